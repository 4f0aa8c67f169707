"""The router of routed experts, whose warps hold 2048 of a row's weights at once, or sixteen of a lane's where rows are many or narrow: widths around that and
around a warp, fewer and more experts than warps, all three scores, both input types, against 64 bits; both forms on either side of the line between them; and the
chain of router and experts, whose kernels start before their predecessors have ended."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width", [1, 33, 2047, 2048, 2049, 4128])
@pytest.mark.parametrize("experts,top", [(2, 1), (8, 2), (19, 6)])
@pytest.mark.parametrize("score,bias,dtype", [(0, False, "f32"), (1, True, "bf16"), (2, True, "f32")])
def test_route_scored_matches_float64(width, experts, top, score, bias, dtype):
    import torch
    from lmdeploy_b200 import _hybrid_lib as H
    lib, n = H.load(), 5
    g = torch.Generator(device="cuda").manual_seed(width + experts)
    T, dt = (torch.float32, H.F32) if dtype == "f32" else (torch.bfloat16, H.BF16)
    x = torch.randn(n, width, generator=g, device="cuda").to(T)
    # logits a step apart, so that the choice is the same in any arithmetic
    router = torch.randn(experts, width, generator=g, device="cuda") * (1e-3 / width ** 0.5)
    steps = torch.randperm(experts, generator=g, device="cuda").float() * 0.25
    shift = steps if bias else None
    if not bias:
        x[:, 0], router[:, 0] = 1.0, steps
    ids, wts = torch.full((n, top), -1, dtype=torch.int32, device="cuda"), torch.empty(n, top, device="cuda")
    H.check(lib.b200h_route_scored(x.data_ptr(), dt, router.data_ptr(), shift.data_ptr() if bias else None, n, width, experts, top, score, ids.data_ptr(), wts.data_ptr(),
                                   torch.cuda.current_stream().cuda_stream), "route")
    z = x.double() @ router.double().T + (shift.double() if bias else 0.0)
    best, at = z.topk(top, -1)
    want = z.softmax(-1).gather(1, at) if score == 0 else best.sigmoid() if score == 1 else best.softmax(-1)
    assert (ids.long() == at).all()
    # float sums of `width` products of about 1e-3 / sqrt(width), and the exponential of a logit of up to five
    assert ((wts.double() - want).abs() <= 2e-6 * want + 1e-7).all()


# rows x width x experts on either side of where the form changes: 3 / 4 of the width, or any number of rows for many experts
@pytest.mark.parametrize("rows,width,experts", [(192, 256, 8), (193, 256, 8), (191, 255, 9), (1056, 1408, 16), (1057, 1408, 16), (1057, 1408, 24), (769, 1024, 63), (769, 1024, 64), (1537, 2048, 8), (1537, 2048, 16)])
@pytest.mark.parametrize("dtype", ["f32", "bf16"])
def test_a_row_does_not_depend_on_the_rows_beside_it(rows, width, experts, dtype):
    import torch
    from lmdeploy_b200 import _hybrid_lib as H
    lib, top = H.load(), 3
    g = torch.Generator(device="cuda").manual_seed(rows + width)
    T, dt = (torch.float32, H.F32) if dtype == "f32" else (torch.bfloat16, H.BF16)
    x, router = torch.randn(rows, width, generator=g, device="cuda").to(T), torch.randn(experts, width, generator=g, device="cuda") * width ** -0.5

    def route(x):
        ids, wts = torch.full((len(x), top), -1, dtype=torch.int32, device="cuda"), torch.empty(len(x), top, device="cuda")
        H.check(lib.b200h_route_scored(x.data_ptr(), dt, router.data_ptr(), None, len(x), width, experts, top, 2, ids.data_ptr(), wts.data_ptr(),
                                       torch.cuda.current_stream().cuda_stream), "route")
        return ids, wts

    (ids, wts), parts = route(x), [route(x[i:i + 100].contiguous()) for i in range(0, rows, 100)]
    assert torch.equal(ids, torch.cat([p[0] for p in parts])) and torch.equal(wts, torch.cat([p[1] for p in parts]))


def test_a_narrow_router_costs_less_than_a_wide_one():
    """4096 rows, 128 experts: an eighth of the width takes 0.36 of the time, and 0.98 where every width takes as many steps."""
    import torch
    from lmdeploy_b200 import _hybrid_lib as H
    lib, n, E, top = H.load(), 4096, 128, 8
    ids, wts = torch.empty(n, top, dtype=torch.int32, device="cuda"), torch.empty(n, top, device="cuda")
    best = {}
    for width in (64, 512):
        x, router = torch.randn(n, width, device="cuda"), torch.randn(E, width, device="cuda") * width ** -0.5
        for i in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(4):
                H.check(lib.b200h_route_scored(x.data_ptr(), H.F32, router.data_ptr(), None, n, width, E, top, 2, ids.data_ptr(), wts.data_ptr(),
                                               torch.cuda.current_stream().cuda_stream), "route")
            b.record()
            torch.cuda.synchronize()
            best[width] = min(best.get(width, 1e9), a.elapsed_time(b))
    assert best[64] <= 0.7 * best[512], best


@pytest.mark.parametrize("rows", [1, 12, 32])
def test_router_and_experts_in_a_row_agree_with_each_alone(rows):
    """The same calls with everything drained in between, many times over: a kernel that read its input early would show."""
    import torch
    from lmdeploy_b200 import _hybrid_lib as H
    import ctypes as C
    lib, W, ff, E, top = H.load(), 512, 384, 8, 2
    g = torch.Generator(device="cuda").manual_seed(rows)
    rand = lambda *s: torch.randn(*s, generator=g, device="cuda")  # noqa: E731
    router, gate, up, down = rand(E, W), rand(E, ff, W).mul(W ** -0.5).bfloat16(), rand(E, ff, W).mul(W ** -0.5).bfloat16(), rand(E, W, ff).mul(ff ** -0.5).bfloat16()
    xs = [rand(rows, W) for _ in range(6)]
    ids, wts = torch.empty(rows, top, dtype=torch.int32, device="cuda"), torch.empty(rows, top, device="cuda")
    mid, lists = torch.empty(rows * top, ff, dtype=torch.bfloat16, device="cuda"), torch.empty(E * (rows * top + 1), dtype=torch.int32, device="cuda")
    xt, out = torch.empty(rows, W, dtype=torch.bfloat16, device="cuda"), torch.empty(rows, top, W, device="cuda")

    def step(x, drain):
        st = torch.cuda.current_stream().cuda_stream
        xt.copy_(x)
        H.check(lib.b200h_route_scored(x.data_ptr(), H.F32, router.data_ptr(), None, rows, W, E, top, 2, ids.data_ptr(), wts.data_ptr(), st), "route")
        if drain:
            torch.cuda.synchronize()
        a = H.ExpertArgs(n=rows, width=W, ff=ff, experts=E, top=top, dtype=H.BF16, act=H.EXPERT_ACT["silu_gate"], scale_input=0)
        a.x, a.gate, a.up, a.down, a.ids, a.wts, a.out = (t.data_ptr() for t in (xt, gate, up, down, ids, wts, out))
        a.mid, a.counts, a.lists, a.stream = mid.data_ptr(), lists.data_ptr(), lists.data_ptr() + 4 * E, st
        H.check(lib.b200h_experts(C.byref(a)), "experts")
        return out.clone()

    alone = [step(x, True) for x in xs]
    chained = [step(x, False) for _ in range(5) for x in xs]
    torch.cuda.synchronize()
    assert all(torch.equal(y, alone[i % len(xs)]) for i, y in enumerate(chained))
