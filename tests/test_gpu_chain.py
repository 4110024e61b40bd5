"""The combined call's basic stage prepares its final stage (sums, counts, the
estimate's non-finite pixels). Results equal the two stages called one after
the other, bit for bit: with non-finite inputs, planes left out by their noise
level, a reference of its own, and sizes that change from call to call."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _planes(n, h, w, kind):
    import torch
    from isp_mw_b200 import synth
    out = []
    for c in range(n):
        p = synth.pair(h, w, 20.0, 70 + c)[1]
        if kind == "nan" and c != 1:
            p = p.copy()
            p[h // 2, w // 3], p[0, 0], p[-1, -1] = np.nan, np.inf, -np.inf
        out.append(torch.from_numpy(p).cuda())
    return out


@pytest.mark.parametrize("profile", ["fast", "vn"])
@pytest.mark.parametrize("kind", ["plain", "nan"])
@pytest.mark.parametrize("sigma", [[30.0, 20.0, 20.0], [30.0, 0.0, 20.0]])
def test_combined_equals_stages(bm3d_lib, profile, kind, sigma):
    import torch
    import isp_mw_b200
    ctx = isp_mw_b200.Context(0)
    b = isp_mw_b200.stage_params_default(profile, False, sigma)
    f = isp_mw_b200.stage_params_default(profile, True, sigma)
    same = lambda x, y: np.array_equal(x.cpu().numpy(), y.cpu().numpy(), equal_nan=True)
    for (h, w) in ((40, 61), (90, 128), (33, 40), (64, 17)):
        src = _planes(3, h, w, kind)
        got = [torch.zeros_like(p) for p in src]
        ctx.full3(b, f, got, src)
        est, want = [p.clone() for p in src], [p.clone() for p in src]
        ctx.stage3(b, False, est, src)
        ctx.stage3(f, True, want, src, est)
        ctx.check()
        assert all(same(x, y) for x, y in zip(got, want))
        ref = _planes(2, h, w, "plain")[1]
        for r in (None, ref):
            got1, est1, want1 = (torch.zeros_like(src[0]) for _ in range(3))
            ctx.full(b, f, got1, src[0], ref=r)
            ctx.stage(b, False, est1, src[0], r)
            ctx.stage(f, True, want1, src[0], est1)
            assert same(got1, want1)
    ctx.close()


def test_no_plane_to_filter(bm3d_lib):
    """Noise levels that are no numbers pass the parameter guard and select no
    plane: the combined call copies, a stage leaves dst alone, in batches too."""
    import torch
    import isp_mw_b200
    ctx = isp_mw_b200.Context(0)
    b = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    f = isp_mw_b200.stage_params_default("fast", True, [30.0] * 3)
    for p in (b, f):
        p.sigma[0], p.sigma[1], p.sigma[2] = float("nan"), 0.0, float("nan")
    src = _planes(3, 40, 61, "plain")
    dst = [torch.full_like(p, -1.0) for p in src]
    for wiener, p in ((False, b), (True, f)):
        ctx.stage3(p, wiener, dst, src)
        assert all(bool((d == -1.0).all()) for d in dst)
    counts = ctx.last_stats()  # the final stage's alone, as after a combined call
    ctx.full3(b, f, dst, src)
    ctx.check()
    assert all(torch.equal(d, s) for d, s in zip(dst, src)) and ctx.last_stats() == counts
    dst = [torch.full_like(p, -1.0) for p in src]
    batch = isp_mw_b200.Batch(ctx, [b], [f], [dst], [src])
    batch.run()
    batch.check()
    batch.close()
    assert all(torch.equal(d, s) for d, s in zip(dst, src))
    ctx.close()


@pytest.mark.parametrize("planes", [1, 3])
def test_no_room_for_the_next_stage_sums(bm3d_lib, planes):
    """Without room for the final stage's own weight sums the stages run one
    after the other: same results, no error, in single calls and batches."""
    import torch
    import isp_mw_b200
    b = isp_mw_b200.stage_params_default("fast", False, [30.0, 20.0, 20.0])
    f = isp_mw_b200.stage_params_default("fast", True, [30.0, 20.0, 20.0])
    src = _planes(planes, 90, 128, "nan")
    same = lambda x, y: all(np.array_equal(p.cpu().numpy(), q.cpu().numpy(), equal_nan=True)
                            for p, q in zip(x, y))
    one = (lambda x: x) if planes == 3 else (lambda x: x[0])
    call = lambda c, *args: (c.full3 if planes == 3 else c.full)(*args)
    ctx = isp_mw_b200.Context(0)
    want = [torch.zeros_like(p) for p in src]
    call(ctx, b, f, one(want), one(src))
    copied = isp_mw_b200.stage_params_default("fast", True, [0.0] * 3)
    short = isp_mw_b200.Context(0)
    got = [torch.zeros_like(p) for p in src]
    call(short, b, copied, one(got), one(src))  # every buffer but those sums
    try:
        for skip in range(planes):
            bm3d_lib.bm3d_inject_alloc_failures_after(skip, 1)
            got = [torch.zeros_like(p) for p in src]
            call(short, b, f, one(got), one(src))
            assert same(got, want)
            bm3d_lib.bm3d_inject_alloc_failures(0)
            short.close()
            short = isp_mw_b200.Context(0)
            call(short, b, copied, one(got), one(src))
        # captured with those sums missing: nothing to allocate
        stream = torch.cuda.Stream()
        got = [torch.zeros_like(p) for p in src]
        torch.cuda.synchronize()
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=stream):
            call(short, b, f, one(got), one(src))
        graph.replay()
        torch.cuda.synchronize()
        assert same(got, want)
        # a batch: estimates, state, marks and consistency counter come first
        got = [torch.zeros_like(p) for p in src]
        bm3d_lib.bm3d_inject_alloc_failures_after(4, 1)
        batch = isp_mw_b200.Batch(ctx, [b], [f], [one(got)], [one(src)])
        batch.run()
        batch.check()
        batch.close()
        assert same(got, want)
    finally:
        bm3d_lib.bm3d_inject_alloc_failures(0)
        short.close()
        ctx.close()
