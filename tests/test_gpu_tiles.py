"""The tile shape a call picks from its size changes nothing but the time:
results equal one fixed shape's bit for bit (sums are exact integers), from
one block to several waves of tiles, for one and three planes and for the
profiles of both kernels."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("planes", [1, 3])
@pytest.mark.parametrize("profile,shape", [("fast", (8, 8)), ("fast", (9, 70)), ("fast", (64, 64)),
                                           ("fast", (203, 301)), ("fast", (520, 519)),
                                           ("fast", (720, 1280)), ("lc", (333, 222)),
                                           ("np", (50, 61)), ("np", (220, 230)), ("vn", (130, 90))])
def test_picked_shape_equals_fixed_shape(bm3d_lib, profile, shape, planes):
    import torch
    import isp_mw_b200
    from isp_mw_b200 import synth
    h, w = shape
    src = [torch.from_numpy(synth.pair(h, w, 20.0, 40 + c)[1]).cuda() for c in range(planes)]
    sp = [30.0, 20.0, 20.0]
    b = isp_mw_b200.stage_params_default(profile, False, sp)
    f = isp_mw_b200.stage_params_default(profile, True, sp)
    out = []
    for fixed in (None, (8, 8, 16), (3, 5, 2)):
        ctx = isp_mw_b200.Context(0)
        if fixed:
            ctx.set_tiling(*fixed)
        dst = [torch.zeros_like(p) for p in src]
        if planes == 1:
            ctx.full(b, f, dst[0], src[0])
        else:
            ctx.full3(b, f, dst, src)
        ctx.check()
        out.append(dst)
        ctx.close()
    for other in out[1:]:
        for p, q in zip(out[0], other):
            assert torch.equal(p, q)


@pytest.mark.parametrize("block", [1, 5, 8, 11, 16])
@pytest.mark.parametrize("shape", [(16, 64), (17, 65), (33, 63), (16, 129), (31, 20), (50, 192)])
def test_normalisation_tile_edges(bm3d_lib, oracle_mod, shape, block):
    """One stage at sizes around the normalisation's 64 x 16 tiles, for the
    block sizes its windows hold, against the oracle."""
    import isp_mw_b200
    from isp_mw_b200 import synth
    h, w = shape
    noisy = synth.pair(h, w, 20.0, 5)[1]
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.block_size, p.block_step, p.group_size, p.bm_range = block, max(1, block // 2), 4, 3
    ctx = isp_mw_b200.Context(0)
    out = np.empty_like(noisy)
    ctx.stage(p, False, out, noisy)
    ctx.close()
    want = oracle_mod.backend("port", np.float32).stage(False, p.as_dict(), noisy)
    want = want[1] if isinstance(want, tuple) else want
    assert np.abs(out - want).max() <= 1e-3


@pytest.mark.parametrize("wiener", [False, True])
@pytest.mark.parametrize("group_size,thmse", [(17, 1500.0), (24, 900.0), (31, 1e5), (32, 1200.0), (32, 1e5)])
def test_groups_of_up_to_32(bm3d_lib, oracle_mod, group_size, thmse, wiener):
    """Group lengths of the generic kernel's 8 x 8 path: full groups of 32 and
    every shorter length that a tight threshold leaves, against the oracle."""
    import isp_mw_b200
    from isp_mw_b200 import synth
    noisy = synth.pair(58, 67, 20.0, 9)[1]
    guide = synth.pair(58, 67, 8.0, 9)[1] if wiener else noisy
    p = isp_mw_b200.stage_params_default("np", wiener, [34.0] * 3)
    p.group_size, p.thMSE = group_size, thmse * (0.2 if wiener and thmse < 1e4 else 1.0)
    ctx = isp_mw_b200.Context(0)
    out = np.empty_like(noisy)
    ctx.stage(p, wiener, out, noisy, guide)
    ctx.close()
    want = oracle_mod.backend("port", np.float32).stage(wiener, p.as_dict(), noisy, guide)
    want = want[1] if isinstance(want, tuple) else want
    assert np.abs(out - want).max() <= 1e-3


# The limit on the search range does not move with the kernels' layouts: the
# largest range taken and the next, by stage_limit_bytes' sum for these parameters
# (one plane, fast profile, 1 x 1 tile: 20 B a window pixel and 8 B a list place;
# batches: 2 x 2 tile). Whole images smaller than the window leave room for more.
@pytest.mark.parametrize("shape,bm_range,ok", [((300, 310), 42, True), ((300, 310), 43, False),
                                               ((40, 300), 60, True), ((40, 300), 90, False)])
def test_search_range_limit(bm3d_lib, shape, bm_range, ok):
    import torch
    import isp_mw_b200
    from isp_mw_b200 import synth
    h, w = shape
    src = torch.from_numpy(synth.pair(h, w, 20.0, 3)[1]).cuda()
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.bm_range, p.block_step = bm_range, 32
    dst = torch.zeros_like(src)
    ctx = isp_mw_b200.Context(0)
    if ok:
        ctx.stage(p, False, dst, src)
        ctx.check()
        assert not torch.equal(dst, torch.zeros_like(dst))
    else:
        with pytest.raises(isp_mw_b200.BM3DError) as e:
            ctx.stage(p, False, dst, src)
        assert e.value.code == isp_mw_b200.BM3D_ERR_UNSUPPORTED
    ctx.close()


@pytest.mark.parametrize("planes", [1, 3])
@pytest.mark.parametrize("block,bm_range", [(8, 1), (8, 32), (11, 9), (11, 30), (5, 1), (5, 32)])
def test_groups_of_one_have_no_search_list(bm3d_lib, oracle_mod, block, bm_range, planes):
    """Groups of one match nothing, at any BMrange within the limit: single calls
    and batches agree bit for bit, and with the oracle."""
    import torch
    import isp_mw_b200
    from isp_mw_b200 import synth
    noisy = [synth.pair(83, 97, 20.0, 3 + c)[1] for c in range(planes)]
    src = [torch.from_numpy(p).cuda() for p in noisy]
    ctx = isp_mw_b200.Context(0)
    b, f = (isp_mw_b200.stage_params_default("fast", w, [30.0] * 3) for w in (False, True))
    for p in (b, f):
        p.block_size, p.group_size, p.bm_range, p.block_step = block, 1, bm_range, block - 1
    dst = [torch.zeros_like(p) for p in src]
    if planes == 1:
        ctx.full(b, f, dst[0], src[0])
    else:
        ctx.full3(b, f, dst, src)
    ctx.check()
    other = [torch.zeros_like(p) for p in src]
    batch = isp_mw_b200.Batch(ctx, [b], [f], other if planes == 1 else [other], src if planes == 1 else [src])
    batch.run()
    batch.check()
    batch.close()
    assert all(torch.equal(p, q) for p, q in zip(dst, other))
    if planes == 1:
        _, want = oracle_mod.backend("port", np.float32).full(b.as_dict(), f.as_dict(), noisy[0])
        assert np.abs(dst[0].cpu().numpy() - want).max() <= 1e-3
    ctx.close()


# block sizes without a kernel of their own: one tile of 2 x 2 reference blocks,
# some, and enough for the shape of 6 x 4 on 12 warps; FP64 to the 9th digit
@pytest.mark.parametrize("shape", [(19, 20), (60, 49), (150, 161)])
@pytest.mark.parametrize("block,step,group_size", [(1, 1, 4), (2, 1, 32), (4, 3, 17), (7, 4, 16), (9, 5, 8), (16, 9, 32)])
@pytest.mark.parametrize("wiener", [False, True])
def test_block_sizes_at_picked_shapes(bm3d_lib, oracle_mod, shape, block, step, group_size, wiener):
    import isp_mw_b200
    from isp_mw_b200 import synth
    p = isp_mw_b200.stage_params_default("fast", wiener, [30.0] * 3)
    p.block_size, p.block_step, p.group_size, p.bm_range = block, step, group_size, 3
    noisy = synth.pair(*shape, 20.0, 5)[1]
    ctx = isp_mw_b200.Context(0)
    for dtype, tol in ((np.float32, 1e-3), (np.float64, 1e-9)):
        src = noisy.astype(dtype)
        out = np.empty_like(src)
        ctx.stage(p, wiener, out, src)
        want = oracle_mod.backend("port", dtype).stage(wiener, p.as_dict(), src)
        want = want[1] if isinstance(want, tuple) else want
        assert np.abs(out - want).max() <= tol
    ctx.close()
