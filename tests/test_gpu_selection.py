"""Group selection at the edges of its paths, against the oracle.

The search list of a reference block is selected through a cut on distances,
a compacted set ranked by counting, and three rarer paths: equal keys, more
candidates under the cut than the compacted set holds, and keys outside the
normal range. Groups (positions, order and keys) equal the oracle's exactly:
both sides evaluate the same correctly rounded operations.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(bm3d_lib):
    import isp_mw_b200
    c = isp_mw_b200.Context(0)
    yield c
    c.close()


def _plane(kind, h=60, w=53):
    from isp_mw_b200 import synth
    noisy = synth.pair(h, w, 20.0, 17)[1]
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    if kind == "quantised":   # equal keys everywhere
        return (np.round(noisy * 10) / 10).astype(np.float32)
    if kind == "columns":     # the best candidates share a column (or a row below)
        return (np.sin(x) + 0.02 * noisy).astype(np.float32)
    if kind == "rows":
        return (np.sin(y) + 0.02 * noisy).astype(np.float32)
    if kind == "flat":        # many candidates at nearly the cut
        return (0.5 + 1e-6 * noisy).astype(np.float32)
    return noisy


# list lengths below, at and above the 384 places held in registers
# (BMrange 9: 362, 10: 442), groups around the one / two minima rule (17, 18)
@pytest.mark.parametrize("bm_range,group_size", [(1, 16), (9, 2), (9, 16), (9, 17), (9, 18),
                                                 (10, 16), (16, 32), (20, 32)])
@pytest.mark.parametrize("kind", ["noisy", "quantised", "columns", "rows", "flat"])
def test_groups_equal_oracle(ctx, oracle_mod, bm_range, group_size, kind):
    import isp_mw_b200
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.bm_range, p.group_size = bm_range, group_size
    _check(ctx, oracle_mod, p, _plane(kind), 1.0)


@pytest.mark.parametrize("value_range", [1e-18, 1e18])
def test_keys_outside_the_normal_range(ctx, oracle_mod, value_range):
    """A plane far below its nominal range: keys round to few values or none."""
    import isp_mw_b200
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    _check(ctx, oracle_mod, p, _plane("noisy"), value_range)


def _check(ctx, oracle_mod, p, plane, value_range):
    count, pos, keys = ctx.debug_groups(p, False, plane, value_range)
    want = oracle_mod.backend("port", np.float32).groups(False, p.as_dict(), plane, value_range)
    assert np.array_equal(count, want[0])
    for r, n in enumerate(count):
        assert np.array_equal(pos[r, :n], want[1][r, :n]), r
        assert np.array_equal(keys[r, :n], want[2][r, :n]), r


# FP32 lists hold approximate distances where their order decides the group.
# Keys scaled by a power of two to just above the subnormal range keep every
# mantissa but lie where the approximation is not used, so the same call with
# value_range * 2^67 and thMSE * 2^-134 takes exact distances throughout.
@pytest.mark.parametrize("wiener", [False, True])
@pytest.mark.parametrize("bm_range,group_size,shape", [(1, 2, (40, 41)), (3, 16, (24, 71)),
                                                       (9, 16, (8, 8)), (9, 16, (75, 91)),
                                                       (9, 17, (50, 64)), (10, 32, (64, 60)),
                                                       (16, 32, (70, 83))])
def test_approximate_order_equals_exact(ctx, bm_range, group_size, shape, wiener):
    import torch
    import isp_mw_b200
    rng = np.random.default_rng(bm_range * 100 + group_size)
    plane = torch.from_numpy((0.5 + 0.09 * rng.standard_normal(shape)).astype(np.float32)).cuda()
    out = []
    for k in (0, 67):
        p = isp_mw_b200.stage_params_default("fast", wiener, [40.0] * 3)
        p.bm_range, p.group_size, p.block_step = bm_range, group_size, 3
        p.thMSE = 1e4 * 2.0 ** (-2 * k)
        dst = torch.zeros_like(plane)
        ctx.stage(p, wiener, dst, plane, plane.clone() if wiener else None, 2.0 ** k)
        out.append(dst)
        stats = ctx.last_stats()
        assert stats[0] > 0
    assert torch.equal(out[0], out[1])
    assert not torch.equal(out[0], plane)


# 11 x 11 blocks match by the same strips and approximate distances (BMstep 1);
# BMstep 2 takes one candidate a lane.
@pytest.mark.parametrize("bm_range,bm_step,group_size,shape", [(1, 1, 2, (40, 41)), (3, 1, 8, (24, 71)),
                                                               (9, 1, 16, (11, 11)), (9, 2, 16, (60, 53)),
                                                               (9, 1, 17, (75, 91)), (16, 1, 32, (70, 83))])
@pytest.mark.parametrize("kind", ["noisy", "quantised", "flat"])
def test_groups_of_11x11_blocks(ctx, oracle_mod, kind, bm_range, bm_step, group_size, shape):
    import torch
    import isp_mw_b200
    rng = np.random.default_rng(bm_range * 100 + group_size)
    plane = torch.from_numpy((0.5 + 0.09 * rng.standard_normal(shape)).astype(np.float32)).cuda()
    out = []
    for k in (0, 67):  # approximate and exact distances, as above
        p = isp_mw_b200.stage_params_default("vn", False, [40.0] * 3)
        p.block_size, p.block_step, p.group_size = 11, 4, group_size
        p.bm_range, p.bm_step = bm_range, bm_step
        if k == 0:
            _check(ctx, oracle_mod, p, _plane(kind), 1.0)
        p.thMSE = 1e4 * 2.0 ** (-2 * k)
        dst = torch.zeros_like(plane)
        ctx.stage(p, False, dst, plane, None, 2.0 ** k)
        out.append(dst)
    assert torch.equal(out[0], out[1])
    assert not torch.equal(out[0], plane)
