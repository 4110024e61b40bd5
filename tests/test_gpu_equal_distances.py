"""Planes whose search lists are full of equal, nearly equal or zero distances
(computer graphics, ramps): the cut that halves its range between elements, lists
that go to the exact placement of equal keys at once, and lists made exact from
what the approximate distances left. Against the oracle."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

KINDS = ["steps", "speckle", "ramp", "tiles"]


@pytest.fixture(scope="module")
def ctx(bm3d_lib):
    import isp_mw_b200
    c = isp_mw_b200.Context(0)
    yield c
    c.close()


def _plane(kind, h, w):
    rng = np.random.default_rng(11)
    y, x = np.mgrid[0:h, 0:w]
    if kind == "ramp":   # distances depend on the displacement alone, up to rounding
        return (0.0011 * x + 0.0017 * y + 0.1).astype(np.float32)
    if kind == "tiles":  # a repeated pattern: equal blocks, a few distances for the rest
        return rng.integers(0, 4, (6, 5))[y % 6, x % 5].astype(np.float32) / 4
    plane = np.full((h, w), 0.3, np.float32)
    for _ in range(40):  # rectangles of six grey levels
        a, b = rng.integers(0, h), rng.integers(0, w)
        plane[a:a + rng.integers(3, h // 2), b:b + rng.integers(3, w // 2)] = rng.integers(0, 6) / 5
    if kind == "speckle":
        plane[rng.random((h, w)) < 0.02] += 1.0 / 255
    return plane


# GroupSize 17 to 32 cut by the lanes' two smallest; lists of up to 384 places are
# held in registers (BMrange 9), longer ones are read again (12, 16)
@pytest.mark.parametrize("block,bm_range,bm_step,group_size", [
    (8, 9, 1, 16), (8, 9, 1, 17), (8, 9, 2, 16), (8, 12, 1, 5), (8, 16, 1, 16), (8, 16, 1, 24),
    (8, 16, 1, 32), (11, 9, 1, 32), (11, 16, 1, 16), (5, 9, 1, 16), (12, 12, 1, 32)])
@pytest.mark.parametrize("kind", KINDS)
def test_positions_equal_oracle(ctx, oracle_mod, kind, block, bm_range, bm_step, group_size):
    import isp_mw_b200
    plane = _plane(kind, 57, 62)
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.block_size, p.bm_range, p.bm_step, p.group_size = block, bm_range, bm_step, group_size
    for th in (0.05 * p.thMSE, p.thMSE, 1e5):
        p.thMSE = th
        count, pos = ctx.debug_positions(p, False, plane)
        want = oracle_mod.backend("port", np.float32).groups(False, p.as_dict(), plane)
        assert np.array_equal(count, want[0])
        for r, n in enumerate(count):
            assert np.array_equal(pos[r, :n], want[1][r, :n]), (th, r)


# FP64 sums in another order than the oracle's differ in the 16th digit
@pytest.mark.parametrize("block,bm_range,group_size", [(8, 9, 16), (8, 16, 32), (5, 9, 16), (11, 16, 32)])
@pytest.mark.parametrize("wiener", [False, True])
@pytest.mark.parametrize("kind", KINDS)
def test_double_stage_equals_oracle(ctx, oracle_mod, kind, wiener, block, bm_range, group_size):
    import isp_mw_b200
    plane = _plane(kind, 45, 51).astype(np.float64)
    p = isp_mw_b200.stage_params_default("fast", wiener, [30.0] * 3)
    p.block_size, p.bm_range, p.group_size, p.block_step = block, bm_range, group_size, 5
    out = np.empty_like(plane)
    ctx.stage(p, wiener, out, plane)
    want = oracle_mod.backend("port", np.float64).stage(wiener, p.as_dict(), plane)
    want = want[1] if isinstance(want, tuple) else want
    assert np.abs(out - want).max() <= 1e-9
