"""Groups as the FP32 stages find them (positions without keys), against the
oracle. The stages decide by approximate distances wherever these are enough;
positions and their order equal the oracle's exactly all the same, because
whatever the approximation cannot tell is decided by exact distances."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx(bm3d_lib):
    import isp_mw_b200
    c = isp_mw_b200.Context(0)
    yield c
    c.close()


def _check(ctx, oracle_mod, p, plane, value_range=1.0):
    """Returns the oracle's group sizes."""
    plane = np.ascontiguousarray(plane, np.float32)
    count, pos = ctx.debug_positions(p, False, plane, value_range)
    want = oracle_mod.backend("port", np.float32).groups(False, p.as_dict(), plane, value_range)
    assert np.array_equal(count, want[0])
    for r, n in enumerate(count):
        assert np.array_equal(pos[r, :n], want[1][r, :n]), r
    return want[0]


def _one_column(block, amplitude, h=47):
    """Blocks match along their own column only: constant columns of 1 at
    irregular places, noise of the given amplitude between them. The plane has
    16 columns of blocks, so the candidates fall to two of a warp's lanes."""
    w = block + 15
    rng = np.random.default_rng(8)
    plane = (amplitude * rng.random((h, w))).astype(np.float32)
    plane[:, [1, 4, 5, 9, 11, 12, 18, 20]] = 1.0
    return plane


# Keys are distances over a power of the value range: far from the usual ranges,
# distances that differ have keys that are subnormal or zero and tie, and ties
# go by list order or std::partial_sort's heap
@pytest.mark.parametrize("value_range", [1.0, 1e10, 1e13, 1e16, 1e18])
@pytest.mark.parametrize("key", [1e-44, 1e-46])
@pytest.mark.parametrize("block,group_size", [(8, 8), (8, 16), (8, 32), (11, 16), (11, 32)])
def test_keys_below_the_normal_range(ctx, oracle_mod, block, group_size, key, value_range):
    import isp_mw_b200
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.block_size, p.group_size, p.block_step, p.bm_range = block, group_size, 5, 16
    scale = block * block * value_range ** 2 / 255.0 ** 2
    p.thMSE = 0.5 * np.sqrt(3.0) / scale  # distances up to 1 / 2
    plane = _one_column(block, np.sqrt(6 * key * scale) / block)
    assert (_check(ctx, oracle_mod, p, plane, value_range) > 1).any() or value_range == 1.0


def _plane(kind, h=60, w=53):
    from isp_mw_b200 import synth
    noisy = synth.pair(h, w, 20.0, 17)[1]
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    if kind == "quantised":   # equal keys everywhere
        return (np.round(noisy * 10) / 10).astype(np.float32)
    if kind == "eight_bit":   # some equal keys
        return (np.round(noisy * 255) / 255).astype(np.float32)
    if kind == "columns":     # the best candidates share a column (or a row below)
        return (np.sin(x) + 0.02 * noisy).astype(np.float32)
    if kind == "rows":
        return (np.sin(y) + 0.02 * noisy).astype(np.float32)
    if kind == "flat":        # many candidates at nearly the cut
        return (0.5 + 1e-6 * noisy).astype(np.float32)
    return noisy


# thresholds that reject most of a list, a part of it and none of it; 8 x 8 and
# 11 x 11 blocks, every BMstep (1: strips of candidates; else one a lane)
@pytest.mark.parametrize("block,bm_range,bm_step,group_size", [
    (8, 1, 1, 16), (8, 9, 1, 2), (8, 9, 1, 16), (8, 9, 1, 17), (8, 9, 1, 18), (8, 10, 1, 16),
    (8, 16, 1, 32), (8, 9, 2, 16), (8, 10, 3, 16), (8, 16, 2, 32), (11, 3, 1, 8), (11, 9, 1, 16),
    (11, 9, 2, 16), (11, 16, 1, 32), (5, 9, 1, 16)])
@pytest.mark.parametrize("kind", ["noisy", "quantised", "eight_bit", "columns", "rows", "flat"])
def test_positions_equal_oracle(ctx, oracle_mod, kind, block, bm_range, bm_step, group_size):
    import isp_mw_b200
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.block_size, p.bm_range, p.bm_step, p.group_size = block, bm_range, bm_step, group_size
    for th in (0.3 * p.thMSE, p.thMSE, 1e5):
        p.thMSE = th
        _check(ctx, oracle_mod, p, _plane(kind))


def _set_threshold(p, block, distance):
    """thMSE whose sum-of-squares threshold is the float `distance`."""
    norm = 1.0 / np.sqrt(3.0)
    scale = float(block * block) / (255.0 * 255.0)
    p.thMSE = float(distance) / scale / norm
    while np.float32(p.thMSE * norm * scale) < distance:
        p.thMSE = np.nextafter(p.thMSE, np.inf)
    while np.float32(p.thMSE * norm * scale) > distance:
        p.thMSE = np.nextafter(p.thMSE, 0.0)


# A candidate exactly at the threshold is taken, one past it is not: the threshold
# put on a distance of the list and one unit to either side
@pytest.mark.parametrize("block,group_size", [(8, 16), (8, 32), (11, 16)])
@pytest.mark.parametrize("rank", [3, 12, 60])
def test_distances_at_the_threshold(ctx, oracle_mod, block, group_size, rank):
    import isp_mw_b200
    plane = _plane("noisy", 44, 46)
    y0, x0 = 16, 16
    ref = plane[y0:y0 + block, x0:x0 + block]
    dist = []
    for dy in range(-9, 10):
        for dx in range(-9, 10):
            d = np.float32(0)
            for r, c in zip(ref.ravel(), plane[y0 + dy:y0 + dy + block, x0 + dx:x0 + dx + block].ravel()):
                e = np.float32(r - c)
                d = np.float32(d + np.float32(e * e))  # the reference's order
            dist.append(d)
    at = np.sort(np.array(dist, np.float32))[rank]
    p = isp_mw_b200.stage_params_default("fast", False, [30.0] * 3)
    p.block_size, p.block_step, p.group_size = block, 8, group_size
    sizes = []
    for d in (np.nextafter(at, np.float32(0)), at, np.nextafter(at, np.float32(np.inf))):
        _set_threshold(p, block, d)
        sizes.append(_check(ctx, oracle_mod, p, plane).sum())
    if rank < group_size:  # that one candidate is the difference
        assert sizes[1] == sizes[0] + 1
