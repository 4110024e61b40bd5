"""Batches of every GroupSize: the launch's shared memory follows the layout
that the kernel works out for itself, so each plane of a batch equals the
single call bit for bit and no tile is left out."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


# 8 x 8 blocks of up to 16 run on the register-resident kernel, the rest on the
# generic ones; basic and final stage differ, as the profiles' do
@pytest.mark.parametrize("planes", [1, 3])
@pytest.mark.parametrize("basic,final", [((8, 1), (8, 32)), ((8, 2), (8, 2)), ((8, 7), (8, 16)),
                                         ((8, 8), (8, 15)), ((8, 15), (8, 17)), ((8, 16), (11, 5)),
                                         ((11, 2), (8, 3)), ((5, 3), (8, 8)), ((8, 24), (8, 1))])
def test_batch_equals_single_calls(bm3d_lib, basic, final, planes):
    import torch
    import isp_mw_b200
    from isp_mw_b200 import synth
    ctx = isp_mw_b200.Context(0)
    shapes = [(40, 53), (17, 90), (71, 36)]
    sigma = [30.0, 20.0, 25.0]
    b = isp_mw_b200.stage_params_default("fast", False, sigma)
    f = isp_mw_b200.stage_params_default("fast", True, sigma)
    b.block_size, b.group_size, b.block_step = basic + (5,)
    f.block_size, f.group_size, f.block_step = final + (4,)
    src = [[torch.from_numpy(synth.pair(h, w, 20.0, 7 * i + c)[1]).cuda() for c in range(planes)]
           for i, (h, w) in enumerate(shapes)]
    want = [[torch.zeros_like(p) for p in image] for image in src]
    for d, s in zip(want, src):
        if planes == 3:
            ctx.full3(b, f, d, s)
        else:
            ctx.full(b, f, d[0], s[0])
    ctx.check()
    flat = (lambda x: x) if planes == 3 else (lambda x: [i[0] for i in x])
    for autotune in (False, True):
        got = [[torch.full_like(p, -1.0) for p in image] for image in src]
        batch = isp_mw_b200.Batch(ctx, [b] * 3, [f] * 3, flat(got), flat(src), autotune=autotune)
        batch.run()
        batch.check()
        batch.close()
        for x, y in zip(got, want):
            assert all(torch.equal(p, q) for p, q in zip(x, y))
    host = [[p.cpu().numpy() for p in image] for image in src]
    got = [[np.full_like(p, -1.0) for p in image] for image in host]
    hb = isp_mw_b200.HostBatch(ctx, [b] * 3, [f] * 3, shapes, planes=planes)
    hb.run(flat(got), flat(host))
    hb.close()
    for x, y in zip(got, want):
        assert all(np.array_equal(p, q.cpu().numpy()) for p, q in zip(x, y))
    ctx.close()
