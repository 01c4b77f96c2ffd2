"""Pageable host frames, staged in chunks by one thread (below 32 MB) or by
several, against the same frames on the device.  Chunks change the tiles of a
launch, so FP64 sums may round differently: 1e-9 A; moved coordinates are
float32 of the same transforms: one ulp of the largest coordinate."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("frames,atoms", [(7, 1001), (700, 1000), (1500, 1001), (330, 9001), (3, 1000003)])
def test_host_frames_equal_device_frames(frames, atoms):
    import torch
    from warp_md import _native as N

    ctx = N.context(0)
    rng = np.random.default_rng(atoms)
    ref = (30 * rng.standard_normal((atoms, 3))).astype(np.float32)
    host = ref + rng.standard_normal((frames, atoms, 3), dtype=np.float32)
    dev = torch.from_numpy(host).cuda()
    r = N.Reference.from_numpy(ctx, ref)
    res = []
    for x in (host.ctypes.data, dev.data_ptr()):
        out = np.empty(frames)
        moved = np.empty_like(host)
        xf = np.empty((frames, 12), np.float32)
        ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x, frames, atoms, 3, None, atoms, r.handle, 1, out.ctypes.data, None))
        ctx.check(ctx.lib.wmd_superpose(ctx.handle, x, frames, atoms, 3, None, atoms, r.handle, 0, moved.ctypes.data,
                                        xf.ctypes.data, None))
        res.append((out, moved))
    np.testing.assert_allclose(res[0][0], res[1][0], rtol=0, atol=1e-9)
    assert np.abs(res[0][1] - res[1][1]).max() <= np.spacing(np.abs(res[1][1]).max())
