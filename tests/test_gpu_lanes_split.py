"""The frames-across-lanes kernel's split: runs that end inside a group, on its edge and
inside one stage, whole groups in one warp, groups added by the last warp and by the
second kernel, frames past the last quad row (1, 2 and 3), batches of frames and sums
left for the superposition; against the FP64 oracle.

Tolerance: FP64 sums in different orders, 1e-9 A on the RMSD; transforms in float32
(rotation 1e-6, the superposition bar, translation 2e-5)."""

import numpy as np
import pytest

import oracle
from warp_md import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stride,frames,atoms", [
    (3, 8000, 33),      # 2 stages a group, whole groups
    (3, 37888, 32),     # one stage a group, one group a warp
    (3, 40000, 36),     # more groups than warps
    (3, 4700, 500),     # few stages a warp
    (3, 3333, 1030),    # quad rows, 1 frame past them
    (3, 2402, 2051),    # 2 past
    (3, 2399, 2500),    # 3... and a last group of 31 frames
    (3, 1003, 9001),    # the second kernel, 3 frames past the quad rows
    (3, 257, 20000),    # 9 groups, the last of one frame
    (4, 3000, 1500),    # xyzw
    (4, 700, 5000),     # xyzw, second kernel
])
def test_split(stride, frames, atoms):
    from warp_md import _native as N

    fr, ref = synth.make_trajectory(atoms, frames, (0.1, 2.0), 17 + atoms)
    fr[frames - 1] = ref
    data = fr if stride == 3 else np.concatenate([fr, np.full(fr.shape[:2] + (1,), 3.0, np.float32)], axis=2)
    x = torch.from_numpy(np.ascontiguousarray(data)).cuda()
    w = np.random.default_rng(1).uniform(0.5, 20.0, atoms).astype(np.float32)
    ctx = N.context(0)
    r, rw = N.Reference.from_numpy(ctx, ref), N.Reference.from_numpy(ctx, ref, weights=w)

    def run(align):
        out = torch.full((frames,), -1.0, dtype=torch.float64, device="cuda")
        ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x.data_ptr(), frames, atoms, stride, None, atoms, r.handle, align,
                                          out.data_ptr(), None))
        torch.cuda.synchronize()
        return out.cpu().numpy()

    try:
        for align in (1, 0):
            got = run(align)
            _, want = oracle.rmsd_frames(fr, ref, align=bool(align))
            np.testing.assert_allclose(got[:-1], want[:-1], rtol=0, atol=1e-9)
            assert got[-1] < 1e-7
            assert np.array_equal(got, run(align))  # the same bits again
        for ref_handle, weights in ((r, None), (rw, w)):
            rows = torch.empty(frames, 12, device="cuda")
            ctx.check(ctx.lib.wmd_superpose_transforms(ctx.handle, x.data_ptr(), frames, atoms, stride, None, atoms,
                                                       ref_handle.handle, 0, rows.data_ptr(), None))
            torch.cuda.synchronize()
            got = rows.cpu().numpy()
            want, _ = oracle.superpose(fr, ref, weights=weights, apply=False)
            np.testing.assert_allclose(got[:, :9], want[:, :9], rtol=0, atol=1e-6)
            np.testing.assert_allclose(got[:, 9:], want[:, 9:], rtol=0, atol=2e-5)
    finally:
        r.close()
        rw.close()
