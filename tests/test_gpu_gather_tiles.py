"""Gathered statistics with tiles chosen by size: list lengths around the tiles and
sub-chunks, enough frames that a warp takes several items, scattered and repeated
indices, unaligned bases; RMSD (fit and no fit) and weighted transforms against the
oracle.

Tolerances: FP64 sums in different orders, 1e-9 A on the RMSD; transforms are written
in float32 (rotation 1e-6, the superposition bar, translation of up to ~100 A 2e-5)."""

import numpy as np
import pytest

import oracle
from warp_md import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("stride", [3, 4])
@pytest.mark.parametrize("frames,atoms,n_sel", [(593, 400, 63), (700, 400, 65), (9000, 300, 127), (5000, 300, 129),
                                                (601, 1500, 1023), (2500, 1500, 1025), (1201, 3001, 2049)])
def test_gathered(frames, atoms, n_sel, stride):
    from warp_md import _native as N

    fr, ref = synth.make_trajectory(atoms, frames, (0.1, 2.0), 11 + n_sel)
    rng = np.random.default_rng(n_sel)
    sel = rng.integers(0, atoms, n_sel).astype(np.uint32)
    sel[0], sel[-1] = atoms - 1, 0
    w = rng.uniform(0.5, 20.0, n_sel).astype(np.float32)
    data = fr if stride == 3 else np.concatenate([fr, np.full(fr.shape[:2] + (1,), 7.0, np.float32)], axis=2)
    flat = torch.zeros(data.size + 1, device="cuda")
    flat[1:] = torch.from_numpy(np.ascontiguousarray(data)).reshape(-1).cuda()
    x = flat[1:]  # 4 bytes off 16-byte alignment
    dsel = torch.from_numpy(sel.astype(np.int32)).cuda()
    ctx = N.context(0)
    r, rw = N.Reference.from_numpy(ctx, ref[sel]), N.Reference.from_numpy(ctx, ref[sel], weights=w)
    try:
        for align in (1, 0):
            out = torch.full((frames,), -1.0, dtype=torch.float64, device="cuda")
            ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x.data_ptr(), frames, atoms, stride, dsel.data_ptr(), n_sel,
                                              r.handle, align, out.data_ptr(), None))
            torch.cuda.synchronize()
            _, want = oracle.rmsd_frames(fr, ref[sel], selection=sel, align=bool(align))
            np.testing.assert_allclose(out.cpu().numpy(), want, rtol=0, atol=1e-9)
        rows = torch.empty(frames, 12, device="cuda")
        ctx.check(ctx.lib.wmd_superpose_transforms(ctx.handle, x.data_ptr(), frames, atoms, stride, dsel.data_ptr(),
                                                   n_sel, rw.handle, 0, rows.data_ptr(), None))
        torch.cuda.synchronize()
    finally:
        r.close()
        rw.close()
    got = rows.cpu().numpy().astype(np.float64)
    want, _ = oracle.superpose(fr, ref[sel], selection=sel, weights=w, apply=False)
    np.testing.assert_allclose(got[:, :9], want[:, :9], rtol=0, atol=1e-6)
    np.testing.assert_allclose(got[:, 9:], want[:, 9:], rtol=0, atol=2e-5)
