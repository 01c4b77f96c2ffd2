"""One CTA per frame for launches too small to fill the GPU: RMSD, its frame
records and its gradient at the kernel's edges and on both sides of the rule's
lines, against the FP64 oracle.

Tolerances: FP64 sums in different orders put lambda off by a few eps of G, so 1e-9 A
(deviations from 0.1 A, coordinates within ~100 A), 1e-7 A where the RMSD is near
zero; the gradient is rounded to float32 once (2^-23 relative, 1e-9 for its zeros)."""

import numpy as np
import pytest

import oracle
from warp_md import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("align", [1, 0])
@pytest.mark.parametrize("stride", [3, 4])
@pytest.mark.parametrize("frames,atoms", [(1, 1), (2, 3), (592, 31), (593, 31), (5, 257), (147, 8192), (9, 8193)])
def test_forward(frames, atoms, stride, align):
    from warp_md import _native as N

    fr, ref = synth.make_trajectory(atoms, frames, (0.1, 2.0), 3 + atoms)
    if frames > 1:
        fr[1] = ref
    data = fr if stride == 3 else np.concatenate([fr, np.full(fr.shape[:2] + (1,), 9.0, np.float32)], axis=2)
    flat = torch.zeros(data.size + 1, device="cuda")
    flat[1:] = torch.from_numpy(np.ascontiguousarray(data)).reshape(-1).cuda()
    sel = np.arange(0, atoms, 2, dtype=np.uint32)[::-1].copy()
    ctx = N.context(0)
    for x, s in ((flat[1:].clone(), None), (flat[1:], None), (flat[1:], sel)):
        r = ref if s is None else np.ascontiguousarray(ref[s])
        ds = None if s is None else torch.from_numpy(s.astype(np.int32)).cuda()
        rr = N.Reference.from_numpy(ctx, r)
        out = torch.full((frames,), -1.0, dtype=torch.float64, device="cuda")
        try:
            ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x.data_ptr(), frames, atoms, stride,
                                              None if s is None else ds.data_ptr(), len(r), rr.handle, align,
                                              out.data_ptr(), None))
            torch.cuda.synchronize()
        finally:
            rr.close()
        _, want = oracle.rmsd_frames(fr, r, selection=s, align=bool(align))
        near = want < 1e-3
        np.testing.assert_allclose(out.cpu().numpy()[~near], want[~near], rtol=0, atol=1e-9)
        np.testing.assert_allclose(out.cpu().numpy()[near], want[near], rtol=0, atol=1e-7)


@pytest.mark.parametrize("frames,atoms,sel", [(1, 4, None), (3, 255, None), (64, 257, None), (592, 1000, None),
                                              (7, 600, 3), (148, 8000, None)])
def test_gradient(frames, atoms, sel):
    from warp_md.torch_ops import rmsd, rmsd_value_and_grad

    fr, ref = synth.make_trajectory(atoms, frames, (0.1, 2.0), 5 + atoms)
    idx = np.arange(atoms) if sel is None else np.arange(0, atoms, sel)
    r = torch.from_numpy(ref[idx]).cuda()
    s = None if sel is None else torch.from_numpy(idx.astype(np.int32)).cuda()
    w = torch.linspace(0.5, 1.5, frames, dtype=torch.float64, device="cuda")
    x = torch.from_numpy(fr).cuda().requires_grad_(True)
    v = rmsd(x, r, s)
    (v * w).sum().backward()
    v2, g2 = rmsd_value_and_grad(x, r, weights=w, selection=s)
    want_v, want_g = oracle.rmsd_grad(fr, ref[idx], selection=None if sel is None else idx)
    want_g = want_g * w.cpu().numpy()[:, None, None]
    for got_v, got_g in ((v.detach(), x.grad), (v2, g2)):
        np.testing.assert_allclose(got_v.cpu().numpy(), want_v, rtol=0, atol=1e-9)
        np.testing.assert_allclose(got_g.cpu().numpy(), want_g, rtol=2**-23, atol=1e-9)
