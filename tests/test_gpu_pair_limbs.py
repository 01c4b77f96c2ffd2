"""The int8 all-pairs modes write a whole matrix themselves (nothing is cleared first)
and pack four atoms' limbs per store: atom counts around the packing and the padding,
frame counts around the 10-frame row groups and the tiles, into a matrix of NaN, after
a call that left other limbs in the workspace; selections in any order and with
repeats, both strides.  Against the oracle at the modes' bars (5e-4 and 1e-4 A)."""

import numpy as np
import pytest

import oracle
from warp_md import _native as N
from warp_md import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("mode,bar", [(N.MODE_I8X2, 5e-4), (N.MODE_I8X3, 1e-4)])
@pytest.mark.parametrize("frames,atoms,n_sel,stride", [
    (2, 2, None, 3), (9, 3, None, 3), (11, 63, None, 3), (40, 64, None, 4), (41, 65, None, 3), (81, 130, 67, 3),
    (123, 200, 129, 4), (50, 515, None, 3)])
def test_whole_matrix(frames, atoms, n_sel, stride, mode, bar):
    fr, _ = synth.make_trajectory(atoms, frames, (0.1, 2.0), 23 + atoms)
    sel = None if n_sel is None else np.random.default_rng(2).integers(0, atoms, n_sel).astype(np.uint32)
    picked = fr if sel is None else np.ascontiguousarray(fr[:, sel])
    data = fr if stride == 3 else np.concatenate([fr, np.full(fr.shape[:2] + (1,), 5.0, np.float32)], axis=2)
    x = torch.from_numpy(np.ascontiguousarray(data)).cuda()
    ds = None if sel is None else torch.from_numpy(sel.astype(np.int32)).cuda()
    ctx = N.context(0)
    junk = torch.randn(150, 300, 3, device="cuda") * 50
    for metric, name in ((N.PAIR_RMS, "rms"), (N.PAIR_NOFIT, "nofit")):
        other = torch.empty(150, 150, device="cuda")
        ctx.check(ctx.lib.wmd_pairwise_rmsd(ctx.handle, junk.data_ptr(), 150, 300, 3, None, 300, N.PAIR_RMS, mode,
                                            other.data_ptr(), None))
        out = torch.full((frames, frames), float("nan"), device="cuda")
        ctx.check(ctx.lib.wmd_pairwise_rmsd(ctx.handle, x.data_ptr(), frames, atoms, stride,
                                            None if ds is None else ds.data_ptr(), picked.shape[1], metric, mode,
                                            out.data_ptr(), None))
        torch.cuda.synchronize()
        got = out.cpu().numpy()
        np.testing.assert_allclose(got, oracle.pairwise(picked, name)[0], rtol=1e-6, atol=bar)
        assert np.all(np.diag(got) == 0.0)
