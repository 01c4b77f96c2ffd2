"""The frames-across-lanes kernel finishing its own frames (the last warp of a 32-frame
group to store its sums finishes the group) and summing the frames past the last quad
row, against the same frames run 16 at a time, which takes other kernels.

Tolerance: both sum in FP64 in different orders, so G and lambda differ by a few
eps of G (coordinates ~50 A from the origin): 1e-9 A, as the batched tests; an
exact copy of the reference is 0 to the residual pass's own rounding."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("align", [1, 0])
@pytest.mark.parametrize("stride,frames,atoms", [
    (3, 9500, 64),     # one tile: finished from registers
    (3, 9507, 65),     # quad rows, tail of 3 frames, one tile
    (3, 4741, 515),    # quad rows, tail of 1
    (3, 4738, 1030),   # tail of 2, several tiles
    (4, 3001, 1000),   # xyzw
    (3, 320, 10000),   # around the most tiles a lane adds up itself
    (3, 321, 9999),
    (3, 100, 20001),   # many tiles: the finalize kernel, tail inside the streaming kernel
])
def test_equals_small_batches(stride, frames, atoms, align):
    import torch
    from warp_md import _native as N

    ctx = N.context(0)
    g = torch.Generator(device="cuda").manual_seed(atoms)
    ref = 50 + 10 * torch.randn(atoms, 3, generator=g, device="cuda")
    x = torch.zeros(frames, atoms, stride, device="cuda")
    x[..., :3] = ref + torch.randn(frames, atoms, 3, generator=g, device="cuda")
    for f in (0, frames // 2, frames - 1):  # residual pass, in a group and in the tail
        x[f, :, :3] = ref
    r = N.Reference(ctx, ref.data_ptr(), atoms, 3, keepalive=ref)

    def run(first, n):
        out = torch.full((n,), float("nan"), dtype=torch.float64, device="cuda")
        ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x[first:].data_ptr(), n, atoms, stride, None, atoms, r.handle, align,
                                          out.data_ptr(), None))
        torch.cuda.synchronize()
        return out.cpu().numpy()

    whole = run(0, frames)
    assert np.array_equal(whole, run(0, frames))  # the same bits again
    some = sorted({0, frames // 3 // 16 * 16, max(0, frames - 16)})
    for f0 in some:
        n = min(16, frames - f0)
        np.testing.assert_allclose(whole[f0:f0 + n], run(f0, n), rtol=0, atol=1e-9)
    assert not np.isnan(whole).any()
    assert whole[0] < 1e-12 and whole[frames // 2] < 1e-12 and whole[-1] < 1e-12
