"""Per-group RMSD of consecutive atoms in aligned packed frames (blocks of at most
512 positions streamed through shared memory): sizes at the block's edges, against
the oracle.  Bar: 1e-5 A plus one float32 ulp, the per-group bar elsewhere."""

import numpy as np
import pytest

import oracle
from warp_md import synth

torch = pytest.importorskip("torch")

pytestmark = pytest.mark.gpu

# (atoms, frames, first atom of the list, group sizes; the last size repeats to the end)
CASES = [
    (512, 1, 0, [512]),  # one full block, one frame, 32 lanes a sum
    (513, 3, 1, [512]),  # the array's end is not on 16 bytes
    (1031, 2, 0, [513, 10]),  # a group past the block: the other kernel
    (1537, 5, 3, [0, 0, 255, 257, 0, 511, 1, 0]),  # exact fits, empty groups at both ends
    (2047, 33, 2, [1]),  # more (frame, group) sums than threads
    (1500, 7, 5, [64, 63, 33, 32, 31, 17, 2, 9]),  # every lane count
    (40, 4, 7, [10, 0, 0, 3]),  # a single short block
    (3001, 601, 0, [10]),  # several items a CTA, CTAs that change block
]


@pytest.mark.parametrize("n,frames,first,sizes", CASES)
def test_staged_groups(n, frames, first, sizes):
    from warp_md import _native as N

    fr, ref = synth.make_trajectory(n, frames, (0.1, 2.0), 7 + n)
    out_sizes, left = [], n - first
    for k in sizes:
        out_sizes.append(min(k, left))
        left -= out_sizes[-1]
    while left > 0:
        out_sizes.append(min(sizes[-1] or 10, left))
        left -= out_sizes[-1]
    out_sizes.append(0)
    goff = np.concatenate([[0], np.cumsum(out_sizes)]).astype(np.uint32)
    groups = [np.arange(first + goff[i], first + goff[i + 1]) for i in range(len(out_sizes))]
    sel = np.arange(0, n, 3, dtype=np.uint32)
    ctx = N.context(0)
    rr = N.Reference.from_numpy(ctx, ref[sel])
    gref = N.GroupRef(ctx, ref, goff, np.arange(first, n, dtype=np.uint32))
    x = torch.from_numpy(fr).cuda()
    dsel = torch.from_numpy(sel.astype(np.int32)).cuda()
    out = torch.full((frames, len(out_sizes)), -1.0, device="cuda")
    try:
        ctx.check(ctx.lib.wmd_rmsd_per_group(ctx.handle, x.data_ptr(), frames, n, 3, dsel.data_ptr(), sel.size,
                                             rr.handle, gref.handle, 1, out.data_ptr(), None))
        torch.cuda.synchronize()
    finally:
        gref.close()
        rr.close()
    got = out.cpu().numpy()
    want = oracle.rmsd_perres(fr, ref, groups, selection=sel, align=True)
    np.testing.assert_allclose(got, want, rtol=1.2e-7, atol=1e-5)
    assert np.all(got[:, np.array(out_sizes) == 0] == 0.0)
