"""The batched lanes forward's equal runs of stages: runs that end inside a unit, units
shared by three and more warps, trajectories without frames or atoms between others,
and the last frames of packed trajectories whose stride is no multiple of 16 bytes
(their group's rows arrive one by one); against the oracle with both tile shapes.

Tolerance: 1e-9 A, FP64 sums in different orders; gradients rounded to float32 once
(2^-23 relative, 1e-9 for zeros)."""

import numpy as np
import pytest

import oracle
from warp_md import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tile", ["512", "1024"])
@pytest.mark.parametrize("sizes", [
    [(1, 40)],                                        # one stage
    [(5000, 3)],                                      # one group over every warp
    [(20000, 33), (7, 1), (20001, 35)],               # many warps a unit
    [(0, 5), (33, 1000), (100, 0), (1029, 131), (1030, 129), (1031, 130), (64, 9)],
    [(300, 2001), (1500, 1003), (2, 64), (513, 702)],
])
def test_equal_runs(monkeypatch, sizes, tile):
    from warp_md.batched import BatchedRmsd

    monkeypatch.setenv("WARPMD_BATCHED_LAYOUT", "lanes")
    monkeypatch.setenv("WARPMD_BATCHED_TILE_ATOMS", tile)
    made = [synth.make_trajectory(max(n, 1), max(f, 1), (0.1, 2.0), 3 + i) for i, (n, f) in enumerate(sizes)]
    coords = [torch.from_numpy(np.ascontiguousarray(x[:f, :n])).cuda() for (n, f), (x, _) in zip(sizes, made)]
    refs = [torch.from_numpy(np.ascontiguousarray(r[:n])).cuda() for (n, f), (_, r) in zip(sizes, made)]
    b = BatchedRmsd(coords, refs, with_grad=True)
    first = [t.clone() for t in b.run()]
    assert b.layout()["layout"] == "lanes"
    again = b.run()
    torch.cuda.synchronize()
    for (n, f), (x, r), got, got2, grad in zip(sizes, made, first, again, b.grads):
        assert torch.equal(got, got2)
        if n < 3 or f == 0:
            continue
        want, want_g = oracle.rmsd_grad(x, r)
        np.testing.assert_allclose(got.cpu().numpy(), want, rtol=0, atol=1e-9)
        np.testing.assert_allclose(grad.cpu().numpy(), want_g, rtol=2**-23, atol=1e-9)
