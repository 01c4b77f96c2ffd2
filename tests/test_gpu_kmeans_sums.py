"""k-means with cluster sizes and feature counts at the edges of the sums' batches (64
rows, then 8) and of the members' blocks (1,024 labels): labels, sizes and centroids
equal to the oracle's (well-separated states, sums added in the same order)."""

import numpy as np
import pytest

import oracle
from warp_md import synth

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("atoms,per", [
    (11, [1, 63, 65]),              # 33 features
    (21, [64, 127, 128, 9]),        # 63
    (22, [1023, 1]),                # 66; one block of labels
    (43, [700, 325, 200]),          # 129; more than one
    (40, [1024, 1025, 8, 7, 72]),
    (12, [30, 31, 32, 33, 40, 63, 64, 65, 71, 100]),  # ten clusters
])
def test_equal_to_oracle(atoms, per):
    import warp_md

    rng = np.random.default_rng(atoms)
    _, ref = synth.make_trajectory(atoms, 1, 0.0, atoms)
    fr = np.concatenate([ref[None] + rng.normal(0, 3.0, ref.shape)[None] + rng.normal(0, 0.1, (m, atoms, 3))
                         for m in per]).astype(np.float32)
    rng.shuffle(fr)
    system = warp_md.System.from_arrays({"name": ["CA"] * atoms, "resid": list(range(1, atoms + 1))})
    traj = warp_md.Trajectory.from_numpy(fr)
    sel = system.select("all")
    for seed in (3, 8):
        out = warp_md.TrajectoryClusterPlan(sel, method="kmeans", n_clusters=len(per), seed=seed).run(traj, system)
        labels, _, sizes = oracle.kmeans(fr, selection=sel.as_array(), n_clusters=len(per), seed=seed)
        np.testing.assert_array_equal(out["labels"], labels)
        np.testing.assert_array_equal(out["sizes"], sizes)
