"""The FP64 all-pairs mode on the tensor cores (40-bit fixed point per frame,
five int8 digits) against the CPU oracle at the sizes where its tiles, chunks
and its lists can go wrong.

Tolerance, per entry v: float32 rounding of the result and of nothing else,
2^-23 v, plus the FP64 cancellation of G_i + G_j - 2 lambda: the MSD carries a
few (8) eps (G_i + G_j) / n, as the SIMT tiles' does."""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


def _run(frames, metric, sel=None, device_sel=False):
    import torch
    from warp_md import _native as N

    ctx = N.context(0)
    x = torch.from_numpy(np.ascontiguousarray(frames, dtype=np.float32)).cuda()
    F, n = x.shape[0], x.shape[1]
    out = torch.full((F, F), float("nan"), dtype=torch.float32, device="cuda")
    m = N.PAIR_RMS if metric == "rms" else N.PAIR_NOFIT
    s = None if sel is None else torch.from_numpy(np.asarray(sel, dtype=np.int32)).cuda()
    ctx.check(ctx.lib.wmd_pairwise_rmsd(ctx.handle, x.data_ptr(), F, n, x.shape[2], None if s is None else s.data_ptr(),
                                        n if s is None else len(sel), m, N.MODE_FP64, out.data_ptr(), None))
    torch.cuda.synchronize()
    return out.cpu().numpy()


def _check(frames, metric, sel=None):
    x = np.asarray(frames[..., :3], dtype=np.float32)
    x = x if sel is None else x[:, np.asarray(sel)]
    got = _run(frames, metric, sel)
    _, want = oracle.pairwise(np.ascontiguousarray(x), metric)
    c = x.astype(np.float64) - x.astype(np.float64).mean(1, keepdims=True)
    g = (c ** 2).sum((1, 2)) / x.shape[1]
    msd_tol = 8 * np.finfo(float).eps * (g[:, None] + g[None])
    if metric == "nofit":  # the centroid offsets are part of the sum
        msd_tol = msd_tol + 8 * np.finfo(float).eps * want.astype(np.float64) ** 2
    v = want.astype(np.float64)
    tol = 2.0 ** -23 * v + np.minimum(np.sqrt(msd_tol), msd_tol / np.maximum(2 * v, 1e-300))
    assert not np.isnan(got).any()
    assert np.array_equal(got, got.T) and not got.diagonal().any()
    assert (np.abs(got - v) <= tol).all(), float((np.abs(got - v) - tol).max())


@pytest.mark.parametrize("metric", ["rms", "nofit"])
@pytest.mark.parametrize("frames,atoms", [(2, 160), (30, 161), (31, 191), (40, 192), (41, 193), (121, 224), (161, 500),
                                          (303, 1000)])
def test_tile_and_chunk_edges(frames, atoms, metric):
    from warp_md import synth

    _check(synth.make_drift_trajectory(atoms, frames, 0.3, seed=frames), metric)


def test_listed_pairs_and_a_full_list():
    """Frames 1e-3 A apart are recomputed in FP64: a few pairs through the list,
    and a trajectory of nothing else (over an eighth of all pairs) through the
    SIMT tiles."""
    from warp_md import synth

    rng = np.random.default_rng(1)
    fr = synth.make_drift_trajectory(300, 90, 0.5, seed=2)
    for k in range(0, 90, 9):
        fr[k + 1] = fr[k] + 1e-3 * rng.standard_normal(fr[k].shape)
        fr[k + 2] = fr[k]
    _check(fr, "rms")
    same = (fr[:1] + 1e-3 * rng.standard_normal((70, 300, 3))).astype(np.float32)
    _check(same, "rms")
    _check(same, "nofit")


def test_frames_of_very_different_extent_and_degenerate_frames():
    """Every frame has its own scale: a frame blown up a thousandfold, one
    shrunk to a point's neighbourhood, a collinear and a planar one, all
    beside ordinary ones; and a selection with a w column."""
    from warp_md import synth

    fr = synth.make_drift_trajectory(200, 60, 0.5, seed=5).astype(np.float64)
    fr[7] *= 1000.0
    fr[11] = 5.0 + 1e-3 * fr[11]
    fr[13][:, 1:] = 2.0
    fr[17][:, 2] = -1.0
    xyzw = np.zeros((60, 200, 4), np.float32)
    xyzw[..., :3] = fr
    _check(xyzw, "rms")
    _check(xyzw, "nofit", sel=np.arange(0, 200)[::-1][:180])


def test_parts_sum_to_the_matrix_also_when_the_list_overflows():
    import torch
    from warp_md import _native as N

    rng = np.random.default_rng(3)
    ctx = N.context(0)
    base = 10 * rng.standard_normal((1, 256, 3))
    for sigma in (1.0, 1e-4):
        x = torch.from_numpy((base + sigma * rng.standard_normal((130, 256, 3))).astype(np.float32)).cuda()
        full = _run(x.cpu().numpy(), "rms")
        total = np.zeros_like(full)
        for part in range(3):
            out = torch.empty((130, 130), dtype=torch.float32, device="cuda")
            ctx.check(ctx.lib.wmd_pairwise_rmsd_part(ctx.handle, x.data_ptr(), 130, 256, 3, None, 256, N.PAIR_RMS,
                                                     N.MODE_FP64, part, 3, out.data_ptr(), None))
            torch.cuda.synchronize()
            o = out.cpu().numpy()
            assert not (total[o != 0]).any()
            total += o
        assert np.array_equal(total, full)
