"""Host-side parts of the tensor-core all-pairs kernels: the tile walk visits
every tile with a pair i < j exactly once and no other frame pair is missed,
and the FP64 epilogue's root (qcp_gap) agrees with the eigenvalue route."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
REPO = os.path.dirname(HERE)


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    out = tmp_path_factory.mktemp("pair64") / "libpair64_host.so"
    subprocess.run(["g++", "-O2", "-std=c++17", "-shared", "-fPIC", "-I", os.path.join(REPO, "warp-md_b200", "csrc"),
                    os.path.join(HERE, "native", "pair_fp64_host.cpp"), "-o", str(out)], check=True)
    L = ctypes.CDLL(str(out))
    L.t_qcp_gap.argtypes = [np.ctypeslib.ndpointer(np.float64, flags="C_CONTIGUOUS"), ctypes.c_double,
                            ctypes.POINTER(ctypes.c_double)]
    L.t_walk.argtypes = [ctypes.c_int, ctypes.c_longlong, ctypes.c_int, ctypes.c_int, ctypes.c_int, ctypes.c_int,
                         np.ctypeslib.ndpointer(np.int32, flags="C_CONTIGUOUS"), ctypes.POINTER(ctypes.c_longlong)]
    L.t_walk.restype = ctypes.c_longlong
    return L


@pytest.mark.parametrize("fn", [30, 40])
@pytest.mark.parametrize("frames", [2, 30, 31, 40, 41, 119, 120, 121, 361, 1000])
def test_tile_walk_covers_every_pair_once(lib, fn, frames):
    ni, nj = -(-frames // 40), -(-frames // fn)
    bi, bj = np.meshgrid(np.arange(ni), np.arange(nj), indexing="ij")
    need = (bi * 40 < np.minimum((bj + 1) * fn, frames) - 1).astype(np.int32)
    for parts in (1, 2, 3, ni + 1):
        total = np.zeros((ni, nj), np.int32)
        for part in range(parts):
            seen = np.zeros((ni, nj), np.int32)
            empty = ctypes.c_longlong(0)
            n = lib.t_walk(int(fn == 40), frames, part, parts, 7, nj, seen, ctypes.byref(empty))
            assert n == seen.sum() + empty.value
            assert not seen[np.arange(ni) % parts != part].any()
            total += seen
        assert np.array_equal(total, need), (frames, parts)


def _rotation(rng):
    q, _ = np.linalg.qr(rng.normal(size=(3, 3)))
    return q * np.sign(np.linalg.det(q))


def test_gap_matches_the_svd(lib):
    """D - 2 lambda_max against the SVD (s1 + s2 + sign(det) s3) in FP64.  Both
    carry a few rounding errors of D (the SVD's singular values, D's own
    cancellation): 64 eps D.  Collinear structures (a double root) are refused,
    general and planar ones are not."""
    rng = np.random.default_rng(3)
    refused = {"general": 0, "planar": 0, "collinear": 0}
    tried = dict(refused)
    for trial in range(600):
        kind = ("general", "general", "planar", "collinear")[trial % 4]
        n = int(rng.integers(4, 400))
        x = 10 ** rng.uniform(-3, 3) * rng.normal(size=(n, 3))
        if kind == "planar":
            x[:, 2] = 0
        if kind == "collinear":
            x[:, 1:] = 0
        x -= x.mean(0)
        y = x @ _rotation(rng).T + np.abs(x).max() * 10 ** rng.uniform(-5, -0.3) * rng.normal(size=(n, 3)) * (kind != "collinear")
        y -= y.mean(0)
        h = np.ascontiguousarray((x.T @ y).reshape(9))
        d = float((x * x).sum() + (y * y).sum())
        u, s, vt = np.linalg.svd(h.reshape(3, 3))
        want = d - 2 * (s[0] + s[1] + np.sign(np.linalg.det(u) * np.linalg.det(vt)) * s[2])
        gap = ctypes.c_double()
        tried[kind] += 1
        if not lib.t_qcp_gap(h, d, ctypes.byref(gap)):
            refused[kind] += 1
            continue
        assert abs(gap.value - max(want, 0.0)) <= 64 * np.finfo(float).eps * d, (trial, kind, n, gap.value, want)
    assert refused["general"] <= tried["general"] // 50 and refused["planar"] <= tried["planar"] // 10, refused
    assert refused["collinear"] >= tried["collinear"] // 2, refused


def test_gap_out_of_range_is_refused(lib):
    gap = ctypes.c_double()
    for d in (0.0, -1.0, 1e300, float("inf"), float("nan")):
        assert not lib.t_qcp_gap(np.zeros(9), d, ctypes.byref(gap))
