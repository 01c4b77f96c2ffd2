"""A reference centred on the device (wmd_reference_prepare, torch_ops) gives what
the uploaded one gives, on any stream and inside a captured graph."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _both(ctx, ref, stride):
    import torch
    from warp_md import _native as N

    y = torch.zeros(max(ref.shape[0], 1), stride, device="cuda")
    y[:ref.shape[0], :3] = torch.from_numpy(ref)
    n = ref.shape[0]
    size = ctx.lib.wmd_reference_workspace(n)
    work = torch.full((size,), 255, dtype=torch.uint8, device="cuda")
    p = N.Reference.prepared(ctx, y.data_ptr(), n, stride, work.data_ptr(), size, None, keepalive=(y, work))
    return p, N.Reference(ctx, y.data_ptr(), n, stride, keepalive=y)


@pytest.mark.parametrize("n,stride", [(1, 3), (3, 4), (31, 3), (32, 3), (33, 4), (511, 3), (512, 3), (513, 3), (4100, 4)])
def test_prepared_equals_uploaded(n, stride):
    """Same centred sums to FP64 rounding: RMSD (fit and raw), covariance and
    transforms agree to 1e-12 of their size (transforms: float32 results, one ulp)."""
    import torch
    from warp_md import _native as N

    rng = np.random.default_rng(n)
    ref = (50 + 20 * rng.standard_normal((n, 3))).astype(np.float32)
    ctx = N.context(0)
    F = 70
    x = torch.from_numpy((ref + rng.standard_normal((F, n, 3))).astype(np.float32)).cuda()
    res = []
    for r in _both(ctx, ref, stride):
        out = [torch.empty(F, dtype=torch.float64, device="cuda") for _ in range(2)]
        xf = torch.empty(F, 12, device="cuda")
        for align in (0, 1):
            ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x.data_ptr(), F, n, 3, None, n, r.handle, align,
                                              out[align].data_ptr(), None))
        ctx.check(ctx.lib.wmd_superpose_transforms(ctx.handle, x.data_ptr(), F, n, 3, None, n, r.handle, 0,
                                                   xf.data_ptr(), None))
        torch.cuda.synchronize()
        res.append([o.cpu().numpy() for o in out] + [xf.cpu().numpy()])
    (raw_p, fit_p, xf_p), (raw_u, fit_u, xf_u) = res
    np.testing.assert_allclose(raw_p, raw_u, rtol=1e-12, atol=0)
    # one or two atoms superpose exactly: only the cancellation of G_x + G_y - 2 lambda is left
    np.testing.assert_allclose(fit_p, fit_u, rtol=1e-11, atol=1e-6 if n < 3 else 0)
    if n >= 3:
        np.testing.assert_allclose(xf_p, xf_u, rtol=2e-6, atol=2e-6 * np.abs(xf_u).max())


def test_workspace_is_checked():
    import torch
    from warp_md import _native as N

    ctx = N.context(0)
    y = torch.randn(40, 3, device="cuda")
    size = ctx.lib.wmd_reference_workspace(40)
    w = torch.empty(size + 256, dtype=torch.uint8, device="cuda")
    h = ctypes.c_void_p()
    args = lambda ptr, ws, b: (ctx.handle, ptr, 40, 3, ws, b, None, ctypes.byref(h))  # noqa: E731
    assert ctx.lib.wmd_reference_prepare(*args(y.data_ptr(), w.data_ptr(), size - 1)) == N.WMD_ERR_INVALID_ARG
    assert ctx.lib.wmd_reference_prepare(*args(y.data_ptr(), w.data_ptr() + 8, size)) == N.WMD_ERR_INVALID_ARG
    host = np.zeros((40, 3), np.float32)
    assert ctx.lib.wmd_reference_prepare(*args(host.ctypes.data, w.data_ptr(), size)) == N.WMD_ERR_INVALID_ARG


def test_streams_views_and_graphs():
    """The cached reference is ordered across streams, a view of another layout
    at the same address is another reference, and a captured call follows the
    reference's values at replay time."""
    import torch
    from warp_md.torch_ops import rmsd, rmsd_value_and_grad

    torch.manual_seed(1)
    x = torch.randn(90, 64, 3, device="cuda")
    pool = torch.randn(128, 3, device="cuda")
    want = [rmsd(x, pool[:64].clone()), rmsd(x, pool[::2].clone())]
    assert torch.equal(rmsd(x, pool[:64]), want[0])
    assert torch.equal(rmsd(x, pool[::2]), want[1])
    side = torch.cuda.Stream()
    for _ in range(3):
        ref = torch.randn(64, 3, device="cuda")
        a = rmsd(x, ref)
        side.wait_stream(torch.cuda.current_stream())
        with torch.cuda.stream(side):
            b = rmsd(x, ref)
        torch.cuda.synchronize()
        assert torch.equal(a, b)
    ref = torch.randn(64, 3, device="cuda")
    out, grad = torch.empty(90, dtype=torch.float64, device="cuda"), torch.empty_like(x)
    with torch.cuda.stream(side):  # sizes the scratch outside the capture
        rmsd_value_and_grad(x, pool[:64], out=out, grad=grad)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        rmsd_value_and_grad(x, ref, out=out, grad=grad)
    for _ in range(2):
        ref.normal_()
        g.replay()
        torch.cuda.synchronize()
        r, d = rmsd_value_and_grad(x, ref.clone())
        assert torch.equal(out, r) and torch.equal(grad, d)
