"""Short kernels launched before the kernel they follow has ended: back-to-back calls
on changing inputs, into the same outputs and scratch, on two streams' contexts and
replayed from a CUDA graph, give the bits of calls that are waited for one by one."""

import numpy as np
import pytest

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

# lanes finished in place / by the second kernel, atom-major, gathered, one CTA a frame
SHAPES = [(3000, 600, None), (500, 12000, None), (800, 1001, None), (900, 3000, 7), (50, 300, None)]


@pytest.mark.parametrize("frames,atoms,every", SHAPES)
def test_in_flight_equals_waited(frames, atoms, every):
    from warp_md import _native as N

    g = torch.Generator(device="cuda").manual_seed(atoms)
    ref = 10 * torch.randn(atoms, 3, generator=g, device="cuda")
    xs = [ref + torch.randn(frames, atoms, 3, generator=g, device="cuda") for _ in range(3)]
    for x in xs:
        x[frames // 2] = ref  # a frame for the residual pass
    sel = None if every is None else torch.arange(0, atoms, every, dtype=torch.int32, device="cuda")
    n_sel = atoms if sel is None else sel.numel()
    picked = ref if sel is None else ref[sel.long()].contiguous()
    ctx = N.context(0)
    r = N.Reference.from_numpy(ctx, picked.cpu().numpy())
    buf = torch.empty_like(xs[0])

    def call(x, out, rows, stream):
        p = None if sel is None else sel.data_ptr()
        ctx.check(ctx.lib.wmd_rmsd_frames(ctx.handle, x.data_ptr(), frames, atoms, 3, p, n_sel, r.handle, 1,
                                          out.data_ptr(), stream))
        ctx.check(ctx.lib.wmd_superpose_transforms(ctx.handle, x.data_ptr(), frames, atoms, 3, p, n_sel, r.handle, 0,
                                                   rows.data_ptr(), stream))

    def fresh():
        return torch.empty(frames, dtype=torch.float64, device="cuda"), torch.empty(frames, 12, device="cuda")

    try:
        want = []
        for x in xs:
            o = fresh()
            call(x, *o, None)
            torch.cuda.synchronize()
            want.append(o)
        s = torch.cuda.Stream()
        s.wait_stream(torch.cuda.current_stream())
        got, shared = [], fresh()
        with torch.cuda.stream(s):
            for _ in range(4):
                for x in xs:
                    buf.copy_(x)  # the input of the call before is overwritten at once
                    call(buf, *shared, s.cuda_stream)
                    got.append(tuple(t.clone() for t in shared))
        torch.cuda.synchronize()
        for i, o in enumerate(got):
            assert torch.equal(o[0], want[i % 3][0]) and torch.equal(o[1], want[i % 3][1]), i
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=s):
            call(buf, *shared, s.cuda_stream)
            call(buf, *shared, s.cuda_stream)
        for x, w in zip(xs, want):
            buf.copy_(x)
            graph.replay()
            torch.cuda.synchronize()
            assert torch.equal(shared[0], w[0]) and torch.equal(shared[1], w[1])
        assert not np.isnan(shared[0].cpu().numpy()).any()
    finally:
        r.close()
