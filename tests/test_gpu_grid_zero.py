"""The dense zero of P2G's targets: every device memset of a step stays inside one
of the grid's arrays, however their addresses fall. Arrays that adjoin need not be
one allocation (cudaMalloc places them back to back where a size is a multiple of
its granule), and a memset across two allocations is an error."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")
cudart = pytest.importorskip("cuda.bindings.runtime")


def _memsets(graph):
    """(address, bytes) of the memset nodes of a captured graph."""
    def ok(r):
        assert int(r[0]) == 0, r[0]
        return r[1:] if len(r) > 2 else r[1]
    _, count = ok(cudart.cudaGraphGetNodes(graph))
    nodes, _ = ok(cudart.cudaGraphGetNodes(graph, count))
    out = []
    for n in nodes:
        if ok(cudart.cudaGraphNodeGetType(n)) == cudart.cudaGraphNodeType.cudaGraphNodeTypeMemset:
            p = ok(cudart.cudaGraphMemsetNodeGetParams(n))
            assert p.height == 1
            out.append((int(p.dst), int(p.width) * int(p.elementSize)))
    return out


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("cells", [(127, 127, 127), (128, 127, 127), (1023, 1023)])  # from 2^20 nodes on
def test_dense_zero_per_array(tb, oracle, dtype, cells):
    from tesserae_b200 import runtime
    D, h = len(cells), 1.0 / 64
    mesh = tb.CartesianMesh(h, *[(0.0, c * h) for c in cells])
    assert mesh.nnodes >= 1 << 20
    rng = np.random.default_rng(3)
    P = tb.Particles(500, D, np.float64)
    P.x[...] = rng.uniform(0.3, 0.6, size=P.x.shape)
    P.v[...] = rng.normal(size=P.v.shape)
    P.V[...] = h ** D
    prm = tb.step_params(1e-5, mass=1.0, V0=h ** D, mu=1.0, lam=1.0)
    stream = torch.cuda.Stream()
    ctx = runtime.Context(0, stream=stream)
    with torch.cuda.stream(stream):
        Pd = P.to("torch", device="cuda", dtype=dtype)
        Po = Pd.to("numpy", dtype=np.float64)
        part = tb.Partition(mesh, P.n, backend="torch", device="cuda")
        G = tb.generate_grid(mesh, dtype, backend="torch", device="cuda")
        # all arrays of the grid back to back, holding what must not survive
        buf = torch.full((1 + 4 * D, mesh.nnodes), 7.0, dtype=G.m.dtype, device="cuda")
        G.m, G.mv, G.f, G.v, G.vn = buf[0], buf[1:1 + D], buf[1 + D:1 + 2 * D], buf[1 + 2 * D:1 + 3 * D], buf[1 + 3 * D:]
        runtime.step(G, Pd, part, mesh, prm, 1, ctx=ctx)
    ctx.synchronize()
    got = {k: v.astype(np.float64) for k, v in G.numpy().items()}
    Go = tb.generate_grid(mesh, np.float64)
    oracle.step(mesh, Po, Go, prm, 1)
    tol = 1e-12 if dtype == np.float64 else 1e-5
    for k in ("m", "mv", "f"):
        ref = getattr(Go, k)
        assert np.abs(got[k].reshape(ref.shape) - ref).max() <= tol * max(np.abs(ref).max(), 1.0), k
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph, stream=stream):
        runtime.step(G, Pd, part, mesh, prm, 1, ctx=ctx)
    row = mesh.nnodes * buf.element_size()
    lo, hi = buf.data_ptr(), buf.data_ptr() + buf.numel() * buf.element_size()
    inside = [(a - lo, b) for a, b in _memsets(graph.raw_cuda_graph()) if lo <= a < hi]
    del graph
    ctx.close()
    for off, size in inside:
        assert off // row == (off + size - 1) // row, (off, size, row)
