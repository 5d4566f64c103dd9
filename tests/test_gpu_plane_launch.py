"""P2G of the 3D FP32 B-spline is one launch on a mesh of any size, with particles at
the faces, edges and corners of a mesh of more than 16384 blocks: the oracle's sums
(FP32, 1e-5 of what a node's terms reach)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_one_launch_on_a_large_mesh(tb, oracle, ctx):
    from tesserae_b200 import runtime
    h, c = 0.125, 102
    mesh = tb.CartesianMesh(h, *[(0.0, c * h)] * 3)
    assert mesh.nblocks_total > 16384
    rng = np.random.default_rng(4)
    n = 4000
    P = tb.Particles(n, 3, np.float32)
    for d in range(3):  # a third of the particles at each end of each axis, a third anywhere
        u = rng.uniform(0.01, 2.0, size=n)
        P.x[d] = h * np.choose(rng.integers(0, 3, size=n), [u, c - u, rng.uniform(0.01, c - 0.01, size=n)])
    P.v[...] = rng.normal(size=P.v.shape)
    P.V[...] = rng.uniform(0.5, 1.5, size=n) * h ** 3
    P.sigma[...] = rng.normal(size=P.sigma.shape)
    prm = tb.step_params(1e-4, mass=1.5, V0=h ** 3, mu=1.0, lam=1.0, gravity=(0.1, -0.2, 0.3))
    Pd = P.to("torch", device="cuda", dtype=np.float32)
    Po = Pd.to("numpy", dtype=np.float64)
    part = tb.Partition(mesh, n, backend="torch", device="cuda")
    G = tb.generate_grid(mesh, np.float32, backend="torch", device="cuda")
    runtime.update(part, Pd, mesh, ctx=ctx)
    before = ctx.launches
    runtime.P2G(G, Pd, part, mesh, prm, grid_half=False, ctx=ctx)
    assert ctx.launches - before == 2  # the grid's zero and P2G
    ctx.synchronize()
    Go = tb.generate_grid(mesh, np.float64)
    oracle.p2g(mesh, Po, Go, prm)
    got = G.numpy()
    for k, scale in (("m", 1.5), ("mv", 1.5), ("f", h ** 2)):
        ref = getattr(Go, k)
        assert np.abs(got[k].reshape(ref.shape) - ref).max() <= 1e-5 * max(np.abs(ref).max(), scale), k
