"""P2G with a partition older than the positions: a particle that has left the
mesh since (or holds NaN) has no support there and adds nothing, in every form of
the quadratic B-spline, at the mesh faces and in interior blocks (3D FP32 raises
an error for a particle that has left an interior block). The sums equal those of
the other particles alone (FP64 1e-12, FP32 1e-5 of the largest)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("outside", [-0.2, -0.7, -3.0, np.nan])
@pytest.mark.parametrize("dim,dtype", [(3, np.float64), (3, np.float32), (2, np.float64), (2, np.float32)])
def test_p2g_leaves_out_particles_outside(tb, ctx, dim, dtype, outside):
    from tesserae_b200 import runtime
    h = 0.125
    cells = (13, 14, 16)[:dim]  # blocks of 4 (2D: 8) cells, the last one cut
    mesh = tb.CartesianMesh(h, *[(0.0, c * h) for c in cells])
    rng = np.random.default_rng(dim)
    n = 40
    P = tb.Particles(n * (2 * dim + 1), dim, np.float64, optional=("m",))
    for d in range(dim):
        P.x[d] = rng.uniform(1.2 * h, (cells[d] - 1.2) * h, size=P.n)
    P.v[...] = rng.normal(size=P.v.shape)
    P.m[...] = rng.uniform(0.5, 1.5, size=P.n)
    P.V[...] = h ** dim
    P.sigma[...] = rng.normal(size=P.sigma.shape)
    faces = [(d, side) for d in range(dim) for side in (0, 1)]
    moved = P.x.copy()
    for k, (d, side) in enumerate(faces):
        sel = slice(k * n, (k + 1) * n)
        P.x[d, sel] = (0.3 * h, (cells[d] - 0.3) * h)[side]
        moved[:, sel] = P.x[:, sel]
        moved[d, sel] = outside * h if side == 0 else (cells[d] - outside) * h
    stays = np.arange(P.n) >= len(faces) * n
    if not (dim == 3 and dtype == np.float32):  # (there, leaving an interior block's tile is an error)
        far = np.flatnonzero(stays)[:8]
        P.x[:, far] = moved[:, far] = 9.5 * h
        moved[0, far] = outside * h
        stays[far] = False
    prm = tb.step_params(1e-4, mass=1.0, V0=h ** dim, mu=1.0, lam=1.0, gravity=(0.1, -0.2, 0.3)[:dim])

    def sums(x, m, V):
        Pd = P.to("torch", device="cuda", dtype=dtype)
        part = tb.Partition(mesh, P.n, backend="torch", device="cuda")
        G = tb.generate_grid(mesh, dtype, backend="torch", device="cuda")
        runtime.update(part, Pd, mesh, ctx=ctx)
        assert part.nassigned == P.n
        Pd.x.copy_(torch.from_numpy(x))
        Pd.m.copy_(torch.from_numpy(m))
        Pd.V.copy_(torch.from_numpy(V))
        runtime.P2G(G, Pd, part, mesh, prm, grid_half=False, ctx=ctx)
        ctx.synchronize()  # raises if the kernel reported an error
        return G.numpy()

    ref = sums(P.x, np.where(stays, P.m, 0.0), np.where(stays, P.V, 0.0))
    got = sums(moved, P.m, P.V)
    tol = 1e-12 if dtype == np.float64 else 1e-5
    for k in ("m", "mv", "f"):
        assert np.abs(got[k] - ref[k]).max() <= tol * np.abs(ref[k]).max(), k
