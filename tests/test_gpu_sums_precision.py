"""Bits that the transfers keep: sums of a crowded block, and the consistency of WLS
weights far from the origin."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("transfer", ["flip", "apic"])
@pytest.mark.parametrize("basis", ["bspline_quadratic", "wls_bspline_quadratic"])
def test_crowded_block_2d_sums_in_fp64(tb, ctx, transfer, basis):
    """2^20 particles at the 64 cell centres of one block, FP32 state: the weights
    (0, 1/4 or 1/2 per axis) and the sums of the particles of one pass are exact in
    FP32, so what is left is how passes are added. WLS and APIC hold a block's sums
    in FP64 until they are added to the grid: at most 8 pieces per block, each
    rounded once and added once in FP32, so 16 * 2^-24 of the node's sum."""
    from helpers import basis_kind
    from tesserae_b200 import runtime
    if transfer == "flip" and basis == "bspline_quadratic":
        pytest.skip("the plain kernel's partials are FP32")
    abi = tb._abi
    h = 0.125
    mesh = tb.CartesianMesh(h, (0.0, 24 * h), (0.0, 24 * h))
    n = 1 << 20
    cell = np.arange(n) // (n // 64)  # every pass takes four particles of each cell
    P = tb.Particles(n, 2, np.float32, optional=("B",))
    P.x[0] = (8.5 + cell % 8) * h
    P.x[1] = (8.5 + cell // 8) * h
    mass = 1.0 + 2.0 ** -17 + 2.0 ** -18 + 2.0 ** -19 + 2.0 ** -21
    P.v[0], P.v[1] = 1.0, -0.5
    P.V[...] = 0.0
    prm = tb.step_params(1e-4, mass=mass, V0=1.0, mu=1.0, lam=1.0, basis=basis_kind(abi, basis),
                         transfer=abi.TB_TRANSFER_APIC if transfer == "apic" else abi.TB_TRANSFER_FLIP)
    Pd = P.to("torch", device="cuda", dtype=np.float32)
    part = tb.Partition(mesh, n, backend="torch", device="cuda")
    G = tb.generate_grid(mesh, np.float32, backend="torch", device="cuda")
    runtime.update(part, Pd, mesh, ctx=ctx)
    runtime.P2G(G, Pd, part, mesh, prm, grid_half=False, ctx=ctx)
    ctx.synchronize()
    nx = mesh.n_nodes[0]
    m = np.zeros((mesh.n_nodes[1], nx))
    for cy in range(8):
        for cx in range(8):
            m[8 + cy:10 + cy, 8 + cx:10 + cx] += 0.25 * mass * (n // 64)
    got = G.numpy()
    on = m > 0
    gm = got["m"].astype(np.float64).reshape(m.shape)
    assert np.all(gm[~on] == 0.0)
    tol = 16 * 2.0 ** -24
    assert np.max(np.abs(gm - m)[on] / m[on]) <= tol
    for d, v in enumerate((1.0, -0.5)):
        gv = got["mv"][d].astype(np.float64).reshape(m.shape)
        assert np.max(np.abs(gv - v * m)[on] / m[on]) <= tol


@pytest.mark.parametrize("basis", ["wls_bspline_quadratic", "wls_ugimp"])
@pytest.mark.parametrize("dim", [2, 3])
def test_wls_weights_reproduce_constants_far_from_the_origin(tb, ctx, dim, basis):
    """FP32: sum N = 1 and sum grad N = 0 wherever WLS fits its moments (uGIMP; B-spline
    windows that the mesh cuts), although a node's coordinate is rounded by up to
    eps |X| (|X| / h = 1300 here, so a weight is off by 1e3 eps). A fitted sum carries
    the rounding of some 40 operations on terms of up to 3 (N) and 6 / h (grad N)."""
    dtype = np.float32
    from helpers import basis_kind
    from tesserae_b200 import runtime
    abi = tb._abi
    h, x0 = 1.0 / 13, 100.3
    cells = (11, 9, 10)[:dim]
    mesh = tb.CartesianMesh(h, *[(x0, x0 + c * h) for c in cells])
    rng = np.random.default_rng(17)
    n = 4000
    P = tb.Particles(n, dim, np.float64)
    for d in range(dim):
        P.x[d] = x0 + rng.uniform(0.02, cells[d] - 0.02, size=n) * h
    P.x[0] = x0 + rng.uniform(0.02, 0.45, size=n) * h  # windows that the mesh cuts on one axis at least
    Pd = P.to("torch", device="cuda", dtype=dtype)
    W = tb.BasisWeights(dim, n, dtype, backend="torch", device="cuda")
    prm = tb.step_params(1e-4, gimp_l=0.45 * h, basis=basis_kind(abi, basis))
    runtime.update(W, Pd, mesh, prm, ctx=ctx)
    ctx.synchronize()
    w = W.w.cpu().numpy().astype(np.float64).reshape(n, -1)
    g = W.grad_w.cpu().numpy().astype(np.float64).reshape(n, w.shape[1], dim)
    eps = float(np.finfo(dtype).eps)
    assert np.abs(w.sum(axis=1) - 1.0).max() <= 40 * 3 * eps
    assert np.abs(g.sum(axis=1)).max() <= 40 * 6 / h * eps


def test_ugimp_quotient_is_the_division_to_one_ulp(tb, ctx):
    """The uGIMP jets divide by the particle's length through its inverse, corrected once.
    At FP32, with offsets that are exact (h = 1/8, positions of few bits) and a second
    axis whose weight is 1/2, grad N gives the jet's derivative itself: 2 a / l or
    (1 + l/2 - a) / l, at most one ulp from the division."""
    from tesserae_b200 import runtime
    abi = tb._abi
    f = np.float32
    h, cells, n = 0.125, 16, 20000
    mesh = tb.CartesianMesh(h, (0.0, cells * h), (0.0, cells * h))
    rng = np.random.default_rng(23)
    P = tb.Particles(n, 2, np.float32, optional=("l",))
    P.x[0] = (rng.integers(4 * 4096, 12 * 4096, size=n) / 4096).astype(f) * f(h)
    P.x[1] = f(8.5 * h)
    P.l[...] = rng.uniform(0.05, 0.95, size=n).astype(f) * f(h)
    Pd = P.to("torch", device="cuda", dtype=np.float32)
    W = tb.BasisWeights(2, n, np.float32, backend="torch", device="cuda")
    runtime.update(W, Pd, mesh, tb.step_params(1e-4, gimp_l=0.5 * h, basis=abi.TB_UGIMP), ctx=ctx)
    ctx.synchronize()
    gx = W.grad_w.cpu().numpy().reshape(n, 3, 3, 2)[..., 0]  # slots: x fastest
    lo = W.window.cpu().numpy()
    xi, l = P.x[0] * f(8), P.l * f(8)
    r = f(1) + l / f(2)
    first = np.floor(xi - r) + f(1)
    checked = 0
    for k in range(3):
        a = np.abs(xi - (first + f(k)))
        hl = l * f(0.5)
        ref = np.where(a < hl, (f(2) * a) / l, np.where(a < f(1) - hl, f(1),
                       np.where(a < f(1) + hl, (f(1) + hl - a) / l, f(0)))).astype(f)
        der = np.abs(gx[:, 0, k]) * f(2) * f(h)  # the first y slot has weight 1/2
        on = (first + f(k)) <= np.floor(xi + r)
        assert np.all(np.abs(der - ref)[on] <= np.spacing(ref)[on]), k
        checked += int(on.sum())
    assert checked > 2 * n and lo.shape[0] == n
