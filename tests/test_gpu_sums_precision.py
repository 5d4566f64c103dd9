"""Bits that the FP32 transfers keep in the sums of a crowded block."""
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
