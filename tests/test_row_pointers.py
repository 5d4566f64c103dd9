"""Row pointers of the (k, n) state arrays: an array with too few rows is refused
(its missing rows would be addresses past its end), a list of row tensors is as good
as one tensor, rows follow the array's stride, and no array or no particles is NULL."""
import numpy as np
import pytest
import torch


def _ints(field, k):
    return [field[i] or 0 for i in range(k)]


@pytest.mark.parametrize("backend", ["numpy", "torch"])
def test_too_few_rows_are_refused(tb, backend):
    P = tb.Particles(7, 3, np.float64, backend=backend, device="cpu", optional=("B",))
    for name, rows in (("x", 3), ("v", 3), ("sigma", 6), ("F", 9), ("B", 9)):
        whole = getattr(P, name)
        setattr(P, name, whole[:rows - 1])
        with pytest.raises(IndexError):
            P.struct()
        setattr(P, name, whole)
    P.struct()
    G = tb.generate_grid(tb.CartesianMesh(0.25, (0.0, 1.0), (0.0, 1.0)), np.float64, backend=backend, device="cpu")
    G.mv = G.mv[:1]
    with pytest.raises(IndexError):
        G.struct()


def test_rows_follow_the_array(tb):
    P = tb.Particles(8, 2, np.float32, backend="torch", device="cpu")
    P.v = [torch.zeros(8), torch.zeros(8)]  # rows that are tensors of their own
    P.x = torch.zeros(4, 10)[::2, 1:9]      # every other row of a wider array
    s = P.struct()
    assert _ints(s.v, 2) == [t.data_ptr() for t in P.v]
    assert _ints(s.x, 2) == [P.x[0].data_ptr(), P.x[1].data_ptr()]
    Q = tb.Particles(8, 2, np.float64)
    Q.x = np.zeros((8, 2)).T[:, ::1]
    assert _ints(Q.struct().x, 2) == [Q.x[0].ctypes.data, Q.x[1].ctypes.data]


def test_no_particles_and_no_array_are_null(tb):
    P = tb.Particles(0, 3, np.float64, backend="torch", device="cpu")
    s = P.struct()
    assert _ints(s.x, 3) == [0, 0, 0]
    assert _ints(s.B, 9) == [0] * 9
