"""The tangent on meshes of any length scale, against the CPU oracle within the parity tolerance (1e-12 of the row's largest
entry).  The basis's denominators carry a guard of 1e-15, so that on elements of width h the functions sum to 1 only
within 1e-15 / h: a kernel that takes the sum for 1 is 2e-7 off on a body of a micrometre, and 3e-12 on a graded mesh of
unit size.  Transient matrices: with equal levels and no inertia the tangent is a quarter of the static one, the history
Jacobians a half and a quarter."""
import numpy as np
import pytest

from cases import tangent_tolerance
from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


def _knots(ne, length, ratio):
    out = []
    for n in ne:
        x = np.concatenate([[0.0], np.cumsum(ratio ** (np.arange(n) / max(n - 1, 1)))])
        x = x / x[-1] * length
        out.append(np.concatenate([[0.0, 0.0], x, [length, length]]))
    return np.concatenate(out)


@pytest.mark.parametrize("length,ratio", [(1e-6, 1.0), (1e-6, 5.0), (1e-3, 2.0), (1.0, 1000.0), (1e6, 1.0)])
@pytest.mark.parametrize("ne", [(1, 1, 1), (3, 5, 4)])
def test_tangents(built, port_oracle, ne, length, ratio):
    import torch
    from igap4standard_b200 import Assembly
    kn = _knots(ne, length, ratio)
    bc = np.ones(36, dtype=np.int32)
    U = np.random.default_rng(4).uniform(-1e-2, 1e-2, mesh.n_dof(ne)) * length
    pm = mesh.par_mat_from_lame(1.0, 1.0, 0.1 * length)
    rp, cols, want = port_oracle.PortCase(ne, kn, pm, bc).tangent(U)
    tol = tangent_tolerance(rp, want)
    A = Assembly(ne, kn, pm, bc)
    assert np.max(np.abs(A.tangent(U, "fp64") - want) / tol) <= 1.0
    pm[5], pm[6], pm[7] = 0.0, 0.0, 1e-3
    T = Assembly(ne, kn, pm, bc, phys="getime")
    T.set_history(1, U)
    T.set_history(2, U)
    Ud = torch.as_tensor(U).cuda()
    V = torch.empty(T.nnz, dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    assert np.max(np.abs(4.0 * T.tangent(U, "fp64") - want) / tol) <= 1.0
    for level, factor in ((1, 2.0), (2, 4.0)):
        T.history_jacobian_device(Ud.data_ptr(), V.data_ptr(), level)
        T.sync()
        assert np.max(np.abs(factor * V.cpu().numpy() - want) / tol) <= 1.0
