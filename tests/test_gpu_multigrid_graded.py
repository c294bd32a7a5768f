"""The V-cycle on graded meshes, whose largest eigenvalue of D^-1 K the power iteration underestimates most (24 elements
a side, the last twice as wide as the first: by 11%).  The smoother has to damp up to the true value, or the V-cycle is
not positive definite and CG breaks down.  The solve stops at a relative residual of 1e-8, which the true residual
(scipy's CSR product) meets up to the rounding of the recurrence, 2e-8 as in the cubic tests."""
import numpy as np
import pytest
import scipy.sparse as sp

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


def _graded_knots(ne, ratio):
    """Open knot vectors whose element widths grow geometrically, the last `ratio` times the first."""
    out = []
    for n in ne:
        x = np.concatenate([[0.0], np.cumsum(ratio ** (np.arange(n) / (n - 1)))])
        out.append(np.concatenate([[0.0, 0.0], x / x[-1], [1.0, 1.0]]))
    return np.concatenate(out)


@pytest.mark.parametrize("method", ["gmres", "cg"])
@pytest.mark.parametrize("ne,ratio", [((24, 24, 24), 2.0), ((24, 16, 20), 3.0), ((24, 24, 24), 5.0)])
def test_graded_mesh(built, ne, ratio, method):
    import torch
    from igap4standard_b200 import Assembly
    A = Assembly(ne, _graded_knots(ne, ratio), mesh.par_mat_from_lame(1.0, 1.0, 0.1), *mesh.bc_config0())
    s = torch.cuda.Stream()
    A.set_stream(s.cuda_stream)
    U = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
    b = torch.as_tensor(np.random.default_rng(1).normal(size=A.ndof)).cuda()
    V = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
    x = torch.empty_like(b)
    torch.cuda.synchronize()
    A.tangent_device(U.data_ptr(), V.data_ptr())
    A.sync()
    its, ok, rn, lev = A.solve_mg_device(V.data_ptr(), b.data_ptr(), x.data_ptr(), "fp64", 1e-8, 0.0, 2000, method)
    rp, cols = A.pattern()
    K = sp.csr_matrix((V.cpu().numpy(), cols, rp), shape=(A.ndof, A.ndof))
    bh = b.cpu().numpy()
    print("%s graded %g %s: levels %d, iterations %d" % (ne, ratio, method, lev, its))
    assert ok
    assert np.linalg.norm(bh - K @ x.cpu().numpy()) <= 2e-8 * np.linalg.norm(bh)
