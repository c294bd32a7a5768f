"""The fused V-cycle on meshes of uneven shape: several levels with different sizes per direction, two levels, and one
level (odd element counts: the Jacobi preconditioner alone).  The solve stops at a relative residual of 1e-8, which the
true residual (scipy's CSR product) meets up to the rounding of the recurrence, 2e-8 as in the cubic tests."""
import numpy as np
import pytest
import scipy.sparse as sp

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["gmres", "cg"])
@pytest.mark.parametrize("ne,levels", [((24, 8, 16), 3), ((12, 4, 8), 2), ((7, 5, 6), 1)])
def test_uneven_levels(built, ne, levels, method):
    import torch
    from igap4standard_b200 import Assembly
    A = Assembly(ne, mesh.knots_for(ne, perturb=0.2, seed=5), mesh.par_mat_from_lame(1.0, 1.0, 0.1),
                 *mesh.bc_config0())
    s = torch.cuda.Stream()
    A.set_stream(s.cuda_stream)
    U = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
    b = torch.as_tensor(np.random.default_rng(1).normal(size=A.ndof)).cuda()
    V = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
    x = torch.empty_like(b)
    torch.cuda.synchronize()
    A.tangent_device(U.data_ptr(), V.data_ptr())
    A.sync()
    its, ok, rn, lev = A.solve_mg_device(V.data_ptr(), b.data_ptr(), x.data_ptr(), "fp64", 1e-8, 0.0, 20000, method)
    rp, cols = A.pattern()
    K = sp.csr_matrix((V.cpu().numpy(), cols, rp), shape=(A.ndof, A.ndof))
    bh = b.cpu().numpy()
    print("%s %s: levels %d, iterations %d" % (ne, method, lev, its))
    assert ok and lev == levels
    assert np.linalg.norm(bh - K @ x.cpu().numpy()) <= 2e-8 * np.linalg.norm(bh)


@pytest.mark.parametrize("ne,n0", [((16, 14, 12), 4032), ((16, 14, 14), 4608)])
def test_rows_loaded_whole_or_in_passes(built, ne, n0):
    """Fine levels on both sides of 4,096 control points (rows loaded whole, or in passes), on the legacy stream too
    (no graph): the two streams' solves run the same kernels, so their solutions are equal."""
    import torch
    from igap4standard_b200 import Assembly
    assert np.prod([n + 2 for n in ne]) == n0
    A = Assembly(ne, mesh.knots_for(ne, perturb=0.2, seed=5), mesh.par_mat_from_lame(1.0, 1.0, 0.1),
                 *mesh.bc_config0())
    U = torch.zeros(A.ndof, dtype=torch.float64, device="cuda")
    b = torch.as_tensor(np.random.default_rng(1).normal(size=A.ndof)).cuda()
    V = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
    s = torch.cuda.Stream()
    torch.cuda.synchronize()
    out = []
    for stream in (s.cuda_stream, 1):
        A.set_stream(stream)
        A.tangent_device(U.data_ptr(), V.data_ptr())
        x = torch.empty_like(b)
        torch.cuda.synchronize()
        ok = A.solve_mg_device(V.data_ptr(), b.data_ptr(), x.data_ptr(), "fp64", 1e-8, 0.0, 20000, "gmres")[1]
        A.sync()
        assert ok
        out.append(x.cpu().numpy())
    rp, cols = A.pattern()
    K = sp.csr_matrix((V.cpu().numpy(), cols, rp), shape=(A.ndof, A.ndof))
    assert np.linalg.norm(b.cpu().numpy() - K @ out[0]) <= 2e-8 * np.linalg.norm(b.cpu().numpy())
    assert np.array_equal(out[0], out[1])
