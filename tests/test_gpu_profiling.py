"""igab_last_kernel_ms reports the last residual and tangent; other calls in between leave its events alone."""
import numpy as np
import pytest

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("ne", [(5, 4, 6), (17, 16, 17)])
def test_history_jacobian_leaves_the_tangent_times(built, ne):
    """Below and above the 4,096 elements up to which the tangent goes through the scratch."""
    import torch
    from igap4standard_b200 import Assembly
    pm = mesh.par_mat_from_lame(1.0, 1.0, 0.1)
    pm[5], pm[6], pm[7] = 1.0, 1.0, 1e-3
    bc, pd = mesh.bc_transient()
    A = Assembly(ne, mesh.knots_for(ne), pm, bc, pd, phys="getime")
    rng = np.random.default_rng(2)
    for level in (1, 2):
        A.set_history(level, rng.uniform(-1e-3, 1e-3, A.ndof))
    U = torch.as_tensor(rng.uniform(-1e-3, 1e-3, A.ndof)).cuda()
    V = torch.empty(A.nnz, dtype=torch.float64, device="cuda")
    J = torch.empty_like(V)
    torch.cuda.synchronize()
    A.set_profiling(True)
    A.tangent_device(U.data_ptr(), V.data_ptr())
    A.sync()
    before = A.last_kernel_ms()
    A.history_jacobian_device(U.data_ptr(), J.data_ptr(), 1)
    A.sync()
    assert A.last_kernel_ms() == before
    A.tangent_device(U.data_ptr(), V.data_ptr())     # the events still work
    A.sync()
    assert A.last_kernel_ms() != before
