"""The sum-factorised tangent (the default kernel) against the direct form on the FMA pipe (kernel
option 0, an independent formulation), at the smallest and at ragged tile shapes, with element scales and a
periodic term.  Tolerances: both kernels sum products of 64-bit values, so they differ by rounding only
(1e-12 of the row's largest entry, the parity criterion); FP32 values round the 64-bit element entries and add
at most 27 of them, 28 half-ulps of 2^-24 of the largest partial sum, which stays below a few times the row's
largest entry (1e-5, the FP32 criterion of the parity suite)."""
import numpy as np
import pytest

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu

SIZES = [(1, 1, 1), (2, 1, 1), (1, 2, 3), (2, 2, 2), (3, 3, 3), (5, 4, 3), (2, 7, 1), (9, 2, 5)]


def _rowwise(rowptr, v, w):
    top = np.maximum.reduceat(np.abs(w), rowptr[:-1])
    return float(np.max(np.maximum.reduceat(np.abs(v - w), rowptr[:-1]) / top))


@pytest.mark.parametrize("ne", SIZES)
def test_against_direct_form(built, ne):
    from igap4standard_b200 import Assembly
    rng = np.random.default_rng(sum(ne))
    bc, pd = mesh.bc_config0()
    A = Assembly(ne, mesh.knots_for(ne, perturb=0.2, seed=2), mesh.par_mat_from_lame(0.7, 1.3, 0.15), bc, pd,
                 rng.uniform(-0.02, 0.02, 9))
    A.set_element_log_scale(rng.normal(0.0, 0.3, A.nelem_total))
    U = rng.uniform(-2e-2, 2e-2, A.ndof)
    rowptr, cols = A.pattern()
    out = {}
    for prec, option in (("fp64", 1), ("fp32", 2)):
        for kernel in (0, 1):
            A.set_option(option, kernel)
            out[prec, kernel] = A.tangent(U, prec)
    assert _rowwise(rowptr, out["fp64", 1], out["fp64", 0]) <= 1e-12
    assert _rowwise(rowptr, out["fp32", 1].astype(np.float64), out["fp64", 0]) <= 1e-5
    # the transposed entry is the same number
    import scipy.sparse as sp
    K = sp.csr_matrix((out["fp64", 1], cols, rowptr), shape=(A.ndof, A.ndof))
    assert abs(K - K.T).max() == 0.0
