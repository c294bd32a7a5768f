"""The transient residual, tangent and history Jacobians against the same in plain torch, 64 bits (perf/cases.py: its own
basis, energy and assembly, none of this library's code), entry by entry: 1e-12 of the largest entry of the row, as the
parity tests take it, and 1e-5 for FP32 values.  One element, odd sizes, a mesh above the 4,096 elements of the scratch."""
import numpy as np
import pytest

from perf import cases as workload

pytestmark = pytest.mark.gpu


def _rowptr(nelem):
    width = [np.minimum(np.arange(n + 2) + 2, n + 1) - np.maximum(np.arange(n + 2) - 2, 0) + 1 for n in nelem]
    per = 3 * (width[0][:, None, None] * width[1][None, :, None] * width[2][None, None, :]).reshape(-1)
    return np.concatenate([[0], np.cumsum(np.repeat(per, 3))])


def _worst(got, want, rowptr, tol):
    got, want = got.cpu().numpy().astype(np.float64), want.cpu().numpy()
    scale = np.repeat(np.maximum.reduceat(np.abs(want), rowptr[:-1]), np.diff(rowptr)) if got.size == rowptr[-1] \
        else np.full(got.size, np.abs(want).max())
    return np.max(np.abs(got - want) / np.maximum(tol * scale, 1e-300))


@pytest.mark.parametrize("kind,prec,tol", [("transient", "fp64", 1e-12), ("transient", "fp32", 1e-5),
                                           ("jacobians", "fp64", 1e-12)])
@pytest.mark.parametrize("ne", [(1, 1, 1), (2, 3, 1), (5, 4, 7), (17, 16, 17)])
def test_entries(built, ne, kind, prec, tol):
    import torch
    case = dict(kind=kind, nx=ne[0], ny=ne[1], nz=ne[2], prec=prec, perturb=0.2)
    state = workload.prepare(case, 11)
    got = workload.run(state)
    state["A"].sync()
    torch.cuda.synchronize()
    want = workload.exact(case, 11)
    rp = _rowptr(ne)
    for g, w in zip(got, want):
        assert g.numel() == w.numel()
        assert _worst(g, w, rp, 1e-12 if g.dtype == torch.float64 else tol) <= 1.0
