"""The host-pointer tangent where it has several parts to download: slabs of tiles (static and transient bounds) and
more steps of layers than there are events, in every colour order, with Dirichlet conditions on all faces.  The values
are those of the one-pass device tangent bit for bit.  The launches are counted, so that a mesh that no longer takes
the path it stands for is noticed."""
import numpy as np
import pytest

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


def _case(ne, phys):
    from igap4standard_b200 import Assembly
    rng = np.random.default_rng(sum(ne))
    pm = mesh.par_mat_from_lame(0.7, 1.3, 0.15)
    pm[5], pm[6], pm[7] = 1.0, 1.0, 1e-3
    A = Assembly(ne, mesh.knots_for(ne, perturb=0.2, seed=7), pm, rng.integers(0, 2, 36).astype(np.int32),
                 rng.uniform(-0.05, 0.05, 9), phys=phys)
    U = rng.uniform(-1e-2, 1e-2, A.ndof)
    if phys == "getime":
        A.set_history(1, U + rng.uniform(-1e-2, 1e-2, A.ndof))
        A.set_history(2, U + rng.uniform(-1e-2, 1e-2, A.ndof))
    assert A.dirichlet_rows().size > 0
    return A, U


@pytest.mark.parametrize("ne,phys,prec,parts,each", [
    ((25, 37, 37), "ge", "fp64", 3, 8),         # slabs of tiles: layers over 1,365 (FP32: 682) elements
    ((40, 26, 27), "ge", "fp32", 3, 8),
    ((24, 37, 38), "getime", "fp64", 2, 8),
    ((24, 27, 27), "getime", "fp32", 2, 8),
    ((100, 20, 20), "ge", "fp64", 50, 2),       # steps of layers: two events' worth of 32
    ((70, 30, 22), "getime", "fp32", 70, 2)])
def test_host_tangent_in_parts(built, ne, phys, prec, parts, each):
    import torch
    A, U = _case(ne, phys)
    Ud = torch.as_tensor(U).cuda()
    V = torch.empty(A.nnz, dtype=torch.float64 if prec == "fp64" else torch.float32, device="cuda")
    out = np.empty(A.nnz, dtype=np.float64 if prec == "fp64" else np.float32)
    for order in (0, 1, 2):
        A.set_option(3, order)
        V.fill_(float("nan"))
        torch.cuda.synchronize()
        A.tangent_device(Ud.data_ptr(), V.data_ptr(), prec)
        A.sync()
        out.fill(np.nan)
        A.tangent(U, prec, out=out)
        assert A.last_launch_count() >= each * parts
        assert torch.equal(torch.from_numpy(out), V.cpu())
