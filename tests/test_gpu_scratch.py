"""Small meshes assemble through scratch arrays and a gather, larger ones (and the x slabs of the host entry
points, and captures by the caller) tile by tile: both add every value in the same order, so results must be
equal bit for bit, on whatever stream and under whichever capture."""
import numpy as np
import pytest

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


def _transient(ne):
    from igap4standard_b200 import Assembly
    rng = np.random.default_rng(sum(ne))
    pm = mesh.par_mat_from_lame(1.0, 1.0, 0.1)
    pm[5], pm[6], pm[7] = 1.0, 1.0, 1e-3
    bc, pd = mesh.bc_transient()
    A = Assembly(ne, mesh.knots_for(ne, perturb=0.1, seed=3), pm, bc, pd, phys="getime")
    U0 = rng.uniform(-1e-2, 1e-2, A.ndof)
    U1 = U0 + rng.uniform(-1e-2, 1e-2, A.ndof)
    A.set_history(1, U1)
    A.set_history(2, U0)
    return A, U1 + rng.uniform(-1e-2, 1e-2, A.ndof)


def _static(ne):
    from igap4standard_b200 import Assembly
    bc, pd = mesh.bc_config0()
    A = Assembly(ne, mesh.knots_for(ne, perturb=0.1, seed=3), mesh.par_mat_from_lame(1.0, 1.0, 0.1), bc, pd)
    return A, np.random.default_rng(sum(ne)).uniform(-1e-2, 1e-2, A.ndof)


def _device(A, U, prec, n=1):
    import torch
    Ud = torch.as_tensor(U).cuda()
    V = torch.full((A.nnz,), float("nan"), dtype=torch.float64 if prec == "fp64" else torch.float32, device="cuda")
    R = torch.full((A.ndof,), float("nan"), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    for _ in range(n):
        A.residual_device(Ud.data_ptr(), R.data_ptr())
        A.tangent_device(Ud.data_ptr(), V.data_ptr(), prec)
    A.sync()
    return Ud, R, V


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
@pytest.mark.parametrize("make", [_static, _transient])
def test_slabs_equal_scratch(built, make, prec):
    """23 or more elements along x: the host tangent goes slab by slab through the tiles."""
    A, U = make((25, 3, 2))
    _, _, V = _device(A, U, prec)
    assert np.array_equal(V.cpu().numpy(), A.tangent(U, prec))


def test_residual_without_scratch(built):
    """igab_residual_noalloc runs the tiles."""
    A, U = _static((3, 5, 4))
    R = np.empty(A.ndof)
    from igap4standard_b200.native import check, vp
    check(A.lib, "igab_residual_noalloc",
          A.lib.igab_residual_noalloc(A.h, U.ctypes.data_as(vp), R.ctypes.data_as(vp)))
    assert np.array_equal(R, A.residual(U))


@pytest.mark.parametrize("make", [_static, _transient])
def test_streams_and_captures(built, make):
    import torch
    A, U = make((6, 5, 7))
    Ud, R, V = _device(A, U, "fp64")
    R0, V0 = R.clone(), V.clone()
    A.graph_capture(Ud.data_ptr(), R.data_ptr(), V.data_ptr(), "fp64")
    for _ in range(3):        # replays and eager calls on changing streams share the scratch arrays
        R.zero_(), V.zero_()
        torch.cuda.synchronize()
        s = torch.cuda.Stream()
        A.set_stream(s.cuda_stream)
        A.graph_launch()
        t = torch.cuda.Stream()
        A.set_stream(t.cuda_stream)
        R2, V2 = torch.empty_like(R), torch.empty_like(V)
        A.residual_device(Ud.data_ptr(), R2.data_ptr())
        A.tangent_device(Ud.data_ptr(), V2.data_ptr())
        torch.cuda.synchronize()
        for r, v in ((R, V), (R2, V2)):
            assert torch.equal(r, R0) and torch.equal(v, V0)
    # a capture by the caller
    R.zero_(), V.zero_()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        A.set_stream(torch.cuda.current_stream().cuda_stream)
        A.residual_device(Ud.data_ptr(), R.data_ptr())
        A.tangent_device(Ud.data_ptr(), V.data_ptr())
    A.set_stream(torch.cuda.Stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(R, R0) and torch.equal(V, V0)


@pytest.mark.parametrize("ne,prec", [((9, 12, 13), "fp64"), ((9, 36, 37), "fp64"), ((11, 26, 26), "fp32"),
                                     ((13, 37, 37), "fp64"), ((14, 26, 27), "fp32")])
def test_host_steps_and_slabs(built, ne, prec):
    """The host tangent by steps of layers through a ring of layers (all of a small mesh, many, three of 1,332 elements,
    six of 676) and, with larger layers, by slabs of tiles: the values of the one-pass tangent."""
    A, U = _static(ne)
    _, _, V = _device(A, U, prec)
    for _ in range(2):
        assert np.array_equal(V.cpu().numpy(), A.tangent(U, prec))
