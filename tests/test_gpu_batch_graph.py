"""A captured batch assembly after a change of the schedule: a replay gives the values of the present colour order, bit
for bit.  Directions with odd numbers of tiles, where the tiles per colour differ."""
import numpy as np
import pytest

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("prec", ["fp64", "fp32"])
def test_replay_after_a_colour_order_change(built, prec):
    import torch
    from igap4standard_b200 import Batch
    inst = []
    for k, ne in enumerate([(5, 6, 10), (9, 10, 6), (1, 2, 5), (6, 5, 1)]):
        bc, pd = mesh.bc_config0()
        inst.append(dict(nelem=ne, knots=mesh.knots_for(ne, perturb=0.2, seed=k),
                         par_mat=mesh.par_mat_from_lame(1.0, 1.0 + 0.1 * k, 0.1), bc_type=bc, par_dirichlet=pd))
    B = Batch(inst)
    U = torch.as_tensor(np.random.default_rng(3).uniform(-1e-2, 1e-2, B.ndof)).cuda()
    dt = torch.float64 if prec == "fp64" else torch.float32
    R = torch.empty_like(U)
    V = torch.empty(B.nnz, dtype=dt, device="cuda")
    torch.cuda.synchronize()
    want = {}
    for order in (0, 1, 2):
        B.set_colour_order(order)
        B.residual_device(U.data_ptr(), R.data_ptr())
        B.tangent_device(U.data_ptr(), V.data_ptr(), prec)
        B.sync()
        want[order] = R.clone(), V.clone()
        torch.cuda.synchronize()
    assert not torch.equal(want[0][1], want[1][1])     # the orders are told apart by the rounding
    B.set_colour_order(0)
    B.graph_capture(U.data_ptr(), R.data_ptr(), V.data_ptr(), prec)
    for order, largest_first in ((0, 0), (1, 0), (2, 1), (0, 1), (1, 1)):
        B.set_colour_order(order)
        B.set_schedule(order=largest_first)
        R.fill_(float("nan")), V.fill_(float("nan"))
        torch.cuda.synchronize()
        B.graph_launch()
        B.sync()
        assert torch.equal(R, want[order][0]) and torch.equal(V, want[order][1]), order
