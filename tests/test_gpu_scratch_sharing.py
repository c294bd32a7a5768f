"""The scratch arrays of the assembly beside other contexts, streams and captures."""
import threading

import numpy as np
import pytest

from igap4standard_b200 import mesh

pytestmark = pytest.mark.gpu

TOTAL = 4 << 30        # bytes that the scratch arrays of all contexts of a device take together, at most


def _mesh(n=16):
    from igap4standard_b200 import Assembly
    ne = (n, n, n)
    return Assembly(ne, mesh.knots_for(ne, perturb=0.1, seed=3), mesh.par_mat_from_lame(1.0, 1.0, 0.1),
                    *mesh.bc_config0())


def _vectors(A, amp=1e-2, seed=1):
    import torch
    U = torch.as_tensor(np.random.default_rng(seed).uniform(-amp, amp, A.ndof)).cuda()
    return U, torch.empty_like(U), torch.empty(A.nnz, dtype=torch.float64, device="cuda")


def test_scratch_of_many_contexts_is_bounded(built):
    """36 meshes of 16^3 would take 5.2 GB.  The ones beyond the bound work without a scratch, with the same values, and
    the scratch of a destroyed context is there for the next one."""
    import torch
    many = [_mesh() for _ in range(36)]
    U, R, V = _vectors(many[0])
    R1, V1 = torch.empty_like(R), torch.empty_like(V)
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    for k, A in enumerate(many):
        r, v = (R, V) if k else (R1, V1)
        r.fill_(float("nan")), v.fill_(float("nan"))
        torch.cuda.synchronize()
        A.residual_device(U.data_ptr(), r.data_ptr())
        A.tangent_device(U.data_ptr(), v.data_ptr())
        A.sync()
        assert torch.equal(r, R1) and torch.equal(v, V1)
    torch.cuda.synchronize()
    grown = free - torch.cuda.mem_get_info()[0]
    print("%.2f GB" % (grown / 1e9))
    assert grown <= TOTAL + (256 << 20)          # the comparisons' and the kernels' own memory beside the scratch
    for A in many:
        A.close()
    A = _mesh()
    torch.cuda.synchronize()
    free = torch.cuda.mem_get_info()[0]
    A.tangent_device(U.data_ptr(), V.data_ptr())
    A.sync()
    assert free - torch.cuda.mem_get_info()[0] >= 16 ** 3 * 4374 * 8
    assert torch.equal(V, V1)


def test_first_call_beside_a_capture(built):
    """A context's first assembly, on its own stream, while another stream is captured in the global mode: the capture
    goes on, and both results are right."""
    import torch
    A, B = _mesh(6), _mesh(6)
    U, R, V = _vectors(A)
    R1, V1 = torch.empty_like(R), torch.empty_like(V)
    x = torch.ones(1000, device="cuda")
    B.residual_device(U.data_ptr(), R1.data_ptr())
    B.tangent_device(U.data_ptr(), V1.data_ptr())
    B.sync()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode="global"):
        x.add_(1.0)
        A.residual_device(U.data_ptr(), R.data_ptr())
        A.tangent_device(U.data_ptr(), V.data_ptr())
        x.mul_(2.0)
    A.sync()
    assert torch.equal(R, R1) and torch.equal(V, V1)
    g.replay()
    torch.cuda.synchronize()
    assert bool((x == 4.0).all())


def test_per_thread_stream_of_two_threads(built):
    """cudaStreamPerThread is one handle and a stream per thread: the second thread's assembly comes after the first
    one's, with which it shares the scratch, although the handles are equal."""
    import torch
    A = _mesh(6)
    U, R, V = _vectors(A)
    V2 = torch.empty_like(V)
    A.tangent_device(U.data_ptr(), V.data_ptr())
    A.sync()
    want = V.clone()
    torch.cuda.synchronize()
    per_thread = 2
    A.set_stream(per_thread)
    done = [None, None]

    def go(i, out, cycles):
        with torch.cuda.stream(torch.cuda.ExternalStream(per_thread)):
            if cycles:
                torch.cuda._sleep(cycles)
            A.tangent_device(U.data_ptr(), out.data_ptr())
            done[i] = torch.cuda.Event()
            done[i].record()

    go(0, V, 400_000_000)          # 0.2 s ahead of the first assembly
    t = threading.Thread(target=go, args=(1, V2, 0))
    t.start()
    t.join()
    done[1].synchronize()
    assert done[0].query()
    torch.cuda.synchronize()
    assert torch.equal(V, want) and torch.equal(V2, want)
