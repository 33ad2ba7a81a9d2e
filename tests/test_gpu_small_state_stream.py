"""What a caller sees of a small state's ops right after applying them.

Ops wait on the host to be launched together. Below 14 qubits the counters
and the stream show them launched all the same: the counters count them, and a
caller that has the stream finds every op on it as it is applied (here: in a
stream capture, whose graph holds one node per CX).
"""

import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

H = np.array([[1, 1], [1, -1]]) / np.sqrt(2)


@pytest.mark.parametrize("n", (3, 9, 13))
@pytest.mark.parametrize("prec,flags", ((64, 0), (64, 1), (32, 1)))
def test_counters_are_current(zc, n, prec, flags):
    be = zc.CudaBackend(n, prec, flags)
    c0 = be.counters()
    for q in range(3):
        be.apply_unitary([q], H)
    c1 = be.counters()
    assert c1["ops"] - c0["ops"] == 3
    assert c1["launches"] > c0["launches"] and c1["bytes_moved"] > c0["bytes_moved"]
    be.close()


def _cudart():
    for name in ("libcudart.so.13", "libcudart.so", "/usr/local/cuda/lib64/libcudart.so"):
        try:
            return ctypes.CDLL(name)
        except OSError:
            pass
    pytest.skip("no shared CUDA runtime")


@pytest.mark.parametrize("prec,flags", ((64, 0), (64, 1), (32, 1)))
def test_ops_are_on_the_stream(zc, prec, flags):
    rt = _cudart()
    be = zc.CudaBackend(5, prec, flags)
    be.apply_unitary([1], H)
    stream = ctypes.c_void_p(be.stream())
    be.apply_cx(1, 3)  # (loads the kernel: that does not go into a capture)
    assert rt.cudaStreamSynchronize(stream) == 0
    graph, nodes = ctypes.c_void_p(), ctypes.c_size_t()
    assert rt.cudaStreamBeginCapture(stream, 2) == 0  # relaxed
    be.apply_cx(3, 4)
    be.apply_cx(4, 2)
    assert rt.cudaStreamEndCapture(stream, ctypes.byref(graph)) == 0
    assert rt.cudaGraphGetNodes(graph, None, ctypes.byref(nodes)) == 0
    assert nodes.value == 2
    assert rt.cudaGraphDestroy(graph) == 0
    v = be.statevector()  # of what ran: H and the first CX
    assert np.allclose(v[[0, 0b01010]], 1 / np.sqrt(2)) and np.allclose(np.delete(v, [0, 0b01010]), 0)
    be.close()


def test_larger_states_keep_their_queue(zc):
    be = zc.CudaBackend(14, 64)
    c0 = be.counters()["launches"]
    be.stream()
    be.apply_unitary([1], H)
    be.apply_unitary([2], H)
    assert be.counters()["launches"] == c0
    be.finish()
    assert be.counters()["launches"] == c0 + 1
    be.close()
