"""caelix_radix_sort_pairs_static in the caller's stream: its first command is ordered after everything that
the caller put there, also where one kernel is the whole sort."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def bind():
    import caelix_b200

    f = caelix_b200.library().lib.caelix_radix_sort_pairs_static
    f.restype = C.c_int
    f.argtypes = [C.c_uint64, C.c_uint64, C.c_uint32, C.c_uint32, C.c_uint64, C.c_uint64]
    return f


@pytest.mark.parametrize("n", [1, 512, 513, 4096, 4097])
def test_keys_of_an_async_copy(cuda_device, n):
    """The keys arrive by a copy enqueued just before."""
    import torch

    sort = bind()
    keys = np.random.default_rng(n).integers(0, 1 << 10, n, dtype=np.uint32)
    host = torch.from_numpy(keys.view(np.int32)).pin_memory()
    d_keys, d_values = (torch.empty(n, dtype=torch.int32, device="cuda") for _ in range(2))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        d_keys.fill_(-1)
        d_keys.copy_(host, non_blocking=True)
        assert sort(d_keys.data_ptr(), d_values.data_ptr(), n, 1, 0, stream.cuda_stream) == 0
    stream.synchronize()
    order = np.argsort(keys, kind="stable")
    assert np.array_equal(d_keys.cpu().numpy().view(np.uint32), keys[order])
    assert np.array_equal(d_values.cpu().numpy().view(np.uint32), order.astype(np.uint32))


@pytest.mark.parametrize("n", [1, 512, 513, 4096])
def test_first_kernel_depends_in_full(cuda_device, n):
    """In a captured stream (nothing is launched) the sort's kernel depends on the kernel before it by a plain
    edge, not by one that lets it start early."""
    import torch
    from cuda.bindings import runtime as rt

    sort = bind()
    d_keys, d_values = (torch.zeros(n, dtype=torch.int32, device="cuda") for _ in range(2))
    assert sort(d_keys.data_ptr(), d_values.data_ptr(), n, 1, 0, 0) == 0  # (lookups of the first call)
    torch.cuda.synchronize()
    stream = torch.cuda.Stream()
    ok = rt.cudaError_t.cudaSuccess
    (e,) = rt.cudaStreamBeginCapture(stream.cuda_stream, rt.cudaStreamCaptureMode.cudaStreamCaptureModeThreadLocal)
    assert e == ok
    for _ in range(2):  # the second sort's kernel follows the first's
        assert sort(d_keys.data_ptr(), d_values.data_ptr(), n, 1, 0, stream.cuda_stream) == 0
    e, graph = rt.cudaStreamEndCapture(stream.cuda_stream)
    assert e == ok
    # (The driver's call by ctypes: the runtime binding's edge data does not outlive its call.)
    nodes, edges, count = (C.c_void_p * 8)(), (C.c_uint8 * 64)(), C.c_size_t(8)  # an edge: from port, to port, type, 5 bytes
    assert C.CDLL("libcuda.so.1").cuGraphGetEdges_v2(C.c_void_p(int(graph)), nodes, (C.c_void_p * 8)(), edges, C.byref(count)) == 0
    assert count.value == 1 and edges[2] == int(rt.cudaGraphDependencyType.cudaGraphDependencyTypeDefault)
    assert rt.cudaGraphDestroy(graph)[0] == ok
