"""Shared helpers of the GPU parity tests."""
import ctypes as C

import numpy as np


def to_dev(torch, a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def captured_grids(torch, queue):
    """The grid's x of every kernel that queue() launches, from a capture of it."""
    queue()                                        # function attributes are set outside the capture
    graph = torch.cuda.CUDAGraph(keep_graph=True)
    with torch.cuda.graph(graph):
        queue()
    driver, handle, count = C.CDLL("libcuda.so.1"), C.c_void_p(graph.raw_cuda_graph()), C.c_size_t(0)
    assert driver.cuGraphGetNodes(handle, None, C.byref(count)) == 0
    nodes = (C.c_void_p * count.value)()
    assert driver.cuGraphGetNodes(handle, nodes, C.byref(count)) == 0
    grids = []
    for node in nodes:
        kind, params = C.c_int(-1), (C.c_uint32 * 32)()   # CUDA_KERNEL_NODE_PARAMS: the function, then gridDimX
        assert driver.cuGraphNodeGetType(C.c_void_p(node), C.byref(kind)) == 0
        if kind.value == 0:
            assert driver.cuGraphKernelNodeGetParams(C.c_void_p(node), params) == 0
            grids.append(params[2])
    return grids


def assert_close_to_f64(got, f32_oracle, sum64, abs64, what=""):
    """The F32 bar of the path: each output within 1e-5 of the magnitude of its
    own block products (sum |block product|, the reference's
    tests/unit/decode_gpu_test.cc style bound), the vector within NMSE 1e-10 of
    the double sum (tests/unit/dsv4_fast_test.cc:875-947), and within 1e-5
    relative of the oracle's F32 evaluation at the vector's scale."""
    got = np.asarray(got, np.float64)
    assert np.isfinite(got).all(), what
    err = np.abs(got - sum64)
    assert (err <= 1e-5 * abs64 + 1e-30).all(), (what, float((err / (abs64 + 1e-30)).max()))
    nmse = float(((got - sum64) ** 2).sum() / max(float((sum64 ** 2).sum()), 1e-300))
    assert nmse <= 1e-10, (what, nmse)
    scale = float(np.abs(f32_oracle).max())
    assert float(np.abs(got - f32_oracle).max()) <= 1e-5 * scale, what
