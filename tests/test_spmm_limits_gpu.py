"""SpMM under capture and without memory for its scratch."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(n, seed=1):
    import torch
    from sparseops_b200 import CSR_Matrix, synth
    rp, ci, v = synth.powerlaw(n, hi=n // 4, seed=seed)
    return CSR_Matrix(n, n, *(torch.from_numpy(a).to("cuda") for a in (rp, ci, v))), (rp, ci, v)


def _runtime():
    for line in open("/proc/self/maps"):
        if "libcudart" in line:
            return ctypes.CDLL(line.split()[-1])
    pytest.skip("no shared CUDA runtime")


def _node_types(graph):
    rt, g, n = _runtime(), ctypes.c_void_p(graph.raw_cuda_graph()), ctypes.c_size_t(0)
    assert rt.cudaGraphGetNodes(g, None, ctypes.byref(n)) == 0
    nodes = (ctypes.c_void_p * n.value)()
    assert rt.cudaGraphGetNodes(g, nodes, ctypes.byref(n)) == 0
    out, t = [], ctypes.c_int()
    for q in nodes:
        assert rt.cudaGraphNodeGetType(ctypes.c_void_p(q), ctypes.byref(t)) == 0
        out.append(t.value)
    return out


@pytest.mark.parametrize("f32", [False, True])
@pytest.mark.parametrize("k", [1, 3, 8, 12, 16, 31, 32])
def test_captured_spmm(cuda, k, f32):
    """A captured SpMM gives the result of a plain call, on new X too, holds no
    allocation nodes (10 and 11), and two graphs of one matrix replay beside each
    other and beside plain calls."""
    import torch
    from sparseops_b200 import CSR_Matrix, SpMM_csr
    A, (rp, ci, v) = _matrix(20000)
    dt = torch.float32 if f32 else torch.float64
    n = A.num_rows
    A = CSR_Matrix(n, n, A.row_offset, A.col_index, A.values.to(dt))
    gen = torch.Generator(device="cuda").manual_seed(k)
    X = [torch.rand(n, k, dtype=dt, device="cuda", generator=gen) for _ in range(2)]
    Y = [torch.zeros(n, k, dtype=dt, device="cuda") for _ in range(2)]
    want = torch.zeros(n, k, dtype=dt, device="cuda")
    SpMM_csr(1.0, A, X[0], 0.0, want)
    graphs, streams = [], [torch.cuda.Stream(), torch.cuda.Stream()]
    for q in range(2):
        g = torch.cuda.CUDAGraph(keep_graph=True)
        with torch.cuda.graph(g, stream=streams[q]):
            SpMM_csr(1.0, A, X[q], 0.0, Y[q])
        assert not {10, 11} & set(_node_types(g))
        graphs.append(g)
    for turn in range(5):
        torch.cuda.synchronize()
        for q in range(2):
            with torch.cuda.stream(streams[q]):
                X[q].uniform_(-1, 1)
                Y[q].fill_(7.0)
                for _ in range(4):
                    graphs[q].replay()
        torch.cuda.synchronize()
        for q in range(2):
            SpMM_csr(1.0, A, X[q], 0.0, want)
            assert torch.equal(Y[q], want), (turn, q)


def test_captured_spmm_outlives_its_graph_only(cuda):
    """The scratch goes with the graph: many captures of one matrix do not add
    up."""
    import torch
    from sparseops_b200 import SpMM_csr
    A, _ = _matrix(300000)
    n, k = A.num_rows, 31
    X = torch.rand(n, k, dtype=torch.float64, device="cuda")
    Y = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    SpMM_csr(1.0, A, X, 0.0, Y)
    s = torch.cuda.Stream()
    free = []
    for _ in range(30):  # 14 MB each
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            SpMM_csr(1.0, A, X, 0.0, Y)
        g.replay()
        torch.cuda.synchronize()
        del g
        free.append(torch.cuda.mem_get_info()[0])
    assert free[2] - free[-1] < 100 << 20


def test_spmm_without_room_for_its_scratch(cuda, orc):
    """k = 31 wants 2k values per tile; where the device has no room for them
    the product is computed all the same."""
    import torch
    from sparseops_b200 import CSR_Matrix, SpMM_csr, Context
    n, per, k = 1 << 18, 128, 31
    rp = torch.arange(0, n * per + 1, per, dtype=torch.int32, device="cuda")
    ci = (torch.arange(n * per, dtype=torch.int64, device="cuda") * 7919 % n).to(torch.int32)
    v = torch.rand(n * per, dtype=torch.float64, device="cuda")
    X = torch.rand(n, k, dtype=torch.float64, device="cuda")
    out = []
    for hog in (False, True):
        A = CSR_Matrix(n, n, rp, ci, v)
        A.device(Context(0, torch.cuda.current_stream().cuda_stream or None))  # a pool of its own
        Y = torch.zeros(n, k, dtype=torch.float64, device="cuda")
        held = []
        torch.cuda.synchronize()
        if hog:  # leave 24 MB: the scratch takes 65 MB
            torch.cuda.empty_cache()
            for size in (1 << 30, 64 << 20, 8 << 20):
                while torch.cuda.mem_get_info()[0] > size + (24 << 20):
                    held.append(torch.empty(size, dtype=torch.uint8, device="cuda"))
        try:
            SpMM_csr(1.0, A, X, 0.0, Y)
            torch.cuda.synchronize()
        finally:
            del held
            torch.cuda.empty_cache()
        out.append(Y)
    err = ((out[1] - out[0]).abs() / out[0].abs()).max()
    assert float(err) <= 1e-13  # sums of 128 positive terms in two orders


def test_scratch_stays_while_its_graph_does(cuda):
    """The scratch of graphs that are kept stays allocated (their instances hold
    it, the captured graphs themselves are gone), and is given back after them."""
    import torch
    from sparseops_b200 import SpMM_csr
    A, _ = _matrix(300000)
    n, k = A.num_rows, 31
    X = torch.rand(n, k, dtype=torch.float64, device="cuda")
    Y = torch.zeros(n, k, dtype=torch.float64, device="cuda")
    SpMM_csr(1.0, A, X, 0.0, Y)
    s = torch.cuda.Stream()
    graphs, free = [], []

    def capture():
        g = torch.cuda.CUDAGraph()
        with torch.cuda.graph(g, stream=s):
            SpMM_csr(1.0, A, X, 0.0, Y)
        torch.cuda.synchronize()
        return g

    for _ in range(10):  # 14 MB each
        graphs.append(capture())
        free.append(torch.cuda.mem_get_info()[0])
    assert free[1] - free[-1] > 8 * (12 << 20)
    graphs.clear()
    torch.cuda.synchronize()
    capture()  # a later capture frees what the graphs left
    assert torch.cuda.mem_get_info()[0] - free[-1] > 8 * (12 << 20)
