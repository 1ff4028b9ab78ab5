"""Handles that go away while other work is under way: a capture on the same
device, products still queued on a stream the context has left."""
import gc
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _csr(n=3000, dtype=np.float64, seed=1, host=False):
    import torch
    from sparseops_b200 import CSR_Matrix, synth
    rp, ci, v = synth.banded_random(n, 16.0, 64, seed=seed)
    a = (rp, ci, v.astype(dtype))
    return CSR_Matrix(n, n, *(a if host else [torch.from_numpy(t).to("cuda") for t in a])), a


def _used(kind):
    """A matrix with everything its products build, ready to be destroyed."""
    import torch
    from sparseops_b200 import SpMM_csr, SpOps_csr, convert_to
    A, _ = _csr(host=kind == "host arrays")
    n = A.num_rows
    x, y = torch.ones(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    SpOps_csr(1.0, A, x, 0.0, y)
    if kind == "spmm":
        X, Y = torch.ones(n, 12, dtype=torch.float64, device="cuda"), torch.zeros(n, 12, dtype=torch.float64, device="cuda")
        SpMM_csr(1.0, A, X, 0.0, Y)
    if kind == "sell":
        return convert_to(A, "sell_c_sigma", sigma=512, chunk=32, layout=1)
    if kind == "array shown":
        S = convert_to(A, "sell_c_sigma", sigma=512, chunk=32, layout=1)
        S.reorder  # its address is asked for
        return S
    return A


@pytest.mark.parametrize("kind", ["borrowed arrays", "host arrays", "spmm", "sell", "array shown"])
@pytest.mark.parametrize("mode", ["global", "thread_local"])
def test_destroy_beside_a_capture(cuda, kind, mode):
    """Destroying a handle leaves a capture on another stream valid, in the
    capturing thread (a handle collected inside the capture) and in another."""
    import torch
    handles = [_used(kind), _used(kind)]
    x = torch.arange(1000, dtype=torch.float64, device="cuda")
    y = torch.zeros_like(x)
    torch.cuda.synchronize()
    gc.collect()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream(), capture_error_mode=mode):
        torch.mul(x, 2.0, out=y)
        handles.pop()
        t = threading.Thread(target=handles.pop)
        t.start()
        t.join()
        gc.collect()
        y.add_(1.0)
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, 2 * x + 1)
    assert _used(kind) is not None  # and the library goes on


def test_destroy_inside_a_captured_stream(cuda):
    """The context's own stream is being captured: its products are recorded,
    another handle goes away, the graph replays."""
    import torch
    from sparseops_b200 import SpOps_csr
    A, _ = _csr()
    n = A.num_rows
    x, y = torch.rand(n, dtype=torch.float64, device="cuda"), torch.zeros(n, dtype=torch.float64, device="cuda")
    SpOps_csr(1.0, A, x, 0.0, y)
    want = y.clone()
    other = [_used("sell")]
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=torch.cuda.Stream()):
        SpOps_csr(1.0, A, x, 0.0, y)
        other.pop()
    for _ in range(2):
        y.zero_()
        g.replay()
        torch.cuda.synchronize()
        assert torch.equal(y, want)
    assert _used("sell") is not None


def test_plan_rebuilt_after_a_stream_change(cuda, orc):
    """A product still queued on the stream the context has left keeps its plan:
    the plan's blocks are handed out again only after it."""
    import torch
    from sparseops_b200 import SpOps_csr, default_context
    A, (rp, ci, v) = _csr(400000)  # above the one-launch limit
    n = A.num_rows
    x = torch.rand(n, dtype=torch.float64, device="cuda")
    ref = orc.spmv_csr(rp, ci, v, x.cpu().numpy())
    den = orc.absdot(rp, ci, v, x.cpu().numpy())
    ctx = default_context()
    ys = [torch.zeros(n, dtype=torch.float64, device="cuda") for _ in range(3)]
    SpOps_csr(1.0, A, x, 0.0, ys[0])
    torch.cuda.synchronize()
    s1, s2 = torch.cuda.Stream(), torch.cuda.Stream()
    try:
        with torch.cuda.stream(s1):
            torch.cuda._sleep(100_000_000)
            SpOps_csr(1.0, A, x, 0.0, ys[1])
        with torch.cuda.stream(s2):
            ctx.set_option("csr_variant", 5)  # tiles of another width: a new plan
            SpOps_csr(1.0, A, x, 0.0, ys[2])
        torch.cuda.synchronize()
    finally:
        ctx.set_option("csr_variant", 0)
    for y in ys:
        assert (np.abs(y.cpu().numpy() - ref) / den).max() <= 1e-12


def test_assembly_gives_its_memory_back(cuda):
    """A one-off assembly of 60M triplets through the global sorts (one row has
    more than 512 entries), about 6 GB of temporaries: the context keeps at most
    2 GB of blocks and 1 GB of temporaries in each of arena and pool (1/8 of
    growth added), and nothing once it is closed."""
    import torch
    from sparseops_b200 import COO_Matrix, Context, coo_to_csr
    n, per = 1_000_000, 60
    rows = torch.arange(n * per, device="cuda", dtype=torch.int64)
    cols = (rows * 48271 % n).to(torch.int32)
    rows = (rows % n).to(torch.int32)
    rows[:600] = 5
    vals = torch.ones(n * per, dtype=torch.float64, device="cuda")
    ctx = Context(0)

    def held():
        torch.cuda.synchronize()
        return start - torch.cuda.mem_get_info()[0]

    start = torch.cuda.mem_get_info()[0]
    for _ in range(2):
        coo = COO_Matrix(n, n, rows, cols, vals)
        coo.device(ctx)
        A = coo_to_csr(coo, compact=True)
        assert A.num_nnzs > n
        del A, coo
        gc.collect()
        assert held() <= 4.4 * 2 ** 30
    ctx.close()
    assert held() <= 64 << 20
