"""Chains of overlapped launches, each reading what the one before wrote: the
same bits as with a wait for the device between them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _chain(step, wait, turns=60):
    import torch
    for t in range(turns):
        step(t)
        if wait:
            torch.cuda.synchronize()


@pytest.mark.parametrize("vtype", [np.float32, np.float64])
@pytest.mark.parametrize("n", [700, 20000, 400000])
@pytest.mark.parametrize("what", ["csr", "sell", "spmm", "adjoint"])
def test_products_of_products(cuda, what, n, vtype):
    """y = A x, x = A y, ... (values and gradients in turn for the adjoint),
    across rows that end in other tiles."""
    import torch
    from sparseops_b200 import CSR_Matrix, SpMM_csr, SpOps_csr, SpOps_sell_c_sigma, csr_to_sell_c_sigma, synth
    from sparseops_b200._lib import call, dbl, vp
    rp, ci, v = synth.powerlaw(n, hi=min(3000, n // 4), seed=2)
    v = (v / np.maximum(np.diff(rp), 1).repeat(np.diff(rp))).astype(vtype)  # rows sum to at most 1
    A = CSR_Matrix(n, n, *(torch.from_numpy(a).to("cuda") for a in (rp, ci, v)))
    S = csr_to_sell_c_sigma(A, slicewidth=512, chunkwidth=32, layout=1) if what == "sell" else None
    dt = torch.from_numpy(v).dtype
    k = 5 if what == "spmm" else 1
    start = torch.rand(n, k, dtype=dt, device="cuda", generator=torch.Generator(device="cuda").manual_seed(3))
    out = []
    for wait in (True, False):
        a = [start.clone().reshape(-1) if k == 1 else start.clone(), torch.zeros_like(start).reshape(-1 if k == 1 else (n, k))]
        vals = A.values.clone()
        B = CSR_Matrix(n, n, A.row_offset, A.col_index, vals)
        h = B.device()

        def step(t):
            x, y = a[t % 2], a[1 - t % 2]
            if what == "csr":
                SpOps_csr(1.0, A, x, 0.0, y)
            elif what == "sell":
                SpOps_sell_c_sigma(1.0, S, x, 0.0, y)
            elif what == "spmm":
                SpMM_csr(1.0, A, x, 0.0, y)
            elif t % 3 == 2:  # the matrix's own values from the two vectors
                call("spops_sddmm", h.ctx.handle, dbl(0.01), h.handle, vp(x.data_ptr()), vp(y.data_ptr()),
                     vp(vals.data_ptr()))
                call("spops_matrix_touch", h.handle)
            elif t % 3 == 1:
                call("spops_spmv_t", h.ctx.handle, dbl(1.0), h.handle, vp(x.data_ptr()), dbl(0.0), vp(y.data_ptr()))
            else:
                SpOps_csr(1.0, B, x, 0.0, y)

        torch.cuda.synchronize()
        _chain(step, wait)
        torch.cuda.synchronize()
        out.append([t.clone() for t in a] + [vals])
    assert all(torch.isfinite(t).all() for t in out[0])
    assert all(torch.equal(p, q) for p, q in zip(*out))
