"""An element of x that no entry of the matrix reads stays out of y, whatever it
is: infinities and NaN in it change nothing.  Checked at sizes above the
one-launch form's limit with an nnz that ends inside a tile, for every CSR
variant, the other formats, a k = 1 batch and the adjoint."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _matrix(vtype, extra):
    """Column 0 and row 0 hold no entry; rows of 0 to 79 entries and one over
    many tiles; the last tile holds `extra` entries."""
    rng = np.random.default_rng(extra)
    n = 30000
    lens = rng.integers(0, 80, n)
    lens[0] = 0
    lens[77] = 9000
    lens[-1] += (extra - int(lens.sum())) % 256
    rp = np.concatenate([[0], np.cumsum(lens)]).astype(np.int32)
    ci = (1 + rng.integers(0, n - 1, rp[-1])).astype(np.int32)
    for r in (77, n - 1):  # the row that would take the entries past the end, without repeats
        ci[rp[r]:rp[r + 1]] = np.sort(rng.choice(np.arange(1, n), lens[r], replace=False))
    return n, rp, ci, rng.standard_normal(len(ci)).astype(vtype)


def _err(orc, rp, ci, v, x, y, transposed=False):
    n = len(rp) - 1
    a = np.abs(v).astype(np.float64)
    if transposed:
        ref, den = orc.spmv_t(rp, ci, v.astype(np.float64), x, n), orc.spmv_t(rp, ci, a, np.abs(x), n)
    else:
        ref, den = orc.spmv_csr(rp, ci, v.astype(np.float64), x), orc.absdot(rp, ci, v.astype(np.float64), x)
    return (np.abs(y.cpu().numpy() - ref) / np.maximum(den, 1e-300)).max()


@pytest.mark.parametrize("bad", [np.inf, np.nan])
@pytest.mark.parametrize("vtype,extra", [(np.float64, 1), (np.float64, 250), (np.float32, 137)])
def test_unread_x(cuda, orc, vtype, extra, bad):
    import torch
    from sparseops_b200 import Batch, CSR_Matrix, SpOps_csr, convert_to, default_context
    from sparseops_b200.spops import _spmv
    n, rp, ci, v = _matrix(vtype, extra)
    tol = 1e-12 if vtype == np.float64 else 1e-5
    rng = np.random.default_rng(1)
    x = rng.uniform(-1, 1, n).astype(vtype)
    xf = x.astype(np.float64)
    xf[0] = 0
    x[0] = bad
    xd = torch.from_numpy(x).to("cuda")
    dev = [torch.from_numpy(a).to("cuda") for a in (rp, ci, v)]
    ctx = default_context()
    try:
        for variant in range(11):
            ctx.set_option("csr_variant", variant)
            y = torch.full((n,), 3.0, dtype=xd.dtype, device="cuda")
            SpOps_csr(1.0, CSR_Matrix(n, n, *dev), xd, 0.0, y)
            assert _err(orc, rp, ci, v, xf, y) <= tol, variant
    finally:
        ctx.set_option("csr_variant", 0)
    A = CSR_Matrix(n, n, *dev)
    for fmt, params in (("csr5", {}), ("coo", {}), ("sell_c_sigma", dict(sigma=512, chunk=32, layout=1)),
                        ("sell_c_sigma", dict(sigma=512, chunk=4)), ("sell_c_R", dict(chunk=32, layout=1))):
        y = torch.full((n,), 3.0, dtype=xd.dtype, device="cuda")
        _spmv(1.0, convert_to(A, fmt, **params), xd, 0.0, y)
        assert _err(orc, rp, ci, v, xf, y) <= tol, fmt
    y = torch.full((n,), 3.0, dtype=xd.dtype, device="cuda")
    batch = Batch([A], k=1)
    batch.set_vectors([xd], [y])
    batch.run()
    assert _err(orc, rp, ci, v, xf, y) <= tol


@pytest.mark.parametrize("bands", [0, 1, 3])
@pytest.mark.parametrize("vtype", [np.float64, np.float32])
def test_unread_gradient(cuda, orc, vtype, bands):
    """A^T g: g of a row without entries, with the values read through the
    permutation (right after they changed) and from the reordered copy."""
    import torch
    from sparseops_b200._lib import call, dbl, vp
    from sparseops_b200 import CSR_Matrix, default_context
    n, rp, ci, v = _matrix(vtype, 91)
    g = np.random.default_rng(2).uniform(-1, 1, n).astype(vtype)
    gf = g.astype(np.float64)
    gf[0] = 0
    g[0] = np.inf
    gd = torch.from_numpy(g).to("cuda")
    ctx = default_context()
    ctx.set_option("adjoint_bands", bands)
    try:
        A = CSR_Matrix(n, n, *(torch.from_numpy(a).to("cuda") for a in (rp, ci, v)))
        h = A.device()
        for turn in range(4):
            if turn == 2:
                call("spops_matrix_touch", h.handle)
            y = torch.full((n,), 3.0, dtype=gd.dtype, device="cuda")
            call("spops_spmv_t", ctx.handle, dbl(1.0), h.handle, vp(gd.data_ptr()), dbl(0.0), vp(y.data_ptr()))
            assert _err(orc, rp, ci, v, gf, y, True) <= (1e-12 if vtype == np.float64 else 1e-5), turn
    finally:
        ctx.set_option("adjoint_bands", 0)
