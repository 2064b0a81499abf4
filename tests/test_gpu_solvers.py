"""The charge solvers at the sizes where their work split changes: fewer rows than warps, ragged blocks of rows, empty and
long rows."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _random_csr(n, seed):
    """A symmetric positive definite (diag(eta) + H): rows of 0 to min(n - 1, 300) entries, |H| well below eta."""
    rng = np.random.default_rng(seed)
    H = np.zeros((n, n))
    for i in range(n):
        m = int(rng.integers(0, min(n, 150)))
        j = rng.choice(n, size=m, replace=False)
        H[i, j] = rng.uniform(0.0, 1.0, size=m)
    H = np.triu(H, 1)
    H += H.T
    eta = H.sum(1) + rng.uniform(1.0, 3.0, size=n)
    rows, cols = np.nonzero(H)
    rs = np.concatenate([[0], np.cumsum(np.bincount(rows, minlength=n))]).astype(np.int32)
    return H, rs, cols.astype(np.int32), H[rows, cols], eta, rng.uniform(-5.0, 5.0, size=n)


@pytest.mark.parametrize("n", [2, 3, 15, 16, 17, 64, 129, 255, 257, 1000, 1999])
def test_static_solve_sizes_match_dense(n):
    """Sizes on both sides of a block's 16 rows and of the cluster's halvings, against the dense FP64 solution. At tol 1e-12
    the residual bounds the error: |x - x*| <= cond * tol * |x|; the matrices are diagonally dominant by a factor that keeps
    cond below 1e3, hence 1e-8 of the largest charge."""
    import torch
    import rxcuda
    H, rs, col, val, eta, chi = _random_csr(n, 100 + n)
    dev = torch.device("cuda", 0)
    up = lambda a: torch.from_numpy(np.ascontiguousarray(a)).to(dev)  # noqa: E731
    nnz = len(col)
    rs_d, col_d, val_d = up(rs), up(np.append(col, 0).astype(np.int32)), up(np.append(val, 0.0))
    eta_d, chi_d = up(eta), up(chi)
    s, t, q = (torch.zeros(n, dtype=torch.float64, device=dev) for _ in range(3))
    it, rel = torch.zeros(2, dtype=torch.int32, device=dev), torch.zeros(2, dtype=torch.float64, device=dev)
    lib = rxcuda.load()
    err = ctypes.create_string_buffer(256)
    rc = lib.rx_qeq_solve_static(n, rs_d.data_ptr(), col_d.data_ptr(), val_d.data_ptr(), eta_d.data_ptr(), chi_d.data_ptr(),
                                 s.data_ptr(), t.data_ptr(), q.data_ptr(), 1e-12, 500, it.data_ptr(), rel.data_ptr(),
                                 torch.cuda.current_stream(dev).cuda_stream, err, 256)
    assert rc == 0, err.value.decode()
    torch.cuda.synchronize(dev)
    A = np.diag(eta) + H
    s_ref, t_ref = np.linalg.solve(A, -chi), np.linalg.solve(A, -np.ones(n))
    q_ref = s_ref - s_ref.sum() / t_ref.sum() * t_ref
    assert nnz == rs[-1]
    assert rel.cpu().numpy().max() <= 1e-12 and it.cpu().numpy().max() < 500
    for got, ref in ((s, s_ref), (t, t_ref), (q, q_ref)):
        assert np.abs(got.cpu().numpy() - ref).max() <= 1e-8 * max(1.0, np.abs(ref).max())
