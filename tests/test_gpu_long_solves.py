"""The FP64 loops over thousands of iterations.

The loops form s = A p from s = A r + beta s, so rounding could add up in s, and with it a gap
between the recursive residual, which ends the solve, and b - A x.  Systems: a tall column
under a free surface, and lattices whose coefficients spread over up to six decades.

Tolerance: the recursive residual ends below eps |b|; the gap may be as large again (factor
2).  eps is such that the CG with the product A p, run beside it in FP64 on the CPU, ends with
a true residual below eps itself.  The iteration counts differ by what rounding does to the
steps of an ill-conditioned solve: 5 %.
"""
import ctypes as C

import numpy as np
import pytest

from openmps_gb300 import _abi as abi

pytestmark = pytest.mark.gpu

# nx, nz, decades of the coefficients, eps
CASES = {
    "column": (30, 1000, 0, 1e-8),
    "two_decades_each_way": (60, 60, 4, 1e-9),
    "six_decades": (50, 100, 6, 1e-8),
    "three_decades": (100, 140, 3, 1e-10),
    "one_cluster": (40, 50, 4, 1e-9),
}


def _lattice(nx, nz, decades, seed):
    """Five-point operator with log-uniform coefficients, Dirichlet along the top row."""
    sp = pytest.importorskip("scipy.sparse")
    rng = np.random.default_rng(seed)
    n = nx * nz
    idx = np.arange(n).reshape(nx, nz)
    row, col, val = [], [], []
    for a, b in ((idx[1:], idx[:-1]), (idx[:, 1:], idx[:, :-1])):
        w = 10.0 ** rng.uniform(-decades / 2, decades / 2, a.size)
        row += [a.ravel(), b.ravel()]
        col += [b.ravel(), a.ravel()]
        val += [-w, -w]
    A = sp.csr_matrix((np.concatenate(val), (np.concatenate(row), np.concatenate(col))), shape=(n, n))
    d = -np.asarray(A.sum(1)).ravel()
    d[idx[:, -1]] += 1.0
    A = (A + sp.diags(d)).tocsr()
    A.sort_indices()
    return A


def _cg(A, b, eps):
    """CG with the product A p; iterations and true relative residual."""
    x, r, p, it = np.zeros_like(b), b.copy(), b.copy(), 0
    rr, thr = r @ r, eps * eps * (b @ b)
    while it < 40_000:
        s = A @ p
        alpha = rr / (p @ s)
        x += alpha * p
        r -= alpha * s
        it += 1
        new = r @ r
        if new < thr:
            break
        p = r + (new / rr) * p
        rr = new
    return it, np.linalg.norm(b - A @ x) / np.linalg.norm(b)


@pytest.mark.parametrize("which", ["cg64", "noalloc"])
@pytest.mark.parametrize("name", list(CASES))
def test_true_residual_after_many_iterations(gpu_lib, name, which):
    nx, nz, decades, eps = CASES[name]
    A = _lattice(nx, nz, decades, seed=1)
    n = A.shape[0]
    b = np.random.default_rng(3).standard_normal(n)
    it_direct, rel_direct = _cg(A, b, eps)
    assert rel_direct <= eps and it_direct >= 900
    ptr, col, val = A.indptr.astype(np.int64), A.indices.astype(np.int32), A.data
    if which == "cg64":
        from openmps_gb300.computer import Computer

        x, it, _ = Computer(abi.make_params()).cg_solve_csr(ptr, col, val, b, np.zeros(n), eps,
                                                            criterion=abi.CRIT_RHS, max_iters=40_000)
    else:
        torch = pytest.importorskip("torch")
        dev = [torch.from_numpy(a).cuda() for a in (ptr, col, val, b)]
        d_x = torch.zeros(n, dtype=torch.float64, device="cuda")
        count = C.c_int32()
        rc = gpu_lib.mps_cg_solve_csr_device_noalloc(n, *[d.data_ptr() for d in dev], d_x.data_ptr(), eps,
                                                     abi.CRIT_RHS, 40_000, None, C.byref(count), None)
        assert rc == abi.MPS_OK
        x, it = d_x.cpu().numpy(), count.value
    rel = np.linalg.norm(b - A @ x) / np.linalg.norm(b)
    print("%s %s: %d iterations (%d with A p), true residual %.3f eps (%.3f)" %
          (name, which, it, it_direct, rel / eps, rel_direct / eps))
    assert rel <= 2 * eps
    assert abs(it - it_direct) <= 0.05 * it_direct
