"""The plain solvers' single-launch loops at the edges of their work split.

mps_cg_solve_csr and the allocation-free solve run on a caller's system, so the systems here choose the
sizes: rows around a chunk (32), around the largest system one cluster takes (80 and 128
chunks), several tiles of chunks per block, more chunks than a block's tables hold, rows
longer than the usual unit, and identity rows (left out of the loop when their residual is
zero, kept when it is not).

Tolerance: each system is symmetric and strictly diagonally dominant with off-diagonal row
sums of at most half the diagonal, so its condition number is at most 3 d_max / d_min <= 6,
and |b - A x| <= 1e-12 |b| leaves |x - x*| <= 6e-12 |x*|; b = A x* adds rounding of 1e-15.
"""
import numpy as np
import pytest

from openmps_gb300 import _abi as abi

pytestmark = pytest.mark.gpu

TOL = 1e-11


def _system(n, offsets, seed, identity=0.0, dense_row=False):
    """CSR of a banded symmetric system, x* and a starting guess."""
    rng = np.random.default_rng(seed)
    idn = rng.random(n) < identity
    rows, cols, vals = [], [], []
    for k in offsets:
        if k >= n:
            continue
        i = np.arange(n - k)
        i = i[~idn[i] & ~idn[i + k]]
        v = rng.uniform(0.1, 1.0, i.size)
        rows += [i, i + k]
        cols += [i + k, i]
        vals += [v, v]
    if dense_row and n > 2:
        j = np.arange(1, n)
        j = j[~idn[j] & ~idn[0]]
        v = rng.uniform(0.1, 1.0, j.size)
        rows += [np.zeros(j.size, np.int64), j]
        cols += [j, np.zeros(j.size, np.int64)]
        vals += [v, v]
    row = np.concatenate(rows) if rows else np.zeros(0, np.int64)
    col = np.concatenate(cols) if cols else np.zeros(0, np.int64)
    val = np.concatenate(vals) if vals else np.zeros(0)
    # scaled so that no row's off-diagonal sum passes half of the diagonal 1 .. 2
    total = np.bincount(row, weights=val, minlength=n)
    val = val * (0.5 / max(total.max(), 1e-300)) if row.size else val
    diag = np.where(idn, 1.0, rng.uniform(1.0, 2.0, n))
    row = np.concatenate([row, np.arange(n)])
    col = np.concatenate([col, np.arange(n)])
    val = np.concatenate([val, diag])
    order = np.lexsort((col, row))
    row, col, val = row[order], col[order], val[order]
    ptr = np.zeros(n + 1, np.int64)
    ptr[1:] = np.cumsum(np.bincount(row, minlength=n))
    xs = rng.standard_normal(n)
    b = np.add.reduceat(val * xs[col], ptr[:-1])
    x0 = xs + rng.standard_normal(n)
    still = idn & (rng.random(n) < 0.5)  # identity rows that start at their solution
    if identity > 0:
        still |= idn & (np.arange(n) // 32 % 2 == 0)
    x0[still] = b[still]
    return ptr, col.astype(np.int32), val, b, xs, x0


CASES = {
    "one_row": dict(n=1, offsets=()),
    "below_chunk": dict(n=31, offsets=(1,)),
    "chunk": dict(n=32, offsets=(1, 7)),
    "above_chunk": dict(n=33, offsets=(1, 7)),
    "cluster64_edge": dict(n=80 * 32, offsets=(1, 2, 50, 51, 52)),
    "cluster64_past": dict(n=80 * 32 + 1, offsets=(1, 2, 50, 51, 52)),
    "cluster32_edge": dict(n=128 * 32, offsets=(1, 2, 64, 65)),
    "cluster32_past": dict(n=128 * 32 + 1, offsets=(1, 2, 64, 65)),
    "identity_rows": dict(n=5000, offsets=(1, 2, 3, 70, 71, 72), identity=0.7),
    "all_but_identity": dict(n=20000, offsets=(1,), identity=0.98),
    "long_row": dict(n=700, offsets=(1, 2), dense_row=True),
    "wide_rows": dict(n=9000, offsets=tuple(range(1, 46))),
    "two_tiles": dict(n=152 * 32 * 45 + 5, offsets=(1, 500)),
    "tables_rebuilt": dict(n=1_700_001, offsets=(1,)),
}


@pytest.mark.parametrize("solver", ["cg64", "mixed"])
@pytest.mark.parametrize("name", list(CASES))
def test_loop_sizes(gpu_lib, name, solver):
    from openmps_gb300.computer import Computer

    ptr, col, val, b, xs, x0 = _system(seed=len(name), **CASES[name])
    c = Computer(abi.make_params())
    which = abi.SOLVER_CG64 if solver == "cg64" else abi.SOLVER_MIXED
    x, it, rel = c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    err = float(np.linalg.norm(x - xs) / np.linalg.norm(xs))
    print("%s %s: n %d, %d iterations, relres %.2e, error %.2e" % (name, solver, len(b), it, rel, err))
    assert rel <= 1.01e-12
    assert err <= TOL
    again, it2, _ = c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    assert it2 == it and np.array_equal(x, again)  # every sum has a fixed order


# past the rows whose chunks a block's tables surely hold: more chunks in the loop than the
# tables (whole chunks walked, some left out, rows of one step and of several), and so many
# left out that the tables hold the rest
PAST_TABLES = {
    "walked": dict(n=1_300_003, offsets=(1, 2, 3, 4, 5, 6)),
    "walked_past_left_out": dict(n=3_200_001, offsets=(1,), identity=0.98),
    "tables_hold_the_rest": dict(n=1_700_001, offsets=(1,), identity=0.98),
}


@pytest.mark.parametrize("solver", ["cg64", "mixed"])
@pytest.mark.parametrize("name", list(PAST_TABLES))
def test_past_the_tables(gpu_lib, name, solver):
    from openmps_gb300.computer import Computer

    ptr, col, val, b, xs, x0 = _system(seed=len(name), **PAST_TABLES[name])
    c = Computer(abi.make_params())
    which = abi.SOLVER_CG64 if solver == "cg64" else abi.SOLVER_MIXED
    x, it, rel = c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    assert rel <= 1.01e-12
    assert float(np.linalg.norm(x - xs) / np.linalg.norm(xs)) <= TOL
    again, it2, _ = c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    assert it2 == it and np.array_equal(x, again)


@pytest.mark.parametrize("n", [168 * 32, 168 * 32 + 1])
def test_mixed_cluster_edge(gpu_lib, n):
    from openmps_gb300.computer import Computer

    ptr, col, val, b, xs, x0 = _system(n, (1, 2, 73, 74), seed=n)
    x, _, rel = Computer(abi.make_params()).cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS,
                                                         solver=abi.SOLVER_MIXED)
    assert rel <= 1.01e-12
    assert np.linalg.norm(x - xs) <= TOL * np.linalg.norm(xs)


# every way the allocation-free solve walks its rows, around the largest system one cluster
# takes (2,048 rows) and at the largest it accepts
NOALLOC = {
    "one_row": dict(n=1, offsets=()),
    "cluster_edge": dict(n=2048, offsets=(1, 2, 50, 51)),
    "cluster_past": dict(n=2049, offsets=(1, 2, 50, 51)),
    "eight_lanes": dict(n=5003, offsets=(1, 2, 70, 71, 72)),
    "four_lanes": dict(n=30001, offsets=(1, 2, 3, 170, 171, 172)),
    "four_by_four": dict(n=100_003, offsets=(1, 2, 3, 4, 315, 316, 317)),
    "four_by_four_wide": dict(n=80_000, offsets=tuple(range(1, 24))),
    "lane_per_row": dict(n=100_003, offsets=(1,)),
    "warp_per_row": dict(n=2001, offsets=tuple(range(1, 100))),
    "long_row": dict(n=700, offsets=(1, 2), dense_row=True),
    "identity_rows": dict(n=20_000, offsets=(1, 2, 3), identity=0.9),
    "largest": dict(n=abi.NOALLOC_MAX_ROWS, offsets=(1, 2, 512)),
}


@pytest.mark.parametrize("name", list(NOALLOC))
def test_noalloc_sizes(gpu_lib, name):
    import ctypes as C

    torch = pytest.importorskip("torch")
    ptr, col, val, b, xs, x0 = _system(seed=len(name), **NOALLOC[name])
    dev = [torch.from_numpy(a).cuda() for a in (ptr, col, val, b)]
    got = []
    for _ in range(2):
        x = torch.from_numpy(x0.copy()).cuda()
        it, rel = C.c_int32(), C.c_double()
        rc = gpu_lib.mps_cg_solve_csr_device_noalloc(len(b), *[a.data_ptr() for a in dev], x.data_ptr(), 1e-12,
                                                     abi.CRIT_RHS, 0, torch.cuda.current_stream().cuda_stream,
                                                     C.byref(it), C.byref(rel))
        assert rc == abi.MPS_OK
        got.append(x.cpu().numpy())
    err = float(np.linalg.norm(got[0] - xs) / np.linalg.norm(xs))
    print("%s: n %d, %d iterations, relres %.2e, error %.2e" % (name, len(b), it.value, rel.value, err))
    assert rel.value <= 1.01e-12
    assert err <= TOL
    assert np.array_equal(got[0], got[1])


# empty rows: an aligned chunk of them, and one at the end of a chunk of padding rows
EMPTY = {"last_row": (33, np.arange(32, 33)), "middle_chunk": (96, np.arange(32, 64)),
         "grid": (80 * 32 + 65, np.arange(3 * 32, 5 * 32))}


@pytest.mark.parametrize("solver", ["cg64", "mixed"])
@pytest.mark.parametrize("name", list(EMPTY))
def test_empty_rows(gpu_lib, name, solver):
    # 0 = b has no solution: the rows' residual stays in r.r whatever the rest does.  With
    # b = 0 there the system is solved, and x keeps its start in those rows.
    from openmps_gb300.computer import Computer, ComputerError

    n, empty = EMPTY[name]
    ptr, col, val, b, xs, x0 = _system(n, (1, 7), seed=n)
    gone = np.zeros(n, bool)
    gone[empty] = True
    row = np.repeat(np.arange(n), np.diff(ptr))
    keep = ~gone[row] & ~gone[col]
    ptr = np.concatenate([[0], np.cumsum(np.bincount(row[keep], minlength=n))]).astype(np.int64)
    col, val = col[keep], val[keep]
    b = np.bincount(row[keep], weights=val * xs[col], minlength=n)
    c = Computer(abi.make_params())
    which = abi.SOLVER_CG64 if solver == "cg64" else abi.SOLVER_MIXED
    x, _, rel = c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    assert rel <= 1.01e-12
    assert np.array_equal(x[empty], x0[empty])
    assert np.linalg.norm((x - xs)[~gone]) <= TOL * np.linalg.norm(xs)
    for size in (1e-3, 1.0):
        b[empty] = size
        with pytest.raises(ComputerError) as e:
            c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, max_iters=200, solver=which)
        assert e.value.code == abi.MPS_ERR_CG_NOT_CONVERGED


@pytest.mark.parametrize("solver", ["cg64", "mixed"])
def test_wait_runs_out(gpu_lib, solver):
    # a bound of 0 cycles: the blocks that arrive first leave the loop, and the call says so
    from openmps_gb300.computer import Computer, ComputerError

    ptr, col, val, b, xs, x0 = _system(20_000, (1, 2, 140, 141), seed=5)
    c = Computer(abi.make_params())
    which = abi.SOLVER_CG64 if solver == "cg64" else abi.SOLVER_MIXED
    c.set_wait_limits(barrier_clocks=0)
    with pytest.raises(ComputerError) as e:
        c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    assert e.value.code == abi.MPS_ERR_TIMEOUT
    c.set_wait_limits()
    x, _, rel = c.cg_solve_csr(ptr, col, val, b, x0, 1e-12, criterion=abi.CRIT_RHS, solver=which)
    assert rel <= 1.01e-12
    assert np.linalg.norm(x - xs) <= TOL * np.linalg.norm(xs)
