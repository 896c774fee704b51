"""The preconditioned solves' single-launch loop at the edges of its work split.

Scenes around the largest system one cluster takes (2,560 rows), with hierarchies whose
single-block levels start at level 1, 2 and deeper, columns of cells much taller and much
shorter than usual (coarse levels one cell high), and cells so full that a block's window overflows (u goes through
global memory).

Tolerance: a column of N particles under a free surface has a condition number of about
4 (2 N / pi)^2 <= 1.7 N^2, and the wider weights raise it by less than 4; both solves leave
|b - A p| <= 1e-10 |b|, so |p - p'| <= 2e-10 * 7 N^2 |p|.
"""
import numpy as np
import pytest

from openmps_gb300 import _abi as abi
from openmps_gb300 import scenes

pytestmark = pytest.mark.gpu

# l0, water w, h, tank w, h, radius
CASES = {
    "cluster": (1e-2, 0.2, 0.4, 0.8, 0.6, 2.1),
    "past_cluster": (7.5e-3, 0.2, 0.4, 0.8, 0.6, 2.1),
    "few_rows": (2e-2, 0.1, 0.06, 0.2, 0.2, 2.1),
    "grid": (4e-3, 0.2, 0.4, 0.8, 0.6, 2.1),
    "flat": (5e-3, 2.0, 0.03, 6.0, 0.06, 2.1),
    "film": (5e-3, 1.0, 0.015, 14.0, 0.02, 2.1),
    "tall": (5e-3, 0.06, 1.0, 0.1, 1.2, 2.1),
    "deep_bottom": (2e-3, 0.2, 0.2, 2.0, 0.8, 2.1),
    "full_cells": (2e-3, 0.1, 0.4, 0.12, 0.4, 6.0),
}


def _step(s, **kw):
    from openmps_gb300.computer import Computer

    c = Computer(s.params(criterion=abi.CRIT_RHS, eps=1e-10, **kw))
    c.add_scene(s)
    c.forward_time(0.02 * s.l0)
    return c.particles()["p"], c.stats()


@pytest.mark.parametrize("name", list(CASES))
def test_loop_matches_cg(gpu_lib, name):
    l0, ww, wh, tw, th, radius = CASES[name]
    s = scenes.dam_break(l0, ww, wh, tw, th)
    mg, st = _step(s, solver=abi.SOLVER_MIXED_MG, re_by_l0=radius)
    cg, _ = _step(s, solver=abi.SOLVER_CG64, re_by_l0=radius)
    err = float(np.linalg.norm(mg - cg) / np.linalg.norm(cg))
    n = wh / l0
    print("%s: %d particles, %d iterations, relres %.1e, error %.1e" %
          (name, s.count, st["cg_iterations"], st["cg_true_relres"], err))
    assert st["fallback"] == 0
    assert st["cg_true_relres"] <= 1e-10
    assert err <= 2e-10 * 7 * n * n
    again, st2 = _step(s, solver=abi.SOLVER_MIXED_MG, re_by_l0=radius)
    assert st2["cg_iterations"] == st["cg_iterations"]
    np.testing.assert_array_equal(mg, again)  # every sum has a fixed order


# around the largest scenes of one cluster (5,376 rows) and of half the SMs (12,288)
FORMS = {
    "cluster_5250": (5e-3, 0.2, 0.4, 0.8, 0.6, 4.0),
    "half_5961": (4.6e-3, 0.2, 0.4, 0.8, 0.6, 4.0),
    "half_10875": (3e-3, 0.06, 1.0, 0.1, 1.2, 4.0),
    "grid": (2.9e-3, 0.2, 0.4, 0.8, 0.6, 4.0),
}


@pytest.mark.parametrize("name", list(FORMS))
def test_forms_match_cg(gpu_lib, name):
    l0, ww, wh, tw, th, radius = FORMS[name]
    s = scenes.dam_break(l0, ww, wh, tw, th)
    mg, st = _step(s, solver=abi.SOLVER_MIXED_MG, re_by_l0=radius)
    cg, _ = _step(s, solver=abi.SOLVER_CG64, re_by_l0=radius)
    n = wh / l0
    print("%s: %d particles" % (name, s.count))
    assert st["fallback"] == 0 and st["cg_true_relres"] <= 1e-10
    assert float(np.linalg.norm(mg - cg) / np.linalg.norm(cg)) <= 2e-10 * 7 * n * n
    again, _ = _step(s, solver=abi.SOLVER_MIXED_MG, re_by_l0=radius)
    np.testing.assert_array_equal(mg, again)


def test_handles_at_once(gpu_lib):
    # four handles stepped from four threads end where one by itself does, in each form
    import threading

    from openmps_gb300.computer import Computer

    for l0 in (5e-3, 3.6e-3, 2.5e-3):
        s = scenes.dam_break(l0, 0.2, 0.4, 0.8, 0.6)
        cs = []
        for _ in range(5):
            c = Computer(s.params(criterion=abi.CRIT_RHS, eps=1e-10, solver=abi.SOLVER_MIXED_MG))
            c.add_scene(s)
            cs.append(c)

        def go(c):
            for _ in range(4):
                c.forward_time(0.01 * l0)

        go(cs[0])
        threads = [threading.Thread(target=go, args=(c,)) for c in cs[1:]]
        for t in threads:
            t.start()
        for t in threads:
            t.join()
        want = cs[0].particles()
        for c in cs[1:]:
            got = c.particles()
            for k in ("x", "z", "u", "w", "p"):
                np.testing.assert_array_equal(got[k], want[k], err_msg=k)
