"""The neighbour walks of small scenes (eight lanes per particle) against the oracle.

Particle counts around a group of lanes and a block, lists of more than the 64 entries
screened at once, more pairs in range than the 48 cached weights, cells of more than 64
particles, and the terms switched off one by one.  Every comparison is bit for bit: the
walks keep the list order of each sum.
"""
import numpy as np
import pytest

from helpers import assert_same_neighbors, assert_same_particles, jittered_tank, make_pair
from openmps_gb300 import _abi as abi
from openmps_gb300 import scenes

pytestmark = pytest.mark.gpu


def _few(nx, nz):
    s = scenes.lattice(nx, nz, 0.01, (-0.2, -0.2, 0.4, 0.4))
    rng = np.random.default_rng(nx * 10 + nz)
    s.x += rng.uniform(-1e-3, 1e-3, s.count)
    s.z += rng.uniform(-1e-3, 1e-3, s.count)
    s.u += rng.uniform(-0.1, 0.1, s.count)
    s.w += rng.uniform(-0.1, 0.1, s.count)
    return s


CASES = {
    "one": (lambda: _few(1, 1), {}),
    "seven": (lambda: _few(7, 1), {}),
    "nine": (lambda: _few(3, 3), {}),
    "block": (lambda: _few(8, 8), {}),
    "wide": (lambda: _few(21, 19), dict(re_by_l0=4.0)),
    "widest": (lambda: _few(23, 22), dict(re_by_l0=7.5)),
    "tank": (lambda: jittered_tank(jitter=0.1), dict(re_by_l0=4.0)),
    "tank_wide": (lambda: jittered_tank(jitter=0.1), dict(re_by_l0=6.5)),
}


@pytest.mark.parametrize("drop", [0, abi.FLAG_HS, abi.FLAG_HL, abi.FLAG_ECS, abi.FLAG_SPP])
@pytest.mark.parametrize("name", list(CASES))
def test_walks_bit_for_bit(gpu_lib, oracle_lib, name, drop):
    make, kw = CASES[name]
    s = make()
    every = abi.FLAG_HS | abi.FLAG_HL | abi.FLAG_ECS | abi.FLAG_SPP
    gpu, cpu = make_pair(s, s.params(flags=every & ~drop, eps=1e-13, **kw))
    for h in (gpu, cpu):
        h.forward_time(1e-4)
    assert_same_neighbors(gpu, cpu, name)
    for a, b in zip(gpu.ppe()[:4], cpu.ppe()[:4]):  # the fifth is the solution by now
        np.testing.assert_array_equal(a, b)
    g, c = gpu.aux(), cpu.aux()
    np.testing.assert_array_equal(g["n_without_spp"], c["n_without_spp"])
    if not drop & abi.FLAG_ECS:
        np.testing.assert_array_equal(g["ecs"], c["ecs"])
    # the gradient from the same pressure
    P = cpu.particles()
    gpu.set_particles(P["type"], *[P[k] for k in ("x", "z", "u", "w", "p", "n")])
    gpu.set_aux(c["n_without_spp"], c["ecs"], c["ox"], c["oz"])
    for h in (gpu, cpu):
        h.stage("search_neighbor")
        h.stage("pressure_gradient")
    assert_same_particles(gpu, cpu, what=name)
