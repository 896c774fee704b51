"""The 3D step's shared neighbour walks against its stage kernels."""
import numpy as np
import pytest

from openmps_gb300 import _abi as abi
from openmps_gb300.computer import Computer
from test_gpu_dim3 import _scene

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("drop", [0, abi.FLAG_HS, abi.FLAG_HL, abi.FLAG_ECS, abi.FLAG_SPP, abi.FLAG_DS])
@pytest.mark.parametrize("re_lap", [0.0, 1.7])
def test_shared_walks_equal_the_stages(gpu_lib, drop, re_lap):
    # the step's walks (density + ECS + explicit, density + assembly) against the stage
    # kernels, bit for bit: the same solver on the same matrix between them
    s = _scene(flags=abi.PRESET_REFERENCE & ~drop, re_lap=re_lap, jitter=0.1)
    a, b = (Computer(s.params()) for _ in range(2))
    for h in (a, b):
        h.add_scene(s)
    flags = s.params().flags
    dt = 1e-4
    for _ in range(2):
        a.forward_time(dt)
        b.begin_step(dt)
        for name, on in (("search_neighbor", True), ("density", True), ("error_correction", flags & abi.FLAG_ECS),
                         ("explicit", True), ("density", True), ("save_x", flags & abi.FLAG_DS), ("set_ppe", True),
                         ("solve_ppe", True), ("assign_pressure", True), ("pressure_gradient", True),
                         ("dynamic_stabilize", flags & abi.FLAG_DS)):
            if on:
                b.stage(name)
    P, Q = a.particles3(), b.particles3()
    for k in P:
        np.testing.assert_array_equal(P[k], Q[k], err_msg=k)
