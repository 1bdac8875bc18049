"""A request's candidate records come from the device's memory pool.

The records of 2,048 slabs are 168 MB in the float lane. Freed through the
pool they stay there for the next request; a free outside it would give them
back to the device, and would wait for everything that runs on it (the other
lane's lattices among it) to do so.
"""
import ctypes

import numpy as np
import pytest

from test_zz_no_alloc import _cudart

pytestmark = pytest.mark.gpu

SLABS = 2048


def _free_bytes():
    free, total = ctypes.c_size_t(), ctypes.c_size_t()
    assert _cudart().cudaMemGetInfo(ctypes.byref(free), ctypes.byref(total)) == 0
    return free.value


def test_a_retired_requests_records_stay_in_the_pool(device):
    from banjo_gb300 import scenes

    case = scenes.impact_block(nx=6, ny=5, nz=4, blocks=1, radius=0.02, speed=8.0, steps=2)
    n = int(case["node_count"][0])
    begin = np.full(SLABS + 1, n, dtype=np.uint32)
    begin[0] = 0
    sched = device.build_lattice_schedule(n, case["bond_a"], case["bond_b"], begin)
    state = device.build_lattice_state(case, sched)
    server = device.Server(device.step_settings(case["settings"]), 1 << 34)
    ticket = server.submit(sched, state, device.sphere_state(case["sphere"]), 8)
    server.step(4)
    assert server.poll(ticket).phase == device.REQUEST_RUNNING
    running = _free_bytes()
    server.step(4)
    assert server.poll(ticket).phase == device.REQUEST_DONE
    assert _free_bytes() - running < 84 << 20  # half of the records
    server.take(ticket, state)
