"""Work lists are for several lattices: one lattice's launches count their items off.

What a settled lattice's first substep prepares is then its graph, whose size
depends on the number of levels and not on the lattice's: a 64-times larger
one (same levels, one slab) is prepared in the same time. With lists, an item
is written and copied for every 32 bonds of the double lane's sweep and every
256 of the rest, about 3 ns each: 1.1 ms for this lattice in the double lane
and 0.2 in the float lane.
"""
import time

import pytest

pytestmark = pytest.mark.gpu


def _prepare_ms(device, shape, precision):
    from banjo_gb300 import scenes

    case = scenes.drop_trial(*shape, compliance=1e-7, break_strain=2e-3, drop_height=0.5)
    n = int(case["node_count"][0])
    sched = device.build_lattice_schedule(n, case["bond_a"], case["bond_b"], case["node_block_begin"])
    state = device.build_lattice_state(case, sched)
    batch = device.Batch(precision)
    batch.add(sched, state, device.sphere_state(case["sphere"]))
    settings = device.step_settings(case["settings"])
    settings.direct_arithmetic = 1 if precision == "double" else 0
    times = []
    for _ in range(15):
        batch.settle(settings)
        t = time.perf_counter()
        kernels = batch.kernels_per_substep()
        times.append((time.perf_counter() - t) * 1e3)
    return min(times), kernels


@pytest.mark.parametrize("precision", ["float", "double"])
def test_one_lattice_prepares_no_list(device, precision):
    small, a = _prepare_ms(device, (33, 32, 16), precision)  # its widest level is past the staged sweep's
    large, b = _prepare_ms(device, (132, 128, 64), precision)
    assert abs(a - b) <= 2
    assert large - small < 0.1
