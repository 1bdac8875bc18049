"""The double lane's sweep levels, dealt out in single warps, against the CPU
checker at the sizes where a warp ends: levels of 1, 31, 32, 33 and 65 bonds,
broken bonds among live ones, a box on the ground struck by a sphere, and a
batch against each of its lattices alone. Bit for bit.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu


def _chain(bonds, iterations=4, dead=0):
    """A chain alternates between two levels of half its bonds each."""
    from banjo_gb300 import scenes

    case = scenes.drop_trial(bonds + 1, 1, 1, compliance=1e-7, break_strain=1.5e-3, drop_height=0.002, steps=2)
    vel = case["vel"].reshape(-1, 3)
    vel[:, 1] = -3.0
    vel[::3, 0] = 0.5
    case["vel"] = vel.reshape(-1)
    case["settings"][scenes.K_ITER] = iterations
    if dead:
        alive = np.ones(int(case["bond_count"][0]), dtype=np.uint8)
        alive[::dead] = 0
        case["alive"] = alive
    return case


@pytest.mark.parametrize("bonds,iterations,dead", [(1, 4, 0), (62, 4, 0), (63, 1, 0), (64, 4, 5), (66, 4, 0),
                                                   (130, 2, 7)])
def test_level_sizes_match_checker(device, port, bonds, iterations, dead):
    case = _chain(bonds, iterations, dead)
    cpu = port.run_port(case, precision="double")
    gpu = device.run_case(case, precision="double")
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_struck_box_matches_checker(device, port):
    from banjo_gb300 import scenes

    case = scenes.impact_block(nx=16, ny=8, nz=12, blocks=3, radius=0.03, speed=12.0, steps=3)
    cpu = port.run_port(case, precision="double", threads=4)
    gpu = device.run_case(case, precision="double")
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_double_batch_equals_each_alone(device):
    cases = [_chain(b) for b in (1, 65, 130)]
    for case, out in zip(cases, device.run_batch(cases, precision="double")):
        alone = device.run_case(case, precision="double")
        assert mismatches(alone, out, STATE_KEYS) == []
        assert status_mismatches(alone, out) == []
