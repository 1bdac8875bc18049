"""The staged sweep (a small lattice swept by one CTA from shared memory)
against the CPU checker, at the sizes where it begins and ends: a level of one
bond, one iteration, a widest level of exactly 1,024 bonds and the first one
above (level-launched), many levels of few bonds, with the ground, plastic flow
and a sphere, and broken bonds among live ones. Bit for bit.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu


def _drop(nx, ny, nz, iterations=4, dead=0, **kw):
    from banjo_gb300 import scenes

    case = scenes.drop_trial(nx, ny, nz, compliance=1e-7, break_strain=1.5e-3, drop_height=0.002, steps=2, **kw)
    vel = case["vel"].reshape(-1, 3)
    vel[:, 1] = -3.0
    case["vel"] = vel.reshape(-1)
    case["settings"][scenes.K_ITER] = iterations
    if dead:
        alive = np.ones(int(case["bond_count"][0]), dtype=np.uint8)
        alive[::dead] = 0
        case["alive"] = alive
    return case


def _cases():
    from banjo_gb300 import scenes

    return {
        "one bond": _drop(2, 1, 1),
        "chain": _drop(67, 1, 1),
        "one iteration": _drop(9, 4, 5, iterations=1),
        "odd": _drop(13, 7, 5, dead=7),
        "widest 1024": _drop(32, 8, 8),
        "widest 1056": _drop(33, 8, 8),
        "plastic impact": scenes.impact_block(nx=16, ny=8, nz=12, blocks=3, radius=0.03, speed=12.0, steps=3),
    }


@pytest.mark.parametrize("name", ["one bond", "chain", "one iteration", "odd", "widest 1024", "widest 1056",
                                  "plastic impact"])
def test_staged_sweep_matches_checker(device, port, name):
    case = _cases()[name]
    cpu = port.run_port(case, threads=4)
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_staged_batch_equals_each_alone(device):
    """Lattices of one to 1,024 bonds a level staged in one launch."""
    cases = [_cases()[k] for k in ("chain", "odd", "widest 1024", "one bond")]
    for case, out in zip(cases, device.run_batch(cases)):
        alone = device.run_case(case)
        assert mismatches(alone, out, STATE_KEYS) == []
        assert status_mismatches(alone, out) == []
