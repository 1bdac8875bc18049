"""Bonds that are degenerate (1e-12 m long or less) in some iterations of a sweep.

The projection leaves such a bond and its multiplier alone, and an iteration
that finds it longer goes on from the multiplier it has: the one of the same
substep, or, when the first iteration passed it by, the one the last substep
ended with. Cells of 2e-12 m whose bonds stretch and shorten across that
length, against the CPU checker bit for bit, by every form of the sweep.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu

OFF = 0xFFFFFFFF


def _minute(nx, ny, nz, seed=6, steps=20):
    from banjo_gb300 import scenes

    case = scenes.drop_trial(nx, ny, nz, compliance=1e-7, break_strain=1.5e-3, drop_height=0.002, h=2e-12, steps=2)
    vel = case["vel"].reshape(-1, 3).copy()
    vel[:, 1] = -1e-9
    case["vel"] = vel.reshape(-1)
    case["pos"] = case["pos"] + (np.random.default_rng(seed).random(case["pos"].size) - 0.5) * 3e-12
    # No bond breaks: they go on being solved.
    case["threshold"] = np.full_like(case["threshold"], np.inf)
    case["steps"] = np.array([steps], dtype=np.uint64)
    return case


def _checked(port, case, precision):
    from banjo_gb300 import scenes

    if precision == "double":
        case["settings"] = case["settings"].copy()
        case["settings"][scenes.K_DIRECT] = 1
    return port.run_port(case, precision=precision, threads=2)


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("shape", [(2, 1, 1), (9, 1, 1), (7, 5, 6), (12, 8, 8), (40, 8, 8)])
def test_lattice_matches_checker(device, port, shape, precision):
    case = _minute(*shape)
    cpu = _checked(port, case, precision)
    gpu = device.run_case(case, precision=precision)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("tuning", [None, "tune", {"whole_max_bonds": 1 << 20, "staged_max_nodes": OFF},
                                    {"whole_max_bonds": 1, "staged_max_nodes": OFF}],
                         ids=["default", "tune", "whole", "levels"])
def test_batch_matches_checker(device, port, tuning, precision):
    cases = [_minute(8, 6, 8), _minute(5, 5, 5, seed=7), _minute(9, 1, 1, seed=8)]
    outs = device.run_batch(cases, precision=precision, tuning=tuning)
    for case, out in zip(cases, outs):
        cpu = _checked(port, case, precision)
        assert mismatches(cpu, out, [k for k in STATE_KEYS if not k.startswith("source")]) == []


def test_tuned_between_runs(device):
    """Tuning times sweeps of the lattices present; their multipliers stay."""
    case = _minute(12, 8, 8)
    sched = device.build_lattice_schedule(int(case["node_count"][0]), case["bond_a"], case["bond_b"],
                                          case["node_block_begin"])
    results = []
    for tuned in (False, True):
        batch = device.Batch()
        states = [device.build_lattice_state(case, sched) for _ in range(2)]
        for state in states:
            batch.add(sched, state, device.sphere_state(case["sphere"]))
        batch.settle(device.step_settings(case["settings"]))
        batch.run(device.RunControl(max_steps=7))
        if tuned:
            batch.tune()
        batch.run(device.RunControl(max_steps=7))
        for k, state in enumerate(states):
            batch.download(k, state)
        results.append(states[0].u.copy())
    assert np.array_equal(*results)
