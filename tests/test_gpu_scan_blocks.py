"""The event scan where a lattice goes from one scan block of tiles to two.

A tile is 256 bonds and a block 1,024 tiles; up to 1,023 tiles (261,888 bonds)
the block's own scan is the whole of it, from there on a second launch follows.
Bond counts on both sides of 1,023, 1,024 and 1,025 tiles, with breaks in the
last tile, against the CPU checker; and all of them in one batch against each
alone.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu

TILE = 256
COUNTS = [1023 * TILE - 1, 1023 * TILE, 1023 * TILE + 1, 1024 * TILE, 1024 * TILE + 1, 1025 * TILE]


def _box(bonds):
    """A box thrown on the ground, its last bonds cut down to `bonds` and the
    very last ones near failure."""
    from banjo_gb300 import scenes

    case = scenes.drop_trial(34, 30, 32, compliance=1e-7, break_strain=1.5e-3, drop_height=0.0002, steps=1)
    total = int(case["bond_count"][0])
    assert total > bonds
    for k in ("bond_a", "bond_b", "rest_length", "compliance"):
        case[k] = case[k][:bonds].copy()
    thr = case["threshold"].reshape(-1, 6)[:bonds].copy()
    thr[-300:, :2] = 1e-9
    case["threshold"] = thr.reshape(-1)
    case["bond_count"] = np.array([bonds], dtype=np.uint32)
    vel = case["vel"].reshape(-1, 3)
    vel[:, 1] = -5.0
    vel[::5, 0] = 0.2
    case["vel"] = vel.reshape(-1)
    return case


@pytest.mark.parametrize("bonds", COUNTS)
def test_bond_counts_match_checker(device, port, bonds):
    case = _box(bonds)
    cpu = port.run_port(case, threads=8)
    assert int(cpu["status_u64"][4]) > 1000 and not cpu["alive"][-TILE:].all()
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_batch_equals_each_alone(device):
    cases = [_box(b) for b in COUNTS[::2]] + [_box(5 * TILE)]
    for case, out in zip(cases, device.run_batch(cases)):
        alone = device.run_case(case)
        assert mismatches(alone, out, STATE_KEYS) == []
        assert status_mismatches(alone, out) == []
