"""The end sample of one lattice, whose CTAs take the tiles of 256 bonds in
stripes, and of its contact halo, whose CTAs each look at several tiles, against
the CPU checker at the sizes where either could go wrong: a single tile, fewer
tiles than levels, a stripe more or less, levels of very different widths, and a
halo of many tiles in a lattice with more tiles than CTAs of one launch round.
Bit for bit.
"""
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu


def _drop(nx, ny, nz):
    from banjo_gb300 import scenes

    case = scenes.drop_trial(nx, ny, nz, compliance=1e-7, break_strain=1.5e-3, drop_height=0.002, steps=2)
    vel = case["vel"].reshape(-1, 3)
    vel[:, 1] = -3.0
    case["vel"] = vel.reshape(-1)
    return case


@pytest.mark.parametrize("size", [(2, 1, 1), (6, 4, 3), (9, 5, 3), (13, 12, 11), (40, 2, 1), (24, 20, 22)])
def test_striped_tiles_match_checker(device, port, size):
    case = _drop(*size)
    cpu = port.run_port(case, threads=4)
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


@pytest.mark.parametrize("size,blocks,radius", [((8, 4, 8), 2, 0.02), ((56, 40, 56), 4, 0.3)])
def test_halo_tiles_match_checker(device, port, size, blocks, radius):
    from banjo_gb300 import scenes

    nx, ny, nz = size
    case = scenes.impact_block(nx=nx, ny=ny, nz=nz, blocks=blocks, radius=radius, speed=12.0, steps=2)
    cpu = port.run_port(case, threads=8)
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []
