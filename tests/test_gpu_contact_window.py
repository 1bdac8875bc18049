"""The narrow phase's window of 32 pairs in registers against the CPU checker:
lists from a few pairs to thousands, fast boxes whose pairs share nodes within
and across windows, deep overlaps (position corrections), the measure mode, and
lattices of different list lengths in one batch. Bit for bit, accumulators
included.
"""
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu

SCENES = [dict(nx=2, ny=2, nz=2, speed=20.0, steps=12), dict(nx=4, ny=3, nz=5, speed=25.0, steps=16),
          dict(nx=7, ny=5, nz=6, speed=15.0, steps=20), dict(nx=12, ny=8, nz=11, speed=30.0, steps=24),
          dict(nx=12, ny=8, nz=11, speed=30.0, steps=12, mode=1)]


@pytest.mark.parametrize("kw", SCENES, ids=lambda k: "x".join(str(k[d]) for d in ("nx", "ny", "nz")) + f"m{k.get('mode', 2)}")
@pytest.mark.parametrize("precision", ["float", "double"])
def test_windows_match_checker(device, port, kw, precision):
    from banjo_gb300 import scenes

    case = scenes.contact_drop(**kw)
    if precision == "double":
        case["settings"] = case["settings"].copy()
        case["settings"][scenes.K_DIRECT] = 1
    cpu = port.run_port(case, precision=precision, threads=2)
    gpu = device.run_case(case, precision=precision)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_batch_equals_each_alone(device):
    from banjo_gb300 import scenes

    cases = [scenes.contact_drop(**dict(kw, steps=16)) for kw in SCENES[:4]]
    for case in cases[1:]:
        case["settings"] = cases[0]["settings"]
    for case, out in zip(cases, device.run_batch(cases)):
        alone = device.run_case(case)
        assert mismatches(alone, out, STATE_KEYS) == []
        assert status_mismatches(alone, out) == []
