"""The warp's serial FP64 sum (foldSerial) against the CPU checker's loop, bit
for bit, through the external-load ledger and the wrench sources' ledgers.

The loads make the running sums do what the fold treats apart: stay in one
binade for hundreds of terms, grow through many, cancel back towards zero term
after term, meet terms far larger and far smaller than themselves, exact zeros
and halves of an ulp (powers of two of mixed size), with list lengths around a
lane's share, a run, a staged chunk and several chunks.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu

SHAPES = {"few": (4, 2, 2), "one run": (17, 4, 4), "past a chunk": (14, 8, 8), "chunks": (24, 11, 9)}


def _forces(kind, n, rng):
    f = np.zeros((n, 3))
    if kind == "one sign":
        f[:] = -9.81e-3 * rng.uniform(0.5, 1.5, (n, 3))
    elif kind == "mixed":
        f[:] = rng.choice([-1.0, 1.0], (n, 3)) * 10.0 ** rng.uniform(-9, 1, (n, 3))
    elif kind == "cancelling":
        f[:] = 1e-2 * np.where(np.arange(n)[:, None] % 2, 1.0, -1.0) * (1.0 + 1e-6 * rng.standard_normal((n, 3)))
    else:  # powers of two: halves of ulps, exact zeros
        f[:] = rng.choice([-1.0, 0.0, 1.0], (n, 3)) * 2.0 ** rng.integers(-30, 1, (n, 3))
        f[::3] = 0.0
    return f


@pytest.mark.parametrize("kind", ["one sign", "mixed", "cancelling", "powers of two"])
@pytest.mark.parametrize("shape", list(SHAPES))
def test_load_ledger_matches_checker(device, port, shape, kind):
    from banjo_gb300 import scenes

    case = scenes.cantilever(*SHAPES[shape], steps=1, substeps=6)
    n = int(case["node_count"][0])
    f = _forces(kind, n, np.random.default_rng(n))
    f[case["pinned"] != 0] = 0.0
    case["forces"] = f.reshape(-1)
    cpu = port.run_port(case, threads=4)
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []
    for k in range(14, 18):  # work and impulse of the external load: serial sums, no tolerance
        assert cpu["status_f64"][k] == gpu["status_f64"][k], k


@pytest.mark.parametrize("shape", ["one run", "past a chunk", "chunks"])
def test_wrench_sources_match_checker(device, port, shape):
    """Sources whose node runs begin and end anywhere in a run or a chunk."""
    from banjo_gb300 import scenes

    nx, ny, nz = SHAPES[shape]
    case = scenes.wrenched_bar(nx, ny, nz, steps=4)
    i = np.arange(nx * ny * nz)
    pos = case["ref_pos"].reshape(-1, 3)
    x = i % nx
    rng = np.random.default_rng(3)
    regions = []
    for k, (lo, hi) in enumerate([(1, 2), (2, 3), (3, nx // 2), (nx // 2, nx)]):
        nodes = np.flatnonzero((x >= lo) & (x < hi))
        regions.append((f"s{k}", nodes, pos[nodes].mean(axis=0), rng.uniform(-0.2, 0.2, 3), rng.uniform(-1e-3, 1e-3, 3)))
    case = scenes.wrenches(case, regions, 4)
    cpu = port.run_port(case, threads=4)
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS + ["source_names", "source_ledgers"]) == []
