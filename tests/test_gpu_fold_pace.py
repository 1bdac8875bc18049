"""The warp's serial FP64 sum where it cannot go by runs, and where it changes over.

A sum that keeps crossing binades is the chain of adds, at the chain's speed;
one that does so for a while goes on as it should after. Loads on thousands of
nodes, several staged chunks, whose sums cancel, settle, cancel again and jump,
against the CPU checker bit for bit; wrench sources whose runs begin on odd
places of a chunk; and the time of a substep bound by such a sum.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu


def _forces(kind, n, rng):
    k = np.arange(n)[:, None]
    f = rng.uniform(-0.5, 0.5, (n, 3)) * 1e-3
    if kind == "alternating":
        f = 1e-3 * np.where(k % 2, 1.0, -1.0) * rng.uniform(0.999, 1.001, (n, 3))
    elif kind == "phases":  # cancelling, then of one sign, then cancelling about a large sum, then a jump
        f[n // 4:n // 2] = -np.abs(f[n // 4:n // 2])
        f[n // 2:3 * n // 4] *= 1e-6
        f[3 * n // 4] = 1e3
    elif kind == "late":  # nothing at all, then one term after another that outweighs those before it
        f[:2 * n // 3] = 0.0
        f[2 * n // 3:] *= 2.0 ** np.minimum((k[2 * n // 3:] - 2 * n // 3) // 64, 40)
    return f


@pytest.mark.parametrize("kind", ["any sign", "alternating", "phases", "late"])
@pytest.mark.parametrize("shape", [(3, 5, 5), (9, 9, 9), (24, 18, 21)])
def test_load_ledger_matches_checker(device, port, shape, kind):
    from banjo_gb300 import scenes

    case = scenes.cantilever(*shape, steps=1, substeps=5)
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


def test_wrench_sources_match_checker(device, port):
    """Nine sources of odd sizes over several chunks, and the total beside them."""
    from banjo_gb300 import scenes

    case = scenes.wrenched_bar(30, 9, 11, steps=4)
    n = int(case["node_count"][0])
    pos = case["ref_pos"].reshape(-1, 3)
    rng = np.random.default_rng(4)
    movable = np.flatnonzero(np.arange(n) % 30 > 0)
    cuts = [0, 61, 160, 333, 500, 901, 1700, 1801, 2500, movable.size - 3]
    regions = []
    for k, (lo, hi) in enumerate(zip(cuts[:-1], cuts[1:])):
        nodes = movable[lo:hi]
        torque = rng.uniform(-1e-3, 1e-3, 3) if nodes.size > 40 else np.zeros(3)
        regions.append((f"s{k}", nodes, pos[nodes].mean(axis=0), rng.uniform(-0.2, 0.2, 3), torque))
    case = scenes.wrenches(case, regions, 4)
    cpu = port.run_port(case, threads=4)
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS + ["source_names", "source_ledgers"]) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_a_sum_of_any_sign_costs_the_chain(device):
    """16,128 loaded nodes: a substep waits for its thirteen sums, 36 ns an add
    and term (73 cycles) when they are chains, 0.58 ms, and has about 40 us
    before and after them. A tenth more bounds it: 0.68 ms."""
    from banjo_gb300 import scenes

    case = scenes.cantilever(64, 16, 16)
    n = int(case["node_count"][0])
    f = np.random.default_rng(3).uniform(-0.5, 0.5, (n, 3)) * 1e-3
    f[case["pinned"] != 0] = 0.0
    sched = device.build_lattice_schedule(n, case["bond_a"], case["bond_b"], case["node_block_begin"])
    state = device.build_lattice_state(case, sched)
    backend = device.make_gb300_lattice_backend(sched)
    backend.upload(state, device.step_settings(case["settings"]), device.sphere_state(case["sphere"]))
    backend.set_external_forces(f.reshape(-1), 10_000)
    backend.run(device.RunControl(max_steps=4))
    times = []
    for _ in range(5):
        before = backend.status().kernel_seconds
        times.append((backend.run(device.RunControl(max_steps=20)).kernel_seconds - before) / 20 * 1e3)
    assert min(times) < 0.68
