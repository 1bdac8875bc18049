"""The pair gather's launch: at most 32 CTAs an SM, each over a run of owners.

The lists against the CPU checker where a CTA takes one owner a warp and where
it takes several, with a short last run, nodes that own no pairs (pinned) and
ones that own many, alone and in a batch; and the idle cost, where no rebuild
is due, on a lattice of many nodes.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu


def _loose(nodes, seed=3, rows=64):
    """Unbonded cells in a flat box, some of them nearer than the cutoff, every
    seventh one pinned: `nodes` owners, most without pairs."""
    from banjo_gb300 import scenes

    case = scenes.contact_drop(nx=2, ny=1, nz=1, drop_height=0.5, speed=0.0, steps=3, restitution=0.1)
    k = np.arange(nodes)
    ref = np.stack([k % rows, np.full(nodes, 60.0), k // rows], axis=1) * 0.013
    ref += (np.random.default_rng(seed).random((nodes, 3)) - 0.5) * 0.006
    case.update({
        "node_count": np.array([nodes], dtype=np.uint32), "bond_count": np.array([0], dtype=np.uint32),
        "ref_pos": ref.reshape(-1), "pos": ref.reshape(-1).copy(), "vel": np.zeros(3 * nodes),
        "mass": np.full(nodes, 1e-3), "bond_a": np.zeros(0, np.uint32), "bond_b": np.zeros(0, np.uint32),
        "rest_length": np.zeros(0), "compliance": np.zeros(0), "threshold": np.zeros(0),
        "node_block_begin": np.array([0, nodes], dtype=np.uint32),
        "pinned": (k % 7 == 0).astype(np.uint8)})
    case["settings"] = scenes.settings(node_contact=scenes.node_contact(2, 0.005, 0.0025, restitution=0.1,
                                                                        node_count=nodes))
    return case


# One run for each warp of at most 152 x 32 CTAs covers 38,912 owners; above, a CTA's run grows.
@pytest.mark.parametrize("nodes", [1, 9, 255, 257, 38_911, 38_913, 100_003])
def test_lists_match_checker(device, port, nodes):
    case = _loose(nodes)
    cpu = port.run_port(case, threads=2)
    gpu = device.run_case(case)
    if nodes > 1000:
        assert int(gpu["status_u64"][16]) > nodes // 20  # pairs listed
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []


def test_batch_equals_each_alone(device):
    cases = [_loose(n, seed=n) for n in (257, 38_913, 9, 5_000)]
    for c in cases[1:]:
        c["settings"] = cases[0]["settings"]
    for case, out in zip(cases, device.run_batch(cases)):
        alone = device.run_case(case)
        assert mismatches(alone, out, STATE_KEYS) == []
        assert status_mismatches(alone, out) == []


def test_idle_cost_of_many_nodes(device):
    """Without a rebuild the two launches cost what starting their CTAs does.
    At 1.05 ns a CTA (145,860 that return at once took 153 us), a CTA per eight
    owners would take 550 us for both at 2,097,152 nodes; the drift test, which
    reads 32 bytes a node, and seven other launches of at most one thread a node
    or bucket come to about 100. Half of that sum bounds the phase."""
    nodes = 1 << 21
    case = _loose(nodes, rows=1 << 10)
    case["ref_pos"] = (np.stack([np.arange(nodes) % 1024, np.full(nodes, 60), np.arange(nodes) // 1024], axis=1)
                       * 0.02).reshape(-1)
    case["pos"] = case["ref_pos"].copy()
    sched = device.build_lattice_schedule(nodes, case["bond_a"], case["bond_b"], case["node_block_begin"])
    state = device.build_lattice_state(case, sched)
    backend = device.make_gb300_lattice_backend(sched)
    settings = device.step_settings(case["settings"])
    settings.gravity[1] = 0.0
    backend.upload(state, settings, device.sphere_state(case["sphere"]))
    before = backend.run(device.RunControl(max_steps=2)).node_contact.rebuilds
    broad = min(backend.profile_phases(5)["node_contact_broad"] / 5 for _ in range(5))
    assert backend.run(device.RunControl(max_steps=1)).node_contact.rebuilds == before
    assert broad < 0.325
