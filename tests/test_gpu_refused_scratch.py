"""A sphere's candidate records that do not fit the device.

The records take 80 KB a slab in the float lane, so 2^22 slabs (nearly all of
them without a node) ask for 344 GB, more than the device has: the allocation
is refused. What was there before the refusal goes on as it was: a batch keeps
the settings it had, an admitted request does not enter, and later calls run.
"""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SLABS = 1 << 22
KEYS = ("u", "v", "alive", "damage", "prev_tensile")


def _case(sphere):
    from banjo_gb300 import scenes

    case = scenes.impact_block(nx=6, ny=5, nz=4, blocks=1, radius=0.02, speed=8.0, steps=2)
    if not sphere:
        case["settings"] = case["settings"].copy()
        case["settings"][scenes.K_SPHERE] = 0
    return case


def _built(device, case, slabs):
    n = int(case["node_count"][0])
    begin = np.full(slabs + 1, n, dtype=np.uint32)
    begin[0] = 0  # every node in the first slab
    sched = device.build_lattice_schedule(n, case["bond_a"], case["bond_b"], begin)
    return sched, device.build_lattice_state(case, sched)


def test_batch_keeps_its_settings_when_the_records_are_refused(device):
    free, impact = _case(sphere=False), _case(sphere=True)
    alone = device.run_case(dict(free, steps=np.array([8], dtype=np.uint64)))
    sched, state = _built(device, free, SLABS)
    batch = device.Batch()
    batch.add(sched, state, device.sphere_state(free["sphere"]))
    batch.settle(device.step_settings(free["settings"]))
    batch.run(device.RunControl(max_steps=3))
    for _ in range(2):
        with pytest.raises(RuntimeError, match="device allocation"):
            batch.settle(device.step_settings(impact["settings"]))
    batch.run(device.RunControl(max_steps=5))
    assert batch.status(0).total_steps == 8
    batch.download(0, state)
    for k in KEYS:
        assert np.array_equal(state.arrays[k], alone[k]), k


def test_refused_request_stays_queued_and_others_are_served(device):
    case = _case(sphere=True)
    alone = device.run_case(dict(case, steps=np.array([12], dtype=np.uint64)))
    sphere = device.sphere_state(case["sphere"])
    large, small = _built(device, case, SLABS), _built(device, case, 1)
    server = device.Server(device.step_settings(case["settings"]), 1 << 40)
    refused = server.submit(*large, sphere, 12)
    for _ in range(2):
        with pytest.raises(RuntimeError, match="device allocation"):
            server.step(4)
        assert server.poll(refused).phase == device.REQUEST_QUEUED
    server.cancel(refused)
    ticket = server.submit(*small, sphere, 12)
    while server.poll(ticket).phase != device.REQUEST_DONE:
        server.step(4)
    _, status = server.take(ticket, small[1])
    assert status.total_steps == 12
    for k in KEYS:
        assert np.array_equal(small[1].arrays[k], alone[k]), k
    stats = server.stats()
    assert stats.queued == 0 and stats.running == 0 and stats.bytes_in_use == 0
