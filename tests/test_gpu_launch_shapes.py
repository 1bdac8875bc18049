"""Every launch shape of a batch's sweep gives the level-launched sweep's results.

The staged sweep is on by default and takes any batch of small lattices, so
each shape here says what it turns off: lattices swept whole by one CTA of
256, 512 or 1,024 threads, some whole beside others level-launched, several
groups of level launches, and the staged sweep itself. Each is told apart by
its number of kernels a substep and held bit for bit to level launches in one
group, which are held to the CPU checker.
"""
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu

OFF = 0xFFFFFFFF
LEVELS = {"whole_max_bonds": 1, "staged_max_nodes": OFF}


def _drops():
    from banjo_gb300 import scenes

    shapes = [(8, 6, 8), (12, 5, 9), (6, 6, 6), (10, 7, 5), (3, 4, 4)]
    cases = []
    for k, shape in enumerate(shapes):
        case = scenes.drop_trial(*shape, compliance=10.0 ** (-7 + 0.5 * k), break_strain=1.0e-3 + 5e-4 * k,
                                 drop_height=0.002, steps=3)
        vel = case["vel"].reshape(-1, 3)
        vel[:, 1] = -4.0
        case["vel"] = vel.reshape(-1)
        cases.append(case)
    return cases


def _impacts():
    from banjo_gb300 import scenes

    kw = dict(radius=0.03, speed=12.0, steps=3)
    cases = [scenes.impact_block(nx=14, ny=8, nz=10, blocks=3, **kw),
             scenes.impact_block(nx=10, ny=8, nz=14, blocks=2, seed_point=5, seed_strength=9, **kw),
             scenes.impact_block(nx=12, ny=8, nz=6, blocks=1, seed_point=7, seed_strength=4, **kw)]
    # (The plane of a block of eight layers is the same for all of them.)
    for c in cases[1:]:
        c["settings"] = cases[0]["settings"]
    return cases


# Scene, substeps, and a reach that takes some of its lattices.
SCENES = {"drops": (_drops, 60, 2000), "plastic impacts": (_impacts, 30, 5000)}
SHAPES = {
    "whole 256": {"sweep_threads": 256, "whole_max_bonds": 1 << 24, "staged_max_nodes": OFF},
    "whole 512": {"sweep_threads": 512, "whole_max_bonds": 1 << 24, "staged_max_nodes": OFF},
    "whole 1024": {"sweep_threads": 1024, "whole_max_bonds": 1 << 24, "staged_max_nodes": OFF},
    "some whole": {"sweep_threads": 1024, "whole_max_bonds": None, "staged_max_nodes": OFF},
    "groups": {"whole_max_bonds": 1, "group_bytes": 1 << 12, "staged_max_nodes": OFF},
    "some whole, groups": {"sweep_threads": 256, "whole_max_bonds": None, "group_bytes": 1 << 12,
                           "staged_max_nodes": OFF},
    "staged": {"whole_max_bonds": 1 << 24, "group_bytes": 1 << 12, "staged_max_nodes": 14336},
}


def _run(device, cases, precision, shape, steps):
    batch = device.Batch(precision)
    states = []
    for c in cases:
        sched = device.build_lattice_schedule(int(c["node_count"][0]), c["bond_a"], c["bond_b"], c["node_block_begin"])
        state = device.build_lattice_state(c, sched)
        batch.add(sched, state, device.sphere_state(c["sphere"]))
        states.append(state)
    settings = device.step_settings(cases[0]["settings"])
    settings.direct_arithmetic = 1 if precision == "double" else 0
    batch.settle(settings)
    batch.set_tuning(**shape)
    kernels = batch.kernels_per_substep()
    batch.run(device.RunControl(max_steps=steps))
    outs = []
    for k, state in enumerate(states):
        sp = batch.download(k, state)
        outs.append(device.state_outputs(state, sp, batch.first_failure_bonds(k), batch.status(k)))
    return outs, kernels


@pytest.fixture(scope="module")
def level_launched(device):
    kept = {}

    def get(scene, precision):
        if (scene, precision) not in kept:
            make, steps, _ = SCENES[scene]
            kept[scene, precision] = _run(device, make(), precision, LEVELS, steps)
        return kept[scene, precision]

    return get


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("scene", list(SCENES))
@pytest.mark.parametrize("name", list(SHAPES))
def test_shape_equals_level_launches(device, level_launched, name, scene, precision):
    make, steps, some = SCENES[scene]
    base, levels = level_launched(scene, precision)
    shape = dict(SHAPES[name])
    shape["whole_max_bonds"] = shape["whole_max_bonds"] or some
    outs, kernels = _run(device, make(), precision, shape, steps)
    if name.startswith("whole") or name == "staged":
        assert kernels < levels - 20  # one launch for the sweep (by staged lattices, in the float lane)
    elif name.endswith("groups"):
        assert kernels > levels + 20  # a sweep for each group
    else:
        assert kernels == levels + 1  # the larger lattices' levels, and the others' one launch
    assert any(int(o["status_u64"][4]) > 0 for o in base)  # bonds broke
    for want, got in zip(base, outs):
        assert mismatches(want, got, STATE_KEYS) == []
        assert status_mismatches(want, got) == []


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("scene", list(SCENES))
def test_level_launches_match_checker(level_launched, port, scene, precision):
    import numpy as np

    make, steps, _ = SCENES[scene]
    base, _ = level_launched(scene, precision)
    for case, out in zip(make(), base):
        case["settings"] = case["settings"].copy()
        if precision == "double":
            from banjo_gb300 import scenes

            case["settings"][scenes.K_DIRECT] = 1
        cpu = port.run_port(dict(case, steps=np.array([steps], dtype=np.uint64)), precision=precision, threads=2)
        assert mismatches(cpu, out, [k for k in STATE_KEYS if not k.startswith("source")]) == []
        assert status_mismatches(cpu, out, ledger_rtol=LEDGER_RTOL) == []
