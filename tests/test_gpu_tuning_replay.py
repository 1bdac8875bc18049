"""What tune reports, set_tuning reproduces, whatever the shape before it.

The number of kernels of a substep tells the shapes apart: a staged or
one-CTA sweep is one launch, a level-launched one as many as levels times
iterations.
"""
import pytest

pytestmark = pytest.mark.gpu

SHAPE = ("sweep_threads", "whole_max_bonds", "group_bytes", "staged_max_nodes")
OFF = 0xFFFFFFFF


def _batch(device, cases, precision):
    batch = device.Batch(precision)
    for c in cases:
        sched = device.build_lattice_schedule(int(c["node_count"][0]), c["bond_a"], c["bond_b"], c["node_block_begin"])
        batch.add(sched, device.build_lattice_state(c, sched), device.sphere_state(c["sphere"]))
    settings = device.step_settings(cases[0]["settings"])
    settings.direct_arithmetic = 1 if precision == "double" else 0
    batch.settle(settings)
    return batch


def _trials(*shapes):
    from banjo_gb300 import scenes

    return [scenes.drop_trial(*s, compliance=1e-7, break_strain=2e-3, drop_height=0.01, steps=2) for s in shapes]


@pytest.mark.parametrize("precision", ["float", "double"])
@pytest.mark.parametrize("shapes", [((28, 24, 26), (25, 24, 20)), ((8, 6, 8), (12, 5, 9), (6, 6, 6))],
                         ids=["wide levels", "staged"])
def test_a_tuned_shape_is_reproduced(device, shapes, precision):
    cases = _trials(*shapes)
    tuned = _batch(device, cases, precision)
    chosen = tuned.tune()
    shape = {k: chosen[k] for k in SHAPE}
    assert all(shape.values())  # a zero would keep what the other batch has
    expected = tuned.kernels_per_substep()
    for before in ({}, {"sweep_threads": 256, "whole_max_bonds": 1 << 24, "staged_max_nodes": OFF},
                   {"whole_max_bonds": 1, "group_bytes": 1 << 12, "staged_max_nodes": 14336}):
        other = _batch(device, cases, precision)
        if before:
            other.set_tuning(**before)
        other.set_tuning(**shape)
        assert other.kernels_per_substep() == expected, before


def test_none_swept_whole_is_level_launched(device):
    cases = _trials((8, 6, 8), (2, 1, 1))
    level = _batch(device, cases, "float")
    level.set_tuning(staged_max_nodes=OFF)
    again = _batch(device, cases, "float")
    again.set_tuning(whole_max_bonds=1 << 20, staged_max_nodes=OFF)
    whole = again.kernels_per_substep()
    again.set_tuning(whole_max_bonds=1)
    assert again.kernels_per_substep() == level.kernels_per_substep() > whole


def test_refused_shapes_stay_refused(device):
    batch = _batch(device, _trials((6, 6, 6), (5, 4, 5)), "float")
    for bad in ({"whole_max_bonds": (1 << 24) + 1}, {"whole_max_bonds": OFF}, {"staged_max_nodes": 14337},
                {"sweep_threads": 128}):
        with pytest.raises(ValueError):
            batch.set_tuning(**bad)
