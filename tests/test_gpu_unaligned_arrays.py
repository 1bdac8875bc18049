"""Caller's arrays that start on no multiple of their element.

The device reads and writes whole elements, a host copy any bytes: such an
array is copied, and gives what an aligned one does, byte for byte. Every
array of doubles is shifted alone, by each number of bytes that leaves it
unaligned in a different way, and then all of them together.
"""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

OUT_DOUBLES = ("u", "u_prev", "v", "damage", "prev_tensile", "prev_compressive", "prev_shear", "plastic_extension",
               "plastic_strain")
OUT_BYTES = ("alive", "failure_mode")
IN_DOUBLES = ("x0", "u", "u_prev", "v", "inv_mass", "mass", "nbr_rest", "nbr_weight", "rest_edge", "rest_length",
              "rest_length_sq_minus", "compliance", "threshold", "damage", "prev_tensile", "prev_compressive",
              "prev_shear", "plastic_extension", "plastic_strain")
IN_INDICES = ("nbr_bond", "nbr_other", "bond_slot_a", "bond_slot_b", "bond_a", "bond_b")


def _shifted(array, by):
    """The same values in memory that starts `by` bytes past a multiple of 64."""
    raw = np.zeros(array.nbytes + 128, dtype=np.uint8)
    at = (-raw.ctypes.data) % 64 + by
    part = raw[at:at + array.nbytes]
    part[:] = np.ascontiguousarray(array).view(np.uint8).reshape(-1)
    return raw, part


def _view(device, state, shifts):
    """A copy of the state's view with the named arrays shifted; what is held, and the arrays' bytes."""
    view = device.StateView()
    C.memmove(C.byref(view), C.byref(state.view), C.sizeof(view))
    types = dict(device._STATE_ARRAYS)
    held, parts = [], {}
    for name, by in shifts.items():
        raw, part = _shifted(state.arrays[name], by)
        held.append(raw)
        parts[name] = part
        setattr(view, name, C.cast(part.ctypes.data, types[name]))
    return view, held, parts


def _scene(device):
    from banjo_gb300 import scenes

    case = scenes.impact_block(nx=13, ny=7, nz=11, blocks=3, radius=0.03, speed=12.0, steps=3)
    n = int(case["node_count"][0])
    sched = device.build_lattice_schedule(n, case["bond_a"], case["bond_b"], case["node_block_begin"])
    return case, sched, device.build_lattice_state(case, sched)


@pytest.mark.parametrize("precision", ["float", "double"])
def test_download_into_unaligned_arrays(device, precision):
    case, sched, state = _scene(device)
    settings = device.step_settings(case["settings"])
    settings.direct_arithmetic = 1 if precision == "double" else 0
    backend = device.make_gb300_lattice_backend(sched, precision)
    backend.upload(state, settings, device.sphere_state(case["sphere"]))
    backend.run(device.RunControl(max_steps=30))
    backend.download(state)
    assert np.any(state.alive == 0) and np.any(state.plastic_strain != 0)
    expected = {k: state.arrays[k].copy() for k in OUT_DOUBLES + OUT_BYTES}
    shifts = [{name: by} for name in OUT_DOUBLES for by in (1, 4)]
    shifts += [{name: by for name in OUT_DOUBLES + OUT_BYTES} for by in (1, 2, 4, 7)]
    for some in shifts:
        for k in expected:
            state.arrays[k][:] = 0
        view, held, parts = _view(device, state, {k: some.get(k, 0) for k in expected})
        for part in parts.values():
            part[:] = 0xA5
        device._call(device.library().gbl_download, backend._h, C.byref(view), None)
        for k, want in expected.items():
            assert np.array_equal(parts[k], want.view(np.uint8).reshape(-1)), (k, some)
        for raw, (k, part) in zip(held, parts.items()):  # and nothing around it
            at = part.ctypes.data - raw.ctypes.data
            assert not raw[:at].any() and not raw[at + part.size:].any(), (k, some)


def test_upload_from_unaligned_arrays(device):
    case, sched, state = _scene(device)
    settings, sphere = device.step_settings(case["settings"]), device.sphere_state(case["sphere"])
    backend = device.make_gb300_lattice_backend(sched)

    def result(view):
        device._call(device.library().gbl_upload, backend._h, C.byref(view), C.byref(settings), C.byref(sphere))
        backend.run(device.RunControl(max_steps=12))
        out = device.build_lattice_state(case, sched)
        backend.download(out)
        return {k: out.arrays[k].copy() for k in OUT_DOUBLES + OUT_BYTES}

    expected = result(state.view)
    assert np.any(expected["u"] != 0)
    shifts = [{name: 4} for name in IN_DOUBLES] + [{name: 2} for name in IN_INDICES]
    shifts += [{name: by for name in IN_DOUBLES + IN_INDICES + OUT_BYTES + ("nbr_alive",)} for by in (1, 6)]
    for some in shifts:
        view, held, _ = _view(device, state, some)
        got = result(view)
        for k, want in expected.items():
            assert np.array_equal(got[k].view(np.uint8), want.view(np.uint8)), (k, some)
