"""The timed workloads of the lattice substep, each through the public API.

A case is one thing a user of the framework has it do, at one size:

  beam    a pinned beam under its own weight as an external load, one frame of
          substeps and a read-back: the interactive call, where launches count
  wrench  a pinned bar gripped by two named wrenches, one frame and a read-back
  plate   a sheet one cell thick on two ledges, struck by a sphere, with plate
          bending: a window or tile being broken
  crack   a box thrown on the ground whose cracked faces meet again
          (node-to-node contact on)
  impact  a block on the ground struck by a rigid sphere, with per-bond
          strengths and plastic flow: the framework's headline scene, in the
          float lane and in the double lane
  bar     a notched bar under a ramped end load (horizon 2, plastic flow), the
          load set anew every step: the long-horizon tensile test
  trial   one box from a caller's arrays to its result: upload, run, download
  batch   independent drop trials of uneven sizes advanced together
  serve   requests through the server: submit, step until done, take

`beam`, `wrench`, `plate`, `crack`, `impact`, `bar` and `batch` go on from where
the last pass left off, as a simulation does; `trial` and `serve` start afresh
every pass. Sizes are those of the benchmark's configurations and of the tests,
and odd ones around them.
"""
from __future__ import annotations

import concurrent.futures
import ctypes
import functools
import math
import os

import numpy as np

from banjo_gb300 import lattice, scenes

H = 0.01  # cell edge, m
DT = scenes.DT_SUBSTEP
GRAVITY = -9.81
ITERATIONS = 4
INF = float("inf")

# What a download writes (include/gbl.h, gbl_state_view): values per node or per bond.
NODE_ARRAYS = {"u": 3, "u_prev": 3, "v": 3}
BOND_ARRAYS = {"alive": np.uint8, "failure_mode": np.uint8, "damage": np.float64, "prev_tensile": np.float64,
               "prev_compressive": np.float64, "prev_shear": np.float64, "plastic_extension": np.float64,
               "plastic_strain": np.float64}


def listed():
    return [
        # The smallest interactive scene: a stub of a beam, a frame at a time.
        {"name": "beam 9x5x3", "kind": "beam", "nx": 9, "ny": 5, "nz": 3, "substeps": 10},
        # The cantilever configuration: 240 frames a second, one frame a pass.
        {"name": "beam 32x8x8", "kind": "beam", "nx": 32, "ny": 8, "nz": 8, "substeps": 10},
        # A driven part: two grips re-spread from the moving geometry every substep.
        {"name": "wrench 24x9x9", "kind": "wrench", "nx": 24, "ny": 9, "nz": 9, "substeps": 10},
        # A tile under a ball, two frames.
        {"name": "plate 64x1x48", "kind": "plate", "nx": 64, "ny": 1, "nz": 48, "substeps": 20},
        # The cracking box of the node-contact tests.
        {"name": "crack 24x10x18", "kind": "crack", "nx": 24, "ny": 10, "nz": 18, "substeps": 20},
        # One trial of the batch configuration's mean size, alone, start to end.
        {"name": "trial 28x28x28", "kind": "trial", "nx": 28, "ny": 28, "nz": 28, "substeps": 240},
        # The double lane, as a user checks a float run with it.
        {"name": "impact 48x24x40 double", "kind": "impact", "nx": 48, "ny": 24, "nz": 40, "slabs": 5,
         "precision": "double", "substeps": 10},
        # The impact scene at the size that fits a tile of a larger scene.
        {"name": "impact 128x64x64", "kind": "impact", "nx": 128, "ny": 64, "nz": 64, "slabs": 32,
         "precision": "float", "substeps": 10},
        # The headline impact, two frames and a read-back.
        {"name": "impact 256x128x128", "kind": "impact", "nx": 256, "ny": 128, "nz": 128, "slabs": 32,
         "precision": "float", "substeps": 20},
        # The notched bar of the precision check, four steps of its ramp.
        {"name": "bar 128x32x32", "kind": "bar", "nx": 128, "ny": 32, "nz": 32, "steps": 4, "substeps": 10},
        # A slice of the batch configuration: edges 8..48 a side.
        {"name": "batch 128 of 8..48", "kind": "batch", "count": 128, "lo": 8, "hi": 48, "substeps": 120},
        # Requests of the served configuration, with one large lattice among them.
        {"name": "serve 12 of 8..48", "kind": "serve", "count": 12, "lo": 8, "hi": 48, "large": 80, "substeps": 40},
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["beam", "beam", "wrench", "plate", "crack", "impact", "impact", "bar", "trial", "batch",
                       "serve"])
    frame = rng.choice([4, 10, 20])
    if kind == "beam":
        return {"kind": kind, "nx": _log_int(rng, 6, 64), "ny": _log_int(rng, 3, 16), "nz": _log_int(rng, 3, 16),
                "substeps": frame}
    if kind == "wrench":
        return {"kind": kind, "nx": _log_int(rng, 8, 48), "ny": _log_int(rng, 4, 14), "nz": _log_int(rng, 4, 14),
                "substeps": frame}
    if kind == "plate":
        return {"kind": kind, "nx": _log_int(rng, 16, 128), "ny": 1, "nz": _log_int(rng, 16, 128), "substeps": frame}
    if kind == "crack":
        return {"kind": kind, "nx": _log_int(rng, 8, 32), "ny": _log_int(rng, 5, 14), "nz": _log_int(rng, 8, 24),
                "substeps": frame}
    if kind == "impact":
        double = rng.random() < 0.3
        top = 64 if double else 160
        nx = _log_int(rng, 24, top)
        ny, nz = _log_int(rng, 16, max(16, nx // 2)), _log_int(rng, 16, max(16, nx // 2))
        return {"kind": kind, "nx": nx, "ny": ny, "nz": nz, "slabs": rng.choice([1, 3, max(1, nz // 4)]),
                "precision": "double" if double else "float", "substeps": frame}
    if kind == "bar":
        return {"kind": kind, "nx": 2 * _log_int(rng, 12, 64), "ny": 2 * _log_int(rng, 5, 16),
                "nz": _log_int(rng, 8, 32), "steps": rng.choice([1, 2, 4]), "substeps": 10}
    if kind == "trial":
        return {"kind": kind, "nx": _log_int(rng, 8, 48), "ny": _log_int(rng, 8, 48), "nz": _log_int(rng, 8, 48),
                "substeps": rng.choice([60, 120, 240])}
    lo = _log_int(rng, 6, 20)
    hi = rng.randint(lo + 4, 48)
    if kind == "batch":
        return {"kind": kind, "count": _log_int(rng, 8, 128), "lo": lo, "hi": hi, "substeps": rng.choice([60, 120])}
    return {"kind": kind, "count": _log_int(rng, 3, 12), "lo": lo, "hi": hi, "large": rng.choice([0, 56, 72]),
            "substeps": rng.choice([20, 40])}


class Result:
    """Arrays a download writes into, for one lattice or several end to end,
    with one state view per lattice."""

    def __init__(self, nodes, bonds, degrees):
        n, b = int(sum(nodes)), int(sum(bonds))
        # Touched once, as a program's own arrays are after its first frame.
        self.arrays = {k: np.zeros(w * n) for k, w in NODE_ARRAYS.items()}
        self.arrays.update({k: np.zeros(b, dtype=t) for k, t in BOND_ARRAYS.items()})
        for a in self.arrays.values():
            a.fill(1)
        self.parts = []
        n0 = b0 = 0
        for n, b, d in zip(nodes, bonds, degrees):
            self.parts.append(_Part(self.arrays, n0, b0, int(n), int(b), int(d)))
            n0 += int(n)
            b0 += int(b)


class _Part:
    def __init__(self, arrays, n0, b0, n, b, degree):
        self.view = lattice.StateView()
        self.view.node_count, self.view.bond_count, self.view.max_degree = n, b, degree
        for name, ptype in lattice._STATE_ARRAYS:
            if name in NODE_ARRAYS:
                at = arrays[name].ctypes.data + 8 * NODE_ARRAYS[name] * n0
            elif name in BOND_ARRAYS:
                at = arrays[name].ctypes.data + arrays[name].itemsize * b0
            else:
                continue
            setattr(self.view, name, ctypes.cast(at, ptype))


def _status(st):
    c, n = st.contact, st.node_contact
    return {
        "counts": np.array([st.total_steps, st.failure_rounds, st.broken_bonds, st.exit_reason,
                            st.rank_deficient_nodes, c.impulse_contacts, c.candidate_overflow, c.ball_support_events,
                            n.contacts, n.pair_tests, n.rebuilds, n.pairs_listed, n.pair_overflow,
                            st.bond_projections], dtype=np.int64),
        "sums": np.array([st.removed_energy_j, st.max_damage, st.plastic_work_j, c.impulse_to_material_x,
                          c.impulse_to_material_y, c.impulse_to_material_z, c.dissipated_kinetic_energy_j,
                          c.maximum_penetration_m, st.external_load.work_j, *st.external_load.impulse_n_s,
                          *st.external_load.angular_impulse_kg_m2_s, n.dissipated_kinetic_energy_j,
                          n.maximum_overlap_m], dtype=np.float64),
    }


@functools.lru_cache(maxsize=1)
def _block(nx, ny, nz, slabs):
    """A block's geometry, built once and struck again and again: a program
    keeps it; an upload only reads it. Strengths and sphere are the strike's."""
    box = lattice.build_box(nx, ny, nz, H, slabs=slabs)
    schedule = lattice.box_schedule(box)
    return schedule, lattice.box_state(box, schedule)


def _impact(case, rng):
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    schedule, state = _block(nx, ny, nz, case["slabs"])
    strength = rng.standard_normal(state.bond_count, dtype=np.float32)
    strength *= np.float32(0.3)
    np.exp(strength, out=strength)
    strength *= np.float32(1.5e-3)
    thr = state.threshold.reshape(-1, 6)
    thr[:, 0] = strength
    thr[:, 1] = strength
    radius = 0.2 * min(nx, 2 * ny) / 256.0
    where = (rng.random(2) - 0.5) * 0.5 * np.array([nx, nz]) * H
    sphere = scenes.sphere((where[0], 0.5 * ny * H + 0.002 + radius, where[1]), (0.0, -10.0, 0.0), radius)
    double = case["precision"] == "double"
    packed = scenes.settings(sphere_enabled=1, direct=1 if double else 0, yield_stretch=0.9e-3,
                             contact=(0.5, 0.4, 0.0, 0.5, 0.5 * H, 1e-5, 0.05 * radius),
                             planes=[scenes.plane((0.0, -0.5 * ny * H, 0.0), node_radius=0.5 * H)])
    return schedule, state, packed, sphere


def _scene(case, rng):
    """A single-lattice scene as a case of banjo_gb300.scenes."""
    nx, ny, nz, kind = case["nx"], case["ny"], case["nz"], case["kind"]
    if kind == "beam":
        c = scenes.cantilever(nx, ny, nz, steps=1)
        f = c["forces"].reshape(-1, 3)
        f *= rng.uniform(0.8, 1.0)
        f[f[:, 1] != 0, 0::2] = 0.2 * rng.uniform(-1, 1, 2) * 1e-3 * GRAVITY
        c["threshold"] *= rng.uniform(1.0, 1.2)
        return c
    if kind == "wrench":
        return scenes.wrenched_bar(nx, ny, nz, grip=(0.0, -4.0 * rng.uniform(0.5, 1.0), rng.uniform(-1, 1)),
                                   twist=(0.04 * rng.uniform(0.5, 1.0), 0.0, 0.0),
                                   hand=(0.0, 0.0, 2.5 * rng.uniform(0.5, 1.0)))
    if kind == "plate":
        return scenes.plate_strike(nx, nz, radius=0.03 * rng.uniform(0.8, 1.2), speed=8.0 * rng.uniform(0.7, 1.2),
                                   seed_strength=int(rng.integers(1 << 30)))
    if kind == "crack":
        return scenes.contact_drop(nx, ny, nz, break_strain=1.5e-3 * rng.uniform(0.8, 1.2),
                                   speed=3.0 * rng.uniform(0.8, 1.2))
    return scenes.notched_bar(nx, ny, nz, load_factor=2.0 * rng.uniform(0.9, 1.1))


def _trial_box(edges, compliance, strain, height, speed=0.0):
    nx, ny, nz = (int(e) for e in edges)
    thr = (strain, strain, INF, INF, INF, INF)
    box = lattice.build_box(nx, ny, nz, H, (0.0, height + 0.5 * ny * H, 0.0), compliance=compliance, threshold=thr)
    schedule = lattice.box_schedule(box)
    state = lattice.box_state(box, schedule)
    if speed:
        state.v.reshape(-1, 3)[:, 1] = -speed
    return schedule, state


def _ground():
    return lattice.step_settings(scenes.settings(planes=[scenes.plane((0.0, 0.0, 0.0), node_radius=0.5 * H)]))


def _edges(case, rng):
    e = rng.integers(case["lo"], case["hi"] + 1, size=(case["count"], 3))
    if case.get("large"):
        e[case["count"] // 2] = case["large"]
    return e


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind = case["kind"]
    none = lattice.sphere_state(scenes.sphere())
    if kind in ("batch", "serve"):
        # Fixed sizes for a case, so that seeds are alike in work: compliance,
        # strength and height are the seed's.
        edges = _edges(case, np.random.default_rng(5))
        n = case["count"]
        draws = np.stack([10.0 ** rng.uniform(-8, -5, n), rng.uniform(1e-3, 5e-3, n), rng.uniform(0.1, 1.0, n)], 1)
        with concurrent.futures.ThreadPoolExecutor(min(8, os.cpu_count() or 1)) as pool:
            built = list(pool.map(lambda k: _trial_box(edges[k], *draws[k]), range(n)))
        result = Result([s.node_count for _, s in built], [s.bond_count for _, s in built],
                        [s.view.max_degree for _, s in built])
        if kind == "serve":
            return {"case": case, "server": lattice.Server(_ground(), 40 << 30), "requests": built, "result": result,
                    "sphere": none}
        batch = lattice.Batch()
        for schedule, state in built:
            batch.add(schedule, state, none)
        batch.settle(_ground())
        return {"case": case, "batch": batch, "result": result}
    if kind == "trial":
        schedule, state = _trial_box((case["nx"], case["ny"], case["nz"]), 10.0 ** rng.uniform(-8, -6),
                                     rng.uniform(1e-3, 3e-3), 0.002, rng.uniform(1.5, 4.0))
        return {"case": case, "backend": lattice.make_gb300_lattice_backend(schedule), "state": state,
                "settings": _ground(), "sphere": none,
                "result": Result([state.node_count], [state.bond_count], [state.view.max_degree])}
    precision = case.get("precision", "float")
    scene = None
    if kind == "impact":
        schedule, state, packed, sphere = _impact(case, rng)
    else:
        scene = _scene(case, rng)
        schedule = lattice.build_lattice_schedule(int(scene["node_count"][0]), scene["bond_a"], scene["bond_b"],
                                                  scene["node_block_begin"])
        state = lattice.build_lattice_state(scene, schedule)
        packed, sphere = scene["settings"], scene["sphere"]
    backend = lattice.make_gb300_lattice_backend(schedule, precision)
    backend.upload(state, lattice.step_settings(packed), lattice.sphere_state(sphere))
    if kind == "beam":
        backend.set_external_forces(scene["forces"], 1 << 40)
    if kind == "wrench":
        backend.set_external_wrenches(lattice.case_wrenches(scene), 1 << 40)
    st = {"case": case, "backend": backend,
          "result": Result([state.node_count], [state.bond_count], [state.view.max_degree])}
    if kind == "bar":
        st["forces"] = scene["forces"]
        st["scale"] = float(scene["force_ramp_scale"][0]) / float(scene["force_ramp_steps"][0])
        st["step"] = 0
    return st


def run(state):
    case, result = state["case"], state["result"]
    kind = case["kind"]
    control = lattice.RunControl(max_steps=case["substeps"])
    if kind == "batch":
        batch = state["batch"]
        batch.run(control)
        for k, part in enumerate(result.parts):
            batch.download(k, part)
        sums = [_status(batch.status(k)) for k in range(len(result.parts))]
        return dict(result.arrays, counts=np.stack([s["counts"] for s in sums]),
                    sums=np.stack([s["sums"] for s in sums]))
    if kind == "serve":
        server = state["server"]
        tickets = [server.submit(schedule, lat, state["sphere"], case["substeps"], borrow=True)
                   for schedule, lat in state["requests"]]
        while server.step(case["substeps"]).done < len(tickets):
            pass
        sums = [_status(server.take(t, part)[1]) for t, part in zip(tickets, result.parts)]
        return dict(result.arrays, counts=np.stack([s["counts"] for s in sums]),
                    sums=np.stack([s["sums"] for s in sums]))
    backend = state["backend"]
    if kind == "trial":
        backend.upload(state["state"], state["settings"], state["sphere"])
        status = backend.run(control)
    elif kind == "bar":
        for _ in range(case["steps"]):
            backend.set_external_forces(state["scale"] * state["step"] * state["forces"], case["substeps"])
            state["step"] += 1
            status = backend.run(control)
    else:
        status = backend.run(control)
    sphere = backend.download(result.parts[0])
    return dict(result.arrays, sphere=lattice.pack_sphere(sphere), **_status(status))


def _size(nx, ny, nz, horizon=1):
    """Nodes and bonds of a full box, bonds counted offset by offset."""
    offsets = scenes.half_offsets(horizon, 2 if horizon == 1 else None)
    bonds = sum(max(0, nx - abs(dx)) * max(0, ny - abs(dy)) * max(0, nz - abs(dz)) for dx, dy, dz, _ in offsets)
    return nx * ny * nz, bonds


def work(case):
    """Per substep: a node's position, velocity, rest position and masses read
    and its position and velocity written, 112 bytes; a bond's ends, rest
    length, edge, compliance, thresholds and sample history read and the
    history written, 96 bytes; values twice as wide in the double lane. A solve
    is about 70 operations, a bond's strain sample 150, a slot's share of a
    node's strain 30. Passes that start from the caller's arrays read those
    once too, and every pass writes the result."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        sizes = [_size(*(int(x) for x in e)) for e in _edges(case, np.random.default_rng(5))]
    else:
        sizes = [_size(case["nx"], case["ny"], case["nz"], 2 if kind == "bar" else 1)]
    n, b = sum(s[0] for s in sizes), sum(s[1] for s in sizes)
    wide = 2 if case.get("precision") == "double" else 1
    substeps = case["substeps"] * case.get("steps", 1)
    out = 72 * n + 50 * b
    fresh = 112 * n + 164 * b + 2 * 41 * b if kind in ("trial", "serve") else 0
    return {"bytes": substeps * wide * (112 * n + 96 * b) + out + fresh,
            "flops": substeps * (b * (ITERATIONS * 70 + 150 + 2 * 30) + 100 * n)}


def exact(case, seed):
    """A pass from the start in 64 bits. A beam is solved here (no bond of it
    fails in its first frame); boxes in free fall have a closed form; the other
    kinds break within a pass, where 32 and 64 bits part, and have none."""
    kind = case["kind"]
    if kind in ("batch", "serve"):
        n = sum(_size(*(int(x) for x in e))[0] for e in _edges(case, np.random.default_rng(5)))

        def fallen(k):
            u = np.zeros((n, 3))
            u[:, 1] = DT * DT * GRAVITY * (0.5 * k * (k + 1))
            return u

        k = case["substeps"]
        v = np.zeros((n, 3))
        v[:, 1] = k * DT * GRAVITY
        got = {"u": fallen(k).reshape(-1), "u_prev": fallen(k - 1).reshape(-1), "v": v.reshape(-1)}
    elif kind == "beam" and case["substeps"] <= 10:
        got = _beam64(case, seed)
    else:
        return None
    return {key: got.get(key) for key in [*NODE_ARRAYS, *BOND_ARRAYS, "counts", "sums"] +
            ([] if kind in ("batch", "serve") else ["sphere"])}


def _beam64(case, seed):
    """The beam's first frame: kick, prediction, XPBD sweeps colour by colour
    (bonds coloured greedily in the box's own order), velocity."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    rng = np.random.default_rng(seed)
    scale, tilt = rng.uniform(0.8, 1.0), 0.2 * rng.uniform(-1, 1, 2)
    n = nx * ny * nz
    i = np.arange(n)
    grid = np.stack([i % nx, (i // nx) % ny, i // (nx * ny)], 1)
    free = grid[:, 0] > 0
    x0 = (grid + 0.5 - 0.5 * np.array([nx, ny, nz])) * H
    offsets = [(dx, dy, dz) for dz in (-1, 0, 1) for dy in (-1, 0, 1) for dx in (-1, 0, 1)
               if (dz, dy, dx) > (0, 0, 0) and dx * dx + dy * dy + dz * dz <= 2]
    colours, taken = [], [0] * n
    for a in range(n):
        for dx, dy, dz in offsets:
            x, y, z = grid[a, 0] + dx, grid[a, 1] + dy, grid[a, 2] + dz
            if not (0 <= x < nx and 0 <= y < ny and 0 <= z < nz):
                continue
            b = int(x + nx * (y + ny * z))
            c, used = 0, taken[a] | taken[b]
            while used >> c & 1:
                c += 1
            taken[a] |= 1 << c
            taken[b] |= 1 << c
            while len(colours) <= c:
                colours.append([])
            colours[c].append((a, b))
    colours = [np.array(c) for c in colours]
    w = np.where(free, 1e3, 0.0)
    alpha = 1e-7 / (DT * DT)
    force = np.zeros((n, 3))
    force[free] = 1e-3 * GRAVITY * np.array([tilt[0], scale, tilt[1]])
    u, v = np.zeros((n, 3)), np.zeros((n, 3))
    for _ in range(case["substeps"]):
        v = v + DT * w[:, None] * force
        before = u
        u = u + DT * v
        lam = [np.zeros(len(c)) for c in colours]
        for _ in range(ITERATIONS):
            for k, c in enumerate(colours):
                a, b = c[:, 0], c[:, 1]
                rest = np.sqrt(np.sum((grid[b] - grid[a]) ** 2, 1)) * H
                edge, du = x0[b] - x0[a], u[b] - u[a]
                delta = edge + du
                length = np.sqrt(np.sum(delta * delta, 1))
                strain = (np.sum(edge * edge, 1) - rest * rest + 2 * np.sum(edge * du, 1) + np.sum(du * du, 1)) / (
                    length + rest)
                total = w[a] + w[b] + alpha
                dl = (-strain - alpha * lam[k]) / total
                lam[k] += dl
                step = (dl / length)[:, None] * delta
                u[a] -= w[a][:, None] * step
                u[b] += w[b][:, None] * step
        v = (u - before) / DT
    return {"u": u.reshape(-1), "u_prev": before.reshape(-1), "v": v.reshape(-1)}
