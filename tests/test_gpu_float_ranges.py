"""Operands outside the branch-free quotients' ranges, against the CPU checker.

The float lane's bond step, sample and contact chains divide branch-free where
every divisor is within 2^-90..2^30, every dividend zero or at least 2^-90 and
every square below 2^60, and form the expression again with `/` and sqrt where
one is not. Each scene here has operands on the far side of one of those
bounds in most of its bonds or contacts (stated beside it), and its results are
the checker's bit for bit. Levels launched one by one and the staged sweep of
one CTA share the step and are both run.
"""
import numpy as np
import pytest

from _util import LEDGER_RTOL, STATE_KEYS, mismatches, status_mismatches

pytestmark = pytest.mark.gpu

LEAST = 2.0 ** -90


def _thrown(nx, ny, nz, speed=4.0, compliance=1e-7, **kw):
    from banjo_gb300 import scenes

    case = scenes.drop_trial(nx, ny, nz, compliance=compliance, break_strain=1.5e-3, drop_height=0.002, steps=2, **kw)
    vel = case["vel"].reshape(-1, 3).copy()
    vel[:, 1] = -speed
    case["vel"] = vel.reshape(-1)
    case["settings"] = case["settings"].copy()
    return case


def _tiny_compliance(shape):
    assert 0 < np.float32(1e-30) < LEAST
    return _thrown(*shape, compliance=1e-30)  # a dividend: compliance over dt^2


def _heavy(shape):
    case = _thrown(*shape, compliance=0.0)
    case["mass"] = np.full_like(case["mass"], 1e30)
    assert np.float32(2e-30) < LEAST  # a divisor: the inverse masses' sum, with no compliance beside it
    return case


def _heavy_among_light(shape):
    case = _heavy(shape)
    case["mass"][::3] = 1e-3  # lanes of a warp on both sides
    return case


def _tiny_displacements(shape):
    # Axis-aligned bonds' other components, and the numerators, of about 1e-31.
    from banjo_gb300 import scenes

    case = _thrown(*shape, speed=0.0)
    rng = np.random.default_rng(5)
    case["vel"] = (rng.random(case["vel"].size) - 0.5) * 1e-27
    case["settings"][scenes.K_GRAVITY:scenes.K_GRAVITY + 3] = 0.0
    assert 1e-27 * scenes.DT_SUBSTEP < LEAST
    return case


def _tiny_timestep(shape):
    from banjo_gb300 import scenes

    case = _thrown(*shape, speed=1e9)
    case["settings"][scenes.K_DT] = 1e-14
    assert np.float32(1e-14) ** 2 < LEAST  # dt^2 itself, a divisor
    return case


def _large_timestep(shape):
    from banjo_gb300 import scenes

    case = _thrown(*shape, speed=1e-8, compliance=1e-3)
    case["settings"][scenes.K_DT] = 65536.0
    case["settings"][scenes.K_GRAVITY:scenes.K_GRAVITY + 3] = (0.0, -1e-13, 0.0)
    assert 65536.0 ** 2 >= 2.0 ** 30
    return case


def _vast(shape):
    # Cells of 4e9 m: squared lengths past 2^60, lengths past 2^30.
    case = _thrown(*shape, speed=2e12, h=4e9)
    assert (4e9) ** 2 > 2.0 ** 60
    return case


BONDS = {f.__name__[1:]: f for f in (_tiny_compliance, _heavy, _heavy_among_light, _tiny_displacements, _tiny_timestep,
                                     _large_timestep, _vast)}


def _equal(device, port, case):
    cpu = port.run_port(case, threads=2)
    assert np.isfinite(cpu["u"]).all() and np.isfinite(cpu["v"]).all()  # a NaN's bits are nobody's
    gpu = device.run_case(case)
    assert mismatches(cpu, gpu, STATE_KEYS) == []
    assert status_mismatches(cpu, gpu, ledger_rtol=LEDGER_RTOL) == []
    return cpu


@pytest.mark.parametrize("shape", [(7, 5, 6), (40, 8, 8)], ids=["staged", "levels"])
@pytest.mark.parametrize("name", list(BONDS))
def test_bonds_match_checker(device, port, name, shape):
    cpu = _equal(device, port, BONDS[name](shape))
    assert float(np.abs(cpu["u"]).max()) > 0.0


@pytest.mark.parametrize("yield_stretch", [0.0, 9e-4])
@pytest.mark.parametrize("kind", ["heavy nodes", "heavy all", "slow", "vast"])
def test_sphere_contacts_match_checker(device, port, kind, yield_stretch):
    """Impulses between masses of 1e30 (the effective inverse mass a divisor
    below 2^-90), speeds whose squares leave the range, and vast cells."""
    from banjo_gb300 import scenes

    h = 4e9 if kind == "vast" else 0.01
    scale = h / 0.01
    case = scenes.impact_block(nx=12, ny=6, nz=10, h=h, blocks=3, radius=0.03 * scale, speed=12.0 * scale,
                               gap=0.0005 * scale, steps=2)
    case["settings"] = case["settings"].copy()
    case["settings"][scenes.K_YIELD] = yield_stretch
    if kind.startswith("heavy"):
        case["mass"] = np.full_like(case["mass"], 1e30)
        case["compliance"] = np.zeros_like(case["compliance"])
        if kind == "heavy all":
            sphere = case["sphere"].copy()
            sphere[-2:] = (1e30, 1e27)  # mass, inertia
            case["sphere"] = sphere
    elif kind == "slow":
        sphere = case["sphere"].copy()
        sphere[1] -= 0.0006  # already touching, at a speed of 1e-20 m/s
        sphere[4] = -1e-20
        case["sphere"] = sphere
        case["settings"][scenes.K_GRAVITY:scenes.K_GRAVITY + 3] = 0.0
    cpu = _equal(device, port, case)
    assert int(cpu["status_u64"][9]) > 0  # impulses


@pytest.mark.parametrize("kind", ["heavy", "heavy among light", "slow"])
def test_node_contacts_match_checker(device, port, kind):
    from banjo_gb300 import scenes

    case = scenes.contact_drop(nx=6, ny=5, nz=5, compliance=0.0, break_strain=5e-4, speed=6.0, steps=24)
    if kind == "slow":
        case["vel"] = (np.random.default_rng(7).random(case["vel"].size) - 0.5) * 1e-20
        case["settings"][scenes.K_GRAVITY:scenes.K_GRAVITY + 3] = 0.0
        case["alive"] = np.zeros(int(case["bond_count"][0]), dtype=np.uint8)
        case["pos"] = case["pos"].reshape(-1, 3) * 0.999
        case["pos"] = case["pos"].reshape(-1)
    else:
        case["mass"] = np.full_like(case["mass"], 1e30)
        if kind == "heavy among light":
            case["mass"][::3] = 1e-3
    cpu = _equal(device, port, case)
    assert int(cpu["status_u64"][13]) > 0  # contacts
