"""The step's streaming pass (one launch that records tiles after a cell-list
build and streams the recorded ones) against the CPU oracle, at the forms it
distinguishes: one, two and four lanes per particle, tiles that do not fit
the stream (too many core particles, crowded blocks, candidate lists that
overflow), steps that only stream and steps that rebuild the list.

Tolerances: the passes sum about 20 pair terms per field in FP64 in another
order than the oracle; with condition numbers up to 1e3 of the summed fields
of a stirred tank that is 20 x 1e3 x 2^-53 = 2e-12 per evaluation, taken to
1e-10 over four steps.  FP32 pairs: 1e-4, as the FP32 parity tests."""
import numpy as np
import pytest

from _util import FLUID_FIELDS, compare_fields
from oracle import oracle as O
from uph_b200 import deck as D
from uph_b200._capi import PREC_FP32_PAIR, PREC_FP64, PROFILE_REF, PROFILE_WCSPH

pytestmark = pytest.mark.gpu

SHORT = ["Position", "Velocity", "density", "ddensitydt", "dvdt"]


def _stirred(n, crowd=0, speed=0.05):
    """A dam break of about n particles in motion, off the lattice; `crowd`
    particles near the middle of the column are drawn together."""
    d = D.dam_break(tank=(2.0, 3.0), column=(1.0, 2.0), dx=(2.0 / n) ** 0.5, layers=2, hydrostatic=True)
    p = D.derive_params(d.params, d.eta_override)
    st = d.initial_state()
    rng = np.random.default_rng(n + crowd)
    nf = d.n_fluid
    pos = st["Position"][:nf]
    pos += rng.uniform(-0.1, 0.1, (nf, 2)) * p["dx"]
    if crowd:
        centre = np.array([0.5, 1.0])
        order = np.argsort(((pos - centre) ** 2).sum(axis=1))[:crowd]
        pos[order] = centre + 0.75 * (pos[order] - centre)
    st["Velocity"][:nf] = speed * p["speed_of_sound"] * np.stack(
        [np.sin(3 * pos[:, 0]) * np.cos(2 * pos[:, 1]), -np.cos(3 * pos[:, 0]) * np.sin(2 * pos[:, 1])], axis=1)
    st["localVelocity"][:nf] = st["Velocity"][:nf]
    st["density"][:nf] *= 1 + 1e-4 * rng.standard_normal(nf)
    st["localDensity"][:nf] = st["density"][:nf]
    st["density_min"][:] = st["density"][:nf]
    return d, st


@pytest.mark.parametrize("profile,precision", [(PROFILE_REF, PREC_FP64), (PROFILE_WCSPH, PREC_FP64),
                                               (PROFILE_WCSPH, PREC_FP32_PAIR)])
@pytest.mark.parametrize("n,crowd,tile", [
    (40, 0, None),       # one tile, most lanes idle
    (900, 0, None),      # small tiles, four lanes per particle
    (2000, 0, 8),        # two lanes per particle
    (2000, 0, 11),       # one lane per particle
    (2000, 0, 13),       # a core of more particles than threads: every tile is hard
    (3000, 300, None),   # a crowd: lists that overflow, hard tiles beside streamed ones
    (3000, 300, 11),     # the same with one lane
])
def test_streamed_steps_match_oracle(profile, precision, n, crowd, tile):
    from uph_b200.sim import Simulation
    d, st = _stirred(n, crowd)
    o = O.Oracle(d.uph_params(profile=profile), st)
    o.step(4)
    with Simulation(d.uph_params(profile=profile, precision=precision)) as s:
        s.upload(st, 0)
        if tile:
            s.set_tuning(2, tile, 3)
        s.step(1)
        s.step(3)
        got = s.download()
        builds = s.stats()["list_builds"]
    assert builds >= 1
    if precision == PREC_FP64:
        compare_fields(got, o.state(), d.n_fluid, 1e-10, fields=FLUID_FIELDS if profile == PROFILE_REF else SHORT)
    else:
        compare_fields(got, o.state(), d.n_fluid, 1e-4, fields=SHORT)


@pytest.mark.parametrize("n", [14950, 15050, 29900, 30100])
def test_lane_rule_boundaries(n):
    """Just below and above the sizes at which a particle's lanes change."""
    from uph_b200.sim import Simulation
    d, st = _stirred(n)
    o = O.Oracle(d.uph_params(profile=PROFILE_REF), st)
    o.step(2)
    with Simulation(d.uph_params(profile=PROFILE_REF)) as s:
        s.upload(st, 0)
        s.step(2)
        compare_fields(s.download(), o.state(), d.n_fluid, 1e-10, fields=FLUID_FIELDS)
