"""A value that is not finite acts only through pairs: a wall particle outside
every fluid particle's radius, but within the distance at which the step's
candidate lists hold it, and the last boundary particle, which the reference's
pair search leaves out, change nothing whatever they hold.  Bit for bit, at
each number of lanes per particle, in both profiles and precisions."""
import numpy as np
import pytest

from uph_b200 import deck as D
from uph_b200._capi import PREC_FP32_PAIR, PREC_FP64, PROFILE_REF, PROFILE_WCSPH

pytestmark = pytest.mark.gpu

# velocity, pressure and (through the reciprocal of a zero) density
POISON = {"Velocity": np.nan, "DynamicPressure": np.inf, "density": 0.0, "mass": np.nan}


def _tank(n):
    d = D.dam_break(tank=(2.0, 3.0), column=(1.0, 2.0), dx=(2.0 / n) ** 0.5, layers=2, hydrostatic=True)
    st = d.initial_state()
    st["Position"][:d.n_fluid] += np.random.default_rng(n).uniform(-0.05, 0.05, (d.n_fluid, 2)) * d.params["dx"]
    return d, st


@pytest.mark.parametrize("profile,precision", [(PROFILE_REF, PREC_FP64), (PROFILE_WCSPH, PREC_FP64),
                                               (PROFILE_WCSPH, PREC_FP32_PAIR)])
@pytest.mark.parametrize("tile", [5, 7, 11])
@pytest.mark.parametrize("who", ["beyond the radius", "last boundary particle"])
def test_partners_outside_the_pairs_do_not_act(profile, precision, tile, who):
    from uph_b200.sim import Simulation
    d, st = _tank(2000)
    p, nf = D.derive_params(d.params, d.eta_override), d.n_fluid
    radius = 2.0 * p["h"]
    pos = st["Position"]
    if who == "last boundary particle":
        k = d.n_all - 1
        poison = {f: v for f, v in POISON.items() if f != "mass"}  # its mass is in the brute-force wall laws
    else:
        k, poison = nf, POISON  # the first wall particle, put in front of the column
    front = np.argmax(pos[:nf, 0] - 10.0 * np.abs(pos[:nf, 1] - 1.0))
    pos[k] = pos[front] + np.array([radius * (1.02 if k == nf else 0.6), 0.0])
    r = np.sqrt(((pos[:nf] - pos[k]) ** 2).sum(axis=1))
    assert k != nf or radius < r.min() < 1.03 * radius
    got = []
    for fields in ({}, poison):
        s_in = {f: a.copy() for f, a in st.items()}
        for f, v in fields.items():
            s_in[f][k] = v
        with Simulation(d.uph_params(profile=profile, precision=precision)) as s:
            s.set_tuning(2, tile, 64)
            s.upload(s_in, 0)
            s.step(1)
            s.step(2)
            got.append(s.download())
    for f in ("Position", "Velocity", "density", "DynamicPressure", "ddensitydt", "dvdt"):
        assert np.all(np.isfinite(got[1][f][:nf])), f
        assert np.array_equal(got[0][f][:nf], got[1][f][:nf]), f
