"""Wide kernels without the k-nearest cap (nearNeighbor 50 to 91): tiles whose
blocks do not fit the step's stream take the tiled pass, a launch of their own
behind the list's, and both forms give the oracle's state.  Tolerance: about
90 pair terms a field with condition numbers up to 1e3 give
90 x 1e3 x 2^-53 = 1e-11 an evaluation, taken to 1e-10 over three steps; FP32
pairs 1e-4, as the FP32 parity tests."""
import math

import numpy as np
import pytest

from _util import FLUID_FIELDS, compare_fields
from oracle import oracle as O
from uph_b200 import deck as D
from uph_b200._capi import PREC_FP32_PAIR, PREC_FP64, PROFILE_REF, PROFILE_WCSPH

pytestmark = pytest.mark.gpu

SHORT = ["Position", "Velocity", "density", "ddensitydt", "dvdt"]


def _tank(n, near):
    d = D.dam_break(tank=(2.0, 3.0), column=(1.0, 2.0), dx=(2.0 / n) ** 0.5, layers=2, hydrostatic=True,
                    eta=math.sqrt(near / (4.0 * math.pi)))
    st = d.initial_state()
    st["Position"][:d.n_fluid] += np.random.default_rng(n).uniform(-0.1, 0.1, (d.n_fluid, 2)) * d.params["dx"]
    return d, st


@pytest.mark.parametrize("profile,precision", [(PROFILE_REF, PREC_FP64), (PROFILE_WCSPH, PREC_FP64),
                                               (PROFILE_WCSPH, PREC_FP32_PAIR)])
@pytest.mark.parametrize("near,tile,streams", [
    (45, 7, True),    # 478 records a lattice block, of 488 that a buffer holds
    (50, 7, False),   # 531
    (61, 6, False),   # the default tiles of larger tanks
    (91, 5, False),
    (91, 3, True),
    (0, 13, False),   # h = 1.3 dx: 538
])
def test_wide_kernels(profile, precision, near, tile, streams):
    from uph_b200.sim import Simulation
    d, st = _tank(2500, near or 4.0 * math.pi * 1.69)
    o = O.Oracle(d.uph_params(profile=profile), st)
    o.step(3)
    with Simulation(d.uph_params(profile=profile, precision=precision)) as s:
        s.set_tuning(2, tile, 64)
        s.upload(st, 0)
        s.step(1)
        before = s.launch_count()
        s.step(2)
        launches = s.launch_count() - before  # the predictor and two steps
        got = s.download()
    assert launches == (3 if streams else 5)
    if precision == PREC_FP64:
        compare_fields(got, o.state(), d.n_fluid, 1e-10, fields=FLUID_FIELDS if profile == PROFILE_REF else SHORT)
    else:
        compare_fields(got, o.state(), d.n_fluid, 1e-4, fields=SHORT)
