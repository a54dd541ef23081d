"""The step pass at each number of lanes per particle, against the CPU oracle:
the tiles and sizes that give four, two and one, hard tiles and overflowing
lists beside two-lane streamed tiles, both sides of the sizes at which the
default changes.  Tolerance as in the streaming tests: 1e-10 over the steps."""
import pytest

from _util import FLUID_FIELDS, compare_fields
from oracle import oracle as O
from test_gpu_stream import SHORT, _stirred
from uph_b200._capi import PREC_FP32_PAIR, PREC_FP64, PROFILE_REF, PROFILE_WCSPH

pytestmark = pytest.mark.gpu


def _check(profile, n, crowd, tile, lanes, steps):
    from uph_b200.sim import Simulation
    d, st = _stirred(n, crowd)
    o = O.Oracle(d.uph_params(profile=profile), st)
    o.step(steps)
    with Simulation(d.uph_params(profile=profile, precision=PREC_FP64)) as s:
        if tile:
            s.set_tuning(2, tile, 3)
        assert s.tuning()[3] == lanes
        s.upload(st, 0)
        s.step(1)
        s.step(steps - 1)
        compare_fields(s.download(), o.state(), d.n_fluid, 1e-10,
                       fields=FLUID_FIELDS if profile == PROFILE_REF else SHORT)


@pytest.mark.parametrize("profile", [PROFILE_REF, PROFILE_WCSPH])
@pytest.mark.parametrize("n,crowd,tile,lanes", [
    (2000, 0, 5, 4), (2000, 0, 6, 2), (2000, 0, 7, 2), (2000, 0, 8, 1),
    (3000, 300, 6, 2), (3000, 300, 7, 2),
])
def test_lanes(profile, n, crowd, tile, lanes):
    _check(profile, n, crowd, tile, lanes, 4)


@pytest.mark.parametrize("profile", [PROFILE_REF, PROFILE_WCSPH])
@pytest.mark.parametrize("n,lanes", [(14950, 4), (15050, 2), (29900, 2), (30100, 1)])
def test_default_lanes(profile, n, lanes):
    _check(profile, n, 0, None, lanes, 2)


def test_fp32_pairs_keep_one_lane():
    from uph_b200.sim import Simulation
    d, _ = _stirred(900)
    with Simulation(d.uph_params(profile=PROFILE_WCSPH, precision=PREC_FP32_PAIR)) as s:
        assert s.tuning()[1:] == (11, 64, 1)
        s.set_tuning(2, 5, 64)
        assert s.tuning() == (2, 5, 64, 1)
