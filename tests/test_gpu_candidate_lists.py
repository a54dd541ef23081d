"""The step's candidate lists: complete whenever they are written, and the same
whether they are kept or written at every step."""
import numpy as np
import pytest

from uph_b200 import deck as D
from uph_b200._capi import PREC_FP32_PAIR, PREC_FP64, PROFILE_REF, PROFILE_WCSPH

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("profile", [PROFILE_REF, PROFILE_WCSPH])
@pytest.mark.parametrize("lists", [True, False])
def test_lists_written_after_the_walls_moved(profile, lists):
    """A rate evaluation bins the particles; the first step then moves a wall
    particle away from where it was binned and writes the lists, the next one
    moves it back past that place while a fluid particle comes to meet it.
    Nobody leaves the skin, so nothing is binned again: the pair, 3.07 skins
    closer than when the lists were written, has to be on them."""
    from uph_b200.sim import Simulation
    dx = 0.02
    params = D.base_params(dx, gravity_flag=0)
    p = D.derive_params(params, 1.3)
    radius, dt = 2.0 * p["h"], p["time_step"]
    skin = 0.025 * radius
    m = 0.97 * skin
    along = np.array([3.0, 1.0]) / np.sqrt(10.0)
    wall = np.array([0.2, 0.2])                                   # as binned
    fluid = wall + [-m, 0.0] + (radius + 2.9 * skin) * along      # from where the lists are written
    mass = p["density0"] * dx * dx
    walls = np.array([wall, wall - 8.0 * radius])                 # the last one is never in a pair
    rows = D._rows(walls[:, 0], walls[:, 1], p["density0"], 0.0, mass, 3)
    d = D.Deck(params, D._rows(fluid[:1], fluid[1:], p["density0"], 0.0, mass, 1), np.zeros((0, 12)),
               np.zeros((0, 12)), rows, eta_override=1.3, domain_lo=(-1.0, -1.0), domain_hi=(1.0, 1.0))
    st = d.initial_state()
    st["Velocity"][0] = st["localVelocity"][0] = -m / dt
    with Simulation(d.uph_params(profile=profile)) as s:
        # x = x0 + hs (1 - cos wt): at dt / 2 where it is binned, at dt 0.97 skins back, at 2 dt as much ahead
        s.set_wall_motion(walls[:, 0] + [m, 0.0], np.array([-m, 0.0]), np.full(2, np.pi / dt))
        s.set_candidate_lists(lists)
        s.upload(st, 0)
        s.derivatives(0.5 * dt)
        builds = s.stats()["list_builds"]
        s.step(1)
        assert s.stats()["niac"] == 0
        s.step(1)
        got = s.stats()
        assert got["list_builds"] == builds  # no particle left its skin
        assert got["niac"] == 1


def _stirred(n):
    d = D.dam_break(tank=(2.0, 3.0), column=(1.0, 2.0), dx=(2.0 / n) ** 0.5, layers=2, hydrostatic=True)
    p = D.derive_params(d.params, d.eta_override)
    st = d.initial_state()
    rng, nf = np.random.default_rng(n), d.n_fluid
    pos = st["Position"][:nf]
    pos += rng.uniform(-0.1, 0.1, (nf, 2)) * p["dx"]
    st["Velocity"][:nf] = 0.05 * p["speed_of_sound"] * np.stack(
        [np.sin(3 * pos[:, 0]) * np.cos(2 * pos[:, 1]), -np.cos(3 * pos[:, 0]) * np.sin(2 * pos[:, 1])], axis=1)
    st["localVelocity"][:nf] = st["Velocity"][:nf]
    return d, st


@pytest.mark.parametrize("profile,precision", [(PROFILE_REF, PREC_FP64), (PROFILE_WCSPH, PREC_FP64),
                                               (PROFILE_WCSPH, PREC_FP32_PAIR)])
@pytest.mark.parametrize("n,tile", [(3000, None), (3000, 7), (3000, 11), (17000, None)])
def test_kept_lists_change_no_bit(profile, precision, n, tile):
    """Default tuning (four lanes per particle at 3,000 particles and two at
    17,000 in FP64), two lanes and one: steps between builds, over several."""
    from uph_b200.sim import Simulation
    d, st = _stirred(n)
    got = []
    for lists in (True, False):
        with Simulation(d.uph_params(profile=profile, precision=precision)) as s:
            if tile:
                s.set_tuning(2, tile, 64)
            s.set_candidate_lists(lists)
            s.upload(st, 0)
            s.step(60)
            got.append(s.download())
            assert s.stats()["list_builds"] > 2
    for f, a in got[0].items():
        assert np.array_equal(a, got[1][f]), f


@pytest.mark.parametrize("precision,tile,launches", [(PREC_FP64, 11, 5), (PREC_FP32_PAIR, None, 5), (PREC_FP64, 7, 3)])
def test_steps_without_kept_lists(precision, tile, launches):
    """With one lane per particle nothing is recorded for one step alone: a
    list launch and the tiled pass, behind the call's predictor."""
    from uph_b200.sim import Simulation
    d, st = _stirred(3000)
    with Simulation(d.uph_params(profile=PROFILE_WCSPH, precision=precision)) as s:
        if tile:
            s.set_tuning(2, tile, 64)
        s.set_candidate_lists(False)
        s.upload(st, 0)
        s.step(1)
        before = s.launch_count()
        s.step(2)
        assert s.launch_count() - before == launches


@pytest.mark.parametrize("profile,precision", [(PROFILE_REF, PREC_FP64), (PROFILE_WCSPH, PREC_FP64),
                                               (PROFILE_WCSPH, PREC_FP32_PAIR)])
@pytest.mark.parametrize("piston_layers", [1, 3])
def test_moving_walls_step_alike(profile, precision, piston_layers):
    """A wave flume's piston (the reference's law, and a table) where steps
    stream and where they take the tiled pass, as single calls and as a graph."""
    from uph_b200.sim import Simulation
    d = D.wave_flume(2.0, 0.4, 0.016, piston_layers=piston_layers, hydrostatic_walls=True)
    st = d.initial_state()
    got = []
    for lists, graph in ((True, 0), (False, 0), (True, 30), (False, 30)):
        with Simulation(d.uph_params(profile=profile, precision=precision)) as s:
            s.set_tuning(2, 11, 64)
            if d.wall_table is not None:
                s.set_wall_motion(*d.wall_table)
            s.set_candidate_lists(lists)
            s.set_graph(graph)
            s.upload(st, 0)
            s.step(1)
            s.step(30)
            s.step(30)
            got.append(s.download())
    assert np.abs(got[0]["Position"] - st["Position"])[d.n_fluid:].max() > 0
    for other in got[1:]:
        for f, a in got[0].items():
            assert np.array_equal(a, other[f]), f
