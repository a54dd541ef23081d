"""The capped pair list of tanks whose lattice has fewer points in radius than
the cap: from 10,000 queries on they are counted a lane each, and only those of a
crowd go on to the warp's selection; below, a warp takes each query.  Against a brute force on the CPU, pair sets exactly equal,
with and without the virtual mirror particles, which count as points too."""
import numpy as np
import pytest

from uph_b200 import deck as D

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


@pytest.mark.parametrize("virtual_type", [77, 8])
@pytest.mark.parametrize("n,crowd", [(30, 0), (700, 60), (9900, 300), (10200, 0), (10200, 60), (12000, 3000)])
def test_counted_cut_matches_brute_force(virtual_type, n, crowd):
    from uph_b200.sim import Simulation
    d = D.dam_break(tank=(2.0, 3.0), column=(1.0, 2.0), dx=(2.0 / n) ** 0.5, layers=2, flat_bottom_length=2.0)
    d.params["virtual_type"] = virtual_type
    st, nf = d.initial_state(), d.n_fluid
    pos = st["Position"]
    pos[:nf] += np.random.default_rng(n).uniform(-0.1, 0.1, (nf, 2)) * d.params["dx"]
    if crowd:  # at the column's foot, beside the mirrors
        order = np.argsort((pos[:nf] ** 2).sum(axis=1))[:crowd]
        pos[order] *= 0.6
    with Simulation(d.uph_params(knn_cap=40)) as s:
        s.upload(st, 1)
        s.derivatives(0.0)
        i, j, r2, _, _ = s.pairs()
        mirrors = s.virtual()[0]
    assert (len(mirrors) > 0) == (virtual_type == 8)
    points = np.concatenate([pos, mirrors])
    dist = (2.0 * D.derive_params(d.params, d.eta_override)["h"]) ** 2
    want, cut = [], 0
    for a in range(nf):
        dx, dy = pos[a, 0] - points[:, 0], pos[a, 1] - points[:, 1]
        q2 = dx * dx + dy * dy
        c = np.flatnonzero((q2 < dist) & (q2 > EPS))
        cut += c.size > 40
        c = c[np.lexsort((c, q2[c]))][:40]
        c = np.sort(c[(c > a) & (c < d.n_all - 1)])
        want += [(a, b, q2[b]) for b in c]
    assert (cut > 0) == (crowd > 0) and cut < nf
    assert list(zip(i.tolist(), j.tolist())) == [(a, b) for a, b, _ in want]
    assert np.array_equal(r2, np.array([w[2] for w in want]))
