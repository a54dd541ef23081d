"""The k-nearest cut of the capped search (a warp per query) against a brute
force on the CPU: pair sets exactly equal, at the forms the selection
distinguishes: fewer and more in-radius points than the cap, rings of equal
distances (ties go to the smaller index), more points in one distance bin than
its list holds, and more equal distances than that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

EPS = np.finfo(np.float64).eps


def brute(pos, nf, pb, dist, k):
    out = []
    for s in range(nf):
        dx, dy = pos[s, 0] - pos[:, 0], pos[s, 1] - pos[:, 1]
        r2 = dx * dx + dy * dy
        c = np.flatnonzero((r2 < dist) & (r2 > EPS))
        c = c[np.lexsort((c, r2[c]))][:k]
        c = np.sort(c[(c > s) & (c < pb)])
        out += [(s, j, r2[j]) for j in c]
    return out


def clouds():
    rng = np.random.default_rng(5)
    x, y = np.meshgrid(np.arange(24.0), np.arange(20.0))
    lattice = np.stack([x.ravel(), y.ravel()], axis=1)
    yield "sparse", rng.uniform(0, 30, (600, 2)), 2.0, 40
    yield "lattice_ties", lattice, 5.5, 40
    yield "lattice_ties_k1", lattice, 2.5, 1
    yield "lattice_ties_k64", lattice, 6.5, 64
    yield "shuffled", (lattice + rng.uniform(-0.3, 0.3, lattice.shape))[rng.permutation(480)], 5.0, 40
    # 300 points at nearly one distance from a centre, and at exactly one
    t = np.linspace(0, 2 * np.pi, 300, endpoint=False)
    ring = np.stack([np.cos(t), np.sin(t)], axis=1)
    yield "near_ring", np.concatenate([np.zeros((1, 2)), ring * (1 + 1e-9 * rng.standard_normal((300, 1)))]), 1.5, 40
    dyadic = np.concatenate([np.tile([[3.0, 4.0], [-3.0, 4.0], [3.0, -4.0], [5.0, 0.0], [0.0, -5.0]], (20, 1))])
    yield "equal_ring", np.concatenate([np.zeros((1, 2)), dyadic, [[1.0, 0.0]]]), 6.0, 40


@pytest.mark.parametrize("name,pos,radius,k", list(clouds()), ids=lambda v: v if isinstance(v, str) else "")
def test_cut_matches_brute_force(name, pos, radius, k):
    from uph_b200.sim import search_neighbors
    n = pos.shape[0]
    nf, pb, dist = max(1, n - 7), n - 1, radius * radius
    i, j, r2 = search_neighbors(pos, nf, pb, dist, k)
    want = brute(pos, nf, pb, dist, k)
    assert list(zip(i.tolist(), j.tolist())) == [(a, b) for a, b, _ in want]
    assert np.array_equal(r2, np.array([w[2] for w in want]))
