"""Rays through the edges and diagonals of the dynamic triangles, many of them grazing their plane, against
the full in-order scan (RC_FLAG_BRUTE_FORCE), bit for bit.  There a trace that tests less than every triangle has
to leave the decision to the exact test: a crossing point that it computes from another rounding of a
plane moves by that over the ray's slope."""
import gzip
import os

import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _rays(st, n, rng):
    """Rays aimed at a point of a triangle's diagonal, of its edges or just beside them; of the origins 40 %
    lie 1e-6 to 0.1 off that triangle's plane and 30 % are cache points', as a frame's are."""
    t = st.T.reshape(-1, 9).astype(np.float64)[rng.integers(0, len(st.T), n)]
    kind, a = rng.integers(0, 3, n), rng.random(n)
    u = np.where(kind == 1, 0.0, a) + rng.choice([0.0, 0.0, 1e-6, 1e-5, 3e-5, 1e-4, 1e-3], n) * rng.choice([-1.0, 1.0], n)
    v = np.where(kind == 0, 1.0 - a, np.where(kind == 1, a, 0.0))
    target = t[:, :3] + t[:, 3:6] * u[:, None] + t[:, 6:] * v[:, None]
    o = rng.uniform(st.P.min(axis=0), st.P.max(axis=0), (n, 3))
    normal = np.cross(t[:, 3:6], t[:, 6:])
    normal /= np.linalg.norm(normal, axis=1, keepdims=True)
    side = ((o - target) * normal).sum(1, keepdims=True)
    near = o - normal * side + normal * (10.0 ** rng.uniform(-6, -1, (n, 1))) * np.where(side < 0, -1.0, 1.0)
    o = np.where(rng.random((n, 1)) < 0.4, near, o)
    i = rng.integers(0, len(st.P), n)
    o = np.where(rng.random((n, 1)) < 0.3, st.P[i] + st.N[i] * np.float32(1e-3), o).astype(np.float32)
    d = (target - o).astype(np.float32)
    length = np.linalg.norm(d, axis=1, keepdims=True)
    d = np.where((rng.random((n, 1)) < 0.5) & (length > 0), d / np.maximum(length, 1e-30), d)
    return np.concatenate([o, d], axis=1).astype(np.float32)


@pytest.mark.parametrize("name", ["room 13", "room 14", "room 12", "main", "stress"])
def test_rays_through_edges_equal_full_scan(name):
    if name.startswith("room"):
        seed = int(name.split()[1])
        sc = S.box_room(points=3000, seed=seed, boxes={12: 6, 13: 4, 14: 9}[seed])
    else:
        sc = S.read(gzip.open(os.path.join(GOLDEN, "scene_%s.bin.gz" % name)).read())
    data = S.write(sc)
    fast, full = N.Context(), N.Context(flags=N.FLAG_BRUTE_FORCE)
    fast.load_bytes(data)
    full.load_bytes(data)
    for state in (0, 2):
        rays = _rays(sc.states[state], 1_500_000, np.random.default_rng(31 + state))
        p0, t0 = fast.trace_rays(state, rays)
        p1, t1 = full.trace_rays(state, rays)
        wrong = np.nonzero((p0 != p1) | (t0.view(np.uint32) != t1.view(np.uint32)))[0]
        assert len(wrong) == 0, (state, len(wrong), rays[wrong[0]], p0[wrong[0]], t0[wrong[0]], p1[wrong[0]], t1[wrong[0]])
        assert (p1 >= 0).mean() > 0.5
    fast.close()
    full.close()
