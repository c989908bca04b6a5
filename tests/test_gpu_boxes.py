"""The box slabs of the dynamic triangles' trace against the full in-order scan
(RC_FLAG_BRUTE_FORCE), bit for bit: rooms, rooms with a wall missing, a lone cube without a room,
overlapping and coincident boxes; rays from anywhere, along the axes, and aimed at what the slabs
cannot decide (edges, corners, diagonals, origins on and inside faces)."""
import gzip
import os

import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu
GOLDEN = os.path.join(os.path.dirname(__file__), "golden")


def _from_quads(quads, points=600):
    """A one-state room file from (o, u, v, n) quads."""
    sc = S.box_room(points=points, seed=0)
    Q = np.array([[*o, *u, *v, *n] for o, u, v, n in quads], np.float32)
    T = np.empty((2 * len(Q), 9), np.float32)
    P, Nn = [], []
    for i, q in enumerate(Q):
        o, u, v, n = q[:3], q[3:6], q[6:9], q[9:]
        T[2 * i] = np.concatenate([o, u, v])
        T[2 * i + 1] = np.concatenate([o + u + v, -u, -v])
        for a in (0.25, 0.75):
            for b in (0.25, 0.75):
                P.append(o + np.float32(a) * u + np.float32(b) * v)
                Nn.append(n)
    nq = len(Q)
    st = S.State(inten=sc.states[0].inten, P=np.array(P, np.float32), N=np.array(Nn, np.float32), Q=Q, dims=np.full((nq, 2), 2, np.int32),
                 off=(4 * np.arange(nq)).astype(np.int32), T=T, TQ=np.repeat(np.arange(nq, dtype=np.int32), 2))
    return S.write(S.Scene(NR=1, L=sc.L, A=np.full(4 * nq, 0.5, np.float32), region=np.zeros(4 * nq, np.int32), states=[st]))


def _scene(name):
    room = S._room_quads()
    a, b = ((1.0, 1.0, 0.0), (2.0, 2.2, 1.0)), ((1.5, 1.4, 0.0), (3.0, 3.0, 0.7))
    if name == "room":
        return S.write(S.box_room(points=3000, seed=5))
    if name == "room 9 boxes":
        return S.write(S.box_room(points=3000, seed=2, boxes=9))
    if name in ("main", "stress"):
        return gzip.open(os.path.join(GOLDEN, "scene_%s.bin.gz" % name)).read()
    if name == "empty room":
        return _from_quads(room)
    if name == "no ceiling":
        return _from_quads(room[:1] + room[2:] + S._box_quads(*a))
    if name == "overlapping":
        return _from_quads(room + S._box_quads(*a) + S._box_quads(*b, with_bottom=True))
    if name == "coincident":
        return _from_quads(room + S._box_quads(*a) + S._box_quads(*a) + S._box_quads((0.0, 0.0, 0.0), (0.5, 0.5, 3.0)))
    if name == "panels":   # lone rectangles, one of them in the plane of a wall
        return _from_quads(room + [((2.0, 1.0, 0.5), (0, 2.0, 0), (0, 0, 1.5), (1, 0, 0)), ((0.0, 1.0, 1.0), (0, 1.0, 0), (0, 0, 1.0), (1, 0, 0)),
                                   ((5.0, 0.0, 2.0), (2.0, 0, 0), (0, 4.0, 0), (0, 0, -1))])
    if name == "cube alone":
        return _from_quads(S._box_quads((3.0, 1.0, 1.0), (4.0, 2.0, 2.0), with_bottom=True))
    if name == "slanted edges":   # a parallelogram in an axis-aligned plane: no rectangle record
        return _from_quads(room + [((2.0, 1.0, 1.0), (1.0, 0.4, 0), (0.2, 1.0, 0), (0, 0, 1))] + S._box_quads(*a))
    raise KeyError(name)


def _rays(data, seed):
    """Origins and directions over the scene's box and a little beyond, and rays aimed at the points
    of its triangles where two answers lie close together."""
    sc = S.read(data)
    st = sc.states[0]
    rng = np.random.default_rng(seed)
    lo, hi = st.P.min(axis=0) - 0.3, st.P.max(axis=0) + 0.3
    n = 4000

    def unit(k):
        d = rng.normal(size=(k, 3))
        return d / np.linalg.norm(d, axis=1, keepdims=True)

    o = [rng.uniform(lo, hi, (n, 3))]
    d = [unit(n)]
    i = rng.integers(0, len(st.P), n)                      # from the cache points, as frames do
    o.append(st.P[i] + st.N[i] * np.float32(1e-3))
    dd = unit(n)
    d.append(np.where((dd * st.N[i]).sum(1, keepdims=True) < 0, -dd, dd))
    axes = np.eye(3)[rng.integers(0, 3, n)] * rng.choice([-1.0, 1.0], (n, 1))
    o.append(rng.uniform(lo, hi, (n, 3)))
    d.append(axes)                                          # along the axes
    o.append(st.P[i])
    d.append(axes + unit(n) * 10.0 ** rng.uniform(-7, -1, (n, 1)))   # nearly along them, from the faces
    t = st.T[rng.integers(0, len(st.T), 3 * n)].astype(np.float64)
    a = rng.choice([0.0, 1.0, 0.5], 3 * n) + rng.choice([0.0, 1e-6, -1e-5, 1e-4, -1e-3], 3 * n)
    b = np.where(rng.random(3 * n) < 0.5, 1.0 - a, rng.uniform(0, 1, 3 * n))
    target = t[:, :3] + t[:, 3:6] * a[:, None] + t[:, 6:] * b[:, None]   # edges, corners, diagonals
    src = rng.uniform(lo, hi, (3 * n, 3))
    src[:n] = st.P[i]
    o.append(src)
    d.append(target - src)                                  # not unit length
    return np.concatenate([np.concatenate(o), np.concatenate(d)], axis=1).astype(np.float32)


@pytest.mark.parametrize("name", ["room", "room 9 boxes", "main", "stress", "empty room", "no ceiling", "overlapping", "coincident", "panels",
                                  "cube alone", "slanted edges"])
def test_boxes_equal_full_scan(name):
    data = _scene(name)
    fast, full = N.Context(), N.Context(flags=N.FLAG_BRUTE_FORCE)
    fast.load_bytes(data)
    full.load_bytes(data)
    for state in range(min(fast.info()["ns"], 3)):
        rays = _rays(data, 17 + state)
        p0, t0 = fast.trace_rays(state, rays)
        p1, t1 = full.trace_rays(state, rays)
        assert (p1 >= 0).mean() > 0.02
        np.testing.assert_array_equal(p0, p1)
        np.testing.assert_array_equal(t0.view(np.uint32), t1.view(np.uint32))
    fast.close()
    full.close()
