"""Frames of rooms whose rays the box slabs often leave undecided cost no more than with the plane filter alone.
The filter's side is the same room with a speck of a quad turned out of the axes in it, which sends the whole
state there; both sides of a comparison run in turn on the same GPU, and the allowance is far below what
undecided rays cost when each scanned every triangle (1.45 and 2.8 times)."""
import statistics
import time

import numpy as np
import pytest

from render_engine_gb300 import methods as M
from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _room(scale, speck):
    sc = S.box_room(points=200_000, seed=3)
    for st in sc.states:
        if speck:
            q = np.array([[4.0, 2.0, 2.9, 1e-3, 1e-3, 0.0, 0.0, 0.0, 1e-3, 0.0, 1.0, 0.0]], np.float32)
            st.Q = np.concatenate([st.Q, q])
            st.dims = np.concatenate([st.dims, [[1, 1]]]).astype(np.int32)
            st.off = np.concatenate([st.off, [len(st.P)]]).astype(np.int32)
            t = np.array([[*q[0, :9]], [*(q[0, :3] + q[0, 3:6] + q[0, 6:9]), *-q[0, 3:9]]], np.float32)
            st.T = np.concatenate([st.T, t])
            st.TQ = np.concatenate([st.TQ, [len(st.Q) - 1] * 2]).astype(np.int32)
            st.P = np.concatenate([st.P, q[:, :3]])
            st.N = np.concatenate([st.N, q[:, 9:]])
        st.P, st.T, st.Q = (st.P * np.float32(scale)), (st.T * np.float32(scale)), st.Q.copy()
        st.Q[:, :9] *= np.float32(scale)
    if speck:
        sc.A = np.concatenate([sc.A, [0.5]]).astype(np.float32)
        sc.region = np.concatenate([sc.region, [0]]).astype(np.int32)
    sc.L = sc.L * np.float32(scale)
    return S.write(sc)


def _compare(scale):
    method = {m.name: m for m in M.timing_methods()}["v4-A2C suivi 1/4"]
    ctxs = []
    for speck in (False, True):
        c = N.Context()
        c.load_bytes(_room(scale, speck))
        c.build_states()
        c.begin(method, 0, 1)
        ctxs.append(c)
    times = ([], [])
    for _ in range(15):
        for c, t in zip(ctxs, times):
            c.sync()
            t0 = time.perf_counter()
            for _ in range(20):
                c.frame(0)
            c.sync()
            t.append(time.perf_counter() - t0)
    for c in ctxs:
        c.close()
    boxes, filt = (statistics.median(t) for t in times)
    assert boxes <= 1.2 * filt, (boxes, filt)


def test_rows_of_undecided_rays():
    """A room of 0.8 x 0.4 x 0.3: its points lie 2 mm apart, and whole rows of them beside the boxes' edges."""
    _compare(0.1)


def test_large_units():
    """A room of 800 x 400 x 300: the slabs' margin passes the 1e-3 that rays start off their surface."""
    _compare(100.0)
