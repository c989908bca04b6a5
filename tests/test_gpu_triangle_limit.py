"""The largest number of dynamic triangles that shared memory holds (48 bytes a triangle, 4 more outside any
plane group, 72 a group, 200 KB in all): a scene just below it loads, traces like the full scan and runs
frames; one above it is refused."""
import numpy as np
import pytest

from render_engine_gb300 import methods as M
from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _scene(loose):
    """The room and a quad whose `loose` triangles are turned out of the axes."""
    sc = S.box_room(points=600, seed=0)
    quads = list(S._room_quads()) + [((3.0, 1.0, 1.0), (1.0, 0.2, 0.0), (0.0, 0.1, 1.0), (0, 1, 0))]
    Q = np.array([[*o, *u, *v, *n] for o, u, v, n in quads], np.float32)
    T = [np.concatenate([np.concatenate([q[:3], q[3:9]]), np.concatenate([q[:3] + q[3:6] + q[6:9], -q[3:9]])]) for q in Q[:6]]
    rng = np.random.default_rng(loose)
    free = np.concatenate([rng.uniform((0.5, 0.5, 0.3), (7.0, 3.5, 2.6), (loose, 3)), rng.uniform(0.02, 0.2, (loose, 6))], axis=1)
    T = np.concatenate([np.array(T).reshape(-1, 9), free]).astype(np.float32)
    TQ = np.concatenate([np.repeat(np.arange(6), 2), np.full(loose, 6)]).astype(np.int32)
    P = np.array([q[:3] + np.float32(a) * q[3:6] + np.float32(b) * q[6:9] for q in Q for b in (0.25, 0.75) for a in (0.25, 0.75)], np.float32)
    st = S.State(inten=sc.states[0].inten, P=P, N=np.repeat(Q[:, 9:], 4, axis=0), Q=Q, dims=np.full((7, 2), 2, np.int32),
                 off=(4 * np.arange(7)).astype(np.int32), T=T, TQ=TQ)
    return S.write(S.Scene(NR=1, L=sc.L, A=np.full(28, 0.5, np.float32), region=np.zeros(28, np.int32), states=[st]))


def test_largest_scene():
    most = (200 * 1024 - 16 - 6 * 72 - 12 * 48) // 52
    data = _scene(most)
    fast, full = N.Context(), N.Context(flags=N.FLAG_BRUTE_FORCE)
    fast.load_bytes(data)
    full.load_bytes(data)
    rng = np.random.default_rng(1)
    d = rng.normal(size=(20_000, 3))
    rays = np.concatenate([rng.uniform((0.1, 0.1, 0.1), (7.9, 3.9, 2.9), (20_000, 3)), d], axis=1).astype(np.float32)
    (p0, t0), (p1, t1) = fast.trace_rays(0, rays), full.trace_rays(0, rays)
    np.testing.assert_array_equal(p0, p1)
    np.testing.assert_array_equal(t0.view(np.uint32), t1.view(np.uint32))
    assert (p1 == 6).any()
    method = {m.name: m for m in M.timing_methods()}["Classique 1.0x"]
    out = []
    for ctx in (fast, full):
        ctx.begin(method, 0, 1)
        for _ in range(3):
            ctx.frame(0)
        out.append(ctx.array(N.A_LC))
    np.testing.assert_array_equal(out[0], out[1])
    assert np.isfinite(out[0]).all() and out[0].any()
    with pytest.raises(N.RCError):
        fast.load_bytes(_scene(most + 1))
    fast.close()
    full.close()
