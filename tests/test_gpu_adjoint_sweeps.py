"""rc_adjoint's sweeps bit for bit against the same FP32 sweeps in numpy, at a size where the sweeps
leave out what no longer changes: few sweeps (all full), many (most points copied), and past the fixed
point; K a multiple of four and not; the objective on few points and on all."""
import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("K,iterations,dense", [(32, 5, True), (32, 6, False), (32, 44, True), (33, 61, False), (32, 150, True)])
def test_sweeps_equal_plain_sweeps(K, iterations, dense):
    sc = S.box_room(points=70_000, seed=3)
    data = S.write(sc)
    ctx = N.Context()
    info = ctx.load_bytes(data)
    n = info["np"]
    assert n * K >= 1 << 21   # followed
    rng = np.random.default_rng(K)
    w = rng.uniform(0.5, 1.5, n).astype(np.float32) / np.float32(n)
    if not dense:
        w[rng.random(n) < 0.95] = 0.0
    g_out, res = ctx.adjoint(0, w, K=K, seed=7, iterations=iterations)
    L, u, hits = ctx.adjoint_arrays()
    E = ctx.state_array(0, N.SA_EDIR).reshape(n, info["nl"])
    A = sc.A.astype(np.float32)
    d = np.zeros(n, np.float32)
    for l in range(info["nl"]):
        d += E[:, l]
    ok = hits >= 0
    flat = hits.reshape(-1)
    keep = np.flatnonzero(flat >= 0)
    target, source = flat[keep], (keep // K).astype(np.int64)
    wL, wu = np.zeros(n, np.float32), w.copy()
    for _ in range(iterations):
        g = A * (d + wL)
        s = np.zeros(n, np.float32)
        for r in range(K):
            s += np.where(ok[:, r], g[hits[:, r]], np.float32(0))
        wL = s / np.float32(K)
        t = np.zeros(n, np.float32)
        np.add.at(t, target, wu[source])   # in ray order, one rounding each
        wu = w + A * t / np.float32(K)
    assert np.array_equal(L.view(np.uint32), wL.view(np.uint32))
    assert np.array_equal(u.view(np.uint32), wu.view(np.uint32))
    J = float((w.astype(np.float64) * wL.astype(np.float64)).sum())
    assert abs(res["J"] - J) <= 1e-12 * abs(J) and abs(res["J_grad"] - J) <= 1e-4 * abs(J) + (0 if iterations > 20 else abs(J))
    assert res["max_incoming"] == int(np.bincount(target, minlength=n).max())
    ctx.close()
