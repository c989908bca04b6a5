"""Reference iterations with several lanes to a point (few points) and with one (many points), light
counts on both sides of the lanes, ray counts that do not fill them: two iterations of both chains
against sums over the frozen rays of the same seeds."""
import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu
M64 = (1 << 64) - 1


def _mix(x):
    x ^= x >> 30
    x = x * 0xbf58476d1ce4e5b9 & M64
    x ^= x >> 27
    x = x * 0x94d049bb133111eb & M64
    return x ^ x >> 31


@pytest.mark.parametrize("points,lights,K", [(600, 1, 1), (600, 3, 7), (5000, 3, 32), (5000, 8, 8), (3001, 16, 13), (700, 32, 9), (700_000, 3, 5)])
def test_reference_iterations(points, lights, K):
    sc = S.box_room(points=points, seed=2, lights=lights)
    rng = np.random.default_rng(points)
    sc.A = rng.uniform(0.2, 0.9, sc.Np).astype(np.float32)
    ctx = N.Context()
    ctx.load_bytes(S.write(sc))
    ctx.build_reference(K=K, warmup=0, block=2, max_iter=2, noise_target=0.0)
    for state in (0, sc.NS - 1):
        E = ctx.state_array(state, N.SA_EDIR).reshape(sc.Np, lights).astype(np.float64)
        got = ctx.state_array(state, N.SA_PW).reshape(sc.Np, lights)
        want = np.zeros((sc.Np, lights))
        for chain in range(2):
            L = np.zeros((sc.Np, lights))
            for it in range(2):
                seed = _mix(0x51 + 7919 * state + 104729 * chain + 31 * it) & 0xFFFFFFFF
                ctx.adjoint(state, np.zeros(sc.Np, np.float32), K=K, seed=seed, iterations=1)
                hits = ctx.adjoint_arrays()[2]
                nxt = np.zeros((sc.Np, lights))
                for r in range(K):
                    h = hits[:, r]
                    nxt += np.where((h >= 0)[:, None], sc.A[h][:, None].astype(np.float64) * (E[h] + L[h]), 0.0)
                L = nxt / K
                want += L / 4
        # FP32: K products and additions and a division in either iteration, the sums of two iterates and chains
        tol = 2 * (K + 6) * 2.0 ** -24
        assert np.all(np.abs(got - want) <= tol * np.abs(want) + 1e-30), state
        assert want.any()
    ctx.close()
