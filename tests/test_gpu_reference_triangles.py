"""Reference iterations of scenes with many dynamic triangles on the plane filter: the staged triangles and the
lanes' exchange rows together pass 48 KB of shared memory where neither does alone (and, for comparison,
below and above it): two iterations of both chains against sums over the frozen rays of the same seeds."""
import numpy as np
import pytest
from test_gpu_reference_lanes import _mix

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _panels(n, lights):
    """The room and n panels in it, the first one turned out of the axes; four points to a quad."""
    sc = S.box_room(points=600, seed=0, lights=lights)
    rng = np.random.default_rng(n)
    quads = list(S._room_quads())
    for k in range(n):
        o = rng.uniform((0.5, 0.5, 0.3), (7.0, 3.0, 2.5))
        quads.append((o, (0.2, 0.05 if k == 0 else 0.0, 0.0), (0.0, 0.0, 0.2), (0, 1, 0)))
    Q = np.array([[*o, *u, *v, *m] for o, u, v, m in quads], np.float32)
    T = np.concatenate([np.concatenate([np.concatenate([q[:3], q[3:9]]), np.concatenate([q[:3] + q[3:6] + q[6:9], -q[3:9]])]) for q in Q])
    cells = [(a, b) for b in (0.25, 0.75) for a in (0.25, 0.75)]
    P = np.array([q[:3] + np.float32(a) * q[3:6] + np.float32(b) * q[6:9] for q in Q for a, b in cells], np.float32)
    nq = len(Q)
    st = S.State(inten=sc.states[0].inten, P=P, N=np.repeat(Q[:, 9:], 4, axis=0), Q=Q, dims=np.full((nq, 2), 2, np.int32),
                 off=(4 * np.arange(nq)).astype(np.int32), T=T.reshape(-1, 9).astype(np.float32), TQ=np.repeat(np.arange(nq, dtype=np.int32), 2))
    A = rng.uniform(0.2, 0.9, 4 * nq).astype(np.float32)
    return S.Scene(NR=1, L=sc.L, A=A, region=np.zeros(4 * nq, np.int32), states=[st])


@pytest.mark.parametrize("panels,lights,K", [(60, 32, 9), (90, 32, 9), (250, 32, 8), (240, 16, 9), (300, 16, 9), (430, 16, 4), (420, 3, 9), (520, 3, 5)])
def test_reference_iterations_of_many_triangles(panels, lights, K):
    sc = _panels(panels, lights)
    ctx = N.Context()
    ctx.load_bytes(S.write(sc))
    ctx.build_reference(K=K, warmup=0, block=2, max_iter=2, noise_target=0.0)
    E = ctx.state_array(0, N.SA_EDIR).reshape(sc.Np, lights).astype(np.float64)
    got = ctx.state_array(0, N.SA_PW).reshape(sc.Np, lights)
    want = np.zeros((sc.Np, lights))
    for chain in range(2):
        L = np.zeros((sc.Np, lights))
        for it in range(2):
            ctx.adjoint(0, np.zeros(sc.Np, np.float32), K=K, seed=_mix(0x51 + 104729 * chain + 31 * it) & 0xFFFFFFFF, iterations=1)
            hits = ctx.adjoint_arrays()[2]
            nxt = np.zeros((sc.Np, lights))
            for r in range(K):
                h = hits[:, r]
                nxt += np.where((h >= 0)[:, None], sc.A[h][:, None].astype(np.float64) * (E[h] + L[h]), 0.0)
            L = nxt / K
            want += L / 4
    # FP32: K products and additions and a division in either iteration, the sums of two iterates and chains
    tol = 2 * (K + 6) * 2.0 ** -24
    assert np.all(np.abs(got - want) <= tol * np.abs(want) + 1e-30)
    assert want.any()
    ctx.close()
