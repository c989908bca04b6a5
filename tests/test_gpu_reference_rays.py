"""The rays of a reference iteration are the frozen rays of the same seed, every one: 43 k points, 32 rays, four
iterations of both chains, among them rays through edges and diagonals that the box slabs leave to the exact
test.  One ray with another hit moves its point's value by 1e-3 of it, the arithmetic by less than 1e-5."""
import numpy as np
import pytest
from test_gpu_reference_lanes import _mix

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [43_000, 90_000])   # eight lanes to a point, and one
def test_reference_rays_are_the_frozen_rays(points):
    K, iterations, lights = 32, 4, 3
    sc = S.box_room(points=points, seed=points % 1009, lights=lights)
    ctx = N.Context()
    ctx.load_bytes(S.write(sc))
    ctx.build_reference(K=K, warmup=0, block=iterations, max_iter=iterations, noise_target=0.0)
    A = sc.A.astype(np.float64)
    for state in (1, 2):
        E = ctx.state_array(state, N.SA_EDIR).reshape(sc.Np, lights).astype(np.float64)
        got = ctx.state_array(state, N.SA_PW).reshape(sc.Np, lights)
        want = np.zeros((sc.Np, lights))
        for chain in range(2):
            L = np.zeros((sc.Np, lights))
            for it in range(iterations):
                seed = _mix(0x51 + 7919 * state + 104729 * chain + 31 * it) & 0xFFFFFFFF
                ctx.adjoint(state, np.zeros(sc.Np, np.float32), K=K, seed=seed, iterations=1)
                hits = ctx.adjoint_arrays()[2]
                nxt = np.zeros((sc.Np, lights))
                for r in range(K):
                    h = hits[:, r]
                    nxt += np.where((h >= 0)[:, None], A[h][:, None] * (E[h] + L[h]), 0.0)
                L = nxt / K
                want += L / (2 * iterations)
        # FP32: K products and additions and a division in each iteration, the sums of the iterates and chains
        tol = iterations * (K + 6) * 2.0 ** -24
        wrong = np.nonzero((np.abs(got - want) > tol * np.abs(want) + 1e-30).any(axis=1))[0]
        assert len(wrong) == 0, (state, wrong, got[wrong], want[wrong])
    ctx.close()
