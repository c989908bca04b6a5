"""A rejected rc_adjoint call (an emission that is not finite) leaves the context as it was: the last
call's arrays can still be read, and the next valid call gives what it gives on a context that never saw
the rejected one.  Rejected: the first call of all, one that asks for more iterations than any before, one
with another K, one right after a scene was loaded again."""
import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points,K", [(700, 3), (70_000, 32)])   # plain sweeps; sweeps whose counts are followed
def test_rejected_call_leaves_the_context_usable(points, K):
    data = S.write(S.box_room(points=points, seed=6))
    ctx, other = N.Context(), N.Context()
    info = ctx.load_bytes(data)
    other.load_bytes(data)
    rng = np.random.default_rng(points)
    w = rng.uniform(0.0, 1.0, info["np"]).astype(np.float32) / np.float32(info["np"])
    bad = np.full(info["nl"], 2.0, np.float32)
    bad[-1] = np.nan

    def reject(**kw):
        with pytest.raises(N.RCError) as e:
            ctx.adjoint(0, w, emission=bad, **kw)
        assert "emission" in str(e.value)

    def same(**kw):
        g, r = ctx.adjoint(0, w, **kw)
        g2, r2 = other.adjoint(0, w, **kw)
        np.testing.assert_array_equal(g, g2)
        assert r == r2
        for a, b in zip(ctx.adjoint_arrays(), other.adjoint_arrays()):
            np.testing.assert_array_equal(a, b)

    reject(K=K, iterations=8)
    with pytest.raises(N.RCError):
        ctx._adj_k = K
        ctx.adjoint_arrays()
    same(K=K, iterations=8)
    kept = ctx.adjoint_arrays()
    reject(K=K, iterations=300)     # more iterations than the buffers hold
    for a, b in zip(kept, ctx.adjoint_arrays()):
        np.testing.assert_array_equal(a, b)
    same(K=K, iterations=8)
    reject(K=K + 2, iterations=8)
    same(K=K, iterations=70)
    same(K=K + 2, iterations=8)
    ctx.load_bytes(data)
    reject(K=K, iterations=8)
    same(K=K, iterations=8)
    ctx.close()
    other.close()
