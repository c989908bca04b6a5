"""An adjoint whose objective starts on few points keeps its full sweeps, one launch an iteration, while the
changes still spread and where recomputing the touched points would not pay; once the iterates rest, nothing
is launched for them until the last sweep."""
import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


def test_spreading_changes_keep_full_sweeps():
    ctx = N.Context()
    n = ctx.load_bytes(S.write(S.box_room(points=270_000, seed=3)))["np"]
    assert 8 * n >= 1 << 21   # followed
    w = np.zeros(n, np.float32)
    w[:512] = 1.0 / 512
    ctx.build_states()
    ctx.adjoint(0, w, K=8, seed=1, iterations=4)

    def launches(iterations):
        before = ctx.stats()["launches"]
        ctx.adjoint(0, w, K=8, seed=1, iterations=iterations)
        return ctx.stats()["launches"] - before

    base = launches(4)
    assert launches(8) == base + 4
    assert launches(14) == base + 10
    assert launches(400) < base + 200
    ctx.close()
