"""The error of a taa frame, summed by the last block of the update to arrive: one block, one more
than a round of the 256 runs, ragged last blocks, frame after frame, against FP64 sums over the
history and the references."""
import numpy as np
import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("points", [150, 256, 700, 65_536, 66_000, 140_001])
def test_taa_error_equals_the_sums(points):
    sc = S.box_room(points=points, seed=1)
    rng = np.random.default_rng(points)
    for s in sc.states:
        s.ref = rng.uniform(0.05, 1.0, sc.Np).astype(np.float32)
        s.valid = (rng.random(sc.Np) < 0.9).astype(np.uint8)
        s.Pw = np.zeros((sc.Np, s.inten.shape[0]), np.float32)
    ctx = N.Context()
    ctx.load_bytes(S.write(sc))
    ctx.taa_begin(0.1, 1.0, 0, 0, 5000)
    for f in range(5):
        e = ctx.taa_frame(0, want_err=f != 2)
        if f == 2:
            assert e is None
            continue
        on = sc.states[0].valid != 0
        ref = sc.states[0].ref[on]
        d = (ctx.taa_array(N.T_H)[on] - ref).astype(np.float64)
        want = np.sqrt((d * d).mean()) / ref.astype(np.float64).mean()
        assert e == pytest.approx(want, rel=1e-6), f   # the value is returned in FP32
    ctx.close()
