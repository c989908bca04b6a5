"""The public count of kernels launched (rc_run_stats.launches) follows the launches that a call makes."""
import numpy as np
import pytest

from render_engine_gb300 import hashgrid as H
from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


def _launches(ctx, call):
    before = ctx.stats()["launches"]
    call()
    return ctx.stats()["launches"] - before


def test_adjoint_launches():
    """Small problems run both sweeps of an iteration in one launch: beside them the frozen rays, the transposed
    lists (3 kernels, and the offsets' scan in 2048s: 1 kernel, or 3 over several blocks), the start of the
    iterates and the gradient's two, and in a state's first call its direct light at unit emission."""
    for points, scan in ((900, 1), (5000, 3)):
        ctx = N.Context()
        n = ctx.load_bytes(S.write(S.box_room(points=points, seed=2)))["np"]
        assert (n + 1 <= 2048) == (scan == 1)
        w = np.full(n, 1.0 / n, np.float32)
        ctx.build_states()
        first = _launches(ctx, lambda: ctx.adjoint(0, w, K=4, iterations=10))
        assert first == 1 + 1 + 3 + scan + 1 + 2 + 10
        assert _launches(ctx, lambda: ctx.adjoint(0, w, K=4, iterations=10)) == first - 1
        assert _launches(ctx, lambda: ctx.adjoint(0, w, K=4, iterations=23)) == first - 1 + 13
        ctx.close()


@pytest.mark.parametrize("voxels", [False, True])
def test_camera_path_launches(voxels):
    """A pass of camera paths: the paths, the insertion, the samples' sums and the marks."""
    ctx = N.Context()
    ctx.load_bytes(S.write(S.box_room(points=2000, seed=2)))
    ctx.build_states()
    hg = H.HashGrid(H.make_config(cell=0.1, capacity=1 << 14, max_depth=4, tracing_distance=50.0))
    if voxels:
        hg.voxels_init(32)
    hg.begin_frame(0, 16)
    cam = N.camera((0.6, 0.6, 1.6), (6.0, 3.0, 1.0), width=64, height=48)
    assert _launches(ctx, lambda: hg.camera_paths(ctx, 0, H.path_params(cam, bounces=2))) == 4
    hg.close()
    ctx.close()
