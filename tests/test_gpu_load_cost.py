"""Loading a room with many boxes costs little more than loading one without: finding the boxes among the
triangles is host work that a caller waits for with every load.  (The allowance is half of a load; comparing
every pair of sides anew for every box took a load's time again.)"""
import statistics
import time

import pytest

from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


def test_many_boxes_load_like_few():
    data = [S.write(S.box_room(points=10_728, seed=3, boxes=b)) for b in (0, 9)]
    ctx = N.Context()
    times = ([], [])
    for _ in range(30):
        for d, t in zip(data, times):
            t0 = time.perf_counter()
            ctx.load_bytes(d)
            ctx.sync()
            t.append(time.perf_counter() - t0)
    few, many = (statistics.median(t[3:]) for t in times)
    assert many <= 1.5 * few, (few, many)
    ctx.close()
