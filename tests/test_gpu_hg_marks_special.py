"""Zone marks and voxel light marks of vertices with infinities, NaN, zeros of both signs, denormal and very
large numbers among their coordinates and directions, bit for bit against the oracle."""
import numpy as np
import pytest
import torch
from test_gpu_hg_marks import BOXES, _dev, _vertices

from oracle import pyhg
from render_engine_gb300 import hashgrid as H

pytestmark = pytest.mark.gpu
FINITE = [1e30, -1e30, 1e-38, 0.0, -0.0, 3e38, 1e-45, 1e10]


@pytest.mark.parametrize("special", [FINITE, FINITE + [np.inf, -np.inf, np.nan]])
@pytest.mark.parametrize("box", sorted(BOXES))
def test_marks_of_special_values(box, special):
    lo, hi = BOXES[box]
    rng = np.random.default_rng(len(box) + len(special))
    cap, npaths, stride = 1 << 16, 30000, 3
    size = float(np.linalg.norm(np.array(hi) - np.array(lo)))
    cfg = H.make_config(zone_lo=lo, zone_hi=hi, capacity=cap, max_depth=4, tracing_distance=6.0 * size)
    v = _vertices(rng, lo, hi, npaths * stride)
    for f in ("origin", "hit", "dir", "to_light"):
        v[f] = np.where(rng.random(v[f].shape) < 0.01, rng.choice(np.array(special, np.float32), v[f].shape), v[f])
    v["light_dist"] = np.where(rng.random(len(v)) < 0.05, np.inf, v["light_dist"])
    v["entry"] = np.arange(len(v)) % cap
    lens = rng.integers(0, stride + 1, npaths).astype(np.int32)
    hg, orc = H.HashGrid(cfg), pyhg.Cache(pyhg.config_from(cfg))
    keep, ptr = _dev(v, True)
    hg.mark_paths_strided(ptr, torch.from_numpy(lens).cuda(), stride, npaths)
    start = np.zeros(npaths + 1, np.int32)
    start[1:] = np.cumsum(lens)
    packed = v.reshape(npaths, stride)[np.arange(stride)[None, :] < lens[:, None]]
    orc.mark_paths(packed, start)
    got, want = hg.download(H.A_BANK0), orc.bank0
    assert np.array_equal(got, want), int((got != want).sum())
    assert want.any()
    hg.close()
    del keep
