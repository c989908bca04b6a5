"""Zone marks and voxel light marks at the places where their stepped samples cannot decide (on and
beside zone faces, degenerate and very long segments, small and far boxes), bit for bit against the
oracle, from 16-byte aligned vertex records and from records that are not."""
import numpy as np
import pytest
import torch

from oracle import pyhg
from render_engine_gb300 import hashgrid as H

pytestmark = pytest.mark.gpu

BOXES = {"room": ((0.0, 0.0, 0.0), (8.0, 4.0, 3.0)), "far": ((-421.3, 873.1, -7.7), (-11.9, 1201.3, 61.3)),
         "small": ((0.1, 0.2, 0.3), (0.11, 0.207, 0.3091)), "odd": ((-1.7, -0.3, 0.1), (5.9, 3.3, 2.7))}


def _coords(rng, lo, hi, n):
    """Points mostly on faces of the 6 x 4 x 4 zones or next to them, some anywhere, some far out."""
    lo, hi = np.array(lo), np.array(hi)
    p = rng.uniform(lo - 0.2 * (hi - lo), hi + 0.2 * (hi - lo), (n, 3))
    G = np.array([6, 4, 4])
    face = (lo + (hi - lo) * rng.integers(0, G + 1, (n, 3)) / G).astype(np.float32)
    off = rng.choice([0.0, 0.0, 1e-7, -1e-7, 1e-6, -1e-5, 1e-4, 1e-3], (n, 3)) * np.abs(hi - lo)
    p = np.where(rng.random((n, 3)) < 0.6, face + off, p).astype(np.float32)
    ulp = rng.integers(-2, 3, (n, 3))
    p = np.where(ulp > 0, np.nextafter(p, np.float32(np.inf)), np.where(ulp < 0, np.nextafter(p, np.float32(-np.inf)), p))
    far = rng.random(n) < 0.03
    p[far] += (rng.normal(size=(int(far.sum()), 3)) * 1e4 * (hi - lo)).astype(np.float32)
    return p.astype(np.float32)


def _vertices(rng, lo, hi, n):
    v = np.zeros(n, H.VERTEX_DTYPE)
    v["origin"], v["hit"] = _coords(rng, lo, hi, n), _coords(rng, lo, hi, n)
    same = rng.random((n, 3)) < 0.25                      # segments along an axis, or no segment at all
    v["hit"] = np.where(same, v["origin"], v["hit"])
    d = rng.normal(size=(n, 3))
    d[rng.random((n, 3)) < 0.2] = 0.0
    d[:, 0] += 1e-3
    v["dir"] = d / np.linalg.norm(d, axis=1, keepdims=True)
    t = np.roll(d, 1, axis=0)
    v["to_light"] = t / np.linalg.norm(t, axis=1, keepdims=True)
    v["light_dist"] = np.linalg.norm(np.array(hi) - np.array(lo)) * 10.0 ** rng.uniform(-3, 2, n)
    v["light_index"] = rng.integers(-1, 70, n)
    v["flags"] = np.where(rng.random(n) < 0.7, H.LIGHT_VISIBLE, 0) | np.where(rng.random(n) < 0.1, H.MISS, 0)
    return v


def _dev(v, aligned):
    raw = np.ascontiguousarray(v).view(np.uint8).reshape(-1)
    buf = torch.zeros(raw.size + 16, dtype=torch.uint8, device="cuda")
    at = 0 if aligned else 4
    buf[at:at + raw.size] = torch.from_numpy(raw).cuda()
    return buf, buf.data_ptr() + at


@pytest.mark.parametrize("aligned", [True, False])
@pytest.mark.parametrize("box", sorted(BOXES))
def test_marks_at_zone_faces(box, aligned):
    lo, hi = BOXES[box]
    rng = np.random.default_rng(len(box))
    cap, npaths, stride = 1 << 16, 20000, 3
    size = float(np.linalg.norm(np.array(hi) - np.array(lo)))
    cfg = H.make_config(zone_lo=lo, zone_hi=hi, capacity=cap, max_depth=4, tracing_distance=6.0 * size)
    v = _vertices(rng, lo, hi, npaths * stride)
    v["entry"] = np.arange(len(v)) % cap
    lens = rng.integers(0, stride + 1, npaths).astype(np.int32)
    hg, orc = H.HashGrid(cfg), pyhg.Cache(pyhg.config_from(cfg))
    hg.voxels_init(37)
    keep, ptr = _dev(v, aligned)
    dl = torch.from_numpy(lens).cuda()
    hg.mark_paths_strided(ptr, dl, stride, npaths)
    hg.voxels_mark(ptr, dl, stride, npaths)
    start = np.zeros(npaths + 1, np.int32)
    start[1:] = np.cumsum(lens)
    packed = v.reshape(npaths, stride)[np.arange(stride)[None, :] < lens[:, None]]
    orc.mark_paths(packed, start)
    assert np.array_equal(hg.download(H.A_BANK0), orc.bank0)
    assert np.array_equal(hg.voxels(), pyhg.voxels_mark(pyhg.config_from(cfg), 37, v, lens, stride))
    assert orc.bank0.any()
    hg.close()
    del keep
