"""Zone masks and voxel light marks of a pass of camera paths, which take one launch: a single
path, one less and one more than a block of paths, an odd image, no bounce and many, bit for bit against
the oracle's marks of the GPU's own vertices; and the zone masks alone, without voxel masks."""
import numpy as np
import pytest
import torch

from oracle import pyhg
from render_engine_gb300 import hashgrid as H
from render_engine_gb300 import native as N
from render_engine_gb300 import scene as S

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("width,height,bounces,res", [(1, 1, 2, 16), (17, 15, 1, 16), (257, 1, 0, 16), (61, 37, 5, 16), (64, 48, 2, 37), (61, 37, 2, 0)])
def test_marks_of_camera_paths(width, height, bounces, res):
    ctx = N.Context()
    ctx.load_bytes(S.write(S.box_room(points=2000, seed=3)))
    cfg = H.make_config(zone_lo=(0, 0, 0), zone_hi=(8, 4, 3), cell=0.1, capacity=1 << 18, max_depth=4, tracing_distance=50.0)
    hg = H.HashGrid(cfg)
    if res:
        hg.voxels_init(res)
    hg.begin_frame(0, 16)
    cam = N.camera((0.6, 0.5, 1.6), (6.0, 3.0, 1.0), width=width, height=height, fov_y_deg=75.0)
    img = torch.zeros(width * height * 3, device="cuda")
    hg.camera_paths(ctx, 0, H.path_params(cam, bounces=bounces, seed=9, frame=3), img)
    torch.cuda.synchronize()
    a = H.camera_arrays(ctx)
    ln, S1 = a["len"], a["stride"]
    oc = pyhg.Cache(pyhg.config_from(cfg))
    oc.keys[:] = hg.download(H.A_KEYS)
    verts = np.concatenate([a["vertices"][p * S1: p * S1 + ln[p]] for p in range(len(ln))])
    oc.mark_paths(verts, np.concatenate([[0], np.cumsum(ln)]).astype(np.int32))
    assert np.array_equal(hg.download(H.A_BANK0), oc.bank0)
    assert oc.bank0.any()
    if res:
        assert np.array_equal(hg.voxels(), pyhg.voxels_mark(pyhg.config_from(cfg), res, a["vertices"], ln, S1))
    hg.close()
    ctx.close()
