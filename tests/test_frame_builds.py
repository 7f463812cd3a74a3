"""Frames of one object on both sides of the sizes where the frame kernel's
build changes (400,000 pixels, 700,000 at width 8, two million, or three for
one of 400,000 triangles and more that follows none on its canvas): its record
comes by value there, the batch kernel reads the same scene from a table, and
the frames are equal byte for byte."""
import numpy as np
import pytest

from test_frame_overlap import _canvas, _same


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("w,h", [(3, 2), (632, 624), (640, 632), (832, 836), (840, 840), (1504, 1328), (1504, 1336), (2000, 1496),
                                 (2000, 1504)])
def test_frames_equal_a_batch_of_one(gpu_ctx, width, w, h):
    _compare(gpu_ctx, (300, 150), width, w, h)


@pytest.mark.gpu
@pytest.mark.parametrize("width", [2, 4, 8])
@pytest.mark.parametrize("w,h", [(640, 632), (1504, 1336), (2000, 1496), (2000, 1504)])
def test_frames_of_a_larger_mesh(gpu_ctx, width, w, h):
    _compare(gpu_ctx, (640, 320), width, w, h)


def _compare(gpu_ctx, grid, width, w, h):
    from j3d_gb300 import Matcap, Mesh, Scene, render_batch, workloads as W
    sc = Scene()
    sc.add_object(Mesh(gpu_ctx, *W.torus(*grid), width=width), db_id=1)
    sc.prepare_scene()
    sc.unzoom()
    mc = Matcap.make(gpu_ctx, 0)
    frame, batch = _canvas(gpu_ctx, w, h), _canvas(gpu_ctx, w, h)
    for pose in W.cameras(3, W.SEED_BASE + 9, 2.5, 4.0):  # the first follows none
        sc.set_pose(pose)
        frame.render_frame(sc, mc)
    for pose in W.cameras(3, W.SEED_BASE + 9, 2.5, 4.0):
        sc.set_pose(pose)
        render_batch(gpu_ctx, [(batch, sc, mc)])
    got = (frame.get_pixels(), frame.get_image())
    _same(got, (batch.get_pixels(), batch.get_image()), f"width {width}, {w}x{h}")
    assert (got[0]["object_id"] != 0xffffffff).any() or w < 10
    assert gpu_ctx.device_status() == 0
    frame.close()
    batch.close()
