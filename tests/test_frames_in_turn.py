"""Frames of several objects in a row on one canvas, with and without overlap:
sizes of each build of the frame kernel (below 400,000 pixels, from there to
two million, above), one view again and again and views in turn. A pixel that
the frame before still holds stays parked; every state is byte for byte that
of frames run one after the other."""
import numpy as np
import pytest

from test_frame_overlap import _canvas, _same


def _scene(ctx, n_obj):
    from j3d_gb300 import Mesh, Scene, workloads as W
    rng = np.random.default_rng(n_obj)
    meshes = [Mesh(ctx, *W.icosphere(level)) for level in (1, 3, 5)]
    sc = Scene()
    for k in range(n_obj):
        cs = np.eye(4, dtype=np.float32)
        cs[3, :3] = rng.uniform(-1.5, 1.5, size=3)
        sc.add_object(meshes[k % 3], cs.reshape(16), k + 1)
    sc.prepare_scene()
    sc.unzoom()
    return sc


@pytest.mark.gpu
@pytest.mark.parametrize("n_obj", [2, 24])
@pytest.mark.parametrize("w,h", [(5, 3), (64, 48), (633, 631), (637, 640), (1504, 1333)])
def test_rows_of_frames_equal_serial(gpu_ctx, n_obj, w, h):
    from j3d_gb300 import Matcap, workloads as W
    sc = _scene(gpu_ctx, n_obj)
    mc = Matcap.make(gpu_ctx, 0)
    views = W.cameras(3, W.SEED_BASE + n_obj, 3.0, 6.0)
    states = []
    try:
        for on in (True, False):
            gpu_ctx.set_frame_overlap(on)
            cv = _canvas(gpu_ctx, w, h)
            got = []
            for row in ([0] * 8, [0, 1, 2] * 4):
                for k in row:
                    sc.set_pose(views[k])
                    cv.render_frame(sc, mc)
                got.append((cv.get_pixels().copy(), cv.get_image().copy()))
            states.append(got)
            cv.close()
    finally:
        gpu_ctx.set_frame_overlap(True)
    assert gpu_ctx.device_status() == 0
    for row, (a, b) in enumerate(zip(*states)):
        _same(a, b, f"{n_obj} objects, {w}x{h}, row {row}")
    assert (states[0][0][0]["object_id"] != 0xffffffff).any()


@pytest.mark.gpu
def test_wait_runs_out(gpu_ctx):
    """A frame of several objects told to wait for a frame that no one wrote:
    its waits run out, the status says so, and the canvas goes on."""
    from j3d_gb300 import J3dgError, Matcap, workloads as W
    sc = _scene(gpu_ctx, 24)
    mc = Matcap.make(gpu_ctx, 0)
    sc.set_pose(W.cameras(1, W.SEED_BASE + 5, 3.0, 6.0)[0])
    cv, ref = _canvas(gpu_ctx, 200, 150), _canvas(gpu_ctx, 200, 150)
    for c in (cv, ref):
        c.render_frame(sc, mc)
        c.get_pixels()
    cv.expect_frame(0x7EADBEEF)
    cv.render_frame(sc, mc)
    with pytest.raises(J3dgError) as e:
        cv.get_pixels()
    assert "16 frame wait timeout" in str(e.value)
    assert gpu_ctx.device_status() == 0
    for c in (cv, ref):
        c.render_frame(sc, mc)
    _same((cv.get_pixels(), cv.get_image()), (ref.get_pixels(), ref.get_image()), "after the timeout")
