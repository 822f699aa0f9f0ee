"""Which opaque content a context holds, whatever drew it: an opaque draw adds
to the current frame's (a replayed one's, a batch's), and starts anew where the
frame has none."""
import numpy as np
import pytest

import parity_util as pu
import vk_order_independent_transparency_gb300 as oit

pytestmark = pytest.mark.gpu

W, H = 75, 45


def meshes():
    """A scene, and a smaller one in front of it and beside it, to be drawn on top."""
    v, i, tpo, sd = pu.scene(24, W, H, seed=4, radius_min=0.1, radius_max=0.3)
    w, j, _, _ = pu.scene(5, W, H, seed=11, radius_min=0.1, radius_max=0.2)
    return oit.DeviceMesh(v, i), tpo, oit.DeviceMesh(w, j), sd


def renderer(sd, alg, aa, flags=0):
    r = oit.Renderer(oit.make_state(alg, W, H, oit_layers=4, nodes_per_pixel=40, aa_type=aa, flags=flags))
    r.update_scene(sd)
    return r


def targets(r):
    return r.read_buffer(oit.OIT_BUF_DEPTH), r.read_buffer(oit.OIT_BUF_OPAQUE_COLOR)


def staged_frame(r, mesh, opaque):
    r.begin_frame()
    r.clear_transparent()
    if opaque:
        r.draw_opaque(mesh, 0, mesh.num_triangles)
    r.draw_transparent_color(mesh, 0, 0)
    r.composite()


def expected(sd, alg, aa, mesh, tpo, percent, extra, count):
    """The targets of the frame and then the draw, in one plain context."""
    with renderer(sd, alg, aa) as r:
        if percent < 100:
            r.render_frame(mesh, tpo, percent)
        else:
            r.begin_frame()
        r.draw_opaque(extra, 0, count)
        return targets(r)


@pytest.mark.parametrize('aa', [oit.OIT_AA_NONE, oit.OIT_AA_MSAA_4X])
@pytest.mark.parametrize('percent', [60, 100])
@pytest.mark.parametrize('whole', [True, False])
def test_opaque_draw_after_a_replayed_frame(engine, aa, percent, whole):
    """A captured frame with and without opaque objects; between the capture
    and the replay a staged frame that has the opposite."""
    mesh, tpo, extra, sd = meshes()
    count = extra.num_triangles if whole else 0
    with renderer(sd, oit.OIT_SIMPLE, aa, oit.OIT_FLAG_CUDA_GRAPH) as r:
        r.render_frame(mesh, tpo, percent)
        staged_frame(r, mesh, opaque=percent == 100)
        r.render_frame(mesh, tpo, percent)
        r.draw_opaque(extra, 0, count)
        got = targets(r)
    for a, b in zip(got, expected(sd, oit.OIT_SIMPLE, aa, mesh, tpo, percent, extra, count)):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize('mode', [-1, 0, 1])
@pytest.mark.parametrize('replays', [0, 1])
def test_opaque_draw_after_a_batch(engine, mode, replays):
    mesh, tpo, extra, sd = meshes()
    algs = [oit.OIT_LINKEDLIST, oit.OIT_LOOP64]
    views = [(renderer(sd, alg, oit.OIT_AA_NONE), mesh, tpo, 60) for alg in algs]
    batch = oit.Batch(parallel_streams=2)
    batch.set_raster_mode(mode)
    batch.set_views(views)
    for _ in range(1 + replays):
        batch.render()
    for (r, *_), alg in zip(views, algs):
        r.draw_opaque(extra, 0, extra.num_triangles)
        for a, b in zip(targets(r), expected(sd, alg, oit.OIT_AA_NONE, mesh, tpo, 60, extra, extra.num_triangles)):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize('staged', [True, False])
@pytest.mark.parametrize('after', [0, 2])
def test_failed_opaque_draw_leaves_cleared_targets(engine, staged, after):
    """A frame (or an opaque draw) that fails for want of memory leaves no
    earlier frame's opaque content for the draws that follow it."""
    mesh, tpo, extra, sd = meshes()
    v, i, big_tpo, _ = pu.scene(400, W, H, seed=8)
    big = oit.DeviceMesh(v, i)
    with renderer(sd, oit.OIT_SIMPLE, oit.OIT_AA_NONE) as r:
        r.render_frame(mesh, tpo, 60)
        if staged:
            r.begin_frame()
            r.clear_transparent()
        oit.debug_fail_allocations(after)  # among the larger mesh's buffers
        try:
            with pytest.raises(oit.OitError) as e:
                if staged:
                    r.draw_opaque(big, 0, big.num_triangles)
                else:
                    r.render_frame(big, big_tpo, 0)
        finally:
            oit.debug_fail_allocations(-1)
        assert e.value.status == oit.OIT_ERR_OUT_OF_MEMORY
        depth, color = targets(r)
        assert depth.size == W * H and (depth == 0x3F800000).all()
        assert color.size == 4 * W * H and (color.view(np.float32) == np.float32(0.2)).all()
        r.clear_transparent()
        r.draw_transparent_color(extra, 0, extra.num_triangles)
        r.composite()
        image = r.output()
    with renderer(sd, oit.OIT_SIMPLE, oit.OIT_AA_NONE) as r:
        r.render_frame(extra, tpo, 100)
        np.testing.assert_array_equal(image, r.output())
