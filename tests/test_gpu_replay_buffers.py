"""Captured frames after their context's buffers have moved: a larger draw, or
another batch over the same contexts, grows them between two replays."""
import numpy as np
import pytest

import parity_util as pu
import vk_order_independent_transparency_gb300 as oit

pytestmark = pytest.mark.gpu

W, H = 96, 64
KW = dict(oit_layers=8, nodes_per_pixel=60)


def scenes(alg, seed):
    """[(mesh, triangles per object, scene constants, image)] of a small and a large scene."""
    out = []
    for n in (12, 600):
        v, i, tpo, sd = pu.scene(n, W, H, seed=seed)
        out.append((oit.DeviceMesh(v, i), tpo, sd, pu.render_gpu(alg, W, H, v, i, tpo, sd, 100, **KW)['image']))
    return out


@pytest.mark.parametrize('alg', [oit.OIT_LINKEDLIST, oit.OIT_SPINLOCK])
def test_replay_after_a_larger_draw(engine, alg):
    (mesh, tpo, sd, ref), (large, _, _, large_ref) = scenes(alg, 3)
    with oit.Renderer(oit.make_state(alg, W, H, flags=oit.OIT_FLAG_CUDA_GRAPH, **KW)) as r:
        r.update_scene(sd)
        for _ in range(2):
            r.render_frame(mesh, tpo, 100)
            np.testing.assert_array_equal(r.output(), ref)
        r.begin_frame()
        r.clear_transparent()
        r.draw_transparent_color(large, 0, large.num_triangles)
        r.composite()
        np.testing.assert_array_equal(r.output(), large_ref)
        for _ in range(2):
            r.render_frame(mesh, tpo, 100)
            np.testing.assert_array_equal(r.output(), ref)
        assert r.get_error() == 0


def test_two_batches_over_the_same_contexts(engine):
    algs = [oit.OIT_LINKEDLIST, oit.OIT_LOOP64, oit.OIT_SIMPLE]
    sc = [scenes(alg, 20 + k) for k, alg in enumerate(algs)]
    renderers = [oit.Renderer(oit.make_state(alg, W, H, **KW)) for alg in algs]
    batches = []
    for size in (0, 1):
        b = oit.Batch(parallel_streams=2)
        b.set_views([(r, s[size][0], s[size][1], 100) for r, s in zip(renderers, sc)])
        batches.append(b)
    for r, s in zip(renderers, sc):
        r.update_scene(s[0][2])
    for size in (0, 0, 1, 1, 0, 0, 1):
        batches[size].render()
        for r, s in zip(renderers, sc):
            np.testing.assert_array_equal(r.output(), s[size][3])
            assert r.get_error() == 0


def test_batch_replay_after_a_resolve_of_other_views(engine):
    """The batched resolve's descriptors are those of its last call's views."""
    algs = [oit.OIT_LINKEDLIST, oit.OIT_LOOP64, oit.OIT_LINKEDLIST]
    cameras = [oit.make_camera(W, H, eye=(x, 0.0, 3.0)) for x in (0.0, 0.7, -0.7)]
    views, refs = [], []
    for k, alg in enumerate(algs):
        v, i, tpo, _ = pu.scene(20, W, H, seed=40 + k)
        refs.append([pu.render_gpu(alg, W, H, v, i, tpo, sd, 100, **KW)['image'] for sd in cameras])
        views.append((oit.Renderer(oit.make_state(alg, W, H, **KW)), oit.DeviceMesh(v, i), tpo, 100))
    batch = oit.Batch(parallel_streams=2)

    def render(which, camera):
        for k in which:
            views[k][0].update_scene(cameras[camera])
        batch.set_views([views[k] for k in which])
        batch.render()
        for k in which:
            np.testing.assert_array_equal(views[k][0].output(), refs[k][camera])

    def resolve(which, camera):
        for k in which:
            views[k][0].update_scene(cameras[camera])
            views[k][0].render_frame(*views[k][1:])
        batch.set_views([views[k] for k in which])
        batch.resolve()
        for k in which:
            np.testing.assert_array_equal(views[k][0].output(), refs[k][camera])

    render((0, 1), 0)
    render((0, 1), 1)
    resolve((2,), 0)
    render((0, 1), 2)
    render((0, 1), 0)
    resolve((0, 1, 2), 1)
    render((0, 1), 0)


def test_batch_with_a_context_made_anew(engine):
    """A destroyed context's successor, at the same address perhaps, is another view."""
    s = scenes(oit.OIT_LOOP64, 60)
    batch = oit.Batch(parallel_streams=2)
    for n in range(4):
        with oit.Renderer(oit.make_state(oit.OIT_LOOP64, W, H, **KW)) as r:
            r.update_scene(s[0][2])
            batch.set_views([(r, s[0][0], s[0][1], 100)])
            for _ in range(2):
                batch.render()
                np.testing.assert_array_equal(r.output(), s[0][3])


@pytest.mark.parametrize('own', [True, False])
def test_overflow_of_a_graph_captured_before_another(engine, own):
    """Bins that a captured frame's scene outgrows are re-sized by its next
    call, also when the context was captured for another batch since."""
    import torch
    alg = oit.OIT_LOOP64
    small, large = [oit.make_scene(200, seed=9, radius_min=a, radius_max=b) for a, b in ((0.01, 0.02), (0.2, 0.35))]
    sd = oit.make_camera(W, H)
    refs = [pu.render_gpu(alg, W, H, *s, sd, 100, **KW)['image'] for s in (small, large)]
    r = oit.Renderer(oit.make_state(alg, W, H, flags=oit.OIT_FLAG_CUDA_GRAPH, **KW))
    r.update_scene(sd)
    mesh, other = [oit.DeviceMesh(small[0], small[1]) for _ in range(2)]

    def batch(m):
        b = oit.Batch(parallel_streams=2)
        b.set_views([(r, m, small[2], 100)])
        return b

    first = None if own else batch(mesh)
    second = batch(other)

    def frame():
        if own:
            r.render_frame(mesh, small[2], 100)
        else:
            first.render()
        return r.output(), r.get_error()

    for _ in range(2):
        image, error = frame()
        np.testing.assert_array_equal(image, refs[0])
    second.render()
    mesh.vertices.copy_(torch.from_numpy(large[0]))  # the scene grows behind the same pointer
    errors = []
    for _ in range(3):
        image, error = frame()
        np.testing.assert_array_equal(image, refs[1])
        errors.append(error)
    assert errors == [oit.OIT_DEVERR_BIN_OVERFLOW, 0, 0]
