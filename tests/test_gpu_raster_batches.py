"""The tile raster's batch edges: a warp processes the triangles that touch its
pixels 32 at a time and queues their fragments 64 (with several samples a
lane, 96) at a time, so stacks of triangles around those counts, over frames
that end inside a tile, a micro-tile and a pixel group, against the oracle.
Small triangles and ones wider than 64 pixels (whose edge functions need 64
bits) alternate."""
import numpy as np
import pytest

import parity_util as pu
import vk_order_independent_transparency_gb300 as oit

pytestmark = pytest.mark.gpu


def stack(n, W, H, seed, large):
    """n triangles in clip space, from a pixel up to the frame's size (large:
    every third one reaches far beyond it)."""
    rng = np.random.default_rng(seed)
    v = np.zeros((n, 3, 10), np.float32)
    centre = rng.uniform(-0.8, 0.8, (n, 1, 2))
    size = rng.uniform(1.0, 8.0, (n, 1, 1)) * 2.0 / np.array([W, H])
    if large:
        size[::3] = 6.0 + 200.0 / np.array([W, H])
    v[:, :, :2] = centre + size * rng.uniform(-1.0, 1.0, (n, 3, 2))
    v[:, :, 2] = rng.uniform(0.05, 0.95, (n, 3))
    v[:, :, 3:6] = rng.normal(size=(n, 3, 3))
    v[:, :, 6:] = rng.random((n, 1, 4))
    return v.reshape(-1, 10), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)


def scene_data():
    sd = oit.OitSceneData()
    for j in range(4):
        sd.proj_view_matrix[5 * j] = 1.0
        sd.view_matrix[5 * j] = 1.0
    return sd


@pytest.mark.parametrize('n,W,H,percent', [(1, 8, 4, 100), (31, 9, 5, 100), (32, 17, 16, 100), (33, 7, 3, 60),
                                           (64, 16, 17, 100), (65, 33, 21, 50), (161, 24, 9, 75)])
@pytest.mark.parametrize('aa', [oit.OIT_AA_NONE, oit.OIT_AA_MSAA_8X, oit.OIT_AA_SSAA_4X])
@pytest.mark.parametrize('alg', range(7))
def test_stacked_triangles(engine, alg, aa, n, W, H, percent):
    L = 4
    v, i = stack(n, W, H, 7 * n + W, large=n % 2 == 1)
    kw = dict(oit_layers=L, nodes_per_pixel=200, aa_type=aa, weighted_precision=oit.OIT_WEIGHTED_FP32)
    g = pu.render_gpu(alg, W, H, v, i, 1, scene_data(), percent, **kw)
    o = pu.render_oracle(alg, W, H, v, i, 1, scene_data(), percent, **kw)
    pu.check_pair(alg, g, o, W, H, L, aa)


@pytest.mark.parametrize('aa', [oit.OIT_AA_NONE, oit.OIT_AA_MSAA_4X])
@pytest.mark.parametrize('cuts', [(0, 90), (0, 1, 90), (0, 0, 45, 90), (0, 90, 90)])
def test_opaque_draws_accumulate(engine, aa, cuts):
    """Opaque draws one after the other (the first one clears, an empty one
    only clears) leave what one draw of all triangles leaves."""
    W, H = 37, 19
    v, i = stack(90, W, H, 5, large=True)
    mesh = oit.DeviceMesh(v, i)

    def targets(bounds):
        with oit.Renderer(oit.make_state(oit.OIT_SIMPLE, W, H, aa_type=aa)) as r:
            r.update_scene(scene_data())
            for _ in range(2):  # the second frame finds the first one's targets
                r.begin_frame()
                r.clear_transparent()
                for a, b in zip(bounds, bounds[1:]):
                    r.draw_opaque(mesh, a, b - a)
                r.draw_transparent_color(mesh, 0, 0)
                r.composite()
            return r.read_buffer(oit.OIT_BUF_DEPTH), r.read_buffer(oit.OIT_BUF_OPAQUE_COLOR), r.output()

    for a, b in zip(targets(cuts), targets((0, 90))):
        np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize('W,H', [(257, 131), (33, 200)])
@pytest.mark.parametrize('alg', [oit.OIT_SIMPLE, oit.OIT_LINKEDLIST, oit.OIT_LOOP64])
def test_many_small_triangles(engine, alg, W, H):
    """Draws large enough for the setup to test micro-tiles (65536 triangles):
    slivers, triangles from a fraction of a pixel to several tiles, some over
    the frame's edge, some split by the near plane, a quarter opaque."""
    n, L = 66000, 8
    rng = np.random.default_rng(W)
    v = np.zeros((n, 3, 10), np.float32)
    centre = rng.uniform(-1.05, 1.05, (n, 1, 2))
    size = np.exp(rng.uniform(np.log(0.2), np.log(12.0), (n, 1, 1))) * 2.0 / np.array([W, H])
    size[::500] *= 5.0
    offset = rng.uniform(-1.0, 1.0, (n, 3, 2))
    offset[::3, 2] = offset[::3, 1] + 0.1 * rng.uniform(-1.0, 1.0, (len(offset[::3]), 2))  # slivers
    v[:, :, :2] = centre + size * offset
    v[:, :, 2] = rng.uniform(0.05, 0.95, (n, 3))
    v[::50, 0, 2] = -0.3  # across the near plane
    v[:, :, 3:6] = rng.normal(size=(n, 3, 3))
    v[:, :, 6:] = rng.random((n, 1, 4))
    v, i = v.reshape(-1, 10), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    kw = dict(oit_layers=L, nodes_per_pixel=200)
    g = pu.render_gpu(alg, W, H, v, i, 1, scene_data(), 75, **kw)
    o = pu.render_oracle(alg, W, H, v, i, 1, scene_data(), 75, **kw)
    pu.check_pair(alg, g, o, W, H, L)


@pytest.mark.parametrize('tail', [True, False])
@pytest.mark.parametrize('L', [1, 2, 16, 32])
@pytest.mark.parametrize('aa', [oit.OIT_AA_NONE, oit.OIT_AA_MSAA_4X, oit.OIT_AA_SSAA_8X])
def test_loop_second_pass(engine, aa, L, tail):
    """Loop32 walks a list a second time only where a pixel dropped a fragment:
    buffers that overflow everywhere, here and there, and nowhere, with equal
    depths among the triangles."""
    n, W, H = 120, 21, 13
    v, i = stack(n, W, H, L, large=True)
    v = v.reshape(n, 3, 10)
    v[1::4, :, 2] = 0.5   # equal depths, within and across the kept ones
    v[3::8, :, 2] = 0.05
    v = v.reshape(-1, 10)
    kw = dict(oit_layers=L, aa_type=aa, tail_blend=tail)
    g = pu.render_gpu(oit.OIT_LOOP, W, H, v, i, 1, scene_data(), 80, **kw)
    o = pu.render_oracle(oit.OIT_LOOP, W, H, v, i, 1, scene_data(), 80, **kw)
    pu.check_pair(oit.OIT_LOOP, g, o, W, H, L, aa)


@pytest.mark.parametrize('n', [12, 24, 1200])
def test_sort_chunks(engine, n):
    """Slivers across the frame, each in thousands of tiles: pairs on both
    sides of the line (65536) from which a frame's sort sums its chunks' counts
    in a launch of their own, and more chunks than one round of it takes."""
    W = H = 1024
    L = 8
    rng = np.random.default_rng(n)
    v = np.zeros((n, 3, 10), np.float32)
    at = rng.uniform(0.9, 0.99, (n, 2))
    sign = rng.choice([-1.0, 1.0], n)
    v[:, 0, 0], v[:, 0, 1] = -at[:, 0], -at[:, 1] * sign
    v[:, 1, 0], v[:, 1, 1] = at[:, 1], at[:, 0] * sign
    v[:, 2] = v[:, 1]
    v[:, 2, 0] += rng.uniform(0.001, 0.003, n)
    v[:, :, 2] = rng.uniform(0.05, 0.95, (n, 3))
    v[:, :, 3:6] = rng.normal(size=(n, 3, 3))
    v[:, :, 6:] = rng.random((n, 1, 4))
    v, i = v.reshape(-1, 10), np.arange(3 * n, dtype=np.uint32).reshape(-1, 3)
    kw = dict(oit_layers=L, nodes_per_pixel=8)
    g = pu.render_gpu(oit.OIT_LOOP64, W, H, v, i, 1, scene_data(), 100, **kw)
    o = pu.render_oracle(oit.OIT_LOOP64, W, H, v, i, 1, scene_data(), 100, **kw)
    pu.check_pair(oit.OIT_LOOP64, g, o, W, H, L)


@pytest.mark.parametrize('aa', [oit.OIT_AA_NONE, oit.OIT_AA_MSAA_4X, oit.OIT_AA_MSAA_8X, oit.OIT_AA_SSAA_8X])
@pytest.mark.parametrize('alg', [oit.OIT_LINKEDLIST, oit.OIT_SPINLOCK, oit.OIT_WEIGHTED])
@pytest.mark.parametrize('W,H', [(128, 96), (101, 83)])
def test_large_triangles(engine, alg, aa, W, H):
    """Triangles wider than 64 pixels: quads whose edges run along pixel and
    micro-tile borders, through pixel centres and just beside them, slivers
    across the frame, the same quad twice (the first one stays), half of them
    opaque, with small ones between them."""
    n, L = 48, 8
    rng = np.random.default_rng(W)
    v = np.zeros((n, 2, 3, 10), np.float32)
    corner = np.array([[0, 0], [1, 0], [1, 1], [0, 1]])
    for k in range(n):
        if k % 8 == 7:  # small
            at, size = rng.uniform(0, 1, 2) * (W, H), rng.uniform(1, 12, 2)
        else:
            size = rng.choice([8, 4, 1, 0.5, 1 / 256]) * rng.integers(-3, 4, 2) + (W, H) - rng.integers(0, 24, 2)
            at = np.floor(rng.uniform(-16, 24, 2)) + rng.choice([0.0, 0.5, 0.5 + 1 / 256, 3 / 16])
        quad = at + corner * size
        if k % 5 == 4:
            quad[2] = quad[0] + rng.uniform(-1, 1, 2)  # a sliver and its back
        z = rng.uniform(0.05, 0.95, 4)
        v[k, :, :, :2] = (quad / (W, H) * 2 - 1)[[[0, 1, 2], [0, 2, 3]]]
        v[k, :, :, 2] = z[[[0, 1, 2], [0, 2, 3]]]
        if k % 12 == 11:
            v[k] = v[k - 2]  # equal depths
    v[:, :, :, 3:6] = rng.normal(size=(n, 1, 1, 3))
    v[:, :, :, 6:] = rng.random((n, 1, 1, 4))
    v[:, :, :, 0] *= rng.choice([1, -1], (n, 1, 1))  # both windings, of which opaque ones keep one
    v, i = v.reshape(-1, 10), np.arange(6 * n, dtype=np.uint32).reshape(-1, 3)
    order = rng.permutation(n)
    i = i.reshape(n, 2, 3)[order].reshape(-1, 3)
    kw = dict(oit_layers=L, nodes_per_pixel=200, aa_type=aa, weighted_precision=oit.OIT_WEIGHTED_FP32)
    g = pu.render_gpu(alg, W, H, v, i, 2, scene_data(), 50, **kw)
    o = pu.render_oracle(alg, W, H, v, i, 2, scene_data(), 50, **kw)
    pu.check_pair(alg, g, o, W, H, L, aa)
