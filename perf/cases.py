"""Performance cases of the transparent pass: what a program that uses this
package has it render, through its public entry points.

A case names an algorithm, an antialiasing mode, a frame size, a scene of
spheres and the way the frame is asked for: one plain call, a captured frame
replayed, the pass's calls one by one, host buffers in and out, or many views
as one batch. The sizes are those of the reference's test sequence (64x40 and
800x512, its default state), of the workloads of bench.py, and odd ones in
between. Scenes are drawn from the seed: every seed places, scales and colours
its spheres anew, at the same counts and radii.

  listed()             the cases
  draw(rng)            one more case of the same ranges
  prepare(case, seed)  scene, camera, renderer(s) and output on the GPU
  run(state)           one frame (or one batch of views): the images
  work(case)           bytes and operations that a frame cannot do without
  exact(case, seed)    the linear image in 64 bits, for the cases that return it
"""
import math

import numpy as np
import torch

import vk_order_independent_transparency_gb300 as oit

ALGORITHMS = {'simple': oit.OIT_SIMPLE, 'linkedlist': oit.OIT_LINKEDLIST, 'loop': oit.OIT_LOOP,
              'loop64': oit.OIT_LOOP64, 'spinlock': oit.OIT_SPINLOCK, 'interlock': oit.OIT_INTERLOCK,
              'weighted': oit.OIT_WEIGHTED}
AA = {'none': oit.OIT_AA_NONE, 'msaa4': oit.OIT_AA_MSAA_4X, 'ssaa4': oit.OIT_AA_SSAA_4X,
      'super4': oit.OIT_AA_SUPER_4X, 'msaa8': oit.OIT_AA_MSAA_8X, 'ssaa8': oit.OIT_AA_SSAA_8X}

# Spheres in [-1, 1]^3 seen from z = 3 (bench.py), or in [-4, 4]^3 seen from
# z = 12 (the reference's own scene).
NEAR_SCENE = dict(half=1.0, eye=3.0, z_far=10.0)
WIDE_SCENE = dict(half=4.0, eye=12.0, z_far=100.0)
FOV_Y = 45.0
Z_NEAR = 0.1

DEFAULTS = dict(algorithm='linkedlist', width=640, height=480, layers=8, nodes=8, aa='none', tail=True,
                spheres=256, stacks=16, rmin=0.05, rmax=0.15, percent=100, alpha_min=0.2, alpha_width=0.6,
                record_fp32=False, weighted_fp32=False, half_color=False, linear=False, call='frame')


def _case(name=None, **kw):
    c = {**DEFAULTS, **NEAR_SCENE, **kw}
    if name:
        c['name'] = name
    return c


def listed():
    return [
        # the smallest call: three objects in a thumbnail, as a test or a preview renders it; the linear image too
        _case('tiny_spinlock_64x40', algorithm='spinlock', width=64, height=40, spheres=3, rmin=0.1, rmax=0.4,
              alpha_width=0.3, linear=True),
        # the reference's default state and scene in its own window, one plain call a frame
        _case('default_spinlock_800x512', algorithm='spinlock', width=800, height=512, spheres=1024, rmin=0.045,
              rmax=0.45, nodes=10, alpha_width=0.3, **WIDE_SCENE),
        # a small interactive frame, captured once and replayed
        _case('linkedlist_640x480', call='graph'),
        # a full-HD frame with opaque objects in front of and behind the transparent ones
        _case('loop64_1920x1080_opaque', algorithm='loop64', width=1920, height=1080, layers=16, spheres=1024,
              rmin=0.03, rmax=0.10, percent=60, call='graph'),
        # coverage records with 8 samples a pixel, a heavy frame
        _case('interlock_2560x1440_msaa8', algorithm='interlock', width=2560, height=1440, aa='msaa8', spheres=4096,
              rmin=0.02, rmax=0.08, call='graph'),
        # the pass's calls one by one, as a renderer with its own frame loop makes them; an odd size
        _case('simple_1283x717_msaa4_staged', algorithm='simple', width=1283, height=717, aa='msaa4', layers=4,
              spheres=500, rmin=0.03, rmax=0.12, percent=70, tail=False, call='staged'),
        # the largest frame: 4K, fp16 accumulators, an instanced scene
        _case('weighted_3840x2160_instanced', algorithm='weighted', width=3840, height=2160, spheres=16384,
              rmin=0.01, rmax=0.05, alpha_min=0.05, alpha_width=0.9, call='instanced'),
        # weighted blending in fp32, the linear image kept for later passes; an odd size
        _case('weighted_fp32_641x359_linear', algorithm='weighted', width=641, height=359, spheres=200, rmin=0.03,
              rmax=0.15, weighted_fp32=True, linear=True),
        # one A-buffer per sample, both passes of the two-pass algorithm; an odd size
        _case('loop_1001x563_ssaa4', algorithm='loop', width=1001, height=563, aa='ssaa4', spheres=300, rmin=0.04,
              rmax=0.12),
        # float records, supersampled
        _case('linkedlist_fp32_700x420_super4', width=700, height=420, layers=4, nodes=10, aa='super4', spheres=400,
              rmin=0.03, rmax=0.10, record_fp32=True),
        # many views a step (a server, a data generator): linked list and Loop64, 4 to 32 layers, mixed sizes
        _case('batch_24views', call='batch', views=24, shapes=2, width=2048, height=2048, spheres=8192, rmin=0.01,
              rmax=0.05, half_color=True),
        # a mesh in host memory, the image back in host memory
        _case('host_linkedlist_1280x720', width=1280, height=720, spheres=200, rmin=0.04, rmax=0.12, call='host'),
    ]


def _log_uniform(rng, lo, hi):
    return lo * (hi / lo) ** rng.random()


def draw(rng):
    """One more frame (or batch) of the listed ranges."""
    call = rng.choice(['frame', 'frame', 'frame', 'graph', 'graph', 'staged', 'instanced', 'host', 'batch'])
    alpha_min = rng.choice([0.05, 0.2])
    if call == 'batch':
        return _case(call=call, views=rng.randint(2, 24), shapes=rng.randint(3, 1 << 20), width=2048, height=2048,
                     spheres=8192, rmin=0.01, rmax=0.05, half_color=True)
    algorithm = rng.choice(sorted(ALGORITHMS))
    area = _log_uniform(rng, 64 * 40, 2560 * 1440)
    aspect = rng.choice([1.0, 4 / 3, 16 / 10, 16 / 9])
    width = max(8, int(math.sqrt(area * aspect)))
    height = max(8, int(math.sqrt(area / aspect)))
    aa = rng.choice(['none', 'none', 'none'] + sorted(AA))
    layers = rng.choice([1, 2, 4, 8, 8, 16, 32])
    samples = {'ssaa4': 4, 'super4': 4, 'ssaa8': 8}.get(aa, 1)
    while width * height * samples * layers > 2560 * 1440 * 16:  # A-buffers within those of the listed frames
        if layers > 4:
            layers //= 2
        else:
            width, height = width * 3 // 4, height * 3 // 4
    spheres = int(_log_uniform(rng, 3, 4096))
    rmax = _log_uniform(rng, 0.04, 0.4)
    c = _case(algorithm=algorithm, width=width, height=height, layers=layers, nodes=10, aa=aa,
              tail=rng.random() < 0.7, spheres=spheres, rmin=rmax / rng.choice([2, 4, 8]), rmax=rmax,
              percent=rng.choice([100, 100, 100, 60, 25]), alpha_min=alpha_min,
              alpha_width=rng.choice([0.3, 0.6, 0.9]), call=call, stacks=rng.choice([16, 16, 16, 8, 11]),
              half_color=rng.random() < 0.2, linear=rng.random() < 0.2, weighted_fp32=rng.random() < 0.5)
    if algorithm in ('linkedlist', 'loop64'):
        c['record_fp32'] = rng.random() < 0.25
    # no more fragments than the listed frames have, and linked-list pools that hold them
    most = min(4e7 / samples, 4.0 * width * height)
    while _fragments(c) > most:
        c['rmax'] *= 0.8
        c['rmin'] *= 0.8
    return c


# ---------------------------------------------------------------------------
# Scenes
# ---------------------------------------------------------------------------
def _template(stacks):
    """Unit UV sphere: positions (also the normals) and outward triangles."""
    slices = 2 * stacks
    th = np.pi * np.arange(stacks + 1) / stacks
    ph = 2.0 * np.pi * np.arange(slices + 1) / slices
    pos = np.stack([np.sin(th)[:, None] * np.cos(ph), np.cos(th)[:, None] + 0 * ph, np.sin(th)[:, None] * np.sin(ph)],
                   -1).reshape(-1, 3)
    i, j = np.meshgrid(np.arange(stacks), np.arange(slices), indexing='ij')
    a = i * (slices + 1) + j
    upper = np.stack([a, a + 1, a + slices + 1], -1)
    lower = np.stack([a + 1, a + slices + 2, a + slices + 1], -1)
    keep = np.stack([i != 0, i != stacks - 1], -1).reshape(-1)
    tri = np.stack([upper, lower], 2).reshape(-1, 3)[keep]
    return pos.astype(np.float32), tri.astype(np.uint32)


def _instances(spheres, half, rmin, rmax, seed):
    """Centre, radius and colour of every sphere."""
    u = np.random.default_rng(seed).random((spheres, 8), np.float32)
    inst = u.copy()
    inst[:, :3] = (2.0 * u[:, :3] - 1.0) * half
    inst[:, 3] = rmin + u[:, 3] * (rmax - rmin)
    return inst


def _flatten(pos, tri, inst):
    """One mesh of every sphere: (vertices [n, 10], triangles [m, 3])."""
    n, k = len(inst), len(pos)
    v = np.empty((n, k, 10), np.float32)
    v[:, :, :3] = pos * inst[:, None, 3:4] + inst[:, None, :3]
    v[:, :, 3:6] = pos
    v[:, :, 6:] = inst[:, None, 4:]
    t = tri[None] + (np.arange(n, dtype=np.uint32) * np.uint32(k))[:, None, None]
    return v.reshape(-1, 10), t.reshape(-1, 3)


def _mesh(case, seed):
    pos, tri = _template(case['stacks'])
    return pos, tri, _instances(case['spheres'], case['half'], case['rmin'], case['rmax'], seed)


def _renderer(case, **kw):
    c = dict(case, **kw)
    flags = (oit.OIT_FLAG_CUDA_GRAPH if c['call'] == 'graph' else 0) | \
        (oit.OIT_FLAG_HALF_COLOR if c['half_color'] else 0) | (oit.OIT_FLAG_LINEAR_OUTPUT if c['linear'] else 0)
    r = oit.Renderer(oit.make_state(
        ALGORITHMS[c['algorithm']], c['width'], c['height'], oit_layers=c['layers'], nodes_per_pixel=c['nodes'],
        tail_blend=c['tail'], aa_type=AA[c['aa']], alpha_min=c['alpha_min'], alpha_width=c['alpha_width'],
        record_format=oit.OIT_RECORD_RGBA32F if c['record_fp32'] else oit.OIT_RECORD_RGBA8,
        weighted_precision=oit.OIT_WEIGHTED_FP32 if c['weighted_fp32'] else oit.OIT_WEIGHTED_FP16, flags=flags))
    r.update_scene(oit.make_camera(c['width'], c['height'], eye=(0.0, 0.0, c['eye']), fov_y=FOV_Y, z_near=Z_NEAR,
                                   z_far=c['z_far']))
    return r


def _view_shapes(case):
    """The views of a batch: square, sides log-uniform in 256..2048, 64..8192
    spheres, linked list and Loop64 in turn, 4 to 32 layers."""
    rng = np.random.default_rng(case['shapes'])
    shapes = []
    for k in range(case['views']):
        side = int(round(256 * 8 ** rng.random()))
        shapes.append(dict(algorithm='linkedlist' if k % 2 == 0 else 'loop64', width=side, height=side,
                           layers=[4, 8, 16, 32][(k // 2) % 4], spheres=int(round(64 * 128 ** rng.random()))))
    return shapes


def _prepare_batch(case, seed):
    pos, tri = _template(case['stacks'])
    template = torch.from_numpy(np.concatenate([pos, pos], 1)).cuda()
    indices = torch.from_numpy(tri.view(np.int32)).cuda()
    views, images = [], []
    for k, shape in enumerate(_view_shapes(case)):
        inst = torch.from_numpy(_instances(shape['spheres'], case['half'], case['rmin'], case['rmax'],
                                           1000 * seed + k)).cuda()
        out = torch.empty((shape['height'], shape['width'], 4), dtype=torch.uint8, device='cuda')
        views.append((_renderer(case, **shape), oit.DeviceInstancedMesh.from_tensors(template, indices, inst),
                      len(tri), case['percent'], out.data_ptr()))
        images.append(out)
    batch = oit.Batch(parallel_streams=16)
    batch.set_views(views)
    return dict(case=case, batch=batch, views=views, images=images)


def prepare(case, seed):
    if case['call'] == 'batch':
        return _prepare_batch(case, seed)
    pos, tri, inst = _mesh(case, seed)
    state = dict(case=case, renderer=_renderer(case), tpo=len(tri))
    if case['call'] == 'instanced':
        state['mesh'] = oit.DeviceInstancedMesh(np.concatenate([pos, pos], 1), tri, inst)
    elif case['call'] == 'host':
        state['vertices'], state['indices'] = _flatten(pos, tri, inst)
        state['image'] = np.zeros((case['height'], case['width'], 4), np.uint8)
        return state
    else:
        state['mesh'] = oit.DeviceMesh(*_flatten(pos, tri, inst))
    state['image'] = torch.empty((case['height'], case['width'], 4), dtype=torch.uint8, device='cuda')
    return state


class _DeviceArray:
    """A device buffer of a renderer, for torch.as_tensor: the tensor holds
    this object, and so the renderer that owns the memory."""

    def __init__(self, owner, ptr, shape, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = dict(data=(ptr, False), shape=shape, typestr=typestr, version=3)


def run(state):
    case = state['case']
    if case['call'] == 'batch':
        state['batch'].render()
        return state['images']
    r, pct = state['renderer'], case['percent']
    if case['call'] == 'host':
        r.render_frame_host(state['vertices'], state['indices'], state['tpo'], pct, state['image'])
        return _outputs(state)
    out = state['image'].data_ptr()
    if case['call'] == 'instanced':
        r.render_frame_instanced(state['mesh'], pct, out_ptr=out)
    elif case['call'] == 'staged':
        mesh, tpo = state['mesh'], state['tpo']
        transparent = case['spheres'] * pct // 100 * tpo
        r.begin_frame()
        r.clear_transparent()
        if transparent < mesh.num_triangles:
            r.draw_opaque(mesh, transparent, mesh.num_triangles - transparent)
        r.draw_transparent_color(mesh, 0, transparent)
        r.composite(out_ptr=out)
    else:
        r.render_frame(state['mesh'], state['tpo'], pct, out_ptr=out)
    return _outputs(state)


def _outputs(state):
    """The image, and the linear image where the case asks for it."""
    case = state['case']
    if not case['linear']:
        return dict(image=state['image'])
    if 'linear' not in state:
        ptr, _ = state['renderer'].buffer(oit.OIT_BUF_OUTPUT_LINEAR)
        state['linear'] = torch.as_tensor(_DeviceArray(state['renderer'], ptr, (case['height'], case['width'], 4),
                                                       '<f4'), device='cuda')
    return dict(image=state['image'], linear=state['linear'])


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _triangles(stacks):
    return 2 * stacks * (2 * stacks - 2)


def _fragments(case):
    """Expected transparent fragments: twice every sphere's disc (front and
    back faces), at the scene's mean distance, within the frame's share."""
    scale = case['height'] / 2 / math.tan(math.radians(FOV_Y / 2)) / case['eye']
    lo, hi = case['rmin'] * scale, case['rmax'] * scale
    r2 = (lo * lo + lo * hi + hi * hi) / 3
    ss = 4 if case['aa'] == 'super4' else 1
    return case['spheres'] * case['percent'] / 100 * 2 * math.pi * r2 * ss


def work(case):
    """The scene read once and the images written once; per triangle its three
    vertices' transforms and its setup, per fragment its interpolation,
    shading and blending."""
    if case['call'] == 'batch':
        every = [work(dict(case, **shape, call='instanced')) for shape in _view_shapes(case)]
        return dict(bytes=sum(w['bytes'] for w in every), flops=sum(w['flops'] for w in every))
    triangles = case['spheres'] * _triangles(case['stacks'])
    vertices = (case['stacks'] + 1) * (2 * case['stacks'] + 1)
    if case['call'] == 'instanced':
        scene = 32 * case['spheres'] + 24 * vertices + 12 * _triangles(case['stacks'])
    else:
        scene = 40 * vertices * case['spheres'] + 12 * triangles
    pixels = case['width'] * case['height']
    samples = {'ssaa4': 4, 'ssaa8': 8}.get(case['aa'], 1)
    return dict(bytes=scene + pixels * (20 if case['linear'] else 4),
                flops=200.0 * triangles + 100.0 * samples * _fragments(case))


# ---------------------------------------------------------------------------
# The linear image in 64 bits
# ---------------------------------------------------------------------------
def _encode(c):
    """sRGB code of a linear value."""
    c = c.clamp(0.0, 1.0)
    return torch.round(255.0 * torch.where(c <= 0.0031308, 12.92 * c, 1.055 * c ** (1 / 2.4) - 0.055))


def _decode(code):
    s = code / 255.0
    return torch.where(s <= 0.04045, s / 12.92, ((s + 0.055) / 1.055) ** 2.4)


def _exact_fragments(case, seed):
    """Every fragment in primitive order: pixel, depth, view depth, colour."""
    W, H = case['width'], case['height']
    vertices, triangles = _flatten(*_mesh(case, seed))
    v = torch.from_numpy(vertices).cuda().double()
    t = torch.from_numpy(triangles.astype(np.int64)).cuda()
    f = 1.0 / math.tan(math.radians(FOV_Y) / 2)
    zn, zf = Z_NEAR, case['z_far']
    p = v[:, :3] - torch.tensor([0.0, 0.0, case['eye']], dtype=torch.float64, device='cuda')
    w = -p[:, 2]
    x, y = p[:, 0] * f * H / W / w, -p[:, 1] * f / w
    z = (zf / (zn - zf) * p[:, 2] + zn * zf / (zn - zf)) / w
    # window positions have 8 subpixel bits
    X = torch.round((x + 1) * W / 2 * 256)[t]
    Y = torch.round((y + 1) * H / 2 * 256)[t]
    z, q = z[t], (1 / w)[t]
    normal, vz, colour = v[:, 3:6][t] * q[..., None], p[:, 2][t] * q, v[:, 6:][t[:, 0]]
    area = (X[:, 1] - X[:, 0]) * (Y[:, 2] - Y[:, 0]) - (Y[:, 1] - Y[:, 0]) * (X[:, 2] - X[:, 0])
    x0 = torch.floor(X.amin(1) / 256).clamp(0, W)
    x1 = torch.floor(X.amax(1) / 256).clamp(-1, W - 1)
    y0 = torch.floor(Y.amin(1) / 256).clamp(0, H)
    y1 = torch.floor(Y.amax(1) / 256).clamp(-1, H - 1)
    wide = (x1 - x0 + 1).clamp(min=0).long()
    count = torch.where(area != 0, wide * (y1 - y0 + 1).clamp(min=0).long(), 0)
    k = torch.repeat_interleave(torch.arange(len(t), device='cuda'), count)
    at = torch.arange(len(k), device='cuda') - (count.cumsum(0) - count)[k]
    px, py = x0[k].long() + at % wide[k], y0[k].long() + at // wide[k]
    sx, sy = px * 256.0 + 128, py * 256.0 + 128
    b, inside = [], torch.ones_like(k, dtype=torch.bool)
    sign = torch.sign(area)[k]
    for i in range(3):
        j, m = (i + 1) % 3, (i + 2) % 3
        dx, dy = (X[:, m] - X[:, j])[k], (Y[:, m] - Y[:, j])[k]
        e = dx * (sy - Y[k, j]) - dy * (sx - X[k, j])
        dx, dy = sign * dx, sign * dy
        top_left = (dy < 0) | ((dy == 0) & (dx > 0))
        inside &= (sign * e > 0) | ((e == 0) & top_left)
        b.append(e / area[k])
    k, px, py = k[inside], px[inside], py[inside]
    b = torch.stack([e[inside] for e in b], 1)
    n = torch.nn.functional.normalize((b[..., None] * normal[k]).sum(1), dim=1)
    warmth = 0.5 + 0.5 * (n * torch.nn.functional.normalize(torch.tensor([[-1.0, 2.0, 1.0]], dtype=torch.float64,
                                                                         device='cuda'))).sum(1)
    rgb = colour[k, :3] * torch.stack([warmth, 0.25 + 0.75 * warmth, 0.75 + 0.25 * warmth], 1)
    alpha = (colour[k, 3] * case['alpha_width'] + case['alpha_min']).clamp(0, 1)
    depth = (b * z[k]).sum(1)
    view = (b * vz[k]).sum(1) / (b * q[k]).sum(1)
    return py * W + px, depth, view, rgb, alpha


def exact(case, seed):
    """The linear image of a single-sample frame without opaque objects, where
    it follows from the fragments alone: weighted blending, or every fragment
    kept. None otherwise."""
    if not case['linear'] or case['aa'] != 'none' or case['percent'] != 100 or case['call'] == 'batch' or \
            _fragments(case) > 4e6:
        return None
    pixels = case['width'] * case['height']
    pixel, depth, view, rgb, alpha = _exact_fragments(case, seed)
    linear = torch.full((pixels, 4), 0.2, dtype=torch.float64, device='cuda')
    if case['algorithm'] == 'weighted':
        c = torch.cat([rgb * alpha[:, None], alpha[:, None]], 1)
        weight = (0.03 / (1e-5 + (-view * 10.0 / 200.0) ** 4)).clamp(1e-2, 3e3)
        weight = weight * (c.amax(1) * 40.0 + 0.01).clamp(max=1.0) ** 2
        total = torch.zeros_like(linear).index_add_(0, pixel, c * weight[:, None])
        reveal = torch.zeros(pixels, dtype=torch.float64, device='cuda')
        reveal = torch.exp(reveal.index_add_(0, pixel, torch.log1p(-alpha)))[:, None]
        colour = torch.cat([total[:, :3] / total[:, 3:].clamp(min=1e-5), reveal], 1)
        linear = colour * (1 - reveal) + linear * reveal
    else:
        if int(torch.bincount(pixel, minlength=pixels).max()) > case['layers']:
            return None
        if not case['record_fp32']:  # records hold 8 bits a channel
            rgb, alpha = _decode(_encode(rgb)), torch.round(alpha * 255) / 255
        far = torch.argsort(depth, descending=True, stable=True)
        far = far[torch.argsort(pixel[far], stable=True)]
        pixel, c = pixel[far], torch.cat([rgb * alpha[:, None], alpha[:, None]], 1)[far]
        first = torch.searchsorted(pixel, pixel)
        rank = torch.arange(len(pixel), device='cuda') - first
        for i in range(int(rank.max()) + 1 if len(rank) else 0):  # each pixel's fragments, farthest first
            m = rank == i
            linear[pixel[m]] = c[m] + linear[pixel[m]] * (1 - c[m][:, 3:])
    return dict(image=None, linear=linear.reshape(case['height'], case['width'], 4))
