"""What this library is timed on: the calls its users make, over the sizes they make them at.

Each case names one public entry point (its "kind") and the sizes of the call:

  query    Session.query: closest hits of a ray list held on the host, as picking, probe and
           visibility tools ask for them
  frame    Session.render: one progressive RtRender pass into the caller's RGBA8 buffer, from the
           interactive front end's one path per pixel to the offline passes of 16
  load     Session.initialize and the first frame: what a user waits for after opening or editing a scene
  batch    Batch.render and every view's image: many views of many scenes per frame
  denoise  Session.denoise: the learned network (net true) or the guided filter (net false) on the
           running sums of a render
  train    Unet.train: Adam steps on a crop set, then the updated parameters
  grad     Unet.loss_grad: loss and gradient, for a training loop that lives outside the library

Scenes are the package's own synthetic ones (scenes.py): the Cornell box with a displaced sphere, the
room with a noisy geodesic sphere of up to a million triangles, rooms of spheres and boxes with glossy
materials, and the multi-scene batch. Their vertices, colours, cameras and sampler seeds come from the
seed alone. Buffers that a user's program keeps (the image, the ray list) are kept here too.
"""
import functools
import math
import sys
from pathlib import Path

import numpy as np
import torch
import torch.nn.functional as F

PACKAGE = Path(__file__).resolve().parent.parent / 'custom-ray-tracing-shader_b200'
if str(PACKAGE) not in sys.path:
    sys.path.insert(0, str(PACKAGE))

import native_api  # noqa: E402
import scenes  # noqa: E402

CROP_CHANNELS = 10
WIDTHS = (32, 48, 64, 96, 128)


def listed():
    return [
        # A picking or probe tool: a few thousand rays into a small scene. Latency of one call.
        dict(name='query_4k', kind='query', scene='cornell', triangles=5132, rays=4096),
        # Light baking and visibility maps: a long ray list into the million-triangle room.
        dict(name='query_1m', kind='query', scene='sphere', triangles=1003532, rays=1_000_000),
        # The stated small configuration (5,132 triangles, 256 x 256, depth 4) as the interactive
        # front end draws it: one path per pixel per pass, launch- and latency-bound.
        dict(name='frame_256_1spp', kind='frame', scene='cornell', triangles=5132, width=256, height=256, spp=1,
             depth=4, glossy=False),
        # An interactive full-HD frame: one path per pixel, a 100K-triangle room with glossy objects,
        # depth of field, sky light and six bounces.
        dict(name='frame_1080p_1spp', kind='frame', scene='room', triangles=100_000, width=1920, height=1080, spp=1,
             depth=6, glossy=True),
        # The stated large configuration: a million triangles, 1920 x 1080, 16 paths per pixel, depth 3.
        dict(name='pass_1080p_16spp', kind='frame', scene='sphere', triangles=1003532, width=1920, height=1080,
             spp=16, depth=3, glossy=False),
        # A scene edit in the front end: a few thousand triangles loaded, then a small first frame.
        dict(name='load_8k', kind='load', scene='room', triangles=8_000, width=640, height=360, spp=1, depth=4,
             glossy=True),
        # Opening the million-triangle scene at full HD.
        dict(name='load_1m', kind='load', scene='sphere', triangles=1003532, width=1920, height=1080, spp=1, depth=3,
             glossy=False),
        # Batched multi-scene rendering, scaled down from the stated 8 scenes and 64 views: uneven
        # scenes, square views of 256 and 512 pixels, 8 paths per pixel, depth 4.
        dict(name='batch_16_views', kind='batch', scenes=4, triangles=60_000, views=16, size=512, spp=8, depth=4),
        # The learned denoiser on a full-HD frame (1080 is no multiple of the network's 16).
        dict(name='denoise_net_1080p', kind='denoise', net=True, width=1920, height=1080, spp=4),
        # The default denoiser (no network attached) on an odd-sized window.
        dict(name='denoise_filter_odd', kind='denoise', net=False, width=1283, height=717, spp=4),
        # The stated training step (batch 32 of 128 x 128 crops, Adam), sixteen of them in one call.
        dict(name='train_32x128', kind='train', crops=64, batch=32, height=128, width=128, steps=16),
        # A small ragged batch for gradients only.
        dict(name='grad_6x80x112', kind='grad', batch=6, height=80, width=112),
    ]


def _log(rng, low, high):
    return int(round(math.exp(rng.uniform(math.log(low), math.log(high)))))


def draw(rng):
    kind = rng.choice(('query', 'frame', 'frame', 'load', 'batch', 'denoise', 'denoise', 'train', 'grad'))
    if kind == 'query':
        return dict(kind=kind, scene=rng.choice(('room', 'sphere')), triangles=_log(rng, 1_000, 1_000_000),
                    rays=_log(rng, 500, 1_000_000))
    if kind in ('frame', 'load'):
        width = _log(rng, 96, 1920)
        height = max(64, min(1080, int(width * rng.uniform(0.5, 1.0))))
        # spp times depth no more than the largest listed pass has.
        spp = 1 if kind == 'load' else rng.choice((1, 1, 2, 3, 4, 8, 16))
        depth = rng.randint(2, 3 if spp > 4 else 6)
        return dict(kind=kind, scene=rng.choice(('room', 'sphere')), triangles=_log(rng, 1_000, 1_000_000), width=width,
                    height=height, spp=spp, depth=depth, glossy=rng.random() < 0.5)
    if kind == 'batch':
        return dict(kind=kind, scenes=rng.randint(2, 4), triangles=_log(rng, 2_000, 60_000), views=rng.randint(3, 16),
                    size=rng.choice((96, 200, 256, 333, 512)), spp=rng.choice((1, 2, 4, 8)), depth=rng.randint(2, 4))
    if kind == 'denoise':
        width = _log(rng, 160, 1920)
        return dict(kind=kind, net=rng.random() < 0.5, width=width, spp=rng.choice((1, 4, 8)),
                    height=max(96, min(1080, int(width * rng.uniform(0.5, 1.0)))))
    height, width = 16 * rng.randint(2, 8), 16 * rng.randint(2, 8)
    if kind == 'grad':
        return dict(kind=kind, batch=rng.randint(1, 16), height=height, width=width)
    return dict(kind=kind, crops=rng.randint(8, 64), batch=rng.choice((1, 4, 7, 16, 32)), height=height, width=width,
                steps=rng.randint(2, 8))


# ---- scenes ----

@functools.lru_cache(maxsize=16)
def _geodesic(subdivisions):
    """Unit points and corner indices of a geodesic sphere (scenes.geodesic_sphere without displacement);
    the same for every seed, so it is made once."""
    rng = np.random.Generator(np.random.PCG64(0))
    v0, v1, v2, _ = scenes.geodesic_sphere(subdivisions, 1.0, (0.0, 0.0, 0.0), 0.0, rng)
    corners = np.stack([v0, v1, v2], 1).reshape(-1, 3)
    keys = np.round(corners * (1 << 20)).astype(np.int64)
    packed = (keys[:, 0] << 42) ^ ((keys[:, 1] & 0x1FFFFF) << 21) ^ (keys[:, 2] & 0x1FFFFF)
    _, first, inverse = np.unique(packed, return_index=True, return_inverse=True)
    return corners[first], inverse.reshape(-1, 3)


def _displaced_room(rng, triangles):
    """scenes.displaced_sphere_room for another seed and size: the noise is drawn per vertex."""
    subdivisions = max(2, int(round(math.sqrt(max(triangles - 12, 80) / 20.0))))
    points, corners = _geodesic(subdivisions)
    colors = rng.uniform(0.2, 0.8, (6, 3))
    room = scenes.open_box((-2.5, 0.0, -2.5), (2.5, 4.0, 2.5), colors[:5], 0.6, 3.98, 15.0)
    factor = 1.0 + rng.uniform(-0.05, 0.05, len(points))
    verts = points * (1.3 * factor)[:, None] + np.array([0.0, 1.45, 0.3])
    v0, v1, v2 = (verts[corners[:, k]] for k in range(3))
    face = np.cross(v1 - v0, v2 - v0)
    normal = np.zeros_like(verts)
    for k in range(3):
        for axis in range(3):
            normal[:, axis] += np.bincount(corners[:, k], weights=face[:, axis], minlength=len(verts))
    normal /= np.maximum(np.linalg.norm(normal, axis=1, keepdims=True), 1e-30)
    sphere = scenes.records(v0, v1, v2, color=colors[5], normals=tuple(normal[corners[:, k]] for k in range(3)), mesh=7)
    return np.concatenate([room, sphere])


def _scene(case, seed):
    """Triangles, camera, settings of a query, frame or load case."""
    rng = np.random.Generator(np.random.PCG64(seed))
    w, h = case.get('width', 256), case.get('height', 256)
    if case['scene'] == 'cornell':
        tris, cam, _, _, _ = scenes.cornell_sphere(seed=seed, width=w, height=h)
    elif case['scene'] == 'sphere':
        tris = _displaced_room(rng, case['triangles'])
        eye = (rng.uniform(-0.4, 0.4), 2.0 + rng.uniform(-0.2, 0.2), -7.0)
        cam = scenes.camera(eye, (0.0, 1.6, 0.0), math.tan(math.radians(24.0)), w / h)
    else:
        tris, cam, _, _ = scenes.random_room(seed, w, h, triangles=case['triangles'])
    glossy = bool(case.get('glossy', False))
    if glossy:
        # Glossy walls beside the objects' own materials, a thin lens and sky light.
        some = rng.random(len(tris)) < 0.2
        tris['smoothness'][some] = np.float32(0.85)
        tris['specularProbability'][some] = np.float32(0.3)
    settings = native_api.Settings(case.get('depth', 4), 1.0, 0.02 if glossy else 0.0, 3.0 if glossy else 1.0,
                                   0.5 if glossy else 0.0, 42 + seed % 1000, case.get('spp', 1))
    return tris, cam, settings


def _rays(rng, count, far):
    """Rays of a probe tool: origins all over the room, directions over the sphere, a finite reach."""
    q = np.zeros(count, native_api.QUERY_DTYPE)
    origin = rng.uniform((-2.4, 0.1, -2.4), (2.4, 3.9, 2.4), (count, 3)).astype(np.float32)
    direction = rng.normal(size=(count, 3))
    direction = (direction / np.linalg.norm(direction, axis=1, keepdims=True)).astype(np.float32)
    for k, axis in enumerate('xyz'):
        q['origin'][axis], q['direction'][axis] = origin[:, k], direction[:, k]
    q['limit'] = np.float32(far)
    return q


def _crops(seed, n, h, w):
    """A crop set as train_denoiser.py's, synthesised: noisy radiance around a smooth target, albedo,
    normals, distance."""
    rng = np.random.default_rng(seed)
    yy, xx = np.mgrid[0:h, 0:w] / max(h, w)
    phase = rng.uniform(0, 6, (n, 1, 1))
    shade = 0.5 + 0.5 * np.sin(rng.uniform(2, 6, (n, 1, 1)) * xx + rng.uniform(2, 6, (n, 1, 1)) * yy + phase)
    target = (rng.uniform(0.1, 2.0, (n, 1, 1, 3)) * shade[..., None]).astype(np.float32)
    aovs = np.empty((n, h, w, CROP_CHANNELS), np.float32)
    aovs[..., 0:3] = target * rng.standard_exponential((n, h, w, 3), np.float32)
    aovs[..., 3:6] = rng.uniform(0, 1, (n, 1, 1, 3))
    normal = rng.normal(size=(n, 1, 1, 3)) + 0.3 * rng.standard_normal((n, h, w, 3), np.float32)
    aovs[..., 6:9] = normal / np.linalg.norm(normal, axis=-1, keepdims=True)
    aovs[..., 9] = 1.0 + 4.0 * yy
    return aovs, target


# ---- the calls ----

class State:
    """What a program holds between calls; the native objects go when it goes."""

    def __init__(self):
        self.session = self.batch = self.net = None

    def __del__(self):
        if self.session is not None:
            if self.net is not None:
                self.session.set_denoiser(None)
            self.session.close()
        if self.batch is not None:
            self.batch.close()
        if self.net is not None:
            self.net.close()


@functools.lru_cache(maxsize=1)
def _library():
    return native_api.load_library()


def prepare(case, seed):
    s = State()
    s.kind = kind = case['kind']
    lib = _library()
    if kind in ('query', 'frame', 'load'):
        s.tris, s.camera, s.settings = _scene(case, seed)
        s.size = (case.get('width', 256), case.get('height', 256))
        s.session = native_api.Session(lib)
        if kind != 'load':
            s.session.initialize(s.tris, *s.size)
        s.image = np.zeros(s.size[0] * s.size[1] * 4, np.uint8)
        if kind == 'query':
            s.rays = _rays(np.random.default_rng(seed + 1), case['rays'], 50.0)
    elif kind == 'batch':
        rng = np.random.Generator(np.random.PCG64(seed))
        s.batch = native_api.Batch(lib)
        # Uneven scenes: each about half the size of the one before.
        ids = [s.batch.add_scene(scenes.random_scene(seed * 100 + k, max(500, case['triangles'] >> k)))
               for k in range(case['scenes'])]
        for v in range(case['views']):
            eye = (rng.uniform(-3.0, 3.0), rng.uniform(0.8, 3.2), rng.uniform(-3.8, -2.5))
            target = (rng.uniform(-1.5, 1.5), rng.uniform(0.5, 2.5), rng.uniform(-1.0, 2.5))
            cam = scenes.camera(eye, target, math.tan(math.radians(rng.uniform(25.0, 45.0))), 1.0)
            size = case['size'] if v % 2 else max(64, case['size'] // 2)
            s.batch.add_view(ids[v % len(ids)], cam, size, size)
        s.settings = native_api.Settings(case['depth'], 1.0, 0.0, 1.0, 0.5, 42 + seed % 1000, case['spp'])
    elif kind == 'denoise':
        w, h = case['width'], case['height']
        tris, cam, settings, environment = scenes.random_room(seed, w, h, triangles=20_000)
        settings.raysPerPixel = case['spp']
        s.session = native_api.Session(lib).initialize(tris, w, h)
        s.session.set_environment(environment)
        s.session.render_device(cam, settings)
        s.image = np.zeros(w * h * 4, np.uint8)
        if case['net']:
            s.net = native_api.Unet(lib)
            s.net.load(native_api.DENOISER_WEIGHTS)
            s.session.set_denoiser(s.net)
    else:
        s.aovs, s.target = _crops(seed, case.get('crops', case['batch']), case['height'], case['width'])
        s.net = native_api.Unet(lib)
        s.net.load(native_api.DENOISER_WEIGHTS)
        s.steps, s.minibatch, s.seed = case.get('steps', 0), case['batch'], seed
    return s


def run(s):
    if s.kind == 'query':
        hits = s.session.query(s.rays)
        return {name: hits[name] for name in ('index', 'distance', 'u', 'v')}
    if s.kind == 'frame':
        return s.session.render(s.camera, s.settings, output=s.image)[0]
    if s.kind == 'load':
        s.session.initialize(s.tris, *s.size)
        return s.session.render(s.camera, s.settings, output=s.image)[0]
    if s.kind == 'batch':
        s.batch.render(s.settings)
        return [s.batch.image(v) for v in range(len(s.batch.views))]
    if s.kind == 'denoise':
        return s.session.denoise(s.image)[0]
    if s.kind == 'train':
        # The learning rate at the end of train_denoiser.py's schedule.
        losses = s.net.train(s.aovs, s.target, s.steps, s.minibatch, 5e-5, s.seed)
        return {'losses': losses, 'params': s.net.params()}
    loss, grads = s.net.loss_grad(s.aovs, s.target)
    return {'loss': loss, 'grads': grads}


# ---- what a pass cannot do without ----

def _network_flops(pixels):
    """Forward FLOPs of the U-Net on `pixels` full-resolution pixels."""
    table, prev = [], 16
    for level, width in enumerate(WIDTHS):
        table += [(prev, width, level), (width, width, level)]
        prev = width
    for level in (3, 2, 1, 0):
        table += [(prev + WIDTHS[level], WIDTHS[level], level), (WIDTHS[level], WIDTHS[level], level)]
        prev = WIDTHS[level]
    return pixels * (sum(18 * ci * co / 4 ** level for ci, co, level in table) + 6 * WIDTHS[0])


def _query_flops(triangles):
    """FLOPs of one ray: eight boxes of 15 on each of about log2(n) / 2 eight-wide nodes, four
    triangles of 45."""
    return 120 * max(1.0, math.log2(max(triangles, 2)) / 2) + 180


def work(case):
    kind = case['kind']
    if kind == 'query':
        return {'bytes': case['rays'] * (28 + 16) + case['triangles'] * 48,
                'flops': case['rays'] * _query_flops(case['triangles'])}
    if kind in ('frame', 'load'):
        pixels = case['width'] * case['height']
        rays = pixels * case['spp'] * case['depth'] * 2  # a path ray and a light ray per bounce
        once = case['triangles'] * (116 if kind == 'load' else 48)
        return {'bytes': once + pixels * 44, 'flops': rays * _query_flops(case['triangles'])}
    if kind == 'batch':
        pixels = sum((case['size'] if v % 2 else max(64, case['size'] // 2)) ** 2 for v in range(case['views']))
        triangles = sum(max(500, case['triangles'] >> k) for k in range(case['scenes']))
        return {'bytes': triangles * 48 + pixels * 44,
                'flops': pixels * case['spp'] * case['depth'] * 2 * _query_flops(case['triangles'])}
    if kind == 'denoise':
        pixels = case['width'] * case['height']
        # The filter: five passes of 25 taps, about 30 operations each.
        return {'bytes': pixels * (44 + 4), 'flops': _network_flops(pixels) if case['net'] else pixels * 5 * 25 * 30}
    pixels = case['batch'] * case['height'] * case['width']
    steps = case.get('steps', 1)
    sets = case.get('crops', case['batch']) * case['height'] * case['width']
    return {'bytes': sets * 4 * (CROP_CHANNELS + 3) + steps * 1_017_379 * 4 * 4,
            'flops': steps * 3 * _network_flops(pixels)}


# ---- the same in 64 bits ----

def _exact_hits(tris, q, device, chunk=128):
    """Closest hits by testing every triangle (Moeller and Trumbore) in 64 bits."""
    def vec(field):
        return torch.from_numpy(np.stack([field[a] for a in 'xyz'], 1).astype(np.float64)).to(device)

    o, d = vec(q['origin']), vec(q['direction'])
    limit = torch.from_numpy(q['limit'].astype(np.float64)).to(device)
    p0, e1, e2 = vec(tris['origin']), vec(tris['edge1']), vec(tris['edge2'])
    one_sided = torch.from_numpy(tris['oneSided'] != 0).to(device)
    out = torch.zeros(3, len(q), dtype=torch.float64, device=device)
    for k in range(0, len(q), chunk):
        ok, dk = o[k:k + chunk, None], d[k:k + chunk, None]
        p = torch.linalg.cross(dk.expand(-1, len(e2), -1), e2[None].expand(dk.shape[0], -1, -1))
        det = (e1 * p).sum(-1)
        keep = (det.abs() >= 1e-7) & ~(one_sided & (det < 0))
        inv = 1.0 / torch.where(keep, det, torch.ones_like(det))
        s = ok - p0
        u = (s * p).sum(-1) * inv
        c = torch.linalg.cross(s, e1[None].expand(s.shape[0], -1, -1))
        v = (dk * c).sum(-1) * inv
        t = (e2 * c).sum(-1) * inv
        keep &= (u >= 0) & (u <= 1) & (v >= 0) & (u + v <= 1) & (t > 1e-4) & (t < limit[k:k + chunk, None])
        t = torch.where(keep, t, torch.full_like(t, math.inf))
        best, at = t.min(1)
        hit, row = torch.isfinite(best), torch.arange(len(at), device=device)
        out[0, k:k + chunk] = torch.where(hit, best, limit[k:k + chunk])
        out[1, k:k + chunk] = torch.where(hit, u[row, at], 0.0)
        out[2, k:k + chunk] = torch.where(hit, v[row, at], 0.0)
    return out.cpu().numpy()


def _parameters(device):
    """The trained network's parameters from its checkpoint, per layer, in 64 bits: [(OIHW, bias)] of the 18
    3x3 layers, then ([32][3], [3])."""
    flat = np.fromfile(native_api.DENOISER_WEIGHTS, np.float32, offset=32)
    table, prev = [], 16
    for width in WIDTHS:
        table += [(prev, width), (width, width)]
        prev = width
    for width in WIDTHS[3::-1]:
        table += [(prev + width, width), (width, width)]
        prev = width
    layers, at = [], 0

    def take(*shape):
        nonlocal at
        n = int(np.prod(shape))
        x = torch.from_numpy(flat[at:at + n].astype(np.float64)).to(device).reshape(shape)
        at += n
        return x

    for ci, co in table:
        w = take(3, 3, ci, co).permute(3, 2, 0, 1).contiguous()
        layers.append((w.requires_grad_(), take(co).requires_grad_()))
    layers.append((take(WIDTHS[0], 3).requires_grad_(), take(3).requires_grad_()))
    return layers


def _exact_gradient(case, seed, device):
    aovs, target = _crops(seed, case['batch'], case['height'], case['width'])
    a = torch.from_numpy(aovs.astype(np.float64)).to(device).permute(0, 3, 1, 2)
    t = torch.log1p(torch.from_numpy(target.astype(np.float64)).to(device).clamp(min=0)).permute(0, 3, 1, 2)
    x = torch.zeros(a.shape[0], 16, *a.shape[2:], dtype=torch.float64, device=device)
    x[:, 0:3], x[:, 3:9], x[:, 9] = torch.log1p(a[:, 0:3].clamp(min=0)), a[:, 3:9], torch.log1p(a[:, 9].clamp(min=0))
    layers = _parameters(device)
    k, skips = 0, []

    def block(x):
        nonlocal k
        for _ in range(2):
            x = F.relu(F.conv2d(x, *layers[k], padding=1))
            k += 1
        return x

    for level in range(5):
        x = block(F.avg_pool2d(x, 2) if level else x)
        skips.append(x)
    for level in (3, 2, 1, 0):
        x = block(torch.cat([F.interpolate(x, scale_factor=2, mode='nearest'), skips[level]], 1))
    wo, bo = layers[-1]
    loss = (torch.einsum('nchw,ck->nkhw', x, wo) + bo[None, :, None, None] - t).abs().mean()
    loss.backward()
    parts = []
    for w, b in layers[:-1]:
        parts += [w.grad.permute(2, 3, 1, 0).reshape(-1), b.grad]
    parts += [wo.grad.reshape(-1), bo.grad]
    return {'loss': float(loss.detach()), 'grads': torch.cat(parts).cpu().numpy()}


def exact(case, seed):
    device = 'cuda' if torch.cuda.is_available() else 'cpu'
    if case['kind'] == 'query' and case['rays'] * case['triangles'] <= 4e8:
        tris, _, _ = _scene(case, seed)
        hits = _exact_hits(tris, _rays(np.random.default_rng(seed + 1), case['rays'], 50.0), device,
                           chunk=max(1, int(4e6 / len(tris))))
        return {'index': None, 'distance': hits[0], 'u': hits[1], 'v': hits[2]}
    if case['kind'] == 'grad':
        return _exact_gradient(case, seed, device)
    return None  # whole bytes, or a chain of rounded training steps, or far too many pairs to test
