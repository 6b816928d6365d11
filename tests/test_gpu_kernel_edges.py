"""Kernels and dispatch rules at the sizes where they can go wrong: edges of
tiles, remainders, the smallest and largest of a range. Needs a GPU.

Tolerances: node arrays, ray queries, accumulated sums and convolutions that
only change how the same products are laid out are bit-exact; the others are
stated at their test."""
import threading

import numpy as np
import pytest
import torch

import scenes
from native_api import QUERY_DTYPE, Session, Unet
from test_gpu_parity import _leaf_sets
from test_gpu_unet import features, forward, layer_table, pack_grads, synthetic, unpack

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def sphere():
    return scenes.cornell_sphere()[0]


@pytest.fixture(scope='module')
def net(lib):
    n = Unet(lib, seed=11)
    yield n
    n.close()


def some_triangles(sphere, n):
    pick = np.random.default_rng(n).permutation(len(sphere))[:n]
    return sphere[np.sort(pick)]


def rays(count, seed=3):
    rng = np.random.default_rng(seed)
    q = np.zeros(count, QUERY_DTYPE)
    d = rng.normal(size=(count, 3))
    d /= np.linalg.norm(d, axis=1, keepdims=True)
    o = rng.uniform(-0.9, 0.9, (count, 3)) + (0, 1, 0)
    for k, ax in enumerate('xyz'):
        q['origin'][ax], q['direction'][ax] = o[:, k], d[:, k]
    q['limit'] = np.where(np.arange(count) % 5 == 0, 0.25, 1e30).astype(np.float32)
    return q


@pytest.mark.parametrize('n', (1, 2, 4, 5, 31, 32, 33, 64, 65, 511, 512, 513, 1025, 2047, 2048, 2049))
def test_build_sizes(session, oracle, sphere, n):
    """Around a warp's subtree (32), the tasks searched from their primitives
    (512) and the tasks binned in one block (2048): the reference's nodes, and
    its answers through the default trees."""
    tris = some_triangles(sphere, n)
    assert len(tris) == n
    scene = oracle.scene(tris)
    session.initialize(tris, 8, 8)
    nodes, order = session.export_bvh(n)
    assert nodes.tobytes() == scene.nodes().tobytes()
    assert _leaf_sets(nodes, order) == _leaf_sets(scene.nodes(), scene.order())
    q = rays(257)
    assert session.query(q).tobytes() == oracle.query(scene, q, False)[0].tobytes()


@pytest.mark.parametrize('far', (1e25, np.inf))
@pytest.mark.parametrize('n', (20, 40, 600, 3000))
def test_build_with_unbounded_boxes(session, oracle, sphere, n, far):
    """A vertex so far out that a box's area is infinite: no split is cheaper
    than the leaf, in the subtree, search and binned forms alike, so the nodes
    are the reference's. Nothing is asked of rays through an infinite box."""
    tris = some_triangles(sphere, n).copy()
    for axis in 'xyz':
        tris['origin'][axis][n // 2] = far
    scene = oracle.scene(tris)
    session.initialize(tris, 8, 8)
    nodes, order = session.export_bvh(n)
    assert nodes.tobytes() == scene.nodes().tobytes()
    assert _leaf_sets(nodes, order) == _leaf_sets(scene.nodes(), scene.order())
    if np.isfinite(far):
        q = rays(257)
        assert session.query(q).tobytes() == oracle.query(scene, q, False)[0].tobytes()


@pytest.mark.parametrize('offset', (-1, 0, 1))
def test_query_counts(session, oracle, sphere, offset):
    """Around a warp, a block and the count from which queries run as blocks
    of 128 (128 rays per multiprocessor), closest and any hit."""
    tris = some_triangles(sphere, 700)
    scene = oracle.scene(tris)
    session.initialize(tris, 8, 8)
    per_wave = 128 * torch.cuda.get_device_properties(0).multi_processor_count
    for base in (2, 32, 128, per_wave):
        q = rays(base + offset)
        assert session.query(q).tobytes() == oracle.query(scene, q, False)[0].tobytes(), len(q)
        any_hit = session.query(q, any_hit=True)['index'] >= 0
        assert (any_hit == (oracle.query(scene, q, True)[0]['index'] >= 0)).all(), len(q)


@pytest.mark.parametrize('w,h,samples', ((1, 1, 1), (45, 31, 3), (128, 12, 2)))
def test_pass_schedules(lib, w, h, samples):
    """A pass in one wave (dependent launches, shadow rays traced with the next
    bounce), in waves that end inside a row of samples or at its end (waves
    hold 1024 paths at least), and in the one-kernel integrator: the same
    sums, over two passes."""
    tris, cam, st, _, _ = scenes.cornell_sphere()
    cam.aspect = w / h
    st.raysPerPixel = samples
    total, out = w * h * samples, []
    for integrator, paths, lanes in ((0, 0, 2), (0, total, 1), (0, total - 1, 2), (0, w * h, 1), (0, 1025, 2),
                                     (1, 0, 1)):
        with Session(lib) as s:
            s.set_integrator(integrator)
            s.set_tuning(lanes=lanes)
            if paths:
                s.set_tuning(paths_in_flight=max(1024, paths))
            s.initialize(tris, w, h)
            for _ in range(2):
                s.render_device(cam, st)
            out.append(s.accumulation().tobytes())
    assert all(o == out[0] for o in out)


def filter_restated(sums, samples, w, h):
    """The guided filter in float64: 5 passes of 25 taps, taps 1 .. 16 apart."""
    def field(name):
        return np.stack([sums[name][ax] for ax in 'xyz'], -1).astype(np.float64).reshape(h, w, 3)
    c, a, n = field('radiance') / samples, field('albedo') / samples, field('normal')
    n = n / np.maximum(np.linalg.norm(n, axis=-1, keepdims=True), 1e-30)
    covered = sums['covered'].reshape(h, w) != 0
    kernel = (3 / 8, 1 / 4, 1 / 16)
    inv_phi = 2.0
    for it in range(5):
        total, weights = np.zeros_like(c), np.zeros((h, w))
        for dy in range(-2, 3):
            for dx in range(-2, 3):
                sy, sx = dy << it, dx << it
                y0, y1, x0, x1 = max(0, -sy), min(h, h - sy), max(0, -sx), min(w, w - sx)
                if y0 >= y1 or x0 >= x1:
                    continue
                here, there = (slice(y0, y1), slice(x0, x1)), (slice(y0 + sy, y1 + sy), slice(x0 + sx, x1 + sx))
                wt = kernel[abs(dx)] * kernel[abs(dy)] * np.exp(-((c[there] - c[here]) ** 2).sum(-1) * inv_phi)
                wt *= np.exp(-((a[there] - a[here]) ** 2).sum(-1) / 0.02)
                wt *= np.maximum(0, (n[there] * n[here]).sum(-1)) ** 64
                wt *= covered[there] & covered[here]
                total[here] += c[there] * wt[..., None]
                weights[here] += wt
        with np.errstate(invalid='ignore', divide='ignore'):
            c = np.where((weights > 0)[..., None], total / weights[..., None], c)
        inv_phi *= 2
    return np.where(covered[..., None], c, 0)


@pytest.mark.parametrize('w,h', ((1, 1), (33, 17), (31, 70), (97, 49)))
def test_filter_tiles(lib, w, h):
    """The filter's tiles (32 x 16 points of a lattice per step) against a
    float64 restatement. A tap's float32 weight is off by at most (64 + 100 +
    4) 2^-23 = 2e-5 of itself (power 64, exponents to -100), so a pass by 4e-5
    of the brightest colour C; a later pass's colour weights turn an error d
    into 2 x 0.56 x 32 d: 5e-3 C bounds the five, and 1e-4 C their mean."""
    tris, cam, st, _, _ = scenes.cornell_sphere()
    cam.aspect = w / h
    st.raysPerPixel = 4
    with Session(lib) as s:
        s.initialize(tris, w, h)
        s.render_device(cam, st)
        s.denoise()
        got = s.denoised_radiance().reshape(h, w, 3)
        expect = filter_restated(s.accumulation(), s.sample_count(), w, h)
    diff, top = np.abs(got - expect), expect.max()
    assert diff.max() <= 5e-3 * top and diff.mean() <= 1e-4 * top, (diff.max() / top, diff.mean() / top)


@pytest.mark.parametrize('h,w', ((16, 16), (16, 1024), (80, 1040), (272, 480), (528, 464), (1088, 96)))
def test_convolutions_identical(lib, net, h, w):
    """Tiles that span rows (images up to 64 pixels wide, column segments of
    small wider ones, the streamed 224 -> 96 layer) accumulate in the order of
    the kernels they stand in for: the same image, at level widths on both
    sides of 64, 128 and the limit on the image's pixels."""
    aovs, _ = synthetic(np.random.default_rng(h + w), 1, h, w)
    try:
        assert lib.RtxSetConvPath(2)
        expect = net.infer(aovs[0])
        assert lib.RtxSetConvPath(0)
        assert np.array_equal(net.infer(aovs[0]), expect)
    finally:
        lib.RtxSetConvPath(0)


@pytest.mark.parametrize('n,h,w', ((1, 16, 16), (3, 16, 176), (1, 144, 16), (2, 80, 112), (1, 32, 272), (5, 128, 256)))
def test_gradients_at_edges(net, n, h, w):
    """Weight gradients (segments of 16 to 128 pixels, column taps along N or
    not), the head, the pre-activation gradients and the data gradients against
    PyTorch, with the bounds of test_gpu_unet (5% of each layer's gradient,
    cosine 0.99). Targets lie far above any prediction, so that rounding flips
    no sign of the L1 loss."""
    aovs, target = synthetic(np.random.default_rng(n * h * w), n, h, w)
    target = target + np.float32(1e4)
    loss, grads = net.loss_grad(aovs, target)
    params = unpack(net.params())
    t = torch.tensor(np.log1p(target)).permute(0, 3, 1, 2)
    ref = (forward(features(aovs), params) - t).abs().mean()
    ref.backward()
    assert abs(loss - ref.item()) <= 5e-3 * ref.item()
    expect, off = pack_grads(params), 0
    for size in [s for ci, co in layer_table() for s in (9 * ci * co, co)] + [96, 3]:
        g, e = grads[off:off + size].astype(np.float64), expect[off:off + size].astype(np.float64)
        off += size
        norm = np.linalg.norm(e)
        assert np.linalg.norm(g - e) <= 5e-2 * norm, (off, np.linalg.norm(g - e) / norm)
        assert norm == 0 or g @ e >= 0.99 * np.linalg.norm(g) * norm, off
    assert off == grads.size


def test_device_memory_is_shared_and_given_back(lib, sphere):
    """Sessions that come and go reuse device memory, also from two threads at
    once, with the results of a session alone; what is kept is given back with
    the last session."""
    _, cam, st, _, _ = scenes.cornell_sphere()
    cam.aspect = 1.0
    st.raysPerPixel = 2

    def run(size):
        with Session(lib) as s:
            s.initialize(sphere, size, size)
            s.render_device(cam, st)
            return s.accumulation().tobytes()
    expect = {size: run(size) for size in (40, 64)}
    free = torch.cuda.mem_get_info()[0]
    results = []

    def worker(sizes):
        for size in sizes:
            results.append(run(size) == expect[size])
    threads = [threading.Thread(target=worker, args=(sizes,)) for sizes in ((40, 64) * 4, (64, 40) * 4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert len(results) == 16 and all(results)
    assert torch.cuda.mem_get_info()[0] >= free - (64 << 20)


def test_queries_beside_a_graph_capture(lib, sphere):
    """A batch that records a CUDA graph for every frame (its settings change)
    in one thread, and queries, scene loads and gradients, whose buffers come
    and go, in others: every call succeeds with its usual result."""
    from native_api import Batch, NativeError, Settings
    _, cam, _, _, _ = scenes.cornell_sphere()
    cam.aspect = 1.0
    q = rays(1500)
    aovs, target = synthetic(np.random.default_rng(1), 1, 32, 32)

    def images(batch, view, frames):
        out = []
        for k in range(frames):
            batch.render(Settings(2, 1.0, 0.0, 1.0, 0.5, 1 + k % 2, 1))
            out.append(batch.image(view).tobytes())
        return out

    def frames(count):
        batch = Batch(lib)
        try:
            view = batch.add_view(batch.add_scene(sphere), cam, 48, 48)
            return images(batch, view, count)
        finally:
            batch.close()

    def queries(count):
        out = []
        for _ in range(count):
            with Session(lib) as s:
                s.initialize(sphere, 8, 8)
                out += [s.query(q).tobytes() for _ in range(8)]
        return out

    def gradients(count):
        n = Unet(lib, seed=2)
        try:
            losses = [n.loss_grad(aovs, target)[0] for _ in range(count)]  # equal to the order of their sums
            return [max(losses) - min(losses) <= 1e-5 * min(losses)]
        finally:
            n.close()
    jobs = ((frames, 2, 150), (queries, 1, 30), (gradients, 1, 100))
    expect = {job: set(job(few)) for job, few, _ in jobs}
    results, errors = {}, []

    def work(job, many):
        try:
            results[job] = set(job(many))
        except NativeError as e:
            errors.append((job.__name__, str(e)))
    threads = [threading.Thread(target=work, args=(job, many)) for job, _, many in jobs]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    assert results == expect


def test_convolution_counts_name_the_kernel(lib, net):
    """The counts go by order of accumulation; the row-spanning kernel's own say
    how many of them it ran: none where a path switch leaves it out."""
    import ctypes
    aovs, _ = synthetic(np.random.default_rng(4), 1, 64, 256)

    def counts():
        pipe, single = ctypes.c_longlong(), ctypes.c_longlong()
        lib.RtxConvLaunchCounts(ctypes.byref(pipe), ctypes.byref(single))
        return np.array((pipe.value, single.value, lib.RtxConvRowSpanLaunches()))
    try:
        got = {}
        for mode in (0, 1, 2):
            assert lib.RtxSetConvPath(mode)
            before = counts()
            net.infer(aovs[0])
            got[mode] = tuple(counts() - before)
    finally:
        lib.RtxSetConvPath(0)
    assert got[1] == (0, 18, 0) and got[2] == (20, 1, 0)
    # Levels 2 to 4 (64, 32 and 16 pixels wide) and 224 -> 96: 6 layers down, 4 up,
    # one of them in two passes, at least.
    assert got[0][:2] == (20, 1) and 11 <= got[0][2] <= 21, got[0]
