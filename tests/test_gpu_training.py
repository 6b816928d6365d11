"""Training (RtxUnetLossGrad, RtxUnetTrain) beyond one layer's tolerance: which
sums are taken together. Needs a GPU.

A network of unit weights makes every product exact: channel 0 of the input's
albedo passes unchanged through layers 0, 1, 16 and 17, channel 1 drives the
prediction, and the gradient at layer 17's pre-activation is +1 or -1 as the
target lies below or above it. The weight gradient between the two channels is
then a sum of chosen numbers over the pixels."""
import numpy as np
import pytest
import torch

from native_api import Unet
from test_gpu_unet import layer_table, synthetic

pytestmark = pytest.mark.gpu


@pytest.fixture(scope='module')
def net(lib):
    n = Unet(lib, seed=3)
    yield n
    n.close()


def offsets():
    """Flat offset of each 3x3 layer's weights, then the output layer's."""
    out, at = [], 0
    for ci, co in layer_table():
        out.append(at)
        at += 9 * ci * co + co
    return out + [at]


CENTRE = 4  # tap (0, 0)


def unit_network(net, pixels):
    """Sets the parameters described above for a batch of `pixels` pixels."""
    table, at = layer_table(), offsets()
    flat = np.zeros(net.param_count, np.float32)
    for layer, first in ((0, 3), (1, 0), (16, 48), (17, 0)):  # albedo is input channels 3-5; layer 16 reads [up 48, skip 32]
        ci, co = table[layer]
        for c in range(2):
            flat[at[layer] + (CENTRE * ci + first + c) * co + c] = 1.0
    # The gradient at the prediction is +-1 / (3 pixels): a weight of 3 pixels
    # makes it +-1 below, and the bias brings the prediction back to 1.
    assert 3 * pixels < 1 << 24
    flat[at[18] + 1 * 3 + 0] = 3 * pixels
    flat[at[18] + 96 + 0] = 1 - 3 * pixels
    net.set_params(flat)


def weight_between(net, values, sign):
    """The gradient of layer 17's centre weight from channel 0 to 1: the sum of
    values * sign over the pixels, as the kernel adds it."""
    n, h, w = values.shape
    unit_network(net, values.size)
    aovs = np.zeros((n, h, w, 10), np.float32)
    aovs[..., 3], aovs[..., 4] = values, 1.0
    target = np.zeros((n, h, w, 3), np.float32)
    target[..., 0] = np.where(sign > 0, 0.0, 1e30)
    _, grads = net.loss_grad(aovs, target)
    return float(grads[offsets()[17] + (CENTRE * 32 + 0) * 32 + 1])


@pytest.mark.parametrize('n,h,w', ((4, 128, 128), (32, 32, 32), (3, 80, 112), (2, 16, 16)))
def test_weight_gradient_groups(net, n, h, w):
    """A weight gradient's pixels are summed in groups of whole image rows in
    order, as many rows each as make two groups for three multiprocessors.
    Training from fresh Adam moments carries the rounding of these sums on, so
    they are part of its result. A number that swallows every 1 added between
    it and its negative shows which rows share a sum."""
    rows = n * h
    groups = min(rows, 2 * torch.cuda.get_device_properties(0).multi_processor_count // 3)
    per = -(-rows // groups)
    groups = -(-rows // per)
    for g in sorted({0, groups // 2, groups - 1}):
        first, last = g * per, min(rows, (g + 1) * per) - 1
        values = np.ones((rows, w), np.float32)
        sign = np.ones((rows, w), np.float32)
        values[first, 0] = values[last, w - 1] = 2.0 ** 40
        sign[last, w - 1] = -1.0
        got = weight_between(net, values.reshape(n, h, w), sign.reshape(n, h, w))
        assert got == (rows - (last - first + 1)) * w, (g, got)


@pytest.mark.parametrize('h,w', ((64, 96), (37, 23)))
def test_inference_after_training_is_the_same(lib, h, w):
    """A gradient of one image leaves buffers that inference of the same padded
    size uses: its result is a fresh network's, byte for byte."""
    aovs, target = synthetic(np.random.default_rng(h), 1, -(-h // 16) * 16, -(-w // 16) * 16)
    nets = [Unet(lib, seed=5), Unet(lib, seed=5)]
    try:
        nets[0].loss_grad(aovs, target)
        got, expect = (n.infer(np.ascontiguousarray(aovs[0, :h, :w])) for n in nets)
        assert np.array_equal(got, expect) and expect.max() > 0
    finally:
        for n in nets:
            n.close()


@pytest.mark.parametrize('n,h,w', ((32, 128, 128), (1, 16, 16), (7, 48, 112)))
def test_weight_gradient_is_exact(net, n, h, w):
    """Sums of small integers are exact in FP32 whatever their order: every row
    segment of every tap is there once, at a training batch as at one image."""
    rng = np.random.default_rng(n)
    values = rng.integers(0, 8, (n, h, w)).astype(np.float32)
    sign = rng.choice((-1.0, 1.0), (n, h, w))
    unit_network(net, values.size)
    aovs = np.zeros((n, h, w, 10), np.float32)
    aovs[..., 3], aovs[..., 4] = values, 1.0
    target = np.zeros((n, h, w, 3), np.float32)
    target[..., 0] = np.where(sign > 0, 0.0, 1e30)
    _, grads = net.loss_grad(aovs, target)
    at = offsets()[17]
    got = grads[at:at + 9 * 32 * 32].reshape(3, 3, 32, 32)[:, :, 0, 1]
    padded = np.pad(values, ((0, 0), (1, 1), (1, 1)))
    expect = [[(padded[:, dy:dy + h, dx:dx + w] * sign).sum() for dx in range(3)] for dy in range(3)]
    assert np.array_equal(got, np.array(expect, np.float32)), (got, expect)


def layer_slices():
    sizes = [s for ci, co in layer_table() for s in (9 * ci * co, co)] + [96, 3]
    ends = np.cumsum(sizes)
    return [slice(e - s, e) for s, e in zip(sizes, ends)]


@pytest.mark.parametrize('n,h,w', ((32, 64, 96), (32, 128, 128), (16, 112, 80)))
def test_batch_gradient_is_the_mean_of_its_images(lib, n, h, w):
    """Images do not see one another, and a batch size that is a power of two
    scales every gradient exactly, so a batch's gradient is the mean of its
    images' up to FP32 summation: at most 336 additions of 2^-23 per accumulator
    (4e-5), taken as 1e-4 of each layer's norm. A strip or segment lost where
    blocks walk many would be a hundred times that."""
    aovs, target = synthetic(np.random.default_rng(n + h), n, h, w)
    net = Unet(lib, seed=5)
    try:
        loss, grads = net.loss_grad(aovs, target)
        each = [net.loss_grad(aovs[i:i + 1], target[i:i + 1]) for i in range(n)]
    finally:
        net.close()
    assert abs(loss - np.mean([e[0] for e in each])) <= 1e-5 * loss
    mean = np.mean([e[1].astype(np.float64) for e in each], axis=0)
    for k, s in enumerate(layer_slices()):
        norm = np.linalg.norm(mean[s])
        assert norm > 0 and np.linalg.norm(grads[s] - mean[s]) <= 1e-4 * norm, (k // 2, np.linalg.norm(grads[s] - mean[s]) / norm)


def test_adam_step_and_its_copies(lib):
    """One step of RtxUnetTrain on one crop against Adam's formula on
    RtxUnetLossGrad's gradient (the crop is not flipped at this seed), and the
    BF16 copies that a step leaves against those of RtxUnetSetParams."""
    lr = np.float32(1e-3)
    seed = next(s for s in range(100) if np.random.RandomState(s).randint(0, 2 ** 32, size=2, dtype=np.uint32)[1] & 3 == 0)
    aovs, target = synthetic(np.random.default_rng(2), 1, 48, 64)
    net, other = Unet(lib, seed=5), Unet(lib, seed=6)
    try:
        p = net.params()
        loss, g = net.loss_grad(aovs, target)
        losses = net.train(aovs, target, steps=1, batch=1, lr=float(lr), seed=seed)
        assert abs(losses[0] - loss) <= 1e-5 * loss
        moved = net.params()
        one, b1, b2 = np.float32(1), np.float32(0.9), np.float32(0.999)
        m, v = (one - b1) * g, (one - b2) * g * g
        expect = p - lr * (m / (one - b1)) / (np.sqrt(v / (one - b2)) + np.float32(1e-8))
        # An update is lr g / (|g| + 1e-8): beyond 1e-6 a gradient's own rounding
        # (1e-6 of it) moves it by 1e-8 of lr.
        sure = np.abs(g) > 1e-6
        assert sure.mean() > 0.5
        assert (np.abs(moved - expect)[sure] <= 2 * np.spacing(np.abs(p[sure])) + 1e-5 * lr).all()
        assert (np.abs(moved - p) <= 1.00001 * lr + 2 * np.spacing(np.abs(p))).all()
        assert np.array_equal(moved[g == 0], p[g == 0]) and (g == 0).any()
        net.train(aovs, target, steps=3, batch=1, lr=float(lr), seed=seed)
        other.set_params(net.params())
        assert np.array_equal(net.infer(aovs[0]), other.infer(aovs[0]))
        a, b = net.loss_grad(aovs, target)[1], other.loss_grad(aovs, target)[1]
        assert np.linalg.norm(a - b) <= 1e-5 * np.linalg.norm(b)
    finally:
        net.close()
        other.close()
