"""Graph-convolution layers of every width against the CPU oracle, at the sizes where a kernel's tiles begin and end."""
import numpy as np
import pytest

import oracle as O
import parity as P
from visualmesh_b200 import workloads as W
from visualmesh_b200.engine import Engine

pytestmark = pytest.mark.gpu


def _rows(n, n_neighbours, seed):
    x = W.uniform(seed, n * 4, -1.0, 1.0).reshape(n, 4).astype(np.float32)
    nb = (W.splitmix64(seed + 1, n * n_neighbours) % np.uint64(n)).astype(np.int32).reshape(n, n_neighbours)
    nb[-1] = n - 1
    return x, nb


def _check(net, n, n_neighbours):
    x, nb = _rows(n, n_neighbours, 31 + n)
    engine = Engine(net)
    got = engine.network(x, nb)
    engine.close()
    assert np.abs(got.astype(np.float64) - O.network(x, nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


# on 148 SMs: part of the outputs per block up to 1036 blocks of 128 rows and eight outputs (24 outputs: up to 44160 rows), one row per
# thread up to 147 blocks of 512 rows (75264 rows), two from there on
@pytest.mark.parametrize("n", [1, 127, 129, 44_160, 44_161, 75_264, 75_265, 75_776, 75_777])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [24, 20, 12, 5]), (6, [7, 13, 3]), (8, [28, 32, 31, 2])])
def test_widths_without_a_kernel_of_their_own(n, n_neighbours, widths):
    _check(W.make_network(41, n_neighbours, widths), n, n_neighbours)


# the same for layers with a kernel of their own: 444 blocks (16 outputs: 28416 rows; 8 outputs: 56832), 148 for 12 outputs (9472 rows)
@pytest.mark.parametrize("n", [1, 128, 129, 9_472, 9_473, 28_416, 28_417, 56_832, 56_833, 75_264, 75_265])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [16, 8, 16, 5]), (6, [8, 16, 12, 12, 8, 3]), (8, [12, 16, 4, 32, 16, 2])])
def test_layers_with_a_kernel_of_their_own(n, n_neighbours, widths, monkeypatch):
    monkeypatch.setenv("VMCUDA_TC", "0")
    _check(W.make_network(53, n_neighbours, widths), n, n_neighbours)


@pytest.mark.parametrize("activation", [W.SELU, W.RELU, W.TANH, W.SOFTMAX])
def test_odd_widths_inside_a_group(activation):
    """Dense layers behind a gather, their widths padded with channels of zeros: a softmax in the middle must not count them."""
    rng = np.random.default_rng(3)
    net, width = [], 4
    for group in ([6, 5], [9, 3]):
        net.append([])
        for i, out in enumerate(group):
            fan_in = width * (7 if i == 0 else 1)
            w = rng.uniform(-1, 1, (fan_in, out)).astype(np.float32) * np.float32(np.sqrt(6.0 / (fan_in + out)))
            net[-1].append(W.Layer(w, rng.uniform(-0.1, 0.1, out).astype(np.float32), activation))
            width = out
    net[-1][-1].activation = W.SOFTMAX
    _check(net, 1000, 6)


# 256-row super-tiles of two 128-row tiles; 9472 rows are 37 super-tiles, 75776 and more are several per SM
@pytest.mark.parametrize("n", [1, 128, 129, 256, 257, 9_472, 90_001])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [32, 32, 32, 3]), (6, [16, 32, 32, 16, 16, 2]), (8, [32, 32, 20, 32, 32])])
def test_layers_of_32_channels(n, n_neighbours, widths):
    _check(W.make_network(43, n_neighbours, widths), n, n_neighbours)


def test_layers_of_32_channels_with_neighbours_close_by():
    """Neighbours inside the window (random ones all over the rows mostly are not)."""
    net = W.make_network(47, 8, [32, 32, 32, 4])
    n = 50_000
    x, _ = _rows(n, 8, 5)
    near = (W.splitmix64(6, n * 8) % np.uint64(61)).astype(np.int64).reshape(n, 8) - 30
    nb = np.clip(np.arange(n)[:, None] + near, 0, n - 1).astype(np.int32)
    engine = Engine(net)
    got = engine.network(x, nb)
    engine.close()
    assert np.abs(got.astype(np.float64) - O.network(x, nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


def _near(n, n_neighbours, reach):
    """Neighbours within `reach` rows, so that most lie in the row's own window."""
    near = (W.splitmix64(6, n * n_neighbours) % np.uint64(2 * reach + 1)).astype(np.int64).reshape(n, n_neighbours) - reach
    return np.clip(np.arange(n)[:, None] + near, 0, n - 1).astype(np.int32)


# tiles of 8 rows, groups of 32, super-tiles of 256; 113 921 rows are two super-tiles for some of 444 CTAs. Every layout in front of
# and behind a 16-channel layer: from the CUDA cores, from the window kernel and from one another, to either of them and to fp32
@pytest.mark.parametrize("n", [1, 7, 9, 31, 33, 255, 257, 9_472, 113_921])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [16, 16, 8, 3]), (6, [8, 16, 32, 32, 16, 16, 8, 2]), (8, [16, 32, 16, 12, 16, 8, 5])])
@pytest.mark.parametrize("activation", [W.SELU, W.TANH])
def test_layers_of_16_channels_with_neighbours_close_by(n, n_neighbours, widths, activation):
    net = W.make_network(59, n_neighbours, widths)
    for group in net[:-1]:
        group[0].activation = activation
    x, _ = _rows(n, n_neighbours, 7)
    nb = _near(n, n_neighbours, 40)
    engine = Engine(net)
    got = engine.network(x, nb)
    engine.close()
    assert np.abs(got.astype(np.float64) - O.network(x, nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


# random neighbours lie outside the window, most of them beyond its halo
@pytest.mark.parametrize("n", [1, 33, 257, 9_473])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [16, 16, 8, 3]), (6, [16, 32, 16, 16, 8, 2]), (8, [16, 16, 8, 5])])
def test_layers_of_16_channels_with_neighbours_anywhere(n, n_neighbours, widths):
    _check(W.make_network(61, n_neighbours, widths), n, n_neighbours)


# super-tiles with 200, 340 and 460 outside rows: more than the staged kernel keeps, than the window kernel's loaders read ahead, than
# the plan has slots for; 64-row tiles and their edges
@pytest.mark.parametrize("reach", [100, 170, 230])
@pytest.mark.parametrize("n", [63, 65, 20_001])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [32, 32, 16, 16, 3]), (6, [16, 16, 32, 32, 8, 3]), (8, [32, 32, 32, 4])])
def test_layers_with_large_halos(n, reach, n_neighbours, widths):
    net = W.make_network(67, n_neighbours, widths)
    x, _ = _rows(n, n_neighbours, 11)
    nb = _near(n, n_neighbours, reach)
    engine = Engine(net)
    got = engine.network(x, nb)
    engine.close()
    assert np.abs(got.astype(np.float64) - O.network(x, nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


# three blocks per SM walk the super-tiles: three or more windows each from 227 329 rows on. Halos of 30 to 520 rows in any order: windows
# that share the pool with the one before, that wait for it, and super-tiles beyond the plan's slots
@pytest.mark.parametrize("n", [227_329, 350_001])
@pytest.mark.parametrize("n_neighbours,widths", [(4, [16, 16, 8, 3]), (6, [16, 32, 16, 16, 3]), (8, [16, 16, 8, 3])])
def test_layers_of_16_channels_with_halos_of_every_size(n, n_neighbours, widths):
    net = W.make_network(83, n_neighbours, widths)
    x, _ = _rows(n, n_neighbours, 19)
    reach = np.array([15, 90, 120, 170, 190, 260])[(W.splitmix64(8, n // 256 + 1) % np.uint64(6)).astype(np.int64)][np.arange(n) // 256]
    step = (W.splitmix64(9, n * n_neighbours) % (2 * reach.astype(np.uint64) + 1).repeat(n_neighbours)).astype(np.int64).reshape(n, n_neighbours)
    nb = np.clip(np.arange(n)[:, None] + step - reach[:, None], 0, n - 1).astype(np.int32)
    engine = Engine(net)
    got = engine.network(x, nb)
    engine.close()
    assert np.abs(got.astype(np.float64) - O.network(x, nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


# 296 blocks of 128 rows (32 channels: half super-tiles), 592 super-tiles or 296 blocks of 512 rows: up to there layers start early
@pytest.mark.parametrize("n", [1, 300, 37_888, 37_889, 151_552, 151_553])
@pytest.mark.parametrize("n_neighbours,widths", [(6, [16, 16, 16, 8, 8, 8, 5]), (8, [32, 32, 32, 16, 8, 4, 3])])
def test_layers_that_start_early(n, n_neighbours, widths):
    """Layers whose buffers take turns, over inputs that take turns: a row read too early would be another input's or another layer's."""
    net = W.make_network(71, n_neighbours, widths)
    x, _ = _rows(n, n_neighbours, 13)
    inputs = [x, np.ascontiguousarray(-x[::-1])]
    nb = _near(n, n_neighbours, 40)
    engine = Engine(net)
    got = [engine.network(inputs[i % 2], nb).copy() for i in range(6)]
    engine.close()
    for i, result in enumerate(got):
        if i >= 2:
            assert np.array_equal(result, got[i - 2])
            continue
        assert np.abs(result.astype(np.float64) - O.network(inputs[i], nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


# neighbours beyond every halo: rows that the layer in front writes are read past the windows, from memory
@pytest.mark.parametrize("n", [300, 37_888])
@pytest.mark.parametrize("n_neighbours,widths", [(6, [16, 16, 32, 32, 16, 16, 5]), (8, [16, 16, 16, 16, 8, 3]), (8, [32, 32, 32, 32, 4])])
def test_layers_that_start_early_with_neighbours_anywhere(n, n_neighbours, widths):
    net = W.make_network(79, n_neighbours, widths)
    x, nb = _rows(n, n_neighbours, 17)
    inputs = [x, np.ascontiguousarray(-x[::-1])]
    engine = Engine(net)
    got = [engine.network(inputs[i % 2], nb).copy() for i in range(6)]
    engine.close()
    for i, result in enumerate(got):
        if i >= 2:
            assert np.array_equal(result, got[i - 2])
            continue
        assert np.abs(result.astype(np.float64) - O.network(inputs[i], nb, net).astype(np.float64)).max() <= P.TOL_CLS / 4


def test_selu_over_its_range():
    """A layer that passes its input through: SELU of floats of every size, against double.

    The kernels write lambda alpha (e^s - 1) as one multiply-add of 2^(s log2 e). Its errors: the hardware's 2^x (2^-22.5 relative), the
    product s log2 e and its constant (together |s| 2^-23 of an exponential of e^s), the multiply-add (half an ulp of at most 1.76) and
    its rounded constant: 1.7581 (e^s 2^-22.5 + |s| e^s 2^-23) + 2^-24 + 2^-24 < 4.2e-7 for every s. The form with an exponential
    function, lambda (alpha exp(s) - alpha), rounds three times behind it and is no closer."""
    import torch
    down = -np.exp2(np.linspace(-30.0, 7.0, 3_000_000)).astype(np.float32)
    extremes = np.array([-0.0, 0.0, -1e-45, -1e-38, -87.0, -104.0, -1e4, -3e38, 1e-45, 1e-38, 3e38, 1.0], np.float32)
    up = np.exp2(np.linspace(-100.0, 100.0, 999_988)).astype(np.float32)
    ones = np.ones(4, np.float32)  # the last row, which every neighbour is: the zero weights of the gather meet finite values
    s = np.concatenate([down, up, extremes, ones]).reshape(-1, 4)
    n = len(s)
    weights = np.zeros((20, 4), np.float32)
    weights[:4] = np.eye(4, dtype=np.float32)
    net = [[W.Layer(weights, np.zeros(4, np.float32), W.SELU)]]
    nb = np.full((n, 4), n - 1, np.int32)
    lam, alpha = 1.0507009873554804934193349852946, 1.6732632423543772848170429916717
    x = s.astype(np.float64)
    want = np.where(x >= 0, lam * x, lam * alpha * np.expm1(np.minimum(x, 0)))
    engine = Engine(net)
    got = engine.network(s, nb).astype(np.float64)
    engine.close()
    error, negative = np.abs(got - want), x < 0
    alpha32 = float(np.float32(alpha))
    plain = (float(np.float32(lam)) * (alpha32 * torch.exp(torch.from_numpy(s).cuda()) - alpha32)).cpu().numpy().astype(np.float64)
    plain_error = np.abs(plain - want)[negative].max()
    print(f"selu: largest error {error[negative].max():.3g}, with an exponential function {plain_error:.3g}")
    assert error[negative].max() <= min(4.2e-7, plain_error)
    positive = x > 1e-37
    assert (error[positive] / want[positive]).max() <= 2.0**-23  # lambda rounded, the product rounded
    assert error[(x >= 0) & ~positive].max() <= 1e-44
