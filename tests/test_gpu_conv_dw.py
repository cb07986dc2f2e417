"""Weight gradients of the network (conv_dw.cu) at image sizes that end inside a tile of the
kernel (4 x 64 pixels) on every level, against the FP64 oracle."""
import warnings

import numpy as np
import pytest

from oracle import unet_oracle as U
from pyom2_b200 import learned, synth
from pyom2_b200.external import ExternalMode
from pyom2_b200.model import ModelState

pytestmark = pytest.mark.gpu


def trainer(nx, ny, params):
    M = ModelState(nx, ny, 1, enable_cyclic_x=False, coord_degree=False)
    M.dxt[2:nx + 2] = M.dyt[2:ny + 2] = 1e4
    M.dzt[:] = 100.0
    synth.calc_grid(M)
    M.kbot[2:nx + 2, 2:ny + 2] = 1
    synth.calc_topo(M)
    E = ExternalMode(M)
    with warnings.catch_warnings():
        warnings.simplefilter("ignore", RuntimeWarning)
        E.streamfunction_init(maxipp=10**6, maxq=10**6)
    return learned.LearnedPreconditioner(E, params=params, training=True)


def layer_slices():
    o, out = 0, []
    for ci, co in learned.LAYERS:
        out.append((slice(o, o + 9 * ci * co), (co, ci, 3, 3)))
        o += 9 * ci * co
    return out, o


SIZES = [(8, 8), (64, 8), (72, 24), (136, 40), (200, 88)]


def copying_params():
    """Weights that copy channels (centre tap 1 for ci = co mod Cin; the output sums its inputs)."""
    p = np.zeros(learned.num_params(), dtype=np.float32)
    sl, _ = layer_slices()
    for k, (s, shape) in enumerate(sl):
        w = np.zeros(shape, dtype=np.float32)
        if k == 11:
            w[0, :, 1, 1] = 1.0
        else:
            for co in range(shape[0]):
                w[co, co % shape[1], 1, 1] = 1.0
        p[s] = w.ravel()
    return p


@pytest.mark.parametrize("nx,ny", SIZES)
def test_gradients_exactly(nx, ny):
    """Every layer, level and tap: with copying weights and inputs and output gradients that are constant on
    8 x 8 blocks (0/1 and -1/0/1), activations and gradients are small integers times powers of two, exact in
    bf16, and every sum of products is an integer multiple of one power of two below 2**24 of it, exact in FP32
    in any order: the gradients equal the oracle's."""
    p = copying_params()
    pc = trainer(nx, ny, p)
    rng = np.random.default_rng(nx)
    blocks = lambda a: np.kron(a, np.ones((8, 8)))
    x0 = np.stack([blocks(rng.integers(0, 2, (ny // 8, nx // 8))) for _ in range(16)])
    gz = blocks(rng.integers(-1, 2, (ny // 8, nx // 8)).astype(float)).astype(np.float32)
    z = pc.forward_backward(U.bf16_bits(U.to_planar(x0)), gz)
    g = pc.get_grads()
    zo, A = U.unet_forward(p, x0, emulate=False)
    want = U.unet_backward(p, A, gz.astype(np.float64), emulate=False)
    assert np.array_equal(z, zo)
    assert np.array_equal(g, want)
    pc.close()


@pytest.mark.parametrize("nx,ny", SIZES)
def test_output_layer_gradient_to_fp32(nx, ny):
    """With zero weights the output layer's input is the constant S1 + c10 bias of a channel, so its gradient
    is that constant times the sum of the output gradient over the tap's window: bf16 operands, FP32 sums
    (1e-5 of the sum of magnitudes)."""
    sl, o = layer_slices()
    p = np.zeros(learned.num_params(), dtype=np.float32)
    b1, b10 = 0.5 + np.arange(16) / 16.0, 1.0 + np.arange(16) / 8.0  # exact in bf16
    off = np.cumsum([0] + [co for _, co in learned.LAYERS])
    p[o + off[1]:o + off[1] + 16] = b1
    p[o + off[10]:o + off[10] + 16] = b10
    pc = trainer(nx, ny, p)
    rng = np.random.default_rng(ny)
    gz = rng.standard_normal((ny, nx)).astype(np.float32)
    pc.forward_backward(np.zeros((2, ny, nx, 8), dtype=np.uint16), gz)
    g = pc.get_grads()
    gb = U.bf16_round(gz.astype(np.float64))
    u1 = U.bf16_round(b1 + b10)
    s, shape = sl[11]
    got = g[s].reshape(shape).astype(np.float64)
    for dy in range(3):
        for dx in range(3):
            # pixels whose neighbour (dy-1, dx-1) lies inside the image
            w = gb[max(0, 1 - dy):ny - max(0, dy - 1), max(0, 1 - dx):nx - max(0, dx - 1)]
            assert np.all(np.abs(got[0, :, dy, dx] - u1 * w.sum()) <= 1e-5 * u1 * np.abs(w).sum()), (dy, dx)
    assert np.all(got[1:] == 0.0)
    assert abs(g[o + off[11]] - gb.sum()) <= 1e-5 * np.abs(gb).sum()
    pc.close()


def test_sums_do_not_drift():
    """The gradient of the output layer against the exact sums of the same bf16 operands, all positive, so that a
    rounding of one sign in the accumulation adds up.  Sums of four products of 16 pixels each may be truncated
    (on average half a unit of 2**-23 of the running sum, at most a whole one): the mean error is at most
    (1/4 + 2/4 + 3/4 + 1) 2**-24 2 = 3e-7 of the sum, and half of that expected; rounded sums on top of them (four
    a tile of 4 x 64 pixels and one a block) scatter by less than sqrt(400) 2**-24 and have no mean."""
    nx, ny = 1440, 720
    sl, _ = layer_slices()
    p = np.zeros(learned.num_params(), dtype=np.float32)
    for k in (0, 1):  # the first level's activations are the input, the coarser levels add nothing
        w = np.zeros(sl[k][1], dtype=np.float32)
        w[np.arange(16), np.arange(16), 1, 1] = 1.0
        p[sl[k][0]] = w.ravel()
    pc = trainer(nx, ny, p)
    rng = np.random.default_rng(2)
    x = U.bf16_round(rng.uniform(0.5, 1.5, (16, ny, nx)))
    gz = np.abs(rng.standard_normal((ny, nx))).astype(np.float32)
    pc.forward_backward(U.bf16_bits(U.to_planar(x)), gz)
    s, shape = sl[11]
    got = pc.get_grads()[s].reshape(shape)[0].astype(np.float64)
    pc.close()
    xp, g = np.pad(x, ((0, 0), (1, 1), (1, 1))), U.bf16_round(gz.astype(np.float64))
    want = np.empty((16, 3, 3))
    for dy in range(3):
        for dx in range(3):
            want[:, dy, dx] = (xp[:, dy:dy + ny, dx:dx + nx] * g).sum(axis=(1, 2))
    err = got / want - 1.0
    assert abs(err.mean()) <= 2.5 * 2.0 ** -23
    assert err.std() <= 20 * 2.0 ** -24
