"""The FP32 policy kernels (csrc/mlp.cu) at the edges of their tiles, each product against FP64 on the inputs the GPU
itself had for it. An output is a chain of K fused multiply-adds (split sums included), so its error is at most
K * 2^-24 times the sum of its terms' magnitudes (K counts the chain and its splits; 2 more for the roundings around
it); tanhf adds 2 ulps, at most 2^-22, and maps an error to at most itself."""
import numpy as np
import pytest

import warporacer3d_gb300 as W

pytestmark = pytest.mark.gpu

U = 2.0 ** -24


def within(got, a, b, chain, extra=0.0, scale=1.0):
    """got is a @ b (times scale elementwise) up to the error of `chain` roundings."""
    want, mag = (a @ b) * scale, (np.abs(a) @ np.abs(b)) * np.abs(scale)
    err = np.abs(got.astype(np.float64) - want)
    assert np.all(err <= (chain + 4) * U * mag + extra + 1e-37), err.max()


# inputs: one k-chunk with a remainder, whole chunks, the widest; samples: one, either side of a 32-sample block, either
# side of the 64-sample kernel's threshold, a split of the batch with a remainder
@pytest.mark.parametrize("beams,cols", [(2, 1), (27, 31), (59, 33), (108, 1023), (108, 19391), (1081, 65), (123, 19457),
                                        (100, 5000)])
def test_fp32_products(beams, cols):
    rng = np.random.default_rng(beams * cols)
    n = beams + 5
    p = W.Policy(5, beams=beams)
    p.set_precision("fp32")
    theta = p.theta.numpy()
    theta[:-2] += rng.normal(0, 0.05, p.P - 2).astype(np.float32)
    p.theta.write(theta)
    p.sync()
    w0 = theta[:p.W1].reshape(64, n).astype(np.float64)
    w1 = theta[p.W1:p.W2].reshape(64, 65).astype(np.float64)
    w2 = theta[p.W2:p.LOGSTD].reshape(3, 65).astype(np.float64)
    x = rng.uniform(-1, 1, (n, cols)).astype(np.float32)
    xd = W.DevArray.empty((n, cols))
    xd.write(x)
    acts = W.Activations(p, cols)
    p.forward(xd, acts)
    h1, h2, o = acts.h1.numpy(), acts.h2.numpy(), acts.o.numpy()
    assert np.all(h1[64] == 1) and np.all(h2[64] == 1)
    for h, w, inp in ((h1, w0, x), (h2, w1, h1)):
        pre = w @ inp.astype(np.float64)
        err = np.abs(h[:64] - np.tanh(pre))
        assert np.all(err <= (inp.shape[0] + 2) * U * (np.abs(w) @ np.abs(inp.astype(np.float64))) + 2.0 ** -22), err.max()
    within(o, w2, h2.astype(np.float64), 65)
    d3 = rng.normal(0, 1 / cols, (3, cols)).astype(np.float32)
    d3d = W.DevArray.empty((3, cols))
    d3d.write(d3)
    back = [W.DevArray.empty((65, cols)), W.DevArray.empty((65, cols)), W.DevArray.empty((p.P,))]
    p.backward(xd, acts, d3d, *back)
    d2, d1, g = (b.numpy() for b in back)
    f64 = np.float64
    within(d2, w2.T, d3.astype(f64), 3, scale=1 - h2.astype(f64) ** 2)
    within(d1, w1.T, d2[:64].astype(f64), 64, scale=1 - h1.astype(f64) ** 2)
    for got, a, b in ((g[:p.W1].reshape(64, n), d1[:64], x), (g[p.W1:p.W2].reshape(64, 65), d2[:64], h1),
                      (g[p.W2:p.LOGSTD].reshape(3, 65), d3, h2)):
        within(got, a.astype(f64), b.astype(f64).T, cols)
    assert np.all(g[p.LOGSTD:] == 0)
