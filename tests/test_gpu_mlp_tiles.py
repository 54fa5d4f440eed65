"""The warm-start MLP's product kernel on 64 x 64 tiles (at least 96 of them and
no sum above 512 terms; smaller calls take 32 x 32) against the oracle, at the
tolerances of the network's other tests: the 2049-wide output layer from 129
rows on with the fused loss, and a network of ragged widths whose paired
backward launches and hidden layers take them, transposed operands included."""
import numpy as np
import pytest

from oracle import mlp_oracle as mo
from pincosimulator_gb300 import twmc

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

FULL, RAGGED = [5, 256, 256, 256, 2049], [5, 501, 509, 333]


def setup_net(widths, batch, seed):
    rng = np.random.default_rng(seed)
    p = mo.init_params(widths, seed=seed)
    offs, _ = mo.offsets(widths)
    for (_, bo), m in zip(offs, widths[1:]):
        p[bo:bo + m] = 0.1 * rng.normal(size=m)
    net = twmc.MLP(widths, batch, 1)
    net.set_params(p)
    x = rng.uniform(-1, 1, size=(batch, widths[0])).astype(np.float32)
    t = rng.normal(size=(batch, widths[-1])).astype(np.float32)
    return net, p, x, t


def nrel(a, b):
    return np.linalg.norm(a - b) / max(np.linalg.norm(b), 1e-30)


@pytest.mark.parametrize("widths,batch", [(FULL, 129), (FULL, 256), (RAGGED, 1021)])
def test_forward(built_lib, widths, batch):
    net, p, x, _ = setup_net(widths, batch, 1)
    xd = torch.as_tensor(x).cuda()
    y = torch.zeros(batch, widths[-1], dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    net.forward(xd.data_ptr(), batch, y.data_ptr())
    torch.cuda.synchronize()
    ref, _ = mo.forward(p, widths, x)
    assert nrel(y.cpu().numpy(), ref) < 2e-3
    net.close()


@pytest.mark.parametrize("widths,batch", [(FULL, 129), (FULL, 256), (RAGGED, 511)])
def test_backward(built_lib, widths, batch):
    net, p, x, t = setup_net(widths, batch, 2)
    w = np.random.default_rng(3).uniform(0.5, 1.5, size=widths[-1]).astype(np.float32)
    xd, td, wd = (torch.as_tensor(a).cuda() for a in (x, t, w))
    torch.cuda.synchronize()
    loss = net.backward(xd.data_ptr(), td.data_ptr(), batch, wd.data_ptr(), want_loss=True)
    g = net.get_grads()
    lref, gref, _ = mo.backward(p, widths, x, t, w)
    assert abs(loss - lref) < 2e-3 * lref
    offs, _ = mo.offsets(widths)
    for l, ((wo, bo), k, m) in enumerate(zip(offs, widths[:-1], widths[1:])):
        assert nrel(g[wo:wo + m * k], gref[wo:wo + m * k]) < 1e-2, f"dW layer {l}"
        assert nrel(g[bo:bo + m], gref[bo:bo + m]) < 1e-2, f"db layer {l}"
    net.close()


def test_a_row_does_not_depend_on_the_tile(built_lib):
    """128 rows of the full network run on 32 x 32 tiles throughout, 129 on 64 x 64
    in the output layer: the same bits, since a sum's terms are added in the
    same order."""
    net, _, x, _ = setup_net(FULL, 129, 4)
    xd = torch.as_tensor(x).cuda()
    y = torch.zeros(2, 129, FULL[-1], dtype=torch.float32, device="cuda")
    torch.cuda.synchronize()
    net.forward(xd.data_ptr(), 128, y[0].data_ptr())
    net.forward(xd.data_ptr(), 129, y[1].data_ptr())
    torch.cuda.synchronize()
    assert torch.equal(y[0, :128], y[1, :128])
    net.close()


@pytest.mark.parametrize("widths", [[5, 64, 48, 37], [5, 256, 256, 256, 513], FULL])
def test_adam_rounds_alike_for_every_size(built_lib, widths):
    """One parameter per thread (small networks) or four: the same operations in
    FP32, m = fma(1 - b1, g, b1 m) and v = fma((1 - b2) g, g, b2 v), bit for
    bit over three steps."""
    net, p, x, t = setup_net(widths, 64, 6)
    xd, td = torch.as_tensor(x).cuda(), torch.as_tensor(t).cuda()
    torch.cuda.synchronize()
    f = np.float32
    lr, b1, b2, eps, one = f(2e-3), f(0.9), f(0.999), f(1e-8), f(1)

    def fma(a, b, c):
        return (np.float64(a) * np.float64(b) + np.float64(c)).astype(f)  # the product is exact

    w = p.astype(f)
    m, v = np.zeros_like(w), np.zeros_like(w)
    for step in range(1, 4):
        net.backward(xd.data_ptr(), td.data_ptr(), 64)
        g = net.get_grads()
        net.adam(2e-3)
        m = fma(one - b1, g, b1 * m)
        v = fma((one - b2) * g, g, b2 * v)
        c1, c2 = f(1 / (1 - float(b1) ** step)), f(1 / (1 - float(b2) ** step))
        w = w - lr * (m * c1) / (np.sqrt(v * c2) + eps)
        assert np.array_equal(net.get_params(), w), step
    net.close()
