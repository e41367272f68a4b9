"""The predictor network: the CPU oracle (oracle/mlp_oracle.py) pinned by
finite differences, and the GPU forward/backward/Adam kernels
(zerork_b200/csrc/mlp.cu) checked against the oracle.

GPU tolerances: products accumulate in FP32 on the GPU and FP64 in the
oracle, which only moves BF16 roundings of the intermediate values; every
gradient tensor must agree within 1e-2 relative (L2) and every output within
1e-2 of the output scale.
"""
import numpy as np
import pytest

import mlp_oracle as mo
from conftest import have_gpu


def _net(rng, n_in, hidden, layers, n_out):
    d = mo.dims(n_in, hidden, layers, n_out)
    w = np.concatenate([
        (rng.standard_normal((d[l], d[l + 1])) / np.sqrt(d[l])).astype(np.float32).ravel()
        for l in range(len(d) - 1)])
    b = (0.1 * rng.standard_normal(sum(d[1:]))).astype(np.float32)
    # zero the padding rows/columns, as the library keeps them
    W, B = mo.unpack(w, b, d)
    for l, Wl in enumerate(W):
        kin = n_in if l == 0 else hidden
        kout = n_out if l == len(W) - 1 else hidden
        Wl[kin:, :] = 0.0
        Wl[:, kout:] = 0.0
        B[l][kout:] = 0.0
    return d, w, b


def test_bf16_rounding():
    x = np.array([1.0, 1.00390625, 1.005859375, -2.5, 3.0e-39, 65504.0], np.float32)
    r = mo.bf16(x)
    assert r[0] == 1.0 and r[1] == 1.0  # tie to even
    assert r[2] == np.float32(1.0078125)
    assert r[3] == -2.5
    assert np.all(np.isfinite(r))


def test_oracle_gradient_matches_finite_differences(monkeypatch):
    rng = np.random.default_rng(1)
    monkeypatch.setattr(mo, "bf16", lambda a: np.asarray(a, np.float32))  # exact arithmetic
    d, w, b = _net(rng, 7, 16, 2, 5)
    x = rng.standard_normal((32, 7)).astype(np.float32)
    t = rng.standard_normal((32, 5))
    _, gw, gb, _ = mo.forward_backward(w, b, d, x, t)
    n, n_out = t.shape
    for idx in rng.choice(np.flatnonzero(w), 12, replace=False):
        e = 1e-3
        wp, wm = w.copy(), w.copy()
        wp[idx] += e
        wm[idx] -= e
        lp = mo.forward_backward(wp, b, d, x, t)[0] / (n * n_out)
        lm = mo.forward_backward(wm, b, d, x, t)[0] / (n * n_out)
        assert abs((lp - lm) / (2 * e) - gw[idx]) <= 2e-3 * max(1e-3, abs(gw[idx]))
    for idx in rng.choice(np.flatnonzero(b), 6, replace=False):
        e = 1e-3
        bp, bm = b.copy(), b.copy()
        bp[idx] += e
        bm[idx] -= e
        lp = mo.forward_backward(w, bp, d, x, t)[0] / (n * n_out)
        lm = mo.forward_backward(w, bm, d, x, t)[0] / (n * n_out)
        assert abs((lp - lm) / (2 * e) - gb[idx]) <= 2e-3 * max(1e-3, abs(gb[idx]))


@pytest.fixture(scope="module")
def torch():
    if not have_gpu():
        pytest.skip("no CUDA device")
    import torch
    return torch


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,n_out,batch", [(163, 161, 64), (14, 12, 48)])
def test_gpu_gradients_match_oracle(torch, n_in, n_out, batch):
    from zerork_b200.predictor import Mlp
    rng = np.random.default_rng(2)
    net = Mlp(n_in, n_out, 256, 3, seed=3)
    d = mo.dims(n_in, 256, 3, n_out)
    _, w, b = _net(rng, n_in, 256, 3, n_out)
    net.set_params(w, b)
    x = rng.standard_normal((batch, n_in)).astype(np.float32)
    t = rng.standard_normal((batch, n_out)).astype(np.float32)
    xd, td = torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda()
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    net.gradients(xd, td, loss)
    gw, gb = net.grads()
    y = net.forward(xd).cpu().numpy()
    lo, ow, ob, yo = mo.forward_backward(w, b, d, x, t.astype(np.float64))
    scale = np.abs(yo).max()
    assert np.max(np.abs(y - yo)) <= 1e-2 * scale
    assert abs(float(loss.item()) - lo) <= 1e-2 * lo
    W, B = mo.unpack(gw, gb, d)
    Wo, Bo = mo.unpack(ow, ob, d)
    for l in range(len(W)):
        for g, go in ((W[l], Wo[l]), (B[l], Bo[l])):
            rel = np.linalg.norm(g - go) / max(np.linalg.norm(go), 1e-30)
            assert rel <= 1e-2, (l, rel)


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,hidden,layers,n_out,batch,rows", [
    (1, 1, 1, 1, 16, 1),          # one fragment of one tile everywhere
    (17, 100, 2, 65, 80, 63),     # ragged tiles in every dimension
    (163, 64, 5, 161, 1040, 65),  # the deepest network, a last slice of 16 rows
    (300, 256, 1, 12, 4096, 129)])
def test_gpu_tiles_and_slices(torch, n_in, hidden, layers, n_out, batch, rows):
    """Tile remainders, batch slices of the weight gradient and depths: the
    bounds of test_gpu_gradients_match_oracle (BF16 products, 2^-9 relative
    each, of which single roundings flip)."""
    from zerork_b200.predictor import Mlp
    rng = np.random.default_rng(5)
    net = Mlp(n_in, n_out, hidden, layers, seed=3)
    d, w, b = _net(rng, n_in, hidden, layers, n_out)
    net.set_params(w, b)
    x = rng.standard_normal((batch, n_in)).astype(np.float32)
    t = rng.standard_normal((batch, n_out)).astype(np.float32)
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    net.gradients(torch.from_numpy(x).cuda(), torch.from_numpy(t).cuda(), loss)
    gw, gb = net.grads()
    lo, ow, ob, yo = mo.forward_backward(w, b, d, x, t.astype(np.float64))
    y = net.forward(torch.from_numpy(x[:rows]).cuda()).cpu().numpy()
    assert np.max(np.abs(y - yo[:rows])) <= 1e-2 * np.abs(yo).max()
    assert abs(float(loss.item()) - lo) <= 1e-2 * lo
    for g, go in zip(mo.unpack(gw, gb, d), mo.unpack(ow, ob, d)):
        for a, o in zip(g, go):
            assert np.linalg.norm(a - o) <= 1e-2 * max(np.linalg.norm(o), 1e-30)


@pytest.mark.gpu
@pytest.mark.parametrize("n_in,hidden,layers,n_out,batch", [
    (3, 16, 1, 2, 2048), (17, 100, 2, 65, 80), (163, 256, 3, 128, 4096)])
def test_gpu_sums_run_over_the_batch_in_order(torch, n_in, hidden, layers, n_out, batch):
    """Gradients are one sum over the rows in order and the loss a fixed tree,
    so training repeats bit for bit whatever tiles and slices a version uses.
    Exact: the bias gradient of the output layer and the loss (up to 128
    outputs: one column a thread) from the outputs, in FP32, in that order."""
    from zerork_b200.predictor import Mlp
    rng = np.random.default_rng(7)
    net = Mlp(n_in, n_out, hidden, layers, seed=3)
    d, w, b = _net(rng, n_in, hidden, layers, n_out)
    net.set_params(w, b)
    x = torch.from_numpy(rng.standard_normal((batch, n_in)).astype(np.float32)).cuda()
    t = rng.standard_normal((batch, n_out)).astype(np.float32)
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    net.gradients(x, torch.from_numpy(t).cuda(), loss)
    e = net.forward(x).cpu().numpy() - t
    scale = np.float32(2.0) / (np.float32(batch) * np.float32(n_out))
    gb = net.grads()[1][-d[-1]:][:n_out]
    assert np.array_equal(gb, np.add.accumulate(scale * e, axis=0, dtype=np.float32)[-1])

    def tree(v):  # 32 lanes, halving distances
        for o in (16, 8, 4, 2, 1):
            v = v + v[..., np.arange(32) ^ o]
        return v[..., 0]

    def in_order(v):
        return np.add.accumulate(v, axis=-1, dtype=np.float32)[..., -1]

    sq = np.zeros((batch, 128), np.float32)
    sq[:, :n_out] = e * e
    rows = np.zeros(-(-batch // 256) * 256, np.float32)
    rows[:batch] = in_order(tree(sq.reshape(batch, 4, 32)))
    assert loss.item() == in_order(tree(in_order(rows.reshape(-1, 256).T).reshape(8, 32)))


@pytest.mark.gpu
def test_gpu_weight_gradient_is_one_chain(torch):
    """A weight gradient adds the batch rows 16 at a time to one accumulator:
    with a first row of 1 and one row of 1.5 * 2^-26 in each following 16, every
    addition is below half a unit of the accumulator and is lost, while partial
    sums of any four of them would not be."""
    from zerork_b200.predictor import Mlp
    net = Mlp(1, 2, 1, 1, seed=3)
    d = mo.dims(1, 1, 1, 2)
    w, b = np.zeros(net.nw, np.float32), np.zeros(net.nb, np.float32)
    b[0] = 1.0  # hidden activation silu(1) in every row, outputs 0
    net.set_params(w, b)
    n = 2048
    t = np.zeros((n, 2), np.float32)
    t[16::16, 0] = -1.5 * 2.0 ** -26
    t[0, 0] = -1.0
    loss = torch.zeros(1, dtype=torch.float32, device="cuda")
    net.gradients(torch.zeros((n, 1), device="cuda"), torch.from_numpy(t).cuda(), loss)
    gw, _ = net.grads()
    silu1 = mo.bf16(np.float32(1.0 / (1.0 + np.exp(-1.0))))
    assert mo.unpack(gw, np.zeros(net.nb, np.float32), d)[0][1][0, 0] == silu1 * np.float32(2.0 / (2 * n))


@pytest.mark.gpu
def test_gpu_capture_after_an_evaluation(torch):
    """An evaluation leaves the workspace that gradients of as many rows need,
    so they can be captured in a CUDA graph, where nothing can be allocated."""
    from zerork_b200.predictor import Mlp
    rng = np.random.default_rng(8)
    nets = [Mlp(56, 54, 64, 2, seed=3) for _ in range(2)]
    x = torch.from_numpy(rng.standard_normal((320, 56)).astype(np.float32)).cuda()
    t = torch.from_numpy(rng.standard_normal((320, 54)).astype(np.float32)).cuda()
    loss = torch.zeros(2, dtype=torch.float32, device="cuda")
    Mlp(56, 54, 64, 2, seed=3).gradients(x, t, loss[:1])  # loads the kernels
    nets[0].forward(x)
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        nets[0].gradients(x, t, loss[:1], stream=torch.cuda.current_stream().cuda_stream)
    g.replay()
    torch.cuda.synchronize()
    nets[1].gradients(x, t, loss[1:])
    assert np.array_equal(nets[0].grads()[0], nets[1].grads()[0]) and loss[0].item() == loss[1].item()


@pytest.mark.gpu
def test_gpu_training_reduces_loss(torch):
    from zerork_b200.predictor import train
    rng = np.random.default_rng(4)
    A = rng.standard_normal((10, 6))
    x = rng.standard_normal((16384, 10))
    t = np.tanh(0.5 * (x @ A)) + 0.1 * (x[:, :6] ** 2)
    net, xs, ts, hist = train(x, t, hidden=256, layers=3, epochs=8, batch=1024, lr=2e-3)
    assert hist[-1] < 0.2 * hist[0], hist
    # the trained network predicts held-out points of the same function
    xv = rng.standard_normal((2048, 10))
    tv = np.tanh(0.5 * (xv @ A)) + 0.1 * (xv[:, :6] ** 2)
    yv = net.forward(torch.from_numpy(xs.fwd(xv).astype(np.float32)).cuda()).cpu().numpy()
    err = np.mean((ts.inv(yv) - tv) ** 2) / np.var(tv)
    assert err < 0.3, err
