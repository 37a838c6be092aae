"""The learned-guess network's tensor-core kernels against the CPU oracle
(GPU tests): forward pass, gradients of one batch, one Adam step, and a
short training run that must lower the loss.

The device products (tcgen05.mma) are BF16 x BF16 with FP32 accumulation
and the oracle rounds to BF16 at the same points in float64, so the two
differ by FP32 accumulation order and by the rare value that lands on the
other side of a BF16 rounding boundary: relative error norms below 2e-3 per
parameter block (measured: at most 2.1e-4, on the 112-256-256-232 network),
and below 1e-4 for the forward output (measured: at most 3.5e-5)."""
import numpy as np
import pytest

from oracle import mlp_ref
from helpers import pfk

pytestmark = pytest.mark.gpu


def _net(dims, seed=0, max_batch=512):
    pfk()
    import importlib
    M = importlib.import_module("planck-refactored_b200.mlp")
    return M.MLP(dims, max_batch, seed=seed)


def _data(dims, n, seed):
    rng = np.random.default_rng(seed)
    X = rng.normal(size=(n, dims[0])).astype(np.float32)
    T = rng.normal(size=(n, dims[-1])).astype(np.float32)
    return X, T


@pytest.mark.parametrize("dims,n", [([112, 256, 256, 232], 300), ([16, 24, 8], 7), ([40, 64, 32, 48], 130)])
def test_forward_and_gradients_match_oracle(dims, n):
    torch = pytest.importorskip("torch")
    net = _net(dims, seed=1)
    X, T = _data(dims, n, 2)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    p = net.params()
    Y = net.forward(Xd).cpu().numpy()
    Yo = mlp_ref.forward(dims, p, X)[0]
    assert np.linalg.norm(Y - Yo) < 1e-4 * np.linalg.norm(Yo)
    g, loss = net.gradients(Xd, Td)
    go, losso = mlp_ref.gradients(dims, p, X, T)
    assert abs(loss - losso) < 1e-4 * losso
    o = 0
    for din, dout in zip(dims[:-1], dims[1:]):
        for size in (din * dout, dout):
            a, b = g[o:o + size], go[o:o + size]
            assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-12
            o += size
    net.close()


def test_adam_step_matches_oracle():
    torch = pytest.importorskip("torch")
    dims = [32, 64, 16]
    net = _net(dims, seed=3)
    X, T = _data(dims, 64, 4)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    p0 = net.params().astype(np.float64)
    g, _ = net.gradients(Xd, Td)           # the gradient the step will use
    net.train_step(Xd, Td, 1e-2)
    p1 = net.params()
    po, _, _ = mlp_ref.adam(p0, g.astype(np.float64), np.zeros_like(p0), np.zeros_like(p0), 1, 1e-2)
    assert np.abs(p1 - po).max() < 1e-5
    net.close()


def test_training_lowers_the_loss():
    torch = pytest.importorskip("torch")
    dims = [16, 64, 64, 8]
    rng = np.random.default_rng(5)
    X = rng.normal(size=(512, 16)).astype(np.float32)
    W = rng.normal(size=(16, 8)) / 4
    T = np.tanh(X @ W).astype(np.float32)            # a smooth target the network can fit
    net = _net(dims, seed=6)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    first = net.gradients(Xd, Td)[1]
    for _ in range(300):
        net.train_step(Xd, Td, 3e-3)
    last = net.gradients(Xd, Td)[1]
    assert last < 0.1 * first
    net.close()


@pytest.mark.parametrize("dims,n", [([8, 8], 1), ([24, 8], 129), ([64, 64, 64], 8), ([72, 136, 8], 127),
                                    ([520, 264, 64], 128), ([16, 8, 8, 8, 8, 8, 8, 8, 8], 65), ([128, 192, 200], 1031)])
def test_tile_edges(dims, n):
    """Widths and batch sizes around the 128 x 64 tile, the 64-deep round and
    the four-stage ring (520 is nine rounds; 1031 rows are 17 rounds of the
    weight gradients in four splits, the last of them short), one to eight
    layers; targets and outputs that are not 16-byte aligned give the same
    bits as aligned ones.  Bounds as above: the roundings of Z, H and dZ are
    the oracle's, the sums differ in order."""
    torch = pytest.importorskip("torch")
    net = _net(dims, seed=9, max_batch=n + 3)
    X, T = _data(dims, n, 10)
    Xd = torch.from_numpy(X).cuda()
    flat = torch.zeros(n * dims[-1] + 1, device="cuda")
    flat[1:] = torch.from_numpy(T).cuda().reshape(-1)
    Tu = flat[1:].view(n, dims[-1])                 # 4 bytes past a 16-byte boundary
    Td = Tu.clone()
    p = net.params()
    Y = net.forward(Xd).cpu().numpy()
    Yo = mlp_ref.forward(dims, p, X)[0]
    assert np.linalg.norm(Y - Yo) < 1e-4 * np.linalg.norm(Yo)
    Yu = torch.zeros(n * dims[-1] + 1, device="cuda")
    net._check(net.L.pfk_mlp_forward(net.h, net._ptr(Xd), n, Yu.data_ptr() + 4, None))
    assert np.array_equal(Yu[1:].view(n, dims[-1]).cpu().numpy(), Y) and float(Yu[0]) == 0.0
    g, loss = net.gradients(Xd, Td)
    gu, lossu = net.gradients(Xd, Tu)
    assert np.array_equal(g, gu) and loss == lossu
    go, losso = mlp_ref.gradients(dims, p, X, T)
    assert abs(loss - losso) < 1e-4 * losso
    o = 0
    for din, dout in zip(dims[:-1], dims[1:]):
        for size in (din * dout, dout):
            a, b = g[o:o + size], go[o:o + size]
            assert np.linalg.norm(a - b) <= 2e-3 * np.linalg.norm(b) + 1e-12
            o += size
    # the update uses these gradients, and the next forward pass its weights
    net.train_step(Xd, Td, 1e-2)
    z = np.zeros_like(p, dtype=np.float64)
    po = mlp_ref.adam(p.astype(np.float64), g.astype(np.float64), z, z, 1, 1e-2)[0]
    p1 = net.params()
    assert np.abs(p1 - po).max() < 1e-5
    Y1o = mlp_ref.forward(dims, p1, X)[0]
    assert np.linalg.norm(net.forward(Xd).cpu().numpy() - Y1o) < 1e-4 * np.linalg.norm(Y1o)
    net.close()


@pytest.mark.parametrize("dims", [[64, 64], [64, 128, 64], [256, 8], [8, 256], [264, 264]])
def test_output_over_the_input(dims):
    """pfk_mlp_forward converts X before it writes Y, so Y may lie anywhere on
    X: the bits of a separate output.  1000 rows are eight row tiles, whose
    outputs land on other tiles' inputs when the widths or the starts differ."""
    torch = pytest.importorskip("torch")
    n = 1000
    net = _net(dims, seed=4, max_batch=n)
    X, _ = _data(dims, n, 6)
    Y = net.forward(torch.from_numpy(X).cuda()).cpu().numpy()
    nx, ny = n * dims[0], n * dims[-1]
    for at in (0, 4, dims[0] * 129, max(nx - ny, 0)):       # Y's start, in floats after X's
        buf = torch.zeros(max(nx, at + ny), device="cuda")
        buf[:nx] = torch.from_numpy(X).cuda().reshape(-1)
        torch.cuda.synchronize()
        net._check(net.L.pfk_mlp_forward(net.h, buf.data_ptr(), n, buf.data_ptr() + 4 * at, None))
        assert np.array_equal(buf[at:at + ny].view(n, -1).cpu().numpy(), Y), at
    net.close()


def test_rows_beyond_a_grid_axis():
    """65535 x 32 rows and a few more through the layer-by-layer path: the
    input conversion's row tiles are not limited to one grid's y axis.  The
    last rows' outputs are those of a small batch (a row's arithmetic does not
    depend on its batch)."""
    torch = pytest.importorskip("torch")
    dims, n = [264, 8], 65535 * 32 + 70
    net = _net(dims, seed=2, max_batch=n)
    X = torch.randn((n, dims[0]), device="cuda", generator=torch.Generator(device="cuda").manual_seed(1))
    Y = net.forward(X)
    for a, b in ((0, 100), (n - 300, n)):
        assert bool((net.forward(X[a:b].contiguous()) == Y[a:b]).all())
    net.close()


@pytest.mark.parametrize("dims,n", [([24, 8], 129), ([72, 136, 8], 127), ([112, 256, 256, 232], 300), ([264, 16], 70)])
def test_unaligned_input(dims, n):
    """X 4 bytes past a 16-byte boundary: the bits of an aligned X."""
    torch = pytest.importorskip("torch")
    net = _net(dims, seed=9, max_batch=n)
    X, T = _data(dims, n, 10)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    flat = torch.zeros(n * dims[0] + 1, device="cuda")
    flat[1:] = Xd.reshape(-1)
    Xu = flat[1:].view(n, dims[0])
    assert Xu.data_ptr() % 16 == 4
    assert bool((net.forward(Xu) == net.forward(Xd)).all())
    g, loss = net.gradients(Xd, Td)
    gu, lossu = net.gradients(Xu, Td)
    assert np.array_equal(g, gu) and loss == lossu
    net.close()


def test_many_networks_share_the_host_slots():
    """150 networks at a time (64 result slots per page-locked slab), made,
    used and closed from several threads, give one network's results."""
    import threading
    torch = pytest.importorskip("torch")
    dims, n = [16, 24, 8], 40
    X, T = _data(dims, n, 3)
    Xd, Td = torch.from_numpy(X).cuda(), torch.from_numpy(T).cuda()
    torch.cuda.synchronize()
    first = _net(dims, seed=1)
    g0, loss0 = first.gradients(Xd, Td)
    bad = []

    def work(k):
        for _ in range(2):
            nets = [_net(dims, seed=1) for _ in range(50)]
            for net in nets[k::3] + nets[:2]:
                g, loss = net.gradients(Xd, Td, stream=torch.cuda.Stream())
                if loss != loss0 or not np.array_equal(g, g0):
                    bad.append(k)
            for net in nets[::-1] if k == 1 else nets:
                net.close()
    threads = [threading.Thread(target=work, args=(k,)) for k in range(3)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not bad
    assert first.gradients(Xd, Td)[1] == loss0
    first.close()
