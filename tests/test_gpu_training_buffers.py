"""hydro_nn_train's work buffers: networks whose buffers share memory where the
layer by layer order allows it, and what the buffers hold after a call."""
import ctypes as C

import numpy as np
import pytest

torch = pytest.importorskip("torch")

from stonefish_gb300 import surrogate as S  # noqa: E402

pytestmark = pytest.mark.gpu

BATCH, STEPS = 128, 3
PARAMS = ("w", "b", "gw", "gb", "mw", "vw", "mb", "vb", "w16", "wt16")


def _problem(hctx, seed, n_out=S.N_OUT, normalise=True):
    """A network, its inputs and targets of `n_out` columns."""
    rng = np.random.default_rng(seed)
    n = BATCH * STEPS
    feats = torch.from_numpy(rng.normal(size=(n, S.N_FEAT)).astype(np.float32)).cuda()
    t6 = torch.from_numpy(rng.normal(size=(n, S.N_OUT)).astype(np.float32) * 4.0 + 1.0).cuda()
    sur = S.Surrogate(hctx, hidden=256, seed=5, batch=BATCH)
    sur.fit_normalisation(feats, t6)
    T = torch.from_numpy(rng.normal(size=(n, n_out)).astype(np.float32)).cuda()
    stats = [torch.from_numpy(rng.uniform(0.5, 1.5, n_out).astype(np.float32)).cuda() for _ in range(2)]
    return sur, sur.prepare_inputs(feats), T, stats if normalise else [None, None]


def _net(sur, n_out, stats):
    net = sur._net()
    net.n_out = n_out
    net.tmean, net.tistd = (t.data_ptr() if t is not None else None for t in stats)
    return net


def _native(hctx, sur, X, T, net, steps=STEPS):
    rows = np.arange(steps, dtype=np.int64) * BATCH
    lrs = np.full(steps, 1e-3, dtype=np.float32)
    sur.loss_d.zero_()
    sur._ck(hctx.lib.hydro_nn_train(hctx.ctx, C.byref(net), S._ptr(X), S._ptr(T), X.shape[0], rows.ctypes.data,
                                    lrs.ctypes.data, steps, 0, 0.9, 0.999, 1e-8, 1e-5, sur._s()))
    torch.cuda.synchronize()


def _step_by_step(hctx, sur, X, T, n_out, stats):
    """The same steps through the single entry points."""
    bf, Ls = sur._bufs(), sur.layers
    z, x, dz, xt = bf["z"], bf["x"], bf["dz"], bf["xt"]
    P = lambda t: S._ptr(t) if t is not None else None  # noqa: E731
    sur.loss_d.zero_()
    for s in range(STEPS):
        ins = [X[s * BATCH:(s + 1) * BATCH], *x]
        for l in range(3):
            sur.gemm(1, ins[l], Ls[l]["k"], Ls[l]["w16"], 256, BATCH, 256, Ls[l]["k"], z=z[l], y=x[l], bias=Ls[l]["b"])
        sur.gemm(2, x[2], 256, Ls[3]["w16"], 64, BATCH, 64, 256, z=z[3], bias=Ls[3]["b"])
        sur._ck(hctx.lib.hydro_nn_mse_grad(hctx.ctx, P(z[3]), P(T[s * BATCH:]), BATCH, 64, n_out, P(stats[0]), P(stats[1]),
                                           P(dz[3]), P(sur.loss_d), sur._s()))
        for l in (3, 2, 1, 0):
            k, n = Ls[l]["k"], Ls[l]["n"]
            sur._ck(hctx.lib.hydro_nn_transpose(hctx.ctx, P(ins[l]), P(xt[l]), BATCH, k, sur._s()))
            sur.gemm(0, xt[l], BATCH, dz[l], n, k, n, BATCH, z=Ls[l]["gw"])
            sur._ck(hctx.lib.hydro_nn_colsum(hctx.ctx, P(dz[l]), BATCH, n, P(Ls[l]["gb"]), sur._s()))
            if l:
                sur.gemm(3, dz[l], n, Ls[l]["wt16"], k, BATCH, k, n, y=dz[l - 1], zprev=z[l - 1])
        sur.optimizer_step(1e-3)
    torch.cuda.synchronize()


def _same(a, b):
    for La, Lb in zip(a.layers, b.layers):
        for f in PARAMS:
            assert torch.equal(La[f], Lb[f]), f


@pytest.mark.parametrize("shared", ["dz in turn", "dz over x", "dz inside one block"])
def test_gradient_buffers_may_take_used_buffers(hctx, shared):
    """dz[0] in dz[2]'s place, each dz[l] in the place of the activation that
    its layer's weight gradient has used, or dz[1] overlapping dz[3] by a part:
    layer by layer these are free by then, so the weights are the same bits."""
    ref, X, T, stats = _problem(hctx, 3)
    _step_by_step(hctx, ref, X, T, S.N_OUT, stats)
    sur, X, T, stats = _problem(hctx, 3)
    net = _net(sur, S.N_OUT, stats)
    if shared == "dz in turn":
        net.dz[0] = net.dz[2]
    elif shared == "dz over x":
        for l in range(3):
            net.dz[l] = net.x[l]
    else:
        block = torch.empty(BATCH * 256 * 2 + 1024, dtype=torch.uint8, device="cuda")
        net.dz[1] = block.data_ptr()
        net.dz[3] = block.data_ptr() + 1024
    _native(hctx, sur, X, T, net)
    _same(sur, ref)


@pytest.mark.parametrize("n_out,normalise", [(6, True), (6, False), (1, True), (64, False)])
def test_fused_step_for_other_targets(hctx, n_out, normalise):
    """Raw targets, and the fewest and the most target columns."""
    ref, X, T, stats = _problem(hctx, 4, n_out, normalise)
    _step_by_step(hctx, ref, X, T, n_out, stats)
    sur, X, T, stats = _problem(hctx, 4, n_out, normalise)
    _native(hctx, sur, X, T, _net(sur, n_out, stats))
    _same(sur, ref)
    assert np.isclose(float(sur.loss_d), float(ref.loss_d), rtol=1e-12)


@pytest.mark.parametrize("n_out,shared_xt", [(6, False), (5, True)])
def test_buffers_hold_the_last_step(hctx, n_out, shared_xt):
    """After a call z (every column), x, dz and xt hold what the last step's
    single entry points leave there, also with one xt for all layers."""
    ref, X, T, stats = _problem(hctx, 6, n_out)
    _step_by_step(hctx, ref, X, T, n_out, stats)
    sur, X, T, stats = _problem(hctx, 6, n_out)
    bufs = sur._bufs()
    for group in bufs.values():
        for t in group:
            t.fill_(7.0)
    net = _net(sur, n_out, stats)
    if shared_xt:
        for l in range(4):
            net.xt[l] = bufs["xt"][1].data_ptr()
    _native(hctx, sur, X, T, net)
    _same(sur, ref)
    want = ref._bufs()
    for key in ("z", "x", "dz"):
        for l, (a, b) in enumerate(zip(bufs[key], want[key])):
            assert torch.equal(a, b), (key, l)
    if shared_xt:   # the first layer's input comes last
        assert torch.equal(bufs["xt"][1].view(-1)[:64 * BATCH], want["xt"][0].view(-1))
    else:
        for l in range(4):
            assert torch.equal(bufs["xt"][l], want["xt"][l]), l
