"""The fused training step of hydro_nn_train over long runs: its kernels are
chained by programmatic dependent launch and each step's update reads the
weights and moments that the step before wrote."""
import os
import re

import numpy as np
import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "stonefish_gb300", "csrc")


def test_update_reads_parameters_behind_its_wait():
    """No branch of the update kernel touches a layer's arrays in front of its
    dependency_wait(): only a kernel that has waited is promised to see what
    the step before wrote."""
    text = open(os.path.join(CSRC, "hydro_train.cu")).read()
    body = re.search(r"\btrain_update_kernel\(.*?\)\n\{(.*?)\n\}\n", text, re.S).group(1)
    weights, biases = body.split("b -= count;")
    for branch in (weights, biases):
        wait = branch.index("dependency_wait();")
        reads = [m.start() for m in re.finditer(r"\bL\.(w|mw|vw|b|mb|vb|part|col)\b", branch)]
        assert reads and min(reads) > wait


@pytest.mark.gpu
def test_hundreds_of_chained_steps_match_step_by_step_calls(hctx):
    """600 fused steps in one call against the single entry points step by
    step: weights, moments and their BF16 copies are the same bits."""
    torch = pytest.importorskip("torch")
    from stonefish_gb300 import surrogate as S
    rng = np.random.default_rng(11)
    batch, steps = 64, 600
    feats = torch.from_numpy(rng.normal(size=(batch * steps, S.N_FEAT)).astype(np.float32)).cuda()
    targ = torch.from_numpy((rng.normal(size=(batch * steps, S.N_OUT)) * 40.0 + 5.0).astype(np.float32)).cuda()
    nets = []
    for native in (True, False):
        sur = S.Surrogate(hctx, hidden=256, seed=5, batch=batch)
        sur.fit_normalisation(feats, targ)
        sur.fit(feats, targ, epochs=1, lr=3e-3, warmup=20, native=native)
        nets.append(sur)
    torch.cuda.synchronize()
    for La, Lb in zip(nets[0].layers, nets[1].layers):
        for f in ("w", "b", "mw", "vw", "mb", "vb", "w16", "wt16"):
            assert torch.equal(La[f], Lb[f]), f


@pytest.mark.gpu
def test_captured_call_behind_a_join(hctx):
    """A call captured into a graph behind a fill and a join of two streams,
    replayed, against the same calls launched one by one."""
    torch = pytest.importorskip("torch")
    import ctypes as C

    from stonefish_gb300 import surrogate as S
    rng = np.random.default_rng(12)
    batch, steps = 256, 3
    feats = torch.from_numpy(rng.normal(size=(batch * steps, S.N_FEAT)).astype(np.float32)).cuda()
    targ = torch.from_numpy((rng.normal(size=(batch * steps, S.N_OUT)) * 4.0).astype(np.float32)).cuda()
    rows, lrs = np.arange(steps, dtype=np.int64) * batch, np.full(steps, 1e-3, dtype=np.float32)
    nets = []
    for _ in range(2):
        sur = S.Surrogate(hctx, hidden=256, seed=5, batch=batch)
        sur.fit_normalisation(feats, targ)
        nets.append((sur, sur.prepare_inputs(feats), sur._net()))

    def train(k, n, stream):
        sur, X, net = nets[k]
        sur._ck(hctx.lib.hydro_nn_train(hctx.ctx, C.byref(net), S._ptr(X), S._ptr(targ), X.shape[0], rows.ctypes.data,
                                        lrs.ctypes.data, n, 0, 0.9, 0.999, 1e-8, 1e-5, stream))

    torch.cuda.synchronize()
    side, fork, junk = torch.cuda.Stream(), torch.cuda.Stream(), torch.zeros(1 << 20, device="cuda")
    train(1, 0, None)                       # the workspace grows outside the capture
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g, stream=side):
        nets[1][0].loss_d.zero_()
        fork.wait_stream(side)
        with torch.cuda.stream(fork):
            junk.add_(1.0)
        side.wait_stream(fork)
        train(1, steps, side.cuda_stream)
    for _ in range(3):
        g.replay()
        nets[0][0].loss_d.zero_()
        train(0, steps, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    for La, Lb in zip(nets[0][0].layers, nets[1][0].layers):
        for f in ("w", "b", "mw", "vw", "mb", "vb", "w16", "wt16"):
            assert torch.equal(La[f], Lb[f]), f
    assert float(junk[0]) == 3.0
