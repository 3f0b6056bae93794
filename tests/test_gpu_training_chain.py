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
