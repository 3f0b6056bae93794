"""Cable forces leave in FP64: their error against extended precision, and
currents that depend on the place."""
import numpy as np
import pytest

from stonefish_gb300 import abi, scenarios

pytestmark = pytest.mark.gpu

U = 2.0 ** -53


def _field(current, kind, speed, radius, radius2=0.0, length=0.0, gamma=0.0, point=(0, 0, 0), direction=(1, 0, 0)):
    current.type, current.enabled, current.speed, current.radius = kind, 1, speed, radius
    current.radius2, current.length, current.gamma = radius2, length, gamma
    for k in range(3):
        current.point[k], current.dir[k] = point[k], direction[k]


@pytest.mark.parametrize("gamma", [1.0 / 7.0, 0.5, 1.0, 2.0, 10.0])
def test_pipe_profile_to_the_last_bits(hctx, gamma):
    """Resting segments beside a straight pipe's axis at distances that FP64
    holds exactly: the skin friction is 2 pi r L (1 - d)^gamma along the pipe.
    The power may be off by two units of the last place (four of 2^-53); the
    products r L, 2 pi (r L) and the force itself round once each."""
    k = np.arange(64)
    n = k.size
    cables = np.zeros(n, dtype=abi.CABLE_DTYPE)
    cables["first_node"], cables["n_nodes"], cables["radius"], cables["mode"] = 2 * k, 2, 0.03, abi.MODE_SUBMERGED
    x = np.zeros((n, 2, 3))
    x[:, 0, 0], x[:, 1, 0] = 1.0, 1.5
    x[:, :, 1] = (k / 64.0)[:, None]
    x[:, :, 2] = 5.0
    ocean = scenarios.flat_ocean()
    ocean.currents_enabled, ocean.n_currents = 1, 1
    _field(ocean.currents[0], abi.CURRENT_PIPE, 1.0, 1.0, 1.0, 40.0, gamma, point=(0, 0, 5.0))
    out = np.zeros(2 * n, dtype=abi.CABLE_FORCES_DTYPE)
    hctx.cable_forces(cables, x.reshape(-1, 3), np.zeros((2 * n, 3)), ocean, scenarios.settings(), out)
    LD = np.longdouble
    pi2 = LD("6.28318530717958647692528676655900577")
    want = pi2 * LD(0.03) * LD(0.5) * (1 - k.astype(LD) / 64) ** LD(gamma)
    got = out["Fdf"].reshape(n, 2, 3)
    assert np.all(got[:, :, 1:] == 0.0)
    for end in (0, 1):
        assert float(np.max(np.abs(got[:, end, 0] / want - 1)) / U) <= 7.0


@pytest.mark.parametrize("gamma", [1.0 / 7.0, 0.7, 2.0])
def test_cables_between_a_jet_and_a_pipe_match_oracle(oracle, hctx, gamma):
    """Cables through a jet and a widening pipe: FP64 per node within 1e-12 of
    the force scale, as without them."""
    sc, st = scenarios.cable_set(n_cables=96, seed=8), scenarios.settings()
    ocean = sc["ocean"]
    ocean.n_currents = 3
    _field(ocean.currents[1], abi.CURRENT_JET, 1.5, 1.0, point=(-3.0, -4.0, 0.5), direction=(0.6, 0.8, 0.0))
    _field(ocean.currents[2], abi.CURRENT_PIPE, 2.0, 3.0, 4.0, 40.0, gamma, (-20.0, 0.0, 1.0), (1.0, 0.0, 0.0))
    gpu = np.zeros(len(sc["x"]), dtype=abi.CABLE_FORCES_DTYPE)
    ref, still = gpu.copy(), gpu.copy()
    hctx.cable_forces(sc["cables"], sc["x"], sc["v"], ocean, st, gpu)
    oracle.cable_forces(sc["cables"], sc["x"], sc["v"], ocean, st, ref)
    ocean.n_currents = 1
    oracle.cable_forces(sc["cables"], sc["x"], sc["v"], ocean, st, still)
    assert np.mean(np.any(ref["Fdf"] != still["Fdf"], axis=1)) > 0.2   # the currents reach many nodes
    scale = max(np.abs(ref[k]).max() for k in ("Fb", "Fdq", "Fdf"))
    for k in ("Fb", "Fdq", "Fdf"):
        assert np.max(np.abs(gpu[k] - ref[k])) <= 1e-12 * scale, k
