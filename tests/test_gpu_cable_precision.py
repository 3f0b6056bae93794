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


def _submerged_volumes(x, r):
    """Volumes of segments between the nodes of x, radius r [n], in extended
    precision (CableEntity.cpp:270-322), and which of them cross the surface,
    neither vertical nor level."""
    LD = np.longdouble
    pi = LD("3.14159265358979323846264338327950288")
    dep = x[:, 2].astype(np.float32).astype(LD)
    x, r = x.astype(LD), r.astype(LD)
    swap = dep[:-1] > dep[1:]
    d1, d2 = np.where(swap, dep[1:], dep[:-1]), np.where(swap, dep[:-1], dep[1:])
    s = x[1:] - x[:-1]
    dxy, length = np.hypot(s[:, 0], s[:, 1]), np.sqrt((s * s).sum(1))
    with np.errstate(all="ignore"):
        alpha = np.arctan((d2 - d1) / dxy)
        ca, sa = np.cos(alpha), np.sin(alpha)
        m, full = r * ca, pi * r * r * length

        def circ(h):
            hh = np.clip(np.where(h > r, 2 * r - h, h), 0, None)
            th = 2 * np.arccos(np.clip((r - hh) / r, -1, 1))
            small = r * r / 2 * (th - np.sin(th))
            return np.where(h <= 0, 0 * r, np.where(h >= 2 * r, pi * r * r, np.where(h > r, pi * r * r - small, small)))
        V = np.select([d2 < -m, d1 > m, (np.abs(d1) <= m) & (np.abs(d2) <= m), (d1 < -m) & (d2 > m), d2 <= m],
                      [0 * full, full, (circ(d1 / ca + r) + circ(d2 / ca + r)) / 2 * length,
                       pi * r * r * ((d2 - m) / sa + m), circ(r + d2 / ca) * (r + d2 / ca) / sa / 2],
                      full - circ(r - d1 / ca) * (r - d1 / ca) / sa / 2)
    return V, (V > 0) & ~(d1 > m) & (dxy > 1e-3) & (d2 - d1 > 1e-3)


def _surface_errors(hctx):
    """Relative errors, in units of 2^-53, of the buoyancy of segments that
    cross the surface, each a cable of its own."""
    q = []
    for seed in range(8):
        rng = np.random.default_rng(seed)
        sc = scenarios.cable_set(n_cables=300, seed=100 + seed, max_nodes=120)
        lo = np.concatenate([c["first_node"] + np.arange(c["n_nodes"] - 1) for c in sc["cables"]])
        r = np.repeat(rng.uniform(0.01, 0.3, len(sc["cables"])), sc["cables"]["n_nodes"] - 1)
        x = np.stack([sc["x"][lo], sc["x"][lo + 1]], 1)
        cables = np.zeros(len(lo), dtype=abi.CABLE_DTYPE)
        cables["first_node"], cables["n_nodes"], cables["radius"] = 2 * np.arange(len(lo)), 2, r
        cables["mode"], cables["buoyancy"] = abi.MODE_SUBMERGED, 1
        out = np.zeros(2 * len(lo), dtype=abi.CABLE_FORCES_DTYPE)
        ocean = sc["ocean"]
        hctx.cable_forces(cables, x.reshape(-1, 3), np.zeros((2 * len(lo), 3)), ocean, scenarios.settings(), out)
        V, part = _submerged_volumes(x.reshape(-1, 3), np.repeat(r, 2)[:-1])
        V, part = V[::2], part[::2]
        want = -V * np.longdouble(ocean.density) * np.longdouble(ocean.gravity)
        q.append(np.abs(out["Fb"][::2, 2][part] / want[part] - 1).astype(float) / U)
    return np.concatenate(q)


def test_segments_in_the_surface_keep_the_references_error(hctx):
    """The mean error is 2.12 units with the reference's operations one by one,
    leaving out the hundredth part where the length itself cancels; with the
    angle's cosine and sine as products of a reciprocal it would be 2.36."""
    q = np.sort(_surface_errors(hctx))
    assert q.size > 5000
    assert np.mean(q[:int(0.99 * q.size)]) <= 2.2
