"""hydro_rigid_step's rotation by large angles, and on both sides of the angle
up to which it is a series."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from oracle import rigid  # noqa: E402
from stonefish_gb300 import abi  # noqa: E402
from stonefish_gb300 import rollout as RO  # noqa: E402

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dt", [0.01, 0.002])
def test_rotation_by_any_angle_matches_oracle(hctx, dt):
    """Spheres (no gyroscopic term) turning by up to three radians a step, none
    at all, and by 1/2 +- a few units of the last place, where half the angle
    is the series' last: positions, orientations and rates within 1e-12."""
    rng = np.random.default_rng(2)
    n = 2000
    s = RO.initial_states(rng, n)
    s["inertia"] = rng.uniform(1.0, 5.0, n)[:, None]
    s["thrust_force"], s["thrust_torque"] = 0.0, 0.0
    axis = rng.normal(size=(n, 3))
    axis /= np.linalg.norm(axis, axis=1)[:, None]
    half = rng.uniform(0.0, 1.5, n)
    half[:600] = 0.25 * (1.0 + rng.integers(-6, 7, 600) * 2.0 ** -52)
    half[600:700] = rng.uniform(0.2, 0.3, 100)
    half[700:710] = 0.0
    half[710:730] = 10.0 ** -np.arange(1, 21, dtype=np.float64)
    s["w"] = axis * (2.0 * half / dt)[:, None]
    q = rng.normal(size=(n, 4))
    s["q"] = q / np.linalg.norm(q, axis=1)[:, None]
    d_s = torch.from_numpy(np.frombuffer(s.tobytes(), dtype=np.uint8).copy()).cuda()
    d_b = torch.from_numpy(np.frombuffer(RO.static_bodies(n, 0).tobytes(), dtype=np.uint8).copy()).cuda()
    assert hctx.lib.hydro_rigid_step(hctx.ctx, RO._ptr(d_s), RO._ptr(d_b), None, None, n, dt, 9.81, None) == 0
    torch.cuda.synchronize()
    got = np.frombuffer(d_s.cpu().numpy().tobytes(), dtype=abi.RIGID_DTYPE)
    ref = rigid.step(s, np.zeros((n, 3)), np.zeros((n, 3)), dt, 9.81)
    for k in ("p", "q", "v"):
        assert np.allclose(got[k], ref[k], rtol=1e-12, atol=1e-12), k
    assert np.allclose(got["w"], ref["w"], rtol=1e-12, atol=1e-12 * np.abs(ref["w"]).max())
