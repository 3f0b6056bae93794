"""GatedPredictor (hydro_nn_predict): what a caller reads beside the outputs,
and how one state's prediction stands to the others of its call."""
import numpy as np
import pytest

torch = pytest.importorskip("torch")

from stonefish_gb300 import scenarios  # noqa: E402
from stonefish_gb300 import surrogate as S  # noqa: E402

pytestmark = pytest.mark.gpu


class Scene:
    """A hull, a wave field, states and untrained networks normalised on
    them, with the gates wide open."""

    def __init__(self, n, nets=1, faces=3000, gravity=None):
        from stonefish_gb300.hydro import HydroContext
        self.h = HydroContext()
        self.mid = self.h.upload_mesh(*S.hull_mesh(faces))
        self.h.set_wave_grid(scenarios.wave_grid(n=256, n_waves=16, seed=5))
        self.ocean, self.st, self.n = S.wave_ocean(), scenarios.settings(), n
        if gravity is not None:
            self.ocean.gravity = gravity
        self.bodies = S.sample_states(np.random.default_rng(n), n, extent=25.6)
        self.bodies["mesh"] = self.mid
        self.d_b = torch.from_numpy(self.bodies.view(np.uint8).copy()).cuda()
        rng = np.random.default_rng(1)
        feats = torch.from_numpy(rng.normal(size=(4096, S.N_FEAT)).astype(np.float32)).cuda()
        targ = torch.from_numpy((rng.normal(size=(4096, S.N_OUT)) * 500.0).astype(np.float32)).cuda()
        self.nets = [S.Surrogate(self.h, batch=256, seed=k) for k in range(nets)]
        for net in self.nets:
            net.fit_normalisation(feats, targ)
            net.gate["lo"].fill_(-1e30), net.gate["hi"].fill_(1e30)
            net.gate["thr"] = 1e30

    def predictor(self, **kw):
        return S.GatedPredictor(self.nets[0], self.h, self.mid, self.n, self.ocean, self.st,
                                second=self.nets[1] if len(self.nets) > 1 else None, **kw)


@pytest.fixture
def scene(built_library):
    open_ = []

    def make(*a, **kw):
        open_.append(Scene(*a, **kw))
        return open_[-1]
    yield make
    for s in open_:
        s.h.close()


def test_one_network_needs_no_scales(scene):
    """Without a second network and without the audit nothing is measured
    against the hull's force scale, which is zero without gravity."""
    s = scene(300, gravity=0.0)
    gp = s.predictor()
    assert gp.fs == 0.0
    got = gp.predict(s.d_b).cpu().numpy()
    z = torch.zeros((300, 16), device="cuda")
    feats = gp.bufs["feats"][:300].contiguous()
    s.nets[0].infer_tc(feats, z, gp.tcw)
    assert np.array_equal(got, z[:, :6].cpu().numpy()) and gp.rejected() == 0
    gp.close()


@pytest.mark.parametrize("n", [600, 6000])
def test_prediction_is_a_states_own(scene, n):
    """A state's output is the same bits however many others of its call take
    the exact step: here the gate's depth limit lets few or most through."""
    s = scene(n)
    gp = s.predictor()
    gp.predict(s.d_b)
    depth = gp.bufs["feats"][:n, 0].clone()
    outs = []
    for q in (0.99, 0.9, 0.2):
        s.nets[0].gate["hi"][0] = float(torch.quantile(depth, q))
        outs.append((gp.predict(s.d_b).clone(), gp.pos.clone() >= 0))
        assert 0 < gp.rejected() < n
    few = outs[0][1]
    for out, exact in outs[1:]:
        assert bool((exact | ~few).all()) and int(exact.sum()) > int(few.sum())
        assert torch.equal(out[few], outs[0][0][few])
        both = ~exact
        assert torch.equal(out[both], outs[0][0][both])
    gp.close()


@pytest.mark.parametrize("n,stride", [(1, 4), (63, 64), (500, 64), (4097, 1024)])
def test_audit_rows_are_recorded(scene, n, stride):
    """audit_idx holds the call's sample: a row for each audited state, -1 for
    one the gate sent to the exact step anyway or a slot past the last state."""
    s = scene(n)
    gp = s.predictor(audit_stride=stride)
    gp.predict(s.d_b)
    s.nets[0].gate["hi"][0] = float(torch.quantile(gp.bufs["feats"][:n, 0], 0.6))
    feats, hi = gp.bufs["feats"][:n].clone(), s.nets[0].gate["hi"]
    admitted = (feats[:, 0] <= hi[0]).cpu().numpy()
    for call in range(1, 4):
        gp.audit_idx.fill_(-7)
        gp.predict(s.d_b)
        rows = call % stride + stride * np.arange(gp.audit_k)
        want = np.where((rows < n) & admitted[np.minimum(rows, n - 1)], rows, -1)
        assert np.array_equal(gp.audit_idx.cpu().numpy(), want)
        assert np.array_equal(gp.audit_err[call].cpu().numpy() >= 0, want >= 0)
    gp.close()


def test_exact_step_is_profiled_and_counted(scene):
    """hydro_batch_profile and hydro_batch_last_launches of the predictor's
    batch see the exact step of a prediction, whose outputs stay the same."""
    s = scene(3000)
    gp = s.predictor()
    gp.predict(s.d_b)
    s.nets[0].gate["hi"][0] = float(torch.quantile(gp.bufs["feats"][:3000, 0], 0.7))
    plain = gp.predict(s.d_b).clone()
    assert gp.batch.last_launches() == 3 and gp.rejected() > 0
    gp.batch.profile(True)
    assert torch.equal(gp.predict(s.d_b), plain)
    ms = gp.batch.kernel_ms()
    assert all(0.0 < ms[k] < 50.0 for k in ("prep", "chunk", "finalize")), ms
    g = torch.cuda.CUDAGraph()          # no events while a stream captures
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.graph(g, stream=side):
        gp.predict(s.d_b)
    gp.out.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(gp.out, plain)
    gp.close()
