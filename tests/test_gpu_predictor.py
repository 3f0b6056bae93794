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


@pytest.mark.parametrize("n,stride", [(257, 7), (3000, 64), (5000, 0)])
def test_disagreement_gate_and_whole_chunks(scene, n, stride):
    """Two networks with a threshold in the middle of their disagreements: the
    gate alone rejects states, some of them audit rows; masks, slots and, with
    whole chunks, every output are the bits of the single entry points'
    chain.  The same call with chunks split stays within 2e-6 of the scales."""
    import ctypes as C
    s = scene(n, nets=2)
    h, lib, ctx, P = s.h, s.h.lib, s.h.ctx, S._ptr
    wide = s.predictor(tau=1e30)
    wide.predict(s.d_b)
    f = wide.bufs["feats"][:n].clone()
    za, zb = torch.zeros((n, 16), device="cuda"), torch.zeros((n, 16), device="cuda")
    s.nets[0].infer_tc(f, za, wide.tcw)
    s.nets[1].infer_tc(f, zb, wide.tcw2)
    d = torch.maximum((za - zb)[:, :3].double().norm(dim=1) / wide.fs, (za - zb)[:, 3:6].double().norm(dim=1) / wide.ts)
    tau = float(torch.quantile(d, 0.9))
    wide.close()
    gp = s.predictor(tau=tau, audit_stride=stride)
    got = gp.predict(s.d_b).clone()
    mask = torch.ones(n, dtype=torch.uint8, device="cuda")
    h._ck(lib.hydro_nn_ensemble(ctx, P(za), P(zb), 16, n, gp.fs, gp.ts, tau, P(mask), None))
    gate = mask.clone()
    idx = torch.zeros(max(gp.audit_k, 1), dtype=torch.int32, device="cuda")
    if stride:
        h._ck(lib.hydro_nn_audit_pick(ctx, P(mask), n, stride, 0, gp.audit_k, P(idx), None))
        rows = torch.arange(0, n, stride, device="cuda")
        assert 0 < int((gate[rows] == 0).sum()) < rows.numel()   # rejected audit rows, and admitted ones
    rejected = int((gate == 0).sum())
    assert 0.05 * n < rejected < 0.15 * n
    clear = (d - tau).abs() > 1e-5 * tau
    assert torch.equal((gate == 0)[clear], (d > tau)[clear])
    cnt = torch.zeros((n + 255) // 256, dtype=torch.int32, device="cuda")
    packed, pos = torch.zeros_like(s.d_b), torch.zeros(n, dtype=torch.int32, device="cuda")
    npk, io = torch.zeros(1, dtype=torch.int32, device="cuda"), torch.zeros(n * 168, dtype=torch.uint8, device="cuda")
    h._ck(lib.hydro_nn_route(ctx, P(s.d_b), P(mask), n, P(cnt), P(packed), P(pos), P(npk), P(io), None))
    gp.batch.compute_device_prefix(packed.data_ptr(), npk.data_ptr(), s.ocean, s.st, io.data_ptr())
    out = torch.zeros((n, 6), device="cuda")
    h._ck(lib.hydro_nn_merge(ctx, P(s.d_b), P(za), 16, P(pos), P(io), n, P(out), None))
    torch.cuda.synchronize()
    assert torch.equal(gp.bufs["mask"][:n], mask) and torch.equal(gp.pos, pos)
    assert torch.equal(got, out)
    if stride:
        err = torch.zeros(gp.audit_k, device="cuda")
        h._ck(lib.hydro_nn_audit_error(ctx, P(s.d_b), P(za), 16, P(pos), P(io), P(idx), gp.audit_k, gp.fs, gp.ts, P(err),
                                       None))
        assert torch.equal(gp.audit_idx, idx) and torch.allclose(gp.audit_err[0], err, rtol=1e-6, atol=1e-9)
    p = gp._predictor(True)             # chunks split where few states are exact
    launches = C.c_uint32()
    h._ck(lib.hydro_nn_predict(ctx, gp.batch.b, C.byref(p), P(s.d_b), C.byref(s.ocean), C.byref(s.st), 0,
                               P(gp.audit_err[1]) if stride else None, C.byref(launches), s.nets[0]._s()))
    torch.cuda.synchronize()
    ex = pos >= 0
    scale = torch.tensor([gp.fs] * 3 + [gp.ts] * 3, device="cuda")
    assert launches.value == 6 and torch.equal(gp.out[~ex], out[~ex])
    if int(ex.sum()) <= 100:          # fewer chunks than half the CTAs
        assert not torch.equal(gp.out[ex], out[ex])
    assert float(((gp.out - out)[ex].abs() / scale).max()) <= 2e-6
    gp.close()


def test_refused_predictors(scene):
    """Arguments that hydro_nn_predict refuses, before anything is launched."""
    import ctypes as C

    from stonefish_gb300 import abi
    s = scene(300, nets=2)
    gp = s.predictor(audit_stride=16)
    other = s.h.upload_mesh(*S.hull_mesh(2000))
    mixed = s.h.batch(np.array([s.mid, other] * 150, dtype=np.uint32))
    short = s.h.batch(np.full(299, s.mid, dtype=np.uint32))
    err, st = gp.audit_err[0], s.nets[0]._s()

    def status(batch=gp.batch, phase=0, err=err, ocean=s.ocean, **changes):
        p = gp._predictor(False)
        for k, v in changes.items():
            setattr(p, k, v)
        return s.h.lib.hydro_nn_predict(s.h.ctx, batch.b, C.byref(p), S._ptr(s.d_b), C.byref(ocean), C.byref(s.st), phase,
                                        S._ptr(err) if err is not None else None, None, st)

    assert status() == 0
    gp.out.fill_(5.0)
    refused = [status(batch=mixed), status(batch=short), status(phase=16), status(err=None), status(n=0), status(n_nets=0),
               status(n_nets=3), status(force_scale=0.0), status(torque_scale=-1.0), status(force_scale=float("nan")),
               status(features=gp.bufs["feats"].data_ptr() + 4), status(out=gp.out.data_ptr() + 8), status(mask=None),
               status(rows=None)]
    assert refused == [abi.HYDRO_ERR_INVALID_ARG] * len(refused)
    torch.cuda.synchronize()
    assert bool((gp.out == 5.0).all())
    gp.close(), mixed.close(), short.close()
