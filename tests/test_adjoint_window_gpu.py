"""The adjoint's windowed kernels (fly-brain_gb300/csrc/fb_adjoint_window.cuh) where their parts meet
their limits, against the oracle's restatement of LIFDiff: checkpoint intervals, truncations and lengths that do
not divide a window; targets with more contributions than a lane (8) or a warp (128) sorts; both
membrane models; refractory times below the three steps a window needs. Tape and spike counts
identical, gradients within the tolerance of tests/test_adjoint_gpu.py (the same arithmetic)."""
import numpy as np
import pytest

from test_adjoint_gpu import _compare_grads, _pair

pytestmark = pytest.mark.gpu


def hub_net(N, hub, seed, deg=6):
    rng = np.random.default_rng(seed)
    rows = [np.unique(np.concatenate([np.arange(hub), rng.integers(0, N, deg)])) for _ in range(N)]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.uint32)
    idx = np.concatenate(rows).astype(np.uint32)
    return dict(N=N, indptr=indptr, indices=idx, counts=rng.integers(1, 9, idx.shape[0]).astype(np.float32),
                sign=np.where(rng.random(N) < 0.7, 1.0, -1.0).astype(np.float32))


CUBA = dict(dt=0.1, coba=False, soft=False, surrogateBeta=0.5, wSyn=0.2, minSyn=2.0, adjClip=50.0)
COBA = dict(dt=0.1, coba=True, soft=False, surrogateBeta=2.0, wSyn=0.4, minSyn=2.0, adaptInc=0.4, depU=0.15, inhGain=1.3)


@pytest.mark.parametrize("model", [CUBA, COBA])
@pytest.mark.parametrize("N,hub,hz", [(60, 3, 900.0), (300, 4, 4000.0)])
@pytest.mark.parametrize("K,truncate,steps", [(7, 0, 61), (18, 0, 90), (100, 23, 130), (16, 16, 64), (1, 0, 20)])
def test_windows_match_oracle(model, N, hub, hz, K, truncate, steps):
    ins = hub_net(N, hub, N)
    rng = np.random.default_rng(3)
    driven = rng.permutation(N)[: N * 3 // 4].astype(np.int32)
    p = dict(model, checkpoint=K)
    prob, net = _pair(ins, p, driven, np.full(driven.shape[0], hz))
    sc0, tape = prob.forward(steps, seed=5, checkpoint=K)
    sc1 = net.forward(steps, seed=5)
    assert sc0.tobytes() == sc1.tobytes()
    off, idx, amp = net.tape()
    np.testing.assert_array_equal(off, tape["off"])
    np.testing.assert_array_equal(idx, tape["idx"])
    dL = rng.normal(0, 1, N).astype(np.float32)
    g0 = prob.backward(tape, dL, truncate=truncate, lossFrom=steps // 3)
    g1 = net.backward(dL, truncate=truncate, lossFrom=steps // 3)
    _compare_grads(g0, g1)
    assert np.abs(g1["edge"]).sum() > 0


@pytest.mark.parametrize("tref", [0.05, 0.25, 0.45])
def test_short_refractory_times(tref):
    ins = hub_net(80, 2, 9)
    driven = np.arange(0, 80, 2, dtype=np.int32)
    p = dict(COBA, tRef=tref, checkpoint=10, vThresh=-50.0)
    prob, net = _pair(ins, p, driven, np.full(40, 500.0))
    sc0, tape = prob.forward(70, seed=2, checkpoint=10)
    assert sc0.tobytes() == net.forward(70, seed=2).tobytes()
    off, idx, _ = net.tape()
    np.testing.assert_array_equal(idx, tape["idx"])
    dL = np.ones(80, np.float32)
    _compare_grads(prob.backward(tape, dL), net.backward(dL))


@pytest.mark.parametrize("nD", [1, 512, 513, 2048, 2049, 4096, 4097])
def test_driven_list_sizes(nD):
    """The chain's layouts; 2,049 and more also shorten the windows (their draws); 4,097 goes step by
    step. Drawn often enough that a step forces hundreds of spikes."""
    ins = hub_net(4500, 1, nD, deg=5)
    rng = np.random.default_rng(nD)
    driven = rng.permutation(4500)[:nD].astype(np.int32)
    hz = rng.uniform(100, 2500, nD)
    prob, net = _pair(ins, dict(CUBA, checkpoint=50, adaptInc=0.3), driven, hz)
    sc0, tape = prob.forward(57, seed=4, checkpoint=50)
    assert sc0.tobytes() == net.forward(57, seed=4).tobytes()
    off, idx, _ = net.tape()
    np.testing.assert_array_equal(off, tape["off"])
    np.testing.assert_array_equal(idx, tape["idx"])


@pytest.mark.parametrize("model", [CUBA, COBA])
@pytest.mark.parametrize("power", [50, 100, 112])
def test_float_sums_scale(model, power):
    """Every operation of the reverse sweep is linear in dL, so with dL times 2^power the gradients
    are the same times 2^power: at 0 every accumulator is summed in floats, at 100 part of them and
    at 112 nearly all go to the double. Each sum of at most 200 terms is off by at most 200 * 2^-53 of its
    terms' magnitudes; a float result rounds by 2^-24."""
    ins = hub_net(300, 4, 11)
    rng = np.random.default_rng(6)
    driven = rng.permutation(300)[:200].astype(np.int32)
    p = dict(model, checkpoint=40, precision="f32", adjClip=0.0, surrogateBeta=5.0)
    _, net = _pair(ins, p, driven, np.full(200, 900.0))
    net.forward(120, seed=5)
    dL = rng.normal(0, 1, 300).astype(np.float32)
    g0 = net.backward(dL)
    net.forward(120, seed=5)
    g1 = net.backward(np.ldexp(dL, power).astype(np.float32))
    for k in ("logGain", "bias", "edge"):
        a, b = np.asarray(g0[k], np.float64), np.ldexp(np.asarray(g1[k], np.float64), -power)
        assert np.isfinite(b).all() and np.abs(a).max() > 0
        assert np.abs(a - b).max() <= 1e-9 * np.abs(a).max() + 2.0 ** -23 * np.abs(a).max(), k
    for k, v in g0["params"].items():
        assert abs(v - np.ldexp(g1["params"][k], -power)) <= 1e-6 * abs(v) + 1e-9, k


@pytest.mark.parametrize("precision", ["f64", "f32"])
@pytest.mark.parametrize("what", ["one", "edge inf", "threshold inf", "threshold nan", "bias inf", "readout"])
def test_what_the_sweep_leaves_out(what, precision):
    """Losses on few neurons, so that most adjoints stay zero, and values with which a product with
    zero is not zero, somewhere in the network. Without them a sweep over every neuron (a loss of the least
    float on each, which marks all of them) gives the same gradients up to that loss's own; with them the
    oracle's double sweep and the kernels agree on which gradients are lost."""
    N = 400
    ins = hub_net(N, 2, 21, deg=8)
    rng = np.random.default_rng(8)
    thr = np.zeros(N, np.float32)
    if what == "edge inf":
        ins["counts"][np.nonzero(ins["indices"] == 77)[0][0]] = np.inf
    if what == "threshold inf":
        thr[50:60] = np.inf
    if what == "threshold nan":
        thr[50:52] = np.nan
    bias = np.zeros(N, np.float32)
    if what == "bias inf":
        bias[90] = np.inf
    driven = rng.permutation(N)[:250].astype(np.int32)
    p = dict(CUBA, checkpoint=30, adjClip=0.0, precision=precision)
    prob, net = _pair(dict(ins, thrOffset=thr), p, driven, np.full(250, 700.0))
    if what == "bias inf":
        from flybrain.diff import DiffNet
        net = DiffNet(dict(N=N, indptr=ins["indptr"], indices=ins["indices"], weights=ins["counts"], sign=ins["sign"]),
                      dict(p, bias=bias, thrOffset=thr))
        for i in driven:
            net.setDriveOne(int(i), 700.0)
    dL = np.zeros(N, np.float32)
    dL[[5, 123]] = 1.0, -2.0
    every = np.where(dL == 0, np.float32(1e-45), dL)
    got = []
    for d in (dL, every):
        net.forward(100, seed=9)
        if what == "readout":
            got.append(net.backward(np.tile(d[[5, 123]], (100, 1)), readout=np.array([5, 123], np.int32))
                       if d is dL else net.backward(d))
        else:
            got.append(net.backward(d))
    a, b = got
    for k in ("logGain", "bias", "edge"):
        x, y = np.asarray(a[k], np.float64), np.asarray(b[k], np.float64)
        np.testing.assert_array_equal(np.isnan(x), np.isnan(y))
        np.testing.assert_array_equal(np.isinf(x), np.isinf(y))
        ok = np.isfinite(x)
        scale = np.abs(x[ok]).max() if ok.any() else 0.0
        assert np.abs(x[ok] - y[ok]).max() <= 1e-6 * scale + 1e-30, k
    assert a["clamped"] == b["clamped"]


@pytest.mark.parametrize("model", [CUBA, COBA])
@pytest.mark.parametrize("K,truncate,steps", [(1, 0, 45), (7, 0, 61), (18, 0, 90), (40, 23, 130)])
def test_losses_on_few_neurons(model, K, truncate, steps):
    """The replay of a segment runs the neurons that the sweep can reach; segments shorter and longer
    than the delay, against the oracle. Values set to what they are between the passes give up the
    selection and nothing else."""
    N = 300
    ins = hub_net(N, 1, K, deg=4)
    rng = np.random.default_rng(K)
    driven = rng.permutation(N)[:60].astype(np.int32)
    p = dict(model, checkpoint=K)
    prob, net = _pair(ins, p, driven, np.full(60, 900.0))
    sc0, tape = prob.forward(steps, seed=5, checkpoint=K)
    assert sc0.tobytes() == net.forward(steps, seed=5).tobytes()
    dL = np.zeros(N, np.float32)
    dL[rng.permutation(N)[:3]] = rng.normal(0, 1, 3)
    g0 = prob.backward(tape, dL, truncate=truncate, lossFrom=0)
    g1 = net.backward(dL, truncate=truncate, lossFrom=0)
    _compare_grads(g0, g1)
    net.set_array("thrOffset", np.zeros(N, np.float32))
    g2 = net.backward(dL, truncate=truncate, lossFrom=0)
    assert g1["params"] == g2["params"]
    for k in ("logGain", "bias", "edge"):
        np.testing.assert_array_equal(g1[k], g2[k])
