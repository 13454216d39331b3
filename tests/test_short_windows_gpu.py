"""One brain whose windows would be short or do not apply -- refractory times of a few steps and of
none, more draws per step than a window's shared memory holds -- on the delay-scheduled kernel of single
steps (fly-brain_gb300/csrc/fb_lagged.cu), alternating with the windowed one (fb_window.cu) and the grid
kernel by the length of the launch. State, generator and ring equal the oracle's after each launch."""
import numpy as np
import pytest

from test_window_gpu import GEN, make, pair, params, same

pytestmark = pytest.mark.gpu

BG = dict(bgRate=40.0, bgAmp=1.5)


def brain(p, N=500, every=5, hz=600.0):
    from flybrain import BrainBatch, DeviceGraph
    g = make(N, 17, deg=20)
    idx = np.arange(0, N, every, dtype=np.int32)
    ob = pair(g, p, 3, idx, np.full(idx.shape[0], hz))
    b = BrainBatch([DeviceGraph(g)], p, [3])
    b.set_drive(0, idx, hz)
    return ob, b


@pytest.mark.parametrize("forced", [False, True])
@pytest.mark.parametrize("over", [dict(), dict(BG, **GEN)])
@pytest.mark.parametrize("tref,delay", [(0.0, 1.8), (0.05, 1.8), (0.15, 0.4), (0.25, 3.2), (0.35, 0.9)])
def test_short_refractory_times(tref, delay, over, forced):
    """8, 16, 64 and 128 steps are where the rule turns for windows of 1 to 4 steps."""
    from flybrain import _native as nat
    ob, b = brain(params(tRef=tref, delay=delay, vThresh=-50.0, **over))
    if forced:
        b.set_schedule(nat.FB_SCHEDULE_LAGGED)
    for n in (30, 1, 5, 7, 8, 15, 1, 16, 63, 64, 2, 128, 1, 200):
        ob.run(n)
        b.step(n)
        if forced or n >= 8:
            assert b.last_schedule() == nat.FB_SCHEDULE_LAGGED
        same(ob, b, 0, (tref, n))
    assert int(ob.spikeCount.sum()) > 100


def test_more_draws_than_a_window_holds():
    """40,000 background events a step; from 2^16 draws on the forced schedule is refused."""
    from flybrain import _native as nat
    p = params(bgRate=40000 / (500 * 0.1e-3), bgAmp=0.001)
    ob, b = brain(p)
    b.set_schedule(nat.FB_SCHEDULE_LAGGED)
    for n in (3, 20):
        ob.run(n)
        b.step(n)
        assert b.last_schedule() == nat.FB_SCHEDULE_LAGGED
        same(ob, b, 0, n)
    b.set_background(0, 66000 / (500 * 0.1e-3), 0.001)
    with pytest.raises(nat.FlyBrainError) as e:
        b.step(8)
    assert e.value.code == nat.FB_EINVAL
    same(ob, b, 0, "refused")
    b.set_schedule(nat.FB_SCHEDULE_AUTO)
    ob.setBackground(66000 / (500 * 0.1e-3), 0.001)
    ob.run(9)
    b.step(9)
    assert b.last_schedule() == nat.FB_SCHEDULE_GRID
    same(ob, b, 0, "auto")


@pytest.mark.parametrize("forced", [False, True])
def test_neurons_that_fire_twice_in_a_step(forced):
    """No refractory time and thresholds under the reset potential: the grid kernel."""
    from flybrain import _native as nat
    ob, b = brain(params(tRef=0.0))
    for i in range(0, 500, 10):
        ob.setThr(i, -9.0)
    b.set_thr(0, np.arange(0, 500, 10, dtype=np.int32), -9.0)
    if forced:
        b.set_schedule(nat.FB_SCHEDULE_LAGGED)
    for n in (20, 40):
        ob.run(n)
        b.step(n)
        assert b.last_schedule() == nat.FB_SCHEDULE_GRID
        same(ob, b, 0, n)
    assert int(ob.spikeCount.max()) > 20


@pytest.mark.parametrize("trip_at", [0, 41])
def test_timeout_leaves_the_brain_as_it_was(trip_at):
    from flybrain import _native as nat
    ob, b = brain(params(tRef=0.15, depU=0.1, **BG))
    for n in (5, 100):
        ob.run(n)
        b.step(n)
    default = b.tuning()["timeout_us"]
    b.set_tuning(timeout_us=2000)
    b.trip_wait(trip_at)
    with pytest.raises(nat.FlyBrainError) as e:
        b.step(60)
    assert e.value.code == nat.FB_ETIMEOUT
    b.set_tuning(timeout_us=default)
    same(ob, b, 0, "after the timeout")
    for n in (1, 1, 4, 60, 1):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, n)


@pytest.mark.parametrize("trefs,n,windows", [((0.05, 0.05, 0.05), 40, False), ((0.15, 0.15, 0.15), 40, True),
                                             ((0.05, 2.2, 2.2), 40, False), ((0.15, 2.2, 2.2), 3, True),
                                             ((2.2, 0.15, 0.05), 2, False), ((2.2, 2.2, 2.2), 2, True)])
def test_batches_of_short_windows(trefs, n, windows):
    """Windows of one step in a batch cost more than the grid kernel's steps."""
    from flybrain import BrainBatch, DeviceGraph
    from flybrain import _native as nat
    gs = [make(300 + 50 * b, 60 + b, deg=15) for b in range(3)]
    ps = [params(tRef=t, depU=0.1) for t in trefs]
    idx = np.arange(0, 300, 4, dtype=np.int32)
    obs = [pair(g, p, b + 1, idx, np.full(75, 700.0)) for b, (g, p) in enumerate(zip(gs, ps))]
    batch = BrainBatch([DeviceGraph(g) for g in gs], ps, [1, 2, 3])
    for b in range(3):
        batch.set_drive(b, idx, 700.0)
    for k in range(3):
        for ob in obs:
            ob.run(n)
        batch.step(n)
        assert batch.last_schedule() == (nat.FB_SCHEDULE_LAGGED if windows else nat.FB_SCHEDULE_GRID)
        for b, ob in enumerate(obs):
            same(ob, batch, b, (trefs, k, b))


@pytest.mark.parametrize("nD,blocks", [(511, 0), (512, 0), (1500, 0), (1500, 1), (33, 2), (2049, 0)])
@pytest.mark.parametrize("bg", [False, True])
def test_driven_lists_over_one_and_two_blocks(nD, blocks, bg):
    """Each driven block's draws follow the other's live entries; launches recorded step by step, too."""
    from flybrain import BrainBatch, DeviceGraph
    from flybrain import _native as nat
    g = make(3000, 23, deg=12)
    p = params(tRef=0.15, **(dict(BG, depU=0.1) if bg else {}))
    idx = np.random.default_rng(nD).permutation(g.N)[:nD].astype(np.int32)
    hz = np.linspace(80.0, 900.0, nD)
    ob = pair(g, p, 9, idx, hz)
    b = BrainBatch([DeviceGraph(g)], p, [9])
    b.set_drive(0, idx, hz)
    b.set_tuning(lag_driven_blocks=blocks)
    for n in (40, 7, 150):
        ob.run(n)
        b.step(n)
        assert n < 16 or b.last_schedule() == nat.FB_SCHEDULE_LAGGED
        same(ob, b, 0, (nD, n))
    counts, raster = ob.run(64, raster=True)
    b.record(64, 1 << 20)
    b.step(64)
    k, r = b.spike_log(0, 64, 1 << 20)
    np.testing.assert_array_equal(k, counts)
    np.testing.assert_array_equal(r, raster)
    same(ob, b, 0, "recorded")


@pytest.mark.parametrize("tref,delay", [(0.25, 3.2), (2.2, 0.4), (0.7, 1.8)])
@pytest.mark.parametrize("over", [dict(), dict(BG, **GEN)])
def test_recorded_launches(tref, delay, over):
    """A record of few windows is written by the windowed kernel, one of many by the other: both sides of
    the rule in turn, last windows whole and partial, counts and lists of every step."""
    ob, b = brain(params(tRef=tref, delay=delay, **over))
    for n in (5, 8, 9, 16, 12, 64, 3, 24, 20, 63, 32):
        counts, raster = ob.run(n, raster=True)
        b.record(n, 1 << 18)
        b.step(n)
        k, r = b.spike_log(0, n, 1 << 18)
        b.record(0, 0)
        np.testing.assert_array_equal(k, counts, err_msg=str(n))
        np.testing.assert_array_equal(r, raster, err_msg=str(n))
        same(ob, b, 0, (tref, n))


@pytest.mark.parametrize("n", [8, 16, 20, 40, 64])
@pytest.mark.parametrize("nD", [60, 600])
def test_recorded_lists_of_many_spikes(n, nD):
    """Every step's list is placed after the record as it was before the launch, also where the length
    after it (an even number of steps) takes the same word and one list is ready long before another."""
    from flybrain import BrainBatch, DeviceGraph
    g = make(794, 3, deg=20)
    p = params(tRef=0.15)
    idx = np.random.default_rng(1).permutation(g.N)[:nD].astype(np.int32)
    ob = pair(g, p, 5, idx, np.full(nD, 1e5))
    b = BrainBatch([DeviceGraph(g)], p, [5])
    b.set_drive(0, idx, 1e5)
    b.record(10 * n, 1 << 18)
    want = [ob.run(n, raster=True) for _ in range(10)]
    for _ in range(10):
        b.step(n)
    k, r = b.spike_log(0, 10 * n, 1 << 18)
    np.testing.assert_array_equal(k, np.concatenate([c for c, _ in want]))
    np.testing.assert_array_equal(r, np.concatenate([x for _, x in want]))
