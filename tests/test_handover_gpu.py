"""Spikes in flight across everything that can stand between two launches of the step kernels: reads
of the ring, resets, new parameters, host writes of the refractory count, launches that time out. The
windowed kernel (fly-brain_gb300/csrc/fb_window.cu) keeps them in its log and the grid kernel
(fb_step.cu) in the ring's lists and slot records; after each single step every state word, the
generator and the ring equal the oracle's."""
import numpy as np
import pytest

from test_window_gpu import GEN, make, pair, params, same

pytestmark = pytest.mark.gpu

DEP = dict(depU=0.2, adaptInc=0.5)


def brains(B, p, N=400, hz=2000.0, every=4, deg=20):
    from flybrain import BrainBatch, DeviceGraph
    gs = [make(N + 30 * b, 40 + b, deg=deg) for b in range(B)]
    batch = BrainBatch([DeviceGraph(g) for g in gs], p, np.arange(1, B + 1))
    obs = []
    for b, g in enumerate(gs):
        idx = np.arange(0, g.N, every, dtype=np.int32)
        obs.append(pair(g, p, b + 1, idx, np.full(idx.shape[0], hz)))
        batch.set_drive(b, idx, hz)
    return obs, batch


def steps(obs, batch, n, where):
    for k in range(n):
        for ob in obs:
            ob.run(1)
        batch.step(1)
        for b, ob in enumerate(obs):
            same(ob, batch, b, (where, k, b))


def set_tref(ob, batch, b, p, tref):
    batch.set_params(b, dict(p, tRef=tref))
    ob._pull()
    ob.hdr.c[4] = float(np.float32(tref))  # the header's tRef
    ob._push()


@pytest.mark.parametrize("what", ["ring", "reset", "params", "timeout"])
@pytest.mark.parametrize("before", [0, 5])  # steps of the grid kernel first: slot records of its own
def test_single_steps_after_a_windowed_launch(what, before):
    """The grid kernel delivers what the windowed one left in flight, also when the ring's lists were
    taken from the log earlier than at its launch."""
    from flybrain import _native as nat
    p = params(**DEP)
    obs, batch = brains(3 if what == "reset" else 1, p)
    batch.set_schedule(nat.FB_SCHEDULE_GRID)
    steps(obs, batch, before, "before")
    forced = what == "timeout"
    batch.set_schedule(nat.FB_SCHEDULE_LAGGED if forced else nat.FB_SCHEDULE_AUTO)
    for ob in obs:
        ob.run(50)
    batch.step(50)
    assert batch.last_schedule() == nat.FB_SCHEDULE_LAGGED
    if what == "ring":
        batch.ring(0)
    elif what == "reset":
        obs[0].reset()
        batch.reset(0)
    elif what == "params":
        set_tref(obs[0], batch, 0, p, 1.3)
    else:
        default = batch.tuning()["timeout_us"]
        batch.set_tuning(timeout_us=2000)
        batch.trip_wait(7)
        with pytest.raises(nat.FlyBrainError) as e:
            batch.step(40)
        assert e.value.code == nat.FB_ETIMEOUT
        batch.set_tuning(timeout_us=default)
        batch.set_schedule(nat.FB_SCHEDULE_AUTO)
    assert sum(int(ob.ringCount.sum()) for ob in obs) > 30
    steps(obs, batch, 25, what)
    assert batch.last_schedule() == nat.FB_SCHEDULE_GRID


@pytest.mark.parametrize("rest", [[[(0, 40), (5, 0), (45, 5)]], [[(3, 25), (60, 70)], [(2, 100), (7, 0), (40, 60), (50, 1)]]])
def test_refractory_write_of_a_brain_that_waits(rest):
    """What a write of refr allows (two spikes of a neuron in flight closer than its refractory time)
    holds for as many steps of that brain, however far the others are taken meanwhile."""
    p = params(**DEP)
    obs, batch = brains(2, p, hz=5000.0)

    def go(n):
        for ob, k in zip(obs, n):
            ob.run(k)
        batch.step_uneven(np.array(n, np.int32))
        for b, ob in enumerate(obs):
            same(ob, batch, b, (n, b))

    go((30, 30))
    for n in rest:
        obs[0].refr[:] = 0.0
        batch.write("refr", 0, np.zeros(obs[0].N, np.float32))
        for m in n:
            go(m)


def test_refractory_write_before_a_launch_that_times_out():
    """The launch leaves the brain as it was, what the write allows included."""
    from flybrain import _native as nat
    obs, batch = brains(1, params(**DEP), hz=5000.0)
    ob = obs[0]
    ob.run(30)
    batch.step(30)
    ob.refr[:] = 0.0
    batch.write("refr", 0, np.zeros(ob.N, np.float32))
    default = batch.tuning()["timeout_us"]
    for trip, n in ((2, 100), (25, 100), (90, 100), (3, 12)):
        batch.set_tuning(timeout_us=2000)
        batch.trip_wait(trip)
        with pytest.raises(nat.FlyBrainError) as e:
            batch.step(n)
        assert e.value.code == nat.FB_ETIMEOUT
        batch.set_tuning(timeout_us=default)
        same(ob, batch, 0, ("timeout", trip))
    for n in (5, 100, 1, 30):
        ob.run(n)
        batch.step(n)
        same(ob, batch, 0, n)


@pytest.mark.parametrize("B", [1, 2])
@pytest.mark.parametrize("n", [2, 12])
def test_refractory_written_before_every_launch(n, B):
    """Every neuron fires in every launch: far more spikes in flight than the refractory time allows."""
    from flybrain import _native as nat
    obs, batch = brains(B, params(), hz=1e5, every=1)
    for k in range(12):
        for b, ob in enumerate(obs):
            ob.refr[:] = 0.0
            batch.write("refr", b, np.zeros(ob.N, np.float32))
            ob.run(n)
        batch.step(n)
        for b, ob in enumerate(obs):
            same(ob, batch, b, (n, k, b))
    if n == 2:
        assert int(obs[0].ringCount.sum()) > 8 * obs[0].N
    for ob in obs:
        ob.run(70)
    batch.step(70)
    assert batch.last_schedule() == nat.FB_SCHEDULE_LAGGED
    for b, ob in enumerate(obs):
        same(ob, batch, b, ("after", b))


@pytest.mark.parametrize("trefs", [(0.15, 2.2, 0.6), (2.2, 0.0, 1.0)])
def test_refractory_time_changed(trefs):
    """The spikes in flight are those of the refractory time before."""
    p = params(depU=0.1)
    obs, batch = brains(2, dict(p, tRef=trefs[0]), hz=1e5, every=1)
    for k, tref in enumerate(trefs):
        if k:
            for b, ob in enumerate(obs):
                set_tref(ob, batch, b, p, tref)
        for n in (6, 30, 64):
            for ob in obs:
                ob.run(n)
            batch.step(n)
            for b, ob in enumerate(obs):
                same(ob, batch, b, (trefs, tref, n, b))


def test_refractory_count_that_is_not_a_number():
    """It is neither over zero nor at most zero (lif.c:61-76): the neuron integrates and never fires."""
    for B in (1, 3):
        obs, batch = brains(B, params(), hz=300.0)
        ix = np.arange(1, 400, 3)
        for b, ob in enumerate(obs):
            ob.setBias(np.arange(ob.N), 9.0)
            batch.set_bias(b, np.arange(ob.N, dtype=np.int32), 9.0)
            r = np.zeros(ob.N, np.float32)
            r[ix] = np.nan
            ob.refr[:] = r
            batch.write("refr", b, r)
        for n in (30, 100, 40):
            for ob in obs:
                ob.run(n)
            batch.step(n)
            for b, ob in enumerate(obs):
                same(ob, batch, b, (B, n, b))
        assert int(obs[0].spikeCount.sum()) > 200


def test_single_steps_take_no_window_buffers():
    """The windowed kernel's buffers (8 bytes per edge and more) come with the first windowed launch."""
    import torch
    from flybrain import BrainBatch, DeviceGraph
    from flybrain import _native as nat
    g = make(1500, 3, deg=4000)
    batch = BrainBatch([DeviceGraph(g)] * 2, params(), [1, 2])
    for b in range(2):
        batch.set_drive(b, np.arange(50, dtype=np.int32), 200.0)
    batch.step(1)
    batch.set_schedule(nat.FB_SCHEDULE_GRID)
    batch.step(20)
    before = torch.cuda.mem_get_info()[0]
    batch.set_schedule(nat.FB_SCHEDULE_AUTO)
    batch.step(20)
    assert batch.last_schedule() == nat.FB_SCHEDULE_LAGGED
    assert before - torch.cuda.mem_get_info()[0] >= 2 * 8 * g.E


@pytest.mark.parametrize("nD", [1, 511, 512, 513, 1700])
@pytest.mark.parametrize("B", [1, 3])
def test_fired_lists_handed_over(nD, B):
    """Lists of as many spikes as the export has threads (512), fewer and more, out of the log and back
    into it, several slots at once."""
    p = params(tRef=0.9, **DEP)
    obs, batch = brains(B, p, N=2000, hz=1e5, every=1)
    for b, ob in enumerate(obs):
        for i in range(nD, ob.N):
            ob.setDriveOne(i, 0.0)
        batch.set_drive(b, np.arange(nD, ob.N, dtype=np.int32), 0.0)
    most = 0
    for n in (13, 1, 1, 24, 1, 3, 40, 1):
        for ob in obs:
            ob.run(n)
        batch.step(n)
        most = max(most, int(obs[0].ringCount.max()))
        for b, ob in enumerate(obs):
            same(ob, batch, b, (nD, n, b))
    assert most >= nD


@pytest.mark.parametrize("N,n,first", [(400, 2, 5), (400, 5, 5), (400, 6, 1), (12000, 3, 2), (12000, 4, 1), (12000, 5, 1)])
def test_short_launches_between_single_steps(N, n, first):
    """They stay on the grid kernel where the way into the log and back costs more: `first` is the
    launch after a single step that takes windows."""
    from flybrain import _native as nat
    obs, batch = brains(1, params(**DEP), N=N, hz=2000.0, deg=6)
    ob = obs[0]
    since = 100
    for k, m in enumerate([30, 1, n, 1] + 7 * [n] + [1, n, n, 1]):
        ob.run(m)
        batch.step(m)
        since = 0 if m == 1 else since + 1
        want = nat.FB_SCHEDULE_LAGGED if m > 1 and since >= first else nat.FB_SCHEDULE_GRID
        assert batch.last_schedule() == want, k
        same(ob, batch, 0, (N, n, k))


@pytest.mark.parametrize("trefs", [(2.2, 3.0, 2.2, 1.6, 2.4), (2.2, 0.0, 2.2, 0.3, 0.2, 1.8)])
def test_new_refractory_times_keep_the_window_buffers(trefs):
    """They are made again only where the log must hold more spikes than before."""
    import torch
    p = params(depU=0.1)
    obs, batch = brains(1, p, N=1500, hz=1e5, every=2, deg=700)
    ob = obs[0]
    free = None
    for k, tref in enumerate(trefs):
        set_tref(ob, batch, 0, p, tref)
        for n in (6, 90, 25):
            ob.run(n)
            batch.step(n)
            same(ob, batch, 0, (tref, n))
        if k == 0:
            free = torch.cuda.mem_get_info()[0]
        elif min(trefs) > 1.0:
            assert torch.cuda.mem_get_info()[0] == free, tref


@pytest.mark.parametrize("B", [1, 2])
def test_driven_lists_replaced(B):
    """The windows' places in the driven lists follow lists that shrink, grow past a block's threads, turn
    around, empty and come back, also past what windows take; background hits look them up."""
    p = params(bgRate=30.0, bgAmp=1.0, **GEN)
    obs, batch = brains(B, p, N=4500, hz=300.0, every=1500, deg=6)
    rng = np.random.default_rng(4)
    now = [list(range(0, ob.N, 1500)) for ob in obs]
    for nD in (3, 1100, 40, 0, 4096, 4200, 1023, 1025, 1):
        for b in range(B if nD != 40 else 1):  # one brain's alone, too
            new = rng.permutation(obs[b].N)[:nD].astype(np.int32)
            for i in now[b]:
                obs[b].setDriveOne(int(i), 0.0)
            batch.set_drive(b, np.array(now[b], np.int32), 0.0)
            for i in new:
                obs[b].setDriveOne(int(i), 150.0)
            batch.set_drive(b, new, 150.0)
            now[b] = new.tolist()
        for n in (4, 30):
            for ob in obs:
                ob.run(n)
            batch.step(n)
            for b, ob in enumerate(obs):
                same(ob, batch, b, (nD, n, b))


@pytest.mark.parametrize("deg,first", [(20, 1), (700, 5)])
def test_first_short_launches(deg, first):
    """The windowed kernel's buffers are made for the fifth short launch where they cost something."""
    from flybrain import _native as nat
    obs, batch = brains(1, params(**DEP), deg=deg)
    ob = obs[0]
    for k, n in enumerate((2, 3, 7, 2, 4, 2, 9, 1)):
        ob.run(n)
        batch.step(n)
        assert batch.last_schedule() == (nat.FB_SCHEDULE_LAGGED if k + 1 >= first and n > 1 else nat.FB_SCHEDULE_GRID), k
        same(ob, batch, 0, (deg, k))
