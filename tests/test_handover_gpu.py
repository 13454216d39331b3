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
