"""The windowed kernel (fly-brain_gb300/csrc/fb_window.cu) where its parts meet their limits, bit for
bit against the oracle: windows cut by the draws that fit in shared memory, by short refractory
times and by the launch's end; driven lists at the edges of the chain's warp layouts; several
background hits on one neuron and step, driven or not; targets with more contributions than a lane
or a warp sorts; batches of unequal delays, lengths and models on few and on many blocks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def make(N, seed, deg=20, hub=0):
    """A CSR graph of N neurons, `deg` targets each (each of the first `hub` targets gets an edge
    from every neuron)."""
    from flybrain import Graph
    rng = np.random.default_rng(seed)
    rows = [np.unique(np.concatenate([np.arange(hub), rng.integers(0, N, deg)])) for _ in range(N)]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])])
    E = int(indptr[-1])
    return Graph(N, indptr, np.concatenate(rows), rng.uniform(0.5, 3.0, E).astype(np.float32),
                 np.where(rng.random(N) < 0.7, 1.0, -1.0).astype(np.float32))


def pair(g, p, seed, driven, hz):
    from oracle import oracle as O
    ob = O.OracleBrain(g.N, g.indptr, g.indices, g.weights, g.sign, p, seed=seed)
    for i, h in zip(driven.tolist(), hz.tolist()):
        ob.setDriveOne(int(i), float(h))
    return ob


def same(ob, batch, b, where):
    for f in ("v", "gE", "gI", "refr", "trace", "adapt", "res", "spikeCount"):
        assert getattr(ob, f).tobytes() == batch.read(f, b).tobytes(), (where, f)
    h, s = ob._pull(), batch.scalars(b)
    assert (s["rng"], s["head"], s["nFired"], s["lastSlot"]) == (h.rng, h.head, h.nFired, h.lastSlot), where
    lists, counts, _ = batch.ring(b)
    np.testing.assert_array_equal(counts, ob.ringCount, err_msg=str(where))
    for k in range(counts.shape[0]):
        np.testing.assert_array_equal(lists[k, :counts[k]], ob.ring[k * ob.N: k * ob.N + counts[k]], err_msg=str(where))


def params(**over):
    from flybrain import SYNTH_PARAMS
    return dict(SYNTH_PARAMS, **over)


GEN = dict(coba=True, adaptInc=1.5, depU=0.15)


@pytest.mark.parametrize("nD", [0, 1, 255, 256, 257, 1023, 1025, 2047, 2049, 4095, 4096])
@pytest.mark.parametrize("gen", [False, True])
def test_driven_list_sizes(nD, gen):
    """Driven lists at the edges of the chain's layouts; 4,096 also cuts the window (their draws)."""
    from flybrain import BrainBatch, DeviceGraph
    g = make(4200, 3)
    p = params(**(dict(GEN, bgRate=6.0, bgAmp=1.0) if gen else {}))
    rng = np.random.default_rng(nD)
    idx = rng.permutation(g.N)[:nD].astype(np.int32)
    hz = rng.uniform(50, 400, nD)
    ob = pair(g, p, 5, idx, hz)
    b = BrainBatch([DeviceGraph(g)], p, [5])
    if nD:
        b.set_drive(0, idx, hz)
    for n in (37, 5):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, (nD, gen, n))


@pytest.mark.parametrize("tref,delay", [(0.05, 1.8), (0.1, 0.4), (0.35, 1.8), (2.2, 3.2), (5.0, 0.5)])
def test_window_lengths(tref, delay):
    """Windows of 1 step (refractory for less than a step) up to the key's 31."""
    from flybrain import BrainBatch, DeviceGraph
    g = make(700, 8, deg=30)
    p = params(tRef=tref, delay=delay, vThresh=-50.0, depU=0.1)
    idx = np.arange(0, 700, 9, dtype=np.int32)
    hz = np.full(idx.shape[0], 300.0)
    ob = pair(g, p, 2, idx, hz)
    b = BrainBatch([DeviceGraph(g)], p, [2])
    b.set_drive(0, idx, hz)
    for n in (50, 3, 64):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, (tref, delay, n))
    assert int(ob.spikeCount.sum()) > 0


@pytest.mark.parametrize("rate", [40.0, 1500.0])
@pytest.mark.parametrize("dt", [0.1, 0.5])
def test_background_hits(rate, dt):
    """Dense background: several hits on one neuron in one step, on driven and other neurons, strong
    enough to fire them (the driven ones' live steps change and the chain runs again)."""
    from flybrain import BrainBatch, DeviceGraph
    g = make(300, 4, deg=10)
    p = params(dt=dt, bgRate=rate, bgAmp=2.5, **GEN)
    idx = np.arange(0, 300, 3, dtype=np.int32)
    hz = np.full(100, 120.0)
    ob = pair(g, p, 9, idx, hz)
    b = BrainBatch([DeviceGraph(g)], p, [9])
    b.set_drive(0, idx, hz)
    for n in (60, 7):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, (rate, dt, n))
    assert int(ob.spikeCount.sum()) > 0


@pytest.mark.parametrize("N", [40, 120, 600])
def test_many_contributions(N):
    """Targets that every neuron reaches, most of them firing in one window: 16 and 128 contributions
    are what a lane and a warp sort."""
    from flybrain import BrainBatch, DeviceGraph
    g = make(N, 6, deg=4, hub=6)
    p = params(**GEN)
    idx = np.arange(1, N, dtype=np.int32)  # hub 0 is not driven, the others are
    hz = np.full(N - 1, 3000.0)
    ob = pair(g, p, 3, idx, hz)
    b = BrainBatch([DeviceGraph(g)], p, [3])
    b.set_drive(0, idx, hz)
    for n in (40, 19):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, (N, n))


@pytest.mark.parametrize("B", [2, 20, 160])
def test_batches(B):
    """Brains of unequal size, delay, model and length in one launch: on blocks of their own, and on
    blocks that also deliver and update, one and two lists each."""
    from flybrain import BrainBatch, DeviceGraph
    rng = np.random.default_rng(B)
    gs = [make(int(n), 10 + k, deg=12) for k, n in enumerate((150, 333, 64))]
    dgs = [DeviceGraph(g) for g in gs]
    ps = [params(), params(dt=0.5, bgRate=20.0, bgAmp=1.5, **GEN), params(delay=0.7, depU=0.2, bgRate=9.0, bgAmp=2.0)]
    obs, drives = [], []
    for b in range(B):
        g = gs[b % 3]
        idx = rng.permutation(g.N)[:int(rng.integers(1, g.N // 2))].astype(np.int32)
        drives.append((idx, rng.uniform(50, 300, idx.shape[0])))
        obs.append(pair(g, ps[(b // 2) % 3], b + 1, *drives[-1]))
    batch = BrainBatch([dgs[b % 3] for b in range(B)], [ps[(b // 2) % 3] for b in range(B)], np.arange(1, B + 1))
    for b, (idx, hz) in enumerate(drives):
        batch.set_drive(b, idx, hz)
    done = np.zeros(B, np.int64)
    for top in (90, 25):
        steps = rng.integers(0, top, B).astype(np.int32)
        done += steps
        for b in range(B):
            obs[b].run(int(steps[b]))
        batch.step_uneven(steps)
        for b in range(B):
            if done[b]:
                same(obs[b], batch, b, (B, top, b))


def test_state_written_between_launches():
    """Refractory counts cleared from the host: neurons fire sooner than their refractory time, while
    spikes of theirs are still in flight."""
    from flybrain import BrainBatch, DeviceGraph
    g = make(400, 12, deg=15)
    p = params(vThresh=-50.5, **GEN)
    idx = np.arange(0, 400, 4, dtype=np.int32)
    hz = np.full(100, 800.0)
    ob = pair(g, p, 7, idx, hz)
    b = BrainBatch([DeviceGraph(g)], p, [7])
    b.set_drive(0, idx, hz)
    for n in (30, 6, 45):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, n)
        ob.refr[:] = 0.0
        b.write("refr", 0, np.zeros(g.N, np.float32))
    b.set_params(0, dict(p, tRef=0.3))
    ob._pull()
    ob.hdr.c[4] = float(np.float32(0.3))  # the header's tRef
    ob._push()
    for n in (25, 40):
        ob.run(n)
        b.step(n)
        same(ob, b, 0, ("tRef", n))
