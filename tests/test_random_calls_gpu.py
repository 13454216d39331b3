"""Random sequences of calls on two batches of the same brains: one left to choose its kernels (windowed,
lagged, grid), one on the grid kernel, which the other tests hold to the oracle. Between launches of all
lengths: resets, host writes of refr, new parameters, drives, background, thresholds, biases, conductances,
reads of the ring and of fired lists, recording. State, generator, rings and records are equal bit for bit."""
import numpy as np
import pytest

from test_window_gpu import make, params

pytestmark = pytest.mark.gpu

FIELDS = ("v", "gE", "gI", "refr", "trace", "adapt", "res", "spikeCount")


def same(a, b, where):
    for k in range(a.B):
        for f in FIELDS:
            assert a.read(f, k).tobytes() == b.read(f, k).tobytes(), (where, k, f)
        assert a.scalars(k) == b.scalars(k), (where, k)


def same_rings(a, b, where):
    for k in range(a.B):
        (la, ca, ha), (lb, cb, hb) = a.ring(k), b.ring(k)
        assert ha == hb and np.array_equal(ca, cb), (where, k)
        for s, c in enumerate(ca):
            assert np.array_equal(la[s, :c], lb[s, :c]), (where, k, s)


def model(rng, dt, delay):
    p = params(dt=dt, delay=delay, tRef=float(rng.choice([2.2, 2.2, 2.2, 0.3, 0.6, 0.12, 1.3, 0.05, 0.0, 4.0])))
    if rng.random() < 0.5:
        p.update(coba=True, adaptInc=float(rng.choice([0, 1.5])), depU=float(rng.choice([0, 0.2])))
    if rng.random() < 0.4:
        p.update(bgRate=float(rng.choice([3, 40, 400])), bgAmp=1.2)
    return p


@pytest.mark.parametrize("seed", range(30))
def test_random_calls(seed):
    from flybrain import BrainBatch, DeviceGraph
    from flybrain import _native as nat
    rng = np.random.default_rng(seed)
    B = int(rng.choice([1, 1, 1, 2, 3, 5]))
    big = seed % 6 == 5  # networks on the other side of the rules for short launches
    N = [int(rng.integers(9000, 13000)) if big else int(rng.integers(40, 900)) for _ in range(B)]
    graphs = [DeviceGraph(make(n, seed * 7 + k, deg=5 if big else int(rng.choice([4, 20, 90])))) for k, n in enumerate(N)]
    dt = float(rng.choice([0.1, 0.5]))
    delays = [float(rng.choice([1.8, 1.8, 3.2, 0.9] if dt == 0.1 else [1.8, 2.5, 9.0])) for _ in range(B)]
    ps = [model(rng, dt, d) for d in delays]
    seeds = rng.integers(1, 1 << 20, B)
    both = a, b = BrainBatch(graphs, ps, seeds), BrainBatch(graphs, ps, seeds)
    b.set_schedule(nat.FB_SCHEDULE_GRID)
    hz = float(rng.choice([50, 300, 2000, 1e5]))

    def each(call):
        return [call(x) for x in both]

    for k in range(B):
        idx = rng.permutation(N[k])[: int(rng.integers(0, N[k] // 2 + 1))].astype(np.int32)
        if idx.size:
            each(lambda x: x.set_drive(k, idx, hz))
    record = 0
    for op in range(50):
        k, r = int(rng.integers(0, B)), rng.random()
        half = rng.permutation(N[k])[: N[k] // 2].astype(np.int32)
        if r < 0.55:
            n = int(rng.choice([1, 1, 2, 2, 3, 4, 5, 6, 7, 8, 12, 20, 33, 64, 100, 150]))
            n = min(n, record) if record else n
            x, y = each(lambda q: q.step(n))
            assert np.array_equal(x, y), op
        elif r < 0.63:
            n = rng.integers(0, 60, B) * (rng.random(B) < 0.7)
            n = np.minimum(n, record) if record else n
            each(lambda q: q.step_uneven(n))
        elif r < 0.67:
            which = k if rng.random() < 0.7 else -1
            each(lambda q: q.reset(which))
        elif r < 0.72:
            refr = np.where(rng.random(N[k]) < 0.7, 0.0, rng.uniform(-1, 3, N[k])).astype(np.float32)
            each(lambda q: q.write("refr", k, refr))
        elif r < 0.76:
            p = model(rng, dt, delays[k])
            each(lambda q: q.set_params(k, p))
        elif r < 0.81:
            some = half[: int(rng.integers(1, max(2, N[k] // 3)))]
            rate = 0.0 if rng.random() < 0.5 else hz
            each(lambda q: q.set_drive(k, some, rate))
        elif r < 0.84:
            rate = float(rng.choice([0, 5, 100]))
            each(lambda q: q.set_background(k, rate, 1.0))
        elif r < 0.87:
            mv = float(rng.choice([-3, 0, 2]))
            each(lambda q: q.set_thr(k, half, mv))
        elif r < 0.90:
            mv = float(rng.choice([0, 4, 9]))
            each(lambda q: q.set_bias(k, half, mv))
        elif r < 0.92:
            each(lambda q: q.add_g(k, half, 2.0, -0.5))
        elif r < 0.95:
            same_rings(a, b, op)
        elif r < 0.97:
            assert np.array_equal(*each(lambda q: q.fired(k))), op
        else:
            record = 0 if record else int(rng.choice([8, 20, 64]))
            each(lambda q: q.record(512 if record else 0, 1 << 18 if record else 0))
        if rng.random() < 0.4:
            same(a, b, op)
        if record and rng.random() < 0.4:
            for q in range(B):
                (ca, ra), (cb, rb) = each(lambda x: x.spike_log(q, 512, 1 << 18))
                assert np.array_equal(ca, cb) and np.array_equal(ra, rb), (op, q)
    same(a, b, "end")
    same_rings(a, b, "end")
