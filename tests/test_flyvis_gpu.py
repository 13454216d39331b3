"""The flyvis kernel (fb_flyvis_*, fly-brain_gb300/csrc/fb_flyvis.cu) against the reference's
fv_step: the golden run bit for bit, full-size eyes against the oracle, input semantics."""
import os

import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _golden():
    z = np.load(os.path.join(GOLDEN, "flyvis", "flyvis_synth.npz"))
    m = dict(N=int(z["N"]), E=int(z["E"]), indptr=z["indptr"], target=z["target"], weight=z["weight"],
             bias=z["bias"], tau=z["tau"], dt=float(z["dt"]))
    return m, z


def test_golden_run_bit_for_bit():
    from flybrain.flyvis import FlyVis
    m, z = _golden()
    B = z["x"].shape[0]
    fv = FlyVis(m, B=B)
    for b in range(B):
        fv.write("x", b, z["x"][b])
        np.testing.assert_array_equal(fv.v(b), m["bias"])
    done = 0
    for k, upto in enumerate(z["steps"]):
        fv.step(int(upto) - done)
        done = int(upto)
        for b in range(B):
            assert fv.v(b).tobytes() == z["v"][k][b].tobytes(), (int(upto), b)


@pytest.mark.parametrize("B", [1, 2, 5, 33, 64])
def test_full_size_eyes_match_the_oracle(B):
    from oracle import oracle as O
    from flybrain.flyvis import FlyVis, synth_flyvis
    m = synth_flyvis(seed=7)
    rng = np.random.default_rng(B)
    x = rng.normal(0.2, 0.6, (B, m["N"])).astype(np.float32)
    fv = FlyVis(m, B=B)
    for b in range(B):
        fv.write("x", b, x[b])
    fv.step(25)
    v = np.tile(m["bias"], (B, 1)).astype(np.float32)
    O.fv_run(m, v, x, 25)
    for b in range(B):
        assert fv.v(b).tobytes() == v[b].tobytes(), b


def test_set_input_and_reset():
    """setInput writes luminance into every input type's nodes, per column (src/flyvis.js:20-21);
    a repeated index keeps its last value; reset puts v back to bias for one eye."""
    from flybrain.flyvis import FlyVis, synth_flyvis
    m = synth_flyvis(N=63 * 12, seed=3, columns=12)
    fv = FlyVis(m, B=2)
    lum = np.linspace(0, 1, 12).astype(np.float32)
    fv.setInput(lum, 1)
    x1 = fv.read("x", 1)
    for ix in m["inputIdx"].values():
        np.testing.assert_array_equal(x1[ix], lum[:ix.shape[0]])
    assert not fv.read("x", 0).any()
    fv.set_input([3, 4, 3], [1.0, 2.0, 5.0], 0)
    x0 = fv.read("x", 0)
    assert x0[3] == 5.0 and x0[4] == 2.0
    fv.step(5)
    assert not np.array_equal(fv.v(1), m["bias"])
    fv.reset(1)
    np.testing.assert_array_equal(fv.v(1), m["bias"])
    assert not np.array_equal(fv.v(0), m["bias"])
    from flybrain import _native as nat
    with pytest.raises(nat.FlyBrainError):
        fv.set_input([m["N"]], [1.0], 0)


@pytest.mark.parametrize("finite", [True, False])
@pytest.mark.parametrize("N", [1, 37, 3000])
@pytest.mark.parametrize("B", [1, 2, 3, 4, 6, 63, 66, 132])
def test_vectors_chunks_and_weights(B, N, finite):
    """Rows of whole and of padded vectors, one and several chunks of them, lists that end within a
    group of four or are empty, several calls of one and more steps; weights that are not finite
    (an inactive source must not meet them)."""
    from oracle import oracle as O
    from flybrain.flyvis import FlyVis
    rng = np.random.default_rng(B * 7 + N)
    deg = rng.integers(0, 12, N) * (rng.random(N) < 0.8)
    indptr = np.concatenate([[0], np.cumsum(deg)]).astype(np.int32)
    E = int(indptr[-1])
    w = rng.normal(0, 0.3, E).astype(np.float32)
    if not finite and E:
        w[:: max(1, E // 5)] = np.inf
    m = dict(N=N, E=E, indptr=indptr, target=rng.integers(0, N, E).astype(np.int32), weight=w,
             bias=rng.normal(0, 0.5, N).astype(np.float32), tau=rng.uniform(0.02, 0.2, N).astype(np.float32), dt=0.02)
    x = rng.normal(0.0, 0.6, (B, N)).astype(np.float32)
    fv = FlyVis(m, B=B)
    v = np.tile(m["bias"], (B, 1)).astype(np.float32)
    for b in range(B):
        fv.write("x", b, x[b])
    for steps in (1, 4, 1):
        fv.step(steps)
        O.fv_run(m, v, x, steps)
        for b in range(B):
            np.testing.assert_array_equal(fv.v(b), v[b])
        v[0] = -v[0]
        fv.write("v", 0, v[0])


@pytest.mark.parametrize("n", [1, 1024, 1025, 8192, 8193])
def test_input_lists(n):
    """Lists that a block holds in registers and longer ones, each index several times (its last
    value stays), a bad index among them (an error, the rest written)."""
    from flybrain import _native as nat
    from flybrain.flyvis import FlyVis, synth_flyvis
    m = synth_flyvis(N=700, seed=3, columns=12)
    rng = np.random.default_rng(n)
    fv = FlyVis(m, B=3)
    for k in range(2):
        idx = rng.integers(0, 700, n).astype(np.int32)
        val = rng.normal(0, 1, n).astype(np.float32)
        bad = k == 1 and n > 1
        if bad:
            idx[n // 2] = 700
        ref = fv.read("x", 1)
        ok = idx < 700
        for i, y in zip(idx[ok], val[ok]):
            ref[i] = y
        if bad:
            with pytest.raises(nat.FlyBrainError):
                fv.set_input(idx, val, 1)
        else:
            fv.set_input(idx, val, 1)
        np.testing.assert_array_equal(fv.read("x", 1), ref)
    assert not fv.read("x", 0).any() and not fv.read("x", 2).any()


@pytest.mark.parametrize("N,B", [(33333, 3), (33334, 3), (25000, 4), (25001, 4), (60000, 5), (60001, 5), (42857, 7),
                                 (42858, 7), (50001, 6),
                                 (45669, 21), (45669, 22), (10001, 101)])
def test_instances_per_lane(N, B):
    """Both sides of where a lane takes two and four instances, calls of one and of several steps."""
    from oracle import oracle as O
    from flybrain.flyvis import FlyVis, synth_flyvis
    m = synth_flyvis(N=N, seed=5, mean_in=6.0)
    rng = np.random.default_rng(N)
    x = rng.normal(0.0, 0.6, (B, N)).astype(np.float32)
    fv = FlyVis(m, B=B)
    v = np.tile(m["bias"], (B, 1)).astype(np.float32)
    for b in range(B):
        fv.write("x", b, x[b])
    for steps in (1, 3):
        fv.step(steps)
        O.fv_run(m, v, x, steps)
        for b in range(B):
            np.testing.assert_array_equal(fv.v(b), v[b])


@pytest.mark.parametrize("N,B", [(1000, 64), (1000, 65), (700, 129), (20000, 17), (20000, 66), (22222, 99), (22223, 99)])
def test_odd_eyes(N, B):
    """Rows whose padding has no lanes, chunks of 64 words and one more, and both sides of where a call
    first makes the rectified rows; calls of one and of several steps."""
    from oracle import oracle as O
    from flybrain.flyvis import FlyVis, synth_flyvis
    m = synth_flyvis(N=N, seed=6, mean_in=5.0)
    rng = np.random.default_rng(N + B)
    x = rng.normal(0.0, 0.6, (B, N)).astype(np.float32)
    fv = FlyVis(m, B=B)
    v = np.tile(m["bias"], (B, 1)).astype(np.float32)
    for b in range(B):
        fv.write("x", b, x[b])
    for steps in (2, 1, 4):
        fv.step(steps)
        O.fv_run(m, v, x, steps)
        for b in range(B):
            np.testing.assert_array_equal(fv.v(b), v[b])


def test_many_input_lists():
    """The lists before, at and after the one that brings the pinned copy (the 32nd), a bad index in
    some."""
    from flybrain import _native as nat
    from flybrain.flyvis import FlyVis, synth_flyvis
    m = synth_flyvis(N=700, seed=4, columns=12)
    rng = np.random.default_rng(9)
    fv = FlyVis(m, B=2)
    ref = np.zeros(700, np.float32)
    for k in range(36):
        idx = rng.integers(0, 700, 500).astype(np.int32)
        val = rng.normal(0, 1, 500).astype(np.float32)
        bad = k % 3 == 1
        if bad:
            idx[77] = -1
        for i, y in zip(idx, val):
            if i >= 0:
                ref[i] = y
        if bad:
            with pytest.raises(nat.FlyBrainError):
                fv.set_input(idx, val, 1)
        else:
            fv.set_input(idx, val, 1)
        np.testing.assert_array_equal(fv.read("x", 1), ref)
    assert not fv.read("x", 0).any()
