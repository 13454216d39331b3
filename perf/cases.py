"""The work this framework is used for, as cases that can be timed and compared: the brain step
(one fly, an ensemble of flies), the differentiable brain's training step and the flyvis optic
lobe, each through the package's public classes.

listed() is a fixed set, draw(rng) one more case of the same ranges, prepare(case, seed) what a
program holds before the call, run(state) one pass, exact(case, seed) the same results from plain
torch in 64 bits, work(case) the bytes and operations of a pass.

Case fields: kind, and per kind
  run       one brain for `steps` steps in one call, then the fired list, spike counts and v
  step      one brain, `steps` calls of step(), each returning its fired list
  embodied  one simulated millisecond of the body loop: the sensory drives rewritten, two steps
            of 0.5 ms, every spike count read back
  ensemble  `trials` flies over one topology, each with its own gains, drive, seed and length
  train     loss and gradients of one differentiable brain through the autograd function
  adjoint   forward and adjoint of one differentiable brain through its own methods
  batch     forward, rasters and adjoint of `trials` differentiable brains of uneven size
  flyvis    `eyes` eyes: luminance in, `steps` steps, activity out
Graphs follow the package's synthetic connectome recipe (flybrain.synth), generated on the GPU.
"""
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
for _p in (ROOT, os.path.join(ROOT, "fly-brain_gb300")):
    if _p not in sys.path:
        sys.path.insert(0, _p)

FULL = 165122          # neurons of the whole connectome
MEAN_DEG = 66.0        # mean out-degree of the recipe (after merging duplicates)
MODELS = dict(
    # current-based, dt 0.1 ms: the synthetic workloads' parameters (flybrain.SYNTH_PARAMS)
    cuba=dict(dt=0.1, adaptInc=0.0, depU=0.0, coba=False),
    # the same at the body loop's 0.5 ms
    cuba_half_ms=dict(dt=0.5, adaptInc=0.0, depU=0.0, coba=False),
    # the application's defaults: adaptation and depression, conductances, background events
    coba=dict(dt=0.5, adaptInc=2.0, depU=0.2, coba=True, bgRate=5.0, bgAmp=1.0),
    coba_fine=dict(dt=0.1, adaptInc=2.0, depU=0.2, coba=True, bgRate=5.0, bgAmp=1.0),
)
# current-based, steep surrogate (slope 25/mV) bounded by adjClip: the benchmark's adjoint settings
DIFF_STEEP = dict(dt=0.1, wSyn=0.275, coba=False, surrogateBeta=0.04, adjClip=100.0, adaptInc=0.0, depU=0.0)
# conductance-based with adaptation and depression: LIFDiff's own model
DIFF_COBA = dict(dt=0.5, wSyn=0.5, coba=True, surrogateBeta=2.0, minSyn=3.0, adaptInc=0.3, depU=0.1)


def listed():
    return [
        # the smallest call: a game loop or script that steps a small brain one step at a time
        dict(name="step one 1.5k", kind="step", N=1501, driven=15, lo=100.0, hi=200.0, steps=1, model="coba", bias=0.0),
        # the body loop over the whole connectome, one simulated millisecond
        dict(name="embodied ms full", kind="embodied", N=FULL, driven=3000, lo=0.0, hi=200.0, model="cuba_half_ms"),
        # plain forward of a 20k subgraph, 100 ms
        dict(name="run 20k 1000", kind="run", N=20000, driven=200, lo=150.0, hi=150.0, steps=1000, model="cuba", bias=0.0),
        # the headline: the whole connectome under sensory drive, 100 ms
        dict(name="run full 1000", kind="run", N=FULL, driven=2000, lo=100.0, hi=200.0, steps=1000, model="cuba", bias=0.0),
        # the same near threshold, where recurrent spikes dominate
        dict(name="run full busy 500", kind="run", N=FULL, driven=2000, lo=100.0, hi=200.0, steps=500, model="cuba", bias=6.0),
        # the application's own model on an odd size, 100 ms
        dict(name="run 60k coba 200", kind="run", N=60013, driven=777, lo=50.0, hi=250.0, steps=200, model="coba", bias=0.0),
        # many flies of the whole connectome at once, uneven lengths
        dict(name="ensemble 96 full", kind="ensemble", N=FULL, trials=96, lo=500, hi=4000, steps=250, model="cuba"),
        # a training step of the whole connectome, fast arithmetic
        dict(name="train full f32 500", kind="train", N=FULL, driven=2000, lo=100.0, hi=200.0, steps=500,
             precision="f32", model="steep"),
        # the reference's own model and double arithmetic on a 20k subgraph
        dict(name="adjoint 20k f64 200", kind="adjoint", N=20000, driven=400, lo=50.0, hi=250.0, steps=200,
             precision="f64", model="coba"),
        # a batch of uneven subgraphs, fast arithmetic
        dict(name="batch 12 uneven f32", kind="batch", N=60000, trials=12, steps=1200, precision="f32", model="steep"),
        # both eyes of one fly, one frame
        dict(name="flyvis 2 eyes 1", kind="flyvis", N=45669, eyes=2, steps=1),
        # the eyes of many flies, two seconds of frames
        dict(name="flyvis 64 eyes 100", kind="flyvis", N=45669, eyes=64, steps=100),
    ]


def _log(rng, lo, hi):
    return int(round(float(np.exp(rng.uniform(np.log(lo), np.log(hi))))))


def draw(rng):
    kind = rng.choice(["step", "embodied", "run", "run", "ensemble", "train", "adjoint", "batch", "flyvis"])
    if kind == "flyvis":
        eyes = _log(rng, 1, 64)
        return dict(kind=kind, N=_log(rng, 3000, 45669), eyes=eyes, steps=_log(rng, 1, 100))
    if kind == "ensemble":
        N = _log(rng, 4000, FULL)
        trials = max(2, min(96, int(96 * FULL / N * rng.uniform(0.1, 1.0))))
        return dict(kind=kind, N=N, trials=trials, lo=max(1, N // 300), hi=max(2, N // 40), steps=_log(rng, 30, 250),
                    model=rng.choice(["cuba", "cuba", "coba", "coba_fine"]))
    if kind == "batch":
        return dict(kind=kind, N=_log(rng, 8000, 60000), trials=rng.randint(2, 12), steps=_log(rng, 100, 1200),
                    precision=rng.choice(["f32", "f32", "f64"]), model=rng.choice(["steep", "coba"]))
    N = _log(rng, 1500, FULL)
    if kind == "embodied":
        return dict(kind=kind, N=N, driven=max(1, int(N * rng.uniform(0.005, 0.03))), lo=0.0, hi=200.0,
                    model=rng.choice(["cuba_half_ms", "coba"]))
    c = dict(kind=kind, N=N, driven=max(1, int(N * rng.uniform(0.004, 0.02))), lo=rng.choice([50.0, 100.0]), hi=200.0)
    if kind == "step":
        return dict(c, steps=rng.randint(1, 8), model=rng.choice(["cuba", "coba"]), bias=0.0)
    if kind == "run":
        return dict(c, steps=_log(rng, 8, 1000), model=rng.choice(["cuba", "cuba", "coba", "coba_fine"]),
                    bias=rng.choice([0.0, 0.0, 3.0, 6.0]))
    return dict(c, steps=_log(rng, 40, 300 if kind == "adjoint" else 500), precision=rng.choice(["f32", "f64"]),
                model="coba" if kind == "adjoint" else "steep")


# ---- inputs -----------------------------------------------------------------------------------

def _graph(N, seed):
    """The synthetic connectome recipe (flybrain.synth) on the GPU: host arrays of a CSR graph.
    The wiring belongs to N (there is one connectome); synapse counts, signs and cell types to the
    seed."""
    from flybrain import Graph
    g = torch.Generator(device="cuda").manual_seed(N)
    z = torch.randn(N, generator=g, device="cuda")
    deg = torch.exp(3.5 + 1.2 * z).round().clamp(1, min(5000, N - 1)).long()
    pre = torch.repeat_interleave(torch.arange(N, device="cuda"), deg)
    tot, half = pre.shape[0], max(1, N // 50)
    near = (pre + torch.randint(-half, half + 1, (tot,), generator=g, device="cuda")) % N
    far = torch.randint(0, N, (tot,), generator=g, device="cuda")
    post = torch.where(torch.rand(tot, generator=g, device="cuda") < 0.8, near, far)
    key = torch.unique(pre * N + post)
    pre, post = key // N, key % N
    indptr = torch.zeros(N + 1, dtype=torch.int64, device="cuda")
    indptr[1:] = torch.cumsum(torch.bincount(pre, minlength=N), 0)
    g.manual_seed(int(seed) * 7919 + N)
    u = torch.rand(key.shape[0], generator=g, device="cuda", dtype=torch.float64).clamp_min(1e-12)
    counts = (5 + torch.floor(torch.log(u) / float(np.log(0.7)))).clamp_max(60)
    sign = torch.where(torch.rand(N, generator=g, device="cuda") < 0.6, 1.0, -1.0)
    ctype = torch.randint(0, 64, (N,), generator=g, device="cuda")
    return Graph(N, indptr.to(torch.int32).cpu().numpy().view(np.uint32),
                 post.to(torch.int32).cpu().numpy().view(np.uint32),
                 (counts * 0.275).float().cpu().numpy(), sign.float().cpu().numpy(),
                 counts.to(torch.int16).cpu().numpy().view(np.uint16), ctype.to(torch.uint8).cpu().numpy())


def _rng(case, seed):
    return np.random.default_rng([int(seed), int(case["N"]), len(case["kind"])])


def _pinned(n, dtype=torch.int32):
    return torch.zeros(n, dtype=dtype).pin_memory().numpy()


def _params(case):
    from flybrain import SYNTH_PARAMS
    return dict(SYNTH_PARAMS, **MODELS[case["model"]])


def _brain_inputs(case, seed):
    rng = _rng(case, seed)
    g = _graph(case["N"], seed)
    idx = np.sort(rng.choice(g.N, case["driven"], replace=False)).astype(np.int32)
    return g, idx, rng.uniform(case["lo"], case["hi"], idx.shape[0])


def _diff_opts(case, **more):
    base = DIFF_STEEP if case["model"] == "steep" else DIFF_COBA
    return dict(base, checkpoint=100 if case["model"] == "steep" else 16, precision=case["precision"], **more)


def _diff_net(g, idx, hz, opts, defer=False):
    from flybrain.diff import DiffNet
    net = DiffNet(dict(N=g.N, indptr=g.indptr, indices=g.indices, weights=g.counts.astype(np.float32), sign=g.sign),
                  opts, _defer=defer)
    for i, h in zip(idx.tolist(), hz.tolist()):
        net.setDriveOne(i, h)
    return net


def _batch_specs(case, seed):
    rng, shape = _rng(case, seed), _rng(case, case["trials"])
    out = []
    for k in range(case["trials"]):
        N = int(shape.integers(max(1000, case["N"] // 12), case["N"] + 1))
        steps = int(shape.integers(max(20, case["steps"] // 4), case["steps"] + 1))
        g = _graph(N, seed * 131 + k)
        idx = rng.choice(N, max(1, N // 100), replace=False)
        ro = np.sort(rng.choice(N, min(200, N), replace=False)).astype(np.int32)
        out.append(dict(g=g, idx=idx, hz=np.full(idx.shape[0], 150.0), steps=steps, readout=ro,
                        dL=rng.normal(0, 1e-3, (steps, ro.shape[0])).astype(np.float32), seed=int(rng.integers(1, 1 << 20))))
    return out


def prepare(case, seed):
    import flybrain as fb
    kind = case["kind"]
    s = dict(case=case)
    if kind in ("run", "step", "embodied"):
        g, idx, hz = _brain_inputs(case, seed)
        b = s["brain"] = fb.LIFCuda(fb.DeviceGraph(g), _params(case), seed=seed % 100003 + 1)
        b.setDrive(idx, 1.0)
        b._batch.set_drive(0, idx, np.maximum(hz, 1e-3))
        if case.get("bias"):
            b.setBias(np.arange(g.N, dtype=np.int32), case["bias"])
        if kind == "embodied":
            s["idx"] = torch.from_numpy(idx).pin_memory().numpy()
            s["rates"] = torch.from_numpy(_rng(case, seed + 1).uniform(0, 200, (16, idx.shape[0]))).pin_memory().numpy()
            s["ms"] = 0
        s["counts"], s["v"] = _pinned(g.N).view(np.uint32), _pinned(g.N, torch.float32)
        s["fired"] = _pinned(g.N)
        if kind == "step":
            s["lists"] = np.full((case["steps"], g.N), -1, np.int32)
    elif kind == "ensemble":
        rng = _rng(case, seed)
        g = _graph(case["N"], seed)
        topo = fb.DeviceGraph(g)
        counts, sign = (torch.from_numpy(x.astype(np.float32)).cuda() for x in (g.counts, g.sign))
        ctype = torch.from_numpy(g.cell_type.astype(np.int64)).cuda()
        graphs = []
        for _ in range(case["trials"]):
            gains = torch.from_numpy(rng.lognormal(0.0, 0.2, 64).astype(np.float32)).cuda()
            graphs.append(topo.compile(counts, sign, dict(_params(case), wSyn=0.275), out_scale=gains[ctype].contiguous()))
        torch.cuda.synchronize()
        b = s["batch"] = fb.BrainBatch(graphs, _params(case), rng.integers(1, 1 << 30, case["trials"]))
        for k in range(case["trials"]):
            idx = np.sort(rng.integers(0, g.N, int(rng.integers(case["lo"], case["hi"] + 1)))).astype(np.int32)
            b.set_drive(k, idx, rng.uniform(50.0, 250.0, idx.shape[0]))
        s["steps"] = rng.integers(max(1, case["steps"] // 4), case["steps"] + 1, case["trials"]).astype(np.int32)
        s["counts"] = torch.zeros((case["trials"], g.N), dtype=torch.int32).pin_memory().numpy()
    elif kind == "train":
        from flybrain.autograd import DiffContext
        g, idx, hz = _brain_inputs(case, seed)
        opts = _diff_opts(case, edgeGain=np.ones(g.E, np.float32), bias=np.zeros(g.N, np.float32),
                          outScale=np.ones(g.N, np.float32))
        rng = _rng(case, seed + 2)
        ro = np.sort(rng.choice(g.N, min(1000, g.N), replace=False))
        s["ctx"] = DiffContext(_diff_net(g, idx, hz, opts), g.cell_type, ro, case["steps"], seed=seed % 1009 + 1)
        s["target"] = torch.as_tensor(rng.uniform(0, 80, (1, ro.shape[0])), dtype=torch.float32, device="cuda")
        s["in"] = [torch.ones(g.E, device="cuda"), torch.zeros(g.N, device="cuda"),
                   torch.as_tensor(rng.lognormal(0, 0.2, 64), dtype=torch.float32, device="cuda")]
        for t in s["in"]:
            t.requires_grad_()
    elif kind == "adjoint":
        g, idx, hz = _brain_inputs(case, seed)
        s["net"] = _diff_net(g, idx, hz, _diff_opts(case))
        s["seed"] = seed % 1009 + 1
        rng = _rng(case, seed + 2)
        s["dL"] = np.zeros(g.N, np.float32)
        s["dL"][rng.choice(g.N, min(500, g.N), replace=False)] = 1e-3
    elif kind == "batch":
        from flybrain.diff import DiffBatch
        specs = s["specs"] = _batch_specs(case, seed)
        members = [_diff_net(q["g"], q["idx"], q["hz"], _diff_opts(case), defer=True) for q in specs]
        s["batch"] = DiffBatch(members, _diff_opts(case))
        s["dL"] = [torch.from_numpy(q["dL"]).cuda() for q in specs]
        s["rasters"] = [torch.zeros((q["steps"], q["readout"].shape[0]), device="cuda") for q in specs]
    else:
        m = _flyvis_model(case, seed)
        rng = _rng(case, seed)
        s["fv"] = fb.FlyVis(m, B=case["eyes"])
        s["lum"] = [rng.uniform(0, 1, 721).astype(np.float32) for _ in range(case["eyes"])]
    return s


def _flyvis_model(case, seed):
    from flybrain import synth_flyvis
    return synth_flyvis(N=case["N"], seed=seed)


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "run":
        b = s["brain"]
        b.run(case["steps"])
        n = b._batch.fired(0, out=s["fired"]).shape[0]
        return dict(n=n, fired=s["fired"], counts=b._batch.read("spikeCount", 0, out=s["counts"]).view(np.int32),
                    v=b._batch.read("v", 0, out=s["v"]))
    if kind == "step":
        b, n = s["brain"], []
        for k in range(case["steps"]):
            f = b.step()
            n.append(f.shape[0])
            s["lists"][k, :f.shape[0]] = f
        return dict(n=n, fired=s["lists"], v=b._batch.read("v", 0, out=s["v"]))
    if kind == "embodied":
        b = s["brain"]._batch
        b.set_drive(0, s["idx"], s["rates"][s["ms"] % 16])
        s["ms"] += 1
        b.step(2)
        return dict(counts=b.read("spikeCount", 0, out=s["counts"]).view(np.int32))
    if kind == "ensemble":
        b = s["batch"]
        last = b.step_uneven(s["steps"])
        for k in range(b.B):
            b.read("spikeCount", k, out=s["counts"][k].view(np.uint32))
        return dict(last=last, counts=s["counts"])
    if kind == "train":
        from flybrain.autograd import rate_loss
        loss = rate_loss(s["ctx"], s["target"], *s["in"])
        edge, bias, types = torch.autograd.grad(loss, s["in"])
        return dict(loss=loss.detach(), edge=edge, bias=bias, types=types)
    if kind == "adjoint":
        net = s["net"]
        counts = net.forward(case["steps"], seed=s["seed"])
        g = net.backward(s["dL"])
        return dict(counts=counts, edge=g["edge"], bias=g["bias"], logGain=g["logGain"],
                    params=np.array(list(g["params"].values())))
    if kind == "batch":
        b, specs = s["batch"], s["specs"]
        counts = b.forward([q["steps"] for q in specs], [q["seed"] for q in specs])
        b.rasters([q["readout"] for q in specs], s["rasters"])
        gs = b.backward(s["dL"], [q["readout"] for q in specs], device="cuda")
        return dict(counts=counts, rasters=s["rasters"], edge=[g["edge"] for g in gs], bias=[g["bias"] for g in gs])
    fv = s["fv"]
    for k, lum in enumerate(s["lum"]):
        fv.setInput(lum, k)
    fv.step(case["steps"])
    return dict(v=np.stack([fv.v(k) for k in range(case["eyes"])]))


# ---- what a pass cannot do without ------------------------------------------------------------

def work(case):
    """Inputs read and outputs written once; operations of the model's arithmetic (about 25 per
    neuron and step forward, 60 for the adjoint's replay and sweep, 2 per synaptic event)."""
    N, steps = case["N"], case.get("steps", 2)
    if case["kind"] == "flyvis":
        E = 33.0 * N
        return dict(bytes=E * 8 + N * 12 + case["eyes"] * N * 12, flops=case["eyes"] * steps * (2 * E + 5 * N))
    dt = (DIFF_STEEP if case["model"] == "steep" else MODELS[case["model"]])["dt"]
    if case["kind"] == "adjoint":
        dt = DIFF_COBA["dt"]
    if case["kind"] == "ensemble":
        ns, T = steps * 0.625 * case["trials"], case["trials"]
        ev = ns * 0.5 * (case["lo"] + case["hi"]) * 150.0 * dt / 1000 * MEAN_DEG
        return dict(bytes=T * (N * 80 + MEAN_DEG * N * 4) + MEAN_DEG * N * 4 + ev * 4, flops=25 * N * ns + 2 * ev)
    if case["kind"] == "batch":
        n = 0.54 * N * case["trials"]
        ev = n * 0.01 * 150.0 * dt / 1000 * steps * 0.625 * MEAN_DEG
        return dict(bytes=n * (80 + MEAN_DEG * 20) + ev * 8, flops=85 * n * steps * 0.625 + 8 * ev)
    ev = steps * case["driven"] * 0.5 * (case["lo"] + case["hi"]) * dt / 1000 * MEAN_DEG
    if case["kind"] in ("train", "adjoint"):
        return dict(bytes=N * (80 + MEAN_DEG * 20) + ev * 8, flops=85 * N * steps + 8 * ev)
    return dict(bytes=N * 80 + min(ev, MEAN_DEG * N) * 8, flops=25 * N * steps + 2 * ev)


# ---- the same results in 64 bits, with plain torch ---------------------------------------------

def _stream(seed, n):
    """The first n outputs of the xorshift32 stream of a brain's seed (the map is linear over
    GF(2): the next block of outputs is the last one under the map's power)."""
    m = 0xFFFFFFFF
    s = int(np.fmod(np.floor(float(seed) * 2654435761.0), 4294967296.0)) or 1

    def nxt(x):
        x ^= (x << 13) & m
        x ^= x >> 17
        return x ^ ((x << 5) & m)
    cols = [nxt(1 << b) for b in range(32)]  # the map's columns
    x = torch.tensor([nxt(s)], dtype=torch.int64, device="cuda")
    while x.shape[0] < n:
        y = torch.zeros_like(x)
        for b in range(32):
            y ^= torch.where((x >> b) & 1 == 1, cols[b], 0)
        x = torch.cat([x, y])

        def sq(v):
            r = 0
            for b in range(32):
                if v >> b & 1:
                    r ^= cols[b]
            return r
        cols = [sq(c) for c in cols]
    return x[:n]


class _Sim64:
    """A LIF network step by step in 64 bits. Refractory counts, which decide how many steps a
    neuron waits, are counted in 32 bits as the model defines them."""

    def __init__(self, g, p, idx, hz, seed, steps, weights, sign, dt32):
        f64, dev = torch.float64, "cuda"
        self.p, self.N, self.steps, self.dt32 = p, g.N, steps, dt32
        N = g.N
        self.ptr = torch.from_numpy(g.indptr.astype(np.int64)).to(dev)
        self.tgt = torch.from_numpy(g.indices.astype(np.int64)).to(dev)
        self.W, self.sign = weights, sign
        full = lambda x: torch.full((N,), float(x), dtype=f64, device=dev)  # noqa: E731
        self.v, self.gE, self.gI, self.ad, self.res = full(p["vRest"]), full(0), full(0), full(0), full(1)
        self.r = torch.zeros(N, dtype=torch.float32, device=dev)
        self.bias, self.count = full(p.get("bias0", 0.0)), full(0)
        self.D = max(1, int(np.floor(p["delay"] / p["dt"] + 0.5)))
        self.idx = torch.from_numpy(np.asarray(idx, np.int64)).to(dev)
        self.hz = torch.from_numpy(np.asarray(hz, np.float64)).to(dev)
        self.acc, self.bgE = np.float32(0), np.float32(float(N) * (p.get("bgRate") or 0.0) * p["dt"] / 1000)
        self.draws = _stream(seed, steps * (len(idx) + int(self.bgE) + 1) + 1)
        self.at = torch.zeros((), dtype=torch.int64, device=dev)
        self.lists = []   # per step: ids fired
        d = p["dt"]
        self.dE, self.dA, self.kR, self.kM = np.exp(-d / p["tauSyn"]), np.exp(-d / p["adaptTau"]), d / p["depTau"], d / p["tauM"]
        self.cE, self.cI = 1 / (p["eExc"] - p["vRest"]), 1 / (p["vRest"] - p["eInh"])

    def edges(self, ids):
        """(arrival of each edge, edge) of the rows of ids."""
        lo, n = self.ptr[ids], self.ptr[ids + 1] - self.ptr[ids]
        k = torch.repeat_interleave(torch.arange(ids.shape[0], device="cuda"), n)
        first = torch.cumsum(n, 0) - n
        return k, lo[k] + torch.arange(k.shape[0], device="cuda") - first[k]

    def step(self, t, tape=None):
        p = self.p
        arr = self.lists[t - self.D] if t >= self.D else self.idx[:0]
        resAt = self.res[arr]
        if arr.shape[0]:
            amp = self.sign[arr] * resAt
            self.res[arr] = resAt - p["depU"] * resAt
            k, j = self.edges(arr)
            c = self.W[j] * amp[k]
            self.gE.index_add_(0, self.tgt[j], torch.where(c > 0, c, 0.0))
            self.gI.index_add_(0, self.tgt[j], torch.where(c > 0, 0.0, c))
        self.acc = np.float32(self.acc + self.bgE)
        nbg = int(self.acc)
        self.acc = np.float32(self.acc - np.float32(nbg))
        if nbg:
            hit = self.draws[self.at + torch.arange(nbg, device="cuda")] % self.N
            self.gE.index_add_(0, hit, torch.full((nbg,), float(p["bgAmp"]), dtype=torch.float64, device="cuda"))
        live = ~(self.r[self.idx] > 0)
        rank = torch.cumsum(live, 0)
        u = (self.draws[(self.at + nbg + rank - 1).clamp_min(0)] >> 8).double() / 16777216.0
        forced = self.idx[live & (u < self.hz * (p["dt"] / 1000))]
        self.at = self.at + nbg + rank[-1]
        self.r[forced] = float(np.float32(np.float32(p["tRef"]) + np.float32(p["dt"])) if self.dt32 else np.float32(p["tRef"] + p["dt"]))
        self.ad[forced] += p["adaptInc"]
        if self.dt32:
            self.v[forced] = p["vReset"]
        was = self.r > 0
        dec = self.r - np.float32(p["dt"]) if self.dt32 else (self.r.double() - p["dt"]).float()
        v0, gE0, gI0 = self.v, self.gE.clone(), self.gI.clone()
        if p["coba"]:
            drive = gE0 * (p["eExc"] - v0) * self.cE + gI0 * (v0 - p["eInh"]) * self.cI
        else:
            drive = gE0 + gI0
        u_ = v0 + (p["vRest"] - v0 + drive + self.bias) * self.kM
        v = torch.where(was, torch.full_like(v0, float(p["vReset"])), u_)
        r = torch.where(was, dec, self.r)
        self.gE, self.gI = self.gE * self.dE, self.gI * self.dE
        self.ad = self.ad * self.dA
        self.res = self.res + (1 - self.res) * self.kR
        thr = p["vThresh"] + self.ad
        cross = (v >= thr) & ((r <= 0) if self.dt32 else ~was)
        if tape is not None:
            mode = was.long()
            mode[forced] = 2
            tape.append((v0, gE0, gI0, thr, cross, mode, arr, resAt))
        self.v = torch.where(cross, torch.full_like(v, float(p["vReset"])), v)
        self.r = torch.where(cross, torch.full_like(r, float(np.float32(p["tRef"]))), r)
        self.ad = self.ad + cross * p["adaptInc"]
        self.count[forced] += 1
        self.count += cross
        self.lists.append(torch.cat([forced, torch.nonzero(cross)[:, 0]]))


def _diff_sim(g, idx, hz, seed, steps, opts, out_scale=None):
    from flybrain.diff import DIFF_DEFAULTS
    p = dict(DIFF_DEFAULTS, **opts)
    cnt = torch.from_numpy(g.counts.astype(np.float64)).cuda()
    cnt = torch.where(cnt >= p["minSyn"], cnt, 0.0)
    sign = torch.from_numpy(g.sign.astype(np.float64)).cuda() * p["wSyn"]
    if out_scale is not None:
        sign = sign * out_scale
    sim = _Sim64(g, p, idx, hz, seed, steps, cnt, sign, dt32=False)
    tape = []
    for t in range(steps):
        sim.step(t, tape)
    return sim, tape


def _sweep64(sim, tape, dL):
    """The surrogate-gradient adjoint over a recorded pass: dLoss/dW per edge (W the effective
    weight), per neuron bias, and per neuron log gain. dL(t): dLoss/dspike of step t, N values."""
    p, N, D = sim.p, sim.N, sim.D
    z = lambda n=N: torch.zeros(n, dtype=torch.float64, device="cuda")  # noqa: E731
    lv, lE, lI, la, lr = z(), z(), z(), z(), z()
    ring = [z() for _ in range(D + 1)]
    gEdge, gBias, gLog = z(sim.tgt.shape[0]), z(), z()
    clip = float(p["adjClip"] or 0.0)
    cl = (lambda x: x.clamp(-clip, clip)) if clip > 0 else (lambda x: x)  # noqa: E731
    beta = p["surrogateBeta"]
    for t in range(sim.steps - 1, -1, -1):
        v0, gE, gI, thr, cross, mode, arr, resAt = tape[t]
        s = cross.double()
        lE, lI, lA, lr = lE * sim.dE, lI * sim.dE, la * sim.dA, lr * (1 - sim.kR)
        ls = ring[t % (D + 1)]
        if p["coba"]:
            u = v0 + (p["vRest"] - v0 + gE * (p["eExc"] - v0) * sim.cE + gI * (v0 - p["eInh"]) * sim.cI) * sim.kM
        else:
            u = v0 + (p["vRest"] - v0 + gE + gI) * sim.kM
        sg = 1 / (beta * (1 + (u - thr).abs() / beta) ** 2)
        lt = ((p["vReset"] - u) * lv + la * p["adaptInc"] + ls + dL(t)) * sg
        lu = lv * (1 - s) + lt
        free = mode == 0
        if p["coba"]:
            dv, dE, dI = 1 + sim.kM * (-1 - gE * sim.cE + gI * sim.cI), sim.kM * (p["eExc"] - v0) * sim.cE, sim.kM * (v0 - p["eInh"]) * sim.cI
        else:
            dv, dE, dI = 1 - sim.kM, sim.kM, sim.kM
        lv = torch.where(free, lu * dv, 0.0)
        lE, lI = torch.where(free, lE + lu * dE, lE), torch.where(free, lI + lu * dI, lI)
        la = torch.where(free, lA - lt * sim.dA, lA)
        gBias += torch.where(free, lu * sim.kM, 0.0)
        ring[t % (D + 1)] = torch.where(mode == 1, ls, 0.0)
        lv, lE, lI, la, lr = cl(lv), cl(lE), cl(lI), cl(la), cl(lr)
        if arr.shape[0]:
            k, j = sim.edges(arr)
            base = sim.sign[arr] * resAt
            lq = torch.where(base[k] > 0, lE[sim.tgt[j]], lI[sim.tgt[j]])
            on = sim.W[j] != 0
            gEdge.index_add_(0, j, torch.where(on, lq * base[k], 0.0))
            raw = torch.zeros(arr.shape[0], dtype=torch.float64, device="cuda").index_add_(0, k, lq * sim.W[j])
            gLog[arr] += raw * base
            tg = ring[(t - D) % (D + 1)]
            tg[arr] = cl(tg[arr] + raw * base)
            lr[arr] = cl(lr[arr] * (1 - p["depU"]) + raw * sim.sign[arr])
    return gEdge, gBias, gLog


def exact(case, seed):
    kind = case["kind"]
    if kind in ("run", "step"):
        # v after the pass; spike lists and counts are whole numbers
        g, idx, hz = _brain_inputs(case, seed)
        p = dict(_params(case), bias0=case.get("bias", 0.0))
        w, sg = (torch.from_numpy(x.astype(np.float64)).cuda() for x in (g.weights, g.sign))
        sim = _Sim64(g, p, idx, np.maximum(hz, 1e-3), seed % 100003 + 1, case["steps"], w, sg, dt32=True)
        for t in range(case["steps"]):
            sim.step(t)
        return dict(v=sim.v)
    if kind in ("embodied", "ensemble"):
        return None  # whole numbers only
    if kind == "flyvis":
        m = _flyvis_model(case, seed)
        rng = _rng(case, seed)
        N, B = case["N"], case["eyes"]
        from flybrain.flyvis import kdt_of
        w = torch.sparse_csr_tensor(torch.from_numpy(m["indptr"].astype(np.int64)), torch.from_numpy(m["target"].astype(np.int64)),
                                    torch.from_numpy(m["weight"].astype(np.float64)), (N, N)).cuda().to_sparse_coo().t().to_sparse_csr()
        col = lambda a: torch.from_numpy(np.asarray(a, np.float64)).cuda()[:, None]  # noqa: E731
        bias, kdt, x = col(m["bias"]), col(kdt_of(m["tau"], 0.02)), torch.zeros((N, B), dtype=torch.float64, device="cuda")
        for k in range(B):
            lum = torch.from_numpy(rng.uniform(0, 1, 721).astype(np.float32)).double().cuda()
            for ix in m["inputIdx"].values():
                x[torch.from_numpy(ix.astype(np.int64)).cuda(), k] = lum[:len(ix)]
        v = bias.expand(N, B).clone()
        for _ in range(case["steps"]):
            v = v + kdt * (-v + bias + w @ v.clamp_min(0) + x)
        return dict(v=v.t())
    if kind == "batch":
        if case["precision"] != "f64" and case["trials"] * case["steps"] > 12000:
            return None  # minutes of small torch steps
        edge, bias = [], []
        for q in _batch_specs(case, seed):
            sim, tape = _diff_sim(q["g"], q["idx"], q["hz"], q["seed"], q["steps"], _diff_opts(case))
            ro, d = torch.from_numpy(q["readout"].astype(np.int64)).cuda(), torch.from_numpy(q["dL"]).double().cuda()
            dl = lambda t: torch.zeros(q["g"].N, dtype=torch.float64, device="cuda").index_copy_(0, ro, d[t])  # noqa: E731,B023
            e, b, _ = _sweep64(sim, tape, dl)
            edge.append(e)
            bias.append(b)
        none = [None] * case["trials"]
        return dict(counts=none, rasters=none, edge=edge, bias=bias)
    g, idx, hz = _brain_inputs(case, seed)
    rng = _rng(case, seed + 2)
    if kind == "adjoint":
        dL = torch.zeros(g.N, dtype=torch.float64, device="cuda")
        dL[torch.from_numpy(rng.choice(g.N, min(500, g.N), replace=False)).cuda()] = float(np.float32(1e-3))
        sim, tape = _diff_sim(g, idx, hz, seed % 1009 + 1, case["steps"], _diff_opts(case))
        e, b, lg = _sweep64(sim, tape, lambda t: dL)
        return dict(counts=None, edge=e, bias=b, logGain=lg, params=None)
    ro = torch.from_numpy(np.sort(rng.choice(g.N, min(1000, g.N), replace=False))).cuda()
    target = torch.as_tensor(rng.uniform(0, 80, (1, ro.shape[0])), dtype=torch.float32, device="cuda").double()
    gains = torch.as_tensor(rng.lognormal(0, 0.2, 64), dtype=torch.float32, device="cuda").double()
    ct = torch.from_numpy(g.cell_type.astype(np.int64)).cuda()
    sim, tape = _diff_sim(g, idx, hz, seed % 1009 + 1, case["steps"], _diff_opts(case), out_scale=gains[ct])
    T, a = case["steps"], float(np.exp(-sim.p["dt"] / 20.0))
    c = (1 - a) / (sim.p["dt"] / 1000.0)
    r, rates = torch.zeros(ro.shape[0], dtype=torch.float64, device="cuda"), []
    for t in range(T):
        s = torch.zeros(g.N, dtype=torch.float64, device="cuda")
        s[sim.lists[t]] = 1.0
        r = a * r + c * s[ro]
        rates.append(r)
    err = torch.stack(rates) - target
    n = float(err.numel())
    d, dr = torch.zeros_like(r), [None] * T
    for t in range(T - 1, -1, -1):  # the filter's own adjoint
        d = 2 * err[t] / n + a * d
        dr[t] = c * d
    dl = lambda t: torch.zeros(g.N, dtype=torch.float64, device="cuda").index_copy_(0, ro, dr[t])  # noqa: E731
    e, b, lg = _sweep64(sim, tape, dl)
    W = torch.from_numpy(g.counts.astype(np.float64)).cuda()
    types = torch.zeros(64, dtype=torch.float64, device="cuda").index_add_(0, ct, lg / gains[ct])
    return dict(loss=(err ** 2).mean(), edge=e * W, bias=b, types=types)
