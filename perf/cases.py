"""The work that a user of this framework has it do, as measurable cases.

Four kinds of work, each through the package's public entry points:

  forward  host input events through ``forward`` (one sample, one call) or
           ``forward_batched`` (many samples, uneven step counts)
  encoded  features encoded on the device, a run created, launched and
           fetched: the data-set evaluation loop
  eprop    one e-prop training minibatch with the weights read back, or the
           gradient of one (a rank's share of a data-parallel update)
  core     one spiking BPTT layer, forward and backward
  lm       one training step of the spiking language model

over four graph families: small feed-forward nets (a sample's state fits one
SM many times over), the recurrent audio net (just fits one SM), torus grids
(need the whole GPU), and ring-local recurrent language-model layers.

Weights of the nets that run in an unordered delivery mode lie on a fixed
grid of 2^-16 or finer, as a fixed-point export has them: their sums are the
same in every order, so a spike train is one value in every mode.
"""
import math

import numpy as np
import torch
import torch.nn.functional as F

from snc_b200 import bptt, eprop, runtime, workloads
from snc_b200.graph import INPUT, INTERNAL, OUTPUT, SNNGraph

MODES = {"sort": runtime.MODE_SORT, "bucket": runtime.MODE_BUCKET, "atomic": runtime.MODE_ATOMIC}


def listed():
    return [
        # one small sample per call, as an online classifier runs it: latency
        {"name": "call_ff784", "kind": "forward", "net": "ff", "n_in": 784, "n_hid": 256, "n_out": 10,
         "fan": 10, "max_delay": 4, "samples": 1, "t_min": 50, "t_max": 50, "rate": 0.1, "mode": "sort"},
        # a batch of image-sized samples with equal lengths
        {"name": "batch_ff784", "kind": "forward", "net": "ff", "n_in": 784, "n_hid": 256, "n_out": 10,
         "fan": 10, "max_delay": 4, "samples": 64, "t_min": 50, "t_max": 50, "rate": 0.1, "mode": "sort"},
        # one long sample of a large recurrent substrate, bit-exact delivery
        {"name": "grid100k_sort", "kind": "forward", "net": "grid", "width": 400, "height": 250,
         "degree": 100, "max_delay": 30, "samples": 1, "t_min": 1000, "t_max": 1000, "rate": 0.02,
         "mode": "sort"},
        # the same with the fastest unordered delivery
        {"name": "grid100k_bucket", "kind": "forward", "net": "grid", "width": 400, "height": 250,
         "degree": 100, "max_delay": 30, "samples": 1, "t_min": 1000, "t_max": 1000, "rate": 0.02,
         "mode": "bucket"},
        # several uneven samples of a mid-size substrate with odd sizes
        {"name": "grid12k_ragged", "kind": "forward", "net": "grid", "width": 123, "height": 97,
         "degree": 50, "max_delay": 11, "samples": 5, "t_min": 60, "t_max": 250, "rate": 0.03,
         "mode": "sort"},
        # evaluation of an audio data set: uneven lengths, Poisson encoding,
        # bit-exact delivery
        {"name": "audio_eval_sort", "kind": "encoded", "net": "audio", "n_in": 700, "n_rec": 1024,
         "n_out": 20, "max_delay": 30, "samples": 256, "t_min": 50, "t_max": 1000, "rate": 0.01,
         "encoder": "poisson", "mode": "sort", "readout": -1.0},
        # the same net with leaky readout units and unordered delivery, a
        # smaller batch
        {"name": "audio_readout_atomic", "kind": "encoded", "net": "audio", "n_in": 700, "n_rec": 1024,
         "n_out": 20, "max_delay": 30, "samples": 100, "t_min": 50, "t_max": 1000, "rate": 0.01,
         "encoder": "poisson", "mode": "atomic", "readout": 0.9},
        # one e-prop minibatch of the audio net (few samples, long, uneven)
        {"name": "eprop_audio", "kind": "eprop", "net": "audio", "n_in": 700, "n_rec": 1024, "n_out": 20,
         "max_delay": 30, "samples": 32, "t_min": 50, "t_max": 1000, "rate": 0.01, "mode": "sort",
         "update": True},
        # the image net's gradient over one rank's shard (many samples, short)
        {"name": "eprop_ff784", "kind": "eprop", "net": "ff", "n_in": 784, "n_hid": 256, "n_out": 10,
         "fan": 10, "max_delay": 4, "samples": 64, "t_min": 50, "t_max": 50, "rate": 0.1, "mode": "sort",
         "update": False},
        # a small BPTT layer with the bridge's default step count, fp32
        {"name": "core_small", "kind": "core", "n_in": 784, "n_hid": 256, "n_top": 10, "fan": 10,
         "max_delay": 1, "batch": 32, "steps": 20, "ckpt": 10, "rate": 0.25},
        # a two-hidden-layer BPTT core at training size
        {"name": "core_mnist", "kind": "core", "n_in": 784, "n_hid": 512, "n_top": 512, "fan": 85,
         "max_delay": 4, "batch": 128, "steps": 100, "ckpt": 10, "rate": 0.1},
        # one training step of the spiking language model, the whole model
        {"name": "lm_step", "kind": "lm", "hidden": 4096, "fan": 64, "max_delay": 8, "vocab": 96,
         "batch": 64, "steps": 256, "ckpt": 16},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["forward", "forward", "grid", "encoded", "eprop", "core", "core", "lm"])
    if kind == "forward":
        t = _log(rng, 10, 200)
        return {"kind": "forward", "net": "ff", "n_in": rng.randint(100, 900), "n_hid": rng.randint(50, 700),
                "n_out": rng.randint(2, 20), "fan": rng.randint(4, 24), "max_delay": rng.randint(1, 9),
                "samples": _log(rng, 1, 256), "t_min": max(1, t - rng.randint(0, t // 2)), "t_max": t,
                "rate": rng.uniform(0.03, 0.15), "mode": rng.choice(["sort", "sort", "atomic"])}
    if kind == "grid":
        t = _log(rng, 50, 1000)
        return {"kind": "forward", "net": "grid", "width": rng.randint(90, 400),
                "height": rng.randint(90, 250), "degree": rng.randint(20, 100),
                "max_delay": rng.randint(4, 30), "samples": 1 if t > 400 else rng.randint(1, 3),
                "t_min": max(1, t - rng.randint(0, t // 2)), "t_max": t, "rate": rng.uniform(0.01, 0.03),
                "mode": rng.choice(["sort", "bucket"])}
    if kind == "encoded":
        t = _log(rng, 60, 1000)
        return {"kind": "encoded", "net": "audio", "n_in": rng.randint(200, 700),
                "n_rec": rng.randint(150, 1024), "n_out": rng.randint(2, 20),
                "max_delay": rng.randint(3, 30), "samples": _log(rng, 4, 200),
                "t_min": max(1, t // rng.randint(1, 20)), "t_max": t, "rate": rng.uniform(0.005, 0.012),
                "encoder": rng.choice(["poisson", "poisson", "latency"]),
                "mode": rng.choice(["sort", "atomic"]), "readout": rng.choice([-1.0, -1.0, 0.9])}
    if kind == "eprop":
        if rng.random() < 0.5:
            t = _log(rng, 50, 800)
            return {"kind": "eprop", "net": "audio", "n_in": rng.randint(200, 700),
                    "n_rec": rng.randint(150, 1000), "n_out": rng.randint(2, 20),
                    "max_delay": rng.randint(3, 30), "samples": _log(rng, 1, 40),
                    "t_min": max(1, t // rng.randint(1, 10)), "t_max": t,
                    "rate": rng.uniform(0.005, 0.012), "mode": "sort", "update": True}
        t = rng.randint(20, 100)
        return {"kind": "eprop", "net": "ff", "n_in": rng.randint(100, 900), "n_hid": rng.randint(50, 500),
                "n_out": rng.randint(2, 20), "fan": rng.randint(4, 20), "max_delay": rng.randint(1, 5),
                "samples": _log(rng, 4, 128), "t_min": t, "t_max": t, "rate": rng.uniform(0.05, 0.15),
                "mode": rng.choice(["sort", "sort", "atomic"]), "update": False}
    if kind == "core":
        return {"kind": "core", "n_in": rng.randint(64, 800), "n_hid": rng.randint(64, 1024),
                "n_top": rng.randint(10, 700), "fan": rng.randint(5, 90), "max_delay": rng.randint(1, 12),
                "batch": _log(rng, 1, 140), "steps": _log(rng, 10, 100),
                "ckpt": rng.choice([0, 4, 10, 16]), "rate": rng.uniform(0.05, 0.3)}
    return {"kind": "lm", "hidden": _log(rng, 300, 4096), "fan": rng.randint(16, 64),
            "max_delay": rng.randint(1, 10), "vocab": rng.randint(64, 128), "batch": _log(rng, 2, 64),
            "steps": _log(rng, 24, 256), "ckpt": rng.choice([8, 16, 16])}


# ---- inputs ------------------------------------------------------------------

def _grid16(w):
    """Weights on a 2^-16 grid (exact sums in fp32 in any order)."""
    return (np.rint(np.asarray(w, np.float64) * 65536.0) / 65536.0).astype(np.float32)


def _ff_graph(c, seed):
    """Layers of LIF neurons with 1-D local receptive fields."""
    sizes = [c["n_in"], c["n_hid"], c["n_out"]]
    pre, post, d = workloads.layered_local_edges(sizes, c["fan"], seed=seed, max_delay=c["max_delay"])
    rng = np.random.default_rng([seed, 21])
    n = sum(sizes)
    w = _grid16(rng.normal(0.02, 0.1, pre.shape[0]))
    role = np.full(n, INTERNAL, np.uint8)
    role[:sizes[0]] = INPUT
    role[sizes[0] + sizes[1]:] = OUTPUT
    channel = np.full(n, -1, np.int32)
    channel[:sizes[0]] = np.arange(sizes[0])
    channel[sizes[0] + sizes[1]:] = np.arange(sizes[2])
    row_ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(pre, minlength=n), out=row_ptr[1:])
    return SNNGraph(n, row_ptr.astype(np.int32), post.astype(np.int32), w, d.astype(np.int32), role,
                    np.ones(n, np.int8), channel)


def _audio_graph(c, seed):
    """One wiring per size, the weights from the seed at each layer pair's
    scale."""
    g = workloads.audio700_graph(seed=1, n_in=c["n_in"], n_rec=c["n_rec"], n_out=c["n_out"],
                                 max_delay=c["max_delay"])
    scale = np.where(g.pre_ids() < c["n_in"], 0.5, 0.1)
    rng = np.random.default_rng([seed, 25])
    g.weights[:] = _grid16(rng.normal(0.0, 1.0, g.num_synapses) * scale)
    return g


# weight scale of the grid nets: w_std * sqrt(3) / 2^16 is the power of two
# 2^-19, so every generated weight lies on that grid
GRID_W_STD = float(np.float32(65536.0 / math.sqrt(3.0) / 2 ** 19))


def _grid_graph(c, seed):
    spec = workloads.grid_graph_spec(seed=seed, width=c["width"], height=c["height"],
                                     out_degree=c["degree"], long_range=max(1, c["degree"] // 20),
                                     w_std=GRID_W_STD, max_delay=c["max_delay"])
    return runtime.DeviceGraph.generate_grid(spec), int(spec["channel"][spec["role"] == INPUT].max()) + 1


def _steps(c, rng):
    return rng.integers(c["t_min"], c["t_max"] + 1, c["samples"]).astype(np.int32)


def _rates(c, rng, n_ch):
    """Poisson rates of one batch: uniform intensities for image and substrate
    drive, lognormal ones for audio channels."""
    if c["net"] == "audio":
        r = rng.lognormal(math.log(c["rate"]) - 0.5, 1.0, (c["samples"], n_ch))
    elif c["net"] == "ff":
        r = rng.random((c["samples"], n_ch)) * (2 * c["rate"])
    else:
        r = np.full((c["samples"], n_ch), c["rate"])
    return np.minimum(r, 1.0).astype(np.float32)


def _events(c, seed, n_ch):
    rng = np.random.default_rng([seed, 22])
    steps = _steps(c, rng)
    rates = _rates(c, rng, n_ch)
    ev = [workloads.poisson_events(np.random.default_rng([seed, 1000 + i]), rates[i], int(steps[i]), sample_id=i)
          for i in range(c["samples"])]
    return np.concatenate(ev), steps


def _core_net(c, seed):
    sizes = [c["n_in"], c["n_hid"], c["n_top"]]
    pre, post, d = workloads.layered_local_edges(sizes, c["fan"], seed=seed, max_delay=c["max_delay"])
    return sum(sizes), pre, post, d


def _core_tensors(c, seed, n, s):
    """(w, ext, upstream gradient) of a core case on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(1000 + seed)
    w = (torch.rand(s, generator=gen, device="cuda") * 2 - 1) * 0.5
    ext = torch.zeros(c["steps"], c["batch"], n, device="cuda")
    inp = torch.rand(c["steps"], c["batch"], c["n_in"], generator=gen, device="cuda")
    ext[:, :, :c["n_in"]] = (inp < c["rate"]).float()
    g = torch.randn(c["steps"], c["batch"], n, generator=gen, device="cuda") / c["batch"]
    return w, ext, g


def prepare(case, seed):
    c = dict(case)
    st = {"c": c, "lif": workloads.lif_tau20()}
    if c["kind"] in ("forward", "encoded"):
        if c["net"] == "grid":
            st["dg"], n_ch = _grid_graph(c, seed)
        else:
            st["g"] = _ff_graph(c, seed) if c["net"] == "ff" else _audio_graph(c, seed)
            st["dg"] = runtime.DeviceGraph(st["g"])
            n_ch = c["n_in"]
        if c["kind"] == "forward":
            st["events"], st["steps"] = _events(c, seed, n_ch)
        else:
            rng = np.random.default_rng([seed, 23])
            st["steps"] = _steps(c, rng)
            rates = _rates(c, rng, n_ch)
            # latency coding reads intensities, Poisson coding rates
            st["features"] = rates if c["encoder"] == "poisson" else \
                rng.random(rates.shape, dtype=np.float32)
            st["seed"] = seed
    elif c["kind"] == "eprop":
        g = _ff_graph(c, seed) if c["net"] == "ff" else _audio_graph(c, seed)
        cfg = eprop.TrainConfig(lif=st["lif"], lr=5e-4, trace_decay=0.95, mode=MODES[c["mode"]], seed=seed)
        st["session"] = eprop.create(g, cfg, c["samples"], weights=g.weights)
        st["events"], st["steps"] = _events(c, seed, c["n_in"])
        if not c["update"]:
            st["grad"] = torch.empty(g.num_synapses, device="cuda")
        st["labels"] = np.random.default_rng([seed, 24]).integers(0, c["n_out"], c["samples"]).astype(np.int32)
    elif c["kind"] == "core":
        n, pre, post, d = _core_net(c, seed)
        st["core"] = bptt.SpikingCore(n, pre, post, d)
        w, ext, st["grad"] = _core_tensors(c, seed, n, len(pre))
        st["w"], st["ext"] = w.requires_grad_(), ext.requires_grad_()
    else:
        net = workloads.char_lm(seed=seed, vocab=c["vocab"], hidden=c["hidden"], fan_in=c["fan"],
                                sigma=c["hidden"] / 64.0, max_delay=c["max_delay"], B=c["batch"], T=c["steps"])
        torch.manual_seed(seed)
        st["net"] = bptt.SpikingLM(net["vocab"], net["H"], net["pre"], net["post"], net["delays"],
                                   w_scale=2.0, seed=seed, ckpt_every=c["ckpt"]).cuda()
        st["net"].core()
        st["x"] = torch.as_tensor(np.ascontiguousarray(net["x"]), device="cuda")
        st["y"] = torch.as_tensor(np.ascontiguousarray(net["y"]), device="cuda")
    return st


def run(st):
    c = st["c"]
    if c["kind"] == "forward":
        mode = MODES[c["mode"]]
        if c["samples"] == 1 and "g" in st:
            r = runtime.forward(st["g"], st["events"], int(st["steps"][0]), st["lif"],
                                backend="b200-" + c["mode"], device_graph=st["dg"])
            return {"logits": r.logits, "spikes": r.stats.spikes, "events": r.stats.synaptic_events}
        r = runtime.forward_batched(st["dg"], st["events"], st["steps"], st["lif"], mode=mode)
        return {"logits": r["logits"], "spikes": r["spikes"], "events": r["events"]}
    if c["kind"] == "encoded":
        inputs = runtime.DeviceInputs.encode(st["dg"], st["features"], st["steps"], encoder=c["encoder"],
                                             max_rate=1.0, seed=st["seed"])
        job = runtime.Run(st["dg"], inputs, vfinal=True)
        if c["readout"] >= 0:
            job.set_readout(c["readout"])
        job.launch(st["lif"], mode=MODES[c["mode"]])
        r = job.fetch(vfinal=True)
        job.release()
        inputs.release()
        return {"logits": r["logits"], "spikes": r["spikes"], "events": r["events"], "v": r["v"]}
    if c["kind"] == "eprop":
        if not c["update"]:
            r = st["session"].gradient(st["events"], st["steps"], st["labels"], st["grad"])
            return {"counts": r["counts"], "spikes": r["spikes"], "events": r["events"], "grad": st["grad"]}
        r = st["session"].run_batch(st["events"], st["steps"], st["labels"], train=True)
        return {"counts": r["counts"], "spikes": r["spikes"], "events": r["events"],
                "weights": st["session"].get_weights()}
    if c["kind"] == "core":
        s = bptt.spiking_core(st["w"], st["ext"], st["core"], threshold=1.0, decay=0.95, slope=25.0,
                              ckpt_every=c["ckpt"])
        gw, ge = torch.autograd.grad(s, (st["w"], st["ext"]), st["grad"])
        return {"spikes": s.detach(), "grad_w": gw, "grad_ext": ge}
    net = st["net"]
    logits = net(st["x"])
    loss = F.cross_entropy(logits.reshape(-1, c["vocab"]), st["y"].reshape(-1))
    names, params = zip(*net.named_parameters())
    grads = torch.autograd.grad(loss, params)
    return {"logits": logits.detach(), "loss": loss.detach(),
            "grads": {n: g for n, g in zip(names, grads)}}


# ---- what the work cannot do without -----------------------------------------

def _sizes(c):
    """(neurons, synapses, spikes per neuron and step) of a case's net; the
    last from the drive alone, a round figure."""
    if c.get("net") == "grid":
        n = c["width"] * c["height"]
        return n, n * c["degree"], 0.1 * c["rate"]
    if c.get("net") == "audio":
        n = c["n_in"] + c["n_rec"] + c["n_out"]
        return n, int(0.1 * (c["n_in"] + c["n_rec"]) * c["n_rec"]) + c["n_rec"] * c["n_out"], 4 * c["rate"]
    if c["kind"] == "lm":
        return c["hidden"], c["hidden"] * c["fan"], 0.05
    top = c["n_out"] if "n_out" in c else c["n_top"]
    s = c["n_in"] * min(c["fan"], c["n_hid"]) + c["n_hid"] * min(c["fan"], top)
    return c["n_in"] + c["n_hid"] + top, s, c["rate"]


def work(case):
    c = dict(case)
    n, s, rate = _sizes(c)
    if c["kind"] in ("core", "lm"):
        t, b = c["steps"], c["batch"]
        plane = 4.0 * t * b * n
        # drive in, spikes out, spike gradient in, drive gradient out; edges,
        # weights and their gradient once each
        nbytes, flops = 4 * plane + 16.0 * s, 0.0
        # forward adds of active synapses, backward multiply-adds of every
        # synapse, weight-gradient adds of active ones, about 20 per neuron-step
        flops += t * b * (2 * rate * s + 2.0 * s + 20.0 * n)
        if c["kind"] == "lm":
            nbytes = 16.0 * s + 8.0 * t * b + 4.0 * t * b * c["vocab"] + 16.0 * n * c["vocab"]
            flops += 6.0 * t * b * n * c["vocab"]
        return {"bytes": nbytes, "flops": flops}
    steps = c["samples"] * 0.5 * (c["t_min"] + c["t_max"])
    if c["kind"] == "encoded":
        inputs = 4.0 * c["samples"] * c["n_in"]
    else:
        ch = 0.1 * n if c["net"] == "grid" else c["n_in"]
        inputs = 16.0 * steps * ch * c["rate"]
    nbytes = inputs + 12.0 * s + 16.0 * n + 4.0 * c["samples"] * (c.get("n_out", 10) + 4)
    flops = steps * (4.0 * n + rate * s)
    if c["kind"] == "encoded":
        nbytes += 4.0 * c["samples"] * n
    if c["kind"] == "eprop":
        # trace and eligibility of every synapse and step, weights in and out
        nbytes += 8.0 * s
        flops += steps * (2.0 * s + 6.0 * n)
    return {"bytes": nbytes, "flops": flops}


# ---- the same in 64 bits -------------------------------------------------------

def _exact_core(c, seed):
    """The spiking layer and its surrogate gradients in float64, step by step
    over the edge list."""
    n, pre, post, d = _core_net(c, seed)
    w, ext, g = (x.double() for x in _core_tensors(c, seed, n, len(pre)))
    t_n, b = c["steps"], c["batch"]
    pre, post, d = (torch.as_tensor(x, device="cuda") for x in (pre, post, d))
    decay = float(np.float32(0.95))
    zero = torch.zeros(b, n, dtype=torch.float64, device="cuda")
    s_all = torch.zeros(t_n, b, n, dtype=torch.float64, device="cuda")
    vp_all = torch.zeros_like(s_all)
    v = zero
    groups = [(k, (d == k).nonzero()[:, 0]) for k in range(1, int(d.max()) + 1)]
    for t in range(t_n):
        cur = zero.clone()
        for k, e in groups:
            if t - k >= 0:
                cur.index_add_(1, post[e], s_all[t - k][:, pre[e]] * w[e])
        vp = decay * v + cur + ext[t]
        s_all[t] = (vp >= 1.0).double()
        vp_all[t] = vp
        v = vp * (1 - s_all[t])
    grad = torch.zeros_like(s_all)
    gw = torch.zeros_like(w)
    gv = zero
    for t in range(t_n - 1, -1, -1):
        gs = g[t].clone()
        for k, e in groups:
            if t + k < t_n:
                gs.index_add_(1, pre[e], grad[t + k][:, post[e]] * w[e])
        gs -= gv * vp_all[t]
        grad[t] = gv * (1 - s_all[t]) + gs / (1 + 25.0 * (vp_all[t] - 1.0).abs()) ** 2
        gv = decay * grad[t]
        for k, e in groups:
            if t - k >= 0:
                gw[e] += (s_all[t - k][:, pre[e]] * grad[t][:, post[e]]).sum(0)
    return {"spikes": s_all, "grad_w": gw, "grad_ext": grad}


def _exact_ff(c, seed):
    """Spike counts of the output channels of a small net in float64."""
    g = _ff_graph(c, seed)
    ev, steps = _events(c, seed, c["n_in"])
    t_n, b, n = int(steps.max()), c["samples"], g.num_neurons
    ext = torch.zeros(t_n, b, n, dtype=torch.float64, device="cuda")
    ext[torch.as_tensor(ev["time"].astype(np.int64)), torch.as_tensor(ev["sample_id"].astype(np.int64)),
        torch.as_tensor(ev["channel_id"].astype(np.int64))] = 1.0
    live = torch.as_tensor(steps, device="cuda")
    pre = torch.as_tensor(np.repeat(np.arange(n), np.diff(g.row_ptr)), device="cuda")
    post = torch.as_tensor(g.post_ids.astype(np.int64), device="cuda")
    w = torch.as_tensor(g.weights, device="cuda").double()
    d = torch.as_tensor(g.delays, device="cuda")
    groups = [(k, (d == k).nonzero()[:, 0]) for k in range(1, int(d.max()) + 1)]
    lif = workloads.lif_tau20()
    v = torch.zeros(b, n, dtype=torch.float64, device="cuda")
    s_all = torch.zeros(t_n, b, n, dtype=torch.float64, device="cuda")
    for t in range(t_n):
        cur = torch.zeros_like(v)
        for k, e in groups:
            if t - k >= 0:
                cur.index_add_(1, post[e], s_all[t - k][:, pre[e]] * w[e])
        v = v * lif.decay + ext[t] + cur
        s = ((v >= lif.threshold) & (t < live)[:, None]).double()
        s_all[t] = s
        v = v - s * lif.threshold
    return s_all[:, :, n - c["n_out"]:].sum(0)


def exact(case, seed):
    """None for the nets whose spike trains depend on every rounding over
    hundreds of steps, and for the whole model."""
    c = dict(case)
    if c["kind"] == "core":
        return _exact_core(c, seed)
    if c["kind"] == "forward" and c["net"] == "ff":
        logits = _exact_ff(c, seed)
        one = c["samples"] == 1
        return {"logits": logits[0] if one else logits, "spikes": None, "events": None}
    return None
