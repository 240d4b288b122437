"""Performance cases of the engine: what a program that uses it has it do, over the range of
sizes it meets.

A case names one of six kinds of call and its sizes:

- ``present``: one readout presentation through ``Network.present`` and its final spikes.
- ``static``: presentations through ``axon_present_static`` on buffers that the caller owns
  (device tensors): a readout, or with ``learn`` one training epoch over the stored patterns.
- ``recall``: a batch of readout trajectories from host cues to host results.
- ``recall_device``: the same with cues and results in device memory.
- ``multi``: ``multi_train``, the whole experiment for several networks in one launch.
- ``serve``: a burst of recall requests answered by a ``Server``.

Networks are trained in ``prepare`` (patterns, weights and cues follow from the seed), so that
readouts run on weights and spike vectors with the statistics of a trained network. The
geometry is the default configuration's (4,096 columns of 32 neurons, 512 of them inputs, 64
active columns) or smaller ones with the same proportions, as the tests use.
"""
import ctypes as C

import numpy as np
import torch

import axon_b200 as ax
from axon_b200 import _capi as A

FIELDS = {"w0": "W0", "w1": "W1", "w2": "W2", "w3": "W3", "conn": "CONN", "bias": "BIAS", "mult": "MULT",
          "refball": "REFBALL", "stim": "STIM", "spk_a": "SPK_A", "spk_b": "SPK_B", "drive": "DRIVE",
          "bbits": "BBITS", "acc": "ACC", "marg": "MARG", "drive_log": "DRIVELOG", "stats": "STATS", "hist": "HIST",
          "theta": "THETA"}


def listed():
    return [
        # one query of a trained network, the smallest call at the default geometry: a 10-step
        # readout of a 75 % cue, as the experiments run for every cue
        dict(name="present_query", kind="present", ncol=4096, load=60, epochs=20, T=10, clamp=5, keep=0.75),
        # the wave readout (35 steps) on caller-owned buffers, at a width that is no power of two
        dict(name="static_wave_2080", kind="static", ncol=2080, load=24, epochs=20, T=35, clamp=5, keep=1.0, learn=False),
        # one training epoch of 12 patterns at the default geometry: the reference's own headline loop
        dict(name="train_epoch", kind="static", ncol=4096, load=12, epochs=3, T=10, clamp=5, keep=1.0, learn=True),
        # one training epoch of a small network: launches and latency
        dict(name="train_small", kind="static", ncol=256, load=5, epochs=3, T=10, clamp=5, keep=1.0, learn=True),
        # a single cue through the batched readout, host to host
        dict(name="recall_1", kind="recall", ncol=4096, load=24, epochs=20, B=1, T=10, clamp=5, keep=0.75, bias=0, records=False),
        # an odd small batch, as an application gathers a few queries
        dict(name="recall_13", kind="recall", ncol=4096, load=24, epochs=20, B=13, T=15, clamp=5, keep=0.75, bias=0, records=False),
        # the completion measurements of one network: every pattern, with every step's spikes, counters
        # and the drive log of the assemblies' members
        dict(name="recall_60_records", kind="recall", ncol=4096, load=60, epochs=20, B=60, T=30, clamp=5, keep=0.75, bias=0, records=True),
        # the benchmark's batch: 300 noisy cues, 10 clamped and 35 free steps, in device memory
        dict(name="recall_300_device", kind="recall_device", ncol=4096, load=60, epochs=20, B=300, T=45, clamp=10, keep=1.0, bias=0),
        # more trajectories than one launch holds, of a long readout, host to host
        dict(name="recall_700", kind="recall", ncol=4096, load=60, epochs=20, B=700, T=35, clamp=5, keep=0.75, bias=0, records=False),
        # training and measuring several networks at once
        dict(name="multi_3", kind="multi", ncol=4096, loads="24 36 60", epochs=10),
        # a light burst of requests on a few networks: tick latency
        dict(name="serve_16", kind="serve", ncol=4096, loads="12 24", epochs=20, requests=16),
        # a saturating burst on several networks: throughput
        dict(name="serve_1200", kind="serve", ncol=4096, loads="12 24 36 60", epochs=10, requests=1200),
    ]


def _log(rng, lo, hi):
    """A whole number of [lo, hi], spread evenly over its logarithm."""
    return min(hi, max(lo, int(round(lo * (hi / lo) ** rng.random()))))


def draw(rng):
    kind = rng.choice(["present", "static", "static", "recall", "recall", "recall_device", "multi", "serve"])
    ncol = 4096 if rng.random() < 0.6 else 32 * _log(rng, 8, 128)
    load = _log(rng, 3, 60)
    T = _log(rng, 5, 50)
    clamp = rng.randint(1, min(T, 10))
    keep = rng.choice([1.0, 0.9, 0.75, 0.5])
    if kind == "present":
        return dict(kind=kind, ncol=ncol, load=load, epochs=10, T=T, clamp=clamp, keep=keep)
    if kind == "static":
        learn = rng.random() < 0.6
        return dict(kind=kind, ncol=ncol, load=_log(rng, 3, 30), epochs=3, T=10 if learn else T, clamp=5 if learn else clamp,
                    keep=1.0 if learn else keep, learn=learn)
    if kind == "recall":
        return dict(kind=kind, ncol=ncol, load=load, epochs=10, B=_log(rng, 1, 600), T=min(T, 35), clamp=min(clamp, 5), keep=keep,
                    bias=int(rng.random() < 0.15), records=rng.random() < 0.25)
    if kind == "recall_device":
        return dict(kind=kind, ncol=ncol, load=load, epochs=10, B=_log(rng, 1, 512), T=T, clamp=clamp, keep=keep, bias=0)
    if kind == "multi":
        return dict(kind=kind, ncol=ncol, loads=" ".join(str(_log(rng, 3, 30)) for _ in range(rng.randint(1, 4))), epochs=rng.randint(2, 8))
    return dict(kind=kind, ncol=ncol, loads=" ".join(str(_log(rng, 3, 30)) for _ in range(rng.randint(1, 4))), epochs=10,
                requests=_log(rng, 1, 800))


def _geometry(ncol):
    """The configuration of a network of ncol columns and the columns per stored pattern."""
    incols = max(32, ncol // 8 // 8 * 8)
    cfg = dict(ax.CONFIG_C, ncol=ncol, incols=incols, target=max(8, ncol // 64))
    return cfg, max(4, incols // 8)


def _loads(case):
    return [int(x) for x in case["loads"].split()] if "loads" in case else [case["load"]]


def _patterns(rng, load, incols, stimcols):
    return np.stack([rng.permutation(incols)[:stimcols] for _ in range(load)]).astype(np.uint32)


def _train(net, pats, epochs, seed):
    net.init(seed & 0x7FFFFFFF)
    stims = [ax.clamp_words(p, net.ncol) for p in pats]
    for _ in range(epochs):
        for s in stims:
            net.present(s, 10, 5, True)


def _cue(rng, pat, keep, ncol):
    """The clamp words of a pattern of which a share `keep` of the active bits is left."""
    words = ax.clamp_words(pat, ncol)
    if keep < 1.0:
        bits = rng.random((len(pat), 32)) < keep
        words[pat] = (bits.astype(np.uint64) << np.arange(32, dtype=np.uint64)).sum(1).astype(np.uint32)
    return words


def _assembly(net, pat):
    """The spikes of a pattern's clamped readout, the reference its recall is measured against."""
    net.present(ax.clamp_words(pat, net.ncol), 10, 10, False)
    return net.final_spikes(10)


def _pinned(words):
    return torch.empty(words, dtype=torch.int32, pin_memory=True)


def prepare(case, seed):
    rng = np.random.default_rng(seed)
    kind, ncol = case["kind"], case["ncol"]
    kw, stimcols = _geometry(ncol)
    cfg = ax.config(**kw)
    state = dict(case=case, cfg=cfg)
    if kind == "multi":  # the networks, and page-locked memory for the trained state
        loads = _loads(case)
        nets = [ax.Network(cfg) for _ in loads]
        state.update(nets=nets, seeds=[(seed + i) & 0x7FFFFFFF for i in range(len(loads))], loads=loads, stimcols=stimcols,
                     host=[{b: _pinned(n.words(b)) for b in ("W0", "W1", "W2", "W3", "BIAS")} for n in nets])
        return state
    nets, pats = [], []
    for i, load in enumerate(_loads(case)):
        pats.append(_patterns(rng, load, cfg.incols, stimcols))
        nets.append(ax.Network(cfg))
        _train(nets[i], pats[i], case["epochs"], seed + i)
    state.update(nets=nets)
    if kind == "serve":  # cues of a quarter to all of a pattern's columns, then 10-60 free steps
        reqs = []
        for tag in range(case["requests"]):
            n = int(rng.integers(len(nets)))
            pat = pats[n][int(rng.integers(len(pats[n])))]
            cols = np.sort(rng.choice(pat, int(rng.integers(max(1, stimcols // 4), stimcols + 1)), replace=False)).astype(np.uint32)
            reqs.append((n, cols, int(rng.integers(10, 61)), tag))
        state.update(reqs=reqs, server=ax.Server(nets, 1 << 30))
        return state
    net, pats = nets[0], pats[0]
    if kind == "present":
        state.update(stim=_cue(rng, pats[0], case["keep"], ncol))
    elif kind == "static":
        bufs = {f: torch.from_numpy(net.read(b).view(np.int32)).cuda() for f, b in FIELDS.items()}
        cues = pats if case["learn"] else pats[:1]
        stims = torch.from_numpy(np.stack([_cue(rng, p, case["keep"], ncol) for p in cues]).view(np.int32)).cuda()
        net.close()
        structs = []
        for i in range(len(cues)):
            ptr = {f: bufs[f].data_ptr() for f in FIELDS}
            ptr["stim"] = stims[i].data_ptr()
            structs.append(A.StateDev(**{f: C.c_void_p(p) for f, p in ptr.items()}))
        state.update(nets=[], bufs=bufs, stims=stims, structs=structs)
    else:
        cues = np.stack([_cue(rng, pats[b % len(pats)], case["keep"] if b % 5 else 1.0, ncol) for b in range(case["B"])])
        if kind == "recall":
            ref = None
            if case["records"]:  # the assembly of each cue's pattern
                refs = [_assembly(net, p) for p in pats]
                ref = np.stack([refs[b % len(pats)] for b in range(case["B"])])
            state.update(cues=cues, ref=ref)
        else:
            state.update(d_cues=torch.from_numpy(cues.view(np.int32)).cuda(),
                         d_final=torch.zeros((case["B"], ncol), dtype=torch.int32, device="cuda"))
    torch.cuda.synchronize()
    return state


def run(state):
    case, kind = state["case"], state["case"]["kind"]
    if kind == "present":
        net = state["nets"][0]
        net.present(state["stim"], case["T"], case["clamp"], False, True, 0)
        return {"spikes": net.final_spikes(case["T"]).view(np.int32)}
    if kind == "static":
        lib, cfg = A.lib(), C.byref(state["cfg"])
        learn = int(case["learn"])
        for st in state["structs"]:
            A.check(lib.axon_present_static(cfg, C.byref(st), case["T"], case["clamp"], learn, 2 if learn else 0))
        return {f: t for f, t in state["bufs"].items() if f not in ("conn", "mult", "refball", "stim")}
    if kind == "recall":
        out = state["nets"][0].recall(state["cues"], case["T"], case["clamp"], use_bias=case["bias"], hist=case["records"],
                                      stats=case["records"], ref_ball=state["ref"])
        return {k: v.view(np.int32) for k, v in out.items() if isinstance(v, np.ndarray)}
    if kind == "recall_device":
        state["nets"][0].recall_device(state["d_cues"].data_ptr(), case["B"], case["T"], case["clamp"],
                                       state["d_final"].data_ptr(), use_bias=case["bias"], graph=True)
        return {"final": state["d_final"]}
    if kind == "multi":
        res, _ = ax.multi_train(state["nets"], state["seeds"], state["loads"], epochs=case["epochs"], stimcols=state["stimcols"])
        for net, host in zip(state["nets"], state["host"]):
            for b, t in host.items():
                A.check(A.lib().axon_read(net._h, A.BUF[b], C.cast(t.data_ptr(), A.U32P), t.numel()))
        return {"results": res, "nets": state["host"]}
    srv, n = state["server"], len(state["reqs"])
    for net, cols, free, tag in state["reqs"]:
        srv.submit(net, cols, 5, free, tag)
    srv.wait_idle(60)
    spikes = np.empty((n, state["cfg"].ncol), dtype=np.int32)
    for res, spk in srv.poll(n):
        spikes[res["tag"]] = spk.view(np.int32)
    return {"spikes": spikes}


def exact(case, seed):
    """Spikes, counters, drives and weights are whole numbers, which have to stay equal bit for
    bit. The only floating outputs are the overlaps and percentages of ``multi``, ratios of
    counts over a whole training run, which plain torch would take minutes for."""
    return None


def work(case):
    """Bytes: each W3 tile (1 KiB per column and branch) that any trajectory's active groups
    touch read once, the four planes of the tiles that learning changes read and written once,
    cues in and spikes out. Operations: an AND and a population count per 32-bit weight word
    that meets a nonzero spike word, for every step, plus those of the bit-serial updates."""
    ncol = case["ncol"]
    kw, stimcols = _geometry(ncol)
    incols, target, inbr = kw["incols"], kw["target"], kw["inbr"]
    grec, gin = (ncol - incols) / 8, incols / 8
    frec, fin = 1 - (1 - 1 / grec) ** target, 1 - (1 - 1 / gin) ** stimcols  # share of groups that spike

    def tiles(B):  # tiles that B different spike vectors touch
        return ncol * ((32 - inbr) * (1 - (1 - frec) ** B) + inbr * (1 - (1 - fin) ** B))

    def step_ops(clamped):  # of one trajectory's step
        return 64.0 * ncol * ((32 - inbr) * target / grec + (inbr * stimcols / gin if clamped else 0.0))

    def readout(B, T, clamp):
        return {"bytes": 1024.0 * tiles(B) + 8.0 * B * ncol, "flops": B * (clamp * step_ops(True) + (T - clamp) * step_ops(False))}

    voted = (32 - inbr) * frec + inbr * fin  # branches of a column that learn

    def epoch(load):  # one training epoch: 10-step presentations, the assemblies' branches updated
        learn = load * (target + stimcols) * voted
        return {"bytes": 1024.0 * tiles(load) + 7168.0 * min(learn, ncol * 32), "flops": load * (5 * step_ops(True) + 5 * step_ops(False)) + learn * 8 * 256 * 20.0}

    kind = case["kind"]
    if kind == "present" or (kind == "static" and not case["learn"]):
        return readout(1, case["T"], case["clamp"])
    if kind == "static":
        return epoch(case["load"])
    if kind in ("recall", "recall_device"):
        w = readout(case["B"], case["T"], case["clamp"])
        if case.get("records"):
            w["bytes"] += case["B"] * (4.0 * ncol * (case["T"] + 1) + 4096 + 1024)
        return w
    total = {"bytes": 0.0, "flops": 0.0}
    loads = _loads(case)
    for load in loads:
        if kind == "multi":
            e, r = epoch(load), readout(2 * load + 24, 15, 5)
            w = {"bytes": e["bytes"] + r["bytes"] + 4 * ncol * 32768.0, "flops": case["epochs"] * e["flops"] + r["flops"]}
        else:
            w = readout(case["requests"] / len(loads), 40, 5)
        total = {k: total[k] + w[k] for k in total}
    return total
