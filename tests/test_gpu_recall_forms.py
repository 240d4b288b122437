"""The batched readout outside the bit planes (facilitation, boosts of 256 and more, the tensor
contraction): every trajectory equals the plain path."""
import ctypes as C

import numpy as np
import pytest

import axon_b200 as ax
import axon_b200._capi as A

pytestmark = pytest.mark.gpu


def trained(seed=0, nstim=6, epochs=3, **kw):
    base = dict(ax.CONFIG_C, ncol=256, incols=64, target=16, k=12)
    base.update(kw)
    net = ax.Network(base)
    net.init(seed)
    pats = ax.stimuli(seed, nstim, base["incols"], max(4, base["incols"] // 4))
    for _ in range(epochs):
        for p in range(nstim):
            net.present(ax.load_stim(pats[p], 1.0, 1000 + p, net.ncol), 10, 5, True)
    return net, pats


def cues_of(net, pats, B):
    keep = (1.0, 0.75, 0.5, 0.35, 0.25, 0.1, 0.0)
    return np.stack([ax.load_stim(pats[b % len(pats)], keep[b % len(keep)], 4400 + b, net.ncol) for b in range(B)])


def same(net, cues, T, clamp, **kw):
    a = net.recall(cues, T, clamp, hist=True, stats=True, **kw)
    plain = {k: v for k, v in kw.items() if k in ("use_bias", "ref_ball")}
    b = net.recall(cues, T, clamp, hist=True, stats=True, method="plain", **plain)
    a["stats"][:, 2] = b["stats"][:, 2] = 0  # branch coincidence: plain method only
    for k in ("final", "hist", "stats"):
        assert np.array_equal(a[k], b[k]), k
    if a["drive_log"] is not None:
        assert np.array_equal(a["drive_log"], b["drive_log"])


# trajectories split over several groups of warps (one CTA per SM, 148 on a B200: batches just above a multiple
# of it, and 512), whose thresholds fall below the recorded drives after the clamp
@pytest.mark.parametrize("B", [3, 149, 300, 512])
def test_split_trajectories(B):
    net, pats = trained()
    cues = cues_of(net, pats, B)
    for slab in ("floor", "floor_always") * 3:
        same(net, cues, 16, 4, contraction="tensor", slab=slab)
    net.close()


# every output of axon_recall is optional: reference assemblies without a log to write are accepted, and ignored
@pytest.mark.parametrize("kw", [dict(), dict(boost=300), dict(facil=7), dict(boost=2000)])
@pytest.mark.parametrize("contraction", [0, 1])
def test_assemblies_without_a_log(kw, contraction):
    net, pats = trained(**kw)
    cues = cues_of(net, pats, 5)
    want = net.recall(cues, 12, 4, method="plain")["final"]
    got, ref = np.zeros_like(cues), np.full_like(cues, 0xFFFFFFFF)
    for method in (0, 1):
        a = A.RecallArgs(T=12, clamp_steps=4, method=method, contraction=contraction)
        A.check(A.lib().axon_recall(net._h, A.u32(cues), 5, C.byref(a), A.u32(ref), A.u32(got), None, None, None, None))
        assert np.array_equal(got, want)
    net.close()


# from boost 256 on a neuron's drive can pass 2^14 and the 16-bit counters take over (up to 1,791), their default
# contraction included: one and two counter buffers (400 trajectories leave room for one), several trajectories per
# CTA, the clamped steps' cache (whole and cut groups), every slab policy, biases, and the member-drive log
@pytest.mark.parametrize("kw", [dict(boost=255), dict(boost=256), dict(boost=1700), dict(boost=300, dthr=9, incols=20)])
@pytest.mark.parametrize("B", [9, 149, 400])
def test_sixteen_bit_counters(kw, B):
    net, pats = trained(**kw)
    cues = cues_of(net, pats, B)
    for slab in ("floor", "floor_always", "full"):
        same(net, cues, 12, 5, slab=slab)
    same(net, cues, 12, 5, use_bias=1)
    rng = np.random.default_rng(B)
    net.write("MULT", rng.integers(0, 3, net.ncol * 32).astype(np.uint32))
    same(net, cues, 9, 1, ref_ball=rng.integers(0, 1 << 32, cues.shape, dtype=np.uint64).astype(np.uint32))
    net.close()


def test_sixteen_bit_counters_at_the_widest_network():
    net, pats = trained(ncol=8192, incols=512, target=64, k=24, epochs=1, boost=600)
    same(net, cues_of(net, pats, 160), 12, 4)
    net.close()


# the server's kernels for these drives: few trajectories of a network in a tick, many, and more than two counter
# buffers hold (366)
@pytest.mark.parametrize("boost", [256, 1700])
@pytest.mark.parametrize("requests", [12, 150, 420])
def test_server_with_sixteen_bit_counters(boost, requests):
    nets, pats = zip(*(trained(seed, boost=boost) for seed in range(2)))
    rng = np.random.default_rng(requests)
    reqs = []
    for tag in range(requests):
        i = int(rng.random() < (0.5 if requests < 400 else 0.05))
        pat = pats[i][tag % len(pats[i])]
        reqs.append((i, np.sort(rng.choice(pat, int(rng.integers(2, len(pat) + 1)), replace=False)).astype(np.uint32), 3 + tag % 9))
    with ax.Server(list(nets), 128 << 20) as srv:
        at = ax.clock_s() + 0.02  # all together
        for tag, (i, cols, free) in enumerate(reqs):
            srv.submit(i, cols, 4, free, tag, at)
        srv.wait_idle(120)
        got = {res["tag"]: spikes for res, spikes in srv.poll(requests)}
        assert srv.stats()["max_batch"] == requests
    for free in range(3, 12):
        for i, n in enumerate(nets):
            tags = [t for t, (j, _, f) in enumerate(reqs) if j == i and f == free]
            if tags:
                want = n.recall(np.stack([ax.clamp_words(reqs[t][1], n.ncol) for t in tags]), 4 + free, 4, method="plain")["final"]
                for t, w in zip(tags, want):
                    assert np.array_equal(got[t], w), t
    for n in nets:
        n.close()
