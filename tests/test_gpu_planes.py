"""The bit-plane batched readout (lane = trajectory) against the plain path, at the edges of
its cases: every form of spike-word record, both ways of reading the tiles, the lane split of
small batches, more candidates and gated columns than a group's memory holds."""
import numpy as np
import pytest

import axon_b200 as ax

pytestmark = pytest.mark.gpu


def trained(seed=0, nstim=6, epochs=3, **kw):
    base = dict(ax.CONFIG_C, ncol=256, incols=64, target=16, k=12)
    base.update(kw)
    net = ax.Network(base)
    net.init(seed)
    stimcols = max(4, base["incols"] // 4)
    pats = ax.stimuli(seed, nstim, base["incols"], stimcols)
    for _ in range(epochs):
        for p in range(nstim):
            net.present(ax.load_stim(pats[p], 1.0, 1000 + p, net.ncol), 10, 5, True)
    return net, pats


def cues_of(net, pats, B, seed):
    """Whole columns, dropped columns and single flipped bits: words of 1 to 32 set bits."""
    rng = np.random.default_rng(seed)
    out = []
    for b in range(B):
        w = ax.clamp_words(pats[b % len(pats)], net.ncol)
        keep = (1.0, 0.95, 0.7, 0.5, 0.3, 0.05)[b % 6]
        if keep < 1.0:
            bits = rng.random((net.ncol, 32)) < keep
            w &= (bits.astype(np.uint64) << np.arange(32, dtype=np.uint64)).sum(1).astype(np.uint32)
        out.append(w)
    return np.stack(out)


def same(net, cues, T, clamp, **kw):
    a = net.recall(cues, T, clamp, hist=True, stats=True, **kw)
    b = net.recall(cues, T, clamp, hist=True, stats=True, method="plain", **kw)
    a["stats"][:, 2] = b["stats"][:, 2] = 0  # branch coincidence: plain method only
    for k in ("final", "hist", "stats"):
        assert np.array_equal(a[k], b[k]), k
    if a["drive_log"] is not None:
        assert np.array_equal(a["drive_log"], b["drive_log"])


# winners per column: sums of the held or of the left-out neurons, of at most 8, 12 or 16 masks
@pytest.mark.parametrize("k", [0, 1, 8, 12, 13, 16, 17, 19, 20, 23, 24, 31, 32, 40])
def test_record_forms(k):
    net, pats = trained(k=k)
    same(net, cues_of(net, pats, 12, k), 16, 4)
    net.close()


@pytest.mark.parametrize("kw", [dict(dthr=3), dict(dthr=40), dict(dthr=600), dict(mode=0), dict(mode=2, dthr=2), dict(boost=255),
                                dict(boost=77), dict(incols=20), dict(target=1), dict(target=250), dict(target=0),
                                dict(target=0, topkpar=0)])
@pytest.mark.parametrize("B", [9, 130])
def test_dendrites_and_thresholds(kw, B):
    net, pats = trained(**kw)
    same(net, cues_of(net, pats, B, B), 14, 3)
    same(net, cues_of(net, pats, B, B + 1), 14, 3, use_bias=1, slab="full")
    net.close()


# both sides of each line of the launch shape: lanes per trajectory, tiles through L2 or staged, one or more launches
@pytest.mark.parametrize("B", [1, 10, 11, 20, 21, 32, 33, 96, 97, 160, 161, 296, 300, 512, 513])
def test_batch_sizes(B):
    net, pats = trained(ncol=608, incols=72, target=24, k=24)
    same(net, cues_of(net, pats, B, B), 9, 3)
    net.close()


def test_wide_networks_with_logs():
    """Several columns per slot and CTA at odd widths, more gated columns than the list holds
    (target near ncol), and the drive log."""
    rng = np.random.default_rng(5)
    for ncol, B, kw in ((2080, 110, {}), (1984, 20, dict(target=1500)), (2208, 100, dict(target=1900)), (8192, 100, {})):
        net, pats = trained(**dict(dict(ncol=ncol, incols=256, target=32, k=24, nstim=4, epochs=1), **kw))
        net.write("MULT", rng.integers(0, 3, ncol * 32).astype(np.uint32))
        ref = rng.integers(0, 1 << 32, (B, ncol), dtype=np.uint64).astype(np.uint32)
        for slab in ("floor", "floor_always", "full"):
            same(net, cues_of(net, pats, B, 3), 9, 3, ref_ball=ref if slab == "floor" else None, slab=slab)
        net.close()


# the input groups' share of the drives, kept over the clamped steps: none, one, all but the last, all
@pytest.mark.parametrize("clamp", [0, 1, 2, 7, 8, 9])
@pytest.mark.parametrize("B", [13, 161, 300])
def test_clamped_steps(clamp, B):
    net, pats = trained(incols=72)
    same(net, cues_of(net, pats, B, clamp), 8, clamp)
    net.close()


# a server whose trajectories end at different steps moves the others to lower lanes: whole blocks of
# staged and of directly read launches, small batches, and columns recomputed in the step of the move
@pytest.mark.parametrize("kw,unit", [(dict(), 1), (dict(target=250), 1), (dict(incols=20, k=0), 1), (dict(), 12)])
def test_server_moves_lanes(kw, unit):
    net, pats = trained(**kw)
    other, _ = trained(seed=1, **kw)
    rng = np.random.default_rng(3)
    reqs = []
    for tag in range(450):
        cols = np.sort(rng.choice(pats[tag % len(pats)], int(rng.integers(1, len(pats[0]) + 1)), replace=False)).astype(np.uint32)
        reqs.append((int(tag % 9 == 0), cols, unit * int(rng.integers(1, 1 + 36 // unit))))
    with ax.Server([net, other], 64 << 20) as srv:
        at = ax.clock_s() + 0.02  # all together
        for tag, (i, cols, free) in enumerate(reqs):
            srv.submit(i, cols, 4, free, tag, at)
        srv.wait_idle(120)
        got = {res["tag"]: spikes for res, spikes in srv.poll(len(reqs))}
    for free in sorted({f for _, _, f in reqs}):
        for i, n in enumerate((net, other)):
            tags = [t for t, (j, _, f) in enumerate(reqs) if j == i and f == free]
            if tags:
                cues = np.stack([ax.clamp_words(reqs[t][1], n.ncol) for t in tags])
                want = n.recall(cues, 4 + free, 4, method="plain")["final"]
                for t, w in zip(tags, want):
                    assert np.array_equal(got[t], w), t
    net.close()
    other.close()


# both sides of the width up to which every column with a drive is a candidate, and sorted tasks with
# several lanes per trajectory (two columns per CTA)
@pytest.mark.parametrize("ncol,target", [(256, 8), (512, 24), (544, 24), (544, 460)])
@pytest.mark.parametrize("B", [40, 96])
def test_small_networks(ncol, target, B):
    net, pats = trained(ncol=ncol, incols=64, target=target, k=24, nstim=12, epochs=2)
    same(net, cues_of(net, pats, B, B), 12, 3, use_bias=1)
    same(net, cues_of(net, pats, B, B + 1), 12, 3, slab="floor_always")
    net.close()


# the widths next to the line up to which every column with a drive is a candidate
@pytest.mark.parametrize("ncol", [576, 608])
@pytest.mark.parametrize("B", [5, 40, 200])
def test_widths_about_the_candidate_line(ncol, B):
    net, pats = trained(ncol=ncol, incols=72, target=9, k=24, nstim=12, epochs=2)
    for bias in (0, 1):
        same(net, cues_of(net, pats, B, B + bias), 12, 3, use_bias=bias)
    net.close()


# more candidates than a group keeps in shared memory (1,024), whose planes are stored: with biases every column
# that passes a low floor; and every column's planes kept beside the candidates
@pytest.mark.parametrize("ncol", [1056, 2080])
def test_more_candidates_than_a_group_holds(ncol):
    net, pats = trained(ncol=ncol, incols=128, target=32, k=24, epochs=2)
    for B in (20, 170):
        for slab in ("floor", "floor_always", "full"):
            for bias in (0, 1):
                same(net, cues_of(net, pats, B, B), 12, 3, slab=slab, use_bias=bias)
    net.close()


# both sides of the lines between this kernel and the former one: winners per column, share of winning columns,
# number of trajectories, width, biases and logs
@pytest.mark.parametrize("kw", [dict(k=6), dict(k=10), dict(k=16), dict(k=22), dict(target=40), dict(target=150), dict(target=0),
                                dict(mode=2, dthr=2), dict(boost=200)])
@pytest.mark.parametrize("ncol", [512, 608, 2080])
def test_lines_between_the_kernels(kw, ncol):
    net, pats = trained(**dict(dict(ncol=ncol, incols=64, target=8, k=24, epochs=1), **kw))
    rng = np.random.default_rng(ncol)
    for B in (20, 21, 48, 49, 97, 129):
        cues = cues_of(net, pats, B, B)
        same(net, cues, 9, 3)
        same(net, cues, 9, 3, use_bias=1)
        same(net, cues, 9, 3, ref_ball=rng.integers(0, 1 << 32, cues.shape, dtype=np.uint64).astype(np.uint32))
    with ax.Server([net], 64 << 20) as srv:
        for tag in range(30):
            srv.submit(0, np.sort(pats[tag % 6][: 4 + tag % 9]).astype(np.uint32), 3, 4 + tag % 3, tag)
        srv.wait_idle(60)
        for res, spikes in srv.poll(30):
            t = res["tag"]
            cue = ax.clamp_words(np.sort(pats[t % 6][: 4 + t % 9]), ncol)[None]
            assert np.array_equal(spikes, net.recall(cue, 7 + t % 3, 3, method="plain")["final"][0]), t
    net.close()


# the same above the width up to which every column is a candidate: a threshold below the floor in the step of the
# move recomputes columns from the old lanes' activity words
@pytest.mark.parametrize("target", [24, 150])
def test_server_moves_lanes_of_wider_networks(target):
    test_server_moves_lanes(dict(ncol=608, incols=72, target=target), 1)


# more gated columns than the list holds, over the forms that keep this kernel for them
@pytest.mark.parametrize("ncol,target,B,bias", [(2208, 1900, 130, 0), (2208, 600, 20, 1), (512, 440, 130, 0), (512, 440, 9, 1)])
def test_more_gated_columns_than_the_list_holds(ncol, target, B, bias):
    net, pats = trained(ncol=ncol, incols=64, target=target, k=24, epochs=1)
    for slab in ("floor", "floor_always", "full"):
        same(net, cues_of(net, pats, B, B), 9, 3, slab=slab, use_bias=bias)
    net.close()
