"""Near the limit of the device's memory a batched recall and a server take the form that needs
less: the bit planes' layout is 162 MiB for 4,096 columns, the older one's 128."""
import gc

import numpy as np
import pytest

import axon_b200 as ax

pytestmark = pytest.mark.gpu

MIB = 1 << 20
CFG = dict(ax.CONFIG_C, ncol=4096, incols=512, target=64)


@pytest.fixture
def leave():
    """Fills the device's memory up to `mib` MiB, until the test ends."""
    import torch

    held = []

    def fill(mib):
        torch.cuda.synchronize()
        free = torch.cuda.mem_get_info()[0]
        if free < (mib + 2) * MIB:
            pytest.skip("another program holds the device's memory")
        held.append(torch.empty(free - mib * MIB, dtype=torch.uint8, device="cuda"))

    yield fill
    held.clear()
    gc.collect()
    torch.cuda.empty_cache()


def network(**kw):
    net = ax.Network(dict(CFG, **kw))
    net.init(3)
    pats = ax.stimuli(3, 4, net.cfg.incols, 32)
    for p in pats:
        net.present(ax.clamp_words(p, net.ncol), 10, 5, True)
    return net, pats


def cues_of(net, pats, B):
    return np.stack([ax.load_stim(pats[b % 4], 0.7, b, net.ncol) for b in range(B)])


def warm():
    """The kernels of both forms are loaded while there is room (with 16-bit counters: boost 300)."""
    for kw in (dict(), dict(boost=300)):
        net, pats = network(ncol=256, incols=64, target=8, **kw)
        net.recall(cues_of(net, pats[:, :8] % 64, 3), 6, 2)
        with ax.Server([net], 16 * MIB) as srv:
            for tag in range(30):
                srv.submit(0, np.sort(pats[0][:8]), 2, 3, tag)
            srv.wait_idle(30)
        net.close()


# room for the bit planes' layout but not for its 22 MiB of scratch, and not even for the layout
@pytest.mark.parametrize("mib", [176, 158])
def test_recall(leave, mib):
    warm()
    net, pats = network()
    cues = cues_of(net, pats, 64)
    want = net.recall(cues, 8, 1, method="plain")["final"]
    leave(mib)
    for _ in range(2):
        assert np.array_equal(net.recall(cues, 8, 1)["final"], want)
    net.close()


# two networks: the layout of one alone fits, and both do but the server's own 40 MiB do not
@pytest.mark.parametrize("mib", [312, 345])
def test_server(leave, mib):
    warm()
    nets, pats = zip(*(network() for _ in range(2)))
    cols = [np.sort(p[0][:20]).astype(np.uint32) for p in pats]
    want = [n.recall(ax.clamp_words(c, 4096)[None], 9, 3, method="plain")["final"][0] for n, c in zip(nets, cols)]
    leave(mib)
    with ax.Server(list(nets), 40 * MIB) as srv:
        for tag in range(60):
            srv.submit(tag % 2, cols[tag % 2], 3, 6, tag)
        srv.wait_idle(60)
        got = srv.poll(60)
    assert len(got) == 60
    for res, spikes in got:
        assert np.array_equal(spikes, want[res["net"]])
    for n in nets:
        n.close()
