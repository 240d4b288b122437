"""Networks of different widths used side by side: what one call or server sets for its kernels
does not refuse another's launches."""
import threading

import numpy as np
import pytest

import axon_b200 as ax

pytestmark = pytest.mark.gpu


def network(ncol, **kw):
    net = ax.Network(dict(ax.CONFIG_C, ncol=ncol, incols=ncol // 8, target=max(4, ncol // 64), **kw))
    net.init(ncol)
    pats = ax.stimuli(1, 3, ncol // 8, max(4, ncol // 64))
    for p in pats:
        net.present(ax.clamp_words(p, ncol), 8, 4, True)
    return net, np.stack([ax.clamp_words(p, ncol) for p in pats])


# one host thread per network: the bit planes, 16-bit counters, and the tensor contraction
@pytest.mark.parametrize("kw,contraction", [(dict(), "popc"), (dict(boost=300), "popc"), (dict(), "tensor")])
def test_threads_with_networks_of_their_own(kw, contraction):
    nets = [network(ncol, **kw) for ncol in (256, 1056)]
    batches = [np.tile(cues, (n, 1)) for (_, cues), n in zip(nets, (55, 70))]
    wants = [net.recall(b, 4, 2, method="plain")["final"] for (net, _), b in zip(nets, batches)]
    errors = []

    def work(i):
        try:
            for _ in range(250):
                got = nets[i][0].recall(batches[i], 4, 2, contraction=contraction)["final"]
                assert np.array_equal(got, wants[i])
        except BaseException as e:  # noqa: BLE001 - reported by the main thread
            errors.append(e)

    threads = [threading.Thread(target=work, args=(i,)) for i in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for net, _ in nets:
        net.close()


# facilitation runs the gather and batched kernels, whose step kernel's shared memory grows with the width
@pytest.mark.parametrize("kw", [dict(facil=5), dict()])
def test_server_of_narrower_networks_beside_a_running_one(kw):
    wide, narrow = network(4096, **kw), network(256, **kw)

    def answer(srv, net, cues, tag):
        cols = np.flatnonzero(cues[0][: net.ncol // 8]).astype(np.uint32)
        srv.submit(0, cols, 3, 5, tag)
        srv.wait_idle(30)
        (res, spikes), = srv.poll(4)
        assert res["tag"] == tag and np.array_equal(spikes, net.recall(cues[:1], 8, 3, method="plain")["final"][0])

    with ax.Server([wide[0]], 64 << 20) as first:
        answer(first, *wide, 1)
        with ax.Server([narrow[0]], 64 << 20) as second:
            answer(second, *narrow, 2)
            answer(first, *wide, 3)
        answer(first, *wide, 4)
    for net, _ in (wide, narrow):
        net.close()
