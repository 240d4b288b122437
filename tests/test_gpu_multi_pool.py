"""The multi-network launch with tiles in a shared-memory pool (threads=0: one or two columns
per warp) leaves every network as the plain path does, for slots of several sizes, uneven
queues and the learning-rule variants."""
import numpy as np
import pytest

import axon_b200 as ax

pytestmark = pytest.mark.gpu


def run(cfg, loads, method, **kw):
    nets = [ax.Network(cfg) for _ in loads]
    try:
        res, rep = ax.multi_train(nets, list(range(len(loads))), loads, epochs=2, stimcols=max(4, cfg["incols"] // 4),
                                  method=method, **kw)
        return res, rep, [{b: n.read(b) for b in ("W0", "W1", "W2", "W3", "BIAS", "SPK_A", "SPK_B")} for n in nets]
    finally:
        for n in nets:
            n.close()


def check(cfg, loads, slots, tiles=0):
    a = run(cfg, loads, "launch", autotune=False, slots=slots, threads=0)
    b = run(cfg, loads, "plain")
    assert a[1]["slots"] == slots and a[1]["tiles"] == tiles
    assert a[0] == b[0]
    for x, y in zip(a[2], b[2]):
        for name in x:
            assert np.array_equal(x[name], y[name]), name


# columns per warp 1 and 2; slots too small for the pool (tiles 4) take the register form
@pytest.mark.parametrize("ncol,incols,loads,slots,tiles", [(32, 8, [1, 2, 1], 2, 0), (512, 64, [3, 5, 2, 6, 4], 3, 0),
                                                           (608, 72, [2, 3, 4], 1, 0), (2080, 256, [2, 3, 2, 1], 3, 0),
                                                           (2080, 256, [2, 3, 2, 1], 4, 4),  # 37 CTAs x 28 warps x 2: 2,072
                                                           (4096, 512, [2, 3, 1], 2, 0), (4096, 512, [1, 2, 1], 3, 4)])
def test_pool_equals_plain(ncol, incols, loads, slots, tiles):
    cfg = dict(ax.CONFIG_C, ncol=ncol, incols=incols, target=max(4, ncol // 32), k=12 if ncol < 600 else 24)
    check(cfg, loads, slots, tiles)


@pytest.mark.parametrize("variant", [dict(margingate=1, hetero=1, ltdrep=2, ltdevery=1), dict(contrast=0),
                                     dict(mode=2, dthr=3, boost=7), dict(topkpar=0), dict(bandlo=9, bandhi=6),
                                     dict(biasdownevery=3, biasshift=2, ktest=8, facil=5)])
def test_pool_rule_variants(variant):
    check(dict(ax.CONFIG_C, ncol=512, incols=64, target=24, **variant), [3, 4, 2], 2)


# the tuner's choice takes no longer than the best of the shapes it chooses from (which are 15 % apart at
# these widths; a tenth is allowed for the time of a launch)
@pytest.mark.parametrize("ncol,load", [(352, 6), (2080, 8)])
def test_tuner_finds_the_fastest_shape(ncol, load):
    cfg = dict(ax.CONFIG_C, ncol=ncol, incols=ncol // 8 // 8 * 8, target=ncol // 64)
    kw = dict(epochs=4, stimcols=ncol // 64, method="launch")
    with ax.Network(cfg) as net:
        forced = min(ax.multi_train([net], [1], [load], autotune=False, slots=1, threads=t, **kw)[1]["gpu_ms"]
                     for t in (0, 512, 896, 1024) for _ in range(2))
        assert ax.multi_train([net], [1], [load], **kw)[1]["gpu_ms"] <= 1.1 * forced
