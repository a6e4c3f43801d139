"""Runs of small boxes in one launch: several boxes, threads and refused launches side by side."""
import json
import threading
import time

import numpy as np
import pytest

import mdpd

pytestmark = pytest.mark.gpu

DPD = dict(style=1, A=25.0, rho_est=0.0)


def batch(n, style=0, seed=1, exact=0):
    kw = dict(DPD) if style else {}
    return mdpd.Batch([mdpd.box_spec(n, (n / (3.0 if style else 6.05)) ** (1 / 3), seed=seed, init_seed=seed + 6,
                                     exact_rng=exact, **kw)])


def same(a, b):
    return all(np.array_equal(p, q) for p, q in zip(a, b))


# pairs of sizes whose runs share a kernel (32, 8 and 2 lanes per row on 148 SMs: up to 24, up to 96 and
# more rows per block) but not the amount of shared memory
@pytest.mark.parametrize("large,small", [(3000, 2000), (9000, 5000), (20000, 15000)])
@pytest.mark.parametrize("style", [0, 1])
def test_boxes_that_share_a_run_kernel(style, large, small):
    """the larger box's batch is made first, then the smaller one's; both step on in turn, then from a
    thread each: every box as it is alone"""
    sizes = (large, small)

    def alone(k):
        b = batch(sizes[k], style, seed=k + 1)
        b.setup()
        for _ in range(6):
            b.step(7)
        s = b.state(0)
        b.close()
        return s

    want = [alone(k) for k in range(2)]
    bs = [batch(sizes[k], style, seed=k + 1) for k in range(2)]
    for b in bs:
        b.setup()
    for _ in range(3):
        for b in bs:
            b.step(7)
    errors = []

    def go(b):
        try:
            for _ in range(3):
                b.step(7)
        except Exception as e:  # seen by the main thread
            errors.append(e)

    th = [threading.Thread(target=go, args=(b,)) for b in bs]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not errors, errors
    for k in range(2):
        assert same(bs[k].state(0), want[k])
        bs[k].close()


def test_a_smaller_box_leaves_an_earlier_box_its_one_launch_runs():
    """the larger box's launch still goes through: with its barrier wait made to run out, its call says so
    (on the step graph it would succeed)"""
    for style, large, small in ((0, 3000, 2000), (0, 20000, 15000), (1, 20000, 15000)):
        a, b = batch(large, style), batch(small, style)
        for q in (a, b):
            q.setup()
            q.step(4)
        assert mdpd.lib().mdpd_batch_test_run_wait(a.h, 8192, 3) == mdpd.OK
        with pytest.raises(mdpd.MdpdError) as e:
            a.step(4)
        assert e.value.code == mdpd.ERR_TIMEOUT
        b.step(4)
        a.close()
        b.close()


def test_a_small_box_beside_a_large_one():
    """calls of 1,000 steps of 2,000 particles from another thread do not keep a box of a million
    particles from stepping, and the small box, stepped partly in one-launch runs and partly by the step
    graph, keeps its bits"""
    big, small, ref = batch(1000000), batch(2000, seed=5), batch(2000, seed=5)
    for q in (big, small, ref):
        q.setup()
        q.step(300)

    def fastest():
        t = []
        for _ in range(5):
            a = time.perf_counter()
            big.step(20)
            t.append(time.perf_counter() - a)
        return min(t)

    alone = fastest()
    stop, calls, errors = threading.Event(), [0], []

    def go():
        try:
            while not stop.is_set():
                small.step(1000)
                calls[0] += 1
        except Exception as e:  # seen by the main thread
            errors.append(e)

    th = threading.Thread(target=go)
    th.start()
    time.sleep(0.05)
    beside = fastest()
    time.sleep(0.1)  # the small box alone again
    stop.set()
    th.join()
    assert not errors and calls[0] > 0
    # one-launch runs beside it: about 20 times as long; step graphs: a few per cent
    assert beside < 4 * alone
    for _ in range(calls[0]):
        ref.step(1000)
    assert same(small.state(0), ref.state(0))
    for q in (big, small, ref):
        q.close()


def test_small_boxes_of_several_threads_in_long_calls():
    """calls long enough to change between one-launch runs and the step graph under way"""
    sizes, steps = (2000, 3000, 2500), (1900, 700, 2600)

    def go(k, out):
        try:
            b = batch(sizes[k], k % 2, seed=k + 1)
            b.setup()
            b.step(steps[k])
            b.time(steps[k])  # plain steps only
            out[k] = b.state(0) + (np.array([b.thermo(0).step]),)
            b.close()
        except Exception as e:  # seen by the main thread
            out[k] = e

    alone, together = {}, {}
    for k in range(3):
        go(k, alone)
    th = [threading.Thread(target=go, args=(k, together)) for k in range(3)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    for k in range(3):
        assert not isinstance(together[k], Exception), together[k]
        assert same(alone[k], together[k]) and alone[k][2][0] == 2 * steps[k]


@pytest.mark.parametrize("style", [0, 1])
@pytest.mark.parametrize("launch", [1, 2, 3])
def test_a_refused_launch_in_the_middle_of_a_run(style, launch):
    """600 steps go in three launches; from the refused one on they go by the step graph: as many steps
    and the same bits"""
    a, b = batch(2500, style), batch(2500, style)
    for q in (a, b):
        q.setup()
    assert mdpd.lib().mdpd_batch_test_refuse_run(a.h, launch) == mdpd.OK
    for q in (a, b):
        q.step(601)
        assert q.thermo(0).step == 601
        q.step(30)
    assert same(a.state(0), b.state(0))
    assert a.thermo(0).step == b.thermo(0).step == 631
    a.close()
    b.close()


# barriers of a step that rebuilds: 1 after integrate, 2 to 10 between and after the rebuild's passes (2: the
# classes are counted, their counts not yet cleared), 11 after the density pass (mDPD), then the force pass's
@pytest.mark.parametrize("style,barrier", [(0, k) for k in range(1, 13)] + [(1, k) for k in (1, 2, 5, 10, 11)])
def test_a_barrier_wait_that_runs_out(style, barrier):
    """one arrival too few with a limit of a few ms: the call says so, whatever was queued behind it is
    skipped or stays in bounds, the box stays refused, and other boxes step on"""
    n = 2000
    kw = dict(DPD) if style else {}
    L = (n / (3.0 if style else 6.05)) ** (1 / 3)
    spec = mdpd.box_spec(n, L, check=0, seed=3, init_seed=4, **kw)  # a rebuild at every step
    other = batch(2500, style)
    other.setup()
    ref = batch(2500, style)
    ref.setup()
    b = mdpd.Batch([spec])
    b.setup()
    b.step(3)

    def refused(f):
        with pytest.raises(mdpd.MdpdError) as e:
            f()
        assert e.value.code == mdpd.ERR_TIMEOUT and "wait" in str(e.value)

    assert mdpd.lib().mdpd_batch_test_run_wait(b.h, 8192, barrier) == mdpd.OK
    refused(lambda: b.step(600))
    assert mdpd.lib().mdpd_batch_test_run_wait(b.h, 0, 0) == mdpd.OK
    other.step(20)
    refused(lambda: b.step(3))
    refused(lambda: b.run_thermo(2))
    refused(lambda: b.time(2))
    refused(lambda: b.setup())
    assert b.thermo(0).status & 128
    b.close()
    other.step(20)
    ref.step(20)
    ref.step(20)
    assert same(other.state(0), ref.state(0))
    other.close()
    ref.close()


def test_tune_cache_keeps_boxes_with_one_launch_runs_apart(tmp_path):
    """140,000 and 250,000 DPD particles lie in one power of two; the first box's runs go in one launch at
    one thread per particle, the second's do not: neither takes the other's stored pick"""
    cache = tmp_path / "tune.json"
    sizes = (140000, 250000)  # one-launch runs: up to 1,400 rows on each of 148 SMs
    for order in (sizes, sizes[::-1]):
        if cache.exists():
            cache.unlink()
        for n in order:
            b = batch(n, 1)
            b.setup()
            d, f, hit = b.tune(cache=cache)
            assert not hit and (n == sizes[1] or (d, f) == (1, 1))
            b.close()
            # what is stored now is another shape than the next box would take by the rule
            j = json.loads(cache.read_text())
            for e in j["entries"].values():
                e["density"], e["force"] = 2, 4
            cache.write_text(json.dumps(j))
        assert len(j["entries"]) == 2
    b = batch(sizes[1], 1)  # an entry of its own class is applied
    b.setup()
    assert b.tune(cache=cache) == (2, 4, True)
    b.close()


def edge(kind):
    """specs of the last box whose runs go in one launch on 148 SMs, and of the first that does not"""
    if kind == "rows mdpd":  # 768 rows per block: each warp of the force pass holds 32
        return [mdpd.box_spec(n, (n / 6.05) ** (1 / 3), seed=2, init_seed=8) for n in (148 * 768, 148 * 768 + 1)]
    if kind == "rows dpd":  # 1,400 rows per block: shared memory is nearly full
        return [mdpd.box_spec(n, (n / 3.0) ** (1 / 3), seed=2, init_seed=8, **DPD) for n in (148 * 1400, 148 * 1400 + 1)]
    # 22^3 bins, mostly empty: as many as particles and 4,096 more
    return [mdpd.box_spec(n, 26.0, seed=2, init_seed=8, fill_lo=(12.2, 0, 0), fill_hi=(13.8, 26, 26))
            for n in (22 ** 3 - 4096, 22 ** 3 - 4097)]


@pytest.mark.parametrize("kind", ["rows mdpd", "rows dpd", "bins"])
def test_the_last_box_with_one_launch_runs_and_the_first_without(kind):
    """plain steps and steps with a thermo line each (always launches of their passes): the same bits"""
    for spec, one_launch in zip(edge(kind), (True, False)):
        a, b = mdpd.Batch([spec]), mdpd.Batch([spec])
        for q in (a, b):
            q.setup()
        a.step(14)
        b.run_thermo(14)
        assert same(a.state(0), b.state(0))
        assert a.thermo(0).nbuild == b.thermo(0).nbuild >= 3 and a.thermo(0).status == 0
        # which way the plain steps went: only one-launch runs meet a barrier
        mdpd.lib().mdpd_batch_test_run_wait(a.h, 8192, 1)
        if one_launch:
            with pytest.raises(mdpd.MdpdError) as e:
                a.step(2)
            assert e.value.code == mdpd.ERR_TIMEOUT
        else:
            a.step(2)
        a.close()
        b.close()
