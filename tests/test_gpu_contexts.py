"""Several contexts in one process, idle SMs of a small context, and contexts of very many chains."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

UP, DOWN, DYN = 0, 1, 2


def _run(hq, e, trips=2):
    for _ in range(trips):
        e.sweep(UP, hq.SWEEP_MEASURE)
        e.sweep(DOWN, hq.SWEEP_MEASURE)
    e.sync()
    return [e.g(0), e.fields(0), e.estimators(0)]


@pytest.mark.parametrize("mode", [0, 1], ids=["launches", "persistent"])
def test_a_context_of_smaller_chains_beside_a_larger_one(hq, mode):
    """The kernels' shared-memory limits are shared by the contexts of a process: a later context of
    smaller chains leaves them where an earlier one needs them."""
    def make(L):
        e = hq.Engine([dict(nl=L, u=4.0, mu=0.1, beta=0.8, nt=8, stabilization_pace=5, seed=L)])
        e.set_sweep_mode(mode)
        e.fields_random()
        e.init()
        return e
    a = make(12)
    want = _run(hq, a)
    a.close()
    a = make(12)
    b = make(4)
    got_small = _run(hq, b)
    for x, y in zip(_run(hq, a), want):
        assert np.array_equal(x, y)
    c = make(4)
    for x, y in zip(_run(hq, c), got_small):
        assert np.array_equal(x, y)
    for e in (a, b, c):
        e.close()


@pytest.mark.parametrize("chains", [1, 3])
def test_few_chains_hold_few_sms(hq, chains):
    """A persistent sweep holds no more SMs than it has chains, the most that can be at work at once: a
    CTA beyond them would only wait (its waits are counted when it takes an item), on an SM that other
    contexts could use. An item's look at the queue takes a few thousand cycles, an interval of ten
    8x8 slices some 400 thousand."""
    e = hq.Engine([dict(nl=8, u=4.0, mu=0.1, beta=20.0, nt=200, stabilization_pace=10, seed=c) for c in range(chains)])
    e.set_sweep_mode(hq.SWEEP_PERSISTENT)
    e.fields_random()
    e.init()
    e.sweep(UP)
    e.phase_cycles(reset=True)
    e.sweep(DOWN, hq.capi.SWEEP_PHASE_CLOCKS)
    pc = e.phase_cycles()
    assert pc["items"] == 20 * chains
    assert pc["wait"] < 0.25 * pc["interval"], pc
    e.close()


@pytest.mark.parametrize("L,per_sm,persistent", [(1, 1.75, True), (1, 1.76, False), (6, 1.75, True), (6, 1.76, False),
                                                 (4, 8.0, False)])
def test_default_mode_of_many_small_chains(hq, L, per_sm, persistent, monkeypatch):
    """Chains that outnumber the SMs by more than 7/4 gain from the launch sequence at any size."""
    import torch
    monkeypatch.delenv("HQ_SWEEP_MODE", raising=False)
    n = int(per_sm * torch.cuda.get_device_properties(0).multi_processor_count + 0.5)
    e = hq.Engine([dict(nl=L, u=4.0, mu=0.1, beta=0.2, nt=2, stabilization_pace=2, seed=c) for c in range(n)])
    assert e.sweep_mode() == (hq.SWEEP_PERSISTENT if persistent else hq.SWEEP_LAUNCHES)
    e.close()


def _many(hq, n, **kw):
    """n chains of 2 x 2, the last one with the parameters of the first and a seed of its own."""
    cfg = [dict(nl=2, u=4.0, mu=0.1, beta=0.3, nt=3, stabilization_pace=2, seed=1 + (c % 7), **kw) for c in range(n)]
    e, one = hq.Engine(cfg), hq.Engine([cfg[0], cfg[n - 1]])
    for x in (e, one):
        x.set_sweep_mode(hq.SWEEP_LAUNCHES)
        x.fields_random()
        x.init()
    return e, one


def test_displaced_sweep_of_22000_chains(hq):
    """Three job lists of the displaced builder in one launch: more than 65535 products."""
    n = 22000
    e, one = _many(hq, n, dynamic=1)
    for x in (e, one):
        x.sweep(DYN, hq.SWEEP_MEASURE)
        x.sweep(DOWN, hq.SWEEP_MEASURE)
    for k, c in ((0, 0), (1, n - 1)):
        assert np.array_equal(e.g(c), one.g(k))
        assert np.array_equal(e.fields(c), one.fields(k))
        for a, b in zip(e.dynamic_estimators(c), one.dynamic_estimators(k)):
            assert np.array_equal(a, b)
    e.close()
    one.close()


def test_adjoint_of_33000_chains(hq):
    """The push with the first builder product in one launch: more than 65535 products."""
    n = 33000
    e, one = _many(hq, n)
    (ld, gr), (ld1, gr1) = e.logdet_adjoint(), one.logdet_adjoint()
    for k, c in ((0, 0), (1, n - 1)):
        assert ld[c] == ld1[k] and gr[c][0] == gr1[k][0] and gr[c][1] == gr1[k][1]
        assert np.array_equal(gr[c][2], gr1[k][2])
    e.close()
    one.close()
