"""Handles that accumulate half of G4 (mirror symmetry) beside handles that accumulate all of it: sharing one G4,
adding into each other, reads of the running and of the finalized G4.  Against the oracle, which always sums the
whole, at the tolerances of the other GPU tests."""

import numpy as np
import pytest

from helpers import rel_err
from dca_b200 import workloads as W

pytestmark = pytest.mark.gpu

FP64_TOL, MIXED_TOL = 1e-12, 1e-6
CLUSTER = W.square_cluster(4)
BETA, NW_HALF, N_SP, MAX_ORDER = 7.0, 4, 8, 40


def _g0(symmetric=True):
    """Symmetric to the bit (all hoppings real), or with a G0(k, w) of no symmetry at all."""
    g = W.make_g0(W.Model("single", tp=-0.1), CLUSTER, BETA, 0.3, N_SP)
    if not symmetric:
        rng = np.random.default_rng(2)
        g = g * (1 + 0.2 * rng.normal(size=g.shape) + 0.2j * rng.normal(size=g.shape))
    return g


def _params(precision=0, k_ex=range(16), channels=(W.PH_MAGNETIC, W.PH_CHARGE), max_batch=None):
    from dca_b200.accumulators import TpParameters
    return TpParameters(1, 16, NW_HALF, N_SP, BETA, list(channels), list(k_ex), [0], CLUSTER.r_vecs, CLUSTER.k_vecs,
                        np.zeros((1, 2)), CLUSTER.k_add, CLUSTER.k_sub, CLUSTER.r_sub, max_order=MAX_ORDER,
                        precision=precision, max_batch=max_batch or (2 if precision else 1))


def _measurements(count, seed):
    rng = np.random.default_rng(seed)
    return [W.Measurement(-1 if i % 3 == 2 else 1,
                          tuple(W.make_sector(rng, int(n), 1, 16, BETA) for n in rng.integers(5, MAX_ORDER, 2)))
            for i in range(count)]


def _feed(acc, measurements):
    for m in measurements:
        acc.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)


class _Fed:
    """A handle and the oracle of everything that it has been fed."""

    def __init__(self, oracle_lib, symmetric=True, **kw):
        from dca_b200.accumulators import TpAccumulator
        self.acc = TpAccumulator(_g0(symmetric), _params(**kw))
        self.acc.resetAccumulation(0)
        self.ora = oracle_lib.OracleTp(_g0(symmetric), _params(**kw))

    def feed(self, count, seed):
        for a in (self.acc, self.ora):
            _feed(a, _measurements(count, seed))
        return self

    def want(self):
        return [np.array(g) for g in self.ora.get_G4()]


def _total(*fed):
    return [sum(gs) for gs in zip(*(f.want() for f in fed))]


def _check(acc, want, tol):
    acc.finalize()
    for got, ref in zip(acc.get_G4(), want):
        assert rel_err(got, ref) <= tol


def _tol(*kinds):
    return MIXED_TOL if any(k.get("precision") for k in kinds) else FP64_TOL


HALF, FULL = dict(), dict(symmetric=False)                            # FP64
MIXED_HALF, MIXED_FULL = dict(precision=1), dict(precision=1, symmetric=False)


def test_modes(oracle_lib):
    """The four kinds of handle that the tests below combine."""
    for kind, mode in ((HALF, 2), (FULL, 0), (MIXED_HALF, 3), (MIXED_FULL, 0)):
        assert _Fed(oracle_lib, **kind).acc.mirror_mode() == mode


@pytest.mark.parametrize("first,second", [(HALF, HALF), (HALF, FULL), (FULL, HALF), (HALF, MIXED_FULL), (MIXED_FULL, HALF),
                                          (MIXED_HALF, MIXED_HALF)])
def test_shared_g4_of_two_kinds(oracle_lib, first, second):
    """Measurements before and after the two share a G4, and a third handle that joins later: the others' modes
    stay as they are, and every contribution arrives."""
    a, b = _Fed(oracle_lib, **first).feed(2, 1), _Fed(oracle_lib, **second).feed(2, 2)
    b.acc.share_G4_with(a.acc)
    modes = a.acc.mirror_mode(), b.acc.mirror_mode()
    a.feed(2, 3)
    b.feed(1, 4)
    joiner = first if first is MIXED_HALF else FULL
    c = _Fed(oracle_lib, **joiner).feed(1, 5)
    c.acc.share_G4_with(a.acc)
    assert (a.acc.mirror_mode(), b.acc.mirror_mode()) == modes
    for fed, seed in ((a, 6), (b, 7), (c, 8)):
        fed.feed(2, seed)
    b.acc.sumTo(a.acc)
    c.acc.sumTo(a.acc)
    _check(a.acc, _total(a, b, c), _tol(first, second))


@pytest.mark.parametrize("owner,joiner", [(HALF, MIXED_HALF), (MIXED_HALF, HALF), (FULL, MIXED_HALF)])
def test_refused_share_changes_nothing(oracle_lib, owner, joiner):
    """A mixed handle with half of G4 shares with handles of its own kind alone."""
    from dca_b200.accumulators import LogicError
    a, b = _Fed(oracle_lib, **owner).feed(2, 1), _Fed(oracle_lib, **joiner).feed(2, 2)
    modes = a.acc.mirror_mode(), b.acc.mirror_mode()
    with pytest.raises(LogicError):
        b.acc.share_G4_with(a.acc)
    assert (a.acc.mirror_mode(), b.acc.mirror_mode()) == modes
    for fed, kind in ((a, owner), (b, joiner)):
        _check(fed.feed(1, 3).acc, fed.want(), _tol(kind))


@pytest.mark.parametrize("source,target", [(FULL, HALF), (HALF, FULL), (HALF, HALF), (MIXED_FULL, HALF), (MIXED_HALF, HALF),
                                           (FULL, MIXED_HALF), (MIXED_FULL, MIXED_HALF), (HALF, MIXED_HALF)])
def test_sum_to_between_kinds(oracle_lib, source, target):
    """The target's G4 is the sum of both, whatever half of it either has accumulated, also after further
    measurements; and so is what a read of the running G4 gives."""
    a, b = _Fed(oracle_lib, **source).feed(3, 1), _Fed(oracle_lib, **target).feed(2, 2)
    a.acc.sumTo(b.acc)
    tol = _tol(source, target)
    size = b.want()[0].size
    for c, ref in enumerate(_total(a, b)):
        assert rel_err(b.acc.peek_G4(c, 0, size), ref) <= tol
    b.feed(3, 3)
    _check(b.acc, _total(a, b), tol)
    a.acc.finalize()
    assert not any(np.any(g) for g in a.acc.get_G4())


def test_sum_to_shared_half_g4(oracle_lib):
    """Into a G4 that mixed handles accumulate by halves: only what has the mirror symmetry."""
    from dca_b200.accumulators import LogicError
    a, b = _Fed(oracle_lib, **MIXED_HALF).feed(2, 1), _Fed(oracle_lib, **MIXED_HALF).feed(2, 2)
    b.acc.share_G4_with(a.acc)
    c, d = _Fed(oracle_lib, **FULL).feed(2, 3), _Fed(oracle_lib, **HALF).feed(2, 4)
    with pytest.raises(LogicError):
        c.acc.sumTo(a.acc)
    d.acc.sumTo(a.acc)
    b.acc.sumTo(a.acc)
    _check(a.acc, _total(a, b, d), MIXED_TOL)
    _check(c.acc, c.want(), FP64_TOL)


@pytest.mark.parametrize("kind", [HALF, MIXED_HALF])
@pytest.mark.parametrize("shared", [False, True])
def test_reads_of_a_running_half_g4(oracle_lib, kind, shared):
    """Windows below and above the one that a handle keeps (65,536 entries), at both ends and between, in one
    private or shared G4 that goes on accumulating; reads that follow one another; and the finalized G4 after them."""
    a = _Fed(oracle_lib, **kind)
    if shared:
        b = _Fed(oracle_lib, **kind)
        b.acc.share_G4_with(a.acc)
    size = a.want()[0].size
    for seed, (offset, count) in enumerate([(5, 100), (7, 65536), (3, 65537), (size - 70000, 70000), (1, size - 1),
                                            (0, size), (size, 0)]):
        a.feed(1, seed)
        for channel in (1, 0):
            got = a.acc.peek_G4(channel, offset, count)
            assert got.size == count and rel_err(got, a.want()[channel][offset:offset + count]) <= _tol(kind)
    # Several reads without an update between them, then another handle's sum, then an update.
    c = _Fed(oracle_lib, **kind).feed(1, 20)
    fed = [a]
    for step in range(3):
        if step == 1:
            c.acc.sumTo(a.acc)
            fed.append(c)
        if step == 2:
            a.feed(1, 21)
        want = _total(*fed)[1]
        for offset, count in [(0, 70000), (70000, 70000), (100, 50), (140000, size - 140000), (30, 90000)]:
            assert rel_err(a.acc.peek_G4(1, offset, count), want[offset:offset + count]) <= _tol(kind)
    _check(a.acc, _total(*fed), _tol(kind))
    a.acc.resetAccumulation(1)
    assert not np.any(a.acc.peek_G4(1, 0, size))


@pytest.mark.parametrize("kind", [HALF, FULL, MIXED_HALF])
def test_finalized_g4_outlives_changes(oracle_lib, kind):
    """get_G4 after finalize gives the finalized sums, read from the device or kept on the host: after a
    sumTo that clears the device's, after a share, and while other handles add to the shared ones."""
    import ctypes

    from dca_b200 import _native as N

    def read(acc, c):
        out = np.empty(a.want()[c].size, np.complex128)
        assert N.lib.dcaacc_tp_get_g4(acc._h, c, out.view(np.float64).ctypes.data_as(
            ctypes.POINTER(ctypes.c_double)), out.size) == 0
        return out

    a, b, c = (_Fed(oracle_lib, **kind).feed(2, seed) for seed in (1, 2, 3))
    want = a.want()
    a.acc.finalize()
    a.acc.peek_G4(0, 0, want[0].size)
    a.acc.sumTo(b.acc)
    for channel in range(2):
        assert rel_err(read(a.acc, channel), want[channel]) <= _tol(kind)
    total = _total(a, b)
    _check(b.acc, total, _tol(kind))
    c.acc.share_G4_with(b.acc)
    c.feed(2, 4)
    c.acc.synchronizeCopy()
    for channel in range(2):
        assert rel_err(read(b.acc, channel), total[channel]) <= _tol(kind)
    _check(c.acc, _total(a, b, c), _tol(kind))


def test_finalize_reuses_only_unreferenced_arrays(oracle_lib):
    """A result that the caller still holds, whole or by a view, stays as it was; one that nothing holds is
    the next result's memory."""
    a = _Fed(oracle_lib)

    def result(seed):
        a.acc.resetAccumulation(seed)
        a.feed(1, seed)
        a.acc.finalize()

    result(1)
    kept = a.acc.get_G4()[0]
    view = a.acc.get_G4()[1][5:9]
    copies = kept.copy(), view.copy()
    result(2)
    assert not np.shares_memory(kept, a.acc.get_G4()[0]) and not np.shares_memory(view, a.acc.get_G4()[1])
    assert np.array_equal(kept, copies[0]) and np.array_equal(view, copies[1])
    addresses = [g.ctypes.data for g in a.acc.get_G4()]
    result(3)
    assert [g.ctypes.data for g in a.acc.get_G4()] == addresses


@pytest.mark.parametrize("precision", [0, 1])
def test_graphs_on_a_shared_stream(precision):
    """A handle on the caller's stream captures its batches while another thread launches on the same stream: the
    other's kernels run once each, and the handle's graphs hold its own alone."""
    import threading

    import torch

    from dca_b200.accumulators import TpAccumulator
    want = TpAccumulator(_g0(), _params(precision))
    want.set_graphs(False)
    got = TpAccumulator(_g0(), _params(precision))
    stream = torch.cuda.Stream()
    got.set_stream(stream.cuda_stream)
    count, stop, calls = torch.zeros(1, dtype=torch.float64, device="cuda"), threading.Event(), [0]
    torch.cuda.synchronize()

    def other():
        with torch.cuda.stream(stream):
            while not stop.is_set():
                count.add_(1.)
                calls[0] += 1

    thread = threading.Thread(target=other)
    thread.start()
    try:
        for acc in (got, want):
            acc.resetAccumulation(0)
            _feed(acc, _measurements(60, 30))
            acc.synchronizeCopy()
    finally:
        stop.set()
        thread.join()
    torch.cuda.synchronize()
    assert got.graph_stats()[0] > 0 and got.graph_stats()[1] > 0
    assert count.item() == calls[0]
    for acc in (got, want):
        acc.finalize()
    for a, b in zip(got.get_G4(), want.get_G4()):
        assert rel_err(a, b) <= (1e-14 if precision == 0 else 1e-7)
    del got  # before its stream
