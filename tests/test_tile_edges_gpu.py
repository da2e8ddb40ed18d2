"""Sizes at which the tiled kernels can go wrong: clusters, bands, frequencies and expansion orders that
do not fill a tile, orbitals without vertices, transfer lists that are cut, unsorted or repeated.  Against
the oracle, at the tolerances of the other GPU tests (the same arithmetic at other sizes)."""

import numpy as np
import pytest

from helpers import rel_err
from dca_b200 import workloads as W

pytestmark = pytest.mark.gpu

FP64_TOL, MIXED_TOL, SP_TOL = 1e-12, 1e-6, 1e-9

CLUSTERS = {"2x1": W.make_cluster((2, 0), (0, 1)), "3x2": W.make_cluster((3, 0), (0, 2)),
            "2x2": W.square_cluster(2), "betts8": W.betts8_cluster(), "4x4": W.square_cluster(4),
            "8x2": W.make_cluster((8, 0), (0, 2)), "5x5": W.square_cluster(5), "6x6": W.square_cluster(6),
            "9x4": W.make_cluster((9, 0), (0, 4))}


def _g0(rng, nb, cl, n_sp):
    """A G0 with the layout of workloads.make_g0 and random band blocks (nb = 1: time-reversal symmetric,
    as the models' is, so that the mirrored path runs)."""
    if nb == 1:
        return W.make_g0(W.Model("single", tp=-0.1), cl, 7.0, 0.3, n_sp)
    nc = cl.nc
    g = np.zeros((2 * n_sp, nc, 2, nb, 2, nb), complex)
    for s in range(2):
        g[:, :, s, :, s, :] = rng.normal(size=(2 * n_sp, nc, nb, nb)) + 1j * rng.normal(size=(2 * n_sp, nc, nb, nb))
    return g


def _measurements(rng, nb, nc, orders):
    # One sign in five negative: with as many of both the beta^2 G0 G0 terms, the same in every measurement,
    # cancel, and their FP32 rounding (6e-8 of the uncancelled sum) is all that a relative error sees.
    return [W.Measurement(-1 if i % 5 == 4 else 1, tuple(W.make_sector(rng, n, nb, nc, 7.0) for n in pair))
            for i, pair in enumerate(orders)]


def _params(nb, cl, nw_half, n_sp, channels, k_ex, w_ex, orders, **kw):
    from dca_b200.accumulators import TpParameters
    a_vecs = np.zeros((1, 2)) if nb == 1 else np.linspace(0, 0.5, 2 * nb).reshape(nb, 2)
    return TpParameters(nb, cl.nc, nw_half, n_sp, 7.0, channels, k_ex, w_ex, cl.r_vecs, cl.k_vecs, a_vecs, cl.k_add,
                        cl.k_sub, cl.r_sub, max_order=max(1, max(max(p) for p in orders)), **kw)


def _compare(oracle_lib, g0, measurements, params, tol):
    from dca_b200.accumulators import TpAccumulator
    ora = oracle_lib.OracleTp(g0, params)
    acc = TpAccumulator(g0, params)
    acc.resetAccumulation(0)
    for m in measurements:
        for a in (ora, acc):
            a.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)
    acc.finalize()
    for got, want in zip(acc.get_G4(), ora.get_G4()):
        assert np.all(np.isfinite(got))
        assert rel_err(got, want) <= tol
    return acc


@pytest.mark.parametrize("precision,tol", [(0, FP64_TOL), (1, MIXED_TOL)])
@pytest.mark.parametrize("cluster,nb,nw_half,w_ex,orders", [
    ("2x1", 1, 1, [0], [(1, 0), (3, 2)]),             # D = 4: less than one tile of rows
    ("3x2", 1, 5, [0, 1], [(33, 31), (1, 64)]),       # 6 sites: no FFT, momenta not a multiple of 8
    ("2x2", 2, 3, [1], [(17, 40), (0, 5)]),           # two bands
    ("2x1", 4, 2, [0], [(9, 30), (32, 1)]),           # more bands than the compiled cases
    ("betts8", 3, 3, [0, 2], [(47, 18), (5, 100)]),   # three bands, rows not a multiple of the tile
    ("4x4", 1, 5, [0], [(1, 33), (130, 7)]),          # 4 x 4 FFT, 10 frequencies, most orbitals empty
    ("5x5", 1, 2, [0], [(40, 70), (2, 25)]),          # 25 sites: matrix transform
    ("8x2", 1, 4, [0], [(40, 21), (97, 5)]),          # 16 and 36 sites without the FFT, half of G
    ("9x4", 1, 2, [0], [(40, 21), (97, 5)]),
    ("6x6", 1, 3, [0], [(40, 0), (97, 5)]),           # 6 x 6 FFT, 6 frequencies
])
def test_front_end_tiles(oracle_lib, precision, tol, cluster, nb, nw_half, w_ex, orders):
    rng = np.random.default_rng(5)
    cl = CLUSTERS[cluster]
    n_sp = nw_half + max(w_ex) + 3
    params = _params(nb, cl, nw_half, n_sp, [W.PH_MAGNETIC], [cl.nc - 1], w_ex, orders, precision=precision,
                     max_batch=2 if precision else 1)
    _compare(oracle_lib, _g0(rng, nb, cl, n_sp), _measurements(rng, nb, cl.nc, orders), params, tol)


@pytest.mark.parametrize("cluster,k_ex,n_meas,max_batch", [
    ("2x2", [3], 20, 20), ("2x2", [2, 0, 2], 3, 2), ("betts8", [1, 5, 2, 7, 0], 15, 15), ("4x4", [15], 8, 7),
    ("4x4", [3, 9, 1, 14, 8], 3, 3), ("6x6", [20], 5, 5), ("6x6", [35, 1], 2, 1)])
@pytest.mark.parametrize("channels", [[2, 3], [4, 2, 1]])
def test_transfer_subsets(oracle_lib, cluster, k_ex, n_meas, max_batch, channels):
    """Mixed path, cut transfer lists (the list's length against the threads' transfers, batches beyond the
    staged measurements), the second-order terms of every channel; PH channels alone run with half of G."""
    rng = np.random.default_rng(6)
    cl = CLUSTERS[cluster]
    orders = [(int(a), int(b)) for a, b in rng.integers(0, 30, (n_meas, 2))]
    nw_half = {"4x4": 8, "6x6": 4}.get(cluster, 2)
    params = _params(1, cl, nw_half, nw_half + 4, channels, k_ex, [0, 1] if cluster == "2x2" else [0], orders,
                     precision=1, max_batch=max_batch)
    _compare(oracle_lib, _g0(rng, 1, cl, nw_half + 4), _measurements(rng, 1, cl.nc, orders), params, MIXED_TOL)


@pytest.mark.parametrize("cluster", ["2x2", "betts8", "4x4"])
def test_all_transfers_all_channels(oracle_lib, cluster):
    """Mixed path, every transfer, four channels in another order than their terms run."""
    rng = np.random.default_rng(7)
    cl = CLUSTERS[cluster]
    orders = [(12, 7), (0, 0), (3, 25), (31, 2)]
    k_ex = list(rng.permutation(cl.nc))
    params = _params(1, cl, 2, 8, [3, 4, 1, 2], k_ex, [0, 1], orders, precision=1, max_batch=3)
    _compare(oracle_lib, _g0(rng, 1, cl, 8), _measurements(rng, 1, cl.nc, orders), params, MIXED_TOL)


@pytest.mark.parametrize("n_meas,max_batch,channels", [(32, 32, [2, 3]), (37, 37, [2]), (41, 33, [3])])
def test_large_cluster_all_transfers(oracle_lib, n_meas, max_batch, channels):
    """6x6, every transfer in another order, batches that do and do not fill the steps of eight measurements."""
    rng = np.random.default_rng(9)
    cl = CLUSTERS["6x6"]
    orders = [(int(a), int(b)) for a, b in rng.integers(0, 30, (n_meas, 2))]
    params = _params(1, cl, 2, 6, channels, list(rng.permutation(36)), [0], orders, precision=1, max_batch=max_batch)
    _compare(oracle_lib, _g0(rng, 1, cl, 6), _measurements(rng, 1, cl.nc, orders), params, MIXED_TOL)


@pytest.mark.parametrize("cluster,k_ex,n_meas,max_batch", [
    ("betts8", [5], 1, 1), ("betts8", [1, 6, 3], 35, 35), ("betts8", [7, 2, 0, 4, 1, 6, 3, 5], 4, 3),
    ("2x2", [2], 31, 31), ("2x2", [3, 0, 1, 2], 2, 2)])
def test_three_band_pairing(oracle_lib, cluster, k_ex, n_meas, max_batch):
    """Items that do and do not fill the passes of 512, runs cut by a pass, batches shorter and longer than the
    27 entries of an item, odd ones against the two measurements of a stage."""
    rng = np.random.default_rng(11)
    cl = CLUSTERS[cluster]
    orders = [(int(a), int(b)) for a, b in rng.integers(0, 25, (n_meas, 2))]
    params = _params(3, cl, 2, 7, [W.PP_UP_DOWN], k_ex, [0, 1], orders, precision=1, max_batch=max_batch)
    _compare(oracle_lib, _g0(rng, 3, cl, 7), _measurements(rng, 3, cl.nc, orders), params, MIXED_TOL)


def test_three_band_pairing_large_batch(oracle_lib):
    """A batch whose signs alone fill what the tiles leave of shared memory: the pairing kernel still takes it (the
    general one reports its launch shapes).  3,000 FP32 additions of four roundings, three fifths of the terms
    surviving the signs: 0.46 u sqrt(3000) = 1.5e-6."""
    rng = np.random.default_rng(15)
    cl = CLUSTERS["betts8"]
    orders = [(int(a), int(b)) for a, b in rng.integers(1, 3, (3000, 2))]
    params = _params(3, cl, 1, 4, [W.PP_UP_DOWN], [2], [0], orders, precision=1, max_batch=3000)
    acc = _compare(oracle_lib, _g0(rng, 3, cl, 4), _measurements(rng, 3, cl.nc, orders), params, 3e-6)
    assert "g4staged" not in acc.tuning_report()


def _symmetric(cl, g0):
    """g0 with G0(-k, -w) = conj G0(k, w) to the bit."""
    identity = [z for z in range(cl.nc) if np.array_equal(cl.k_add[z], np.arange(cl.nc))][0]
    minus = cl.k_sub[:, identity]
    return 0.5 * (g0 + np.conj(g0[::-1][:, minus]))


@pytest.mark.parametrize("cluster,k_ex,w_ex,channels,mode", [
    ("2x1", [1], [0, 2], [3], 1),      # frequency transfers not closed under negation: half of G alone
    ("3x2", [5], [0], [2], 1),         # nor is this momentum transfer
    ("3x2", [5, 3], [0], [2], 3),      # each the other's negative
    ("4x4", [15], [-1, 1], [2, 3], 3),
    ("3x2", [0, 1, 2, 3, 4, 5], [0], [3, 2], 2)])  # half of G4 alone: with this many transfers the update reads all of G
def test_fp64_half_g(monkeypatch, cluster, k_ex, w_ex, channels, mode):
    """FP64: G4 and G with half of G or G4 against all of it.  The two halves come from different
    terms' roundings of one sum: a few ulps of the largest entries."""
    from dca_b200.accumulators import TpAccumulator
    rng = np.random.default_rng(12)
    cl = CLUSTERS[cluster]
    orders = [(33, 7), (0, 18)]
    params = _params(1, cl, 3, 9, channels, k_ex, w_ex, orders)
    g0 = _symmetric(cl, _g0(rng, 1, cl, 9))
    measurements, got = _measurements(rng, 1, cl.nc, orders), []
    for full in ("0", "1"):
        monkeypatch.setenv("DCAACC_TP_FULL_G", full)
        acc = TpAccumulator(g0, params)
        assert acc.mirror_mode() == (0 if full == "1" else mode)
        acc.resetAccumulation(0)
        for m in measurements:
            acc.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)
        gs = [acc.get_G(spin) for spin in range(2)]
        acc.finalize()
        got.append(gs + acc.get_G4())
    for a, b in zip(*got):
        assert rel_err(a, b) <= FP64_TOL


def test_fp64_whole_g_when_not_symmetric():
    """An asymmetry of G0 beyond rounding: the whole of G and G4."""
    from dca_b200.accumulators import TpAccumulator
    cl = CLUSTERS["4x4"]
    g0 = _symmetric(cl, _g0(None, 1, cl, 9))
    params = _params(1, cl, 3, 9, [2], [15], [0], [(1, 1)])
    assert TpAccumulator(g0, params).mirror_mode() == 3
    g0[9, 3, 0, 0, 0, 0] += 1e-14 * np.abs(g0).max()
    assert TpAccumulator(g0, params).mirror_mode() == 0


@pytest.mark.parametrize("cluster,max_order,fp32", [("2x2", 512, True), ("2x2", 513, False), ("2x1", 600, False),
                                                    ("3x2", 600, True)])
def test_front_end_of_small_clusters(oracle_lib, cluster, max_order, fp32):
    """Up to four sites: the FP32 front-end up to 512 vertices, orders up to the handle's limit."""
    rng = np.random.default_rng(17)
    cl = CLUSTERS[cluster]
    orders = [(max_order, 3), (0, max_order - 1), (127, 257)]
    params = _params(1, cl, 5, 9, [2, 4], [0], [0, 1], orders, precision=1, max_batch=3)
    acc = _compare(oracle_lib, _g0(rng, 1, cl, 9), _measurements(rng, 1, cl.nc, orders), params, MIXED_TOL)
    assert ("row32" in acc.tuning_report()) == fp32 and ("tc_row_order" in acc.tuning_report()) != fp32


@pytest.mark.parametrize("cluster,channels,k_ex,fp32,mode", [
    ("8x2", [2], [15], True, 3), ("8x2", [4], [15], True, 0), ("8x2", [2, 3], list(range(16)), False, 3),
    ("9x4", [2], [35], True, 1), ("9x4", [4], [35], False, 0), ("9x4", [2, 4], [35, 1, 2], False, 0),
    ("9x4", [3], list(range(36)), False, 3)])
def test_front_end_of_clusters_without_fft(oracle_lib, cluster, channels, k_ex, fp32, mode):
    """16 and 36 sites off the square clusters: which front-end runs (the launch-shape tuner names its kernels),
    with half of G where it applies (half of D a whole number of 128-row tiles on the tensor cores)."""
    rng = np.random.default_rng(14)
    cl = CLUSTERS[cluster]
    orders = [(40, 21), (97, 5), (0, 3)]
    nw_half = 32 if len(k_ex) == 36 else 8
    params = _params(1, cl, nw_half, nw_half + 3, channels, k_ex, [0], orders, precision=1, max_batch=2)
    acc = _compare(oracle_lib, _g0(rng, 1, cl, nw_half + 3), _measurements(rng, 1, cl.nc, orders), params, MIXED_TOL)
    assert ("row32" in acc.tuning_report()) == fp32 and ("tc_row_order" in acc.tuning_report()) != fp32
    assert acc.mirror_mode() == mode


@pytest.mark.parametrize("twist", [(0.0, 0.0), (0.3, -0.7)])
@pytest.mark.parametrize("order", ["sorted", "shuffled"])
def test_fp64_phases_of_the_given_momenta(oracle_lib, twist, order):
    """4x4, FP64: the phases are those of the momenta as given, here 2 pi m / 4 + 8 ulps or a twisted boundary's, not of
    exact quarters (off by 3e-15 rms in the first case).  Between different frequencies, where G is M's part
    alone: sums of 10 to 100 rounded terms twice over, in both codes, leave 10 u = 1.1e-15 at most."""
    from dca_b200.accumulators import TpAccumulator
    rng = np.random.default_rng(13)
    cl = CLUSTERS["4x4"]
    orders = [(120, 45)]
    params = _params(1, cl, 5, 9, [2], [15], [0], orders)
    params.k_vecs = cl.k_vecs + np.array(twist)
    if order == "shuffled":
        sites = rng.permutation(16)
        params.r_vecs, params.r_sub = cl.r_vecs[sites], None
    acc, ora = TpAccumulator(_g0(rng, 1, cl, 9), params), oracle_lib.OracleTp(_g0(rng, 1, cl, 9), params)
    acc.resetAccumulation(0)
    for m in _measurements(rng, 1, cl.nc, orders):
        for a in (acc, ora):
            a.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)
    for spin in range(2):
        got, want = (np.asarray(a.get_G(spin)).reshape(10, 10, -1) for a in (acc, ora))  # w2, w1
        off = ~np.eye(10, dtype=bool)
        print("error:", rel_err(got[off], want[off]))
        assert rel_err(got[off], want[off]) <= 10 * 2.0 ** -53


def test_fp64_graphs():
    """FP64 with and without captured graphs, orders on both sides of the launch shapes' steps of 128."""
    from dca_b200.accumulators import TpAccumulator
    rng = np.random.default_rng(10)
    cl = CLUSTERS["2x2"]
    orders = [(3, 128), (129, 0), (1, 127), (130, 140), (128, 128), (5, 7), (200, 129), (0, 0), (17, 2)]
    params = _params(1, cl, 2, 6, [2, 4], [1, 3], [0, 1], orders)
    measurements, got = _measurements(rng, 1, cl.nc, orders), []
    for graphs in (True, False):
        acc = TpAccumulator(_g0(rng, 1, cl, 6), params)
        acc.set_graphs(graphs)
        for _ in range(2):
            acc.resetAccumulation(0)
            for m in measurements:
                acc.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)
        acc.finalize()
        assert (acc.graph_stats()[0] > 0) == graphs
        got.append(acc.get_G4())
    for a, b in zip(*got):
        assert np.array_equal(a, b)


@pytest.mark.parametrize("cluster,nb,n_sp,orders", [
    ("2x2", 1, 5, [(0, 1), (2, 0)]), ("betts8", 3, 37, [(31, 32), (33, 65)]), ("3x2", 2, 64, [(7, 129)])])
def test_single_particle_pairs(oracle_lib, cluster, nb, n_sp, orders):
    """Pair counts around the warps' 32, frequency counts that do not fill the finalize passes."""
    from dca_b200.accumulators import SpAccumulator, SpParameters
    rng = np.random.default_rng(8)
    cl = CLUSTERS[cluster]
    params = SpParameters(nb, cl.nc, n_sp, 7.0, cl.r_sub, max_order=max(max(p) for p in orders))
    acc, ora = SpAccumulator(params, True), oracle_lib.OracleSp(params, True)
    acc.resetAccumulation()
    for m in _measurements(rng, nb, cl.nc, orders):
        for a in (acc, ora):
            a.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)
    acc.finalize()
    ora.finalize()
    assert rel_err(acc.get_sign_times_M_r_w(), ora.get()) <= SP_TOL
    assert rel_err(acc.get_sign_times_M_r_w_sqr(), ora.get(True)) <= SP_TOL
