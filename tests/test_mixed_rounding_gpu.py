"""Mixed precision: rounding errors that add up over a batch or that every entry shares, against the FP64 path."""

import numpy as np
import pytest

from helpers import rel_err
from dca_b200 import workloads as W

pytestmark = pytest.mark.gpu

U = 2.0 ** -24  # unit roundoff of FP32


def _run(cluster, precision, channels, k_ex, measurements, beta, nw_half=4, max_batch=1):
    from dca_b200.accumulators import TpAccumulator, TpParameters
    nc, n_sp = cluster.nc, nw_half + 3
    params = TpParameters(1, nc, nw_half, n_sp, beta, channels, k_ex, [0], cluster.r_vecs, cluster.k_vecs,
                          np.zeros((1, 2)), cluster.k_add, cluster.k_sub, cluster.r_sub,
                          max_order=max(s.n for m in measurements for s in m.sectors), precision=precision,
                          max_batch=max_batch)
    acc = TpAccumulator(W.make_g0(W.Model("single", tp=-0.15), cluster, beta, 0.3, n_sp), params)
    acc.resetAccumulation(0)
    for m in measurements:
        acc.accumulate([s.M for s in m.sectors], list(m.sectors), m.sign)
    acc.finalize()
    return acc


@pytest.mark.parametrize("length,channels,transfers", [
    (6, [W.PH_MAGNETIC], 1), (6, [W.PP_UP_DOWN], 1), (4, [W.PH_TRANSVERSE], 2), (6, [W.PH_TRANSVERSE], 36),
    (4, [W.PP_UP_DOWN], 16), (4, [W.PH_TRANSVERSE], 16)])
def test_batch_sums_round_once_a_measurement(length, channels, transfers):
    """64 measurements of nearly the same G: a sum that grows as j of 64 and is rounded once a measurement is
    off by 0.23 u sqrt(64) = 1.1e-7 (roundings of 0.4 u of the partial sum, as a random walk), four times a measurement
    by 2.2e-7.  The entries' own errors, 0.7e-7, come in quadrature: 1.4e-7 and 2.3e-7."""
    cluster = W.square_cluster(length)
    rng = np.random.default_rng(3)
    ms = [W.Measurement(1, tuple(W.make_sector(rng, int(n), 1, cluster.nc, 36.0) for n in rng.integers(21, 25, 2)))
          for _ in range(64)]
    k_ex = list(range(cluster.nc))[-transfers:]
    exact = _run(cluster, 0, channels, k_ex, ms, 36.0)
    got = _run(cluster, 1, channels, k_ex, ms, 36.0, max_batch=64)
    err = rel_err(got.get_G4()[0], exact.get_G4()[0])
    print("error:", err)
    assert err <= 1.8e-7


@pytest.mark.parametrize("cluster", [W.square_cluster(2), W.betts8_cluster(), W.square_cluster(4), W.square_cluster(6)])
def test_delta_term_rounds_once(cluster):
    """G = beta G0 delta (M = 0), with a beta whose rounding to FP32 is the largest there is, u: G rounded once
    leaves 0.4 u (2 G's: 0.6 u) and their product as much again, 0.8 u = 5e-8; a rounded beta would add 2 u in every entry."""
    beta = 4 * (1 + 2.0 ** -24)
    rng = np.random.default_rng(4)
    sectors = tuple(W.make_sector(rng, 1, 1, cluster.nc, beta) for _ in range(2))
    for s in sectors:
        s.M[:] = 0.
    ms = [W.Measurement(1, sectors)]
    exact = _run(cluster, 0, [W.PP_UP_DOWN], [0], ms, beta)
    got = _run(cluster, 1, [W.PP_UP_DOWN], [0], ms, beta)
    err = rel_err(got.get_G4()[0], exact.get_G4()[0])
    print("error:", err)
    assert err <= 8e-8
