"""The work that programs have the measurement accumulators do, as cases that can be timed and checked.

A two-particle case is one bin of measurements: resetAccumulation, the measurements of the bin (one
accumulate call each, or accumulate_batch for a queue of walkers), and the read of the whole G4,
either with finalize / get_G4 (the end of a DCA iteration) or with peek_G4_async into pinned memory
that the program keeps (a bin of a longer accumulation).  A single-particle case is the same with
M(r, w).  A "g" case is dcaacc_tp_compute_g_noalloc: G of one measurement, device to device.

M matrices are on the device, as a walker on the GPU leaves them, and of the form (I + A)^-1 with
A_ij ~ N(0, 0.1 / n), the values that workloads.py gives them.
"""

from __future__ import annotations

import ctypes
import functools
import math

import numpy as np
import torch

from dca_b200 import _native as N
from dca_b200 import workloads as W
from dca_b200.accumulators import (SpAccumulator, SpParameters, TpAccumulator, TpParameters, _check, _make_sectors)

_CLUSTERS = {"2x1": ("rect", (2, 0), (0, 1)), "2x2": ("square", 2), "betts8": ("betts8",), "4x4": ("square", 4),
             "6x6": ("square", 6)}
_SITES = {"2x1": 2, "2x2": 4, "betts8": 8, "4x4": 16, "6x6": 36}
_CHANNELS = {"magnetic": (W.PH_MAGNETIC,), "magnetic+charge": (W.PH_MAGNETIC, W.PH_CHARGE),
             "transverse": (W.PH_TRANSVERSE,), "pp": (W.PP_UP_DOWN,),
             "all": (W.PH_TRANSVERSE, W.PH_MAGNETIC, W.PH_CHARGE, W.PP_UP_DOWN)}


def _tp(name, cluster, model, precision, channels, q, wex, nw, lo, hi, beta, count, batch, read):
    return dict(name=name, kind="tp", cluster=cluster, model=model, precision=precision, channels=channels, q=q,
                wex=wex, nw=nw, lo=lo, hi=hi, beta=beta, count=count, batch=batch, read=read)


def _sp(name, cluster, model, n_sp, lo, hi, beta, count, squares):
    return dict(name=name, kind="sp", cluster=cluster, model=model, n_sp=n_sp, lo=lo, hi=hi, beta=beta, count=count,
                squares=squares)


def _g(name, cluster, model, nw, lo, hi, beta):
    return dict(name=name, kind="g", cluster=cluster, model=model, nw=nw, lo=lo, hi=hi, beta=beta)


def listed():
    """q: "all" momentum transfers or one (an index into the cluster's momenta); wex: frequency transfers 0 .. wex;
    nw: four-point frequencies; lo, hi: range of the expansion orders; count: measurements in the bin."""
    return [
        # The smallest call: one measurement of a 2x2 cluster in double precision, and its G4 (latency).
        _tp("fp64_2x2_one", "2x2", "hubbard", "fp64", "magnetic", "0", 0, 16, 20, 60, 10.0, 1, 1, "finalize"),
        # Double precision, one call per measurement, every momentum transfer: a 4x4 study of both
        # particle-hole channels.
        _tp("fp64_4x4_allq", "4x4", "hubbard", "fp64", "magnetic+charge", "all", 0, 64, 100, 300, 20.0, 48, 1, "peek"),
        # The commonest production setting: double precision, the transfer (pi, pi) alone.
        _tp("fp64_4x4_oneq", "4x4", "hubbard", "fp64", "magnetic", "15", 0, 64, 100, 300, 20.0, 64, 1, "finalize"),
        # Pairing in the three-band model in double precision, zero momentum transfer.
        _tp("fp64_emery_pp", "betts8", "emery", "fp64", "pp", "0", 1, 16, 100, 300, 16.0, 16, 1, "finalize"),
        # Mixed precision, batches of a queue of walkers, uneven orders: the throughput setting.
        _tp("mixed_4x4_allq", "4x4", "hubbard", "mixed", "magnetic+charge", "all", 0, 64, 50, 400, 20.0, 1024, 64,
            "peek"),
        # Mixed precision with one transfer.
        _tp("mixed_4x4_oneq", "4x4", "hubbard", "mixed", "magnetic", "15", 0, 64, 50, 400, 20.0, 512, 64, "finalize"),
        # Three-band pairing over all transfers, four frequency transfers.
        _tp("mixed_emery_pp", "betts8", "emery", "mixed", "pp", "all", 3, 16, 100, 500, 16.0, 256, 32, "peek"),
        # The large cluster at high order.
        _tp("mixed_6x6_allq", "6x6", "hubbard_tp", "mixed", "magnetic", "all", 0, 32, 300, 1000, 40.0, 384, 128,
            "peek"),
        # All four channels of an 8-site cluster with a frequency transfer.
        _tp("mixed_betts8_all", "betts8", "hubbard", "mixed", "all", "all", 1, 24, 50, 250, 10.0, 128, 32, "peek"),
        # Single-particle accumulation: every measurement of every run does this.
        _sp("sp_4x4", "4x4", "hubbard", 512, 50, 400, 20.0, 64, False),
        # The same on the large cluster, with the squares for the error bars.
        _sp("sp_6x6_squares", "6x6", "hubbard_tp", 512, 300, 1000, 40.0, 12, True),
        # G of one measurement for a program that does its own two-particle work.
        _g("g_4x4", "4x4", "hubbard", 64, 100, 400, 20.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["tp"] * 6 + ["sp"] * 2 + ["g"])
    cluster = rng.choice(["2x2", "betts8", "4x4", "4x4", "6x6"])
    nc = _SITES[cluster]
    beta = round(rng.uniform(5.0, 40.0), 2)
    hi = _log(rng, 20, 700 if nc == 36 else 450)
    lo = rng.randint(0, hi)
    if kind == "sp":
        model = rng.choice(["hubbard", "hubbard_tp", "emery"]) if nc < 36 else "hubbard_tp"
        case = _sp("", cluster, model, _log(rng, 32, 512), lo, hi, beta, rng.randint(1, 24), rng.random() < 0.3)
    elif kind == "g":
        case = _g("", cluster, rng.choice(["hubbard", "hubbard_tp"]), 2 * rng.randint(4, 32 if nc <= 16 else 8), lo,
                  max(1, min(hi, 400 if nc <= 16 else 150)), beta)
        case["lo"] = min(case["lo"], case["hi"])
        if nc == 36:
            case["cluster"] = "4x4"
    else:
        model = rng.choice(["hubbard", "hubbard", "hubbard_tp", "emery"]) if nc <= 8 else \
            rng.choice(["hubbard", "hubbard_tp"])
        nb = 3 if model == "emery" else 1
        channels = rng.choice(sorted(_CHANNELS)) if nc <= 8 and nb == 1 else \
            rng.choice(["magnetic", "magnetic+charge", "pp"])
        q = "all" if rng.random() < 0.5 else str(rng.randrange(nc))
        wex = rng.choice([0, 0, 0, 1, 2])
        nw = 2 * _log(rng, 2, 32)
        precision = rng.choice(["fp64", "mixed", "mixed"])
        entries = len(_CHANNELS[channels]) * nb ** 4 * nc ** 2 * (nc if q == "all" else 1) * (wex + 1)
        while entries * nw * nw > 30e6 and nw > 2:  # half a GB of G4 at most
            nw = 2 * max(1, nw // 4)
        if precision == "fp64" or nb == 3:
            count, batch = rng.randint(1, 24), rng.choice([1, 1, 4]) if precision == "fp64" else rng.choice([8, 16])
        else:
            count, batch = _log(rng, 8, 192 if nc == 36 else 384), rng.choice([16, 32, 64])
        case = _tp("", cluster, model, precision, channels, q, wex, nw, lo, hi, beta, count, batch,
                   rng.choice(["peek", "finalize"]))
    del case["name"]
    return case


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
_MODELS = {"hubbard": dict(kind="single", t=1.0, U=6.0), "hubbard_tp": dict(kind="single", t=1.0, tp=-0.15, U=7.0),
           "emery": dict(kind="threeband", U=6.0)}


def _device():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


@functools.lru_cache(maxsize=None)
def _cluster(cluster):
    kind = _CLUSTERS[cluster]
    return W.make_cluster(kind[1], kind[2]) if kind[0] == "rect" else \
        W.betts8_cluster() if kind[0] == "betts8" else W.square_cluster(kind[1])


@functools.lru_cache(maxsize=32)
def _g0(cluster, model, beta, n_sp):
    m = W.Model(**_MODELS[model])
    mu = 0.0 if model == "hubbard" else W.find_mu(m, beta)
    return W.make_g0(m, _cluster(cluster), beta, mu, n_sp)


def _bands(case):
    return 3 if case["model"] == "emery" else 1


def _workload(case):
    """The case as a Workload (sizes, frequencies, channels)."""
    tp = case["kind"] == "tp"
    wex = case["wex"] if tp else 0
    nw_half = case.get("nw", 2) // 2
    n_sp = case.get("n_sp", nw_half + wex + 16)
    q = case["q"] if tp else "0"
    return W.Workload("case", W.Model(**_MODELS[case["model"]]), _CLUSTERS[case["cluster"]], case["beta"], nw_half,
                      n_sp, True, wex, 0 if q == "all" else int(q),
                      _CHANNELS[case["channels"]] if tp else (W.PH_MAGNETIC,), (case["lo"], case["hi"]),
                      case.get("batch", 1), mu=0.0)


def _tp_parameters(case):
    w = _workload(case)
    q = case.get("q", "all")
    nc = _SITES[case["cluster"]]
    p = TpParameters.from_workload(w, _cluster(case["cluster"]), k_ex=list(range(nc)) if q == "all" else [int(q)],
                                   max_order=max(1, case["hi"]), max_batch=case.get("batch", 1))
    p.precision = N.PRECISION_MIXED if case.get("precision") == "mixed" else N.PRECISION_FP64
    return p


def _inverses(orders, gen, device):
    """M = (I + A)^-1 of each order, column major on the device.  A's norm is below one half, so
    Newton's iteration X <- X (2 - (I + A) X) from X = I - A squares the residual each time."""
    out = []
    chunk = max(1, int(2e8 // max(1, max(orders) ** 2 * 8)))
    for c in range(0, len(orders), chunk):
        ns = orders[c:c + chunk]
        top = max(1, max(ns))
        A = torch.zeros(len(ns), top, top, dtype=torch.float64, device=device)
        for i, n in enumerate(ns):
            if n:
                A[i, :n, :n] = torch.randn(n, n, generator=gen, dtype=torch.float64, device=device) * math.sqrt(0.1 / n)
        eye = torch.eye(top, dtype=torch.float64, device=device)
        A += eye
        X = 2 * eye - A
        for _ in range(8):
            X = torch.matmul(X, 2 * eye - torch.matmul(A, X))
        for i, n in enumerate(ns):
            out.append(X[i, :n, :n].contiguous().t())
    return out


def _measurements(case, seed):
    """Signs, vertex configurations and device M matrices of the bin, from the seed alone."""
    count = case.get("count", 1)
    rng = np.random.default_rng([77, seed])
    device = _device()
    gen = torch.Generator(device=device)
    gen.manual_seed(1000003 * seed + 17)
    orders = [int(n) for n in rng.integers(case["lo"], case["hi"] + 1, 2 * count)]
    nc, nb = _SITES[case["cluster"]], _bands(case)
    configs = []
    for n in orders:
        tau = rng.uniform(0.0, case["beta"], n)
        site = rng.integers(0, nc, n).astype(np.int32)
        band = rng.integers(0, nb, n).astype(np.int32)
        configs.append(W.Sector(tau, band, band.copy(), site, site.copy(), None))
    signs = np.where(rng.uniform(size=count) < 0.95, 1, -1)
    Ms = _inverses(orders, gen, device)
    return [int(s) for s in signs], [configs[2 * i:2 * i + 2] for i in range(count)], \
        [Ms[2 * i:2 * i + 2] for i in range(count)]


def _tp_config(p, keep):
    arrays = [np.ascontiguousarray(a, np.int32) for a in (p.k_ex, p.w_ex, p.channels)] + \
        [np.ascontiguousarray(a, np.float64) for a in (p.r_vecs, p.k_vecs, p.a_vecs)] + \
        [np.ascontiguousarray(np.asarray(a, np.int32).T) for a in (p.k_add, p.k_sub)]
    keep.extend(arrays)
    ints = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_int32)) for a in arrays[:3] + arrays[6:]]
    reals = [a.ctypes.data_as(ctypes.POINTER(ctypes.c_double)) for a in arrays[3:6]]
    return N.TpConfig(p.n_bands, p.n_sites, p.n_w_half, p.n_sp_freq, len(p.k_ex), ints[0], len(p.w_ex), ints[1],
                      len(p.channels), ints[2], p.beta, reals[0], reals[1], reals[2], ints[3], ints[4], 0, 0, 1,
                      p.max_order, 1)


def prepare(case, seed):
    """Measurements on the device, the accumulator, and for "peek" the pinned memory that G4 is read into."""
    signs, configs, Ms = _measurements(case, seed)
    state = dict(case=case, signs=signs, configs=configs, Ms=Ms)
    if case["kind"] == "sp":
        state["acc"] = SpAccumulator(SpParameters.from_workload(_workload(case), _cluster(case["cluster"]),
                                                                max_order=max(1, case["hi"])),
                                     accumulate_m_squared=case["squares"])
    else:
        p = _tp_parameters(case)
        g0 = _g0(case["cluster"], case["model"], case["beta"], p.n_sp_freq)
        if case["kind"] == "g":
            keep = []
            state["cfg"] = _tp_config(p, keep)
            state["keep"] = keep
            state["G0"] = torch.from_numpy(np.ascontiguousarray(g0)).cuda()
            D = p.n_bands * p.n_sites * 2 * p.n_w_half
            state["G"] = torch.empty(2, D, D, dtype=torch.complex128, device="cuda")
        else:
            state["acc"] = TpAccumulator(g0, p)
            if case["read"] == "peek":
                state["out"] = [torch.empty(int(np.prod(p.g4_shape())), dtype=torch.complex128, pin_memory=True)
                                for _ in p.channels]
    torch.cuda.synchronize()
    return state


def run(state):
    case = state["case"]
    signs, configs, Ms = state["signs"], state["configs"], state["Ms"]
    if case["kind"] == "g":
        keep = []
        sectors = _make_sectors(Ms[0], configs[0], keep)
        _check(N.lib.dcaacc_tp_compute_g_noalloc(
            ctypes.byref(state["cfg"]), ctypes.c_void_p(state["G0"].data_ptr()), sectors,
            ctypes.c_void_p(state["G"].data_ptr()), ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return state["G"]
    acc = state["acc"]
    acc.resetAccumulation()
    if case["kind"] == "sp":
        for sign, config, M in zip(signs, configs, Ms):
            acc.accumulate(M, config, sign)
        acc.finalize()
        out = [acc.get_sign_times_M_r_w()]
        if case["squares"]:
            out.append(acc.get_sign_times_M_r_w_sqr())
        return out
    if case["precision"] == "fp64":
        for sign, config, M in zip(signs, configs, Ms):
            acc.accumulate(M, config, sign)
    else:
        for c in range(0, len(signs), case["batch"]):
            acc.accumulate_batch(Ms[c:c + case["batch"]], configs[c:c + case["batch"]], signs[c:c + case["batch"]])
    if case["read"] == "finalize":
        acc.finalize()
        return acc.get_G4()
    for channel, out in enumerate(state["out"]):
        acc.peek_G4_async(channel, 0, out.numpy())
    return state["out"]


# ---------------------------------------------------------------------------------------------
# Work and tolerances
# ---------------------------------------------------------------------------------------------
def work(case):
    """M and the vertices in, the result out; the per-orbital NDFTs, the cluster transforms as FFTs,
    the G0 products, and per G4 entry the products of its channel (both spins)."""
    nc, nb = _SITES[case["cluster"]], _bands(case)
    lo, hi = case["lo"], case["hi"]
    n1 = (lo + hi) / 2
    n2 = n1 * n1 + ((hi - lo + 1) ** 2 - 1) / 12
    count = case.get("count", 1)
    read = 2 * count * (8 * n2 + 24 * n1)
    if case["kind"] == "sp":
        sets = 2 if case["squares"] else 1
        out = sets * (2 * nb) ** 2 * nc * 2 * case["n_sp"] * 16
        # 16 taps of four table entries for every pair of vertices, then one FFT per label.
        padded = 8 * case["n_sp"]
        return {"bytes": read + out,
                "flops": 2 * count * n2 * 16 * (6 + 2 * sets) + sets * 2 * nb * nb * nc * 5 * padded * math.log2(padded)}
    ext = case["wex"] if case["kind"] == "tp" else 0
    nwe = case["nw"] + 2 * ext
    D = nb * nc * nwe
    fft = 5 * math.log2(nc)
    per_spin = 4 * nwe * n2 + fft * D * n1 + 8 * D * nwe * n1 + fft * D * D + (14 if nb == 1 else 16 * nb) * D * D
    flops = 2 * count * per_spin
    if case["kind"] == "g":
        return {"bytes": read + 2 * D * D * 16, "flops": flops}
    per = {W.PH_TRANSVERSE: 16, W.PH_MAGNETIC: 24, W.PH_CHARGE: 24, W.PP_UP_DOWN: 16}
    entries = nb ** 4 * nc ** 2 * case["nw"] ** 2 * (nc if case["q"] == "all" else 1) * (ext + 1)
    flops += count * entries * sum(per[c] for c in _CHANNELS[case["channels"]])
    return {"bytes": read + 16 * entries * len(_CHANNELS[case["channels"]]), "flops": flops}


def tolerance(case):
    if case["kind"] == "tp" and case["precision"] == "mixed":
        return {"rel": 2.5e-6, "max": 1e-4}  # G in 32 bits, its products summed in 32 bits over a batch
    if case["kind"] == "sp":
        return {"rel": 1e-12, "max": 1e-10}
    return {"rel": 1e-13, "max": 1e-11}


# ---------------------------------------------------------------------------------------------
# The results in 64 bits, by definition
# ---------------------------------------------------------------------------------------------
def _exact_sp(case, signs, configs, Ms):
    """M(r, w) = 1 / Nc sum over pairs of a label of sign M_ij e^{i w (tau_i - tau_j)}."""
    cl = _cluster(case["cluster"])
    nc, nb, n_sp = _SITES[case["cluster"]], _bands(case), case["n_sp"]
    device = _device()
    w = torch.from_numpy(W.matsubara(case["beta"], n_sp)).to(device)[n_sp:]
    r_of = np.zeros((nc, nc), np.int64)  # [r_j, r_i] -> index of r_i - r_j
    for rj in range(nc):
        for ri in range(nc):
            r_of[rj, ri] = cl.r_sub[rj, ri]
    results = []
    for power in range(1, 3 if case["squares"] else 2):
        out = torch.zeros(2 * n_sp, nc, 2, nb, 2, nb, dtype=torch.complex128, device=device)
        for spin in range(2):
            S = torch.zeros(n_sp, nb * nc, nb * nc, dtype=torch.complex128, device=device)
            for sign, config, M in zip(signs, configs, Ms):
                c = config[spin]
                if not c.n:
                    continue
                orb = torch.from_numpy(c.right_band.astype(np.int64) + nb * c.right_site).to(device)
                T = torch.exp(1j * torch.outer(w, torch.from_numpy(c.tau).to(device)))
                onehot = torch.nn.functional.one_hot(orb, nb * nc).t().to(torch.complex128)
                Mc = (sign * M[spin] ** power).to(torch.complex128)
                step = max(1, int(1e9 // (16 * c.n * nb * nc)))
                for a in range(0, n_sp, step):
                    B = onehot[None] * T[a:a + step, None, :]
                    S[a:a + step] += B @ Mc @ B.conj().transpose(1, 2)
            S = S.reshape(n_sp, nc, nb, nc, nb)  # r_i, b_i, r_j, b_j
            for ri in range(nc):
                for rj in range(nc):
                    r = int(r_of[rj, ri])
                    part = S[:, ri, :, rj, :].transpose(1, 2) / nc  # [w, b_j, b_i]
                    out[n_sp:, r, spin, :, spin, :] += part
                    out[:n_sp, r, spin, :, spin, :] += part.conj().flip(0)
        results.append(out.reshape(-1))
    return results


def _exact_g(case, config, M, spin, nwe):
    """G(w1 k1 b1; w2 k2 b2) = -G0 M~ G0 + beta G0 delta of one spin, as a (D, D) matrix."""
    cl = _cluster(case["cluster"])
    nc, nb = _SITES[case["cluster"]], _bands(case)
    device = _device()
    half = nwe // 2
    n_sp = _workload(case).n_sp
    g0 = torch.from_numpy(_g0(case["cluster"], case["model"], case["beta"], n_sp)).to(device)
    g0 = g0[n_sp - half:n_sp + half, :, spin, :, spin, :].transpose(2, 3)  # [w, k, b1, b2]
    D = nwe * nc * nb
    G0 = torch.zeros(nwe * nc, nb, nwe * nc, nb, dtype=torch.complex128, device=device)
    at = torch.arange(nwe * nc, device=device)
    G0[at, :, at, :] = g0.reshape(nwe * nc, nb, nb)
    G = case["beta"] * G0.reshape(D, D)
    if config.n:
        w = torch.from_numpy(W.matsubara(case["beta"], half)).to(device)
        k = torch.from_numpy(cl.k_vecs).to(device)
        a = torch.from_numpy(W.Model(**_MODELS[case["model"]]).a_vecs()).to(device)
        band = torch.from_numpy(config.right_band.astype(np.int64)).to(device)
        pos = torch.from_numpy(cl.r_vecs).to(device)[torch.from_numpy(config.right_site.astype(np.int64)).to(device)]
        A = torch.exp(1j * ((w[:, None] * torch.from_numpy(config.tau).to(device))[:, None, :]
                            + (k @ (pos + a[band]).t())[None]))  # [w, k, i]
        # G0(b1, b_i) e^{...} on the left, its counterpart on the right.
        P = torch.einsum("wkbi,wki->wkbi", g0[:, :, :, band], A).reshape(D, -1)
        Q = torch.einsum("wkib,wki->wkbi", g0[:, :, band, :], A.conj()).reshape(D, -1)
        G = G - (P @ M.to(torch.complex128)) @ Q.t() / nc
    return G


def _exact_g4(case, signs, configs, Ms):
    p = _tp_parameters(case)
    nc, nb, nw, ext = p.n_sites, p.n_bands, case["nw"], case["wex"]
    nwe = nw + 2 * ext
    device = _device()
    add = torch.from_numpy(np.asarray(p.k_add, np.int64)).to(device)
    sub = torch.from_numpy(np.asarray(p.k_sub, np.int64)).to(device)
    X = nw * nc
    kk = torch.arange(nc, device=device).repeat(nw)  # compact index x = (w, k), k fastest
    ww = torch.arange(nw, device=device).repeat_interleave(nc)
    out = [torch.zeros(len(p.w_ex), len(p.k_ex), X, X, nb, nb, nb, nb, dtype=torch.complex128, device=device)
           for _ in p.channels]  # [wq, q, (w2 k2), (w1 k1), b4, b3, b2, b1]
    chunk = max(1, int(4e9 // (2 * 16 * (nwe * nc * nb) ** 2)))
    for c in range(0, len(signs), chunk):
        m = range(c, min(len(signs), c + chunk))
        # Gs[s][m, x_left, x_right, a, b] = G_(a, b; ...); the formulas' G(b1, b2) is its band transpose.
        Gs = [torch.stack([_exact_g(case, configs[i][s], Ms[i][s], s, nwe) for i in m])
              .reshape(len(m), nwe * nc, nb, nwe * nc, nb).permute(0, 1, 3, 2, 4) for s in range(2)]
        empty = torch.tensor([configs[i][0].n + configs[i][1].n == 0 for i in m], device=device)
        sg = 0.5 * torch.tensor([float(signs[i]) for i in m], dtype=torch.float64, device=device)
        sg = torch.where(empty, torch.zeros_like(sg), sg)

        def pick(G, left, right):  # [m, len(left), len(right), a, b]
            return G[:, left][:, :, right]

        x = kk + nc * (ww + ext)
        for iq, q in enumerate(p.k_ex):
            for iw, wq in enumerate(p.w_ex):
                y = add[kk, q] + nc * (ww + ext + wq)
                z = sub[kk, q] + nc * (wq + nw - 1 - ww + ext)

                def direct(F, H, scale, eq):  # sum over m of F[m, x1, x2] H[m, x1, x2] over bands
                    if nb == 1:
                        return (scale[:, None, None] * F[..., 0, 0] * H[..., 0, 0]).sum(0).t()[
                            ..., None, None, None, None]
                    return torch.einsum("m,mxy%s,mxy%s->yx%s" % eq, scale.to(F.dtype), F, H)

                def disc(F, H, eq):  # F[m, x1], H[m, x2] over bands
                    return torch.einsum("m,mx%s,my%s->yx%s" % eq, sg.to(F.dtype), F, H)

                at = torch.arange(X, device=device)
                for ic, ch in enumerate(p.channels):
                    acc = out[ic][iw, iq]
                    if ch in (W.PH_MAGNETIC, W.PH_CHARGE):
                        f = -1.0 if ch == W.PH_MAGNETIC else 1.0
                        # G(k1, k1 + q)(b2, b1) and G(k2 + q, k2)(b3, b4), stored band-transposed.
                        L = Gs[0][:, x[at], y[at]] + f * Gs[1][:, x[at], y[at]]  # [m, x1, b1, b2]
                        R = Gs[0][:, y[at], x[at]] + f * Gs[1][:, y[at], x[at]]  # [m, x2, b4, b3]
                        acc += disc(L, R, ("ab", "dc", "dcba"))
                    for s in range(2):
                        F = pick(Gs[s], x, x)
                        if ch == W.PH_TRANSVERSE:
                            H = pick(Gs[1 - s], y, y).transpose(1, 2)
                            acc += direct(F, H, -sg, ("db", "ac", "dcba"))
                        elif ch == W.PH_MAGNETIC:
                            H = pick(Gs[s], y, y).transpose(1, 2)
                            acc += direct(F, H, -sg, ("ac", "db", "dcba"))
                        elif ch == W.PH_CHARGE:
                            H = pick(Gs[s], y, y).transpose(1, 2)
                            acc += direct(F, H, -sg, ("da", "cb", "dcba"))
                        else:
                            H = pick(Gs[1 - s], z, z)
                            acc += direct(F, H, sg, ("ca", "db", "dcba"))
        del Gs
    return [o.reshape(-1) for o in out]


def exact(case, seed):
    """The definition's sums in 64 bits, in the layout of run's outputs."""
    signs, configs, Ms = _measurements(case, seed)
    if case["kind"] == "sp":
        return _exact_sp(case, signs, configs, Ms)
    if case["kind"] == "g":
        nw, nc = case["nw"], _SITES[case["cluster"]]
        D = nw * nc * _bands(case)
        R = D // nw
        # Blocks (w1, w2) of R x R entries.
        return torch.stack([_exact_g(case, configs[0][s], Ms[0][s], s, nw).reshape(nw, R, nw, R).permute(0, 2, 1, 3)
                            .reshape(D, D) for s in range(2)])
    return _exact_g4(case, signs, configs, Ms)
