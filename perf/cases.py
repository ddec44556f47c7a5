"""Timed cases of the KDE / VKDE proposal path, each through the Python mirror of the C-ABI.

What an ensemble sampler does with this library on every half-move: it hands over the
walkers of one half (`set_sample`), prepares the density estimate or fits its weights
(`prepare`, `prepare_interp`), draws proposals (`sample`) and evaluates -2 ln p at proposals
and walkers (`eval_m2lnp`).  The cases time those calls one by one and one whole half-move.

A case is a dict of plain values:
  op         eval | prepare | fit | step
  kind       kde | vkde              kernel  gauss | st (Student-t, nu = 3)
  dim, n, m  dimension, sample size, points evaluated
  precision  fp64 | mixed            where   host | device (the points' memory)
  data       gauss | banana | gmm    cov     sample | robust_diag | robust
  cv         none | split_nofit
"""
from __future__ import annotations

import math

import numpy as np
import torch

from numcosmo_gb300 import (Precision, StatsDistCV, StatsDistKDE, StatsDistKDECovType, StatsDistKernelGauss,
                            StatsDistKernelST, StatsDistVKDE)

NU = 3.0
LOCAL_FRAC = 0.05
_BASE = {"kind": "vkde", "kernel": "st", "precision": "fp64", "where": "host", "data": "gauss", "cov": "sample",
         "cv": "none", "m": 0}


def _case(name: str, op: str, **kw) -> dict:
    return {"name": name, "op": op, **_BASE, **kw}


def listed() -> list[dict]:
    return [
        # one walker's density, the reference's per-walker call: all latency
        _case("point_kde_gauss_d4", "eval", kind="kde", kernel="gauss", dim=4, n=1000, m=1),
        # the plain Gaussian KDE at its benchmark size, FP64 as a new handle has it
        _case("eval_kde_gauss_d4", "eval", kind="kde", kernel="gauss", dim=4, n=1000, m=1000),
        # the headline size in the default precision: a curved posterior, heavy-tailed kernels
        _case("eval_vkde_st_d16", "eval", dim=16, n=8192, m=8192, data="banana"),
        # many parameters, a ragged ensemble
        _case("eval_vkde_gauss_d27", "eval", kernel="gauss", dim=27, n=3001, m=5003),
        # the headline size in the mixed form, points resident on the device
        _case("eval_mixed_vkde_st_d16", "eval", dim=16, n=8192, m=8192, data="banana", precision="mixed",
              where="device"),
        # a long chain's points against one ensemble, fixed-shape kernels, mixed form
        _case("eval_mixed_kde_st_d11", "eval", kind="kde", dim=11, n=5000, m=20011, precision="mixed"),
        # the density of one half of a large ensemble: neighbours, local covariances, factors
        _case("prepare_vkde_st_d16", "prepare", dim=16, n=8192, m=256, data="banana"),
        # bandwidth by the held-out half, fixed-shape kernels
        _case("prepare_kde_split_d6", "prepare", kind="kde", dim=6, n=2000, m=100, cv="split_nofit"),
        # outlier-resistant local covariances
        _case("prepare_vkde_robust_d8", "prepare", dim=8, n=2048, m=64, cov="robust"),
        # the weight fit in the default precision
        _case("fit_vkde_gauss_d12", "fit", kernel="gauss", dim=12, n=2048, data="gmm"),
        # the weight fit at its benchmark size, mixed form
        _case("fit_mixed_vkde_gauss_d12", "fit", kernel="gauss", dim=12, n=4096, data="gmm", precision="mixed"),
        # a whole half-move of a small ensemble: fit, proposals, densities at proposals and walkers
        _case("step_mixed_vkde_st_d8", "step", dim=8, n=512, precision="mixed"),
    ]


def _log_int(rng, lo: int, hi: int) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _vkde_min_n(dim: int) -> int:
    """Ensembles large enough that the neighbourhoods (5 %) determine a covariance."""
    return max(64, 60 * dim)


def draw(rng) -> dict:
    op = rng.choices(["eval", "prepare", "fit", "step"], [8, 4, 3, 2])[0]
    c = dict(_BASE, op=op)
    c["kernel"] = rng.choice(["gauss", "st"])
    c["kind"] = rng.choice(["kde", "vkde"]) if op in ("eval", "prepare") else "vkde"

    if op == "eval":
        c["dim"] = rng.randint(2, 32)
        lo = _vkde_min_n(c["dim"]) if c["kind"] == "vkde" else 64
        c["n"] = _log_int(rng, lo, 12000)
        # no more pair work than the largest listed eval
        cap = int(8192 * 8192 * (16 * 16 + 5 * 16) / (c["n"] * (c["dim"] ** 2 + 5 * c["dim"])))
        c["m"] = 1 if rng.random() < 0.1 else _log_int(rng, 16, max(17, min(20011, cap)))
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["where"] = rng.choice(["host", "device"])
        c["data"] = rng.choice(["gauss", "banana"])
    elif op == "prepare":
        c["dim"] = rng.randint(2, 24)
        lo = _vkde_min_n(c["dim"]) if c["kind"] == "vkde" else 64
        c["n"] = _log_int(rng, lo, 6000)
        c["m"] = rng.randint(16, 256)
        c["data"] = rng.choice(["gauss", "banana"])
        c["cov"] = rng.choices(["sample", "robust_diag", "robust"], [6, 1, 1])[0]
        if c["cov"] != "sample":
            c["n"] = min(c["n"], 2048)
        elif rng.random() < 0.25:
            c["cv"] = "split_nofit"
    else:
        c["dim"] = rng.randint(8, 20)
        c["n"] = _log_int(rng, _vkde_min_n(c["dim"]), 2600 if op == "fit" else 1500)
        c["precision"] = rng.choice(["fp64", "mixed"])
        c["data"] = rng.choice(["gauss", "gmm"]) if op == "fit" else "gauss"

    return c


# ---------------------------------------------------------------------------- inputs


def _spd(d: int, rng, cond: float = 100.0) -> np.ndarray:
    """Random orientation, eigenvalues log-spaced over `cond`."""
    q, _ = np.linalg.qr(rng.standard_normal((d, d)))
    s = (q * np.logspace(0.0, math.log10(cond), d)) @ q.T
    return 0.5 * (s + s.T)


def _inputs(case: dict, seed: int) -> dict:
    """Sample, evaluation points, target -2 ln L at the sample and replay draws, all float64 numpy."""
    rng = np.random.default_rng([int(seed), 20])
    d, n, m = case["dim"], case["n"], case["m"]
    if case["data"] == "banana":
        def law(k):
            x = rng.standard_normal((k, d))
            x[:, 0] *= 10.0
            x[:, 1] += 0.1 * (x[:, 0] ** 2 - 100.0)
            return x
        X, P, m2 = law(n), law(m), None
    elif case["data"] == "gmm":
        wts, covs = np.array([0.5, 0.3, 0.2]), [_spd(d, rng) for _ in range(3)]
        sig = max(math.sqrt(np.max(np.diag(c))) for c in covs)
        mus = [np.zeros(d), np.zeros(d), np.zeros(d)]
        mus[1][0], mus[2][1] = 3.0 * sig, 3.0 * sig
        ls = [np.linalg.cholesky(c) for c in covs]
        comp = rng.choice(3, size=n, p=wts)
        z = rng.standard_normal((n, d))
        X = np.empty((n, d))
        for k in range(3):
            X[comp == k] = mus[k] + z[comp == k] @ ls[k].T
        t = np.array([math.log(wts[k]) - 0.5 * (np.sum(np.linalg.solve(ls[k], (X - mus[k]).T) ** 2, axis=0)
                                                + 2.0 * np.sum(np.log(np.diag(ls[k]))) + d * math.log(2 * math.pi))
                      for k in range(3)])
        top = t.max(axis=0)
        m2 = -2.0 * (top + np.log(np.exp(t - top).sum(axis=0)))
        P = np.empty((0, d))
    else:
        L = np.linalg.cholesky(_spd(d, rng))
        # walkers of a chain that has not quite settled are a little wider than the target
        X, P = 1.2 * rng.standard_normal((n, d)) @ L.T, rng.standard_normal((m, d)) @ L.T
        m2 = np.sum(np.linalg.solve(L, X.T) ** 2, axis=0)
    out = {"X": np.ascontiguousarray(X), "P": np.ascontiguousarray(P), "m2lnL": m2}
    if case["op"] == "step":
        out["W"] = np.ascontiguousarray(1.2 * rng.standard_normal((n, d)) @ L.T)  # the other half's walkers
        out["u"], out["z"] = rng.random(n), rng.standard_normal((n, d))
        out["chisq"] = rng.chisquare(NU, n) if case["kernel"] == "st" else None
    return out


def _handle(case: dict):
    kernel = StatsDistKernelST(case["dim"], NU) if case["kernel"] == "st" else StatsDistKernelGauss(case["dim"])
    cv = StatsDistCV.SPLIT_NOFIT if case["cv"] == "split_nofit" else StatsDistCV.NONE
    sd = (StatsDistVKDE if case["kind"] == "vkde" else StatsDistKDE)(kernel, cv)
    sd.set_precision(Precision.MIXED if case["precision"] == "mixed" else Precision.FP64)
    sd.set_cov_type({"sample": StatsDistKDECovType.SAMPLE, "robust_diag": StatsDistKDECovType.ROBUST_DIAG,
                     "robust": StatsDistKDECovType.ROBUST}[case["cov"]])
    if case["kind"] == "vkde":
        sd.set_local_frac(LOCAL_FRAC)
    return sd


_stream = None


def _program_stream():
    """The one stream that a program with device-resident points works on."""
    global _stream
    if _stream is None:
        _stream = torch.cuda.Stream()
    return _stream


def prepare(case: dict, seed: int) -> dict:
    s = {"case": case, "sd": _handle(case), **_inputs(case, seed)}
    if case["op"] == "eval":
        if case["where"] == "device":
            s["sd"].set_stream(_program_stream().cuda_stream)
            s["dP"] = torch.from_numpy(s["P"]).cuda()
            s["out"] = torch.empty(case["m"], dtype=torch.float64, device="cuda")
            torch.cuda.synchronize()
        s["sd"].set_sample(s["X"])
        s["sd"].prepare()
    return s


def run(s: dict):
    case, sd = s["case"], s["sd"]
    op = case["op"]
    if op == "eval":
        if case["where"] == "device":
            sd.eval_m2lnp_device(s["dP"].data_ptr(), case["m"], s["out"].data_ptr())
            return s["out"]
        return sd.eval_m2lnp(s["P"][0]) if case["m"] == 1 else sd.eval_m2lnp(s["P"])
    sd.set_sample(s["X"])
    if op == "prepare":
        if case["cv"] != "none":
            sd.set_over_smooth(1.0)  # the fit leaves its bandwidth in the handle
        sd.prepare()
        return {"cov": sd.peek_full_cov(), "href": sd.get_href(), "m2lnp": sd.eval_m2lnp(s["P"])}
    sd.prepare_interp(s["m2lnL"])
    if op == "fit":
        return {"weights": sd.peek_weights(), "rnorm": sd.get_rnorm()}
    x, idx = sd.sample(s["u"], s["z"], s["chisq"])
    return {"weights": sd.peek_weights(), "x": x, "idx": idx, "m2lnp": sd.eval_m2lnp(np.concatenate([x, s["W"]]))}


# ---------------------------------------------------------------------------- work


def _eval_flops(case: dict, n: int, m: int) -> float:
    """Differences, triangular whitening and squared norm of a pair (VKDE) or difference and norm (KDE)."""
    d = case["dim"]
    return float(n) * m * ((d * d + 3 * d) if case["kind"] == "vkde" else 3 * d)


def _prepare_flops(case: dict) -> float:
    d, n = case["dim"], case["n"]
    f = float(n) * d * (d + 1) + n * d * d
    if case["kind"] == "vkde":
        f += float(n) * n * 3 * d + n * (LOCAL_FRAC * n) * d * (d + 1) + n * 2 * d ** 3 / 3
    return f


def work(case: dict) -> dict:
    d, n, m = case["dim"], case["n"], case["m"]
    vk = case["kind"] == "vkde"
    kernels = 8.0 * n * (d + (d * (d + 1) // 2 if vk else 0) + 1)
    if case["op"] == "eval":
        return {"bytes": kernels + 8.0 * m * (d + 1), "flops": _eval_flops(case, n, m)}
    if case["op"] == "prepare":
        f = _prepare_flops(case) + _eval_flops(case, n, m)
        if case["cv"] != "none":
            f += 20 * _eval_flops(case, n // 2, n - n // 2)  # a simplex fit takes about that many objectives
        return {"bytes": 8.0 * n * d + 8.0 * m * (d + 1), "flops": f}
    # the interpolation matrix, its normal matrix and at least one factorisation
    f = _prepare_flops(case) + _eval_flops(case, n, n) + float(n) ** 3 + float(n) ** 3 / 3
    if case["op"] == "fit":
        return {"bytes": 8.0 * n * (d + 2), "flops": f}
    return {"bytes": 8.0 * n * (4 * d + 6), "flops": f + _eval_flops(case, n, 2 * n)}


# ---------------------------------------------------------------------------- 64-bit values


def _lnnorm(case: dict, lndet: torch.Tensor) -> torch.Tensor:
    d = case["dim"]
    if case["kernel"] == "gauss":
        return 0.5 * (d * math.log(2 * math.pi) + lndet)
    return (math.lgamma(0.5 * NU) - math.lgamma(0.5 * (NU + d))) + 0.5 * d * math.log(math.pi * NU) + 0.5 * lndet


def _rot_bandwidth(case: dict, n: int) -> float:
    d = case["dim"]
    if case["kernel"] == "gauss":
        return (4.0 / (n * (d + 2.0))) ** (1.0 / (d + 4.0))
    v = max(NU, 3.0)
    return (16.0 * (v - 2) ** 2 * (1 + d + v) * (3 + d + v)
            / ((2 + d) * (d + v) * (2 + d + v) * (d + 2 * v) * (2 + d + 2 * v) * n)) ** (1.0 / (d + 4.0))


def _exact_density(case: dict, X: torch.Tensor, P: torch.Tensor):
    """(global covariance, bandwidth, -2 ln p at P) of the unweighted estimate on the sample X."""
    d, n = case["dim"], X.shape[0]
    mid = X.mean(0)
    cov = (X - mid).T @ (X - mid) / (n - 1)
    low = torch.linalg.cholesky(cov)
    y = torch.linalg.solve_triangular(low, X.T, upper=False).T.contiguous()
    h = 1.0 if case["kind"] == "vkde" else _rot_bandwidth(case, n)
    if case["kind"] == "vkde":
        k = max(int(LOCAL_FRAC * n), 2)
        near = torch.empty((n, k), dtype=torch.int64, device=X.device)
        for i in range(0, n, 256):
            d2 = torch.zeros((min(256, n - i), n), dtype=torch.float64, device=X.device)
            for c in range(d):
                d2 += (y[i:i + 256, c, None] - y[None, :, c]) ** 2
            near[i:i + 256] = torch.topk(d2, k, dim=1, largest=False).indices
        loc = torch.empty((n, d, d), dtype=torch.float64, device=X.device)
        for i in range(0, n, 512):
            z = X[near[i:i + 512]]
            z = z - z.mean(1, keepdim=True)
            loc[i:i + 512] = z.transpose(1, 2) @ z / (k - 1)
        factor = torch.linalg.cholesky(loc)
        lndet = 2.0 * torch.log(torch.diagonal(factor, dim1=1, dim2=2)).sum(1)
        whiten = torch.linalg.solve_triangular(factor, torch.eye(d, dtype=torch.float64, device=X.device).expand(n, d, d),
                                               upper=False)
    else:
        lndet = 2.0 * torch.log(torch.diagonal(low)).sum().expand(n)
        yp = torch.linalg.solve_triangular(low, P.T, upper=False).T.contiguous()
    c = -math.log(n) - _lnnorm(case, lndet) - d * math.log(h)
    lse = torch.full((P.shape[0],), -math.inf, dtype=torch.float64, device=X.device)
    step = max(1, (1 << 24) // max(1, P.shape[0] * d))
    for i in range(0, n, step):
        if case["kind"] == "vkde":
            chi2 = (((P[None] - X[i:i + step, None]) @ whiten[i:i + step].transpose(1, 2)) ** 2).sum(2)
        else:
            chi2 = ((yp[None] - y[i:i + step, None]) ** 2).sum(2)
        chi2 = chi2 / (h * h)
        lnk = -0.5 * chi2 if case["kernel"] == "gauss" else -0.5 * (NU + d) * torch.log1p(chi2 / NU)
        lse = torch.logaddexp(lse, torch.logsumexp(lnk + c[i:i + step, None], 0))
    return cov, h, -2.0 * lse


def exact(case: dict, seed: int):
    # a fitted bandwidth, robust covariances and fitted weights have no closed form
    if case["op"] not in ("eval", "prepare") or case["cov"] != "sample" or case["cv"] != "none":
        return None
    s = _inputs(case, seed)
    dev = "cuda" if torch.cuda.is_available() else "cpu"
    X, P = torch.from_numpy(s["X"]).to(dev), torch.from_numpy(s["P"]).to(dev)
    cov, h, m2 = _exact_density(case, X, P)
    if case["op"] == "prepare":
        return {"cov": cov.cpu().numpy(), "href": h, "m2lnp": m2.cpu().numpy()}
    return m2 if case["where"] == "device" else (float(m2[0]) if case["m"] == 1 else m2.cpu().numpy())
