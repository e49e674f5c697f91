"""Performance cases of the library: what its users call, over the range of sizes.

Every case goes through a device entry point of hsspack_gb300 with its inputs in HBM.
A case carries the configuration (hsspack_gb300.set_config) that its program would set
once; entries that it does not name keep the library's defaults.  Entry points that
overwrite an input get a fresh copy of it in every pass.

listed()  the cases, with what each stands for
draw      one more case of the same ranges
prepare   inputs on the GPU, from a seed
run       one pass
work      bytes and operations that a pass cannot do without
exact     the results in 64 bits from torch / numpy alone (singular and eigenvectors have
          no value there: their signs are free)
"""
import math

import numpy as np
import torch

import hsspack_gb300 as hp

# the configuration entries a case may name
OPTIONS = ("precision", "predictor", "smlsiz", "split_min_m")
DEFAULT = hp.get_config()


def listed():
    return [
        # a small tridiagonal with the library's defaults (FP64 products, standard
        # secular start): launches and latency are all there is
        {"name": "tridiagonal_257", "kind": "tridiagonal", "n": 257},
        # the second half of a dense symmetric eigensolver, DSYTRD + DORGTR before it:
        # COMPZ = 'V', defaults, FP64 products
        {"name": "tridiagonal_v_2048", "kind": "tridiagonal_v", "n": 2048},
        # the reference's test matrix D = 2, E = 1 (TEST/Testedc.f90) with a little
        # disorder: extended eigenvectors, almost nothing deflates, the largest merges
        # go through HSS
        {"name": "tridiagonal_chain_3000", "kind": "chain", "n": 3000, "precision": 1,
         "predictor": 2},
        # the benchmark's tridiagonal under its tuned configuration: localized
        # eigenvectors, small merges, 8.6 GB of output
        {"name": "tridiagonal_32768", "kind": "tridiagonal", "n": 32768, "precision": 1,
         "predictor": 2, "smlsiz": 12},
        # the benchmark's uneven batch: 512 problems in one call
        {"name": "tridiagonal_batch_512", "kind": "batch", "count": 512, "lo": 256, "hi": 4096,
         "precision": 1, "predictor": 3, "smlsiz": 16, "split_min_m": 64},
        # bidiagonal SVD of an ordinary odd size with the defaults, and the benchmark's
        {"name": "bidiagonal_svd_1001", "kind": "bidiagonal", "n": 1001},
        {"name": "bidiagonal_svd_16384", "kind": "bidiagonal", "n": 16384, "precision": 1,
         "predictor": 2},
        # symmetric band, the tests' and benchmark's bandwidth
        {"name": "band_16384_kd4", "kind": "band", "n": 16384, "kd": 4, "precision": 1},
        # banded SVD, the reference's test case (TEST/test_bdc1.f90)
        {"name": "banded_svd_5000_sb5", "kind": "banded_svd", "n": 5000, "sb": 5, "smlsiz_arg": 75,
         "precision": 1, "predictor": 2},
        # Cauchy-like matrix in HSS form times a dense one, on the reference's
        # interlacing grid (TEST/testCauchyHss_serial.f90)
        {"name": "cauchy_hss_3000", "kind": "cauchy", "n": 3000, "ncb": 3000, "ni": 128,
         "tol": 1e-14, "precision": 1},
        # dense matrix to HSS form and its product: the reference's FMM test
        # (TEST/testfmm.f90)
        {"name": "dhssmm_2000", "kind": "dhssmm", "n": 2000, "ncb": 2000, "ni": 64, "tol": 1e-11,
         "precision": 1},
        # HSS Cholesky of a kernel matrix, factored and solved for several right-hand
        # sides, as a preconditioner is set up
        {"name": "hss_cholesky_8192", "kind": "cholesky", "n": 8192, "nrhs": 16, "ni": 32,
         "tol": 1e-8, "prank": 20},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    fast = rng.choice([{}, {"precision": 1, "predictor": 2}])
    kind = rng.choice(["tridiagonal", "tridiagonal", "tridiagonal_v", "chain", "batch",
                       "bidiagonal", "bidiagonal", "band", "banded_svd", "cauchy", "dhssmm",
                       "cholesky"])
    c = {"kind": kind}
    if kind == "tridiagonal":
        c.update(n=_log(rng, 100, 32768), **fast)
        if fast and rng.random() < 0.5:
            c["smlsiz"] = rng.choice([8, 12, 16])
    elif kind == "tridiagonal_v":
        c.update(n=_log(rng, 300, 4096), **fast)
    elif kind == "chain":
        c.update(n=_log(rng, 400, 3000), **fast)
    elif kind == "batch":
        c.update(count=_log(rng, 8, 256), lo=256, hi=4096, precision=1,
                 predictor=rng.choice([2, 3]), smlsiz=rng.choice([8, 12, 16]),
                 split_min_m=rng.choice([0, 64]))
    elif kind == "bidiagonal":
        c.update(n=_log(rng, 300, 16384), **fast)
    elif kind == "band":
        c.update(n=_log(rng, 300, 8192), kd=rng.choice([2, 3, 4, 8]), **fast)
    elif kind == "banded_svd":
        c.update(n=_log(rng, 500, 5000), sb=rng.randint(2, 5), smlsiz_arg=rng.choice([25, 75]),
                 precision=1, predictor=2)
    elif kind == "cauchy":
        n = _log(rng, 1000, 3000)
        c.update(n=n, ncb=_log(rng, 64, n), ni=rng.choice([64, 128]), tol=1e-14,
                 precision=rng.choice([0, 1]))
    elif kind == "dhssmm":
        n = _log(rng, 700, 2000)
        c.update(n=n, ncb=_log(rng, 5, n), ni=rng.choice([50, 64, 96]), tol=1e-11,
                 precision=rng.choice([0, 1]))
    else:
        c.update(n=_log(rng, 1000, 8192), nrhs=rng.randint(1, 16), ni=32, tol=1e-8, prank=20)
    return c


def _configure(case):
    hp.restore_config(DEFAULT)
    hp.set_config(**{k: case[k] for k in OPTIONS if k in case})


def _uniform(gen, lo, hi, *shape):
    return torch.rand(*shape, dtype=torch.float64, device="cuda", generator=gen) * (hi - lo) + lo


def _sizes(case, seed):
    rng = np.random.default_rng(seed)
    return np.round(np.exp(rng.uniform(math.log(case["lo"]), math.log(case["hi"]),
                                       case["count"]))).astype(np.int32)


def _grid(n):
    """The interlacing grid of TEST/testCauchyHss_serial.f90: column poles F, row poles D."""
    gap = 8.9 / (2 * n)
    f = 0.1 + gap * (2.0 * torch.arange(1, n + 1, dtype=torch.float64, device="cuda") - 1.0)
    return f, f + gap


def _inputs(case, seed):
    """The case's matrices and vectors on the GPU, by name."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("tridiagonal", "tridiagonal_v"):
        x = {"d": _uniform(g, -1.0, 1.0, n), "e": _uniform(g, -1.0, 1.0, n)}
        if kind == "tridiagonal_v":
            # an orthogonal matrix as a reduction leaves it, column-major
            x["q"] = torch.linalg.qr(torch.randn(n, n, dtype=torch.float64, device="cuda",
                                                 generator=g))[0].contiguous()
        return x
    if kind == "chain":
        return {"d": 2.0 + _uniform(g, -1e-3, 1e-3, n), "e": 1.0 + _uniform(g, -1e-3, 1e-3, n)}
    if kind == "batch":
        # the sizes are the workload's own, the same for every seed
        sizes = _sizes(case, 2)
        total = int(sizes.sum())
        return {"sizes": sizes, "d": _uniform(g, -1.0, 1.0, total),
                "e": _uniform(g, -1.0, 1.0, total)}
    if kind == "bidiagonal":
        return {"d": 1.0 - _uniform(g, 0.0, 1.0, n), "e": 1.0 - _uniform(g, 0.0, 1.0, n)}
    if kind == "band":
        return {"ab": _uniform(g, -1.0, 1.0, n, case["kd"] + 1)}
    if kind == "banded_svd":
        return {"ab": _uniform(g, 0.0, 1.0, n, case["sb"] + 1)}
    if kind == "cauchy":
        f, d = _grid(n)
        u, v = (torch.randn(n, dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
        b = torch.randn(case["ncb"], n, dtype=torch.float64, device="cuda", generator=g)
        return {"d": d, "f": f, "u": u, "v": v, "b": b}
    if kind == "dhssmm":
        f, d = _grid(n)
        z, v = _uniform(g, 0.0, 1.0, n), _uniform(g, 0.0, 1.0, n)
        # A_ij = z_i v_j / (f_i - d_j), column-major
        a = ((z[:, None] * v[None, :]) / (f[:, None] - d[None, :])).T.contiguous()
        return {"a": a, "b": _uniform(g, 0.0, 1.0, case["ncb"], n)}
    x = torch.sort(_uniform(g, 0.0, 1.0, n))[0]
    a = torch.exp(-0.5 * ((x[:, None] - x[None, :]) / 0.01) ** 2)
    a.diagonal().add_(1e-2)
    b = torch.randn(case["nrhs"], n, dtype=torch.float64, device="cuda", generator=g)
    return {"a": a, "b": b}


def prepare(case, seed):
    _configure(case)
    x = _inputs(case, seed)
    kind, n = case["kind"], case.get("n", 0)

    def new(count):
        return torch.empty(count, dtype=torch.float64, device="cuda")

    if kind in ("tridiagonal", "chain"):
        x["z"] = new(n * n)
    elif kind == "batch":
        x["z"] = new(int((x["sizes"].astype(np.int64) ** 2).sum()))
    elif kind in ("bidiagonal", "banded_svd"):
        x.update(s=new(n), uo=new(n * n), vo=new(n * n))
    elif kind == "band":
        x.update(w=new(n), z=new(n * n))
    return {"case": case, **x}


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind in ("tridiagonal", "chain"):
        w = s["d"].clone()
        hp.mdstedc_dev(w, s["e"], s["z"])
        return w, s["z"]
    if kind == "tridiagonal_v":
        w, q = s["d"].clone(), s["q"].clone()
        hp.mdstedc_v_dev(w, s["e"], q)
        return w, q
    if kind == "batch":
        w = s["d"].clone()
        hp.mdstedc_batch_dev(s["sizes"], w, s["e"], s["z"])
        return w, s["z"]
    if kind == "bidiagonal":
        w = s["d"].clone()
        hp.mdbdsdc_dev(w, s["e"], s["uo"], s["vo"])
        return w, s["uo"], s["vo"]
    if kind == "band":
        hp.mdsbevd_dev(case["kd"], s["ab"], s["w"], s["z"])
        return s["w"], s["z"]
    if kind == "banded_svd":
        hp.mdbdsvd_dev(case["sb"], s["ab"], s["s"], s["uo"], s["vo"], smlsiz=case["smlsiz_arg"])
        return s["s"], s["uo"], s["vo"]
    if kind == "cauchy":
        b = s["b"].clone()
        hp.cauchyhssmm_dev(s["d"], s["f"], s["u"], s["v"], b, case["ni"], case["tol"])
        return b
    if kind == "dhssmm":
        b = s["b"].clone()
        hp.dhssmm_dev(s["a"], b, case["ni"], case["tol"])
        return b
    b = s["b"].clone()
    f = hp.HssChol(s["a"], case["ni"], case["tol"], case["prank"])
    f.solve(b)
    f.free()
    return b


def work(case):
    kind, n = case["kind"], float(case.get("n", 0))
    if kind in ("tridiagonal", "chain"):
        return {"bytes": 8.0 * (n * n + 3 * n), "flops": 4.0 * n * n}
    if kind == "tridiagonal_v":
        # Q0 in, the product out
        return {"bytes": 8.0 * (2 * n * n + 3 * n), "flops": 4.0 * n * n}
    if kind == "batch":
        z = _sizes(case, 2).astype(np.float64)
        nn = float((z * z).sum())
        return {"bytes": 8.0 * (nn + 3 * float(z.sum())), "flops": 4.0 * nn}
    if kind == "bidiagonal":
        return {"bytes": 8.0 * (2 * n * n + 3 * n), "flops": 8.0 * n * n}
    if kind == "band":
        kd = case["kd"]
        return {"bytes": 8.0 * (n * n + (kd + 2) * n), "flops": 4.0 * n * n * kd}
    if kind == "banded_svd":
        sb = case["sb"]
        return {"bytes": 8.0 * (2 * n * n + (sb + 2) * n), "flops": 8.0 * n * n * sb}
    if kind == "cauchy":
        m = float(case["ncb"])
        return {"bytes": 8.0 * (2 * n * m + 4 * n), "flops": 2.0 * n * m * case["ni"]}
    if kind == "dhssmm":
        m = float(case["ncb"])
        return {"bytes": 8.0 * (n * n + 2 * n * m), "flops": 2.0 * n * m * case["ni"]}
    return {"bytes": 8.0 * (n * n + 2 * n * case["nrhs"]),
            "flops": n * case["ni"] ** 2 + 4.0 * n * case["ni"] * case["nrhs"]}


def exact(case, seed):
    kind, n = case["kind"], case.get("n", 0)
    if kind == "batch" or (kind in ("tridiagonal", "bidiagonal", "band") and n > 4096):
        return None  # dense solvers would take too long
    x = _inputs(case, seed)
    if kind in ("tridiagonal", "tridiagonal_v", "chain"):
        e = x["e"][:n - 1]
        t = torch.diag(x["d"]) + torch.diag(e, 1) + torch.diag(e, -1)
        return torch.linalg.eigvalsh(t), None
    if kind == "bidiagonal":
        a = torch.diag(x["d"]) + torch.diag(x["e"][:n - 1], 1)
        return torch.from_numpy(np.linalg.svd(a.cpu().numpy(), compute_uv=False)), None, None
    if kind in ("band", "banded_svd"):
        # x["ab"][j, k + i - j] = A(i, j), j - k <= i <= j
        k = x["ab"].shape[1] - 1
        a = torch.diag(x["ab"][:, k])
        for o in range(1, k + 1):
            a += torch.diag(x["ab"][o:, k - o], o)
        if kind == "banded_svd":
            return torch.from_numpy(np.linalg.svd(a.cpu().numpy(), compute_uv=False)), None, None
        return torch.linalg.eigvalsh(a, UPLO="U"), None
    if kind == "cauchy":
        c = x["u"][:, None] * x["v"][None, :] / (x["d"][:, None] - x["f"][None, :])
        return x["b"] @ c.T
    if kind == "dhssmm":
        return x["b"] @ x["a"]
    return torch.linalg.solve(x["a"], x["b"].T).T.contiguous()
