"""Timed cases of the SVM engine: training, cross-validation, the request loop and prediction.

A case is a plain dict: what is called (`do`), the shape of the data, and the
options a caller sets.  Inputs are synthetic, made from a seed with the
distributions of the engine's own workloads (svmb200.datagen), as float32
numbers.  Training and prediction go through svm.h (svm_train,
svm_cross_validation, svm_predict_values) and the svmb_* C-ABI exactly as a
C program calls them: the svm_node rows or CSR arrays are in the caller's
memory before the call, the model or the coefficients after it.

The autotuner is off: it tries other launch shapes on a caller's first calls,
while a program that trains one model gets the fixed rules measured here.
"""
import ctypes as C
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "libsvm-cuda_b200"))

from svmb200 import cabi  # noqa: E402
from svmb200.lib import Engine, ServerConfig, SolveStats, make_params  # noqa: E402

FORMS = {"exact": 0, "fp32": 1, "bf16x3": 2, "fp16x3": 3, "tf32": 4}
KERNELS = {"linear": 0, "poly": 1, "rbf": 2, "sigmoid": 3}
SVMS = {"c_svc": 0, "nu_svc": 1, "one_class": 2, "eps_svr": 3, "nu_svr": 4}

_libc = C.CDLL(None)
_libc.malloc.restype = C.c_void_p
_libc.malloc.argtypes = [C.c_size_t]
_engine = None


def engine():
    global _engine
    if _engine is None:
        _engine = Engine()
        _engine.set_option("autotune", 0)
    return _engine


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _train(name, data, n, d, **more):
    c = dict(name=name, do="train", data=data, n=n, d=d, svm="c_svc", kernel="rbf", C=1.0, gamma=1.0 / d, form="exact")
    c.update(more)
    return {k: v for k, v in c.items() if k != "name" or v}


def listed():
    return [
        # one decision value at a time: a service that answers single rows with a loaded model
        dict(name="predict_one_row", do="predict_one", n=1, sv=1500, d=64, classes=2, form="exact", kernel="rbf", gamma=1.0 / 64),
        # the smallest training jobs of the request mix: 500 rows, 16 features
        _train("train_500x16", "gauss", 500, 16),
        # the plain binary workload: 4,000 x 64, C = 1, gamma = 1/64
        _train("train_4000x64", "gauss", 4000, 64),
        # the request mix's sparse nu-SVC with a cubic kernel, at an odd size
        _train("train_nu_poly_sparse_3001x512", "sparse", 3001, 512, nnz=40, svm="nu_svc", kernel="poly", gamma=1.0, nu=0.3),
        # epsilon-SVR: twice as many variables as rows
        _train("train_svr_2500x8", "regression", 2500, 8, svm="eps_svr", C=4.0),
        # model selection on a small multi-class problem: 5 folds x 3 pairs side by side
        dict(name="cv5_3class_1800x32", do="cv", data="classes", classes=3, n=1800, d=32, svm="c_svc", kernel="rbf", C=2.0,
             gamma=1.0 / 32, form="exact", folds=5),
        # rows of text: 20,000 features, about 40 nonzeros
        _train("train_text_6000x20000", "sparse", 6000, 20000, nnz=40, C=4.0, gamma=0.5),
        # the headline: 45 one-vs-one problems of 10 uneven classes (53,558 rows x 256)
        _train("train_ovo10_53558x256", "classes", 53558, 256, classes=10),
        # the pixel workload's shape on the tensor cores, rows resident on the device
        dict(name="solve_pixels_10000x784_fp16x3", do="solve", data="pixels", n=10000, d=784, svm="c_svc", kernel="rbf", C=10.0,
             gamma=1.0 / 784, form="fp16x3", cache_mb=400.0),
        # mixed jobs sent to the request loop together
        dict(name="serve_16_jobs", do="serve", jobs=16, n=500, n_hi=5000, d=16, d_hi=512, form="exact"),
        # a held-out set through a 10-class model, the reference's decision values bit for bit
        dict(name="predict_6000_rows_10class", do="predict", n=6000, sv=20000, d=256, classes=10, form="exact", kernel="rbf",
             gamma=1.0 / 256),
        # decision values of pixel rows as block products on the tensor cores
        dict(name="predict_10000_pixels_fp16x3", do="predict", n=10000, sv=30011, d=784, classes=2, form="fp16x3", kernel="rbf",
             gamma=1.0 / 784),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    what = rng.choice(["small", "dense", "dense", "sparse", "text", "svr", "classes", "cv", "pixels", "one", "predict", "serve"])
    if what in ("small", "dense"):
        n, d = (_log(rng, 500, 1500), rng.randint(9, 80)) if what == "small" else (_log(rng, 1500, 9000), _log(rng, 16, 300))
        svm, kernel = rng.choice([("c_svc", "rbf"), ("c_svc", "rbf"), ("nu_svc", "rbf"), ("c_svc", "poly")])
        return _train("", "gauss", n, d, svm=svm, kernel=kernel, C=rng.choice([0.5, 1.0, 4.0]), nu=0.3,
                      form=rng.choice(["exact", "exact", "fp32"]))
    if what == "sparse":
        svm, kernel = rng.choice([("c_svc", "rbf"), ("nu_svc", "poly"), ("c_svc", "poly")])
        return _train("", "sparse", _log(rng, 500, 5000), _log(rng, 64, 2000), nnz=rng.randint(10, 40), svm=svm, kernel=kernel,
                      gamma=1.0, nu=0.3)
    if what == "text":
        return _train("", "sparse", _log(rng, 2000, 7000), rng.randint(15000, 25000), nnz=rng.randint(20, 60), C=4.0, gamma=0.5)
    if what == "svr":
        return _train("", "regression", _log(rng, 400, 2500), rng.randint(4, 12), svm=rng.choice(["eps_svr", "nu_svr"]),
                      C=rng.choice([1.0, 4.0]), nu=0.4)
    if what == "classes":
        return _train("", "classes", _log(rng, 4000, 50000), rng.randint(60, 256), classes=rng.randint(3, 10))
    if what == "cv":
        return dict(do="cv", data="classes", classes=rng.randint(2, 4), n=_log(rng, 400, 2500), d=rng.randint(8, 64), svm="c_svc",
                    kernel="rbf", C=rng.choice([1.0, 2.0]), gamma=1.0 / 32, form="exact", folds=5)
    if what == "pixels":
        return dict(do="solve", data="pixels", n=_log(rng, 2000, 9000), d=rng.choice([196, 784, rng.randint(300, 800)]), svm="c_svc",
                    kernel="rbf", C=10.0, gamma=1.0 / 784, form=rng.choice(["fp16x3", "exact", "tf32"]),
                    cache_mb=rng.choice([100.0, 400.0]))
    if what == "one":
        return dict(do="predict_one", n=1, sv=_log(rng, 300, 5000), d=rng.randint(8, 300), classes=rng.randint(2, 4), form="exact",
                    kernel="rbf", gamma=1.0 / 64)
    if what == "predict":
        form = rng.choice(["exact", "exact", "fp16x3"])
        return dict(do="predict", n=_log(rng, 200, 8000), sv=_log(rng, 1000, 20000), d=_log(rng, 16, 784),
                    classes=rng.randint(2, 10), form=form, kernel=rng.choice(["rbf", "rbf", "poly"]), gamma=1.0 / 256)
    return dict(do="serve", jobs=rng.randint(6, 16), n=500, n_hi=_log(rng, 1500, 5000), d=16, d_hi=512, form="exact")


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _data(kind, n, d, seed, classes=2, nnz=40):
    """(X, y) with X a float32 matrix, or a CSR triple for sparse data."""
    if kind == "sparse":
        return _sparse(n, d, nnz, seed)
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*s):
        return torch.randn(*s, device="cuda", generator=g)

    def uniform(*s):
        return torch.rand(*s, device="cuda", generator=g)

    if kind == "gauss":
        y = torch.where(uniform(n) < 0.5, 1.0, -1.0)
        X = normal(n, d) + 0.5 * y[:, None]
        y = torch.where(uniform(n) < 0.05, -y, y)
    elif kind == "pixels":
        k = torch.floor(uniform(n, d) * 256) * (uniform(n, d) >= 0.7)
        X = k / 255
        s = torch.tanh((X - X.mean(0)) @ normal(d, 64) / math.sqrt(0.1 * d) + 0.1 * normal(64)) @ normal(64)
        y = torch.where(s >= s.median(), 1.0, -1.0)
        y = torch.where(uniform(n) < 0.1, -y, y)
    elif kind == "regression":
        X = normal(n, d)
        y = torch.sin(X @ normal(d) / math.sqrt(d)) + 0.5 * (X @ normal(d)) ** 2 / d + 0.1 * normal(n)
    else:   # classes of geometric sizes (ratio 0.8) around N(0, 4) centres
        share = torch.tensor([0.8 ** k for k in range(classes)], device="cuda")
        edge = torch.cumsum(share / share.sum() * n, 0).round().long()
        lab = torch.searchsorted(edge, torch.arange(n, device="cuda"), right=True).clamp_(max=classes - 1)
        lab = lab[torch.randperm(n, device="cuda", generator=g)]
        X = (2 * normal(classes, d))[lab] + normal(n, d)
        y = lab.float() + 1
    return X.cpu().numpy().astype(np.float32), y.cpu().numpy().astype(np.float64)


def _sparse(n, d, nnz, seed):
    """About nnz nonzeros a row, lognormal values, rows of length one; labels by a sparse hyperplane, 10% flipped."""
    rng = np.random.default_rng(seed)
    lens = np.clip(rng.poisson(min(nnz, d // 2), n), 1, d)
    rows = np.repeat(np.arange(n), lens)
    key = np.unique(rows.astype(np.int64) * d + rng.integers(0, d, rows.size))
    rows, col = key // d, (key % d).astype(np.int32)
    val = rng.lognormal(0.0, 1.0, rows.size)
    val = (val / np.sqrt(np.bincount(rows, val * val, n))[rows]).astype(np.float32)
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(rows, minlength=n), out=ptr[1:])
    w = np.where(rng.random(d) < max(0.01, 32 / d), rng.standard_normal(d), 0.0)
    y = np.where(np.bincount(rows, val * w[col], n) >= 0, 1.0, -1.0)
    return (ptr, col, val), np.where(rng.random(n) < 0.1, -y, y)


def _csr(X):
    if isinstance(X, tuple):
        return X
    n, d = X.shape
    r, c = np.nonzero(X)
    ptr = np.zeros(n + 1, np.int64)
    np.cumsum(np.bincount(r, minlength=n), out=ptr[1:])
    return ptr, c.astype(np.int32), np.ascontiguousarray(X[r, c])


class Nodes:
    """svm_node rows (1-based indices, zeros left out, each row ended by -1) and the svm_problem over them."""

    def __init__(self, X, y=None):
        if not isinstance(X, tuple) and np.all(X):
            n, d = X.shape
            buf = np.zeros((n, d + 1), cabi.NODE_DTYPE)
            buf["index"][:, :d] = np.arange(1, d + 1, dtype=np.int32)
            buf["index"][:, d] = -1
            buf["value"][:, :d] = X
            start = np.arange(n, dtype=np.int64) * (d + 1)
        else:
            ptr, col, val = _csr(X)
            n = ptr.size - 1
            buf = np.zeros(col.size + n, cabi.NODE_DTYPE)
            at = np.arange(col.size) + np.repeat(np.arange(n), np.diff(ptr))
            buf["index"][at] = col + 1
            buf["value"][at] = val
            buf["index"][ptr[1:] + np.arange(n)] = -1
            start = ptr[:-1] + np.arange(n)
        self.buf, self.n = buf, n
        self.addrs = (buf.ctypes.data + 16 * start).astype(np.uint64)
        self.y = np.ascontiguousarray(np.zeros(n) if y is None else y, np.float64)
        self.prob = cabi.svm_problem()
        self.prob.l = n
        self.prob.y = self.y.ctypes.data_as(C.POINTER(C.c_double))
        self.prob.x = C.cast(C.c_void_p(self.addrs.ctypes.data), C.POINTER(C.POINTER(cabi.svm_node)))


def _model_inputs(case, seed):
    """Support vectors grouped by class, their coefficients and the pairs' offsets, with test rows."""
    k = case["classes"]
    kind = "pixels" if case["d"] >= 512 else "classes"
    X, y = _data(kind, case["sv"] + case["n"], case["d"], seed, k)
    rng = np.random.default_rng(seed)
    lab = np.sort(rng.integers(0, k, case["sv"]))
    S = X[:case["sv"]]
    if kind == "classes":
        order = np.argsort(y[:case["sv"]], kind="stable")
        S, lab = S[order], y[:case["sv"]][order].astype(np.int64) - 1
    count = np.bincount(lab, minlength=k).astype(np.int32)
    coef = rng.random((k - 1, case["sv"])) * (rng.random((k - 1, case["sv"])) < 0.7)
    coef *= np.where(np.arange(k - 1)[:, None] >= lab[None, :], 1.0, -1.0)
    rho = rng.standard_normal(k * (k - 1) // 2)
    return np.ascontiguousarray(S), coef, count, rho, np.ascontiguousarray(X[case["sv"]:])


class Model:
    """An svm_model in malloc'ed memory, as svm_load_model builds one; freed by svm_free_and_destroy_model."""

    def __init__(self, case, seed):
        S, coef, count, rho, self.rows = _model_inputs(case, seed)
        self.sv = Nodes(S)
        k = case["classes"]

        def block(a):
            a = np.ascontiguousarray(a)
            p = _libc.malloc(max(a.nbytes, 1))
            C.memmove(p, a.ctypes.data, a.nbytes)
            return p

        m = cabi.svm_model()
        m.param = cabi.make_param(kernel_type=KERNELS[case["kernel"]], gamma=case["gamma"])
        m.nr_class, m.l, m.free_sv = k, len(S), 0
        m.SV = C.cast(block(self.sv.addrs), type(m.SV))
        m.sv_coef = C.cast(block(np.array([block(c) for c in coef], np.uint64)), type(m.sv_coef))
        m.rho = C.cast(block(rho), type(m.rho))
        m.label = C.cast(block(np.arange(1, k + 1, dtype=np.int32)), type(m.label))
        m.nSV = C.cast(block(count), type(m.nSV))
        p = _libc.malloc(C.sizeof(m))
        C.memmove(p, C.byref(m), C.sizeof(m))
        self.ptr = C.cast(C.c_void_p(p), C.POINTER(cabi.svm_model))

    def __del__(self):
        engine().lib.svm_free_and_destroy_model(C.byref(self.ptr))


def _svm_param(case):
    return cabi.make_param(svm_type=SVMS[case["svm"]], kernel_type=KERNELS[case["kernel"]], gamma=case["gamma"], C_=case["C"],
                           nu=case.get("nu", 0.5), cache_size=case.get("cache_mb", 100.0))


def _jobs(case, seed):
    """The jobs of the request mix: 60% dense, 70% C-SVC, RBF or cubic; sizes spread evenly over their logarithm."""
    rng = np.random.default_rng(seed)
    sizes = np.exp(np.linspace(math.log(case["n"]), math.log(case["n_hi"]), case["jobs"])).astype(int)
    dims = [d for d in (16, 64, 256, 512) if case["d"] <= d <= case["d_hi"]]
    jobs = []
    for k, n in enumerate(sizes):
        dense, d = k % 5 < 3, dims[k % len(dims)]
        d = d if dense else max(d, 64)
        X, y = _data("gauss" if dense else "sparse", int(n), d, int(rng.integers(1 << 30)))
        jobs.append((_csr(X), y, d, dict(svm_type=1 if k % 10 in (2, 5, 9) else 0, kernel_type=2 if k % 2 else 1,
                                        gamma=1.0 / d, C_pos=10.0 if k % 4 == 3 else 1.0, nu=0.3)))
    order = rng.permutation(len(jobs))
    return [jobs[i] for i in order]


class Rows:
    """Rows kept on the device by svmb_rows_upload_csr."""

    def __init__(self, X):
        n, d = X.shape
        ptr, col, val = _csr(X)
        self.h = C.c_void_p()
        if engine().lib.svmb_rows_upload_csr(n, d, ptr.ctypes.data, col.ctypes.data, val.ctypes.data, -1, C.byref(self.h)):
            raise RuntimeError(engine().error())

    def __del__(self):
        engine().lib.svmb_rows_free(self.h)


class Loop:
    """A request loop (svmb_server_create)."""

    def __init__(self, form):
        cfg = ServerConfig(8 << 30, 0, 0, FORMS[form], 0, 0)
        self.h = C.c_void_p()
        if engine().lib.svmb_server_create(C.byref(cfg), C.byref(self.h)):
            raise RuntimeError(engine().error())

    def __del__(self):
        engine().lib.svmb_server_destroy(self.h)


def prepare(case, seed):
    e, do, form = engine(), case["do"], FORMS[case["form"]]
    s = {"case": case}
    if do in ("predict", "predict_one"):
        e.set_option("predict_form", form)
        s["model"] = Model(case, seed)
        s["rows"] = Nodes(s["model"].rows)
    elif do == "serve":
        s["jobs"], s["loop"] = _jobs(case, seed), Loop(case["form"])
    else:
        e.set_option("form", form)
        X, s["y"] = _data(case["data"], case["n"], case["d"], seed, case.get("classes", 2), case.get("nnz", 40))
        if do == "solve":
            s["rows"] = Rows(X)
        else:
            s["nodes"], s["param"] = Nodes(X, s["y"]), _svm_param(case)
    return s


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _ptr(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _train_once(s):
    e, n = engine(), s["nodes"].n
    p = e.lib.svm_train(C.byref(s["nodes"].prob), C.byref(s["param"]))
    if not p:
        raise RuntimeError(e.error())
    m = p.contents
    k, l = m.nr_class, m.l
    at = np.ctypeslib.as_array(m.sv_indices, (l,)) - 1
    out = {"rho": np.ctypeslib.as_array(m.rho, (k * (k - 1) // 2,)).copy(), "coef": np.zeros((k - 1, n))}
    for j in range(k - 1):      # by training row: zero where a row is no support vector
        out["coef"][j, at] = np.ctypeslib.as_array(m.sv_coef[j], (l,))
    e.lib.svm_free_and_destroy_model(C.byref(p))
    return out


def _solve_once(s):
    e, case = engine(), s["case"]
    n = case["n"]
    prm = make_params(svm_type=SVMS[case["svm"]], kernel_type=KERNELS[case["kernel"]], gamma=case["gamma"], C_pos=case["C"],
                      cache_mb=case["cache_mb"], form=FORMS[case["form"]])
    ptr, at, alpha, st = np.array([0, n], np.int32), np.arange(n, dtype=np.int32), np.zeros(n), SolveStats()
    if e.lib.svmb_rows_solve_many(s["rows"].h, 1, ptr.ctypes.data, at.ctypes.data, s["y"].ctypes.data, C.byref(prm),
                                  alpha.ctypes.data, C.byref(st)):
        raise RuntimeError(e.error())
    return {"alpha": alpha, "rho": np.array([st.rho]), "iters": int(st.iters)}


def _serve_once(s):
    e = engine()
    tickets = []
    for (ptr, col, val), y, d, more in s["jobs"]:
        prm = make_params(form=FORMS[s["case"]["form"]], **more)
        tickets.append(e.lib.svmb_server_submit(s["loop"].h, y.size, d, ptr.ctypes.data, col.ctypes.data, val.ctypes.data,
                                                y.ctypes.data, C.byref(prm)))
    alphas, rho = [], []
    for t, (_, y, _, _) in zip(tickets, s["jobs"]):
        alpha, st, lat = np.zeros(y.size), SolveStats(), C.c_double()
        if t < 0 or e.lib.svmb_server_wait(s["loop"].h, t, alpha.ctypes.data, C.byref(st), C.byref(lat)):
            raise RuntimeError(e.error())
        alphas.append(alpha)
        rho.append(st.rho)
    return {"alpha": np.concatenate(alphas), "rho": np.array(rho)}


def run(s):
    e, case = engine(), s["case"]
    if case["do"] == "train":
        return _train_once(s)
    if case["do"] == "solve":
        return _solve_once(s)
    if case["do"] == "serve":
        return _serve_once(s)
    if case["do"] == "cv":
        target = np.zeros(s["nodes"].n)
        _libc.srand(1)      # the folds are drawn with rand(): those of a program's first call
        e.lib.svm_cross_validation(C.byref(s["nodes"].prob), C.byref(s["param"]), case["folds"], _ptr(target))
        return {"target": target}
    n, pairs = case["n"], case["classes"] * (case["classes"] - 1) // 2
    dec = np.zeros((n, pairs))
    if case["do"] == "predict_one":
        row = C.cast(C.c_void_p(int(s["rows"].addrs[0])), C.POINTER(cabi.svm_node))
        return {"label": e.lib.svm_predict_values(s["model"].ptr, row, _ptr(dec)), "dec": dec}
    label = np.zeros(n)
    if e.lib.svmb_predict_batch(s["model"].ptr, C.c_void_p(s["rows"].addrs.ctypes.data), n, _ptr(label), _ptr(dec)):
        raise RuntimeError(e.error())
    return {"label": label, "dec": dec}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def work(case):
    n, d = case["n"], case["d"]
    if case["do"] in ("predict", "predict_one"):
        pairs, sv = case["classes"] * (case["classes"] - 1) // 2, case["sv"]
        per = 3 if case["kernel"] == "rbf" and case["form"] == "exact" else 2
        return {"bytes": 16.0 * n * (d + 1) + 4.0 * sv * d + 8.0 * n * (pairs + 1), "flops": float(per) * n * sv * d}
    # training: the rows once, and one kernel row over the problem for each
    # support vector; their share is about what the data kind gives
    if case["do"] == "serve":
        sizes = np.exp(np.linspace(math.log(n), math.log(case["n_hi"]), case["jobs"]))
        return {"bytes": float(np.sum(sizes)) * 8 * 40, "flops": float(np.sum(0.4 * sizes * sizes)) * 2 * 64}
    share = {"gauss": 0.35, "sparse": 0.6, "pixels": 0.6, "regression": 0.5, "classes": 0.05}[case["data"]]
    width = case["nnz"] if case["data"] == "sparse" else d
    k = case.get("classes", 2)
    size = [n * 0.8 ** i / sum(0.8 ** j for j in range(k)) for i in range(k)]
    pairs = [size[i] + size[j] for i in range(k) for j in range(i + 1, k)] if k > 2 else [n]
    rounds = case.get("folds", 1)
    part = (1 - 1 / rounds) if rounds > 1 else 1.0
    node = 4 if case["do"] == "solve" else 16
    return {"bytes": float(node) * n * width + 8.0 * n, "flops": 2.0 * width * share * rounds * sum((part * l) ** 2 for l in pairs)}


# ---------------------------------------------------------------------------
# the same results in 64 bits without the engine
# ---------------------------------------------------------------------------
def _dense64(X, n, d):
    if not isinstance(X, tuple):
        return X.astype(np.float64)
    ptr, col, val = X
    out = np.zeros((n, d))
    out[np.repeat(np.arange(n), np.diff(ptr)), col] = val
    return out


def _gram(A, B, kernel, gamma):
    dot = A @ B.T
    if kernel == "poly":
        return (gamma * dot) ** 3
    if kernel == "linear":
        return dot
    sq = lambda M: (M * M).sum(1)  # noqa: E731
    return torch.exp(-gamma * (sq(A)[:, None] + sq(B)[None, :] - 2 * dot))


def _smo(K, y, cost, eps=1e-3, most=40000):
    """Two-variable descent with second-order selection on the whole kernel matrix (Fan, Chen and Lin 2005)."""
    n = y.size
    a, G, diag = np.zeros(n), -np.ones(n), np.diagonal(K).copy()
    for _ in range(most):
        up = np.where(y > 0, a < cost, a > 0)
        low = np.where(y > 0, a > 0, a < cost)
        v = -y * G
        i = int(np.argmax(np.where(up, v, -np.inf)))
        b = v[i] - v
        ok = low & (b > 0)
        if v[i] - np.min(np.where(low, v, np.inf)) < eps:
            return a * y
        quad = np.maximum(diag[i] + diag - 2 * K[i], 1e-12)
        j = int(np.argmin(np.where(ok, -b * b / quad, np.inf)))
        step = b[j] / quad[j]
        step = min(step, cost - a[i] if y[i] > 0 else a[i], a[j] if y[j] > 0 else cost - a[j])
        a[i] = min(max(a[i] + y[i] * step, 0.0), cost)
        a[j] = min(max(a[j] - y[j] * step, 0.0), cost)
        G += step * y * (K[i] - K[j])
    return None


def exact(case, seed):
    if case["do"] in ("predict", "predict_one"):
        S, coef, count, rho, rows = _model_inputs(case, seed)
        k, out = case["classes"], []
        S64, W = torch.from_numpy(S).cuda().double(), torch.from_numpy(coef).cuda()
        edge = np.concatenate([[0], np.cumsum(count)])
        for part in torch.from_numpy(rows).split(2000):
            K = _gram(part.cuda().double(), S64, case["kernel"], case["gamma"])
            cols = [K[:, edge[i]:edge[i + 1]] @ W[j - 1, edge[i]:edge[i + 1]] + K[:, edge[j]:edge[j + 1]] @ W[i, edge[j]:edge[j + 1]]
                    for i in range(k) for j in range(i + 1, k)]
            out.append(torch.stack(cols, 1))
        dec = torch.cat(out).cpu().numpy() - rho
        return {"label": None, "dec": dec}
    # a trained model stops anywhere within its tolerance: only small binary
    # problems follow the same steps in 64 bits
    if case["do"] != "train" or case["svm"] != "c_svc" or case.get("classes", 2) > 2 or case["n"] > 4500:
        return None
    X, y = _data(case["data"], case["n"], case["d"], seed, 2, case.get("nnz", 40))
    A = torch.from_numpy(_dense64(X, case["n"], case["d"])).cuda()
    alpha = _smo(_gram(A, A, case["kernel"], case["gamma"]).cpu().numpy(), y, case["C"])
    return None if alpha is None else {"rho": None, "coef": alpha[None]}
