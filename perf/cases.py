"""Workloads for timing and comparing the library through its public Python API.

Each case is one call sequence that a program makes for one signal (or one batch, image,
recording): hand the values over, run the solver for a fixed number of iterations, read the
whole solution back.  The stopping tolerance is 0, so that every pass does the same work; the
solver still polls its stopping rule as it does in any other call.  Host arrays are
page-locked, as the library's documentation advises.

Kinds
  qp        gamma-step QP of one 1-D signal (SPGQPSolver), mixed or FP64 precision
  ts        alternating theta / gamma loop of one 1-D signal (TSSolver), optionally with the FEM
            temporal coarsening of the gamma step
  mc        TSSolver on a multichannel recording (n channels)
  batch     gamma-step QPs of many signals of uneven length, K and epssqr in one handle
  image     gamma-step QP of an image on its pixel grid
  adjoint   reconstruction loss and its gradient through a converged gamma step
"""
import math

import numpy as np
import torch

from pasc_inference_gb300 import PASC_PREC_FP64, PASC_PREC_MIXED, Batch, BGMGraphGrid2D, Problem, capi

GLL = 10  # GLL memory of every solve (the benchmark's)


def listed():
    return [
        # a short sensor trace classified interactively: T = 1e4, K = 2 is the reference's plain
        # Signal1D example; one call is a few dozen microsecond-sized iterations
        {"name": "qp_t1e4_k2", "kind": "qp", "T": 10_000, "K": 2, "epssqr": 1.0, "its": 40, "precision": "mixed"},
        # an ordinary recording of odd length with more clusters
        {"name": "qp_t123457_k5", "kind": "qp", "T": 123_457, "K": 5, "epssqr": 1.0, "its": 40, "precision": "mixed"},
        # the size of the differentiable workload's forward solve
        {"name": "qp_t1e6_k3", "kind": "qp", "T": 1_000_000, "K": 3, "epssqr": 1.0, "its": 40, "precision": "mixed"},
        # the benchmark's headline: T = 1e7, K = 3, from host buffer to host buffer
        {"name": "qp_t1e7_k3", "kind": "qp", "T": 10_000_000, "K": 3, "epssqr": 1.0, "its": 50, "precision": "mixed"},
        # the plain method in FP64 at the reference example's size, and at the size where it is
        # used to certify a mixed solution
        {"name": "qp64_t1e4_k2", "kind": "qp", "T": 10_000, "K": 2, "epssqr": 10.0, "its": 40, "precision": "fp64"},
        {"name": "qp64_t1e6_k3", "kind": "qp", "T": 1_000_000, "K": 3, "epssqr": 10.0, "its": 20, "precision": "fp64"},
        # clustering of a signal with unknown levels: theta and gamma steps in turn
        {"name": "ts_t50001_k4", "kind": "ts", "T": 50_001, "K": 4, "epssqr": 1.0, "its": 20, "outer": 3, "fem": 1.0},
        # the same on a long signal with the gamma step on a 10x coarser grid
        {"name": "ts_fem_t2e6_k3", "kind": "ts", "T": 2_000_000, "K": 3, "epssqr": 1.0, "its": 20, "outer": 3, "fem": 0.1},
        # the multichannel recording of the benchmark
        {"name": "mc_t1e6_n128_k8", "kind": "mc", "T": 1_000_000, "n": 128, "K": 8, "epssqr": 50.0, "its": 20, "outer": 2},
        # many signals of uneven length in one handle
        {"name": "batch_64", "kind": "batch", "n": 64, "tmin": 1000, "tmax": 100_000, "its": 30},
        # a full-HD frame
        {"name": "image_1920x1080_k3", "kind": "image", "W": 1920, "H": 1080, "K": 3, "epssqr": 2.0, "its": 30},
        # the backward pass: gradient of the reconstruction loss through the solution
        {"name": "adjoint_t1e6_k3", "kind": "adjoint", "T": 1_000_000, "K": 3, "epssqr": 30.0},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["qp", "qp", "qp", "qp64", "ts", "ts", "mc", "batch", "image", "adjoint"])
    if kind == "qp":
        K = rng.randint(2, 8)
        return {"kind": "qp", "T": _log(rng, 1000, 30_000_000 // K), "K": K, "epssqr": rng.choice([1.0, 3.0]),
                "its": rng.randint(20, 40), "precision": "mixed"}
    if kind == "qp64":
        K = rng.randint(2, 5)
        return {"kind": "qp", "T": _log(rng, 1000, 3_000_000 // K), "K": K, "epssqr": float(_log(rng, 1, 100)),
                "its": rng.randint(10, 40), "precision": "fp64"}
    if kind == "ts":
        fem = rng.choice([1.0, 1.0, 0.5, 0.1])
        return {"kind": "ts", "T": _log(rng, 5000, 2_000_000), "K": rng.randint(2, 5), "epssqr": rng.choice([1.0, 3.0]),
                "its": rng.randint(10, 20), "outer": rng.randint(2, 3), "fem": fem}
    if kind == "mc":
        return {"kind": "mc", "T": _log(rng, 5000, 1_000_000), "n": rng.choice([2, 17, 64, 100, 128]), "K": rng.randint(2, 8),
                "epssqr": 50.0, "its": rng.randint(10, 20), "outer": 2}
    if kind == "batch":
        return {"kind": "batch", "n": rng.randint(8, 64), "tmin": 1000, "tmax": _log(rng, 10_000, 100_000),
                "its": rng.randint(15, 30)}
    if kind == "image":
        return {"kind": "image", "W": _log(rng, 60, 1920), "H": _log(rng, 40, 1080), "K": rng.randint(2, 4), "epssqr": 2.0,
                "its": rng.randint(10, 30)}
    return {"kind": "adjoint", "T": _log(rng, 2000, 1_000_000), "K": rng.randint(2, 4), "epssqr": float(_log(rng, 1, 30))}


# ------------------------------------------------------------------------------------------
# inputs
# ------------------------------------------------------------------------------------------
def _rng(seed, stream=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1_000_003 + stream)
    return g


def _signal(seed, T, K, levels, sigma, stream=0):
    """Piecewise-constant signal on `levels` plus Gaussian noise: FP32 data, clean copy, labels."""
    g = _rng(seed, stream)
    mean = max(20, min(50_000, T // 40))
    nseg = 3 * (T // mean) + 8
    length = torch.randint(max(1, mean // 2), mean + mean // 2 + 1, (nseg,), generator=g, device="cuda")
    ends = torch.cumsum(length, 0)
    step = torch.randint(1, K, (nseg,), generator=g, device="cuda") if K > 1 else torch.zeros_like(length)
    state = torch.cumsum(step, 0) % K
    labels = state[torch.searchsorted(ends, torch.arange(T, device="cuda"), right=True).clamp_(max=nseg - 1)]
    lev = torch.as_tensor(levels, dtype=torch.float32, device="cuda")
    clean = lev[labels]
    data = clean + sigma * torch.randn(T, generator=g, device="cuda")
    return data, clean, labels


def _blocked(g):
    """T x K weights as the flat blocked array (k*T + t) that a TSSolver permutes first."""
    return g.t().contiguous().reshape(-1)


def _guess(seed, labels, K, share):
    """Start weights of a clustering from a rough labelling: a share of the mass on it, the rest
    random (T x K, rows sum to 1)."""
    u = torch.rand(labels.numel(), K, generator=_rng(seed, 77), device="cuda")
    u *= (1.0 - share) / u.sum(1, keepdim=True)
    u[torch.arange(labels.numel(), device="cuda"), labels] += share
    return u


def _host(t):
    """Page-locked host copy."""
    h = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    h.copy_(t)
    return h.numpy()


def _host_like(n, dtype):
    return torch.empty(n, dtype=dtype, pin_memory=True).numpy()


def _levels(K):
    return [float(k) for k in range(K)]


def _inputs(case, seed):
    """Tensors (on the GPU) that prepare() hands over and exact() computes from."""
    kind = case["kind"]
    if kind in ("qp", "ts", "adjoint"):
        T, K = case["T"], case["K"]
        data, clean, labels = _signal(seed, T, K, _levels(K), 0.5)
        out = {"data": data, "theta": torch.as_tensor(_levels(K), dtype=torch.float64)}
        if kind == "qp":
            out["gamma0"] = torch.rand(T * K, generator=_rng(seed, 5), device="cuda")
        elif kind == "ts":
            out["gamma0"] = _blocked(_guess(seed, labels, K, 0.5))
        else:
            out["clean"] = clean
            out["gamma0"] = _smooth_solution(data.double(), out["theta"].cuda(), case["epssqr"]).float().reshape(-1)
        return out
    if kind == "mc":
        T, n, K = case["T"], case["n"], case["K"]
        g = _rng(seed)
        centroids = torch.randn(K, n, generator=g, device="cuda")
        _, _, labels = _signal(seed, T, K, _levels(K), 0.0, 9)
        X = torch.empty(T, n, device="cuda")
        for i in range(0, T, 1 << 18):
            j = min(T, i + (1 << 18))
            X[i:j] = centroids[labels[i:j]] + 0.8 * torch.randn(j - i, n, generator=g, device="cuda")
        return {"data": X, "gamma0": _blocked(_guess(seed, labels, K, 0.1))}
    if kind == "batch":
        r = np.random.default_rng([int(seed), 11])
        sizes = np.random.default_rng([case["n"], case["tmax"]])  # the same lengths for every seed: one handle's shape
        n = case["n"]
        T = np.exp(sizes.uniform(math.log(case["tmin"]), math.log(case["tmax"]), n)).astype(np.int64)
        T[0] = case["tmax"]
        K = sizes.integers(2, 6, n).astype(np.int32)
        eps = np.exp(sizes.uniform(0.0, math.log(3.0), n))
        data, gamma0, theta = [], [], []
        for i in range(n):
            lev = np.sort(r.uniform(0.0, 4.0, K[i]))
            data.append(_signal(seed, int(T[i]), int(K[i]), lev, float(r.uniform(0.2, 1.0)), 100 + i)[0].double())
            gamma0.append(torch.rand(int(T[i]) * int(K[i]), generator=_rng(seed, 10_000 + i), device="cuda").double())
            theta.append(torch.as_tensor(lev))
        return {"T": T, "K": K, "epssqr": eps, "data": data, "gamma0": gamma0, "theta": theta}
    W, H, K = case["W"], case["H"], case["K"]
    g = _rng(seed)
    yy, xx = torch.meshgrid(torch.arange(H, device="cuda"), torch.arange(W, device="cuda"), indexing="ij")
    lab = ((xx - 0.4 * W) ** 2 + (yy - 0.5 * H) ** 2 < (0.3 * min(W, H)) ** 2).long()
    lab[(xx > 0.75 * W) & (xx < 0.9 * W)] = K - 1
    img = lab.float() + 0.4 * torch.randn(H, W, generator=g, device="cuda")
    return {"data": img.reshape(-1), "theta": torch.as_tensor(_levels(K), dtype=torch.float64),
            "gamma0": torch.rand(W * H * K, generator=_rng(seed, 5), device="cuda")}


def prepare(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    s = {"kind": kind, "case": dict(case)}
    if kind == "qp":
        f64 = case["precision"] == "fp64"
        dt = torch.float64 if f64 else torch.float32
        s["p"] = Problem(case["T"], case["K"], case["epssqr"], PASC_PREC_FP64 if f64 else PASC_PREC_MIXED)
        s["data"], s["gamma0"], s["theta"] = _host(x["data"].to(dt)), _host(x["gamma0"].to(dt)), x["theta"].numpy()
        s["out"] = _host_like(case["T"] * case["K"], dt)
        s["spg"] = capi.spgqp_opts(m=GLL, maxit=case["its"], eps=0.0)
    elif kind in ("ts", "mc"):
        T, K = case["T"], case["K"]
        s["p"] = Problem(T, K, case["epssqr"], PASC_PREC_MIXED, xdim=case.get("n", 1))
        if case.get("fem", 1.0) < 1.0:
            s["p"].set_fem(case["fem"], 0)
        if kind == "mc":  # the recording is handed over once and clustered from several starts
            s["p"].set_data_f32(_host(x["data"].reshape(-1)))
        else:
            s["data"] = _host(x["data"])
        s["gamma0"] = _host(x["gamma0"])
        s["out"] = _host_like(T * K, torch.float32)
        s["ts"] = capi.ts_opts(maxit=case["outer"], eps=0.0)
        s["spg"] = capi.spgqp_opts(m=GLL, maxit=case["its"], eps=0.0)
    elif kind == "batch":
        s["b"] = Batch(x["T"], x["K"], x["epssqr"])
        for i in range(s["b"].n):  # the signals stay in the handle and are solved from several starts
            s["b"].set_data(i, x["data"][i].cpu().numpy())
            s["b"].set_theta(i, x["theta"][i].numpy())
        s["gamma0"] = [_host(t) for t in x["gamma0"]]
        s["end"] = np.cumsum(x["T"] * x["K"])
        s["out"] = np.zeros(int(s["end"][-1]), dtype=np.float32)
        s["spg"] = capi.spgqp_opts(m=GLL, maxit=case["its"], eps=0.0)
    elif kind == "image":
        W, H, K = case["W"], case["H"], case["K"]
        grid = BGMGraphGrid2D(W, H)
        grid.process_grid()
        s["p"] = Problem(1, K, case["epssqr"], PASC_PREC_MIXED, graph=grid)
        s["data"], s["gamma0"], s["theta"] = _host(x["data"]), _host(x["gamma0"]), x["theta"].numpy()
        s["out"] = _host_like(W * H * K, torch.float32)
        s["spg"] = capi.spgqp_opts(m=GLL, maxit=case["its"], eps=0.0)
    else:
        s["p"] = Problem(case["T"], case["K"], case["epssqr"], PASC_PREC_MIXED)
        s["p"].set_data_f32(_host(x["data"]))
        s["p"].set_theta(x["theta"].numpy())
        s["gamma"] = _host(x["gamma0"])
        s["clean"] = _host(x["clean"].double())
        # a step of a learning loop: the gradient is wanted to far below the step's own noise
        s["opts"] = capi.adjoint_opts(cg_tol=1e-10)
    return s


def run(state):
    kind = state["kind"]
    if kind == "qp":
        p = state["p"]
        if state["out"].dtype == np.float64:
            p.set_data(state["data"])
            p.set_gamma(state["gamma0"])
            p.set_theta(state["theta"])
            p.update_b()
            st = p.spgqp_solve(state["spg"])
            return {"gamma": p.get_gamma_into(state["out"]), "fx": st.fx, "it": st.it}
        p.set_data_f32(state["data"])
        p.set_gamma_f32(state["gamma0"])
        p.set_theta(state["theta"])
        st = p.spgqp_solve(state["spg"])
        # (the mixed path sums its objective and theta from FP32 terms and FP32 weights; they
        # are kept in the type of the solution they belong to)
        return {"gamma": p.get_gamma_f32_into(state["out"]), "fx": np.float32(st.fx), "it": st.it}
    if kind in ("ts", "mc"):
        p = state["p"]
        if kind == "ts":
            p.set_data_f32(state["data"])
        p.set_gamma_f32(state["gamma0"])
        st = p.ts_solve(state["ts"], state["spg"])
        return {"gamma": p.get_gamma_f32_into(state["out"]), "theta": p.get_theta().astype(np.float32),
                "L": np.float32(st.L), "it": st.spg_it_sum}
    if kind == "batch":
        b = state["b"]
        for i in range(b.n):
            b.set_gamma(i, state["gamma0"][i])
        st = b.spgqp_solve(state["spg"])
        for i, end in enumerate(state["end"]):
            g = b.get_gamma(i)
            state["out"][end - g.size:end] = g
        return {"gamma": state["out"], "fx": np.array([r.fx for r in st], dtype=np.float32), "it": np.array([r.it for r in st])}
    if kind == "image":
        p = state["p"]
        p.set_data_f32(state["data"])
        p.set_gamma_f32(state["gamma0"])
        p.set_theta(state["theta"])
        st = p.spgqp_solve(state["spg"])
        return {"gamma": p.get_gamma_f32_into(state["out"]), "fx": np.float32(st.fx), "it": st.it}
    p = state["p"]
    p.set_gamma_f32(state["gamma"])
    loss = p.recon_mse(state["clean"])
    deps, ddata, dtheta, _ = p.adjoint(None, state["opts"])
    return {"loss": loss, "depssqr": deps, "ddata": ddata, "dtheta": dtheta}


# ------------------------------------------------------------------------------------------
# necessary work
# ------------------------------------------------------------------------------------------
#: arithmetic of one SPG iteration for one gamma entry: step, projection (about 6), operator
#: product, three dots, two updates, objective
_SPG_FLOPS = 30


def work(case):
    kind = case["kind"]
    if kind == "qp":
        T, K = case["T"], case["K"]
        w = 8 if case["precision"] == "fp64" else 4
        return {"bytes": w * (2 * T * K + T), "flops": _SPG_FLOPS * T * K * case["its"]}
    if kind == "ts":
        T, K = case["T"], case["K"]
        return {"bytes": 4 * (2 * T * K + T),
                "flops": case["outer"] * T * K * (8 + case["fem"] * _SPG_FLOPS * case["its"])}
    if kind == "mc":
        T, K, n = case["T"], case["K"], case["n"]
        return {"bytes": 2 * T * n + 8 * T * K, "flops": case["outer"] * T * K * (4 * n + _SPG_FLOPS * case["its"])}
    if kind == "batch":
        sizes = np.random.default_rng([case["n"], case["tmax"]])
        T = np.exp(sizes.uniform(math.log(case["tmin"]), math.log(case["tmax"]), case["n"])).astype(np.int64)
        T[0] = case["tmax"]
        K = sizes.integers(2, 6, case["n"])
        return {"bytes": float(np.sum(4 * (2 * T * K + T))), "flops": float(_SPG_FLOPS * case["its"] * np.sum(T * K))}
    if kind == "image":
        R, K = case["W"] * case["H"], case["K"]
        return {"bytes": 4 * (2 * R * K + R), "flops": (_SPG_FLOPS + 4) * R * K * case["its"]}
    T, K = case["T"], case["K"]
    return {"bytes": 4 * T * K + 4 * T + 8 * 2 * T, "flops": 14 * T * K * 100}  # about 100 CG iterations at least


# ------------------------------------------------------------------------------------------
# the same in 64 bits
# ------------------------------------------------------------------------------------------
def _project(y):
    """Rows of y onto the simplex: the threshold is the largest of (sum of the j largest - 1) / j."""
    K = y.shape[1]
    s = [y[:, k].clone() for k in range(K)]
    for r in range(K):  # descending odd-even transposition
        for a in range(r & 1, K - 1, 2):
            hi, lo = torch.maximum(s[a], s[a + 1]), torch.minimum(s[a], s[a + 1])
            s[a], s[a + 1] = hi, lo
    acc, tau = torch.zeros_like(s[0]), None
    for j in range(K):
        acc = acc + s[j]
        t = (acc - 1.0) / (j + 1)
        tau = t if tau is None else torch.maximum(tau, t)
    return (y - tau[:, None]).clamp_(min=0.0)


def _chain(x):
    """2 sum of (x_t - x_neighbour) along the time axis (rows)."""
    y = torch.zeros_like(x)
    d = 2.0 * (x[1:] - x[:-1])
    y[1:] += d
    y[:-1] -= d
    return y


def _grid(W, H):
    def apply(x):
        v = x.reshape(H, W, -1)
        y = torch.zeros_like(v)
        d = v[1:] - v[:-1]
        y[1:] += d
        y[:-1] -= d
        d = v[:, 1:] - v[:, :-1]
        y[:, 1:] += d
        y[:, :-1] -= d
        return y.reshape(x.shape)
    return apply


def _spg(x, b, apply, coeff, its):
    """its iterations of the spectral projected gradient method with the GLL line search."""
    x = _project(x)
    g = coeff * apply(x) - b
    fx = 0.5 * float(((g - b) * x).sum())
    fs, last, alpha = [fx] * GLL, 0, 2.0
    for _ in range(its):
        d = _project(x - alpha * g) - x
        Ad = coeff * apply(d)
        dd, dAd, gd = float((d * d).sum()), float((d * Ad).sum()), float((g * d).sum())
        if not (dd > 0.0 and dAd > 0.0):
            break
        xi, bar = (max(fs) - fx) / dAd, -gd / dAd
        beta = min(max(0.9 * bar + math.sqrt(0.81 * bar * bar + 2.0 * xi), 0.0), 1.0)
        x = x + beta * d
        g = g + beta * Ad
        fx = 0.5 * float(((g - b) * x).sum())
        last = (last + 1) % GLL
        fs[last] = fx
        alpha = dd / dAd
    return x, fx


def _smooth_solution(data, theta, epssqr, its=200):
    """Near-solution of the gamma step (accelerated projected gradient), T x K."""
    T = data.numel()
    coeff, b = epssqr / T, -((data[:, None] - theta) ** 2) / T
    x = _project(b * (T / 2.0))
    y, t, step = x, 1.0, 1.0 / (8.0 * coeff)
    for _ in range(its):
        xn = _project(y - step * (coeff * _chain(y) - b))
        tn = 0.5 * (1.0 + math.sqrt(1.0 + 4.0 * t * t))
        y = xn + ((t - 1.0) / tn) * (xn - x)
        x, t = xn, tn
    return x


def _exact_qp(data, gamma0, theta, T, K, epssqr, its):
    b = -((data[:, None] - theta) ** 2) / T
    return _spg(gamma0.reshape(T, K), b, _chain, epssqr / T, its)


def _exact_ts(case, x):
    T, K = case["T"], case["K"]
    gamma = x["gamma0"].double().reshape(K, T).t().contiguous()
    X = x["data"].bfloat16().double() if case["kind"] == "mc" else x["data"].double()[:, None]
    T2 = int(math.ceil(T * case.get("fem", 1.0)))
    if T2 < T:  # block sums over [round(j*T/T2), round((j+1)*T/T2))
        cut = torch.floor(torch.arange(T2 + 1, dtype=torch.float64, device="cuda") * (T / T2) + 0.5).long()
        block = torch.searchsorted(cut, torch.arange(T, device="cuda"), right=True) - 1

        def reduce(v):
            return torch.zeros(T2, v.shape[1], dtype=v.dtype, device="cuda").index_add_(0, block, v)
    for _ in range(case["outer"]):
        theta = (gamma.t() @ X) / gamma.sum(0)[:, None]
        res = torch.stack([((X - theta[k]) ** 2).sum(1) for k in range(K)], 1)
        if T2 < T:
            small, L = _spg(reduce(gamma), -reduce(res) / T2, _chain, case["epssqr"] / T, case["its"])
            gamma = small[block]
        else:
            gamma, L = _spg(gamma, -res / T, _chain, case["epssqr"] / T, case["its"])
    return gamma, theta, L


def _exact_adjoint(case, x):
    T, K = case["T"], case["K"]
    data, theta, clean = x["data"].double(), x["theta"].cuda(), x["clean"].double()
    gamma = x["gamma0"].double().reshape(T, K)
    coeff, bscale = case["epssqr"] / T, -1.0 / T
    e = gamma @ theta - clean
    z = _project(gamma - (coeff * _chain(gamma) - bscale * (data[:, None] - theta) ** 2) / (8.0 * coeff + abs(bscale)))
    free = (z > 1e-7).double()
    nf = free.sum(1, keepdim=True).clamp_(min=1.0)

    def P(v):
        v = v * free
        return free * (v - v.sum(1, keepdim=True) / nf)
    r = P(2.0 / T * e[:, None] * theta)
    lam, p, rr = torch.zeros_like(r), r.clone(), float((r * r).sum())
    stop = 1e-30 * rr
    for _ in range(5000):
        if rr <= stop:
            break
        q = P(coeff * _chain(p))
        a = rr / float((p * q).sum())
        lam += a * p
        r -= a * q
        new = float((r * r).sum())
        p = r + (new / rr) * p
        rr = new
    db = 2.0 * bscale * (data[:, None] - theta)
    direct = 2.0 / T * (gamma.t() @ e)  # the loss's own dependence on the levels
    return {"loss": float((e * e).sum()) / T, "depssqr": float(-(lam * _chain(gamma)).sum() / T),
            "ddata": (lam * db).sum(1), "dtheta": direct - (lam * db).sum(0)}


def exact(case, seed):
    kind, x = case["kind"], _inputs(case, seed)
    if kind == "qp":
        gamma, fx = _exact_qp(x["data"].double(), x["gamma0"].double(), x["theta"].cuda(), case["T"], case["K"],
                              case["epssqr"], case["its"])
        return {"gamma": gamma.reshape(-1), "fx": fx, "it": None}
    if kind in ("ts", "mc"):
        gamma, theta, L = _exact_ts(case, x)
        return {"gamma": gamma.reshape(-1), "theta": theta.reshape(-1), "L": L, "it": None}
    if kind == "batch":
        got = [_exact_qp(x["data"][i], x["gamma0"][i], x["theta"][i].cuda(), int(x["T"][i]), int(x["K"][i]),
                         float(x["epssqr"][i]), case["its"]) for i in range(case["n"])]
        return {"gamma": torch.cat([g.reshape(-1) for g, _ in got]), "fx": torch.tensor([f for _, f in got], dtype=torch.float64),
                "it": None}
    if kind == "image":
        W, H, K = case["W"], case["H"], case["K"]
        b = -(x["data"].double()[:, None] - x["theta"].cuda()) ** 2
        gamma, fx = _spg(x["gamma0"].double().reshape(W * H, K), b, _grid(W, H), case["epssqr"], case["its"])
        return {"gamma": gamma.reshape(-1), "fx": fx, "it": None}
    return _exact_adjoint(case, x)
