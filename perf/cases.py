"""Performance cases of the SHORE fit: what a user's program has it do, through the public entry points.

``listed()`` holds the named cases, ``draw(rng)`` one more case of the same ranges, ``prepare(case, seed)`` the
inputs a program holds before the call, ``run(state)`` one pass, ``work(case)`` the bytes and operations a pass
cannot do without, and ``exact(case, seed)`` the same outputs in 64 bits from plain torch and numpy.

Inputs are the package's synthetic acquisition: its CS-DSI gradient table (a seeded subset of the integer q-grid
behind one b = 0 volume) and one to three fibre tensors plus free water with Rician noise at SNR 25, S0 = 1000.
The gradient table of a case is fixed, as a study's protocol is; the voxels change with the seed.
"""

from __future__ import annotations

import math

import numpy as np
import torch

import cs_dmri_b200 as csd
from cs_dmri_b200.autograd import DifferentiableShore
from cs_dmri_b200.graddev import shore_fit_graddev
from cs_dmri_b200.phantom import BIG_DELTA, SMALL_DELTA, S0, SNR, brain_mask, gradient_table

ZETA = 700.0
DEFAULTS = dict(order=6, dirs=258, reg="l1", alpha_mode="fixed", precision="fp64", alpha=0.01, fill="full")


def listed():
    return [
        # A handful of voxels (the package's smoke volume): an interactive check of one region, all latency.
        dict(name="fit-108", kind="volume", x=6, y=6, z=3),
        # The reference's default call on host arrays, every diagnostic map asked for, on a 4,000-voxel block.
        dict(name="default-host-4k", kind="host", x=20, y=20, z=10, alpha_mode="l2-anchored"),
        # A whole brain, fixed alpha, resident on the GPU: the headline workload.
        dict(name="fit-brain300k", kind="volume", x=96, y=114, z=96, fill="brain"),
        # Radial order 8 (145 coefficients) on a slab of a volume.
        dict(name="fit-order8-32k", kind="volume", x=40, y=40, z=20, order=8),
        # The reference's default alpha selection on a ragged mask and an odd table of 181 samples.
        dict(name="default-path-50k", kind="volume", x=61, y=47, z=37, fill="brain", dirs=180,
             alpha_mode="l2-anchored"),
        # Tikhonov on a whole brain.
        dict(name="tikhonov-brain300k", kind="volume", x=96, y=114, z=96, fill="brain", reg="l2", lam=0.05),
        # The amplitude-positivity QP on a 64,000-voxel block.
        dict(name="nonneg-64k", kind="volume", x=40, y=40, z=40, reg="nonneg"),
        # The KKT-certified optimum on a whole brain, TF32 iterations and FP64 polish.
        dict(name="optimum-brain300k", kind="volume", x=96, y=114, z=96, fill="brain", precision="mixed-kkt"),
        # A training step through the L1 fit: fit, RTOP and ODF forward, and back to signals and alpha.
        dict(name="train-l1-50k", kind="grad", v=50000),
        # A small training step through the Tikhonov fit at radial order 8, odd batch.
        dict(name="train-l2-order8-3001", kind="grad", v=3001, order=8, reg="l2", lam=0.05),
        # Gradient nonlinearity: every voxel its own design, radial order 8, dropped samples.
        dict(name="graddev-order8-12k", kind="graddev", v=12288, order=8),
        # Maps of a fitted host volume: predicted signals, ODF SH, ODF peaks and the propagator scalars.
        dict(name="maps-32k", kind="maps", x=32, y=32, z=32),
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    def grid(v):
        x = max(1, min(96, int(round(v ** (1 / 3) * rng.uniform(0.7, 1.4)))))
        y = max(1, min(114, int(round(math.sqrt(v / x) * rng.uniform(0.8, 1.25)))))
        return dict(x=x, y=y, z=max(1, min(128, v // (x * y))), fill=rng.choice(["full", "brain"]))

    dirs = rng.choice([size(80, 514), size(80, 514), 258])
    what = rng.choice(["fit", "fit", "path", "l2", "nonneg", "optimum", "grad", "grad", "graddev", "host", "maps"])
    order = rng.choice([4, 6, 6, 8])
    if what == "fit":
        return dict(kind="volume", dirs=dirs, order=order, alpha=rng.choice([0.01, 0.05]),
                    **grid(size(64, 30000 if order == 8 else 300000)))
    if what == "path":
        return dict(kind="volume", dirs=dirs, order=min(order, 6), **grid(size(64, 30000)),
                    alpha_mode=rng.choice(["l2-anchored", "path-bic", "alpha-ratio"]))
    if what == "l2":
        return dict(kind="volume", dirs=dirs, order=order, reg="l2", lam=rng.choice([0.05, 0.01]),
                    **grid(size(64, 300000)))
    if what == "nonneg":
        return dict(kind="volume", dirs=max(dirs, 120), order=min(order, 6), reg="nonneg", **grid(size(64, 64000)))
    if what == "optimum":
        return dict(kind="volume", dirs=dirs, order=min(order, 6), precision=rng.choice(["mixed-kkt", "fp64-kkt"]),
                    **grid(size(64, 300000)))
    if what == "grad":
        reg = rng.choice(["l1", "l2"])
        return dict(kind="grad", dirs=dirs, order=order, reg=reg, lam=0.05, v=size(16, 5000 if order == 8 else 50000))
    if what == "graddev":
        return dict(kind="graddev", dirs=min(dirs, 300), order=max(order, 6), v=size(64, 8000),
                    precision=rng.choice(["fp64", "fp64-kkt", "mixed-kkt"]))
    if what == "host":
        return dict(kind="host", dirs=dirs, order=min(order, 6), alpha_mode=rng.choice(["fixed", "l2-anchored"]),
                    **grid(size(64, 8000)))
    return dict(kind="maps", order=order, dirs=dirs, **grid(size(64, 32768)))


# ------------------------------------------------------------------ inputs

def _full(case):
    return {**DEFAULTS, **case}


def _table(c):
    """(bvals (N,), bvecs (N, 3)) of the case's protocol, the b = 0 volume first."""
    return gradient_table(seed=1, n_dirs=c["dirs"])


def _n_coeffs(order):
    return sum(2 * l + 1 for n in range(order + 1) for l in range(0, n + 1, 2))


def _signals(gen, V, bvals, bvecs):
    """Rician multi-tensor signals (V, N) float32 on the GPU."""
    dev = torch.device("cuda")
    b, g = (torch.as_tensor(a, device=dev) for a in (bvals, bvecs))
    out = torch.empty((V, len(bvals)), dtype=torch.float32, device=dev)
    for lo in range(0, V, 32768):
        v = min(32768, V - lo)

        def u(*shape):
            return torch.rand(shape, generator=gen, device=dev, dtype=torch.float64)

        nf = 1 + torch.clamp((u(v) * 3).long(), max=2)
        e = -torch.log1p(-u(v, 3)) * (torch.arange(3, device=dev)[None] < nf[:, None])
        frac = e / e.sum(1, keepdim=True)
        iso = 0.3 * u(v)
        z, ph = 2 * u(v, 3) - 1, 2 * math.pi * u(v, 3)
        r = torch.sqrt(torch.clamp(1 - z * z, min=0))
        d = torch.stack([r * torch.cos(ph), r * torch.sin(ph), z], -1)
        cos2 = (d @ g.T).square()
        att = torch.exp(-b * (0.3e-3 + 1.4e-3 * cos2))
        s = (1 - iso)[:, None] * (frac[:, :, None] * att).sum(1) + iso[:, None] * torch.exp(-b * 3e-3)
        n1, n2 = (torch.randn(s.shape, generator=gen, device=dev, dtype=torch.float64) for _ in range(2))
        s, sigma = s * S0, S0 / SNR
        out[lo:lo + v] = torch.sqrt((s + sigma * n1).square() + (sigma * n2).square()).float()
    return out


def _mask(c):
    shape = (c["x"], c["y"], c["z"])
    return brain_mask(shape) if c["fill"] == "brain" and min(shape) > 2 else np.ones(shape, bool)


def _n_voxels(c):
    return c["v"] if "v" in c else int(_mask(c).sum())


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _volume(c, seed):
    """(signals of the masked voxels (V, N), volume (X, Y, Z, N), mask) on the GPU."""
    bvals, bvecs = _table(c)
    mask = torch.from_numpy(_mask(c)).cuda()
    sig = _signals(_generator(seed), int(mask.sum()), bvals, bvecs)
    data = torch.zeros(mask.shape + (len(bvals),), dtype=torch.float32, device="cuda")
    data[mask] = sig
    return sig, data, mask


def _fit_kwargs(c):
    kw = dict(big_delta=BIG_DELTA, small_delta=SMALL_DELTA, radial_order=c["order"], zeta=ZETA,
              regularization=c["reg"], precision=c["precision"])
    if c["reg"] == "l1":
        kw.update(alpha_mode=c["alpha_mode"], alpha=c["alpha"])
    elif c["reg"] == "l2":
        kw.update(lambda_n=c["lam"], lambda_l=c["lam"])
    return kw


def _deviation(c, seed):
    """Deviation tensors (V, 3, 3) and kept samples (V, N): up to 15 % of a voxel's weighted samples dropped."""
    gen, (bvals, _) = _generator(seed + 1_000_003), _table(c)
    V, N = c["v"], len(bvals)
    T = torch.eye(3, dtype=torch.float64, device="cuda") + 0.02 * torch.randn(
        (V, 3, 3), generator=gen, device="cuda", dtype=torch.float64)
    frac = 0.15 * torch.rand((V, 1), generator=gen, device="cuda")
    keep = torch.rand((V, N), generator=gen, device="cuda") >= frac
    keep[:, 0] = True
    return T, keep


def _coefficient_volume(c, seed):
    """A fitted coefficient volume: the Tikhonov solution of synthetic signals, plain torch."""
    sig, _, mask = _volume(c, seed)
    M = _design(*_table(c), c["order"])
    coef = _tikhonov(M, sig.double() @ M, c["order"], 0.05)
    vol = torch.zeros(mask.shape + (M.shape[1],), dtype=torch.float32, device="cuda")
    vol[mask] = coef.float()
    return vol.cpu().numpy(), mask.cpu().numpy()


def prepare(case, seed):
    c = _full(case)
    bvals, bvecs = _table(c)
    s = dict(case=c, bvals=bvals, bvecs=bvecs)
    if c["kind"] in ("volume", "host"):
        _, s["data"], s["mask"] = _volume(c, seed)
        if c["kind"] == "host":
            s["data"], s["mask"] = s["data"].cpu().numpy(), s["mask"].cpu().numpy()
    elif c["kind"] == "grad":
        s["signals"] = _signals(_generator(seed), c["v"], bvals, bvecs).requires_grad_(True)
        s["model"] = DifferentiableShore(bvals, bvecs, big_delta=BIG_DELTA, small_delta=SMALL_DELTA,
                                         radial_order=c["order"], zeta=ZETA, regularization=c["reg"])
        values = [c["alpha"]] if c["reg"] == "l1" else [c["lam"], c["lam"]]
        s["hyper"] = [torch.tensor(v, dtype=torch.float64, device="cuda", requires_grad=True) for v in values]
    elif c["kind"] == "graddev":
        s["signals"] = _signals(_generator(seed), c["v"], bvals, bvecs)
        s["T"], s["keep"] = _deviation(c, seed)
    else:
        s["coef"], s["mask"] = _coefficient_volume(c, seed)
    return s


# -------------------------------------------------------------------- pass

MAPS = ("coefficients", "r2", "residual_l2", "rmse", "iterations", "alpha", "bic", "rss_l2")


def run(state):
    c = state["case"]
    if c["kind"] == "volume":
        return csd.shore_fit_device(state["data"], state["mask"], state["bvals"], state["bvecs"], **_fit_kwargs(c))[0]
    if c["kind"] == "host":
        out = csd.shore_fit(state["data"], state["bvals"], state["bvecs"], state["mask"], diagnostics=True,
                            **_fit_kwargs(c))
        return {k: out[k] for k in MAPS if k in out}
    if c["kind"] == "grad":
        model, signals, hyper = state["model"], state["signals"], state["hyper"]
        coef = model.fit(signals, *hyper) if c["reg"] == "l1" else \
            model.fit(signals, lambda_n=hyper[0], lambda_l=hyper[1])
        rtop, odf = model.rtop(coef), model.odf(coef)
        loss = rtop.mean() + odf.square().mean()
        grads = torch.autograd.grad(loss, [signals, *hyper])
        return {"coef": coef.detach(), "loss": loss.detach(), "signals_grad": grads[0], "hyper_grad": list(grads[1:])}
    if c["kind"] == "graddev":
        out = shore_fit_graddev(state["signals"], state["bvals"], state["bvecs"], state["T"], state["keep"],
                                alpha=c["alpha"], radial_order=c["order"], zeta=ZETA, big_delta=BIG_DELTA,
                                small_delta=SMALL_DELTA, precision=c["precision"])
        # the certified modes time their iteration count on the call and report a low-order eigenvalue estimate
        keys = ("coefficients", "converged", "n_samples") + (("iterations", "lipschitz") if c["precision"] == "fp64"
                                                             else ())
        return {k: out[k] for k in keys}
    coef, mask, order = state["coef"], state["mask"], c["order"]
    out = csd.shore_odf_peaks(coef, order, ZETA, mask, npeaks=3)
    out["predict"] = csd.shore_predict(coef, order, ZETA, state["bvals"], state["bvecs"], big_delta=BIG_DELTA,
                                       small_delta=SMALL_DELTA)
    out["odf_sh"] = csd.shore_odf_sh(coef, order, ZETA, order, mask)
    out.update(csd.shore_microstructure(coef, order, ZETA, mask))
    return {k: v for k, v in out.items() if k not in ("rtap", "rtpp")}  # no directions are given


def work(case):
    """Signals (or coefficients) read once, results written once; the operations of the right-hand side and of the
    solver's own iteration at the mean counts the synthetic acquisition takes."""
    c = _full(case)
    V, N, K = _n_voxels(c), c["dirs"] + 1, _n_coeffs(c["order"])
    rhs, step = 2 * N * K, 2 * K * K + 8 * K
    nvol = c["x"] * c["y"] * c["z"] if "x" in c else V
    if c["kind"] in ("volume", "host"):
        bytes_ = 4 * V * N + 4 * nvol * K + nvol
        if c["kind"] == "host":
            bytes_ += 24 * nvol
        if c["reg"] == "l2":
            flops = V * rhs
        elif c["reg"] == "nonneg":
            flops = V * (rhs + 2 * K * K + 10 * 2 * 5 * (321 + K))
        elif c["precision"] in ("mixed-kkt", "fp64-kkt"):
            flops = V * (rhs + 2 * K * K)
        else:
            iters = {"fixed": 140, "alpha-ratio": 200, "l2-anchored": 2200, "path-bic": 4000}[c["alpha_mode"]]
            flops = V * (rhs + iters * step)
    elif c["kind"] == "grad":
        bytes_ = V * (4 * N + 8 * K + 4 * N + 8 * K)
        flops = V * (2 * rhs + 4 * 362 * K + (140 * step if c["reg"] == "l1" else 0))
    elif c["kind"] == "graddev":
        bytes_ = V * (4 * N + N + 72 + 8 * K)
        flops = V * (2 * N * K * K + rhs + (120 if c["precision"] == "fp64" else 20) * step)
    else:
        R = (c["order"] + 1) * (c["order"] + 2) // 2
        bytes_ = nvol * (4 * K + 4 * N + 4 * R + 4 * 16 + 4 * 6 + 1)
        flops = nvol * 2 * K * (N + 1) + V * 2 * K * 181
    return {"bytes": float(bytes_), "flops": float(flops)}


# ------------------------------------------------- the same in 64 bits, plain

def _columns(order):
    return [(n, l, k) for n in range(order + 1) for l in range(0, n + 1, 2) for k in range(2 * l + 1)]


def _legendre(l, m, x):
    """P_l^m with the Condon-Shortley phase, by the upward recurrence in l."""
    p = np.ones_like(x)
    for i in range(m):
        p = -p * (2 * i + 1) * np.sqrt(np.maximum(1 - x * x, 0))
    prev, cur = np.zeros_like(x), p
    for j in range(m + 1, l + 1):
        prev, cur = cur, ((2 * j - 1) * x * cur - (j + m - 1) * prev) / (j - m)
    return cur


def _laguerre(n, a, x):
    prev, cur = np.zeros_like(x), np.ones_like(x)
    for k in range(n):
        prev, cur = cur, ((2 * k + 1 + a - x) * cur - (k + a) * prev) / (k + 1)
    return cur


def _sh(l, m, theta, cos_phi):
    """Real spherical harmonic: cosine for m > 0, sine for m < 0, both from the Condon-Shortley P_l^|m|."""
    am = abs(m)
    norm = math.sqrt((2 * l + 1) / (4 * math.pi) * math.factorial(l - am) / math.factorial(l + am))
    p = norm * _legendre(l, am, cos_phi)
    if m == 0:
        return p
    return math.sqrt(2) * p * (np.cos(am * theta) if m > 0 else np.sin(am * theta))


def _order_of(l, k):
    """(signed order m, sign) of column k of a BrainSuite block: cosines l..1, zero, signed sines 1..l."""
    if k <= l:
        return l - k, 1.0
    return l - k, 1.0 if (k - l) % 2 == 1 else -1.0


def _design_rows(bvals, dirs, order):
    """SHORE design (rows, K) of b-values and unit directions, numpy."""
    tau = BIG_DELTA - SMALL_DELTA / 3
    q2 = np.where(bvals <= 50.0, 0.0, bvals / (4 * math.pi ** 2 * tau))
    u = q2 / ZETA
    q = np.sqrt(q2)[..., None] * dirs
    r = np.linalg.norm(q, axis=-1)
    cos_phi = np.where(r > 0, q[..., 2] / np.where(r > 0, r, 1), 1.0)
    theta = np.arctan2(q[..., 1], q[..., 0])
    radial, angular, cols = {}, {}, []
    for n, l, k in _columns(order):
        if (n, l) not in radial:
            kappa = math.sqrt(2 * math.factorial(n - l) / (ZETA ** 1.5 * math.gamma(n + 1.5)))
            radial[n, l] = kappa * _laguerre(n - l, l + 0.5, u) * np.exp(-u / 2) * u ** (l / 2)
        if (l, k) not in angular:
            m, sign = _order_of(l, k)
            angular[l, k] = sign * _sh(l, m, theta, cos_phi)
        cols.append(radial[n, l] * angular[l, k])
    return np.stack(cols, -1)


def _design(bvals, bvecs, order):
    return torch.from_numpy(_design_rows(bvals, bvecs, order)).cuda()


def _tikhonov(M, B, order, lam_n, lam_l=None):
    lam_l = lam_n if lam_l is None else lam_l
    w = [lam_n * (n * (n + 1)) ** 2 + lam_l * (l * (l + 1)) ** 2 for n, l, _ in _columns(order)]
    H = M.T @ M + torch.diag(torch.tensor(w, dtype=torch.float64, device=M.device))
    return torch.linalg.solve(H, B.T).T


def _fista(G, B, n, L, alpha, warm=None, tol=1e-6, max_iter=1000):
    """FISTA with the relative-change rule; G (K, K) or one per voxel (V, K, K), n, L, alpha per voxel.
    Returns (x, iterations, converged)."""
    V, K = B.shape
    X = torch.zeros_like(B) if warm is None else warm.clone()
    iters = torch.zeros(V, dtype=torch.int64, device=B.device)
    conv = torch.zeros(V, dtype=torch.bool, device=B.device)
    idx, x, y, b = torch.arange(V, device=B.device), X.clone(), X.clone(), B
    g, t = G, 1.0
    n, step, thr = n[:, None], (1 / L)[:, None], (alpha / L)[:, None]
    for it in range(1, max_iter + 1):
        gy = y @ g if g.dim() == 2 else torch.bmm(g, y[:, :, None])[:, :, 0]
        z = y - step * ((gy - b) / n)
        xn = torch.sign(z) * torch.clamp(z.abs() - thr, min=0)
        tn = (1 + math.sqrt(1 + 4 * t * t)) / 2
        d = xn - x
        y, x, t = xn + ((t - 1) / tn) * d, xn, tn
        done = d.norm(dim=1) / torch.clamp(xn.norm(dim=1), min=1e-12) < tol
        stop = done if it < max_iter else torch.ones_like(done)
        if bool(stop.any()):
            at = idx[stop]
            X[at], iters[at], conv[at] = x[stop], it, done[stop]
            live = ~stop
            idx, x, y, b, n, step, thr = (a[live] for a in (idx, x, y, b, n, step, thr))
            g = g if g.dim() == 2 else g[live]
            if not idx.numel():
                break
    return X, iters, conv


def _nnqp(H, q, lam):
    """min 1/2 l'Hl + q'l, l >= 0, one q per row, from the feasible rows of lam: the Lawson-Hanson active-set
    method, every row at its own step."""
    V, scale = q.shape[0], float(q.abs().max())
    live = torch.arange(V, device=q.device)
    free = lam > 0
    add = ~free.any(1)
    for _ in range(600):
        l, f, ql = lam[live], free[live], q[live]
        w = -(l @ H + ql)
        w[f] = -torch.inf
        best, j = w.max(1)
        stop = add[live] & (best <= 1e-13 * scale)
        f[add[live] & ~stop, j[add[live] & ~stop]] = True
        m = max(1, int(f.sum(1).max()))
        pos = torch.argsort(~f, dim=1, stable=True)[:, :m]
        on = torch.gather(f, 1, pos)
        A = H[pos[:, :, None], pos[:, None, :]] * (on[:, :, None] & on[:, None, :])
        A = A + torch.diag_embed((~on).double())
        z = torch.linalg.solve(A, (-torch.gather(ql, 1, pos) * on)[:, :, None])[:, :, 0]
        cur = torch.gather(l, 1, pos)
        bad = on & (z <= 0)
        ratio = torch.where(bad, cur / torch.clamp(cur - z, min=1e-300), torch.inf)
        a = torch.clamp(ratio.min(1).values, max=1.0)[:, None]
        new = cur + a * (z - cur)
        new = torch.where(bad & (ratio <= a), 0.0, new) * on
        full = torch.zeros_like(l).scatter_(1, pos, new)
        lam[live] = torch.where(stop[:, None], l, full)
        free[live] = (full > 0) & f
        add[live] = ~bad.any(1)
        live = live[~stop]
        if not live.numel():
            return lam
    raise RuntimeError("the active-set method did not end")


def _lasso(G, B, n, alpha, start):
    """The LASSO minimiser itself, from the support of `start`."""
    K = G.shape[0]
    H = torch.cat([torch.cat([G, -G], 1), torch.cat([-G, G], 1)])
    out = torch.empty_like(B)
    for lo in range(0, B.shape[0], 40000):
        b, s = B[lo:lo + 40000], start[lo:lo + 40000]
        q = torch.cat([n * alpha - b, n * alpha + b], 1)
        lam = _nnqp(H, q, torch.cat([torch.clamp(s, min=0), torch.clamp(-s, min=0)], 1))
        out[lo:lo + 40000] = lam[:, :K] - lam[:, K:]
    return out


def _hemisphere():
    """One of each antipodal pair of the 642-vertex icosphere (three midpoint subdivisions)."""
    g = (1 + math.sqrt(5)) / 2
    v = [(s * 1.0, t * g, 0.0) for s in (-1, 1) for t in (-1, 1)]
    v = np.array(v + [(0.0, a, b) for a, b, _ in v] + [(b, 0.0, a) for a, b, _ in v])
    v /= np.linalg.norm(v, axis=1, keepdims=True)
    edge = np.sort(np.linalg.norm(v[0] - v, axis=1))[1]
    near = lambda a, b: abs(np.linalg.norm(v[a] - v[b]) - edge) < 1e-9  # noqa: E731
    faces = [(a, b, c) for a in range(12) for b in range(a) for c in range(b)
             if near(a, b) and near(b, c) and near(a, c)]
    tri = v[np.array(faces)]
    for _ in range(3):
        a, b, c = tri[:, 0], tri[:, 1], tri[:, 2]
        ab, bc, ca = (m / np.linalg.norm(m, axis=1, keepdims=True) for m in (a + b, b + c, c + a))
        tri = np.concatenate([np.stack(t, 1) for t in ((a, ab, ca), (b, bc, ab), (c, ca, bc), (ab, bc, ca))])
    p = tri.reshape(-1, 3)
    p = p[np.unique(np.round(p, 9), axis=0, return_index=True)[1]]
    z, y, x = (np.where(np.abs(p[:, i]) > 1e-12, p[:, i], 0) for i in (2, 1, 0))
    return p[(z > 0) | ((z == 0) & (y > 0)) | ((z == 0) & (y == 0) & (x > 0))]


def _odf_factor(n, l):
    """Radial factor of the analytic SHORE ODF."""
    term, f = 1.0, 1.0
    for k in range(n - l):
        term *= (l - n + k) * (l / 2 + 1.5 + k) / ((l + 1.5 + k) * (k + 1)) * 2
        f += term
    c = (-1) ** (n - l // 2) * math.sqrt(2 * math.factorial(n - l) / (ZETA ** 1.5 * math.gamma(n + 1.5)))
    g = math.gamma(l / 2 + 1.5) * math.gamma(n + 1.5) / (math.gamma(l + 1.5) * math.factorial(n - l))
    return c * g * 0.5 ** (-l / 2 - 1.5) * f


def _odf_matrix(dirs, order):
    """ODF amplitudes of each coefficient on unit directions; the SH table is float32, as the interface has it."""
    theta, z = np.arctan2(dirs[:, 1], dirs[:, 0]), dirs[:, 2]
    cols = []
    for n, l, k in _columns(order):
        m, sign = _order_of(l, k)
        cols.append(_sh(l, m, theta, z).astype(np.float32).astype(np.float64) * sign * _odf_factor(n, l))
    return torch.from_numpy(np.stack(cols, 1)).cuda()


def _nonneg(M, B, order):
    """The amplitude-positivity fit along the reference's Goldfarb-Idnani path, whose end its multiplier rule sets
    (a full step gives the new constraint that step's length)."""
    G = M.T @ M + 1e-10 * torch.eye(M.shape[1], dtype=torch.float64, device=M.device)
    C = _odf_matrix(_hemisphere(), order)
    U = torch.linalg.solve(G, C.T)
    gam, tol, out = C @ U, 1e-9, torch.linalg.solve(G, B.T).T
    for lo in range(0, B.shape[0], 16384):
        x = out[lo:lo + 16384]
        s, live = x @ C.T, torch.arange(x.shape[0], device=x.device)
        u, act = torch.zeros_like(s), torch.zeros_like(s, dtype=torch.bool)
        p, fresh = torch.zeros_like(live), torch.ones_like(live, dtype=torch.bool)
        while True:
            val, j = torch.where(act[live], torch.inf, s[live]).min(1)
            stop = fresh[live] & (val >= -tol)
            p[live] = torch.where(fresh[live], j, p[live])
            live = live[~stop]
            if not live.numel():
                break
            a, pl = act[live], p[live]
            m = max(1, int(a.sum(1).max()))
            pos = torch.argsort(~a, dim=1, stable=True)[:, :m]
            on = torch.gather(a, 1, pos)
            A = gam[pos[:, :, None], pos[:, None, :]] * (on[:, :, None] & on[:, None, :])
            col = torch.gather(gam[pl], 1, pos) * on
            r = torch.linalg.solve(A + torch.diag_embed((~on).double()), col[:, :, None])[:, :, 0]
            zn = gam[pl, pl] - (col * r).sum(1)
            ratio = torch.where(on & (r > tol), torch.gather(u[live], 1, pos) / r, torch.inf)
            t1, d = ratio.min(1)
            t2 = torch.where(zn > tol, -s[live, pl] / zn, torch.inf)
            t = torch.minimum(t1, t2)
            full_r = torch.zeros_like(u[live]).scatter_(1, pos, r * on)
            step = torch.where(torch.isfinite(t), t, 0.0)[:, None]
            u[live] -= step * full_r
            s[live] += step * (gam[pl] - full_r @ gam)
            x[live] += step * (U.T[pl] - full_r @ U.T)
            full = t == t2
            act[live[full], pl[full]] = True
            u[live[full], pl[full]] = t[full]
            gone = torch.gather(pos, 1, d[:, None])[:, 0]
            act[live[~full], gone[~full]] = False
            fresh[live] = full
            live = live[torch.isfinite(t)]
    return out


def _path(M, B, S, mode, order, alpha_max):
    """The reference's alpha path: (coefficients, alpha, iterations, rss of the Tikhonov fit or None)."""
    n, L = M.shape[0], _lipschitz(M)
    G, V, dev = M.T @ M, B.shape[0], B.device
    rss = lambda x: (S - x @ M.T).square().sum(1)  # noqa: E731
    eps, ref = (1e-3, None) if mode == "path-bic" else (1e-4, rss(_tikhonov(M, B, order, 1e-8)))
    best = torch.full((V,), torch.inf, dtype=torch.float64, device=dev)
    X, A, I = torch.zeros_like(B), torch.zeros_like(best), torch.zeros(V, dtype=torch.int64, device=dev)
    idx, x = torch.arange(V, device=dev), torch.zeros_like(B)
    ones = torch.ones(V, dtype=torch.float64, device=dev)
    for i in range(20):
        lmax, lmin = torch.log(alpha_max[idx]), torch.log(alpha_max[idx] * eps)
        a = torch.exp(lmax + (i / 19) * (lmin - lmax))
        x, it, _ = _fista(G, B[idx], ones[idx] * n, ones[idx] * L, a, warm=x)
        r = (S[idx] - x @ M.T).square().sum(1)
        if ref is None:
            score = n * torch.log(torch.clamp(r, min=2.2250738585072014e-308) / n) + math.log(n) * (x != 0).sum(1)
            take, out = score < best[idx], torch.zeros_like(r, dtype=torch.bool)
        else:
            out, score = r <= 1.05 * ref[idx], r
            take = out | (r < best[idx])
        at = idx[take]
        best[at], X[at], A[at], I[at] = score[take], x[take], a[take], it[take]
        idx, x = idx[~out], x[~out]
        if not idx.numel():
            break
    return X, A, I, ref


def _lipschitz(M):
    return float(torch.linalg.eigvalsh(M.T @ M)[-1]) / M.shape[0]


def _l1_fixed(M, B, alpha):
    V = B.shape[0]
    ones = torch.ones(V, dtype=torch.float64, device=B.device)
    return _fista(M.T @ M, B, ones * M.shape[0], ones * _lipschitz(M), ones * alpha)


def _solve(c, sig):
    """(coefficients of the case's fit, alpha per voxel or None, rss of the Tikhonov reference or None)."""
    M, S = _design(*_table(c), c["order"]), sig.double()
    B = S @ M
    if c["reg"] == "l2":
        return _tikhonov(M, B, c["order"], c["lam"]), None, None
    if c["reg"] == "nonneg":
        return _nonneg(M, B, c["order"]), None, None
    alpha = torch.full((B.shape[0],), c["alpha"], dtype=torch.float64, device=B.device)
    n = M.shape[0]
    if c["alpha_mode"] != "fixed":
        amax = B.abs().max(1).values / n
        if c["alpha_mode"] in ("l2-anchored", "path-bic"):
            x, alpha, _, ref = _path(M, B, S, c["alpha_mode"], c["order"], amax)
            return x, alpha, ref
        alpha = amax * 1e-3
    ones = torch.ones_like(alpha)
    x = _fista(M.T @ M, B, ones * n, ones * _lipschitz(M), alpha)[0]
    if c["precision"] in ("mixed-kkt", "fp64-kkt"):
        x = _lasso(M.T @ M, B, n, c["alpha"], x)
    return x, alpha, None


def _in_volume(mask, v):
    out = torch.zeros(tuple(mask.shape) + tuple(v.shape[1:]), dtype=torch.float64, device=v.device)
    out[mask] = v
    return out


def _exact_host(c, seed):
    sig, _, mask = _volume(c, seed)
    x, alpha, ref = _solve(c, sig)
    M, S = _design(*_table(c), c["order"]), sig.double()
    n = M.shape[0]
    rss = (S - x @ M.T).square().sum(1)
    sst = (S - S.mean(1, keepdim=True)).square().sum(1)
    bic = n * torch.log(rss / n) + math.log(n) * (x != 0).sum(1)
    out = dict(coefficients=x, r2=1 - rss / sst, residual_l2=rss.sqrt(), rmse=(rss / n).sqrt(), alpha=alpha, bic=bic)
    if ref is not None:
        out["rss_l2"] = ref
    out = {k: _in_volume(mask, v).cpu().numpy() for k, v in out.items()}
    out["iterations"] = None
    return out


def _rtop_weights(order):
    """(e0, w): E(0) = e0 . c and RTOP = w . c / E(0)."""
    e0 = torch.zeros(_n_coeffs(order), dtype=torch.float64)
    w = torch.zeros_like(e0)
    for i, (n, l, _) in enumerate(_columns(order)):
        if l == 0:
            kappa = math.sqrt(2 * math.factorial(n) / (ZETA ** 1.5 * math.gamma(n + 1.5)))
            e0[i] = kappa * float(_laguerre(n, 0.5, np.zeros(1))[0]) / math.sqrt(4 * math.pi)
            w[i] = (-1) ** n * math.sqrt(16 * math.pi * ZETA ** 1.5 * math.gamma(n + 1.5) / math.factorial(n))
    return e0.cuda(), w.cuda()


def _exact_grad(c, seed):
    bvals, bvecs = _table(c)
    sig = _signals(_generator(seed), c["v"], bvals, bvecs)
    M = _design(bvals, bvecs, c["order"])
    B, V = sig.double() @ M, c["v"]
    coef = (_l1_fixed(M, B, c["alpha"])[0] if c["reg"] == "l1" else _tikhonov(M, B, c["order"], c["lam"]))
    x = coef.clone().requires_grad_(True)
    e0, w = _rtop_weights(c["order"])
    # the 362 directions are the call's default argument; here they are an input
    from cs_dmri_b200.autograd import geodesic_sphere
    odf = x @ _odf_matrix(geodesic_sphere(6), c["order"]).T
    loss = torch.clamp((x @ w) / (x @ e0), min=0).mean() + odf.square().mean()
    g, = torch.autograd.grad(loss, x)
    G = M.T @ M
    if c["reg"] == "l2":
        wv = _tikhonov(M, g, c["order"], c["lam"])
        nn, ll = (torch.tensor([float((s[i] * (s[i] + 1)) ** 2) for s in _columns(c["order"])], dtype=torch.float64,
                               device=M.device) for i in (0, 1))
        hyper = [-(wv * nn * coef).sum(), -(wv * ll * coef).sum()]
    else:
        wv = torch.zeros_like(coef)
        for lo in range(0, V, 8192):
            on = coef[lo:lo + 8192] != 0
            A = G[None] * (on[:, :, None] & on[:, None, :]) + torch.diag_embed((~on).double())
            wv[lo:lo + 8192] = torch.linalg.solve(A, (g[lo:lo + 8192] * on)[:, :, None])[:, :, 0]
        hyper = [-M.shape[0] * (torch.sign(coef) * wv).sum()]
    return {"coef": coef, "loss": loss.detach(), "signals_grad": wv @ M.T, "hyper_grad": hyper}


def _exact_graddev(c, seed):
    bvals, bvecs = _table(c)
    S = _signals(_generator(seed), c["v"], bvals, bvecs).double()
    T, keep = _deviation(c, seed)
    coef = torch.empty((c["v"], _n_coeffs(c["order"])), dtype=torch.float64, device="cuda")
    lip = torch.empty(c["v"], dtype=torch.float64, device="cuda")
    for lo in range(0, c["v"], 1024):
        t, k, s = T[lo:lo + 1024], keep[lo:lo + 1024], S[lo:lo + 1024]
        q = torch.einsum("vji,nj->vni", t, torch.as_tensor(bvecs, device="cuda"))
        norm = q.norm(dim=-1)
        b = torch.as_tensor(bvals, device="cuda") * norm.square()
        M = torch.from_numpy(_design_rows(b.cpu().numpy(), (q / torch.clamp(norm, min=1e-300)[..., None]).cpu().numpy(),
                                          c["order"])).cuda() * k[..., None]
        G, B, n = M.transpose(1, 2) @ M, torch.einsum("vnk,vn->vk", M, s), k.sum(1).double()
        L = torch.linalg.eigvalsh(G)[:, -1] / n
        coef[lo:lo + 1024] = _fista(G, B, n, L, torch.full_like(n, c["alpha"]))[0]
        lip[lo:lo + 1024] = L
    return {"coefficients": coef, "converged": None, "n_samples": None, "iterations": None, "lipschitz": lip}


def _exact_maps(c, seed):
    vol, mask = _coefficient_volume(c, seed)
    x, m = torch.from_numpy(vol).cuda().double(), torch.from_numpy(mask).cuda()
    P = torch.zeros((x.shape[-1], (c["order"] + 1) * (c["order"] + 2) // 2), dtype=torch.float64, device="cuda")
    for i, (n, l, k) in enumerate(_columns(c["order"])):
        order, sign = _order_of(l, k)
        P[i, l * (l + 1) // 2 + order] = sign * _odf_factor(n, l)
    e0, w = _rtop_weights(c["order"])
    rtop = torch.where(m, torch.clamp((x @ w) / (x @ e0), min=0) * 1e-9, 0)
    out = dict(gfa=None, peak_dirs=None, peak_values=None, peak_qa=None, msd=None, qiv=None, ng=None,
               predict=(x @ _design(*_table(c), c["order"]).T).cpu().numpy(), odf_sh=((x @ P) * m[..., None]).cpu().numpy())
    top = 10 * rtop[m].quantile(0.99, interpolation="nearest") if int(m.sum()) < 16_000_000 else math.inf
    out["rtop"] = torch.where(rtop > top, math.nan, rtop).cpu().numpy()
    return out


def exact(case, seed):
    c = _full(case)
    if c["kind"] == "volume":
        sig, _, mask = _volume(c, seed)
        return _in_volume(mask, _solve(c, sig)[0])
    if c["kind"] == "host":
        return _exact_host(c, seed)
    if c["kind"] == "grad":
        return _exact_grad(c, seed)
    if c["kind"] == "graddev":
        if c["precision"] != "fp64":
            return None  # the minimiser of a design per voxel: too long in plain batched algebra
        return _exact_graddev(c, seed)
    return _exact_maps(c, seed)
