"""Performance cases: what programs built on this package call, over the sizes they call it with.

A case names one pass through a public entry point. The sizes come from the package's own workloads (`entropical_gb300.workloads`), its tests and the
benchmark: single densities of 1 to 3 dimensions, all-pairs mutual information, all-ordered-pairs transfer entropy, uneven entropy batches, the AMISE
bandwidth search, `dens` over all triples, the reference's own mutual-information formula, and a trajectory load.

Inputs are synthetic, drawn on the GPU from the seed with the distributions of those workloads; time series are concatenated trajectories of 1,000 frames.
"""
import math
import tempfile

import numpy as np
import torch

from entropical_gb300.densities import Context, default_context, write_xtc
from entropical_gb300.estimators import ReferenceEstimators

DEV = "cuda"
SEGMENT = 1000  # frames of one trajectory


def listed():
    return [
        # one marginal of a short recording: the smallest call, where launches and waits count
        {"name": "density_1d_1000", "kind": "density", "d": 1, "n": 1000, "lag": 0},
        # one joint density of two columns, as the reference's dens mode asks for it
        {"name": "density_2d_100003", "kind": "density", "d": 2, "n": 100003, "lag": 0},
        # one (x, x lagged, y) density, as the reference's transs mode asks for it, on an odd length
        {"name": "density_3d_lag_50021", "kind": "density", "d": 3, "n": 50021, "lag": 5},
        # an interactive all-pairs MI of a few columns held in host memory
        {"name": "mi_8x4000_host", "kind": "mi", "m": 8, "n": 4000, "host": True},
        # the benchmark's all-pairs MI
        {"name": "mi_64x100000", "kind": "mi", "m": 64, "n": 100000, "host": False},
        # transfer entropy of a small system
        {"name": "te_6x30011", "kind": "te", "m": 6, "n": 30011, "lags": "1,5"},
        # the largest job: transfer entropy of 32 coordinates at three lags
        {"name": "te_32x200000", "kind": "te", "m": 32, "n": 200000, "lags": "1,5,10"},
        # independent samples of very uneven size and dimension in one batch
        {"name": "uneven_64", "kind": "uneven", "count": 64, "n_min": 2000, "n_max": 200000},
        # bandwidths of all columns before an MI job
        {"name": "amise_64x100000", "kind": "amise", "m": 64, "n": 100000},
        # dens -D 3: every triple of a few columns, left on the device
        {"name": "dens_all_8x20011", "kind": "dens_all", "m": 8, "n": 20011, "dims": 3},
        # the reference's own MI formula over host columns
        {"name": "ref_mi_10x25000", "kind": "ref_mi", "m": 10, "n": 25000},
        # a compressed trajectory file decoded into the coordinate matrix
        {"name": "xtc_300x4000", "kind": "xtc", "atoms": 300, "frames": 4000},
    ]


def _log_int(rng, lo, hi):
    """Log-uniform in [lo, hi], odd more often than not."""
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v | 1 if rng.random() < 0.7 else v))


def draw(rng):
    kind = rng.choice(["density", "density", "mi", "mi", "te", "te", "uneven", "amise", "dens_all", "ref_mi", "xtc"])
    if kind == "density":
        d = rng.randint(1, 3)
        return {"kind": kind, "d": d, "n": _log_int(rng, 1000, 200000), "lag": rng.randint(1, 20) if d > 1 and rng.random() < 0.5 else 0}
    if kind == "mi":
        m = _log_int(rng, 4, 64)
        return {"kind": kind, "m": m, "n": _log_int(rng, 4000, 100000), "host": rng.random() < 0.5}
    if kind == "te":
        m = _log_int(rng, 4, 24)
        return {"kind": kind, "m": m, "n": _log_int(rng, 10000, 120000), "lags": ",".join(str(v) for v in sorted(rng.sample(range(1, 21), rng.randint(1, 3))))}
    if kind == "uneven":
        return {"kind": kind, "count": _log_int(rng, 8, 128), "n_min": 2000, "n_max": _log_int(rng, 20000, 200000)}
    if kind == "amise":
        return {"kind": kind, "m": _log_int(rng, 1, 64), "n": _log_int(rng, 2000, 200000)}
    if kind == "dens_all":
        return {"kind": kind, "m": rng.randint(3, 10), "n": _log_int(rng, 2000, 30000), "dims": rng.randint(2, 3)}
    if kind == "ref_mi":
        return {"kind": kind, "m": _log_int(rng, 3, 32), "n": _log_int(rng, 4000, 60000)}
    return {"kind": kind, "atoms": _log_int(rng, 30, 1000), "frames": _log_int(rng, 200, 8000)}


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _mixture(rng, d, n):
    """One mixture of 1 to 6 normal components, (d, n) float32 (workloads.mixture_instance)."""
    k = int(rng.integers(1, 7))
    w = torch.tensor(rng.dirichlet(np.ones(k)), device=DEV)
    mu = torch.tensor(rng.uniform(-2.0, 2.0, (k, d)), device=DEV, dtype=torch.float32)
    sd = torch.tensor(rng.uniform(0.1, 0.8, (k, d)), device=DEV, dtype=torch.float32)
    g = _gen(rng.integers(1 << 40))
    edges = torch.cumsum(w, 0)
    comp = torch.bucketize(torch.rand(n, device=DEV, generator=g, dtype=torch.float64), edges).clamp_(max=k - 1)
    return (mu[comp] + sd[comp] * torch.randn(n, d, device=DEV, generator=g)).T.contiguous()


def _tanh_columns(seed, m, n):
    """tanh(A z) of a 16-dimensional AR(1) process, standardised columns, (m, n) float32 (workloads.mi_coords)."""
    g = _gen(seed)
    seg = -(-n // SEGMENT)
    a = torch.randn(16, m, device=DEV, generator=g)
    z = torch.randn(seg, 16, device=DEV, generator=g) / math.sqrt(1.0 - 0.95 * 0.95)
    e = torch.randn(SEGMENT, seg, 16, device=DEV, generator=g)
    for t in range(SEGMENT):
        z = torch.add(e[t], z, alpha=0.95)
        e[t] = z
    x = torch.tanh(e.transpose(0, 1).reshape(-1, 16)[:n] @ a).T.double()
    x = (x - x.mean(1, keepdim=True)) / x.std(1, unbiased=False, keepdim=True)
    return x.float().contiguous()


def _langevin(seed, m, n):
    """Coupled double-well Langevin coordinates, (m, n) float32 (workloads.langevin)."""
    g = _gen(seed)
    seg = -(-n // SEGMENT)
    c = torch.where(torch.rand(m, m, device=DEV, generator=g) < 0.1, torch.rand(m, m, device=DEV, generator=g) * 0.6 - 0.3, 0.0)
    c.fill_diagonal_(0.0)
    x = torch.randint(0, 2, (seg, m), device=DEV, generator=g) * 2.0 - 1.0 + 0.1 * torch.randn(seg, m, device=DEV, generator=g)
    out = torch.empty(SEGMENT, seg, m, device=DEV)
    drift = torch.eye(m, device=DEV) * 1.01 + 0.01 * c.T
    for t in range(-300, SEGMENT):
        x = torch.addmm(0.05 * torch.randn(seg, m, device=DEV, generator=g), x, drift).sub_(x * x * x, alpha=0.01)
        if t >= 0:
            out[t] = x
    return out.transpose(0, 1).reshape(-1, m)[:n].T.contiguous()


def _scott(x, d):
    """Scott's rule for every row of x, float32 values as Python floats."""
    s = x.double().std(1, unbiased=False).cpu().numpy() * x.shape[1] ** (-1.0 / (d + 4))
    return [float(v) for v in s.astype(np.float32)]


def _sizes(case, seed):
    """(d, n) of every instance of an uneven batch."""
    rng = np.random.default_rng([int(seed), 1])
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    return [(int(rng.integers(1, 4)), int(math.exp(rng.uniform(lo, hi)))) for _ in range(case["count"])]


def _trajectory(case, seed):
    """(3 atoms, frames) float32: atoms along a chain, moving a little from frame to frame."""
    rng = np.random.default_rng(int(seed))
    at = np.cumsum(rng.normal(0.0, 0.15, (case["atoms"], 3)), axis=0) + 4.0
    x = at[None] + np.cumsum(rng.normal(0.0, 0.01, (case["frames"], 1, 3)), axis=0) + rng.normal(0.0, 0.03, (case["frames"], case["atoms"], 3))
    return np.ascontiguousarray(x.reshape(case["frames"], -1).T.astype(np.float32))


def _inputs(case, seed):
    """The coordinates and bandwidths of a case, on the GPU."""
    kind = case["kind"]
    if kind == "density":
        if case["lag"]:  # (x, x lagged, y)
            x = _langevin(seed, 2, case["n"] + case["lag"])
            cols, tau = ([0, 0, 1], [0, case["lag"], 0]) if case["d"] == 3 else ([0, 1], [case["lag"], 0])
        else:
            x = _mixture(np.random.default_rng(int(seed)), case["d"], case["n"])
            cols, tau = list(range(case["d"])), None
        h = _scott(x, case["d"])
        return x, cols, tau, [h[c] for c in cols]
    if kind == "uneven":
        rng = np.random.default_rng(int(seed))
        xs = [_mixture(rng, d, n) for d, n in _sizes(case, seed)]
        return xs, [_scott(x, x.shape[0]) for x in xs]
    if kind == "te":
        x = _langevin(seed, case["m"], case["n"])
        return x, _scott(x, 3)
    x = _tanh_columns(seed, case["m"], case["n"])
    return x, _scott(x, case.get("dims", 2))


def prepare(case, seed):
    kind = case["kind"]
    ctx: Context = default_context()
    state = {"case": case, "ctx": ctx}
    if kind == "density":
        x, cols, tau, h = _inputs(case, seed)
        state.update(x=x, cols=cols, tau=tau, h=h, out=torch.empty(case["n"], device=DEV, dtype=torch.float64))
    elif kind == "uneven":
        xs, hs = _inputs(case, seed)
        state.update(xs=xs, inst=[(x.data_ptr(), x.shape[0], x.shape[1], h) for x, h in zip(xs, hs)])
    elif kind == "xtc":
        f = tempfile.NamedTemporaryFile(suffix=".xtc")
        write_xtc(f.name, _trajectory(case, seed))
        state.update(file=f, out=torch.empty(3 * case["atoms"], case["frames"], device=DEV))
    else:
        x, h = _inputs(case, seed)
        state.update(x=x.cpu().numpy() if kind == "ref_mi" or case.get("host") else x, h=h)
        if kind == "te":
            state["taus"] = [int(v) for v in case["lags"].split(",")]
        elif kind == "dens_all":
            state["out"] = torch.empty(math.comb(case["m"], case["dims"]), case["n"], device=DEV, dtype=torch.float64)
        elif kind == "ref_mi":
            state["est"] = ReferenceEstimators(ctx)
    torch.cuda.synchronize()
    return state


def run(state):
    case, ctx = state["case"], state["ctx"]
    kind = case["kind"]
    if kind == "density":
        x = state["x"]
        ctx.combined_densities_device(x.data_ptr(), x.shape[1], x.shape[0], state["cols"], state["h"], state["tau"], state["out"].data_ptr())
        return state["out"]
    if kind == "mi":
        if case["host"]:
            return ctx.mi_all_pairs(state["x"], state["h"])
        return ctx.mi_all_pairs_device(state["x"].data_ptr(), case["n"], case["m"], state["h"])
    if kind == "te":
        return ctx.te_all_pairs_device(state["x"].data_ptr(), case["n"], case["m"], state["h"], state["taus"])
    if kind == "uneven":
        return ctx.entropy_batch(state["inst"], device=True)
    if kind == "amise":
        return ctx.hestimate_device(state["x"].data_ptr(), case["n"], case["m"])[0]
    if kind == "dens_all":
        ctx.dens_all_device(state["x"].data_ptr(), case["n"], case["m"], state["h"], case["dims"], state["out"].data_ptr())
        return state["out"]
    if kind == "ref_mi":
        return state["est"].mi(state["x"], state["h"])
    ctx.load_xtc_device(state["file"].name, state["out"].data_ptr())
    return state["out"]


# ------------------------------------------------------------ least work
def _density_work(d, n):
    """(bytes, flops) beside the coordinates of one density: at d <= 2 a sum over a sorted range per point (two searches and some 30 operations), at d = 3
    the pairs inside the support, each once for both points (14 operations), for Scott bandwidths on normal columns."""
    if d < 3:
        return 0.0, n * (2.0 * d * math.log2(n) + 30.0 * d)
    return 0.0, 7.0 * n * n * (2.0 * n ** (-1.0 / 7.0) * 0.282) ** 3


def work(case):
    kind = case["kind"]
    b = f = 0.0
    dens = []
    if kind == "density":
        n = case["n"]
        b, dens = 4.0 * n * case["d"] + 8.0 * n, [(case["d"], n, 1)]
    elif kind in ("mi", "ref_mi"):
        m, n = case["m"], case["n"]
        b, dens = 4.0 * m * n + 8.0 * m * m, [(1, n, m), (2, n, m * (m - 1) // 2)]
    elif kind == "te":
        m, n, q = case["m"], case["n"], len(case["lags"].split(","))
        b, dens = 4.0 * m * n + 8.0 * q * m * m, [(1, n, q * m), (2, n, q * m * (m + 1) // 2), (3, n, q * m * (m - 1))]
    elif kind == "uneven":
        dens = [(d, n, 1) for d, n in _sizes(case, 0)]
        b = sum(4.0 * d * n for d, n, _ in dens) + 8.0 * case["count"]
    elif kind == "amise":  # sort, then 16 convolutions of one search and a few operations per point
        m, n = case["m"], case["n"]
        b, f = 4.0 * m * n + 4.0 * m, m * n * (math.log2(n) + 16.0 * (math.log2(n) + 8.0))
    elif kind == "dens_all":
        m, n, d = case["m"], case["n"], case["dims"]
        b, dens = 4.0 * m * n + 8.0 * n * math.comb(m, d), [(d, n, math.comb(m, d))]
    else:  # about 1.6 bytes of file per coordinate
        v = 3.0 * case["atoms"] * case["frames"]
        b, f = 5.6 * v, 10.0 * v
    for d, n, count in dens:
        f += _density_work(d, n)[1] * count
    return {"bytes": b, "flops": f}


# ---------------------------------------------------------- 64-bit values
def _density64(cols, h):
    """Product-Epanechnikov densities in 64 bits: each target against the sources within h of it in dimension 0."""
    n = cols[0].numel()
    xs, order = torch.sort(cols[0].double())
    pts = [xs] + [c.double()[order] for c in cols[1:]]
    out = torch.empty(n, device=xs.device, dtype=torch.float64)
    lo = torch.searchsorted(xs, xs - h[0]).cpu().numpy()
    hi = torch.searchsorted(xs, xs + h[0], right=True).cpu().numpy()
    a = 0
    while a < n:
        b = min(n, a + max(1, int(2.5e7 / max(1, hi[a] - lo[a]))))
        while b > a + 1 and (b - a) * (hi[b - 1] - lo[a]) > 5e7:
            b = a + (b - a) // 2
        w = None
        for x, hj in zip(pts, h):
            k = ((x[a:b, None] - x[None, lo[a]:hi[b - 1]]) / hj).square_().neg_().add_(1.0).clamp_(min=0.0)
            w = k if w is None else w.mul_(k)
        out[a:b] = w.sum(1) * (0.75 ** len(h) / (n * math.prod(h)))
        a = b
    back = torch.empty_like(out)
    back[order] = out
    return back


def _entropy64(cols, h):
    return -float(_density64(cols, h).log().mean())


def _amise64(x):
    """The reference's AMISE bracket search over one column."""
    xs = torch.sort(x.double())[0]
    n = xs.numel()
    centred = xs - xs[n // 2]
    prefix = torch.cat([centred.new_zeros(1), centred.cumsum(0)])
    at = torch.arange(n, device=xs.device)

    def amise(h):
        e = torch.searchsorted(xs, xs + 2.0 * h, right=True)
        c = (e - 1 - at).double()
        s = prefix[e] - prefix[at + 1] - c * centred
        conv = (4.5 * n + 2.0 * float((4.5 * c - 2.25 * s / h).sum())) / (float(n) * n)
        return (0.04 / h ** 5 * conv) ** 0.2 * 1.25 * 0.6 ** 0.8 / float(n) ** 0.8

    h0 = n ** (-1.0 / 7.0) * float(xs.var(unbiased=False).sqrt())
    lo, hi = 0.1 * h0, 2.0 * h0
    for _ in range(20):
        delta = hi - lo
        mid = lo + 0.5 * delta
        if delta <= 0.01 * h0:
            break
        if amise(mid - 0.25 * delta) < amise(mid + 0.25 * delta):
            hi = mid
        else:
            lo = mid
    return lo + 0.5 * (hi - lo)


def _pairs64(case):
    """Source-target pairs that the 64-bit values of a case take, in units of n^2 of the largest density."""
    kind, m = case["kind"], case.get("m", 1)
    if kind in ("mi", "ref_mi"):
        return math.comb(m, 2) * float(case["n"]) ** 2
    if kind == "te":
        return len(case["lags"].split(",")) * 1.5 * m * m * float(case["n"]) ** 2
    if kind == "dens_all":
        return math.comb(m, case["dims"]) * float(case["n"]) ** 2
    if kind == "uneven":
        return sum(float(n) ** 2 for _, n in _sizes(case, 0))
    return 0.0


def exact(case, seed):
    kind = case["kind"]
    if _pairs64(case) > 4e11:
        return None
    if kind == "xtc":
        return torch.from_numpy(np.round(_trajectory(case, seed).astype(np.float64) * 1000.0) / 1000.0)
    if kind == "density":
        x, cols, tau, h = _inputs(case, seed)
        tau = tau or [0] * case["d"]
        return _density64([x[c, t:t + case["n"]] for c, t in zip(cols, tau)], h)
    if kind == "uneven":
        xs, hs = _inputs(case, seed)
        return np.array([_entropy64(list(x), h) for x, h in zip(xs, hs)])
    x, h = _inputs(case, seed)
    m, n = case["m"], case["n"]
    if kind == "amise":
        return np.array([_amise64(c) for c in x])
    if kind == "mi":
        hx = np.array([_entropy64([x[i]], [h[i]]) for i in range(m)])
        mi = np.zeros((m, m))
        for i in range(m):
            for j in range(i + 1, m):
                mi[i, j] = mi[j, i] = hx[i] + hx[j] - _entropy64([x[i], x[j]], [h[i], h[j]])
        return mi, hx
    if kind == "ref_mi":
        p = [_density64([x[i]], [h[i]]) for i in range(m)]
        out = np.zeros((m, m))
        for i in range(m):
            for j in range(i + 1, m):
                pij = _density64([x[i], x[j]], [h[i], h[j]])
                out[i, j] = out[j, i] = float((pij * (pij / p[i] / p[j]).log()).sum())
        return out
    if kind == "te":
        taus = [int(v) for v in case["lags"].split(",")]
        out = np.zeros((len(taus), m, m))
        for q, tau in enumerate(taus):
            y, yp = x[:, :n - tau], x[:, tau:]
            h1 = [_entropy64([y[i]], [h[i]]) for i in range(m)]
            hl = [_entropy64([yp[i], y[i]], [h[i], h[i]]) for i in range(m)]
            hj = {(i, j): _entropy64([y[i], y[j]], [h[i], h[j]]) for i in range(m) for j in range(i + 1, m)}
            for i in range(m):
                for j in range(m):
                    if i != j:
                        out[q, i, j] = hj[min(i, j), max(i, j)] + hl[i] - _entropy64([y[j], yp[i], y[i]], [h[j], h[i], h[i]]) - h1[i]
        return out
    rows = []  # dens_all
    for i in range(m):
        for j in range(i + 1, m):
            for k in range(j + 1, m) if case["dims"] == 3 else [None]:
                c = [i, j] if k is None else [i, j, k]
                p = _density64([x[q] for q in c], [h[q] for q in c])
                rows.append(p / p.sum())
    return torch.stack(rows)
