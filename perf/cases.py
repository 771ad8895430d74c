"""The work that users of the library have it do, as measurable cases.

Each case is one call (or the few calls of one task) through the public Python
binding of the C API: encoding images as Fisher vectors or VLAD, projecting
descriptors, and learning the mixture model.  ``prepare`` makes what a program
has in hand before the call, ``run`` is one pass, ``work`` the bytes and
operations it cannot do without, and ``exact`` the same results in 64 bits.

Kinds (``op``):

* ``fv_host``   vl_fisher_encode on host arrays: a program relinked from VLFeat.
* ``fv_image``  one image already on the device, encoded in a serving loop.
* ``fv_batch``  a batch of uneven images encoded in one call.
* ``fv_plan``   a batch layout that repeats, encoded through a plan.
* ``gmm``       vl_gmm_cluster on host data: initialisation and EM.
* ``em``        EM on descriptors that are on the device, from given parameters.
* ``vlad``      a batch of uneven images encoded as VLAD.
* ``pca``       the descriptor prologue: projection, renormalisation, position.
"""
import math

import numpy as np
import torch

from vlfeat_b200 import capi
from vlfeat_b200 import workloads as W

DEV = "cuda"


def listed():
    return [
        # One small image through VLFeat's own call, default arithmetic: the
        # smallest call there is, all latency.
        {"name": "fv_host_small", "op": "fv_host", "n": 500, "d": 64, "k": 64, "flags": 3, "double": False},
        # The same call in double, plain vectors (the binding's default for
        # double descriptors), an odd row count.
        {"name": "fv_host_double", "op": "fv_host", "n": 2001, "d": 64, "k": 64, "flags": 0, "double": True},
        # One image of a serving loop, descriptors already on the device.
        {"name": "fv_image_fp32", "op": "fv_image", "n": 3000, "d": 80, "k": 256, "flags": 3, "precision": "fp32"},
        # A batch in the default arithmetic (VLFeat's float results).
        {"name": "fv_batch_exact", "op": "fv_batch", "images": 256, "median": 3000, "d": 80, "k": 256, "flags": 3,
         "precision": "exact"},
        # The recognition pipeline's descriptors: 80 PCA dimensions and x, y.
        {"name": "fv_batch_xy_fp32", "op": "fv_batch", "images": 512, "median": 3000, "d": 82, "k": 256, "flags": 3,
         "precision": "fp32"},
        # The benchmark's batch: 4,096 uneven images through a plan.
        {"name": "fv_plan_fp32", "op": "fv_plan", "images": 4096, "median": 3000, "d": 80, "k": 256, "flags": 3,
         "precision": "fp32"},
        # Learning a model with the defaults: Rand initialisation, EM on host data.
        {"name": "gmm_rand", "op": "gmm", "n": 100000, "d": 64, "k": 64, "init": "rand", "iters": 10},
        # Learning as the recognition pipeline does: KMeans initialisation.
        {"name": "gmm_kmeans", "op": "gmm", "n": 60001, "d": 80, "k": 256, "init": "kmeans", "iters": 5},
        # EM at scale on SIFT-shaped descriptors.
        {"name": "em_fp32", "op": "em", "n": 1000000, "d": 128, "k": 256, "iters": 5, "precision": "fp32"},
        # A large vocabulary, single-part posteriors.
        {"name": "em_bf16_k1024", "op": "em", "n": 150000, "d": 128, "k": 1024, "iters": 3, "precision": "bf16"},
        # VLAD of a batch with hard assignments, the usual intra-normalisation.
        {"name": "vlad_batch", "op": "vlad", "images": 256, "median": 3000, "d": 80, "k": 256, "flags": 1},
        # SIFT descriptors to 80 whitened dimensions with positions.
        {"name": "pca_batch", "op": "pca", "images": 512, "median": 3000, "d": 128, "m": 80, "xy": True},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["fv_host", "fv_image", "fv_batch", "fv_plan", "gmm", "em", "vlad", "pca"])
    dim = rng.choice([64, 64, 80, 80, 128, 128, rng.randint(24, 126)])
    flags = rng.choice([3, 3, 3, 0, 2])
    if op == "fv_host":
        return {"op": op, "n": _log(rng, 100, 20000), "d": dim, "k": rng.choice([32, 64, 100, 128, 256]),
                "flags": flags, "double": rng.random() < 0.4}
    if op == "fv_image":
        return {"op": op, "n": _log(rng, 100, 20000), "d": dim, "k": rng.choice([64, 128, 256, 512]),
                "flags": flags, "precision": rng.choice(["fp32", "fp32", "bf16"])}
    if op in ("fv_batch", "fv_plan"):
        big = op == "fv_plan"
        prec = rng.choice(["fp32", "fp32", "bf16"]) if big else rng.choice(["exact", "exact", "fp32", "bf16"])
        return {"op": op, "images": _log(rng, 16, 3000 if big else 400), "median": _log(rng, 500, 4000),
                "d": rng.choice([64, 80, 128]) if big else dim, "k": rng.choice([64, 128, 256]),
                "flags": flags, "precision": prec}
    if op == "gmm":
        return {"op": op, "n": _log(rng, 5000, 150000), "d": dim, "k": rng.choice([32, 64, 100, 128]),
                "init": rng.choice(["rand", "kmeans"]), "iters": rng.randint(3, 12)}
    if op == "em":
        k = rng.choice([64, 256, 512])
        return {"op": op, "n": _log(rng, 20000, 800000 // max(1, k // 256)), "d": rng.choice([64, 80, 128]), "k": k,
                "iters": rng.randint(2, 5), "precision": rng.choice(["exact", "fp32", "bf16"])}
    if op == "vlad":
        return {"op": op, "images": _log(rng, 16, 256), "median": _log(rng, 500, 4000), "d": dim,
                "k": rng.choice([64, 128, 256]), "flags": rng.choice([1, 0, 3])}
    return {"op": op, "images": _log(rng, 16, 512), "median": _log(rng, 500, 4000), "d": 128,
            "m": rng.choice([32, 64, 80, 96]), "xy": rng.random() < 0.7}


# ------------------------------------------------------------------ inputs
def _offsets(case):
    """Row offsets of the case's images: uneven, the same for every seed."""
    counts = W.image_counts(case["images"], seed=300 + case["images"], median=float(case["median"]))
    return np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)


def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed) * 7919 + 17)
    return g


def _pca_like(n, d, seed, dtype=torch.float32):
    """Rows of N(0, diag(lambda)), lambda_i = (1 + i)^-0.8 (PCA-projected descriptors)."""
    x = torch.empty((n, d), dtype=torch.float32, device=DEV)
    x.normal_(generator=_gen(seed))
    x *= torch.from_numpy(np.sqrt(W.pca_lambdas(d))).to(DEV, torch.float32)
    return x.to(dtype)


def _fv_model(case, seed):
    pr, mu, cv = W.fv_gmm(case["k"], case["d"], seed=11 + int(seed) % 100003, dtype=np.float32)
    return pr, mu, cv


def _mixture(case, seed):
    """Points of a seeded mixture of the case's shape, on the device."""
    means, sigma, priors = W.mixture_params(case["k"], case["d"], 100 + int(seed) % 100003)
    g = _gen(seed)
    p = torch.from_numpy(priors).to(DEV)
    c = torch.multinomial(p, case["n"], replacement=True, generator=g)
    m = torch.from_numpy(means.astype(np.float32)).to(DEV)
    s = torch.from_numpy(sigma.astype(np.float32)).to(DEV)
    return m[c] + s[c] * torch.randn((case["n"], case["d"]), generator=g, device=DEV)


def _em_inputs(case, seed):
    x = W.sift_like_device(case["n"], case["d"], seed=int(seed) * 31 + 5)
    pr, mu, cv, lb = W.custom_init_device(x, case["k"], seed=201 + int(seed) % 100003)
    return x, pr, mu, cv, lb


def _vlad_inputs(case, seed):
    off = _offsets(case)
    n, d, k = int(off[-1]), case["d"], case["k"]
    x = _pca_like(n, d, seed)
    means = torch.from_numpy(_fv_model(case, seed)[1]).to(DEV)
    a = torch.zeros((n, k), dtype=torch.float32, device=DEV)
    half = 0.5 * (means * means).sum(1)
    for i in range(0, n, 1 << 20):
        near = (half[None, :] - x[i:i + (1 << 20)] @ means.T).argmin(1)
        a[i:i + (1 << 20)].scatter_(1, near[:, None], 1.0)
    return off, x, means, a


def _pca_inputs(case, seed):
    off = _offsets(case)
    n = int(off[-1])
    x = W.sift_like_device(n, case["d"], seed=int(seed) * 31 + 7)
    # The projection as the recognition pipeline learns it: whitened principal
    # axes of a sample, each with its largest entry positive.
    t = x[:20000].double()
    mean = t.mean(0)
    ev, vec = torch.linalg.eigh(((t - mean).T @ (t - mean) / t.shape[0]).cpu())
    ev, vec = ev.flip(0)[:case["m"]], vec.flip(1)[:, :case["m"]].T
    vec = vec * torch.sign(vec.gather(1, vec.abs().argmax(1, keepdim=True)))
    proj = (vec / torch.sqrt(ev + 0.01 * ev[0])[:, None]).float().contiguous().to(DEV)
    centre = mean.float()
    frames = sizes = None
    if case["xy"]:
        g = _gen(seed + 1)
        frames = torch.rand((n, 2), generator=g, device=DEV) * 500.0
        sizes = torch.full((case["images"], 2), 500.0, device=DEV)
    return off, x, proj, centre, frames, sizes


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op == "fv_host":
        dt = np.float64 if case["double"] else np.float32
        x = _pca_like(case["n"], case["d"], seed, torch.float64 if case["double"] else torch.float32)
        s["x"] = x.cpu().numpy()
        s["gmm"] = tuple(v.astype(dt) for v in _fv_model(case, seed))
    elif op in ("fv_image", "fv_batch", "fv_plan"):
        pr, mu, cv = (torch.from_numpy(v).to(DEV) for v in _fv_model(case, seed))
        s["gmm"] = (pr, mu, cv)
        off = np.array([0, case["n"]], np.int64) if op == "fv_image" else _offsets(case)
        s["off"] = off
        s["x"] = _pca_like(int(off[-1]), case["d"], seed)
        s["enc"] = torch.zeros((len(off) - 1, 2 * case["k"] * case["d"]), dtype=torch.float32, device=DEV)
        s["nt"] = torch.zeros(len(off) - 1, dtype=torch.int64, device=DEV)
        if op == "fv_plan":
            s["plan"] = capi.FisherPlan(case["d"], case["k"], off, case["flags"], case["precision"])
            s["plan"].set_gmm(mu, cv, pr)
    elif op == "gmm":
        x = _mixture(case, seed)
        s["x"] = x.cpu().numpy()
        s["lb"] = 1e-4 * float(x.double().var(0).max())
        s["seed"] = 1 + int(seed) % 100003
        s["g"] = capi.GMM(case["d"], case["k"], np.float32)
        s["g"].set_initialization(case["init"])
        s["g"].set_max_num_iterations(case["iters"])
        s["g"].set_covariance_lower_bound(s["lb"])
    elif op == "em":
        s["x"], pr, mu, cv, lb = _em_inputs(case, seed)
        s["init"] = (pr, mu, cv)
        s["g"] = capi.GMM(case["d"], case["k"], np.float32)
        s["g"].set_initialization("custom")
        s["g"].set_max_num_iterations(case["iters"])
        s["g"].set_covariance_lower_bound(lb)
    elif op == "vlad":
        s["off"], s["x"], s["means"], s["a"] = _vlad_inputs(case, seed)
        s["enc"] = torch.zeros((case["images"], case["k"] * case["d"]), dtype=torch.float32, device=DEV)
    else:
        s["off"], s["x"], s["proj"], s["centre"], s["frames"], s["sizes"] = _pca_inputs(case, seed)
        s["out"] = torch.zeros((int(s["off"][-1]), case["m"] + (2 if case["xy"] else 0)), dtype=torch.float32,
                               device=DEV)
    torch.cuda.synchronize()
    return s


def _model_of(g, ll):
    return {"means": g.means, "covs": g.covariances, "priors": g.priors, "ll": float(ll)}


def run(s):
    case, op = s["case"], s["case"]["op"]
    if op == "fv_host":
        pr, mu, cv = s["gmm"]
        enc, nt = capi.fisher_encode(s["x"], mu, cv, pr, case["flags"])
        return {"enc": enc, "nt": nt}
    if op == "fv_image":
        pr, mu, cv = s["gmm"]
        nt = capi.fisher_encode_device(s["enc"], mu, cv, pr, s["x"], case["flags"], case["precision"])
        return {"enc": s["enc"], "nt": nt}
    if op == "fv_batch":
        pr, mu, cv = s["gmm"]
        capi.fisher_encode_batch_device(s["enc"], mu, cv, pr, s["x"], s["off"], case["flags"], case["precision"],
                                        s["nt"])
        return {"enc": s["enc"], "nt": s["nt"]}
    if op == "fv_plan":
        s["plan"].execute(s["enc"], s["x"], s["nt"])
        return {"enc": s["enc"], "nt": s["nt"]}
    if op == "gmm":
        capi.rand_seed(s["seed"])
        return _model_of(s["g"], s["g"].cluster(s["x"]))
    if op == "em":
        g, (pr, mu, cv) = s["g"], s["init"]
        g.set_priors(pr)
        g.set_means(mu)
        g.set_covariances(cv)
        return _model_of(g, g.em_device(s["x"], case["precision"]))
    if op == "vlad":
        capi.vlad_encode_batch_device(s["enc"], s["means"], s["x"], s["a"], s["off"], case["flags"])
        return {"enc": s["enc"]}
    capi.pca_project_device(s["out"], s["x"], s["proj"], s["centre"], True, s["frames"], s["off"], s["sizes"])
    return {"out": s["out"]}


# -------------------------------------------------------------------- work
def work(case):
    op, d = case["op"], case["d"]
    k = case.get("k", 0)
    n = case["n"] if "n" in case else int(_offsets(case)[-1])
    if op.startswith("fv"):
        b = 8 if case.get("double") else 4
        images = case.get("images", 1)
        return {"bytes": b * (n * d + (2 * d + 1) * k + images * 2 * k * d), "flops": 8.0 * k * d * n}
    if op in ("gmm", "em"):
        flops = (8.0 * case["iters"] + 4.0) * k * d * n
        if op == "gmm":  # one distance per row and centre to seed; about six assignments of every row for KMeans
            flops += (1 if case["init"] == "rand" else 6) * 3.0 * k * d * n
        return {"bytes": 4 * (n * d + 2 * (2 * d + 1) * k), "flops": flops}
    if op == "vlad":
        return {"bytes": 4 * (n * (d + k) + k * d + case["images"] * k * d), "flops": 2.0 * n * d}
    m, xy = case["m"], 2 if case["xy"] else 0
    return {"bytes": 4 * (n * (d + xy + m + xy) + m * d), "flops": 2.0 * n * d * m}


# ------------------------------------------------------------------- exact
def _logits(x, pr, mu, cv):
    """log(pi_k N(x_i; mu_k, cv_k)) in 64 bits; -inf for priors below 1e-6."""
    d = x.shape[1]
    iv = 1.0 / cv
    c = torch.log(pr) - 0.5 * (d * math.log(2 * math.pi) + torch.log(cv).sum(1) + (mu * mu * iv).sum(1))
    c = torch.where(pr >= 1e-6, c, torch.full_like(c, -math.inf))
    return c + x @ (mu * iv).T - 0.5 * (x * x) @ iv.T


def _fisher64(x, off, pr, mu, cv, flags):
    k, d = mu.shape
    out = torch.empty((len(off) - 1, 2 * k * d), dtype=torch.float64, device=DEV)
    sd = torch.sqrt(cv)
    for j in range(len(off) - 1):
        a, b = int(off[j]), int(off[j + 1])
        xj = x[a:b].double()
        q = torch.softmax(_logits(xj, pr, mu, cv), 1)
        q = torch.where((q >= 1e-6) & (pr >= 1e-6), q, torch.zeros_like(q))
        s0, s1, s2 = q.sum(0)[:, None], q.T @ xj, q.T @ (xj * xj)
        nn = max(1, b - a)
        u = (s1 - mu * s0) / sd / (nn * torch.sqrt(pr))[:, None]
        v = ((s2 - 2 * mu * s1 + mu * mu * s0) / cv - s0) / (nn * torch.sqrt(2 * pr))[:, None]
        keep = (pr >= 1e-6)[:, None]
        z = torch.cat([torch.where(keep, u, 0 * u).reshape(-1), torch.where(keep, v, 0 * v).reshape(-1)])
        if flags & 1:
            z = torch.sign(z) * torch.sqrt(z.abs())
        if flags & 2:
            z = z / z.norm().clamp_min(1e-12)
        out[j] = z
    return out


def _em64(x, pr, mu, cv, lb, iters):
    n, (k, d) = x.shape[0], mu.shape
    step = max(4096, (1 << 27) // k)
    cv = cv.clamp_min(lb)
    for it in range(iters + 1):
        ll = 0.0
        s0 = torch.zeros((k, 1), dtype=torch.float64, device=DEV)
        s1, s2 = torch.zeros_like(mu), torch.zeros_like(mu)
        for i in range(0, n, step):
            xb = x[i:i + step].double()
            lg = _logits(xb, pr, mu, cv)
            lse = torch.logsumexp(lg, 1)
            ll += float(lse.sum())
            q = torch.exp(lg - lse[:, None])
            q = torch.where(q >= 1e-2 / k, q, torch.zeros_like(q))
            s0 += q.sum(0)[:, None]
            s1 += q.T @ xb
            s2 += q.T @ (xb * xb)
        if it == iters:
            return pr, mu, cv, ll
        live = s0 >= 1e-6 / k
        div = torch.where(live, s0, torch.ones_like(s0))
        new = s1 / div
        v = (s2 - 2 * mu * s1 + mu * mu * s0) / div
        v = torch.where(live, v - (new - mu) ** 2, v)
        mu, cv = new, v.clamp_min(lb)
        pr = s0[:, 0] / s0.sum().clamp_min(1e-12)
    return None


def exact(case, seed):
    op = case["op"]
    if op.startswith("fv"):
        pr, mu, cv = (torch.from_numpy(v).to(DEV).double() for v in _fv_model(case, seed))
        off = np.array([0, case["n"]], np.int64) if "n" in case else _offsets(case)
        x = _pca_like(int(off[-1]), case["d"], seed)
        enc = _fisher64(x, off, pr, mu, cv, case["flags"])
        return {"enc": enc[0] if op == "fv_host" else enc, "nt": None}
    if op == "em":
        x, pr, mu, cv, lb = _em_inputs(case, seed)
        pr, mu, cv = (torch.from_numpy(v).to(DEV).double() for v in (pr, mu, cv))
        pr, mu, cv, ll = _em64(x, pr, mu, cv, lb, case["iters"])
        return {"means": mu, "covs": cv, "priors": pr, "ll": ll}
    if op == "vlad":
        off, x, means, a = _vlad_inputs(case, seed)
        k, d = means.shape
        out = torch.empty((case["images"], k * d), dtype=torch.float64, device=DEV)
        for j in range(case["images"]):
            b0, b1 = int(off[j]), int(off[j + 1])
            aj = a[b0:b1].double()
            v = aj.T @ x[b0:b1].double() - aj.sum(0)[:, None] * means.double()
            if case["flags"] & 2:
                v = torch.sign(v) * torch.sqrt(v.abs())
            if case["flags"] & 1:
                v = v / v.norm(dim=1, keepdim=True).clamp_min(1e-12)
            out[j] = (v / v.norm().clamp_min(1e-12)).reshape(-1)
        return {"enc": out}
    if op == "pca":
        off, x, proj, centre, frames, sizes = _pca_inputs(case, seed)
        out = torch.empty((x.shape[0], case["m"] + (2 if case["xy"] else 0)), dtype=torch.float64, device=DEV)
        for i in range(0, x.shape[0], 1 << 20):
            y = (x[i:i + (1 << 20)].double() - centre.double()) @ proj.double().T
            out[i:i + (1 << 20), :case["m"]] = y / y.norm(dim=1, keepdim=True).clamp_min(1e-12)
        if case["xy"]:
            img = torch.repeat_interleave(torch.arange(case["images"], device=DEV),
                                          torch.from_numpy(np.diff(off)).to(DEV))
            wh = sizes.double()[img]
            out[:, case["m"]:] = (frames.double() - wh / 2) / wh
        return {"out": out}
    # The initialisations draw from the library's own generator and order.
    return None
