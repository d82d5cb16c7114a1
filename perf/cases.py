"""Performance cases of the annealed EM step, through the package's public entry points.

Five kinds of call, as programs make them:

* ``em``: the temperature loop itself (``Context.set_Y`` on the starting
  centres, then ``anneal`` for ``iters`` iterations, then ``Context.get_Y``),
  in every precision form, on 0/1 fingerprints and on real-valued mixtures,
  with either M-step solver, annealed (``isda`` 1) or plain EM (``isda`` 0).
* ``map``: what a run writes at its end: the E-step on the final centres, the
  posterior-mean map of every point and rows of the responsibilities.
* ``ctemp``: the AUTO schedule's next critical temperature, after an E-step.
* ``fe``: the free energy of a batch and its gradients in the centres, the
  data and beta, through autograd.
* ``project``: held-out points moved onto a fixed map (forward and gradient,
  ``steps`` times).

The data are seeded stand-ins with the shapes the package's configurations
name: a Gaussian mixture, or binary vectors copied from prototypes with bits
flipped.  The starting centres lie on a smooth random sheet through the data,
as they do in the middle of a run, and the basis width (0.5 times the spacing
of the basis centres) keeps the normal equations well conditioned, so that W
and Y are determined by the data.
"""
import importlib
import math

import numpy as np
import torch

pkg = importlib.import_module("da-gtm_gb300")
autograd = importlib.import_module("da-gtm_gb300.autograd")

WIDTH = 0.5


def listed():
    return [
        # A small real-valued data set run to the end on the defaults: the size of the
        # reference's own sample (N = 1000, D = 12); latency and launches decide.
        dict(name="em_small", kind="em", form="fp64", data="gmm", n=1000, d=12, latent=2, g=20, m=4,
             solver="cholesky", isda=1, iters=20, beta=60.0, temp=1.5),
        # The same kind of run with the reference's pseudo-inverse in place of Cholesky,
        # on a ragged size.
        dict(name="em_small_svd", kind="em", form="fp64", data="gmm", n=877, d=9, latent=2, g=15, m=5,
             solver="svd", isda=1, iters=10, beta=60.0, temp=1.2),
        # Mid-sized real-valued data in full FP64, plain EM after the annealing.
        dict(name="em_mid", kind="em", form="fp64", data="gmm", n=20011, d=37, latent=2, g=45, m=7,
             solver="cholesky", isda=0, iters=3, beta=25.0, temp=1.0),
        # 100,000 fingerprints of 166 bits on a 20^3 map (the fp_n100k configuration) in the
        # FP32 form and in the FP64 form.
        dict(name="em_fp32", kind="em", form="fp32", data="fp", n=100000, d=166, latent=3, g=20, m=4,
             solver="cholesky", isda=1, iters=2, beta=6.0, temp=2.0),
        dict(name="em_fp64_bits", kind="em", form="fp64", data="fp", n=100000, d=166, latent=3, g=20, m=4,
             solver="cholesky", isda=1, iters=2, beta=6.0, temp=2.0),
        # The headline: 1,000,000 fingerprints on a 20^3 map in the split form (fp_n1m).
        dict(name="em_headline", kind="em", form="bf16x3", data="fp", n=1000000, d=166, latent=3, g=20, m=4,
             solver="cholesky", isda=1, iters=4, beta=6.0, temp=2.0),
        # Real-valued data in the split form (the shape of gmm_n65k).
        dict(name="em_split_gmm", kind="em", form="bf16x3", data="gmm", n=65536, d=64, latent=2, g=64, m=4,
             solver="cholesky", isda=1, iters=5, beta=20.0, temp=1.5),
        # The large map: 32^3 centres, 8^3 basis functions (fp_n4m's K and M), on a sample
        # of the points.
        dict(name="em_large_basis", kind="em", form="bf16x3", data="fp", n=100000, d=166, latent=3, g=32, m=8,
             solver="cholesky", isda=1, iters=2, beta=6.0, temp=2.0),
        # The end of a fingerprint run: map of every point and rows of R for the output file.
        dict(name="map_output", kind="map", form="bf16x3", data="fp", n=50000, d=166, latent=3, g=20, m=4,
             beta=8.0, temp=1.0, rows=16),
        # One step of the AUTO schedule on real-valued data in FP64.
        dict(name="ctemp_auto", kind="ctemp", form="fp64", data="gmm", n=20000, d=64, latent=3, g=5, m=2,
             beta=2.0, temp=6.0),
        # Gradient-based refinement: free energy and all gradients (the shape of gmm_n65k).
        dict(name="fe_grad", kind="fe", n=65536, d=64, k=4096, beta=20.0, temp=1.5),
        # Projection of a batch of held-out points onto a trained map.
        dict(name="project", kind="project", n=10007, d=64, k=1024, steps=10, beta=20.0, temp=1.0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _cost_ms(c):
    """A rough time of one pass, to keep drawn cases within the listed ones."""
    if c["kind"] in ("fe", "project"):
        return c["n"] * c["k"] * (c["d"] + 60) * 3e-11 * c.get("steps", 1)
    pairs, d = c["n"] * c["g"] ** c["latent"], c["d"]
    bits = c["data"] == "fp"
    if c["kind"] == "map":
        return pairs * (d + 40) * 3e-9
    if c["kind"] == "ctemp":
        return pairs * d * d * (6e-9 if c["form"] == "fp64" else 3e-10)
    per = {"fp64": 2e-8 if bits else (3 * d + 75) * 3e-9, "fp32": (3 * d + 60) * 2e-10,
           "bf16x3": (d + 60) * 8e-12}[c["form"]]
    m1 = c["m"] ** c["latent"] + 1
    solve = c["g"] ** c["latent"] * m1 * (m1 + 2 * d) * 2.5e-9
    return c["iters"] * (pairs * per + solve)


def draw(rng):
    while True:
        c = _draw(rng)
        w = work(c)
        if _cost_ms(c) <= 30.0 and w["flops"] <= 8e12:
            return c


def _draw(rng):
    kind = rng.choice(["em"] * 7 + ["map", "map", "ctemp", "fe", "project"])
    if kind == "fe":
        return dict(kind=kind, n=_log_int(rng, 300, 65536), d=_log_int(rng, 2, 189), k=_log_int(rng, 64, 4096),
                    beta=rng.choice([10.0, 20.0]), temp=rng.choice([1.0, 1.5, 2.0]))
    if kind == "project":
        return dict(kind=kind, n=_log_int(rng, 300, 30000), d=_log_int(rng, 2, 189), k=_log_int(rng, 64, 4096),
                    steps=rng.randint(3, 12), beta=rng.choice([10.0, 20.0]), temp=1.0)
    data = rng.choice(["gmm", "fp"])
    d = _log_int(rng, 32, 189) if data == "fp" else _log_int(rng, 3, 120)
    latent = rng.choice([2, 3])
    if kind == "ctemp":
        g = rng.randint(4, 12) if latent == 2 else rng.randint(3, 6)
        return dict(kind=kind, form=rng.choice(["fp64", "fp64", "bf16x3"]), data=data, n=_log_int(rng, 300, 30000),
                    d=d, latent=latent, g=g, m=2, beta=2.0, temp=6.0)
    g = _log_int(rng, 8, 64) if latent == 2 else _log_int(rng, 5, 24)
    form = rng.choice(["fp64", "fp64", "fp32", "bf16x3"])
    beta = 6.0 if data == "fp" else rng.choice([10.0, 20.0])
    temp = rng.choice([1.2, 1.5, 2.0])
    if kind == "map":
        return dict(kind=kind, form=form, data=data, n=_log_int(rng, 300, 100000), d=d, latent=latent, g=g,
                    m=rng.randint(2, 4), beta=beta, temp=temp, rows=rng.randint(1, 16))
    m = rng.randint(3, min(9, g // 2)) if latent == 2 else rng.randint(2, min(6, g // 2))
    return dict(kind=kind, form=form, data=data, n=_log_int(rng, 300, 300000), d=d, latent=latent, g=g, m=m,
                solver=rng.choice(["cholesky", "cholesky", "svd"]) if m ** latent <= 64 else "cholesky",
                isda=rng.choice([1, 1, 0]), iters=rng.randint(2, 6), beta=beta, temp=temp)


# ---- inputs (plain torch / numpy) ---------------------------------------------------

def _axes(latent, g):
    return np.stack(np.meshgrid(*[np.linspace(-1.0, 1.0, g)] * latent, indexing="ij"), axis=-1).reshape(-1, latent)


def _basis(latent, g, m):
    """Latent grid (g^latent points) and Gaussian basis functions on m^latent centres, and a bias."""
    x = _axes(latent, g)
    mu = _axes(latent, m) * (m / (m - 1.0))
    sigma = WIDTH * 2.0 / (m - 1.0) * (m / (m - 1.0))
    e = np.exp(((x[:, None, :] - mu[None, :, :]) ** 2).sum(2) * (-0.5 / sigma ** 2))
    return x, np.concatenate([e, np.ones((len(x), 1))], axis=1)


def _data(gen, kind, n, d):
    if kind == "gmm":
        means = torch.rand((16, d), generator=gen, device="cuda", dtype=torch.float64)
        at = torch.randint(0, 16, (n,), generator=gen, device="cuda")
        return means[at] + 0.2 * torch.randn((n, d), generator=gen, device="cuda", dtype=torch.float64)
    p = 0.05 + 0.45 * torch.rand(d, generator=gen, device="cuda", dtype=torch.float64)
    protos = torch.rand((20, d), generator=gen, device="cuda", dtype=torch.float64) < p
    out = torch.empty((n, d), device="cuda", dtype=torch.float64)
    for s in range(0, n, 1 << 17):
        e = min(n, s + (1 << 17))
        at = torch.randint(0, 20, (e - s,), generator=gen, device="cuda")
        out[s:e] = protos[at] ^ (torch.rand((e - s, d), generator=gen, device="cuda") < 0.1)
    return out


def _sheet(gen, t, x):
    """Centres on a smooth random sheet over the latent points x, with the data's mean and spread."""
    x = torch.from_numpy(x).cuda()
    d = t.shape[1]
    freq = torch.randn((x.shape[1], 12), generator=gen, device="cuda", dtype=torch.float64) * 1.5
    phase = 6.2832 * torch.rand(12, generator=gen, device="cuda", dtype=torch.float64)
    mix = torch.randn((12, d), generator=gen, device="cuda", dtype=torch.float64) / math.sqrt(6.0)
    return t.mean(0) + 0.8 * t.std(0) * (torch.sin(x @ freq + phase) @ mix)


def _inputs(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    if case["kind"] in ("fe", "project"):
        t = _data(gen, "gmm", case["n"], case["d"])
        y = _sheet(gen, t, 2.0 * torch.rand((case["k"], 2), generator=gen, device="cuda", dtype=torch.float64).cpu().numpy() - 1.0)
        return t.float(), y.float(), None, None
    x, fi = _basis(case["latent"], case["g"], case["m"])
    t = _data(gen, case["data"], case["n"], case["d"])
    return t, _sheet(gen, t, x), x, fi


# ---- the measured passes ------------------------------------------------------------

def prepare(case, seed):
    t, y, x, fi = _inputs(case, seed)
    if case["kind"] == "fe":
        beta = torch.tensor(case["beta"], dtype=torch.float64, device="cuda", requires_grad=True)
        return dict(case=case, t=t.requires_grad_(True), y=y.requires_grad_(True), beta=beta)
    if case["kind"] == "project":
        return dict(case=case, t=t, y=y)
    ctx = pkg.Context(t.cpu().numpy(), fi, case["form"], case.get("solver", "cholesky"))
    y = y.cpu().numpy()
    ctx.set_Y(y)
    return dict(case=case, ctx=ctx, y=y, x=x)


def run(state):
    c = state["case"]
    if c["kind"] == "fe":
        f = autograd.free_energy(state["y"], state["t"], state["beta"], c["temp"])
        dy, dt, db = torch.autograd.grad(f, (state["y"], state["t"], state["beta"]))
        return dict(f=f.detach(), dy=dy, dt=dt, db=db)
    if c["kind"] == "project":
        return dict(t=autograd.project(state["t"], state["y"], c["beta"], c["temp"], steps=c["steps"]))
    ctx = state["ctx"]
    if c["kind"] == "em":
        ctx.set_Y(state["y"])
        res = pkg.anneal(ctx, c["beta"], c["temp"], isDA=c["isda"], eps=0.0, maxloop=c["iters"])
        return dict(nfree=np.array(res.nfree_trace), llh=np.array(res.llh_trace), beta=np.array(res.beta_trace[1:] + [res.beta]),
                    w=res.W, y=ctx.get_Y())
    llh, nfree = ctx.estep(c["beta"], 1, c["temp"])
    if c["kind"] == "map":
        return dict(q=np.array([llh, nfree]), m=ctx.map(state["x"]), r=ctx.R_block(0, c["rows"], 0, c["n"]))
    ctemp, per_centre = ctx.next_ctemp(c["temp"], c["beta"], 1e-6, per_centre=True)
    return dict(q=np.array([llh, nfree]), ctemp=np.array([ctemp]), per_centre=per_centre)


def work(case):
    n, d = case["n"], case["d"]
    if case["kind"] in ("fe", "project"):
        k, steps = case["k"], case.get("steps", 1)
        products = 3 if case["kind"] == "fe" else 2  # distances, R T and R^T Y (project: distances and R^T Y)
        return {"bytes": steps * 8.0 * (n + k) * d, "flops": steps * products * 2.0 * n * k * d}
    k, m1 = case["g"] ** case["latent"], case["m"] ** case["latent"] + 1
    held = {"fp64": 8, "fp32": 4, "bf16x3": 2 if case["data"] == "fp" else 4}[case["form"]]  # bytes of a resident value of T
    if case["kind"] == "em":
        return {"bytes": case["iters"] * (held * n * d + 8.0 * (k * m1 + k * d + m1 * d)),
                "flops": case["iters"] * (4.0 * n * k * d + 2.0 * k * m1 * (m1 / 2 + 2 * d))}
    if case["kind"] == "map":
        return {"bytes": held * n * d + 8.0 * (k * d + n * case["latent"] + n * case["rows"]),
                "flops": 2.0 * n * k * (d + case["latent"])}
    return {"bytes": held * n * d + 8.0 * k * d, "flops": 2.0 * n * k * (d + d * (d + 1))}


# ---- the same in 64 bits, in plain torch ----------------------------------------------

def _blocks(n, k):
    step = max(256, (1 << 28) // k)
    return [(s, min(n, s + step)) for s in range(0, n, step)]


def _distances(t, y):
    return ((t * t).sum(1)[:, None] - 2.0 * (t @ y.T)) + (y * y).sum(1)[None, :]


def _quality(beta, temp, isda, n, d, k, s1, s2):
    base = n * (d / 2.0 * math.log(beta / (2.0 * math.pi)) - math.log(k))
    llh = (base + s1) / n
    return llh, (base + temp * s2) / n if isda else -llh


def _step(t, y, beta, temp, isda, fi):
    """One EM iteration: qualities, W, Y and beta."""
    n, d = t.shape
    k = y.shape[0]
    g = torch.zeros(k, device="cuda", dtype=torch.float64)
    rt = torch.zeros_like(y)
    s1 = s2 = 0.0
    for s, e in _blocks(n, k):
        v = _distances(t[s:e], y).mul_(-0.5 * beta)
        s1 += float(torch.logsumexp(v, 1).sum())
        if isda:
            v /= temp
        lse = torch.logsumexp(v, 1)
        s2 += float(lse.sum())
        v = v.sub_(lse[:, None]).exp_()
        g += v.sum(0)
        rt += v.T @ t[s:e]
    llh, nfree = _quality(beta, temp, isda, n, d, k, s1, s2)
    w = torch.linalg.solve(fi.T @ (g[:, None] * fi), fi.T @ rt)
    y = fi @ w
    cross = float((g * (y * y).sum(1)).sum() - 2.0 * (y * rt).sum() + (t * t).sum())
    return llh, nfree, w, y, n * d / cross


def exact(case, seed):
    t, y, x, fi = _inputs(case, seed)
    t, y = t.double(), y.double()
    n, d = t.shape
    k = y.shape[0]
    beta, temp = case["beta"], case["temp"]
    if case["kind"] == "em":
        if 6.0 * n * k * d * case["iters"] > 1.2e13:
            return None
        fi = torch.from_numpy(fi).cuda()
        out = dict(nfree=[], llh=[], beta=[])
        for _ in range(case["iters"]):
            llh, nfree, w, y, beta = _step(t, y, beta, temp, case["isda"], fi)
            out["nfree"].append(nfree)
            out["llh"].append(llh)
            out["beta"].append(beta)
        return dict({key: np.array(v) for key, v in out.items()}, w=w.cpu().numpy(), y=y.cpu().numpy())
    if case["kind"] == "project":
        for _ in range(case["steps"]):
            for s, e in _blocks(n, k):
                r = torch.softmax(_distances(t[s:e], y) * (-beta / (2.0 * temp)), 1)
                t[s:e] -= t[s:e] - r @ y
        return dict(t=t)
    s1 = s2 = 0.0
    m = torch.zeros((n, case.get("latent", 1)), device="cuda", dtype=torch.float64)
    rows = torch.zeros((case.get("rows", 1), n), device="cuda", dtype=torch.float64)
    dt, rt = torch.zeros_like(t), torch.zeros_like(y)
    g = torch.zeros(k, device="cuda", dtype=torch.float64)
    full, rd = [], 0.0
    for s, e in _blocks(n, k):
        v = _distances(t[s:e], y)
        s1 += float(torch.logsumexp(v * (-0.5 * beta), 1).sum())
        lse = torch.logsumexp(v * (-0.5 * beta / temp), 1)
        s2 += float(lse.sum())
        r = torch.exp(v * (-0.5 * beta / temp) - lse[:, None])
        if case["kind"] == "map":
            m[s:e] = r @ torch.from_numpy(x).cuda()
            rows[:, s:e] = r[:, :case["rows"]].T
        elif case["kind"] == "ctemp":
            full.append(r.T.contiguous())
        else:
            dt[s:e] = -beta * (t[s:e] - r @ y)
            g += r.sum(0)
            rt += r.T @ t[s:e]
            rd += float((r * v).sum())
    q = np.array(_quality(beta, temp, 1, n, d, k, s1, s2))
    if case["kind"] == "map":
        return dict(q=q, m=m.cpu().numpy(), r=rows.cpu().numpy())
    if case["kind"] == "fe":
        base = n * (d / 2.0 * math.log(beta / (2.0 * math.pi)) - math.log(k))
        return dict(f=base + temp * s2, dy=-beta * (g[:, None] * y - rt), dt=dt, db=n * d / (2.0 * beta) - 0.5 * rd)
    r = torch.cat(full, 1)
    vals = []
    for j in range(k):
        z = t - y[j]
        a = (z * r[j][:, None]).T @ z
        b = (z * (r[j] ** 2)[:, None]).T @ z
        lam = torch.linalg.eigvalsh(torch.stack([2.0 * a, 2.0 * (a - b)]))
        gk = float(r[j].sum())
        lam = torch.where(lam >= (temp - 1e-6) * 2.0 * gk / beta, torch.zeros_like(lam), lam)
        vals.append(beta / 2.0 / gk * float(lam.max()))
    return dict(q=q, ctemp=np.array([max(vals)]), per_centre=np.array(vals))
