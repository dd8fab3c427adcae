"""The work that users of this framework have it do, through its public entry
points, as a set of measurable cases.

A case names a kind of work and its sizes:

  ops     one hand-written Krylov step on device vectors: b = M T (+ dt F),
          y = A x, z = y / diag, x.y (build_rhs_ptr, apply_ptr, precond_ptr,
          dot_ptr) -- what a program that brings its own solver calls;
  pcg     one Jacobi-PCG solve of A x = b on device vectors (pcg_ptr);
  solve   implicit-Euler steps of a host field (solve_host): the drop-in;
  case    a detector run with its per-step records (run_case), against a kept
          reference trajectory: the fault-study form;
  batch   an ensemble of independent solves through the batched
          mixed-precision engine: admitted, stepped to the end, read back and
          removed (add, step, field, remove);
  field   a lognormal conductivity field generated on the device
          (field_lognormal).

Fields are the reference generator's law (lognormal, Gaussian correlation),
drawn here with torch; `exact` solves the same problems with plain torch in
64 bits (dense 8x8 element matrices, PCG to a much tighter tolerance).
"""
import math

import numpy as np
import torch

from mnhack8_b200 import _lib

SIGMA_IC = 0.15


def listed():
    return [
        # a small grid in a user's own Krylov loop: call latency is all there is
        {"name": "ops-n16", "kind": "ops", "n": 16, "form": "wht", "scatter": "colored", "dt": 1e-3, "sigma": 1.0,
         "corr": 4.0},
        # the same at the size of the FP64 benchmark problem
        {"name": "ops-n128", "kind": "ops", "n": 128, "form": "wht", "scatter": "colored", "dt": 1e-4, "sigma": 1.0,
         "corr": 8.0},
        # the reference's own defaults: dense element matrices, atomic scatter
        {"name": "ops-atomic-n64", "kind": "ops", "n": 64, "form": "fast", "scatter": "atomic", "dt": 1e-3,
         "sigma": 1.0, "corr": 8.0},
        # one small solve: a coarse model inside an outer loop
        {"name": "pcg-n24", "kind": "pcg", "n": 24, "dt": 1e-3, "sigma": 1.0, "corr": 4.0, "rtol": 1e-8},
        # one mid-size solve on an odd grid
        {"name": "pcg-n65", "kind": "pcg", "n": 65, "dt": 2e-4, "sigma": 1.0, "corr": 8.0, "rtol": 1e-10},
        # the smallest named configuration: 8^3 elements, homogeneous, dense form, 10 steps, checksum on
        {"name": "solve-n8", "kind": "solve", "n": 8, "form": "fast", "dt": 1e-3, "sigma": 0.0, "corr": 1.0,
         "rtol": 1e-10, "steps": 10},
        # the benchmark trajectory's problem (N=128, lognormal, rtol 1e-10), ten of its steps
        {"name": "solve-n128", "kind": "solve", "n": 128, "form": "wht", "dt": 1e-4, "sigma": 1.0, "corr": 8.0,
         "rtol": 1e-10, "steps": 10},
        # the large named grid, strongly heterogeneous
        {"name": "solve-n256", "kind": "solve", "n": 256, "form": "wht", "dt": 1e-4, "sigma": 1.5, "corr": 16.0,
         "rtol": 1e-8, "steps": 2},
        # a fault-study run: source on, dense form, every detector, snapshots against a kept reference
        {"name": "case-n48", "kind": "case", "n": 48, "form": "fast", "dt": 1e-3, "sigma": 1.0, "corr": 6.0,
         "rtol": 1e-8, "steps": 10},
        # an uneven ensemble, N uniform in 16..96, 20 steps: the batching configuration at a tenth of its count
        {"name": "batch-16-96", "kind": "batch", "count": 24, "n_lo": 16, "n_hi": 96, "dt": 1e-4, "sigma": 1.0,
         "steps": 20},
        # one large strongly heterogeneous instance: the precision form
        {"name": "batch-n160", "kind": "batch", "count": 1, "n_lo": 160, "n_hi": 160, "dt": 1e-4, "sigma": 1.5,
         "steps": 10},
        # a conductivity field for a served request
        {"name": "field-n128", "kind": "field", "n": 128, "corr": 8.0, "sigma": 1.0},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["ops", "ops", "pcg", "pcg", "solve", "solve", "case", "batch", "field"])
    dt = 10.0 ** rng.uniform(-4.0, -3.0)
    sigma = rng.choice([0.5, 1.0, 1.5])
    if kind == "ops":
        scatter = rng.choice(["colored", "colored", "atomic"])
        return {"kind": kind, "n": size(8, 200), "form": rng.choice(["wht", "wht", "fast"]), "scatter": scatter,
                "dt": dt, "sigma": sigma, "corr": rng.choice([4.0, 8.0])}
    if kind == "pcg":
        return {"kind": kind, "n": size(12, 160), "dt": dt, "sigma": sigma, "corr": rng.choice([4.0, 8.0]),
                "rtol": rng.choice([1e-8, 1e-10])}
    if kind == "solve":
        n = size(8, 160)
        return {"kind": kind, "n": n, "form": rng.choice(["wht", "wht", "fast"]) if n < 100 else "wht", "dt": dt,
                "sigma": sigma, "corr": rng.choice([4.0, 8.0]), "rtol": rng.choice([1e-8, 1e-10]),
                "steps": rng.randint(1, 4) if n > 64 else rng.randint(2, 10)}
    if kind == "case":
        return {"kind": kind, "n": size(8, 72), "form": rng.choice(["wht", "fast", "gauss"]), "dt": dt,
                "sigma": sigma, "corr": 6.0, "rtol": 1e-8, "steps": rng.randint(3, 8)}
    if kind == "batch":
        lo = size(12, 48)
        return {"kind": kind, "count": rng.randint(2, 16), "n_lo": lo, "n_hi": min(96, 2 * lo + rng.randint(0, 9)),
                "dt": dt, "sigma": sigma, "steps": rng.randint(3, 12)}
    return {"kind": kind, "n": size(16, 160), "corr": rng.choice([4.0, 8.0, 16.0]), "sigma": sigma}


# ---- inputs ------------------------------------------------------------------
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) & 0x7FFFFFFF)
    return g


def _field(n, sigma, corr, gen):
    """k, rho*c of n^3 elements (device, float64): lognormal k with Gaussian
    correlation of `corr` elements, rho*c = 1 (the reference generator's law);
    sigma 0 is the homogeneous field k = 1."""
    one = torch.ones(n ** 3, dtype=torch.float64, device="cuda")
    if sigma == 0.0:
        return one.clone(), one
    w = torch.randn(n, n, n, dtype=torch.float64, device="cuda", generator=gen)
    f = 2.0 * math.pi * torch.fft.fftfreq(n, dtype=torch.float64, device="cuda")
    fz = 2.0 * math.pi * torch.fft.rfftfreq(n, dtype=torch.float64, device="cuda")
    k2 = (f[:, None, None] ** 2 + f[None, :, None] ** 2 + fz[None, None, :] ** 2) * corr ** 2 / 8.0
    g = torch.fft.irfftn(torch.fft.rfftn(w) * torch.exp(-k2), s=(n, n, n))
    g = (g - g.mean()) / g.std(unbiased=False)
    return torch.exp(sigma * g).reshape(-1), one


def _interior(n):
    m = torch.zeros(n + 1, n + 1, n + 1, dtype=torch.float64, device="cuda")
    m[1:-1, 1:-1, 1:-1] = 1.0
    return m


def _bump(n, gen, shift=0.05):
    """A Gaussian bump of width SIGMA_IC near the centre, zero on the faces."""
    c = 0.5 + shift * (torch.rand(3, dtype=torch.float64, device="cuda", generator=gen) - 0.5) * 2.0
    t = torch.linspace(0.0, 1.0, n + 1, dtype=torch.float64, device="cuda")
    e = [torch.exp(-((t - c[i]) ** 2) / (2.0 * SIGMA_IC ** 2)) for i in range(3)]
    return (e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :] * _interior(n)).reshape(-1)


def _sizes(case):
    rng = np.random.default_rng(1000 + case["count"])
    return [int(v) for v in rng.integers(case["n_lo"], case["n_hi"] + 1, size=case["count"])]


def _inputs(case, seed):
    gen = _gen(seed)
    n = case["n"]
    k, r = _field(n, case["sigma"], case["corr"], gen)
    return gen, n, k, r


def _batch_inputs(case, seed):
    gen = _gen(seed)
    out = []
    for n in _sizes(case):
        k, r = _field(n, case["sigma"], n / 8.0, gen)
        out.append((n, k, r, _bump(n, gen)))
    return out


def prepare(case, seed):
    kind = case["kind"]
    if kind == "field":
        n = case["n"]
        return {"case": case, "seed": int(seed), "k": torch.empty(n ** 3, dtype=torch.float64, device="cuda"),
                "r": torch.empty(n ** 3, dtype=torch.float64, device="cuda")}
    if kind == "batch":
        inst = [(n, k.cpu().numpy(), r.cpu().numpy(), t.cpu().numpy()) for n, k, r, t in _batch_inputs(case, seed)]
        return {"case": case, "batch": _lib.Batch(rtol=1e-8), "inst": inst}
    gen, n, k, r = _inputs(case, seed)
    kw = {"kernel": case.get("form", "wht"), "scatter": case.get("scatter", "colored"), "detect": True,
          "no_source": kind != "case", "ic": "gaussian", "ic_sigma": SIGMA_IC, "rtol": case.get("rtol", 1e-8),
          "max_iter": 1000}
    s = {"case": case, "solver": _lib.Solver(n, case["dt"], k.cpu().numpy(), r.cpu().numpy(), **kw)}
    if kind == "ops":
        s["T"] = _bump(n, gen)
        s["x"] = torch.randn((n + 1) ** 3, dtype=torch.float64, device="cuda", generator=gen) * _interior(n).reshape(-1)
        for name in ("b", "y", "z"):
            s[name] = torch.zeros_like(s["T"])
    elif kind == "pcg":
        # a warm start near the solution's scale and a smooth right-hand side, as a time step has them
        s["x0"] = _bump(n, gen)
        s["b"] = _bump(n, gen) / n ** 3
        s["x"] = torch.empty_like(s["x0"])
    elif kind == "solve":
        s["T0"] = _bump(n, gen).cpu().numpy()
    else:
        s["solver"].run_case(case["steps"], snap_every=5, keep_reference=True, want_T=False)
    torch.cuda.synchronize()
    return s


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "field":
        n = case["n"]
        _lib.field_lognormal(n, 0.0, case["sigma"], case["corr"] / n, s["seed"], 1.0, s["k"].data_ptr(),
                             s["r"].data_ptr())
        return {"k": s["k"], "rhoc": s["r"]}
    if kind == "batch":
        b = s["batch"]
        slots = [b.add(n, case["dt"], k, r, T0=t, steps=case["steps"]) for n, k, r, t in s["inst"]]
        while b.step()[0]:
            pass
        out = [b.field(i) for i in slots]
        for i in slots:
            b.remove(i)
        return out
    g = s["solver"]
    if kind == "ops":
        x, y = s["x"].data_ptr(), s["y"].data_ptr()
        g.build_rhs_ptr(s["T"].data_ptr(), s["b"].data_ptr())
        g.apply_ptr(x, y)
        g.precond_ptr(y, s["z"].data_ptr())
        return {"b": s["b"], "y": s["y"], "z": s["z"], "dot": g.dot_ptr(x, y)}
    if kind == "pcg":
        s["x"].copy_(s["x0"])
        torch.cuda.current_stream().synchronize()       # the solver works on a stream of its own
        it = g.pcg_ptr(s["b"].data_ptr(), s["x"].data_ptr(), 1000, case["rtol"])
        return {"x": s["x"], "iterations": it}
    if kind == "solve":
        T, it, _ = g.solve_host(s["T0"], case["steps"])
        return {"T": T, "iterations": it}
    res = g.run_case(case["steps"], snap_every=5)
    st = res["steps"]
    rec = {key: np.array([v[key] for v in st]) for key in ("d1", "d2", "tmin", "tmax", "E", "spread")}
    return {"T": res["T"], "iterations": np.array([v["cg_iters"] for v in st]), "records": rec}


# ---- what a pass cannot do without --------------------------------------------
def _cg_iterations(n, dt, sigma, rtol):
    """Jacobi-PCG iterations of one step, to about 20 %."""
    return math.log(2.0 / rtol) * (1.9 + 1.6 * math.sqrt(dt) * n * math.exp(2.0 * (sigma - 1.0) if sigma > 1 else 0.0))


_FLOPS_ITER = 110.0      # per node and CG iteration, element operator in its factored form
_DENSE = 270.0           # with the dense 8x8 element matrices


def work(case):
    kind = case["kind"]
    if kind == "field":
        ne = case["n"] ** 3
        return {"bytes": 16.0 * ne, "flops": 2.0 * ne * 3 * 6 * case["corr"] + 60.0 * ne}
    if kind == "batch":
        by = fl = 0.0
        for n in _sizes(case):
            it = 1.2 * _cg_iterations(n, case["dt"], case["sigma"], 1e-8)
            nn, ne = (n + 1) ** 3, n ** 3
            by += 16.0 * ne + 16.0 * nn + case["steps"] * (it * (40.0 * nn + 8.0 * ne) + 3 * (40.0 * nn + 16.0 * ne))
            fl += case["steps"] * it * _FLOPS_ITER * nn
        return {"bytes": by, "flops": fl}
    n = case["n"]
    nn, ne = (n + 1) ** 3, n ** 3
    per = _FLOPS_ITER if case.get("form", "wht") == "wht" else _DENSE
    if kind == "ops":
        return {"bytes": 2 * (24.0 * nn + 16.0 * ne) + 24.0 * nn + 16.0 * nn, "flops": (2 * per + 3) * nn}
    it = _cg_iterations(n, case["dt"], case["sigma"], case["rtol"]) + 2
    step_bytes, step_flops = it * (80.0 * nn + 16.0 * ne), it * per * nn
    steps = case.get("steps", 1)
    return {"bytes": steps * step_bytes + 16.0 * nn, "flops": steps * step_flops}


# ---- the same in plain 64-bit torch --------------------------------------------
class _Plain:
    """(M + dt K) with dense Q1 element matrices, Dirichlet-projected."""

    def __init__(self, n, dt, k, r):
        self.n, self.dt = n, dt
        h = 1.0 / n
        m1 = h / 6.0 * torch.tensor([[2.0, 1.0], [1.0, 2.0]], dtype=torch.float64, device="cuda")
        k1 = 1.0 / h * torch.tensor([[1.0, -1.0], [-1.0, 1.0]], dtype=torch.float64, device="cuda")

        def kron(a, b, c):
            return torch.kron(torch.kron(a, b), c)

        self.M = kron(m1, m1, m1)
        self.K = kron(k1, m1, m1) + kron(m1, k1, m1) + kron(m1, m1, k1)
        self.k, self.r = k.reshape(n, n, n), r.reshape(n, n, n)
        self.mask = _interior(n)
        d = self._scatter([self.r * self.M[q, q] + dt * self.k * self.K[q, q] for q in range(8)])
        self.diag = torch.where(self.mask > 0, d, torch.ones_like(d))

    def _corner(self, x, q):
        n = self.n
        a, b, c = (q >> 2) & 1, (q >> 1) & 1, q & 1
        return x[a:n + a, b:n + b, c:n + c]

    def _scatter(self, v):
        y = torch.zeros(self.n + 1, self.n + 1, self.n + 1, dtype=torch.float64, device="cuda")
        for q in range(8):
            self._corner(y, q).add_(v[q])
        return y

    def apply(self, x, dt):
        x = x.reshape(self.mask.shape)
        v = torch.stack([self._corner(x, q) for q in range(8)]).reshape(8, -1)
        out = (self.M @ v) * self.r.reshape(-1)
        if dt:
            out += (self.K @ v) * (dt * self.k).reshape(-1)
        return self._scatter(out.reshape(8, self.n, self.n, self.n)) * self.mask

    def source(self):
        n = self.n
        h = 1.0 / n
        gp = 0.5 / math.sqrt(3.0)
        at = [(torch.arange(n, dtype=torch.float64, device="cuda") + 0.5 + s * gp) * h for s in (-1.0, 1.0)]
        shape = [[0.5 + gp, 0.5 - gp], [0.5 - gp, 0.5 + gp]]        # shape[point][corner]
        v = [torch.zeros(n, n, n, dtype=torch.float64, device="cuda") for _ in range(8)]
        for g in range(8):
            a, b, c = (g >> 2) & 1, (g >> 1) & 1, g & 1
            e = [torch.exp(-((at[i] - 0.5) ** 2) / (2.0 * 0.1 ** 2)) for i in (a, b, c)]
            Q = 1000.0 * e[0][:, None, None] * e[1][None, :, None] * e[2][None, None, :] * h ** 3 / 8.0
            for q in range(8):
                v[q] += Q * (shape[a][(q >> 2) & 1] * shape[b][(q >> 1) & 1] * shape[c][q & 1])
        return self._scatter(v) * self.mask

    def pcg(self, b, x, tol=1e-14, cap=4000):
        """To a relative residual far below any tolerance the cases use; the
        residual is looked at every 16 iterations."""
        b, x = b.reshape(self.mask.shape), x.reshape(self.mask.shape).clone()
        r = b - self.apply(x, self.dt)
        z = r / self.diag
        p, rho = z.clone(), (r * z).sum()
        stop = (tol * b.norm()) ** 2
        for i in range(cap):
            q = self.apply(p, self.dt)
            a = rho / (p * q).sum()
            x += a * p
            r -= a * q
            if i % 16 == 15 and bool((r * r).sum() <= stop):
                break
            z = r / self.diag
            new = (r * z).sum()
            p = z + (new / rho) * p
            rho = new
        return x

    def steps(self, T, count, src=None):
        T = T.reshape(self.mask.shape)
        for _ in range(count):
            b = self.apply(T, 0.0)
            if src is not None:
                b = b + self.dt * src
            T = self.pcg(b, T)
        return T.reshape(-1)


def _exact_field(case, seed):
    n = case["n"]
    ne = n ** 3

    def mix(x):
        x = x + np.uint64(0x9E3779B97F4A7C15)
        x = (x ^ (x >> np.uint64(30))) * np.uint64(0xBF58476D1CE4E5B9)
        x = (x ^ (x >> np.uint64(27))) * np.uint64(0x94D049BB133111EB)
        return x ^ (x >> np.uint64(31))

    with np.errstate(over="ignore"):
        c = mix(np.array([seed], dtype=np.uint64)) + np.uint64(2) * np.arange(ne, dtype=np.uint64)
        u = [((mix(c + np.uint64(i)) >> np.uint64(11)).astype(np.float64) + 1.0) * 2.0 ** -53 for i in (0, 1)]
    g = torch.from_numpy(np.sqrt(-2.0 * np.log(u[0])) * np.cos(2.0 * np.pi * u[1])).cuda().reshape(n, n, n)
    s = 0.5 * case["corr"]
    R = max(1, int(math.ceil(6.0 * (0.5 * (case["corr"] / n) * n))))
    for axis in (2, 1, 0):
        acc = torch.zeros_like(g)
        for t in range(-R, R + 1):
            acc += math.exp(-t * t / (2.0 * s * s)) * torch.roll(g, -t, dims=axis)
        g = acc
    g = (g - g.mean()) / g.std(unbiased=False)
    return {"k": torch.exp(case["sigma"] * g).reshape(-1), "rhoc": torch.ones(ne, dtype=torch.float64)}


def exact(case, seed):
    kind = case["kind"]
    if kind == "field":
        return _exact_field(case, int(seed))
    if kind == "batch":
        if case["count"] * case["steps"] > 250:
            return None                     # more than 20 s of small torch solves
        return [_Plain(n, case["dt"], k, r).steps(t, case["steps"]) for n, k, r, t in _batch_inputs(case, seed)]
    gen, n, k, r = _inputs(case, seed)
    A = _Plain(n, case["dt"], k, r)
    if kind == "ops":
        T = _bump(n, gen)
        x = torch.randn((n + 1) ** 3, dtype=torch.float64, device="cuda", generator=gen) * _interior(n).reshape(-1)
        y = A.apply(x, case["dt"])
        return {"b": A.apply(T, 0.0).reshape(-1), "y": y.reshape(-1), "z": (y / A.diag).reshape(-1),
                "dot": float((x.reshape(y.shape) * y).sum())}
    if kind == "pcg":
        x0 = _bump(n, gen)
        b = _bump(n, gen) / n ** 3
        return {"x": A.pcg(b, x0).reshape(-1), "iterations": None}
    if kind == "solve":
        return {"T": A.steps(_bump(n, gen), case["steps"]), "iterations": None}
    t = torch.linspace(0.0, 1.0, n + 1, dtype=torch.float64, device="cuda")
    e = torch.exp(-((t - 0.5) ** 2) / (2.0 * SIGMA_IC ** 2))
    T0 = e[:, None, None] * e[None, :, None] * e[None, None, :] * _interior(n)
    return {"T": A.steps(T0, case["steps"], A.source()), "iterations": None, "records": None}
