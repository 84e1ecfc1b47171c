"""The workloads that this framework's speed is judged on: what its users have it do, through its
public Python entry points, from one live filter of a few thousand particles to 2^24 particles.

``listed()`` names the cases, ``draw(rng)`` gives more of the same ranges, ``prepare`` builds what a
program holds before the call (its filter and its observations), ``run`` is one pass, ``work`` what
a pass cannot do without, and ``exact`` the same outputs in 64 bits from plain torch: the same
model, the same counter-based PCG32 draws and the same systematic resampling, in FP64 throughout.
Observations come from the matched stochastic-volatility generator (gpubpf.dgp) that the tests and
the benchmark use; the filter's parameters are the generator's.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "bootstrap-particle-filter-in-ptx_b200"))
import gpubpf  # noqa: E402
from gpubpf import dgp  # noqa: E402


def _case(name, kind, **kw):
    base = {"kind": kind, "n": 4096, "ticks": 64, "ess": 0.5, "nu_state": 0.0, "nu_obs": 0.0, "filters": 1,
            "cpmmh": 0.0, "mu": -1.0, "rho": 0.97, "sigma": 0.2}
    base.update(kw)
    return {"name": name, **base}


def listed():
    return [
        # one live filter: every observation is a call that waits for its result (trading loop, 4096 particles)
        _case("live_4096", "live", n=4096, ticks=64),
        # benchmark configuration 1: the textbook filter, resampling on every tick
        _case("series_4096_always", "series", n=4096, ticks=1000, ess=0.0),
        # the matched-DGP suite's filter: 50000 particles, not a multiple of a tile, default ESS rule
        _case("series_50000", "series", n=50000, ticks=1000),
        # the conditional-resampling study: 300000 particles, always resampling (its costliest row) ...
        _case("series_300000_always", "series", n=300000, ticks=500, ess=0.0, mu=-4.5, rho=0.98, sigma=0.16),
        # ... and heavy tails in state and observation at an odd size of about a million
        _case("series_1000003_t", "series", n=1000003, ticks=256, nu_state=5.0, nu_obs=5.0),
        # the headline size: 2^24 particles, device-resident series, ESS < N/2
        _case("device_16777216", "device", n=1 << 24, ticks=256),
        # auxiliary particle filter at the matched-DGP size
        _case("apf_50000", "apf", n=50000, ticks=300, ess=0.0),
        # one iteration of gradient-based estimation: log-likelihood and its gradient, 2^20 particles
        _case("grad_1048576", "grad", n=1 << 20, ticks=200, ess=0.0),
        # many parameter vectors at once (inner loop of SMC^2 / PMMH): ragged particle counts 512..16384
        _case("batch_1024_mixed", "batch", n=0, filters=1024, ticks=200),
        # the same with gradients, equal sizes
        _case("batch_grad_256x8192", "batch_grad", n=8192, filters=256, ticks=100, ess=0.0),
        # interacting multiple models stepped live
        _case("imm_8x4096", "imm", n=4096, filters=8, ticks=64),
        # online posterior over the parameters: a whole SMC^2 run
        _case("smc2_256x512", "smc2", n=512, filters=256, ticks=150),
    ]


def _log_int(rng, lo, hi):
    v = int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))
    return min(hi, max(lo, v))


def draw(rng):
    kind = rng.choice(("live", "series", "series", "series", "device", "apf", "grad", "batch", "batch_grad", "imm",
                       "smc2"))
    c = {"kind": kind, "ess": rng.choice((0.0, 0.5, 0.5)), "nu_state": 0.0, "nu_obs": rng.choice((0.0, 0.0, 0.0, 5.0)),
         "filters": 1, "cpmmh": 0.0, "mu": round(rng.uniform(-4.5, 0.0), 3), "rho": round(rng.uniform(0.85, 0.99), 4),
         "sigma": round(rng.uniform(0.05, 0.4), 3)}
    if kind == "live":
        c.update(n=_log_int(rng, 1000, 1 << 20), ticks=rng.randint(16, 128))
    elif kind == "series":
        c.update(n=_log_int(rng, 1000, 1 << 22), ticks=rng.randint(64, 500), nu_state=rng.choice((0.0, 0.0, 0.0, 5.0, 6.0)))
    elif kind == "device":
        c.update(n=_log_int(rng, 4000, 1 << 24), ticks=rng.randint(32, 200))
    elif kind == "apf":
        c.update(n=_log_int(rng, 1000, 1 << 20), ticks=rng.randint(64, 300), ess=0.0)
    elif kind == "grad":
        c.update(n=_log_int(rng, 4096, 1 << 20), ticks=rng.randint(32, 200), ess=0.0)
    elif kind == "batch":
        c.update(n=rng.choice((0, 0, _log_int(rng, 100, 16384))), filters=_log_int(rng, 16, 1024), ticks=rng.randint(50, 200))
    elif kind == "batch_grad":
        c.update(n=_log_int(rng, 200, 8192), filters=_log_int(rng, 16, 256), ticks=rng.randint(32, 100), ess=0.0)
    elif kind == "imm":
        c.update(n=_log_int(rng, 500, 16384), filters=rng.randint(2, 16), ticks=rng.randint(16, 128), ess=0.5, nu_obs=0.0)
    else:
        c.update(n=_log_int(rng, 64, 1024), filters=rng.randint(32, 384), ticks=rng.randint(50, 150), ess=0.5,
                 nu_obs=0.0, cpmmh=rng.choice((0.0, 0.99)))
    return c


def _series(case, seed, ticks):
    _, y = dgp.matched_series(ticks, case["rho"], case["sigma"], case["mu"], 1 + seed % 1000003,
                              nu_state=case["nu_state"], nu_obs=case["nu_obs"])
    return np.asarray(y, dtype=np.float32)


def _seed(seed):
    return 1 + (seed * 2654435761) % 1000000007


def _sizes(case, seed):
    """Particle counts of a batch: equal, or log-uniform on 512..16384 (benchmark configuration 4)."""
    if case["n"]:
        return [case["n"]] * case["filters"]
    r = np.random.RandomState(4)                    # the counts are part of the case, not of the inputs
    return [int(round(math.exp(v))) for v in r.uniform(math.log(512.0), math.log(16384.0), case["filters"])]


def _batch_filters(case, seed):
    r = np.random.RandomState(seed % (1 << 31))
    fl = []
    for b, n in enumerate(_sizes(case, seed)):
        fl.append({"mu": case["mu"] + 0.3 * r.standard_normal(), "rho": r.uniform(0.85, 0.995),
                   "sigma_z": r.uniform(0.05, 0.4), "n_particles": n, "seed": _seed(seed) % 1000003 + b,
                   "nu_obs": case["nu_obs"]})
    return fl


def _imm_models(case):
    k = case["filters"]
    return [{"rho": 0.90 + 0.09 * (i % 4) / 3.0, "sigma_z": 0.1 + 0.05 * (i % 3),
             "mu": case["mu"] + 0.5 * (i - (k - 1) / 2.0) / k} for i in range(k)]


def prepare(case, seed):
    kind, n, T = case["kind"], case["n"], case["ticks"]
    th = (case["rho"], case["sigma"], case["mu"])
    s = {"case": case, "seed": _seed(seed)}
    if kind in ("live", "series", "device"):
        s["f"] = gpubpf.GpuBpf(n, *th, nu_state=case["nu_state"], nu_obs=case["nu_obs"], seed=s["seed"],
                               ess_threshold=case["ess"])
        y = _series(case, seed, T)
        if kind == "device":
            s["y"] = torch.from_numpy(y).cuda()
            s["rec"] = torch.zeros(T, 40, dtype=torch.uint8, device="cuda")
        else:
            s["y"] = y.tolist()
    elif kind == "apf":
        s["f"] = gpubpf.GpuApf(n, *th, nu_state=case["nu_state"], nu_obs=case["nu_obs"], seed=s["seed"])
        s["y"] = _series(case, seed, T).tolist()
    elif kind == "grad":
        s["y"] = torch.from_numpy(_series(case, seed, T)).cuda()
        r = np.random.RandomState(seed % (1 << 31))   # an optimiser's iterate near the generator's parameters
        s["theta"] = torch.tensor([th[2] + 0.1 * r.standard_normal(), th[0] - 0.01 * r.uniform(),
                                   th[1] * (1.0 + 0.1 * r.uniform())], dtype=torch.float64, requires_grad=True)
    elif kind == "batch":
        s["b"] = gpubpf.GpuBpfBatch(_batch_filters(case, seed), ess_threshold=case["ess"])
        s["y"] = _series(case, seed, T).tolist()
    elif kind == "batch_grad":
        fl = _batch_filters(case, seed)
        s["n"] = [f["n_particles"] for f in fl]
        s["theta"] = torch.tensor([[f["mu"], f["rho"], f["sigma_z"]] for f in fl], dtype=torch.float64,
                                  device="cuda", requires_grad=True)
        s["y"] = torch.from_numpy(_series(case, seed, T)).cuda()
    elif kind == "imm":
        s["f"] = gpubpf.Imm(_imm_models(case), n, seed=s["seed"])
        s["y"] = _series(case, seed, 4 * T).tolist()
        s["at"] = 0
    else:
        s["y"] = _series(case, seed, T).tolist()
    return s


def _results(res):
    return {"h_mean": np.array([r.h_mean for r in res], dtype=np.float32),
            "log_lik": np.array([r.log_lik for r in res], dtype=np.float32)}


def run(s):
    case, kind = s["case"], s["case"]["kind"]
    if kind == "live":
        f = s["f"]
        f.reset(s["seed"])
        return _results([f.step(v) for v in s["y"]])
    if kind == "series":
        s["f"].reset(s["seed"])
        return _results(s["f"].step_many(s["y"]))
    if kind == "device":
        s["f"].reset(s["seed"])
        s["f"].step_many_device(s["y"].data_ptr(), case["ticks"], s["rec"].data_ptr())
        f64, f32, i32 = s["rec"].view(torch.float64), s["rec"].view(torch.float32), s["rec"].view(torch.int32)
        return {"loglik": f64[:, 0:3], "h_mean_ess": f32[:, 6:8], "resampled_tick": i32[:, 8:10]}
    if kind == "apf":
        return _results(s["f"].step_many(s["y"]))      # no reset in its API: the next pass goes on from here
    if kind == "grad":
        s["theta"].grad = None
        ll = gpubpf.bpf_loglik(s["theta"], s["y"], case["n"], seed=s["seed"], nu_obs=case["nu_obs"])
        ll.backward()
        return {"loglik": ll.detach(), "grad": s["theta"].grad}
    if kind == "batch":
        ll, hm = s["b"].run(s["y"])
        return {"loglik": np.array(ll), "h_mean": np.array(hm, dtype=np.float32)}
    if kind == "batch_grad":
        s["theta"].grad = None
        ll = gpubpf.bpf_batch_loglik(s["theta"], s["y"], s["n"], nu_obs=case["nu_obs"])   # its default seeds
        ll.sum().backward()
        return {"loglik": ll.detach(), "grad": s["theta"].grad}
    if kind == "imm":
        T, y = case["ticks"], s["y"]
        res = [s["f"].step(y[(s["at"] + t) % len(y)]) for t in range(T)]
        s["at"] += T
        return {"h_mean": np.array([r.h_mean for r in res], dtype=np.float32),
                "log_lik": np.array([r.log_lik for r in res], dtype=np.float32),
                "probs": np.array(s["f"].probs(), dtype=np.float32)}
    f = gpubpf.Smc2(case["filters"], case["n"], case["ticks"], seed=s["seed"])
    if case["cpmmh"] > 0.0:
        f.set_cpmmh_rho(case["cpmmh"])
    ess = np.array([f.update(v) for v in s["y"]], dtype=np.float32)
    theta, logw, loglik = f.particles()
    f.close()
    return {"ess": ess, "theta": theta, "logw": logw, "loglik": loglik}


def work(case):
    """Observations in and results out once; per particle and tick the arithmetic of one draw (uniform 3,
    inverse normal CDF 23), the transition (4), the density (6) and the weight sums (8), and 12 more
    where the particle is resampled. Particles that no chip could hold between ticks (more than
    60 MB of them) are read and written with their weights on every tick."""
    T, B = case["ticks"], case["filters"]
    total = sum(_sizes(case, 0)) if case["kind"] in ("batch", "batch_grad", "imm", "smc2") else case["n"]
    per = 44.0 + (12.0 if case["ess"] == 0.0 else 1.0) + (30.0 if case["nu_state"] > 0.0 else 0.0)
    per += 12.0 if case["kind"] in ("grad", "batch_grad") else 0.0
    per *= 2.0 if case["kind"] == "apf" else 1.0
    state = 16.0 * total * T if 8.0 * total > 60e6 else 0.0
    return {"bytes": 4.0 * T + 40.0 * T * B + state, "flops": per * total * T}


# ---------------------------------------------------------------------------------------------------
# The same outputs in 64 bits
# ---------------------------------------------------------------------------------------------------
_M64 = (1 << 64) - 1
_A = 6364136223846793005


def _i64(v):
    v &= _M64
    return v - (1 << 64) if v >> 63 else v


def _lsr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _pcg(s):
    """PCG32 XSH-RR output of 64-bit states held as int64."""
    x = _lsr(_lsr(s, 18) ^ s, 27) & 0xFFFFFFFF
    r = _lsr(s, 59)
    return ((x >> r) | (x << (32 - r))) & 0xFFFFFFFF


def _pcg_int(old):
    x = (((old >> 18) ^ old) >> 27) & 0xFFFFFFFF
    r = old >> 59
    return ((x >> r) | (x << ((32 - r) & 31))) & 0xFFFFFFFF


def _uniform(s):
    u = (_pcg(s) >> 9).double() * 2.0 ** -23
    return u.clamp(float(np.uint32(0x358637BD).view(np.float32)), float(np.uint32(0x3F7FFBCE).view(np.float32)))


def _f32(v):
    return float(np.float32(v))


class _Filters:
    """Rows of independent filters [B, N] in FP64 (row b uses its first n[b] slots)."""

    def __init__(self, rows, nu_state=0.0, nu_obs=0.0, tangents=False):
        self.dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
        col = lambda k: torch.tensor([[_f32(r[k])] for r in rows], dtype=torch.float64, device=self.dev)  # noqa: E731
        self.mu, self.rho, self.sig = col("mu"), col("rho"), col("sigma_z")
        self.n = torch.tensor([[float(r["n_particles"])] for r in rows], dtype=torch.float64, device=self.dev)
        self.seeds = [int(r["seed"]) for r in rows]
        N = max(int(r["n_particles"]) for r in rows)
        self.i = torch.arange(N, device=self.dev)[None, :]
        self.live = None if all(int(r["n_particles"]) == N for r in rows) else self.i < self.n
        self.nu_state, self.nu_obs = nu_state, nu_obs
        self.t, self.At, self.Bt = 0, 1, 0
        self.u = [(s * 67890 + 12345) & _M64 for s in self.seeds]
        self.logw = -torch.log(self.n).expand(len(rows), N)
        one_m = (1.0 - self.rho * self.rho).clamp_min(1e-6)
        z = self._normal(2 * self.i + 1)
        self.h = self.mu + self.sig / one_m.sqrt() * z
        self.tan = None
        if tangents:
            self.tan = [torch.ones_like(self.h), z * self.sig * self.rho / one_m ** 1.5, z / one_m.sqrt()]

    def _state(self, inc):
        k1 = torch.tensor([[_i64(self.At * _A * _A * s)] for s in self.seeds], device=self.dev)
        return k1 + inc * _i64(self.At * (_A + 1) + self.Bt)

    def _normal(self, inc):
        return torch.special.ndtri(_uniform(self._state(inc)))

    def _noise(self):
        inc = 2 * self.i + 1
        z = self._normal(inc)
        if self.nu_state > 0.0:
            k = int(self.nu_state + 0.5)
            chi2 = torch.zeros_like(z)
            for c in range(k // 2):
                chi2 -= 2.0 * torch.log(_uniform(self._state(inc + ((c + 1) << 33))))
            if k & 1:
                chi2 += self._normal(inc + ((k // 2 + 1) << 33)) ** 2
            z = z * torch.sqrt(self.nu_state / chi2)
        return z

    def logpdf(self, y, h):
        q = (y * y) * torch.exp(-h)
        if self.nu_obs > 0.0:
            nu = self.nu_obs
            c = math.lgamma((nu + 1) / 2) - math.lgamma(nu / 2) - 0.5 * math.log(nu * math.pi)
            return c - 0.5 * (nu + 1) * torch.log1p(q / nu) - 0.5 * h
        return -0.5 * math.log(2 * math.pi) - 0.5 * q - 0.5 * h

    def score(self, y, h):
        q = (y * y) * torch.exp(-h)
        if self.nu_obs > 0.0:
            return -0.5 + 0.5 * (self.nu_obs + 1) * (q / self.nu_obs) / (1 + q / self.nu_obs)
        return -0.5 + 0.5 * q

    def propagate(self):
        if self.t > 0:
            z = self._noise()
            if self.tan is not None:
                a, b, c = self.tan
                self.tan = [self.rho * a + (1 - self.rho), self.rho * b + (self.h - self.mu), self.rho * c + z]
            self.h = self.mu + self.rho * (self.h - self.mu) + self.sig * z

    def advance(self):
        self.t += 1
        self.At = self.At * _A & _M64
        self.Bt = (self.Bt * _A + 1) & _M64

    def normalise(self, lw):
        """Normalised log-weights and the log of their sum before."""
        if self.live is not None:
            lw = lw.masked_fill(~self.live, -math.inf)
        S = torch.logsumexp(lw, dim=1, keepdim=True)
        return lw - S, S

    def resample(self, lw, rows):
        """Systematic resampling of the rows in `rows` (bools) by normalised log-weights lw."""
        which = [b for b, r in enumerate(rows) if r]
        if not which:
            return
        at = torch.tensor(which, device=self.dev)
        us = []
        for b in which:
            old = self.u[b]
            self.u[b] = (old * _A + 1442695040888963407) & _M64
            us.append((_pcg_int(old) >> 9) / 8388608.0)
        cdf = torch.cumsum(torch.exp(lw[at]), dim=1)
        last = cdf[:, -1:]
        t = (torch.tensor(us, dtype=torch.float64, device=self.dev)[:, None] + self.i) / self.n[at] * last
        anc = torch.searchsorted(cdf, t, right=True)
        anc = torch.minimum(anc, (self.n[at] - 1).long())
        self.h[at] = torch.gather(self.h[at], 1, anc)
        if self.tan is not None:
            for x in self.tan:
                x[at] = torch.gather(x[at], 1, anc)

    def tick(self, y, ess_threshold):
        """One bootstrap tick: (increment, filtered mean, ESS, resampled, gradient of the increment), by row."""
        self.propagate()
        lw, S = self.normalise(self.logw + self.logpdf(y, self.h))
        W = torch.exp(lw)
        hm = (W * self.h).sum(1)
        ess = 1.0 / (W * W).sum(1)
        g = None
        if self.tan is not None:
            Wg = W * self.score(y, self.h)
            g = torch.stack([(Wg * x).sum(1) for x in self.tan], dim=1)
        res = [True] * len(self.seeds) if ess_threshold <= 0.0 else (ess / self.n[:, 0] < ess_threshold).tolist()
        if self.tan is not None:
            self.tan = [x.expand_as(self.h).clone() for x in self.tan]
        self.resample(lw, res)
        r = torch.tensor(res, device=self.dev)[:, None]
        self.logw = torch.where(r, -torch.log(self.n), lw)
        self.advance()
        return S[:, 0], hm, ess, res, g


def _row(case, seed):
    return {"mu": case["mu"], "rho": case["rho"], "sigma_z": case["sigma"], "n_particles": case["n"], "seed": seed}


def _exact_plain(case, seed, records):
    f = _Filters([_row(case, _seed(seed))], case["nu_state"], case["nu_obs"])
    ll, hm, ess, res = [], [], [], []
    for y in _series(case, seed, case["ticks"]).tolist():
        a, b, c, d, _ = f.tick(y, case["ess"])
        ll.append(a); hm.append(b); ess.append(c); res.append(d[0])
    ll, hm, ess = (torch.cat(v).cpu() for v in (ll, hm, ess))
    if not records:
        return {"h_mean": hm, "log_lik": ll}
    ref, run_, prev = [], 0.0, True
    for v, r in zip(ll.tolist(), res):
        run_ = (0.0 if prev else run_) + v
        ref.append(run_)
        prev = r
    rec = torch.stack([ll, torch.tensor(ref, dtype=torch.float64), torch.cumsum(ll, 0)], dim=1)
    return {"loglik": rec, "h_mean_ess": torch.stack([hm, ess], dim=1), "resampled_tick": None}


def _exact_apf(case, seed):
    f = _Filters([_row(case, _seed(seed))], case["nu_state"], case["nu_obs"])
    hms, lls = [], []
    for t, y in enumerate(_series(case, seed, case["ticks"]).tolist()):
        if t == 0:
            S, hm, _, _, _ = f.tick(y, 0.0)
        else:
            mean = lambda: f.mu + f.rho * (f.h - f.mu)  # noqa: E731
            lv, _ = f.normalise(f.logw + f.logpdf(y, mean()))
            f.resample(lv, [True])
            m = mean()
            f.h = m + f.sig * f._noise()
            lw, S = f.normalise(f.logw + f.logpdf(y, f.h) - f.logpdf(y, m))
            hm = (torch.exp(lw) * f.h).sum(1)
            f.resample(lw, [True])
            f.advance()
        hms.append(hm)
        lls.append(S if S.dim() == 1 else S[:, 0])
    return {"h_mean": torch.cat(hms).cpu(), "log_lik": torch.cat(lls).cpu()}


def _exact_batch(case, seed, grad):
    fl = _batch_filters(case, seed)
    if grad:
        fl = [dict(r, seed=42 + b) for b, r in enumerate(fl)]
    f = _Filters(fl, 0.0, case["nu_obs"], tangents=grad)
    tot, g, hm = 0.0, 0.0, None
    for y in _series(case, seed, case["ticks"]).tolist():
        a, hm, _, _, gg = f.tick(y, case["ess"])
        tot = tot + a
        if grad:
            g = g + gg
    return {"loglik": tot.cpu(), "grad": g.cpu()} if grad else {"loglik": tot.cpu(), "h_mean": hm.cpu()}


def _exact_grad(case, seed):
    th = prepare(dict(case, kind="grad"), seed)["theta"].tolist()
    row = {"mu": th[0], "rho": th[1], "sigma_z": th[2], "n_particles": case["n"], "seed": _seed(seed)}
    f = _Filters([row], 0.0, case["nu_obs"], tangents=True)
    tot, g = 0.0, 0.0
    for y in _series(case, seed, case["ticks"]).tolist():
        a, _, _, _, gg = f.tick(y, 0.0)
        tot, g = tot + a, g + gg
    return {"loglik": tot[0].cpu(), "grad": g[0].cpu()}


def _exact_imm(case, seed):
    models = _imm_models(case)
    k = len(models)
    f = _Filters([dict(m, n_particles=case["n"], seed=_seed(seed) + 7919 * j) for j, m in enumerate(models)])
    logT = np.log(np.where(np.eye(k) > 0, 0.95, 0.05 / max(k - 1, 1)))
    lp = np.full(k, -math.log(k))
    out = {"h_mean": [], "log_lik": []}
    for y in _series(case, seed, 4 * case["ticks"]).tolist()[:case["ticks"]]:
        a, hm, _, _, _ = f.tick(y, 0.5)
        joint = np.logaddexp.reduce(logT + lp[:, None], axis=0) + a.cpu().numpy()
        z = np.logaddexp.reduce(joint)
        lp = joint - z
        out["h_mean"].append(float((np.exp(lp) * hm.cpu().numpy()).sum()))
        out["log_lik"].append(float(z))
    return {"h_mean": np.array(out["h_mean"]), "log_lik": np.array(out["log_lik"]), "probs": np.exp(lp)}


def exact(case, seed):
    kind = case["kind"]
    if kind in ("live", "series"):
        return _exact_plain(case, seed, False)
    if kind == "device":
        return _exact_plain(case, seed, True)
    if kind == "apf":
        return _exact_apf(case, seed)
    if kind == "grad":
        return _exact_grad(case, seed)
    if kind in ("batch", "batch_grad"):
        return _exact_batch(case, seed, kind == "batch_grad")
    if kind == "imm":
        return _exact_imm(case, seed)
    return None          # SMC^2: accept / reject decisions on noisy estimates have no 64-bit value
