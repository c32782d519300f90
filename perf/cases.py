"""The work that a user of this sampler has it do, as measurable cases.

A pass is what the user's program calls in its loop: a number of sweeps of one
study's chain (``Sampler.run``), of many chains or studies at once, the
reference's own loop of host-driven steps (``Sampler.step_host``), a chain
with the white-matter coefficient and the DIC / Qhat pass, the t and logistic
links and the FP64 chain, and the state that the program reads afterwards.
The studies have the shapes of ``bsglmm_gb300.synth``: ellipsoid masks, an
intercept, a +-0.5 group column and further covariates, smooth coefficient
fields with a rare outcome.

Chains start near their stationary state (the coefficients that the outcomes
were drawn from, with voxel noise), as all but the first sweeps of a chain of
thousands do.  Omega and the posterior maps of FP32 chains are handed on in
single precision: the sweep reads Omega so, and they are computed from single
precision coefficients.
"""
import math

import numpy as np
import torch

KINDS = ("run", "step", "wmdic", "logit", "t", "fp64")


# ------------------------------------------------------------- the cases ----
def _case(name, kind, grid, fill, N, P, sweeps, chains=1, studies=1, S=1):
    return {"name": name, "kind": kind, "X": grid[0], "Y": grid[1], "Z": grid[2],
            "fill": fill, "N": N, "P": P, "S": S, "sweeps": sweeps, "chains": chains,
            "studies": studies}


BRAIN, MM1, CUBE20 = (91, 109, 91), (182, 218, 182), (20, 20, 20)


def listed():
    return [
        # the reference's loop on a small study: Omega in, one sweep, Omega and
        # column means out, once per sweep (latency of one call)
        _case("sphere20_step", "step", CUBE20, 0.90, 50, 3, 16),
        # one chain of a small study, all sweeps kept, and its maps
        _case("sphere20_run", "run", CUBE20, 0.90, 50, 3, 64),
        # convergence study: 64 chains of the small study in one context
        _case("sphere20_chains64", "run", CUBE20, 0.90, 50, 3, 128, chains=64),
        # a simulation study: replicates of uneven size, N and P
        _case("replicates24", "run", (47, 47, 47), 0.75, 173, 4, 16, studies=24),
        # the brain-sized study, one production chain
        _case("brain_p5", "run", BRAIN, 0.787, 1000, 5, 32),
        # the large cohort with nuisance covariates
        _case("brain_p8", "run", BRAIN, 0.787, 2000, 8, 12),
        # 1 mm maps
        _case("volume_1mm", "run", MM1, 0.735, 500, 6, 16),
        # the command-line program's chain: white-matter coefficient, DIC and
        # Qhat on every kept sweep, two group columns, N not a multiple of 32
        _case("brain_wm_dic", "wmdic", BRAIN, 0.787, 403, 5, 12, S=2),
        # the reference's other two links
        _case("brain_logit", "logit", BRAIN, 0.787, 301, 5, 12),
        _case("mid_t", "t", (64, 64, 64), 0.85, 251, 3, 24),
        # the FP64 reference chain of a mid-sized study
        _case("mid_fp64", "fp64", (40, 44, 40), 0.80, 117, 4, 6),
    ]


def draw(rng):
    kind = rng.choice(("run",) * 4 + KINDS)
    log = lambda a, b: int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))  # noqa: E731
    fill = round(rng.uniform(0.6, 0.95), 3)
    P = rng.randint(2, 8)
    S = rng.randint(1, min(3, P)) if kind == "wmdic" else 1
    top = 64 if kind == "fp64" else 182
    side = log(14, top)
    grid = [max(10, min(top, int(side * rng.uniform(0.8, 1.25)))) for _ in range(3)]
    V = 4.0 / 3.0 * math.pi * np.prod([0.5 * fill * g for g in grid])
    # subject-voxels of a sweep stay below the largest listed study's
    most = {"fp64": 4e6, "logit": 7e7, "t": 7e7, "wmdic": 1e8}.get(kind, 4e8)
    N = log(20, max(21, min(2000, most / V)))
    chains = studies = 1
    if kind == "run" and N * V < 1e7 and rng.random() < 0.5:
        if rng.random() < 0.5:
            chains = log(2, 64)
        else:
            studies = log(2, 24)
    per = N * V * chains * studies * {"fp64": 150.0, "logit": 4.0, "t": 3.0}.get(kind, 1.0)
    sweeps = max(2, min(64, int(4e9 / per)))
    return {"kind": kind, "X": grid[0], "Y": grid[1], "Z": grid[2], "fill": fill, "N": N,
            "P": P, "S": S, "sweeps": sweeps, "chains": chains, "studies": studies}


# ------------------------------------------------------------ the studies ----
def _sizes(case, k):
    """Grid, fill, N and P of study k: the case's own, or (several studies)
    uneven ones around them."""
    if case["studies"] == 1:
        return (case["X"], case["Y"], case["Z"]), case["fill"], case["N"], case["P"]
    r = np.random.default_rng(7919 * k + 13)
    s = r.uniform(0.7, 1.3)
    g = tuple(max(8, int(case[a] * s)) for a in "XYZ")
    return (g, float(r.uniform(0.6, 0.9)), max(20, int(case["N"] * r.uniform(0.25, 1.75))),
            int(np.clip(case["P"] + r.integers(-2, 3), 2, 8)))


def _mask(grid, fill):
    X, Y, Z = grid
    z, y, x = np.meshgrid(*[(np.arange(n) - (n - 1) / 2) / (0.5 * fill * n) for n in (Z, Y, X)],
                          indexing="ij", sparse=True)
    return (x * x + y * y + z * z <= 1.0).astype(np.uint8)


def _voxels(mask):
    """Number of in-mask voxels per colour (0: odd sum of 1-based coordinates)."""
    z, y, x = np.nonzero(mask)
    odd = int(((x + y + z + 1) & 1).sum())
    return odd, len(x) - odd


def _study(grid, fill, N, P, S, seed, wm):
    """mask, covar [P][N], data [N][V], wm [V] or None, beta0 [P][V],
    omega0 [P][P]; made on the GPU from the seed."""
    dev = "cuda"
    g = torch.Generator(device=dev)
    g.manual_seed(seed)
    mask = _mask(grid, fill)
    m = torch.from_numpy(mask).to(dev).bool()
    V = int(m.sum())
    rnd = lambda *s: torch.randn(*s, generator=g, device=dev)  # noqa: E731
    X, Y, Z = grid

    # smooth fields, standardised in the mask
    t = torch.arange(-4, 5, device=dev, dtype=torch.float32)
    w = torch.exp(-0.5 * (t / 1.7) ** 2)
    w /= w.sum()
    f = rnd(P, 1, Z, Y, X)
    for d in range(3):
        sh, pad = [1, 1, 1, 1, 1], [0, 0, 0]
        sh[2 + d], pad[d] = 9, 4
        f = torch.nn.functional.conv3d(f, w.reshape(sh), padding=pad)
    f = f[:, 0][:, m]
    f = (f - f.mean(1, keepdim=True)) / (f.std(1, keepdim=True) + 1e-12)
    beta = 0.3 * f
    beta[0] = 0.5 * f[0] - 1.7
    covar = rnd(P, N)
    half = (torch.rand(N, generator=g, device=dev) < 0.5).float()
    if S >= 2:  # indicator columns of the groups cover every subject
        which = torch.randint(0, S, (N,), generator=g, device=dev)
        for s in range(S):
            covar[s] = (which == s).float()
            beta[s] = 0.5 * f[s] - 1.7
    else:
        covar[0] = 1.0
        if P > 1:
            covar[1] = half - 0.5
    wmv = torch.rand(V, generator=g, device=dev) if wm else None
    data = torch.empty(N, V, dtype=torch.uint8)
    step = max(1, (1 << 26) // V)
    for i in range(0, N, step):
        eta = covar[:, i:i + step].T @ beta
        if wm:
            eta += 0.3 * wmv
        u = torch.rand(eta.shape, generator=g, device=dev)
        data[i:i + step] = (u < torch.special.ndtr(eta)).to(torch.uint8).cpu()
    beta0 = beta + 0.1 * rnd(P, V)
    omega0 = 4.0 * torch.eye(P, dtype=torch.float64) + 0.3
    return {"mask": mask, "covar": covar.cpu().numpy(), "data": data.numpy(),
            "wm": None if wmv is None else wmv.cpu().numpy(), "beta0": beta0.cpu().numpy(),
            "omega0": omega0.numpy()}


def _studies(case, seed):
    for k in range(case["studies"]):
        grid, fill, N, P = _sizes(case, k)
        yield _study(grid, fill, N, P, case["S"], 1000003 * seed + k, case["kind"] == "wmdic")


BETA_WM0 = 0.25


def prepare(case, seed):
    import bsglmm_gb300 as bsg

    kind = case["kind"]
    s = bsg.Sampler(0)
    chains = []
    for k, st in enumerate(_studies(case, seed)):
        ds = s.add_dataset(st["mask"], st["covar"], st["data"], case["S"], st["wm"])
        info, lat = s.info(ds), s.lattice(ds)
        b = np.zeros((info["P"], info["Vp"]), np.float32)
        inmask = lat["idx"] >= 0
        b[:, lat["idxsc"][inmask]] = st["beta0"]
        for c in range(case["chains"]):
            ch = s.add_chain(ds, seed=seed * 7 + 1 + 100 * k + c, burnin=-1, thin=1,
                             beta_wm=BETA_WM0 if kind == "wmdic" else 0.0)
            if kind in ("logit", "t"):
                s.set_model(ch, "logistic" if kind == "logit" else "t")
            if kind == "fp64":
                s.set_precision(ch, 64)
            if kind == "wmdic":
                s.set_wm_update(ch, True)
                s.set_predictive(ch, True)
            s.set_beta(ch, b)
            s.set_omega(ch, st["omega0"])
            chains.append(ch)
    s.sync()
    return {"s": s, "chains": chains, "case": case}


# ---------------------------------------------------------------- a pass ----
def run(state):
    s, chains, case = state["s"], state["chains"], state["case"]
    kind, n = case["kind"], case["sweeps"]
    f4 = lambda a: np.asarray(a, dtype=np.float32)  # noqa: E731
    if kind == "step":
        om = None
        for _ in range(n):
            om, cm = s.step_host(chains[0], om, 1)
        return {"omega": f4(om), "colmeans": cm, "beta": s.beta(chains[0])}
    s.run(n, sync=False)
    if kind == "fp64":
        return {"beta": s.beta64(chains[0]), "omega": s.omega(chains[0])}
    out = {"beta": [s.beta(c) for c in chains], "omega": [f4(s.omega(c)) for c in chains]}
    if len(chains) > 12:  # at most 64 outputs
        out = {"beta": np.concatenate([b.ravel() for b in out["beta"]]),
               "omega": np.concatenate([o.ravel() for o in out["omega"]])}
    if kind == "wmdic":
        q, ed, _ = s.predictive(chains[0])
        out |= {"qhat": f4(q), "ed": f4(ed), "beta_wm": f4(s.beta_wm(chains[0])[0])}
    elif _maps_too(case):
        mean, var, prb, _ = s.posterior(chains[0])
        out |= {"mean": f4(mean), "var": f4(var), "prb": f4(prb)}
    return out


def _maps_too(case):
    """A chain of a small study reads its posterior summaries too."""
    return (case["kind"] == "run" and case["chains"] == case["studies"] == 1
            and case["X"] * case["Y"] * case["Z"] <= 32 ** 3)


# ------------------------------------------------------------- the work ----
def work(case):
    """Bytes: outcome bits, design, coefficients of a voxel and its
    neighbours, neighbour table, the posterior sums, the link's weights.
    Operations: 4 P of the two products of a subject and voxel and 40 of the
    truncated normal draw (the count of this project's benchmark), the other
    links' weighted products and gamma draw, and the DIC pass's."""
    kind, S, bts, flops = case["kind"], case["S"], 0.0, 0.0
    for k in range(case["studies"]):
        grid, fill, N, P = _sizes(case, k)
        V = sum(_voxels(_mask(grid, fill)))
        b = N * V / 8 + 4.0 * P * N + V * (8 * P + 29) + 16.0 * V * (2 * P + S)
        f = N * V * (4.0 * P + 40)
        if kind in ("logit", "t"):
            b += 8.0 * N * V
            f += N * V * (P * (P + 1) + (40 if kind == "logit" else 10))
        if kind == "wmdic":
            b += N * V / 8 + 4.0 * P * V
            f += N * V * S * 20.0
        bts += b * case["chains"] * case["sweeps"]
        flops += f * case["chains"] * case["sweeps"]
    return {"bytes": bts, "flops": flops}


# ---------------------------------------------- the same chains in 64 bits ----
_M32 = 0xFFFFFFFF


def _philox(c, k0, k1):
    """Philox-4x32-10 (Salmon et al., SC'11) on int64 tensors of 32-bit words."""
    x, y, z, w = c
    for r in range(10):
        p0, p1 = x * 0xD2511F53, z * 0xCD9E8D57
        a = (k0 + r * 0x9E3779B9) & _M32
        b = (k1 + r * 0xBB67AE85) & _M32
        x, y, z, w = ((p1 >> 32) & _M32) ^ y ^ a, p1 & _M32, ((p0 >> 32) & _M32) ^ w ^ b, p0 & _M32
    return x, y, z, w


def _u(k):
    return (k.double() + 0.5) * 2.0 ** -32


def _normal(k):
    lo = k < 0x80000000
    t = torch.special.ndtri(_u(torch.where(lo, k, k ^ _M32)))
    return torch.where(lo, t, -t)


def _tn(a, k):
    """N(0, 1) on (a, inf) from the word k by inversion."""
    T = torch.special.ndtr(-a.abs())
    u, uc = _u(k), _u(k ^ _M32)
    lower = T * uc + u                      # the CDF of the draw where a < 0
    neg = a < 0
    lo = neg & (lower < 0.5)
    t = torch.special.ndtri(torch.where(lo, lower, torch.where(neg, uc - T * uc, T * uc)))
    return torch.where(lo, t, -t)


class _Exact:
    """Chains of one study (leading index: the chain) in FP64."""

    def __init__(self, st, S, seeds, ids, model, beta_wm, wm_update):
        dev = "cuda"
        self.S, self.model, self.wm_update = S, model, wm_update
        mask = st["mask"].astype(bool)
        pad = np.pad(mask, 1)
        Y, X = pad.shape[1:]
        dil = pad.copy()
        at = np.flatnonzero(pad.ravel())
        offs = (-1, 1, -X, X, -X * Y, X * Y)
        for o in offs:
            dil.ravel()[at + o] = True
        idx = np.full(pad.size, len(at), np.int64)
        idx[at] = np.arange(len(at))
        sc = np.cumsum(dil.ravel()) - 1
        self.V, self.Vp, self.sc = len(at), int(dil.sum()), torch.from_numpy(sc[at]).to(dev)
        z, y, x = np.unravel_index(at, pad.shape)
        nb = torch.from_numpy(np.stack([idx[at + o] for o in offs])).to(dev)
        odd = torch.from_numpy(((x + y + z) & 1).astype(bool)).to(dev)
        self.col = [torch.nonzero(odd)[:, 0], torch.nonzero(~odd)[:, 0]]
        self.nb = [nb[:, c] for c in self.col]
        self.X = torch.from_numpy(st["covar"]).to(dev).double()
        self.P, self.N = self.X.shape
        self.Yd = torch.from_numpy(st["data"]).to(dev)
        self.wm = (torch.ones(self.V, device=dev, dtype=torch.float64) if st["wm"] is None
                   else torch.from_numpy(st["wm"]).to(dev).double())
        C = len(seeds)
        self.C = C
        self.b = torch.zeros(C, self.P, self.V + 1, device=dev, dtype=torch.float64)
        self.b[:, :, :self.V] = torch.from_numpy(st["beta0"]).to(dev).double()
        self.om = torch.from_numpy(st["omega0"]).to(dev).expand(C, -1, -1).clone()
        self.k0 = torch.tensor([q & _M32 for q in seeds], device=dev)
        self.k1 = torch.tensor([q >> 32 for q in seeds], device=dev)
        self.cid = torch.tensor([q << 8 for q in ids], device=dev)
        self.bw = torch.full((C,), float(np.float32(beta_wm)), device=dev, dtype=torch.float64)
        self.sweep = 0
        self.df = float({0: 8, 1: 0, 2: 3}[model])
        if model != 1:
            self.phi = [torch.ones(C, self.N, len(c), device=dev, dtype=torch.float64)
                        for c in self.col]
        z = lambda *s: torch.zeros(*s, device=dev, dtype=torch.float64)  # noqa: E731
        self.sum, self.sq = z(C, self.P, self.V), z(C, self.P, self.V)
        self.prb, self.kept = z(C, S, self.V), 0
        self.qhat, self.ed = z(self.N, S), 0.0

    def words(self, c0, v, tag, key=None):
        """Philox words of counters (c0, v, sweep, chain | tag): [C][len c0][len v]."""
        sh = (self.C, -1, -1)
        x = c0[None, :, None].expand(self.C, -1, len(v))
        y = v[None, None, :].expand(self.C, len(c0), -1)
        w = (self.cid + tag)[:, None, None].expand(sh[0], len(c0), len(v))
        return _philox((x, y, torch.full_like(x, self.sweep), w), self.k0[:, None, None],
                       self.k1[:, None, None])

    def tail(self, a, i, v, c):
        """Robert (1995) rejection beyond 5 sigma; a, i, v, c: flat."""
        r = torch.zeros_like(a)
        todo = torch.ones_like(a, dtype=torch.bool)
        s = 0.5 * (a + torch.sqrt(a * a + 4.0))
        for q in range(8):
            w = _philox((i * 8 + q, v, torch.full_like(i, self.sweep), self.cid[c] + 2),
                        self.k0[c], self.k1[c])
            for j in (0, 2):
                x = a - torch.log(_u(w[j])) / s
                ok = todo & (torch.log(_u(w[j + 1])) < -0.5 * (x - s) ** 2)
                r = torch.where(ok, x, r)
                todo = todo & ~ok
        return r

    def gamma(self, i, v):
        """Gamma((nu + 1) / 2, 1) of subjects i (even start) and voxels v."""
        half = torch.arange(int(i[0]) // 2, (int(i[-1]) + 2) // 2, device="cuda")
        w = self.words(half, v, 7)
        inter = lambda a, b: torch.stack((a, b), 2).reshape(self.C, -1, len(v))[:, :len(i)]  # noqa: E731
        kn, ku = inter(w[0], w[2]), inter(w[1], w[3])
        if self.model == 2:
            return -torch.log(_u(kn) * _u(ku))
        d = 0.5 * (self.df + 1.0) - 1.0 / 3.0
        g, ok = self.mt(d, kn, ku)
        bad = torch.nonzero(~ok)
        if len(bad):
            c, ii, jj = bad.T
            todo, val = torch.ones(len(bad), device="cuda", dtype=torch.bool), torch.full((len(bad),), d, device="cuda", dtype=torch.float64)
            for q in range(31):
                w = _philox((i[ii] * 32 + q, v[jj], torch.full_like(ii, self.sweep),
                             self.cid[c] + 8), self.k0[c], self.k1[c])
                for j in (0, 2):
                    gg, o = self.mt(d, w[j], w[j + 1])
                    o = o & todo
                    val, todo = torch.where(o, gg, val), todo & ~o
                if not bool(todo.any()):
                    break
            g[c, ii, jj] = val
        return g

    @staticmethod
    def mt(d, kn, ku):
        x, u = _normal(kn), _u(ku)
        v = 1.0 + x / math.sqrt(9.0 * d)
        v3 = v ** 3
        ok = (v > 0) & ((u < 1.0 - 0.0331 * x ** 4)
                        | (torch.log(u) < 0.5 * x * x + d * (1.0 - v3 + torch.log(v3.clamp_min(1e-300)))))
        return d * v3, ok

    def colour(self, c):
        col, P, C, dev = self.col[c], self.P, self.C, "cuda"
        n = len(col)
        beta = self.b[:, :, col]
        bwm = self.bw[:, None] * self.wm[col]
        acc = torch.zeros(C, P, n, device=dev, dtype=torch.float64)
        zsum = torch.zeros(C, n, device=dev, dtype=torch.float64)
        mix = self.model != 1
        if mix:
            Q = torch.zeros(C, P, P, n, device=dev, dtype=torch.float64)
        step = max(4, min(1 << 20, ((1 << 24) // max(1, C * n)) & ~3))
        for i0 in range(0, self.N, step):
            i = torch.arange(i0, min(i0 + step, self.N), device=dev)
            quad = torch.arange(i0 // 4, (int(i[-1]) + 4) // 4, device=dev)
            k = torch.stack(self.words(quad, col, 1), 2).reshape(C, -1, n)[:, :len(i)]
            x = self.X[:, i]
            m0 = torch.einsum("pi,cpn->cin", x, beta)
            y = self.Yd[i][:, col].bool()
            sgn = torch.where(y, 1.0, -1.0).double()
            mu = m0 + bwm[:, None]
            if mix:
                ph = self.phi[c][:, i]
                sd = ph.rsqrt()
            a = -sgn * mu
            if mix:
                a = a / sd
            t = _tn(a.clamp_max(5.0), k)
            far = torch.nonzero(a > 5.0)
            if len(far):
                f = far.T
                t[f[0], f[1], f[2]] = self.tail(a[f[0], f[1], f[2]], i[f[1]], col[f[2]], f[0])
            if mix:
                t = t * sd
            r = sgn * t
            zr = m0 + r
            if mix:
                phn = 2.0 * self.gamma(i, col) / (r * r + self.df)
                self.phi[c][:, i] = phn
                zr = phn * zr
                for p in range(P):
                    for q in range(p + 1):
                        Q[:, p, q] += torch.einsum("i,cin->cn", x[p] * x[q], phn)
            acc += torch.einsum("pi,cin->cpn", x, zr)
            if self.wm_update:
                zsum += zr.sum(1)
        nb = self.nb[c]
        nn = (nb < self.V).sum(0).double()
        sumV = self.b[:, :, nb].sum(2)
        b = [acc[:, p] + torch.einsum("cq,cqn->cn", self.om[:, p], sumV) for p in range(P)]
        XX = self.X @ self.X.T
        G = [[(Q[:, p, q] if mix else XX[p, q]) + nn * self.om[:, p, q, None]
              for q in range(p + 1)] for p in range(P)]
        for p in range(P):
            for q in range(p + 1):
                s = G[p][q]
                for t in range(q):
                    s = s - G[p][t] * G[q][t]
                G[p][q] = torch.sqrt(s) if p == q else s / G[q][q]
        w = [self.words(torch.tensor([j], device=dev), col, 3) for j in range((P + 3) // 4)]
        e = [_normal(w[p // 4][p % 4])[:, 0] for p in range(P)]
        for p in range(P):
            for q in range(p):
                b[p] = b[p] - G[p][q] * b[q]
            b[p] = b[p] / G[p][p]
        b = [b[p] + e[p] for p in range(P)]
        for p in reversed(range(P)):
            for q in range(p + 1, P):
                b[p] = b[p] - G[q][p] * b[q]
            b[p] = b[p] / G[p][p]
        b = torch.stack(b, 1)
        self.b[:, :, col] = b
        self.sum[:, :, col] += b
        self.sq[:, :, col] += b * b
        for g in range(self.S):
            e = b[:, g] / 0.634 if self.model == 0 else b[:, g] if self.model == 2 else b[:, g] + bwm
            self.prb[:, g, col] += torch.sigmoid(e) if self.model != 1 else torch.exp(_as_log(e))
        if self.wm_update:
            xs = self.X.sum(1)
            return (self.wm[col] * (zsum + self.N * bwm
                                    - torch.einsum("p,cpn->cn", xs, b))).sum(1)
        return 0.0

    def advance(self):
        wmt = self.colour(0) + self.colour(1)
        P, C = self.P, self.C
        d = self.b[:, :, self.col[1]][:, :, None] - self.b[:, :, self.nb[1]]
        d = d * (self.nb[1] < self.V)
        S = torch.einsum("cpkn,cqkn->cpq", d, d).cpu()
        T = torch.zeros(C, P, P, dtype=torch.float64)
        tri = [(i, j) for i in range(1, P) for j in range(i)]
        z = torch.tensor([0], device="cuda")
        for c in range(C):
            one = lambda c0, tag: [int(w) for w in _philox(  # noqa: E731
                (c0, 0, self.sweep, int(self.cid[c]) + tag), int(self.k0[c]), int(self.k1[c]))]
            for i in range(P):
                a = 0.5 * (self.V + P - i)
                dd = a - 1.0 / 3.0
                for t in range(64):
                    w = one(i * 64 + t, 5)
                    x = float(_normal(torch.tensor(w[0])))
                    v = 1.0 + x / math.sqrt(9.0 * dd)
                    if v > 0 and math.log((w[1] + 0.5) * 2.0 ** -32) < 0.5 * x * x + dd * (
                            1.0 - v ** 3 + 3.0 * math.log(v)):
                        T[c, i, i] = math.sqrt(2.0 * dd * v ** 3)
                        break
            for q, (i, j) in enumerate(tri):
                T[c, i, j] = float(_normal(torch.tensor(one(q // 4, 4)[q % 4])))
            if self.wm_update:
                var = 1.0 / (self.N * float((self.wm ** 2).sum()))
                n = float(_normal(torch.tensor(one(0, 6)[0])))
                self.bw[c] = var * float(wmt[c]) + math.sqrt(var) * n
        L = torch.linalg.cholesky(torch.linalg.inv(S + torch.eye(P, dtype=torch.float64)))
        B = L @ T
        self.om = (B @ B.transpose(1, 2)).to(z.device)
        self.sweep += 1
        self.kept += 1

    def predict(self):
        """The DIC / Qhat pass of chain 0 after a kept sweep."""
        P, S, N = self.P, self.S, self.N
        b, bwm = self.b[0, :, :self.V], self.bw[0] * self.wm
        m = torch.zeros(N, S, device="cuda", dtype=torch.float64)
        step = max(1, (1 << 24) // self.V)
        for i in range(0, N, step):
            x, y = self.X[:, i:i + step], self.Yd[i:i + step].bool()
            rest = x[S:].T @ b[S:] + bwm
            for g in range(S):
                eta = rest + b[g]
                m[i:i + step, g] = _as_log(torch.where(y, eta, -eta)).sum(1)
        own = (self.X[:S] != 0).double().argmax(0)
        o = m.gather(1, own[:, None])
        d = m - o
        first = self.kept == 1
        new = torch.logaddexp(self.qhat, d)
        if first:
            new[:, 0] = d[:, 0]
        self.qhat = new
        self.ed += float(o.sum())

    def beta(self):
        out = torch.zeros(self.C, self.P, self.Vp, device="cuda", dtype=torch.float64)
        out[:, :, self.sc] = self.b[:, :, :self.V]
        return out.cpu().numpy()


def _as_log(a):
    """log of the Abramowitz & Stegun 26.2.17 normal CDF, on the side of a."""
    t = 1.0 / (1.0 + 0.2316419 * a.abs())
    p = 0.39894228 * t * (0.319381530 + t * (-0.356563782 + t * (
        1.781477937 + t * (-1.821255978 + t * 1.330274429))))
    return torch.where(a < 0, torch.log(p) - 0.5 * a * a, torch.log1p(-p * torch.exp(-0.5 * a * a)))


def exact(case, seed):
    kind = case["kind"]
    if not torch.cuda.is_available():
        return None
    model = {"logit": 0, "t": 2}.get(kind, 1)
    betas, omegas, last, first_id = [], [], None, 0
    for k, st in enumerate(_studies(case, seed)):
        C = case["chains"]
        seeds = [seed * 7 + 1 + 100 * k + c for c in range(C)]
        e = _Exact(st, case["S"], seeds, list(range(first_id, first_id + C)), model,
                   BETA_WM0 if kind == "wmdic" else 0.0, kind == "wmdic")
        first_id += C
        for _ in range(case["sweeps"]):
            e.advance()
            if kind == "wmdic":
                e.predict()
        betas += list(e.beta())
        omegas += list(e.om.cpu().numpy())
        last = e
    if kind == "step":
        return {"omega": omegas[0], "colmeans": last.b[0, :, :last.V].mean(1).cpu().numpy(),
                "beta": betas[0]}
    if kind == "fp64":
        return {"beta": betas[0], "omega": omegas[0]}
    out = {"beta": betas, "omega": omegas}
    if len(betas) > 12:
        out = {"beta": np.concatenate([b.ravel() for b in betas]),
               "omega": np.concatenate([o.ravel() for o in omegas])}
    if kind == "wmdic":
        out |= {"qhat": last.qhat.cpu().numpy(), "ed": np.float64(last.ed),
                "beta_wm": np.float64(float(last.bw[0]))}
    elif _maps_too(case):
        n, mean = last.kept, last.sum[0] / last.kept
        var = (last.sq[0] - n * mean ** 2) / (n - 1)
        out |= {"mean": mean.cpu().numpy(), "var": var.cpu().numpy(),
                "prb": (last.prb[0] / n).cpu().numpy()}
    return out
