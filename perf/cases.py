"""Performance cases: what programs run with this library, and the exact results of it.

A case is one pass of a simulation program's loop: the coordinates of its jobs
go up from pinned host memory, the jobs advance by some Langevin steps, the
coordinates come back (an interactive or sampling program, a serving quantum,
a trajectory writer).  The kinds:

  replicas  independent chains without hydrodynamics, one or hundreds of them,
            force clamp or force ramp (the plain pull and the ragged batch);
  shell     one capsid-like shell indented by a tip against a surface;
  tea       one chain with Truncated Expansion hydrodynamics;
  exact     one chain with exact hydrodynamics (Cholesky of the diffusion
            tensor every `refresh` steps).

Physical parameters are those of the benchmark workloads: T = 0.6 kcal/mol,
dt = 0.08 tau_H, pairlist every 10 steps at 20 A.
"""
import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.abspath(__file__)), os.pardir, "sop-gpu_b200"))

import sopb  # noqa: E402
import sopb_synth  # noqa: E402

JITTER = 0.1      # A: thermal displacement of the starting coordinates
CHAINS = 32       # distinct chains of a batch of replicas


# ---------------------------------------------------------------------------
# the cases
# ---------------------------------------------------------------------------
def _case(kind, steps, lo, hi=None, jobs=1, mode="ramp", refresh=1, copies=0):
    return {"kind": kind, "steps": steps, "jobs": jobs, "lo": lo, "hi": hi or lo, "mode": mode, "refresh": refresh,
            "copies": copies}


def listed():
    return [
        # an interactive pull of a small domain: a few steps per call, latency counts
        dict(_case("replicas", 20, 64, mode="clamp"), name="pull_64"),
        # the plain configuration: one 200-bead force-ramp pull
        dict(_case("replicas", 200, 200), name="pull_200"),
        # a handful of force-clamp replicas of different proteins
        dict(_case("replicas", 200, 60, 600, jobs=24, mode="clamp"), name="clamp_24"),
        # the ragged batch: 512 force-clamp replicas of 60 to 600 beads
        dict(_case("replicas", 200, 60, 600, jobs=512, mode="clamp"), name="clamp_512"),
        # one large protein complex below the one-job-per-block limit
        dict(_case("replicas", 100, 1733), name="pull_1733"),
        # one complex of the largest size that is served (50 to 5000 beads)
        dict(_case("replicas", 100, 5011, mode="clamp"), name="clamp_5011"),
        # capsid nanoindentation, 180 chains of 1100 beads
        dict(_case("shell", 20, 1100, copies=3, mode="indent"), name="shell_198000"),
        # hydrodynamics by TEA: a domain, and the benchmark's globule
        dict(_case("tea", 20, 517), name="tea_517"),
        dict(_case("tea", 20, 4000), name="tea_4000"),
        # exact hydrodynamics: a small domain with a new factor every step, a
        # served size, and the benchmark's globule with a factor every 10 steps
        dict(_case("exact", 20, 90), name="exact_90"),
        dict(_case("exact", 10, 601, refresh=5), name="exact_601"),
        dict(_case("exact", 10, 4000, refresh=10), name="exact_4000"),
    ]


def draw(rng):
    """One more case of the ranges above (rng: random.Random)."""
    def size(a, b):
        return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))

    kind = rng.choice(["one", "one", "batch", "batch", "grid", "shell", "tea", "exact_small", "exact"])
    mode = rng.choice(["clamp", "ramp"])
    if kind == "one":
        return _case("replicas", rng.choice([10, 30, 100, 200]), size(50, 2048), mode=mode)
    if kind == "batch":
        lo = size(50, 200)
        return _case("replicas", rng.choice([50, 100, 200]), lo, lo + size(20, 400), jobs=size(2, 512), mode=mode)
    if kind == "grid":
        return _case("replicas", rng.choice([20, 50, 100]), size(2049, 9000), mode=mode)
    if kind == "shell":
        return _case("shell", rng.choice([10, 20]), size(100, 1100), copies=rng.choice([1, 2, 3]), mode="indent")
    if kind == "tea":
        return _case("tea", rng.choice([10, 20]), size(50, 4000))
    if kind == "exact_small":
        return _case("exact", rng.choice([10, 20]), size(20, 128), refresh=rng.choice([1, 1, 5]))
    return _case("exact", 10, size(129, 3000), refresh=rng.choice([5, 10]))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _key(case):
    """The chains' seed: a function of the case's sizes."""
    return 1000 + 7 * case["lo"] + 13 * case["hi"] + case["jobs"]


@functools.lru_cache(maxsize=256)
def _chain(n, seed):
    return sopb_synth.make_system(n, seed)


@functools.lru_cache(maxsize=4)
def _shell(copies, chain_n):
    start = 7.3 * math.sqrt(copies * chain_n)
    return sopb_synth.make_capsid(copies_per_unit=copies, chain_n=chain_n, radius=start)[0]


def _systems(case):
    """The base system of every job."""
    if case["kind"] == "shell":
        return [_shell(case["copies"], case["lo"])]
    lo, hi, jobs, key = case["lo"], case["hi"], case["jobs"], _key(case)
    if lo == hi:
        return [_chain(lo, key)] * jobs
    sizes = sopb_synth.lognormal_sizes(min(jobs, CHAINS), lo, hi, key)
    sizes[0], sizes[-1] = lo, hi
    chains = [_chain(int(n), key + k) for k, n in enumerate(sizes)]
    return [chains[k % len(chains)] for k in range(jobs)]


def _inputs(case, seed):
    """Per job: (system, starting coordinates [n, 3], random states [n, 4], clamp force)."""
    rng = np.random.default_rng([seed, 20240])
    out = []
    for s in _systems(case):
        xyz = (s.xyz + JITTER * rng.standard_normal(s.xyz.shape)).astype(np.float32)
        states = rng.integers(1024, 2 ** 32, size=(s.n, 4), dtype=np.uint32)
        out.append((s, xyz, states, float(np.float32(rng.uniform(100.0, 300.0) / 70.0))))
    return out


def _params(case, sys_, force):
    """Config keys of a job (units of the library: A, kcal/mol, tau_H)."""
    n = sys_.n
    p = dict(timestep=0.08, zeta=50.0, temperature=0.6, kspring_cov=20.0, R_limit=2.0, a=3.8, el=1.0,
             pairs_cutoff=20.0, pairlist_cutoff=20.0, pairs_freq=10, pairs_threshold=200.0, nav=1000)
    if case["kind"] == "shell":
        x = sys_.xyz.astype(np.float64)
        c = x.mean(axis=0)
        tip = [float(c[0]), float(x[:, 1].max() + 104.0), float(c[2])]
        p.update(pairs_threshold=40.0, max_possiblePairs=2048, max_pairs=512, nav=100, indentation=1,
                 indentationTipR=100.0, indentationKs=0.07, indentationDeltaX=0.012, indentationTip=tip,
                 indentationChip=tip, indentationDirection=[0.0, -1.0, 0.0],
                 indentationSurfaceR0=[0.0, float(x[:, 1].min() - 10.0), 0.0], indentationSurfaceN=[0.0, 1.0, 0.0],
                 indentationTipZeta=5000.0, indentationTipSigma=1.0, indentationTipEl=1.0, indentationTipA=0.0,
                 indentationTipB=1.0, indentationSurfSigma=10.0, indentationSurfEl=0.2, indentationSurfA=1.0,
                 indentationSurfB=-2.0, indentationFixTrans=1)
        return p
    if n > 4096:   # above the default capacity of a bead's possible pairs
        p.update(max_possiblePairs=n)
    p.update(pulling=1, fixedEnd=0, pulledEnd=n - 1)
    if case["mode"] == "clamp":
        p.update(fconst=force)
    else:
        p.update(deltax=0.5, k_trans=0.05, pullFreq=1000)
    if case["kind"] != "replicas":
        p.update(hi_on=1, hi_a=3.8, hi_exact=int(case["kind"] == "exact"), hi_refresh=case["refresh"],
                 hi_epsilon_freq=10, hi_capricious=0)
    return p


_context = None


def _ctx():
    """The program's one device context."""
    global _context
    if _context is None:
        _context = sopb.Context(0)
    return _context


class _State:
    """The jobs of a program and its pinned coordinate buffers."""

    def __init__(self, case, seed):
        self.ctx, self.kind, self.steps, self.jobs = _ctx(), case["kind"], case["steps"], []
        coords = []
        for sys_, xyz, states, force in _inputs(case, seed):
            ends = [] if case["kind"] == "shell" else [0]
            spec = sopb.JobSpec(xyz, sys_.bonds, sys_.bonds_r0, sys_.natives, sys_.natives_r0, sys_.natives_eh,
                                sopb.default_params(**_params(case, sys_, force)), fixed=ends,
                                pulled=[sys_.n - 1] if ends else [], seeds=states)
            self.jobs.append(self.ctx.job(spec))
            coords.append(np.concatenate([xyz, np.zeros((sys_.n, 1), np.float32)], axis=1))
        self.start = torch.from_numpy(np.concatenate(coords)).pin_memory()
        self.end = torch.empty_like(self.start).pin_memory()

    def __del__(self):
        for j in self.jobs:
            j.destroy()
            self.ctx.jobs.remove(j)


def prepare(case, seed):
    return _State(case, seed)


def run(state):
    """Coordinates up, the steps, coordinates back; of a long job's pass also
    the kinetic temperatures that its program prints."""
    ctx, jobs = state.ctx, state.jobs
    ctx.upload_coords(jobs, state.start.numpy())
    ctx.run(jobs, state.steps)
    ctx.download_coords(jobs, state.end.numpy())
    if state.kind == "replicas":
        return {"x": state.end}
    return {"x": state.end, "T": jobs[0].read(sopb.TEMP)}


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _partners(n):
    """Beads within 20 A of a bead of an n-bead globule (uniform sphere)."""
    u = min(2.0, 20.0 / sopb_synth.target_radius(n))
    return (n - 1) * (u ** 3 - 9.0 / 16.0 * u ** 4 + u ** 6 / 32.0)


def work(case):
    """State in and out and maps once; per step the pair, bonded and noise
    arithmetic, and the hydrodynamic products."""
    if case["kind"] == "shell":
        sizes = [60 * case["copies"] * case["lo"]]
        partners = [145.0]
    else:
        sizes = [s.n for s in _systems(case)]
        partners = [_partners(n) for n in sizes]
    steps = case["steps"]
    nbytes = flops = 0.0
    for n, q in zip(sizes, partners):
        nbytes += n * (16 * 4 + 4 * 2 + 2 * 8 + 8 * 12)
        flops += steps * n * (18.0 * q + 2 * 20.0 + 8 * 18.0 + 80.0)
        if case["kind"] == "tea":
            flops += steps * 45.0 * n * n + -(-steps // 10) * 40.0 * n * n
        if case["kind"] == "exact":
            refreshes = -(-steps // case["refresh"])
            flops += refreshes * 9.0 * n ** 3 + steps * (45.0 * n * n + 9.0 * n * n)
            nbytes += refreshes * 18.0 * n * n
    return {"bytes": nbytes, "flops": flops}


# ---------------------------------------------------------------------------
# the same pass in 64 bits, plain torch
# ---------------------------------------------------------------------------
def _dev():
    return torch.device("cuda" if torch.cuda.is_available() else "cpu")


def _near_pairs(x, job, cut):
    """Index pairs (i, j), i and j of the same job, closer than `cut`, once each."""
    dev, n = x.device, x.shape[0]
    size = cut * 1.001
    c = ((x - x.min(dim=0).values) / size).floor().to(torch.int64) + 1
    dx, dy, dz = (int(v) + 2 for v in c.max(dim=0).values)
    cid = ((job * dz + c[:, 2]) * dy + c[:, 1]) * dx + c[:, 0]
    key, order = torch.sort(cid)
    me = torch.arange(n, device=dev)
    got = []
    for oz in (0, 1):
        for oy in (-1, 0, 1):
            for ox in (-1, 0, 1):
                if (oz, oy, ox) < (0, 0, 0):
                    continue
                want = cid + (oz * dy + oy) * dx + ox
                s = torch.searchsorted(key, want)
                cnt = torch.searchsorted(key, want, right=True) - s
                i = torch.repeat_interleave(me, cnt)
                first = torch.cumsum(cnt, 0) - cnt
                j = order[s[i] + torch.arange(i.numel(), device=dev) - first[i]]
                ok = (x[i] - x[j]).square().sum(1) < cut * cut
                if (oz, oy, ox) == (0, 0, 0):
                    ok &= i < j
                got.append((i[ok], j[ok]))
    return torch.cat([g[0] for g in got]), torch.cat([g[1] for g in got])


def _taus(s):
    """One draw of the combined Tausworthe + LCG generator from states s [n, 4]
    (int64 holding 32 bits), in place."""
    m32 = 0xFFFFFFFF
    for k, (s1, s2, s3, m) in enumerate(((13, 19, 12, 4294967294), (2, 25, 4, 4294967288), (3, 11, 17, 4294967280))):
        z = s[:, k]
        b = (((z << s1) & m32) ^ z) >> s2
        s[:, k] = (((z & m) << s3) & m32) ^ b
    s[:, 3] = (1664525 * s[:, 3] + 1013904223) & m32
    u = ((s[:, 0] ^ s[:, 1] ^ s[:, 2] ^ s[:, 3]) & 0x7FFFFF).double() / 2.0 ** 23
    return torch.where(u == 0, torch.full_like(u, 1e-8), u)


def _gauss(s):
    """Three of the four Gaussians a step draws per bead (Box-Muller)."""
    r1, t1 = (-2.0 * _taus(s).log()).sqrt(), 2.0 * math.pi * _taus(s)
    r2, t2 = (-2.0 * _taus(s).log()).sqrt(), 2.0 * math.pi * _taus(s)
    return torch.stack([r1 * t1.sin(), r1 * t1.cos(), r2 * t2.sin()], dim=1)


def _rpy(xi, xj, a):
    """Normalised RPY blocks [p, q, 3, 3] between rows of xi and of xj (zero on itself)."""
    d = xj[None, :, :] - xi[:, None, :]
    r = d.square().sum(-1).sqrt()
    same = r == 0
    r = torch.where(same, torch.ones_like(r), r)
    e, ra = d / r[..., None], r / a
    far = ra > 2.0
    crr = torch.where(far, 0.75 / ra * (1.0 - 2.0 / ra ** 2), 3.0 * ra / 32.0)
    cii = torch.where(far, 0.75 / ra * (1.0 + 2.0 / 3.0 / ra ** 2), 1.0 - 9.0 * ra / 32.0)
    crr, cii = crr * ~same, cii * ~same
    return e[..., :, None] * e[..., None, :] * crr[..., None, None] + cii[..., None, None] * torch.eye(3, dtype=xi.dtype, device=xi.device)


def _rows(n):
    """Row chunks of an n x n block sweep."""
    step = max(1, 2_000_000 // n)
    return [(k, min(n, k + step)) for k in range(0, n, step)]


def exact(case, seed):
    dev = _dev()
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    jobs = _inputs(case, seed)
    off = np.cumsum([0] + [s.n for s, *_ in jobs])
    T = lambda a, dt=torch.float64: torch.as_tensor(np.ascontiguousarray(a), device=dev).to(dt)  # noqa: E731
    x = T(np.concatenate([j[1] for j in jobs]))
    states = T(np.concatenate([j[2] for j in jobs]).astype(np.int64), torch.int64)
    job = T(np.repeat(np.arange(len(jobs)), np.diff(off)), torch.int64)
    bonds = T(np.concatenate([s.bonds + o for (s, *_), o in zip(jobs, off)]).astype(np.int64), torch.int64)
    b_r0 = T(np.concatenate([s.bonds_r0 for s, *_ in jobs]))
    nat = T(np.concatenate([s.natives + o for (s, *_), o in zip(jobs, off)]).astype(np.int64), torch.int64)
    n_r0 = T(np.concatenate([s.natives_r0 for s, *_ in jobs]))
    n_eh = T(np.concatenate([s.natives_eh for s, *_ in jobs]))
    n = x.shape[0]
    p = [_params(case, s, f) for s, _, _, f in jobs]
    P = p[0]
    h, zeta = f32(P["timestep"]), P["zeta"]
    mob, var = h / zeta, math.sqrt(2.0 * f32(P["temperature"]) * zeta / h)
    c8 = -6.0 * P["el"] * f32(P["a"]) ** 6
    skip = torch.sort(torch.cat([bonds, nat]).min(1).values * n + torch.cat([bonds, nat]).max(1).values).values
    pulled = fixed = None
    if P.get("pulling"):
        fixed, pulled = T(off[:-1], torch.int64), T(off[1:] - 1, torch.int64)
        x0 = x.clone()
        v = x0[pulled] - x0[fixed]
        pull = v / v.norm(dim=1, keepdim=True) * T([q.get("fconst", 0.0) for q in p])[:, None]

    def add(f, i, j, w, d):
        t = w[:, None] * d
        f.index_add_(0, i, t)
        f.index_add_(0, j, -t)

    def forces(pi, pj):
        f = torch.zeros_like(x)
        d = x[bonds[:, 1]] - x[bonds[:, 0]]
        r = d.norm(dim=1)
        w = r - b_r0
        add(f, bonds[:, 0], bonds[:, 1], P["kspring_cov"] * w / (r * (1.0 - w * w / P["R_limit"] ** 2)), d)
        d = x[nat[:, 1]] - x[nat[:, 0]]
        w = n_r0 ** 2 / d.square().sum(1)
        add(f, nat[:, 0], nat[:, 1], w * (w ** 6 - w ** 3) * (-12.0 * n_eh / n_r0 ** 2), d)
        d = x[pj] - x[pi]
        r2 = d.square().sum(1)
        add(f, pi, pj, torch.where(r2 < P["pairs_cutoff"] ** 2, c8 / r2 ** 4, torch.zeros_like(r2)), d)
        if P.get("indentation"):
            d = x - T([f32(v) for v in P["indentationTip"]])
            r = d.norm(dim=1)
            g = r - P["indentationTipR"]
            w = (12.0 * P["indentationTipA"] / g ** 6 + 6.0 * P["indentationTipB"]) / g ** 6 / (r * g)
            f += w[:, None] * P["indentationTipEl"] * d
            nn = T(P["indentationSurfaceN"])
            g = ((x - T([f32(v) for v in P["indentationSurfaceR0"]])) * nn).sum(1)
            sg, el = P["indentationSurfSigma"], f32(P["indentationSurfEl"])
            w = 12.0 * el * P["indentationSurfA"] * sg ** 12 / g ** 6 + 6.0 * el * P["indentationSurfB"] * sg ** 6
            f += (w / g ** 8)[:, None] * nn
        return f

    a = f32(P.get("hi_a", 0.0))
    L = ci = beta = None
    temp = torch.zeros_like(x[:, 0])
    # the updaters run at the smallest of their periods
    stride = case["refresh"] if case["kind"] == "exact" and case["refresh"] > 1 else 10
    for step in range(case["steps"]):
        if step % 10 == 0:
            pi, pj = _near_pairs(x, job, P["pairlist_cutoff"])
            k = torch.minimum(pi, pj) * n + torch.maximum(pi, pj)
            at = torch.searchsorted(skip, k).clamp(max=skip.numel() - 1)
            keep = skip[at] != k
            pi, pj = pi[keep], pj[keep]
        if step % stride == 0:
            if case["mode"] == "ramp":
                pull = f32(P["k_trans"]) * (x0[pulled] - x[pulled])
            if case["kind"] == "tea":   # epsilon and beta of the updater
                sq, tot = torch.empty_like(x), 0.0
                for r0, r1 in _rows(n):
                    D = _rpy(x[r0:r1], x, a)
                    sq[r0:r1] = D.square().sum((1, 3))
                    tot += float(D.sum())
                eps = min(1.0, tot / (3.0 * n * (3.0 * n - 3.0)))
                q = (3.0 * n - 1.0) * eps * eps - (3.0 * n - 2.0) * eps
                beta = 0.5 if abs(q) < 1e-7 else (1.0 - math.sqrt(1.0 - q)) / q
                ci = 1.0 / (1.0 + beta * beta * sq).sqrt()
        f, noise = forces(pi, pj), var * _gauss(states)
        if case["kind"] in ("replicas", "shell"):
            f += noise
        if pulled is not None:
            f[pulled] += pull
            f[fixed] = 0.0
        if case["kind"] == "tea":
            tot = f + ci * noise
            for r0, r1 in _rows(n):
                D = _rpy(x[r0:r1], x, a)
                tot[r0:r1] += torch.einsum("ijcd,jd->ic", D, f) + beta * torch.einsum(
                    "ijcd,id,jd->ic", D, ci[r0:r1], noise)
            f = tot
        elif case["kind"] == "exact":
            fresh = step % case["refresh"] == 0
            D = torch.eye(3 * n, dtype=x.dtype, device=dev) if fresh else None
            tot = f.clone()
            for r0, r1 in _rows(n):
                B = _rpy(x[r0:r1], x, a)
                tot[r0:r1] += torch.einsum("ijcd,jd->ic", B, f)
                if fresh:
                    D[3 * r0:3 * r1] += B.permute(0, 2, 1, 3).reshape(3 * (r1 - r0), 3 * n)
            if fresh:
                L = None
                L = torch.linalg.cholesky(D)
                del D
            f = tot + (L @ noise.reshape(-1)).reshape(n, 3)
        if fixed is not None:
            f[fixed] = 0.0
        x = x + mob * f
        temp = temp + f32(zeta / (6.0 * h)) * (mob * f).square().sum(1)
    out = {"x": torch.cat([x, torch.zeros_like(x[:, :1])], dim=1), "T": temp}
    return out if case["kind"] != "replicas" else {"x": out["x"]}
