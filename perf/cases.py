"""What this library is timed on: its public entry points at the sizes its users call them with.

The screen (a few stars to a benchmark chunk, both precisions, arrays and text lines), the clone Monte Carlo (one
pulsar against 64 clusters, a stage-2 list, one pair with very many clones, a whole pulsar job with its draws), the
prefilter that selects a pulsar's clusters, and the draws on the GPU.  Inputs are the synthetic catalogues of
phygas_gb300.synth (the benchmark's distributions), drawn from the case's seed.

listed() the cases, draw(rng) one more of the same ranges, prepare(case, seed) inputs and handles as a program holds
them, run(state) one pass, work(case) what the pass cannot do without, exact(case, seed) the same outputs by torch and
numpy in 64 bits.
"""
import math
import os
import shutil
import tempfile

import numpy as np
import torch

import phygas_gb300 as pg
from phygas_gb300 import synth

NC = 4087                      # clusters of the benchmark's table
CUT = 25.0                     # the screen's default chi2_max


def listed():
    return [
        # one star looked up against the resident table: the smallest call, latency
        dict(name="screen_1", kind="screen", nt=1, nc=NC, cut=CUT, r_kernel=2.0, control=False),
        # a small odd batch against a part of the catalogue, kernel radius rtot, a tighter cut
        dict(name="screen_301x1021", kind="screen", nt=301, nc=1021, cut=9.0, r_kernel=0.0, control=False),
        # the reference's `screen` profile: one work unit of 2,000 stars
        dict(name="screen_2000", kind="screen", nt=2000, nc=NC, cut=CUT, r_kernel=2.0, control=False),
        # the benchmark's chunk
        dict(name="screen_20000", kind="screen", nt=20000, nc=NC, cut=CUT, r_kernel=2.0, control=False),
        # the plain FP64 screen (its own option of the calls, the CLI and the request loop) on a small batch
        dict(name="screen_fp64_250", kind="fp64", nt=250, nc=NC, cut=CUT, r_kernel=2.0, control=False),
        # the screen CLI's path: records in, text lines out, chunks pipelined; the chance-alignment control run
        dict(name="text_3000", kind="text", nt=3000, nc=NC, cut=CUT, r_kernel=2.0, control=True, chunk=1250),
        # the clone Monte Carlo's small configuration: one pulsar x 64 clusters x 200 clones, 400 steps
        dict(name="pair_64x200", kind="pair", n_pairs=64, clones=200, dt=0.05, tmax=20.0, stars=False),
        # the reference's `stage2` profile: 300 star pairs x 1,000 clones, up to 2,000 steps each
        dict(name="pair_300x1000", kind="pair", n_pairs=300, clones=1000, dt=0.05, tmax=0.0, stars=True),
        # one close pair studied with very many clones
        dict(name="pair_1x20000", kind="pair", n_pairs=1, clones=20000, dt=0.05, tmax=100.0, stars=True),
        # a whole pulsar job as the pair CLI and the request loop run it: draws and tracing of every given cluster
        dict(name="pulsar_job_3500x1000", kind="job", nc=3500, clones=1000, dt=0.05),
        # which clusters a few pulsars can have met (the catalogue's side is resident after the first call)
        dict(name="prefilter_3", kind="prefilter", nt=3, nc=NC),
        # the clones of a stage-2 list drawn on the GPU
        dict(name="draws_300x1000", kind="draws", n_pairs=300, clones=1000),
    ]


def _log(rng, lo, hi):
    return min(hi, max(lo, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["screen", "screen", "screen", "fp64", "text", "pair", "pair", "pair", "job", "prefilter", "draws"])
    if kind in ("screen", "fp64", "text"):
        nt, nc = _log(rng, 1, 20000), _log(rng, 64, NC)
        if kind == "fp64":
            nt = max(1, min(nt, 250 * NC // nc, 4000))
        if kind == "text":
            nt = min(nt, 3000)
        c = dict(kind=kind, nt=nt, nc=nc, cut=rng.choice([9.0, CUT]), r_kernel=rng.choice([2.0, 2.0, 0.0]),
                 control=rng.random() < 0.3)
        if kind == "text":
            c["chunk"] = _log(rng, 500, 4000)
        return c
    if kind == "pair":
        if rng.random() < 0.25:                # few pairs with more clones than one warp reduces
            return dict(kind=kind, n_pairs=rng.randint(1, 4), clones=_log(rng, 1025, 20000), dt=0.05,
                        tmax=rng.choice([0.0, 20.0, 100.0]), stars=rng.random() < 0.5)
        n = _log(rng, 1, 3000)
        return dict(kind=kind, n_pairs=n, clones=_log(rng, 10, max(10, min(1000, 600000 // n))),
                    dt=rng.choice([0.05, 0.05, 0.02, 0.1]), tmax=rng.choice([0.0, 0.0, 20.0]),
                    stars=rng.random() < 0.5)
    if kind == "job":
        return dict(kind=kind, nc=_log(rng, 64, 3500), clones=_log(rng, 100, 1000), dt=0.05)
    if kind == "prefilter":
        return dict(kind=kind, nt=_log(rng, 1, 36), nc=_log(rng, 64, NC))
    n = _log(rng, 1, 2000)
    return dict(kind=kind, n_pairs=n, clones=_log(rng, 10, max(10, min(1000, 600000 // n))))


# ---- inputs ------------------------------------------------------------------------------------------------------
def _records(lines, read):
    d = tempfile.mkdtemp(prefix="phygas_cases_")
    try:
        path = os.path.join(d, "in.txt")
        with open(path, "w") as f:
            f.write("\n".join(lines) + "\n")
        return read(path)
    finally:
        shutil.rmtree(d, ignore_errors=True)


def _clusters(n, seed, tmax=0.0):
    return _records(synth.clusters(n, seed, n_no_rv=int(round(878 * n / NC)), tmax_fixed=tmax or None),
                    pg.read_clusters)


def _stars(n, seed, control=False):
    t = _records(synth.stars(n, seed), pg.read_targets)
    return pg.control_targets(t) if control else t


def _pulsars(n, seed):
    return _records(synth.pulsars(n, seed), pg.read_targets)


def _tmax(clusters):
    return max(c.tmax_myr for c in clusters)


def _pairs(case, seed):
    """The records and the pair list of the Monte Carlo kinds: stars cycle over the clusters, or one pulsar meets all."""
    n = case["n_pairs"]
    clusters = _clusters(n, seed, case.get("tmax", 0.0))
    if case.get("stars", True):
        targets, ti = _stars(min(n, 50), seed), np.arange(n, dtype=np.int32) % min(n, 50)
    else:
        targets, ti = _pulsars(1, seed), np.zeros(n, np.int32)
    return targets, ti, clusters, np.arange(n, dtype=np.int32)


def _room(case):
    """Rows a screen's buffer holds: every pair of a small one, a fifth of a large one's (about a tenth is kept)."""
    pairs = case["nt"] * case["nc"]
    return pairs if pairs < 1 << 20 else (1 << 19) + pairs // 5


class Held(np.ndarray):
    """Rows in page-locked memory that stays allocated while an array of them is in use."""

    def __array_finalize__(self, other):
        self.owner = getattr(other, "owner", None)


class State:
    """A case's inputs and the context a program keeps open."""

    def __init__(self, case):
        self.kind, self.case = case["kind"], dict(case)
        self.ctx = pg.Context(0)

    def __del__(self):
        self.ctx.close()


def prepare(case, seed):
    s = State(case)
    kind = s.kind
    if kind in ("screen", "fp64", "text"):
        s.clusters = _clusters(case["nc"], seed)
        s.stars = _stars(case["nt"], seed + 1, case["control"])
        s.tmax = _tmax(s.clusters)
        s.ctx.set_clusters(s.clusters, r_kernel=case["r_kernel"])
        if kind == "text":
            s.text = np.zeros(_room(case) * 100, np.uint8)
        else:
            s.draws = pg.draw_targets(s.stars)
            s.out = pg.HostRows(_room(case))
            s.out.rows[:] = 0
    elif kind == "pair":
        t, ti, c, ci = _pairs(case, seed)
        s.args = pg.draw_pair_batch(t, ti, c, ci, case["clones"], case["dt"])
    elif kind == "draws":
        s.args = _pairs(case, seed)
    elif kind == "job":
        s.clusters, s.targets = _clusters(case["nc"], seed), _pulsars(1, seed)
        s.ci = np.arange(case["nc"], dtype=np.int32)
    else:
        s.clusters, s.targets = _clusters(case["nc"], seed), _pulsars(case["nt"], seed)
        s.ctx.prefilter(s.targets, s.clusters)          # the catalogue's tracks stay in the context
        s.targets = _pulsars(case["nt"], seed + 1)
        s.pairs = np.full((2, case["nt"] * case["nc"]), -1, np.int32)
    return s


# ---- one pass ----------------------------------------------------------------------------------------------------
def _columns(rows):
    return {k: rows[k] for k in rows.dtype.names if k != "pad"}


def run(s):
    case, kind = s.case, s.kind
    if kind in ("screen", "fp64"):
        n = len(s.ctx.screen_into(*s.draws, s.tmax, s.out, case["cut"],
                                  pg.PGX_MIXED if kind == "screen" else pg.PGX_FP64))
        rows = s.out.rows.view(Held)                    # the whole buffer: zeros past the n rows
        rows.owner = s.out
        return dict(_columns(rows), n=n)
    if kind == "text":
        size = 0

        def emit(first, text, n):
            nonlocal size
            s.text[size:size + len(text)] = np.frombuffer(text, np.uint8)
            size += len(text)
        s.ctx.screen_chunks_text(s.stars, s.clusters, case["chunk"], s.tmax, emit, case["cut"])
        return dict(text=s.text, n=size)
    if kind == "pair":
        res, clones = s.ctx.pair(*s.args, want_clones=True)
        return dict(_columns(res), clones=clones)
    if kind == "draws":
        off, ps, steps, dt, r50, rt = s.ctx.draw_pair_batch(*s.args, case["clones"])
        return dict(off=off, ps=ps, steps=steps, dt=dt)
    if kind == "job":
        return _columns(s.ctx.pair_targets(s.targets, np.zeros(len(s.ci), np.int32), s.clusters, s.ci, case["clones"],
                                           case["dt"]))
    ti, ci = s.ctx.prefilter(s.targets, s.clusters)
    s.pairs[0, :len(ti)], s.pairs[1, :len(ti)] = ti, ci
    return dict(pairs=s.pairs, n=len(ti))


# ---- what a pass cannot do without -------------------------------------------------------------------------------
def work(case):
    """Flops: 104 per orbit step, 215 per clone-step, 126 per pair-point, about 240 per Gaussian triple and 600 per
    drawn clone; mean track lengths and kept fractions of the synthetic catalogues."""
    k = case["kind"]
    points, kept = 154, 0.109
    if k in ("screen", "fp64", "text"):
        nt, pairs = case["nt"], case["nt"] * case["nc"]
        rows = kept * pairs * (1.0 if case["cut"] >= CUT else 0.6)
        return {"bytes": nt * 28 * 8 + case["nc"] * points * 96 + rows * (94 if k == "text" else 80),
                "flops": nt * 7 * 2000 * 104 + pairs * points * 126.0 + rows * 512 * 240}
    if k in ("pair", "job"):
        n = (case["n_pairs"] if k == "pair" else case["nc"]) * case["clones"]
        steps = (case.get("tmax") or 40.0) / case["dt"]
        return {"bytes": n * (96 + 24) if k == "pair" else n * 96 + 96 * case["nc"], "flops": n * steps * 215.0}
    if k == "draws":
        n = case["n_pairs"] * case["clones"]
        return {"bytes": n * 96, "flops": n * 600}
    pairs = case["nt"] * case["nc"]
    return {"bytes": case["nc"] * 81 * 24 + pairs, "flops": case["nt"] * 2000 * 104 + pairs * 80 * 45}


# ---- the same outputs in 64 bits, by torch and numpy -------------------------------------------------------------
KMS = 977.7922216807892
G = 4.30091e-6 / (KMS * KMS) * 2.325e7
BULGE, DISK, HALO = G * 606.0, G * 3690.0, G * 4615.0
GOLDEN, MUL1, MUL2 = 0x9E3779B97F4A7C15, 0xBF58476D1CE4E5B9, 0x94D049BB133111EB


def _accel(p):
    """Allen & Santillan (1991) at p [3, ...]."""
    x, y, z = p
    R2 = x * x + y * y
    r2 = R2 + z * z
    rb = r2 + 0.3873 ** 2
    s = torch.sqrt(z * z + 0.25 ** 2)
    D2 = R2 + (5.3178 + s) ** 2
    r = torch.sqrt(r2).clamp_min(1e-12)
    h = r.clamp_max(100.0) / 12.0
    q = h ** (2.02 - 1.0)
    g = -BULGE / (rb * torch.sqrt(rb)) - HALO * h * q / (1.0 + q) / (r * r * r)
    d = -DISK / (D2 * torch.sqrt(D2))
    return torch.stack([x * (g + d), y * (g + d), z * (g + d * ((5.3178 + s) / s))])


def _kdk(p, v, a, dt):
    v = v + 0.5 * dt * a
    p = p + dt * v
    a = _accel(p)
    return p, v + 0.5 * dt * a, a


def _device(a):
    return torch.from_numpy(np.ascontiguousarray(a)).cuda()


def _exact_clones(args):
    off, ps, steps, dt = args[0], args[1].reshape(-1, 12), args[2], args[3]
    pair = np.repeat(np.arange(len(steps)), np.diff(off))
    order = np.argsort(-steps[pair], kind="stable")
    n_steps, h = steps[pair][order], _device(dt[pair][order])
    st = _device(ps[order]).T.reshape(2, 2, 3, -1)                    # body, (pos, vel), xyz, clone
    p, v = st[:, 0].transpose(0, 1).contiguous(), st[:, 1].transpose(0, 1).contiguous()     # [3, body, clone]
    a = _accel(p)
    r0 = p[:, 0] - p[:, 1]
    best, tbest = torch.sqrt((r0 * r0).sum(0)), torch.zeros_like(h)
    w = v[:, 0] - v[:, 1]
    vbest = torch.sqrt((w * w).sum(0))
    for i in range(1, int(n_steps[0]) + 1 if len(n_steps) else 0):
        m = int(np.searchsorted(-n_steps, -i, side="right"))          # clones that take step i: a prefix
        if m < p.shape[-1]:
            p, v, a, r0 = p[..., :m], v[..., :m], a[..., :m], r0[..., :m]
        p, v, a = _kdk(p, v, a, h[:m])
        r1 = p[:, 0] - p[:, 1]
        d = r1 - r0
        dd = (d * d).sum(0)
        s = torch.where(dd > 0, (-(r0 * d).sum(0) / dd).clamp(0.0, 1.0), torch.zeros_like(dd))
        x = r0 + d * s
        dm = torch.sqrt((x * x).sum(0))
        w = v[:, 0] - v[:, 1]
        hit = dm < best[:m]
        best[:m] = torch.where(hit, dm, best[:m])
        tbest[:m] = torch.where(hit, (i - 1 + s) * -h[:m], tbest[:m])
        vbest[:m] = torch.where(hit, torch.sqrt((w * w).sum(0)), vbest[:m])
        r0 = r1
    out = np.empty((3, len(order)))
    out[:, order] = torch.stack([best, tbest, vbest]).cpu().numpy()
    return out


def _exact_pair(case, seed):
    t, ti, c, ci = _pairs(case, seed)
    args = pg.draw_pair_batch(t, ti, c, ci, case["clones"], case["dt"])
    off, clones = args[0], _exact_clones(args)
    res = {k: np.zeros(len(off) - 1) for k in pg.RESULT_DTYPE.names if k != "n"}
    for q in range(len(off) - 1):
        part = clones[:, off[q]:off[q + 1]]
        m = part.shape[1]
        if not m:
            continue
        for name, x in (("d", part[0] * 1000.0), ("t", part[1]), ("v", part[2] * KMS)):
            x = np.sort(x)
            for pc, f in (("05", 0.05), ("50", 0.5), ("95", 0.95)):
                at = f * (m - 1)
                i = min(int(at), m - 1)
                res[name + pc][q] = x[i] if i >= m - 1 else x[i] + (at - i) * (x[i + 1] - x[i])
        res["f_r50"][q] = np.count_nonzero(part[0] * 1000.0 < c[q].r50_pc) / m
        res["f_rtot"][q] = np.count_nonzero(part[0] * 1000.0 < c[q].rtot_pc) / m
    return dict(res, n=None, clones=clones)


def _exact_tracks(ps0, sig, npts):
    """[npts][12][n]: position, velocity and covariance of each 0.5 Myr point of n objects."""
    n = len(ps0)
    base = _device(ps0).T
    st = base[:, None, :].repeat(1, 7, 1)                             # [6][orbit][n]
    for j in range(6):
        st[j, j + 1] += 1e-5
    p, v = st[:3].contiguous(), st[3:].contiguous()
    a = _accel(p)
    sg = _device(sig).reshape(n, 6, 6)
    out = torch.empty((npts, 12, n), dtype=torch.float64, device="cuda")
    for k in range(npts):
        if k:
            for _ in range(10):
                p, v, a = _kdk(p, v, a, -0.05)
        A = ((p[:, 1:] - p[:, :1]) / 1e-5).permute(2, 0, 1)
        S = torch.matmul(torch.matmul(A, sg), A.transpose(1, 2))
        out[k, :3], out[k, 3:6] = p[:, 0], v[:, 0]
        out[k, 6:] = torch.stack([S[:, 0, 0], S[:, 0, 1], S[:, 0, 2], S[:, 1, 1], S[:, 1, 2], S[:, 2, 2]])
    return out


def _forms(M, *xs):
    """x^T M^-1 x for symmetric M = (xx xy xz yy yz zz), by the adjugate; infinite where M is singular."""
    a, b, c, d, e, f = M
    i00, i01, i02 = d * f - e * e, c * e - b * f, b * e - c * d
    i11, i12, i22 = a * f - c * c, b * c - a * e, a * d - b * b
    det = a * i00 + b * i01 + c * i02
    for x, y, z in xs:
        q = (x * (i00 * x + i01 * y + i02 * z) + y * (i01 * x + i11 * y + i12 * z) +
             z * (i02 * x + i12 * y + i22 * z)) / det
        yield torch.where((det > 0) & (q >= 0), q, torch.full_like(q, math.inf))


def _signed(u):
    return u - (1 << 64) if u >= 1 << 63 else u


def _uniform(seed, call):
    """Output `call` of each row's splitmix64 stream as a number in [0, 1)."""
    def right(z, k):
        return (z >> k) & ((1 << (64 - k)) - 1)
    z = seed + call * _signed(GOLDEN)
    z = (z ^ right(z, 30)) * _signed(MUL1)
    z = (z ^ right(z, 27)) * _signed(MUL2)
    z = z ^ right(z, 31)
    return right(z, 11).double() / 9007199254740992.0


def _gauss(seed, call):
    u1 = _uniform(seed, call).clamp_min(2.0 ** -64)
    return torch.sqrt(-2.0 * torch.log(u1)) * torch.cos(2.0 * math.pi * _uniform(seed, call + 1))


def _exact_screen(case, seed):
    cl, stars = _clusters(case["nc"], seed), _stars(case["nt"], seed + 1, case["control"])
    ps0, sig, prefix = pg.draw_targets(stars)
    tmax = np.array([c.tmax_myr for c in cl])
    cn = np.ceil(tmax / 0.5).astype(int) + 1
    r50, rt = np.array([c.r50_pc for c in cl]) / 1e3, np.array([c.rtot_pc for c in cl]) / 1e3
    R2 = _device((case["r_kernel"] * r50 if case["r_kernel"] > 0 else rt) ** 2)
    npts = int(cn.max())
    T, C = _exact_tracks(ps0, sig, npts), _exact_tracks(*pg.draw_clusters(cl), npts)
    names = np.zeros((len(cl), 40), np.uint8)
    for i, c in enumerate(cl):
        names[i, :len(c.name)] = np.frombuffer(c.name, np.uint8)
    past = torch.arange(npts, device="cuda")[:, None, None] >= _device(cn)[None, None, :]
    step, cols = max(1, int(2e7 // (npts * len(cl)))), []
    for s0 in range(0, len(stars), step):
        t = T[:, :, s0:s0 + step, None]
        m0 = [t[:, i] - C[:, i, None, :] for i in range(3)]
        M = [t[:, 6 + i] + C[:, 6 + i, None, :] + (R2 if i in (0, 3, 5) else 0.0) for i in range(6)]
        last = _device(cn - 1)
        dr = [torch.cat([x[1:] - x[:-1], torch.zeros_like(x[:1])]) for x in m0]
        for x in dr:
            x.scatter_(0, last[None, None, :].expand(1, x.shape[1], -1), 0.0)
        dd = dr[0] ** 2 + dr[1] ** 2 + dr[2] ** 2
        f = -(m0[0] * dr[0] + m0[1] * dr[1] + m0[2] * dr[2]) / dd
        f = torch.where(dd > 0, f.clamp(0.0, 1.0), torch.zeros_like(dd))
        q0, q1 = _forms(M, m0, [a + b * f for a, b in zip(m0, dr)])
        f = torch.where(q1 < q0, f, torch.zeros_like(f))
        q = torch.minimum(q0, q1).masked_fill_(past, math.inf)
        best, kb = q.min(0)
        st, ci = torch.nonzero(best < case["cut"], as_tuple=True)
        k = kb[st, ci]
        sb = f[k, st, ci]
        m = torch.stack([a[k, st, ci] + b[k, st, ci] * sb for a, b in zip(m0, dr)])
        v = torch.stack([T[k, 3 + i, s0 + st] - C[k, 3 + i, ci] for i in range(3)])
        S = [T[k, 6 + i, s0 + st] + C[k, 6 + i, ci] for i in range(6)]
        l00 = torch.sqrt(S[0].clamp_min(0))
        l10, l20 = S[1] / l00, S[2] / l00
        l11 = torch.sqrt((S[3] - l10 * l10).clamp_min(0))
        l21 = torch.where(l11 > 0, (S[4] - l20 * l10) / l11, torch.zeros_like(l11))
        l22 = torch.sqrt((S[5] - l20 * l20 - l21 * l21).clamp_min(0))
        hi, ch = prefix[s0 + st.cpu().numpy()], names[ci.cpu().numpy()]
        with np.errstate(over="ignore"):
            for b in range(40):
                on = ch[:, b] != 0
                if not on.any():
                    break
                hi = np.where(on, (hi ^ ch[:, b].astype(np.uint64)) * np.uint64(1099511628211), hi)
        h = _device(hi.view(np.int64))[:, None]
        i50, irt = _device(r50)[ci], _device(rt)[ci]
        n50, nrt = torch.zeros_like(i50), torch.zeros_like(irt)
        for d0 in range(0, 512, 64):
            call = 6 * torch.arange(d0, d0 + 64, device="cuda")[None, :] + 1
            z = [_gauss(h, call + 2 * i) for i in range(3)]
            x = m[0][:, None] + l00[:, None] * z[0]
            y = m[1][:, None] + l10[:, None] * z[0] + l11[:, None] * z[1]
            w = m[2][:, None] + l20[:, None] * z[0] + l21[:, None] * z[1] + l22[:, None] * z[2]
            r = torch.sqrt(x * x + y * y + w * w)
            n50 += (r < i50[:, None]).sum(1)
            nrt += (r < irt[:, None]).sum(1)
        cols.append([x.cpu().numpy() for x in (
            sb, best[st, ci], (k + sb) * 0.5, torch.sqrt((m * m).sum(0)) * 1e3,
            torch.sqrt((S[0] + S[3] + S[5]) / 3.0) * 1e3, n50 / 512, nrt / 512, torch.sqrt((v * v).sum(0)) * KMS)])
    out = {}
    for name, x in zip(("sb", "chi2", "t_myr", "d_nom_pc", "sig_pc", "p_r50", "p_rtot", "vrel_kms"), zip(*cols)):
        out[name] = np.zeros(_room(case))
        x = np.concatenate(x)
        out[name][:len(x)] = x
    return dict(out, star=None, cluster=None, kb=None, n=None)


ROT = synth.ROT
SUN_V = np.array([11.1, 229.0 + 12.24, 7.25]) / KMS
AU_YR = 1.495978707e8 / 3.15576e7


def _phase_space(ra, dec, plx, pmra, pmdec, rv):
    ra, dec = np.radians(ra), np.radians(dec)
    er = np.stack([np.cos(dec) * np.cos(ra), np.cos(dec) * np.sin(ra), np.sin(dec)])
    ea = np.stack([-np.sin(ra), np.cos(ra), np.zeros_like(ra)])
    ed = np.stack([-np.sin(dec) * np.cos(ra), -np.sin(dec) * np.sin(ra), np.cos(dec)])
    pos = ROT @ (er / plx) + np.array([[-synth.SUN_R0], [0.0], [synth.SUN_Z0]])
    vel = ROT @ ((er * rv + ea * (AU_YR * pmra / plx) + ed * (AU_YR * pmdec / plx)) / KMS) + SUN_V[:, None]
    return pos, vel


def _rotation_rv(pos):
    """Line-of-sight velocity (km/s) of the circular orbit through pos's cylindrical radius."""
    flat = torch.from_numpy(np.stack([pos[0], pos[1], np.zeros_like(pos[0])]))
    a, R = _accel(flat).numpy(), np.hypot(pos[0], pos[1])
    vc = np.sqrt(np.maximum(-(a[0] * pos[0] + a[1] * pos[1]) / R, 0.0) * R)
    v = np.stack([vc * pos[1] / R, -vc * pos[0] / R, np.zeros_like(R)]) - SUN_V[:, None]
    los = pos - np.array([[-synth.SUN_R0], [0.0], [synth.SUN_Z0]])
    return (v * los).sum(0) / np.sqrt((los * los).sum(0)) * KMS


def _exact_draws(case, seed):
    t, ti, c, ci = _pairs(case, seed)
    n, m = case["n_pairs"], case["clones"]
    state = torch.from_numpy(np.array([_fnv(t[j].id + b"|" + c[i].name) for j, i in zip(ti, ci)],
                                      np.uint64).view(np.int64))
    calls = torch.zeros(n, dtype=torch.int64)

    def gauss(on=None):
        z = _gauss(state, calls + 1).numpy()
        calls.add_(2 if on is None else 2 * torch.from_numpy(on.astype(np.int64)))
        return z

    def positive(value):
        """value(z) drawn until positive, each object from its own stream."""
        x = value(gauss())
        while (bad := ~(x > 0)).any():
            x = np.where(bad, value(gauss(bad)), x)
        return x

    def columns(seq, idx):
        return {f: np.array([float(getattr(seq[i], f)) for i in idx])
                for f, kind in type(seq[0])._fields_ if getattr(kind, "_type_", "") in ("d", "i")}

    def body(o, plx, prior):
        pmra, pmdec = o["pmra"] + o["e_pmra"] * gauss(), o["pmdec"] + o["e_pmdec"] * gauss()
        z = gauss()
        pos, _ = _phase_space(o["ra"], o["dec"], plx, pmra, pmdec, np.zeros(n))
        rv = np.where(o["has_rv"] > 0, o["rv"] + o["e_rv"] * z, _rotation_rv(pos) + prior * z)
        return np.concatenate(_phase_space(o["ra"], o["dec"], plx, pmra, pmdec, rv)).T

    T, K, out = columns(t, ti), columns(c, ci), np.empty((n, m, 12))
    prior = np.array([265.0 if t[j].kind == b"P" else 30.0 for j in ti])
    with np.errstate(divide="ignore", over="ignore"):
        for j in range(m):
            plx = positive(lambda z: np.where(T["plx"] > 0, T["plx"] + T["e_plx"] * z,
                                              1000.0 / (T["dist_pc"] * np.exp(T["e_lndist"] * z))))
            out[:, j, :6] = body(T, plx, prior)
            out[:, j, 6:] = body(K, 1000.0 / positive(lambda z: K["dist_pc"] + K["e_dist_pc"] * z), 10.0)
    tmax = np.array([x.tmax_myr for x in c])
    return dict(off=None, steps=None, ps=out.reshape(-1), dt=-tmax / np.ceil(tmax / 0.05))


def _fnv(text):
    h = 1469598103934665603       # the offset the reference seeds with
    for b in text:
        h = (h ^ b) * 1099511628211 % (1 << 64)
    return h


def exact(case, seed):
    # a larger screen has pairs whose covariance is singular to 64 bits: whether they are kept is rounding alone
    if case["kind"] in ("screen", "fp64") and case["nt"] * case["nc"] < 1 << 20:
        return _exact_screen(case, seed)
    if case["kind"] == "pair":
        return _exact_pair(case, seed)
    if case["kind"] == "draws":
        return _exact_draws(case, seed)
    return None
