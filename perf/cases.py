"""Workloads the engine is timed on, each through the public entry points of
amdat_gb300.engine and amdat_gb300.autograd.

A case is a dict of plain values; `kind` names the analysis:

  disp         msd + ngp moments, optionally F_s shells and the self van Hove
               histogram of one list (Engine.disp); with `upload`, the pass
               starts from the trajectory in pinned host memory
  lists        the same over many nested lists through a prepared plan
  isf_lattice  rho_k over every lattice vector with |k| <= kmax, then F(k,t), S(k)
  isf_list     rho_k over q-vector shells, then F(k,t), S(k)
  rdf, vhd     g(r) counts and distinct van Hove counts
  structure    the loss of the differentiable structure and its gradient
  bins         msd + ngp (+ F_s) of every bin of a 3-d grid

Trajectories are seeded Gaussian random walks at the number density 0.8436 of
the repository's benchmark workloads.
"""
import math

import numpy as np
import torch

from amdat_gb300 import autograd as AG
from amdat_gb300 import engine as E
from amdat_gb300 import synth

DENSITY = 0.8436
TWO_PI = 2.0 * math.pi


def listed():
    return [
        # one short analysis of a small system: launches and host latency are the cost
        dict(name="msd_small", kind="disp", n=500, blocks=5, steps=10, shells="none", bins=0, upload=False),
        # the repository's MSD + NGP + F_s workload: 4000 atoms, one whole lattice shell (2,246 vectors)
        dict(name="msd_fs_4k", kind="disp", n=4000, blocks=10, steps=27, shells="lattice", bins=0, upload=False),
        # self van Hove over a long list, every time pair of a linear trajectory
        dict(name="vhs_64k", kind="disp", n=64000, blocks=49, steps=1, shells="none", bins=200, upload=False),
        # a fresh trajectory arrives in host memory and gets its MSD: ingestion, planning and the pass
        dict(name="upload_msd_32k", kind="disp", n=32000, blocks=12, steps=10, shells="none", bins=0, upload=True),
        # 64 nested lists of a 200,000-atom trajectory (per-species, per-region lists): moments
        dict(name="lists_msd_200k", kind="lists", n=200000, blocks=12, steps=30, lists=64, shells="none"),
        # the same lists with F_s on q-vector shells
        dict(name="lists_fs_200k", kind="lists", n=200000, blocks=12, steps=30, lists=64, shells="vectors"),
        # coherent scattering on the whole lattice |k| <= 20 (2.56 M vectors) of 32,000 atoms
        dict(name="isf_lattice_32k", kind="isf_lattice", n=32000, frames=20, kmax=20.0),
        # coherent scattering on the q-vector shells 1..20 of a script's isf command
        dict(name="isf_shells_32k", kind="isf_list", n=32000, frames=100, shells=20),
        # g(r) to half the box, every frame
        dict(name="rdf_64k", kind="rdf", n=64000, frames=50, bins=500, reach=0.5, lists="all"),
        # distinct van Hove to 5.0 over every time pair
        dict(name="vhd_64k", kind="vhd", n=64000, frames=50, bins=200, r_max=5.0, lists="all"),
        # loss and gradient of smoothed g(r) and S(k), 100,000 atoms
        dict(name="structure_100k", kind="structure", n=100000, frames=2, kmax=12.0, bins=400, sigma=0.02),
        # dynamics resolved by region: 4 x 4 x 4 bins, moments and two F_s shells
        dict(name="bins_fs_200k", kind="bins", n=200000, blocks=12, steps=30, grid=4, shells=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["disp", "disp", "lists", "isf_lattice", "isf_list", "rdf", "vhd", "structure", "bins"])
    c = dict(kind=kind)
    if kind == "disp":
        c["shells"] = rng.choice(["none", "none", "lattice", "vectors"])
        c["n"] = _log_int(rng, 200, 64000 if c["shells"] == "none" else 8000)
        c["blocks"], c["steps"] = rng.choice([(rng.randint(9, 49), 1), (rng.randint(2, 12), rng.randint(4, 30))])
        c["bins"] = rng.choice([0, rng.randint(20, 400)])
        c["upload"] = rng.choice([False, False, True])
    elif kind == "lists":
        c["shells"] = rng.choice(["none", "vectors"])
        c.update(n=_log_int(rng, 2000, 200000), blocks=rng.randint(2, 12), steps=rng.randint(4, 30),
                 lists=_log_int(rng, 2, 64))
    elif kind == "isf_lattice":
        c["kmax"] = round(rng.uniform(4.0, 20.0), 2)
        c["n"] = _log_int(rng, 500, 32000)
        c["frames"] = min(_log_int(rng, 2, 100), max(2, int(1.6e12 / (c["n"] * _half_space(c)))))
    elif kind == "isf_list":
        c["shells"] = rng.randint(2, 20)
        c["n"] = _log_int(rng, 500, 32000)
        c["frames"] = min(_log_int(rng, 4, 200), max(4, 3200000 // c["n"]))
    elif kind == "rdf":
        c["n"] = _log_int(rng, 300, 64000)
        c["frames"] = min(_log_int(rng, 1, 50), max(1, int(2e11 / c["n"] ** 2)))
        c.update(bins=rng.randint(50, 1000), reach=round(rng.uniform(0.2, 0.5), 3), lists=rng.choice(["all", "types"]))
    elif kind == "vhd":
        c.update(n=_log_int(rng, 1000, 64000), frames=rng.randint(5, 40), bins=rng.randint(50, 400),
                 r_max=round(rng.uniform(1.5, 5.0), 2), lists=rng.choice(["all", "types"]))
    elif kind == "structure":
        c.update(n=_log_int(rng, 1200, 100000), frames=rng.randint(1, 2), kmax=round(rng.uniform(4.0, 12.0), 2),
                 bins=rng.randint(100, 400), sigma=round(rng.uniform(0.02, 0.05), 3))
    else:
        c.update(n=_log_int(rng, 2000, 200000), blocks=rng.randint(2, 12), steps=rng.randint(4, 30),
                 grid=rng.randint(2, 5), shells=rng.choice([0, 0, 1, 2]))
    return c


# --- inputs ----------------------------------------------------------------
def _box(case):
    return float(np.float32(round((case["n"] / DENSITY) ** (1.0 / 3.0), 1)))


def _half_space(case):
    r = case["kmax"] * _box(case) / TWO_PI
    return max(1.0, 2.0 / 3.0 * math.pi * r ** 3)


def _scheme(case):
    if "frames" in case:
        return synth.TimeScheme.linear(case["frames"], 1.0)
    if case["steps"] == 1:
        return synth.TimeScheme.linear(case["blocks"] + 1, 1.0)
    return synth.TimeScheme.exponential(case["blocks"], case["steps"], 1.25, 0, 0, 0.005)


def _walk(case, seed):
    """Unwrapped float32 positions [frames][atoms][3] on the GPU."""
    sc = _scheme(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    n, L = case["n"], _box(case)
    dt = np.diff(sc.timelist().astype(np.float64))
    step = np.full_like(dt, 0.1) if sc.kind == "linear" else 0.05 * np.sqrt(np.maximum(dt, 0.0))
    pos = torch.rand((n, 3), generator=g, device="cuda", dtype=torch.float64) * L
    out = torch.empty((sc.n_timesteps, n, 3), device="cuda", dtype=torch.float32)
    out[0] = pos
    for t in range(1, sc.n_timesteps):
        pos += step[t - 1] * torch.randn((n, 3), generator=g, device="cuda", dtype=torch.float64)
        out[t] = pos
    return out


def _wrapped(u, L):
    """The engine's wrapped coordinates: u - L floor(u / L), every step in float32."""
    l32 = torch.tensor(L, dtype=torch.float32, device=u.device)
    return u - l32 * torch.floor(u / l32)


def _sphere(nmax):
    r = np.arange(-nmax, nmax + 1)
    g = np.stack(np.meshgrid(r, r, r, indexing="ij"), -1).reshape(-1, 3)
    return g, np.sqrt((g.astype(np.float64) ** 2).sum(1))


def _vector_shells(first, count):
    """q-vector shells like the reference's files: shell m holds up to 300 vectors
    of the half space with m + 1/2 <= |n| < m + 3/2, spread over the shell."""
    g, r = _sphere(first + count + 1)
    x, y, z = g.T
    half = (z > 0) | ((z == 0) & ((y > 0) | ((y == 0) & (x > 0))))
    kv, off = [], [0]
    rng = np.random.default_rng(1)
    for m in range(first, first + count):
        v = g[half & (r >= m + 0.5) & (r < m + 1.5)]
        v = v[np.sort(rng.permutation(len(v))[:min(300, len(v))])]
        kv.append(v)
        off.append(off[-1] + len(v))
    return np.concatenate(kv).astype(np.int32), np.asarray(off, np.int32)


def _lattice_shell(L, k0, k1):
    g, r = _sphere(int(math.ceil(k1 * L / TWO_PI)) + 1)
    k = TWO_PI * r / L
    v = g[(k >= k0) & (k <= k1)].astype(np.int32)
    return v, np.asarray([0, len(v)], np.int32)


def _shells(case):
    """(vectors, offsets) or None"""
    s = case.get("shells", "none")
    if s == "lattice":
        return _lattice_shell(_box(case), 7.0, 7.2)
    if s == "vectors":
        return _vector_shells(7, 5)
    if case["kind"] == "isf_list":
        return _vector_shells(1, s)
    if case["kind"] == "bins" and s:
        return _vector_shells(9, s)
    return None


def _nested(case, seed):
    """Sizes (ascending) and the permutation whose prefixes are the lists."""
    rng = np.random.default_rng(seed)
    top = case["n"] // 4
    sizes = np.exp(rng.uniform(math.log(100), math.log(top), case["lists"])).astype(np.int64)
    return np.sort(sizes), rng.permutation(case["n"])


def _types(case):
    """80:20 mixture: the atoms of each type."""
    n_a = (8 * case["n"]) // 10
    return np.arange(n_a), np.arange(n_a, case["n"])


class State:
    pass


def prepare(case, seed):
    s = State()
    s.case, s.L = case, _box(case)
    u = _walk(case, seed)
    if case["kind"] == "structure":
        s.pos = _wrapped(u, s.L).requires_grad_(True)
        s.box = [s.L] * 3
        with torch.no_grad():
            tgt = _wrapped(_walk(case, seed + 500009), s.L)
            h = AG.gsmooth(tgt, s.box, case["sigma"], 4.0, case["bins"])
            r = AG.structure_factor_raw(tgt, s.box, case["kmax"], 0.1)
            s.g_t = AG.g_of_r(h, case["n"], case["frames"], s.box, 4.0)
            s.s_t = AG.s_of_k(r, case["n"], case["frames"])
        return s
    s.eng = E.Engine(0)
    torch.cuda.synchronize()
    s.T, s.n = u.shape[0], u.shape[1]
    s.eng.upload_device(u.data_ptr(), s.T, s.n, [s.L] * 3)
    s.eng.set_scheme(_scheme(case))
    s.frames = np.arange(s.T, dtype=np.int32)
    s.shells = _shells(case)
    kind = case["kind"]
    if kind == "disp" and case["upload"]:
        s.host = torch.empty(u.shape, dtype=torch.float32, pin_memory=True)
        s.host.copy_(u)
    elif kind == "lists":
        sizes, perm = _nested(case, seed)
        handles = [s.eng.list(np.sort(perm[:m])) for m in sizes]
        s.plan = s.eng.plan(handles, shells=s.shells, period=s.L, flags=E.PLAN_GRAPH)
    elif kind == "isf_lattice":
        h, nk, ns = s.eng.wave_density_lattice(0, case["kmax"], 0.1, s.L, s.frames[:1])
        s.off = s.eng.wave_density_vectors(h, nk, ns)[1]
        s.eng.wave_density_free(h)
    elif kind in ("rdf", "vhd"):
        s.l1, s.l2 = (0, 0) if case["lists"] == "all" else [s.eng.list(a) for a in _types(case)]
    elif kind == "bins":
        s.bins = s.eng.bins_create([case["grid"]] * 3, [0.0] * 3, [s.L] * 3)
        s.eng.synchronize()
    return s


def _full(d):
    return {k: v for k, v in d.items() if v is not None and v.size}


def run(s):
    c, eng = s.case, getattr(s, "eng", None)
    kind = c["kind"]
    if kind == "disp":
        if c["upload"]:
            eng.upload_ptr(s.host.data_ptr(), s.T, s.n, [s.L] * 3)
        return _full(eng.disp(0, shells=s.shells, period=s.L, n_bins=c["bins"], bin_max=5.0 if c["bins"] else 0.0))
    if kind == "lists":
        s.plan.run()
        return _full(s.plan.read())
    if kind in ("isf_lattice", "isf_list"):
        if kind == "isf_lattice":
            h, off = eng.wave_density_lattice(0, c["kmax"], 0.1, s.L, s.frames)[0], s.off
        else:
            h, off = eng.wave_density(0, s.shells[0], s.L, s.frames), s.shells[1]
        corr, pairs = eng.isf(h, h, off)
        sk = eng.structure_factor(h, h, off)
        eng.wave_density_free(h)
        return dict(corr=corr, pairs=pairs, sk=sk)
    if kind == "rdf":
        return eng.rdf(s.l1, s.l2, s.frames, c["reach"] * s.L, c["bins"])
    if kind == "vhd":
        return eng.vhd(s.l1, s.l2, c["r_max"], c["bins"])
    if kind == "structure":
        loss, g, sk = AG.structure_loss(s.pos, s.box, s.g_t, s.s_t, c["sigma"], 4.0, c["bins"], c["kmax"], 0.1)
        grad, = torch.autograd.grad(loss, s.pos)
        return dict(loss=loss.detach(), g=g.detach(), s=sk.detach(), grad=grad)
    return _full(eng.disp_bins(0, s.bins, c["grid"] ** 3, shells=s.shells, period=s.L))


# --- work ------------------------------------------------------------------
def _pairs(case):
    """(gap, t0, t1) of the reference's time-pair scheduler (fullblock 0, frt 0)."""
    sc = _scheme(case)
    K, B = sc.n_exponential_steps, sc.n_exponentials
    out = [(g, K * b, K * b + g) for g in range(K) for b in range(B)]
    for g in range(K, K + B - 1):
        out += [(g, K * b, K * b + K * (g - K + 1)) for b in range(B - (g - K + 1))]
    out.append((K + B - 1, 0, sc.n_timesteps - 1))
    return out, K + B


def _n_frames(case):
    return _scheme(case).n_timesteps


def work(case):
    n, kind = case["n"], case["kind"]
    T = _n_frames(case)
    xyz = 12.0 * n * T
    pairs = float(len(_pairs(case)[0]))
    if kind in ("disp", "lists", "bins"):
        sh = _shells(case)
        atoms = n
        if kind == "lists":
            atoms = int(_nested(case, 0)[0][-1])
            xyz = 12.0 * atoms * T
        if kind == "bins":
            xyz += 4.0 * n * T
        # |dr|^2 and |dr|^4: 10 flops; a phase and a cosine per vector (8), or 3 per
        # octant representative of a shell closed under sign flips
        per = 10.0
        if sh is not None:
            per += 3.0 * len(sh[0]) / 8.0 if case["shells"] == "lattice" else 8.0 * len(sh[0])
        return dict(bytes=xyz, flops=per * pairs * atoms)
    if kind == "isf_lattice":
        # two real multiply-adds per atom and vector (cosine and sine products are
        # shared by the sign images of a vector), four flops per time pair and vector
        nk = _half_space(case)
        return dict(bytes=xyz, flops=4.0 * n * T * nk + 4.0 * pairs * nk)
    if kind == "isf_list":
        nk = len(_shells(case)[0])
        return dict(bytes=xyz, flops=8.0 * n * T * nk + 4.0 * pairs * nk)
    if kind == "rdf":
        a, b = (n, n / 2.0) if case["lists"] == "all" else [float(len(x)) for x in _types(case)]
        return dict(bytes=xyz, flops=10.0 * a * b * T)
    if kind == "vhd":
        a, b = (n, n) if case["lists"] == "all" else [float(len(x)) for x in _types(case)]
        near = min(1.0, 4.0 / 3.0 * math.pi * case["r_max"] ** 3 / _box(case) ** 3)
        return dict(bytes=xyz, flops=10.0 * pairs * a * b * near)
    near = n * 4.0 / 3.0 * math.pi * (4.0 + 6 * case["sigma"]) ** 3 * DENSITY
    span = 12.0 * case["sigma"] * case["bins"] / 4.0
    nk = _half_space(case)
    return dict(bytes=2.0 * xyz, flops=T * (1.5 * near * (10.0 + 4.0 * span) + 4.0 * n * nk + 8.0 * n * nk))


# --- 64-bit values -----------------------------------------------------------
def exact(case, seed):
    kind = case["kind"]
    if kind in ("rdf", "vhd"):
        return None  # counts
    if kind in ("disp", "lists", "bins"):
        return _exact_disp(case, seed)
    if kind in ("isf_lattice", "isf_list"):
        return _exact_isf(case, seed)
    return _exact_structure(case, seed)


def _exact_disp(case, seed):
    u = _walk(case, seed)
    L = _box(case)
    pairs, G = _pairs(case)
    sh = _shells(case)
    n, kind = case["n"], case["kind"]
    S = 0 if sh is None else len(sh[1]) - 1
    dev = u.device
    order, group = None, None
    if kind == "lists":
        sizes, perm = _nested(case, seed)
        order = torch.as_tensor(perm[:sizes[-1]], device=dev)
        ends = torch.as_tensor(sizes - 1, device=dev)
        rows = len(sizes)
    elif kind == "bins":
        rows = case["grid"] ** 3
        w = _wrapped(u, L)
        eps = float(np.finfo(np.float32).eps)
        ax = ((w.double() + 10.0 * eps) / (L + 20.0 * eps) * case["grid"]).long()
        group = (ax[..., 0] * case["grid"] + ax[..., 1]) * case["grid"] + ax[..., 2]
        group = torch.where(((w > 0) & (w < L)).all(-1), group, rows)
    else:
        rows = 1
    if sh is not None:
        kv = torch.as_tensor(sh[0].astype(np.float64) * (TWO_PI / L), device=dev).T.contiguous()

    def reduce(v, t0):
        if order is not None:
            return torch.cumsum(v, 0)[ends]
        if group is not None:
            return torch.zeros(rows + 1, dtype=torch.float64, device=dev).index_add_(0, group[t0], v)[:rows]
        return v.sum()[None]

    d2 = torch.zeros((rows, G), dtype=torch.float64, device=dev)
    d4 = torch.zeros_like(d2)
    fs = torch.zeros((rows, G, max(S, 1)), dtype=torch.float64, device=dev)
    for g, t0, t1 in pairs:
        a, b = (u[t0], u[t1]) if order is None else (u[t0][order], u[t1][order])
        dr = b.double() - a.double()
        q = (dr * dr).sum(1)
        d2[:, g] += reduce(q, t0)
        d4[:, g] += reduce(q * q, t0)
        if S:
            f = torch.empty((dr.shape[0], S), dtype=torch.float64, device=dev)
            step = max(1, 60000000 // kv.shape[1])
            for i in range(0, dr.shape[0], step):
                c = torch.cos(dr[i:i + step] @ kv)
                for k in range(S):
                    f[i:i + step, k] = c[:, sh[1][k]:sh[1][k + 1]].mean(1)
            for k in range(S):
                fs[:, g, k] += reduce(f[:, k], t0)
    if kind == "disp":
        d2, d4, fs = d2[0], d4[0], fs[0]
    out = dict(sum_d2=d2.cpu().numpy(), sum_d4=d4.cpu().numpy())
    if S:
        out["fs_sum"] = fs.cpu().numpy()
    out.update({"count": None} if kind == "bins" else {"atom_pairs": None})
    if kind == "disp" and case["bins"]:
        out["gs_counts"] = None
    return out


def _lattice_rho(q, row_vec, nz):
    """rho of (row, +-row) x nz from the real products of W = X Y and Z:
    returns rho(row, nz) and rho(-row, nz)."""
    nmax = int(row_vec.abs().max())
    ang = TWO_PI * q  # [3][N] turns -> radians
    k = torch.arange(-nmax, nmax + 1, device=q.device, dtype=torch.float64)
    px, py = torch.outer(k, ang[0]), torch.outer(k, ang[1])
    ph = px[row_vec[:, 0] + nmax] + py[row_vec[:, 1] + nmax]
    z = torch.outer(nz.double(), ang[2])
    A = torch.cat([torch.cos(ph), torch.sin(ph)])
    B = torch.cat([torch.cos(z), torch.sin(z)])
    P = A @ B.T
    R, Z = len(row_vec), len(nz)
    rr, ri, ir, ii = P[:R, :Z], P[:R, Z:], P[R:, :Z], P[R:, Z:]
    return torch.complex(rr - ii, ri + ir), torch.complex(rr + ii, ri - ir)


def _exact_isf(case, seed):
    L = _box(case)
    w = _wrapped(_walk(case, seed), L).double() / L
    w = w - torch.round(w)
    T, n = w.shape[0], w.shape[1]
    dev = w.device
    if case["kind"] == "isf_lattice":
        if n * T * _half_space(case) > 1.7e12:
            return None
        R = float(np.float32(case["kmax"])) * L / TWO_PI
        nmax = int(math.floor(R))
        r = torch.arange(-nmax, nmax + 1, device=dev)
        gx, gy = torch.meshgrid(r, r, indexing="ij")
        half = ((gy > 0) | ((gy == 0) & (gx >= 0))) & (gx * gx + gy * gy <= R * R)
        rows = torch.stack([gx[half], gy[half]], 1)
        nz = torch.arange(0, nmax + 1, device=dev)
        n2 = (rows ** 2).sum(1)[:, None].double() + (nz ** 2)[None].double()
        zero = (nz == 0)[None] & torch.ones_like(n2, dtype=torch.bool)
        origin = (rows == 0).all(1)[:, None]
        plus = (n2 <= R * R) & ~(zero & origin)
        minus = (n2 <= R * R) & ~zero & ~origin
        dk = float(np.float32(0.1))
        ns = int(math.floor(float(np.float32(case["kmax"])) / dk)) + 1
        shell = torch.clamp(torch.floor(TWO_PI * torch.sqrt(n2) / L / dk).long(), max=ns - 1)
        idx = torch.cat([shell[plus], shell[minus]])
        rho = torch.empty((T, len(idx)), dtype=torch.complex128, device=dev)
        for t in range(T):
            a, b = [], []
            for i in range(0, len(rows), 4096):
                p, m = _lattice_rho(w[t].T.contiguous(), rows[i:i + 4096], nz)
                a.append(p[plus[i:i + 4096]])
                b.append(m[minus[i:i + 4096]])
            rho[t] = torch.cat(a + b)
    else:
        kv, off = _shells(case)
        ns = len(off) - 1
        idx = torch.as_tensor(np.repeat(np.arange(ns), np.diff(off)), device=dev)
        k64 = torch.as_tensor(kv.astype(np.float64), device=dev)
        rho = torch.empty((T, len(kv)), dtype=torch.complex128, device=dev)
        for t in range(T):
            for i in range(0, len(kv), 1024):
                turn = k64[i:i + 1024] @ w[t].T
                turn -= torch.round(turn)
                rho[t, i:i + 1024] = torch.complex(torch.cos(TWO_PI * turn).sum(1), torch.sin(TWO_PI * turn).sum(1))
    cnt = torch.zeros(ns, dtype=torch.float64, device=dev).index_add_(
        0, idx, torch.ones(len(idx), dtype=torch.float64, device=dev))
    cnt = torch.where(cnt > 0, cnt, torch.ones_like(cnt))

    def shell_mean(v):
        return torch.zeros(ns, dtype=torch.float64, device=dev).index_add_(0, idx, v) / cnt

    pairs, G = _pairs(case)
    by = [[] for _ in range(G)]
    for g, a, b in pairs:
        by[g].append((a, b))
    corr = torch.zeros((G, ns), dtype=torch.float64, device=dev)
    for g in range(G):
        acc = torch.zeros(rho.shape[1], dtype=torch.float64, device=dev)
        for a, b in by[g]:
            acc += rho[a].real * rho[b].real + rho[a].imag * rho[b].imag
        corr[g] = shell_mean(acc)
    sk = shell_mean((rho.real ** 2 + rho.imag ** 2).sum(0))
    return dict(corr=corr.cpu().numpy(), pairs=None, sk=sk.cpu().numpy())


def _g_parts(pos, L, sigma, bins, weight):
    """h of one frame, and with weights dL/dh its gradient (float64)."""
    n = len(pos)
    dev = pos.device
    r_max, norm = 4.0, 1.0 / (math.sqrt(TWO_PI) * sigma)
    dr = r_max / bins
    cut, span = r_max + 6 * sigma, int(math.ceil(6.0 * sigma / dr))
    h = torch.zeros(bins, dtype=torch.float64, device=dev)
    grad = torch.zeros((n, 3), dtype=torch.float64, device=dev)
    order = torch.argsort(pos[:, 2])
    p = pos[order]
    z = p[:, 2].contiguous()
    step = 1024
    off = torch.arange(-span, span + 1, device=dev)
    for i in range(0, n, step):
        a = p[i:i + step]
        lo, hi = float(a[0, 2]) - cut, float(a[-1, 2]) + cut
        near = (z >= lo) & (z <= hi) | (z <= hi - L) | (z >= lo + L)
        cand = torch.nonzero(near)[:, 0]
        d = a[:, None, :] - p[cand][None]
        d -= L * torch.round(d / L)
        r = torch.sqrt((d * d).sum(-1))
        ii, jj = torch.nonzero((r < cut) & (r > 0), as_tuple=True)
        for k in range(0, len(ii), 2000000):
            rr, dd = r[ii[k:k + 2000000], jj[k:k + 2000000]], d[ii[k:k + 2000000], jj[k:k + 2000000]]
            b = torch.floor(rr / dr).long()[:, None] + off[None]
            ok = (b >= 0) & (b < bins)
            x = (b.double() + 0.5) * dr - rr[:, None]
            G = torch.where(ok, norm * torch.exp(-x * x / (2 * sigma * sigma)), torch.zeros_like(x))
            bc = b.clamp(0, bins - 1)
            if weight is None:
                h.index_add_(0, bc.reshape(-1), 0.5 * G.reshape(-1))
            else:
                psi = (weight[bc] * x * G).sum(1) / (sigma * sigma)
                grad.index_add_(0, ii[k:k + 2000000] + i, (psi / rr)[:, None] * dd)
    out = torch.empty_like(grad)
    out[order] = grad
    return h, out


def _exact_structure(case, seed):
    n, F, L = case["n"], case["frames"], _box(case)
    if F * n * _half_space(case) > 4e11:
        return None
    bins, sigma = case["bins"], float(np.float32(case["sigma"]))
    here, there = [_wrapped(_walk(case, s), L).double() for s in (seed, seed + 500009)]
    dev = here.device
    R = float(np.float32(case["kmax"])) * L / TWO_PI
    nmax = int(math.floor(R))
    r = torch.arange(-nmax, nmax + 1, device=dev)
    gx, gy = torch.meshgrid(r, r, indexing="ij")
    half = ((gy > 0) | ((gy == 0) & (gx >= 0))) & (gx * gx + gy * gy <= R * R)
    rows = torch.stack([gx[half], gy[half]], 1)
    nz = torch.arange(0, nmax + 1, device=dev)
    n2 = (rows ** 2).sum(1)[:, None].double() + (nz ** 2)[None].double()
    flat, origin = (nz == 0)[None], (rows == 0).all(1)[:, None]
    plus = (n2 <= R * R) & ~(flat & origin)
    minus = (n2 <= R * R) & ~(flat | origin)
    dk = float(np.float32(0.1))
    ns = int(math.floor(float(np.float32(case["kmax"])) / dk)) + 1
    shell = torch.clamp(torch.floor(TWO_PI * torch.sqrt(n2) / L / dk).long(), max=ns - 1)
    one = torch.ones_like(n2)
    cnt = torch.zeros(ns, dtype=torch.float64, device=dev)
    cnt.index_add_(0, shell[plus], one[plus]).index_add_(0, shell[minus], one[minus])
    cnt = torch.where(cnt > 0, cnt, torch.ones_like(cnt))

    def forward(pos):
        h = torch.zeros(bins, dtype=torch.float64, device=dev)
        s = torch.zeros(ns, dtype=torch.float64, device=dev)
        rho = []
        for f in range(F):
            h += _g_parts(pos[f], L, sigma, bins, None)[0]
            q = (pos[f] / L).T.contiguous()
            both = [_lattice_rho(q, rows[i:i + 1024], nz) for i in range(0, len(rows), 1024)]
            p, m = torch.cat([b[0] for b in both]), torch.cat([b[1] for b in both])
            rho.append((p, m))
            s.index_add_(0, shell[plus], (p.abs() ** 2)[plus]).index_add_(0, shell[minus], (m.abs() ** 2)[minus])
        b = (torch.arange(bins, dtype=torch.float64, device=dev) + 0.5) * (4.0 / bins)
        ideal = F * 0.5 * n * (n - 1) / L ** 3 * 4.0 * math.pi * b * b
        return h / ideal, s / cnt / (F * n), rho, ideal

    g_t, s_t, _, _ = forward(there)
    g, s, rho, ideal = forward(here)
    loss = ((g - g_t) ** 2).sum() + ((s - s_t) ** 2).sum()
    w_h = 2.0 * (g - g_t) / ideal
    w_s = 2.0 * (s - s_t) / (F * n)
    u = (2.0 * w_s / cnt)[shell]
    grad = torch.zeros((F, n, 3), dtype=torch.float64, device=dev)
    for f in range(F):
        grad[f] = _g_parts(here[f], L, sigma, bins, w_h)[1]
        q = (here[f] / L).T.contiguous()
        cp = torch.where(plus, u, 0 * u) * rho[f][0].conj()
        cm = torch.where(minus, u, 0 * u) * rho[f][1].conj()
        z = TWO_PI * torch.outer(nz.double(), q[2])
        zc, zs = torch.cos(z), torch.sin(z)
        acc = torch.zeros((3, n), dtype=torch.float64, device=dev)
        nzc = nz.double()[None]
        for i in range(0, len(rows), 512):
            row = rows[i:i + 512].double()
            ph = TWO_PI * (torch.outer(row[:, 0], q[0]) + torch.outer(row[:, 1], q[1]))
            wr, wi = torch.cos(ph), torch.sin(ph)
            a, b = cp[i:i + 512], cm[i:i + 512]
            d, e = a - b, a + b  # Im(W T+) -+ Im(conj(W) T-)
            v = wr * (d.real @ zs + d.imag @ zc) + wi * (e.real @ zc - e.imag @ zs)
            acc[0] += (row[:, :1] * v).sum(0)
            acc[1] += (row[:, 1:] * v).sum(0)
            d, e = d * nzc, e * nzc
            acc[2] += (wr * (e.real @ zs + e.imag @ zc) + wi * (d.real @ zc - d.imag @ zs)).sum(0)
        grad[f] -= (TWO_PI / L) * acc.T
    return dict(loss=loss.cpu(), g=g.cpu(), s=s.cpu(), grad=grad.cpu())
