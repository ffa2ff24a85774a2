"""What the performance of this framework is measured on.

Twelve listed calls of the correlation path, each through the public entry
points of ``corr_gb300``, and a generator of further ones of the same ranges.
Sizes are those of the repository's workloads (a water molecule and a 20-water
cluster in def2-SVP / def2-SVP-RI, nocc=40 nvir=360 naux=1200, the adjoint at
nocc=64 nvir=512 naux=2048, the batch of uneven instances) and odd ones between
them; every input is made on the GPU from the seed.

Two kinds of inputs:

* B^Q_ia = G s_Q with G ~ N(0, 1) and s_Q = 0.05 exp(-Q/400), occupied energies
  U[-1.5, -0.3] and virtual ones U[0.05, 3], the distribution of the
  repository's RI-MP2 workloads;
* for the calls that start from integrals, the Coulomb integrals of s Gaussians
  on random centres at the density of a water cluster, in closed form: a real
  metric with its ill-conditioning, real (P|mn) and (ab|cd) with their decay
  over distance, and orbitals orthonormal in the Gaussians' overlap.
"""
import json
import math
import os

import numpy as np
import torch

import corr_gb300
from corr_gb300 import autograd

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
F64 = torch.float64
BOHR = 1.0 / 0.52917721067  # bohr per angstrom


def listed():
    return [
        # one water molecule, the plain form: the smallest call, all latency
        {"name": "energy_fp64_h2o", "kind": "energy", "precision": "fp64",
         "nocc": 5, "nvir": 19, "naux": 76},
        # the plain form on a medium molecule, no size a multiple of a tile
        {"name": "energy_fp64_medium", "kind": "energy", "precision": "fp64",
         "nocc": 23, "nvir": 211, "naux": 743},
        # the benchmark's workload in its default precision form
        {"name": "energy_fp16_o40v360", "kind": "energy", "precision": "split_fp16",
         "nocc": 40, "nvir": 360, "naux": 1200},
        # the more accurate precision form (autograd's default), ragged sizes
        {"name": "energy_bf16_ragged", "kind": "energy", "precision": "split_bf16",
         "nocc": 27, "nvir": 151, "naux": 529},
        # 32 uneven molecules at once: a screening run
        {"name": "batch_fp16_32", "kind": "batch", "precision": "split_fp16",
         "count": 32, "sizes_seed": 505},
        # from the integrals to the energy at the size of the 20-water cluster
        {"name": "pipeline_fp16_cluster", "kind": "pipeline", "precision": "split_fp16",
         "nbf": 480, "nocc": 100, "naux": 1520},
        # the same in the plain form on a smaller molecule
        {"name": "pipeline_fp64_small", "kind": "pipeline", "precision": "fp64",
         "nbf": 131, "nocc": 19, "naux": 433},
        # the reference's own route through its drop-in calls: J^-1/2 and
        # BPQ = J^-1/2 (Q|mn), then B^Q_ia
        {"name": "calculate_ri_medium", "kind": "calculate_ri",
         "nbf": 227, "nocc": 43, "naux": 715},
        # (P|Q) and (P|mn) of the 20-water cluster from its basis shells
        {"name": "integrals_cluster", "kind": "integrals", "waters": 20},
        # canonical MP2 of one water molecule: build_FMo, MOtrans, the energy
        {"name": "canonical_h2o", "kind": "canonical", "nbf": 24, "nocc": 5},
        # a training-style step: energy and its adjoint by torch's autograd
        {"name": "autograd_o64v512", "kind": "autograd", "precision": "split_bf16",
         "nocc": 64, "nvir": 512, "naux": 2048},
        # the plain form's gradient, odd sizes
        {"name": "gradient_fp64_small", "kind": "gradient",
         "nocc": 13, "nvir": 83, "naux": 311},
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["energy", "energy", "energy", "batch", "pipeline", "pipeline",
                       "calculate_ri", "integrals", "canonical", "autograd", "gradient"])
    if kind == "integrals":
        return {"kind": kind, "waters": _between(rng, 1, 20)}
    if kind == "batch":
        return {"kind": kind, "precision": rng.choice(["split_fp16", "split_bf16"]),
                "count": _between(rng, 2, 40), "sizes_seed": rng.randrange(1 << 30)}
    if kind == "canonical":
        n = _between(rng, 10, 80)
        return {"kind": kind, "nbf": n, "nocc": max(1, int(n * rng.uniform(0.15, 0.4)))}
    if kind in ("pipeline", "calculate_ri"):
        p = rng.choice(["split_fp16", "split_bf16", "fp64"])
        n = _between(rng, 24, 240 if kind == "pipeline" and p == "fp64" else 480)
        case = {"kind": kind, "nbf": n, "nocc": max(1, int(n * rng.uniform(0.15, 0.25))),
                "naux": int(n * rng.uniform(3.0, 3.4))}
        return dict(case, precision=p) if kind == "pipeline" else case
    o = _between(rng, 4, {"energy": 64, "autograd": 64, "gradient": 24}[kind])
    v = min({"energy": 400, "autograd": 512, "gradient": 130}[kind],
            max(5, int(o * rng.uniform(4.0, 9.0))))
    case = {"kind": kind, "nocc": o, "nvir": v, "naux": int(v * rng.uniform(3.0, 4.0))}
    if kind == "energy":
        case["precision"] = rng.choice(["fp64", "split_fp16", "split_bf16"])
        if case["precision"] == "fp64":  # at most about the cost of the largest listed case
            case["nocc"] = min(o, 40)
            case["nvir"] = min(v, 360)
            case["naux"] = min(case["naux"], 1200)
    elif kind == "autograd":
        case["precision"] = rng.choice(["split_bf16", "split_fp16"])
    return case


# ---------------------------------------------------------------- inputs
def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)
    return g


def _rand(g, lo, hi, *shape):
    return lo + (hi - lo) * torch.rand(shape, generator=g, device="cuda", dtype=F64)


def _energies(g, nocc, nvir):
    return torch.cat([torch.sort(_rand(g, -1.5, -0.3, nocc))[0],
                      torch.sort(_rand(g, 0.05, 3.0, nvir))[0]])


def _rimp2(nocc, nvir, naux, seed, dtype=F64):
    """(B[Q][i][a], eps) of the RI-MP2 workloads."""
    g = _gen(seed)
    s = 0.05 * torch.exp(-torch.arange(naux, device="cuda", dtype=F64) / 400.0)
    B = torch.randn((naux, nocc, nvir), generator=g, device="cuda", dtype=F64)
    B *= s[:, None, None]
    return B.to(dtype), _energies(g, nocc, nvir)


def _batch_sizes(count, seed):
    r = np.random.Generator(np.random.PCG64(seed))
    out = []
    for _ in range(count):
        o = int(r.integers(5, 61))
        v = o * int(r.integers(4, 9))
        out.append((o, v, int(round(3.5 * v))))
    return out


def _spread(r, count, volume, apart):
    """`count` points (bohr) in a cube of `volume` each, `apart` from one another."""
    box = (volume * count) ** (1.0 / 3.0)
    pts = []
    while len(pts) < count:
        p = r.uniform(0.0, box, 3)
        if all(np.sum((p - q) ** 2) >= apart * apart for q in pts):
            pts.append(p)
    return np.array(pts)


def _f0(t):
    """The Boys function F_0(t) = erf(sqrt t) sqrt(pi / t) / 2."""
    s = torch.sqrt(torch.clamp(t, min=1e-16))
    return torch.where(t < 1e-8, 1.0 - t / 3.0, 0.5 * math.sqrt(math.pi) * torch.erf(s) / s)


class _Gaussians:
    """Normalised s Gaussians on random centres: `nbf` orbital functions (four
    exponents per centre) and `naux` auxiliary ones on three times as many; the
    metric's condition number is that of the cluster's (about 6e5 at naux = 1520)."""

    def __init__(self, nbf, naux, seed):
        r = np.random.Generator(np.random.PCG64(seed))
        nc = -(-nbf // 4)

        def functions(n, centres, volume, apart, a0, ratio):
            c = _spread(r, centres, volume, apart)
            k = np.arange(n)
            a = a0 * ratio ** (k // centres) * np.exp(r.uniform(-0.1, 0.1, n))
            return torch.from_numpy(a).cuda(), torch.from_numpy(c[k % centres]).cuda()

        self.a, self.A = functions(nbf, nc, 60.0, 2.2, 0.18, 3.6)
        self.d, self.D = functions(naux, 3 * nc, 20.0, 1.5, 0.4, 3.0)

    def _pairs(self):
        """Product exponents, centres and factors of the orbital pairs."""
        a, A = self.a, self.A
        p = a[:, None] + a[None, :]
        P = (a[:, None, None] * A[:, None] + a[None, :, None] * A[None]) / p[..., None]
        r2 = ((A[:, None] - A[None]) ** 2).sum(-1)
        n = (2.0 * a / math.pi) ** 0.75
        K = n[:, None] * n[None] * torch.exp(-a[:, None] * a[None] / p * r2)
        return p, P, K

    def overlap(self):
        p, _, K = self._pairs()
        return K * (math.pi / p) ** 1.5

    def orbitals(self):
        """Rows orthonormal in the overlap: S^-1/2, ordered by kinetic energy."""
        S = self.overlap().cpu().numpy()
        w, V = np.linalg.eigh(S)
        C = (V / np.sqrt(w)) @ V.T
        return torch.from_numpy(np.ascontiguousarray(C[np.argsort(self.a.cpu().numpy())])).cuda()

    def metric(self):
        d, D = self.d, self.D
        n = (2.0 * d / math.pi) ** 0.75
        t = d[:, None] * d[None] / (d[:, None] + d[None])
        r2 = ((D[:, None] - D[None]) ** 2).sum(-1)
        pre = 2.0 * math.pi ** 2.5 / (d[:, None] * d[None] * torch.sqrt(d[:, None] + d[None]))
        J = n[:, None] * n[None] * pre * _f0(t * r2)
        return (0.5 * (J + J.T)).contiguous()

    def three_index(self):
        p, P, K = self._pairs()
        n = (2.0 * self.d / math.pi) ** 0.75
        out = torch.empty((len(self.d),) + tuple(p.shape), device="cuda", dtype=F64)
        for q in range(len(self.d)):
            s = p + self.d[q]
            r2 = ((P - self.D[q]) ** 2).sum(-1)
            v = n[q] * K * (2.0 * math.pi ** 2.5) / (p * self.d[q] * torch.sqrt(s)) \
                * _f0(p * self.d[q] / s * r2)
            out[q] = 0.5 * (v + v.T)
        return out

    def four_index(self, ab, cd):
        """(ab|cd) for pair indices a*nbf+b and c*nbf+d."""
        p, P, K = (x.reshape(-1, 3) if x.dim() == 3 else x.reshape(-1) for x in self._pairs())
        s = p[ab] + p[cd]
        r2 = ((P[ab] - P[cd]) ** 2).sum(-1)
        return K[ab] * K[cd] * (2.0 * math.pi ** 2.5) / (p[ab] * p[cd] * torch.sqrt(s)) \
            * _f0(p[ab] * p[cd] / s * r2)


class _Packed:
    """The reference's packed list of unique AO integrals: values, index
    quadruples, and the ends of the classes (aa|aa), (aa|cc), (ab|ab), (aa|cd)."""

    def __init__(self, gs, n):
        a, b = torch.tril_indices(n, n, device="cuda")
        x, y = torch.tril_indices(len(a), len(a), device="cuda")
        q = torch.stack([a[x], b[x], a[y], b[y]], 1)
        val = gs.four_index(q[:, 0] * n + q[:, 1], q[:, 2] * n + q[:, 3])
        keep = val.abs() > 1e-12
        q, val = q[keep], val[keep]
        late = (q[:, 2] == q[:, 3]) & (q[:, 0] != q[:, 1])  # (ab|cc) is listed as (cc|ab)
        q = torch.where(late[:, None], q[:, [2, 3, 0, 1]], q)
        e01, e23 = q[:, 0] == q[:, 1], q[:, 2] == q[:, 3]
        cls = torch.full_like(val, 4, dtype=torch.int64)
        cls[e01] = 3
        cls[(q[:, 0] == q[:, 2]) & (q[:, 1] == q[:, 3])] = 2
        cls[e01 & e23] = 1
        cls[e01 & e23 & (q[:, 0] == q[:, 2])] = 0
        order = torch.argsort(cls, stable=True)
        self.intval = val[order].contiguous()
        self.intnums = q[order].to(torch.int16).contiguous()
        self.nrofint = int(len(val))
        ends = torch.cumsum(torch.bincount(cls, minlength=5), 0)[:4].cpu().numpy()
        self.sortcount = np.ascontiguousarray(ends, dtype=np.int64)

    def dense(self, n):
        out = torch.zeros((n,) * 4, device="cuda", dtype=F64)
        a, b, c, d = (self.intnums[:, k].long() for k in range(4))
        for i, j in ((a, b), (b, a)):
            for k, l in ((c, d), (d, c)):
                out[i, j, k, l] = self.intval
                out[k, l, i, j] = self.intval
        return out


def _symmetric(n, seed):
    m = torch.randn((n, n), generator=_gen(seed), device="cuda", dtype=F64)
    return (m + m.T).contiguous()


def _shells(basis, waters, seed):
    """Shell arrays (l, nprim, poff, center, exps, coefs) of a water cluster."""
    with open(os.path.join(ROOT, "oracle", "basis_h2o.json")) as f:
        db = json.load(f)["basis"][basis]
    r = np.random.Generator(np.random.PCG64(seed))
    t = math.radians(104.52) / 2
    oh = np.array([[math.sin(t), 0.0, math.cos(t)], [-math.sin(t), 0.0, math.cos(t)]])
    cols = [[], [], [], [], [], []]
    # the density of 20 waters in a 9 angstrom cube, O-O distances >= 2.6 angstrom
    for c in _spread(r, waters, 9.0 ** 3 / 20 * BOHR ** 3, 2.6 * BOHR):
        rot, _ = np.linalg.qr(r.standard_normal((3, 3)))
        h = c + 0.9572 * BOHR * oh @ rot.T
        for el, xyz in (("O", c), ("H", h[0]), ("H", h[1])):
            for sh in db[el]:
                for col, val in zip(cols, ([sh["l"]], [len(sh["exps"])], [len(cols[4])],
                                           list(xyz), sh["exps"], sh["coefs"])):
                    col.extend(val)
    return cols


def _inputs(case, seed):
    """The arrays of a case, before any handle of the framework."""
    k = case["kind"]
    if k in ("energy", "gradient"):
        return _rimp2(case["nocc"], case["nvir"], case["naux"], seed)
    if k == "autograd":  # FP32 storage, as a training program keeps it
        B, eps = _rimp2(case["nocc"], case["nvir"], case["naux"], seed, torch.float32)
        return B, eps
    if k == "batch":
        return [_rimp2(o, v, x, seed * 1000 + n) + (o, v)
                for n, (o, v, x) in enumerate(_batch_sizes(case["count"], case["sizes_seed"]))]
    if k in ("pipeline", "calculate_ri"):
        gs = _Gaussians(case["nbf"], case["naux"], seed)
        eps = _energies(_gen(seed), case["nocc"], case["nbf"] - case["nocc"])
        return gs.orbitals(), eps, gs.metric(), gs.three_index()
    if k == "canonical":
        n = case["nbf"]
        gs = _Gaussians(n, 1, seed)
        eps = _energies(_gen(seed), case["nocc"], n - case["nocc"])
        return gs.orbitals(), _symmetric(n, seed), eps, _Packed(gs, n)
    return [_shells(b, case["waters"], seed) for b in ("def2-svp", "def2-svp-ri")]


def prepare(case, seed):
    x = _inputs(case, seed)
    if case["kind"] == "integrals":
        x = [corr_gb300.Basis(*cols) for cols in x]
    elif case["kind"] == "autograd":
        x = [t.requires_grad_() for t in x]
    torch.cuda.synchronize()
    return case, corr_gb300.default_context(), x


# ---------------------------------------------------------------- one pass
def _mp2(*es):
    """[E_SS, E_OS, E, E_SCS] of each molecule."""
    return np.array([[e.e_ss, e.e_os, e.e_total, e.e_scs] for e in es])


def run(state):
    case, ctx, x = state
    k, o = case["kind"], case.get("nocc")
    if k == "energy":
        return _mp2(ctx.rimp2_energy(x[0], x[1], o, case["nvir"], case["naux"],
                                     case["precision"]))
    if k == "batch":
        return _mp2(*ctx.rimp2_energy_batched(x, case["precision"]))
    if k == "pipeline":
        e, _ = ctx.rimp2_energy_from_3index(2 * o, *x, precision=case["precision"])
        return _mp2(e)
    if k == "calculate_ri":
        mos, _, J, pmn = x
        bpq = ctx.calculate_ri(J, pmn)
        return bpq, ctx.transform_ri(2 * o, mos, bpq)
    if k == "integrals":
        return ctx.ri_integrals(*x)
    if k == "canonical":
        mos, fmat, eps, packed = x
        fmo = ctx.build_fmo(mos, fmat)
        prec = ctx.motrans(2 * o, mos, packed)
        return _mp2(ctx.canonical_mp2(2 * o, prec, eps)), fmo, prec
    if k == "autograd":
        e = autograd.rimp2_energy(x[0], x[1], o, case["nvir"], case["precision"])
        dB, deps = torch.autograd.grad(e, x)
        return e.detach(), dB, deps
    e, dB, deps = ctx.rimp2_gradient(x[0], x[1], o, case["nvir"], case["naux"])
    return e, dB, deps


# ---------------------------------------------------------------- what it takes
def _sizes(case):
    k = case["kind"]
    if k == "batch":
        return _batch_sizes(case["count"], case["sizes_seed"])
    v = case.get("nvir", case.get("nbf", 0) - case["nocc"])
    return [(case["nocc"], v, case.get("naux", 0))]


def work(case):
    """Bytes: every input read once, every output written once.  Operations:
    the contractions with the symmetries that any method can use ((ia|jb) =
    (jb|ia); J^-1/2 counted as 10 X^3, of an eigendecomposition)."""
    k = case["kind"]
    if k == "integrals":
        # per (P|mn) about 60 operations for each of ~1.7 x 1.7 primitive pairs
        n, x = 24 * case["waters"], 76 * case["waters"]
        return {"bytes": 8.0 * (x * n * n + x * x), "flops": 60.0 * 3.0 * (x * n * n / 2.0 + x * x)}
    e_bytes = sum(8.0 * (o * v * x + o + v) for o, v, x in _sizes(case))
    e_flops = sum(float(o * v) ** 2 * x + 6.0 * (o * v) ** 2 for o, v, x in _sizes(case))
    o, v, x = _sizes(case)[0]
    n = case.get("nbf", 0)
    if k in ("energy", "batch"):
        return {"bytes": e_bytes, "flops": e_flops}
    if k == "pipeline":
        return {"bytes": 8.0 * (x * n * n + x * x + n * n),
                "flops": e_flops + 2.0 * x * o * n * n + 2.0 * x * o * v * n
                + x ** 3 / 3.0 + 1.0 * x * x * o * v}
    if k == "calculate_ri":
        return {"bytes": 8.0 * (2 * x * n * n + x * x + n * n + x * o * v),
                "flops": 10.0 * x ** 3 + 1.0 * x * x * n * (n + 1) + 2.0 * x * o * n * n
                + 2.0 * x * o * v * n}
    if k == "canonical":
        return {"bytes": 8.0 * (n ** 4 / 8.0 + n ** 4 + 3 * n * n) + n ** 4,
                "flops": 8.0 * n ** 5 / 4.0}
    b = 4.0 if k == "autograd" else 8.0
    # the adjoint: (ia|jb) once (half by symmetry), then G B for every row
    return {"bytes": 2 * b * o * v * x + 16.0 * (o + v), "flops": e_flops + 2.0 * (o * v) ** 2 * x}


# ---------------------------------------------------------------- 64 bits
def _exact_mp2(B, eps, o, v):
    B = B.to(F64)
    eps = eps.to(F64)
    X = B.shape[0]
    eo, ev = eps[:o], eps[o:]
    os_ = ss = 0.0
    for i in range(o):
        M = (B[:, i, :].T @ B[:, i:, :].reshape(X, -1)).reshape(v, o - i, v)
        D = ev[:, None, None] + ev[None, None, :] - eo[i] - eo[i:][None, :, None]
        w = torch.full((o - i,), 2.0, device=B.device, dtype=F64)
        w[0] = 1.0
        os_ = os_ - (w * (M * M / D).sum((0, 2))).sum()
        ss = ss - (w * ((M - M.transpose(0, 2)) * M / D).sum((0, 2))).sum()
    return _four(float(ss), float(os_))


def _four(ss, os_):
    return np.array([[ss, os_, ss + os_, ss / 3.0 + 1.2 * os_]])


def _exact_gradient(B, eps, o, v):
    B = B.to(F64)
    eps = eps.to(F64)
    X = B.shape[0]
    eo, ev = eps[:o], eps[o:]
    flat = B.reshape(X, -1)
    dB, deps = torch.empty_like(B), torch.zeros_like(eps)
    e = 0.0
    for i in range(o):
        M = (B[:, i, :].T @ flat).reshape(v, o, v)
        D = ev[:, None, None] + ev[None, None, :] - eo[i] - eo[None, :, None]
        T = M.transpose(0, 2)
        e = e - float(((2.0 * M - T) * M / D).sum())
        G = -(4.0 * M - 2.0 * T) / D
        dB[:, i, :] = 2.0 * flat @ G.reshape(v, -1).T
        W = (2.0 * M - T) * M / (D * D)
        deps[i] -= 2.0 * W.sum()
        deps[o:] += 2.0 * W.sum((1, 2))
    return e, dB, deps


def _inv_sqrt(J):
    w, V = np.linalg.eigh(J.cpu().numpy())
    keep = (w > 0) & (w / w.max() >= 1e-10)
    s = np.where(keep, 1.0 / np.sqrt(np.where(keep, w, 1.0)), 0.0)
    return torch.from_numpy((V * s) @ V.T).cuda()


def _mo_block(P, mos, o):
    """sum_mn C_im (P|mn) C_an as P[Q][i][a]."""
    X, n = P.shape[0], P.shape[1]
    h = torch.matmul(mos[:o], P)
    return (h.reshape(-1, n) @ mos[o:].T).reshape(X, o, n - o)


# Real solid harmonics m = -l..l as polynomials {(lx, ly, lz): coefficient}.
_HARMONICS = [
    [{(0, 0, 0): 1}],
    [{(0, 1, 0): 1}, {(0, 0, 1): 1}, {(1, 0, 0): 1}],
    [{(1, 1, 0): 1}, {(0, 1, 1): 1}, {(0, 0, 2): 2, (2, 0, 0): -1, (0, 2, 0): -1},
     {(1, 0, 1): 1}, {(2, 0, 0): 1, (0, 2, 0): -1}],
    [{(2, 1, 0): 3, (0, 3, 0): -1}, {(1, 1, 1): 1},
     {(0, 1, 2): 4, (2, 1, 0): -1, (0, 3, 0): -1},
     {(0, 0, 3): 2, (2, 0, 1): -3, (0, 2, 1): -3},
     {(1, 0, 2): 4, (3, 0, 0): -1, (1, 2, 0): -1}, {(2, 0, 1): 1, (0, 2, 1): -1},
     {(3, 0, 0): 1, (1, 2, 0): -3}],
]


def _boys(n, t):
    """F_0..F_n(t) from the incomplete gamma function and downward recursion."""
    big = torch.clamp(t, min=1e-10)
    h = n + 0.5
    top = torch.special.gammainc(torch.full_like(big, h), big) * math.gamma(h) / (2 * big ** h)
    out = [torch.where(t < 1e-3, 1 / (2 * n + 1) - t / (2 * n + 3) + t * t / (4 * n + 10)
                       - t ** 3 / (12 * n + 42) + t ** 4 / (48 * n + 216), top)]
    for m in range(n - 1, -1, -1):
        out.append((2 * t * out[-1] + torch.exp(-t)) / (2 * m + 1))
    return out[::-1]


def _hermite(la, lb, p, xpa, xpb):
    """E[i][j][t]: x_A^i x_B^j exp(..) in Hermite Gaussians of exponent p (1-d)."""
    E = {(0, 0): [torch.ones_like(p)]}

    def up(src, x):
        n = len(src)
        z = torch.zeros_like(p)
        return [(src[t - 1] / (2 * p) if t else z) + (x * src[t] if t < n else z)
                + ((t + 1) * src[t + 1] if t + 1 < n else z) for t in range(n + 1)]

    for i in range(la + 1):
        if i:
            E[i, 0] = up(E[i - 1, 0], xpa)
        for j in range(1, lb + 1):
            E[i, j] = up(E[i, j - 1], xpb)
    return E


class _Shell:
    def __init__(self, cols, s):
        l, nprim, poff, cen, ex, co = cols
        self.l, self.c = l[s], np.array(cen[3 * s:3 * s + 3])
        self.ex = np.array(ex[poff[s]:poff[s] + nprim[s]])
        # coefficients of normalised primitives; the contraction normalised below
        self.co = np.array(co[poff[s]:poff[s] + nprim[s]]) * self.ex ** ((2 * self.l + 3) / 4)
        r = self.co[:, None] * self.co[None] * (self.ex[:, None] + self.ex[None]) ** -(self.l + 1.5)
        self.co = self.co / math.sqrt(r.sum() * math.pi ** 1.5)


def _odd(n):
    return math.prod(range(n, 0, -2)) if n > 0 else 1


def _harmonic_rows(l):
    """Coefficients of the harmonics over the Cartesian powers, normalised with
    the radial part of _Shell."""
    cart = [(i, j, l - i - j) for i in range(l, -1, -1) for j in range(l - i, -1, -1)]
    rows = np.zeros((2 * l + 1, len(cart)))
    for m, poly in enumerate(_HARMONICS[l]):
        for c, f in poly.items():
            rows[m, cart.index(c)] = f
        n = sum(f * g * math.prod(_odd(x + y - 1) if (x + y) % 2 == 0 else 0
                                  for x, y in zip(c, d)) / 2.0 ** l
                for c, f in poly.items() for d, g in poly.items())
        rows[m] /= math.sqrt(n)
    return cart, torch.from_numpy(rows).cuda()


def _classes(cols):
    """Shells of one basis grouped by (l, primitives): {key: (indices, first function)}."""
    sh = [_Shell(cols, s) for s in range(len(cols[0]))]
    first = np.cumsum([0] + [2 * s.l + 1 for s in sh])
    groups = {}
    for n, s in enumerate(sh):
        groups.setdefault((s.l, len(s.ex)), []).append(n)
    return sh, first, groups


def _dev(rows):
    return torch.from_numpy(np.array(rows)).cuda()


def _exact_integrals(obs, aux):
    """(P|Q) and (P|mn) by the McMurchie-Davidson scheme in torch, one batch
    per class of shells: Hermite expansions of the pair and of the auxiliary
    shell, Hermite Coulomb integrals from the Boys function."""
    A, fa, ga = _classes(obs)
    D, fd, gd = _classes(aux)
    N, X = int(fa[-1]), int(fd[-1])
    pmn = torch.zeros((X, N, N), device="cuda", dtype=F64)
    J = torch.zeros((X, X), device="cuda", dtype=F64)

    def side(shells, la, lb, pairs, first):
        """Primitive pairs of a list of shell pairs (second None: a single shell)."""
        a = _dev([shells[i].ex for i, _ in pairs])
        ca = _dev([shells[i].co for i, _ in pairs])
        Ac = _dev([shells[i].c for i, _ in pairs])
        if lb is None:
            p, K, P = a, ca, Ac[:, None].expand(-1, a.shape[1], -1)
            E = [_hermite(la, 0, p, torch.zeros_like(p), torch.zeros_like(p)) for _ in range(3)]
            cb, rb = [(0, 0, 0)], torch.ones((1, 1), device="cuda", dtype=F64)
        else:
            b = _dev([shells[j].ex for _, j in pairs])
            cbv = _dev([shells[j].co for _, j in pairs])
            Bc = _dev([shells[j].c for _, j in pairs])
            a, b = a[:, :, None], b[:, None, :]
            p = (a + b).flatten(1)
            P = ((a[..., None] * Ac[:, None, None] + b[..., None] * Bc[:, None, None])
                 / (a + b)[..., None]).flatten(1, 2)
            K = (ca[:, :, None] * cbv[:, None, :]
                 * torch.exp(-a * b / (a + b) * ((Ac - Bc) ** 2).sum(-1)[:, None, None])).flatten(1)
            E = [_hermite(la, lb, p, P[..., x] - Ac[:, None, x], P[..., x] - Bc[:, None, x])
                 for x in range(3)]
            cb, rb = _harmonic_rows(lb)
        ca_, ra = _harmonic_rows(la)
        L = la + (lb or 0)
        hs = [(t, u, L2 - t - u) for L2 in range(L + 1) for t in range(L2, -1, -1)
              for u in range(L2 - t, -1, -1)]
        # H[pair][prim][(function pair)][hermite]
        H = torch.zeros(p.shape + (len(ca_), len(cb), len(hs)), device="cuda", dtype=F64)
        for i, x in enumerate(ca_):
            for j, y in enumerate(cb):
                for h, tuv in enumerate(hs):
                    if all(t <= x[d] + y[d] for d, t in enumerate(tuv)):
                        H[..., i, j, h] = E[0][x[0], y[0]][tuv[0]] * E[1][x[1], y[1]][tuv[1]] \
                            * E[2][x[2], y[2]][tuv[2]]
        H = torch.einsum("mi,nj,zpijh->zpmnh", ra, rb, H) * K[:, :, None, None, None]
        return p, P, H.flatten(2, 3), hs, L

    def coulomb(s1, s2):
        """sum over primitives of (pair 1 | pair 2): [pairs 2][pairs 1][f2][f1]."""
        p, P, H1, h1, L1 = s1
        q, Q, H2, h2, L2 = s2
        out = torch.zeros((q.shape[0], p.shape[0], H2.shape[2], H1.shape[2]), device="cuda",
                          dtype=F64)
        L = L1 + L2
        for i in range(p.shape[1]):
            for k in range(q.shape[1]):
                pi, qk = p[None, :, i], q[:, None, k]
                al = pi * qk / (pi + qk)
                r = P[None, :, i] - Q[:, None, k]
                F = _boys(L, al * (r * r).sum(-1))
                pre = 2 * math.pi ** 2.5 / (pi * qk * torch.sqrt(pi + qk))
                R = {(0, 0, 0, m): (-2 * al) ** m * F[m] * pre for m in range(L + 1)}
                for tot in range(1, L + 1):
                    for t in range(tot, -1, -1):
                        for u in range(tot - t, -1, -1):
                            c = (t, u, tot - t - u)
                            d = next(x for x in range(3) if c[x])
                            lo = tuple(v - (x == d) for x, v in enumerate(c))
                            lo2 = tuple(v - 2 * (x == d) for x, v in enumerate(c))
                            for m in range(L - tot + 1):
                                v = r[..., d] * R[lo + (m + 1,)]
                                if c[d] > 1:
                                    v = v + (c[d] - 1) * R[lo2 + (m + 1,)]
                                R[c + (m,)] = v
                for y, hy in enumerate(h2):
                    W = torch.zeros_like(out[:, :, 0])
                    for x, hx in enumerate(h1):
                        c = tuple(s + t for s, t in zip(hx, hy)) + (0,)
                        W += R[c][..., None] * H1[None, :, i, :, x]
                    out += (-1) ** sum(hy) * H2[:, None, k, :, y, None] * W[:, :, None, :]
        return out

    def functions(first, idx, l):
        return (torch.from_numpy(np.array([first[i] for i in idx])).cuda()[:, None]
                + torch.arange(2 * l + 1, device="cuda")[None])

    aux_sides = {k: (side(D, k[0], None, [(i, None) for i in idx], fd), functions(fd, idx, k[0]))
                 for k, idx in gd.items()}
    for k1, (s1, f1) in aux_sides.items():
        for k2, (s2, f2) in aux_sides.items():
            J[f2[:, None, :, None], f1[None, :, None, :]] = coulomb(s1, s2)
    for ka, ia in ga.items():
        for kb, ib in ga.items():
            if ka < kb:
                continue
            pairs = [(i, j) for i in ia for j in ib]
            for c0 in range(0, len(pairs), 4096):
                part = pairs[c0:c0 + 4096]
                s1 = side(A, ka[0], kb[0], part, fa)
                m = functions(fa, [i for i, _ in part], ka[0])
                n = functions(fa, [j for _, j in part], kb[0])
                for s2, f2 in aux_sides.values():
                    v = coulomb(s1, s2).reshape(f2.shape[0], len(part), f2.shape[1], m.shape[1],
                                                n.shape[1])
                    q = f2[:, None, :, None, None]
                    pmn[q, m[None, :, None, :, None], n[None, :, None, None, :]] = v
                    pmn[q, n[None, :, None, None, :], m[None, :, None, :, None]] = v
    return J, pmn


def exact(case, seed):
    k, o = case["kind"], case.get("nocc")
    x = _inputs(case, seed)
    if k == "integrals":
        return _exact_integrals(*x)
    if k == "energy":
        return _exact_mp2(*x, o, case["nvir"])
    if k == "batch":
        return np.concatenate([_exact_mp2(*b) for b in x])
    if k == "pipeline":
        mos, eps, J, P = x
        n = case["nbf"]
        B = (_inv_sqrt(J) @ _mo_block(P, mos, o).reshape(len(J), -1)).reshape(-1, o, n - o)
        return _exact_mp2(B, eps, o, n - o)
    if k == "calculate_ri":
        mos, _, J, P = x
        bpq = (_inv_sqrt(J) @ P.reshape(len(J), -1)).reshape(P.shape)
        return bpq, _mo_block(bpq, mos, o)
    if k == "canonical":
        mos, fmat, eps, packed = x
        n = case["nbf"]
        t = packed.dense(n)
        for _ in range(4):  # transform the first index and move it to the end
            t = (mos @ t.reshape(n, -1)).reshape((n,) * 4).permute(1, 2, 3, 0).contiguous()
        M = t[:o, o:, :o, o:]
        D = eps[o:][None, :, None, None] + eps[o:][None, None, None, :] \
            - eps[:o][:, None, None, None] - eps[:o][None, None, :, None]
        os_ = -float((M * M / D).sum())
        ss = -float(((M - M.permute(0, 3, 2, 1)) * M / D).sum())
        return _four(ss, os_), mos @ fmat @ mos.T, t
    e, dB, deps = _exact_gradient(*(t.detach() for t in x), o, case["nvir"])
    if k == "autograd":
        return torch.tensor(e, dtype=F64, device="cuda"), dB, deps
    return e, dB, deps
