"""Performance cases of the spherical-shell transform core.

Each case is the work a program hands to the public entry points of
redondito_b200.sphp: transform pairs of scalar and vector fields in the three
array forms (FP64 plans, mixed plans on FP64 arrays, mixed plans on
single-precision arrays), the nonlinear step and the RK3 step, the radial
operators with the boundary solve, and a batch of unequal problems.  A case
is a dict of plain values:

  kind   "chain"  2D synthesis, 2D analysis, radial derivative
         "pair"   3D inverse and 3D forward of the named fields, in place
         "nl"     the right-hand sides of the nonlinear step
         "rk3"    one RK3 step of the state, in place
         "radial" two radial derivatives, D_l and v_imposebc
         "batch"  `problems` shells of unequal size as one batch
  form   "fp64", "mixed" or "f32" (mixed plan, single-precision arrays)
  fields "scalar", "vector" or "both" (pairs)

listed() and draw() give the cases, prepare() a program's arrays and plan,
run() one pass, work() the bytes and operations a pass cannot do without,
exact() the result in FP64 from plain torch and numpy.
"""
import math
import os
import random

import numpy as np
import torch

from redondito_b200 import sphp as S

CZ, OZ, RINT, REXT = 25, 5, 0.35, 1.0
NU, DT = 1e-3, 1e-6
KMAX = 8  # radial modes of the seeded fields
TABLES = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "redondito_b200", "tables")


def _size(lmax, nz, nlat=None, nphi=None):
    nlat = nlat or 4 * ((3 * (lmax + 1) + 7) // 8)
    return {"lmax": lmax, "nlat": nlat, "nphi": nphi or 2 * nlat, "nz": nz}


def listed():
    return [
        # the smallest shells: a chain of single calls on one field, where
        # launches and latency count; nz = 33 = 3 11 and 58 = 2 29 are the
        # reference's own radial sizes
        {"name": "chain31_nz33_fp64", "kind": "chain", "form": "fp64", **_size(31, 33, 48, 96)},
        {"name": "chain31_nz58_fp64", "kind": "chain", "form": "fp64", **_size(31, 58, 48, 96)},
        # a small shell of a serving mix: one scalar field on a mixed plan
        {"name": "pair63_scalar_mixed", "kind": "pair", "form": "mixed", "fields": "scalar", **_size(63, 64, 96, 192)},
        # a medium shell: the vector field of a solver in FP64
        {"name": "pair127_vector_fp64", "kind": "pair", "form": "fp64", "fields": "vector", **_size(127, 64, 192, 384)},
        # a truncation off the usual ones: the grid rule gives 260 x 520 = 8 5 13, and nz = 90 = 2 9 5
        {"name": "pair170_both_ragged_fp64", "kind": "pair", "form": "fp64", "fields": "both", **_size(170, 90)},
        # the nonlinear step of a production solver, FP64 and mixed
        {"name": "rk3_255_fp64", "kind": "rk3", "form": "fp64", **_size(255, 128, 384, 768)},
        {"name": "nl_255_mixed", "kind": "nl", "form": "mixed", **_size(255, 128, 384, 768)},
        # the radial operators and the boundary solve of the same solver
        {"name": "radial_255_fp64", "kind": "radial", "form": "fp64", **_size(255, 96, 384, 768)},
        # one GPU's share of an ensemble of unequal shells
        {"name": "batch8_mixed", "kind": "batch", "form": "mixed", "problems": 8, "shape_seed": 4},
        # the large shell: a scalar and a vector field, in the three array forms
        {"name": "pair511_both_fp64", "kind": "pair", "form": "fp64", "fields": "both", **_size(511, 256, 768, 1536)},
        {"name": "pair511_both_mixed", "kind": "pair", "form": "mixed", "fields": "both", **_size(511, 256, 768, 1536)},
        {"name": "pair511_both_f32", "kind": "pair", "form": "f32", "fields": "both", **_size(511, 256, 768, 1536)},
    ]


def _smooth(n, most=31):
    """whether n has no prime factor above `most`"""
    for q in range(2, most + 1):
        while n % q == 0:
            n //= q
    return n == 1


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["chain", "pair", "pair", "pair", "pair", "pair", "nl", "rk3", "radial", "batch"])
    form = rng.choice(["fp64", "mixed", "f32"] if kind == "pair" else
                      ["fp64"] if kind in ("chain", "radial") else ["fp64", "mixed"])
    if kind == "batch":
        return {"kind": kind, "form": form, "problems": rng.randint(2, 8), "shape_seed": rng.randint(10, 10 ** 6)}
    top = {"chain": 63, "pair": 511, "nl": 255, "rk3": 255, "radial": 255}[kind]
    while True:
        lmax = _log_int(rng, 31, top)
        size = _size(lmax, 0)
        if form != "fp64":  # mixed plans: nphi = 3 2^a
            nphi = 48
            while nphi < size["nphi"]:
                nphi *= 2
            size = _size(lmax, 0, nphi // 2, nphi)
        if _smooth(size["nphi"]):
            break
    while True:
        nz = _log_int(rng, 33, 256 if kind == "pair" else 128)
        if kind in ("nl", "rk3", "radial"):
            nz = max(nz, 48)
        if rng.random() < 0.5:  # half of them the lengths that programs like best
            nz = min((48, 64, 96, 128, 192, 256), key=lambda v: abs(math.log(v / nz)))
        if _smooth(nz) and (kind == "pair" or nz <= 128):
            break
    case = {"kind": kind, "form": form, **size, "nz": nz}
    if kind == "pair":
        case["fields"] = rng.choice(["scalar", "vector", "both"])
    return case


def _problems(case):
    """The shells of a batch: (lmax, nz, fields), lmax 63, 127 or 255, nz 32, 64, 96 or 128."""
    r = random.Random(case["shape_seed"])
    return [(r.choice((63, 127, 255)), r.choice((32, 64, 96, 128)), r.randint(1, 3)) for _ in range(case["problems"])]


def _nfields(case):
    return {"scalar": 1, "vector": 3, "both": 4}[case["fields"]]


# ---------------------------------------------------------------- inputs
def _dir():
    """The FC-Gram continuation operator A Q^T, (CZ, OZ)."""
    a = np.fromfile(os.path.join(TABLES, f"A{CZ}-{OZ}.dat")).reshape(OZ, CZ).T
    q = np.fromfile(os.path.join(TABLES, f"Q{OZ}.dat")).reshape(OZ, OZ).T
    return torch.from_numpy(a @ q.T).cuda()


def _radii(nz):
    return RINT + (REXT - RINT) / (nz - CZ - 1) * torch.arange(nz, dtype=torch.float64, device="cuda")


def _lm(lmax):
    ell = torch.cat([torch.arange(m, lmax + 1, dtype=torch.float64) for m in range(lmax + 1)]).cuda()
    emm = torch.cat([torch.full((lmax + 1 - m,), m) for m in range(lmax + 1)]).cuda()
    return ell, emm


def _field(lmax, nz, gen, power, basis):
    """A smooth random spectral field in (r, lm): sum_k c_k,lm basis_k(r), with
    c ~ N(0, 1) (l+1)^-power (k+1)^-2, real for m = 0."""
    ell, emm = _lm(lmax)
    nk, nlm = basis.shape[1], ell.numel()
    c = torch.randn((2, nk, nlm), generator=gen, device="cuda", dtype=torch.float64)
    c *= (ell + 1.0) ** -power * (torch.arange(nk, device="cuda", dtype=torch.float64)[:, None] + 1.0) ** -2
    c[1][:, emm == 0] = 0.0
    return torch.complex(basis @ c[0], basis @ c[1])


def _cosines(nz):
    x = (_radii(nz) - RINT) / (REXT - RINT)
    return torch.cos(math.pi * x[:, None] * torch.arange(KMAX + 1, device="cuda", dtype=torch.float64))


def _continued(a, d):
    """a (rows, ...) with its last CZ rows the continuation of the others."""
    n = a.shape[0] - CZ
    flat = a[:n].reshape(n, -1)
    cont = d.to(a.dtype) @ flat[n - OZ:] + d.flip(0).to(a.dtype) @ flat[:OZ].flip(0)
    return torch.cat([a[:n], cont.reshape((CZ,) + a.shape[1:])])


def _forward_z(a, d):
    return torch.fft.fft(_continued(a, d), dim=0, norm="forward")


def _derivative(a, d, order):
    nz = a.shape[0]
    kz = torch.fft.fftfreq(nz, 1.0 / nz, device="cuda", dtype=torch.float64)
    kz *= 2.0 * math.pi / ((REXT - RINT) / (nz - CZ - 1) * nz)
    return torch.fft.ifft((1j * kz)[:, None] ** order * _forward_z(a, d), dim=0, norm="forward")


def _dl(a, lmax, d):
    ell, _ = _lm(lmax)
    return _derivative(a, d, 2) - (ell * (ell + 1.0)) / _radii(a.shape[0])[:, None] ** 2 * a


def _walls(nz):
    """Radial modes that vanish at both walls with their first derivative."""
    x = (_radii(nz) - RINT) / (REXT - RINT)
    return torch.sin(math.pi * x)[:, None] ** 2 * _cosines(nz)


def _state(lmax, nz, gen, d):
    """(Z, W, phi = D_l W) of a flow at rest on both walls."""
    Z, W = (_field(lmax, nz, gen, 3.0, _walls(nz)) for _ in range(2))
    W[:, 0] = 0.0
    return Z, W, _dl(W, lmax, d)


def _inputs(case, seed):
    """The seeded spectra of a case, FP64."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    d = _dir()
    if case["kind"] == "batch":
        return [[_forward_z(_field(l, nz, gen, 2.0, _cosines(nz)), d) for _ in range(nf)] for l, nz, nf in _problems(case)]
    lmax, nz = case["lmax"], case["nz"]
    if case["kind"] == "chain":
        return [_field(lmax, nz, gen, 2.0, _cosines(nz))]
    if case["kind"] == "pair":
        return [_forward_z(_field(lmax, nz, gen, 2.0, _cosines(nz)), d) for _ in range(_nfields(case))]
    return list(_state(lmax, nz, gen, d))


# ---------------------------------------------------------------- a program's state and one pass
_kept = {}  # the plans of the sizes in use: a program lays them out once


def _plans(key, make):
    if key not in _kept:
        _kept.clear()
        _kept[key] = make()
    return _kept[key]


def _plan(lmax, nz, nlat, nphi, form):
    return S.Plan(lmax, nz, nlat=nlat, nphi=nphi, Cz=CZ, oz=OZ, rint=RINT, rext=REXT,
                  precision=S.SPH_FP64 if form == "fp64" else S.SPH_MIXED)


def prepare(case, seed):
    x = _inputs(case, seed)
    form = case["form"]
    if case["kind"] == "batch":
        probs = _problems(case)
        plans = _plans(("batch", form, tuple(probs)), lambda: [
            _plan(l, nz, 3 * (l + 1) // 2, 3 * (l + 1), form) for l, nz, _ in probs])
        batch = S.Batch(plans, [nf for _, _, nf in probs])
        for dst, src in zip(batch.spec, x):
            for a, b in zip(dst, src):
                a.copy_(b)
        return {"kind": "batch", "batch": batch}
    size = (case["lmax"], case["nz"], case["nlat"], case["nphi"])
    flow = case["kind"] in ("nl", "rk3", "radial")

    def make():
        plan = _plan(*size, form)
        if flow:
            S.setup_bc(plan)
        return plan
    plan = _plans((size, form, flow), make)
    st = {"kind": case["kind"], "form": form, "fields": case.get("fields"), "plan": plan}
    if form == "f32":
        st["spec"] = [a.to(torch.complex64).contiguous() for a in x]
        st["grid"] = [plan.new_grid32() for _ in x]
    else:
        st["spec"] = [a.contiguous() for a in x]
        grids = {"chain": 1, "pair": len(x)}.get(case["kind"], 0)
        st["grid"] = [plan.new_grid() for _ in range(grids)]
        st["out"] = [plan.new_spec() for _ in range({"chain": 2, "nl": 2, "radial": 3}.get(case["kind"], 0))]
    return st


def run(st):
    kind = st["kind"]
    if kind == "batch":
        B = st["batch"]
        B.run()
        return {"spec": B.spec, "grid": B.grid, "dspec": B.dspec}
    P, a, g = st["plan"], st["spec"], st["grid"]
    if kind == "chain":
        s, d = st["out"]
        S.fftp2d_complex_to_real_xy(P, a[0], g[0])
        S.fftp2d_real_to_complex_xy(P, g[0], s)
        S.derivr(P, s, d, 1, "r")
        return {"grid": g[0], "spec": s, "derivative": d}
    if kind == "pair":
        tail = "_f32" if st["form"] == "f32" else ""
        inv, fwd, vinv, vfwd = (getattr(S, n + tail) for n in (
            "fftp3d_complex_to_real", "fftp3d_real_to_complex", "fftp3d_qst_to_vec", "fftp3d_vec_to_qst"))
        scalar = st["fields"] != "vector"
        if scalar:
            inv(P, a[0], g[0])
        if st["fields"] != "scalar":
            v = slice(1, 4) if scalar else slice(0, 3)
            vinv(P, *a[v], *g[v])
        if scalar:
            fwd(P, g[0], a[0])
        if st["fields"] != "scalar":
            vfwd(P, *g[v], *a[v])
        return {"grid": g, "spec": a}
    Z, W, phi = a
    if kind == "nl":
        rz, rp = st["out"]
        e = S.nl_rhs(P, Z, W, phi, NU, rz, rp)
        return {"rhs_z": rz, "rhs_phi": rp, "energy": e}
    if kind == "rk3":
        e = S.rk3_step(P, Z, W, phi, NU, DT)
        return {"Z": Z, "W": W, "phi": phi, "energy": e}
    d1, d2, dl = st["out"]
    S.derivr(P, Z, d1, 1, "r")
    S.derivr(P, W, d2, 2, "r")
    S.dlr(P, W, dl)
    S.v_imposebc(P, Z, phi, W)
    return {"d1": d1, "d2": d2, "dl": dl, "Z": Z, "phi": phi, "W": W}


# ---------------------------------------------------------------- what a pass cannot do without
def _cost(lmax, nlat, nphi, nz, nfield, nvec, f32=False):
    """(bytes, flops) of one direction of `nfield` fields, nvec of them vector components 2 and 3."""
    nlm = (lmax + 1) * (lmax + 2) // 2
    item = 4 if f32 else 8
    size = nfield * nz * item * (nlat * nphi + 2 * nlm)
    leg = 4.0 * nz * (nlat // 2) * nlm * ((nfield - nvec) + 2 * nvec)
    fft = nfield * nz * nlat * 2.5 * nphi * math.log2(nphi) + nfield * nlm * 5.0 * nz * math.log2(nz)
    return size, leg + fft


def work(case):
    if case["kind"] == "batch":
        b = f = 0.0
        for l, nz, nf in _problems(case):
            size, flops = _cost(l, 3 * (l + 1) // 2, 3 * (l + 1), nz, nf, 0)
            nlm = (l + 1) * (l + 2) // 2
            b += 2 * size + nf * 16.0 * nz * nlm
            f += 2 * flops + nf * 10.0 * nlm * nz * math.log2(nz)
        return {"bytes": b, "flops": f}
    size = (case["lmax"], case["nlat"], case["nphi"], case["nz"])
    nz, nlm = case["nz"], (case["lmax"] + 1) * (case["lmax"] + 2) // 2
    spec, zfft = 16.0 * nz * nlm, 5.0 * nlm * nz * math.log2(nz)
    solve = 4.0 * nlm * (nz - CZ) * (nz - CZ - 4)
    if case["kind"] == "chain":
        b, f = _cost(*size, 1, 0)
        return {"bytes": 2 * b + 2 * spec, "flops": 2 * f + 2 * zfft}
    if case["kind"] == "pair":
        n = _nfields(case)
        b, f = _cost(*size, n, 2 if n > 1 else 0, case["form"] == "f32")
        return {"bytes": 2 * b, "flops": 2 * f}
    if case["kind"] == "radial":  # Z, W in; three derivatives out; Z, phi, W out; the matrices
        binv = 8.0 * case["lmax"] * (nz - CZ) * (nz - CZ - 4)
        return {"bytes": 9 * spec + binv, "flops": 8 * zfft + solve}
    _, f = _cost(*size, 3, 2)
    rhs = 3 * f + 10 * zfft
    if case["kind"] == "nl":  # Z, W, phi in; two right-hand sides out
        return {"bytes": 5 * spec, "flops": rhs}
    binv = 8.0 * case["lmax"] * (nz - CZ) * (nz - CZ - 4)
    return {"bytes": 6 * spec + 3 * binv, "flops": 3 * (rhs + solve + 2 * zfft)}


# ---------------------------------------------------------------- the results in FP64, without the library
def _gauss(nlat):
    """Gauss-Legendre nodes (descending) and weights, Newton in long double."""
    i = np.arange(nlat, dtype=np.longdouble)
    x = np.cos(np.longdouble(math.pi) * (i + 0.75) / (nlat + 0.5))
    for _ in range(8):
        a, b = np.ones_like(x), x
        for k in range(2, nlat + 1):
            a, b = b, ((2 * k - 1) * x * b - (k - 1) * a) / k
        dp = nlat * (x * b - a) / (x * x - 1)
        x = x - b / dp
    return x, 2 / ((1 - x * x) * dp * dp)


class _Sphere:
    """Orthonormal spherical harmonics on the Gauss grid, dense FP64 tables."""

    def __init__(self, lmax, nlat, nphi):
        self.lmax, self.nlat, self.nphi = lmax, nlat, nphi
        x, w = _gauss(nlat)
        s = torch.from_numpy(np.sqrt((1 - x) * (1 + x)).astype(np.float64)).cuda()
        self.w = torch.from_numpy((w * 2 * np.longdouble(math.pi) / nphi).astype(np.float64)).cuda()
        x = torch.from_numpy(x.astype(np.float64)).cuda()
        m = torch.arange(lmax + 1, device="cuda", dtype=torch.float64)[:, None]
        p = torch.zeros((lmax + 1, lmax + 1, nlat), device="cuda", dtype=torch.float64)  # [l][m][node]
        dp = torch.zeros_like(p)
        top = torch.full((nlat,), math.sqrt(0.25 / math.pi), device="cuda", dtype=torch.float64)
        for l in range(lmax + 1):
            if l:
                top = top * s * math.sqrt((2.0 * l + 1.0) / (2.0 * l))
            k = m[:l]
            if l:
                a = torch.sqrt((4.0 * l * l - 1.0) / (l * l - k * k))
                b = torch.sqrt(((l - 1.0) ** 2 - k * k).clamp(min=0) / (4.0 * (l - 1.0) ** 2 - 1.0)) if l > 1 else 0.0 * k
                p[l, :l] = a * (x * p[l - 1, :l] - (b * p[l - 2, :l] if l > 1 else 0.0))
            p[l, l] = top
            k = m[:l + 1]
            c = torch.sqrt((2.0 * l + 1.0) * (l * l - k * k) / max(2.0 * l - 1.0, 1.0))
            dp[l, :l + 1] = (l * x * p[l, :l + 1] - (c * p[l - 1, :l + 1] if l else 0.0)) / s
        self.p, self.dp, self.mp = p, dp, p * m / s
        self.at = [mm * (2 * lmax + 1 - mm) // 2 + mm for mm in range(lmax + 1)]

    def _cols(self, a, m):
        return a[:, self.at[m]:self.at[m] + self.lmax + 1 - m]

    def _grid(self, terms):
        """terms: [(spectra, tables, factor)] summed -> the physical field."""
        nz = terms[0][0].shape[0]
        F = torch.zeros((nz, self.nphi // 2 + 1, self.nlat), device="cuda", dtype=torch.complex128)
        for m in range(self.lmax + 1):
            for a, tab, f in terms:
                F[:, m] += f * (self._cols(a, m) @ tab[m:, m].to(torch.complex128))
        return torch.fft.irfft(F, n=self.nphi, dim=1, norm="forward")

    def _spec(self, terms):
        """terms: [(Fourier coefficients, tables, factor)] summed -> spectra."""
        out = [sum(f * ((F[:, m] * self.w) @ tab[m:, m].T.to(torch.complex128)) for F, tab, f in terms)
               for m in range(self.lmax + 1)]
        out[0] = out[0].real.to(torch.complex128)
        return torch.cat(out, dim=1)

    def _fourier(self, g):
        return torch.fft.rfft(g, dim=1)[:, :self.lmax + 1]

    def scalar_grid(self, a):
        return self._grid([(a, self.p, 1.0)])

    def scalar_spec(self, g):
        return self._spec([(self._fourier(g), self.p, 1.0)])

    def vector_grid(self, q, s, t):
        return (self.scalar_grid(q), self._grid([(s, self.dp, 1.0), (t, self.mp, 1j)]),
                self._grid([(s, self.mp, 1j), (t, self.dp, -1.0)]))

    def vector_spec(self, vr, vt, vp):
        ell, _ = _lm(self.lmax)
        f = 1.0 / (ell * (ell + 1.0)).clamp(min=1.0) * (ell > 0)
        Ft, Fp = self._fourier(vt), self._fourier(vp)
        return (self.scalar_spec(vr), f * self._spec([(Ft, self.dp, 1.0), (Fp, self.mp, -1j)]),
                f * self._spec([(Ft, self.mp, -1j), (Fp, self.dp, -1.0)]))


def _exact_pair(x, sph, d, fields):
    r = [torch.fft.ifft(a, dim=0, norm="forward") for a in x]
    grid = []
    if fields != "vector":
        grid.append(sph.scalar_grid(r[0]))
    if fields != "scalar":
        grid += sph.vector_grid(*r[-3:])
    spec = []
    if fields != "vector":
        spec.append(sph.scalar_spec(grid[0]))
    if fields != "scalar":
        spec += sph.vector_spec(*grid[-3:])
    return r, grid, [_forward_z(a, d) for a in spec]


def _exact_nl(Z, W, phi, sph, d):
    ell, _ = _lm(sph.lmax)
    nz, ll = Z.shape[0], ell * (ell + 1.0)
    r = _radii(nz)[:, None]
    n = nz - CZ
    u = sph.vector_grid(ll * W / r ** 2, _derivative(W, d, 1) / r, Z / r)
    o = sph.vector_grid(ll * Z / r ** 2, _derivative(Z, d, 1) / r, -phi / r)
    trap = torch.ones(n, device="cuda", dtype=torch.float64)
    trap[0] = trap[-1] = 0.5
    shell = sum((c[:n] ** 2 * sph.w).sum(dim=(1, 2)) for c in u)
    e = 0.5 * float((trap * _radii(nz)[:n] ** 2 * shell).sum()) * (REXT - RINT) / (n - 1)
    N = [u[(i + 1) % 3] * o[(i + 2) % 3] - u[(i + 2) % 3] * o[(i + 1) % 3] for i in range(3)]
    for c in N:
        c[n:] = 0.0
    q, s, t = sph.vector_spec(*N)
    return (r * t + NU * _dl(Z, sph.lmax, d), _derivative(r * s, d, 1) - q + NU * _dl(phi, sph.lmax, d), e)


class _Walls:
    """v_imposebc for no-slip walls: one dense solve per degree."""

    def __init__(self, lmax, nz, d):
        n, self.lmax, self.d = nz - CZ, lmax, d
        eye = torch.zeros((nz, n), device="cuda", dtype=torch.complex128)
        eye[:n] = torch.eye(n, device="cuda", dtype=torch.float64).to(torch.complex128)
        d1, d2 = (_derivative(eye, d, k).real[:n] for k in (1, 2))
        l = torch.arange(1, lmax + 1, device="cuda", dtype=torch.float64)
        B = d2.repeat(lmax, 1, 1) - torch.diag_embed((l * (l + 1.0))[:, None] / _radii(nz)[:n] ** 2)
        B[:, 0], B[:, 1], B[:, n - 2], B[:, n - 1] = 0.0, d1[0], d1[n - 1], 0.0
        B[:, 0, 0] = B[:, n - 1, n - 1] = 1.0
        scale = B.abs().amax(dim=2, keepdim=True)
        self.inv = (torch.linalg.inv(B / scale) / scale.transpose(1, 2))[:, :, 2:n - 2]

    def __call__(self, Z, phi):
        ell, _ = _lm(self.lmax)
        n = Z.shape[0] - CZ
        Z = Z.clone()
        Z[0] = Z[n - 1] = 0.0
        W = torch.zeros_like(phi)
        for l in range(1, self.lmax + 1):
            c = (ell == l).nonzero()[:, 0]
            W[:n, c] = self.inv[l - 1].to(torch.complex128) @ phi[2:n - 2, c]
        return Z, W, _dl(W, self.lmax, self.d)


def exact(case, seed):
    if case.get("lmax", 0) > 260:
        return None  # the dense tables and transforms of the large shells take too long
    x, d = _inputs(case, seed), _dir()
    if case["form"] == "f32":
        x = [a.to(torch.complex64).to(torch.complex128) for a in x]
    kind = case["kind"]
    if kind == "batch":
        out = {"spec": [], "grid": [], "dspec": []}
        for (l, nz, _), xs in zip(_problems(case), x):
            sph = _Sphere(l, 3 * (l + 1) // 2, 3 * (l + 1))
            got = [_exact_pair([a], sph, d, "scalar") for a in xs]
            out["spec"].append([s[0] for _, _, s in got])
            out["grid"].append([g[0] for _, g, _ in got])
            out["dspec"].append([_derivative(r[0], d, 1) for r, _, _ in got])
        return out
    if kind == "radial":
        Z, W, phi = x
        Zb, Wb, phib = _Walls(case["lmax"], case["nz"], d)(Z, phi)
        return {"d1": _derivative(Z, d, 1), "d2": _derivative(W, d, 2), "dl": _dl(W, case["lmax"], d),
                "Z": Zb, "phi": phib, "W": Wb}
    sph = _Sphere(case["lmax"], case["nlat"], case["nphi"])
    if kind == "chain":
        g = sph.scalar_grid(x[0])
        s = sph.scalar_spec(g)
        return {"grid": g, "spec": s, "derivative": _derivative(s, d, 1)}
    if kind == "pair":
        _, grid, spec = _exact_pair(x, sph, d, case["fields"])
        return {"grid": grid, "spec": spec}
    Z, W, phi = x
    if kind == "nl":
        rz, rp, e = _exact_nl(Z, W, phi, sph, d)
        return {"rhs_z": rz, "rhs_phi": rp, "energy": e}
    walls, Z0, F0, energy = _Walls(case["lmax"], case["nz"], d), Z, phi, None
    for o in (3, 2, 1):
        rz, rp, e = _exact_nl(Z, W, phi, sph, d)
        energy = e if o == 3 else energy
        Z, W, phi = walls(Z0 + DT / o * rz, F0 + DT / o * rp)
    return {"Z": Z, "W": W, "phi": phi, "energy": energy}
