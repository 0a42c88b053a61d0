"""Performance cases of the spherical-transform framework.

Every case is work that a time-stepping program has the library do through its
public entry points: the full cycle (backward transform, grid products, forward
transform) in the three precision tiers, the separable backward and forward
transforms, the spectral post-processing of one step, host-resident spectra and
batched instances, from the smallest shells to the largest angular grids.

``exact`` restates each path in 64 bits with plain numpy / torch: Schmidt
functions by their recurrence in extended precision, the Legendre sums as dense
products, the longitudinal transforms by torch.fft.
"""
from __future__ import annotations

import math
from concurrent.futures import ThreadPoolExecutor

import numpy as np
import torch

from kemorin_mhd_b200.config import (FIELD_SETS, PROD_CROSS, PROD_DOT, PROD_VEC_SCALAR, R_CMB, R_ICB, TIER_FP32ACC,
                                     TIER_FP64, TIER_SPLIT_I8, SphConfig)
from kemorin_mhd_b200.sph_trans import SphTransform, batch_cycle

TIERS = {"fp64": TIER_FP64, "split": TIER_SPLIT_I8, "fp32acc": TIER_FP32ACC}
# field sets of the MHD transforms, and the two- and three-field sets of a
# convection or a non-magnetic run
SETS = dict(FIELD_SETS)
SETS["heat"] = dict(nvb=1, nsb=1, nvf=1, nsf=0, products=((PROD_VEC_SCALAR, 0, 0, 1.0),))
SETS["convection"] = dict(nvb=2, nsb=1, nvf=2, nsf=1,
                          products=((PROD_CROSS, 1, 0, 1.0), (PROD_VEC_SCALAR, 0, 0, 1.0), (PROD_DOT, 0, 1, 1.0)))

# grid values times components of the largest drawn case
DRAW_CAP = 24 * 768 * 1536 * 20


def listed():
    c = []
    # smallest shell in use (the dynamo benchmark's truncation): launches and host time count
    c.append(dict(name="cycle_fp64_L31_Nr33", kind="cycle", tier="fp64", L=31, nth=48, nph=96, nr=33))
    # truncation and grid off every tile size: odd latitudes, longitudes with a factor 81, odd radii
    c.append(dict(name="cycle_fp64_L106_Nr47_odd", kind="cycle", tier="fp64", L=106, nth=161, nph=324, nr=47))
    # grid output: fields on the sphere for diagnostics and for products formed by the caller
    c.append(dict(name="btrans_split_L127_Nr65", kind="b_trans", tier="split", L=127, nth=192, nph=384, nr=65))
    # forces the caller formed on the grid back to spectra, plain FP64
    c.append(dict(name="ftrans_fp64_L127_Nr65", kind="f_trans", tier="fp64", L=127, nth=192, nph=384, nr=65))
    # a host program (Fortran time loop) with page-locked spectra in and out
    c.append(dict(name="host_split_L127_Nr65", kind="host", tier="split", L=127, nth=192, nph=384, nr=65))
    # ordinary production size, split tier
    c.append(dict(name="cycle_split_L255_Nr129", kind="cycle", tier="split", L=255, nth=384, nph=768, nr=129))
    # the same size, plain FP64, with the Coriolis curl inside the cycle as the time loop has it
    c.append(dict(name="cycle_fp64_coriolis_L255_Nr129", kind="cycle", tier="fp64", L=255, nth=384, nph=768, nr=129,
                  coriolis=True))
    # curls, divergence, Coriolis and buoyancy of one time step on the spectra
    c.append(dict(name="post_L255_Nr129", kind="post", tier="fp64", L=255, nth=384, nph=768, nr=129))
    # dynamo field set with the Lorentz force on the largest lines that fit shared memory
    c.append(dict(name="dynamo_split_L511_Nr33", kind="cycle", tier="split", L=511, nth=768, nph=1536, nr=33,
                  fields="dynamo"))
    # the cheapest tier, for runs that need 1e-6
    c.append(dict(name="cycle_fp32acc_L511_Nr65", kind="cycle", tier="fp32acc", L=511, nth=768, nph=1536, nr=65))
    # largest angular grid (wide lines), plain FP64
    c.append(dict(name="cycle_fp64_L1023_Nr17", kind="cycle", tier="fp64", L=1023, nth=1536, nph=3072, nr=17))
    # largest work: the benchmark's angular grid with half its radii
    c.append(dict(name="cycle_split_L511_Nr129", kind="cycle", tier="split", L=511, nth=768, nph=1536, nr=129))
    return c


def _smooth(n):
    """Smallest even 2^a 3^b 5^c >= n."""
    while True:
        r = n
        for q in (2, 3, 5):
            while r % q == 0:
                r //= q
        if r == 1 and n % 2 == 0:
            return n
        n += 1


def draw(rng):
    kind = rng.choice(["cycle"] * 6 + ["b_trans", "f_trans", "post", "host", "batch"])
    while True:
        c = dict(kind=kind, tier=rng.choice(["fp64", "split", "split", "fp32acc"]))
        if kind == "batch":
            c.update(L=rng.choice([31, 63, 127]), nr=rng.randint(9, 33), n=rng.randint(3, 8), nth=0, nph=0)
            c["nth"], c["nph"] = 3 * (c["L"] + 1) // 2, 3 * (c["L"] + 1)
            return c
        if rng.random() < 0.5:  # the usual dealiased grids
            L = rng.choice([31, 63, 127, 255, 511])
            nth, nph = 3 * (L + 1) // 2, 3 * (L + 1)
        else:  # any truncation, odd latitude counts, wider longitudes
            L = int(round(math.exp(rng.uniform(math.log(15), math.log(511)))))
            nth = 3 * (L + 1) // 2 + rng.randint(0, 5)
            nph = _smooth(3 * L + 1 + rng.randint(0, L // 4))
        nr = int(round(math.exp(rng.uniform(math.log(5), math.log(129)))))
        c.update(L=L, nth=nth, nph=nph, nr=nr)
        if kind in ("cycle", "host"):
            c["fields"] = rng.choice(["default", "default", "dynamo", "full", "convection", "heat"])
            c["coriolis"] = c["fields"] != "heat" and rng.random() < 0.25
        if kind == "cycle" and c["tier"] == "fp64":
            c["otf"] = rng.random() < 0.2
        if kind == "post":
            c["tier"] = "fp64"
        cfg = _cfg(c)
        if nr * nth * nph * (cfg.ncb + cfg.ncf) <= DRAW_CAP:
            return c


def _cfg(case):
    return SphConfig(case["L"], case["nth"], case["nph"], case["nr"], **SETS[case.get("fields", "default")])


def _batch_cfgs(case):
    """Uneven instances: falling truncations and radii, alternating field sets."""
    out = []
    for i in range(case["n"]):
        L = max(15, ((case["L"] + 1) >> (i % 3)) - 1)
        out.append(SphConfig(L, 3 * (L + 1) // 2, 3 * (L + 1), max(5, case["nr"] - 2 * i),
                             **SETS[("default", "convection", "heat")[i % 3]]))
    return out


# ---------------------------------------------------------------------------
# inputs

def _lm(L):
    m = np.concatenate([np.full(L - abs(k) + 1, k) for k in range(-L, L + 1)])
    l = np.concatenate([np.arange(abs(k), L + 1) for k in range(-L, L + 1)])
    return l, m


def _spectra(cfg, gen, extra=0):
    """(ncb + extra, nr, J) spectra: Gaussian amplitudes falling as (l + 1)^-2, four radial modes per
    coefficient, the radial derivative column consistent with its poloidal column."""
    dev = torch.device("cuda")
    l = torch.from_numpy(_lm(cfg.ltr)[0]).to(dev)
    decay = (l.double() + 1.0) ** -2
    r = torch.from_numpy(cfg.radius()).to(dev)
    x = math.pi * (r - R_ICB) / (R_CMB - R_ICB)
    q = torch.arange(1, 5, device=dev, dtype=torch.float64)
    s = torch.sin(q[None, :] * x[:, None] + 0.3) / q ** 2                                     # (nr, 4)
    ds = (math.pi / (R_CMB - R_ICB)) * torch.cos(q[None, :] * x[:, None] + 0.3) / q
    out = torch.zeros((cfg.ncb + extra, cfg.nr, cfg.J), dtype=torch.float64, device=dev)

    def amp(vec):
        a = torch.randn((4, cfg.J), generator=gen, dtype=torch.float64, device=dev) * decay
        return torch.where(l == 0, torch.zeros_like(a), a) if vec else a

    for v in range(cfg.nvb):
        a = amp(True)
        torch.matmul(s, a, out=out[3 * v])
        torch.matmul(ds, a, out=out[3 * v + 1])
        torch.matmul(s, amp(True), out=out[3 * v + 2])
    for k in range(cfg.nsb):
        torch.matmul(s, amp(False), out=out[3 * cfg.nvb + k])
    return out


def _grid(cfg, gen):
    """(ncf, nph, nth, nr) smooth grid fields: sums of separable band-limited waves."""
    dev = torch.device("cuda")

    def wave(n, k):  # (ncf, k, n)
        t = torch.arange(n, device=dev, dtype=torch.float64) * (2.0 * math.pi / n)
        f = torch.randint(0, max(2, n // 6), (cfg.ncf, k, 1), generator=gen, device=dev).double()
        p = torch.rand((cfg.ncf, k, 1), generator=gen, dtype=torch.float64, device=dev) * 6.0
        return torch.cos(f * t + p)

    k = 6
    tr = torch.einsum("ckt,ckr->cktr", wave(cfg.nth, k), wave(cfg.nr, k)).reshape(cfg.ncf, k, -1)
    return torch.bmm(wave(cfg.nph, k).transpose(1, 2), tr).contiguous()


def prepare(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    tier = TIERS[case["tier"]]
    f64 = dict(dtype=torch.float64, device="cuda")
    if kind == "batch":
        cfgs = _batch_cfgs(case)
        trs = [SphTransform(c, tier=tier) for c in cfgs]
        ins = [_spectra(c, gen).reshape(c.ncb, -1) for c in cfgs]
        outs = [torch.zeros((c.ncf, c.J * c.nr), **f64) for c in cfgs]
        torch.cuda.synchronize()
        return dict(kind=kind, tr=trs, d=ins, out=outs)
    cfg = _cfg(case)
    tr = SphTransform(cfg, tier=tier, p_on_the_fly=bool(case.get("otf")))
    st = dict(kind=kind, tr=tr, coriolis=bool(case.get("coriolis")), ncf=cfg.ncf)
    n = cfg.J * cfg.nr
    ncol = cfg.ncf + (3 if case.get("coriolis") else 0)
    if case.get("coriolis"):
        tr.set_coriolis(_COR, 0, 1, cfg.ncf)
    if kind in ("cycle", "host"):
        st["d"] = _spectra(cfg, gen).reshape(cfg.ncb, -1)
        st["out"] = torch.zeros((ncol, n), **f64)
        if kind == "host":
            st["d"] = st["d"].cpu().pin_memory()
            st["out"] = st["out"].cpu().pin_memory()
    elif kind == "b_trans":
        st["d"] = _spectra(cfg, gen).reshape(cfg.ncb, -1)
        st["out"] = torch.empty((cfg.ncb, cfg.nr * cfg.nth * cfg.nph), **f64)
    elif kind == "f_trans":
        st["d"] = _grid(cfg, gen).reshape(cfg.ncf, -1)
        st["out"] = torch.zeros((cfg.ncf, n), **f64)
    else:
        # columns: 0-2 u, 3-5 omega (input for Coriolis), 6-8 B, 9 T, then the results
        st["d"] = _spectra(cfg, gen, extra=_POST_COLS).reshape(cfg.ncb + _POST_COLS, -1)
    torch.cuda.synchronize()
    return st


_COR = 2000.0
_POST_COLS = 19
_POST_OUT = [(10, 13), (13, 16), (16, 19), (19, 22), (22, 23), (23, 24), (25, 26), (26, 27), (28, 29)]


def run(st):
    kind, tr, d = st["kind"], st["tr"], st["d"]
    if kind == "batch":
        batch_cycle(tr, d, st["out"])
        return st["out"]
    if kind in ("cycle", "host"):
        tr.nonlinear_cycle(d, st["out"])
    elif kind == "b_trans":
        tr.sph_b_trans(d, st["out"])
    elif kind == "f_trans":
        tr.sph_f_trans(d, st["out"])
    else:
        tr.vorticity(d, 0, 10)                # curl u, non-slip rows
        tr.current(d, 6, 13)                  # curl B, insulating rows
        tr.rot_force(d, 0, 16, 1, 0)          # curl of a force, free slip inside
        tr.rot_induction(d, 3, 19)            # curl of u x B, insulating rows
        tr.div_flux_bc(d, 5, 22, 0, 1)        # divergence of a flux, fixed field / fixed flux
        tr.div_force(d, 2, 23)
        tr.rot_buoyancy(d, 9, 1.5, 25)
        tr.rot_coriolis(d, 0, 3, 26, _COR)    # columns 26 and 28
        return [d[a:b] for a, b in _POST_OUT]
    if st["coriolis"]:  # forward fields, then the poloidal and toroidal columns of the curl
        return [st["out"][:st["ncf"]], st["out"][st["ncf"]::2]]
    return st["out"]


# ---------------------------------------------------------------------------
# what a pass cannot do without

def _cycle_work(cfg, back, fwd, grid_io):
    nnod = cfg.nr * cfg.nth * cfg.nph
    leg = 2.0 * cfg.nh * cfg.J * cfg.nr
    fft = 2.5 * nnod * math.log2(cfg.nph)
    n, fl = 0.0, 0.0
    if back:
        n += 8.0 * cfg.J * cfg.nr * cfg.ncb + (8.0 * nnod * cfg.ncb if grid_io else 0.0)
        fl += leg * (5 * cfg.nvb + cfg.nsb) + fft * cfg.ncb
    if fwd:
        n += 8.0 * cfg.J * cfg.nr * cfg.ncf + (8.0 * nnod * cfg.ncf if grid_io else 0.0)
        fl += leg * (5 * cfg.nvf + cfg.nsf) + fft * cfg.ncf
    return n, fl


def work(case):
    kind = case["kind"]
    if kind == "batch":
        w = [_cycle_work(c, True, True, False) for c in _batch_cfgs(case)]
        return dict(bytes=sum(x[0] for x in w), flops=sum(x[1] for x in w))
    cfg = _cfg(case)
    if kind == "post":
        # u, omega, B and T read once, eighteen columns written
        n = cfg.J * cfg.nr
        return dict(bytes=8.0 * n * (10 + 18), flops=120.0 * n)
    b, f = _cycle_work(cfg, kind != "f_trans", kind != "b_trans", kind in ("b_trans", "f_trans"))
    if case.get("coriolis"):
        b += 8.0 * cfg.J * cfg.nr * 2
        f += 40.0 * cfg.J * cfg.nr
    return dict(bytes=b, flops=f)


def tolerance(case):
    # 2-norm errors against `exact`, about four times the largest seen over the
    # listed cases and thirty drawn ones
    if case["kind"] == "post":
        # second differences on radii that crowd at the boundaries
        return {"rel": 2.5e-13}
    return {"rel": {"fp64": 4e-13, "split": 4e-13, "fp32acc": 1e-7}[case["tier"]]}


# ---------------------------------------------------------------------------
# 64-bit restatement

def _gauss(n):
    """Colatitudes and weights (x_1 near -1): Newton on P_n until |dz| < 3e-12, the weight taken with P'_n of
    the previous iterate, as the transform defines its quadrature."""
    i = np.arange(1, (n + 1) // 2 + 1, dtype=np.float64)
    z = np.cos(np.pi * (i - 0.25) / (n + 0.5))
    pp = np.ones_like(z)
    live = np.ones(z.shape, bool)
    for _ in range(100):
        p1, p2 = np.ones_like(z), np.zeros_like(z)
        for j in range(1, n + 1):
            p1, p2 = ((2.0 * j - 1.0) * z * p1 - (j - 1.0) * p2) / j, p1
        ppn = n * (z * p1 - p2) / (z * z - 1.0)
        pp = np.where(live, ppn, pp)
        zn = np.where(live, z - p1 / ppn, z)
        live &= np.abs(zn - z) >= 3.0e-12
        z = zn
        if not live.any():
            break
    w = 2.0 / ((1.0 - z * z) * pp * pp)
    th, wt = np.empty(n), np.empty(n)
    th[:len(z)], wt[:len(z)] = np.arccos(-z), w
    th[n - len(z):], wt[n - len(z):] = np.arccos(z)[::-1], w[::-1]
    return th, wt


def _schmidt(L, theta, m0, m1):
    """P and dP/dtheta of orders m0 <= m < m1, arrays (m, l, theta), zero for l < m."""
    ld = np.longdouble
    ct, st = np.cos(theta.astype(ld)), np.sin(theta.astype(ld))
    ms = np.arange(m0 - 1, m1 + 1)  # neighbours too
    # P_m^m = sqrt(2 (2m-1)!!/(2m)!!) sin^m
    pmm = np.zeros((len(ms), len(theta)), ld)
    c = ld(1)
    for m in range(0, m1 + 1):
        if m > 0:
            c = c * ld(2 * m - 1) / ld(2 * m)
        if m >= m0 - 1:
            pmm[m - (m0 - 1)] = 1 if m == 0 else np.sqrt(2 * c) * st ** m
    P = np.zeros((len(ms), L + 1, len(theta)), np.float64)
    dP = np.zeros((m1 - m0, L + 1, len(theta)), np.float64)
    a, b = np.zeros_like(pmm), np.zeros_like(pmm)  # P_{l-1}, P_{l-2}: zero until l = m
    m2 = (ms[:, None].astype(ld)) ** 2
    m = np.arange(m0, m1).astype(ld)[:, None]
    for l in range(max(0, m0 - 1), L + 1):
        lo = np.sqrt(np.maximum(ld(l) * l - m2, 1))
        v = ((ld(2 * l - 1) / lo) * ct) * a - (np.sqrt(np.maximum(ld(l - 1) * (l - 1) - m2, 0)) / lo) * b
        if m0 - 1 <= l <= m1:
            v[l - (m0 - 1)] = pmm[l - (m0 - 1)]
        a, b = v, a
        P[:, l] = v
        # dP_l^m = (sqrt((l+m)(l-m+1)) P^{m-1} - sqrt((l-m)(l+m+1)) P^{m+1}) / 2, Schmidt factors at m = 0, 1
        e = np.sqrt(np.maximum((l + m) * (l - m + 1), 0)) / 2
        f = np.sqrt(np.maximum((l - m) * (l + m + 1), 0)) / 2
        if m0 == 0:
            e[0] = 0
            f[0] *= np.sqrt(ld(2))
        if m0 <= 1 < m1:
            e[1 - m0] *= np.sqrt(ld(2))
        dP[:, l] = e * v[:-2] - f * v[2:]
    return P[1:-1], dP


class _Exact:
    """Dense transforms of one configuration, fields as (component, radius, order, [cos, sin], theta) spectra."""

    def __init__(self, cfg):
        self.cfg = cfg
        self.dev = torch.device("cuda")
        self.th, self.w = _gauss(cfg.nth)
        L = cfg.ltr
        l, m = _lm(L)
        pos = np.full((2, L + 1, L + 1), -1, np.int64)  # [slot][m][l] -> j
        pos[(m < 0).astype(int), np.abs(m), l] = np.arange(cfg.J)
        self.pos = torch.from_numpy(pos).to(self.dev)
        self.r = torch.from_numpy(cfg.radius()).to(self.dev)
        self.mb = 64
        self.tables = None

    def blocks(self):
        """(m0, m1, P, dP) per block of orders, tensors (m, l, theta) on the GPU for the whole meridian."""
        if self.tables is None:
            L, th = self.cfg.ltr, self.th[:self.cfg.nh]

            def block(m0):
                m1 = min(L + 1, m0 + self.mb)
                p, dp = _schmidt(L, th, m0, m1)
                return m0, m1, torch.from_numpy(p).to(self.dev), torch.from_numpy(dp).to(self.dev)

            with ThreadPoolExecutor(8) as pool:
                self.tables = list(pool.map(block, range(0, L + 1, self.mb)))
        sg = torch.where((torch.arange(self.cfg.ltr + 1, device=self.dev)) % 2 == 0, 1.0, -1.0).double()
        for m0, m1, p, dp in self.tables:
            s = (sg[None, :] * sg[m0:m1, None])[:, :, None]
            tail = self.cfg.nth // 2
            yield (m0, m1, torch.cat([p, (p * s)[:, :, :tail].flip(2)], 2),
                   torch.cat([dp, (-dp * s)[:, :, :tail].flip(2)], 2))

    def spec(self, d, m0, m1):
        """(k, nr, J) -> (m, slot, l, k, nr) with zeros where no mode exists."""
        q = self.pos[:, m0:m1]                                   # slot, m, l
        x = d[:, :, q.clamp(min=0)] * (q >= 0)                   # k, nr, slot, m, l
        return x.permute(3, 2, 4, 0, 1)

    def bwd(self, d):
        """(ncb, rc, J) spectra of radii self.rr -> (ncb, rc, nth, nph)."""
        c, rr = self.cfg, self.rr
        rc = d.shape[1]
        L = c.ltr
        co = torch.zeros((c.ncb, rc, c.nth, c.nph // 2 + 1), dtype=torch.complex128, device=self.dev)
        ms_ = torch.from_numpy(1.0 / np.sin(self.th)).to(self.dev)
        lg = torch.arange(L + 1, device=self.dev, dtype=torch.float64)
        g3 = torch.where(lg == 0, 0.5, lg * (lg + 1))
        for m0, m1, p, dp in self.blocks():
            nm = m1 - m0
            x = self.spec(d, m0, m1)                             # m, 2, l, ncb, rc

            def mul(t, v):  # (m, l, th), (m, 2, l, k, rc) -> (m, 2, k, rc, th)
                v = v.reshape(nm, 2, L + 1, -1)
                return torch.einsum("mlt,mslc->msct", t, v).reshape(nm, 2, -1, rc, c.nth)

            mm = torch.arange(m0, m1, device=self.dev, dtype=torch.float64).reshape(-1, 1, 1, 1) * ms_
            out = torch.zeros((nm, 2, c.ncb, rc, c.nth), dtype=torch.float64, device=self.dev)
            if c.nvb:
                v = x[:, :, :, :3 * c.nvb].reshape(nm, 2, L + 1, c.nvb, 3, rc)
                a = v[..., 0, :] * g3.reshape(1, 1, -1, 1, 1) / (rr * rr)
                b, t = v[..., 1, :] / rr, v[..., 2, :] / rr
                pb, pt, db, dt = mul(p, b), mul(p, t), mul(dp, b), mul(dp, t)
                out[:, :, 0:3 * c.nvb:3] = mul(p, a)
                out[:, 0, 1:3 * c.nvb:3] = db[:, 0] + mm * pt[:, 1]
                out[:, 1, 1:3 * c.nvb:3] = db[:, 1] - mm * pt[:, 0]
                out[:, 0, 2:3 * c.nvb:3] = -dt[:, 0] + mm * pb[:, 1]
                out[:, 1, 2:3 * c.nvb:3] = -dt[:, 1] - mm * pb[:, 0]
            if c.nsb:
                out[:, :, 3 * c.nvb:] = mul(p, x[:, :, :, 3 * c.nvb:])
            z = torch.complex(out[:, 0], -out[:, 1]) * 0.5       # x = sum 2 Re z e^{i m phi}
            co[..., m0:m1] = z.permute(1, 2, 3, 0)
        co[..., 0] = torch.complex(2.0 * co[..., 0].real, torch.zeros_like(co[..., 0].real))
        return torch.fft.irfft(co, n=c.nph, dim=-1, norm="forward")

    def fwd(self, g):
        """(ncf, rc, nth, nph) -> (ncf, rc, J)."""
        c, rr = self.cfg, self.rr
        rc, L = g.shape[1], c.ltr
        z = torch.fft.rfft(g, dim=-1, norm="forward")[..., :L + 1]
        z = z * torch.from_numpy(self.w).to(self.dev).reshape(1, 1, -1, 1)
        sc = torch.full((L + 1,), 2.0, dtype=torch.float64, device=self.dev)
        sc[0] = 1.0
        f = torch.stack([z.real * sc, -z.imag * sc])             # slot, ncf, rc, th, m
        f[1, ..., 0] = 0.0
        f = f.permute(4, 0, 1, 2, 3).contiguous()                # m, slot, ncf, rc, th
        out = torch.zeros((c.ncf, rc, c.J), dtype=torch.float64, device=self.dev)
        isin = torch.from_numpy(1.0 / np.sin(self.th)).to(self.dev)
        lg = torch.arange(L + 1, device=self.dev, dtype=torch.float64)
        for m0, m1, p, dp in self.blocks():
            nm = m1 - m0
            x = f[m0:m1]
            mm = torch.arange(m0, m1, device=self.dev, dtype=torch.float64)
            n0 = torch.where(mm == 0, 2.0, 4.0).reshape(-1, 1, 1, 1)
            l4 = lg.reshape(1, 1, 1, -1)
            g7 = (2 * l4 + 1) / (n0 * torch.where(l4 == 0, torch.ones_like(l4), l4 * (l4 + 1)))
            g7 = torch.where(l4 == 0, torch.ones_like(g7), g7)
            g6 = (2 * l4 + 1) / n0
            m4 = mm.reshape(-1, 1, 1, 1)

            def mul(t, v):  # (m, l, th), (m, 2, k, rc, th) -> (m, 2, k, rc, l)
                k = v.shape[2]
                return torch.einsum("mlt,msct->mscl", t, v.reshape(nm, 2, -1, c.nth)).reshape(nm, 2, k, rc, L + 1)

            res = torch.zeros((nm, 2, c.ncf, rc, L + 1), dtype=torch.float64, device=self.dev)
            if c.nvf:
                vr, vt, vp = (x[:, :, q:3 * c.nvf:3] for q in range(3))
                r1 = rr.reshape(1, 1, -1, 1)
                zz, wt, wp = mul(p, vr), mul(dp, vt), mul(dp, vp)
                up, ut = mul(p, vp * isin), mul(p, vt * isin)
                fac = r1 * g7
                for s, sg in ((0, 1.0), (1, -1.0)):
                    res[:, s, 0:3 * c.nvf:3] = zz[:, s] * r1 * fac
                    res[:, s, 1:3 * c.nvf:3] = (wt[:, s] - sg * m4 * up[:, 1 - s]) * fac
                    res[:, s, 2:3 * c.nvf:3] = (-sg * m4 * ut[:, 1 - s] - wp[:, s]) * fac
            if c.nsf:
                res[:, :, 3 * c.nvf:] = mul(p, x[:, :, 3 * c.nvf:]) * g6.reshape(nm, 1, 1, 1, -1)
            q = self.pos[:, m0:m1]
            slot, mi, li = torch.nonzero(q >= 0, as_tuple=True)
            out[:, :, q[slot, mi, li]] = res[mi, slot, :, :, li].permute(1, 2, 0)
        return out

    def products(self, g):
        c = self.cfg
        vec = [g[3 * v:3 * v + 3] for v in range(c.nvb)]
        scl = [g[3 * c.nvb + s] for s in range(c.nsb)]
        vout, sout = [], []
        for kind, a, b, cf in c.products:
            if kind == PROD_CROSS:
                vout.append(cf * torch.linalg.cross(vec[a], vec[b], dim=0))
            elif kind == PROD_VEC_SCALAR:
                vout.append(cf * vec[a] * scl[b])
            elif kind == PROD_DOT:
                sout.append(cf * (vec[a] * vec[b]).sum(0, keepdim=True))
            else:
                sout.append(cf * (scl[a] * scl[b])[None])
        return torch.cat(vout + sout)

    def over_radii(self, fn):
        """fn(r0, r1) over chunks of radii that keep the working set small."""
        c = self.cfg
        per = 16.0 * c.nth * c.nph * (c.ncb + c.ncf) * 4
        step = max(1, min(c.nr, int(6e9 / per)))
        for r0 in range(0, c.nr, step):
            r1 = min(c.nr, r0 + step)
            self.rr = self.r[r0:r1]
            fn(r0, r1)


def _exact_cycle(cfg, d):
    ex = _Exact(cfg)
    d = d.reshape(cfg.ncb, cfg.nr, cfg.J)
    out = torch.zeros((cfg.ncf, cfg.nr, cfg.J), dtype=torch.float64, device="cuda")

    def step(r0, r1):
        out[:, r0:r1] = ex.fwd(ex.products(ex.bwd(d[:, r0:r1])))

    ex.over_radii(step)
    return out.reshape(cfg.ncf, -1)


def _fdm(r):
    """Radial 3-point rows: interior first and second derivatives (nr, 3) and boundary Taylor inverses."""
    nr = len(r)
    d1, d2 = np.zeros((nr, 3)), np.zeros((nr, 3))
    for k in range(1, nr - 1):
        p, n = r[k + 1] - r[k], r[k] - r[k - 1]
        inv = np.linalg.inv(np.array([[1, -n, n * n / 2], [1, 0, 0], [1, p, p * p / 2]]))
        d1[k], d2[k] = inv[1], inv[2]
    return d1, d2


def _exact_post(cfg, d):
    dev = d.device
    nr, J = cfg.nr, cfg.J
    x = d.reshape(-1, nr, J)
    r = cfg.radius()
    rt = torch.from_numpy(r).to(dev)[:, None]
    l = torch.from_numpy(_lm(cfg.ltr)[0]).to(dev).double()
    g3 = l * (l + 1)
    d1, d2 = (torch.from_numpy(t).to(dev) for t in _fdm(r))
    h0, h1 = r[1] - r[0], r[-1] - r[-2]
    one = np.linalg.inv(np.array([[1, 0, 0], [1, r[1] - r[0], (r[1] - r[0]) ** 2 / 2],
                                  [1, r[2] - r[0], (r[2] - r[0]) ** 2 / 2]]))[1]
    out1 = np.linalg.inv(np.array([[1, 0, 0], [1, r[-2] - r[-1], (r[-2] - r[-1]) ** 2 / 2],
                                   [1, r[-3] - r[-1], (r[-3] - r[-1]) ** 2 / 2]]))[1]

    def inner(c3, f):
        o = torch.zeros_like(f)
        o[1:-1] = c3[1:-1, 0:1] * f[:-2] + c3[1:-1, 1:2] * f[1:-1] + c3[1:-1, 2:3] * f[2:]
        return o

    def bnd_rows(f):  # one-sided first derivatives at the two boundaries
        return one[0] * f[0] + one[1] * f[1] + one[2] * f[2], out1[0] * f[-1] + out1[1] * f[-2] + out1[2] * f[-3]

    def curl(c, second, kind):
        S, dS, T = x[c], x[c + 1], x[c + 2]
        dp = inner(d1, T)
        tr = -(inner(d2, S) if second else inner(d1, dS)) + g3 * S / rt ** 2
        i0, i1 = bnd_rows(T)
        # d2S/dr2 with the slope given at the boundary: 2 (S1 - S0 - h s) / h^2
        sl0 = torch.zeros_like(l)
        sl1 = torch.zeros_like(l)
        if kind == "ins_s":
            sl0, sl1 = (l + 1) / r[0] * S[0], -l / r[-1] * S[-1]
        dd0 = 2.0 * (S[1] - S[0] - h0 * sl0) / h0 ** 2
        dd1 = 2.0 * (S[-2] - S[-1] + h1 * sl1) / h1 ** 2
        if kind == "free_in":  # S extrapolated to zero at r = 0, dT/dr = 2 T / r
            vp = np.linalg.inv(np.array([[1, 0, 0], [1, -r[0], r[0] ** 2 / 2], [1, h0, h0 ** 2 / 2]]))
            vt = np.linalg.inv(np.array([[1, 0, 0], [2, -r[0], 0], [1, h0, h0 ** 2 / 2]]))
            dd0 = vp[2, 0] * S[0] + vp[2, 2] * S[1]
            i0 = vt[1, 0] * T[0]
        if kind == "ins":
            dp[0], dp[-1] = (l + 1) * T[0] / r[0], -l * T[-1] / r[-1]
            tr[0], tr[-1] = 0.0, 0.0
        else:
            dp[0], dp[-1] = i0, i1
            tr[0], tr[-1] = -(dd0 - g3 * S[0] / r[0] ** 2), -(dd1 - g3 * S[-1] / r[-1] ** 2)
        return [T, dp, tr]

    def div(c, own):
        S, dS = x[c], x[c + 1]
        o = inner(d1, S)
        if own:
            o[0], o[-1] = bnd_rows(S)
        else:  # zero fixed field inside, zero fixed flux outside
            o[0] = one[1] * S[1] + one[2] * S[2]
            o[-1] = 0.0
        return (o - dS) * torch.clamp(g3, min=0.5) / rt ** 2

    cols = curl(0, True, "rigid") + curl(6, True, "ins_s") + curl(0, False, "free_in") + curl(3, False, "ins")
    cols += [div(5, False), div(2, True), torch.zeros_like(x[0]), 1.5 * x[9] * rt]
    # Coriolis: closed-form Adams-Gaunt and Elsasser integrals of the degree-1 rotation
    L = cfg.ltr
    ln, mn = _lm(L)
    lookup = {(a, b): i for i, (a, b) in enumerate(zip(ln.tolist(), mn.tolist()))}
    jl = np.array([lookup.get((a - 1, b), -1) for a, b in zip(ln.tolist(), mn.tolist())])
    jh = np.array([lookup.get((a + 1, b), -1) for a, b in zip(ln.tolist(), mn.tolist())])
    jm = np.array([lookup[(a, -b)] for a, b in zip(ln.tolist(), mn.tolist())])
    lf, mf = ln.astype(float), mn.astype(float)
    ok1, ok2 = (ln >= 2) & (jl >= 0), (ln >= 1) & (jh >= 0)
    k1 = np.where(ok1, 4 * np.sqrt(np.maximum(lf ** 2 - mf ** 2, 0)) / ((2 * lf - 1) * (2 * lf + 1)), 0.0)
    k2 = np.where(ok2, 4 * np.sqrt((lf + 1) ** 2 - mf ** 2) / ((2 * lf + 1) * (2 * lf + 3)), 0.0)
    el = np.where(ln >= 1, -4 * mf / (2 * lf + 1), 0.0)
    n3 = np.where(ln == 0, 0.5, lf * (lf + 1))
    n4, n5 = (lf - 1) * lf, (lf + 1) * (lf + 2)
    gg = np.where(ln == 0, 0.0, (2 * lf + 1) / np.maximum(4 * lf * (lf + 1), 1.0))

    def t(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)

    jl, jh, jm = t(np.maximum(jl, 0)), t(np.maximum(jh, 0)), t(jm)
    vS, vd, wS, wd, wT = x[0], x[1], x[3], x[4], x[5]
    w0, w1 = 0.5 * rt ** 2, rt
    pol = (t((2 - n4 - n3) * k1 * gg) * w0 * vd[:, jl] + t((2 - n5 - n3) * k2 * gg) * w0 * vd[:, jh]
           + t(2 * el * gg) * w0 * wS[:, jm] + t(n4 * (2 - n4 + n3) * k1 * gg / 2) * w1 * vS[:, jl]
           + t(n5 * (2 - n5 + n3) * k2 * gg / 2) * w1 * vS[:, jh])
    d2v = t(n3) * vS[:, jm] / rt ** 2 - wT[:, jm]
    tor = (t(-2 * el * gg) * w0 * d2v + t(n3 * el * gg) * vS[:, jm]
           - t((n3 * (2 + n4 - n3) + 2 * (-2 + n4 + n3)) * k1 * gg / 2) * w1 * wS[:, jl]
           - t((n3 * (2 + n5 - n3) + 2 * (-2 + n5 + n3)) * k2 * gg / 2) * w1 * wS[:, jh]
           - t((-2 + n4 + n3) * k1 * gg) * w0 * (wd[:, jl] - 2 / rt * wS[:, jl])
           - t((-2 + n5 + n3) * k2 * gg) * w0 * (wd[:, jh] - 2 / rt * wS[:, jh]))
    cols += [-_COR * pol / rt ** 2, torch.zeros_like(x[0]), -_COR * tor / rt ** 2]
    return torch.stack(cols).reshape(len(cols), -1)


def exact(case, seed):
    gen = torch.Generator(device="cuda").manual_seed(seed)
    kind = case["kind"]
    if kind == "batch":
        cfgs = _batch_cfgs(case)
        ins = [_spectra(c, gen) for c in cfgs]
        return [_exact_cycle(c, d) for c, d in zip(cfgs, ins)]
    cfg = _cfg(case)
    if kind == "post":
        x = _exact_post(cfg, _spectra(cfg, gen, extra=_POST_COLS).reshape(cfg.ncb + _POST_COLS, -1))
        return [x[a - 10:b - 10] for a, b in _POST_OUT]
    if kind == "f_trans":
        g = _grid(cfg, gen).reshape(cfg.ncf, cfg.nph, cfg.nth, cfg.nr)
        ex = _Exact(cfg)
        out = torch.zeros((cfg.ncf, cfg.nr, cfg.J), dtype=torch.float64, device="cuda")

        def fstep(r0, r1):
            out[:, r0:r1] = ex.fwd(g[..., r0:r1].permute(0, 3, 2, 1).contiguous())

        ex.over_radii(fstep)
        return out.reshape(cfg.ncf, -1)
    d = _spectra(cfg, gen)
    if kind == "b_trans":
        ex = _Exact(cfg)
        out = torch.empty((cfg.ncb, cfg.nph, cfg.nth, cfg.nr), dtype=torch.float64, device="cuda")

        def bstep(r0, r1):
            out[..., r0:r1] = ex.bwd(d[:, r0:r1]).permute(0, 3, 2, 1)

        ex.over_radii(bstep)
        return out.reshape(cfg.ncb, -1)
    res = _exact_cycle(cfg, d)
    if case.get("coriolis"):
        # the same curl as the post-processing's last three columns, u and omega in the first six columns
        cor = _exact_post(_post_cfg(cfg), _post_input(cfg, d))[-3:]
        res = [res, cor[::2]]
        return [x.cpu() for x in res] if kind == "host" else res
    return res.cpu() if kind == "host" else res


def _post_cfg(cfg):
    return SphConfig(cfg.ltr, cfg.nth, cfg.nph, cfg.nr)


def _post_input(cfg, d):
    x = torch.zeros((10, cfg.nr, cfg.J), dtype=torch.float64, device=d.device)
    x[:6] = d[:6]
    return x
