"""Record layout and longitudinal FFT variants at the sizes where they can go
wrong: truncations that do not fill the eight-order blocks of the rtm records,
odd component counts (a half pair at the end of a record), composite FFT radices
(every one of them, first, middle and last), the short, staged, in-place and
half line kernels, and radial blocks of the separable transforms that end inside
a block.  Reference: the CPU FP64 oracle; bounds as in the FP64 tier's tests."""
import numpy as np
import pytest

from kemorin_mhd_b200.config import FIELD_SETS, SphConfig
from kemorin_mhd_b200.synthetic import make_d_rj
from oracle.oracle import Oracle
from tests.gpu_util import col_relerr, from_dev_fortran, to_dev_fortran

TOL = 1e-13  # FP64 tier against the oracle, max-norm per column

HEAT = dict(nvb=1, nsb=1, nvf=1, nsf=0, products=((1, 0, 0, 1.0),))
ODD = dict(nvb=2, nsb=2, nvf=2, nsf=2,  # 8 + 8 components, a list no kernel knows
           products=((0, 1, 0, 0.5), (1, 1, 1, 2.0), (2, 0, 1, 1.0), (3, 0, 1, -1.0)))
ONE2 = dict(nvb=1, nsb=2, nvf=1, nsf=1, products=((1, 0, 1, 0.5), (3, 0, 1, 2.0)))  # components paired in order
FIVE = dict(nvb=5, nsb=0, nvf=5, nsf=0,
            products=tuple((0, a, (a + 1) % 5, 1.0) for a in range(5)))


def run(kind, cfg, tier=0, **kw):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    tr = SphTransform(cfg, tier=tier, **kw)
    orc = Oracle(cfg, nthreads=8)
    n = cfg.J * cfg.nr
    if kind == "cycle":
        d = make_d_rj(cfg, seed=21)
        out = torch.zeros((cfg.ncf, n), dtype=torch.float64, device="cuda")
        tr.nonlinear_cycle(to_dev_fortran(d), out)
        ref = orc.cycle(d)
    elif kind == "b_trans":
        d = make_d_rj(cfg, seed=22)
        out = torch.empty((cfg.ncb, cfg.nr * cfg.nth * cfg.nph), dtype=torch.float64, device="cuda")
        tr.sph_b_trans(to_dev_fortran(d), out)
        ref = orc.b_trans(d)
    else:
        rng = np.random.default_rng(23)
        f = np.asfortranarray(rng.standard_normal((cfg.nr * cfg.nth * cfg.nph, cfg.ncf)))
        out = torch.zeros((cfg.ncf, n), dtype=torch.float64, device="cuda")
        tr.sph_f_trans(to_dev_fortran(f), out)
        ref = orc.f_trans(f)
    return col_relerr(from_dev_fortran(out), ref).max()


# truncation: block edges of eight orders; longitudes: every radix of the run-time
# passes (90 = 10 9, 108 = 12 9, 128 = 16 8, 162 = 9 6 3, 400 = 10 8 5, 450 = 10 9 5,
# 750 = 10 15 5, 20 = 5 4 or 10 2, 40 = 8 5)
LINES = [(3, 6, 8), (7, 12, 16), (8, 13, 20), (9, 15, 40), (15, 24, 90), (16, 26, 108), (23, 36, 128), (24, 37, 162),
         (30, 48, 96), (39, 60, 400), (41, 64, 450), (47, 72, 750)]


@pytest.mark.gpu
@pytest.mark.parametrize("fields", ["default", "heat", "dynamo", "odd", "one2"])
@pytest.mark.parametrize("L,nth,nph", LINES)
def test_cycle_lines(L, nth, nph, fields):
    sets = dict(FIELD_SETS, heat=HEAT, odd=ODD, one2=ONE2)
    assert run("cycle", SphConfig(L, nth, nph, 3, **sets[fields])) <= TOL


# short lines of the specialised kernels: an odd count, pruned and unpruned
@pytest.mark.gpu
@pytest.mark.parametrize("L,nph", [(31, 96), (30, 96), (63, 192), (50, 192), (127, 384), (100, 384)])
def test_cycle_specialised_odd_set(L, nph):
    assert run("cycle", SphConfig(L, 3 * (L + 1) // 2, nph, 3, nvb=2, nsb=1, nvf=2, nsf=1,
                                  products=((0, 1, 0, 1.0), (1, 0, 0, 1.0), (2, 0, 1, 1.0)))) <= TOL


# lines whose grid alone fits (in place), with sets of their own and without, and
# unpruned half lines (3072); lines that go pair by pair: test_gpu_wide.py
@pytest.mark.gpu
@pytest.mark.parametrize("L,nph,fields", [(L, nph, f) for L, nph in ((40, 1536), (511, 1536), (60, 1440), (40, 3072))
                                          for f in ("dynamo", "full", "five", "odd", "heat", "one2")
                                          if L != 511 or f not in ("odd", "heat", "one2")])  # those are staged
def test_cycle_long_lines(L, nph, fields):
    sets = dict(FIELD_SETS, odd=ODD, five=FIVE, heat=HEAT, one2=ONE2)
    nth = 64 if L < 100 else 96
    assert run("cycle", SphConfig(L, nth, nph, 3, **sets[fields])) <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("nr", [1, 2, 3, 4, 5, 7, 8, 9, 17])
def test_separable_radial_blocks(nr):
    # with one or two radii the synthetic profile vanishes: values from the grid instead
    cfg = SphConfig(23, 37, 90, nr, **FIELD_SETS["dynamo"])
    radius = 0.6 + 0.1 * np.arange(nr)
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    tr, orc = SphTransform(cfg, radius=radius), Oracle(cfg, nthreads=4, radius=radius)
    rng = np.random.default_rng(nr)
    d = np.asfortranarray(rng.standard_normal((cfg.J * nr, cfg.ncb)))
    d[0:1, :] = 0.0
    fld = torch.empty((cfg.ncb, nr * cfg.nth * cfg.nph), dtype=torch.float64, device="cuda")
    tr.sph_b_trans(to_dev_fortran(d), fld)
    assert col_relerr(from_dev_fortran(fld), orc.b_trans(d)).max() <= TOL
    f = np.asfortranarray(rng.standard_normal((nr * cfg.nth * cfg.nph, cfg.ncf)))
    out = torch.zeros((cfg.ncf, cfg.J * nr), dtype=torch.float64, device="cuda")
    tr.sph_f_trans(to_dev_fortran(f), out)
    assert col_relerr(from_dev_fortran(out), orc.f_trans(f)).max() <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("kind", ["b_trans", "f_trans"])
@pytest.mark.parametrize("fields", ["default", "heat", "one2"])
@pytest.mark.parametrize("L,nth,nph,nr", [(31, 48, 96, 9), (20, 32, 3072, 5), (20, 32, 1536, 6), (20, 33, 450, 8)])
def test_separable_lines(kind, L, nth, nph, nr, fields):
    sets = dict(FIELD_SETS, heat=HEAT, one2=ONE2)
    assert run(kind, SphConfig(L, nth, nph, nr, **sets[fields])) <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("fields", ["default", "convection"])
@pytest.mark.parametrize("back", [0, 1, 2])
def test_noalloc_smaller_record_blocks(fields, back):
    """L + 1 = 33 orders pad to 40 in blocks of eight: the largest shells that the
    static work area takes (and the next smaller ones) need smaller blocks, down to
    one order, where an odd component count leaves the sectors on 16 bytes."""
    import ctypes
    import torch
    from kemorin_mhd_b200 import sph_trans as st
    conv = dict(nvb=2, nsb=1, nvf=2, nsf=1, products=((0, 1, 0, 1.0), (1, 0, 0, 1.0), (2, 0, 1, 1.0)))
    lib = st.load_library()

    def call(nr):
        cfg = SphConfig(32, 50, 108, nr, **(conv if fields == "convection" else {}))
        d = make_d_rj(cfg, seed=6)
        n = cfg.J * cfg.nr
        out = torch.zeros((cfg.ncf, n), dtype=torch.float64, device="cuda")
        src = to_dev_fortran(d)
        r = np.ascontiguousarray(cfg.radius())
        prods = (st.Product * len(cfg.products))(*[st.Product(*q) for q in cfg.products])
        de = st.Desc()
        de.ltr, de.nth, de.nph, de.nr = cfg.ltr, cfg.nth, cfg.nph, cfg.nr
        de.radius = r.ctypes.data_as(ctypes.POINTER(ctypes.c_double))
        de.nvector_b, de.nscalar_b, de.nvector_f, de.nscalar_f = cfg.nvb, cfg.nsb, cfg.nvf, cfg.nsf
        de.nproduct, de.products = len(cfg.products), prods
        cb, cf = st._i32(cfg.cols_b()), st._i32(cfg.cols_f())
        torch.cuda.synchronize()
        rc = lib.kmhd_sph_cycle_noalloc(ctypes.byref(de), src.data_ptr(), n, cb, out.data_ptr(), n, cf, None)
        return rc, cfg, d, out

    nr = 80
    while call(nr)[0] == 2:  # KMHD_ERR_SIZE
        nr -= 1
    # with one order per block the work area holds what it always held
    assert nr == {"default": 46, "convection": 66}[fields]
    rc, cfg, d, out = call(nr - back)
    assert rc == 0
    assert col_relerr(from_dev_fortran(out), Oracle(cfg, nthreads=8).cycle(d)).max() <= TOL


@pytest.mark.gpu
@pytest.mark.parametrize("L,nr,fields", [(130, 21, f) for f in ("heat", "convection", "default", "dynamo", "full", "five",
                                                                "one2")] + [(160, 33, "default"), (255, 9, "default")])
def test_fp64_sixteen_row_kernels(L, nr, fields):
    """The FP64 Legendre kernels of large launches: truncations that end inside
    their 16- and 64-degree blocks, latitudes inside a block of 16 (odd: an equator
    row), odd radial block counts, every field group."""
    conv = dict(nvb=2, nsb=1, nvf=2, nsf=1, products=((0, 1, 0, 1.0), (1, 0, 0, 1.0), (2, 0, 1, 1.0)))
    sets = dict(FIELD_SETS, heat=HEAT, convection=conv, five=FIVE, one2=ONE2)
    assert run("cycle", SphConfig(L, 3 * (L + 1) // 2 + 1, 3 * (L + 1) if L == 255 else 480, nr, **sets[fields])) <= TOL


# 17 components back, the most a set can have: the same line kernels as with 16,
# so a scalar that no product uses changes no bit; against the oracle with it used
@pytest.mark.gpu
@pytest.mark.parametrize("L,nph", [(300, 1536), (40, 3072)])  # in place, half lines
def test_seventeen_components(L, nph):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    prods = tuple((0, a, (a + 1) % 5, 1.0) for a in range(5)) + ((2, 0, 1, 1.0),)
    res = []
    for nsb in (1, 2):
        cfg = SphConfig(L, 64, nph, 3, nvb=5, nsb=nsb, nvf=5, nsf=1, products=prods)
        d = make_d_rj(SphConfig(L, 64, nph, 3, nvb=5, nsb=2, nvf=5, nsf=1, products=prods), seed=24)[:, :cfg.ncb]
        out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
        SphTransform(cfg).nonlinear_cycle(to_dev_fortran(np.asfortranarray(d)), out)
        res.append(out)
    assert torch.equal(res[0], res[1])
    used = dict(nvb=5, nsb=2, nvf=4, nsf=2, products=((0, 0, 4, 1.0), (0, 1, 2, 1.0), (1, 3, 1, 1.0), (1, 4, 0, 1.0),
                                                       (2, 0, 3, 1.0), (3, 0, 1, 1.0)))
    assert run("cycle", SphConfig(L, 64, nph, 3, **used)) <= TOL
