"""What shares a complex FFT shares its rounding error.  With an odd number of
vectors the first scalar goes with theta of the last vector, not with its much
larger r (forward: unless the scalar is a dot product, as large as r): where
theta is zero the scalar must come out the same, bit for bit, whatever r is --
and the other way round -- in every line kernel."""
import numpy as np
import pytest

from kemorin_mhd_b200.config import FIELD_SETS, SphConfig, TIER_FP64, TIER_SPLIT_I8
from kemorin_mhd_b200.synthetic import make_d_rj
from tests.gpu_util import from_dev_fortran, to_dev_fortran

HEAT = dict(nvb=1, nsb=1, nvf=1, nsf=1, products=((1, 0, 0, 1.0), (3, 0, 0, 1.0)))
FIVE1 = dict(nvb=5, nsb=1, nvf=5, nsf=1,  # the last vector in the first two products only
             products=((0, 3, 4, 1.0), (0, 2, 4, 1.0), (1, 0, 0, 1.0), (1, 1, 0, 1.0), (0, 0, 1, 1.0), (3, 0, 0, 1.0)))
SETS = dict(FIELD_SETS, heat=HEAT, five1=FIVE1)


def transform(cfg, tier=TIER_FP64):
    from kemorin_mhd_b200.sph_trans import SphTransform
    return SphTransform(cfg, tier=tier)


def radial_last_vector(cfg, scale):
    """Spectra whose last vector has a radial component alone, times scale."""
    d = make_d_rj(cfg, seed=81)
    v = 3 * (cfg.nvb - 1)
    d[:, v] *= scale
    d[:, v + 1:v + 3] = 0.0
    return d


# separable kernels: the run-time passes at any length
@pytest.mark.gpu
@pytest.mark.parametrize("tier", [TIER_FP64, TIER_SPLIT_I8], ids=["fp64", "split"])
@pytest.mark.parametrize("fields", ["default", "heat", "five1"])
def test_backward_scalar_apart_from_r(fields, tier):
    import torch
    cfg = SphConfig(31, 48, 96, 9, **SETS[fields])
    tr, res = transform(cfg, tier), []
    for scale in (0.0, 1e3):
        fld = torch.empty((cfg.ncb, cfg.nr * cfg.nth * cfg.nph), dtype=torch.float64, device="cuda")
        tr.sph_b_trans(to_dev_fortran(radial_last_vector(cfg, scale)), fld)
        res.append(fld)
    assert torch.equal(res[0][3 * cfg.nvb], res[1][3 * cfg.nvb])
    assert float(res[1][3 * cfg.nvb].abs().max()) > 0.0


@pytest.mark.gpu
@pytest.mark.parametrize("fields", ["heat", "five1"])
def test_forward_scalar_apart_from_r(fields):
    import torch
    cfg = SphConfig(31, 48, 96, 9, **SETS[fields])
    v, s = 3 * (cfg.nvf - 1), 3 * cfg.nvf
    f = np.random.default_rng(82).standard_normal((cfg.nr * cfg.nth * cfg.nph, cfg.ncf))
    f[:, v + 1:v + 3] = 0.0
    tr = transform(cfg)

    def run(r, sc):
        g = np.asfortranarray(f)
        g[:, v] *= r
        g[:, s] *= sc
        out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
        tr.sph_f_trans(to_dev_fortran(g), out)
        return from_dev_fortran(out)

    a, b, c = run(1.0, 1.0), run(1.0, 1e4), run(0.0, 1.0)
    assert np.array_equal(a[:, v], b[:, v])
    assert np.array_equal(a[:, s], c[:, s])


# the cycle kernels: staged pruned and unpruned, run-time radices staged, half
# lines, pair by pair, and in place with run-time field counts
@pytest.mark.gpu
@pytest.mark.parametrize("L,nph,fields", [(31, 96, "default"), (30, 96, "default"), (127, 384, "default"),
                                          (40, 1536, "default"), (20, 90, "default"), (40, 3072, "default"),
                                          (40, 3000, "default"), (40, 1536, "five1"), (40, 3072, "five1"),
                                          (60, 1440, "five1")])
def test_cycle_scalar_apart_from_r(L, nph, fields):
    import torch
    cfg = SphConfig(L, 3 * (L + 1) // 2, nph, 3, **SETS[fields])
    tr, res = transform(cfg), []
    for scale in (0.0, 1e3):
        out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
        tr.nonlinear_cycle(to_dev_fortran(radial_last_vector(cfg, scale)), out)
        res.append(from_dev_fortran(out))
    # the products without the last vector know nothing of its rounding error
    free = list(range(6, 10)) if fields == "default" else list(range(6, 16))
    assert np.abs(res[1][:, free]).max(axis=0).min() > 0.0
    assert np.array_equal(res[0][:, free], res[1][:, free])


@pytest.mark.gpu
@pytest.mark.parametrize("L,nph", [(31, 96), (40, 1536), (20, 90), (40, 3072)])
def test_cycle_forward_r_apart_from_scalar(L, nph):
    """u s1 and s0 s1: u has r alone, so u s1's poloidal column knows nothing of s0."""
    import torch
    cfg = SphConfig(L, 3 * (L + 1) // 2, nph, 3, nvb=1, nsb=2, nvf=1, nsf=1,
                    products=((1, 0, 1, 0.5), (3, 0, 1, 2.0)))
    tr, res = transform(cfg), []
    for scale in (1.0, 1e4):
        d = radial_last_vector(cfg, 1.0)
        d[:, 3] *= scale
        out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
        tr.nonlinear_cycle(to_dev_fortran(d), out)
        res.append(from_dev_fortran(out)[:, 0])
    assert np.array_equal(res[0], res[1])
