"""The result at a radius does not depend on how the shell is cut.  The FP64
Legendre launchers choose between an 8-row and a 16-row kernel by the size of
the launch, which a radial window (host-pointer chunks), a slab of a parallel
run or a shell of a few radii changes; both sides of each choice must agree bit
for bit.  The sizes lie on both sides of the thresholds for two SMs' and one SM's
worth of CTAs at 148 SMs."""
import numpy as np
import pytest

from kemorin_mhd_b200.config import FIELD_SETS, SphConfig, TIER_FP64, TIER_SPLIT_I8
from kemorin_mhd_b200.synthetic import make_d_rj
from tests.gpu_util import from_dev_fortran, to_dev_fortran

CONV = dict(nvb=2, nsb=1, nvf=2, nsf=1, products=((0, 1, 0, 1.0), (1, 0, 0, 1.0), (2, 0, 1, 1.0)))


def cycle(cfg, d, tier, radius=None):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
    tr = SphTransform(cfg, tier=tier, radius=radius)
    tr.nonlinear_cycle(to_dev_fortran(d), out)
    tr.close()
    return from_dev_fortran(out)


@pytest.mark.gpu
@pytest.mark.parametrize("fields", ["default", "dynamo", "full", "convection"])
def test_few_radii_equal_the_shell(fields):
    sets = dict(FIELD_SETS, convection=CONV)
    # 65 radii: 16-row kernels both ways; 4 radii: 256 backward and 128 forward CTAs, 8-row kernels
    cfg, few = (SphConfig(127, 192, 384, nr, **sets[fields]) for nr in (65, 4))
    d, r = make_d_rj(cfg, seed=71), cfg.radius()
    n = cfg.J * few.nr
    whole = cycle(cfg, d, TIER_FP64)
    assert np.array_equal(cycle(few, np.asfortranarray(d[:n]), TIER_FP64, radius=r[:few.nr].copy()), whole[:n])


@pytest.mark.gpu
@pytest.mark.parametrize("L,nr,tier", [(63, 129, TIER_FP64),         # 1088 CTAs backward, chunks of 128
                                       (255, 129, TIER_SPLIT_I8)],  # dipole orders forward: 198 CTAs, chunks of 24
                         ids=["fp64", "split_dipole"])
def test_host_chunks_equal_device_call(L, nr, tier):
    from kemorin_mhd_b200.sph_trans import SphTransform
    cfg = SphConfig(L, 3 * (L + 1) // 2, 3 * (L + 1), nr)
    d = make_d_rj(cfg, seed=72)
    ref = cycle(cfg, d, tier)
    tr = SphTransform(cfg, tier=tier)
    h_out = np.full((cfg.J * nr, cfg.ncf), np.nan, order="F")
    tr.nonlinear_cycle(np.asfortranarray(d), h_out)
    assert tr.last_timing()["fft_nl"] == 0.0  # chunked: no stage times
    tr.close()
    assert np.array_equal(h_out, ref)


@pytest.mark.gpu
@pytest.mark.parametrize("nr,world", [(33, 2), (65, 3)])  # 320 and 576 CTAs, slabs of 192
def test_slabs_equal_the_shell(nr, world):
    from kemorin_mhd_b200.slabs import radial_slab
    cfg = SphConfig(63, 96, 192, nr)
    d, r, J = make_d_rj(cfg, seed=73), cfg.radius(), cfg.J
    whole = cycle(cfg, d, TIER_FP64)
    for rank in range(world):
        s = radial_slab(nr, world, rank)
        got = cycle(SphConfig(63, 96, 192, s.nr_local), np.asfortranarray(d[s.lo * J:s.hi * J]), TIER_FP64,
                    radius=r[s.lo:s.hi].copy())
        a = (s.r0 - s.lo) * J
        assert np.array_equal(got[a:a + (s.r1 - s.r0) * J], whole[s.r0 * J:s.r1 * J]), rank
