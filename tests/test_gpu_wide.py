"""Lines too wide for shared memory.  N = 3072 goes through in halves, every other
length one component pair at a time.  At small truncations the reference is the
CPU oracle; the pruned half lines (N = 3 (L + 1), so L = 1023) are compared with
the separable transforms, whose run-time passes are other code, around products
formed here."""
import numpy as np
import pytest

from kemorin_mhd_b200.config import FIELD_SETS, SphConfig
from kemorin_mhd_b200.synthetic import make_d_rj
from oracle.oracle import Oracle
from tests.gpu_util import col_relerr, from_dev_fortran, to_dev_fortran

TOL = 1e-13  # FP64 tier against the oracle, max-norm per column

FIVE1 = dict(nvb=5, nsb=1, nvf=5, nsf=1,  # a list that no kernel knows, split pairs both ways
             products=((0, 3, 4, 1.0), (0, 2, 4, 1.0), (1, 0, 0, 1.0), (1, 1, 0, 1.0), (0, 0, 1, 1.0), (3, 0, 0, 1.0)))
# at L = 1023 a set holds at most eleven components: lists read at run time, with and without split forward pairs
SQUARE = dict(nvb=3, nsb=1, nvf=3, nsf=1, products=((0, 1, 0, 1.0), (1, 0, 0, 1.0), (1, 2, 0, 1.0), (3, 0, 0, 1.0)))
ODD = dict(nvb=2, nsb=2, nvf=2, nsf=2, products=((0, 1, 0, 0.5), (1, 1, 1, 2.0), (2, 0, 1, 1.0), (3, 0, 1, -1.0)))
SETS = dict(FIELD_SETS, five1=FIVE1, square=SQUARE, odd=ODD)


@pytest.mark.gpu
@pytest.mark.parametrize("fields", ["default", "dynamo", "full", "five1"])
@pytest.mark.parametrize("nph", [3000, 4096])
def test_pair_by_pair(nph, fields):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    cfg = SphConfig(40, 64, nph, 3, **SETS[fields])
    # no line of every pair fits in the 227 KB of shared memory
    assert 16 * ((max(cfg.ncb, cfg.ncf) + 1) // 2) * nph > 227 * 1024
    d = make_d_rj(cfg, seed=51)
    out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
    SphTransform(cfg).nonlinear_cycle(to_dev_fortran(d), out)
    assert col_relerr(from_dev_fortran(out), Oracle(cfg, nthreads=8).cycle(d)).max() <= TOL


def products(cfg, g):
    """Grid products of the configuration's list, components first."""
    import torch
    vec = [g[3 * v:3 * v + 3] for v in range(cfg.nvb)]
    scl = [g[3 * cfg.nvb + s] for s in range(cfg.nsb)]
    vout, sout = [], []
    for kind, a, b, cf in cfg.products:
        if kind == 0:
            x, y = vec[a], vec[b]
            vout.append(cf * torch.stack([x[1] * y[2] - x[2] * y[1], x[2] * y[0] - x[0] * y[2], x[0] * y[1] - x[1] * y[0]]))
        elif kind == 1:
            vout.append(cf * vec[a] * scl[b])
        elif kind == 2:
            sout.append(cf * (vec[a] * vec[b]).sum(0, keepdim=True))
        else:
            sout.append(cf * (scl[a] * scl[b])[None])
    return torch.cat(vout + sout).contiguous()


# the same comparison where the unpruned half lines are pinned to the oracle
# elsewhere (L = 40), and where nothing but the order L + 1 is missing (L = 1022)
@pytest.mark.gpu
@pytest.mark.parametrize("L,fields", [(40, "five1")] + [(L, f) for L in (40, 1022, 1023)
                                                       for f in ("default", "square", "odd")])
def test_half_lines_equal_separable_passes(L, fields):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    cfg = SphConfig(L, 3 * (L + 1) // 2, 3072, 2, **SETS[fields])
    l = np.concatenate([np.arange(abs(k), L + 1) for k in range(-L, L + 1)])
    rng = np.random.default_rng(52)
    d = rng.standard_normal((cfg.ncb, cfg.nr, cfg.J)) * (l + 1.0) ** -2
    d[:3 * cfg.nvb, :, l == 0] = 0.0
    d = torch.from_numpy(d.reshape(cfg.ncb, -1)).cuda()
    tr = SphTransform(cfg, radius=np.array([0.7, 1.1]))
    out = torch.zeros((cfg.ncf, cfg.J * cfg.nr), dtype=torch.float64, device="cuda")
    fld = torch.empty((cfg.ncb, cfg.nr * cfg.nth * cfg.nph), dtype=torch.float64, device="cuda")
    tr.nonlinear_cycle(d, out)
    tr.sph_b_trans(d, fld)
    frc = products(cfg, fld)
    torch.cuda.synchronize()
    ref = torch.zeros_like(out)
    tr.sph_f_trans(frc, ref)
    tr.close()
    err = col_relerr(from_dev_fortran(out), from_dev_fortran(ref))
    assert err.max() <= TOL, err
