"""A NaN or an infinity among the spectra in the INT8-sliced tiers.  A column of
operands (one order, radius and field) is scaled by its largest finite entry, and
what is not finite has no digits: it counts as zero and leaves the other modes
of its column as they were."""
import numpy as np
import pytest

from kemorin_mhd_b200.config import SphConfig, TIER_FP32ACC, TIER_SPLIT_I8
from kemorin_mhd_b200.synthetic import make_d_rj
from tests.gpu_util import to_dev_fortran


@pytest.mark.gpu
@pytest.mark.parametrize("tier", [TIER_SPLIT_I8, TIER_FP32ACC], ids=["split", "fp32acc"])
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf])
@pytest.mark.parametrize("col", [0, 1, 2, 9])  # the radial column of u, its two vector columns, T
def test_counts_as_zero(tier, value, col):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    cfg = SphConfig(31, 48, 96, 5)
    d = make_d_rj(cfg, seed=91)
    lm = [(b, a) for a in range(-cfg.ltr, cfg.ltr + 1) for b in range(abs(a), cfg.ltr + 1)]
    row = cfg.J + lm.index((6, 3))  # radius 1
    tr, res = SphTransform(cfg, tier=tier), []
    for v in (0.0, value):
        d[row, col] = v
        fld = torch.empty((cfg.ncb, cfg.nr * cfg.nth * cfg.nph), dtype=torch.float64, device="cuda")
        tr.sph_b_trans(to_dev_fortran(d), fld)
        res.append(fld)
    assert float(res[0].abs().max()) > 0.0
    assert torch.equal(res[0], res[1])
