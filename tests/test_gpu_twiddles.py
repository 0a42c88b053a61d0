"""Twiddle factors of the run-time FFT passes.  A scalar whose radius m - 1 holds
the sectoral mode (m, m) alone is A cos(m phi) on every latitude circle: one
frequency goes through the passes as a product of twiddles, so the grid shows
their error and little else.  With u = 2^-53, in units of A u and as the root mean
square over frequencies and points: 0.64 .. 0.79 with every twiddle read from the
table, 0.76 .. 0.85 with at most three running products between table values and
1.01 .. 1.07 with seven (a numpy restatement of the passes, without fused
multiply-adds: 0.7 .. 0.9, 1.0 .. 1.1 and 1.6 .. 1.8)."""
import numpy as np
import pytest

from kemorin_mhd_b200.config import SphConfig
from tests.gpu_util import from_dev_fortran, to_dev_fortran


@pytest.mark.gpu
@pytest.mark.parametrize("N", [384, 450, 768])
def test_one_frequency(N):
    import torch
    from kemorin_mhd_b200.sph_trans import SphTransform
    L = N // 3 - 1
    cfg = SphConfig(L, 8, N, L, nvb=1, nsb=1, nvf=1, nsf=0, products=((1, 0, 0, 1.0),))
    d = np.zeros((cfg.J * cfg.nr, cfg.ncb), order="F")
    m_of = np.concatenate([np.full(L - abs(k) + 1, k) for k in range(-L, L + 1)])
    l_of = np.concatenate([np.arange(abs(k), L + 1) for k in range(-L, L + 1)])
    for m in range(1, L + 1):
        j = np.flatnonzero((m_of == m) & (l_of == m))[0]
        d[(m - 1) * cfg.J + j, 3] = 1.0
    fld = torch.empty((cfg.ncb, cfg.nr * cfg.nth * cfg.nph), dtype=torch.float64, device="cuda")
    tr = SphTransform(cfg, radius=1.0 + np.arange(L) / L)
    tr.sph_b_trans(to_dev_fortran(d), fld)
    # (phi, r) at the latitude next to the equator; m = r + 1
    f = from_dev_fortran(fld)[:, 3].reshape(N, cfg.nth, L)[:, 4].astype(np.longdouble)
    k = np.outer(np.arange(N), np.arange(1, L + 1)) % N
    c = np.cos(2 * np.longdouble("3.14159265358979323846264338327950288") * k / N)
    amp = 2 * (f * c).mean(axis=0)
    err = (f / amp - c).astype(float)
    rms = np.sqrt((err ** 2).mean()) * 2.0 ** 53
    assert rms < 0.95
