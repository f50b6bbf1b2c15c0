"""The unit of the gridded phase sum's integer cells (grid_tables_kernel, csrc/phase_grid.cu), for every
largest factor: no cell overflows, and a weight's rounding and what six of them leave in an amplitude stay
within the bounds that the kernel's comment states."""
import math
import re

import numpy as np
import pytest

from test_grid_weights import SRC, weights


def scale(bmax, slice_atoms, peak, total, single):
    most = min(total / (peak * slice_atoms), single / peak)
    return 2.0 ** (math.frexp(most / bmax)[1] - 1)


def rule():
    m = re.search(r"fmin\(([0-9.e]+) / \(kGridPeak \* s\.slice_atoms\), ([0-9.e]+) / kGridPeak\)", open(SRC).read())
    return float(m.group(1)), float(m.group(2))


@pytest.mark.parametrize("atoms,half,rms", [(4096, 1.1e-6, 2.1e-6), (16384, 4.4e-6, 8.4e-6)])
def test_unit(atoms, half, rms):
    w, peak = weights()
    total, single = rule()
    bmax = np.exp(np.linspace(math.log(1e-6), math.log(1e6), 3001))
    s = np.array([scale(b, atoms, peak, total, single) for b in bmax])
    assert (s * bmax * peak * atoms < 2**31).all()  # every atom on one grid point
    assert (s * bmax * peak < 2**22).all()  # the magic number's mantissa
    assert (0.5 / (s * bmax)).max() <= half
    # six independent roundings, divided by D at the largest shell of the coarser set
    z = np.linspace(-0.5, 0.5, 401)
    c = np.stack([np.polynomial.polynomial.polyval(z, k) for k in w[0]], axis=1)
    c = np.concatenate([c, c[::-1, ::-1]], axis=1)
    D = (c * np.cos(np.pi / 3 * (np.arange(6) - 2.5 - z[:, None]))).sum(axis=1).mean()
    assert math.sqrt(6 / 12) * (1 / (s * bmax)).max() / D <= rms
    assert (1 / s[np.argmin(abs(bmax - 1))]) * math.sqrt(6 / 12) == pytest.approx({4096: 1.35e-6, 16384: 5.4e-6}[atoms], rel=0.01)
