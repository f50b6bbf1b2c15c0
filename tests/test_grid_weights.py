"""The gridded phase sum's weights (csrc/phase_grid.cu): sum_n c_n(z) exp(i l (o_n - z)) is the same
D(l) for every z to the errors that the kernel's comment states, every weight is positive and
below the peak that the integer grid's unit assumes."""
import os
import re

import numpy as np
import pytest

SRC = os.path.join(os.path.dirname(__file__), "..", "sassena_gb300", "csrc", "phase_grid.cu")


def weights():
    src = open(SRC).read()
    body = src[src.index("constexpr float grid_coef("):]
    body = body[:body.index("return w[set]")]
    v = [float(x) for x in re.findall(r"-?\d\.\d+e[-+]\d+", body)]
    peak = float(re.search(r"kGridPeak = ([0-9.]+)f", src).group(1))
    return np.array(v, dtype=np.float32).astype(np.float64).reshape(2, 3, 6), peak


@pytest.mark.parametrize("s,sigma,rms,most", [(0, 3.0, 5.6e-7, 4.6e-6), (1, 4.0, 7.0e-8, 6.0e-7)])
def test_alias_error(s, sigma, rms, most):
    w, peak = weights()
    z = np.linspace(-0.5, 0.5, 401)
    half = np.stack([np.polynomial.polynomial.polyval(z, c) for c in w[s]], axis=1)
    c = np.concatenate([half, half[::-1, ::-1]], axis=1)  # c_{5-n}(z) = c_n(-z)
    assert c.min() > 0 and c.max() < peak
    lam = np.linspace(0, np.pi / sigma, 300)
    o = np.arange(6) - 2.5
    e = np.einsum("zn,zln->zl", c, np.exp(1j * lam[None, :, None] * (o[None, None] - z[:, None, None])))
    r = np.abs(e / e.real.mean(axis=0) - 1)
    assert np.sqrt((r ** 2).mean()) < rms and r.max() < most
