"""The last eight lags of a coherent autocorrelation from 128 frames on, against the sums of products of
the library's own amplitudes: the phases' rounding is on both sides, so that the bars hold the products'
alone, which the transforms' (times NF / (NF - tau)) does not meet."""
import numpy as np
import pytest

import oracle
from sassena_gb300 import abi, synth

from test_gpu_multipole import case, check

pytestmark = pytest.mark.gpu


def products(w, precision, method):
    """S(q, t) and its last eight lags summed in FP64 from the amplitudes."""
    shell = np.repeat(np.arange(w.nq, dtype=np.int32), w.nm)
    with abi.Plan(w.na, w.nf, len(w.class_names), "all", "autocorrelate", method, precision) as p:
        p.stage(w.coords)
        p.set_classes(w.atom_class)
        p.set_recurrence(-1)  # the direct kernel, as the amplitudes' own call
        got = p.compute(w.sub_offsets(), w.subvectors(), w.class_factors)[0]
        A = p.amplitudes(w.subvectors(), shell, w.class_factors).reshape(w.nq, w.nm, w.nf)
    lags = []
    for n in range(8, 0, -1):  # n products a series
        x = np.conj(A[:, :, :n]) * A[:, :, w.nf - n:]
        lags.append((np.conj(x) if method == "direct" else x).sum(axis=2).mean(axis=1) / n)
    return got, np.stack(lags, axis=1)


# FP64: a product is off by 4 x 2^-53 of |A|^2 and the sum of n <= 8 of them over NM series by 12 x 2^-53 more
# at the most; FP32: a product and the sum of n by 10 x 2^-24 at the most, 2 x 2^-24 in the mean of its
# signs.
@pytest.mark.parametrize("precision,bar", [("fp64", 2e-15), ("fp32", 1.2e-7)])
@pytest.mark.parametrize("method", ["fftw", "direct"])
@pytest.mark.parametrize("nf,nm", [(128, 1), (129, 40), (250, 60), (700, 7), (300, 1100)])
def test_last_lags(native_lib, nf, nm, method, precision, bar):
    w = synth.small("all", "autocorrelate", seed=nf, na=40, nf=nf, nq=2, nm=nm)
    got, lags = products(w, precision, method)
    assert (np.abs(got[:, -8:] - lags).max(axis=1) <= bar * np.abs(got[:, 0])).all()


@pytest.mark.parametrize("kind", ["sphere", "cylinder"])
@pytest.mark.parametrize("method", ["fftw", "direct"])
def test_last_lags_of_multipole_amplitudes(native_lib, kind, method):
    w, q = case(7, na=30, nf=150, nq=2)
    moments = oracle.sphere_moments(4) if kind == "sphere" else oracle.cylinder_moments(4)
    check(w, q, kind, moments, method=method)
