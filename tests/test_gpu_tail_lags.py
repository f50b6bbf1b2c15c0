"""The last lags of the FP32 coherent autocorrelation, summed directly from 128 frames on, against
the FP64 oracle. Bar per lag: phases of at most 60 rad in FP32 (3.6e-6) on both factors of a
product, so 1e-5 of S(q, 0), whatever the number of frames."""
import dataclasses

import numpy as np
import pytest

import oracle
from sassena_gb300 import abi, synth

from helpers import cplx

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("nf,nm", [(127, 3), (128, 1), (129, 40), (700, 7), (300, 1100)])
def test_last_lags(native_lib, nf, nm):
    w = synth.small("all", "autocorrelate", seed=nf, na=40, nf=nf, nq=2, nm=nm)
    for method in ("fftw", "direct"):
        got = abi.compute_workload(w, "fp32", method=method)[0]
        ref = cplx(oracle.all_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), 0, method == "direct",
                                      nthreads=8)[0])
        assert (np.abs(got - ref)[:, -16:].max(axis=1) <= 1e-5 * np.abs(ref[:, 0])).all()


def test_a_frame_that_is_not_finite(native_lib):
    w = synth.small("all", "autocorrelate", seed=1, na=40, nf=200, nq=2, nm=5)
    c = w.coords.copy()
    c[100, 3, 1] = np.nan  # in no product of the last lags
    assert all(np.isnan(a).all() for a in abi.compute_workload(dataclasses.replace(w, coords=c), "fp32"))
