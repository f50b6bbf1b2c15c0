"""Fixed-point incoherent autocorrelation of the FP64 form (csrc/corr_fx.cu) against the oracle: every
padded length it takes, directions that do not fill a warp's series, chunks that end inside an
atom, and the largest sums its integers hold. Bar 1e-12, as for every FP64 path
(max_t |S - S_ref| / |S_ref(q, 0)|)."""
import dataclasses

import numpy as np
import pytest

import oracle
from sassena_gb300 import abi, synth

from helpers import cplx, rel_err_sqt, rel_err_vec

pytestmark = pytest.mark.gpu


def check(w, method="fftw"):
    got = abi.compute_workload(w, "fp64", method=method)
    ref = oracle.self_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), 0, method == "direct", nthreads=8)
    assert rel_err_sqt(got[0], ref[0]).max() <= 1e-12
    assert max(rel_err_vec(got[1], cplx(ref[1])), rel_err_vec(got[2], cplx(ref[2]))) <= 1e-12


@pytest.mark.parametrize("nf", [17, 31, 32, 33, 64, 65, 100, 127, 128])
@pytest.mark.parametrize("na,nm", [(1, 1), (5, 3), (23, 17)])
def test_lengths_and_remainders(native_lib, nf, na, nm):
    check(synth.small("self", "autocorrelate", seed=nf + na, na=na, nf=nf, nq=2, nm=nm))


def test_many_pairs_and_direct_method(native_lib):
    # about as many (atom, direction) pairs per warp as fit several folds, and one left over
    check(synth.small("self", "autocorrelate", seed=1, na=301, nf=128, nq=3, nm=33))
    check(synth.small("self", "autocorrelate", seed=2, na=40, nf=60, nq=400, nm=3), method="direct")


@pytest.mark.parametrize("nf", [32, 64, 128])
def test_still_atoms_fill_the_integers(native_lib, nf):
    # every term of a series is the same: |X| = NF at one bin; at the origin exactly 1
    w = synth.small("self", "autocorrelate", seed=3, na=12, nf=nf, nq=2, nm=5)
    c = np.repeat(w.coords[:1], nf, axis=0)
    c[:, :4] = 0.0
    check(dataclasses.replace(w, coords=c))


@pytest.mark.parametrize("scale", [1e-20, 1e-3, 100.0, 2e6])
def test_coordinate_scales(native_lib, scale):
    # subnormal offsets, residuals below the 32-bit grid, and beyond the fixed-point range (FP64 path)
    w = synth.small("self", "autocorrelate", seed=4, na=9, nf=50, nq=2, nm=4)
    c = (w.coords - 6.0) * np.float32(scale)
    check(dataclasses.replace(w, coords=c, shells=w.shells * min(1.0, 10.0 / scale)))


def test_non_finite_coordinates(native_lib):
    w = synth.small("self", "autocorrelate", seed=5, na=9, nf=50, nq=2, nm=4)
    c = w.coords.copy()
    c[7, 3, 1] = np.nan
    assert all(np.isnan(a).all() for a in abi.compute_workload(dataclasses.replace(w, coords=c), "fp64"))


def test_batch_of_one_length(native_lib):
    ws = [synth.small("self", "autocorrelate", seed=60 + i, na=na, nf=nf, nq=nq, nm=nm)
          for i, (na, nf, nq, nm) in enumerate([(15, 70, 5, 33), (61, 128, 3, 8), (40, 66, 2, 7)])]
    with abi.Batch(ws, precision="fp64") as b:
        b.run()
        b.sync()
        for i, w in enumerate(ws):
            ref = oracle.self_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), 0, 0, nthreads=8)
            assert rel_err_sqt(b.results(i)[0], ref[0]).max() <= 1e-12
