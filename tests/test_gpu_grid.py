"""Gridded phase sum of the FP32 form (csrc/phase_grid.cu) against the oracle, at the edges of its
tiles: directions left over (32, 16 x 2 and 8 x 4 lanes), frames, atom slices, shells per pass,
factors that weight the atoms and factors that are applied per class.

Bar: a phase is off by at most 3 x 2^-24 q r (FP32 products and sums of u.r; q r <= 70 here) and the
weights and the grid's unit add 2e-6, so an amplitude is off by at most 1.5e-5 of sum |b|; at
random phases that is 1.5e-5 of |A|, and S(q, t) = <A* A> / S(q, 0) at most twice that: 3e-5."""
import dataclasses

import numpy as np
import pytest

import oracle
from sassena_gb300 import abi, synth

from helpers import rel_err_sqt

pytestmark = pytest.mark.gpu

BAR = 3e-5


def case(na, nf, nq, nm, seed, shells="random", factors="constant", nclass=4):
    w = synth.small("all", "square", seed=seed, na=na, nf=nf, nq=nq, nm=nm, box=24.0)
    rng = np.random.default_rng(seed)
    q = np.linspace(0.2, 2.5, nq) if shells == "linear" else np.sort(rng.uniform(0.1, 2.5, nq))
    b = np.array([6.6, -3.7, 9.4, 5.8])[:nclass]
    if factors == "wide":
        b = np.array([25.3, 0.09, 2.0, 0.3])[:nclass]
    cf = np.tile(b, (nq, 1))
    if factors == "varying":
        cf = cf * (1.0 + 0.1 * np.arange(nq))[:, None]
    cls = np.minimum(w.atom_class, nclass - 1)
    return dataclasses.replace(w, shells=q, class_factors=cf, atom_class=cls, class_names=w.class_names[:nclass])


def check(w, gridded=True, **kw):
    sch = {}
    got = abi.compute_workload(w, "fp32", schedule=sch, **kw)
    if gridded:
        assert sch["rec_tiles"] > 0 and sch["rec_shells"] == w.nq and sch["rec_shells_per_lane"] == 0
    ref = oracle.all_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), {"autocorrelate": 0, "square": 1,
                             "plain": 2}[w.dsp], 0, nthreads=8)
    assert rel_err_sqt(got[0], ref[0]).max() <= BAR
    return sch


@pytest.mark.parametrize("nm", [1, 8, 9, 16, 24, 25, 32, 33, 47])
def test_direction_remainders(native_lib, nm):
    check(case(600, 5, 20, nm, nm), gridded=nm >= 4)  # one direction would leave 7 of 8 lanes idle


@pytest.mark.parametrize("nf", [1, 7, 8, 9, 33])
def test_frames(native_lib, nf):
    check(case(520, nf, 18, 13, 100 + nf))


@pytest.mark.parametrize("na", [512, 1025, 4096, 4097, 9001])
@pytest.mark.parametrize("factors", ["constant", "varying", "wide"])
def test_slices_and_factors(native_lib, na, factors):
    check(case(na, 3, 24, 20, na, factors=factors))


@pytest.mark.parametrize("nq", [9, 16, 17, 64])
def test_shell_passes(native_lib, nq):
    check(case(700, 4, nq, 40, nq))


def test_linear_scan_and_slices_of_a_batch(native_lib):
    check(case(3000, 4, 60, 40, 7, shells="linear"))
    ws = [dataclasses.replace(case(na, nf, nq, nm, na), dsp="square") for na, nf, nq, nm in
          ((700, 6, 20, 33), (5000, 3, 30, 10), (60, 5, 12, 9))]
    with abi.Batch(ws, precision="fp32") as b:
        b.run()
        b.sync()
        for i, w in enumerate(ws):
            ref = oracle.all_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), 1, 0, nthreads=8)
            assert rel_err_sqt(b.results(i)[0], ref[0]).max() <= BAR


def test_clustered_atoms_do_not_overflow(native_lib):
    # every atom within a thousandth of one place: the largest sum that a grid point can take
    w = case(4096, 2, 20, 16, 3, nclass=1)
    c = np.full_like(w.coords, 3.0) + np.random.default_rng(1).uniform(-1e-3, 1e-3, w.coords.shape).astype(np.float32)
    c[:, 0] = -9.0  # the extent of an ordinary box
    c[:, 1] = 15.0
    check(dataclasses.replace(w, coords=c))


def test_non_finite_coordinates_take_the_other_kernels(native_lib):
    w = case(600, 6, 20, 16, 11)
    c = w.coords.copy()
    c[3, 17, 1] = np.inf
    got = abi.compute_workload(dataclasses.replace(w, coords=c), "fp32")[0]
    ref = abi.compute_workload(w, "fp32")[0]
    assert np.isnan(got[:, 3]).all()
    keep = [0, 1, 2, 4, 5]
    assert (np.abs(got[:, keep] - ref[:, keep]) <= 2 * BAR * np.abs(ref).max()).all()


@pytest.mark.parametrize("na", [9001, 20000])
@pytest.mark.parametrize("factors", ["constant", "varying", "wide"])
def test_long_slices(native_lib, na, factors):
    # one slice asked for: one grid up to 16,384 atoms, then several, one after the other
    w = case(na, 3, 18, 20, 77, factors=factors)
    with abi.Plan(w.na, w.nf, len(w.class_names), "all", "square", precision="fp32") as p:
        p.stage(w.coords)
        p.set_classes(w.atom_class)
        p.set_tile(0, 0, 0, 1)
        got = p.compute(w.sub_offsets(), w.subvectors(), w.class_factors)
        assert p.schedule()["rec_tiles"] > 0 and p.schedule()["atom_splits"] == 1
    ref = oracle.all_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), 1, 0, nthreads=8)
    assert rel_err_sqt(got[0], ref[0]).max() <= BAR
