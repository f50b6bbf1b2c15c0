"""Fixed-point phase sum of the FP64 form (csrc/phase_fx.cu) against the numpy oracle's amplitudes
(pairwise sums; the C++ oracle adds the atoms one after another, as the reference does, and at
phases near 0 that drift alone exceeds the bound below).

The bound is the oracle's own rounding: its FP64 phase q.r (three products, two sums, each
rounded to at most P = sum_c |q_c| max|r_c|) is off by at most 5 x 2^-53 P, its cos, sin and
sums by a few 2^-53 more, so |A - A_ref| <= sum_j |b_j| (5 x 2^-53 P + 2^-50)."""
import numpy as np
import pytest

from oracle import numpy_oracle
from sassena_gb300 import abi

pytestmark = pytest.mark.gpu


def amplitudes(coords, cls, nclass, sv, shell, cf):
    with abi.Plan(coords.shape[1], coords.shape[0], nclass, precision="fp64") as p:
        p.stage(coords)
        p.set_classes(cls)
        return p.amplitudes(sv, shell, cf), p.schedule()


def check(coords, sv, nclass=3, seed=0):
    rng = np.random.default_rng(seed)
    na = coords.shape[1]
    cls = rng.integers(0, nclass, na).astype(np.int32)
    shell = np.sort(rng.integers(0, 4, len(sv))).astype(np.int32)
    cf = rng.uniform(-10, 10, (4, nclass))
    got, sch = amplitudes(coords, cls, nclass, sv, shell, cf)
    fac = cf[:, cls]
    ref = np.stack([numpy_oracle.amplitude(coords, q, fac[s]) for q, s in zip(sv, shell)])
    P = (np.abs(sv)[:, None, :] * np.abs(coords.astype(np.float64)).max(axis=1)[None]).sum(-1)  # [nv, nf]
    bound = np.abs(fac).sum(axis=1)[shell][:, None] * (5 * 2.0 ** -53 * P + 2.0 ** -50)
    assert (np.abs(got - ref) <= bound).all(), np.max(np.abs(got - ref) / bound)
    assert sch["direct_tiles"] > 0


@pytest.mark.parametrize("na,nf,nv", [(1, 1, 1), (31, 7, 31), (32, 8, 32), (33, 9, 33), (129, 3, 65), (700, 17, 100)])
def test_sizes(native_lib, na, nf, nv):
    rng = np.random.default_rng(na)
    check(rng.uniform(-20, 60, (nf, na, 3)).astype(np.float32), rng.normal(size=(nv, 3)) * 1.5, seed=nv)


@pytest.mark.parametrize("scale", [1e-30, 1e-6, 0.3, 40.0, 3e3, 9e5, 2e6, 1e12])
def test_coordinate_scales(native_lib, scale):
    # below 1, across several binades of the block exponent, and beyond the fixed-point range
    rng = np.random.default_rng(5)
    c = rng.uniform(-1, 1, (4, 150, 3)) * scale * 2.0 ** -rng.integers(0, 30, (4, 150, 3))
    check(c.astype(np.float32), rng.normal(size=(40, 3)) * min(1.0, 1e6 / scale))


@pytest.mark.parametrize("q", [0.0, 1e-300, 1e-9, 3e4, 5e6])
def test_q_scales(native_lib, q):
    rng = np.random.default_rng(6)
    sv = rng.normal(size=(37, 3)) * q
    sv[0] = 0.0
    check(rng.uniform(-1, 1, (5, 90, 3)).astype(np.float32) * np.float32(8.0), sv)


def test_non_finite_frames_stay_apart(native_lib):
    rng = np.random.default_rng(7)
    c = rng.uniform(0, 30, (6, 70, 3)).astype(np.float32)
    sv, cls, shell, cf = rng.normal(size=(33, 3)), np.zeros(70, np.int32), np.zeros(33, np.int32), np.ones((1, 1))
    good, _ = amplitudes(c, cls, 1, sv, shell, cf)
    bad = c.copy()
    bad[2, 40, 1], bad[4, 3, 0] = np.nan, np.inf
    got, _ = amplitudes(bad, cls, 1, sv, shell, cf)
    assert np.isnan(got[:, [2, 4]]).all()
    keep = [0, 1, 3, 5]
    assert (got[:, keep] == good[:, keep]).all()
