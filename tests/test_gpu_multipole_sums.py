"""The sphere's integer contraction and its basis (csrc/multipole.cu) against the FP64 oracle, where
they can go wrong: atoms that do not fill a lane or a tile, more sums than one round of the
integers holds, q-vectors over several CTAs, groups of one to eight pairs, moments of negative m
alone or given twice, and rows of tiny values. Bar 1e-12, as for every FP64 path
(max_t |S - S_ref| / |S_ref(q, 0)|)."""
import dataclasses

import numpy as np
import pytest

import oracle
from sassena_gb300 import abi

from test_gpu_multipole import case, check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("na,nf,nq", [(1, 3, 1), (31, 4, 2), (33, 5, 10), (255, 2, 11), (257, 2, 21), (20000, 2, 3)])
def test_atoms_and_q(native_lib, na, nf, nq):
    w, q = case(70 + nq, na=na, nf=nf, nq=nq, box=2.0 * na ** (1.0 / 3.0) + 2.0)
    check(w, q, "sphere", oracle.sphere_moments(9 if na < 1000 else 3))


@pytest.mark.parametrize("count", [1, 2, 3, 4, 5, 6, 7, 8, 9, 17])
def test_pairs_of_one_l(native_lib, count):
    w, q = case(81, na=100, nf=4, nq=2)
    check(w, q, "sphere", [(17, m if m % 2 else -m) for m in range(count)])


def test_negative_m_and_repeated_moments(native_lib):
    w, q = case(82, na=50, nf=5, nq=3)
    check(w, q, "sphere", [(5, -3), (5, -4), (2, -1)])
    with abi.Plan(w.na, w.nf, len(w.class_names), precision="fp64") as p:
        p.stage(w.coords)
        p.set_classes(w.atom_class)
        once = p.multipole("sphere", q, w.class_factors, [(4, 2), (3, -1)])
        twice = p.multipole("sphere", q, w.class_factors, [(4, 2), (3, -1), (4, 2), (3, -1)])
    for a, b in zip(once, twice):
        np.testing.assert_allclose(b, 2 * a, rtol=1e-14)


@pytest.mark.parametrize("scale", [1e-4, 1e-2, 0.3, 3.0, 60.0])
@pytest.mark.parametrize("moments", [[(9, 4), (9, -9)], [(40, 0), (40, 39)], [(0, 0), (1, 1)]])
def test_scales_of_the_bessel_rows(native_lib, scale, moments):
    # arguments from the power series through Miller's recurrence to the upward one; tiny rows alone
    w, q = case(83, na=64, nf=4, nq=2)
    c = (w.coords - 6.0) * np.float32(scale)
    if scale ** moments[0][0] < 1e-60:
        return  # the correlation of amplitudes below 1e-154 underflows in FP64
    check(dataclasses.replace(w, coords=c), q, "sphere", moments)


def test_atom_at_the_origin_and_not_finite(native_lib):
    w, q = case(84, na=40, nf=6, nq=2)
    c = w.coords.copy()
    c[:, 7] = 0.0
    check(dataclasses.replace(w, coords=c), q, "sphere", oracle.sphere_moments(4))
    c[3, 5, 2] = np.nan
    with abi.Plan(w.na, w.nf, len(w.class_names), precision="fp64") as p:
        p.stage(c)
        p.set_classes(w.atom_class)
        assert all(np.isnan(a).all() for a in p.multipole("sphere", q, w.class_factors, oracle.sphere_moments(4)))
