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


AXIS = (0.2, -1.0, 0.4)


@pytest.mark.parametrize("na,nf,nq", [(1, 3, 1), (31, 4, 2), (33, 5, 5), (255, 2, 6), (257, 2, 13), (20000, 2, 3)])
def test_cylinder_atoms_and_q(native_lib, na, nf, nq):
    w, q = case(90 + nq, na=na, nf=nf, nq=nq, box=2.0 * na ** (1.0 / 3.0) + 2.0)
    check(w, q, "cylinder", oracle.cylinder_moments(9 if na < 1000 else 3), AXIS)


@pytest.mark.parametrize("count", [1, 2, 3, 5, 8, 9, 17])
def test_cylinder_orders(native_lib, count):
    w, q = case(91, na=100, nf=4, nq=2)
    moments = [(1 + k // 2, 2 * (k % 2) + (k % 3 == 0)) for k in range(count)]
    check(w, q, "cylinder", moments + moments[:1], AXIS)


def angle(x, y):
    """The reference's azimuth: its float pi where x < 0 (CylinderCoor3D, coor3d.cpp:116-141)."""
    phi = np.arctan(y / x) + np.where(x < 0, np.where(y < 0, -1.0, 1.0) * np.float64(np.float32(np.pi)), 0.0)
    return np.where(phi < 0, phi + 2 * np.pi, phi)


def cylinder_reference(w, coords, q, moments, axis):
    """F(q, t) from scipy's Bessel functions (the oracle's are 3e-12 off for n = 80 just below x = n)."""
    from scipy.special import jv
    ez = np.asarray(axis) / np.linalg.norm(axis)
    er = np.cross([0.0, 0.0, 1.0], ez)
    er /= np.linalg.norm(er)
    base = np.array([er, np.cross(ez, er), ez])
    c = np.einsum("kx,tjx->ktj", base, coords.astype(np.float64))
    r = np.hypot(c[0], c[1]).astype(np.float32).astype(np.float64)
    phi = angle(c[0], c[1]).astype(np.float32).astype(np.float64)
    z = c[2].astype(np.float32).astype(np.float64)
    out = []
    for k in range(len(q)):
        qx, qy, qz = base @ q[k]
        x = w.factors()[k] * np.exp(1j * np.abs(z * qz))
        series = []
        for l, m in moments:
            n = 2 * l if m < 2 else 2 * l - 1
            t = (np.cos if m in (0, 2) else np.sin)(n * (phi - angle(qx, qy)))
            f = 1.0 if l == 0 else np.sqrt(2.0) * ((-1) ** l if m < 2 else 1j * (-1) ** (l - 1))
            a = np.sqrt(2 * np.pi) * f * (x * jv(n, np.hypot(qx, qy) * r) * t).sum(axis=1)
            series.append([np.mean(np.conj(a[: w.nf - tau]) * a[tau:]) for tau in range(w.nf)])
        out.append(np.sum(series, axis=0) / (2 * np.pi))
    return np.array(out)


@pytest.mark.parametrize("scale", [1e-4, 1e-2, 0.3, 3.0, 8.0, 60.0])
@pytest.mark.parametrize("moments", [[(4, 0), (5, 3)], [(40, 0), (40, 2)], [(0, 0), (1, 2)]])
def test_cylinder_scales(native_lib, scale, moments):
    # arguments below, around and above Hankel's range and the orders; tiny rows alone
    w, q = case(92, na=64, nf=4, nq=2)
    c = (w.coords - 6.0) * np.float32(scale)
    if scale ** (2 * moments[0][0]) < 1e-60:
        return  # the correlation of amplitudes below 1e-154 underflows in FP64
    ref = cylinder_reference(w, c, q, moments, AXIS)
    with abi.Plan(w.na, w.nf, len(w.class_names), precision="fp64") as p:
        p.stage(c)
        p.set_classes(w.atom_class)
        fqt, fq, fq2 = p.multipole("cylinder", q, w.class_factors, moments, AXIS)
    assert (np.abs(fqt - ref).max(axis=1) <= 1e-12 * np.abs(ref[:, 0])).all()
    assert (np.abs(fq - ref.mean(axis=1)) <= 1e-12 * np.abs(fq)).all()
