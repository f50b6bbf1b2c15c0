"""Multipole amplitudes that are small beside the bounds of both of their factors, which the integer
contractions' digits do not reach (MpRedo in csrc/multipole.cu): against the FP64 oracle at the bar of
1e-12, single moments alone, so that no larger one hides the error."""
import dataclasses

import numpy as np
import pytest

from test_gpu_multipole import case, check

pytestmark = pytest.mark.gpu


def column(seed, na, nf, nq, z0, z1, width):
    """Atoms in a column along z, jittering from frame to frame."""
    w, q = case(seed, na=na, nf=nf, nq=nq)
    rng = np.random.default_rng(seed)
    c = np.empty((nf, na, 3))
    c[:, :, 2] = rng.uniform(z0, z1, na)
    c[:, :, :2] = rng.normal(scale=width, size=(na, 2))
    c += rng.normal(scale=0.05 * width, size=c.shape)
    return dataclasses.replace(w, coords=c.astype(np.float32)), q


@pytest.mark.parametrize("na", [33, 500])
@pytest.mark.parametrize("moment", [(4, 4), (6, -6), (8, 8), (10, 10), (12, -12), (20, 20), (20, 13)])
def test_column_on_the_axis(native_lib, na, moment):
    w, q = column(120, na, 5, 2, 20.0, 100.0, 2.0)
    check(w, q, "sphere", [moment])


@pytest.mark.parametrize("moment", [(6, 6), (12, 12)])
def test_column_through_the_origin(native_lib, moment):
    # near the origin the harmonics are large and the Bessel functions small, far away the reverse
    w, q = column(121, 300, 4, 2, -100.0, 100.0, 0.5)
    check(w, q, "sphere", [moment])


def test_some_frames_and_some_q(native_lib):
    # frames on the axis among frames in the open: only the former are summed again
    w, q = column(122, 70, 6, 3, 20.0, 60.0, 0.3)
    c = w.coords.copy()
    c[1::2, :, 0] += np.random.default_rng(5).uniform(-30, 30, (3, 70)).astype(np.float32)
    w = dataclasses.replace(w, coords=c)
    check(w, q, "sphere", [(9, 9), (9, -8)])
    for f in (0, 1):
        check(dataclasses.replace(w, coords=c[f : f + 1]), q, "sphere", [(9, 9), (9, -8)])


@pytest.mark.parametrize("height", [1e-9, 1e-5, 1e-2])
@pytest.mark.parametrize("moment", [(2, 1), (3, 3)])
def test_sine_moments_of_one_half_plane(native_lib, height, moment):
    w, q = case(123, na=40, nf=4, nq=2)
    rng = np.random.default_rng(9)
    c = rng.uniform(2.0, 14.0, w.coords.shape)
    c[:, :, 1] = height * rng.uniform(0.5, 1.5, c.shape[:2])
    q = q.copy()
    q[:, 0], q[:, 1] = np.abs(q[:, 0]), 0.0
    check(dataclasses.replace(w, coords=c.astype(np.float32)), q, "cylinder", [moment])


@pytest.mark.parametrize("l", [3, 6, 10])
def test_invisible_atoms_hold_the_large_bessel_functions(native_lib, l):
    w, q = case(124, na=64, nf=4, nq=2)
    c = w.coords.copy()
    far = w.atom_class == w.atom_class[0]
    c[:, ~far, :2] *= 0.03
    c[:, far, :2] += 9.0
    cf = w.class_factors.copy()
    cf[:, w.atom_class[0]] = 0.0
    check(dataclasses.replace(w, coords=c, class_factors=cf), q, "cylinder", [(l, 0)])
