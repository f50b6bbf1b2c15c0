"""When the gridded phase sum is chosen for systems of several classes (choose_grid, csrc/engine.cu): each
class is padded to 32 atoms, and factors that vary with q have a grid for each. The kernel that the
schedule names, the memory of the class-sorted copy, and the results at the bar of test_gpu_grid."""
import dataclasses

import numpy as np
import pytest
import torch

import oracle
from sassena_gb300 import abi

from helpers import cplx, rel_err_sqt
from test_gpu_grid import BAR, case

pytestmark = pytest.mark.gpu


def system(na, nf, nq, nm, nclass, shells="linear", factors="constant", seed=5, qmax=2.5):
    w = case(na, nf, nq, nm, seed, shells=shells)
    rng = np.random.default_rng(seed)
    q = np.linspace(0.2, qmax, nq) if shells == "linear" else w.shells
    cf = np.tile(rng.uniform(2.0, 9.0, nclass), (nq, 1))
    if factors == "varying":
        cf = cf * (1.0 + 0.05 * np.arange(nq))[:, None]
    cls = rng.permutation(np.arange(na) % nclass).astype(np.int32)
    return dataclasses.replace(w, shells=q, class_factors=cf, atom_class=cls, class_names=[str(i) for i in range(nclass)])


def kernel(sch):
    if sch["rec_tiles"] == 0:
        return "direct"
    return "recurrence" if sch["rec_shells_per_lane"] else "gridded"


def reference(w):
    return oracle.all_vectors(w.coords, w.sub_offsets(), w.subvectors(), w.factors(), 1, 0, nthreads=8)[0]


@pytest.mark.parametrize("na,nclass,nq,shells,factors,want", [
    (600, 5, 20, "linear", "constant", "gridded"),
    (600, 5, 20, "linear", "varying", "recurrence"),
    (600, 5, 20, "random", "constant", "gridded"),
    (600, 20, 20, "random", "varying", "direct"),
    (4000, 40, 20, "random", "constant", "gridded"),
    (4000, 40, 5, "random", "varying", "direct"),
    (600, 600, 20, "random", "constant", "direct"),  # one atom a class: 32 slots for each
    (600, 600, 20, "linear", "varying", "direct"),
])
def test_choice(native_lib, na, nclass, nq, shells, factors, want):
    w = system(na, 6, nq, 32, nclass, shells, factors)
    sch = {}
    got = abi.compute_workload(w, "fp32", schedule=sch)
    assert kernel(sch) == want
    assert rel_err_sqt(got[0], reference(w)).max() <= BAR


@pytest.mark.parametrize("device", [False, True])
def test_factors_of_each_call(native_lib, device):
    # one plan, factors that are alike at all shells and that are not, in turn
    ws = [system(600, 6, 20, 32, 5, factors=f) for f in ("constant", "varying", "constant")]
    with abi.Plan(600, 6, 5, "all", "square", precision="fp32") as p:
        p.stage(ws[0].coords)
        p.set_classes(ws[0].atom_class)
        for w, want in zip(ws, ("gridded", "recurrence", "gridded")):
            if device:
                sv = torch.from_numpy(np.ascontiguousarray(w.subvectors())).cuda()
                cf = torch.from_numpy(np.ascontiguousarray(w.class_factors)).cuda()
                out = [torch.zeros(n, dtype=torch.float64, device="cuda") for n in ((20, 6, 2), (20, 2), (20, 2))]
                torch.cuda.synchronize()
                p.compute_device(w.sub_offsets(), sv.data_ptr(), cf.data_ptr(), *[o.data_ptr() for o in out])
                got = out[0].cpu().numpy()
                got = got[..., 0] + 1j * got[..., 1]
            else:
                got = p.compute(w.sub_offsets(), w.subvectors(), w.class_factors)[0]
            if not device:  # read on the device: the kernel stays the one that the first factors chose
                assert kernel(p.schedule()) == want
            assert rel_err_sqt(got, reference(w)).max() <= BAR


@pytest.mark.parametrize("shells", ["random", "linear"])
def test_no_memory_for_the_sorted_copy(native_lib, shells):
    # the copy is as large as the staged frames; where it finds no memory the direct kernel needs none
    w = system(2000, 8, 16, 32, 2, shells)
    nf = 16384
    rng = np.random.default_rng(1)
    coords = np.tile(w.coords, (nf // 8, 1, 1)) + rng.normal(scale=0.01, size=(1, 2000, 3)).astype(np.float32)
    with abi.Plan(2000, nf, 2, "all", "square", precision="fp32") as p:
        p.stage(coords)
        p.set_classes(w.atom_class)
        p.set_recurrence(-1)
        args = w.sub_offsets(), w.subvectors(), w.class_factors
        ref = p.compute(*args)[0]
        torch.cuda.empty_cache()
        hold = torch.empty(torch.cuda.mem_get_info()[0] - (300 << 20), dtype=torch.uint8, device="cuda")
        try:
            p.set_recurrence(0)
            got = p.compute(*args)[0]
            assert kernel(p.schedule()) == "direct"
        finally:
            del hold
            torch.cuda.empty_cache()
        assert (got == ref).all()


def test_one_large_factor(native_lib):
    # One atom of 16 among 4,000 of 1. A weight is rounded to 9e-7 of the largest factor of its grid: by
    # class, an amplitude is off by 1.35e-6 of its norm (and by 1e-6 for FP32's phases), of which S(q) takes
    # 2 / sqrt(2) / sqrt(20 directions) = 5.3e-7 rms; in one grid the former is up to 16 times that.
    w = system(4001, 20, 18, 20, 2, "random")
    cls = np.zeros(w.na, dtype=np.int32)
    cls[77] = 1
    w = dataclasses.replace(w, atom_class=cls, class_factors=np.tile([1.0, 16.0], (w.nq, 1)))
    sch = {}
    got = abi.compute_workload(w, "fp32", schedule=sch)[0]
    assert kernel(sch) == "gridded"
    ref = cplx(reference(w))
    assert np.sqrt(np.mean(np.abs(got / ref - 1) ** 2)) <= 1e-6
