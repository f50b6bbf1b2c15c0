"""Memory of a batch whose systems are cut into slices of atoms: the partial amplitudes of all of its
systems together stay within 4 GiB (prepare_full, csrc/engine.cu)."""
import numpy as np
import pytest
import torch

from sassena_gb300 import abi

from helpers import rel_err_sqt
from test_gpu_grid import BAR, case, check

pytestmark = pytest.mark.gpu


def test_partials_of_a_batch(native_lib):
    # 80 systems of 65,536 sub-vectors x 64 frames: 34 MB of amplitudes each, and as much again for
    # each of two slices of 4,200 atoms
    w = case(4200, 64, 64, 1024, 21)
    nsys, amplitudes = 80, 80 * 64 * 1024 * 64 * 8
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    with abi.Batch([w] * nsys, precision="fp32") as b:
        b.run()
        b.sync()
        used = free - torch.cuda.mem_get_info()[0]
        first, last = b.results(0)[0], b.results(nsys - 1)[0]
        assert b.schedule()["rec_shells"] == nsys * w.nq
    assert used < amplitudes + (4 << 30) + (1 << 30)
    assert rel_err_sqt(first, abi.compute_workload(w, "fp32")[0]).max() <= BAR
    assert rel_err_sqt(last, first).max() <= BAR


@pytest.mark.parametrize("factors", ["constant", "varying"])
def test_a_system_alone_keeps_its_slices(native_lib, factors):
    sch = check(case(9001, 3, 18, 20, 22, factors=factors))
    assert sch["atom_splits"] > 1
