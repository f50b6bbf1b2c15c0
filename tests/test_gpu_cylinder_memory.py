"""What a plan keeps on the device after a cylinder call (csrc/multipole.cu): a basis of at most 4 GiB,
however many frames, which are then taken in parts with the same results."""
import dataclasses

import numpy as np
import pytest
import torch

import oracle
from sassena_gb300 import abi

from test_gpu_multipole import case

pytestmark = pytest.mark.gpu


def test_basis_kept_by_a_plan(native_lib):
    w, q = case(130, na=2000, nf=400, nq=20, dsp="square")  # 20 q x 41 orders: 15 MB a frame
    moments = oracle.cylinder_moments(20)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    free = torch.cuda.mem_get_info()[0]
    out = []
    for frames in (slice(0, 400), slice(130, 150)):
        c = np.ascontiguousarray(w.coords[frames])
        with abi.Plan(w.na, len(c), len(w.class_names), "all", "square", precision="fp64") as p:
            p.stage(c)
            p.set_classes(w.atom_class)
            out.append(p.multipole("cylinder", q, w.class_factors, moments, (0.1, 0.2, 1.0))[0])
            if not out[1:]:
                assert free - torch.cuda.mem_get_info()[0] < 5 << 30
    np.testing.assert_allclose(out[0][:, 130:150], out[1], rtol=1e-12)
