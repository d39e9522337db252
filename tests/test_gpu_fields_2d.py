"""Transforms of one 2D field at the sizes with kernels of their own (c2r 64 and 128, r2c 810), FP32.

Against the FP64 oracle with the tolerance of one FP32 transform (test_gpu_sweeps.py),
the mean and the Nyquist modes (of size up to 1) by themselves.
"""

import numpy as np
import pytest
import torch

import oracle as O
import symcode as S
from _util import rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (64, 128, 810))
def test_one_2d_field_to_and_fro(n):
    g, go = S.Grid(2, n, dtype=torch.float32, device="cuda:0"), O.Grid(2, n)
    x = np.random.default_rng(n).standard_normal(go.phys_shape).astype(np.float32).astype(np.float64) + 0.5
    spec = S.to_spec_(S.scalarfield(g), to_dev(x, g), g)
    ref = O.to_spec(x, go)
    assert rel_l2(to_np(spec), ref) < 1e-6
    for k in ((0, 0), (0, n // 2), (n // 2, 0), (n // 2, n // 2)):  # [ky][kx]
        assert abs(complex(to_np(spec)[k]) - ref[k]) < 1e-6
    back = S.to_phys_(S.spacescalarfield(g), to_dev(ref, g), g)
    assert rel_l2(to_np(back), x) < 1e-6
    g.close()
