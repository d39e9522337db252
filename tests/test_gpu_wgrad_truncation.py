"""The tensor cores' truncated sums leave no common factor in the weight gradient.

A network that passes (u + 16) on exactly: centre taps of 1, and where gelu is the
identity in FP32.  The last layer's weight gradient is then sum g u with the same g and
u in the tensor-core network and in the FP32 one on CUDA cores, and their ratio shows
what the sums of the first lose.
"""

import numpy as np
import pytest
import torch

import oracle as O
import symcode as S
from _util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", (64, 128))
def test_the_weight_gradient_keeps_its_size(n):
    dt, nu = 1e-12, 1e-3  # dt: the four stages are at u0 itself
    g, go = S.Grid(3, n, dtype=torch.float32, device="cuda:0"), O.Grid(3, n)
    u = O.random_field(go, seed=48, kpeak=4)
    s = 1 / np.sqrt(sum(float(np.sum(np.abs(c) ** 2)) for c in u))
    u0 = [to_dev(s * c, g) for c in u]
    ws, bs = S.kaiming_cnn_weights(5)
    ws, bs = [w.copy() for w in ws], [np.zeros_like(b) for b in bs]
    for w in ws[:3]:
        w[:] = 0
        for c in range(3):
            w[c, c, 1, 1, 1] = 1.0
    bs[0][:3] = 16.0
    target = S.rollout_record(g, None, [to_dev(c, g) for c in O.random_field(go, seed=49, kpeak=4)], dt, nu, 1)
    args = (4 * go.l / n, nu, g, ws, bs)
    grads = []
    for cl in (S.create_cnn_closure(*args, split=True), S.create_cnn_fp_closure(*args)):
        _, grad = S.rollout_adjoint(g, cl, u0, target, dt, nu, 1, ckpt_every=1)
        grads.append(grad[-(ws[3].size + 6):-6].reshape(6, 32, 27)[:, :3])
        cl.close()
    g.close()
    tc, fp = grads
    # what is given back is within 20 % of what was lost (2.4e-8); FP32 sums rounded to
    # nearest are off by up to 4e-8 on either side
    assert abs(float((tc * fp).sum() / (fp * fp).sum()) - 1) < 6e-8
