"""The one-pass BF16 network has the same input in the adjoint as in the forward evaluation.

Another transform of the same state, as exact but rounded otherwise, tips BF16
roundings of the input.  A field that does not depend on y shows it: where the
evaluation gives every x row of a plane the same values, a first layer that takes
differences along y sees zeros, and any difference that the adjoint's own transform
made would be magnified 2^14 times.
"""

import numpy as np
import pytest
import torch

import oracle as O
import symcode as S
from _util import to_dev

pytestmark = pytest.mark.gpu


def test_the_adjoint_sees_the_input_of_the_evaluation():
    n, dt, nu = 128, 1e-12, 1e-3  # dt: the four stages are at u0 itself
    g, go = S.Grid(3, n, dtype=torch.float32, device="cuda:0"), O.Grid(3, n)
    u = O.random_field(go, seed=46, kpeak=4)
    for c in u:
        c[:, 1:, :] = 0  # [kz][ky][kx]: ky = 0 only
    s = 1 / np.sqrt(sum(float(np.sum(np.abs(c) ** 2)) for c in u))
    u0 = [to_dev(s * c, g) for c in u]
    ws, bs = S.kaiming_cnn_weights(5)
    ws = [w.copy() for w in ws]
    bs = [np.zeros_like(b) for b in bs]
    ws[0][:] = 0
    for c in range(3):
        ws[0][c, c, 1, 1, 1], ws[0][c, c, 1, 2, 1] = 2.0 ** 14, -(2.0 ** 14)
        bs[0][c] = 1.0
    cl = S.create_cnn_closure(4 * go.l / n, nu, g, ws, bs, mu=5.0, sigma=2.0)
    # one difference would lift a layer-1 activation from 0.84 to tens; the sums of equal
    # terms in another order, which the rows of the later layers do differ by, are far below
    tau = cl(u0, None)  # [6][z][y][x]
    if (tau - tau[:, :, :1]).abs().max() > 0.05 * tau.abs().max():
        cl.close()
        g.close()
        pytest.skip("the evaluation itself tells the rows apart")
    target = S.rollout_record(g, None, [to_dev(c, g) for c in O.random_field(go, seed=47, kpeak=4)], dt, nu, 1)
    _, grad = S.rollout_adjoint(g, cl, u0, target, dt, nu, 1, ckpt_every=1)
    # channels 0 to 2 of the second layer's input are the constant a = BF16(gelu(1)), so each
    # of their 27 taps has the gradient a sum g, and sum g is the bias gradient
    sizes = [(w.size, b.size) for w, b in zip(ws, bs)]
    o = sum(sizes[0])
    gw1 = grad[: sizes[0][0]].reshape(ws[0].shape)
    gw2 = grad[o: o + sizes[1][0]].reshape(32, 32, 27)
    gb2 = grad[o + sizes[1][0]: o + sum(sizes[1])]
    a = float(torch.nn.functional.gelu(torch.tensor(1.0), approximate="tanh").bfloat16())
    # FP32 sums of at most a few hundred terms (16 accumulations in tensor memory) before FP64:
    # 1e-5 of sum |g|, which is about sqrt(n^3) = 1448 times the size of the first layer's
    # gradient, sum g u with u of unit size and random signs
    scale = np.abs(gw1[:3, :3]).max()
    assert scale > 0
    assert np.abs(gw2[:, :3] - a * gb2[:, None, None]).max() < 1.5e-2 * scale
    cl.close()
    g.close()
