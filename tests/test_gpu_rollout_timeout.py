"""The bounded waits of the tensor-core network's training kernels, made to run out on purpose.

With the plan option SC_OPT_WAIT_LIMIT = 0 the convolutions (the fused launch of a
split-precision layer included) and the weight-gradient kernel give up at their
first wait, free their tensor memory and return (test_gpu_cnn_timeout.py has the
plain evaluation).  What they leave out is missing from states, loss and gradient,
so a rollout has to say so.
"""

import numpy as np
import pytest
import torch

import oracle as O
import symcode as S
from symcode import _lib as L
from _util import to_dev

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("split", (True, False))
def test_a_rollout_reports_a_wait_that_ran_out(split):
    n, dt, nu, steps = 64, 5e-3, 1e-3, 2
    g, go = S.Grid(3, n, dtype=torch.float32, device="cuda:0"), O.Grid(3, n)
    u0 = [to_dev(c, g) for c in O.random_field(go, seed=45, kpeak=4)]
    ws, bs = S.kaiming_cnn_weights(5)

    def closure():
        return S.create_cnn_closure(4 * go.l / n, nu, g, ws, bs, mu=5.0, sigma=2.0, split=split)

    target = S.rollout_record(g, None, u0, dt, nu, steps)
    cl = closure()
    loss, grad = S.rollout_adjoint(g, cl, u0, target, dt, nu, steps, ckpt_every=1)
    cl.close()

    S.set_option(g, L.SC_OPT_WAIT_LIMIT, 0)
    job = dict(grid=g, u0=u0, traj=target, dt=dt, visc=nu, nsteps=steps, ckpt_every=1)
    for call in (lambda c: S.rollout_adjoint(g, c, u0, target, dt, nu, steps, ckpt_every=1),
                 lambda c: S.rollout_adjoint_batch([dict(closure=c, **job)]),
                 lambda c: S.rollout_loss(g, c, u0, target, dt, nu, steps),
                 lambda c: S.rollout_record(g, c, u0, dt, nu, steps)):
        cl = closure()
        with pytest.raises(S.SymcodeError) as err:
            call(cl)
        assert err.value.status == L.SC_ERR_TIMEOUT
        torch.cuda.synchronize()  # the kernels returned: no hang, no fault
        cl.close()

    # back to the default bound: a fresh closure gives what it gave before (sums
    # over blocks are FP64 atomics: their order is free and may tip an FP32 rounding)
    S.set_option(g, L.SC_OPT_WAIT_LIMIT, -1)
    cl = closure()
    loss2, grad2 = S.rollout_adjoint(g, cl, u0, target, dt, nu, steps, ckpt_every=1)
    assert abs(loss2 - loss) <= 1e-9 * loss
    assert np.linalg.norm(grad2 - grad) <= 1e-8 * np.linalg.norm(grad)
    cl.close()
    g.close()
