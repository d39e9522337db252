"""The filter's reduced grids: one DNS plan filtered to LES grids that need different ones.

160 -> 64 forms the DNS products on 128 points and 160 -> 32 on 120 (96 -> 36 and
96 -> 20: 80 and 72).  Tolerances as in test_gpu_filter.py: tau against the size of
the products it cancels.
"""

import math

import numpy as np
import pytest
import torch

import oracle as O
import symcode as S
from _util import rel_l2, to_dev, to_np

pytestmark = pytest.mark.gpu

DTYPES = (torch.float32, torch.float64)


def _check(u, od, ol, d, ub, tau, tol):
    rb, rt = O.sfs(u, od, ol, d)
    assert rel_l2([to_np(c) for c in ub], rb) < tol
    s1 = [O.twothirds(O.gaussianfilter(O.cutoff(c, od, ol), d, ol), ol) for c in O.nonlinearity(u, od)]
    scale = math.sqrt(sum(float(np.sum(np.abs(c) ** 2)) for c in s1))
    assert math.sqrt(sum(float(np.sum(np.abs(to_np(x) - y) ** 2)) for x, y in zip(tau, rt))) < tol * scale


@pytest.mark.parametrize("n,m,other", ((160, 64, 32), (160, 32, 64), (96, 36, 20)))
@pytest.mark.parametrize("dtype", DTYPES)
def test_a_captured_filter_keeps_its_grid(n, m, other, dtype):
    """A call for another LES grid between capture and replay changes nothing."""
    tol = 1e-12 if dtype == torch.float64 else 1e-5
    gd, gl, go = (S.Grid(3, k, dtype=dtype, device="cuda:0") for k in (n, m, other))
    od, ol, oo = O.Grid(3, n), O.Grid(3, m), O.Grid(3, other)
    u = O.random_field(od, seed=6, kpeak=4)
    ud = [to_dev(c, gd) for c in u]
    d, do = 2 * ol.l / m, 2 * oo.l / other
    ub, tau = S.vectorfield(gl), S.tensorfield(gl)
    S.sfs_(ub, tau, ud, gd, gl, d)  # from here on the reduced grid is there for a capture
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        S.sfs_(ub, tau, ud, gd, gl, d)
    ub2, tau2 = S.vectorfield(go), S.tensorfield(go)
    S.sfs_(ub2, tau2, ud, gd, go, do)
    for c in (*ub, *tau):
        c.zero_()
    graph.replay()
    _check(u, od, ol, d, ub, tau, tol)
    _check(u, od, oo, do, ub2, tau2, tol)


def test_the_first_call_does_not_wait_for_the_stream():
    """A stream-ordered call returns while the work queued before it still runs, the
    first one for an LES grid too (about a second of queued work)."""
    n = 160
    out, keep = [], []  # a plan that went away meanwhile would wait for the device
    for busy in (False, True):  # the first round loads the kernels
        gd = S.Grid(3, n, dtype=torch.float32, device="cuda:0")
        u = [to_dev(c, gd) for c in O.random_field(O.Grid(3, n), seed=7, kpeak=4)]
        gls = [S.Grid(3, m, dtype=torch.float32, device="cuda:0") for m in (64, 32)]
        ubs, taus = [S.vectorfield(g) for g in gls], [S.tensorfield(g) for g in gls]
        keep.append((gd, gls))
        torch.cuda.synchronize()
        queued = torch.cuda.Event()
        if busy:
            torch.cuda._sleep(2_000_000_000)
        queued.record()
        for g, ub, tau in zip(gls, ubs, taus):
            S.sfs_(ub, tau, u, gd, g, 2 * g.spacing)
        assert not busy or not queued.query()
        torch.cuda.synchronize()
        out.append([c.clone() for f in (*ubs, *taus) for c in f])
    assert all(torch.equal(a, b) for a, b in zip(*out))
