"""The warp-per-row-pair x sweeps at every size they have, against the oracles.

Every size is 2^a 3^b 5^c with its own split into lanes and points per lane, so
each has its own remainders: lanes left over in a warp, work items left over in
a round, the block of modes that straddles the 2/3 cut.  2D grids run the 2D
product sweep, the plain transforms in the full layout and the CFL maximum; 3D
grids run the 3D product sweep on a sparse field that reaches the cube's faces
and corners, against exact triad sums.

Tolerances (as in test_gpu_solver.py): FP64 1e-12 relative L2; FP32 1e-5 for a
right-hand side and 1e-6 for one transform (a length-N transform in FP32 is off
by about 6e-8 sqrt(log2 N^D) <= 3e-7).
"""

import math

import numpy as np
import pytest
import torch

import oracle as O
import symcode as S
from _util import rel_l2, to_dev, to_np
from oracle import triad as T
from test_gpu_les import KINDS, _models

pytestmark = pytest.mark.gpu

SIZES = (32, 36, 40, 48, 60, 64, 72, 80, 90, 96, 120, 128, 160, 180, 192, 240, 256, 270, 320, 360, 384, 512, 540, 640,
         720, 768, 810, 1024)
DTYPES = (torch.float32, torch.float64)


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", SIZES)
def test_2d_sweeps_match_the_oracle(n, dtype):
    g, go = S.Grid(2, n, dtype=dtype, device="cuda:0"), O.Grid(2, n, 2 * math.pi)
    tol, ftol = (1e-12, 1e-12) if dtype == torch.float64 else (1e-5, 1e-6)
    u = O.random_field(go, 3, kpeak=5.0)
    du = S.convectiondiffusion_(S.vectorfield(g), [to_dev(c, g) for c in u], g, 1e-3)
    ref = [O.twothirds(c, go) for c in O.convectiondiffusion(u, go, 1e-3)]
    assert rel_l2([to_np(c) for c in du], ref) < tol
    dt = S.propose_timestep([to_dev(c, g) for c in u], g, 1e-6)
    assert abs(dt / O.propose_timestep(u, go, 1e-6) - 1) < ftol
    x = np.random.default_rng(n).standard_normal(go.phys_shape)
    xd = to_dev(x, g)
    spec = S.to_spec_(S.scalarfield(g), xd, g)
    assert rel_l2(to_np(spec), O.to_spec(to_np(xd), go)) < ftol
    back = S.to_phys_(S.spacescalarfield(g), spec, g)
    assert rel_l2(to_np(back), to_np(xd)) < ftol


@pytest.mark.parametrize("n", (32, 48, 90, 128))
@pytest.mark.parametrize("dtype", DTYPES)
def test_3d_transforms_match_pocketfft(n, dtype):
    """One field in 3D: the last warp's pencils are partly empty."""
    g, go = S.Grid(3, n, dtype=dtype, device="cuda:0"), O.Grid(3, n, 2 * math.pi)
    tol = 1e-12 if dtype == torch.float64 else 1e-6
    xd = to_dev(np.random.default_rng(n).standard_normal(go.phys_shape), g)
    spec = S.to_spec_(S.scalarfield(g), xd, g)
    assert rel_l2(to_np(spec), O.to_spec(to_np(xd), go)) < tol
    assert rel_l2(to_np(S.to_phys_(S.spacescalarfield(g), spec, g)), to_np(xd)) < tol


@pytest.mark.parametrize("dtype", DTYPES)
@pytest.mark.parametrize("n", SIZES)
def test_3d_product_sweep_matches_triad_sums(n, dtype):
    if n == 1024 and dtype == torch.float64:
        pytest.skip("the plan and its fields do not fit one GPU")
    k = n // 3
    edges = ((k, 0, 0), (0, k, 0), (0, 0, k), (k, k, k), (k, -k, 1), (1, 0, 0), (0, 1, -1))
    kk, uu = T.random_sparse_field(n, 40, n, extra=edges)
    kout, ref = T.convectiondiffusion(kk, uu, n, 1e-3)
    g = S.Grid(3, n, dtype=dtype, device="cuda:0")
    kf, uf = T.full_modes(kk, uu)
    half = kf[:, 0] >= 0
    at = tuple(torch.from_numpy(a).to(g.device) for a in T.to_rfft_index(kf[half], n))
    u = S.vectorfield(g)
    for c in range(3):
        u[c][at] = torch.from_numpy(uf[half][:, c]).to(g.cdtype).to(g.device)
    du = S.convectiondiffusion_(S.vectorfield(g), u, g, 1e-3)
    ot = tuple(torch.from_numpy(a).to(g.device) for a in T.to_rfft_index(kout, n))
    num = den = 0.0
    for c in range(3):
        r = torch.from_numpy(ref[:, c]).to(g.device)
        num += float((du[c][ot].to(torch.complex128) - r).abs().square().sum())
        den += float(r.abs().square().sum())
        du[c][ot] = 0  # what is left must be zero, and counts as error
        num += float(torch.linalg.vector_norm(du[c]).double() ** 2)
    assert math.sqrt(num / den) < (1e-12 if dtype == torch.float64 else 1e-5)
    g.close()


@pytest.mark.parametrize("captured", (False, True))
@pytest.mark.parametrize("n,m", ((96, 36), (60, 20), (120, 36), (160, 64), (192, 32)))
@pytest.mark.parametrize("dtype", DTYPES)
def test_sfs_on_the_reduced_grid_matches_the_oracle(n, m, dtype, captured):
    """DNS products formed on fewer points than the DNS grid has (96 -> 80, 60 ->
    48, 120 -> 96, 160 -> 128, 192 -> 160), and on the DNS grid where the first
    call is being captured.  Tolerances as in test_gpu_filter.py: tau against the
    size of the products it cancels."""
    gd, gl = (S.Grid(3, k, dtype=dtype, device="cuda:0") for k in (n, m))
    od, ol = O.Grid(3, n), O.Grid(3, m)
    u = O.random_field(od, seed=5, kpeak=4)
    d = 2 * ol.l / m
    ud = [to_dev(c, gd) for c in u]
    ub, tau = S.vectorfield(gl), S.tensorfield(gl)
    if captured:
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph):
            S.sfs_(ub, tau, ud, gd, gl, d)
        graph.replay()
    else:
        S.sfs_(ub, tau, ud, gd, gl, d)
    rb, rt = O.sfs(u, od, ol, d)
    tol = 1e-12 if dtype == torch.float64 else 1e-5
    assert rel_l2([to_np(c) for c in ub], rb) < tol
    s1 = [O.twothirds(O.gaussianfilter(O.cutoff(c, od, ol), d, ol), ol) for c in O.nonlinearity(u, od)]
    scale = math.sqrt(sum(float(np.sum(np.abs(c) ** 2)) for c in s1))
    assert math.sqrt(sum(float(np.sum(np.abs(to_np(x) - y) ** 2)) for x, y in zip(tau, rt))) < tol * scale


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("D,n,dtype", ((3, 32, torch.float64), (3, 36, torch.float32), (3, 60, torch.float64),
                                       (3, 64, torch.float32), (3, 72, torch.float64), (3, 90, torch.float32),
                                       (3, 96, torch.float64), (3, 128, torch.float32), (2, 90, torch.float32),
                                       (2, 160, torch.float64)))
def test_closure_sweeps_match_the_oracle(kind, D, n, dtype):
    """The closures' point functions inside the x sweep and the test filter inside
    the z sweep.  A right-hand side, so the tolerances of one."""
    if kind == "verstappen" and D == 2:
        pytest.skip("Q-R model is only defined in 3D")
    g, go = S.Grid(D, n, dtype=dtype, device="cuda:0"), O.Grid(D, n)
    u = O.random_field(go, seed=21, kpeak=3)
    delta = 2 * go.l / n
    cl, model = _models(kind, delta, g, D)
    ref = [O.twothirds(c, go) for c in O.les_rhs(u, go, lambda uu, GG: model(uu, GG, go), 1e-3)]
    du = S.vectorfield(g)
    S.les_(du, [to_dev(c, g) for c in u], g, cl, 1e-3)
    assert rel_l2([to_np(c) for c in du], ref) < (1e-12 if dtype == torch.float64 else 1e-5)


def test_split_training_gradient_at_128():
    """Forward passes, input gradients and weight gradients of the tensor-core
    network at its larger size against FP64.  Tolerance of the 64^3 case in
    test_gpu_adjoint.py: one step with weights 100 % off leaves a misfit of the
    size that its 40 steps with 1 % do, so the FP32 rounding of the states weighs
    the same."""
    n, dt, nu = 128, 2.5e-3, 1e-3
    go = O.Grid(3, n)
    u = O.random_field(go, seed=7, kpeak=4)
    ws, bs = S.kaiming_cnn_weights(5)
    theta = S.pack_cnn_params(ws, bs)
    off = theta * (1 + np.random.default_rng(8).standard_normal(theta.size))
    res = []
    for dtype in DTYPES:
        g = S.Grid(3, n, dtype=dtype, device="cuda:0")
        if dtype == torch.float32:
            cl = S.create_cnn_closure(4 * go.l / n, nu, g, ws, bs, mu=5.0, sigma=2.0, split=True)
        else:
            cl = S.create_cnn_fp_closure(4 * go.l / n, nu, g, ws, bs, mu=5.0, sigma=2.0)
        u0 = [to_dev(c, g) for c in u]
        S.closure_set_params(cl, off)
        traj = S.rollout_record(g, cl, u0, dt, nu, 1)
        S.closure_set_params(cl, theta)
        res.append(S.rollout_adjoint(g, cl, u0, traj, dt, nu, 1, ckpt_every=1))
        cl.close()
        g.close()
    (l32, g32), (l64, g64) = res
    assert abs(l32 - l64) < 1e-4 * l64
    assert np.linalg.norm(g32 - g64) < 1e-4 * np.linalg.norm(g64)
