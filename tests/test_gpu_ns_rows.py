"""The row-of-four stencil kernels of the flow solver (momentum, pressure gradient,
divergence) on ragged rows and unaligned fields."""
import numpy as np
import pytest

from oracle import ns as ons, tfops, weights as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(3, 3, 3), (3, 5, 4), (4, 9, 132), (5, 7, 130), (6, 4, 33)])
@pytest.mark.parametrize("offset", [0, 1])
def test_momentum_gradient_divergence(hfm, shape, offset):
    import torch
    ns = hfm.ns
    rng = np.random.default_rng(11)
    n = int(np.prod(shape))

    def dev(a):  # `offset` floats past a 16-byte boundary
        t = torch.zeros(n + 4, device="cuda")[offset:offset + n].view(shape)
        return t.copy_(torch.from_numpy(np.ascontiguousarray(a)))

    u, v, w, p = (rng.standard_normal(shape).astype(np.float32) for _ in range(4))
    Kd, (Kx, Ky, Kz) = W.w1_diffusion27(0.1, 0.25, 1.0), W.advection_kernels(0.1)
    K = [rng.standard_normal((3, 3, 3)).astype(np.float32) for _ in range(3)]  # no zero weights
    # sums of at most 109 products of O(1) values: 109 roundings of 6e-8 of sum |products|
    tol = lambda ref: 1e-5 * max(1.0, np.abs(ref).max())
    for Kq in ((Kd, Kx, Ky, Kz), (Kd, *K)):
        out = [dev(np.zeros(shape, np.float32)) for _ in range(3)]
        vel = [dev(a) for a in (u, v, w)]
        ns.momentum_stage(vel, vel, out, *Kq, 0.5)
        for f, got in zip((u, v, w), out):
            ref = f + 0.5 * ons.momentum_rhs(f.astype(np.float64), u, v, w, *Kq, dt=np.float64)
            assert np.abs(got.cpu().numpy() - ref).max() <= tol(ref) * 10
    g = ns.pressure_gradient(dev(p), dev(u), dev(v), dev(w), *K)
    for got, f, k in zip(g, (u, v, w), K):
        ref = f - tfops.conv3d_same(p, k, np.float64)
        assert np.abs(got.cpu().numpy() - ref).max() <= tol(ref)
    for bc in (False, True):
        b = ns.divergence(dev(u), dev(v), dev(w), dev(np.zeros(shape, np.float32)), *K, bc_source=bc)
        ref = -sum(tfops.conv3d_same(f, k, np.float64) for f, k in zip((u, v, w), K))
        if bc:
            ref = ons.bc_source(ref)
        assert np.abs(b.cpu().numpy() - ref).max() <= tol(ref)
