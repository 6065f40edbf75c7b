"""Infinite and NaN cells under a zero weight of a 27-point kernel: they reach no other cell in
the ragged sweeps and residuals and in the restricted residual."""
import numpy as np
import pytest

from oracle import weights as W

pytestmark = pytest.mark.gpu


# one, two and four cells per thread in the register-queue kernels, the plane-marching
# restriction (X >= 48), and rows for the one-thread-per-cell kernels
@pytest.mark.parametrize("shape", [(6, 8, 9), (5, 6, 10), (6, 8, 26), (6, 8, 20), (8, 16, 64), (4, 4, 6)])
@pytest.mark.parametrize("bad", [np.inf, np.nan])
def test_zero_weights_leave_out_what_is_not_finite(hfm, shape, bad):
    import torch
    ops, L = hfm.ops, hfm._lib
    rng = np.random.default_rng(53)
    K = np.asarray(W.w2_7point(), np.float32).reshape(3, 3, 3)
    assert (K == 0).sum() == 20
    x, f = (torch.from_numpy(rng.standard_normal(shape).astype(np.float32)).cuda() for _ in range(2))
    cell = tuple(n // 2 for n in shape)
    y = x.clone()
    y[cell] = float(bad)
    op = ops.Stencil27(K)
    even, ragged = not any(n & 1 for n in shape), shape[2] % 4 != 0

    def run(t):
        out = {}
        if ragged:
            out["jacobi"] = ops.jacobi(op, t, f, 0.8)
            out["residual"] = ops.residual(op, t, f)
            out["conv"] = ops.conv3d_same(t.view((1,) + shape + (1,)), K).view(shape)
        if even:
            out["restricted"] = ops.residual_restrict(op, t, f)[0]
        return {k: v.cpu().numpy() for k, v in out.items()}

    good, got = run(x), run(y)
    for name, a in got.items():
        hit = np.zeros(shape, bool)  # the cell and its neighbours under the seven weights
        for d in np.argwhere(K != 0) - 1:
            n = np.array(cell) + d
            if ((n >= 0) & (n < shape)).all():
                hit[tuple(n)] = True
        if name == "restricted":
            s = tuple(n // 2 for n in shape)
            hit = hit.reshape(s[0], 2, s[1], 2, s[2], 2).any(axis=(1, 3, 5))
        np.testing.assert_array_equal(a[~hit], good[name][~hit])
        assert not np.isfinite(a[hit]).any()
