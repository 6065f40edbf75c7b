"""Handles whose levels floor odd extents (``n_levels`` given): the last cells of an odd extent
have no coarse cell; the restriction drops them and the prolongation is zero there."""
import numpy as np
import pytest

from oracle import mg, tfops, weights as W

pytestmark = pytest.mark.gpu


def _prolong(w, shape):
    """Nearest prolongation onto ``shape``, zero past the last coarse cell."""
    out = np.zeros(shape, w.dtype)
    up = tfops.prolong_nearest(w, w.dtype.type)
    z, y, x = (min(a, b) for a, b in zip(up.shape, shape))
    out[:z, :y, :x] = up[:z, :y, :x]
    return out


def _sawtooth(ops, phi, b, fine_smooth):
    r = [mg.residual(ops[0], phi, b)]
    for _ in ops[1:]:
        r.append(tfops.restrict_avg(r[-1], np.float64))
    w = mg.jacobi_ref(ops[-1], np.zeros_like(r[-1]), r[-1])
    for l in range(len(ops) - 2, -1, -1):
        w = _prolong(w, r[l].shape)
        if l or fine_smooth:
            w = mg.jacobi_ref(ops[l], w, r[l])
    return mg.jacobi_ref(ops[0], phi - w, b), np.abs(w).max()


# rows of whole and of partial vectors, an odd extent along each axis and on a coarse level,
# two slots (a read past the first one's last coarse plane is a read of the second's)
@pytest.mark.parametrize("shape,levels", [((9, 8, 12), 2), ((8, 9, 16), 3), ((12, 10, 44), 3), ((5, 6, 7), 2),
                                          ((17, 16, 64), 3), ((10, 8, 26), 3)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7", "sigma7-bf16"])
@pytest.mark.parametrize("fine_smooth", [True, False])
def test_sawtooth_on_odd_extents(hfm, shape, levels, form, fine_smooth):
    import torch
    M, ops = hfm.multigrid, hfm.ops
    rng = np.random.default_rng(41)
    B, bf16 = 2, form.endswith("bf16")
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    f = rng.standard_normal((B,) + shape).astype(np.float32)
    sig = np.exp(0.5 * rng.standard_normal((3, B) + shape)).astype(np.float32)
    if bf16:  # exact in 16 bits, so that only the cycle's own roundings are left
        sig = np.exp2(np.round(rng.standard_normal((3, B) + shape))).astype(np.float32)
    K = W.w5_pressure27()
    op, oracle = {"const7": (lambda: ops.Const7(0.5, 1.0, 2.0), lambda b: mg.const7(0.5, 1.0, 2.0, dtype=np.float64)),
                  "k27": (lambda: ops.Stencil27(K), lambda b: mg.Stencil27(np.asarray(K, np.float32), dtype=np.float64)),
                  "sigma7": (lambda: ops.Sigma7(*(dev(s) for s in sig)),
                             lambda b: mg.Sigma7(*(s[b].astype(np.float64) for s in sig), dtype=np.float64))}[form[:6] if bf16 else form]
    op = op()
    cfg = M.SolverConfig.reference(n_levels=levels, cycles=100, fine_smooth=fine_smooth)
    cfg.storage = "bf16" if bf16 else "f32"
    with M.Multigrid(shape, op.kind, cfg, slots=B) as h:
        h.set_operator(op)
        for s in range(B):
            h.load(s, dev(f[s]), dev(f[s]))
        h.run(1)
        got = [h.fetch(s).cpu().numpy() for s in range(B)]
    for s in range(B):
        ref, w = _sawtooth(mg.hierarchy(oracle(s), levels), f[s].astype(np.float64), f[s].astype(np.float64), fine_smooth)
        # a sweep of omega 1 averages: an error of the values it reads passes with weight <= 2;
        # a few dozen roundings of them, or some eight of the storage's 2^-9
        scale = max(np.abs(ref).max(), np.abs(f[s]).max(), w)
        assert np.abs(got[s] - ref).max() <= (16 * 2.0 ** -9 if bf16 else 1e-5) * scale


def _vcycle(ops, l, f, phi, coarse_sweeps=5):
    if l == len(ops) - 1:
        for _ in range(coarse_sweeps):
            phi = mg.jacobi(ops[l], phi, f, 2.0 / 3.0)
        return phi
    for _ in range(2):
        phi = mg.jacobi(ops[l], phi, f, 2.0 / 3.0)
    r = tfops.restrict_avg(mg.residual(ops[l], phi, f), np.float64)
    phi = phi - _prolong(_vcycle(ops, l + 1, r, np.zeros_like(r), coarse_sweeps), phi.shape)
    for _ in range(2):
        phi = mg.jacobi(ops[l], phi, f, 2.0 / 3.0)
    return phi


ODD_BELOW = [((24, 24, 24), 5), ((20, 12, 40), 4), ((28, 20, 24), 4)]


@pytest.mark.parametrize("shape,levels", ODD_BELOW)
@pytest.mark.parametrize("cycle,slots,fused", [("V", 1, True), ("V", 7, True), ("V", 1, False), ("V", 8, False),
                                               ("F", 1, True), ("F", 8, True), ("F", 1, False)])
def test_v_and_f_cycles_refuse_odd_levels(hfm, shape, levels, cycle, slots, fused):
    import torch
    cfg = hfm.multigrid.SolverConfig(cycle=cycle, n_levels=levels, tol=1e-300, fused_coarse=fused)
    op = hfm.ops.Const7(0.5, 1.0, 2.0)
    with hfm.multigrid.Multigrid(shape, op.kind, cfg, slots=slots) as h:
        h.set_operator(op)
        h.load(0, torch.ones(shape, device="cuda"))
        with pytest.raises(hfm._lib.HfmError, match="BAD_ARG"):
            h.run(1)


# the last two: thin levels that fill an SM's shared memory, and a long coarsest solve
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("shape,levels,coarse_sweeps", [s + (5,) for s in ODD_BELOW] + [((4, 6, 1156), 3, 5), ((20, 12, 40), 4, 300)])
def test_many_slot_v_cycles_floor_odd_levels(hfm, shape, levels, form, coarse_sweeps):
    import torch
    ops, rng = hfm.ops, np.random.default_rng(43)
    B = 8
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    f = rng.standard_normal((B,) + shape).astype(np.float32)
    sig = np.exp(0.5 * rng.standard_normal((3, B) + shape)).astype(np.float32)
    K = W.w5_pressure27()
    op = {"const7": lambda: ops.Const7(0.5, 1.0, 2.0), "k27": lambda: ops.Stencil27(K),
          "sigma7": lambda: ops.Sigma7(*(dev(s) for s in sig))}[form]()
    cfg = hfm.multigrid.SolverConfig(cycle="V", n_levels=levels, tol=1e-300, coarse_sweeps=coarse_sweeps)
    with hfm.multigrid.Multigrid(shape, op.kind, cfg, slots=B) as h:
        h.set_operator(op)
        for s in range(B):
            h.load(s, dev(f[s]))
        h.run(1)
        got = [h.fetch(s).cpu().numpy() for s in range(B)]
    for s in (0, B - 1):
        oracle = {"const7": lambda: mg.const7(0.5, 1.0, 2.0, dtype=np.float64),
                  "k27": lambda: mg.Stencil27(np.asarray(K, np.float32), dtype=np.float64),
                  "sigma7": lambda: mg.Sigma7(*(a[s].astype(np.float64) for a in sig), dtype=np.float64)}[form]()
        f64 = f[s].astype(np.float64)
        ref = _vcycle(mg.hierarchy(oracle, levels, 0.5), 0, f64, np.zeros_like(f64), coarse_sweeps)
        assert np.abs(got[s] - ref).max() <= 1e-5 * max(np.abs(ref).max(), np.abs(f64).max())
