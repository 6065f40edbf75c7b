"""Ragged rows (two cells or one per thread in the register-queue kernels): 16-bit storage in every
pass, and the masked launches of a handle with partial sums and shared grids."""
import ctypes as C

import numpy as np
import pytest

from oracle import mg, tfops, weights as W

pytestmark = pytest.mark.gpu

ULP = {"bf16": 2.0 ** -8, "f16": 2.0 ** -11}


@pytest.fixture(scope="module")
def T(hfm):
    import torch
    return torch


# rows of 4 k + 2 cells, odd rows, and whole vectors at a pointer 1 or 2 elements off
@pytest.mark.parametrize("shape,offset", [((4, 6, 10), 0), ((9, 8, 34), 0), ((6, 20, 70), 0), ((5, 7, 9), 0),
                                          ((3, 33, 31), 0), ((9, 8, 101), 0), ((6, 8, 24), 1), ((6, 8, 24), 2),
                                          ((4, 16, 64), 1), ((4, 16, 64), 2)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("dtype", ["bf16", "f16"])
def test_typed_passes_match_oracle(hfm, T, shape, offset, form, dtype):
    L = hfm._lib
    tdt, code = {"bf16": (T.bfloat16, L.BF16), "f16": (T.float16, L.F16)}[dtype]
    rng = np.random.default_rng(61)
    B, n = 2, 2 * int(np.prod(shape))

    def field(a, off=offset):
        """Rounded to the storage type, `off` elements past an aligned allocation; and its value."""
        t = T.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda().to(tdt)
        store = T.empty(t.numel() + 8, dtype=tdt, device="cuda")
        view = store[off:off + t.numel()].view(t.shape)
        view.copy_(t)
        return view, view.double().cpu().numpy()

    x, x64 = field(rng.standard_normal((B,) + shape))
    f, f64 = field(rng.standard_normal((B,) + shape))
    op = L.HfmOperator()
    op.coef_dtype, op.scale = code, 1.0
    keep = []
    if form == "sigma7":
        op.kind = L.OP_SIGMA7
        s64 = []
        for k in range(3):
            t, v = field(np.exp(rng.standard_normal((B,) + shape)))
            keep.append(t)
            s64.append(v)
            op.coef[k], op.c[k] = t.data_ptr(), (0.5, 1.0, 2.0)[k]
        ops = [mg.Sigma7(*(s[b] for s in s64), c=(0.5, 1.0, 2.0), dtype=np.float64) for b in range(B)]
    elif form == "const7":
        op.kind = L.OP_CONST7
        op.k[0], op.k[1], op.k[2] = 0.5, 1.0, 2.0
        ops = [mg.const7(0.5, 1.0, 2.0, dtype=np.float64)] * B
    else:
        K = W.w5_pressure27().astype(np.float32)
        op.kind = L.OP_K27
        for i, v in enumerate(K.reshape(27)):
            op.k[i] = float(v)
        ops = [mg.Stencil27(K.astype(np.float64), dtype=np.float64)] * B
    P, dims, st = (lambda t: C.c_void_p(t.data_ptr())), (B,) + shape, hfm.ops._stream()
    even = not any(e & 1 for e in shape)
    half = tuple(e // 2 for e in shape)
    out = {}

    def call(name, *args):
        o, _ = field(np.zeros((B,) + (half if name == "restricted" else shape)), 0 if name == "restricted" else offset)
        args = [P(o) if a is out else a for a in args]
        L.call(*args)
        out[name] = o

    call("jacobi", "hfm_op_jacobi_typed", C.byref(op), code, P(x), P(f), out, *dims, 2.0 / 3.0, 0, st)
    call("residual", "hfm_op_residual_typed", C.byref(op), code, P(x), P(f), out, *dims, 0, st)
    if even:
        w, w64 = field(rng.standard_normal((B,) + half))
        call("restricted", "hfm_residual_restrict_typed", C.byref(op), code, P(x), P(f), C.c_void_p(0), out, *dims, 0, st)
        call("corrected", "hfm_prolong_correct_smooth_typed", C.byref(op), code, P(x), P(w), P(f), out, *dims, 2.0 / 3.0, 0, st)
    ref = {"jacobi": [mg.jacobi(o, x64[b], f64[b], 2.0 / 3.0) for b, o in enumerate(ops)],
           "residual": [mg.residual(o, x64[b], f64[b]) for b, o in enumerate(ops)]}
    scale = max(np.abs(v).max() for v in ref["residual"])
    if even:
        ref["restricted"] = [tfops.restrict_avg(r, np.float64) for r in ref["residual"]]
        ref["corrected"] = [mg.jacobi(o, x64[b] - tfops.prolong_nearest(w64[b], np.float64), f64[b], 2.0 / 3.0)
                            for b, o in enumerate(ops)]
    for name, t in out.items():
        want = np.stack(ref[name])
        # computed in float32 and rounded once to the storage type
        excess = np.abs(t.double().cpu().numpy() - want) - ULP[dtype] * np.abs(want)
        assert excess.max() <= 1e-5 * max(scale, np.abs(want).max()), name


# a slot's bits alone, in a few and with every slot at work; the first check's residual norm
# against the oracle (two sweeps from zero).  Rows for two cells per thread with coarser levels
# below, odd rows (one level) for one cell per thread, whole vectors for comparison; the table of
# one and of several active counts per entry
@pytest.mark.parametrize("shape,slots", [((18, 20, 22), 33), ((12, 10, 70), 5), ((34, 36, 38), 70), ((15, 20, 21), 9),
                                         ((17, 30, 63), 40), ((16, 24, 32), 12), ((16, 32, 64), 6)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("accel", ["none", "cg"])
def test_masked_launches_share_the_grid(hfm, T, shape, slots, form, accel):
    ops, rng = hfm.ops, np.random.default_rng(67)
    dev = lambda a: T.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    sig = np.exp(0.5 * rng.standard_normal((3,) + shape)).astype(np.float32)
    K = W.w5_pressure27()
    op = {"const7": lambda: ops.Const7(0.5, 1.0, 2.0), "k27": lambda: ops.Stencil27(K),
          "sigma7": lambda: ops.Sigma7(*(dev(s) for s in sig))}[form]()
    oracle = {"const7": lambda: mg.const7(0.5, 1.0, 2.0, dtype=np.float64),
              "k27": lambda: mg.Stencil27(np.asarray(K, np.float32), dtype=np.float64),
              "sigma7": lambda: mg.Sigma7(*(s.astype(np.float64) for s in sig), dtype=np.float64)}[form]()
    f = rng.standard_normal((slots,) + shape).astype(np.float32)
    rhs = dev(f)
    cfg = hfm.multigrid.SolverConfig(cycle="V", accel=accel, tol=1e-300, max_cycles=1000, coarse_sweeps=4)
    probe = sorted({0, slots // 2, slots - 1})
    with hfm.multigrid.Multigrid(shape, op.kind, cfg, slots=slots) as h:
        for k in range(slots):
            h.set_operator(op, slot=k)

        def run(which, cycles):
            for k in range(slots):
                h.cancel(k)
            for k in which:
                h.load(k, rhs[k])
            h.run(cycles)
            st = h.query()
            return {k: (h.fetch(k).cpu().numpy(), st[k]["cycles"], st[k]["rel_resid"]) for k in probe if k in which}

        every, few = run(range(slots), 3), run(probe, 3)
        for k in probe:
            alone = run([k], 3)[k]
            # (cycles of a single level make no check)
            assert alone[1] == (0 if accel == "none" and len(h.levels) == 1 else 3) and np.isfinite(alone[0]).all()
            for other in (few[k], every[k]):
                np.testing.assert_array_equal(alone[0], other[0])
                assert alone[1:] == other[1:]
        if accel == "none" and len(h.levels) > 1:
            first = run(range(slots), 1)
            for k in probe:
                phi = np.zeros(shape)
                for _ in range(2):
                    phi = mg.jacobi(oracle, phi, f[k].astype(np.float64), 2.0 / 3.0)
                want = np.linalg.norm(mg.residual(oracle, phi, f[k])) / np.linalg.norm(f[k].astype(np.float64))
                assert abs(first[k][2] - want) <= 1e-5 * want
