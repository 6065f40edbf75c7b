"""Kernels and launch rules for grids that leave most of the GPU idle (one instance, small or
ragged extents)."""
import numpy as np
import pytest

from oracle import mg, weights as W

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def T(hfm):
    import torch
    return torch


def dev(T, a):
    return T.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()


# one instance marches one plane per block (two for the restriction), 700 instances the
# whole column: the same cells, the same bits
@pytest.mark.parametrize("shape", [(2, 2, 4), (6, 4, 8), (10, 6, 12), (16, 16, 16), (34, 8, 44)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
def test_result_does_not_depend_on_the_chunk_length(hfm, T, shape, form):
    B = 700
    rng = np.random.default_rng(3)
    x = rng.standard_normal((4,) + shape)
    f = rng.standard_normal((4,) + shape)
    sig = np.exp(rng.standard_normal((3, 4) + shape))
    ops = hfm.ops

    def op(rep):
        if form == "const7":
            return ops.Const7(0.5, 1.0, 2.0)
        if form == "k27":
            return ops.Stencil27(W.w5_pressure27())
        return ops.Sigma7(*(rep(dev(T, sig[k])) for k in range(3)))

    def run(rep):
        o, xd, fd = op(rep), rep(dev(T, x)), rep(dev(T, f))
        y = ops.jacobi(o, xd, fd, 2.0 / 3.0, sweeps=2)
        return y, ops.residual(o, y, fd), ops.residual_restrict(o, y, fd)

    one = run(lambda t: t[:1].contiguous())
    many = run(lambda t: t.repeat(B // 4, 1, 1, 1))
    for a, b in zip(one, many):
        np.testing.assert_array_equal(a[0].cpu().numpy(), b[0].cpu().numpy())
        np.testing.assert_array_equal(a[0].cpu().numpy(), b[B - 4].cpu().numpy())


# the 27-point residual + restriction: plane-marching (X >= 48), register-queue and generic
# kernels; the x-end rule comes with the handle's outflow rule
@pytest.mark.parametrize("shape", [(2, 2, 4), (4, 6, 8), (6, 34, 20), (10, 8, 48), (12, 18, 64), (6, 16, 68), (4, 4, 6)])
@pytest.mark.parametrize("xend", [False, True])
def test_pressure_residual_restriction(hfm, T, shape, xend):
    rng = np.random.default_rng(5)
    B = 3
    x = rng.standard_normal((B,) + shape).astype(np.float32)
    f = rng.standard_normal((B,) + shape).astype(np.float32)
    K = rng.standard_normal((3, 3, 3))
    rc, rf = hfm.ops.residual_restrict(hfm.ops.Stencil27(K), dev(T, x), dev(T, f),
                                       flags=hfm._lib.FLAG_ZERO_XEND if xend else 0, want_fine=True)
    op = mg.Stencil27(np.asarray(K, np.float32), dtype=np.float64)
    for b in range(B):
        ref = mg.residual(op, x[b], f[b])
        if xend:
            ref[..., -1] = 0
        scale = np.abs(ref).max()  # 27 products of O(1): 28 roundings of 6e-8 of it
        assert np.abs(rf[b].cpu().numpy() - ref).max() <= 1e-5 * scale
        c = ref.reshape(shape[0] // 2, 2, shape[1] // 2, 2, shape[2] // 2, 2).mean(axis=(1, 3, 5))
        assert np.abs(rc[b].cpu().numpy() - c).max() <= 1e-5 * scale


# the fused coarse levels against one launch per level step: first fused level in quads
# (X % 4 == 0) and cell by cell (X % 4 != 0), one level and several below it, every operator,
# V and F cycles (the F-cycle's second visit starts from a non-zero iterate)
@pytest.mark.parametrize("shape", [(16, 16, 16), (32, 24, 40), (20, 20, 20), (12, 36, 28), (8, 64, 24)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("cycle,nu", [("V", (2, 2)), ("V", (0, 1)), ("V", (1, 0)), ("F", (2, 2)), ("F", (1, 2))])
def test_fused_coarse_levels_few_slots(hfm, T, shape, form, cycle, nu):
    M, ops = hfm.multigrid, hfm.ops
    rng = np.random.default_rng(17)
    B = 2
    f = dev(T, rng.standard_normal((B,) + shape))
    sig = np.exp(rng.standard_normal((3, B) + shape))
    op = {"const7": lambda: ops.Const7(0.5, 1.0, 2.0), "k27": lambda: ops.Stencil27(W.w5_pressure27()),
          "sigma7": lambda: ops.Sigma7(*(dev(T, sig[k]) for k in range(3)))}[form]()
    outs = []
    for fused in (True, False):
        cfg = M.SolverConfig(cycle=cycle, nu_pre=nu[0], nu_post=nu[1], tol=1e-300, max_cycles=10,
                             coarse_sweeps=5, min_coarse_edge=3, fused_coarse=fused)
        with M.Multigrid(shape, op.kind, cfg, slots=B) as h:
            h.set_operator(op)
            for s in range(B):
                h.load(s, f[s].contiguous())
            h.run(3)
            outs.append(np.stack([h.fetch(s).cpu().numpy() for s in range(B)]))
    # three cycles of a few dozen float32 roundings per value, damped by the smoothing
    assert np.abs(outs[0] - outs[1]).max() <= 1e-5 * np.abs(outs[1]).max()


# the reference cycle with its small levels in one launch against one launch per step: the
# iterate and every level's restricted residual and correction
@pytest.mark.parametrize("shape", [(16, 16, 16), (64, 64, 64), (40, 8, 8), (24, 12, 20), (64, 128, 128)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("sweeps,xend", [(1, False), (2, False), (1, True)])
def test_fused_sawtooth_levels(hfm, T, shape, form, sweeps, xend):
    M, ops = hfm.multigrid, hfm.ops
    rng = np.random.default_rng(23)
    f = dev(T, rng.standard_normal(shape))
    sig = np.exp(0.5 * rng.standard_normal((3,) + shape))
    op = {"const7": lambda: ops.Const7(0.5, 1.0, 2.0), "k27": lambda: ops.Stencil27(W.w5_pressure27()),
          "sigma7": lambda: ops.Sigma7(*(dev(T, sig[k]) for k in range(3)))}[form]()
    n_levels = int(np.log2(min(shape))) + 1
    outs = []
    for fused in (True, False):
        cfg = M.SolverConfig.reference(n_levels=n_levels, cycles=100, coarse_sweeps=sweeps, zero_xend=xend,
                                       fine_smooth=not xend)
        cfg.fused_coarse = fused
        with M.Multigrid(shape, op.kind, cfg, slots=1) as h:
            h.set_operator(op)
            h.load(0, f, f)
            h.run(3)
            got = [h.fetch(0)]
            for l in range(1, len(h.levels)):
                got += [h.read_level(0, l, 0), h.read_level(0, l, 1)]
            outs.append([g.cpu().numpy() for g in got])
    for a, b in zip(*outs):  # float32 rounding of three cycles, as the other parity tests allow
        assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-3 * np.abs(outs[1][0]).max())


# rows that are no multiple of 4 cells, and views off a 16-byte boundary: two cells or one per
# thread in the register-queue kernels
@pytest.mark.parametrize("shape", [(3, 4, 8), (5, 7, 9), (4, 6, 10), (6, 33, 31), (8, 10, 34), (9, 8, 101), (34, 20, 70)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("offset", [0, 1, 2])
def test_ragged_rows(hfm, T, shape, form, offset):
    ops, L = hfm.ops, hfm._lib
    rng = np.random.default_rng(29)
    B, n = 2, 2 * int(np.prod(shape))

    def field(a):  # `offset` floats past a 16-byte boundary
        t = T.zeros(n + 4, device="cuda")[offset:offset + n].view((B,) + shape)
        return t.copy_(T.from_numpy(np.ascontiguousarray(a, dtype=np.float32)))

    x, f = (rng.standard_normal((B,) + shape).astype(np.float32) for _ in range(2))
    sig = np.exp(rng.standard_normal((3, B) + shape)).astype(np.float32)
    K = rng.standard_normal((3, 3, 3)).astype(np.float32)
    K[1, 1, 1] = 20.0
    op = {"const7": lambda: ops.Const7(0.5, 1.0, 2.0), "k27": lambda: ops.Stencil27(K),
          "sigma7": lambda: ops.Sigma7(*(field(sig[k]) for k in range(3)))}[form]()
    even = not any(e & 1 for e in shape)
    w = rng.standard_normal((B,) + tuple(e // 2 for e in shape)).astype(np.float32)
    for flags in (0, L.FLAG_ZERO_XEND, L.FLAG_TOP_COPY):
        y = ops.jacobi(op, field(x), field(f), 2.0 / 3.0, flags=flags)
        r = ops.residual(op, field(x), field(f), flags=flags & L.FLAG_ZERO_XEND)
        if even:
            c = ops.residual_restrict(op, field(x), field(f), flags=flags & L.FLAG_ZERO_XEND)
            p = ops.prolong_correct_smooth(op, field(x), dev(T, w), field(f), 2.0 / 3.0)
        for b in range(B):
            o = {"const7": lambda: mg.const7(0.5, 1.0, 2.0, dtype=np.float64),
                 "k27": lambda: mg.Stencil27(K, dtype=np.float64),
                 "sigma7": lambda: mg.Sigma7(*(sig[k, b] for k in range(3)), dtype=np.float64)}[form]()
            xb = x[b].astype(np.float64)
            if flags == L.FLAG_ZERO_XEND:
                xb[..., -1] = 0
            ref = mg.jacobi(o, xb, f[b], 2.0 / 3.0)
            if flags == L.FLAG_TOP_COPY:
                ref[0] = ref[1]
            res = mg.residual(o, x[b], f[b])
            if flags == L.FLAG_ZERO_XEND:
                res[..., -1] = 0
            pairs = [(y, ref), (r, res)]
            if even:
                s = tuple(e // 2 for e in shape)
                pairs.append((c, res.reshape(s[0], 2, s[1], 2, s[2], 2).mean(axis=(1, 3, 5))))
                up = w[b].repeat(2, 0).repeat(2, 1).repeat(2, 2)
                pairs.append((p, mg.jacobi(o, x[b] - up.astype(np.float64), f[b], 2.0 / 3.0)))
            for got, want in pairs:  # at most 28 roundings of 6e-8 of the largest term
                scale = max(np.abs(want).max(), np.abs(res).max())
                assert np.abs(got[b].cpu().numpy() - want).max() <= 1e-5 * scale


# the 2D fused coarse cycle against one launch per level step, bit for bit: levels in quads
# with whole and straddling rows, one cell per thread, ringed levels (X % 4 != 0 above 512
# cells), coarsest levels on a warp (a full one too) and above
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("shape,min_edge", [((64, 64), 4), ((56, 56), 4), ((48, 80), 5), ((52, 46), 23), ((40, 24), 3),
                                            ((16, 128), 4), ((64, 32), 8), ((60, 44), 30)])
def test_2d_fused_levels_same_bits(hfm, T, periodic, shape, min_edge):
    KM = hfm.kolmogorov
    rng = np.random.default_rng(31)
    w = KM.laplace5(0.1)
    w += 0.02 * rng.standard_normal((3, 3))  # no zero weights
    w[1, 1] *= 1.2
    f = T.from_numpy(rng.standard_normal((2,) + shape).astype(np.float32)).cuda()
    outs = []
    for fused in (True, False):
        m = KM.Multigrid2D(shape, w, periodic=periodic, slots=2, min_edge=min_edge, fused_coarse=fused, coarse_sweeps=7)
        p = T.zeros((2,) + shape, device="cuda")
        for _ in range(2):
            m.iterate(p, f)
        outs.append(p.cpu().numpy())
    np.testing.assert_array_equal(outs[0], outs[1])


# the fine level's two legs with the outer defect and the update inside, against the separate
# launches, bit for bit: tile edges, axes shorter than a ring
@pytest.mark.parametrize("periodic", [True, False])
@pytest.mark.parametrize("storage", ["f32", "bf16"])
@pytest.mark.parametrize("shape", [(2, 2), (2, 34), (4, 6), (8, 32), (10, 66), (130, 96)])
def test_2d_outer_legs_same_bits(hfm, T, periodic, storage, shape):
    L, KM = hfm._lib, hfm.kolmogorov
    code, dt = KM._DT[storage]
    Y, X = shape
    rng = np.random.default_rng(37)
    w = KM._w9(KM.laplace5(0.3) + 0.1 * rng.standard_normal((3, 3)))
    fl = L.FLAG_PERIODIC if periodic else 0
    st, P = hfm.ops._stream(), KM._p
    p, f = (T.from_numpy(rng.standard_normal((2, Y, X)).astype(np.float32)).cuda() for _ in range(2))
    wc = T.from_numpy(rng.standard_normal((2, Y // 2, X // 2)).astype(np.float32)).cuda().to(dt)
    new = lambda *s: T.zeros((2,) + s, device="cuda", dtype=dt)
    a, b = [(new(Y, X), new(Y, X), new(Y // 2, X // 2)) for _ in range(2)]
    L.call("hfm_outer_pre2_restrict2d", code, w, P(p), P(f), *(P(t) for t in a), 2, Y, X, 0.8, fl, st)
    L.call("hfm_outer_residual2d", w, P(p), P(f), code, P(b[0]), 2, Y, X, fl, None, None, st)
    L.call("hfm_pre2_restrict2d", code, w, P(b[0]), P(b[1]), P(b[2]), 2, Y, X, 0.8, fl, st)
    for s, t in zip(a, b):
        assert T.equal(s, t)
    pa, pb, out = p.clone(), p.clone(), new(Y, X)
    L.call("hfm_post2_update2d", code, w, P(a[1]), P(wc), -1.0, P(a[0]), P(pa), -1.0, 2, Y, X, 0.8, fl, st)
    L.call("hfm_jacobi2d", code, w, P(a[1]), P(wc), -1.0, P(a[0]), P(out), 2, Y, X, 0.8, fl | L.FLAG_TWO_SWEEPS, st)
    L.call("hfm_update2d", P(pb), code, P(out), -1.0, 2 * Y * X, st)
    assert T.equal(pa, pb)


# the blocks of a many-slot handle are dealt to its active slots: a slot's solve has the same
# bits alone, in a few and with every slot at work (table of one and of several counts per
# entry, more slots than are listed; register-queue and plane-marching kernels; planes that
# are no multiple of a segment)
@pytest.mark.parametrize("shape,slots,accel,storage", [
    ((16, 16, 16), 2, "cg", "f32"), ((18, 12, 20), 33, "cg", "f32"), ((8, 8, 8), 70, "cg", "f32"),
    ((8, 8, 8), 300, "cg", "f32"), ((32, 32, 32), 64, "ir", "bf16"), ((18, 32, 64), 3, "ir", "bf16"),
    ((36, 16, 48), 40, "ir", "bf16"), ((16, 64, 64), 7, "cg", "f32"), ((20, 16, 72), 65, "none", "f32")])
def test_active_slots_share_the_grid_same_bits(hfm, T, shape, slots, accel, storage):
    rng = np.random.default_rng(9)
    cfg = hfm.multigrid.SolverConfig(cycle="V", accel=accel, storage=storage, tol=1e-6, max_cycles=60,
                                     inner_tol=1e-3)
    sig = dev(T, np.exp(0.5 * rng.standard_normal((3,) + shape)))
    rhs = dev(T, rng.standard_normal((slots,) + shape))
    with hfm.multigrid.Multigrid(shape, hfm._lib.OP_SIGMA7, cfg, slots=slots) as h:
        for k in range(slots):
            h.set_operator(hfm.ops.Sigma7(sig[0], sig[1], sig[2]), slot=k)

        def solve(which):
            for k in which:
                h.load(k, rhs[k])
            for _ in range(40):
                h.run(4)
                st = h.query()
                if not any(st[k]["active"] for k in which):
                    break
            return {k: (h.fetch(k).cpu().numpy(), st[k]["status"], st[k]["cycles"], st[k]["rel_resid"])
                    for k in which}

        probe = sorted({0, slots // 2, slots - 1})
        every = solve(range(slots))
        few = solve(probe)
        for k in probe:
            alone = solve([k])[k]
            assert alone[1] == hfm._lib.OK and alone[3] <= 1e-6
            for other in (few[k], every[k]):
                np.testing.assert_array_equal(alone[0], other[0])
                assert alone[1:] == other[1:]


def test_cancel_on_another_stream_leaves_the_other_slots_alone(hfm, T):
    """The blocks of a launch share out the active slots: a cancel from another stream takes
    effect between launches, and the slots that stay keep their bits."""
    shape, slots = (24, 32, 48), 6
    rng = np.random.default_rng(13)
    cfg = hfm.multigrid.SolverConfig(cycle="V", accel="cg", tol=1e-6, max_cycles=60)
    sig = dev(T, np.exp(0.5 * rng.standard_normal((3,) + shape)))
    rhs = dev(T, rng.standard_normal((slots,) + shape))
    other = T.cuda.Stream()
    with hfm.multigrid.Multigrid(shape, hfm._lib.OP_SIGMA7, cfg, slots=slots) as h:
        for k in range(slots):
            h.set_operator(hfm.ops.Sigma7(sig[0], sig[1], sig[2]), slot=k)

        def solve(cancel):
            for k in range(slots):
                h.load(k, rhs[k])
            for it in range(15):
                h.run(4)
                if cancel and it < slots - 2:
                    with T.cuda.stream(other):
                        h.cancel(it + 1)
            st = h.query()
            return h.fetch(0).cpu().numpy(), h.fetch(slots - 1).cpu().numpy(), st

        a, b = solve(False), solve(True)
        assert b[2][0]["status"] == hfm._lib.OK and b[2][slots - 1]["status"] == hfm._lib.OK
        assert not any(s["active"] for s in b[2])
        for x, y in zip(a[:2], b[:2]):
            np.testing.assert_array_equal(x, y)
