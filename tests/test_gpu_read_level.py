"""The level buffers that ``hfm_mg_read_level`` shows, with the small levels in one launch."""
import numpy as np
import pytest

from oracle import weights as W

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(16, 16, 16), (32, 24, 40), (20, 20, 20)])
@pytest.mark.parametrize("form", ["const7", "k27", "sigma7"])
@pytest.mark.parametrize("cycle,slots", [("V", 1), ("V", 8), ("F", 1), ("F", 8)])
def test_levels_after_a_cycle(hfm, shape, form, cycle, slots):
    import torch
    M, ops = hfm.multigrid, hfm.ops
    rng = np.random.default_rng(47)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    f = dev(rng.standard_normal((slots,) + shape))
    sig = np.exp(0.5 * rng.standard_normal((3, slots) + shape))
    op = {"const7": lambda: ops.Const7(0.5, 1.0, 2.0), "k27": lambda: ops.Stencil27(W.w5_pressure27()),
          "sigma7": lambda: ops.Sigma7(*(dev(s) for s in sig))}[form]()
    got = []
    for fused in (True, False):
        cfg = M.SolverConfig(cycle=cycle, tol=1e-300, coarse_sweeps=6, min_coarse_edge=3, fused_coarse=fused)
        with M.Multigrid(shape, op.kind, cfg, slots=slots) as h:
            h.set_operator(op)
            for s in range(slots):
                h.load(s, f[s].contiguous())
            h.run(1)
            got.append([h.read_level(s, l, which).cpu().numpy() for s in {0, slots - 1}
                        for l in range(1, len(h.levels)) for which in (0, 1)])
    # float32 rounding of one cycle, relative to the level's values or a thousandth of the data's
    for a, b in zip(*got):
        assert np.abs(a - b).max() <= 1e-5 * max(np.abs(b).max(), 1e-3 * float(f.abs().max()))
