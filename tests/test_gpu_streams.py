"""Loads, runs and cancels of a many-slot handle on several streams.  A stream is held up by a
bounded device-side sleep, so that the order the calls keep (or need not keep) can be observed."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
SHAPE, SLOTS = (24, 32, 48), 4
HOLD = 600_000_000  # clock ticks: about 0.3 s


@pytest.fixture(scope="module")
def rig(hfm):
    import torch
    rng = np.random.default_rng(59)
    cfg = hfm.multigrid.SolverConfig(cycle="V", tol=1e-300, max_cycles=1000)
    dev = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).cuda()
    sig = [dev(a) for a in np.exp(0.5 * rng.standard_normal((3,) + SHAPE))]
    rhs = dev(rng.standard_normal((SLOTS,) + SHAPE))
    with hfm.multigrid.Multigrid(SHAPE, hfm._lib.OP_SIGMA7, cfg, slots=SLOTS) as h:
        for k in range(SLOTS):
            h.set_operator(hfm.ops.Sigma7(*sig), slot=k)
            h.load(k, rhs[k])
        h.run(20)  # the graph exists from here on
        torch.cuda.synchronize()
        yield torch, h, rhs


def _loaded(torch, h, rhs):
    for k in range(SLOTS):
        h.load(k, rhs[k])
    torch.cuda.synchronize()


def _done(torch, stream):
    e = torch.cuda.Event()
    e.record(stream)
    return e


def _plain(torch, h, rhs, cycles=20):
    _loaded(torch, h, rhs)
    h.run(cycles)
    return [h.fetch(k).cpu().numpy() for k in range(SLOTS)]


def test_cancel_waits_for_no_run_and_ends_the_slot_within_it(rig):
    torch, h, rhs = rig
    want = _plain(torch, h, rhs)
    _loaded(torch, h, rhs)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(HOLD)
        h.run(20)
    ran = _done(torch, a)
    with torch.cuda.stream(b):
        h.cancel(1)
        _done(torch, b).synchronize()
    assert not ran.query()
    torch.cuda.synchronize()
    st = h.query()
    assert [s["cycles"] for s in st] == [20, 0, 20, 20] and not st[1]["active"]
    for k in (0, 2, 3):
        np.testing.assert_array_equal(h.fetch(k).cpu().numpy(), want[k])
    h.run(20)  # no more work for it
    assert [s["cycles"] for s in h.query()] == [40, 0, 40, 40]


def test_cancel_on_the_runs_stream_is_over_before_the_next_run(rig):
    torch, h, rhs = rig
    _loaded(torch, h, rhs)
    h.run(4)
    h.cancel(2)
    before = h.fetch(2).cpu().numpy()
    assert not h.query()[2]["active"]
    h.run(4)
    assert [s["cycles"] for s in h.query()] == [8, 8, 4, 8]
    np.testing.assert_array_equal(h.fetch(2).cpu().numpy(), before)


def test_loads_and_runs_wait_for_each_other(rig):
    torch, h, rhs = rig
    _loaded(torch, h, rhs)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(a):
        torch.cuda._sleep(HOLD)
        h.run(20)
    with torch.cuda.stream(b):  # a load after a run
        h.load(1, rhs[1])
    loaded = _done(torch, b)
    assert not loaded.query()
    torch.cuda.synchronize()
    assert [s["cycles"] for s in h.query()] == [20, 0, 20, 20]
    with torch.cuda.stream(b):  # a run after a load
        torch.cuda._sleep(HOLD)
        h.load(3, rhs[3])
    with torch.cuda.stream(a):
        h.run(20)
    ran = _done(torch, a)
    assert not ran.query()
    torch.cuda.synchronize()
    assert [s["cycles"] for s in h.query()] == [40, 20, 40, 20]


def test_loads_and_cancels_keep_their_order(rig):
    torch, h, rhs = rig
    _loaded(torch, h, rhs)
    a, b = torch.cuda.Stream(), torch.cuda.Stream()
    with torch.cuda.stream(b):  # a load after a cancel
        torch.cuda._sleep(HOLD)
        h.cancel(1)
    with torch.cuda.stream(a):
        h.load(1, rhs[1])
        h.run(20)
    torch.cuda.synchronize()
    assert [s["cycles"] for s in h.query()] == [20] * SLOTS
    with torch.cuda.stream(b):  # a cancel after a load
        torch.cuda._sleep(HOLD)
        h.load(2, rhs[2])
    with torch.cuda.stream(a):
        h.cancel(2)
        h.run(20)
    torch.cuda.synchronize()
    assert [s["cycles"] for s in h.query()] == [40, 40, 0, 40]

