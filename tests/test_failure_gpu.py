"""The failure paths of the waits for other CTAs (the persistent pressure solve's, the bitmask
scan's), exercised without faulting the GPU.

The solve runs as one cooperative launch whose CTAs meet at grid barriers (the reference runs its
iterations as host dispatches instead, fluid.wgsl:572-577, src/sim.rs:634-647). Every wait at a
barrier is bounded: after a limit of polls the CTA sets an error flag, returns, and the step
reports NTR_E_TIMEOUT. Here one CTA skips its first arrival (a flag nothing else sets) under a
short limit of 4096 polls: the step must fail promptly with NTR_E_TIMEOUT, the context must stay
usable, and a normal step from a restored snapshot must again equal the oracle bit for bit.

The scan of the block bitmask is one launch whose CTAs wait for the counts of those before them,
with the same bound. Here one CTA keeps its count: the step must end there, none of the steps queued
behind it may run, and a restore must bring the simulation back.
"""
import time

import pytest

from natray_b200 import World
from natray_b200._abi import NatrayError, check, lib
from natray_b200.sim import Sim
from oracle.py import Oracle

from test_parity_gpu import assert_worlds_equal, measured, small

pytestmark = pytest.mark.gpu

NTR_E_TIMEOUT = 5


def test_solver_barrier_timeout_is_reported_and_recoverable():
    w = measured(small())
    s = Sim(world=w)
    assert s.step(2) == 2
    saved = s.snapshot()
    check(lib().ntr_sim_test_barrier(s._h, 4096, 0))
    t0 = time.perf_counter()
    with pytest.raises(NatrayError) as e:
        s.step(1)
    assert e.value.status == NTR_E_TIMEOUT
    assert time.perf_counter() - t0 < 10.0
    # Back to the default limit and no skipped arrival; the context still works.
    check(lib().ntr_sim_test_barrier(s._h, 0, 0xFFFFFFFF))
    s.restore(saved)
    o = Oracle(saved.blob)
    assert s.step(3) == o.step(3) == 3
    assert_worlds_equal(World(o.snapshot()), s.snapshot(), "after a solve whose barrier gave up")
    s.close()


@pytest.mark.parametrize("cta", [0, 1, 2])
def test_scan_timeout_ends_the_step_and_is_recoverable(cta):
    w = measured(small(resolution=40))  # four CTAs of 2,048 words
    words = -(-(w.h.params.bdims[0] * w.h.params.bdims[1] * w.h.params.bdims[2]) // 32)
    assert -(-words // 2048) == 4
    s = Sim(world=w)
    assert s.step(2) == 2
    saved = s.snapshot()
    check(lib().ntr_sim_test_scan(s._h, 4096, cta))
    t0 = time.perf_counter()
    with pytest.raises(NatrayError) as e:
        s.step(4)
    assert e.value.status == NTR_E_TIMEOUT
    assert time.perf_counter() - t0 < 10.0
    # The first of the four began and found no blocks; the others, and those of a later call, are not taken.
    st = s.state
    assert (st["step"], st["n_blocks"], st["dt_ns"]) == (saved.state["step"] + 1, 0, 0)
    check(lib().ntr_sim_test_scan(s._h, 0, 0xFFFFFFFF))
    with pytest.raises(NatrayError) as e:
        s.step(1)
    assert e.value.status == NTR_E_TIMEOUT and s.state["step"] == saved.state["step"] + 1
    # What the steps move is where it was: particles, membrane.
    for sec in ("PARTICLES", "MEM_X"):
        assert s.snapshot().sec(sec).tobytes() == saved.sec(sec).tobytes(), sec
    s.restore(saved)
    o = Oracle(saved.blob)
    assert s.step(3) == o.step(3) == 3
    assert_worlds_equal(World(o.snapshot()), s.snapshot(), "after a scan that gave up")
    s.close()
