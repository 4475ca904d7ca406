"""The step's paths that depend on sizes: the pressure solve with one block a warp (registers),
several (records in shared memory) and more than the shared memory holds (records in global memory);
bullets waiting, flying and gone in one launch, and scenes with different numbers of them in one
batch. All bit for bit."""
import subprocess

import numpy as np
import pytest

from natray_b200 import Params, World, build_world
from natray_b200._abi import NatrayError
from natray_b200.batch import Batch
from natray_b200.sim import Sim
from oracle.py import Oracle

SAME = ("PARTICLES", "MEM_X", "MEM_V", "MEM_PUSH", "ALIVE", "BULLETS", "SECTIONS", "BULLET_HIT", "POSE_LOG", "BLOCKS_PREV", "BLOCK_ACTIVE", "AIR")


def same(a: World, b: World):
    assert a.state == b.state
    for s in SAME:
        assert a.sec(s).tobytes() == b.sec(s).tobytes(), s


def world(p: Params) -> World:
    return World(Oracle(build_world(p).blob).snapshot())  # the measuring substep taken once, on the CPU


@pytest.mark.gpu
@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("ctas", [1, 2, 7, 40])
def test_solve_with_blocks_in_registers_shared_and_global_memory(ctas, fp64):
    w = world(Params(resolution=40, mesh_level=3, block_cap=4096, spray_cap=50000, dt_max=2e-6))
    out = []
    for n in (0, ctas):
        s = Sim(world=w, fp64_reductions=fp64)
        if n:
            s.tuning = {"solve_ctas": n, "cell_ctas_per_sm": 0, "block_ctas_per_sm": 0}
        assert s.step(3) == 3 and s.step(3) == 3
        out.append(s.snapshot())
        assert s.state["n_blocks"] > 12 * 7  # 1 and 2 CTAs: more blocks than records in shared memory
        s.close()
    same(*out)


@pytest.mark.gpu
@pytest.mark.parametrize("preset", ["Four sides", "Crossfire", "Bounce"])
def test_bullets_equal_the_oracle(preset):
    w = world(Params.preset(preset, resolution=24, mesh_level=3, block_cap=8192, spray_cap=50000))
    o, s = Oracle(w.blob), Sim(world=w)
    for _ in range(12):  # the first arrival and the others still waiting (0.5 ms apart)
        assert o.step(8) == s.step(8) == 8
    same(World(o.snapshot()), s.snapshot())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("z", [1e30, -1e30, float("inf"), float("-inf")])
@pytest.mark.parametrize("what", ["particle", "vertex"])
def test_a_coordinate_past_the_cell_numbers_marks_no_block(what, z):
    # A live particle, or a dry vertex (its triangles gone, so that nothing else feels it), at the
    # domain's far corner in x and y and out of the range of 32-bit cell numbers in z: the row of
    # blocks along z is inverted. (A row taken as its length would mark the blocks after it, and past
    # the bitmask's end.)
    w = World(world(Params(resolution=20, mesh_level=3, block_cap=4096, spray_cap=50000)).blob)
    u = w.h.params
    x, y = (u.origin[k] + (u.dims[k] - 0.5) * u.origin[3] for k in (0, 1))
    if what == "particle":
        w.sec("PARTICLES")[7, :3] = (x, y, z)
        assert w.sec("PARTICLES")[7, 7] >= 0.5
    else:
        j = int(np.flatnonzero(w.sec("MEM_PUSH").reshape(-1, 2)[:, 1] > 0)[5])
        w.sec("MEM_X")[j, :3] = (x, y, z)
        w.sec("MEM_WATER")[j, 3] = 0.0
        off = w.sec("VTRI_OFF")
        w.sec("ALIVE")[w.sec("VTRI")[off[j] : off[j + 1]]] = 0
    o, s = Oracle(w.blob), Sim(world=w)
    assert o.step(2) == s.step(2) == 2
    same(World(o.snapshot()), s.snapshot())
    s.close()


@pytest.mark.gpu
@pytest.mark.parametrize("cut", [1, 4, 8])
def test_steps_past_an_overflow_equal_the_oracle(cut):
    # A low balloon falling, with fewer blocks of capacity than it takes: the steps go on with the blocks
    # that fit (the call reports the overflow), and a block past the capacity in one step is no block of
    # the steps after unless they mark it too. One call on either side: nothing adapts in between.
    p = dict(resolution=16, mesh_level=3, spray_cap=100000, height=0.12)
    o = Oracle(world(Params(block_cap=4096, **p)).blob)
    o.step(1)
    w = world(Params(block_cap=World(o.snapshot()).state["n_blocks"] - cut, **p))
    o, s = Oracle(w.blob), Sim(world=w)
    with pytest.raises(RuntimeError):
        o.step(120)
    with pytest.raises(NatrayError) as e:
        s.step(120)
    assert e.value.status == 3  # NTR_E_OVERFLOW
    same(World(o.snapshot()), s.snapshot())
    s.close()


@pytest.mark.gpu
def test_batch_of_scenes_with_different_numbers_of_bullets():
    ws = [world(Params.preset(p, resolution=18, mesh_level=3, block_cap=8192, spray_cap=50000)) for p in ("Four sides", "Bounce", "Crossfire")]
    with Batch(max_scenes=4) as b:
        slots = [b.admit(w, 32) for w in ws]
        while b.step(8):
            pass
        got = [b.snapshot(k) for k in slots]
    for w, g in zip(ws, got):
        s = Sim(world=w)
        for _ in range(4):
            s.step(8)
        same(s.snapshot(), g)
        s.close()


def test_quotient_by_the_reciprocal_is_the_quotient(tmp_path):
    # div_by of dev.cuh restated: a / b for |a| in [2^-80, 2^40], b in [2^-60, 2^40], ends of the
    # mantissas included.
    src = tmp_path / "d.cpp"
    src.write_text(r"""
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
int main() {
    uint64_t s = 88172645463325252ull; long bad = 0;
    for (long t = 0; t < 20000000; t++) {
        s ^= s << 13, s ^= s >> 7, s ^= s << 17;
        uint32_t ma = s & 0x7fffff, mb = (s >> 23) & 0x7fffff;
        const int ea = (int)((s >> 46) % 121) - 80, eb = (int)((s >> 54) % 101) - 60;
        if ((t & 7) == 0) mb = 0x7fffff;
        if ((t & 7) == 1) mb = (s >> 40) & 0xff;
        if ((t & 7) == 2) ma = 0x7fffff - ((s >> 50) & 3);
        float a = std::ldexp(1.0f + ma * 0x1p-23f, ea);
        const float b = std::ldexp(1.0f + mb * 0x1p-23f, eb);
        if (s >> 63) a = -a;
        const float y = 1.0f / b, want = a / b;
        float q = a * y;
        float e = std::fma(-q, b, a);
        q = std::fma(e, y, q);
        e = std::fma(-q, b, a);
        q = std::fma(e, y, q);
        bad += std::memcmp(&q, &want, 4) != 0;
    }
    std::printf("%ld\n", bad);
}
""")
    subprocess.run(["g++", "-O2", "-march=native", "-ffp-contract=off", str(src), "-o", str(tmp_path / "d")], check=True)
    assert subprocess.run([str(tmp_path / "d")], capture_output=True, text=True, check=True).stdout.strip() == "0"
