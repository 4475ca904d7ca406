"""The step's paths that depend on sizes: the pressure solve with one block a warp (registers),
several (records in shared memory) and more than the shared memory holds (records in global memory);
bullets waiting, flying and gone in one launch, and scenes with different numbers of them in one
batch; coordinates and block counts past their range; the quotients. All bit for bit."""
import ctypes as C
import re
import subprocess
from pathlib import Path

import numpy as np
import pytest

from natray_b200 import Params, World, build_world
from natray_b200._abi import NatrayError
from natray_b200.batch import Batch
from natray_b200.build import ARCH, NVCC
from natray_b200.sim import Sim
from oracle.py import Oracle

SAME = ("PARTICLES", "MEM_X", "MEM_V", "MEM_PUSH", "ALIVE", "BULLETS", "SECTIONS", "BULLET_HIT", "POSE_LOG", "BLOCKS_PREV", "BLOCK_ACTIVE", "AIR")


def same(a: World, b: World):
    assert a.state == b.state
    for s in SAME:
        assert a.sec(s).tobytes() == b.sec(s).tobytes(), s


def world(p: Params) -> World:
    return World(Oracle(build_world(p).blob).snapshot())  # the measuring substep taken once, on the CPU


def solve_storage(n_blocks: int, ctas: int) -> set:
    """Where the CTAs of a solve of `n_blocks` keep their blocks: CTA c owns those of residues c, c + ctas,
    ... (mod 256); registers while each warp has at most one, then the records its shared memory holds."""
    src = (Path(__file__).resolve().parent.parent / "natray_b200" / "csrc" / "kernels_solve.cuh").read_text()
    warps = int(re.search(r"constexpr int SOLVE_W = (\d+);", src).group(1))
    records = int(re.search(r"SOLVE_DYN = (\d+)u \* sizeof\(SolveRec\);", src).group(1))
    mine = np.bincount(np.arange(n_blocks) % 256 % ctas, minlength=ctas)
    return {"registers" if m <= warps else "shared" if m <= records else "global" for m in mine}


@pytest.mark.gpu
@pytest.mark.parametrize("fp64", [True, False])
@pytest.mark.parametrize("ctas,where", [(1, {"global"}), (2, {"global"}), (4, {"global"}), (5, {"shared"}), (7, {"shared"}), (16, {"registers", "shared"}),
                                        (40, {"registers"})])
def test_solve_with_blocks_in_registers_shared_and_global_memory(ctas, where, fp64):
    w = world(Params(resolution=40, mesh_level=3, block_cap=4096, spray_cap=50000, dt_max=2e-6))
    out = []
    for n in (0, ctas):
        s = Sim(world=w, fp64_reductions=fp64)
        if n:
            s.tuning = {"solve_ctas": n, "cell_ctas_per_sm": 0, "block_ctas_per_sm": 0}
        for _ in range(2):
            assert s.step(3) == 3
            assert solve_storage(s.state["n_blocks"], n or 43) == (where if n else {"registers"})  # by default 43: 512 blocks, 12 a CTA
        out.append(s.snapshot())
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


# div_by (quotient.cuh) over pairs (a, b), with y = 1 / b as its callers keep it, against a / b.
QUOTIENTS = r"""
#ifdef __CUDACC__
#include "quotient.cuh"
__global__ void quotients(const float* a, const float* b, float* q, float* want, long n) {
    for (long i = blockIdx.x * (long)blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
        q[i] = ntr::div_by(a[i], b[i], 1.0f / b[i]), want[i] = a[i] / b[i];
}
extern "C" int run(const float* a, const float* b, float* q, float* want, long n) {
    quotients<<<1184, 256>>>(a, b, q, want, n);
    return (int)cudaDeviceSynchronize();
}
#else
#include <cmath>
#define __device__
#define __noinline__ __attribute__((noinline))
#define __forceinline__ inline
static inline float __fmaf_rn(float a, float b, float c) { return std::fmaf(a, b, c); }
#include "quotient.cuh"
extern "C" int run(const float* a, const float* b, float* q, float* want, long n) {
    for (long i = 0; i < n; i++) q[i] = ntr::div_by(a[i], b[i], 1.0f / b[i]), want[i] = a[i] / b[i];
    return 0;
}
#endif
"""


def quotient_pairs() -> tuple[np.ndarray, np.ndarray]:
    """Numerators and denominators: every pair of the ends of div_by's range (2^-80, 2^-60, 2^40) with a
    few ulp to either side, zeros of both signs, subnormals, the largest and infinite, NaN; and random
    ones around the range and of any size, mantissas at their ends among them."""
    ends = [np.float32(2.0) ** e for e in (-149, -126, -80, -60, 0, 40, 127)]
    special = [0.0, 1e-40, 3.0, 7.0, 1.0 / 3.0, np.finfo(np.float32).max, np.inf, np.nan]
    near = [np.uint32(np.float32(e).view(np.uint32) + d).view(np.float32) for e in ends for d in (0, 1, 2)]
    near += [np.uint32(np.float32(e).view(np.uint32) - d).view(np.float32) for e in ends[1:] for d in (1, 2)]
    v = np.array(special + near, dtype=np.float32)
    v = np.concatenate([v, -v])
    a, b = (x.ravel() for x in np.meshgrid(v, v))
    r = np.random.default_rng(5)
    n = 1 << 22

    def some(lo: int, hi: int) -> np.ndarray:
        m = r.integers(0, 1 << 23, n, dtype=np.uint32)
        m[::8] = 0x7FFFFF
        m[1::8] = r.integers(0, 256, m[1::8].size)
        m[2::8] = 0x7FFFFF - r.integers(0, 4, m[2::8].size)
        return r.permutation((m | (r.integers(lo + 127, hi + 127, n, dtype=np.uint32) << np.uint32(23))).view(np.float32))

    sign = np.where(r.random(2 * n) < 0.5, np.float32(-1), np.float32(1))
    return (np.concatenate([a, np.concatenate([some(-84, 44), some(-126, 128)]) * sign]).astype(np.float32),
            np.concatenate([b, some(-63, 43), some(-126, 128)]).astype(np.float32))


@pytest.mark.parametrize("where", ["host", pytest.param("device", marks=pytest.mark.gpu)])
def test_quotient_by_the_reciprocal_is_the_quotient(tmp_path, where):
    # The step's own source, compiled for the host (IEEE division and fused multiply-add there) and for
    # the device: the same bits as a / b, NaN for NaN.
    csrc = Path(__file__).resolve().parent.parent / "natray_b200" / "csrc"
    src, so = tmp_path / ("q.cu" if where == "device" else "q.cpp"), tmp_path / "q.so"
    src.write_text(QUOTIENTS)
    if where == "device":
        cmd = [NVCC, *ARCH, "-O3", "-fmad=false", "-shared", "-Xcompiler", "-fPIC"]
    else:
        cmd = ["g++", "-O2", "-march=native", "-ffp-contract=off", "-shared", "-fPIC"]
    subprocess.run([*cmd, "-I", str(csrc), str(src), "-o", str(so)], check=True)
    a, b = quotient_pairs()
    if where == "device":
        import torch
        t = [torch.from_numpy(x).cuda() for x in (a, b)] + [torch.empty(a.size, dtype=torch.float32, device="cuda") for _ in range(2)]
        torch.cuda.synchronize()
        assert C.CDLL(str(so)).run(*(C.c_void_p(x.data_ptr()) for x in t), C.c_long(a.size)) == 0
        q, want = t[2].cpu().numpy(), t[3].cpu().numpy()
        with np.errstate(all="ignore"):
            assert np.array_equal(want, a / b, equal_nan=True)  # the device's division itself
    else:
        q, want = np.empty_like(a), np.empty_like(a)
        assert C.CDLL(str(so)).run(*(C.c_void_p(x.ctypes.data) for x in (a, b, q, want)), C.c_long(a.size)) == 0
    bad = np.flatnonzero((q.view(np.uint32) != want.view(np.uint32)) & ~(np.isnan(q) & np.isnan(want)))
    assert bad.size == 0, [(a[i], b[i], q[i], want[i]) for i in bad[:4]]
