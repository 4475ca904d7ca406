"""Timed cases of the simulation, through the calls a program makes.

`listed()` names the cases, `draw()` gives more of the same ranges; `prepare()` builds what a
program holds before the call (a scene on the GPU, some steps into its run), `run()` is one pass.
A simulation goes on from pass to pass, as in use: every pass starts where the last one ended.

Kinds of case:
  step   n steps of one scene in one call (`Sim.step`), then its particles in the reference's
         layout in a buffer of the caller's, as a renderer takes them once a frame
  bake   the application's loop: the simulation runs ahead at its own step length and stores
         keyframes (`Cache.bake`), scenes at the library's defaults and its presets
  show   playback: the state between two stored keyframes into the buffers a renderer reads
  batch  n steps of many scenes of uneven size in one batch (`Batch.step`), every scene polled and
         one scene's world handed back, as a server does after a chunk of steps
  serve  whole requests: worlds admitted into a batch, stepped to their end in chunks, their
         worlds handed back, their slots freed
  sort   `ntr_sort_by_block_noalloc`, particles grouped by block in the caller's buffers

Every result is the same bits in every correct version of this library: block and sort order are
canonical, the transfer sums are integers, every other sum has a fixed order (the tests compare the
step bit for bit with the CPU restatement). So the tolerance is "exact", and there is no error
against 64 bits to measure where a pass is some steps of a whole simulation (`exact` is None).
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from natray_b200 import Params
from natray_b200._abi import SHOWN, check, lib
from natray_b200.batch import Batch
from natray_b200.cache import Cache
from natray_b200.serve import build_worlds, mixed_scenes, scene_params
from natray_b200.sim import Sim
from natray_b200.world import sized_for


def listed() -> list[dict]:
    return [
        # `particles` sets the lattice's resolution, as `sized_for` has it.
        # The tests' scene (resolution 20): the smallest in use, a step a call (interactive, latency).
        dict(name="step 4k", kind="step", particles=4200, diameter=16.0, mesh=3, speed=350.0, steps=1, ahead=10, fp64=True),
        # The size of the bench's small scene (8 cm, resolution 51), a step a call.
        dict(name="step 66k", kind="step", particles=69500, diameter=8.0, mesh=4, speed=300.0, steps=1, ahead=40, fp64=True),
        # A served scene's size (the requests' median) in its chunk of steps, with the reference's
        # FP32 sums in the solver.
        dict(name="step 128k fp32 sums", kind="step", particles=128000, diameter=11.0, mesh=5, speed=250.0, steps=8, ahead=16, fp64=False),
        # The bench scene: 1M particles, in flight and impact (ahead 5) and with the bullet inside
        # the water (ahead 150).
        dict(name="step 1M", kind="step", particles=1000000, diameter=16.0, mesh=6, speed=350.0, steps=4, ahead=5, fp64=True),
        dict(name="step 1M inside", kind="step", particles=1000000, diameter=16.0, mesh=6, speed=350.0, steps=4, ahead=150, fp64=True),
        # The largest scene the requests are clipped to.
        dict(name="step 2M", kind="step", particles=2000000, diameter=20.0, mesh=6, speed=400.0, steps=2, ahead=20, fp64=True),
        # The application: default resolution and membrane; one default shot, and four of them.
        dict(name="bake default", kind="bake", preset="Backlit", resolution=64, steps=8, ahead=48),
        dict(name="bake four sides", kind="bake", preset="Four sides", resolution=64, steps=8, ahead=160),
        # Playback of the bench scene.
        dict(name="show 1M", kind="show", particles=1000000, diameter=16.0, mesh=6, speed=350.0, keys=6, ahead=60),
        # The batched workload: 64 scenes, 16k-512k particles, two chunks of 8 steps.
        dict(name="batch 64", kind="batch", scenes=64, lo=16000, hi=512000, steps=8, calls=2, ahead=16),
        # Three requests of small to median size, 96 steps each in chunks of 8.
        dict(name="serve 3", kind="serve", scenes=3, lo=16000, hi=128000, steps=96, chunk=8),
        # The allocation-free sort at the bench scene's size and block count.
        dict(name="sort 1M", kind="sort", n=976915, blocks=2997),
    ]


def _log(rng, lo: float, hi: float) -> float:
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng) -> dict:
    kind = rng.choice(["step", "step", "step", "step", "bake", "bake", "show", "batch", "serve", "sort"])
    if kind == "step":
        n = int(_log(rng, 4000, 2e6))
        return dict(kind=kind, particles=n, diameter=round(rng.uniform(6.5, 22.0), 2), mesh=rng.choice([3, 4, 5, 6]),
                    speed=round(_log(rng, 40, 600), 1), steps=rng.randint(1, max(1, min(16, int(8e6 / n)))), ahead=rng.randint(1, 200),
                    fp64=rng.random() < 0.75)
    if kind == "bake":
        return dict(kind=kind, preset=rng.choice(["Backlit", "Tumbling rifle round", "Crossfire", "Four sides", "Moon gravity",
                                                  "Weightless", "Slow pellet", "Bounce"]),
                    resolution=rng.randint(24, 100), steps=rng.randint(4, 16), ahead=rng.randint(8, 200))
    if kind == "show":
        return dict(kind=kind, particles=int(_log(rng, 4000, 2e6)), diameter=round(rng.uniform(6.5, 20.0), 2),
                    mesh=rng.choice([3, 4, 5, 6]), speed=round(_log(rng, 100, 600), 1), keys=rng.randint(2, 8), ahead=rng.randint(4, 120))
    if kind == "batch":
        lo = int(_log(rng, 4000, 32000))
        return dict(kind=kind, scenes=rng.randint(2, 40), lo=lo, hi=int(lo * _log(rng, 2, 16)), steps=rng.randint(2, 8), calls=2,
                    ahead=rng.randint(1, 48))
    if kind == "serve":
        lo = int(_log(rng, 4000, 32000))
        return dict(kind=kind, scenes=rng.randint(1, 4), lo=lo, hi=int(lo * _log(rng, 2, 8)), steps=rng.randint(24, 96),
                    chunk=rng.choice([4, 8, 16]))
    return dict(kind="sort", n=int(_log(rng, 1000, 1048576)), blocks=int(_log(rng, 20, 65535)))


# ---- inputs ------------------------------------------------------------------------------------


class _Lent:
    """A device buffer lent by the library, for torch; the tensor keeps its owner alive."""

    def __init__(self, owner, ptr: int, shape: tuple, typestr: str):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": typestr, "version": 3, "strides": None}


def _lent(owner, ptr: int, shape: tuple, typestr: str = "<f4") -> torch.Tensor:
    return torch.as_tensor(_Lent(owner, ptr, shape, typestr), device="cuda")


def _scene(case: dict, seed: int) -> Params:
    """The case's scene: the particles' jitter, where the bullet strikes and its speed are the seed's."""
    r = np.random.default_rng(seed)
    d = case["diameter"]
    return Params(diameter=d, resolution=sized_for(case["particles"], d), mesh_level=case["mesh"], bullet=6, caliber=8,
                  bullet_speed=case["speed"] * r.uniform(0.97, 1.03), impact_offset=r.uniform(-1.0, 1.0), dt_max=2e-6, seed=seed + 1)


def _preset(case: dict, seed: int) -> Params:
    r = np.random.default_rng(seed)
    p = Params.preset(case["preset"], resolution=case["resolution"], seed=seed + 1)
    return p.set("impact_offset", p.shots[0].impact_offset_cm + r.uniform(-0.5, 0.5))


def _mixed(case: dict, seed: int, n: int) -> list[Params]:
    """Scenes log-uniform in particles between the case's ends. The sizes are the case's (so that
    the seeds cost the same), the balloons, shots and jitter the seed's."""
    sizes = np.exp(np.random.default_rng(n).uniform(math.log(case["lo"]), math.log(case["hi"]), n))
    r = np.random.default_rng(seed)
    diameters = np.random.default_rng(n + 1).uniform(6.5, 16.0, n)
    return [scene_params(int(p), float(d), float(r.uniform(0.95, 1.05) * v), seed * 1000 + i + 1)
            for i, (p, d, v) in enumerate(zip(sizes, diameters, np.random.default_rng(n + 2).uniform(150.0, 400.0, n)))]


def _ahead(step, n: int) -> None:
    """n steps in chunks, as a program takes them (the substeps adapt between chunks)."""
    while n > 0:
        step(min(n, 8))
        n -= 8


def _sim_views(st: dict) -> None:
    """The simulation's buffers as torch tensors, and the caller's buffer of packed particles."""
    s, i = st["sim"], st["sim"].info
    st["packed"] = torch.empty((i.n_particles, 20), dtype=torch.float32, device="cuda")
    # (Past the step's blocks and drops they hold what earlier steps left there, or zeros.)
    st["views"] = {"mem_pos": _lent(s, s.buffer("MEM_POS")[0], (i.n_verts, 4)), "alive": _lent(s, s.buffer("ALIVE")[0], (i.n_tris,), "<i4"),
                   "air": _lent(s, s.buffer("AIR")[0], (5, i.block_cap, 64)), "spray": _lent(s, s.buffer("SPRAY")[0], (i.spray_cap, 12))}
    p, n = s.buffer("TOUCH")
    st["views"]["touch"] = _lent(s, p, (n // 4,), "<i4")


def prepare(case: dict, seed: int) -> dict:
    kind = case["kind"]
    if kind == "sort":
        # Particles in lattice order: neighbours in the list mostly share a block, some are dead.
        g = torch.Generator(device="cuda").manual_seed(seed)
        n, nb = case["n"], case["blocks"]
        base = torch.arange(n, device="cuda", dtype=torch.float64) * (nb / n)
        k = (base + torch.randn(n, device="cuda", generator=g, dtype=torch.float64) * (0.02 * nb)).long().clamp(0, nb - 1).int()
        k[torch.randperm(n, device="cuda", generator=g)[: n // 100]] = -1
        return dict(case=case, keys=k, live=n - n // 100, sorted=torch.empty(n, dtype=torch.int32, device="cuda"),
                    start=torch.empty(nb + 1, dtype=torch.int32, device="cuda"))
    if kind in ("batch", "serve"):
        worlds = build_worlds(_mixed(case, seed, case["scenes"]), threads=8)
        b = Batch(max_scenes=max(8, case["scenes"]))
        st = dict(case=case, batch=b, worlds=worlds)
        if kind == "batch":
            st["slots"] = [b.admit(w, 1 << 30) for w in worlds]
            _ahead(b.step, case["ahead"])
            st["smallest"] = min(range(len(worlds)), key=lambda k: worlds[k].h.n_particles)
            del st["worlds"]
        return st
    if kind == "step":
        sim = Sim(_scene(case, seed), fp64_reductions=case["fp64"])
        _ahead(sim.step, case["ahead"])
        st = dict(case=case, sim=sim)
        _sim_views(st)
        return st
    if kind == "bake":
        p = _preset(case, seed)
        sim = Sim(p)
        sim.set_batch_steps(8)  # batches end where a count says, not the clock: runs repeat
        cache = Cache(sim, p)
        _ahead(cache.bake, case["ahead"])
        st = dict(case=case, sim=sim, cache=cache)
        _sim_views(st)
        return st
    # show
    sim = Sim(_scene(case, seed))
    sim.set_batch_steps(4)
    sim.advance(0.0, 1)
    _ahead(sim.step, case["ahead"])
    cache = Cache(sim)
    for _ in range(case["keys"]):
        sim.step(2)
        sim.advance(sim._info().t, 0)  # the clock the keyframes carry follows the steps
        cache.store()
    keys = cache.keys()[1:]
    times = [a["t"] + f * (b["t"] - a["t"]) for a, b in zip(keys[:-1], keys[1:]) for f in (0.25, 0.5, 0.8)] or [keys[0]["t"]]
    i = sim.info
    buf = {}
    for name, shape, t in (("PARTICLES", (i.n_particles, 8), "<f4"), ("MEM_POS", (i.n_verts, 4), "<f4"), ("ALIVE", (i.n_tris,), "<i4"),
                           ("WET", None, "<i4")):
        p, n = C.c_void_p(), C.c_size_t()
        check(lib().ntr_cache_buffer(cache._h, SHOWN[name], C.byref(p), C.byref(n)))
        buf[name] = _lent((cache, sim), p.value, shape or (n.value // 4,), t)
    return dict(case=case, sim=sim, cache=cache, times=times, at=0, shown=buf)


# ---- a pass ------------------------------------------------------------------------------------


def _state(s: dict) -> np.ndarray:
    """The state's words (f64 holds each exactly)."""
    return np.array(list(s.values()), dtype=np.float64)


def _frame(st: dict) -> dict:
    """The frame a renderer takes: the particles packed into its buffer, the rest as lent."""
    s, v = st["sim"], st["views"]
    packed = st["packed"]
    check(lib().ntr_sim_pack_particles(s._h, C.c_void_p(packed.data_ptr()), packed.numel() * 4, None))
    return {"particles": packed, "state": _state(s.state), **v}


def _sections(w) -> dict:
    """A world handed back: its state and its sections, those whose length the scene fixes."""
    names = ("PARTICLES", "MEM_X", "MEM_V", "MEM_WATER", "MEM_LAYER", "MEM_PUSH", "ALIVE", "BULLETS", "SECTIONS", "POSE_LOG", "TOUCH")
    return {"state": _state(w.state), **{k: w.sec(k) for k in names}}


def run(st: dict):
    case = st["case"]
    kind = case["kind"]
    if kind == "step":
        st["sim"].step(case["steps"])
        return _frame(st)
    if kind == "bake":
        st["cache"].bake(case["steps"])
        return _frame(st)
    if kind == "show":
        st["cache"].show(st["times"][st["at"] % len(st["times"])])
        st["at"] += 1
        return st["shown"]
    if kind == "batch":
        b = st["batch"]
        for _ in range(case["calls"]):
            b.step(case["steps"])
        return {"states": np.stack([_state(b.poll(k)["state"]) for k in st["slots"]]),
                "world": _sections(b.snapshot(st["slots"][st["smallest"]]))}
    if kind == "serve":
        b = st["batch"]
        slots = [b.admit(w, case["steps"]) for w in st["worlds"]]
        while b.step(case["chunk"]):
            pass
        out = [_sections(b.snapshot(k)) for k in slots]
        for k in slots:
            b.retire(k)
        return out
    stream = torch.cuda.current_stream().cuda_stream
    check(lib().ntr_sort_by_block_noalloc(st["keys"].data_ptr(), case["n"], case["blocks"], st["sorted"].data_ptr(), st["start"].data_ptr(),
                                          C.c_void_p(stream)))
    # The entries past the last block's end (as many as there are dead particles) are not meaningful.
    return {"sorted": st["sorted"][: st["live"]], "start": st["start"]}


# ---- what a pass takes at the least ---------------------------------------------------------------


def _step_bytes(n: float, mesh: int) -> float:
    """A step's state read and written once: 160 B a particle; its cells (8 particles each) 160 B;
    two rubber substeps' 256 B a vertex and 32 B a triangle."""
    v = 10 * 4**mesh + 2
    return 160.0 * n + 160.0 * n / 8 + 2 * (256.0 * v + 32.0 * 2 * v)


def work(case: dict) -> dict:
    kind = case["kind"]
    if kind == "sort":
        return {"bytes": 8.0 * case["n"] + 4.0 * case["blocks"], "flops": 0.0}
    if kind == "step":
        n = case["particles"]
        return {"bytes": case["steps"] * _step_bytes(n, case["mesh"]) + 160.0 * n, "flops": 0.0}
    if kind == "bake":
        n = math.pi / 6 * case["resolution"] ** 3
        return {"bytes": case["steps"] * _step_bytes(n, 6) + 188.0 * n, "flops": 0.0}
    if kind == "show":
        v = 10 * 4 ** case["mesh"] + 2
        return {"bytes": 48.0 * case["particles"] + 32.0 * v + 8.0 * v + 8.0 * 1024 * 1024, "flops": 0.0}
    # The sizes are log-uniform: their mean.
    mean = (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"])
    steps = case["steps"] * (case["calls"] if kind == "batch" else 1)
    return {"bytes": case["scenes"] * steps * _step_bytes(mean, 5), "flops": 0.0}


def tolerance(case: dict):
    return "exact"


def exact(case: dict, seed: int):
    """The sort's result by numpy (whole numbers); None for the rest, some steps of a simulation."""
    if case["kind"] != "sort":
        return None
    k = prepare(case, seed)["keys"].cpu().numpy().astype(np.int64)
    order = np.argsort(np.where(k < 0, case["blocks"], k), kind="stable")[: int((k >= 0).sum())]
    start = np.searchsorted(np.sort(np.where(k < 0, case["blocks"], k)), np.arange(case["blocks"] + 1))
    return {"sorted": torch.from_numpy(order.astype(np.int32)), "start": torch.from_numpy(start.astype(np.int32))}
