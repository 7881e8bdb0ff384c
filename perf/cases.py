"""Timed cases of the Brownian-dynamics framework, through its public entry points.

A case is a dict with a ``kind``:

* ``step``      a resident system advanced by ``steps`` timesteps, its records taken over on the
                device into the caller's buffer (``System.step`` + ``System.state_pointer``).
                ``network`` is the c2 or c3 network of ``gpusmoldyn_gb300.configs`` at its density.
* ``ensemble``  a batch of c2 instances of uneven sizes, stepped and read the same way.
* ``job``       a whole simulation with host arrays on a handle that is kept: upload, ``steps``
                timesteps, event counts, readback.
* ``release``   a job whose A molecules all start at one point, so a few cells hold thousands.
* ``diffuse``   a system without reactions: every molecule only diffuses.
* ``serve``     requests through the continuous-batching server, more of them than slots, each with
                its own size and step count (``steps`` to ``steps`` + 30).
* ``io``        particles up to the handle and back to the host.
* ``sort``      the allocation-free cell sort on the caller's device buffers.

The particle count changes with the reactions, so results go into the caller's own buffers, which
have room for more; the count is returned beside them.

Positions are uniform in the box from numpy's Philox generator with the case's seed, as the
benchmark's are; species are at the network's stationary composition.
"""
import ctypes as C
import math

import numpy as np
import torch

from gpusmoldyn_gb300 import _lib as L
from gpusmoldyn_gb300 import configs
from gpusmoldyn_gb300.serve import Server
from gpusmoldyn_gb300.system import System

C2_DENSITY = configs.C2_DENSITY
C3_DENSITY = 2.0
C1_DENSITY = 40.0


def listed():
    return [
        # one update of a small reversible system, as an interactive or coupled program calls it
        # once per frame: all launches and latency
        dict(name="step_c2_4k_x1", kind="step", network="c2", n=4001, steps=1, normals="boxmuller", sort="auto",
             surfaces=False),
        # the reference-scale run A + B -> C: upload, 100 steps, counts and particles back
        dict(name="job_c1_40k_x100", kind="job", n=40000, steps=100),
        # the same system with its 20,000 A released at one point: crowded cells
        dict(name="release_c1_40k_x20", kind="release", n=40000, steps=20),
        # 8 species and 12 reactions at a size that stays in the L2 cache, between two looks at it
        dict(name="step_c3_300k_x16", kind="step", network="c3", n=300007, steps=16, normals="boxmuller", sort="auto",
             surfaces=False),
        # the reversible million-particle configuration
        dict(name="step_c2_1m_x16", kind="step", network="c2", n=1000000, steps=16, normals="boxmuller", sort="auto",
             surfaces=False),
        # the 8-species network inside a cell: membrane and a nucleus of 1,280 triangles
        dict(name="step_c3_cell_2m_x8", kind="step", network="c3", n=2000003, steps=8, normals="boxmuller",
             sort="auto", surfaces=True),
        # the headline configuration
        dict(name="step_c3_16m_x8", kind="step", network="c3", n=16000000, steps=8, normals="boxmuller", sort="auto",
             surfaces=False),
        # a parameter sweep in one batch: 64 instances of 1e3 to 1e6 particles, D and k_on scaled
        dict(name="ensemble_c4_64_x4", kind="ensemble", instances=64, n_lo=1000, n_hi=1000000, mix=4, steps=4),
        # tracer diffusion without reactions
        dict(name="diffuse_1m_x16", kind="diffuse", n=1000003, steps=16, normals="boxmuller"),
        # 12 requests through 8 slots of the server
        dict(name="serve_c5_12_x60", kind="serve", jobs=12, slots=8, n_lo=1000, n_hi=500000, steps=60),
        # set-up and checkpoint traffic: particles in and out through pinned host arrays
        dict(name="io_c3_4m", kind="io", n=4000000, pinned=True),
        # cell lists for a host program that owns all device memory
        dict(name="sort_2m", kind="sort", n=2000003),
    ]


def _size(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi))))) | 1


def draw(rng):
    kind = rng.choice(["step", "step", "step", "step", "ensemble", "job", "release", "diffuse", "serve", "io", "sort"])
    if kind == "step":
        network = rng.choice(["c2", "c3"])
        n = _size(rng, 1000, 8000000)
        steps = rng.choice([s for s in (1, 2, 3, 5, 8, 16, 19, 32) if s == 1 or n * s <= 64000000])
        return dict(kind=kind, network=network, n=n, steps=steps, normals=rng.choice(["boxmuller"] * 5 + ["table"]),
                    sort=rng.choice(["auto"] * 5 + ["compact"]), surfaces=network == "c3" and rng.random() < 0.2)
    if kind == "ensemble":
        inst = rng.randint(3, 64)
        return dict(kind=kind, instances=inst, n_lo=1000, n_hi=_size(rng, 5000, 500000), mix=rng.randint(1, 999),
                    steps=rng.randint(1, 8))
    if kind == "job":
        return dict(kind=kind, n=2 * _size(rng, 500, 100000), steps=rng.randint(10, 150))
    if kind == "release":
        return dict(kind=kind, n=2 * _size(rng, 500, 25000), steps=rng.randint(5, 20))
    if kind == "diffuse":
        return dict(kind=kind, n=_size(rng, 1000, 4000000), steps=rng.choice([1, 3, 16, 25]),
                    normals=rng.choice(["boxmuller"] * 4 + ["table"]))
    if kind == "serve":
        slots = rng.randint(3, 8)
        return dict(kind=kind, jobs=slots + rng.randint(0, 4), slots=slots, n_lo=1000,
                    n_hi=_size(rng, 5000, 300000), steps=rng.randint(10, 60))
    if kind == "io":
        return dict(kind=kind, n=_size(rng, 1000, 4000000), pinned=rng.random() < 0.75)
    return dict(kind=kind, n=_size(rng, 1000, 3000000))


# ------------------------------------------------------------------ helpers
class _Records:
    """The records of a System as the caller's program sees them: device memory, (slots, 4) float32
    words x, y, z, w.  The System owns that memory, so whoever looks at it keeps the System."""

    def __init__(self, system):
        pointer, self.slots = system.state_pointer()
        self.system = system
        self.__cuda_array_interface__ = dict(shape=(self.slots, 4), typestr="<f4", data=(pointer, False), version=3)


def _room(n):
    """Slots of a caller's buffer for a system of about n particles."""
    return n + n // 4 + 1024


def _take(system, buffer):
    """The system's records in the caller's device buffer."""
    rec = _Records(system)
    buffer[: rec.slots].copy_(torch.as_tensor(rec, device="cuda"))
    return {"xyz": buffer[:, :3], "w": buffer.view(torch.int32)[:, 3], "slots": rec.slots}


def _side(n, density):
    return float((n / density) ** (1.0 / 3.0))


def _pack(pos):
    xyz4 = np.ones((len(pos), 4), np.float32)
    xyz4[:, :3] = pos
    return xyz4


def _c1_system(n, seed):
    side = _side(n, C1_DENSITY)
    s = System((0, 0, 0), (side, side, side), dt=1e-3, seed=seed)
    a, b, c = s.add_species(1.0), s.add_species(1.0), s.add_species(0.5)
    s.add_reaction(2, [a, b], [c], 0.01)
    s.finalize()
    return s, side


def _diffusing(case, seed):
    """Box side, diffusion coefficients, positions and species of a diffuse case."""
    n = case["n"]
    side = _side(n, C3_DENSITY)
    D, _ = configs.c3_network()
    g = configs.rng(seed)
    pos = configs.uniform_positions(g, n, (0, 0, 0), (side, side, side))
    return side, D, pos, g.integers(0, len(D), n).astype(np.int32)


def _sort_input(case, seed):
    n = case["n"]
    dims = [max(1, min(101, round((n / 3.0) ** (1.0 / 3.0))))] * 3
    g = torch.Generator(device="cuda").manual_seed(int(seed))
    side = _side(n, C3_DENSITY)
    rec = torch.rand((n, 4), generator=g, device="cuda") * side
    rec.view(torch.int32)[:, 3] = torch.randint(0, 8, (n,), generator=g, device="cuda", dtype=torch.int32)
    return rec, side, dims


def _serve_jobs(case):
    """(particles, steps) of the requests: sizes spread over the range by a fixed stride, so that
    large and small ones mix."""
    k = case["jobs"]
    stride = next(s for s in (5, 7, 3, 1) if math.gcd(s, k) == 1)
    lo, hi = math.log(case["n_lo"]), math.log(case["n_hi"])
    return [(int(math.exp(lo + (hi - lo) * ((j * stride) % k + 0.5) / k)), case["steps"] + 10 * (j % 4))
            for j in range(k)]


# ------------------------------------------------------------------ prepare
def prepare(case, seed):
    seed = int(seed)
    kind, n = case["kind"], case.get("n")
    if kind == "step":
        if case["network"] == "c2":
            side = _side(n, C2_DENSITY)
            s = configs.c2_system(side, seed, case["normals"], sort=case["sort"])
            s.set_particles(*configs.c2_particles(n // 2, n - n // 2, side, seed))
        else:
            s = configs.build_c3(n, _side(n, C3_DENSITY), seed, case["normals"], surfaces=case["surfaces"],
                                 sort=case["sort"])
        return dict(kind=kind, system=s, steps=case["steps"], buffer=torch.zeros((_room(n), 4), device="cuda"))
    if kind == "ensemble":
        inst, counts = configs.c4_instances(case["instances"], case["mix"], case["n_lo"], case["n_hi"])
        for k, d in enumerate(inst):
            d["seed"] = 1000 * seed + k
        s = System(dt=5e-4, seed=seed, instances=inst)
        configs.c2_network(s)
        s.finalize()
        pos, sp = configs.c4_positions(inst, counts, seed)
        s.set_ensemble_particles(pos, sp, counts)
        return dict(kind=kind, system=s, steps=case["steps"],
                    buffer=torch.zeros((_room(int(counts.sum())), 4), device="cuda"))
    if kind in ("job", "release"):
        s, side = _c1_system(n, seed)
        pos = configs.uniform_positions(configs.rng(seed), n, (0, 0, 0), (side, side, side))
        if kind == "release":
            pos[: n // 2] = np.float32(side / 2)
        sp = np.repeat(np.arange(2, dtype=np.int32), [n // 2, n - n // 2])
        return dict(kind=kind, system=s, steps=case["steps"], xyz4=_pack(pos), species=sp,
                    out=(np.zeros((n, 4), np.float32), np.zeros(n, np.int32)))
    if kind == "diffuse":
        side, D, pos, sp = _diffusing(case, seed)
        s = System((0, 0, 0), (side, side, side), dt=1e-3, seed=seed, normals=case["normals"])
        for d in D:
            s.add_species(float(d))
        s.finalize()
        s.set_particles(pos, sp)
        return dict(kind=kind, system=s, steps=case["steps"], buffer=torch.zeros((n, 4), device="cuda"))
    if kind == "serve":
        _, frac = configs.c3_steady_state(configs.c3_network()[1], C3_DENSITY)
        jobs, out = [], []
        for j, (m, steps) in enumerate(_serve_jobs(case)):
            side = _side(m, C3_DENSITY)
            desc = dict(box_lo=(0.0, 0.0, 0.0), box_hi=(side, side, side), seed=100 * seed + j)
            pos = configs.uniform_positions(configs.rng(desc["seed"]), m, desc["box_lo"], desc["box_hi"])
            jobs.append(dict(id=j, arrival=0.0, n=m, steps=steps, seed=desc["seed"],
                             payload=(desc, pos, configs.c3_species(m, frac), steps)))
            out.append((np.zeros((_room(m), 3), np.float32), np.zeros(_room(m), np.int32)))
        return dict(kind=kind, server=Server(max_instances=case["slots"]), jobs=jobs, out=out)
    if kind == "io":
        side = _side(n, C3_DENSITY)
        pos, sp = configs.c3_particles(n, side, seed)
        xyz4, species = torch.from_numpy(_pack(pos)), torch.from_numpy(sp)
        out = torch.empty((n, 4), dtype=torch.float32), torch.empty(n, dtype=torch.int32)
        if case["pinned"]:
            xyz4, species, out = xyz4.pin_memory(), species.pin_memory(), tuple(t.pin_memory() for t in out)
        return dict(kind=kind, system=configs.c3_system(n, side, seed), xyz4=xyz4.numpy(), species=species.numpy(),
                    out=tuple(t.numpy() for t in out), keep=(xyz4, species, out))
    if kind == "sort":
        rec, side, dims = _sort_input(case, seed)
        cells = dims[0] * dims[1] * dims[2]
        return dict(kind=kind, n=n, input=rec, output=torch.empty_like(rec),
                    start=torch.empty(cells + 1, dtype=torch.int32, device="cuda"), lib=L.load(),
                    lo=(C.c_float * 3)(0.0, 0.0, 0.0), hi=(C.c_float * 3)(side, side, side),
                    dims=(C.c_uint32 * 3)(*dims))
    raise ValueError(kind)


# ---------------------------------------------------------------------- run
def run(state):
    kind = state["kind"]
    if kind == "sort":
        out, start = state["output"], state["start"]
        rc = state["lib"].bd_cell_sort_static(
            C.c_void_p(state["input"].data_ptr()), state["n"], state["lo"], state["hi"], state["dims"],
            C.c_void_p(out.data_ptr()), C.c_void_p(start.data_ptr()),
            C.c_void_p(torch.cuda.current_stream().cuda_stream))
        L.check(rc, "bd_cell_sort_static")
        return {"xyz": out[:, :3], "w": out.view(torch.int32)[:, 3], "cell_start": start}
    if kind == "serve":
        done = state["server"].run([dict(j) for j in state["jobs"]], time_scale=0.0, keep_results=True)["done"]
        got = []
        for j in sorted(done, key=lambda j: j["id"]):
            pos, sp = state["out"][j["id"]]
            m = j["n_final"]
            pos[:m], sp[:m] = j["result"]
            got.append({"pos": pos, "species": sp, "n": m})
        return got
    s = state["system"]
    if kind in ("job", "release"):
        s.set_particles(state["xyz4"], state["species"])
        s.step(state["steps"])
        pos, sp = state["out"]
        m = len(s.particles4(out=(pos, sp))[1])
        return {"pos": pos, "species": sp, "n": m, "events": s.event_counts().astype(np.int64)}
    if kind == "io":
        s.set_particles(state["xyz4"], state["species"])
        pos, sp = s.particles4(out=state["out"])
        return {"pos": pos, "species": sp}
    # after the copy of the last pass, which reads the records on the caller's stream
    s.step(state["steps"], stream=torch.cuda.current_stream().cuda_stream)
    return _take(s, state["buffer"])


# --------------------------------------------------------------------- work
def work(case):
    """A step has to read and write every 16-byte record (all others decide where it goes) and
    draws three normals and a cell for it; molecules that only diffuse need one read and one write
    whatever the number of steps; uploads and readbacks move float4 positions and int species."""
    kind = case["kind"]
    n, steps = case.get("n"), case.get("steps", 1)
    if kind == "diffuse":
        return dict(bytes=32 * n, flops=60 * n * steps)
    if kind == "io":
        return dict(bytes=2 * (20 + 16) * n, flops=n)
    if kind == "sort":
        return dict(bytes=32 * n + 4 * n // 3, flops=10 * n)
    if kind == "ensemble":
        n = int(configs.c4_instances(case["instances"], case["mix"], case["n_lo"], case["n_hi"])[1].sum())
    if kind == "serve":
        jobs = _serve_jobs(case)
        n, moves = sum(m for m, _ in jobs), sum(m * t for m, t in jobs)
    else:
        moves = n * steps
    host = 2 * 20 * n if kind in ("job", "release", "serve") else 0
    return dict(bytes=32 * moves + host, flops=60 * moves)


# -------------------------------------------------------------------- exact
def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 on uint64 arrays of 32-bit words (Salmon et al., SC'11)."""
    m = np.uint64(0xFFFFFFFF)
    sh = np.uint64(32)
    for _ in range(10):
        p0, p1 = c0 * np.uint64(0xD2511F53), c2 * np.uint64(0xCD9E8D57)
        c0, c1, c2, c3 = (p1 >> sh) ^ c1 ^ k0, p1 & m, (p0 >> sh) ^ c3 ^ k1, p0 & m
        k0, k1 = (k0 + np.uint64(0x9E3779B9)) & m, (k1 + np.uint64(0xBB67AE85)) & m
    return c0, c1, c2, c3


def _exact_diffuse(case, seed):
    """The positions of a diffuse case after its steps, in 64 bits: the step's own Philox words,
    Box-Muller and reflecting walls."""
    side, D, pos, sp = _diffusing(case, seed)
    side = float(np.float32(side))
    n = case["n"]
    sigma = np.sqrt(2.0 * D.astype(np.float64) * float(np.float32(1e-3)))[sp]
    x = pos.astype(np.float64)
    slot = np.arange(n, dtype=np.uint64)
    k0, k1 = np.uint64(seed & 0xFFFFFFFF), np.uint64(seed >> 32)
    s8, byte = np.uint64(8), np.uint64(0xFF)

    def unit(w):
        return (w >> s8).astype(np.float64) * 2.0 ** -24

    for t in range(case["steps"]):
        a, b, c, _ = _philox(slot, np.uint64(t), np.full(n, 1 << 24, np.uint64), np.uint64(0), k0, k1)
        ra = np.sqrt(-2.0 * np.log(unit(a) + 2.0 ** -25))
        rc = np.sqrt(-2.0 * np.log(unit(c) + 2.0 ** -25))
        low = ((a & byte) << np.uint64(24)) | ((b & byte) << np.uint64(16)) | ((c & byte) << s8)
        angle = 2.0 * math.pi * unit(b)
        for axis, g in enumerate((ra * np.cos(angle), ra * np.sin(angle), rc * np.cos(2.0 * math.pi * unit(low)))):
            y = np.abs(x[:, axis] + sigma * g)
            x[:, axis] = np.where(y > side, 2.0 * side - y, y)
    return {"xyz": torch.from_numpy(x), "w": torch.from_numpy(sp), "slots": n}


def _exact_sort(case, seed):
    """The records in cell order, inside a cell by their words as unsigned integers.  The cell of a
    record is defined by float32 operations, so they are repeated in float32."""
    rec, side, dims = _sort_input(case, seed)
    side = float(np.float32(side))
    words = rec.view(torch.int32).long() & 0xFFFFFFFF
    key = torch.zeros(len(rec), dtype=torch.int64, device="cuda")
    for a in (2, 1, 0):
        inv = torch.tensor(float(np.float32(dims[a]) / np.float32(side)), dtype=torch.float32, device="cuda")
        cell = torch.clamp(torch.floor(rec[:, a] * inv).long(), 0, dims[a] - 1)
        key = key * dims[a] + cell
    order = torch.arange(len(rec), device="cuda")
    for col in (words[:, 3], words[:, 2], words[:, 1], words[:, 0], key):
        order = order[torch.sort(col[order], stable=True).indices]
    counts = torch.bincount(key, minlength=dims[0] * dims[1] * dims[2])
    start = torch.cat([torch.zeros(1, dtype=torch.int64, device="cuda"), counts.cumsum(0)])
    return {"xyz": rec[order, :3].double(), "w": words[order, 3].int(), "cell_start": start.int()}


def exact(case, seed):
    """Box-Muller diffusion, the cell sort and a round trip of the particles have 64-bit values.  A
    reacting step has none: which records share a cell, their order by the bits of float32
    coordinates and with it every later random number are defined in 32 bits."""
    seed = int(seed)
    kind = case["kind"]
    if kind == "diffuse" and case["normals"] == "boxmuller" and case["n"] * case["steps"] <= 40000000:
        return _exact_diffuse(case, seed)
    if kind == "sort":
        return _exact_sort(case, seed)
    if kind == "io":
        pos, sp = configs.c3_particles(case["n"], _side(case["n"], C3_DENSITY), seed)
        return {"pos": torch.from_numpy(_pack(pos)).double(), "species": torch.from_numpy(sp)}
    return None
