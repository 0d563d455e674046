"""The work a user of tigerpm_b200 has it do, as cases that can be timed and compared.

A case names one call sequence of the public interface (tigerpm_b200.api) on one
synthetic box or ensemble.  prepare() makes the inputs and the context a program
would keep, run() is one pass, exact() the same results in 64 bits from plain torch.

Kinds:
  step    a whole PME kick of a resident box: restore the particles from device
          arrays, chain-mesh sort, long-range solve, interpolation + pair sum + kick
  sort    the chain-mesh sort alone (chainmesh_create)
  long    the long-range solve alone (gravity_long_compute) on a sorted box
  batch   an ensemble of boxes kicked together (Batch.step)
  host    a stream of boxes from and to pinned host memory (pme_steps_host)
"""
import math

import numpy as np
import torch

from tigerpm_b200.api import GRAVITY_LONG_PM, GRAVITY_LONG_PME, Batch, TigerPM, make_options
from tigerpm_b200.workloads import ParticleSet, accurate_box_params, fft_friendly, log_uniform_sides

# A big step shorter than any particle's own time step: every new rung is then
# whole whatever the rounding of the force, and velocities follow the forces
# continuously (a rung on a power-of-two boundary would double one half-kick).
SHORT = 1e-9


def _accurate(side):
    """The form that meets 1e-4 force error: cloud4, mesh >= 3 points per spacing, r_s = 2/3 spacing, cutoff 6 r_s."""
    p = accurate_box_params(side)
    return {"grid": p["grid"], "rs": p["rs_cells"], "rcut": p["rcut_over_rs"], "assign": p["assign"], "chain": 0}


def _literal(grid, assign):
    """Mesh = particle lattice, r_s = 1.25 cells, cutoff 4.5 r_s."""
    return {"grid": grid, "rs": 1.25, "rcut": 4.5, "assign": assign, "chain": 0}


def _reference(side):
    """The reference's own defaults: mesh = lattice / 3, chain mesh = mesh / 5, r_s = 1 cell, no cutoff."""
    return {"grid": side // 3, "rs": 1.0, "rcut": 0.0, "assign": "cloud4", "chain": side // 15}


def _step(dist, n, form, **more):
    c = {"kind": "step", "dist": dist, "n": n, "sort": "parity", "deposit": 0, "min_rung": 0, "first": True, "t0": SHORT}
    c.update(form)
    c.update(more)
    return c


def listed():
    return [
        # the headline configuration: 256^3 Zel'dovich box in the accurate form, 768^3 mesh
        _step("zeldovich", 256 ** 3, _accurate(256), name="headline 256^3"),
        # the same particles with the configuration's literal mesh parameters: more pairs, a small mesh
        _step("zeldovich", 256 ** 3, _literal(256, "tsc"), name="literal 256^3"),
        # the 64^3 configuration, with the rungs of a whole time unit
        _step("uniform", 64 ** 3, _literal(64, "cic"), t0=1.0, name="uniform 64^3"),
        # the smallest box of the served and batched pools, alone: launches and latency
        _step("zeldovich", 32 ** 3, _accurate(32), name="served 32^3"),
        # late times: most particles in halos, cells hundreds of times the mean
        _step("halos", 128 ** 3, _accurate(128), name="clustered 128^3"),
        # the reference's default options: 3,375 particles a chain cell, all pairs of 27 cells
        _step("uniform", 90 ** 3, _reference(90), name="reference options 90^3"),
        # one substep of a block time-step scheme: a quarter of the particles is due
        _step("zeldovich", 128 ** 3, _accurate(128), min_rung=2, first=False, name="active subset 128^3"),
        # a run that has to be repeatable bit for bit: integer deposit; a count that is no cube
        _step("uniform", 1234567, _accurate(107), deposit=2, name="repeatable 1.23M"),
        # re-sorting a box after its particles came in no order; an odd chain mesh
        {"kind": "sort", "dist": "uniform", "n": 7654321, "grid": 64, "rs": 1.0, "rcut": 0.0, "assign": "cloud4",
         "chain": 49, "sort": "parity", "name": "sort 7.65M"},
        # a particle-mesh code's own step: only the long-range field, on a mesh that is 16 x 25
        {"kind": "long", "dist": "zeldovich", "n": 200 ** 3, "grid": 400, "rs": 1.0, "rcut": 0.0, "assign": "tsc",
         "chain": 80, "deposit": 0, "pme": False, "name": "mesh field 400^3"},
        # the batched ensemble: boxes of many sizes kicked together
        {"kind": "batch", "boxes": 12, "lo": 32, "hi": 96, "name": "ensemble of 12"},
        # boxes that live in host memory: upload, kick, download, one after another
        {"kind": "host", "dist": "zeldovich", "n": 128 ** 3, **_accurate(128), "steps": 3, "name": "host stream 128^3"},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["step"] * 6 + ["literal", "literal", "halos", "reference", "subset", "sort", "long", "batch", "host"])
    deposit = rng.choice([0, 0, 1, 2])
    if kind == "step":
        side = _log(rng, 24, 240)
        n = side ** 3 if rng.random() < 0.5 else rng.randint(side ** 3 // 2, side ** 3)
        dist = "zeldovich" if n == side ** 3 else "uniform"
        return _step(dist, n, _accurate(side), deposit=deposit, sort=rng.choice(["parity", "parity", "fast"]))
    if kind == "literal":
        side = _log(rng, 24, 240)
        n = rng.randint(side ** 3 // 2, side ** 3)
        return _step("uniform", n, _literal(rng.choice([side, fft_friendly(side)]), rng.choice(["cic", "tsc", "cloud4"])),
                     deposit=deposit)
    if kind == "halos":
        side = _log(rng, 32, 112)
        return _step("halos", side ** 3, _accurate(side))
    if kind == "reference":
        side = 15 * rng.randint(3, 5)
        return _step("uniform", rng.randint(side ** 3 // 2, side ** 3), _reference(side))
    if kind == "subset":
        side = _log(rng, 32, 160)
        return _step("zeldovich", side ** 3, _accurate(side), min_rung=rng.randint(1, 3), first=False)
    if kind == "sort":
        n = _log(rng, 20000, 16000000)
        chain = max(3, round((n / rng.uniform(20, 300)) ** (1 / 3)))
        dist, order = rng.choice([("uniform", "parity"), ("halos", "parity"), ("uniform", "fast")])
        return {"kind": "sort", "dist": dist, "n": n, "grid": 64, "rs": 1.0, "rcut": 0.0, "assign": "cloud4",
                "chain": chain, "sort": order}
    if kind == "long":
        grid = _log(rng, 32, 700)
        if rng.random() < 0.7:
            grid = fft_friendly(grid)
        n = min(12000000, max(1000, int(grid ** 3 / rng.uniform(1, 27))))
        return {"kind": "long", "dist": "uniform", "n": n, "grid": grid, "rs": 1.25, "rcut": 0.0,
                "assign": rng.choice(["cic", "tsc", "cloud4"]), "chain": max(3, int(grid / rng.uniform(5, 12.5))),
                "deposit": deposit, "pme": rng.random() < 0.7}
    if kind == "batch":
        lo = _log(rng, 24, 48)
        return {"kind": "batch", "boxes": rng.randint(3, 16), "lo": lo, "hi": rng.randint(lo + 8, 100)}
    side = _log(rng, 32, 150)
    return {"kind": "host", "dist": "zeldovich", "n": side ** 3, **_accurate(side), "steps": rng.randint(2, 4)}


# ------------------------------------------------------------------ inputs
def _raw(pos):
    """fixed32 of (3, n) positions in box units, as the int32 tensors that hold the uint32 bits."""
    v = torch.floor((pos - torch.floor(pos)) * 4294967296.0).clamp_(max=4294967295.0).to(torch.int64)
    return torch.where(v >= 2 ** 31, v - 2 ** 32, v).to(torch.int32).contiguous()


def _zeldovich(side, g):
    """A lattice displaced by the Zel'dovich field of P(k) ~ k^-2 cut at k_Nyq / 2, rms 0.3 spacings."""
    dev = "cuda"
    dk = torch.fft.rfftn(torch.randn((side, side, side), generator=g, device=dev))
    k = torch.fft.fftfreq(side, device=dev) * side
    kz = torch.fft.rfftfreq(side, device=dev) * side
    k2 = k[:, None, None] ** 2 + k[None, :, None] ** 2 + kz[None, None, :] ** 2
    k2[0, 0, 0] = 1.0
    dk *= torch.exp(-torch.sqrt(k2) / (0.5 * side)) / torch.sqrt(k2) / k2
    dk[0, 0, 0] = 0
    disp = torch.stack([torch.fft.irfftn(1j * K * dk, s=(side,) * 3) for K in
                        (k[:, None, None], k[None, :, None], kz[None, None, :])])
    disp *= 0.3 / side / torch.sqrt((disp * disp).sum(0).mean())
    q = (torch.arange(side, device=dev, dtype=torch.float64) + 0.5) / side
    pos = torch.empty((3, side, side, side), dtype=torch.float64, device=dev)
    pos[0], pos[1], pos[2] = q[:, None, None], q[None, :, None], q[None, None, :]
    return (pos + disp).reshape(3, -1)


def _halos(n, g):
    """70 % of the particles in NFW halos (masses log-uniform over three decades, c in 5..15), the rest uniform."""
    dev = "cuda"
    nh, nhalo = int(0.7 * n), max(8, int(2000 * n / 256 ** 3))
    w = torch.exp(torch.rand(nhalo, generator=g, device=dev, dtype=torch.float64) * math.log(1000.0))
    hid = torch.searchsorted(torch.cumsum(w, 0) / w.sum(), torch.rand(nh, generator=g, device=dev, dtype=torch.float64))
    hid = hid.clamp_(max=nhalo - 1)
    centre = torch.rand((3, nhalo), generator=g, device=dev, dtype=torch.float64)
    conc = (5 + 10 * torch.rand(nhalo, generator=g, device=dev, dtype=torch.float64))[hid]
    r200 = ((w / w.sum() * nh) * 3 / (800 * math.pi * n)) ** (1 / 3)
    mu = lambda s: torch.log1p(s) - s / (1 + s)  # noqa: E731
    u = torch.rand(nh, generator=g, device=dev, dtype=torch.float64) * mu(conc)
    lo, hi = torch.zeros_like(conc), conc.clone()
    for _ in range(45):
        s = 0.5 * (lo + hi)
        below = mu(s) < u
        lo, hi = torch.where(below, s, lo), torch.where(below, hi, s)
    v = torch.randn((3, nh), generator=g, device=dev, dtype=torch.float64)
    v *= (0.5 * (lo + hi) / conc * r200[hid]) / torch.linalg.vector_norm(v, dim=0)
    return torch.cat([centre[:, hid] + v, torch.rand((3, n - nh), generator=g, device=dev, dtype=torch.float64)], 1)


def _particles(dist, n, seed, moving):
    """Device particle arrays x, y, z, vx, vy, vz, rung."""
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1000003 + n)
    if dist == "zeldovich":
        pos = _zeldovich(round(n ** (1 / 3)), g)
    elif dist == "halos":
        pos = _halos(n, g)
    else:
        pos = torch.rand((3, n), generator=g, device="cuda", dtype=torch.float64)
    raw = _raw(pos)
    if moving:  # half the particles on rung 0, a quarter on rung 1, ...
        v = torch.randn((3, n), generator=g, device="cuda") * 1e-3
        u = torch.rand(n, generator=g, device="cuda")
        rung = torch.floor(-torch.log2(u.clamp_(min=1e-9))).clamp_(max=6).to(torch.int8)
    else:
        v = torch.zeros((3, n), device="cuda")
        rung = torch.zeros(n, dtype=torch.int8, device="cuda")
    return [raw[0], raw[1], raw[2], v[0], v[1], v[2], rung]


def _moving(case):
    return not case.get("first", True) or case["kind"] == "sort"


def _options(case):
    return make_options(max(2, round(case["n"] ** (1 / 3))), case["grid"], chain=case["chain"] or None, rs_cells=case["rs"],
                        rcut_over_rs=case["rcut"], assign=case["assign"], sort=case.get("sort", "parity"),
                        deterministic_deposit=case.get("deposit", 0))


class _Span:
    """A device array of a context for torch; keeps the context alive."""

    def __init__(self, owner, ptr, count, typestr):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": typestr, "data": (ptr, False), "version": 2}


class _Views:
    """Tensors over a context's arrays, made once per address (the sort swaps two sets of them)."""

    TYPES = {"x": "<i4", "y": "<i4", "z": "<i4", "vx": "<f4", "vy": "<f4", "vz": "<f4", "rung": "|i1", "gx": "<f4",
             "gy": "<f4", "gz": "<f4", "pot": "<f4", "cell_begin": "<i4", "phi": "<f4"}

    def __init__(self, ctx, owner):
        self.ctx, self.owner, self.made = ctx, owner, {}

    def __call__(self, fields):
        d, out = self.ctx.device_arrays(), {}
        for f in fields:
            ptr = getattr(d, f)
            if ptr not in self.made:
                o = self.ctx.opts
                count = {"cell_begin": o.chain_dim ** 3 + 1, "phi": o.four_dim ** 3}.get(f, d.n)
                self.made[ptr] = torch.as_tensor(_Span(self.owner, ptr, count, self.TYPES[f]), device="cuda")
            out[f] = self.made[ptr]
        return out


KICKED = ("x", "y", "z", "vx", "vy", "vz", "rung", "gx", "gy", "gz", "pot")
SORTED = ("x", "y", "z", "vx", "vy", "vz", "rung", "cell_begin")


def _boxes(case, seed):
    """(sides, options) of an ensemble; the sides belong to the case, the particles to the seed."""
    sides = [int(s) for s in log_uniform_sides(case["boxes"], case["lo"], case["hi"], 4)]
    return sides, [_options({"n": s ** 3, **_accurate(s)}) for s in sides]


def prepare(case, seed):
    s = {"case": case}
    if case["kind"] == "batch":
        sides, opts = _boxes(case, seed)
        b = Batch(opts, [n ** 3 for n in sides])
        for i, n in enumerate(sides):
            b.set_input(i, _host(_particles("zeldovich", n ** 3, seed * 100 + i, False)))
        s["batch"], s["stream"] = b, torch.cuda.ExternalStream(b.stream())
        s["arrays"] = [_Views(b.box(i), b)(KICKED) for i in range(len(sides))]
    elif case["kind"] == "host":
        s["ctx"] = TigerPM(_options(case), case["n"])
        s["in"], s["out"], s["tensors"] = [], [], []
        for k in range(case["steps"]):
            src = [t.cpu().pin_memory() for t in _particles(case["dist"], case["n"], seed * 100 + k, False)]
            dst = [torch.empty_like(t).pin_memory() for t in src]
            s["in"].append(_set(src))
            s["out"].append(_set(dst))
            s["tensors"].append((src, dst))
    else:
        s["ctx"] = TigerPM(_options(case), case["n"])
        s["parts"] = _particles(case["dist"], case["n"], seed, _moving(case))
        s["ptrs"] = [t.data_ptr() for t in s["parts"]]
        s["views"] = _Views(s["ctx"], s["ctx"])
        if case["kind"] == "long":
            torch.cuda.synchronize()
            s["ctx"].set_particles_device(case["n"], s["ptrs"])
            s["ctx"].chainmesh_create()
            s["ctx"].synchronize()
    torch.cuda.synchronize()
    return s


def _set(tensors):
    a = [t.numpy() for t in tensors]
    return ParticleSet(*(v.view(np.uint32) for v in a[:3]), *a[3:])


def _host(tensors):
    return _set([t.cpu() for t in tensors])


def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "step":
        ctx = s["ctx"]
        ctx.set_particles_device(case["n"], s["ptrs"])
        ctx.pme_step(case["min_rung"], 1.0, case["t0"], case["first"])
        return s["views"](KICKED)
    if kind == "sort":
        ctx = s["ctx"]
        ctx.set_particles_device(case["n"], s["ptrs"])
        ctx.chainmesh_create()
        return s["views"](SORTED)
    if kind == "long":
        s["ctx"].gravity_long_compute(GRAVITY_LONG_PME if case["pme"] else GRAVITY_LONG_PM)
        return s["views"](("phi",))
    if kind == "batch":
        s["batch"].step(restore=True, graph=True, t0=SHORT)
        with torch.cuda.stream(s["stream"]):  # the ensemble's particles as one array per field
            return {f: torch.cat([a[f] for a in s["arrays"]]) for f in KICKED}
    s["ctx"].pme_steps_host(s["in"], s["out"], t0=SHORT)
    return [dict(zip(KICKED, dst)) for _, dst in s["tensors"]]


# -------------------------------------------------------------------- work
def _pairs(n, grid, rs, rcut, chain):
    """Sink-source pairs of a box that is even in the mean (fewer than a clustered one has)."""
    volume = 4.0 / 3.0 * math.pi * (rcut * rs / grid) ** 3 if rcut > 0 else 27.0 / chain ** 3
    return float(n) * n * min(1.0, volume)


def _mesh_flops(grid):
    return 2 * 2.5 * grid ** 3 * math.log2(grid ** 3)  # real transforms, there and back


def _step_work(c):
    active = 0.5 ** c.get("min_rung", 0)
    flops = active * 44 * _pairs(c["n"], c["grid"], c["rs"], c["rcut"], c["chain"]) + _mesh_flops(c["grid"]) + 700 * c["n"]
    return {"bytes": c["n"] * (25 + 41), "flops": flops}  # particles in, particles and forces out


def work(case):
    if case["kind"] == "sort":
        return {"bytes": case["n"] * 50 + 4 * case["chain"] ** 3, "flops": 0}
    if case["kind"] == "long":
        return {"bytes": case["n"] * 12 + 4 * case["grid"] ** 3, "flops": _mesh_flops(case["grid"]) + 200 * case["n"]}
    if case["kind"] == "batch":
        sides, _ = _boxes(case, 0)
        w = [_step_work({"n": s ** 3, **_accurate(s)}) for s in sides]
        return {k: sum(v[k] for v in w) for k in ("bytes", "flops")}
    if case["kind"] == "host":
        w = _step_work(case)
        return {"bytes": case["steps"] * case["n"] * 50, "flops": case["steps"] * w["flops"]}
    return _step_work(case)


def tolerance(case):
    if case["kind"] == "sort":
        return "exact"
    if case.get("t0") == 1.0:
        # a rung on its power-of-two boundary doubles one half-kick: rel ~ 1 / sqrt(n) a particle
        return {"rel": 3e-3, "max": 0.99, "differ": 1e-4}
    if case["kind"] == "batch" or case["dist"] == "zeldovich":
        # forces of a near-lattice box are small differences of the mesh potential, whose FP32 rounding they
        # carry: against 64 bits 3e-6 at 32^3, 1.3e-5 at 128^3; two runs (sums in another order) 2.7e-5 at 256^3
        side = case["hi"] if case["kind"] == "batch" else case["n"] ** (1 / 3)
        return {"rel": 1e-5 + 4e-7 * side, "max": 1e-3, "differ": 1e-4}
    # against 64 bits 2e-7 to 5.3e-6
    return {"rel": 2e-5, "max": 1e-3, "differ": 1e-4}


# ------------------------------------------------------- 64-bit references
def _u32(t):
    return t.to(torch.int64) & 0xFFFFFFFF


def _partition(raw, C, fast):
    """The chain-mesh order: (permutation, cell of each sorted position, cell offsets).  The box is bisected along z,
    then y, then x; each node's range is partitioned in place by the two-pointer pass that swaps the i-th misplaced
    element from the left with the i-th from the right."""
    dev = raw[0].device
    thr = torch.tensor([int(4294967296.0 * (m * (1.0 / C))) for m in range(C)], device=dev)
    cell = [torch.searchsorted(thr, r, right=True) - 1 for r in raw]
    key = (cell[2] * C + cell[1]) * C + cell[0]
    offs = torch.zeros(C ** 3 + 1, dtype=torch.int64, device=dev)
    offs[1:] = torch.cumsum(torch.bincount(key, minlength=C ** 3), 0)
    n = key.numel()
    if fast:
        return torch.argsort(key, stable=True), None, offs
    at = torch.repeat_interleave(torch.arange(C ** 3, device=dev), offs[1:] - offs[:-1])  # final cell of each position
    perm = torch.arange(n, device=dev)
    p = torch.arange(n, device=dev)
    span = [[] for _ in range(C)]
    for c in range(C):
        lo, hi = 0, C
        while hi - lo > 1:
            mid = lo + (hi - lo) // 2
            span[c].append((lo, mid, hi))
            lo, hi = (lo, mid) if c < mid else (mid, hi)
    for unit in (C * C, C, 1):
        here = at // unit % C
        base = at // (unit * C) * (unit * C)
        for level in range(max(len(t) for t in span)):
            tab = torch.tensor([t[level] if level < len(t) else (c, c + 1, c + 1) for c, t in enumerate(span)], device=dev)
            lo, mid, hi = (offs[base + tab[here, k] * unit] for k in range(3))
            left = (key[perm] // unit % C < tab[here, 1]).to(torch.int64)
            before = torch.zeros(n + 1, dtype=torch.int64, device=dev)
            before[1:] = torch.cumsum(left, 0)
            a = (p < mid) & (left == 0)
            b = (p >= mid) & (left == 1)
            pa, pb = p[a], p[b]
            ia = lo[a] + (pa - lo[a]) - (before[pa] - before[lo[a]])
            ib = lo[b] + before[hi[b]] - before[pb] - 1
            slot = torch.empty(n, dtype=torch.int64, device=dev)
            slot[ib] = pb
            pb = slot[ia]
            perm[pa], perm[pb] = perm[pb], perm[pa]
    return perm, at, offs


def _weights(f, assign):
    if assign == "cloud4":
        g = 1 - f
        return [g ** 3 / 6, (4 - 6 * f * f + 3 * f ** 3) / 6, (4 - 6 * g * g + 3 * g ** 3) / 6, f ** 3 / 6]
    if assign == "cic":
        return [1 - f, f]
    d = f - (f >= 0.5).to(f.dtype)
    return [0.5 * (0.5 - d) ** 2, 0.75 - d * d, 0.5 * (0.5 + d) ** 2]


def _potential(raw, case, pme):
    N, dev = case["grid"], raw[0].device
    rho = torch.zeros(N ** 3, dtype=torch.float64, device=dev)
    start, w = [], []
    for r in raw:
        t = r * N
        f = (t & 0xFFFFFFFF).double() / 4294967296.0
        first = (t >> 32) - (0 if case["assign"] == "cic" else 1)
        if case["assign"] == "tsc":
            first = first + (f >= 0.5).to(torch.int64)
        start.append(first)
        w.append(_weights(f, case["assign"]))
    for i in range(len(w[0])):
        for j in range(len(w[0])):
            row = ((start[0] + i) % N * N + (start[1] + j) % N) * N
            for k in range(len(w[0])):
                rho.index_add_(0, row + (start[2] + k) % N, w[0][i] * w[1][j] * w[2][k])
    spec = torch.fft.rfftn((rho * (4 * math.pi * N)).view(N, N, N))
    i = torch.arange(N, device=dev, dtype=torch.float64)
    k = torch.where(i < N / 2, i, i - N) * (2 * math.pi / N)
    order = {"cic": 2, "tsc": 3, "cloud4": 4}[case["assign"]]
    sinc = torch.where(k == 0, torch.ones_like(k), torch.sin(0.5 * k) / torch.where(k == 0, torch.ones_like(k), 0.5 * k))
    g = sinc ** -order * (torch.exp(-k * k * case["rs"] ** 2) if pme else 1.0)
    h = N // 2 + 1
    k2 = (k * k)[:, None, None] + (k * k)[None, :, None] + (k * k)[None, None, :h]
    k2[0, 0, 0] = 1.0
    spec *= -(g[:, None, None] * g[None, :, None] * g[None, None, :h]) / k2
    spec[0, 0, 0] = 0
    return torch.fft.irfftn(spec, s=(N, N, N)).reshape(-1)


def _quintic(x):
    c = [[0, 1 / 12, -1 / 24, -3 / 8, 13 / 24, -5 / 24], [0, -2 / 3, 2 / 3, 13 / 8, -8 / 3, 25 / 24],
         [1, 0, -5 / 4, -35 / 12, 21 / 4, -25 / 12], [0, 2 / 3, 2 / 3, 11 / 4, -31 / 6, 25 / 12],
         [0, -1 / 12, -1 / 24, -11 / 8, 61 / 24, -25 / 24], [0, 0, 0, 7 / 24, -1 / 2, 5 / 24]]
    return ([sum(a * x ** m for m, a in enumerate(r) if a) for r in c],
            [sum(m * a * x ** (m - 1) for m, a in enumerate(r) if a and m) for r in c])


def _long_range(phi, raw, N):
    """(3, n) force and (n) potential of the mesh at the particles, 6-point quintic."""
    out = []
    for lo in range(0, raw[0].numel(), 1 << 20):
        w, dw, base = [], [], []
        for r in raw:
            t = r[lo:lo + (1 << 20)] * N
            a, b = _quintic((t & 0xFFFFFFFF).double() / 4294967296.0)
            w.append(a)
            dw.append(b)
            base.append((t >> 32) - 2)
        s = torch.zeros((4, base[0].numel()), dtype=torch.float64, device=phi.device)
        for i in range(6):
            for j in range(6):
                row = ((base[0] + i) % N * N + (base[1] + j) % N) * N
                v = [phi[row + (base[2] + k) % N] for k in range(6)]
                z = sum(a * b for a, b in zip(w[2], v))
                dz = sum(a * b for a, b in zip(dw[2], v))
                s += torch.stack([-N * dw[0][i] * w[1][j] * z, -N * w[0][i] * dw[1][j] * z, -N * w[0][i] * w[1][j] * dz,
                                  w[0][i] * w[1][j] * z])
        out.append(s)
    out = torch.cat(out, 1)
    return out[:3], out[3]


def _pair_sums(raw, offs, C, opts):
    """(3, n) force and (n) potential of the short-range pair sum, or None where it would take too long."""
    dev, n = raw[0].device, raw[0].numel()
    count = offs[1:] - offs[:-1]
    most = int(count.max())
    if 27.0 * C ** 3 * most * most > 1.5e10:
        return None, None
    rcut = opts.rcut_over_rs * opts.rs if opts.rcut_over_rs > 0 else 1e9
    h, inv2rs = opts.hsoft, 0.5 / opts.rs
    slot = torch.arange(most, device=dev)
    have = slot[None, :] < count[:, None]
    index = torch.where(have, offs[:-1, None] + slot[None, :], 0)
    pos = torch.stack([r.double() / 4294967296.0 for r in raw])
    g = torch.zeros((3, n), dtype=torch.float64, device=dev)
    ph = torch.zeros(n, dtype=torch.float64, device=dev)
    cells = torch.arange(C ** 3, device=dev)
    step = max(1, int(2e7) // (most * most))
    for lo in range(0, C ** 3, step):
        mine = cells[lo:lo + step]
        x, y, z = mine % C, mine // C % C, mine // (C * C)
        i0, m0 = index[mine], have[mine]
        for d in range(27):
            near = ((z + d // 9 - 1) % C * C + (y + d // 3 % 3 - 1) % C) * C + (x + d % 3 - 1) % C
            i1, m1 = index[near], have[near]
            r2 = None
            for k in range(3):
                dx = pos[k][i0][:, :, None] - pos[k][i1][:, None, :]
                dx -= torch.round(dx)
                r2 = dx * dx if r2 is None else r2.addcmul_(dx, dx)
            a, b, c = torch.nonzero((r2 < rcut * rcut) & m0[:, :, None] & m1[:, None, :], as_tuple=True)
            r2 = r2[a, b, c]
            sink, source = i0[a, b], i1[a, c]
            r = torch.sqrt(r2)
            x0 = r * inv2rs
            t = 1 / (1 + 0.3275911 * x0)  # Abramowitz and Stegun 7.1.26, the method's own erfc
            e = torch.exp(-x0 * x0)
            erfc = t * (0.254829592 + t * (-0.284496736 + t * (1.421413741 + t * (-1.453152027 + t * 1.061405429)))) * e
            q2 = r2 / (h * h)
            soft = r <= h
            f = torch.where(soft, (35 / 8 - 21 / 4 * q2 + 15 / 8 * q2 * q2) / h ** 3,
                            (erfc + 2 / math.sqrt(math.pi) * x0 * e) / (r2 * r))
            p = torch.where(soft, (35 / 16 - 35 / 16 * q2 + 21 / 16 * q2 ** 2 - 5 / 16 * q2 ** 3) / h, erfc / r)
            ph.index_add_(0, sink, -p)
            for k in range(3):
                dx = pos[k][sink] - pos[k][source]
                g[k].index_add_(0, sink, -(dx - torch.round(dx)) * f)
    return g, ph


def _kicked(case, parts):
    """What a step leaves of one box, in 64 bits; None for whole numbers and where the pair sum would take too long."""
    opts = _options(case)
    raw = [_u32(t) for t in parts[:3]]
    perm, _, offs = _partition(raw, opts.chain_dim, case.get("sort") == "fast")
    raw = [r[perm] for r in raw]
    v, rung = [t[perm].double() for t in parts[3:6]], parts[6][perm].to(torch.int64)
    g, pot = _pair_sums(raw, offs, opts.chain_dim, opts)
    if g is None:
        return None
    gl, pl = _long_range(_potential(raw, case, True), raw, case["grid"])
    due = rung >= case.get("min_rung", 0)
    g, pot = (g + gl) * opts.GM * due, (pot + pl) * opts.GM * due
    out = {f: None for f in KICKED}
    out.update(gx=g[0], gy=g[1], gz=g[2], pot=pot)
    t0 = case.get("t0", SHORT)
    if t0 == SHORT:
        half = 0.5 * t0 * torch.pow(2.0, -rung.double())
        later = 0.5 * t0 * torch.pow(2.0, -(rung - 1).clamp(min=0).double())
        dt = (later if case.get("first", True) else half + later) * due
        out.update({f: a + b * dt for f, a, b in zip(("vx", "vy", "vz"), v, g)})
    return out


def exact(case, seed):
    if case["kind"] == "batch":
        sides, _ = _boxes(case, seed)
        boxes = [_kicked({"n": s ** 3, **_accurate(s)}, _particles("zeldovich", s ** 3, seed * 100 + i, False))
                 for i, s in enumerate(sides)]
        if any(b is None for b in boxes):
            return None
        return {f: None if boxes[0][f] is None else torch.cat([b[f] for b in boxes]) for f in KICKED}
    if case["kind"] == "host":
        sets = [_particles(case["dist"], case["n"], seed * 100 + k, False) for k in range(case["steps"])]
        boxes = [_kicked(case, p) for p in sets]
        return None if boxes[0] is None else [{f: b[f] for f in KICKED[:7]} for b in boxes]
    parts = _particles(case["dist"], case["n"], seed, _moving(case))
    if case["kind"] == "step":
        return _kicked(case, parts)
    raw = [_u32(t) for t in parts[:3]]
    if case["kind"] == "long":
        return {"phi": _potential(raw, case, case["pme"])}
    perm, _, offs = _partition(raw, case["chain"], case["sort"] == "fast")
    out = {f: t[perm] for f, t in zip(SORTED, parts)}
    out["cell_begin"] = offs.to(torch.int32)
    return out
