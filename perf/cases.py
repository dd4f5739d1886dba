"""Cases of the simulation step at the sizes its users run it: the step's stages through the C ABI
(`olc_stage_*`: diffusion of one field in each storage type, contact, the key sort), and whole steps of a
solo engine and of a batch.

Every state is made from the seed alone.  A pass continues from the state the previous one left, as a
simulation does.  The populations grow slowly (doubling in about 100 days, a slow solid tumour) and no drug
dose is lethal, so a long run keeps its size with births, uptake and contact in the path; the columns come at
their full capacity, whose rows past the population are zero.
"""
import ctypes as C
import math
from types import SimpleNamespace

import numpy as np
import torch

from oncolytica_b200 import _lib
from oncolytica_b200 import workloads as W

DEV = "cuda"
STORAGE = {"f32": (0, torch.float32), "bf16": (1, torch.bfloat16), "f16": (2, torch.float16),
           "bf16_sr": (3, torch.bfloat16), "f16_sr": (4, torch.float16)}
GROWTH = 2.9e-4   # 1/h: ln 2 / 2400 h
STIFFNESS, MOBILITY, MAX_DISP, MARGIN, DT = 1.0, 10.0, 1.0, 0.1, 0.1


def listed():
    return [
        # a whole step of the small configuration (10,000 agents, one 64^3 field), metrics read each step:
        # the smallest simulation in use, where launches and latency count
        dict(name="engine_small", kind="engine", agents=10_000, grid=64, storage="f32", drug=False, graphs=False),
        # a whole step of the large configuration (1,000,000 agents, two 256^3 fields), as CUDA graphs
        dict(name="engine_scale", kind="engine", agents=1_000_000, grid=256, storage="f32", drug=True, graphs=True),
        # 16 members of a parameter sweep in one batch, FP16 fields with stochastic rounding (the sweep's form)
        dict(name="batch_sweep", kind="batch", members=16, storage="f16_sr"),
        # one step of one O2 field of the small configuration: 79 substeps, uptake deposited by 10,000 agents
        dict(name="diffuse_small", kind="diffuse", nx=64, ny=64, nz=64, substeps=79, storage="f32",
             encoding=0, decay=0.0, uptakes=10_000),
        # a sweep member's O2 field (96^3)
        dict(name="diffuse_mid", kind="diffuse", nx=96, ny=96, nz=96, substeps=88, storage="f32",
             encoding=0, decay=0.0, uptakes=40_000),
        # a tissue sample of no round size: rows that are no multiple of 16 bytes
        dict(name="diffuse_odd", kind="diffuse", nx=117, ny=75, nz=131, substeps=21, storage="f32",
             encoding=0, decay=0.1, uptakes=0),
        # the drug field of the large configuration: 21 substeps with decay, no uptake
        dict(name="diffuse_large", kind="diffuse", nx=256, ny=256, nz=256, substeps=21, storage="f32",
             encoding=0, decay=0.1, uptakes=0),
        # a 128^3 sweep field stored as FP16 with stochastic rounding
        dict(name="diffuse16_f16", kind="diffuse", nx=128, ny=128, nz=128, substeps=79, storage="f16_sr",
             encoding=0, decay=0.1, uptakes=100_000),
        # the large configuration's drug field stored as BF16 with its default encoding (three offsets)
        dict(name="diffuse16_bf16", kind="diffuse", nx=256, ny=256, nz=256, substeps=21, storage="bf16_sr",
             encoding=2, decay=0.1, uptakes=0),
        # the contact pass of the large configuration
        dict(name="contact_large", kind="contact", agents=1_000_000, r_lo=4.0, r_hi=6.0, crowding=1.0),
        # a small population's key sort (random order: a first step)
        dict(name="sort_small", kind="sort", n=10_007, bits=16, disorder=1.0),
        # a large batch's key sort: nearly sorted rows with this step's moves
        dict(name="sort_large", kind="sort", n=4_000_000, bits=30, disorder=0.05),
    ]


def draw(rng):
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["diffuse", "diffuse", "diffuse", "diffuse16", "diffuse16", "contact", "sort", "engine"])
    if kind in ("diffuse", "diffuse16"):
        f32 = kind == "diffuse"
        nx, ny, nz = (log_int(20, 256) for _ in range(3))
        if not f32:
            nx = max(24, nx // 8 * 8)
        elif rng.random() < 0.6:
            nx = max(20, nx // 4 * 4)
        most = max(3, min(120, int(21 * 256 ** 3 / (nx * ny * nz))))
        storage = "f32" if f32 else rng.choice(["bf16_sr", "f16_sr", "f16", "bf16"])
        # BF16 keeps three offsets, FP16 values: what storage= alone gives
        return dict(kind="diffuse", nx=nx, ny=ny, nz=nz, substeps=rng.randint(3, most), storage=storage,
                    encoding=2 if storage.startswith("bf16") else 0, decay=rng.choice([0.0, 0.1]),
                    uptakes=rng.choice([0, log_int(100, min(100_000, nx * ny * nz // 8))]))
    if kind == "contact":
        return dict(kind="contact", agents=log_int(1_000, 1_000_000), r_lo=4.0, r_hi=rng.choice([4.5, 6.0]),
                    crowding=round(rng.uniform(0.4, 1.8), 3))
    if kind == "sort":
        return dict(kind="sort", n=log_int(500, 4_000_000), bits=rng.randint(9, 30), disorder=rng.choice([1.0, 0.05]))
    grid, drug = rng.choice([32, 48, 64, 96, 128]), rng.random() < 0.7
    return dict(kind="engine", agents=log_int(1_000, min(100_000, int(_density(drug) * (1.6 * grid) ** 3 * 4.18))),
                grid=grid, storage=rng.choice(["f32", "f16_sr", "bf16_sr"]), drug=drug, graphs=rng.random() < 0.5)


# ---------------------------------------------------------------- one field through its stage entry point
# D dt / (S dx^2) = 0.152: the default margin above the stability bound
def _spec(case):
    d = _lib.OlcDiffusion()
    d.diffusion = 0.152 * case["substeps"] / DT
    d.decay = case["decay"]
    d.boundary = 1.0
    d.substeps = case["substeps"]
    d.has_sink = int(case["uptakes"] > 0)
    d.storage = STORAGE[case["storage"]][0]
    d.encoding = case["encoding"]
    return d


def _field(case, seed):
    """A field in mid-run, [z, y, x] in double: a depleted core under its boundary value plus local variation."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    ax = [torch.linspace(-1, 1, n, device=DEV, dtype=torch.float64) for n in (nz, ny, nx)]
    r2 = ax[0][:, None, None] ** 2 + ax[1][None, :, None] ** 2 + ax[2][None, None, :] ** 2
    f = (0.15 + 0.8 * (r2 / 3.0).sqrt()).clamp_(0.0, 0.98)
    f += 0.04 * (torch.rand(f.shape, generator=g, device=DEV, dtype=torch.float64) - 0.5)
    f[0], f[-1], f[:, 0], f[:, -1], f[:, :, 0], f[:, :, -1] = 1, 1, 1, 1, 1, 1
    idx = torch.empty(0, dtype=torch.int64, device=DEV)
    rate = torch.empty(0, dtype=torch.float32, device=DEV)
    if case["uptakes"]:
        idx = torch.randperm(nx * ny * nz, generator=g, device=DEV)[:case["uptakes"]].sort().values
        rate = 0.01 + 0.1 * torch.rand(case["uptakes"], generator=g, device=DEV, dtype=torch.float32)
    return f, idx, rate


def _bits(f, encoding, dtype):
    """The elements a host program uploads: values, or distances to the nearest of 0, 1/2 and 1 under two flag bits."""
    f = f.to(torch.float32)
    if encoding == 0:
        return f.to(dtype)
    low, high = f < 0.25, f > 0.75
    d = f - 0.5
    mag = torch.where(low, f, torch.where(high, 1.0 - f, d.abs())).to(dtype).view(torch.int16).to(torch.int32)
    code = torch.where(low, 0, torch.where(high, 0xC000, torch.where(d < 0, 0x8000, 0x4000)))
    w = mag | code
    return torch.where(w >= 0x8000, w - 0x10000, w).to(torch.int16).view(dtype)


def _prepare_diffuse(case, seed):
    f, idx, rate = _field(case, seed)
    dtype = STORAGE[case["storage"]][1]
    s = SimpleNamespace(kind="diffuse", lib=_lib.load(), step=0, f16=dtype != torch.float32, case=case)
    s.f = f.to(dtype).contiguous() if not s.f16 else _bits(f, case["encoding"], dtype).contiguous()
    s.tmp = torch.zeros_like(s.f)
    s.sink = torch.zeros(f.shape, dtype=torch.float32, device=DEV) if case["uptakes"] else None
    s.comp = torch.zeros(f.shape, dtype=torch.float32, device=DEV) if s.f16 else None
    s.idx, s.rate = idx, rate
    s.spec = _spec(case)
    s.dims = (C.c_int32 * 3)(case["nx"], case["ny"], case["nz"])
    return s


def _ptr(t):
    return C.c_void_p(t.data_ptr()) if t is not None else None


def _stream():
    return C.c_void_p(torch.cuda.current_stream().cuda_stream)


def _run_diffuse(s):
    if s.sink is not None:  # the agents' uptake of this step
        s.sink.view(-1).index_copy_(0, s.idx, s.rate)
    if s.f16:
        rc = s.lib.olc_stage_diffuse16(_ptr(s.f), _ptr(s.tmp), _ptr(s.sink), _ptr(s.comp), C.byref(s.dims), 1.0, DT,
                                       C.byref(s.spec), s.step, 0, _stream())
        s.step += 1
        _lib.check(rc)
        return [s.f.view(torch.int16) if s.case["encoding"] else s.f, s.comp]
    _lib.check(s.lib.olc_stage_diffuse(_ptr(s.f), _ptr(s.tmp), _ptr(s.sink), C.byref(s.dims), 1.0, DT,
                                       C.byref(s.spec), _stream()))
    return [s.f]


def _exact_diffuse(case, seed):
    if case["encoding"]:
        return None  # flagged bit patterns, equal or not
    f, idx, rate = _field(case, seed)
    dtype = STORAGE[case["storage"]][1]
    f = f.to(torch.float32).to(dtype).double()
    spec = _spec(case)
    r = float(spec.diffusion) * DT / case["substeps"]
    inv = 1.0 / (1.0 + float(spec.decay) * DT / case["substeps"])
    if case["uptakes"]:
        k = torch.zeros(f.numel(), dtype=torch.float64, device=DEV)
        k[idx] = rate.double()
        k = k.view(f.shape)[1:-1, 1:-1, 1:-1]
        f[1:-1, 1:-1, 1:-1] /= 1.0 + k * DT
    for _ in range(case["substeps"]):
        c = f[1:-1, 1:-1, 1:-1]
        s = f[1:-1, 1:-1, :-2] + f[1:-1, 1:-1, 2:]
        s += f[1:-1, :-2, 1:-1]
        s += f[1:-1, 2:, 1:-1]
        s += f[:-2, 1:-1, 1:-1]
        s += f[2:, 1:-1, 1:-1]
        s -= 6.0 * c
        f = f.clone()
        f[1:-1, 1:-1, 1:-1] = ((c + r * s) * inv).clamp_(min=0.0)
    return [f, None] if dtype != torch.float32 else [f]


# ---------------------------------------------------------------- contact over sorted agents
def _morton(cx, cy, cz):
    """Bin keys: the Morton key of the coarse coordinate above the three parity bits."""
    k = torch.zeros_like(cx)
    for b in range(9):
        for a, c in enumerate((cx, cy, cz)):
            k |= ((c >> (b + 1)) & 1) << (3 * b + 3 + a)
    return k | (cx & 1) | ((cy & 1) << 1) | ((cz & 1) << 2)


def _agents(case, seed):
    """Agents uniform in a ball, in bin-key order: (x, y, z, radius), bin coordinates, keys, bins per axis."""
    g = torch.Generator(device=DEV).manual_seed(seed)
    n = case["agents"]
    # crowding 1: the large configuration's 1e6 agents in a ball of radius 400 um
    ball = 400.0 * (n / 1e6 / case["crowding"]) ** (1.0 / 3.0)
    nb = max(4, int(math.ceil(2.5 * ball / 10.0)))
    nb = min(nb + nb % 2, 240)
    v = torch.randn(n, 3, generator=g, device=DEV)
    u = torch.rand(n, 1, generator=g, device=DEV)
    pos = nb * 5.0 + ball * u ** (1.0 / 3.0) * v / v.norm(dim=1, keepdim=True)
    rad = case["r_lo"] + (case["r_hi"] - case["r_lo"]) * torch.rand(n, 1, generator=g, device=DEV)
    posr = torch.cat([pos, rad], 1).float()
    c = (posr[:, :3] / 10.0).to(torch.int64).clamp_(0, nb - 1)
    key = _morton(c[:, 0], c[:, 1], c[:, 2])
    order = torch.sort(key, stable=True).indices
    return posr[order].contiguous(), c[order], key[order], nb


def _prepare_contact(case, seed):
    posr, _, key, nb = _agents(case, seed)
    s = SimpleNamespace(kind="contact", lib=_lib.load(), n=case["agents"], posr=posr)
    e = torch.full((3,), nb, dtype=torch.int64, device=DEV)
    table = int(_morton(e[:1], e[1:2], e[2:])[0])
    lo = torch.searchsorted(key, torch.arange(table, device=DEV))
    hi = torch.searchsorted(key, torch.arange(table, device=DEV), right=True)
    empty = hi == lo
    s.ranges = torch.stack([lo.masked_fill(empty, 0), hi.masked_fill(empty, 0)], 1).to(torch.int32).contiguous()
    s.geom = _lib.OlcGeom()
    s.geom.tissue_dims[:] = (nb, nb, nb)
    s.geom.tissue_voxel_size = 10.0
    s.geom.domain_hi[:] = (10.0 * nb,) * 3
    s.spec = _lib.OlcContact()
    s.spec.enabled, s.spec.radius_field = 1, 3
    s.spec.stiffness, s.spec.mobility, s.spec.max_disp, s.spec.margin = STIFFNESS, MOBILITY, MAX_DISP, MARGIN
    s.out = [torch.zeros(s.n, device=DEV) for _ in range(3)]
    return s


def _run_contact(s):
    _lib.check(s.lib.olc_stage_contact(_ptr(s.posr), _ptr(s.ranges), s.n, C.byref(s.geom), C.byref(s.spec), DT,
                                       _ptr(s.out[0]), _ptr(s.out[1]), _ptr(s.out[2]), _stream()))
    return list(s.out)


def _exact_contact(case, seed):
    posr, c, _, nb = _agents(case, seed)
    n = case["agents"]
    lin = (c[:, 2] * nb + c[:, 1]) * nb + c[:, 0]
    order = torch.sort(lin, stable=True).indices
    starts = torch.searchsorted(lin[order], torch.arange(nb ** 3 + 1, device=DEV))
    p = posr.double()
    force = torch.zeros(n, 3, dtype=torch.float64, device=DEV)
    me = torch.arange(n, device=DEV)
    for off in range(27):
        d = torch.tensor([off % 3 - 1, off // 3 % 3 - 1, off // 9 - 1], device=DEV)
        q = c + d
        ok = ((q >= 0) & (q < nb)).all(1)
        b = torch.where(ok, (q[:, 2] * nb + q[:, 1]) * nb + q[:, 0], 0)
        first, count = starts[b], torch.where(ok, starts[b + 1] - starts[b], 0)
        for slot in range(int(count.max())):
            row = torch.nonzero(count > slot).view(-1)
            j = order[first[row] + slot]
            keep = j != me[row]
            row, j = row[keep], j[keep]
            delta = p[row, :3] - p[j, :3]
            dist = delta.norm(dim=1)
            over = p[row, 3] + p[j, 3] - dist
            near = (over > 0) & (dist > 1e-5)
            row, delta, dist, over = row[near], delta[near], dist[near], over[near]
            force.index_add_(0, row, delta * (STIFFNESS * over * over.sqrt() / dist)[:, None])
    move = force * (MOBILITY * DT)
    length = move.norm(dim=1, keepdim=True)
    move = torch.where(length > MAX_DISP, move * (MAX_DISP / length), move)
    out = (p[:, :3] + move).clamp_(MARGIN, 10.0 * nb - MARGIN)
    return [out[:, a].contiguous() for a in range(3)]


# ---------------------------------------------------------------- the key sort
def _prepare_sort(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    n, bits = case["n"], case["bits"]
    key = torch.randint(0, 1 << bits, (n,), generator=g, device=DEV, dtype=torch.int64)
    if case["disorder"] < 1.0:
        fresh = torch.rand(n, generator=g, device=DEV) < case["disorder"]
        key = torch.where(fresh, key, key.sort().values)
    s = SimpleNamespace(kind="sort", lib=_lib.load(), n=n, bits=bits, key=key.to(torch.int32))
    s.kout, s.vout = torch.empty_like(s.key), torch.empty_like(s.key)
    s.bytes = s.lib.olc_sort_scratch_bytes(n, bits)
    s.scratch = torch.empty(s.bytes, dtype=torch.uint8, device=DEV)
    return s


def _run_sort(s):
    _lib.check(s.lib.olc_stage_sort_pairs(_ptr(s.key), None, _ptr(s.kout), _ptr(s.vout), s.n, s.bits,
                                          _ptr(s.scratch), s.bytes, _stream()))
    return [s.kout, s.vout]


# ---------------------------------------------------------------- whole steps
def _density(drug):
    """Agents per cubic um: the large configuration's ball with a drug field, the small one's without."""
    return 1e6 / (4.18879 * 400.0 ** 3) if drug else 1e4 / (4.18879 * 60.0 ** 3)


def _tumour(case, seed):
    n, grid = case["agents"], case["grid"]
    domain = 1000.0 if grid == 256 else 4.0 * grid
    ball = min(0.45 * domain, (n / _density(case["drug"]) / 4.18879) ** (1.0 / 3.0))
    return W.TumourSpec(name="case", n_agents=n, domain=domain, ball_radius=ball, field_dims=(grid,) * 3,
                        r_lo=4.0 if case["drug"] else 5.0, r_hi=6.0 if case["drug"] else 5.0, has_drug=case["drug"],
                        growth=GROWTH, death_k=0.0, storage=case["storage"], seed=seed,
                        capacity=2 * n + 4096)


def _prepare_engine(case, seed):
    eng = W.build_engine(_tumour(case, seed))
    if case["graphs"]:
        eng.set_graphs(True)
    return SimpleNamespace(kind="engine", eng=eng, drug=case["drug"])


def _run_engine(s):
    back = s.eng._backend_impl
    pending = s.eng.run_step(collect_metrics=True, wait=False)
    metrics = pending.result()
    out = {"metrics": {k: int(v) for k, v in metrics.items()}, "rows": pending.counters["n_agents"],
           "fields": [back.field_tensor(f) for f in (("o2", "drug") if s.drug else ("o2",))],
           "residuals": [c for c in back.comp_dev if c is not None],
           "agents": [back.column_tensor(c) for c in ("pos.x", "pos.y", "pos.z", "radius", "volume", "state",
                                                      "_rng_state")]}
    out["fields"] = [f if f.dtype == torch.float32 else f.view(torch.int16) for f in out["fields"]]
    return out


def _sweep(case, seed):
    # the sweep's own sizes and parameters (one draw of them), another population per seed
    specs = W.batched_specs(case["members"], seed=0)
    return [W.scaled(sp, growth=GROWTH, death_k=0.0, storage=case["storage"], seed=seed * 1000 + k)
            for k, sp in enumerate(specs)]


def _prepare_batch(case, seed):
    batch = W.build_batch(_sweep(case, seed))
    batch.set_graphs(True)
    return SimpleNamespace(kind="batch", batch=batch, n=case["members"])


def _run_batch(s):
    b = s.batch
    b.run_steps(1, collect_metrics=True)
    par = b._field_parity()
    ab = b._agent_buf()
    off = b.field_off
    fields = [b.fields_dev[i][int(par[k, i])][int(off[k]):int(off[k + 1])] for i in range(2) for k in range(s.n)]
    return {"live": np.array([[e._metrics.live, e._metrics.proliferating, e._metrics.quiescent, e._metrics.necrotic]
                              for e in b.engines]),
            "agents": [c[ab] for c in b.cols_dev],
            "fields": [f if f.dtype == torch.float32 else f.view(torch.int16) for f in fields],
            "residuals": [c for c in b.comp_dev if c is not None]}


# ---------------------------------------------------------------- the interface
_PREPARE = {"diffuse": _prepare_diffuse, "contact": _prepare_contact, "sort": _prepare_sort,
            "engine": _prepare_engine, "batch": _prepare_batch}
_RUN = {"diffuse": _run_diffuse, "contact": _run_contact, "sort": _run_sort, "engine": _run_engine,
        "batch": _run_batch}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return _RUN[state.kind](state)


def exact(case, seed):
    if case["kind"] == "diffuse":
        return _exact_diffuse(case, seed)
    if case["kind"] == "contact":
        return _exact_contact(case, seed)
    return None


def work(case):
    """Bytes: each input read and each output written once.  Operations: 12 per voxel and substep (six neighbour
    sums, the update, decay and clamp), 12 per contact candidate (the distance test)."""
    def field(nvox, substeps, storage, uptakes):
        elem = 4 if storage == "f32" else 2
        # 16-bit storage carries an FP32 residual per voxel, read and written
        return (nvox * (2 * elem + (8 if elem == 2 else 0)) + 8 * uptakes, 12 * nvox * substeps)

    def agents(n):
        return 2 * 28 * n, 12 * 90 * n

    kind = case["kind"]
    if kind == "diffuse":
        b, f = field(case["nx"] * case["ny"] * case["nz"], case["substeps"], case["storage"], case["uptakes"])
    elif kind == "contact":
        b, f = 28 * case["agents"], 12 * 90 * case["crowding"] * case["agents"]
    elif kind == "sort":
        b, f = 12 * case["n"], 0
    else:
        specs = [_tumour(case, 0)] if kind == "engine" else _sweep(case, 0)
        b = f = 0
        for sp in specs:
            nvox = int(np.prod(sp.field_dims))
            for substeps in [sp.S_o2] + ([sp.S_drug] if sp.has_drug else []):
                fb, ff = field(nvox, substeps, sp.storage, 0)
                b, f = b + fb, f + ff
            ab, af = agents(sp.n_agents)
            b, f = b + ab, f + af
    return {"bytes": b, "flops": f}
