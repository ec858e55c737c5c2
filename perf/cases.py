"""The work that users of the framework have it do, as cases that can be timed.

A case is a dict of plain values; :func:`prepare` makes what a program holds
before the call (a grid with its particles, a halo plan, a cotangent),
:func:`run` makes one pass through the public entry points of
``dsdecompx_b200`` and :func:`exact` says what that pass returns, restated
with plain torch in 64 bits.  The kinds of pass:

``wrap``     the single-rank drop-in's migrate (``rank_migrate``)
``step``     one queued batched step (``VirtualGrid.step_async``)
``calls``    the same step one call at a time, as a dsDecompX program has it:
             out_of_domain, migrate, exchange_halo(rebuild), reverse_halo
``refresh``  a step along a plan that stays valid: exchange_halo, reverse_halo
``fields``   reverse_exchange and forward_exchange of registered fields
``adjoint``  ``halo_backward``, the backward pass of the ghost copy
``owner``    ``owner_rank`` of positions that belong to nobody yet

The user's own share of a step (an integrator, a force loop) is kept as small
as it can be: particles move by their velocity times +dt and -dt in turn, so
that every pass migrates the same few particles and the distribution stays
what it is, and the ghosts' forces are copied from a table.
"""
import functools
import gc
import weakref

import torch

import dsdecompx_b200 as dsx

CORE = ["x", "y", "z", "vx", "vy", "vz", "fx", "fy", "fz", "mass", "charge"]
BYTES = {"int32": 4, "int64": 8, "uint32": 4, "uint64": 8, "float32": 4, "float64": 8}
# unsigned fields are looked at as signed ones of their size: the same bits
TORCH = {"int32": torch.int32, "int64": torch.int64, "uint32": torch.int32,
         "uint64": torch.int64, "float32": torch.float32, "float64": torch.float64}
TYPESTR = {torch.int32: "<i4", torch.int64: "<i8", torch.float32: "<f4", torch.float64: "<f8"}

ID = "id64:int64:1"
MESH = "charge2:float64:1,vec:float32:3"
FLUID = "energy:float64:1,pressure:float64:1,dipole:float64:3,species:int32:1,id64:int64:1"
MIXED = "a:int32:1,b:int64:1,c:uint32:2,d:uint64:1,e:float32:3,f:float64:1"


def _case(kind, n, dims="1x1x1", **more):
    """The defaults of a case: a periodic box of `dims` equal cells holding n
    uniform particles at `density`, halo width 2.8, velocities N(0, drift)."""
    case = dict(kind=kind, n=n, dims=dims, policy="manual", open="", edges=True, density=0.85,
                halo=2.8, drift=0.1, blobs=0, fields="", ops="", forward="", tune=False,
                positions_only=False, results=True)
    case.update(more)
    return case


def listed():
    return [
        # the drop-in of one rank that owns the whole box: 1M particles
        dict(_case("wrap", 1_000_000, density=1.0), name="wrap_1m"),
        # a small system of 8 subdomains: what a step costs when launches and latency are all
        dict(_case("step", 4_000, "2x2x2", density=0.5, halo=1.5, drift=0.2, fields=MESH),
             name="step_8_4k"),
        # a film with open faces and face neighbors only, an odd count, one axis unsplit
        dict(_case("step", 262_147, "3x1x4", open="xz", edges=False, fields=ID),
             name="step_12_262k"),
        # 2x2x2 at 8M with field exchanges inside the step (particle-mesh codes), fast particles
        dict(_case("step", 8_000_000, "2x2x2", density=1.0, drift=0.5, fields=MESH,
                   ops="vec:sum", forward="charge2"), name="step_8_8m"),
        # the benchmark: clustered particles, Dynamic boundaries, tuned as a long run would be
        dict(_case("step", 16_000_000, "4x4x4", policy="dynamic", density=0.9537, blobs=32,
                   fields=ID, tune=True), name="step_64_16m"),
        # the largest: 256 subdomains and a wide record
        dict(_case("step", 27_200_000, "8x8x4", drift=0.05, fields=FLUID, tune=True),
             name="step_256_27m"),
        # a program that makes one call at a time and reads every result; every field type
        dict(_case("calls", 1_000_003, "3x3x3", fields=MIXED), name="calls_27_1m"),
        # the inner loop between two rebuilds: positions out, forces back
        dict(_case("refresh", 16_000_000, "4x4x4", policy="dynamic", density=0.9537, blobs=32,
                   fields=ID, positions_only=True, results=False), name="refresh_64_16m"),
        # the same where the ghosts need velocities and every field, with the call's report read
        dict(_case("refresh", 13_600_007, "8x4x4", fields=FLUID), name="refresh_128_13m"),
        # partial sums, extrema and owners' values of fields over the halo (SPH, particle-mesh)
        dict(_case("fields", 2_000_003, "3x2x2", fields=MIXED, ops="a:max,b:sum,e:sum,f:min",
                   forward="c,d,f"), name="fields_12_2m"),
        # gradients of a differentiable energy through the halo: 262,144 particles at density 0.8
        dict(_case("adjoint", 262_144, "2x2x2", density=0.8), name="adjoint_8_262k"),
        # inserted particles (an inlet, a restart): who owns them under uneven cuts
        dict(_case("owner", 5_000_011, "4x4x4", policy="dynamic", blobs=32), name="owner_64_5m"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["wrap", "step", "step", "step", "calls", "refresh", "refresh", "fields",
                       "adjoint", "owner"])
    if kind == "wrap":
        return _case("wrap", _log(rng, 4_000, 20_000_000), density=round(rng.uniform(0.5, 1.2), 3))
    small = {"step": 2_400, "calls": 2_400, "refresh": 5_000, "fields": 5_000, "adjoint": 10_000,
             "owner": 2_400}[kind]
    n = _log(rng, small, 16_000_000)
    grids = ["2x2x2", "3x1x4", "4x2x1", "1x2x3", "5x1x1", "3x3x3", "3x2x2", "4x4x4", "5x4x3",
             "8x4x4", "8x8x4"]
    # at least 450 particles a subdomain, so that the halo is narrower than half a cell
    dims = rng.choice([d for d in grids if n >= 450 * _volume(d)])
    case = _case(kind, n, dims, density=round(rng.uniform(0.5, 1.1), 3),
                 drift=round(rng.uniform(0.03, 0.5), 3), fields=rng.choice(["", ID, MESH, FLUID, MIXED]))
    case["halo"] = round(min(rng.choice([1.5, 2.5, 2.8, 3.5]), 0.4 * _cell(case)), 3)
    if kind != "adjoint":
        case["open"] = rng.choice(["", "", "", "z", "xz"])
        case["edges"] = rng.random() < 0.85
    if kind in ("step", "refresh", "owner") and n > 100_000 and rng.random() < 0.3:
        case.update(policy="dynamic", blobs=rng.choice([5, 32]), open="")
    if kind == "step":
        case["tune"] = n > 4_000_000 and rng.random() < 0.5
    if kind == "refresh":
        case.update(positions_only=rng.random() < 0.6, results=rng.random() < 0.4)
    if kind == "fields":
        case.update(fields=MIXED, forward=rng.choice(["c", "c,d", "c,d,f"]),
                    ops=rng.choice(["e:sum", "b:sum,f:min", "a:max,b:sum,e:sum", "a:replace,f:max"]))
    return case


# ------------------------------------------------------------------- geometry

def _dims(case):
    return [int(d) for d in case["dims"].split("x")]


def _volume(dims):
    a, b, c = (int(d) for d in dims.split("x"))
    return a * b * c


def _cell(case):
    return (case["n"] / (_volume(case["dims"]) * case["density"])) ** (1.0 / 3.0)


def _box(case):
    return [d * _cell(case) for d in _dims(case)]


def _periodic(case):
    return ["xyz"[a] not in case["open"] for a in range(3)]


def _fields(case):
    return [(f.split(":")[0], f.split(":")[1], int(f.split(":")[2]))
            for f in case["fields"].split(",") if f]


def _record(case):
    return 96 + sum(BYTES[t] * c for _, t, c in _fields(case))


def _ghosts(case):
    """Ghosts of uniform particles under equal cells (both faces of every split axis)."""
    grow = 1.0
    for d, p in zip(_dims(case), _periodic(case)):
        faces = 0.0 if d == 1 else 2.0 if p else 2.0 * (d - 1) / d
        grow *= 1.0 + faces * case["halo"] / _cell(case)
    return case["n"] * (grow - 1.0)


def _room(case):
    """Ghost slots that a program's own loops cover: the ghosts of any pass."""
    return int((1.4 if case["blobs"] else 1.05) * _ghosts(case)) + 2_000


def work(case):
    """Bytes of a pass: records in and out, ghosts out, and the user's share."""
    n, g, s = case["n"], _ghosts(case), _record(case)
    if case["kind"] == "wrap":
        return {"bytes": 24 * n, "flops": 0}   # few positions change
    if case["kind"] == "owner":
        return {"bytes": 28 * n, "flops": 0}
    if case["kind"] == "adjoint":
        return {"bytes": 48 * n + 24 * g, "flops": 3 * g}
    exchanged = sum(BYTES[t] * c for f, t, c in _fields(case)
                    if f in case["forward"].split(",") or f in _ops(case))
    if case["kind"] == "fields":
        return {"bytes": 2 * exchanged * g, "flops": g}
    owners = min(g, n)
    back = 24 * g + 48 * owners + 48 * g          # the reverse sum, and the user's ghost forces
    if case["kind"] == "refresh":
        copied = 24 if case["positions_only"] else s - 48
        return {"bytes": 2 * copied * g + 24 * g + back, "flops": 6 * g}
    return {"bytes": 2 * s * n + s * g + back + 72 * n + 2 * exchanged * g, "flops": 6 * (n + g)}


def _ops(case):
    return dict(o.split(":") for o in case["ops"].split(",") if o)


# ------------------------------------------------------------------- particles

def _axis_cell(v, cuts):
    return (torch.bucketize(v, cuts, right=True) - 1).clamp_(0, cuts.numel() - 2)


def _cuts(case):
    return [torch.tensor([L * i / d for i in range(d + 1)], dtype=torch.float64, device="cuda")
            for L, d in zip(_box(case), _dims(case))]


def _owner(case, pos):
    d = _dims(case)
    c = [_axis_cell(v, cuts) for v, cuts in zip(pos, _cuts(case))]
    return (c[0] * d[1] + c[1]) * d[2] + c[2]


def _particles(case, seed):
    """(counts per subdomain, arrays by name): the particles of every subdomain
    of equal cells, in rank order, as `VirtualGrid.upload_flat` takes them."""
    n, box = case["n"], _box(case)
    gen = torch.Generator("cuda").manual_seed(seed)
    rand = functools.partial(torch.rand, generator=gen, dtype=torch.float64, device="cuda")
    randn = functools.partial(torch.randn, generator=gen, dtype=torch.float64, device="cuda")
    pos = [rand(n) * L for L in box]
    if case["blobs"]:
        # 80% in Gaussian blobs of 1/32 of the box, scattered over the storage
        inside = rand(n) < 0.8
        blob = torch.randint(0, case["blobs"], (n,), generator=gen, device="cuda")
        for a, L in enumerate(box):
            v = torch.remainder((rand(case["blobs"]) * L)[blob] + randn(n) * (L / 32), L)
            pos[a] = torch.where(inside & (v < L), v, pos[a])
    order = torch.sort(_owner(case, pos), stable=True)[1]
    counts = torch.bincount(_owner(case, pos), minlength=_volume(case["dims"])).cpu().numpy()
    out = {"xyz"[a]: pos[a][order] for a in range(3)}
    for a in "xyz":
        out["v" + a] = randn(n)
    out["mass"] = torch.ones(n, dtype=torch.float64, device="cuda")
    out["global_id"] = torch.arange(n, dtype=torch.int32, device="cuda")
    for name, t, c in _fields(case):
        if t.startswith("float"):
            out[name] = randn(n, c).to(TORCH[t])
        else:
            out[name] = torch.randint(0, 1 << 20, (n, c), generator=gen, device="cuda").to(TORCH[t])
    return counts, out


def _table(seed, ghosts):
    """Values that a user's force loop leaves on the ghosts."""
    gen = torch.Generator("cuda").manual_seed(seed + 7919)
    return list(torch.randn(3, ghosts, generator=gen, dtype=torch.float64, device="cuda"))


class _Address:
    """`shape` elements of a grid's storage, for torch.as_tensor: the tensor
    keeps this object, and with it the grid, alive."""

    def __init__(self, grid, address, shape, dtype):
        self.grid = grid
        self.__cuda_array_interface__ = {"data": (int(address), False), "shape": tuple(shape),
                                         "typestr": TYPESTR[dtype], "version": 3}


def _tensor(grid, address, shape, dtype):
    return torch.as_tensor(_Address(grid, address, shape, dtype), device="cuda")


class _Arrays:
    """A grid's particle arrays as tensors, owned or ghosts, by name."""

    def __init__(self, case, grid):
        v, self.grid = grid.view(), grid
        kinds = [(a, torch.float64, 1) for a in CORE] + [("type", torch.int32, 1),
                                                         ("global_id", torch.int32, 1)]
        kinds += [(name, TORCH[t], c) for name, t, c in _fields(case)]
        self.base = {name: (v.base[k], dtype, c) for k, (name, dtype, c) in enumerate(kinds)}
        self.ghost_offset, self.capacity = v.ghost_offset, v.ghost_capacity
        self.owned_offset, self.n = v.owned_offset, v.particles

    def slice(self, name, first, count):
        base, dtype, c = self.base[name]
        return _tensor(self.grid, base + first * c * dtype.itemsize, (count,) if c == 1 else (count, c), dtype)

    def owned(self, name):
        return self.slice(name, self.owned_offset, self.n)

    def ghosts(self, name, count):
        return self.slice(name, self.ghost_offset, count)


# --------------------------------------------------------------------- prepare

class State:
    pass


def _settled(case, counts, arrays, room=0):
    """(grid, ghosts): the grid with its halo plan, Dynamic cuts where they stay."""
    grid = _grid(case, counts, arrays, room)
    if case["policy"] == "dynamic":
        for _ in range(12):
            grid.migrate(results=False)
    if case["tune"]:
        grid.autotune()
    return grid, int(grid.exchange_halo(rebuild=True)[:, 0].sum())


def _grid(case, counts, arrays, room=0):
    n = case["n"]
    if not room:
        room = int(1.5 * _ghosts(case)) + 20_000
        if case["blobs"]:
            room = max(room, int(0.9 * n))
    grid = dsx.VirtualGrid(_volume(case["dims"]), dims=_dims(case), policy=case["policy"],
                           upper=_box(case), periodic=_periodic(case), halo_width=case["halo"],
                           edges_and_corners=case["edges"], fields=_fields(case), particles=n,
                           ghost_capacity=room)
    names = CORE + ["type", "global_id"] + [f for f, _, _ in _fields(case)]
    torch.cuda.synchronize()   # the arrays were made on another stream than the grid's
    grid.upload_flat(counts, [arrays[k].data_ptr() if k in arrays else None for k in names])
    return grid


def prepare(case, seed):
    gc.collect()   # a grid that steps with a callback is in a reference cycle with it
    s = State()
    s.case, s.stream = case, torch.cuda.Stream()
    if case["kind"] == "wrap":
        _, a = _particles(case, seed)
        s.pos = [a[k] + case["drift"] * a["v" + k] for k in "xyz"]
        s.box = _box(case)
        return s
    if case["kind"] == "owner":
        # positions around the box, under cuts that clustered particles have moved
        n = max(2_400, case["n"] // 8)
        few = dict(case, n=n, density=case["density"] * n / case["n"])
        s.grid = _grid(few, *_particles(few, seed))
        for _ in range(8):
            s.grid.migrate(results=False)
        gen = torch.Generator("cuda").manual_seed(seed + 1)
        s.pos = [(torch.rand(case["n"], generator=gen, dtype=torch.float64, device="cuda") * 1.1
                  - 0.05) * L for L in _box(case)]
        s.out = torch.empty(case["n"], dtype=torch.int32, device="cuda")
        return s
    counts, arrays = _particles(case, seed)
    s.grid, ghosts = _settled(case, counts, arrays)
    if 1.5 * ghosts > s.grid.view().ghost_capacity:   # storage must not move under a program's tensors
        s.grid, ghosts = _settled(case, counts, arrays, 2 * ghosts)
    del arrays
    if case["kind"] == "adjoint":
        gen = torch.Generator("cuda").manual_seed(seed + 1)
        draw_ = functools.partial(torch.randn, generator=gen, dtype=torch.float64, device="cuda")
        s.upstream, s.cotangent = draw_(3, case["n"]), draw_(3, ghosts)
        return s
    a = _Arrays(case, s.grid)
    for name in a.base:
        a.ghosts(name, a.capacity).zero_()
    s.room = _room(case)
    s.table = _table(seed, s.room)
    s.ghost_forces = [a.ghosts(k, s.room) for k in ("fx", "fy", "fz")]
    s.deposit = [a.ghosts(f, s.room) for f in _ops(case)]
    s.ops, s.forward = list(_ops(case).items()), [f for f in case["forward"].split(",") if f]
    # the two owned halves and the two layouts of the counts that migrates swap
    s.halves, s.moved = [], []
    for _ in range(2):
        a, v = _Arrays(case, s.grid), s.grid.view()
        out = {"owned." + k: a.owned(k) for k in a.base}
        out.update({"ghosts." + k: a.ghosts(k, s.room) for k in a.base})
        out["n"] = _tensor(s.grid, v.n, (v.nranks,), torch.int32)
        out["g"] = _tensor(s.grid, v.g, (v.nranks,), torch.int32)
        s.halves.append(out)
        s.moved.append(([out["owned." + k] for k in ("x", "y", "z")],
                        [out["owned." + k] for k in ("vx", "vy", "vz")]))
        s.grid.migrate(results=False)
    s.half = 0
    if case["kind"] in ("refresh", "fields"):
        s.grid.exchange_halo(rebuild=True)
        for t in s.deposit:
            _deposit(t)
    else:
        _drift(s, 0, 1.0)     # the first pass has particles to migrate
    if case["kind"] == "step":
        first = a.owned_offset     # of half 1
        state = weakref.ref(s)     # the grid keeps the callback, and s keeps the grid

        def callback(view, _stream):
            s = state()
            half = 1 if view.owned_offset == first else 0
            with torch.cuda.stream(s.stream):
                _user(s, half, 1.0 if half == 0 else -1.0)
                if s.ops:
                    s.grid.reverse_exchange(s.ops)
                if s.forward:
                    s.grid.forward_exchange(s.forward)
        s.callback = callback
    return s


def _deposit(t):
    t.fill_(0.25 if t.is_floating_point() else 3)


def _drift(s, half, sign):
    pos, vel = s.moved[half]
    torch._foreach_add_(pos, vel, alpha=sign * s.case["drift"])


def _user(s, half, sign):
    """What a program does between the halo and the reverse sum: forces on the
    ghosts, partial field values on the ghosts, and the integrator."""
    torch._foreach_copy_(s.ghost_forces, s.table)
    for t in s.deposit:
        _deposit(t)
    _drift(s, half, sign)


# ------------------------------------------------------------------------- run

def run(s):
    kind = s.case["kind"]
    if kind == "step":
        s.grid.step_async(s.callback, stream=s.stream)
        s.half ^= 1
        return s.halves[s.half]
    with torch.cuda.stream(s.stream):
        if kind == "wrap":
            dsx.rank_migrate(*s.pos, s.case["n"], (0.0, 0.0, 0.0), s.box)
            return s.pos
        if kind == "owner":
            s.grid.owner_rank(*s.pos, s.out)
            return s.out
        if kind == "adjoint":
            grad = s.upstream.clone()
            s.grid.halo_backward(s.cotangent, grad)
            return grad
        if kind == "fields":
            s.grid.reverse_exchange(s.ops)
            s.grid.forward_exchange(s.forward)
            return s.halves[s.half]
        if kind == "refresh":
            s.grid.exchange_halo(positions_only=s.case["positions_only"], results=s.case["results"])
            torch._foreach_copy_(s.ghost_forces, s.table)
            s.grid.reverse_halo()
            return s.halves[s.half]
        # calls
        if s.grid.out_of_domain()[1]:
            migrated = s.grid.migrate()
            s.half ^= 1
        else:
            migrated = None
        built = s.grid.exchange_halo(rebuild=True)
        _user(s, s.half, 1.0 if s.half == 0 else -1.0)
        s.grid.reverse_halo()
        return dict(s.halves[s.half], migrated=migrated, built=built)


# ----------------------------------------------------------------------- exact

def _wrap(case, pos):
    return [v - torch.floor(v / L) * L if p else v.clone()
            for v, L, p in zip(pos, _box(case), _periodic(case))]


def _migrate(case, counts, a):
    """Retained particles of every subdomain in their order, then immigrants
    by source subdomain and source order."""
    source = torch.repeat_interleave(torch.arange(len(counts), device="cuda"), counts)
    w = _wrap(case, [a[k] for k in "xyz"])
    dest = _owner(case, _wrap(case, w))
    order = torch.sort(dest * 2 + (dest != source), stable=True)[1]
    a = dict(a, x=w[0], y=w[1], z=w[2])
    return torch.bincount(dest, minlength=len(counts)), {k: v[order] for k, v in a.items()}


def _halo(case, counts, a):
    """(owner, shift per axis, direction) of every ghost, receiver by receiver
    and block by block in the receiver's neighbor order, senders in owned order."""
    d, box, periodic, w = _dims(case), _box(case), _periodic(case), case["halo"]
    cuts = _cuts(case)
    rank = torch.repeat_interleave(torch.arange(len(counts), device="cuda"), counts)
    c = [rank // (d[1] * d[2]), (rank // d[2]) % d[1], rank % d[2]]
    low = [a["xyz"[k]] < cuts[k][c[k]] + w for k in range(3)]
    high = [a["xyz"[k]] > cuts[k][c[k] + 1] - w for k in range(3)]
    offsets = [(i, j, k) for i in (-1, 0, 1) for j in (-1, 0, 1) for k in (-1, 0, 1)
               if (i or j or k) and (case["edges"] or abs(i) + abs(j) + abs(k) == 1)]
    blocks = []
    for m, back in enumerate(offsets):          # the receiver's block toward its sender
        step = [-o for o in back]
        hit = torch.ones_like(rank, dtype=torch.bool)
        for k in range(3):
            if step[k]:
                if d[k] == 1:
                    hit.zero_()
                to = c[k] + step[k]
                hit &= (low[k] if step[k] < 0 else high[k])
                if not periodic[k]:
                    hit &= (to >= 0) & (to < d[k])
        i = hit.nonzero()[:, 0]
        to, shift = [], []
        for k in range(3):
            t = c[k][i] + step[k]
            shift.append(((t < 0).double() - (t >= d[k]).double()) * box[k])
            to.append(t % d[k])
        n = offsets.index(tuple(step))          # the sender's list
        blocks.append(((to[0] * d[1] + to[1]) * d[2] + to[2], i, shift, torch.full_like(i, n)))
    receiver = torch.cat([b[0] for b in blocks])
    order = torch.sort(receiver, stable=True)[1]
    return (torch.cat([b[1] for b in blocks])[order],
            [torch.cat([b[2][k] for b in blocks])[order] for k in range(3)],
            torch.cat([b[3] for b in blocks])[order])


def _reverse(values, owner, direction, ghost, op="sum"):
    """Owners' values with their images', in the order of the sender's lists."""
    for n in torch.unique(direction).tolist():
        at = (direction == n).nonzero()[:, 0]
        o, g = values[owner[at]], ghost[at]
        values[owner[at]] = (o + g if op == "sum" else torch.minimum(o, g) if op == "min" else
                             torch.maximum(o, g) if op == "max" else g)


def exact(case, seed):
    if case["kind"] == "owner" or case["policy"] != "manual":
        return None    # whole numbers; cuts that only the framework's own rebalance gives
    counts, a = _particles(case, seed)
    if case["kind"] == "wrap":
        return _wrap(case, [a[k] + case["drift"] * a["v" + k] for k in "xyz"])
    counts = torch.from_numpy(counts).cuda()
    for k in CORE:
        a.setdefault(k, torch.zeros_like(a["x"]))
    owner, shift, direction = _halo(case, counts, a)
    ghosts = owner.numel()
    if case["kind"] == "adjoint":
        gen = torch.Generator("cuda").manual_seed(seed + 1)
        draw_ = functools.partial(torch.randn, generator=gen, dtype=torch.float64, device="cuda")
        grad, cot = draw_(3, case["n"]), draw_(3, ghosts)
        for k in range(3):
            _reverse(grad[k], owner, direction, cot[k])
        return grad
    room = _room(case)
    table = _table(seed, room)
    if case["kind"] in ("step", "calls"):
        for k in "xyz":
            a[k] = a[k].add(a["v" + k], alpha=case["drift"])
        counts, a = _migrate(case, counts, a)
        owner, shift, direction = _halo(case, counts, a)
        ghosts = owner.numel()
    real = [k for k in CORE] + [f for f, t, _ in _fields(case) if t.startswith("float")]
    g = {k: a[k][owner] for k in real}
    for k in range(3):
        g["xyz"[k]] = g["xyz"[k]] + shift[k]
        g["f" + "xyz"[k]] = table[k][:ghosts].clone()
    if case["kind"] in ("step", "calls"):
        for k in "xyz":
            a[k] = a[k].add(a["v" + k], alpha=-case["drift"])
    if case["kind"] != "fields":
        for k in ("fx", "fy", "fz"):
            _reverse(a[k], owner, direction, g[k])
    else:
        for k in ("fx", "fy", "fz"):
            g[k].zero_()
    if case["kind"] in ("step", "fields"):
        for f, op in _ops(case).items():
            if f in g:
                a[f] = a[f].double()
                _deposit(g[f])
                _reverse(a[f], owner, direction, g[f].double(), op)
        for f in case["forward"].split(","):
            if f in g:
                g[f] = a[f][owner]
    out = {"owned." + k: a[k].squeeze(-1) if a[k].dim() == 2 and a[k].shape[1] == 1 else a[k]
           for k in real}
    for k in real:
        # slots past the ghosts: zero, or what the user's own loops leave there
        v = g[k].squeeze(-1) if g[k].dim() == 2 and g[k].shape[1] == 1 else g[k]
        whole = torch.zeros((room,) + v.shape[1:], dtype=v.dtype, device="cuda")
        whole[:ghosts] = v
        if k in ("fx", "fy", "fz") and case["kind"] != "fields":
            whole[ghosts:] = table["xyz".index(k[1])][ghosts:]
        if k in _ops(case):
            _deposit(whole[ghosts:])
        out["ghosts." + k] = whole
    return out
