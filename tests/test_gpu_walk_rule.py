"""Which walk of the ghosts a refresh and a forward exchange take, and that the
one by list leaves what the one in slot order does (which the parity tests
hold to the oracle) in every ghost slot of every array, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

NAMES = ["x", "y", "z", "vx", "vy", "vz", "fx", "fy", "fz", "mass", "charge", "type", "global_id"]
DTYPES = ["f8"] * 11 + ["i4"] * 2


class Address:
    def __init__(self, grid, address, count, typestr):
        self.grid = grid     # the storage stays alive
        self.__cuda_array_interface__ = {"data": (int(address), False), "shape": (int(count),),
                                         "typestr": "<" + typestr, "version": 3}


def make(dims, n, halo, periodic, fields, ghost_capacity=0, particles=0, edge=0.0):
    """A grid of unit cells with n uniform particles (edge: their x that far
    above a cell's lower face at most) and its halo plan."""
    import torch

    import dsdecompx_b200 as dsx

    gen = torch.Generator("cuda").manual_seed(n)
    P = dims[0] * dims[1] * dims[2]
    pos = [torch.rand(n, generator=gen, dtype=torch.float64, device="cuda") * d for d in dims]
    if edge:
        pos[0] = pos[0].floor() + edge * (pos[0] - pos[0].floor())
    cell = [v.long().clamp(max=d - 1) for v, d in zip(pos, dims)]
    owner = (cell[0] * dims[1] + cell[1]) * dims[2] + cell[2]
    order = torch.sort(owner, stable=True)[1]
    counts = torch.bincount(owner, minlength=P).cpu().numpy()
    arrays = {"xyz"[a]: pos[a][order] for a in range(3)}
    for name in ("vx", "vy", "vz"):
        arrays[name] = torch.randn(n, generator=gen, dtype=torch.float64, device="cuda")
    for name, kind, comps in fields:
        words = comps * (2 if kind.endswith("64") else 1)
        arrays[name] = torch.randint(0, 1 << 30, (n * words,), generator=gen, device="cuda", dtype=torch.int32)
    grid = dsx.VirtualGrid(P, dims=dims, upper=[float(d) for d in dims], periodic=periodic, halo_width=halo,
                           fields=fields, particles=particles or n, ghost_capacity=ghost_capacity)
    torch.cuda.synchronize()
    grid.upload_flat(counts, [arrays[k].data_ptr() if k in arrays else None
                              for k in NAMES + [f[0] for f in fields]])
    ghosts = int(grid.exchange_halo(rebuild=True)[:, 0].sum())
    return grid, ghosts


def ghost_words(grid, ghosts, fields):
    """The ghost region of every array as 32-bit words (a view, by name)."""
    import torch

    v = grid.view()
    widths = [8] * 11 + [4] * 2 + [c * (8 if k.endswith("64") else 4) for _, k, c in fields]
    return {name: torch.as_tensor(Address(grid, v.base[k] + v.ghost_offset * width, ghosts * width // 4, "i4"),
                                  device="cuda")
            for k, (name, width) in enumerate(zip(NAMES + [f[0] for f in fields], widths))}


def kernels(call):
    """Names of the library's kernels that `call` launches."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        call()
        torch.cuda.synchronize()
    return [e.key for e in p.key_averages() if "k_halo_refresh" in e.key or "k_forward" in e.key]


def check_walks(grid, ghosts, fields, positions_only):
    """auto against slot order: a refresh, and a forward exchange of every field."""
    import torch

    words = ghost_words(grid, ghosts, fields)
    results = []
    for kind in ("ghosts", "auto"):
        grid.set_refresh_kind(kind)
        for name, w in words.items():
            if name not in ("mass", "charge", "type", "global_id") and not (
                    positions_only and name not in ("x", "y", "z", "fx", "fy", "fz")):
                w.fill_(-1)     # what the refresh has to overwrite
        torch.cuda.synchronize()
        grid.exchange_halo(positions_only=positions_only, results=False)
        torch.cuda.synchronize()
        results.append({k: w.clone() for k, w in words.items()})
    for k in words:
        assert torch.equal(results[0][k], results[1][k]), k
    if positions_only or not fields:
        return
    for name, _, _ in fields:
        words[name].fill_(-1)
    torch.cuda.synchronize()
    grid.forward_exchange([f[0] for f in fields])
    torch.cuda.synchronize()
    for name, _, _ in fields:
        assert torch.equal(results[0][name], words[name]), name


FLUID = [("energy", "float64", 1), ("pressure", "float64", 1), ("dipole", "float64", 3),
         ("species", "int32", 1), ("id64", "int64", 1)]
WIDE = [("w", "float32", 300_001)]


@pytest.mark.parametrize("dims,n,halo,periodic,fields,positions_only", [
    ((10, 10, 10), 9_000_011, 0.12, (True, True, True), FLUID, False),   # short lists, many in a row
    ((3, 1, 4), 6_000_017, 0.05, (False, True, False), FLUID, False),    # empty lists at open faces
    ((2, 2, 2), 251, 0.1, (True, True, True), WIDE, False),              # a few ghosts, of 1.2 MB
    ((2, 2, 2), 3_000_001, 0.25, (True, True, True), FLUID, False),      # several passes of full rows
    ((4, 2, 1), 8_000_009, 0.1, (True, True, True), [], True),           # positions alone
    ((1, 2, 3), 8_000_003, 0.1, (True, True, False), [], True),
], ids=["short_lists", "open_faces", "few_ghosts", "many_ghosts", "positions", "positions_open"])
def test_list_walk_leaves_what_slot_order_does(cuda, dims, n, halo, periodic, fields, positions_only):
    grid, ghosts = make(dims, n, halo, periodic, fields)
    names = kernels(lambda: grid.exchange_halo(positions_only=positions_only, results=False))
    assert any(f"k_halo_refresh<{str(positions_only).lower()}, true>" in k for k in names), names
    if fields:
        names = kernels(lambda: grid.forward_exchange([f[0] for f in fields]))
        assert any("k_forward_by_list" in k for k in names), names
    check_walks(grid, ghosts, fields, positions_only)
    grid.close()


@pytest.mark.parametrize("n,halo,ghost_capacity,fields,positions_only", [
    (3_000_001, 0.02, 16_000_000, FLUID, False),    # far fewer ghosts than the capacity's split
    (8_000_003, 0.06, 16_000_000, [], True),
    (8_000_009, 0.15, 0, [], True),                 # whole rows over the whole grid
    (2_000_003, 0.28, 40_000_000, FLUID, False),
], ids=["reserved", "reserved_positions", "window_positions", "window_reserved"])
def test_list_walk_splits_by_the_plan(cuda, n, halo, ghost_capacity, fields, positions_only):
    grid, ghosts = make((2, 2, 2), n, halo, (True, True, True), fields, ghost_capacity=ghost_capacity)
    names = kernels(lambda: grid.exchange_halo(positions_only=positions_only, results=False))
    assert any(f"k_halo_refresh<{str(positions_only).lower()}, true>" in k for k in names), names
    check_walks(grid, ghosts, fields, positions_only)
    grid.close()


@pytest.mark.parametrize("dims,n,halo,fields,call", [
    # what slot order touches between two of a sender's receivers fits the L2
    ((8, 8, 4), 4_000_000, 0.05, [], "positions"),
    ((2, 2, 2), 4_000_000, 0.01, [], "positions"),
    ((2, 1, 1), 12_000_000, 0.08, [], "positions"),
    ((8, 8, 4), 6_000_000, 0.08, [("c", "uint32", 2), ("d", "uint64", 2), ("f", "float64", 1)], "forward"),
    ((2, 2, 2), 6_000_000, 0.01, [("c", "uint32", 2), ("d", "uint64", 2), ("f", "float64", 1)], "forward"),
], ids=["plane", "thin", "one_axis", "forward_plane", "forward_thin"])
def test_small_reuse_distances_keep_slot_order(cuda, dims, n, halo, fields, call):
    grid, _ = make(dims, n, halo, (True, True, True), fields)
    if call == "positions":
        names = kernels(lambda: grid.exchange_halo(positions_only=True, results=False))
        assert any("k_halo_refresh_slots<true>" in k for k in names), names
    else:
        names = kernels(lambda: grid.forward_exchange([f[0] for f in fields]))
        assert any("k_forward_fields" in k for k in names), names
    grid.close()


def test_capacity_does_not_choose_the_walk(cuda):
    """A program that reserves far more than it holds walks as one that does not."""
    grid, _ = make((2, 2, 2), 300_000, 0.05, (True, True, True), FLUID, particles=8_000_000)
    names = kernels(lambda: grid.exchange_halo(results=False))
    assert any("k_halo_refresh<false, false>" in k for k in names), names
    grid.close()


@pytest.mark.parametrize("fields", [[], FLUID[:2], FLUID[:3]], ids=["none", "two", "three"])
@pytest.mark.parametrize("positions_only", [False, True], ids=["full", "positions"])
def test_slot_order_by_ghost_and_by_row(cuda, fields, positions_only):
    """Both forms of the walk in slot order against the walk owner by owner."""
    import torch

    grid, ghosts = make((3, 2, 2), 40_003, 0.2, (True, False, True), fields)
    words = ghost_words(grid, ghosts, fields)
    results = []
    for kind in ("owners", "ghosts"):
        grid.set_refresh_kind(kind)
        for name in ["x", "y", "z", "fx", "fy", "fz"] + ([] if positions_only else
                                                         ["vx", "vy", "vz"] + [f[0] for f in fields]):
            words[name].fill_(-1)
        torch.cuda.synchronize()
        names = kernels(lambda: grid.exchange_halo(positions_only=positions_only, results=False))
        results.append({k: w.clone() for k, w in words.items()})
    by_row = len(fields) >= 3 and not positions_only
    assert any(("k_halo_refresh<" if by_row else "k_halo_refresh_slots<") in k for k in names), names
    for k in words:
        assert torch.equal(results[0][k], results[1][k]), k
    grid.close()


def test_reverse_sum_of_more_owners_than_expected(cuda):
    """Every particle on the boundary, where the mean cell has a ninth there."""
    import torch

    grid, ghosts = make((2, 2, 2), 1_000_003, 0.02, (True, True, True), [], edge=0.015)
    assert grid.totals()["boundary"] == 1_000_003
    words = ghost_words(grid, ghosts, [])
    v = grid.view()
    owned = [torch.as_tensor(Address(grid, v.base[6 + a] + v.owned_offset * 8, v.particles, "f8"), device="cuda")
             for a in range(3)]
    gen = torch.Generator("cuda").manual_seed(3)
    force = torch.randn(3, ghosts, generator=gen, dtype=torch.float64, device="cuda")
    results = []
    for per_sm in (32, 0):
        grid.set_tuning(reverse_ctas_per_sm=per_sm)
        for a in range(3):
            owned[a].fill_(0.5)
            words["f" + "xyz"[a]].copy_(force[a].view(torch.int32))
        torch.cuda.synchronize()
        grid.reverse_halo()
        torch.cuda.synchronize()
        results.append([t.clone() for t in owned])
    for a in range(3):
        assert not torch.equal(results[0][a], torch.full_like(owned[a], 0.5))
        assert torch.equal(results[0][a], results[1][a]), a
    grid.close()


@pytest.mark.parametrize("dims,n,halo,periodic,by_tile", [
    ((2, 2, 2), 6_500_003, 0.2, (True, True, True), True),      # thick lists of few large subdomains
    ((3, 2, 2), 9_000_001, 0.18, (True, False, True), True),
    ((2, 1, 1), 12_000_017, 0.2, (True, True, True), False),    # lists in one dimension
    ((2, 2, 2), 6_500_003, 0.05, (True, True, True), False),    # thin ones
], ids=["thick", "open", "one_axis", "thin"])
def test_thick_lists_of_wide_records_go_tile_by_tile(cuda, dims, n, halo, periodic, by_tile):
    grid, ghosts = make(dims, n, halo, periodic, FLUID)
    names = kernels(lambda: grid.exchange_halo(results=False))
    assert any("k_halo_refresh_staged" in k for k in names) == by_tile, names
    check_walks(grid, ghosts, FLUID, False)
    grid.close()
