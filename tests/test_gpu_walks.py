"""Walks of the ghosts list by list (chosen where the copied arrays exceed the
L2) against the walk in slot order, which the parity tests hold to the oracle:
the same values in every ghost slot, bit for bit (both only copy)."""
import numpy as np
import pytest

from helpers import same, uniform_particles

pytestmark = pytest.mark.gpu

# a field of 5,000 bytes makes 30,000 particles exceed the L2, and 1,250
# four-byte words leave a remainder of the three-word groups
WIDE = [("w", "float32", 1250), ("v", "float64", 3), ("s", "int32", 1)]


@pytest.mark.parametrize("dims,halo,periodic,n", [
    ((10, 10, 10), 0.12, (True, True, True), 30_011),     # more lists in a row than one window
    ((3, 1, 4), 0.05, (False, True, False), 28_001),      # empty lists at open faces
    ((2, 2, 2), 0.0005, (True, True, True), 27_999),      # fewer ghosts than one warp's rows
    ((2, 2, 2), 0.25, (True, True, True), 27_777),        # several passes of full rows
], ids=["short_lists", "open_faces", "few_ghosts", "many_ghosts"])
def test_list_walk_equals_slot_walk(cuda, dims, halo, periodic, n):
    import dsdecompx_b200 as dsx

    P = dims[0] * dims[1] * dims[2]
    rng = np.random.default_rng(11)
    data = uniform_particles(rng, n, (0, 0, 0), dims, WIDE)
    cell = [np.minimum(np.floor(data[a]).astype(int), d - 1) for a, d in zip("xyz", dims)]
    owner = (cell[0] * dims[1] + cell[1]) * dims[2] + cell[2]
    order = np.argsort(owner, kind="stable")
    per_rank = [{k: v[order][owner[order] == r] for k, v in data.items()} for r in range(P)]
    grid = dsx.VirtualGrid(P, dims=dims, upper=[float(d) for d in dims], periodic=periodic,
                           halo_width=halo, fields=WIDE, particles=n, ghost_capacity=8 * n)
    grid.upload(per_rank)
    ghosts = int(grid.exchange_halo(rebuild=True)[:, 0].sum())
    assert ghosts > 0
    check = sorted(rng.choice(P, min(P, 4), replace=False).tolist())

    def values():
        return [{k: v for k, v in grid.snapshot(r).items()} for r in check]

    results = {}
    for kind in ("ghosts", "auto"):
        grid.set_refresh_kind(kind)
        for r in check:      # what a refresh has to overwrite
            o, g = grid.counts(r)
            for name in ("x", "vy", "fz", "w", "v", "s"):
                c = grid.components(name)
                grid.write(r, name, o, np.zeros((g, c), dtype=grid.dtype_of(name)))
        grid.exchange_halo()
        results[kind] = values()
    for a, b in zip(results["ghosts"], results["auto"]):
        for k in a:
            assert same(a[k], b[k]), k
    # forward_exchange of the same fields leaves what the refresh left there
    for r in check:
        o, g = grid.counts(r)
        for name in ("w", "v", "s"):
            grid.write(r, name, o, np.zeros((g, grid.components(name)), dtype=grid.dtype_of(name)))
    grid.forward_exchange(["s", "w", "v"])
    for a, b in zip(results["ghosts"], values()):
        for k in ("w", "v", "s"):
            assert same(a[k], b[k]), k
    grid.close()
