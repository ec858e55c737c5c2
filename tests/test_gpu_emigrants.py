"""Both ways of placing emigrants (one CTA per destination up to 1,024 tiles,
the chain of kernels beyond) and the counters around them, against the oracle:
list lengths around the four entries a thread reads, more immigrants than one
pass of a CTA takes, and few enough
subdomains for copies of the immigrant counters; and the scan of the tiles'
counters around its rows."""
import numpy as np
import pytest

from helpers import Pair, split_by_owner, uniform_particles

pytestmark = pytest.mark.gpu


def check(pair, rng, sigma, steps=2):
    import torch

    stream = torch.cuda.Stream()
    for step in range(steps):
        pair.displace(rng, sigma)
        torch.cuda.synchronize()
        if step:      # the batched step, then the calls it stands for
            # the callback's first launch is the library's own: it must wait
            # for the emigrants' branch as well as for the move
            callback = None
            if pair.fields:
                def callback(view, s):
                    pair.gpu.reverse_exchange([("q", "sum")], stream=s)
            assert pair.gpu.step(callback, capture=True, stream=stream) == 0
            pair.ref.migrate()
            pair.ref.exchange_halo(rebuild=True)
            if pair.fields:
                pair.ref.reverse_exchange([("q", "sum")])
            pair.ref.reverse_halo()
        else:
            assert (pair.gpu.migrate() == pair.ref.migrate()).all()
            hg, hr = pair.gpu.exchange_halo(rebuild=True), pair.ref.exchange_halo(rebuild=True)
            assert (hg[:, 0] == hr[:, 0]).all()
        pair.compare(f"step {step}")


@pytest.mark.parametrize("dims,n,sigma", [
    ((2, 1, 1), 7, 0.6),             # a list shorter than one thread's entries
    ((5, 1, 1), 2_049, 0.02),        # a few emigrants
    ((2, 2, 2), 4_097, 3.0),         # most leave: a destination's passes and list passes
    ((3, 2, 2), 40_000, 0.3),
    ((2, 1, 2), 530_000, 0.2),       # more than 1,024 tiles: the chain, two counter copies
], ids=["tiny", "few", "most", "mid", "chain"])
def test_emigrants_follow_the_oracle(cuda, dims, n, sigma):
    rng = np.random.default_rng(n)
    fields = [("q", "float64", 1), ("v", "float32", 3)] if n < 100_000 else []
    L = [4.0 * d for d in dims]
    pair = Pair(int(np.prod(dims)), dims, "manual", (0, 0, 0), L, (True, True, True), 0.5, True,
                None, fields, particles=n, ghost_capacity=3 * n + 1000)
    try:
        data = uniform_particles(rng, n, (0, 0, 0), L, fields)
        owner = pair.ref.owner_rank(np.stack([data["x"], data["y"], data["z"]], 1))
        pair.upload(split_by_owner(owner, data, pair.P))
        check(pair, rng, sigma)
    finally:
        pair.close()


@pytest.mark.parametrize("dims,n,sigma", [
    ((2, 2, 2), 30_011, 3.0),        # eight CTAs of 256 threads, several passes each
    ((3, 3, 2), 20_003, 4.0),        # four
    ((2, 1, 1), 9_001, 1.8),         # a list that one CTA takes
    ((2, 1, 1), 11_003, 3.0),        # a list just past it
    ((2, 1, 1), 140_001, 3.0),       # more than 256 tiles: eight CTAs of 512 threads
    ((3, 2, 2), 135_007, 3.0),       # two
], ids=["eight", "four", "one", "just_past", "wide_eight", "wide_two"])
def test_many_emigrants_share_a_cluster(cuda, dims, n, sigma):
    rng = np.random.default_rng(n)
    fields = [("q", "float64", 1), ("v", "float32", 3)] if n < 100_000 else []
    L = [4.0 * d for d in dims]
    pair = Pair(int(np.prod(dims)), dims, "manual", (0, 0, 0), L, (True, True, True), 0.5, True,
                None, fields, particles=n, ghost_capacity=3 * n + 1000)
    try:
        data = uniform_particles(rng, n, (0, 0, 0), L, fields)
        owner = pair.ref.owner_rank(np.stack([data["x"], data["y"], data["z"]], 1))
        pair.upload(split_by_owner(owner, data, pair.P))
        check(pair, rng, sigma)
        assert (pair.gpu.totals()["emigrants"] > 4_096) == (n != 9_001)
    finally:
        pair.close()


@pytest.mark.parametrize("tiles", [4_095, 4_097, 32_767, 32_770])
def test_tile_scans_around_their_rows(cuda, tiles):
    """A migrate of as many tiles as fill the scan's rows (4,096 tiles to a row
    of the block, eight rows a pass), one less and a few more: every id where
    a stable sort by destination, retained particles first, puts it."""
    import torch

    import dsdecompx_b200 as dsx
    from test_gpu_walk_rule import Address

    n, P = tiles * 512 - 700, 2    # the subdomains' last tiles are not full
    gen = torch.Generator("cuda").manual_seed(tiles)
    x = torch.rand(n, generator=gen, dtype=torch.float64, device="cuda")
    source = (x >= 0.5).long()
    order = torch.sort(source, stable=True)[1]
    x, source = x[order], source[order]
    counts = torch.bincount(source, minlength=P)
    assert int(((counts + 511) // 512).sum()) in (tiles, tiles - 1)
    ids = torch.arange(n, dtype=torch.int32, device="cuda")
    moved = x + 0.01 * torch.randn(n, generator=gen, dtype=torch.float64, device="cuda")
    moved = moved - torch.floor(moved)
    half = torch.full_like(moved, 0.5)
    grid = dsx.VirtualGrid(P, dims=(2, 1, 1), upper=(1.0, 1.0, 1.0), halo_width=0.01, particles=n,
                           ghost_capacity=n // 8)
    torch.cuda.synchronize()
    arrays = {0: moved, 1: half, 2: half, 12: ids}
    grid.upload_flat(counts.cpu().numpy(), [arrays[k].data_ptr() if k in arrays else None for k in range(13)])
    res = grid.migrate()
    dest = (moved >= 0.5).long()
    want = ids[torch.sort(dest * 2 + (dest != source).long(), stable=True)[1]]
    assert (res[:, 5] == torch.bincount(dest, minlength=P).cpu().numpy()).all()
    v = grid.view()
    got = torch.as_tensor(Address(grid, v.base[12] + v.owned_offset * 4, n, "i4"), device="cuda")
    assert torch.equal(got, want)
    grid.close()


@pytest.mark.parametrize("program", ["emigrant_sanity", "join_sanity"])
def test_cpp_programs(cuda, program):
    """tests/cpp/emigrant_sanity.cu: more or fewer leavers than the layout
    counted raise the status bit, and only the counted slots are written.
    tests/cpp/join_sanity.cpp: the first launch after a captured stream was
    joined with another one (as a step's emigrants' branch is) waits for both
    in full, whatever was launched in between."""
    import os
    import subprocess

    import dsdecompx_b200 as dsx
    exe = os.path.join(os.path.dirname(dsx.library_path()), program)
    assert os.path.exists(exe), "tests/cpp programs are built by __graft_entry__.build()"
    proc = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert proc.returncode == 0, proc.stdout + proc.stderr
    assert f"{program}: ok" in proc.stdout
