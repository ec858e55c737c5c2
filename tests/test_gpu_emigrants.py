"""Both ways of placing emigrants (one CTA per destination up to 1,024 tiles,
the chain of kernels beyond) and the counters around them, against the oracle:
list lengths around the four entries a thread reads, more immigrants than one
pass of a CTA takes, tile counts around the scan's rows, and few enough
subdomains for copies of the immigrant counters."""
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
