"""The counted owner search and the one-box wrap at their edges."""
import numpy as np
import pytest

from helpers import Pair, same

pytestmark = pytest.mark.gpu


def edge_values(lower, extent):
    """Multiples of the extent, their neighbors, signed zeros, denormals and
    what is not a number."""
    with np.errstate(all="ignore"):
        out = [np.array([-0.0, 0.0, 5e-324, -5e-324, -1e-310, -1e-200, 1e300, np.nan, np.inf, -np.inf])]
        for k in (-3, -2, -1, 0, 1, 2, 3):
            up = down = k * extent + lower
            for _ in range(4):
                out.append(np.array([up, down]))
                up, down = np.nextafter(up, np.inf), np.nextafter(down, -np.inf)
    return np.concatenate(out)


@pytest.mark.parametrize("lower,extent", [(0.0, 100.0), (-3.7, 11.3), (0.0, 3.0), (5.0, 0.1),
                                          (0.0, 2.0 ** -600), (0.0, 1.7e308), (1e10, 7.0)])
def test_wrap_one_box_away_is_the_divided_wrap(cuda, lower, extent):
    """The wrap without its division against the formula it stands for,
    v - lower - floor((v - lower) / extent) * extent + lower, in IEEE doubles."""
    import torch

    import dsdecompx_b200 as dsx

    upper = lower + extent
    extent = upper - lower
    rng = np.random.default_rng(3)
    with np.errstate(all="ignore"):
        v = np.concatenate([edge_values(lower, extent), rng.uniform(-3, 3, 20_001) * extent + lower,
                            lower - extent * 2.0 ** rng.uniform(-1080, 0, 2_000)])
        t = v - lower
        inside = (t >= 0) & (t < extent)
        want = np.where(inside, np.where(t == 0, 0.0, t) + lower,
                        (t - np.floor(t / extent) * extent) + lower)
    dev = [torch.as_tensor(v, device="cuda").clone() for _ in range(3)]
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    dsx.rank_migrate(*dev, v.size, (lower,) * 3, (upper,) * 3, stream=stream)
    stream.synchronize()
    for d in dev:
        got = d.cpu().numpy()
        nan = np.isnan(want)
        assert (np.isnan(got) == nan).all()
        assert same(got[~nan], want[~nan])


@pytest.mark.parametrize("dims,lower", [((4, 4, 4), 0.0), ((8, 1, 5), 0.0), ((2, 7, 3), -2.5),
                                        ((9, 2, 2), 0.0)])
def test_owner_rank_counts_and_alignments(cuda, dims, lower):
    """Uneven cuts, axes up to the counted length and one past it, positions
    and results off their 16-byte boundaries, odd counts and single ones."""
    import torch

    rng = np.random.default_rng(5)
    L = np.array([12.0, 10.0, 9.0])
    pair = Pair(int(np.prod(dims)), dims, "manual", (lower,) * 3, tuple(lower + L),
                (True, False, True), 0.5, True, None, (), particles=10)
    try:
        cuts = [np.concatenate([[lower], lower + np.sort(rng.uniform(0.02, 0.98, d - 1)) * l, [lower + l]])
                for d, l in zip(dims, L)]
        pair.gpu.set_cuts(cuts)
        pair.ref.set_cuts(cuts)
        flat = np.concatenate(cuts)
        special = np.concatenate([flat, np.nextafter(flat, -np.inf), np.nextafter(flat, np.inf),
                                  *[edge_values(lower, l) for l in L]])
        pos = rng.uniform(lower - 15, lower + 25, size=(5_003, 3))
        pick = rng.random(pos.shape) < 0.4
        pos[pick] = rng.choice(special, pick.sum())
        dev = [torch.as_tensor(np.ascontiguousarray(pos[:, a]), device="cuda") for a in range(3)]
        for first, n in ((0, 5_003), (0, 5_002), (1, 5_001), (2, 1), (3, 2)):
            out = torch.full((5_004,), -7, dtype=torch.int32, device="cuda")
            pair.gpu.owner_rank(*[d[first:first + n] for d in dev], out[first:first + n])
            torch.cuda.synchronize()
            assert (out[first:first + n].cpu().numpy() == pair.ref.owner_rank(pos[first:first + n])).all()
            assert (out[:first] == -7).all() and (out[first + n:] == -7).all()
    finally:
        pair.close()
