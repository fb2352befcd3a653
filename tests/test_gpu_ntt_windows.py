"""LDE windows at their switch points against the oracle, over every 64-bit word.

Transform lengths around the first window's limits (2^11 to 2^13 points, with the blowup's copy lanes in a
full tile, in a partial one and alone), lengths whose windows leave every remainder phase (1 to 3 stages), blowup 1 (the
forward transform reads the inverse's words as they are), and inputs that are all 2^64 - 1, all p, p - 1 or random
words with those among them: the butterflies leave out canonicalisations that these would need.
"""
import numpy as np
import pytest

import oracle

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(pkg):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg.init(0)
    return pkg, torch


CASES = [(n, n + b) for n in range(1, 12) for b in (0, 1, 3)] + [(12, 12), (11, 13), (12, 13), (12, 14), (13, 13), (13, 14),
                                                                 (10, 14), (14, 15), (15, 17), (16, 17)]


@pytest.mark.parametrize("nbits,nbits_ext", CASES)
def test_lde_over_all_words(dev, orc, nbits, nbits_ext):
    pkg, torch = dev
    n, p = 1 << nbits, oracle.P
    rng = np.random.RandomState(nbits * 31 + nbits_ext)
    mixed = rng.randint(0, 1 << 63, n).astype(np.uint64) * np.uint64(2) + rng.randint(0, 2, n).astype(np.uint64)
    edge = np.array([2**64 - 1, 2**64 - 2**32, p, p - 1, p + 1, 2**32 - 1, 2**32, 0], dtype=np.uint64)
    pick = rng.randint(0, 3, n) == 0
    mixed[pick] = edge[rng.randint(0, 8, int(pick.sum()))]
    m = np.stack([np.full(n, 2**64 - 1, np.uint64), np.full(n, p, np.uint64), np.full(n, p - 1, np.uint64), mixed,
                  edge[rng.randint(0, 8, n)]], axis=1)
    exp = orc.lde(m % np.uint64(p), nbits_ext)
    ncols = m.shape[1]
    d_trace = torch.from_numpy(np.ascontiguousarray(m).view(np.int64)).cuda()
    d_lde = torch.full((ncols, 1 << nbits_ext), -1, dtype=torch.int64, device="cuda")
    d_scr = torch.empty(pkg.lde_scratch_words(nbits, ncols), dtype=torch.int64, device="cuda")
    pkg.lde_device(d_lde, d_trace, nbits, nbits_ext, ncols, d_scr)
    torch.cuda.synchronize()
    got = d_lde.cpu().numpy().view(np.uint64).T
    assert (got == exp).all(), (nbits, nbits_ext, np.argwhere(got != exp)[:4])


# Both sides of the rule for first windows that fill no tile (one copy lane a CTA, or all of them): 2048 CTAs below 2^5
# points, 4096 from there, no limit from 2^9.
EDGES = [(1, 8, 16), (1, 8, 17), (2, 4, 512), (2, 4, 513), (4, 8, 128), (4, 8, 129), (5, 12, 32), (5, 12, 33), (8, 12, 256),
         (8, 12, 257), (9, 12, 513)]


@pytest.mark.parametrize("nbits,nbits_ext,ncols", EDGES)
def test_lde_at_the_lane_rule(dev, orc, nbits, nbits_ext, ncols):
    pkg, torch = dev
    rng = np.random.RandomState(nbits * 31 + ncols)
    m = rng.randint(0, 1 << 63, (1 << nbits, ncols)).astype(np.uint64) * np.uint64(2) + np.uint64(1)
    m[:, ::3] = np.uint64(2**64 - 1)
    m[::2, 1::3] = np.uint64(oracle.P)
    exp = orc.lde(m % np.uint64(oracle.P), nbits_ext)
    d_trace = torch.from_numpy(np.ascontiguousarray(m).view(np.int64)).cuda()
    d_lde = torch.full((ncols, 1 << nbits_ext), -1, dtype=torch.int64, device="cuda")
    d_scr = torch.empty(pkg.lde_scratch_words(nbits, ncols), dtype=torch.int64, device="cuda")
    pkg.lde_device(d_lde, d_trace, nbits, nbits_ext, ncols, d_scr)
    torch.cuda.synchronize()
    got = d_lde.cpu().numpy().view(np.uint64).T
    assert (got == exp).all(), np.argwhere(got != exp)[:4]


def test_few_rows_at_a_high_blowup_take_no_longer(dev):
    """2^1 -> 2^8 writes what 2^7 -> 2^8 does with fewer stages; with a CTA of two points a copy lane it took three times
    as long (41 us against 13).  Best of several runs each."""
    pkg, torch = dev
    ncols, next_ = 512, 1 << 8
    lde = torch.empty(ncols * next_, dtype=torch.int64, device="cuda")

    def best(nbits):
        trace = torch.zeros(ncols << nbits, dtype=torch.int64, device="cuda")
        scr = torch.empty(pkg.lde_scratch_words(nbits, ncols), dtype=torch.int64, device="cuda")
        ms = []
        for _ in range(8):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for _ in range(20):
                pkg.lde_device(lde, trace, nbits, 8, ncols, scr, trace_rowmajor=False)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms[1:])

    few, many = best(1), best(7)
    assert few < 1.5 * many, (few, many)
