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
