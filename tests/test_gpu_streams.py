"""Commits beside other work on the device: a higher-priority stream gets in while a tree is hashed, and commits that
run on several streams at once give the roots that they give one after another."""
import time

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def dev(pkg):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    pkg.init(0)
    yield pkg, torch
    pkg.set_native_hash_family(2)


def _empty(torch, n):
    return torch.empty(n, dtype=torch.int64, device="cuda")


def test_higher_priority_work_enters_a_long_hash_launch(dev):
    """The sponge of 2^20 rows x 256 columns is one launch of some 16 ms; openings at high priority, issued once it runs,
    wait for the CTAs then on the SMs (about 1.2 ms: 22 permutations a tile), not for the launch.  A third of the tree's time
    separates the two; the median of five takes out a descheduled host thread."""
    pkg, torch = dev
    rows, ncols, small = 1 << 20, 256, 1 << 12
    src, tree = _empty(torch, rows * ncols), _empty(torch, pkg.tree_num_elements(rows, 4))
    lde, ltree = _empty(torch, 120 * small), _empty(torch, pkg.tree_num_elements(small, 4))
    for t in (src, lde, ltree):
        pkg.fill_random_device(t, t.numel(), 3)
    q = torch.arange(64, device="cuda")
    out = _empty(torch, 64 * pkg.query_proof_words(small, 120, 4, 0))
    low, high = torch.cuda.Stream(priority=0), torch.cuda.Stream(priority=-1)
    waits, trees = [], []
    for _ in range(6):
        torch.cuda.synchronize()
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record(low)
        pkg.merkletree_device(tree, src, 1, rows, ncols, rows, 4, stream=low)
        b.record(low)
        time.sleep(0.001)
        t0 = time.perf_counter()
        pkg.query_openings_device(out, lde, small, 120, ltree, 4, q, 64, stream=high)
        high.synchronize()
        waits.append((time.perf_counter() - t0) * 1e3)
        low.synchronize()
        trees.append(a.elapsed_time(b))
    assert np.median(waits[1:]) < np.median(trees[1:]) / 3, (waits, trees)
