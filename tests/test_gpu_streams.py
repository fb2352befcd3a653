"""Commits beside other work on the device: a higher-priority stream gets in while a tree is hashed, and commits that
run on several streams at once give the roots that they give one after another."""
import threading
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


# log2 rows, log2 extended rows, columns, arity: cooperative and tiled sponges of every width, on an SM's whole tensor memory
SHAPES = [(8, 9, 20, 4), (12, 13, 40, 4), (13, 14, 30, 2), (12, 13, 25, 3), (14, 15, 13, 4), (11, 14, 9, 2)]


@pytest.mark.parametrize("family", [1, 2])
def test_commits_on_several_streams(dev, family):
    """Six commits at once, each on its stream and from its own host thread, several times over."""
    pkg, torch = dev
    pkg.set_native_hash_family(family)
    work = []
    for i, (nb, nbe, nc, ar) in enumerate(SHAPES):
        trace = _empty(torch, nc << nb)
        pkg.fill_random_device(trace, trace.numel(), 50 + i)
        work.append((trace, _empty(torch, nc << nb), _empty(torch, nc << nbe), _empty(torch, pkg.tree_num_elements(1 << nbe, ar))))

    def commit(i, stream, want_root):
        nb, nbe, nc, ar = SHAPES[i]
        trace, scratch, lde, tree = work[i]
        return pkg.commit_device(lde, tree, trace, nb, nbe, nc, ar, scratch, stream=stream, want_root=want_root)

    alone = [commit(i, None, True) for i in range(len(SHAPES))]
    trees = [w[3].clone() for w in work]
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in SHAPES]
    roots = [None] * len(SHAPES)

    def worker(i):
        work[i][3].fill_(-1)
        torch.cuda.current_stream().synchronize()
        for _ in range(3):
            commit(i, streams[i], False)
        roots[i] = commit(i, streams[i], True)

    threads = [threading.Thread(target=worker, args=(i,)) for i in range(len(SHAPES))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    torch.cuda.synchronize()
    for i in range(len(SHAPES)):
        assert (roots[i] == alone[i]).all(), SHAPES[i]
        assert torch.equal(work[i][3], trees[i]), SHAPES[i]
    assert pkg.load().b200_tma_wait_errors() == 0


def test_small_launches_share_the_sms(dev):
    """Eight streams of arity-2 commits whose sponges are 128 tiles each: CTAs of one group share an SM, so they take
    0.42 of the time of the same commits on one stream; while a CTA of eight groups took the SM for one tile, 0.72."""
    pkg, torch = dev
    pkg.set_native_hash_family(2)
    nb, nbe, nc, ar, n = 13, 14, 100, 2, 8
    work = [(_empty(torch, nc << nb), _empty(torch, nc << nb), _empty(torch, nc << nbe),
             _empty(torch, pkg.tree_num_elements(1 << nbe, ar))) for _ in range(n)]
    for i, w in enumerate(work):
        pkg.fill_random_device(w[0], w[0].numel(), i)
    torch.cuda.synchronize()
    streams = [torch.cuda.Stream() for _ in range(n)]
    main = torch.cuda.current_stream()

    def run(over):
        ms = []
        for _ in range(6):
            a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
            a.record()
            for s in over:
                s.wait_event(a)
            for k in range(3 * n):
                trace, scratch, lde, tree = work[k % n]
                pkg.commit_device(lde, tree, trace, nb, nbe, nc, ar, scratch, stream=over[k % n % len(over)], want_root=False)
            for s in over:
                main.wait_stream(s)
            b.record()
            torch.cuda.synchronize()
            ms.append(a.elapsed_time(b))
        return min(ms[1:])

    together, apart = run(streams), run(streams[:1])
    assert together < 0.57 * apart, (together, apart)
