"""The tensor core hashing kernels (tc_hash.cuh) against the oracle, above the cooperative kernels' range.

Edges: the first row counts past that range (4096; 8192 at arity 2), one row into a new 128-row tile, one tile more than the resident groups (148 SMs x 4), sponges of no,
one and more blocks with a full and a ragged last one, both strides, a tree at an odd word of its buffer
(8-byte stores), words from 0 to 2^64 - 1, and a level whose last parent has missing children.
Whole trees are compared, bit for bit.
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
    yield pkg, torch
    pkg.set_native_hash_family(2)
    assert pkg.load().b200_tma_wait_errors() == 0  # no bounded wait ran out


# rows, columns in sponge blocks (blocks, extra columns)
ROWS = [4097, 8193, 8320, 148 * 4 * 128 + 1]
COLS = [(0, 0), (1, 0), (1, 1), (2, -1)]


@pytest.mark.parametrize("family", [1, 2])
@pytest.mark.parametrize("arity", [2, 3, 4])
@pytest.mark.parametrize("nrows", ROWS)
def test_tree_at_the_tiles_edges(dev, arity, family, nrows):
    pkg, torch = dev
    orc = oracle.Oracle(family=family)
    pkg.set_native_hash_family(family)
    rate = 4 * arity - 4
    blocks, extra = COLS[(nrows + arity + family) % len(COLS)]
    for k, (b, x) in enumerate([(blocks, extra), (1, 0)]):
        ncols = b * rate + x
        m = oracle.random_field((nrows, ncols), nrows + ncols + family)
        if ncols:
            m[0] = np.uint64(2**64 - 1)
            m[-1] = np.uint64(oracle.P - 1)
        exp = orc.merkletree(m % np.uint64(oracle.P), arity)
        colmajor = k == 0
        src = np.ascontiguousarray(m.T if colmajor else m)
        d_src = torch.from_numpy((src if src.size else np.zeros(1, np.uint64)).view(np.int64)).cuda()
        buf = torch.zeros(exp.size + 1, dtype=torch.int64, device="cuda")
        tree = buf[k:k + exp.size]  # the second at an odd word
        rs, cs = (1, nrows) if colmajor else (ncols, 1)
        pkg.merkletree_device(tree, d_src, rs, cs, ncols, nrows, arity)
        torch.cuda.synchronize()
        bad = np.nonzero(tree.cpu().numpy().view(np.uint64) != exp)[0]
        assert bad.size == 0, (nrows, ncols, arity, family, bad[:8])


# Every sponge shape at every width and family, and three blocks with a ragged last one.
@pytest.mark.parametrize("family", [1, 2])
@pytest.mark.parametrize("arity", [2, 3, 4])
@pytest.mark.parametrize("blocks,extra", COLS + [(3, 1), (4, -1)])
def test_sponge_shapes(dev, arity, family, blocks, extra):
    pkg, torch = dev
    orc = oracle.Oracle(family=family)
    pkg.set_native_hash_family(family)
    nrows, ncols = 8320, blocks * (4 * arity - 4) + extra
    m = oracle.random_field((nrows, ncols), ncols + 10 * arity + family)
    if ncols:
        m[0], m[-1] = np.uint64(2**64 - 1), np.uint64(oracle.P - 1)
    exp = orc.merkletree(m % np.uint64(oracle.P), arity)
    d_src = torch.from_numpy((m.reshape(-1) if m.size else np.zeros(1, np.uint64)).view(np.int64)).cuda()
    tree = torch.zeros(exp.size, dtype=torch.int64, device="cuda")
    pkg.merkletree_device(tree, d_src, ncols, 1, ncols, nrows, arity)
    torch.cuda.synchronize()
    bad = np.nonzero(tree.cpu().numpy().view(np.uint64) != exp)[0]
    assert bad.size == 0, bad[:8]


# CTAs of one group up to a tile an SM at widths 8 and 12, of two up to two tiles at width 8: the last rows of each and the next.
@pytest.mark.parametrize("family", [1, 2])
@pytest.mark.parametrize("arity,nrows", [(2, 148 * 128), (2, 148 * 128 + 1), (2, 2 * 148 * 128), (2, 2 * 148 * 128 + 1),
                                         (3, 148 * 128), (3, 148 * 128 + 1)])
def test_tree_at_the_group_rule(dev, arity, nrows, family):
    pkg, torch = dev
    orc = oracle.Oracle(family=family)
    pkg.set_native_hash_family(family)
    ncols = 4 * arity - 3
    m = oracle.random_field((nrows, ncols), nrows + family)
    exp = orc.merkletree(m, arity)
    d_src = torch.from_numpy(np.ascontiguousarray(m.T).view(np.int64)).cuda()
    tree = torch.zeros(exp.size, dtype=torch.int64, device="cuda")
    pkg.merkletree_device(tree, d_src, 1, nrows, ncols, nrows, arity)
    torch.cuda.synchronize()
    bad = np.nonzero(tree.cpu().numpy().view(np.uint64) != exp)[0]
    assert bad.size == 0, bad[:8]


# One tile past a whole wave of CTAs that take a single tile a group (16 permutations a row and more), and past one of
# CTAs that take two (8 permutations): the next wave's first CTA, with one group at work.
@pytest.mark.parametrize("arity,nrows,blocks", [(4, 148 * 4 * 128 + 1, 17), (2, 148 * 8 * 128 + 1, 16),
                                                (3, 2 * 148 * 4 * 128 + 1, 8)])
def test_tree_past_a_wave(dev, orc, arity, nrows, blocks):
    pkg, torch = dev
    pkg.set_native_hash_family(2)
    ncols = blocks * (4 * arity - 4) - 1
    m = oracle.random_field((nrows, ncols), nrows)
    exp = orc.merkletree(m, arity)
    d_src = torch.from_numpy(np.ascontiguousarray(m.T).view(np.int64)).cuda()
    tree = torch.zeros(exp.size, dtype=torch.int64, device="cuda")
    pkg.merkletree_device(tree, d_src, 1, nrows, ncols, nrows, arity)
    torch.cuda.synchronize()
    bad = np.nonzero(tree.cpu().numpy().view(np.uint64) != exp)[0]
    assert bad.size == 0, bad[:8]


# Levels by subtrees of the tree (coop.cuh): one CTA's last parent and one more (16, 9, 32 parents at arity 4, 3, 2), a
# launch's top level ending on one digest or leaving two, and missing children at every level.
LEVELS = [(4, n) for n in (2, 4, 5, 63, 64, 65, 255, 257, 1025, 4096, 4099, 16384)] + \
    [(3, n) for n in (2, 3, 4, 27, 28, 81, 82, 730, 6562)] + [(2, n) for n in (2, 3, 64, 65, 127, 2049, 16384, 16387)]


@pytest.mark.parametrize("family", [1, 2])
@pytest.mark.parametrize("arity,nrows", LEVELS)
def test_levels_by_subtrees(dev, arity, nrows, family):
    pkg, torch = dev
    orc = oracle.Oracle(family=family)
    pkg.set_native_hash_family(family)
    digests = oracle.random_field((nrows, 4), nrows + arity)
    digests[0] = np.uint64(oracle.P - 1)
    tree = torch.zeros(pkg.tree_num_elements(nrows, arity), dtype=torch.int64, device="cuda")
    tree[:4 * nrows] = torch.from_numpy(digests.reshape(-1).view(np.int64)).cuda()
    pkg.merkletree_reduce_device(tree[:4 * nrows].clone(), nrows, arity, tree)
    torch.cuda.synchronize()
    got = tree.cpu().numpy().view(np.uint64)
    level, at = digests.reshape(-1), 0
    while level.size > 4:
        n = level.size // 4
        level = np.concatenate([level, np.zeros(4 * (-n % arity), np.uint64)])
        assert (got[at:at + level.size] == level).all(), (arity, nrows, n)
        at += level.size
        level = np.concatenate([orc.permute(level[i:i + 4 * arity])[:4] for i in range(0, level.size, 4 * arity)])
    assert (got[at:at + 4] == level).all()
