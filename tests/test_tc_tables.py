"""The byte tables of the tensor core permutations (csrc/tc_tables.h), on the host.

A plain C++ walk through the tables, with the kernel's own arithmetic (byte products, column pairs, the
32-bit and 64-bit Montgomery steps), must give the oracle's permutation for every width and family, and
the bounds the kernel relies on must hold for the largest bytes: every column pair below 2^31, and added
constants that leave room for the joined word.
"""
import os
import shutil
import subprocess
import tempfile

import numpy as np
import pytest

import oracle

REPO = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

DRIVER = r"""
#include <cstdio>
#include <cstdlib>
#include "tc_tables.h"
using namespace tch;
using detail::add;
using detail::mul;
typedef uint64_t u64;
typedef uint32_t u32;
static const u64 EPS = 0xffffffffu;

static u64 mont(u64 x, u64 y)
{
    const unsigned __int128 v = (unsigned __int128)x * y;
    const u64 lo = (u64)v, hi = (u64)(v >> 64), a = lo + (lo << 32), e = a < lo, b = a - (a >> 32) - e, r = hi - b;
    return hi < b ? r - EPS : r;
}
static u64 mont_pow7(u64 x) { const u64 x2 = mont(x, x), x3 = mont(x2, x), x4 = mont(x2, x2); return mont(x3, x4); }
static u64 pow7(u64 x) { const u64 x2 = mul(x, x), x3 = mul(x2, x), x4 = mul(x2, x2); return mul(x3, x4); }

static void pairs(const uint8_t *tab, int N, int K, const u64 *words, int out, u32 *t)
{
    for (int i = 0; i < 4; i++) {
        u64 v = 0;
        for (int h = 0; h < 2; h++) {
            u64 c = 0;
            for (int b = 0; b < K; b++)
                c += ((words[b / 8] >> (8 * (b % 8))) & 255) * tab[(size_t)(b >> 4) * N * 16 + (8 * out + 2 * i + h) * 16 + (b & 15)];
            v += c << (8 * h);
        }
        if (v >> 31) { std::printf("FAIL pair bound\n"); std::exit(1); }
        t[i] = (u32)v;
    }
}
static u64 join_word(const u32 *t, u64 c)
{
    if (c >= 0 - (1ull << 50)) { std::printf("FAIL constant headroom\n"); std::exit(1); }
    const u64 x = (u64)t[0] + (u32)(t[1] << 16);
    const u32 x0 = (u32)x, u = t[2] + (t[1] >> 16) + (u32)(x >> 32);
    const u64 y = (u64)t[3] * 65536 + c + u + x0, s = (u64)x0 << 32;
    return y < s ? y - s - EPS : y - s;
}

template <int W>
static void permute(int fam, u64 *s)
{
    typedef Shape<W> S;
    std::vector<uint8_t> tab(S::BYTES);
    Consts c;
    build_tables<W>(fam, tab.data(), c);
    u64 w[W + 12];
    u32 t4[4];
    for (int i = 0; i < W + 12; i++) w[i] = i < W ? s[i] : ~0ull;  // y rows not written yet: any bytes
    auto layer = [&](int off, int K, const u64 *k, bool sbox) {
        u64 o[W];
        for (int i = 0; i < W; i++) {
            pairs(tab.data() + off, S::KX, K, w, i, t4);
            o[i] = join_word(t4, k[i]);
            if (sbox) o[i] = mont_pow7(o[i]);
        }
        for (int i = 0; i < W; i++) w[i] = o[i];
    };
    if (fam == 1)
        for (int i = 0; i < W; i++) w[i] = pow7(add(w[i] % detail::P, c.lay[0][i]));
    for (int l = fam == 1 ? 1 : 0; l < 9; l++) {
        if (l != 4 && l != 5) {
            layer(S::OFF_L, S::KX, c.lay[l], true);
            continue;
        }
        const int b = l - 4;
        int nq = 0;
        for (int run = 0; run < 2; run++)
            for (int f = run ? RUN0 : 0, n = run ? RUN1 : RUN0, t = 0; t < n; t++) {
                pairs(tab.data() + b * S::BLOCK + (run ? S::OFF_Z1 : S::OFF_Z0), NZ, run ? S::K_Z1 : S::K_Z0, w, t, t4);
                u64 z;
                if (t == 0) {
                    z = join_word(t4, c.z[b][f]);
                } else {
                    unsigned __int128 v = 0;
                    for (int i = 3; i >= 0; i--) v = (v << 16) + t4[i];
                    z = add((u64)(v % detail::P), c.z[b][f + t]);
                    for (int u = 0; u < t; u++) z = add(z, mul(c.q[b][nq++], w[W + f + u]));
                }
                w[W + f + t] = mont_pow7(z);
            }
        layer(S::OFF_U + b * S::BLOCK, S::K_U, c.lay[l], b == 1);
    }
    for (int i = 0; i < 4; i++) {
        pairs(tab.data() + S::OFF_F, S::NF, S::KX, w, i, t4);
        s[i] = join_word(t4, 0) % detail::P;
    }
    // the largest bytes: pairs() checks every column pair of every table
    for (int i = 0; i < W + 12; i++) w[i] = ~0ull;
    for (int i = 0; i < W; i++) {
        pairs(tab.data() + S::OFF_L, S::KX, S::KX, w, i, t4);
        for (int b = 0; b < BLOCKS; b++) pairs(tab.data() + b * S::BLOCK + S::OFF_U, S::KX, S::K_U, w, i, t4);
    }
    for (int b = 0; b < BLOCKS; b++)
        for (int t = 0; t < 6; t++) {
            pairs(tab.data() + b * S::BLOCK + S::OFF_Z0, NZ, S::K_Z0, w, t, t4);
            pairs(tab.data() + b * S::BLOCK + S::OFF_Z1, NZ, S::K_Z1, w, t, t4);
        }
}

int main(int argc, char **argv)
{
    const int W = std::atoi(argv[1]), fam = std::atoi(argv[2]);
    u64 s[16];
    for (int i = 0; i < W; i++) s[i] = std::strtoull(argv[3 + i], nullptr, 10);
    if (W == 8) permute<8>(fam, s);
    if (W == 12) permute<12>(fam, s);
    if (W == 16) permute<16>(fam, s);
    for (int i = 0; i < 4; i++) std::printf("%llu ", (unsigned long long)s[i]);
    return 0;
}
"""


@pytest.fixture(scope="module")
def binary():
    cxx = shutil.which("g++")
    if not cxx:
        pytest.skip("no host C++ compiler")
    with tempfile.TemporaryDirectory() as d:
        src, exe = os.path.join(d, "t.cpp"), os.path.join(d, "t")
        with open(src, "w") as f:
            f.write(DRIVER)
        subprocess.run([cxx, "-O2", "-std=c++17", "-I", os.path.join(REPO, "pil2-proofman_b200", "csrc"), "-o", exe, src],
                       check=True)
        yield exe


@pytest.mark.parametrize("family", [1, 2])
@pytest.mark.parametrize("width", [8, 12, 16])
def test_tables_give_the_permutation(binary, width, family):
    orc = oracle.Oracle(family=family)
    states = [oracle.random_field((width,), 5), np.zeros(width, np.uint64), np.full(width, oracle.P - 1, np.uint64),
              np.full(width, 2**64 - 1, np.uint64)]
    for s in states:
        out = subprocess.run([binary, str(width), str(family)] + [str(int(x)) for x in s], capture_output=True, text=True)
        assert out.returncode == 0, out.stdout
        exp = orc.permute(s % np.uint64(oracle.P))[:4]
        assert [int(x) for x in out.stdout.split()] == [int(x) for x in exp]
