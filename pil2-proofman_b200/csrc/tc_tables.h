// Byte tables that turn the linear layers of a Poseidon permutation into 8-bit integer matrix
// products (host side; tc_hash.cuh is the kernel that uses them).
//
// A 64-bit word is its eight bytes, so a linear map over GF(p) is an integer matrix over bytes:
//   sum_i c_i x_i = sum_{i,b} byte_b(x_i) * (c_i 2^(8b) mod p)  (mod p),
// and with the constant (c_i 2^(8b) mod p) cut into bytes too, column k of an output word collects
// sum byte_b(x_i) * byte_k(c_i 2^(8b) mod p), an integer below K * 255^2 < 2^24 (K <= 256 input bytes);
// the word is sum_k column_k 2^(8k).  One row of the left matrix is a state as it lies in memory.
//
// A permutation is four full rounds (x^7 on every word, a linear layer, constants), 22 partial rounds
// (x^7 on word 0 only) and four full rounds.  Through the partial rounds everything but the one
// S-box is linear: with y_t the S-box output of partial round t, the S-box input z_t is a linear
// function of the state before and of y_0..y_{t-1}, and so is the state after.  The 22 rounds are taken in
// two blocks of 11 and each block in runs of 6 and 5: a run's z_t come from one matrix product (over the
// block's first state and the earlier run's y) plus the run's own y by a few field multiplications,
// and one product per block gives the state after it.  The layer after the fourth full round is folded
// into the first block.
//
// Scales.  The kernel's S-box uses Montgomery products, S(x) = x^7 2^(-384), so a word that enters it is kept times
// k = 2^(384/7) (the seventh root exists: 7 is prime to p - 1): S(k x) = x^7.  A joined word comes out of one 32-bit
// Montgomery step, times 2^-32.  Both are undone in the tables and constants, so they cost nothing: a layer into an
// S-box is stored times 2^32 k, one that leaves the state (the output, the state between the blocks) times 2^32.
//
// Round structure: poseidon2_goldilocks.cpp:9-41, poseidon_goldilocks.cpp:13-51.
#ifndef PIL2_B200_TC_TABLES_H
#define PIL2_B200_TC_TABLES_H
#include <stdint.h>
#include <string.h>

#include <vector>

#include "poseidon1_constants.h"
#include "poseidon2_constants.h"

namespace tch {

constexpr int BLOCKS = 2, LEN = 11, RUN0 = 6, RUN1 = 5;  // 22 partial rounds = 2 x (6 + 5)
constexpr int NZ = 48;                                  // columns of a run's product: 6 words
constexpr int YCH = 6;                                  // 16-byte chunks of a block's y rows (12 words)
constexpr int NQ = RUN0 * (RUN0 - 1) / 2 + RUN1 * (RUN1 - 1) / 2;

// Table sizes and offsets of width W.  A table of N columns and K input bytes is stored as the matrix unit
// reads it: 16-byte pieces of a column's bytes, [K/16][N][16].
template <int W>
struct Shape {
    static constexpr int KX = 8 * W;  // bytes of a state
    static constexpr int CHX = W / 2;
    static constexpr int K_Z0 = KX, K_Z1 = KX + 64, K_U = KX + 96;  // y_0..y_7 (6 used), y_0..y_11 (11 used)
    static constexpr int NF = 32;    // columns of the output's product: 4 words
    static constexpr int OFF_L = 0;
    static constexpr int SIZE_L = KX * KX, SIZE_Z0 = NZ * K_Z0, SIZE_Z1 = NZ * K_Z1, SIZE_U = KX * K_U;
    static constexpr int BLOCK = SIZE_Z0 + SIZE_Z1 + SIZE_U, SIZE_F = NF * KX;
    static constexpr int OFF_Z0 = SIZE_L, OFF_Z1 = OFF_Z0 + SIZE_Z0, OFF_U = OFF_Z1 + SIZE_Z1;  // + b * BLOCK
    static constexpr int OFF_F = SIZE_L + BLOCKS * BLOCK;
    static constexpr int BYTES = OFF_F + SIZE_F;
};
constexpr int MAX_BYTES = Shape<16>::BYTES;

// Words added after the products, and the field multipliers inside a run.
struct Consts {
    uint64_t lay[9][16];       // 0 before round 1; 1-3 after rounds 1-3; 4, 5 after the blocks; 6-8 after rounds 5-7
    uint64_t z[BLOCKS][LEN];   // added to z_t
    uint64_t q[BLOCKS][NQ];    // z_t += q y_u: run 0 t = 1..5, u < t, then run 1
};

namespace detail {

constexpr uint64_t P = 0xFFFFFFFF00000001ULL;
inline uint64_t mul(uint64_t a, uint64_t b) { return (uint64_t)((unsigned __int128)a * b % P); }
inline uint64_t add(uint64_t a, uint64_t b) { return (uint64_t)(((unsigned __int128)a + b) % P); }

typedef std::vector<uint64_t> Vec;  // coefficients over (state words, y_0..y_10, 1)

inline uint64_t power(uint64_t b, uint64_t e)
{
    uint64_t r = 1;
    for (; e; e >>= 1, b = mul(b, b))
        if (e & 1) r = mul(r, b);
    return r;
}

inline void axpy(Vec &d, uint64_t c, const Vec &s)
{
    for (size_t i = 0; i < d.size(); i++) d[i] = add(d[i], mul(c, s[i]));
}

// bytes of column word `out` of a table (K input bytes, N columns) for input word `word`
inline void put(uint8_t *tab, int N, int word, int out, uint64_t coef)
{
    for (int b = 0; b < 8; b++) {
        const int kb = 8 * word + b;
        const uint64_t c = mul(coef, (uint64_t)1 << (8 * b));
        for (int k = 0; k < 8; k++) tab[(size_t)(kb >> 4) * N * 16 + (8 * out + k) * 16 + (kb & 15)] = (uint8_t)(c >> (8 * k));
    }
}

template <int W> struct Raw;
template <> struct Raw<8> {
    static const uint64_t *C2() { static const uint64_t v[] = {P2_C8_LIST}; return v; }
    static const uint64_t *D2() { static const uint64_t v[] = {P2_D8_LIST}; return v; }
    static const uint64_t *C1() { static const uint64_t v[] = {P1_C8_LIST}; return v; }
    static const uint64_t *M1() { static const uint64_t v[] = {P1_M8_LIST}; return v; }
    static const uint64_t *P1() { static const uint64_t v[] = {P1_P8_LIST}; return v; }
    static const uint64_t *S1() { static const uint64_t v[] = {P1_S8_LIST}; return v; }
};
template <> struct Raw<12> {
    static const uint64_t *C2() { static const uint64_t v[] = {P2_C12_LIST}; return v; }
    static const uint64_t *D2() { static const uint64_t v[] = {P2_D12_LIST}; return v; }
    static const uint64_t *C1() { static const uint64_t v[] = {P1_C12_LIST}; return v; }
    static const uint64_t *M1() { static const uint64_t v[] = {P1_M12_LIST}; return v; }
    static const uint64_t *P1() { static const uint64_t v[] = {P1_P12_LIST}; return v; }
    static const uint64_t *S1() { static const uint64_t v[] = {P1_S12_LIST}; return v; }
};
template <> struct Raw<16> {
    static const uint64_t *C2() { static const uint64_t v[] = {P2_C16_LIST}; return v; }
    static const uint64_t *D2() { static const uint64_t v[] = {P2_D16_LIST}; return v; }
    static const uint64_t *C1() { static const uint64_t v[] = {P1_C16_LIST}; return v; }
    static const uint64_t *M1() { static const uint64_t v[] = {P1_M16_LIST}; return v; }
    static const uint64_t *P1() { static const uint64_t v[] = {P1_P16_LIST}; return v; }
    static const uint64_t *S1() { static const uint64_t v[] = {P1_S16_LIST}; return v; }
};

}  // namespace detail

// Tables (Shape<W>::BYTES bytes at tab) and constants of hash family fam (1 Poseidon1, 2 Poseidon2).
template <int W>
inline void build_tables(int fam, uint8_t *tab, Consts &c)
{
    using namespace detail;
    typedef Shape<W> S;
    memset(tab, 0, S::BYTES);
    memset(&c, 0, sizeof(c));
    const int NP = BLOCKS * LEN;
    // 1/7 mod p - 1: the smallest (1 + j (p - 1)) / 7
    uint64_t seventh = 0;
    for (unsigned __int128 j = 1; j < 7; j++)
        if ((1 + j * (P - 1)) % 7 == 0) seventh = (uint64_t)((1 + j * (P - 1)) / 7);
    const uint64_t two32 = 1ull << 32, k = power(power(two32, 12), seventh), k32 = mul(k, two32);
    // full-round layer L (out_i = sum_j L[i][j] x_j) and the layer L4 after the fourth round
    static const int M4[4][4] = {{5, 7, 1, 3}, {4, 6, 1, 1}, {1, 3, 5, 7}, {1, 1, 4, 6}};
    std::vector<Vec> L(W, Vec(W)), L4(W, Vec(W));
    for (int i = 0; i < W; i++)
        for (int j = 0; j < W; j++) {
            L[i][j] = fam == 1 ? Raw<W>::M1()[j * W + i] : (uint64_t)M4[i & 3][j & 3] * (i / 4 == j / 4 ? 2 : 1);
            L4[i][j] = fam == 1 ? Raw<W>::P1()[j * W + i] : L[i][j];
        }
    for (int i = 0; i < W; i++)
        for (int j = 0; j < W; j++) put(tab + S::OFF_L, S::KX, j, i, mul(k32, L[i][j]));
    for (int i = 0; i < 4; i++)
        for (int j = 0; j < W; j++) put(tab + S::OFF_F, S::NF, j, i, mul(two32, L[i][j]));
    // constants of the full rounds: Poseidon2 adds them before the S-boxes, Poseidon1 after them (so they
    // pass through the next layer) and once before round 1
    auto through = [&](const std::vector<Vec> &m, const uint64_t *k, uint64_t *out) {
        for (int i = 0; i < W; i++) {
            uint64_t a = 0;
            for (int j = 0; j < W; j++) a = add(a, mul(m[i][j], k[j]));
            out[i] = a;
        }
    };
    const uint64_t *C = fam == 1 ? Raw<W>::C1() : Raw<W>::C2();
    Vec post(W, 0);  // Poseidon1: constants entering the state with the layer after round 4
    for (int i = 0; i < W; i++) c.lay[0][i] = C[i];
    for (int r = 1; r <= 3; r++) {
        if (fam == 1)
            through(L, C + r * W, c.lay[r]);
        else
            for (int i = 0; i < W; i++) c.lay[r][i] = C[r * W + i];
        const uint64_t *k2 = fam == 1 ? C + 5 * W + NP + (r - 1) * W : C + 4 * W + NP + r * W;
        if (fam == 1)
            through(L, k2, c.lay[5 + r]);
        else
            for (int i = 0; i < W; i++) c.lay[5 + r][i] = k2[i];
    }
    if (fam == 1) through(L4, C + 4 * W, post.data());
    for (int b = 0; b < BLOCKS; b++) {
        const int ONE = W + LEN;
        std::vector<Vec> x(W, Vec(ONE + 1, 0)), z(LEN);
        for (int i = 0; i < W; i++) {
            if (b == 0) {
                for (int j = 0; j < W; j++) x[i][j] = L4[i][j];
                x[i][ONE] = post[i];
            } else {
                x[i][i] = 1;
            }
        }
        for (int t = 0; t < LEN; t++) {
            const int pr = b * LEN + t;
            z[t] = x[0];
            Vec y(ONE + 1, 0);
            y[W + t] = 1;
            if (fam == 1) {
                const uint64_t *Sr = Raw<W>::S1() + (2 * W - 1) * pr;
                y[ONE] = C[5 * W + pr];
                Vec x0(ONE + 1, 0);
                axpy(x0, Sr[0], y);
                for (int i = 1; i < W; i++) axpy(x0, Sr[i], x[i]);
                for (int i = 1; i < W; i++) axpy(x[i], Sr[W - 1 + i], y);
                x[0] = x0;
            } else {
                z[t][ONE] = add(z[t][ONE], C[4 * W + pr]);
                Vec sum = y;
                for (int i = 1; i < W; i++) axpy(sum, 1, x[i]);
                for (int i = 0; i < W; i++) {
                    Vec n = sum;
                    axpy(n, Raw<W>::D2()[i], i == 0 ? y : x[i]);
                    x[i] = n;
                }
            }
        }
        uint8_t *blk = tab + b * S::BLOCK, *z0 = blk + S::OFF_Z0, *z1 = blk + S::OFF_Z1, *u = blk + S::OFF_U;
        int nq = 0;
        for (int t = 0; t < LEN; t++) {
            const int first = t < RUN0 ? 0 : RUN0;
            uint8_t *zt = t < RUN0 ? z0 : z1;
            // a run's first z is a joined word; the others also add the run's own y and are reduced as a whole
            const uint64_t sc = t == first ? k32 : k;
            for (int j = 0; j < W; j++) put(zt, NZ, j, t - first, mul(sc, z[t][j]));
            for (int v = 0; v < first; v++) put(zt, NZ, W + v, t - first, mul(sc, z[t][W + v]));
            for (int v = first; v < t; v++) c.q[b][nq++] = mul(k, z[t][W + v]);
            c.z[b][t] = mul(k, z[t][ONE]);
        }
        for (int i = 0; i < W; i++) {
            const uint64_t sc = b == 1 ? k32 : two32;
            for (int j = 0; j < W; j++) put(u, S::KX, j, i, mul(sc, x[i][j]));
            for (int v = 0; v < LEN; v++) put(u, S::KX, W + v, i, mul(sc, x[i][W + v]));
            c.lay[4 + b][i] = x[i][ONE];
            if (b == 1 && fam != 1) c.lay[5][i] = add(c.lay[5][i], C[4 * W + NP + i]);
        }
    }
    // scale the added words (the first constants of Poseidon1 are added before a plain x^7)
    for (int l = fam == 1 ? 1 : 0; l < 9; l++)
        for (int i = 0; i < W; i++)
            if (l != 4) c.lay[l][i] = mul(k, c.lay[l][i]);
}

}  // namespace tch
#endif
