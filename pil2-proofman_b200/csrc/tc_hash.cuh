// Poseidon permutations with the linear layers on the tensor cores (8-bit integer tcgen05.mma).
//
// The tables of tc_tables.h turn every linear layer (the external / MDS layers of the full rounds, and all
// of the partial rounds but their S-boxes) into products of a state's bytes with a constant byte matrix.
// One group of 256 threads (128 at width 8) owns 128 states: the states' bytes are the 128 rows of the left operand in shared
// memory (16-byte piece c of row r at c * 2048 + r * 16, so a thread's 16-byte accesses are conflict-free and
// a state word is stored as it is), the accumulators are the 128 lanes of tensor memory, and a thread reads
// its row's columns back and joins them to 64-bit words (join_word).
//
// What bounds it: the S-boxes' integer products (150 x^7 a width-16 permutation, at 0.82 clocks an SM each in a loop of
// nothing else 122 of the 206 clocks a permutation takes on a B200; IMAD.WIDE issues 25 lanes a clock and SM).  The
// tensor pipe is 13 % busy, so no product is shaped for it: every layer goes through, also those with small coefficients, because
// joining eight columns costs a third of the 128-bit sums that it replaces.  The S-boxes and joins run in
// Montgomery form because that reduction needs no multiplication (gl64.cuh).
//
// At width 12 and 16 a CTA is four groups, one CTA an SM (fewer groups where a launch has few tiles, few_groups): the
// tables take 106 KB of shared memory at width 16, each group 28 KB and a quarter of the tensor memory (128 columns, a
// whole layer's).  Two threads share a row (each takes half its words, and every other run of partial rounds), so 32 warps hide the barriers and latencies: 1000 rows of
// 40 columns take 16 % less than with one thread a row, large launches the same.  At width 8 a layer has 64
// columns and the tables take 44 KB, so eight groups fit with one thread a row: 2^20 rows x 64 columns 7.5 -> 7.0 ms.
// Groups run independently, so one's products and barriers run under the others' S-boxes.
#pragma once
#include "gl64.cuh"
#include "tc_tables.h"
#include "wait_error.cuh"

// Table bytes and constants by [family - 1][width / 4 - 2], uploaded once per device.
__device__ __align__(16) uint8_t g_tc_tab[2][3][tch::MAX_BYTES];
__constant__ tch::Consts c_tc[2][3];

namespace tch {

// Groups of a CTA, threads that share a row, and a group's tensor memory columns (a whole layer's): what shared
// memory and the 512 columns hold, with 1024 threads either way.  (Width 12 with five groups of one thread a row: 9.65 against
// 9.75 ms for 2^20 rows x 128 columns, but 32 against 28 us for 5000 rows x 8.)
template <int W>
struct Cfg {
    static constexpr int GROUPS = W == 8 ? 8 : 4, SPLIT = W == 8 ? 1 : 2;
    static constexpr int GTHREADS = 128 * SPLIT, THREADS = GTHREADS * GROUPS, COLS = 8 * W;
    static_assert(GROUPS * COLS <= 512 && GROUPS <= 15, "tensor memory columns, barriers");
    // an allocation is a power of two
    static __device__ __forceinline__ uint32_t columns(uint32_t groups)
    {
        const uint32_t n = groups * COLS;
        return n > 256 ? 512 : n > 128 ? 256 : n > 64 ? 128 : 64;
    }
};
constexpr int MAX_GROUPS = 8;
constexpr uint32_t WAIT_LIMIT = 1u << 20;  // try_wait rounds before a thread gives up

template <int W>
struct Smem {
    static constexpr int GROUP = (Shape<W>::CHX + YCH) * 2048;  // state rows and a block's y rows
    static constexpr int bytes(int groups) { return Shape<W>::BYTES + groups * GROUP; }
    static constexpr int BYTES = bytes(Cfg<W>::GROUPS);
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// Shared-memory matrix descriptor, no swizzle: 8-row x 16-byte cores, `lbo` bytes between cores along K,
// 128 bytes between cores along the rows.
__device__ __forceinline__ uint64_t matrix_desc(uint32_t addr, uint32_t lbo)
{
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | ((uint64_t)(128 >> 4) << 32) | (1ull << 46);
}

// u8 x u8 -> s32, 128 rows, n columns
__host__ __device__ constexpr uint32_t instr_desc(uint32_t n) { return (2u << 4) | ((n >> 3) << 17) | ((128u >> 4) << 24); }

__device__ __forceinline__ void mma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

// 16 columns (two words) of this thread's row
__device__ __forceinline__ void ld_cols16(uint32_t (&r)[16], uint32_t t)
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(t)
        : "memory");
}

__device__ __forceinline__ void sts128(uint32_t a, uint64_t x, uint64_t y)
{
    asm volatile("st.shared.v2.b64 [%0], {%1, %2};" ::"r"(a), "l"(x), "l"(y) : "memory");
}

// 160-bit little-endian value
struct Wide {
    uint32_t w[5];
};

// Column pairs: t_i = col[2i] + 256 col[2i+1], below 2^31 for every table, the word is sum_i t_i 2^(16 i).
__device__ __forceinline__ void pairs(const uint32_t *col, uint32_t (&t)[4])
{
#pragma unroll
    for (int i = 0; i < 4; i++) t[i] = col[2 * i] + (col[2 * i + 1] << 8);
}

// sum_i t_i 2^(16 i) + c in 96 bits
__device__ __forceinline__ void join96(const uint32_t *col, uint64_t c, uint32_t &w0, uint32_t &w1, uint32_t &w2)
{
    uint32_t t[4];
    pairs(col, t);
    const uint64_t lo = (uint64_t)t[1] * 65536u + t[0], hi = (uint64_t)t[3] * 65536u + t[2];
    asm("add.cc.u32  %0, %3, %7;\n\t"
        "addc.cc.u32 %1, %4, %8;\n\t"
        "addc.u32    %2, %6, 0;\n\t"
        "add.cc.u32  %1, %1, %5;\n\t"
        "addc.u32    %2, %2, 0;\n\t"
        : "=&r"(w0), "=&r"(w1), "=&r"(w2)
        : "r"(gl::lo32(lo)), "r"(gl::hi32(lo)), "r"(gl::lo32(hi)), "r"(gl::hi32(hi)), "r"(gl::lo32(c)), "r"(gl::hi32(c)));
}

// (sum_i t_i 2^(16 i)) 2^-32 + c, loose.  With x0 the sum's low word, one Montgomery step by 32 bits is
// (sum - x0 p) / 2^32 = sum >> 32 + x0 - x0 2^32; c < 2^64 - 2^50 leaves room for the rest, so only the last
// subtraction can wrap, once, and the result is at most gl::MONT_MAX.
__device__ __forceinline__ uint64_t join_word(const uint32_t *col, uint64_t c)
{
    uint32_t t[4], x0, u;
    pairs(col, t);
    asm("add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32   %1, %4, %5;\n\t"
        : "=&r"(x0), "=&r"(u)
        : "r"(t[0]), "r"(t[1] << 16), "r"(t[2]), "r"(t[1] >> 16));
    const uint64_t y = (uint64_t)t[3] * 65536u + c + u + x0;
    uint32_t z1, m;
    asm("sub.cc.u32 %0, %2, %3;\n\t"
        "subc.u32   %1, 0, 0;\n\t"
        : "=r"(z1), "=r"(m)
        : "r"(gl::hi32(y)), "r"(x0));
    return gl::mk64(gl::lo32(y), z1) - (uint64_t)m;
}

__device__ __forceinline__ void wide_mul_add(Wide &a, uint64_t x, uint64_t y)
{
    uint32_t r0, r1, r2, r3;
    gl::mul128(x, y, r0, r1, r2, r3);
    asm("add.cc.u32  %0, %0, %5;\n\t"
        "addc.cc.u32 %1, %1, %6;\n\t"
        "addc.cc.u32 %2, %2, %7;\n\t"
        "addc.cc.u32 %3, %3, %8;\n\t"
        "addc.u32    %4, %4, 0;\n\t"
        : "+r"(a.w[0]), "+r"(a.w[1]), "+r"(a.w[2]), "+r"(a.w[3]), "+r"(a.w[4])
        : "r"(r0), "r"(r1), "r"(r2), "r"(r3));
}

// 2^128 = -2^32 (mod p): reduce the low 128 bits, subtract w4 * 2^32 (< p)
__device__ __forceinline__ uint64_t wide_reduce(const Wide &a)
{
    return gl::sub_c(gl::reduce128(a.w[0], a.w[1], a.w[2], a.w[3]), (uint64_t)a.w[4] << 32);
}

// Canonical words to p: 16-byte stores where p is aligned for them (a tree may start at any word of a caller's
// buffer), else 8-byte ones.
template <int N>
__device__ __forceinline__ void store_words(uint64_t *p, const uint64_t (&v)[N])
{
    const bool aligned = (reinterpret_cast<uintptr_t>(p) & 15) == 0;
#pragma unroll
    for (int i = 0; i < N; i += 2) {
        const uint64_t a = gl::canon(v[i]), b = gl::canon(v[i + 1]);
        if (aligned) {
            *reinterpret_cast<ulonglong2 *>(p + i) = make_ulonglong2(a, b);
        } else {
            p[i] = a;
            p[i + 1] = b;
        }
    }
}

// A CTA's barriers and tensor memory address.
struct Shared {
    uint64_t mbar[MAX_GROUPS];
    uint32_t tmem, columns;
};

// A thread's view of its group.
template <int W, int FAM>
struct Group {
    uint32_t row;      // shared address of this thread's row (piece 0)
    uint32_t tab;      // shared address of the tables
    uint32_t tmem;     // the group's first tensor memory column, this warp's lanes
    uint32_t mbar;     // the group's barrier
    uint32_t phase;
    uint32_t id;       // group index
    uint32_t half;     // this thread's share of the row's words
    bool issuer, dead;

    static constexpr int GROUPS = Cfg<W>::GROUPS, SPLIT = Cfg<W>::SPLIT, GTHREADS = Cfg<W>::GTHREADS,
                         THREADS = Cfg<W>::THREADS;
    static constexpr int OUT = 4 / SPLIT;  // output words of a thread

    static __device__ __forceinline__ const Consts &consts() { return c_tc[FAM - 1][W / 4 - 2]; }

    // words i and i + 1 (i even) of this thread's row
    __device__ __forceinline__ void store_row(int i, uint64_t x, uint64_t y) const
    {
        sts128(row + (uint32_t)(i >> 1) * 2048, x, y);
    }

    // Tables into shared memory, tensor memory, barriers.  All threads of the CTA, which has `groups` groups.
    __device__ __forceinline__ void setup(uint8_t *sm, Shared &sh, uint32_t groups = GROUPS)
    {
        const uint32_t warp = threadIdx.x >> 5;
        const uint8_t *src = g_tc_tab[FAM - 1][W / 4 - 2];
        tab = smem_addr(sm);
        // asynchronous copies: with one group a CTA, loads through registers took 3 us longer
        for (uint32_t i = threadIdx.x * 16; i < (uint32_t)Shape<W>::BYTES; i += groups * GTHREADS * 16)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tab + i), "l"(__cvta_generic_to_global(src + i)) : "memory");
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (warp == 0) {
            const uint32_t columns = Cfg<W>::columns(groups);
            if (threadIdx.x == 0) sh.columns = columns;
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&sh.tmem)),
                         "r"(columns)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        if (threadIdx.x < GROUPS)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(sh.mbar + threadIdx.x)) : "memory");
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        id = threadIdx.x / GTHREADS;
        half = (threadIdx.x >> 7) % SPLIT;
        const uint32_t r = threadIdx.x & 127;
        row = tab + Shape<W>::BYTES + id * Smem<W>::GROUP + r * 16;
        tmem = sh.tmem + id * Cfg<W>::COLS + ((warp & 3) << 21);
        mbar = smem_addr(sh.mbar + id);
        phase = 0;
        issuer = threadIdx.x % GTHREADS == 0;
        dead = false;
    }

    // barrier of the group's threads
    __device__ __forceinline__ void sync() const { asm volatile("bar.sync %0, %1;" ::"r"(id + 1), "n"(GTHREADS) : "memory"); }

    // the same barrier, and whether any of them has given up: the same answer to all, so that they leave a loop together
    __device__ __forceinline__ bool gave_up() const
    {
        uint32_t any;
        asm volatile(
            "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 p, %1, 0;\n\t"
            "bar.red.or.pred q, %2, %3, p;\n\t"
            "selp.u32 %0, 1, 0, q;\n\t}"
            : "=r"(any)
            : "r"((uint32_t)dead), "r"(id + 1), "n"(GTHREADS)
            : "memory");
        return any != 0;
    }

    __device__ __forceinline__ bool wait(uint32_t limit = WAIT_LIMIT) const
    {
        for (uint32_t i = 0; i < limit; i++) {
            uint32_t done;
            asm volatile(
                "{\n\t.reg .pred p;\n\t"
                "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                "selp.u32 %0, 1, 0, p;\n\t}"
                : "=r"(done)
                : "r"(mbar), "r"(phase)
                : "memory");
            if (done) return true;
        }
        return false;
    }

    // The group's rows times a table of K bytes (K / 32 steps of 32) whose pieces hold `ld` columns, the first
    // n of them into the group's tensor memory.  Ends with the columns readable.  If the product does not
    // complete within the wait bound the thread flags the error and gives up: it waits for and issues nothing
    // more, and its phase stays that of the product it gave up on, which finish() waits for once more.  It goes
    // through the motions up to the end of the tile (the barriers need every thread; what a late product then
    // reads from the rows no longer matters), stores no digest, and the group leaves at the next gave_up().
    // `issue` and `limit` are for the probe of that path.
    __device__ __forceinline__ void product(uint32_t off, uint32_t ksteps, uint32_t ld, uint32_t idesc, bool issue = true,
                                            uint32_t limit = WAIT_LIMIT)
    {
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        sync();
        if (issuer && !dead && issue) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint64_t a = matrix_desc(row, 2048), b = matrix_desc(tab + off, ld * 16);
            for (uint32_t k = 0; k < ksteps; k++) {
                mma_i8(tmem, a, b, idesc, k != 0);
                a += 2 * 2048 / 16;
                b += 2 * ld;
            }
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(mbar) : "memory");
        }
        if (!dead) {
            if (wait(limit)) {
                phase ^= 1;
            } else {
                dead = true;
                wait_error::raise();
            }
        }
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }

    // Frees the tensor memory once every group is done with it.  All threads of the CTA.
    __device__ __forceinline__ void finish(const Shared &sh, uint32_t limit = WAIT_LIMIT)
    {
        // A late product gets one more bound to land.  The issuer's wait covers every product issued: those before
        // the one it gave up on it saw complete, and it has issued none since.
        if (issuer && dead) wait(limit);
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(sh.tmem), "r"(sh.columns));
        }
    }

    // One run of N partial rounds: z_t from the product's words and the run's earlier y, y_t = z_t^7 into the
    // block's y rows from y_{first}.  A chain, so one thread of a row does it: the first run's by one half of the
    // threads, the second's by the other.
    template <int N>
    __device__ __forceinline__ void run(uint32_t off, uint32_t ksteps, int first, const uint64_t *kz, const uint64_t *q)
    {
        product(off, ksteps, NZ, instr_desc(NZ));
        if (SPLIT == 2 && half != (N == RUN0 ? 0 : 1)) return;
        uint64_t y[N];
        uint32_t col[16];
#pragma unroll
        for (int t = 0; t < N; t++) {
            if (t % 2 == 0) ld_cols16(col, tmem + 8 * t);
            if (t == 0) {
                y[0] = gl::mont_pow7(join_word(col, kz[0]));
            } else {
                Wide a;
                join96(col + 8 * (t & 1), kz[t], a.w[0], a.w[1], a.w[2]);
                a.w[3] = a.w[4] = 0;
#pragma unroll
                for (int u = 0; u < t; u++) wide_mul_add(a, y[u], q[t * (t - 1) / 2 + u]);
                y[t] = gl::mont_pow7(gl::canon(wide_reduce(a)));
            }
        }
#pragma unroll
        for (int t = 0; t < N; t += 2) store_row(W + first + t, y[t], t + 1 < N ? y[t + 1] : 0ull);
    }

    // The permutation of the states in the rows (Poseidon2: the state; Poseidon1: x^7 of the state plus the
    // first constants, which has no layer before it).  out: words 0..3 of the result, loose.
    __device__ __forceinline__ void permute(uint64_t (&out)[OUT])
    {
        typedef Shape<W> S;
        const Consts &C = consts();
#pragma unroll 1
        for (int s = FAM == 2 ? 0 : 1; s < 9; s++) {
            if (s == 4 || s == 5) {
                const int b = s - 4;
                run<RUN0>(S::OFF_Z0 + b * S::BLOCK, S::K_Z0 / 32, 0, C.z[b], C.q[b]);
                run<RUN1>(S::OFF_Z1 + b * S::BLOCK, S::K_Z1 / 32, RUN0, C.z[b] + RUN0, C.q[b] + RUN0 * (RUN0 - 1) / 2);
                product(S::OFF_U + b * S::BLOCK, S::K_U / 32, S::KX, instr_desc(S::KX));
            } else {
                product(S::OFF_L, S::KX / 32, S::KX, instr_desc(S::KX));
            }
            const uint64_t *k = C.lay[s];
#pragma unroll 1
            for (int i = 0; i < W / SPLIT; i += 2) {
                const int g = half * (W / SPLIT) + i;
                uint32_t col[16];
                ld_cols16(col, tmem + 8 * g);
                uint64_t x[2];
#pragma unroll
                for (int j = 0; j < 2; j++) x[j] = join_word(col + 8 * j, k[g + j]);
                if (s != 4) {
#pragma unroll
                    for (int j = 0; j < 2; j++) x[j] = gl::mont_pow7(x[j]);
                }
#pragma unroll
                for (int j = 0; j < 2; j += 2) store_row(g + j, x[j], x[j + 1]);
            }
        }
        product(S::OFF_F, S::KX / 32, S::NF, instr_desc(S::NF));
#pragma unroll
        for (int j = 0; j < OUT; j += 2) {
            uint32_t col[16];
            ld_cols16(col, tmem + 8 * (OUT * half + j));
            out[j] = join_word(col, 0);
            out[j + 1] = join_word(col + 8, 0);
        }
    }

    // words g and g + 1 of a state into the rows (g even)
    __device__ __forceinline__ void put2(int g, uint64_t a, uint64_t b) const
    {
        if (FAM == 1) {
            const uint64_t *k = consts().lay[0];
            a = gl::pow7(gl::add_c(a, k[g]));
            b = gl::pow7(gl::add_c(b, k[g + 1]));
        }
        store_row(g, a, b);
    }
};

// Tiles of a launch over its CTAs of `groups` groups: waves of `lanes` CTAs, `rounds` tiles a group and wave; a wave's
// first tiles go to different CTAs, so that few tiles spread over the SMs.
struct Split {
    uint32_t lanes, rounds, ctas, groups;
};

// A group's tiles: for (t = first; t < end; t += step).
template <int W>
struct TileRange {
    uint64_t first, end, step;
    __device__ __forceinline__ TileRange(const Split &s, uint32_t group, uint64_t tiles)
    {
        step = (uint64_t)s.lanes * s.groups;
        const uint64_t wave = step * s.rounds, begin = blockIdx.x / s.lanes * wave;
        first = begin + (uint64_t)group * s.lanes + blockIdx.x % s.lanes;
        end = tiles - begin < wave ? tiles : begin + wave;
    }
};

// Row sponge of up to 128 rows (capacity zeroed at the start; every block of RATE columns overwrites words
// [0, RATE), zero past the last column, and carries words [0, 4) into the capacity; 0 columns give the zero digest:
// poseidon2_goldilocks.cpp:42-77).  `resume`: the digests hold the four words of the blocks before.  Threads past the last
// row hash it again and store nothing.
template <int W, int FAM>
__device__ __forceinline__ void leaf_tile(Group<W, FAM> &G, uint64_t *__restrict__ digests,
                                          const uint64_t *__restrict__ src, uint64_t rs, uint64_t cs, uint64_t ncols,
                                          uint64_t nrows, uint64_t tile, bool resume)
{
    constexpr int RATE = W - 4, MINE = RATE / Cfg<W>::SPLIT, OUT = Group<W, FAM>::OUT;
    uint64_t row = tile * 128 + (threadIdx.x & 127);
    const bool valid = row < nrows;
    if (!valid) row = nrows - 1;
    const int first = (int)G.half * MINE;
    const uint64_t *p = src + row * rs;
    uint64_t *d = digests + row * 4 + G.half * OUT;
    uint64_t cap[OUT] = {};
    if (resume) {
#pragma unroll
        for (int i = 0; i < OUT; i++) cap[i] = d[i];
    }
    for (uint64_t done = 0; done < ncols; done += RATE) {
        const uint64_t at = done + first;
        uint64_t v[MINE];
#pragma unroll
        for (int i = 0; i < MINE; i++) v[i] = at + i < ncols ? __ldg(p + (at + i) * cs) : 0ull;
#pragma unroll
        for (int i = 0; i < MINE; i += 2) G.put2(first + i, v[i], v[i + 1]);
#pragma unroll
        for (int i = 0; i < OUT; i += 2) G.put2(RATE + (int)G.half * OUT + i, cap[i], cap[i + 1]);
        G.permute(cap);
    }
    if (valid && !G.dead) store_words(d, cap);
}

// Parents of up to 128 nodes of one tree level (poseidon2_goldilocks.cpp:129-175): `pending` child digests at
// `level`, `pad` zero digests after them (written by the last parent), parents written to `out`; parent i hashes the
// W words of its children, zero past `pending`.
template <int W, int FAM>
__device__ __forceinline__ void node_tile(Group<W, FAM> &G, uint64_t *__restrict__ level, uint64_t pending, uint64_t pad,
                                          uint64_t parents, uint64_t *__restrict__ out, uint64_t tile)
{
    constexpr int MINE = W / Cfg<W>::SPLIT, OUT = Group<W, FAM>::OUT;
    const uint64_t i = tile * 128 + (threadIdx.x & 127);
    const uint64_t first = i * W + G.half * MINE, end = pending * 4;
    if (i == parents - 1 && G.half == 0)
        for (uint64_t z = 0; z < pad * 4; z++) level[end + z] = 0;
    uint64_t v[MINE];
    const uint64_t *q = level + first;
    if ((reinterpret_cast<uintptr_t>(q) & 15) == 0 && first + MINE <= end) {
#pragma unroll
        for (int j = 0; j < MINE; j += 2) {
            const ulonglong2 w = *reinterpret_cast<const ulonglong2 *>(q + j);
            v[j] = w.x;
            v[j + 1] = w.y;
        }
    } else {
#pragma unroll
        for (int j = 0; j < MINE; j++) v[j] = first + j < end ? q[j] : 0ull;
    }
#pragma unroll
    for (int j = 0; j < MINE; j += 2) G.put2((int)G.half * MINE + j, v[j], v[j + 1]);
    uint64_t o[OUT];
    G.permute(o);
    if (i < parents && !G.dead) store_words(out + i * 4 + G.half * OUT, o);
}

// Probe of a product that does not complete: every group runs `before` products, waits a few rounds for one that is
// never issued, and calls product `after` times more.  counts: threads that gave up; threads whose phase says the
// missing product has landed; threads told to leave.
__global__ void __launch_bounds__(Cfg<16>::THREADS, 1) product_wait_probe_kernel(uint32_t before, uint32_t after, uint32_t *counts)
{
    typedef Shape<16> S;
    constexpr uint32_t LIMIT = 8;
    extern __shared__ __align__(128) uint8_t tc_sm[];
    __shared__ Shared sh;
    Group<16, 2> G;
    G.setup(tc_sm, sh);
    if (G.half == 0)
        for (int i = 0; i < 16; i += 2) G.store_row(i, 1, 2);
    for (uint32_t i = 0; i < before; i++) G.product(S::OFF_L, S::KX / 32, S::KX, instr_desc(S::KX));
    G.product(S::OFF_L, S::KX / 32, S::KX, instr_desc(S::KX), false, LIMIT);
    for (uint32_t i = 0; i < after; i++) G.product(S::OFF_L, S::KX / 32, S::KX, instr_desc(S::KX));
    atomicAdd(counts, G.dead ? 1u : 0u);
    atomicAdd(counts + 1, G.wait(LIMIT) ? 1u : 0u);
    atomicAdd(counts + 2, G.gave_up() ? 1u : 0u);
    G.finish(sh, LIMIT);
}

// ------------------------------------------------------------------ host side ----

template <int W>
inline cudaError_t upload(int fam)
{
    static uint8_t tab[MAX_BYTES];
    Consts c;
    build_tables<W>(fam, tab, c);
    const size_t i = (size_t)(fam - 1) * 3 + (W / 4 - 2);
    cudaError_t e = cudaMemcpyToSymbol(g_tc_tab, tab, Shape<W>::BYTES, i * MAX_BYTES);
    if (e != cudaSuccess) return e;
    return cudaMemcpyToSymbol(c_tc, &c, sizeof(c), i * sizeof(Consts));
}

template <int W>
inline cudaError_t upload()
{
    const cudaError_t e = upload<W>(1);
    return e != cudaSuccess ? e : upload<W>(2);
}

// the tables of every width and family on the current device
inline cudaError_t init_tables()
{
    cudaError_t e;
    if ((e = upload<8>()) != cudaSuccess) return e;
    if ((e = upload<12>()) != cudaSuccess) return e;
    return upload<16>();
}

// Groups of a CTA of a launch over `tiles` tiles.  Up to one tile an SM (two at width 8) as many as it has, so that launches
// of different streams share an SM where tables, rows and tensor memory columns fit more than once: three CTAs of 64 KB and
// 64 columns at width 8 (two of 84 KB with two groups), two of 96 KB and 128 columns at width 12.  With all groups they
// queued, one of eight or four at work: 48 commits of 2^13 x 40 on 16 streams 10.1 -> 6.1 ms at arity 2 (7.7 with the
// one-thread-a-row kernels) and 6.0 -> 4.4 at arity 3 (6.3), on one stream 17.2 -> 17.0 and 12.3 -> 12.2.  At width 16 the
// tables keep a second CTA out (2 x 134 KB).
template <int W>
inline uint32_t few_groups(uint64_t tiles, uint64_t sms)
{
    if (W < 16 && tiles <= sms) return 1;
    return W == 8 && tiles <= 2 * sms ? 2 : Cfg<W>::GROUPS;
}

// Launch over `tiles` 128-row tiles of `perms` permutations a row.  A CTA holds its SM to its end, and a kernel of a
// higher-priority stream enters at CTA ends only, so a group takes the tiles of 16 permutations (0.9-1.0 ms with every
// group at work) or one wider tile, and the next CTA goes on.  With one CTA an SM for all tiles, query openings issued
// at high priority 1 ms into a tree of 2^20 x 256 waited 14.9 ms (whole sponge 16.4), with these 0.08; the trees take the
// same (16.60 and 16.61 ms; 2^20 x 24: 1.86 both); at most 1 % more where a second wave is short of tiles (a commit of
// 2^16 x 126 at arity 3: 1.86 -> 1.88).  Half as many permutations a CTA take 2 % more at 24 columns: a table
// load and tensor memory setup are a few microseconds each.
constexpr uint64_t CTA_PERMS = 16;
template <int W>
inline Split split(uint64_t tiles, uint64_t perms, uint64_t sms)
{
    const uint64_t rounds = perms >= CTA_PERMS ? 1 : perms ? CTA_PERMS / perms : CTA_PERMS;
    const uint32_t groups = few_groups<W>(tiles, sms);
    const uint64_t lanes = tiles < sms ? tiles : sms, wave = rounds * groups * lanes;
    const uint64_t rest = tiles % wave;
    return Split{(uint32_t)lanes, (uint32_t)rounds, (uint32_t)(tiles / wave * lanes + (rest < lanes ? rest : lanes)), groups};
}

// the same on the current device
template <int W>
inline Split split(uint64_t tiles, uint64_t perms)
{
    int dev = 0, sms = 0;
    if (cudaGetDevice(&dev) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || sms < 1)
        sms = 1;
    return split<W>(tiles, perms, (uint64_t)sms);
}

}  // namespace tch
