// Row sponge ("linear hash") and arity-k Merkle tree levels, Poseidon2 or Poseidon1.
//
// Semantics follow the reference CPU path bit for bit:
//   linear hash  poseidon2_goldilocks.cpp:42-77 — capacity zeroed at the start; every
//                block overwrites words [0, n) with input, zero-fills [n, RATE) and carries
//                the previous output words [0, 4) into the capacity; no length padding;
//                0 columns give the zero digest.
//   tree         poseidon2_goldilocks.cpp:129-175 — digests of a level are contiguous
//                4-word groups; (arity - pending % arity) % arity zero digests pad the level
//                inside the buffer; parent i is the first 4 words of the permutation of the
//                W = 4*arity words of its children; the root is the last 4 words
//                (goldilocks_tooling.hpp:9-21 gives the buffer size).
//
// Layout: the extended trace is addressed as element (row, col) = src[row*rs + col*cs], so
// the same kernel reads the column-major device LDE (rs = 1, cs = nrows; warp loads are
// 256 B contiguous) or a row-major buffer (rs = ncols, cs = 1).
#pragma once
#include "coop.cuh"
#include "poseidon1.cuh"
#include "poseidon2.cuh"
#include "prof.cuh"
#include "tc_hash.cuh"

namespace merkle {

constexpr int TPB = 128;  // threads per CTA of permute_kernel (one state each)

// Hash family (the reference's set_hash_family): 1 = Poseidon1, 2 = Poseidon2.  Both use the same sponge and
// tree.  permute_kernel, which returns every word of a state, runs the one-thread-a-state permutations; the
// Poseidon1 one needs a second W x TPB shared area for its matrix steps, right after the state area.
template <int FAM>
struct Family {
    static constexpr int SMEM_AREAS = FAM == 1 ? 2 : 1;
    // resident CTAs per SM the register budget must allow (registers <= 64 K / (MIN_CTAS * 128)):
    // Poseidon1's 32 KB of shared memory per CTA fits 7 CTAs, so its registers are capped to
    // match (72); Poseidon2 keeps 12 resident CTAs (<= 42 registers, the 40 it needs)
    static constexpr int MIN_CTAS = FAM == 1 ? 7 : 12;
};

template <int W, int FAM>
__device__ __forceinline__ void permute_fam(uint64_t *st)
{
    if constexpr (FAM == 1)
        p1::permute_smem<W, TPB>(st, st + W * TPB);
    else
        p2::permute_smem<W, TPB>(st);
}

// Row sponges of `nrows` rows, 128-row tiles over the groups of every CTA (tc_hash.cuh).  Against one thread a row with
// the state in shared memory and every layer on the integer pipes, 2^20 rows (B200): Poseidon2 W16 x 256 columns 24.6 ->
// 16.3 ms (937 -> 1413 M permutations/s), W12 x 128 13.9 -> 9.8, W8 x 64 9.6 -> 7.0; Poseidon1 W16 39.0 -> 16.4, W12 19.4 -> 9.7, W8 12.5 -> 7.0.
template <int W, int FAM = 2>
__global__ void __launch_bounds__(tch::Cfg<W>::THREADS, 1) leaf_hash_kernel(uint64_t *__restrict__ digests,
                                                                    const uint64_t *__restrict__ src, uint64_t rs,
                                                                    uint64_t cs, uint64_t ncols, uint64_t nrows,
                                                                    int resume, tch::Split split)
{
    extern __shared__ __align__(128) uint8_t tc_sm[];
    __shared__ tch::Shared sh;
    tch::Group<W, FAM> G;
    G.setup(tc_sm, sh, split.groups);
    const tch::TileRange<W> r(split, G.id, (nrows + 127) / 128);
    for (uint64_t t = r.first; t < r.end; t += r.step) {
        tch::leaf_tile(G, digests, src, rs, cs, ncols, nrows, t, resume != 0);
        if (G.gave_up()) break;
    }
    G.finish(sh);
}

// One tree level of `parents` parents.
template <int W, int FAM = 2>
__global__ void __launch_bounds__(tch::Cfg<W>::THREADS, 1) node_kernel(uint64_t *__restrict__ level, uint64_t pending, uint64_t pad,
                                                               uint64_t parents, uint64_t *__restrict__ out,
                                                               tch::Split split)
{
    extern __shared__ __align__(128) uint8_t tc_sm[];
    __shared__ tch::Shared sh;
    tch::Group<W, FAM> G;
    G.setup(tc_sm, sh, split.groups);
    const tch::TileRange<W> r(split, G.id, (parents + 127) / 128);
    for (uint64_t t = r.first; t < r.end; t += r.step) {
        tch::node_tile(G, level, pending, pad, parents, out, t);
        if (G.gave_up()) break;
    }
    G.finish(sh);
}

// Whole permutations of n independent states (permute / permuteTrunc checks).
template <int W, int FAM = 2>
__global__ void __launch_bounds__(TPB, Family<FAM>::MIN_CTAS) permute_kernel(uint64_t *__restrict__ out, const uint64_t *__restrict__ in,
                                                      uint64_t n)
{
    __shared__ uint64_t sm[Family<FAM>::SMEM_AREAS * W * TPB];
    uint64_t *st = sm + threadIdx.x;
    const uint64_t i = (uint64_t)blockIdx.x * TPB + threadIdx.x;
    if (i >= n) return;
#pragma unroll
    for (int j = 0; j < W; j++) st[j * TPB] = in[i * W + j];
    permute_fam<W, FAM>(st);
#pragma unroll
    for (int j = 0; j < W; j++) out[i * W + j] = gl::canon(st[j * TPB]);
}

inline uint64_t tree_num_elements(uint64_t nrows, uint64_t arity)
{
    uint64_t total = nrows, level = nrows;
    while (level > 1) {
        total += (arity - level % arity) % arity;
        level = (level + arity - 1) / arity;
        total += level;
    }
    return total * 4;
}

// Launches of at most this many states x lanes (4096 states at W = 12 and 16, 8192 at W = 8) run cooperatively
// (coop.cuh): below it the tiled kernels leave most of the GPU idle and take the latency of whole permutations, above
// it the cooperative ones' instructions take longer.  One W16 permutation of 4096 / 6144 rows: 23 / 32 us cooperative,
// 30 / 30 tiled; W8 of 8192 / 12288 rows: 21 / 30 and 26 / 26.
constexpr uint64_t COOP_MAX_LANES = 65536;
template <int W>
constexpr uint64_t coop_max_states()
{
    return COOP_MAX_LANES / coop::Tab<W>::G;
}

// Every tree level above `nrows` leaf digests already at the start of d_tree, on `stream`.
// Levels of more than coop_max_states parents in 128-parent tiles, smaller ones cooperatively, several to a
// launch (coop::subtree_kernel); both hash families.
template <int W, int FAM = 2>
cudaError_t build_levels(uint64_t *d_tree, uint64_t nrows, cudaStream_t stream)
{
    constexpr uint64_t ARITY = W / 4;
    prof::Scope ps(prof::TREE_LEVELS, stream);
    uint64_t pending = nrows, base = 0;
    while (pending > 1) {
        const uint64_t pad = (ARITY - pending % ARITY) % ARITY;
        const uint64_t parents = (pending + ARITY - 1) / ARITY;
        const uint64_t before = pending;
        uint64_t *lvl = d_tree + base;
        if (parents <= coop_max_states<W>()) {
            constexpr uint64_t P = coop::Subtree<W>::PARENTS;
            const int levels = coop::subtree_advance<W>(pending, base);
            coop::subtree_kernel<W, FAM><<<(unsigned)((parents + P - 1) / P), coop::CTA_THREADS, 0, stream>>>(
                lvl, before, levels);
            prof::count();
            continue;
        }
        const tch::Split split = tch::split<W>((parents + 127) / 128, 1);
        node_kernel<W, FAM><<<split.ctas, tch::Cfg<W>::GTHREADS * split.groups, tch::Smem<W>::bytes(split.groups), stream>>>(
            lvl, pending, pad, parents, lvl + (pending + pad) * 4, split);
        prof::count();
        base += (pending + pad) * 4;
        pending = parents;
    }
    return cudaGetLastError();
}

// Row sponges into `digests` (resume: continuing from the words there), on `stream`.
template <int W, int FAM = 2>
cudaError_t hash_rows(uint64_t *digests, const uint64_t *src, uint64_t rs, uint64_t cs, uint64_t ncols, uint64_t nrows,
                      bool resume, cudaStream_t stream)
{
    const tch::Split split = tch::split<W>((nrows + 127) / 128, (ncols + W - 5) / (W - 4));
    leaf_hash_kernel<W, FAM><<<split.ctas, tch::Cfg<W>::GTHREADS * split.groups, tch::Smem<W>::bytes(split.groups), stream>>>(
        digests, src, rs, cs, ncols, nrows, resume ? 1 : 0, split);
    prof::count();
    return cudaGetLastError();
}

// Leaf digests and every level up to the root, on `stream`.
template <int W, int FAM = 2>
cudaError_t build_tree(uint64_t *d_tree, const uint64_t *d_src, uint64_t rs, uint64_t cs, uint64_t ncols,
                       uint64_t nrows, cudaStream_t stream)
{
    if (nrows == 0) return cudaSuccess;
    {
        prof::Scope ps(prof::LEAF_HASH, stream);
        if (nrows <= coop_max_states<W>()) {
            const uint64_t threads = nrows * coop::Tab<W>::G;
            coop::leaf_coop_kernel<W, FAM><<<(unsigned)((threads + coop::CTA_THREADS - 1) / coop::CTA_THREADS),
                                             coop::CTA_THREADS, 0, stream>>>(d_tree, d_src, rs, cs, ncols, nrows);
            prof::count();
        } else {
            const cudaError_t e = hash_rows<W, FAM>(d_tree, d_src, rs, cs, ncols, nrows, false, stream);
            if (e != cudaSuccess) return e;
        }
    }
    return build_levels<W, FAM>(d_tree, nrows, stream);
}

// family: 1 = Poseidon1, otherwise Poseidon2; W = 4 * arity (MerkleTreeGL::merkelize)
inline cudaError_t build_tree_arity(uint64_t arity, uint64_t *d_tree, const uint64_t *d_src, uint64_t rs,
                                    uint64_t cs, uint64_t ncols, uint64_t nrows, cudaStream_t stream, int family = 2)
{
    if (family == 1) {
        switch (arity) {
        case 2: return build_tree<8, 1>(d_tree, d_src, rs, cs, ncols, nrows, stream);
        case 3: return build_tree<12, 1>(d_tree, d_src, rs, cs, ncols, nrows, stream);
        case 4: return build_tree<16, 1>(d_tree, d_src, rs, cs, ncols, nrows, stream);
        default: return cudaErrorInvalidValue;
        }
    }
    switch (arity) {
    case 2: return build_tree<8>(d_tree, d_src, rs, cs, ncols, nrows, stream);
    case 3: return build_tree<12>(d_tree, d_src, rs, cs, ncols, nrows, stream);
    case 4: return build_tree<16>(d_tree, d_src, rs, cs, ncols, nrows, stream);
    default: return cudaErrorInvalidValue;
    }
}

// tables and kernel attributes of the current device
template <int W, int FAM>
inline cudaError_t set_attrs()
{
    const cudaError_t e = cudaFuncSetAttribute(leaf_hash_kernel<W, FAM>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                               tch::Smem<W>::BYTES);
    if (e != cudaSuccess) return e;
    return cudaFuncSetAttribute(node_kernel<W, FAM>, cudaFuncAttributeMaxDynamicSharedMemorySize, tch::Smem<W>::BYTES);
}

inline cudaError_t init()
{
    cudaError_t e = tch::init_tables();
    if (e == cudaSuccess) e = set_attrs<8, 1>();
    if (e == cudaSuccess) e = set_attrs<8, 2>();
    if (e == cudaSuccess) e = set_attrs<12, 1>();
    if (e == cudaSuccess) e = set_attrs<12, 2>();
    if (e == cudaSuccess) e = set_attrs<16, 1>();
    if (e == cudaSuccess) e = set_attrs<16, 2>();
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(tch::product_wait_probe_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 tch::Smem<16>::BYTES);
    return e;
}

}  // namespace merkle
