// The reference's MT19937 walk baselines on sm_100a with exact uint32 visit counters:
//   scalar  src/rw_experiment.cpp:34-47      walk i, hop j takes draw i * depth + j
//   simd    src/rw_experiment_simd.cpp:44-83 bouquet b (walks 8b .. 8b+7) steps together; hop j
//                                            of lane l takes draw 8 b depth + 8 j + l
// from every vertex with a neighbour, with std::mt19937 reseeded to 42 + src per source
// (src/rw_experiment.cpp:110) and k = draw % degree(cur) per hop.  They are the comparison rows of
// the walk experiment (not the SABA walk): same counters as the reference's routines, integer
// instead of float.
//
// Layout.  One warp per source (grid-stride over the sources).  The generator is the Mersenne
// Twister of Matsumoto & Nishimura (ACM TOMACS 8(1), 1998) with the C++ standard's seeding.  Its
// 624-word state lives in shared memory as a ring of two generations: generation t (t = 0 the
// seeded state, t >= 1 the state after t regenerations, whose tempered words are draws
// 624 (t-1) .. 624 t - 1) sits in half t & 1.  Generation t + 1 is built from t into the other
// half by the 32 lanes together: word i needs old words i and i + 1 and either old word i + 397
// (i < 227) or new word i - 227 -- at least 227 places back, so runs of 224 words (seven a lane)
// never depend on one another.  The lanes walk side by side, up to kSlots walks each (scalar) or
// kSlots bouquets per 8 lanes (simd), as long as the draws one hop of all active walks takes span
// at most 624 consecutive numbers: they then lie in the two generations the ring holds.
//
// What bounds it is the dependent random load per hop, so the walks run on the degree-renumbered
// copies of the walk counter (saba.cu): one 8-byte load per hop over the packed copy (the class table
// in shared memory), kSlots of them in flight per lane, most counters in shared memory; r % d is
// two multiplications with floor((2^32 - 1) / d) kept beside d.  The seeding recurrence is
// sequential (623 dependent steps), so kSeedAhead sources are seeded at once, one per lane, into a
// scratch in global memory.  R-MAT scale 16 (n = 46,703, m = 1,819,968), D = 5, W = 2,048:
// 3.1 ms in both draw orders (20.8 over the graph's own arrays with one walk in flight per lane).
#include <algorithm>

#include "common.cuh"
#include "internal.hpp"

namespace tgtp {
namespace {

constexpr uint32_t kMtWords = 624;
constexpr uint32_t kMtShift = 397;
constexpr int kMtThreads = 1024;
constexpr int kSlots = 4;       // walks (bouquets) in flight per lane (8 lanes)
constexpr int kSeedAhead = 4;   // sources a warp seeds at once
constexpr uint32_t kMtHot = 12288;

__device__ __forceinline__ uint32_t mt_temper(uint32_t y) {
    y ^= y >> 11;
    y ^= (y << 7) & 0x9d2c5680u;
    y ^= (y << 15) & 0xefc60000u;
    y ^= y >> 18;
    return y;
}

// Generation 0 of one generator into 16-byte aligned global memory (one lane; the recurrence is
// sequential).
__device__ __forceinline__ void mt_seed(uint32_t* state, uint32_t seed) {
    uint32_t x = seed;
    for (uint32_t i = 0; i < kMtWords; i += 4) {
        uint32_t w[4];
#pragma unroll
        for (uint32_t k = 0; k < 4; ++k) {
            w[k] = x;
            x = 1812433253u * (x ^ (x >> 30)) + (i + k + 1);
        }
        *reinterpret_cast<uint4*>(state + i) = make_uint4(w[0], w[1], w[2], w[3]);
    }
}

// Generation t + 1 from generation t, all lanes of the warp, 224 words at a time.
__device__ __forceinline__ void mt_regenerate(uint32_t* ring, uint32_t t, uint32_t lane) {
    const uint32_t* o = ring + (t & 1u) * kMtWords;
    uint32_t* w = ring + ((t + 1u) & 1u) * kMtWords;
    __syncwarp();  // the draws of the generation this one replaces have been read
#pragma unroll
    for (uint32_t base = 0; base < kMtWords; base += 224) {
        uint32_t v[7];
#pragma unroll
        for (uint32_t c = 0; c < 7; ++c) {
            const uint32_t i = base + c * 32 + lane;
            v[c] = 0;
            if (i < kMtWords) {
                const uint32_t nx = i + 1 < kMtWords ? o[i + 1] : w[0];
                const uint32_t y = (o[i] & 0x80000000u) | (nx & 0x7fffffffu);
                const uint32_t far = i + kMtShift < kMtWords ? o[i + kMtShift] : w[i + kMtShift - kMtWords];
                v[c] = far ^ (y >> 1) ^ ((y & 1u) ? 0x9908b0dfu : 0u);
            }
        }
#pragma unroll
        for (uint32_t c = 0; c < 7; ++c) {
            const uint32_t i = base + c * 32 + lane;
            if (i < kMtWords) w[i] = v[c];
        }
        __syncwarp();
    }
}

// floor((2^32 - 1) / d); then r - umulhi(r, inv) * d lies in [r mod d, r mod d + d], see mt_mod.
__device__ __forceinline__ uint32_t mt_inverse(uint32_t d) { return d ? 0xffffffffu / d : 0u; }

// r mod d with inv = floor((2^32 - 1) / d): 2^32 / d - inv is at most 1, so umulhi(r, inv) is at most
// one below floor(r / d) and one subtraction of d corrects it.
__device__ __forceinline__ uint32_t mt_mod(uint32_t r, uint32_t d, uint32_t inv) {
    const uint32_t rem = r - __umulhi(r, inv) * d;
    return rem >= d ? rem - d : rem;
}

// PACKED: over the packed copy; else over the plain renumbered adjacency and the row records.
template <bool SIMD, bool PACKED>
__global__ void __launch_bounds__(kMtThreads)
mt_walk_kernel(const PackedWalk g, const uint32_t* __restrict__ adjp, uint64_t n, uint32_t depth,
               uint32_t n_walks, WalkCounters cnt, uint32_t hot, uint32_t* seeds) {
    // the class table (8 bytes a class), its inverses, the counters, then per warp the ring
    extern __shared__ __align__(16) uint32_t s_mt[];
    const uint32_t lane = threadIdx.x & 31;
    uint2* s_cls = reinterpret_cast<uint2*>(s_mt);
    uint32_t* s_inv = reinterpret_cast<uint32_t*>(s_cls + (PACKED ? g.ncls : 0u));
    uint32_t* s_cnt = s_inv + (PACKED ? g.ncls : 0u);
    uint32_t* ring = s_mt + (((PACKED ? 3u * g.ncls : 0u) + hot + 3u) & ~3u) + size_t(threadIdx.x >> 5) * 2 * kMtWords;
    if (PACKED)
        for (uint32_t i = threadIdx.x; i < g.ncls; i += blockDim.x) {
            s_cls[i] = __ldg(g.classes + i);
            s_inv[i] = mt_inverse(s_cls[i].y);
        }
    for (uint32_t i = threadIdx.x; i < hot; i += blockDim.x) s_cnt[i] = 0;
    __syncthreads();
    const uint32_t pmask = (1u << g.pbits) - 1u;
    const uint64_t warp = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nwarps = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    uint32_t* my_seeds = seeds + warp * kSeedAhead * kMtWords;
    // a group is one walk (scalar) or one bouquet of 8 walks (simd); it takes `per` draws a hop
    constexpr uint32_t per = SIMD ? 8u : 1u;
    constexpr uint32_t side = SIMD ? 4u : 32u;  // groups of one slot across the warp
    const uint64_t gdraws = uint64_t(per) * depth;  // draws of one group's whole walk
    const uint32_t groups = n_walks / per;
    // groups side by side: the draws of one hop span (G - 1) * gdraws + per <= 624 numbers
    const uint32_t G = uint32_t(min(uint64_t(side) * kSlots, (kMtWords - per) / gdraws + 1));
    const uint32_t grp = SIMD ? lane >> 3 : lane, sub = SIMD ? lane & 7u : 0u;
    uint32_t off[kSlots];  // a slot's draw relative to the first group's (below 624 where active)
#pragma unroll
    for (int u = 0; u < kSlots; ++u) off[u] = uint32_t((u * side + grp) * gdraws) + sub;
    uint32_t seeded = 0;   // sources of this warp already in my_seeds, counted from its first
    uint32_t turn = 0;
    for (uint64_t src = warp; src < n; src += nwarps, ++turn) {
        if (turn == seeded) {  // seed the next kSeedAhead sources, one per lane
            __syncwarp();
            const uint64_t mine = src + lane * nwarps;
            if (lane < kSeedAhead && mine < n) mt_seed(my_seeds + lane * kMtWords, 42u + __ldg(g.info + mine).z);
            seeded += kSeedAhead;
            __syncwarp();
        }
        const uint4 home = __ldg(g.info + src);
        if (home.y == 0) continue;  // isolated (warp-uniform)
        const uint32_t home_inv = mt_inverse(home.y);
        {
            const uint4* from = reinterpret_cast<const uint4*>(my_seeds + (turn % kSeedAhead) * kMtWords);
            __syncwarp();
            for (uint32_t i = lane; i < kMtWords / 4; i += 32) reinterpret_cast<uint4*>(ring)[i] = __ldcg(from + i);
            __syncwarp();
        }
        uint64_t gen = 0;  // newest generation in the ring (the one before it sits in the other half)
        for (uint32_t g0 = 0; g0 < groups; g0 += G) {
            const uint32_t gact = min(G, groups - g0);
            const uint64_t first = uint64_t(g0) * gdraws;  // the first group's first draw
            const uint64_t top = (uint64_t(g0) + gact - 1) * gdraws + (per - 1);
            uint32_t beg[kSlots], d[kSlots], inv[kSlots];
#pragma unroll
            for (int u = 0; u < kSlots; ++u) {
                beg[u] = home.x;
                d[u] = home.y;
                inv[u] = home_inv;
            }
            for (uint32_t j = 0; j < depth; ++j) {
                // the hop's largest draw decides the newest generation needed (warp-uniform); its
                // smallest is less than 624 before, so within the generation before
                const uint64_t kmax = top + uint64_t(j) * per;
                while (gen * kMtWords <= kmax) {
                    mt_regenerate(ring, uint32_t(gen), lane);
                    ++gen;
                }
                // the hop's first draw relative to the newest generation's first (>= -624)
                const int rel = int(int64_t(first + uint64_t(j) * per - (gen - 1) * kMtWords));
                const uint32_t newest = uint32_t(gen & 1u) * kMtWords;
                uint32_t at[kSlots];
                uint2 e[kSlots];
#pragma unroll
                for (int u = 0; u < kSlots; ++u) {
                    if (u * side + grp < gact) {
                        const int x = rel + int(off[u]);
                        const uint32_t r =
                            mt_temper(ring[x >= 0 ? newest + uint32_t(x)
                                                  : kMtWords - newest + uint32_t(x + int(kMtWords))]);
                        at[u] = beg[u] + mt_mod(r, d[u], inv[u]);
                    }
                }
#pragma unroll
                for (int u = 0; u < kSlots; ++u)
                    if (u * side + grp < gact) {
                        if (PACKED) e[u] = __ldg(g.slots + at[u]);
                        else e[u].x = __ldg(adjp + at[u]);
                    }
#pragma unroll
                for (int u = 0; u < kSlots; ++u)
                    if (u * side + grp < gact) {
                        const uint32_t p = PACKED ? e[u].x & pmask : e[u].x;
                        if (j + 1 < depth) {
                            if (PACKED) {
                                const uint32_t c = e[u].x >> g.pbits;
                                const uint2 k = s_cls[c];
                                beg[u] = k.x + p * k.y;
                                d[u] = k.y;
                                inv[u] = s_inv[c];
                            } else {
                                const uint4 k = __ldg(g.info + p);
                                beg[u] = k.x;
                                d[u] = k.y;
                                inv[u] = mt_inverse(k.y);
                            }
                        }
                        if (p < hot) atomicAdd(s_cnt + p, 1u);
                        else atomicAdd(cnt.at(p), 1u);
                    }
            }
        }
    }
    __syncthreads();
    for (uint32_t i = threadIdx.x; i < hot; i += blockDim.x) {
        const uint32_t c = s_cnt[i];
        if (c) atomicAdd(cnt.at(i), c);
    }
}

}  // namespace

void mt_walk_run(tgtp_graph* g, uint32_t depth, uint32_t n_walks, bool simd,
                 uint32_t* device_counters) {
    cudaStream_t s = g->stream;
    const WalkCounters cnt = walk_counters(g);
    if (n_walks == 0 || depth == 0) {
        TGTP_CUDA(cudaMemsetAsync(device_counters, 0, sizeof(uint32_t) * g->n, s));
        return;
    }
    saba_prepare(g);
    const bool packed = saba_prepare_copy(g, saba_packable(g));
    PackedWalk w{};
    if (packed) w = saba_prepare_packed(g);
    else w.info = g->saba_info.as<uint4>();
    auto kern = simd ? (packed ? mt_walk_kernel<true, true> : mt_walk_kernel<true, false>)
                     : (packed ? mt_walk_kernel<false, true> : mt_walk_kernel<false, false>);
    // shared memory: the rings, the classes (12 bytes each), and counters in what is left of it
    // Warps per block: a source each on graphs too small for 32 on every SM (n = 1,000, depth 700, 8
    // walks: 3.36 ms with 32 on each of 32 SMs, 2.39 with seven on each of 143).
    const int warps = int(std::min<uint64_t>(kMtThreads / 32, (g->n + g->num_sms - 1) / g->num_sms));
    const size_t rings = size_t(warps) * 2 * kMtWords;  // words, as are the next two
    const size_t room = size_t(227) * 256 - rings - 3 * size_t(w.ncls) - 4;
    const uint32_t hot = uint32_t(std::min<uint64_t>({g->n, kMtHot, room}));
    const size_t smem = sizeof(uint32_t) * (((3 * size_t(w.ncls) + hot + 3) & ~size_t(3)) + rings);
    const int per_sm = std::max(1, blocks_per_sm(reinterpret_cast<const void*>(kern), warps * 32, smem));
    uint64_t blocks = std::min<uint64_t>(uint64_t(g->num_sms) * per_sm, (g->n + warps - 1) / warps);
    // the generators' states (10 KB a warp); fewer blocks where the device has no room for all
    for (bool there = false; !there;) {
        try {
            g->mt_seeds.reserve(blocks * warps * kSeedAhead * kMtWords * sizeof(uint32_t));
            there = true;
        } catch (const Error& e) {
            if (e.code != TGTP_ERR_OUT_OF_MEMORY || blocks <= 1) throw;
            blocks /= 2;
        }
    }
    {
        ScopedKernel k(g->prof, s, "mt_walk");
        kern<<<unsigned(blocks), unsigned(warps * 32), smem, s>>>(w, g->saba_adj.as<uint32_t>(), g->n, depth, n_walks,
                                                        cnt, hot, g->mt_seeds.as<uint32_t>());
        TGTP_LAUNCH_CHECK("mt_walk_kernel");
    }
    scatter_counters(g, cnt, device_counters);
}

}  // namespace tgtp
