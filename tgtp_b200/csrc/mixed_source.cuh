// Per-source stage of the mixed form: one source per block (included by aesc.cu, inside its
// namespace, after the walk queue's types).
//
// The residual vector lives
//   kShared  in shared memory (graphs up to about 27,900 vertices), as in push_shared_kernel;
//   kGlobal  in global memory, one 64-bit word per vertex and block: sums are added with 64-bit
//            reductions in L2, the touched vertices marked in a bitmap (shared memory up to 819,200
//            vertices), so a round costs its frontier's rows, not n;
//   kColumn  in a column left by a block push, which ran the rounds already.
// Everything after the push (the edge bound, chi and the walk counts, the walks) is shared by the
// block's threads too: with one warp per source the largest source of the 4,039-vertex graph (2,055
// neighbours) alone took as long as the whole kernel.  Against one source per warp (four warps per
// SM in shared memory, twelve with their vectors in HBM), ms: 4,039-vertex graph, eps = 0.005,
// 1.92 -> 0.49; Chung-Lu n = 200,000, m = 4e6, eps = 0.05, 287 -> 133; 16 graphs of 1,000-3,500
// vertices as one batch 9.1 -> 2.25.

enum MixedMode { kShared, kGlobal, kColumn };
constexpr uint32_t kSetMax = 64;              // members of the top-gamma set compared pair by pair
constexpr uint32_t kCandMax = 256;            // candidates for the top-gamma set
constexpr uint64_t kBitsInSmem = 100 * 1024;  // bytes of the bitmap kept in shared memory

struct MixedParams {
    const uint32_t* idx;
    const uint32_t* adj;
    const uint2* adjd;
    const double* dinv;
    uint32_t n;
    const int* taus;
    double* preds;
    unsigned* work;        // [1] error flags, [2] list length
    const uint32_t* rows;  // the listed sources
    double eps, logmd;
    int gamma;
    unsigned long long* stats;
    uint64_t budget_ns;
    unsigned* claim;
    uint32_t* trace_nr;
    uint32_t* trace_ell;
    // per-block scratch, laid out for scratch_n vertices and max_degree slots
    uint32_t scratch_n, max_degree;
    uint4* lists;              // the frontier
    WalkItem* items;
    unsigned long long* sums;  // kGlobal: scratch_n words, all zero between sources
    uint32_t* touched;         // kGlobal: scratch_n vertices
    uint32_t* gbits;           // kGlobal: the bitmap when it is not in shared memory; kShared: see round_with_zeros
    unsigned char* clean;      // kGlobal, per block: 1 = its sums and bitmap are all zero
    // kColumn
    uint32_t list_base, list_cap;
    const PrePush* pre;
    const float* pre_cols;
    const uint32_t* pre_final;
    WalkItem* walk_queue;
    unsigned* walk_count;
    uint32_t walk_cap;
};

template <int N>
struct MixedPack {
    static constexpr int kMax = N;
    uint32_t count;
    MixedParams g[N];
};

struct SourceScratch {
    PushScratch push;
    unsigned long long st[3], ph[8];
    uint32_t hist[kCandMax];  // digit histogram, or the candidates' residuals
    uint32_t cand_v[kCandMax];
    uint32_t set_v[kSetMax], set_r[kSetMax];  // set_r: first the groups' maxima
    uint32_t set_count, cand_count, nth, best, nitems, next_item, smax, smin, bin, rest, graph;
    uint32_t late;  // past the deadline at the claim (push.late: at a round's start; see GsScratch)
};
inline size_t mixed_words(uint64_t n) { return (n + 31) / 32; }
inline size_t mixed_shared_bytes(int mode, uint64_t n) {
    if (mode == kShared) return sizeof(SourceScratch) + 8 * ((n + 3) & ~uint64_t(3));
    if (mode == kGlobal && 4 * mixed_words(n) <= kBitsInSmem) return sizeof(SourceScratch) + 4 * mixed_words(n);
    return sizeof(SourceScratch);
}

// Whether a graph's sums fit beside the scratch and the item prefix (static).
inline bool mixed_fits_shared(uint64_t n) { return mixed_shared_bytes(kShared, n) + 1024 <= 227 * 1024; }

// The rg-th largest (counting repeats) of the positive values value(i), i < count, as FP32 bits:
// the digits are fixed eight bits at a time from a histogram of the values that share the digits
// fixed so far; 0 when fewer than rg values are positive.  All threads of the block call it.
template <class Value>
__device__ __forceinline__ uint32_t block_nth_largest(SourceScratch& s, uint32_t count, uint32_t rg, Value value) {
    uint32_t prefix = 0, rest = rg;
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) s.hist[i] = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
            const uint32_t x = value(i);
            if (x != 0 && (shift == 24 || (x >> (shift + 8)) == prefix)) atomicAdd(s.hist + ((x >> shift) & 255u), 1u);
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // the bin, from the top, where the running count reaches rest
            const uint32_t lane = threadIdx.x;
            uint32_t h[8], sum = 0;  // lane l holds bins 255 - 8 l .. 248 - 8 l
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                h[k] = s.hist[255u - 8u * lane - uint32_t(k)];
                sum += h[k];
            }
            uint32_t incl = sum;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= uint32_t(o)) incl += y;
            }
            const unsigned reach = __ballot_sync(kFullMask, incl >= rest);
            if (!reach && lane == 0) s.rest = 0;  // too few (seen at the first digit)
            if (lane == uint32_t(__ffs(int(reach)) - 1)) {
                uint32_t left = rest - (incl - sum);
                int k = 0;
                while (k < 7 && left > h[k]) left -= h[k++];
                s.bin = 255u - 8u * lane - uint32_t(k);
                s.rest = left;
            }
        }
        __syncthreads();
        prefix = (prefix << 8) | s.bin;
        rest = s.rest;
        if (rest == 0) return 0;
    }
    return prefix;
}

// The rg-th largest of 32 K values, K per lane of one warp (0: none), counting repeats; rg of them
// are positive.
template <int K>
__device__ __forceinline__ uint32_t warp_nth_largest(uint32_t (&x)[K], uint32_t rg) {
    uint32_t top = 0;
    for (uint32_t left = rg;;) {
        uint32_t mx = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) mx = max(mx, x[k]);
        top = __reduce_max_sync(kFullMask, mx);
        uint32_t c = 0;
#pragma unroll
        for (int k = 0; k < K; ++k)
            if (x[k] == top) {
                ++c;
                x[k] = 0;
            }
        c = __reduce_add_sync(kFullMask, c);
        if (c >= left || top == 0) return top;
        left -= c;
    }
}

// The top-gamma set of the edge bound: the rg-th largest t (rg <= kSetMax) of the positive values
// value(i), i < count, of which there are at least rg, and the set {value > t} in set_v / set_r
// (set_count of them); returns t.  64 groups of threads take their maxima; the rg-th largest of
// those is at most t, so two passes over the values find the few candidates at or above it.  When
// too many tie with it (more than kCandMax candidates) the digits of t are found instead.
template <class Value, class Vertex>
__device__ __forceinline__ uint32_t block_top_set(SourceScratch& s, uint32_t count, uint32_t rg, Value value,
                                                  Vertex vertex) {
    constexpr int U = 4;
    const uint32_t tid = threadIdx.x, lane = tid & 31, per_group = blockDim.x / 64u;
    uint32_t mx = 0;
    for (uint32_t i0 = tid; i0 < count; i0 += U * blockDim.x) {
        uint32_t x[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const uint32_t i = i0 + k * blockDim.x;
            x[k] = i < count ? value(i) : 0u;
        }
#pragma unroll
        for (int k = 0; k < U; ++k) mx = max(mx, x[k]);
    }
    for (uint32_t o = per_group >> 1; o; o >>= 1) mx = max(mx, __shfl_xor_sync(kFullMask, mx, int(o)));
    if (tid % per_group == 0) s.set_r[tid / per_group] = mx;
    __syncthreads();
    uint32_t g[2] = {s.set_r[lane], s.set_r[32 + lane]};
    const uint32_t low = max(1u, warp_nth_largest<2>(g, rg));  // the same in every warp
    for (uint32_t i0 = tid; i0 < count; i0 += U * blockDim.x) {
        uint32_t x[U];
#pragma unroll
        for (int k = 0; k < U; ++k) {
            const uint32_t i = i0 + k * blockDim.x;
            x[k] = i < count ? value(i) : 0u;
        }
#pragma unroll
        for (int k = 0; k < U; ++k)
            if (x[k] >= low) {
                const uint32_t at = atomicAdd(&s.cand_count, 1u);
                if (at < kCandMax) {
                    s.hist[at] = x[k];
                    s.cand_v[at] = vertex(i0 + k * blockDim.x);
                }
            }
    }
    __syncthreads();
    const uint32_t c = s.cand_count;
    if (c > kCandMax) {
        const uint32_t t = block_nth_largest(s, count, rg, value);
        for (uint32_t i = tid; i < count; i += blockDim.x) {
            const uint32_t x = value(i);
            if (x > t) {
                const uint32_t at = atomicAdd(&s.set_count, 1u);
                s.set_r[at] = x;
                s.set_v[at] = vertex(i);
            }
        }
        __syncthreads();
        return t;
    }
    if (tid < 32) {
        uint32_t x[kCandMax / 32];
#pragma unroll
        for (int k = 0; k < int(kCandMax / 32); ++k) x[k] = 32u * k + lane < c ? s.hist[32u * k + lane] : 0u;
        const uint32_t t = warp_nth_largest<kCandMax / 32>(x, rg);
        for (uint32_t i = lane; i < c; i += 32)
            if (s.hist[i] > t) {
                const uint32_t at = atomicAdd(&s.set_count, 1u);
                s.set_r[at] = s.hist[i];
                s.set_v[at] = s.cand_v[i];
            }
        if (lane == 0) s.nth = t;
    }
    __syncthreads();
    return s.nth;
}

// Exclusive prefix over the block of the set bits of `words` words; their positions in increasing
// order per thread's run of words go to out, the words are cleared.  Returns the count.
__device__ __forceinline__ uint32_t drain_bits(PushScratch& s, uint32_t* bits, uint32_t words, uint32_t* out) {
    const uint32_t per = (words + blockDim.x - 1) / blockDim.x;
    const uint32_t w0 = min(words, threadIdx.x * per), w1 = min(words, w0 + per);
    uint32_t c = 0;
    for (uint32_t w = w0; w < w1; ++w) c += __popc(bits[w]);
    uint32_t at = block_exclusive_scan(c, s.chunk.tmp, &s.chunk.total);
    for (uint32_t w = w0; w < w1; ++w) {
        uint32_t b = bits[w];
        if (b) bits[w] = 0u;
        while (b) {
            out[at++] = w * 32u + uint32_t(__ffs(int(b)) - 1);
            b &= b - 1;
        }
    }
    return s.chunk.total;
}

// A round of kShared in which a residual may be 0.  Every vertex a frontier vertex reaches is in the
// next frontier, also one whose residual rounds to 0 (below 2^-62) or is a sum of such.  A vertex's sum
// is at least one frontier residual, so its residual is above 0 while the smallest of them is at least
// the largest degree in 2^-62; the other rounds (far vertices of grids and the like, after 30 rounds
// and more) come here, where the neighbours of the frontier's zeros have bits of their own (all clear
// between rounds).  The block pushes leave vertices with residual 0 out, so where there are some a
// source may stop at another round than here.  A function of its own, because the other rounds pay
// for code around them: 4,039-vertex graph, eps = 0.005, 484 us without it, 490 so, 487 to 503 with the
// marking inside take_residuals or the push; batch of 16 graphs 2.18 ms, 2.21, 2.23 to 2.33.
__device__ __noinline__ void round_with_zeros(PushScratch& s, uint32_t* lo, uint32_t* hi, uint32_t* bits,
                                              const uint32_t* __restrict__ idx, const uint32_t* __restrict__ adj,
                                              const double* __restrict__ dinv, uint32_t n, const Frontier& f,
                                              uint32_t nl, uint32_t nh) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    push_frontier(s, f, nl, nh, adj, [&](uint32_t u, unsigned long long v) { add_fixed(lo, hi, u, v); });
    for (uint32_t i = warp; i < nl + nh; i += nw) {
        const uint4 v = f.list[i < nl ? i : f.cap - 1u - (i - nl)];
        if (v.z) continue;
        for (uint32_t o = lane; o < v.y; o += 32) {
            const uint32_t u = __ldg(adj + v.x + o);
            atomicOr(bits + (u >> 5), 1u << (u & 31u));
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) reset_sums(s);
    __syncthreads();
    FrontierSums t;
    for (uint32_t w = warp; w < (n + 31u) / 32u; w += nw) {
        const uint32_t x = __ldcg(bits + w);
        const uint32_t v = w * 32u + lane;
        uint32_t u[1] = {kNoVertex}, b[1] = {0u}, d[1] = {1u};
        float r[1] = {0.f};
        if (v < n) {
            const uint32_t sl = lo[v], sh = hi[v];
            b[0] = __ldg(idx + v);
            d[0] = __ldg(idx + v + 1) - b[0];
            if (sl | sh) {
                r[0] = from_fixed(sh, sl, d[0], __ldg(dinv + v));
                lo[v] = __float_as_uint(r[0]);
                hi[v] = 0u;
            }
            if ((sl | sh) || ((x >> lane) & 1u)) u[0] = v;
        }
        append_frontier<1, true>(s, f, t, u, b, d, r);
        if (lane == 0 && x) bits[w] = 0u;
    }
    add_sums(s, t);
}

template <int MODE, class Pack>
__global__ void __launch_bounds__(1024, 1) mixed_source_kernel(const Pack pk) {
    extern __shared__ __align__(16) unsigned char mixed_smem[];
    __shared__ uint32_t s_pre[Pack::kMax + 1];  // item prefix over the pack's row lists
    SourceScratch& S = *reinterpret_cast<SourceScratch*>(mixed_smem);
    PushScratch& s = S.push;
    const MixedParams& p0 = pk.g[0];
    const uint32_t tid = threadIdx.x, lane = tid & 31, nw = blockDim.x >> 5;
    const uint32_t sn = p0.scratch_n, pad = (sn + 3u) & ~3u;
    uint32_t* const smem_words = reinterpret_cast<uint32_t*>(mixed_smem + sizeof(SourceScratch));
    uint32_t* const lo = smem_words;        // kShared
    uint32_t* const hi = smem_words + pad;  // kShared
    const uint32_t bwords = (sn + 31u) / 32u;
    const bool bits_here = MODE == kGlobal && !p0.gbits;
    uint32_t* const gbits = MODE == kShared || (MODE == kGlobal && !bits_here)
                                ? p0.gbits + size_t(blockIdx.x) * bwords
                                : nullptr;
    unsigned long long* const sums = MODE == kGlobal ? p0.sums + size_t(blockIdx.x) * sn : nullptr;
    uint32_t* const touched = MODE == kGlobal ? p0.touched + size_t(blockIdx.x) * sn : nullptr;
    const Frontier f{p0.lists + size_t(blockIdx.x) * sn, sn};
    WalkItem* const items = p0.items + size_t(blockIdx.x) * p0.max_degree;
    if (MODE == kShared)
        for (uint32_t u = tid; u < 2 * pad; u += blockDim.x) lo[u] = 0u;
    if (bits_here)
        for (uint32_t w = tid; w < bwords; w += blockDim.x) smem_words[w] = 0u;
    pdl_launch_dependents();
    pdl_wait();  // taus and row lists of the tau kernels; the columns of a block push
    if (MODE == kShared)
        for (uint32_t w = tid; w < bwords; w += blockDim.x) gbits[w] = 0u;
    if (MODE == kGlobal && !p0.clean[blockIdx.x]) {
        for (uint32_t u = tid; u < sn; u += blockDim.x) sums[u] = 0ull;
        if (gbits)
            for (uint32_t w = tid; w < bwords; w += blockDim.x) gbits[w] = 0u;
    }
    // items: the listed rows of the pack's graphs one after another (kColumn: this wave's rows)
    if (tid < 32) {
        uint32_t carry = 0;
        for (uint32_t k0 = 0; k0 < pk.count; k0 += 32) {
            uint32_t incl = k0 + lane < pk.count ? pk.g[k0 + lane].work[2] : 0u;
            if (MODE == kColumn) incl = incl > p0.list_base ? min(incl - p0.list_base, p0.list_cap) : 0u;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
                if (lane >= uint32_t(o)) incl += y;
            }
            if (k0 + lane < pk.count) s_pre[k0 + lane + 1] = carry + incl;
            carry += __shfl_sync(kFullMask, incl, 31);
        }
        if (lane == 0) s_pre[0] = 0;
    }
    const uint64_t deadline = globaltimer_ns() + p0.budget_ns;
    // run counters: the push's (rounds, vertices, traversals) and the phases' by thread 0 in shared
    // memory, the walks' per thread
    if (tid < 3) S.st[tid] = 0;
    if (tid < 8) S.ph[tid] = 0;
    unsigned long long st_we = 0, st_wc = 0, st_wh = 0, st_fb = 0;
    // SM cycles per phase as thread 0 sees them, counted once per warp of the block
    long long tmark = clock64();
    auto lap = [&](int i) {
        if (tid == 0) {
            const long long now = clock64();
            S.ph[i] += (unsigned long long)(now - tmark) * nw;
            tmark = now;
        }
    };
    auto flush_stats = [&](unsigned long long* stats) {
        st_we = warp_sum_u64(st_we);
        st_wc = warp_sum_u64(st_wc);
        st_wh = warp_sum_u64(st_wh);
        st_fb = warp_sum_u64(st_fb);
        if (lane == 0) {
            stat_add(stats, kStWalkEdges, st_we);
            stat_add(stats, kStWalkCount, st_wc);
            stat_add(stats, kStWalkHops, st_wh);
            stat_add(stats, kStFallback, st_fb);
        }
        if (tid == 0) {
            stat_add(stats, kStPushRounds, S.st[0]);
            stat_add(stats, kStPushVertices, S.st[1]);
            stat_add(stats, kStPushTraversals, S.st[2]);
            for (int i = 0; i < 8; ++i) stat_add(stats, kStPhase0 + i, S.ph[i]);
            for (int i = 0; i < 3; ++i) S.st[i] = 0;
            for (int i = 0; i < 8; ++i) S.ph[i] = 0;
        }
        st_we = st_wc = st_wh = st_fb = 0;
    };
    uint32_t last_gi = 0xffffffffu;
    bool dirty = false;
    while (true) {
        __syncthreads();  // s_pre is complete, or the previous source is done with the scratch
        if (tid == 0) {
            const uint32_t k = atomicAdd(p0.claim, 1u);
            uint32_t gi = 0;  // the item's graph: the last list whose prefix is at most k
            for (uint32_t h = pk.count; h - gi > 1;) {
                const uint32_t mid = (gi + h) >> 1;
                if (s_pre[mid] <= k) gi = mid;
                else h = mid;
            }
            s.k = k;
            S.graph = gi;
            S.late = globaltimer_ns() > deadline;
            reset_sums(s);
            S.nitems = S.next_item = S.set_count = S.cand_count = 0;
            S.smax = S.best = 0;
            S.smin = __float_as_uint(FLT_MAX);
        }
        __syncthreads();
        const uint32_t item = s.k, gi = S.graph;
        if (item >= s_pre[pk.count]) break;
        const MixedParams& p = pk.g[gi];
        if (gi != last_gi) {
            if (last_gi != 0xffffffffu) flush_stats(pk.g[last_gi].stats);
            last_gi = gi;
        }
        if (S.late) {
            if (tid == 0) atomicOr(p.work + 1, kErrDeadline);
            break;
        }
        const uint32_t n = p.n;
        const uint32_t* __restrict__ idx = p.idx;
        const uint32_t* __restrict__ adj = p.adj;
        const uint32_t entry = (item - s_pre[gi]) + (MODE == kColumn ? p.list_base : 0u);
        const uint32_t src = __ldg(p.rows + entry);
        const uint32_t rb = __ldg(idx + src), dsi = __ldg(idx + src + 1) - rb;
        const float ds = float(dsi);
        const float* col = nullptr;
        if (MODE == kColumn) col = pre_column(p.pre_cols, p.pre_final, entry - p.list_base, n);
        // the residual of vertex u (between rounds)
        auto pv = [&](uint32_t u) -> float {
            if (MODE == kShared) return __uint_as_float(lo[u]);
            if (MODE == kGlobal) return __uint_as_float(__ldcg(reinterpret_cast<const uint32_t*>(sums + u)));
            return __ldg(col + u);
        };
        lap(0);
        uint32_t nl = 0, nh = 0, qs = 0;
        int ell = 1;
        float gmax, gmin;
        bool timed_out = false;
        if (MODE == kColumn) {
            const PrePush r = p.pre[entry];
            ell = r.ell;
            gmax = r.gmax;
            qs = r.support;
            gmin = qs < n ? 0.f : r.gmin;
        } else {
            // ---- push (src/aesc.h:456-503) ----
            first_round(s, f, p.adjd, idx, rb, dsi, p.preds, [&](uint32_t u, float r) {
                if (MODE == kShared) lo[u] = __float_as_uint(r);
                else sums[u] = __float_as_uint(r);
            });
            if (tid == 0) {
                S.st[1] += 1;
                S.st[2] += dsi;
            }
            lap(1);
            while (true) {
                if (tid == 0) s.late = globaltimer_ns() > deadline;
                __syncthreads();
                nl = s.light;
                nh = s.heavy;
                qs = nl + nh;
                gmax = __uint_as_float(s.gmax);
                gmin = qs < n ? 0.f : __uint_as_float(s.gmin);
                const bool stop = block_stops(s, p.taus, rb, dsi, ell, gmax, gmin, p.eps, p.logmd);
                lap(3);
                timed_out = s.late != 0 && !stop;
                if (stop || timed_out) break;
                if (tid == 0) {
                    S.st[1] += qs;
                    S.st[2] += s.picost;
                }
                // the old residuals leave the vector before the round's sums start
                if (MODE == kShared && qs * 4u > n) {
                    for (uint32_t u = tid; u < n; u += blockDim.x) lo[u] = 0u;
                } else {
                    for (uint32_t i = tid; i < qs; i += blockDim.x) {
                        const uint32_t u = f.list[i < nl ? i : sn - 1u - (i - nl)].w;
                        if (MODE == kShared) lo[u] = 0u;
                        else sums[u] = 0ull;
                    }
                }
                __syncthreads();
                if (MODE == kShared && to_fixed(__uint_as_float(s.gmin)) < p0.max_degree) {
                    round_with_zeros(s, lo, hi, gbits, idx, adj, p.dinv, n, f, nl, nh);
                } else {
                    push_frontier(s, f, nl, nh, adj, [&](uint32_t u, unsigned long long v) {
                        if (MODE == kShared) {
                            add_fixed(lo, hi, u, v);
                        } else {
                            atomicAdd(sums + u, v);
                            if (bits_here) atomicOr(smem_words + (u >> 5), 1u << (u & 31u));
                            else atomicOr(gbits + (u >> 5), 1u << (u & 31u));
                        }
                    });
                    __syncthreads();
                    if (tid == 0) reset_sums(s);
                    __syncthreads();
                    if (MODE == kShared) {
                        take_residuals(s, lo, hi, idx, p.dinv, n, f);
                    } else {
                        const uint32_t count = drain_bits(s, bits_here ? smem_words : gbits, (n + 31u) / 32u, touched);
                        __syncthreads();
                        constexpr int K = 4;
                        FrontierSums t;
                        for (uint32_t i0 = tid - lane; i0 < count; i0 += K * blockDim.x) {
                            uint32_t u[K], b[K], d[K];
                            float r[K];
                            unsigned long long sum[K];
                            double inv[K];
#pragma unroll
                            for (int k = 0; k < K; ++k) {
                                const uint32_t i = i0 + k * blockDim.x + lane;
                                u[k] = i < count ? touched[i] : kNoVertex;
                            }
#pragma unroll
                            for (int k = 0; k < K; ++k) {
                                sum[k] = 0;
                                b[k] = 0;
                                d[k] = 1;
                                inv[k] = 1.0;
                                if (u[k] != kNoVertex) {
                                    sum[k] = __ldcg(sums + u[k]);
                                    b[k] = __ldg(idx + u[k]);
                                    d[k] = __ldg(idx + u[k] + 1);
                                    inv[k] = __ldg(p.dinv + u[k]);
                                }
                            }
#pragma unroll
                            for (int k = 0; k < K; ++k) {
                                r[k] = 0.f;
                                d[k] -= b[k];
                                if (sum[k]) {
                                    r[k] = from_fixed(uint32_t(sum[k] >> 32), uint32_t(sum[k]), d[k], inv[k]);
                                    sums[u[k]] = __float_as_uint(r[k]);
                                }
                            }
                            append_frontier<K, true>(s, f, t, u, b, d, r);
                        }
                        add_sums(s, t);
                    }
                }
                __syncthreads();
                lap(1);
                // preds[row] += (r[src] - r[t]) / ds (:235-237)
                const float ps = pv(src);
                for (uint32_t o = tid; o < dsi; o += blockDim.x) {
                    const uint32_t w = __ldg(adj + rb + o);
                    p.preds[rb + o] = row_update<float, double>(p.preds[rb + o], ps, pv(w), ds);
                }
                ++ell;
                lap(2);
            }
            if (timed_out) {
                if (tid == 0) atomicOr(p.work + 1, kErrDeadline);
                dirty = true;
                break;
            }
            if (tid == 0) S.st[0] += uint64_t(ell);
        }
        if (p.trace_ell && tid == 0) p.trace_ell[src] = uint32_t(ell);

        // ---- slots that still need walks (rest = tau - ell > 0), with the row's extremes ----
        {
            uint32_t mx = 0, mn = __float_as_uint(FLT_MAX);
            for (uint32_t o0 = tid - lane; o0 < dsi; o0 += blockDim.x) {
                const uint32_t o = o0 + lane;
                uint32_t v = 0;
                int rest = 0;
                if (o < dsi) {
                    v = __ldg(adj + rb + o);
                    rest = __ldg(p.taus + rb + o) - ell;
                    const uint32_t x = __float_as_uint(pv(v));
                    mx = max(mx, x);
                    mn = min(mn, x);
                }
                const unsigned hb = __ballot_sync(kFullMask, rest > 0);
                if (hb) {
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(&S.nitems, uint32_t(__popc(hb)));
                    at = __shfl_sync(kFullMask, at, 0) + uint32_t(__popc(hb & ((1u << lane) - 1u)));
                    if (rest > 0) items[at] = WalkItem{rb + o, v, uint32_t(rest), entry, 0ull};
                }
            }
            mx = __reduce_max_sync(kFullMask, mx);
            mn = __reduce_min_sync(kFullMask, mn);
            if (lane == 0) {
                atomicMax(&S.smax, mx);
                atomicMin(&S.smin, mn);
            }
        }
        __syncthreads();
        const uint32_t nitems = S.nitems;
        if (nitems) {
            // ---- edge bound (:414-442, :504-506) ----
            // edge_max starts at gmax + min(1, t), t the gamma-th largest residual, and is raised by
            // pairs of adjacent vertices of the top-gamma set.  A member equal to t cannot raise it
            // (residuals do not exceed gmax, rounding is monotone), so the set is {r > t}.
            float edge_max;
            // the values: the list, or the whole vector where it is the shorter or the nearer
            const bool dense = MODE == kColumn || (MODE == kShared && qs * 4u > n);
            const uint32_t total = dense ? n : qs;
            auto at_list = [&](uint32_t i) -> uint32_t { return i < nl ? i : sn - 1u - (i - nl); };
            auto value = [&](uint32_t i) -> uint32_t {  // bits of a non-negative residual
                return dense ? __float_as_uint(pv(i)) : f.list[at_list(i)].z;
            };
            auto vertex = [&](uint32_t i) -> uint32_t { return dense ? i : f.list[at_list(i)].w; };
            if (p.gamma == 1) {
                edge_max = __fmul_rn(2.f, gmax);
            } else {
                const bool all = uint32_t(p.gamma) >= qs;  // every frontier vertex is in the set
                const bool small = (all ? qs : uint32_t(p.gamma)) <= kSetMax;
                uint32_t t = 0;
                if (!all && small) {
                    t = block_top_set(S, total, uint32_t(p.gamma), value, vertex);
                } else if (!all) {
                    t = block_nth_largest(S, total, uint32_t(p.gamma), value);
                } else if (small) {
                    for (uint32_t i = tid; i < total; i += blockDim.x) {
                        const uint32_t x = value(i);
                        if (x) {
                            const uint32_t at = atomicAdd(&S.set_count, 1u);
                            S.set_r[at] = x;
                            S.set_v[at] = vertex(i);
                        }
                    }
                    __syncthreads();
                }
                edge_max = __fadd_rn(gmax, all ? 0.f : std_min(1.f, __uint_as_float(t)));
                uint32_t best = 0;
                if (small) {
                    const uint32_t c = S.set_count;
                    for (uint32_t q = tid; q < c * c; q += blockDim.x) {
                        const uint32_t i = q / c, j = q % c;
                        if (i >= j) continue;
                        if (adjacent(idx, adj, S.set_v[i], S.set_v[j]))
                            best = max(best, __float_as_uint(__fadd_rn(__uint_as_float(S.set_r[i]),
                                                                       __uint_as_float(S.set_r[j]))));
                    }
                } else {
                    // the members' rows, each neighbour's residual compared with t
                    const uint32_t per = min(kChunk, blockDim.x);
                    for (uint32_t i0 = 0; i0 < total; i0 += blockDim.x) {
                        const uint32_t i = i0 + tid;
                        const uint32_t x = i < total ? value(i) : 0u;
                        const uint32_t v = x > t ? vertex(i) : 0u;
                        // this step's members to the front of the block, per at a time
                        uint32_t count;
                        __syncthreads();
                        const uint32_t rank = block_exclusive_scan(x > t ? 1u : 0u, s.chunk.tmp, &s.chunk.total);
                        count = s.chunk.total;
                        __syncthreads();
                        for (uint32_t c0 = 0; c0 < count; c0 += per) {
                            const uint32_t cnt = min(per, count - c0);
                            if (x > t && rank >= c0 && rank - c0 < cnt) {
                                s.chunk.base[rank - c0] = v;
                                s.chunk.val[rank - c0] = x;
                            }
                            __syncthreads();
                            uint32_t beg = 0, deg = 0;
                            unsigned long long r = 0;
                            if (tid < cnt) {
                                const uint32_t m = s.chunk.base[tid];
                                beg = __ldg(idx + m);
                                deg = __ldg(idx + m + 1) - beg;
                                r = s.chunk.val[tid];
                            }
                            __syncthreads();
                            for_entries(
                                s.chunk, cnt, beg, deg, r,
                                [&](uint32_t slot, bool in) { return in ? __ldg(adj + slot) : 0u; },
                                [&](uint32_t w, unsigned long long m, uint32_t, bool in) {
                                    const float y = in ? pv(w) : 0.f;
                                    if (__float_as_uint(y) > t)
                                        best = max(best, __float_as_uint(__fadd_rn(
                                                             __uint_as_float(uint32_t(m)), y)));
                                });
                            __syncthreads();
                        }
                    }
                }
                best = __reduce_max_sync(kFullMask, best);
                if (lane == 0 && best) atomicMax(&S.best, best);
                __syncthreads();
                edge_max = std_max(edge_max, __uint_as_float(S.best));
            }
            lap(4);

            // ---- chi and walk counts per edge (:392-412, :508-521) ----
            const float smax = __uint_as_float(S.smax), smin = __uint_as_float(S.smin);
            const float dse = __double2float_rn(__dmul_rn(double(ds), p.eps));
            const double den = double(__fmul_rn(dse, dse));
            const uint32_t per = min(kChunk, blockDim.x);
            for (uint32_t i0 = 0; i0 < nitems; i0 += per) {
                const uint32_t cnt = min(per, nitems - i0);
                uint32_t beg = 0, deg = 0;
                if (tid < cnt) {
                    const uint32_t v = items[i0 + tid].v;
                    beg = __ldg(idx + v);
                    deg = __ldg(idx + v + 1) - beg;
                }
                __syncthreads();  // the previous chunk's scratch is no longer read
                // val holds the target's neighbourhood: largest residual in the low word, smallest
                // in the high one
                uint32_t* const ext = reinterpret_cast<uint32_t*>(s.chunk.val);
                for_entries(
                    s.chunk, cnt, beg, deg, static_cast<unsigned long long>(__float_as_uint(FLT_MAX)) << 32,
                    [&](uint32_t slot, bool in) { return in ? __float_as_uint(pv(__ldg(adj + slot))) : 0u; },
                    [&](uint32_t x, unsigned long long, uint32_t k, bool in) {
                        const uint32_t k0 = __shfl_sync(kFullMask, k, 0);  // lane 0 always has an entry
                        if (__all_sync(kFullMask, !in || k == k0)) {  // one row: reduced across the warp
                            const uint32_t mx = __reduce_max_sync(kFullMask, x);
                            const uint32_t mn = __reduce_min_sync(kFullMask, in ? x : 0xffffffffu);
                            if (lane == 0) {
                                atomicMax(ext + 2 * k, mx);
                                atomicMin(ext + 2 * k + 1, mn);
                            }
                        } else if (in) {
                            atomicMax(ext + 2 * k, x);
                            atomicMin(ext + 2 * k + 1, x);
                        }
                    });
                __syncthreads();
                if (tid < cnt) {
                    WalkItem it = items[i0 + tid];
                    const float tmax = __uint_as_float(ext[2 * tid]), tmin = __uint_as_float(ext[2 * tid + 1]);
                    // get_chi (:410): float terms rounded as in the reference, summed in double
                    const int Li = int(it.len);
                    const double A = __dadd_rn(double(gmax), __ddiv_rn(double(__fadd_rn(smax, tmax)), 2.0));
                    const double B = __dadd_rn(A, double(__fmul_rn(float(Li - 1), edge_max)));
                    const double C = __dsub_rn(__dsub_rn(B, double(smin)), double(tmin));
                    const double E = __dsub_rn(C, double(__fmul_rn(float(2 * (Li - 1)), gmin)));
                    const float chi = __double2float_rn(E);
                    // nr (:519-521)
                    const double num = __dmul_rn(double(__fmul_rn(8.f, __fmul_rn(chi, chi))), p.logmd);
                    const double nrd = std_max(ceil(__ddiv_rn(num, den)), 1.0);
                    unsigned long long nr = (unsigned long long)nrd;
                    nr += 8ull - (nr % 8ull);
                    if (nr > kMaxWalks) {
                        atomicOr(p.work + 1, kErrWalkCount);
                        nr = 0;  // skipped by the walk loop
                    } else {
                        st_we += 1;
                        st_wc += nr;
                        st_wh += nr * (unsigned long long)it.len;
                    }
                    items[i0 + tid].nr = nr;
                    if (p.trace_nr) p.trace_nr[it.pos] = uint32_t(nr);
                    if (MODE == kColumn) {
                        // handed to walk_queue_kernel / heavy_walk_kernel: light items from the
                        // front, heavy ones from the back
                        it.nr = nr;
                        const bool heavy = nr >= kHeavyNr && it.len <= kHeavyLen;
                        const uint32_t at = atomicAdd(p.walk_count + (heavy ? 2 : 0), 1u);
                        p.walk_queue[heavy ? p.walk_cap - 1u - at : at] = it;
                    }
                }
            }
            __syncthreads();
            lap(5);

            // ---- 2-way bouquet walks (:241-391): an 8-lane group per item, as walk_queue_kernel ----
            if (MODE != kColumn) {
                const uint32_t j = lane & 7, grp = lane >> 3;
                bool has = false, start = false, primary = true, done = false;
                WalkItem it{};
                unsigned long long bi = 0;
                uint32_t len = 0, step = 0, cur = 0, cur2 = 0, sec = 0, sec2 = 0, state = 0;
                float x = 0.f, pa = 0.f, pb = 0.f;
                bool pend = false;
                while (true) {
                    if (!has && !done) {
                        uint32_t my = 0;
                        if (j == 0) my = atomicAdd(&S.next_item, 1u);
                        my = __shfl_sync(0xffu << (grp * 8), my, int(grp * 8));
                        if (my >= nitems) {
                            done = true;
                        } else {
                            it = items[my];
                            if (it.nr) {
                                has = true;
                                start = true;
                                bi = 0;
                                x = 0.f;
                                step = uint32_t(0xffffffffull / it.nr);
                            }
                        }
                    }
                    if (!__any_sync(kFullMask, has || !done)) break;
                    if (has && start) {
                        cur = src;
                        cur2 = it.v;
                        sec = (uint32_t(bi) + j + 1u) * step;
                        sec2 = sec;
                        state = sec;
                        primary = true;
                        len = 0;
                        start = false;
                    }
                    const unsigned z = __ballot_sync(kFullMask, has && primary && (sec == 0u || sec2 == 0u));
                    if (has && primary && ((z >> (grp * 8)) & 0xffu)) {
                        primary = false;
                        if (j == 0) ++st_fb;
                    }
                    bool item_done = false;
                    if (has) {
                        const uint32_t b1 = __ldg(idx + cur), d1 = __ldg(idx + cur + 1) - b1;
                        const uint32_t b2 = __ldg(idx + cur2), d2 = __ldg(idx + cur2 + 1) - b2;
                        if (pend) x = __fadd_rn(x, __fsub_rn(pa, pb));
                        uint32_t k1, k2;
                        if (primary) {
                            k1 = __umulhi(sec ^ fmix32(cur), d1);
                            k2 = __umulhi(sec2 ^ fmix32(cur2), d2);
                            sec *= d1;
                            sec2 *= d2;
                        } else {
                            const uint32_t r1 = splitmix32(state);
                            const uint32_t r2 = splitmix32(state);
                            k1 = r1 % d1;
                            k2 = r2 % d2;
                        }
                        cur = __ldg(adj + b1 + k1);
                        cur2 = __ldg(adj + b2 + k2);
                        pa = pv(cur);
                        pb = pv(cur2);
                        pend = true;
                        if (++len == it.len) {
                            bi += 8;
                            start = true;
                            item_done = bi >= it.nr;
                        }
                    }
                    if (__any_sync(kFullMask, item_done)) {
                        if (item_done && pend) {
                            x = __fadd_rn(x, __fsub_rn(pa, pb));
                            pend = false;
                        }
                        double sum = 0;
#pragma unroll
                        for (int b = 0; b < 8; ++b) sum += double(__shfl_sync(kFullMask, x, int(grp * 8 + b)));
                        if (item_done && j == 0) p.preds[it.pos] += sum / (double(ds) * double(it.nr));
                        if (item_done) has = false;
                    }
                }
                __syncthreads();
            }
            lap(6);
        }
        // ---- the next source starts from an all-zero vector ----
        if (MODE == kShared && qs * 4u > n) {
            for (uint32_t u = tid; u < n; u += blockDim.x) lo[u] = 0u;
        } else if (MODE != kColumn) {
            for (uint32_t i = tid; i < qs; i += blockDim.x) {
                const uint32_t u = f.list[i < nl ? i : sn - 1u - (i - nl)].w;
                if (MODE == kShared) lo[u] = 0u;
                else sums[u] = 0ull;
            }
        }
        lap(7);
    }
    if (MODE == kGlobal && tid == 0) p0.clean[blockIdx.x] = dirty ? 0 : 1;
    flush_stats(pk.g[last_gi == 0xffffffffu ? 0u : last_gi].stats);
}
