// Per-source stage of the FP32 and FP64 forms (included by aesc.cu, inside its namespace): one source
// per block.  Warp 0 pushes, in the reference's sequential (Gauss-Seidel) order; everything else --
// the first round, the row updates, the cost test, the edge bound, chi and the walk counts, the
// walks -- is shared by the block's threads.
//
// The push is a chain of dependent updates, so what counts is the latency of one 32-entry step and
// the number of sources in flight.  A discovered vertex is marked by the sign bit of its residual
// (residuals are never negative), so an entry touches one word and not a residual and a flag; window
// membership is looked up in a bit filter in shared memory; the adjacency is read two steps ahead
// and, where the residuals live in HBM, the words of the next step are brought to L1 while a step is
// applied; r / deg(u) is formed from the vertex's reciprocal (div_fixed).
//
// Against one warp per source, half as many sources in flight and a flag array beside the residuals
// (per call): FP64, n = 4,039, 44 neighbours, eps = 0.005, 1.55 -> 0.87 ms; FP32 there, eps = 0.01, 0.62
// -> 0.36 ms; FP64, n = 25,860, 9 neighbours, eps = 0.05 (HBM tier), 290 -> 145 ms.  A step still waits
// on a shared-memory or L2 round trip: 0.14 (shared memory) and 0.22 (HBM) instructions per cycle and
// scheduler, no unit above 26 % of its rate.

constexpr int kGsRows = 128;       // rows concatenated at a time by the block (its threads, at most)
constexpr uint32_t kGsCand = 128;  // candidates for the top-gamma set
constexpr uint32_t kGsFilter = 256;  // words of the window filter (8,192 bits)

// A residual with the "discovered this round" mark in its sign bit.
__device__ __forceinline__ bool found(float x) { return __float_as_int(x) < 0; }
__device__ __forceinline__ bool found(double x) { return __double2hiint(x) < 0; }
__device__ __forceinline__ float magnitude(float x) { return fabsf(x); }
__device__ __forceinline__ double magnitude(double x) { return fabs(x); }
__device__ __forceinline__ float with_mark(float x) { return -x; }  // x >= +0
__device__ __forceinline__ double with_mark(double x) { return -x; }

// r / d, correctly rounded; inv = RN(1 / d) in FP64.
__device__ __forceinline__ float push_share(float r, uint32_t d, double) { return rdiv(r, from_u64<float>(d)); }
__device__ __forceinline__ double push_share(double r, uint32_t d, double inv) {
    return div_fixed(r, double(d), inv);
}

// A load whose value is not used: it brings the word's line to L1.  gone() marks the point where the
// loaded register may be reused.
__device__ __forceinline__ uint32_t touch(const void* p) {
    uint32_t v;
    asm volatile("ld.global.u32 %0, [%1];" : "=r"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ void gone(uint32_t v) { asm volatile("" ::"r"(v)); }

// Extremes of residuals as 64-bit keys (ord_bits).
__device__ __forceinline__ unsigned long long warp_max_u64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(kFullMask, x, o);
        x = x > y ? x : y;
    }
    return x;
}
__device__ __forceinline__ unsigned long long warp_min_u64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(kFullMask, x, o);
        x = x < y ? x : y;
    }
    return x;
}

struct GsScratch {
    ChunkScratchOf<kGsRows> chunk;
    unsigned long long gmax, gmin, smax, smin, best, nth, st[3], ph[8];
    unsigned long long set_k[kSetMax];
    uint32_t set_v[kSetMax];
    double rw[4];
    alignas(8) uint32_t filter[kGsFilter];
    // late: past the deadline at the claim, round_late: at a round's start.  Two words: a warp may read
    // the one after thread 0 has written the other, and every warp must leave the loops with the rest.
    uint32_t k, graph, late, round_late, picost, found, nitems, next_item, set_count, cand_count, bin, rest;
};
static_assert(sizeof(unsigned long long) * kGsRows == 4 * kGsFilter, "the chi step keeps its minima in the filter");
template <class Real>
inline size_t gs_shared_bytes(bool smem, uint64_t n) {
    return sizeof(GsScratch) + (smem ? (sizeof(Real) * n + 15) / 16 * 16 : 0);
}

// What the push reads of a graph.
struct GsGraph {
    const uint32_t* idx;
    const uint2* adjd;    // (neighbour, neighbour's degree) per slot
    const double* dinv;
};

// ---- diffuse (src/aesc.h:218-239), windowed, by one warp ----
// The reference drains the frontier one vertex at a time: r = pvec[v], pvec[v] = 0, then pvec[u] +=
// r / deg(u) for u in N(v) in row order, discovering each u on its first visit.  Here up to 32
// consecutive frontier vertices form a window whose residuals are taken at once and whose rows are
// concatenated and processed 32 entries per step, in order.  That gives the reference's values as
// long as no entry of a window vertex j targets a later window vertex k (it would have changed r_k
// before k was drained): such an entry cuts the window before k -- found before anything of its step
// is applied, the cut vertices get their residuals back and are drained by a later window.  Entries
// targeting the vertex itself or an earlier window vertex are ordinary adds (those were drained first
// in the reference too).  Lanes of one step that hit the same neighbour form a group whose lowest
// lane adds the group's contributions one by one in lane (= the reference's) order; the lowest lane
// is also the first visit, so discovery order is the reference's.  Returns the number of discovered
// vertices (in qn); their degree sum and the traversals are added to pcost and trav.
template <class Real, bool SMEM>
__device__ uint32_t push_window(const GsGraph& g, Real* pvec, const uint32_t* q, uint32_t qs, uint32_t* qn,
                                uint32_t* filter, uint32_t& pcost, unsigned long long& trav) {
    constexpr uint32_t NONE = 0xffffffffu;
    const uint32_t lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t qns = 0;
    uint32_t t_idx = 0, t_pv = 0;
    for (uint32_t i0 = 0; i0 < qs;) {
        const uint32_t cnt = min(32u, qs - i0);
        uint32_t myv = 0, vb = 0, vd = 0;
        Real x = Real(0);
        if (lane < cnt) {
            myv = q[i0 + lane];
            vb = __ldg(g.idx + myv);
            vd = __ldg(g.idx + myv + 1) - vb;
            x = pvec[myv];
        }
        if (!SMEM) {  // the next window's row offsets and residuals
            gone(t_idx);
            gone(t_pv);
            if (i0 + 32u + lane < qs) {
                const uint32_t nv = q[i0 + 32u + lane];
                t_idx = touch(g.idx + nv);
                t_pv = touch(pvec + nv);
            }
        }
        const Real rv = magnitude(x);
        __syncwarp();
        if (lane < cnt) {
            pvec[myv] = found(x) ? with_mark(Real(0)) : Real(0);
            atomicOr(filter + ((myv >> 5) & (kGsFilter - 1u)), 1u << (myv & 31u));
        }
        uint32_t incl = vd;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        const uint32_t excl = incl - vd, base = vb - excl;
        __syncwarp();
        uint32_t wend = cnt;  // the window: frontier vertices i0 .. i0 + wend - 1
        struct Step {
            uint32_t sg, u, du;
        };
        auto load = [&](uint32_t at) {
            Step t{32u, NONE, 1u};
            if (at < total) {
                const unsigned upto = __ballot_sync(kFullMask, excl <= at);
                const uint32_t rel = excl - at;
                const unsigned mask = __reduce_or_sync(kFullMask, rel - 1u < 31u ? 1u << rel : 0u);
                const uint32_t k = uint32_t(__popc(upto)) - 1u + uint32_t(__popc(mask & ((2u << lane) - 1u)));
                const uint32_t slot = __shfl_sync(kFullMask, base, int(k & 31u)) + at + lane;
                if (at + lane < total) {
                    const uint2 a = __ldg(g.adjd + slot);
                    t.sg = k;
                    t.u = a.x;
                    t.du = a.y;
                }
            }
            return t;
        };
        auto inverse = [&](const Step& t) {
            return std::is_same<Real, double>::value && t.sg < 32u ? __ldg(g.dinv + t.u) : 1.0;
        };
        Step s0 = load(0u), s1 = load(32u);
        uint32_t t0 = 0;
        if (!SMEM && s0.sg < 32u) t0 = touch(pvec + s0.u);
        double inv0 = inverse(s0);
        for (uint32_t e0 = 0; e0 < total; e0 += 32) {
            gone(t0);
            if (!SMEM && s1.sg < 32u) t0 = touch(pvec + s1.u);
            const double inv1 = inverse(s1);
            const Step s2 = load(e0 + 64u);
            if (__all_sync(kFullMask, s0.sg >= wend)) break;  // past the (cut) window
            const uint32_t u = s0.u, sg = s0.sg;
            Real px = sg < wend ? pvec[u] : Real(0);
            const bool maybe = sg < wend && ((filter[(u >> 5) & (kGsFilter - 1u)] >> (u & 31u)) & 1u);
            unsigned mb = __ballot_sync(kFullMask, maybe);
            if (mb) {
                uint32_t kmin = 32u;
                while (mb) {  // is the target a later window vertex?
                    const int l = __ffs(int(mb)) - 1;
                    mb &= mb - 1;
                    const uint32_t uu = __shfl_sync(kFullMask, u, l), ss = __shfl_sync(kFullMask, sg, l);
                    const unsigned hit = __ballot_sync(kFullMask, lane < wend && myv == uu);
                    if (hit) {
                        const uint32_t k = uint32_t(__ffs(int(hit)) - 1);
                        if (k > ss) kmin = min(kmin, k);
                    }
                }
                if (kmin < wend) {  // window vertices kmin .. wend - 1 leave the window undrained
                    if (lane >= kmin && lane < wend) pvec[myv] = x;
                    wend = kmin;
                    __syncwarp();
                    px = sg < wend ? pvec[u] : Real(0);
                }
            }
            const bool apply = sg < wend;
            const unsigned grp = __match_any_sync(kFullMask, apply ? u : (0xffffffe0u | lane));
            const bool lead = apply && lane == uint32_t(__ffs(int(grp)) - 1);
            const Real r = __shfl_sync(kFullMask, rv, int(sg & 31u));
            const Real c = apply ? push_share(r, s0.du, inv0) : Real(0);
            const bool fresh = lead && !found(px);
            const unsigned bal = __ballot_sync(kFullMask, fresh);
            if (fresh) {
                qn[qns + __popc(bal & lt)] = u;
                pcost += s0.du;
            }
            qns += __popc(bal);
            const unsigned others = __ballot_sync(kFullMask, apply && !lead);
            Real pv = radd(magnitude(px), c);
            for (unsigned mm = others; mm; mm &= mm - 1) {
                const int t = __ffs(int(mm)) - 1;
                const Real ct = __shfl_sync(kFullMask, c, t);
                if ((grp >> t) & 1u) pv = radd(pv, ct);
            }
            if (lead) pvec[u] = with_mark(pv);
            __syncwarp();
            s0 = s1;
            s1 = s2;
            inv0 = inv1;
        }
        gone(t0);
        if (lane < cnt) filter[(myv >> 5) & (kGsFilter - 1u)] = 0u;
        trav += __shfl_sync(kFullMask, incl, int(wend - 1));
        __syncwarp();
        i0 += wend;
    }
    gone(t_idx);
    gone(t_pv);
    return qns;
}

// The same one frontier vertex at a time (rows without repeated neighbours): the entries of a row are
// distinct, so up to 128 of them are applied at once, 32 where no more are left (a step costs its
// instructions: FP64, n = 1,200, 20 neighbours, eps = 0.005, 1.31 -> 1.23 ms against four groups
// always); the next step's entries are loaded meanwhile.
template <class Real>
__device__ uint32_t push_single(const GsGraph& g, Real* pvec, const uint32_t* q, uint32_t qs, uint32_t* qn,
                                uint32_t& pcost, unsigned long long& trav) {
    constexpr int K = 4;
    const uint32_t lane = threadIdx.x & 31;
    const unsigned lt = (1u << lane) - 1u;
    uint32_t qns = 0;
    uint32_t v = 0;
    Real r = Real(0);
    // KK groups of 32 entries of v's row, of which `left` are left; the first ones drain v
    auto apply = [&](auto width, const uint2* in, uint32_t left, bool first) {
        constexpr int KK = decltype(width)::value;
        uint2 a[KK];
        double inv[KK];
        Real px[KK];
#pragma unroll
        for (int k = 0; k < KK; ++k) a[k] = in[k];
#pragma unroll
        for (int k = 0; k < KK; ++k)
            inv[k] = std::is_same<Real, double>::value && a[k].y ? __ldg(g.dinv + a[k].x) : 1.0;
        if (first) {
            const Real x = pvec[v];
            r = magnitude(x);
            __syncwarp();
            if (lane == 0) pvec[v] = found(x) ? with_mark(Real(0)) : Real(0);
        }
#pragma unroll
        for (int k = 0; k < KK; ++k) px[k] = a[k].y ? pvec[a[k].x] : Real(0);
#pragma unroll
        for (int k = 0; k < KK; ++k) {
            if (k && 32u * k >= left) break;
            const bool fresh = a[k].y && !found(px[k]);
            const unsigned bal = __ballot_sync(kFullMask, fresh);
            if (fresh) {
                qn[qns + __popc(bal & lt)] = a[k].x;
                pcost += a[k].y;
            }
            qns += __popc(bal);
            if (a[k].y) pvec[a[k].x] = with_mark(radd(magnitude(px[k]), push_share(r, a[k].y, inv[k])));
        }
        __syncwarp();
    };
    for (uint32_t i0 = 0; i0 < qs; i0 += 32) {
        const uint32_t cnt = min(32u, qs - i0);
        uint32_t myv = 0, vb = 0, vd = 0;
        if (lane < cnt) {
            myv = q[i0 + lane];
            vb = __ldg(g.idx + myv);
            vd = __ldg(g.idx + myv + 1) - vb;
        }
        trav += __reduce_add_sync(kFullMask, vd);
        uint2 nxt[K];
        uint32_t b = 0, d = 0;  // the loaded entries' row
        auto load = [&](uint32_t c0) {
            const uint32_t o = c0 + lane;
            nxt[0] = o < d ? __ldg(g.adjd + b + o) : make_uint2(0u, 0u);
            if (d - c0 > 32u) {
#pragma unroll
                for (int k = 1; k < K; ++k)
                    nxt[k] = o + 32u * k < d ? __ldg(g.adjd + b + o + 32u * k) : make_uint2(0u, 0u);
            }
        };
        b = __shfl_sync(kFullMask, vb, 0);
        d = __shfl_sync(kFullMask, vd, 0);
        load(0u);
        for (uint32_t t = 0; t < cnt; ++t) {
            v = __shfl_sync(kFullMask, myv, int(t));
            uint2 a[K];
            uint32_t c0 = 0, left = d;
            while (left > 32u * K) {
#pragma unroll
                for (int k = 0; k < K; ++k) a[k] = nxt[k];
                c0 += 32u * K;
                load(c0);
                apply(std::integral_constant<int, K>{}, a, 32u * K, c0 == 32u * K);
                left -= 32u * K;
            }
#pragma unroll
            for (int k = 0; k < K; ++k) a[k] = nxt[k];
            if (t + 1 < cnt) {
                b = __shfl_sync(kFullMask, vb, int(t + 1));
                d = __shfl_sync(kFullMask, vd, int(t + 1));
                load(0u);
            }
            if (left <= 32u) apply(std::integral_constant<int, 1>{}, a, left, c0 == 0);
            else apply(std::integral_constant<int, K>{}, a, left, c0 == 0);
        }
    }
    return qns;
}

// The rg-th largest of 32 K 64-bit keys, K per lane of one warp (0: none), counting repeats.
template <int K>
__device__ __forceinline__ unsigned long long warp_nth_largest_u64(unsigned long long (&x)[K], uint32_t rg) {
    unsigned long long top = 0;
    for (uint32_t left = rg;;) {
        unsigned long long mx = 0;
#pragma unroll
        for (int k = 0; k < K; ++k) mx = x[k] > mx ? x[k] : mx;
        top = warp_max_u64(mx);
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

// The rg-th largest key (counting repeats) of value(i), i < count, by digits of eight bits (see
// block_nth_largest); 0 when fewer than rg keys are positive (a vertex that is drained after its last
// visit of the round stays in the frontier with residual 0).
template <int BITS, class Value>
__device__ __forceinline__ unsigned long long gs_nth_largest(GsScratch& s, uint32_t count, uint32_t rg, Value value) {
    unsigned long long prefix = 0;
    uint32_t rest = rg;
    for (int shift = BITS - 8; shift >= 0; shift -= 8) {
        uint32_t* const hist = reinterpret_cast<uint32_t*>(s.chunk.val);
        static_assert(sizeof(s.chunk.val) >= 1024, "256 counters");
        for (uint32_t i = threadIdx.x; i < 256; i += blockDim.x) hist[i] = 0;
        __syncthreads();
        for (uint32_t i = threadIdx.x; i < count; i += blockDim.x) {
            const unsigned long long x = value(i);
            if (x != 0 && (shift == BITS - 8 || (x >> (shift + 8)) == prefix))
                atomicAdd(hist + (uint32_t(x >> shift) & 255u), 1u);
        }
        __syncthreads();
        if (threadIdx.x < 32) {  // the bin, from the top, where the running count reaches rest
            const uint32_t lane = threadIdx.x;
            uint32_t h[8], sum = 0;  // lane l holds bins 255 - 8 l .. 248 - 8 l
#pragma unroll
            for (int k = 0; k < 8; ++k) {
                h[k] = hist[255u - 8u * lane - uint32_t(k)];
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

// The gamma-th largest residual t of the frontier (rg <= kSetMax of qs > rg) and the set {r > t} in
// set_v / set_k, as block_top_set.
template <class Real>
__device__ __forceinline__ unsigned long long gs_top_set(GsScratch& s, const uint32_t* q, uint32_t qs, uint32_t rg,
                                                         const Real* pvec) {
    constexpr int U = 4;
    const uint32_t tid = threadIdx.x, lane = tid & 31, per_group = blockDim.x / 64u;
    auto value = [&](uint32_t i) { return ord_bits(pvec[q[i]]); };
    unsigned long long mx = 0;
    auto sweep = [&](auto use) {
        for (uint32_t i0 = tid; i0 < qs; i0 += U * blockDim.x) {
            uint32_t u[U];
            unsigned long long x[U];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                const uint32_t i = i0 + k * blockDim.x;
                u[k] = i < qs ? q[i] : 0xffffffffu;
            }
#pragma unroll
            for (int k = 0; k < U; ++k) x[k] = u[k] != 0xffffffffu ? ord_bits(pvec[u[k]]) : 0ull;
#pragma unroll
            for (int k = 0; k < U; ++k) use(u[k], x[k]);
        }
    };
    sweep([&](uint32_t, unsigned long long x) { mx = x > mx ? x : mx; });
    for (uint32_t o = per_group >> 1; o; o >>= 1) {
        const unsigned long long y = __shfl_xor_sync(kFullMask, mx, int(o));
        mx = mx > y ? mx : y;
    }
    if (tid % per_group == 0) s.chunk.val[tid / per_group] = mx;
    __syncthreads();
    unsigned long long g[2] = {s.chunk.val[lane], s.chunk.val[32 + lane]};
    unsigned long long low = warp_nth_largest_u64<2>(g, rg);  // the same in every warp
    if (low == 0) low = 1;
    __syncthreads();  // the maxima have been read: candidates take their place
    unsigned long long* const cand = s.chunk.val;
    uint32_t* const cand_v = s.chunk.base;
    static_assert(kGsCand <= kGsRows, "candidates share the chunk's arrays");
    sweep([&](uint32_t u, unsigned long long x) {
        if (x >= low) {
            const uint32_t at = atomicAdd(&s.cand_count, 1u);
            if (at < kGsCand) {
                cand[at] = x;
                cand_v[at] = u;
            }
        }
    });
    __syncthreads();
    const uint32_t c = s.cand_count;
    if (c > kGsCand) {
        const unsigned long long t = gs_nth_largest<8 * sizeof(Real)>(s, qs, rg, value);
        sweep([&](uint32_t u, unsigned long long x) {
            if (x > t) {
                const uint32_t at = atomicAdd(&s.set_count, 1u);
                s.set_k[at] = x;
                s.set_v[at] = u;
            }
        });
        __syncthreads();
        return t;
    }
    if (tid < 32) {
        unsigned long long x[kGsCand / 32];
#pragma unroll
        for (int k = 0; k < int(kGsCand / 32); ++k) x[k] = 32u * k + lane < c ? cand[32u * k + lane] : 0ull;
        const unsigned long long t = warp_nth_largest_u64<kGsCand / 32>(x, rg);
        for (uint32_t i = lane; i < c; i += 32)
            if (cand[i] > t) {
                const uint32_t at = atomicAdd(&s.set_count, 1u);
                s.set_k[at] = cand[i];
                s.set_v[at] = cand_v[i];
            }
        if (lane == 0) s.nth = t;
    }
    __syncthreads();
    return s.nth;
}

template <class Real>
struct SourceParams {
    const uint32_t* idx;
    const uint32_t* adj;
    const uint2* adjd;     // (neighbour, neighbour degree) per slot
    const double* dinv;    // 1 / degree
    uint32_t n;
    const int* taus;
    Real* preds;           // pre-symmetric row scores
    unsigned* work;        // [1] error flags, [2] list length
    const uint32_t* rows;  // the sources to run (rows with a slot of tau > 1), in any order
    double eps;
    double logmd;          // log(m / delta), formed on the host
    int gamma;
    unsigned long long* stats;
    uint64_t budget_ns;    // device time budget; past it every block stops and flags a timeout
    unsigned* claim;       // the claim counter of this launch
    // Optional run trace (null when off): the walk count nr of every walking slot, and the rounds
    // pushed (ell) of every listed row.
    uint32_t* trace_nr;
    uint32_t* trace_ell;
    // The graph has rows that repeat a neighbour or hold their own vertex (the reference's loader
    // keeps duplicate edges and self-loops, src/graph.h:63-66, 75-78): the first round takes the
    // general path and the push is the windowed one.
    bool multi;
    bool gs_window;        // the windowed push (else one vertex at a time)
    // per-block scratch, laid out for scratch_n vertices (the graph's n, or the largest n of a
    // batch whose graphs share one persistent launch) and max_degree slots
    uint32_t scratch_n, max_degree;
    uint32_t* qbuf;        // 2 * scratch_n
    WalkItem* items;       // max_degree
    Real* pvec_g;          // scratch_n (HBM tier), all +0 between sources
    unsigned char* clean;  // HBM tier, per block: 1 = its vector is all zero (left so by its last run)
};

// The source kernel's parameters: one graph (N = 1), or up to N graphs whose listed rows one
// persistent launch works through as a single queue of (graph, row) items.  Every entry shares the
// first entry's per-block scratch and claim counter.  The pack travels in the kernel's parameter
// space, so a block reads its graph's fields from the constant bank with a uniform index.
template <class Real, int N>
struct SourcePack {
    static constexpr int kMax = N;
    uint32_t count;
    SourceParams<Real> g[N];
};
constexpr int kBatchPack = 64;  // graphs per persistent batch launch

// Threads per block and the blocks per SM its registers are limited for: in shared memory four warps
// share the stages after the push (two where many small vectors fit, see gs_layout); in HBM, where
// the push is nearly all of the time, two, and as many blocks as the vectors' way through L1 and L2
// stands (FP64, n = 10,000, 10 neighbours: 6, 8, 10, 12, 16 blocks 19.6, 17.3, 16.6, 18.3, 18.6 ms; n = 25,860:
// 179, 156, 145, 147, 150; FP32 there, 8 .. 20 blocks: 127, 118 (10), 117 (12), 114 (16), 118 (20)).
template <class Real, bool SMEM>
struct GsShape {
    static constexpr int kThreads = SMEM ? 128 : 64;
    static constexpr int kBlocks = SMEM ? (sizeof(Real) == 8 ? 6 : 8) : (sizeof(Real) == 8 ? 10 : 16);
};

template <class Real, bool SMEM, class Pack>
__global__ void __launch_bounds__(GsShape<Real, SMEM>::kThreads, GsShape<Real, SMEM>::kBlocks)
source_kernel(const Pack pk) {
    extern __shared__ __align__(16) unsigned char gs_smem[];
    __shared__ uint32_t s_pre[Pack::kMax + 1];  // item prefix over the pack's row lists
    GsScratch& s = *reinterpret_cast<GsScratch*>(gs_smem);
    const SourceParams<Real>& p0 = pk.g[0];
    const uint32_t tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const uint32_t sn = p0.scratch_n;
    Real* const pvec = SMEM ? reinterpret_cast<Real*>(gs_smem + sizeof(GsScratch)) : p0.pvec_g + size_t(blockIdx.x) * sn;
    uint32_t* const qa = p0.qbuf + size_t(blockIdx.x) * 2 * sn;
    WalkItem* const items = p0.items + size_t(blockIdx.x) * p0.max_degree;
    pdl_launch_dependents();
    pdl_wait();  // taus, row lists and their lengths from the tau kernels
    // items: the listed rows of the pack's graphs one after another
    if (tid < 32) {
        uint32_t carry = 0;
        for (uint32_t k0 = 0; k0 < pk.count; k0 += 32) {
            uint32_t incl = k0 + lane < pk.count ? pk.g[k0 + lane].work[2] : 0u;
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
    __syncthreads();
    // a block's first item is its index, further ones are claimed
    const uint32_t items_all = s_pre[pk.count];
    if (blockIdx.x >= items_all) return;
    for (uint32_t i = tid; i < kGsFilter; i += blockDim.x) s.filter[i] = 0u;
    if (SMEM || !p0.clean[blockIdx.x])
        for (uint32_t i = tid; i < sn; i += blockDim.x) pvec[i] = Real(0);
    const uint64_t deadline = globaltimer_ns() + p0.budget_ns;
    // run counters: the push's (rounds, vertices, traversals) and the phases' by thread 0 in shared
    // memory, the walks' per thread
    if (tid < 3) s.st[tid] = 0;
    if (tid < 8) s.ph[tid] = 0;
    unsigned long long st_we = 0, st_wc = 0, st_wh = 0, st_fb = 0;
    // SM cycles per phase as thread 0 sees them, counted once per warp of the block
    long long tmark = clock64();
    auto lap = [&](int i) {
        if (tid == 0) {
            const long long now = clock64();
            s.ph[i] += (unsigned long long)(now - tmark) * nw;
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
            stat_add(stats, kStPushRounds, s.st[0]);
            stat_add(stats, kStPushVertices, s.st[1]);
            stat_add(stats, kStPushTraversals, s.st[2]);
            for (int i = 0; i < 8; ++i) stat_add(stats, kStPhase0 + i, s.ph[i]);
            for (int i = 0; i < 3; ++i) s.st[i] = 0;
            for (int i = 0; i < 8; ++i) s.ph[i] = 0;
        }
        st_we = st_wc = st_wh = st_fb = 0;
    };
    // extremes of the block's keys into two words of the scratch (reset by the caller)
    auto add_extremes = [&](unsigned long long mx, unsigned long long mn, unsigned long long* to_max,
                            unsigned long long* to_min) {
        mx = warp_max_u64(mx);
        mn = warp_min_u64(mn);
        if (lane == 0) {
            atomicMax(to_max, mx);
            atomicMin(to_min, mn);
        }
    };
    uint32_t last_gi = 0xffffffffu;
    bool dirty = false;
    for (bool first = true;; first = false) {
        __syncthreads();  // the previous source is done with the scratch
        if (tid == 0) {
            const uint32_t k = first ? blockIdx.x : gridDim.x + atomicAdd(p0.claim, 1u);
            uint32_t gi = 0;  // the item's graph: the last list whose prefix is at most k
            for (uint32_t h = pk.count; h - gi > 1;) {
                const uint32_t mid = (gi + h) >> 1;
                if (s_pre[mid] <= k) gi = mid;
                else h = mid;
            }
            s.k = k;
            s.graph = gi;
            s.late = globaltimer_ns() > deadline;
            s.picost = s.nitems = s.next_item = s.set_count = s.cand_count = 0;
            s.gmax = s.smax = s.best = 0;
            s.gmin = ord_bits(Real(1));
            s.smin = ord_bits(Real(FLT_MAX));
        }
        __syncthreads();
        const uint32_t item = s.k, gi = s.graph;
        if (item >= items_all) break;
        const SourceParams<Real>& p = pk.g[gi];
        if (gi != last_gi) {
            if (last_gi != 0xffffffffu) flush_stats(pk.g[last_gi].stats);
            last_gi = gi;
        }
        if (s.late) {
            if (tid == 0) atomicOr(p.work + 1, kErrDeadline);
            break;
        }
        const uint32_t n = p.n;
        const uint32_t* __restrict__ idx = p.idx;
        const uint32_t* __restrict__ adj = p.adj;
        const GsGraph graph{p.idx, p.adjd, p.dinv};
        const uint32_t src = __ldg(p.rows + (item - s_pre[gi]));
        const uint32_t rb = __ldg(idx + src), dsi = __ldg(idx + src + 1) - rb;
        const Real ds = from_u64<Real>(dsi);
        // preds = 1.0 / ds (:468-470); stored together with the first round's update below
        const Real pinit = from_f64<Real>(__ddiv_rn(1.0, double(ds)));
        uint32_t* q = qa;
        uint32_t* qn = qa + sn;
        uint32_t qs = 0;
        lap(0);
        // ---- round 1 (:457-503, first pass of the loop) ----
        // The frontier is {src} with residual 1 (pvec[src] = 1.0, then zeroed as it is drained):
        // every neighbour u is discovered in row order and receives 0 + 1/deg(u) = 1/deg(u), so
        // the round's new frontier, residuals, degree sum, max / min and row update
        // preds = 1/ds + (0 - 1/deg(u)) / ds follow from one pass over the row when the
        // neighbours are distinct.
        if (p.multi) {
            // each run of one neighbour u (rows are sorted, so repeats are adjacent) is handled by
            // its first slot: k repeats add 1/deg(u) k times in order, as the reference's sequential
            // += does; that slot discovers u (first-occurrence order) and adds deg(u) to picost.
            // pvec[src] starts at 0 (it was drained), so a self-loop run adds to it like to any
            // neighbour.
            if (warp == 0) {
                uint32_t count = 0, pc = 0;
                unsigned long long mx = 0, mn = ord_bits(Real(1));
                for (uint32_t c = 0; c < dsi; c += 32) {
                    const uint32_t o = c + lane;
                    const bool in = o < dsi;
                    const uint2 a = in ? __ldg(p.adjd + rb + o) : make_uint2(0u, 1u);
                    const bool lead = in && (o == 0 || __ldg(adj + rb + o - 1) != a.x);
                    if (lead) {
                        const Real x = rdiv(Real(1), from_u64<Real>(a.y));
                        Real pu = radd(Real(0), x);
                        for (uint32_t k = o + 1; k < dsi && __ldg(adj + rb + k) == a.x; ++k) pu = radd(pu, x);
                        pvec[a.x] = pu;
                        pc += a.y;
                        mx = max(mx, ord_bits(pu));
                        mn = min(mn, ord_bits(pu));
                    }
                    const unsigned bl = __ballot_sync(kFullMask, lead);
                    if (lead) q[count + __popc(bl & ((1u << lane) - 1u))] = a.x;
                    count += __popc(bl);
                }
                pc = __reduce_add_sync(kFullMask, pc);
                if (lane == 0) {
                    s.picost = pc;
                    s.found = count;
                }
                add_extremes(mx, mn, &s.gmax, &s.gmin);
            }
            __syncthreads();
            qs = s.found;
            // preds[s -> t] = 1/ds + (pvec[s] - pvec[t]) / ds with the round's residuals
            const Real ps = pvec[src];
            for (uint32_t o = tid; o < dsi; o += blockDim.x)
                p.preds[rb + o] = row_update<Real, Real>(pinit, ps, pvec[__ldg(adj + rb + o)], ds);
        } else {
            uint32_t pc = 0;
            unsigned long long mx = 0, mn = ord_bits(Real(1));
            for (uint32_t o = tid; o < dsi; o += blockDim.x) {
                const uint2 a = __ldg(p.adjd + rb + o);
                const Real pu = rdiv(Real(1), from_u64<Real>(a.y));
                pvec[a.x] = pu;
                q[o] = a.x;
                pc += a.y;
                mx = max(mx, ord_bits(pu));
                mn = min(mn, ord_bits(pu));
                p.preds[rb + o] = row_update<Real, Real>(pinit, Real(0), pu, ds);
            }
            pc = __reduce_add_sync(kFullMask, pc);
            if (lane == 0 && pc) atomicAdd(&s.picost, pc);
            add_extremes(mx, mn, &s.gmax, &s.gmin);
            qs = dsi;
        }
        if (tid == 0) {
            s.st[1] += 1;
            s.st[2] += dsi;
        }
        int ell = 1;
        Real gmax, gmin;
        bool timed_out = false;
        lap(1);
        while (true) {
            // ---- the push/walk cost test (:483-502) ----
            // The walk counts are whole numbers, so their sum does not depend on the order while it
            // is below 2^53; beyond that it exceeds any push cost either way.
            if (tid == 0) s.round_late = globaltimer_ns() > deadline;
            __syncthreads();
            gmax = from_ord<Real>(s.gmax);
            gmin = qs < n ? Real(0) : from_ord<Real>(s.gmin);
            const double picost = double(s.picost);
            const double dse0 = __dmul_rn(double(ds), p.eps);
            const double dse2 = __dmul_rn(dse0, dse0);
            double rw = 0;
            for (uint32_t o = tid; o < dsi; o += blockDim.x) {
                const int rest = __ldg(p.taus + rb + o) - ell;
                if (rest > 0) {
                    const double chi = __dmul_rn(__dmul_rn(2.0, double(rest)), __dsub_rn(double(gmax), double(gmin)));
                    const double num = __dmul_rn(__dmul_rn(8.0, __dmul_rn(chi, chi)), p.logmd);
                    rw += std_max(ceil(__ddiv_rn(num, dse2)), 1.0);
                }
            }
#pragma unroll
            for (int o = 16; o; o >>= 1) rw += __shfl_xor_sync(kFullMask, rw, o);
            if (lane == 0) s.rw[warp] = rw;
            __syncthreads();
            rw = 0;
            for (uint32_t w = 0; w < nw; ++w) rw += s.rw[w];
            const bool stop = picost >= __dmul_rn(25.0, rw);
            timed_out = s.round_late != 0 && !stop;
            lap(3);
            if (stop || timed_out) break;
            if (warp == 0) {
                uint32_t pc = 0;
                unsigned long long trav = 0;
                const uint32_t qns = p.gs_window || p.multi
                                         ? push_window<Real, SMEM>(graph, pvec, q, qs, qn, s.filter, pc, trav)
                                         : push_single<Real>(graph, pvec, q, qs, qn, pc, trav);
                pc = __reduce_add_sync(kFullMask, pc);
                if (lane == 0) {
                    s.st[1] += qs;
                    s.st[2] += trav;
                    s.picost = pc;
                    s.found = qns;
                    s.gmax = 0;
                    s.gmin = ord_bits(Real(1));
                }
            }
            __syncthreads();
            lap(1);
            { uint32_t* t = q; q = qn; qn = t; }
            qs = s.found;
            // the new frontier's marks are cleared and its residual max / min taken (:484-491)
            {
                constexpr int U = 4;
                unsigned long long mx = 0, mn = ord_bits(Real(1));
                for (uint32_t i0 = tid; i0 < qs; i0 += U * blockDim.x) {
                    uint32_t u[U];
                    Real x[U];
#pragma unroll
                    for (int k = 0; k < U; ++k) {
                        const uint32_t i = i0 + k * blockDim.x;
                        u[k] = i < qs ? q[i] : 0xffffffffu;
                    }
#pragma unroll
                    for (int k = 0; k < U; ++k) x[k] = u[k] != 0xffffffffu ? pvec[u[k]] : Real(0);
#pragma unroll
                    for (int k = 0; k < U; ++k)
                        if (u[k] != 0xffffffffu) {
                            const Real y = magnitude(x[k]);
                            pvec[u[k]] = y;
                            mx = max(mx, ord_bits(y));
                            mn = min(mn, ord_bits(y));
                        }
                }
                add_extremes(mx, mn, &s.gmax, &s.gmin);
            }
            __syncthreads();
            // preds[row] += (pvec[src] - pvec[adj]) / ds (:235-237)
            {
                const Real ps = pvec[src];
                for (uint32_t o = tid; o < dsi; o += blockDim.x) {
                    const uint32_t w = __ldg(adj + rb + o);
                    p.preds[rb + o] = row_update<Real, Real>(p.preds[rb + o], ps, pvec[w], ds);
                }
            }
            ++ell;
            lap(2);
        }
        if (timed_out) {
            if (tid == 0) atomicOr(p.work + 1, kErrDeadline);
            dirty = true;
            break;
        }
        if (tid == 0) s.st[0] += uint64_t(ell);
        if (p.trace_ell && tid == 0) p.trace_ell[src] = uint32_t(ell);

        // ---- slots that still need walks (rest = tau - ell > 0), with the row's extremes ----
        {
            unsigned long long mx = 0, mn = ord_bits(Real(FLT_MAX));
            for (uint32_t o0 = tid - lane; o0 < dsi; o0 += blockDim.x) {
                const uint32_t o = o0 + lane;
                uint32_t v = 0;
                int rest = 0;
                if (o < dsi) {
                    v = __ldg(adj + rb + o);
                    rest = __ldg(p.taus + rb + o) - ell;
                    const unsigned long long x = ord_bits(pvec[v]);
                    mx = max(mx, x);
                    mn = min(mn, x);
                }
                const unsigned hb = __ballot_sync(kFullMask, rest > 0);
                if (hb) {
                    uint32_t at = 0;
                    if (lane == 0) at = atomicAdd(&s.nitems, uint32_t(__popc(hb)));
                    at = __shfl_sync(kFullMask, at, 0) + uint32_t(__popc(hb & ((1u << lane) - 1u)));
                    if (rest > 0) items[at] = WalkItem{rb + o, v, uint32_t(rest), 0u, 0ull};
                }
            }
            add_extremes(mx, mn, &s.smax, &s.smin);
        }
        __syncthreads();
        const uint32_t nitems = s.nitems;
        if (nitems) {
            // ---- edge bound (:414-442, :504-506) ----
            // edge_max starts at gmax + min(1, t), t the gamma-th largest residual, and is raised by
            // pairs of adjacent vertices of the top-gamma set: the residuals above t, then those
            // equal to t in frontier order until there are gamma.  While t is at most 1 a member
            // equal to t cannot raise it (residuals do not exceed gmax, rounding is monotone), so
            // those are left out.
            Real edge_max;
            if (p.gamma == 1) {
                edge_max = rmul(Real(2), gmax);
            } else {
                const uint32_t gamma = uint32_t(p.gamma);
                const bool all = gamma >= qs;  // every frontier vertex is in the set
                auto value = [&](uint32_t i) { return ord_bits(pvec[q[i]]); };
                unsigned long long t = 0;
                bool pairs = (all ? qs : gamma) <= kSetMax;
                if (!all && pairs) t = gs_top_set<Real>(s, q, qs, gamma, pvec);
                else if (!all) t = gs_nth_largest<8 * sizeof(Real)>(s, qs, gamma, value);
                const bool ties = !all && from_ord<Real>(t) > Real(1);
                edge_max = radd(gmax, all ? Real(0) : std_min(Real(1), from_ord<Real>(t)));
                unsigned long long best = 0;
                if (ties) pairs = false;
                if (pairs && all) {
                    for (uint32_t i = tid; i < qs; i += blockDim.x) {
                        s.set_k[i] = value(i);
                        s.set_v[i] = q[i];
                    }
                    if (tid == 0) s.set_count = qs;
                    __syncthreads();
                }
                if (pairs) {
                    const uint32_t c = s.set_count;
                    for (uint32_t x = tid; x < c * c; x += blockDim.x) {
                        const uint32_t i = x / c, j = x % c;
                        // a vertex is its own neighbour only in a graph with self-loops
                        if (p.multi ? i > j : i >= j) continue;
                        if (adjacent(idx, adj, s.set_v[i], s.set_v[j]))
                            best = max(best, ord_bits(radd(from_ord<Real>(s.set_k[i]), from_ord<Real>(s.set_k[j]))));
                    }
                } else {
                    // the members are marked in the vector, then their rows are searched for marks
                    __syncthreads();
                    for (uint32_t i = tid; i < qs; i += blockDim.x) {
                        const uint32_t u = q[i];
                        const Real x = pvec[u];
                        if (all || ord_bits(x) > t) pvec[u] = with_mark(x);
                    }
                    __syncthreads();
                    if (ties && warp == 0) {
                        uint32_t above = 0;
                        for (uint32_t i = lane; i < qs; i += 32) above += found(pvec[q[i]]);
                        uint32_t left = gamma - __reduce_add_sync(kFullMask, above);
                        for (uint32_t i0 = 0; i0 < qs && left; i0 += 32) {
                            const bool eq = i0 + lane < qs && ord_bits(pvec[q[i0 + lane]]) == t;
                            const unsigned be = __ballot_sync(kFullMask, eq);
                            if (eq && uint32_t(__popc(be & ((1u << lane) - 1u))) < left)
                                pvec[q[i0 + lane]] = with_mark(pvec[q[i0 + lane]]);
                            left -= min(left, uint32_t(__popc(be)));
                        }
                    }
                    __syncthreads();
                    for (uint32_t i0 = 0; i0 < qs; i0 += blockDim.x) {
                        const uint32_t i = i0 + tid;
                        const uint32_t u = i < qs ? q[i] : 0u;
                        const Real x = i < qs ? pvec[u] : Real(0);
                        const bool member = i < qs && found(x);
                        const uint32_t rank = block_exclusive_scan(member ? 1u : 0u, s.chunk.tmp, &s.chunk.total);
                        const uint32_t cnt = s.chunk.total;
                        __syncthreads();
                        if (cnt == 0) continue;
                        if (member) {
                            s.chunk.base[rank] = u;
                            s.chunk.val[rank] = ord_bits(magnitude(x));
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
                                const Real y = in ? pvec[w] : Real(0);
                                if (found(y)) best = max(best, ord_bits(radd(from_ord<Real>(m), magnitude(y))));
                            });
                        __syncthreads();
                    }
                    for (uint32_t i = tid; i < qs; i += blockDim.x) pvec[q[i]] = magnitude(pvec[q[i]]);
                }
                best = warp_max_u64(best);
                if (lane == 0 && best) atomicMax(&s.best, best);
                __syncthreads();
                edge_max = std_max(edge_max, from_ord<Real>(s.best));
            }
            lap(4);

            // ---- chi and walk counts per edge (:392-412, :508-521) ----
            const Real smax = from_ord<Real>(s.smax), smin = from_ord<Real>(s.smin);
            const Real dse = from_f64<Real>(__dmul_rn(double(ds), p.eps));
            const double den = double(rmul(dse, dse));
            for (uint32_t i0 = 0; i0 < nitems; i0 += blockDim.x) {
                const uint32_t cnt = min(blockDim.x, nitems - i0);
                uint32_t beg = 0, deg = 0;
                if (tid < cnt) {
                    const uint32_t v = items[i0 + tid].v;
                    beg = __ldg(idx + v);
                    deg = __ldg(idx + v + 1) - beg;
                }
                __syncthreads();  // the previous chunk's scratch is no longer read
                // the targets' neighbourhoods: largest residual in the chunk's values, smallest in
                // the push's filter (not in use here); a step's entries of one target are reduced
                // across their lanes first
                unsigned long long* const tmaxs = s.chunk.val;
                unsigned long long* const tmins = reinterpret_cast<unsigned long long*>(s.filter);
                tmins[tid] = ord_bits(Real(FLT_MAX));
                for_entries(
                    s.chunk, cnt, beg, deg, 0ull,
                    [&](uint32_t slot, bool in) { return in ? __ldg(adj + slot) : 0u; },
                    [&](uint32_t w, unsigned long long, uint32_t k, bool in) {
                        const unsigned long long x = in ? ord_bits(pvec[w]) : 0ull;
                        unsigned long long mx = x, mn = in ? x : ~0ull;
                        const uint32_t seg = in ? k : 0xffffffffu;
#pragma unroll
                        for (int o = 1; o < 32; o <<= 1) {
                            const unsigned long long ymx = __shfl_down_sync(kFullMask, mx, o);
                            const unsigned long long ymn = __shfl_down_sync(kFullMask, mn, o);
                            const uint32_t ys = __shfl_down_sync(kFullMask, seg, o);
                            if (lane + o < 32 && ys == seg) {
                                mx = max(mx, ymx);
                                mn = min(mn, ymn);
                            }
                        }
                        const uint32_t before = __shfl_up_sync(kFullMask, seg, 1);
                        if (in && (lane == 0 || before != seg)) {
                            atomicMax(tmaxs + k, mx);
                            atomicMin(tmins + k, mn);
                        }
                    });
                __syncthreads();
                const Real tmax = from_ord<Real>(tmaxs[min(tid, cnt - 1u)]);
                const Real tmin = from_ord<Real>(tmins[min(tid, cnt - 1u)]);
                if (tid < cnt) {
                    const WalkItem it = items[i0 + tid];
                    // get_chi (:410): float terms rounded as in the reference, summed in double
                    const int Li = int(it.len);
                    const double A = __dadd_rn(double(gmax), __ddiv_rn(double(radd(smax, tmax)), 2.0));
                    const double B = __dadd_rn(A, double(rmul(Real(Li - 1), edge_max)));
                    const double C = __dsub_rn(__dsub_rn(B, double(smin)), double(tmin));
                    const double E = __dsub_rn(C, double(rmul(Real(2 * (Li - 1)), gmin)));
                    const Real chi = from_f64<Real>(E);
                    // nr (:519-521)
                    const Real c8 = rmul(Real(8), rmul(chi, chi));
                    const double num = __dmul_rn(double(c8), p.logmd);
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
                }
            }
            __syncthreads();
            lap(5);

            // ---- 2-way bouquet walks (:241-391): an 8-lane group per item ----
            // Each hop's residual difference is added to x one hop later (after the next hop's row
            // offsets are requested), so the residual loads overlap the next hop instead of stalling
            // it; the adds stay in hop order, and the last one is made before the item's lanes are
            // summed.
            const uint32_t j = lane & 7, grp = lane >> 3;
            bool has = false, start = false, primary = true, done = false;
            WalkItem it{};
            unsigned long long bi = 0;
            uint32_t len = 0, step = 0, cur = 0, cur2 = 0, sec = 0, sec2 = 0, state = 0;
            Real x = Real(0), pa = Real(0), pb = Real(0);
            bool pend = false;
            while (true) {
                if (!has && !done) {
                    uint32_t my = 0;
                    if (j == 0) my = atomicAdd(&s.next_item, 1u);
                    my = __shfl_sync(0xffu << (grp * 8), my, int(grp * 8));
                    if (my >= nitems) {
                        done = true;
                    } else {
                        it = items[my];
                        if (it.nr) {
                            has = true;
                            start = true;
                            bi = 0;
                            x = Real(0);
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
                    if (pend) x = radd(x, rsub(pa, pb));
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
                    pa = pvec[cur];
                    pb = pvec[cur2];
                    pend = true;
                    if (++len == it.len) {
                        bi += 8;
                        start = true;
                        item_done = bi >= it.nr;
                    }
                }
                if (__any_sync(kFullMask, item_done)) {
                    if (item_done && pend) {
                        x = radd(x, rsub(pa, pb));
                        pend = false;
                    }
                    // the eight lanes summed 0..7, then preds += xij / (ds * nr) (:386-390, :525)
                    Real sum = Real(0);
#pragma unroll
                    for (int b = 0; b < 8; ++b) sum = radd(sum, __shfl_sync(kFullMask, x, int(grp * 8 + b)));
                    if (item_done && j == 0)
                        p.preds[it.pos] = radd(p.preds[it.pos], rdiv(sum, rmul(ds, from_u64<Real>(it.nr))));
                    if (item_done) has = false;
                }
            }
            __syncthreads();
            lap(6);
        }
        // ---- the next source starts from an all-zero residual vector (and filter) ----
        if (nitems)
            for (uint32_t i = tid; i < kGsFilter; i += blockDim.x) s.filter[i] = 0u;
        for (uint32_t i = tid; i < qs; i += blockDim.x) pvec[q[i]] = Real(0);
        if (tid == 0) pvec[src] = Real(0);
        lap(7);
    }
    if (!SMEM && tid == 0) p0.clean[blockIdx.x] = dirty ? 0 : 1;
    flush_stats(pk.g[last_gi == 0xffffffffu ? 0u : last_gi].stats);
}
