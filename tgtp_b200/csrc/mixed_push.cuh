// Push of the mixed form by a whole block per source (included by aesc.cu, inside its namespace).
//
// A round of the mixed form takes the frontier's residuals together: a vertex u receives the exact
// integer sum of its frontier neighbours' residuals in 2^-62 fixed point, divided (rounding down) by
// deg(u) and rounded once to FP32 (from_fixed).  The sum does not depend on the order of the
// additions, so the threads of a block share one source and add with shared-memory atomics: a
// 64-bit sum as two 32-bit words, the low word's old value giving the carry.  Measured on random
// vertices, that is 1.5e12 additions a second over the chip, against 5e11 for the 64-bit shared
// atomic and 1.9e11 for 64-bit atomics in L2.
//
// A frontier is a list of (row start, degree, residual, vertex) in global memory.  Light vertices are
// taken 32 at a time by each warp, which concatenates their rows in registers and needs no barrier;
// vertices of more than kHeavyRow entries (at the list's other end) are shared by the whole block:
// their adjacency is concatenated (block-wide prefix sum) and each warp takes a contiguous run of
// it.  The push of the sparse Chung-Lu graph (n = 25,860, eps = 0.005, 2.0e9 frontier vertices of 10.7
// entries on average) took 120 ms with every vertex going through the block-wide concatenation, 79 ms
// now: 55 in the additions, 20 in take_residuals.

constexpr uint32_t kHeavyRow = 256;
constexpr uint32_t kChunk = 512;  // frontier vertices whose adjacency is concatenated at a time

// Shared scratch of the concatenation of up to C rows: entry offsets (C + 1, and 33 words read but
// not used past them), row start minus offset, the vertex's value.
template <int C>
struct ChunkScratchOf {
    static constexpr uint32_t kRows = C;
    uint32_t offs[C + 34];
    uint32_t base[C];
    unsigned long long val[C];
    uint32_t tmp[32];
    uint32_t total;
};
using ChunkScratch = ChunkScratchOf<kChunk>;

// The segment of entry e among cnt segments starting at offs[0 .. cnt) (offs[cnt] = total > e):
// the last one that starts at or before e.  All lanes of a warp call it with the same e.
template <int C>
__device__ __forceinline__ uint32_t find_segment(const uint32_t* offs, uint32_t cnt, uint32_t e) {
    const uint32_t lane = threadIdx.x & 31;
    constexpr uint32_t R = C / 32;
    static_assert(R >= 1 && R <= 32 && R * 32 == C, "a step over 32 runs of R, a step inside one");
    const uint32_t c0 = lane * R;
    const unsigned b0 = __ballot_sync(kFullMask, c0 < cnt && offs[c0] <= e);
    const uint32_t coarse = (uint32_t(__popc(b0)) - 1u) * R;
    const uint32_t c1 = coarse + (lane & (R - 1u));
    const unsigned b1 = __ballot_sync(kFullMask, lane < R && c1 < cnt && offs[c1] <= e);
    return coarse + uint32_t(__popc(b1)) - 1u;
}

// Concatenates the rows of up to C vertices: thread i < cnt passes vertex i's row start, its
// degree (at least 1) and a value.  Every entry is loaded, load(slot, whether there is an entry), and
// then used, use(loaded, value of its vertex, the vertex's index in the chunk, whether there is an
// entry), by all lanes of a warp together, on consecutive entries.  All threads of the block call it;
// the scratch is free again after the caller's next __syncthreads.
template <int C, class Load, class Use>
__device__ __forceinline__ uint32_t for_entries(ChunkScratchOf<C>& s, uint32_t cnt, uint32_t beg, uint32_t deg,
                                                unsigned long long val, Load load, Use use) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const uint32_t off = block_exclusive_scan(deg, s.tmp, &s.total);
    if (threadIdx.x < cnt) {
        s.offs[threadIdx.x] = off;
        s.base[threadIdx.x] = beg - off;
        s.val[threadIdx.x] = val;
    }
    if (threadIdx.x == 0) s.offs[cnt] = s.total;
    __syncthreads();
    const uint32_t total = s.total;
    const uint32_t per = ((total + nw - 1) / nw + 31u) & ~31u;
    const uint32_t e0 = warp * per, end = min(total, e0 + per);
    if (e0 < end) {
        uint32_t seg = find_segment<C>(s.offs, cnt, e0);
        uint32_t e = e0;
        // lane's segment in the step of entries e .. e + 31, and the step's next first segment
        auto step = [&](uint32_t at, uint32_t& first) {
            const uint32_t rel = s.offs[min(first + 1u + lane, cnt)] - at;
            const unsigned mask = __reduce_or_sync(kFullMask, rel < 32u ? 1u << rel : 0u);
            const uint32_t k = first + uint32_t(__popc(mask & ((2u << lane) - 1u)));
            first += uint32_t(__popc(mask));
            if (s.offs[first + 1u] == at + 32u) ++first;
            return k;
        };
        uint32_t k = step(e, seg);
        bool in = e + lane < end;
        uint32_t slot = in ? s.base[k] + e + lane : 0u;
        uint32_t x = load(slot, in);
        while (true) {
            const uint32_t en = e + 32u;
            uint32_t kn = 0, slotn = 0;
            bool inn = false;
            uint32_t xn = 0;
            const bool more = en < end;
            if (more) {  // the next step's load is in flight while this one is used
                kn = step(en, seg);
                inn = en + lane < end;
                slotn = inn ? s.base[kn] + en + lane : 0u;
                xn = load(slotn, inn);
            }
            use(x, in ? s.val[k] : 0ull, k, in);
            if (!more) break;
            e = en;
            k = kn;
            in = inn;
            slot = slotn;
            x = xn;
        }
    }
    return total;
}

// Whether w is in u's row or u in w's (a hand-built CSR may hold an edge in one direction only); the
// shorter row is searched first.
__device__ __forceinline__ bool adjacent(const uint32_t* __restrict__ idx, const uint32_t* __restrict__ adj,
                                         uint32_t u, uint32_t w) {
    const uint32_t ub = __ldg(idx + u), ue = __ldg(idx + u + 1), wb = __ldg(idx + w), we = __ldg(idx + w + 1);
    for (int k = 0; k < 2; ++k) {
        const bool in_u = (ue - ub <= we - wb) == (k == 0);
        const uint32_t e = in_u ? ue : we, v = in_u ? w : u;
        const uint32_t at = lower_bound_u32(adj, in_u ? ub : wb, e, v);
        if (at < e && __ldg(adj + at) == v) return true;
    }
    return false;
}

// Adds a 64-bit value to the sum kept as lo[u], hi[u].
__device__ __forceinline__ void add_fixed(uint32_t* lo, uint32_t* hi, uint32_t u, unsigned long long v) {
    const uint32_t l = uint32_t(v);
    const uint32_t o = atomicAdd(lo + u, l);
    atomicAdd(hi + u, uint32_t(v >> 32) + uint32_t(o + l < l));
}

// A source's push state shared by the block.
struct PushScratch {
    ChunkScratch chunk;
    uint32_t picost, gmax, gmin, light, heavy, next, k, late;
    double rw[32];
};

// The push/walk cost test (src/aesc.h:483-502) of the current round: true when the source stops.
// The walk counts nr are whole numbers, so their sum does not depend on the order while it is
// below 2^53; beyond that it exceeds any push cost (at most the slot count) either way.
__device__ __forceinline__ bool block_stops(PushScratch& s, const int* __restrict__ taus, uint32_t rb,
                                            uint32_t dsi, int ell, float gmax, float gmin, double eps,
                                            double logmd) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const double dse0 = __dmul_rn(double(float(dsi)), eps);
    const double dse2 = __dmul_rn(dse0, dse0);
    double rw = 0;
    for (uint32_t o = threadIdx.x; o < dsi; o += blockDim.x) {
        const int rest = __ldg(taus + rb + o) - ell;
        if (rest > 0) {
            const double chi = __dmul_rn(__dmul_rn(2.0, double(rest)), __dsub_rn(double(gmax), double(gmin)));
            const double num = __dmul_rn(__dmul_rn(8.0, __dmul_rn(chi, chi)), logmd);
            rw += std_max(ceil(__ddiv_rn(num, dse2)), 1.0);
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) rw += __shfl_xor_sync(kFullMask, rw, o);
    if (lane == 0) s.rw[warp] = rw;
    __syncthreads();
    rw = lane < nw ? s.rw[lane] : 0.0;
#pragma unroll
    for (int o = 16; o; o >>= 1) rw += __shfl_xor_sync(kFullMask, rw, o);
    return double(s.picost) >= __dmul_rn(25.0, rw);
}

// The lists of one block: cap entries, light vertices from the front, heavy ones from the back.
struct Frontier {
    uint4* list;
    uint32_t cap;
};

// Appends the lanes' vertices with r > 0 (K of them per lane; REACHED: those with a number, also where
// r is 0) to the frontier and adds up what the cost test needs.  All lanes of a warp call it.
struct FrontierSums {
    uint32_t pc = 0, mx = 0, mn = 0x3f800000u;  // degree sum, bits of the largest and smallest residual
};
constexpr uint32_t kNoVertex = 0xffffffffu;
template <int K, bool REACHED = false>
__device__ __forceinline__ void append_frontier(PushScratch& s, const Frontier& f, FrontierSums& t,
                                                const uint32_t (&u)[K], const uint32_t (&beg)[K],
                                                const uint32_t (&deg)[K], const float (&r)[K]) {
    const uint32_t lane = threadIdx.x & 31;
    const unsigned below = (1u << lane) - 1u;
    unsigned bl[K], bh[K];
    uint32_t nl = 0, nh = 0;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        const bool live = REACHED ? u[k] != kNoVertex : r[k] > 0.f, big = live && deg[k] > kHeavyRow;
        bl[k] = __ballot_sync(kFullMask, live && !big);
        bh[k] = __ballot_sync(kFullMask, big);
        nl += __popc(bl[k]);
        nh += __popc(bh[k]);
    }
    if (!(nl | nh)) return;
    uint32_t at = 0, hat = 0;
    if (lane == 0) {
        if (nl) at = atomicAdd(&s.light, nl);
        if (nh) hat = atomicAdd(&s.heavy, nh);
    }
    at = __shfl_sync(kFullMask, at, 0);
    if (nh) hat = __shfl_sync(kFullMask, hat, 0);
#pragma unroll
    for (int k = 0; k < K; ++k) {
        if (REACHED ? u[k] != kNoVertex : r[k] > 0.f) {
            const bool big = (bh[k] >> lane) & 1u;
            f.list[big ? f.cap - 1u - (hat + uint32_t(__popc(bh[k] & below)))
                       : at + uint32_t(__popc(bl[k] & below))] =
                make_uint4(beg[k], deg[k], __float_as_uint(r[k]), u[k]);
            t.pc += deg[k];
            t.mx = max(t.mx, __float_as_uint(r[k]));
            t.mn = min(t.mn, __float_as_uint(r[k]));
        }
        at += uint32_t(__popc(bl[k]));
        hat += uint32_t(__popc(bh[k]));
    }
}
__device__ __forceinline__ void add_sums(PushScratch& s, const FrontierSums& t) {
    const uint32_t pc = __reduce_add_sync(kFullMask, t.pc);
    const uint32_t mx = __reduce_max_sync(kFullMask, t.mx);
    const uint32_t mn = __reduce_min_sync(kFullMask, t.mn);
    if ((threadIdx.x & 31) == 0) {
        if (pc) atomicAdd(&s.picost, pc);
        atomicMax(&s.gmax, mx);
        atomicMin(&s.gmin, mn);
    }
}
// One thread, before a barrier: nothing counted yet.
__device__ __forceinline__ void reset_sums(PushScratch& s) {
    s.picost = 0;
    s.gmax = 0;
    s.gmin = 0x3f800000u;
    s.light = s.heavy = s.next = 0;
}

// add(u, residual in fixed point) for every entry of the rows of the frontier's light and heavy
// vertices (nl and nh of them; s.next is 0).
template <class Add>
__device__ __forceinline__ void push_frontier(PushScratch& s, const Frontier& f, uint32_t nl, uint32_t nh,
                                              const uint32_t* __restrict__ adj, Add add) {
    const uint32_t lane = threadIdx.x & 31;
    const uint32_t per = min(kChunk, blockDim.x);
    for (uint32_t i0 = 0; i0 < nh; i0 += per) {
        const uint32_t cnt = min(per, nh - i0);
        uint4 q = make_uint4(0u, 0u, 0u, 0u);
        if (threadIdx.x < cnt) q = f.list[f.cap - 1u - (i0 + threadIdx.x)];
        if (i0) __syncthreads();  // the previous chunk's scratch is no longer read
        for_entries(
            s.chunk, cnt, q.x, q.y, to_fixed(__uint_as_float(q.z)),
            [&](uint32_t slot, bool in) { return in ? __ldg(adj + slot) : 0u; },
            [&](uint32_t u, unsigned long long v, uint32_t, bool in) {
                if (in) add(u, v);
            });
    }
    // light vertices: batches of 32 claimed by the warps, the next one loaded while one is pushed
    auto claim = [&]() {
        uint32_t i = 0;
        if (lane == 0) i = atomicAdd(&s.next, 32u);
        return __shfl_sync(kFullMask, i, 0);
    };
    auto fetch = [&](uint32_t i) {
        return i + lane < nl ? f.list[i + lane] : make_uint4(0u, 0u, 0u, 0u);
    };
    uint32_t i0 = claim();
    if (i0 >= nl) return;
    uint4 q = fetch(i0);
    while (true) {
        const uint32_t i1 = claim();
        uint4 qn = make_uint4(0u, 0u, 0u, 0u);
        if (i1 < nl) qn = fetch(i1);
        uint32_t incl = q.y;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
            if (lane >= uint32_t(o)) incl += y;
        }
        const uint32_t total = __shfl_sync(kFullMask, incl, 31);
        const uint32_t excl = incl - q.y, base = q.x - excl;
        const unsigned long long val = to_fixed(__uint_as_float(q.z));
        const uint32_t vl = uint32_t(val), vh = uint32_t(val >> 32);
        // lane's vertex in the step of entries at .. at + 31: the one that starts last at or before
        // its entry (empty lanes at the end start at total, past every entry)
        auto step = [&](uint32_t at) {
            const unsigned upto = __ballot_sync(kFullMask, excl <= at);
            const uint32_t rel = excl - at;
            const unsigned mask = __reduce_or_sync(kFullMask, rel - 1u < 31u ? 1u << rel : 0u);
            return uint32_t(__popc(upto)) - 1u + uint32_t(__popc(mask & ((2u << lane) - 1u)));
        };
        uint32_t k = step(0u);
        uint32_t slot = __shfl_sync(kFullMask, base, int(k & 31u)) + lane;
        uint32_t u = lane < total ? __ldg(adj + slot) : 0u;
        for (uint32_t e = 0; e < total; e += 32) {
            const unsigned long long v = (static_cast<unsigned long long>(__shfl_sync(kFullMask, vh, int(k & 31u))) << 32) |
                                         __shfl_sync(kFullMask, vl, int(k & 31u));
            const uint32_t cu = u;
            const uint32_t en = e + 32u;
            if (en < total) {  // the next step's entries are in flight while this one's are added
                k = step(en);
                slot = __shfl_sync(kFullMask, base, int(k & 31u)) + en + lane;
                u = en + lane < total ? __ldg(adj + slot) : 0u;
            }
            if (e + lane < total) add(cu, v);
        }
        if (i1 >= nl) break;
        i0 = i1;
        q = qn;
    }
}

// The new frontier of a round from the sums in lo / hi: every vertex with a nonzero residual goes
// to the frontier, its residual replaces the sum's low word (so lo is the residual vector until the
// next round) and the high word is cleared.
__device__ __forceinline__ void take_residuals(PushScratch& s, uint32_t* lo, uint32_t* hi,
                                               const uint32_t* __restrict__ idx,
                                               const double* __restrict__ dinv, uint32_t n,
                                               const Frontier& f) {
    constexpr int K = 4;  // vertices in flight per lane: the pass is a chain of loads otherwise
    const uint32_t lane = threadIdx.x & 31;
    FrontierSums t;
    for (uint32_t u0 = threadIdx.x - lane; u0 < n; u0 += K * blockDim.x) {
        uint32_t u[K], b[K], d[K], sl[K], sh[K];
        float r[K];
        double inv[K];
#pragma unroll
        for (int k = 0; k < K; ++k) {
            u[k] = u0 + k * blockDim.x + lane;
            sl[k] = sh[k] = b[k] = 0;
            d[k] = 1;
            inv[k] = 1.0;
            if (u[k] < n) {
                sl[k] = lo[u[k]];
                sh[k] = hi[u[k]];
                b[k] = __ldg(idx + u[k]);
                d[k] = __ldg(idx + u[k] + 1);
                inv[k] = __ldg(dinv + u[k]);
            }
        }
#pragma unroll
        for (int k = 0; k < K; ++k) {
            r[k] = 0.f;
            d[k] -= b[k];
            if (sl[k] | sh[k]) {
                r[k] = from_fixed(sh[k], sl[k], d[k], inv[k]);
                lo[u[k]] = __float_as_uint(r[k]);
                hi[u[k]] = 0u;
            }
        }
        append_frontier<K>(s, f, t, u, b, d, r);
    }
    add_sums(s, t);
}

struct PushSharedParams {
    const uint32_t* idx;
    const uint32_t* adj;
    const uint2* adjd;
    const double* dinv;    // 1 / degree
    uint32_t n;
    const int* taus;
    double* preds;
    unsigned* work;        // [1] error flags, [2] list length
    const uint32_t* rows;  // the list of sources
    uint32_t base, cap;    // this launch runs list entries [base, base + cap)
    unsigned* claim;
    double eps, logmd;
    uint4* lists;          // per block: the frontier, n entries
    float* cols;           // per entry of the launch: n floats, the final residual vector
    PrePush* pre;          // per list entry
    unsigned long long* stats;
    uint64_t budget_ns;
};

// Shared memory of the block push over n vertices: the scratch, then lo and hi.
inline size_t push_shared_bytes(uint64_t n) { return sizeof(PushScratch) + 8 * ((n + 3) & ~uint64_t(3)); }

// Round 1 in closed form: the frontier {src} pushes 1 / deg(u) to every neighbour u, which is the
// next frontier; put(u, residual) stores the residual.  preds = 1 / ds + (0 - 1 / deg(u)) / ds.
template <class Put>
__device__ __forceinline__ void first_round(PushScratch& s, const Frontier& f, const uint2* __restrict__ adjd,
                                            const uint32_t* __restrict__ idx, uint32_t rb, uint32_t dsi,
                                            double* preds, Put put) {
    const uint32_t lane = threadIdx.x & 31;
    const float ds = float(dsi);
    const double pinit = __ddiv_rn(1.0, double(ds));
    FrontierSums t;
    for (uint32_t o0 = threadIdx.x - lane; o0 < dsi; o0 += blockDim.x) {
        const uint32_t o = o0 + lane;
        float r[1] = {0.f};
        uint32_t u[1] = {0u}, b[1] = {0u}, d[1] = {1u};
        if (o < dsi) {
            const uint2 a = __ldg(adjd + rb + o);
            u[0] = a.x;
            b[0] = __ldg(idx + a.x);
            d[0] = a.y;
            r[0] = from_fixed(kFixOne, a.y);
            put(a.x, r[0]);
            preds[rb + o] = row_update<float, double>(pinit, 0.f, r[0], ds);
        }
        append_frontier<1>(s, f, t, u, b, d, r);
    }
    add_sums(s, t);
}

// Mixed form, graphs whose sums fit in shared memory: the push of one listed source at a time per
// block, which leaves the source's final residual vector in cols and its outcome in pre, as
// push_block_kernel does for larger graphs (the same values: the sums are exact).
__global__ void __launch_bounds__(1024, 1) push_shared_kernel(PushSharedParams p) {
    extern __shared__ __align__(16) unsigned char push_smem[];
    PushScratch& s = *reinterpret_cast<PushScratch*>(push_smem);
    const uint32_t n = p.n, pad = (n + 3u) & ~3u;
    uint32_t* const lo = reinterpret_cast<uint32_t*>(push_smem + sizeof(PushScratch));
    uint32_t* const hi = lo + pad;
    pdl_launch_dependents();
    for (uint32_t u = threadIdx.x; u < 2 * pad; u += blockDim.x) lo[u] = 0u;
    pdl_wait();  // the list, the taus, and the previous wave's readers of the columns
    const unsigned len = p.work[2];
    const uint32_t count = len > p.base ? min(len - p.base, p.cap) : 0u;
    const Frontier f{p.lists + size_t(blockIdx.x) * n, n};
    const uint64_t deadline = globaltimer_ns() + p.budget_ns;
    unsigned long long st_pv = 0, st_tr = 0, st_rounds = 0;
    while (true) {
        __syncthreads();
        if (threadIdx.x == 0) {
            s.k = atomicAdd(p.claim, 1u);
            reset_sums(s);
        }
        __syncthreads();
        const uint32_t k = s.k;
        if (k >= count) break;
        const uint32_t src = __ldg(p.rows + p.base + k);
        const uint32_t rb = __ldg(p.idx + src), dsi = __ldg(p.idx + src + 1) - rb;
        const float ds = float(dsi);
        first_round(s, f, p.adjd, p.idx, rb, dsi, p.preds,
                    [&](uint32_t u, float r) { lo[u] = __float_as_uint(r); });
        int ell = 1;
        if (threadIdx.x == 0) {
            st_pv += 1;
            st_tr += dsi;
        }
        while (true) {
            if (threadIdx.x == 0) s.late = globaltimer_ns() > deadline;
            __syncthreads();
            const uint32_t nl = s.light, nh = s.heavy, qs = nl + nh;
            const float gmax = __uint_as_float(s.gmax);
            const float gmin = qs < n ? 0.f : __uint_as_float(s.gmin);
            const bool stop = block_stops(s, p.taus, rb, dsi, ell, gmax, gmin, p.eps, p.logmd);
            const bool late = s.late != 0;
            if (threadIdx.x == 0) {
                if (stop || late) {
                    PrePush r;
                    r.ell = ell;
                    r.gmax = gmax;
                    r.gmin = __uint_as_float(s.gmin);
                    r.support = qs;
                    p.pre[p.base + k] = r;
                    st_rounds += uint64_t(ell);
                    if (late && !stop) atomicOr(p.work + 1, kErrDeadline);
                } else {
                    st_pv += qs;
                    st_tr += s.picost;
                }
            }
            if (stop || late) break;
            // the old residuals leave the vector before the round's sums start
            if (qs * 4u > n) {
                for (uint32_t u = threadIdx.x; u < n; u += blockDim.x) lo[u] = 0u;
            } else {
                for (uint32_t i = threadIdx.x; i < qs; i += blockDim.x)
                    lo[f.list[i < nl ? i : n - 1u - (i - nl)].w] = 0u;
            }
            __syncthreads();
            push_frontier(s, f, nl, nh, p.adj,
                          [&](uint32_t u, unsigned long long v) { add_fixed(lo, hi, u, v); });
            __syncthreads();
            if (threadIdx.x == 0) reset_sums(s);
            __syncthreads();
            take_residuals(s, lo, hi, p.idx, p.dinv, n, f);
            __syncthreads();
            // preds[row] += (r[src] - r[t]) / ds (src/aesc.h:235-237)
            const float ps = __uint_as_float(lo[src]);
            for (uint32_t o = threadIdx.x; o < dsi; o += blockDim.x) {
                const uint32_t w = __ldg(p.adj + rb + o);
                p.preds[rb + o] =
                    row_update<float, double>(p.preds[rb + o], ps, __uint_as_float(lo[w]), ds);
            }
            ++ell;
        }
        __syncthreads();
        float* const col = p.cols + size_t(k) * n;
        for (uint32_t u = threadIdx.x; u < n; u += blockDim.x) {
            col[u] = __uint_as_float(lo[u]);
            lo[u] = 0u;
        }
    }
    if (threadIdx.x == 0) {
        stat_add(p.stats, kStPushRounds, st_rounds);
        stat_add(p.stats, kStPushVertices, st_pv);
        stat_add(p.stats, kStPushTraversals, st_tr);
    }
}
