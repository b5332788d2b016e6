// tgtp() on sm_100a: the TGT+ approximate edge spanning centrality of src/aesc.h:113-551.
//
// Stages (all on the graph's stream, consecutive kernels joined by programmatic dependent launch):
//   1. tau per undirected edge (u <= v): the omega-eigenvector walk-length bound (calculate_taus,
//      :164-216), written to both CSR slots; rows with a slot of tau > 1 are listed.
//        FP32 form           tau_kernel: the reference's sequential sums, two lanes per edge.
//        FP64 / mixed forms  tau_sums_kernel (eight lanes per edge gather the rows) then
//                            tau_bound_kernel (lane per edge evaluates the bound).
//   2. the listed sources: push rounds until the push/walk cost test stops them (:456-503), the
//      top-gamma edge bound (:414-442), the per-edge chi and walk count (:392-412, :508-521) and
//      the 2-way bouquet walks (:241-391), accumulating each source's CSR row (:524-525).
//        source_kernel        FP32 / FP64 forms: one source at a time per block, pushed by one of
//                             its warps (gs_source.cuh);
//        mixed_source_kernel  mixed form: one source at a time per block (mixed_source.cuh);
//        push_shared_kernel, push_block_kernel  mixed form, deep pushes: the push alone, one source
//                             per block in shared memory, or 32 sources per CTA as a pull product;
//                             then mixed_source_kernel for the rest and the walk kernels.
//   3. finish_kernel: score[q] = row[q] + row[reverse slot] (:532-550), with the rows of unlisted
//      sources (every tau <= 1: one push round, no walks) in closed form.
//
// The parity forms (FP32 = the reference's own arithmetic, FP64 = every real held in double)
// keep the reference's evaluation order wherever a rounding depends on it:
//   * the push of one source is sequential over its frontier, in discovery order; the lanes of the
//     warp share one frontier vertex's adjacency (distinct neighbours update distinct words; a run
//     of one repeated neighbour is applied by its first lane, one add per repeat, in order);
//   * float sums run in the reference's order (walk lanes per bouquet lane in bouquet order, the
//     eight lanes summed 0..7; the FP32 form's tau dot products per edge in index order, the FP64
//     form's in its fixed eight-way split);
//   * every operation is a correctly rounded intrinsic, never contracted into an FMA except the
//     FP64 form's tau terms, which are defined as fused multiply-adds.
// Max/min/integer reductions are order-free and run across lanes.
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <string>
#include <memory>
#include <vector>
#include <type_traits>

#include <cub/device/device_radix_sort.cuh>

#include "common.cuh"
#include "internal.hpp"

namespace tgtp {
namespace {

constexpr int kTauThreads = 32;      // FP32 form's tau: one warp per block
constexpr int kTauBlocks = 20;       // per SM: 96 registers (16 blocks: 78 us for 70; 24 spill: 70)
constexpr int kTauTableRows = 64;    // rows of the eigen_t_1 power table (api.cu)
constexpr uint64_t kMaxWalks = 0xffffffffull;  // nr beyond the 32-bit grid is not supported

enum : unsigned { kErrDeadline = 1u, kErrWalkCount = 2u };

enum StatIdx {
    kStPushRounds = 0, kStPushVertices, kStPushTraversals, kStWalkEdges, kStWalkCount,
    kStWalkHops, kStFallback, kStTauIters, kStTauAmbiguous, kStPhase0,
    kStCount = kStPhase0 + 8
};
// The run counters are striped over kStStripes copies (block index modulo kStStripes) so that the
// warps of a launch do not all meet on one address; the host adds the copies up.
constexpr int kStStripes = 32;
static_assert(kStCount <= kRunStatSlots, "aesc_read_stats writes kStCount counters");

// Forms with their own tuned source-kernel layout on a handle: FP32, FP64, MIXED over F32 rows,
// MIXED over BF16 rows.  A layout is (kLayoutSmem if the residual vectors live in shared memory) |
// warps per block; 0 = the default rule.
constexpr uint16_t kLayoutSmem = 0x100;
constexpr uint16_t kLayoutBlock = 0x200;  // mixed form: multi-source block push
// parity forms: bit 0x400 set = the windowed sequential push, 0x800 = one vertex at a time (neither
// set: the default rule, by average degree)
constexpr uint16_t kLayoutWindow = 0x400;
constexpr uint16_t kLayoutNoWindow = 0x800;
// block push: the frontier size below which a round is compacted, as m / list_div, in bits 12-13
// (0 = the default list_div of 4, 1 = 2, 2 = 16, 3 = never compacted)
constexpr int kLayoutListShift = 12;
inline uint32_t layout_list_div(uint16_t layout) {
    switch ((layout >> kLayoutListShift) & 3) {
        case 1: return 2;
        case 2: return 16;
        case 3: return 0;
        default: return 4;
    }
}
inline int form_key(const tgtp_config& cfg) {
    if (cfg.precision == TGTP_PRECISION_FP32) return 0;
    if (cfg.precision == TGTP_PRECISION_FP64) return 1;
    return cfg.vec_dtype == TGTP_VEC_BF16 ? 3 : 2;
}

// The run's work words ([0] next list entry, [1] error flags, [2] list length, [3] unused) sit
// behind the striped counters in the same buffer, and the per-row marks behind them.
constexpr int kWorkWords = 4;
inline unsigned* run_work(tgtp_graph* g) {
    return reinterpret_cast<unsigned*>(g->stats.as<unsigned char>() +
                                       sizeof(unsigned long long) * kStCount * kStStripes);
}

__device__ __forceinline__ void stat_add(unsigned long long* stats, int i, unsigned long long v) {
    if (v) atomicAdd(stats + size_t(blockIdx.x % kStStripes) * kStCount + i, v);
}

struct TauConst {
    double one_m_l1sq, b1;  // 1 - lambda_1^2, log(1/|lambda_1|)
    double one_m_l2sq, b2;  // the same for lambda_{omega-1}
};

__device__ __forceinline__ uint64_t globaltimer_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Programmatic dependent launch: a kernel lets the next one in the stream start its blocks early
// (launch_dependents) and the next one waits for it to finish, with its memory visible, before it
// touches its results (wait).  Without the launch attribute wait returns at once.
__device__ __forceinline__ void pdl_launch_dependents() {
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// get_tau (src/aesc.h:129-135).  p1/p2 in the reference's parameter order (its callers pass
// (degree(u), degree(v)) into parameters named (dv, du)).  The 1 - lambda^2 and log(1/|lambda|)
// constants are formed on the host with the same libm as the reference.
template <class Real>
__device__ int get_tau(uint32_t p1, uint32_t p2, Real epsilon, double one_m_lam2, double b,
                       Real delta, Real upsilon, unsigned long long& ambiguous) {
    const Real ed = rsub(epsilon, delta);
    const Real eps_delta = double(ed) > 0.0 ? ed : epsilon;
    const double d1 = double(p1), d2 = double(p2);
    const double x = __dsub_rn(__dsub_rn(__dadd_rn(__ddiv_rn(1.0, d2), __ddiv_rn(1.0, d1)),
                                         __ddiv_rn(__ddiv_rn(2.0, d2), d1)),
                               double(upsilon));
    const double y = __ddiv_rn(__ddiv_rn(x, double(eps_delta)), one_m_lam2);
    const double a = log(std_max(y, 1.0));
    const double q = __dsub_rn(__ddiv_rn(a, b), 1.0);
    // A last-place difference between this log and the host's can only move ceil() when q sits
    // within rounding of an integer; count such edges so a caller can see that it never happens.
    if (a != 0.0 && fabs(q - rint(q)) <= 1e-12 * fmax(1.0, fabs(q))) ++ambiguous;
    const int tau = x86_f64_to_i32(std_max(ceil(q), 1.0));
    return tau % 2 == 0 ? int(tau + 1) : int(tau);
}

// eigen_t_1[i] cast to float after k multiplications by lambda_i^2.
__device__ __forceinline__ float etab_value(const float* tab, const double* tabd, uint32_t stride,
                                            uint32_t k, uint32_t i) {
    if (k < uint32_t(kTauTableRows)) return __ldg(tab + size_t(k) * stride + i);
    double e = __ldg(tabd + size_t(kTauTableRows - 1) * stride + i);
    const double sq = __ldg(tabd + i);
    for (uint32_t r = kTauTableRows - 1; r < k; ++r) e = __dmul_rn(e, sq);
    return from_f64<float>(e);
}

// Rows whose every tau is at most 1 stop after their first push round: with ell = 1 every slot has
// rest = tau - ell <= 0, so rwcost = 0 <= picost (src/aesc.h:483-502) and no slot walks
// (:508-526).  Their scores follow from the closed-form first round and they skip the source
// kernel.  The tau kernels mark each row that has a slot with tau > 1 (mark[r] == epoch) and append
// it, once per run, to the list the source kernel claims its sources from.
struct RowMarks {
    uint32_t* mark;
    uint32_t* list;
    unsigned* len;
    uint32_t epoch;
};

__device__ __forceinline__ void mark_row(const RowMarks& rm, uint32_t r) {
    if (*reinterpret_cast<volatile const uint32_t*>(rm.mark + r) == rm.epoch) return;
    if (atomicExch(rm.mark + r, rm.epoch) != rm.epoch) rm.list[atomicAdd(rm.len, 1u)] = r;
}

// ---- stage 1: tau per undirected edge ------------------------------------------------------------
// The FP32 form keeps the reference's sums: upsilon and the first delta term of an edge, each a chain
// of dependent additions over the eigen index in order, and a delta per further sweep.  A warp takes
// 16 forward slots.  The terms do not depend on one another, so all 32 lanes form them, one edge and
// 32 consecutive indices at a time (coalesced row pieces, a lane's constants loaded once per 32
// indices), and leave them in shared memory; then each lane adds up one chain, lanes 0 .. 15 the
// edges' upsilon and lanes 16 .. 31 their delta.
//
// What bounds it: issue slots at many warps per SM, else the chains (an addition and two conversions
// an index) and the divisions' latency, which is why four edges' terms are formed side by side and the
// next pieces fetched before they are used.  One edge per lane, terms and sums (a sweep costs a warp
// the same however few of its edges want it), took on the 88,234-edge graph 70 us at eps = 0.05 (one
// sweep) and 133 us at 0.01 (1.15 sweeps an edge, two or more in most warps); this takes 49 and 70.
// x / y for a divisor known in advance, 1e-150 < y <= 2^32, correctly rounded (round to nearest
// even), with Markstein's method (P. Markstein, IBM J. Res. Dev. 34(1), 1990): from r = RN(1/y), q0 =
// x * r is within 1.5 ulp, one correction q1 = q0 + r * (x - q0 y) within an ulp (remainders are exact
// by FMA), and his theorem says that a correction of such a quotient by a correctly rounded
// reciprocal is RN(x / y).  Nothing under- or overflows while 2^-913 <= x < 2^513 (known_range); any
// other x (zero and negative ones too) takes the correctly rounded division.  With a check of
// q1's remainder against half an ulp in place of the second correction a call on the 4,039-vertex
// graph (FP64, eps = 0.005) took 0.98 ms, so 0.87.
__device__ __forceinline__ double div_known(double x, double y, double r) {
    const double q0 = __dmul_rn(x, r);
    const double q1 = __fma_rn(__fma_rn(-q0, y, x), r, q0);
    return __fma_rn(__fma_rn(-q1, y, x), r, q1);
}
__device__ __forceinline__ bool known_range(double x) {
    return (unsigned(__double2hiint(x)) >> 20) - 110u < 0x600u - 110u;  // the sign bit counts as large
}
__device__ __forceinline__ double div_fixed(double x, double y, double r) {
    return known_range(x) ? div_known(x, y, r) : __ddiv_rn(x, y);
}

constexpr int kSumsEdges = 2, kSumsThreads = 256, kSumsBlocks = 4, kSumsUnroll = 4;  // tau_sums_kernel
constexpr uint32_t kTauEdges = 16;  // forward slots per warp: two chains each

__global__ void __launch_bounds__(kTauThreads, kTauBlocks)
tau_kernel(const uint32_t* __restrict__ idx, const uint32_t* __restrict__ adj,
           const uint32_t* __restrict__ row_of, const uint32_t* __restrict__ rev,
           const uint32_t* __restrict__ forward, uint64_t num_forward,
           const float* __restrict__ vec, uint32_t stride, uint32_t omega,
           const double* __restrict__ onep, const double* __restrict__ onem,
           const float* __restrict__ etab, const double* __restrict__ etabd, float epsilon,
           uint64_t m, TauConst c, int* __restrict__ taus, RowMarks rm,
           unsigned long long* __restrict__ stats) {
    __shared__ double terms[2][kTauEdges][33];  // upsilon's and delta's, of 32 indices
    pdl_launch_dependents();
    const uint32_t lane = threadIdx.x;
    const uint32_t half = lane / kTauEdges, mine = lane % kTauEdges;
    const float mreal = from_u64<float>(m);
    unsigned long long iters = 0, ambiguous = 0;
    for (uint64_t base = uint64_t(blockIdx.x) * kTauEdges; base < num_forward; base += uint64_t(gridDim.x) * kTauEdges) {
        // both halves of the warp hold the edges' state
        const uint64_t e = base + mine;
        uint32_t pos = 0, u = 0, v = 0, du = 1, dv = 1;
        bool done = e >= num_forward;
        if (!done) {
            pos = __ldg(forward + e);
            u = __ldg(row_of + pos);
            v = __ldg(adj + pos);
            du = __ldg(idx + u + 1) - __ldg(idx + u);
            dv = __ldg(idx + v + 1) - __ldg(idx + v);
        }
        float ups = 0.0f;
        int tau = 0, t = 1;
        for (uint32_t k = 0;; ++k) {
            const unsigned left = __ballot_sync(kFullMask, !done) & ((1u << kTauEdges) - 1u);
            if (!left) break;
            // get_upsilon (:151-162) with get_delta (:137-150) at eigen_t_1 = lambda^2, or get_delta
            // alone at lambda^(2(k+1)); indices 1 .. omega - 2
            float acc = 0.0f;
            const bool full = left == (1u << kTauEdges) - 1u;
            auto inside = [&](uint32_t i) { return i > 0 && i < omega - 1; };
            // one edge's row elements; a place that loads nothing divides 1
            auto piece = [&](int slot, uint32_t i, float& xu, float& xv) {
                const uint32_t uq = __shfl_sync(kFullMask, u, slot), vq = __shfl_sync(kFullMask, v, slot);
                xu = inside(i) ? __ldg(vec + size_t(uq) * stride + i) : 1.0f;
                xv = inside(i) ? __ldg(vec + size_t(vq) * stride + i) : 0.0f;
            };
            // the next indices' constants and first pieces are fetched before the sums of these
            struct {
                float et;
                double w, y;
            } next;
            auto constants = [&](uint32_t i) {
                next.et = inside(i) ? etab_value(etab, etabd, stride, k, i) : 1.0f;
                next.w = inside(i) ? __ldg(onep + i) : 1.0;
                next.y = inside(i) ? __ldg(onem + i) : 1.0;
            };
            float nu[4], nv[4];
            constants(lane);
            if (full) {
#pragma unroll
                for (int q = 0; q < 4; ++q) piece(q, lane, nu[q], nv[q]);
            }
            for (uint32_t i0 = 0; i0 < omega - 1; i0 += 32) {
                const uint32_t i = i0 + lane;
                const float et = next.et;
                const double w = next.w, y = next.y;
                const bool known = y > 1e-150 && y < 8.0;
                const double r = __drcp_rn(y);
                // the terms of four edges from their row pieces
                auto form = [&](const float (&xu)[4], const float (&xv)[4], const int (&slot)[4]) {
                    float d2[4];
                    double x[4], z[4];
                    bool ok = known;
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const float d = rsub(xu[q], xv[q]);
                        d2[q] = rmul(d, d);
                        x[q] = double(rmul(d2[q], et));
                        ok = ok && known_range(x[q]);
                        z[q] = div_known(x[q], y, r);
                    }
                    if (!ok) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) z[q] = __ddiv_rn(x[q], y);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        if (slot[q] >= 0) {
                            if (k == 0) terms[0][slot[q]][lane] = __dmul_rn(double(d2[q]), w);
                            terms[1][slot[q]][lane] = z[q];
                        }
                };
                if (full) {
#pragma unroll
                    for (int g = 0; g < int(kTauEdges); g += 4) {
                        float xu[4], xv[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            xu[q] = nu[q];
                            xv[q] = nv[q];
                            if (g + 4 < int(kTauEdges)) piece(g + 4 + q, i, nu[q], nv[q]);
                            else piece(q, i + 32, nu[q], nv[q]);
                        }
                        if (g + 4 == int(kTauEdges)) constants(i + 32);
                        const int slot[4] = {g, g + 1, g + 2, g + 3};
                        form(xu, xv, slot);
                    }
                } else {
                    constants(i + 32);
                    for (unsigned rest = left; rest;) {
                        float xu[4], xv[4];
                        int slot[4];
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            slot[q] = __ffs(int(rest)) - 1;
                            rest &= rest - 1;
                            xu[q] = 1.0f;
                            xv[q] = 0.0f;
                            if (slot[q] >= 0) piece(slot[q], i, xu[q], xv[q]);
                        }
                        form(xu, xv, slot);
                    }
                }
                __syncwarp();
                if (!done && (half || k == 0)) {
                    const double* const mt = terms[half][mine];
                    const uint32_t lo = i0 == 0 ? 1u : 0u, hi = min(32u, omega - 1 - i0);
                    if (lo == 0 && hi == 32) {
#pragma unroll 8
                        for (uint32_t j = 0; j < 32; ++j) acc = from_f64<float>(__dadd_rn(double(acc), mt[j]));
                    } else {
                        for (uint32_t j = lo; j < hi; ++j) acc = from_f64<float>(__dadd_rn(double(acc), mt[j]));
                    }
                }
                __syncwarp();
            }
            acc = rdiv(acc, mreal);
            if (k == 0) ups = __shfl_sync(kFullMask, acc, int(mine));
            // lanes 16 .. 31: the bound of this delta; lanes 0 .. 15, first sweep: tau from lambda_1
            int bound = 0;
            if (!done && (half || k == 0))
                bound = get_tau<float>(du, dv, epsilon, half ? c.one_m_l2sq : c.one_m_l1sq, half ? c.b2 : c.b1,
                                       half ? acc : 0.0f, half ? ups : 0.0f, ambiguous);
            if (k == 0) tau = __shfl_sync(kFullMask, bound, int(mine));
            const int tp = __shfl_sync(kFullMask, bound, int(mine + kTauEdges));
            if (!done) {
                iters += half;
                if (t <= tp && tp < tau) {
                    tau = tp;
                    t += 2;
                } else {
                    done = true;
                    taus[half ? __ldg(rev + pos) : pos] = tau;
                    if (tau > 1) mark_row(rm, half ? v : u);
                }
            }
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        iters += __shfl_xor_sync(kFullMask, iters, o);
        ambiguous += __shfl_xor_sync(kFullMask, ambiguous, o);
    }
    if (lane == 0) {
        stat_add(stats, kStTauIters, iters);
        stat_add(stats, kStTauAmbiguous, ambiguous);
    }
}

// ---- stage 1 helpers of the mixed form: compensated FP32 sums, FP64 bound, fixed-point residuals
// d_i^2 = (x_u[i] - x_v[i])^2 and the weighted terms d_i^2 (1 + lambda_i) and
// d_i^2 lambda_i^(2(k+1)) / (1 - lambda_i) are formed in FP32 from F32 or BF16 eigenvectors; the
// bound itself (get_tau: logs, ceil, odd rounding, the delta iteration) is evaluated in FP64.

__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bp)), __fsub_rn(b, bp));
}

// Residual arithmetic of the mixed form's push: the residual a vertex u receives in a round is the
// exact integer sum of its frontier neighbours' residuals in 2^-62 fixed point, divided (rounding
// down) by deg(u), then rounded once to FP32.  The sum does not depend on the order of the
// additions, so the per-source push and the block pushes add up the same bits.
// Sums are 64 bits wide, so they are taken modulo 4.  A round conserves the sum of deg(u) r(u), not
// that of r(u): a vertex whose neighbours have few others (a hub with leaves) can be sent up to the
// source's degree, and where that passes 4 its residual becomes (sum mod 4) / deg(u).  All pushes do
// so alike and the scores of this form are defined with it; the FP32 and FP64 forms have no such
// limit.  Sparse Chung-Lu graph (n = 25,860, exponent 2.1): 723 sources are sent more than 4 in round
// 2; scores next to them are 8e-4 off the exact values on average, 3.6e-4 in the FP64 form (eps = 0.005).
constexpr unsigned long long kFixOne = 1ull << 62;
__device__ __forceinline__ unsigned long long to_fixed(float r) {
    return __float2ull_rn(__fmul_rn(r, 0x1p62f));
}
__device__ __forceinline__ float from_fixed(unsigned long long s, uint32_t d) {
    return __fmul_rn(__ull2float_rn(s / d), 0x1p-62f);
}

// from_fixed of the sum hi * 2^32 + lo with inv = RN(1 / d) at hand.  q = RN(RN(s) * inv) is within 4
// ulps of s / d, and floor(s / d) is at most one below s / d, so q and the floor round to the same
// FP32 unless a midpoint between two FP32 lies within 4 ulps and one unit of q: the midpoints are
// where the 29 bits of q's significand below FP32's read 2^28.  Then, and for q below 2^30 (where one
// unit is no longer small against FP32's spacing), the quotient is taken exactly: q truncated is off
// by at most one while q is below 2^50, and the remainder tells; above that the 64-bit division.
__device__ __forceinline__ float from_fixed(uint32_t shi, uint32_t slo, uint32_t d, double inv) {
    // s in double with one rounding: 2^84 + hi 2^32 and 2^52 + lo by their bit patterns
    const double a = __dadd_rn(__hiloint2double(0x45300000, int(shi)), -19342813118337666422669312.0);
    const double q = __dmul_rn(__dadd_rn(a, __hiloint2double(0x43300000, int(slo))), inv);
    const int e = (__double2hiint(q) >> 20) - 1023;  // q is positive
    const int t = int(uint32_t(__double2loint(q)) & 0x1fffffffu) - 0x10000000;
    const int margin = 4 + (e < 53 ? int(1u << ((52 - e) & 31)) : 1);
    if (e < 30 || abs(t) <= margin) {
        const unsigned long long s = (static_cast<unsigned long long>(shi) << 32) | slo;
        if (e >= 50) return from_fixed(s, d);
        unsigned long long f = __double2ull_rz(q);
        const long long rem = (long long)(s - f * d);
        f = rem < 0 ? f - 1 : (rem >= (long long)d ? f + 1 : f);
        return __fmul_rn(__ull2float_rn(f), 0x1p-62f);
    }
    return __fmul_rn(__double2float_rn(q), 0x1p-62f);
}

__device__ __forceinline__ float vec_load(const float* p) { return __ldg(p); }
__device__ __forceinline__ float vec_load(const __nv_bfloat16* p) {
    return __bfloat162float(__ushort_as_bfloat16(__ldg(reinterpret_cast<const unsigned short*>(p))));
}

// get_tau (src/aesc.h:129-135) in FP64 for the mixed form (no bit-level parity asked): the degree
// terms from reciprocals, one division and the precomputed 1 / log(1/|lambda|).
__device__ __forceinline__ int get_tau_mixed(double inv1, double inv2, double epsilon,
                                             double one_m_lam2, double inv_b, double delta,
                                             double ups) {
    const double ed = epsilon - delta;
    const double eps_delta = ed > 0.0 ? ed : epsilon;
    const double x = (inv2 + inv1) - 2.0 * inv2 * inv1 - ups;
    const double a = log(std_max(x / (eps_delta * one_m_lam2), 1.0));
    const int tau = x86_f64_to_i32(std_max(ceil(a * inv_b - 1.0), 1.0));
    return tau % 2 == 0 ? tau + 1 : tau;
}

// Error-free combination of the eight partial sums of a lane group (TwoSum tree, the rounding
// errors carried and added back).
__device__ __forceinline__ double group_reduce(float a) {
    float ca = 0.f;
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) {
        const float a2 = __shfl_xor_sync(kFullMask, a, o);
        const float ca2 = __shfl_xor_sync(kFullMask, ca, o);
        float t, e;
        two_sum(a, a2, t, e);
        a = t;
        ca = __fadd_rn(__fadd_rn(ca, ca2), e);
    }
    return double(a) + double(ca);
}

// ---- stage 1 (FP64 and mixed forms): tau with eight lanes per edge ---------------------------------
// A warp takes four forward slots at a time, one per group of eight lanes.  Lane s of a group owns
// the index pieces {C j + P s, ..., C j + P s + P - 1} of the slot's two eigen rows (P = 2 FP64,
// 4 F32, 8 BF16 elements: one 16-byte load per row and piece; C = 8 P) and accumulates the terms
// d_i^2 w_i over them with fused multiply-adds, in index order, where d_i = x_u[i] - x_v[i] and
// w_i = 1 + lambda_i (upsilon, src/aesc.h:151-162) or lambda_i^(2(k+1)) / (1 - lambda_i) (delta_k,
// :137-150).  The weights are exactly zero at the indices the reference leaves out (0 and
// omega - 1) and past omega, so those terms add nothing.  The eight partial sums are combined by a
// fixed tree: ((S0 + S1) + (S2 + S3)) + ((S4 + S5) + (S6 + S7)) in FP64 for the FP64 form, the
// compensated group_reduce into FP64 for the mixed form.  The bound and the delta iteration follow
// :164-216 (get_tau, t += 2 while t <= tau' < tau).
template <class Vec> struct Split;
template <> struct Split<double> {
    static constexpr uint32_t P = 2;
    using Part = double;
};
template <> struct Split<float> {
    static constexpr uint32_t P = 4;
    using Part = float;
};
template <> struct Split<__nv_bfloat16> {
    static constexpr uint32_t P = 8;
    using Part = float;
};

// P consecutive elements starting at i0 (a multiple of P below omega); one 16-byte load when the
// row stride keeps pieces aligned, else element loads masked at omega.
__device__ __forceinline__ void load_piece(const double* __restrict__ row, uint32_t i0,
                                           uint32_t omega, bool vec_ok, double (&x)[2]) {
    if (vec_ok) {
        const double2 t = __ldg(reinterpret_cast<const double2*>(row + i0));
        x[0] = t.x;
        x[1] = t.y;
    } else {
        x[0] = __ldg(row + i0);
        x[1] = i0 + 1 < omega ? __ldg(row + i0 + 1) : 0.0;
    }
}
__device__ __forceinline__ void load_piece(const float* __restrict__ row, uint32_t i0,
                                           uint32_t omega, bool vec_ok, float (&x)[4]) {
    if (vec_ok) {
        const float4 t = __ldg(reinterpret_cast<const float4*>(row + i0));
        x[0] = t.x;
        x[1] = t.y;
        x[2] = t.z;
        x[3] = t.w;
    } else {
#pragma unroll
        for (uint32_t e = 0; e < 4; ++e) x[e] = i0 + e < omega ? __ldg(row + i0 + e) : 0.f;
    }
}
__device__ __forceinline__ void load_piece(const __nv_bfloat16* __restrict__ row, uint32_t i0,
                                           uint32_t omega, bool vec_ok, float (&x)[8]) {
    if (vec_ok) {
        const uint4 t = __ldg(reinterpret_cast<const uint4*>(row + i0));
        const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
        for (int h = 0; h < 4; ++h) {  // a bf16 is the upper half of its float
            x[2 * h] = __uint_as_float(w[h] << 16);
            x[2 * h + 1] = __uint_as_float(w[h] & 0xffff0000u);
        }
    } else {
#pragma unroll
        for (uint32_t e = 0; e < 8; ++e) x[e] = i0 + e < omega ? vec_load(row + i0 + e) : 0.f;
    }
}

// P consecutive elements from 16-byte aligned shared memory (the bulk-copied rows).
__device__ __forceinline__ void load_piece_shared(const double* p, double (&x)[2]) {
    const double2 t = *reinterpret_cast<const double2*>(p);
    x[0] = t.x;
    x[1] = t.y;
}
__device__ __forceinline__ void load_piece_shared(const float* p, float (&x)[4]) {
    const float4 t = *reinterpret_cast<const float4*>(p);
    x[0] = t.x;
    x[1] = t.y;
    x[2] = t.z;
    x[3] = t.w;
}
__device__ __forceinline__ void load_piece_shared(const __nv_bfloat16* p, float (&x)[8]) {
    const uint4 t = *reinterpret_cast<const uint4*>(p);
    const uint32_t w[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
    for (int h = 0; h < 4; ++h) {
        x[2 * h] = __uint_as_float(w[h] << 16);
        x[2 * h + 1] = __uint_as_float(w[h] & 0xffff0000u);
    }
}

__device__ __forceinline__ double split_fma(double a, double w, double s) {
    const double d2 = __dmul_rn(a, a);
    return __fma_rn(d2, w, s);
}
__device__ __forceinline__ float split_fma(float a, float w, float s) {
    const float d2 = __fmul_rn(a, a);
    return __fmaf_rn(d2, w, s);
}
__device__ __forceinline__ double split_sub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ float split_sub(float a, float b) { return __fsub_rn(a, b); }

__device__ __forceinline__ double split_reduce(double s) {
    s = __dadd_rn(s, __shfl_xor_sync(kFullMask, s, 1));
    s = __dadd_rn(s, __shfl_xor_sync(kFullMask, s, 2));
    return __dadd_rn(s, __shfl_xor_sync(kFullMask, s, 4));
}
__device__ __forceinline__ double split_reduce(float s) { return group_reduce(s); }

// Weight of index i in delta_k: row k + 1 of the padded table while k < kTauTableRows, beyond it
// the FP64 power chain continued from the last row of the eigen_t_1 table (src/aesc.h:201-203).
template <class Part>
__device__ __forceinline__ Part split_weight(const Part* __restrict__ wtab, uint32_t wpad,
                                             uint32_t k, uint32_t i, uint32_t omega,
                                             const double* __restrict__ etabd, uint32_t stride,
                                             const double* __restrict__ onem) {
    if (k < uint32_t(kTauTableRows)) return __ldg(wtab + size_t(k + 1) * wpad + i);
    if (i < 1 || i + 1 >= omega) return Part(0);
    double e = __ldg(etabd + size_t(kTauTableRows - 1) * stride + i);
    const double sq = __ldg(etabd + i);
    for (uint32_t r = kTauTableRows - 1; r < k; ++r) e = __dmul_rn(e, sq);
    return Part(__ddiv_rn(e, __ldg(onem + i)));
}

// Pass of one 8-lane group over the rows of one edge: lane sl's partial sums of d_i^2 wa_i and
// d_i^2 wb_i (two weight rows at once) or of d_i^2 w(k, i) alone.
template <class Vec, int ROWS>
__device__ __forceinline__ void split_pass(const Vec* __restrict__ ur, const Vec* __restrict__ vr,
                                           uint32_t omega, bool vec_ok, uint32_t sl,
                                           const typename Split<Vec>::Part* wa,
                                           const typename Split<Vec>::Part* wb,
                                           typename Split<Vec>::Part& sa,
                                           typename Split<Vec>::Part& sb) {
    using Part = typename Split<Vec>::Part;
    constexpr uint32_t P = Split<Vec>::P, C = 8 * P;
#pragma unroll 4
    for (uint32_t i0 = sl * P; i0 < omega; i0 += C) {
        Part xu[P], xv[P];
        load_piece(ur, i0, omega, vec_ok, xu);
        load_piece(vr, i0, omega, vec_ok, xv);
#pragma unroll
        for (uint32_t j = 0; j < P; ++j) {
            const Part d = split_sub(xu[j], xv[j]);
            if (ROWS == 2) sa = split_fma(d, wa[i0 + j], sa);
            sb = split_fma(d, wb[i0 + j], sb);
        }
    }
}

// Both sums of N edges at a time by one 8-lane group: the weights are read once for all of them, and
// one u row where the edges share it (SAME).
template <class Vec, int N, bool SAME>
__device__ __forceinline__ void split_pass_n(const Vec* const (&ur)[SAME ? 1 : N], const Vec* const (&vr)[N],
                                             uint32_t omega, bool vec_ok, uint32_t sl,
                                             const typename Split<Vec>::Part* wa,
                                             const typename Split<Vec>::Part* wb,
                                             typename Split<Vec>::Part (&sa)[N],
                                             typename Split<Vec>::Part (&sb)[N]) {
    using Part = typename Split<Vec>::Part;
    constexpr uint32_t P = Split<Vec>::P, C = 8 * P;
#pragma unroll kSumsUnroll
    for (uint32_t i0 = sl * P; i0 < omega; i0 += C) {
        Part xu[SAME ? 1 : N][P], xv[N][P];
#pragma unroll
        for (int q = 0; q < (SAME ? 1 : N); ++q) load_piece(ur[q], i0, omega, vec_ok, xu[q]);
#pragma unroll
        for (int q = 0; q < N; ++q) load_piece(vr[q], i0, omega, vec_ok, xv[q]);
#pragma unroll
        for (uint32_t j = 0; j < P; ++j) {
            const Part a = wa[i0 + j], b = wb[i0 + j];
#pragma unroll
            for (int q = 0; q < N; ++q) {
                const Part d = split_sub(xu[SAME ? 0 : q][j], xv[q][j]);
                sa[q] = split_fma(d, a, sa[q]);
                sb[q] = split_fma(d, b, sb[q]);
            }
        }
    }
}

// Stage 1a: the first sweep of every forward edge (upsilon and delta_0 sums), a pure gather.  A
// group takes two consecutive edges at a time (slots are in row order, so they mostly share their u);
// the next ones' vertices are fetched one step ahead.
//
// What bounds it: the rows come from L2, half of them from L1, and half of the L1's cycles went to
// the weights, read from shared memory for every edge.  Two edges per read and one u row for both took
// (with the launch) 21 -> 17 us on 88,234 edges in FP64, 249 -> 177 us on 2,000,000 in F32 rows.  Four edges
// a group need 80 registers, so 24 warps an SM: 20 us, 182 us; five blocks an SM spill: 18 us.
template <class Vec>
__global__ void __launch_bounds__(kSumsThreads, kSumsBlocks)
tau_sums_kernel(const uint4* __restrict__ fedge, uint64_t num_forward, const Vec* __restrict__ vec,
                uint32_t stride, uint32_t omega, const typename Split<Vec>::Part* __restrict__ wtab,
                uint32_t wpad, double2* __restrict__ sums, uint32_t* __restrict__ zero, uint64_t zero_words) {
    using Part = typename Split<Vec>::Part;
    constexpr int N = kSumsEdges;
    extern __shared__ __align__(16) unsigned char ssm[];
    pdl_launch_dependents();
    // the run's counters, work words and row marks, which the later kernels use
    for (uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < zero_words; i += uint64_t(gridDim.x) * blockDim.x)
        zero[i] = 0u;
    Part* wu = reinterpret_cast<Part*>(ssm);  // upsilon weights, then delta_0 weights
    Part* wd = wu + wpad;
    for (uint32_t i = threadIdx.x; i < 2 * wpad; i += blockDim.x) wu[i] = __ldg(wtab + i);
    __syncthreads();
    const uint32_t lane = threadIdx.x & 31, grp = lane >> 3, sl = lane & 7;
    const uint64_t gw = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    const bool vec_ok = stride % Split<Vec>::P == 0;
    // the N edges from e on (past the end: the last edge again)
    uint2 next[N];
    auto fetch = [&](uint64_t e) {
#pragma unroll
        for (int q = 0; q < N; ++q)
            next[q] = __ldg(reinterpret_cast<const uint2*>(fedge + min(e + q, num_forward - 1)));
    };
    if (gw * 4 * N < num_forward) fetch(gw * 4 * N + grp * N);
    for (uint64_t base = gw * 4 * N; base < num_forward; base += nw * 4 * N) {
        const uint64_t e = base + grp * N;
        const Vec* vr[N];
        uint32_t u[N];
        bool one = true;
#pragma unroll
        for (int q = 0; q < N; ++q) {
            u[q] = next[q].x;
            vr[q] = vec + size_t(next[q].y) * stride;
            one = one && u[q] == u[0];
        }
        if (base + nw * 4 * N < num_forward) fetch(e + nw * 4 * N);
        Part su[N], sd[N];
#pragma unroll
        for (int q = 0; q < N; ++q) su[q] = sd[q] = Part(0);
        if (__all_sync(kFullMask, one)) {
            const Vec* const ur[1] = {vec + size_t(u[0]) * stride};
            split_pass_n<Vec, N, true>(ur, vr, omega, vec_ok, sl, wu, wd, su, sd);
        } else {
#pragma unroll
            for (int h = 0; h < N; h += 2) {
                const Vec* const ur[2] = {vec + size_t(u[h]) * stride, vec + size_t(u[h + 1]) * stride};
                const Vec* const v2[2] = {vr[h], vr[h + 1]};
                Part a[2] = {Part(0), Part(0)}, b[2] = {Part(0), Part(0)};
                split_pass_n<Vec, 2, false>(ur, v2, omega, vec_ok, sl, wu, wd, a, b);
                su[h] = a[0];
                su[h + 1] = a[1];
                sd[h] = b[0];
                sd[h + 1] = b[1];
            }
        }
#pragma unroll
        for (int q = 0; q < N; ++q) {
            const double x = split_reduce(su[q]), y = split_reduce(sd[q]);
            if (sl == 0 && e + q < num_forward) sums[e + q] = make_double2(x, y);
        }
    }
}

// ---- bulk-copy pipeline helpers (cp.async.bulk + mbarrier, CTA scope, no multicast) -------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) {
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        " selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void fence_proxy_async() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
// bytes (a multiple of 16) from 16-byte aligned global memory into 16-byte aligned shared memory,
// completing on the mbarrier
__device__ __forceinline__ void bulk_g2s(uint32_t dst, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(dst), "l"(src), "r"(bytes), "r"(bar)
        : "memory");
}
// Bounded wait on an mbarrier phase: false (and the run's error flag set) if it never completes.
__device__ __forceinline__ bool mbar_wait_bounded(uint32_t bar, uint32_t parity, unsigned* work) {
    for (uint32_t it = 0; it < (1u << 22); ++it)
        if (mbar_try_wait(bar, parity)) return true;
    atomicOr(work + 1, kErrDeadline);
    return false;
}

// Stage 1a over bulk copies: each warp runs its own NST-stage pipeline; a stage holds the two
// eigen rows (omega elements, a multiple of 16 bytes) of the warp's next four edges, brought into
// shared memory by one lane per edge with cp.async.bulk and completed on the stage's mbarrier.
// The eight lanes of group g then sum edge g's terms from shared memory exactly as
// tau_sums_kernel does from global memory (same pieces, same order), so the sums are identical.
template <class Vec> struct BulkShape;
template <> struct BulkShape<double> { static constexpr int WPB = 2; };
template <> struct BulkShape<float> { static constexpr int WPB = 4; };
template <> struct BulkShape<__nv_bfloat16> { static constexpr int WPB = 8; };
constexpr int kBulkStages = 4;

template <class Vec>
__global__ void __launch_bounds__(32 * BulkShape<Vec>::WPB)
tau_sums_bulk_kernel(const uint4* __restrict__ fedge, uint64_t num_forward,
                     const Vec* __restrict__ vec, uint32_t stride, uint32_t omega,
                     const typename Split<Vec>::Part* __restrict__ wtab, uint32_t wpad,
                     double2* __restrict__ sums, unsigned* __restrict__ work) {
    using Part = typename Split<Vec>::Part;
    constexpr uint32_t P = Split<Vec>::P, C = 8 * P;
    constexpr int NST = kBulkStages;
    extern __shared__ __align__(128) unsigned char bsm[];
    pdl_launch_dependents();
    const uint32_t rowb = omega * uint32_t(sizeof(Vec));
    const uint32_t lane = threadIdx.x & 31, wib = threadIdx.x >> 5, grp = lane >> 3, sl = lane & 7;
    // layout: per warp NST stages x 4 edges x 2 rows, then the warp's NST mbarriers; the weights
    // after all warps
    const size_t per_warp = size_t(NST) * 8 * rowb + NST * 8;
    unsigned char* wbase = bsm + size_t(wib) * per_warp;
    const uint32_t bars = smem_u32(wbase + size_t(NST) * 8 * rowb);
    Part* wu = reinterpret_cast<Part*>(bsm + size_t(blockDim.x >> 5) * per_warp);
    Part* wd = wu + wpad;
    for (uint32_t i = threadIdx.x; i < 2 * wpad; i += blockDim.x) wu[i] = __ldg(wtab + i);
    if (lane == 0) {
        for (int st = 0; st < NST; ++st) mbar_init(bars + 8 * st, 1);
        mbar_fence_init();
    }
    __syncthreads();
    const uint64_t gw = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    auto step_base = [&](uint64_t t) { return (gw + t * nw) * 4; };
    // lane l < 4 holds the record of edge l of a step, fetched a step before the copies need it
    auto fetch = [&](uint64_t t) {
        const uint64_t e = step_base(t) + lane;
        return (lane < 4 && e < num_forward) ? __ldg(fedge + e) : make_uint4(0, 0, 0, 0);
    };
    // stage st <- the rows of step t's edges (records in r)
    auto issue = [&](uint64_t t, int st, uint4 r) {
        const uint64_t eb = step_base(t);
        if (eb >= num_forward) return;
        const uint32_t cnt = uint32_t(min(uint64_t(4), num_forward - eb));
        const uint32_t bar = bars + 8 * st;
        if (lane == 0) {
            fence_proxy_async();  // the stage's previous contents were read through the generic proxy
            mbar_expect_tx(bar, cnt * 2 * rowb);
        }
        __syncwarp();
        if (lane < cnt) {
            unsigned char* dst = wbase + (size_t(st) * 8 + lane * 2) * rowb;
            bulk_g2s(smem_u32(dst), vec + size_t(r.x) * stride, rowb, bar);
            bulk_g2s(smem_u32(dst + rowb), vec + size_t(r.y) * stride, rowb, bar);
        }
    };
    for (int st = 0; st < NST; ++st) issue(uint64_t(st), st, fetch(uint64_t(st)));
    uint4 ahead = fetch(uint64_t(NST));
    bool ok = true;
    uint64_t t = 0;
    for (; step_base(t) < num_forward; ++t) {
        const int st = int(t % NST);
        const uint4 next_rec = ahead;
        ahead = fetch(t + NST + 1);
        if (!mbar_wait_bounded(bars + 8 * st, uint32_t((t / NST) & 1), work)) {
            ok = false;
            break;
        }
        const uint64_t e = step_base(t) + grp;
        Part su = Part(0), sd = Part(0);
        if (e < num_forward) {
            const Vec* ur = reinterpret_cast<const Vec*>(wbase + (size_t(st) * 8 + grp * 2) * rowb);
            const Vec* vr = ur + omega;
#pragma unroll 4
            for (uint32_t i0 = sl * P; i0 < omega; i0 += C) {
                Part xu[P], xv[P];
                load_piece_shared(ur + i0, xu);
                load_piece_shared(vr + i0, xv);
#pragma unroll
                for (uint32_t j = 0; j < P; ++j) {
                    const Part d = split_sub(xu[j], xv[j]);
                    su = split_fma(d, wu[i0 + j], su);
                    sd = split_fma(d, wd[i0 + j], sd);
                }
            }
        }
        const double us = split_reduce(su), ds = split_reduce(sd);
        if (sl == 0 && e < num_forward) sums[e] = make_double2(us, ds);
        __syncwarp();  // every lane is done with the stage
        issue(t + NST, st, next_rec);
    }
    if (!ok) {  // drain what is still in flight before the shared memory goes away (bounded)
        for (uint64_t u = t + 1; u < t + NST && step_base(u) < num_forward; ++u)
            if (!mbar_wait_bounded(bars + 8 * int(u % NST), uint32_t((u / NST) & 1), work)) break;
    }
}

// The bound of one edge per lane (src/aesc.h:181-207): tau_0 from lambda_1, then tau' from
// delta_k while t <= tau' < tau (t += 2).  Edges that need a further delta sweep are served four
// at a time by the warp's 8-lane groups.  Writes tau to both slots and marks the two rows when
// tau > 1.  All 32 lanes of the warp call it together; act says whether the lane holds an edge.
template <class Vec>
struct BoundArgs {
    const uint32_t* deg;
    const Vec* vec;
    uint32_t stride, omega;
    const typename Split<Vec>::Part* wtab;
    uint32_t wpad;
    const double* etabd;
    const double* onem;
    double eps_half, mdbl;
    TauConst c;
    int* taus;
    RowMarks rm;
};

template <class Vec>
__device__ __forceinline__ void bound_lanes(const BoundArgs<Vec>& A, bool act, uint4 rec, double2 sm,
                                            unsigned long long& iters,
                                            unsigned long long& ambiguous) {
    using Part = typename Split<Vec>::Part;
    constexpr bool kF64 = std::is_same<Vec, double>::value;
    constexpr uint32_t P = Split<Vec>::P, C = 8 * P;
    const uint32_t lane = threadIdx.x & 31, grp = lane >> 3, sl = lane & 7;
    const bool vec_ok = A.stride % P == 0;
    const double inv_b1 = 1.0 / A.c.b1, inv_b2 = 1.0 / A.c.b2;
    uint32_t du = 1, dv = 1;
    if (act) {
        du = __ldg(A.deg + rec.x);
        dv = __ldg(A.deg + rec.y);
    }
    const double inv1 = 1.0 / double(du), inv2 = 1.0 / double(dv);
    auto bound = [&](double one_m_lam2, double b, double inv_b, double dl, double up) {
        if constexpr (kF64) {
            return get_tau<double>(du, dv, A.eps_half, one_m_lam2, b, dl, up, ambiguous);
        } else {
            return get_tau_mixed(inv1, inv2, A.eps_half, one_m_lam2, inv_b, dl, up);
        }
    };
    int tau = 0, t = 1;
    uint32_t k = 1;
    bool need = false;
    double ups = 0;
    if (act) {
        ups = kF64 ? __ddiv_rn(sm.x, A.mdbl) : sm.x / A.mdbl;
        const double del = kF64 ? __ddiv_rn(sm.y, A.mdbl) : sm.y / A.mdbl;
        tau = bound(A.c.one_m_l1sq, A.c.b1, inv_b1, 0.0, 0.0);
        ++iters;
        const int tp = bound(A.c.one_m_l2sq, A.c.b2, inv_b2, del, ups);
        if (t <= tp && tp < tau) {
            tau = tp;
            t += 2;
            need = true;
        }
    }
    // further delta sweeps (:191-204), four edges at a time
    unsigned nb;
    while ((nb = __ballot_sync(kFullMask, need)) != 0) {
        int sel[4];
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            sel[g] = nb ? __ffs(nb) - 1 : -1;
            if (nb) nb &= nb - 1;
        }
        const uint32_t src_lane = sel[grp] < 0 ? 0u : uint32_t(sel[grp]);
        const uint32_t gu = __shfl_sync(kFullMask, rec.x, src_lane);
        const uint32_t gv = __shfl_sync(kFullMask, rec.y, src_lane);
        const uint32_t gk = __shfl_sync(kFullMask, k, src_lane);
        Part s2 = Part(0);
        if (sel[grp] >= 0) {
            const Vec* ur = A.vec + size_t(gu) * A.stride;
            const Vec* vr = A.vec + size_t(gv) * A.stride;
            if (gk < uint32_t(kTauTableRows)) {
                split_pass<Vec, 1>(ur, vr, A.omega, vec_ok, sl, nullptr,
                                   A.wtab + size_t(gk + 1) * A.wpad, s2, s2);
            } else {
                for (uint32_t i0 = sl * P; i0 < A.omega; i0 += C) {
                    Part xu[P], xv[P];
                    load_piece(ur, i0, A.omega, vec_ok, xu);
                    load_piece(vr, i0, A.omega, vec_ok, xv);
#pragma unroll
                    for (uint32_t j = 0; j < P; ++j)
                        s2 = split_fma(split_sub(xu[j], xv[j]),
                                       split_weight<Part>(A.wtab, A.wpad, gk, i0 + j, A.omega,
                                                          A.etabd, A.stride, A.onem),
                                       s2);
                }
            }
        }
        const double dsum = split_reduce(s2);
        double mine = 0.0;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            const double r = __shfl_sync(kFullMask, dsum, g * 8);
            if (sel[g] == int(lane)) mine = r;
        }
        bool served = false;
#pragma unroll
        for (int g = 0; g < 4; ++g) served |= sel[g] == int(lane);
        if (served) {
            const double del = kF64 ? __ddiv_rn(mine, A.mdbl) : mine / A.mdbl;
            ++iters;
            const int tp = bound(A.c.one_m_l2sq, A.c.b2, inv_b2, del, ups);
            if (t <= tp && tp < tau) {
                tau = tp;
                t += 2;
                ++k;
            } else {
                need = false;
            }
        }
    }
    if (act) {
        A.taus[rec.z] = tau;
        A.taus[rec.w] = tau;
        if (tau > 1) {
            mark_row(A.rm, rec.x);
            mark_row(A.rm, rec.y);
        }
    }
}

__device__ __forceinline__ void flush_tau_stats(unsigned long long iters, unsigned long long ambiguous,
                                                unsigned long long* stats) {
#pragma unroll
    for (int o = 16; o; o >>= 1) {
        iters += __shfl_xor_sync(kFullMask, iters, o);
        ambiguous += __shfl_xor_sync(kFullMask, ambiguous, o);
    }
    if ((threadIdx.x & 31) == 0) {
        stat_add(stats, kStTauIters, iters);
        stat_add(stats, kStTauAmbiguous, ambiguous);
    }
}

// Stage 1b: the bound per edge, one lane per edge (a variant that evaluated the bounds inside the
// gather kernel, 32 edges per warp at a time, measured slower: the bound's FP64 chains then sit on
// the gather's critical path).
template <class Vec>
__global__ void __launch_bounds__(256)
tau_bound_kernel(const uint4* __restrict__ fedge, uint64_t num_forward,
                 const double2* __restrict__ sums, BoundArgs<Vec> A, uint32_t per_warp,
                 unsigned long long* __restrict__ stats) {
    const uint32_t lane = threadIdx.x & 31;
    const uint64_t gw = (uint64_t(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
    const uint64_t nw = (uint64_t(gridDim.x) * blockDim.x) >> 5;
    unsigned long long iters = 0, ambiguous = 0;
    pdl_launch_dependents();
    pdl_wait();  // the sums of tau_sums_kernel
    for (uint64_t base = gw * per_warp; base < num_forward; base += nw * per_warp) {
        const uint64_t e = base + lane;
        const bool act = lane < per_warp && e < num_forward;
        uint4 rec = make_uint4(0, 0, 0, 0);
        double2 sm = make_double2(0.0, 0.0);
        if (act) {
            rec = __ldg(fedge + e);
            sm = sums[e];
        }
        bound_lanes<Vec>(A, act, rec, sm, iters, ambiguous);
    }
    flush_tau_stats(iters, ambiguous, stats);
}

// ---- stage 2: per-source push, edge bound and walks -----------------------------------------------
struct WalkItem {
    uint32_t pos, v, len, pad;  // pad: in a walk queue, the item's list entry (its source)
    unsigned long long nr;
};

// Outcome of the push of one listed source in push_block_kernel or push_shared_kernel.
struct PrePush {
    int ell;           // rounds pushed
    float gmax, gmin;  // residual max / min over the final frontier (gmin before the |q| < n rule)
    uint32_t support;  // size of the final frontier
};


template <class Real>
__device__ __forceinline__ Real warp_max(Real x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x = std_max(x, __shfl_xor_sync(kFullMask, x, o));
    return x;
}
template <class Real>
__device__ __forceinline__ Real warp_min(Real x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x = std_min(x, __shfl_xor_sync(kFullMask, x, o));
    return x;
}
__device__ __forceinline__ unsigned long long warp_sum_u64(unsigned long long x) {
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(kFullMask, x, o);
    return x;
}

// preds[pos] += (pvec[src] - pvec[w]) / ds (:236): in the row's own real type in the parity forms,
// accumulated in FP64 in the mixed form.
template <class Real, class Acc>
__device__ __forceinline__ Acc row_update(Acc old, Real ps, Real pv, Real ds) {
    if constexpr (std::is_same<Real, Acc>::value) {
        return radd(old, rdiv(rsub(ps, pv), ds));
    } else {
        return __dadd_rn(old, __ddiv_rn(__dsub_rn(double(ps), double(pv)), double(ds)));
    }
}

// Order-preserving integer images of non-negative reals (residuals are never negative), so that
// shared-memory integer atomics give max / min.
__device__ __forceinline__ unsigned long long ord_bits(float x) { return __float_as_uint(x); }
__device__ __forceinline__ unsigned long long ord_bits(double x) {
    return (unsigned long long)__double_as_longlong(x);
}
template <class Real> __device__ __forceinline__ Real from_ord(unsigned long long b);
template <> __device__ __forceinline__ float from_ord<float>(unsigned long long b) {
    return __uint_as_float(unsigned(b));
}
template <> __device__ __forceinline__ double from_ord<double>(unsigned long long b) {
    return __longlong_as_double((long long)b);
}

// ---- stage 2a (mixed form, large graphs): multi-source Jacobi push as a pull product -----------
// In the mixed form a push round drains the whole frontier at once (Jacobi), so a round is exactly
// r <- D^-1 A r: with r supported on the frontier q, every vertex u receives the residuals of its
// frontier neighbours divided by deg(u), and the frontier's own residuals are pushed out.  For
// graphs whose residual vector does not fit in shared memory, each CTA takes S = 32 listed sources
// at a time and keeps their residual vectors as the columns of an n x S row-major block in HBM; a
// round is one pass over the CSR in which warp w pulls rows u = w, w + 32, ...: lane j adds the
// column-j entries of u's neighbours in CSR order (one coalesced 128-byte row read per neighbour)
// and divides by deg(u).  The same pass accumulates each column's frontier statistics (degree sum,
// max, min, size of the support), so the stop test of src/aesc.h:483-502 needs no further pass.
// Columns whose source has stopped are carried over unchanged, so when the last one stops every
// column holds its source's final residual vector; the edge bound, chi and walk counts of those
// sources then run in mixed_source_kernel<kColumn>, which reads the column in place, and their walks
// in kernels of their own.
constexpr int kBlockCols = 32;

// The final residual vector (n contiguous floats) of list entry list_base + slot after a block push:
// with finals, a column of its 32-source CTA's spare block (finals[cta] tells which of the two
// blocks is the spare), else the entry's own.
__device__ __forceinline__ const float* pre_column(const float* cols, const uint32_t* finals,
                                                   uint32_t slot, uint32_t n) {
    if (!finals) return cols + size_t(slot) * n;
    const uint32_t cta = slot / kBlockCols, col = slot % kBlockCols;
    return cols + (size_t(cta) * 2 + (1u - finals[cta])) * size_t(n) * kBlockCols + size_t(col) * n;
}
// Walk items of the block push's sources with at least kHeavyNr walks of at most kHeavyLen hops
// go to heavy_walk_kernel, which walks 32 of their bouquets at once instead of one after another.
constexpr unsigned long long kHeavyNr = 512;
constexpr uint32_t kHeavyLen = 32;
// rows a warp of push_block_kernel claims at a time (their dependent loads are issued together).
// Measured on three graphs (n = 25,860 / 143,522 / 199,772): 1 row is 3-6 % faster than the plain
// loop (the row's own value and first adjacency chunk are requested before its neighbours are
// read), 2 and 4 rows 0-25 % slower (the kernel is at its 64-register cap).
constexpr int kRowBatch = 1;


struct PushBlockParams {
    const uint32_t* idx;
    const uint32_t* adj;
    const uint32_t* deg;
    const uint2* adjd;
    uint32_t n;
    uint64_t m;
    const int* taus;
    double* preds;
    unsigned* work;        // [1] error flags, [2] list length
    const uint32_t* rows;  // the list of sources
    uint32_t base;         // first list entry of this wave
    double eps, logmd;
    float* cols;           // per CTA: two n x S blocks
    uint32_t* final_buf;   // per CTA: the block that holds the final columns
    PrePush* pre;          // per list entry
    bool bits;             // the three row masks fit in shared memory (else they live in gbits)
    bool cur_smem;         // (when !bits) the current round's mask alone fits in shared memory
    uint32_t* gbits;       // per CTA: three n-bit row masks in global memory (L2), when not in smem
    uint32_t* lists;       // per CTA: four row lists of n entries (see push_block_kernel)
    uint32_t list_div;     // a round is compacted when its live rows' degree sum * list_div < m
    int rounds_mode;       // 0 = by that rule, 1 = every round compacted, 2 = every round full
    unsigned long long* stats;
    uint64_t budget_ns;
};

// Exclusive prefix sum over the block's threads (blockDim.x a multiple of 32, at most 1024); the
// block total goes to *total.  Uses `tmp` (32 words of shared memory).
__device__ __forceinline__ uint32_t block_exclusive_scan(uint32_t v, uint32_t* tmp, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    uint32_t incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(kFullMask, incl, o);
        if (lane >= uint32_t(o)) incl += y;
    }
    if (lane == 31) tmp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
        const uint32_t w = lane < nwarp ? tmp[lane] : 0u;
        uint32_t wi = w;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(kFullMask, wi, o);
            if (lane >= uint32_t(o)) wi += y;
        }
        if (lane < nwarp) tmp[lane] = wi - w;
        if (lane == 31) *total = wi;
    }
    __syncthreads();
    const uint32_t out = tmp[warp] + incl - v;
    __syncthreads();
    return out;
}

// The rows whose bit is set in `mask` (words of 32 rows), in increasing order, into `out`; the
// count goes to *count.  Each thread takes a contiguous run of words.
__device__ __forceinline__ void compact_mask(const uint32_t* mask, uint32_t words, uint32_t n,
                                             uint32_t* out, uint32_t* tmp, uint32_t* count) {
    const uint32_t per = (words + blockDim.x - 1) / blockDim.x;
    const uint32_t w0 = min(words, threadIdx.x * per), w1 = min(words, w0 + per);
    uint32_t c = 0;
    for (uint32_t w = w0; w < w1; ++w) c += __popc(mask[w]);
    uint32_t pos = block_exclusive_scan(c, tmp, count);
    for (uint32_t w = w0; w < w1; ++w) {
        uint32_t b = mask[w];
        while (b) {
            const uint32_t r = w * 32u + uint32_t(__ffs(b) - 1);
            b &= b - 1;
            if (r < n) out[pos++] = r;
        }
    }
}

__global__ void __launch_bounds__(1024, 1)
push_block_kernel(PushBlockParams p) {
    constexpr int S = kBlockCols;
    // Row masks, one bit per row: bcur / bnxt mark the rows with a nonzero running column in the
    // cur / nxt block (the pull skips the 128-byte reads of neighbour rows whose bit is clear);
    // tmask marks the rows a compacted round processes.  In shared memory while the three fit
    // (p.bits), else in this CTA's part of p.gbits (L2-resident).
    //
    // Row lists (n entries each, in p.lists): Lc = rows with any nonzero column in cur, Lp = the
    // same for the block nxt still holds from the round before, Ln = those of the round being
    // formed, P = the rows a compacted round processes.  A round is either a full pass over all n
    // rows (dense frontiers) or a compacted one over P = (neighbours of the running-live rows of
    // cur) U Lc U Lp, in increasing row order: a row outside the neighbourhood of the live rows
    // receives nothing, Lc carries the stopped columns and zeroes the running ones, and Lp covers
    // every row nxt still holds from two rounds before, so no stale row survives.  Both give the
    // same values; the choice per round is by the live rows' degree sum (the scatter work of the
    // compaction) against m / list_div.
    extern __shared__ uint32_t s_bits[];
    __shared__ uint32_t s_src[S], s_rb[S], s_ds[S], s_support[S], s_ell[S];
    __shared__ unsigned long long s_picost[S];
    __shared__ unsigned s_max[S], s_min[S];  // float bits of non-negative residuals
    __shared__ int s_active[S];
    __shared__ int s_any;
    __shared__ uint32_t s_tmp[32];
    __shared__ uint32_t s_lc, s_lp, s_ln, s_pn;  // list lengths
    __shared__ uint32_t s_next;                  // next row of the round (claimed by warps)
    __shared__ unsigned long long s_live_deg;   // degree sum of the running-live rows of cur
    pdl_launch_dependents();
    pdl_wait();  // the list, and the previous wave's readers of these blocks
    const uint32_t lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarp = blockDim.x >> 5;
    const uint32_t n = p.n;
    const unsigned len = p.work[2];
    const uint64_t first = uint64_t(p.base) + uint64_t(blockIdx.x) * S;
    if (first >= len) return;
    const uint32_t cnt = uint32_t(min(uint64_t(S), len - first));
    float* A = p.cols + size_t(blockIdx.x) * 2 * size_t(n) * S;
    float* B = A + size_t(n) * S;
    const uint64_t deadline = globaltimer_ns() + p.budget_ns;
    unsigned long long st_pv = 0, st_tr = 0, st_rounds = 0;

    // both blocks start at zero (a compacted round writes only the rows it processes)
    for (size_t i = threadIdx.x; i < size_t(n) * S / 2; i += blockDim.x)
        reinterpret_cast<float4*>(A)[i] = make_float4(0.f, 0.f, 0.f, 0.f);
    const uint32_t words = (n + 31) / 32;
    // Mask placement: all three in shared memory; or (cur_smem) bcur in shared memory -- it is
    // read for every neighbour chunk of the pull -- with bnxt and tmask in global memory, bnxt
    // copied into bcur at each round's end; or all three in global memory.
    uint32_t* const gb = p.gbits ? p.gbits + size_t(blockIdx.x) * 3 * words : nullptr;
    uint32_t* bcur = (p.bits || p.cur_smem) ? s_bits : gb;
    uint32_t* bnxt = p.bits ? s_bits + words : gb + words;
    uint32_t* tmask = p.bits ? s_bits + 2 * words : gb + 2 * words;
    for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) {
        bcur[i] = 0u;
        bnxt[i] = 0u;
        tmask[i] = 0u;
    }
    uint32_t* const lbase = p.lists + size_t(blockIdx.x) * 4 * size_t(n);
    uint32_t* Lc = lbase;
    uint32_t* Lp = lbase + n;
    uint32_t* Ln = lbase + 2 * size_t(n);
    uint32_t* const P = lbase + 3 * size_t(n);
    if (threadIdx.x < S) {
        const uint32_t j = threadIdx.x;
        s_active[j] = j < cnt;
        s_src[j] = j < cnt ? __ldg(p.rows + first + j) : 0;
        s_picost[j] = 0;
        s_max[j] = 0;
        s_min[j] = __float_as_uint(1.f);
        s_ell[j] = 1;
    }
    if (threadIdx.x == 0) {
        s_lp = 0;
        s_live_deg = 0;
    }
    __syncthreads();
    // round 1 in closed form: the frontier {src} pushes 1 / deg(u) to every neighbour u
    if (warp < cnt) {
        const uint32_t j = warp, src = s_src[j];
        const uint32_t rb = __ldg(p.idx + src), dsi = __ldg(p.idx + src + 1) - rb;
        const float ds = float(dsi);
        const double pinit = __ddiv_rn(1.0, double(ds));
        unsigned long long pc = 0;
        float mx = 0.f, mn = 1.f;
        for (uint32_t o = lane; o < dsi; o += 32) {
            const uint2 a = __ldg(p.adjd + rb + o);
            const float pu = from_fixed(kFixOne, a.y);
            A[size_t(a.x) * S + j] = pu;
            atomicOr(bcur + (a.x >> 5), 1u << (a.x & 31));
            pc += a.y;
            mx = fmaxf(mx, pu);
            mn = fminf(mn, pu);
            p.preds[rb + o] = row_update<float, double>(pinit, 0.f, pu, ds);
        }
        pc = warp_sum_u64(pc);
        mx = warp_max(mx);
        mn = warp_min(mn);
        if (lane == 0) {
            s_rb[j] = rb;
            s_ds[j] = dsi;
            s_picost[j] = pc;
            s_max[j] = __float_as_uint(mx);
            s_min[j] = __float_as_uint(mn);
            s_support[j] = dsi;
        }
        st_pv += lane == 0 ? 1 : 0;
        st_tr += lane == 0 ? dsi : 0;
    }
    __syncthreads();
    // Lc after round 1: the rows of bcur (every column runs, so a nonzero row is running-live)
    compact_mask(bcur, words, n, Lc, s_tmp, &s_lc);
    __syncthreads();
    {
        unsigned long long d = 0;
        for (uint32_t k = threadIdx.x; k < s_lc; k += blockDim.x) d += __ldg(p.deg + Lc[k]);
        d = warp_sum_u64(d);
        if (lane == 0 && d) atomicAdd(&s_live_deg, d);
    }
    __syncthreads();
    float* cur = A;
    float* nxt = B;
    uint32_t fin = 0;
    while (true) {
        // ---- stop test of every running source (one warp per source) ----
        if (threadIdx.x == 0) s_any = 0;
        __syncthreads();
        if (warp < cnt && s_active[warp]) {
            const uint32_t j = warp, rb = s_rb[j], dsi = s_ds[j];
            const int ell = int(s_ell[j]);
            const float gmax = __uint_as_float(s_max[j]);
            const float gmin = s_support[j] < n ? 0.f : __uint_as_float(s_min[j]);
            const double dse0 = __dmul_rn(double(float(dsi)), p.eps);
            const double dse2 = __dmul_rn(dse0, dse0);
            double rw = 0;
            for (uint32_t c = 0; c < dsi; c += 32) {
                const uint32_t o = c + lane;
                const int rest = o < dsi ? __ldg(p.taus + rb + o) - ell : 0;
                double nrd = 0;
                const bool has = rest > 0;
                if (has) {
                    const double chi = __dmul_rn(__dmul_rn(2.0, double(rest)),
                                                 __dsub_rn(double(gmax), double(gmin)));
                    const double num = __dmul_rn(__dmul_rn(8.0, __dmul_rn(chi, chi)), p.logmd);
                    nrd = std_max(ceil(__ddiv_rn(num, dse2)), 1.0);
                }
                unsigned hb = __ballot_sync(kFullMask, has);
                while (hb) {  // rwcost += nr in slot order
                    const int l = __ffs(hb) - 1;
                    hb &= hb - 1;
                    rw = __dadd_rn(rw, __shfl_sync(kFullMask, nrd, l));
                }
            }
            const bool stop = double(s_picost[j]) >= __dmul_rn(25.0, rw);
            const bool late = globaltimer_ns() > deadline;
            if (lane == 0) {
                if (stop || late) {
                    s_active[j] = 0;
                    PrePush r;
                    r.ell = ell;
                    r.gmax = gmax;
                    r.gmin = __uint_as_float(s_min[j]);
                    r.support = s_support[j];
                    p.pre[first + j] = r;
                    st_rounds += uint64_t(ell);
                    if (late && !stop) atomicOr(p.work + 1, kErrDeadline);
                } else {
                    s_any = 1;
                    st_pv += s_support[j];
                    st_tr += s_picost[j];
                }
            }
        }
        __syncthreads();
        if (!s_any) break;
        // ---- the rows this round processes: all n, or the compacted list P ----
        const bool compact = p.rounds_mode == 1 ||
                             (p.rounds_mode == 0 &&
                              double(s_live_deg) * double(p.list_div) < double(p.m));
        __syncthreads();  // every thread has read s_live_deg before it is reset below
        if (compact) {
            for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) tmask[i] = 0u;
            __syncthreads();
            for (uint32_t k = threadIdx.x; k < s_lp; k += blockDim.x)
                atomicOr(tmask + (Lp[k] >> 5), 1u << (Lp[k] & 31));
            for (uint32_t k = warp; k < s_lc; k += nwarp) {
                const uint32_t w = Lc[k];
                if (lane == 0) atomicOr(tmask + (w >> 5), 1u << (w & 31));
                if (!((bcur[w >> 5] >> (w & 31)) & 1u)) continue;  // only stopped columns here
                const uint32_t wb = __ldg(p.idx + w), we = __ldg(p.idx + w + 1);
                for (uint32_t o = wb + lane; o < we; o += 32) {
                    const uint32_t u = __ldg(p.adj + o);
                    atomicOr(tmask + (u >> 5), 1u << (u & 31));
                }
            }
            __syncthreads();
            compact_mask(tmask, words, n, P, s_tmp, &s_pn);
        }
        // ---- one Jacobi round for the running columns; stopped columns are carried over ----
        if (threadIdx.x < S) {
            s_picost[threadIdx.x] = 0;
            s_max[threadIdx.x] = 0;
            s_min[threadIdx.x] = __float_as_uint(1.f);
            s_support[threadIdx.x] = 0;
        }
        if (threadIdx.x == 0) {
            s_ln = 0;
            s_live_deg = 0;
            s_next = nwarp * kRowBatch;
        }
        for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) bnxt[i] = 0u;
        __syncthreads();
        const uint32_t nrows = compact ? s_pn : n;
        const bool run = lane < cnt && s_active[lane];
        unsigned long long pc = 0, live_deg = 0;
        uint32_t sup = 0;
        float mx = 0.f, mn = 1.f;
        // Rows are claimed kRowBatch at a time from a shared counter (rows warp * kRowBatch .. first),
        // so a warp that meets a hub row does not hold the others at the round's barrier.  The
        // batch's row ids, offsets, first adjacency chunks and own values are loaded together, so
        // their dependent loads are paid once per batch, not once per row.
        for (uint32_t kb = warp * kRowBatch; kb < nrows;) {
            uint32_t myu = 0, myb = 0, myd = 0;
            if (lane < kRowBatch && kb + lane < nrows) {
                myu = compact ? P[kb + lane] : kb + lane;
                myb = __ldg(p.idx + myu);
                myd = __ldg(p.idx + myu + 1) - myb;
            }
            uint32_t nb0[kRowBatch];
            float own[kRowBatch];
#pragma unroll
            for (int i = 0; i < kRowBatch; ++i) {
                const uint32_t ui = __shfl_sync(kFullMask, myu, i);
                const uint32_t bi = __shfl_sync(kFullMask, myb, i);
                const uint32_t di = __shfl_sync(kFullMask, myd, i);
                const bool has = kb + uint32_t(i) < nrows;
                nb0[i] = has && lane < di ? __ldg(p.adj + bi + lane) : 0u;
                own[i] = has ? cur[size_t(ui) * S + lane] : 0.f;
            }
            unsigned nk = 0;
            if (lane == 0) nk = atomicAdd(&s_next, uint32_t(kRowBatch));
#pragma unroll
            for (int i = 0; i < kRowBatch; ++i) {
            if (kb + uint32_t(i) >= nrows) break;
            const uint32_t u = __shfl_sync(kFullMask, myu, i);
            const uint32_t ub = __shfl_sync(kFullMask, myb, i);
            const uint32_t ud = __shfl_sync(kFullMask, myd, i);
            unsigned long long acc = 0;
            for (uint32_t c = 0; c < ud; c += 32) {
                const uint32_t nb =
                    c == 0 ? nb0[i] : (c + lane < ud ? __ldg(p.adj + ub + c + lane) : 0u);
                // neighbours whose running columns are all zero add nothing: they are dropped, and
                // the live ones compacted into lanes 0 .. popc(live) - 1 (the fixed-point sum does
                // not depend on the order)
                const bool in = c + lane < ud;
                const unsigned live =
                    __ballot_sync(kFullMask, in && ((bcur[nb >> 5] >> (nb & 31)) & 1u));
                const uint32_t nth =
                    lane < uint32_t(__popc(live)) ? __fns(live, 0, int(lane) + 1) : 0u;
                const uint32_t packed = __shfl_sync(kFullMask, nb, nth);
                const uint32_t kk = __popc(live);
                // eight independent 128-byte row loads in flight per step; the last step's loads
                // past kk are predicated off (a zero adds nothing), so a row's remainder costs one
                // load latency, not one per neighbour
                for (uint32_t t = 0; t < kk; t += 8) {
                    float x[8];
#pragma unroll
                    for (int h = 0; h < 8; ++h) {
                        const uint32_t v = __shfl_sync(kFullMask, packed, int((t + h) & 31u));
                        x[h] = t + h < kk ? cur[size_t(v) * S + lane] : 0.f;
                    }
#pragma unroll
                    for (int h = 0; h < 8; ++h) acc += to_fixed(x[h]);
                }
            }
            float r = own[i];
            if (run) {
                r = acc ? from_fixed(acc, ud) : 0.f;
                if (r > 0.f) {
                    pc += ud;
                    ++sup;
                    mx = fmaxf(mx, r);
                    mn = fminf(mn, r);
                }
            }
            const bool running_live = __any_sync(kFullMask, run && r > 0.f);
            const bool any_nz = __any_sync(kFullMask, r != 0.f);
            if (lane == 0) {
                if (running_live) {
                    atomicOr(bnxt + (u >> 5), 1u << (u & 31));
                    live_deg += ud;
                }
                if (any_nz) Ln[atomicAdd(&s_ln, 1u)] = u;
            }
            nxt[size_t(u) * S + lane] = r;
            }
            kb = __shfl_sync(kFullMask, nk, 0);
        }
        if (run) {
            atomicAdd(s_picost + lane, pc);
            atomicAdd(s_support + lane, sup);
            atomicMax(s_max + lane, __float_as_uint(mx));
            atomicMin(s_min + lane, __float_as_uint(mn));
        }
        if (lane == 0 && live_deg) atomicAdd(&s_live_deg, live_deg);
        __syncthreads();
        // ---- preds[row] += (r[src] - r[t]) / ds for every slot of each running source ----
        if (warp < cnt && s_active[warp]) {
            const uint32_t j = warp, src = s_src[j], rb = s_rb[j], dsi = s_ds[j];
            const float ds = float(dsi);
            const float ps = nxt[size_t(src) * S + j];
            for (uint32_t o = lane; o < dsi; o += 32) {
                const uint32_t w = __ldg(p.adj + rb + o);
                p.preds[rb + o] = row_update<float, double>(p.preds[rb + o], ps,
                                                            nxt[size_t(w) * S + j], ds);
            }
            if (lane == 0) ++s_ell[j];
        }
        if (threadIdx.x == 0) {
            s_lp = s_lc;
            s_lc = s_ln;
        }
        __syncthreads();
        float* t = cur;
        cur = nxt;
        nxt = t;
        if (!p.bits && p.cur_smem) {
            // bcur stays in shared memory: take the new round's mask into it
            for (uint32_t i = threadIdx.x; i < words; i += blockDim.x) bcur[i] = bnxt[i];
            __syncthreads();
        } else {
            uint32_t* tb = bcur;
            bcur = bnxt;
            bnxt = tb;
        }
        uint32_t* tl = Lp;
        Lp = Lc;
        Lc = Ln;
        Ln = tl;
        fin ^= 1u;
    }
    // The final columns, transposed into the other buffer: column j becomes n contiguous floats
    // at spare + j * n, so the per-source stage reads its residual vector with unit stride.  Warp
    // w takes tiles of 32 rows; lane l loads row (tile + l) whole (eight 16-byte loads of one
    // 128-byte row) and the 32 stores of the tile (one per column) are each 128 contiguous bytes.
    {
        float* spare = fin ? A : B;
        for (uint32_t t0 = warp * 32u; t0 < n; t0 += nwarp * 32u) {
            const uint32_t u = t0 + lane;
            float v[S];
            if (u < n) {
                const float4* row = reinterpret_cast<const float4*>(cur + size_t(u) * S);
#pragma unroll
                for (int k = 0; k < S / 4; ++k) {
                    const float4 f = row[k];
                    v[4 * k] = f.x;
                    v[4 * k + 1] = f.y;
                    v[4 * k + 2] = f.z;
                    v[4 * k + 3] = f.w;
                }
#pragma unroll
                for (int c = 0; c < S; ++c) spare[size_t(c) * n + u] = v[c];
            }
        }
    }
    if (threadIdx.x == 0) p.final_buf[blockIdx.x] = fin;
    st_pv = warp_sum_u64(st_pv);
    st_tr = warp_sum_u64(st_tr);
    st_rounds = warp_sum_u64(st_rounds);
    if (lane == 0) {
        stat_add(p.stats, kStPushRounds, st_rounds);
        stat_add(p.stats, kStPushVertices, st_pv);
        stat_add(p.stats, kStPushTraversals, st_tr);
    }
}

#include "mixed_push.cuh"

// Sort key of each row for the multi-source push: the row's largest tau if it is listed, else 0.
// A source stops pushing once ell reaches that tau (rwcost = 0 then), so CTAs whose 32 sources
// share a tau bound push for about the same number of rounds.
__global__ void row_key_kernel(const uint32_t* __restrict__ idx, const int* __restrict__ taus,
                               const uint32_t* __restrict__ mark, uint32_t n,
                               uint32_t* __restrict__ key, uint32_t* __restrict__ ids) {
    pdl_wait();  // taus and marks of the tau kernels
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t v = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; v < n;
         v += (gridDim.x * blockDim.x) >> 5) {
        int t = 0;
        if (mark[v]) {
            const uint32_t b = __ldg(idx + v), e = __ldg(idx + v + 1);
            for (uint32_t o = b + lane; o < e; o += 32) t = max(t, __ldg(taus + o));
#pragma unroll
            for (int o = 16; o; o >>= 1) t = max(t, __shfl_xor_sync(kFullMask, t, o));
        }
        if (lane == 0) {
            key[v] = uint32_t(t);
            ids[v] = v;
        }
    }
}

// ---- walks of the block push's sources, as their own launch --------------------------------------
// After a block push the per-source stage leaves each source's walking slots in a queue; this lean
// kernel walks them with many more warps in flight.  Everything a lane computes is what the
// per-source kernel's walk loop computes for the same item:
// an 8-lane group takes one item, lane j walks the item's walks j, j + 8, ... in order over the
// source's residual column, each hop's residual difference added to x in hop order, then the
// group's eight x are summed in lane order into preds[slot] (src/aesc.h:241-391, 524-525).
struct WalkQueueParams {
    const uint32_t* idx;
    const uint32_t* adj;
    const uint32_t* rows;      // list entry -> source
    const float* pre_cols;     // the block push's column blocks
    const uint32_t* pre_final;
    uint32_t list_base;        // first list entry of this wave
    uint32_t n;
    double* preds;
    const WalkItem* items;
    const unsigned* count;     // items in the queue
    unsigned* claim;           // next item (zeroed before the launch)
    unsigned long long* stats;
};
constexpr int kWalkThreads = 256;

__global__ void __launch_bounds__(kWalkThreads, 5) walk_queue_kernel(const WalkQueueParams q) {
    pdl_launch_dependents();
    pdl_wait();  // the queue and the columns of this wave
    const uint32_t lane = threadIdx.x & 31, j = lane & 7, grp = lane >> 3;
    const uint32_t total = *q.count;
    const uint32_t* __restrict__ idx = q.idx;
    const uint32_t* __restrict__ adj = q.adj;
    unsigned long long st_fb = 0;
    bool has = false, start = false, primary = true, done = false;
    WalkItem it{};
    unsigned long long bi = 0;
    uint32_t len = 0, step = 0, cur = 0, cur2 = 0, sec = 0, sec2 = 0, state = 0, src = 0;
    float ds = 0.f;
    const float* pvec = nullptr;
    float x = 0.f, pa = 0.f, pb = 0.f;
    bool pend = false;
    while (true) {
        // a group without an item claims the next one (items with nr = 0 are skipped)
        if (!has && !done) {
            unsigned my = 0;
            if (j == 0) my = atomicAdd(q.claim, 1u);
            my = __shfl_sync(0xffu << (grp * 8), my, int(grp * 8));
            if (my >= total) {
                done = true;
            } else {
                it = q.items[my];
                if (it.nr) {
                    has = true;
                    start = true;
                    bi = 0;
                    x = 0.f;
                    step = uint32_t(0xffffffffull / it.nr);
                    src = __ldg(q.rows + it.pad);
                    ds = float(__ldg(idx + src + 1) - __ldg(idx + src));
                    pvec = pre_column(q.pre_cols, q.pre_final, it.pad - q.list_base, q.n);
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
            double sum = 0;
#pragma unroll
            for (int b = 0; b < 8; ++b) sum += double(__shfl_sync(kFullMask, x, int(grp * 8 + b)));
            if (item_done && j == 0) q.preds[it.pos] += sum / (double(ds) * double(it.nr));
            if (item_done) has = false;
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) st_fb += __shfl_xor_sync(kFullMask, st_fb, o);
    if (lane == 0) stat_add(q.stats, kStFallback, st_fb);
}

// Heavy walk items (at least kHeavyNr walks of at most kHeavyLen hops; a few per wave, which would
// otherwise hold a whole wave for one 8-lane group walking them one bouquet after another; on large
// graphs low-degree sources reach 10^6 walks and more).  One 1,024-thread block per item walks 128
// bouquets at once: thread 8r + j walks walk bi + j of bouquet r (bi = the bouquet's first walk)
// and keeps each hop's residual difference in shared memory; then thread j (the item's lane j)
// adds its walks' differences to x in walk order and hop order -- the adds, values and order of
// walk_queue_kernel's lane j -- and the eight x are summed as there.
constexpr int kHeavyThreads = 1024;
constexpr size_t kHeavySmem = sizeof(float) * kHeavyThreads * (kHeavyLen + 1);

__global__ void __launch_bounds__(kHeavyThreads) heavy_walk_kernel(const WalkQueueParams q,
                                                                   uint32_t cap) {
    extern __shared__ float s_heavy[];
    float (*s_d)[kHeavyLen + 1] = reinterpret_cast<float (*)[kHeavyLen + 1]>(s_heavy);
    __shared__ unsigned s_item;
    pdl_launch_dependents();
    pdl_wait();
    const uint32_t tid = threadIdx.x, lane = tid & 31, j = tid & 7, grp = lane >> 3;
    const uint32_t r = tid >> 3;  // bouquet of the chunk
    const uint32_t total = *q.count;
    const uint32_t* __restrict__ idx = q.idx;
    const uint32_t* __restrict__ adj = q.adj;
    unsigned long long st_fb = 0;
    while (true) {
        if (tid == 0) s_item = atomicAdd(q.claim, 1u);
        __syncthreads();
        const unsigned my = s_item;
        __syncthreads();
        if (my >= total) break;
        const WalkItem it = q.items[cap - 1u - my];
        const uint32_t src = __ldg(q.rows + it.pad);
        const float ds = float(__ldg(idx + src + 1) - __ldg(idx + src));
        const float* pvec = pre_column(q.pre_cols, q.pre_final, it.pad - q.list_base, q.n);
        const uint32_t step = uint32_t(0xffffffffull / it.nr);
        const uint32_t L = it.len;
        float x = 0.f;  // threads 0..7
        for (unsigned long long c0 = 0; c0 < it.nr; c0 += kHeavyThreads) {
            const unsigned long long bi = c0 + 8ull * r;
            const bool active = bi < it.nr;
            uint32_t cur = src, cur2 = it.v;
            uint32_t sec = (uint32_t(bi) + j + 1u) * step, sec2 = sec, state = sec;
            bool primary = true;
            // each hop's residual pair is stored one hop later, after the next hop's row offsets
            // are requested, so the residual loads stay off the walk's chain of dependent loads
            float pa = 0.f, pb = 0.f;
            for (uint32_t h = 0; h < L; ++h) {
                const unsigned z =
                    __ballot_sync(kFullMask, active && primary && (sec == 0u || sec2 == 0u));
                if (active && primary && ((z >> (grp * 8)) & 0xffu)) {
                    primary = false;
                    if (j == 0) ++st_fb;
                }
                if (active) {
                    const uint32_t b1 = __ldg(idx + cur), d1 = __ldg(idx + cur + 1) - b1;
                    const uint32_t b2 = __ldg(idx + cur2), d2 = __ldg(idx + cur2 + 1) - b2;
                    if (h > 0) s_d[tid][h - 1] = rsub(pa, pb);
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
                }
            }
            if (active && L > 0) s_d[tid][L - 1] = rsub(pa, pb);
            __syncthreads();
            if (tid < 8) {
                for (uint32_t b = 0; b < kHeavyThreads / 8 && c0 + 8ull * b < it.nr; ++b)
                    for (uint32_t h = 0; h < L; ++h) x = radd(x, s_d[8 * b + tid][h]);
            }
            __syncthreads();
        }
        if (tid < 32) {
            double sum = 0;
#pragma unroll
            for (int b = 0; b < 8; ++b) sum += double(__shfl_sync(kFullMask, x, b));
            if (tid == 0) q.preds[it.pos] += sum / (double(ds) * double(it.nr));
        }
    }
#pragma unroll
    for (int o = 16; o; o >>= 1) st_fb += __shfl_xor_sync(kFullMask, st_fb, o);
    if (lane == 0) stat_add(q.stats, kStFallback, st_fb);
}

#include "mixed_source.cuh"
#include "gs_source.cuh"

// ---- stage 3: symmetrise (src/aesc.h:532-550) -----------------------------------------------------
// score[q] = p[q] + p[q'] with q' the slot that lands on q (sym_src; none in a row without its
// reverse).  p comes from the source kernel for listed rows, and in closed form for the others:
// after the first round of source s, pvec[s] = 0 and pvec[u] = 1 / deg(u) for each neighbour u, so
// p[s -> u] = 1 / ds + (0 - 1 / deg(u)) / ds in the form's arithmetic.  Those rows' work counters
// (one round, one frontier vertex, ds traversals) are added here.
template <class Real, class Acc>
__device__ __forceinline__ Acc closed_row_score(uint32_t ds, uint32_t du) {
    const Real d = from_u64<Real>(ds);
    const Acc pinit = from_f64<Acc>(__ddiv_rn(1.0, double(d)));
    // the mixed form (FP32 residuals, FP64 scores) forms 1 / deg(u) as its push does
    constexpr bool kMixed = std::is_same<Real, float>::value && std::is_same<Acc, double>::value;
    const Real pu = kMixed ? Real(from_fixed(kFixOne, du)) : rdiv(Real(1), from_u64<Real>(du));
    return row_update<Real, Acc>(pinit, Real(0), pu, d);
}

template <class Real, class Acc>
__global__ void __launch_bounds__(256)
finish_kernel(const Acc* __restrict__ preds, const uint32_t* __restrict__ sym_src,
              const uint32_t* __restrict__ row_of, const uint2* __restrict__ adjd,
              const uint32_t* __restrict__ deg, const uint32_t* __restrict__ mark, uint32_t epoch,
              uint64_t m, float* __restrict__ out, unsigned long long* __restrict__ stats) {
    unsigned long long rows = 0, trav = 0;
    pdl_wait();  // pre-symmetric scores of the source kernel
    for (uint64_t q = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x; q < m;
         q += uint64_t(gridDim.x) * blockDim.x) {
        // first level: the slot's row, its (neighbour, degree) and the slot landing on it
        const uint32_t s = __ldg(row_of + q);
        const uint2 tv = __ldg(adjd + q);
        const uint32_t o = __ldg(sym_src + q);
        const bool first = q == 0 || __ldg(row_of + q - 1) != s;
        // second level, all at once: both rows' marks, both pre-symmetric scores, and the degree of
        // s (the reverse slot's neighbour degree; only graphs without repeated neighbours or
        // self-loops have rows in closed form, every row of the others is listed)
        const uint32_t r = o ? o - 1 : 0;
        const bool ls = __ldg(mark + s) == epoch;
        const bool lt = o && __ldg(mark + tv.x) == epoch;  // slot r lies in row tv.x
        const Acc pq = preds[q];
        const Acc pr = o ? preds[r] : Acc(0);
        const uint32_t ds = o ? __ldg(adjd + r).y : __ldg(deg + s);
        Acc a = ls ? pq : closed_row_score<Real, Acc>(ds, tv.y);
        if (!ls && first) {
            ++rows;
            trav += ds;
        }
        if (o) a = radd(a, lt ? pr : closed_row_score<Real, Acc>(tv.y, ds));
        out[q] = float(a);
    }
    rows = warp_sum_u64(rows);
    trav = warp_sum_u64(trav);
    if ((threadIdx.x & 31) == 0) {
        stat_add(stats, kStPushRounds, rows);
        stat_add(stats, kStPushVertices, rows);
        stat_add(stats, kStPushTraversals, trav);
    }
}

unsigned grid_cap(uint64_t work, int threads, int num_sms, int per_sm) {
    const uint64_t b = (work + threads - 1) / threads;
    return unsigned(std::max<uint64_t>(1, std::min<uint64_t>(b, uint64_t(num_sms) * per_sm)));
}

uint64_t deadline_from_env() {
    double s = 30.0;
    if (const char* e = std::getenv("TGTP_KERNEL_DEADLINE_S")) {
        const double v = std::atof(e);
        if (v > 0) s = v;
    }
    return uint64_t(s * 1e9);
}

// Buffer growth of a run.  A graph captured in a live batch must keep every buffer the batch's
// CUDA graph points at, so a run on it that would need a larger buffer is refused.
void grow(tgtp_graph* g, DeviceBuffer& b, size_t want) {
    if (g->batch_refs > 0 && (!b.ptr || b.bytes < want))
        fail(TGTP_ERR_INVALID_ARGUMENT,
             "this graph belongs to a live batch and the run needs larger buffers than the batch's; "
             "free the batch first");
    b.reserve(want);
}

// Weight tables of the split tau kernel for the configured omega, cached on the graph and formed
// on the device: row 0 = 1 + lambda_i, row k + 1 = lambda_i^(2(k+1)) / (1 - lambda_i) from the
// parity forms' eigen_t_1 table, zero at the indices the reference leaves out (0 and omega - 1)
// and in the padding of each row to a multiple of 64.  FP64 for the FP64 form, FP32 (rounded from
// the FP64 values) for the mixed form.
uint32_t split_pad(uint32_t omega) { return (omega + 63u) & ~63u; }

__global__ void split_tables_kernel(const double* __restrict__ onep, const double* __restrict__ onem,
                                    const double* __restrict__ etab, uint32_t stride,
                                    uint32_t omega, uint32_t wpad, uint32_t total,
                                    double* __restrict__ t64, float* __restrict__ t32) {
    const uint32_t x = blockIdx.x * blockDim.x + threadIdx.x;
    if (x >= total) return;
    const uint32_t k = x / wpad, i = x % wpad;
    double v = 0.0;
    if (i >= 1 && i + 1 < omega)
        v = k == 0 ? onep[i] : __ddiv_rn(etab[size_t(k - 1) * stride + i], onem[i]);
    t64[x] = v;
    t32[x] = __double2float_rn(v);
}

void prepare_split_tables(tgtp_graph* g, uint32_t omega) {
    if (g->split_omega == omega && g->wtab32.ptr && g->wtab64.ptr) return;
    if (g->batch_refs > 0)
        fail(TGTP_ERR_INVALID_ARGUMENT,
             "this graph belongs to a live batch built for another omega; free the batch first");
    const uint32_t rows = 1 + kTauTableRows, wpad = split_pad(omega);
    g->wtab64.reserve(sizeof(double) * rows * wpad);
    g->wtab32.reserve(sizeof(float) * rows * wpad);
    const uint32_t total = rows * wpad;
    split_tables_kernel<<<(total + 255) / 256, 256, 0, g->stream>>>(
        g->onep.as<double>(), g->onem.as<double>(), g->etab.as<double>(), g->omega, omega, wpad,
        total, g->wtab64.as<double>(), g->wtab32.as<float>());
    TGTP_LAUNCH_CHECK("split_tables_kernel");
    g->split_omega = omega;
}

// Graphs with repeated neighbours or self-loops: every row is listed before the tau kernels run
// (so none is scored in closed form, which assumes distinct neighbours and pvec[s] = 0 after the
// first round), and the tau kernels, finding every row marked, append none.
__global__ void list_all_rows_kernel(RowMarks rm, uint32_t n) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x) {
        rm.mark[r] = rm.epoch;
        rm.list[r] = r;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) *rm.len = n;
}

// Row marks of this run: they sit behind the work words in the counter buffer, so the run's one
// zeroing clears them too (a captured run replays correctly), and a marked row holds 1.
RowMarks begin_row_marks(tgtp_graph* g) {
    grow(g, g->row_list, sizeof(uint32_t) * (g->n + 1));
    RowMarks rm;
    rm.mark = run_work(g) + kWorkWords;
    rm.list = g->row_list.as<uint32_t>();
    rm.len = run_work(g) + 2;
    rm.epoch = 1;
    return rm;
}

// Kernel launch on the handle's stream; with pdl the launch may begin while the previous kernel
// finishes (the kernel waits for it with pdl_wait).  TGTP_PDL=0 turns the overlap off.
bool pdl_enabled() {
    static const bool on = [] {
        const char* e = std::getenv("TGTP_PDL");
        return !(e && std::string(e) == "0");
    }();
    return on;
}

template <class... KArgs, class... Args>
void launch(void (*kern)(KArgs...), unsigned grid, unsigned block, size_t smem, cudaStream_t s,
            bool pdl, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = (pdl && pdl_enabled()) ? 1 : 0;
    TGTP_CUDA(cudaLaunchKernelEx(&cfg, kern, std::forward<Args>(args)...));
}

// Symmetrisation of one run (stage 3) on the graph's stream.
template <class Real, class Acc>
void launch_finish(tgtp_graph* g, float* out) {
    ScopedKernel k(g->prof, g->stream, "finish");
    launch(finish_kernel<Real, Acc>, grid_cap(g->m, 256, g->num_sms, 8), 256, 0, g->stream, true,
           g->preds.as<Acc>(), g->sym_src.as<uint32_t>(), g->row_of.as<uint32_t>(),
           g->adjd.as<uint2>(), g->deg.as<uint32_t>(), run_work(g) + kWorkWords, 1u, g->m, out,
           g->stats.as<unsigned long long>());
    TGTP_LAUNCH_CHECK("finish_kernel");
}

}  // namespace

// ---- batched runs: one persistent source kernel over the rows of many graphs --------------------
// While a batch is captured (batch.cu), each run_form of a graph whose per-source stage is one kernel
// (no block push) stops after its tau kernels and leaves that stage and the symmetrisation to the
// batch: the batch joins every graph's branch, launches one persistent source kernel per
// (arithmetic form, residual-vector tier) over the listed rows of all its graphs, then launches
// each graph's finish kernel on the graph's own stream again.  The graphs of a group share one
// per-block scratch laid out for the group's largest graph.
struct BatchEntry {
    tgtp_graph* g;
    float* out;
    int key;    // form_key of the run
    bool smem;  // residual vectors in shared memory
    std::vector<unsigned char> params;  // the run's SourceParams<Real> or MixedParams
};
struct BatchGroup {
    int key;
    bool smem;
    std::vector<size_t> members;  // indices into BatchPlan::entries
    DeviceBuffer scratch, wclean, claims;
};
struct BatchPlan {
    std::vector<BatchEntry> entries;
    std::vector<std::unique_ptr<BatchGroup>> groups;
};
namespace {
thread_local BatchPlan* t_collect = nullptr;

template <class Params>
bool defer_to_batch(tgtp_graph* g, const tgtp_config& cfg, float* out, bool smem, const Params& p) {
    if (!t_collect) return false;
    BatchEntry e;
    e.g = g;
    e.out = out;
    e.key = form_key(cfg);
    e.smem = smem;
    e.params.resize(sizeof(p));
    std::memcpy(e.params.data(), &p, sizeof(p));
    t_collect->entries.push_back(std::move(e));
    return true;
}

// Graphs of more than 22,680 vertices (five bytes a vertex and 1,280 beyond 112 KB, what a warp had
// for its vector when pushes were made by single warps): those whose mixed push is chosen by
// measurement, see learn_push_hint.
bool mixed_push_chosen(uint64_t n) {
    return ((n * 4 + 15) & ~uint64_t(15)) + ((n + 15) & ~uint64_t(15)) + 1280 > uint64_t(112) * 1024;
}
void poll_push_hint(tgtp_graph* g);
void post_push_hint(tgtp_graph* g, int key, double eps);

// How a mixed run pushes.
struct MixedPlan {
    bool block_mode = false, shared_push = false;
    uint32_t block_ctas = 0, wave_cap = 0, waves = 0;
};
MixedPlan plan_mixed(tgtp_graph* g, const tgtp_config& cfg) {
    const uint64_t n = g->n;
    const int key = form_key(cfg);
    MixedPlan p;
    poll_push_hint(g);
    // A block push (the push alone, in waves of listed sources with a claim counter each, then the
    // other stages) or the per-source kernel for all of it: the handle's tuned layout, else
    // TGTP_MIXED_BLOCK, else what the last completed mixed run on this graph at this epsilon showed
    // (push_hint), else the block push on graphs of more than 22,680 vertices at eps <= 0.01.  Scores
    // are the same while no residual rounds to 0 (see round_with_zeros).  learn_push_hint has the
    // figures: the line is the former kernels'.
    if (g->src_layout[key]) p.block_mode = (g->src_layout[key] & kLayoutBlock) != 0;
    else if (const char* e = std::getenv("TGTP_MIXED_BLOCK")) p.block_mode = std::atoi(e) != 0;
    else if (g->push_hint[key] && g->push_hint_eps[key] == cfg.epsilon)
        p.block_mode = g->push_hint[key] == 2;
    else p.block_mode = mixed_push_chosen(n) && cfg.epsilon <= 0.01;
    // Graphs whose sums fit in shared memory push one source per block (push_shared_kernel), all
    // listed sources in waves of at most 4 GiB of residual vectors, or of half the device memory free
    // now (beside what the columns already hold) where that is less, but not below what the 32-source
    // push takes; in a live batch, which pins the columns, of what they hold.  A knob of the 32-source
    // block push asks for that one.  Sparse Chung-Lu graph (n = 25,860), eps = 0.005 / 0.05: push 208 / 109 ms
    // with the 32-source block push (six waves), 79 / 19 ms with this one (its inner loop takes 55 ms of the 79:
    // 21.6e9 additions of two shared atomics each).
    const bool block_knob = std::getenv("TGTP_BLOCK_CTAS") || std::getenv("TGTP_BLOCK_ROUNDS") ||
                            std::getenv("TGTP_BLOCK_MASKS") || std::getenv("TGTP_BLOCK_LIST_DIV");
    p.shared_push = p.block_mode && push_shared_bytes(n) <= size_t(227) * 1024 && !block_knob;
    uint32_t shared_wave =
        uint32_t(std::min<uint64_t>(n, std::max<uint64_t>(1, (uint64_t(4) << 30) / (sizeof(float) * n))));
    const uint64_t held_wave = g->block_cols.bytes / (sizeof(float) * n);
    if (p.shared_push && held_wave < shared_wave) {
        uint64_t wave = held_wave;
        if (g->batch_refs == 0 || wave == 0) {
            size_t free_b = 0, total_b = 0;
            TGTP_CUDA(cudaMemGetInfo(&free_b, &total_b));
            const uint64_t budget = (std::min(free_b, alloc_limit()) + g->block_cols.bytes) / 2;
            wave = std::max<uint64_t>({wave, budget / (sizeof(float) * n), 2 * kBlockCols * uint64_t(g->num_sms)});
        }
        shared_wave = uint32_t(std::min<uint64_t>(shared_wave, wave));
    }
    // CTAs of the 32-source block push: one per SM, within a budget for their residual blocks of 24 GB or
    // half the device memory free now (beside what the blocks already hold), whichever is larger
    // (TGTP_BLOCK_CTAS lowers the count, e.g. to exercise many waves on small graphs)
    p.block_ctas = uint32_t(g->num_sms);
    if (p.block_mode && !p.shared_push) {
        const size_t per_cta = 2 * size_t(n) * kBlockCols * sizeof(float);
        size_t free_b = 0, total_b = 0;
        TGTP_CUDA(cudaMemGetInfo(&free_b, &total_b));
        const size_t budget = std::max(size_t(24) << 30, (free_b + g->block_cols.bytes) / 2);
        p.block_ctas = uint32_t(std::max<size_t>(1, std::min<size_t>(p.block_ctas, budget / per_cta)));
        if (const char* e = std::getenv("TGTP_BLOCK_CTAS"))
            p.block_ctas = std::max(1u, std::min(p.block_ctas, uint32_t(std::atoi(e))));
    }
    p.wave_cap = p.shared_push ? shared_wave : p.block_ctas * kBlockCols;
    p.waves = p.block_mode ? uint32_t((n + uint64_t(p.wave_cap) - 1) / p.wave_cap) : 0u;
    return p;
}

// The per-block "vector is all zero" marks of a run that carves the handle's scratch as `kind` says.
// They hold while the same carving of the same scratch runs again; a run that reads them after
// another one clears them first.  A captured run can be replayed between any two later runs, which
// the host does not see, so it clears them inside the capture, and from then on every run on the
// handle does.
unsigned char* clean_marks(tgtp_graph* g, uint64_t kind, unsigned blocks, bool reads) {
    const uint64_t sig[5] = {kind, blocks, g->n, uint64_t(reinterpret_cast<uintptr_t>(g->scratch.ptr)),
                             uint64_t(g->scratch.bytes)};
    grow(g, g->wclean, blocks + 16);
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    TGTP_CUDA(cudaStreamIsCapturing(g->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) g->captured = true;
    if (reads && (g->captured || std::memcmp(sig, g->wclean_sig, sizeof(sig)) != 0))
        TGTP_CUDA(cudaMemsetAsync(g->wclean.ptr, 0, blocks + 16, g->stream));
    std::memcpy(g->wclean_sig, sig, sizeof(sig));
    return g->wclean.as<unsigned char>();
}

// Blocks of the mixed form's per-source kernel in one of its modes over up to n vertices.
struct MixedLayout {
    unsigned blocks, threads;
    size_t smem, list_bytes, item_bytes, sum_bytes, touched_bytes, bit_bytes;
    size_t scratch() const { return list_bytes + item_bytes + sum_bytes + touched_bytes + bit_bytes + 256; }
};
template <class Pack>
const void* mixed_kernel(int mode) {
    return mode == kShared   ? reinterpret_cast<const void*>(mixed_source_kernel<kShared, Pack>)
           : mode == kGlobal ? reinterpret_cast<const void*>(mixed_source_kernel<kGlobal, Pack>)
                             : reinterpret_cast<const void*>(mixed_source_kernel<kColumn, Pack>);
}
template <class Pack>
MixedLayout mixed_layout(int mode, uint64_t n, uint64_t max_degree, uint64_t rows, int num_sms) {
    MixedLayout l;
    l.smem = mixed_shared_bytes(mode, n);
    // about 1,024 resident threads per SM (64 registers each): as many sources at once as shared
    // memory holds vectors of; in HBM two.  Threads per block in HBM, Chung-Lu n = 200,000 / 60,000,
    // eps = 0.05, ms: 128 166 / 12.6, 256 143.9 / 11.6, 512 143.5 / 10.9, 1,024 158 / 15.2 (fewer
    // sources at once wait for each other's barriers, more push each other's words out of L2)
    if (mode == kShared)
        l.threads = l.smem > size_t(113) * 1024  ? 1024u
                    : l.smem > size_t(56) * 1024 ? 512u
                    : l.smem > size_t(28) * 1024 ? 256u
                                                 : 128u;
    else
        l.threads = mode == kGlobal ? 512u : 256u;
    const int per_sm = blocks_per_sm(mixed_kernel<Pack>(mode), int(l.threads), l.smem);
    if (per_sm < 1) fail(TGTP_ERR_UNSUPPORTED, "source kernel does not fit on an SM");
    l.blocks = unsigned(std::max<uint64_t>(1, std::min<uint64_t>(uint64_t(num_sms) * per_sm, rows)));
    auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
    l.list_bytes = mode == kColumn ? 0 : align(sizeof(uint4) * size_t(n) * l.blocks);
    l.item_bytes = align(sizeof(WalkItem) * std::max<uint64_t>(max_degree, 1) * l.blocks);
    l.sum_bytes = mode == kGlobal ? align(sizeof(unsigned long long) * size_t(n) * l.blocks) : 0;
    l.touched_bytes = mode == kGlobal ? align(sizeof(uint32_t) * size_t(n) * l.blocks) : 0;
    // the bitmap in HBM: beyond kBitsInSmem, or as TGTP_BLOCK_MASKS=global asks (kShared: always)
    const char* masks = std::getenv("TGTP_BLOCK_MASKS");
    const bool gbits = mode == kShared || (mode == kGlobal && (4 * mixed_words(n) > kBitsInSmem ||
                                                               (masks && std::string(masks) == "global")));
    l.bit_bytes = gbits ? align(4 * mixed_words(n) * l.blocks) : 0;
    return l;
}
void carve_mixed(MixedParams& p, const MixedLayout& l, unsigned char* base, uint64_t n, uint64_t max_degree) {
    p.scratch_n = uint32_t(n);
    p.max_degree = uint32_t(std::max<uint64_t>(max_degree, 1));
    p.lists = l.list_bytes ? reinterpret_cast<uint4*>(base) : nullptr;
    base += l.list_bytes;
    p.items = reinterpret_cast<WalkItem*>(base);
    base += l.item_bytes;
    p.sums = l.sum_bytes ? reinterpret_cast<unsigned long long*>(base) : nullptr;
    base += l.sum_bytes;
    p.touched = l.touched_bytes ? reinterpret_cast<uint32_t*>(base) : nullptr;
    base += l.touched_bytes;
    p.gbits = l.bit_bytes ? reinterpret_cast<uint32_t*>(base) : nullptr;
}
template <class Pack>
void launch_mixed(int mode, const MixedLayout& l, cudaStream_t s, bool pdl, const Pack& pk) {
    if (mode == kShared) launch(mixed_source_kernel<kShared, Pack>, l.blocks, l.threads, l.smem, s, pdl, pk);
    else if (mode == kGlobal) launch(mixed_source_kernel<kGlobal, Pack>, l.blocks, l.threads, l.smem, s, pdl, pk);
    else launch(mixed_source_kernel<kColumn, Pack>, l.blocks, l.threads, l.smem, s, pdl, pk);
    TGTP_LAUNCH_CHECK("mixed_source_kernel");
}

// Per-source stage of the mixed form; false when it is left to a batch.
bool run_mixed(tgtp_graph* g, const tgtp_config& cfg, float* out, const RowMarks& rm, const MixedPlan& mp,
               double logmd) {
    cudaStream_t s = g->stream;
    const uint64_t n = g->n, m = g->m;
    const int key = form_key(cfg);
    auto* stats = g->stats.as<unsigned long long>();
    auto* work = run_work(g);
    // sums in shared memory while they fit (the tuned layout's tier, else TGTP_PVEC_TIER)
    int mode = kColumn;
    if (!mp.block_mode) {
        bool shared = mixed_fits_shared(n);
        if (g->src_layout[key]) shared = shared && (g->src_layout[key] & kLayoutSmem) != 0;
        else if (const char* t = std::getenv("TGTP_PVEC_TIER")) shared = shared && std::string(t) != "global";
        mode = shared ? kShared : kGlobal;
    }
    const MixedLayout lay = mixed_layout<MixedPack<1>>(mode, n, g->max_degree, n, g->num_sms);
    grow(g, g->scratch, lay.scratch());
    MixedParams p{};
    carve_mixed(p, lay, g->scratch.as<unsigned char>(), n, g->max_degree);
    p.idx = g->idx.as<uint32_t>();
    p.adj = g->adj.as<uint32_t>();
    p.adjd = g->adjd.as<uint2>();
    p.dinv = g->dinv.as<double>();
    p.n = uint32_t(n);
    p.taus = g->taus.as<int>();
    p.preds = g->preds.as<double>();
    p.work = work;
    p.rows = rm.list;
    p.eps = cfg.epsilon;
    p.logmd = logmd;
    p.gamma = cfg.gamma;
    p.stats = stats;
    p.budget_ns = deadline_from_env();
    if (g->trace_on) {
        grow(g, g->trace, sizeof(uint32_t) * (m + n));
        TGTP_CUDA(cudaMemsetAsync(g->trace.ptr, 0, sizeof(uint32_t) * (m + n), s));
        p.trace_nr = g->trace.as<uint32_t>();
        p.trace_ell = p.trace_nr + m;
        g->trace_valid = true;
    }
    MixedPack<1> pk;
    pk.count = 1;
    if (!mp.block_mode) {
        p.claim = work;
        if (defer_to_batch(g, cfg, out, mode == kShared, p)) return false;
    }
    const uint64_t carving = uint64_t(key) | (uint64_t(mode) << 8) | (uint64_t(lay.bit_bytes != 0) << 16);
    p.clean = clean_marks(g, carving | (uint64_t(1) << 63), lay.blocks, mode == kGlobal);
    if (!mp.block_mode) {
        pk.g[0] = p;
        ScopedKernel k(g->prof, s, "source");
        launch_mixed(mode, lay, s, true, pk);
        return true;
    }
    grow(g, g->block_pre, sizeof(PrePush) * (n + 1));
    PushBlockParams bp;
    PushSharedParams sp;
    size_t bsm = 0;
    unsigned push_blocks = mp.block_ctas;
    unsigned push_threads = 1024u;
    if (mp.shared_push) {
        // the block's threads by its shared memory: 1,024 resident threads per SM
        bsm = push_shared_bytes(n);
        push_threads = bsm > size_t(113) * 1024 ? 1024u : (bsm > size_t(56) * 1024 ? 512u : 256u);
        const int per_sm =
            blocks_per_sm(reinterpret_cast<const void*>(push_shared_kernel), int(push_threads), bsm);
        if (per_sm < 1) fail(TGTP_ERR_UNSUPPORTED, "block push does not fit on an SM");
        push_blocks = unsigned(std::min<uint64_t>(uint64_t(g->num_sms) * per_sm, mp.wave_cap));
        grow(g, g->block_cols, sizeof(float) * size_t(n) * mp.wave_cap);
        grow(g, g->block_lists, sizeof(uint4) * size_t(n) * push_blocks + 16);
        sp.idx = p.idx;
        sp.adj = p.adj;
        sp.adjd = p.adjd;
        sp.dinv = g->dinv.as<double>();
        sp.n = uint32_t(n);
        sp.taus = p.taus;
        sp.preds = p.preds;
        sp.work = work;
        sp.eps = cfg.epsilon;
        sp.logmd = logmd;
        sp.lists = g->block_lists.as<uint4>();
        sp.cols = g->block_cols.as<float>();
        sp.pre = g->block_pre.as<PrePush>();
        sp.stats = stats;
        sp.budget_ns = p.budget_ns;
        sp.cap = mp.wave_cap;
    } else {
        grow(g, g->block_cols, 2 * size_t(n) * kBlockCols * sizeof(float) * mp.block_ctas);
        grow(g, g->block_final, sizeof(uint32_t) * (mp.block_ctas + 1));
        bp.idx = p.idx;
        bp.adj = p.adj;
        bp.deg = g->deg.as<uint32_t>();
        bp.adjd = p.adjd;
        bp.n = uint32_t(n);
        bp.taus = p.taus;
        bp.preds = p.preds;
        bp.work = work;
        bp.rows = rm.list;
        bp.eps = cfg.epsilon;
        bp.logmd = logmd;
        bp.cols = g->block_cols.as<float>();
        bp.final_buf = g->block_final.as<uint32_t>();
        bp.pre = g->block_pre.as<PrePush>();
        bp.stats = stats;
        bp.budget_ns = p.budget_ns;
        // three row masks in shared memory while they fit beside the kernel's static 1.5 KB, else
        // the current round's mask alone (n up to about 1.6 million), else none; the others in
        // global memory; four row lists of n entries per CTA.  TGTP_BLOCK_MASKS=global|cur picks
        // the placement of larger graphs on small ones.
        const size_t mask_bytes = sizeof(uint32_t) * ((size_t(n) + 31) / 32);
        const size_t bits_bytes = 3 * mask_bytes;
        bp.bits = bits_bytes <= size_t(200) * 1024;
        bp.cur_smem = !bp.bits && mask_bytes <= size_t(200) * 1024;
        if (const char* e = std::getenv("TGTP_BLOCK_MASKS")) {
            if (std::string(e) == "global") bp.bits = bp.cur_smem = false;
            else if (std::string(e) == "cur") {
                bp.bits = false;
                bp.cur_smem = true;
            }
        }
        bsm = bp.bits ? bits_bytes : (bp.cur_smem ? mask_bytes : 0);
        if (!bp.bits) grow(g, g->block_bits, bits_bytes * mp.block_ctas + 16);
        bp.gbits = bp.bits ? nullptr : g->block_bits.as<uint32_t>();
        grow(g, g->block_lists, sizeof(uint32_t) * 4 * size_t(n) * mp.block_ctas + 16);
        bp.lists = g->block_lists.as<uint32_t>();
        bp.m = m;
        // a round is compacted when its live rows' degree sum is below m / list_div (the tuned
        // layout's threshold, else TGTP_BLOCK_LIST_DIV, else 4); TGTP_BLOCK_ROUNDS=compact|full
        // fixes the choice (the values do not depend on it)
        bp.list_div = layout_list_div(g->src_layout[key]);
        if (const char* e = std::getenv("TGTP_BLOCK_LIST_DIV"))
            if (!g->src_layout[key]) bp.list_div = uint32_t(std::atoi(e));
        bp.rounds_mode = bp.list_div == 0 ? 2 : 0;
        if (const char* e = std::getenv("TGTP_BLOCK_ROUNDS")) {
            if (std::string(e) == "compact") bp.rounds_mode = 1;
            else if (std::string(e) == "full") bp.rounds_mode = 2;
        }
        if (bsm) (void)blocks_per_sm(reinterpret_cast<const void*>(push_block_kernel), 1024, bsm);
    }
    p.pre = g->block_pre.as<PrePush>();
    p.pre_cols = g->block_cols.as<float>();
    p.pre_final = mp.shared_push ? nullptr : g->block_final.as<uint32_t>();
    // the listed rows ordered by their largest tau (unlisted rows sort last, key 0)
    grow(g, g->block_keys, sizeof(uint32_t) * 4 * (n + 1));
    uint32_t* rkey = g->block_keys.as<uint32_t>();
    uint32_t* ids = rkey + (n + 1);
    uint32_t* skey = ids + (n + 1);
    uint32_t* sorted = skey + (n + 1);
    size_t tbytes = 0;
    TGTP_CUDA(cub::DeviceRadixSort::SortPairsDescending(nullptr, tbytes, rkey, skey, ids, sorted,
                                                        int(n), 0, 32, s));
    grow(g, g->block_tmp, tbytes + 16);
    {
        ScopedKernel k(g->prof, s, "row_key");
        launch(row_key_kernel, grid_cap(uint64_t(n) * 32, 256, g->num_sms, 8), 256u, size_t(0), s,
               true, g->idx.as<uint32_t>(), g->taus.as<int>(), rm.mark, uint32_t(n), rkey, ids);
        TGTP_LAUNCH_CHECK("row_key_kernel");
    }
    TGTP_CUDA(cub::DeviceRadixSort::SortPairsDescending(g->block_tmp.ptr, tbytes, rkey, skey, ids,
                                                        sorted, int(n), 0, 32, s));
    bp.rows = sp.rows = sorted;
    p.rows = sorted;
    unsigned* claims = work + kWorkWords + n + 1;
    // the walks of each wave's sources: a queue of (slot, its source's list entry) items that
    // walk_queue_kernel works through (a wave's sources hold at most m slots), and per wave a
    // queue length and a claim counter
    grow(g, g->walk_queue, sizeof(WalkItem) * (m + 1));
    grow(g, g->walk_ctl, sizeof(unsigned) * 4 * (mp.waves + 1));
    unsigned* ctl = g->walk_ctl.as<unsigned>();
    TGTP_CUDA(cudaMemsetAsync(ctl, 0, sizeof(unsigned) * 4 * (mp.waves + 1), s));
    p.walk_queue = g->walk_queue.as<WalkItem>();
    p.walk_cap = uint32_t(m + 1);
    WalkQueueParams wq;
    wq.idx = p.idx;
    wq.adj = p.adj;
    wq.rows = sorted;
    wq.pre_cols = p.pre_cols;
    wq.pre_final = p.pre_final;
    wq.n = uint32_t(n);
    wq.preds = p.preds;
    wq.items = p.walk_queue;
    wq.stats = stats;
    const int walk_per_sm =
        blocks_per_sm(reinterpret_cast<const void*>(walk_queue_kernel), kWalkThreads, 0);
    const unsigned walk_blocks = unsigned(g->num_sms) * unsigned(std::max(walk_per_sm, 1));
    const int heavy_per_sm = blocks_per_sm(reinterpret_cast<const void*>(heavy_walk_kernel),
                                           kHeavyThreads, kHeavySmem);
    const unsigned heavy_blocks = unsigned(g->num_sms) * unsigned(std::max(heavy_per_sm, 1));
    // These kernels run for milliseconds each, and the next one's blocks started early take slots
    // from them: without programmatic dependent launch the whole run on the sparse Chung-Lu graph
    // (n = 25,860, eps = 0.005) takes 95 ms, with it 109 ms.
    for (uint32_t w = 0; w < mp.waves; ++w) {
        bp.base = sp.base = w * mp.wave_cap;
        {
            ScopedKernel k(g->prof, s, "push_block");
            if (mp.shared_push) {
                sp.claim = claims + mp.waves + w;
                launch(push_shared_kernel, push_blocks, push_threads, bsm, s, false, sp);
            } else {
                launch(push_block_kernel, mp.block_ctas, 1024u, bsm, s, false, bp);
            }
            TGTP_LAUNCH_CHECK("push_block_kernel");
        }
        p.claim = claims + w;
        p.list_base = bp.base;
        p.list_cap = mp.wave_cap;
        p.walk_count = ctl + 4 * w;
        pk.g[0] = p;
        {
            ScopedKernel k(g->prof, s, "source");
            launch(mixed_source_kernel<kColumn, MixedPack<1>>, lay.blocks, lay.threads, lay.smem, s, false, pk);
            TGTP_LAUNCH_CHECK("mixed_source_kernel");
        }
        wq.list_base = p.list_base;
        wq.count = ctl + 4 * w;
        wq.claim = ctl + 4 * w + 1;
        {
            ScopedKernel k(g->prof, s, "walk_queue");
            launch(walk_queue_kernel, walk_blocks, unsigned(kWalkThreads), size_t(0), s, false, wq);
            TGTP_LAUNCH_CHECK("walk_queue_kernel");
        }
        WalkQueueParams wh = wq;
        wh.count = ctl + 4 * w + 2;
        wh.claim = ctl + 4 * w + 3;
        ScopedKernel k(g->prof, s, "heavy_walk");
        launch(heavy_walk_kernel, heavy_blocks, unsigned(kHeavyThreads), kHeavySmem, s, false, wh,
               uint32_t(m + 1));
        TGTP_LAUNCH_CHECK("heavy_walk_kernel");
    }
    return true;
}

// Blocks of the FP32 / FP64 forms' per-source kernel over up to n vertices.
struct GsLayout {
    unsigned blocks, threads;
    size_t smem, q_bytes, item_bytes, vec_bytes;
    size_t scratch() const { return q_bytes + item_bytes + vec_bytes + 256; }
};
template <class Real, class Pack>
GsLayout gs_layout(bool use_smem, uint64_t n, uint64_t max_degree, uint64_t rows, int num_sms) {
    GsLayout l;
    l.threads = unsigned(use_smem ? GsShape<Real, true>::kThreads : GsShape<Real, false>::kThreads);
    l.smem = gs_shared_bytes<Real>(use_smem, n);
    const void* kern = use_smem ? reinterpret_cast<const void*>(source_kernel<Real, true, Pack>)
                                : reinterpret_cast<const void*>(source_kernel<Real, false, Pack>);
    int per_sm = blocks_per_sm(kern, int(l.threads), l.smem);
    if (per_sm < 1) fail(TGTP_ERR_UNSUPPORTED, "source kernel does not fit on an SM");
    // Small vectors: where registers and not shared memory limit the 128-thread blocks and there are
    // sources for more than one round of them, blocks of half the threads, so that more sources push
    // at a time (FP64, eps = 0.005: n = 2,000, 20 neighbours 2.81 ms against 3.13; n = 1,000, 14 and 6
    // neighbours, 888 blocks of 128 threads or all sources at once, 1.13 against 1.39 and 4.27 against
    // 6.03; n = 600, one round, 0.626 against 0.610; at n = 5,500, shared memory the limit, 17.3 against
    // 16.7).
    if (use_smem && rows > uint64_t(num_sms) * per_sm) {
        const int half = blocks_per_sm(kern, int(l.threads) / 2, l.smem);
        if (half > per_sm) {
            l.threads /= 2;
            per_sm = half;
        }
    }
    // vectors and lists in HBM: eight blocks per SM where more would take over 16 GB
    if (!use_smem && uint64_t(num_sms) * per_sm * n * (8 + sizeof(Real)) > (uint64_t(16) << 30))
        per_sm = std::min(per_sm, 8);
    l.blocks = unsigned(std::max<uint64_t>(1, std::min<uint64_t>(uint64_t(num_sms) * per_sm, rows)));
    auto align = [](size_t x) { return (x + 255) & ~size_t(255); };
    l.q_bytes = align(size_t(l.blocks) * 2 * size_t(n) * 4);
    l.item_bytes = align(size_t(l.blocks) * std::max<uint64_t>(max_degree, 1) * sizeof(WalkItem));
    l.vec_bytes = use_smem ? 0 : align(size_t(l.blocks) * size_t(n) * sizeof(Real));
    return l;
}
template <class Real>
void carve_gs(SourceParams<Real>& p, const GsLayout& l, unsigned char* base, uint64_t n, uint64_t max_degree) {
    p.scratch_n = uint32_t(n);
    p.max_degree = uint32_t(std::max<uint64_t>(max_degree, 1));
    p.qbuf = reinterpret_cast<uint32_t*>(base);
    base += l.q_bytes;
    p.items = reinterpret_cast<WalkItem*>(base);
    base += l.item_bytes;
    p.pvec_g = l.vec_bytes ? reinterpret_cast<Real*>(base) : nullptr;
}
template <class Real, class Pack>
void launch_gs(bool use_smem, const GsLayout& l, cudaStream_t s, bool pdl, const Pack& pk) {
    if (use_smem) launch(source_kernel<Real, true, Pack>, l.blocks, l.threads, l.smem, s, pdl, pk);
    else launch(source_kernel<Real, false, Pack>, l.blocks, l.threads, l.smem, s, pdl, pk);
    TGTP_LAUNCH_CHECK("source_kernel");
}

// Largest shared memory of a block that keeps its residual vector there by default.  Shared memory
// shortens a step of the push and limits the sources in flight; the HBM tier's windowed push gains
// on it as rows get shorter.  Measured, shared memory against HBM, in ms:
//   44 neighbours  FP64  51 KB 1.55 / 1.73,  63 KB 2.53 / 2.31;  FP32  55 KB 3.12 / 3.77
//   30             FP64  31 KB 1.73 / 2.62,  51 KB 4.35 / 4.94
//   20             FP64  23 KB 2.81 / 3.12,  39 KB 8.31 / 8.30,  51 KB 16.7 / 12.8
//                  FP32  31 KB 5.43 / 6.89,  39 KB 7.56 / 8.83,  51 KB 12.7 / 12.8
//   15, 14         FP64  23 KB 2.78 / 2.95,  35 KB 7.91 / 7.18;  FP32  21 KB 4.34 / 4.94,  35 KB 12.7 / 12.1
//   9.5            FP64  19 KB 2.03 / 2.24,  39 KB 8.55 / 7.19
inline size_t gs_smem_most(uint64_t n, uint64_t m) {
    return size_t(m >= 24 * n ? 56 : m >= 18 * n ? 40 : 24) * 1024;
}

// Per-source stage of the FP32 and FP64 forms; false when it is left to a batch.
template <class Real>
bool run_sources(tgtp_graph* g, const tgtp_config& cfg, float* out, const RowMarks& rm, bool multi, double logmd) {
    cudaStream_t s = g->stream;
    const uint64_t n = g->n, m = g->m;
    const int key = form_key(cfg);
    const uint16_t lay = g->src_layout[key];
    // Shared-memory tier: the residual vector in shared memory; HBM tier: in HBM.  The tuned
    // layout's, else shared memory while a block takes at most gs_smem_most; TGTP_PVEC_TIER=smem|global
    // overrides the rule.
    const size_t smem = gs_shared_bytes<Real>(true, n);
    const bool fits = smem + 512 <= size_t(227) * 1024;
    bool use_smem = smem <= gs_smem_most(n, m);
    if (lay) use_smem = fits && (lay & kLayoutSmem) != 0;
    else if (const char* t = std::getenv("TGTP_PVEC_TIER")) {
        if (std::string(t) == "global") use_smem = false;
        else if (std::string(t) == "smem" && fits) use_smem = true;
    }
    using Pack1 = SourcePack<Real, 1>;
    const GsLayout l = gs_layout<Real, Pack1>(use_smem, n, g->max_degree, n, g->num_sms);
    grow(g, g->scratch, l.scratch());
    SourceParams<Real> p{};
    carve_gs(p, l, g->scratch.as<unsigned char>(), n, g->max_degree);
    p.idx = g->idx.as<uint32_t>();
    p.adj = g->adj.as<uint32_t>();
    p.adjd = g->adjd.as<uint2>();
    p.dinv = g->dinv.as<double>();
    p.n = uint32_t(n);
    p.taus = g->taus.as<int>();
    p.preds = g->preds.as<Real>();
    p.work = run_work(g);
    p.rows = rm.list;
    p.eps = cfg.epsilon;
    p.logmd = logmd;
    p.gamma = cfg.gamma;
    p.stats = g->stats.as<unsigned long long>();
    p.budget_ns = deadline_from_env();
    p.multi = multi;
    if (g->trace_on) {
        grow(g, g->trace, sizeof(uint32_t) * (m + n));
        TGTP_CUDA(cudaMemsetAsync(g->trace.ptr, 0, sizeof(uint32_t) * (m + n), s));
        p.trace_nr = g->trace.as<uint32_t>();
        p.trace_ell = p.trace_nr + m;
        g->trace_valid = true;
    }
    {
        // The windowed push pays off when rows are short: several frontier vertices share a 32-entry
        // step.  With long rows each vertex fills its steps anyway and adjacent frontier vertices cut
        // windows often.  In shared memory the line is at 15 neighbours (one vertex at a time /
        // windowed, ms: 9.5 neighbours 2.96 / 2.02; 14: 3.04 / 2.78; 16: 2.37 / 2.39; 20: 2.81 / 3.17;
        // 44: 0.73 / 1.42), in HBM, where a step waits for its words, at 32 (20: 18.7 / 12.8; 30:
        // 5.18 / 4.94; 44: 1.73 / 2.44).  Where two vertices are neighbours with a chance of 1 in 25 or
        // more, half of the windows of eight are cut and it does not pay (n = 150, 6 neighbours: FP64
        // 0.305 / 0.336, FP32 0.289 / 0.346; n = 150, 12: FP64 0.187 / 0.324; n = 300, 12: FP64 0.63 / 0.84,
        // FP32 0.59 / 0.85; at 1 in 50, n = 300, 6 neighbours: FP64 1.05 / 0.88, FP32 0.96 / 0.88).  The tuned
        // layout, then TGTP_GS_WINDOW=0/1, override the rule.
        const char* e = std::getenv("TGTP_GS_WINDOW");
        if (lay & kLayoutWindow) p.gs_window = true;
        else if (lay & kLayoutNoWindow) p.gs_window = false;
        else if (e) p.gs_window = std::string(e) != "0";
        else p.gs_window = m < (use_smem ? 15 : 32) * n && 25 * m < n * n;
    }
    p.claim = run_work(g);
    if (defer_to_batch(g, cfg, out, use_smem, p)) return false;
    p.clean = clean_marks(g, uint64_t(key) | (uint64_t(use_smem) << 8) | (uint64_t(1) << 62), l.blocks, !use_smem);
    Pack1 pk;
    pk.count = 1;
    pk.g[0] = p;
    ScopedKernel k(g->prof, s, "source");
    launch_gs<Real>(use_smem, l, s, true, pk);
    return true;
}

// One tgtp() run.  Real = residual type, MIXED = the mixed form (scores accumulated in FP64), Vec =
// eigenvector storage of the split tau kernels.
template <class Real, bool MIXED, class Vec>
void run_form(tgtp_graph* g, const tgtp_config& cfg, float* out) {
    using Acc = typename std::conditional<MIXED, double, Real>::type;
    cudaStream_t s = g->stream;
    const uint64_t n = g->n, m = g->m;
    const uint32_t omega = uint32_t(cfg.omega);
    // host-side constants with the host libm (as the reference evaluates them)
    TauConst c;
    const double l1 = g->values[1], l2 = g->values[omega - 1];
    c.one_m_l1sq = 1.0 - (l1 * l1);
    c.b1 = std::log(double(1.0) / std::fabs(l1));
    c.one_m_l2sq = 1.0 - (l2 * l2);
    c.b2 = std::log(double(1.0) / std::fabs(l2));
    const double logmd = std::log(double(m) / cfg.delta);

    grow(g, g->taus, sizeof(int) * (m + 1));
    grow(g, g->preds, sizeof(Acc) * (m + 1));
    // one zeroing for the striped counters, the work words and the row marks behind them
    const size_t stat_bytes = sizeof(unsigned long long) * kStCount * kStStripes;
    const int key = form_key(cfg);
    MixedPlan mp;
    if (MIXED) mp = plan_mixed(g, cfg);
    g->last_key = key;
    g->last_eps = cfg.epsilon;
    const size_t zero_bytes = stat_bytes + sizeof(unsigned) * (kWorkWords + n + 1 + 2 * size_t(mp.waves));
    grow(g, g->stats, zero_bytes);
    auto* stats = g->stats.as<unsigned long long>();
    auto* work = run_work(g);
    const bool multi = !MIXED && g->has_multi_edges;
    const char* bulk_env = std::getenv("TGTP_TAU_BULK");
    const bool want_bulk = bulk_env && std::atoi(bulk_env) == 1;
    // tau_sums_kernel, where it runs first, zeroes them on its way (a launch less: 30.5 -> 27 us for
    // a call on the 4,039-vertex graph, FP64, eps = 0.05)
    const bool zero_in_sums = (MIXED || std::is_same<Real, double>::value) && !multi && !want_bulk;
    if (!zero_in_sums) TGTP_CUDA(cudaMemsetAsync(stats, 0, zero_bytes, s));

    const RowMarks rm = begin_row_marks(g);
    if (multi) {
        // the reference leaves tau = 0 in the slots no forward edge writes (the later repeats of
        // a neighbour u < v in row v, src/aesc.h:179-209), and every row goes to the source kernel
        TGTP_CUDA(cudaMemsetAsync(g->taus.ptr, 0, sizeof(int) * m, s));
        list_all_rows_kernel<<<grid_cap(n, 256, g->num_sms, 8), 256, 0, s>>>(rm, uint32_t(n));
        TGTP_LAUNCH_CHECK("list_all_rows_kernel");
    }
    if constexpr (MIXED || std::is_same<Real, double>::value) {
        // FP64 and mixed forms: eight lanes per edge over F64 / F32 / BF16 rows
        prepare_split_tables(g, omega);
        using Part = typename Split<Vec>::Part;
        const Vec* vec = std::is_same<Vec, double>::value ? (const Vec*)g->vec_f64.ptr
                         : std::is_same<Vec, float>::value ? (const Vec*)g->vec_f32.ptr
                                                           : (const Vec*)g->vec_bf16.ptr;
        const Part* wtab = std::is_same<Part, double>::value ? (const Part*)g->wtab64.ptr
                                                             : (const Part*)g->wtab32.ptr;
        const uint32_t wpad = split_pad(omega);
        const size_t ssmem = 2 * sizeof(Part) * wpad;
        BoundArgs<Vec> ba;
        ba.deg = g->deg.as<uint32_t>();
        ba.vec = vec;
        ba.stride = g->omega;
        ba.omega = omega;
        ba.wtab = wtab;
        ba.wpad = wpad;
        ba.etabd = g->etab.as<double>();
        ba.onem = g->onem.as<double>();
        ba.eps_half = cfg.epsilon / 2.0;
        ba.mdbl = double(m);
        ba.c = c;
        ba.taus = g->taus.as<int>();
        ba.rm = rm;
        {
            const int per_sm =
                blocks_per_sm(reinterpret_cast<const void*>(tau_sums_kernel<Vec>), kSumsThreads, ssmem);
            if (per_sm < 1) fail(TGTP_ERR_UNSUPPORTED, "omega too large for the tau kernel");
            grow(g, g->tau_sums, sizeof(double2) * (g->num_forward + 1));
            constexpr uint64_t kStep = kSumsThreads / 8 * kSumsEdges;  // edges per block and step
            const uint64_t need = (g->num_forward + kStep - 1) / kStep;
            const unsigned blocks = unsigned(std::max<uint64_t>(
                1, std::min<uint64_t>(need, uint64_t(g->num_sms) * per_sm)));
            // TGTP_TAU_BULK=1: the bulk-copy pipeline instead of the gather (rows whose bytes are a
            // multiple of 16, with a row stride that keeps them aligned).  On the 4,039-vertex graph
            // it measured 0.056 ms per FP64 step against the gather's 0.046: the rows are
            // L2-resident, so the gather's 32 warps per SM hide the latency better than six
            // pipelined warps, and the bulk copies fetch each edge's u row again.
            const bool bulk = want_bulk &&
                              (size_t(omega) * sizeof(Vec)) % 16 == 0 &&
                              (size_t(g->omega) * sizeof(Vec)) % 16 == 0;
            constexpr int WPB = BulkShape<Vec>::WPB;
            const size_t bsmem = size_t(WPB) * (size_t(kBulkStages) * 8 * omega * sizeof(Vec) +
                                                kBulkStages * 8) + ssmem;
            const int bper_sm = bulk ? blocks_per_sm(
                reinterpret_cast<const void*>(tau_sums_bulk_kernel<Vec>), 32 * WPB, bsmem) : 0;
            if (bulk && bper_sm >= 1) {
                const uint64_t bneed = (g->num_forward + 4 * WPB - 1) / (4 * WPB);
                const unsigned bblocks = unsigned(std::max<uint64_t>(
                    1, std::min<uint64_t>(bneed, uint64_t(g->num_sms) * bper_sm)));
                ScopedKernel k(g->prof, s, "tau_sums");
                launch(tau_sums_bulk_kernel<Vec>, bblocks, unsigned(32 * WPB), bsmem, s, false,
                       g->fedge.as<uint4>(), g->num_forward, vec, g->omega, omega, wtab, wpad,
                       g->tau_sums.as<double2>(), work);
                TGTP_LAUNCH_CHECK("tau_sums_bulk_kernel");
            } else {
                ScopedKernel k(g->prof, s, "tau_sums");
                launch(tau_sums_kernel<Vec>, blocks, unsigned(kSumsThreads), ssmem, s, false,
                    g->fedge.as<uint4>(), g->num_forward, vec, g->omega, omega, wtab, wpad,
                    g->tau_sums.as<double2>(), reinterpret_cast<uint32_t*>(stats),
                    zero_in_sums ? uint64_t(zero_bytes / sizeof(uint32_t)) : uint64_t(0));
                TGTP_LAUNCH_CHECK("tau_sums_kernel");
            }
            ScopedKernel k(g->prof, s, "tau_bound");
            // Edges per warp: a further delta sweep serves four of a warp's edges at a time, one round
            // after another, so graphs with few edges spread them over more warps (12,000 edges, most
            // with a second sweep: 32 a warp 29 us, 16 19, 8 16, 4 15; 29,700: 23, 21, 17, 19; 88,234 with
            // one sweep: 10.7, 12.7, 16.5, 25; 2,000,000: 88, 123, 184, 299).
            const uint64_t at_once = uint64_t(g->num_sms) * 32;
            const uint32_t per_warp = g->num_forward <= 8 * at_once ? 8u : g->num_forward <= 16 * at_once ? 16u : 32u;
            launch(tau_bound_kernel<Vec>, grid_cap(g->num_forward * (32 / per_warp), 256, g->num_sms, 8), 256u,
                   size_t(0), s, true, g->fedge.as<uint4>(), g->num_forward,
                   static_cast<const double2*>(g->tau_sums.as<double2>()), ba, per_warp, stats);
            TGTP_LAUNCH_CHECK("tau_bound_kernel");
        }
    } else {
        // FP32 form: the reference's arithmetic and summation order
        const Real* vec = (const Real*)g->vec_f32.ptr;
        const Real* etab = (const Real*)g->etab_f.ptr;
        const Real eps_half = Real(cfg.epsilon / 2.0);
        // the largest omega this form takes (6,736); the kernel itself keeps 32 indices at a time
        if (32 * size_t(omega) + 4 * 32 * 33 * sizeof(Real) > size_t(227) * 1024)
            fail(TGTP_ERR_UNSUPPORTED, "omega too large for the FP32 form");
        const unsigned tau_blocks = unsigned(std::max<uint64_t>(
            1, std::min<uint64_t>((g->num_forward + kTauEdges - 1) / kTauEdges, uint64_t(1) << 30)));
        ScopedKernel k(g->prof, s, "tau");
        tau_kernel<<<tau_blocks, kTauThreads, 0, s>>>(
            g->idx.as<uint32_t>(), g->adj.as<uint32_t>(), g->row_of.as<uint32_t>(),
            g->rev.as<uint32_t>(), g->forward.as<uint32_t>(), g->num_forward, vec, g->omega, omega,
            g->onep.as<double>(), g->onem.as<double>(), etab, g->etab.as<double>(), eps_half, m, c,
            g->taus.as<int>(), rm, stats);
        TGTP_LAUNCH_CHECK("tau_kernel");
    }
    if constexpr (MIXED) {
        if (!run_mixed(g, cfg, out, rm, mp, logmd)) return;
    } else {
        if (!run_sources<Real>(g, cfg, out, rm, multi, logmd)) return;
    }
    launch_finish<Real, Acc>(g, out);
}

// The persistent source kernel of one batch group: per-block scratch for the group's largest
// graph, packs of up to kBatchPack graphs, each pack one launch on `s` with its own claim counter.
template <class Real>
void launch_group(BatchPlan& plan, BatchGroup& grp, cudaStream_t s, int num_sms) {
    using Pack = SourcePack<Real, kBatchPack>;
    static_assert(sizeof(Pack) < 32000, "pack must fit in the kernel parameter space");
    uint64_t sn = 1, maxd = 1, rows = 0;
    for (size_t i : grp.members) {
        const tgtp_graph* g = plan.entries[i].g;
        sn = std::max<uint64_t>(sn, g->n);
        maxd = std::max<uint64_t>(maxd, g->max_degree);
        rows += g->n;
    }
    const GsLayout lay = gs_layout<Real, Pack>(grp.smem, sn, maxd, rows, num_sms);
    grp.scratch.reserve(lay.scratch());
    grp.wclean.reserve(lay.blocks + 16);
    const size_t packs = (grp.members.size() + kBatchPack - 1) / kBatchPack;
    grp.claims.reserve(sizeof(unsigned) * (packs + 1));
    // each replay starts from "vectors not known to be zero" and fresh claim counters
    TGTP_CUDA(cudaMemsetAsync(grp.wclean.ptr, 0, lay.blocks + 16, s));
    TGTP_CUDA(cudaMemsetAsync(grp.claims.ptr, 0, sizeof(unsigned) * (packs + 1), s));
    for (size_t pk0 = 0; pk0 < grp.members.size(); pk0 += kBatchPack) {
        auto pk = std::make_unique<Pack>();
        pk->count = uint32_t(std::min<size_t>(kBatchPack, grp.members.size() - pk0));
        for (uint32_t j = 0; j < pk->count; ++j) {
            SourceParams<Real> p;
            std::memcpy(&p, plan.entries[grp.members[pk0 + j]].params.data(), sizeof(p));
            carve_gs(p, lay, grp.scratch.as<unsigned char>(), sn, maxd);
            p.clean = grp.wclean.as<unsigned char>();
            p.claim = grp.claims.as<unsigned>() + pk0 / kBatchPack;
            pk->g[j] = p;
        }
        launch_gs<Real>(grp.smem, lay, s, false, *pk);
    }
}

// The same for the mixed form: one block per source, per-block scratch for the group's largest graph.
void launch_mixed_group(BatchPlan& plan, BatchGroup& grp, cudaStream_t s, int num_sms) {
    using Pack = MixedPack<kBatchPack>;
    static_assert(sizeof(Pack) < 32000, "pack must fit in the kernel parameter space");
    uint64_t sn = 1, maxd = 1, rows = 0;
    for (size_t i : grp.members) {
        const tgtp_graph* g = plan.entries[i].g;
        sn = std::max<uint64_t>(sn, g->n);
        maxd = std::max<uint64_t>(maxd, g->max_degree);
        rows += g->n;
    }
    const int mode = grp.smem ? kShared : kGlobal;
    const MixedLayout lay = mixed_layout<Pack>(mode, sn, maxd, rows, num_sms);
    grp.scratch.reserve(lay.scratch());
    grp.wclean.reserve(lay.blocks + 16);
    const size_t packs = (grp.members.size() + kBatchPack - 1) / kBatchPack;
    grp.claims.reserve(sizeof(unsigned) * (packs + 1));
    // each replay starts from "sums not known to be zero" and fresh claim counters
    TGTP_CUDA(cudaMemsetAsync(grp.wclean.ptr, 0, lay.blocks + 16, s));
    TGTP_CUDA(cudaMemsetAsync(grp.claims.ptr, 0, sizeof(unsigned) * (packs + 1), s));
    for (size_t pk0 = 0; pk0 < grp.members.size(); pk0 += kBatchPack) {
        auto pk = std::make_unique<Pack>();
        pk->count = uint32_t(std::min<size_t>(kBatchPack, grp.members.size() - pk0));
        for (uint32_t j = 0; j < pk->count; ++j) {
            MixedParams p;
            std::memcpy(&p, plan.entries[grp.members[pk0 + j]].params.data(), sizeof(p));
            carve_mixed(p, lay, grp.scratch.as<unsigned char>(), sn, maxd);
            p.clean = grp.wclean.as<unsigned char>();
            p.claim = grp.claims.as<unsigned>() + pk0 / kBatchPack;
            pk->g[j] = p;
        }
        launch_mixed(mode, lay, s, false, *pk);
    }
}

}  // namespace

BatchPlan* batch_plan_new() { return new BatchPlan(); }
void batch_plan_free(BatchPlan* plan) { delete plan; }
void batch_plan_collect(BatchPlan* plan) {
    if (plan) plan->entries.clear();
    t_collect = plan;
}

size_t batch_plan_deferred(const BatchPlan* plan) { return plan->entries.size(); }

void batch_plan_launch(BatchPlan* plan, cudaStream_t s, int num_sms) {
    plan->groups.clear();
    for (size_t i = 0; i < plan->entries.size(); ++i) {
        const BatchEntry& e = plan->entries[i];
        BatchGroup* grp = nullptr;
        for (auto& g : plan->groups)
            if (g->key == e.key && g->smem == e.smem) grp = g.get();
        if (!grp) {
            plan->groups.push_back(std::make_unique<BatchGroup>());
            grp = plan->groups.back().get();
            grp->key = e.key;
            grp->smem = e.smem;
        }
        grp->members.push_back(i);
    }
    for (auto& grp : plan->groups) {
        switch (grp->key) {
            case 0: launch_group<float>(*plan, *grp, s, num_sms); break;
            case 1: launch_group<double>(*plan, *grp, s, num_sms); break;
            default: launch_mixed_group(*plan, *grp, s, num_sms); break;
        }
    }
}

void batch_plan_finish(BatchPlan* plan) {
    for (const BatchEntry& e : plan->entries) {
        if (e.key == 0) launch_finish<float, float>(e.g, e.out);
        else if (e.key == 1) launch_finish<double, double>(e.g, e.out);
        else launch_finish<float, double>(e.g, e.out);
    }
}

std::vector<tgtp_graph*> batch_plan_graphs(const BatchPlan* plan) {
    std::vector<tgtp_graph*> v;
    for (const BatchEntry& e : plan->entries) v.push_back(e.g);
    return v;
}


void aesc_run(tgtp_graph* g, const tgtp_config& cfg, float* device_scores) {
    if (!(cfg.epsilon > 0 && cfg.epsilon < 1))
        fail(TGTP_ERR_INVALID_ARGUMENT, "require 0 < epsilon < 1, integer omega >= 2, integer gamma >= 1");
    if (cfg.gamma < 1)
        fail(TGTP_ERR_INVALID_ARGUMENT, "require 0 < epsilon < 1, integer omega >= 2, integer gamma >= 1");
    if (cfg.omega < 2 || uint64_t(cfg.omega) > g->n)
        fail(TGTP_ERR_INVALID_ARGUMENT, "omega must be between 2 and vertex count");
    if (g->omega == 0 || uint32_t(cfg.omega) > g->omega)
        fail(TGTP_ERR_INVALID_ARGUMENT, "eigenpairs for this omega were not uploaded");
    if (!(cfg.delta > 0)) fail(TGTP_ERR_INVALID_ARGUMENT, "delta must be positive");
    if (g->min_degree == 0)
        fail(TGTP_ERR_INVALID_ARGUMENT,
             "graph vertex IDs must be contiguous with no isolated vertices");
    if (g->has_multi_edges && cfg.precision == TGTP_PRECISION_MIXED)
        fail(TGTP_ERR_UNSUPPORTED,
             "the mixed form does not take rows with repeated neighbours or self-loops; "
             "use the FP32 or FP64 form");
    switch (cfg.precision) {
        case TGTP_PRECISION_FP32:
            if (!g->has_f32) fail(TGTP_ERR_INVALID_ARGUMENT, "FP32 form needs F32 eigenvectors");
            run_form<float, false, float>(g, cfg, device_scores);
            break;
        case TGTP_PRECISION_FP64:
            if (!g->has_f64) fail(TGTP_ERR_INVALID_ARGUMENT, "FP64 form needs F64 eigenvectors");
            run_form<double, false, double>(g, cfg, device_scores);
            break;
        case TGTP_PRECISION_MIXED:
            if (cfg.vec_dtype == TGTP_VEC_BF16) {
                if (!g->has_bf16) fail(TGTP_ERR_INVALID_ARGUMENT, "MIXED/BF16 needs BF16 eigenvectors");
                run_form<float, true, __nv_bfloat16>(g, cfg, device_scores);
            } else if (cfg.vec_dtype == TGTP_VEC_F32) {
                if (!g->has_f32) fail(TGTP_ERR_INVALID_ARGUMENT, "MIXED/F32 needs F32 eigenvectors");
                run_form<float, true, float>(g, cfg, device_scores);
            } else {
                fail(TGTP_ERR_INVALID_ARGUMENT, "MIXED form stores eigenvectors as F32 or BF16");
            }
            post_push_hint(g, form_key(cfg), cfg.epsilon);
            break;
        default:
            fail(TGTP_ERR_UNSUPPORTED, "unknown precision form");
    }
    g->last_precision = cfg.precision;
    g->have_run = true;
}

void aesc_check_flags(tgtp_graph* g) {
    unsigned flags[2];
    TGTP_CUDA(cudaMemcpyAsync(flags, run_work(g), sizeof(flags), cudaMemcpyDeviceToHost, g->stream));
    TGTP_CUDA(cudaStreamSynchronize(g->stream));
    if (flags[1] & kErrDeadline)
        fail(TGTP_ERR_TIMEOUT, "device time budget exceeded (TGTP_KERNEL_DEADLINE_S)");
    if (flags[1] & kErrWalkCount)
        fail(TGTP_ERR_UNSUPPORTED, "a walk count exceeds the 32-bit walk grid");
}

namespace {

// Mixed form, graphs of more than 22,680 vertices: the block push when a run's rounds average more than
// m / 40 traversals.  That line was drawn where a dense round of the 32-source push, which reads
// every slot once per 32 sources, became cheaper than pushes made by single warps.  With the present
// kernels, ms, per-source kernel / block push at eps = 0.05, 0.01, 0.005 (Chung-Lu, neighbours and
// exponent; * where the rule takes the block push):
//   one-source block push, up to 27,900 vertices
//     9.3, 2.1   n = 9,000 4.2/3.2, 11/8.3, 16/11; 16,000 23/11, 60/30, 81/40; 20,000 36/17, 100/47, 135/63;
//                23,000 44/21*, 128/58*, 178/78*; 25,860 55/24*, 160/68*, 222/92*
//     20, 2.3    16,000 3.7/3.1, 11/8.3, 17/13; 27,800 4.1/6.8, 24/18*, 48/31*
//   32-source block push
//     9.3, 2.1   28,500 62/143*, 196/253*, 272/307*; 60,000 355/710*, 1,068/1,258*
//     20, 2.3    28,500 4.4/36, 25/70*, 50/83*; 60,000 16/127, 99/256*; 200,000 137/1,125
//     R-MAT, n = 90,000   101/808, 717/1,578*
// So up to 27,900 vertices the block push is the faster one from about 9,000 on unless the pushes are
// shallow, and above that the per-source kernel everywhere; the rule is still the former one.
void learn_push_hint(tgtp_graph* g, int key, double eps, unsigned long long rounds,
                     unsigned long long traversals) {
    if (key < 2 || rounds == 0) return;
    const double per_round = double(traversals) / double(rounds);
    g->push_hint[key] = (mixed_push_chosen(g->n) && per_round * 40.0 > double(g->m)) ? 2 : 1;
    g->push_hint_eps[key] = eps;
}

// The counters of a completed mixed run copied to pinned memory (see tgtp_graph::hint_host), if
// that copy has finished; never waits.
void poll_push_hint(tgtp_graph* g) {
    if (g->hint_key < 0 || !g->hint_event) return;
    const cudaError_t e = cudaEventQuery(g->hint_event);
    if (e == cudaErrorNotReady) {
        (void)cudaGetLastError();
        return;
    }
    TGTP_CUDA(e);
    unsigned long long rounds = 0, trav = 0;
    for (int c = 0; c < kStStripes; ++c) {
        rounds += g->hint_host[size_t(c) * kStCount + kStPushRounds];
        trav += g->hint_host[size_t(c) * kStCount + kStPushTraversals];
    }
    learn_push_hint(g, g->hint_key, g->hint_eps, rounds, trav);
    g->hint_key = -1;
}

// After a mixed run on the handle's stream (not while capturing) on a graph whose push is chosen by
// measurement: copy its counters to pinned memory and record the event poll_push_hint looks at.
void post_push_hint(tgtp_graph* g, int key, double eps) {
    if (!mixed_push_chosen(g->n)) return;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    TGTP_CUDA(cudaStreamIsCapturing(g->stream, &cs));
    if (cs != cudaStreamCaptureStatusNone) return;
    const size_t bytes = sizeof(unsigned long long) * kStCount * kStStripes;
    if (!g->hint_host) {
        void* h = nullptr;
        TGTP_CUDA(cudaHostAlloc(&h, bytes, cudaHostAllocDefault));
        g->hint_host = static_cast<unsigned long long*>(h);
    }
    if (!g->hint_event) TGTP_CUDA(cudaEventCreateWithFlags(&g->hint_event, cudaEventDisableTiming));
    TGTP_CUDA(cudaMemcpyAsync(g->hint_host, g->stats.ptr, bytes, cudaMemcpyDeviceToHost, g->stream));
    TGTP_CUDA(cudaEventRecord(g->hint_event, g->stream));
    g->hint_key = key;
    g->hint_eps = eps;
}

}  // namespace

void aesc_read_stats(tgtp_graph* g, unsigned long long* st) {
    // the striped counters and the work words behind them, in one copy
    unsigned long long stripes[kStCount * kStStripes + 2];
    TGTP_CUDA(cudaMemcpyAsync(stripes, g->stats.ptr, sizeof(stripes), cudaMemcpyDeviceToHost,
                              g->stream));
    TGTP_CUDA(cudaStreamSynchronize(g->stream));
    unsigned work[4];
    std::memcpy(work, stripes + kStCount * kStStripes, sizeof(work));
    if (work[1] & kErrDeadline)
        fail(TGTP_ERR_TIMEOUT, "device time budget exceeded (TGTP_KERNEL_DEADLINE_S)");
    if (work[1] & kErrWalkCount)
        fail(TGTP_ERR_UNSUPPORTED, "a walk count exceeds the 32-bit walk grid");
    for (int i = 0; i < kStCount; ++i) st[i] = 0;
    for (int c = 0; c < kStStripes; ++c)
        for (int i = 0; i < kStCount; ++i) st[i] += stripes[size_t(c) * kStCount + i];
    learn_push_hint(g, g->last_key, g->last_eps, st[kStPushRounds], st[kStPushTraversals]);
}

int aesc_tune(tgtp_graph* g, const tgtp_config& cfg, float* device_scores, int trials) {
    const int key = form_key(cfg);
    const bool mixed = cfg.precision == TGTP_PRECISION_MIXED;
    std::vector<uint16_t> cand;
    if (mixed) {
        // one source per block with its sums in shared memory or in HBM, and the block push at each
        // compaction threshold of its 32-source form (one while the sums fit in shared memory)
        const bool shared = mixed_fits_shared(g->n);
        if (shared) cand.push_back(uint16_t(kLayoutSmem | 1));
        cand.push_back(4);
        for (int ld = 0; ld < (push_shared_bytes(g->n) <= size_t(227) * 1024 ? 1 : 4); ++ld)
            cand.push_back(uint16_t(kLayoutBlock | 4 | (ld << kLayoutListShift)));
    } else {
        // residual vectors in shared memory (four warps a block) or in HBM (two), windowed or
        // one-vertex push
        const bool f64 = cfg.precision == TGTP_PRECISION_FP64;
        const size_t smem = f64 ? gs_shared_bytes<double>(true, g->n) : gs_shared_bytes<float>(true, g->n);
        for (uint16_t pk : {kLayoutWindow, kLayoutNoWindow}) {
            if (smem + 512 <= size_t(227) * 1024) cand.push_back(uint16_t(pk | kLayoutSmem | 4));
            cand.push_back(uint16_t(pk | 2));
        }
    }
    cudaEvent_t e0, e1;
    TGTP_CUDA(cudaEventCreate(&e0));
    TGTP_CUDA(cudaEventCreate(&e1));
    const bool prof = g->prof.enabled;
    g->prof.enabled = false;
    float best = 0;
    uint16_t pick = 0;
    try {
        for (uint16_t c : cand) {
            g->src_layout[key] = c;
            try {
                aesc_run(g, cfg, device_scores);  // warm-up (and scratch for this layout)
            } catch (const Error&) {
                continue;  // the layout does not fit this graph
            }
            float t = 0;
            for (int i = 0; i < std::max(trials, 1); ++i) {
                TGTP_CUDA(cudaEventRecord(e0, g->stream));
                aesc_run(g, cfg, device_scores);
                TGTP_CUDA(cudaEventRecord(e1, g->stream));
                TGTP_CUDA(cudaEventSynchronize(e1));
                float ms = 0;
                TGTP_CUDA(cudaEventElapsedTime(&ms, e0, e1));
                t = i == 0 ? ms : std::min(t, ms);
            }
            if (!pick || t < best) {
                best = t;
                pick = c;
            }
        }
    } catch (...) {
        g->src_layout[key] = 0;
        g->prof.enabled = prof;
        cudaEventDestroy(e0);
        cudaEventDestroy(e1);
        throw;
    }
    g->src_layout[key] = pick;
    g->prof.enabled = prof;
    TGTP_CUDA(cudaEventDestroy(e0));
    TGTP_CUDA(cudaEventDestroy(e1));
    if (!pick) fail(TGTP_ERR_UNSUPPORTED, "no source-kernel layout fits this graph");
    return pick;
}

}  // namespace tgtp

using namespace tgtp;

namespace {
void finish_run(tgtp_graph* g) { aesc_check_flags(g); }
}  // namespace

extern "C" {

tgtp_status tgtp_run_device(tgtp_graph* g, const tgtp_config* cfg, float* device_scores) {
    return guarded([&] {
        if (!g || !cfg || !device_scores) fail(TGTP_ERR_INVALID_ARGUMENT, "null argument");
        aesc_run(g, *cfg, device_scores);
    });
}

tgtp_status tgtp_run(tgtp_graph* g, const tgtp_config* cfg, float* host_scores) {
    return guarded([&] {
        if (!g || !cfg || !host_scores) fail(TGTP_ERR_INVALID_ARGUMENT, "null argument");
        g->out.reserve(sizeof(float) * (g->m + 1));
        aesc_run(g, *cfg, g->out.as<float>());
        TGTP_CUDA(cudaMemcpyAsync(host_scores, g->out.ptr, sizeof(float) * g->m,
                                  cudaMemcpyDeviceToHost, g->stream));
        unsigned long long st[kStCount];
        aesc_read_stats(g, st);  // synchronises once for scores, counters and error flags
    });
}

tgtp_status tgtp_last_run_stats(tgtp_graph* g, tgtp_run_stats* out) {
    return guarded([&] {
        if (!g || !out) fail(TGTP_ERR_INVALID_ARGUMENT, "null argument");
        if (!g->have_run) fail(TGTP_ERR_INVALID_ARGUMENT, "no run on this graph yet");
        finish_run(g);
        unsigned long long st[kStCount] = {};
        aesc_read_stats(g, st);
        out->push_rounds = st[kStPushRounds];
        out->push_vertices = st[kStPushVertices];
        out->push_traversals = st[kStPushTraversals];
        out->walk_edges = st[kStWalkEdges];
        out->walk_count = st[kStWalkCount];
        out->walk_hops = st[kStWalkHops];
        out->fallback_bouquets = st[kStFallback];
        out->tau_iterations = st[kStTauIters];
        out->tau_ambiguous = st[kStTauAmbiguous];
        for (int i = 0; i < 8; ++i) out->phase_cycles[i] = st[kStPhase0 + i];
    });
}

tgtp_status tgtp_last_taus(tgtp_graph* g, int32_t* host_taus) {
    return guarded([&] {
        if (!g || !host_taus) fail(TGTP_ERR_INVALID_ARGUMENT, "null argument");
        if (!g->have_run) fail(TGTP_ERR_INVALID_ARGUMENT, "no run on this graph yet");
        TGTP_CUDA(cudaMemcpyAsync(host_taus, g->taus.ptr, sizeof(int32_t) * g->m,
                                  cudaMemcpyDeviceToHost, g->stream));
        TGTP_CUDA(cudaStreamSynchronize(g->stream));
    });
}

}  // extern "C"
