// Exact spanning centrality of sampled edges on sm_100a: the quantity of src/exact_sc.cpp:24-49
// (and scripts/paper_accuracy.py:13-54), R(u, v) = (e_u - e_v)^T L^+ (e_u - e_v) on the simple
// undirected graph of the CSR (a repeated neighbour counts once, self-loops are ignored), for graphs
// beyond a dense factorisation.  It is the accuracy reference of the approximate scores: each
// sampled slot's resistance comes from Jacobi-preconditioned conjugate gradients on the graph
// Laplacian in FP64, 32 slots at a time as the 32 columns of an n x 32 block (one 256-byte row per
// vertex, lane j of a warp = column j).
//
// One iteration is three grid-wide passes (each a kernel, so every pass sees the previous one's
// results complete):
//   spmv     lp = L p (pull over the simple neighbours of each row) and the column sums of p * lp
//            and of lp;
//   update   alpha = rz / (p . Lp); x += alpha p; r = r - alpha lp - mean, where mean is that of
//            r - alpha lp from the measured column sums of r and lp (b is orthogonal to the constant
//            vector, and so is every exact residual; this removes the rounding drift); the column
//            sums of r, r * r / d (= r . z) and r * r;
//   direct   beta = rz_new / rz; p = r / d + beta p.
// A column whose residual norm has reached tol * ||b|| takes alpha = 0 from then on, so converged
// columns stop moving while the others continue.  Column sums are FP64 atomics over one partial
// per block, so their last bits may vary between runs; the iteration is a solver, not a parity
// path, and its results are checked against the dense oracle to 1e-9.
//
// What bounds a pass is the latency of the gathered 256-byte rows, not their bytes (the blocks of a
// batch stay in L2 up to n of about 10^5), so the work is cut to keep loads in flight: a warp has
// eight neighbour rows in flight, rows of more than kSeg slots are cut into segments for different
// warps (a hub row would hold the whole pass), and several batches run side by side while their
// blocks fit in L2 together.  256 slots of the Chung-Lu graph with n = 25,860, m = 239,944: 9.7 ms;
// with one batch at a time, whole rows per warp and one neighbour row in flight 373.
#include <algorithm>
#include <cmath>
#include <vector>

#include "common.cuh"
#include "internal.hpp"

namespace tgtp {
namespace {

constexpr int kCols = 32;      // slots per batch (block columns)
constexpr int kScThreads = 256;
constexpr int kScWarps = kScThreads / 32;
// Longest run of a row's slots one warp adds up.  256 slots of Chung-Lu graphs, n = 25,860 / 4,039 /
// 200,000 (64 slots): 9.8 / 1.14 / 12.4 ms with 64, 10.2 / 1.20 / 12.0 with 128, 11.6 / 1.35 / 11.9
// with 256.
constexpr uint32_t kSeg = 64;
// Bytes of the blocks (x, r, p, lp) of the batches that run side by side, and their largest number
// (their sums and flags).  n = 25,860 / 4,039, 256 slots: one batch after another 14.6 / 3.7 ms,
// 40 MB 14.6 / 1.13, 80 MB 9.7 / 1.13, 160 MB (beyond L2) 9.5 / 1.13.
constexpr uint64_t kSideBySide = uint64_t(80) << 20;
constexpr uint64_t kMostSide = 256;
constexpr int kCheck = 8;       // iterations between two looks at the residuals from the host
// Column sums of one iteration (kCols doubles each).  An iteration reads the sums of the one
// before (rz, r . r, sum of r) and adds up its own; kCheck + 1 of them form a batch's table, whose
// entry 0 is the last of the previous kCheck iterations.
enum SumIdx { kSumRz = 0, kSumRr, kSumR, kSumPlp, kSumLp, kSums };
constexpr size_t kTable = size_t(kCheck + 1) * kSums * kCols;

// Column sums: every warp keeps its lane's partials (lane = column), the block adds its warps'
// partials in shared memory and lane j of warp 0 adds the block's totals to out[k][j].
template <int N>
__device__ __forceinline__ void block_column_sums(const double (&v)[N], double* const (&out)[N]) {
    __shared__ double part[N][kScWarps][kCols];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
#pragma unroll
    for (int i = 0; i < N; ++i) part[i][w][lane] = v[i];
    __syncthreads();
    if (w < N) {
        double s = 0;
#pragma unroll
        for (int k = 0; k < kScWarps; ++k) s += part[w][k][lane];
        double* o = out[0];
#pragma unroll
        for (int i = 1; i < N; ++i)
            if (w == i) o = out[i];
        if (s != 0.0) atomicAdd(o + lane, s);
    }
}

// Simple degree (neighbours other than the vertex itself, each distinct id once; rows are sorted),
// one warp per row, and the list of the segments (row, first slot) of the rows beyond kSeg slots.
__global__ void simple_degree_kernel(const uint32_t* __restrict__ idx, const uint32_t* __restrict__ adj,
                                     uint32_t n, double* __restrict__ ds, uint2* __restrict__ segs,
                                     uint32_t* __restrict__ num_segs) {
    const uint32_t lane = threadIdx.x & 31;
    for (uint32_t u = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; u < n;
         u += (gridDim.x * blockDim.x) >> 5) {
        const uint32_t b = __ldg(idx + u), e = __ldg(idx + u + 1);
        uint32_t c = 0;
        for (uint32_t q = b + lane; q < e; q += 32) {
            const uint32_t w = __ldg(adj + q);
            if (w != u && (q == b || __ldg(adj + q - 1) != w)) ++c;
        }
#pragma unroll
        for (int o = 16; o; o >>= 1) c += __shfl_xor_sync(kFullMask, c, o);
        if (lane == 0) ds[u] = double(c);
        if (e - b > kSeg) {
            const uint32_t k = (e - b + kSeg - 1) / kSeg;
            uint32_t at = 0;
            if (lane == 0) at = atomicAdd(num_segs, k);
            at = __shfl_sync(kFullMask, at, 0);
            for (uint32_t i = lane; i < k; i += 32) segs[at + i] = make_uint2(u, b + i * kSeg);
        }
    }
}

// The blocks and sums of the batches that run side by side: batch i (blockIdx.y) uses the i-th
// n x kCols block of each and the i-th table of sums.
struct ScBatches {
    uint32_t n;
    const double* ds;
    double *x, *r, *p, *lp;
    double* tables;  // kTable doubles per batch
    double* bb;      // b . b, kCols per batch
    double tol2;
    __device__ __forceinline__ size_t block(uint32_t i) const { return size_t(i) * n * kCols; }
    // sums `which` of iteration `it` (1 .. kCheck; 0: the last of the previous kCheck)
    __device__ __forceinline__ double* sum(uint32_t i, int it, int which) const {
        return tables + size_t(i) * kTable + (size_t(it) * kSums + which) * kCols;
    }
    __device__ __forceinline__ bool converged(uint32_t i, int it, uint32_t j) const {
        return sum(i, it, kSumRr)[j] <= tol2 * bb[i * kCols + j];
    }
};

// Right-hand sides of one batch per block: column j is e_u - e_v for slot slots[j] (zero for
// padding columns and self-loop slots); r = b, p = z = b / d, rz = b . z, bb = b . b.  x, r, p, lp
// and the tables are zero on entry.
__global__ void sc_init_kernel(const ScBatches B, const uint32_t* __restrict__ slots, uint32_t count,
                               const uint32_t* __restrict__ row_of, const uint32_t* __restrict__ adj,
                               uint32_t* __restrict__ ends) {
    const uint32_t i = blockIdx.x, j = threadIdx.x, k = i * kCols + j;
    double rz = 0, bb = 0;
    uint32_t u = 0xffffffffu, v = 0xffffffffu;
    if (k < count) {
        const uint32_t q = slots[k];
        u = row_of[q];
        v = adj[q];
        if (u != v) {
            double* r = B.r + B.block(i);
            double* p = B.p + B.block(i);
            r[size_t(u) * kCols + j] = 1.0;
            r[size_t(v) * kCols + j] = -1.0;
            p[size_t(u) * kCols + j] = 1.0 / B.ds[u];
            p[size_t(v) * kCols + j] = -1.0 / B.ds[v];
            rz = 1.0 / B.ds[u] + 1.0 / B.ds[v];
            bb = 2.0;
        }
    }
    ends[2 * k] = u;
    ends[2 * k + 1] = v;
    B.sum(i, 0, kSumRz)[j] = rz;
    B.sum(i, 0, kSumRr)[j] = bb;  // r . r (so the first test sees an unconverged column)
    B.bb[k] = bb;
}

// Sum of p[t] over the simple neighbours t among the slots [c0, c1) of row u, which starts at slot
// b; lane = column.  Eight rows of p are in flight at a time.
__device__ __forceinline__ double neighbour_sum(const uint32_t* __restrict__ adj,
                                                const double* __restrict__ p, uint32_t u, uint32_t b,
                                                uint32_t c0, uint32_t c1) {
    const uint32_t lane = threadIdx.x & 31;
    double acc = 0;
    for (uint32_t c = c0; c < c1; c += 32) {
        const uint32_t q = c + lane;
        const uint32_t w = q < c1 ? __ldg(adj + q) : u;
        uint32_t before = __shfl_up_sync(kFullMask, w, 1);
        if (lane == 0) before = c > b ? __ldg(adj + c - 1) : 0xffffffffu;
        const unsigned keep = __ballot_sync(kFullMask, w != u && w != before);
        const uint32_t k = __popc(keep);
        // the kept neighbours packed into lanes 0 .. k - 1
        const uint32_t nth = lane < k ? __fns(keep, 0, int(lane) + 1) : 0u;
        const uint32_t packed = __shfl_sync(kFullMask, w, int(nth));
        for (uint32_t t = 0; t < k; t += 8) {
            double x[8];
#pragma unroll
            for (int h = 0; h < 8; ++h) {
                const uint32_t v = __shfl_sync(kFullMask, packed, int((t + h) & 31u));
                x[h] = t + h < k ? p[size_t(v) * kCols + lane] : 0.0;
            }
#pragma unroll
            for (int h = 0; h < 8; ++h) acc += x[h];
        }
    }
    return acc;
}

__global__ void __launch_bounds__(kScThreads)
sc_spmv_kernel(const ScBatches B, int it, const uint32_t* __restrict__ idx,
               const uint32_t* __restrict__ adj, const uint2* __restrict__ segs,
               const uint32_t* __restrict__ num_segs) {
    const uint32_t lane = threadIdx.x & 31, i = blockIdx.y;
    if (__all_sync(kFullMask, B.converged(i, it - 1, lane))) return;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const double* __restrict__ p = B.p + B.block(i);
    double* __restrict__ lp = B.lp + B.block(i);
    const uint32_t ns = *num_segs;
    double dot = 0, sum = 0;
    // the segments of the long rows first, then the other rows
    for (uint64_t k = warp; k < uint64_t(ns) + B.n; k += nw) {
        const uint2 sg = k < ns ? __ldg(segs + k) : make_uint2(uint32_t(k - ns), 0u);
        const uint32_t u = sg.x;
        const uint32_t b = __ldg(idx + u), e = __ldg(idx + u + 1);
        if (k >= ns && e - b > kSeg) continue;
        const uint32_t c0 = k < ns ? sg.y : b, c1 = min(e, c0 + kSeg);
        const size_t o = size_t(u) * kCols + lane;
        const double pu = p[o];
        const double acc = neighbour_sum(adj, p, u, b, c0, c1);
        const double y = c0 == b ? B.ds[u] * pu - acc : -acc;
        if (k < ns) atomicAdd(lp + o, y);  // lp is zero in long rows (init, sc_direct_kernel)
        else lp[o] = y;
        dot += pu * y;
        sum += y;
    }
    const double v[2] = {dot, sum};
    double* const out[2] = {B.sum(i, it, kSumPlp), B.sum(i, it, kSumLp)};
    block_column_sums<2>(v, out);
}

__global__ void __launch_bounds__(kScThreads)
sc_update_kernel(const ScBatches B, int it) {
    const uint32_t lane = threadIdx.x & 31, i = blockIdx.y;
    const bool still = B.converged(i, it - 1, lane);
    if (__all_sync(kFullMask, still)) return;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const double rz = B.sum(i, it - 1, kSumRz)[lane], plp = B.sum(i, it, kSumPlp)[lane];
    const double alpha = (still || !(plp > 0.0)) ? 0.0 : rz / plp;
    const double mean =
        (B.sum(i, it - 1, kSumR)[lane] - alpha * B.sum(i, it, kSumLp)[lane]) / double(B.n);
    const double* __restrict__ p = B.p + B.block(i);
    const double* __restrict__ lp = B.lp + B.block(i);
    double* __restrict__ x = B.x + B.block(i);
    double* __restrict__ r = B.r + B.block(i);
    double s = 0, sz = 0, sr = 0;
    for (uint32_t u = warp; u < B.n; u += nw) {
        const size_t o = size_t(u) * kCols + lane;
        x[o] += alpha * p[o];
        const double rv = (r[o] - alpha * lp[o]) - mean;
        r[o] = rv;
        const double d = B.ds[u];
        s += rv;
        sz += d > 0.0 ? rv * rv / d : 0.0;  // a vertex with no simple neighbour keeps z = 0
        sr += rv * rv;
    }
    const double v[3] = {sz, sr, s};
    double* const out[3] = {B.sum(i, it, kSumRz), B.sum(i, it, kSumRr), B.sum(i, it, kSumR)};
    block_column_sums<3>(v, out);
}

__global__ void __launch_bounds__(kScThreads)
sc_direct_kernel(const ScBatches B, int it, const uint32_t* __restrict__ idx, double beta_guard) {
    const uint32_t lane = threadIdx.x & 31, i = blockIdx.y;
    if (__all_sync(kFullMask, B.converged(i, it - 1, lane))) return;
    const uint32_t warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const uint32_t nw = (gridDim.x * blockDim.x) >> 5;
    const double rz = B.sum(i, it - 1, kSumRz)[lane], rz_new = B.sum(i, it, kSumRz)[lane];
    const double beta = rz > beta_guard ? rz_new / rz : 0.0;
    const double* __restrict__ r = B.r + B.block(i);
    double* __restrict__ p = B.p + B.block(i);
    double* __restrict__ lp = B.lp + B.block(i);
    for (uint32_t u = warp; u < B.n; u += nw) {
        const size_t o = size_t(u) * kCols + lane;
        const double d = B.ds[u];
        p[o] = (d > 0.0 ? r[o] / d : 0.0) + beta * p[o];
        if (__ldg(idx + u + 1) - __ldg(idx + u) > kSeg) lp[o] = 0.0;  // its segments add to it
    }
}

// Entry 0 of each batch's table <- its entry `last`, the others cleared; done[i] = every column of
// batch i has converged.
__global__ void sc_roll_kernel(const ScBatches B, int last, uint32_t* __restrict__ done) {
    double* t = B.tables + size_t(blockIdx.x) * kTable;
    constexpr uint32_t per = kSums * kCols;
    if (threadIdx.x < 32) {
        const bool all = __all_sync(kFullMask, B.converged(blockIdx.x, last, threadIdx.x));
        if (threadIdx.x == 0) done[blockIdx.x] = all;
    }
    __syncthreads();
    for (uint32_t k = threadIdx.x; k < per; k += blockDim.x) t[k] = t[size_t(last) * per + k];
    __syncthreads();
    for (uint32_t k = per + threadIdx.x; k < kTable; k += blockDim.x) t[k] = 0.0;
}

__global__ void sc_answer_kernel(const ScBatches B, const uint32_t* __restrict__ ends, uint32_t count,
                                 double* __restrict__ out) {
    const uint32_t i = blockIdx.x, j = threadIdx.x, k = i * kCols + j;
    if (k >= count) return;
    const double* x = B.x + B.block(i);
    const uint32_t u = ends[2 * k], v = ends[2 * k + 1];
    out[k] = u == v ? 0.0 : x[size_t(u) * kCols + j] - x[size_t(v) * kCols + j];
}

}  // namespace

void exact_sc_slots(tgtp_graph* g, const uint32_t* host_slots, uint32_t count, double tol,
                    uint32_t max_iter, double* host_out, uint32_t* host_iters) {
    if (count == 0) return;
    if (!(tol > 0) || max_iter == 0) fail(TGTP_ERR_INVALID_ARGUMENT, "require tol > 0 and max_iter > 0");
    for (uint32_t i = 0; i < count; ++i)
        if (host_slots[i] >= g->m) fail(TGTP_ERR_INVALID_ARGUMENT, "slot id out of range");
    cudaStream_t s = g->stream;
    const uint32_t n = uint32_t(g->n);
    const size_t blk = sizeof(double) * size_t(n) * kCols;
    // batches side by side: as many as keep their four blocks within kSideBySide bytes of L2
    const uint32_t batches = (count + kCols - 1) / kCols;
    const uint32_t side =
        uint32_t(std::max<uint64_t>(1, std::min<uint64_t>({batches, kMostSide, kSideBySide / (4 * blk)})));
    DeviceBuffer ds, segs, blocks, tables, slots, ends, out;
    ds.reserve(sizeof(double) * n);
    segs.reserve(sizeof(uint2) * (2 * (g->m / kSeg) + 2));  // ceil(d / kSeg) < 2 d / kSeg for d > kSeg
    blocks.reserve(4 * blk * side);
    // tables, then b . b, then the number of segments and the batches' done flags
    const size_t table_bytes = sizeof(double) * (kTable + kCols) * side;
    tables.reserve(table_bytes + sizeof(uint32_t) * (1 + side));
    slots.reserve(sizeof(uint32_t) * count);
    ends.reserve(sizeof(uint32_t) * 2 * kCols * side);
    out.reserve(sizeof(double) * count);
    auto* num_segs = reinterpret_cast<uint32_t*>(tables.as<unsigned char>() + table_bytes);
    TGTP_CUDA(cudaMemsetAsync(num_segs, 0, sizeof(uint32_t), s));
    TGTP_CUDA(cudaMemcpyAsync(slots.ptr, host_slots, sizeof(uint32_t) * count, cudaMemcpyHostToDevice, s));
    const unsigned grid = unsigned(std::max<uint64_t>(
        1, std::min<uint64_t>((uint64_t(n) + kScWarps - 1) / kScWarps, uint64_t(g->num_sms) * 8)));
    simple_degree_kernel<<<grid, kScThreads, 0, s>>>(g->idx.as<uint32_t>(), g->adj.as<uint32_t>(), n,
                                                     ds.as<double>(), segs.as<uint2>(), num_segs);
    TGTP_LAUNCH_CHECK("simple_degree_kernel");
    ScBatches B;
    B.n = n;
    B.ds = ds.as<double>();
    B.x = blocks.as<double>();
    B.r = B.x + size_t(n) * kCols * side;
    B.p = B.r + size_t(n) * kCols * side;
    B.lp = B.p + size_t(n) * kCols * side;
    B.tables = tables.as<double>();
    B.bb = B.tables + kTable * side;
    B.tol2 = tol * tol;
    uint32_t* done = num_segs + 1;
    std::vector<uint32_t> hdone(side);
    for (uint32_t b0 = 0; b0 < batches; b0 += side) {
        const uint32_t nb = std::min(side, batches - b0);
        const uint32_t first = b0 * kCols, bc = std::min<uint32_t>(nb * kCols, count - first);
        TGTP_CUDA(cudaMemsetAsync(blocks.ptr, 0, 4 * blk * side, s));
        TGTP_CUDA(cudaMemsetAsync(tables.ptr, 0, table_bytes, s));
        sc_init_kernel<<<nb, kCols, 0, s>>>(B, slots.as<uint32_t>() + first, bc, g->row_of.as<uint32_t>(),
                                            g->adj.as<uint32_t>(), ends.as<uint32_t>());
        TGTP_LAUNCH_CHECK("sc_init_kernel");
        std::vector<uint32_t> took(nb, 0);  // iterations of each batch, once it has converged
        const dim3 g2(grid, nb);
        uint32_t it = 0, open = nb;
        while (open) {
            if (it >= max_iter)
                fail(TGTP_ERR_TIMEOUT, "conjugate gradients did not converge within max_iter");
            const int k = int(std::min<uint32_t>(kCheck, max_iter - it));
            for (int i = 1; i <= k; ++i) {
                sc_spmv_kernel<<<g2, kScThreads, 0, s>>>(B, i, g->idx.as<uint32_t>(), g->adj.as<uint32_t>(),
                                                         segs.as<uint2>(), num_segs);
                sc_update_kernel<<<g2, kScThreads, 0, s>>>(B, i);
                sc_direct_kernel<<<g2, kScThreads, 0, s>>>(B, i, g->idx.as<uint32_t>(), 1e-300);
            }
            sc_roll_kernel<<<nb, 256, 0, s>>>(B, k, done);
            TGTP_LAUNCH_CHECK("exact spanning centrality iteration");
            it += uint32_t(k);
            TGTP_CUDA(cudaMemcpyAsync(hdone.data(), done, sizeof(uint32_t) * nb, cudaMemcpyDeviceToHost, s));
            TGTP_CUDA(cudaStreamSynchronize(s));
            for (uint32_t b = 0; b < nb; ++b)
                if (!took[b] && hdone[b]) {
                    took[b] = it;
                    --open;
                }
        }
        sc_answer_kernel<<<nb, kCols, 0, s>>>(B, ends.as<uint32_t>(), bc, out.as<double>() + first);
        TGTP_LAUNCH_CHECK("sc_answer_kernel");
        if (host_iters) std::copy(took.begin(), took.end(), host_iters + b0);
    }
    TGTP_CUDA(cudaMemcpyAsync(host_out, out.ptr, sizeof(double) * count, cudaMemcpyDeviceToHost, s));
    TGTP_CUDA(cudaStreamSynchronize(s));
}

}  // namespace tgtp

extern "C" tgtp_status tgtp_exact_sc_slots(tgtp_graph* g, const uint32_t* host_slots, uint32_t count,
                                           double tol, uint32_t max_iter, double* host_resistance,
                                           uint32_t* host_iterations) {
    using namespace tgtp;
    return guarded([&] {
        if (!g || (count && (!host_slots || !host_resistance)))
            fail(TGTP_ERR_INVALID_ARGUMENT, "null argument");
        exact_sc_slots(g, host_slots, count, tol, max_iter, host_resistance, host_iterations);
    });
}
