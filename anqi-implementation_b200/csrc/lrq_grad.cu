// LRQ radius-reconstruction objective: CUDA forward and backward (FP64).
//
// The quantity the reference trainer's rounds minimise
// (tools/train_final_m8_u8.py:90-157, 206-218): for cutoff rows T (n x nk),
// mean mu (nk), rank-M basis G (m x nk) and per-rank codebook B (nk x cs,
// rows ascending),
//   c[o,:]  = (T[o,:] - mu) G^T                    (reconstruct, :90-93)
//   base    = mu + c G
//   a[o,k]  = decode_nearest(T - base)             (:146-156: the insertion
//             point of the value in row k, then the closer of the two
//             neighbours, the lower one on ties)
//   r       = base + B[k, a] - T
//   loss    = sum(r^2) / (n nk)
// With the codes held fixed (a is piecewise constant in the parameters):
//   dL/dB[k,j] = 2/(n nk) sum_{o: a[o,k]=j} r[o,k]
//   dL/dmu[k]  = 2/(n nk) sum_o (r[o,k] - sum_m G[m,k] s[o,m]),  s = r G^T
//   dL/dG[m,k] = 2/(n nk) sum_o (r[o,k] c[o,m] + (T[o,k] - mu[k]) s[o,m])
//
// Forward and the basis half of the backward: one warp per row, lanes over the
// nk columns, one resident block per SM; the codebook half of the backward: a
// histogram per column.  Entry points take device pointers and a stream and
// allocate nothing.
#include <algorithm>

#include "common.cuh"
#include "internal.h"

namespace anqi {
namespace {

constexpr uint32_t kMaxCols = 4;  // per-lane columns: nk <= 128
constexpr unsigned kWarp = 0xFFFFFFFFu;

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kWarp, v, o);
    return v;
}

// Warp sums of M values at once (M = 8 or 16): every step halves the values a
// lane still carries, so M = 8 takes 9 exchanges instead of 40.  Each value is
// summed in warp_sum's tree (partners 16, 8, 4, 2, 1 apart), so the bits are
// the same.  Returns the sum of value sum_index<M>(lane).
template <uint32_t M>
__device__ __forceinline__ double warp_sum_many(double (&v)[M], uint32_t lane) {
    uint32_t o = 16;
#pragma unroll
    for (uint32_t h = M / 2; h > 0; h >>= 1, o >>= 1) {
        const bool up = (lane & o) != 0;
#pragma unroll
        for (uint32_t i = 0; i < h; i++) {
            const double mine = up ? v[i + h] : v[i];
            const double other = up ? v[i] : v[i + h];
            v[i] = mine + __shfl_xor_sync(kWarp, other, o);
        }
    }
    for (; o > 0; o >>= 1) v[0] += __shfl_xor_sync(kWarp, v[0], o);
    return v[0];
}
// The value a lane receives, and the first lane that receives value i.
template <uint32_t M>
__device__ __forceinline__ uint32_t sum_index(uint32_t lane) {
    return lane / (32 / M);
}
template <uint32_t M>
__device__ __forceinline__ uint32_t sum_lane(uint32_t i) {
    return i * (32 / M);
}

struct ObjParams {
    const double* T;
    uint64_t n;
    uint32_t nk, m, cs;
    const double* mu;
    const double* G;
    const double* B;
    const uint8_t* codes_in;  // optional: use these codes instead of the nearest ones
    double* r;
    double* c;
    uint8_t* a;
    double* loss;             // one accumulator, zeroed by the host
    uint32_t bcols, bpitch;   // codebook rows kept in shared memory (whole groups of 32 columns, or all), and their
                              // pitch: the next power of two plus one (odd: lanes on different banks)
};

extern __shared__ __align__(16) double s_lrq[];

// decode_nearest on the lane's column of each group of 32: first index with
// row[i] >= v, then the closer of it and its predecessor, the lower on ties.
// The kMaxCols searches run side by side.
template <class Row>
__device__ __forceinline__ void nearest_codes(const Row& row, uint32_t nk, uint32_t cs, uint32_t lane, uint32_t j0,
                                              uint32_t j1, const double (&v)[kMaxCols], uint32_t (&code)[kMaxCols]) {
    uint32_t lo[kMaxCols];
#pragma unroll
    for (uint32_t j = 0; j < kMaxCols; j++) lo[j] = 0;
#pragma unroll 1
    for (uint32_t step = 256; step > 0; step >>= 1) {
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) {
            if (j < j0 || j >= j1 || lane + 32 * j >= nk) continue;
            if (lo[j] + step <= cs && row(j)[lo[j] + step - 1] < v[j]) lo[j] += step;
        }
    }
#pragma unroll
    for (uint32_t j = 0; j < kMaxCols; j++) {
        if (j < j0 || j >= j1 || lane + 32 * j >= nk) continue;
        const uint32_t high = lo[j] < cs ? lo[j] : cs - 1;
        const uint32_t low = lo[j] > 0 ? lo[j] - 1 : 0;
        code[j] = fabs(row(j)[high] - v[j]) < fabs(v[j] - row(j)[low]) ? high : low;
    }
}

// The same on codebook rows in shared memory, padded with +inf to a power of
// two: a halving step is one load at a constant offset from the running
// position, a compare and a predicated add, without bounds.
// Lanes past the last of the `rows` rows search that one (their codes are not
// used).
__device__ __forceinline__ void nearest_codes_padded(const double* sB, uint32_t pitch, uint32_t cs, uint32_t rows,
                                                     uint32_t lane, const double (&v)[kMaxCols],
                                                     uint32_t (&code)[kMaxCols]) {
    const uint32_t top = pitch - 1;  // the padded row length
    uint32_t at[kMaxCols];
#pragma unroll
    for (uint32_t j = 0; j < kMaxCols; j++) at[j] = min(lane + 32 * j, rows - 1) * pitch;
#pragma unroll
    for (uint32_t step = 128; step > 0; step >>= 1) {
        if (step >= top) continue;
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++)
            if (sB[at[j] + step - 1] < v[j]) at[j] += step;
    }
#pragma unroll
    for (uint32_t j = 0; j < kMaxCols; j++) {
        const uint32_t r0 = min(lane + 32 * j, rows - 1) * pitch;
        const uint32_t lo = at[j] - r0 + (sB[at[j]] < v[j] ? 1u : 0u);
        const uint32_t high = lo < cs ? lo : cs - 1;
        const uint32_t low = lo > 0 ? lo - 1 : 0;
        code[j] = fabs(sB[r0 + high] - v[j]) < fabs(v[j] - sB[r0 + low]) ? high : low;
    }
}

// M: compile-time bound on the rank (m <= M).  One block per SM holds the
// codebook in shared memory (as many columns as fit; the rest is read through
// L1) and the basis, and walks the rows with the next row's cutoffs on their
// way.  Bound by latency and issue of the nine dependent shared-memory gathers
// of the code search (lanes in different codebook rows, about four bank
// conflicts each).  120,000 x 100, rank 8, 256 codes: 526 us with the codebook
// read from global memory by 8 blocks of 8 warps an SM, 174 us now.
template <uint32_t M, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads, 1) lrq_objective_forward_kernel(ObjParams p) {
    const uint32_t lane = threadIdx.x & 31u;
    const uint64_t w = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * kThreads) >> 5;
    double* sG = s_lrq;                              // M x 128 (columns past nk and ranks past m zero)
    double* sB = s_lrq + M * 32 * kMaxCols;          // bcols x bpitch
    for (uint32_t t = threadIdx.x; t < M * 32 * kMaxCols; t += kThreads) {
        const uint32_t mm = t / (32 * kMaxCols), k = t % (32 * kMaxCols);
        sG[t] = mm < p.m && k < p.nk ? p.G[(size_t)mm * p.nk + k] : 0.0;
    }
    if (!p.codes_in)
        for (uint32_t k = threadIdx.x >> 5; k < p.bcols; k += kThreads / 32)
            for (uint32_t i = lane; i < p.bpitch; i += 32)
                sB[k * p.bpitch + i] = i < p.cs ? p.B[(size_t)k * p.cs + i] : __longlong_as_double(0x7ff0000000000000ll);
    __syncthreads();
    double mu[kMaxCols];
#pragma unroll
    for (uint32_t j = 0; j < kMaxCols; j++) mu[j] = lane + 32 * j < p.nk ? p.mu[lane + 32 * j] : 0.0;
    // the lane's columns of the basis stay in registers up to rank 8
    double gr[M == 8 ? M : 1][kMaxCols];
    if constexpr (M == 8) {
#pragma unroll
        for (uint32_t mm = 0; mm < M; mm++)
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++) gr[mm][j] = sG[mm * 32 * kMaxCols + 32 * j + lane];
    }
    auto g = [&](uint32_t mm, uint32_t j) {
        if constexpr (M == 8) return gr[mm][j];
        else return sG[mm * 32 * kMaxCols + 32 * j + lane];
    };
    const uint32_t jb = (p.bcols + 31) / 32;  // column groups in shared memory
    double part = 0.0;
    double nxt[kMaxCols];
    auto load = [&](uint64_t o) {
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++)
            nxt[j] = o < p.n && lane + 32 * j < p.nk ? p.T[o * p.nk + lane + 32 * j] : 0.0;
    };
    load(w);
    for (uint64_t o = w; o < p.n; o += nw) {
        double tv[kMaxCols], v[kMaxCols], base[kMaxCols];
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) {
            tv[j] = nxt[j];
            v[j] = lane + 32 * j < p.nk ? tv[j] - mu[j] : 0.0;
            base[j] = mu[j];
        }
        load(o + nw);
        double s[M];
#pragma unroll
        for (uint32_t mm = 0; mm < M; mm++) {
            s[mm] = 0.0;
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++)
                if (32 * j < p.nk) s[mm] = fma(v[j], g(mm, j), s[mm]);
        }
        const double cm = warp_sum_many<M>(s, lane);
        const uint32_t ci = sum_index<M>(lane);
        if (lane == sum_lane<M>(ci) && ci < p.m) p.c[o * p.m + ci] = cm;
#pragma unroll
        for (uint32_t mm = 0; mm < M; mm++) {
            if (mm >= p.m) break;
            const double cv = __shfl_sync(kWarp, cm, sum_lane<M>(mm));
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++)
                if (32 * j < p.nk) base[j] = fma(cv, g(mm, j), base[j]);
        }
        uint32_t code[kMaxCols] = {0, 0, 0, 0};
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) v[j] = tv[j] - base[j];
        if (p.codes_in) {
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++)
                if (lane + 32 * j < p.nk) code[j] = min((uint32_t)p.codes_in[o * p.nk + lane + 32 * j], p.cs - 1);
        } else {
            auto in_global = [&](uint32_t j) { return p.B + (size_t)(lane + 32 * j) * p.cs; };
            if (p.bcols) nearest_codes_padded(sB, p.bpitch, p.cs, p.bcols, lane, v, code);
            if (32 * jb < p.nk) nearest_codes(in_global, p.nk, p.cs, lane, jb, kMaxCols, v, code);
        }
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) {
            const uint32_t k = lane + 32 * j;
            if (k >= p.nk) continue;
            const double b = !p.codes_in && j < jb ? sB[(size_t)k * p.bpitch + code[j]] : p.B[(size_t)k * p.cs + code[j]];
            const double rv = base[j] + b - tv[j];
            p.r[o * p.nk + k] = rv;
            p.a[o * p.nk + k] = (uint8_t)code[j];
            part = fma(rv, rv, part);
        }
    }
    part = warp_sum(part);
    if (lane == 0 && part != 0.0) atomicAdd(p.loss, part);
}

struct GradParams {
    const double* T;
    uint64_t n;
    uint32_t nk, m, cs;
    const double* mu;
    const double* G;
    const double* r;
    const double* c;
    const uint8_t* a;
    double scale;  // dL/d(sum r^2) times the incoming gradient
    double* g_mu;
    double* g_G;
    double* g_B;
    bool zero_others;  // lrq_codebook_grad_kernel: zero g_mu and g_G
};

// Gradients of mu and G.  A warp keeps its lanes' columns of both in registers
// over all its rows; mu's needs only the sums of s over the rows,
// sum_o r - G^T (sum_o s).  The block's warps add up in shared memory first:
// per-warp atomics to the same m nk + nk addresses, with the codebook's, were
// most of the backward's 529 us at 120,000 x 100; now 95 us, bound by the FP64
// and shuffle work of a row.
template <uint32_t M, uint32_t kThreads>
__global__ void __launch_bounds__(kThreads, 1) lrq_objective_backward_kernel(GradParams p) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    const uint64_t w = ((uint64_t)blockIdx.x * kThreads + threadIdx.x) >> 5;
    const uint64_t nw = ((uint64_t)gridDim.x * kThreads) >> 5;
    constexpr uint32_t kRow = 32 * kMaxCols;
    double* sG = s_lrq;               // M x 128
    double* acc = s_lrq + M * kRow;   // (M + 1) x 128: block sums of g_G, then g_mu
    for (uint32_t t = threadIdx.x; t < M * kRow; t += kThreads) {
        const uint32_t mm = t / kRow, k = t % kRow;
        sG[t] = mm < p.m && k < p.nk ? p.G[(size_t)mm * p.nk + k] : 0.0;
    }
    for (uint32_t t = threadIdx.x; t < (M + 1) * kRow; t += kThreads) acc[t] = 0.0;
    __syncthreads();
    double mu[kMaxCols], gmu[kMaxCols], gG[M][kMaxCols], ssum = 0.0;
#pragma unroll
    for (uint32_t j = 0; j < kMaxCols; j++) {
        mu[j] = lane + 32 * j < p.nk ? p.mu[lane + 32 * j] : 0.0;
        gmu[j] = 0.0;
#pragma unroll
        for (uint32_t mm = 0; mm < M; mm++) gG[mm][j] = 0.0;
    }
    // the next row's residuals, cutoffs and coefficients are on their way while
    // this one is added
    double nr[kMaxCols], nt[kMaxCols], nc = 0.0;
    auto load = [&](uint64_t o) {
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) {
            const bool in = o < p.n && lane + 32 * j < p.nk;
            nr[j] = in ? p.r[o * p.nk + lane + 32 * j] : 0.0;
            nt[j] = in ? p.T[o * p.nk + lane + 32 * j] : 0.0;
        }
        nc = o < p.n && lane < p.m ? p.c[o * p.m + lane] : 0.0;
    };
    load(w);
    for (uint64_t o = w; o < p.n; o += nw) {
        double rv[kMaxCols], cen[kMaxCols], s[M];
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) {
            rv[j] = nr[j];
            cen[j] = lane + 32 * j < p.nk ? nt[j] - mu[j] : 0.0;
            gmu[j] += rv[j];
        }
        const double cl = nc;
        load(o + nw);
#pragma unroll
        for (uint32_t mm = 0; mm < M; mm++) {
            s[mm] = 0.0;
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++)
                if (32 * j < p.nk) s[mm] = fma(sG[mm * kRow + 32 * j + lane], rv[j], s[mm]);
        }
        const double sm = warp_sum_many<M>(s, lane);
        ssum += sm;
#pragma unroll
        for (uint32_t mm = 0; mm < M; mm++) {
            if (mm >= p.m) break;
            const double sv = __shfl_sync(kWarp, sm, sum_lane<M>(mm));
            const double cv = __shfl_sync(kWarp, cl, mm);
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++)
                if (32 * j < p.nk) gG[mm][j] = fma(rv[j], cv, fma(cen[j], sv, gG[mm][j]));
        }
    }
#pragma unroll
    for (uint32_t mm = 0; mm < M; mm++) {
        if (mm >= p.m) break;  // zero times an infinite residual there
        const double sv = __shfl_sync(kWarp, ssum, sum_lane<M>(mm));
#pragma unroll
        for (uint32_t j = 0; j < kMaxCols; j++) gmu[j] = fma(-sG[mm * kRow + 32 * j + lane], sv, gmu[j]);
    }
    for (uint32_t turn = 0; turn < kThreads / 32; turn++) {
        if (turn == warp) {
#pragma unroll
            for (uint32_t j = 0; j < kMaxCols; j++) {
#pragma unroll
                for (uint32_t mm = 0; mm < M; mm++) acc[mm * kRow + 32 * j + lane] += gG[mm][j];
                acc[M * kRow + 32 * j + lane] += gmu[j];
            }
        }
        __syncthreads();
    }
    for (uint32_t t = threadIdx.x; t < (M + 1) * kRow; t += kThreads) {
        const uint32_t mm = t / kRow, k = t % kRow;
        if (k >= p.nk) continue;
        if (mm == M) atomicAdd(p.g_mu + k, p.scale * acc[t]);
        else if (mm < p.m) atomicAdd(p.g_G + (size_t)mm * p.nk + k, p.scale * acc[t]);
    }
}

// Gradient of B: the sums of r by code.  A block has the histograms of 32
// columns in shared memory, lane l of every warp adding to column l's (bank
// pair l: no conflicts inside a warp, hardly any collisions between warps), and
// adds them to g_B once (43 us at 120,000 x 100 x 256); one that has a column's rows
// to itself stores them.  Adding every r to g_B in global memory took an atomic per
// matrix entry.  Launched before the other half (zero_others) it also zeroes that
// one's outputs.
constexpr uint32_t kHistThreads = 1024;
__global__ void __launch_bounds__(kHistThreads, 1) lrq_codebook_grad_kernel(GradParams p) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5, k0 = blockIdx.x * 32, k = k0 + lane;
    if (p.zero_others && blockIdx.x == 0 && blockIdx.y == 0) {
        for (uint32_t t = threadIdx.x; t < p.nk; t += kHistThreads) p.g_mu[t] = 0.0;
        for (uint32_t t = threadIdx.x; t < p.m * p.nk; t += kHistThreads) p.g_G[t] = 0.0;
    }
    for (uint32_t t = threadIdx.x; t < p.cs * 32; t += kHistThreads) s_lrq[t] = 0.0;
    __syncthreads();
    constexpr uint32_t kAhead = 4, kWarps = kHistThreads / 32;
    if (k < p.nk) {
        for (uint64_t o = (uint64_t)blockIdx.y * kWarps + warp; o < p.n; o += (uint64_t)gridDim.y * kWarps * kAhead) {
            double rv[kAhead];
            uint32_t a[kAhead];
#pragma unroll
            for (uint32_t q = 0; q < kAhead; q++) {
                const uint64_t row = o + (uint64_t)q * gridDim.y * kWarps;
                const bool ok = row < p.n;
                rv[q] = ok ? p.r[row * p.nk + k] : 0.0;
                a[q] = ok ? min((uint32_t)p.a[row * p.nk + k], p.cs - 1) : 0u;
            }
#pragma unroll
            for (uint32_t q = 0; q < kAhead; q++) atomicAdd(s_lrq + a[q] * 32 + lane, rv[q]);
        }
    }
    __syncthreads();
    // diagonally, so that a warp's reads fall on all banks
    for (uint32_t t = threadIdx.x; t < p.cs * 32; t += kHistThreads) {
        const uint32_t a = t >> 5, kk = ((t & 31u) + a) & 31u;
        const double v = s_lrq[a * 32 + kk];
        if (k0 + kk >= p.nk) continue;
        double* out = p.g_B + (size_t)(k0 + kk) * p.cs + a;
        if (gridDim.y == 1) *out = p.scale * v;
        else if (v != 0.0) atomicAdd(out, p.scale * v);
    }
}

uint32_t sm_count() {
    int dev = 0, sms = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return (uint32_t)sms;
}

constexpr size_t kSmemMax = 227 * 1024;

// allow_smem where a launch needs it (the calls are a fifth of a small step's host
// time).
template <class Kernel>
cudaError_t large_smem(Kernel kern, size_t smem) {
    return smem > 48 * 1024 ? allow_smem(kern) : cudaSuccess;
}

// A block an SM, fewer only where a warp would have no row: rows one after the other
// cost a warp more than filling another SM's shared memory (forward and backward of
// 1,000 x 100, rank 8, 256 codes: 17.2 and 10.8 us with four rows a warp, 11.0 and
// 7.5 with one; 300 x 100: 17.0 and 10.6, 10.3 and 6.8).
template <uint32_t M, uint32_t kThreads>
cudaError_t launch_forward(ObjParams p, cudaStream_t st) {
    const size_t fixed = (size_t)M * 32 * kMaxCols * 8;
    uint32_t top = 1;
    while (top < p.cs) top <<= 1;
    p.bpitch = top + 1;
    const uint64_t fit = (kSmemMax - fixed) / (p.bpitch * 8ull);
    p.bcols = fit >= p.nk ? p.nk : (uint32_t)fit / 32 * 32;
    const size_t smem = fixed + (p.codes_in ? 0 : (size_t)p.bcols * p.bpitch * 8);
    auto kern = lrq_objective_forward_kernel<M, kThreads>;
    cudaError_t e = large_smem(kern, smem);
    if (e != cudaSuccess) return e;
    constexpr uint64_t rows = kThreads / 32;
    kern<<<(unsigned)std::min<uint64_t>((p.n + rows - 1) / rows, sm_count()), kThreads, smem, st>>>(p);
    return cudaGetLastError();
}

template <uint32_t M, uint32_t kThreads>
cudaError_t launch_backward(GradParams p, cudaStream_t st) {
    // the codebook's: one block an SM, at least 64 rows a block
    const size_t hist = (size_t)p.cs * 32 * 8;
    cudaError_t e = large_smem(lrq_codebook_grad_kernel, hist);
    if (e != cudaSuccess) return e;
    const uint32_t sms = sm_count(), groups = (p.nk + 31) / 32;
    const uint64_t rowgroups = std::min<uint64_t>((p.n + 63) / 64, std::max(1u, sms / groups));
    if (rowgroups > 1 && (e = cudaMemsetAsync(p.g_B, 0, (size_t)p.nk * p.cs * sizeof(double), st)) != cudaSuccess)
        return e;
    auto codebook = [&] {
        lrq_codebook_grad_kernel<<<dim3(groups, (unsigned)rowgroups), kHistThreads, hist, st>>>(p);
        return cudaGetLastError();
    };
    // before the other half while T and r stay in L2, which saves two memsets (a step of
    // 1,000 x 100: 37.8 and 33.8 us); past that after it, which reads T and r itself
    // and leaves the end of r behind (120,000 x 100: 352 us before, 338 after)
    p.zero_others = 2 * p.n * p.nk * sizeof(double) <= 64ull << 20;
    if (p.zero_others) {
        if ((e = codebook()) != cudaSuccess) return e;
    } else if ((e = cudaMemsetAsync(p.g_mu, 0, p.nk * sizeof(double), st)) != cudaSuccess ||
               (e = cudaMemsetAsync(p.g_G, 0, (size_t)p.m * p.nk * sizeof(double), st)) != cudaSuccess) {
        return e;
    }
    const size_t smem = (size_t)(2 * M + 1) * 32 * kMaxCols * 8;
    auto kern = lrq_objective_backward_kernel<M, kThreads>;
    if ((e = large_smem(kern, smem)) != cudaSuccess) return e;
    constexpr uint64_t rows = kThreads / 32;
    kern<<<(unsigned)std::min<uint64_t>((p.n + rows - 1) / rows, sms), kThreads, smem, st>>>(p);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    return p.zero_others ? cudaSuccess : codebook();
}

}  // namespace
}  // namespace anqi

using namespace anqi;

extern "C" {

int anqi_lrq_objective_forward(const double* T, uint64_t n, uint32_t nk, uint32_t m, const double* mu,
                               const double* G, const double* B, uint32_t cs, const uint8_t* codes_in, double* r,
                               double* c, uint8_t* a, double* loss, void* stream) {
    if (!T || !mu || !G || !B || !r || !c || !a || !loss || n == 0) return ANQI_ERR_ARGS;
    if (nk == 0 || nk > 32 * kMaxCols || m == 0 || m > 16 || cs == 0 || cs > 256) return ANQI_ERR_ARGS;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (cudaMemsetAsync(loss, 0, sizeof(double), st) != cudaSuccess) return ANQI_ERR_DEVICE;
    ObjParams p{T, n, nk, m, cs, mu, G, B, codes_in, r, c, a, loss, 0, 0};
    const cudaError_t e = m <= 8 ? launch_forward<8, 384>(p, st) : launch_forward<16, 384>(p, st);
    return e == cudaSuccess ? ANQI_OK : ANQI_ERR_DEVICE;
}

int anqi_lrq_objective_backward(const double* T, uint64_t n, uint32_t nk, uint32_t m, const double* mu,
                                const double* G, const double* r, const double* c, const uint8_t* a, uint32_t cs,
                                double scale, double* g_mu, double* g_G, double* g_B, void* stream) {
    if (!T || !mu || !G || !r || !c || !a || !g_mu || !g_G || !g_B || n == 0) return ANQI_ERR_ARGS;
    if (nk == 0 || nk > 32 * kMaxCols || m == 0 || m > 16 || cs == 0 || cs > 256) return ANQI_ERR_ARGS;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    GradParams p{T, n, nk, m, cs, mu, G, r, c, a, scale, g_mu, g_G, g_B, false};
    const cudaError_t e = m <= 8 ? launch_backward<8, 384>(p, st) : launch_backward<16, 256>(p, st);
    return e == cudaSuccess ? ANQI_OK : ANQI_ERR_DEVICE;
}

}  // extern "C"
