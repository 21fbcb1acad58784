// The AKNN gather (nndindex::gather_candidates and the top-K after it,
// include/index.h:1347-1366, 1491-1525) for rows whose list graph falls into
// small components.
//
// A row's search only ever reaches rows of its own component of the list graph
// (lists and reverse lists taken together), so on clustered data, where a
// component is one cluster, all it needs fits two small tables:
//   - the component's distance matrix, every pair once, in the same FP32 lane
//     order as the general gather (comp_gram_kernel);
//   - the component's adjacency as bitmaps over its own rows (comp_adj_kernel).
// comp_search_kernel then runs the search on them, a warp per row, one bit per
// row of the component: an expansion ORs one bitmap into the visited set.
//
// It is the general gather's search, not a brute-force answer.  That beam keeps
// the ef best visited entries and expands the best unexpanded one, so an entry
// e is expanded when it is the closest visited unexpanded one and its rank
// among the visited is below ef; every visited entry closer than e is expanded
// already, so that rank is the number of expanded entries closer than e.  The
// search ends when no such entry is left, when the pool has reached its cap
// after an expansion, or -- what makes it short -- when the whole component is
// visited, since nothing new can be found from there on.  The result is the
// out_k + 1 best visited entries without the row itself, in the (dist,
// original id) order, as in the general gather.
//
// Components that hold a non-finite distance, and larger ones, stay with the
// general gather.
//
// At 1M x 128 in clusters of 1,000 the gather takes 38.6 ms on the device (Gram
// 14.3, bitmaps 0.5, search 23.8) instead of the general gather's 599 ms, whose
// rows each read 1,000 vectors and walked 120,000 list entries.
//
// The G48 build's select and commit (gather_candidates, the alpha-RNG prune and
// commit_edges, include/index.h:267-281, 772-829, 907-930) run on the same
// tables when every row lies in a small component: comp_select_kernel searches
// and prunes, comp_commit_kernel prunes each row's chosen and reverse edges.
// Both prune against rows of the distance matrix instead of recomputing a
// product per candidate and selected edge.  200k x 130 in clusters of 200:
// 5.9 ms (with the tables) instead of 74.2 ms.
#include <algorithm>
#include <cfloat>
#include <vector>

#include "common.cuh"
#include "component.h"
#include "util.cuh"

namespace anqi {
namespace {

constexpr uint32_t kGT = 32;         // Gram tile: 32 x 32 pairs per block
constexpr uint32_t kKC = 128;        // floats of each row staged at a time
constexpr uint32_t kGS = kKC + 16;   // staged row stride: neighbouring rows half the banks apart
constexpr uint32_t kPad = 0xFFFFFFFFu;

// Order-preserving map of finite floats to unsigned keys.
__device__ __forceinline__ uint32_t key_of(float f) {
    const uint32_t u = __float_as_uint(f);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float value_of(uint32_t k) {
    return __uint_as_float((k >> 31) ? (k & 0x7FFFFFFFu) : ~k);
}

// Distances of all pairs of every component of the batch: block = one 32 x 32
// tile on or above the diagonal, written to both sides.  A 4-thread group owns
// 4 x 4 pairs, thread gt the AVX lanes gt, gt + 4, gt + 8, gt + 12 of each (the
// chunk column order of common.cuh), so the lane accumulators, the fold tree
// and the tail are those of group_ip and the bits are the same; the product is
// symmetric in its rows.  Compute-bound: 64 FMAs per 8 shared loads of a
// thread, rows staged 128 floats at a time.
__global__ void __launch_bounds__(256, 2) comp_gram_kernel(const float* __restrict__ x,
                                                           const float* __restrict__ norms, uint32_t stride,
                                                           uint32_t dim, uint32_t cols,
                                                           const CompDesc* __restrict__ comps, uint32_t ncomps,
                                                           float* __restrict__ G, uint32_t* __restrict__ bad) {
    __shared__ __align__(16) float sa[kGT * kGS];
    __shared__ __align__(16) float sb[kGT * kGS];
    // the component of this tile: the last one whose first tile is <= blockIdx.x
    uint32_t lo = 0, hi = ncomps;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (comps[mid].tile0 <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const CompDesc cd = comps[lo];
    // tile number -> (ti <= tj), row by row of the upper triangle by tj
    const uint32_t t = blockIdx.x - cd.tile0;
    uint32_t tj = (uint32_t)((sqrtf(8.0f * (float)t + 1.0f) - 1.0f) * 0.5f);
    while (tj * (tj + 1) / 2 > t) tj--;
    while ((tj + 1) * (tj + 2) / 2 <= t) tj++;
    const uint32_t ti = t - tj * (tj + 1) / 2;
    const uint32_t i0 = ti * kGT, j0 = tj * kGT;

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u, gt = lane & 3u, gw = lane >> 2;
    // 64 groups as 8 x 8, a warp's as 2 x 4; group (gr, gc) owns rows gr + 8 a,
    // columns gc + 8 b (neighbouring groups' rows fall on different bank halves)
    const uint32_t gr = (warp >> 1) * 2 + (gw >> 2), gc = (warp & 1) * 4 + (gw & 3u);
    const uint32_t q16 = dim >> 4, rem = dim & 15u, nch = q16 + (rem ? 1u : 0u);
    float acc[4][4][4];
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++)
#pragma unroll
            for (int l = 0; l < 4; l++) acc[a][b][l] = 0.f;
    float res[4][4];
    auto fold = [&](const float (&c)[4]) {
        const float t6 = __fadd_rn(__fadd_rn(c[3], c[1]), __fadd_rn(c[2], c[0]));
        const float t8 = __fadd_rn(__shfl_xor_sync(kAll, t6, 2, 4), t6);
        return __fadd_rn(__shfl_xor_sync(kAll, t8, 1, 4), t8);
    };
    for (uint32_t c0 = 0; c0 < nch; c0 += kKC / 16) {
        const uint32_t cn = min(kKC / 16, nch - c0);
        __syncthreads();
        // stage 16 cn floats of the tile's rows and columns in chunk column
        // order, zero past dim; rows past the component repeat its first one
        for (uint32_t e = threadIdx.x; e < 2 * kGT * cn * 4; e += blockDim.x) {
            const uint32_t q = e & 3u, c = (e >> 2) % cn, r = (e >> 2) / cn;  // quarter q of chunk c of staged row r
            const uint32_t rr = r & (kGT - 1);
            const uint32_t loc = (r < kGT ? i0 : j0) + rr;
            const float* src = x + (uint64_t)(cd.start + (loc < cd.size ? loc : 0u)) * stride;
            const uint32_t col = (c0 + c) * 16 + 4 * q;
            float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
            if (col < dim) v = *reinterpret_cast<const float4*>(src + col);  // the row is padded to 8 floats
            float* dst = (r < kGT ? sa : sb) + rr * kGS + c * 16;
            if (cols) {
                *reinterpret_cast<float4*>(dst + 4 * q) = v;
            } else {
                dst[q] = v.x;
                dst[4 + q] = col + 1 < dim ? v.y : 0.f;
                dst[8 + q] = col + 2 < dim ? v.z : 0.f;
                dst[12 + q] = col + 3 < dim ? v.w : 0.f;
            }
        }
        __syncthreads();
        const uint32_t full = c0 + cn > q16 ? q16 - c0 : cn;
#pragma unroll 2
        for (uint32_t c = 0; c < full; c++) {
            float4 av[4], bv[4];
#pragma unroll
            for (int a = 0; a < 4; a++) av[a] = *reinterpret_cast<const float4*>(sa + (gr + 8 * a) * kGS + c * 16 + 4 * gt);
#pragma unroll
            for (int b = 0; b < 4; b++) bv[b] = *reinterpret_cast<const float4*>(sb + (gc + 8 * b) * kGS + c * 16 + 4 * gt);
#pragma unroll
            for (int a = 0; a < 4; a++)
#pragma unroll
                for (int b = 0; b < 4; b++) {
                    acc[a][b][0] = __fmaf_rn(av[a].x, bv[b].x, acc[a][b][0]);
                    acc[a][b][1] = __fmaf_rn(av[a].y, bv[b].y, acc[a][b][1]);
                    acc[a][b][2] = __fmaf_rn(av[a].z, bv[b].z, acc[a][b][2]);
                    acc[a][b][3] = __fmaf_rn(av[a].w, bv[b].w, acc[a][b][3]);
                }
        }
    }
#pragma unroll
    for (int a = 0; a < 4; a++)
#pragma unroll
        for (int b = 0; b < 4; b++) res[a][b] = fold(acc[a][b]);
    if (rem) {
        // the masked tail, the last staged chunk: products without FMA, folded
        // by the same tree and added last
        const uint32_t c = q16 % (kKC / 16);
#pragma unroll
        for (int a = 0; a < 4; a++) {
            const float4 av = *reinterpret_cast<const float4*>(sa + (gr + 8 * a) * kGS + c * 16 + 4 * gt);
#pragma unroll
            for (int b = 0; b < 4; b++) {
                const float4 bv = *reinterpret_cast<const float4*>(sb + (gc + 8 * b) * kGS + c * 16 + 4 * gt);
                const float p[4] = {__fmul_rn(av.x, bv.x), __fmul_rn(av.y, bv.y), __fmul_rn(av.z, bv.z),
                                    __fmul_rn(av.w, bv.w)};
                res[a][b] = __fadd_rn(res[a][b], fold(p));
            }
        }
    }
    // through shared memory, so both orientations are written in whole rows
    __syncthreads();
    float* tile = sa;  // kGT x (kGT + 1)
    bool nonfinite = false;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const uint32_t i = gr + 8 * a;
        const float ni = norms[cd.start + (i0 + i < cd.size ? i0 + i : 0u)];
#pragma unroll
        for (int b = 0; b < 4; b++) {
            if ((uint32_t)a != gt) continue;  // all four threads hold the value; thread a writes row a
            const uint32_t j = gc + 8 * b;
            const float d = norm_d2(ni, norms[cd.start + (j0 + j < cd.size ? j0 + j : 0u)], res[a][b]);
            tile[i * (kGT + 1) + j] = d;
            nonfinite |= !(fabsf(d) <= FLT_MAX);
        }
    }
    if (__syncthreads_or(nonfinite) && threadIdx.x == 0) atomicExch(bad + cd.index, 1u);
    const uint32_t pitch = cd.words * 32;
    float* out = G + cd.goff;
    for (uint32_t e = threadIdx.x; e < kGT * kGT; e += blockDim.x) {
        const uint32_t r = e / kGT, s = e % kGT;
        if (i0 + r < cd.size && j0 + s < cd.size) out[(uint64_t)(i0 + r) * pitch + j0 + s] = tile[r * (kGT + 1) + s];
        if (ti != tj && j0 + r < cd.size && i0 + s < cd.size)
            out[(uint64_t)(j0 + r) * pitch + i0 + s] = tile[s * (kGT + 1) + r];
    }
}

// Adjacency bitmap of each row of the batch over its component: the row's list
// and its reverse list.  Warp per row.
__global__ void __launch_bounds__(128) comp_adj_kernel(uint64_t row_lo, uint64_t row_hi,
                                                       const uint32_t* __restrict__ row_comp,
                                                       const CompDesc* __restrict__ comps, uint32_t first,
                                                       uint32_t ncomps, const uint32_t* __restrict__ g_ids, uint32_t K,
                                                       const uint64_t* __restrict__ rev_off,
                                                       const uint32_t* __restrict__ rev_ids,
                                                       uint32_t* __restrict__ adj) {
    __shared__ uint32_t s_bits[4][kCompMaxWords];
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t row = row_lo + (uint64_t)blockIdx.x * 4 + wib;
    if (row >= row_hi) return;
    const uint32_t ci = row_comp[row] - first;  // kEmpty wraps past ncomps
    if (ci >= ncomps) return;
    const CompDesc cd = comps[ci];
    uint32_t* bits = s_bits[wib];
    for (uint32_t w = lane; w < cd.words; w += 32) bits[w] = 0u;
    __syncwarp();
    for (uint32_t t = lane; t < K; t += 32) {
        const uint32_t e = g_ids[row * K + t] - cd.start;
        if (e < cd.size) atomicOr(bits + (e >> 5), 1u << (e & 31u));
    }
    const uint64_t r1 = rev_off[row + 1];
    for (uint64_t t = rev_off[row] + lane; t < r1; t += 32) {
        const uint32_t e = rev_ids[t] - cd.start;
        if (e < cd.size) atomicOr(bits + (e >> 5), 1u << (e & 31u));
    }
    __syncwarp();
    uint32_t* out = adj + cd.aoff + (uint64_t)(row - cd.start) * cd.words;
    for (uint32_t w = lane; w < cd.words; w += 32) out[w] = bits[w];
}

struct CompSearchParams {
    uint64_t row_lo, row_hi;
    const uint32_t* row_comp;
    const CompDesc* comps;
    uint32_t first, ncomps;
    const float* G;
    const uint32_t* adj;
    const uint32_t* bad;
    const uint32_t* g_ids;
    const float* g_vals;
    uint32_t K, ef, cap, out_k, mcap;
    const uint32_t* perm;
    uint32_t* out_ids;
    float* out_d;
    unsigned long long* pool_total;
};

__host__ __device__ constexpr uint32_t comp_search_words(uint32_t mcap) { return 4 * mcap + kCompMaxWords; }

// The search of one row on its component's tables, one warp per row.  Lane l
// holds the row's distances to the component rows 32 j + l (j < W) as ordered
// keys in registers; word j of a bitmap covers rows 32 j .. 32 j + 31.  The
// out_k + 1 closest rows are selected and sorted first: the search expands
// close rows first, so the next row to expand is found by a ballot over that
// short list (a scan of all keys serves when none of it is left).  Bound by
// instruction issue: a load of the row's distances, a selection (one count when
// the row's own list already is its exact top-K), a rank sort and, per
// expansion, one bitmap row.
template <int W>
__global__ void __launch_bounds__(128) comp_search_kernel(CompSearchParams p) {
    extern __shared__ __align__(16) uint32_t s_search[];
    constexpr int NL = (W + 31) / 32;  // bitmap words per lane
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t row = p.row_lo + (uint64_t)blockIdx.x * 4 + wib;
    if (row >= p.row_hi) return;
    const uint32_t ci = p.row_comp[row] - p.first;
    if (ci >= p.ncomps) return;
    const CompDesc cd = p.comps[ci];
    if (p.bad[cd.index]) return;
    uint32_t* ukey = s_search + wib * comp_search_words(p.mcap);  // selected, unsorted
    uint32_t* uid = ukey + p.mcap;
    uint32_t* skey = uid + p.mcap;  // selected, ascending (dist, original id)
    uint32_t* sid = skey + p.mcap;
    uint32_t* fr = sid + p.mcap;    // frontier: visited, not expanded
    const uint32_t li = (uint32_t)row - cd.start;
    const uint32_t* perm = p.perm + cd.start;

    uint32_t v[W];
    const float* drow = p.G + cd.goff + (uint64_t)li * (cd.words * 32);
#pragma unroll
    for (int j = 0; j < W; j++) {
        const uint32_t e = 32 * j + lane;
        v[j] = e < cd.size ? key_of(drow[e]) : kPad;
    }
    // the row's own list: the seeds, and a guess of the selection's threshold
    uint32_t guess = 0;
    for (uint32_t w = lane; w < NL * 32; w += 32) fr[w] = 0u;
    __syncwarp();
    for (uint32_t t = lane; t < p.K; t += 32) {
        const uint32_t e = p.g_ids[row * p.K + t] - cd.start;
        if (e < cd.size) {
            atomicOr(fr + (e >> 5), 1u << (e & 31u));
            guess = max(guess, key_of(p.g_vals[row * p.K + t]));
        }
    }
    guess = __reduce_max_sync(kAll, guess);
    __syncwarp();
    uint32_t vis[NL], exp_[NL];
    uint32_t npool = 0;
#pragma unroll
    for (int w = 0; w < NL; w++) {
        vis[w] = fr[lane + 32 * w];
        exp_[w] = 0u;
        npool += __popc(vis[w]);
    }
    npool = __reduce_add_sync(kAll, npool);

    auto count_le = [&](uint32_t t) {
        uint32_t c = 0;
#pragma unroll
        for (int j = 0; j < W; j++) c += v[j] <= t ? 1u : 0u;
        return __reduce_add_sync(kAll, c);
    };
    const uint32_t m_all = min(p.out_k + 1, cd.size);
    uint32_t m = m_all;
    for (int pass = 0; pass < 2; pass++) {
        // ---- the m smallest keys (ties at the last one by original id):
        // thr with count(<= thr) >= m, the smallest such unless it is exactly m
        uint32_t thr = guess, cnt = count_le(thr);
        if (cnt != m) {
            uint32_t a = kPad, b = 0;
#pragma unroll
            for (int j = 0; j < W; j++) {
                a = min(a, v[j]);
                if (v[j] != kPad) b = max(b, v[j]);
            }
            a = __reduce_min_sync(kAll, a);
            b = __reduce_max_sync(kAll, b);
            if (cnt > m) b = min(b, thr);
            else if (thr >= a) a = thr + 1;
            while (a < b) {
                const uint32_t mid = a + (b - a) / 2;
                cnt = count_le(mid);
                if (cnt == m) {
                    a = b = mid;
                    break;
                }
                if (cnt > m) b = mid;
                else a = mid + 1;
            }
            thr = a;
            cnt = count_le(thr);
        }
        uint32_t plim = kPad;  // of the entries at thr, those with original ids <= plim
        if (cnt > m) {
            uint32_t below = 0;
#pragma unroll
            for (int j = 0; j < W; j++) below += v[j] < thr ? 1u : 0u;
            const uint32_t need = m - __reduce_add_sync(kAll, below);
            uint32_t a = 0, b = kPad - 1;
            while (a < b) {
                const uint32_t mid = a + (b - a) / 2;
                uint32_t c = 0;
#pragma unroll
                for (int j = 0; j < W; j++)
                    if (v[j] == thr && perm[32 * j + lane] <= mid) c++;
                if (__reduce_add_sync(kAll, c) >= need) b = mid;
                else a = mid + 1;
            }
            plim = a;
        }
        uint32_t at = 0;
#pragma unroll
        for (int j = 0; j < W; j++) {
            const bool in = v[j] < thr || (v[j] == thr && (plim == kPad || perm[32 * j + lane] <= plim));
            const unsigned b = __ballot_sync(kAll, in);
            if (in) {
                const uint32_t pos = at + __popc(b & lane_lt_mask());
                ukey[pos] = v[j];
                uid[pos] = 32 * j + lane;
            }
            at += __popc(b);
        }
        __syncwarp();
        // ---- rank sort (by key; by original id too when two keys tie)
        for (uint32_t e0 = 0; e0 < m; e0 += 128) {
            uint32_t k[4], rank[4] = {0, 0, 0, 0}, same = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) k[q] = e0 + 32 * q + lane < m ? ukey[e0 + 32 * q + lane] : kPad;
            for (uint32_t s = 0; s < m; s++) {
                const uint32_t ks = ukey[s];
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    rank[q] += ks < k[q] ? 1u : 0u;
                    same += ks == k[q] ? 1u : 0u;
                }
            }
            uint32_t own = 0;
#pragma unroll
            for (int q = 0; q < 4; q++) own += e0 + 32 * q + lane < m ? 1u : 0u;
            if (__any_sync(kAll, same != own)) {
#pragma unroll
                for (int q = 0; q < 4; q++) {
                    if (e0 + 32 * q + lane >= m) continue;
                    const uint32_t mine = perm[uid[e0 + 32 * q + lane]];
                    rank[q] = 0;
                    for (uint32_t s = 0; s < m; s++) {
                        const uint32_t ks = ukey[s];
                        rank[q] += (ks < k[q] || (ks == k[q] && perm[uid[s]] < mine)) ? 1u : 0u;
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const uint32_t e = e0 + 32 * q + lane;
                if (e < m) {
                    skey[rank[q]] = k[q];
                    sid[rank[q]] = uid[e];
                }
            }
        }
        __syncwarp();
        if (pass == 1) break;

        // ---- the search
        uint32_t nexp = 0;
        while (npool < cd.size) {
            uint32_t node = kEmpty;
            for (uint32_t e0 = 0; e0 < m; e0 += 32) {
                const uint32_t id = sid[min(e0 + lane, m - 1)];
                const unsigned b = __ballot_sync(kAll, e0 + lane < m && ((fr[id >> 5] >> (id & 31u)) & 1u));
                if (b) {
                    node = __shfl_sync(kAll, id, __ffs(b) - 1);
                    break;
                }
            }
            if (node == kEmpty) {
                // none of the closest out_k + 1 rows: the best of the whole frontier
                uint32_t bk = kPad, be = kPad, bp = kPad;
#pragma unroll
                for (int j = 0; j < W; j++) {
                    if (!((fr[j] >> lane) & 1u)) continue;
                    const uint32_t e = 32 * j + lane;
                    if (v[j] < bk || (v[j] == bk && perm[e] < bp)) {
                        bk = v[j];
                        be = e;
                        bp = perm[e];
                    }
                }
                const uint32_t kmin = __reduce_min_sync(kAll, bk);
                if (kmin == kPad) break;  // nothing left to expand
                const uint32_t pmin = __reduce_min_sync(kAll, bk == kmin ? bp : kPad);
                const unsigned b = __ballot_sync(kAll, bk == kmin && bp == pmin);
                node = __shfl_sync(kAll, be, __ffs(b) - 1);
            }
            if (nexp >= p.ef) {
                // its rank among the visited: the expanded rows closer than it
                const uint32_t nk = key_of(drow[node]), np = perm[node];
                uint32_t closer = 0;
#pragma unroll
                for (int j = 0; j < W; j++) {
                    const uint32_t word = __shfl_sync(kAll, exp_[j / 32], j % 32);
                    if (((word >> lane) & 1u) && (v[j] < nk || (v[j] == nk && perm[32 * j + lane] < np))) closer++;
                }
                if (__reduce_add_sync(kAll, closer) >= p.ef) break;
            }
            const uint32_t* arow = p.adj + cd.aoff + (uint64_t)node * cd.words;
            uint32_t fresh = 0;
#pragma unroll
            for (int w = 0; w < NL; w++) {
                const uint32_t word = lane + 32 * w;
                const uint32_t add = (word < cd.words ? arow[word] : 0u) & ~vis[w];
                vis[w] |= add;
                fresh += __popc(add);
                if (word == (node >> 5)) exp_[w] |= 1u << (node & 31u);
                fr[word] = vis[w] & ~exp_[w];
            }
            npool += __reduce_add_sync(kAll, fresh);
            nexp++;
            __syncwarp();
            if (npool >= p.cap) break;
        }
        if (npool >= cd.size) break;  // the whole component: the list stands
        // else: the list again, over the visited rows
#pragma unroll
        for (int j = 0; j < W; j++) {
            const uint32_t word = __shfl_sync(kAll, vis[j / 32], j % 32);
            if (!((word >> lane) & 1u)) v[j] = kPad;
        }
        m = min(p.out_k + 1, npool);
        __syncwarp();
    }
    // ---- index.h:1355-1361: the first K ids != row
    uint32_t self_pos = kEmpty;
    for (uint32_t t = lane; t < m; t += 32)
        if (sid[t] == li) self_pos = t;
    self_pos = __reduce_min_sync(kAll, self_pos);
    const uint64_t orow = perm[li];
    for (uint32_t t = lane; t < p.out_k; t += 32) {
        const uint32_t src = t >= self_pos ? t + 1 : t;
        const bool ok = src < m;
        p.out_ids[orow * p.out_k + t] = ok ? perm[sid[src]] : kEmpty;
        p.out_d[orow * p.out_k + t] = ok ? value_of(skey[src]) : FLT_MAX;
    }
    if (lane == 0) atomicAdd(p.pool_total, (unsigned long long)npool);
}

template <int W>
int launch_search(Ctx* c, const CompSearchParams& p, uint32_t blocks) {
    const size_t smem = 4ull * 4 * comp_search_words(p.mcap);
    ANQI_CUDA(c, allow_smem(comp_search_kernel<W>));
    comp_search_kernel<W><<<blocks, 128, smem, c->stream>>>(p);
    ANQI_CUDA(c, cudaGetLastError());
    return ANQI_OK;
}

struct CompSelectParams {
    uint64_t row_lo, row_hi;
    const uint32_t* row_comp;
    const CompDesc* comps;
    uint32_t first, ncomps;
    const float* G;
    const uint32_t* adj;
    const uint32_t* bad;
    const uint32_t* g_ids;
    uint32_t K, ef, cap, M;
    float alpha;
    const uint32_t* perm;
    uint32_t* edges;  // select: chosen edges and their reverse, bitmaps laid out as adj (zeroed before)
    uint32_t* links;  // commit: n x M and degrees, original numbering
    uint32_t* deg;
    unsigned long long* pool_total;
};

// Lane l's bits of W bitmap words (word j bit l -> bit j), the words spread over
// the lanes (word j in words[j / 32] of lane j % 32).
template <int W>
__device__ __forceinline__ uint64_t lane_bits(const uint32_t (&words)[(W + 31) / 32], uint32_t lane) {
    uint64_t m = 0;
#pragma unroll
    for (int j = 0; j < W; j++) {
        const uint32_t w = __shfl_sync(kAll, words[j / 32], j % 32);
        m |= (uint64_t)((w >> lane) & 1u) << j;
    }
    return m;
}

// The best (dist, original id) of the lanes' marked entries: its component row,
// or kEmpty when nothing is marked.  Warp-collective.
template <int W>
__device__ __forceinline__ uint32_t best_marked(const float (&v)[W], uint64_t mark, const uint32_t* perm,
                                                uint32_t lane) {
    float bd = 0.f;
    uint32_t be = kEmpty;
#pragma unroll
    for (int j = 0; j < W; j++) {
        if (!((mark >> j) & 1u)) continue;
        const uint32_t e = 32 * j + lane;
        if (be == kEmpty || v[j] < bd || (v[j] == bd && perm[e] < perm[be])) {
            bd = v[j];
            be = e;
        }
    }
    const uint32_t key = be == kEmpty ? kPad : key_of(bd);
    const uint32_t kmin = __reduce_min_sync(kAll, key);
    if (kmin == kPad) return kEmpty;
    unsigned b = __ballot_sync(kAll, key == kmin);
    if (b & (b - 1)) {
        const uint32_t p = key == kmin ? perm[be] : kPad;
        b = __ballot_sync(kAll, p == __reduce_min_sync(kAll, p) && key == kmin);
    }
    return __shfl_sync(kAll, be, __ffs(b) - 1);
}

// alpha-RNG prune (index.h:267-281) of the marked entries of a row with
// distances v into sel: the best one left is taken and drops every entry it
// occludes, found in its row of the distance matrix.
template <int W>
__device__ __forceinline__ uint32_t comp_prune(const float (&v)[W], uint64_t alive, const CompDesc& cd,
                                               const float* G, const uint32_t* perm, uint32_t M, float alpha,
                                               uint32_t* sel, uint32_t lane) {
    uint32_t nsel = 0;
    while (nsel < M) {
        const uint32_t c = best_marked<W>(v, alive, perm, lane);
        if (c == kEmpty) break;
        if (lane == 0) sel[nsel] = c;
        nsel++;
        if (lane == (c & 31u)) alive &= ~(1ull << (c >> 5));
        const float* crow = G + cd.goff + (uint64_t)c * (cd.words * 32);
#pragma unroll
        for (int j = 0; j < W; j++)
            if ((alive >> j) & 1u)
                if (__fmul_rn(alpha, crow[32 * j + lane]) < v[j]) alive &= ~(1ull << j);
    }
    __syncwarp();
    return nsel;
}

// Select: the row's search (as comp_search_kernel's, the next row to expand
// found by a scan of the marked distances: the queue here is short) and the
// prune of everything it visited.  Warp per row.
template <int W>
__global__ void __launch_bounds__(128) comp_select_kernel(CompSelectParams p) {
    __shared__ uint32_t s_words[4][kCompMaxWords], s_sel[4][64];
    constexpr int NL = (W + 31) / 32;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t row = p.row_lo + (uint64_t)blockIdx.x * 4 + wib;
    if (row >= p.row_hi) return;
    const uint32_t ci = p.row_comp[row] - p.first;
    if (ci >= p.ncomps) return;
    const CompDesc cd = p.comps[ci];
    if (p.bad[cd.index]) return;
    uint32_t* words = s_words[wib];
    uint32_t* sel = s_sel[wib];
    const uint32_t li = (uint32_t)row - cd.start;
    const uint32_t* perm = p.perm + cd.start;
    const float* drow = p.G + cd.goff + (uint64_t)li * (cd.words * 32);
    float v[W];
#pragma unroll
    for (int j = 0; j < W; j++) v[j] = 32 * j + lane < cd.size ? drow[32 * j + lane] : 0.f;
    for (uint32_t w = lane; w < NL * 32; w += 32) words[w] = 0u;
    __syncwarp();
    for (uint32_t t = lane; t < p.K; t += 32) {
        const uint32_t e = p.g_ids[row * p.K + t] - cd.start;
        if (e < cd.size) atomicOr(words + (e >> 5), 1u << (e & 31u));
    }
    __syncwarp();
    uint64_t vis = 0;  // the lane's visited entries
#pragma unroll
    for (int j = 0; j < W; j++) vis |= (uint64_t)((words[j] >> lane) & 1u) << j;
    uint64_t front = vis;  // visited, not expanded
    uint32_t npool = __reduce_add_sync(kAll, (uint32_t)__popcll(vis)), nexp = 0;
    while (npool < cd.size) {
        const uint32_t node = best_marked<W>(v, front, perm, lane);
        if (node == kEmpty) break;
        if (nexp >= p.ef) {
            // its rank among the visited: the expanded rows closer than it
            const float nd = drow[node];
            const uint32_t np = perm[node];
            uint32_t closer = 0;
#pragma unroll
            for (int j = 0; j < W; j++)
                if (((vis & ~front) >> j) & 1u)
                    closer += v[j] < nd || (v[j] == nd && perm[32 * j + lane] < np) ? 1u : 0u;
            if (__reduce_add_sync(kAll, closer) >= p.ef) break;
        }
        const uint32_t* arow = p.adj + cd.aoff + (uint64_t)node * cd.words;
        uint32_t aw[NL];
#pragma unroll
        for (int w = 0; w < NL; w++) aw[w] = lane + 32 * w < cd.words ? arow[lane + 32 * w] : 0u;
        const uint64_t fresh = lane_bits<W>(aw, lane) & ~vis;
        vis |= fresh;
        front |= fresh;
        if (lane == (node & 31u)) front &= ~(1ull << (node >> 5));
        npool += __reduce_add_sync(kAll, (uint32_t)__popcll(fresh));
        nexp++;
        if (npool >= p.cap) break;
    }
    if (lane == (li & 31u)) vis &= ~(1ull << (li >> 5));  // never the row itself
    const uint32_t nsel = comp_prune<W>(v, vis, cd, p.G, perm, p.M, p.alpha, sel, lane);
    uint32_t* edges = p.edges + cd.aoff;
    for (uint32_t t = lane; t < nsel; t += 32) {
        const uint32_t c = sel[t];
        atomicOr(edges + (uint64_t)li * cd.words + (c >> 5), 1u << (c & 31u));
        atomicOr(edges + (uint64_t)c * cd.words + (li >> 5), 1u << (li & 31u));
    }
    if (lane == 0) atomicAdd(p.pool_total, (unsigned long long)npool);
}

// Commit: prunes each row's chosen and reverse edges into its final links.
template <int W>
__global__ void __launch_bounds__(128) comp_commit_kernel(CompSelectParams p) {
    __shared__ uint32_t s_sel[4][64];
    constexpr int NL = (W + 31) / 32;
    const uint32_t lane = threadIdx.x & 31u, wib = threadIdx.x >> 5;
    const uint64_t row = p.row_lo + (uint64_t)blockIdx.x * 4 + wib;
    if (row >= p.row_hi) return;
    const uint32_t ci = p.row_comp[row] - p.first;
    if (ci >= p.ncomps) return;
    const CompDesc cd = p.comps[ci];
    if (p.bad[cd.index]) return;
    uint32_t* sel = s_sel[wib];
    const uint32_t li = (uint32_t)row - cd.start;
    const uint32_t* perm = p.perm + cd.start;
    const float* drow = p.G + cd.goff + (uint64_t)li * (cd.words * 32);
    const uint32_t* erow = p.edges + cd.aoff + (uint64_t)li * cd.words;
    uint32_t ew[NL];
#pragma unroll
    for (int w = 0; w < NL; w++) ew[w] = lane + 32 * w < cd.words ? erow[lane + 32 * w] : 0u;
    const uint64_t cand = lane_bits<W>(ew, lane);
    float v[W];
#pragma unroll
    for (int j = 0; j < W; j++) v[j] = (cand >> j) & 1u ? drow[32 * j + lane] : 0.f;
    const uint32_t nsel = comp_prune<W>(v, cand, cd, p.G, perm, p.M, p.alpha, sel, lane);
    const uint64_t orow = perm[li];
    for (uint32_t t = lane; t < p.M; t += 32) p.links[orow * p.M + t] = t < nsel ? perm[sel[t]] : kEmpty;
    if (lane == 0) p.deg[orow] = nsel;
}

template <int W>
int launch_select(Ctx* c, const CompSelectParams& p, uint32_t blocks) {
    comp_select_kernel<W><<<blocks, 128, 0, c->stream>>>(p);
    comp_commit_kernel<W><<<blocks, 128, 0, c->stream>>>(p);
    ANQI_CUDA(c, cudaGetLastError());
    return ANQI_OK;
}

// Components in batches whose matrices fit the context's init_knn key buffer
// (kept between builds and idle here; at least 256 MB are allowed), with each
// row's component.
struct CompBatch {
    size_t c0, c1;
    uint32_t tiles, words;
    uint64_t aoff;
};

int plan_batches(Ctx* c, const CompGather& g, const std::vector<CompRange>& ranges, std::vector<CompBatch>& batches,
                 TmpBuf& descs_d, DevBuf& row_comp, DevBuf& bad) {
    int rc;
    std::vector<uint32_t> rows(g.n, kEmpty);
    std::vector<CompDesc> descs(ranges.size());
    const uint64_t budget = std::max<uint64_t>(c->init_cid.bytes, 256ull << 20) / 4;
    for (size_t k = 0; k < ranges.size();) {
        CompBatch b{k, k, 0, 1, 0};
        uint64_t goff = 0;
        while (b.c1 < ranges.size()) {
            const CompRange& r = ranges[b.c1];
            const uint32_t words = (r.size + 31) / 32;
            const uint64_t need = (uint64_t)r.size * words * 32;
            if (b.c1 > b.c0 && goff + need > budget) break;
            const uint32_t tiles = (r.size + kGT - 1) / kGT;
            descs[b.c1] = {r.start, r.size, words, b.tiles, goff, b.aoff, (uint32_t)b.c1, 0};
            b.tiles += tiles * (tiles + 1) / 2;
            b.words = std::max(b.words, words);
            goff += need;
            b.aoff += (uint64_t)r.size * words;
            for (uint32_t t = 0; t < r.size; t++) rows[r.start + t] = (uint32_t)b.c1;
            b.c1++;
        }
        if ((rc = ensure(c, c->init_cid, goff * 4)) || (rc = ensure(c, c->init_key, b.aoff * 4))) return rc;
        batches.push_back(b);
        k = b.c1;
    }
    if ((rc = h2d(c, row_comp, rows.data(), g.n * 4)) ||
        (rc = h2d(c, descs_d, descs.data(), descs.size() * sizeof(CompDesc))) ||
        (rc = ensure(c, bad, (ranges.size() + 1) * 4)))
        return rc;
    ANQI_CUDA(c, cudaMemsetAsync(bad.p, 0, (ranges.size() + 1) * 4, c->stream));
    return sync(c);  // the host arrays go out of scope
}

// The distance matrices and adjacency bitmaps of a batch's components.
int launch_tables(Ctx* c, const CompGather& g, const CompBatch& b, const CompDesc* comps, uint64_t lo, uint64_t hi,
                  const DevBuf& row_comp, const DevBuf& bad) {
    const uint32_t nc = (uint32_t)(b.c1 - b.c0);
    comp_gram_kernel<<<b.tiles, 256, 0, c->stream>>>(g.x, g.norms, g.stride, g.dim, g.cols, comps, nc,
                                                     c->init_cid.as<float>(), bad.as<uint32_t>());
    comp_adj_kernel<<<(unsigned)((hi - lo + 3) / 4), 128, 0, c->stream>>>(
        lo, hi, row_comp.as<uint32_t>(), comps, (uint32_t)b.c0, nc, g.g_ids, g.K, g.rev_off, g.rev_ids,
        c->init_key.as<uint32_t>());
    ANQI_CUDA(c, cudaGetLastError());
    return ANQI_OK;
}

int any_flag(Ctx* c, const DevBuf& bad, size_t n, bool* any) {
    std::vector<uint32_t> hb(n);
    int rc;
    if ((rc = d2h(c, hb.data(), bad, hb.size() * 4)) || (rc = sync(c))) return rc;
    for (uint32_t f : hb) *any |= f != 0;
    return ANQI_OK;
}

}  // namespace

int run_component_gather(Ctx* c, const CompGather& g, const std::vector<CompRange>& ranges, DevBuf& row_comp,
                         DevBuf& bad, bool* any_bad) {
    *any_bad = false;
    if (ranges.empty()) return ANQI_OK;
    int rc;
    std::vector<CompBatch> batches;
    TmpBuf dc(c);
    if ((rc = plan_batches(c, g, ranges, batches, dc, row_comp, bad))) return rc;
    for (const CompBatch& b : batches) {
        const CompDesc* comps = dc.as<CompDesc>() + b.c0;
        const uint64_t lo = ranges[b.c0].start, hi = (uint64_t)ranges[b.c1 - 1].start + ranges[b.c1 - 1].size;
        const uint32_t blocks = (uint32_t)((hi - lo + 3) / 4);
        if ((rc = launch_tables(c, g, b, comps, lo, hi, row_comp, bad))) return rc;
        CompSearchParams p{};
        p.row_lo = lo;
        p.row_hi = hi;
        p.row_comp = row_comp.as<uint32_t>();
        p.comps = comps;
        p.first = (uint32_t)b.c0;
        p.ncomps = (uint32_t)(b.c1 - b.c0);
        p.G = c->init_cid.as<float>();
        p.adj = c->init_key.as<uint32_t>();
        p.bad = bad.as<uint32_t>();
        p.g_ids = g.g_ids;
        p.g_vals = g.g_vals;
        p.K = g.K;
        p.ef = g.ef;
        p.cap = g.cap;
        p.out_k = g.out_k;
        p.mcap = round_up(g.out_k + 1, 32);
        p.perm = g.perm;
        p.out_ids = g.out_ids;
        p.out_d = g.out_d;
        p.pool_total = g.pool_total;
        // the instance whose registers hold the batch's longest row
        rc = b.words <= 8    ? launch_search<8>(c, p, blocks)
             : b.words <= 20 ? launch_search<20>(c, p, blocks)
             : b.words <= 36 ? launch_search<36>(c, p, blocks)
                             : launch_search<kCompMaxWords>(c, p, blocks);
        if (rc) return rc;
    }
    return any_flag(c, bad, ranges.size(), any_bad);
}

int run_component_select_commit(Ctx* c, const CompGather& g, const std::vector<CompRange>& ranges, uint32_t M,
                                float alpha, uint32_t* links, uint32_t* deg, bool* any_bad) {
    *any_bad = false;
    int rc;
    std::vector<CompBatch> batches;
    TmpBuf dc(c), row_comp(c), bad(c), edges(c);
    if ((rc = plan_batches(c, g, ranges, batches, dc, row_comp, bad))) return rc;
    uint64_t most = 0;
    for (const CompBatch& b : batches) most = std::max(most, b.aoff);
    if ((rc = ensure(c, edges, most * 4))) return rc;
    for (const CompBatch& b : batches) {
        const CompDesc* comps = dc.as<CompDesc>() + b.c0;
        const uint64_t lo = ranges[b.c0].start, hi = (uint64_t)ranges[b.c1 - 1].start + ranges[b.c1 - 1].size;
        const uint32_t blocks = (uint32_t)((hi - lo + 3) / 4);
        if ((rc = launch_tables(c, g, b, comps, lo, hi, row_comp, bad))) return rc;
        ANQI_CUDA(c, cudaMemsetAsync(edges.p, 0, b.aoff * 4, c->stream));
        CompSelectParams p{};
        p.row_lo = lo;
        p.row_hi = hi;
        p.row_comp = row_comp.as<uint32_t>();
        p.comps = comps;
        p.first = (uint32_t)b.c0;
        p.ncomps = (uint32_t)(b.c1 - b.c0);
        p.G = c->init_cid.as<float>();
        p.adj = c->init_key.as<uint32_t>();
        p.bad = bad.as<uint32_t>();
        p.g_ids = g.g_ids;
        p.K = g.K;
        p.ef = g.ef;
        p.cap = g.cap;
        p.M = M;
        p.alpha = alpha;
        p.perm = g.perm;
        p.edges = edges.as<uint32_t>();
        p.links = links;
        p.deg = deg;
        p.pool_total = g.pool_total;
        rc = b.words <= 8    ? launch_select<8>(c, p, blocks)
             : b.words <= 20 ? launch_select<20>(c, p, blocks)
             : b.words <= 36 ? launch_select<36>(c, p, blocks)
                             : launch_select<kCompMaxWords>(c, p, blocks);
        if (rc) return rc;
    }
    return any_flag(c, bad, ranges.size(), any_bad);
}

}  // namespace anqi
