// Nearest-centroid assignment of many rows (k-means steps and add) on the
// tcgen05 tensor cores, with the answer of the exact rule: the first minimum,
// in centroid order, of the sequential FP32 scores (coarse_scores_kernel and
// argmin_kernel; src/IVFScan.hpp:108-138, src/Clustering.cpp:93-118).
//
// Rows and centroids are split as hi + lo, two bf16 each, and the accumulator
// sums hi.hi + lo.hi + hi.lo, so a score s_c = |c|^2 - 2 x.c (L2; -x.c for
// inner product) lies within E of the exact one, E about 2^-15 |x||c| (below).
// The exact winner's s_c is therefore at most the smallest s_c + 2 E.  The
// kernel keeps each row's three smallest scores: when the second is above
// that bound, the first is the label; when the third is, the two candidates
// get their exact scores (assign_exact_kernel); else the row is listed for
// the exact scores of every centroid.
//
// E, with r = v - hi - lo the part of a value the split drops, A the norm of
// |hi| + |lo|, u = 2^-24 and the centroid terms at their maxima over all
// centroids: the dropped products |x_r||c| + |x||c_r| + |x_lo||c_lo|, the f32
// accumulation of 3d products (tc::accum_units), twice that for L2, plus the rounding of the
// norms, of s_c and of the exact sums: (3d + 16) u (|x|^2 + |c|^2), or
// (d + 4) u |x||c| for inner product; all inflated by 2^-7; and 2^-17 |s| for
// the column index that a score carries in its low mantissa bits.  Rows whose E or
// largest |s| could leave [1e-30, 1e37] (overflow, infinities, NaN,
// underflow) are listed for the exact scores.
//
// Bound by L2 reads of the centroid image: a persistent CTA keeps 128 rows
// (their hi and lo k-blocks, converted while the tile before is scanned) in
// shared memory and streams every centroid tile once: 512 KB per 128 rows at
// 1024 x 128.  MMAs of N = 256 read 12 KB of shared memory in 128 cycles of
// math; N = 128 (8 KB in 64) ran at 40 % of the tensor rate.  Measured, 1M x
// 128 to 1024 lists (20 steps on 262,144 rows, then add): 5.5 ms here and
// 1.0 ms of exact scores, where scoring every centroid exactly and the argmin
// took 100.6 ms; the whole build and a first search 117 -> 21.7 ms.
#include <cuda_bf16.h>

#include <algorithm>
#include <cfloat>

#include "hy_assign.cuh"
#include "hy_common.cuh"
#include "hy_tc.cuh"

namespace hy {
namespace {

constexpr int METRIC_L2 = 1;  // include/hy.h's HY_METRIC_L2
constexpr int TM = 128;       // rows per tile
constexpr int TN = 256;       // centroids per accumulator (two tiles of the centroid image)
constexpr int KB = 16384;     // bytes of one k-block (128 rows x 64 bf16)
constexpr int NSTG = 2;       // stages of the centroid ring (a k-block of TN centroids each)
constexpr int W_MMA = 1, W_EPI0 = 4, N_EPI = 8, W_CONV0 = 12, N_CONV = 4;
constexpr int ASSIGN_THREADS = 32 * (W_CONV0 + N_CONV);

struct AssignParams {
    const float* x;
    const unsigned char* cimg;
    const float* cxn;
    const float* cmax;
    int64_t* labels;
    int32_t *second, *hard, *hard_count;
    int* err;
    int n, d, nlist, nkb, nbuf;  // nkb: 64-dimension blocks; nbuf: row tiles held
    int ntc, nit;                     // accumulators per row tile; 128-row tiles of the centroid image
    uint32_t wait_limit;              // polls of a wait before it gives up
    float cK, cN;                     // accum_units u, (3d + 16) u or (d + 4) u, inflated
};

// A bounded wait; one that gives up raises the status word and the abort flag,
// on which every role leaves.  Roles run by a whole warp vote on the result,
// so that no lane is left alone at a warp-wide step.
__device__ inline bool wait_abort(uint64_t* bar, uint32_t parity, const AssignParams& p, volatile int* abort) {
    for (uint32_t i = 0; i < p.wait_limit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 1023u && *abort) return false;
    }
    if (p.err) atomicCAS(p.err, 0, DEV_ERR_TIMEOUT);
    *abort = 1;
    return false;
}

// The three smallest scores of a row and the first two's centroids.
struct Best {
    float m1, m2, m3;
    int i1, i2;
    __device__ void init() {
        m1 = m2 = m3 = INFINITY;
        i1 = i2 = 0;
    }
    __device__ void insert(float s, int c) {
        if (s < m2) {
            m3 = m2;
            if (s < m1) {
                m2 = m1;
                i2 = i1;
                m1 = s;
                i1 = c;
            } else {
                m2 = s;
                i2 = c;
            }
        } else if (s < m3) {
            m3 = s;
        }
    }
};

template <int METRIC>
__global__ void __launch_bounds__(ASSIGN_THREADS, 1) assign_kernel(const __grid_constant__ AssignParams p) {
    extern __shared__ unsigned char sm_raw[];
    unsigned char* sA =
        reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sm_raw) + 1023) & ~uintptr_t(1023));
    const int nkb = p.nkb, nbuf = p.nbuf;
    const size_t tileA = static_cast<size_t>(nkb) * 2 * KB;  // per 64 dimensions: hi k-block, lo k-block
    unsigned char* sB = sA + nbuf * tileA;                   // NSTG x 2 centroid k-blocks
    __shared__ uint64_t afull[2], afree[2], full[NSTG], empty[NSTG], accf[2], acce[2], folded[2], drain;
    __shared__ uint32_t tbase;
    __shared__ int s_abort;
    __shared__ float4 s_row[2][TM];          // per row {|x|, |x_lo|, |x_r|, A_x}
    __shared__ __align__(16) float s_cn[N_EPI][TN / 2];  // a warp's 128 centroid terms
    __shared__ uint32_t s_lo[2];             // it + 1 when some row of tile it has a lo part
    __shared__ float s_m[2][3][TM];          // the second column half's best, for the fold
    __shared__ int s_i[2][2][TM];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    volatile int* vabort = &s_abort;
    constexpr bool l2 = METRIC == METRIC_L2;

    if (threadIdx.x == 0) {
        for (int i = 0; i < 2; ++i) {
            mbar_init(&afull[i], 32 * N_CONV);
            mbar_init(&afree[i], 1 + N_EPI);  // MMA commit + every epilogue warp
            mbar_init(&accf[i], 1);
            mbar_init(&acce[i], N_EPI);
            mbar_init(&folded[i], N_EPI / 2);  // the second half's warps
        }
        for (int i = 0; i < NSTG; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        mbar_init(&drain, 1);
        s_abort = 0;
        s_lo[0] = s_lo[1] = 0;
        fence_mbar_init();
    }
    if (warp == W_MMA) tc::tmem_alloc(&tbase, 2 * TN);
    tc::fence_before_sync();
    __syncthreads();
    tc::fence_after_sync();
    const uint32_t tmem = tbase;
    const int ntiles = (p.n + TM - 1) / TM;

    if (warp >= W_CONV0) {
        // ---------------- converters: rows to hi / lo k-blocks, 8 lanes per row
        const int cw = warp - W_CONV0;
        const bool v4 = (p.d & 3) == 0 && (reinterpret_cast<uintptr_t>(p.x) & 15) == 0;
        uint32_t it = 0;
        for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++it) {
            const int b = static_cast<int>(it % nbuf);
            if (!__all_sync(FULL, wait_abort(&afree[b], ((it / nbuf) & 1u) ^ 1u, p, vabort))) break;
            unsigned char* A = sA + b * tileA;
            uint32_t lo_any = 0;
            for (int r0 = cw * 4; r0 < TM; r0 += N_CONV * 4) {
                const int r = r0 + (lane >> 3), ch = lane & 7;
                const int64_t row = static_cast<int64_t>(t) * TM + r;
                const float* src = p.x + row * p.d;
                float nn = 0.0f, ll = 0.0f, rr = 0.0f, aa = 0.0f;
                for (int kb = 0; kb < nkb; ++kb) {
                    const int j0 = kb * 64 + ch * 8;
                    float v[8];
                    if (row < p.n && v4 && j0 + 8 <= p.d) {
                        const float4 a = __ldg(reinterpret_cast<const float4*>(src + j0));
                        const float4 c = __ldg(reinterpret_cast<const float4*>(src + j0 + 4));
                        v[0] = a.x, v[1] = a.y, v[2] = a.z, v[3] = a.w;
                        v[4] = c.x, v[5] = c.y, v[6] = c.z, v[7] = c.w;
                    } else {
#pragma unroll
                        for (int i = 0; i < 8; ++i) v[i] = row < p.n && j0 + i < p.d ? __ldg(src + j0 + i) : 0.0f;
                    }
                    uint32_t h[4], l[4];
#pragma unroll
                    for (int i = 0; i < 8; i += 2) {
                        const __nv_bfloat16 h0 = __float2bfloat16_rn(v[i]), h1 = __float2bfloat16_rn(v[i + 1]);
                        const float f0 = __bfloat162float(h0), f1 = __bfloat162float(h1);
                        const __nv_bfloat16 l0 = __float2bfloat16_rn(v[i] - f0), l1 = __float2bfloat16_rn(v[i + 1] - f1);
                        const float g0 = __bfloat162float(l0), g1 = __bfloat162float(l1);
                        h[i >> 1] = static_cast<uint32_t>(__bfloat16_as_ushort(h0)) |
                                    static_cast<uint32_t>(__bfloat16_as_ushort(h1)) << 16;
                        l[i >> 1] = static_cast<uint32_t>(__bfloat16_as_ushort(l0)) |
                                    static_cast<uint32_t>(__bfloat16_as_ushort(l1)) << 16;
                        const float e0 = (v[i] - f0) - g0, e1 = (v[i + 1] - f1) - g1;
                        const float a0 = fabsf(f0) + fabsf(g0), a1 = fabsf(f1) + fabsf(g1);
                        nn = fmaf(v[i], v[i], fmaf(v[i + 1], v[i + 1], nn));
                        ll = fmaf(g0, g0, fmaf(g1, g1, ll));
                        rr = fmaf(e0, e0, fmaf(e1, e1, rr));
                        aa = fmaf(a0, a0, fmaf(a1, a1, aa));
                    }
                    lo_any |= l[0] | l[1] | l[2] | l[3];
                    unsigned char* dst = A + static_cast<size_t>(2 * kb) * KB + r * 128 + ((ch ^ (r & 7)) << 4);
                    *reinterpret_cast<uint4*>(dst) = make_uint4(h[0], h[1], h[2], h[3]);
                    *reinterpret_cast<uint4*>(dst + KB) = make_uint4(l[0], l[1], l[2], l[3]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) {
                    nn += __shfl_xor_sync(FULL, nn, o);
                    ll += __shfl_xor_sync(FULL, ll, o);
                    rr += __shfl_xor_sync(FULL, rr, o);
                    aa += __shfl_xor_sync(FULL, aa, o);
                }
                if (ch == 0) s_row[b][r] = make_float4(sqrtf(nn), sqrtf(ll), sqrtf(rr), sqrtf(aa));
            }
            if (lo_any << 1) s_lo[b] = it + 1;
            fence_proxy_async();  // generic-proxy writes -> tensor-core reads
            mbar_arrive_cta(&afull[b]);
        }
    } else if (warp == 0) {
        // ---------------- producer: every centroid k-block, once per row tile
        if (lane == 0) {
            uint32_t i = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x) {
                // CTAs start at different accumulators, so they do not all
                // read the same lines at once.
                int ct = static_cast<int>(blockIdx.x % p.ntc);
                for (int n = 0; n < p.ntc && ok; ++n) {
                    const uint32_t halves = min(2, p.nit - 2 * ct);
                    for (int k = 0; k < 2 * nkb; ++k, ++i) {
                        const uint32_t st = i % NSTG;
                        if (!wait_abort(&empty[st], ((i / NSTG) & 1u) ^ 1u, p, vabort)) {
                            ok = false;
                            break;
                        }
                        mbar_expect_tx(&full[st], halves * KB);
                        for (uint32_t hf = 0; hf < halves; ++hf)
                            bulk_g2s(sB + (st * 2 + hf) * KB,
                                     p.cimg + (static_cast<size_t>(2 * ct + hf) * 2 * nkb + k) * KB, KB, &full[st]);
                    }
                    if (++ct == p.ntc) ct = 0;
                }
            }
            // No copy may outlive the CTA: wait for the last ones (bounded).
            for (uint32_t j = i > NSTG ? i - NSTG : 0; j < i; ++j)
                for (uint32_t w = 0; w < WAIT_LIMIT && !mbar_try_wait(&full[j % NSTG], (j / NSTG) & 1u); ++w) {
                }
        }
    } else if (warp == W_MMA) {
        if (lane == 0) {
            uint32_t i = 0, acc = 0, it = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++it) {
                const int b = static_cast<int>(it % nbuf);
                if (!wait_abort(&afull[b], (it / nbuf) & 1u, p, vabort)) break;
                tc::fence_after_sync();
                const uint32_t a0 = smem_u32(sA + b * tileA);
                // Rows without a lo part (integers to 256, bf16 values) need
                // no lo.hi product.
                const bool lo = *reinterpret_cast<volatile uint32_t*>(&s_lo[b]) == it + 1;
                int tile = static_cast<int>(blockIdx.x % p.ntc);
                for (int ct = 0; ct < p.ntc && ok; ++ct, ++acc) {
                    const int buf = acc & 1;
                    const uint32_t idesc = tc::idesc_bf16_f32(TM, 2 * tile + 1 < p.nit ? TN : TN / 2);
                    if (++tile == p.ntc) tile = 0;
                    if (!wait_abort(&acce[buf], ((acc >> 1) & 1u) ^ 1u, p, vabort)) {
                        ok = false;
                        break;
                    }
                    tc::fence_after_sync();
                    const uint32_t dcol = tmem + static_cast<uint32_t>(buf * TN);
                    for (int k = 0; k < 2 * nkb; ++k, ++i) {
                        const uint32_t st = i % NSTG;
                        if (!wait_abort(&full[st], (i / NSTG) & 1u, p, vabort)) {
                            ok = false;
                            break;
                        }
                        tc::fence_after_sync();
                        const uint32_t bs = smem_u32(sB + st * 2 * KB);
                        const uint32_t ah = a0 + static_cast<uint32_t>(k & ~1) * KB;  // this dimension block's hi
                        // The centroids' hi block meets the rows' hi and lo,
                        // their lo block the rows' hi.
#pragma unroll
                        for (int kk = 0; kk < 4; ++kk) {
                            const uint64_t bd = tc::sdesc_sw128(bs + kk * 32);
                            tc::mma_bf16(dcol, tc::sdesc_sw128(ah + kk * 32), bd, idesc, (k | kk) != 0 ? 1u : 0u);
                            if (lo && (k & 1) == 0) tc::mma_bf16(dcol, tc::sdesc_sw128(ah + KB + kk * 32), bd, idesc, 1u);
                        }
                        tc::mma_commit(&empty[st]);
                    }
                    if (ok) tc::mma_commit(&accf[buf]);
                }
                if (ok) tc::mma_commit(&afree[b]);
            }
            // No tensor-core instruction outlives the CTA either (one is
            // still in flight here only after a wait gave up).
            tc::mma_commit(&drain);
            mbar_wait_bounded(&drain, 0, p.err);
        }
    } else if (warp >= W_EPI0 && warp < W_EPI0 + N_EPI) {
        // ---------------- epilogue: thread = row; each half scans 128 of an
        // accumulator's 256 columns, 64 at a time.
        const int e = warp - W_EPI0, quad = warp & 3, half = e >> 2;
        const int r = quad * 32 + lane;
        const float cf = l2 ? -2.0f : -1.0f;
        const float4 cm = make_float4(p.cmax[0], p.cmax[1], p.cmax[2], p.cmax[3]);
        const float inflate = 1.0f + 0.0078125f;
        uint32_t acc = 0, it = 0;
        bool ok = true;
        for (int t = blockIdx.x; t < ntiles && ok; t += gridDim.x, ++it) {
            const int b = static_cast<int>(it % nbuf);
            Best best;
            best.init();
            int tile = static_cast<int>(blockIdx.x % p.ntc);
            for (int ct = 0; ct < p.ntc; ++ct, ++acc) {
                const int buf = acc & 1;
                const int c00 = tile * TN + half * (TN / 2);
                if (++tile == p.ntc) tile = 0;
                __syncwarp();
#pragma unroll
                for (int j = 0; j < TN / 2; j += 32) {
                    const int c = c00 + lane + j;
                    s_cn[e][lane + j] = c < p.nlist ? (l2 ? __ldg(p.cxn + c) : 0.0f) : FLT_MAX;
                }
                __syncwarp();
                ok = __all_sync(FULL, wait_abort(&accf[buf], (acc >> 1) & 1u, p, vabort));
                if (!ok) break;
                tc::fence_after_sync();
#pragma unroll 1
                for (int ch = 0; ch < TN / 128; ++ch) {
                const int c0 = c00 + 64 * ch;
                // Columns past the centroids: the image's zero rows score
                // FLT_MAX; a half without any centroid was not computed.
                const bool any = c0 < p.nlist;
                uint32_t v[64];
                tc::tmem_ld64(tmem + (static_cast<uint32_t>(quad * 32) << 16) +
                                  static_cast<uint32_t>(buf * TN + half * (TN / 2) + 64 * ch),
                              v);
                if (ch == TN / 128 - 1) {
                    tc::fence_before_sync();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_cta(&acce[buf]);
                }
                if (!any) continue;
                // The 64 columns' three smallest by min / max alone, two
                // at a time (the k-th of two sorted lists is the least of
                // max(a_i, b_j), i + j = k): the column rides in the six low
                // mantissa bits, which E allows for.  (Branches on each
                // column's insertion took 5,000 cycles per 64 columns, most
                // warps always having a lane that inserts; this 2,000.)
                float t1 = INFINITY, t2 = INFINITY, t3 = INFINITY;
#pragma unroll
                for (int j = 0; j < 64; j += 4) {
                    const float4 cn = *reinterpret_cast<const float4*>(&s_cn[e][64 * ch + j]);
                    const float c4[4] = {cn.x, cn.y, cn.z, cn.w};
                    float s[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint32_t w = __float_as_uint(fmaf(cf, __uint_as_float(v[j + i]), c4[i]));
                        s[i] = __uint_as_float((w & ~63u) | static_cast<uint32_t>(j + i));
                    }
#pragma unroll
                    for (int i = 0; i < 4; i += 2) {
                        const float lo = fminf(s[i], s[i + 1]), hi = fmaxf(s[i], s[i + 1]);
                        const float n3 = fminf(fminf(t3, fmaxf(t2, lo)), fmaxf(t1, hi));
                        t2 = fminf(fminf(t2, hi), fmaxf(t1, lo));
                        t1 = fminf(t1, lo);
                        t3 = n3;
                    }
                }
                best.insert(t1, c0 + static_cast<int>(__float_as_uint(t1) & 63u));
                best.insert(t2, c0 + static_cast<int>(__float_as_uint(t2) & 63u));
                best.insert(t3, c0 + static_cast<int>(__float_as_uint(t3) & 63u));
                }  // column chunks
            }
            // Fold the halves: the second writes, the first finishes the row.
            // (Two buffers: the second half reaches tile it + 2 only after
            // the first has released tile it's rows below.)
            const int xb = static_cast<int>(it & 1u);
            if (half == 1) {
                s_m[xb][0][r] = best.m1;
                s_m[xb][1][r] = best.m2;
                s_m[xb][2][r] = best.m3;
                s_i[xb][0][r] = best.i1;
                s_i[xb][1][r] = best.i2;
                __syncwarp();
                if (lane == 0) mbar_arrive_cta(&folded[xb]);
            } else {
                ok = ok && __all_sync(FULL, wait_abort(&folded[xb], (it >> 1) & 1u, p, vabort));
            }
            if (half == 0 && ok) {
                best.insert(s_m[xb][0][r], s_i[xb][0][r]);
                best.insert(s_m[xb][1][r], s_i[xb][1][r]);
                best.insert(s_m[xb][2][r], 0);  // at most the third: its centroid is not kept
                const int64_t row = static_cast<int64_t>(t) * TM + r;
                const float4 q = s_row[b][r];
                if (row < p.n) {
                    float E = fmaf(q.z, cm.x, fmaf(q.x, cm.z, fmaf(q.y, cm.y, p.cK * q.w * cm.w)));
                    E = l2 ? 2.0f * E + p.cN * fmaf(q.x, q.x, cm.x * cm.x) : E + p.cN * q.x * cm.x;
                    // The column in the low mantissa bits: 2^-17 |s|.
                    const float smax = l2 ? fmaf(2.0f * q.x, cm.x, cm.x * cm.x) : q.x * cm.x;
                    E += 7.7e-6f * smax;
                    const float top = fmaf(2.0f * inflate, E, best.m1);
                    const bool sane = E > 1e-30f && smax < 1e37f && E < 1e37f;
                    const bool one = sane && best.m2 > top, two = sane && best.m3 > top;
                    // (A padding column wins where every real score overflows:
                    // a listed row's label is still read as a centroid.)
                    p.labels[row] = min(best.i1, p.nlist - 1);
                    p.second[row] = one || !two ? -1 : best.i2;
                    if (!two) p.hard[atomicAdd(p.hard_count, 1)] = static_cast<int32_t>(row);
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_cta(&afree[b]);  // the row terms are read
        }
    }
    tc::fence_before_sync();
    __syncthreads();
    if (warp == W_MMA) tc::tmem_dealloc(tmem, 2 * TN);
}

// Exact scores (coarse_scores_kernel's arithmetic) of 32 rows per warp, lane =
// row: 32 dimensions of the rows and of their centroids are staged at a time.
// Bound by the read of the rows when every score is wanted.
constexpr int EX_WARPS = 4;
template <int METRIC>
__global__ void __launch_bounds__(32 * EX_WARPS) assign_exact_kernel(const float* __restrict__ x, int n, int d,
                                                                     const float* __restrict__ cent,
                                                                     const int32_t* __restrict__ second,
                                                                     int64_t* __restrict__ labels,
                                                                     float* __restrict__ score) {
    __shared__ float sx[EX_WARPS][32][33], sc[EX_WARPS][32][33];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t r0 = (static_cast<int64_t>(blockIdx.x) * EX_WARPS + warp) * 32;
    if (r0 >= n) return;  // whole warp
    const int64_t row = r0 + lane;
    const int c1 = row < n ? static_cast<int>(labels[row]) : 0;
    const int c2 = row < n ? second[row] : -1;
    const unsigned pairs = __ballot_sync(FULL, c2 >= 0);
    const unsigned rows = score ? __ballot_sync(FULL, row < n) : pairs;
    if (!rows) return;
    float (*X)[33] = sx[warp], (*Y)[33] = sc[warp];
    auto dist = [&](int c, unsigned mask) {
        float a = 0.0f;
        for (int j0 = 0; j0 < d; j0 += 32) {
            const int jn = min(32, d - j0);
            __syncwarp();
#pragma unroll 4
            for (int i = 0; i < 32; ++i) {
                const int ci = __shfl_sync(FULL, c, i);
                if (((mask >> i) & 1u) && lane < jn) {
                    X[i][lane] = x[(r0 + i) * d + j0 + lane];
                    Y[i][lane] = cent[static_cast<size_t>(ci) * d + j0 + lane];
                }
            }
            __syncwarp();
            if ((mask >> lane) & 1u)
                for (int j = 0; j < jn; ++j)
                    a = METRIC == METRIC_L2 ? sq_add(a, X[lane][j], Y[lane][j]) : ip_add(a, X[lane][j], Y[lane][j]);
        }
        return METRIC == METRIC_L2 ? a : -a;
    };
    float best = dist(c1, rows);
    int c = c1;
    if (pairs) {
        const float s2 = dist(max(c2, 0), pairs);
        if (c2 >= 0 && (s2 < best || (s2 == best && c2 < c1))) {
            best = s2;
            c = c2;
        }
    }
    if ((rows >> lane) & 1u) {
        if (c != c1) labels[row] = c;
        if (score) score[row] = best;
    }
}

}  // namespace

cudaError_t launch_assign(const float* x, int n, int d, int nlist, int metric, const AssignWork& w, int nsm,
                          int64_t* labels, cudaStream_t s) {
    if (d > ASSIGN_DMAX || n < 1) return cudaErrorInvalidValue;
    AssignParams p;
    p.x = x;
    p.cimg = static_cast<const unsigned char*>(w.cimg);
    p.cxn = w.cxn;
    p.cmax = w.cmax;
    p.labels = labels;
    p.second = w.second;
    p.hard = w.hard;
    p.hard_count = w.hard_count;
    p.err = w.err;
    p.wait_limit = w.wait_limit;
    p.n = n;
    p.d = d;
    p.nlist = nlist;
    p.nkb = (d + 63) / 64;
    p.nbuf = p.nkb <= 2 ? 2 : 1;  // two row tiles while they leave room for the ring
    p.nit = (nlist + TM - 1) / TM;
    p.ntc = (p.nit + 1) / 2;
    const double u = 1.0 / 16777216.0, inflate = 1.0 + 1.0 / 128.0;
    p.cK = static_cast<float>(tc::accum_units(3 * d, 16) * u * inflate);
    p.cN = static_cast<float>((metric == METRIC_L2 ? 3.0 * d + 16 : d + 4.0) * u * inflate);
    const size_t smem = 1024 + static_cast<size_t>(p.nbuf) * p.nkb * 2 * KB + NSTG * 2 * KB;
    cudaError_t e = cudaMemsetAsync(w.hard_count, 0, sizeof(int32_t), s);
    if (e != cudaSuccess) return e;
    auto run = [&](auto kern) -> cudaError_t {
        cudaError_t le = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(smem));
        if (le != cudaSuccess) return le;
        kern<<<std::min(nsm, (n + TM - 1) / TM), ASSIGN_THREADS, smem, s>>>(p);
        return cudaGetLastError();
    };
    return metric == METRIC_L2 ? run(assign_kernel<1>) : run(assign_kernel<0>);
}

cudaError_t launch_assign_exact(const float* x, int n, int d, const float* cent, int metric, const AssignWork& w,
                                int64_t* labels, float* score, cudaStream_t s) {
    const int grid = (n + 32 * EX_WARPS - 1) / (32 * EX_WARPS);
    if (metric == METRIC_L2)
        assign_exact_kernel<1><<<grid, 32 * EX_WARPS, 0, s>>>(x, n, d, cent, w.second, labels, score);
    else
        assign_exact_kernel<0><<<grid, 32 * EX_WARPS, 0, s>>>(x, n, d, cent, w.second, labels, score);
    return cudaGetLastError();
}

}  // namespace hy
