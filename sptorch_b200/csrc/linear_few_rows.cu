// linear_few_rows.cu -- Linear for a handful of input rows: C[m, n] = act(alpha * sum_k A[m,k] W[n,k] + bias[n]) (+ / * R[m,n]),
// M <= 64, bf16 operands, bf16 or f32 output.  This is the shape of every projection of a decode step (M = sequences in flight;
// crates/nn/src/lib.rs:706-760 and 1119-1131 run them once per generated token).
//
// With so few rows the product is a stream over the weight matrix and nothing else: 2 * N * K bytes read once, a few FLOP per
// byte.  The 128-row tcgen05 tiles of gemm.cu put such a problem on N / 256 .. N / 64 SMs (3 to 48 of 148) with a pipeline
// prologue and a TMEM allocation in front of a few microseconds of work; here the weight rows are spread over N / 8 .. N / 32
// CTAs, every warp takes every eighth 32-element slice of K, issues its weight loads (16 bytes per lane, up to eight slices
// in flight) before it touches the activations, and multiplies with mma.sync m16n8k16 -- the tensor unit is idle either way,
// the warp-level instruction needs no allocation and no barrier.  The eight warps' partial sums meet in shared memory and are
// added in warp order (the result does not depend on scheduling).  Where the weight rows alone do not cover the SMs (the
// projections back to the model width: N = d, K up to 4 d) a cluster of 2 or 4 CTAs splits K and the CTAs' sums meet in the
// cluster's first CTA through distributed shared memory, again in a fixed order.  The RMSNorm in front of a
// projection is applied on the fly to up to 12 rows, the LayerNorm to up to 8 where linear_row_kernel takes the product or rows are longer than
// norm_few_rows_kernel's; the others take that kernel, below, as a launch of its own.
//
// k order inside a 32-element slice: lane t of a quad loads the 8 consecutive elements 8t .. 8t+7 of a weight row and of an
// activation row; the first mma takes elements 0..3 of every lane as its k = {2t, 2t+1, 2t+8, 2t+9}, the second elements 4..7.
// A sum over k does not care about the order as long as both operands use the same one.
//
// A row or a few whose weights all fit the registers of a launch take linear_row_kernel below instead, a warp per weight row and no barrier;
// linear_stream.cu takes over where the weights are many or the rows more than 16 (linear_stream_preferred).  What stays here beside the short
// projections of 3 .. 16 rows, and ordinary launches of up to 3 M weights, are the block-diagonal products and the activation on A.
#include "gemm.h"
#include "epilogue_math.cuh"
#include "pdl.cuh"
#include "sm100.cuh"
#include <algorithm>
#include <cooperative_groups.h>

namespace spt {

namespace {

constexpr int kWarps = 8;
// Row counts up to this take this kernel or linear_stream.cu's by default (the limit of four 16-row groups here, of 64 columns there) and not
// the 128-row tiles of gemm.cu.  Decode step of a 12-layer, 768-wide model at 64 sequences: 0.99 ms with these tiles, 0.92 ms with this
// kernel, where every CTA re-reads more activation bytes from L2 than it streams weight bytes, 0.53 ms with linear_stream.cu's.
constexpr int kDefaultMaxRows = 64;

__device__ __forceinline__ uint4 ld_stream(const void* p) {     // weights: read once, do not keep in L1
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

__device__ __forceinline__ void mma_bf16_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Every CTA normalises all M rows itself: for a few rows that is noise, at 64 rows it cost more than the launch it saves
// (decode step of a 12-layer, 768-wide model at 64 sequences: 2.30 ms with, 1.0 ms without).
constexpr int kNormMaxRows = 16;
// ... and below that the launch of norm_few_rows_kernel, 2.0 us, still pays for more than this many rows: RMSNorm inside, 3072 x 768 in a chain, 16 rows
// 7.4 us, without 3.6; 8 rows 5.1 against 3.5.  LayerNorm, whose two reductions lie behind each other, is taken inside only where a warp does
// it in its registers (linear_row_kernel): 8 rows 2304 x 768 6.5 against 3.4, 2 rows 5120 x 768 5.9 against 3.6, one row 6144 x 2048 8.8 against 5.9.
int norm_inside_rows(const RowNorm& nrm) { return nrm.kind == 1 ? 8 : 12; }
constexpr int kNormLaunchMaxK = 4096;        // the rows norm_few_rows_kernel takes
// Neither does a head pay for it, whose CTAs come in several waves and normalise the rows in each (one row, 50304 x 768 with LayerNorm 22.1 us,
// without 12.5; eight rows, 32000 x 2048 with RMSNorm 29.7, without 21.5; 16384 x 2048 14 against 12.5 beside the launch of about 3).
constexpr long long kNormInsideWeights = 36ll << 20;
// GemmDesc's block-diagonal form
struct FewRowsGroups { int group; long long group_a, group_c; const __nv_bfloat16* gate; long long ld_gate; };
// its activation on A, f32 output and second output
struct FewRowsExtra { int act_from; long long act_off; int c_f32; __nv_bfloat16* c2; };

// a * max(g, 0) on eight bf16 values
__device__ __forceinline__ uint4 relu_mul8(uint4 a, uint4 g) {
    const __nv_bfloat162 zero = __float2bfloat162_rn(0.0f);
    __nv_bfloat162* x = reinterpret_cast<__nv_bfloat162*>(&a);
    const __nv_bfloat162* y = reinterpret_cast<const __nv_bfloat162*>(&g);
#pragma unroll
    for (int i = 0; i < 4; i++) x[i] = __hmul2(x[i], __hmax2(y[i], zero));
    return a;
}

// MT: 16-row groups of A (M <= 16 MT); NT: 8-row groups of W per CTA; S: weight slices a warp has in flight.
// NORM: A holds un-normalised rows; every CTA normalises them itself into shared memory (kind 1: LayerNorm, gamma * ((x - mean) *
// inv) + beta with inv = 1 / sqrt(var + eps); kind 2: RMSNorm, x * inv * gamma with inv = 1 / sqrt(mean(x^2) + eps)), rounded to
// bf16 as the stand-alone kernels store them.  M rows of K values per CTA is little work next to the launch it saves.
template <int MT, int NT, int S, int NORM>
__global__ void __launch_bounds__(kWarps * 32) linear_few_rows_kernel(const __nv_bfloat16* A, long long lda,
                                                                     const __nv_bfloat16* __restrict__ W, long long ldb,
                                                                     __nv_bfloat16* C, long long ldc, const float* __restrict__ bias,
                                                                     const __nv_bfloat16* R, int M, int N, int K, float alpha, int epilogue,
                                                                     RowNorm nrm, int ksplit, FewRowsGroups grp, FewRowsExtra ext) {
    __shared__ float red[kWarps][MT * 16][NT * 8 + 1];
    extern __shared__ __align__(16) uint8_t dyn[];                       // NORM: M rows of (K + 8) bf16
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // ksplit > 1: a cluster of ksplit CTAs shares the weight rows of one block, CTA r of it takes the r-th part of K
    const int krank = blockIdx.x % ksplit;
    const int n0 = (blockIdx.x / ksplit) * (NT * 8);
    const int all_slices = (K + 31) >> 5, per_cta = (all_slices + ksplit - 1) / ksplit;
    const int s_lo = krank * per_cta, slices = min(all_slices, s_lo + per_cta);
    const int gi = grp.group ? n0 / grp.group : 0;          // a CTA's weight rows lie in one group
    A += gi * grp.group_a;
    C += gi * (grp.group_c - grp.group);
    constexpr bool SPLITS = NORM == 0 && MT == 1;            // the instantiations that a cluster may share
    if (SPLITS && ksplit > 1) sm100::cluster_arrive();
    const int k_mine = K - 8 * t;               // a slice s holds elements of this lane while 32 s < k_mine (K is a multiple of 8)
    pdl_release();

    const __nv_bfloat16* wrow[NT];
#pragma unroll
    for (int j = 0; j < NT; j++) wrow[j] = W + (long long)min(n0 + 8 * j + g, N - 1) * ldb + 8 * t;
    float acc[MT][NT][4];
#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][j][q] = 0.0f;

    uint4 wv[S][NT];
    auto load_weights = [&](int s0) {
#pragma unroll
        for (int u = 0; u < S; u++) {
            const int s = s0 + u * kWarps;
#pragma unroll
            for (int j = 0; j < NT; j++) wv[u][j] = s < slices && 32 * s < k_mine ? ld_stream(wrow[j] + 32 * s) : make_uint4(0, 0, 0, 0);
        }
    };
    load_weights(s_lo + warp);       // the weights do not depend on the kernel before this one
    // the output elements this thread finishes at the end: their bias and residual are requested now, not after the reduction
    constexpr int EI = (MT * 16 * NT * 8 + kWarps * 32 - 1) / (kWarps * 32);
    float bpre[EI], rpre[EI];
#pragma unroll
    for (int it = 0; it < EI; it++) {
        const int e = tid + it * kWarps * 32, n = n0 + e % (NT * 8);
        bpre[it] = (bias && e < MT * 16 * NT * 8 && n < N) ? __ldg(bias + n) : 0.0f;
    }
    pdl_acquire();
#pragma unroll
    for (int it = 0; it < EI; it++) {
        const int e = tid + it * kWarps * 32, m = e / (NT * 8), n = n0 + e % (NT * 8);
        rpre[it] = !(R && krank == 0 && m < M && n < N) ? 0.0f
                   : ext.c_f32                          ? reinterpret_cast<const float*>(R)[(long long)m * ldc + n]
                                                        : __bfloat162float(R[(long long)m * ldc + n]);
    }

    const long long a_ld = NORM ? (long long)(K + 8) : lda;
    const __nv_bfloat16* a_base = NORM ? reinterpret_cast<const __nv_bfloat16*>(dyn) : A;
    if constexpr (NORM == 1) {
        // Warps are dealt over (row, part of the row): eight rows or more, one warp per row; a single row, eight warps on its eighths.
        // The partial sums of a row's parts meet in shared memory.
        __shared__ float part[kNormMaxRows][kWarps], part2[kNormMaxRows][kWarps];
        const int P = M >= 8 ? 1 : M >= 4 ? 2 : M >= 2 ? 4 : 8, RP = kWarps / P;
        const int my_p = warp % P, my_r = warp / P;
        const int nvec = K >> 3, per = (nvec + P - 1) / P;
        const int c_begin = my_p * per, c_end = min(nvec, c_begin + per);
        const bool ln = nrm.kind == 1;
#pragma unroll 1
        for (int r = my_r; r < M; r += RP) {
            const uint4* src = reinterpret_cast<const uint4*>(A + (long long)r * lda);
            uint4* row = reinterpret_cast<uint4*>(dyn + (size_t)r * (K + 8) * 2);
            float acc1 = 0.0f;                                      // LayerNorm: sum; RMSNorm: sum of squares
            for (int c = c_begin + lane; c < c_end; c += 32) {
                const uint4 d = src[c];
                row[c] = d;
                const uint32_t wd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float lo = __uint_as_float(wd[j] << 16), hi = __uint_as_float(wd[j] & 0xffff0000u);
                    acc1 += ln ? lo + hi : lo * lo + hi * hi;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) acc1 += __shfl_xor_sync(0xffffffffu, acc1, o);
            if (lane == 0) part[r][my_p] = acc1;
        }
        if (P == 1) __syncwarp(); else __syncthreads();      // one warp per row: its sums never leave the warp
        if (ln) {
#pragma unroll 1
            for (int r = my_r; r < M; r += RP) {
                float tot = 0.0f;
                for (int q = 0; q < P; q++) tot += part[r][q];
                const float mean = tot / (float)K;
                const uint4* row = reinterpret_cast<const uint4*>(dyn + (size_t)r * (K + 8) * 2);
                float var = 0.0f;                                   // centred second pass over this warp's part of the copy in shared memory
                for (int c = c_begin + lane; c < c_end; c += 32) {
                    const uint4 d = row[c];
                    const uint32_t wd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float lo = __uint_as_float(wd[j] << 16) - mean, hi = __uint_as_float(wd[j] & 0xffff0000u) - mean;
                        var += lo * lo + hi * hi;
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) var += __shfl_xor_sync(0xffffffffu, var, o);
                if (lane == 0) part2[r][my_p] = var;
            }
            if (P == 1) __syncwarp(); else __syncthreads();
        }
#pragma unroll 1
        for (int r = my_r; r < M; r += RP) {
            float tot = 0.0f, tot2 = 0.0f;
            for (int q = 0; q < P; q++) { tot += part[r][q]; tot2 += part2[r][q]; }
            const float mean = ln ? tot / (float)K : 0.0f;
            const float inv = 1.0f / sqrtf((ln ? tot2 : tot) / (float)K + nrm.eps);
            uint4* row = reinterpret_cast<uint4*>(dyn + (size_t)r * (K + 8) * 2);
            for (int c = c_begin + lane; c < c_end; c += 32) {
                const uint4 d = row[c];
                const uint32_t wd[4] = {d.x, d.y, d.z, d.w};
                const float4 g0 = __ldg(reinterpret_cast<const float4*>(nrm.gamma + 8 * c)), g1 = __ldg(reinterpret_cast<const float4*>(nrm.gamma + 8 * c + 4));
                const float gg[8] = {g0.x, g0.y, g0.z, g0.w, g1.x, g1.y, g1.z, g1.w};
                float bb[8] = {0, 0, 0, 0, 0, 0, 0, 0};
                if (ln) {
                    const float4 b0 = __ldg(reinterpret_cast<const float4*>(nrm.beta + 8 * c)), b1 = __ldg(reinterpret_cast<const float4*>(nrm.beta + 8 * c + 4));
                    bb[0] = b0.x; bb[1] = b0.y; bb[2] = b0.z; bb[3] = b0.w; bb[4] = b1.x; bb[5] = b1.y; bb[6] = b1.z; bb[7] = b1.w;
                }
                uint4 o;
                __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    const float lo = __uint_as_float(wd[j] << 16), hi = __uint_as_float(wd[j] & 0xffff0000u);
                    float y0, y1;
                    if (ln) { y0 = fmaf(gg[2 * j], (lo - mean) * inv, bb[2 * j]); y1 = fmaf(gg[2 * j + 1], (hi - mean) * inv, bb[2 * j + 1]); }
                    else { y0 = lo * inv * gg[2 * j]; y1 = hi * inv * gg[2 * j + 1]; }
                    oh[j] = __floats2bfloat162_rn(y0, y1);
                }
                row[c] = o;
            }
        }
        __syncthreads();
    }

    for (int s0 = s_lo + warp; s0 < slices; s0 += kWarps * S) {
        if (s0 != s_lo + warp) load_weights(s0);
#pragma unroll
        for (int u = 0; u < S; u++) {
            const int s = s0 + u * kWarps;
            if (s >= slices) break;
#pragma unroll
            for (int i = 0; i < MT; i++) {
                const int r0 = 16 * i + g, r1 = r0 + 8;
                uint4 a0 = make_uint4(0, 0, 0, 0), a1 = make_uint4(0, 0, 0, 0);
                const bool live = 32 * s < k_mine;
                if (live && r0 < M) a0 = *reinterpret_cast<const uint4*>(a_base + (long long)r0 * a_ld + 32 * s + 8 * t);
                if (live && r1 < M) a1 = *reinterpret_cast<const uint4*>(a_base + (long long)r1 * a_ld + 32 * s + 8 * t);
                if (NORM == 0 && ext.act_off && live && 32 * s + 8 * t >= ext.act_from) {
                    if (r0 < M) a0 = relu_mul8(a0, *reinterpret_cast<const uint4*>(a_base + (long long)r0 * a_ld + ext.act_off + 32 * s + 8 * t));
                    if (r1 < M) a1 = relu_mul8(a1, *reinterpret_cast<const uint4*>(a_base + (long long)r1 * a_ld + ext.act_off + 32 * s + 8 * t));
                }
#pragma unroll
                for (int j = 0; j < NT; j++) {
                    mma_bf16_16x8x16(acc[i][j], a0.x, a1.x, a0.y, a1.y, wv[u][j].x, wv[u][j].y);
                    mma_bf16_16x8x16(acc[i][j], a0.z, a1.z, a0.w, a1.w, wv[u][j].z, wv[u][j].w);
                }
            }
        }
    }

#pragma unroll
    for (int i = 0; i < MT; i++)
#pragma unroll
        for (int j = 0; j < NT; j++) {
            red[warp][16 * i + g][8 * j + 2 * t] = acc[i][j][0];
            red[warp][16 * i + g][8 * j + 2 * t + 1] = acc[i][j][1];
            red[warp][16 * i + g + 8][8 * j + 2 * t] = acc[i][j][2];
            red[warp][16 * i + g + 8][8 * j + 2 * t + 1] = acc[i][j][3];
        }
    __syncthreads();
    float tot[EI];
#pragma unroll
    for (int it = 0; it < EI; it++) {
        const int e = tid + it * kWarps * 32;
        const int m = e / (NT * 8), nn = e % (NT * 8);
        tot[it] = 0.0f;
        if (m < MT * 16) {
            float sum = red[0][m][nn];
#pragma unroll
            for (int w = 1; w < kWarps; w++) sum += red[w][m][nn];
            tot[it] = sum;
        }
    }
    if constexpr (SPLITS) {
    if (ksplit > 1) {
        // the CTAs send their sums to the cluster's first one, which adds them in rank order (read by it instead, with a third barrier to keep
        // them: one sequence of a 12-layer, 768-wide model, 32 steps 9.95 against 9.75 ms)
        __shared__ float inbox[3][MT * 16][NT * 8 + 1];
        namespace cg = cooperative_groups;
        cg::cluster_group cluster = cg::this_cluster();
        sm100::cluster_wait();                            // every CTA of the cluster runs (arrived at the start)
        if (krank != 0) {
            float* to = cluster.map_shared_rank(&inbox[krank - 1][0][0], 0);
#pragma unroll
            for (int it = 0; it < EI; it++) {
                const int e = tid + it * kWarps * 32;
                if (e < MT * 16 * NT * 8) to[(e / (NT * 8)) * (NT * 8 + 1) + e % (NT * 8)] = tot[it];
            }
        }
        sm100::cluster_arrive();
        sm100::cluster_wait();
        if (krank != 0) return;
#pragma unroll
        for (int it = 0; it < EI; it++) {
            const int e = tid + it * kWarps * 32;
            if (e < MT * 16 * NT * 8)
                for (int r = 1; r < ksplit; r++) tot[it] += inbox[r - 1][e / (NT * 8)][e % (NT * 8)];
        }
    }
    }
#pragma unroll
    for (int it = 0; it < EI; it++) {
        const int e = tid + it * kWarps * 32;
        const int m = e / (NT * 8), nn = e % (NT * 8), n = n0 + nn;
        if (m >= M || n >= N || m >= MT * 16) continue;
        float v = fmaf(tot[it], alpha, bpre[it]);
        if (epilogue == EPI_GELU || epilogue == EPI_GELU_MUL) v = gelu_fast2(make_float2(v, 0.0f)).x;
        else if (epilogue == EPI_SWIGLU) v = silu_fast(v);
        else if (epilogue == EPI_RELU_MUL) v = fmaxf(v, 0.0f);
        if (R) v = epilogue_multiplies(epilogue) ? v * rpre[it] : v + rpre[it];
        if (grp.gate) v *= 1.0f / (1.0f + __expf(-__bfloat162float(grp.gate[(long long)m * grp.ld_gate + gi])));
        if (ext.c_f32) reinterpret_cast<float*>(C)[(long long)m * ldc + n] = v;
        else C[(long long)m * ldc + n] = __float2bfloat16_rn(v);
        if (ext.c2) ext.c2[(long long)m * ldc + n] = __float2bfloat16_rn(v);
    }
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// One row or a few: a warp takes R weight rows whole and, where the norm is inside (K <= 2048), normalises the input row by itself, in registers.
// What bounds such a launch is the chain behind its wait: the kernel above stages a row to normalise in shared memory, meets at four barriers and
// fetches the norm's weights behind them, and its warps' partial products meet once more; here nothing but the row itself is left to load, the
// two moments and the products are warp reductions, and there is no barrier.  Same values as there: centred deviations, rounded to bf16 before the
// product, f32 sums in another order.  Several rows: the warps of a CTA are dealt over (row, R weight rows), the same weights for its M warps
// next to each other.  NV: vectors of eight values a lane holds.
template <int NV, int R, bool NORM>
__global__ void __launch_bounds__(kWarps * 32, 2) linear_row_kernel(const __nv_bfloat16* A, long long lda, const __nv_bfloat16* __restrict__ W, long long ldb, void* C,
                                                                   long long ldc, const float* __restrict__ bias, const void* res, int M, int N, int K, float alpha,
                                                                   int epilogue, RowNorm nrm, int c_f32, __nv_bfloat16* c2) {
    pdl_release();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, m = warp % M, n0 = (blockIdx.x * (kWarps / M) + warp / M) * R, nvec = K >> 3;
    const bool ln = nrm.kind == 1;
    // weights, the norm's weights and the bias do not depend on the kernel before this one
    uint4 wv[R][NV];
#pragma unroll
    for (int j = 0; j < R; j++) {
        const __nv_bfloat16* w = W + (long long)min(n0 + j, N - 1) * ldb;
#pragma unroll
        for (int i = 0; i < NV; i++) {
            wv[j][i] = make_uint4(0, 0, 0, 0);
            if (32 * i + lane < nvec) wv[j][i] = M == 1 ? ld_stream(w + 8 * (32 * i + lane)) : __ldg(reinterpret_cast<const uint4*>(w + 8 * (32 * i + lane)));
        }
    }
    __shared__ float4 gg[2][NORM ? 32 * NV : 1], bb[2][NORM ? 32 * NV : 1];      // halves of every lane's vector (in registers they would cost the launch behind its place)
    if constexpr (NORM) for (int c = threadIdx.x; c < 64 * NV; c += blockDim.x) {
        const int e = c >> 1, h = c & 1;
        gg[h][e] = e < nvec ? __ldg(reinterpret_cast<const float4*>(nrm.gamma) + c) : make_float4(0, 0, 0, 0);
        if (ln) bb[h][e] = e < nvec ? __ldg(reinterpret_cast<const float4*>(nrm.beta) + c) : make_float4(0, 0, 0, 0);
    }
    const int n = n0 + lane;                                             // lane j finishes weight row j
    const bool mine = lane < R && n < N;
    const float b_mine = bias && mine ? __ldg(bias + n) : 0.0f;
    if constexpr (NORM) __syncthreads();
    pdl_acquire();
    auto widen = [](uint4 d, float2 (&f)[4]) {
        const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&d);
#pragma unroll
        for (int q = 0; q < 4; q++) f[q] = bf16x2_to_float2(e[q]);
    };
    uint4 x[NV];
#pragma unroll
    for (int i = 0; i < NV; i++) x[i] = 32 * i + lane < nvec ? *reinterpret_cast<const uint4*>(A + (long long)m * lda + 8 * (32 * i + lane)) : make_uint4(0, 0, 0, 0);
    const float r_mine = !(res && mine) ? 0.0f : c_f32 ? static_cast<const float*>(res)[(long long)m * ldc + n]
                                                       : __bfloat162float(static_cast<const __nv_bfloat16*>(res)[(long long)m * ldc + n]);
    float mean = 0.0f, inv = 1.0f;
    if constexpr (NORM) {
        // LayerNorm: the sum, then the squares of the deviations; RMSNorm: the squares
        float2 s2 = make_float2(0.0f, 0.0f), f[4];
        if (ln) {
#pragma unroll
            for (int i = 0; i < NV; i++) {
                widen(x[i], f);
#pragma unroll
                for (int q = 0; q < 4; q++) s2 = __fadd2_rn(s2, f[q]);
            }
            mean = warp_sum(s2.x + s2.y) / (float)K;
            s2 = make_float2(0.0f, 0.0f);
        }
#pragma unroll
        for (int i = 0; i < NV; i++) {
            if (32 * i + lane < nvec) {
                widen(x[i], f);
#pragma unroll
                for (int q = 0; q < 4; q++) { f[q] = __fadd2_rn(f[q], make_float2(-mean, -mean)); s2 = __ffma2_rn(f[q], f[q], s2); }
            }
        }
        inv = 1.0f / sqrtf(warp_sum(s2.x + s2.y) / (float)K + nrm.eps);
    }
    float2 dot[R];
#pragma unroll
    for (int j = 0; j < R; j++) dot[j] = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int i = 0; i < NV; i++) {
        float2 v[4], wf[4];
        widen(x[i], v);
        if constexpr (NORM) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const float4 g4 = gg[h][32 * i + lane], b4 = ln ? bb[h][32 * i + lane] : make_float4(0, 0, 0, 0);
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const float2 t = __fmul2_rn(__fadd2_rn(v[2 * h + q], make_float2(-mean, -mean)), make_float2(inv, inv)), g = q ? make_float2(g4.z, g4.w) : make_float2(g4.x, g4.y);
                    const float2 y = ln ? __ffma2_rn(g, t, q ? make_float2(b4.z, b4.w) : make_float2(b4.x, b4.y)) : __fmul2_rn(t, g);
                    v[2 * h + q] = bf16x2_to_float2(__floats2bfloat162_rn(y.x, y.y));       // as the stand-alone kernels store it
                }
            }
        }
#pragma unroll
        for (int j = 0; j < R; j++) {
            widen(wv[j][i], wf);
#pragma unroll
            for (int q = 0; q < 4; q++) dot[j] = __ffma2_rn(v[q], wf[q], dot[j]);
        }
    }
    float tot = 0.0f;
#pragma unroll
    for (int j = 0; j < R; j++) {
        const float d = warp_sum(dot[j].x + dot[j].y);
        if (lane == j) tot = d;
    }
    if (!mine) return;
    float y = fmaf(tot, alpha, b_mine);
    if (epilogue == EPI_GELU || epilogue == EPI_GELU_MUL) y = gelu_fast2(make_float2(y, 0.0f)).x;
    else if (epilogue == EPI_SWIGLU) y = silu_fast(y);
    else if (epilogue == EPI_RELU_MUL) y = fmaxf(y, 0.0f);
    if (res) y = epilogue_multiplies(epilogue) ? y * r_mine : y + r_mine;
    if (c_f32) static_cast<float*>(C)[(long long)m * ldc + n] = y;
    else static_cast<__nv_bfloat16*>(C)[(long long)m * ldc + n] = __float2bfloat16_rn(y);
    if (c2) c2[(long long)m * ldc + n] = __float2bfloat16_rn(y);
}
// Weight rows per warp: as few as leave twelve warps to an SM, and as the registers hold (up to 12 vectors of weights a lane; of 16 a few are spilled).
int row_group(const GemmDesc& d) {
    const long long outputs = (long long)d.M * d.N, warps = 12ll * rt().sm_count;
    const int most = d.K <= 1024 ? 4 : d.K <= 2048 ? 2 : 1;
    return std::min(most, outputs > 2 * warps ? 4 : outputs > warps ? 2 : 1);
}
// ... taken while all its CTAs are resident, two to an SM: every weight byte is then on its way before the wait, and a second wave would normalise
// the rows again.  One of a chain of launches with weights of its own, us (the kernel above or linear_stream.cu's / this one):
//   1 row:  768 x 768 2.8 / 1.6, 3072 x 768 3.2 / 2.0, 5120 x 768 3.5 / 2.2, 768 x 3072 3.8 / 2.3, 2048 x 2048 3.8 / 2.5; LayerNorm inside 2304 x 768
//           5.1 / 3.3, 5120 x 1024 6.5 / 3.9, RMSNorm inside 2304 x 768 4.2 / 2.9, 2048 x 2048 5.6 / 3.9
//   4 rows: 2304 x 768 3.3 / 2.4, 1024 x 2048 4.3 / 2.5, 768 x 3072 (384 CTAs) 3.8 / 4.0; LayerNorm inside 2304 x 768 6.0 / 3.7, 3072 x 768 (384) 5.9 / 6.4
//   8 rows: 1024 x 1024 3.2 / 2.3, 2304 x 768 (576) 3.4 / 4.0; LayerNorm inside 1024 x 1024 6.9 / 4.1, 2304 x 768 (576) 6.5 / 7.0
// Above 3072 a lane holds 13 .. 16 vectors of weights, which its 128 registers do not quite (72 bytes spilled); seven and eight rows then pay only with
// one CTA to an SM (8 rows, 148 x 4096 4.34 / 4.07, 296 x 4096 4.50 / 5.04; 6 rows, 296 x 4096 4.48 / 4.45; 4 rows, 592 x 4096 6.28 / 5.03; one row, 2368 x
// 4096 9.61 / 6.49, ordinary launches).
bool row_preferred(const GemmDesc& d, bool norm) {
    const int per_sm = d.K > 3072 && d.M > 6 ? 1 : 2;
    return !d.group && !d.act_off && d.M <= kWarps && d.K <= (norm ? 2048 : 4096) && ceil_div(d.N, kWarps / d.M * row_group(d)) <= per_sm * rt().sm_count;
}
template <int NV, bool NORM>
int launch_row(const GemmDesc& d, const RowNorm& nrm, bool dependent) {
    auto go = [&](auto kern, int r) {
        SPT_CUDA(launch_dependent(kern, dim3(ceil_div(d.N, kWarps / d.M * r)), dim3(kWarps / d.M * d.M * 32), 0, dependent, 1, static_cast<const __nv_bfloat16*>(d.A), d.lda,
                                  static_cast<const __nv_bfloat16*>(d.B), d.ldb, d.C, d.ldc, d.bias, d.R, d.M, d.N, d.K, d.alpha, d.epilogue, nrm, d.out_dtype == F32 ? 1 : 0,
                                  static_cast<__nv_bfloat16*>(d.C2)));
        note_submit();
        return 0;
    };
    const int r = row_group(d);
    if constexpr (NV <= 4) if (r == 4) return go(linear_row_kernel<NV, 4, NORM>, 4);
    if constexpr (NV <= 8) if (r == 2) return go(linear_row_kernel<NV, 2, NORM>, 2);
    return go(linear_row_kernel<NV, 1, NORM>, 1);
}
template <bool NORM>
int row(const GemmDesc& d, const RowNorm& nrm, bool dependent) {
    const int nv = ceil_div(d.K, 256);
    if (nv == 1) return launch_row<1, NORM>(d, nrm, dependent);
    if (nv == 2) return launch_row<2, NORM>(d, nrm, dependent);
    if (nv == 3) return launch_row<3, NORM>(d, nrm, dependent);
    if (nv == 4) return launch_row<4, NORM>(d, nrm, dependent);
    if (nv <= 6) return launch_row<6, NORM>(d, nrm, dependent);
    if constexpr (NORM) return launch_row<8, NORM>(d, nrm, dependent);
    else return nv <= 8 ? launch_row<8, NORM>(d, nrm, dependent) : nv <= 12 ? launch_row<12, NORM>(d, nrm, dependent) : launch_row<16, NORM>(d, nrm, dependent);
}

constexpr size_t kNormSmemLimit = 160 * 1024;
size_t norm_smem(const GemmDesc& d) { return (size_t)d.M * (d.K + 8) * 2; }

template <int MT, int NT, int NORM>
int launch(const GemmDesc& d, const RowNorm& nrm, bool dependent) {
    // Few weight rows and a long K (the projections back to the model width): clusters of 2 or 4 CTAs split K, so that the launch
    // still covers the SMs and a warp's share of K is one round of loads.  Not above 16 rows: what comes here then has a K of 512 at most (the
    // block-diagonal products over a latent), too little to split.
    int ksplit = 1;
    if constexpr (NORM == 0 && MT == 1) {
        const long long blocks = ceil_div(d.N, NT * 8);
        // (768 x 768 with one row: 2.8 us in a chain without the cluster, 3.2 with two CTAs; 768 x 3072 4.9 -> 4.3 with four)
        while (ksplit < 4 && blocks * ksplit * 2 <= 3ll * rt().sm_count && d.K / (ksplit * 2) >= 64 * kWarps) ksplit *= 2;
    }
    constexpr int S = NT == 1 ? 8 : NT == 2 ? 4 : 2;
    auto kern = linear_few_rows_kernel<MT, NT, S, NORM>;
    const size_t smem = NORM ? norm_smem(d) : 0;
    if constexpr (NORM) {
        static bool granted = false;                                   // per instantiation
        if (!granted) { SPT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kNormSmemLimit)); granted = true; }
    }
    const int grid = ceil_div(d.N, NT * 8) * ksplit;
    SPT_CUDA(launch_dependent(kern, dim3(grid), dim3(kWarps * 32), smem, dependent, ksplit,
                              static_cast<const __nv_bfloat16*>(d.A), d.lda, static_cast<const __nv_bfloat16*>(d.B), d.ldb, static_cast<__nv_bfloat16*>(d.C), d.ldc,
                              d.bias, static_cast<const __nv_bfloat16*>(d.R), d.M, d.N, d.K, d.alpha, d.epilogue, nrm, ksplit,
                              FewRowsGroups{d.group, d.group_a, d.group_c, static_cast<const __nv_bfloat16*>(d.gate), d.ld_gate},
                              FewRowsExtra{d.act_from, d.act_off, d.out_dtype == F32 ? 1 : 0, static_cast<__nv_bfloat16*>(d.C2)}));
    note_submit();
    return 0;
}

template <int NORM>
int dispatch(const GemmDesc& d, const RowNorm& nrm, bool dependent) {
    // CTAs: 8, 16 or 32 weight rows each, the widest that still gives every SM two CTAs (a short kernel: spread first)
    const long long want = 2ll * rt().sm_count;
    const int mt = d.M <= 16 ? 1 : d.M <= 32 ? 2 : 4;
    int nt = 1;
    if (ceil_div(d.N, 16) >= want && d.group % 16 == 0) nt = 2;
    if (mt <= 2 && ceil_div(d.N, 32) >= want && d.group % 32 == 0) nt = 4;
    if constexpr (NORM != 0) {       // at most kNormMaxRows = 16 rows: one row group
        return nt == 1 ? launch<1, 1, NORM>(d, nrm, dependent) : nt == 2 ? launch<1, 2, NORM>(d, nrm, dependent) : launch<1, 4, NORM>(d, nrm, dependent);
    } else {
        switch (mt * 10 + nt) {
            case 11: return launch<1, 1, 0>(d, nrm, dependent);
            case 12: return launch<1, 2, 0>(d, nrm, dependent);
            case 14: return launch<1, 4, 0>(d, nrm, dependent);
            case 21: return launch<2, 1, 0>(d, nrm, dependent);
            case 22: return launch<2, 2, 0>(d, nrm, dependent);
            case 24: return launch<2, 4, 0>(d, nrm, dependent);
            case 41: return launch<4, 1, 0>(d, nrm, dependent);
            default: return launch<4, 2, 0>(d, nrm, dependent);
        }
    }
}

// LayerNorm / RMSNorm of a handful of rows as a launch of its own (the row counts where normalising inside every CTA of the
// projection costs more than it saves; the pipelined kernel of rowops.cu spends longer setting up its ring than these rows take).
// What bounds it is the chain load - reduce - store: one CTA per row, NV vectors of eight values a thread, the norm weights requested
// ahead of the wait, one barrier (LayerNorm: every warp's mean and squared deviations, merged by Chan, Golub and LeVeque's update).  64 rows of
// 768 with LayerNorm in a chain of dependent launches: 3.4 us with a warp per row, two reductions and the weights fetched last, 2.0 us so.
template <int NV>
__global__ void __launch_bounds__(256) norm_few_rows_kernel(const __nv_bfloat16* x, __nv_bfloat16* out, int K, RowNorm nrm) {
    __shared__ float part[8][2];
    pdl_release();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, nvec = K >> 3, threads = blockDim.x;
    const bool ln = nrm.kind == 1;
    float gg[NV][8], bb[NV][8];
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int c = i * threads + tid;
#pragma unroll
        for (int j = 0; j < 8; j++) { gg[i][j] = 0.0f; bb[i][j] = 0.0f; }
        if (c < nvec) {
            const float4 g0 = __ldg(reinterpret_cast<const float4*>(nrm.gamma + 8 * c)), g1 = __ldg(reinterpret_cast<const float4*>(nrm.gamma + 8 * c + 4));
            gg[i][0] = g0.x; gg[i][1] = g0.y; gg[i][2] = g0.z; gg[i][3] = g0.w; gg[i][4] = g1.x; gg[i][5] = g1.y; gg[i][6] = g1.z; gg[i][7] = g1.w;
            if (ln) {
                const float4 b0 = __ldg(reinterpret_cast<const float4*>(nrm.beta + 8 * c)), b1 = __ldg(reinterpret_cast<const float4*>(nrm.beta + 8 * c + 4));
                bb[i][0] = b0.x; bb[i][1] = b0.y; bb[i][2] = b0.z; bb[i][3] = b0.w; bb[i][4] = b1.x; bb[i][5] = b1.y; bb[i][6] = b1.z; bb[i][7] = b1.w;
            }
        }
    }
    pdl_acquire();
    const uint4* src = reinterpret_cast<const uint4*>(x + (size_t)blockIdx.x * K);
    float v[NV][8];
    float sum = 0.0f;                                                    // LayerNorm: of the values, RMSNorm: of their squares
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int c = i * threads + tid;
        const uint4 d = c < nvec ? src[c] : make_uint4(0, 0, 0, 0);
        const uint32_t wd[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int j = 0; j < 4; j++) {
            v[i][2 * j] = __uint_as_float(wd[j] << 16); v[i][2 * j + 1] = __uint_as_float(wd[j] & 0xffff0000u);
            sum += ln ? v[i][2 * j] + v[i][2 * j + 1] : v[i][2 * j] * v[i][2 * j] + v[i][2 * j + 1] * v[i][2 * j + 1];
        }
    }
    // values of the row that warp w holds
    auto held = [&](int w) { int n = 0; for (int i = 0; i < NV; i++) n += 8 * max(0, min(32, nvec - i * threads - 32 * w)); return (float)n; };
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float n_mine = held(warp);
    if (ln) {
        const float mean = n_mine > 0.0f ? sum / n_mine : 0.0f;
        float m2 = 0.0f;
#pragma unroll
        for (int i = 0; i < NV; i++)
            if (i * threads + tid < nvec) {
#pragma unroll
                for (int j = 0; j < 8; j++) m2 += (v[i][j] - mean) * (v[i][j] - mean);
            }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m2 += __shfl_xor_sync(0xffffffffu, m2, o);
        if (lane == 0) { part[warp][0] = mean; part[warp][1] = m2; }
    } else if (lane == 0) part[warp][1] = sum;
    __syncthreads();
    // merged from the first warp's moments on: an empty set has no mean to be far from, and the square of a large mean need not be an f32
    float mean = ln ? part[0][0] : 0.0f, m2 = part[0][1], n = held(0);
    for (int w = 1; w < threads / 32; w++) {
        if (!ln) { m2 += part[w][1]; continue; }
        const float nw = held(w), d = part[w][0] - mean;
        if (nw == 0.0f) continue;
        const float f = nw / (n + nw);
        m2 += part[w][1] + d * d * n * f;
        mean += d * f;
        n += nw;
    }
    const float inv = 1.0f / sqrtf(m2 / (float)K + nrm.eps);
    uint4* dst = reinterpret_cast<uint4*>(out + (size_t)blockIdx.x * K);
#pragma unroll
    for (int i = 0; i < NV; i++) {
        const int c = i * threads + tid;
        if (c < nvec) {
            uint4 o;
            __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float y[2];
#pragma unroll
                for (int q = 0; q < 2; q++) {
                    const int e = 2 * j + q;
                    y[q] = ln ? fmaf(gg[i][e], (v[i][e] - mean) * inv, bb[i][e]) : v[i][e] * inv * gg[i][e];
                }
                oh[j] = __floats2bfloat162_rn(y[0], y[1]);
            }
            dst[c] = o;
        }
    }
}

}  // namespace

bool linear_few_rows_supported(const GemmDesc& d) {
    // SPTORCH_B200_FEW_ROWS: the largest row count that takes this kernel (0 = never; experiments)
    static const int max_rows = [] { const char* e = getenv("SPTORCH_B200_FEW_ROWS"); const int v = e ? atoi(e) : kDefaultMaxRows; return v < 0 ? 0 : v > 64 ? 64 : v; }();
    const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return d.mode == MM_BF16 && (d.out_dtype == BF16 || !d.group) && d.act_off % 8 == 0 && d.act_from % 8 == 0 && d.M >= 1 && d.M <= max_rows && d.N >= 1 && d.K >= 8 && d.K % 8 == 0 && d.nb1 * d.nb2 == 1 &&
           !d.causal_lower && !d.causal_k && !d.norm_axis && !d.reduce && d.lda % 8 == 0 && d.ldb % 8 == 0 && d.lda >= d.K && d.ldb >= d.K &&
           (d.group ? d.group > 0 && d.group % 8 == 0 && d.N % d.group == 0 && d.group_a % 8 == 0 && !d.R : d.ldc >= d.N) && al16(d.A) && al16(d.B) && d.C != nullptr;
}

bool linear_few_rows_norm_supported(const GemmDesc& d, const RowNorm& nrm) {
    if (d.act_off) return false;
    const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return linear_few_rows_supported(d) && (nrm.kind == 1 || nrm.kind == 2) && nrm.gamma && al16(nrm.gamma) && (nrm.kind == 2 || (nrm.beta && al16(nrm.beta))) &&
           (nrm.kind == 2 || d.K > kNormLaunchMaxK || row_preferred(d, true)) && d.M <= norm_inside_rows(nrm) && (long long)d.N * d.K <= kNormInsideWeights &&
           norm_smem(d) <= kNormSmemLimit;
}

bool norm_few_rows_supported(const void* x, const void* out, int rows, int K, const RowNorm& nrm) {
    const auto al16 = [](const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15) == 0; };
    return rows >= 1 && rows <= 64 && K % 8 == 0 && K >= 8 && K <= kNormLaunchMaxK && (nrm.kind == 1 || nrm.kind == 2) && nrm.gamma && al16(nrm.gamma) &&
           (nrm.kind == 2 || (nrm.beta && al16(nrm.beta))) && al16(x) && al16(out);
}

int norm_few_rows(const void* x, void* out, int rows, int K, const RowNorm& nrm, bool dependent) {
    if (!norm_few_rows_supported(x, out, rows, K, nrm)) return fail("norm_few_rows: unsupported problem");
    const dim3 grid(rows), block(std::min(256, ceil_div(K / 8, 32) * 32));
    const __nv_bfloat16* xp = static_cast<const __nv_bfloat16*>(x);
    __nv_bfloat16* op = static_cast<__nv_bfloat16*>(out);
    if (K <= 2048) SPT_CUDA(launch_dependent(norm_few_rows_kernel<1>, grid, block, 0, dependent, 1, xp, op, K, nrm));
    else SPT_CUDA(launch_dependent(norm_few_rows_kernel<2>, grid, block, 0, dependent, 1, xp, op, K, nrm));
    note_submit();
    return 0;
}

int linear_few_rows(const GemmDesc& d, const RowNorm* nrm, bool dependent) {
    if (nrm && nrm->kind) {
        if (!linear_few_rows_norm_supported(d, *nrm)) return fail("linear_few_rows: unsupported problem (normalised rows)");
        if (row_preferred(d, true)) return row<true>(d, *nrm, dependent);
        if (linear_stream_preferred(d, nrm, dependent)) return linear_stream(d, nrm, dependent);
        return dispatch<1>(d, *nrm, dependent);
    }
    if (!linear_few_rows_supported(d)) return fail("linear_few_rows: unsupported problem");
    if (row_preferred(d, false)) return row<false>(d, RowNorm{}, dependent);
    if (linear_stream_preferred(d, nullptr, dependent)) return linear_stream(d, nullptr, dependent);
    return dispatch<0>(d, RowNorm{}, dependent);
}

}  // namespace spt
