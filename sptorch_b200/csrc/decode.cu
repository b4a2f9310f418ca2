// decode.cu -- single-token attention over a key/value cache (crates/nn/src/lib.rs:706-760, causal_attention_last_token).
//
// One warp per (sequence, head).  The query (hd values) sits in shared memory; lanes take cached positions p = lane,
// lane+32, ... for the scores (each reads one contiguous K row of hd elements), the scores are normalised with two warp
// reductions, and for the weighted sum every lane owns hd/32 output columns and walks the positions (coalesced V rows).
// HBM-bound: the cache is read once: 2 * n * hd * sizeof(T) bytes per (sequence, head).
// Cache layout: [layer][sequence][position][H*hd] (position-major rows, as the HAL spec describes for devices:
// crates/hal/src/lib.rs:129-303), so appending a token is one row write per layer.
#include "common.h"
#include "pdl.cuh"
#include "sm100.cuh"
#include "../../include/sptorch_b200_ext.h"
#include <math.h>

namespace spt {

constexpr int kDecThreads = 128;    // 4 warps = 4 (sequence, head) pairs per CTA

template <typename T>
__global__ void __launch_bounds__(kDecThreads) attention_last_token_kernel(const T* __restrict__ q, long long ld_q, const T* __restrict__ kc,
                                                                           const T* __restrict__ vc, T* __restrict__ out, long long ld_out,
                                                                           int B, int H, int hd, int n, long long seq_stride, long long row_stride,
                                                                           float scale, const int* __restrict__ state, int n_cap) {
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // decode graphs: the number of valid positions lives in a device word; shared memory is sized for the cache capacity
    if (state) n = state[1];
    float* qs = sm + warp * (hd + (state ? n_cap : n));
    float* sc = qs + hd;
    const int pair = blockIdx.x * (kDecThreads / 32) + warp;
    if (pair >= B * H) return;
    const int b = pair / H, h = pair % H;
    const T* qp = q + (long long)b * ld_q + (long long)h * hd;
    for (int d = lane; d < hd; d += 32) qs[d] = (float)qp[d];
    __syncwarp();
    const T* kb = kc + (long long)b * seq_stride + (long long)h * hd;
    const T* vb = vc + (long long)b * seq_stride + (long long)h * hd;
    float mx = -INFINITY;
    for (int p = lane; p < n; p += 32) {
        const T* kr = kb + (long long)p * row_stride;
        float dot = 0.0f;
        for (int d = 0; d < hd; d++) dot += qs[d] * (float)kr[d];
        dot *= scale;
        sc[p] = dot;
        mx = fmaxf(mx, dot);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    float den = 0.0f;
    for (int p = lane; p < n; p += 32) { float e = expf(sc[p] - mx); sc[p] = e; den += e; }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) den += __shfl_xor_sync(0xffffffffu, den, o);
    __syncwarp();
    const float inv = 1.0f / den;
    T* op = out + (long long)b * ld_out + (long long)h * hd;
    for (int d = lane; d < hd; d += 32) {
        float acc = 0.0f;
        for (int p = 0; p < n; p++) acc += (sc[p] * inv) * (float)vb[(long long)p * row_stride + d];
        op[d] = (T)acc;
    }
}

// q: [B, ld_q] (head h at columns h*hd); kc/vc: first cached row of this layer, rows of H*hd elements, sequences
// seq_stride apart; n cached positions (the newest included); out: [B, ld_out]
// The same function for head sizes up to 128 whose rows are 16 .. 512 bytes (a power of two): the form the decode step uses.
// One CTA of 4 or 16 warps per (sequence, head).  A row of K or V is read by LPR = row bytes / 16 neighbouring lanes with one
// 16-byte load each, so a warp fetches 32 / LPR whole rows per instruction, fully coalesced, and four positions are in flight per
// lane (sixteen warps cover 256 positions of 128-byte rows per turn: the walk over a 1024-position cache is four dependent
// rounds of loads, not thirty); the dot product is finished with log2(LPR) shuffles.  Every row group keeps a running (maximum,
// sum, weighted value sum) over the positions it visits (online softmax), the groups of a warp and then the warps are merged at
// the end.  Same result as the kernel above up to the order of the f32 sums.
// What bounds it with few sequences is the chain from q to the output: the four positions of a round share one update of the maximum,
// warps are merged one output column per thread, and a cluster's CTAs send their results to the first one, counted on its barrier as they land.
// rope (optional): base^(2p / hd); q and the fresh key are rotated to position state[0], the angles ahead of the wait.
// fresh_k / fresh_v (optional): the newest token's key / value, still in the projection output (rows of ld_fresh elements, head h
// at columns h*hd).  The CTA copies its head's part into cache row `slot` and uses the fresh rows for that position, which
// saves the append launch in front of the attention.
// The first round of cache rows is requested before the programmatic-launch wait: cache rows other than `slot` were written by
// earlier steps, only q and the fresh rows come from the kernel before this one.
// HBM traffic: 2 * n * hd * sizeof(T) bytes per (sequence, head), read once.
constexpr int kRowsMaxWarps = 16;
// The warps' (maximum, sum, value sums) -> the CTA's, one output column per thread, and the CTAs' of the cluster, sent to the first one
template <int NW, typename F>
__device__ __forceinline__ void merge_parts(const float* sm, float* res, uint64_t* inbox, volatile int* abort_flag, uint32_t* status, int splits, int rank, int hd, F store) {
    const int col = threadIdx.x;
    float cm = -INFINITY, cl = 0.0f, co = 0.0f;
    auto gather = [&](const float* set, int count) {
        cm = -INFINITY; cl = 0.0f; co = 0.0f;
        for (int w = 0; w < count; w++) cm = fmaxf(cm, set[w * 130]);
        for (int w = 0; w < count; w++) {
            const float f = set[w * 130] == -INFINITY ? 0.0f : expf(set[w * 130] - cm);
            cl += f * set[w * 130 + 1];
            co += f * set[w * 130 + 2 + col];
        }
    };
    if (col < hd) gather(sm, NW);
    if (splits > 1) {
        sm100::cluster_wait();                           // every CTA of the cluster runs and has its barrier (arrived at the start)
        if (col < hd) {
            const uint32_t bar = sm100::mapa(sm100::smem_u32(inbox), 0), to = sm100::mapa(sm100::smem_u32(res + rank * 130), 0);
            if (col == 0) { sm100::send4(to, bar, cm); sm100::send4(to + 4, bar, cl); }
            sm100::send4(to + 8 + 4 * col, bar, co);
        }
        if (rank != 0) return;
        if (!sm100::mbar_wait_warp(sm100::ClusterBar{sm100::smem_u32(inbox)}, 0, abort_flag, status, sm100::kErrEpilogueWait)) {
            // given up: the others may still send here.  This CTA stays until they have left, which is their arrival, and what they sent has landed
            sm100::cluster_sync();
            const unsigned long long t0 = sm100::globaltimer();
            while (sm100::globaltimer() - t0 < 200000ull) { }
            return;
        }
        if (col < hd) gather(res, splits);
    }
    if (col < hd) store(col, co * (1.0f / cl));
}
// NW: warps per CTA.  Four-warp CTAs are held to 80 registers so that six share an SM (888 CTA slots: the 768 (sequence, head)
// pairs of 64 sequences x 12 heads run as one wave; at 92 registers and five per SM they made two).
template <typename T, int NW>
__global__ void __launch_bounds__(NW * 32, NW == 4 ? 6 : 1) attention_last_token_rows_kernel(const T* q, long long ld_q, const T* kc,
                                                                                      const T* vc, T* out, long long ld_out, int H, int hd,
                                                                                      int n, long long seq_stride, long long row_stride, float scale,
                                                                                      const int* __restrict__ state, const T* fresh_k,
                                                                                      const T* fresh_v, long long ld_fresh, int slot, T* kc_w, T* vc_w, int splits,
                                                                                      const float* __restrict__ rope, uint32_t* status) {
    constexpr int VE = 16 / (int)sizeof(T);              // elements per 16-byte segment
    constexpr int U = 4;                                 // positions in flight per row group
    __shared__ float res[8 * 130];                       // the cluster's first CTA: maximum, sum and value sums of every CTA
    __shared__ float sm[NW * 130];                       // per warp: maximum, sum, up to 128 value sums
    __shared__ __align__(8) uint64_t inbox;              // the first CTA: counts what lands in res
    __shared__ volatile int abort_flag;
    pdl_release();
    if (splits > 1) {
        if (threadIdx.x == 0) {
            abort_flag = 0;
            sm100::mbar_init(sm100::smem_u32(&inbox), 1);
            sm100::fence_barrier_init();
            sm100::mbar_expect_tx(sm100::smem_u32(&inbox), (uint32_t)(splits * (hd + 2) * 4));
        }
        sm100::cluster_arrive();
    }
    if (state) { n = state[1]; slot = state[2]; }        // written before the step's first kernel was launched
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    constexpr int nw = NW;
    const int lpr = hd / VE;                             // lanes per row
    const int rpi = 32 / lpr;                            // rows per warp instruction
    const int seg = lane % lpr, grp = lane / lpr;
    // a cluster of `splits` CTAs shares one (sequence, head): CTA r of it walks the r-th part of the positions
    const int pair = blockIdx.x / splits, rank = blockIdx.x % splits;
    const int b = pair / H, h = pair % H;
    const int part = (n + splits - 1) / splits, lo = rank * part, hi = min(n, lo + part);
    auto widen = [](uint4 raw, float (&f)[VE]) {
        if constexpr (sizeof(T) == 2) {
            const __nv_bfloat162* e = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int i = 0; i < 4; i++) { const float2 a = bf16x2_to_float2(e[i]); f[2 * i] = a.x; f[2 * i + 1] = a.y; }
        } else {
            f[0] = __uint_as_float(raw.x); f[1] = __uint_as_float(raw.y); f[2] = __uint_as_float(raw.z); f[3] = __uint_as_float(raw.w);
        }
    };
    const T* kb = kc + (long long)b * seq_stride + (long long)h * hd + seg * VE;
    const T* vb = vc + (long long)b * seq_stride + (long long)h * hd + seg * VE;
    const int stride = nw * rpi;
    uint4 kr[U], vr[U];
    // dead positions get no weight and read row 0 (always valid); values of bf16 caches are zeros there, so that an infinite one in row 0 stays in its column
    // (with it f32 is 1 to 2 % behind)
    auto fetch_k = [&](int base) {
#pragma unroll
        for (int u = 0; u < U; u++) { const int p = base + u * stride + grp; kr[u] = *reinterpret_cast<const uint4*>(kb + (p < hi ? p : 0) * row_stride); }
    };
    auto fetch_v = [&](int base) {
#pragma unroll
        for (int u = 0; u < U; u++) { const int p = base + u * stride + grp; vr[u] = p < hi || sizeof(T) == 4 ? *reinterpret_cast<const uint4*>(vb + (p < hi ? p : 0) * row_stride) : make_uint4(0, 0, 0, 0); }
    };
    const int first = lo + warp * rpi;
    if (first < hi) { fetch_k(first); fetch_v(first); }
    // rotation of the query and of the key about to be cached, as rope.cu does it in place: the angles depend on the position alone
    float sn[VE / 2], cs[VE / 2];
    if (rope) {
        const float pos = (float)state[0];
#pragma unroll
        for (int i = 0; i < VE / 2; i++) sincosf(pos / rope[seg * (VE / 2) + i], &sn[i], &cs[i]);
    }
    auto rotate = [&](uint4& raw) {
        if constexpr (sizeof(T) == 2) {
            __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 a = bf16x2_to_float2(e[i]);
                e[i] = __floats2bfloat162_rn(__fsub_rn(__fmul_rn(a.x, cs[i]), __fmul_rn(a.y, sn[i])), __fadd_rn(__fmul_rn(a.x, sn[i]), __fmul_rn(a.y, cs[i])));
            }
        } else {
            float* e = reinterpret_cast<float*>(&raw);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const float ev = e[2 * i], od = e[2 * i + 1];
                e[2 * i] = __fsub_rn(__fmul_rn(ev, cs[i]), __fmul_rn(od, sn[i]));
                e[2 * i + 1] = __fadd_rn(__fmul_rn(ev, sn[i]), __fmul_rn(od, cs[i]));
            }
        }
    };
    pdl_acquire();
    uint4 q_raw = *reinterpret_cast<const uint4*>(q + (long long)b * ld_q + (long long)h * hd + seg * VE);
    uint4 fk = make_uint4(0, 0, 0, 0), fv = fk;
    if (fresh_k) {
        fk = *reinterpret_cast<const uint4*>(fresh_k + (long long)b * ld_fresh + (long long)h * hd + seg * VE);
        fv = *reinterpret_cast<const uint4*>(fresh_v + (long long)b * ld_fresh + (long long)h * hd + seg * VE);
    }
    if (rope) { rotate(q_raw); rotate(fk); }
    float qf[VE];
    widen(q_raw, qf);
    if (fresh_k && rank == 0 && warp == 0 && grp == 0) {
        const long long dst = (long long)b * seq_stride + (long long)slot * row_stride + (long long)h * hd + seg * VE;
        *reinterpret_cast<uint4*>(kc_w + dst) = fk;
        *reinterpret_cast<uint4*>(vc_w + dst) = fv;
    }
    float m = -INFINITY, l = 0.0f, o[VE];
#pragma unroll
    for (int i = 0; i < VE; i++) o[i] = 0.0f;
    // Warp-uniform trip count (the shuffles are warp-wide).  The positions of a round share one update of the running maximum, and the next
    // round's keys and values are requested as soon as this one's have been read.
    for (int base = first; base < hi; base += U * stride) {
        const int next = base + U * stride;
        float s[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool is_fresh = fresh_k != nullptr && base + u * stride + grp == slot;
            float kf[VE];
            widen(is_fresh ? fk : kr[u], kf);
            s[u] = 0.0f;
#pragma unroll
            for (int i = 0; i < VE; i++) s[u] += qf[i] * kf[i];
        }
        if (next < hi) fetch_k(next);
        for (int off = lpr >> 1; off > 0; off >>= 1) {
#pragma unroll
            for (int u = 0; u < U; u++) s[u] += __shfl_xor_sync(0xffffffffu, s[u], off);
        }
        float mn = m;
#pragma unroll
        for (int u = 0; u < U; u++) {
            s[u] = base + u * stride + grp < hi ? s[u] * scale : -INFINITY;
            mn = fmaxf(mn, s[u]);
        }
        const float ref = mn == -INFINITY ? 0.0f : mn;               // nothing seen yet: every weight below is exp(-inf) = 0
        const float corr = expf(m - ref);
        l *= corr;
#pragma unroll
        for (int i = 0; i < VE; i++) o[i] *= corr;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const bool is_fresh = fresh_k != nullptr && base + u * stride + grp == slot;
            const float pr = expf(s[u] - ref);
            float vf[VE];
            widen(is_fresh ? fv : vr[u], vf);
            l += pr;
#pragma unroll
            for (int i = 0; i < VE; i++) o[i] += pr * vf[i];
        }
        if (next < hi) fetch_v(next);
        m = mn;
    }
    // merge the row groups of the warp (groups that saw no position carry m = -inf, l = 0)
    {
        float mx = m;
        for (int off = lpr; off < 32; off <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, off));
        const float f = m == -INFINITY ? 0.0f : expf(m - mx);
        l *= f;
#pragma unroll
        for (int i = 0; i < VE; i++) o[i] *= f;
        for (int off = lpr; off < 32; off <<= 1) {
            l += __shfl_xor_sync(0xffffffffu, l, off);
#pragma unroll
            for (int i = 0; i < VE; i++) o[i] += __shfl_xor_sync(0xffffffffu, o[i], off);
        }
        m = mx;
    }
    // ... then the warps, one output column per thread, and the CTAs of the cluster, whose results are sent to the first one
    float* mine = sm + warp * 130;
    if (grp == 0) {
        if (seg == 0) { mine[0] = m; mine[1] = l; }
#pragma unroll
        for (int i = 0; i < VE; i++) mine[2 + seg * VE + i] = o[i];
    }
    __syncthreads();
    merge_parts<NW>(sm, res, &inbox, &abort_flag, status, splits, rank, hd, [&](int col, float v) { out[(long long)b * ld_out + (long long)h * hd + col] = (T)v; });
}

// The same for bf16 caches on mma.sync, heads of 64 and 128 above all (fragments_preferred).  With the rows of 64 sequences in flight the walk above is bound by its instructions (two widenings and two
// multiply-adds an element pair, three shuffles a position): here a warp takes sixteen positions at a time, keys and values go from global memory
// straight into fragments (a sum over k does not care about its order), and neither the query nor a weight loses a bit: the query and the
// rows are bf16 as they are, a weight is three bf16 parts that add up to its 24 bits, in three columns of one instruction.
//   S = K q: rows = positions g and g + 8, k slot (lane 4 g + t; elements 8 t .. 8 t + 7 of a 32-element slice), column 0 = the query
//   o = V^T p: row g of tile j = dimension 64 (j / 4) + 8 g + 2 (j % 4), row g + 8 the one behind it, k = positions, columns 0 .. 2 = the parts of p
// NS: 32-element slices, NB: 64-element blocks of a head.  One of a chain of launches, us (the walk above / this one): 12 pairs of heads of 64, 520
// positions 3.7 / 2.8, 1000 positions 3.7 / 3.1; 96 pairs, 520 6.5 / 5.9; 192 pairs, 400 7.0 / 6.2; 768 pairs, 144 8.2 / 7.2;
// 128 pairs of heads of 128, 272 7.7 / 6.9; 512 pairs, 200 17.2 / 15.8.
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// A lane's part of a pair of weights -- column 0: their upper eight bits, 1: the next eight, 2: the last eight, each exact (the others are not read).  The
// lower parts are kept from being zero (2^-126 is far below what an f32 weight can say), so that an infinite value stays one.
struct WeightPart {
    uint32_t past_first, past_second;
    __device__ __forceinline__ explicit WeightPart(int column) : past_first(column >= 1 ? 0xffff0000u : 0u), past_second(column >= 2 ? 0xffff0000u : 0u) {}
    __device__ __forceinline__ float one(float x) const {
        x -= __uint_as_float(__float_as_uint(x) & past_first);
        x -= __uint_as_float(__float_as_uint(x) & past_second);
        return x + __uint_as_float(0x00800000u & past_first);
    }
    __device__ __forceinline__ uint32_t pair(float x, float y) const { return __byte_perm(__float_as_uint(one(x)), __float_as_uint(one(y)), 0x7632); }
};
// CTAs of NW warps that an SM holds, which the rule below counts on and the compiler is held to: heads of 128 took 175 registers where three CTAs of four
// warps leave 168, and what was to run at once ran as two waves (8 layers with 16 heads of 128, a prompt and 32 steps: 12 sequences behind 1024
// positions 29.9 ms, 27.4 so; 10 behind 256 16.3, 15.1; 6 behind 1024 20.8, 18.8).
constexpr int mma_ctas_per_sm(int hd, int warps) { return hd <= 64 ? (warps == 4 ? 6 : warps == 8 ? 2 : 1) : warps == 4 ? 3 : 1; }
template <int NS, int NB, int NW>
__global__ void __launch_bounds__(NW * 32, mma_ctas_per_sm(NS * 32, NW)) attention_last_token_mma_kernel(const __nv_bfloat16* q, long long ld_q, const __nv_bfloat16* kc,
                                                                                                    const __nv_bfloat16* vc, __nv_bfloat16* out, long long ld_out, int H, int hd,
                                                                                                    int n, long long seq_stride, long long row_stride, float scale,
                                                                                                    const int* __restrict__ state, const __nv_bfloat16* fresh_k,
                                                                                                    const __nv_bfloat16* fresh_v, long long ld_fresh, int slot,
                                                                                                    __nv_bfloat16* kc_w, __nv_bfloat16* vc_w, int splits,
                                                                                                    const float* __restrict__ rope, uint32_t* status) {
    __shared__ float res[8 * 130];                       // as above
    __shared__ __align__(8) float sm[NW * 130];          // as above; pairs of value sums are stored at once
    __shared__ __align__(16) float cs[64], sn[64];
    __shared__ __align__(16) __nv_bfloat16 kf[NS * 32], vf[NB * 64];         // the newest position's rows
    __shared__ __align__(8) uint64_t inbox;
    __shared__ volatile int abort_flag;
    pdl_release();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    if (splits > 1) {
        if (tid == 0) {
            abort_flag = 0;
            sm100::mbar_init(sm100::smem_u32(&inbox), 1);
            sm100::fence_barrier_init();
            sm100::mbar_expect_tx(sm100::smem_u32(&inbox), (uint32_t)(splits * (hd + 2) * 4));
        }
        sm100::cluster_arrive();
    }
    if (state) { n = state[1]; slot = state[2]; }        // written before the step's first kernel was launched
    const int pair = blockIdx.x / splits, rank = blockIdx.x % splits, b = pair / H, h = pair % H;
    const int part = ((n + splits - 1) / splits + 15) / 16 * 16, lo = rank * part, hi = min(n, lo + part);
    const __nv_bfloat16* kb = kc + (long long)b * seq_stride + (long long)h * hd;
    const __nv_bfloat16* vb = vc + (long long)b * seq_stride + (long long)h * hd;
    const uint4 zero4 = make_uint4(0, 0, 0, 0);
    uint4 kr[2][NS], vr[4][NB];
    // keys k0 + g and k0 + 8 + g; values of positions k0 + 2t, 2t + 1, 2t + 8, 2t + 9
    auto fetch_keys = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int p = k0 + 8 * i + g;
            const __nv_bfloat16* row = kb + (long long)p * row_stride + 8 * t;
#pragma unroll
            for (int s = 0; s < NS; s++) kr[i][s] = p < hi && 32 * s + 8 * t < hd ? *reinterpret_cast<const uint4*>(row + 32 * s) : zero4;
        }
    };
    auto fetch_values = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int p = k0 + 2 * t + (i & 1) + 8 * (i >> 1);
            const __nv_bfloat16* row = vb + (long long)p * row_stride + 8 * g;
#pragma unroll
            for (int s = 0; s < NB; s++) vr[i][s] = p < hi && 64 * s + 8 * g < hd ? *reinterpret_cast<const uint4*>(row + 64 * s) : zero4;
        }
    };
    constexpr int step = NW * 16;
    const int first = lo + warp * 16;
    // rows other than `slot` were written by earlier steps: requested ahead of the wait
    if (first < hi) { fetch_keys(first); fetch_values(first); }
    if (rope) {
        if (tid < hd / 2) sincosf((float)state[0] / rope[tid], &sn[tid], &cs[tid]);
        __syncthreads();
    }
    // the warp that meets the newest position takes its rows from the projections, the cluster's first warp puts them into the cache
    const bool meets = fresh_k != nullptr && slot >= lo && slot < hi && ((slot - lo) / 16) % NW == warp, writes = fresh_k != nullptr && rank == 0 && warp == 0;
    pdl_acquire();
    uint4 qf[NS];
#pragma unroll
    for (int s = 0; s < NS; s++) qf[s] = 32 * s + 8 * t < hd ? *reinterpret_cast<const uint4*>(q + (long long)b * ld_q + (long long)h * hd + 32 * s + 8 * t) : zero4;
    uint4 fk[NS], fv[NB];
    if (meets || writes) {
#pragma unroll
        for (int s = 0; s < NS; s++) fk[s] = 32 * s + 8 * t < hd ? *reinterpret_cast<const uint4*>(fresh_k + (long long)b * ld_fresh + (long long)h * hd + 32 * s + 8 * t) : zero4;
#pragma unroll
        for (int s = 0; s < NB; s++) fv[s] = 64 * s + 8 * g < hd ? *reinterpret_cast<const uint4*>(fresh_v + (long long)b * ld_fresh + (long long)h * hd + 64 * s + 8 * g) : zero4;
    }
    if (rope) {
        auto rotate = [&](uint4& raw, int s) {
            __nv_bfloat162* e = reinterpret_cast<__nv_bfloat162*>(&raw);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 a = bf16x2_to_float2(e[i]);
                const int at = min(16 * s + 4 * t + i, 63);
                const float c = cs[at], w = sn[at];
                e[i] = __floats2bfloat162_rn(__fsub_rn(__fmul_rn(a.x, c), __fmul_rn(a.y, w)), __fadd_rn(__fmul_rn(a.x, w), __fmul_rn(a.y, c)));
            }
        };
#pragma unroll
        for (int s = 0; s < NS; s++)
            if (32 * s + 8 * t < hd) { rotate(qf[s], s); if (meets || writes) rotate(fk[s], s); }
    }
    if (writes) {
        const long long dst = (long long)b * seq_stride + (long long)slot * row_stride + (long long)h * hd;
#pragma unroll
        for (int s = 0; s < NS; s++) if (g == 0 && 32 * s + 8 * t < hd) *reinterpret_cast<uint4*>(kc_w + dst + 32 * s + 8 * t) = fk[s];
#pragma unroll
        for (int s = 0; s < NB; s++) if (t == 0 && 64 * s + 8 * g < hd) *reinterpret_cast<uint4*>(vc_w + dst + 64 * s + 8 * g) = fv[s];
    }
    if (meets) {
#pragma unroll
        for (int s = 0; s < NS; s++) if (g == 0) *reinterpret_cast<uint4*>(kf + 32 * s + 8 * t) = fk[s];
#pragma unroll
        for (int s = 0; s < NB; s++) if (t == 0) *reinterpret_cast<uint4*>(vf + 64 * s + 8 * g) = fv[s];
        __syncwarp();
    }
#pragma unroll
    for (int s = 0; s < NS; s++) if (g != 0) qf[s] = zero4;              // column 0 alone
    float acc[4 * NB][4];
#pragma unroll
    for (int j = 0; j < 4 * NB; j++)
#pragma unroll
        for (int e = 0; e < 4; e++) acc[j][e] = 0.0f;
    const WeightPart mine_of(g);
    float m = -INFINITY, l = 0.0f;
    for (int k0 = first; k0 < hi; k0 += step) {
        if (meets && slot - k0 >= 0 && slot - k0 < 16) {
            const int d = slot - k0;
#pragma unroll
            for (int i = 0; i < 2; i++)
                if (8 * i + g == d) {
#pragma unroll
                    for (int s = 0; s < NS; s++) kr[i][s] = *reinterpret_cast<const uint4*>(kf + 32 * s + 8 * t);
                }
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (2 * t + (i & 1) + 8 * (i >> 1) == d) {
#pragma unroll
                    for (int s = 0; s < NB; s++) vr[i][s] = *reinterpret_cast<const uint4*>(vf + 64 * s + 8 * g);
                }
        }
        float s4[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
        for (int s = 0; s < NS; s++) {
            mma_16x8x16(s4, kr[0][s].x, kr[1][s].x, kr[0][s].y, kr[1][s].y, qf[s].x, qf[s].y);
            mma_16x8x16(s4, kr[0][s].z, kr[1][s].z, kr[0][s].w, kr[1][s].w, qf[s].z, qf[s].w);
        }
        if (k0 + step < hi) fetch_keys(k0 + step);                       // in flight while the softmax and P V run
        // column 0 lies with the lanes t = 0: every lane takes the four positions whose values it holds
        float p[4];
        p[0] = __shfl_sync(0xffffffffu, s4[0], 8 * t); p[1] = __shfl_sync(0xffffffffu, s4[0], 8 * t + 4);
        p[2] = __shfl_sync(0xffffffffu, s4[2], 8 * t); p[3] = __shfl_sync(0xffffffffu, s4[2], 8 * t + 4);
        float mn = m;
#pragma unroll
        for (int i = 0; i < 4; i++) {
            p[i] = k0 + 2 * t + (i & 1) + 8 * (i >> 1) < hi ? p[i] * scale : -INFINITY;
            mn = fmaxf(mn, p[i]);
        }
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 1));
        mn = fmaxf(mn, __shfl_xor_sync(0xffffffffu, mn, 2));
        const float ref = mn == -INFINITY ? 0.0f : mn;
        const float corr = expf(m - ref);
        m = mn;
        l *= corr;
#pragma unroll
        for (int i = 0; i < 4; i++) { p[i] = expf(p[i] - ref); l += p[i]; }
        const uint32_t b0 = mine_of.pair(p[0], p[1]), b1 = mine_of.pair(p[2], p[3]);
#pragma unroll
        for (int j = 0; j < 4 * NB; j++) {
            const uint32_t* v0 = reinterpret_cast<const uint32_t*>(&vr[0][j / 4]);
            const uint32_t* v1 = reinterpret_cast<const uint32_t*>(&vr[1][j / 4]);
            const uint32_t* v2 = reinterpret_cast<const uint32_t*>(&vr[2][j / 4]);
            const uint32_t* v3 = reinterpret_cast<const uint32_t*>(&vr[3][j / 4]);
#pragma unroll
            for (int e = 0; e < 4; e++) acc[j][e] *= corr;
            mma_16x8x16(acc[j], __byte_perm(v0[j % 4], v1[j % 4], 0x5410), __byte_perm(v0[j % 4], v1[j % 4], 0x7632), __byte_perm(v2[j % 4], v3[j % 4], 0x5410),
                        __byte_perm(v2[j % 4], v3[j % 4], 0x7632), b0, b1);
        }
        if (k0 + step < hi) fetch_values(k0 + step);
    }
    l += __shfl_xor_sync(0xffffffffu, l, 1);
    l += __shfl_xor_sync(0xffffffffu, l, 2);
    // the parts' columns: 0 and 1 lie with t = 0, 2 with t = 1 (the others hold zeros times the values, which are not zeros if a value is infinite)
    float* mine = sm + warp * 130;
    if (lane == 0) { mine[0] = m; mine[1] = l; }
#pragma unroll
    for (int j = 0; j < 4 * NB; j++) {
        float x = acc[j][0] + (t == 0 ? acc[j][1] : 0.0f), y = acc[j][2] + (t == 0 ? acc[j][3] : 0.0f);
        x += __shfl_xor_sync(0xffffffffu, x, 1);
        y += __shfl_xor_sync(0xffffffffu, y, 1);
        if (t == 0 && 64 * (j / 4) + 8 * g < hd) *reinterpret_cast<float2*>(mine + 2 + 64 * (j / 4) + 8 * g + 2 * (j % 4)) = make_float2(x, y);
    }
    __syncthreads();
    merge_parts<NW>(sm, res, &inbox, &abort_flag, status, splits, rank, hd, [&](int col, float v) { out[(long long)b * ld_out + (long long)h * hd + col] = __float2bfloat16_rn(v); });
}

// Device-resident state of a decode step replayed as a CUDA graph: {absolute position, valid cached positions (new token
// included), ring slot the new token's key / value go to, row of the position table}.
__global__ void decode_state_kernel(int* state, int pos, int n, int slot, int pos_row) {
    state[0] = pos; state[1] = n; state[2] = slot; state[3] = pos_row;
}
int decode_state_launch(int* state, int pos, int n, int slot, int pos_row) {
    decode_state_kernel<<<1, 1, 0, rt().stream>>>(state, pos, n, slot, pos_row);
    SPT_LAUNCH_CHECK("decode_state");
    return 0;
}

// key and value of the new token of every sequence ([q | k | v] rows of 3*dl elements) into cache row `slot` (slot_dev overrides)
template <typename T>
__global__ void __launch_bounds__(256) kv_append_kernel(const T* __restrict__ qkv, T* __restrict__ kc, T* __restrict__ vc, int B, int dl, long long seq_stride,
                                                        int slot, const int* __restrict__ state) {
    if (state) slot = state[2];
    const int vec = 16 / (int)sizeof(T);
    const int per_row = dl / vec;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < B * per_row; i += gridDim.x * blockDim.x) {
        const int b = i / per_row, c = (i - b * per_row) * vec;
        const T* src = qkv + (long long)b * 3 * dl;
        const long long dst = (long long)b * seq_stride + (long long)slot * dl + c;
        *reinterpret_cast<uint4*>(kc + dst) = *reinterpret_cast<const uint4*>(src + dl + c);
        *reinterpret_cast<uint4*>(vc + dst) = *reinterpret_cast<const uint4*>(src + 2 * dl + c);
    }
}
int kv_append_launch(const void* qkv, void* kc, void* vc, int B, int dl, long long seq_stride, int slot, const int* state, int dtype) {
    const int vec = dtype == BF16 ? 8 : 4;
    if (dl % vec) return fail("kv_append: row width %d is not a multiple of %d", dl, vec);
    const int work = B * (dl / vec);
    const int grid = (work + 255) / 256;
    if (dtype == BF16) kv_append_kernel<__nv_bfloat16><<<grid, 256, 0, rt().stream>>>((const __nv_bfloat16*)qkv, (__nv_bfloat16*)kc, (__nv_bfloat16*)vc, B, dl, seq_stride, slot, state);
    else kv_append_kernel<float><<<grid, 256, 0, rt().stream>>>((const float*)qkv, (float*)kc, (float*)vc, B, dl, seq_stride, slot, state);
    SPT_LAUNCH_CHECK("kv_append");
    return 0;
}

// Keys and values of a whole prompt ([q | k | v] rows of 3*dl elements, T per sequence) into cache rows 0 .. T-1 of every sequence.  HBM-bound;
// one launch per layer (64 sequences of 128 tokens took 128 strided copies of 4 us each).
__global__ void __launch_bounds__(256) kv_fill_kernel(const uint4* qkv, uint4* kc, uint4* vc, long long rows, int T, int per_row,
                                                      long long seq_stride) {
    pdl_release();
    pdl_acquire();
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= rows * per_row) return;
    const long long r = i / per_row, c = i - r * per_row, b = r / T, dst = b * seq_stride + (r - b * T) * per_row + c;
    const uint4 k = qkv[(3 * r + 1) * per_row + c], v = qkv[(3 * r + 2) * per_row + c];
    kc[dst] = k;
    vc[dst] = v;
}
// false: the rows are no multiples of 16 bytes
bool kv_fill_supported(const void* qkv, const void* kc, const void* vc, size_t row_bytes) {
    return row_bytes % 16 == 0 && ((reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc)) & 15) == 0;
}
int kv_fill_launch(const void* qkv, void* kc, void* vc, int B, int T, size_t row_bytes, long long cache_rows) {
    const int per_row = (int)(row_bytes / 16);
    const long long work = (long long)B * T * per_row;
    SPT_CUDA(launch_dependent(kv_fill_kernel, dim3((unsigned)((work + 255) / 256)), dim3(256), 0, short_launch(0.0, 64.0 * work), 1, (const uint4*)qkv, (uint4*)kc, (uint4*)vc, (long long)B * T, T, per_row, cache_rows * per_row));
    note_submit();
    return 0;
}

// true when the coalesced kernel (the one that can also take the newest token's key / value rows straight from the projection
// output) serves this head size: rows of 16 .. 512 bytes, a power of two
bool attention_last_token_takes_fresh(int hd, int dtype) {
    const size_t rb = (size_t)hd * (dtype == BF16 ? 2 : 4);
    return rb >= 16 && rb <= 512 && hd <= 128 && (rb & (rb - 1)) == 0;
}

// bf16: whether tensor-core fragments or the walk by rows serves heads of hd over span positions, `pairs` (sequence, head)s at once.  Fragments are sixteen
// positions of 64 or 128 elements whatever hd is, a row group of the walk is as many lanes as a row has: small heads leave the fragments
// empty, and four-warp CTAs of the walk share an SM by sixes where heads of 128 take three.  One of a chain of launches, us (walk / fragments):
//   heads of 8:    33 pairs 64 positions 2.31 / 2.15, 520 3.50 / 3.81, 2000 3.60 / 5.07; 2112 pairs 64 positions 8.8 / 8.3, 520 17.9 / 38.9
//   heads of 32:   16 pairs 1000 positions 3.93 / 3.28; 48 pairs 256 3.40 / 2.77, 400 3.41 / 3.70, 1000 4.68 / 5.33; 768 pairs 64 4.09 / 3.54, 520 11.4 / 16.9
//   heads of 64:   fragments throughout (12 pairs 520 positions 3.80 / 2.93; 768 pairs 144 8.1 / 7.4)
//   heads of 128:  384 pairs 64 positions 5.3 / 4.3; 512 pairs 64 6.1 / 7.1, 144 12.3 / 13.4, 256 18.4 / 18.2; 1024 pairs 16 6.0 / 8.6, 256 31.1 / 30.0
static bool fragments_preferred(int hd, int span, long long pairs) {
    if (hd > 64) return pairs <= (long long)mma_ctas_per_sm(hd, 4) * rt().sm_count || span >= 200;
    return hd > 32 || span <= 64 || (hd > 16 && pairs * span <= 16384);
}

// state / n_cap: when state is given, n and the ring slot are read from state[1] / state[2] at run time; n_cap is the cache capacity
// fresh_k / fresh_v / ld_fresh / slot: see the kernel; dependent: launched as a programmatic dependent of the kernel before it
int attention_last_token(const void* q, long long ld_q, const void* kc, const void* vc, void* out, long long ld_out, int B, int H, int hd,
                         int n, long long seq_stride, long long row_stride, int dtype, const int* state, int n_cap,
                         const void* fresh_k, const void* fresh_v, long long ld_fresh, int slot, bool dependent, const float* rope) {
    if (B <= 0 || H <= 0 || n <= 0) return fail("attention_last_token: empty cache or batch");
    {
        // rows of 16 .. 512 bytes, a power of two, everything 16-byte aligned: the coalesced kernel
        const size_t es = dtype == BF16 ? 2 : 4;
        const bool aligned = ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(kc) | reinterpret_cast<uintptr_t>(vc) | reinterpret_cast<uintptr_t>(out) |
                               reinterpret_cast<uintptr_t>(fresh_k) | reinterpret_cast<uintptr_t>(fresh_v)) & 15) == 0 &&
                             (ld_q * es) % 16 == 0 && (ld_out * es) % 16 == 0 && (seq_stride * es) % 16 == 0 && (row_stride * es) % 16 == 0 && (ld_fresh * es) % 16 == 0;
        if (attention_last_token_takes_fresh(hd, dtype) && aligned) {
            const float scale = 1.0f / sqrtf((float)hd);
            // Few (sequence, head) pairs: a cluster of up to eight CTAs shares each pair, with four, eight or sixteen warps per CTA -- whichever
            // combination walks the cache in the fewest dependent rounds while all CTAs are resident at once.  A round costs about as much
            // as four doublings of the cluster size; clusters of eight fill three quarters of the SMs at most (16 of them with a CTA alone on its
            // SM made two waves), seven eighths with six CTAs to an SM (2000 positions, 96 pairs 16 warps x 1 13.6, 4 x 8 11.0; 108 pairs 14.0, 16.7).  Measured in a chain, us: 12 pairs of heads of 64, 520 positions: 16 warps x 4 2.96, 8 x 8 2.88, 8 x 4 3.60, 16 x 1
            // 5.2; 96 pairs, 520: 4 x 8 6.0, 16 x 1 6.5, 4 x 4 7.1; 192 pairs, 400: 4 x 4 6.6, 8 x 1 7.5, 4 x 8 (1536 CTAs) 8.8; 16 pairs of heads of
            // 128, 2000: 4 x 8 8.8, 8 x 8 12.2.
            const int span = state ? n_cap : n;
            const long long pairs = (long long)B * H, sms = rt().sm_count;
            const bool mma = dtype == BF16 && fragments_preferred(hd, span, pairs);
            const int per_warp_round = mma ? 16 : (32 / (hd / (16 / (int)es))) * 4;
            int splits = 1, threads = 128, best = INT32_MAX;
            for (int sp = 1, log2sp = 0; sp <= 8; sp *= 2, log2sp++)
                for (int nw = 4; nw <= kRowsMaxWarps; nw *= 2) {
                    if (mma ? nw == 16 && hd > 64 : nw == 8) continue;
                    const long long slots = sms * (mma ? mma_ctas_per_sm(hd, nw) : nw == 4 ? 6 : 1);
                    const long long ctas = pairs * sp, cap = mma && sp == 8 ? slots * (hd <= 64 && nw == 4 ? 7 : 6) / 8 : slots;
                    if (ctas > cap && !(sp == 1 && nw == 4)) continue;
                    const int rounds = ceil_div(span, (long long)sp * nw * per_warp_round);
                    const int score = rounds * 8 + (nw == 16 ? 2 : 0) + (mma ? 2 : 6) * log2sp;
                    if (score < best) { best = score; splits = sp; threads = nw * 32; }
                }
#define SPT_ROWS_LAUNCH(T_, NW_)                                                                                                                  \
    SPT_CUDA(launch_dependent(attention_last_token_rows_kernel<T_, NW_>, dim3(B * H * splits), dim3(NW_ * 32), 0, dependent, splits, (const T_*)q, ld_q,  \
                              (const T_*)kc, (const T_*)vc, (T_*)out, ld_out, H, hd, n, seq_stride, row_stride, scale, state, (const T_*)fresh_k,         \
                              (const T_*)fresh_v, ld_fresh, slot, (T_*)const_cast<void*>(kc), (T_*)const_cast<void*>(vc), splits, rope, rt().dev_status))
#define SPT_MMA_LAUNCH(NS_, NB_, NW_)                                                                                                                 \
    SPT_CUDA(launch_dependent(attention_last_token_mma_kernel<NS_, NB_, NW_>, dim3(B * H * splits), dim3(NW_ * 32), 0, dependent, splits,                     \
                              (const __nv_bfloat16*)q, ld_q, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc, (__nv_bfloat16*)out, ld_out, H, hd, n, seq_stride,  \
                              row_stride, scale, state, (const __nv_bfloat16*)fresh_k, (const __nv_bfloat16*)fresh_v, ld_fresh, slot,                              \
                              (__nv_bfloat16*)const_cast<void*>(kc), (__nv_bfloat16*)const_cast<void*>(vc), splits, rope, rt().dev_status))
            if (mma) {
                if (hd <= 64) { if (threads == 128) SPT_MMA_LAUNCH(2, 1, 4); else if (threads == 256) SPT_MMA_LAUNCH(2, 1, 8); else SPT_MMA_LAUNCH(2, 1, 16); }
                else { if (threads == 128) SPT_MMA_LAUNCH(4, 2, 4); else SPT_MMA_LAUNCH(4, 2, 8); }
            } else if (dtype == BF16) { if (threads == 128) SPT_ROWS_LAUNCH(__nv_bfloat16, 4); else SPT_ROWS_LAUNCH(__nv_bfloat16, kRowsMaxWarps); }
            else if (threads == 128) SPT_ROWS_LAUNCH(float, 4);
            else SPT_ROWS_LAUNCH(float, kRowsMaxWarps);
#undef SPT_MMA_LAUNCH
#undef SPT_ROWS_LAUNCH
            note_submit();
            return 0;
        }
    }
    if (fresh_k || fresh_v || rope) return fail("attention_last_token: the newest token's rows can only be taken from the projection output for 16 .. 512-byte head rows");
    const size_t smem = (size_t)(kDecThreads / 32) * (hd + (state ? n_cap : n)) * sizeof(float);
    if (smem > 200 * 1024) return fail("attention_last_token: %d cached positions exceed the shared-memory score buffer", n);
    const int grid = ceil_div((long long)B * H, kDecThreads / 32);
    const float scale = 1.0f / sqrtf((float)hd);
    if (dtype == BF16) {
        auto kern = attention_last_token_kernel<__nv_bfloat16>;
        if (smem > 48 * 1024) SPT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, kDecThreads, smem, rt().stream>>>((const __nv_bfloat16*)q, ld_q, (const __nv_bfloat16*)kc, (const __nv_bfloat16*)vc,
                                                       (__nv_bfloat16*)out, ld_out, B, H, hd, n, seq_stride, row_stride, scale, state, n_cap);
    } else {
        auto kern = attention_last_token_kernel<float>;
        if (smem > 48 * 1024) SPT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        kern<<<grid, kDecThreads, smem, rt().stream>>>((const float*)q, ld_q, (const float*)kc, (const float*)vc, (float*)out, ld_out, B, H, hd, n,
                                                       seq_stride, row_stride, scale, state, n_cap);
    }
    SPT_LAUNCH_CHECK("attention_last_token");
    return 0;
}

}  // namespace spt

using namespace spt;

extern "C" int sptorch_ext_attention_last_token(const void* q, const void* k_cache, const void* v_cache, void* out, size_t B, size_t H, size_t hd,
                                                size_t n, size_t cache_positions, int dtype) {
    if (enter()) return 1;
    if (!q || !k_cache || !v_cache || !out) return fail("attention_last_token: null handle");
    if (dtype != SPT_F32 && dtype != SPT_BF16) return fail("attention_last_token: unknown dtype %d", dtype);
    if (n == 0 || n > cache_positions) return fail("attention_last_token: n must be in 1..cache_positions");
    const long long d = (long long)(H * hd);
    return attention_last_token(q, d, k_cache, v_cache, out, d, (int)B, (int)H, (int)hd, (int)n, (long long)cache_positions * d, d, dtype, nullptr, 0,
                                nullptr, nullptr, 0, 0, false, nullptr);
}
