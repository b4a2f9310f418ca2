// linear_stream.cu -- Linear for at most 64 input rows on the tensor cores, the weights as the wide operand:
//   C[m, n] = act(alpha * sum_k A[m,k] W[n,k] + bias[n]) (+ / * R[m,n]),   M <= 64, bf16 operands, bf16 or f32 output.
//
// With so few rows the product is a stream over the weight matrix: 2 N K bytes read once.  One CTA takes 128 weight rows and a part of
// K; a cluster of up to eight CTAs shares the 128 rows and splits K, so that the launch covers the SMs whatever N is.
//   warp 0      TMA producer: 128 x 64 weight tiles (and the TN x 64 tile of A beside each) into a ring; the ring is filled with weights
//               before the programmatic-launch wait, since no earlier kernel writes them
//   warp 1      tcgen05.mma with the weights as the 128-row operand and the input rows as its N = TN columns, accumulator in TMEM
//   all warps   TMEM -> the sums [input row][weight row] f32, each sent into the shared memory of the CTA that finishes the row and counted on
//               its barrier (a barrier of the cluster behind remote stores took 0.8 us longer); there they are added in rank order, so the
//               result does not depend on scheduling
// PAIR: two weight matrices against the same rows, two accumulators; the second product is the factor of the gated epilogue.
// NORM (at most 12 rows): the rows are normalised on the way in (RowNorm kinds 1 and 2).  Every CTA takes the statistics of the whole
// rows and normalises its own part of K into the operand tiles.
#include "gemm.h"
#include "epilogue_math.cuh"
#include "pdl.cuh"
#include "sm100.cuh"
#include <algorithm>

namespace spt {

using namespace sm100;

namespace {

constexpr int kTileRows = 128, kBK = 64;
// 64 input rows: what lies behind the products is a few hundred instructions a thread, and four warps a scheduler hide what two cannot (768 x 768
// 4.7 -> 4.5 us in a chain, 2304 x 768 5.7 -> 5.3, 3072 x 768 5.4 -> 5.0, 2048 x 2048 5.8 -> 5.4; 32 rows 768 x 768 3.4 -> 3.5, so not there)
constexpr int threads_of(int tn) { return tn == 64 ? 512 : 256; }
constexpr int kWeightBytes = kTileRows * kBK * 2;
constexpr int kMaxStages = 8, kMaxSplit = 8, kNormRows = 16;

struct StreamParams {
    void* C; const float* bias; const void* R; __nv_bfloat16* c2; const float* bias2;
    int M, N, K;
    long long ldc;
    float alpha;
    int epilogue, c_f32, ahead;              // ahead: weights beyond the ring are requested into L2 before the wait
    int split, per_cta, num_kb, stages;      // CTAs per cluster, k-blocks (of 64) per CTA and in all, ring depth
    int share, inbox;                        // input rows every CTA of the cluster finishes; offset of the partial sums in shared memory
    const __nv_bfloat16* A; long long lda;   // NORM: the rows before normalisation
    RowNorm nrm;
    uint32_t* status;
};

// sum, mean and squared deviations of two sets of values -> of their union (Chan, Golub and LeVeque's update)
struct Moments { float n, mean, m2; };
__device__ __forceinline__ Moments merge(const Moments& a, const Moments& b) {
    const float n = a.n + b.n;
    if (a.n == 0.0f || b.n == 0.0f) return a.n == 0.0f ? b : a;             // an empty set has no mean to be far from
    const float d = b.mean - a.mean, f = b.n / n;
    return {n, a.mean + d * f, a.m2 + b.m2 + d * d * a.n * f};
}
__device__ __forceinline__ void widen8(uint4 d, float (&v)[8]) {
    const uint32_t w[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
    for (int j = 0; j < 4; j++) { v[2 * j] = __uint_as_float(w[j] << 16); v[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u); }
}

template <int TN, bool NORM, bool PAIR>
__global__ void __launch_bounds__(threads_of(TN)) linear_stream_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmW2, const __grid_constant__ CUtensorMap tmA,
                                                                 const __grid_constant__ StreamParams p) {
    constexpr int ROW_BYTES = TN * kBK * 2;                                  // one k-block of A
    constexpr int WEIGHTS = PAIR ? 2 * kWeightBytes : kWeightBytes, STAGE = WEIGHTS + (NORM ? 0 : ROW_BYTES);
    constexpr uint32_t IDESC = make_idesc(false, kTileRows, TN);
    constexpr uint32_t COLS = (PAIR ? 2 : 1) * TN < 32 ? 32 : (PAIR ? 2 : 1) * TN;
    constexpr int THREADS = threads_of(TN), HALF = TN / (THREADS / 128);     // TMEM columns a warp reads
    extern __shared__ __align__(1024) uint8_t smem[];                        // [ring | NORM: k-blocks of A | partial sums, see below]
    __shared__ __align__(8) uint64_t bars[2 * kMaxStages + 2];
    __shared__ uint32_t tmem_slot;
    __shared__ volatile int abort_flag;
    const uint32_t base = smem_u32(smem), bar_full = smem_u32(bars), bar_empty = bar_full + 8 * kMaxStages, bar_done = bar_empty + 8 * kMaxStages,
                   bar_inbox = bar_done + 8;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int split = p.split, rank = (int)(blockIdx.x % (unsigned)split), n0 = (int)(blockIdx.x / (unsigned)split) * kTileRows;
    const int kb_lo = rank * p.per_cta, n_kb = min(p.num_kb, kb_lo + p.per_cta) - kb_lo, stages = p.stages;

    if (tid == 0) {
        for (int s = 0; s < stages; s++) { mbar_init(bar_full + 8 * s, 1); mbar_init(bar_empty + 8 * s, 1); }
        mbar_init(bar_done, 1);
        mbar_init(bar_inbox, 1);
        abort_flag = (base & 1023u) ? 1 : 0;
        if (base & 1023u) atomicOr(p.status, 0x200u);
        fence_barrier_init();
        // all sums of the rows this CTA finishes, its own among them: [sender][four rows][weight row][row] f32
        // (a CTA without a cluster stores its own)
        const int quads_mine = max(0, min(p.share, p.M - rank * p.share) + 3) >> 2;
        mbar_expect_tx(bar_inbox, (uint32_t)(split * quads_mine * kTileRows * 16 * (PAIR ? 2 : 1)));
    }
    if (warp == 1) { tmem_alloc(smem_u32(&tmem_slot), COLS); tmem_relinquish(); }
    if (warp == 0 && lane == 0) { tma_prefetch_desc(&tmW); if (!NORM) tma_prefetch_desc(&tmA); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    bool ok = abort_flag == 0;
    if (split > 1) cluster_arrive();      // met again before the first sum is sent: a CTA's shared memory is only written once it runs
    pdl_release();           // after the TMEM allocation: a successor that holds TMEM waits for this grid, never the other way round

    const int first = min(stages, n_kb);
    if (warp == 0 && ok && elect_one_sync()) {
        for (int s = 0; s < first; s++) {
            mbar_expect_tx(bar_full + 8 * s, STAGE);
            tma_load_4d(base + s * STAGE, &tmW, bar_full + 8 * s, (kb_lo + s) * kBK, n0, 0, 0);
            if constexpr (PAIR) tma_load_4d(base + s * STAGE + kWeightBytes, &tmW2, bar_full + 8 * s, (kb_lo + s) * kBK, n0, 0, 0);
        }
        // what the ring does not hold yet waits in L2: the memory works on while the launch before this one finishes
        for (int i = first; i < n_kb && p.ahead; i++) {
            tma_prefetch_l2_4d(&tmW, (kb_lo + i) * kBK, n0, 0, 0);
            if constexpr (PAIR) tma_prefetch_l2_4d(&tmW2, (kb_lo + i) * kBK, n0, 0, 0);
        }
    }
    __syncwarp();
    // NORM: this thread's 16-byte column piece of the CTA's part of K, with its norm weights (not written by any kernel), and the rows it takes
    const int nch = n_kb * 8, across = min(nch, THREADS), down = THREADS / across, c_mine = tid % across, r_mine = tid / across;
    const bool ln = p.nrm.kind == 1;
    float gg[8], bb[8];
    auto norm_weights = [&](int c) {
        const int k = kb_lo * kBK + 8 * c;
#pragma unroll
        for (int j = 0; j < 8; j++) { gg[j] = 0.0f; bb[j] = 0.0f; }
        if (k < p.K) {
            const float4 g0 = __ldg(reinterpret_cast<const float4*>(p.nrm.gamma + k)), g1 = __ldg(reinterpret_cast<const float4*>(p.nrm.gamma + k + 4));
            gg[0] = g0.x; gg[1] = g0.y; gg[2] = g0.z; gg[3] = g0.w; gg[4] = g1.x; gg[5] = g1.y; gg[6] = g1.z; gg[7] = g1.w;
            if (ln) {
                const float4 b0 = __ldg(reinterpret_cast<const float4*>(p.nrm.beta + k)), b1 = __ldg(reinterpret_cast<const float4*>(p.nrm.beta + k + 4));
                bb[0] = b0.x; bb[1] = b0.y; bb[2] = b0.z; bb[3] = b0.w; bb[4] = b1.x; bb[5] = b1.y; bb[6] = b1.z; bb[7] = b1.w;
            }
        }
    };
    if constexpr (NORM) norm_weights(c_mine);
    pdl_acquire();
    if constexpr (!NORM) {
        if (warp == 0 && ok && elect_one_sync())
            for (int s = 0; s < first; s++) tma_load_4d(base + s * STAGE + WEIGHTS, &tmA, bar_full + 8 * s, (kb_lo + s) * kBK, 0, 0, 0);
        __syncwarp();
    }
    const uint32_t rows_base = NORM ? base + stages * STAGE : 0u;            // NORM: k-block i of A at rows_base + i * ROW_BYTES
    if constexpr (NORM) {
        __shared__ Moments part[kNormRows][8];
        __shared__ float2 stat[kNormRows];                                   // (mean, 1 / sqrt(var + eps)); RMSNorm: mean 0
        constexpr int KEEP = 4;                                              // pieces requested with the rows' statistics
        uint4 kept[KEEP];
        auto piece = [&](int r, int c) {
            const int k = kb_lo * kBK + 8 * c;
            return r < p.M && r_mine < down && k < p.K ? *reinterpret_cast<const uint4*>(p.A + (long long)r * p.lda + k) : make_uint4(0, 0, 0, 0);
        };
#pragma unroll
        for (int i = 0; i < KEEP; i++) kept[i] = piece(r_mine + i * down, c_mine);
        const int P = p.M >= 8 ? 1 : p.M >= 4 ? 2 : p.M >= 2 ? 4 : 8, RP = 8 / P, my_p = warp % P, my_r = warp / P;
        const int nvec = p.K >> 3, per = (nvec + P - 1) / P, c_begin = my_p * per, c_end = min(nvec, c_begin + per);
        for (int r = my_r; r < p.M; r += RP) {
            const uint4* src = reinterpret_cast<const uint4*>(p.A + (long long)r * p.lda);
            Moments mo = {0.0f, 0.0f, 0.0f};
            for (int c0 = c_begin + lane; c0 - lane < c_end; c0 += 256) {
                uint4 d[8];
#pragma unroll
                for (int u = 0; u < 8; u++) d[u] = c0 + 32 * u < c_end ? src[c0 + 32 * u] : make_uint4(0, 0, 0, 0);
                Moments mc = {0.0f, 0.0f, 0.0f};
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    float v[8];
                    widen8(d[u], v);
                    if (c0 + 32 * u < c_end) mc.n += 8.0f;
#pragma unroll
                    for (int j = 0; j < 8; j++) mc.mean += ln ? v[j] : v[j] * v[j];
                }
                if (ln) {
                    mc.mean = mc.n > 0.0f ? mc.mean / mc.n : 0.0f;
#pragma unroll
                    for (int u = 0; u < 8; u++) {
                        float v[8];
                        widen8(d[u], v);
                        if (c0 + 32 * u < c_end) {
#pragma unroll
                            for (int j = 0; j < 8; j++) mc.m2 += (v[j] - mc.mean) * (v[j] - mc.mean);
                        }
                    }
                    mo = merge(mo, mc);
                } else mo.m2 += mc.mean;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                Moments other = {__shfl_xor_sync(0xffffffffu, mo.n, o), __shfl_xor_sync(0xffffffffu, mo.mean, o), __shfl_xor_sync(0xffffffffu, mo.m2, o)};
                if (ln) mo = merge(mo, other); else mo.m2 += other.m2;
            }
            if (lane == 0) part[r][my_p] = mo;
        }
        __syncthreads();
        if (tid < p.M) {
            Moments mo = part[tid][0];
            for (int q = 1; q < P; q++) { if (ln) mo = merge(mo, part[tid][q]); else mo.m2 += part[tid][q].m2; }
            stat[tid] = make_float2(mo.mean, 1.0f / sqrtf(mo.m2 / (float)p.K + p.nrm.eps));
        }
        __syncthreads();
        auto normalise = [&](int r, int c, uint4 d) {
            float v[8];
            widen8(d, v);
            const float2 st = stat[r];
            uint4 o;
            __nv_bfloat162* oh = reinterpret_cast<__nv_bfloat162*>(&o);
#pragma unroll
            for (int j = 0; j < 4; j++) {
                float y[2];
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const int q = 2 * j + i;
                    y[i] = ln ? fmaf(gg[q], (v[q] - st.x) * st.y, bb[q]) : v[q] * st.y * gg[q];
                }
                oh[j] = __floats2bfloat162_rn(y[0], y[1]);
            }
            if (kb_lo * kBK + 8 * c >= p.K) o = make_uint4(0, 0, 0, 0);
            *reinterpret_cast<uint4*>(smem + (uint32_t)(stages * STAGE + (c >> 3) * ROW_BYTES + r * 128 + (((c & 7) ^ (r & 7)) << 4))) = o;
        };
        if (r_mine < down) {
#pragma unroll
            for (int i = 0; i < KEEP; i++) if (r_mine + i * down < p.M) normalise(r_mine + i * down, c_mine, kept[i]);
            for (int r = r_mine + KEEP * down; r < p.M; r += down) normalise(r, c_mine, piece(r, c_mine));
            for (int c = c_mine + THREADS; c < nch; c += THREADS) {        // parts of K of more than 256 pieces: down is 1
                norm_weights(c);
                for (int r = 0; r < p.M; r++) normalise(r, c, piece(r, c));
            }
        }
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();
    }

    if (warp == 0) {                                     // one thread, like the issuer below
        if (ok && elect_one_sync()) {
            int stage = 0; uint32_t phase = 0;
            for (int i = first; i < n_kb; i++) {
                ok = mbar_wait(bar_empty + 8 * stage, phase, &abort_flag, p.status, kErrProducerWait);
                if (!ok) break;
                mbar_expect_tx(bar_full + 8 * stage, STAGE);
                tma_load_4d(base + stage * STAGE, &tmW, bar_full + 8 * stage, (kb_lo + i) * kBK, n0, 0, 0);
                if constexpr (PAIR) tma_load_4d(base + stage * STAGE + kWeightBytes, &tmW2, bar_full + 8 * stage, (kb_lo + i) * kBK, n0, 0, 0);
                if constexpr (!NORM) tma_load_4d(base + stage * STAGE + WEIGHTS, &tmA, bar_full + 8 * stage, (kb_lo + i) * kBK, 0, 0, 0);
                if (++stage == stages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        if (ok && elect_one_sync()) {
            int stage = 0; uint32_t phase = 0;
            for (int i = 0; i < n_kb; i++) {
                if (!wait_alone(bar_full + 8 * stage, phase, &abort_flag, p.status, kErrMmaWait)) break;
                tc_fence_after();
                const uint64_t wd = make_kmajor_sw128_desc(base + stage * STAGE);
                const uint64_t ad = make_kmajor_sw128_desc(NORM ? rows_base + i * ROW_BYTES : base + stage * STAGE + WEIGHTS);
#pragma unroll
                for (int k = 0; k < kBK / 16; k++) mma_ss<false>(tmem, wd + 2 * k, ad + 2 * k, IDESC, (i | k) != 0 ? 1u : 0u);
                if constexpr (PAIR) {
                    const uint64_t wd2 = make_kmajor_sw128_desc(base + stage * STAGE + kWeightBytes);
#pragma unroll
                    for (int k = 0; k < kBK / 16; k++) mma_ss<false>(tmem + TN, wd2 + 2 * k, ad + 2 * k, IDESC, (i | k) != 0 ? 1u : 0u);
                }
                mma_commit(bar_empty + 8 * stage);
                if (i == n_kb - 1) mma_commit(bar_done);
                if (++stage == stages) { stage = 0; phase ^= 1; }
            }
        }
        __syncwarp();
    }
    // What the rows this thread finishes are joined with, requested before their sums are there: item i is (four rows, weight row) number tid + THREADS i
    // of this CTA's share: all there are from a split of two up (a load left for the end costs 0.7 us).
    const int quads = p.share >> 2, set = split * quads * kTileRows;         // PAIR: the second product's sums are a set of their own
    constexpr int AHEAD = 2;
    float bias_pre[AHEAD];
    uint32_t res_pre[AHEAD][4];                                                  // as they come: f32 or bf16 bits
    auto joined = [&](int e, float& b, uint32_t (&x)[4]) {
        const int m0 = rank * p.share + (e / kTileRows) * 4, n = n0 + (e & (kTileRows - 1));
        const bool live = e < quads * kTileRows && n < p.N;
        const long long at = (long long)m0 * p.ldc + n;
        b = live && p.bias ? __ldg(p.bias + n) : 0.0f;
#pragma unroll
        for (int j = 0; j < 4; j++)
            x[j] = PAIR || !(live && p.R && m0 + j < p.M) ? 0u : p.c_f32 ? reinterpret_cast<const uint32_t*>(p.R)[at + j * p.ldc] : reinterpret_cast<const uint16_t*>(p.R)[at + j * p.ldc];
    };
#pragma unroll
    for (int i = 0; i < AHEAD; i++) joined(tid + i * THREADS, bias_pre[i], res_pre[i]);
    // Every CTA finishes `share` of the input rows (a multiple of four): all send it their sums of those rows, sixteen bytes a thread, a warp's
    // stores 512 contiguous bytes, counted on the receiver's barrier as they land.
    if (split > 1) cluster_wait();
    ok = mbar_wait_warp(bar_done, 0, &abort_flag, p.status, kErrEpilogueWait);
    tc_fence_after();
    const float4* sums = reinterpret_cast<const float4*>(smem + p.inbox);
    for (int which = 0; which < (PAIR ? 2 : 1) && ok; which++) {
        const int quarter = warp & 3, c0 = (warp >> 2) * HALF;
        uint32_t v[HALF];
        tmem_ld_32xN(tmem + ((uint32_t)(quarter * 32) << 16) + which * TN + c0, v);
        tmem_ld_wait();
        int owner = c0 / p.share, quad = (c0 - owner * p.share) >> 2;
        const uint32_t mine = base + p.inbox + (uint32_t)(which * set + rank * quads * kTileRows + quarter * 32 + lane) * 16;
#pragma unroll
        for (int j = 0; j < HALF; j += 4) {
            if (c0 + j < p.M) {
                if (split > 1) send16(mapa(mine + quad * kTileRows * 16, owner), mapa(bar_inbox, owner), v[j], v[j + 1], v[j + 2], v[j + 3]);
                else *reinterpret_cast<uint4*>(smem + p.inbox + (which * set + quad * kTileRows + quarter * 32 + lane) * 16) = make_uint4(v[j], v[j + 1], v[j + 2], v[j + 3]);
            }
            if (++quad == quads) { quad = 0; owner++; }
        }
    }
    if (split > 1) {
        cluster_arrive_relaxed();                    // met again at the end
        const bool all = mbar_wait_warp(ClusterBar{bar_inbox}, 0, &abort_flag, p.status, kErrEpilogueWait);
        ok = ok && all;
    } else __syncthreads();                          // (the asynchronous stores are for launches with clusters alone)
    auto finish = [&](int e, float b, const uint32_t (&r)[4]) {
        const int m0 = rank * p.share + (e / kTileRows) * 4, n = n0 + (e & (kTileRows - 1));
        if (e >= quads * kTileRows || n >= p.N || m0 >= p.M) return;
        float4 part[kMaxSplit];
#pragma unroll
        for (int i = 0; i < kMaxSplit; i++) part[i] = i < split ? sums[i * quads * kTileRows + e] : make_float4(0, 0, 0, 0);
        const long long at = (long long)m0 * p.ldc + n;
        float f[4] = {part[0].x, part[0].y, part[0].z, part[0].w}, x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) x[j] = __uint_as_float(p.c_f32 ? r[j] : r[j] << 16);
#pragma unroll
        for (int i = 1; i < kMaxSplit; i++) {
            if (i < split) { f[0] += part[i].x; f[1] += part[i].y; f[2] += part[i].z; f[3] += part[i].w; }
        }
        if constexpr (PAIR) {
#pragma unroll
            for (int i = 0; i < kMaxSplit; i++) part[i] = i < split ? sums[set + i * quads * kTileRows + e] : make_float4(0, 0, 0, 0);
            float4 u = part[0];
#pragma unroll
            for (int i = 1; i < kMaxSplit; i++) {
                if (i < split) { u.x += part[i].x; u.y += part[i].y; u.z += part[i].z; u.w += part[i].w; }
            }
            const float b2 = p.bias2 ? __ldg(p.bias2 + n) : 0.0f, uu[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] = __bfloat162float(__float2bfloat16_rn(fmaf(uu[j], p.alpha, b2)));
        }
        // every choice is made once for the four rows: with two warps a scheduler a branch per value is what this phase waits for
#pragma unroll
        for (int j = 0; j < 4; j++) f[j] = fmaf(f[j], p.alpha, b);
        if (p.epilogue == EPI_GELU || p.epilogue == EPI_GELU_MUL) {
#pragma unroll
            for (int j = 0; j < 4; j += 2) { const float2 y = gelu_fast2(make_float2(f[j], f[j + 1])); f[j] = y.x; f[j + 1] = y.y; }
        } else if (p.epilogue == EPI_SWIGLU) {
#pragma unroll
            for (int j = 0; j < 4; j++) f[j] = silu_fast(f[j]);
        } else if (p.epilogue == EPI_RELU_MUL) {
#pragma unroll
            for (int j = 0; j < 4; j++) f[j] = fmaxf(f[j], 0.0f);
        }
        if (PAIR || (p.R && epilogue_multiplies(p.epilogue))) {
#pragma unroll
            for (int j = 0; j < 4; j++) f[j] *= x[j];
        } else if (p.R) {
#pragma unroll
            for (int j = 0; j < 4; j++) f[j] += x[j];
        }
        const int rows = p.M - m0;
        if (p.c_f32) {
#pragma unroll
            for (int j = 0; j < 4; j++) if (j < rows) reinterpret_cast<float*>(p.C)[at + j * p.ldc] = f[j];
        } else {
#pragma unroll
            for (int j = 0; j < 4; j++) if (j < rows) reinterpret_cast<__nv_bfloat16*>(p.C)[at + j * p.ldc] = __float2bfloat16_rn(f[j]);
        }
        if (p.c2) {
#pragma unroll
            for (int j = 0; j < 4; j++) if (j < rows) p.c2[at + j * p.ldc] = __float2bfloat16_rn(f[j]);
        }
    };
    if (ok) {
#pragma unroll
        for (int i = 0; i < AHEAD; i++) finish(tid + i * THREADS, bias_pre[i], res_pre[i]);
        for (int e = tid + AHEAD * THREADS; e < quads * kTileRows; e += THREADS) {
            float b;
            uint32_t r[4];
            joined(e, b, r);
            finish(e, b, r);
        }
    }

    // teardown: every thread of every CTA arrives here, also after an aborted wait
    tc_fence_before();
    __syncthreads();
    if (split > 1) cluster_wait();       // no CTA leaves before all have sent: only an aborted one can still be waited for here
    if (abort_flag) {
        // loads and other CTAs' sums that may still be in flight land before shared memory is released
        const unsigned long long t0 = globaltimer();
        while (globaltimer() - t0 < 200000ull) { }
        __syncthreads();
    }
    if (warp == 1) { tc_fence_after(); tmem_dealloc(tmem, COLS); }
}

size_t stage_bytes(int tn, bool norm, bool pair) { return (size_t)kWeightBytes * (pair ? 2 : 1) + (norm ? 0 : (size_t)tn * kBK * 2); }

struct Split { int split, per_cta, num_kb, stages, share, inbox; size_t smem; };

// K is split into the most parts of 8, 6, 4, 3, 2 that make at most 9/5 CTAs per SM (one of a chain of launches, us): clusters of up to eight do
// not fill two per SM to the last slot, a second wave doubles the time, and clusters of five or seven leave SMs with two CTAs beside SMs with
// one (8 rows, 6144 x 2048: 4 parts 5.9, 5 parts 6.5, 6 parts, 288 CTAs, 9.2; 64 rows, 5632 x 2048: 4 parts 9.2, 5 parts 9.7, 6 parts, 264 CTAs,
// 8.4, 8 parts 14; 9728 x 2048: 2 parts 14.0, 3 parts 11.5, 4 parts, 304 CTAs, 18.9).  With more than 32 rows a CTA sends up to 28 KB of sums and all
// that send at once share the way: where three parts and more fit half the SMs, no more are taken (3072 x 768: 3 parts 5.5, 4 parts 6.1, 6
// parts 6.3; 2048 x 2048: 4 parts 5.6, 8 parts 6.1; 2048 x 7680: 11.8 / 11.6), unless they are three alone and K is long (3072 x 3072: 3 parts 8.3, 8 parts
// 7.9; 3072 x 5632: 12.4, 10.9).  17 .. 32 rows on more CTAs than SMs want three k-blocks each (5632 x 768: 6 parts 5.5, 4 parts 5.0).  With the norm inside, up to 7/4 CTAs per SM of at least three
// k-blocks: more parts are less to normalise for each (8 rows, 6144 x 2048: 4 parts 8.1, 5 parts 7.9; 4 rows, 5120 x 768: 4 parts 6.2, 6 parts 6.8).
// A CTA takes half of an SM's shared memory at most: the other half is for the next launch, which fills its ring while this one still computes
// (rings of up to 200 KB: 2048 x 5632 7.4 -> 12.8 us).  A launch that covers no more than half the SMs leaves the next one the others and takes a
// whole SM's (768 x 3072, 48 CTAs: 64 rows 5.6 -> 4.7, 32 rows 4.4 -> 4.0).  A pair of matrices is long enough to want the whole of it on every
// SM (8 rows, 2 x 5632 x 2048: 110 KB 13.7 us, 195 KB 9.4 us, two CTAs per SM 10.4 us; one matrix after the other 12.5 us, with RMSNorm
// 16.3 against 11.2 us; 2 x 3072 x 768 7.0 against 4.6 us).
Split choose_split(const GemmDesc& d, int tn, bool norm, bool pair) {
    const int sms = rt().sm_count, tiles = ceil_div(d.N, kTileRows), num_kb = ceil_div(d.K, kBK);
    int s = pair ? std::min(sms / tiles, num_kb) : norm ? std::min(7 * sms / 4 / tiles, std::max(num_kb / 3, 1)) : 0;
    if (!pair && !norm) {
        const int most = std::min(kMaxSplit, num_kb), half = sms / 2 / tiles;
        const auto fits = [&](int t) { return t <= most && 5 * t * tiles <= 9 * sms && !(d.M > 16 && d.M <= 32 && t * tiles > sms && num_kb < 3 * t); };
        if (d.M > 32 && (half > 3 || (half == 3 && num_kb <= 32))) s = std::min(half, most);
        else for (int t : {8, 6, 4, 3, 2}) if (!s && fits(t)) s = t;
    }
    s = std::max(1, std::min(s, kMaxSplit));
    Split r;
    r.num_kb = num_kb; r.per_cta = ceil_div(num_kb, s); r.split = ceil_div(num_kb, r.per_cta);
    r.share = 4 * ceil_div(d.M, 4ll * r.split);
    const int ctas = tiles * r.split, resident = std::min(3, ceil_div((long long)ctas, sms));
    const size_t sums = (size_t)r.split * r.share * kTileRows * 4 * (pair ? 2 : 1), norm_rows = norm ? (size_t)r.per_cta * tn * kBK * 2 : 0;
    const size_t room = ((pair && resident == 1) || 2 * ctas <= sms ? 195 : resident <= 2 ? 110 : 73) * 1024, inbox = r.split > 1 ? sums : 0, fixed = norm_rows + inbox;
    const int fit = (int)((room > fixed ? room - fixed : 0) / stage_bytes(tn, norm, pair));
    r.stages = std::max(std::min(2, r.per_cta), std::min({fit, r.per_cta, kMaxStages}));
    // a CTA that has the rows to itself keeps its sums where the ring was
    r.inbox = r.split > 1 ? (int)(r.stages * stage_bytes(tn, norm, pair) + norm_rows) : 0;
    r.smem = std::max(r.stages * stage_bytes(tn, norm, pair) + norm_rows + inbox, sums);
    return r;
}

template <int TN, bool NORM, bool PAIR = false>
int launch(const GemmDesc& d, const RowNorm& nrm, bool dependent) {
    const Split s = choose_split(d, TN, NORM, PAIR);
    CUtensorMap tmW, tmW2, tmA;
    if (gemm_encode_operand(&tmW, d.B, false, d.K, d.N, d.ldb, 1, 1, 0, 0, kTileRows)) return 1;
    tmW2 = tmW;
    if (PAIR && gemm_encode_operand(&tmW2, d.B2, false, d.K, d.N, d.ldb, 1, 1, 0, 0, kTileRows)) return 1;
    if (NORM) tmA = tmW;
    else if (gemm_encode_operand(&tmA, d.A, false, d.K, d.M, d.lda, 1, 1, 0, 0, TN)) return 1;
    auto kern = linear_stream_kernel<TN, NORM, PAIR>;
    static std::atomic<bool> granted{false};                                 // per instantiation
    if (!granted.load()) { SPT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024)); granted.store(true); }
    StreamParams p;
    p.bias2 = d.bias2;
    p.C = d.C; p.bias = d.bias; p.R = d.R; p.c2 = static_cast<__nv_bfloat16*>(d.C2);
    p.M = d.M; p.N = d.N; p.K = d.K; p.ldc = d.ldc; p.alpha = d.alpha; p.epilogue = d.epilogue; p.c_f32 = d.out_dtype == F32;
    p.ahead = ceil_div(d.N, kTileRows) * s.split <= rt().sm_count;          // (8 rows, 2048 x 5632: 7.4 -> 6.9 us; 32000 x 2048, all resident: 20.7 -> 25 us, hence the line)
    p.split = s.split; p.per_cta = s.per_cta; p.num_kb = s.num_kb; p.stages = s.stages; p.share = s.share; p.inbox = s.inbox;
    p.A = static_cast<const __nv_bfloat16*>(d.A); p.lda = d.lda; p.nrm = nrm; p.status = rt().dev_status;
    SPT_CUDA(launch_dependent(kern, dim3(ceil_div(d.N, kTileRows) * s.split), dim3(threads_of(TN)), s.smem, dependent, s.split, tmW, tmW2, tmA, p));
    note_submit();
    return 0;
}

}  // namespace

// From 17 rows up always; below that linear_few_rows.cu's direct loads have the shorter way to a result and lose where the weights are many, or
// K is long and a warp makes several rounds of loads (a row or a few whose weights fit its registers are taken there before this is asked).
// One of a chain of dependent launches, each with weights of its own, us (direct loads / this kernel):
//   M 64:  768 x 768 6.2 / 4.5, 768 x 3072 12.3 / 4.8
//   M 16:  2304 x 768 3.5 / 3.4, 768 x 2048 3.5 / 3.5, 1024 x 2048 4.6 / 3.6, 768 x 3072 4.1 / 3.7, 1024 x 3072 5.7 / 4.2
//   M 8:   3072 x 768 3.4 / 3.5, 2048 x 512 2.7 / 3.3, 768 x 2048 3.4 / 3.4, 1024 x 2048 4.3 / 3.6, 2048 x 1024 3.8 / 3.5, 1024 x 3072 5.5 / 4.1,
//          2048 x 2048 6.0 / 3.9, 6144 x 2048 11.9 / 5.9  -- hence 3 M weights, and 2 M where K is 1024 or more
//          (6144 x 512, 3 M exactly, behind a LayerNorm 6.7 / 5.2)
//   An ordinary launch has nothing to fill its ring behind: 8 rows, 2304 x 1024 4.2 / 6.3, 768 x 3072 4.7 / 6.1, 1024 x 2048 4.9 / 5.7 -- 3 M there
//   RMSNorm inside, M 8: 3072 x 768 5.0 / 5.4, 2048 x 2048 8.6 / 5.9, 6144 x 2048 11.3 / 7.9
//   LayerNorm inside, M 4: 3072 x 1024 6.3 / 6.4, 4096 x 1024 10.3 / 7.1 (forced: LayerNorm comes here with rows of more than 4096 values alone)
bool linear_stream_preferred(const GemmDesc& d, const RowNorm* nrm, bool dependent) {
    if (d.group || d.act_off || d.M > 64 || d.K <= kBK) return false;
    const long long weights = (long long)d.N * d.K;
    if (nrm && nrm->kind) return d.M <= kNormRows && d.K <= 16384 && weights > (d.M >= 4 ? 3ll << 20 : 8ll << 20);
    return d.M > 16 || weights > (3ll << 20) || (dependent && weights >= (d.K >= 1024 ? 2ll << 20 : 3ll << 20));
}

// The pair exists for one tile of 16 input rows: 17 .. 64 rows take the two products one after the other.
bool linear_pair_supported(const GemmDesc& d, const RowNorm* nrm) {
    if (!linear_few_rows_supported(d) || d.M > kNormRows || d.group || d.act_off || d.C2 || d.R || d.out_dtype != BF16 || !epilogue_multiplies(d.epilogue) || d.K <= kBK ||
        d.N < kTileRows || !d.B2 || (reinterpret_cast<uintptr_t>(d.B2) & 15)) return false;
    const bool norm = nrm && nrm->kind;
    if (norm && !linear_few_rows_norm_supported(d, *nrm)) return false;
    const Split s = choose_split(d, 16, norm, true);
    return s.smem <= 200 * 1024 && s.per_cta <= 32;                          // the normalised rows lie in shared memory whole
}
int linear_pair(const GemmDesc& d, const RowNorm* nrm) {
    if (!linear_pair_supported(d, nrm)) return fail("linear_pair: unsupported problem");
    return nrm && nrm->kind ? launch<16, true, true>(d, *nrm, true) : launch<16, false, true>(d, RowNorm{}, true);
}

int linear_stream(const GemmDesc& d, const RowNorm* nrm, bool dependent) {
    if (nrm && nrm->kind) return launch<16, true>(d, *nrm, dependent);
    if (d.M <= 16) return launch<16, false>(d, RowNorm{}, dependent);
    if (d.M <= 32) return launch<32, false>(d, RowNorm{}, dependent);
    return launch<64, false>(d, RowNorm{}, dependent);
}

}  // namespace spt
