// attention.cu -- causal multi-head attention core (crates/nn/src/lib.rs:600-637).
//
// Reference composition: reshape_to_heads x3 -> batch_transpose(K) -> batch_matmul(Q,K^T) -> scale ->
// masked_fill(j>i,-inf) -> softmax rows -> batch_matmul(P,V) -> reshape_from_heads, each a separate host
// pass with its own copy.  Here the head permutations are strides of the tensor maps (no kernel, no
// copy); f32 sequences of up to 128 tokens run attention_short_kernel, bf16 heads of 64 and 128 attention_fused.cu, and the
// "materialised" form below runs three launches per layer:
//   S = Q K^T      batched tcgen05 GEMM over (head, sequence), tiles above the diagonal skipped
//   P = causal_softmax(scale * S)   in place, reads only j <= i
//   O = P V        batched tcgen05 GEMM, k-blocks above the diagonal skipped, V supplied as V^T [hd, T]
#include "gemm.h"
#include "pdl.cuh"
#include "../../include/sptorch_b200_ext.h"

namespace spt {

// v [B*T, ld] (head h at columns h*hd..) -> vt [B, H, hd, T]
template <typename T>
__global__ void head_transpose_kernel(const T* __restrict__ v, T* __restrict__ vt, int Tn, int H, int hd, long long ld) {
    __shared__ T tile[32][33];
    const int bh = blockIdx.z, b = bh / H, h = bh % H;
    const int t0 = blockIdx.x * 32, e0 = blockIdx.y * 32;
    const T* src = v + ((long long)b * Tn) * ld + (long long)h * hd;
    T* dst = vt + (long long)bh * hd * Tn;
    for (int j = threadIdx.y; j < 32; j += 8) {
        int t = t0 + j, e = e0 + threadIdx.x;
        if (t < Tn && e < hd) tile[j][threadIdx.x] = src[(long long)t * ld + e];
    }
    __syncthreads();
    for (int j = threadIdx.y; j < 32; j += 8) {
        int e = e0 + j, t = t0 + threadIdx.x;
        if (t < Tn && e < hd) dst[(long long)e * Tn + t] = tile[threadIdx.x][j];
    }
}

// Short f32 sequences in one launch, f32 multiply-adds throughout: a CTA owns 32 query rows of one (sequence, head) and walks the keys up to
// the diagonal 64 at a time with a running row maximum and sum.  A thread holds 4 x 4 scores (keys 4 tx .., rows 4 ty ..) and the rows' 4 x C
// output columns; a row's sixteen threads are neighbours in the warp.  Bound by the FMA pipe where there are many sequences, by the chain
// load - scores - softmax - product where there are few.
constexpr int kShortThreads = 128, kShortQ = 32, kShortK = 64;
template <int C>                                                            // output columns a thread holds: head sizes up to 16 C
__global__ void __launch_bounds__(kShortThreads) attention_short_kernel(const float* q, const float* k, const float* v, float* out, int Tn, int H, int hd, long long ld,
                                                                        long long ld_out, float scale) {
    constexpr int QP = kShortQ + 4, KP = kShortK + 4, VP = 16 * C + 4, PP = kShortK + 4;
    extern __shared__ __align__(16) float sh[];
    float* qs = sh;                        // [hd][QP], scaled
    float* ks = qs + 16 * C * QP;          // [hd][KP]
    float* vs = ks + 16 * C * KP;          // [kShortK][VP]
    float* ps = vs + kShortK * VP;         // [kShortQ][PP]
    pdl_release();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, tiles = (Tn + kShortQ - 1) / kShortQ, bh = blockIdx.x / tiles, h = bh % H, b = bh / H,
              q0 = (blockIdx.x - bh * tiles) * kShortQ, vecs = hd / 4, pairs = (vecs + 1) / 2;
    const long long base = (long long)b * Tn * ld + (long long)h * hd;
    pdl_acquire();
    // Queries and keys are stored by column: a warp takes sixteen rows of two pieces side by side, a sector of each row, and its lanes' words lie in 32
    // banks.  (A row's pieces side by side lay in two of them: 64 x 16 heads of 128, 128 tokens, 353 us, so 274; 8 x 12 heads of 64 25.4, 22.7.)
    auto piece = [&](int i, int rows, int& r, int& c) { r = (i >> 1) % rows; c = ((i >> 1) / rows * 2 + (i & 1)) * 4; };
    constexpr int QV = kShortQ * 4 * C / kShortThreads;                      // pieces of the queries a thread brings
    float4 qv[QV];                                                           // requested with the first keys
#pragma unroll
    for (int u = 0; u < QV; u++) {
        int r, c;
        piece(tid + u * kShortThreads, kShortQ, r, c);
        qv[u] = c < hd && q0 + r < Tn ? *reinterpret_cast<const float4*>(q + base + (long long)(q0 + r) * ld + c) : make_float4(0, 0, 0, 0);
    }
    float m[4], l[4];
    float2 o[4][C / 2];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        m[i] = -INFINITY; l[i] = 0.0f;
#pragma unroll
        for (int c = 0; c < C / 2; c++) o[i][c] = make_float2(0.0f, 0.0f);
    }
    const int last = min(q0 + kShortQ, Tn);                                  // keys 0 .. last - 1 are seen by some row
    for (int k0 = 0; k0 < last; k0 += kShortK) {
        if (k0) __syncthreads();                                             // the block before has been read
        for (int i0 = tid; i0 < kShortK * 2 * pairs; i0 += 4 * kShortThreads) {      // four keys' and values' pieces requested before the first is stored
            float4 x[4], y[4];
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = i0 + u * kShortThreads, rv = i / vecs, cv = (i - rv * vecs) * 4;
                int r, c;
                piece(i, kShortK, r, c);
                x[u] = c < hd && k0 + r < last ? *reinterpret_cast<const float4*>(k + base + (long long)(k0 + r) * ld + c) : make_float4(0, 0, 0, 0);
                y[u] = rv < kShortK && k0 + rv < last ? *reinterpret_cast<const float4*>(v + base + (long long)(k0 + rv) * ld + cv) : make_float4(0, 0, 0, 0);
            }
            if (k0 == 0 && i0 == tid) {
#pragma unroll
                for (int u = 0; u < QV; u++) {
                    int r, c;
                    piece(tid + u * kShortThreads, kShortQ, r, c);
                    if (c < hd) { qs[c * QP + r] = qv[u].x * scale; qs[(c + 1) * QP + r] = qv[u].y * scale; qs[(c + 2) * QP + r] = qv[u].z * scale; qs[(c + 3) * QP + r] = qv[u].w * scale; }
                }
            }
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = i0 + u * kShortThreads, rv = i / vecs, cv = (i - rv * vecs) * 4;
                int r, c;
                piece(i, kShortK, r, c);
                if (c < hd) { ks[c * KP + r] = x[u].x; ks[(c + 1) * KP + r] = x[u].y; ks[(c + 2) * KP + r] = x[u].z; ks[(c + 3) * KP + r] = x[u].w; }
                if (rv < kShortK) *reinterpret_cast<float4*>(vs + rv * VP + cv) = y[u];
            }
        }
        __syncthreads();
        float2 s2[4][2] = {};                                                // two products an instruction here and below (the two calls above 247 and 21.2 us): the same roundings
#pragma unroll 4
        for (int d = 0; d < hd; d++) {
            const float4 a = *reinterpret_cast<const float4*>(qs + d * QP + 4 * ty), x = *reinterpret_cast<const float4*>(ks + d * KP + 4 * tx);
            const float aa[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                s2[i][0] = __ffma2_rn(make_float2(aa[i], aa[i]), make_float2(x.x, x.y), s2[i][0]);
                s2[i][1] = __ffma2_rn(make_float2(aa[i], aa[i]), make_float2(x.z, x.w), s2[i][1]);
            }
        }
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int row = q0 + 4 * ty + i;
            float s[4] = {s2[i][0].x, s2[i][0].y, s2[i][1].x, s2[i][1].y}, mx = m[i];
#pragma unroll
            for (int j = 0; j < 4; j++) { if (k0 + 4 * tx + j > row) s[j] = -INFINITY; mx = fmaxf(mx, s[j]); }
#pragma unroll
            for (int w = 8; w > 0; w >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, w));
            const float ref = mx == -INFINITY ? 0.0f : mx, corr = expf(m[i] - ref);      // a row below the first block sees key 0: finite
            float sum = 0.0f;
#pragma unroll
            for (int j = 0; j < 4; j++) { s[j] = expf(s[j] - ref); sum += s[j]; }
            l[i] = l[i] * corr + sum;                                        // this thread's keys; the row's threads meet at the end
            m[i] = mx;
#pragma unroll
            for (int c = 0; c < C / 2; c++) { o[i][c].x *= corr; o[i][c].y *= corr; }
            *reinterpret_cast<float4*>(ps + (4 * ty + i) * PP + 4 * tx) = make_float4(s[0], s[1], s[2], s[3]);
        }
        __syncwarp();                                                        // a row's weights are written and read by one half warp
        const int keys = min(kShortK, last - k0);                            // rounded up to four below: the weights past them are zero
        for (int j = 0; j < keys; j += 4) {
            float w[4][4];
#pragma unroll
            for (int i = 0; i < 4; i++) *reinterpret_cast<float4*>(w[i]) = *reinterpret_cast<const float4*>(ps + (4 * ty + i) * PP + j);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                float2 vv[C / 2];
                if constexpr (C % 4 == 0) {
#pragma unroll
                    for (int c = 0; c < C; c += 4) {
                        const float4 x = *reinterpret_cast<const float4*>(vs + (j + u) * VP + (c / 4 * 16 + tx) * 4);
                        vv[c / 2] = make_float2(x.x, x.y); vv[c / 2 + 1] = make_float2(x.z, x.w);
                    }
                } else vv[0] = *reinterpret_cast<const float2*>(vs + (j + u) * VP + tx * 2);
#pragma unroll
                for (int i = 0; i < 4; i++)
#pragma unroll
                    for (int c = 0; c < C / 2; c++) o[i][c] = __ffma2_rn(make_float2(w[i][u], w[i][u]), vv[c], o[i][c]);
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int row = q0 + 4 * ty + i;
        float sum = l[i];
#pragma unroll
        for (int w = 8; w > 0; w >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, w);
        if (row >= Tn) continue;
        const float inv = 1.0f / sum;
        float* dst = out + ((long long)b * Tn + row) * ld_out + (long long)h * hd;
        if constexpr (C % 4 == 0) {
#pragma unroll
            for (int c = 0; c < C; c += 4) {
                const int col = (c / 4 * 16 + tx) * 4;
                if (col < hd) *reinterpret_cast<float4*>(dst + col) = make_float4(o[i][c / 2].x * inv, o[i][c / 2].y * inv, o[i][c / 2 + 1].x * inv, o[i][c / 2 + 1].y * inv);
            }
        } else if (2 * tx < hd) *reinterpret_cast<float2*>(dst + 2 * tx) = make_float2(o[i][0].x * inv, o[i][0].y * inv);
    }
}

// The rule knows the sequence alone: a sequence's result does not depend on how many there are.  A layer of an f32 model with this kernel / with the
// four launches, us, for 1, 8 and 64 sequences:
//   heads of 64, width 768:    64 tokens 64 / 78, 77 / 87, 187 / 218;       128 tokens 77 / 83, 95 / 97, 355 / 376
//   heads of 128, width 2048:  64 tokens 117 / 135, 153 / 172, 555 / 583;   96 tokens 125 / 137, 197 / 202, 824 / 817;   128 tokens 129 / 138, 251 / 249, 1087 / 1047
// The attention alone, public operation: 12 heads of 64 10.0 / 16.1, 21.2 / 20.2, 88.9 / 104.8 at 128 tokens; 16 heads of 128 9.0 / 16.1, 12.4 / 20.4, 90.6 / 98.2 at
// 64 and 17.5 / 17.4, 40.3 / 25.6, 247 / 172 at 128.  So heads above 64 with more than 96 tokens are behind from about sixteen sequences on, where the
// tensor pipe's TF32 products are many: they stay here for the bits of f32 (the four launches round the operands to eleven).
bool attention_short_supported(const void* q, const void* k, const void* v, const void* out, int Tn, int hd, long long ld, long long ld_out, int dtype) {
    return dtype == F32 && Tn <= 128 && hd % 4 == 0 && hd <= 128 && ld % 4 == 0 && ld_out % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k) | reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
}

int attention_short(const float* q, const float* k, const float* v, float* out, int B, int Tn, int H, int hd, long long ld, long long ld_out) {
    const long long ctas = (long long)ceil_div(Tn, kShortQ) * B * H;
    if (ctas > INT32_MAX) return fail("attention: %lld query tiles exceed one launch", ctas);
    ProfScope ps(PROF_ATTN_FUSED);
    auto launch = [&](auto kern, int c) -> int {
        const size_t smem = (size_t)(16 * c * (kShortQ + 4 + kShortK + 4) + kShortK * (16 * c + 4) + kShortQ * (kShortK + 4)) * 4;
        SPT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        SPT_CUDA(launch_dependent(kern, dim3((unsigned)ctas), dim3(kShortThreads), smem, short_launch(0.0, 16.0 * B * Tn * H * hd), 1, q, k, v, out, Tn, H, hd, ld, ld_out,
                                  1.0f / sqrtf((float)hd)));
        note_submit();
        return 0;
    };
    return hd <= 32 ? launch(attention_short_kernel<2>, 2) : hd <= 64 ? launch(attention_short_kernel<4>, 4) : launch(attention_short_kernel<8>, 8);
}

int attention_materialized(const void* q, const void* k, const void* vt, long long vt_ld, long long vt_s_head, long long vt_s_batch,
                           void* out, void* scores, int B, int Tn, int H, int hd, long long ld_qk, long long ld_out, int dtype);
bool attention_fused_supported(int T, int hd, long long ld_q, long long ld_kv);
int attention_fused(const void* q, const void* k, const void* v, void* out, int B, int T, int H, int hd, long long ld_q, long long ld_k,
                    long long ld_v, long long ld_out);

static std::atomic<int> g_attn_mode{0};   // 0 = fused kernel whenever it applies, 1 = always the materialised three-launch form
int attention_mode() { return g_attn_mode.load(); }

// true when the fused kernel takes this problem (bf16, head_dim 64 or 128, 16-byte aligned row pitches, not switched off)
bool attention_uses_fused(int dtype, int Tn, int hd, long long ld_q, long long ld_kv) {
    return dtype == BF16 && g_attn_mode.load() == 0 && attention_fused_supported(Tn, hd, ld_q, ld_kv);
}

// q,k: [B*T, ld_qk]; vt: V^T with element (b,h,e,t) at vt[b*vt_s_batch + h*vt_s_head + e*vt_ld + t];
// scores: workspace of B*H*T*T elements; out: [B*T, ld_out]
int attention_materialized(const void* q, const void* k, const void* vt, long long vt_ld, long long vt_s_head, long long vt_s_batch,
                           void* out, void* scores, int B, int Tn, int H, int hd, long long ld_qk, long long ld_out, int dtype) {
    const int mode = dtype == BF16 ? MM_BF16 : MM_TF32;
    GemmDesc s;
    s.A = q; s.B = k; s.C = scores;
    s.M = Tn; s.N = Tn; s.K = hd;
    s.lda = ld_qk; s.ldb = ld_qk; s.ldc = Tn;
    s.nb1 = H; s.nb2 = B;
    s.sA1 = hd; s.sA2 = (long long)Tn * ld_qk;
    s.sB1 = hd; s.sB2 = (long long)Tn * ld_qk;
    s.sC1 = (long long)Tn * Tn; s.sC2 = (long long)H * Tn * Tn;
    s.mode = mode; s.out_dtype = dtype; s.causal_lower = 1;
    GemmPlan ps;
    if (gemm_plan(s, &ps)) return 1;
    { ProfScope pr(PROF_ATTN_GEMM); if (gemm_run(ps)) return 1; }
    // scale -> mask -> softmax exactly in the reference's order (crates/nn/src/lib.rs:614-632)
    { ProfScope pr(PROF_SOFTMAX); if (sptorch_ext_causal_softmax(scores, scores, (size_t)B * H, (size_t)Tn, 1.0f / sqrtf((float)hd), dtype)) return 1; }
    GemmDesc o;
    o.A = scores; o.B = vt; o.C = out;
    o.M = Tn; o.N = hd; o.K = Tn;
    o.lda = Tn; o.ldb = vt_ld; o.ldc = ld_out;
    o.nb1 = H; o.nb2 = B;
    o.sA1 = (long long)Tn * Tn; o.sA2 = (long long)H * Tn * Tn;
    o.sB1 = vt_s_head; o.sB2 = vt_s_batch;
    o.sC1 = hd; o.sC2 = (long long)Tn * ld_out;
    o.mode = mode; o.out_dtype = dtype; o.causal_k = 1;
    GemmPlan po;
    if (gemm_plan(o, &po)) return 1;
    { ProfScope pr(PROF_ATTN_GEMM); if (gemm_run(po)) return 1; }
    return 0;
}

}  // namespace spt

using namespace spt;

extern "C" {

size_t sptorch_ext_attention_workspace(size_t B, size_t T, size_t H, size_t hd, int dtype) {
    size_t es = dtype == SPT_BF16 ? 2 : 4;
    size_t scores = ((B * H * T * T * es + 255) / 256) * 256;
    size_t vt = ((B * H * hd * T * es + 255) / 256) * 256;
    return scores + vt;
}

int sptorch_ext_attention_causal(const void* q, const void* k, const void* v, void* out, void* workspace, size_t B, size_t T, size_t H,
                                 size_t hd, size_t ld_qkv, int dtype) {
    if (enter()) return 1;
    if (B == 0 || T == 0 || H == 0 || hd == 0) return 0;
    if (!q || !k || !v || !out || !workspace) return fail("attention: null handle");
    if (dtype != SPT_F32 && dtype != SPT_BF16) return fail("attention: unknown dtype %d", dtype);
    if (B * H > 65535) return fail("attention: B*H exceeds one launch of the V transpose");
    size_t es = dtype == SPT_BF16 ? 2 : 4;
    const bool fused = attention_uses_fused(dtype, (int)T, (int)hd, (long long)ld_qkv, (long long)ld_qkv);
    if (!fused && (T * es) % 16) return fail("attention: T must be a multiple of %zu for this dtype", 16 / es);
    size_t scores_bytes = ((B * H * T * T * es + 255) / 256) * 256;
    void* scores = workspace;
    void* vt = (uint8_t*)workspace + scores_bytes;
    if (fused)
        return attention_fused(q, k, v, out, (int)B, (int)T, (int)H, (int)hd, (long long)ld_qkv, (long long)ld_qkv, (long long)ld_qkv, (long long)(H * hd));
    // The one launch writes a tile's rows while others still read keys and values, and reads only its own rows of q: an output over one of them takes the
    // several launches, the last of which reads the workspace alone.
    const size_t in_bytes = ((B * T - 1) * ld_qkv + H * hd) * es, out_bytes = B * T * H * hd * es;
    auto apart = [&](const void* p) { return (const uint8_t*)p + in_bytes <= (const uint8_t*)out || (const uint8_t*)out + out_bytes <= (const uint8_t*)p; };
    const bool separate = apart(k) && apart(v) && (apart(q) || (q == out && ld_qkv == H * hd));
    if (separate && g_attn_mode.load() == 0 && attention_short_supported(q, k, v, out, (int)T, (int)hd, (long long)ld_qkv, (long long)(H * hd), dtype))
        return attention_short((const float*)q, (const float*)k, (const float*)v, (float*)out, (int)B, (int)T, (int)H, (int)hd, (long long)ld_qkv, (long long)(H * hd));
    dim3 grid((unsigned)((T + 31) / 32), (unsigned)((hd + 31) / 32), (unsigned)(B * H));
    if (dtype == SPT_BF16)
        head_transpose_kernel<__nv_bfloat16><<<grid, dim3(32, 8), 0, rt().stream>>>((const __nv_bfloat16*)v, (__nv_bfloat16*)vt, (int)T, (int)H, (int)hd, (long long)ld_qkv);
    else
        head_transpose_kernel<float><<<grid, dim3(32, 8), 0, rt().stream>>>((const float*)v, (float*)vt, (int)T, (int)H, (int)hd, (long long)ld_qkv);
    SPT_LAUNCH_CHECK("head_transpose");
    return attention_materialized(q, k, vt, (long long)T, (long long)(hd * T), (long long)(H * hd * T), out, scores, (int)B, (int)T, (int)H,
                                  (int)hd, (long long)ld_qkv, (long long)(H * hd), dtype);
}

int sptorch_ext_set_attention_mode(int mode) {
    if (mode != 0 && mode != 1) return fail("set_attention_mode: 0 = fused when possible, 1 = materialised");
    g_attn_mode.store(mode);
    bump_config_epoch();          // a captured forward holds the other path's launches
    return 0;
}

}  // extern "C"
