// Attention and the small per-head kernels around it, fp32 throughout (the KV cache stays fp32, as in the reference).
//
//   k_attn_decode   one token: per-head q/k RMSNorm + RoPE + KV store fused in front of a split-K flash decode; all
//                   q heads of a KV group share one pass over K/V; splits meet in a scratch buffer summed by the
//                   last CTA to arrive, in split order (deterministic).
//   k_qkv_post      prompt chunk: per-head q/k RMSNorm + RoPE in place, K/V rows stored to the cache.
//   k_attn_prefill  prompt chunk: causal tiled attention, 32 queries of one head per CTA, online softmax.
// Semantics follow CpuModel::forward of the reference (src/model.cpp:176-214): scale = 1/sqrt(float(D)), scores
// accumulated in dimension order without FMA contraction, max-subtracted softmax.
#include <algorithm>
#include <cmath>
#include <cstdlib>

#include "common.cuh"
#include "split.cuh"
#include "attn_core.cuh"

namespace elb {

constexpr int D = 128;  // head_dim (checked at model creation)

// RMSNorm over one 128-wide head followed by NEOX RoPE (rmsnorm + rope, src/ops.cpp:155-160, src/model.cpp:23-32).
// One warp per head; lane owns elements lane, lane+32, lane+64, lane+96. Result goes to dst (shared or global).
__device__ __forceinline__ void head_norm_rope(const float* src, const float* w, const float2* cs, int rope_dim,
                                               float eps, float* dst, int lane) {
    float v[4];
    double ss = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[j] = src[lane + 32 * j];
        ss += double(v[j]) * v[j];
    }
    ss = warp_sum(ss);
    const float inv = float(1.0 / sqrt(ss / D + double(eps)));
#pragma unroll
    for (int j = 0; j < 4; ++j) v[j] = __fmul_rn(__fmul_rn(v[j], inv), w[lane + 32 * j]);
    if (rope_dim == D) {  // pairs (i, i+64): both halves of a pair live in this lane
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 c = cs[lane + 32 * j];
            const float a = v[j], b = v[j + 2];
            v[j] = __fsub_rn(__fmul_rn(a, c.x), __fmul_rn(b, c.y));
            v[j + 2] = __fadd_rn(__fmul_rn(a, c.y), __fmul_rn(b, c.x));
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[lane + 32 * j] = v[j];
    } else {  // partial rotary: pairs (i, i + rope_dim/2), the rest passes through
#pragma unroll
        for (int j = 0; j < 4; ++j) dst[lane + 32 * j] = v[j];
        __syncwarp();
        const int half = rope_dim / 2;
        for (int i = lane; i < half; i += 32) {
            const float2 c = cs[i];
            const float a = dst[i], b = dst[i + half];
            dst[i] = __fsub_rn(__fmul_rn(a, c.x), __fmul_rn(b, c.y));
            dst[i + half] = __fadd_rn(__fmul_rn(a, c.y), __fmul_rn(b, c.x));
        }
    }
    __syncwarp();
}

// ---------------------------------------------------------------- decode

constexpr int AD_THREADS = 256, AD_KT = 32, AD_MAXG = 8, AD_LDK = D + 1, AD_MAXSPLIT = 32;

struct AttnDecodeParams {
    const float* qkv;  // [QD + 2 KD] of this token, q and k not yet normalised
    const float *q_norm, *k_norm;
    const float2* rope;  // [n_ctx][rope_dim/2] (cos, sin)
    const int* pos;      // device scalar
    float *kc, *vc;      // this layer's cache [n_ctx][KD]
    float* att;          // [QD]
    float* part;         // [HKV][nsplit][group][D + 2]
    unsigned* counters;  // [HKV]
    int H, HKV, rope_dim, nsplit;
    float eps, scale;
    PostOp post;
};

__global__ void __launch_bounds__(AD_THREADS) k_attn_decode(const AttnDecodeParams p) {
    __shared__ float qs[AD_MAXG][D];
    __shared__ float knew[D], vnew[D];
    __shared__ float Ks[AD_KT][AD_LDK];
    __shared__ float Vs[AD_KT][D];
    __shared__ float Ps[AD_MAXG][AD_KT];
    __shared__ float corr_s[AD_MAXG], m_s[AD_MAXG], l_s[AD_MAXG];
    __shared__ int s_last;
    __shared__ double red8[8];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int kvh = blockIdx.x, split = blockIdx.y, group = p.H / p.HKV, QD = p.H * D, KD = p.HKV * D;
    pdl_launch_dependents();
    pdl_wait();
    const int pos = *p.pos, T = pos + 1;
    const float2* cs = p.rope + size_t(pos) * (p.rope_dim / 2);

    for (int h = warp; h < group + 1; h += AD_THREADS / 32) {
        if (h < group) head_norm_rope(p.qkv + (kvh * group + h) * D, p.q_norm, cs, p.rope_dim, p.eps, qs[h], lane);
        else head_norm_rope(p.qkv + QD + kvh * D, p.k_norm, cs, p.rope_dim, p.eps, knew, lane);
    }
    if (tid < D) vnew[tid] = p.qkv[QD + KD + kvh * D + tid];
    __syncthreads();
    if (split == 0 && tid < D) {  // KV append (src/model.cpp:186-189): only row `pos` is written
        p.kc[size_t(pos) * KD + kvh * D + tid] = knew[tid];
        p.vc[size_t(pos) * KD + kvh * D + tid] = vnew[tid];
    }
    if (tid < AD_MAXG) { m_s[tid] = -INFINITY; l_s[tid] = 0.f; }

    // this split's key range, in whole tiles
    const int tiles = (T + AD_KT - 1) / AD_KT, per = (tiles + p.nsplit - 1) / p.nsplit;
    const int t_begin = min(T, split * per * AD_KT), t_end = min(T, (split + 1) * per * AD_KT);
    float acc[4] = {0.f, 0.f, 0.f, 0.f};  // outputs (head tid/128 + 2i, dim tid%128)
    const int od = tid & (D - 1), oh = tid >> 7;

    for (int t0 = t_begin; t0 < t_end; t0 += AD_KT) {
        const int nk = min(AD_KT, t_end - t0);
        __syncthreads();
        for (int idx = tid; idx < AD_KT * (D / 4); idx += AD_THREADS) {
            const int j = idx / (D / 4), c = (idx % (D / 4)) * 4;
            float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
            if (j < nk) {
                const int t = t0 + j;
                if (t == pos) {  // the row this kernel appends: take it from shared memory, not from the cache
                    kv = *reinterpret_cast<const float4*>(&knew[c]);
                    vv = *reinterpret_cast<const float4*>(&vnew[c]);
                } else {
                    kv = *reinterpret_cast<const float4*>(p.kc + size_t(t) * KD + kvh * D + c);
                    vv = *reinterpret_cast<const float4*>(p.vc + size_t(t) * KD + kvh * D + c);
                }
            }
            Ks[j][c] = kv.x; Ks[j][c + 1] = kv.y; Ks[j][c + 2] = kv.z; Ks[j][c + 3] = kv.w;
            *reinterpret_cast<float4*>(&Vs[j][c]) = vv;
        }
        __syncthreads();
        // scores: warp = head, lane = key; dimension order, multiply then add (no contraction), as the CPU path does
        if (warp < group) {
            float s = -INFINITY;
            if (lane < nk) {
                float a = 0.f;
#pragma unroll 8
                for (int i = 0; i < D; ++i) a = __fadd_rn(a, __fmul_rn(qs[warp][i], Ks[lane][i]));
                s = __fmul_rn(a, p.scale);
            }
            const float m_old = m_s[warp], m_new = fmaxf(m_old, warp_max(s));
            const float pj = lane < nk ? expf(s - m_new) : 0.f;
            const float sum = warp_sum(pj);
            Ps[warp][lane] = pj;
            if (lane == 0) {
                const float c = m_old == -INFINITY ? 0.f : expf(m_old - m_new);
                corr_s[warp] = c;
                l_s[warp] = l_s[warp] * c + sum;
                m_s[warp] = m_new;
            }
        }
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int h = oh + 2 * i;
            if (h >= group) continue;
            float a = acc[i] * corr_s[h];
            for (int j = 0; j < nk; ++j) a = fmaf(Ps[h][j], Vs[j][od], a);
            acc[i] = a;
        }
    }
    __syncthreads();

    if (p.nsplit == 1) {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int h = oh + 2 * i;
            if (h < group) p.att[(kvh * group + h) * D + od] = acc[i] / l_s[h];
        }
    } else {
        // partial result of this split: [group][D] accumulators, then m and l per head
        float* mine = p.part + (size_t(kvh) * p.nsplit + split) * group * (D + 2);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int h = oh + 2 * i;
            if (h < group) mine[h * (D + 2) + od] = acc[i];
        }
        if (tid < group) {
            mine[tid * (D + 2) + D] = m_s[tid];
            mine[tid * (D + 2) + D + 1] = l_s[tid];
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            const unsigned old = atomicAdd(&p.counters[kvh], 1u);
            s_last = old == unsigned(p.nsplit - 1);
            if (s_last) p.counters[kvh] = 0;
        }
        __syncthreads();
        if (s_last) {
            __threadfence();
            const float* base = p.part + size_t(kvh) * p.nsplit * group * (D + 2);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int h = oh + 2 * i;
                if (h >= group) continue;
                // all loads of a pass are issued before the first use (the split count is at most AD_MAXSPLIT)
                float ms[AD_MAXSPLIT], ls[AD_MAXSPLIT], as[AD_MAXSPLIT];
#pragma unroll
                for (int s = 0; s < AD_MAXSPLIT; ++s) {
                    const float* ps = base + (size_t(s < p.nsplit ? s : 0) * group + h) * (D + 2);
                    ms[s] = s < p.nsplit ? __ldcg(ps + D) : -INFINITY;
                    ls[s] = __ldcg(ps + D + 1);
                    as[s] = __ldcg(ps + od);
                }
                float M = -INFINITY;
#pragma unroll
                for (int s = 0; s < AD_MAXSPLIT; ++s) M = fmaxf(M, ms[s]);
                float L = 0.f, o = 0.f;
#pragma unroll
                for (int s = 0; s < AD_MAXSPLIT; ++s) {  // fixed split order
                    if (ms[s] == -INFINITY) continue;
                    const float w = expf(ms[s] - M);
                    L = fmaf(ls[s], w, L);
                    o = fmaf(as[s], w, o);
                }
                p.att[(kvh * group + h) * D + od] = o / L;
            }
        }
    }
    post_op(p.post, gridDim.x * gridDim.y, &s_last, red8);
}

// ---------------------------------------------------------------- prompt chunk

// grid (B, ceil((H + 2 HKV) / 8)), blocks of 8 warps, one warp per (token, head). q heads: norm + rope in place. k heads: norm + rope in place and
// store to the cache row pos0 + b. v heads: store.
// posv / seqv (both or neither): row b sits at position posv[b] of sequence seqv[b], whose cache starts seq_stride
// floats after kc / vc; without them row b sits at position pos0 + b of the cache at kc / vc.
__global__ void __launch_bounds__(256) k_qkv_post(float* qkv, int64_t ld, const float* q_norm, const float* k_norm,
                                                 const float2* rope, int pos0, float* kc, float* vc, int H, int HKV,
                                                 int rope_dim, float eps, const int* posv, const int* seqv,
                                                 size_t seq_stride) {
    const int b = blockIdx.x, hd = blockIdx.y * 8 + threadIdx.y, lane = threadIdx.x, QD = H * D, KD = HKV * D;
    pdl_launch_dependents();
    pdl_wait();
    if (hd >= H + 2 * HKV) return;  // (warps only: nothing below synchronises the block)
    const int pos = posv ? posv[b] : pos0 + b;
    if (seqv) { kc += size_t(seqv[b]) * seq_stride; vc += size_t(seqv[b]) * seq_stride; }
    float* row = qkv + int64_t(b) * ld;
    const float2* cs = rope + size_t(pos) * (rope_dim / 2);
    if (hd < H) {
        head_norm_rope(row + hd * D, q_norm, cs, rope_dim, eps, row + hd * D, lane);
    } else if (hd < H + HKV) {
        float* k = row + QD + (hd - H) * D;
        head_norm_rope(k, k_norm, cs, rope_dim, eps, k, lane);
        for (int i = lane; i < D; i += 32) kc[size_t(pos) * KD + (hd - H) * D + i] = k[i];
    } else {
        const float* v = row + QD + KD + (hd - H - HKV) * D;
        for (int i = lane; i < D; i += 32) vc[size_t(pos) * KD + (hd - H - HKV) * D + i] = v[i];
    }
}

constexpr int AP_Q = 32, AP_K = 32, AP_THREADS = 256, AP_LD = D + 1;
constexpr size_t AP_SMEM = size_t(AP_Q * AP_LD + AP_K * AP_LD + AP_K * D + AP_Q * (AP_K + 1)) * sizeof(float);

// grid (H, ceil(B/32)). Query b of the chunk sits at position pos0 + b and sees keys 0..pos0+b (causal).
__global__ void __launch_bounds__(AP_THREADS) k_attn_prefill(const float* __restrict__ qkv, int64_t ld,
                                                             const float* __restrict__ kc, const float* __restrict__ vc,
                                                             float* __restrict__ att, int64_t ld_att, int pos0, int B, int H,
                                                             int HKV, float scale) {
    extern __shared__ __align__(16) float sm[];
    float (*Qs)[AP_LD] = reinterpret_cast<float (*)[AP_LD]>(sm);
    float (*Ks)[AP_LD] = reinterpret_cast<float (*)[AP_LD]>(sm + AP_Q * AP_LD);
    float (*Vs)[D] = reinterpret_cast<float (*)[D]>(sm + AP_Q * AP_LD + AP_K * AP_LD);
    float (*Ps)[AP_K + 1] = reinterpret_cast<float (*)[AP_K + 1]>(sm + AP_Q * AP_LD + AP_K * AP_LD + AP_K * D);
    const int tid = threadIdx.x, hd = blockIdx.x, q0 = blockIdx.y * AP_Q, KD = HKV * D, kvh = hd / (H / HKV);
    const int qi = tid >> 3, sub = tid & 7;  // 8 threads per query row
    const int nq = min(AP_Q, B - q0);
    for (int idx = tid; idx < AP_Q * D; idx += AP_THREADS) {
        const int r = idx / D, c = idx % D;
        Qs[r][c] = r < nq ? qkv[int64_t(q0 + r) * ld + hd * D + c] : 0.f;
    }
    float m = -INFINITY, l = 0.f, acc[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) acc[i] = 0.f;
    const int my_last = pos0 + q0 + qi;            // last key this query may see
    const int T = pos0 + q0 + nq;                  // keys needed by the tile
    for (int t0 = 0; t0 < T; t0 += AP_K) {
        __syncthreads();
        for (int idx = tid; idx < AP_K * (D / 4); idx += AP_THREADS) {
            const int j = idx / (D / 4), c = (idx % (D / 4)) * 4;
            float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
            if (t0 + j < T) {
                kv = *reinterpret_cast<const float4*>(kc + size_t(t0 + j) * KD + kvh * D + c);
                vv = *reinterpret_cast<const float4*>(vc + size_t(t0 + j) * KD + kvh * D + c);
            }
            Ks[j][c] = kv.x; Ks[j][c + 1] = kv.y; Ks[j][c + 2] = kv.z; Ks[j][c + 3] = kv.w;
            *reinterpret_cast<float4*>(&Vs[j][c]) = vv;
        }
        __syncthreads();
        float s[4] = {0.f, 0.f, 0.f, 0.f};  // keys sub + 8i
#pragma unroll 4
        for (int d = 0; d < D; ++d) {
            const float q = Qs[qi][d];
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] = __fadd_rn(s[i], __fmul_rn(q, Ks[sub + 8 * i][d]));
        }
        float mx = -INFINITY;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s[i] = t0 + sub + 8 * i <= my_last ? __fmul_rn(s[i], scale) : -INFINITY;
            mx = fmaxf(mx, s[i]);
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m, mx);
        float sum = 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float pj = s[i] == -INFINITY ? 0.f : expf(s[i] - m_new);
            Ps[qi][sub + 8 * i] = pj;
            sum += pj;
        }
#pragma unroll
        for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float corr = m == -INFINITY ? 0.f : expf(m - m_new);
        l = l * corr + sum;
        m = m_new;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < 16; ++i) acc[i] *= corr;
        const int nk = min(AP_K, T - t0);
        for (int j = 0; j < nk; ++j) {
            const float pj = Ps[qi][j];
#pragma unroll
            for (int i = 0; i < 16; ++i) acc[i] = fmaf(pj, Vs[j][sub + 8 * i], acc[i]);
        }
    }
    if (qi < nq) {
        const float inv = 1.0f / l;
#pragma unroll
        for (int i = 0; i < 16; ++i) att[int64_t(q0 + qi) * ld_att + hd * D + sub + 8 * i] = acc[i] * inv;
    }
}

// Prompt chunk, all query heads of one KV head together: a CTA holds 64 query rows (group heads x 64/group tokens), so
// every K/V tile is loaded once for the whole group, and each thread keeps a 4-row x 2-key block of scores and a
// 4-row x 8-dim block of outputs in registers. Same arithmetic as k_attn_prefill: scores in dimension order, multiply
// then add, online softmax over 32-key tiles, causal.
// The keys of a query tile are cut into chunks of `kchunk` key tiles, one CTA per (query tile, chunk): late query tiles
// see many more keys than early ones, and without the cut the longest tile alone sets the kernel's duration. A query
// tile with one chunk writes its output directly; otherwise every chunk leaves (acc, m, l) in `part` and the last
// chunk to arrive adds them in chunk order (deterministic). grid (HKV, number of (query tile, chunk) items).
constexpr int AG_ROWS = 64, AG_K = 32, AG_LD = D + 4, AG_THREADS = 256, AG_LDP = AG_K + 1, AG_MAXCHUNK = 8;
constexpr size_t AG_SMEM = size_t(AG_ROWS * AG_LD + AG_K * AG_LD + AG_K * D + AG_ROWS * AG_LDP) * sizeof(float);
constexpr int AG_PART = AG_ROWS * (D + 2);  // floats per partial result

__host__ __device__ __forceinline__ int ag_chunks(int pos0, int B, int TQ, int i, int kchunk) {  // chunks of query tile i
    const int T = pos0 + min(B, (i + 1) * TQ);
    return ((T + AG_K - 1) / AG_K + kchunk - 1) / kchunk;
}

__global__ void __launch_bounds__(AG_THREADS) k_attn_prefill_gqa(const float* __restrict__ qkv, int64_t ld,
                                                                 const float* __restrict__ kc, const float* __restrict__ vc,
                                                                 float* __restrict__ att, int64_t ld_att, int pos0, int B,
                                                                 int H, int HKV, float scale, int kchunk, float* part,
                                                                 unsigned* counters) {
    extern __shared__ __align__(16) float sm[];
    float* Qs = sm;                        // [64][AG_LD]
    float* Ks = Qs + AG_ROWS * AG_LD;      // [32][AG_LD]
    float* Vs = Ks + AG_K * AG_LD;         // [32][D]
    float* Ps = Vs + AG_K * D;             // [64][33]
    __shared__ int s_last;
    const int tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int kvh = blockIdx.x, group = H / HKV, TQ = AG_ROWS / group, KD = HKV * D, n_qt = (B + TQ - 1) / TQ;
    int qt = 0, chunk = int(blockIdx.y), n_chunks = ag_chunks(pos0, B, TQ, 0, kchunk);  // item -> (query tile, chunk)
    while (chunk >= n_chunks && qt + 1 < n_qt) {
        chunk -= n_chunks;
        ++qt;
        n_chunks = ag_chunks(pos0, B, TQ, qt, kchunk);
    }
    const int q0 = qt * TQ;
    const int nq = min(TQ, B - q0);
    for (int idx = tid; idx < AG_ROWS * (D / 4); idx += AG_THREADS) {  // row r = head * TQ + token
        const int r = idx / (D / 4), c = (idx % (D / 4)) * 4, h = r / TQ, t = r - h * TQ;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < nq) v = *reinterpret_cast<const float4*>(qkv + int64_t(q0 + t) * ld + (kvh * group + h) * D + c);
        *reinterpret_cast<float4*>(Qs + r * AG_LD + c) = v;
    }
    int last[4];  // last key each of this thread's rows may see
    float m[4], l[4], acc[4][8];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i, t = r % TQ;
        last[i] = t < nq ? pos0 + q0 + t : -1;
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 8; ++c) acc[i][c] = 0.f;
    }
    const int T = min(pos0 + q0 + nq, (chunk + 1) * kchunk * AG_K);  // keys of this chunk: [chunk * kchunk * 32, T)
    for (int t0 = chunk * kchunk * AG_K; t0 < T; t0 += AG_K) {
        __syncthreads();
        for (int idx = tid; idx < AG_K * (D / 4); idx += AG_THREADS) {
            const int j = idx / (D / 4), c = (idx % (D / 4)) * 4;
            float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
            if (t0 + j < T) {
                kv = *reinterpret_cast<const float4*>(kc + size_t(t0 + j) * KD + kvh * D + c);
                vv = *reinterpret_cast<const float4*>(vc + size_t(t0 + j) * KD + kvh * D + c);
            }
            *reinterpret_cast<float4*>(Ks + j * AG_LD + c) = kv;
            *reinterpret_cast<float4*>(Vs + j * D + c) = vv;
        }
        __syncthreads();
        float sc[4][2];  // rows ty*4+i, keys tx and tx+16
#pragma unroll
        for (int i = 0; i < 4; ++i) sc[i][0] = sc[i][1] = 0.f;
#pragma unroll 4
        for (int d4 = 0; d4 < D / 4; ++d4) {
            float4 q[4], k[2];
#pragma unroll
            for (int i = 0; i < 4; ++i) q[i] = *reinterpret_cast<const float4*>(Qs + (ty * 4 + i) * AG_LD + d4 * 4);
#pragma unroll
            for (int j = 0; j < 2; ++j) k[j] = *reinterpret_cast<const float4*>(Ks + (tx + 16 * j) * AG_LD + d4 * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    float a = sc[i][j];
                    a = __fadd_rn(a, __fmul_rn(q[i].x, k[j].x));
                    a = __fadd_rn(a, __fmul_rn(q[i].y, k[j].y));
                    a = __fadd_rn(a, __fmul_rn(q[i].z, k[j].z));
                    a = __fadd_rn(a, __fmul_rn(q[i].w, k[j].w));
                    sc[i][j] = a;
                }
        }
        float corr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float mx = -INFINITY;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                sc[i][j] = t0 + tx + 16 * j <= last[i] ? __fmul_rn(sc[i][j], scale) : -INFINITY;
                mx = fmaxf(mx, sc[i][j]);
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_new = fmaxf(m[i], mx);
            float sum = 0.f;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float pj = sc[i][j] == -INFINITY ? 0.f : expf(sc[i][j] - m_new);
                Ps[(ty * 4 + i) * AG_LDP + tx + 16 * j] = pj;
                sum += pj;
            }
#pragma unroll
            for (int o = 1; o < 16; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            corr[i] = m[i] == -INFINITY ? 0.f : expf(m[i] - m_new);
            l[i] = l[i] * corr[i] + sum;
            m[i] = m_new;
        }
        __syncwarp();  // a row's 16 threads are half a warp
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 8; ++c) acc[i][c] *= corr[i];
        const int nk = min(AG_K, T - t0);
        for (int j = 0; j < nk; ++j) {  // outputs: dims tx*4..+3 and 64+tx*4..+3
            const float4 v0 = *reinterpret_cast<const float4*>(Vs + j * D + tx * 4);
            const float4 v1 = *reinterpret_cast<const float4*>(Vs + j * D + 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float pj = Ps[(ty * 4 + i) * AG_LDP + j];
                acc[i][0] = fmaf(pj, v0.x, acc[i][0]); acc[i][1] = fmaf(pj, v0.y, acc[i][1]);
                acc[i][2] = fmaf(pj, v0.z, acc[i][2]); acc[i][3] = fmaf(pj, v0.w, acc[i][3]);
                acc[i][4] = fmaf(pj, v1.x, acc[i][4]); acc[i][5] = fmaf(pj, v1.y, acc[i][5]);
                acc[i][6] = fmaf(pj, v1.z, acc[i][6]); acc[i][7] = fmaf(pj, v1.w, acc[i][7]);
            }
        }
        __syncwarp();
    }
    if (n_chunks > 1) {  // leave this chunk's result; the last chunk of the query tile to arrive adds them all
        float* base = part + (size_t(kvh) * n_qt + qt) * AG_MAXCHUNK * AG_PART;
        float* mine = base + size_t(chunk) * AG_PART;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float* o = mine + (ty * 4 + i) * (D + 2);
            *reinterpret_cast<float2*>(o + tx * 4) = make_float2(acc[i][0], acc[i][1]);  // rows of D + 2 floats: 8-byte aligned
            *reinterpret_cast<float2*>(o + tx * 4 + 2) = make_float2(acc[i][2], acc[i][3]);
            *reinterpret_cast<float2*>(o + 64 + tx * 4) = make_float2(acc[i][4], acc[i][5]);
            *reinterpret_cast<float2*>(o + 64 + tx * 4 + 2) = make_float2(acc[i][6], acc[i][7]);
            if (tx == 0) { o[D] = m[i]; o[D + 1] = l[i]; }
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) {
            unsigned* cnt = counters + size_t(kvh) * n_qt + qt;
            const unsigned old = atomicAdd(cnt, 1u);
            s_last = old == unsigned(n_chunks - 1);
            if (s_last) *cnt = 0;
        }
        __syncthreads();
        if (!s_last) return;
        __threadfence();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = ty * 4 + i;
            float M = -INFINITY;
            for (int c = 0; c < n_chunks; ++c) M = fmaxf(M, __ldcg(base + size_t(c) * AG_PART + r * (D + 2) + D));
            float L = 0.f;
#pragma unroll
            for (int c8 = 0; c8 < 8; ++c8) acc[i][c8] = 0.f;
            for (int c = 0; c < n_chunks; ++c) {  // fixed chunk order
                const float* ps = base + size_t(c) * AG_PART + r * (D + 2);
                const float mc = __ldcg(ps + D);
                if (mc == -INFINITY) continue;
                const float w = expf(mc - M);
                L = fmaf(__ldcg(ps + D + 1), w, L);
                const float2 a0 = __ldcg(reinterpret_cast<const float2*>(ps + tx * 4)), a1 = __ldcg(reinterpret_cast<const float2*>(ps + tx * 4 + 2));
                const float2 b0 = __ldcg(reinterpret_cast<const float2*>(ps + 64 + tx * 4)), b1 = __ldcg(reinterpret_cast<const float2*>(ps + 64 + tx * 4 + 2));
                acc[i][0] = fmaf(a0.x, w, acc[i][0]); acc[i][1] = fmaf(a0.y, w, acc[i][1]);
                acc[i][2] = fmaf(a1.x, w, acc[i][2]); acc[i][3] = fmaf(a1.y, w, acc[i][3]);
                acc[i][4] = fmaf(b0.x, w, acc[i][4]); acc[i][5] = fmaf(b0.y, w, acc[i][5]);
                acc[i][6] = fmaf(b1.x, w, acc[i][6]); acc[i][7] = fmaf(b1.y, w, acc[i][7]);
            }
            l[i] = L;
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i, h = r / TQ, t = r - h * TQ;
        if (t >= nq) continue;
        const float inv = 1.0f / l[i];
        float* o = att + int64_t(q0 + t) * ld_att + (kvh * group + h) * D;
        *reinterpret_cast<float4*>(o + tx * 4) = make_float4(acc[i][0] * inv, acc[i][1] * inv, acc[i][2] * inv, acc[i][3] * inv);
        *reinterpret_cast<float4*>(o + 64 + tx * 4) = make_float4(acc[i][4] * inv, acc[i][5] * inv, acc[i][6] * inv, acc[i][7] * inv);
    }
}

// ---------------------------------------------------------------- rows of several sequences

// Row b of the batch is one token of sequence seqv[b] at position posv[b]; its q heads are normalised and rotated and
// its K/V row is in the cache already (k_qkv_post). Grid (B, HKV, most splits of a row): all q heads of a KV group share
// one pass over keys 0..posv[b] of that sequence (attn_core.cuh), cut into ranges of about `per_split` keys so that rows
// of different context lengths give CTAs of like work; the splits of a row meet in `part` and the last one to arrive
// adds them in split order.
// Bound by the K/V rows' bytes: 64 rows with 100-1000 keys on the 1.7B shape 111 -> 65 us per layer, 16 rows with 64-700
// keys on the 4B shape 51 -> 27 us, against tiles staged in shared memory, scores by one warp per head and a CTA per row.
struct AttnRowsParams {
    const float* qkv;
    int64_t ld;
    const float *kc, *vc;  // this layer's cache of sequence 0; sequence s starts seq_stride floats later
    size_t seq_stride;
    const int *posv, *seqv;
    float* att;
    int64_t ld_att;
    float* part;         // [B][HKV][nsplit][group][D + 2]
    unsigned* counters;  // [B][HKV]
    int H, HKV, nsplit, per_split;
    float scale;
};

constexpr int AR_WARPS = 8, AR_THREADS = 32 * AR_WARPS;

template <int GP>
__global__ void __launch_bounds__(AR_THREADS, 2) k_attn_rows(const AttnRowsParams p) {
    __shared__ __align__(16) float qs[GP * D];
    __shared__ __align__(16) float work[ac_smem_floats(GP, AR_WARPS)];
    __shared__ int s_last;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.x, kvh = blockIdx.y, split = blockIdx.z, group = p.H / p.HKV, KD = p.HKV * D;
    pdl_wait();
    const int T = p.posv[b] + 1, ns = min(p.nsplit, (T + p.per_split - 1) / p.per_split);
    if (split >= ns) return;
    const float* kc = p.kc + size_t(p.seqv[b]) * p.seq_stride + kvh * D;
    const float* vc = p.vc + size_t(p.seqv[b]) * p.seq_stride + kvh * D;
    for (int idx = tid; idx < GP * D; idx += AR_THREADS) qs[idx] = idx < group * D ? p.qkv[int64_t(b) * p.ld + (kvh * group) * D + idx] : 0.f;
    const AcSmem s = ac_smem(work, qs, GP, AR_WARPS);
    const int t0 = int(int64_t(T) * split / ns), t1 = int(int64_t(T) * (split + 1) / ns);
    float* out = p.att + int64_t(b) * p.ld_att + kvh * group * D;
    float* base = p.part + (size_t(b) * p.HKV + kvh) * p.nsplit * group * (D + 2);
    float* mine = base + size_t(split) * group * (D + 2);
    constexpr int KT = 32 / GP < 8 ? 32 / GP : 8;
    AcKeys<GP, KT, AR_WARPS> keys(kc, vc, size_t(KD), t0, t1, warp, lane);
    keys.first(-1);
    __syncthreads();
    keys.walk(-1, nullptr, nullptr, s, p.scale);
    ac_finish<GP, KT, AR_WARPS>(keys.w, s, group, warp, lane, [] { __syncthreads(); }, [&](int h, int d, float o) {
        if (ns == 1) out[h * D + d] = o / s.l[h];
        else mine[h * (D + 2) + d] = o;
    });
    if (ns == 1) return;
    if (tid < group) {
        mine[tid * (D + 2) + D] = s.m[tid];
        mine[tid * (D + 2) + D + 1] = s.l[tid];
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned* cnt = p.counters + size_t(b) * p.HKV + kvh;
        const unsigned old = atomicAdd(cnt, 1u);
        s_last = old == unsigned(ns - 1);
        if (s_last) *cnt = 0;
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int e = tid; e < group * D; e += AR_THREADS) {
        const int h = e / D, od = e % D;
        float M = -INFINITY;
        for (int q = 0; q < ns; ++q) M = fmaxf(M, __ldcg(base + (size_t(q) * group + h) * (D + 2) + D));
        float L = 0.f, o = 0.f;
#pragma unroll 4
        for (int q = 0; q < ns; ++q) {  // fixed split order
            const float* ps = base + (size_t(q) * group + h) * (D + 2);
            const float w = expf(__ldcg(ps + D) - M);
            L = fmaf(__ldcg(ps + D + 1), w, L);
            o = fmaf(__ldcg(ps + od), w, o);
        }
        out[e] = o / L;
    }
}

// Most splits a row can have when the batch has B rows: the partial results of AR_ROW_SPLITS (row, split) pairs fit.
constexpr int AR_ROW_SPLITS = 2048, AR_MAXSPLIT = 32;
static int attn_rows_most_splits(int B) { return std::max(1, std::min(AR_MAXSPLIT, AR_ROW_SPLITS / std::max(B, 1))); }
size_t attn_rows_part_floats(int H) { return size_t(AR_ROW_SPLITS) * H * (D + 2); }

// posv_host: the rows' positions on the host (they decide how the keys are cut)
int attn_rows_launch(const float* qkv, int64_t ld, const float* kc, const float* vc, size_t seq_stride, const int* posv,
                     const int* seqv, const int* posv_host, float* att, int64_t ld_att, float* part, unsigned* counters, int B, int H,
                     int HKV, float scale, int sm_count, cudaStream_t s, bool pdl) {
    if (H % HKV || H / HKV > AD_MAXG) return fail(ELB_ERR_UNSUPPORTED, "attention: at most 8 query heads per KV head");
    // Ranges of 256 keys, halved (down to 64: below that the fixed cost of a CTA and of the combination outweighs its keys)
    // until the GPU has two CTAs per SM.
    int Tmax = 1;
    for (int b = 0; b < B; ++b) Tmax = std::max(Tmax, posv_host[b] + 1);
    int per = 256;
    for (; per > 64; per /= 2) {
        int64_t ctas = 0;
        for (int b = 0; b < B; ++b) ctas += (posv_host[b] + per) / per;
        if (ctas * HKV >= 2 * int64_t(sm_count)) break;
    }
    const int most = attn_rows_most_splits(B);
    if ((Tmax + per - 1) / per > most) per = (Tmax + most - 1) / most;
    const int nsplit = (Tmax + per - 1) / per;
    AttnRowsParams p{qkv, ld, kc, vc, seq_stride, posv, seqv, att, ld_att, part, counters, H, HKV, nsplit, per, scale};
    const dim3 grid{unsigned(B), unsigned(HKV), unsigned(nsplit)};
    const int group = H / HKV;
    return launch_after(group <= 2 ? k_attn_rows<2> : group <= 4 ? k_attn_rows<4> : k_attn_rows<8>, grid, dim3(AR_THREADS), 0, s, pdl, p);
}

// ---------------------------------------------------------------- RMSNorm over rows (el::rmsnorm, src/ops.cpp:155-160)
__global__ void __launch_bounds__(256) k_rmsnorm_rows(float* out, const float* x, const float* w, int n, float eps) {
    __shared__ double red8[8];
    const int tid = threadIdx.x;
    const float* xr = x + int64_t(blockIdx.x) * n;
    float* o = out + int64_t(blockIdx.x) * n;
    double ss = 0.0;
    for (int i = tid; i < n; i += 256) { const double v = xr[i]; ss += v * v; }
    ss = warp_sum(ss);
    if ((tid & 31) == 0) red8[tid >> 5] = ss;
    __syncthreads();
    ss = 0.0;
    for (int i = 0; i < 8; ++i) ss += red8[i];
    const float inv = float(1.0 / sqrt(ss / n + double(eps)));
    for (int i = tid; i < n; i += 256) o[i] = __fmul_rn(__fmul_rn(xr[i], inv), w[i]);
}

// ---------------------------------------------------------------- logits post-processing
// What the reference's generate loop does on the host with the n_vocab logits of every token (src/main.cpp:309-320):
// log-sum-exp in double precision and the k best tokens ordered by (logit descending, id ascending).
// allowed != nullptr: bit i of the array says whether token i may be picked (the log-sum-exp still covers all tokens).
// Row b: logits + b * ld -> out + b * TOP_BYTES.

// An order-preserving integer of (value descending, index ascending): the larger key comes first. 0: no candidate (NaN
// never is one; -0 and +0 are the same value).
__device__ __forceinline__ unsigned long long top_key(float v, int i) {
    if (v != v) return 0ull;
    const unsigned u = __float_as_uint(v + 0.0f);
    return (unsigned long long)(u & 0x80000000u ? ~u : u | 0x80000000u) << 32 | unsigned(~i);
}
// the largest key of the warp's lanes, on every lane
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
    const unsigned hi = __reduce_max_sync(0xffffffffu, unsigned(k >> 32));
    const unsigned lo = __reduce_max_sync(0xffffffffu, unsigned(k >> 32) == hi ? unsigned(k) : 0u);
    return (unsigned long long)hi << 32 | lo;
}

// Grid (chunk, row). A CTA takes a chunk of TP_CHUNK logits (TP_PER per lane, in registers): its maximum, its sum of
// exponentials and its k best, which each warp finds for its own part and warp 0 merges. The last CTA of a row to arrive
// merges the chunks in chunk order. One block per row was bound by its single SM's exponentials in double and by k + 2
// passes of one block over the row: 100 us for 64 rows at k = 1, 186 us for 16 rows at k = 4 (151 936 logits each).
constexpr int TP_WARPS = 8, TP_THREADS = 32 * TP_WARPS, TP_PER = 10, TP_CHUNK = TP_THREADS * TP_PER;
constexpr int TP_HEADS = TP_WARPS * TOP_MAXK * 8;  // most chunks of a row: one byte of the list area each (10 million logits)
struct TopChunk { double sum; float mx; int pad; };
__global__ void __launch_bounds__(TP_THREADS) k_logits_top(const float* __restrict__ logits, int n, int k, uint8_t* __restrict__ out,
                                                           const uint32_t* __restrict__ allowed, int64_t ld, TopChunk* __restrict__ parts,
                                                           unsigned long long* __restrict__ cand, unsigned* __restrict__ arrived) {
    const int chunks = gridDim.x, c = blockIdx.x, row = blockIdx.y;
    logits += int64_t(row) * ld;
    out += size_t(row) * TOP_BYTES;
    parts += size_t(row) * chunks;
    cand += size_t(row) * chunks * k;
    __shared__ unsigned long long lists[TP_WARPS * TOP_MAXK];
    __shared__ float red_f[TP_WARPS];
    __shared__ double red_d[TP_WARPS];
    __shared__ bool s_last;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    float v[TP_PER];
    const int base = c * TP_CHUNK + tid;
    float mx = -INFINITY;
#pragma unroll
    for (int j = 0; j < TP_PER; ++j) {
        const int i = base + j * TP_THREADS;
        v[j] = i < n ? __ldcg(logits + i) : -INFINITY;
        mx = fmaxf(mx, v[j]);
    }
    mx = warp_max(mx);
    if (lane == 0) red_f[warp] = mx;
    __syncthreads();
    mx = red_f[0];
#pragma unroll
    for (int w = 1; w < TP_WARPS; ++w) mx = fmaxf(mx, red_f[w]);
    const double from = mx == -INFINITY ? 0.0 : double(mx);  // (no finite logit: the sum is then 0, or NaN if one of them is)
    double sum = 0.0;
#pragma unroll 1
    for (int j = 0; j < TP_PER; ++j) {
        const int i = base + j * TP_THREADS;
        if (i < n) sum += exp(double(__ldcg(logits + i)) - from);
    }
    sum = warp_sum(sum);
    if (lane == 0) red_d[warp] = sum;
    unsigned long long key[TP_PER];
#pragma unroll
    for (int j = 0; j < TP_PER; ++j) {
        const int i = base + j * TP_THREADS;
        key[j] = i < n && (!allowed || ((allowed[i >> 5] >> (i & 31)) & 1u)) ? top_key(v[j], i) : 0ull;
    }
    for (int r = 0; r < k; ++r) {  // the warp's k best, in order
        unsigned long long best = key[0];
#pragma unroll
        for (int j = 1; j < TP_PER; ++j) best = key[j] > best ? key[j] : best;
        best = warp_max_key(best);
        if (lane == 0) lists[warp * k + r] = best;
#pragma unroll
        for (int j = 0; j < TP_PER; ++j)
            if (key[j] == best) key[j] = 0ull;
    }
    __syncthreads();
    if (warp == 0) {
        int at = 0;
        for (int r = 0; r < k; ++r) {  // merge of the sorted lists: lane w holds the head of warp w's
            const unsigned long long head = lane < TP_WARPS && at < k ? lists[lane * k + at] : 0ull;
            const unsigned long long best = warp_max_key(head);
            if (best && head == best) ++at;
            if (lane == 0) __stcg(cand + size_t(c) * k + r, best);
        }
        if (lane == 0) {
            double t = 0.0;
            for (int w = 0; w < TP_WARPS; ++w) t += red_d[w];  // fixed order
            __stcg(&parts[c].sum, t);
            __stcg(&parts[c].mx, mx);
            __threadfence();
            const unsigned seen = atomicAdd(arrived + row, 1u);
            s_last = seen == unsigned(chunks - 1);
            if (s_last) arrived[row] = 0;  // ready for the next launch
        }
    }
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (warp == 1) {  // log-sum-exp over the chunks (a lane's chunks in order, then the lanes in a fixed tree)
        float M = -INFINITY;
        for (int i = lane; i < chunks; i += 32) M = fmaxf(M, __ldcg(&parts[i].mx));
        M = warp_max(M);
        double t = 0.0;
        for (int i = lane; i < chunks; i += 32) t += __ldcg(&parts[i].sum) * exp(double(__ldcg(&parts[i].mx)) - double(M));
        t = warp_sum(t);
        if (lane == 0) *reinterpret_cast<double*>(out) = double(M) + log(t);
    }
    if (warp == 0) {
        int32_t* ids = reinterpret_cast<int32_t*>(out + 8);
        float* vals = reinterpret_cast<float*>(out + 8 + 4 * TOP_MAXK);
        // lane's lists: chunks lane, lane + 32, ...; the best head of the lane's lists is kept, and looked for again only
        // on the lane whose list gave a pick (heads[]: how far list i has been used up)
        uint8_t* heads = reinterpret_cast<uint8_t*>(lists);
        for (int i = lane; i < chunks; i += 32) heads[i] = 0;
        auto look = [&](int& from) {
            unsigned long long b = 0ull;
            for (int i = lane; i < chunks; i += 32) {
                const unsigned long long h = heads[i] < k ? __ldcg(cand + size_t(i) * k + heads[i]) : 0ull;
                if (h > b) { b = h; from = i; }
            }
            return b;
        };
        int from = 0;
        unsigned long long head = look(from);
        for (int r = 0; r < k; ++r) {
            const unsigned long long best = warp_max_key(head);
            if (lane == 0) {
                const int i = int(~unsigned(best));
                ids[r] = best ? i : -1;  // fewer than k tokens allowed: -1 from here on
                vals[r] = best ? __ldcg(logits + i) : -INFINITY;
            }
            if (best && head == best) { ++heads[from]; head = look(from); }
        }
    }
}

// scratch of logits_top_launch for up to `rows` rows of n logits: arrival counters (zero at first, and between launches),
// then candidates and sums of the chunks
static size_t top_counter_bytes(int rows) { return (size_t(rows) * sizeof(unsigned) + 15) / 16 * 16; }
size_t logits_top_scratch_bytes(int n, int rows) {
    const size_t chunks = size_t(n + TP_CHUNK - 1) / TP_CHUNK;
    return top_counter_bytes(rows) + size_t(rows) * chunks * (TOP_MAXK * 8 + sizeof(TopChunk));
}

// rows of logits [rows][ld] -> out [rows][TOP_BYTES]; scratch: logits_top_scratch_bytes(n, scratch_rows) bytes
int logits_top_launch(const float* logits, int n, int64_t ld, int rows, int k, uint8_t* out, void* scratch, int scratch_rows,
                      cudaStream_t s, const uint32_t* d_allowed) {
    if (!logits || !out || !scratch || n < 1 || rows < 1 || rows > scratch_rows || k < 1 || k > TOP_MAXK || k > n)
        return fail(ELB_ERR_INVALID, "logits_top: bad argument");
    const int chunks = (n + TP_CHUNK - 1) / TP_CHUNK;
    if (chunks > TP_HEADS) return fail(ELB_ERR_UNSUPPORTED, "logits_top: vocabulary too large");
    auto* cand = reinterpret_cast<unsigned long long*>(static_cast<uint8_t*>(scratch) + top_counter_bytes(scratch_rows));
    auto* parts = reinterpret_cast<TopChunk*>(cand + size_t(rows) * chunks * TOP_MAXK);
    k_logits_top<<<dim3(unsigned(chunks), unsigned(rows)), TP_THREADS, 0, s>>>(logits, n, k, out, d_allowed, ld, parts, cand,
                                                                              static_cast<unsigned*>(scratch));
    ELB_CUDA(cudaGetLastError());
    return ELB_OK;
}

// ---------------------------------------------------------------- host side

int attn_decode_launch(const AttnDecodeArgs& a, cudaStream_t s) {
    if (a.H % a.HKV || a.H / a.HKV > AD_MAXG) return fail(ELB_ERR_UNSUPPORTED, "attention: at most 8 query heads per KV head");
    if (a.nsplit < 1 || a.nsplit > AD_MAXSPLIT) return fail(ELB_ERR_INVALID, "attention: split count out of range");
    AttnDecodeParams p{a.qkv, a.q_norm, a.k_norm, reinterpret_cast<const float2*>(a.rope), a.pos, a.kc, a.vc, a.att, a.part,
                       a.counters, a.H, a.HKV, a.rope_dim, a.nsplit, a.eps, a.scale, a.post};
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(a.HKV, a.nsplit);
    cfg.blockDim = dim3(AD_THREADS);
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = a.pdl ? 1 : 0;
    ELB_CUDA(cudaLaunchKernelEx(&cfg, k_attn_decode, p));
    return ELB_OK;
}

int qkv_post_launch(float* qkv, int64_t ld, const float* q_norm, const float* k_norm, const float* rope, int pos0, int B,
                    float* kc, float* vc, int H, int HKV, int rope_dim, float eps, cudaStream_t s, const int* posv,
                    const int* seqv, size_t seq_stride, bool pdl) {
    return launch_after(k_qkv_post, dim3(B, (H + 2 * HKV + 7) / 8), dim3(32, 8), 0, s, pdl, qkv, ld, q_norm, k_norm,
                        reinterpret_cast<const float2*>(rope), pos0, kc, vc, H, HKV, rope_dim, eps, posv, seqv, seq_stride);
}

size_t attn_prefill_scratch_floats(int max_batch, int H, int HKV) {  // partial results of the chunked prompt attention
    const int group = std::max(1, H / HKV), TQ = AG_ROWS % group == 0 ? AG_ROWS / group : AG_ROWS;
    return size_t(HKV) * size_t((max_batch + TQ - 1) / TQ) * AG_MAXCHUNK * AG_PART;
}
size_t attn_prefill_counters(int max_batch, int H, int HKV) {
    const int group = std::max(1, H / HKV), TQ = AG_ROWS % group == 0 ? AG_ROWS / group : AG_ROWS;
    return size_t(HKV) * size_t((max_batch + TQ - 1) / TQ);
}

int attn_prefill_launch(const float* qkv, int64_t ld, const float* kc, const float* vc, float* att, int64_t ld_att,
                        int pos0, int B, int H, int HKV, float scale, cudaStream_t s, float* part, unsigned* counters) {
    ELB_TRY(ensure_dyn_smem((const void*)k_attn_prefill, AP_SMEM));
    ELB_TRY(ensure_dyn_smem((const void*)k_attn_prefill_gqa, AG_SMEM));
    const int group = H / HKV;
    static const bool old_kernel = [] { const char* v = std::getenv("ELB_ATTN_SIMPLE"); return v && v[0] == '1'; }();
    if (!old_kernel && H % HKV == 0 && AG_ROWS % group == 0 && ld % 4 == 0 && ld_att % 4 == 0) {
        const int TQ = AG_ROWS / group, n_qt = (B + TQ - 1) / TQ;
        // chunks of 4 key tiles (128 keys), longer when the context is long enough to need more than AG_MAXCHUNK of them;
        // without scratch memory one chunk per query tile
        const int tiles_max = (pos0 + B + AG_K - 1) / AG_K;
        const int kchunk = part && counters ? std::max(4, (tiles_max + AG_MAXCHUNK - 1) / AG_MAXCHUNK) : tiles_max;
        int items = 0;
        for (int i = 0; i < n_qt; ++i) items += ag_chunks(pos0, B, TQ, i, kchunk);
        k_attn_prefill_gqa<<<dim3(HKV, items), AG_THREADS, AG_SMEM, s>>>(qkv, ld, kc, vc, att, ld_att, pos0, B, H, HKV, scale,
                                                                         kchunk, part, counters);
        ELB_CUDA(cudaGetLastError());
        return ELB_OK;
    }
    k_attn_prefill<<<dim3(H, (B + AP_Q - 1) / AP_Q), AP_THREADS, AP_SMEM, s>>>(qkv, ld, kc, vc, att, ld_att, pos0, B, H, HKV,
                                                                             scale);
    ELB_CUDA(cudaGetLastError());
    return ELB_OK;
}

int rmsnorm_launch(float* out, const float* x, const float* w, int n, float eps, int rows, cudaStream_t s) {
    k_rmsnorm_rows<<<rows, 256, 0, s>>>(out, x, w, n, eps);
    ELB_CUDA(cudaGetLastError());
    return ELB_OK;
}

}  // namespace elb
