// Attention of one query token over a range of cached keys, by all warps of a block (src/model.cpp:191-214 of the
// reference): shared by the one-GPU decode kernel (decode_one.cu) and the batched rows kernel (attn.cu).
//
// Bound by the bytes of the key and value rows, each read once for all query heads of its KV head, and at short contexts
// by the chain of latencies: so every warp walks its own tiles of a few keys with its own running maximum, sum and
// outputs, asks for the next tile's rows while it works on the current one, and the warps meet once, at the end.
// Within a tile:
//   scores   16 lanes share a key (2 keys per pass), a lane holds 8 dimensions of up to 4 query heads; the sums over the
//            16 lanes are a transposing butterfly (5 exchanges for 4 heads, not 16);
//   softmax  lane = (key, head);
//   values   lane = 4 dimensions of every head, probabilities broadcast from shared memory: no shuffles.
// Scores by one warp per head over tiles shared by the block, three block barriers per tile, took 37 us per layer of the
// decode kernel at 4375 keys on the 4B shape (36 MB of rows: 5.6 us at the copy rate).
#pragma once

#include "common.cuh"

namespace elb {

constexpr int AC_D = 128;  // head_dim
// GP: query heads of a KV head, rounded up to 2, 4 or 8
__host__ __device__ constexpr int ac_red_heads(int GP) { return GP < 4 ? GP : 4; }  // heads whose partial outputs meet in shared memory together
__host__ __device__ constexpr int ac_smem_floats(int GP, int warps) {
    return warps * ac_red_heads(GP) * AC_D  // partial outputs; during the tiles: 32 probabilities per warp
           + 2 * warps * 8 + 2 * 8;         // maximum and sum of every (warp, head), then of every head
}

struct AcSmem {
    const float* qs;  // [GP][128] query heads (heads beyond the group: anything finite)
    float* red;
    float *mw, *lw;   // [warps][8]
    float *m, *l;     // [8]: of the block's keys, valid for every thread once the outputs are emitted
};
__device__ __forceinline__ AcSmem ac_smem(float* base, const float* qs, int GP, int warps) {
    AcSmem s;
    s.qs = qs;
    s.red = base;
    s.mw = base + warps * ac_red_heads(GP) * AC_D;
    s.lw = s.mw + warps * 8;
    s.m = s.lw + warps * 8;
    s.l = s.m + 8;
    return s;
}

__device__ __forceinline__ float4 ac_ld(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float ac_dot(const float4& a, const float4& b, float s) {
    return fmaf(a.x, b.x, fmaf(a.y, b.y, fmaf(a.z, b.z, fmaf(a.w, b.w, s))));
}

// One warp's running state and its tile step. KT: keys of a tile (KT * GP <= 32).
template <int GP, int KT> struct AcWarp {
    static constexpr int SG = GP < 4 ? GP : 4;  // heads scored together
    float4 acc[GP];  // outputs, dimensions 4 * lane ..
    float m, l;      // lane = (key, head): of head lane % GP (the same on all lanes of a head)

    __device__ __forceinline__ void init() {
#pragma unroll
        for (int h = 0; h < GP; ++h) acc[h] = make_float4(0.f, 0.f, 0.f, 0.f);
        m = -INFINITY;
        l = 0.f;
    }

    // scores of the tile's keys: lane key * GP + head gets score (key, head). k[u][i]: dimensions 64 i + 4 (lane % 16) ..
    // of key 2 u + lane / 16.
    __device__ __forceinline__ float scores(const float4 (&k)[KT / 2][2], const float* qs, float scale, int lane) {
        const int c = lane & 15;
        const int head = lane % GP, key = lane / GP;
        float out = 0.f;
#pragma unroll
        for (int h0 = 0; h0 < GP; h0 += SG) {
            float4 q[SG][2];
#pragma unroll
            for (int h = 0; h < SG; ++h)
#pragma unroll
                for (int i = 0; i < 2; ++i) q[h][i] = ac_ld(qs + (h0 + h) * AC_D + 64 * i + 4 * c);
#pragma unroll
            for (int u = 0; u < KT / 2; ++u) {
                // A lane's 8 products are added in fp32, the 16 lanes of a key in double: a score is then rounded about
                // once, and softmax passes its rounding on undamped.
                double a[SG];
#pragma unroll
                for (int h = 0; h < SG; ++h) a[h] = double(ac_dot(q[h][0], k[u][0], 0.f) + ac_dot(q[h][1], k[u][1], 0.f));
                double r;  // a lane ends up with one head (SG == 4: head c / 4, SG == 2: head c / 8)
                const bool up = c & 8;
                if (SG == 4) {
                    const bool up2 = c & 4;
                    const double s0 = up ? a[0] : a[2 % SG], s1 = up ? a[1 % SG] : a[3 % SG];
                    const double k0 = up ? a[2 % SG] : a[0], k1 = up ? a[3 % SG] : a[1 % SG];
                    const double b0 = k0 + __shfl_xor_sync(0xffffffffu, s0, 8), b1 = k1 + __shfl_xor_sync(0xffffffffu, s1, 8);
                    r = (up2 ? b1 : b0) + __shfl_xor_sync(0xffffffffu, up2 ? b0 : b1, 4);
                } else {
                    r = (up ? a[1 % SG] : a[0]) + __shfl_xor_sync(0xffffffffu, up ? a[0] : a[1 % SG], 8);
                    r += __shfl_xor_sync(0xffffffffu, r, 4);
                }
                r += __shfl_xor_sync(0xffffffffu, r, 2);
                r += __shfl_xor_sync(0xffffffffu, r, 1);
                const float got = __shfl_sync(0xffffffffu, float(r * double(scale)), (key & 1) * 16 + (head % SG) * (16 / SG));
                if ((key >> 1) == u && head >= h0 && head < h0 + SG) out = got;
            }
        }
        return out;
    }

    // softmax of the tile's nk <= KT keys and v rows of it; v[j]: dimensions 4 * lane .. of key j; ps: 32 floats of this warp
    __device__ __forceinline__ void add(float score, const float4 (&v)[KT], int nk, float* ps, int lane) {
        const bool on = lane / GP < nk && lane < KT * GP;
        float mx = on ? score : -INFINITY;
#pragma unroll
        for (int o = GP; o < 32; o *= 2) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
        const float m_new = fmaxf(m, mx);
        const float from = m_new == -INFINITY ? 0.f : m_new;  // (keys at -infinity: probability 0, also when no other has come yet)
        const float p = on ? expf(score - from) : 0.f;
        float sum = p;
#pragma unroll
        for (int o = GP; o < 32; o *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, o);
        const float corr = expf(m - from);  // (0 for the first tile)
        const bool moved = m_new != m;
        l = l * corr + sum;
        m = m_new;
        __syncwarp();
        ps[lane] = p;
        if (__any_sync(0xffffffffu, moved)) {
#pragma unroll
            for (int h = 0; h < GP; ++h) {
                const float c = __shfl_sync(0xffffffffu, corr, h);
                acc[h].x *= c; acc[h].y *= c; acc[h].z *= c; acc[h].w *= c;
            }
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < KT; ++j) {  // (rows past nk have probability 0)
            float w[GP];
            if (GP == 2) {
                const float2 x = *reinterpret_cast<const float2*>(ps + j * GP);
                w[0] = x.x; w[1] = x.y;
            } else {
#pragma unroll
                for (int i = 0; i < GP / 4; ++i) {
                    const float4 x = ac_ld(ps + j * GP + 4 * i);
                    w[4 * i % GP] = x.x; w[(4 * i + 1) % GP] = x.y; w[(4 * i + 2) % GP] = x.z; w[(4 * i + 3) % GP] = x.w;
                }
            }
#pragma unroll
            for (int h = 0; h < GP; ++h) {
                acc[h].x = fmaf(w[h], v[j].x, acc[h].x);
                acc[h].y = fmaf(w[h], v[j].y, acc[h].y);
                acc[h].z = fmaf(w[h], v[j].z, acc[h].z);
                acc[h].w = fmaf(w[h], v[j].w, acc[h].w);
            }
        }
    }
};

// The warps of the block meet: calls emit(head, dimension, value) once for every output of the group, by the thread that
// holds it: value = sum over the block's keys of exp(score - s.m[head]) * v. sync: a barrier of the block's WARPS warps.
template <int GP, int KT, int WARPS, class Sync, class Emit>
__device__ __forceinline__ void ac_finish(const AcWarp<GP, KT>& w, const AcSmem& s, int group, int warp, int lane, Sync sync, Emit emit) {
    constexpr int RH = ac_red_heads(GP);
    if (lane < GP) { s.mw[warp * 8 + lane] = w.m; s.lw[warp * 8 + lane] = w.l; }
#pragma unroll
    for (int h0 = 0; h0 < GP; h0 += RH) {
        if (h0 >= group) break;
        sync();  // every warp's maximum is there; the probabilities (or the previous heads' outputs) have been used
        float c = 0.f;  // lane h < RH: this warp's factor for head h0 + h
        if (lane < RH) {
            float M = -INFINITY;
#pragma unroll
            for (int i = 0; i < WARPS; ++i) M = fmaxf(M, s.mw[i * 8 + h0 + lane]);
            const float mine = s.mw[warp * 8 + h0 + lane];
            c = mine == -INFINITY ? 0.f : expf(mine - M);
            if (warp == 0) {
                float L = 0.f;
#pragma unroll
                for (int i = 0; i < WARPS; ++i) {
                    const float mi = s.mw[i * 8 + h0 + lane];
                    L += mi == -INFINITY ? 0.f : s.lw[i * 8 + h0 + lane] * expf(mi - M);
                }
                s.m[h0 + lane] = M;
                s.l[h0 + lane] = L;
            }
        }
#pragma unroll
        for (int h = 0; h < RH; ++h) {
            const float f = __shfl_sync(0xffffffffu, c, h);
            const float4 a = w.acc[h0 + h];
            *reinterpret_cast<float4*>(s.red + (warp * RH + h) * AC_D + 4 * lane) = make_float4(a.x * f, a.y * f, a.z * f, a.w * f);
        }
        sync();
#pragma unroll 1
        for (int e = warp * 32 + lane; e < RH * AC_D; e += WARPS * 32) {
            const int h = e / AC_D, d = e % AC_D;
            if (h0 + h >= group) continue;
            float o = 0.f;
#pragma unroll
            for (int i = 0; i < WARPS; ++i) o += s.red[(i * RH + h) * AC_D + d];  // fixed order
            emit(h0 + h, d, o);
        }
    }
}

// One warp's walk over its tiles of the block's keys [t0, t1), rows straight from global memory into registers. Row t_last
// comes from knew / vnew (shared memory, or null when t_last < 0): this step appends it. first() asks for the first tile,
// which needs nothing of the step's own results; walk() works through all of them.
template <int GP, int KT, int WARPS> struct AcKeys {
    AcWarp<GP, KT> w;
    float4 k[KT / 2][2], v[KT];
    const float *kc, *vc;
    size_t stride;
    int t, t1, warp, lane;
    __device__ __forceinline__ AcKeys(const float* kc_, const float* vc_, size_t stride_, int t0, int t1_, int warp_, int lane_)
        : kc(kc_), vc(vc_), stride(stride_), t(t0 + warp_ * KT), t1(t1_), warp(warp_), lane(lane_) {
        w.init();
    }
    __device__ __forceinline__ void load_k(int at, int t_last, const float* knew) {
#pragma unroll
        for (int u = 0; u < KT / 2; ++u) {
            const int j = min(at + 2 * u + (lane >> 4), t1 - 1);
            const float* row = (knew && j == t_last ? knew : kc + size_t(j) * stride) + 4 * (lane & 15);
            k[u][0] = ac_ld(row);
            k[u][1] = ac_ld(row + 64);
        }
    }
    __device__ __forceinline__ void load_v(int at, int t_last, const float* vnew) {
#pragma unroll
        for (int u = 0; u < KT; ++u) {
            const int j = min(at + u, t1 - 1);
            v[u] = ac_ld((vnew && j == t_last ? vnew : vc + size_t(j) * stride) + 4 * lane);
        }
    }
    __device__ __forceinline__ void first(int t_last) {
        if (t < t1 && !(t_last >= t && t_last < t + KT)) { load_k(t, -1, nullptr); load_v(t, -1, nullptr); }
    }
    __device__ __forceinline__ void walk(int t_last, const float* knew, const float* vnew, const AcSmem& s, float scale) {
        if (t < t1 && t_last >= t && t_last < t + KT) { load_k(t, t_last, knew); load_v(t, t_last, vnew); }
#pragma unroll 1
        while (t < t1) {
            const int next = t + WARPS * KT;
            const float score = w.scores(k, s.qs, scale, lane);
            if (next < t1) load_k(next, t_last, knew);
            w.add(score, v, t1 - t, s.red + warp * 32, lane);
            if (next < t1) load_v(next, t_last, vnew);
            t = next;
        }
    }
};

}  // namespace elb
