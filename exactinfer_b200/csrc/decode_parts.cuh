// What the two persistent decode kernels (decode_one.cu: one GPU; decode.cu: tensor parallel) share: the split of an
// activation into limbs, the unit stream of a working warp with its ring in shared memory and the producer warp that
// fills it, and the per-head norm + RoPE.
#pragma once

#include "common.cuh"
#include "split.cuh"
#include "gemv_core.cuh"
#include "decode.cuh"

namespace elb {

constexpr int DK_THREADS = 512, DK_WARPS = DK_THREADS / 32;  // the working warps
constexpr int DK_NBAR = 8;  // mbarriers per warp = most units a warp can have requested and not yet consumed
// How long the producer warp sleeps when no ring has room (ns). It shares a scheduler with four working warps:
// 500-1000 ns measured 0.6 % faster per step than 40 ns, 2000 ns 2 % slower (the rings run dry).
#ifndef DK_PRODUCER_NAP
#define DK_PRODUCER_NAP 500
#endif
constexpr int DK_HD = 128, DK_MAXG = 8;
constexpr int DK_MAXSPLIT = 18;         // key splits of one KV head
constexpr int DK_PS = DK_HD + 4;        // floats per (split, head) of the attention's partial results: 128 outputs, m, l, padding
constexpr unsigned DK_SPIN_LIMIT = 1u << 22;
constexpr unsigned DK_MBAR_LIMIT = 1u << 17;   // tries of one wait for a weight unit (each try blocks for a while in hardware)

// CTA barrier of the working warps (the producer warp runs on its own): a named barrier over DK_THREADS threads
__device__ __forceinline__ void dk_sync() { asm volatile("bar.sync 1, %0;" ::"n"(DK_THREADS) : "memory"); }

// ---------------------------------------------------------------- activation -> limbs in shared memory

// The split activation of a matvec: int8 limbs [4][n_pad], the sums of each limb over the 32-wide (Q4_K's min term) and
// 16-wide (Q6_K's offset) sub-blocks as two balanced base-256 digits each, in the layout the matvec's extra MMA reads
// (split.cuh), and one power-of-two scale per 256-block: here every 256-block is split on its own, with the shift
// k = 8 nl - 2 - e of its own largest magnitude (k_split8 of the reference, src/cuda/model_cuda.cu:701-729, applied per
// block; the matvec multiplies each block's exact integer sums by 2^-k of that block). A block is then converted
// without knowing anything about the rest of the vector: no maximum over the whole vector has to be agreed on.
struct ActSmem {
    int8_t* lim;    // [4][n_pad]
    int8_t* sd32;   // [n/256][8][8]
    int8_t* sd16;   // [n/256][8][16]
    float* bscale;  // [n/256] 2^-k of each block
    int n_pad;
};
__host__ __device__ inline size_t dk_act_bytes(int n) {  // limbs, sums, scales (a multiple of 16)
    return (size_t(4) * (n + 32) + size_t(n / 256) * 192 + size_t(n / 256) * 4 + 15) / 16 * 16;
}
__device__ __forceinline__ ActSmem act_at(int8_t* base, int n) {
    ActSmem a;
    a.lim = base;
    a.n_pad = n + 32;
    a.sd32 = a.lim + 4 * a.n_pad;
    a.sd16 = a.sd32 + (n / 256) * 64;
    a.bscale = reinterpret_cast<float*>(a.sd16 + (n / 256) * 128);
    return a;
}
__device__ __forceinline__ int sd_need(int type) { return type == ELB_Q4_K ? 1 : type == ELB_Q6_K ? 2 : 0; }
__device__ __forceinline__ int unit_bytes_of(int type) { return type == ELB_Q4_K ? Q4K_UNIT : type == ELB_Q6_K ? Q6K_UNIT : Q8_UNIT; }
// 1 / sqrt(x) in double from the single-precision estimate and two Newton steps (relative error ~1e-27 of the exact
// value before the last rounding): what the reference's 1.0 / sqrt(x) in double gives, after rounding to float,
// without the division and square root routines; those only beyond the range of a float (values of more than 1e19)
static __device__ __noinline__ double rsqrt_far(double x) { return 1.0 / sqrt(x); }
__device__ __forceinline__ double rsqrt_d(double x) {
    if (!(x > 1e-37 && x < 1e38)) return rsqrt_far(x);
    double y = double(rsqrtf(float(x)));
    y = y * fma(-0.5 * x, y * y, 1.5);
    y = y * fma(-0.5 * x, y * y, 1.5);
    return y;
}
__device__ __forceinline__ float pow2_neg(int k) { return k <= 126 ? __int_as_float((127 - k) << 23) : ldexpf(1.0f, -k); }

// Four consecutive fixed-point values -> one packed word of each of the 4 limbs (balanced base-256 digits: adding 128 at
// every byte position turns them into the ordinary digits of v + 0x80808080; a 4x4 byte transpose groups them by limb).
__device__ __forceinline__ void limb_words(const float4& f, const Pow2 sc, uint32_t (&w)[4]) {
    const uint32_t a = (uint32_t(__float2int_rn(f.x * sc.s1 * sc.s2)) + 0x80808080u) ^ 0x80808080u;
    const uint32_t b = (uint32_t(__float2int_rn(f.y * sc.s1 * sc.s2)) + 0x80808080u) ^ 0x80808080u;
    const uint32_t c = (uint32_t(__float2int_rn(f.z * sc.s1 * sc.s2)) + 0x80808080u) ^ 0x80808080u;
    const uint32_t d = (uint32_t(__float2int_rn(f.w * sc.s1 * sc.s2)) + 0x80808080u) ^ 0x80808080u;
    const uint32_t ab01 = __byte_perm(a, b, 0x5140), ab23 = __byte_perm(a, b, 0x7362);  // a0 b0 a1 b1 | a2 b2 a3 b3
    const uint32_t cd01 = __byte_perm(c, d, 0x5140), cd23 = __byte_perm(c, d, 0x7362);
    w[0] = __byte_perm(ab01, cd01, 0x5410);
    w[1] = __byte_perm(ab01, cd01, 0x7632);
    w[2] = __byte_perm(ab23, cd23, 0x5410);
    w[3] = __byte_perm(ab23, cd23, 0x7632);
}

// One warp splits 256-block b of a vector: lane holds its values 8*lane .. 8*lane+7 in v0, v1. Writes limbs, sub-block
// sums (shuffles over the 2 / 4 neighbouring lanes that hold the rest of a sub-block; the sums of two limbs travel in
// the halves of one word: |sum of 32 int8| < 2^12) and the block's scale. Every lane of the warp must call this together.
__device__ __forceinline__ void split_block(const float4& v0, const float4& v1, const int b, const int nl, const ActSmem& a,
                                            const int sd_mask, const int lane) {
    float m = fmaxf(absmax4(v0), absmax4(v1));
    m = warp_max(m);
    const int k = split_shift(m, nl);
    const Pow2 sc = make_pow2(k);
    uint32_t w0[4], w1[4];
    limb_words(v0, sc, w0);
    limb_words(v1, sc, w1);
    const int idx = b * 256 + lane * 8;
#pragma unroll
    for (int l = 0; l < 4; ++l) *reinterpret_cast<uint2*>(a.lim + l * a.n_pad + idx) = make_uint2(w0[l], w1[l]);
    if (sd_mask) {
#pragma unroll
        for (int h = 0; h < 2; ++h) {  // limbs 2h and 2h+1 together
            const int sa = __dp4a(int(w1[2 * h]), 0x01010101, __dp4a(int(w0[2 * h]), 0x01010101, 0));
            const int sb = __dp4a(int(w1[2 * h + 1]), 0x01010101, __dp4a(int(w0[2 * h + 1]), 0x01010101, 0));
            int pk = sa + (sb << 16);  // (the low half may borrow from the high one: undone when they are taken apart)
            const int p16 = pk + __shfl_xor_sync(0xffffffffu, pk, 1);
            const int p32 = p16 + __shfl_xor_sync(0xffffffffu, p16, 2);
#pragma unroll
            for (int wd = 0; wd < 2; ++wd) {
                if (!(sd_mask & (wd ? 1 : 2))) continue;
                const int pw = wd ? p32 : p16, per = wd ? 8 : 16, si = wd ? lane >> 2 : lane >> 1;
                if ((lane & (wd ? 3 : 1)) != 0) continue;
                int8_t* sd = wd ? a.sd32 : a.sd16;
                const int s_lo = int(short(pw & 0xFFFF)), s_hi = (pw - s_lo) >> 16;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int sum = e ? s_hi : s_lo, l = 2 * h + e;
                    const int lo = ((sum + 128) & 255) - 128;
                    sd[(b * 8 + l) * per + si] = int8_t(lo);
                    sd[(b * 8 + 4 + l) * per + si] = int8_t((sum - lo) >> 8);
                }
            }
        }
    }
    if (lane == 0) a.bscale[b] = pow2_neg(k);
}

// ---------------------------------------------------------------- the unit stream of one warp

// Matrices of the step in execution order: per layer qkv segments, wo, gate|up, down; then the head. Matrix `i` of
// layer `l` (l == n_layer, i == 0: the head). Every layer has the same shapes, so the way a matrix is shared between
// CTAs and warps depends only on its kind.
__device__ __forceinline__ int kind_li(const DkParams& p, int l, int i) { return l >= p.n_layer ? 6 : i < p.n_qkv ? i : 3 + i - p.n_qkv; }

// The CTA's share of a matrix as a range of units [cA, cB), cut into equal ranges for its warps [wA, wB).
// Whole tiles of the matrix's group by default (no tile is shared between CTAs: the phase ends without any exchange;
// a group with fewer tiles than CTAs occupies the first CTAs only); equal unit ranges for a balanced matrix.
struct WarpRange { int cA, cB, wA, wB; };
__host__ __device__ inline WarpRange cut_range(const DkKind& m, int c, int ctas, int warp, int warps) {
    WarpRange r;
    if (m.balanced) {
        const int U = m.tiles * m.upt;
        r.cA = range_lo(U, ctas, c);
        r.cB = range_lo(U, ctas, c + 1);
    } else {
        const int G = min(ctas, m.group_tiles);
        if (m.group_cost > 0) {  // CTA c takes the tiles whose cost position lies in [C c / G, C (c + 1) / G)
            auto bound = [&](int cc) {  // first tile of this matrix at or behind the cost position of boundary cc
                const long long rel = (long long)m.group_cost * cc / G - m.group_cost_off;
                return rel <= 0 ? 0 : int(min((rel + m.cost - 1) / m.cost, (long long)m.tiles));
            };
            r.cA = (c < G ? bound(c) : m.tiles) * m.upt;
            r.cB = (c < G ? bound(c + 1) : m.tiles) * m.upt;
        } else {
            const int gA = c < G ? range_lo(m.group_tiles, G, c) : 0, gB = c < G ? range_lo(m.group_tiles, G, c + 1) : 0;
            r.cA = min(max(gA - m.group_off, 0), m.tiles) * m.upt;
            r.cB = min(max(gB - m.group_off, 0), m.tiles) * m.upt;
        }
    }
    r.wA = r.cA + range_lo(r.cB - r.cA, warps, warp);
    r.wB = r.cA + range_lo(r.cB - r.cA, warps, warp + 1);
    return r;
}
static __device__ __noinline__ WarpRange warp_range(const DkKind& m, int warp, int warps = DK_WARPS) {
    return cut_range(m, int(blockIdx.x), int(gridDim.x), warp, warps);
}

// Most row tiles that the share of a CTA, and of one of its warps, touches. Taken from the cut itself: q, k and v are cut as
// one group and by cost, so that a CTA can hold many more tiles of a cheap format than its share by count.
struct CutExtent { int cta, warp; };
inline CutExtent cut_extent(const DkKind& m, int ctas, int warps) {
    CutExtent e{0, 1};
    auto touched = [&](int a, int b) { return a < b ? (b - 1) / m.upt - a / m.upt + 1 : 0; };
    for (int c = 0; c < ctas; ++c)
        for (int w = 0; w < warps; ++w) {
            const WarpRange r = cut_range(m, c, ctas, w, warps);
            if (w == 0) e.cta = max(e.cta, touched(r.cA, r.cB));
            e.warp = max(e.warp, touched(r.wA, r.wB));
        }
    return e;
}

// The shares of a warp (and of its CTA) in the matrices of every kind are computed once, when the kernel starts, and
// kept in shared memory: warp[kind] = {wA, wB} and tiles[kind] = {first row tile, last row tile} of this warp's share,
// cta[kind] = {cA, cB}.
struct Sched {
    const int2* warp;   // this warp's [DK_KINDS]
    const int2* tiles;  // all warps' [DK_WARPS][DK_KINDS]
    const int2* cta;    // [DK_KINDS]
};

// Prefetch cursor: the next unit of a warp's stream that has not been requested yet.
struct Cursor {
    int l, i, u, end, unit_bytes;  // matrix i of layer l (l > n_layer: the stream has ended)
    const uint8_t* W;
};
__device__ __forceinline__ bool cursor_live(const DkParams& p, const Cursor& c) { return c.l <= p.n_layer; }
__device__ __forceinline__ void cursor_next_matrix(const DkParams& p, Cursor& c) {
    if (c.l >= p.n_layer || ++c.i == p.n_qkv + 3) { c.i = 0; ++c.l; }
}
__device__ __forceinline__ void cursor_seek(const DkParams& p, Cursor& c, const int2* sched_warp) {  // first non-empty range from (l, i) on
    while (cursor_live(p, c)) {
        const int2 r = sched_warp[kind_li(p, c.l, c.i)];
        if (r.x < r.y) {
            c.u = r.x; c.end = r.y; c.W = p.W[c.l][c.i]; c.unit_bytes = unit_bytes_of(p.wtype[c.l][c.i]);
            return;
        }
        cursor_next_matrix(p, c);
    }
}

// The ring of one working warp: `bytes` bytes of shared memory that the units of the warp's stream pass through in
// order. A unit is requested with one bulk copy (global -> shared, completion counted in bytes on an mbarrier) by the
// producer warp (its lane w serves working warp w) and consumed by the working warp; its place is given up when the
// arithmetic on it is done. Units are placed back to back; one that would cross the end of the ring starts at offset 0
// instead and the bytes left over count as used until the consumer has passed them too (consumer and producer walk the
// same sequence of unit sizes, so both take the same decisions). Unit number q of the warp (counted from the start of
// the kernel) reports to mbarrier q % DK_NBAR, whose phase for it has parity (q / DK_NBAR) & 1; the ring is at most
// DK_NBAR of the smallest units long, so no more than DK_NBAR units are ever on request. The consumer tells the producer
// how far it has come through one word of shared memory: the number of bytes it has given up since the kernel started.
struct RingShared {       // in shared memory, one set for the CTA
    unsigned freed[DK_WARPS];    // bytes given up by working warp w so far (gaps included)
    unsigned issued[DK_WARPS];   // units requested for warp w in all, written when the producer ends
    int producer_done;
};
struct Ring {             // consumer side, in registers of the working warp
    uint32_t base;        // shared-memory addresses (32 bit) of the ring's first byte and of its first mbarrier
    uint32_t bars;
    int bytes;
    int c_off;            // offset of the next unit to consume (before the wrap rule is applied)
    unsigned c_seq;       // units given up so far
    unsigned freed;       // bytes given up so far
    uint32_t freed_out;   // where the producer reads it (shared-memory address)
};

__device__ __forceinline__ uint32_t dk_smem_u32(const void* p) { return uint32_t(__cvta_generic_to_shared(p)); }
__device__ __forceinline__ const uint8_t* dk_smem_ptr(uint32_t a) { return static_cast<const uint8_t*>(__cvta_shared_to_generic(size_t(a))); }

__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(bar), "r"(parity)
        : "memory");
    return done != 0;
}

// The producer warp: lane w < DK_WARPS walks the stream of working warp w and requests its units as room appears in that
// warp's ring. All lanes run in step, so the bookkeeping is paid once for the sixteen rings. Ends when every stream
// has been requested to its end, when the step is given up (dead flag), or when nothing has moved for too long.
static __device__ __noinline__ void producer_warp(const DkParams& p, const uint32_t ring0, const int ring_bytes, const uint32_t bars0,
                                           const int2* sched_all, RingShared* rs, const int* s_dead, const int lane) {
    const bool mine = lane < DK_WARPS;
    const int2* sched_warp = sched_all + (mine ? lane : 0) * DK_KINDS;
    Cursor c;
    c.l = 0;
    c.i = 0;
    c.u = c.end = c.unit_bytes = 0;
    c.W = nullptr;
    if (mine) cursor_seek(p, c, sched_warp);
    else c.l = p.n_layer + 1;
    const uint32_t base = ring0 + uint32_t(lane * ring_bytes), bars = bars0 + uint32_t(lane * DK_NBAR) * 8u;
    unsigned issued = 0, seq = 0, idle = 0;
    int off = 0;
    const volatile unsigned* freed = rs->freed + (mine ? lane : 0);
    while (true) {
        const bool live = cursor_live(p, c);
        if (!__any_sync(0xffffffffu, live)) break;
        bool did = false;
        if (live) {
            const int ub = c.unit_bytes;
            const bool wrap = off + ub > ring_bytes;
            const int need = wrap ? ring_bytes - off + ub : ub;
            if (int(issued - *freed) + need <= ring_bytes) {
                if (wrap) off = 0;
                const uint32_t bar = bars + (seq % DK_NBAR) * 8u;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(ub) : "memory");
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                             ::"r"(base + uint32_t(off)), "l"(c.W + size_t(c.u) * ub), "r"(ub), "r"(bar)
                             : "memory");
                issued += unsigned(need);
                off += ub;
                ++seq;
                did = true;
                if (++c.u == c.end) {
                    cursor_next_matrix(p, c);
                    cursor_seek(p, c, sched_warp);
                }
            }
        }
        if (__any_sync(0xffffffffu, did)) {
            idle = 0;
        } else {
            if (*reinterpret_cast<const volatile int*>(s_dead) || ++idle > DK_SPIN_LIMIT) break;
            __nanosleep(DK_PRODUCER_NAP);
        }
    }
    if (mine) rs->issued[lane] = seq;
    __syncwarp();
    if (lane == 0) {
        __threadfence_block();
        *reinterpret_cast<volatile int*>(&rs->producer_done) = 1;
    }
}

// Wait (bounded) until the oldest requested unit, of `ub` bytes, has arrived; returns where it lies. On timeout the
// dead flag and the error word are raised and the caller goes on with whatever the ring holds: the next grid barrier
// ends the step.
__device__ __forceinline__ uint32_t ring_front(const DkParams& p, Ring& r, int ub, int* s_dead) {
    if (r.c_off + ub > r.bytes) {  // the producer skipped the end of the ring for this unit
        r.freed += unsigned(r.bytes - r.c_off);
        r.c_off = 0;
    }
    const uint32_t bar = r.bars + (r.c_seq % DK_NBAR) * 8u, parity = (r.c_seq / DK_NBAR) & 1u;
    bool done = false;
#pragma unroll 1
    for (unsigned it = 0; it < DK_MBAR_LIMIT && !done; ++it) {
        done = mbar_try(bar, parity);
        if ((it & 255u) == 255u && *reinterpret_cast<const volatile int*>(s_dead)) break;
    }
    if (!done && !*s_dead) {
        *s_dead = 1;
        atomicExch(p.err, 1);
    }
    return r.base + uint32_t(r.c_off);
}
// The unit at the front has been used up by every lane (the caller has synchronised the warp): its bytes are free again.
__device__ __forceinline__ void ring_pop(Ring& r, int ub, int lane) {
    r.c_off += ub;
    r.freed += unsigned(ub);
    ++r.c_seq;
    if (lane == 0) asm volatile("st.release.cta.shared::cta.u32 [%0], %1;" ::"r"(r.freed_out), "r"(r.freed) : "memory");
}
// Before the kernel ends: the producer must have stopped and every copy it requested must have landed (bounded waits).
static __device__ __noinline__ void ring_drain(Ring& r, const RingShared* rs, int warp) {
    unsigned it = 0;
    while (!*reinterpret_cast<const volatile int*>(&rs->producer_done) && ++it < DK_SPIN_LIMIT) __nanosleep(100);
    const unsigned end = *reinterpret_cast<const volatile unsigned*>(&rs->issued[warp]);
    for (; r.c_seq != end; ++r.c_seq) {
        const uint32_t bar = r.bars + (r.c_seq % DK_NBAR) * 8u, parity = (r.c_seq / DK_NBAR) & 1u;
        bool done = false;
        for (unsigned j = 0; j < DK_MBAR_LIMIT && !done; ++j) done = mbar_try(bar, parity);
    }
}

// RMSNorm over one 128-wide head followed by NEOX RoPE (src/ops.cpp:155-160, src/model.cpp:23-32 of the reference);
// one warp per head, lane owns elements lane, lane+32, lane+64, lane+96.
__device__ __forceinline__ void dk_head_norm_rope(const float* src, const float* w, const float2* cs, int rope_dim, float eps,
                                                  float* dst, int lane) {
    float v[4], wn[4];
    float2 c[2];  // cos / sin of this lane's rotation pairs: asked for together with the head, used last
    const int half = rope_dim / 2;
#pragma unroll
    for (int j = 0; j < 2; ++j) c[j] = lane + 32 * j < half ? __ldg(cs + lane + 32 * j) : make_float2(1.f, 0.f);
    double ss = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        v[j] = __ldcg(src + lane + 32 * j);
        wn[j] = __ldg(w + lane + 32 * j);
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) ss += double(v[j]) * v[j];
    ss = warp_sum(ss);
    const float inv = float(rsqrt_d(ss / DK_HD + double(eps)));
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[lane + 32 * j] = __fmul_rn(__fmul_rn(v[j], inv), wn[j]);
    __syncwarp();
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = lane + 32 * j;
        if (i < half) {
            const float a = dst[i], b = dst[i + half];
            dst[i] = __fsub_rn(__fmul_rn(a, c[j].x), __fmul_rn(b, c[j].y));
            dst[i + half] = __fadd_rn(__fmul_rn(a, c[j].y), __fmul_rn(b, c[j].x));
        }
    }
    __syncwarp();
}

}  // namespace elb
