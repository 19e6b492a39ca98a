// One decode step (one token, batch 1) on one GPU as ONE persistent kernel without grid barriers.
//
// At batch 1 every layer is a chain of five dependent steps (q|k|v, attention, output projection, gate|up, down), each a
// few microseconds of HBM traffic: what bounds the step is the latency of handing a vector of a few thousand values from
// every SM to every SM, five times per layer. Here one CTA per SM stays resident for the whole step and
//   * a value travels with the number of the layer pass it belongs to, in ONE 8-byte word written by one store: a consumer
//     loads its words and asks again for those that do not carry the number it waits for. There is no barrier, no fence and
//     no counter between a producer's store and a consumer's load, a word of another layer or step is never taken for this
//     one's, whatever the order in which stores arrive, and a block of the activation is converted as soon as its own words
//     are there. One buffer per vector is enough: whoever reads exchange s of layer n afterwards writes something that,
//     going from exchange to exchange, every writer of exchange s of layer n + 1 has waited for (a CTA reads nothing in a
//     stage in which it has no share, except the rows of the residual stream that its next share adds to). With the grid
//     barriers of decode.cu (release, poll, then load: 2.5 us from the last store to the first use, against about 1 us) the
//     4B-shape layer took 48.7 us, here 34.7 us. (Partial sums in 16-byte words of three values and the number, a quarter
//     fewer bytes: a step 2 % slower on the 0.6B and 1.7B shapes, 1 % faster on the 4B and 32B shapes. All vectors so: 5 %
//     slower on the 0.6B and 4B shapes; two producers then share a 32-byte sector of the feed-forward vector.);
//   * every working warp owns a fixed, contiguous share of the (row tile, k block) units of every weight matrix of the
//     step, in execution order, and a producer warp keeps every working warp's ring in shared memory as full as it gets,
//     no matter what the CTA is doing: HBM streams through exchanges, attention and conversion;
//   * the activation of a matvec is converted redundantly by every CTA: to int8 limbs in shared memory (quantized
//     weights, split block by block) or to an fp32 vector there (F16 weights); the residual stream is added up
//     redundantly too, so nothing but partial sums crosses between CTAs, in a fixed order: deterministic;
//   * q, k, v and gate|up are cut in whole row tiles; attn_output and ffn_down, with few row tiles and long rows, in equal
//     unit ranges: a row tile then has at most two contributing CTAs, whose sums the next conversion adds;
//   * an ffn_down activation too long for shared memory (25 600 values of the 32B shape: 121 KB of limbs) is worked
//     off in down_parts equal ranges of k: convert one, multiply it, convert the next.
// All waits are bounded: on timeout the kernel raises an error word, drains its copies and leaves.
#include <cuda.h>

#include <algorithm>
#include <cstring>

#include "decode_parts.cuh"
#include "attn_core.cuh"
#include "layout.cuh"

namespace elb {

namespace {

// 15 working warps and the producer: 16 warps can have 128 registers a thread, which the attention's rows in flight need
// (with 16 working warps the seventeenth warp would leave 96).
constexpr int D1_WARPS = 15, D1_WORKERS = 32 * D1_WARPS, D1_THREADS = D1_WORKERS + 32;
static_assert(D1_WARPS <= DK_WARPS, "the ring bookkeeping has one place per warp");
__device__ __forceinline__ void d1_sync() { asm volatile("bar.sync 1, %0;" ::"n"(D1_WORKERS) : "memory"); }
constexpr unsigned D1_POLL_LIMIT = 1u << 20;    // loads of one wait for an exchange word: about a second
constexpr int D1_SPLIT_KEYS = 4 * D1_WARPS;     // keys of one attention split: one tile of 4 keys per warp
constexpr int D1_F16_UNIT = 16 * 128 * 2;       // F16: 16 rows x 128 k

__device__ __forceinline__ int d1_unit_bytes(int type) { return type == ELB_F16 ? D1_F16_UNIT : unit_bytes_of(type); }

// barrier of the working warps that also agrees on whether a wait has run out anywhere in the CTA
__device__ __forceinline__ bool d1_sync_dead(const int* dead) {
    int out;
    asm volatile(
        "{\n .reg .pred p, q;\n setp.ne.s32 p, %1, 0;\n bar.red.or.pred q, 1, %2, p;\n selp.s32 %0, 1, 0, q;\n}\n"
        : "=r"(out)
        : "r"(*reinterpret_cast<const volatile int*>(dead)), "n"(D1_WORKERS)
        : "memory");
    return out != 0;
}

// ---------------------------------------------------------------- exchange words

// A word is one memory location: loads and stores are relaxed, at GPU scope, 64 bits each.
__device__ __forceinline__ DkEx ex_word(unsigned long long w) { return DkEx{__uint_as_float(unsigned(w)), unsigned(w >> 32)}; }
__device__ __forceinline__ DkEx ex_ld(const DkEx* p) {
    unsigned long long a;
    asm volatile("ld.relaxed.gpu.global.b64 %0, [%1];" : "=l"(a) : "l"(p) : "memory");
    return ex_word(a);
}
__device__ __forceinline__ void ex_ld2(const DkEx* p, DkEx& x, DkEx& y) {  // two words (p: 16-byte aligned)
    unsigned long long a, b;
    asm volatile("ld.relaxed.gpu.global.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "l"(p) : "memory");
    x = ex_word(a);
    y = ex_word(b);
}
__device__ __forceinline__ void ex_st(DkEx* p, float v, unsigned num) {
    asm volatile("st.relaxed.gpu.global.b64 [%0], %1;" ::"l"(p), "l"((unsigned long long)num << 32 | __float_as_uint(v)) : "memory");
}
struct Ex8 {  // eight consecutive words (64-byte aligned)
    unsigned long long w[8];
    __device__ __forceinline__ void load(const DkEx* p) {
#pragma unroll
        for (int j = 0; j < 8; j += 4)
            asm volatile("ld.relaxed.gpu.global.v4.b64 {%0, %1, %2, %3}, [%4];"
                         : "=l"(w[j]), "=l"(w[j + 1]), "=l"(w[j + 2]), "=l"(w[j + 3]) : "l"(p + j) : "memory");
    }
    __device__ __forceinline__ bool missing(unsigned num) const {
        bool m = false;
#pragma unroll
        for (int j = 0; j < 8; ++j) m = m || unsigned(w[j] >> 32) != num;
        return m;
    }
    __device__ __forceinline__ float4 get(int j) const { return make_float4(ex_word(w[j]).v, ex_word(w[j + 1]).v, ex_word(w[j + 2]).v, ex_word(w[j + 3]).v); }
};
struct Wait {  // of one place where a thread waits for words; false: give up (a wait has run out here or elsewhere in the CTA)
    unsigned it = 0;
    __device__ __forceinline__ bool again(const DkParams& p, int* dead) {
        if ((++it & 63u) == 0u) {
            if (*reinterpret_cast<volatile int*>(dead)) return false;
            if (it > D1_POLL_LIMIT) {
                *dead = 1;
                atomicExch(p.err, 1);
                return false;
            }
        }
        return true;
    }
};

__device__ __forceinline__ void d1_stamp(const DkParams& p, int l, int ev) {
    if (p.prof && blockIdx.x == 0 && threadIdx.x == 0) {
        unsigned long long t;
        asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
        p.prof[l * 32 + ev] = t;
    }
}

// ---------------------------------------------------------------- shares and unit stream

// Kinds of matrices: 0..2 q|k|v segments, then attn_output, gate|up, head, and the parts of ffn_down along k.
enum { K1_WO = 3, K1_GU = 4, K1_HEAD = 5, K1_DOWN = 6, K1_KINDS = K1_DOWN + DK_MAX_PARTS };
static_assert(K1_KINDS == DK_ONE_KINDS, "tables of the parameter block");

__host__ __device__ __forceinline__ const DkKind& d1_whole(const DkParams& p, int kind) { return kind < K1_HEAD ? p.kind[kind] : kind == K1_HEAD ? p.kind[6] : p.kind[5]; }
// Matrices of a layer in execution order: q|k|v segments, attn_output, gate|up, the parts of ffn_down; layer n_layer: the head.
__device__ __forceinline__ int d1_kind_of(const DkParams& p, int l, int i) {
    if (l >= p.n_layer) return K1_HEAD;
    return i < p.n_qkv ? i : i < p.n_qkv + 2 ? K1_WO + i - p.n_qkv : K1_DOWN + i - p.n_qkv - 2;
}
__device__ __forceinline__ int d1_weight_of(const DkParams& p, int i) { return min(i, p.n_qkv + 2); }  // index into W / wtype

// Tables in shared memory, computed once when the kernel starts. Of a warp's share of a kind: {units, k block of the
// first unit within its row tile, first row tile}; of the CTA's: {first row tile, row tiles, holds the first tile's first
// unit, holds the last tile's last unit}; of every row tile of the CTA: the warps that have units of it, lo | hi << 8, and
// which of warp lo's row tiles it is, << 16 (of the warps behind lo it is the first).
struct Share { int units, b0, tile, pad; };
struct CtaShare { int tile, tiles, first, last; };

// F16 units are tiles of a row-major matrix: one tensor copy each (16 bulk copies of a row's 256 bytes kept the producer
// warp busy for longer than HBM needed: 47 us per layer of the 0.6B shape, 31 MB). Maps in execution order, in global memory.
__device__ __forceinline__ void d1_tensor_copy(uint32_t dst, const void* map, int k, int row, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(k), "r"(row), "r"(bar)
                 : "memory");
}

// Prefetch cursor: the next unit of a warp's stream that has not been requested yet.
struct Cursor1 {
    int l, i, left, b, upt, ub, skip, tile;  // left: units of this range; b: k block within the row tile's part
    int k0;                                  // F16: k block at which the part starts (quantized: src is there already)
    const uint8_t* src;                      // the unit (F16: the matrix's tensor map)
};
__device__ __forceinline__ void d1_seek(const DkParams& p, Cursor1& c, const Share* shares) {  // first non-empty range from (l, i) on
    while (c.l <= p.n_layer) {
        const int kind = d1_kind_of(p, c.l, c.i);
        const Share sh = shares[kind];
        if (sh.units > 0) {
            const int wi = d1_weight_of(p, c.i), type = p.wtype[c.l][wi];
            const DkKind& full = d1_whole(p, kind);
            c.upt = p.upt1[kind];
            c.left = sh.units;
            c.b = sh.b0;
            c.ub = d1_unit_bytes(type);
            const uint8_t* W = p.W[c.l][wi];
            c.tile = sh.tile;
            const int part0 = kind >= K1_DOWN ? (kind - K1_DOWN) * c.upt : 0;  // first unit of the part within a row tile
            if (type == ELB_F16) {
                c.k0 = part0;
                c.src = p.f16_maps + size_t(c.l * DK_LAYER_MATS + wi) * 128;
            } else {
                c.skip = (full.upt - c.upt) * c.ub;
                c.src = W + (size_t(sh.tile) * full.upt + part0 + c.b) * c.ub;
            }
            return;
        }
        if (c.l >= p.n_layer || ++c.i == p.n_qkv + 2 + p.down_parts) { c.i = 0; ++c.l; }
    }
}

// The producer warp: lane w walks the stream of working warp w and requests its units as room appears in that warp's ring.
template <bool F16M>
__device__ __noinline__ void d1_producer(const DkParams& p, const uint32_t ring0, const int ring_bytes, const uint32_t bars0,
                                         const Share* shares, RingShared* rs, const int* s_dead, const int lane) {
    const bool mine = lane < D1_WARPS;
    shares += (mine ? lane : 0) * K1_KINDS;
    Cursor1 c{};
    if (mine) d1_seek(p, c, shares);
    else c.l = p.n_layer + 1;
    const uint32_t base = ring0 + uint32_t(lane * ring_bytes), bars = bars0 + uint32_t(lane * DK_NBAR) * 8u;
    unsigned issued = 0, seq = 0, idle = 0;
    int off = 0;
    const volatile unsigned* freed = rs->freed + (mine ? lane : 0);
    while (true) {
        const bool live = c.l <= p.n_layer;
        if (!__any_sync(0xffffffffu, live)) break;
        bool did = false;
        if (live) {
            const int ub = c.ub;
            const bool wrap = off + ub > ring_bytes;
            const int need = wrap ? ring_bytes - off + ub : ub;
            if (int(issued - *freed) + need <= ring_bytes) {
                if (wrap) off = 0;
                const uint32_t bar = bars + (seq % DK_NBAR) * 8u, dst = base + uint32_t(off);
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(ub) : "memory");
                if (F16M) {
                    d1_tensor_copy(dst, c.src, (c.k0 + c.b) * 128, c.tile * 16, bar);
                } else {
                    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                                 ::"r"(dst), "l"(c.src), "r"(ub), "r"(bar)
                                 : "memory");
                }
                issued += unsigned(need);
                off += ub;
                ++seq;
                did = true;
                if (!F16M) c.src += ub;
                if (++c.b == c.upt) {
                    c.b = 0;
                    if (F16M) ++c.tile;
                    else c.src += c.skip;
                }
                if (--c.left == 0) {
                    if (c.l >= p.n_layer || ++c.i == p.n_qkv + 2 + p.down_parts) { c.i = 0; ++c.l; }
                    d1_seek(p, c, shares);
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

// ---------------------------------------------------------------- activation of a matvec

// What a conversion has to hand on of the residual stream
struct Rows {
    float* keep;  // shared memory: rows [r0, r1), which this CTA's next row-parallel matvec adds to
    int r0, r1;
    float* out;   // global: this CTA's slice of the whole stream (the last one: p.x), or null
};

// Blocks [blk0, blk0 + nblk) of the exchanged vector A (NORM: of A + B, the two buffers of partial sums a row-parallel
// matvec left, the first of which carries the old residual stream; B null: A alone) -> blocks 0.. of the activation:
// limbs, or fp32 values (F16M). NORM multiplies by norm_w; the factor 1 / sqrt(mean(x^2) + eps) of the RMSNorm
// (src/ops.cpp:155-160 of the reference, sum of squares in double) is applied to the row sums of the matvec, and every
// warp leaves its share of the sum of squares in red8: no block waits for the sum over the vector. Warp w takes blocks
// w, w + 15, ...; the words of the next block (plain: of the two next) are asked for before the current one is converted,
// into the registers of the words just used (a loop, not unrolled: the code of a conversion runs once or twice per stage, as
// fast as it can be fetched).
template <bool NORM, bool F16M>
__device__ __forceinline__ void d1_convert(const DkParams& p, const DkEx* A, const DkEx* B, const unsigned num, const float* norm_w,
                                           const int blk0, const int nblk, const int nl, const ActSmem& a, const int sd_mask, double* red8,
                                           const Rows& rows, int* dead) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    A += blk0 * 256 + lane * 8;
    if (NORM) { norm_w += lane * 8; if (B) B += lane * 8; }
    double ss = 0.0;
    Ex8 va{}, vb{};   // the current block's words (plain: vb, the next block's)
    if (warp < nblk) {
        va.load(A + warp * 256);
        if (NORM && B) vb.load(B + warp * 256);
    }
    if (!NORM && warp + D1_WARPS < nblk) vb.load(A + (warp + D1_WARPS) * 256);
#pragma unroll 1
    for (int b = warp; b < nblk; b += D1_WARPS) {
        const int at = b * 256;
        float4 n0, n1;
        if (NORM) { n0 = __ldg(reinterpret_cast<const float4*>(norm_w + at)); n1 = __ldg(reinterpret_cast<const float4*>(norm_w + at + 4)); }
        Wait wait;
        while (__any_sync(0xffffffffu, va.missing(num) || (NORM && B && vb.missing(num)))) {
            va.load(A + b * 256);
            if (NORM && B) vb.load(B + b * 256);
            if (__any_sync(0xffffffffu, !wait.again(p, dead))) break;
        }
        float4 v0 = va.get(0), v1 = va.get(4);
        const int next = b + D1_WARPS;
        if (NORM) {
            if (B) {
                const float4 w0 = vb.get(0), w1 = vb.get(4);
                v0 = make_float4(__fadd_rn(v0.x, w0.x), __fadd_rn(v0.y, w0.y), __fadd_rn(v0.z, w0.z), __fadd_rn(v0.w, w0.w));
                v1 = make_float4(__fadd_rn(v1.x, w1.x), __fadd_rn(v1.y, w1.y), __fadd_rn(v1.z, w1.z), __fadd_rn(v1.w, w1.w));
            }
            if (next < nblk) {
                va.load(A + next * 256);
                if (B) vb.load(B + next * 256);
            }
            ss += double(v0.x) * v0.x + double(v0.y) * v0.y + double(v0.z) * v0.z + double(v0.w) * v0.w;
            ss += double(v1.x) * v1.x + double(v1.y) * v1.y + double(v1.z) * v1.z + double(v1.w) * v1.w;
            const int i = at + lane * 8;
            if (i >= rows.r0 && i < rows.r1) {
                *reinterpret_cast<float4*>(rows.keep + i - rows.r0) = v0;
                *reinterpret_cast<float4*>(rows.keep + i - rows.r0 + 4) = v1;
            }
            if (rows.out && b == int(blockIdx.x)) {  // (there are at least as many CTAs as blocks)
                *reinterpret_cast<float4*>(rows.out + i) = v0;
                *reinterpret_cast<float4*>(rows.out + i + 4) = v1;
            }
            v0 = make_float4(__fmul_rn(v0.x, n0.x), __fmul_rn(v0.y, n0.y), __fmul_rn(v0.z, n0.z), __fmul_rn(v0.w, n0.w));
            v1 = make_float4(__fmul_rn(v1.x, n1.x), __fmul_rn(v1.y, n1.y), __fmul_rn(v1.z, n1.z), __fmul_rn(v1.w, n1.w));
        } else {
            va = vb;
            if (next + D1_WARPS < nblk) vb.load(A + (next + D1_WARPS) * 256);
        }
        if (F16M) {
            float* dst = reinterpret_cast<float*>(a.lim) + at + lane * 8;
            *reinterpret_cast<float4*>(dst) = v0;
            *reinterpret_cast<float4*>(dst + 4) = v1;
        } else {
            split_block(v0, v1, b, nl, a, sd_mask, lane);
        }
    }
    if (NORM) {
        ss = warp_sum(ss);
        if (lane == 0) red8[warp] = ss;
    }
}

// A CTA without a share in the matrices of a stage still needs its rows of the residual stream, and CTA b block b of the
// last one.
__device__ __noinline__ void d1_keep_rows(const DkParams& p, const DkEx* A, const DkEx* B, const unsigned num, const Rows rows, int* dead) {
    auto get = [&](int i, float* dst) {
        Ex8 a, b{};
        a.load(A + i);
        if (B) b.load(B + i);
        Wait wait;
        while ((a.missing(num) || (B && b.missing(num))) && wait.again(p, dead)) {
            a.load(A + i);
            if (B) b.load(B + i);
        }
        float4 v0 = a.get(0), v1 = a.get(4);
        if (B) {
            const float4 w0 = b.get(0), w1 = b.get(4);
            v0 = make_float4(__fadd_rn(v0.x, w0.x), __fadd_rn(v0.y, w0.y), __fadd_rn(v0.z, w0.z), __fadd_rn(v0.w, w0.w));
            v1 = make_float4(__fadd_rn(v1.x, w1.x), __fadd_rn(v1.y, w1.y), __fadd_rn(v1.z, w1.z), __fadd_rn(v1.w, w1.w));
        }
        *reinterpret_cast<float4*>(dst) = v0;
        *reinterpret_cast<float4*>(dst + 4) = v1;
    };
#pragma unroll 1
    for (int i = rows.r0 + int(threadIdx.x) * 8; i < rows.r1; i += D1_WORKERS * 8) get(i, rows.keep + i - rows.r0);
    const int o = blockIdx.x * 256 + int(threadIdx.x) * 8;
    if (rows.out && threadIdx.x < 32 && o < p.E) get(o, rows.out + o);
}

// ---------------------------------------------------------------- matvec

struct Smem1 {
    const Share* shares;    // this warp's [K1_KINDS]
    const CtaShare* cta;    // [K1_KINDS]
    const int* who;         // [row tiles of all kinds, p.tile_base] which warps have units of a row tile
    float* red;    // [D1_WARPS][slots][16] row sums of each warp's share, per row tile it touches
    double* red8;  // [D1_WARPS]
    float* xrow;   // [2][row tiles of a share * 16]
    int* flags;    // [2]: a wait has run out; [3]: the step's position
};

template <int TYPE>
__device__ __forceinline__ void d1_units(const DkParams& p, const int upt, const Share sh, Ring& rg, const ActSmem& act, float* red, int* dead,
                                         int lane) {
    const int g = lane >> 2, t = lane & 3;
    constexpr int UB = TYPE == ELB_Q4_K ? Q4K_UNIT : TYPE == ELB_Q6_K ? Q6K_UNIT : Q8_UNIT;
    const int8_t* sd = TYPE == ELB_Q6_K ? act.sd16 : act.sd32;
    Acc a{{0.f, 0.f}, {0.f, 0.f}};
    int b = sh.b0;
    const float wt = t < 2 ? (t & 1 ? 65536.0f : 1.0f) : 0.0f;
    const float wtm = (t & 1 ? 65536.0f : 1.0f) * (t & 2 ? 256.0f : 1.0f);
    DbgOut dbg{nullptr, nullptr, nullptr, 0, 0, 0, 0};
#pragma unroll 1
    for (int left = sh.units; left > 0; --left) {
        Unit<TYPE> cur;
        load_unit(cur, dk_smem_ptr(ring_front(p, rg, UB, dead)), lane);
        compute_unit<false, false>(cur, b, act.lim, act.n_pad, sd, lane, a, dbg, act.bscale);
        __syncwarp();  // every lane has its fragments of the unit in registers and has used them
        ring_pop(rg, UB, lane);
        if (++b == upt || left == 1) {
            float v0 = a.acc[0] * wt - a.accm[0] * wtm, v1 = a.acc[1] * wt - a.accm[1] * wtm;
            v0 += __shfl_xor_sync(0xffffffffu, v0, 1);
            v1 += __shfl_xor_sync(0xffffffffu, v1, 1);
            v0 += __shfl_xor_sync(0xffffffffu, v0, 2);
            v1 += __shfl_xor_sync(0xffffffffu, v1, 2);
            if (t == 0) { red[g] = v0; red[g + 8] = v1; }
            red += 16;
            a = Acc{{0.f, 0.f}, {0.f, 0.f}};
            b = 0;
        }
    }
}

// F16 weights, fp32 multiply-adds: half a warp per row (rows r and r + 8), lane = 8 values of the unit's 128 k
__device__ __forceinline__ void d1_units_f16(const DkParams& p, const int upt, const Share sh, Ring& rg, const ActSmem& as, float* red, int* dead,
                                             int lane) {
    const int c = lane & 15, half = lane >> 4;
    const float* act = reinterpret_cast<const float*>(as.lim) + 8 * c;
    float acc[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) acc[r] = 0.f;
    int b = sh.b0;
#pragma unroll 1
    for (int left = sh.units; left > 0; --left) {
        const uint8_t* src = dk_smem_ptr(ring_front(p, rg, D1_F16_UNIT, dead)) + half * 2048 + c * 16;
        const float4 x0 = *reinterpret_cast<const float4*>(act + b * 128), x1 = *reinterpret_cast<const float4*>(act + b * 128 + 4);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const uint4 q = lds4(src + r * 256);
            const float2 f0 = __half22float2(*reinterpret_cast<const __half2*>(&q.x)), f1 = __half22float2(*reinterpret_cast<const __half2*>(&q.y));
            const float2 f2 = __half22float2(*reinterpret_cast<const __half2*>(&q.z)), f3 = __half22float2(*reinterpret_cast<const __half2*>(&q.w));
            float v = acc[r];
            v = fmaf(f0.x, x0.x, v); v = fmaf(f0.y, x0.y, v); v = fmaf(f1.x, x0.z, v); v = fmaf(f1.y, x0.w, v);
            v = fmaf(f2.x, x1.x, v); v = fmaf(f2.y, x1.y, v); v = fmaf(f3.x, x1.z, v); v = fmaf(f3.y, x1.w, v);
            acc[r] = v;
        }
        __syncwarp();
        ring_pop(rg, D1_F16_UNIT, lane);
        if (++b == upt || left == 1) {
            // the 16 lanes of a half hold 8 row sums in parts: a transposing butterfly leaves row (c >> 1) on lanes c and c ^ 1
            float v4[4], v2[2];
#pragma unroll
            for (int r = 0; r < 4; ++r) v4[r] = (c & 8 ? acc[r + 4] : acc[r]) + __shfl_xor_sync(0xffffffffu, c & 8 ? acc[r] : acc[r + 4], 8);
#pragma unroll
            for (int r = 0; r < 2; ++r) v2[r] = (c & 4 ? v4[r + 2] : v4[r]) + __shfl_xor_sync(0xffffffffu, c & 4 ? v4[r] : v4[r + 2], 4);
            float v = (c & 2 ? v2[1] : v2[0]) + __shfl_xor_sync(0xffffffffu, c & 2 ? v2[0] : v2[1], 2);
            v += __shfl_xor_sync(0xffffffffu, v, 1);
            if ((c & 1) == 0) red[half * 8 + (c >> 1)] = v;
            red += 16;
#pragma unroll
            for (int r = 0; r < 8; ++r) acc[r] = 0.f;
            b = 0;
        }
    }
}

template <bool F16M>
__device__ __forceinline__ void d1_matvec(const DkParams& p, const int type, const int kind, Ring& rg, const ActSmem& act, const Smem1& s) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, upt = p.upt1[kind];
    const Share sh = s.shares[kind];
    float* const red = s.red + (warp * p.slots + p.slot_base[kind]) * 16;
    int* const dead = &s.flags[2];
    if (sh.units == 0 && lane < 16) red[lane] = 0.f;  // (it may lie between two warps with units of one row tile)
    if (F16M) {
        d1_units_f16(p, upt, sh, rg, act, red, dead, lane);
    } else {
        switch (type) {
            case ELB_Q4_K: d1_units<ELB_Q4_K>(p, upt, sh, rg, act, red, dead, lane); break;
            case ELB_Q6_K: d1_units<ELB_Q6_K>(p, upt, sh, rg, act, red, dead, lane); break;
            default: d1_units<ELB_Q8_0>(p, upt, sh, rg, act, red, dead, lane); break;
        }
    }
}

// Row sums of the CTA's share of `kind` (and of parts - 1 kinds behind it: parts along k of the same rows) and what
// becomes of them, by stage:
//   0 q|k|v    -> exchange                        1, 3 attn_output, ffn_down: the CTA that holds a tile's first unit adds
//   2 gate|up  -> silu(gate) * up -> exchange       the residual stream and writes vector 0, the one that holds its last
//   4 head     -> logits                            unit vector 1 (a CTA that holds the whole tile: zeros)
__device__ __forceinline__ void d1_epilogue(const DkParams& p, const int stage, const int kind, const int parts, const int seg, const unsigned num,
                                            const float inv, const Smem1& s, const float* xrow) {
    const int lane = threadIdx.x & 31;
    const CtaShare cs = s.cta[kind];
    const int rows = d1_whole(p, kind).rows, total = cs.tiles * 16;
#pragma unroll 1
    for (int e0 = threadIdx.x & ~31; e0 < total; e0 += D1_WORKERS) {
        const int e = e0 + lane, lt = e >> 4, row = e & 15;
        const bool on = e < total;
        float v = 0.f;
        if (on) {
#pragma unroll 1
            for (int part = 0; part < parts; ++part) {  // fixed order: parts, then warps
                const int who = s.who[p.tile_base[kind + part] + lt], lo = who & 255, hi = (who >> 8) & 255;
                const float* r = s.red + p.slot_base[kind + part] * 16 + row;
                v += r[(lo * p.slots + (who >> 16)) * 16];
#pragma unroll 4
                for (int w = lo + 1; w <= hi; ++w) v += r[w * p.slots * 16];
            }
        }
        v *= inv;
        const int R = 16 * cs.tile + e;
        if (stage == 2) {  // rows 0..7 of a tile gate, 8..15 up (SwiGLU, src/model.cpp:222-225 of the reference)
            const float up = __shfl_down_sync(0xffffffffu, v, 8);
            if (on && row < 8) ex_st(p.ex_g + 8 * (cs.tile + lt) + row, __fmul_rn(__fdiv_rn(v, 1.0f + expf(-v)), up), num);
        } else if (on && R < rows) {
            if (stage == 0) {
                ex_st(p.ex_q + p.qkv_col[seg] + R, v, num);
            } else if (stage == 4) {
                p.logits_peer[0][R] = v;
            } else {
                DkEx* buf = stage == 1 ? p.ex_p1 : p.ex_p2;
                const bool first = lt > 0 || cs.first, last = lt + 1 < cs.tiles || cs.last;
                if (first) v = __fadd_rn(xrow[e], v);
                if (first && last) ex_st(buf + p.E + R, 0.f, num);
                ex_st(buf + (first ? 0 : p.E) + R, v, num);
            }
        }
    }
}

// ---------------------------------------------------------------- attention

// RMSNorm over one 128-wide head followed by NEOX RoPE (src/ops.cpp:155-160, src/model.cpp:23-32 of the reference), as
// dk_head_norm_rope, from exchange words; one warp per head, lane owns elements lane, lane+32, lane+64, lane+96.
__device__ __forceinline__ void d1_head(const DkParams& p, const DkEx* src, const unsigned num, const float* w, const float2* cs, float* dst, int lane, int* dead) {
    const int half = p.rope_dim / 2;
    DkEx x[4];
    float wn[4];
    float2 c[2];
#pragma unroll
    for (int j = 0; j < 4; ++j) x[j] = ex_ld(src + lane + 32 * j);
#pragma unroll
    for (int j = 0; j < 4; ++j) wn[j] = __ldg(w + lane + 32 * j);
#pragma unroll
    for (int j = 0; j < 2; ++j) c[j] = lane + 32 * j < half ? __ldg(cs + lane + 32 * j) : make_float2(1.f, 0.f);
    Wait wait;
    while (__any_sync(0xffffffffu, x[0].num != num || x[1].num != num || x[2].num != num || x[3].num != num)) {
#pragma unroll
        for (int j = 0; j < 4; ++j) x[j] = ex_ld(src + lane + 32 * j);
        if (__any_sync(0xffffffffu, !wait.again(p, dead))) break;
    }
    double ss = 0.0;
#pragma unroll
    for (int j = 0; j < 4; ++j) ss += double(x[j].v) * x[j].v;
    ss = warp_sum(ss);
    const float inv = float(rsqrt_d(ss * (1.0 / DK_HD) + double(p.eps)));
#pragma unroll
    for (int j = 0; j < 4; ++j) dst[lane + 32 * j] = __fmul_rn(__fmul_rn(x[j].v, inv), wn[j]);
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
}

// CTA c < HKV * splits works on KV head c / splits, key split c % splits: the first keys and values are asked for, then
// q/k norm + RoPE, KV append, attention over its keys (attn_core.cuh). Several splits leave their partial results in an
// exchange buffer, each adds a slice of the outputs in split order and writes it to att. Semantics: src/model.cpp:176-214 of the
// reference.
template <int GP>
__device__ __forceinline__ void d1_attention(const DkParams& p, const int l, const unsigned num, float* scratch, const int* s_pos, int* dead) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, c = blockIdx.x;
    // (read here, and not kept from layer to layer: what follows from it would take registers from the matvecs)
    const int pos = *reinterpret_cast<const volatile int*>(s_pos), T = pos + 1, ns = max(1, min(p.nsplit, (T + D1_SPLIT_KEYS - 1) / D1_SPLIT_KEYS));
    if (c >= p.HKV * ns) return;
    const int kvh = c / ns, split = c - kvh * ns, group = p.H / p.HKV, QD = p.H * DK_HD, KD = p.HKV * DK_HD;
    float* const qs = scratch;               // [DK_MAXG][128]
    float* const knew = qs + DK_MAXG * DK_HD;  // [128]
    float* const vnew = knew + DK_HD;          // [128]
    const AcSmem as = ac_smem(vnew + DK_HD, qs, GP, D1_WARPS);
    float* const kc = p.kc + size_t(l) * p.kv_stride + kvh * DK_HD;
    float* const vc = p.vc + size_t(l) * p.kv_stride + kvh * DK_HD;
    const int t0 = range_lo(T, ns, split), t1 = range_lo(T, ns, split + 1);  // equal key ranges
    const float* const q_norm = p.norms + size_t(l) * p.norm_stride + 2 * p.E;
    const float2* const cs = reinterpret_cast<const float2*>(p.rope) + size_t(pos) * (p.rope_dim / 2);
    const DkEx* const qkv = p.ex_q;
    const int pstride = group * DK_PS;       // words of one split's partial results
    DkEx* const part = p.ex_s + size_t(kvh) * p.nsplit * pstride;

    AcKeys<GP, 4, D1_WARPS> keys(kc, vc, size_t(KD), t0, t1, warp, lane);
    keys.first(pos);
    if (warp <= group) {
        const bool key = warp == group;
        d1_head(p, qkv + (key ? QD + kvh * DK_HD : (kvh * group + warp) * DK_HD), num, key ? q_norm + DK_HD : q_norm, cs, key ? knew : qs + warp * DK_HD, lane, dead);
    } else if (warp <= GP) *reinterpret_cast<float4*>(qs + (warp - 1) * DK_HD + 4 * lane) = make_float4(0.f, 0.f, 0.f, 0.f);  // heads the group does not have
    if (warp == D1_WARPS - 1) {
        const DkEx* src = qkv + QD + KD + kvh * DK_HD + 4 * lane;
        DkEx v[4];
        ex_ld2(src, v[0], v[1]);
        ex_ld2(src + 2, v[2], v[3]);
        Wait wait;
        while ((v[0].num != num || v[1].num != num || v[2].num != num || v[3].num != num) && wait.again(p, dead)) {
            ex_ld2(src, v[0], v[1]);
            ex_ld2(src + 2, v[2], v[3]);
        }
        *reinterpret_cast<float4*>(vnew + 4 * lane) = make_float4(v[0].v, v[1].v, v[2].v, v[3].v);
    }
    d1_sync();
    if (split == ns - 1 && threadIdx.x < DK_HD) {  // KV append (src/model.cpp:186-189): only row `pos` is written
        kc[size_t(pos) * KD + threadIdx.x] = knew[threadIdx.x];
        vc[size_t(pos) * KD + threadIdx.x] = vnew[threadIdx.x];
    }
    d1_stamp(p, l, 12);
    keys.walk(pos, knew, vnew, as, p.scale);
    d1_stamp(p, l, 13);
    DkEx* const att = p.ex_a;
    ac_finish<GP, 4, D1_WARPS>(keys.w, as, group, warp, lane, [] { d1_sync(); }, [&](int h, int d, float o) {
        if (ns == 1) {
            ex_st(att + (kvh * group + h) * DK_HD + d, o / as.l[h], num);
        } else {
            ex_st(part + split * pstride + h * DK_PS + d, o, num);
            if (d < 2) ex_st(part + split * pstride + h * DK_PS + DK_HD + d, d ? as.l[h] : as.m[h], num);
        }
    });
    if (ns > 1) {
        // The splits of a KV head share its outputs: each waits for everybody's results of its slice (groups of 4
        // dimensions; one thread per split and group, one trip through L2) and adds them in split order. By split 0 alone,
        // four splits at a time, it took 18 of the 24 us of this phase at 1024 keys on the 32B shape.
        const int f0 = range_lo(group * 32, ns, split), cnt = range_lo(group * 32, ns, split + 1) - f0;
        float4* const so = reinterpret_cast<float4*>(as.red);             // [ns][cnt]
        float2* const sm = reinterpret_cast<float2*>(so + ns * cnt);       // [ns][cnt] maximum, sum
        d1_sync();
        const int idx = threadIdx.x;
        if (idx < ns * cnt) {
            const int q = idx / cnt, f = f0 + idx - q * cnt, h = f >> 5;
            const DkEx* src = part + q * pstride + h * DK_PS;
            DkEx o[4], m, l2;
            auto get = [&] {
                ex_ld2(src + (f & 31) * 4, o[0], o[1]);
                ex_ld2(src + (f & 31) * 4 + 2, o[2], o[3]);
                ex_ld2(src + DK_HD, m, l2);
            };
            get();
            Wait wait;
            while ((o[0].num != num || o[1].num != num || o[2].num != num || o[3].num != num || m.num != num || l2.num != num) && wait.again(p, dead)) get();
            so[idx] = make_float4(o[0].v, o[1].v, o[2].v, o[3].v);
            sm[idx] = make_float2(m.v, l2.v);
        }
        d1_sync();
#pragma unroll 1
        for (int e = idx; e < cnt * 4; e += D1_WORKERS) {
            const int f = e >> 2;
            float M = -INFINITY, L = 0.f, o = 0.f;
#pragma unroll 1
            for (int q = 0; q < ns; ++q) M = fmaxf(M, sm[q * cnt + f].x);
#pragma unroll 2
            for (int q = 0; q < ns; ++q) {
                const float w = expf(sm[q * cnt + f].x - M);
                L = fmaf(sm[q * cnt + f].y, w, L);
                o = fmaf(reinterpret_cast<const float*>(so + q * cnt)[e], w, o);
            }
            ex_st(att + kvh * group * DK_HD + f0 * 4 + e, o / L, num);
        }
    }
    d1_sync();  // the scratch area is the next conversion's
}

// ---------------------------------------------------------------- the step

__host__ __device__ inline int d1_group_pad(int group) { return group <= 2 ? 2 : group <= 4 ? 4 : 8; }
__host__ __device__ inline size_t d1_scratch_bytes(int n_max, int group, bool f16) {
    const size_t act = f16 ? size_t(n_max) * 4 : dk_act_bytes(n_max);
    const size_t attn = size_t(DK_MAXG * DK_HD + 2 * DK_HD + ac_smem_floats(d1_group_pad(group), D1_WARPS)) * 4;
    return ((act > attn ? act : attn) + 15) / 16 * 16;
}

template <bool F16M, int GP>  // F16M: all matrices F16 (else all quantized); GP: query heads per KV head, rounded up to 2, 4 or 8
__global__ void __launch_bounds__(D1_THREADS, 1) k_decode_one(const __grid_constant__ DkParams p, const int ring_bytes) {
    extern __shared__ __align__(128) uint8_t smem[];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // shared memory: rings | scratch (the running matvec's activation, or the attention's) | row sums | kept rows | sums of
    // squares | flags | mbarriers | tables
    float* scratch = reinterpret_cast<float*>(smem + size_t(D1_WARPS) * ring_bytes);
    Smem1 s;
    s.red = reinterpret_cast<float*>(reinterpret_cast<uint8_t*>(scratch) + d1_scratch_bytes(p.n_max, p.H / p.HKV, F16M));
    s.xrow = s.red + D1_WARPS * p.slots * 16;
    s.red8 = reinterpret_cast<double*>(s.xrow + 2 * p.cta_tiles * 16);
    s.flags = reinterpret_cast<int*>(s.red8 + D1_WARPS + 1);
    uint64_t* bars0 = reinterpret_cast<uint64_t*>(s.flags + 4);
    Share* shares = reinterpret_cast<Share*>(bars0 + D1_WARPS * DK_NBAR);
    CtaShare* cta = reinterpret_cast<CtaShare*>(shares + D1_WARPS * K1_KINDS);
    int* who = reinterpret_cast<int*>(cta + K1_KINDS);
    RingShared* rshared = reinterpret_cast<RingShared*>(who + p.tile_base[K1_KINDS]);
    const int wk = warp < D1_WARPS ? warp : 0;
    s.shares = shares + wk * K1_KINDS;
    s.cta = cta;
    s.who = who;
    Ring rg;
    rg.base = dk_smem_u32(smem) + uint32_t(wk * ring_bytes);
    rg.bars = dk_smem_u32(bars0 + wk * DK_NBAR);
    rg.bytes = ring_bytes;
    rg.c_off = 0;
    rg.c_seq = rg.freed = 0u;
    rg.freed_out = dk_smem_u32(rshared->freed + wk);
    if (tid == 0) { s.flags[2] = 0; s.flags[3] = p.pos[p.ctl[0]]; rshared->producer_done = 0; }
    if (tid < D1_WARPS) { rshared->freed[tid] = 0u; rshared->issued[tid] = 0u; }
    if (warp < D1_WARPS && lane < K1_KINDS) {  // this warp's share of every kind of matrix (kinds the model does not have: empty)
        const int kind = lane;
        WarpRange r{0, 0, 0, 0};
        int upt = 1;
        if (kind < p.n_qkv || (kind >= K1_WO && kind < K1_DOWN + p.down_parts)) {
            DkKind k = d1_whole(p, kind);
            k.upt = upt = p.upt1[kind];
            r = warp_range(k, warp, D1_WARPS);
        }
        shares[warp * K1_KINDS + kind] = Share{r.wB - r.wA, r.wA % upt, r.wA / upt, 0};
        if (warp == 0) {
            const int t0 = r.cA / upt, t1 = r.cA < r.cB ? (r.cB - 1) / upt + 1 : t0;
            cta[kind] = CtaShare{t0, t1 - t0, r.cA % upt == 0, r.cB % upt == 0};
        }
    }
    if (warp < D1_WARPS && lane == 0) {
#pragma unroll 1
        for (int i = 0; i < DK_NBAR; ++i)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(rg.bars + i * 8u), "r"(1));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();  // the only barrier of all sixteen warps

    // the weight stream starts here: from now to the end of the step the producer warp keeps every ring as full as it gets
    if (warp >= D1_WARPS) {
        d1_producer<F16M>(p, dk_smem_u32(smem), ring_bytes, dk_smem_u32(bars0), shares, rshared, &s.flags[2], lane);
        return;
    }
    if (warp < K1_KINDS) {  // which warps have units of a row tile (used behind the first stage's barrier)
        const CtaShare cs = cta[warp];
        const int upt = p.upt1[warp];
        for (int t = lane; t < cs.tiles; t += 32) {
            int lo = 255, hi = 0, slot = 0;
            for (int w = 0; w < D1_WARPS; ++w) {
                const Share sh = shares[w * K1_KINDS + warp];
                const int at = cs.tile + t - sh.tile;  // which of the warp's row tiles this one is
                if (sh.units == 0 || at < 0 || at * upt >= sh.b0 + sh.units) continue;
                if (lo == 255) { lo = w; slot = at; }
                hi = w;
            }
            who[p.tile_base[warp] + t] = lo | hi << 8 | slot << 16;
        }
    }
    int* dead = &s.flags[2];
    const unsigned num0 = p.ctl[2] * unsigned(p.n_layer) + 1u;  // the number of layer 0's pass: layers are numbered through all launches
    {   // token embedding (get_row, src/ops.cpp:76-82 of the reference): the CTAs decode slices of the row into an exchange buffer
        const int64_t R = p.token[p.ctl[0]];
        const int lo = range_lo(p.E, gridDim.x, blockIdx.x), hi = range_lo(p.E, gridDim.x, blockIdx.x + 1);
#pragma unroll 1
        for (int k = lo + tid; k < hi; k += D1_WORKERS)
            ex_st(p.ex_e + k,
                  p.embd_type == ELB_F16 ? __half2float(reinterpret_cast<const __half*>(p.embd)[R * p.E + k])
                                         : elem_value(p.embd_type, tiled_elem(p.embd_type, p.embd, p.E, R, k)),
                  num0);
    }

    // The step as ONE loop over its matvec stages - per layer q|k|v (0), attn_output (1), gate|up (2), ffn_down (3), then
    // the head (4) - so that conversion, matvec and attention exist once in the kernel.
    const int n_stages = 4 * p.n_layer + 1;
    int kept = 0;  // which half of xrow holds the rows that the next row-parallel matvec adds to
#pragma unroll 1
    for (int stage = 0; stage < n_stages; ++stage) {
        const bool head = stage + 1 == n_stages;
        const int l = head ? p.n_layer : stage >> 2, k = head ? 4 : stage & 3;
        const unsigned num = num0 + unsigned(l);
        const unsigned num_in = (k == 0 || head) && stage > 0 ? num - 1u : num;  // (q|k|v and the head read the layer before)
        if (k == 0) d1_stamp(p, l, 0);
        if (k == 1) {  // attention sits between q|k|v and attn_output
            d1_attention<GP>(p, l, num, scratch, &s.flags[3], dead);
            d1_stamp(p, l, 3);
        }
        const float* const layer_norms = p.norms + size_t(l) * p.norm_stride;  // (not read for the head)
        const DkEx *A, *B = nullptr;
        const float* norm_w = nullptr;
        int n = p.E, nl = 4, nm = 1, i0, kind0;
        switch (k) {
            case 0:
                A = stage == 0 ? p.ex_e : p.ex_p2;
                norm_w = layer_norms; nl = p.nl_qkv; i0 = 0; kind0 = 0; nm = p.n_qkv;
                break;
            case 1: A = p.ex_a; n = p.H * DK_HD; nl = p.nl_wo; i0 = p.n_qkv; kind0 = K1_WO; break;
            case 2: A = p.ex_p1; norm_w = layer_norms + p.E; nl = p.nl_gu; i0 = p.n_qkv + 1; kind0 = K1_GU; break;
            case 3: A = p.ex_g; n = p.F; nl = p.nl_down; i0 = p.n_qkv + 2; kind0 = K1_DOWN; nm = p.down_parts; break;
            default: A = p.ex_p2; norm_w = p.output_norm; i0 = 0; kind0 = K1_HEAD; break;
        }
        if (norm_w && stage > 0) B = A + p.E;
        int need = 0;
        bool mine = false;  // has this CTA a share of the stage's matrices?
        for (int i = 0; i < nm; ++i) {
            if (!F16M) need |= sd_need(p.wtype[l][d1_weight_of(p, i0 + i)]);
            mine = mine || s.cta[kind0 + i].tiles > 0;
        }
        Rows rows{nullptr, 0, 0, nullptr};
        if (norm_w) {
            kept ^= 1;
            rows.keep = s.xrow + kept * p.cta_tiles * 16;
            if (head) {
                rows.out = p.x;
            } else {
                const CtaShare next = s.cta[k == 0 ? K1_WO : K1_DOWN];
                rows.r0 = next.tile * 16;
                rows.r1 = rows.r0 + next.tiles * 16;
            }
        }
        float inv = 1.0f;
        if (mine) {
            const int parts = k == 3 ? p.down_parts : 1, mats = k == 3 ? 1 : nm, per = p.down_parts > 1 && k == 3 ? p.down_blocks : n / 256;
            const ActSmem act = act_at(reinterpret_cast<int8_t*>(scratch), per * 256);
#pragma unroll 1
            for (int part = 0; part < parts; ++part) {
                if (part) d1_sync();  // the activation of the part before has been used
                if (norm_w) d1_convert<true, F16M>(p, A, B, num_in, norm_w, 0, per, nl, act, need, s.red8, rows, dead);
                else d1_convert<false, F16M>(p, A, nullptr, num_in, nullptr, part * per, per, nl, act, need, s.red8, rows, dead);
                d1_sync();
                if (part == 0) d1_stamp(p, l, k == 0 ? 1 : 3 * k + 1);
#pragma unroll 1
                for (int i = 0; i < mats; ++i) d1_matvec<F16M>(p, p.wtype[l][i0 + i], kind0 + part + i, rg, act, s);
            }
            if (norm_w) {
                double S = lane < D1_WARPS ? s.red8[lane] : 0.0;
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) S += __shfl_xor_sync(0xffffffffu, S, o);
                S = __shfl_sync(0xffffffffu, S, 0);
                inv = float(rsqrt_d(S * p.inv_E + double(p.eps)));
            }
        } else if (norm_w) {
            d1_keep_rows(p, A, B, num_in, rows, dead);
        }
        if (d1_sync_dead(dead)) break;  // (the row sums are in place; all warps agree to stop when a wait has run out)
        if (mine) {
            const int segs = k == 0 ? nm : 1;
#pragma unroll 1
            for (int i = 0; i < segs; ++i) d1_epilogue(p, k, kind0 + i, k == 0 ? 1 : nm, i, num, inv, s, s.xrow + kept * p.cta_tiles * 16);
        }
        d1_stamp(p, l, k == 0 ? 2 : k == 1 ? 5 : k == 2 ? 8 : 11);
    }
    ring_drain(rg, rshared, warp);  // (nothing is left in flight after a whole step; after a timeout the copies still land here)
    if (tid == 0) {  // the last CTA to finish moves the step on: every CTA has read ctl by then
        const unsigned step = __ldcg(p.ctl), epoch = __ldcg(p.ctl + 2);
        __threadfence();
        const unsigned old = atomicAdd(p.fin, 1u);
        if (old == gridDim.x - 1) {
            *p.fin = 0u;
            p.ctl[2] = epoch + 1;
            if (p.ctl[1]) p.ctl[0] = step + 1;
        }
    }
}

const void* d1_kernel(const DkParams& p) {
    const int gp = d1_group_pad(p.H / p.HKV);
#define ELB_D1(G) (p.f16 ? reinterpret_cast<const void*>(k_decode_one<true, G>) : reinterpret_cast<const void*>(k_decode_one<false, G>))
    return gp == 2 ? ELB_D1(2) : gp == 4 ? ELB_D1(4) : ELB_D1(8);
#undef ELB_D1
}
size_t d1_fixed_smem(const DkParams& p) {  // everything but the rings
    return d1_scratch_bytes(p.n_max, p.H / p.HKV, p.f16 != 0) + size_t(D1_WARPS) * p.slots * 16 * 4 + size_t(2) * p.cta_tiles * 16 * 4 +
           (D1_WARPS + 1) * 8 + 4 * 4 + size_t(D1_WARPS) * DK_NBAR * 8 + size_t(D1_WARPS) * K1_KINDS * sizeof(Share) + K1_KINDS * sizeof(CtaShare) +
           size_t(p.tile_base[K1_KINDS]) * 4 + sizeof(RingShared);
}

}  // namespace

int decode_one_f16_unit() { return D1_F16_UNIT; }

// Tensor maps of an F16 model's matrices (row-major fp16, tiles of 16 rows x 128 k) in execution order, [n_layer + 1][6];
// false: tensor maps cannot be made here.
bool decode_one_f16_maps(const DkParams& p, void* host) {
    using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) {
        cudaGetLastError();
        return false;
    }
    for (int l = 0; l <= p.n_layer; ++l)
        for (int i = 0; i < (l < p.n_layer ? p.n_qkv + 3 : 1); ++i) {
            const DkKind& k = l == p.n_layer ? p.kind[6] : i < p.n_qkv ? p.kind[i] : p.kind[3 + i - p.n_qkv];
            CUtensorMap map;
            const cuuint64_t dims[2] = {cuuint64_t(k.n), cuuint64_t(k.tiles) * 16}, strides[1] = {cuuint64_t(k.n) * 2};
            const cuuint32_t box[2] = {128, 16}, estr[2] = {1, 1};
            if (reinterpret_cast<EncodeFn>(fn)(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 2, const_cast<uint8_t*>(p.W[l][i]), dims, strides, box, estr,
                                               CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                                               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
                return false;
            std::memcpy(static_cast<uint8_t*>(host) + (size_t(l) * DK_LAYER_MATS + i) * 128, &map, 128);
        }
    return true;
}

// Bytes of the exchange buffers; sets the pointers of `p` when base is not null. All words zero: number 0 is no layer's.
size_t decode_one_exchange(DkParams& p, uint8_t* base) {
    size_t at = 0;
    auto take = [&](DkEx** out, size_t words) {
        if (base) *out = reinterpret_cast<DkEx*>(base + at);
        at += (words * sizeof(DkEx) + 255) / 256 * 256;
    };
    const size_t E = size_t(p.E);
    take(&p.ex_e, E);
    take(&p.ex_q, size_t(p.qkv_len));
    take(&p.ex_a, size_t(p.H) * DK_HD);
    take(&p.ex_p1, 2 * E);
    take(&p.ex_g, size_t(p.F));
    take(&p.ex_p2, 2 * E);
    take(&p.ex_s, size_t(p.HKV) * p.nsplit * (p.H / p.HKV) * DK_PS);
    return at;
}
// Steps after which the numbers of the layers' passes would start again.
int64_t decode_one_steps(const DkParams& p) { return (int64_t(0xFFFFFFFFu) - 1) / p.n_layer; }

// Bytes per warp ring when the kernel takes all the shared memory a CTA can have (a multiple of 128), capped so that a
// warp cannot have more than DK_NBAR of the smallest units on request; 0 when not even two of the largest units fit.
static int ring_bytes_of(const DkParams& p, int max_unit, int min_unit, size_t smem_optin) {
    const size_t fixed = d1_fixed_smem(p);
    if (smem_optin < fixed + size_t(D1_WARPS) * 2 * max_unit) return 0;
    size_t per = (smem_optin - fixed) / D1_WARPS / 128 * 128;
    per = std::min(per, size_t(DK_NBAR) * min_unit / 128 * 128);
    return per >= size_t(2) * max_unit ? int(per) : 0;
}

// How a step's shared memory is used, from the shapes in `p` (kind, n_qkv, E, F, H, HKV, f16): parts of ffn_down, sizes of the
// activation, of the reduction buffer and of the tables. Returns the bytes of a warp's ring, 0: the shape does not fit.
// Rings and activation share an SM's memory: ffn_down's activation is worked off in as many equal parts as leave the rings
// 8 KB per warp (three to four units of weights).
int decode_one_plan(DkParams& p, int grid, int max_unit, int min_unit, size_t smem_optin) {
    for (p.down_parts = 1; p.down_parts <= DK_MAX_PARTS; ++p.down_parts) {
        if (p.kind[5].upt % p.down_parts || (p.F / 256) % p.down_parts) continue;
        p.n_max = std::max({p.E, p.H * DK_HD, p.F / p.down_parts});
        p.down_blocks = p.F / 256 / p.down_parts;
        p.slots = p.cta_tiles = 0;
        int table = 0, qkv = 0, down = 0;  // entries of the row-tile table; row-tile slots of q|k|v and of the parts, side by side
        for (int i = 0; i < DK_ONE_KINDS; ++i) {
            DkKind k = d1_whole(p, i);
            k.upt = p.upt1[i] = i < K1_DOWN ? k.upt : k.upt / p.down_parts;
            p.tile_base[i] = table;
            p.slot_base[i] = 0;
            if (i < 3 ? i < p.n_qkv : i < K1_DOWN + p.down_parts) {
                const CutExtent e = cut_extent(k, grid, D1_WARPS);
                int* side = i < 3 ? &qkv : i >= K1_DOWN ? &down : nullptr;
                if (side) { p.slot_base[i] = *side; *side += e.warp; }
                p.slots = std::max(p.slots, p.slot_base[i] + e.warp);
                table += e.cta;
                if (i == K1_WO || i == K1_DOWN) p.cta_tiles = std::max(p.cta_tiles, e.cta);  // rows of the residual stream a CTA keeps
            }
            p.tile_base[i + 1] = table;
        }
        const int ring = ring_bytes_of(p, max_unit, min_unit, smem_optin);
        if (ring >= std::max(8192, 2 * max_unit)) return ring;
    }
    return 0;
}

// Self-test without a GPU. shape: {n_embd, n_ff, n_head, n_head_kv, n_vocab}; types: block formats of q, k, v, attn_output,
// gate|up, ffn_down, head; out: {parts of ffn_down, ring bytes, slots per warp, tiles kept}, then the first table entry and the
// first slot of every kind of matrix (q, k, v, attn_output, gate|up, head, four parts of ffn_down), then the table's length.
int decode_one_selftest_plan(const int* shape, const int* types, int ctas, size_t smem, int* out) {
    DkParams p{};
    p.E = shape[0]; p.F = shape[1]; p.H = shape[2]; p.HKV = shape[3]; p.n_qkv = 3;
    p.f16 = types[6] == ELB_F16;
    const int QD = p.H * DK_HD, KD = p.HKV * DK_HD, rows[7] = {QD, KD, KD, p.E, 2 * p.F, p.E, shape[4]}, n[7] = {p.E, p.E, p.E, QD, p.E, p.F, p.E};
    int unit_max = 0, unit_min = 1 << 30;
    long long cost[3];
    for (int i = 0; i < 7; ++i) {
        const int tiles = (rows[i] + 15) / 16, upt = n[i] / (types[i] == ELB_F16 || types[i] == ELB_Q8_0 ? 128 : 256);
        const int ub = types[i] == ELB_F16 ? D1_F16_UNIT : types[i] == ELB_Q4_K ? Q4K_UNIT : types[i] == ELB_Q6_K ? Q6K_UNIT : Q8_UNIT;
        p.kind[i] = DkKind{tiles, upt, rows[i], n[i], tiles, 0, 0, 0};
        p.kind[i].balanced = (i == 3 || i == 5) && tiles >= ctas;
        if (i < 3) cost[i] = decode_unit_cost(types[i]);
        unit_max = std::max(unit_max, ub);
        unit_min = std::min(unit_min, ub);
    }
    decode_cut_qkv(p, cost);
    out[1] = decode_one_plan(p, ctas, unit_max, unit_min, smem);
    out[0] = out[1] ? p.down_parts : 0;
    out[2] = p.slots;
    out[3] = p.cta_tiles;
    for (int i = 0; i < DK_ONE_KINDS; ++i) { out[4 + i] = p.tile_base[i]; out[4 + DK_ONE_KINDS + i] = p.slot_base[i]; }
    out[4 + 2 * DK_ONE_KINDS] = p.tile_base[DK_ONE_KINDS];
    return ELB_OK;
}

int decode_one_launch(const DkParams& p, int ring_bytes, int grid, cudaStream_t s) {
    const size_t smem = size_t(D1_WARPS) * ring_bytes + d1_fixed_smem(p);
    ELB_TRY(ensure_dyn_smem(d1_kernel(p), smem));
    void* args[] = {const_cast<DkParams*>(&p), const_cast<int*>(&ring_bytes)};
    ELB_CUDA(cudaLaunchCooperativeKernel(d1_kernel(p), dim3(grid), dim3(D1_THREADS), args, smem, s));
    return ELB_OK;
}

// can one CTA per SM be resident with rings of this size?
int decode_one_fits(const DkParams& p, int ring_bytes, int device, bool* fits) {
    DeviceInfo di;
    ELB_TRY(device_info(device, &di));
    const size_t smem = size_t(D1_WARPS) * ring_bytes + d1_fixed_smem(p);
    *fits = false;
    if (smem > di.smem_optin) return ELB_OK;
    ELB_TRY(ensure_dyn_smem(d1_kernel(p), smem));
    int per_sm = 0;
    ELB_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, d1_kernel(p), D1_THREADS, smem));
    *fits = per_sm >= 1;
    return ELB_OK;
}

}  // namespace elb
