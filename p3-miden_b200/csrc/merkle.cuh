// Lifted Merkle tree (LMCS) kernels: leaf sponge absorption with virtual
// lifting, and layer compression.
//
// Leaf semantics (p3-miden-lmcs/src/lifted_tree.rs:385-483): leaf j of a tree
// of height H absorbs, for every matrix m in ascending-height order, row
// j >> log2(H/h_m) of m, each row in its own absorb call (overwrite mode,
// rate 8, zero-padded partial chunk; field_sponge.rs:164-182), then squeezes
// state[0..4]. Matrices are processed one height class at a time: the
// states of a class of height h are computed from the states of the
// previous class at index j >> log2(h/h_prev); nothing is upsampled in
// memory.
//
// Digest layers of a tree of height H live in one buffer of 2H-1 digests
// (4 words each), layer l (H >> l digests) at digest offset 2H - 2(H >> l).
#pragma once
#include "gl.cuh"
#include "poseidon2.cuh"

__constant__ uint64_t c_p2[p2::N_DEVICE];

// Device permutation: one looped copy of the round body per call site, so
// that kernels stay small enough for the instruction cache (the fully
// unrolled form stalled on instruction fetch). Rounds 0-3 and 26-29 are
// external, 4-25 internal; constants come from the __constant__ table.
//
// Arithmetic is lazy: state words are kept weakly reduced (any value below
// 2^64 congruent mod p); the linear layers reduce once per output; s*mu + sum
// is reduced once from 128 bits. Products are reduced in Montgomery form
// (R = 2^64): R^3 = 1 mod p, so x^7 needs no conversion and a product with a
// constant takes the constant times R. Callers canonicalise words that leave
// the permutation (p2w::canon). Measured 1.38 G permutations/s against 1.27
// with plain reductions (B200, 1965 MHz, chained permutations); p2tc.cuh's
// form is faster where a launch has enough states.
namespace p2w {
constexpr uint64_t EPS = 0xFFFFFFFFull;
struct W {  // lo + hi * 2^64
    uint64_t lo;
    uint32_t hi;
};
// a * b / 2^64 mod p, weakly reduced
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t b) { return gl::mont_mul(a, b); }
__device__ __forceinline__ uint64_t canon(uint64_t a) { return gl::canon_dev(a); }
// weak + canonical: one wrap at most (a + c - 2^64 + eps < 2^64)
__device__ __forceinline__ uint64_t add_c(uint64_t a, uint64_t c) {
    uint32_t r0, r1;
    asm("{\n\t.reg .u32 k;\n\t"
        "add.cc.u32 %0, %2, %4;\n\t"
        "addc.cc.u32 %1, %3, %5;\n\t"
        "addc.u32 k, 0, 0;\n\t"
        "neg.s32 k, k;\n\t"
        "add.cc.u32 %0, %0, k;\n\t"
        "addc.u32 %1, %1, 0;\n\t}"
        : "=&r"(r0), "=&r"(r1)
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)c), "r"((uint32_t)(c >> 32)));
    return ((uint64_t)r1 << 32) | r0;
}
__device__ __forceinline__ W wide(uint64_t a) { return W{a, 0}; }
__device__ __forceinline__ W wadd(W a, W b) {
    uint32_t r0, r1, h;
    asm("add.cc.u32 %0, %3, %6;\n\t"
        "addc.cc.u32 %1, %4, %7;\n\t"
        "addc.u32 %2, %5, %8;"
        : "=&r"(r0), "=&r"(r1), "=&r"(h)
        : "r"((uint32_t)a.lo), "r"((uint32_t)(a.lo >> 32)), "r"(a.hi), "r"((uint32_t)b.lo),
          "r"((uint32_t)(b.lo >> 32)), "r"(b.hi));
    return W{((uint64_t)r1 << 32) | r0, h};
}
__device__ __forceinline__ W wadd1(W a, uint64_t b) {
    uint32_t r0, r1, h;
    asm("add.cc.u32 %0, %3, %6;\n\t"
        "addc.cc.u32 %1, %4, %7;\n\t"
        "addc.u32 %2, %5, 0;"
        : "=&r"(r0), "=&r"(r1), "=&r"(h)
        : "r"((uint32_t)a.lo), "r"((uint32_t)(a.lo >> 32)), "r"(a.hi), "r"((uint32_t)b), "r"((uint32_t)(b >> 32)));
    return W{((uint64_t)r1 << 32) | r0, h};
}
__device__ __forceinline__ W wdbl(uint64_t a) { return wadd1(wide(a), a); }
// lo + hi * 2^64 with hi < 2^32: lo + hi * eps, one wrap at most
__device__ __forceinline__ uint64_t wreduce(W a) {
    uint32_t r0, r1;
    asm("{\n\t.reg .u32 u0, u1, c;\n\t"
        "sub.cc.u32 u0, 0, %4;\n\t"  // hi*eps = (hi << 32) - hi
        "subc.u32 u1, %4, 0;\n\t"
        "add.cc.u32 %0, %2, u0;\n\t"
        "addc.cc.u32 %1, %3, u1;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "neg.s32 c, c;\n\t"          // on carry add eps
        "add.cc.u32 %0, %0, c;\n\t"
        "addc.u32 %1, %1, 0;\n\t}"
        : "=&r"(r0), "=&r"(r1)
        : "r"((uint32_t)a.lo), "r"((uint32_t)(a.lo >> 32)), "r"(a.hi));
    return ((uint64_t)r1 << 32) | r0;
}
// x^7: the four products leave a factor 2^(-64 * 6) = (2^192)^-2 = 1 mod p
__device__ __forceinline__ uint64_t sbox(uint64_t x) {
    uint64_t x2 = mul(x, x), x4 = mul(x2, x2), x3 = mul(x2, x);
    return mul(x4, x3);
}
// a*b + c for a, b < 2^64 and a 96-bit c below 2^68: c enters the product's
// carry chain whole (its top word on the third limb, where the product chain
// starts from zero), so a sum shared by several products is never reduced on
// its own. a*b + c <= (2^64-1)^2 + 2^68 < 2^128; weakly reduced.
__device__ __forceinline__ uint64_t mul_add_w(uint64_t a, uint64_t b, W c) {
    uint32_t r0, r1, r2, r3;
    asm("mad.lo.cc.u32 %0, %4, %6, %8;\n\t"
        "madc.hi.cc.u32 %1, %4, %6, %9;\n\t"
        "addc.u32 %2, %10, 0;\n\t"
        "mad.lo.cc.u32 %1, %4, %7, %1;\n\t"
        "madc.hi.cc.u32 %2, %4, %7, %2;\n\t"
        "addc.u32 %3, 0, 0;\n\t"
        "mad.lo.cc.u32 %1, %5, %6, %1;\n\t"
        "madc.hi.cc.u32 %2, %5, %6, %2;\n\t"
        "addc.u32 %3, %3, 0;\n\t"
        "mad.lo.cc.u32 %2, %5, %7, %2;\n\t"
        "madc.hi.u32 %3, %5, %7, %3;"
        : "=&r"(r0), "=&r"(r1), "=&r"(r2), "=&r"(r3)
        : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)), "r"((uint32_t)b), "r"((uint32_t)(b >> 32)),
          "r"((uint32_t)c.lo), "r"((uint32_t)(c.lo >> 32)), "r"(c.hi));
    return gl::reduce4_dev(r0, r1, r2, r3);
}
// M4 = circ(2,3,1,1) on sums modulo 2^64 and on 32-bit sums
template <typename T>
__device__ __forceinline__ void m4(T a, T b, T c, T d, T *y) {
    const T t01 = a + b, t23 = c + d, t = t01 + t23, t1 = t + b, t3 = t + d;
    y[0] = t1 + t01;      // 2a + 3b + c + d
    y[1] = t1 + (c + c);  // a + 2b + 3c + d
    y[2] = t3 + t23;      // a + b + 2c + 3d
    y[3] = t3 + (a + a);  // 3a + b + c + 2d
}
// A sum of at most 29 words, given modulo 2^64 (w) and as the sum h of the
// words' top 27 bits (h <= 29 (2^27 - 1) < 2^32): the sum is
// 2^37 h + d 2^37 + ... with 0 <= d < 29, and w >> 37 = h + d mod 2^27, so
// g = ceil((h - (w >> 37)) / 2^27) counts its wraps of 2^64. The value is
// w + g * eps, with one wrap at most.
__device__ __forceinline__ uint64_t fold_wraps(uint64_t w, uint32_t h) {
    const uint32_t g = (h - (uint32_t)(w >> 37) + 31) >> 27;
    const uint64_t u = (uint64_t)g * 0xFFFFFFFFu;
    uint32_t r0, r1;
    asm("{\n\t.reg .u32 c;\n\t"
        "add.cc.u32 %0, %2, %4;\n\t"
        "addc.cc.u32 %1, %3, %5;\n\t"
        "addc.u32 c, 0, 0;\n\t"
        "neg.s32 c, c;\n\t"
        "add.cc.u32 %0, %0, c;\n\t"
        "addc.u32 %1, %1, 0;\n\t}"
        : "=&r"(r0), "=&r"(r1)
        : "r"((uint32_t)w), "r"((uint32_t)(w >> 32)), "r"((uint32_t)u), "r"((uint32_t)(u >> 32)));
    return ((uint64_t)r1 << 32) | r0;
}
// circ(2*M4, M4, M4). Every output is a sum of 28 words (and a constant): it
// is formed modulo 2^64, with 64-bit additions, beside the sum of the words'
// top 27 bits, which gives the number of wraps (fold_wraps). 171 ALU and 106
// multiplier-pipe instructions per layer against 230 and 69 for 96-bit carry
// chains: 392 against 468 cycles per warp (B200, 8 warps per scheduler). With
// rc_off >= 0 the next round's constants c_p2[rc_off + i] join the sums.
// capacity_only: words 0..7 are left undefined.
__device__ __forceinline__ void ext_linear(uint64_t *s, int rc_off = -1, bool capacity_only = false) {
    uint64_t y[12];
    uint32_t z[12];
#pragma unroll
    for (int c = 0; c < 12; c += 4) {
        m4<uint64_t>(s[c], s[c + 1], s[c + 2], s[c + 3], y + c);
        m4<uint32_t>((uint32_t)(s[c] >> 37), (uint32_t)(s[c + 1] >> 37), (uint32_t)(s[c + 2] >> 37),
                     (uint32_t)(s[c + 3] >> 37), z + c);
    }
#pragma unroll
    for (int k = 0; k < 4; k++) {
        const uint64_t t = y[k] + y[k + 4] + y[k + 8];
        const uint32_t u = z[k] + z[k + 4] + z[k + 8];
#pragma unroll
        for (int j = 8; j >= 0; j -= 4) {
            if (j == 4 && capacity_only) break;
            uint64_t w = y[k + j] + t;
            uint32_t h = z[k + j] + u;
            if (rc_off >= 0) {
                const uint64_t rc = c_p2[rc_off + k + j];
                w += rc;
                h += (uint32_t)(rc >> 37);
            }
            s[k + j] = fold_wraps(w, h);
        }
    }
}
}  // namespace p2w

// External rounds take their constants inside the preceding linear layer
// (rounds 0-3 and 27-29); round 26 follows the internal rounds and adds its own.
// `stop` is asked before each external round and ends the permutation with the
// state undefined (the proof-of-work search; never for the hashes).
template <typename Stop>
__device__ __forceinline__ void p2_permute_until(uint64_t *s, Stop &stop) {
    p2w::ext_linear(s, p2::OFF_INIT);
#pragma unroll 1
    for (int r = 0; r < 30; r++) {
        if (r < 4 || r >= 26) {
            if (stop()) return;
            if (r == 26) {
#pragma unroll
                for (int i = 0; i < 12; i++) s[i] = p2w::add_c(s[i], c_p2[p2::OFF_TERM + i]);
            }
#pragma unroll
            for (int i = 0; i < 12; i++) s[i] = p2w::sbox(s[i]);
            p2w::ext_linear(s, r < 3 ? p2::OFF_INIT + 12 * (r + 1) : (r >= 26 && r < 29) ? p2::OFF_TERM + 12 * (r - 25) : -1);
        } else {
            s[0] = p2w::sbox(p2w::add_c(s[0], c_p2[p2::OFF_INT + r - 4]));
            p2w::W acc = p2w::wide(s[0]);
#pragma unroll
            for (int i = 1; i < 12; i++) acc = p2w::wadd1(acc, s[i]);  // below 12 * 2^64
            // the sum times 2^64: 2^64 lo + 2^128 hi = 2^64 lo - 2^32 hi (mod p)
            const uint64_t c = gl::sub_dev(gl::reduce4_dev(0, 0, (uint32_t)acc.lo, (uint32_t)(acc.lo >> 32)),
                                           (uint64_t)acc.hi << 32);
#pragma unroll
            for (int i = 0; i < 12; i++) s[i] = gl::mont_mul(s[i], c_p2[p2::OFF_DIAG_M + i], c);
        }
    }
}
struct NeverStop {
    __device__ __forceinline__ bool operator()() const { return false; }
};
__device__ __forceinline__ void p2_permute_dev(uint64_t *s) {
    NeverStop stop;
    p2_permute_until(s, stop);
}

// Permutation shared by 16 lanes, for latency-bound work (a few states at a
// time; about 0.28 of the single-thread latency). Lane l < 12 holds word
// l; what lanes 12..15 hold nobody reads. External rounds run one S-box per
// lane and move the M4 and cross-block sums through shuffles. In the internal
// rounds every lane carries a copy z of s_0: the S-box runs on z while the
// sum R of s_1..s_11 is formed by a 4-step butterfly, and
// s_0 <- (mu_0 + 1) * S(z) + R, s_i <- mu_i s_i + R + S(z) are one product in
// every lane, with the next round's constant in lane 0's sum; lane 0's word is
// then broadcast. A lone warp is bound by its own issue as much as by the
// chain, so the shared product pays for the broadcast: a chained permutation
// takes 12.8 k cycles, 17.0 k with a second product for z in every lane. Same
// lazy arithmetic as p2_permute_dev (results agree mod p); the diagonal
// products take the plain reduction, whose 96-bit addend needs no reduction of
// its own. Two states per warp; all 32 lanes must call it. `sc` is the
// constant table staged in shared memory (stage_consts).
namespace p2x {
// copy the constant table into shared memory (all threads of the block call it)
__device__ __forceinline__ void stage_consts(uint64_t *sc) {
    for (int i = threadIdx.x; i < p2::N_PARAMS; i += blockDim.x) sc[i] = c_p2[i];
    __syncthreads();
}
__device__ __forceinline__ uint64_t shfl64(uint64_t v, int src) {
    const uint32_t lo = __shfl_sync(0xffffffffu, (uint32_t)v, src, 16);
    const uint32_t hi = __shfl_sync(0xffffffffu, (uint32_t)(v >> 32), src, 16);
    return ((uint64_t)hi << 32) | lo;
}
__device__ __forceinline__ p2w::W shflW_xor(p2w::W v, int m) {
    const uint32_t lo = __shfl_xor_sync(0xffffffffu, (uint32_t)v.lo, m, 16);
    const uint32_t hi = __shfl_xor_sync(0xffffffffu, (uint32_t)(v.lo >> 32), m, 16);
    return p2w::W{((uint64_t)hi << 32) | lo, __shfl_xor_sync(0xffffffffu, v.hi, m, 16)};
}
struct Lane {
    uint64_t mu;  // diagonal word l; mu_0 + 1 mod p in lane 0; 0 for l >= 12
};
__device__ __forceinline__ Lane lane_consts(const uint64_t *sc, int l) {
    return Lane{l == 0 ? gl::add_dev(sc[p2::OFF_DIAG], 1) : l < 12 ? sc[p2::OFF_DIAG + l] : 0};
}
// circ(2*M4, M4, M4) for word l: M4 of v = x_l + the sum of the three blocks'
// words at position l mod 4, with sums modulo 2^64 beside those of the top 27
// bits as in p2w::ext_linear (28 words in all). rc: the lane's constant of the
// next round (0 for none). Lanes 12..15 return values nobody reads.
__device__ __forceinline__ uint64_t ext_linear(uint64_t x, int l, uint64_t rc = 0) {
    const uint64_t xa = shfl64(x, l < 8 ? l + 4 : l - 8), xb = shfl64(x, l < 4 ? l + 8 : l - 4);
    const uint64_t v = x + x + xa + xb;
    const uint32_t h = 2 * (uint32_t)(x >> 37) + (uint32_t)(xa >> 37) + (uint32_t)(xb >> 37);
    const int base = l & ~3;
    uint64_t w = v + v + rc;
    uint32_t u = h + h + (uint32_t)(rc >> 37);
#pragma unroll
    for (int d = 1; d < 4; d++) {
        const int src = base | ((l + d) & 3);
        const uint64_t vd = shfl64(v, src);
        const uint32_t hd = __shfl_sync(0xffffffffu, h, src, 16);
        w += d == 1 ? vd + vd + vd : vd;
        u += d == 1 ? 3 * hd : hd;
    }
    return p2w::fold_wraps(w, u);
}
// four external rounds whose first constant is already in x; each linear
// layer takes in the next round's constant
__device__ __forceinline__ uint64_t ext_rounds(uint64_t x, int l, const uint64_t *rc) {
    const int li = l < 12 ? l : 11;
#pragma unroll 1
    for (int r = 0; r < 4; r++) x = ext_linear(p2w::sbox(x), l, r < 3 ? rc[12 * (r + 1) + li] : 0);
    return x;
}
__device__ __forceinline__ uint64_t permute(uint64_t x, int l, const uint64_t *sc, const Lane &k) {
    using namespace p2w;
    const int li = l < 12 ? l : 11;
    x = ext_rounds(ext_linear(x, l, sc[p2::OFF_INIT + li]), l, sc + p2::OFF_INIT);
    const bool first = l == 0, rest = l >= 1 && l < 12;
    if (first) x = add_c(x, sc[p2::OFF_INT]);
#pragma unroll 1
    for (int r = 0; r < 22; r++) {
        const uint64_t zs = sbox(shfl64(x, 0)), rc = r < 21 ? sc[p2::OFF_INT + r + 1] : 0;
        W P = wide(rest ? x : 0);
#pragma unroll
        for (int m = 1; m < 16; m <<= 1) P = wadd(P, shflW_xor(P, m));
        x = mul_add_w(first ? zs : x, k.mu, wadd1(P, first ? rc : zs));  // sum < 12 * 2^64
    }
    return ext_rounds(add_c(x, sc[p2::OFF_TERM + li]), l, sc + p2::OFF_TERM);
}
}  // namespace p2x

// Permutation shared by 4 lanes, for launches of a few thousand states: lane
// l holds words l, l + 4 and l + 8 (position l of the three M4 blocks), so an
// S-box layer is three S-boxes per lane, the block sums are local and M4 is
// one exchange of the four positions, y_l = 2 v_l + 3 v_{l+1} + v_{l+2} +
// v_{l+3}. Internal rounds as p2x::permute. About 800 warp instructions per
// state against 545 for one thread per state and 2450 for 16 lanes; alone, a
// chained permutation takes 17.7 k cycles against 44.9 and 12.8. 8 states per
// warp; all 32 lanes must call it. `sc`: p2x::stage_consts.
namespace p2q {
__device__ __forceinline__ uint32_t from(uint32_t v, int d) {  // lane l + d of the quad
    return __shfl_sync(0xffffffffu, v, (threadIdx.x & 3) + d & 3, 4);
}
// next: index of the lane's first constant of the next round in sc, or -1
__device__ __forceinline__ void ext_linear(uint64_t *x, const uint64_t *sc, int next) {
    const uint32_t h0 = (uint32_t)(x[0] >> 37), h1 = (uint32_t)(x[1] >> 37), h2 = (uint32_t)(x[2] >> 37);
    const uint64_t tw = x[0] + x[1] + x[2];
    const uint32_t ts = h0 + h1 + h2;
    const uint32_t hs[3] = {h0, h1, h2};
#pragma unroll
    for (int k = 0; k < 3; k++) {
        const uint64_t v = x[k] + tw;  // the M4 input of block k, sums as in p2w::ext_linear
        const uint32_t h = hs[k] + ts;
        uint64_t w = v + v;
        uint32_t u = h + h;
#pragma unroll
        for (int d = 1; d < 4; d++) {
            const uint64_t vd = ((uint64_t)from((uint32_t)(v >> 32), d) << 32) | from((uint32_t)v, d);
            const uint32_t hd = from(h, d);
            w += d == 1 ? vd + vd + vd : vd;
            u += d == 1 ? 3 * hd : hd;
        }
        if (next >= 0) {
            const uint64_t rc = sc[next + 4 * k];
            w += rc;
            u += (uint32_t)(rc >> 37);
        }
        x[k] = p2w::fold_wraps(w, u);
    }
}
struct Lane {
    uint64_t mu[3];  // diagonal words of the lane; mu_0 + 1 mod p for word 0
};
__device__ __forceinline__ Lane lane_consts(const uint64_t *sc, int l) {
    return Lane{{l ? sc[p2::OFF_DIAG + l] : gl::add_dev(sc[p2::OFF_DIAG], 1), sc[p2::OFF_DIAG + l + 4],
                 sc[p2::OFF_DIAG + l + 8]}};
}
__device__ __forceinline__ void permute(uint64_t *x, const uint64_t *sc, const Lane &k) {
    using namespace p2w;
    const int l = threadIdx.x & 3;
    ext_linear(x, sc, p2::OFF_INIT + l);
#pragma unroll 1
    for (int r = 0; r < 8; r++) {
        if (r == 4) {
            if (l == 0) x[0] = add_c(x[0], sc[p2::OFF_INT]);
#pragma unroll 1
            for (int q = 0; q < 22; q++) {
                const uint64_t z = ((uint64_t)__shfl_sync(0xffffffffu, (uint32_t)(x[0] >> 32), 0, 4) << 32) |
                                   __shfl_sync(0xffffffffu, (uint32_t)x[0], 0, 4);
                const uint64_t zs = sbox(z), rc = q < 21 ? sc[p2::OFF_INT + q + 1] : 0;
                W P = wadd1(wadd1(wide(l ? x[0] : 0), x[1]), x[2]);
#pragma unroll
                for (int m = 1; m < 4; m <<= 1) P = wadd(P, p2x::shflW_xor(P, m));
                const W t = wadd1(P, zs);  // < 12 * 2^64
                x[0] = mul_add_w(l ? x[0] : zs, k.mu[0], l ? t : wadd1(P, rc));
                x[1] = mul_add_w(x[1], k.mu[1], t);
                x[2] = mul_add_w(x[2], k.mu[2], t);
            }
#pragma unroll
            for (int i = 0; i < 3; i++) x[i] = add_c(x[i], sc[p2::OFF_TERM + l + 4 * i]);
        }
#pragma unroll
        for (int i = 0; i < 3; i++) x[i] = sbox(x[i]);
        ext_linear(x, sc, r < 3 ? p2::OFF_INIT + 12 * (r + 1) + l : r == 3 || r == 7 ? -1 : p2::OFF_TERM + 12 * (r - 3) + l);
    }
}
}  // namespace p2q

namespace merkle {

constexpr int MAX_MATS = 8;

struct ClassArgs {
    const uint64_t *data[MAX_MATS];
    uint64_t width[MAX_MATS];
    uint64_t ld[MAX_MATS];  // row stride in words (>= width; a column slab of a wider matrix)
    int n_mats;
    uint32_t log_h;         // height of this class
    const uint64_t *prev;   // states of the previous class (12 words each), or null
    uint32_t prev_log_h;
    uint64_t *states_out;   // 12 words per leaf, or null when squeezing
    uint64_t *digests_out;  // 4 words per leaf, or null
    // optional column-major copy of the absorbed rows (n_mats == 1): word c
    // of row j < cm_rows is also written to cm[c * cm_ld + j] (the cells the
    // generated constraint kernels read; a warp's 32 rows make one 256-byte run)
    uint64_t *cm;
    uint64_t cm_ld, cm_rows;
};

// absorb one row (rate 8, overwrite mode, zero-padded last chunk); a single
// permutation call site
// permutation call site; with CM, each word is also stored at cmj[c * cm_ld]
// (cmj = cm + row index, or null for rows past cm_rows)
template <bool CM>
__device__ __forceinline__ void absorb_row(uint64_t *s, const uint64_t *row, uint64_t w, uint64_t *cmj,
                                           uint64_t cm_ld) {
#pragma unroll 1
    for (uint64_t i = 0; i < w; i += 8) {
        if (i + 8 <= w) {
#pragma unroll
            for (int j = 0; j < 8; j++) s[j] = __ldg(row + i + j);
            if (CM && cmj) {
#pragma unroll
                for (int j = 0; j < 8; j++) cmj[(i + j) * cm_ld] = s[j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < 8; j++) s[j] = i + j < w ? __ldg(row + i + j) : 0;
            if (CM && cmj) {
#pragma unroll
                for (int j = 0; j < 8; j++)
                    if (i + j < w) cmj[(i + j) * cm_ld] = s[j];
            }
        }
        p2_permute_dev(s);
    }
}

// At most 64 registers: eight 128-thread blocks per SM (measured: 66
// registers, seven blocks, made the slab's tree 9 % slower).
template <bool CM>
__global__ void __launch_bounds__(128, 8) leaf_class_kernel(const __grid_constant__ ClassArgs a) {
    uint64_t j = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >> a.log_h) return;
    uint64_t s[12];
    if (a.prev) {
        const uint64_t *p = a.prev + (j >> (a.log_h - a.prev_log_h)) * 12;
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = p[i];
    } else {
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = 0;
    }
    for (int m = 0; m < a.n_mats; m++)
        absorb_row<CM>(s, a.data[m] + j * a.ld[m], a.width[m], CM && j < a.cm_rows ? a.cm + j : nullptr, a.cm_ld);
    if (a.digests_out) {
#pragma unroll
        for (int i = 0; i < 4; i++) a.digests_out[j * 4 + i] = p2w::canon(s[i]);
    } else {
#pragma unroll
        for (int i = 0; i < 12; i++) a.states_out[j * 12 + i] = s[i];
    }
}

// The same leaf sponge with one 16-lane group per leaf (p2x), for classes
// with few leaves, where one thread per leaf leaves the GPU nearly empty and
// each of a row's chained permutations costs the full single-thread latency.
// States are weakly reduced like leaf_class_kernel's (congruent mod p, not
// always the same words), so classes may mix the two kernels.
constexpr uint64_t kCoopLeaves = 2048;
template <bool CM>
__global__ void __launch_bounds__(128) leaf_class_coop_kernel(const __grid_constant__ ClassArgs a) {
    __shared__ uint64_t sc[p2::N_PARAMS];
    p2x::stage_consts(sc);
    const int l = threadIdx.x & 15;
    const p2x::Lane k = p2x::lane_consts(sc, l);
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (((t & ~31ull) >> 4) >> a.log_h) return;  // warp-uniform: the warp's first leaf is past the class
    const uint64_t j = t >> 4;
    const bool ok = (j >> a.log_h) == 0;
    uint64_t x = 0;
    if (ok && a.prev && l < 12) x = a.prev[(j >> (a.log_h - a.prev_log_h)) * 12 + l];
    for (int m = 0; m < a.n_mats; m++) {
        const uint64_t w = a.width[m];
        const uint64_t *row = a.data[m] + (ok ? j : 0) * a.ld[m];
        uint64_t next = l < 8 && ok && l < w ? __ldg(row + l) : 0;  // loaded a permutation ahead
#pragma unroll 1
        for (uint64_t i = 0; i < w; i += 8) {
            if (l < 8) x = next;
            if (CM && l < 8 && ok && i + l < w && j < a.cm_rows) a.cm[(i + l) * a.cm_ld + j] = x;
            next = l < 8 && ok && i + 8 + l < w ? __ldg(row + i + 8 + l) : 0;
            x = p2x::permute(x, l, sc, k);
        }
    }
    if (!ok) return;
    if (a.digests_out) {
        if (l < 4) a.digests_out[j * 4 + l] = p2w::canon(x);
    } else if (l < 12) {
        a.states_out[j * 12 + l] = x;
    }
}

// The leaf sponge with four lanes per leaf (p2q), for classes of 2^12 to 2^14
// leaves: one thread per leaf leaves most schedulers without a warp there, and
// 16 lanes per leaf more than fill them. Trees of 2^11 / 2^12 / 2^13 / 2^14 /
// 2^15 leaves x 512 columns took 0.69 / 1.05 / 1.63 / 2.96 / 5.61 ms with 16
// lanes, - / 0.70 / 0.93 / 1.59 / 2.55 with four and 1.59 / 1.62 / 1.64 / 1.65
// / 2.37 with one thread. The next chunk's words are loaded before the
// permutation of this one.
template <bool CM>
__global__ void __launch_bounds__(128) leaf_class_quad_kernel(const __grid_constant__ ClassArgs a) {
    __shared__ uint64_t sc[p2::N_PARAMS];
    p2x::stage_consts(sc);
    const int l = threadIdx.x & 3;
    const p2q::Lane k = p2q::lane_consts(sc, l);
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (((t & ~31ull) >> 2) >> a.log_h) return;  // warp-uniform: the warp's first leaf is past the class
    const uint64_t j = t >> 2;
    const bool ok = (j >> a.log_h) == 0;
    uint64_t x[3] = {0, 0, 0};
    if (ok && a.prev) {
        const uint64_t *p = a.prev + (j >> (a.log_h - a.prev_log_h)) * 12 + l;
        x[0] = p[0], x[1] = p[4], x[2] = p[8];
    }
    for (int m = 0; m < a.n_mats; m++) {
        const uint64_t w = ok ? a.width[m] : 0, n = a.width[m];
        const uint64_t *row = a.data[m] + (ok ? j : 0) * a.ld[m];
        uint64_t c0 = l < w ? __ldg(row + l) : 0, c1 = 4 + l < w ? __ldg(row + 4 + l) : 0;
#pragma unroll 1
        for (uint64_t i = 0; i < n; i += 8) {
            x[0] = c0, x[1] = c1;
            if (CM && j < a.cm_rows) {
                if (i + l < w) a.cm[(i + l) * a.cm_ld + j] = c0;
                if (i + 4 + l < w) a.cm[(i + 4 + l) * a.cm_ld + j] = c1;
            }
            c0 = i + 8 + l < w ? __ldg(row + i + 8 + l) : 0;
            c1 = i + 12 + l < w ? __ldg(row + i + 12 + l) : 0;
            p2q::permute(x, sc, k);
        }
    }
    if (!ok) return;
    if (a.digests_out) {
        a.digests_out[j * 4 + l] = p2w::canon(x[0]);
    } else {
        uint64_t *p = a.states_out + j * 12 + l;
        p[0] = x[0], p[4] = x[1], p[8] = x[2];
    }
}

__device__ __forceinline__ void compress2(const uint64_t *l, const uint64_t *r, uint64_t *out) {
    uint64_t s[12];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        s[i] = l[i];
        s[4 + i] = r[i];
        s[8 + i] = 0;
    }
    p2_permute_dev(s);
#pragma unroll
    for (int i = 0; i < 4; i++) out[i] = p2w::canon(s[i]);
}

// One block compresses 2*blockDim.x digests of layer `l_in` through `levels`
// layers (2^levels <= 2*blockDim.x), writing every produced layer.
__global__ void __launch_bounds__(256) compress_kernel(uint64_t *layers, uint64_t H, uint32_t l_in, uint32_t levels) {
    __shared__ uint64_t sm[256 * 4];
    const uint64_t n_in = H >> l_in;
    const uint64_t off_in = 2 * H - 2 * (H >> l_in);
    const uint32_t t = threadIdx.x;
    const uint64_t parent = (uint64_t)blockIdx.x * blockDim.x + t;  // index in layer l_in+1
    uint64_t d[4];
    if (2 * parent + 1 < n_in) {
        compress2(layers + 4 * (off_in + 2 * parent), layers + 4 * (off_in + 2 * parent + 1), d);
        uint64_t off1 = 2 * H - 2 * (H >> (l_in + 1));
#pragma unroll
        for (int i = 0; i < 4; i++) {
            layers[4 * (off1 + parent) + i] = d[i];
            sm[4 * t + i] = d[i];
        }
    }
    __syncthreads();
    uint32_t active = blockDim.x;
    for (uint32_t lv = 1; lv < levels; lv++) {
        active >>= 1;
        uint64_t n_l = H >> (l_in + lv + 1);
        uint64_t pidx = (uint64_t)blockIdx.x * active + t;
        if (t < active && pidx < n_l) {
            compress2(sm + 4 * (2 * t), sm + 4 * (2 * t + 1), d);
            uint64_t off = 2 * H - 2 * (H >> (l_in + lv + 1));
#pragma unroll
            for (int i = 0; i < 4; i++) layers[4 * (off + pidx) + i] = d[i];
        }
        __syncthreads();
        if (t < active && pidx < n_l) {
#pragma unroll
            for (int i = 0; i < 4; i++) sm[4 * t + i] = d[i];
        }
        __syncthreads();
    }
}

// Levels with few parents are bound by the latency of one permutation, not
// by throughput: there one 16-lane group compresses one parent (p2x), about
// a third of the single-thread latency. Children 2p and 2p + 1 are adjacent
// digests, so lanes 0..7 load the eight input words with one access each.
__device__ __forceinline__ void compress_parent_coop(uint64_t *layers, uint64_t off_in, uint64_t off_out, uint64_t p,
                                                     bool ok, int l, const uint64_t *sc, const p2x::Lane &k) {
    uint64_t x = 0;
    if (ok && l < 8) x = __ldcg(layers + 4 * (off_in + 2 * p) + l);
    x = p2x::permute(x, l, sc, k);
    if (ok && l < 4) layers[4 * (off_out + p) + l] = p2w::canon(x);
}

// One level: parents of layer l_in + 1, one 16-lane group each.
__global__ void __launch_bounds__(128) compress_level_coop_kernel(uint64_t *layers, uint64_t H, uint32_t l_in) {
    __shared__ uint64_t sc[p2::N_PARAMS];
    p2x::stage_consts(sc);
    const int l = threadIdx.x & 15;
    const p2x::Lane k = p2x::lane_consts(sc, l);
    const uint64_t p = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const uint64_t n = H >> (l_in + 1);
    compress_parent_coop(layers, 2 * H - 2 * (H >> l_in), 2 * H - 2 * (H >> (l_in + 1)), p, p < n, l, sc, k);
}

// The same with four lanes per parent (a multiple of 32 parents).
__global__ void __launch_bounds__(128) compress_level_quad_kernel(uint64_t *layers, uint64_t H, uint32_t l_in) {
    __shared__ uint64_t sc[p2::N_PARAMS];
    p2x::stage_consts(sc);
    const int l = threadIdx.x & 3;
    const p2q::Lane k = p2q::lane_consts(sc, l);
    const uint64_t p = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 2;
    const uint64_t *in = layers + 4 * (2 * H - 2 * (H >> l_in) + 2 * p);
    uint64_t x[3] = {in[l], in[4 + l], 0};
    p2q::permute(x, sc, k);
    layers[4 * (2 * H - 2 * (H >> (l_in + 1)) + p) + l] = p2w::canon(x[0]);
}

__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// The top of a tree, layer l_in up to the root, in one launch of one
// 8-CTA cluster (128 groups; two warps per scheduler at the level of 128
// parents, which cost 4 us more in two passes of 64 groups): a level's parents
// are spread over the groups, and the hardware cluster barrier
// (release / acquire) orders one level's stores before the next level's
// loads, which read L2 (__ldcg). Warps without a parent in a pass skip it.
constexpr uint32_t kTopCtas = 8, kTopThreads = 256, kTopGroups = kTopCtas * kTopThreads / 16;
__global__ void __cluster_dims__(kTopCtas, 1, 1) __launch_bounds__(kTopThreads)
    compress_top_kernel(uint64_t *layers, uint64_t H, uint32_t l_in, uint32_t depth) {
    __shared__ uint64_t sc[p2::N_PARAMS];
    p2x::stage_consts(sc);
    const int l = threadIdx.x & 15;
    const p2x::Lane k = p2x::lane_consts(sc, l);
    const uint32_t gid = (blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    for (uint32_t lv = l_in; lv < depth; lv++) {
        const uint64_t n = H >> (lv + 1);
        const uint64_t off_in = 2 * H - 2 * (H >> lv), off_out = 2 * H - 2 * (H >> (lv + 1));
        for (uint64_t base = 0; base < n; base += kTopGroups)
            if (base + (gid & ~1u) < n)  // warp-uniform: the warp's first group has a parent
                compress_parent_coop(layers, off_in, off_out, base + gid, base + gid < n, l, sc, k);
        cluster_sync();
    }
}

// Digest layers of a tree whose layer l holds one digest c_l repeated:
// digest g (0 <= g < 2H - 1) belongs to layer l with H >> l = 2^(ceil(log2(2H - g)) - 1).
__global__ void fill_const_layers_kernel(uint64_t *layers, uint64_t H, uint32_t depth, const uint64_t *c) {
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= 2 * H - 1) return;
    const uint64_t r1 = 2 * H - g;  // >= 2
    const uint32_t lg = 64 - __clzll(r1 - 1);
    const uint32_t l = depth - (lg - 1);
#pragma unroll
    for (int k = 0; k < 4; k++) layers[4 * g + k] = c[4 * l + k];
}

}  // namespace merkle
