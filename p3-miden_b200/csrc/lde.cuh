// Coset LDE kernels: radix-8 rounds over groups of rows staged in shared
// memory, three global trips per transform of up to 2^20 rows.
//
// A matrix is h x w, row-major, one polynomial per column; h = 2^L. The
// bit positions [0, L) of a row index are split into ranges of at most 10
// bits. For a range [blo, blo + k) a block loads one group (the 2^k rows
// whose index agrees outside the range; stride 2^blo) for a tile of C
// columns, runs the k radix-2 stages of that range as rounds of up to three
// stages, and stores the group back.
//
// The LDE of a trace on s*K, |K| = h*B (p3-dft/src/traits.rs coset_lde_batch
// semantics: natural-order evaluations in, bit-reversed coset evaluations
// out) is
//   - inverse transform, decimation in time, ranges in ascending order; the
//     first range reads row bitrev_L(i) for position i, so the result is in
//     natural coefficient order (times h);
//   - for every coset c of K over H, (s*w_{hB}^c)*H: coefficient i times
//     (s*w_{hB}^c)^i / h, then a forward transform, decimation in frequency,
//     ranges in descending order, whose bit-reversed output is exactly the
//     committed layout of coset c (rows [bitrev_B(c)*h, +h)).
// The top range is the same set of rows for the last inverse range and the
// first forward range, so one kernel does both: it keeps the group's
// coefficients in shared memory and runs the forward range once per coset
// (lde_fused_kernel). A transform of L <= 10 is that kernel alone; L <= 20 is
// three launches (inverse low range, fused top range, forward low range over
// all cosets).
//
// Round arithmetic. For a round over global bits [b, b+R) and positions
// x_j = a[hi + j*2^b + l] (l = position mod 2^b), the R stages of
// decimation in frequency equal a size-2^R transform with the small root
// w_{2^R} followed by multiplying output p by t^{bitrev_R(p)},
// t = w_{2^{b+R}}^l; decimation in time is the transpose (multiply input p
// by t^{bitrev_R(p)}, then the small transform). The small roots are powers
// of two modulo p: w_8 = 2^120 = -2^24, w_4 = 2^48 (forward) and
// w_8^-1 = 2^72, w_4^-1 = -2^48 (inverse), so the small transforms cost
// shifts, not multiplications. The powers t^e of every round are built once
// per block in a shared table (2^k - 1 entries per direction).
//
// All values stay canonical (< p). Twiddles and scales are kept in Montgomery
// form (times R = 2^64): a product with one is a Montgomery product, 16
// instructions and canonical, against 26 for a canonical plain product. As
// R^3 = 1 mod p, a product of two plain table words comes into that form by
// one Montgomery product and one bare reduction (mont_of).
#pragma once
#include "gl.cuh"
#include "ntt.cuh"

namespace lde {

// a + b as a - (p - b): seven instructions against nine for add_dev (p - b
// = p when b = 0; the borrow then adds p back). add_dev stays where it is the
// faster one: the generated constraint kernels took 25.5 ms with this form,
// 18.7 with add_dev (2^18-row Keccak proof).
__device__ __forceinline__ uint64_t add(uint64_t a, uint64_t b) { return gl::sub_dev(a, gl::P - b); }
__device__ __forceinline__ uint64_t sub(uint64_t a, uint64_t b) { return gl::sub_dev(a, b); }
// a times the word whose Montgomery form is m
__device__ __forceinline__ uint64_t mul(uint64_t a, uint64_t m) { return gl::mont_mul(a, m); }
// Montgomery form of x * y: x y R^-1, then R^-1 once more (R^-2 = R)
__device__ __forceinline__ uint64_t mont_of(uint64_t x, uint64_t y) {
    const uint64_t v = gl::mont_mul(x, y);
    return gl::mont_reduce_dev((uint32_t)v, (uint32_t)(v >> 32), 0, 0);
}
// Montgomery form of a table's power
__device__ __forceinline__ uint64_t mont_at(const ntt::PowTab &t, uint64_t e) {
    return mont_of(__ldg(t.lo + (e & ((1ull << t.lo_bits) - 1))), __ldg(t.hi + (e >> t.lo_bits)));
}

// x * 2^24 mod p (canonical): (x >> 40) * 2^64 + (x << 24) reduced with
// 2^64 = eps; the last step folds the carry and the comparison with p into
// one select.
__device__ __forceinline__ uint64_t mul_2_24(uint64_t x) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    uint32_t r0, r1;
    asm("{\n\t.reg .u32 m, u0, u1, t0, t1;\n\t.reg .pred q;\n\t"
        "sub.cc.u32 u0, 0, %4;\n\t"    // h0*eps
        "subc.u32 u1, %4, 0;\n\t"
        "add.cc.u32 %0, %2, u0;\n\t"
        "addc.cc.u32 %1, %3, u1;\n\t"
        "addc.u32 m, 0, 0;\n\t"
        "add.cc.u32 t0, %0, 0xFFFFFFFF;\n\t"  // r + eps: r - p, or the value of a wrapped sum
        "addc.cc.u32 t1, %1, 0;\n\t"
        "addc.u32 m, m, 0;\n\t"
        "setp.ne.u32 q, m, 0;\n\t"
        "selp.b32 %0, t0, %0, q;\n\t"
        "selp.b32 %1, t1, %1, q;\n\t}"
        : "=&r"(r0), "=&r"(r1)
        : "r"(x0 << 24), "r"(__funnelshift_l(x0, x1, 24)), "r"(x1 >> 8));
    return ((uint64_t)r1 << 32) | r0;
}
// Divisions by 2^s, s < 64, for x < p: x - m p with m = x p^-1 mod 2^s is a
// multiple of 2^s, and (x - m p) / 2^s lies in (-p, p), so one conditional
// addition of p makes it canonical. p^-1 = 1 + 2^32 (mod 2^64).
//
// x * 2^-24 = -x * 2^72: m = x mod 2^24 = l, (x >> 24) + l 2^8 - l 2^40.
__device__ __forceinline__ uint64_t div_2_24(uint64_t x) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32), s = x0 << 8;  // l << 8
    uint32_t r0, r1;
    asm("{\n\t.reg .u32 m;\n\t"
        "add.cc.u32 %0, %2, %4;\n\t"
        "addc.u32 %1, %3, 0;\n\t"
        "sub.cc.u32 %1, %1, %4;\n\t"
        "subc.u32 m, 0, 0;\n\t"      // borrow: 0xFFFFFFFF = eps
        "sub.cc.u32 %0, %0, m;\n\t"  // + p = - eps (mod 2^64)
        "subc.u32 %1, %1, 0;\n\t}"
        : "=&r"(r0), "=&r"(r1)
        : "r"(__funnelshift_r(x0, x1, 24)), "r"(x1 >> 24), "r"(s));
    return ((uint64_t)r1 << 32) | r0;
}
// x * 2^-48 = -x * 2^48: with t = x0 + x1 (33 bits), m = (t mod 2^16) 2^32 + x0
// and the quotient is (t >> 16) + (t mod 2^16) 2^16 - m 2^16; the first two
// terms are t's low word rotated by 16 plus its carry times 2^16. 13
// instructions against 19 for x * 2^48 from its 112-bit product.
__device__ __forceinline__ uint64_t div_2_48(uint64_t x) {
    const uint32_t x0 = (uint32_t)x, x1 = (uint32_t)(x >> 32);
    uint32_t t, c, r0, r1;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, 0, 0;" : "=&r"(t), "=&r"(c) : "r"(x0), "r"(x1));
    asm("{\n\t.reg .u32 m;\n\t"
        "add.cc.u32 %0, %2, %3;\n\t"
        "addc.u32 %1, 0, 0;\n\t"
        "sub.cc.u32 %0, %0, %4;\n\t"
        "subc.cc.u32 %1, %1, %5;\n\t"
        "subc.u32 m, 0, 0;\n\t"
        "sub.cc.u32 %0, %0, m;\n\t"
        "subc.u32 %1, %1, 0;\n\t}"
        : "=&r"(r0), "=&r"(r1)
        : "r"(__funnelshift_l(t, t, 16)), "r"(c << 16), "r"(x0 << 16), "r"(__byte_perm(x0, t, 0x5432)));
    return ((uint64_t)r1 << 32) | r0;
}

__host__ __device__ constexpr uint32_t brev(uint32_t p, int R) {
    return R == 3 ? ((p & 1) << 2) | (p & 2) | ((p >> 2) & 1) : R == 2 ? ((p & 1) << 1) | ((p >> 1) & 1) : p;
}

// Size-2^R transforms with power-of-two roots. dif: natural input, output
// position p holds frequency bitrev_R(p) (forward roots). dit: input
// position p holds bitrev_R(p), natural output (inverse roots).
template <int R>
__device__ __forceinline__ void dft_dif(uint64_t *x) {
    if (R == 3) {
        const uint64_t a0 = add(x[0], x[4]), a4 = sub(x[0], x[4]);
        const uint64_t a1 = add(x[1], x[5]), a5 = mul_2_24(sub(x[5], x[1]));  // * w8 = -2^24
        const uint64_t a2 = add(x[2], x[6]), a6 = div_2_48(sub(x[6], x[2]));  // * w8^2 = 2^48
        const uint64_t a3 = add(x[3], x[7]), a7 = div_2_24(sub(x[3], x[7]));  // * w8^3 = -2^72
        const uint64_t b0 = add(a0, a2), b2 = sub(a0, a2);
        const uint64_t b1 = add(a1, a3), b3 = div_2_48(sub(a3, a1));
        const uint64_t b4 = add(a4, a6), b6 = sub(a4, a6);
        const uint64_t b5 = add(a5, a7), b7 = div_2_48(sub(a7, a5));
        x[0] = add(b0, b1), x[1] = sub(b0, b1);
        x[2] = add(b2, b3), x[3] = sub(b2, b3);
        x[4] = add(b4, b5), x[5] = sub(b4, b5);
        x[6] = add(b6, b7), x[7] = sub(b6, b7);
    } else if (R == 2) {
        const uint64_t a0 = add(x[0], x[2]), a2 = sub(x[0], x[2]);
        const uint64_t a1 = add(x[1], x[3]), a3 = div_2_48(sub(x[3], x[1]));  // * w4 = 2^48
        x[0] = add(a0, a1), x[1] = sub(a0, a1);
        x[2] = add(a2, a3), x[3] = sub(a2, a3);
    } else {
        const uint64_t a0 = add(x[0], x[1]), a1 = sub(x[0], x[1]);
        x[0] = a0, x[1] = a1;
    }
}
template <int R>
__device__ __forceinline__ void dft_dit(uint64_t *x) {
    if (R == 3) {
        const uint64_t a0 = add(x[0], x[1]), a1 = sub(x[0], x[1]);
        const uint64_t a2 = add(x[2], x[3]), a3 = sub(x[2], x[3]);
        const uint64_t a4 = add(x[4], x[5]), a5 = sub(x[4], x[5]);
        const uint64_t a6 = add(x[6], x[7]), a7 = sub(x[6], x[7]);
        uint64_t v = div_2_48(a3);  // * w4^-1 = -2^48
        const uint64_t c0 = add(a0, a2), c2 = sub(a0, a2);
        const uint64_t c1 = add(a1, v), c3 = sub(a1, v);
        v = div_2_48(a7);
        const uint64_t c4 = add(a4, a6), c6 = sub(a4, a6);
        const uint64_t c5 = add(a5, v), c7 = sub(a5, v);
        x[0] = add(c0, c4), x[4] = sub(c0, c4);
        v = div_2_24(c5);  // * w8^-1 = 2^72, negated
        x[1] = sub(c1, v), x[5] = add(c1, v);
        v = div_2_48(c6);  // * w8^-2 = -2^48
        x[2] = add(c2, v), x[6] = sub(c2, v);
        v = mul_2_24(c7);  // * w8^-3 = 2^24
        x[3] = add(c3, v), x[7] = sub(c3, v);
    } else if (R == 2) {
        const uint64_t a0 = add(x[0], x[1]), a1 = sub(x[0], x[1]);
        const uint64_t a2 = add(x[2], x[3]), a3 = sub(x[2], x[3]);
        const uint64_t v = div_2_48(a3);  // * w4^-1 = -2^48
        x[0] = add(a0, a2), x[2] = sub(a0, a2);
        x[1] = add(a1, v), x[3] = sub(a1, v);
    } else {
        const uint64_t a0 = add(x[0], x[1]), a1 = sub(x[0], x[1]);
        x[0] = a0, x[1] = a1;
    }
}

// Rounds of a k-bit range: decimation in time ascends from bit 0 in rounds
// of 3 (the last one shorter), decimation in frequency descends from bit k
// (the last one, at bit 0, shorter).
__device__ __forceinline__ void round_bits(bool dif, uint32_t k, uint32_t rd, uint32_t &q_lo, uint32_t &r) {
    if (dif) {
        const int hi = (int)k - 3 * (int)rd;
        q_lo = hi >= 3 ? hi - 3 : 0;
        r = hi - q_lo;
    } else {
        q_lo = 3 * rd;
        r = k - q_lo < 3 ? k - q_lo : 3;
    }
}

// Shared twiddle table of a k-bit range at global bit blo for a group with
// low position bits base_lo: the round at local bit q_lo with R bits
// occupies entries [2^q_lo - 1, 2^(q_lo+R) - 1); entry (l, e), e in
// [1, 2^R), is t_l^e with t_l = w_{2^(b+R)}^(base_lo + l*2^blo), b = blo + q_lo.
template <bool DIF>
__device__ void fill_table(uint64_t *T, uint32_t k, uint32_t blo, uint64_t base_lo, uint32_t L,
                           const ntt::PowTab &root, uint32_t tid, uint32_t nthreads) {
    const uint32_t nr = (k + 2) / 3;
    for (uint32_t rd = 0; rd < nr; rd++) {
        uint32_t q_lo, r;
        round_bits(DIF, k, rd, q_lo, r);
        const uint32_t em1 = (1u << r) - 1, b = blo + q_lo;
        const uint64_t emask = (1ull << (b + r)) - 1;
        uint64_t *Tr = T + ((1u << q_lo) - 1);
        for (uint32_t rel = tid; rel < (em1 << q_lo); rel += nthreads) {
            const uint32_t li = r == 3 ? rel / 7 : r == 2 ? rel / 3 : rel;
            const uint32_t e = rel - li * em1 + 1;
            const uint64_t l = base_lo + ((uint64_t)li << blo);
            Tr[rel] = mont_at(root, ((l * e) & emask) << (L - b - r));
        }
    }
}

// One round over the group in shared memory (element m of column c at
// sm[m*C + c]); T is the round's table, or null when every t is 1.
template <int C, int R, bool DIF>
__device__ __forceinline__ void round(uint64_t *sm, const uint64_t *T, uint32_t q_lo, uint32_t k, uint32_t c,
                                      uint32_t t, uint32_t TPC) {
    constexpr uint32_t E = 1u << R;
    const uint32_t tasks = (1u << k) >> R;
    const uint32_t stride = C << q_lo;
    for (uint32_t task = t; task < tasks; task += TPC) {
        const uint32_t low = task & ((1u << q_lo) - 1);
        const uint32_t mb = low | ((task >> q_lo) << (q_lo + R));
        uint64_t *px = sm + mb * C + c;
        uint64_t x[E];
#pragma unroll
        for (uint32_t j = 0; j < E; j++) x[j] = px[j * stride];
        const uint64_t *Tl = T ? T + low * (E - 1) : nullptr;
        if (!DIF && Tl) {
#pragma unroll
            for (uint32_t p = 1; p < E; p++) x[p] = mul(x[p], Tl[brev(p, R) - 1]);
        }
        if (DIF) dft_dif<R>(x);
        else dft_dit<R>(x);
        if (DIF && Tl) {
#pragma unroll
            for (uint32_t p = 1; p < E; p++) x[p] = mul(x[p], Tl[brev(p, R) - 1]);
        }
#pragma unroll
        for (uint32_t j = 0; j < E; j++) px[j * stride] = x[j];
    }
}

// All rounds of a k-bit range; every round ends with a block barrier.
// tw_low: whether the round at bit 0 has a nontrivial table (base_lo != 0).
template <int C, bool DIF>
__device__ __forceinline__ void run_rounds(uint64_t *sm, const uint64_t *T, bool tw_low, uint32_t k, uint32_t c,
                                           uint32_t t, uint32_t TPC) {
    const uint32_t nr = (k + 2) / 3;
    for (uint32_t rd = 0; rd < nr; rd++) {
        uint32_t q_lo, r;
        round_bits(DIF, k, rd, q_lo, r);
        const uint64_t *Tr = (q_lo == 0 && !tw_low) ? nullptr : T + ((1u << q_lo) - 1);
        if (r == 3) round<C, 3, DIF>(sm, Tr, q_lo, k, c, t, TPC);
        else if (r == 2) round<C, 2, DIF>(sm, Tr, q_lo, k, c, t, TPC);
        else round<C, 1, DIF>(sm, Tr, q_lo, k, c, t, TPC);
        __syncthreads();
    }
}

struct PassArgs {
    const uint64_t *src;
    uint64_t *dst;
    uint64_t ld_src, ld_dst;      // row strides in words
    uint64_t src_blk, dst_blk;    // words between the blocks of blockIdx.y (cosets of forward passes)
    uint64_t w;                   // columns
    uint32_t L, blo, k;           // transform size 2^L; range [blo, blo + k)
    uint32_t n_tiles;             // column tiles; blockIdx.x = group * n_tiles + tile
    uint32_t tile_step;           // tile kernels: blocks per group; blockIdx.x = group * tile_step + first tile
    uint32_t src_bitrev;          // position i is read from row bitrev_L(i)
    ntt::PowTab root;             // powers of w_h (forward) or w_h^-1 (inverse)
};

struct FusedArgs {
    const uint64_t *src;
    uint64_t *dst;
    uint64_t ld_src, ld_dst;
    uint64_t w;
    uint32_t L, blo, k, n_tiles, tile_step, src_bitrev;
    uint32_t log_cosets;          // B = 2^log_cosets output cosets of h rows each
    ntt::PowTab inv_root, fwd_root;
    ntt::PowTab coset_root;       // powers of w_{hB} (tile kernel)
    // scale of coset c: coefficient i times scale_lo[c*2^lo_bits + (i mod 2^lo_bits)] *
    // scale_hi[c*scale_hi_len + (i >> lo_bits)] = (s*w_{hB}^c)^i / h
    const uint64_t *scale_lo, *scale_hi;
    uint32_t scale_lo_bits;
    uint64_t scale_hi_len;
    // optional per-column factor: coefficient i of column col times
    // colpow(col/2)^i (quotient chunks); null when absent
    const uint64_t *cp_lo, *cp_hi;
    uint32_t cp_lo_bits;
    uint64_t cp_hi_len;
};

__device__ __forceinline__ void group_of(uint64_t g, uint32_t blo, uint32_t k, uint64_t &base, uint64_t &base_lo) {
    const uint64_t S = 1ull << blo;
    base = (g & (S - 1)) | ((g >> blo) << (blo + k));
    base_lo = base & (S - 1);
}

// One range of the inverse (DIF = false) or forward (DIF = true) transform,
// any bit count: narrow matrices (C < 8) and ranges of fewer than
// kTileMinBits bits.
template <int C, bool DIF>
__global__ void __launch_bounds__(1024) lde_pass_kernel(const __grid_constant__ PassArgs a) {
    extern __shared__ uint64_t sm[];
    const uint32_t kk = a.k;
    const uint32_t G = 1u << kk;
    uint64_t *T = sm + (size_t)G * C;
    const uint32_t tile = blockIdx.x % a.n_tiles;
    uint64_t base, base_lo;
    group_of(blockIdx.x / a.n_tiles, a.blo, kk, base, base_lo);
    const uint64_t col0 = (uint64_t)tile * C;
    const uint32_t tid = threadIdx.x, c = tid % C, t = tid / C, TPC = blockDim.x / C;
    const bool col_ok = col0 + c < a.w;
    const uint64_t *src = a.src + blockIdx.y * a.src_blk + col0 + c;
    uint64_t *dst = a.dst + blockIdx.y * a.dst_blk + col0 + c;
    for (uint32_t m = t; m < G; m += TPC) {
        const uint64_t P = base + ((uint64_t)m << a.blo);
        const uint64_t row = a.src_bitrev ? gl::bitrev(P, a.L) : P;
        sm[m * C + c] = col_ok ? __ldg(src + row * a.ld_src) : 0;
    }
    fill_table<DIF>(T, kk, a.blo, base_lo, a.L, a.root, tid, blockDim.x);
    __syncthreads();
    run_rounds<C, DIF>(sm, T, base_lo != 0, kk, c, t, TPC);
    if (!col_ok) return;
    for (uint32_t m = t; m < G; m += TPC) {
        const uint64_t P = base + ((uint64_t)m << a.blo);
        dst[P * a.ld_dst] = sm[m * C + c];
    }
}

// The top range: inverse rounds, then per coset the scale and the forward
// rounds, written to the coset's block of the output.
template <int C>
__global__ void __launch_bounds__(1024) lde_fused_kernel(const __grid_constant__ FusedArgs a) {
    extern __shared__ uint64_t sm[];
    const uint32_t kk = a.k;
    const uint32_t G = 1u << kk;
    uint64_t *A = sm, *Bf = A + (size_t)G * C, *Ti = Bf + (size_t)G * C, *Tf = Ti + G, *sc = Tf + G;
    const uint32_t tile = blockIdx.x % a.n_tiles;
    uint64_t base, base_lo;
    group_of(blockIdx.x / a.n_tiles, a.blo, kk, base, base_lo);
    const uint64_t col0 = (uint64_t)tile * C;
    const uint32_t tid = threadIdx.x, c = tid % C, t = tid / C, TPC = blockDim.x / C;
    const uint64_t col = col0 + c;
    const bool col_ok = col < a.w;
    for (uint32_t m = t; m < G; m += TPC) {
        const uint64_t P = base + ((uint64_t)m << a.blo);
        const uint64_t row = a.src_bitrev ? gl::bitrev(P, a.L) : P;
        A[m * C + c] = col_ok ? __ldg(a.src + row * a.ld_src + col) : 0;
    }
    fill_table<false>(Ti, kk, a.blo, base_lo, a.L, a.inv_root, tid, blockDim.x);
    fill_table<true>(Tf, kk, a.blo, base_lo, a.L, a.fwd_root, tid, blockDim.x);
    __syncthreads();
    run_rounds<C, false>(A, Ti, base_lo != 0, kk, c, t, TPC);
    const uint64_t h = 1ull << a.L;
    const uint32_t B = 1u << a.log_cosets;
    const uint64_t lo_mask = (1ull << a.scale_lo_bits) - 1;
    for (uint32_t cs = 0; cs < B; cs++) {
        const uint64_t *slo = a.scale_lo + ((uint64_t)cs << a.scale_lo_bits);
        const uint64_t *shi = a.scale_hi + cs * a.scale_hi_len;
        for (uint32_t m = tid; m < G; m += blockDim.x) {
            const uint64_t P = base + ((uint64_t)m << a.blo);
            sc[m] = mont_of(__ldg(slo + (P & lo_mask)), __ldg(shi + (P >> a.scale_lo_bits)));
        }
        __syncthreads();
        for (uint32_t m = t; m < G; m += TPC) {
            uint64_t v = mul(A[m * C + c], sc[m]);
            if (a.cp_lo && col_ok) {
                const uint64_t P = base + ((uint64_t)m << a.blo), tc = col / 2;
                v = mul(v, mont_of(__ldg(a.cp_lo + (tc << a.cp_lo_bits) + (P & ((1ull << a.cp_lo_bits) - 1))),
                                   __ldg(a.cp_hi + tc * a.cp_hi_len + (P >> a.cp_lo_bits))));
            }
            Bf[m * C + c] = v;
        }
        __syncthreads();
        run_rounds<C, true>(Bf, Tf, base_lo != 0, kk, c, t, TPC);
        if (col_ok) {
            uint64_t *dst = a.dst + (uint64_t)gl::bitrev(cs, a.log_cosets) * h * a.ld_dst + col;
            for (uint32_t m = t; m < G; m += TPC) {
                const uint64_t P = base + ((uint64_t)m << a.blo);
                dst[P * a.ld_dst] = Bf[m * C + c];
            }
        }
        // the next coset writes sc (not read by the stores) and, after a
        // barrier, Bf
    }
}

// ---------------------------------------------------------- tile kernels
// The same two kernels for 8-column tiles and a bit count fixed at compile
// time, bound by the integer pipes. A thread keeps its 8 elements of a column
// in registers from global memory through the first round and from the last
// round to global memory; only the rounds between go through shared memory
// (two exchanges for 7..9 bits instead of four), and all index arithmetic is
// compile-time offsets from a few pointers. A block takes several column
// tiles of its group, so the twiddle table is built once for them.
// The fused kernel holds the coefficients in registers: the last inverse
// round and the first forward round work on the same elements
// (t + j * 2^(k-3)), and coset c's scale (s w_{hB}^c)^i / h is the previous
// one's times w_{hB}^i, one product per element and coset from one table.
// Measured (B200): 2^18 x 336, blowup 2, 5.55 -> 3.53 ms; 2^20 x 37, blowup
// 8, 9.57 -> 6.0 ms, with the ALU pipe at 76..79 % of its peak.
constexpr int kTileMinBits = 5;

// Element m of column c: rows are paired into 128-byte lines, and the half a
// row takes is the parity of its low four bits, so that the two rows a
// half-warp touches in any round lie in different halves.
__device__ __forceinline__ uint32_t row_parity(uint32_t m) { return __popc(m & 15) & 1; }
__host__ __device__ constexpr uint32_t cparity(uint32_t m) { return (m ^ (m >> 1) ^ (m >> 2) ^ (m >> 3)) & 1; }

template <int KT, bool DIF, int RD>
struct Round {
    static constexpr int NR = (KT + 2) / 3;
    static constexpr int HI = KT - 3 * RD;
    static constexpr int Q = DIF ? (HI >= 3 ? HI - 3 : 0) : 3 * RD;
    static constexpr int R = DIF ? HI - Q : (KT - Q < 3 ? KT - Q : 3);
    static constexpr int E = 1 << R, N = 8 >> R;  // elements of a task, tasks of a thread
    static constexpr uint32_t TPC = 1u << (KT - 3);
    // first element of task i of thread t
    static __device__ __forceinline__ uint32_t first(uint32_t t, int i) {
        const uint32_t task = t + i * TPC, low = task & ((1u << Q) - 1);
        return low | ((task >> Q) << (Q + R));
    }
    // v[i * E + e] = element first(t, i) + e * 2^Q
    template <bool LOAD>
    static __device__ __forceinline__ void exchange(uint64_t *sm, uint64_t *v, uint32_t t, uint32_t c) {
#pragma unroll
        for (int i = 0; i < N; i++) {
            const uint32_t m = first(t, i), par = row_parity(m);
            uint64_t *line = sm + (m >> 1) * 16 + c, *h0 = line + par * 8, *h1 = line + 8 - par * 8;
#pragma unroll
            for (int e = 0; e < E; e++) {
                uint64_t *p = (cparity((e << Q) & 15) ? h1 : h0) + ((e << Q) >> 1) * 16;
                if (LOAD) v[i * E + e] = *p;
                else *p = v[i * E + e];
            }
        }
    }
    // T: the range's table; tw_low: whether the round at bit 0 has twiddles
    static __device__ __forceinline__ void run(uint64_t *v, const uint64_t *T, bool tw_low, uint32_t t) {
        const uint64_t *Tr = T + ((1u << Q) - 1);
#pragma unroll
        for (int i = 0; i < N; i++) {
            uint64_t *x = v + i * E;
            const uint64_t *Tl = Tr + ((t + i * TPC) & ((1u << Q) - 1)) * (E - 1);
            if (!DIF && (Q != 0 || tw_low)) {
#pragma unroll
                for (int p = 1; p < E; p++) x[p] = mul(x[p], Tl[brev(p, R) - 1]);
            }
            if (DIF) dft_dif<R>(x);
            else dft_dit<R>(x);
            if (DIF && (Q != 0 || tw_low)) {
#pragma unroll
                for (int p = 1; p < E; p++) x[p] = mul(x[p], Tl[brev(p, R) - 1]);
            }
        }
    }
};
// Rounds RD.. of a range: on entry v holds the inputs of round RD in its
// order, on return the outputs of the last round in that one's order.
template <int KT, bool DIF, int RD = 0>
__device__ __forceinline__ void tile_rounds(uint64_t *sm, const uint64_t *T, bool tw_low, uint64_t *v, uint32_t t,
                                            uint32_t c) {
    using Rd = Round<KT, DIF, RD>;
    Rd::run(v, T, tw_low, t);
    if constexpr (RD + 1 < Rd::NR) {
        Rd::template exchange<false>(sm, v, t, c);
        __syncthreads();
        Round<KT, DIF, RD + 1>::template exchange<true>(sm, v, t, c);
        tile_rounds<KT, DIF, RD + 1>(sm, T, tw_low, v, t, c);
    }
}

// 1536 resident threads per SM (at most 40 registers; 1024 threads with 62
// registers measured 4 % slower on 2^18 x 2633); the fused kernel, with the
// coefficients in registers, keeps 1024.
template <bool DIF, int KT>
__global__ void __launch_bounds__(1 << KT, 1536 >> KT) lde_pass_tile_kernel(const __grid_constant__ PassArgs a) {
    extern __shared__ uint64_t sm[];
    constexpr uint32_t G = 1u << KT;
    uint64_t *T = sm + (size_t)G * 8;
    using First = Round<KT, DIF, 0>;
    using Last = Round<KT, DIF, First::NR - 1>;
    const uint32_t group = blockIdx.x / a.tile_step;
    uint64_t base, base_lo;
    group_of(group, a.blo, KT, base, base_lo);
    const uint32_t c = threadIdx.x % 8, t = threadIdx.x / 8;
    fill_table<DIF>(T, KT, a.blo, base_lo, a.L, a.root, threadIdx.x, G);
    const uint64_t *src = a.src + blockIdx.y * a.src_blk + c;
    uint64_t *dst = a.dst + blockIdx.y * a.dst_blk + c;
    for (uint32_t tile = blockIdx.x % a.tile_step; tile < a.n_tiles; tile += a.tile_step) {
        const uint64_t col0 = (uint64_t)tile * 8;
        const bool col_ok = col0 + c < a.w;
        uint64_t v[8];
#pragma unroll
        for (int i = 0; i < First::N; i++) {
            // rows of the task, ascending; read in bit-reversed order, bit b
            // of e in the position is bit L - 1 - blo - Q - b of the row
            const uint64_t pos = base + ((uint64_t)First::first(t, i) << a.blo);
            const uint64_t *p = src + (a.src_bitrev ? gl::bitrev(pos, a.L) : pos) * a.ld_src + col0;
            const uint64_t step = a.ld_src << (a.src_bitrev ? a.L - a.blo - First::Q - First::R : a.blo + First::Q);
            uint64_t x[First::E];
#pragma unroll
            for (int e = 0; e < First::E; e++) x[e] = col_ok ? __ldg(p + e * step) : 0;
#pragma unroll
            for (int e = 0; e < First::E; e++) v[i * First::E + e] = a.src_bitrev ? x[brev(e, First::R)] : x[e];
        }
        __syncthreads();  // the table; the last tile's reads
        tile_rounds<KT, DIF>(sm, T, base_lo != 0, v, t, c);
        if (col_ok) {
#pragma unroll
            for (int i = 0; i < Last::N; i++) {
                uint64_t *p = dst + (base + ((uint64_t)Last::first(t, i) << a.blo)) * a.ld_dst + col0;
                const uint64_t step = a.ld_dst << (a.blo + Last::Q);
#pragma unroll
                for (int e = 0; e < Last::E; e++) p[e * step] = v[i * Last::E + e];
            }
        }
    }
}

template <int KT>
__global__ void __launch_bounds__(1 << KT, 1024 >> KT) lde_fused_tile_kernel(const __grid_constant__ FusedArgs a) {
    extern __shared__ uint64_t sm[];
    constexpr uint32_t G = 1u << KT, TPC = G / 8;
    uint64_t *Ti = sm + (size_t)G * 8, *Tf = Ti + G, *s0 = Tf + G, *om = s0 + G;
    using First = Round<KT, false, 0>;
    using LastI = Round<KT, false, First::NR - 1>;
    using LastF = Round<KT, true, First::NR - 1>;
    const uint32_t group = blockIdx.x / a.tile_step;
    uint64_t base, base_lo;
    group_of(group, a.blo, KT, base, base_lo);
    const uint32_t c = threadIdx.x % 8, t = threadIdx.x / 8;
    fill_table<false>(Ti, KT, a.blo, base_lo, a.L, a.inv_root, threadIdx.x, G);
    fill_table<true>(Tf, KT, a.blo, base_lo, a.L, a.fwd_root, threadIdx.x, G);
    const uint64_t h = 1ull << a.L;
    const uint32_t B = 1u << a.log_cosets;
    {
        // coset 0's scale s^i / h and the step to the next coset's, w_{hB}^i
        const uint32_t m = threadIdx.x;
        const uint64_t pos = base + ((uint64_t)m << a.blo), lo = pos & ((1ull << a.scale_lo_bits) - 1),
                       hi = pos >> a.scale_lo_bits;
        s0[m] = mont_of(__ldg(a.scale_lo + lo), __ldg(a.scale_hi + hi));
        om[m] = mont_at(a.coset_root, pos);
    }
    for (uint32_t tile = blockIdx.x % a.tile_step; tile < a.n_tiles; tile += a.tile_step) {
        const uint64_t col = (uint64_t)tile * 8 + c;
        const bool col_ok = col < a.w;
        uint64_t v[8], x[8];
#pragma unroll
        for (int i = 0; i < First::N; i++) {
            const uint64_t pos = base + ((uint64_t)First::first(t, i) << a.blo);
            const uint64_t *p = a.src + (a.src_bitrev ? gl::bitrev(pos, a.L) : pos) * a.ld_src + col;
            const uint64_t step = a.ld_src << (a.src_bitrev ? a.L - a.blo - First::Q - First::R : a.blo + First::Q);
#pragma unroll
            for (int e = 0; e < First::E; e++) x[i * First::E + e] = col_ok ? __ldg(p + e * step) : 0;
#pragma unroll
            for (int e = 0; e < First::E; e++)
                v[i * First::E + e] = a.src_bitrev ? x[i * First::E + brev(e, First::R)] : x[i * First::E + e];
        }
        __syncthreads();  // the tables; the last tile's reads
        tile_rounds<KT, false>(sm, Ti, base_lo != 0, v, t, c);
        // v[i * E + e] is element t + (i + e * N) * TPC
#pragma unroll
        for (int i = 0; i < LastI::N; i++)
#pragma unroll
            for (int e = 0; e < LastI::E; e++) x[i + e * LastI::N] = v[i * LastI::E + e];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = mul(x[j], s0[t + j * TPC]);
        if (a.cp_lo && col_ok) {
            const uint64_t tc = col / 2;
            const uint64_t *clo = a.cp_lo + (tc << a.cp_lo_bits), *chi = a.cp_hi + tc * a.cp_hi_len;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint64_t pos = base + ((uint64_t)(t + j * TPC) << a.blo);
                x[j] = mul(x[j], mont_of(__ldg(clo + (pos & ((1ull << a.cp_lo_bits) - 1))),
                                         __ldg(chi + (pos >> a.cp_lo_bits))));
            }
        }
#pragma unroll 1
        for (uint32_t cs = 0; cs < B; cs++) {
#pragma unroll
            for (int j = 0; j < 8; j++) v[j] = x[j];
            __syncthreads();  // the last round's reads
            tile_rounds<KT, true>(sm, Tf, base_lo != 0, v, t, c);
            if (col_ok) {
                uint64_t *dst = a.dst + (uint64_t)gl::bitrev(cs, a.log_cosets) * h * a.ld_dst + col;
#pragma unroll
                for (int i = 0; i < LastF::N; i++) {
                    uint64_t *p = dst + (base + ((uint64_t)LastF::first(t, i) << a.blo)) * a.ld_dst;
                    const uint64_t step = a.ld_dst << (a.blo + LastF::Q);
#pragma unroll
                    for (int e = 0; e < LastF::E; e++) p[e * step] = v[i * LastF::E + e];
                }
            }
            if (cs + 1 < B) {
#pragma unroll
                for (int j = 0; j < 8; j++) x[j] = mul(x[j], om[t + j * TPC]);
            }
        }
    }
}

}  // namespace lde
