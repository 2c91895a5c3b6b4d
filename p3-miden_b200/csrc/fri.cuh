// FRI commit-phase kernels (p3-miden-lifted-fri/src/fri/prover.rs:190-292,
// fri/fold/arity{2,4,8}.rs) and the proof-of-work grind.
//
// Round r commits the evaluations (bit-reversed, n_r EF) as an
// (n_r/a) x 2a base matrix (EF flattened), one leaf per row, unaligned
// tree. Folding row k (the coset s*<w_a>, s = w_{n_r}^{bitrev(k)}) with
// challenge beta gives (1/a) sum_j (beta/s)^j sum_t y_t w_a^{-jt}, where the
// row holds y_t at position bitrev_{log a}(t).
//
// The fold of round r is fused with the leaf hash of round r+1: one thread
// folds a consecutive rows, stores the a folded values and hashes them as
// one leaf of the next tree.
#pragma once
#include "gl.cuh"
#include "lde.cuh"
#include "merkle.cuh"
#include "ntt.cuh"

namespace fri {

__device__ __forceinline__ uint64_t merkle_shfl(uint64_t v, int src) { return p2x::shfl64(v, src); }

struct FoldArgs {
    const uint64_t *in;  // n_in EF
    uint64_t n_out;      // n_in / a
    uint32_t log_a;
    uint32_t log_nin;     // log2 n_in
    uint32_t log_n0;      // log2 of the root of the s_inv table
    ntt::PowTab w0inv;    // powers of w_{n0}^{-1}
    gl::ef beta;
    const uint64_t *beta_dev;  // if set, the challenge is read from here (device-side transcript)
    uint64_t inv_a;       // 1/a
    uint64_t *out;        // n_out EF
    uint64_t *digests;    // (n_out / a) digests of the next round, or null
};

// Output k. The row holds y_t at bit-reversed positions, so the sums over t
// are one decimation-in-time transform of each coordinate with the inverse
// small roots (powers of two, lde.cuh): u_j = sum_t y_t w_a^{-jt}; then
// Horner in beta/s. At arity 4 that is 8 sums and a shift per coordinate in
// place of 16 products.
template <int LA>
__device__ __forceinline__ gl::ef fold_one(const FoldArgs &a, gl::ef beta, uint64_t k) {
    constexpr int A = 1 << LA;
    // s_inv = w_{n_in}^{-bitrev_{log n_out}(k)} = w_{n0}^{-(bitrev << (log n0 - log n_in))}
    const uint64_t e = gl::bitrev(k, a.log_nin - LA) << (a.log_n0 - a.log_nin);
    const uint64_t *row = a.in + 2 * k * A;
    uint64_t y0[A], y1[A];
#pragma unroll
    for (int p = 0; p < A; p++) y0[p] = row[2 * p], y1[p] = row[2 * p + 1];
    const gl::ef x = gl::ef_mulf(beta, a.w0inv.at(e));
    lde::dft_dit<LA>(y0);
    lde::dft_dit<LA>(y1);
    gl::ef r{y0[A - 1], y1[A - 1]};
#pragma unroll
    for (int j = A - 2; j >= 0; j--) r = gl::ef_add(gl::ef_mul(r, x), gl::ef{y0[j], y1[j]});
    return gl::ef_mulf(r, a.inv_a);
}
__device__ __forceinline__ gl::ef fold_any(const FoldArgs &a, gl::ef beta, uint64_t k) {
    return a.log_a == 1 ? fold_one<1>(a, beta, k) : a.log_a == 2 ? fold_one<2>(a, beta, k) : fold_one<3>(a, beta, k);
}

// The fold alone, one thread per output (2^20 values at arity 4: 44 us with
// the row sums as products and four outputs per thread). Bound by latency and
// launch below about 2^20 values, by the integer pipes above.
template <int LA>
__global__ void __launch_bounds__(128) fold_kernel(const __grid_constant__ FoldArgs a) {
    const uint64_t k = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= a.n_out) return;
    const gl::ef v = fold_one<LA>(a, a.beta, k);
    a.out[2 * k] = v.c0;
    a.out[2 * k + 1] = v.c1;
}

// thread g folds outputs [g*a, g*a + a)
__global__ void __launch_bounds__(128) fold_hash_kernel(const __grid_constant__ FoldArgs a) {
    const uint32_t A = 1u << a.log_a;
    const uint64_t g = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g * A >= a.n_out) return;
    uint64_t buf[16];
    const uint32_t cnt = (uint32_t)((a.n_out - g * A) < A ? (a.n_out - g * A) : A);
    const gl::ef beta = a.beta_dev ? gl::ef{a.beta_dev[0], a.beta_dev[1]} : a.beta;
    for (uint32_t u = 0; u < cnt; u++) {
        gl::ef v = fold_any(a, beta, g * A + u);
        a.out[2 * (g * A + u)] = v.c0;
        a.out[2 * (g * A + u) + 1] = v.c1;
        buf[2 * u] = v.c0;
        buf[2 * u + 1] = v.c1;
    }
    if (a.digests && cnt == A) {
        uint64_t s[12];
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = 0;
        const uint32_t W = 2 * A;
        for (uint32_t i = 0; i < W; i += 8) {
#pragma unroll
            for (uint32_t j = 0; j < 8; j++) s[j] = (i + j < W) ? buf[i + j] : 0;
            p2_permute_dev(s);
        }
#pragma unroll
        for (int i = 0; i < 4; i++) a.digests[4 * g + i] = p2w::canon(s[i]);
    }
}

// Device copy of the host Challenger (transcript.cuh) for the FRI commit
// loop: the same observe / sample / duplex rules on canonical words, so the
// state read back after the loop continues the host transcript unchanged.
struct DevCh {
    uint64_t state[12], in[8], out[8];
    int32_t n_in, n_out;
    int32_t err;  // a grind witness was missing or did not satisfy its bits
};
// Warp-cooperative challenger: the DevCh is staged in shared memory beside the
// constant table (stage_consts, by the whole block), both 16-lane groups of
// the warp run the duplex permutation (p2x; the second group duplicates the
// first), group 0 writes the state back and lane 0 does the counters. The
// observe / sample / duplex rules are the host Challenger's.
struct WarpChShared {
    DevCh c;
    uint64_t sc[p2::N_PARAMS];
};
struct WarpCh {
    WarpChShared &s;
    p2x::Lane k;
    int l;
    __device__ __forceinline__ WarpCh(WarpChShared &sh, const DevCh *g) : s(sh), l(threadIdx.x & 15) {
        const uint32_t *src = (const uint32_t *)g;
        uint32_t *dst = (uint32_t *)&s.c;
        for (uint32_t i = threadIdx.x; i < sizeof(DevCh) / 4; i += 32) dst[i] = src[i];
        __syncwarp();
        k = p2x::lane_consts(s.sc, l);
    }
    __device__ __forceinline__ void duplex() {
        __syncwarp();
        uint64_t x = 0;
        if (l < 12) x = l < s.c.n_in ? s.c.in[l] : s.c.state[l];
        x = p2w::canon(p2x::permute(x, l, s.sc, k));
        __syncwarp();
        if (threadIdx.x < 12) s.c.state[l] = x;
        if (threadIdx.x < 8) s.c.out[l] = x;
        if (threadIdx.x == 0) s.c.n_in = 0, s.c.n_out = 8;
        __syncwarp();
    }
    __device__ __forceinline__ void observe(uint64_t x) {
        __syncwarp();
        if (threadIdx.x == 0) s.c.n_out = 0, s.c.in[s.c.n_in++] = x;
        __syncwarp();
        if (s.c.n_in == 8) duplex();
    }
    __device__ __forceinline__ uint64_t sample() {
        __syncwarp();
        if (s.c.n_in > 0 || s.c.n_out == 0) duplex();
        const uint64_t v = s.c.out[s.c.n_out - 1];
        __syncwarp();
        if (threadIdx.x == 0) s.c.n_out--;
        __syncwarp();
        return v;
    }
};
// A round of the commit loop between the layer's root and its fold:
// send_commit(root), grind(bits) with the witness found by grind_kernel, and
// the folding challenge. What the transcript records is left in the logs.
struct RoundArgs {
    const DevCh *ch;  // at the start of the round
    DevCh *next;      // and at its end: another slot, as every block reads ch
    const uint64_t *root;
    uint32_t bits;
    const unsigned long long *found;
    uint64_t *log_root, *log_w;
    uint64_t *beta;
};
// By one warp; `writes`: this warp stores the results.
__device__ __forceinline__ gl::ef round_beta(WarpChShared &sh, const RoundArgs &a, bool writes) {
    // all loads first: each would wait for memory on its own
    uint64_t root[4], x = a.bits ? *a.found : 0;
#pragma unroll
    for (int i = 0; i < 4; i++) root[i] = a.root[i];
    WarpCh w(sh, a.ch);
    writes = writes && threadIdx.x == 0;
#pragma unroll
    for (int i = 0; i < 4; i++) {
        if (writes) a.log_root[i] = root[i];
        w.observe(root[i]);
    }
    if (a.bits == 0) {
        if (writes) *a.log_w = 0;
    } else {
        if (x == ~0ull) {
            if (threadIdx.x == 0) sh.c.err = 1;
            x = 0;
        }
        if (writes) *a.log_w = x;
        w.observe(x);
        if ((w.sample() & ((1ull << a.bits) - 1)) != 0 && threadIdx.x == 0) sh.c.err = 1;
    }
    gl::ef beta;
    beta.c0 = w.sample();
    beta.c1 = w.sample();
    if (writes) {
        a.beta[0] = beta.c0, a.beta[1] = beta.c1;
        *a.next = sh.c;
    }
    return beta;
}
__global__ void __launch_bounds__(32) fri_round_kernel(const __grid_constant__ RoundArgs a) {
    __shared__ WarpChShared sh;
    p2x::stage_consts(sh.sc);
    round_beta(sh, a, true);
}

// The same fold and leaf hash with one 16-lane group per leaf, for rounds
// with few leaves (latency-bound): lane u < a folds output g*a + u, the leaf
// words (output i >> 1, component i & 1) are gathered by shuffles, and the
// group absorbs them (overwrite mode, zero-padded 8-word chunks) with the
// cooperative permutation. Every block's first warp runs the round's challenger
// itself, which costs no more than a kernel for it would and spares two
// launches a round (commit phase of 10 / 17 rounds: 1.66 -> 1.55 / 4.62 ->
// 4.45 ms).
__global__ void __launch_bounds__(128) fold_hash_coop_kernel(const __grid_constant__ FoldArgs a,
                                                             const __grid_constant__ RoundArgs r) {
    __shared__ WarpChShared sh;
    __shared__ gl::ef beta_sh;
    const uint64_t *sc = sh.sc;
    p2x::stage_consts(sh.sc);
    if (threadIdx.x < 32) {
        const gl::ef b = round_beta(sh, r, blockIdx.x == 0);
        if (threadIdx.x == 0) beta_sh = b;
    }
    __syncthreads();
    const gl::ef beta = beta_sh;
    const int l = threadIdx.x & 15;
    const p2x::Lane k = p2x::lane_consts(sc, l);
    const uint32_t A = 1u << a.log_a;
    const uint64_t g = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 4;
    const bool ok = g * A < a.n_out;
    const uint32_t cnt = ok ? (uint32_t)((a.n_out - g * A) < A ? (a.n_out - g * A) : A) : 0;
    uint64_t c0 = 0, c1 = 0;
    if ((uint32_t)l < cnt) {
        const gl::ef v = fold_any(a, beta, g * A + l);
        a.out[2 * (g * A + l)] = v.c0;
        a.out[2 * (g * A + l) + 1] = v.c1;
        c0 = v.c0, c1 = v.c1;
    }
    if (!a.digests) return;  // uniform over the grid
    const uint32_t W = 2 * A;
    uint64_t x = 0;
    for (uint32_t i = 0; i < W; i += 8) {
        const uint32_t idx = i + (l & 7);
        const uint64_t w0 = merkle_shfl(c0, (int)(idx >> 1) & 15), w1 = merkle_shfl(c1, (int)(idx >> 1) & 15);
        if (l < 8) x = idx < W ? ((idx & 1) ? w1 : w0) : 0;
        x = p2x::permute(x, l, sc, k);
    }
    if (cnt == A && l < 4) a.digests[4 * g + l] = p2w::canon(x);
}

// Proof-of-work search over witnesses [base, base + count): the challenger
// with `n_pending` buffered inputs observes w and samples; success when the
// sampled word (state[7] after the duplex) has its low `bits` bits zero.
struct GrindArgs {
    uint64_t state[12];
    uint64_t pending[8];
    uint32_t n_pending;
    uint32_t bits;
    uint64_t base;
    uint64_t count;
    unsigned long long *found;  // atomicMin target, initialised to ~0
    const DevCh *ch;            // if set, the state is read from this device challenger, which has no pending input
    const uint64_t *root;       // (challenges were sampled last) before the four words of this root
};
// A witness below every one this thread could still find is there: the word
// is asked for a round ahead of its use (it lies in L2).
struct WitnessFound {
    const volatile unsigned long long *found;
    uint64_t w, seen;
    __device__ __forceinline__ bool operator()() {
        const bool stop = w >= seen;
        seen = *found;
        return stop;
    }
};
// Candidates are tried in order, a grid's worth at a time, so that the least
// witness is found. Bound by the latency of a permutation and its integer
// pipes. Two blocks per SM while a search is a few turns: a turn of 38 k
// candidates takes 36 us, and more blocks try more candidates past the least
// witness (16 bits, mean of 300 states with the call: 1 / 2 / 3 / 4 / 8 blocks
// 133 / 109 / 115 / 125 / 158 us; 130 us with two when a turn begun beside the
// find ran to its end). A long search is bound by the pipes, which two blocks
// do not fill: 21 / 22 / 23 / 24 / 26 bits take 2.22 / 4.22 / 9.43 / 12.8 / 80.3
// ms with two and 2.29 / 3.99 / 8.34 / 11.1 / 67.9 with eight.
inline unsigned grind_grid(uint32_t bits) { return 148 * (bits < 22 ? 2 : 8); }
__global__ void __launch_bounds__(128) grind_kernel(const __grid_constant__ GrindArgs a) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    const uint64_t mask = (1ull << a.bits) - 1;
    WitnessFound stop{a.found, 0, ~0ull};
    for (uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; t < a.count; t += stride) {
        const uint64_t w = a.base + t;
        stop.w = w;
        if (stop()) return;
        uint64_t s[12];
        if (a.ch) {
#pragma unroll
            for (int i = 0; i < 12; i++) s[i] = i < 4 ? a.root[i] : i == 4 ? w : a.ch->state[i];
        } else {
#pragma unroll
            for (int i = 0; i < 12; i++) s[i] = a.state[i];
            for (uint32_t i = 0; i < a.n_pending; i++) s[i] = a.pending[i];
            s[a.n_pending] = w;
        }
        p2_permute_until(s, stop);  // stopped: the state is noise, but w is above the found one
        if ((p2w::canon(s[7]) & mask) == 0) atomicMin(a.found, (unsigned long long)w);
    }
}

}  // namespace fri
