// DEEP quotient kernels (p3-miden-lifted-fri/src/deep/{interpolate,prover}.rs).
//
//  q[i][j] = 1 / (z_j - x_i) for the bit-reversed coset points
//  x_i = g * w_n^{bitrev(i)} of gK, j in {0, 1}: chunked Montgomery batch
//  inversion (one EF inversion per CHUNK points per thread).
//
//  OOD evaluation of a committed matrix of LDE height h_m (trace degree
//  d_m = h_m / B) at z_j^{n/h_m}: f = s_j * sum_{i < d_m} W_{d_m}[i][j] * M[i],
//  with W_d[i][j] = x_i q[i][j] for the top degree and smaller degrees folded
//  by summing consecutive blocks (interpolate.rs:123-201).
//
//  DEEP polynomial: Q(x_i) = sum_j beta^j q[i][j] (f_red(z_j) - f_red(x_i))
//  with f_red(x_i) = sum_m dot(coef_m, M_m[i >> lift_m])
//  (deep/prover.rs:304-405).
#pragma once
#include "gl.cuh"
#include "ntt.cuh"

namespace deep {

constexpr int CHUNK = 8;

struct PQArgs {
    uint64_t n;
    uint32_t log_n;
    ntt::PowTab wn;  // powers of w_n
    gl::ef z[2];
    uint64_t *q;  // n x 2 EF
};

// 1 / (z - x) = (z - x)^conj / N(z - x) with the norm N = (z_0 - x)^2 - 7 z_1^2
// in the base field, so the batch inversion runs on base-field words: per
// point and z one square, three products of the batch and two for the
// quotient, against 12 for products of extension elements. One inversion per
// 16 quotients (46 -> 20 us at 2^18 points with gl::inv's chain, B200).
__global__ void __launch_bounds__(128) point_quotients_kernel(const __grid_constant__ PQArgs a) {
    const uint64_t i0 = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) * CHUNK;
    if (i0 >= a.n) return;
    const int cnt = (int)((a.n - i0) < (uint64_t)CHUNK ? (a.n - i0) : (uint64_t)CHUNK);
    uint64_t d[2 * CHUNK], norm[2 * CHUNK], pre[2 * CHUNK];
    uint64_t c[2], run = 1;
#pragma unroll
    for (int j = 0; j < 2; j++) c[j] = gl::mul7(gl::sqr(a.z[j].c1));
#pragma unroll
    for (int t = 0; t < CHUNK; t++) {
        if (t >= cnt) break;
        const uint64_t x = gl::mul(gl::GEN, a.wn.at(gl::bitrev(i0 + t, a.log_n)));
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int e = 2 * t + j;
            d[e] = gl::sub(a.z[j].c0, x);
            norm[e] = gl::sub(gl::sqr(d[e]), c[j]);
            pre[e] = run;
            run = gl::mul(run, norm[e]);
        }
    }
    uint64_t inv = gl::inv(run);
#pragma unroll
    for (int t = CHUNK - 1; t >= 0; t--) {
        if (t >= cnt) continue;
#pragma unroll
        for (int j = 1; j >= 0; j--) {
            const int e = 2 * t + j;
            const uint64_t ni = gl::mul(inv, pre[e]);
            inv = gl::mul(inv, norm[e]);
            uint64_t *o = a.q + 4 * (i0 + t) + 2 * j;
            o[0] = gl::mul(d[e], ni);
            o[1] = gl::mul(gl::neg(a.z[j].c1), ni);
        }
    }
}

// W[i][j] = x_i * q[i][j] for i < d
__global__ void top_weights_kernel(const uint64_t *q, uint64_t d, uint32_t log_n, ntt::PowTab wn, uint64_t *W) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= d) return;
    uint64_t x = gl::mul(gl::GEN, wn.at(gl::bitrev(i, log_n)));
#pragma unroll
    for (int k = 0; k < 4; k++) W[4 * i + k] = gl::mul(q[4 * i + k], x);
}
// Wsmall[i] = sum_{c < r} Wbig[i*r + c], eight lanes per i (r is a power of
// two; a serial sum of 32 was 20 us of load latency)
__global__ void __launch_bounds__(256) fold_weights_kernel(const uint64_t *Wb, uint64_t n_small, uint64_t r,
                                                           uint64_t *Ws) {
    const uint64_t t = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x, i = t >> 3;
    const uint32_t lane = threadIdx.x & 7;
    uint64_t s[4] = {0, 0, 0, 0};
    if (i < n_small)
        for (uint64_t c = lane; c < r; c += 8)
#pragma unroll
            for (int k = 0; k < 4; k++) s[k] = gl::add(s[k], Wb[4 * (i * r + c) + k]);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int k = 0; k < 4; k++) s[k] = gl::add(s[k], __shfl_xor_sync(0xffffffffu, s[k], m));
    if (lane < 4 && i < n_small) Ws[4 * i + lane] = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
}

// Column sums: partial[chunk][col][0..4) = sum over rows of chunk of
// W[i][j] * M[i][col] (EF for j = 0, 1). Block: 32 columns x 8 row lanes.
__global__ void __launch_bounds__(256) colsum_kernel(const uint64_t *M, uint64_t w, uint64_t d, const uint64_t *W,
                                                     uint64_t rows_per_chunk, uint64_t *partial) {
    __shared__ uint64_t red[8][32][4];
    const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
    // grid: x = column tile (fastest), y = row chunk
    const uint64_t col = (uint64_t)blockIdx.x * 32 + cl;
    const uint64_t r0 = (uint64_t)blockIdx.y * rows_per_chunk;
    const uint64_t r1 = min(d, r0 + rows_per_chunk);
    gl::SplitAcc acc[4];
    if (col < w) {
        // four rows per step: their loads are issued together, so that each
        // thread keeps several DRAM reads in flight
        uint64_t i = r0 + rl;
        for (; i + 24 < r1; i += 32) {
            uint64_t v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = __ldg(M + (i + 8 * u) * w + col);
#pragma unroll
            for (int u = 0; u < 4; u++)
#pragma unroll
                for (int k = 0; k < 4; k++) acc[k].mac(v[u], __ldg(W + 4 * (i + 8 * u) + k));
        }
        for (; i < r1; i += 8) {
            uint64_t v = __ldg(M + i * w + col);
#pragma unroll
            for (int k = 0; k < 4; k++) acc[k].mac(v, __ldg(W + 4 * i + k));
        }
    }
    uint64_t s[4];
#pragma unroll
    for (int k = 0; k < 4; k++) red[rl][cl][k] = s[k] = acc[k].reduce();
    __syncthreads();
    if (rl == 0 && col < w) {
        for (int r = 1; r < 8; r++)
#pragma unroll
            for (int k = 0; k < 4; k++) s[k] = gl::add(s[k], red[r][cl][k]);
#pragma unroll
        for (int k = 0; k < 4; k++) partial[(blockIdx.y * w + col) * 4 + k] = s[k];
    }
}
// out[col][0..4) = s_j * sum_chunk partial[chunk][col]: a block sums 8 columns
// (32 words, contiguous in a chunk) with 16 rows of threads over the chunks;
// with one thread per column, 296 chunks of a narrow matrix took 157 us.
__global__ void __launch_bounds__(512) colsum_finish_kernel(const uint64_t *partial, uint64_t n_chunks, uint64_t w,
                                                            gl::ef s0, gl::ef s1, uint64_t *out) {
    __shared__ uint64_t red[16][32];
    const uint32_t e = threadIdx.x & 31, r = threadIdx.x >> 5;
    const uint64_t word = (uint64_t)blockIdx.x * 32 + e;
    uint64_t s = 0;
    if (word < 4 * w)
#pragma unroll 4
        for (uint64_t c = r; c < n_chunks; c += 16) s = gl::add(s, __ldg(partial + c * w * 4 + word));
    red[r][e] = s;
    __syncthreads();
    if (r) return;
#pragma unroll
    for (int k = 1; k < 16; k++) s = gl::add(s, red[k][e]);
    // the four words of a column are four neighbouring lanes
    const uint64_t c1 = __shfl_down_sync(0xffffffffu, s, 1);
    if (word < 4 * w && !(e & 1)) {
        const gl::ef v = gl::ef_mul(gl::ef{s, c1}, (e & 2) ? s1 : s0);
        out[word] = v.c0;
        out[word + 1] = v.c1;
    }
}

// The column coefficients -ac^{W-1-c} over the aligned columns of all
// matrices, and the reduced openings f_red(z_j) = sum_c ac^{W-1-c} f_c(z_j)
// (padding columns are zero). One block: ac^0..ac^1023 by doubling in shared
// memory, then 1024 columns at a time from the last (at 1338 columns 22 us cold,
// 33 with a power per column; on the host it was an upload and two waits).
constexpr int MAX_DOTS = 24;
struct CoefArgs {
    int n_mats;
    uint64_t w[MAX_DOTS], off[MAX_DOTS], aligned_off[MAX_DOTS];  // columns and their places in evals and coef
    uint64_t total_aligned;
    gl::ef ac;
    const uint64_t *evals;  // 4 words per column: f(z_0), f(z_1)
    uint64_t *coef;         // 2 words per aligned column; the padding's are not written
    uint64_t *fred;         // 4 words
};
__global__ void __launch_bounds__(1024) coef_kernel(const __grid_constant__ CoefArgs a) {
    __shared__ gl::ef pw[1024];
    __shared__ uint64_t red[32][4];
    const uint32_t tid = threadIdx.x;
    if (tid == 0) pw[0] = gl::ef_one();
    gl::ef step = a.ac;  // ac^(2^s)
    for (uint32_t n = 1; n < 1024; n *= 2) {
        __syncthreads();
        if (tid >= n && tid < 2 * n) pw[tid] = gl::ef_mul(pw[tid - n], step);
        step = gl::ef_sqr(step);
    }
    __syncthreads();
    gl::ef p = pw[tid], f[2] = {gl::ef_zero(), gl::ef_zero()};
    for (uint64_t e = tid; e < a.total_aligned; e += 1024) {
        const uint64_t c = a.total_aligned - 1 - e;
        int m = a.n_mats - 1;
        while (a.aligned_off[m] > c) m--;
        const uint64_t col = c - a.aligned_off[m];
        if (col < a.w[m]) {
            const gl::ef n = gl::ef_neg(p);
            a.coef[2 * c] = n.c0;
            a.coef[2 * c + 1] = n.c1;
            const uint64_t *v = a.evals + 4 * (a.off[m] + col);
            f[0] = gl::ef_add(f[0], gl::ef_mul(p, gl::ef{v[0], v[1]}));
            f[1] = gl::ef_add(f[1], gl::ef_mul(p, gl::ef{v[2], v[3]}));
        }
        p = gl::ef_mul(p, step);  // ac^1024
    }
    uint64_t s[4] = {f[0].c0, f[0].c1, f[1].c0, f[1].c1};
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int m = 16; m; m >>= 1) s[k] = gl::add(s[k], __shfl_xor_sync(0xffffffffu, s[k], m));
    if ((tid & 31) == 0)
#pragma unroll
        for (int k = 0; k < 4; k++) red[tid >> 5][k] = s[k];
    __syncthreads();
    if (tid < 4) {
        uint64_t t = 0;
        for (int i = 0; i < 32; i++) t = gl::add(t, red[i][tid]);
        a.fred[tid] = t;
    }
}

// Row dot products dots[i] = sum_col coef[col] * M[i][col] (EF coef), G lanes
// per row (about eight columns per lane at least, so that the reduction over
// the lanes does not count: 2^18 x 64 took 111 us with 32 lanes per row, 47
// with 8; 2^16 x 250 74 us with 32, 42 with 16), coefficients staged in shared
// memory. Bound by the integer pipes (two lazy products per word).
template <int G>
__global__ void __launch_bounds__(256) rowdot_lanes_kernel(const uint64_t *M, uint64_t h, uint64_t w,
                                                           const uint64_t *coef, uint64_t *dots) {
    extern __shared__ __align__(16) uint64_t sc[];
    const uint64_t padded = (w + 4 * G - 1) / (4 * G) * (4 * G);  // zero coefficients up to whole steps
    for (uint64_t k = threadIdx.x; k < 2 * padded; k += blockDim.x) sc[k] = k < 2 * w ? coef[k] : 0;
    __syncthreads();
    const uint32_t lane = threadIdx.x % G;
    const uint64_t rows = (uint64_t)gridDim.x * (blockDim.x / G);
    const uint64_t first = ((uint64_t)blockIdx.x * blockDim.x + threadIdx.x) / G;
    // every lane of a warp takes the same number of turns
    for (uint64_t base = first - (threadIdx.x % 32) / G; base < h; base += rows) {
        const uint64_t i = base + (threadIdx.x % 32) / G;
        const uint64_t *row = M + (i < h ? i : h - 1) * w;
        gl::SplitAcc a0, a1;
        for (uint64_t col = lane; col < padded; col += 4 * G) {  // four loads in flight per lane
            uint64_t v[4];
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = col + G * u < w ? __ldg(row + col + G * u) : 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const ulonglong2 k = *(const ulonglong2 *)(sc + 2 * (col + G * u));
                a0.mac(v[u], k.x);
                a1.mac(v[u], k.y);
            }
        }
        uint64_t c0 = a0.reduce(), c1 = a1.reduce();
#pragma unroll
        for (int off = G / 2; off; off >>= 1) {
            c0 = gl::add(c0, __shfl_xor_sync(0xffffffffu, c0, off));
            c1 = gl::add(c1, __shfl_xor_sync(0xffffffffu, c1, off));
        }
        if (lane == 0 && i < h) {
            dots[2 * i] = c0;
            dots[2 * i + 1] = c1;
        }
    }
}
// Narrow matrices: one thread per row.
__global__ void rowdot_thread_kernel(const uint64_t *M, uint64_t h, uint64_t w, const uint64_t *coef, uint64_t *dots) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= h) return;
    const uint64_t *row = M + i * w;
    gl::SplitAcc a0, a1;
    for (uint64_t col = 0; col < w; col++) {
        uint64_t v = __ldg(row + col);
        a0.mac(v, __ldg(coef + 2 * col));
        a1.mac(v, __ldg(coef + 2 * col + 1));
    }
    dots[2 * i] = a0.reduce();
    dots[2 * i + 1] = a1.reduce();
}

struct AssembleArgs {
    const uint64_t *dots[MAX_DOTS];
    uint32_t lift[MAX_DOTS];
    int n_dots;
    const uint64_t *q;
    uint64_t n;
    const uint64_t *fred;  // f_red(z_0), f_red(z_1)
    gl::ef beta;
    uint64_t *out;  // n EF
};
__global__ void __launch_bounds__(256) assemble_kernel(const __grid_constant__ AssembleArgs a) {
    uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    gl::ef negf = gl::ef_zero();
    for (int m = 0; m < a.n_dots; m++) {
        const uint64_t *d = a.dots[m] + 2 * (i >> a.lift[m]);
        negf = gl::ef_add(negf, gl::ef{__ldg(d), __ldg(d + 1)});
    }
    const uint64_t *q = a.q + 4 * i;
    gl::ef r = gl::ef_mul(gl::ef{q[0], q[1]}, gl::ef_add(gl::ef{__ldg(a.fred), __ldg(a.fred + 1)}, negf));
    gl::ef r1 = gl::ef_mul(gl::ef{q[2], q[3]}, gl::ef_add(gl::ef{__ldg(a.fred + 2), __ldg(a.fred + 3)}, negf));
    r = gl::ef_add(r, gl::ef_mul(a.beta, r1));
    a.out[2 * i] = r.c0;
    a.out[2 * i + 1] = r.c1;
}

}  // namespace deep
