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
#include "context.cuh"
#include "gl.cuh"
#include "ntt.cuh"

namespace deep {

constexpr int CHUNK = 8;
constexpr int MAX_DOTS = 24;  // matrices of a launch

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
            ((ulonglong2 *)a.q)[2 * (i0 + t) + j] = ulonglong2{gl::mul(d[e], ni), gl::mul(gl::neg(a.z[j].c1), ni)};
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
// A launch over parts of different sizes, at most MAX_DOTS: part k has the
// blocks first[k] <= b < first[k + 1].
struct Parts {
    int n = 0;
    uint32_t first[MAX_DOTS + 1] = {0};
    int add(uint64_t blocks) {  // the new part's index
        if (n == MAX_DOTS) throw p3g::CudaError{p3g::ERR_INVALID, "too many parts in one launch"};
        first[n + 1] = first[n] + (uint32_t)blocks;
        return n++;
    }
    uint32_t blocks() const { return first[n]; }
    __device__ __forceinline__ int find(uint32_t &b) const {  // b: the block within its part
        int k = 0;
        while (k + 1 < n && first[k + 1] <= b) k++;
        b -= first[k];
        return k;
    }
};

// W_d of the smaller degrees: Wsmall[i] = sum_{c < r} Wbig[i*r + c], eight
// lanes per i (r is a power of two; a serial sum of 32 was 20 us of load
// latency). All degrees in one launch.
struct FoldWeightsArgs {
    Parts parts;
    const uint64_t *Wb;
    uint64_t n_small[MAX_DOTS], r[MAX_DOTS];
    uint64_t *Ws[MAX_DOTS];
};
__global__ void __launch_bounds__(256) fold_weights_kernel(const __grid_constant__ FoldWeightsArgs a) {
    uint32_t b = blockIdx.x;
    const int p = a.parts.find(b);
    const uint64_t t = (uint64_t)b * blockDim.x + threadIdx.x, i = t >> 3, r = a.r[p];
    const uint32_t lane = threadIdx.x & 7;
    uint64_t s[4] = {0, 0, 0, 0};
    if (i < a.n_small[p])
        for (uint64_t c = lane; c < r; c += 8)
#pragma unroll
            for (int k = 0; k < 4; k++) s[k] = gl::add(s[k], a.Wb[4 * (i * r + c) + k]);
#pragma unroll
    for (int m = 1; m < 8; m <<= 1)
#pragma unroll
        for (int k = 0; k < 4; k++) s[k] = gl::add(s[k], __shfl_xor_sync(0xffffffffu, s[k], m));
    if (lane < 4 && i < a.n_small[p]) a.Ws[p][4 * i + lane] = lane == 0 ? s[0] : lane == 1 ? s[1] : lane == 2 ? s[2] : s[3];
}

// Column sums of all matrices: partial[chunk][col][0..4) = sum over the
// chunk's rows of W[i][j] * M[i][col] (EF for j = 0, 1). A block takes 32
// columns x 8 row lanes of one chunk; all chunks have the same number of rows,
// so that the blocks of all matrices, one wave, end together. Four rows per
// step, loaded a step ahead; the weights of kTileRows rows in shared memory,
// a tile ahead. Bound by the integer pipes and latency (floors at 2^17 x 2633
// words: 0.42 ms of memory, 0.62 of products): the opening call over one such
// matrix takes 1.17 ms; 1.26 with both loads waited for in each step, 1.45
// with only the words ahead, 1.31 with eight rows per step (two blocks per
// SM), 1.58 at 64 registers (four).
struct ColsumArgs {
    Parts parts;
    const uint64_t *M[MAX_DOTS], *W[MAX_DOTS];
    uint64_t w[MAX_DOTS], d[MAX_DOTS];
    uint64_t *partial[MAX_DOTS];
    uint64_t rows_per_chunk;
};
constexpr int kTileRows = 128;
__global__ void __launch_bounds__(256) colsum_kernel(const __grid_constant__ ColsumArgs a) {
    __shared__ uint64_t red[8][32][4];
    __shared__ ulonglong2 wt[2][2 * kTileRows];
    uint32_t b = blockIdx.x;
    const int p = a.parts.find(b);
    const uint64_t w = a.w[p];
    const uint32_t tiles = (uint32_t)((w + 31) / 32), chunk = b / tiles;
    const int cl = threadIdx.x & 31, rl = threadIdx.x >> 5;
    const uint64_t col = (uint64_t)(b - chunk * tiles) * 32 + cl;
    const uint64_t r0 = chunk * a.rows_per_chunk, r1 = min(a.d[p], r0 + a.rows_per_chunk);
    const uint64_t *M = a.M[p] + col;
    const ulonglong2 *W = (const ulonglong2 *)a.W[p];
    // a tile of kTileRows weights: half a row (16 bytes) per thread
    auto weights = [&](uint64_t tile) {
        const uint64_t e = 2 * tile + threadIdx.x;
        return e < 2 * r1 ? __ldg(W + e) : ulonglong2{0, 0};
    };
    auto word = [&](uint64_t i) { return col < w && i < r1 ? __ldg(M + i * w) : 0; };
    gl::SplitAcc acc[4];
    uint64_t v[4], nv[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = word(r0 + rl + 8 * u);
    ulonglong2 nw = weights(r0);
    for (uint64_t tile = r0; tile < r1; tile += kTileRows) {
        const int buf = (int)((tile - r0) / kTileRows) & 1;
        wt[buf][threadIdx.x] = nw;
        __syncthreads();  // also: the tile before last is read
        nw = weights(tile + kTileRows);
#pragma unroll
        for (int q = 0; q < kTileRows; q += 32) {
#pragma unroll
            for (int u = 0; u < 4; u++) nv[u] = word(tile + q + 32 + rl + 8 * u);
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const ulonglong2 w0 = wt[buf][2 * (q + rl + 8 * u)], w1 = wt[buf][2 * (q + rl + 8 * u) + 1];
                acc[0].mac(v[u], w0.x), acc[1].mac(v[u], w0.y), acc[2].mac(v[u], w1.x), acc[3].mac(v[u], w1.y);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = nv[u];
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
        for (int k = 0; k < 4; k++) a.partial[p][(chunk * w + col) * 4 + k] = s[k];
    }
}
// out[col][0..4) = s_j * sum_chunk partial[chunk][col]: a block sums 8 columns
// (32 words, contiguous in a chunk) with 16 rows of threads over the chunks;
// with one thread per column, 296 chunks of a narrow matrix took 157 us.
struct ColsumFinishArgs {
    Parts parts;
    const uint64_t *partial[MAX_DOTS];
    uint64_t n_chunks[MAX_DOTS], w[MAX_DOTS];
    uint64_t *out[MAX_DOTS];
    gl::ef s0, s1;
};
__global__ void __launch_bounds__(512) colsum_finish_kernel(const __grid_constant__ ColsumFinishArgs a) {
    __shared__ uint64_t red[16][32];
    uint32_t b = blockIdx.x;
    const int p = a.parts.find(b);
    const uint64_t w = a.w[p], n_chunks = a.n_chunks[p], *partial = a.partial[p];
    const uint32_t e = threadIdx.x & 31, r = threadIdx.x >> 5;
    const uint64_t word = (uint64_t)b * 32 + e;
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
        const gl::ef v = gl::ef_mul(gl::ef{s, c1}, (e & 2) ? a.s1 : a.s0);
        a.out[p][word] = v.c0;
        a.out[p][word + 1] = v.c1;
    }
}

// The column coefficients -ac^{W-1-c} over the aligned columns of all
// matrices, and the reduced openings f_red(z_j) = sum_c ac^{W-1-c} f_c(z_j)
// (padding columns are zero). One block: ac^0..ac^1023 by doubling in shared
// memory with the powers ac^(2^s) from the host (squared in every thread they
// were half of the block's products), then 1024 columns at a time from the
// last (at 1338 columns 12 us cold, 22 with the squarings; on the host it was
// an upload and two waits).
struct CoefArgs {
    int n_mats;
    uint64_t w[MAX_DOTS], off[MAX_DOTS], aligned_off[MAX_DOTS];  // columns and their places in evals and coef
    uint64_t total_aligned;
    gl::ef step[11];  // ac^(2^s)
    const uint64_t *evals;  // 4 words per column: f(z_0), f(z_1)
    uint64_t *coef;         // 2 words per aligned column; the padding's are not written
    uint64_t *fred;         // 4 words
};
__global__ void __launch_bounds__(1024) coef_kernel(const __grid_constant__ CoefArgs a) {
    __shared__ gl::ef pw[1024];
    __shared__ uint64_t red[32][4];
    const uint32_t tid = threadIdx.x;
    if (tid == 0) pw[0] = gl::ef_one();
#pragma unroll 1
    for (int s = 0; s < 10; s++) {
        __syncthreads();
        if (tid >> s == 1) pw[tid] = gl::ef_mul(pw[tid - (1u << s)], a.step[s]);
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
        p = gl::ef_mul(p, a.step[10]);
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
// per row: about 32 columns per lane at least, as the reduction over the lanes
// costs as much as the products of eleven columns (the quotient call over
// 2^18 x 64 / 2^17 x 128 / 2^16 x 256 / 2^16 x 512 / 2^15 x 800 takes 133 / 131
// / 128 / 149 / 139 us, with twice as many lanes 141 / 132 / 131 / 158 / 146).
// Coefficients staged in shared memory. Bound by memory at large widths and the integer pipes (two lazy
// products per word): the quotient call over 2^18 x 2633 words takes 1.11 ms,
// 1.23 with the loads of a step waited for.
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
    // every lane of a warp takes the same number of turns; a step's words are
    // loaded during the step before, the next row's first ones included
    const uint32_t sub = (threadIdx.x % 32) / G;
    auto row_at = [&](uint64_t i) { return M + (i < h ? i : h - 1) * w; };
    const uint64_t *row = row_at(first);
    uint64_t v[4];
#pragma unroll
    for (int u = 0; u < 4; u++) v[u] = lane + G * u < w ? __ldg(row + lane + G * u) : 0;
    for (uint64_t base = first - sub; base < h; base += rows) {
        const uint64_t i = base + sub;
        const uint64_t *next_row = row_at(i + rows);
        gl::SplitAcc a0, a1;
        for (uint64_t col = lane; col < padded; col += 4 * G) {
            const bool more = col + 4 * G < padded;
            const uint64_t *from = more ? row : next_row;
            const uint64_t c = more ? col + 4 * G : lane;
            uint64_t nv[4];
#pragma unroll
            for (int u = 0; u < 4; u++) nv[u] = c + G * u < w ? __ldg(from + c + G * u) : 0;
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const ulonglong2 k = *(const ulonglong2 *)(sc + 2 * (col + G * u));
                a0.mac(v[u], k.x);
                a1.mac(v[u], k.y);
            }
#pragma unroll
            for (int u = 0; u < 4; u++) v[u] = nv[u];
        }
        row = next_row;
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
