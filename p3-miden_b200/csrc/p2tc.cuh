// Poseidon2-12 with the linear part of its internal rounds on the tensor
// cores, for the throughput-bound hash kernels.
//
// What bounds the permutation: the integer pipes. One permutation is 118
// S-boxes (472 products) plus linear layers; with the internal diagonal as
// 264 more general products it took 19.7 k instructions per state and ran at
// 1.27 G permutations/s (B200, 1965 MHz), the ALU pipe at 70 % and the
// IMAD pipe at 81 %. The internal layer is linear in everything but word 0,
// so the inputs u_0..u_21 of the 22 internal S-boxes and the 12 words after
// them are fixed linear forms of
//   y_0..y_11  the S-box outputs of the last initial external round,
//   z_0..z_21  the internal S-box outputs (z_r enters u_{r+1} and later),
//   1          (round constants).
// Those forms run as exact 8-bit integer matrix products (tcgen05.mma
// kind::i8, unsigned, 32-bit accumulators): a state is a row of bytes (8 per
// word), and the column of byte j of word w holds the 8 bytes of
// coefficient * 2^(8j) mod p, so an output is 8 accumulators L_l with value
// sum_l L_l 2^(8l) mod p, put together and reduced once (recombine). The
// products that stay on the CUDA cores are the S-boxes and one diagonal
// product per two internal rounds: 12.4 k instructions per state, measured
// 1.91 G permutations/s against 1.27 (chained permutations, no memory).
//
// Mapping. A group is 128 threads, one state per thread, thread = TMEM lane.
// The y bytes of a group are the K-major A operand in shared memory (12 KB);
// 1 and the z's are the A operand in TMEM (48 columns), the accumulators 16
// columns beside them: 64 columns per group, 7 groups (896 threads, 72
// registers) per SM. 8 groups at 64 registers measured the same rate and
// spilled, 6 groups 1 % less. Batch q (16 x K) gives u_2q whole and u_{2q+1}
// without z_2q (one product, mu_0 + 1, adds it): one tensor-core round trip
// per two rounds (one per round measured 8 % slower). The last six batches
// give the 12 words after the internal rounds, with the first terminal round
// constants. Tables: 17 batches of 4608 bytes per CTA.
//
// Products are reduced in Montgomery form (R = 2^64): R^3 = 2^192 = 1 mod p,
// so the four reductions of x^7 = (x^2 x) (x^2)^2 contribute R^-6 = 1 and an
// S-box needs no conversion.
#pragma once
#include <cstdint>
#include <cstring>
#include <vector>

#include "gl.cuh"
#include "merkle.cuh"
#include "poseidon2.cuh"

namespace p2t {

constexpr int kGroups = 7, kThreads = kGroups * 128;
constexpr int kWords = 36;                    // y_0..y_11, 1, z_0..z_21, one unused
constexpr int kK = kWords * 8;                // bytes of a row
constexpr int kBatches = 17, kBatchBytes = 16 * kK, kTableBytes = kBatches * kBatchBytes;
constexpr int kABytes = 128 * 96;             // y rows of a group
constexpr int kSmemBytes = kTableBytes + kGroups * kABytes;
constexpr uint32_t kColsPerGroup = 64, kAccCol = 48;

// Shared-memory order of an 8-bit K-major operand without swizzle: core
// matrices of 8 rows x 16 bytes. Table: [K / 16][row group of 8][8][16];
// y rows: [K / 16][row group of 16][8][16].
//
// The tables for the constants `c` (poseidon2.cuh's layout). False when an
// accumulator could exceed what recombine holds (its byte weights add up to
// more than 2^32 / 257 / 255): such constants hash with p2_permute_dev.
inline bool build_tables(const uint64_t *c, std::vector<uint8_t> &img) {
    struct Form {
        uint64_t c[kWords];
    };
    img.assign(kTableBytes, 0);
    uint64_t worst = 0;
    auto put = [&](int batch, int half, const Form &f) {
        uint8_t *b = img.data() + (size_t)batch * kBatchBytes + half * 128;
        uint64_t sum[8] = {0};
        for (int w = 0; w < kWords; w++) {
            uint64_t v = f.c[w];
            for (int j = 0; j < 8; j++, v = gl::mul(v, 256)) {
                if (w == 12 && j) v = 0;  // the word 1 has one nonzero byte
                const int k = 8 * w + j;
                for (int l = 0; l < 8; l++) {
                    const uint8_t byte = (uint8_t)(v >> (8 * l));
                    b[(k / 16) * 256 + l * 16 + k % 16] = byte;
                    sum[l] += byte;
                }
            }
        }
        for (uint64_t s : sum) worst = s > worst ? s : worst;
    };
    static const int m4[4][4] = {{2, 3, 1, 1}, {1, 2, 3, 1}, {1, 1, 2, 3}, {3, 1, 1, 2}};
    Form st[12];
    memset(st, 0, sizeof(st));
    for (int i = 0; i < 12; i++)
        for (int j = 0; j < 12; j++) st[i].c[j] = (uint64_t)m4[i % 4][j % 4] * (i / 4 == j / 4 ? 2 : 1);
    for (int r = 0; r < 22; r++) {
        Form u = st[0];
        u.c[12] = gl::add(u.c[12], c[p2::OFF_INT + r]);
        if (r & 1) u.c[12 + r] = 0;  // z_{r-1}, added by the product with mu_0 + 1
        put(r / 2, r & 1, u);
        memset(&st[0], 0, sizeof(Form));
        st[0].c[13 + r] = 1;
        Form sum;
        memset(&sum, 0, sizeof(sum));
        for (int i = 0; i < 12; i++)
            for (int w = 0; w < kWords; w++) sum.c[w] = gl::add(sum.c[w], st[i].c[w]);
        for (int i = 0; i < 12; i++)
            for (int w = 0; w < kWords; w++)
                st[i].c[w] = gl::add(sum.c[w], gl::mul(c[p2::OFF_DIAG + i] % gl::P, st[i].c[w]));
    }
    for (int i = 0; i < 12; i++) {
        st[i].c[12] = gl::add(st[i].c[12], c[p2::OFF_TERM + i]);
        put(11 + i / 2, i & 1, st[i]);
    }
    return worst * 255 * 257 < (1ull << 32);
}

// A wait gives up after 0.1 s; a product takes about a microsecond.
constexpr uint32_t kWaitNs = 100000000;
struct Args {
    const uint8_t *table;  // kTableBytes, device
    uint32_t *err;         // set when a wait gave up
    uint32_t wait_ns;      // kWaitNs, or less; 0: every wait gives up at once
};

// One group's handles.
struct Group {
    uint32_t tm;       // TMEM address: the group's columns, the warp's lanes
    uint32_t table;    // shared addresses
    uint32_t a_rows;
    uint32_t mbar;
    uint32_t bar;      // named barrier of the group
    uint32_t phase;
    uint32_t warp;     // warp of the group, 0..3
    bool dead;
    uint8_t *my_row;   // this thread's 16-byte column of y rows
    uint32_t *err;
    uint32_t wait_ns;
};

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void st4(uint32_t a, uint64_t x, uint64_t y) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x4.b32 [%0], {%1, %2, %3, %4};\n\t"
                 "tcgen05.wait::st.sync.aligned;" ::"r"(a),
                 "r"((uint32_t)x), "r"((uint32_t)(x >> 32)), "r"((uint32_t)y), "r"((uint32_t)(y >> 32))
                 : "memory");
}
__device__ __forceinline__ void ld16(uint32_t a, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, "
                 "%14, %15}, [%16];\n\t"
                 "tcgen05.wait::ld.sync.aligned;"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                   "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]),
                   "=r"(v[15])
                 : "r"(a)
                 : "memory");
}
// One poll; with SUSPEND the hardware may hold the thread for some time first.
template <bool SUSPEND = true>
__device__ __forceinline__ bool try_wait(uint32_t mbar, uint32_t phase) {
    uint32_t ok;
    if (SUSPEND)
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(mbar), "r"(phase)
                     : "memory");
    else
        asm volatile("{\n\t.reg .pred p;\n\t"
                     "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                     "selp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok)
                     : "r"(mbar), "r"(phase)
                     : "memory");
    return ok != 0;
}

__device__ __forceinline__ uint64_t now_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}
// Whether the phase ends within ns. kGrace more polls come after the time is
// up (a fraction of a millisecond), so that a context switch in between, after
// which the group's other warps still have to reach the barrier, does not
// count as a wait.
constexpr int kGrace = 4096;
__device__ __forceinline__ bool wait(uint32_t mbar, uint32_t phase, uint32_t ns) {
    if (ns == 0) return false;
    if (try_wait(mbar, phase)) return true;
    const uint64_t t0 = now_ns();
    while (now_ns() - t0 < ns)
        if (try_wait(mbar, phase)) return true;
#pragma unroll 1
    for (int i = 0; i < kGrace; i++)
        if (try_wait<false>(mbar, phase)) return true;
    return false;
}

// Tables, barriers, TMEM and the constant word; every thread of the CTA.
// smem: kSmemBytes of dynamic shared memory.
__device__ __forceinline__ Group setup(uint8_t *smem, const Args &a) {
    __shared__ uint32_t tmem_base;
    __shared__ __align__(8) uint64_t mbars[kGroups];
    for (int i = threadIdx.x * 16; i < kTableBytes; i += kThreads * 16)
        *(uint4 *)(smem + i) = __ldg((const uint4 *)(a.table + i));
    if (threadIdx.x < kGroups)
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_addr(&mbars[threadIdx.x])) : "memory");
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(smem_addr(&tmem_base))
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the tables, read by the tensor cores
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t grp = threadIdx.x >> 7, warp = (threadIdx.x >> 5) & 3;
    Group g;
    g.tm = tmem_base + grp * kColsPerGroup + (warp << 21);  // lane field: 32 * warp, bits 16 and up
    g.table = smem_addr(smem);
    uint8_t *rows = smem + kTableBytes + grp * kABytes;
    g.a_rows = smem_addr(rows);
    g.my_row = rows + (threadIdx.x & 127) * 16;
    g.mbar = smem_addr(&mbars[grp]);
    g.bar = 1 + grp;
    g.phase = 0;
    g.warp = warp;
    g.dead = false;
    g.err = a.err;
    g.wait_ns = a.wait_ns;
    st4(g.tm, 1, 0);
    return g;
}
__device__ __forceinline__ void teardown(Group &g) {
    fence_before();
    __syncthreads();
    fence_after();
    if (threadIdx.x < 32)  // warp 0 of group 0: its address is the allocation's base
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(g.tm));
}

// Batch `batch` over the y rows and the first 4 * z_steps words of the z
// part; the whole group calls it, and one thread issues once the group's
// earlier accesses to its operands are complete. All four warps wait at the
// barrier, although only the issuing one needs the others: threads that gave up
// are not paced by the batches any more, and with bare arrivals one warp's next
// could complete this batch's barrier in another's place and leave a third
// waiting for good (this costs 0.2 to 0.6 %: a 2^18 x 336 slab's commit 12.95
// against 12.88 ms). The warps take turns (a batch is about 75 instructions to issue): with the
// same warp of every group, that scheduler alone had 10 % more to do, 1.79
// against 1.91 G permutations/s.
__device__ __forceinline__ void issue(Group &g, int batch, int z_steps) {
    fence_before();
    asm volatile("bar.sync %0, 128;" ::"r"(g.bar) : "memory");
    if (((batch + g.bar) & 3) == g.warp) {
        if ((threadIdx.x & 31) == 0 && !g.dead) {
            fence_after();
            const uint32_t tm = g.tm & 0xFFFF;  // lane 0
            // instruction: 32-bit accumulators, unsigned bytes, N = 16, M = 128
            const uint32_t idesc = (2u << 4) | ((16u >> 3) << 17) | ((128u >> 4) << 24);
            const uint64_t fixed = 1ull << 46;  // descriptor version; no swizzle
            const uint64_t bd = fixed | ((g.table + batch * kBatchBytes) >> 4) | ((uint64_t)(256 >> 4) << 16) |
                                ((uint64_t)(128 >> 4) << 32);
            const uint64_t ad = fixed | (g.a_rows >> 4) | ((uint64_t)(2048 >> 4) << 16) | ((uint64_t)(128 >> 4) << 32);
#pragma unroll
            for (int s = 0; s < 3; s++)
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\t"
                             "tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tm + kAccCol),
                             "l"(ad + s * (4096 >> 4)), "l"(bd + s * (512 >> 4)), "r"(idesc), "r"(s)
                             : "memory");
#pragma unroll 1
            for (int s = 0; s < z_steps; s++)
                asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, 1, 0;\n\t"
                             "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(tm + kAccCol),
                             "r"(tm + 8 * s), "l"(bd + (s + 3) * (512 >> 4)), "r"(idesc)
                             : "memory");
            asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(g.mbar)
                         : "memory");
        }
        __syncwarp();
    }
}
// Waits for the batch in flight and reads its two outputs' accumulators. A
// wait that runs out marks the launch as failed (the host checks err), and the
// thread neither issues nor waits for a further batch, but keeps to the group's
// barriers, to a bounded end (a batch that is not issued makes the other
// threads' waits run out too). It goes on only after a second bounded wait for
// the batch itself, which would otherwise read shared memory and write TMEM
// that the CTA has given back: every batch is waited for by the warp that
// issued it, so none is in flight at teardown.
__device__ __forceinline__ void collect(Group &g, uint32_t *L) {
    if (!g.dead && !wait(g.mbar, g.phase, g.wait_ns)) {
        *g.err = 1;
        g.dead = true;
        wait(g.mbar, g.phase, kWaitNs);
    }
    g.phase ^= 1;
    __syncwarp();
    fence_after();
    ld16(g.tm + kAccCol, L);
}
// sum_l L_l 2^(8l) (+ t), weakly reduced; every L_l < 2^32 / 257
template <bool ADD>
__device__ __forceinline__ uint64_t recombine(const uint32_t *L, uint64_t t = 0) {
    const uint32_t t1 = L[1] * 256 + L[0], t3 = L[3] * 256 + L[2], t5 = L[5] * 256 + L[4], t7 = L[7] * 256 + L[6];
    const uint64_t lo = (uint64_t)t3 * 65536 + t1, hi = (uint64_t)t7 * 65536 + t5;
    uint32_t r1, r2;
    asm("add.cc.u32 %0, %2, %3;\n\taddc.u32 %1, %4, 0;"
        : "=&r"(r1), "=&r"(r2)
        : "r"((uint32_t)(lo >> 32)), "r"((uint32_t)hi), "r"((uint32_t)(hi >> 32)));
    const p2w::W w{((uint64_t)r1 << 32) | (uint32_t)lo, r2};
    return p2w::wreduce(ADD ? p2w::wadd1(w, t) : w);
}

// The permutation; the whole group calls it. `capacity_only`: only words
// 8..11 of the result are wanted (the next absorb overwrites the others).
__device__ __forceinline__ void permute(Group &g, uint64_t *s, bool capacity_only) {
    p2w::ext_linear(s, p2::OFF_INIT);
#pragma unroll 1
    for (int r = 0; r < 8; r++) {
#pragma unroll
        for (int i = 0; i < 12; i++) s[i] = p2w::sbox(s[i]);
        if (r == 3) {
#pragma unroll
            for (int q = 0; q < 6; q++)
                *(ulonglong2 *)(g.my_row + q * 2048) = make_ulonglong2(s[2 * q], s[2 * q + 1]);
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            uint32_t L[16];
#pragma unroll 1
            for (int q = 0; q < 11; q++) {
                issue(g, q, (2 * q + 4) / 4);
                collect(g, L);
                const uint64_t z0 = p2w::sbox(recombine<false>(L));
                const uint64_t z1 = p2w::sbox(recombine<true>(L + 8, p2w::mul(z0, c_p2[p2::OFF_MU0P1_M])));
                st4(g.tm + 2 + 4 * q, z0, z1);
            }
            issue(g, 11, 6);
#pragma unroll
            for (int q = 0; q < 6; q++) {
                collect(g, L);
                if (q < 5) issue(g, 12 + q, 6);
                s[2 * q] = recombine<false>(L);
                s[2 * q + 1] = recombine<false>(L + 8);
            }
        } else {
            p2w::ext_linear(s, r < 3 ? p2::OFF_INIT + 12 * (r + 1) : r < 7 ? p2::OFF_TERM + 12 * (r - 3) : -1,
                            capacity_only && r == 7);
        }
    }
}

}  // namespace p2t

namespace merkle {

// Leaf sponge and compression of many states with p2t::permute. A CTA runs
// `active` groups (at most p2t::kGroups), each on blocks of 128 leaves or
// parents: block (it * gridDim.x + blockIdx.x) * active + group, it < iters.
struct TcShape {
    uint64_t n_blocks;
    uint32_t active, iters;
};

// leaf_class_kernel's sponge (same arguments and results mod p); the class
// has a multiple of 128 leaves. Bound by the integer pipes; rows are read
// once, 64 bytes per thread and permutation.
template <bool CM>
__global__ void __launch_bounds__(p2t::kThreads, 1)
    leaf_class_tc_kernel(const __grid_constant__ ClassArgs a, const __grid_constant__ p2t::Args t,
                         const __grid_constant__ TcShape sh) {
    extern __shared__ __align__(1024) uint8_t smem[];
    p2t::Group g = p2t::setup(smem, t);
    const uint32_t grp = threadIdx.x >> 7;
    uint32_t chunks = 0;  // permutations per leaf
    for (int m = 0; m < a.n_mats; m++) chunks += (uint32_t)((a.width[m] + 7) / 8);
    for (uint32_t it = 0; it < sh.iters && grp < sh.active; it++) {
        const uint64_t b = ((uint64_t)it * gridDim.x + blockIdx.x) * sh.active + grp;
        if (b >= sh.n_blocks) break;
        const uint64_t j = b * 128 + (threadIdx.x & 127);
        uint64_t s[12];
        if (a.prev) {
            const uint64_t *p = a.prev + (j >> (a.log_h - a.prev_log_h)) * 12;
#pragma unroll
            for (int i = 0; i < 12; i++) s[i] = p[i];
        } else {
#pragma unroll
            for (int i = 0; i < 12; i++) s[i] = 0;
        }
        uint32_t left = chunks;
        for (int m = 0; m < a.n_mats; m++) {
            const uint64_t w = a.width[m];
            const uint64_t *row = a.data[m] + j * a.ld[m];
            uint64_t *cmj = CM && j < a.cm_rows ? a.cm + j : nullptr;
#pragma unroll 1
            for (uint64_t i = 0; i < w; i += 8) {
#pragma unroll
                for (int k = 0; k < 8; k++) s[k] = i + k < w ? __ldg(row + i + k) : 0;
                if (CM && cmj) {
#pragma unroll
                    for (int k = 0; k < 8; k++)
                        if (i + k < w) cmj[(i + k) * a.cm_ld] = s[k];
                }
                p2t::permute(g, s, --left != 0);
            }
        }
        if (a.digests_out) {
#pragma unroll
            for (int i = 0; i < 4; i++) a.digests_out[j * 4 + i] = p2w::canon(s[i]);
        } else {
#pragma unroll
            for (int i = 0; i < 12; i++) a.states_out[j * 12 + i] = s[i];
        }
    }
    p2t::teardown(g);
}

// One level: every parent of layer l_in + 1 (a multiple of 128 of them).
__global__ void __launch_bounds__(p2t::kThreads, 1)
    compress_level_tc_kernel(uint64_t *layers, uint64_t H, uint32_t l_in, const __grid_constant__ p2t::Args t,
                             const __grid_constant__ TcShape sh) {
    extern __shared__ __align__(1024) uint8_t smem[];
    p2t::Group g = p2t::setup(smem, t);
    const uint32_t grp = threadIdx.x >> 7;
    const uint64_t off_in = 2 * H - 2 * (H >> l_in), off_out = 2 * H - 2 * (H >> (l_in + 1));
    for (uint32_t it = 0; it < sh.iters && grp < sh.active; it++) {
        const uint64_t b = ((uint64_t)it * gridDim.x + blockIdx.x) * sh.active + grp;
        if (b >= sh.n_blocks) break;
        const uint64_t p = b * 128 + (threadIdx.x & 127);
        const uint64_t *in = layers + 4 * (off_in + 2 * p);
        uint64_t s[12];
#pragma unroll
        for (int i = 0; i < 8; i++) s[i] = in[i];
#pragma unroll
        for (int i = 8; i < 12; i++) s[i] = 0;
        p2t::permute(g, s, false);
#pragma unroll
        for (int i = 0; i < 4; i++) layers[4 * (off_out + p) + i] = p2w::canon(s[i]);
    }
    p2t::teardown(g);
}

}  // namespace merkle
