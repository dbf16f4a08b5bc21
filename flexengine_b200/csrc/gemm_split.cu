// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) for float32 operands on the fifth-generation tensor cores, as exact as the chain of
// float32 multiply-adds of gemm_fp32.cu or more so.
//
// A float32 has 24 bits of mantissa: cut off after 8 and after 16 of them it is the sum of three bfloat16 numbers, exactly (a = a0 + a1 +
// a2; a0 the upper half of the word, a1 the upper half of what is left, a2 the rest).  Products of two such parts are exact in float32, so
// a.w is the sum of nine products that tcgen05.mma forms exactly; the three smallest (a1 w2, a2 w1, a2 w2: below 2^-22 of a.w together) are
// left out.  What remains is how sums are rounded.  The tensor cores round their running sum towards zero, so it is kept short: a chunk of 64
// k's starts from zero, in one sum for the largest products and two for the others, and is then added to a float32 sum in
// registers, rounded to nearest.
//
// Every output is formed in the same steps whatever the batch: the chunks of a segment of K in order, then the segments in
// order, their number chosen by N and K alone.  Rows of W are the 128 rows of the MMA tile, rows of A its columns (16 or 64 by
// M), so that a handful of rows streams W once.
//
// Blocks stay for tile after tile.  Two groups of eight warps read float32 rows, chunk about, and write the three parts into
// 128-byte-swizzled tiles; one thread issues 12 MMAs a chunk into one of several accumulators in tensor memory; eight more warps add the
// others to their registers and write the tile out at the end.  A result that is no finite number is formed again as a chain of
// multiply-adds (an infinity has no three parts).
//
// A chunk's way (rows from memory, cut up, through shared memory, 12 MMAs, sums) takes 1.1 to 1.5 us and is what bounds the kernel: a third of
// the stalls are loads on their way, the tensor cores are busy 26 % and 19 % of the time (tiles of 16 and of 64 rows).  17,920 x 1,536: 33 us with
// 1 to 16 rows (the chain of multiply-adds 24 to 41), 42 with 64 (107), 144 with 256 (278); 1,536 x 8,960: 33 (31 to 69), 40 (125), 78 (244).
// Relative error against 64 bits, K = 1,536 / 8,960: 1.5e-7 / 1.5e-7, the chain 7.0e-7 / 1.7e-6.
#include "common.cuh"

using namespace fe;

namespace {

constexpr int TILE_W = 128;             // rows of W in a tile = UMMA M
constexpr int CHUNK = 64;               // k's of a chunk: 128 bytes of bfloat16, one swizzle atom wide
constexpr int GROUP_WARPS = 8, SPLIT_WARPS = 2 * GROUP_WARPS, SUM_WARPS = 8, THREADS = 32 * (SPLIT_WARPS + SUM_WARPS);
constexpr long long WAIT_LIMIT = 4000000000LL;      // clock cycles

__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(unsigned long long* bar, int count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(unsigned long long* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ bool mbar_test(unsigned long long* bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool mbar_wait(unsigned long long* bar, unsigned parity) {
    if (mbar_test(bar, parity)) return true;
    const long long t0 = clock64();
    while (!mbar_test(bar, parity)) {
        if (clock64() - t0 > WAIT_LIMIT) return false;
    }
    return true;
}

// K-major operand, 128-byte swizzle, rows 128 bytes apart, groups of 8 rows 1024 bytes apart (as in gemm_tcgen05.cu).
__device__ __forceinline__ unsigned long long smem_desc(unsigned addr) {
    return (((unsigned long long)addr & 0x3FFFFull) >> 4) | ((1024ull >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// float accumulator, bfloat16 operands, both K-major, 128 x n tile
__host__ __device__ constexpr unsigned instr_desc(int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((unsigned)(n >> 3) << 17) | ((unsigned)(TILE_W >> 4) << 24); }
__device__ __forceinline__ void umma(unsigned tmem_d, unsigned long long adesc, unsigned long long bdesc, unsigned idesc, unsigned accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n"
                 ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void umma_commit(unsigned long long* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory"); }

// eight accumulator columns of this thread's TMEM lane (wait::ld is the caller's)
__device__ __forceinline__ void tmem_load8(unsigned taddr, unsigned* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// Eight floats -> their three parts, eight bfloat16 each.
__device__ __forceinline__ void split8(const float4& p, const float4& q, uint4& hi, uint4& mid, uint4& lo) {
    const float v[8] = {p.x, p.y, p.z, p.w, q.x, q.y, q.z, q.w};
    unsigned h[4], m[4], l[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const unsigned a = __float_as_uint(v[2 * i]), b = __float_as_uint(v[2 * i + 1]);
        const float a1 = v[2 * i] - __uint_as_float(a & 0xffff0000u), b1 = v[2 * i + 1] - __uint_as_float(b & 0xffff0000u);
        const unsigned ua = __float_as_uint(a1), ub = __float_as_uint(b1);
        const float a2 = a1 - __uint_as_float(ua & 0xffff0000u), b2 = b1 - __uint_as_float(ub & 0xffff0000u);
        h[i] = __byte_perm(a, b, 0x7632);
        m[i] = __byte_perm(ua, ub, 0x7632);
        l[i] = __byte_perm(__float_as_uint(a2), __float_as_uint(b2), 0x7632);
    }
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

template <int BN> struct Sizes {
    static constexpr int STAGES = BN == 16 ? 3 : 2;             // no more: loads on their way take lines of what is left of the SM's memory
    static constexpr int W_PART = TILE_W * CHUNK * 2, X_PART = BN * CHUNK * 2;
    static constexpr int STAGE = 3 * (W_PART + X_PART);
    static constexpr int BYTES = STAGES * STAGE + 1024;
    static constexpr int BUFFERS = BN == 16 ? 4 : 2;            // chunks' accumulators, of 3 BN columns of tensor memory each
    static constexpr int COLUMNS = BN == 16 ? 256 : 512;
};

// ``part`` (null with one segment): the segments' sums, [segments][M][N].
template <int BN, bool VEC>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                  float* __restrict__ part, const int M, const int N, const int K, const int m_tiles, const int tiles, const int segments,
                  int* __restrict__ status) {
    using S = Sizes<BN>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long full_bar[S::STAGES], empty_bar[S::STAGES], acc_full[S::BUFFERS], acc_empty[S::BUFFERS];
    __shared__ unsigned tmem_holder;
    __shared__ volatile int give_up;
    const unsigned base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int chunks = (K + CHUNK - 1) / CHUNK;
    // tile t: a segment of the chunks (fastest), a tile of A's rows, a tile of W's rows
    auto place = [&](int t, int& w0, int& m0, int& c0, int& c1, int& s) {
        s = t % segments;
        const int u = t / segments;
        m0 = u % m_tiles * BN;
        w0 = u / m_tiles * TILE_W;
        c0 = (int)((long long)chunks * s / segments);
        c1 = (int)((long long)chunks * (s + 1) / segments);
    };
    if (tid == 0) {
        for (int s = 0; s < S::STAGES; ++s) { mbar_init(&full_bar[s], GROUP_WARPS); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < S::BUFFERS; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], SUM_WARPS); }
        give_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == SPLIT_WARPS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_u32(&tmem_holder)), "n"(S::COLUMNS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    griddep_wait();
    griddep_launch_dependents();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_holder;

    if (warp < SPLIT_WARPS) {
        // ---- float32 rows into three bfloat16 parts: an item is eight k's of a row ----
        constexpr int ITEMS_W = TILE_W * 8 / (32 * GROUP_WARPS), ITEMS_X = BN >= 32 ? BN * 8 / (32 * GROUP_WARPS) : 1;
        // two groups of eight warps take turns: while one waits for its loads, a free stage or its stores, the other is at work
        const int turn = warp / GROUP_WARPS, row = (tid >> 3) & 31, at = tid & 7;      // item i: row + 32 i, eight k's ``at``
        const bool has_x = BN >= 32 || row < BN;
        const size_t apart = (size_t)32 * K;
        auto eight = [&](const float* __restrict__ s, bool in, int k, float4& p, float4& q) {
            p = q = make_float4(0.f, 0.f, 0.f, 0.f);
            if (!in || k >= K) return;
            if (VEC) {                                            // K a multiple of 4, 16-byte addresses
                p = __ldg(reinterpret_cast<const float4*>(s + k));
                if (k + 4 < K) q = __ldg(reinterpret_cast<const float4*>(s + k + 4));
            } else {
                float v[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) v[i] = k + i < K ? __ldg(s + k + i) : 0.f;
                p = make_float4(v[0], v[1], v[2], v[3]);
                q = make_float4(v[4], v[5], v[6], v[7]);
            }
        };
        auto store = [&](unsigned to, int part_bytes, int r, const float4& p, const float4& q) {
            uint4 hi, mid, lo;
            split8(p, q, hi, mid, lo);
            const unsigned a = to + (r >> 3) * 1024 + (r & 7) * 128 + ((at ^ (r & 7)) << 4);
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(a), "r"(hi.x), "r"(hi.y), "r"(hi.z), "r"(hi.w) : "memory");
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(a + part_bytes), "r"(mid.x), "r"(mid.y), "r"(mid.z), "r"(mid.w) : "memory");
            asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n" ::"r"(a + 2 * part_bytes), "r"(lo.x), "r"(lo.y), "r"(lo.z), "r"(lo.w) : "memory");
        };
        // what is loaded next: chunk ``nc`` of tile ``nt``
        int nt = blockIdx.x, w0 = 0, m0 = 0, nc = 0, nc1 = 0, ns = 0;
        const float *wr = W, *xr = A;                             // this thread's first rows of the tile
        auto settle = [&]() {
            if (nt >= tiles) return;
            place(nt, w0, m0, nc, nc1, ns);
            wr = W + (size_t)(w0 + row) * K;
            xr = A + (size_t)(m0 + row) * K;
        };
        settle();
        auto step = [&]() { if (++nc >= nc1) { nt += gridDim.x; settle(); } };
        if (turn == 1 && nt < tiles) step();
        auto load_w = [&](float4 (&v)[2 * ITEMS_W]) {
#pragma unroll
            for (int i = 0; i < ITEMS_W; ++i) eight(wr + i * apart, w0 + row + 32 * i < N, nc * CHUNK + 8 * at, v[2 * i], v[2 * i + 1]);
        };
        auto load_x = [&](float4 (&v)[2 * ITEMS_X]) {
            if (has_x) {
#pragma unroll
                for (int i = 0; i < ITEMS_X; ++i) eight(xr + i * apart, m0 + row + 32 * i < M, nc * CHUNK + 8 * at, v[2 * i], v[2 * i + 1]);
            }
        };
        auto put_w = [&](unsigned to, const float4 (&v)[2 * ITEMS_W]) {
#pragma unroll
            for (int i = 0; i < ITEMS_W; ++i) store(to, S::W_PART, row + 32 * i, v[2 * i], v[2 * i + 1]);
        };
        auto put_x = [&](unsigned to, const float4 (&v)[2 * ITEMS_X]) {
            if (has_x) {
#pragma unroll
                for (int i = 0; i < ITEMS_X; ++i) store(to + 3 * S::W_PART, S::X_PART, row + 32 * i, v[2 * i], v[2 * i + 1]);
            }
        };
        auto done = [&](int s) {
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");      // the parts are read by the tensor cores
            __syncwarp();
            if (lane == 0) mbar_arrive(&full_bar[s]);
        };
        int at_chunk = turn;
        auto stage_free = [&](int& s) {
            s = at_chunk % S::STAGES;
            if (!mbar_wait(&empty_bar[s], ((at_chunk / S::STAGES) & 1) ^ 1)) { give_up = 1; return false; }
            at_chunk += 2;
            return true;
        };
        // the rows of W of the next chunk are asked for before the rows of A of this one are cut up, and the other way round
        float4 vw[2 * ITEMS_W], vx[2 * ITEMS_X];
        if (nt < tiles) { load_w(vw); load_x(vx); }
        while (nt < tiles && !give_up) {
            int s;
            if (!stage_free(s)) break;
            const unsigned to = base + s * S::STAGE;
            step();
            if (nt < tiles) step();
            put_w(to, vw);
            if (nt < tiles) load_w(vw);
            put_x(to, vx);
            if (nt < tiles) load_x(vx);
            done(s);
        }
    } else {
        // ---- sums: warp w reads TMEM lanes 32 (w % 4) .. + 31 (rows of W), one half of the columns (rows of A) ----
        constexpr int COLS = BN / 2;
        const int quarter = warp & 3, col0 = ((warp - SPLIT_WARPS) >> 2) * COLS;
        // one thread issues the MMAs, a chunk or two ahead of the one it adds up
        int it = blockIdx.x, ic = 0, ic1 = 0, issued = 0;
        auto issue = [&]() {
            if (it >= tiles || give_up) return;
            if (ic >= ic1) {
                int w0, m0, seg;
                place(it, w0, m0, ic, ic1, seg);
            }
            const int s = issued % S::STAGES, buf = issued % S::BUFFERS;
            if (!mbar_wait(&full_bar[s], (issued / S::STAGES) & 1) || !mbar_wait(&acc_empty[buf], ((issued / S::BUFFERS) & 1) ^ 1)) { give_up = 1; return; }
            tc_fence_after();
            const unsigned w = base + s * S::STAGE, x = w + 3 * S::W_PART, acc = tmem + buf * 3 * BN;
            // The parts of A's rows lie one after the other like 3 BN rows: a part of W meets as many of them as count at once.  Column
            // block 0 of the accumulator takes w0 a0, block 1 w0 a1 + w1 a0, block 2 w0 a2 + w1 a1 + w2 a0.
#pragma unroll
            for (int k = 0; k < CHUNK / 16; ++k)
#pragma unroll
                for (int p = 0; p < 3; ++p)
                    umma(acc + p * BN, smem_desc(w + p * S::W_PART) + 2 * k, smem_desc(x) + 2 * k, instr_desc((3 - p) * BN), (p > 0 || k > 0) ? 1u : 0u);
            umma_commit(&empty_bar[s]);
            umma_commit(&acc_full[buf]);
            ++issued;
            if (++ic >= ic1) it += gridDim.x;
        };
        const bool issuer = tid == SPLIT_WARPS * 32;
        if (issuer) {
            issue();
            if (S::BUFFERS > 2) issue();
        }
        int i = 0;
        for (int t = blockIdx.x; t < tiles && !give_up; t += gridDim.x) {
            int w0, m0, c0, c1, seg;
            place(t, w0, m0, c0, c1, seg);
            float sum[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
            bool ok = true;
            for (int c = c0; c < c1; ++c, ++i) {
                const int buf = i % S::BUFFERS;
                if (issuer) issue();
                __syncwarp();
                if (!mbar_wait(&acc_full[buf], (i / S::BUFFERS) & 1)) { give_up = 1; ok = false; break; }
                tc_fence_after();
                const unsigned from = tmem + buf * 3 * BN + col0 + ((unsigned)(quarter * 32) << 16);
#pragma unroll
                for (int j = 0; j < COLS; j += 8) {
                    unsigned r[3][8];
#pragma unroll
                    for (int h = 0; h < 3; ++h) tmem_load8(from + h * BN + j, r[h]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
#pragma unroll
                    for (int e = 0; e < 8; ++e) sum[j + e] += __uint_as_float(r[0][e]) + (__uint_as_float(r[1][e]) + __uint_as_float(r[2][e]));
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[buf]);
            }
            if (!ok) break;
            const int n = w0 + quarter * 32 + lane;
            if (n >= N) continue;
            const float add = part == nullptr && bias != nullptr ? bias[n] : 0.f;
            float* const out = part == nullptr ? C : part + (size_t)seg * M * N;
#pragma unroll
            for (int j = 0; j < COLS; ++j) {
                const int m = m0 + col0 + j;
                if (m >= M) continue;
                float v = sum[j];
                if (!(fabsf(v) <= 3.402823466e38f)) {
                    v = 0.f;
                    for (int k = c0 * CHUNK; k < min(K, c1 * CHUNK); ++k) v = fmaf(A[(size_t)m * K + k], W[(size_t)n * K + k], v);
                }
                out[(size_t)m * N + n] = v + add;
            }
        }
    }
    __syncthreads();
    if (give_up && tid == 0 && status) atomicOr(status, FE_STATUS_WAIT_EXPIRED);
    tc_fence_before();
    __syncthreads();
    if (warp == SPLIT_WARPS) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "n"(S::COLUMNS) : "memory");
}

// C = the segments' sums in order, + bias.
__global__ void __launch_bounds__(256) add_segments_kernel(const float* __restrict__ part, const float* __restrict__ bias, float* __restrict__ C,
                                                           const long long total, const int N, const int segments) {
    griddep_wait();
    griddep_launch_dependents();
    const long long i = ((long long)blockIdx.x * 256 + threadIdx.x) * 4;
    if (i >= total) return;
    if ((total & 3) == 0 && (N & 3) == 0) {
        float4 v = *reinterpret_cast<const float4*>(part + i);
        for (int s = 1; s < segments; ++s) {
            const float4 p = *reinterpret_cast<const float4*>(part + s * total + i);
            v.x += p.x; v.y += p.y; v.z += p.z; v.w += p.w;
        }
        if (bias) {
            const int n = (int)(i % N);
            v.x += bias[n]; v.y += bias[n + 1]; v.z += bias[n + 2]; v.w += bias[n + 3];
        }
        C[i] = v.x; C[i + 1] = v.y; C[i + 2] = v.z; C[i + 3] = v.w;
        return;
    }
    for (long long j = i; j < min(total, i + 4); ++j) {
        float v = part[j];
        for (int s = 1; s < segments; ++s) v += part[s * total + j];
        C[j] = v + (bias ? bias[j % N] : 0.f);
    }
}

template <int BN, bool VEC>
int launch_split(const float* A, const float* W, const float* bias, float* C, float* part, int M, int N, int K, int segments, int* status, cudaStream_t stream) {
    const auto kernel = gemm_split_kernel<BN, VEC>;
    cudaError_t err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Sizes<BN>::BYTES);
    if (err == cudaSuccess) err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (Sizes<BN>::BYTES + 2048) * 100 / (228 * 1024) + 1);
    FE_REQUIRE(err == cudaSuccess, "gemm_split: %s", cudaGetErrorString(err));
    const long long m_tiles = (M + BN - 1) / BN, tiles = m_tiles * ((N + TILE_W - 1) / TILE_W) * segments;
    FE_REQUIRE(tiles < (1LL << 30), "gemm_split: too many tiles");
    const int sms = fe_sm_count();
    fe::launch(kernel, (unsigned)(tiles < sms ? tiles : sms), THREADS, Sizes<BN>::BYTES, stream, A, W, bias, C, segments > 1 ? part : (float*)nullptr, M, N, K,
               (int)m_tiles, (int)tiles, segments, status);
    return fe_check_launch("gemm_split");
}

}  // namespace

// Into how many segments K is cut, by N and K alone: as many as give every SM a tile with 256 rows, of four chunks or more.
extern "C" int fe_gemm_split_segments(int N, int K) {
    const int sms = fe_sm_count(), tiles = 2 * ((N + TILE_W - 1) / TILE_W), chunks = (K + CHUNK - 1) / CHUNK;
    int s = sms / tiles;
    if (s > chunks / 4) s = chunks / 4;
    return s < 1 ? 1 : s;
}

// ``part``: room for segments x M x N floats (16-byte aligned); not read with one segment.
extern "C" int fe_gemm_split(const float* A, const float* W, const float* bias, float* C, float* part, int M, int N, int K, int* status,
                             cudaStream_t stream) {
    FE_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_split: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return 0;
    const int segments = fe_gemm_split_segments(N, K);
    FE_REQUIRE(segments == 1 || (part != nullptr && ((size_t)part & 15) == 0), "gemm_split: no room for the sums of %d segments", segments);
    const bool vec = (K & 3) == 0 && (((size_t)A | (size_t)W) & 15) == 0;
    int rc;
#define FE_SPLIT(BN) rc = vec ? launch_split<BN, true>(A, W, bias, C, part, M, N, K, segments, status, stream) \
                              : launch_split<BN, false>(A, W, bias, C, part, M, N, K, segments, status, stream)
    if (M <= 16) FE_SPLIT(16);
    else FE_SPLIT(64);
#undef FE_SPLIT
    if (rc || segments == 1) return rc;
    const long long total = (long long)M * N;
    fe::launch(add_segments_kernel, (unsigned)((total + 1023) / 1024), 256, 0, stream, (const float*)part, bias, C, total, N, segments);
    return fe_check_launch("gemm_split (segments)");
}
