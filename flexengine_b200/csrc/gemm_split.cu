// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) for float32 operands on the fifth-generation tensor cores, with the error of float32
// multiply-adds (gemm_fp32.cu) or less.
//
// A float32 has 24 bits of mantissa: cut off after 8 and after 16 of them it is the sum of three bfloat16 numbers (a = a0 + a1 + a2; a0 the
// upper half of the word, a1 the upper half of what is left, a2 the rest), exactly from 2^-110 on; of a smaller number less than 2^-133 is
// lost, bfloat16's last place.  a1 is below 2^-7 of a's power of two and a2 below 2^-15.  Products of two parts are exact in float32, so a.w is
// the sum of nine products that tcgen05.mma forms exactly; a2 w2, below 2^-30 of a.w, is left out.  (Without a1 w2 and a2 w1 too, up to
// 2^-21 of a product was missing, always to the same side: rows with few numbers other than 0 were further from 64 bits than the multiply-adds.)
// What remains is how sums are rounded.  The tensor cores round their running sum towards zero.  Of the largest products, w0 a0, it is
// kept short: a chunk of 64 k's starts from zero and is then added to a float32 sum in registers, rounded to nearest.  The others, from
// 2^-7 of a product down, have three sums in tensor memory, by their sizes, over all chunks of a tile, and meet the first one at its end: what they lose
// by then is below what the first loses, and a result of few products is rounded about once.  Segments of K hand on their sums with what their rounding
// lost, and are added up in 64 bits.
//
// Results that this does not serve are formed again from the rows themselves, in 64 bits: what is no finite number (an infinity has no three
// parts), and what is below LEAST, where the lost places of small numbers could count.  They cannot for any other result: a number of LARGE
// or more is made a NaN in shared memory, so that its results are formed again, and with all others below it a sum of K products has
// lost less than 2 K 2^-133 LARGE, below 2^-24 of LEAST up to K = 2^16.
//
// Every output is formed in the same steps whatever the batch: the chunks of a segment of K in order, then the segments in
// order, their number chosen by N and K alone.  Rows of W are the 128 rows of the MMA tile, rows of A its columns (16 or 64 by
// M), so that a handful of rows streams W once.
//
// Blocks stay for tile after tile.  Two groups of eight warps read float32 rows, chunk about, and write the three parts into
// 128-byte-swizzled tiles; a thread of its own issues 16 MMAs a chunk; eight more warps add the chunks' sums to their registers and
// write the tile out at the end, while MMAs of the next one run.
//
// A chunk's way (rows from memory, cut up, through shared memory, 16 MMAs, sums) takes 1.0 to 1.3 us and is what bounds the kernel: with no MMA
// but one a step 17,920 x 1,536 takes 30 and 122 us (4 and 256 rows), with no stores to shared memory 27 and 107; asking rows into L2 ahead of time
// makes it slower (33, 138).  17,920 x 1,536: 31 us with 1 to 16 rows (the chain of multiply-adds 24 to 40), 40 with 64 (106), 135 with 256 (278).
// Relative error against 64 bits, K = 1,536 / 8,960: 1.2e-7 / 1.0e-7, the chain 7.0e-7 / 1.7e-6; rows of 1, 2, 8 and 32 numbers other than 0:
// 2.5e-8, 2.6e-8, 2.8e-8, 4.2e-8, the chain 2.5e-8, 3.1e-8, 5.2e-8, 1.0e-7.
// Forming again is for what hardly ever is: all of 256 x 1,536 results (K = 8,960) take 3.4 ms; a row of NaN among 256 rows 156 us instead of 85, 128 rows
// of W that are 0 395, looked through 16 numbers a lane at a time.  (Flags of the rows that lost places, which would tell such rows from others, cost
// every product 5 to 9 %, by the registers of the warps that cut up.)
#include "tcgen05.cuh"

using namespace fe;

namespace {

constexpr int TILE_W = 128;             // rows of W in a tile = UMMA M
constexpr int CHUNK = 64;               // k's of a chunk: 128 bytes of bfloat16, one swizzle atom wide
constexpr int GROUP_WARPS = 8, SPLIT_WARPS = 2 * GROUP_WARPS, SUM_WARPS = 8, THREADS = 32 * (SPLIT_WARPS + SUM_WARPS + 4);
constexpr float LEAST = 8.673617380e-19f, MOST = 3.402823466e38f;      // 2^-60; results outside of these bounds are formed again
constexpr unsigned LARGE = 0x4f80;                  // 2^32, the upper half of the word

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
    unsigned most = 0;                                // of the eight, two by two: the upper halves without their signs
#pragma unroll
    for (int i = 0; i < 4; ++i) most = __vmaxu2(most, h[i] & 0x7fff7fffu);
    if ((most >> 16) >= LARGE || (most & 0xffffu) >= LARGE) h[0] = 0x7fc07fc0u;
    hi = make_uint4(h[0], h[1], h[2], h[3]);
    mid = make_uint4(m[0], m[1], m[2], m[3]);
    lo = make_uint4(l[0], l[1], l[2], l[3]);
}

template <int BN> struct Sizes {
    static constexpr int STAGES = BN == 16 ? 3 : 2;             // no more: loads on their way take lines of what is left of the SM's memory
    static constexpr int W_PART = TILE_W * CHUNK * 2, X_PART = BN * CHUNK * 2;
    static constexpr int STAGE = 3 * (W_PART + X_PART);
    static constexpr int BYTES = STAGES * STAGE + 1024;
    // Columns of tensor memory: the sums of the smaller products (3 BN) of two tiles, then chunks' sums of the largest (BN each)
    static constexpr int BUFFERS = BN == 16 ? 4 : 2;
    static constexpr int COLUMNS = BN == 16 ? 256 : 512;
    static_assert(6 * BN + BUFFERS * BN <= COLUMNS, "tensor memory");
};

// ---- results formed again; every lane of a warp takes part ----
__device__ bool all_zero(const float* __restrict__ row, int K) {
    const int lane = threadIdx.x & 31;
    for (int k0 = lane; k0 < K + lane; k0 += 512) {      // sixteen loads at once: a row of W that is 0 is looked through to its end
        float v[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) v[i] = row[min(k0 + 32 * i, K - 1)];
        unsigned any = 0;
#pragma unroll
        for (int i = 0; i < 16; ++i) any |= __float_as_uint(v[i]) << 1;
        if (__any_sync(0xffffffffu, any != 0)) return false;
    }
    return true;
}
__device__ float product64(const float* __restrict__ a, const float* __restrict__ w, int K) {
    const int lane = threadIdx.x & 31;
    double v = 0.;
    for (int k0 = lane; k0 < K + lane; k0 += 512) {
        float x[16], y[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int k = k0 + 32 * i;
            x[i] = k < K ? a[k] : 0.f;
            y[i] = k < K ? w[k] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < 16; ++i) v = fma((double)x[i], (double)y[i], v);
        if (__any_sync(0xffffffffu, v != v)) return __uint_as_float(0x7fc00000u);      // and stays so
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return (float)v;
}
// Whether a sum of products has to be formed again.  A sum of 0 may be one that lost all its places; where a whole row is 0 it is not.
__device__ __forceinline__ bool outside(float v) { return !(fabsf(v) >= LEAST && fabsf(v) <= MOST); }

// Rows m0 .. (32 at most) of A with each lane's row n of W: bit j of ``which`` for row m0 + j, of ``zero`` where the sum came to 0.
__device__ __noinline__ void form_again(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                                        int m0, int n, int N, int K, unsigned which, unsigned zero) {
    unsigned w_known = 0, w_zero = 0;                  // lanes whose row of W was looked through, and is 0
    for (unsigned columns = __reduce_or_sync(0xffffffffu, which); columns; columns &= columns - 1) {
        const int j = __ffs(columns) - 1;
        const float* a = A + (size_t)(m0 + j) * K;
        const unsigned zeros = __ballot_sync(0xffffffffu, zero >> j & 1u);
        unsigned lanes = __ballot_sync(0xffffffffu, which >> j & 1u);
        if (zeros && all_zero(a, K)) lanes &= ~zeros;
        for (; lanes; lanes &= lanes - 1) {
            const int l = __ffs(lanes) - 1, nl = __shfl_sync(0xffffffffu, n, l);
            const unsigned bit = 1u << l;
            const float* w = W + (size_t)nl * K;
            if (zeros & bit) {
                if (!(w_known & bit)) {
                    w_known |= bit;
                    if (all_zero(w, K)) w_zero |= bit;
                }
                if (w_zero & bit) continue;
            }
            const float v = product64(a, w, K);
            if ((threadIdx.x & 31) == l) C[(size_t)(m0 + j) * N + nl] = v + (bias ? bias[nl] : 0.f);
        }
    }
}

// ``part`` (null with one segment): the segments' sums, [segments][M / 4, rounded up][N][4], and ``rest`` what their rounding lost: a thread has
// rows of A one after the other, and writes four at once.
template <int BN, bool VEC>
__global__ void __launch_bounds__(THREADS, 1)
gemm_split_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                  float4* __restrict__ part, uint2* __restrict__ rest, const int M, const int N, const int K, const int m_tiles, const int tiles,
                  const int segments, int* __restrict__ status) {
    using S = Sizes<BN>;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    __shared__ __align__(8) unsigned long long full_bar[S::STAGES], empty_bar[S::STAGES], acc_full[S::BUFFERS], acc_empty[S::BUFFERS], small_empty[2];
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
        c0 = (int)((unsigned)chunks * s / segments);           // 2^25 chunks and 64 segments at most
        c1 = (int)((unsigned)chunks * (s + 1) / segments);
    };
    if (tid == 0) {
        for (int s = 0; s < S::STAGES; ++s) { mbar_init(&full_bar[s], GROUP_WARPS); mbar_init(&empty_bar[s], 1); }
        for (int b = 0; b < S::BUFFERS; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], SUM_WARPS); }
        for (int b = 0; b < 2; ++b) mbar_init(&small_empty[b], SUM_WARPS);
        give_up = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == SPLIT_WARPS) tmem_alloc<S::COLUMNS>(&tmem_holder);
    griddep_wait();
    griddep_launch_dependents();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_holder;

    // After a wait that ran out, here or in another warp, all lanes of a warp leave together: their votes and barriers are the warp's.
    auto go_on = [&](bool arrived) {
        if (__all_sync(0xffffffffu, arrived && !give_up)) return true;
        give_up = 1;
        return false;
    };

    // Registers: 28 warps of 72 at launch, 64,512 together.  The sixteen that cut up hold 48 numbers on their way and take 80 each (with 72, 256 rows x
    // 17,920 x 1,536: 191 us instead of 143), which the issuing thread's four warps give: 16 x 80 + 8 x 72 + 4 x 40 = 28 x 72.
    if (warp < SPLIT_WARPS) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 80;\n" ::: "memory");
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
            if (!go_on(mbar_wait(&empty_bar[s], ((at_chunk / S::STAGES) & 1) ^ 1))) return false;
            at_chunk += 2;
            return true;
        };
        // the rows of W of the next chunk are asked for before the rows of A of this one are cut up, and the other way round
        float4 vw[2 * ITEMS_W], vx[2 * ITEMS_X];
        if (nt < tiles) { load_w(vw); load_x(vx); }
        while (nt < tiles) {
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
    } else if (warp < SPLIT_WARPS + SUM_WARPS) {
        // ---- sums: warp w reads TMEM lanes 32 (w % 4) .. + 31 (rows of W), one half of the columns (rows of A) ----
        constexpr int COLS = BN / 2;
        const int quarter = warp & 3, col0 = ((warp - SPLIT_WARPS) >> 2) * COLS;
        int i = 0, turn = 0;
        for (int t = blockIdx.x; t < tiles; t += gridDim.x, ++turn) {
            int w0, m0, c0, c1, seg;
            place(t, w0, m0, c0, c1, seg);
            float sum[COLS];
#pragma unroll
            for (int j = 0; j < COLS; ++j) sum[j] = 0.f;
            const unsigned lanes = (unsigned)(quarter * 32) << 16;
            bool ok = true;
            for (int c = c0; c < c1; ++c, ++i) {
                const int buf = i % S::BUFFERS;
                if (!(ok = go_on(mbar_wait(&acc_full[buf], (i / S::BUFFERS) & 1)))) break;
                tc_fence_after();
                const unsigned from = tmem + (6 + buf) * BN + col0 + lanes;
                constexpr int PART = COLS < 16 ? COLS : 16;
#pragma unroll
                for (int j0 = 0; j0 < COLS; j0 += PART) {
                    unsigned r[PART];
#pragma unroll
                    for (int j = 0; j < PART; j += 8) tmem_load8(from + j0 + j, r + j);
                    tmem_arrived<PART>(r);
#pragma unroll
                    for (int j = 0; j < PART; ++j) sum[j0 + j] += __uint_as_float(r[j]);
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&acc_empty[buf]);
            }
            if (!ok) break;
            // the last chunk's MMAs are done, and so are those of the small sums
            const int n = w0 + quarter * 32 + lane, rows = n < N ? M - m0 - col0 : 0;
            const bool whole = part == nullptr;              // else the segments' sums are looked at when they are added up
            const float add = whole && bias != nullptr && n < N ? bias[n] : 0.f;
            float* out = C + (size_t)(m0 + col0) * N + n;
            size_t four = ((size_t)seg * ((M + 3) / 4) + (m0 + col0) / 4) * N + n;
            unsigned which = 0, zero = 0;
            const unsigned from = tmem + (turn & 1) * 3 * BN + col0 + lanes;
#pragma unroll
            for (int j0 = 0; j0 < COLS; j0 += 8) {
                unsigned r[3][8];
#pragma unroll
                for (int h = 0; h < 3; ++h) tmem_load8(from + h * BN + j0, r[h]);
                tmem_arrived<24>(&r[0][0]);
#pragma unroll
                for (int e = 0; e < 8; ++e) r[0][e] = __float_as_uint(__uint_as_float(r[0][e]) + (__uint_as_float(r[1][e]) + __uint_as_float(r[2][e])));
                if (whole) {
#pragma unroll
                    for (int e = 0; e < 8; ++e, out += N) {
                        const int j = j0 + e;
                        const float v = sum[j] + __uint_as_float(r[0][e]);
                        if (j >= rows) continue;
                        *out = v + add;
                        if (outside(v)) which |= 1u << j;
                        if (v == 0.f) zero |= 1u << j;
                    }
                } else {
#pragma unroll
                    for (int e = 0; e < 8; e += 4, four += N) {
                        float v[4], lost[4];
#pragma unroll
                        for (int i4 = 0; i4 < 4; ++i4) {     // and what large + small lose (Knuth's two-sum)
                            const float large = sum[j0 + e + i4], small = __uint_as_float(r[0][e + i4]);
                            v[i4] = large + small;
                            const float p = v[i4] - large;
                            lost[i4] = (large - (v[i4] - p)) + (small - p);
                        }
                        if (j0 + e >= rows) continue;
                        part[four] = make_float4(v[0], v[1], v[2], v[3]);
                        const __nv_bfloat162 a = __floats2bfloat162_rn(lost[0], lost[1]), b = __floats2bfloat162_rn(lost[2], lost[3]);
                        rest[four] = make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&small_empty[turn & 1]);
            if (whole && __any_sync(0xffffffffu, which != 0)) form_again(A, W, bias, C, m0 + col0, n, N, K, which, zero);
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 40;\n" ::: "memory");
        if (warp == SPLIT_WARPS + SUM_WARPS && lane == 0) {
            // ---- one thread issues the MMAs; three warps only give registers ----
            int issued = 0, tile = 0;
            bool ok = true;
            for (int t = blockIdx.x; t < tiles && ok; t += gridDim.x, ++tile) {
                int w0, m0, c0, c1, seg;
                place(t, w0, m0, c0, c1, seg);
                for (int c = c0; c < c1; ++c, ++issued) {
                    const int s = issued % S::STAGES, buf = issued % S::BUFFERS;
                    ok = mbar_wait(&full_bar[s], (issued / S::STAGES) & 1) && mbar_wait(&acc_empty[buf], ((issued / S::BUFFERS) & 1) ^ 1) &&
                         (c > c0 || mbar_wait(&small_empty[tile & 1], ((tile >> 1) & 1) ^ 1)) && !give_up;
                    if (!ok) break;
                    tc_fence_after();
                    const unsigned w = base + s * S::STAGE, x = w + 3 * S::W_PART;
                    const unsigned small = tmem + (tile & 1) * 3 * BN, large = tmem + (6 + buf) * BN;
                    // The parts of A's rows lie one after the other like 3 BN rows: a part of W meets as many of them as count at once.
                    // Block 0 of the small sums takes w0 a1 + w1 a0, block 1 w0 a2 + w1 a1 + w2 a0, block 2 w1 a2 + w2 a1.
                    const unsigned long long dw0 = desc_k_major(w), dw1 = desc_k_major(w + S::W_PART), dw2 = desc_k_major(w + 2 * S::W_PART);
                    const unsigned long long dx0 = desc_k_major(x), dx1 = desc_k_major(x + S::X_PART);
#pragma unroll
                    for (int k = 0; k < CHUNK / 16; ++k) {
                        umma(small, dw1 + 2 * k, dx0 + 2 * k, instr_desc(TILE_W, 3 * BN), (k > 0 || c > c0) ? 1u : 0u);
                        umma(small, dw0 + 2 * k, dx1 + 2 * k, instr_desc(TILE_W, 2 * BN), 1u);
                        umma(small + BN, dw2 + 2 * k, dx0 + 2 * k, instr_desc(TILE_W, 2 * BN), 1u);
                        umma(large, dw0 + 2 * k, dx0 + 2 * k, instr_desc(TILE_W, BN), k > 0 ? 1u : 0u);
                    }
                    umma_commit(&empty_bar[s]);
                    umma_commit(&acc_full[buf]);
                }
            }
            if (!ok) give_up = 1;
            // Only after a wait that ran out are any MMAs still at work when the sums are done: they end before the tensor memory is given back
            if (issued > 0) mbar_wait(&acc_full[(issued - 1) % S::BUFFERS], ((issued - 1) / S::BUFFERS) & 1);
        }
    }
    __syncthreads();
    if (give_up && tid == 0 && status) atomicOr(status, FE_STATUS_WAIT_EXPIRED);
    tc_fence_before();
    __syncthreads();
    if (warp == SPLIT_WARPS) tmem_dealloc<S::COLUMNS>(tmem);
}

// C = the segments' sums in order, + bias.  A thread takes four rows of A and a row of W; a warp what is to be formed again.
constexpr int ADDING = 64;               // threads: blocks on many SMs at few rows, too
__global__ void __launch_bounds__(ADDING) add_segments_kernel(const float4* __restrict__ part, const uint2* __restrict__ rest, const float* __restrict__ A,
                                                           const float* __restrict__ W, const float* __restrict__ bias, float* __restrict__ C,
                                                           const int M, const int N, const int K, const int segments) {
    griddep_wait();
    griddep_launch_dependents();
    const long long i = (long long)blockIdx.x * ADDING + threadIdx.x, all = (long long)((M + 3) / 4) * N;
    const int m = i < all ? (int)(i / N) * 4 : M, n = (int)(i % N);
    double sum[4] = {0., 0., 0., 0.};
    if (m < M) {
#pragma unroll 4
        for (int s = 0; s < segments; ++s) {
            const float4 p = part[s * all + i];
            const uint2 q = rest[s * all + i];
            sum[0] += (double)p.x + (double)__uint_as_float(q.x << 16);
            sum[1] += (double)p.y + (double)__uint_as_float(q.x & 0xffff0000u);
            sum[2] += (double)p.z + (double)__uint_as_float(q.y << 16);
            sum[3] += (double)p.w + (double)__uint_as_float(q.y & 0xffff0000u);
        }
    }
    unsigned which = 0, zero = 0;
    const float add = bias ? bias[n] : 0.f;
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        if (m + e >= M) continue;
        const float v = (float)sum[e];
        C[(size_t)(m + e) * N + n] = v + add;
        if (outside(v)) which |= 1u << e;
        if (v == 0.f) zero |= 1u << e;
    }
    if (!__any_sync(0xffffffffu, which != 0)) return;
    // The lanes' rows of W meet the same four rows of A, unless the warp reaches over the end of them
    const int first = __shfl_sync(0xffffffffu, m, 0);
    form_again(A, W, bias, C, first, n, N, K, m == first ? which : 0u, m == first ? zero : 0u);
    for (unsigned others = __ballot_sync(0xffffffffu, m != first && which != 0); others; others &= others - 1) {
        const int l = __ffs(others) - 1;
        const bool mine = (threadIdx.x & 31) == l;
        form_again(A, W, bias, C, __shfl_sync(0xffffffffu, m, l), n, N, K, mine ? which : 0u, mine ? zero : 0u);
    }
}

template <int BN, bool VEC>
int launch_split(const float* A, const float* W, const float* bias, float* C, float4* part, uint2* rest, int M, int N, int K, int segments, int* status, cudaStream_t stream) {
    const auto kernel = gemm_split_kernel<BN, VEC>;
    cudaError_t err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, Sizes<BN>::BYTES);
    if (err == cudaSuccess) err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributePreferredSharedMemoryCarveout, (Sizes<BN>::BYTES + 2048) * 100 / (228 * 1024) + 1);
    FE_REQUIRE(err == cudaSuccess, "gemm_split: %s", cudaGetErrorString(err));
    const long long m_tiles = (M + BN - 1) / BN, tiles = m_tiles * ((N + TILE_W - 1) / TILE_W) * segments;
    FE_REQUIRE(tiles < (1LL << 30), "gemm_split: too many tiles");
    const int sms = fe_sm_count();
    fe::launch(kernel, (unsigned)(tiles < sms ? tiles : sms), THREADS, Sizes<BN>::BYTES, stream, A, W, bias, C, segments > 1 ? part : (float4*)nullptr, rest, M, N, K,
               (int)m_tiles, (int)tiles, segments, status);
    return fe_check_launch("gemm_split");
}

// Into how many segments K is cut, by N and K alone, so that a step of few rows has every SM at work: the least of rounds over the SMs x (a
// segment's chunks and one to begin), two for adding up and one for every 16,384 numbers added, in the time of a chunk.  (As many
// as gave every SM a tile of 128 rows with 256 of them were taken before: tiles have 64 rows, or 16, and 72 blocks stood on 148 SMs for
// 1,536 x 8,960.)  Segments before and now, us with 4, 64 and 256 rows before and now, and the chain's with 4: 1,536 x 8,960 6, 12: 34, 43, 77 and 26, 30, 78 (31);
// 4,608 x 3,584 2, 4: 36, 47, 88 and 25, 30, 88 (21); 3,584 x 18,944 2, 5: 154, 195, 385 and 70, 90, 315 (99); 5,120 x 13,824 1, 7: 238, 279, 564 and
// 75, 96, 335 (116); 27,648 x 5,120 1, 2: 166, 213, 615 and 132, 181, 661 (122).
int segments_of(int N, int K) {
    const int sms = fe_sm_count(), tiles = (N + TILE_W - 1) / TILE_W, chunks = (K + CHUNK - 1) / CHUNK;
    int best = 1;
    long long least = 0;
    for (int s = 1; s <= 64 && s <= chunks / 4; ++s) {
        const unsigned rounds = ((unsigned)tiles * s + sms - 1) / sms, each = ((unsigned)chunks + s - 1) / s + 1;
        const long long cost = 16384LL * ((long long)rounds * each + (s > 1 ? 2 : 0)) + (s > 1 ? (long long)s * N : 0);
        if (s == 1 || cost < least) best = s, least = cost;
    }
    return best;
}
// The segments' sums of all rows of a long prompt are a large part of the memory that is left beside the pages (302 MB for 8,192 rows x 1,536 x
// 8,960): rows go in parts of nearly the same size, whole tiles each, which share one room.
constexpr long long ROOM = 64LL << 20;              // bytes at most, or those of 64 rows
int rows_at_once(int M, int N, int segments) {
    if (segments == 1) return M;
    long long most = ROOM / (6LL * segments * N) / 64 * 64;
    if (most < 64) most = 64;
    const long long parts = (M + most - 1) / most;
    return (int)((M + parts * 64 - 1) / (parts * 64) * 64);
}

}  // namespace

extern "C" int fe_gemm_split_segments(int N, int K) { return segments_of(N, K); }

// Bytes of room that a product needs for its segments' sums: bounded, whatever the rows.
extern "C" long long fe_gemm_split_room(int M, int N, int K) {
    const int segments = segments_of(N, K);
    if (segments == 1 || M <= 0) return 0;
    const long long rows = rows_at_once(M, N, segments);
    return 24LL * segments * N * (((rows < M ? rows : M) + 3) / 4);
}

// ``part``: 16-byte aligned room of fe_gemm_split_room bytes; not read with one segment.
extern "C" int fe_gemm_split(const float* A, const float* W, const float* bias, float* C, float* part, int M, int N, int K, int* status,
                             cudaStream_t stream) {
    FE_REQUIRE(M >= 0 && N > 0 && K > 3 * CHUNK, "gemm_split: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return 0;
    const int segments = segments_of(N, K);
    FE_REQUIRE(segments == 1 || (part != nullptr && ((size_t)part & 15) == 0), "gemm_split: no room for the sums of %d segments", segments);
    const bool vec = (K & 3) == 0 && (((size_t)A | (size_t)W) & 15) == 0;
    const int at_once = rows_at_once(M, N, segments);
    for (long long m0 = 0; m0 < M; m0 += at_once) {
        const int rows = (int)(M - m0 < at_once ? M - m0 : at_once);
        const float* a = A + m0 * K;
        float* c = C + m0 * N;
        const long long fours = (long long)((rows + 3) / 4) * N;
        float4* sums = reinterpret_cast<float4*>(part);
        uint2* rest = reinterpret_cast<uint2*>(sums + segments * fours);
        int rc;
#define FE_SPLIT(BN) rc = vec ? launch_split<BN, true>(a, W, bias, c, sums, rest, rows, N, K, segments, status, stream) \
                              : launch_split<BN, false>(a, W, bias, c, sums, rest, rows, N, K, segments, status, stream)
        if (rows <= 16) FE_SPLIT(16);
        else FE_SPLIT(64);
#undef FE_SPLIT
        if (rc) return rc;
        if (segments == 1) continue;
        fe::launch(add_segments_kernel, (unsigned)((fours + ADDING - 1) / ADDING), ADDING, 0, stream, (const float4*)sums, (const uint2*)rest, a, W, bias, c, rows, N, K, segments);
        rc = fe_check_launch("gemm_split (segments)");
        if (rc) return rc;
    }
    return 0;
}
