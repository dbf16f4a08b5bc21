// C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]) in true float32 on CUDA cores: no tensor cores, no
// reduced-precision mode.  Every output element is one chain of fused multiply-adds over
// k = 0..K-1 in ascending order, so a row's result does not depend on how many rows are in
// the batch nor on which of the kernels below ran.  The reference runs these products through nn.Linear in
// float32 (inference/models/qwen2.py:99-101,129-130,135 with dtype float32).
#include "common.cuh"

namespace {

__device__ __forceinline__ void copy16(void* smem_dst, const void* src, int bytes) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copy4(void* smem_dst, const void* src, int bytes) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// ---- many rows ---------------------------------------------------------------------------------------------------------
// A block owns a 128 x 128 tile of C, a thread 8 x 8 of it.  What bounds the loop is the FMA pipe, if little else takes issue
// slots, and shared memory, which gives 128 bytes a clock to the registers: 8 x 8 outputs a thread want 64 bytes for 64 multiply-adds,
// which takes as long as those do (8 x 16 want less, but leave one block an SM: 342 us where this takes 279).  Two multiply-adds an instruction (a pair of rows against one
// column), operands from shared memory as 16-byte loads (k-major tiles, so a thread's rows and columns lie side by side), the
// next k step's tiles on their way from memory into registers meanwhile and from there into the other buffer, one barrier a
// step of 16.  256 x 17,920 x 1,536: 467 us with 64 x 64 tiles of 4 x 4 and scalar loads, 279 us with 128 x 128.
constexpr int BM = 128, BN = 128, BK = 16, TM = 8, TN = 8, THREADS = (BM / TM) * (BN / TN);

template <bool VEC>
__global__ void __launch_bounds__(THREADS, 2)
gemm_fp32_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                 float* __restrict__ C, int M, int N, int K) {
    constexpr int RG = TM / 4, CG = TN / 4;              // groups of four rows / columns a thread owns, BM / RG (BN / CG) apart
    constexpr int PAD = 4;
    constexpr int A_LOADS = (BM * BK / 4 + THREADS - 1) / THREADS, W_LOADS = (BN * BK / 4 + THREADS - 1) / THREADS, Q = BK / 4;
    __shared__ __align__(16) float As[2][BK][BM + PAD];
    __shared__ __align__(16) float Ws[2][BK][BN + PAD];
    fe::griddep_wait();
    fe::griddep_launch_dependents();
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // a warp is 4 (rows) x 8 (columns) threads: its loads of a k's operands touch each bank once
    constexpr int WARPS_N = BN / TN / 8;
    const int tx = (warp % WARPS_N) * 8 + (lane & 7), ty = (warp / WARPS_N) * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    float2 acc[TM / 2][TN];
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = make_float2(0.f, 0.f);

    float4 ra[A_LOADS], rw[W_LOADS];
    // four values of row ``row``, zeros beyond the matrix
    auto four = [&](const float* __restrict__ base, int row, int rows, int k) -> float4 {
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (row < rows) {
            const float* p = base + (size_t)row * K + k;
            if (VEC) {                                   // K is a multiple of 4, rows start on 16-byte boundaries
                if (k < K) v = __ldg(reinterpret_cast<const float4*>(p));
            } else {
                if (k < K) v.x = __ldg(p);
                if (k + 1 < K) v.y = __ldg(p + 1);
                if (k + 2 < K) v.z = __ldg(p + 2);
                if (k + 3 < K) v.w = __ldg(p + 3);
            }
        }
        return v;
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            const int idx = tid + i * THREADS;
            if (idx < BM * BK / 4) ra[i] = four(A, m0 + idx / Q, M, k0 + (idx % Q) * 4);
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            const int idx = tid + i * THREADS;
            if (idx < BN * BK / 4) rw[i] = four(W, n0 + idx / Q, N, k0 + (idx % Q) * 4);
        }
    };
    auto keep = [&](int b) {
#pragma unroll
        for (int i = 0; i < A_LOADS; ++i) {
            const int idx = tid + i * THREADS, row = idx / Q, k = (idx % Q) * 4;
            if (idx < BM * BK / 4) { As[b][k][row] = ra[i].x; As[b][k + 1][row] = ra[i].y; As[b][k + 2][row] = ra[i].z; As[b][k + 3][row] = ra[i].w; }
        }
#pragma unroll
        for (int i = 0; i < W_LOADS; ++i) {
            const int idx = tid + i * THREADS, row = idx / Q, k = (idx % Q) * 4;
            if (idx < BN * BK / 4) { Ws[b][k][row] = rw[i].x; Ws[b][k + 1][row] = rw[i].y; Ws[b][k + 2][row] = rw[i].z; Ws[b][k + 3][row] = rw[i].w; }
        }
    };
    fetch(0);
    keep(0);
    __syncthreads();
    int b = 0;
    for (int k0 = 0; k0 < K; k0 += BK, b ^= 1) {
        const bool more = k0 + BK < K;
        if (more) fetch(k0 + BK);
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float2 a[TM / 2];
            float w[TN];
#pragma unroll
            for (int g = 0; g < RG; ++g) {
                const float4 v = *reinterpret_cast<const float4*>(&As[b][k][g * (BM / RG) + ty * 4]);
                a[2 * g] = make_float2(v.x, v.y), a[2 * g + 1] = make_float2(v.z, v.w);
            }
#pragma unroll
            for (int g = 0; g < CG; ++g) {
                const float4 v = *reinterpret_cast<const float4*>(&Ws[b][k][g * (BN / CG) + tx * 4]);
                w[4 * g] = v.x, w[4 * g + 1] = v.y, w[4 * g + 2] = v.z, w[4 * g + 3] = v.w;
            }
#pragma unroll
            for (int i = 0; i < TM / 2; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = __ffma2_rn(a[i], make_float2(w[j], w[j]), acc[i][j]);
        }
        if (more) keep(b ^ 1);                           // read last a step ago, before the barrier that ended it
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + (i >> 2) * (BM / RG) + ty * 4 + (i & 3);
        if (gm >= M) continue;
#pragma unroll
        for (int g = 0; g < CG; ++g) {
            const int gn = n0 + g * (BN / CG) + tx * 4;
            float v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                v[j] = (i & 1) ? acc[i >> 1][4 * g + j].y : acc[i >> 1][4 * g + j].x;
                if (bias && gn + j < N) v[j] += bias[gn + j];
            }
            float* dst = C + (size_t)gm * N + gn;
            if (VEC && gn + 4 <= N && (N & 3) == 0) *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            else
                for (int j = 0; j < 4; ++j)
                    if (gn + j < N) dst[j] = v[j];
        }
    }
}

// ---- a ring of tiles (few rows, or few tiles) ----------------------------------------------------------------------------
// What bounds these shapes is how much is on its way from memory, not the FMA rate: a decode step is a stream of W, and a
// narrow product has fewer blocks than SMs, each with a long loop.  So a block brings the rows of A and W of its tile in
// asynchronous copies through a ring of STAGES chunks of CHUNK k and every SM keeps tens of kilobytes on their way; the
// kernel above, one step of 16 k ahead in registers, took 1,800 cycles a step at one block an SM.  Rows lie in shared
// memory as in memory, a thread reads four k of a row at a time (rows CHUNK + 4 floats apart: eight of them touch each
// bank once).
template <int BM, int BN, int TM, int TN, int STAGES, int CHUNK, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN))
gemm_fp32_ring_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                      float* __restrict__ C, int M, int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / TN), TX = BN / TN, TY = BM / TM;
    constexpr int PITCH = CHUNK + 4, STAGE = (BM + BN) * PITCH;
    constexpr int AHEAD = TM * TN <= 4 ? 4 : 1;          // a short chain of its own: four 16-byte loads of a row go out together
    extern __shared__ __align__(16) float ring_smem[];
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int chunks = (K + CHUNK - 1) / CHUNK;
    auto start = [&](int i) {
        if (i < chunks) {
            float* dst = ring_smem + (i % STAGES) * STAGE;
            const int k0 = i * CHUNK;
            constexpr int PER = VEC ? CHUNK / 4 : CHUNK, WIDTH = VEC ? 4 : 1;
#pragma unroll
            for (int idx = tid; idx < (BM + BN) * PER; idx += THREADS) {
                const int r = idx / PER, c = (idx % PER) * WIDTH;
                const bool of_w = r < BN;
                const int row = of_w ? n0 + r : m0 + r - BN;
                const float* base = of_w ? W : A;
                const bool real = row < (of_w ? N : M) && k0 + c < K;
                const float* src = real ? base + (size_t)row * K + k0 + c : base;
                if (VEC) copy16(dst + r * PITCH + c, src, real ? 16 : 0);
                else copy4(dst + r * PITCH + c, src, real ? 4 : 0);
            }
        }
        copies_commit();
    };
    fe::griddep_wait();
    fe::griddep_launch_dependents();
#pragma unroll
    for (int i = 0; i < STAGES - 1; ++i) start(i);
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int i = 0; i < chunks; ++i) {
        copies_wait<STAGES - 2>();
        __syncthreads();                                 // chunk i is there for all, and chunk i - 1 has been read by all
        start(i + STAGES - 1);
        const float* w_s = ring_smem + (i % STAGES) * STAGE + tx * PITCH;
        const float* a_s = ring_smem + (i % STAGES) * STAGE + (BN + ty) * PITCH;
#pragma unroll
        for (int k = 0; k < CHUNK; k += 4 * AHEAD) {
            float4 a[AHEAD][TM], w[AHEAD][TN];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
#pragma unroll
                for (int r = 0; r < TM; ++r) a[u][r] = *reinterpret_cast<const float4*>(a_s + r * TY * PITCH + k + 4 * u);
#pragma unroll
                for (int c = 0; c < TN; ++c) w[u][c] = *reinterpret_cast<const float4*>(w_s + c * TX * PITCH + k + 4 * u);
            }
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) {
#pragma unroll
                for (int r = 0; r < TM; ++r)
#pragma unroll
                    for (int c = 0; c < TN; ++c) acc[r][c] = fmaf(a[u][r].x, w[u][c].x, acc[r][c]);
#pragma unroll
                for (int r = 0; r < TM; ++r)
#pragma unroll
                    for (int c = 0; c < TN; ++c) acc[r][c] = fmaf(a[u][r].y, w[u][c].y, acc[r][c]);
#pragma unroll
                for (int r = 0; r < TM; ++r)
#pragma unroll
                    for (int c = 0; c < TN; ++c) acc[r][c] = fmaf(a[u][r].z, w[u][c].z, acc[r][c]);
#pragma unroll
                for (int r = 0; r < TM; ++r)
#pragma unroll
                    for (int c = 0; c < TN; ++c) acc[r][c] = fmaf(a[u][r].w, w[u][c].w, acc[r][c]);
            }
        }
    }
    copies_wait<0>();
#pragma unroll
    for (int r = 0; r < TM; ++r) {
        const int m = m0 + ty + r * TY;
        if (m >= M) continue;
#pragma unroll
        for (int c = 0; c < TN; ++c) {
            const int n = n0 + tx + c * TX;
            if (n < N) C[(size_t)m * N + n] = acc[r][c] + (bias ? bias[n] : 0.f);
        }
    }
}

// ---- few columns (a router, a low-rank projection) for any number of rows, and few rows where the rings do not pay -------------
// A block of 128 threads owns 8 rows x 16 columns, one output a thread, and walks K in chunks of 64 that it stages in
// shared memory: the tiles above would be few blocks with long loops.
constexpr int SR = 8, SC = 16, SK = 64;

__global__ void __launch_bounds__(128)
gemm_fp32_narrow_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                        float* __restrict__ C, int M, int N, int K) {
    fe::griddep_wait();
    fe::griddep_launch_dependents();
    __shared__ __align__(16) float As[SR][SK];
    __shared__ __align__(16) float Ws[SC][SK + 4];
    const int tid = threadIdx.x;
    const int m = tid / SC, n = tid % SC;
    const int m0 = blockIdx.y * SR, n0 = blockIdx.x * SC;
    // the next chunk is on its way from global memory into registers while this one is multiplied
    float next_a[(SR * SK) / 128], next_w[(SC * SK) / 128];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < (SR * SK) / 128; ++i) {
            const int idx = tid + i * 128;
            const int r = idx / SK, c = idx % SK;
            const bool real = m0 + r < M && k0 + c < K;
            next_a[i] = real ? A[(size_t)(m0 + r) * K + k0 + c] : 0.f;
        }
#pragma unroll
        for (int i = 0; i < (SC * SK) / 128; ++i) {
            const int idx = tid + i * 128;
            const int r = idx / SK, c = idx % SK;
            const bool real = n0 + r < N && k0 + c < K;
            next_w[i] = real ? W[(size_t)(n0 + r) * K + k0 + c] : 0.f;
        }
    };
    float acc = 0.f;
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += SK) {
#pragma unroll
        for (int i = 0; i < (SR * SK) / 128; ++i) {
            const int idx = tid + i * 128;
            As[idx / SK][idx % SK] = next_a[i];
        }
#pragma unroll
        for (int i = 0; i < (SC * SK) / 128; ++i) {
            const int idx = tid + i * 128;
            Ws[idx / SK][idx % SK] = next_w[i];
        }
        __syncthreads();
        if (k0 + SK < K) fetch(k0 + SK);
#pragma unroll
        for (int k = 0; k < SK; k += 4) {           // four at a time from shared memory; the chain stays in ascending k
            const float4 a = *reinterpret_cast<const float4*>(&As[m][k]);
            const float4 w = *reinterpret_cast<const float4*>(&Ws[n][k]);
            acc = fmaf(a.x, w.x, acc);
            acc = fmaf(a.y, w.y, acc);
            acc = fmaf(a.z, w.z, acc);
            acc = fmaf(a.w, w.w, acc);
        }
        __syncthreads();
    }
    if (m0 + m < M && n0 + n < N) C[(size_t)(m0 + m) * N + n0 + n] = acc + (bias ? bias[n0 + n] : 0.f);
}

// ---- rows that start on no 16-byte boundary ------------------------------------------------------------------------------
// A block of 256 threads owns 64 x 64 of C, a thread 4 x 4 of it; every value of a step of 16 is a load of its own, which is all
// that such rows allow, and the many blocks an SM hide them better than the larger tiles' few or a ring of 4-byte copies.
constexpr int UM = 64, UN = 64, UK = 16, UT = 4;

__global__ void __launch_bounds__(256)
gemm_fp32_unaligned_kernel(const float* __restrict__ A, const float* __restrict__ W, const float* __restrict__ bias,
                           float* __restrict__ C, int M, int N, int K) {
    fe::griddep_wait();
    fe::griddep_launch_dependents();
    __shared__ float As[UK][UM + 4];
    __shared__ float Ws[UK][UN + 4];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = blockIdx.y * UM, n0 = blockIdx.x * UN;
    float acc[UT][UT];
#pragma unroll
    for (int i = 0; i < UT; ++i)
#pragma unroll
        for (int j = 0; j < UT; ++j) acc[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += UK) {
#pragma unroll
        for (int i = 0; i < UM * UK / 256; ++i) {
            const int idx = tid + i * 256, row = idx / UK, col = idx % UK;
            const int gm = m0 + row, gn = n0 + row, gk = k0 + col;
            As[col][row] = (gm < M && gk < K) ? A[(size_t)gm * K + gk] : 0.f;
            Ws[col][row] = (gn < N && gk < K) ? W[(size_t)gn * K + gk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < UK; ++k) {
            float a[UT], w[UT];
#pragma unroll
            for (int i = 0; i < UT; ++i) a[i] = As[k][ty * UT + i];
#pragma unroll
            for (int j = 0; j < UT; ++j) w[j] = Ws[k][tx * UT + j];
#pragma unroll
            for (int i = 0; i < UT; ++i)
#pragma unroll
                for (int j = 0; j < UT; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < UT; ++i) {
        const int gm = m0 + ty * UT + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < UT; ++j) {
            const int gn = n0 + tx * UT + j;
            if (gn < N) C[(size_t)gm * N + gn] = acc[i][j] + (bias ? bias[gn] : 0.f);
        }
    }
}

template <int BM, int BN, int TM, int TN, int STAGES, int CHUNK, bool VEC>
int launch_ring(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    constexpr size_t smem = (size_t)STAGES * (BM + BN) * (CHUNK + 4) * sizeof(float);
    const cudaError_t err = cudaFuncSetAttribute(gemm_fp32_ring_kernel<BM, BN, TM, TN, STAGES, CHUNK, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    FE_REQUIRE(err == cudaSuccess, "gemm_fp32: %s", cudaGetErrorString(err));
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    FE_REQUIRE(grid.y <= 65535, "gemm_fp32: too many rows (%d)", M);
    fe::launch(gemm_fp32_ring_kernel<BM, BN, TM, TN, STAGES, CHUNK, VEC>, grid, (BM / TM) * (BN / TN), smem, stream, A, W, bias, C, M, N, K);
    return fe_check_launch("gemm_fp32 (ring)");
}

int launch_narrow(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + SC - 1) / SC, (M + SR - 1) / SR);
    FE_REQUIRE(grid.y <= 65535, "gemm_fp32: too many rows (%d)", M);
    fe::launch(gemm_fp32_narrow_kernel, grid, 128, 0, stream, A, W, bias, C, M, N, K);
    return fe_check_launch("gemm_fp32 (narrow)");
}

// Up to 16 rows: whether blocks of 8 rows and 16 columns are done before the rings' (the same bits either way).  The lines lie
// where the rings' blocks go into another round over the SMs and these do not, or where a copy takes more than it brings:
//   rows of 16 bytes: K of one chunk from three rows on (5 rows x 4,864 x 64: 3.0 us, ring 3.7); 5 to 8 rows a little over a
//     round of the ring's 32 columns (x 4,864 x 2,048: 28.3, ring 32.3; x 8,000: 36.3 against 32.7); 9 to 16 rows with these
//     blocks on different SMs (x 1,152 x 2,048: 15.9 against 18.8; x 1,536: 22.9 against 18.8), or the ring's 16 columns, one
//     block an SM, in their second round (x 3,072: 28.9 against 34.2; x 4,864: 44.8 against 33.0)
//   other rows, whose ring takes a copy for every value: nearly always (16 rows x 515 x 515: 5.9 us, ring 13.2; 8 x 40,000 x 131:
//     16.0 against 26.2), but for four rows in the middle (x 10,000 x 515: 14.3 against 11.1) and for 9 to 16 rows of many
//     columns, which these blocks fetch twice (x 10,000 x 1,539: 61.8 against 43.8; from twice as many on with a short K)
template <bool VEC>
bool narrow_pays(int M, int N, int K) {
    const int sms = fe_sm_count();
    if (VEC) {
        if (K <= SK) return M > 2 && N <= (M <= 8 ? 128 : 64) * sms;
        if (M <= 8) return M > 4 && N > 32 * sms && N <= 44 * sms;
        return N <= 8 * sms || (N > 16 * sms && N <= 32 * sms);
    }
    if (M <= 4) return N <= 44 * sms || N > 256 * sms;
    return M <= 8 || N <= (K <= 256 ? 64 : 32) * sms;
}

template <bool VEC>
int few_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    if (narrow_pays<VEC>(M, N, K)) return launch_narrow(A, W, bias, C, M, N, K, stream);
    // 16 columns a block while 32 would leave SMs without one; a deeper ring there (fewer blocks an SM).  A vocabulary's worth of
    // columns fills the device with blocks of 128 columns, whose threads use each value of W for four rows or more.  As few
    // threads a block as the rows allow: what a block reads from shared memory is what its threads' outputs do not share.
    const int sms = fe_sm_count();
    if constexpr (VEC) {
        if (N <= 32 * sms) {
            if (M <= 4) return launch_ring<4, 16, 1, 1, 8, 128, VEC>(A, W, bias, C, M, N, K, stream);
            if (M <= 8) return launch_ring<8, 16, 2, 1, 8, 128, VEC>(A, W, bias, C, M, N, K, stream);
            return launch_ring<16, 16, 2, 2, 8, 128, VEC>(A, W, bias, C, M, N, K, stream);
        }
        if (N <= 256 * sms && M > 4 && M <= 8) return launch_ring<8, 32, 2, 2, 4, 64, VEC>(A, W, bias, C, M, N, K, stream);
        if (N > 256 * sms) {
            if (M <= 4) return launch_ring<4, 128, 4, 1, 3, 64, VEC>(A, W, bias, C, M, N, K, stream);
            if (M <= 8) return launch_ring<8, 128, 8, 1, 3, 64, VEC>(A, W, bias, C, M, N, K, stream);
        }
    }
    if (M <= 4) return launch_ring<4, 32, 2, 1, 4, 64, VEC>(A, W, bias, C, M, N, K, stream);
    return launch_ring<16, 32, 4, 2, 4, 64, VEC>(A, W, bias, C, M, N, K, stream);
}

template <bool VEC>
int launch_tiles(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    FE_REQUIRE(grid.y <= 65535, "gemm_fp32: too many rows (%d)", M);
    fe::launch(gemm_fp32_kernel<VEC>, grid, THREADS, 0, stream, A, W, bias, C, M, N, K);
    return fe_check_launch("gemm_fp32");
}

int launch_unaligned(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    const dim3 grid((N + UN - 1) / UN, (M + UM - 1) / UM);
    FE_REQUIRE(grid.y <= 65535, "gemm_fp32: too many rows (%d)", M);
    fe::launch(gemm_fp32_unaligned_kernel, grid, 256, 0, stream, A, W, bias, C, M, N, K);
    return fe_check_launch("gemm_fp32 (unaligned rows)");
}

// The tile whose blocks are done first: rounds of blocks over the SMs times what a block takes, which is its area over
// how close to the FMA rate it comes (measured: alone on an SM, and where the SMs hold two or more; per mille for rows of 16 bytes).
struct Shape { int bm, bn, alone, several; };
inline int first_done(const Shape* shapes, int count, int M, int N) {
    const int sms = fe_sm_count();
    int best = 0;
    long long least = 0;
    for (int i = 0; i < count; ++i) {
        const Shape& s = shapes[i];
        const long long tiles = (long long)((M + s.bm - 1) / s.bm) * ((N + s.bn - 1) / s.bn), rounds = (tiles + sms - 1) / sms;
        const long long cost = rounds * 1000LL * s.bm * s.bn / (rounds > 1 ? s.several : s.alone);
        if (i == 0 || cost < least) best = i, least = cost;
    }
    return best;
}

int many_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    static constexpr Shape SHAPES[6] = {{128, 128, 690, 720}, {64, 48, 460, 530}, {64, 32, 390, 485},
                                        {32, 64, 380, 490}, {32, 32, 300, 430}, {32, 16, 170, 290}};
    switch (first_done(SHAPES, 6, M, N)) {
        case 0: return launch_tiles<true>(A, W, bias, C, M, N, K, stream);
        case 1: return launch_ring<64, 48, 4, 6, 3, 64, true>(A, W, bias, C, M, N, K, stream);
        case 2: return launch_ring<64, 32, 4, 4, 4, 64, true>(A, W, bias, C, M, N, K, stream);
        case 3: return launch_ring<32, 64, 4, 4, 3, 64, true>(A, W, bias, C, M, N, K, stream);
        case 4: return launch_ring<32, 32, 4, 2, 4, 64, true>(A, W, bias, C, M, N, K, stream);
        default: return launch_ring<32, 16, 4, 1, 4, 64, true>(A, W, bias, C, M, N, K, stream);
    }
}

// Rows that start on no 16-byte boundary: the tiles' order is another, since a ring's copies are of four bytes (relative rates
// over 132 sizes with K of 131 to 1,539: within 2 % of the best of them on average, nowhere behind the 64 x 64 tiles.  33 rows x
// 40,000 x 131: 42 us, by the rates of aligned rows 49; 129 rows: 102, 134; 300 x 3,072 x 515: 64, 69).
int many_unaligned_rows(const float* A, const float* W, const float* bias, float* C, int M, int N, int K, cudaStream_t stream) {
    static constexpr Shape SHAPES[5] = {{128, 128, 130, 167}, {64, 48, 42, 66}, {32, 32, 43, 49}, {32, 16, 26, 45}, {UM, UN, 66, 82}};
    switch (first_done(SHAPES, 5, M, N)) {
        case 0: return launch_tiles<false>(A, W, bias, C, M, N, K, stream);
        case 1: return launch_ring<64, 48, 4, 6, 3, 64, false>(A, W, bias, C, M, N, K, stream);
        case 2: return launch_ring<32, 32, 4, 2, 4, 64, false>(A, W, bias, C, M, N, K, stream);
        case 3: return launch_ring<32, 16, 4, 1, 4, 64, false>(A, W, bias, C, M, N, K, stream);
        default: return launch_unaligned(A, W, bias, C, M, N, K, stream);
    }
}

}  // namespace

extern "C" int fe_gemm_fp32(const float* A, const float* W, const float* bias, float* C, int M, int N, int K,
                            cudaStream_t stream) {
    FE_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_fp32: bad sizes M=%d N=%d K=%d", M, N, K);
    if (M == 0) return 0;
    const bool vec = (K & 3) == 0 && (((size_t)A | (size_t)W | (size_t)C) & 15) == 0;
    if (M <= 16)
        return vec ? few_rows<true>(A, W, bias, C, M, N, K, stream) : few_rows<false>(A, W, bias, C, M, N, K, stream);
    if (N <= 128) return launch_narrow(A, W, bias, C, M, N, K, stream);
    return vec ? many_rows(A, W, bias, C, M, N, K, stream) : many_unaligned_rows(A, W, bias, C, M, N, K, stream);
}
