// y[M, N] = x[M, K] . W[N, K]^T for a handful of rows (decode): the product is a stream of the
// weight matrix, so the kernel is built around reading W once at full HBM speed.
//
// One block takes 16 rows of W (swap-AB: the rows of W are the 16 rows of mma.sync.m16n8k16,
// the batch is its 8 columns).  Its eight warps split K; every lane reads 32 contiguous bytes
// of "its" two W rows per step straight into MMA fragments.  The fragment layout wants
// k = {2t, 2t+1, 2t+8, 2t+9} per lane; since a dot product does not care in which order k is
// summed, lane t instead takes the 16 contiguous elements k0 + 16t .. +15 of a 64-wide step and
// the activations are read with the same pattern, so both operands are 16-byte loads.  The eight
// partial sums of a block are added in shared memory in a fixed order (deterministic).
//
// Epilogues: bfloat16 output; float output (vocabulary projection); SwiGLU, where a block pairs
// 8 gate rows with their 8 up rows of a [2I, K] matrix and writes silu(gate) * up; the fused
// query/key/value epilogue; and the residual epilogue, which ends a branch of a layer and begins
// the norm that follows it (below).
// The reference runs these products through cuBLAS (inference/models/qwen2.py:99-101,129-135).
//
// Residual add and RMSNorm without a kernel of their own.  In a decode step a norm moves a few kilobytes
// between two products that stream hundreds of megabytes; as a kernel it costs a launch and a few trips to
// memory.  Instead the product that ends a branch (output projection, down projection) adds its result to the
// float residual stream in its epilogue, writes the new residual times the next norm's weight as bfloat16,
// and leaves each block's share of the rows' sums of squares in a small table; the product that consumes the
// norm (query/key/value, gate/up) adds the table up in a fixed order while its first weights are on their way
// and multiplies its accumulators by rsqrt(mean square + eps): a row's scale is a factor of every term of its
// dot products, so it may be applied after them.
#define FE_PDL_CLASS 1      // FE_PDL_STREAMING_GEMM
#include <cuda.h>
#include <atomic>

#include "common.cuh"

using namespace fe;

namespace {

constexpr int WARPS = 8;
constexpr int KSTEP = 32;       // k elements of a step (2 MMAs); the stream brings two steps at a time: 128 bytes of a row
constexpr int LARGE_RING = 13312, SMALL_RING = 10240, MAX_DEPTH = 8;        // bytes (and units) of a warp's ring

enum { EPI_BF16 = 0, EPI_F32 = 1, EPI_SWIGLU = 2, EPI_QKV = 3, EPI_RESID = 4, EPI_GEGLU = 5, EPI_RELU2 = 6, EPI_REGLU = 7, EPI_GELU = 8 };   // 5: gated, the tanh form of GELU
constexpr int ACT_RELU2 = 3;            // ``gate_act`` of the bfloat16 epilogue: the square of relu(product), no gate (entry code 6)
constexpr int ACT_RELU = 4;             // ``gate_act`` of the gated epilogue: relu (entry code 7)
constexpr int ACT_GELU = 5;             // ``gate_act`` of the bfloat16 epilogue: the exact GELU of the product, no gate (entry code 8)

// The gate's function of the gated epilogue: 0 silu, 1 the tanh form of GELU, z/2 (1 + tanh(sqrt(2/pi) (z + 0.044715 z^3))).
__device__ __forceinline__ float gate_function(float z, int act) {
    return act == 0 ? z / (1.f + expf(-z)) : act == ACT_RELU ? fmaxf(z, 0.f) : 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}

// The residual epilogue: out[m][n] is not written; residual[m][n] += product, scaled[m][n] = bfloat16(residual *
// norm_weight[n]), sumsq[tile][m] = this tile's share of the sum of squares of row m of the new residual.
struct ResidEpilogue {
    float* residual;            // [M, N] float, updated in place (every element by the one block that owns it)
    const float* norm_weight;   // [N]
    bf16* scaled;               // [M, N]
    float* sumsq;               // [tiles of 16 columns][8]
};

// What a consumer of such a norm gets instead of normalised rows: the table of partial sums of squares.
// ``next``: memory that the kernel after this one streams first (may be null): as a block leaves its loop it asks for its
// share of the first ``next_bytes`` to be brought into L2, so that the next kernel's first loads, which would
// otherwise go out to an idle memory system after the launch gap, are met there.
// ``held``: W belongs to a model, whose steps begin with other kernels: it stands in memory before the kernel ahead of this one
// began.  Any other W may be that very kernel's output, and is read when that has ended, like x.
struct RowScale {
    const float* sumsq;         // [tiles][8] or nullptr: the input is normalised already
    int tiles;
    float eps;
    int width;                  // elements of a row (the mean is over them)
    const void* next;
    long long next_bytes;
    int held, beside;
};

// What the fused query/key/value epilogue needs beside the product: bias, rotary table, where the
// new keys and values go in the paged cache (see elementwise.cu for the unfused form of the same).
struct QkvEpilogue {
    const float* bias;          // [(nq + 2 nkv) d] or nullptr
    const int* positions;       // [M]
    const float* inv_freq;      // [d / 2]
    const int* slot_mapping;    // [M] or nullptr (no cache write)
    bf16* kc;
    bf16* vc;
    int nq, nkv, d, ps;
    long long num_slots;
    int* status;
};

__device__ __forceinline__ void mma16816(float* c, unsigned a0, unsigned a1, unsigned a2, unsigned a3, unsigned b0,
                                         unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ld_shared16(unsigned at) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ bool bar_test(unsigned bar, unsigned parity) {
    unsigned ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
constexpr long long WAIT_LIMIT = 4000000000LL;      // clock cycles

// Where accumulator (row 0..15, column 0..7) of a tile lies among the tile's 128 floats of shared memory: the writes of a
// fragment's lanes and the reads of 16 (or 8) rows a column each fall on 32 banks.
__device__ __forceinline__ int red_at(int row, int col) {
    return (col >> 1) * 32 + (((col ^ (col >> 2)) & 1) << 4) + (row ^ ((col & 2) << 2));
}

constexpr int RED_FLOATS = 4 * 128;      // accumulator tiles a warp leaves at a time x their floats

// How a launch cuts the matrix: ``items`` (rows, or pairs of rows) over the blocks, a block's (or a warp's) in groups of at most ``rows`` of
// them; a unit of the stream is ``rows`` items x KB steps of k, ``plane`` bytes two steps, ``slot`` bytes in all, ``depth`` units a warp's ring.
// Rows of 128 bytes, since the copy engine takes about as long for a row of 64 (271 MB: 54 us), swizzled.
struct Cut {
    int items, rows, plane, slot, depth, ring;
};

// TILES: the 16-row tiles a group has at most (1 or 2); KB = 4 / TILES steps of k are one unit, so that a unit is always four
// (tile, step) pairs: eight 16-byte reads and eight multiplications that wait for one another in pairs at most.
// ONE: a single row of x.  WIDE: a block has so many items that every warp takes an eighth of them over all of K, adds nothing up with
// the others and meets them at no barrier; else the warps share K.
template <int NT, int EPI, bool ONE, int TILES, bool WIDE>
__global__ void __launch_bounds__(WARPS * 32, NT == 1 ? 2 : 1)
skinny_gemm_kernel(const __grid_constant__ CUtensorMap map, const bf16* __restrict__ x, void* __restrict__ out, const int M, const int N, const int K,
                   const Cut cut, const QkvEpilogue qkv, const ResidEpilogue resid, const RowScale scale, const int gate_act, int* __restrict__ status) {
    constexpr bool PAIRS = EPI == EPI_SWIGLU || EPI == EPI_QKV;
    constexpr int ITEMS = PAIRS ? 8 : 16;         // items a tile takes: pairs of rows, or rows
    constexpr int KB = 4 / TILES, AHEAD = 8 / KB;           // AHEAD: units whose rows of x are on their way
    extern __shared__ __align__(1024) unsigned char shared[];
    __shared__ __align__(8) unsigned long long bars[WARPS][MAX_DEPTH];
    __shared__ float scale_part[WARPS][8];
    __shared__ float square_part[TILES][8];
    float* const red = reinterpret_cast<float*>(shared + WARPS * cut.ring);       // [WARPS][RED_FLOATS]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
    // the block's groups of items; for queries, keys and values a group lies within a head
    const int block0 = (int)((long long)cut.items * blockIdx.x / gridDim.x), block1 = (int)((long long)cut.items * (blockIdx.x + 1) / gridDim.x);
    const int item0 = EPI == EPI_QKV ? 0 : WIDE ? block0 + (block1 - block0) * warp / WARPS : block0;
    const int item1 = EPI == EPI_QKV ? cut.items : WIDE ? block0 + (block1 - block0) * (warp + 1) / WARPS : block1;
    const int first_item = EPI == EPI_QKV ? (int)blockIdx.x * cut.rows : item0, group_step = EPI == EPI_QKV ? (int)gridDim.x * cut.rows : cut.rows;
    // a warp's share of the units along K
    const int units = (K / KSTEP + KB - 1) / KB;
    const int u_begin = WIDE ? 0 : warp * units / WARPS, u_end = WIDE ? units : (warp + 1) * units / WARPS;

    // ---- the stream of weights: one lane a warp asks for units, into the warp's own ring ------------------------------
    const unsigned ring = smem_u32(shared) + warp * cut.ring, bar0 = smem_u32(&bars[warp][0]);
    if (lane == 0) {
        for (int i = 0; i < MAX_DEPTH; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(bar0 + 8 * i) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    __syncwarp();
    int at_item = u_begin < u_end ? first_item : item1, at_u = u_begin;
    auto issue = [&](int slot) {                  // lane 0
        if (at_item >= item1) return;
        const unsigned bar = bar0 + 8 * slot, dst = ring + slot * cut.slot;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(cut.plane * (KB / 2)) : "memory");
        if constexpr (EPI == EPI_SWIGLU) {
            asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];\n"
                         ::"r"(dst), "l"(&map), "r"(bar), "r"(0), "r"(at_item), "r"(0), "r"(at_u * (KB / 2)) : "memory");
        } else if constexpr (EPI == EPI_QKV) {
            const int half = qkv.d >> 1, head = at_item / half;
            asm volatile("cp.async.bulk.tensor.5d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, %7}], [%2];\n"
                         ::"r"(dst), "l"(&map), "r"(bar), "r"(0), "r"(at_item - head * half), "r"(0), "r"(head), "r"(at_u * (KB / 2)) : "memory");
        } else {
            asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];\n"
                         ::"r"(dst), "l"(&map), "r"(bar), "r"(0), "r"(at_item), "r"(at_u * (KB / 2)) : "memory");
        }
        if (++at_u == u_end) {
            at_u = u_begin;
            at_item += group_step;
        }
    };
    if (!scale.held) griddep_wait();
    if (lane == 0)
        for (int s = 0; s < cut.depth; ++s) issue(s);
    if (scale.held) griddep_wait();
    griddep_launch_dependents();

    // ---- what the previous kernel wrote ---------------------------------------------------------------------------------
    // ONE row: a lane's register set holds step g of eight of them (a load then brings 512 bytes of the row, SETS of them are on their
    // way at once) and a step's fragments come from its four lanes by shuffles; the product's other seven columns repeat the row.
    constexpr int SETS = 5;
    const int k_begin = u_begin * KB, k_end = min(u_end * KB, K / KSTEP);        // in steps
    uint4 xs[ONE ? SETS : 1], xa[ONE ? 1 : 8][NT];
    const bf16* xr[NT];
    auto load_set = [&](int k) {
        return k + g < k_end ? __ldcg(reinterpret_cast<const uint4*>(x + (size_t)(k + g) * KSTEP + 8 * t)) : make_uint4(0, 0, 0, 0);
    };
    // step ``k`` of this group into place i of eight, or, past the group's end, the step that the next group begins with there
    auto load_step = [&](int i, int k) {
        if (k >= k_end) k = k_begin + i;
#pragma unroll
        for (int nt = 0; nt < NT; ++nt)
            xa[i][nt] = xr[nt] != nullptr && k < k_end ? __ldcg(reinterpret_cast<const uint4*>(xr[nt] + (size_t)k * KSTEP)) : make_uint4(0, 0, 0, 0);
    };
    int set_k = k_begin;                          // ONE: the first step of the set that is loaded next; the groups follow one another in a ring
    auto next_set = [&]() {
        const uint4 v = load_set(set_k);
        set_k += 8;
        if (set_k >= k_end) set_k = k_begin;
        return v;
    };
#pragma unroll
    for (int nt = 0; nt < NT; ++nt) xr[nt] = nt * 8 + g < M ? x + (size_t)(nt * 8 + g) * K + 8 * t : nullptr;
    if constexpr (ONE) {
#pragma unroll
        for (int i = 0; i < SETS; ++i) xs[i] = next_set();
    } else {
#pragma unroll
        for (int i = 0; i < 8; ++i) load_step(i, k_begin + i);
    }
    // a thread's column of the batch in the epilogues of one column tile: the same for every group
    const int my_m = PAIRS ? (tid >> 3) & 7 : (tid >> 4) & 7;
    if (scale.sumsq != nullptr) {
        // thread = (row m, a share of the table): its entries in ascending order, then the shares in a fixed order
        float sum = 0.f;
        for (int part = tid >> 3; part < scale.tiles; part += WARPS * 4) sum += __ldcg(scale.sumsq + (size_t)part * 8 + (tid & 7));
        sum += __shfl_xor_sync(0xffffffffu, sum, 8);
        sum += __shfl_xor_sync(0xffffffffu, sum, 16);
        if (lane < 8) scale_part[warp][lane] = sum;
    }
    float row_scale = 1.f, squares = 0.f, scales[2] = {1.f, 1.f};
    int slot = 0;
    unsigned parity = 0;
    bool dead = false;                            // a wait has run out: no more waiting, the status word says so

    for (int start = first_item; start < item1; start += group_step) {
        const int end = EPI == EPI_QKV ? start + cut.rows : min(start + cut.rows, item1), n = (end - start + ITEMS - 1) / ITEMS;
        const bool first = start == first_item, more = start + group_step < item1;
        // what the residual epilogue reads, asked for before the products
        float before[2] = {0.f, 0.f}, weight[2] = {0.f, 0.f};
        if (EPI == EPI_RESID) {
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int idx = tid + i * WARPS * 32, col = start + (idx >> 7) * 16 + (idx & 15);
                if (idx < n * 128 && my_m < M && col < end) {
                    before[i] = __ldcg(resid.residual + (size_t)my_m * N + col);
                    weight[i] = __ldg(resid.norm_weight + col);
                }
            }
        }
        constexpr int CHAINS = TILES == 1 ? 2 : TILES;          // a tile alone: two chains of multiplications instead of one
        float acc[CHAINS][NT][4];
#pragma unroll
        for (int r = 0; r < CHAINS; ++r)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt) acc[r][nt][0] = acc[r][nt][1] = acc[r][nt][2] = acc[r][nt][3] = 0.f;
#pragma unroll 1
        for (int u0 = u_begin; u0 < u_end; u0 += AHEAD) {
#pragma unroll
            for (int v = 0; v < AHEAD; ++v) {
                if (u0 + v >= u_end) break;
                const unsigned bar = bar0 + 8 * slot;
                if (!bar_test(bar, parity) && !dead) {
                    const long long since = clock64();
                    while (!bar_test(bar, parity))
                        if (clock64() - since > WAIT_LIMIT) { dead = true; break; }
                }
                const unsigned from = ring + slot * cut.slot;
                uint4 a0[KB][TILES], a1[KB][TILES];
                // row ``r`` of a unit: its 16-byte piece c lies at c ^ (r & 7).  Lanes of odd and even rows that read together take the row's two
                // halves in opposite order, so that they meet on no bank
                auto two_steps = [&](int r, uint4& first, uint4& second) {
                    const unsigned at = from + r * 128, odd = r & 1;
                    const uint4 one = ld_shared16(at + (((t + 4 * odd) ^ (r & 7)) << 4)), two = ld_shared16(at + (((t + 4 - 4 * odd) ^ (r & 7)) << 4));
                    first = odd ? two : one;
                    second = odd ? one : two;
                };
#pragma unroll
                for (int pl = 0; pl < KB / 2; ++pl)
#pragma unroll
                    for (int j = 0; j < TILES; ++j) {
                        const int r = pl * cut.rows * (PAIRS ? 2 : 1) + j * ITEMS + g;
                        two_steps(r, a0[2 * pl][j], a0[2 * pl + 1][j]);
                        two_steps(r + (PAIRS ? cut.rows : 8), a1[2 * pl][j], a1[2 * pl + 1][j]);
                    }
#pragma unroll
                for (int kk = 0; kk < KB; ++kk) {
                    const int step = v * KB + kk;             // of the eight whose rows of x are here
                    uint4 b[NT];
                    if constexpr (ONE) {
                        const int src = step * 4 + t;
                        b[0] = make_uint4(__shfl_sync(0xffffffffu, xs[0].x, src), __shfl_sync(0xffffffffu, xs[0].y, src),
                                          __shfl_sync(0xffffffffu, xs[0].z, src), __shfl_sync(0xffffffffu, xs[0].w, src));
                    } else {
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) b[nt] = xa[step][nt];
                    }
#pragma unroll
                    for (int j = 0; j < TILES; ++j)
#pragma unroll
                        for (int nt = 0; nt < NT; ++nt) {
                            float* c = acc[TILES == 1 ? kk & 1 : j][nt];
                            mma16816(c, a0[kk][j].x, a1[kk][j].x, a0[kk][j].y, a1[kk][j].y, b[nt].x, b[nt].y);
                            mma16816(c, a0[kk][j].z, a1[kk][j].z, a0[kk][j].w, a1[kk][j].w, b[nt].z, b[nt].w);
                        }
                    if constexpr (!ONE) load_step(step, (u0 + AHEAD + v) * KB + kk);
                }
                __syncwarp();                                 // every lane has read the slot
                if (lane == 0) issue(slot);
                if (++slot == cut.depth) slot = 0, parity ^= 1;
            }
            if constexpr (ONE) {                              // the next eight steps
#pragma unroll
                for (int i = 0; i + 1 < SETS; ++i) xs[i] = xs[i + 1];
                xs[SETS - 1] = next_set();
            }
        }
        if (TILES == 1) {
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) acc[0][nt][e] += acc[CHAINS - 1][nt][e];
        }
        if constexpr (WIDE) {
            if (scale.sumsq != nullptr && first) {
                __syncthreads();                  // the shares of the rows' sums are there
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    float sum = 0.f;
#pragma unroll
                    for (int w = 0; w < WARPS; ++w) sum += scale_part[w][2 * t + c];
                    scales[c] = rsqrtf(sum / (float)scale.width + scale.eps);
                }
            }
#pragma unroll
            for (int j = 0; j < TILES; ++j)
#pragma unroll
                for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                    for (int c = 0; c < 2; ++c) {
                        const int m = nt * 8 + 2 * t + c;
                        const float lo = acc[j][nt][c] * scales[c], hi = acc[j][nt][2 + c] * scales[c];       // accumulator rows g and g + 8
                        if (m >= M) continue;
                        if (EPI == EPI_SWIGLU) {
                            const int item = start + j * 8 + g;
                            if (item < end) reinterpret_cast<bf16*>(out)[(size_t)m * cut.items + item] = __float2bfloat16_rn(gate_function(lo, gate_act) * hi);
                        } else {
#pragma unroll
                            for (int h = 0; h < 2; ++h) {
                                const int col = start + j * 16 + g + 8 * h;
                                float v = h ? hi : lo;
                                if (col >= end) continue;
                                if (EPI == EPI_BF16 && gate_act == ACT_RELU2) v = v > 0.f ? v * v : 0.f;
                                if (EPI == EPI_BF16 && gate_act == ACT_GELU) v = gelu_erf(v);
                                if (EPI == EPI_F32) reinterpret_cast<float*>(out)[(size_t)m * N + col] = v;
                                else reinterpret_cast<bf16*>(out)[(size_t)m * N + col] = __float2bfloat16_rn(v);
                            }
                        }
                    }
            continue;
        }
        float* const mine = red + warp * RED_FLOATS;
        if (!first) __syncthreads();              // the group before has been read out of ``red``
#pragma unroll
        for (int r = 0; r < TILES; ++r)
#pragma unroll
            for (int nt = 0; nt < NT; ++nt)
#pragma unroll
                for (int e = 0; e < 4; ++e) mine[(r * NT + nt) * 128 + red_at(g + 8 * (e >> 1), 2 * t + (e & 1))] = acc[r][nt][e];
        __syncthreads();
        if (scale.sumsq != nullptr && first) {
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) sum += scale_part[w][my_m];
            row_scale = rsqrtf(sum / (float)scale.width + scale.eps);
        }
        auto total = [&](int tile, int row, int col) {            // the warps' partial sums in order
            const float* p = red + tile * 128 + red_at(row, col);
            float v = 0.f;
#pragma unroll
            for (int w = 0; w < WARPS; ++w) v += p[w * RED_FLOATS];
            return v * row_scale;
        };
        if (EPI == EPI_QKV) {
            // bias, rotation by the token's position, and the write of new keys and values to their pages
            for (int idx = tid; idx < n * 64; idx += WARPS * 32) {
                const int m = my_m, r = idx & 7, item = start + (idx >> 6) * 8 + r;
                if (m >= M || item >= end) continue;
                float a = total(idx >> 6, r, m), c = total(idx >> 6, r + 8, m);
                const int half = qkv.d >> 1, head = item / half, j = item - head * half;
                const int f0 = head * qkv.d + j, f1 = f0 + half;             // features of the two values
                if (qkv.bias) { a += qkv.bias[f0]; c += qkv.bias[f1]; }
                if (head < qkv.nq + qkv.nkv) {
                    float sn, cs;
                    sincosf((float)qkv.positions[m] * qkv.inv_freq[j], &sn, &cs);
                    const float ra = a * cs - c * sn, rc = c * cs + a * sn;
                    a = ra; c = rc;
                }
                const bf16 ba = __float2bfloat16_rn(a), bc = __float2bfloat16_rn(c);
                bf16* o = reinterpret_cast<bf16*>(out) + (size_t)m * N;
                o[f0] = ba; o[f1] = bc;
                if (head >= qkv.nq && qkv.slot_mapping) {
                    const long long at = qkv.slot_mapping[m];
                    if (at >= qkv.num_slots) {
                        if (qkv.status) atomicOr(qkv.status, FE_STATUS_BAD_SLOT);
                    } else if (at >= 0) {
                        const bool is_k = head < qkv.nq + qkv.nkv;
                        const int kvh = is_k ? head - qkv.nq : head - qkv.nq - qkv.nkv;
                        bf16* dst = (is_k ? qkv.kc : qkv.vc) + (((at / qkv.ps) * qkv.nkv + kvh) * qkv.ps + (at % qkv.ps)) * qkv.d;
                        dst[j] = ba;
                        dst[j + half] = bc;
                    }
                }
            }
        } else if (EPI == EPI_SWIGLU) {
            for (int idx = tid; idx < n * NT * 64; idx += WARPS * 32) {
                const int part = idx >> 6, m = (part % NT) * 8 + my_m, r = idx & 7, item = start + part / NT * 8 + r;
                if (m >= M || item >= end) continue;
                const float gate = total(part, r, my_m), up = total(part, r + 8, my_m);
                reinterpret_cast<bf16*>(out)[(size_t)m * cut.items + item] = __float2bfloat16_rn(gate_function(gate, gate_act) * up);
            }
        } else if (EPI == EPI_RESID) {
            // the 16 columns of a (tile, row of the batch) sit in 16 consecutive lanes, which add their squares up with shuffles
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int idx = tid + i * WARPS * 32, col = start + (idx >> 7) * 16 + (idx & 15);
                float square = 0.f;
                if (idx < n * 128 && my_m < M && col < end) {
                    const size_t at = (size_t)my_m * N + col;
                    const float sum = before[i] + total(idx >> 7, idx & 15, my_m);
                    resid.residual[at] = sum;
                    resid.scaled[at] = __float2bfloat16_rn(sum * weight[i]);
                    square = sum * sum;
                }
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) square += __shfl_xor_sync(0xffffffffu, square, o);
                if ((idx & 15) == 0 && idx < TILES * 128) square_part[idx >> 7][my_m] = square;
            }
            __syncthreads();
            if (tid < 8) {
                for (int r = 0; r < n; ++r) squares += square_part[r][tid];
                if (!more) resid.sumsq[(size_t)blockIdx.x * 8 + tid] = squares;
            }
        } else {
            for (int idx = tid; idx < n * NT * 128; idx += WARPS * 32) {
                const int part = idx >> 7, m = (part % NT) * 8 + my_m, row = idx & 15, col = start + part / NT * 16 + row;
                if (m >= M || col >= end) continue;
                float v = total(part, row, my_m);
                if (EPI == EPI_BF16 && gate_act == ACT_RELU2) v = v > 0.f ? v * v : 0.f;
                if (EPI == EPI_BF16 && gate_act == ACT_GELU) v = gelu_erf(v);
                if (EPI == EPI_F32) reinterpret_cast<float*>(out)[(size_t)m * N + col] = v;
                else reinterpret_cast<bf16*>(out)[(size_t)m * N + col] = __float2bfloat16_rn(v);
            }
        }
    }
    if (dead && lane == 0 && status) atomicOr(status, FE_STATUS_WAIT_EXPIRED);
}

// Both sizes of a launch's shared memory: one block of each fits an SM, two of the larger do not.  Warps that add nothing up with the others
// have the room for longer rings.
constexpr int LARGE_BYTES = WARPS * (LARGE_RING + RED_FLOATS * 4), SMALL_BYTES = WARPS * (SMALL_RING + RED_FLOATS * 4);

int blocks_for(int items) { const int sms = fe_sm_count(); return items < sms ? items : sms; }

typedef CUresult (*EncodeTiled)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
    static EncodeTiled fn = nullptr;
    if (!fn) {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess)
            fn = (EncodeTiled)p;
    }
    return fn;
}

// Launches a kernel; gives it its shared memory first, once a device.
template <int NT, int EPI, bool ONE, int TILES, bool WIDE, typename... Args>
int launch_kernel(int blocks, int bytes, cudaStream_t stream, const CUtensorMap& map, Args... args) {
    static std::atomic<unsigned long long> allowed{0};
    const auto kernel = skinny_gemm_kernel<NT, EPI, ONE, TILES, WIDE>;
    int device = 0;
    cudaGetDevice(&device);
    if (!(allowed.load() >> (device & 63) & 1)) {
        const cudaError_t err = cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LARGE_BYTES);
        FE_REQUIRE(err == cudaSuccess, "skinny_gemm: %s", cudaGetErrorString(err));
        allowed.fetch_or(1ull << (device & 63));
    }
    fe::launch(kernel, blocks, WARPS * 32, bytes, stream, map, args...);
    return fe_check_launch("skinny_gemm");
}

template <int EPI>
int launch(const void* x, const void* W, void* out, int M, int N, int K, int items, cudaStream_t stream, int* status,
           const QkvEpilogue& qkv = QkvEpilogue{}, const ResidEpilogue& resid = ResidEpilogue{}, const RowScale& scale = RowScale{},
           int gate_act = 0) {
    constexpr bool PAIRS = EPI == EPI_SWIGLU || EPI == EPI_QKV;
    constexpr int ITEMS = PAIRS ? 8 : 16;
    const int sms = fe_sm_count(), most = 2;                       // tiles a group may have
    int blocks, rows;
    bool wide = false;
    if (EPI == EPI_QKV) {
        // groups that lie within a head: a divisor of d / 2; as few rounds of rows over the SMs as possible
        const int half = qkv.d / 2;
        rows = 8;
        for (int r = 16; r <= 8 * most; r += 8)
            if (half % r == 0 && (items / r + sms - 1) / sms * r <= (items / rows + sms - 1) / sms * rows) rows = r;
        blocks = items / rows < sms ? items / rows : sms;
    } else {
        blocks = blocks_for(items);
        const int block_own = (items + blocks - 1) / blocks;
        wide = EPI != EPI_RESID && block_own > 4 * ITEMS;          // more than half a tile for each warp
        const int own = wide ? (block_own + WARPS - 1) / WARPS : block_own, groups = (own + ITEMS * most - 1) / (ITEMS * most);
        rows = (own + groups - 1) / groups;
    }
    const int tiles = (rows + ITEMS - 1) / ITEMS, T = tiles, KB = 4 / T;
    const int plane = rows * (PAIRS ? 2 : 1) * 128, slot = (plane * (KB / 2) + 1023) / 1024 * 1024;
    const int ring = (scale.beside ? SMALL_RING : LARGE_RING) + (wide ? RED_FLOATS * 4 : 0), depth = ring / slot < MAX_DEPTH ? ring / slot : MAX_DEPTH;
    const Cut cut{items, rows, plane, slot, depth, ring};
    EncodeTiled encode = encode_fn();
    FE_REQUIRE(encode != nullptr, "skinny_gemm: cuTensorMapEncodeTiled is not available from this driver");
    CUtensorMap map;
    const cuuint64_t row = (cuuint64_t)K * 2, ks = (cuuint64_t)K / 64;
    const cuuint32_t ones[5] = {1, 1, 1, 1, 1};
    auto make = [&](int rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
        return encode(&map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(W), dims, strides, box, ones, CU_TENSOR_MAP_INTERLEAVE_NONE,
                      CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult rc;
    if constexpr (EPI == EPI_SWIGLU) {
        const cuuint64_t dims[4] = {64, (cuuint64_t)items, 2, ks}, strides[3] = {row, row * items, 128};
        const cuuint32_t box[4] = {64, (cuuint32_t)rows, 2, (cuuint32_t)KB / 2};
        rc = make(4, dims, strides, box);
    } else if constexpr (EPI == EPI_QKV) {
        const cuuint64_t half = qkv.d / 2, dims[5] = {64, half, 2, (cuuint64_t)items / half, ks}, strides[4] = {row, row * half, row * 2 * half, 128};
        const cuuint32_t box[5] = {64, (cuuint32_t)rows, 2, 1, (cuuint32_t)KB / 2};
        rc = make(5, dims, strides, box);
    } else {
        const cuuint64_t dims[3] = {64, (cuuint64_t)N, ks}, strides[2] = {row, 128};
        const cuuint32_t box[3] = {64, (cuuint32_t)rows, (cuuint32_t)KB / 2};
        rc = make(3, dims, strides, box);
    }
    FE_REQUIRE(rc == CUDA_SUCCESS, "skinny_gemm: cuTensorMapEncodeTiled failed with code %d", (int)rc);
#define FE_SKINNY(NT, ONE, TILES, WIDE) \
    return launch_kernel<NT, EPI, ONE, TILES, WIDE>(blocks, scale.beside ? SMALL_BYTES : LARGE_BYTES, stream, map, (const bf16*)x, out, M, N, K, cut, qkv, resid, scale, gate_act, status)
#define FE_SKINNY_TILES(NT, ONE, WIDE) \
    do { \
        if (T == 1) FE_SKINNY(NT, ONE, 1, WIDE); \
        FE_SKINNY(NT, ONE, 2, WIDE); \
    } while (0)
    if constexpr (EPI != EPI_RESID && EPI != EPI_QKV) {
        if (wide && M == 1) FE_SKINNY_TILES(1, true, true);
        if (wide && M <= 8) FE_SKINNY_TILES(1, false, true);
        if (wide) FE_SKINNY_TILES(2, false, true);
        if (M > 8) FE_SKINNY_TILES(2, false, false);
    }
    if (M == 1) FE_SKINNY_TILES(1, true, false);
    if (M <= 8) FE_SKINNY_TILES(1, false, false);
    return 1;                                     // refused by the entry point already
#undef FE_SKINNY
#undef FE_SKINNY_TILES
}

}  // namespace

// The input rows' scales, when the input is a residual times a norm's weight and not yet divided by its root mean
// square (see the top of this file): ``sumsq`` [sumsq_tiles][8] is the table the residual epilogue left.
static int check_scale(const char* what, const float* sumsq, int sumsq_tiles, int M, int K) {
    if (sumsq == nullptr) return 0;
    FE_REQUIRE(M <= 8, "%s: rows are scaled from a table of sums of squares for up to 8 rows, got %d", what, M);
    FE_REQUIRE(sumsq_tiles == blocks_for(K), "%s: the table of sums of squares has %d entries; the product that makes rows of %d elements leaves %d",
               what, sumsq_tiles, K, blocks_for(K));
    FE_REQUIRE(sumsq_tiles <= 1024 && ((size_t)sumsq & 15) == 0, "%s: the table of sums of squares must be 16-byte aligned "
               "and hold at most 1024 tiles (rows of up to 16384 elements)", what);
    return 0;
}

// epilogue: 0 bfloat16 [M, N]; 1 float [M, N]; 2 SwiGLU: W is [2 I, K] (gate rows, then up rows), out bfloat16 [M, I]; 5 the
// same with the tanh form of GELU as the gate's function, 7 with relu; 6 out = relu(x W^T)^2 as bfloat16 [M, N], 8 the exact GELU.
// ``sumsq`` (may be null): see check_scale.  ``held``: see RowScale (the same for the entry points below).
extern "C" int fe_skinny_gemm_scaled(const void* x, const void* W, void* out, int M, int N, int K, int epilogue,
                                     const float* sumsq, int sumsq_tiles, float eps, const void* next, long long next_bytes,
                                     int* status, int beside, int held, cudaStream_t stream) {
    FE_REQUIRE(M >= 1 && M <= 16, "skinny_gemm: %d rows; this kernel takes 1 to 16", M);
    FE_REQUIRE(N > 0 && K > 0 && K % 64 == 0, "skinny_gemm: K = %d must be a positive multiple of 64", K);
    FE_REQUIRE((((size_t)x | (size_t)W) & 15) == 0, "skinny_gemm: operands must be 16-byte aligned");
    if (check_scale("skinny_gemm", sumsq, sumsq_tiles, M, K)) return 1;
    FE_REQUIRE(next_bytes >= 0, "skinny_gemm: negative byte count");
    const RowScale scale{sumsq, sumsq_tiles, eps, K, next, next_bytes, held, beside};
    if (epilogue == EPI_BF16) return launch<EPI_BF16>(x, W, out, M, N, K, N, stream, status, QkvEpilogue{}, ResidEpilogue{}, scale);
    if (epilogue == EPI_F32) return launch<EPI_F32>(x, W, out, M, N, K, N, stream, status, QkvEpilogue{}, ResidEpilogue{}, scale);
    if (epilogue == EPI_RELU2 || epilogue == EPI_GELU)
        return launch<EPI_BF16>(x, W, out, M, N, K, N, stream, status, QkvEpilogue{}, ResidEpilogue{}, scale, epilogue == EPI_GELU ? ACT_GELU : ACT_RELU2);
    if (epilogue == EPI_SWIGLU || epilogue == EPI_GEGLU || epilogue == EPI_REGLU) {
        FE_REQUIRE(N % 2 == 0, "skinny_gemm: a gated epilogue needs an even number of weight rows, got %d", N);
        return launch<EPI_SWIGLU>(x, W, out, M, N, K, N / 2, stream, status, QkvEpilogue{}, ResidEpilogue{}, scale,
                                  epilogue == EPI_GEGLU ? 1 : epilogue == EPI_REGLU ? ACT_RELU : 0);
    }
    FE_REQUIRE(false, "skinny_gemm: unknown epilogue %d", epilogue);
}

extern "C" int fe_skinny_gemm(const void* x, const void* W, void* out, int M, int N, int K, int epilogue,
                              cudaStream_t stream) {
    return fe_skinny_gemm_scaled(x, W, out, M, N, K, epilogue, nullptr, 0, 0.f, nullptr, 0, nullptr, 0, 0, stream);
}

// The product that ends a branch of a layer: residual[M, N] += x W^T (float, in place); scaled[M, N] = bfloat16(new
// residual * norm_weight); sumsq_out[ceil(N / 16)][8] = each 16-column tile's share of the rows' sums of squares.
// ``sumsq_in`` (may be null): the scales of the input rows, as for fe_skinny_gemm_scaled.  M <= 8.
extern "C" int fe_skinny_gemm_residual(const void* x, const void* W, float* residual, const float* norm_weight, void* scaled,
                                       float* sumsq_out, int M, int N, int K, const float* sumsq_in, int sumsq_tiles,
                                       float eps, const void* next, long long next_bytes, int* status, int beside, int held, cudaStream_t stream) {
    FE_REQUIRE(M >= 1 && M <= 8, "skinny_gemm_residual: %d rows; this kernel takes 1 to 8", M);
    FE_REQUIRE(N > 0 && K > 0 && K % 64 == 0, "skinny_gemm_residual: K = %d must be a positive multiple of 64", K);
    FE_REQUIRE((((size_t)x | (size_t)W) & 15) == 0, "skinny_gemm_residual: operands must be 16-byte aligned");
    FE_REQUIRE(residual && norm_weight && scaled && sumsq_out, "skinny_gemm_residual: a null pointer");
    if (check_scale("skinny_gemm_residual", sumsq_in, sumsq_tiles, M, K)) return 1;
    const ResidEpilogue resid{residual, norm_weight, (bf16*)scaled, sumsq_out};
    FE_REQUIRE(next_bytes >= 0, "skinny_gemm_residual: negative byte count");
    return launch<EPI_RESID>(x, W, nullptr, M, N, K, N, stream, status, QkvEpilogue{}, resid,
                             RowScale{sumsq_in, sumsq_tiles, eps, K, next, next_bytes, held, beside});
}

// The query/key/value projection of an attention layer with its epilogue fused: y = x W^T + bias,
// half-split rotation of the query and key heads by the tokens' positions, in place into
// out [M, (nq + 2 nkv) d] (bfloat16), and the write of the new keys and values into their cache
// slots.  The whole head is rotated (rotary width = head size, a multiple of 16); M <= 8.
// ``sumsq`` (may be null): the scales of the input rows, as for fe_skinny_gemm_scaled.
extern "C" int fe_skinny_qkv(const void* x, const void* W, void* out, const float* bias, const int* positions,
                             const float* inv_freq, const int* slot_mapping, void* kc, void* vc, int M, int K, int nq,
                             int nkv, int d, int ps, long long num_slots, const float* sumsq, int sumsq_tiles, float eps,
                             int* status, int beside, int held, cudaStream_t stream) {
    FE_REQUIRE(M >= 1 && M <= 8, "skinny_qkv: %d rows; this kernel takes 1 to 8", M);
    FE_REQUIRE(K > 0 && K % 64 == 0, "skinny_qkv: K = %d must be a positive multiple of 64", K);
    FE_REQUIRE(d >= 16 && d % 16 == 0 && nq > 0 && nkv > 0 && ps > 0, "skinny_qkv: bad head size or counts");
    FE_REQUIRE(positions != nullptr && inv_freq != nullptr, "skinny_qkv: positions and the rotary table are required");
    FE_REQUIRE((((size_t)x | (size_t)W) & 15) == 0, "skinny_qkv: operands must be 16-byte aligned");
    if (check_scale("skinny_qkv", sumsq, sumsq_tiles, M, K)) return 1;
    QkvEpilogue e{bias, positions, inv_freq, slot_mapping, (bf16*)kc, (bf16*)vc, nq, nkv, d, ps, num_slots, status};
    return launch<EPI_QKV>(x, W, out, M, (nq + 2 * nkv) * d, K, (nq + 2 * nkv) * (d / 2), stream, status, e, ResidEpilogue{},
                           RowScale{sumsq, sumsq_tiles, eps, K, nullptr, 0, held, beside});
}

// How many entries of 8 floats the residual epilogue of a product with N columns leaves in ``sumsq_out``.
extern "C" int fe_skinny_sumsq_parts(int N) { return blocks_for(N); }
