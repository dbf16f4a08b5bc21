// Paged causal grouped-query attention on CUDA cores, float arithmetic throughout.
//
// Keys are taken in blocks of 32 or 64 that are aligned to absolute position 0; scores, running maximum, running
// sum and the value accumulator are float (online softmax, as the reference's block-wise path:
// inference/attention/paged.py:50-70).  Key t is visible to the query at position p iff t <= p
// (and t > p - window, or t < keep, when window > 0; t in the chunk of -window positions that holds p when window < 0)
// (paged.py:31-32).  ``sink``: the softmax starts as if a key of score 0 and value 0 had been seen, which adds
// 1 to its denominator.  ``mode`` bit 1 (bit 0 is the sink): no softmax; the weight of a visible key is
// sigmoid(score + per_head[h]), not normalised over the keys.  Bit 2: scores are multiplied by per_head[h] (null: by 1) and, with
// softcap > 0, become softcap * tanh(score / softcap).  Query head h reads key/value head
// h / (nq / nkv) (paged.py:29-30).  Because the blocks are aligned to position 0 and taken in
// order, the result for a query does not depend on how its request was cut into steps.
//
// Two kernels.  The tiled one serves the true 32-bit path for head sizes up to 128: a block of 32 rows shares every key it
// loads (below).  The other, one warp per (token, query head), serves calls of the same heads that have little to share
// (rows_pay), larger heads in 32 bits, and bfloat16 for shapes the tensor core kernels do not take (head sizes beyond 256: the
// rows of a wide cached latent).
#include <math_constants.h>

#include "common.cuh"

using namespace fe;

// A score from the dot product: times the scale, squashed where there is a cap.  Rounded after each step, so that no compiler
// folds the product into what follows in one kernel and not in another.
__device__ __forceinline__ float score_of(float dot, float scale, float cap) {
    const float s = __fmul_rn(dot, scale);
    return cap > 0.f ? __fmul_rn(cap, tanhf(s / cap)) : s;
}

// One warp per (token, query head), PER keys a lane at a time: lane l takes keys l, l + 32, ... of a block of 32 PER.  With
// PER = 2 it does the arithmetic of the tiled kernel below for one row, operation by operation (blocks of 64 keys; the sum of
// a block's weights first over keys 16 apart, then 32, then within 16), so that a row's result is the same bit for bit
// whichever of the two takes it.
template <typename T, int DPL, int PER>
__global__ void paged_attention_simt_kernel(const T* __restrict__ q, long long q_stride, T* __restrict__ out,
                                            long long out_stride, const T* __restrict__ kc,
                                            const T* __restrict__ vc, const int* __restrict__ block_table,
                                            int bt_stride, const int* __restrict__ cu_q,
                                            const int* __restrict__ q_start, const int* __restrict__ token_req,
                                            int T_tokens, int nq, int nkv, int d, int ps, int num_pages, float scale,
                                            int window, int keep, int mode, const float* __restrict__ per_head, float softcap, int* __restrict__ status) {
    griddep_wait();
    griddep_launch_dependents();
    extern __shared__ float q_smem[];
    constexpr int KEYS = 32 * PER;
    const int lane = threadIdx.x & 31;
    const int warp_in_block = threadIdx.x >> 5;
    const long long warp = (long long)blockIdx.x * (blockDim.x >> 5) + warp_in_block;
    if (warp >= (long long)T_tokens * nq) return;
    const int tok = (int)(warp / nq), h = (int)(warp % nq);
    const int r = token_req[tok];
    const int pos = q_start[r] + (tok - cu_q[r]);
    const int kvh = h / (nq / nkv);
    float* qs = q_smem + (size_t)warp_in_block * d;
    const T* qp = q + (size_t)tok * q_stride + (size_t)h * d;
    for (int j = lane; j < d; j += 32) qs[j] = to_float(qp[j]);
    __syncwarp();

    const bool sink = mode & 1, sigmoid = mode & 2;
    const float bias = (sigmoid && per_head) ? per_head[h] : 0.f;
    if ((mode & 4) && per_head) scale *= per_head[h];
    const float cap = mode & 4 ? softcap : 0.f;
    float m = sink ? 0.f : -CUDART_INF_F, l = sink ? 1.f : 0.f;
    float acc[DPL];
#pragma unroll
    for (int i = 0; i < DPL; ++i) acc[i] = 0.f;

    const int lo = first_visible(pos, window);
    const int* table = block_table + (size_t)r * bt_stride;
    const int kept = kept_tiles<KEYS>(lo, keep), blocks = kept + pos / KEYS - lo / KEYS + 1;
    for (int at = 0; at < blocks; ++at) {
        const int kb = listed_tile<KEYS>(at, kept, lo) * KEYS;
        bool valid[PER];
        float s[PER], p[PER];
        long long base[PER];
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const int t = kb + 32 * u + lane;
            valid[u] = (t >= lo || t < keep) && t <= pos;
            s[u] = -CUDART_INF_F;
            base[u] = 0;
            if (valid[u]) {
                const int page = table[t / ps];
                if (page < 0 || page >= num_pages) {
                    if (status) atomicOr(status, FE_STATUS_BAD_PAGE);
                    valid[u] = false;
                } else {
                    base[u] = (((long long)page * nkv + kvh) * ps + (t % ps)) * d;
                    const T* kp = kc + base[u];
                    float dot = 0.f;
                    for (int j = 0; j < d; j += 8) {
                        float kv[8];
                        load8<T>(kp + j, kv);
#pragma unroll
                        for (int e = 0; e < 8; ++e) dot = fmaf(qs[j + e], kv[e], dot);
                    }
                    s[u] = score_of(dot, scale, cap);
                }
            }
        }
        if (sigmoid) {
#pragma unroll
            for (int u = 0; u < PER; ++u) p[u] = valid[u] ? 1.f / (1.f + expf(-(s[u] + bias))) : 0.f;
            l = 1.f;                                   // the sum is not divided by anything
        } else {
            float bm = s[0];
#pragma unroll
            for (int u = 1; u < PER; ++u) bm = fmaxf(bm, s[u]);
            bm = warp_max(bm);
            if (bm == -CUDART_INF_F) continue;         // nothing visible in this block (bad pages only)
            const float m_new = fmaxf(m, bm);
            const float alpha = expf(m - m_new);       // exp(-inf) = 0 on the first block
            float sum = 0.f;
#pragma unroll
            for (int u = 0; u < PER; ++u) {
                p[u] = valid[u] ? expf(s[u] - m_new) : 0.f;
                const float pair = p[u] + __shfl_xor_sync(0xffffffffu, p[u], 16);
                sum = u == 0 ? pair : sum + pair;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l = fmaf(l, alpha, sum);
#pragma unroll
            for (int i = 0; i < DPL; ++i) acc[i] *= alpha;
            m = m_new;
        }
#pragma unroll
        for (int u = 0; u < PER; ++u) {
            const unsigned weighs = __ballot_sync(0xffffffffu, p[u] != 0.f);      // all from the window's edge to the diagonal, as a rule
            if (weighs == 0u) continue;
            const int count = 32 - __clz(weighs);
            for (int tt = __ffs(weighs) - 1; tt < count; ++tt) {
                const float pt = __shfl_sync(0xffffffffu, p[u], tt);
                const long long vb = __shfl_sync(0xffffffffu, base[u], tt);
                if (pt != 0.f) {
                    const T* vp = vc + vb;
#pragma unroll
                    for (int i = 0; i < DPL; ++i) {
                        const int j = lane + 32 * i;
                        if (j < d) acc[i] = fmaf(pt, to_float(vp[j]), acc[i]);
                    }
                }
            }
        }
    }
    T* op = out + (size_t)tok * out_stride + (size_t)h * d;
    const float inv = l > 0.f ? 1.f / l : 0.f;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
        const int j = lane + 32 * i;
        if (j < d) op[j] = from_float<T>(acc[i] * inv);
    }
}

// ---- the tiled kernel ------------------------------------------------------------------------------------------------------
// A block of 256 threads takes 32 rows of one (request, key/value head); row m is the pair (query m / G, head m % G of the
// group).  Keys and values come to shared memory 64 keys at a time (aligned to position 0) in asynchronous 16-byte copies, the
// next tile's while this one is worked on.  A thread owns two rows throughout: the scores of four keys of them (the dot product over ascending
// elements), their softmax statistics (reduced over the half warp that shares the rows), and eight value columns.  Where a
// lane per key read keys 512 bytes apart and a warp per head read each of them again, memory set the pace (296 us a layer
// at 256 tokens, 12 heads of 128 in 2 groups); now shared memory's latency and bandwidth do (48 us; with
// half as many threads of four rows each, which read less but wait longer, 69 us; tiles of 32 keys, 109 us).
// A row's result does not depend on the rows beside it: a block of keys of which it sees none leaves it as it was.
namespace {

constexpr int TILE_ROWS = 32, TILE_KEYS = 64, TILE_THREADS = 256, TILE_MAX_D = 128;

__device__ __forceinline__ void copy16(void* smem_dst, const void* src, int bytes) {
    const unsigned dst = (unsigned)__cvta_generic_to_shared(smem_dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst), "l"(src), "r"(bytes));
}

__global__ void __launch_bounds__(TILE_THREADS)
paged_attention_tiled_kernel(const float* __restrict__ q, long long q_stride, float* __restrict__ out, long long out_stride,
                             const float* __restrict__ kc, const float* __restrict__ vc, const int* __restrict__ block_table,
                             int bt_stride, const int* __restrict__ cu_q, const int* __restrict__ q_start, int requests, int nq,
                             int nkv, int d, int ps, int num_pages, float scale, int window, int keep, int mode,
                             const float* __restrict__ per_head, float softcap, int* __restrict__ status) {
    griddep_wait();
    griddep_launch_dependents();
    extern __shared__ __align__(16) float tile_smem[];
    __shared__ __align__(16) float probs[TILE_KEYS][TILE_ROWS + 4];
    const int pitch = d + 4;                                  // rows of a tile are shifted by one bank group against each other
    float* q_s = tile_smem;                                   // [TILE_ROWS][pitch]
    float* kv_s = q_s + TILE_ROWS * pitch;                    // two stages of keys [64][pitch] and values [64][pitch]
    const int tid = threadIdx.x, lane = tid & 31, tx = tid & 15, ty = tid >> 4;
    const int G = nq / nkv, kvh = blockIdx.y;

    // which request and which of its tiles of 32 rows: every warp adds up the requests' tiles, 32 at a time
    int r = -1, tile = 0;
    for (int base = 0, seen = 0; base < requests; base += 32) {
        const int i = base + lane;
        const int mine = i < requests ? ((cu_q[i + 1] - cu_q[i]) * G + TILE_ROWS - 1) / TILE_ROWS : 0;
        int upto = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const int at = (int)blockIdx.x - seen;
        const unsigned here = __ballot_sync(0xffffffffu, at >= upto - mine && at < upto);
        if (here) {
            const int who = __ffs(here) - 1;
            r = base + who;
            tile = at - __shfl_sync(0xffffffffu, upto - mine, who);
            break;
        }
        seen += __shfl_sync(0xffffffffu, upto, 31);
    }
    if (r < 0) return;                                        // the grid is an upper bound
    const int tok0 = cu_q[r], n_q = cu_q[r + 1] - tok0, start = q_start[r];
    const int m0 = tile * TILE_ROWS, rows = min(TILE_ROWS, n_q * G - m0);

    const bool sink = mode & 1, sigmoid = mode & 2, mapped = mode & 4;
    const float cap = mapped ? softcap : 0.f;
    int pos[2], lo[2];
    float bias[2], factor[2], m[2], l[2];
    float2 acc[2][4];                                         // row, value columns 4 tx .. + 3 and 64 + 4 tx .. + 3
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = ty * 2 + i;
        const bool real = row < rows;
        const int head = kvh * G + (real ? (m0 + row) % G : 0);
        pos[i] = real ? start + (m0 + row) / G : -1;
        lo[i] = real ? first_visible(pos[i], window) : 0;
        bias[i] = (sigmoid && per_head) ? per_head[head] : 0.f;
        factor[i] = (mapped && per_head) ? scale * per_head[head] : scale;
        m[i] = sink ? 0.f : -CUDART_INF_F;
        l[i] = sink ? 1.f : 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = make_float2(0.f, 0.f);
    }
    for (int idx = tid; idx < TILE_ROWS * d; idx += TILE_THREADS) {
        const int row = idx / d, j = idx - row * d;
        q_s[row * pitch + j] = row < rows ? q[(size_t)(tok0 + (m0 + row) / G) * q_stride + (size_t)(kvh * G + (m0 + row) % G) * d + j] : 0.f;
    }
    const int first_pos = start + m0 / G, last_pos = start + (m0 + rows - 1) / G;
    const int block_lo = first_visible(first_pos, window);
    const int* table = block_table + (size_t)r * bt_stride;
    const int kept = kept_tiles<TILE_KEYS>(block_lo, keep), tiles = kept + last_pos / TILE_KEYS - block_lo / TILE_KEYS + 1;
    const int chunks = d >> 2;
    const bool idle = (ty & ~1) * 2 >= rows;                  // of the whole warp: it owns four rows
    // four threads a key: each copies every fourth 16 bytes of its row; a key beyond the tile's last query reads as zeros
    auto fetch = [&](int at) {
        float* k_s = kv_s + (at & 1) * 2 * TILE_KEYS * pitch;
        float* v_s = k_s + TILE_KEYS * pitch;
        const int row = tid >> 2, key = listed_tile<TILE_KEYS>(at, kept, block_lo) * TILE_KEYS + row;
        long long from = -1;
        if (key <= last_pos) {
            const int page = table[key / ps];
            if (page < 0 || page >= num_pages) {
                // a page that is gone is a fault only where a query sees the key
                if (status && (key >= block_lo || key < keep) && (tid & 3) == 0) atomicOr(status, FE_STATUS_BAD_PAGE);
            } else {
                from = (((long long)page * nkv + kvh) * ps + key % ps) * d;
            }
        }
        for (int c = tid & 3; c < chunks; c += 4) {
            copy16(k_s + row * pitch + c * 4, from >= 0 ? kc + from + c * 4 : kc, from >= 0 ? 16 : 0);
            copy16(v_s + row * pitch + c * 4, from >= 0 ? vc + from + c * 4 : vc, from >= 0 ? 16 : 0);
        }
        // whether the key is there at all
        return from >= 0;
    };
    __shared__ unsigned there[2][TILE_THREADS / 32];
    auto start_tile = [&](int at) {
        const unsigned mask = __ballot_sync(0xffffffffu, at < tiles && fetch(at));
        if (lane == 0) there[at & 1][tid >> 5] = mask;
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    start_tile(0);
    for (int at = 0; at < tiles; ++at) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                                      // tile ``at`` is there; the other stage has been read by all
        if (at + 1 < tiles) start_tile(at + 1);
        const float* k_s = kv_s + (at & 1) * 2 * TILE_KEYS * pitch;
        const float* v_s = k_s + TILE_KEYS * pitch;
        const int key0 = listed_tile<TILE_KEYS>(at, kept, block_lo) * TILE_KEYS;
        if (idle) continue;                                   // a warp whose rows are all padding only helps with the copies
        float s[2][4] = {};
        {
            const float* qp = q_s + ty * 2 * pitch;
            const float* kp = k_s + tx * pitch;
#pragma unroll 4
            for (int j = 0; j < d; j += 4) {
                float4 k4[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) k4[u] = *reinterpret_cast<const float4*>(kp + 16 * u * pitch + j);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(qp + i * pitch + j);
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        s[i][u] = fmaf(a.x, k4[u].x, s[i][u]);
                        s[i][u] = fmaf(a.y, k4[u].y, s[i][u]);
                        s[i][u] = fmaf(a.z, k4[u].z, s[i][u]);
                        s[i][u] = fmaf(a.w, k4[u].w, s[i][u]);
                    }
                }
            }
        }
        // keys tx, tx + 16, tx + 32, tx + 48; four threads looked at a key: bit 4 k of the warp that copied it
        bool see[2][4];
        float p[2][4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const bool have = there[at & 1][2 * u + (tx >> 3)] >> ((tx & 7) * 4) & 1;
            const int t = key0 + tx + 16 * u;
#pragma unroll
            for (int i = 0; i < 2; ++i) see[i][u] = have & ((t >= lo[i]) | (t < keep)) & (t <= pos[i]);
        }
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            float top = -CUDART_INF_F;
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                s[i][u] = score_of(s[i][u], factor[i], cap);
                if (see[i][u]) top = fmaxf(top, s[i][u]);
            }
            if (sigmoid) {
#pragma unroll
                for (int u = 0; u < 4; ++u) p[i][u] = see[i][u] ? 1.f / (1.f + expf(-(s[i][u] + bias[i]))) : 0.f;
                l[i] = 1.f;                                   // the sum is not divided by anything
                continue;
            }
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, o));
            const bool some = top != -CUDART_INF_F;           // else the row sees nothing of this tile (the same for the 16 lanes)
            const float m_new = fmaxf(m[i], top);
            const float alpha = some ? expf(m[i] - m_new) : 1.f;        // exp(-inf) = 0 on the first tile
#pragma unroll
            for (int u = 0; u < 4; ++u) p[i][u] = see[i][u] && some ? expf(s[i][u] - m_new) : 0.f;
            float sum = (p[i][0] + p[i][1]) + (p[i][2] + p[i][3]);
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            l[i] = fmaf(l[i], alpha, sum);
#pragma unroll
            for (int c = 0; c < 4; ++c) { acc[i][c].x *= alpha; acc[i][c].y *= alpha; }
            m[i] = m_new;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u) *reinterpret_cast<float2*>(&probs[tx + 16 * u][ty * 2]) = make_float2(p[0][u], p[1][u]);
        __syncwarp();                                         // a half warp reads the rows it wrote itself
        // a weight of 0 adds nothing, whatever the value (keys beyond what the row sees may hold anything)
        const bool left = tx * 4 < d, right = 64 + tx * 4 < d;
#pragma unroll 4
        for (int key = 0; key < TILE_KEYS; ++key) {
            const float2 w2 = *reinterpret_cast<const float2*>(&probs[key][ty * 2]);
            const float w[2] = {w2.x, w2.y};
            const float* vp = v_s + key * pitch + tx * 4;
            const float4 va = left ? *reinterpret_cast<const float4*>(vp) : make_float4(0.f, 0.f, 0.f, 0.f);
            const float4 vb = right ? *reinterpret_cast<const float4*>(vp + 64) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                if (w[i] != 0.f) {
                    const float2 ww = make_float2(w[i], w[i]);
                    acc[i][0] = __ffma2_rn(ww, make_float2(va.x, va.y), acc[i][0]);
                    acc[i][1] = __ffma2_rn(ww, make_float2(va.z, va.w), acc[i][1]);
                    acc[i][2] = __ffma2_rn(ww, make_float2(vb.x, vb.y), acc[i][2]);
                    acc[i][3] = __ffma2_rn(ww, make_float2(vb.z, vb.w), acc[i][3]);
                }
            }
        }
        __syncwarp();                                         // all have read the weights before the next ones are written
    }
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int row = ty * 2 + i;
        if (row >= rows) continue;
        float* op = out + (size_t)(tok0 + (m0 + row) / G) * out_stride + (size_t)(kvh * G + (m0 + row) % G) * d;
        const float inv = l[i] > 0.f ? 1.f / l[i] : 0.f;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int j = (c >> 1) * 64 + tx * 4 + (c & 1) * 2;
            if (j < d) { op[j] = acc[i][c].x * inv; op[j + 1] = acc[i][c].y * inv; }
        }
    }
}

int launch_tiled(const float* q, long long q_stride, float* out, long long out_stride, const float* kc, const float* vc,
                 const int* block_table, int bt_stride, const int* cu_q, const int* q_start, int requests, int T_tokens, int nq,
                 int nkv, int d, int ps, int num_pages, float scale, int window, int keep, int mode, const float* per_head,
                 float softcap, int* status, cudaStream_t stream) {
    const size_t smem = (size_t)(TILE_ROWS + 4 * TILE_KEYS) * (d + 4) * sizeof(float);
    const cudaError_t err = cudaFuncSetAttribute(paged_attention_tiled_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    FE_REQUIRE(err == cudaSuccess, "paged_attention: %s", cudaGetErrorString(err));
    // a request's last tile may be short: at most one tile a request beyond what the rows fill
    const long long tiles = ((long long)T_tokens * (nq / nkv)) / TILE_ROWS + requests;
    FE_REQUIRE(tiles <= 2147483647LL && nkv <= 65535, "paged_attention: grid too large");
    fe::launch(paged_attention_tiled_kernel, dim3((unsigned)tiles, nkv), TILE_THREADS, smem, stream, q, q_stride, out, out_stride, kc, vc,
               block_table, bt_stride, cu_q, q_start, requests, nq, nkv, d, ps, num_pages, scale, window, keep, mode, per_head, softcap, status);
    return fe_check_launch("paged_attention_tiled");
}

// Whether a call's rows are taken one warp each and not 32 a block (the same bits either way).  A block of the tiled kernel costs its
// 8 us however few of its rows and keys are real, and one or two are resident on an SM; a warp a row costs by the key.  So: where no
// row sees more than a few keys (40 prompts of 9, 12 heads of 128 in two groups: 12.7 us, tiled 26.9; one prompt of 9: 9.0, 15.2; a
// window of 5 over 1,024 tokens: 29, 50; small heads a few more keys); and where the blocks make several rounds with little in each
// (``seen`` keys times a block's rows below what a block costs: 128 requests of 64 keys, 32 heads of 128: 76 us, tiled 237; 48 of 130
// keys: 110, 195; beyond the line 128 of 256 keys, 16 heads of 96 in eight groups: 201, tiled 159), if there are rows enough to hide
// a warp's walk (16 requests of 256 keys, 32 heads of 128: 189 us, tiled 96).
bool rows_pay(int T_tokens, int requests, int nq, int nkv, int d, long long context, int window, int keep) {
    const long long G = nq / nkv, portion = (T_tokens + requests - 1) / requests;
    const long long rows = portion * G, tiles = (rows + TILE_ROWS - 1) / TILE_ROWS, blocks = tiles * nkv * requests;
    long long seen = context - (portion - 1) / 2;                     // by a row, on average of a portion
    if (window > 0) seen = min(seen, (long long)window + keep);
    if (window < 0) seen = min(seen, (1LL - window) / 2);
    if (seen <= (d <= 32 ? 24 : 16)) return true;
    const long long resident = (long long)fe_sm_count() * (d <= 80 ? 2 : 1);
    return blocks > resident && seen * rows <= tiles * (280 + seen / 2) && seen * resident <= 50 * blocks;
}

}  // namespace

template <typename T>
static int launch_simt(const void* q, long long q_stride, void* out, long long out_stride, const void* kc,
                       const void* vc, const int* block_table, int bt_stride, const int* cu_q, const int* q_start,
                       const int* token_req, int T_tokens, int nq, int nkv, int d, int ps, int num_pages,
                       float scale, int window, int keep, int sink, const float* per_head, float softcap, int* status, cudaStream_t stream) {
    const int warps = 4;
    const long long total = (long long)T_tokens * nq;
    const int blocks = (int)((total + warps - 1) / warps);
    const size_t smem = (size_t)warps * d * sizeof(float);
    constexpr int PER = sizeof(T) == 4 ? 2 : 1;               // in 32 bits the blocks of the tiled kernel, for the heads that it takes
#define FE_LAUNCH_SIMT(DPL, PER)                                                                                 \
    fe::launch(paged_attention_simt_kernel<T, DPL, PER>, blocks, warps * 32, smem, stream,                               \
        (const T*)q, q_stride, (T*)out, out_stride, (const T*)kc, (const T*)vc, block_table, bt_stride, cu_q,   \
        q_start, token_req, T_tokens, nq, nkv, d, ps, num_pages, scale, window, keep, sink, per_head, softcap, status)
    static_assert(TILE_MAX_D == 128, "heads up to this size walk blocks of PER * 32 keys");
    if (d <= 32) FE_LAUNCH_SIMT(1, PER);
    else if (d <= 64) FE_LAUNCH_SIMT(2, PER);
    else if (d <= 128) FE_LAUNCH_SIMT(4, PER);
    else if (d <= 256) FE_LAUNCH_SIMT(8, 1);
    else if (d <= 512) FE_LAUNCH_SIMT(16, 1);
    else FE_LAUNCH_SIMT(32, 1);
#undef FE_LAUNCH_SIMT
    return fe_check_launch("paged_attention_simt");
}

// ``context``: the longest context among the requests, 0 if it is not known (the block table's width then stands for it).
extern "C" int fe_paged_attention_simt(const void* q, long long q_stride, void* out, long long out_stride,
                                       const void* kc, const void* vc, const int* block_table, int bt_stride,
                                       const int* cu_q, const int* q_start, const int* token_req, int requests, int T_tokens, int context,
                                       int nq, int nkv, int d, int ps, int num_pages, float scale, int window, int keep,
                                       int sink, int dtype, int* status, const float* per_head, float softcap, cudaStream_t stream) {
    FE_REQUIRE(T_tokens >= 0 && nq > 0 && nkv > 0 && nq % nkv == 0, "paged_attention: bad head counts %d/%d", nq, nkv);
    FE_REQUIRE(d >= 16 && d <= 1024 && d % 16 == 0, "paged_attention: head size %d is not a multiple of 16 in [16, 1024]", d);
    FE_REQUIRE(ps > 0 && num_pages > 0, "paged_attention: bad page size or page count");
    FE_REQUIRE(q_stride % 8 == 0, "paged_attention: query row stride %lld must be a multiple of 8 elements", q_stride);
    if (T_tokens == 0) return 0;
    FE_REQUIRE(((size_t)kc & 15) == 0, "paged_attention: the cache's keys must be 16-byte aligned");
    FE_REQUIRE(requests > 0 && context >= 0, "paged_attention: %d requests, longest context %d", requests, context);
    // the tiled kernel copies values 16 bytes at a time as well
    if (dtype == FE_F32 && d <= TILE_MAX_D && ((size_t)vc & 15) == 0 && nkv <= 65535 &&
        !rows_pay(T_tokens, requests, nq, nkv, d, context > 0 ? context : (long long)bt_stride * ps, window, keep))
        return launch_tiled((const float*)q, q_stride, (float*)out, out_stride, (const float*)kc, (const float*)vc, block_table,
                            bt_stride, cu_q, q_start, requests, T_tokens, nq, nkv, d, ps, num_pages, scale, window, keep, sink,
                            per_head, softcap, status, stream);
    if (dtype == FE_F32)
        return launch_simt<float>(q, q_stride, out, out_stride, kc, vc, block_table, bt_stride, cu_q, q_start,
                                  token_req, T_tokens, nq, nkv, d, ps, num_pages, scale, window, keep, sink, per_head, softcap, status, stream);
    if (dtype == FE_BF16)
        return launch_simt<bf16>(q, q_stride, out, out_stride, kc, vc, block_table, bt_stride, cu_q, q_start,
                                 token_req, T_tokens, nq, nkv, d, ps, num_pages, scale, window, keep, sink, per_head, softcap, status, stream);
    FE_REQUIRE(false, "paged_attention: unknown dtype %d", dtype);
}
