// Causal attention without softmax over a paged cache whose keys and values may differ in size:
//   weight(query i, key j <= i) = sigmoid(scale * q_i . k_j + bias[head]),   out_i = sum_j weight * v_j
// (weights are not normalised over keys).  Scores, weights and the sums are fp32.
//
// rotate_store: rotate-half rotation of the first `rotary` elements of every query and key head (pair (i, i +
// rotary / 2), angle = float(position) * inv_freq[i] in fp32), queries to q_out, keys and values into the request's
// pages: k_pool [pages, kv_heads, page, D], v_pool [pages, kv_heads, page, V].
// attend: one block per (tile of consecutive queries of a run, heads of one key/value head): 16 (token, head) rows;
// keys are walked in tiles of 32 in ascending order (the tensor-core form: of 64), so an output's sum has the same order
// however the tokens were cut into steps and whatever else a step holds.
#include <type_traits>

#include "common.cuh"

EMBER_DEFINE_LAST_ERROR

namespace ember {

template <typename T>
__global__ void rotate_store_kernel(const float* __restrict__ qkv, int ld, int H, int G, int D, int V,
                                    const float* __restrict__ inv_freq, int rotary,
                                    const int* __restrict__ positions, const int* __restrict__ seq_of,
                                    const int* __restrict__ block_table, int max_blocks, int page, int num_pages,
                                    T* __restrict__ q_out, T* __restrict__ k_pool, T* __restrict__ v_pool, int write_kv,
                                    int* __restrict__ err) {
    extern __shared__ float cs[];           // cos [rotary / 2], sin [rotary / 2]
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, pos = positions[t], half = rotary >> 1;
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float sn, c;
        sincosf((float)pos * inv_freq[i], &sn, &c);
        cs[i] = c; cs[half + i] = sn;
    }
    __syncthreads();
    const float* row = qkv + (size_t)t * ld;
    const int blk = block_table[(size_t)seq_of[t] * max_blocks + pos / page], slot = pos % page;
    const bool page_ok = blk >= 0 && blk < num_pages;
    if (write_kv && !page_ok && threadIdx.x == 0 && err) atomicOr(err, EMBER_ERR_PAGE_RANGE);
    // query and key heads: H + G heads of D
    for (int e = threadIdx.x; e < (H + G) * D; e += blockDim.x) {
        const int head = e / D, i = e - head * D;
        float v = row[e];
        if (i < rotary) {
            const int f = i < half ? i : i - half;
            const float other = row[head * D + (i < half ? i + half : i - half)];
            v = i < half ? v * cs[f] - other * cs[half + f] : v * cs[f] + other * cs[half + f];
        }
        if (head < H) q_out[(size_t)t * H * D + e] = from_float<T>(v);
        else if (write_kv && page_ok)
            k_pool[(((size_t)blk * G + (head - H)) * page + slot) * D + i] = from_float<T>(v);
    }
    if (write_kv && page_ok) {
        const float* vr = row + (size_t)(H + G) * D;
        for (int e = threadIdx.x; e < G * V; e += blockDim.x) {
            const int head = e / V, i = e - head * V;
            v_pool[(((size_t)blk * G + head) * page + slot) * V + i] = from_float<T>(vr[e]);
        }
    }
}

constexpr int SA_ROWS = 16, SA_KEYS = 32, SA_THREADS = 128;

// 8 consecutive elements of a cache row as floats (16-byte loads where the row allows them)
__device__ __forceinline__ void load_row_chunk(const __nv_bfloat16* src, float* dst, int n, bool whole) {
    if (whole) {
        const uint4 u = *reinterpret_cast<const uint4*>(src);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&u);
#pragma unroll
        for (int i = 0; i < 4; i++) { const float2 f = __bfloat1622float2(h[i]); dst[2 * i] = f.x; dst[2 * i + 1] = f.y; }
    } else {
        for (int i = 0; i < n; i++) dst[i] = __bfloat162float(src[i]);
    }
}
__device__ __forceinline__ void load_row_chunk(const float* src, float* dst, int n, bool whole) {
    if (whole) {
        const float4 a = reinterpret_cast<const float4*>(src)[0], b = reinterpret_cast<const float4*>(src)[1];
        dst[0] = a.x; dst[1] = a.y; dst[2] = a.z; dst[3] = a.w; dst[4] = b.x; dst[5] = b.y; dst[6] = b.z; dst[7] = b.w;
    } else {
        for (int i = 0; i < n; i++) dst[i] = src[i];
    }
}

// A block's rows are (query token, query head) pairs of one key/value head: `hpb` heads (a divisor of the group, at
// most 16) of 16 / hpb consecutive tokens, so a decode step reads a request's keys once for all heads of the group
// and a prompt portion fills the 16 rows.  Scores: a thread takes one key and four rows, four elements at a time;
// read-out: a thread takes value columns tid, tid + 128, ... of all rows, four keys at a time.
// CM: value columns per thread (V <= 128 CM).  Head sizes that are multiples of 8 are fetched with 16-byte loads.
template <typename T, int CM>
__global__ void __launch_bounds__(SA_THREADS)
sigmoid_attention_kernel(const T* __restrict__ q, const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                         T* __restrict__ out, int H, int G, int D, int V, int hpb, const int* __restrict__ tiles,
                         const int* __restrict__ block_table, int max_blocks, int page, int num_pages, float scale,
                         const float* __restrict__ head_bias, int* __restrict__ err) {
    extern __shared__ __align__(16) float smem[];
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 4 * blockIdx.x;
    const int run = tile[0], row0 = tile[1], nq = tile[2], pos0 = tile[3];
    const int h0 = blockIdx.y * hpb, kv = h0 / (H / G);
    const int n_rows = nq * hpb;                        // row rr: token rr / hpb, head h0 + rr % hpb
    const int DP = (D + 3) / 4 * 4 + 4, VP = (V + 3) / 4 * 4;
    float* qs = smem;                                   // [SA_ROWS][DP]
    float* ks = qs + SA_ROWS * DP;                      // [SA_KEYS][DP]
    float* vs = ks + SA_KEYS * DP;                      // [SA_KEYS][VP]
    float* ws = vs + SA_KEYS * VP;                      // [SA_ROWS][SA_KEYS]
    for (int e = threadIdx.x; e < SA_ROWS * DP; e += SA_THREADS) {
        const int r = e / DP, i = e - r * DP;
        qs[e] = (r < n_rows && i < D) ? to_float(q[((size_t)(row0 + r / hpb) * H + h0 + r % hpb) * D + i]) : 0.0f;
    }
    for (int e = threadIdx.x; e < SA_KEYS * (DP - D); e += SA_THREADS)       // the padding of key rows stays zero
        ks[(e / (DP - D)) * DP + D + e % (DP - D)] = 0.0f;
    float acc[SA_ROWS][CM];
#pragma unroll
    for (int r = 0; r < SA_ROWS; r++)
#pragma unroll
        for (int m = 0; m < CM; m++) acc[r][m] = 0.0f;
    const int n_keys = pos0 + nq;                       // keys 0 .. position of the last query
    const int* bt = block_table + (size_t)run * max_blocks;
    const int kk = threadIdx.x & 31, rg = threadIdx.x >> 5;
    const int dchunks = (D + 7) / 8, vchunks = (V + 7) / 8;
    const bool d8 = (D & 7) == 0, v8 = (V & 7) == 0;
    for (int k0 = 0; k0 < n_keys; k0 += SA_KEYS) {
        __syncthreads();
        // keys and values of this tile as floats (rows beyond the last key are zero)
        for (int e = threadIdx.x; e < SA_KEYS * dchunks; e += SA_THREADS) {
            const int r = e / dchunks, c = e - r * dchunks, kp = k0 + r, n = min(8, D - 8 * c);
            float* dst = ks + r * DP + 8 * c;
            const int blk = kp < n_keys ? bt[kp / page] : -1;
            if (blk >= 0 && blk < num_pages) {
                load_row_chunk(k_pool + (((size_t)blk * G + kv) * page + kp % page) * D + 8 * c, dst, n, d8);
            } else {
                if (kp < n_keys && err) atomicOr(err, EMBER_ERR_PAGE_RANGE);
                for (int i = 0; i < n; i++) dst[i] = 0.0f;
            }
        }
        for (int e = threadIdx.x; e < SA_KEYS * vchunks; e += SA_THREADS) {
            const int r = e / vchunks, c = e - r * vchunks, kp = k0 + r, n = min(8, V - 8 * c);
            float* dst = vs + r * VP + 8 * c;
            const int blk = kp < n_keys ? bt[kp / page] : -1;
            if (blk >= 0 && blk < num_pages) {
                load_row_chunk(v_pool + (((size_t)blk * G + kv) * page + kp % page) * V + 8 * c, dst, n, v8);
            } else {
                for (int i = 0; i < n; i++) dst[i] = 0.0f;
            }
        }
        __syncthreads();
        // weights: thread (key kk, rows rg, rg + 4, rg + 8, rg + 12)
        if (rg < n_rows) {
            float sc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
            const float4* kp4 = reinterpret_cast<const float4*>(ks + kk * DP);
            for (int i = 0; i < DP / 4 - 1; i++) {
                const float4 kx = kp4[i];
#pragma unroll
                for (int m = 0; m < 4; m++) {
                    const float4 qx = reinterpret_cast<const float4*>(qs + (rg + 4 * m) * DP)[i];
                    sc[m] = fmaf(qx.x, kx.x, fmaf(qx.y, kx.y, fmaf(qx.z, kx.z, fmaf(qx.w, kx.w, sc[m]))));
                }
            }
#pragma unroll
            for (int m = 0; m < 4; m++) {
                const int r = rg + 4 * m;
                const bool seen = r < n_rows && k0 + kk <= pos0 + r / hpb;
                const float b = head_bias ? head_bias[h0 + r % hpb] : 0.0f;
                ws[r * SA_KEYS + kk] = seen ? 1.0f / (1.0f + expf(-(sc[m] * scale + b))) : 0.0f;
            }
        }
        __syncthreads();
        for (int x = 0; x < SA_KEYS; x += 4) {
            if (k0 + x >= n_keys) break;
            float vv[4][CM];
#pragma unroll
            for (int y = 0; y < 4; y++)
#pragma unroll
                for (int m = 0; m < CM; m++) {
                    const int c = threadIdx.x + m * SA_THREADS;
                    vv[y][m] = c < V ? vs[(x + y) * VP + c] : 0.0f;
                }
#pragma unroll
            for (int r = 0; r < SA_ROWS; r++) {
                if (r >= n_rows) break;
                const float4 w = *reinterpret_cast<const float4*>(ws + r * SA_KEYS + x);
#pragma unroll
                for (int m = 0; m < CM; m++)
                    acc[r][m] = fmaf(w.w, vv[3][m], fmaf(w.z, vv[2][m], fmaf(w.y, vv[1][m], fmaf(w.x, vv[0][m], acc[r][m]))));
            }
        }
    }
#pragma unroll
    for (int r = 0; r < SA_ROWS; r++) {
        if (r >= n_rows) break;
#pragma unroll
        for (int m = 0; m < CM; m++) {
            const int c = threadIdx.x + m * SA_THREADS;
            if (c < V) out[((size_t)(row0 + r / hpb) * H + h0 + r % hpb) * V + c] = from_float<T>(acc[r][m]);
        }
    }
}

// Query heads per block: the largest divisor of the group that is at most 16.
inline int heads_per_block(int group) {
    int h = group < SA_ROWS ? group : SA_ROWS;
    while (group % h) h--;
    return h;
}

// ------------------------------------------------------------------------ bfloat16 cache: tensor-core tiles
// The same attention for bfloat16 queries and cache with head sizes the tiles take (D a multiple of 16, V of 32).
// q . k runs on the tensor cores (mma.sync m16n8k16, bf16 operands, fp32 accumulation: what the fp32 multiply-adds
// of the kernel above compute from the same bf16 values).  Scores, sigmoid and weights are fp32; for the weight x
// value product a weight is cut into three bf16 pieces p = p1 + p2 + p3 (24 bits of mantissa: the fp32 weight, not a
// rounded one) and the three products are added in the fp32 accumulator.  A block: 16 (token, head) rows, 64-key
// tiles fetched with cp.async into two buffers; warp w takes keys 16 w .. 16 w + 15 of a tile for the scores and a
// quarter of the value columns for the read-out; the weights pass through shared memory.
// Blocks start with the tiles of most keys.
constexpr int TC_KEYS = 64, TC_PITCH = TC_KEYS + 8;      // (a row of weights in shared memory)

__device__ __forceinline__ void mma_bf16_16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}
// the three bf16 pieces of two fp32 weights, packed pairwise
__device__ __forceinline__ void split3(float x, float y, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const float x1 = __bfloat162float(__float2bfloat16_rn(x)), y1 = __bfloat162float(__float2bfloat16_rn(y));
    const float xr = x - x1, yr = y - y1;
    const float x2 = __bfloat162float(__float2bfloat16_rn(xr)), y2 = __bfloat162float(__float2bfloat16_rn(yr));
    p1 = pack_bf16(x1, y1); p2 = pack_bf16(x2, y2); p3 = pack_bf16(xr - x2, yr - y2);
}

// The queries of rows g and g + 8 as A operands, kept for the whole key range, with what their scores need.
template <int DK>          // most 16-element steps of a head (D <= 16 DK)
struct TileQueries {
    uint32_t a[DK][4];
    float bias0, bias1;
    int pos0, pos1;

    __device__ __forceinline__ void load(const __nv_bfloat16* __restrict__ q, const float* __restrict__ head_bias, int H, int D, int hpb,
                                         int h0, int row0, int n_rows, int first, int g, int c) {
        const int r0 = g, r1 = g + 8, dk = D >> 4;
        const __nv_bfloat16* q0 = q + ((size_t)(row0 + r0 / hpb) * H + h0 + r0 % hpb) * D;
        const __nv_bfloat16* q1 = q + ((size_t)(row0 + r1 / hpb) * H + h0 + r1 % hpb) * D;
#pragma unroll
        for (int ks = 0; ks < DK; ks++) {
            if (ks < dk) {
                a[ks][0] = r0 < n_rows ? *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + 2 * c) : 0u;
                a[ks][1] = r1 < n_rows ? *reinterpret_cast<const uint32_t*>(q1 + ks * 16 + 2 * c) : 0u;
                a[ks][2] = r0 < n_rows ? *reinterpret_cast<const uint32_t*>(q0 + ks * 16 + 8 + 2 * c) : 0u;
                a[ks][3] = r1 < n_rows ? *reinterpret_cast<const uint32_t*>(q1 + ks * 16 + 8 + 2 * c) : 0u;
            }
        }
        bias0 = (head_bias && r0 < n_rows) ? head_bias[h0 + r0 % hpb] : 0.0f;
        bias1 = (head_bias && r1 < n_rows) ? head_bias[h0 + r1 % hpb] : 0.0f;
        pos0 = first + r0 / hpb;
        pos1 = first + r1 / hpb;
    }
};

// Scores of this warp's 16 keys of the tile at k0 (its keys in Kt), their weights in three pieces to Ps [3][16][TC_PITCH].
template <int DK>
__device__ __forceinline__ void weigh_tile(const TileQueries<DK>& q, const __nv_bfloat16* Kt, __nv_bfloat16* Ps, int D, int k0, int n_rows,
                                           float scale, int warp, int g, int c) {
    const int DP = D + 8, dk = D >> 4;
#pragma unroll
    for (int nb = 0; nb < 2; nb++) {
        float sc[4] = {0.0f, 0.0f, 0.0f, 0.0f};
        const __nv_bfloat16* krow = Kt + (size_t)(16 * warp + 8 * nb + g) * DP + 2 * c;
#pragma unroll
        for (int ks = 0; ks < DK; ks++) {
            if (ks < dk) {
                const uint32_t b0 = *reinterpret_cast<const uint32_t*>(krow + ks * 16);
                const uint32_t b1 = *reinterpret_cast<const uint32_t*>(krow + ks * 16 + 8);
                mma_bf16_16816(sc, q.a[ks], b0, b1);
            }
        }
        const int col = 16 * warp + 8 * nb + 2 * c;                 // this thread's columns: keys k0 + col and the next
        float w[4];
#pragma unroll
        for (int i = 0; i < 4; i++) {
            const int kp = k0 + col + (i & 1), qp = i < 2 ? q.pos0 : q.pos1;
            const bool seen = (i < 2 ? g : g + 8) < n_rows && kp <= qp;
            w[i] = seen ? 1.0f / (1.0f + expf(-(sc[i] * scale + (i < 2 ? q.bias0 : q.bias1)))) : 0.0f;
        }
        uint32_t p1, p2, p3;
        split3(w[0], w[1], p1, p2, p3);
        *reinterpret_cast<uint32_t*>(Ps + (0 * 16 + g) * TC_PITCH + col) = p1;
        *reinterpret_cast<uint32_t*>(Ps + (1 * 16 + g) * TC_PITCH + col) = p2;
        *reinterpret_cast<uint32_t*>(Ps + (2 * 16 + g) * TC_PITCH + col) = p3;
        split3(w[2], w[3], p1, p2, p3);
        *reinterpret_cast<uint32_t*>(Ps + (0 * 16 + g + 8) * TC_PITCH + col) = p1;
        *reinterpret_cast<uint32_t*>(Ps + (1 * 16 + g + 8) * TC_PITCH + col) = p2;
        *reinterpret_cast<uint32_t*>(Ps + (2 * 16 + g + 8) * TC_PITCH + col) = p3;
    }
}
// The weights of 16 keys (step kb of a tile) as A operands, a piece at a time.
__device__ __forceinline__ void load_pieces(uint32_t (&pa)[3][4], const __nv_bfloat16* Ps, int kb, int g, int c) {
#pragma unroll
    for (int part = 0; part < 3; part++) {
        const __nv_bfloat16* pr = Ps + (size_t)(part * 16 + g) * TC_PITCH + kb * 16 + 2 * c;
        pa[part][0] = *reinterpret_cast<const uint32_t*>(pr);
        pa[part][1] = *reinterpret_cast<const uint32_t*>(pr + 8 * TC_PITCH);
        pa[part][2] = *reinterpret_cast<const uint32_t*>(pr + 8);
        pa[part][3] = *reinterpret_cast<const uint32_t*>(pr + 8 * TC_PITCH + 8);
    }
}
// Eight columns of 16 values as a B operand (`row`: this lane's row of them), and weights times values added to acc,
// smallest pieces first.
__device__ __forceinline__ void load_values(uint32_t (&b)[2], const __nv_bfloat16* row) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x2.trans.shared.b16 {%0,%1}, [%2];\n"
                 : "=r"(b[0]), "=r"(b[1]) : "r"((uint32_t)__cvta_generic_to_shared(row)));
}
__device__ __forceinline__ void add_values(float (&acc)[4], const uint32_t (&pa)[3][4], const uint32_t (&b)[2]) {
    mma_bf16_16816(acc, pa[2], b[0], b[1]);
    mma_bf16_16816(acc, pa[1], b[0], b[1]);
    mma_bf16_16816(acc, pa[0], b[0], b[1]);
}
__device__ __forceinline__ void copy_piece(__nv_bfloat16* dst, const __nv_bfloat16* src, int bytes = 16) {      // the rest of 16 is zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes));
}
__device__ __forceinline__ void zero_piece(__nv_bfloat16* dst) { *reinterpret_cast<uint4*>(dst) = make_uint4(0u, 0u, 0u, 0u); }
// Columns col, col + 1 of rows g and g + 8 -> the output.
__device__ __forceinline__ void store_pairs(__nv_bfloat16* __restrict__ out, const float (&acc)[4], int H, int V, int hpb, int h0, int row0,
                                            int n_rows, int g, int col) {
    if (g < n_rows)
        *reinterpret_cast<uint32_t*>(out + ((size_t)(row0 + g / hpb) * H + h0 + g % hpb) * V + col) = pack_bf16(acc[0], acc[1]);
    if (g + 8 < n_rows)
        *reinterpret_cast<uint32_t*>(out + ((size_t)(row0 + (g + 8) / hpb) * H + h0 + (g + 8) % hpb) * V + col) = pack_bf16(acc[2], acc[3]);
}

template <int DK, int NBV>          // NBV: most 8-column blocks a warp reads out
__global__ void __launch_bounds__(128)
sigmoid_attention_tc_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_pool,
                            const __nv_bfloat16* __restrict__ v_pool, __nv_bfloat16* __restrict__ out, int H, int G, int D,
                            int V, int hpb, const int* __restrict__ tiles, const int* __restrict__ block_table, int max_blocks,
                            int page, int num_pages, float scale, const float* __restrict__ head_bias, int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 4 * (gridDim.x - 1 - blockIdx.x);        // later tiles of a run have more keys
    const int run = tile[0], row0 = tile[1], nq = tile[2], pos0 = tile[3];
    const int h0 = blockIdx.y * hpb, kv = h0 / (H / G);
    const int n_rows = nq * hpb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int DP = D + 8, VP = V + 8;                               // row pitches in elements
    __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smem_raw);                 // [2][64][DP]
    __nv_bfloat16* Vs = Ks + 2 * TC_KEYS * DP;                                      // [2][64][VP]
    __nv_bfloat16* Ps = Vs + 2 * TC_KEYS * VP;                                      // [3][16][TC_PITCH]
    const int vw = V >> 2, nbv = vw >> 3;                           // columns and 8-column blocks per warp
    const int n_keys = pos0 + nq;
    const int* bt = block_table + (size_t)run * max_blocks;

    // a thread fetches pieces of one key row (two threads a row, 32 bytes side by side): one look at the block table
    auto fetch = [&](int k0, int buf) {
        const int dch = D >> 3, vch = V >> 3;                      // 16-byte chunks a row (both even)
        const int r = threadIdx.x >> 1, kp = k0 + r;
        const int blk = kp < n_keys ? bt[kp / page] : -1;
        const bool ok = blk >= 0 && blk < num_pages;
        if (!ok && kp < n_keys && err && (threadIdx.x & 1) == 0) atomicOr(err, EMBER_ERR_PAGE_RANGE);
        const size_t at = ok ? ((size_t)blk * G + kv) * page + kp % page : 0;
        const __nv_bfloat16* ksrc = k_pool + at * D;
        const __nv_bfloat16* vsrc = v_pool + at * V;
        __nv_bfloat16* kdst = Ks + ((size_t)buf * TC_KEYS + r) * DP;
        __nv_bfloat16* vdst = Vs + ((size_t)buf * TC_KEYS + r) * VP;
        for (int ch = threadIdx.x & 1; ch < dch + vch; ch += 2) {
            const bool is_k = ch < dch;
            __nv_bfloat16* dst = is_k ? kdst + 8 * ch : vdst + 8 * (ch - dch);
            if (ok) copy_piece(dst, is_k ? ksrc + 8 * ch : vsrc + 8 * (ch - dch));
            else zero_piece(dst);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };

    TileQueries<DK> queries;
    queries.load(q, head_bias, H, D, hpb, h0, row0, n_rows, pos0, g, c);
    float acc[NBV][4];
#pragma unroll
    for (int nb = 0; nb < NBV; nb++) acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.0f;

    fetch(0, 0);
    int buf = 0;
    for (int k0 = 0; k0 < n_keys; k0 += TC_KEYS, buf ^= 1) {
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();                                            // the tile is in; the other buffer and P are free
        if (k0 + TC_KEYS < n_keys) fetch(k0 + TC_KEYS, buf ^ 1);
        const __nv_bfloat16* Vt = Vs + (size_t)buf * TC_KEYS * VP;
        weigh_tile<DK>(queries, Ks + (size_t)buf * TC_KEYS * DP, Ps, D, k0, n_rows, scale, warp, g, c);
        __syncthreads();
        // read-out of this warp's value columns
        const int kbs = min(TC_KEYS, n_keys - k0 + 15) >> 4;        // 16-key steps that hold a visible key
#pragma unroll
        for (int kb = 0; kb < TC_KEYS / 16; kb++) {
            if (kb < kbs) {
                uint32_t pa[3][4];
                load_pieces(pa, Ps, kb, g, c);
#pragma unroll
                for (int nb = 0; nb < NBV; nb++) {
                    if (nb < nbv) {
                        uint32_t b[2];
                        load_values(b, Vt + (size_t)(kb * 16 + (lane & 15)) * VP + warp * vw + nb * 8);
                        add_values(acc[nb], pa, b);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int nb = 0; nb < NBV; nb++)
        if (nb < nbv) store_pairs(out, acc[nb], H, V, hpb, h0, row0, n_rows, g, warp * vw + nb * 8 + 2 * c);
}

// Steps of few blocks (a decoded token: one per request and key/value head) are bound by their longest key range: a tile of
// 64 keys takes the block above about 3 us whatever else runs.  Such a step runs each tile of queries on a cluster of S
// blocks (gridDim.z), S key tiles a round: block z makes the weights of the round's tile z and hands them to all blocks
// through shared memory, then every block reads out its share of the value columns over the S tiles in key order.  So
// an output's sum is the very one of the kernel above, and S may follow the step.  Two cluster barriers a round: weights
// are written once everybody has read the round before, and read once everybody has written.  A round of eight tiles takes
// 5 us (the chain of 96 dependent products a third of it); a layer of 16/8 heads of 128, one request, us: 200 keys 13.3 with
// the kernel above, 6.0 with this; 1,500 keys 70 / 18.5; 8,000 keys 353 / 89; eight requests of 1,500 keys 71 / 37.
template <int DK, int NBW>          // NBW: most 8-column blocks a warp reads out
__global__ void __launch_bounds__(128)
sigmoid_attention_rounds_kernel(const __nv_bfloat16* __restrict__ q, const __nv_bfloat16* __restrict__ k_pool,
                                const __nv_bfloat16* __restrict__ v_pool, __nv_bfloat16* __restrict__ out, int H, int G, int D,
                                int V, int hpb, const int* __restrict__ tiles, const int* __restrict__ block_table, int max_blocks,
                                int page, int num_pages, float scale, const float* __restrict__ head_bias, int* __restrict__ err) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    constexpr int WEIGHTS = 3 * 16 * TC_PITCH;                      // elements of a tile's weights
    const int S = (int)gridDim.z, z = (int)blockIdx.z;              // (S: a power of two)
    pdl_launch_dependents();
    pdl_wait();
    const int* tile = tiles + 4 * (gridDim.x - 1 - blockIdx.x);
    const int run = tile[0], row0 = tile[1], nq = tile[2], pos0 = tile[3];
    const int h0 = blockIdx.y * hpb, kv = h0 / (H / G);
    const int n_rows = nq * hpb;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, c = lane & 3;
    const int nbb = (V / 8 + S - 1) / S, col0 = z * nbb * 8;       // this block's 8-column blocks, from col0 on
    const int DP = D + 8, VP = nbb * 8 + 8;
    __nv_bfloat16* Ks = reinterpret_cast<__nv_bfloat16*>(smem_raw);                 // [64][DP]
    __nv_bfloat16* Vs = Ks + TC_KEYS * DP;                                          // [S * 64][VP]
    __nv_bfloat16* Ps = Vs + S * TC_KEYS * VP;                                      // [S][3][16][TC_PITCH]
    const int n_keys = pos0 + nq, round_keys = S * TC_KEYS;         // (at least one key: the query's own)
    const int* bt = block_table + (size_t)run * max_blocks;

    // The keys of the block's own tile: eight lanes a row, rows (thread / 8) + 16 i; its value columns of all the round's tiles:
    // 16 / S lanes a row, rows (thread / lanes) + (128 / lanes) i.  Pages are looked up a round ahead of the copies.
    const int shift = __ffs(page) - 1;                              // (pages of powers of two only)
    auto page_of = [&](int kp) {                                    // (volatile: not to be put off until it is used)
        kp = min(kp, n_keys - 1);
        int blk;
        asm volatile("ld.global.b32 %0, [%1];" : "=r"(blk) : "l"(bt + (kp >> shift)));
        return blk;
    };
    auto row_of = [&](int blk, int kp, int& bytes) {                // in the pools; bytes: 16, 0 for a row of zeros
        const bool ok = kp < n_keys && blk >= 0 && blk < num_pages;
        bytes = ok ? 16 : 0;
        return ok ? (unsigned)(blk * G + kv) * (unsigned)page + (unsigned)(kp & (page - 1)) : 0u;
    };
    // (straight-line over the rows: a scheduler has one warp, so what a copy costs is its chain of instructions)
    auto copy_rows = [&](auto n_c, const __nv_bfloat16* pool, int width, const int* pages, int first, int step, __nv_bfloat16* dst, int pitch,
                         int chunk, int chunk_step, int chunks) {
        constexpr int N = decltype(n_c)::value;
        const __nv_bfloat16* src[N];
        int bytes[N];
#pragma unroll
        for (int i = 0; i < N; i++) src[i] = pool + (size_t)row_of(pages[i], first + step * i, bytes[i]) * width;
        for (int ch = chunk; ch < chunks; ch += chunk_step)
#pragma unroll
            for (int i = 0; i < N; i++) copy_piece(dst + (size_t)(step * i) * pitch + 8 * ch, src[i] + 8 * ch, bytes[i]);
    };
    const int k_row = threadIdx.x >> 3, v_lanes = 16 / S, v_rows = 8 * S, v_row = (int)threadIdx.x / v_lanes, v_lane = (int)threadIdx.x % v_lanes;
    const int v_chunks = min(nbb, V / 8 - z * nbb);
    int k_page[4], v_page[8];
    auto look_k = [&](int r0) {
#pragma unroll
        for (int i = 0; i < 4; i++) k_page[i] = page_of(r0 + z * TC_KEYS + k_row + 16 * i);
    };
    auto look_v = [&](int r0) {
#pragma unroll
        for (int i = 0; i < 8; i++) v_page[i] = page_of(r0 + v_row + v_rows * i);
    };
    auto fetch_k = [&](int r0) {
        const int first = r0 + z * TC_KEYS + k_row;
        bool outside = false;
#pragma unroll
        for (int i = 0; i < 4; i++) outside |= first + 16 * i < n_keys && (k_page[i] < 0 || k_page[i] >= num_pages);
        if (outside && err && (threadIdx.x & 7) == 0) atomicOr(err, EMBER_ERR_PAGE_RANGE);
        copy_rows(std::integral_constant<int, 4>(), k_pool, D, k_page, first, 16, Ks + (size_t)k_row * DP, DP, threadIdx.x & 7, 8, D / 8);
    };
    auto fetch_v = [&](int r0) {
        copy_rows(std::integral_constant<int, 8>(), v_pool + col0, V, v_page, r0 + v_row, v_rows, Vs + (size_t)v_row * VP, VP, v_lane, v_lanes, v_chunks);
    };
    // rows past n_rows have no weights: those of other blocks' tiles are zeroed once and not handed over
    for (int e = (int)threadIdx.x; e < S * WEIGHTS / 8; e += 128) zero_piece(Ps + 8 * e);
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");           // (waited for before the first weights go out)

    look_k(0);
    look_v(0);
    TileQueries<DK> queries;
    queries.load(q, head_bias, H, D, hpb, h0, row0, n_rows, pos0, g, c);
    fetch_k(0);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    look_k(round_keys);
    float acc[NBW][4];
#pragma unroll
    for (int nb = 0; nb < NBW; nb++) acc[nb][0] = acc[nb][1] = acc[nb][2] = acc[nb][3] = 0.0f;
    for (int r0 = 0; r0 < n_keys; r0 += round_keys) {
        const bool more = r0 + round_keys < n_keys;
        fetch_v(r0);                                                // (every warp of the block has read the round before)
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        look_v(r0 + round_keys);
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();                                            // the keys are in
        const int k0 = r0 + z * TC_KEYS;
        __nv_bfloat16* mine = Ps + (size_t)z * WEIGHTS;
        if (k0 < n_keys) weigh_tile<DK>(queries, Ks, mine, D, k0, n_rows, scale, warp, g, c);
        __syncthreads();                                            // the weights are there, the keys free
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");         // everybody has read the round before
        if (k0 < n_keys) {
            // 16-byte pieces, eight a row, to every other block
            const int pieces = 3 * n_rows * 8;
            for (int e = (int)threadIdx.x; e < pieces * (S - 1); e += 128) {
                const int peer = (z + 1 + e / pieces) & (S - 1), r = (e % pieces) >> 3;
                __nv_bfloat16* piece = mine + (size_t)(r / n_rows * 16 + r % n_rows) * TC_PITCH + (e & 7) * 8;
                const uint4 v = *reinterpret_cast<const uint4*>(piece);
                uint32_t there;
                asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(there) : "r"((uint32_t)__cvta_generic_to_shared(piece)), "r"(peer));
                asm volatile("st.shared::cluster.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(there), "r"(v.x), "r"(v.y), "r"(v.z), "r"(v.w) : "memory");
            }
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");      // this thread's values are in
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        if (more) fetch_k(r0 + round_keys);                         // (while the others arrive)
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        look_k(r0 + 2 * round_keys);
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");         // the round's weights and values are here
        for (int j = 0; j < S && r0 + j * TC_KEYS < n_keys; j++) {
            const int kbs = min(TC_KEYS, n_keys - (r0 + j * TC_KEYS) + 15) >> 4;
            const __nv_bfloat16* Vt = Vs + (size_t)(j * TC_KEYS + (lane & 15)) * VP;
            const __nv_bfloat16* Pt = Ps + (size_t)j * WEIGHTS;
#pragma unroll
            for (int half = 0; half < 2; half++) {
                // two steps of 16 keys: all that they read is asked for before their products
                uint32_t pa[2][3][4], b[2][NBW][2];
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    load_pieces(pa[u], Pt, 2 * half + u, g, c);
#pragma unroll
                    for (int i = 0; i < NBW; i++)
                        load_values(b[u][i], Vt + (size_t)(2 * half + u) * 16 * VP + (warp + 4 * i < nbb ? warp + 4 * i : 0) * 8);
                }
#pragma unroll
                for (int u = 0; u < 2; u++)
#pragma unroll
                    for (int i = 0; i < NBW; i++)
                        if (2 * half + u < kbs) add_values(acc[i], pa[u], b[u][i]);
            }
        }
        if (more) asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < NBW; i++) {
        const int nb = warp + 4 * i;
        if (nb < nbb && col0 + 8 * nb < V) store_pairs(out, acc[i], H, V, hpb, h0, row0, n_rows, g, col0 + nb * 8 + 2 * c);
    }
}

inline bool tc_attend_on() {
    static int on = -1;
    if (on < 0) { const char* e = getenv("EMBER_SIGMOID_ATTENTION_TC"); on = (e && e[0] == '0') ? 0 : 1; }
    return on != 0;
}

// Blocks of a cluster for the kernel of rounds, 1 for the other one: as many as the SMs hold at once (two a block where
// shared memory allows it), while a round is not half empty.
inline size_t rounds_smem(int S, int D, int V) {
    const int nbb = (V / 8 + S - 1) / S;
    return ((size_t)TC_KEYS * (D + 8) + (size_t)S * TC_KEYS * (nbb * 8 + 8) + (size_t)S * 3 * 16 * TC_PITCH) * sizeof(__nv_bfloat16);
}
inline int cluster_blocks(long long blocks, int D, int V, int page, long long most_keys, int num_sms) {
    if (page & (page - 1)) return 1;
    for (int S = 8; S > 1; S >>= 1) {
        const size_t smem = rounds_smem(S, D, V);
        if (smem <= 227 * 1024 && blocks * S <= (long long)num_sms * (smem <= 112 * 1024 ? 2 : 1) && most_keys > (long long)(S / 2) * TC_KEYS) return S;
    }
    return 1;
}

template <int DK, int NBV>
int launch_attend_tc(const void* q, const void* k_pool, const void* v_pool, void* out, int H, int G, int D, int V, int hpb,
                     const int* tiles, int n_tiles, const int* bt, int max_blocks, int page, int num_pages, float scale,
                     const float* head_bias, int num_sms, int* err, cudaStream_t st) {
    const int S = cluster_blocks((long long)n_tiles * (H / hpb), D, V, page, (long long)max_blocks * page, num_sms);
    if (S > 1) {
        const size_t smem = rounds_smem(S, D, V);
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(n_tiles, H / hpb, S);
        cfg.blockDim = dim3(128);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute attrs[2];
        attrs[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attrs[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
        attrs[1].id = cudaLaunchAttributeClusterDimension;
        attrs[1].val.clusterDim.x = 1; attrs[1].val.clusterDim.y = 1; attrs[1].val.clusterDim.z = (unsigned)S;
        cfg.attrs = attrs; cfg.numAttrs = 2;
        const auto run = [&](auto kernel) -> int {
            const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
            if (e != cudaSuccess) return fail("sigmoid_attention: shared memory %zu: %s", smem, cudaGetErrorString(e));
            cudaLaunchKernelEx(&cfg, kernel, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool,
                               (__nv_bfloat16*)out, H, G, D, V, hpb, tiles, bt, max_blocks, page, num_pages, scale, head_bias, err);
            return check_launch("sigmoid_attention");
        };
        const int most = ((V / 8 + S - 1) / S + 3) / 4;             // 8-column blocks of a warp
        return most <= 1 ? run(sigmoid_attention_rounds_kernel<DK, 1>)
                         : (most <= 2 ? run(sigmoid_attention_rounds_kernel<DK, 2>) : run(sigmoid_attention_rounds_kernel<DK, 8>));
    }
    const size_t smem = ((size_t)2 * TC_KEYS * (D + 8) + (size_t)2 * TC_KEYS * (V + 8) + 3 * 16 * TC_PITCH) * sizeof(__nv_bfloat16);
    if (smem > 48 * 1024) cudaFuncSetAttribute(sigmoid_attention_tc_kernel<DK, NBV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    launch_kernel(sigmoid_attention_tc_kernel<DK, NBV>, dim3(n_tiles, H / hpb), 128, smem, st, (const __nv_bfloat16*)q,
                  (const __nv_bfloat16*)k_pool, (const __nv_bfloat16*)v_pool, (__nv_bfloat16*)out, H, G, D, V, hpb, tiles, bt, max_blocks,
                  page, num_pages, scale, head_bias, err);
    return check_launch("sigmoid_attention");
}

template <typename T>
int launch_attend(const void* q, const void* k_pool, const void* v_pool, void* out, int H, int G, int D, int V,
                  const int* tiles, int n_tiles, const int* bt, int max_blocks, int page, int num_pages, float scale,
                  const float* head_bias, int* err, cudaStream_t st) {
    const int DP = (D + 3) / 4 * 4 + 4, VP = (V + 3) / 4 * 4, hpb = heads_per_block(H / G);
    const size_t smem = ((size_t)(SA_ROWS + SA_KEYS) * DP + (size_t)SA_KEYS * VP + SA_ROWS * SA_KEYS) * sizeof(float);
    if (smem > 200 * 1024) return fail("sigmoid_attention: heads of %d / %d do not fit in shared memory", D, V);
    const int cm = (V + SA_THREADS - 1) / SA_THREADS;
#define EMBER_SA_LAUNCH(CM)                                                                                              \
    do {                                                                                                                 \
        if (smem > 48 * 1024)                                                                                            \
            cudaFuncSetAttribute(sigmoid_attention_kernel<T, CM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        launch_kernel(sigmoid_attention_kernel<T, CM>, dim3(n_tiles, H / hpb), SA_THREADS, smem, st, (const T*)q, (const T*)k_pool, \
                      (const T*)v_pool, (T*)out, H, G, D, V, hpb, tiles, bt, max_blocks, page, num_pages, scale, head_bias, err); \
    } while (0)
    if (cm <= 1) EMBER_SA_LAUNCH(1);
    else if (cm == 2) EMBER_SA_LAUNCH(2);
    else if (cm <= 4) EMBER_SA_LAUNCH(4);
    else return fail("sigmoid_attention: value heads of %d are wider than 512", V);
#undef EMBER_SA_LAUNCH
    return check_launch("sigmoid_attention");
}

}  // namespace ember

using namespace ember;

EMBER_API int ember_sigmoid_attention_tile_queries(int group) { return group > 0 ? SA_ROWS / heads_per_block(group) : 0; }

EMBER_API int ember_rotate_store(const float* qkv, int ld, int T, int H, int G, int D, int V, const float* inv_freq, int rotary,
                                 const int* positions, const int* seq_of, const int* block_table, int max_blocks, int page,
                                 int num_pages, void* q_out, void* k_pool, void* v_pool, int dtype, int write_kv, int* err,
                                 void* stream) {
    if (T <= 0) return 0;
    if (H <= 0 || G <= 0 || D <= 0 || V <= 0 || ld < (H + G) * D + G * V) return fail("rotate_store: %d/%d heads of %d / %d in rows of %d", H, G, D, V, ld);
    if (rotary < 0 || rotary > D || (rotary & 1) || (rotary && !inv_freq)) return fail("rotate_store: rotation of %d in heads of %d", rotary, D);
    if (page <= 0 || max_blocks <= 0 || num_pages <= 0) return fail("rotate_store: bad cache geometry");
    cudaStream_t st = (cudaStream_t)stream;
    const size_t smem = (size_t)(rotary > 0 ? rotary : 2) * sizeof(float);
    if (dtype == EMBER_F32)
        launch_kernel(rotate_store_kernel<float>, T, 256, smem, st, qkv, ld, H, G, D, V, inv_freq, rotary, positions, seq_of, block_table,
                      max_blocks, page, num_pages, (float*)q_out, (float*)k_pool, (float*)v_pool, write_kv, err);
    else if (dtype == EMBER_BF16)
        launch_kernel(rotate_store_kernel<__nv_bfloat16>, T, 256, smem, st, qkv, ld, H, G, D, V, inv_freq, rotary, positions, seq_of,
                      block_table, max_blocks, page, num_pages, (__nv_bfloat16*)q_out, (__nv_bfloat16*)k_pool, (__nv_bfloat16*)v_pool,
                      write_kv, err);
    else
        return fail("rotate_store: unsupported dtype %d", dtype);
    return check_launch("rotate_store");
}

EMBER_API int ember_sigmoid_attention(const void* q, const void* k_pool, const void* v_pool, void* out, int dtype, int H, int G,
                                      int D, int V, const int* tiles, int n_tiles, const int* block_table, int max_blocks, int page,
                                      int num_pages, float scale, const float* head_bias, int num_sms, int* err, void* stream) {
    if (n_tiles <= 0) return 0;
    if (H <= 0 || G <= 0 || H % G || D <= 0 || V <= 0) return fail("sigmoid_attention: %d/%d heads of %d / %d", H, G, D, V);
    if (H > 65535) return fail("sigmoid_attention: too many heads for one launch");
    cudaStream_t st = (cudaStream_t)stream;
    if (dtype == EMBER_F32)
        return launch_attend<float>(q, k_pool, v_pool, out, H, G, D, V, tiles, n_tiles, block_table, max_blocks, page, num_pages, scale, head_bias, err, st);
    if (dtype == EMBER_BF16 && tc_attend_on() && D % 16 == 0 && V % 32 == 0 && D <= 256 && V <= 512) {
        const int hpb = heads_per_block(H / G);
#define EMBER_SA_TC(DK, NBV) launch_attend_tc<DK, NBV>(q, k_pool, v_pool, out, H, G, D, V, hpb, tiles, n_tiles, block_table, \
                                                       max_blocks, page, num_pages, scale, head_bias, num_sms, err, st)
        if (D <= 128) return V <= 128 ? EMBER_SA_TC(8, 4) : EMBER_SA_TC(8, 16);
        return V <= 128 ? EMBER_SA_TC(16, 4) : EMBER_SA_TC(16, 16);
#undef EMBER_SA_TC
    }
    if (dtype == EMBER_BF16)
        return launch_attend<__nv_bfloat16>(q, k_pool, v_pool, out, H, G, D, V, tiles, n_tiles, block_table, max_blocks, page, num_pages, scale, head_bias, err, st);
    return fail("sigmoid_attention: unsupported dtype %d", dtype);
}
