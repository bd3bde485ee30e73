// What turns runs of new tokens of latent attention (see latent_attention.cu for the mechanism) into plain attention with a key and
// a value a head, for attention_prefill_tc.cu's form with keys of 192 and values of 128.
//
// The walk over the latents costs 2 H (E + R) operations a visible pair (1,088 numbers a head at R 512, P 64) and applies the heads'
// matrices to every query; with the keys W_uk c and the values W_uv c written out it costs 2 H (192 + 128) a pair, on the tensor
// pipe, and the matrices are applied once a cached vector, by one product.  For single tokens the walk reads far less.
//
//   latent_gather    the cached vectors a step's sequences see, from their pages into rows: the latents [keys, R] (what that product
//                    reads) and the rotated parts [keys, 64] (zeros behind P).  A sequence's keys start on a multiple of 128
//                    positions and end on one; rows of positions it does not see are zeros, so that its last tile holds nothing of
//                    another sequence.
//   latent_queries   q [rows, H (128 + P)] float32 -> [rows, H * 192] bfloat16, the rotated part turned by the row's position in
//                    float32 (zeros behind P), rounded once.
// Both are bound by the bytes they move (16 bytes a thread and access).
//
// A layer of 32 heads, R 512, P 64 over one prompt of 2,048 tokens: 10 us gathering, 16 us for the queries, 40 us for the product, 68 us
// of attention; before, 1,145 us for the walk and 337 us for the heads' matrices.
#include "api.h"
#include "common.cuh"

namespace citlali {

constexpr int kKeyTile = 128;

// Tiles of 128 positions that a sequence's new rows see: the first one and the one behind the last.
__device__ __forceinline__ int2 seen_tiles(int past, int n, int window) {
    const int lo = window > 0 ? max(0, past - window + 1) : 0;
    return make_int2(lo / kKeyTile, n > 0 ? (past + n - 1) / kKeyTile + 1 : lo / kKeyTile);
}

// Whether one of eight bfloat16 has all bits of its exponent set.
__device__ __forceinline__ bool not_all_finite(uint4 v) {
    auto pair = [](uint32_t w) { return (w & 0x7f800000u) == 0x7f800000u || (w & 0x7f80u) == 0x7f80u; };
    return pair(v.x) || pair(v.y) || pair(v.z) || pair(v.w);
}

__global__ void __launch_bounds__(256)
latent_gather_kernel(const __nv_bfloat16* __restrict__ pool, const int32_t* __restrict__ page_table, int table_stride, int page_size,
                     const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_slot, const int32_t* __restrict__ seq_past,
                     int R, int P, int window, __nv_bfloat16* __restrict__ latents, __nv_bfloat16* __restrict__ shared_keys,
                     int32_t* __restrict__ key_rows, int key_total) {
    __shared__ int first_row;
    __shared__ int spoilt[32];                                // this block's rows whose latents are not all finite
    dependents_may_launch();
    wait_for_predecessor();
    const int seq = blockIdx.y, lane = threadIdx.x & 31;
    const int past = seq_past[seq], n = seq_start[seq + 1] - seq_start[seq];
    const int2 mine = seen_tiles(past, n, window);
    const int tile = mine.x + blockIdx.x / 4;                 // four blocks a tile: 32 rows each
    if (tile >= mine.y) return;
    if (threadIdx.x < 32) {                                   // the rows of the sequences before this one
        spoilt[lane] = 0;
        int before = 0;
        for (int s = lane; s < seq; s += 32) {
            const int2 t = seen_tiles(seq_past[s], seq_start[s + 1] - seq_start[s], window);
            before += t.y - t.x;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (lane == 0) first_row = (before - mine.x) * kKeyTile;
    }
    __syncthreads();
    if (blockIdx.x == 0 && threadIdx.x == 0) key_rows[seq] = first_row;
    const int lo = window > 0 ? max(0, past - window + 1) : 0, hi = past + n;        // the positions seen
    const int E = R + P, chunks = (R + 64) / 8, r_chunks = R / 8, e_chunks = E / 8;
    const int32_t* table = page_table + (size_t)seq_slot[seq] * table_stride;
    const int key0 = tile * kKeyTile + (blockIdx.x & 3) * 32;
    for (int i = threadIdx.x; i < 32 * chunks; i += 256) {
        const int r = i / chunks, key = key0 + r, ch = i % chunks, row = first_row + key;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (key >= lo && key < hi && ch < e_chunks)
            v = *reinterpret_cast<const uint4*>(pool + ((size_t)table[key / page_size] * page_size + key % page_size) * E + ch * 8);
        if (row >= key_total) continue;                       // (a caller that counted otherwise: nothing is written past its buffers)
        if (ch < r_chunks) {
            *reinterpret_cast<uint4*>(latents + (size_t)row * R + ch * 8) = v;
            if (not_all_finite(v)) spoilt[r] = 1;
        } else {
            *reinterpret_cast<uint4*>(shared_keys + (size_t)row * 64 + (ch - r_chunks) * 8) = v;
        }
    }
    __syncthreads();
    // A latent that is not all finite (and was written: those rows alone are marked): its values would meet the zeros that rows which do
    // not see it have for weights.  They become zero, and a key that is not a number says the same to the rows that do see it.
    for (int r = threadIdx.x >> 5; r < 32; r += 8) {
        if (!spoilt[r]) continue;
        const size_t row = first_row + key0 + r;
        for (int ch = threadIdx.x & 31; ch < r_chunks; ch += 32) *reinterpret_cast<uint4*>(latents + row * R + ch * 8) = make_uint4(0u, 0u, 0u, 0u);
        if ((threadIdx.x & 31) < 8)
            *reinterpret_cast<uint4*>(shared_keys + row * 64 + (threadIdx.x & 31) * 8) = make_uint4(0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu, 0x7fff7fffu);
    }
}

// A block a row; a thread four neighbouring elements (192 and 128 + P are multiples of four).
__global__ void __launch_bounds__(256)
latent_queries_kernel(const float* __restrict__ q, int H, int P, const float* __restrict__ inv_freq, int rot_dims, int rot_halves,
                      const int32_t* __restrict__ row_pos, __nv_bfloat16* __restrict__ out) {
    __shared__ float2 turn[32];                               // the row's cosines and sines
    dependents_may_launch();
    wait_for_predecessor();
    const int row = blockIdx.x, half = rot_dims >> 1;
    if (threadIdx.x < half) {
        float sn, cs;
        sincosf((float)row_pos[row] * inv_freq[threadIdx.x], &sn, &cs);
        turn[threadIdx.x] = make_float2(cs, sn);
    }
    __syncthreads();
    const float* src = q + (size_t)row * H * (128 + P);
    __nv_bfloat16* dst = out + (size_t)row * H * 192;
    for (int i = threadIdx.x; i < H * 48; i += 256) {
        const int h = i / 48, e = (i % 48) * 4;
        const float* head = src + (size_t)h * (128 + P);
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (e < 128 + P) v = *reinterpret_cast<const float4*>(head + e);
        if (e >= 128 && e < 128 + P) {
            const int r = e - 128;                            // place in the rotated part
            float x[4] = {v.x, v.y, v.z, v.w};
            if (rot_halves) {
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int k = r + c;
                    if (k >= rot_dims) break;
                    const bool first = k < half;
                    const float2 t = turn[first ? k : k - half];
                    const float other = head[128 + (first ? k + half : k - half)];
                    x[c] = first ? x[c] * t.x - other * t.y : x[c] * t.x + other * t.y;
                }
            } else {
#pragma unroll
                for (int c = 0; c < 4; c += 2) {
                    if (r + c >= rot_dims) break;
                    const float2 t = turn[(r + c) >> 1];
                    const float a = x[c] * t.x - x[c + 1] * t.y, b = x[c + 1] * t.x + x[c] * t.y;
                    x[c] = a; x[c + 1] = b;
                }
            }
            v = make_float4(x[0], x[1], x[2], x[3]);
        }
        __nv_bfloat162 lo = __floats2bfloat162_rn(v.x, v.y), hi = __floats2bfloat162_rn(v.z, v.w);
        *reinterpret_cast<uint2*>(dst + h * 192 + e) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    }
}

}  // namespace citlali

using namespace citlali;

extern "C" int citlali_latent_gather(const void* pool, const int32_t* page_table, int table_stride, int page_size,
                                     const int32_t* seq_start, const int32_t* seq_slot, const int32_t* seq_past, int sequences,
                                     int max_tiles, int R, int P, int window, void* latents, void* shared_keys, int32_t* key_rows,
                                     int key_total, cudaStream_t stream) {
    if (sequences <= 0 || max_tiles <= 0) return 0;
    if (R <= 0 || R % 8 != 0 || P < 0 || P > 64 || P % 8 != 0 || sequences > 65535) {
        set_last_error("latent_gather: a latent of %d and a shared key part of %d (multiples of eight, the part at most 64), %d sequences", R, P, sequences);
        return kBadShape;
    }
    if (((uintptr_t)pool | (uintptr_t)latents | (uintptr_t)shared_keys) & 15u) {
        set_last_error("latent_gather: operands must be 16-byte aligned");
        return kBadAlignment;
    }
    dim3 grid(max_tiles * 4, sequences);
    launch_kernel(latent_gather_kernel, grid, 256, 0, stream, (const __nv_bfloat16*)pool, page_table, table_stride, page_size, seq_start,
                  seq_slot, seq_past, R, P, window, (__nv_bfloat16*)latents, (__nv_bfloat16*)shared_keys, key_rows, key_total);
    return CITLALI_LAUNCH_CHECK();
}

extern "C" int citlali_latent_queries(const float* q, int H, int P, const float* inv_freq, int rot_dims, int rot_halves,
                                      const int32_t* row_pos, void* out, int rows, cudaStream_t stream) {
    if (rows <= 0) return 0;
    if (H <= 0 || P < 0 || P > 64 || P % 4 != 0 || rot_dims < 0 || rot_dims > P || (rot_dims & 1)) {
        set_last_error("latent_queries: %d rotated dimensions of a part of %d (a multiple of four, at most 64)", rot_dims, P);
        return kBadShape;
    }
    if (((uintptr_t)q | (uintptr_t)out) & 15u) {
        set_last_error("latent_queries: operands must be 16-byte aligned");
        return kBadAlignment;
    }
    launch_kernel(latent_queries_kernel, rows, 256, 0, stream, q, H, P, inv_freq, rot_dims, rot_halves, row_pos, (__nv_bfloat16*)out);
    return CITLALI_LAUNCH_CHECK();
}
