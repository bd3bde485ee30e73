// y[M, N] = x[M, K] . w[N, K]^T on CUDA cores: float accumulation, k strictly ascending.
//
// This is the matrix product of the true 32-bit path, and the bfloat16 path's product for
// shapes the tensor-core kernel refuses.  One output element is one chain of fused
// multiply-adds over k = 0 .. K-1; the chain does not depend on M, on N, on where the
// element lies in a tile or on what else is in the batch, so a row's result is the same
// however the rows were cut into steps.  (The reference's product is one block per output
// row with a tree reduction, matvec_fp16_kernel, kernels.cu:381-449.)
#include "api.h"
#include "common.cuh"

namespace citlali {

constexpr int kTileM = 64, kTileN = 64, kTileK = 16;

template <typename TX, typename TW, typename TY, bool kAccumulate>
__global__ void __launch_bounds__(256)
gemm_simt_kernel(const TX* __restrict__ x, const TW* __restrict__ w, TY* __restrict__ y, int M, int N, int K) {
    __shared__ float xs[kTileK][kTileM + 4];
    __shared__ float ws[kTileK][kTileN + 4];
    dependents_may_launch();
    wait_for_predecessor();
    const int m0 = blockIdx.y * kTileM, n0 = blockIdx.x * kTileN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 x 16 threads, 4 x 4 outputs each
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;

    for (int k0 = 0; k0 < K; k0 += kTileK) {
        // 64 rows x 16 k of each operand; 256 threads load 4 elements each, k fastest.
        for (int e = threadIdx.x; e < kTileM * kTileK; e += 256) {
            const int r = e / kTileK, kk = e % kTileK;
            const int gm = m0 + r, gn = n0 + r, gk = k0 + kk;
            xs[kk][r] = (gm < M && gk < K) ? ldf(x, (size_t)gm * K + gk) : 0.0f;
            ws[kk][r] = (gn < N && gk < K) ? ldf(w, (size_t)gn * K + gk) : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kTileK; ++kk) {
            float a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = xs[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn >= N) continue;
            const size_t o = (size_t)gm * N + gn;
            if (kAccumulate) stf(y, o, ldf(y, o) + acc[i][j]);
            else stf(y, o, acc[i][j]);
        }
    }
}

// The same product for float32 operands and many rows: the same chain an element (k ascending, the last 16 k filled up with
// zeros), so the same bits as the kernel above.
// What bounds it: the FMA units.  A thread owns 8 x RN outputs, so that a k costs it four (three) 16-byte reads of shared memory
// for 64 (32) multiply-adds, two of them an instruction (fma.rn.f32x2 rounds each half like fmaf); both operands lie transposed
// [k][row] in shared memory, put there element by element by asynchronous copies (any alignment, any K) three tiles deep.
// TN = 128 for matrices with tiles enough for every SM twice, TN = 64 for some that cannot be copied in pieces; the others run the
// kernel behind this one (see launch_wide).  682 rows, K 1,024: N 5,632
// 212 us, N 32,768 977 (18.6 and 23.4 T multiply-adds a second of 37).
__device__ __forceinline__ void cp_async4_or_zero(uint32_t dst, const float* src, bool there) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(there ? 4 : 0) : "memory");
}
__device__ __forceinline__ unsigned long long fma2(unsigned long long a, unsigned long long b, unsigned long long c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ unsigned long long both(float v) {
    unsigned long long d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}

template <int TN, bool kAccumulate>
__global__ void __launch_bounds__(128, 3)
gemm_simt_wide_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K) {
    constexpr int TM = 64, STAGES = 3, TX = 16, RN = TN / TX, LX = TM + 4, LW = TN + 4;
    __shared__ __align__(16) float xs[STAGES][kTileK][LX];
    __shared__ __align__(16) float ws[STAGES][kTileK][LW];
    dependents_may_launch();
    wait_for_predecessor();
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;   // 16 x 8 threads
    const int lk = threadIdx.x & 15, lr = threadIdx.x >> 4;   // loading: 16 k of 8 rows a pass
    const uint32_t xs_a = (uint32_t)__cvta_generic_to_shared(&xs[0][0][0]), ws_a = (uint32_t)__cvta_generic_to_shared(&ws[0][0][0]);
    const int tiles = (K + kTileK - 1) / kTileK;
    auto fetch = [&](int tile) {
        if (tile < tiles) {
            const int st = tile % STAGES, gk = tile * kTileK + lk;
#pragma unroll
            for (int r = 0; r < TM; r += 8) {
                const bool there = m0 + lr + r < M && gk < K;
                cp_async4_or_zero(xs_a + (uint32_t)(((st * kTileK + lk) * LX + lr + r) * 4), there ? x + (size_t)(m0 + lr + r) * K + gk : x, there);
            }
#pragma unroll
            for (int r = 0; r < TN; r += 8) {
                const bool there = n0 + lr + r < N && gk < K;
                cp_async4_or_zero(ws_a + (uint32_t)(((st * kTileK + lk) * LW + lr + r) * 4), there ? w + (size_t)(n0 + lr + r) * K + gk : w, there);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    unsigned long long acc[8][RN / 2];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < RN / 2; ++j) acc[i][j] = 0ull;
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    for (int t = 0; t < tiles; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                          // the tile has landed for every thread; the one before it is no longer read
        fetch(t + STAGES - 1);
        const int st = t % STAGES;
#pragma unroll
        for (int kk = 0; kk < kTileK; ++kk) {
            float a[8];
            unsigned long long b[RN / 2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {         // rows 4 ty .. 4 ty + 3 of either half of the tile
                const float4 v = *reinterpret_cast<const float4*>(&xs[st][kk][h * 32 + ty * 4]);
                a[4 * h] = v.x; a[4 * h + 1] = v.y; a[4 * h + 2] = v.z; a[4 * h + 3] = v.w;
            }
#pragma unroll
            for (int h = 0; h < RN / 4; ++h) {
                const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(&ws[st][kk][h * 64 + tx * 4]);
                b[2 * h] = v.x; b[2 * h + 1] = v.y;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long ai = both(a[i]);
#pragma unroll
                for (int j = 0; j < RN / 2; ++j) acc[i][j] = fma2(ai, b[j], acc[i][j]);
            }
        }
    }
    const bool quads = N % 4 == 0 && (reinterpret_cast<uintptr_t>(y) & 15) == 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int gm = m0 + (i >> 2) * 32 + ty * 4 + (i & 3);
        if (gm >= M) continue;
#pragma unroll
        for (int h = 0; h < RN / 4; ++h) {
            const int gn = n0 + h * 64 + tx * 4;
            float v[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) v[e] = __uint_as_float((uint32_t)(acc[i][2 * h + (e >> 1)] >> (32 * (e & 1))));
            float* dst = y + (size_t)gm * N + gn;
            if (quads && gn < N) {
                if (kAccumulate) {
                    const float4 old = *reinterpret_cast<const float4*>(dst);
                    v[0] = old.x + v[0]; v[1] = old.y + v[1]; v[2] = old.z + v[2]; v[3] = old.w + v[3];
                }
                *reinterpret_cast<float4*>(dst) = make_float4(v[0], v[1], v[2], v[3]);
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (gn + e < N) dst[e] = kAccumulate ? dst[e] + v[e] : v[e];
            }
        }
    }
}

// The same product again, the same chains, for matrices of few tiles: 64 rows x 16 RN columns a block of
// 2 x 2 warps, RN chosen so that the tiles go round the SMs as evenly as they can (narrow_columns).
// What bounds it: a block or two an SM, a warp or two a scheduler, so the chain of reads and multiply-adds of a thread.  Rows of both
// operands lie in shared memory as they do in memory, 32 k of each, copied in 16-byte pieces (kPieces; else element by element) three
// tiles deep; a thread's 16-byte reads are four k of a row, so a copy costs a quarter of the instructions, and 8 RN multiply-adds a k
// need no moves.  Element by element a warp copies 32 k of one row (eight lanes a row, four k apart: 49 -> 45 us at 682 rows, N 1,024, K 1,022).
// Lanes are placed as in the delta rule's scan: two that read the same place are neighbours or two apart, and a read
// costs two wavefronts.
// 682 rows one product after another, 64 x 64 tiles of the kernel above -> here: N 1,024, K 1,024 / 2,816 (143 tiles of 64 x 80 instead of
// 176) 94 / 223 -> 43 / 112 us; N 1,536, K 1,024 97 -> 62; 200 rows, N 1,024 / 1,536 47 / 71 -> 22 / 29; 33 rows, N 1,024 41 -> 21.
template <int RN, bool kPieces, bool kAccumulate>
__global__ void __launch_bounds__(128, 3)
gemm_simt_narrow_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K) {
    constexpr int RM = 8, TM = 64, TN = 16 * RN, TK = 32, LD = TK + 4, STAGES = 3;
    constexpr int kCopies = (TM + TN) / 16;                 // pieces a thread and tile: 16 rows of 8 pieces a pass
    extern __shared__ __align__(16) float narrow_tiles[];   // [STAGES][rows of x, rows of w][LD]
    dependents_may_launch();
    wait_for_predecessor();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = (lane & 1) | ((lane >> 1) & 2) | ((lane >> 2) & 4), ty = ((lane >> 1) & 1) | ((lane >> 2) & 2);    // lane bits 0 2 4; 1 3
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN;
    const int count = (K + TK - 1) / TK;
    // in pieces: eight threads a row, a thread's rows 16 apart; element by element: a warp a row, so that a copy asks for four or five
    // sectors, its rows four apart
    const int lk = kPieces ? (tid & 7) * 4 : lane, lr = kPieces ? tid >> 3 : warp;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(narrow_tiles) + (uint32_t)((lr * LD + lk) * 4);
    const float* src[kPieces ? kCopies : 1];
    bool in[kPieces ? kCopies : 1];
    if constexpr (kPieces) {
#pragma unroll
        for (int i = 0; i < kCopies; ++i) {
            const int r = 16 * i + lr, row = r < TM ? m0 + r : n0 + r - TM;      // (TM a multiple of 16: a pass is all x or all w)
            in[i] = row < (r < TM ? M : N);
            src[i] = (r < TM ? x : w) + (in[i] ? (size_t)row * K : 0) + lk;
        }
    }
    auto fetch = [&](int tile) {
        if (tile < count) {
            const uint32_t dst = base + (uint32_t)((tile % STAGES) * (TM + TN) * LD * 4);
            const int k = tile * TK;
            if constexpr (kPieces) {
#pragma unroll
                for (int i = 0; i < kCopies; ++i) {
                    const bool there = in[i] && k + lk < K;
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + (uint32_t)(i * 16 * LD * 4)),
                                 "l"(there ? src[i] + k : src[i] - lk), "r"(there ? 16 : 0) : "memory");
                }
            } else {
                const bool k_in = k + lk < K;
                const float *xr = x + (size_t)(m0 + lr) * K + k + lk, *wr = w + (size_t)(n0 + lr) * K + k + lk;
#pragma unroll
                for (int i = 0; i < TM / 4; ++i, xr += (size_t)4 * K) {
                    const bool there = k_in && m0 + lr + 4 * i < M;
                    cp_async4_or_zero(dst + (uint32_t)(i * 4 * LD * 4), there ? xr : x, there);
                }
#pragma unroll
                for (int i = 0; i < TN / 4; ++i, wr += (size_t)4 * K) {
                    const bool there = k_in && n0 + lr + 4 * i < N;
                    cp_async4_or_zero(dst + (uint32_t)((TM + i * 4) * LD * 4), there ? wr : w, there);
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    float acc[RM][RN];
#pragma unroll
    for (int i = 0; i < RM; ++i)
#pragma unroll
        for (int j = 0; j < RN; ++j) acc[i][j] = 0.0f;
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    // rows ty + 4 i of this warp's 32, columns tx + 8 j of its 8 RN
    const int row0 = (warp >> 1) * 32 + ty, col0 = (warp & 1) * 8 * RN + tx;
    for (int t = 0; t < count; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                          // the tile has landed for every thread; the one before it is no longer read
        fetch(t + STAGES - 1);
        const float* xs = narrow_tiles + (t % STAGES) * (TM + TN) * LD + row0 * LD;
        const float* ws = narrow_tiles + (t % STAGES) * (TM + TN) * LD + (TM + col0) * LD;
#pragma unroll
        for (int k = 0; k < TK; k += 4) {
            float4 a[RM], b[RN];
#pragma unroll
            for (int i = 0; i < RM; ++i) a[i] = *reinterpret_cast<const float4*>(xs + i * 4 * LD + k);
#pragma unroll
            for (int j = 0; j < RN; ++j) b[j] = *reinterpret_cast<const float4*>(ws + j * 8 * LD + k);
#pragma unroll
            for (int j = 0; j < RN; ++j)
#pragma unroll
                for (int i = 0; i < RM; ++i) acc[i][j] = fmaf(a[i].x, b[j].x, acc[i][j]);
#pragma unroll
            for (int j = 0; j < RN; ++j)
#pragma unroll
                for (int i = 0; i < RM; ++i) acc[i][j] = fmaf(a[i].y, b[j].y, acc[i][j]);
#pragma unroll
            for (int j = 0; j < RN; ++j)
#pragma unroll
                for (int i = 0; i < RM; ++i) acc[i][j] = fmaf(a[i].z, b[j].z, acc[i][j]);
#pragma unroll
            for (int j = 0; j < RN; ++j)
#pragma unroll
                for (int i = 0; i < RM; ++i) acc[i][j] = fmaf(a[i].w, b[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < RM; ++i) {
        const int gm = m0 + row0 + 4 * i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < RN; ++j) {
            const int gn = n0 + col0 + 8 * j;
            if (gn >= N) continue;
            float* dst = y + (size_t)gm * N + gn;
            *dst = kAccumulate ? *dst + acc[i][j] : acc[i][j];
        }
    }
}

// The same product for float32 operands and few rows (decoding, short ends of prompts): the same chains again.  One output a thread, 8 rows
// x 16 columns a block, so that a matrix of 1,024 rows reaches 64 blocks and every k costs a thread half of a 16-byte read; four tiles of
// 64 k are on their way.  kPieces: K a multiple of four and operands on 16-byte boundaries, copied in 16-byte pieces, else element by
// element.  Few blocks wait for their rounds of copies and the chain (four clocks a k); many are bound by shared memory, three
// wavefronts of reads for every four multiply-adds of a warp (by count 28 us at N 32,768, beside 20 for the bytes of w).  Every eight rows of x
// read w again.
// 8 rows, K 1,024, N 1,024 / 5,632 / 32,768: 7 / 16 / 56 us (the first kernel here: 103 / 104 / 342), 16 rows 7 / 29 / 105, 31 rows
// 11 / 39 / 203.
template <bool kPieces, bool kAccumulate>
__global__ void __launch_bounds__(128)
gemm_simt_few_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y, int M, int N, int K) {
    constexpr int TK = 64, LD = TK + 4, STAGES = 4, TM = 8, TN = 16;
    __shared__ __align__(16) float tiles[STAGES][TM + TN][LD];     // rows of x, then rows of w
    dependents_may_launch();
    wait_for_predecessor();
    const int m0 = blockIdx.y * TM, n0 = blockIdx.x * TN, tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int count = (K + TK - 1) / TK;
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(&tiles[0][0][0]);
    auto fetch = [&](int tile) {
        if (tile < count) {
            constexpr int PER = kPieces ? 4 : 1;
#pragma unroll 4
            for (int i = tid; i < (TM + TN) * (TK / PER); i += 128) {
                const int r = i / (TK / PER), k = (i % (TK / PER)) * PER, gk = tile * TK + k;
                const bool of_x = r < TM;
                const int row = of_x ? m0 + r : n0 + r - TM;
                const bool there = gk < K && row < (of_x ? M : N);
                const float* src = there ? (of_x ? x : w) + (size_t)row * K + gk : w;
                const uint32_t dst = base + (uint32_t)((((tile % STAGES) * (TM + TN) + r) * LD + k) * 4);
                if constexpr (kPieces)
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
                else
                    cp_async4_or_zero(dst, src, there);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int s = 0; s < STAGES - 1; ++s) fetch(s);
    float acc = 0.0f;
    for (int t = 0; t < count; ++t) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();
        fetch(t + STAGES - 1);
        const float* xr = tiles[t % STAGES][ty];
        const float* wr = tiles[t % STAGES][TM + tx];
#pragma unroll
        for (int k = 0; k < TK; k += 4) {
            const float4 a = *reinterpret_cast<const float4*>(xr + k), b = *reinterpret_cast<const float4*>(wr + k);
            acc = fmaf(a.x, b.x, acc); acc = fmaf(a.y, b.y, acc);
            acc = fmaf(a.z, b.z, acc); acc = fmaf(a.w, b.w, acc);
        }
    }
    const int m = m0 + ty, n = n0 + tx;
    if (m < M && n < N) {
        float* dst = y + (size_t)m * N + n;
        *dst = kAccumulate ? *dst + acc : acc;
    }
}

static int launch_few(const float* x, const float* w, float* y, int M, int N, int K, int accumulate, cudaStream_t stream) {
    dim3 grid((N + 15) / 16, (M + 7) / 8);
    const bool pieces = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15u) == 0;
    auto kernel = pieces ? (accumulate ? gemm_simt_few_kernel<true, true> : gemm_simt_few_kernel<true, false>)
                         : (accumulate ? gemm_simt_few_kernel<false, true> : gemm_simt_few_kernel<false, false>);
    launch_kernel(kernel, grid, 128, 0, stream, x, w, y, M, N, K);
    return CITLALI_LAUNCH_CHECK();
}

// From kWideRows rows on.  A tile of 64 rows takes the same time however few of them are there: K 1,024, N 1,024 / 5,632 / 32,768, 33
// to 64 rows 21 / 29 / 112 us, where the kernel above takes 11 / 39 / 203 (31 rows) and 21 / 74 / 398 (64).  So the line lies where
// the two meet for matrices of some 5,000 rows; narrow ones would keep the kernel above to 64 rows, the widest to 16.
// Tiles of 64 x 128 where they give every SM at least two, else narrower ones.
constexpr int kWideRows = 32;

// Columns a thread of the narrow kernel: the RN of 2 to 6 that gives an SM the shortest share.  A share costs a first part and a part a
// tile; measured in pieces at K 1,024 (us; element by element some 15 % more, the order is the same).  An SM with one tile waits for its
// one warp a scheduler, hence the first part: two tiles of 48 columns beat one of 96 where K is short (130 rows, N 4,096, K 64 / 96
// 7.4 / 8.8 -> 4.9 / 6.3 us) and come out even where it is long.
constexpr int kNarrowTile[5] = {15, 21, 27, 32, 39}, kNarrowFirst[5] = {5, 5, 7, 7, 9};
static int narrow_columns(long rows, int N, int sm_count, long* least) {
    int best = 2;
    *least = -1;
    for (int rn = 2; rn <= 6; ++rn) {
        const long tiles = rows * ((N + 16 * rn - 1) / (16 * rn));
        const long share = (tiles + sm_count - 1) / sm_count * kNarrowTile[rn - 2] + kNarrowFirst[rn - 2];
        if (*least < 0 || share < *least) { *least = share; best = rn; }
    }
    return best;
}

// Operands that cannot be copied in pieces: whether the transposed tiles of 64 columns are quicker than the narrow kernel, whose deeper
// tiles are filled up further and take an SM's shared memory, so that short products end before they pay.  `share`: the narrow kernel's.
// Narrow -> transposed at 26 (260 rows, N 1,280), K 33 / 50 5.1 / 5.0 -> 4.5 / 6.7 us; 88, three tiles of 64 columns an SM (1,400 rows,
// N 1,280), K 130 / 333 18.1 / 35.9 -> 16.3 / 34.9; 103, three of 80 (1,000 rows, N 2,048), K 130 / 333 22.7 / 43.8 -> 21.2 / 45.6; 115, four of
// 64 (N 2,304), K 130 / 333 / 667 28 / 58 / 88 -> 21 / 46 / 87.
static bool transposed_tiles_are_quicker(long share, int K) { return K < (share >= 104 ? 640 : share >= 88 ? 160 : 49); }

template <int RN, bool kPieces>
static int launch_narrow(const float* x, const float* w, float* y, int M, int N, int K, int accumulate, cudaStream_t stream) {
    // The blocks begin while the kernel ahead still runs, on whichever SMs have room by then, and stay there: an SM that was idle takes
    // several of them and works as many times as long.  So a block asks for as much shared memory as leaves an SM no room for more than
    // its even share of the blocks (682 rows, N 1,024, one after another: K 1,024 86 -> 43 us, K 2,816 229 -> 111).
    constexpr size_t needed = (size_t)3 * (64 + 16 * RN) * 36 * 4, of_an_sm = 228 * 1024, alone = of_an_sm / 2 + 256;
    dim3 grid((N + 16 * RN - 1) / (16 * RN), (M + 63) / 64);
    const long tiles = (long)grid.x * grid.y, sms = device_sm_count();
    const size_t spread = of_an_sm / (size_t)((tiles + sms - 1) / sms + 1) + 256, smem = spread > needed ? spread : needed;
    auto kernel = accumulate ? gemm_simt_narrow_kernel<RN, kPieces, true> : gemm_simt_narrow_kernel<RN, kPieces, false>;
    if (int code = raise_shared_limit(kernel, alone, alone)) return code;
    launch_kernel(kernel, grid, 128, smem, stream, x, w, y, M, N, K);
    return CITLALI_LAUNCH_CHECK();
}

template <bool kPieces>
static int launch_narrow(int rn, const float* x, const float* w, float* y, int M, int N, int K, int accumulate, cudaStream_t stream) {
    switch (rn) {
        case 2: return launch_narrow<2, kPieces>(x, w, y, M, N, K, accumulate, stream);
        case 3: return launch_narrow<3, kPieces>(x, w, y, M, N, K, accumulate, stream);
        case 4: return launch_narrow<4, kPieces>(x, w, y, M, N, K, accumulate, stream);
        case 5: return launch_narrow<5, kPieces>(x, w, y, M, N, K, accumulate, stream);
        default: return launch_narrow<6, kPieces>(x, w, y, M, N, K, accumulate, stream);
    }
}

template <int TN>
static int launch_wide(const float* x, const float* w, float* y, int M, int N, int K, int accumulate, cudaStream_t stream) {
    dim3 grid((N + TN - 1) / TN, (M + 63) / 64);
    if (accumulate) launch_kernel(gemm_simt_wide_kernel<TN, true>, grid, 128, 0, stream, x, w, y, M, N, K);
    else launch_kernel(gemm_simt_wide_kernel<TN, false>, grid, 128, 0, stream, x, w, y, M, N, K);
    return CITLALI_LAUNCH_CHECK();
}

static int launch_wide(const float* x, const float* w, float* y, int M, int N, int K, int accumulate, cudaStream_t stream) {
    const long rows = (M + 63) / 64, sms = device_sm_count();
    if (rows * ((N + 127) / 128) >= 2 * sms) return launch_wide<128>(x, w, y, M, N, K, accumulate, stream);
    const bool pieces = K % 4 == 0 && (((uintptr_t)x | (uintptr_t)w) & 15u) == 0;
    long share;
    const int rn = narrow_columns(rows, N, (int)sms, &share);
    if (pieces) return launch_narrow<true>(rn, x, w, y, M, N, K, accumulate, stream);
    if (transposed_tiles_are_quicker(share, K)) return launch_wide<64>(x, w, y, M, N, K, accumulate, stream);
    return launch_narrow<false>(rn, x, w, y, M, N, K, accumulate, stream);
}

template <typename TX, typename TW, typename TY>
static int launch(const void* x, const void* w, void* y, int M, int N, int K, int accumulate, cudaStream_t stream) {
    dim3 grid((N + kTileN - 1) / kTileN, (M + kTileM - 1) / kTileM);
    if (grid.y > 65535) {
        set_last_error("gemm_simt: %d rows exceed the grid limit", M);
        return kTooLarge;
    }
    if constexpr (sizeof(TX) == 4 && sizeof(TW) == 4 && sizeof(TY) == 4) {
        return M >= kWideRows ? launch_wide((const float*)x, (const float*)w, (float*)y, M, N, K, accumulate, stream)
                              : launch_few((const float*)x, (const float*)w, (float*)y, M, N, K, accumulate, stream);
    } else if (accumulate) {
        launch_kernel(gemm_simt_kernel<TX, TW, TY, true>, grid, 256, 0, stream, (const TX*)x, (const TW*)w, (TY*)y, M, N, K);
    } else {
        launch_kernel(gemm_simt_kernel<TX, TW, TY, false>, grid, 256, 0, stream, (const TX*)x, (const TW*)w, (TY*)y, M, N, K);
    }
    return CITLALI_LAUNCH_CHECK();
}

}  // namespace citlali

using namespace citlali;

extern "C" int citlali_gemm_simt(const void* x, int x_dtype, const void* w, int w_dtype, void* y, int y_dtype,
                                 int M, int N, int K, int accumulate, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) {
        set_last_error("gemm_simt: inner size %d must be positive", K);
        return kBadShape;
    }
    if (accumulate && y_dtype != kF32) {
        set_last_error("gemm_simt: accumulation needs a float32 output");
        return kBadDType;
    }
    return CITLALI_DISPATCH_FLOAT(x_dtype, TX, [&] {
        return CITLALI_DISPATCH_FLOAT(w_dtype, TW, [&] {
            return CITLALI_DISPATCH_FLOAT(y_dtype, TY, [&] {
                return launch<TX, TW, TY>(x, w, y, M, N, K, accumulate, stream);
            });
        });
    });
}
