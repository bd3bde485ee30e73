// The gated delta rule (see delta_rule.cu for the mechanism) over runs of many tokens, 32 tokens at a time.
//
// The walk of delta_rule.cu takes two tokens a step, and a step is a chain of sums whose latency nothing hides: 0.4 us a token whatever
// the device could do beside it.  A chunk of 32 tokens is a few small matrix products instead.  With S the state before the chunk, G_i = g_1 .. g_i, and r_ij = g_(j+1) .. g_i (products of decays, never
// quotients: a decay of zero is only that),
//   u_i = beta_i (v_i - G_i S^T k_i - sum_(j<i) r_ij (k_i . k_j) u_j),      so   U = T (V - G K S),  T = (I + A)^-1 diag(beta),
//                                                                            A_ij = beta_i r_ij (k_i . k_j) below the diagonal;
//   o_i = G_i S^T q_i + sum_(j<=i) M_ij u_j,                                 M_ij = r_ij (q_i . k_j);
//   S  <- G_32 S + sum_j e_j k_j u_j^T,                                      e_j = r_(32)j.
// Everything is float32 (fused multiply-adds on CUDA cores): the state and the sums keep the precision of the walk, whose numbers these
// are up to the order of the sums.
//
//   delta_chunk_coefficients   one block a (chunk, key head): K K^T and Q K^T, then a warp a head makes T (by forward substitution,
//                              a lane a column) and M.  All chunks at once.
//   delta_chunk_scan           one block a (sequence, head, VS columns of the values): the chunks in order, S in registers and in shared
//                              memory.  [K; Q] S is the bulk: 256 threads, 8 x 4 outputs each over a slice of the 128 k, the slices'
//                              sums added through shared memory; the next chunk's rows arrive meanwhile.  VS is 32, or 16 where that
//                              leaves SMs idle.  Two warps a scheduler and four barriers a chunk: latency, beside 5,000 wavefronts of
//                              shared memory and 3,600 FMA issues a scheduler in a chunk's 9,000 clocks.
// One sequence of 2,048 tokens, 32 heads over 16 key heads, 128 x 128: 316 us for both kernels (31 of them the coefficients); the walk of
// two tokens a step 948.
#include "api.h"
#include "common.cuh"

namespace citlali {

constexpr int kChunk = 32, kHead = 128;                      // tokens a chunk; key size (smaller ones are filled up with zeros)
constexpr int kCoef = 2 * kChunk * kChunk + 2 * kChunk;      // floats a (chunk, head): T | M | G | e
constexpr int kRow = kHead + 4;                              // a key's stride in shared memory: rows side by side in different banks
constexpr int kMatRow = kChunk + 4;                          // a row of T's and M's in shared memory, for the same reason
static_assert(4 * kChunk * (kChunk + 4) <= 2 * kChunk * kRow, "four warps' A lie over the keys and queries");

// The first chunk of a sequence among all chunks' places: sequences of n tokens have at most n / 32 + 1 (rounded down) of them.
__device__ __forceinline__ int first_chunk(int row0, int seq) { return row0 / kChunk + seq; }

__device__ __forceinline__ void cp_async16_or_zero(float* dst, const float* src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}

// prep: see citlali_delta_prepare (one decay a head).  coef [chunk place][H][kCoef].
__global__ void __launch_bounds__(128)
delta_chunk_coefficients_kernel(const float* __restrict__ prep, int prep_stride, const int32_t* __restrict__ seq_start, int H, int KH,
                                int D, int V, float* __restrict__ coef) {
    __shared__ __align__(16) float kq[2 * kChunk][kRow];     // keys, then queries
    __shared__ float kk[kChunk][kChunk + 1], qk[kChunk][kChunk + 1];
    dependents_may_launch();
    wait_for_predecessor();
    const int seq = blockIdx.z, kh = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int row0 = seq_start[seq], r0 = row0 + blockIdx.x * kChunk, n = min(kChunk, seq_start[seq + 1] - r0);
    if (n <= 0) return;
    for (int i = tid; i < 2 * kChunk * (kHead / 4); i += 128) {
        const int r = i / (kHead / 4), c = (i % (kHead / 4)) * 4, token = r & (kChunk - 1);
        const bool there = token < n && c < D;
        const float* src = prep + (size_t)(r0 + token) * prep_stride + ((r < kChunk ? KH : 0) + kh) * D + c;
        cp_async16_or_zero(&kq[r][c], there ? src : prep, there);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();
    {   // 4 x 4 outputs a thread: threads 0-63 K K^T, 64-127 Q K^T; rows and columns eight apart.  An output is a sum of sums of 16
        // products.  Off float64, one chain of 128 / this / the walk's sums, in 1e-7: random keys 2.2 / 1.3 / 1.2, decays near zero
        // 2.1 / 0.9 / 0.9, keys that lean one way 3.3 / 3.2 / 3.1, one key over and over, now and then turned round, 5.9 / 4.6 / 2.6.
        // 32 heads of 128 x 128: 64 rows 22.7 -> 23.7 us in both kernels, 2,048 rows 322 as before.
        const int a0 = (tid >> 6) * kChunk + ((tid >> 3) & 7), b0 = tid & 7;
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = 0.0f;
#pragma unroll 1
        for (int k0 = 0; k0 < D; k0 += 32) {                  // (zeros behind D)
            float part[4][4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) part[i][j][0] = part[i][j][1] = 0.0f;
#pragma unroll
            for (int k = k0; k < k0 + 32; k += 4) {
                float4 a[4], b[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    a[i] = *reinterpret_cast<const float4*>(&kq[a0 + 8 * i][k]);
                    b[i] = *reinterpret_cast<const float4*>(&kq[b0 + 8 * i][k]);
                }
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        part[i][j][0] = fmaf(a[i].y, b[j].y, fmaf(a[i].x, b[j].x, part[i][j][0]));
                        part[i][j][1] = fmaf(a[i].w, b[j].w, fmaf(a[i].z, b[j].z, part[i][j][1]));
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] += part[i][j][0] + part[i][j][1];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) (tid < 64 ? kk : qk)[((tid >> 3) & 7) + 8 * i][b0 + 8 * j] = acc[i][j];
    }
    __syncthreads();
    const int C = 2 * KH * D + H * V, group = H / KH;
    const int place = first_chunk(row0, seq) + blockIdx.x;
    for (int j = warp; j < group; j += 4) {
        const int h = kh * group + j;
        // lane: token `lane` for beta and g, then column `lane` of every matrix
        const float* scalars = prep + (size_t)(r0 + lane) * prep_stride + C;
        const float beta = lane < n ? scalars[h] : 0.0f, g = lane < n ? scalars[H + h] : 1.0f;
        float* dst = coef + ((size_t)place * H + h) * kCoef;
        // (the keys and queries have been read: their place serves for A)
        float(*a)[kChunk + 4] = reinterpret_cast<float(*)[kChunk + 4]>(&kq[0][0]) + warp * kChunk;
        __syncwarp();                                         // the head before has been read
        float r = 1.0f, G = 1.0f, mine = 1.0f;
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
            const float gi = __shfl_sync(0xffffffffu, g, i), bi = __shfl_sync(0xffffffffu, beta, i);
            G *= gi;
            if (i == lane) mine = G;
            if (i > lane) r *= gi;
            dst[kChunk * kChunk + i * kChunk + lane] = i >= lane ? r * qk[i][lane] : 0.0f;
            a[i][lane] = i > lane ? bi * r * kk[i][lane] : 0.0f;
        }
        dst[2 * kChunk * kChunk + lane] = mine;
        dst[2 * kChunk * kChunk + kChunk + lane] = r;
        __syncwarp();
        // column `lane` of (I + A)^-1: row i is e_i minus the rows above it
        float t[kChunk];
#pragma unroll
        for (int i = 0; i < kChunk; ++i) {
            float s0 = 0.0f, s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;
#pragma unroll
            for (int m = 0; m < i; m += 4) {                  // (A is zero on and above the diagonal)
                const float4 w = *reinterpret_cast<const float4*>(&a[i][m]);
                s0 = fmaf(w.x, t[m], s0);
                if (m + 1 < i) s1 = fmaf(w.y, t[m + 1], s1);
                if (m + 2 < i) s2 = fmaf(w.z, t[m + 2], s2);
                if (m + 3 < i) s3 = fmaf(w.w, t[m + 3], s3);
            }
            t[i] = (i == lane ? 1.0f : 0.0f) - ((s0 + s1) + (s2 + s3));
            dst[i * kChunk + lane] = t[i] * beta;
        }
    }
}

template <int VS>
struct ScanShared {
    float kq[2][2 * kChunk][kRow];        // the chunk's keys and queries, and the next one's
    float coef[2][2 * kChunk * kMatRow + 2 * kChunk];           // T | M, rows kMatRow apart | G | e
    float v[2][kChunk][VS];
    float s[kHead][VS];
    float part[128 / VS][2 * kChunk][VS]; // [K; Q] S over a slice of k
    float r[kChunk][VS], u[kChunk][VS], eu[kChunk][VS];
};

// N (two or four) floats from their natural boundary.
template <int N>
struct Floats { float f[N]; };
template <int N>
__device__ __forceinline__ Floats<N> load_floats(const float* p) {
    Floats<N> r;
    if constexpr (N == 4) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        r.f[0] = v.x; r.f[1] = v.y; r.f[2] = v.z; r.f[3] = v.w;
    } else {
        const float2 v = *reinterpret_cast<const float2*>(p);
        r.f[0] = v.x; r.f[1] = v.y;
    }
    return r;
}
template <int N>
__device__ __forceinline__ void store_floats(float* p, const float (&f)[N]) {
    if constexpr (N == 4) *reinterpret_cast<float4*>(p) = make_float4(f[0], f[1], f[2], f[3]);
    else *reinterpret_cast<float2*>(p) = make_float2(f[0], f[1]);
}

// sum += W[row, 0 .. row] X[0 .. row, col ..], rows in order.  What W holds above its diagonal (zeros, or not a number where a later
// token is none) and X's later rows must not meet: a token reaches no earlier one, infinite or not.  A warp has four rows, so only its
// last four of W's columns need to ask.
template <int N, int VS>
__device__ __forceinline__ void add_rows_up_to(float (&sum)[N], const float* W, const float (&X)[kChunk][VS], int row, int col) {
    auto tile = [&](int j, bool ask) {
        const Floats<4> w = load_floats<4>(W + row * kMatRow + j);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const Floats<N> x = load_floats<N>(&X[j + e][col]);
            if (!ask || j + e <= row) {
#pragma unroll
                for (int c = 0; c < N; ++c) sum[c] = fmaf(w.f[e], x.f[c], sum[c]);
            }
        }
    };
    const int own = row & ~3;
    for (int j = 0; j < own; j += 4) tile(j, false);
    tile(own, true);
}

template <int VS>
__global__ void __launch_bounds__(256)
delta_chunk_scan_kernel(const float* __restrict__ prep, int prep_stride, const float* __restrict__ coef, float* __restrict__ state,
                        size_t state_stride, const int32_t* __restrict__ seq_start, const int32_t* __restrict__ seq_slot, int H, int KH,
                        int D, int V, float* __restrict__ out) {
    constexpr int CG = VS / 4, SLICES = 128 / VS, KS = kHead / SLICES, RS = VS / 8;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    ScanShared<VS>& sm = *reinterpret_cast<ScanShared<VS>*>(smem_raw);
    dependents_may_launch();
    wait_for_predecessor();
    const int tid = threadIdx.x, h = blockIdx.y, v0 = blockIdx.x * VS;
    // the longest sequences' blocks first: where there are more blocks than SMs, the last ones to begin are then the shortest (five
    // sequences of 155 to 540 tokens, 16 heads: a step of three such layers 1.70 -> 1.63 ms)
    int seq = blockIdx.z;
    const int sequences = gridDim.z;
    if (sequences > 1 && sequences <= 256) {
        __shared__ int chosen;
        if (tid < sequences) {
            const int n = seq_start[tid + 1] - seq_start[tid];
            int rank = 0;
            for (int s = 0; s < sequences; ++s) {
                const int m = seq_start[s + 1] - seq_start[s];
                rank += m > n || (m == n && s < tid);
            }
            if (rank == (int)blockIdx.z) chosen = tid;
        }
        __syncthreads();
        seq = chosen;
    }
    const int row0 = seq_start[seq], tokens = seq_start[seq + 1] - row0;
    if (tokens <= 0) return;
    const int kh = h / (H / KH);
    const int chunks = (tokens + kChunk - 1) / kChunk;
    const float* coef_h = coef + ((size_t)first_chunk(row0, seq) * H + h) * kCoef;
    auto fetch = [&](int ch) {
        if (ch < chunks) {
            const int buf = ch & 1, r0 = row0 + ch * kChunk, n = min(kChunk, tokens - ch * kChunk);
            for (int i = tid; i < 2 * kChunk * (kHead / 4); i += 256) {
                const int r = i / (kHead / 4), c = (i % (kHead / 4)) * 4, token = r & (kChunk - 1);
                const bool there = token < n && c < D;
                const float* src = prep + (size_t)(r0 + token) * prep_stride + ((r < kChunk ? KH : 0) + kh) * D + c;
                cp_async16_or_zero(&sm.kq[buf][r][c], there ? src : prep, there);
            }
            for (int i = tid; i < kChunk * CG; i += 256) {
                const int token = i / CG, c = (i % CG) * 4;
                const bool there = token < n && v0 + c < V;
                cp_async16_or_zero(&sm.v[buf][token][c], there ? prep + (size_t)(r0 + token) * prep_stride + 2 * KH * D + h * V + v0 + c : prep, there);
            }
            for (int i = tid; i < kCoef / 4; i += 256) {
                const int row = i / (kChunk / 4), at = row < 2 * kChunk ? row * kMatRow + (i % (kChunk / 4)) * 4 : i * 4 + 2 * kChunk * (kMatRow - kChunk);
                cp_async16_or_zero(&sm.coef[buf][at], coef_h + (size_t)ch * H * kCoef + i * 4, true);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    fetch(0);
    // Where a warp's lanes stand in a product.  Of a 16-byte read of shared memory two neighbours (or two lanes two apart) that read the
    // same place are served together, lanes further apart are not: columns in the lane's low bits and rows above them cost the columns'
    // operand four wavefronts a read, columns in every other bit and rows in those between cost either operand two.  (By the counters
    // 5,000 wavefronts a chunk instead of 6,000, 800 of them bank conflicts instead of 200; with the coefficients, columns in the low bits -> every other bit: one sequence of
    // 2,048 tokens, 32 heads 323 -> 316 us, 8 heads (16 columns a block) 232 -> 214, five of 155 to 540 tokens, 16 heads 149 -> 145.)
    const int lane = tid & 31, warp = tid >> 5;
    const int even = (lane & 1) | ((lane >> 1) & 2) | ((lane >> 2) & 4), odd = ((lane >> 1) & 1) | ((lane >> 2) & 2);    // bits 0 2 4; 1 3
    const int lane_c = CG == 8 ? even : even & 3, lane_r = CG == 8 ? odd : odd | ((lane >> 2) & 4);
    constexpr int LR = 32 / CG;                // rows a warp has beside its CG columns
    // this thread's part of S: rows sk .. sk + RS - 1, columns 4 sc .. 4 sc + 3
    const int sc = lane_c, sk = (warp * LR + lane_r) * RS;
    float* S_g = state + (size_t)seq_slot[seq] * state_stride + (size_t)h * D * V + v0 + sc * 4;
    float S[RS][4];
#pragma unroll
    for (int i = 0; i < RS; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            S[i][e] = sk + i < D && v0 + sc * 4 + e < V ? S_g[(size_t)(sk + i) * V + e] : 0.0f;
            sm.s[sk + i][sc * 4 + e] = S[i][e];
        }
    // [K; Q] S: slice `slice` of k, columns 4 xc .. 4 xc + 3, rows xr + 8 i (i < 4: keys, else queries)
    const int slice = warp * LR / 8, xc = lane_c, xr = (warp * LR + lane_r) & 7;
    // the 32 x VS matrices: row `ur`, UC columns from `uc` (a warp four rows)
    constexpr int UC = VS / 8;
    const int ur = warp * 4 + odd, uc = even * UC;
    for (int ch = 0; ch < chunks; ++ch) {
        const int buf = ch & 1;
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                       // the chunk has landed, S is written, the other buffers are no longer read
        fetch(ch + 1);
        {
            float acc[8][4];
#pragma unroll
            for (int i = 0; i < 8; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;
#pragma unroll 2
            for (int k = slice * KS; k < slice * KS + KS; k += 4) {
                float4 s4[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) s4[e] = *reinterpret_cast<const float4*>(&sm.s[k + e][xc * 4]);
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(&sm.kq[buf][xr + 8 * i][k]);
                    acc[i][0] = fmaf(a.w, s4[3].x, fmaf(a.z, s4[2].x, fmaf(a.y, s4[1].x, fmaf(a.x, s4[0].x, acc[i][0]))));
                    acc[i][1] = fmaf(a.w, s4[3].y, fmaf(a.z, s4[2].y, fmaf(a.y, s4[1].y, fmaf(a.x, s4[0].y, acc[i][1]))));
                    acc[i][2] = fmaf(a.w, s4[3].z, fmaf(a.z, s4[2].z, fmaf(a.y, s4[1].z, fmaf(a.x, s4[0].z, acc[i][2]))));
                    acc[i][3] = fmaf(a.w, s4[3].w, fmaf(a.z, s4[2].w, fmaf(a.y, s4[1].w, fmaf(a.x, s4[0].w, acc[i][3]))));
                }
            }
#pragma unroll
            for (int i = 0; i < 8; ++i)
                *reinterpret_cast<float4*>(&sm.part[slice][xr + 8 * i][xc * 4]) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        const float* T = sm.coef[buf];
        const float* M = T + kChunk * kMatRow;
        const float* G = M + kChunk * kMatRow;
        const float* E = G + kChunk;
        float y[UC], r[UC], u[UC], eu[UC];
#pragma unroll
        for (int c = 0; c < UC; ++c) r[c] = y[c] = u[c] = 0.0f;
#pragma unroll
        for (int s = 0; s < SLICES; ++s) {
            const Floats<UC> a = load_floats<UC>(&sm.part[s][ur][uc]), b = load_floats<UC>(&sm.part[s][kChunk + ur][uc]);
#pragma unroll
            for (int c = 0; c < UC; ++c) { r[c] += a.f[c]; y[c] += b.f[c]; }
        }
        const float Gi = G[ur], Ei = E[ur];
        const Floats<UC> v = load_floats<UC>(&sm.v[buf][ur][uc]);
#pragma unroll
        for (int c = 0; c < UC; ++c) { r[c] = fmaf(-Gi, r[c], v.f[c]); y[c] *= Gi; }
        store_floats<UC>(&sm.r[ur][uc], r);
        __syncthreads();
        add_rows_up_to<UC>(u, T, sm.r, ur, uc);
#pragma unroll
        for (int c = 0; c < UC; ++c) eu[c] = Ei * u[c];
        store_floats<UC>(&sm.u[ur][uc], u);
        store_floats<UC>(&sm.eu[ur][uc], eu);
        __syncthreads();
        add_rows_up_to<UC>(y, M, sm.u, ur, uc);
        const int token = ch * kChunk + ur;
        if (token < tokens && v0 + uc < V) store_floats<UC>(out + (size_t)(row0 + token) * H * V + h * V + v0 + uc, y);
        const float G_all = G[kChunk - 1];
#pragma unroll
        for (int i = 0; i < RS; ++i)
#pragma unroll
            for (int e = 0; e < 4; ++e) S[i][e] *= G_all;
#pragma unroll 8
        for (int j = 0; j < kChunk; ++j) {
            const float4 w = *reinterpret_cast<const float4*>(&sm.eu[j][sc * 4]);
            float k[RS];
            if constexpr (RS == 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(&sm.kq[buf][j][sk]);
                k[0] = k4.x; k[1] = k4.y; k[2] = k4.z; k[3] = k4.w;
            } else {
                const float2 k2 = *reinterpret_cast<const float2*>(&sm.kq[buf][j][sk]);
                k[0] = k2.x; k[1] = k2.y;
            }
#pragma unroll
            for (int i = 0; i < RS; ++i) {
                S[i][0] = fmaf(k[i], w.x, S[i][0]); S[i][1] = fmaf(k[i], w.y, S[i][1]);
                S[i][2] = fmaf(k[i], w.z, S[i][2]); S[i][3] = fmaf(k[i], w.w, S[i][3]);
            }
        }
#pragma unroll
        for (int i = 0; i < RS; ++i) *reinterpret_cast<float4*>(&sm.s[sk + i][sc * 4]) = make_float4(S[i][0], S[i][1], S[i][2], S[i][3]);
    }
#pragma unroll
    for (int i = 0; i < RS; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (sk + i < D && v0 + sc * 4 + e < V) S_g[(size_t)(sk + i) * V + e] = S[i][e];
}

}  // namespace citlali

using namespace citlali;

extern "C" size_t citlali_delta_chunks_scratch_floats(int rows, int sequences, int H) {
    return (size_t)(rows / kChunk + sequences + 1) * H * kCoef;
}

template <int VS>
static int launch_scan(const float* prep, int prep_stride, const float* coef, float* state, size_t state_stride, const int32_t* seq_start,
                       const int32_t* seq_slot, int sequences, int H, int KH, int D, int V, float* out, cudaStream_t stream) {
    static bool configured = false;
    auto kernel = delta_chunk_scan_kernel<VS>;
    if (!configured) {
        cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(ScanShared<VS>));
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    dim3 grid((V + VS - 1) / VS, H, sequences);
    launch_kernel(kernel, grid, 256, sizeof(ScanShared<VS>), stream, prep, prep_stride, coef, state, state_stride, seq_start, seq_slot, H,
                  KH, D, V, out);
    return CITLALI_LAUNCH_CHECK();
}

extern "C" int citlali_delta_chunks(const float* prep, int prep_stride, float* state, size_t state_stride, const int32_t* seq_start,
                                    const int32_t* seq_slot, int sequences, int max_new, int H, int KH, int D, int V, float* out,
                                    float* scratch, size_t scratch_floats, int rows, cudaStream_t stream) {
    if (sequences <= 0 || rows <= 0 || max_new <= 0) return 0;
    if (H <= 0 || KH <= 0 || H % KH != 0 || D <= 0 || D > kHead || D % 4 != 0 || V <= 0 || V % 4 != 0 || prep_stride % 4 != 0 ||
        H > 65535 || sequences > 65535) {
        set_last_error("delta_chunks: %d heads over %d key heads of %d, values of %d, rows of %d (sizes in fours, keys of at most 128)", H, KH, D, V, prep_stride);
        return kBadShape;
    }
    if (((uintptr_t)prep | (uintptr_t)out | (uintptr_t)scratch) & 15u) {
        set_last_error("delta_chunks: buffers must be 16-byte aligned");
        return kBadAlignment;
    }
    if (scratch_floats < citlali_delta_chunks_scratch_floats(rows, sequences, H)) {
        set_last_error("delta_chunks: %zu floats of scratch are needed, %zu were given", citlali_delta_chunks_scratch_floats(rows, sequences, H), scratch_floats);
        return kBadShape;
    }
    dim3 grid((max_new + kChunk - 1) / kChunk, KH, sequences);
    launch_kernel(delta_chunk_coefficients_kernel, grid, 128, 0, stream, prep, prep_stride, seq_start, H, KH, D, V, scratch);
    int code = CITLALI_LAUNCH_CHECK();
    if (code != 0) return code;
    // 32 columns a block where that gives the SMs a block each, else 16
    const bool broad = (long)sequences * H * ((V + 31) / 32) >= device_sm_count() * 3 / 4;
    return broad ? launch_scan<32>(prep, prep_stride, scratch, state, state_stride, seq_start, seq_slot, sequences, H, KH, D, V, out, stream)
                 : launch_scan<16>(prep, prep_stride, scratch, state, state_stride, seq_start, seq_slot, sequences, H, KH, D, V, out, stream);
}
