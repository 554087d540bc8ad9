// True 32-bit matrix product for the float32 path of the model:
//   C[M,N] = A[M,K] . B[N,K]^T   (both operands row-major with K contiguous)
// the orientation of every projection in the reference (src/model.cpp:932-944).
// FFMA only: no tensor cores, no reduced-precision mode.  K is cut into segments (a rule of K alone, see segments()); in
// each the even and the odd k are summed in k order and the two sums added, and the segments' sums are added in order.
// The order does not depend on M, N or the kernel that runs, so a row's result is the same whatever else is in the
// batch; and even and odd k are what a packed multiply-add (fma.rn.f32x2, two k at once) takes from 16-byte words as
// they lie in memory.  Shorter chains also round less: 4.5e-6 from 64 bits over 36 layers of the 4B sizes, 1.4e-5 with one
// chain over all of K.
//
// Three kernels share that order:
//  * sgemm_rows_kernel, up to 16 token rows: a stream of weights from HBM;
//  * sgemm_tile_kernel, more rows: bound by the FFMA rate (70 TFLOP/s measured with registers alone);
//  * sgemm_ragged_kernel: operands whose rows do not begin on 16-byte boundaries.
// The plain bfloat16 product, for operands that TMA cannot address, has a kernel of its own (one chain, 32-bit sums).
#include "common.cuh"

#include <cooperative_groups.h>

namespace {
constexpr int BM = 64, BN = 64, BK = 16, TM = 4, TN = 4;

template <typename TO>
__global__ __launch_bounds__(256) void gemm_plain_kernel(const __nv_bfloat16* __restrict__ A, const __nv_bfloat16* __restrict__ B,
                                                       TO* __restrict__ C, int M, int N, int K, long long lda,
                                                       long long ldb, long long ldc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lr = tid >> 2, lk = (tid & 3) * 4;  // this thread loads row lr, k-lanes lk..lk+3 of both tiles
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
        const int k = k0 + lk;
        if (m0 + lr < M) {
            const __nv_bfloat16* p = A + (long long)(m0 + lr) * lda + k;
#pragma unroll
            for (int i = 0; i < 4; ++i) if (k + i < K) a[i] = to_f32(p[i]);
        }
        if (n0 + lr < N) {
            const __nv_bfloat16* p = B + (long long)(n0 + lr) * ldb + k;
#pragma unroll
            for (int i = 0; i < 4; ++i) if (k + i < K) b[i] = to_f32(p[i]);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            As[lk + i][lr] = a[i];
            Bs[lk + i][lr] = b[i];
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 av = *reinterpret_cast<const float4*>(&As[kk][ty * TM]);
            const float4 bv = *reinterpret_cast<const float4*>(&Bs[kk][tx * TN]);
            const float ar[4] = {av.x, av.y, av.z, av.w};
            const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(ar[i], br[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            if (n < N) C[(long long)m * ldc + n] = from_f32<TO>(acc[i][j]);
        }
    }
}

// Segments of K, of 256 lanes and more (the last one may be shorter), and how long they are.
constexpr int SEGMENTS = 8, SEG_STEP = 32;
inline int segments(int K) { return K < 1024 ? 1 : K < 2048 ? 2 : K < 4096 ? 4 : SEGMENTS; }
inline int segment(int K) { const int n = segments(K); return n == 1 ? K : ((K + n - 1) / n + SEG_STEP - 1) / SEG_STEP * SEG_STEP; }

// acc += a * b for two k: the even one in the low half, the odd one in the high half
__device__ __forceinline__ void fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}
__device__ __forceinline__ float even_plus_odd(unsigned long long v) {
    return __uint_as_float((unsigned int)v) + __uint_as_float((unsigned int)(v >> 32));
}

// 16 bytes from global to shared memory, asynchronously; of the four numbers the first `there` are read, the others zeros
// (a row may end within the 16 bytes)
__device__ __forceinline__ void copy16(float* to, const float* from, int there) {
    const uint32_t dst = (uint32_t)__cvta_generic_to_shared(to);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(from), "r"(4 * there) : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int LEFT> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(LEFT) : "memory"); }

// ---- rows of any alignment ----
// 64 x 64 tiles, 16 lanes of K at a time through registers into shared memory.  Bound by the latency of its loads, so it wants
// many blocks an SM: the segments before the running one wait in shared memory (in registers they left two blocks an SM,
// where now there are four: 19,456 features of 9,727 lanes, three rows 2,094 -> 1,201 us, 9,728 with 201 rows 3,085 -> 2,445;
// one chain over all of K, five blocks an SM, 1,276 and 2,002).
__global__ __launch_bounds__(256, 4) void sgemm_ragged_kernel(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C,
                                                              int M, int N, int K, long long lda, long long ldb, long long ldc, int seg) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Bs[BK][BN + 4];
    __shared__ float done[TM * TN][256];
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int lr = tid >> 2, lk = (tid & 3) * 4;  // this thread loads row lr, k-lanes lk..lk+3 of both tiles
    float acc[2][TM][TN];       // even and odd k of the running segment
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[0][i][j] = acc[1][i][j] = 0.f;

    for (int s0 = 0; s0 < K; s0 += seg) {       // (segments are multiples of BK lanes long, the last one may be shorter)
        if (s0 > 0) {
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    float& d = done[i * TN + j][tid];
                    const float v = acc[0][i][j] + acc[1][i][j];
                    d = s0 == seg ? v : d + v;
                    acc[0][i][j] = acc[1][i][j] = 0.f;
                }
        }
        const int s1 = min(K, s0 + seg);
        for (int k0 = s0; k0 < s1; k0 += BK) {
            float a[4] = {0.f, 0.f, 0.f, 0.f}, b[4] = {0.f, 0.f, 0.f, 0.f};
            const int k = k0 + lk;
            if (m0 + lr < M) {
                const float* p = A + (long long)(m0 + lr) * lda + k;
#pragma unroll
                for (int i = 0; i < 4; ++i) if (k + i < K) a[i] = p[i];
            }
            if (n0 + lr < N) {
                const float* p = B + (long long)(n0 + lr) * ldb + k;
#pragma unroll
                for (int i = 0; i < 4; ++i) if (k + i < K) b[i] = p[i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                As[lk + i][lr] = a[i];
                Bs[lk + i][lr] = b[i];
            }
            __syncthreads();
#pragma unroll
            for (int kk = 0; kk < BK; ++kk) {
                const float4 av = *reinterpret_cast<const float4*>(&As[kk][ty * TM]);
                const float4 bv = *reinterpret_cast<const float4*>(&Bs[kk][tx * TN]);
                const float ar[4] = {av.x, av.y, av.z, av.w};
                const float br[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[kk & 1][i][j] = fmaf(ar[i], br[j], acc[kk & 1][i][j]);
            }
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx * TN + j;
            const float last = acc[0][i][j] + acc[1][i][j];
            if (n < N) C[(long long)m * ldc + n] = K > seg ? done[i * TN + j][tid] + last : last;
        }
    }
}

// ---- up to 16 token rows ----
// Bound by the weights' way from HBM (19,456 x 2,560 of them: 30 us at the copy bandwidth).  A block takes as many features,
// 32 at most, as give every SM the same number of blocks; its warps take a segment of K each, with a ring of STAGES
// tiles of 32 lanes of K of their own: no barrier until the segments' sums meet, and a segment is as long as the chain of
// dependent multiply-adds gets.  A lane is a feature and sums all token rows; tile rows are padded by 16 bytes, so eight lanes
// read eight features without bank conflicts, and all lanes read the same words of the token rows.
// Three rows, from a cold L2, launch included: 6,144 x 2,560 27 us, 19,456 x 2,560 55, 2,560 x 9,728 35, 151,936 x 2,560 266
// (5.8 TB/s); 64 x 64 tiles without copies ahead took 386 on average.
// `early`: nothing that may still run writes B, so its first tiles are fetched before the kernel ahead has ended.
constexpr int RW_FEATURES = 32, RW_BK = 32, RW_PITCH = RW_BK + 4, RW_MAX_M = 16;

template <int MT, int STAGES>
__global__ __launch_bounds__(32 * SEGMENTS, 2) void sgemm_rows_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                                      float* __restrict__ C, int M, int N, int K, long long lda,
                                                                      long long ldb, long long ldc, int features, int seg, int early) {
    extern __shared__ float4 smem4[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int stage_floats = (features + M) * RW_PITCH;
    float* ring = reinterpret_cast<float*>(smem4) + warp * STAGES * stage_floats;
    const int n0 = blockIdx.x * features, n_here = min(features, N - n0);
    const int kb = min(K, warp * seg), ke = min(K, kb + seg);
    const int steps = (ke - kb + RW_BK - 1) / RW_BK;
    // a row's eight chunks of 16 bytes go to eight lanes
    const int c4 = (lane & 7) * 4, r0 = lane >> 3;
    const float* b_row = B + (long long)n0 * ldb;
    auto load_b = [&](int slot, int k) {
        float* st = ring + slot * stage_floats + c4;
        const int there = min(4, max(0, ke - k - c4));
        const float* from = b_row + (there > 0 ? k + c4 : 0);
#pragma unroll
        for (int i = 0; i < RW_FEATURES / 4; ++i) {
            const int r = r0 + 4 * i;
            if (r < n_here) copy16(st + r * RW_PITCH, from + r * ldb, there);
        }
    };
    auto load_a = [&](int slot, int k) {
        float* st = ring + slot * stage_floats + features * RW_PITCH + c4;
        const int there = min(4, max(0, ke - k - c4));
        const float* from = A + (there > 0 ? k + c4 : 0);
#pragma unroll
        for (int i = 0; i < (MT + 3) / 4; ++i) {
            const int r = r0 + 4 * i;
            if (r < M) copy16(st + r * RW_PITCH, from + r * lda, there);
        }
    };
    pdl_trigger();
    if (!early) pdl_wait();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t)
        if (t < steps) load_b(t, kb + t * RW_BK);
    if (early) pdl_wait();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < steps) load_a(t, kb + t * RW_BK);
        copies_commit();
    }
    unsigned long long acc[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) acc[i] = 0ull;
    // (a lane without a feature of its own repeats the last one, a row beyond M the last row: their sums are not stored)
    const int w_at = min(lane, n_here - 1) * RW_PITCH, a_at = features * RW_PITCH;
    int use = 0, fill = STAGES - 1;
    for (int t = 0; t < steps; ++t) {
        copies_wait<STAGES - 2>();
        __syncwarp();           // the warp's copies of this stage are there, and its reads of the stage refilled next are over
        if (t + STAGES - 1 < steps) {
            load_b(fill, kb + (t + STAGES - 1) * RW_BK);
            load_a(fill, kb + (t + STAGES - 1) * RW_BK);
        }
        copies_commit();
        const float* st = ring + use * stage_floats;
#pragma unroll
        for (int k = 0; k < RW_BK; k += 4) {       // (lanes of K beyond the segment hold zeros)
            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(st + w_at + k);
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(st + a_at + min(i, M - 1) * RW_PITCH + k);
                fma2(acc[i], a.x, b.x);
                fma2(acc[i], a.y, b.y);
            }
        }
        use = use + 1 == STAGES ? 0 : use + 1;
        fill = fill + 1 == STAGES ? 0 : fill + 1;
    }
    copies_wait<0>();
    __syncthreads();
    float* sums = reinterpret_cast<float*>(smem4);      // [segment][token row][feature]
    const int nseg = blockDim.x >> 5;
#pragma unroll
    for (int i = 0; i < MT; ++i)
        if (i < M && lane < n_here) sums[(warp * M + i) * features + lane] = even_plus_odd(acc[i]);
    __syncthreads();
    for (int i = threadIdx.x; i < M * features; i += blockDim.x) {
        const int m = i / features, f = i % features;
        if (f >= n_here) continue;
        float v = sums[i];
        for (int s = 1; s < nseg; ++s) v += sums[s * M * features + i];
        C[m * ldc + n0 + f] = v;
    }
}

// ---- more token rows ----
// Bound by the FFMA rate.  A block is a tile of 8 TMR token rows x 64 features and one segment of K; the blocks of a
// tile's segments are a cluster that adds its sums through shared memory in segment order, which also makes small work
// items (201 rows against 2,560 features of 9,728 lanes: 1,280 blocks) that fill the SMs evenly.  A thread keeps TMR x 4
// pairs of sums; per four lanes of K it reads TMR + 4 16-byte words for 8 TMR packed multiply-adds.  Tiles lie as in global
// memory, rows padded by 16 bytes (eight features: eight different groups of four banks), two stages of 32 lanes of K.
// Four blocks an SM, or three (BLOCKS), whose threads then have 168 registers instead of 128.  What bounds it is the multiply-add
// pipe, kept waiting by operands in the same register banks.  Over many rounds of blocks four an SM are the better ones, but in 128
// registers tiles of 56 and 64 rows spill, and where all blocks are resident at once that is not hidden: two to three an SM with single
// multiply-adds take 64 rows against 6,144 x 2,560 from 79.0 to 59.8 us, against 2,560 x 9,728 from 140.8 to 108.8 (four an SM over
// more blocks: 100 rows against 2,560 x 4,096 70.4, three 85.0).  Tiles of 72 rows need them, packed: 201 rows against 19,456 x
// 2,560 565 -> 526.
// 256 rows against 19,456 x 2,560: 565 us, 45 TFLOP/s (stages of 16 lanes 612; 16 TFLOP/s in 64 x 64 tiles without copies ahead); one chain
// without packing, 8 x 8 sums a thread or 16 x 16 threads ran at 36 to 46.
namespace cg = cooperative_groups;
constexpr int TL_BN = 64, TL_BK = 32, TL_PITCH = TL_BK + 4, TL_STAGES = 2, TL_THREADS = 128;

template <int TMR, int BLOCKS>
__global__ __launch_bounds__(TL_THREADS, BLOCKS) void sgemm_tile_kernel(const float* __restrict__ A, const float* __restrict__ B,
                                                                   float* __restrict__ C, int M, int N, int K, long long lda,
                                                                   long long ldb, long long ldc, int seg, int nseg, int m_tiles) {
    constexpr int TL_BM = 8 * TMR, ROWS = TL_BM + TL_BN, STAGE = ROWS * TL_PITCH;
    constexpr int SUM_PITCH = TL_BN + 4;
    static_assert(TL_BM * SUM_PITCH <= TL_STAGES * STAGE, "the sums fit into the ring");
    __shared__ __align__(16) float ring[TL_STAGES * STAGE];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int s = blockIdx.x % nseg, tile = blockIdx.x / nseg;
    // token tiles fastest: the blocks that read the same weights run at the same time
    const int m0 = (tile % m_tiles) * TL_BM, n0 = (tile / m_tiles) * TL_BN;
    const int ty = (warp >> 1) * 4 + (lane >> 3), tx = (warp & 1) * 8 + (lane & 7);
    const int kb = min(K, s * seg), ke = min(K, kb + seg);
    const int steps = (ke - kb + TL_BK - 1) / TL_BK;
    const int c4 = (tid & 7) * 4;
    auto load = [&](int t) {
        float* st = ring + (t % TL_STAGES) * STAGE;
        const int k = kb + t * TL_BK + c4;
#pragma unroll
        for (int r = tid >> 3; r < ROWS; r += TL_THREADS / 8) {
            const int row = r < TL_BM ? m0 + r : n0 + r - TL_BM;
            // (rows that are not there are not read: all blocks would ask L2 for one line, 17 rows against 151,936 x 64 took 71 us, not 32)
            const int there = row < (r < TL_BM ? M : N) ? min(4, max(0, ke - k)) : 0;
            const float* from = r < TL_BM ? A + (long long)(there > 0 ? row : 0) * lda : B + (long long)(there > 0 ? row : 0) * ldb;
            copy16(st + r * TL_PITCH + c4, from + (there > 0 ? k : 0), there);
        }
    };
    pdl_trigger();
    pdl_wait();
#pragma unroll
    for (int t = 0; t < TL_STAGES - 1; ++t) {
        if (t < steps) load(t);
        copies_commit();
    }
    constexpr bool SINGLE = BLOCKS == 3 && TMR <= 8;
    unsigned long long acc[SINGLE ? 1 : TMR][4];       // packed: the even k in the low half, the odd ones in the high half
    float even[SINGLE ? TMR : 1][4], odd[SINGLE ? TMR : 1][4];
#pragma unroll
    for (int i = 0; i < TMR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if constexpr (SINGLE) even[i][j] = odd[i][j] = 0.f;
            else acc[i][j] = 0ull;
        }
    for (int t = 0; t < steps; ++t) {
        copies_wait<TL_STAGES - 2>();
        __syncthreads();
        if (t + TL_STAGES - 1 < steps) load(t + TL_STAGES - 1);
        copies_commit();
        const float* a_s = ring + (t % TL_STAGES) * STAGE + ty * TL_PITCH;
        const float* b_s = ring + (t % TL_STAGES) * STAGE + (TL_BM + tx) * TL_PITCH;
#pragma unroll
        for (int k = 0; k < TL_BK; k += 4) {
            if constexpr (SINGLE) {
                float4 b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const float4*>(b_s + 16 * j * TL_PITCH + k);
#pragma unroll
                for (int i = 0; i < TMR; ++i) {
                    const float4 a = *reinterpret_cast<const float4*>(a_s + 8 * i * TL_PITCH + k);
#pragma unroll
                    for (int j = 0; j < 4; ++j) { even[i][j] = fmaf(a.x, b[j].x, even[i][j]); odd[i][j] = fmaf(a.y, b[j].y, odd[i][j]); }
#pragma unroll
                    for (int j = 0; j < 4; ++j) { even[i][j] = fmaf(a.z, b[j].z, even[i][j]); odd[i][j] = fmaf(a.w, b[j].w, odd[i][j]); }
                }
            } else {
                ulonglong2 b[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) b[j] = *reinterpret_cast<const ulonglong2*>(b_s + 16 * j * TL_PITCH + k);
#pragma unroll
                for (int i = 0; i < TMR; ++i) {
                    const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(a_s + 8 * i * TL_PITCH + k);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(acc[i][j], a.x, b[j].x);
#pragma unroll
                    for (int j = 0; j < 4; ++j) fma2(acc[i][j], a.y, b[j].y);
                }
            }
        }
    }
    copies_wait<0>();
    __syncthreads();
#pragma unroll
    for (int i = 0; i < TMR; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            float v;
            if constexpr (SINGLE) v = even[i][j] + odd[i][j];
            else v = even_plus_odd(acc[i][j]);
            ring[(ty + 8 * i) * SUM_PITCH + tx + 16 * j] = v;
        }
    if (nseg == 1) {
        __syncthreads();
    } else {
        cg::this_cluster().sync();
    }
    // each block of the cluster adds and stores every nseg-th row of the tile
    for (int i = tid; i < (TL_BM / nseg) * TL_BN; i += TL_THREADS) {
        const int r = (i / TL_BN) * nseg + s, c = i % TL_BN;
        float v;
        if (nseg == 1) {
            v = ring[r * SUM_PITCH + c];
        } else {
            float part[SEGMENTS];
#pragma unroll
            for (int q = 0; q < SEGMENTS; ++q)
                if (q < nseg) part[q] = cg::this_cluster().map_shared_rank(ring, q)[r * SUM_PITCH + c];
            v = part[0];
#pragma unroll
            for (int q = 1; q < SEGMENTS; ++q)
                if (q < nseg) v += part[q];
        }
        if (m0 + r < M && n0 + c < N) C[(long long)(m0 + r) * ldc + n0 + c] = v;
    }
    if (nseg > 1) cg::this_cluster().sync();       // nobody leaves while its sums may still be read
}

int num_sms() {
    static int n = 0;
    if (n == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0) n = 148;
    }
    return n;
}

template <int MT, int STAGES>
cudaError_t launch_rows(const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                        int features, size_t smem, int early, cudaStream_t stream) {
    cudaError_t e = cudaFuncSetAttribute(sgemm_rows_kernel<MT, STAGES>, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024);
    if (e != cudaSuccess) return e;
    return launch_pdl(sgemm_rows_kernel<MT, STAGES>, dim3((N + features - 1) / features), dim3(32 * segments(K)), smem, stream, A, B, C, M, N, K,
                      lda, ldb, ldc, features, segment(K), early);
}

template <int MT>
cudaError_t choose_rows(const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                        int early, cudaStream_t stream) {
    // features a block: in as few rounds of a block per SM as 32 features allow, the same for every SM
    const int sms = num_sms(), rounds = (N + sms * RW_FEATURES - 1) / (sms * RW_FEATURES);
    int features = (N + sms * rounds - 1) / (sms * rounds);
    if (features < 8) features = 8;
    // stages: a block alone on its SM takes up to six, blocks that share it (more than one round) what fits twice
    const size_t stage = (size_t)segments(K) * (features + M) * RW_PITCH * sizeof(float);
    const size_t room = rounds == 1 ? 220 * 1024 : 112 * 1024;
    if (6 * stage <= room) return launch_rows<MT, 6>(A, B, C, M, N, K, lda, ldb, ldc, features, 6 * stage, early, stream);
    if (4 * stage <= room) return launch_rows<MT, 4>(A, B, C, M, N, K, lda, ldb, ldc, features, 4 * stage, early, stream);
    return launch_rows<MT, 3>(A, B, C, M, N, K, lda, ldb, ldc, features, 3 * stage, early, stream);
}

template <int TMR, int BLOCKS>
cudaError_t launch_tile(const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb, long long ldc,
                        cudaStream_t stream) {
    const int m_tiles = (M + 8 * TMR - 1) / (8 * TMR), nseg = segments(K);
    const long long blocks = (long long)m_tiles * ((N + TL_BN - 1) / TL_BN) * nseg;
    if (blocks > 0x7fffffffll) return cudaErrorInvalidValue;
    return launch_pdl_clusters(sgemm_tile_kernel<TMR, BLOCKS>, dim3((unsigned)blocks), dim3(TL_THREADS), 0, stream, (unsigned)nseg, A, B, C, M, N, K,
                               lda, ldb, ldc, segment(K), nseg, m_tiles);
}
}  // namespace

// b_ready: no kernel that may still be running writes B (a weight matrix): its first tiles may be fetched early.
VCB_API int vcb_sgemm_tn(const float* A, const float* B, float* C, int M, int N, int K, long long lda, long long ldb,
                         long long ldc, int b_ready, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    VCB_CHECK_ARG(M > 0 && N > 0 && K > 0, "sgemm_tn: bad sizes M=%d N=%d K=%d", M, N, K);
    VCB_CHECK_ARG(lda >= K && ldb >= K && ldc >= N, "sgemm_tn: a leading dimension is smaller than its row");
    VCB_CHECK_ARG((M + BM - 1) / BM <= 65535, "sgemm_tn: M=%d exceeds %d rows per launch", M, 65535 * BM);
    const bool aligned = lda % 4 == 0 && ldb % 4 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)B % 16 == 0;
    cudaError_t e = cudaSuccess;
    if (!aligned) {
        sgemm_ragged_kernel<<<dim3((N + BN - 1) / BN, (M + BM - 1) / BM), 256, 0, stream>>>(A, B, C, M, N, K, lda, ldb, ldc, segment(K));
    } else if (M <= (K <= 256 ? 8 : RW_MAX_M)) {
        // (16 rows against 151,936 features: K = 32 44 us against 23 in tiles, 128 70 and 45, 256 96 and 78, 512 146 and 140, 2,048 436 and 532)
        auto rows = M == 1 ? choose_rows<1> : M == 2 ? choose_rows<2> : M <= 4 ? choose_rows<4> : M <= 8 ? choose_rows<8> : choose_rows<16>;
        e = rows(A, B, C, M, N, K, lda, ldb, ldc, b_ready, stream);
    } else {
        // token rows a thread: what pads the rows least, the larger where two pad alike
        int best = 8, padded = (M + 63) / 64 * 64;
        for (int t = 7; t >= 4; --t) {
            const int p = (M + 8 * t - 1) / (8 * t) * (8 * t);
            if (p < padded) { best = t; padded = p; }
        }
        // blocks of a tile of 64 features, all segments; see above for three blocks an SM and tiles of 72 rows.  Against four blocks an SM and no
        // tiles of 72 rows, over 560 products (18 matrices of 256 to 12,288 lanes, 17 to 2,048 rows, weights from HBM) this rule is 2 % faster on
        // average and nowhere more than 1.3 % slower.  Three wherever they hold all blocks lost up to 22 % with less than two an SM (100 rows against
        // 3,072 x 1,024 34 -> 42 us: alone on its way a block waits for its own multiply-adds, and packed ones are half as many; clusters of
        // two segments lose up to there, the others up to one an SM), tiles of 72 rows up to 9 % where others pad as little (400 rows against
        // 2,560 x 9,728 517 -> 565).
        const int nseg = segments(K), high = (M + 71) / 72;
        const long long columns = (long long)((N + TL_BN - 1) / TL_BN) * nseg, sms = num_sms(), blocks = padded / (8 * best) * columns;
        if (high * columns > 12 * sms && (72ll * high * 100 <= 97ll * padded || (72ll * high <= padded && nseg <= 4))) best = 9;
        const bool resident = blocks <= 3 * sms && (2 * blocks <= sms || blocks > (nseg == 2 ? 2 : 1) * sms);
        auto tile = best == 9 ? launch_tile<9, 3> : best == 8 ? (resident ? launch_tile<8, 3> : launch_tile<8, 4>)
                    : best == 7 ? (resident ? launch_tile<7, 3> : launch_tile<7, 4>)
                    : best == 6 ? launch_tile<6, 4> : best == 5 ? launch_tile<5, 4> : launch_tile<4, 4>;
        e = tile(A, B, C, M, N, K, lda, ldb, ldc, stream);
    }
    VCB_CHECK_ARG(e == cudaSuccess, "sgemm_tn: M=%d N=%d K=%d: %s", M, N, K, cudaGetErrorString(e));
    VCB_CHECK_LAUNCH("sgemm_tn");
    return 0;
}

// The same loop for bfloat16 operands whose rows are not 16-byte multiples (which the TMA kernel cannot
// address): bfloat16 in, 32-bit accumulation in k order, bfloat16 or 32-bit out.  Slow; exists so that no
// configuration is refused.
VCB_API int vcb_gemm_bf16_plain(const void* A, const void* B, void* C, int out_dtype, int M, int N, int K, long long lda,
                                long long ldb, long long ldc, cudaStream_t stream) {
    if (M == 0 || N == 0) return 0;
    VCB_CHECK_ARG(M > 0 && N > 0 && K > 0, "gemm_bf16_plain: bad sizes M=%d N=%d K=%d", M, N, K);
    const int gy = (M + BM - 1) / BM, gx = (N + BN - 1) / BN;
    VCB_CHECK_ARG(gy <= 65535, "gemm_bf16_plain: M=%d exceeds %d rows per launch", M, 65535 * BM);
    if (out_dtype == VCB_F32)
        gemm_plain_kernel<float><<<dim3(gx, gy), 256, 0, stream>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)B, (float*)C, M, N, K, lda, ldb, ldc);
    else
        gemm_plain_kernel<__nv_bfloat16><<<dim3(gx, gy), 256, 0, stream>>>((const __nv_bfloat16*)A, (const __nv_bfloat16*)B, (__nv_bfloat16*)C, M, N, K, lda, ldb, ldc);
    VCB_CHECK_LAUNCH("gemm_bf16_plain");
    return 0;
}
