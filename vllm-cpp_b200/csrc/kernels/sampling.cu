// Next-token choice from rows of 32-bit logits, one block or one cluster of blocks per row.
//
// Order of operations as the reference's sample_token (src/model.cpp:1291-1352):
// repetition penalty once per earlier occurrence of a token (positive scores are
// divided, negative multiplied), division by the temperature, softmax, nucleus cut
// at top_p, draw.  temperature <= 0 takes the arg-max, lowest index on ties
// (src/mlx_backend.cpp:516-524).  The draw is argmax_i(score_i + Gumbel(u_i)) over
// the kept tokens, u_i a counter-based uniform of (seed, step, i): one pass, no
// sort, and the same token on any machine for equal logits.  The nucleus is the
// set {p_i >= c} for the largest c whose set has mass >= top_p (the shortest
// descending prefix, with ties at the cut all kept), found by narrowing a range of
// the scores' ordered bit patterns; masses are summed in 64-bit.
#include "common.cuh"

#include <cooperative_groups.h>

#include <math_constants.h>

namespace {

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
    z += 0x9E3779B97F4A7C15ull;
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

__device__ __forceinline__ float uniform01(unsigned long long key, unsigned int index) {
    const unsigned long long bits = mix64(key ^ (unsigned long long)index);
    return ((float)(bits >> 41) + 0.5f) * (1.0f / 8388608.0f);
}

// uniform01 lies in [2^-24, 1 - 2^-24], so -log(-log(u)) is no more than this: a score that cannot reach the best draw so
// far even with it needs no logarithms (rounding keeps the order, so the token is the same)
constexpr float GUMBEL_MAX = 16.75f;

// Whether score s with uniform u may draw as much as `best`, which takes a hash and an exponential where the draw itself takes two
// logarithms more: -log(u) >= 1 - u, so the draw is at most s - log(1 - u).  What is let through in vain costs time only; the
// margins (a hundredth of the exponential, 1e-3 and five units of 2^-23 of `best`) are far above what rounding adds to either side.
// Infinities and NaN are let through.
__device__ __forceinline__ bool may_draw(float s, float u, float best) {
    const float d = best - s - fmaf(fabsf(best), 6e-7f, 1e-3f);
    return !(1.f - u > 1.01f * __expf(-d));
}

// order-preserving map float -> uint32
__device__ __forceinline__ unsigned int ordered_key(float f) {
    const unsigned int u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}

// the score of a key; no score is less than minus infinity (keys of NaN below it)
__device__ __forceinline__ float score_of(unsigned int key) {
    const float f = __uint_as_float((key & 0x80000000u) ? (key & 0x7fffffffu) : ~key);
    return f == f ? f : -CUDART_INF_F;
}

__device__ __forceinline__ double block_sum_f64(double v, double* scratch /* 33 */) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if (lane == 0) scratch[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double t = lane < nwarps ? scratch[lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
        if (lane == 0) scratch[32] = t;
    }
    __syncthreads();
    return scratch[32];
}

// arg-max with lowest index on ties; every thread gets the result
__device__ __forceinline__ void block_argmax(float& v, int& idx, float* sv, int* si) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
    __syncthreads();
    if (lane == 0) { sv[warp] = v; si[warp] = idx; }
    __syncthreads();
    if (warp == 0) {
        float tv = lane < nwarps ? sv[lane] : -CUDART_INF_F;
        int ti = lane < nwarps ? si[lane] : 0x7fffffff;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, tv, o);
            const int oi = __shfl_xor_sync(0xffffffffu, ti, o);
            if (ov > tv || (ov == tv && oi < ti)) { tv = ov; ti = oi; }
        }
        if (lane == 0) { sv[32] = tv; si[32] = ti; }
    }
    __syncthreads();
    v = sv[32];
    idx = si[32];
}

struct RowParams {  // one per row, 32 bytes
    float temperature, top_p, repeat_penalty;
    int slot;              // row of the occurrence-count table, or -1
    unsigned int seed_lo, seed_hi, step, pad;
};

__device__ __forceinline__ float penalised(float s, int count, float penalty) {
    if (count > 0) {
        const float f = powf(penalty, (float)count);
        s = s > 0.f ? s / f : s * f;
    }
    return s;
}

__device__ __forceinline__ float score_at(const float* logits, const int* counts, float penalty, float inv_t, int i) {
    float s = logits[i];
    if (counts) s = penalised(s, counts[i], penalty);
    return s * inv_t;
}

__global__ __launch_bounds__(1024) void sample_kernel(const float* __restrict__ logits, long long row_stride, int V,
                                                      const RowParams* __restrict__ params,
                                                      const int* __restrict__ counts_table, int* __restrict__ out) {
    __shared__ float sv[33];
    __shared__ int si[33];
    __shared__ double sd[33];
    const int row = blockIdx.x;
    const RowParams p = params[row];
    const float* lg = logits + (size_t)row * row_stride;
    const int* counts = (counts_table && p.slot >= 0 && p.repeat_penalty != 1.0f) ? counts_table + (size_t)p.slot * V : nullptr;
    const bool greedy = !(p.temperature > 0.f);
    const float inv_t = greedy ? 1.f : 1.0f / p.temperature;

    // maximum of the scores (also the greedy answer)
    float best = -CUDART_INF_F;
    int best_i = 0x7fffffff;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float s = score_at(lg, counts, p.repeat_penalty, inv_t, i);
        if (s > best || (s == best && i < best_i)) { best = s; best_i = i; }
    }
    block_argmax(best, best_i, sv, si);
    if (greedy) {
        if (threadIdx.x == 0) out[row] = best_i;
        return;
    }
    const float m = best;

    unsigned int cut = 0;  // keep scores whose ordered key is >= cut
    if (p.top_p < 1.0f) {
        double z = 0.0;
        for (int i = threadIdx.x; i < V; i += blockDim.x) z += (double)expf(score_at(lg, counts, p.repeat_penalty, inv_t, i) - m);
        z = block_sum_f64(z, sd);
        const double need = (double)p.top_p * z;
        unsigned int lo = 0, hi = ordered_key(m);  // mass(lo) >= need holds; answer in [lo, hi]
        while (lo < hi) {
            const unsigned int mid = lo + (hi - lo + 1) / 2;
            double mass = 0.0;
            for (int i = threadIdx.x; i < V; i += blockDim.x) {
                const float s = score_at(lg, counts, p.repeat_penalty, inv_t, i);
                if (ordered_key(s) >= mid) mass += (double)expf(s - m);
            }
            mass = block_sum_f64(mass, sd);
            if (mass >= need) lo = mid; else hi = mid - 1;
        }
        cut = lo;
    }

    const unsigned long long key = mix64(((unsigned long long)p.seed_lo << 32) | (unsigned long long)p.step);
    float zbest = m - logf(-logf(uniform01(key, (unsigned int)best_i)));       // the largest score's draw, which all others have to reach
    int zi = best_i;
    for (int i = threadIdx.x; i < V; i += blockDim.x) {
        const float s = score_at(lg, counts, p.repeat_penalty, inv_t, i);
        if (ordered_key(s) < cut || s + GUMBEL_MAX < zbest) continue;
        const float u = uniform01(key, (unsigned int)i);
        if (!may_draw(s, u, zbest)) continue;
        const float zv = s - logf(-logf(u));
        if (zv > zbest || (zv == zbest && i < zi)) { zbest = zv; zi = i; }
    }
    block_argmax(zbest, zi, sv, si);
    if (threadIdx.x == 0) out[row] = zi;
}

// Rows of large vocabularies with a nucleus cut: a cluster of blocks per row, the row's scores computed once and kept in
// the blocks' shared memory.
//
// What bounds it: the logits and the counts are read once (64 rows of 151,936: 78 MB, 12 us at the copy bandwidth); the
// rest is a chain of hand-overs between the cluster's blocks, two rows to an SM's worth of blocks at a time.  The cut is
// therefore not bisected bit by bit (32 passes, expf and powf again in each: sample_kernel, a block a row) but closed in
// on by NT thresholds a pass: the first pass puts them at distances below the maximum, where the mass of a softmax lies,
// later ones spread them evenly over the remaining range of ordered keys.  Once the range holds at most CAND scores, every
// block takes the cluster's list of them, ranks it, and reads the cut off the running sum -- in a model's logits after the
// first pass.  All sums are taken in a fixed order, so equal logits give equal tokens.
// The passes over a block's scores are bound by instructions (128 a score before, of which every score's ordered key, eight
// predicated sums and a comparison of places were most), so a score that reaches no threshold is left at one comparison of floats.
// 64 rows of 151,936 with penalty, temperature and nucleus: 1,620 us with a block a row, 56 here (71 with keys and sums for every
// score); with a temperature alone 41 (56 with two logarithms for every score near the maximum).
// Scores like noise, most of which reach thresholds, lose where a block has an SM to itself (a few rows, or more than 192,000 scores: one
// row of 151,936 62 -> 64 us, of 262,144 91 -> 98) and gain elsewhere (32 rows of 151,936 123 -> 112); a model's gain in both (one row 20.5 -> 18.7, of
// 262,144 28.0 -> 24.5).  Sums under predicates instead of branches take back half of either.
namespace cg = cooperative_groups;
constexpr size_t CLUSTER_MAX_SMEM = 192 * 1024;      // beside ClusterShared (18 KB)
constexpr int CL_THREADS = 512, CL_WARPS = CL_THREADS / 32, CL_BLOCKS = 8, NT = 7, CAND = 1024;
// distances of the first pass's thresholds below the maximum, ascending thresholds
__device__ constexpr float FIRST_CUTS[NT] = {20.f, 14.f, 10.f, 7.f, 4.5f, 2.5f, 1.f};

struct ClusterShared {
    double warp_mass[CL_WARPS][NT + 1];
    double gathered[CL_BLOCKS * (NT + 1)];
    double mass[2][NT + 1];        // this block's sums, for the cluster; the passes use the two halves in turn
    float best_v[2];
    int best_i[2];
    int n_cand;                    // scores of this block in the range (not all listed if more than CAND)
    unsigned int cand_key[CAND], sorted_key[CAND];
    __align__(16) unsigned int all_key[CAND];
    float sorted_mass[CAND];
    double scan[CL_WARPS];
    int first;
    float sv[33];
    int si[33];
};

// sums of NT + 1 values over the cluster, in a fixed order; every thread gets them
__device__ __forceinline__ void cluster_sums(cg::cluster_group& cluster, ClusterShared& sh, int half, double (&v)[NT + 1]) {
    static_assert(NT + 1 == 8, "the exchange below reduces eight values");
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    // eight values over 32 lanes: lanes swap halves of what they hold as they add; lane l ends with value l & 7
#pragma unroll
    for (int w = 4; w >= 1; w >>= 1) {
        const bool up = lane & w;
#pragma unroll
        for (int j = 0; j < w; ++j) {
            const double give = up ? v[j] : v[j + w], keep = up ? v[j + w] : v[j];
            v[j] = keep + __shfl_xor_sync(0xffffffffu, give, w);
        }
    }
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 8);
    v[0] += __shfl_xor_sync(0xffffffffu, v[0], 16);
    if (lane < NT + 1) sh.warp_mass[warp][lane] = v[0];
    __syncthreads();
    if (threadIdx.x < NT + 1) {
        double t = 0.0;
#pragma unroll
        for (int w = 0; w < CL_WARPS; ++w) t += sh.warp_mass[w][threadIdx.x];
        sh.mass[half][threadIdx.x] = t;
    }
    cluster.sync();
    // each block's sums through one thread a value (64 reads in flight), the rest through shared memory
    if (threadIdx.x < CL_BLOCKS * (NT + 1))
        sh.gathered[threadIdx.x] = cluster.map_shared_rank(sh.mass[half], threadIdx.x / (NT + 1))[threadIdx.x % (NT + 1)];
    __syncthreads();
#pragma unroll
    for (int j = 0; j <= NT; ++j) {
        double t = 0.0;
#pragma unroll
        for (int b = 0; b < CL_BLOCKS; ++b) t += sh.gathered[b * (NT + 1) + j];
        v[j] = t;
    }
}

// arg-max over the cluster, lowest index on ties; every thread gets it
__device__ __forceinline__ void cluster_argmax(cg::cluster_group& cluster, ClusterShared& sh, int half, float& v, int& idx) {
    block_argmax(v, idx, sh.sv, sh.si);
    if (threadIdx.x == 0) { sh.best_v[half] = v; sh.best_i[half] = idx; }
    cluster.sync();
    const unsigned int b = threadIdx.x & (CL_BLOCKS - 1);
    v = *cluster.map_shared_rank(&sh.best_v[half], b);
    idx = *cluster.map_shared_rank(&sh.best_i[half], b);
#pragma unroll
    for (int o = CL_BLOCKS / 2; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, v, o);
        const int oi = __shfl_xor_sync(0xffffffffu, idx, o);
        if (ov > v || (ov == v && oi < idx)) { v = ov; idx = oi; }
    }
}

// The largest key c in [lo, hi) with mass_hi + (mass of the cluster's scores with c <= key < hi) >= need, lo if none,
// read off the ranked list of those scores.  False, for all threads of the cluster, if they are more than CAND.
__device__ bool cut_from_list(cg::cluster_group& cluster, ClusterShared& sh, const float* scores, int n, float m,
                              unsigned int lo, unsigned int hi, double mass_hi, double need, unsigned int& cut) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    cluster.sync();                // the lists of an earlier call have been read
    if (tid == 0) sh.n_cand = 0;
    __syncthreads();
    const float4* scores4 = reinterpret_cast<const float4*>(scores);
    const float least = score_of(lo);
    for (int q = tid; q < (n + 3) / 4; q += CL_THREADS) {
        const float4 f = scores4[q];       // (lanes beyond n: the buffer holds a multiple of 4)
        const float e[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            if (e[j] < least) continue;
            const unsigned int k = ordered_key(e[j]);
            if (k >= lo && k < hi && 4 * q + j < n) {
                const int at = atomicAdd(&sh.n_cand, 1);
                if (at < CAND) sh.cand_key[at] = k;
            }
        }
    }
    cluster.sync();
    // two warps take the list of each block
    static_assert(CL_WARPS == 2 * CL_BLOCKS, "two warps a block's list");
    int total = 0, base = 0, mine = 0;
    {
        const int b = lane & (CL_BLOCKS - 1);
        const int c = *cluster.map_shared_rank(&sh.n_cand, (unsigned int)b);
#pragma unroll
        for (int j = 0; j < CL_BLOCKS; ++j) {
            const int cj = __shfl_sync(0xffffffffu, c, j);
            if (j < warp / 2) base += cj;
            if (j == warp / 2) mine = cj;
            total += cj;
        }
    }
    if (total > CAND) return false;
    {
        const unsigned int* keys = cluster.map_shared_rank(sh.cand_key, (unsigned int)(warp / 2));
        for (int i = (warp & 1) * 32 + lane; i < mine; i += 64) sh.all_key[base + i] = keys[i];
    }
    if (tid < 4 && total + tid < (total + 3) / 4 * 4) sh.all_key[total + tid] = 0u;   // ranks below every score
    if (tid == 0) sh.first = total;
    __syncthreads();
    // ranks, largest key first (equal keys have equal masses, so their order among themselves changes nothing);
    // eight lanes count for a score
    for (int i0 = 0; i0 < total; i0 += CL_THREADS / 8) {
        const int i = i0 + tid / 8;
        const unsigned int k = i < total ? sh.all_key[i] : 0u;
        int rank = 0;
        for (int j = (tid & 7) * 4; j < total; j += 32) {
            const uint4 o = *reinterpret_cast<const uint4*>(&sh.all_key[j]);
            rank += (o.x > k || (o.x == k && j < i)) + (o.y > k || (o.y == k && j + 1 < i)) +
                    (o.z > k || (o.z == k && j + 2 < i)) + (o.w > k || (o.w == k && j + 3 < i));
        }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) rank += __shfl_xor_sync(0xffffffffu, rank, o);
        if ((tid & 7) == 0 && i < total) {
            sh.sorted_key[rank] = k;
            sh.sorted_mass[rank] = expf(__uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k) - m);
        }
    }
    __syncthreads();
    // running sums, CL_THREADS scores a round; the first position that reaches what is needed
    double before = mass_hi;
    for (int r0 = 0; r0 < total; r0 += CL_THREADS) {
        const int r = r0 + tid;
        double run = r < total ? (double)sh.sorted_mass[r] : 0.0;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double t = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += t;
        }
        if (lane == 31) sh.scan[warp] = run;
        __syncthreads();
        double warps_before = 0.0, all = 0.0;
#pragma unroll
        for (int w = 0; w < CL_WARPS; ++w) {
            if (w == warp) warps_before = all;
            all += sh.scan[w];
        }
        if (r < total && before + (warps_before + run) >= need) atomicMin(&sh.first, r);
        before += all;
        __syncthreads();
    }
    cut = sh.first < total ? sh.sorted_key[sh.first] : lo;
    return true;
}

__global__ __launch_bounds__(CL_THREADS, 2) void sample_cluster_kernel(const float* __restrict__ logits, long long row_stride,
                                                                       int V, int chunk, int vec,
                                                                       const RowParams* __restrict__ params,
                                                                       const int* __restrict__ counts_table,
                                                                       int* __restrict__ out) {
    extern __shared__ float4 scores4[];      // the block's part of the row: `chunk` scores (a multiple of 4)
    __shared__ ClusterShared sh;
    float* scores = reinterpret_cast<float*>(scores4);
    cg::cluster_group cluster = cg::this_cluster();
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.y, tid = threadIdx.x;
    const RowParams p = params[row];
    const int i0 = min(V, (int)cluster.block_rank() * chunk), n = min(V, i0 + chunk) - i0;
    const float* lg = logits + (size_t)row * row_stride + i0;
    const int* counts = (counts_table && p.slot >= 0 && p.repeat_penalty != 1.0f) ? counts_table + (size_t)p.slot * V + i0 : nullptr;
    const bool greedy = !(p.temperature > 0.f);
    const float inv_t = greedy ? 1.f : 1.0f / p.temperature;

    // scores, and their maximum (also the greedy answer)
    float best = -CUDART_INF_F;
    int best_i = 0x7fffffff;
    if (vec) {
        constexpr int U = 5;       // 16-byte words in flight a thread, of each array
        for (int q0 = tid; q0 < n / 4; q0 += U * CL_THREADS) {
            float4 l[U];
            int4 c[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int q = q0 + u * CL_THREADS;
                l[u] = q < n / 4 ? reinterpret_cast<const float4*>(lg)[q] : make_float4(0.f, 0.f, 0.f, 0.f);
                c[u] = counts && q < n / 4 ? reinterpret_cast<const int4*>(counts)[q] : make_int4(0, 0, 0, 0);
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int q = q0 + u * CL_THREADS;
                if (q >= n / 4) break;
                float f[4] = {l[u].x, l[u].y, l[u].z, l[u].w};
                if ((c[u].x | c[u].y | c[u].z | c[u].w) != 0) {
                    f[0] = penalised(f[0], c[u].x, p.repeat_penalty);
                    f[1] = penalised(f[1], c[u].y, p.repeat_penalty);
                    f[2] = penalised(f[2], c[u].z, p.repeat_penalty);
                    f[3] = penalised(f[3], c[u].w, p.repeat_penalty);
                }
#pragma unroll
                for (int j = 0; j < 4; ++j) f[j] *= inv_t;
                scores4[q] = make_float4(f[0], f[1], f[2], f[3]);
                // (a thread's places ascend: only more than its best so far, or its first score, takes the lead)
                const float most = fmaxf(fmaxf(f[0], f[1]), fmaxf(f[2], f[3]));
                if (most > best || (most == best && best_i == 0x7fffffff)) {
                    best = most;
                    best_i = i0 + 4 * q + (f[0] == most ? 0 : f[1] == most ? 1 : f[2] == most ? 2 : 3);
                }
            }
        }
    } else {
        for (int i = tid; i < n; i += CL_THREADS) {
            const float s = score_at(lg, counts, p.repeat_penalty, inv_t, i);
            if (s > best || (s == best && i0 + i < best_i)) { best = s; best_i = i0 + i; }
            scores[i] = s;
        }
        if (tid < 4 && n + tid < (n + 3) / 4 * 4) scores[n + tid] = -CUDART_INF_F;      // no mass where there is no score
    }
    cluster_argmax(cluster, sh, 0, best, best_i);      // (its barriers order the scores too)
    const float m = best;
    if (!greedy) {
        unsigned int cut = 0;  // keep scores whose ordered key is >= cut
        if (p.top_p < 1.0f) {
            // the answer lies in [lo, hi); mass_hi: of the keys from hi on
            unsigned int lo = 0, hi = ordered_key(m) + 1u;
            double mass_hi = 0.0, need = 0.0;
            for (int pass = 0;; ++pass) {
                unsigned int t[NT];
                if (pass == 0) {
#pragma unroll
                    for (int j = 0; j < NT; ++j) t[j] = ordered_key(m - FIRST_CUTS[j]);
                } else {
#pragma unroll
                    for (int j = 0; j < NT; ++j) {
                        const unsigned int step = (unsigned int)(((unsigned long long)(hi - lo) * (j + 1)) / (NT + 1));
                        t[j] = lo + (step > 0u ? step : 1u);
                    }
                }
                // v[j]: mass of t[j] <= key < hi, v[NT]: of the whole range (all of the row in the first pass)
                double v[NT + 1];
#pragma unroll
                for (int j = 0; j <= NT; ++j) v[j] = 0.0;
                // Bound by instructions: a score below all thresholds costs its exponential and one sum (the first pass) or a
                // comparison (later ones), and a branch each for the thresholds it reaches, most often none.
                const float least = score_of(t[0]);
                auto above = [&](float x, double e) {
                    const unsigned int k = ordered_key(x);
                    if (k >= t[0] && k < hi) {
                        if (pass > 0) v[NT] += e;
                        v[0] += e;
                        if (k >= t[1]) { v[1] += e;
                        if (k >= t[2]) { v[2] += e;
                        if (k >= t[3]) { v[3] += e;
                        if (k >= t[4]) { v[4] += e;
                        if (k >= t[5]) { v[5] += e;
                        if (k >= t[6]) v[6] += e; } } } } }
                    }
                };
                for (int q = tid; q < (n + 3) / 4; q += CL_THREADS) {
                    const float4 f = scores4[q];
                    const float s[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (pass == 0) {
                            const double e = (double)expf(s[c] - m);
                            v[NT] += e;
                            if (!(s[c] < least)) above(s[c], e);
                        } else if (!(s[c] < least) && 4 * q + c < n) {
                            above(s[c], (double)expf(s[c] - m));
                        }
                    }
                }
                cluster_sums(cluster, sh, pass & 1, v);
                if (pass == 0) need = (double)p.top_p * v[NT];
                unsigned int new_lo = lo, new_hi = hi;
                double new_mass = mass_hi;
#pragma unroll
                for (int j = 0; j < NT; ++j) {         // thresholds ascend, masses descend
                    if (mass_hi + v[j] >= need) new_lo = t[j];
                }
#pragma unroll
                for (int j = NT - 1; j >= 0; --j) {
                    if (!(mass_hi + v[j] >= need)) { new_hi = t[j]; new_mass = mass_hi + v[j]; }
                }
                lo = new_lo; hi = new_hi; mass_hi = new_mass;
                if (hi - lo <= 1u) { cut = lo; break; }
                if (cut_from_list(cluster, sh, scores, n, m, lo, hi, mass_hi, need, cut)) break;
            }
        }
        const unsigned long long key = mix64(((unsigned long long)p.seed_lo << 32) | (unsigned long long)p.step);
        best = m - logf(-logf(uniform01(key, (unsigned int)best_i)));      // the largest score's draw, which all others have to reach
        const float least = score_of(cut);
        for (int q = tid; q < (n + 3) / 4; q += CL_THREADS) {
            const float4 f = scores4[q];
            const float s[4] = {f.x, f.y, f.z, f.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int i = i0 + 4 * q + j;
                if (s[j] < least || s[j] + GUMBEL_MAX < best || 4 * q + j >= n || ordered_key(s[j]) < cut) continue;
                const float u = uniform01(key, (unsigned int)i);
                if (!may_draw(s[j], u, best)) continue;
                const float zv = s[j] - logf(-logf(u));
                if (zv > best || (zv == best && i < best_i)) { best = zv; best_i = i; }
            }
        }
        cluster_argmax(cluster, sh, 1, best, best_i);
    }
    if (cluster.block_rank() == 0 && tid == 0) out[row] = best_i;
    cluster.sync();        // nobody leaves while its shared memory may still be read
}

// Two-stage variant for rows that need no nucleus cut (top_p >= 1 or greedy): the vocabulary is dealt to
// `nb` blocks per row, each leaves its best (value, index), and the last stage picks among them with the same
// lowest-index rule, so the token equals the single-block kernel's.
// BOUNDED: may_draw before the logarithms.  A thread's best draw has to rise before that spares any: with 28 to 43 scores a thread it
// costs 5 to 10 % more (31 rows of 190,000 37 us without it, 41 with; 100 of 32,000 32 and 36), at 57 to 64 a percent less (128 of 65,536
// 58.7 and 58.1), from 128 on it saves 12 to 15 % (64 of 262,144 129 and 112, 128 of 262,144 237 and 203).
constexpr int BOUNDED_FROM = 56;
template <bool BOUNDED>
__global__ __launch_bounds__(512) void sample_part_kernel(const float* __restrict__ logits, long long row_stride, int V,
                                                          const RowParams* __restrict__ params,
                                                          const int* __restrict__ counts_table, float* __restrict__ part_v,
                                                          int* __restrict__ part_i) {
    __shared__ float sv[33];
    __shared__ int si[33];
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x, nb = gridDim.y, b = blockIdx.y;
    const RowParams p = params[row];
    const float* lg = logits + (size_t)row * row_stride;
    const int* counts = (counts_table && p.slot >= 0 && p.repeat_penalty != 1.0f) ? counts_table + (size_t)p.slot * V : nullptr;
    const bool greedy = !(p.temperature > 0.f);
    const float inv_t = greedy ? 1.f : 1.0f / p.temperature;
    const unsigned long long key = mix64(((unsigned long long)p.seed_lo << 32) | (unsigned long long)p.step);
    const int chunk = (V + nb - 1) / nb;
    const int lo = b * chunk, hi = min(V, lo + chunk);
    float best = -CUDART_INF_F;
    int best_i = 0x7fffffff;
    for (int i = lo + threadIdx.x; i < hi; i += blockDim.x) {
        float s = score_at(lg, counts, p.repeat_penalty, inv_t, i);
        if (!greedy) {
            if (s + GUMBEL_MAX < best) continue;
            const float u = uniform01(key, (unsigned int)i);
            if (BOUNDED && !may_draw(s, u, best)) continue;
            s -= logf(-logf(u));
        }
        if (s > best || (s == best && i < best_i)) { best = s; best_i = i; }
    }
    block_argmax(best, best_i, sv, si);
    if (threadIdx.x == 0) {
        part_v[row * nb + b] = best;
        part_i[row * nb + b] = best_i;
    }
}

__global__ void sample_pick_kernel(const float* __restrict__ part_v, const int* __restrict__ part_i, int nb,
                                   int* __restrict__ out) {
    pdl_trigger();
    pdl_wait();
    const int row = blockIdx.x;
    float best = -CUDART_INF_F;
    int best_i = 0x7fffffff;
    for (int b = threadIdx.x; b < nb; b += 32) {
        const float v = part_v[row * nb + b];
        const int i = part_i[row * nb + b];
        if (v > best || (v == best && i < best_i)) { best = v; best_i = i; }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ov > best || (ov == best && oi < best_i)) { best = ov; best_i = oi; }
    }
    if (threadIdx.x == 0) out[row] = best_i;
}

__global__ void count_tokens_kernel(const int* __restrict__ ids, const int* __restrict__ slots, int* __restrict__ counts,
                                    int n, int V, int slot_bias) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= n) return;
    const int id = ids[t], slot = slots[t] - slot_bias;
    if (slot >= 0 && id >= 0 && id < V) atomicAdd(counts + (size_t)slot * V + id, 1);
}

}  // namespace

// params: n_rows records of 8 x 32-bit words: temperature, top_p, repeat_penalty (floats), count-table row or -1,
// seed (low 32 bits, high 32 bits, high unused), step, pad
// cluster: a cluster of blocks a row (V up to 393,216: its blocks' shared memory holds the row's scores), else a block a row
VCB_API int vcb_sample(const float* logits, long long row_stride, int n_rows, int V, const void* params,
                       const int* counts_table, int cluster, int* out, cudaStream_t stream) {
    if (n_rows == 0) return 0;
    VCB_CHECK_ARG(n_rows > 0 && V > 0 && row_stride >= V, "sample: bad sizes rows=%d V=%d stride=%lld", n_rows, V, row_stride);
    if (cluster) {
        const int chunk = ((V + CL_BLOCKS - 1) / CL_BLOCKS + 3) / 4 * 4;
        const size_t smem = (size_t)chunk * sizeof(float);
        VCB_CHECK_ARG(smem <= CLUSTER_MAX_SMEM && n_rows <= 65535, "sample: %d rows of %d scores are more than clusters take", n_rows, V);
        VCB_CHECK_ARG(cudaFuncSetAttribute(sample_cluster_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLUSTER_MAX_SMEM) == cudaSuccess,
                      "sample: %zu bytes of shared memory refused", CLUSTER_MAX_SMEM);
        const int vec = row_stride % 4 == 0 && (uintptr_t)logits % 16 == 0 && V % 4 == 0 && (uintptr_t)counts_table % 16 == 0;
        launch_pdl_clusters(sample_cluster_kernel, dim3(CL_BLOCKS, n_rows), dim3(CL_THREADS), smem, stream, (unsigned)CL_BLOCKS,
                            logits, row_stride, V, chunk, vec, (const RowParams*)params, counts_table, out);
        VCB_CHECK_LAUNCH("sample_cluster");
        return 0;
    }
    const int threads = V >= 8192 ? 1024 : 256;
    sample_kernel<<<n_rows, threads, 0, stream>>>(logits, row_stride, V, (const RowParams*)params, counts_table, out);
    VCB_CHECK_LAUNCH("sample");
    return 0;
}

// counts[slots[t] - slot_bias][ids[t]] += 1 for every token whose slot entry, less the bias, is >= 0
VCB_API int vcb_count_tokens(const int* ids, const int* slots, int* counts, int n, int V, int slot_bias, cudaStream_t stream) {
    if (n == 0) return 0;
    count_tokens_kernel<<<(n + 255) / 256, 256, 0, stream>>>(ids, slots, counts, n, V, slot_bias);
    VCB_CHECK_LAUNCH("count_tokens");
    return 0;
}

// For batches in which no row cuts a nucleus: `nb` blocks per row; part_v / part_i hold n_rows * nb entries.
VCB_API int vcb_sample_split(const float* logits, long long row_stride, int n_rows, int V, const void* params,
                             const int* counts_table, float* part_v, int* part_i, int nb, int* out,
                             cudaStream_t stream) {
    if (n_rows == 0) return 0;
    VCB_CHECK_ARG(n_rows > 0 && V > 0 && row_stride >= V && nb >= 1 && nb <= 1024, "sample_split: bad sizes");
    auto part = (V + nb - 1) / nb > BOUNDED_FROM * 512 ? sample_part_kernel<true> : sample_part_kernel<false>;
    launch_pdl(part, dim3(n_rows, nb), dim3(512), 0, stream, logits, row_stride, V, (const RowParams*)params, counts_table, part_v, part_i);
    VCB_CHECK_LAUNCH("sample_part");
    launch_pdl(sample_pick_kernel, dim3(n_rows), dim3(32), 0, stream, part_v, part_i, nb, out);
    VCB_CHECK_LAUNCH("sample_pick");
    return 0;
}
