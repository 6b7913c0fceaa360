// The small kernels either side of the seed mat-vec on the MoE path: router top-k, SwiGLU, the two combines, grouping
// of (token, expert) pairs by expert, activation packing, and the expert cache's admit and copy.
// Reference behaviour they reproduce: engine/kernels_qwen4.cu:385-422 (router), :506-515 (combine);
// engine/kernels_moe.cu:775-788 (SwiGLU, MoVA combine), :527-573 (grouping), :2023-2112 (cache), :2196-2201 (pack).
#include <math.h>

#include "common.cuh"
#include "route.cuh"
#include "seed_block.cuh"

namespace nsl {

__device__ __forceinline__ bool aligned16_dev(const void* p) { return ((unsigned long long) p & 15ull) == 0; }

// ---- router ------------------------------------------------------------------------------------------------------------
// One warp per row (route_row in route.cuh).
template <int PER>                   // experts per lane held in registers: E <= 32 * PER
__global__ void __launch_bounds__(128) route_kernel(int E, int k, const float* logits, int ld,
                                                    int32_t* __restrict__ ind, float* __restrict__ wt, int T) {
    const int lane = threadIdx.x & 31, t = blockIdx.x * 4 + (threadIdx.x >> 5);
    grid_dependency_wait();
    grid_dependents_go();   // only now: the next kernel's blocks would otherwise sit on the SMs the previous one still needs
    if (t >= T) return;
    route_row<PER>(E, k, logits + (size_t) t * ld, lane, ind + (size_t) t * k, wt + (size_t) t * k);
}

// ---- elementwise --------------------------------------------------------------------------------------------------------
__device__ __forceinline__ float silu_bf16(float g) {
    const float s = bf16_round(1.0f / (1.0f + expf(-g)));
    return bf16_round(g * s);
}
__global__ void swiglu_kernel(const float* __restrict__ g, const float* __restrict__ u, float* __restrict__ a, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        a[i] = bf16_round(silu_bf16(g[i]) * u[i]);
}

// The same values as bf16 bits (they are bf16 values already): the packed input of the down projection's GEMM.
__global__ void swiglu_packed_kernel(const float* __restrict__ g, const float* __restrict__ u, uint16_t* __restrict__ a, int n) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n / 2; i += gridDim.x * blockDim.x) {
        const float2 gv = ((const float2*) g)[i], uv = ((const float2*) u)[i];
        const uint32_t lo = __float_as_uint(bf16_round(silu_bf16(gv.x) * uv.x)) >> 16, hi = __float_as_uint(bf16_round(silu_bf16(gv.y) * uv.y)) & 0xFFFF0000u;
        ((uint32_t*) a)[i] = lo | hi;
    }
}

// out[t][i] = sigmoid(sg[t*sgld]) sh[t][i] + sum_j wt[t][j] D[t*k+j][i], plain f32, j ascending; sh == NULL: no shared
// expert term.
__global__ void q4_combine_kernel(int d, int k, const float* D, const float* wt,
                                  const float* sh, const float* sg, int sgld, float* __restrict__ out) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    grid_dependents_go();
    grid_dependency_wait();
    if (i >= d) return;
    float a = 0.0f;
    if (sh) a = (1.0f / (1.0f + expf(-sg[(size_t) t * sgld]))) * sh[(size_t) t * d + i];
    for (int j = 0; j < k; ++j) a += wt[t * k + j] * D[((size_t) t * k + j) * d + i];
    out[(size_t) t * d + i] = a;
}

// The end of a decoder layer and the start of the next: the combine above, x = bf16(x + its result) (nsl_residual_add) and y = the
// grouped RMSNorm of x (kc_gnorm), a block a row, each value formed as those three kernels form it.  For a decode batch
// each of them is a launch's latency and little else.
__global__ void __launch_bounds__(256) combine_residual_gnorm_kernel(int d, int k, const float* D, const float* wt,
                                                                     const float* sh, const float* sg, int sgld,
                                                                     float* __restrict__ x, float eps,
                                                                     const uint16_t* __restrict__ w, float* __restrict__ y) {
    __shared__ float part[8];
    grid_dependency_wait();
    grid_dependents_go();
    const int t = blockIdx.x, half = threadIdx.x >> 7, i0 = threadIdx.x & 127, hw = d / 2;      // (kc_gnorm's split of a row)
    const size_t at = (size_t) t * d + (size_t) half * hw;
    const float* const Dr = D + (size_t) t * k * d + (size_t) half * hw;
    const float gate = 1.0f / (1.0f + expf(-sg[(size_t) t * sgld]));
    float s = 0.0f;
    for (int c0 = i0; c0 < hw; c0 += 8 * 128) {      // eight values a thread side by side
        float a[8], xv[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = c0 + 128 * q;
            if (c < hw) { a[q] = gate * sh[at + c]; xv[q] = x[at + c]; }
        }
#pragma unroll 4
        for (int j = 0; j < k; ++j) {
            const float wj = wt[t * k + j];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int c = c0 + 128 * q;
                if (c < hw) a[q] += wj * Dr[(size_t) j * d + c];
            }
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int c = c0 + 128 * q;
            if (c < hw) {
                const float v = bf16_round(xv[q] + a[q]);
                x[at + c] = v;
                s = fmaf(v, v, s);
            }
        }
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xFFFFFFFFu, s, o);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    const float tot = ((part[4 * half] + part[4 * half + 1]) + part[4 * half + 2]) + part[4 * half + 3];
    const float r = rsqrtf(tot / (float) hw + eps);
    const uint16_t* wr = w + (size_t) half * hw;
    for (int c = i0; c < hw; c += 128) y[at + c] = bf16_round(__uint_as_float((uint32_t) wr[c] << 16) * (x[at + c] * r));      // (x: this thread's own stores)
}
void launch_combine_residual_gnorm(cudaStream_t s, int d, int k, const float* D, const float* wt, const float* sh, const float* sg, int sgld, float* x,
                                   float eps, const uint16_t* w, float* y, int T) {
    launch(combine_residual_gnorm_kernel, (unsigned) T, 256, 0, s, d, k, D, wt, sh, sg, sgld, x, eps, w, y);
    count_launch();
}

// The same without a shared expert over packed bf16 rows (d a multiple of 8: 16 bytes of each of the k rows a thread).  vec: out is
// 16-byte aligned (the caller's pointer may be any).
__global__ void __launch_bounds__(256) combine_packed_kernel(int d8, int k, const uint4* D, const float* wt,
                                                             float* __restrict__ out, int n, int vec) {
    grid_dependency_wait();
    grid_dependents_go();
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= n) return;
    const int t = i / d8, c = i - t * d8;
    float a[8] = {};
    for (int j0 = 0; j0 < k; j0 += 8) {      // eight rows requested side by side, added in order
        uint4 v[8];
        float w[8];
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (j0 + q < k) {
                v[q] = D[((size_t) t * k + j0 + q) * d8 + c];
                w[q] = wt[t * k + j0 + q];
            }
#pragma unroll
        for (int q = 0; q < 8; ++q)
            if (j0 + q < k) {
                const uint32_t u[4] = {v[q].x, v[q].y, v[q].z, v[q].w};
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    a[2 * e] += w[q] * __uint_as_float(u[e] << 16);
                    a[2 * e + 1] += w[q] * __uint_as_float(u[e] & 0xFFFF0000u);
                }
            }
    }
    float* const o = out + 8 * (size_t) i;
    if (vec) {
        ((float4*) o)[0] = make_float4(a[0], a[1], a[2], a[3]);
        ((float4*) o)[1] = make_float4(a[4], a[5], a[6], a[7]);
    } else {
#pragma unroll
        for (int e = 0; e < 8; ++e) o[e] = a[e];
    }
}
void launch_combine_packed(cudaStream_t s, int d, int k, const uint16_t* D, const float* wt, float* out, int T) {
    const int n = T * (d / 8);
    launch(combine_packed_kernel, (unsigned) (n + 255) / 256, 256, 0, s, d / 8, k, (const uint4*) D, wt, out, n, (int) aligned16(out));
    count_launch();
}

// x = bf16(x + bf16(bf16(sum_j bf16(D_j bf16(w_j))) + shared))
__global__ void moe_combine_kernel(const float* __restrict__ D, const float* __restrict__ w, const float* __restrict__ shared,
                                   float* __restrict__ x, int d, int k) {
    const int c = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    if (c >= d) return;
    float s = 0.0f;
    for (int j = 0; j < k; ++j) s += bf16_round(__fmul_rn(D[((size_t) t * k + j) * d + c], bf16_round(w[t * k + j])));
    const size_t i = (size_t) t * d + c;
    x[i] = bf16_round(x[i] + bf16_round(bf16_round(s) + shared[i]));
}

__device__ __forceinline__ void pack_bf16(const float* x, uint16_t* __restrict__ y, size_t n, unsigned block, unsigned blocks) {
    const size_t n8 = n / 8;
    for (size_t i = (size_t) block * blockDim.x + threadIdx.x; i < n8; i += (size_t) blocks * blockDim.x) {
        const float4 a = ((const float4*) x)[2 * i], b = ((const float4*) x)[2 * i + 1];
        ((uint4*) y)[i] = make_uint4(bf16x2_bits(a.x, a.y), bf16x2_bits(a.z, a.w), bf16x2_bits(b.x, b.y), bf16x2_bits(b.z, b.w));
    }
    if (block == 0 && threadIdx.x < (n & 7)) y[n8 * 8 + threadIdx.x] = bf16_bits(x[n8 * 8 + threadIdx.x]);
}
__global__ void pack_bf16_kernel(const float* x, uint16_t* __restrict__ y, size_t n) {
    grid_dependency_wait();
    grid_dependents_go();
    pack_bf16(x, y, n, blockIdx.x, gridDim.x);
}

// Packed bf16 rows in the order of the pairs by expert: row at[t * k + j] of y = row t of x for each of its k pairs (d a multiple of 8;
// a thread: 8 values, read and converted once).  Bound by the writes: 32768 rows of 2048 from 4096 in 26 us (168 MB); a row of y at a time, its
// inputs read again for every pair, took 51.
__global__ void __launch_bounds__(256) pack_sorted_kernel(const float4* x, const int32_t* at, uint4* __restrict__ y, int k, int d8,
                                                          int T) {
    __shared__ int pos[32];
    grid_dependency_wait();
    grid_dependents_go();
    for (int t = blockIdx.x; t < T; t += gridDim.x) {
        __syncthreads();      // the previous row's places are no longer read
        if ((int) threadIdx.x < k) pos[threadIdx.x] = at[(size_t) t * k + threadIdx.x];
        __syncthreads();
        const float4* xp = x + (size_t) t * d8 * 2;
        for (int c = threadIdx.x; c < d8; c += 256) {
            const float4 a = xp[2 * c], b = xp[2 * c + 1];
            const uint4 v = make_uint4(bf16x2_bits(a.x, a.y), bf16x2_bits(a.z, a.w), bf16x2_bits(b.x, b.y), bf16x2_bits(b.z, b.w));
            for (int j = 0; j < k; ++j)
                if ((unsigned) pos[j] < (unsigned) (T * k)) y[(size_t) pos[j] * d8 + c] = v;      // (a pair of no expert has no place)
        }
    }
}
void launch_pack_sorted(cudaStream_t s, const float* x, const int32_t* at, uint16_t* y, int T, int k, int d) {
    const int cap = sm_count() * 8;
    launch(pack_sorted_kernel, (unsigned) (T < cap ? T : cap), 256, 0, s, (const float4*) x, at, (uint4*) y, k, d / 8, T);
    count_launch();
}

// ---- grouping ---------------------------------------------------------------------------------------------------------
// work (2n+3 ints): [0] tile count, [1..n+1] pair offset of each expert, [n+2..2n+2] tile offset of each expert.
// One block: histogram by shared-memory atomics, then an exclusive scan of pairs and tiles over the experts (both in one 64-bit
// word, by warp shuffles: two barriers).
// The block's 1024 threads: pairs of expert tid (count_e), pairs (low half) and tiles (high half) of the experts before it, of all.
__device__ __forceinline__ unsigned long long bucket_offsets(const int32_t* inds, int count, int n, int& count_e, unsigned long long& all) {
    __shared__ int cnt[BUCKET_MAX_EXPERTS];
    __shared__ unsigned long long wsum[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    cnt[tid] = 0;
    __syncthreads();
    auto add = [&](int e) { if (e >= 0 && e < n) atomicAdd(&cnt[e], 1); };
    const int n4 = aligned16_dev(inds) ? count / 4 : 0;
    for (int i = tid; i < n4; i += 1024) { const int4 e = ((const int4*) inds)[i]; add(e.x); add(e.y); add(e.z); add(e.w); }
    for (int i = n4 * 4 + tid; i < count; i += 1024) add(inds[i]);
    __syncthreads();
    const int c = tid < n ? cnt[tid] : 0, tl = (c + MMT_BN - 1) / MMT_BN;
    const unsigned long long mine = ((unsigned long long) tl << 32) | (unsigned) c;
    unsigned long long inc = mine;
    for (int o = 1; o < 32; o <<= 1) { const unsigned long long v = __shfl_up_sync(FULL, inc, o); if (lane >= o) inc += v; }
    if (lane == 31) wsum[w] = inc;
    __syncthreads();
    const unsigned long long ws = wsum[lane];      // every warp scans the 32 warp sums itself
    unsigned long long wi = ws;
    for (int o = 1; o < 32; o <<= 1) { const unsigned long long v = __shfl_up_sync(FULL, wi, o); if (lane >= o) wi += v; }
    all = __shfl_sync(FULL, wi, 31);
    count_e = c;
    return __shfl_sync(FULL, wi - ws, w) + inc - mine;
}
__device__ __forceinline__ void bucket_work(int32_t* work, int n, unsigned long long before, unsigned long long all) {
    const int tid = threadIdx.x;
    if (tid < n) {
        work[1 + tid] = (int) (unsigned) before;
        work[2 + n + tid] = (int) (before >> 32);
    }
    if (tid == 0) {
        work[1 + n] = (int) (unsigned) all;
        work[2 + 2 * n] = work[0] = (int) (all >> 32);
    }
}
__global__ void __launch_bounds__(1024) bucket_count_kernel(const int32_t* inds, int count, int n,
                                                            int32_t* __restrict__ work) {
    grid_dependency_wait();
    grid_dependents_go();
    int c;
    unsigned long long all;
    const unsigned long long before = bucket_offsets(inds, count, n, c, all);
    bucket_work(work, n, before, all);
}
// One block per expert.  Each warp owns a contiguous range of the pair list (a multiple of 128, four entries a lane): it counts its
// matches, the block scans the 32 counts, then each warp writes its matches in order (ballot prefixes), so perm is ascending
// within the expert.
__device__ __forceinline__ void bucket_place(const int32_t* inds, int count, int e, int begin, int total, int t0, int32_t* __restrict__ perm,
                                             MmTile* __restrict__ tiles, int32_t* __restrict__ at_out) {
    __shared__ int wcount[32];
    const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5;
    if (total <= 0) return;
    const bool vec = aligned16_dev(inds);
    const int per = ((count + 31) / 32 + 127) & ~127;
    const int lo = w * per, hi = lo + per < count ? lo + per : count;
    auto four = [&](int i, bool* f) {      // the lane's entries i .. i + 3
        if (vec && i + 3 < hi) {
            const int4 v = *(const int4*) (inds + i);
            f[0] = v.x == e; f[1] = v.y == e; f[2] = v.z == e; f[3] = v.w == e;
        } else {
#pragma unroll
            for (int q = 0; q < 4; ++q) f[q] = i + q < hi && inds[i + q] == e;
        }
    };
    int mine = 0;
    for (int i = lo + 4 * lane; i - 4 * lane < hi; i += 128) {
        bool f[4];
        four(i, f);
        mine += (int) f[0] + (int) f[1] + (int) f[2] + (int) f[3];
    }
    mine = __reduce_add_sync(FULL, mine);
    if (lane == 0) wcount[w] = mine;
    __syncthreads();
    if (mine) {
        int at = begin + __reduce_add_sync(FULL, lane < w ? wcount[lane] : 0);
        const uint32_t below = (1u << lane) - 1u;
        for (int i = lo + 4 * lane; i - 4 * lane < hi; i += 128) {
            bool f[4];
            four(i, f);
            if (!__any_sync(FULL, f[0] || f[1] || f[2] || f[3])) continue;
            uint32_t m[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) m[q] = __ballot_sync(FULL, f[q]);
            int pos = at + __popc(m[0] & below) + __popc(m[1] & below) + __popc(m[2] & below) + __popc(m[3] & below);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                if (f[q]) {
                    if (at_out) at_out[i + q] = pos;      // the inverse of perm
                    perm[pos++] = i + q;
                }
            at += __popc(m[0]) + __popc(m[1]) + __popc(m[2]) + __popc(m[3]);
        }
    }
    for (int t = tid; t * MMT_BN < total; t += 1024) {
        MmTile tl = {e, begin + t * MMT_BN, total - t * MMT_BN < MMT_BN ? total - t * MMT_BN : MMT_BN, 0};
        tiles[t0 + t] = tl;
    }
}
__global__ void __launch_bounds__(1024) bucket_place_kernel(const int32_t* inds, int count,
                                                            const int32_t* work, int32_t* __restrict__ perm,
                                                            MmTile* __restrict__ tiles, int32_t* __restrict__ at_out) {
    const int e = blockIdx.x, n = gridDim.x;
    grid_dependency_wait();
    grid_dependents_go();
    const int begin = work[1 + e];
    bucket_place(inds, count, e, begin, work[2 + e] - begin, work[2 + n + e], perm, tiles, at_out);
}
// Short pair lists: both in one launch, every block counting the whole list itself (8 entries a thread at BUCKET_ONE_PAIRS); the blocks
// beyond the experts' pack the layer's inputs (pack_n values of x), which nothing here needs.  Three launches in a row cost a prompt
// of a few hundred rows three latencies, 3 us each.
constexpr int BUCKET_ONE_PAIRS = 8192;
__global__ void __launch_bounds__(1024) bucket_pack_kernel(const int32_t* inds, int count, int n, int32_t* __restrict__ work, int32_t* __restrict__ perm,
                                                           MmTile* __restrict__ tiles, const float* x, uint16_t* __restrict__ xp, size_t pack_n) {
    __shared__ int mine[3];
    grid_dependency_wait();      // (its dependents go when it ends: the persistent GEMM's blocks would come in wherever an SM is free, and two with one unit more share one: 298 us for 512 rows instead of 274)
    const int e = blockIdx.x;
    if (e >= n) {
        pack_bf16(x, xp, pack_n, (unsigned) (e - n), gridDim.x - (unsigned) n);
        return;
    }
    int c;
    unsigned long long all;
    const unsigned long long before = bucket_offsets(inds, count, n, c, all);
    if (e == 0) bucket_work(work, n, before, all);
    if ((int) threadIdx.x == e) { mine[0] = (int) (unsigned) before; mine[1] = c; mine[2] = (int) (before >> 32); }
    __syncthreads();
    bucket_place(inds, count, e, mine[0], mine[1], mine[2], perm, tiles, NULL);
}

void bucket(cudaStream_t s, const int32_t* inds, int count, int n, int32_t* perm, MmTile* tiles, int32_t* ntiles, int32_t* at);
// kc_bucket and kc_pack_input_bf16 (x -> xp, pack_n values) of a prompt.
void bucket_pack(cudaStream_t s, const int32_t* inds, int count, int n, int32_t* perm, MmTile* tiles, int32_t* ntiles, const float* x, uint16_t* xp, size_t pack_n) {
    if (n < 1 || n > BUCKET_MAX_EXPERTS || count > BUCKET_ONE_PAIRS) {
        bucket(s, inds, count, n, perm, tiles, ntiles, NULL);
        kc_pack_input_bf16(s, x, xp, pack_n);
        return;
    }
    const size_t blocks = (pack_n / 8 + 1023) / 1024 + 1;
    launch(bucket_pack_kernel, (unsigned) n + (unsigned) (blocks < (size_t) sm_count() * 4 ? blocks : (size_t) sm_count() * 4), 1024, 0, s, inds, count, n, ntiles, perm,
           tiles, x, xp, pack_n);
    count_launch();
}
// kc_bucket; at (optional, count ints): every pair's place in perm.
void bucket(cudaStream_t s, const int32_t* inds, int count, int n, int32_t* perm, MmTile* tiles, int32_t* ntiles, int32_t* at) {
    if (n < 1 || n > BUCKET_MAX_EXPERTS) { set_error("kc_bucket: %d experts, at most %d", n, BUCKET_MAX_EXPERTS); return; }
    launch(bucket_count_kernel, 1, 1024, 0, s, inds, count, n, ntiles);
    launch(bucket_place_kernel, (unsigned) n, 1024, 0, s, inds, count, (const int32_t*) ntiles, perm, tiles, at);
    count_launch(2);
}

// ---- expert cache -----------------------------------------------------------------------------------------------------
// Policy (engine/kernels_cuda.h:26-55): the units a call needs are marked; hits get the new tick; misses, in expert order,
// take the least recently used slots (ties: lowest slot) among those this call has not touched and, with
// CACHE_PROTECT_PREV, the previous admit did not touch; a taken slot's old unit is evicted, the unit's slice tables are
// pointed at the slot and a (unit, slot) copy job is queued.  When fewer slots may be replaced than there are misses,
// the remaining misses are left out (njobs = admitted count).
//
// How it is computed here (one block, no serial loop over the misses).  Taking the LRU slot m times in a row is the
// same as taking the m smallest (last use, slot) keys among the replaceable slots, in order.  So: (1) an MSB-first
// radix select over the 32-bit last-use ticks finds the tick of the m-th victim and how many slots lie below it;
// (2) one ordered pass in slot order collects the victims: every replaceable slot below that tick, and of those equal to
// it the lowest slots that are still needed; (3) the victims (at most 1024, in shared memory) are ranked by counting;
// (4) thread r pairs the r-th miss with the victim of rank r and rewrites the tables for it -- all misses at once.
constexpr int ADMIT_T = CACHE_MAX_PER_LAYER;   // threads of the block = the most units one layer has

__device__ __forceinline__ bool slot_replaceable(uint32_t last, uint32_t now, uint32_t prev) { return last != now && last != prev; }

// Exclusive position of this thread's flag among the block's flags (thread order) and their total; `carry` is shared.
__device__ __forceinline__ int block_rank(bool flag, int* wsum, int& total) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t m = __ballot_sync(FULL, flag);
    __syncthreads();            // wsum may still be read from the previous call
    if (lane == 0) wsum[w] = __popc(m);
    __syncthreads();
    int before = 0, all = 0;
    for (int q = 0; q < ADMIT_T / 32; ++q) { const int c = wsum[q]; if (q < w) before += c; all += c; }
    total = all;
    return before + __popc(m & ((1u << lane) - 1u));
}

__global__ void __launch_bounds__(ADMIT_T) cache_admit_kernel(CachePool p, int sl, const int32_t* __restrict__ inds,
                                                              int count, int flags) {
    __shared__ int need[ADMIT_T];                    // expert -> needed by this call
    __shared__ int miss_of[ADMIT_T];                 // r -> the r-th missing expert (ascending)
    __shared__ unsigned long long vict[ADMIT_T];     // victims' (last use, slot) keys, in slot order
    __shared__ int hist[256];
    __shared__ int wsum[ADMIT_T / 32];
    __shared__ uint32_t sel_prefix;
    __shared__ int sel_remaining;
    const int tid = threadIdx.x;
    const uint32_t prev = (flags & CACHE_PROTECT_PREV) ? p.tick[0] : 0xFFFFFFFFu;
    const uint32_t now = p.tick[0] + 1;
    need[tid] = 0;
    __syncthreads();
    for (int i = tid; i < count; i += ADMIT_T) {
        const int e = inds[i];
        if (e >= 0 && e < p.per_layer) need[e] = 1;
    }
    __syncthreads();
    // hits are touched, misses listed in expert order
    const bool wanted = tid < p.per_layer && need[tid];
    const int held = wanted ? p.unit_slot[(size_t) sl * p.per_layer + tid] : -1;
    if (wanted && held >= 0) p.slot_last[held] = now;
    int n_need, n_miss;
    block_rank(wanted, wsum, n_need);
    const bool missing = wanted && held < 0;
    const int mpos = block_rank(missing, wsum, n_miss);
    if (missing) miss_of[mpos] = tid;
    __syncthreads();          // the hits' new ticks are visible to the whole block from here on
    // how many slots may be replaced
    int mine = 0;
    for (int s = tid; s < p.slots; s += ADMIT_T) mine += slot_replaceable(p.slot_last[s], now, prev);
    if (tid < 256) hist[tid] = 0;
    __syncthreads();
    if (mine) atomicAdd(&hist[0], mine);
    __syncthreads();
    const int n_free = hist[0];
    const int n_adm = n_miss < n_free ? n_miss : n_free;      // victims wanted
    if (tid == 0) {
        p.tick[0] = now;
        p.stats[0] += (uint32_t) (n_need - n_miss);
        p.stats[1] += (uint32_t) n_miss;
        *p.njobs = n_adm;
        sel_prefix = 0u;
        sel_remaining = n_adm;
    }
    __syncthreads();
    if (n_adm == 0) return;
    // (1) the tick of the n_adm-th smallest replaceable slot, one byte per pass from the top
    uint32_t known = 0u;      // mask of the bits already fixed
    for (int shift = 24; shift >= 0; shift -= 8) {
        if (tid < 256) hist[tid] = 0;
        __syncthreads();
        const uint32_t prefix = sel_prefix;
        for (int s = tid; s < p.slots; s += ADMIT_T) {
            const uint32_t last = p.slot_last[s];
            if (slot_replaceable(last, now, prev) && (last & known) == prefix) atomicAdd(&hist[(last >> shift) & 255u], 1);
        }
        __syncthreads();
        if (tid == 0) {
            int left = sel_remaining, b = 0;
            while (b < 255 && hist[b] < left) left -= hist[b++];
            sel_remaining = left;                 // rank inside bin b, 1-based
            sel_prefix = prefix | ((uint32_t) b << shift);
        }
        known |= 255u << shift;
        __syncthreads();
    }
    const uint32_t cut = sel_prefix;               // every replaceable slot older than `cut` is a victim,
    const int want_eq = sel_remaining;             // and the `want_eq` lowest slots whose tick equals it
    // (2) the victims, gathered in slot order
    int n_lt = 0, n_eq = 0;
    for (int base = 0; base < p.slots; base += ADMIT_T) {
        const int s = base + tid;
        const uint32_t last = s < p.slots ? p.slot_last[s] : now;
        const bool ok = s < p.slots && slot_replaceable(last, now, prev);
        int t_lt, t_eq;
        const int r_lt = block_rank(ok && last < cut, wsum, t_lt);
        const int r_eq = block_rank(ok && last == cut, wsum, t_eq);
        const unsigned long long key = ((unsigned long long) last << 32) | (uint32_t) s;
        // older slots fill the list's front part from the left, equal ones its last want_eq entries
        if (ok && last < cut) vict[n_lt + r_lt] = key;
        if (ok && last == cut && n_eq + r_eq < want_eq) vict[(n_adm - want_eq) + n_eq + r_eq] = key;
        n_lt += t_lt;
        n_eq += t_eq;
    }
    __syncthreads();
    // (3) + (4): thread t owns victim t, finds its rank among the victims and serves the miss of that rank
    if (tid < n_adm) {
        const unsigned long long key = vict[tid];
        int rank = 0;
        for (int j = 0; j < n_adm; ++j) rank += vict[j] < key;
        const int slot = (int) (key & 0xFFFFFFFFu), x = miss_of[rank], u = sl * p.per_layer + x;
        const int old = p.slot_unit[slot];
        if (old >= 0) p.unit_slot[old] = -1;
        p.slot_unit[slot] = u;
        p.unit_slot[u] = slot;
        p.slot_last[slot] = now;
        p.jobs[2 * rank] = u;
        p.jobs[2 * rank + 1] = slot;
        uint8_t* base = p.vram + (uint64_t) slot * p.unit_bytes;
        for (int i = 0; i < p.ntens; ++i) {
            WSlice* t = p.tab + ((size_t) sl * p.ntens + i) * p.per_layer + x;
            for (int st = 0; st < 4; ++st)
                if (p.off[i][st] != 0xFFFFFFFFu) t->p[st] = base + p.off[i][st];
        }
    }
}

// Copy (grid = the caller's block count): the queued units, as one long run of 16-byte words (job after job), are dealt
// to the blocks in contiguous shares, so a block streams a few long host ranges (mapped pinned memory, read over PCIe by
// the kernel itself) instead of striding over every unit; eight loads in flight per thread.
__global__ void __launch_bounds__(512) cache_copy_kernel(CachePool p) {
    const int nj = *p.njobs;
    if (nj <= 0) return;
    const uint64_t per_unit = p.unit_bytes / 16, total = per_unit * (uint64_t) nj;
    const uint64_t lo = total * blockIdx.x / gridDim.x, hi = total * (blockIdx.x + 1) / gridDim.x;
    uint64_t at = lo;
    while (at < hi) {
        const int j = (int) (at / per_unit);
        const uint64_t w0 = at - (uint64_t) j * per_unit;
        const uint64_t n = (hi - at) < (per_unit - w0) ? (hi - at) : (per_unit - w0);     // words of job j in this share
        const uint4* src = (const uint4*) (p.host + (uint64_t) p.jobs[2 * j] * p.unit_bytes) + w0;
        uint4* dst = (uint4*) (p.vram + (uint64_t) p.jobs[2 * j + 1] * p.unit_bytes) + w0;
        uint64_t i = threadIdx.x;
        for (; i + 7 * 512 < n; i += 8 * 512) {
            uint4 v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = src[i + q * 512];
#pragma unroll
            for (int q = 0; q < 8; ++q) dst[i + q * 512] = v[q];
        }
        for (; i < n; i += 512) dst[i] = src[i];
        at += n;
    }
}


// ---- grouping without caller-provided work memory ---------------------------------------------------------------------
// The offsets that bucket_count_kernel hands to bucket_place_kernel (2 n + 3 ints) live here instead of in a buffer the
// caller allocates.  One array per GPU that loads the library, held until the process exits; sized for the largest
// expert count the grouping accepts.
constexpr int BUCKET_SCRATCH_INTS = 2 * BUCKET_MAX_EXPERTS + 3;
static __device__ __align__(256) int32_t g_bucket_scratch[BUCKET_SCRATCH_INTS];

__global__ void bucket_publish_kernel(const int32_t* work, int32_t* __restrict__ ntiles_out) {
    grid_dependency_wait();
    grid_dependents_go();
    if (threadIdx.x == 0 && blockIdx.x == 0) ntiles_out[0] = work[0];
}

// The array's device address on the current device.  In host code the symbol's name is only a host-side handle, not an
// address a kernel can use, so the address is asked for once per device with that device current.
static int32_t* bucket_scratch_ptr() {
    static int32_t* ptr[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) { set_error("nsl_bucket_noalloc: no current device"); return NULL; }
    if (!ptr[dev]) {
        void* p = NULL;
        const cudaError_t rc = cudaGetSymbolAddress(&p, g_bucket_scratch);
        if (rc != cudaSuccess || !p) { set_error("nsl_bucket_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(rc)); return NULL; }
        ptr[dev] = (int32_t*) p;
    }
    return ptr[dev];
}

}   // namespace nsl

using namespace nsl;

extern "C" {

void nsl_route(cudaStream_t s, int n_exp, int top_k, const float* logits, int ld, int32_t* ind, float* wt, int T) {
    if (T <= 0) return;
    if (n_exp < 1 || n_exp > 32 * ROUTE_PER_LANE || top_k < 1 || top_k > 32 || top_k > n_exp) {
        set_error("router: %d experts (at most %d), top %d (at most 32)", n_exp, 32 * ROUTE_PER_LANE, top_k);
        return;
    }
    FollowScope follow;
    const dim3 grid((unsigned) (T + 3) / 4);
    if (n_exp <= 128) launch(route_kernel<4>, grid, 128, 0, s, n_exp, top_k, logits, ld, ind, wt, T);
    else if (n_exp <= 512) launch(route_kernel<16>, grid, 128, 0, s, n_exp, top_k, logits, ld, ind, wt, T);
    else launch(route_kernel<32>, grid, 128, 0, s, n_exp, top_k, logits, ld, ind, wt, T);
    count_launch();
}
void kq4_route_ld(cudaStream_t s, const void* cfg, const float* logits, int ld, int32_t* ind, float* wt, int T) {
    const int* c = (const int*) cfg;   // Qwen4Cfg: n_exp and top_k are its 22nd and 23rd ints
    nsl_route(s, c[21], c[22], logits, ld, ind, wt, T);
}
void kq4_route(cudaStream_t s, const void* cfg, const float* logits, int32_t* ind, float* wt, int T) {
    kq4_route_ld(s, cfg, logits, ((const int*) cfg)[21], ind, wt, T);
}

void kq4_moe_combine(cudaStream_t s, int d, int k, const float* D, const float* wt, const float* sh, const float* sg,
                     int sgld, float* out, int T) {
    if (T <= 0 || d <= 0) return;
    FollowScope follow;
    launch(q4_combine_kernel, dim3((unsigned) (d + 255) / 256, (unsigned) T), 256, 0, s, d, k, D, wt, sh, sg, sgld, out);
    count_launch();
}

void kc_swiglu(cudaStream_t s, const float* g, const float* u, float* a, int n) {
    if (n <= 0) return;
    const int blocks = (n + 255) / 256;
    swiglu_kernel<<<blocks < sm_count() * 16 ? blocks : sm_count() * 16, 256, 0, s>>>(g, u, a, n);
    count_launch();
}

// kc_swiglu with the result as packed bf16 (n even): what kc_mm_grouped_packed reads.
void nsl_swiglu_packed(cudaStream_t s, const float* g, const float* u, uint16_t* a, int n) {
    if (n <= 0) return;
    const int blocks = (n / 2 + 255) / 256;
    swiglu_packed_kernel<<<blocks < sm_count() * 16 ? blocks : sm_count() * 16, 256, 0, s>>>(g, u, a, n);
    count_launch();
}

void kc_moe_combine(cudaStream_t s, const float* D, const float* w, const float* shared, float* x, int d, int k, int T) {
    if (T <= 0 || d <= 0) return;
    moe_combine_kernel<<<dim3((unsigned) (d + 255) / 256, (unsigned) T), 256, 0, s>>>(D, w, shared, x, d, k);
    count_launch();
}

void kc_pack_input_bf16(cudaStream_t s, const float* x, uint16_t* y, size_t n) {
    if (!n) return;
    const size_t blocks = (n / 8 + 255) / 256 + 1;
    launch(pack_bf16_kernel, (unsigned) (blocks < (size_t) sm_count() * 16 ? blocks : (size_t) sm_count() * 16), 256, 0, s, x, y, n);
    count_launch();
}

void kc_bucket(cudaStream_t s, const int32_t* inds, int count, int n, int32_t* perm, MmTile* tiles, int32_t* ntiles) { nsl::bucket(s, inds, count, n, perm, tiles, ntiles, NULL); }

void nsl_bucket_noalloc(cudaStream_t s, const int32_t* inds, int count, int n, int32_t* perm, MmTile* tiles, int32_t* ntiles_out) {
    if (n < 1 || n > BUCKET_MAX_EXPERTS) {
        set_error("nsl_bucket_noalloc: %d experts, the built-in work array holds at most %d", n, BUCKET_MAX_EXPERTS);
        return;
    }
    int32_t* work = bucket_scratch_ptr();
    if (!work) return;
    // every entry the placement reads is rewritten by the count kernel, so nothing has to be cleared between calls
    launch(bucket_count_kernel, 1, 1024, 0, s, inds, count, n, work);
    launch(bucket_place_kernel, (unsigned) n, 1024, 0, s, inds, count, (const int32_t*) work, perm, tiles, (int32_t*) NULL);
    launch(bucket_publish_kernel, 1, 32, 0, s, (const int32_t*) work, ntiles_out);
    count_launch(3);
}

void kc_cache_admit(cudaStream_t s, const CachePool* p, int sl, const int32_t* inds, int count, int flags) {
    if (p->per_layer > CACHE_MAX_PER_LAYER) { set_error("expert cache: %d experts per layer, at most %d", p->per_layer, CACHE_MAX_PER_LAYER); return; }
    cache_admit_kernel<<<1, CACHE_MAX_PER_LAYER, 0, s>>>(*p, sl, inds, count, flags);
    count_launch();
}
void kc_cache_copy(cudaStream_t s, const CachePool* p, int blocks) {
    if (blocks < 1) blocks = 1;
    cache_copy_kernel<<<(unsigned) blocks, 512, 0, s>>>(*p);
    count_launch();
}

}   // extern "C"
