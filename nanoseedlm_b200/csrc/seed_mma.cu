// Dense seed products of a few rows (up to 32 a tile) on warp-level tensor instructions: the projections of a decode batch.
//
// Y[n][r] = sum_k W[r][k] X[n][k], weights expanded exactly and rounded to bf16, inputs bf16, f32 accumulation.
//
// What bounds it is the expansion (82 instructions a block of 8 weights, 47 of them on the half-rate logic pipe; alone in a loop
// 0.96 clk a block and SM), whatever the number of rows: so nothing else may cost instructions.  The weights never leave the
// registers: the A fragments of mma.sync.m16n8k16 are whole blocks, because the products' k index is free to be permuted as long
// as the inputs follow.  Lane (g, t) of a warp owns chunk 4 S + t (64 weights = one 16-byte load of seeds, one of coefficient
// words, 4 bytes of codes) of rows g and g + 8 of its tile; step j of super-step S multiplies block j of the four lanes' chunks:
// the block's weights {0..3} are the lane's k slots of the first MMA, {4..7} those of the second, and the B fragments of both
// are the 16 bytes of inputs at k = 64 (4 S + t) + 8 j.  A super-step (256 inputs a row) of inputs lies in shared memory as it
// lies in global memory but for an exclusive-or that spreads the lanes' 16-byte loads over the banks.  All of the tile's inputs
// are resident where they fit (8 rows of 2048: 32 KB), so that a warp runs through its rows without a barrier; else two buffers
// of whole super-steps take turns.
// The products of an expert layer do not come here: the pieces of a routed batch have any number of rows, each 32 of them would be
// expanded again, and a row's bits would depend on how many others its expert got.  (A form for few rows an expert was 8 % faster for
// 64 rows, top 10 of 512 experts, routed evenly, and 1.8 times slower where most rows went to a few experts: 231 / 127 us.)
#include "common.cuh"
#include "seed_block.cuh"
#include "seed_mma.cuh"

namespace nsl {

constexpr int SMM_THREADS = 256, SMM_WARPS = 8, SMM_SS = 256;      // inputs of a row per super-step
constexpr int SMM_TILE = 32;                                       // rows of inputs of a pass at most

struct SmmParams {
    MmParams m;
    int rw, kw;          // warps over rows, warps over K
    int per, bufs;       // steps of kw super-steps a buffer holds for `rows` rows of inputs, buffers
    int rows;
};

__device__ __forceinline__ void mma16816(float* c, uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

struct MmaChunk { uint4 s, c; uint32_t cd; };

template <int P>
__device__ __forceinline__ MmaChunk load_mma_chunk(const WSlice& w, uint32_t i) {
    MmaChunk k;
    k.s = __ldg((const uint4*) w.p[0] + i);
    k.c = __ldg((const uint4*) w.p[1] + i);
    k.cd = P == 4 ? __ldg((const uint32_t*) w.p[3] + i) : 0u;
    return k;
}

// Two blocks (an even one and its successor) of one row -> their bf16 pairs: f[0..3] of the even block, f[4..7] of the odd one.
template <int P>
__device__ __forceinline__ void pair_fragments(const StreamTab& tab, uint32_t sw, uint32_t cw, u64 e2, float base, const KConst& kc, uint32_t* f) {
    u64 w2[8];
    pair_weights<P>(tab, sw, cw, e2, base, kc, w2);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float a0, a1, b0, b1;
        unpack2(w2[2 * i], a0, b0);
        unpack2(w2[2 * i + 1], a1, b1);
        f[i] = bf16x2_bits(a0, a1);
        f[4 + i] = bf16x2_bits(b0, b1);
    }
}

// 16-byte unit u (k = 8 u .. 8 u + 7) of row n of a super-step's inputs: for one step j = u & 7 the eight lanes (two rows, four
// t = u >> 3) of a load phase fall into eight bank groups.
__device__ __forceinline__ int unit_at(int n, int u) { return n * 32 + ((u & 24) | ((u & 7) ^ ((u >> 3) | ((n & 1) << 2)))); }

struct SmmShared {
    StreamTab tab;
    int soff[SMM_TILE], drow[SMM_TILE];      // a row's inputs (offset in units of 16 bytes; -1: none), its place in the output
};

// One pass: up to 8 NT rows of inputs for this block's rows of weights.
// DEP: may be a dependent launch, whose inputs the kernel beside it may still be writing (common.cuh).
template <int NT, int P, bool DEP>
__device__ __forceinline__ void smm_pass(const SmmParams& sp, const KConst& kc, SmmShared& sh, unsigned char* xs, int r0) {
    const MmParams& a = sp.m;
    const int kw = sp.kw, rw = sp.rw;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int kg = warp / rw, rg = warp - kg * rw;             // the warp's share of K and of the block's rows
    const int ch = a.K / 64, nss = (ch + 3) / 4, iters = (nss + kw - 1) / kw;
    const int rowA = r0 + rg * 16 + g, rowB = rowA + 8;
    const WSlice& w = a.w0;
    const bool okA = rowA < a.R, okB = rowB < a.R;
    constexpr int SS_BYTES = NT * 8 * 512;
    const int per = sp.per * (sp.rows / 8) / NT;      // a buffer holds more steps of fewer rows
    const uint32_t buf_bytes = (uint32_t) (per * kw * SS_BYTES);
    const float base = exact_base<P>(w.eb);
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.0f;

    // Staging: this thread's unit u of rows tid / 32, + 8, ...; rows beyond the count and inputs beyond K are zeros (a copy of
    // size 0).
    const int u = tid & 31, n_lo = tid >> 5;
    const uint32_t xs32 = (uint32_t) __cvta_generic_to_shared(xs);
    auto stage = [&](int it0, int buf) {      // the steps it0 .. it0 + per - 1
        for (int q = 0; q < per * kw && it0 * kw + q < nss; ++q) {
            const int k = (it0 * kw + q) * SMM_SS + 8 * u;
            const bool kok = k < a.K;
            const uint32_t dst = xs32 + (uint32_t) buf * buf_bytes + (uint32_t) (q * SS_BYTES + unit_at(n_lo, u) * 16);      // (n_lo and n_lo + 8 i share the swizzle)
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const int so = sh.soff[n_lo + 8 * i];
                const bool ok = kok && so >= 0;
                if (a.packed) {
                    const uint16_t* src = (const uint16_t*) a.X + ((size_t) (uint32_t) (ok ? so : 0) * 8 + (ok ? k : 0));
                    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst + i * 4096), "l"(src), "r"(ok ? 16 : 0) : "memory");
                } else {
                    uint4 o = make_uint4(0u, 0u, 0u, 0u);
                    if (ok) {
                        const float4* xp = (const float4*) ((const float*) a.X + ((size_t) (uint32_t) so * 4 + k));
                        const float4 x0 = DEP ? xp[0] : __ldg(xp), x1 = DEP ? xp[1] : __ldg(xp + 1);
                        o = make_uint4(bf16x2_bits(x0.x, x0.y), bf16x2_bits(x0.z, x0.w), bf16x2_bits(x1.x, x1.y), bf16x2_bits(x1.z, x1.w));
                    }
                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + i * 4096), "r"(o.x), "r"(o.y), "r"(o.z), "r"(o.w) : "memory");
                }
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    auto chunk_ok = [&](int it) { return it < iters && (it * kw + kg) * 4 + t < ch; };
    auto load = [&](int it, MmaChunk& ca, MmaChunk& cb) {      // (a chunk that is not there stays zero: zero coefficients, zero weights)
        const int c = (it * kw + kg) * 4 + t;
        if (okA) ca = load_mma_chunk<P>(w, (uint32_t) (rowA * ch + c));
        if (okB) cb = load_mma_chunk<P>(w, (uint32_t) (rowB * ch + c));
    };
    MmaChunk ca = {}, cb = {};
    if (chunk_ok(0)) load(0, ca, cb);
    stage(0, 0);
    int in_buf = 0, buf = 0;      // the step's place in its buffer
    for (int it = 0; it < iters; ++it) {
        MmaChunk na = {}, nb = {};
        if (chunk_ok(it + 1)) load(it + 1, na, nb);
        if (in_buf == 0) {      // a new buffer: its inputs are there; the other one's are requested
            if (sp.bufs == 2 && it + per < iters) {
                stage(it + per, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
        }
        // the lane's unit of step 0: row g, chunk t (128-byte aligned), the swizzle in bits 4..6; step j is an exclusive-or away
        const uint32_t xb = xs32 + (uint32_t) buf * buf_bytes + (uint32_t) ((in_buf * kw + kg) * SS_BYTES + (g * 32 + t * 8) * 16) + (uint32_t) ((t | ((g & 1) << 2)) << 4);
        const uint32_t sA[4] = {ca.s.x, ca.s.y, ca.s.z, ca.s.w}, cA[4] = {ca.c.x, ca.c.y, ca.c.z, ca.c.w};
        const uint32_t sB[4] = {cb.s.x, cb.s.y, cb.s.z, cb.s.w}, cB[4] = {cb.c.x, cb.c.y, cb.c.z, cb.c.w};
        if ((it * kw + kg) * 4 < ch) {      // (warp-uniform)
#pragma unroll
            for (int jj = 0; jj < 4; ++jj) {
                uint32_t fa[8], fb[8];
                pair_fragments<P>(sh.tab, sA[jj], cA[jj], P == 4 ? code_scale_pair(ca.cd, jj, kc) : code_scale_pair3(cA[jj], kc), base, kc, fa);
                pair_fragments<P>(sh.tab, sB[jj], cB[jj], P == 4 ? code_scale_pair(cb.cd, jj, kc) : code_scale_pair3(cB[jj], kc), base, kc, fb);
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const uint32_t at = xb ^ (uint32_t) ((2 * jj + e) << 4);
#pragma unroll
                    for (int i = 0; i < NT; ++i) {
                        uint4 x;
                        asm volatile("ld.shared.v4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(x.x), "=r"(x.y), "=r"(x.z), "=r"(x.w) : "r"(at + i * 4096));
                        mma16816(acc[i], fa[4 * e], fb[4 * e], fa[4 * e + 1], fb[4 * e + 1], x.x, x.y);
                        mma16816(acc[i], fa[4 * e + 2], fb[4 * e + 2], fa[4 * e + 3], fb[4 * e + 3], x.z, x.w);
                    }
                }
            }
        }
        ca = na;
        cb = nb;
        if (++in_buf == per && it + 1 < iters) {
            in_buf = 0;
            __syncthreads();      // this buffer's reads are done
            if (sp.bufs == 2) buf ^= 1;
            else stage(it + 1, 0);
        }
    }
    if (kw > 1) {      // the K shares' sums meet in shared memory, added in order by the first share's warps
        __syncthreads();
        float* part = (float*) xs;
        if (kg > 0) {
#pragma unroll
            for (int i = 0; i < NT; ++i) *(float4*) (part + ((((kg - 1) * rw + rg) * NT + i) * 32 + lane) * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        }
        __syncthreads();
        if (kg > 0) return;
        for (int q = 1; q < kw; ++q)
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                const float4 v = *(const float4*) (part + ((((q - 1) * rw + rg) * NT + i) * 32 + lane) * 4);
                acc[i][0] += v.x; acc[i][1] += v.y; acc[i][2] += v.z; acc[i][3] += v.w;
            }
    }
    // lane (g, t): rows 8 i + 2 t and + 1 of the inputs (elements 0, 1 of weight row A; 2, 3 of row B)
#pragma unroll
    for (int i = 0; i < NT; ++i) {
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int dst = sh.drow[8 * i + 2 * t + e];
            const float va = acc[i][e], vb = acc[i][2 + e];
            if (dst < 0) continue;
            float* y = (float*) a.Y + (size_t) dst * a.ys;
            if (okA) y[rowA] = a.add ? bf16_round(y[rowA] + bf16_round(va)) : bf16_round(va);   // engine/kernels_moe.cu:214
            if (okB) y[rowB] = a.add ? bf16_round(y[rowB] + bf16_round(vb)) : bf16_round(vb);
        }
    }
}

// 128 registers: the pass of 32 rows spills some (P = 4 84 / 144 bytes of stores / loads, 72 / 112 without DEP; P = 3 8 / 12).
template <int P, bool DEP>
__global__ void __launch_bounds__(SMM_THREADS, 2) seed_mma_kernel(SmmParams sp, KConst kc) {
    extern __shared__ __align__(128) unsigned char smm_smem[];
    __shared__ SmmShared sh;
    const MmParams& a = sp.m;
    const int tid = threadIdx.x;
    if (DEP) tab_and_wait(sh.tab, a.G, a.late, tid, SMM_THREADS, !a.late);
    else load_stream_tab(sh.tab, a.G, tid, SMM_THREADS);
    const int start = (int) blockIdx.y * SMM_TILE, count = min(a.T - start, SMM_TILE), r0 = (int) blockIdx.x * sp.rw * 16;
    if (tid < SMM_TILE) {
        const int d = tid >= count ? -1 : start + tid;
        sh.soff[tid] = d < 0 ? -1 : (int) ((long long) d * a.xs / (a.packed ? 8 : 4));
        sh.drow[tid] = d;
    }
    __syncthreads();
    if (count <= 8) smm_pass<1, P, DEP>(sp, kc, sh, smm_smem, r0);
    else if (count <= 16) smm_pass<2, P, DEP>(sp, kc, sh, smm_smem, r0);
    else smm_pass<4, P, DEP>(sp, kc, sh, smm_smem, r0);
}

template <int P, bool DEP>
static void launch_smm_v(cudaStream_t s, const SmmParams& a, dim3 grid, size_t smem) {
    static bool done[16];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!done[dev & 15]) {
        cudaFuncSetAttribute(seed_mma_kernel<P, DEP>, cudaFuncAttributeMaxDynamicSharedMemorySize, max_smem_optin() - 8192);
        done[dev & 15] = true;
    }
    launch(seed_mma_kernel<P, DEP>, grid, SMM_THREADS, smem, s, a, kconst());
    count_launch();
}

bool smm_serves(int K, const void* X, int xs, int packed) {
    return K >= 64 && K % 64 == 0 && aligned16(X) && xs % (packed ? 8 : 4) == 0;
}

void launch_seed_mma(cudaStream_t s, int fmt, const MmParams& m) {
    if (m.T <= 0 || m.R <= 0) return;
    SmmParams a = {m, SMM_WARPS, 1, 1, 2, SMM_TILE};
    // 16 rows of weights a warp leave most SMs idle on a matrix of a few thousand rows, so the block's warps share K until the
    // blocks fill the SMs (a function of the matrix alone).
    while (a.kw < 8 && (m.R + 16 * SMM_WARPS / a.kw - 1) / (16 * SMM_WARPS / a.kw) < sm_count() * 3 / 4 && m.K >= SMM_SS * 2 * a.kw) a.kw *= 2;
    a.rw = SMM_WARPS / a.kw;
    // All of K in one buffer where two blocks of that size fit an SM, else two buffers of 48 KB, else (K shared by many warps) one
    // step at a time.  The sizes are those of the most rows a tile may have; fewer rows make a buffer hold more steps.
    a.rows = m.T > 16 ? 32 : m.T > 8 ? 16 : 8;
    const size_t step = (size_t) a.kw * a.rows * 512, room = 96 * 1024;
    const int iters = (m.K + SMM_SS * a.kw - 1) / (SMM_SS * a.kw);
    if ((size_t) iters * step <= room) { a.per = iters; a.bufs = 1; }
    else if (2 * step <= room) a.per = (int) (room / 2 / step);
    else a.bufs = 1;
    size_t smem = (size_t) a.bufs * a.per * step;
    const size_t red = (size_t) (a.kw - 1) * a.rw * (a.rows / 8) * 512;
    if (red > smem) smem = red;
    const int wrows = a.rw * 16;
    const dim3 grid((unsigned) ((m.R + wrows - 1) / wrows), (unsigned) ((m.T + SMM_TILE - 1) / SMM_TILE));
    // Blocks of two calls beside one another leave some SMs with two and others with none, and a grid of long and short tiles of rows is dealt unevenly
    // wherever it comes in behind another kernel.  So where kc_mm chose a dependent launch itself, the next kernel's blocks come in when this one ends,
    // and the choice falls only where the blocks are alike or each has an SM of its own.  us, calls one behind the other, ordinary / dependent with the
    // next call's blocks let in at once / now: 17858 x 2880, 9 rows 45.1 / 71.0 / 41.9; 8192 x 4096, 48 rows 61.7 / 69.7 / 60.2; 22888 x 768, 35 rows
    // 31.0 / 34.4 / 31.0; 1138 x 512, 11 rows 6.5 / 6.1 / 6.1.  (In a decoder's chain, whose kernels differ, letting them in at once is no slower.)
    const bool even = grid.y == 1 || (long long) grid.x * grid.y <= sm_count();
    if (even || !m.late) {
        if (fmt == MF_SEED4) launch_smm_v<3, true>(s, a, grid, smem);
        else launch_smm_v<4, true>(s, a, grid, smem);
    } else {
        PdlScope off(false);
        if (fmt == MF_SEED4) launch_smm_v<3, false>(s, a, grid, smem);
        else launch_smm_v<4, false>(s, a, grid, smem);
    }
}

}   // namespace nsl
