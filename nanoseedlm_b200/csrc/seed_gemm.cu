// Prompt-row GEMM over seed weights on the 5th-generation tensor cores (tcgen05 + TMEM), dense and grouped by expert.
// Replaces the SEED4P4 paths of the reference's k_mm / k_mm3 / k_mm_packed and their grouped forms
// (engine/kernels_moe.cu:405-525, 2354-2395), which stage one 64 x 32 weight tile per K step for mma.sync.
//
// Y[n][r] = sum_k W[r][k] X[n][k] for a unit of 128 weight rows x up to 128 rows of inputs (one entry of the tile table: one
// expert's run of pairs, or 128 consecutive rows of a dense call), or up to 384 of one expert or dense call.
//
// The expansion is the cost (82 instructions per 8 weights, 0.96 clk a block of weights and SM alone in a loop, against
// 2 x 8 x N flops of tensor work), so the weights are written where the MMA reads them with the fewest instructions: tensor
// memory.  A producer thread owns one row (its tensor memory lane) and the 64 weights of a K step: 8 blocks from one 16-byte load
// of seeds, one of coefficient words and 4 bytes of codes, converted to bf16 pairs and stored by two tcgen05.st; no address
// arithmetic, no swizzle, no proxy fence.  The four warps of a warpgroup make a step; the warpgroups take the steps in turn, so
// a step waits for one warp of each scheduler (eight warps a step left the producers waiting for one another a third of the
// time).  The inputs (B operand) come through shared memory (128-byte swizzle), fetched by loader warps; one elected thread
// issues tcgen05.mma (M 128, K 16, N = the tile's count rounded up to 16) and commits the stage back through an mbarrier.
// Blocks are persistent: the stream table, the tensor memory and the barriers are set up once.
//   TT = 1, packed inputs: 8 producer warps, two blocks an SM (256 of the 512 columns each).
//   dense f32 inputs, K a multiple of 64, streams 8-byte aligned, two or three tiles or at most a unit an SM: 8 producer warps and 11 or 15
//   loaders, one block an SM (launch_dense_f32).
//   otherwise: 16 producer warps, one block an SM (three terms: 8).  TT = 3: up to three tiles of an expert share one expansion, which a prompt of
//   thousands of rows needs (each tile expands its expert's weights again).
// The accumulator is read back with tcgen05.ld by the producer warps (lane = weight row, column = row of inputs), rounded as the
// reference's store_y does and written so that a warp stores 32 consecutive rows of one row of outputs: after each warpgroup's
// first step of the next unit, under which the last MMAs run.  Units that fill at most half of the accumulator columns alternate
// between the halves, so the next unit's MMAs need not wait for that.
// Gate + up + SwiGLU (GU): lane 2 i holds row i of the gate matrix, lane 2 i + 1 of the up matrix, so both sums meet in
// neighbouring lanes and the result leaves as packed bf16: no f32 intermediates, no third kernel.
//
// Weight precision: default, seed weights rounded to bf16 (one term); kc_seed_gemm_f32(1), three bf16 terms whose sum is
// the f32 weight exactly (three MMAs per step), as the reference's two modes (engine/kernels_moe.cu:405-412).
//
// Every wait on an mbarrier is bounded: after the limit the block records a status word, stops issuing work, lets its copies and MMAs in
// flight end, frees its TMEM and returns.
#include <cuda.h>

#include <type_traits>

#include "common.cuh"
#include "seed_block.cuh"
#include "seed_mma.cuh"

namespace nsl {

constexpr int GM_BM = 128, GM_BN = 128, GM_BK = 64, GM_STAGES = 4;
constexpr int GM_MAX_HEADS = 2048;      // tiles of a launch whose experts' tiles share expansions (their list sits in shared memory)
constexpr uint32_t GM_WAIT_LIMIT = 1u << 24;
constexpr unsigned long long GM_WAIT_NS = 1000000000ull;
// How the inputs reach shared memory.  IN_LIST: packed rows picked by a list (cp.async by the loader warps); IN_F32: f32 rows,
// converted by the loaders, whose loads of a whole K step are held in registers meanwhile (IN_F32_FEW: grouped, units of any number of
// rows up to a tile); IN_TMA: packed rows that follow one
// another (dense, or sorted by expert), by one thread.  IN_F32_DENSE: as IN_F32, with more loaders than producers.
enum { IN_LIST = 0, IN_F32 = 1, IN_TMA = 2, IN_F32_FEW = 3, IN_F32_DENSE = 4 };
// One block: PW producer warps, the MMA warp, LW loader warps.  Tensor memory: the accumulators (128 columns per tile of inputs),
// then the stages' weights (32 columns per term: 64 k values as bf16 pairs).
// LAUNCH_REGS: registers a thread at launch (what the launch bounds leave); PREGS, LREGS: of the producers' and of the other
// warpgroups after the split, whose sum over the block is at most what the launch gave it.
template <int TERMS, int TT, int IN>
struct GmCfg {
    static constexpr bool DENSE = IN == IN_F32_DENSE, F32 = IN == IN_F32 || IN == IN_F32_FEW || DENSE;
    static constexpr int CTAS = TERMS == 1 && TT == 1 && !F32 ? 2 : 1, PW = TERMS == 3 || CTAS == 2 || DENSE ? 8 : 16;
    static constexpr int LW = DENSE ? (TT == 1 ? 11 : 15) : TERMS == 1 && F32 ? 7 : 3;
    static constexpr int WARPS = PW + 1 + LW, THREADS = WARPS * 32, GROUPS = PW / 4;
    static constexpr int ACC = GM_BN * TT, A_COLS = 32 * TERMS, COLS = ACC + GM_STAGES * A_COLS <= 256 ? 256 : 512;
    static constexpr int X_BYTES = TT * GM_BN * GM_BK * 2;      // a stage's inputs
    static constexpr bool SPLIT = TERMS == 1;
    static constexpr int LAUNCH_REGS = CTAS == 1 && WARPS == 20 ? 96 : 80, LREGS = F32 ? 64 : 40, PREGS = DENSE ? 112 : F32 ? 88 : LAUNCH_REGS == 96 ? 104 : 96;
    static_assert(ACC + GM_STAGES * A_COLS <= COLS && CTAS * COLS <= 512, "tensor memory");
    static_assert(!SPLIT || PW * PREGS + (LW + 1) * LREGS <= WARPS * LAUNCH_REGS, "registers");
    static_assert(GM_STAGES >= GROUPS, "every warpgroup owns a stage");
};

// The inputs' tensor map, a parameter of the kernels that use one.
struct NoMap {};
template <int IN>
using GmMap = typename std::conditional<IN == IN_TMA, CUtensorMap, NoMap>::type;

__device__ int g_mm_status;   // 0, or the code of the first bounded wait that ran out

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t) __cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count));
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
// Bounded wait: false after GM_WAIT_NS or GM_WAIT_LIMIT attempts (the caller records the code and stops).  The suspended form: a warp that polls
// takes issue slots from the producers (bare polls with short sleeps: 343 us a config-2 layer, this: 328; long sleeps wake too
// late: 376).
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
    unsigned long long t0 = 0;
    for (uint32_t i = 0; i < GM_WAIT_LIMIT; ++i) {
        if (mbar_try(bar, parity)) return true;
        if ((i & 63u) == 63u) {
            unsigned long long t;
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (!t0) t0 = t;
            if (*abort_flag || t - t0 > GM_WAIT_NS) return false;
        }
    }
    return false;
}

__device__ __forceinline__ uint64_t umma_desc(uint32_t saddr) {
    // K-major operand tile, 128-byte swizzle: start address >> 4; leading byte offset (unused with swizzle) 1;
    // stride byte offset 1024 (8 rows of 128 bytes) >> 4; descriptor version 1; layout type 2 = SWIZZLE_128B
    return (uint64_t) ((saddr & 0x3FFFFu) >> 4) | ((uint64_t) 1 << 16) | ((uint64_t) (1024 >> 4) << 32) | ((uint64_t) 1 << 46) |
           ((uint64_t) 2 << 61);
}
__device__ __forceinline__ uint32_t umma_idesc(int n) {
    // D f32 (bits 4-5 = 1), A and B bf16 (bits 7-9, 10-12 = 1), both K-major, N >> 3 at bit 17, M >> 4 at bit 24
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t) (n >> 3) << 17) | ((uint32_t) (GM_BM >> 4) << 24);
}
__device__ __forceinline__ void umma_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t* v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
                   "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
                 : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// tcgen05.mma with the weights (A) in tensor memory and the inputs (B) in shared memory.
__device__ __forceinline__ void umma_ts(uint32_t tmem_d, uint32_t tmem_a, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
                 ::"r"(tmem_d), "r"(tmem_a), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                   "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}

// A thread's share of one K step: the 8 blocks (64 weights) of its row.
struct ChunkIn { uint4 s, c; uint32_t cd; };

// VEC, how the streams may be read.  2: rows of whole chunks, streams aligned to 16, 16 and 4 bytes (stream_wide).  1: rows of whole half
// chunks (K a multiple of 32), streams aligned to 8, 8 and 2 bytes.  0: anything.
template <bool P3>
__device__ __forceinline__ bool stream_wide(const WSlice& w) {
    return (((unsigned long long) w.p[0] | (unsigned long long) w.p[1]) & 15ull) == 0 && (P3 || ((unsigned long long) w.p[3] & 3ull) == 0);
}
template <bool P3, int VEC>
__device__ __forceinline__ ChunkIn load_row_chunk(const WSlice& w, int row, int chunk, int R, int NB) {
    ChunkIn q = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u), 0u};      // zero coefficients: zero weights
    if (row >= R || chunk * 8 >= NB) return q;
    if (VEC == 2) {
        const uint32_t i = (uint32_t) row * (uint32_t) (NB / 8) + (uint32_t) chunk;
        q.s = __ldg((const uint4*) w.p[0] + i);
        q.c = __ldg((const uint4*) w.p[1] + i);
        if (!P3) q.cd = __ldg((const uint32_t*) w.p[3] + i);
    } else if (VEC) {
        const size_t i = ((size_t) row * NB + chunk * 8) / 4;      // the chunk's first half
        const uint2 s0 = __ldg((const uint2*) w.p[0] + i), c0 = __ldg((const uint2*) w.p[1] + i);
        uint2 s1 = make_uint2(0u, 0u), c1 = s1;
        if (!P3) q.cd = __ldg((const uint16_t*) w.p[3] + i);
        if (chunk * 8 + 4 < NB) {
            s1 = __ldg((const uint2*) w.p[0] + i + 1);
            c1 = __ldg((const uint2*) w.p[1] + i + 1);
            if (!P3) q.cd |= (uint32_t) __ldg((const uint16_t*) w.p[3] + i + 1) << 16;
        }
        q.s = make_uint4(s0.x, s0.y, s1.x, s1.y);
        q.c = make_uint4(c0.x, c0.y, c1.x, c1.y);
    } else {
        uint32_t sw[4] = {0u, 0u, 0u, 0u}, cw[4] = {0u, 0u, 0u, 0u};
        const size_t g = (size_t) row * NB + chunk * 8;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            if (chunk * 8 + j >= NB) break;
            sw[j >> 1] |= (uint32_t) __ldg((const uint16_t*) w.p[0] + g + j) << (16 * (j & 1));
            cw[j >> 1] |= (uint32_t) __ldg((const uint16_t*) w.p[1] + g + j) << (16 * (j & 1));
            if (!P3) q.cd |= (uint32_t) ((__ldg((const uint8_t*) w.p[3] + ((g + j) >> 1)) >> (((g + j) & 1) * 4)) & 15) << (4 * j);
        }
        q.s = make_uint4(sw[0], sw[1], sw[2], sw[3]);
        q.c = make_uint4(cw[0], cw[1], cw[2], cw[3]);
    }
    return q;
}

// Where a unit of work lies: 128 rows of weights x up to TT consecutive tiles of one slice.
struct UnitPos { WSlice wa, wb; int start, count, r0; };

// heads: the tiles that start a unit (TT > 1, grouped); otherwise every tile does.
template <int TT, bool GU>
__device__ __forceinline__ UnitPos unit_pos(const MmParams& a, int unit, int row_tiles, const uint16_t* heads) {
    UnitPos u;
    const int y = unit / row_tiles, x = unit - y * row_tiles;
    u.r0 = x * (GU ? GM_BM / 2 : GM_BM);
    if (a.grouped) {
        const MmTile tl = a.tiles[TT > 1 ? heads[y] : y];
        u.start = tl.start;
        u.count = TT > 1 ? min(a.offs[tl.slice + 1] - tl.start, GM_BN * TT) : min(tl.count, GM_BN);
        u.wa = a.ws[tl.slice];
        u.wb = GU ? a.wu[tl.slice] : u.wa;
    } else {
        u.start = y * GM_BN * TT;
        u.count = min(a.T - u.start, GM_BN * TT);
        u.wa = a.w0;
        u.wb = a.w0;
    }
    return u;
}
__device__ __forceinline__ int input_row_of(const MmParams& a, const UnitPos& u, int n) {      // rows beyond the count repeat the last one
    const int p = u.start + min(n, u.count - 1);
    return a.grouped ? a.perm[p] / a.xdiv : p;
}
// 16-byte unit uu (8 inputs) of row n of a stage: 128-byte swizzle.
__device__ __forceinline__ uint32_t input_at(uint32_t stage, int n, int uu) {
    return stage + (uint32_t) (n * 128 + ((uu ^ (n & 7)) << 4));
}

// 1 / (1 + e^-g).  The hardware's reciprocal and one Newton-Raphson step r + r (1 - d r): for every bf16 g above -87.3 the division's
// value.  Below, the result is subnormal, which the approximation flushes to zero, or e^-g is infinite: largest collects the denominators,
// so that the caller can go back and divide.
template <bool DIVIDE>
__device__ __forceinline__ float sigmoid(float g, float& largest) {
    const float d = 1.0f + expf(-g);
    if (DIVIDE) return 1.0f / d;
    largest = fmaxf(largest, d);
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(d));
    return fmaf(r, fmaf(-d, r, 1.0f), r);
}

__device__ __forceinline__ uint32_t mul_bf16x2(uint32_t a, uint32_t b) {      // each product rounded once
    uint32_t d;
    asm("mul.rn.bf16x2 %0, %1, %2;" : "=r"(d) : "r"(a), "r"(b));
    return d;
}

// SwiGLU of 16 columns of a warp: two = bf16 pairs of the gate's (even lanes) and the up matrix's (odd lanes) sums, two columns a word.
// Even lanes finish columns 0..7, odd lanes 8..15, into the warp's box at `at`.  Returns the largest denominator.
template <bool DIVIDE, int ROWS>
__device__ __forceinline__ float swiglu_columns(const uint32_t* two, bool odd, uint16_t* at) {
    float largest = 0.0f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const uint32_t mine = odd ? two[j + 4] : two[j], from = __shfl_xor_sync(0xFFFFFFFFu, odd ? two[j] : two[j + 4], 1);
        const uint32_t g = odd ? from : mine, up = odd ? mine : from;
        const uint32_t sg = bf16x2_bits(sigmoid<DIVIDE>(__uint_as_float(g << 16), largest), sigmoid<DIVIDE>(__uint_as_float(g & 0xFFFF0000u), largest));
        const uint32_t o = mul_bf16x2(mul_bf16x2(g, sg), up);
        at[2 * j * ROWS] = (uint16_t) o;
        at[(2 * j + 1) * ROWS] = (uint16_t) (o >> 16);
    }
    return largest;
}
template <int ROWS>
__device__ __noinline__ void swiglu_columns_divide(uint4 a, uint4 b, bool odd, uint16_t* at) {
    const uint32_t two[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
    swiglu_columns<true, ROWS>(two, odd, at);
}

// The results of a unit, by the producer warps: warp w reads the tensor memory lanes of its quarter, 16 columns at a time, the
// warpgroups taking turns.  col: the unit's first column.  bf16 results are turned round in 1 KB of shared memory a warp (box), so
// that a lane stores 16 bytes of one row of outputs: with 2-byte stores straight from the registers the results of a 256-row unit
// took 8400 clk, a quarter of its expansion.  No MMA of the next unit runs meanwhile where a unit fills the accumulators, so the
// instructions count: two columns at a time from the first rounding on (SwiGLU column by column: 6000 clk a unit), the places of
// the next columns' rows requested ahead (AHEAD).
template <bool GU, int GROUPS, bool AHEAD>
__device__ __forceinline__ void unit_results(const MmParams& a, uint32_t tmem, uint16_t* box, int col, int start, int count, int r0) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, lq = warp & 3;
    constexpr int ROWS = GU ? 16 : 32;      // rows of outputs' values a warp makes of its 32 lanes
    const int row0 = r0 + lq * ROWS;
    auto place = [&](int c0) {      // lane j: column c0 + j's row of outputs
        const int p = start + min(c0 + (lane & 15), count - 1);
        return a.grouped && !a.out_sorted ? a.perm[p] : p;
    };
    int dst_next = AHEAD ? place((warp >> 2) * 16) : 0;
    for (int c0 = (warp >> 2) * 16; c0 < count; c0 += GROUPS * 16) {
        uint32_t v[16];
        const int dst_lane = AHEAD ? dst_next : place(c0);
        tmem_ld16(tmem + ((uint32_t) (lq * 32) << 16) + (uint32_t) (col + c0), v);
        if (AHEAD) dst_next = place(c0 + GROUPS * 16);
        if (GU || a.out_bf16) {      // (R and ys are multiples of 8 here)
            uint32_t two[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) two[j] = bf16x2_bits(__uint_as_float(v[2 * j]), __uint_as_float(v[2 * j + 1]));
            if (GU) {
                const bool odd = lane & 1;
                uint16_t* const at = box + (odd ? 8 * ROWS : 0) + (lane >> 1);      // even lanes finish columns 0..7, odd lanes 8..15
                if (__any_sync(0xFFFFFFFFu, swiglu_columns<false, ROWS>(two, odd, at) > 8e37f))      // (rare: out of line; a branch at every value cost a layer 1024 / 1024 wide 5 %)
                    swiglu_columns_divide<ROWS>(make_uint4(two[0], two[1], two[2], two[3]), make_uint4(two[4], two[5], two[6], two[7]), odd, at);
            } else {
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    box[2 * j * ROWS + lane] = (uint16_t) two[j];
                    box[(2 * j + 1) * ROWS + lane] = (uint16_t) (two[j] >> 16);
                }
            }
            __syncwarp();
#pragma unroll
            for (int i = 0; i < ROWS / 16; ++i) {      // the lane's 8 rows of column c
                const int e = lane + 32 * i, c = e / (ROWS / 8), r = row0 + (e % (ROWS / 8)) * 8;
                const int dst = __shfl_sync(0xFFFFFFFFu, dst_lane, c);
                if (c0 + c < count && r + 8 <= a.R) *(uint4*) ((uint16_t*) a.Y + (size_t) dst * a.ys + r) = *(const uint4*) (box + e * 8);
            }
            __syncwarp();
        } else {
            const int grow = row0 + lane;
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const int dst = __shfl_sync(0xFFFFFFFFu, dst_lane, j);
                if (c0 + j >= count || grow >= a.R) continue;
                const float acc = __uint_as_float(v[j]);
                float* yo = (float*) a.Y + (size_t) dst * a.ys + grow;
                *yo = a.add ? bf16_round(*yo + bf16_round(acc)) : bf16_round(acc);   // engine/kernels_moe.cu:214
            }
        }
    }
}

// WF: the weights' form.  0: SEED4P4 blocks; 1: stored BF16 values; 2: SEED4 (P = 3) blocks.  TERMS: bf16 terms a weight (1, or 3:
// exact).  TT: tiles of 128 rows of inputs that share one expansion.  VEC: how the streams are read (load_row_chunk; 2: slices that are not
// aligned for it as 1).
// GU: gate + up + SwiGLU; row i of the gate matrix on lane 2 i, of the up matrix on lane 2 i + 1.
template <int TERMS, int WF, int TT, int VEC, bool GU, int IN>
__global__ void __launch_bounds__(GmCfg<TERMS, TT, IN>::THREADS, GmCfg<TERMS, TT, IN>::CTAS) seed_gemm_kernel(MmParams a, KConst kc, const __grid_constant__ GmMap<IN> tm) {
    using Cfg = GmCfg<TERMS, TT, IN>;
    constexpr bool F32 = Cfg::F32, FEW = IN == IN_F32_FEW;
    constexpr bool BF16W = WF == 1, P3 = WF == 2;
    constexpr int PW = Cfg::PW, GROUPS = Cfg::GROUPS, HALF = Cfg::ACC / 2;
    extern __shared__ uint8_t smem_raw[];
    __shared__ StreamTab tab;
    __shared__ __align__(8) uint64_t bars[2 * GM_STAGES + 3];
    __shared__ uint32_t tmem_slot;
    __shared__ int srow[FEW ? Cfg::LW * 20 : GM_BN * TT];      // the unit's rows of inputs (FEW: 20 places a warp)
    __shared__ int abort_flag, n_heads;
    __shared__ uint16_t heads[TT > 1 ? GM_MAX_HEADS : 1];

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    uint16_t* const box = (uint16_t*) (((uintptr_t) smem_raw + 1023) & ~(uintptr_t) 1023) + GM_STAGES * Cfg::X_BYTES / 2;      // 1 KB a producer warp
    const uint32_t smem_base = smem_u32((uint8_t*) (((uintptr_t) smem_raw + 1023) & ~(uintptr_t) 1023));
    const uint32_t bar_full = smem_u32(&bars[0]), bar_empty = bar_full + 8 * GM_STAGES, bar_done = bar_empty + 8 * GM_STAGES, bar_read = bar_done + 8;
    if (!BF16W && !a.late) load_stream_tab(tab, a.G, tid, Cfg::THREADS);
    if (tid == 0) {
        abort_flag = 0;
        for (int s = 0; s < GM_STAGES; ++s) {
            mbar_init(bar_full + 8 * s, 4 + (IN == IN_TMA ? 1 : Cfg::LW));      // one arrival per warp of the stage's warpgroup and per loader
            mbar_init(bar_empty + 8 * s, 1);
        }
        mbar_init(bar_done, 1);                            // a unit's MMAs are done
        mbar_init(bar_read, PW);                           // the results in a half of the accumulators have been read
        mbar_init(bar_read + 8, PW);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == PW) {   // the MMA warp owns the tensor memory
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(Cfg::COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    grid_dependents_go();
    grid_dependency_wait();
    if (!BF16W && a.late) load_stream_tab(tab, a.G, tid, Cfg::THREADS);
    if (TT > 1 && a.grouped && warp == 0) {      // the tiles that start a unit: every TT-th of a slice, in order
        const int nt = a.ntiles ? *a.ntiles : a.T;
        int n = 0;
        for (int y0 = 0; y0 < nt; y0 += 32) {
            const int y = y0 + lane;
            bool head = false;
            if (y < nt) { const MmTile tl = a.tiles[y]; head = ((tl.start - a.offs[tl.slice]) / GM_BN) % TT == 0; }
            const uint32_t m = __ballot_sync(0xFFFFFFFFu, head);
            if (head) heads[n + __popc(m & ((1u << lane) - 1u))] = (uint16_t) y;
            n += __popc(m);
        }
        if (lane == 0) n_heads = n;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = tmem_slot, tmem_w = tmem + Cfg::ACC;
    const int NB = a.K / 8, KT = (a.K + GM_BK - 1) / GM_BK, rows_u = GU ? GM_BM / 2 : GM_BM;
    const int row_tiles = (a.R + rows_u - 1) / rows_u;
    const int n_units = row_tiles * (a.grouped ? (TT > 1 ? n_heads : a.ntiles ? *a.ntiles : a.T) : (a.T + GM_BN * TT - 1) / (GM_BN * TT));
    // Units of up to half_max rows alternate between the accumulators' halves.  Their MMAs do not wait for the previous unit's results to
    // be read, so every warpgroup must still owe a step of unit u + 1 when it waits for unit u's MMAs (bar_done: two phases are told
    // apart, a third would look like the first): results(u) follows its first step of u + 1, so it needs a second one.  With fewer
    // steps every unit takes both halves, whose MMAs wait for the readers.
    const int half_max = KT < 2 * GROUPS ? 0 : HALF;
    // Every role walks the same units and counts the same K steps (kr: its stage and the stage's phase) and units.
    int kr0 = 0, unit_run = 0;
    bool ok = true;
    auto fail = [&](int code) { abort_flag = 1; atomicCAS(&g_mm_status, 0, code); ok = false; };

    if (warp < PW) {
        if (Cfg::SPLIT) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::PREGS));
        // ---- producers: thread = one row's 64 weights of a K step; warpgroup g makes the steps with kr % GROUPS = g -----------------
        const int group = warp >> 2, lq = warp & 3, rl = lq * 32 + lane;      // rl: tensor memory lane = row of the tile
        int p_start = 0, p_count = 0, p_r0 = 0, p_col = 0;                      // the unit whose results are still to be read
        int small_run = 0;                                                      // units so far that filled a half
        auto results = [&]() {      // of the pending unit, the unit_run-th
            if (!mbar_wait(bar_done, (unit_run - 1) & 1, &abort_flag)) fail(2);
            ok = __all_sync(0xFFFFFFFFu, ok);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                unit_results<GU, GROUPS, (TT > 1)>(a, tmem, box + warp * 512, p_col, p_start, p_count, p_r0);
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    if (p_count > half_max || p_col == 0) mbar_arrive(bar_read);
                    if (p_count > half_max || p_col != 0) mbar_arrive(bar_read + 8);
                }
            }
            p_count = 0;
        };
        for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
            const UnitPos u = unit_pos<TT, GU>(a, unit, row_tiles, heads);
            if (u.count <= 0) continue;
            const WSlice w = GU && (lane & 1) ? u.wb : u.wa;
            const int grow = GU ? u.r0 + (rl >> 1) : u.r0 + rl;
            const float base = BF16W ? 0.0f : exact_base<P3 ? 3 : 4>(w.eb);
            auto steps = [&](auto how) {      // the unit's K steps of this warpgroup
                constexpr int V = decltype(how)::value;
                int kt = (group - kr0 % GROUPS + GROUPS) % GROUPS;
                ChunkIn cur = {};
                if (!BF16W && kt < KT) cur = load_row_chunk<P3, V>(w, grow, kt, a.R, NB);
                for (; kt < KT && ok; kt += GROUPS) {
                    const int kr = kr0 + kt, s = kr % GM_STAGES;
                    const uint32_t ta = tmem_w + ((uint32_t) (lq * 32) << 16) + (uint32_t) (s * Cfg::A_COLS);
                    ChunkIn nxt = {};
                    if (!BF16W && kt + GROUPS < KT) nxt = load_row_chunk<P3, V>(w, grow, kt + GROUPS, a.R, NB);
                    const uint32_t sw[4] = {cur.s.x, cur.s.y, cur.s.z, cur.s.w}, cw[4] = {cur.c.x, cur.c.y, cur.c.z, cur.c.w};
#pragma unroll
                    for (int q = 0; q < 2; ++q) {      // 32 weights = 16 words
                        uint32_t v[TERMS][16];
                        if (BF16W) {
#pragma unroll
                            for (int i = 0; i < 4; ++i) {
                                const int k = kt * GM_BK + q * 32 + 8 * i;
                                const uint4 t = grow < a.R && k < a.K ? __ldg((const uint4*) ((const uint16_t*) w.p[0] + (size_t) grow * a.K + k)) : make_uint4(0u, 0u, 0u, 0u);
                                v[0][4 * i] = t.x; v[0][4 * i + 1] = t.y; v[0][4 * i + 2] = t.z; v[0][4 * i + 3] = t.w;
                            }
                        } else {
#pragma unroll
                            for (int b = 0; b < 2; ++b) {
                                const int bp = 2 * q + b;
                                u64 w2[8];
                                const u64 e2 = P3 ? code_scale_pair3(cw[bp], kc) : code_scale_pair(cur.cd, bp, kc);
                                pair_weights<P3 ? 3 : 4>(tab, sw[bp], cw[bp], e2, base, kc, w2);
                                float wa[8], wb[8];
#pragma unroll
                                for (int i = 0; i < 8; ++i) unpack2(w2[i], wa[i], wb[i]);
#pragma unroll
                                for (int t = 0; t < TERMS; ++t) {      // term t = the bf16 value of what remains (exact subtraction)
#pragma unroll
                                    for (int i = 0; i < 4; ++i) {
                                        const uint32_t o = bf16x2_bits(wa[2 * i], wa[2 * i + 1]), p = bf16x2_bits(wb[2 * i], wb[2 * i + 1]);
                                        v[t][8 * b + i] = o;
                                        v[t][8 * b + 4 + i] = p;
                                        if (t + 1 < TERMS) {
                                            wa[2 * i] -= __uint_as_float(o << 16); wa[2 * i + 1] -= __uint_as_float(o & 0xFFFF0000u);
                                            wb[2 * i] -= __uint_as_float(p << 16); wb[2 * i + 1] -= __uint_as_float(p & 0xFFFF0000u);
                                        }
                                    }
                                }
                            }
                        }
                        if (q == 0) {      // the stage has to be free only now: half of the step is in registers
                            if (kr >= GM_STAGES && !mbar_wait(bar_empty + 8 * s, ((kr / GM_STAGES) - 1) & 1, &abort_flag)) fail(1);
                            ok = __all_sync(0xFFFFFFFFu, ok);
                            if (!ok) break;
                            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        }
#pragma unroll
                        for (int t = 0; t < TERMS; ++t) tmem_st16(ta + t * 32 + q * 16, v[t]);
                    }
                    if (!ok) break;
                    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_full + 8 * s);
                    cur = nxt;
                    if (p_count) results();      // the previous unit's: its last MMAs ran under this step
                }
            };
            // A table's slices are looked at a unit at a time (512 / 4096 rows of config 1's layer 276.8 / 454.8 us, without the look 274.9 / 453.5; with
            // predicated loads in one loop 276.8 / 461.3).
            if (VEC != 2) steps(std::integral_constant<int, VEC>{});
            else if (__all_sync(0xFFFFFFFFu, stream_wide<P3>(w))) steps(std::integral_constant<int, 2>{});
            else steps(std::integral_constant<int, 1>{});
            if (ok && p_count) results();      // (a unit with fewer steps than warpgroups)
            kr0 += KT;
            ++unit_run;
            p_start = u.start; p_count = u.count; p_r0 = u.r0;
            p_col = u.count <= half_max ? (small_run++ & 1) * HALF : 0;
            if (ok && KT < GROUPS) results();
        }
        if (ok && p_count) results();
    } else {
        if (Cfg::SPLIT) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::LREGS));      // (one instruction for the whole warpgroup)
        if (warp == PW) {
            // ---- the MMA issuer --------------------------------------------------------------------------------------------------
            if (lane == 0) {
                const uint64_t desc0 = umma_desc(smem_base);      // + bytes / 16 for another place in the 256 KB window
                int small_run = 0, uses[2] = {0, 0};               // units so far in each half of the accumulators
                for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
                    const UnitPos u = unit_pos<TT, GU>(a, unit, row_tiles, heads);
                    if (u.count <= 0) continue;
                    const int half = u.count <= half_max ? small_run++ & 1 : 0, col = half * HALF;
                    for (int h = 0; h < 2 && ok; ++h)
                        if (u.count > half_max || h == half) {
                            if (uses[h] > 0 && !mbar_wait(bar_read + 8 * h, (uses[h] - 1) & 1, &abort_flag)) fail(3);
                            ++uses[h];
                        }
                    for (int kt = 0; kt < KT && ok; ++kt) {
                        const int kr = kr0 + kt, s = kr % GM_STAGES;
                        if (!mbar_wait(bar_full + 8 * s, (kr / GM_STAGES) & 1, &abort_flag)) { fail(3); break; }
                        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                        const uint32_t sa = tmem_w + (uint32_t) (s * Cfg::A_COLS);
#pragma unroll 1
                        for (int n0 = 0; n0 < GM_BN * TT && n0 < u.count; n0 += 256) {      // (the tiles of a stage follow one another)
                            const uint32_t idesc = umma_idesc((min(u.count - n0, 256) + 15) & ~15);
                            const uint64_t db = desc0 + (uint64_t) ((s * Cfg::X_BYTES + n0 * 128) >> 4);
#pragma unroll
                            for (int q = 0; q < TERMS; ++q)
#pragma unroll
                                for (int k16 = 0; k16 < GM_BK / 16; ++k16)
                                    umma_ts(tmem + col + n0, sa + q * 32 + k16 * 8, db + (uint64_t) (k16 * 2), idesc, (kt | q | k16) != 0);
                        }
                        umma_commit(bar_empty + 8 * s);   // the stage is free when these MMAs have read it
                    }
                    if (ok) umma_commit(bar_done);
                    kr0 += KT;
                }
            }
        } else if (IN == IN_TMA) {
            // ---- loader: one thread asks for a K step's inputs, 32 rows at a time (rows beyond the unit's belong to others) ---------------
            if (tid == (PW + 1) * 32) {
                for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
                    const UnitPos u = unit_pos<TT, GU>(a, unit, row_tiles, heads);
                    if (u.count <= 0) continue;
                    for (int kt = 0; kt < KT && ok; ++kt) {
                        const int kr = kr0 + kt, s = kr % GM_STAGES;
                        if (kr >= GM_STAGES && !mbar_wait(bar_empty + 8 * s, ((kr / GM_STAGES) - 1) & 1, &abort_flag)) { fail(4); break; }
                        const uint32_t bar = bar_full + 8 * s, dst = smem_base + (uint32_t) (s * Cfg::X_BYTES);
                        asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1;\n\t}"
                                     ::"r"(bar), "r"((uint32_t) (((u.count + 31) & ~31) * GM_BK * 2)) : "memory");
                        for (int n = 0; n < u.count; n += 32)
                            asm volatile("cp.async.bulk.tensor.2d.shared::cta.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                                         ::"r"(dst + n * 128), "l"(&tm), "r"(kt * GM_BK), "r"(u.start + n), "r"(bar) : "memory");
                    }
                    kr0 += KT;
                }
            }
        } else {
            // ---- loaders: a K step's inputs -------------------------------------------------------------------------------------------
            const int lt = tid - (PW + 1) * 32;
            constexpr int LT = Cfg::LW * 32, RPP = LT / 8;      // threads; rows a pass
            const int uu = lt & 7, n_lo = lt >> 3;              // this thread's 16-byte unit of the K step's 64 inputs, its first row
            int pending = -1;                                   // packed: the stage whose copies are in flight
            auto settle = [&]() {      // a stage's inputs are complete
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");   // generic-proxy writes -> visible to the MMA's reads
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_full + 8 * pending);
            };
            for (int unit = blockIdx.x; unit < n_units && ok; unit += gridDim.x) {
                const UnitPos u = unit_pos<TT, GU>(a, unit, row_tiles, heads);
                if (u.count <= 0) continue;
                const int n16 = (u.count + 15) & ~15;
                __syncwarp();
                // FEW, units of few rows: groups of warps take the K steps in turn, so that two or three steps' rows are in flight instead of
                // one (a memory latency a step).  us, 128 experts, 512 x 2048: 512 / 4096 pairs 122 / 154 -> 105 / 117; 7000 and 12000 (units
                // of more than 60 rows) 162 / 174 -> 168 / 179.  The places of a warp's rows are its own: groups may be in different units.
                int groups = 1, grp = 0, wi = lt >> 5, rpp = RPP, n_first = n_lo;
                if (FEW) {
                    if (n16 <= 40) { groups = 3; grp = min(wi >> 1, 2); wi -= 2 * grp; rpp = grp == 2 ? 12 : 8; }
                    else if (n16 <= 60) { groups = 2; grp = wi >> 2; wi -= 4 * grp; rpp = grp ? 12 : 16; }
                    n_first = 4 * wi + (lane >> 3);
                }
                const int mine = FEW ? (lt >> 5) * 20 : 0;
                for (int i = lane;; i += 32) {      // this warp's own rows: 4 w .. 4 w + 3, then every RPP on
                    const int n = (wi << 2) + (i & 3) + (i >> 2) * (FEW ? rpp : RPP);
                    if (n >= n16) break;
                    srow[FEW ? mine + i : n] = input_row_of(a, u, n);
                }
                __syncwarp();
                constexpr int FLIGHT = !Cfg::DENSE ? 5 : TT == 1 ? 3 : TT == 2 ? 5 : 4;      // F32: 16-byte results in flight a thread (5 x 28 rows, DENSE 3 x 44: a tile; 5 x 60: two)
                float4 x[F32 ? 2 * FLIGHT : 1];
                auto request = [&](int kt, int n0) {
                    const int k = kt * GM_BK + 8 * uu;
#pragma unroll
                    for (int i = 0; i < FLIGHT; ++i) {
                        const int n = n0 + i * (FEW ? rpp : RPP);
                        x[2 * i] = x[2 * i + 1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                        if (n < n16 && k < a.K) {
                            const float4* xp = (const float4*) ((const float*) a.X + ((size_t) srow[FEW ? mine + 4 * i + (lane >> 3) : n] * a.xs + k));
                            x[2 * i] = ld_in_order(xp);      // (C++ loads: 1.5 to 3 % slower)
                            x[2 * i + 1] = ld_in_order(xp + 1);
                        }
                    }
                };
                if (F32 && grp < KT) request(grp, n_first);
                int turn = 0;      // the group whose step this is
                for (int kt = 0; kt < KT && ok; ++kt) {
                    const int kr = kr0 + kt, s = kr % GM_STAGES;
                    if (kr >= GM_STAGES && !mbar_wait(bar_empty + 8 * s, ((kr / GM_STAGES) - 1) & 1, &abort_flag)) fail(4);
                    ok = __all_sync(0xFFFFFFFFu, ok);
                    if (!ok) break;
                    const uint32_t stage = smem_base + (uint32_t) (s * Cfg::X_BYTES);
                    if (!F32) {      // copies of this step, then the arrival of the previous one's
                        const int k = kt * GM_BK + 8 * uu;
                        const bool in = k < a.K;
                        const uint16_t* xk = (const uint16_t*) a.X + (in ? k : 0);
#pragma unroll 4
                        for (int n = n_lo; n < n16; n += RPP)
                            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(input_at(stage, n, uu)), "l"(xk + (size_t) srow[n] * a.xs), "r"(in ? 16 : 0) : "memory");
                        asm volatile("cp.async.commit_group;" ::: "memory");
                        if (pending >= 0) {
                            asm volatile("cp.async.wait_group 1;" ::: "memory");
                            settle();
                        }
                        pending = s;
                    } else if (FEW) {
                        pending = s;
                        if (turn == grp) {
#pragma unroll
                            for (int i = 0; i < FLIGHT; ++i) {
                                const int n = n_first + i * rpp;
                                if (n < n16)
                                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(input_at(stage, n, uu)), "r"(bf16x2_bits(x[2 * i].x, x[2 * i].y)),
                                                 "r"(bf16x2_bits(x[2 * i].z, x[2 * i].w)), "r"(bf16x2_bits(x[2 * i + 1].x, x[2 * i + 1].y)),
                                                 "r"(bf16x2_bits(x[2 * i + 1].z, x[2 * i + 1].w)) : "memory");
                            }
                            if (kt + groups < KT) request(kt + groups, n_first);
                        }
                        settle();
                        if (++turn == groups) turn = 0;
                    } else {
                        for (int n0 = n_lo;;) {
#pragma unroll
                            for (int i = 0; i < FLIGHT; ++i) {
                                const int n = n0 + i * RPP;
                                if (n < n16)
                                    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(input_at(stage, n, uu)), "r"(bf16x2_bits(x[2 * i].x, x[2 * i].y)),
                                                 "r"(bf16x2_bits(x[2 * i].z, x[2 * i].w)), "r"(bf16x2_bits(x[2 * i + 1].x, x[2 * i + 1].y)),
                                                 "r"(bf16x2_bits(x[2 * i + 1].z, x[2 * i + 1].w)) : "memory");
                            }
                            n0 += FLIGHT * RPP;
                            const bool more = __any_sync(0xFFFFFFFFu, n0 < n16);      // (warp-uniform)
                            if (more) request(kt, n0);
                            else if (kt + 1 < KT) request(kt + 1, n_lo);
                            if (!more) break;
                        }
                        pending = s;
                        settle();
                    }
                }
                kr0 += KT;
            }
            if (!F32 && pending >= 0 && ok) {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
                settle();
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (abort_flag) {      // a wait ran out: the block's copies and MMAs in flight have no barrier left to report to, so they get a millisecond before its memory goes
        asm volatile("cp.async.wait_all;" ::: "memory");
        unsigned long long t0, t;
        asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t0));
        for (int i = 0; i < 4096; ++i) {
            asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
            if (t - t0 > 1000000ull) break;
            __nanosleep(1000);
        }
        __syncthreads();
    }
    if (warp == PW) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::COLS) : "memory");
}

bool launch_bf16_mm_skinny(cudaStream_t s, const WSlice& w, int K, int R, const float* x, int xs, float* y, int ys, int T, int add);

static int g_exact;   // kc_seed_gemm_f32: process-wide, as the reference's switch (engine/kernels_moe.cu:2354)
bool seed_gemm_exact() { return g_exact != 0; }

// The tensor map of packed rows that follow one another: K bf16 values a row, xs apart, boxes of 32 rows x 64 values with the 128-byte
// swizzle; what lies beyond K or the last row arrives as zeros.
static bool encode_inputs(CUtensorMap* tm, const MmParams& a) {
    typedef CUresult (*Encode)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                               CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
    static const Encode encode = [] {
        void* f = NULL;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) != cudaSuccess || q != cudaDriverEntryPointSuccess) f = NULL;
        return (Encode) f;
    }();
    const cuuint64_t dims[2] = {(cuuint64_t) a.K, (cuuint64_t) (a.grouped ? a.T_in : a.T)}, strides[1] = {(cuuint64_t) a.xs * 2};
    const cuuint32_t box[2] = {64, 32}, step[2] = {1, 1};
    return encode && encode(tm, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(a.X), dims, strides, box, step, CU_TENSOR_MAP_INTERLEAVE_NONE,
                            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// false (nothing launched): IN_TMA inputs that a tensor map cannot describe.
template <int TERMS, int WF, int TT, int VEC, bool GU, int IN>
static bool launch_gemm_v(cudaStream_t s, const MmParams& a, int units) {
    using Cfg = GmCfg<TERMS, TT, IN>;
    const size_t smem = (size_t) GM_STAGES * Cfg::X_BYTES + Cfg::PW * 1024 + 1024;
    static bool attr_set[16];
    int dev = 0;
    cudaGetDevice(&dev);
    if (!attr_set[dev & 15]) {
        cudaFuncSetAttribute(seed_gemm_kernel<TERMS, WF, TT, VEC, GU, IN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) smem);
        attr_set[dev & 15] = true;
    }
    GmMap<IN> tm = {};
    if constexpr (IN == IN_TMA) {
        if (a.xs < a.K || !encode_inputs(&tm, a)) return false;
    }
    const int slots = sm_count() * Cfg::CTAS;
    launch(seed_gemm_kernel<TERMS, WF, TT, VEC, GU, IN>, (unsigned) (units < slots ? units : slots), Cfg::THREADS, smem, s, a, kconst(), tm);
    count_launch();
    return true;
}
static void no_map(const MmParams& a) { set_error("seed GEMM: no tensor map for sorted inputs of row stride %d", a.xs); }
// How many tiles of a dense call share an expansion: a unit takes the time of its expansion (twice that where two blocks share an
// SM) or of its inputs' conversion, and the units go round the SMs.  f32, us a round of units at K = 2048: one tile 34-35 in either kernel form
// (launch_dense_f32) where a block has several units, two tiles 45-48, three 62-72; a block's only unit of one tile 31.  Three rounds of one tile and two
// of two are a tie that the steps of a unit decide, one tile / two: 20000 x 2048, 200 rows 103.1 / 88.0, x 1024 55.9 / 51.1, x 512 32.9 / 33.0; 1906 x 1088,
// 3673 rows 59.5 / 57.9; 5019 x 640, 1156 rows 39.5 / 40.7; 4869 x 512, 1218 rows 34.2 / 36.1.  Two rounds of one tile against one of three: 7120 x 1216,
// 617 rows 44.9 / 47.9, 3235 x 2176, 1365 rows 72.7 / 76.1, 6943 x 576, 553 rows 25.7 / 29.7, 1698 x 3840, 2588 rows 133 / 126.
static int dense_tiles(const MmParams& a, int row_tiles) {
    int best = 1;
    double best_cost = 0.0;
    for (int tt = 1; tt <= 3; ++tt) {
        if (a.packed && tt == 2) continue;
        const int units = row_tiles * ((a.T + GM_BN * tt - 1) / (GM_BN * tt)), slots = sm_count() * (a.packed && tt == 1 ? 2 : 1);
        const double unit = a.packed ? (tt == 1 && units > sm_count() ? 2.0 : 1.0) : tt == 1 && units > sm_count() && a.K >= 1024 ? 0.97 : 0.45 + 0.5 * tt;
        const double cost = (double) ((units + slots - 1) / slots) * unit;
        if (tt == 1 || cost < best_cost) { best = tt; best_cost = cost; }
    }
    return best;
}
// Dense f32 inputs.  Their loaders set the pace (load, convert, store and report a step, while the producers take most issue slots), and with
// 16 producers and 7 loaders a step's rows also came in two or three passes, each a memory latency.  8 producers and 11 loaders take a tile
// in one pass, 8 and 15 two tiles; both fit their registers, the 16 and 7 spill.  us, 16 + 7 / now: 2048 x 2048, 65 rows 34.8 / 34.4, 777 rows
// 38.6 / 36.8, 2048 rows 58.8 / 50.7, 4096 rows 131.0 / 99.1; 8192 x 2048, 1024 rows 119 / 97; 8192 x 4096, 700 rows 154 / 131 (the last five with two or
// three tiles).  One tile and several units a block: the results are read by the producers, which 16 do faster where a unit has few steps (16 + 7 / 8 + 11:
// 20000 x 512, 100 rows 22.6 / 24.6, 40000 x 512 32.2 / 35.4, 151936 x 512 92.8 / 101.9; K = 1024 37.9 / 39.4, 54.7 / 57.4, 157.6 / 166.7; K = 2048 69.1 / 68.9,
// 101.5 / 101.8; 20000 x 4096 130.1 / 127.7).
template <int WF>
static void launch_dense_f32(cudaStream_t s, const MmParams& a, int tt, int units) {
    if (tt == 1 && units > sm_count()) launch_gemm_v<1, WF, 1, 2, false, IN_F32>(s, a, units);
    else if (tt == 1) launch_gemm_v<1, WF, 1, 2, false, IN_F32_DENSE>(s, a, units);
    else if (tt == 2) launch_gemm_v<1, WF, 2, 2, false, IN_F32_DENSE>(s, a, units);
    else launch_gemm_v<1, WF, 3, 2, false, IN_F32_DENSE>(s, a, units);
}
// Whether a slice's seeds and coefficient words are aligned to n bytes and its codes to n / 4.
template <int WF>
static bool streams_aligned(const WSlice& w, unsigned n) {
    return (((uintptr_t) w.p[0] | (uintptr_t) w.p[1]) & (n - 1)) == 0 && (WF == 2 || ((uintptr_t) w.p[3] & (n / 4 - 1)) == 0);
}
template <int WF>
static void launch_gemm_seed(cudaStream_t s, const MmParams& a, int row_tiles, int tiles_y) {
    const int units = row_tiles * tiles_y;
    // how the streams can be read; slices in a device table (8-byte aligned) are looked at by the kernel
    const int vec = a.K % 32 || (!a.grouped && !streams_aligned<WF>(a.w0, 8)) ? 0 : a.K % 64 ? 1 : 2;
    if (g_exact) {
        if (a.packed) { if (vec) launch_gemm_v<3, WF, 1, 1, false, IN_LIST>(s, a, units); else launch_gemm_v<3, WF, 1, 0, false, IN_LIST>(s, a, units); }
        else if (vec == 2) launch_gemm_v<3, WF, 1, 2, false, IN_F32>(s, a, units);
        else if (vec) launch_gemm_v<3, WF, 1, 1, false, IN_F32>(s, a, units);
        else launch_gemm_v<3, WF, 1, 0, false, IN_F32>(s, a, units);
    } else if (vec < 2) {
        if (a.packed) { if (vec) launch_gemm_v<1, WF, 1, 1, false, IN_LIST>(s, a, units); else launch_gemm_v<1, WF, 1, 0, false, IN_LIST>(s, a, units); }
        else if (vec) launch_gemm_v<1, WF, 1, 1, false, IN_F32>(s, a, units);
        else launch_gemm_v<1, WF, 1, 0, false, IN_F32>(s, a, units);
    } else if (a.grouped) {
        if (!a.packed) launch_gemm_v<1, WF, 1, 2, false, IN_F32_FEW>(s, a, units);
        else if (a.in_sorted && a.offs) { if (!launch_gemm_v<1, WF, 3, 2, false, IN_TMA>(s, a, units)) no_map(a); }
        else launch_gemm_v<1, WF, 1, 2, false, IN_LIST>(s, a, units);
    } else {
        const int tt = dense_tiles(a, row_tiles), u = row_tiles * ((a.T + GM_BN * tt - 1) / (GM_BN * tt));
        if (a.packed) {
            if (!(tt == 1 ? launch_gemm_v<1, WF, 1, 2, false, IN_TMA>(s, a, u) : launch_gemm_v<1, WF, 3, 2, false, IN_TMA>(s, a, u)))
                launch_gemm_v<1, WF, 1, 2, false, IN_LIST>(s, a, units);      // rows that overlap
        }
        else launch_dense_f32<WF>(s, a, tt, u);
    }
}
void launch_gemm_gu(cudaStream_t s, const MmParams& a, int tiles_y) {
    const int units = (a.R + GM_BM / 2 - 1) / (GM_BM / 2) * tiles_y;
    if (a.offs) { if (!launch_gemm_v<1, 0, 3, 2, true, IN_TMA>(s, a, units)) no_map(a); }
    else launch_gemm_v<1, 0, 1, 2, true, IN_LIST>(s, a, units);
}
bool gemm_shares_tiles(int max_tiles) { return max_tiles <= GM_MAX_HEADS; }

void launch_gemm(cudaStream_t s, int fmt, const char* who, MmParams a, int tiles_y) {
    if (fmt != MF_SEED4P4 && fmt != MF_SEED4 && fmt != MF_BF16) {
        set_error("%s: weight format %d is not served by this library (SEED4P4 = %d, SEED4 = %d and BF16 = %d only)", who, fmt, (int) MF_SEED4P4,
                  (int) MF_SEED4, (int) MF_BF16);
        return;
    }
    if (a.K <= 0 || a.K % 8 || a.R <= 0) { set_error("%s: K = %d (a multiple of 8), R = %d", who, a.K, a.R); return; }
    if (fmt == MF_BF16 && ((a.ws == NULL && !aligned16(a.w0.p[0])))) { set_error("%s: BF16 weights must be 16-byte aligned", who); return; }
    if (tiles_y <= 0) return;
    if (!aligned16(a.X) || (a.packed ? a.xs % 8 : a.xs % 4)) {
        set_error("%s: inputs must be 16-byte aligned with a row stride that is a multiple of 16 bytes", who);
        return;
    }
    if (a.grouped && !a.ntiles) a.T = tiles_y;
    // A dense call of a few rows: the weights stay in registers.  The line lies where the second tile of 32 rows has used up what that saves
    // (us, this kernel / that one: 2048 x 2048, 9 rows 34.9 / 12.5, 32 rows 34.9 / 16.5, 64 rows 37.0 / 30.6; 512 x 2048, 64 rows 36.8 / 16.5;
    // 8192 x 4096, 9 rows 62.5 / 36.3, 48 rows 64.5 / 63.5, 64 rows 65.7 / 73.2; a third tile adds half as much again; one call behind the other
    // that kernel now takes 9.2, 14.3, 27.7; 14.1; 33.5, 60.5 and 70.5).  A row's bits differ
    // between the two (the order of its sums), not within either.
    if (fmt != MF_BF16 && !g_exact && !a.grouped && a.T <= 64 && (fmt == MF_SEED4 ? streams_aligned<2>(a.w0, 16) : streams_aligned<0>(a.w0, 16)) &&
        smm_serves(a.K, a.X, a.xs, a.packed)) { launch_seed_mma(s, fmt, a); return; }
    const int row_tiles = (a.R + GM_BM - 1) / GM_BM;
    if (fmt == MF_BF16) {      // stored BF16 weights (p[0] = [R][K]): no expansion, one term
        if (a.packed) launch_gemm_v<1, 1, 1, 0, false, IN_LIST>(s, a, row_tiles * tiles_y);
        else launch_gemm_v<1, 1, 1, 0, false, IN_F32>(s, a, row_tiles * tiles_y);
    } else if (fmt == MF_SEED4) launch_gemm_seed<2>(s, a, row_tiles, tiles_y);
    else launch_gemm_seed<0>(s, a, row_tiles, tiles_y);
}

}   // namespace nsl

using namespace nsl;

extern "C" {

void kc_seed_gemm_f32(int on) { g_exact = on; }

void kc_mm(cudaStream_t s, int fmt, WSlice w, int K, int R, const float* x, int xs, float* y, int ys, int T, int add,
           const uint32_t* G) {
    if (fmt == MF_BF16 && launch_bf16_mm_skinny(s, w, K, R, x, xs, y, ys, T, add)) return;      // a decode batch (dense_bf16.cu)
    FollowScope follow(fmt != MF_BF16);      // (products of stored weights have not been measured as such)
    MmParams a = {NULL, w, x, y, NULL, NULL, NULL, G, K, R, T, xs, ys, 1, add, 0, 0, NULL, 0, NULL, 0, 0, 0, follow.own()};
    launch_gemm(s, fmt, "kc_mm", a, (T + GM_BN - 1) / GM_BN);
}
void kc_mm_packed(cudaStream_t s, int fmt, WSlice w, int K, int R, const uint16_t* x, int xs, float* y, int ys, int T, int add,
                  const uint32_t* G) {
    MmParams a = {NULL, w, x, y, NULL, NULL, NULL, G, K, R, T, xs, ys, 1, add, 0, 1, NULL, 0, NULL, 0, 0, 0};
    launch_gemm(s, fmt, "kc_mm_packed", a, (T + GM_BN - 1) / GM_BN);
}
void kc_mm_grouped(cudaStream_t s, int fmt, const WSlice* ws, int K, int R, const float* x, int xs, float* y, int ys,
                   int xdiv, const int32_t* perm, const MmTile* tiles, int ntiles, const uint32_t* G) {
    MmParams a = {ws, WSlice{}, x, y, perm, tiles, NULL, G, K, R, 0, xs, ys, xdiv, 0, 1, 0, NULL, 0, NULL, 0, 0, 0};
    launch_gemm(s, fmt, "kc_mm_grouped", a, ntiles);
}
void kc_mm_grouped_dev(cudaStream_t s, int fmt, const WSlice* ws, int K, int R, const float* x, int xs, float* y, int ys,
                       int xdiv, const int32_t* perm, const MmTile* tiles, const int32_t* ntiles, int max_tiles,
                       const uint32_t* G) {
    MmParams a = {ws, WSlice{}, x, y, perm, tiles, ntiles, G, K, R, 0, xs, ys, xdiv, 0, 1, 0, NULL, 0, NULL, 0, 0, 0};
    launch_gemm(s, fmt, "kc_mm_grouped_dev", a, max_tiles);
}
void kc_mm_grouped_packed(cudaStream_t s, int fmt, const WSlice* ws, int K, int R, const uint16_t* x, int xs, float* y, int ys,
                          int xdiv, const int32_t* perm, const MmTile* tiles, const int32_t* nt, int max_tiles,
                          const uint32_t* G) {
    MmParams a = {ws, WSlice{}, x, y, perm, tiles, nt, G, K, R, 0, xs, ys, xdiv, 0, 1, 1, NULL, 0, NULL, 0, 0, 0};
    launch_gemm(s, fmt, "kc_mm_grouped_packed", a, max_tiles);
}

// 0, or the code of the first bounded wait that ran out in a GEMM block since the last call (1 producer waiting for a
// free stage, 2 results waiting for the accumulators, 3 MMA issuer waiting for a full stage or for the results to have been read, 4 loader
// waiting for a free stage).  Reads device memory: call it after the stream has been synchronised.
int nsl_mm_status(void) {
    int v = 0, zero = 0;
    cudaMemcpyFromSymbol(&v, g_mm_status, sizeof v);
    if (v) cudaMemcpyToSymbol(g_mm_status, &zero, sizeof zero);
    return v;
}

}   // extern "C"
