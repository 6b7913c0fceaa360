// Seed-decode mat-vec kernels for sm_100a: dense (kc_mv), gathered (kc_mv_sel), fused gate+up+SwiGLU (kc_mv_gu), the
// raw-f32 variant and the bit-exact decode.  Replaces the SEED4P4 paths of the reference's k_mv / k_mv1 / k_mv_gu
// (engine/kernels_moe.cu:130-159, 222-348, 2308-2328) and the weight reader used by its tests.
//
// Data movement.  A row of K weights is K/8 blocks; a "chunk" is 8 consecutive blocks = one 16-byte load of seeds, one
// of coefficient words and one 4-byte load of exponent codes.  A lane takes one chunk of a row at a time (64 inputs), so a
// warp reads a row's streams as contiguous runs; the inputs sit in shared memory.  Rows shorter than 32 chunks share a warp
// (K = 512: four rows per step, eight lanes each); rows of another length than 2^j <= 32 chunks are cut into groups of lanes.
//
// Arithmetic per block: the dot form of seed_block.cuh for gathers (32 fused multiply-adds on 32 masked stream words, then the
// four coefficients and the block's 2^code), the weight form for dense calls, whose rows of inputs share each expansion.  A
// token's sum is formed in the same order whatever the number of tokens in the call, so a row of a multi-token call equals the
// single-token call bit for bit, as the reference requires (tests/test_mova_kernels.c:173-183).
#include <math.h>

#include <algorithm>

#include "common.cuh"
#include "route.cuh"
#include "seed_block.cuh"

namespace nsl {

constexpr int MV_WARPS = 8;
constexpr int MV_THREADS = 32 * MV_WARPS;
enum { MODE_ROUND = 0, MODE_GU = 2 };   // the raw-f32 store is a run-time flag of MODE_ROUND

struct MvParams {
    const WSlice* ws;     // slice table on the device (gather), or NULL: w0
    const WSlice* wu;     // gate+up: the up slices
    WSlice w0;            // dense: the slice by value
    const int32_t* sel;   // pair -> slice, or NULL (dense)
    const float* x;
    float* y;
    const uint32_t* G;
    int K, R, P, xdiv, xs, ys, add, raw;
    const int32_t* xrow;    // optional: pair p reads input row xrow[p] (instead of p / xdiv)
    const int32_t* count;   // optional: the pair count is read on the device (<= P)
    int xbf16;              // inputs are packed bf16 rows (row stride xs in bf16 elements)
    int late = 0;         // G may be read only after the wait for the previous kernel
};

__device__ __forceinline__ float silu_bf(float g) {   // each op rounded to bf16 (engine/kernels_moe.cu:28-31)
    const float s = bf16_round(1.0f / (1.0f + expf(-g)));
    return bf16_round(g * s);
}

struct Chunk { uint4 s, c; uint32_t cd; };

// The conversion constants (seed_block.cuh: KConst) as a module constant for code outside the kernels' own bodies: a
// function that is not inlined cannot take them as constant-bank kernel arguments.
constexpr float pow2_f(int e) {
    float v = 1.0f;
    for (int i = 0; i < (e < 0 ? -e : e); ++i) v = e < 0 ? v * 0.5f : v * 2.0f;
    return v;
}
constexpr KConst kconst_static() {
    KConst k = {};
    for (int p = 0; p < 4; ++p) {
        k.cxor[p] = ((uint32_t) (215 - 5 * p) << 23) | (8u << (4 * p));
        k.coff[p] = -(pow2_f(88 - 5 * p) + pow2_f(68 - p));
        k.cxor_x[p] = ((uint32_t) (253 - 5 * p) << 23) | (8u << (4 * p));
        k.coff_x[p] = -(pow2_f(126 - 5 * p) + pow2_f(106 - p));
    }
    k.cor = 112u << 23;
    return k;
}
__constant__ KConst c_kc = kconst_static();

// What the loop over the units' items needs, by value (it runs in a function of its own: see unit_items).
struct UnitCall {
    float* y;
    int ys, R, raw, add;
    int lpr_log2, items;      // items of the window's units of this size
};
__device__ __forceinline__ Chunk load_chunk3(const uint4* s, const uint4* c, const uint32_t* d, size_t chunk_index) {
    Chunk k;
    k.s = __ldg(s + chunk_index);
    k.c = __ldg(c + chunk_index);
    k.cd = __ldg(d + chunk_index);
    return k;
}

template <int PF = 4>      // PF = 3: the SEED4 format has no code stream (a block's code rides in its nibble word)
__device__ __forceinline__ Chunk load_chunk(const WSlice& w, size_t chunk_index) {
    Chunk k;
    k.s = __ldg((const uint4*) w.p[0] + chunk_index);
    k.c = __ldg((const uint4*) w.p[1] + chunk_index);
    k.cd = PF == 4 ? __ldg((const uint32_t*) w.p[3] + chunk_index) : 0u;
    return k;
}

// Eight 16-bit values of a stream of any alignment.  (P = 3 gathers over rows that are not 2^j <= 32 chunks take slices from any address; the
// other forms of a device table have always been read 16 bytes at a time.)
__device__ __forceinline__ bool chunk_aligned(const void* s, const void* c) { return (((unsigned long long) s | (unsigned long long) c) & 15ull) == 0; }
__device__ __noinline__ uint4 load_any_16(const void* p, uint32_t chunk) {
    const uint16_t* q = (const uint16_t*) p + (size_t) chunk * 8;
    uint32_t w[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) w[i] = (uint32_t) __ldg(q + 2 * i) | ((uint32_t) __ldg(q + 2 * i + 1) << 16);
    return make_uint4(w[0], w[1], w[2], w[3]);
}

__device__ __forceinline__ float pair_total(u64 acc2) {
    float lo, hi;
    unpack2(acc2, lo, hi);
    return lo + hi;
}

__device__ __forceinline__ float group_sum(float v, int lpr) {
    for (int o = lpr >> 1; o > 0; o >>= 1) v += __shfl_xor_sync(0xFFFFFFFFu, v, o);
    return v;
}

template <int MODE>
__device__ __forceinline__ void store_out(const MvParams& a, int pair, int r, float s, float su) {
    float* yo = a.y + (size_t) pair * a.ys + r;
    if (MODE == MODE_GU) *yo = a.raw ? (s / (1.0f + expf(-s))) * su : bf16_round(silu_bf(bf16_round(s)) * bf16_round(su));
    else if (a.raw) *yo = s;
    else *yo = a.add ? bf16_round(*yo + bf16_round(s)) : bf16_round(s);   // engine/kernels_moe.cu:214
}

// Inputs in shared memory.  A staged chunk (64 inputs) is CX 16-byte units: the f32x2 operands of the block pairs
// ({x of the even block, x of the odd block}, scaled by input_scale; unit 4 bp + cq holds operands 2 cq and 2 cq + 1 of block
// pair bp), then the block pairs' input sums (unscaled, two u64 a unit), and one unit of padding: chunks are 304 bytes apart,
// so that the 16-byte loads of eight neighbouring lanes (one chunk each) touch all 32 banks once.  Every offset inside a
// chunk is an immediate.
constexpr int CX = 19;

// The centring of pair_expand_dot: xm[p] = -32768 2^(p-85) sum(x), from the (unscaled) input sums of the pair's blocks.
__device__ __forceinline__ void offsets_from_sum(u64 s2, u64* xm2) {
    xm2[0] = mul2(s2, pack2(-8.470329472543003e-22f, -8.470329472543003e-22f));     // -2^-70
    xm2[1] = mul2(s2, pack2(-1.6940658945086007e-21f, -1.6940658945086007e-21f));   // -2^-69
    xm2[2] = mul2(s2, pack2(-3.3881317890172014e-21f, -3.3881317890172014e-21f));   // -2^-68
    xm2[3] = mul2(s2, pack2(-6.776263578034403e-21f, -6.776263578034403e-21f));     // -2^-67
}
__device__ __forceinline__ float input_sum(const float* x) { return ((x[0] + x[4]) + (x[1] + x[5])) + ((x[2] + x[6]) + (x[3] + x[7])); }

// 16 inputs (chunk j of the row, block pair bp): from memory, and into a staged row.
template <bool CG = false>      // CG: memory that other blocks of this grid have written (the loads bypass the L1)
__device__ __forceinline__ void stage_load(const void* row, int bf16, int j, int bp, float* x) {
    if (bf16) {
        const uint4* xp = (const uint4*) ((const uint16_t*) row + (size_t) j * 64 + bp * 16);
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const uint4 t = xp[i];
            const uint32_t u[4] = {t.x, t.y, t.z, t.w};
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                x[8 * i + 2 * q] = __uint_as_float(u[q] << 16);
                x[8 * i + 2 * q + 1] = __uint_as_float(u[q] & 0xFFFF0000u);
            }
        }
    } else {
        const float4* xp = (const float4*) ((const float*) row + (size_t) j * 64 + bp * 16);
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float4 t = CG ? __ldcg(xp + i) : xp[i];
            x[4 * i] = t.x; x[4 * i + 1] = t.y; x[4 * i + 2] = t.z; x[4 * i + 3] = t.w;
        }
    }
}
template <int PF>
__device__ __forceinline__ void stage_store(const float* x, int j, int bp, ulonglong2* sx) {
    ulonglong2* c = sx + j * CX;
#pragma unroll
    for (int cq = 0; cq < 4; ++cq) {
        const float s0 = input_scale<PF>(2 * cq), s1 = input_scale<PF>(2 * cq + 1);
        ulonglong2 t;
        t.x = pack2(x[2 * cq] * s0, x[8 + 2 * cq] * s0);
        t.y = pack2(x[2 * cq + 1] * s1, x[8 + 2 * cq + 1] * s1);
        c[bp * 4 + cq] = t;
    }
    ((u64*) (c + 16))[bp] = pack2(input_sum(x), input_sum(x + 8));
}
__device__ __forceinline__ const void* input_row(const MvParams& a, int xr) {
    return a.xbf16 ? (const void*) ((const uint16_t*) a.x + (size_t) xr * a.xs) : (const void*) (a.x + (size_t) xr * a.xs);
}
// The operands of block pair bp of a staged chunk.
__device__ __forceinline__ void staged_pair(const ulonglong2* c, int bp, u64* x2) {
#pragma unroll
    for (int cq = 0; cq < 4; ++cq) { const ulonglong2 t = c[bp * 4 + cq]; x2[2 * cq] = t.x; x2[2 * cq + 1] = t.y; }
}
__device__ __forceinline__ u64 staged_sum(const ulonglong2* c, int bp) { return ((const u64*) (c + 16))[bp]; }

struct RouteFuse {        // the router folded into the prologue (logits == NULL: the pair list comes from MvParams.sel)
    const float* logits;
    int ld, n_exp, top_k, T;
    int32_t* ind_out;
    float* wt_out;
};

// How a row is cut.  Its sum is defined on 32 VIRTUAL lanes: virtual lane v sums chunks v, v + 32, ... in order, and the 32 sums
// are added by the tree of a butterfly (distance 16 first).  A warp may give a row any power of two lpr of real lanes: lane jc
// then plays the virtual lanes jc + i lpr one after the other (in the order in which the tree adds them) and adds them as the
// tree does, so the split never shows in the bits.  Virtual lanes beyond the row's chunks are zeros: lv = log2 of those kept.
//   fewer lanes a row: more rows a step, so fewer shuffles and fewer distinct 16-byte inputs a load of the warp fetches, and
//   less idling when the chunks do not fill 32 lanes (45 chunks: 64 lane slots with 32 lanes, 48 with 8);
//   more lanes a row: more steps to deal to the warps of a small call.
struct RowShape { int ch, lpr_log2, lv, groups; };

__host__ __device__ __forceinline__ int pass_offset(int pass, int lv) {      // the first virtual lane of a pass: the pass number's bits reversed
    return ((pass & 1) << lv >> 1) | ((pass >> 1 & 1) << lv >> 2) | ((pass >> 2 & 1) << lv >> 3);
}
// s = the sum of pass `pass`: the tree's partial sums that it completes, or into the stack to wait for their other half.
__device__ __forceinline__ float tree_push(float* stk, int pass, float s) {
    if (pass & 1) s = stk[0] + s; else stk[0] = s;
    if ((pass & 1) && (pass & 2)) s = stk[1] + s; else if (pass & 1) stk[1] = s;
    if ((pass & 3) == 3 && (pass & 4)) s = stk[2] + s; else if ((pass & 3) == 3) stk[2] = s;
    return s;      // the whole lane's sum after its last pass
}

// One chunk of the gate (or only) matrix and of the up matrix against its staged inputs.
template <int MODE, int PF>
__device__ __forceinline__ void chunk_dots(const StreamTab& tab, const KConst& kc, const Chunk& ka, const Chunk& kb, const ulonglong2* cx, u64& acc, u64& accu) {
    const uint32_t swa[4] = {ka.s.x, ka.s.y, ka.s.z, ka.s.w}, cwa[4] = {ka.c.x, ka.c.y, ka.c.z, ka.c.w};
    const uint32_t swb[4] = {kb.s.x, kb.s.y, kb.s.z, kb.s.w}, cwb[4] = {kb.c.x, kb.c.y, kb.c.z, kb.c.w};
#pragma unroll
    for (int bp = 0; bp < 4; ++bp) {
        u64 x2[8], xm2[4];
        staged_pair(cx, bp, x2);
        offsets_from_sum(staged_sum(cx, bp), xm2);
        if (PF == 4) {
            u64 q[4];
            pair_coefs(cwa[bp], kc, q);
            acc = fma2(pair_expand_dot(tab, swa[bp], q, x2, xm2), code_scale_pair(ka.cd, bp, kc), acc);
        } else {
            u64 q[3];
            pair_coefs3(cwa[bp], kc, q);
            acc = fma2(pair_expand_dot3(tab, swa[bp], q, x2, xm2), code_scale_pair3(cwa[bp], kc), acc);
        }
        if (MODE == MODE_GU && PF == 4) {
            u64 q[4];
            pair_coefs(cwb[bp], kc, q);
            accu = fma2(pair_expand_dot(tab, swb[bp], q, x2, xm2), code_scale_pair(kb.cd, bp, kc), accu);
        } else if (MODE == MODE_GU) {
            u64 q[3];
            pair_coefs3(cwb[bp], kc, q);
            accu = fma2(pair_expand_dot3(tab, swb[bp], q, x2, xm2), code_scale_pair3(cwb[bp], kc), accu);
        }
    }
}

// Butterfly sums of N values over the lpr lanes of a row (distance lpr / 2 first), each finished by lpr / N lanes only: at the first
// distances a lane sends the values it will not finish and keeps the others.  Returns the sum of value jc / (lpr / N), bit for
// bit what a whole butterfly gives, for 5 (N = 2) or 6 (N = 4) shuffles at 32 lanes instead of 5 N.
template <int N>
__device__ __forceinline__ float split_sum(const float* v, int lpr, int jc) {
    int o = lpr >> 1;
    float a[2] = {v[0], v[1]};
    if (N == 4) {
        const bool up = jc & o;
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const float keep = up ? v[N - 2 + i] : v[i], send = up ? v[i] : v[N - 2 + i];
            a[i] = keep + __shfl_xor_sync(0xFFFFFFFFu, send, o);
        }
        o >>= 1;
    }
    const bool up = jc & o;
    float m = (up ? a[1] : a[0]) + __shfl_xor_sync(0xFFFFFFFFu, up ? a[0] : a[1], o);
    for (o >>= 1; o > 0; o >>= 1) m += __shfl_xor_sync(0xFFFFFFFFu, m, o);
    return m;
}

// Rows of 2^j = 1 .. 32 chunks: a row step = the 32 / lpr rows a warp expands at once, a lane owning one chunk of its row; the
// steps [s_lo, s_hi) of a pair go to the block's warps in turn.  A warp takes two rows of streams at a time against the same
// inputs (an ITEM): a row of the gate and of the up matrix, or two of its steps of the one matrix.
template <int MODE>
struct RowItem {
    static constexpr int STEPS = MODE == MODE_GU ? 1 : 2;      // row steps of the warp an item takes
};
// An item's streams: its first step st, row r.
template <int MODE, int PF>
__device__ __forceinline__ void load_item(const WSlice& wa, const WSlice& wb, int st, int r, int s_hi, int R, int lpr_log2, int jc, Chunk& ka, Chunk& kb) {
    const int S = MV_WARPS * (32 >> lpr_log2);
    if (st < s_hi && r < R) {
        ka = load_chunk<PF>(wa, (size_t) ((r << lpr_log2) + jc));
        if (MODE == MODE_GU) kb = load_chunk<PF>(wb, (size_t) ((r << lpr_log2) + jc));
    }
    if (MODE != MODE_GU && st + MV_WARPS < s_hi && r + S < R) kb = load_chunk<PF>(wa, (size_t) (((r + S) << lpr_log2) + jc));
}
// The items of one pair that fall to this warp, whose first step is st.  ka / kb: the first item's streams, requested by the caller before the inputs were
// staged; the next ones are requested before the current ones are expanded.  The sums stay in the lanes that finish them until
// every lane has one: SwiGLU, rounding and stores then run once for lpr / 2 items (once an item, with one lane in work, they
// and the reductions took 17 of 90 instructions a block).
// store(r, s, su): row r's sum (and the up matrix's).
template <int MODE, int PF, typename Store>
__device__ __forceinline__ void pair_rows(const StreamTab& tab, const KConst& kc, const WSlice& wa, const WSlice& wb, const ulonglong2* sx,
                                          int lpr_log2, int R, int st, int s_hi, Chunk ka, Chunk kb, Store store) {
    constexpr int STEPS = RowItem<MODE>::STEPS;
    const int lane = threadIdx.x & 31;
    const int lpr = 1 << lpr_log2, rpw = 32 >> lpr_log2, S = MV_WARPS * rpw, h = lpr >> 1;
    const int jc = lane & (lpr - 1), slot = jc & (h - 1);
    const bool upper = jc & h;
    const float sca = slice_scale(wa.eb + (8 - PF)), scb = slice_scale(wb.eb + (8 - PF));      // P = 3 products are half as large
    const ulonglong2* cx = sx + jc * CX;
    int r = st * rpw + (lane >> lpr_log2), cnt = 0;
    float keep = 0.0f;
    auto flush = [&](int st0, int r0) {      // the kept items' results; st0, r0: the first one's
        if (MODE == MODE_GU) {
            const float su = __shfl_xor_sync(0xFFFFFFFFu, keep, h);
            const int row = r0 + slot * S;
            if (!upper && slot < cnt && row < R) store(row, keep * sca, su * scb);
        } else {
            const int e = 2 * slot + (upper ? 1 : 0), row = r0 + e * S;
            if (slot < cnt && st0 + e * MV_WARPS < s_hi && row < R) store(row, keep * sca, 0.0f);
        }
    };
    for (; st < s_hi; st += STEPS * MV_WARPS, r += STEPS * S) {
        Chunk na, nb;
        load_item<MODE, PF>(wa, wb, st + STEPS * MV_WARPS, r + STEPS * S, s_hi, R, lpr_log2, jc, na, nb);
        u64 acc[2] = {0ull, 0ull};
        if (r < R) {
            if (MODE == MODE_GU || st + MV_WARPS < s_hi) chunk_dots<MODE_GU, PF>(tab, kc, ka, kb, cx, acc[0], acc[1]);
            else chunk_dots<MODE_ROUND, PF>(tab, kc, ka, kb, cx, acc[0], acc[1]);
        }
        const float v[2] = {pair_total(acc[0]), pair_total(acc[1])};
        if (lpr == 1) {      // rows of one chunk: every lane has its rows' sums
            if (r < R) store(r, v[0] * sca, MODE == MODE_GU ? v[1] * scb : 0.0f);
            if (MODE != MODE_GU && st + MV_WARPS < s_hi && r + S < R) store(r + S, v[1] * sca, 0.0f);
        } else {
            const float mine = split_sum<2>(v, lpr, jc);
            if (slot == cnt) keep = mine;
            if (++cnt == h) {
                flush(st - (h - 1) * STEPS * MV_WARPS, r - (h - 1) * STEPS * S);
                cnt = 0;
            }
        }
        ka = na;
        kb = nb;
    }
    if (cnt) flush(st - cnt * STEPS * MV_WARPS, r - cnt * STEPS * S);
}

// Rows of any other number of chunks: a row is cut into groups of lpr chunks (item_shape), a group's sum is the butterfly over its
// lanes, the row's the groups' sum in order.
constexpr int PART_FLOATS = 4096, PART_FLOATS_MIN = 2048;      // groups' sums that wait in shared memory, if the inputs leave room for them (the longest rows: at least the ch floats of a step of 8 lanes a row)
__host__ __device__ __forceinline__ int part_steps(int floats, int groups, int lpr_log2, int mats) { return floats / (groups * (32 >> lpr_log2) * mats); }

// The router in a kernel's prologue: warp t picks token t's top-k experts; block 0 also stores ids and weights for the kernels that
// follow.  Ends with a barrier.
__device__ __forceinline__ void route_prologue(const RouteFuse& rf, int32_t* r_ind, float* r_wt) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (warp < rf.T) {
        const float* l = rf.logits + (size_t) warp * rf.ld;
        if (rf.n_exp <= 128) route_row<4>(rf.n_exp, rf.top_k, l, lane, r_ind + warp * rf.top_k, r_wt + warp * rf.top_k);
        else if (rf.n_exp <= 512) route_row<16>(rf.n_exp, rf.top_k, l, lane, r_ind + warp * rf.top_k, r_wt + warp * rf.top_k);
        else route_row<32>(rf.n_exp, rf.top_k, l, lane, r_ind + warp * rf.top_k, r_wt + warp * rf.top_k);
    }
    __syncthreads();
    if (blockIdx.x == 0 && (int) threadIdx.x < rf.T * rf.top_k) {
        rf.ind_out[threadIdx.x] = r_ind[threadIdx.x];
        rf.wt_out[threadIdx.x] = r_wt[threadIdx.x];
    }
}

// ---- one expansion per pair, inputs in shared memory, one block of 16 warps per SM -----------------------------------------
// Rows of 1, 2, 4 .. 32 chunks.  The work is the pair-major sequence of items (RowItem); blocks take contiguous equal
// shares of it, and a block's warps fetch its items one by one from a counter in shared memory: the schedulers favour some warps,
// and with items dealt in advance the favoured ones left the others alone for the last third of the launch (13.5 of 16 warps
// active on average).  Inputs, stream addresses and scales of up to PAIR_WIN pairs are staged at a time.
// Bound: the logic pipe (38 LOP3 + 4 PRMT + 2 SHF a block of 8 weights) together with the register file's read ports (a packed
// multiply-add reads three register pairs, three cycles alone, 2.4 with one of them shared by neighbours): the arithmetic
// alone runs at 0.875 clk a block and SM (16 warps, a loop without streams).
// Optionally the block first ROUTES: with logits given, warp t picks token t's top-k experts (route.cuh) and the pair
// list is the T * top_k (token, expert) pairs.
// PF: coefficients per block.  4: SEED4P4; 3: SEED4 (24 states, the nibble word).
constexpr int PAIR_WARPS = 16, PAIR_THREADS = 32 * PAIR_WARPS, PAIR_WIN = 8;

struct PairDesc {      // what an item needs of its pair
    const void *sa, *ca, *da, *sb, *cb, *db;
    float sca, scb;
    int pair, any;      // any: bit 0 / 1: the first / second matrix's streams are not 16-byte aligned (mv_items_kernel, P = 3)
};

// ONE: rows of one chunk (lpr_log2 = 0), a form of its own: the branch in the loop of the others cost config 1 at 8 rows 5 %.
// SINGLE: an item of the one matrix is one row step, not two: small calls, whose warps would not all have an item.  (Two steps one after the
// other beside idle warps: 3 pairs of 1024 / 256 13.8 us a layer, 12.7 with one.)
template <int MODE, int PF, bool ONE, bool SINGLE>
__global__ void __launch_bounds__(PAIR_THREADS, 1) mv_pair_kernel(MvParams a, KConst kc, int lpr_log2, int win, RouteFuse rf) {
    constexpr bool TWO = MODE != MODE_GU && !SINGLE;
    extern __shared__ __align__(16) ulonglong2 pair_sx[];      // [win][lpr * CX]
    __shared__ StreamTab tab;
    __shared__ int32_t r_ind[256];   // the fused router's picks
    __shared__ float r_wt[256];
    __shared__ PairDesc desc[PAIR_WIN];
    __shared__ int next_item;
    constexpr int STEPS = TWO ? 2 : 1;
    tab_and_wait(tab, a.G, a.late, threadIdx.x, PAIR_THREADS);   // everything below may read what the previous kernel in the stream wrote
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lpr = 1 << lpr_log2, rpw = 32 >> lpr_log2, h = lpr >> 1;
    const int jc = lane & (lpr - 1), ro = lane >> lpr_log2, slot = jc & (h - 1);
    const bool upper = jc & h;
    int P = a.count ? min(*a.count, a.P) : a.P;
    if (rf.logits) {
        route_prologue(rf, r_ind, r_wt);
        P = rf.T * rf.top_k;
    }
    const int rs = (a.R + rpw - 1) / rpw, ips = (rs + STEPS - 1) / STEPS;      // row steps, items of a pair
    const long long total = (long long) P * ips;
    const long long begin = (long long) blockIdx.x * total / gridDim.x, end = (long long) (blockIdx.x + 1) * total / gridDim.x;
    if (begin >= end) return;
    const float inv = 1.0f / (float) ips;
    const ulonglong2* const cx0 = pair_sx + jc * CX;
    for (int p0 = (int) (begin / ips); (long long) p0 * ips < end; p0 += win) {
        // items of this window, counted from pair p0's first: [lo, hi)
        const int lo = (int) (begin - (long long) p0 * ips > 0 ? begin - (long long) p0 * ips : 0);
        const int hi = (int) (end - (long long) p0 * ips < (long long) win * ips ? end - (long long) p0 * ips : (long long) win * ips);
        const int np = (hi + ips - 1) / ips;
        __syncthreads();      // the previous window is no longer read
        if ((int) threadIdx.x < np) {
            const int pair = p0 + threadIdx.x, slice = rf.logits ? r_ind[pair] : (a.sel ? a.sel[pair] : 0);
            const WSlice wa = a.ws ? a.ws[slice] : a.w0;
            PairDesc d = {wa.p[0], wa.p[1], wa.p[3], NULL, NULL, NULL, slice_scale(wa.eb + (8 - PF)), 0.0f, pair, 0};      // P = 3 products are half as large
            if (MODE == MODE_GU) {
                const WSlice wb = a.wu[slice];
                d.sb = wb.p[0]; d.cb = wb.p[1]; d.db = wb.p[3];
                d.scb = slice_scale(wb.eb + (8 - PF));
            }
            desc[threadIdx.x] = d;
        }
        if (threadIdx.x == PAIR_THREADS - 1) next_item = lo + PAIR_WARPS;
        for (int i = threadIdx.x; i < np * lpr * 4; i += PAIR_THREADS) {
            const int t = i >> (lpr_log2 + 2), e = i - (t << (lpr_log2 + 2)), pair = p0 + t;
            float x[16];
            stage_load(input_row(a, a.xrow ? a.xrow[pair] : pair / a.xdiv), a.xbf16, e >> 2, e & 3, x);
            stage_store<PF>(x, e >> 2, e & 3, pair_sx + (size_t) t * lpr * CX);
        }
        __syncthreads();      // (and, the first time, the stream table is loaded)
        auto locate = [&](int it, int& t, int& r) {      // item -> its pair in the window, this lane's first row
            t = (int) ((float) it * inv);
            if (t * ips > it) --t;
            if ((t + 1) * ips <= it) ++t;
            r = (it - t * ips) * (STEPS * rpw) + ro;
        };
        auto load = [&](int it, Chunk& ka, Chunk& kb) {
            int t, r;
            locate(it, t, r);
            if (it >= hi || r >= a.R) return;
            const PairDesc& d = desc[t];
            const uint32_t at = (uint32_t) ((r << lpr_log2) + jc);
            ka.s = __ldg((const uint4*) d.sa + at);
            ka.c = __ldg((const uint4*) d.ca + at);
            if (PF == 4) ka.cd = __ldg((const uint32_t*) d.da + at);
            if (MODE == MODE_GU) {
                kb.s = __ldg((const uint4*) d.sb + at);
                kb.c = __ldg((const uint4*) d.cb + at);
                if (PF == 4) kb.cd = __ldg((const uint32_t*) d.db + at);
            } else if (TWO && r + rpw < a.R) {
                kb.s = __ldg((const uint4*) d.sa + at + 32);      // the next row step: 32 chunks on
                kb.c = __ldg((const uint4*) d.ca + at + 32);
                if (PF == 4) kb.cd = __ldg((const uint32_t*) d.da + at + 32);
            }
        };
        // The sums stay in the lanes that finish them until every lane has one: SwiGLU, rounding and stores then run once for
        // lpr / 2 items (once an item, with one lane in work, they and the reductions took 17 of 90 instructions a block).
        float keep = 0.0f;
        int kept = -1, cnt = 0;      // kept: the item's number
        auto flush = [&]() {
            int t, r;
            locate(kept < 0 ? lo : kept, t, r);
            const PairDesc& d = desc[t];
            if (MODE == MODE_GU) {
                const float su = __shfl_xor_sync(0xFFFFFFFFu, keep, h);
                if (!upper && kept >= 0 && r < a.R) store_out<MODE>(a, d.pair, r, keep * d.sca, su * d.scb);
            } else {
                r += TWO && upper ? rpw : 0;
                if (kept >= 0 && (TWO || !upper) && r < a.R) store_out<MODE>(a, d.pair, r, keep * d.sca, 0.0f);
            }
            kept = -1;
            cnt = 0;
        };
        int it = lo + warp;
        Chunk ka, kb;
        load(it, ka, kb);
        while (it < hi) {
            int nx = 0;
            if (lane == 0) nx = atomicAdd(&next_item, 1);
            nx = __shfl_sync(0xFFFFFFFFu, nx, 0);
            Chunk na, nb;
            load(nx, na, nb);
            int t, r;
            locate(it, t, r);
            u64 acc[2] = {0ull, 0ull};
            if (r < a.R) {
                const ulonglong2* cx = cx0 + t * (lpr * CX);
                if (MODE == MODE_GU || (TWO && (it - t * ips + 1) * STEPS <= rs)) chunk_dots<MODE_GU, PF>(tab, kc, ka, kb, cx, acc[0], acc[1]);
                else chunk_dots<MODE_ROUND, PF>(tab, kc, ka, kb, cx, acc[0], acc[1]);      // (a pair's last, single step)
            }
            const float v[2] = {pair_total(acc[0]), pair_total(acc[1])};
            if (ONE) {      // rows of one chunk: every lane has its rows' sums (two lanes a row in mv_items_kernel, one idle: 1300 pairs of 640 rows 103 / 55 us)
                const PairDesc& d = desc[t];
                if (r < a.R) store_out<MODE>(a, d.pair, r, v[0] * d.sca, MODE == MODE_GU ? v[1] * d.scb : 0.0f);
                if (MODE != MODE_GU && r + rpw < a.R) store_out<MODE>(a, d.pair, r + rpw, v[1] * d.sca, 0.0f);
                it = nx;
                ka = na;
                kb = nb;
                continue;
            }
            const float mine = split_sum<2>(v, lpr, jc);
            if (slot == cnt) { keep = mine; kept = it; }
            if (++cnt == h) flush();
            it = nx;
            ka = na;
            kb = nb;
        }
        if (cnt) flush();
    }
}

// ---- the same for rows of any number of chunks ------------------------------------------------------------------------------
// An ITEM is one group of the 32 / lpr rows of a row step (or, with spi = 2, of two steps of the one matrix, which then share the inputs'
// loads), so the work is even to within one chunk a warp whatever the row's length; the warps fetch the items of a
// window of row steps one by one.  The groups' sums wait in shared memory until the window is done: the end of a window is a
// barrier, and a small call's share is one window.  (Two blocks of 8 warps an SM with the items dealt in advance: 47.9 us
// for 5 rows, top 4, of a layer 1536 / 704 wide.)
template <int MODE, int PF>
__global__ void __launch_bounds__(PAIR_THREADS, 1) mv_items_kernel(MvParams a, KConst kc, RowShape sh, int win, int part_floats, int spi, RouteFuse rf) {
    extern __shared__ __align__(16) ulonglong2 pair_sx[];      // [win][ch * CX], then the sums
    __shared__ StreamTab tab;
    __shared__ int32_t r_ind[256];   // the fused router's picks
    __shared__ float r_wt[256];
    __shared__ PairDesc desc[PAIR_WIN];
    __shared__ int next_item;
    constexpr int MATS = MODE == MODE_GU ? 2 : 1;
    tab_and_wait(tab, a.G, a.late, threadIdx.x, PAIR_THREADS);   // everything below may read what the previous kernel in the stream wrote
    const int lane = threadIdx.x & 31, ch = sh.ch, groups = sh.groups;
    const int lpr = 1 << sh.lpr_log2, rpw = 32 >> sh.lpr_log2;
    const int jc = lane & (lpr - 1), ro = lane >> sh.lpr_log2;
    int P = a.count ? min(*a.count, a.P) : a.P;
    if (rf.logits) {
        route_prologue(rf, r_ind, r_wt);
        P = rf.T * rf.top_k;
    }
    float* const part = (float*) (pair_sx + (size_t) win * ch * CX);
    const int rs = (a.R + rpw - 1) / rpw, span = part_steps(part_floats, groups, sh.lpr_log2, MATS);
    const long long total = (long long) P * rs;
    const long long begin = (long long) blockIdx.x * total / gridDim.x, end = (long long) (blockIdx.x + 1) * total / gridDim.x;
    const float inv_rs = 1.0f / (float) rs, inv_groups = 1.0f / (float) groups;
    auto divide = [](int v, float inv, int d) {      // v / d for v < 2^23
        int q = (int) ((float) v * inv);
        if (q * d > v) --q;
        return (q + 1) * d <= v ? q + 1 : q;
    };
    for (long long w0 = begin; w0 < end;) {
        const int p0 = (int) (w0 / rs), lo = (int) (w0 - (long long) p0 * rs);      // the window's first pair, its first step there
        const long long most = (long long) win * rs - lo;
        const int n = (int) min(min(end - w0, (long long) span), most), np = (lo + n + rs - 1) / rs;
        const int items = (n + spi - 1) / spi * groups;
        if (w0 != begin) __syncthreads();      // the previous window is no longer read
        if ((int) threadIdx.x < np) {
            const int pair = p0 + threadIdx.x, slice = rf.logits ? r_ind[pair] : (a.sel ? a.sel[pair] : 0);
            const WSlice wa = a.ws ? a.ws[slice] : a.w0;
            PairDesc d = {wa.p[0], wa.p[1], wa.p[3], NULL, NULL, NULL, slice_scale(wa.eb + (8 - PF)), 0.0f, pair, 0};
            if (MODE == MODE_GU) {
                const WSlice wb = a.wu[slice];
                d.sb = wb.p[0]; d.cb = wb.p[1]; d.db = wb.p[3];
                d.scb = slice_scale(wb.eb + (8 - PF));
            }
            if (PF == 3) d.any = (int) !chunk_aligned(d.sa, d.ca) | (MODE == MODE_GU && !chunk_aligned(d.sb, d.cb) ? 2 : 0);
            desc[threadIdx.x] = d;
        }
        if (threadIdx.x == 0) next_item = PAIR_WARPS;
        for (int i = threadIdx.x; i < np * ch * 4; i += PAIR_THREADS) {
            const int t = i / (ch * 4), e = i - t * (ch * 4), pair = p0 + t;
            float x[16];
            stage_load(input_row(a, a.xrow ? a.xrow[pair] : pair / a.xdiv), a.xbf16, e >> 2, e & 3, x);
            stage_store<PF>(x, e >> 2, e & 3, pair_sx + (size_t) t * ch * CX);
        }
        __syncthreads();      // (and, the first time, the stream table is loaded)
        auto locate = [&](int k, int& t, int& r) {      // the window's step k -> its pair, this lane's row
            t = divide(lo + k, inv_rs, rs);
            r = (lo + k - t * rs) * rpw + ro;
        };
        auto fetch = [&](const void* sp, const void* cp, const void* dp, bool any, uint32_t at, Chunk& k) {
            if (PF == 3 && any) {
                k.s = load_any_16(sp, at);
                k.c = load_any_16(cp, at);
                return;
            }
            k.s = __ldg((const uint4*) sp + at);
            k.c = __ldg((const uint4*) cp + at);
            if (PF == 4) k.cd = __ldg((const uint32_t*) dp + at);
        };
        auto fetch_a = [&](const PairDesc& d, uint32_t at, Chunk& k) { fetch(d.sa, d.ca, d.da, d.any & 1, at, k); };
        struct At { int k, g, t, r; };      // an item: its (first) step, group, the step's pair, this lane's row
        auto load = [&](int it, At& at_it, Chunk& ka, Chunk& kb) {
            if (it >= items) return;
            const int u = divide(it, inv_groups, groups), g = it - u * groups, j = g * lpr + jc;
            int t, r;
            locate(u * spi, t, r);
            at_it = At{u * spi, g, t, r};
            if (j >= ch) return;
            if (r < a.R) {
                const PairDesc& d = desc[t];
                const uint32_t at = (uint32_t) (r * ch + j);
                fetch_a(d, at, ka);
                if (MODE == MODE_GU) fetch(d.sb, d.cb, d.db, d.any & 2, at, kb);
            }
            if (MODE != MODE_GU && spi == 2 && u * 2 + 1 < n) {
                locate(u * 2 + 1, t, r);
                if (r < a.R) fetch_a(desc[t], (uint32_t) (r * ch + j), kb);
            }
        };
        int it = threadIdx.x >> 5;
        Chunk ka, kb;
        At cur = {0, 0, 0, 0};
        load(it, cur, ka, kb);
        while (it < items) {
            int nx = 0;
            if (lane == 0) nx = atomicAdd(&next_item, 1);
            nx = __shfl_sync(0xFFFFFFFFu, nx, 0);
            Chunk na, nb;
            const At now = cur;
            load(nx, cur, na, nb);
            const int k = now.k, g = now.g, t = now.t, r = now.r, j = g * lpr + jc;
            u64 acc[2] = {0ull, 0ull};
            const ulonglong2* const cx = pair_sx + (size_t) (t * ch + j) * CX;
            const bool two = MODE != MODE_GU && spi == 2 && k + 1 < n;
            int t2 = t, r2 = r;
            if (two) locate(k + 1, t2, r2);
            if (j < ch) {
                if (MODE == MODE_GU) {
                    if (r < a.R) chunk_dots<MODE_GU, PF>(tab, kc, ka, kb, cx, acc[0], acc[1]);
                } else if (two && t2 == t) {      // (r2 > r; a row that is not there: whatever the registers hold, never stored)
                    if (r < a.R) chunk_dots<MODE_GU, PF>(tab, kc, ka, kb, cx, acc[0], acc[1]);
                } else {
                    if (r < a.R) chunk_dots<MODE_ROUND, PF>(tab, kc, ka, ka, cx, acc[0], acc[1]);
                    if (two && r2 < a.R) chunk_dots<MODE_ROUND, PF>(tab, kc, kb, kb, pair_sx + (size_t) (t2 * ch + j) * CX, acc[1], acc[0]);
                }
            }
            const float v[2] = {pair_total(acc[0]), pair_total(acc[1])};
            const float mine = split_sum<2>(v, lpr, jc);      // value 0 ends in the row's lower lanes, value 1 in the upper ones
            if (MODE == MODE_GU) {
                if ((jc & (lpr / 2 - 1)) == 0) part[((k * rpw + ro) * groups + g) * 2 + (jc ? 1 : 0)] = mine;
            } else if (jc == 0 || (two && jc == lpr / 2)) part[((k + (jc ? 1 : 0)) * rpw + ro) * groups + g] = mine;
            it = nx;
            ka = na;
            kb = nb;
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n * rpw; i += PAIR_THREADS) {
            const int k = i >> (5 - sh.lpr_log2), t = divide(lo + k, inv_rs, rs), r = (lo + k - t * rs) * rpw + (i & (rpw - 1));
            const float* const at = part + (size_t) i * groups * MATS;
            float s = at[0], su = MODE == MODE_GU ? at[1] : 0.0f;
            for (int q = 1; q < groups; ++q) {
                s += at[q * MATS];
                if (MODE == MODE_GU) su += at[q * MATS + 1];
            }
            if (r < a.R) store_out<MODE>(a, desc[t].pair, r, s * desc[t].sca, su * desc[t].scb);
        }
        w0 += n;
    }
}


// ---- the whole decode step of an expert layer in one launch -----------------------------------------------------------------
// Router, gate + up + SwiGLU, down projection and weighted combine as three phases of one grid of two blocks an SM, instead
// of three dependent launches: a launch boundary costs the step its predecessor's tail (the last blocks' row steps with
// the other SMs idle), the successor's ramp and the prologue (stream table, router) again, ~4 us each on a step of
// 26 .. 114 us.  Here a block that has finished its share of a phase starts on the next one at once; what it needs from
// other blocks it waits for on counters in device memory:
//   ready[p]  row steps of pair p's gate + up rows stored           (the down projection of pair p reads all of them)
//   done[t]   row steps of token t's down projections stored        (the combine of token t reads all top_k of them)
// Each phase is the pair kernel's: the pair-major sequence of row steps cut into contiguous equal shares, so block b
// works on the same pairs in phases 1 and 2 and waits for its neighbours b - 1 and b + 1 at most; blocks are dispatched
// in index order and no block waits for a higher-numbered block other than b + 1 before it has finished phase 2, so the
// grid makes progress even when not all of it is resident.  Every wait is bounded: when one runs out the block records
// status 1, every other wait ends on seeing it, and the launch returns with its counters cleared (the last block to
// finish clears them for the next launch; fin counts finished blocks and wraps to zero by itself).
// Arithmetic and rounding points are those of the three kernels it replaces, operation for operation.
// Measured (config 1, us per step at 8 / 4 / 1 rows): 119 / 65 / 24.8 against 98.8 / 56.9 / 23.7 for the three dependent launches, so the
// host layer does not use it by default.  It keeps the blocks of 8 warps with row steps dealt in advance that the pair kernel had (the
// same 75.0 M instructions then; 126 against 114 us), and at each phase change a block waits for the slowest of the ~6 blocks that share
// its pairs (barrier stalls 0.78 per issued instruction against 0.10).
struct StepSync {
    unsigned* ready;      // [T * top_k]
    unsigned* done;       // [T]
    unsigned* fin;
    int* status;
};
struct StepParams {
    const WSlice *wg, *wu, *wd;
    const float* x;       // [T][d]
    const float* logits;  // [T][ld]
    float* A;             // [T * top_k][ff]
    float* D;             // [T * top_k][d]
    float* out;           // [T][d]
    int32_t* ind_out;
    float* wt_out;
    const uint32_t* G;
    int xs, ld, n_exp, top_k, T, d, ff, raw;
    StepSync sy;
};
constexpr unsigned STEP_WAIT_LIMIT = 1u << 19;      // polls of ~0.1 us

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
// false: the limit ran out, or another block has reported that its wait did
__device__ __forceinline__ bool step_wait(const unsigned* counter, unsigned target, int* status) {
    for (unsigned i = 0; i < STEP_WAIT_LIMIT; ++i) {
        if (ld_acquire(counter) >= target) return true;
        if ((i & 63u) == 63u && *(volatile int*) status) return false;
        __nanosleep(i < 16 ? 32 : 128);
    }
    atomicCAS(status, 0, 1);
    return false;
}

struct StepShared {
    StreamTab tab;
    int32_t r_ind[256];
    float r_wt[256];
    __align__(16) ulonglong2 sx[32 * CX];
    int abort;
};

// One phase: MODE_GU (x -> A, signals ready[pair]) or MODE_ROUND (A -> D, waits for ready[pair], signals done[token]).
template <int MODE>
__device__ __forceinline__ void step_phase(const StepParams& p, const KConst& kc, StepShared& sh, int P, int lpr_log2, unsigned rs_gu) {
    const int R = MODE == MODE_GU ? p.ff : p.d;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lpr = 1 << lpr_log2, rpw = 32 >> lpr_log2;
    const int jc = lane & (lpr - 1), ro = lane >> lpr_log2;
    const int rs = (R + rpw - 1) / rpw;
    const long long total = (long long) P * rs;
    const long long begin = (long long) blockIdx.x * total / gridDim.x, end = (long long) (blockIdx.x + 1) * total / gridDim.x;
    if (begin >= end) return;
    const int p_first = (int) (begin / rs), p_last = (int) ((end - 1) / rs);
    MvParams a = {};
    a.y = MODE == MODE_GU ? p.A : p.D;
    a.ys = R;
    a.R = R;
    a.raw = p.raw;
    for (int pair = p_first; pair <= p_last; ++pair) {
        const int s_lo = pair == p_first ? (int) (begin - (long long) pair * rs) : 0;
        const int s_hi = pair == p_last ? (int) (end - (long long) pair * rs) : rs;
        const int slice = sh.r_ind[pair];
        const WSlice wa = MODE == MODE_GU ? p.wg[slice] : p.wd[slice];
        WSlice wb = wa;
        if (MODE == MODE_GU) wb = p.wu[slice];
        int st = s_lo + warp;
        int r = st * rpw + ro;
        Chunk ka, kb;
        load_item<MODE, 4>(wa, wb, st, r, s_hi, R, lpr_log2, jc, ka, kb);      // the streams do not depend on other blocks: requested before any wait
        if (MODE == MODE_ROUND && threadIdx.x == 0 && !step_wait(p.sy.ready + pair, rs_gu, p.sy.status)) sh.abort = 1;
        __syncthreads();   // the previous pair's inputs are no longer read; the wait's outcome is known
        if (sh.abort) return;
        if (threadIdx.x < lpr * 4) {
            float x[16];
            if (MODE == MODE_GU) stage_load(p.x + (size_t) (pair / p.top_k) * p.xs, 0, threadIdx.x >> 2, threadIdx.x & 3, x);
            else stage_load<true>(p.A + (size_t) pair * p.ff, 0, threadIdx.x >> 2, threadIdx.x & 3, x);
            stage_store<4>(x, threadIdx.x >> 2, threadIdx.x & 3, sh.sx);
        }
        __syncthreads();
        pair_rows<MODE, 4>(sh.tab, kc, wa, wb, sh.sx, lpr_log2, R, st, s_hi, ka, kb,
                                  [&](int rr, float s, float su) { store_out<MODE>(a, pair, rr, s, su); });
        // this block's row steps of the pair are stored: publish their number
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) atomicAdd(MODE == MODE_GU ? p.sy.ready + pair : p.sy.done + pair / p.top_k, (unsigned) (s_hi - s_lo));
    }
}

__global__ void __launch_bounds__(MV_THREADS, 2) mv_step_kernel(StepParams p, KConst kc, int lg_d, int lg_ff) {
    __shared__ StepShared sh;
    load_stream_tab(sh.tab, p.G, threadIdx.x, MV_THREADS);
    if (threadIdx.x == 0) sh.abort = 0;
    grid_dependents_go();
    grid_dependency_wait();   // everything below may read what the previous kernel in the stream wrote
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int P = p.T * p.top_k;
    if (warp < p.T) {         // the router: one warp per token, every block the same picks; block 0 stores them
        const float* l = p.logits + (size_t) warp * p.ld;
        if (p.n_exp <= 128) route_row<4>(p.n_exp, p.top_k, l, lane, sh.r_ind + warp * p.top_k, sh.r_wt + warp * p.top_k);
        else if (p.n_exp <= 512) route_row<16>(p.n_exp, p.top_k, l, lane, sh.r_ind + warp * p.top_k, sh.r_wt + warp * p.top_k);
        else route_row<32>(p.n_exp, p.top_k, l, lane, sh.r_ind + warp * p.top_k, sh.r_wt + warp * p.top_k);
    }
    __syncthreads();
    if (blockIdx.x == 0 && (int) threadIdx.x < P) {
        p.ind_out[threadIdx.x] = sh.r_ind[threadIdx.x];
        p.wt_out[threadIdx.x] = sh.r_wt[threadIdx.x];
    }
    const unsigned rs_gu = (unsigned) ((p.ff + (32 >> lg_d) - 1) / (32 >> lg_d));      // row steps of a pair's gate + up rows
    step_phase<MODE_GU>(p, kc, sh, P, lg_d, rs_gu);
    if (!sh.abort) step_phase<MODE_ROUND>(p, kc, sh, P, lg_ff, rs_gu);
    // combine: out[t][i] = sum_j wt[t][j] D[t * k + j][i], plain f32, j ascending (q4_combine_kernel's sum); item = (token, 256 columns)
    if (!sh.abort) {
        const int cpr = (p.d + MV_THREADS - 1) / MV_THREADS, rpw_d = 32 >> lg_ff;
        const unsigned rs_down = (unsigned) ((p.d + rpw_d - 1) / rpw_d) * (unsigned) p.top_k;
        for (int item = blockIdx.x; item < p.T * cpr; item += gridDim.x) {
            const int t = item / cpr, i = (item - t * cpr) * MV_THREADS + (int) threadIdx.x;
            if (threadIdx.x == 0 && !step_wait(p.sy.done + t, rs_down, p.sy.status)) sh.abort = 1;
            __syncthreads();
            if (sh.abort) break;
            if (i < p.d) {
                float acc = 0.0f;
                for (int j = 0; j < p.top_k; ++j) acc += sh.r_wt[t * p.top_k + j] * __ldcg(p.D + ((size_t) t * p.top_k + j) * p.d + i);
                p.out[(size_t) t * p.d + i] = acc;
            }
        }
    }
    // the last block to finish clears the counters for the next launch
    __syncthreads();
    if (threadIdx.x == 0) sh.abort = atomicInc(p.sy.fin, gridDim.x - 1) == gridDim.x - 1 ? 2 : 0;
    __syncthreads();
    if (sh.abort == 2) {
        for (int i = threadIdx.x; i < P; i += MV_THREADS) p.sy.ready[i] = 0u;
        for (int i = threadIdx.x; i < p.T; i += MV_THREADS) p.sy.done[i] = 0u;
    }
}


// ---- pairs grouped by expert: one expansion per distinct slice ---------------------------------------------------------
// Rows of 4, 8, 16 or 32 chunks (K = 256 .. 2048: grp_serves).  Every block builds the same plan in its prologue: the pair list is
// sorted by slice in shared memory, runs of pairs that use the same slice are cut into UNITS of at most GRP_NT pairs, and
// a unit's rows are expanded once for all its pairs (the logic-pipe work is shared; each pair keeps its own sums, formed in
// the same order as when it is alone, so a pair's result does not depend on its partners).  The work is the sequence of
// (unit, row step) items, an item of a unit with n pairs weighing GRP_W[n]; blocks take contiguous equal shares of the
// weighted sequence.  A block stages the inputs of as many of its units as GRP_SLOTS pairs are; its 16 warps then fetch the
// items (RowItem) of the two-pair units and after them those of the single ones one by one, as in the pair kernel.
constexpr int GRP_NT = 2;                         // pairs that share one expansion at most
constexpr int GRP_MAX_PAIRS = 1024;               // pairs a block can sort; longer lists run ungrouped
constexpr int GRP_SMALL = 128;                    // lists up to this length are ranked by counting (no sorting network)
__device__ constexpr int GRP_W[GRP_NT + 1] = {0, 8, 12};   // relative cost of a row step for a unit of n pairs
constexpr int GRP_SX = 32 * CX;                    // one pair's staged inputs
constexpr int GRP_SLOTS = 12;                     // pairs staged at a time (a share of the longest sorted list is 7 and two parts)
constexpr int GRP_WARPS = 16, GRP_THREADS = 32 * GRP_WARPS;

struct GrpUnit {      // what an item needs of its unit
    const uint4 *sa, *ca, *sb, *cb;
    const uint32_t *da, *db;
    float sca, scb;
    int pid[2];                                    // its pairs
    int slot, s_lo, s_hi;                          // its first pair's staged inputs; the block's row steps of it
};
struct GrpShared {
    StreamTab tab;
    uint32_t key[GRP_MAX_PAIRS];                  // sorted (slice << 10 | pair)
    int32_t prefix[GRP_MAX_PAIRS + 1];            // weight of the units that start before sorted position i
    uint32_t tmp[GRP_SMALL];                      // short lists: unsorted keys, then unit weights
    GrpUnit unit[GRP_NT][GRP_SLOTS];              // the window's units of 1, 2 pairs ...
    int start[GRP_NT][32];                        // ... their first items (beyond the last unit: never reached)
    int next[GRP_NT];                             // the next item to fetch
    int slot_pair[GRP_SLOTS];
    __align__(16) ulonglong2 sx[GRP_SLOTS][GRP_SX];
};


// The state-value pairs of weights 4H .. 4H+3 of two adjacent blocks (half of a pair's): v[4 (c - 4H) + p].
template <int H>
__device__ __forceinline__ void half_states(const Words& wa, const Words& wb, u64* v) {
#define NSL_VH(C)                                                                                \
    {                                                                                            \
        constexpr int B = state_bit<4, C>(), W = 2 * H + C / 2;                                  \
        v[4 * C + 0] = pack2(state_at<B, 0>(wa.w[W]), state_at<B, 0>(wb.w[W]));                  \
        v[4 * C + 1] = pack2(state_at<B, 1>(wa.w[W]), state_at<B, 1>(wb.w[W]));                  \
        v[4 * C + 2] = pack2(state_at<B, 2>(wa.w[W]), state_at<B, 2>(wb.w[W]));                  \
        v[4 * C + 3] = pack2(state_at<B, 3>(wa.w[W]), state_at<B, 3>(wb.w[W]));                  \
    }
    NSL_VH(0) NSL_VH(1) NSL_VH(2) NSL_VH(3)
#undef NSL_VH
}
// One half of a block pair (weights 4H .. 4H+3) against every pair's inputs.
template <int NT, int H>
__device__ __forceinline__ void unit_half(const Words& wa, const Words& wb, int bp, const ulonglong2* const* cx, u64 (*d)[4]) {
    u64 v[16];
    half_states<H>(wa, wb, v);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
#pragma unroll
        for (int cq = 0; cq < 2; ++cq) {
            const ulonglong2 u = cx[t][bp * 4 + 2 * H + cq];
#pragma unroll
            for (int p = 0; p < 4; ++p) d[t][p] = fma2(u.x, v[8 * cq + p], d[t][p]);
#pragma unroll
            for (int p = 0; p < 4; ++p) d[t][p] = fma2(u.y, v[8 * cq + 4 + p], d[t][p]);
        }
    }
}
// One row step of one matrix for NT pairs: each block pair is expanded once, half of its weights at a time (so that only
// 16 state-value pairs are held while every pair's inputs pass), and dotted with every pair's inputs.  Per pair the
// operations and their order are those of pair_expand_dot.
template <int NT>
__device__ __forceinline__ void unit_chunk(const StreamTab& tab, const KConst& kc, const Chunk& k, const ulonglong2* const* cx, u64* acc) {
    const uint32_t sw[4] = {k.s.x, k.s.y, k.s.z, k.s.w}, cw[4] = {k.c.x, k.c.y, k.c.z, k.c.w};
#pragma unroll
    for (int bp = 0; bp < 4; ++bp) {
        uint32_t g0, g1;
        pair_stream(tab, sw[bp], g0, g1);
        const Words wa = window_words<4, 0>(sw[bp], g0), wb = window_words<4, 1>(sw[bp], g1);
        u64 d[NT][4];
#pragma unroll
        for (int t = 0; t < NT; ++t) offsets_from_sum(staged_sum(cx[t], bp), d[t]);
        unit_half<NT, 0>(wa, wb, bp, cx, d);
        unit_half<NT, 1>(wa, wb, bp, cx, d);
        u64 q[4];
        pair_coefs(cw[bp], kc, q);
        const u64 e2 = code_scale_pair(k.cd, bp, kc);
#pragma unroll
        for (int t = 0; t < NT; ++t)
            acc[t] = fma2(fma2(q[3], d[t][3], fma2(q[2], d[t][2], fma2(q[1], d[t][1], mul2(q[0], d[t][0])))), e2, acc[t]);
    }
}

template <int MODE>
__device__ __forceinline__ void store_unit(const UnitCall& uc, int pair, int r, float s, float su) {
    float* yo = uc.y + (size_t) pair * uc.ys + r;
    if (MODE == MODE_GU) *yo = uc.raw ? (s / (1.0f + expf(-s))) * su : bf16_round(silu_bf(bf16_round(s)) * bf16_round(su));
    else if (uc.raw) *yo = s;
    else *yo = uc.add ? bf16_round(*yo + bf16_round(s)) : bf16_round(s);   // engine/kernels_moe.cu:214
}

// The items of the window's units of NT pairs, fetched one by one by the block's warps.
template <int MODE, int NT>
__device__ __noinline__ void unit_items(UnitCall uc) {
    // Not inlined on purpose: each unit size gets a register allocation of its own (inlined into one body, the larger
    // size's pressure spilled the single-pair loop too).  Shared memory and the constants are reached by name.
    static_assert(NT == 1 || NT == 2, "units of one or two pairs");
    extern __shared__ __align__(16) unsigned char grp_smem[];
    GrpShared& sh = *reinterpret_cast<GrpShared*>(grp_smem);
    const KConst& kc = c_kc;
    constexpr int STEPS = RowItem<MODE>::STEPS;
    const int lane = threadIdx.x & 31, lpr_log2 = uc.lpr_log2;
    const int lpr = 1 << lpr_log2, rpw = 32 >> lpr_log2;
    const int jc = lane & (lpr - 1), ro = lane >> lpr_log2;
    // an item's 2 NT sums (pair by pair: A, B) end in lpr / (2 NT) = h lanes of the row each, and stay there until each has one
    const int h = lpr / (2 * NT), slot = jc & (h - 1), part = jc / h;
    const int my_start = sh.start[NT - 1][lane];
    auto fetch = [&]() {
        int i = 0;
        if (lane == 0) i = atomicAdd(&sh.next[NT - 1], 1);
        return __shfl_sync(0xFFFFFFFFu, i, 0);
    };
    int u, st;      // the current item's unit and first row step
    auto locate = [&](int it) {
        u = __popc(__ballot_sync(0xFFFFFFFFu, my_start <= it)) - 1;
        st = sh.unit[NT - 1][u].s_lo + (it - __shfl_sync(0xFFFFFFFFu, my_start, u)) * STEPS;
    };
    auto load_a = [&](Chunk& k, const GrpUnit& d, int r) {
        if (r < uc.R) k = load_chunk3(d.sa, d.ca, d.da, (size_t) ((r << lpr_log2) + jc));
    };
    auto load_b = [&](Chunk& k, const GrpUnit& d, int s, int r) {
        if (MODE == MODE_GU) { if (r < uc.R) k = load_chunk3(d.sb, d.cb, d.db, (size_t) ((r << lpr_log2) + jc)); }
        else if (s + 1 < d.s_hi && r + rpw < uc.R) k = load_chunk3(d.sa, d.ca, d.da, (size_t) ((r << lpr_log2) + jc + 32));
    };
    float keep = 0.0f;
    int kept_u = 0, kept_r = 0, cnt = 0;
    auto flush = [&]() {
        const GrpUnit& d = sh.unit[NT - 1][kept_u];
        const int pid = part & 2 ? d.pid[1] : d.pid[0];
        if (MODE == MODE_GU) {
            const float su = __shfl_xor_sync(0xFFFFFFFFu, keep, h);
            if (!(part & 1) && slot < cnt && kept_r < uc.R) store_unit<MODE>(uc, pid, kept_r, keep * d.sca, su * d.scb);
        } else {
            const int r = kept_r + (part & 1 ? rpw : 0);
            if (slot < cnt && r < min(d.s_hi * rpw, uc.R)) store_unit<MODE>(uc, pid, r, keep * d.sca, 0.0f);
        }
        cnt = 0;
    };
    int it = fetch();
    if (it >= uc.items) return;
    Chunk ka, kb;
    locate(it);
    load_a(ka, sh.unit[NT - 1][u], st * rpw + ro);
    load_b(kb, sh.unit[NT - 1][u], st, st * rpw + ro);
    for (;;) {
        const int nx = fetch(), u0 = u, r = st * rpw + ro;
        const GrpUnit& d = sh.unit[NT - 1][u];
        const bool ok = r < uc.R, okb = ok && (MODE == MODE_GU || st + 1 < d.s_hi);
        const ulonglong2* const cx = sh.sx[d.slot] + jc * CX;
        const bool more = nx < uc.items;
        if (more) locate(nx);
        const GrpUnit& dn = sh.unit[NT - 1][u];
        const int rn = st * rpw + ro;
        float mine;
        if (NT == 1) {
            Chunk na, nb;
            if (more) { load_a(na, dn, rn); load_b(nb, dn, st, rn); }
            u64 acc[2] = {0ull, 0ull};
            if (okb) chunk_dots<MODE_GU, 4>(sh.tab, kc, ka, kb, cx, acc[0], acc[1]);
            else if (ok) chunk_dots<MODE_ROUND, 4>(sh.tab, kc, ka, kb, cx, acc[0], acc[1]);
            ka = na;
            kb = nb;
            const float v[2] = {pair_total(acc[0]), pair_total(acc[1])};
            mine = split_sum<2>(v, lpr, jc);
        } else {
            // the next item's streams are requested as soon as this item's have been used up, into the registers they leave free
            const ulonglong2* const cx2[2] = {cx, cx + GRP_SX};
            u64 acc[2] = {0ull, 0ull}, accb[2] = {0ull, 0ull};
            if (ok) unit_chunk<2>(sh.tab, kc, ka, cx2, acc);
            if (more) load_a(ka, dn, rn);
            if (okb) unit_chunk<2>(sh.tab, kc, kb, cx2, accb);
            if (more) load_b(kb, dn, st, rn);
            const float v[4] = {pair_total(acc[0]), pair_total(accb[0]), pair_total(acc[1]), pair_total(accb[1])};
            mine = split_sum<4>(v, lpr, jc);
        }
        if (slot == cnt) { keep = mine; kept_u = u0; kept_r = r; }
        if (++cnt == h) flush();
        if (!more) break;
    }
    if (cnt) flush();
}

// Ascending bitonic sort of n (a power of two) keys in shared memory by the whole block.
__device__ __forceinline__ void block_sort(uint32_t* key, int n) {
    for (int k = 2; k <= n; k <<= 1)
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = threadIdx.x; i < n; i += GRP_THREADS) {
                const int o = i ^ j;
                if (o > i) {
                    const uint32_t x = key[i], y = key[o];
                    if ((x > y) == ((i & k) == 0)) { key[i] = y; key[o] = x; }
                }
            }
            __syncthreads();
        }
}

// In-place exclusive prefix sum of a[0..n) by the whole block, a[n] = the total (n <= GRP_MAX_PAIRS).
__device__ __forceinline__ void block_exclusive_scan(int32_t* a, int n) {
    __shared__ int wtot[GRP_WARPS];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int per = (n + GRP_THREADS - 1) / GRP_THREADS, lo = threadIdx.x * per;      // a contiguous run per thread
    int sum = 0;
    for (int i = lo; i < lo + per && i < n; ++i) sum += a[i];
    int inc = sum;
    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xFFFFFFFFu, inc, o); if (lane >= o) inc += v; }
    if (lane == 31) wtot[warp] = inc;
    __syncthreads();
    int base = inc - sum;
    for (int w = 0; w < warp; ++w) base += wtot[w];
    for (int i = lo; i < lo + per && i < n; ++i) { const int v = a[i]; a[i] = base; base += v; }
    if (threadIdx.x == GRP_THREADS - 1) { int t = 0; for (int w = 0; w < GRP_WARPS; ++w) t += wtot[w]; a[n] = t; }
    __syncthreads();
}


template <int MODE>
__global__ void __launch_bounds__(GRP_THREADS, 1) mv_grp_kernel(MvParams a, KConst kc, int lpr_log2) {
    extern __shared__ __align__(16) unsigned char grp_smem[];
    GrpShared& sh = *reinterpret_cast<GrpShared*>(grp_smem);
    tab_and_wait(sh.tab, a.G, a.late, threadIdx.x, GRP_THREADS);   // everything below may read what the previous kernel in the stream wrote
    const int lpr = 1 << lpr_log2, rpw = 32 >> lpr_log2;
    int P = a.count ? min(*a.count, a.P) : a.P;
    if (P <= 0) return;
    const int rs = (a.R + rpw - 1) / rpw;             // row steps per unit
    const bool grouped = P <= GRP_MAX_PAIRS;
    long long total;
    if (grouped) {
        const bool small = P <= GRP_SMALL;
        auto slice_of = [&](int i) { return a.sel ? a.sel[i] : 0; };
        if (small) {      // every thread ranks one key among all: two barriers instead of a sorting network's dozens
            const int i = threadIdx.x;
            uint32_t mine = 0xFFFFFFFFu;
            if (i < P) {
                const int sl = slice_of(i);
                mine = ((uint32_t) sl << 10) | (uint32_t) i;
                sh.tmp[i] = mine;
                if (a.ws) {      // the slice's table entries on their way into L2 while the plan is made
                    asm volatile("prefetch.global.L2 [%0];" ::"l"(a.ws + sl));
                    if (MODE == MODE_GU) asm volatile("prefetch.global.L2 [%0];" ::"l"(a.wu + sl));
                }
            }
            __syncthreads();
            if (i < P) {
                int rank = 0;
                for (int j = 0; j < P; ++j) rank += sh.tmp[j] < mine;
                sh.key[rank] = mine;
            }
            __syncthreads();
        } else {
            int n = 32;
            while (n < P) n <<= 1;
            for (int i = threadIdx.x; i < n; i += GRP_THREADS) sh.key[i] = i < P ? ((uint32_t) slice_of(i) << 10) | (uint32_t) i : 0xFFFFFFFFu;
            __syncthreads();
            block_sort(sh.key, n);
        }
        // a sorted position starts a unit when it is a multiple of GRP_NT pairs into its slice's run
        for (int i = threadIdx.x; i < P; i += GRP_THREADS) {
            const uint32_t first = sh.key[i] & ~1023u;          // the smallest key of this slice
            int lo = 0, hi = i;                                  // lower bound of `first`
            while (lo < hi) { const int mid = (lo + hi) >> 1; if (sh.key[mid] < first) lo = mid + 1; else hi = mid; }
            int w = 0;
            if ((i - lo) % GRP_NT == 0) {
                int cnt = 1;
                while (cnt < GRP_NT && i + cnt < P && (sh.key[i + cnt] >> 10) == (sh.key[i] >> 10)) ++cnt;
                w = GRP_W[cnt];
            }
            if (small) sh.tmp[i] = (uint32_t) w; else sh.prefix[i] = w;
        }
        __syncthreads();
        if (small) {
            for (int i = threadIdx.x; i <= P; i += GRP_THREADS) {
                int before = 0;
                for (int j = 0; j < i; ++j) before += (int) sh.tmp[j];
                sh.prefix[i] = before;
            }
            __syncthreads();
        } else block_exclusive_scan(sh.prefix, P);
        total = (long long) sh.prefix[P] * rs;
    } else {
        __syncthreads();
        total = (long long) P * GRP_W[1] * rs;
    }
    const long long begin = (long long) blockIdx.x * total / gridDim.x, end = (long long) (blockIdx.x + 1) * total / gridDim.x;
    if (begin >= end) return;
    // position in the weighted sequence -> (sorted position of the unit's first pair, row step)
    auto locate = [&](long long x, int& u, int& step) {
        if (!grouped) { u = (int) (x / ((long long) GRP_W[1] * rs)); step = (int) ((x - (long long) u * GRP_W[1] * rs) / GRP_W[1]); return; }
        int lo = 0, hi = P;                                      // the last position whose prefix * rs <= x
        while (hi - lo > 1) { const int mid = (lo + hi) >> 1; if ((long long) sh.prefix[mid] * rs <= x) lo = mid; else hi = mid; }
        u = lo;
        step = (int) ((x - (long long) sh.prefix[lo] * rs) / (sh.prefix[lo + 1] - sh.prefix[lo]));
    };
    int u_first, s_first, u_last, s_last;
    locate(begin, u_first, s_first);
    if (end >= total) { u_last = P; s_last = 0; } else locate(end, u_last, s_last);
    auto unit_size = [&](int u) { return grouped && sh.prefix[u + 1] - sh.prefix[u] != GRP_W[1] ? 2 : 1; };
    auto pair_of = [&](int u, int t) { return grouped ? (int) (sh.key[u + t] & 1023u) : u; };
    if (u_first < P && s_first >= rs) { u_first += unit_size(u_first); s_first = 0; }
    constexpr int STEPS = RowItem<MODE>::STEPS;
    auto mine = [&](int u) { return u < P && (u < u_last || (u == u_last && s_last > 0)); };
    for (int u = u_first; mine(u);) {
        if (u != u_first) __syncthreads();      // the previous window is no longer read
        if (threadIdx.x < 32 * GRP_NT) sh.start[threadIdx.x >> 5][threadIdx.x & 31] = 0x7FFFFFFF;
        __syncthreads();
        int slots = 0, units[GRP_NT] = {0, 0}, items[GRP_NT] = {0, 0};
        for (; mine(u); ) {
            const int n = unit_size(u), s_lo = u == u_first ? s_first : 0, s_hi = u == u_last ? s_last : rs;
            if (slots + n > GRP_SLOTS) break;
            const int at = n == 2 ? units[1] : units[0];
            if ((int) threadIdx.x == 32 * slots) {      // one warp a unit: the slices' table entries arrive side by side
                const int slice = grouped ? (int) (sh.key[u] >> 10) : (a.sel ? a.sel[u] : 0);
                GrpUnit d;
                const WSlice wa = a.ws ? a.ws[slice] : a.w0;
                d.sa = (const uint4*) wa.p[0]; d.ca = (const uint4*) wa.p[1]; d.da = (const uint32_t*) wa.p[3];
                d.sca = d.scb = slice_scale(wa.eb + 4);
                d.sb = d.cb = NULL;
                d.db = NULL;
                if (MODE == MODE_GU) {
                    const WSlice wb = a.wu[slice];
                    d.sb = (const uint4*) wb.p[0]; d.cb = (const uint4*) wb.p[1]; d.db = (const uint32_t*) wb.p[3];
                    d.scb = slice_scale(wb.eb + 4);
                }
                d.pid[0] = sh.slot_pair[slots] = pair_of(u, 0);
                d.pid[1] = pair_of(u, n - 1);
                if (n == 2) sh.slot_pair[slots + 1] = d.pid[1];
                d.slot = slots; d.s_lo = s_lo; d.s_hi = s_hi;
                sh.unit[n - 1][at] = d;
                sh.start[n - 1][at] = n == 2 ? items[1] : items[0];
            }
            const int more = (s_hi - s_lo + STEPS - 1) / STEPS;
            if (n == 2) { ++units[1]; items[1] += more; } else { ++units[0]; items[0] += more; }
            slots += n;
            u += n;
        }
        if (threadIdx.x < GRP_NT) sh.next[threadIdx.x] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < slots * lpr * 4; i += GRP_THREADS) {
            const int t = i >> (lpr_log2 + 2), e = i & (lpr * 4 - 1), p = sh.slot_pair[t];
            float x[16];
            stage_load(input_row(a, a.xrow ? a.xrow[p] : p / a.xdiv), a.xbf16, e >> 2, e & 3, x);
            stage_store<4>(x, e >> 2, e & 3, sh.sx[t]);
        }
        __syncthreads();
        UnitCall uc = {a.y, a.ys, a.R, a.raw, a.add, lpr_log2, items[1]};
        if (items[1]) unit_items<MODE, 2>(uc);
        uc.items = items[0];
        if (items[0]) unit_items<MODE, 1>(uc);
    }
}

// ---- dense products: NT rows of inputs share each expansion ---------------------------------------------------------------
// The weights of a block pair are formed once (weight form) and multiplied into every row of inputs; the inputs of all rows
// sit in shared memory.  Every number of rows uses the same form, so a row's bits do not depend on the others.  The row steps
// are dealt to the warps of the grid block by block, so a small matrix still spreads over the SMs.
// Bound: as the pair kernel for one row (0.93 clk a block and SM in a loop without streams); a further row adds 4 packed
// multiply-adds a block and its share of the input loads (16 bytes a lane for two weights of two blocks: with 32 lanes a row
// 0.25 clk a block of the shared-memory pipe, half of that with 16).
template <int PF, int NT, int C>
__device__ __forceinline__ void dense_two_weights(const Words& wa, const Words& wb, const u64* q, const ulonglong2* const* cx, int bp, u64* d) {
    const u64 w0 = pair_weight<PF, 2 * C>(wa, wb, q), w1 = pair_weight<PF, 2 * C + 1>(wa, wb, q);
#pragma unroll
    for (int t = 0; t < NT; ++t) {
        const ulonglong2 u = cx[t][bp * 4 + C];
        d[t] = fma2(u.x, w0, d[t]);
        d[t] = fma2(u.y, w1, d[t]);
    }
}

template <int PF, int NT>
__global__ void __launch_bounds__(MV_THREADS, 2) mv_dense_kernel(MvParams a, KConst kc, RowShape sh, DenseSet set) {
    extern __shared__ __align__(16) ulonglong2 dense_sx[];
    __shared__ StreamTab tab;
    int block = blockIdx.x, blocks = gridDim.x;
    a.x += (size_t) blockIdx.y * NT * a.xs;      // a small matrix: groups of NT rows of inputs side by side
    a.y += (size_t) blockIdx.y * NT * a.ys;
    if (set.n > 1) {      // several matrices share the launch
        const int m = set_member(set, block);
        block -= set.first[m];
        blocks = set.first[m + 1] - set.first[m];
        a.w0 = set.w[m];
        a.R = a.ys = set.R[m];
        a.y = set.y[m];
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int lpr = 1 << sh.lpr_log2, rpw = 32 >> sh.lpr_log2, passes = 1 << (sh.lv - sh.lpr_log2);
    const int jc = lane & (lpr - 1), ro = lane >> sh.lpr_log2, ch = sh.ch;
    const int steps = (a.R + rpw - 1) / rpw, stride = blocks * MV_WARPS;
    int st = warp * blocks + block, r = st * rpw + ro, base = 0, pass = 0;
    Chunk k;
    if (st < steps && r < a.R && jc < ch) k = load_chunk<PF>(a.w0, (size_t) r * ch + jc);      // weights never change: requested before the wait
    load_stream_tab(tab, a.G, threadIdx.x, MV_THREADS);
    grid_dependents_go();
    grid_dependency_wait();   // everything below may read what the previous kernel in the stream wrote
    for (int i = threadIdx.x; i < NT * ch * 4; i += MV_THREADS) {
        const int t = i / (ch * 4), e = i - t * (ch * 4);
        float x[16];
        stage_load(a.x + (size_t) t * a.xs, 0, e >> 2, e & 3, x);
        stage_store<PF>(x, e >> 2, e & 3, dense_sx + (size_t) t * ch * CX);
    }
    __syncthreads();
    const float sc = slice_scale(a.w0.eb + (8 - PF));
    u64 acc[NT];
    float stk[NT][3];
#pragma unroll
    for (int t = 0; t < NT; ++t) acc[t] = 0ull;
    while (st < steps) {
        int sn = st, rn = r, bn = base + 32, pn = pass;
        if (bn >= ch) {
            if (pass + 1 < passes) { pn = pass + 1; bn = pass_offset(pn, sh.lv); }      // (possibly a pass without chunks: zeros)
            else { sn = st + stride; rn = r + stride * rpw; bn = 0; pn = 0; }
        }
        Chunk n;
        if (sn < steps && rn < a.R && bn + jc < ch) n = load_chunk<PF>(a.w0, (uint32_t) (rn * ch + bn + jc));
        const bool ok = r < a.R;
        if (ok && base + jc < ch) {
            const ulonglong2* cx[NT];
#pragma unroll
            for (int t = 0; t < NT; ++t) cx[t] = dense_sx + (size_t) (t * ch + base + jc) * CX;
            const uint32_t sw[4] = {k.s.x, k.s.y, k.s.z, k.s.w}, cw[4] = {k.c.x, k.c.y, k.c.z, k.c.w};
#pragma unroll
            for (int bp = 0; bp < 4; ++bp) {
                uint32_t g0, g1;
                pair_stream(tab, sw[bp], g0, g1);
                const Words wa = window_words<PF, 0>(sw[bp], g0), wb = window_words<PF, 1>(sw[bp], g1);
                u64 q[4], d[NT];
                if (PF == 4) pair_coefs(cw[bp], kc, q); else pair_coefs3(cw[bp], kc, q);
                const u64 kq = pair_centre<PF>(q), e2 = PF == 4 ? code_scale_pair(k.cd, bp, kc) : code_scale_pair3(cw[bp], kc);
#pragma unroll
                for (int t = 0; t < NT; ++t) d[t] = mul2(kq, staged_sum(cx[t], bp));
                dense_two_weights<PF, NT, 0>(wa, wb, q, cx, bp, d);
                dense_two_weights<PF, NT, 1>(wa, wb, q, cx, bp, d);
                dense_two_weights<PF, NT, 2>(wa, wb, q, cx, bp, d);
                dense_two_weights<PF, NT, 3>(wa, wb, q, cx, bp, d);
#pragma unroll
                for (int t = 0; t < NT; ++t) acc[t] = fma2(d[t], e2, acc[t]);
            }
        }
        if (pn != pass || sn != st) {      // the pass's last chunk
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                float s = tree_push(stk[t], pass, pair_total(acc[t]));
                acc[t] = 0ull;
                if (sn != st) {      // and the row's
                    s = group_sum(s, lpr) * sc;
                    if (ok && jc == 0) store_out<MODE_ROUND>(a, t, r, s, 0.0f);
                }
            }
        }
        k = n;
        st = sn; r = rn; base = bn; pass = pn;
    }
}

// ---- any K that is a multiple of 8, any alignment: one warp per (pair or dense, row), lanes over single blocks -------
// P = 4 (SEED4P4) or 3 (SEED4: the exponent code rides in the nibble word, there is no code stream).
template <int MODE, int P>
__global__ void __launch_bounds__(MV_THREADS) mv_generic_kernel(MvParams a, KConst kc, int T) {
    __shared__ StreamTab tab;
    // (The next kernel's blocks come in when this one ends: beside these two an SM they leave the next call's unevenly dealt, us, calls one behind the
    // other: gate + up of 64 pairs, K 1000, P = 3 122.8 with, 93.4 without, 93.8 as ordinary launches; a layer of 8 rows, 1000 / 520, 109.0 / 96.0.)
    tab_and_wait(tab, a.G, a.late, threadIdx.x, MV_THREADS, false);   // everything below may read what the previous kernel in the stream wrote
    __syncthreads();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nb = a.K / 8, dense = a.sel == NULL;
    const long long ntask = (long long) (dense ? 1 : a.P) * a.R;
    for (long long task = (long long) blockIdx.x * MV_WARPS + warp; task < ntask; task += (long long) gridDim.x * MV_WARPS) {
        const int pair = (int) (task / a.R), r = (int) (task % a.R);
        const int slice = a.sel ? a.sel[pair] : 0;
        const WSlice wa = a.ws ? a.ws[slice] : a.w0;
        WSlice wb = wa;
        if (MODE == MODE_GU) wb = a.wu[slice];
        float s[MV_MAXT], su[MV_MAXT];
#pragma unroll
        for (int t = 0; t < MV_MAXT; ++t) s[t] = su[t] = 0.0f;
        for (int j = lane; j < nb; j += 32) {
            const size_t gidx = (size_t) r * nb + j;
#pragma unroll
            for (int half = 0; half < (MODE == MODE_GU ? 2 : 1); ++half) {
                const WSlice& w = half ? wb : wa;
                const uint32_t seed = ((const uint16_t*) w.p[0])[gidx], cwi = ((const uint16_t*) w.p[1])[gidx];
                const uint32_t code = P == 4 ? (((const uint8_t*) w.p[3])[gidx >> 1] >> ((gidx & 1) * 4)) & 15u : cwi & 15u;
                const uint32_t g = stream_bits(tab, seed);
                const uint32_t aw = seed | (g << 16);
                float v[32], q[4];
                if (P == 4) { block_states(aw, g, v); block_coefs(cwi, kc, q); }
                else { block_states3(aw, g, v); block_coefs3(cwi, kc, q); }
                const float e2 = __uint_as_float((code << 23) | 0x38000000u);
#pragma unroll
                for (int t = 0; t < MV_MAXT; ++t) {
                    if (t >= T) break;
                    const float* xp = a.x + (size_t) (dense ? t : pair / a.xdiv) * a.xs + (size_t) j * 8;
                    float xr[8], xo[4];
#pragma unroll
                    for (int c = 0; c < 8; ++c) xr[c] = ld_in_order(xp + c);      // (C++ loads: 4 % slower, spills)
#pragma unroll
                    for (int c = 0; c < 8; ++c) xr[c] *= NSL_XSCALE;
                    block_offsets(xr, xo);
                    const float d = P == 4 ? states_dot(v, q, xr, xo) : states_dot3(v, q, xr, xo);
                    if (half) su[t] = fmaf(d, e2, su[t]);
                    else s[t] = fmaf(d, e2, s[t]);
                }
            }
        }
        const float sca = slice_scale(wa.eb + (4 - P)), scb = slice_scale(wb.eb + (4 - P));   // P = 3 products are half as large
#pragma unroll
        for (int t = 0; t < MV_MAXT; ++t) {
            if (t >= T) break;
            const float st = group_sum(s[t], 32) * sca;
            float sut = 0.0f;
            if (MODE == MODE_GU) sut = group_sum(su[t], 32) * scb;
            if (lane == 0) store_out<MODE>(a, dense ? t : pair, r, st, sut);
        }
    }
}

// ---- bit-exact decode: one thread per block ---------------------------------------------------------------------------
template <bool BF16, int P>
__global__ void __launch_bounds__(256) decode_kernel(WSlice w, KConst kc, int K, int R, void* out, const uint32_t* G) {
    __shared__ StreamTab tab;
    load_stream_tab(tab, G, threadIdx.x, 256);
    __syncthreads();
    const size_t nblk = (size_t) R * (K / 8);
    for (size_t gidx = (size_t) blockIdx.x * 256 + threadIdx.x; gidx < nblk; gidx += (size_t) gridDim.x * 256) {
        const uint32_t seed = ((const uint16_t*) w.p[0])[gidx], cw = ((const uint16_t*) w.p[1])[gidx];
        const int code = P == 4 ? (((const uint8_t*) w.p[3])[gidx >> 1] >> ((gidx & 1) * 4)) & 15 : (int) (cw & 15u);
        const uint32_t g = stream_bits(tab, seed);
        float wv[8];
        if (P == 4) block_weights(seed | (g << 16), g, cw, exact_scale<42>(w.eb + code), kc, wv);
        else block_weights3(seed | (g << 16), g, cw, exact_scale<43>(w.eb + code), kc, wv);
        if (BF16) {
            uint4 o;
            o.x = bf16_bits(wv[0]) | ((uint32_t) bf16_bits(wv[1]) << 16);
            o.y = bf16_bits(wv[2]) | ((uint32_t) bf16_bits(wv[3]) << 16);
            o.z = bf16_bits(wv[4]) | ((uint32_t) bf16_bits(wv[5]) << 16);
            o.w = bf16_bits(wv[6]) | ((uint32_t) bf16_bits(wv[7]) << 16);
            ((uint4*) out)[gidx] = o;
        } else {
            ((float4*) out)[2 * gidx] = make_float4(wv[0], wv[1], wv[2], wv[3]);
            ((float4*) out)[2 * gidx + 1] = make_float4(wv[4], wv[5], wv[6], wv[7]);
        }
    }
}

// ---- launch selection ---------------------------------------------------------------------------------------------------
static int log2_floor(int v) { int l = 0; while ((2 << l) <= v) ++l; return l; }

template <typename K>
static void allow_smem(K kernel, bool* done, size_t bytes) {      // once per device and kernel
    int dev = 0;
    cudaGetDevice(&dev);
    if (!done[dev & 15]) {
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bytes);
        done[dev & 15] = true;
    }
}

// How many lanes a row gets: the fewest chunk slots that a warp spends on its share, the rows dealt to all warps of the grid.
// Rows of 2^j <= 32 chunks keep a lane a chunk: its loop is the shorter one (config 1 at 8 rows: 132 us a step, 135.5 with 16
// lanes a row).
static RowShape row_shape(int ch, long long rows, int warps) {
    int lv = 0;
    while ((1 << lv) < (ch < 32 ? ch : 32)) ++lv;
    RowShape best = {ch, lv, lv, 1};
    if (ch == 1 << lv) return best;
    double best_cost = 0.0;
    for (int l = lv; l >= 0 && l >= lv - 3; --l) {
        int slots = 0;      // chunk rounds of a row step
        for (int p = 0; p < (1 << (lv - l)); ++p) {
            const int off = pass_offset(p, lv);
            slots += off < ch ? (ch - off + 31) / 32 : 0;
        }
        const long long steps = (rows * (1 << l) + 31) / 32;
        const double cost = (double) ((steps + warps - 1) / warps) * (slots + 0.4);      // 0.4: a step's shuffles and stores
        if (l == lv || cost < best_cost) { best.lpr_log2 = l; best_cost = cost; }
    }
    return best;
}

static size_t staged_bytes(int ch) { return (size_t) ch * CX * 16; }
// Rows that are not 2^j <= 32 chunks: groups of 8, 4 or 2 lanes, whichever leaves the fewest lane slots empty (fewer lanes read
// shorter runs of the streams: they have to save a twentieth).  A function of the row's length alone, so a row's bits do not
// depend on the list it is part of.
static RowShape item_shape(int ch) {
    RowShape best = {ch, 0, 0, ch};
    double best_cost = 1e30;
    for (int l = 3; l >= 1; --l) {
        const int groups = (ch + (1 << l) - 1) >> l;
        const double cost = (double) (groups << l) / ch + 0.05 * (3 - l);
        if (cost < best_cost && part_steps(PART_FLOATS_MIN, groups, l, 2) >= 1) { best.lpr_log2 = l; best.groups = groups; best_cost = cost; }
    }
    return best;
}
template <int MODE, int PF>
static void launch_pair(cudaStream_t s, const MvParams& a, const RouteFuse& rf) {
    const int ch = a.K / 64, sms = sm_count();
    static bool attr_set[16], attr_set_one[16], attr_set_single[16], attr_set_items[16];
    if (ch <= 32 && (ch & (ch - 1)) == 0) {
        const int lpr_log2 = log2_floor(ch);
        int win = a.P / sms + 2;      // a share's pairs, whole or in part
        if (win > PAIR_WIN) win = PAIR_WIN;
        if (win > a.P) win = a.P;
        const size_t smem = win * staged_bytes(ch);
        auto go = [&](auto kernel, bool* done) {
            allow_smem(kernel, done, (size_t) PAIR_WIN * 32 * CX * 16);
            launch(kernel, sms, PAIR_THREADS, smem, s, a, kconst(), lpr_log2, win, rf);
        };
        const bool single = MODE != MODE_GU && (long long) a.P * ((a.R * ch + 31) / 32) <= (long long) PAIR_WARPS * sms;      // a warp each for all row steps
        if (ch == 1) go(mv_pair_kernel<MODE, PF, true, false>, attr_set_one);
        else if (single) go(mv_pair_kernel<MODE, PF, false, MODE != MODE_GU>, attr_set_single);
        else go(mv_pair_kernel<MODE, PF, false, false>, attr_set);
    } else {
        const RowShape sh = item_shape(ch);
        const size_t room = (size_t) max_smem_optin() - 6144, one = staged_bytes(ch);      // 6144: the kernel's other shared memory (launch_mv has made sure that one row and the fewest sums fit)
        const int rpw = 32 >> sh.lpr_log2;
        const long long steps = ((long long) a.P * ((a.R + rpw - 1) / rpw) + sms - 1) / sms;      // of a block
        int win = a.P / sms + 2;
        if (win > PAIR_WIN) win = PAIR_WIN;
        if (win > a.P) win = a.P;
        while (win > 1 && win * one + PART_FLOATS * 4 > room) --win;
        size_t part = (room - win * one) / 4;
        if (part > PART_FLOATS) part = PART_FLOATS;
        const size_t need = (size_t) (steps + 1) * sh.groups * rpw * (MODE == MODE_GU ? 2 : 1);
        if (part > need) part = need;
        // Two steps of the one matrix an item where a warp still gets eight items: they share the inputs' loads, but fewer items are
        // dealt less evenly.
        const int spi = MODE != MODE_GU && steps * sh.groups >= 16 * PAIR_WARPS ? 2 : 1;
        allow_smem(mv_items_kernel<MODE, PF>, attr_set_items, room);
        launch(mv_items_kernel<MODE, PF>, sms, PAIR_THREADS, win * one + part * 4, s, a, kconst(), sh, win, (int) part, spi, rf);
    }
    count_launch();
}

// Which pair lists go to the grouped kernel (one expansion per distinct slice, up to GRP_NT pairs a unit): its plan (and the router's
// launch of its own) costs ~15 us a layer and its second pair half of a single one, so enough pairs have to meet on a slice.
// P pairs of E slices meet P^2 / 2E times, and the line lies at 40 of them: config 1's layer with 64 pairs of 16 / 32 / 64 / 128
// slices 90.4 / 93.8 / 100.0 / 105.5 us grouped, 98.9 / 99.2 / 99.3 / 99.6 pair by pair; two decoder layers with 96 pairs of 64 /
// 128 / 512 397 / 408 / 429 and 416 / 416 / 422, with 160 of 512 605 and 589, with 200 719 and 714; 320 of 512 are faster
// grouped.  Fewer than 48 pairs stay pair by pair, where the two are within 5 % (config 1's widths, grouped / pair by pair, us: 28 and 32
// pairs of 4 slices 51.4 / 49.9 and 53.2 / 56.0, 28 of 8 52.1 / 49.9, 40 of 8 63.9 / 66.6, 42 of 16 69.0 / 70.0; 48 of 8 and of 16 71.2 /
// 76.4 and 73.2 / 76.4).  Where the number of slices is not known: more than GRP_MIN_PAIRS pairs.
constexpr int GRP_MIN_PAIRS = 64;
static bool pairs_meet(int P, int slices) { return slices > 0 ? P >= 48 && (long long) P * P >= 80ll * slices : P > GRP_MIN_PAIRS; }
static bool grp_serves(int K) { return K % 64 == 0 && K >= 256 && K <= 2048 && (K & (K - 1)) == 0; }
bool mv_groups(int K, int P, int slices) { return grp_serves(K) && pairs_meet(P, slices); }

template <int MODE>
static void launch_grp(cudaStream_t s, const MvParams& a, int lpr_log2) {
    static bool attr_set[16];
    allow_smem(mv_grp_kernel<MODE>, attr_set, sizeof(GrpShared));
    launch(mv_grp_kernel<MODE>, sm_count(), GRP_THREADS, sizeof(GrpShared), s, a, kconst(), lpr_log2);
    count_launch();
}

template <int PF, int NT>
static void launch_dense_v(cudaStream_t s, const MvParams& a, size_t smem, DenseSet* set, int groups = 1) {
    static bool attr_set[16];
    const int bps = smem > 100 * 1024 ? 1 : 2;
    long long rows = a.R;
    for (int m = 1; set && m < set->n; ++m) rows += set->R[m];
    const RowShape sh = row_shape(a.K / 64, rows, sm_count() * bps * MV_WARPS);
    auto steps_of = [&](long long r) { return (int) ((r * (1 << sh.lpr_log2) + 31) / 32); };
    int blocks = std::min(steps_of(rows), std::max(sm_count() * bps / groups, 1));
    if (set) {      // each matrix gets its share of the blocks, at least one
        int left = blocks > set->n ? blocks : set->n;
        long long rest = rows;
        for (int m = 0; m < DENSE_SET; ++m) {
            int n = 0;
            if (m < set->n) {
                n = (int) ((2 * left * (long long) set->R[m] + rest) / (2 * rest));
                n = std::max(1, std::min(n, left - (set->n - 1 - m)));
                left -= n;
                rest -= set->R[m];
            }
            set->first[m + 1] = set->first[m] + n;
        }
        blocks = set->first[DENSE_SET];
    }
    if (smem > 40 * 1024) allow_smem(mv_dense_kernel<PF, NT>, attr_set, (size_t) max_smem_optin() - 8192);
    launch(mv_dense_kernel<PF, NT>, dim3((unsigned) blocks, (unsigned) groups), MV_THREADS, smem, s, a, kconst(), sh, set ? *set : DenseSet{1});
    count_launch();
}
// T rows on one slice; more rows than their inputs fit shared memory go in two launches (a row's bits do not depend on the rest).
template <int PF>
static void launch_dense(cudaStream_t s, MvParams a, int T, DenseSet* set = NULL) {
    const size_t one = staged_bytes(a.K / 64), room = (size_t) max_smem_optin() - 8192;
    // A matrix of fewer row steps than half the warps: its rows of inputs are shared out too (a P = 3 matrix of 512 x 2048, 8 rows: 12.3 us in one
    // group, 9.1 in four, which is the call itself; 256 x 4096, 8 rows 13.0 and 9.2).
    if (!set && T > 1) {
        const int warps = sm_count() * 2 * MV_WARPS, ch = a.K / 64, per_step = ch < 32 ? 32 / ch : 1, steps = (a.R + per_step - 1) / per_step;
        int g = T;
        while (g > 1 && (T % g || (long long) steps * g > warps)) --g;
        if (g > 1 && (size_t) (T / g) * one <= room) {
            const int n = T / g;
            switch (n) {
                case 1: launch_dense_v<PF, 1>(s, a, n * one, NULL, g); return;
                case 2: launch_dense_v<PF, 2>(s, a, n * one, NULL, g); return;
                case 3: launch_dense_v<PF, 3>(s, a, n * one, NULL, g); return;
                default: launch_dense_v<PF, 4>(s, a, n * one, NULL, g); return;
            }
        }
    }
    while (T > 0) {
        int n = T;
        while (n > 1 && n * one > room) n = (n + 1) / 2;
        switch (n) {
#define NSL_CASE(N) case N: launch_dense_v<PF, N>(s, a, N * one, set); break;
            NSL_CASE(1) NSL_CASE(2) NSL_CASE(3) NSL_CASE(4) NSL_CASE(5) NSL_CASE(6) NSL_CASE(7) NSL_CASE(8)
#undef NSL_CASE
        }
        a.x += (size_t) n * a.xs;
        a.y += (size_t) n * a.ys;
        for (int m = 0; set && m < set->n; ++m) set->y[m] += (size_t) n * set->R[m];
        T -= n;
    }
}

// The streams of a slice given by value (a dense call) are checked on the host.  Slices in a device table are not: their streams must be
// 16-byte aligned (codes 4) in every form but the one that load_any_16 serves.
static bool slice_aligned(const WSlice& w, int pf) {
    return aligned16(w.p[0]) && aligned16(w.p[1]) && (pf == 3 || ((uintptr_t) w.p[3] & 3u) == 0);
}

// PF = 4: SEED4P4; 3: SEED4.  The chunked kernels read whole chunks with 16-byte loads: rows of inputs and (checked where
// the slice is on the host) the streams must be aligned for that, and one row of inputs must fit shared memory; anything else
// goes to the any-shape kernel.
template <int MODE, int PF>
static void launch_mv(cudaStream_t s, const MvParams& a, int T, const RouteFuse& rf = RouteFuse{}, int slices = 0) {      // slices that sel chooses from (0: not known)
    if (a.R <= 0 || a.P <= 0 || T <= 0) return;
    if (a.K <= 0 || a.K % 8) { set_error("seed mat-vec: K = %d is not a multiple of 8", a.K); return; }
    if (T > MV_MAXT) { set_error("seed mat-vec: %d tokens, at most %d", T, MV_MAXT); return; }
    const bool dense = a.sel == NULL && rf.logits == NULL;
    const int ch = a.K / 64;
    const bool chunked = a.K % 64 == 0 && aligned16(a.x) && a.xs % (a.xbf16 ? 8 : 4) == 0 && (a.ws != NULL || slice_aligned(a.w0, PF)) &&
                         staged_bytes(ch) <= (size_t) max_smem_optin() - 10240;
    if (!chunked) {
        if (a.xrow || a.count || a.xbf16 || rf.logits) {
            set_error("seed mat-vec: the routed / row-index / device-count / bf16-input forms need K a multiple of 64 and aligned rows (K = %d)", a.K);
            return;
        }
        launch(mv_generic_kernel<MODE, PF>, sm_count() * 2, MV_THREADS, 0, s, a, kconst(), dense ? T : 1);
        count_launch();
        return;
    }
    if constexpr (MODE == MODE_ROUND) {
        if (dense) { launch_dense<PF>(s, a, T); return; }
    }
    if constexpr (PF == 4) {
        if (!rf.logits && mv_groups(a.K, a.P, slices)) { launch_grp<MODE>(s, a, log2_floor(ch)); return; }
    }
    launch_pair<MODE, PF>(s, a, rf);
}

// kc_mv_gu / nsl_mv_gu_raw and kc_mv_sel / nsl_mv_raw over a layer of n_exp SEED4P4 experts.
void mv_gu_of(cudaStream_t s, const WSlice* wg, const WSlice* wu, int K, int R, const float* x, int xs, float* out, int ys, const int32_t* sel, int P, int xdiv, int raw,
              int n_exp, const uint32_t* G) {
    launch_mv<MODE_GU, 4>(s, MvParams{wg, wu, WSlice{}, sel, x, out, G, K, R, P, xdiv, xs, ys, 0, raw, NULL, NULL, 0}, 1, RouteFuse{}, n_exp);
}
void mv_sel_of(cudaStream_t s, const WSlice* ws, int K, int R, const float* x, int xs, float* y, int ys, const int32_t* sel, int P, int xdiv, int raw, int n_exp,
               const uint32_t* G) {
    launch_mv<MODE_ROUND, 4>(s, MvParams{ws, NULL, WSlice{}, sel, x, y, G, K, R, P, xdiv, xs, ys, 0, raw, NULL, NULL, 0}, 1, RouteFuse{}, n_exp);
}

// A set of SEED4P4 matrices for up to MV_MAXT rows; false: a shape that needs the any-shape kernel.
bool launch_seed_set(cudaStream_t s, DenseSet set, int K, const float* x, int T, const uint32_t* G) {
    if (T < 1 || T > MV_MAXT || K < 64 || K % 64 || !aligned16(x) || staged_bytes(K / 64) > (size_t) max_smem_optin() - 10240) return false;
    for (int m = 0; m < set.n; ++m)
        if (set.R[m] < 1 || !slice_aligned(set.w[m], 4)) return false;
    MvParams a = {NULL, NULL, set.w[0], NULL, x, set.y[0], G, K, set.R[0], T, 1, K, set.R[0], 0, 0, NULL, NULL, 0};
    launch_dense<4>(s, a, T, &set);
    return true;
}

// The decode step in one launch; false (nothing launched) when a size is outside what the pair kernel serves.
static bool launch_mv_step(cudaStream_t s, const StepParams& p) {
    const int cd = p.d / 64, cf = p.ff / 64;
    if (p.T < 1 || p.T > MV_MAXT || p.top_k < 1 || p.top_k > 32 || p.T * p.top_k > 256 || p.n_exp < p.top_k || p.n_exp > 32 * ROUTE_PER_LANE) return false;
    if (p.d % 64 || p.ff % 64 || cd < 1 || cf < 1 || (cd & (cd - 1)) || (cf & (cf - 1)) || cd > 32 || cf > 32) return false;
    if (!aligned16(p.x) || p.xs % 4 || !aligned16(p.A) || !aligned16(p.D)) return false;
    launch(mv_step_kernel, sm_count() * 2, MV_THREADS, 0, s, p, kconst(), log2_floor(cd), log2_floor(cf));
    count_launch();
    return true;
}

bool launch_q4_mv(cudaStream_t s, const WSlice& w, int K, int R, const float* x, int xs, float* y, int ys, int T, int add);
void launch_bf16_mv(cudaStream_t s, const WSlice& w, int K, int R, const float* x, int xs, float* y, int ys, int T, int add);
bool launch_bf16_mm_skinny(cudaStream_t s, const WSlice& w, int K, int R, const float* x, int xs, float* y, int ys, int T, int add);

static bool seed_fmt(int fmt, const char* who) {      // the mat-vec entry points: P = 4 and P = 3 seeds
    if (fmt == MF_SEED4P4 || fmt == MF_SEED4) return true;
    set_error("%s: weight format %d is not served by this library (SEED4P4 = %d, SEED4 = %d)", who, fmt, (int) MF_SEED4P4, (int) MF_SEED4);
    return false;
}

}   // namespace nsl

using namespace nsl;

extern "C" {

void kc_mv(cudaStream_t s, int fmt, WSlice w, int K, int R, const float* x, int xs, float* y, int ys, int T, int add,
           const uint32_t* G) {
    if (fmt == MF_Q4) {      // the LM head's affine int4 (q4_head.cu)
        FollowScope follow;
        if (T > MV_MAXT) set_error("kc_mv (Q4): %d tokens, at most %d", T, (int) MV_MAXT);
        else launch_q4_mv(s, w, K, R, x, xs, y, ys, T, add);
        return;
    }
    if (fmt == MF_BF16) {      // stored BF16 weights (dense_bf16.cu): the tensor-core kernel where its shape rules allow, else a warp per row
        if (!launch_bf16_mm_skinny(s, w, K, R, x, xs, y, ys, T, add)) launch_bf16_mv(s, w, K, R, x, xs, y, ys, T, add);
        return;
    }
    if (!seed_fmt(fmt, "kc_mv")) return;
    MvParams a = {NULL, NULL, w, NULL, x, y, G, K, R, T, 1, xs, ys, add, 0, NULL, NULL, 0};
    if (fmt == MF_SEED4) launch_mv<MODE_ROUND, 3>(s, a, T);
    else launch_mv<MODE_ROUND, 4>(s, a, T);
}

void kc_mv_sel(cudaStream_t s, int fmt, const WSlice* ws, int K, int R, const float* x, int xs, float* y, int ys,
               const int32_t* sel, int P, int xdiv, const uint32_t* G) {
    if (!seed_fmt(fmt, "kc_mv_sel")) return;
    FollowScope follow;
    MvParams a = {ws, NULL, WSlice{}, sel, x, y, G, K, R, P, xdiv, xs, ys, 0, 0, NULL, NULL, 0, follow.own()};
    if (fmt == MF_SEED4) launch_mv<MODE_ROUND, 3>(s, a, 1);
    else launch_mv<MODE_ROUND, 4>(s, a, 1);
}

void kc_mv_gu(cudaStream_t s, int fmt, const WSlice* wg, const WSlice* wu, int K, int R, const float* x, int xs, float* out,
              int ys, const int32_t* sel, int P, int xdiv, const uint32_t* G) {
    if (!seed_fmt(fmt, "kc_mv_gu")) return;
    FollowScope follow;
    MvParams a = {wg, wu, WSlice{}, sel, x, out, G, K, R, P, xdiv, xs, ys, 0, 0, NULL, NULL, 0, follow.own()};
    if (fmt == MF_SEED4) launch_mv<MODE_GU, 3>(s, a, 1);
    else launch_mv<MODE_GU, 4>(s, a, 1);
}

void nsl_mv_raw(cudaStream_t s, const WSlice* ws, int K, int R, const float* x, int xs, float* y, int ys,
                const int32_t* sel, int P, int xdiv, const uint32_t* G) {
    MvParams a = {sel ? ws : NULL, NULL, WSlice{}, sel, x, y, G, K, R, P, xdiv > 0 ? xdiv : 1, xs, ys, 0, 1, NULL, NULL, 0};
    if (!sel) a.w0 = *ws;   // dense: ws is a host pointer to the one slice
    launch_mv<MODE_ROUND, 4>(s, a, sel ? 1 : P);
}

void nsl_mv_gu_raw(cudaStream_t s, const WSlice* wg, const WSlice* wu, int K, int R, const float* x, int xs, float* out,
                   int ys, const int32_t* sel, int P, int xdiv, const uint32_t* G) {
    MvParams a = {wg, wu, WSlice{}, sel, x, out, G, K, R, P, xdiv, xs, ys, 0, 1, NULL, NULL, 0};
    launch_mv<MODE_GU, 4>(s, a, 1);
}

// kc_mv_gu with the router folded into its prologue: T <= MV_MAXT rows of logits -> ind / wt [T][top_k] and
// a [T * top_k][R]; pair t * top_k + j uses expert ind[t][j] and input row t.
void nsl_mv_gu_routed(cudaStream_t s, const WSlice* wg, const WSlice* wu, int K, int R, const float* x, int xs, float* out, int ys,
                      int n_exp, int top_k, const float* logits, int ld, int T, int32_t* ind, float* wt, int raw, const uint32_t* G) {
    if (T <= 0) return;
    if (T > MV_MAXT || n_exp < 1 || n_exp > 32 * ROUTE_PER_LANE || top_k < 1 || top_k > 32 || top_k > n_exp) {
        set_error("nsl_mv_gu_routed: %d rows (at most %d), %d experts (at most %d), top %d (at most 32)", T, MV_MAXT, n_exp,
                  32 * ROUTE_PER_LANE, top_k);
        return;
    }
    MvParams a = {wg, wu, WSlice{}, NULL, x, out, G, K, R, T * top_k, top_k, xs, ys, 0, raw, NULL, NULL, 0};
    const RouteFuse rf = {logits, ld, n_exp, top_k, T, ind, wt};
    launch_mv<MODE_GU, 4>(s, a, 1, rf);
}

// The whole decode step of an expert layer (router, gate + up + SwiGLU, down, combine) as one launch: 1 = launched, 0 = a
// size is outside what it serves (nothing launched: the caller issues the three launches).  sync: 4 * (2 + T + T * top_k)
// bytes of device memory, zero before the first call; every call leaves its counters zero.  sync[0] is the status word:
// 1 after a launch in which a bounded wait ran out (its output is not valid), for the caller to read and clear.
// A and D are the caller's work buffers [T * top_k][ff] and [T * top_k][d].
int nsl_mv_step(cudaStream_t s, const WSlice* wg, const WSlice* wu, const WSlice* wd, int d, int ff, const float* x, int xs, int n_exp,
                int top_k, const float* logits, int ld, int T, int32_t* ind, float* wt, float* A, float* D, float* out, int raw,
                unsigned* sync, const uint32_t* G) {
    if (!sync || T < 1 || top_k < 1) return 0;
    StepParams p = {wg, wu, wd, x, logits, A, D, out, ind, wt, G, xs, ld, n_exp, top_k, T, d, ff, raw,
                    {sync + 2 + T, sync + 2, sync + 1, (int*) sync}};
    return launch_mv_step(s, p) ? 1 : 0;
}

// Expert-parallel forms: a compacted pair list whose length lives on the device.  Pair p uses slice sel[p] and input
// row xrow[p] of x, which holds packed bf16 rows when x_bf16 is set; at most max_pairs pairs, *count of them valid.
void nsl_mv_gu_rows(cudaStream_t s, const WSlice* wg, const WSlice* wu, int K, int R, const void* x, int xs, int x_bf16,
                    float* out, int ys, const int32_t* sel, const int32_t* xrow, int max_pairs, const int32_t* count,
                    int raw, const uint32_t* G) {
    MvParams a = {wg, wu, WSlice{}, sel, (const float*) x, out, G, K, R, max_pairs, 1, xs, ys, 0, raw, xrow, count, x_bf16};
    launch_mv<MODE_GU, 4>(s, a, 1);
}
void nsl_mv_sel_rows(cudaStream_t s, const WSlice* ws, int K, int R, const float* x, int xs, float* y, int ys,
                     const int32_t* sel, int max_pairs, const int32_t* count, int raw, const uint32_t* G) {
    MvParams a = {ws, NULL, WSlice{}, sel, x, y, G, K, R, max_pairs, 1, xs, ys, 0, raw, NULL, count, 0};
    launch_mv<MODE_ROUND, 4>(s, a, 1);
}


void nsl_decode_f32(cudaStream_t s, WSlice w, int K, int R, float* out, const uint32_t* G) {
    if (K <= 0 || K % 8 || R <= 0) { if (K % 8) set_error("nsl_decode_f32: K = %d is not a multiple of 8", K); return; }
    const size_t nblk = (size_t) R * (K / 8);
    const int grid = (int) ((nblk + 255) / 256 < (size_t) sm_count() * 8 ? (nblk + 255) / 256 : (size_t) sm_count() * 8);
    decode_kernel<false, 4><<<grid, 256, 0, s>>>(w, kconst(), K, R, out, G);
    count_launch();
}

void nsl_decode_bf16(cudaStream_t s, WSlice w, int K, int R, uint16_t* out, const uint32_t* G) {
    if (K <= 0 || K % 8 || R <= 0) { if (K % 8) set_error("nsl_decode_bf16: K = %d is not a multiple of 8", K); return; }
    const size_t nblk = (size_t) R * (K / 8);
    const int grid = (int) ((nblk + 255) / 256 < (size_t) sm_count() * 8 ? (nblk + 255) / 256 : (size_t) sm_count() * 8);
    decode_kernel<true, 4><<<grid, 256, 0, s>>>(w, kconst(), K, R, out, G);
    count_launch();
}

// P = 3 (SEED4) slices decoded bit for bit: w.p[0] seeds, w.p[1] nibble words, w.eb the exponent bias.
void nsl_decode3_f32(cudaStream_t s, WSlice w, int K, int R, float* out, const uint32_t* G) {
    if (K <= 0 || K % 8 || R <= 0) { if (K % 8) set_error("nsl_decode3_f32: K = %d is not a multiple of 8", K); return; }
    const size_t nblk = (size_t) R * (K / 8);
    const int grid = (int) ((nblk + 255) / 256 < (size_t) sm_count() * 8 ? (nblk + 255) / 256 : (size_t) sm_count() * 8);
    decode_kernel<false, 3><<<grid, 256, 0, s>>>(w, kconst(), K, R, out, G);
    count_launch();
}

void nsl_decode3_bf16(cudaStream_t s, WSlice w, int K, int R, uint16_t* out, const uint32_t* G) {
    if (K <= 0 || K % 8 || R <= 0) { if (K % 8) set_error("nsl_decode3_bf16: K = %d is not a multiple of 8", K); return; }
    const size_t nblk = (size_t) R * (K / 8);
    const int grid = (int) ((nblk + 255) / 256 < (size_t) sm_count() * 8 ? (nblk + 255) / 256 : (size_t) sm_count() * 8);
    decode_kernel<true, 3><<<grid, 256, 0, s>>>(w, kconst(), K, R, out, G);
    count_launch();
}

}   // extern "C"
