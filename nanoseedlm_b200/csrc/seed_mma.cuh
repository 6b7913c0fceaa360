// Arguments of the seed GEMMs, for the launchers that choose between them: seed_gemm.cu (tcgen05) and seed_mma.cu (a few rows).
#pragma once
#include "common.cuh"

namespace nsl {

struct MmParams {
    const WSlice* ws;        // grouped: device table; dense: NULL
    WSlice w0;
    const void* X;           // f32, or packed bf16
    void* Y;                 // f32; packed bf16 with wu or out_bf16
    const int32_t* perm;
    const MmTile* tiles;
    const int32_t* ntiles;   // device tile count, or NULL: T
    const uint32_t* G;
    int K, R, T, xs, ys, xdiv, add, grouped, packed;      // T: dense rows; grouped without a device count: the number of tiles
    const WSlice* wu;        // gate + up + SwiGLU (SEED4P4, grouped): the up table (ws: the gate's), Y = packed bf16 [pair][R]
    int out_bf16;
    const int32_t* offs;     // grouped: the slices' first pairs (kc_bucket's work), or NULL; given (with in_sorted): up to three tiles of a slice share an expansion
    int in_sorted, out_sorted, T_in;      // grouped, packed: row n of the inputs (of the outputs) belongs to pair perm[n]; T_in: rows of inputs
    int late = 0;            // G may be read only after the wait for the previous kernel
};

bool seed_gemm_exact();      // kc_seed_gemm_f32's switch
// Gate + up + SwiGLU of a grouped prompt (packed inputs, sorted where offs is given; K a multiple of 64); the GEMM; whether MmParams.offs may be given.
void launch_gemm_gu(cudaStream_t s, const MmParams& a, int tiles_y);
void launch_gemm(cudaStream_t s, int fmt, const char* who, MmParams a, int tiles_y);
bool gemm_shares_tiles(int max_tiles);

// The same for a dense call of a few rows (seed_mma.cu; K a multiple of 64).
bool smm_serves(int K, const void* X, int xs, int packed);
void launch_seed_mma(cudaStream_t s, int fmt, const MmParams& m);

}   // namespace nsl
