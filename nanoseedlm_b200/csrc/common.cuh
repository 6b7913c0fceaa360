// Host-side helpers shared by the launchers: error record, launch counter, device properties.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/nslm_kernels.h"

namespace nsl {

void set_error(const char* fmt, ...);
void count_launch(int n = 1);
int sm_count();
int max_smem_optin();

inline bool aligned16(const void* p) { return ((uintptr_t) p & 15u) == 0; }

// Programmatic dependent launch.  While a PdlScope(true) is alive on the calling thread, launch() marks the kernel as
// allowed to start before the previous kernel in its stream has finished: its blocks become resident as the previous
// kernel's blocks retire and run their prologue (the stream table, index arithmetic) until grid_dependency_wait(),
// which returns once the previous kernel has completed and its writes are visible.  Every kernel that launch() may start
// so calls grid_dependency_wait() before it reads or writes anything a neighbouring kernel touches; without the
// scope, and outside the entry points that open one themselves, the launch is an ordinary one and the wait returns at once.
// What a neighbour may have written (activations, logits, routing, partial sums, cache rows) is read with ordinary loads: ld.global.nc (__ldg, and what
// the compiler makes of a kernel's const __restrict__ parameters) is for memory that nobody writes while the kernel runs, and a dependent kernel runs
// beside the one that writes its inputs.  Weight streams and other constants take it.
// The thread's state is one of: each entry point's own choice (until the caller says otherwise), ordinary launches, dependent ones.
enum { PDL_OWN = -1, PDL_OFF = 0, PDL_ON = 1 };
extern thread_local int tl_pdl;
struct PdlScope {
    int prev;
    explicit PdlScope(bool on) : prev(tl_pdl) { tl_pdl = on ? PDL_ON : PDL_OFF; }
    ~PdlScope() { tl_pdl = prev; }
};
// For entry points whose kernels follow another of this library's kernels as a rule: a dependent launch unless the caller has asked for ordinary ones
// (nsl_dependent_launch(0)).  After a copy, and after a kernel that does not let its dependents go early, nothing starts before the predecessor has ended.
// Which ones: the calls of a layer, of a head with its tokens and of a prompt product, as an engine queues them (us, calls one behind the other, ordinary /
// dependent: a P = 3 layer of 8 rows 89.9 / 82.3, head and arg-max 52.4 / 49.7, 777 x (2048 x 2048) 39.0 / 37.4; with new inputs copied in before each, the
// copies included, 97.8 / 89.8, 56.5 / 53.2, 43.1 / 41.0).  kc_mm_packed, kc_mm_grouped*, nsl_mv_raw, nsl_mv_gu_raw,
// nsl_mv_gu_routed and the stored-BF16 products start the same or similar kernels, have not been measured that way and stay ordinary.
// Such a kernel reads nothing at all before its wait, the stream table included (tab_and_wait): a caller that has asked for nothing may have made the
// table in the kernel before, whose writes are visible after the wait and not sooner.
struct FollowScope {
    int prev;
    explicit FollowScope(bool follows = true) : prev(tl_pdl) { if (prev == PDL_OWN && follows) tl_pdl = PDL_ON; }
    int own() const { return prev == PDL_OWN; }
    ~FollowScope() { tl_pdl = prev; }
};

template <typename... KArgs, typename... Args>
inline cudaError_t launch(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = tl_pdl == PDL_ON ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<KArgs>(args)...);
}

// Up to three matrices of one width applied to the same rows of inputs in one launch (the attention's q, k, v; the shared expert's
// gate and up): a block works on one of them, matrix m has the blocks first[m] .. first[m + 1] - 1.
constexpr int DENSE_SET = 3;
struct DenseSet {
    int n;
    int first[DENSE_SET + 1];
    WSlice w[DENSE_SET];
    int R[DENSE_SET];
    float* y[DENSE_SET];      // [T][R]
};

#ifdef __CUDACC__
__device__ __forceinline__ int set_member(const DenseSet& set, int block) {
    int m = 0;
#pragma unroll
    for (int i = 1; i < DENSE_SET; ++i) m += i < set.n && block >= set.first[i];
    return m;
}
__device__ __forceinline__ void grid_dependency_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Ordinary loads that stay in the order they are written in, for loops where the compiler's own order costs registers and time.
__device__ __forceinline__ float ld_in_order(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ float4 ld_in_order(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ void grid_dependents_go() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
#endif

}   // namespace nsl
