// chan_internal.h -- calls between the solver (chanrhs.cu) and the closure
// MLP (closure.cu) translation units of libchanrhs.so, and the early launches
// both use.  Not part of the C ABI.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>

struct chan_ctx;
struct chan_closure;

// Closure inputs and targets: 13 features (the 9 velocity gradients du_a/dx_b
// with a, b over (x, spanwise, wall-normal), the 3 temperature gradients and
// y+) and 9 subgrid fluxes (tau_uu, tau_vv, tau_ww, tau_uv, tau_uw, tau_vw,
// q_u, q_v, q_w).
constexpr int kClIn = 13, kClOut = 9;

// Append samples of the filtered state of context c to X [n][13] / T [n][9]
// (device arrays, room for `capacity` rows); *added receives the count.
// Sample points every (sx, sy, sz) grid points; box filter of width fw in
// x and spanwise.  Queued on the context's stream, which is synchronised.
int chan_internal_sample(chan_ctx *c, float *X, float *T, long long capacity, int sx, int sy, int sz, int fw,
                         long long *added);

// MLP inference on device arrays: Y [n][9] in physical units from X [n][13]
// (soa: X [13][n] and Y [9][n]); sets *flag (device) when a normalised output
// exceeds the closure's limit, and *err (null: the closure's own word) when an MMA did
// not complete in time.  Queued on `stream`, not synchronised.
int chan_internal_infer(chan_closure *m, const float *X, float *Y, long long n, bool soa, cudaStream_t stream,
                        int *flag, bool early, int *err = nullptr);
int chan_internal_closure_device(chan_closure *m);

// ---- early launches.  A kernel of a step takes 5..30 us on a small grid, and a plain
// launch starts it only when the kernel before has drained and been flushed.  Launched
// with programmatic serialisation its CTAs are placed as soon as every CTA of the one
// before has started and there is room, and wait there (grid_dep_wait).

// all kernels before this one are complete and their writes visible (no-op in a plain launch)
__device__ __forceinline__ void grid_dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the next kernel of the stream may be placed; it still waits for this one's end
__device__ __forceinline__ void grid_dep_launch() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// first statement of a kernel that is launched early.  The next kernel is let in only
// after the one before has ended: let in at once, a stage kernel's CTAs are placed beside
// the last ones of the stage before, two on some SMs and none on others
__device__ __forceinline__ void grid_dep_enter()
{
    grid_dep_wait();
    grid_dep_launch();
}

// launch k, early or plainly; an early k must begin with grid_dep_enter, or call
// grid_dep_wait before its first access to memory that an earlier kernel touches
template <typename... KArgs, typename... Args>
cudaError_t launch_kernel(bool early, void (*k)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, Args... args)
{
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = early ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, k, KArgs(args)...);
}
