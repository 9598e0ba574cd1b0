// Shared host-side helpers of the C-ABI translation units: error reporting and launch checks.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>

#include "../../include/coset_b200.h"

namespace coset {

// Stores a message for coset_last_error_string() (thread local) and returns `code`.
int fail(int code, const char* fmt, ...);
// cudaGetLastError() after a launch -> 0 or a positive cudaError_t (message stored).
int check_launch(const char* what);
int check_cuda(cudaError_t e, const char* what);

// Number of SMs of the current device (cached per device).
int sm_count();

// Device pointer to the q=4 single-level residual table of the current device:
// 65536 entries x 8 bytes = twice the residual G b - 4 Q(G b / 4) of level word `b`, plus 7.
// Built once per device by the library's own literal decoder; nullptr on failure (message stored).
const uint2* residual_table_q4(cudaStream_t stream);
// The same residuals packed into 4 bytes per level word (layout at e8::biased_bytes_q4m2), 256 KB:
// mostly L1-resident, for the bandwidth-bound decoder whose gathers otherwise wait on L2.  Kernels
// bound by instruction issue keep the 8-byte entries, which unpack with 12 fewer instructions.
const uint32_t* residual_table_q4_packed(cudaStream_t stream);

// The same residuals in 2 bytes per level word (layout at e8::compact_residues), 128 KB: for the kernels that keep
// the whole table in shared memory.
const uint16_t* residual_table_q4_compact(cudaStream_t stream);

inline bool aligned(const void* p, size_t a) { return (reinterpret_cast<uintptr_t>(p) % a) == 0; }

// s += v, and what the rounded sum lacks to e (Knuth's two-sum)
__device__ __forceinline__ void add_exactly(float& s, float& e, float v) {
    const float t = s + v, z = t - s;
    e += (s - (t - z)) + (v - z);
    s = t;
}

// Programmatic dependent launch.  A kernel launched with the attribute may start while the kernel before it in the stream still
// runs; grid_wait returns once that kernel (and with it every earlier one) has finished and its writes are visible, and grid_trigger
// lets the next such kernel start.  A kernel calls grid_wait before its first access to memory that others write, and grid_trigger
// only behind it, so that a kernel that has started early knows all but its direct predecessor to be complete.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
// The same value, which the compiler knows only behind every volatile statement before: loads through the read-only path (__ldg, const
// __restrict__) count as invariant and could otherwise be moved in front of grid_wait.  An address that is read depends on one, or the read is conditional on a bound.
__device__ __forceinline__ int behind_wait(int v) {
    asm volatile("" : "+r"(v) : : "memory");
    return v;
}
template <typename T>
__device__ __forceinline__ T* behind_wait(T* p) {
    asm volatile("" : "+l"(p) : : "memory");
    return p;
}

// Launches a kernel that calls grid_wait as a programmatic dependent of the one before it.
template <typename... Params, typename... Args>
int launch_dependent(const char* what, void (*kernel)(Params...), dim3 grid, unsigned threads, size_t smem, cudaStream_t stream, Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return check_cuda(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...), what);
}

}  // namespace coset
