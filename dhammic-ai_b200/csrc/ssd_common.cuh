// Shared device helpers and the problem descriptor used by every SSD kernel.
#pragma once
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ssd {

// Problem dimensions; c = T / l, hpg = heads per group.
struct Dims {
    int b, T, h, p, n, g, l, c, hpg;
};

__device__ __forceinline__ float to_f(float v) { return v; }
// A bf16 value as fp32 by a mixed-precision addition (sm_100), which takes either half of a register as it is and runs at the rate of an fp32 one
// (1.1 cycles a warp), where the shift or mask that makes an fp32 number of a half takes two, on the pipe that the conversions to bf16 need.  For the
// element-wise kernels (gated norm's backward of (16384, 4096) 120 -> 111 us, rotation with the running angle 723 -> 696 at (16, 4096, 64 heads), the rotation's
// backward of pairs that are no whole vectors, (4, 2048, 24, 66), 57.6 -> 47.4 although it spills 20 bytes, its forward 30.2 both ways), and where the fp32
// multiply-add kernels read bf16 rows that are no whole vectors (no difference: 970 -> 970 us forward and backward of (4, 1984, 20, 64), d_state 64); the
// tile kernels, which wait for latencies, lose 1 % by it and keep shifts and masks.
__device__ __forceinline__ float to_f(__nv_bfloat16 v) {
    float r;
    asm("add.rn.f32.bf16 %0, %1, %2;" : "=f"(r) : "h"(__bfloat16_as_ushort(v)), "f"(-0.f));
    return r;
}
template <class T> __device__ __forceinline__ T from_f(float v);
template <> __device__ __forceinline__ float from_f<float>(float v) { return v; }
template <> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float v) { return __float2bfloat16_rn(v); }

// Element offsets of the dense layouts.
__device__ __forceinline__ size_t x_off(const Dims& d, int bb, int t, int hh) {  // (b,T,h,p) row start
    return ((size_t)((size_t)bb * d.T + t) * d.h + hh) * d.p;
}
__device__ __forceinline__ size_t bc_off(const Dims& d, int bb, int t, int gg) {  // (b,T,g,n) row start
    return ((size_t)((size_t)bb * d.T + t) * d.g + gg) * d.n;
}
__device__ __forceinline__ size_t cum_off(const Dims& d, int bb, int hh, int k) {  // (b,h,c,l) chunk start
    return ((size_t)((size_t)bb * d.h + hh) * d.c + k) * d.l;
}
__device__ __forceinline__ size_t st_off(const Dims& d, int bb, int k, int hh) {  // (b,c,h,p,n) state start
    return ((size_t)((size_t)bb * d.c + k) * d.h + hh) * (size_t)d.p * d.n;
}

// Launch of a kernel that the GPU may set up while the one before it on the stream still runs (programmatic dependent launch).  Its
// blocks wait in dep_wait() until that kernel is complete and its writes are visible.  Every thread of every kernel launched this way
// calls dep_wait() before it touches global memory in any way, also where it has nothing to do: a kernel that could be complete
// before the one ahead of it would hand the next one memory that is still being written.  With that, the order of
// everything on the stream is what it is with plain launches.  `after`: what is on the stream directly before is a kernel of the same
// pass; what follows a memset, or work of the caller's, is launched plainly.  Saved is the time from the end of one kernel to the first work of the
// next: one slice of 512 positions and 24 heads 26.6 -> 22.5 us a call, one prompt of 16,384 positions 189.6 -> 183.5, a training
// step of (8, 2048, 24 heads) 260.8 -> 248.0.
template <class... K, class... A>
inline void launch_dep(bool after, void (*kernel)(K...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t c{};
    c.gridDim = grid;
    c.blockDim = block;
    c.dynamicSmemBytes = smem;
    c.stream = st;
    c.attrs = &at;
    c.numAttrs = after ? 1 : 0;
    cudaLaunchKernelEx(&c, kernel, static_cast<K>(args)...);  // (the caller looks at cudaGetLastError)
}
__device__ __forceinline__ void dep_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// Also lets the blocks of the kernel behind come to the SMs as soon as all of this one's have, instead of when they end.  For the SIMT
// kernels, whose blocks are small and short: forward + backward as a captured graph (called one by one they wait for the host and show
// nothing), fp32, with dep_wait and with this: (2, 512, 8 heads, 32), d_state 8, 79.9 -> 73.8 us, (1, 1024, 4 heads, 32), d_state 16,
// 53.3 -> 51.3, (1, 1984, 20 heads, 64), d_state 64, 299 -> 294.  Not ahead of the forward's scan, whose large blocks then come to SMs that
// the state pass half fills: forward of (2, 512, 8 heads, 64), d_state 64, 26.7 -> 32.8.  The kernels with a block per SM lose by it
// (prefill 183.5 -> 197 us, (8, 2048, 24 heads) 248 -> 268).
__device__ __forceinline__ void dep_wait_early() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

// Whether two buffers of so many bytes share memory.  A state that is updated in place (init and final_state the same buffer) must be read before it is
// written, and only a walk that one block takes from end to end sees to that.
inline bool overlap(const void* a, const void* b, size_t bytes) { return a && b && (const char*)a < (const char*)b + bytes && (const char*)b < (const char*)a + bytes; }

// Sum over a block of THREADS threads, valid in all of them; red: one float per warp.
template <int THREADS>
__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    __syncthreads();
    float s = 0.f;
#pragma unroll
    for (int w = 0; w < THREADS / 32; ++w) s += red[w];
    return s;
}

namespace prof {
// Kernel slots for launch accounting / optional per-kernel timing (definitions in ssd_b200_api.cu).
enum Kernel {
    K_CUMSUM = 0, K_CHUNK_STATE, K_STATE_PASS, K_CHUNK_SCAN, K_CHUNK_DSTATE, K_STATE_PASS_REV, K_CHUNK_BWD,
    K_DECAY, K_REDUCE, K_CACHE_L, K_CACHE_DC, K_PREFIX, K_TC_FWD, K_TC_BWD_STATE, K_TC_BWD, K_TC_AUX, K_TC_SUMMARY,
    K_EXCHANGE, K_COUNT
};
void begin(int k, cudaStream_t st);
void end(cudaStream_t st);
}  // namespace prof

// Wrap one kernel launch statement: counts it and, when profiling is on, brackets it with events.
#define SSD_LAUNCH(kidx, st, ...)     \
    do {                              \
        ::ssd::prof::begin(kidx, st); \
        __VA_ARGS__;                  \
        ::ssd::prof::end(st);         \
    } while (0)

}  // namespace ssd
