// osc_common.cuh -- shared types and helpers of the B200 space-charge library.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include <string>

namespace osc {

// Complex vector types: float2 / double2 keep 8- and 16-byte aligned loads.
template <typename T> struct VecT;
template <> struct VecT<float> { typedef float2 type; typedef float4 type4; };
template <> struct VecT<double> { typedef double2 type; typedef double4 type4; };
template <typename T> using cplx = typename VecT<T>::type;
template <typename T> using vec4 = typename VecT<T>::type4;

template <typename T> __host__ __device__ __forceinline__ cplx<T> mk(T re, T im) {
    cplx<T> r;
    r.x = re;
    r.y = im;
    return r;
}
template <typename V> __host__ __device__ __forceinline__ V cadd(V a, V b) {
    a.x += b.x;
    a.y += b.y;
    return a;
}
template <typename V> __host__ __device__ __forceinline__ V csub(V a, V b) {
    a.x -= b.x;
    a.y -= b.y;
    return a;
}
template <typename V> __host__ __device__ __forceinline__ V cmul(V a, V b) {
    V r;
    r.x = a.x * b.x - a.y * b.y;
    r.y = a.x * b.y + a.y * b.x;
    return r;
}
// a * conj(b)
template <typename V> __host__ __device__ __forceinline__ V cmulc(V a, V b) {
    V r;
    r.x = a.x * b.x + a.y * b.y;
    r.y = a.y * b.x - a.x * b.y;
    return r;
}
template <typename V> __host__ __device__ __forceinline__ V cconj(V a) {
    a.y = -a.y;
    return a;
}
template <typename V, typename S> __host__ __device__ __forceinline__ V cscale(V a, S s) {
    a.x *= s;
    a.y *= s;
    return a;
}
// multiply by s*i (s = +1 or -1)
template <typename V> __host__ __device__ __forceinline__ V cmul_si(V a, int s) {
    V r;
    if (s > 0) {
        r.x = -a.y;
        r.y = a.x;
    } else {
        r.x = a.y;
        r.y = -a.x;
    }
    return r;
}

// Programmatic dependent launch.  A kernel started by launch_pdl may begin while the kernel queued
// before it on the stream is still finishing: its blocks come up, load their twiddles and work
// out their indexes, and pdl_wait holds them until that kernel is complete and its
// writes are visible.  Every kernel started this way calls pdl_wait before it touches anything that
// an earlier kernel writes or reads (the pointers that go through it cannot be read
// ahead of it), and only then pdl_trigger, so that when the next kernel's blocks come up, all
// kernels before this one are complete.  What the kernel before may still be writing when this one
// comes up is read with plain loads (__ldca), not through the read-only path, whose data has to be
// constant while the kernel runs.
template <typename Ptr> __device__ __forceinline__ void pdl_wait(Ptr &p) {
    asm volatile("griddepcontrol.wait;" : "+l"(p)::"memory");
}
// The same where the compiler has to go on knowing that p points to global memory: loads through the
// pointer that comes out of pdl_wait are generic ones, which keep their order with stores to
// shared memory, so that a loop that copies rows there has one load in flight at a time.
template <typename Ptr> __device__ __forceinline__ void pdl_wait_global(Ptr &p) {
    size_t g = __cvta_generic_to_global(p);
    pdl_wait(g);
    p = reinterpret_cast<Ptr>(__cvta_global_to_generic(g));
}
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }

// Kernels with dynamic shared memory start this way up to 2400 CTAs, the others (particle and
// clearing kernels, Green cells) up to 600.  A kernel that starts early comes up with the
// shared-memory split of the one before it and keeps it for its whole run, so a gather loses its
// L1 and a transform its resident CTAs: with every launch early, the gather of 1e7 particles on
// 128 x 128 x 256 takes 700 us against 220 and the z pass 180 against 140.  What it gains is a few
// us per launch however large the grid is.  Steps in us with limits 0, 300, 600, 1200, 2400, 5000
// (600 at most for the kernels without dynamic shared memory; "all" without a limit): 32 x 32 x 48
// with refit 91 79 75 75 74 74 (all: 69), 64 x 64 x 128 117 114 114 114 110 110 (all: 106), 64^3
// cathode with refit 350 342 339 333 329 329 (all: 323), 128^3 FP64 589 589 588 585 579 580 (all: 688),
// 128 x 128 x 256 691 691 692 690 685 685 (all: 1227).
inline bool pdl_early(uint64_t ctas, size_t smem) { return ctas <= (smem > 0 ? 2400u : 600u); }
template <typename... KP, typename... A>
inline void launch_pdl(void (*kern)(KP...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A &&...args) {
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = pdl_early((uint64_t)grid.x * grid.y * grid.z, smem) ? 1 : 0;
    cudaLaunchKernelEx(&cfg, kern, KP(args)...);  // the caller checks cudaGetLastError
}

inline int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

}  // namespace osc

// Status codes mirror include/opensc_gpu.h.
#define OSC_OK 0
#define OSC_E_INVALID 1
#define OSC_E_BOUNDS 2
#define OSC_E_FFT_SIZE 3
#define OSC_E_ALLOC 4
#define OSC_E_CUDA 5
#define OSC_E_TIMEOUT 6
#define OSC_E_NAN 7
#define OSC_E_NOCHARGE 8
#define OSC_E_UNSUPPORTED 9
#define OSC_E_STATE 10
