// Shared device/host helpers for the sm_103a kernels of the ADRT oblique inverses.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "adrt_pinv_gb300.h"

namespace adrt {

// ------------------------------------------------------------------ complex arithmetic on interleaved pairs
template <typename real> struct cx;
template <> struct cx<float> { using t = float2; };
template <> struct cx<double> { using t = double2; };
template <typename real> using cplx = typename cx<real>::t;

template <typename real> __host__ __device__ __forceinline__ cplx<real> mk(real re, real im) {
    cplx<real> r; r.x = re; r.y = im; return r;
}
template <typename C> __device__ __forceinline__ C cadd(C a, C b) { C r; r.x = a.x + b.x; r.y = a.y + b.y; return r; }
template <typename C> __device__ __forceinline__ C csub(C a, C b) { C r; r.x = a.x - b.x; r.y = a.y - b.y; return r; }
// a + w * b (complex multiply-add, 4 FMAs)
template <typename C> __device__ __forceinline__ C cfma(C w, C b, C a) {
    C r;
    r.x = fma(w.x, b.x, fma(-w.y, b.y, a.x));
    r.y = fma(w.x, b.y, fma(w.y, b.x, a.y));
    return r;
}
// w * b
template <typename C> __device__ __forceinline__ C cmul(C w, C b) {
    C r;
    r.x = fma(w.x, b.x, -w.y * b.y);
    r.y = fma(w.x, b.y, w.y * b.x);
    return r;
}
// conj(w) * b
template <typename C> __device__ __forceinline__ C cmulc(C w, C b) {
    C r;
    r.x = fma(w.x, b.x, w.y * b.y);
    r.y = fma(w.x, b.y, -w.y * b.x);
    return r;
}
// conj(w0) * a + conj(w1) * b
template <typename C> __device__ __forceinline__ C cdot2c(C w0, C a, C w1, C b) {
    C r;
    r.x = fma(w0.x, a.x, fma(w0.y, a.y, fma(w1.x, b.x, w1.y * b.y)));
    r.y = fma(w0.x, a.y, fma(-w0.y, a.x, fma(w1.x, b.y, -w1.y * b.x)));
    return r;
}
template <typename C, typename S> __device__ __forceinline__ C cscale(S s, C a) { C r; r.x = s * a.x; r.y = s * a.y; return r; }

// ------------------------------------------------------------------ bit utilities (usable in constant expressions)
__host__ __device__ constexpr int brev(int x, int bits) {
    int r = 0;
    for (int i = 0; i < bits; ++i) r |= ((x >> i) & 1) << (bits - 1 - i);
    return r;
}
__host__ __device__ constexpr int imax(int a, int b) { return a > b ? a : b; }
__host__ __device__ constexpr int imin(int a, int b) { return a < b ? a : b; }

// ------------------------------------------------------------------ error reporting shared by the C ABI
void set_error(const char* fmt, ...);
int cuda_status(cudaError_t e, const char* where);
int launch_status(const char* where);
// the status of a cudaLaunchKernelEx call: its own return value (cluster launches can be refused there), then the
// launch error state
int launch_ex_status(cudaError_t launched, const char* where);

inline cudaStream_t as_stream(void* s) { return reinterpret_cast<cudaStream_t>(s); }

// ------------------------------------------------------------------ chained launches (programmatic dependent launch)
// The kernels of a packed pass and the outer step follow one another on a stream, a few microseconds each. Launched with
// launch_chained, a kernel may be set up on the SMs once every CTA of its predecessor has exited, while the predecessor's
// writes drain; it touches global memory only after chain_wait (the predecessor has completed and its writes are visible),
// so a kernel that has completed has all earlier ones complete before it. In a plain launch chain_wait does nothing. Whole
// inverses as graphs, plain / chained launches: FP64 N = 64 single 467 / 424 us, N = 256 single 995 / 936, N = 512 b6 7248 /
// 7182, N = 256 b64 9147 / 9128. (With griddepcontrol.launch_dependents at the top of every kernel: 744, 1280, 7378 and 9774;
// the next grid's CTAs then crowd onto the SMs that have room beside the running ones.)
__device__ __forceinline__ void chain_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// a const __restrict__ parameter as the predecessor left it: loads through the result stay behind chain_wait and are
// ordinary ones (the non-coherent path is for data no one writes while the kernel exists)
template <typename T> __device__ __forceinline__ T* after_wait(T* p) {
    asm volatile("" : "+l"(p)::"memory");
    return p;
}
template <typename... P, typename... A>
inline int launch_chained(const char* where, void (*kern)(P...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return launch_ex_status(cudaLaunchKernelEx(&cfg, kern, static_cast<P>(args)...), where);
}

// number of kernels this library has launched (all threads), for launch accounting
void count_launch();

}  // namespace adrt
