// Shared by the wave stencils on periodic grids (pm.cu, wave_march.cu): vectors of x-cells, the
// arithmetic of one cell with every rounding written out, programmatic dependent launches.
#pragma once

#include "kernels.cuh"

namespace rrg {

// V consecutive x-cells of a row
template <typename R, int V>
struct alignas(sizeof(R) * V) Cells {
    R v[V];
};

__device__ __forceinline__ float radd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double radd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float rmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double rmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float rfma(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ double rfma(double a, double b, double c) { return __fma_rn(a, b, c); }

// km (sum of the six neighbours) + ka c + ko po, in wave_cell's order and roundings
template <typename R>
__device__ __forceinline__ R wave_cell_adj(R l, R r, R ym, R yp, R zm, R zp, R c, R po, R km,
                                           R ka, R ko) {
    const R nb = radd(radd(radd(radd(radd(l, r), ym), yp), zm), zp);
    return rfma(po, ko, rfma(c, ka, rmul(nb, km)));
}

// Programmatic dependent launch: a kernel launched by launch_pdl may start while the kernel before
// it still runs. pdl_next lets the next kernel's blocks start; pdl_wait returns when the kernel
// before has completed and its writes are visible. Every block of such a kernel waits, so a
// kernel that has completed leaves none of its predecessors running.
__device__ __forceinline__ void pdl_next() { asm volatile("griddepcontrol.launch_dependents;" ::); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

// Loads of data that the kernel before may have written: plain (coherent) global loads, volatile
// so that none moves ahead of pdl_wait.
__device__ __forceinline__ float4 ldv(const float4* p) {
    float4 v;
    asm volatile("ld.global.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 ldv(const float2* p) {
    float2 v;
    asm volatile("ld.global.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ float ldv(const float* p) {
    float v;
    asm volatile("ld.global.f32 %0, [%1];" : "=f"(v) : "l"(p));
    return v;
}
__device__ __forceinline__ double2 ldv(const double2* p) {
    double2 v;
    asm volatile("ld.global.v2.f64 {%0, %1}, [%2];" : "=d"(v.x), "=d"(v.y) : "l"(p));
    return v;
}
__device__ __forceinline__ double ldv(const double* p) {
    double v;
    asm volatile("ld.global.f64 %0, [%1];" : "=d"(v) : "l"(p));
    return v;
}

template <typename R, int V>
__device__ __forceinline__ Cells<R, V> load_cells(const R* p) {
    Cells<R, V> c;
    if constexpr (V == 1) {
        c.v[0] = ldv(p);
    } else if constexpr (V == 4) {
        const float4 t = ldv(reinterpret_cast<const float4*>(p));
        c.v[0] = t.x;
        c.v[1] = t.y;
        c.v[2] = t.z;
        c.v[3] = t.w;
    } else if constexpr (sizeof(R) == 4) {
        const float2 t = ldv(reinterpret_cast<const float2*>(p));
        c.v[0] = t.x;
        c.v[1] = t.y;
    } else {
        const double2 t = ldv(reinterpret_cast<const double2*>(p));
        c.v[0] = t.x;
        c.v[1] = t.y;
    }
    return c;
}

template <typename... Params, typename... Args>
void launch_pdl(void (*kernel)(Params...), dim3 grid, dim3 block, size_t smem, cudaStream_t s,
                Args... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    RRG_CUDA(cudaLaunchKernelEx(&cfg, kernel, static_cast<Params>(args)...));
}

}  // namespace rrg
