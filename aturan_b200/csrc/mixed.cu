// FP32 instantiation of the aturan_b200 kernels: the mixed-precision path.
//
// State, n-copies, stage buffers, accumulator and forcing are stored and updated in FP32 and the
// stencils are FP32 arithmetic (FMA contraction allowed). The pressure family (p_dyn, p_hydro,
// p_baro, p_b0, p_bfollow) stays FP64: their gradients enter the momentum equations as
// differences of O(10) values and are formed in FP64 before rounding to FP32. The saturation
// adjustment computes in FP64 whatever the storage (satadj.cuh).
#include "launch.h"
#include "launch_impl.cuh"

namespace aturan {
ATURAN_DEFINE_LAUNCHERS(float, float)

__global__ void f64_to_f32_kernel(const double* in, float* out, size_t n){
    chain_wait();
    for(size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
        out[t] = (float)in[t];
}
__global__ void f32_to_f64_kernel(const float* in, double* out, size_t n){
    chain_wait();
    for(size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
        out[t] = (double)in[t];
}
__global__ void scale_copy_f32_kernel(const float* in, float* out, size_t n, double coeff){
    chain_wait();
    for(size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
        out[t] = (float)(coeff * (double)in[t]);
}
void launch_scale_copy_f32(const float* in, float* out, size_t n, double coeff, cudaStream_t st){
    chain(scale_copy_f32_kernel, 148 * 8, 256, 0, st, in, out, n, coeff);
}

// Contiguous [im][jm][km] FP64 <-> padded [im][jm][kp] fields, the layout change and (FP32 fields, the
// temperature pair of common.cuh) the conversion in one pass, every field of a batch in one launch
// (blockIdx.y). A pure copy, bound by HBM: a thread moves PACK_U values of the contiguous side, a block
// apart, all loads before the stores, so each warp access covers whole 128-byte lines of the contiguous
// side and the rows' breaks cost nothing (the row by a multiply-shift division). One launch per field with
// one value per thread moved 41x181x361 FP64 fields at 3.2 TB/s, this form moves them at the measured copy
// rate (6.5 TB/s).
constexpr int PACK_NT = 256, PACK_U = 8;
template <bool IN>
__global__ void __launch_bounds__(PACK_NT) pack_kernel(const __grid_constant__ PackBatch p){
    chain_wait();
    const int f = blockIdx.y;
    const unsigned base = blockIdx.x * (PACK_NT * PACK_U) + threadIdx.x;
    const double* const cin = p.flat[f];
    double* const cout = const_cast<double*>(p.flat[f]);
    unsigned q[PACK_U];                              // the values' places in the padded field
    bool on[PACK_U];
#pragma unroll
    for(int u = 0; u < PACK_U; u++){
        const unsigned e = base + u * PACK_NT;
        on[u] = e < p.n;
        const unsigned r = (unsigned)(((unsigned long long)e * p.div_m) >> p.div_s);      // e / km
        q[u] = r * (unsigned)(p.kp - p.km) + e;
    }
    if(p.kind[f] == PACK_F64){
        double* const d = reinterpret_cast<double*>(p.dev[f]);
        double v[PACK_U];
#pragma unroll
        for(int u = 0; u < PACK_U; u++) if(on[u]) v[u] = IN ? cin[base + u * PACK_NT] : d[q[u]];
#pragma unroll
        for(int u = 0; u < PACK_U; u++) if(on[u]){ if(IN) d[q[u]] = v[u]; else cout[base + u * PACK_NT] = v[u]; }
    } else if(IN){
        float* const d = reinterpret_cast<float*>(p.dev[f]);
        float* const lo = p.kind[f] == PACK_PAIR ? p.lo[f] : nullptr;
        double v[PACK_U];
#pragma unroll
        for(int u = 0; u < PACK_U; u++) if(on[u]) v[u] = cin[base + u * PACK_NT];
#pragma unroll
        for(int u = 0; u < PACK_U; u++) if(on[u]) t_st(d, lo, q[u], v[u]);
    } else {
        const float* const d = reinterpret_cast<const float*>(p.dev[f]);
        const float* const lo = p.kind[f] == PACK_PAIR ? p.lo[f] : nullptr;
        double v[PACK_U];
#pragma unroll
        for(int u = 0; u < PACK_U; u++) if(on[u]) v[u] = t_ld(d, lo, q[u]);
#pragma unroll
        for(int u = 0; u < PACK_U; u++) if(on[u]) cout[base + u * PACK_NT] = v[u];
    }
}
void launch_pack(PackBatch& p, int nf, int km, int kp, size_t rows, bool in, cudaStream_t st){
    p.km = km; p.kp = kp; p.n = (unsigned)(rows * km);         // a context's fields hold < 2^31 values
    int s = 0;
    while((1u << s) < (unsigned)km) s++;
    p.div_s = 31 + s;                                          // exact for e < 2^31: m = ceil(2^(31 + s) / km) < 2^32
    p.div_m = (unsigned)(((1ull << (31 + s)) + km - 1) / km);
    const dim3 grid((p.n + PACK_NT * PACK_U - 1) / (PACK_NT * PACK_U), nf);
    if(in) chain(pack_kernel<true>, grid, PACK_NT, 0, st, p);
    else   chain(pack_kernel<false>, grid, PACK_NT, 0, st, p);
}
__global__ void scale_copy_pair_kernel(const float* hi, const float* lo, float* ohi, float* olo, size_t n, double coeff){
    chain_wait();
    for(size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < n; t += (size_t)gridDim.x * blockDim.x)
        t_st(ohi, olo, t, coeff * t_ld(hi, lo, t));
}
void launch_scale_copy_pair(const float* hi, const float* lo, float* ohi, float* olo, size_t n, double coeff, cudaStream_t st){
    chain(scale_copy_pair_kernel, 148 * 8, 256, 0, st, hi, lo, ohi, olo, n, coeff);
}

void launch_f64_to_f32(const double* in, float* out, size_t n, cudaStream_t st){
    chain(f64_to_f32_kernel, 148 * 8, 256, 0, st, in, out, n);
}
void launch_f32_to_f64(const float* in, double* out, size_t n, cudaStream_t st){
    chain(f32_to_f64_kernel, 148 * 8, 256, 0, st, in, out, n);
}
}  // namespace aturan
