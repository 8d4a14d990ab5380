// Device layout, per-(i,j) geometry and derived constants shared by every aturan_b200 kernel.
//
// HBM layout: one field is a block [i][j][kp] with the longitude row padded from km to kp (a
// multiple of 32 elements) so that every row starts on a 256-byte boundary for FP64 (128-byte
// for FP32) and a warp's 32 consecutive k land in whole sectors. Field f of an arena starts at
// base + f * fstride. k = km-1 is the seam copy of k = 0; padding columns are never read.
#pragma once
#include <utility>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stddef.h>
#include "aturan_b200.h"

namespace aturan {

// a / d by the reciprocal y = 1 / d that the caller holds (itself a division's result), correctly
// rounded, the same bits as the division: after one correction the quotient is faithful, and the
// remainder of a faithful quotient is exact, so the second rounds as the division does (Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", 1990). For a, d and
// a / d well inside the normal range (or a = +0); elsewhere the last bit, or an infinity, may differ.
// Five multiply-adds without a branch, against ~10, a reciprocal estimate and a branch for a division.
__host__ __device__ __forceinline__ double div_by(double a, double d, double y){
    double q = a * y;
    q = fma(fma(-q, d, a), y, q);
    return fma(fma(-q, d, a), y, q);
}

// Launches of one stream follow one another by programmatic stream serialisation: the next kernel's
// blocks are placed once the last block of the kernel before has exited, beside the flush of its
// writes and the launch's own latency, and every kernel waits (chain_wait, its first statement) until
// that flush is done before it touches what another launch writes. An empty kernel launched after another in a stream
// took 4.1 us and takes 2.0 so; eight dependent loads a thread, 600 blocks: 6.2 and 3.5. Only the point passes of
// the pressure solves let their successor in before they end (sor_colour_kernel): elsewhere that was no
// faster (3.5 to 4.6 us), and so a block never starts while one that may hold the successor's input in
// its L1 still reads. A kernel that does not begin with chain_wait, reads what launches write by the read-only
// path (ldr below), or follows a point pass, is launched the plain way.
__device__ __forceinline__ void chain_wait(){ cudaGridDependencySynchronize(); }

template <typename... E, typename... A>
inline cudaError_t chain_if(bool chained, void (*kernel)(E...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args){
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = chained ? 1 : 0;
    return cudaLaunchKernelEx(&cfg, kernel, static_cast<E>(args)...);
}
template <typename... E, typename... A>
inline cudaError_t chain(void (*kernel)(E...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, A&&... args){
    return chain_if(true, kernel, grid, block, smem, st, std::forward<A>(args)...);
}

// Lets a kernel be launched with `bytes` of dynamic shared memory. Above the default 48 KB the kernel has to be
// given a higher limit, which belongs to it on the current device, whatever context or thread asked for it
// last. So every launch that needs it asks for the most a block can have, and nothing remembers that it did:
// a flag per process would leave the kernels of a second device without it, and a limit fitted to one
// context would take it from a larger one. False: the device does not allow it.
constexpr int SMEM_BLOCK_MAX = 227 * 1024;
template <typename... E>
inline bool smem_opt_in(void (*kernel)(E...), size_t bytes){
    if(bytes <= 48 * 1024) return true;
    if(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BLOCK_MAX) == cudaSuccess) return true;
    cudaGetLastError();
    return false;
}

// A value that a launch writes, by a plain load. The read-only path (__ldg, or a const pointer with
// __restrict__) wants memory that nobody writes while the kernel lives, and a chained kernel lives before
// the one ahead of it has flushed its writes: the wait holds back neither a read-only load that the compiler
// moves ahead of it nor one's cache. That path is for the tables formed with the context, for what the point
// pass reads before its wait, and for kernels launched the plain way (ldr). Two of them gain more by it than
// the chaining gave them: the FP64 momentum stage (the RK4 step at 41x181x361 with its transfers: 2.75 ms
// chained with plain loads, 2.69 so) and the adjoint's reverse stage (dry gradient: 1.34 and 1.33 ms). The
// others take the same time with either load.
template <typename T>
__device__ __forceinline__ T ld(const T* p){ return *p; }
template <typename T>
__device__ __forceinline__ T ldr(const T* p){ return __ldg(p); }

constexpr int IM_MAX = 512;        // levels of a context's grid
struct Grid {
    int im, jm, km, kp;
    size_t fstride;            // elements per field (im * jm * kp)
};

__host__ __device__ __forceinline__ size_t gidx(const Grid& g, int i, int j, int k){
    return ((size_t)i * g.jm + j) * g.kp + k;
}

// ATPhys.h:135-139, the periodic seam: ring of km-1 distinct meridians.
__host__ __device__ __forceinline__ int phi_wrap(int kk, int km){
    const int n = km - 1;
    return kk < 0 ? kk + n : (kk >= n ? kk - n : kk);
}

// Per-(i,j) metric of RungeKutta_Uran_Turb.cpp:258-283 plus the products of it the RHS forms
// (RHS_Uran_Turb.cpp:224-331), computed once on the host in FP64 in the reference's operand
// order and uploaded, so the device reads exactly the CPU's values.
template <typename T>
struct GeoIJ {
    T inv_rm, inv_rm2, inv_rmsinthe, inv_rm2sinthe, inv_rm2sinthe2, costhe_inv_rm2sinthe;
    T costhe, cotanthe, v_metric, two_inv_rm, sinthe_bf, cent_rad, cent_the, sponge;
};

// Scalars of the RHS and the RK4 update, precomputed on the host in the operand order in which
// the reference forms them (each product noted beside its field).
template <typename T>
struct RhsConst {
    T inv_2dr, inv_2dthe, inv_2dphi, inv_dr2, inv_dthe2, inv_dphi2;
    T ce_sp;            // coeff_energy_p * scale_p
    T scale_p;
    T m2om, p2om;       // -2 omega, +2 omega
    T cor_sc;           // Coriolis * scale_Cor
    T cor_rad_f;        // cor_rad_on * Coriolis * scale_Cor  (0: CORIOLIS_SPLIT)
    T cen_f;            // 1.0 * centrifugal * cent_mom * scale_cen
    T re, re_pr, re_eff, inv_re;
    T turb_coupling, precip_coupling, chemical_reaction;
    T tmf;              // tmf_scale * chemical_reaction
    T precip_L;         // L_atm * 1e3
    T precip_den;       // r_mix * cp_mix * u_0 * t_ref
    T sc_re[5];         // sc * re for ch4, h2o, h2s, nh3, nh4sh
    T stokes_a;         // (2/9) r_p r_p
    T rho_cond_nh4sh, g, mue_mix, u_0;
    T cp_mix, t_ref;
    T cp_rh2, cp_he_term, cp_ch4_term, cp_rsum, cp_h2_const;   // cp(T), CpH2.h:122-134
    T tke_max, dis_min, t_min, t_max, dt;
    T heat_scale;       // (L_atm * 1e3 / u_0) / t_ref: a heating rate in K/s as a tendency of t
    // reciprocals of the divisors above, for the mixed form's multiplications (qdiv)
    T inv_re_eff, inv_re_pr, inv_sc_re[5], inv_mue_mix, inv_u_0, inv_precip_den, inv_cp_rsum;
    int cp_dyn, cp_gas, cp_mode, turb_active;
};

// Constants of the buoyancy reference level and the hydrostatic column integral
// (RungeKutta_Uran_Turb.cpp:18-177).
struct HydroConst {
    double g, rR, t_ref;       // b = g p / (rR T t_ref), rR = r_mix * R_mix
    double m_nd_rel_b;         // -nd_rel * buoy_scale * buoyancy (buoy_scale = 1)
    double dr, follow_tau;
    int follow_on;
};

// Scratch of the exact (reference-order) level means: the terms, per-chunk sums and flags, and the
// per-chunk binades and units (rk4.cuh, buoy_terms_kernel to buoy_serial_pass_kernel).
struct BuoyScratch {
    double* terms;          // [im][2][jm*km]
    double* bpart;          // [im][nbx][3]
    int* bexp;              // [im][nbx][2]
    long long* bunits;      // [im][nbx][4]
    int nbx;                // chunks per level
};

constexpr int CP_TABLE_N = 2991;   // (1500 - 5) / 0.5 + 1, CpH2.h:66-75

// The mixed form carries the temperature (t and its start-of-step copy tn) as an FP32 pair: the
// stored FP32 value hi, which every stencil reads, and lo = the FP32-rounded remainder T - hi, so
// that T = hi + lo to about 2^-48 relative. The kernels that write T (the RK4 final update, the
// saturation adjustment, the passes after RK4, the layout kernels) form it in FP64 from hi + lo
// and store both halves. Without lo the FP32 rounding of T (~6e-8) moves the adjustment's
// relative 1e-3 stopping test (SaturationAdjustment.h:250-251) to another pass in some cells of
// the CH4 band, a jump of ~1e-5 in T there. lo is null in an FP64 context (and ignored).
template <typename S>
__device__ __forceinline__ double t_ld(const S* hi, const float* lo, size_t q){
    double v = (double)hi[q];
    if(lo) v += (double)lo[q];
    return v;
}
template <typename S>
__device__ __forceinline__ void t_st(S* hi, float* lo, size_t q, double v){
    const S h = (S)v;
    hi[q] = h;
    if(lo) lo[q] = (float)(v - (double)h);
}

}  // namespace aturan
