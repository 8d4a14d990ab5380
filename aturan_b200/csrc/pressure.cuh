// Poisson pressure solves of the dynamic pressure p_dyn (always FP64 on the device).
//
// GS_LEX reproduces PressureSolverUran::run() (planet/PressureSolverUran.h:33-250): ONE
// lexicographic Gauss-Seidel sweep i -> j -> k over the interior, in place. A serial sweep
// makes cell (i,j,k) see the NEW values of (i-1,j,k), (i,j-1,k), (i,j,k-1) and the OLD values of
// (i+1,j,k), (i,j+1,k), (i,j,k+1); at the seam k = 0 reads the old k = km-2 and k = km-2 reads
// the new k = 0. Every one of those relations is preserved by sweeping the hyperplanes
// s = i + j + k in increasing order (gs_wave_kernel), all cells of one hyperplane in parallel: a neighbour with a
// smaller coordinate sum is already new, one with a larger sum is still old (the seam pair
// included: k = km-2 lies km-2 hyperplanes after k = 0). So the wavefront computes exactly the
// serial sweep's values, cell for cell, with no change in any arithmetic.
//
// RB_SHARED reproduces PressureSolver<Planet>::run() (planet/PressureSolver.h:145-766) with
// N sweeps: red-black colouring on (i+j+k)&1, the div(aux) source clamped at den*p_dyn_cap, the
// model's projection boundaries first (planet/Pressure_Uran.cpp:30-146) and the p_dyn boundary
// passes inside the sweep loop.
#pragma once
#include <climits>
#include "common.cuh"

namespace aturan {

constexpr double C43 = 4.0 / 3.0, C13 = 1.0 / 3.0;   // cUranusModel.h:866

// Per-(i,j) weights of PressureSolverUran (sweep and defect-correction source; :139-199).
struct GSW {
    double num1, num2, num3, inv_denom;           // sweep, :180-190
    double inv_rm, inv_rmsinthe;                  // both sources
    double n1, n2, n3, denom;                     // incr_src, :151-157
};

// Per-(i,j) weights of the shared solver (:326-353) and its clamp bound den * p_dyn_cap.
struct RBW {
    double num1, num2, num3, den, inv_rm, inv_rmsinthe, src_max;
};

struct PressConst {
    double inv_2dr, inv_2dthe, inv_2dphi, two_dr, two_dthe, two_dphi, src_scale;   // inv_x: 1 / two_x
    int press_incr;
};

// ---- PressureSolverUran.h:70-81: aux radial planes ----
template <typename S>
__global__ void gs_aux_bc_kernel(Grid g, S* au, S* av, S* aw){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    if(k > g.km - 2 || j > g.jm - 2) return;
    S* A[3] = {au, av, aw};
    // every load before the first store (which each of them would otherwise wait for)
    S lo[3], hi[3];
#pragma unroll
    for(int q = 0; q < 3; q++){
        const S* a = A[q];
        lo[q] = (S)(C43 * (double)a[gidx(g, 1, j, k)] - C13 * (double)a[gidx(g, 2, j, k)]);
        hi[q] = (S)(C43 * (double)a[gidx(g, g.im - 2, j, k)] - C13 * (double)a[gidx(g, g.im - 3, j, k)]);
    }
#pragma unroll
    for(int q = 0; q < 3; q++){ A[q][gidx(g, 0, j, k)] = lo[q]; A[q][gidx(g, g.im - 1, j, k)] = hi[q]; }
}

// ---- PressureSolverUran.h:139-175: incr_src = src_scale div(rhs) + Lc(p_old), the radial
// end planes of rhs_u read as their 2-point extrapolation ----
template <typename S>
__global__ void gs_incr_kernel(Grid g, const S* ru, const S* rv, const S* rw, const double* P,
                               const GSW* w, PressConst c, double* incr){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    const int i = 1 + blockIdx.z;
    if(k > g.km - 2 || j > g.jm - 2) return;
    const GSW W = w[i * g.jm + j];
    const int kw = phi_wrap(k - 1, g.km), ke = phi_wrap(k + 1, g.km);
    auto RU = [&](int ii) -> double {
        if(ii == 0) return C43 * (double)ru[gidx(g, 1, j, k)] - C13 * (double)ru[gidx(g, 2, j, k)];
        if(ii == g.im - 1) return C43 * (double)ru[gidx(g, g.im - 2, j, k)] - C13 * (double)ru[gidx(g, g.im - 3, j, k)];
        return (double)ru[gidx(g, ii, j, k)];
    };
    const double du = RU(i + 1) - RU(i - 1);
    const double dv = (double)rv[gidx(g, i, j + 1, k)] - (double)rv[gidx(g, i, j - 1, k)];
    const double dw = (double)rw[gidx(g, i, j, ke)] - (double)rw[gidx(g, i, j, kw)];
    double div_rhs = div_by(du, c.two_dr, c.inv_2dr) + div_by(dv, c.two_dthe, c.inv_2dthe) * W.inv_rm
                   + div_by(dw, c.two_dphi, c.inv_2dphi) * W.inv_rmsinthe;
    if(!isfinite(div_rhs))                    // an infinity's quotient (div_by makes it a NaN)
        div_rhs = du / c.two_dr + dv / c.two_dthe * W.inv_rm + dw / c.two_dphi * W.inv_rmsinthe;
    const double lc_old =
          (P[gidx(g, i + 1, j, k)] + P[gidx(g, i - 1, j, k)]) * W.n1
        + (P[gidx(g, i, j + 1, k)] + P[gidx(g, i, j - 1, k)]) * W.n2
        + (P[gidx(g, i, j, ke)] + P[gidx(g, i, j, kw)]) * W.n3
        - W.denom * P[gidx(g, i, j, k)];
    incr[gidx(g, i, j, k)] = c.src_scale * div_rhs + lc_old;
}

// The source of the sweep without the defect correction (press_incr = 0): src_scale div(aux), formed
// before the sweep (it reads no pressure).
template <typename S>
__global__ void gs_src_kernel(Grid g, const S* au, const S* av, const S* aw, const GSW* w, PressConst c, double* src){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    const int i = 1 + blockIdx.z;
    if(k > g.km - 2 || j > g.jm - 2) return;
    const GSW W = w[i * g.jm + j];
    const int kw = phi_wrap(k - 1, g.km), ke = phi_wrap(k + 1, g.km);
    const double du_dr   = ((double)au[gidx(g, i + 1, j, k)] - (double)au[gidx(g, i - 1, j, k)]) * c.inv_2dr;
    const double dv_dthe = ((double)av[gidx(g, i, j + 1, k)] - (double)av[gidx(g, i, j - 1, k)]) * c.inv_2dthe * W.inv_rm;
    const double dw_dphi = ((double)aw[gidx(g, i, j, ke)] - (double)aw[gidx(g, i, j, kw)]) * c.inv_2dphi * W.inv_rmsinthe;
    src[gidx(g, i, j, k)] = c.src_scale * (du_dr + dv_dthe + dw_dphi);
}

// ---- PressureSolverUran.h:177-211: the lexicographic sweep as ONE launch ----
// The sweep's dependency chain is (im-2)+(jm-2)+(km-1) cells long, so what bounds it is the time of
// one hyperplane. As a launch per hyperplane that was 2.3 us (576 launches, 1.31 ms at 41x181x361);
// here a hyperplane step is one block barrier and one trip through shared memory: 0.235 ms (0.041
// against 0.244 ms at 21x37x73). A step takes 0.17 us with 4 sweeping warps per block, 0.23 us with 8
// and 0.32 us with 12 (the shared-memory pipe is then 60 % busy). A band lags the one before by its own
// rows' steps and a hand-over of ~2 us, so at 41x181x361 the chain is 577 steps and 22 hand-overs.
//
// A block owns a band of B rows j and all levels i; its thread (i, j) walks its row along k, at step
// s on cell k = s - i - j. The rows lie in a ring of 32 values in shared memory, the new value
// written over the old one, so at step s the slot k of the neighbour rows (i-1, j) and (i, j-1)
// holds the new value (written at step s - 1) and the slot k of (i+1, j) and (i, j+1) still the old
// one: the wavefront's order, read by one barrier per step. A row of 16 lanes has 16 consecutive i,
// so its lanes' slots fall in 16 different bank pairs.
//   Memory: per row 16 values at a time, by the mover warps. When a row has passed k = 16 c + 1 its
// chunk c - 1 is finished and read by nobody any more; the movers write it out and fetch chunk c + 1
// into its place (cp.async), at least 10 steps ahead of the chunk's first reader. Levels 0 and im-1
// and the row after the band are rows that are only fetched.
//   Between bands: the band's last row also leaves each new value in a global edge buffer, as two
// 8-byte words of half the value and a tag (the launch's number), so a reader sees from the word
// itself whether it has been written, without a fence. The receiver warps of the next band poll
// these words up to 32 steps ahead and put the values into a ring of steps in shared memory. Bands
// are taken in the order in which blocks start (a ticket), so a band waits only for one that runs.
// Every wait is bounded: on running out it sets *err and waits no more.
constexpr int GSR = 32;                           // ring: values per row, and steps of the incoming edge
constexpr int GSC = 16;                           // values per chunk
constexpr int GSB_MAX = 8;
struct GsEdge { unsigned lo, tag_lo, hi, tag_hi; };
constexpr int GS_MOVERS = 128;                    // threads of the mover warps
struct GsPlan { int ipad, B, nb, steps, nc; size_t smem; };   // nb = 0: a column does not fit, no plan

// Rows per band: as many as the shared memory holds, at most 8 (more rows per band make fewer bands
// to wait for, but more warps per barrier). nc: the sweeping threads, one of the three counts the
// kernel is built for (a barrier whose count is not a constant costs 160 cycles, else 40).
inline GsPlan gs_plan(const Grid& g){
    GsPlan p{};
    p.ipad = (g.im + GSC - 1) / GSC * GSC;
    auto smem = [&](int B){ return (size_t)p.ipad * (2 * B + 1) * GSR * 8 + (size_t)p.ipad * GSR * 8 + 256; };
    int B = GSB_MAX;
    while(B > 0 && (smem(B) > SMEM_BLOCK_MAX || p.ipad * B > 384)) B--;
    if(B == 0) return p;
    if(B > g.jm - 2) B = g.jm - 2;
    p.B = B; p.nb = (g.jm - 2 + B - 1) / B; p.steps = g.im + B + g.km; p.smem = smem(B);
    p.nc = (p.ipad * B + 127) / 128 * 128;
    return p;
}
inline int gs_threads(const GsPlan& p){ return p.nc + GS_MOVERS + (p.ipad + 31) / 32 * 32; }
inline size_t gs_edge_bytes(const GsPlan& p){ return (size_t)p.nb * p.steps * p.ipad * sizeof(GsEdge); }

__device__ __forceinline__ void gs_cp16(void* smem, const void* gmem){
    const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" :: "r"(sa), "l"(gmem) : "memory");
}
__device__ __forceinline__ bool gs_edge_get(const GsEdge* e, unsigned tag, double& v){
    unsigned lo, t0, hi, t1;
    asm volatile("ld.volatile.global.v4.u32 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(lo), "=r"(t0), "=r"(hi), "=r"(t1) : "l"(e) : "memory");
    v = __longlong_as_double((long long)(((unsigned long long)hi << 32) | lo));
    return t0 == tag && t1 == tag;
}

// tag: this launch's number (from 1); ticket counts blocks over all launches (base: before this one).
// NC sweeping threads, then the mover warps, then the receiver warps.
template <int NC>
static __global__ void __launch_bounds__(768, 1) gs_wave_kernel(Grid g, double* P, const double* src, const GSW* w,
                                                                GsPlan pl, GsEdge* edge, unsigned* ticket, unsigned base,
                                                                unsigned tag, int* err){
    chain_wait();
    extern __shared__ __align__(16) double gs_sm[];
    const int ipad = pl.ipad, B = pl.B;
    double* ringP = gs_sm;                                    // [B + 1][ipad][GSR]
    double* ringS = ringP + (B + 1) * ipad * GSR;             // [B][ipad][GSR]
    double* ringE = ringS + B * ipad * GSR;                   // [GSR steps][ipad]
    volatile int* sync_ = reinterpret_cast<volatile int*>(ringE + ipad * GSR);
    volatile int* prog = sync_;                               // steps the rows have finished
    volatile int* recv = sync_ + 1;                           // per receiver warp: the last step received (<= 32 warps)
    volatile int* landed = sync_ + 33;                        // per mover warp: the last step whose chunks are in
    volatile int* band_s = sync_ + 40;
    const int t = threadIdx.x;
    if(t == 0) *band_s = (int)(atomicAdd(ticket, 1u) - base);
    __syncthreads();
    const int b = *band_s;
    if(b < 0 || b >= pl.nb) return;
    const int j0 = 1 + b * B, j1 = min(j0 + B - 1, g.jm - 2);
    const int s_lo = 1 + j0, s_hi = (g.im - 2) + j1 + (g.km - 2);
    if(t == 0) *prog = s_lo - 1;
    if(t < 32) recv[t] = s_lo - 1;
    if(t < GS_MOVERS / 32) landed[t] = s_lo - 1;
    constexpr int LIMIT = 1 << 22;
    const int PL = g.jm * g.kp;                                // elements of a plane (a context holds < 2^31)

    // chunk work of 16 lanes on the 16 rows i0 .. i0 + 15 of row jb (ipad is a multiple of 16): four
    // lanes per row, four values each as two 16-byte accesses (km - 1 is even, so the pairs of the
    // swept cells k <= km - 2 are whole). Row jb is swept for jb <= j1 - j0, fetched for one more.
    const int e = t & (GSC - 1), e4 = (e & 3) * 4;
    auto fetch = [&](int jb, int ir, int kn){                  // values kn .. kn + 3 of row (ir, j0 + jb)
        const int q = (jb * ipad + ir) * GSR + (kn & (GSR - 1)), o = ir * PL + (j0 + jb) * g.kp + kn;
        const bool sw = j0 + jb <= j1 && ir >= 1 && ir <= g.im - 2;
#pragma unroll
        for(int h = 0; h < 4; h += 2)
            if(kn + h <= g.km - 2){
                gs_cp16(ringP + q + h, P + o + h);
                if(sw) gs_cp16(ringS + q + h, src + o + h);
            }
    };
    auto flush = [&](int jb, int ir, int kf){                  // values kf .. kf + 3 of a swept row
        const int q = (jb * ipad + ir) * GSR + (kf & (GSR - 1)), o = ir * PL + (j0 + jb) * g.kp + kf;
#pragma unroll
        for(int h = 0; h < 4; h += 2)
            if(kf + h <= g.km - 2)
                *reinterpret_cast<double2*>(P + o + h) = *reinterpret_cast<const double2*>(ringP + q + h);
    };
    const int gpr = ipad / GSC, ngrp = gpr * (j1 - j0 + 2);    // groups of 16 rows: the swept rows and one more
    // chunks 0 and 1 of every row, and each row's old value at km - 2 (the west neighbour of k = 0)
    for(int q = t / GSC; q < ngrp; q += (int)blockDim.x / GSC){
        const int jb = q / gpr, i0 = (q - jb * gpr) * GSC;
        for(int r = e >> 2; r < GSC && i0 + r < g.im; r += 4){ fetch(jb, i0 + r, e4); fetch(jb, i0 + r, GSC + e4); }
    }
    const int jb = t / ipad, i = t - jb * ipad, j = j0 + jb;   // a sweeping thread's row
    const bool act = t < NC && jb < B && j <= j1 && i >= 1 && i <= g.im - 2;
    double kw = 0.0, new0 = 0.0;
    GSW W{};
    if(act){ W = w[i * g.jm + j]; kw = P[gidx(g, i, j, g.km - 2)]; }
    asm volatile("cp.async.commit_group;\n cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();

    if(t >= NC + GS_MOVERS){
        // receiver warps: lane <-> i, four steps at a time
        const int wr = (t - NC - GS_MOVERS) >> 5, lane = t & 31;
        const int i = wr * 32 + lane;
        const bool on = i >= 1 && i <= g.im - 2;
        // band b - 1's edge: its step numbering starts at 1 + (j0 - B)
        const GsEdge* E = edge + (size_t)(b - 1) * pl.steps * ipad + i;
        const int e_lo = 1 + (j0 - B);
        bool dead = false;
        auto room = [&](int last){        // the slots up to step `last` are free once step last - GSR is done
            for(int n = 0; !dead && *prog < last - GSR; n++){ __nanosleep(100); if(n > LIMIT){ dead = true; *err = 1; } }
        };
        auto publish = [&](int s){
            __threadfence_block();
            __syncwarp();
            if(lane == 0) recv[wr] = s;
        };
        if(b == 0){                       // the row j = 0: never swept, read as it is, 8 steps at a time
            const double* P0 = P + gidx(g, i < g.im ? i : 0, 0, 0);
            for(int s = s_lo; s <= s_hi; s += 8){
                const int k0 = s - i - j0;
                double v[8];
#pragma unroll
                for(int u = 0; u < 8; u++) v[u] = (on && k0 + u >= 0 && k0 + u <= g.km - 2) ? P0[k0 + u] : 0.0;
                room(s + 7);
                if(i < ipad)
#pragma unroll
                    for(int u = 0; u < 8; u++) ringE[((s + u) & (GSR - 1)) * ipad + i] = v[u];
                publish(s + 7);
            }
            return;
        }
        for(int s = s_lo; s <= s_hi; s += 4){
            const int k0 = s - i - j0;
            double v[4];
            bool got[4];
#pragma unroll
            for(int u = 0; u < 4; u++){ v[u] = 0.0; got[u] = !(on && k0 + u >= 0 && k0 + u <= g.km - 2); }
            int done = 0;                 // steps of the four handed on, in order
            for(int n = 0; done < 4; n++){
#pragma unroll
                for(int u = 0; u < 4; u++)
                    if(!got[u]) got[u] = gs_edge_get(E + (size_t)(s + u - 1 - e_lo) * ipad, tag, v[u]) || dead;
                if(n == 0) room(s + 3);
                const int before = done;
#pragma unroll
                for(int u = 0; u < 4; u++){
                    const bool all = __all_sync(0xffffffffu, got[u]);
                    if(done == u && all){
                        if(i < ipad) ringE[((s + u) & (GSR - 1)) * ipad + i] = v[u];
                        done = u + 1;
                    }
                }
                if(done > before) publish(s + done - 1);
                if(n > LIMIT){ dead = true; *err = 1; }
                dead = __any_sync(0xffffffffu, dead);
            }
        }
        return;
    }

    if(t >= NC){
        // mover warps: four steps at a time, the rows that have passed k = 16 c + 1 .. 16 c + 4
        const int hw = (t - NC) / GSC, mw = (t - NC) >> 5, d = e >> 2;
        bool dead = false;
        for(int s = s_lo + 3; s <= s_hi; s += 4){
            for(int n = 0; !dead && *prog < s; n++){ __nanosleep(100); if(n > LIMIT){ dead = true; *err = 1; } }
            __threadfence_block();
            for(int q = hw; q < ngrp; q += GS_MOVERS / GSC){
                const int mb = q / gpr, i0 = (q - mb * gpr) * GSC;
                const int ir = i0 + ((s - 1 - j0 - mb - i0 - d) & (GSC - 1));
                const int c = (s - 1 - j0 - mb - ir) >> 4;
                if(ir < g.im && c >= 1){
                    if(j0 + mb <= j1 && ir >= 1 && ir <= g.im - 2) flush(mb, ir, (c - 1) * GSC + e4);
                    fetch(mb, ir, (c + 1) * GSC + e4);
                }
            }
            asm volatile("cp.async.commit_group;\n cp.async.wait_group 1;\n" ::: "memory");
            __threadfence_block();
            __syncwarp();
            if((t & 31) == 0) landed[mw] = s - 4;
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __threadfence_block();
        __syncwarp();
        if((t & 31) == 0) landed[mw] = INT_MAX;
        return;
    }

    // shared-memory addresses of the row's ring and its neighbours' (an idle thread reads along row 1
    // and writes nothing)
    const int r0 = act ? jb * ipad + i : 1;
    const unsigned aP = (unsigned)__cvta_generic_to_shared(ringP + r0 * GSR);
    const unsigned dJp = ipad * GSR * 8, dS = (unsigned)__cvta_generic_to_shared(ringS + r0 * GSR) - aP;
    const bool row0 = !act || jb == 0;                         // its poleward neighbour is the incoming edge, by step
    const unsigned aE = (unsigned)__cvta_generic_to_shared(ringE + (act ? i : 1));
    const bool lastrow = act && j == j1 && b + 1 < pl.nb;
    GsEdge* const Eo = edge + (size_t)b * pl.steps * ipad + (act ? i : 0);
    const double n1 = W.num1, n2 = W.num2, n3 = W.num3, inv = W.inv_denom;
    auto lds = [](unsigned p){ double v; asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(p)); return v; };
    // predicated stores: a branch around each would cost a step more than the store does
    auto sts_if = [](bool c, unsigned p, double v){
        asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q st.shared.f64 [%0], %1; }" :: "r"(p), "d"(v), "r"((unsigned)c));
    };
    auto edge_put_if = [tag](bool c, GsEdge* e, double v){
        const unsigned long long x = (unsigned long long)__double_as_longlong(v);
        asm volatile("{ .reg .pred q; setp.ne.u32 q, %5, 0; @q st.volatile.global.v4.u32 [%0], {%1, %2, %3, %4}; }"
                     :: "l"(e), "r"((unsigned)x), "r"(tag), "r"((unsigned)(x >> 32)), "r"(tag), "r"((unsigned)c) : "memory");
    };
    const unsigned a_prog = (unsigned)__cvta_generic_to_shared((void*)prog);
    auto prog_if = [a_prog](bool c, int v){
        asm volatile("{ .reg .pred q; setp.ne.u32 q, %2, 0; @q st.volatile.shared.u32 [%0], %1; }" :: "r"(a_prog), "r"(v), "r"((unsigned)c) : "memory");
    };
    // before the barrier that opens a step (and orders what follows): the row-0 threads wait for the step's incoming edge, warp 0
    // for the chunks the step reads first (the movers' chunks of 13 steps ago)
    int edge_in = act && jb == 0 ? s_lo - 1 : INT_MAX, chunk_in = t < 32 ? s_lo - 1 : INT_MAX - 13;
    int ready = min(edge_in, chunk_in + 13);                   // the steps this thread need not wait for
    auto wait_for = [&](int s){
        if(ready >= s) return;
        for(int n = 0; edge_in < s; n++){
            edge_in = recv[i >> 5];
            if(n > LIMIT){ edge_in = INT_MAX; *err = 1; }
        }
        for(int n = 0; chunk_in + 13 < s; n++){
            chunk_in = min(min(min(landed[0], landed[1]), min(landed[2], landed[3])), INT_MAX - 13);
            if(n > LIMIT){ chunk_in = INT_MAX - 13; *err = 1; }
        }
        ready = min(edge_in, chunk_in + 13);
    };
    wait_for(s_lo);
    // What a step reads that is not new -- the east, upper and poleward old values and the source --
    // is loaded during the step before it; after the barrier only the two new neighbours are left.
    const unsigned nk = act ? g.km - 1 : 0;                    // the row's cells
    const int klast = g.km - 2;
    int k = s_lo - i - j;
    constexpr unsigned MASK = (GSR - 1) * 8;
    unsigned a0 = aP + ((8u * (unsigned)k) & MASK), a1 = aP + ((8u * (unsigned)k + 8) & MASK);   // slots k, k + 1
    double ip = lds(a0 + GSR * 8), jp = lds(a0 + dJp), sr = lds(a0 + dS), ke = lds(a1);
    unsigned a_jm = row0 ? aE + (s_lo & (GSR - 1)) * ipad * 8 : a0 - dJp;
    for(int s = s_lo; s <= s_hi; s++){
        asm volatile("bar.sync 1, %0;\n" :: "n"(NC) : "memory");
        const double im_ = lds(a0 - GSR * 8), jm_ = lds(a_jm);
        const double kpart = ((k == klast ? new0 : ke) + kw) * n3;   // under the loads' latency
        const double v = ((ip + im_) * n1 + (jp + jm_) * n2 + kpart - sr) * inv;
        const bool in = (unsigned)k < nk;
        sts_if(in, a0, v);
        edge_put_if(in && lastrow, Eo + (unsigned)((s - s_lo) * ipad), v);
        prog_if(t == 0, s - 1);
        kw = k >= 0 ? v : kw;
        new0 = k == 0 ? v : new0;
        k++;
        a0 = a1;
        a1 = aP + ((8u * (unsigned)k + 8) & MASK);
        a_jm = row0 ? aE + ((s + 1) & (GSR - 1)) * ipad * 8 : a0 - dJp;
        ip = lds(a0 + GSR * 8); jp = lds(a0 + dJp); sr = lds(a0 + dS); ke = lds(a1);
        wait_for(s < s_hi ? s + 1 : s_hi);
    }
    asm volatile("bar.sync 1, %0;\n" :: "n"(NC) : "memory");
    if(t == 0) *prog = s_hi;
    // what is left in the rings: at most the last two chunks of each swept row
    for(int q = t / GSC; q < gpr * (j1 - j0 + 1); q += NC / GSC){
        const int mb = q / gpr, i0 = (q - mb * gpr) * GSC;
        for(int r = e >> 2; r < GSC; r += 4){
            const int ir = i0 + r;
            if(ir < 1 || ir > g.im - 2) continue;
            for(int c = max(0, ((g.km - 2) >> 4) - 1); c * GSC <= g.km - 2; c++) flush(mb, ir, c * GSC + e4);
        }
    }
}

// ---- the same sweep, one hyperplane s = i + j + k per launch: for columns too deep for gs_wave_kernel's
// shared memory ----
static __global__ void __launch_bounds__(256) gs_hyperplane_kernel(Grid g, double* P, const double* src, const GSW* w, int s){
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    const int nj = g.jm - 2;
    if(t >= (g.im - 2) * nj) return;
    const int i = 1 + t / nj, j = 1 + (t - (i - 1) * nj);
    const int k = s - i - j;
    if(k < 0 || k > g.km - 2) return;
    const GSW W = w[i * g.jm + j];
    const int kw = phi_wrap(k - 1, g.km), ke = phi_wrap(k + 1, g.km);
    P[gidx(g, i, j, k)] =
        ((P[gidx(g, i + 1, j, k)] + P[gidx(g, i - 1, j, k)]) * W.num1
       + (P[gidx(g, i, j + 1, k)] + P[gidx(g, i, j - 1, k)]) * W.num2
       + (P[gidx(g, i, j, ke)] + P[gidx(g, i, j, kw)]) * W.num3
       - src[gidx(g, i, j, k)]) * W.inv_denom;
}

// ---- p_dyn boundary passes, in the reference's order: radial planes over every (j,k), then
// the polar rows over every (i,k), then the seam copy (PressureSolverUran.h:213-244,
// PressureSolver.h:718-746) ----
static __global__ void pdyn_bc_r_kernel(Grid g, double* P){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if(k >= g.km) return;
    P[gidx(g, 0, j, k)]        = C43 * P[gidx(g, 1, j, k)] - C13 * P[gidx(g, 2, j, k)];
    P[gidx(g, g.im - 1, j, k)] = C43 * P[gidx(g, g.im - 2, j, k)] - C13 * P[gidx(g, g.im - 3, j, k)];
}
static __global__ void pdyn_bc_t_kernel(Grid g, double* P){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if(k >= g.km) return;
    P[gidx(g, i, 0, k)]        = C43 * P[gidx(g, i, 1, k)] - C13 * P[gidx(g, i, 2, k)];
    P[gidx(g, i, g.jm - 1, k)] = C43 * P[gidx(g, i, g.jm - 2, k)] - C13 * P[gidx(g, i, g.jm - 3, k)];
}
static __global__ void pdyn_bc_p_kernel(Grid g, double* P){
    chain_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if(c >= g.im * g.jm) return;
    const int i = c / g.jm, j = c - i * g.jm;
    P[gidx(g, i, j, g.km - 1)] = P[gidx(g, i, j, 0)];
}

// ---- Pressure_Uran.cpp:30-146, prepareProjectionBoundaries(rigid_lid), periodic phi.
// The radial and polar passes touch disjoint cells and read only interior ones, so they may
// run in one launch; the seam copy follows. ----
template <typename S>
__global__ void prep_rt_kernel(Grid g, S* au, S* av, S* aw, S* ru, S* rv, S* rw, int rigid_lid){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int y = blockIdx.y;                       // y < jm-2: radial pass row j = y+1, else polar pass level
    if(k > g.km - 2) return;
    S* A[6] = {au, av, aw, ru, rv, rw};
    auto cub = [&](S* X, size_t a3, size_t a2, size_t a1) -> S {
        return (S)((double)X[a3] - 3.0 * (double)X[a2] + 3.0 * (double)X[a1]);
    };
    if(y < g.jm - 2){
        const int j = y + 1;
        for(int q = 0; q < 6; q++){
            S* X = A[q];
            if(q == 0 && rigid_lid){
                X[gidx(g, 0, j, k)] = (S)0.0; X[gidx(g, g.im - 1, j, k)] = (S)0.0;
            } else {
                X[gidx(g, 0, j, k)] = cub(X, gidx(g, 3, j, k), gidx(g, 2, j, k), gidx(g, 1, j, k));
                X[gidx(g, g.im - 1, j, k)] = cub(X, gidx(g, g.im - 4, j, k), gidx(g, g.im - 3, j, k), gidx(g, g.im - 2, j, k));
            }
        }
    } else {
        const int i = y - (g.jm - 2) + 1;
        if(i > g.im - 2) return;
        for(int q = 0; q < 6; q += 3){              // aux_u / rhs_u: cubic; v, w: zero at the poles
            S* X = A[q];
            X[gidx(g, i, 0, k)] = cub(X, gidx(g, i, 3, k), gidx(g, i, 2, k), gidx(g, i, 1, k));
            X[gidx(g, i, g.jm - 1, k)] = cub(X, gidx(g, i, g.jm - 4, k), gidx(g, i, g.jm - 3, k), gidx(g, i, g.jm - 2, k));
            A[q + 1][gidx(g, i, 0, k)] = (S)0.0; A[q + 2][gidx(g, i, 0, k)] = (S)0.0;
            A[q + 1][gidx(g, i, g.jm - 1, k)] = (S)0.0; A[q + 2][gidx(g, i, g.jm - 1, k)] = (S)0.0;
        }
    }
}
template <typename S>
__global__ void prep_seam_kernel(Grid g, S* au, S* av, S* aw, S* ru, S* rv, S* rw){
    chain_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if(c >= g.im * g.jm) return;
    const int i = c / g.jm, j = c - i * g.jm;
    S* A[6] = {au, av, aw, ru, rv, rw};
    S v[6];
#pragma unroll
    for(int q = 0; q < 6; q++) v[q] = A[q][gidx(g, i, j, 0)];
#pragma unroll
    for(int q = 0; q < 6; q++) A[q][gidx(g, i, j, g.km - 1)] = v[q];
}

// ---- PressureSolver.h:370-487: div(aux) source, clamped, non-finite guard ----
template <typename S>
__global__ void rb_src_kernel(Grid g, const S* au, const S* av, const S* aw, const RBW* w,
                              PressConst c, double* src){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    const int i = 1 + blockIdx.z;
    if(k > g.km - 2 || j > g.jm - 2) return;
    const RBW W = w[i * g.jm + j];
    const int kw = phi_wrap(k - 1, g.km), ke = phi_wrap(k + 1, g.km);
    const double du_dr   = ((double)au[gidx(g, i + 1, j, k)] - (double)au[gidx(g, i - 1, j, k)]) * c.inv_2dr;
    const double dv_dthe = ((double)av[gidx(g, i, j + 1, k)] - (double)av[gidx(g, i, j - 1, k)]) * c.inv_2dthe;
    const double dw_dphi = ((double)aw[gidx(g, i, j, ke)] - (double)aw[gidx(g, i, j, kw)]) * c.inv_2dphi;
    double d = du_dr * 1.0 + dv_dthe * W.inv_rm + dw_dphi * W.inv_rmsinthe;
    if(!isfinite(d)) d = 0.0;
    else if(d >  W.src_max) d =  W.src_max;
    else if(d < -W.src_max) d = -W.src_max;
    src[gidx(g, i, j, k)] = d;
}

// ---- PressureSolver.h:320-495: one colour of the red-black relaxation. omega = 1 is the
// reference's update p = (acc - src) / den; other omega over-relax it (RB_SOR). ----
static __global__ void __launch_bounds__(256) rb_colour_kernel(Grid g, double* P, const double* src, const RBW* w,
                                                        int colour, double omega){
    chain_wait();
    const int half = g.km / 2;                       // km-1 even: each row holds half of each colour
    const int k2 = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    const int i = 1 + blockIdx.z;
    if(k2 >= half || j > g.jm - 2) return;
    const int k = 2 * k2 + ((i + j + colour) & 1);
    if(k > g.km - 2) return;
    const RBW W = w[i * g.jm + j];
    const int kw = phi_wrap(k - 1, g.km), ke = phi_wrap(k + 1, g.km);
    const size_t o = gidx(g, i, j, k);
    const double acc = (P[o + (size_t)g.jm * g.kp] + P[o - (size_t)g.jm * g.kp]) * W.num1
                     + (P[o + g.kp] + P[o - g.kp]) * W.num2
                     + (P[o - k + ke] + P[o - k + kw]) * W.num3;
    const double pn = (acc - src[o]) / W.den;
    P[o] = (omega == 1.0) ? pn : P[o] + omega * (pn - P[o]);
}

}  // namespace aturan
