// The moist convective adjustment (planet/ConvectiveAdjustment.h:402-849,
// MoistConvectiveAdjustment<cUranusModel>::run) with the reference's default knobs: Ledoux test
// with condensate loading, relaxation 1, no latitude smoothing (cUranusModel.h:572), at most 64
// sweeps, no phase split (SATADJ_BERGERON = 2), interior levels only (cUranusModel.h:566); the gas
// list H2O, NH3, H2S (its liquid set for both phases), CH4 and the NH4SH tracer of
// cUranusModel.cpp:1276-1290.
//
// Every (j, k) column is independent, and within a column the reference's sweep is a serial chain of
// equilibrium solves (Illinois regula falsi on the energy balance, FP64 whatever the storage: FP32
// storage in the mixed form is widened, T read as its FP32 pair). Four launches take out of that
// chain everything that is not part of it:
//   mca_prep_kernel    per cell: liquid-water static energy, total mixing ratios, weight;
//   mca_test_kernel    per pair (i, i+1): the upper cell's own equilibrium, the parcel's, the pair
//                      test: all of a sweep's tests at its start, one thread each;
//   mca_grow_kernel    per column with an unstable pair: the segments' growth, G lanes per column,
//                      32 / G columns per warp, a column taken from a counter when one is finished;
//   mca_finish_kernel  per mixed cell: its equilibrium at the final means, the write-back.
// What makes this the reference's sweep:
//   * A growth step reads only the equilibrium of the segment's lowest cell (the test below) and of
//     the cell above it (unmixed, so the one of the start), and two parcels: three solves on three
//     lanes at once. The other cells' equilibria are overwritten by the next step, so they are formed
//     once, at the end. A solve can fail only on a non-finite energy (with cp(T); without, on a
//     non-positive temperature, first at the top cell), which each step checks for the whole segment.
//   * A segment stops growing when both its edge pairs test stable, so the reference's re-test of its
//     upper edge is that same test again: the walk continues above it.
//   * After one sweep every pair is stable: pairs inside a segment hold equal values, so the parcel
//     and the upper cell's equilibrium are one solve and their difference is exactly zero; a segment's
//     edge pairs were tested with the values they still have; every other pair was stable at the start
//     and has not changed. The reference's further sweep finds nothing, so there is none here.
// Measured at 41x181x361 (mixed, synthetic state): 4.2 ms -- prep 0.10, tests 1.18, growth 2.48, finish
// 0.46 -- against 44.7 ms for one warp per column running the whole sweep with every settle and a
// verifying sweep; 1.1 against 8.1 ms at 37x83x167, 0.34 against 0.88 ms at 21x37x73. Same bits in FP64; the
// mixed form, whose multiply-adds contract, moved by 1e-15 of a field's maximum with the expressions. (With
// every quotient a division and a column's whole state in shared memory: 6.0, 1.28 and 0.63 ms.)
// The growth chain is what is left of the serial part: bound by the latency of its solves on small
// grids, by that and FP64 issue on large ones, so it takes as many warps an SM as 128 registers allow
// (16; the state in shared memory left room for 12). G = 4 keeps three of four lanes busy; few columns
// take more lanes each, the chain of a warp being that of its slowest column (21x37x73: 0.25 ms with
// G = 8, 0.30 with 4, 0.27 with 16, 0.45 with 32; 37x83x167: 0.61 with 4, 1.07 with 8).
// Every loop is bounded: 60 regula-falsi steps, 30 Newton steps of the enthalpy inverse, and a
// segment grows by at least one level per step within the column.
#pragma once
#include "common.cuh"

namespace aturan {

constexpr int MCA_NG = 4;
// Up to as many columns as the chip holds at once with 8 lanes each in the growth (16 warps an SM).
constexpr long MCA_SMALL_COLUMNS = 148 * 64;
constexpr double CP_T_LO_D = 5.0, CP_T_HI_D = 1500.0, CP_DT_D = 0.5;   // CpH2.h:13

struct McaGas { double ep, lv, ls, t_0, C, L0, R, del_alf, del_bet, C_i, L0_i, del_alf_i, del_bet_i;
                double rd, yrd, tv; };   // 1e-3 R and its reciprocal; 1 / ep - 1

struct McaConst {
    McaGas G[MCA_NG];                // H2O, NH3, H2S, CH4
    double L_tr, t_ref, grav, cp_mix, r_mix, cp_h2, r_h2, r_he, r_ch4, cp_he, cp_ch4;
    double k_h2, den, yden;          // r_h2 / r_mix; r_h2 + r_he + r_ch4 and its reciprocal
    float hz;                        // level spacing [km] as the model stores it (float)
    int cp_dyn, cp_mode, cp_gas, local_rho;
    const double *cp_tab, *H_tab;    // H2 cp table and its running integral (CpH2.h:66-75)
};

template <typename S>
struct McaArgs {
    Grid g;
    McaConst c;
    S* t;
    float* tlo;                      // the mixed form's temperature pair (common.cuh), else null
    S* sp[MCA_NG][3];                // vapour, cloud, ice
    S* nh4sh;
    const S *ps, *rho;
    // work fields in the padded layout: energy, NH4SH ratio, weight (0: the column is left alone), total
    // ratios, the upper cells' own equilibria (Teq = 0: the solve failed) and their condensates
    double *hL, *qr, *w, *qt[MCA_NG], *Teq, *ceq[MCA_NG];
    unsigned char* flag;             // per cell: 1 the pair (i, i+1) is unstable at the start; 2 the cell was mixed
    unsigned* next;                  // columns handed out to mca_grow_kernel's groups
};

__device__ __forceinline__ double mca_mx(double a, double b){ return (a < b) ? b : a; }   // std::max

// CpH2.h:88-101, 122-157
static __device__ double mca_cp_h2(const McaConst& A, double T){
    if(A.cp_mode <= 0) return A.cp_h2;
    const double Tc = T < CP_T_LO_D ? CP_T_LO_D : T;
    const double x = ((Tc > CP_T_HI_D ? CP_T_HI_D : Tc) - CP_T_LO_D) / CP_DT_D;
    int i = (int)x; if(i > CP_TABLE_N - 2) i = CP_TABLE_N - 2;
    if(i < 0) i = 0;                                 // a NaN's index (the value stays NaN through f)
    const double f = x - i;
    return A.cp_tab[i] + f * (A.cp_tab[i + 1] - A.cp_tab[i]);
}
static __device__ double mca_enth_h2(const McaConst& A, double T){
    if(A.cp_mode <= 0) return A.cp_h2 * T;
    const int n = CP_TABLE_N;
    if(T <= CP_T_LO_D) return A.cp_tab[0] * T;
    if(T >= CP_T_HI_D) return A.H_tab[n - 1] + A.cp_tab[n - 1] * (T - CP_T_HI_D);
    const double x = (T - CP_T_LO_D) / CP_DT_D;
    int i = (int)x; if(i > n - 2) i = n - 2;
    if(i < 0) i = 0;
    const double f = x - i;
    return A.H_tab[i] + CP_DT_D * f * (A.cp_tab[i] + 0.5 * f * (A.cp_tab[i + 1] - A.cp_tab[i]));
}
static __device__ double mca_cp(const McaConst& A, double T){
    if(!A.cp_dyn) return A.cp_mix;
    const double ch = mca_cp_h2(A, T);
    if(A.cp_gas) return div_by(A.r_h2 * ch + A.r_he * A.cp_he + A.r_ch4 * A.cp_ch4, A.den, A.yden);
    return A.cp_mix + A.k_h2 * (ch - A.cp_h2);
}
static __device__ double mca_enth(const McaConst& A, double T){
    if(!A.cp_dyn) return A.cp_mix * T;
    const double hh = mca_enth_h2(A, T);
    if(A.cp_gas) return div_by(A.r_h2 * hh + (A.r_he * A.cp_he + A.r_ch4 * A.cp_ch4) * T, A.den, A.yden);
    return (A.cp_mix - A.k_h2 * A.cp_h2) * T + A.k_h2 * hh;
}
static __device__ __noinline__ double mca_enth_inv(const McaConst& A, double h, double T0){
    if(!A.cp_dyn) return h / A.cp_mix;
    double T = (T0 > 0.0) ? T0 : h / A.cp_mix;
    for(int it = 0; it < 30; it++){
        const double f = mca_enth(A, T) - h, c = mca_cp(A, T);
        const double dT = f / c;
        T -= dT; if(T < 1.0) T = 1.0;
        if(fabs(dT) < 1.0e-10 * T) break;
    }
    return T;
}

// ATPhys.h:49-53 (the saturation pressure) and ConvectiveAdjustment.h:437-453 without the phase
// split; lg = log(T), yT = 1 / T, ypr = 1 / pr, the same for every gas at one T, formed once by the
// caller. Its three quotients a gas, and those by constants elsewhere, are products with reciprocals
// (div_by): the divisions' bits, and the four gases' chains run side by side instead of one after the
// other's branches. Where E leaves the normal range q is 0 or far below what qt holds.
__device__ __forceinline__ double mca_qsat(const McaGas& s, double T, double lg, double yT, double pr, double ypr){
    const bool liq = T >= s.t_0;                     // one expression for both sets: the lanes' phases differ
    const double C = liq ? s.C : s.C_i, L0 = liq ? s.L0 : s.L0_i;
    const double al = liq ? s.del_alf : s.del_alf_i, be = liq ? s.del_bet : s.del_bet_i;
    const double E = exp(C + div_by(div_by(-L0, T, yT) + al * lg + be * T, s.rd, s.yrd));
    const double q = div_by(s.ep * E, pr, ypr);
    return isfinite(q) ? q : 0.0;
}
__device__ __forceinline__ double mca_lat(const McaGas& s, double T){ return T >= s.t_0 ? s.lv : s.ls; }

// Level height as the model stores it (float).
__device__ __forceinline__ double mca_z(const McaConst& A, int i){ return (double)((float)i * A.hz) * 1.0e3; }
__device__ __forceinline__ double mca_rho(const McaConst& A, double r_){     // rho_at, cUranusModel.h:526-531
    if(!A.local_rho) return A.r_mix;
    return (r_ > 0.0 && isfinite(r_)) ? r_ : A.r_mix;
}

// :455-488, the equilibrium of (hL, qt) at (p, z): Illinois regula falsi on the energy balance. The
// balance is evaluated at one place in the code -- at the dry temperature T_lo (stage 0), the upper
// bracket (stage 1), then the regula-falsi points -- so that lanes at different stages run together,
// and the values at the returned T are kept rather than formed again.
static __device__ __forceinline__ bool mca_equil(const McaConst& A, double hL, const double (&qt)[MCA_NG], double pr, double z,
                                                 double& T, double (&cond)[MCA_NG]){
    const double cp = A.cp_mix, tol_T = 1.0e-10;
    const double T_lo = A.cp_dyn ? mca_enth_inv(A, hL - A.grav * z, 0.0) : (hL - A.grav * z) / cp;
    if(!(T_lo > 0.0) || !(pr > 0.0)) return false;
    double a = T_lo, b = T_lo, fa = 0.0, fb = 0.0, x = T_lo;
    int side = 0;
    const double ypr = 1.0 / pr;
    for(int n = -2; ; n++){                          // n = it of the reference's loop from 0 on
        const double e = mca_enth(A, x);
        const double lg = log(x), yT = 1.0 / x;
        double f = e + A.grav * z - hL;
        double d[MCA_NG];
        bool any = false;
#pragma unroll
        for(int g = 0; g < MCA_NG; g++){
            const double q = mca_qsat(A.G[g], x, lg, yT, pr, ypr);
            any |= qt[g] > q;
            d[g] = mca_mx(0.0, qt[g] - q);
            f -= mca_lat(A.G[g], x) * d[g];
        }
        bool keep = true;                            // x is the upper bracket: its condensates are the result's
        bool stop = false;
        if(n == -2){
            if(!any){ T = T_lo; for(int g = 0; g < MCA_NG; g++) cond[g] = 0.0; return true; }
            fa = f;
            double span = 0.0;
#pragma unroll
            for(int g = 0; g < MCA_NG; g++) span += mca_mx(A.G[g].lv, A.G[g].ls) * mca_mx(0.0, qt[g]);
            b = A.cp_dyn ? mca_enth_inv(A, e + span, T_lo) + 1.0e-9 : T_lo + span / cp + 1.0e-9;
            x = b;
            continue;
        }
        if(n == -1) fb = f;
        else {
            if(f < 0.0){ a = x; fa = f; if(side == -1) fb *= 0.5; side = -1; keep = false; }
            else       { b = x; fb = f; if(side == +1) fa *= 0.5; side = +1; }
            if(fabs(f) <= cp * tol_T){ a = b = x; keep = stop = true; }
        }
        if(keep){
#pragma unroll
            for(int g = 0; g < MCA_NG; g++) cond[g] = d[g];
        }
        if(stop || !(n + 1 < 60 && b - a > tol_T)) break;
        x = (fb - fa != 0.0) ? b - fb * (b - a) / (fb - fa) : 0.5 * (a + b);
        if(!(x > a && x < b)) x = 0.5 * (a + b);
    }
    T = b;
    return true;
}
__device__ __forceinline__ double mca_trE(const McaConst& A, double qr){ double e = 0.0; e += A.L_tr * qr; return e; }

// :613-624, Ledoux virtual temperature with condensate loading; NH4SH is a condensed tracer
static __device__ __forceinline__ double mca_tv(const McaConst& A, double TT, const double (&v_)[MCA_NG], const double (&cnd)[MCA_NG], double qr){
    double f = 1.0;
#pragma unroll
    for(int g = 0; g < MCA_NG; g++){ f += v_[g] * A.G[g].tv; f -= cnd[g]; }
    f -= qr;
    return TT * f;
}
// :627-644, the test of a pair: the parcel (the lower cell's qt_a, qr_a at the upper cell's level: Tp, pc)
// against the upper cell (qt_b, qr_b, its own equilibrium Tb, ec).
static __device__ __forceinline__ bool mca_decide(const McaConst& A, double Tp, const double (&pc)[MCA_NG], const double (&qta)[MCA_NG], double qra,
                                                  double Tb, const double (&ec)[MCA_NG], const double (&qtb)[MCA_NG], double qrb){
    const double tol_K = 1.0e-7;
    double pv[MCA_NG], ev[MCA_NG];
#pragma unroll
    for(int g = 0; g < MCA_NG; g++){ pv[g] = qta[g] - pc[g]; ev[g] = qtb[g] - ec[g]; }
    const double dTv = mca_tv(A, Tp, pv, pc, qra) - mca_tv(A, Tb, ev, ec, qrb);
    return dTv > tol_K;
}

// The arguments stay in the constant bank (__grid_constant__): the out-of-line enthalpy inverse takes the
// constants by reference, which otherwise copies the whole argument block to every thread's stack.
template <typename S>
__global__ void __launch_bounds__(128) mca_prep_kernel(const __grid_constant__ McaArgs<S> a){
    chain_wait();
    const Grid& g = a.g;
    const McaConst& A = a.c;
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = blockIdx.z;
    if(k >= g.km) return;
    const size_t o = gidx(g, i, j, k);
    const int i0 = 1, i1 = g.im - 2;
    a.flag[o] = 0;
    if(i < i0 || i > i1) return;
    const double T = t_ld(a.t, a.tlo, o) * A.t_ref, p = (double)a.ps[o];
    const double rho = mca_rho(A, A.local_rho ? (double)a.rho[o] : 0.0), z = mca_z(A, i);
    bool ok = (T > 0.0) && (p > 0.0) && (rho > 0.0) && isfinite(T + p + rho);
    const double lo = (i > i0) ? 0.5 * (mca_z(A, i - 1) + z) : mca_z(A, i0);
    const double hi = (i < i1) ? 0.5 * (z + mca_z(A, i + 1)) : mca_z(A, i1);
    const double w = rho * (hi - lo);
    if(!(w > 0.0)) ok = false;
    if(!ok){ a.w[o] = 0.0; return; }                 // its column is left alone: nothing else is read
    double h = mca_enth(A, T) + A.grav * z;
    // every load before the first store, which the compiler must assume to alias them
    double x[MCA_NG][3];
#pragma unroll
    for(int q = 0; q < MCA_NG; q++)
#pragma unroll
        for(int n = 0; n < 3; n++) x[q][n] = (double)a.sp[q][n][o];
    const double qr = (double)a.nh4sh[o] / rho;
#pragma unroll
    for(int q = 0; q < MCA_NG; q++){
        const double qv = mca_mx(0.0, x[q][0]) / rho;
        const double qc = mca_mx(0.0, x[q][1]) / rho;
        const double qi = mca_mx(0.0, x[q][2]) / rho;
        a.qt[q][o] = qv + qc + qi;
        h -= A.G[q].lv * qc + A.G[q].ls * qi;
    }
    h -= A.L_tr * qr;
    a.qr[o] = qr;
    a.hL[o] = h;
    a.w[o] = w;
}

// Thread (i, j, k): cell i + 1's own equilibrium and the test of the pair (i, i + 1), i = 1 .. im-3.
template <typename S>
__global__ void __launch_bounds__(128, 4) mca_test_kernel(const __grid_constant__ McaArgs<S> a){
    chain_wait();
    const Grid& g = a.g;
    const McaConst& A = a.c;
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = 1 + blockIdx.z;
    if(k >= g.km) return;
    const size_t o = gidx(g, i, j, k), ob = o + (size_t)g.jm * g.kp;
    if(!(a.w[o] > 0.0) || !(a.w[ob] > 0.0)) return;  // a column that is left alone
    double qa[MCA_NG], qb[MCA_NG];
#pragma unroll
    for(int q = 0; q < MCA_NG; q++){ qa[q] = a.qt[q][o]; qb[q] = a.qt[q][ob]; }
    const double qra = a.qr[o], qrb = a.qr[ob];
    const double ha = a.hL[o] + mca_trE(A, qra), hb = a.hL[ob] + mca_trE(A, qrb);
    const double pr = (double)a.ps[ob], z = mca_z(A, i + 1);
    double Tp = 0.0, pc[MCA_NG] = {0.0, 0.0, 0.0, 0.0}, Tb = 0.0, ec[MCA_NG] = {0.0, 0.0, 0.0, 0.0};
    bool okp = false, okb = false;
#pragma unroll 1
    for(int s = 0; s < 2; s++){                      // the upper cell, then the parcel: one call site
        double x[MCA_NG], T = 0.0, c[MCA_NG] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
        for(int q = 0; q < MCA_NG; q++) x[q] = s ? qa[q] : qb[q];
        const bool ok = mca_equil(A, s ? ha : hb, x, pr, z, T, c);
        if(s){ okp = ok; Tp = T; } else { okb = ok; Tb = T; }
#pragma unroll
        for(int q = 0; q < MCA_NG; q++){ if(s) pc[q] = c[q]; else ec[q] = c[q]; }
    }
    a.Teq[ob] = okb ? Tb : 0.0;
#pragma unroll
    for(int q = 0; q < MCA_NG; q++) a.ceq[q][ob] = ec[q];
    a.flag[o] = okp && okb && mca_decide(A, Tp, pc, qa, qra, Tb, ec, qb, qrb) ? 1 : 0;
}

// What a group keeps of its column in shared memory, and its bytes: the weights and a flag per level.
struct McaCol { double* w; unsigned char* flag; };
__host__ __device__ constexpr size_t mca_col_bytes(int im){ return (size_t)im * sizeof(double) + ((size_t)im + 7) / 8 * 8; }

// Blocks of one warp, G (4 to 16) lanes per column. A group walks up its column from unstable pair to unstable
// pair; every turn of the loop is one growth step of each group's segment, its three solves on three
// lanes through one call site. The cells of a growing segment all hold its means, which stay in
// registers until it has stopped growing and go to the work fields then; of the other cells a step
// reads only those next to the segment, from the work fields. So shared memory holds no more than the
// weights (the column's whole state there left room for 12 warps an SM, and the solves are latency).
template <typename S, int G>
__global__ void __launch_bounds__(32, 16) mca_grow_kernel(const __grid_constant__ McaArgs<S> a){
    chain_wait();
    extern __shared__ __align__(16) char mca_smem[];
    const Grid& g = a.g;
    const McaConst& A = a.c;
    const int lane = threadIdx.x, gl = lane % G, grp = lane / G;
    const unsigned gm = ((1u << G) - 1u) << (grp * G);
    const int im = g.im, i0 = 1, i1 = im - 2;
    const unsigned ncol = (unsigned)(g.jm * g.km);
    const size_t pl = (size_t)g.jm * g.kp;
    McaCol C;
    C.w = reinterpret_cast<double*>(mca_smem + grp * mca_col_bytes(im));
    C.flag = reinterpret_cast<unsigned char*>(C.w + im);
    // the sums a lane forms: lane 0 w and w hL; lanes 1, 2 two of w qt; lane 3 w qr
    const double* const x0 = gl == 0 ? a.hL : gl == 1 ? a.qt[0] : gl == 2 ? a.qt[2] : a.qr;
    const double* const x1 = gl == 1 ? a.qt[1] : gl == 2 ? a.qt[3] : x0;
    bool active = false, done = false, have = false;     // a segment is growing; no column left; a column is loaded
    int i = i0, lo = 0, hi = 0;
    int ml = 0, mh = -1;                                 // the cells that hold the means s0, s1 of the last step
    double s0 = 0.0, s1 = 0.0;
    size_t o0 = 0;
    while(true){
        // a group without a segment: the next unstable pair of its column, or of the next column
        while(!active && !done){
            if(!have){
                unsigned c = 0;
                if(gl == 0) c = atomicAdd(a.next, 1u);
                c = __shfl_sync(gm, c, 0, G);
                if(c >= ncol){ done = true; break; }
                const int j = (int)(c / (unsigned)g.km), k = (int)(c - (unsigned)j * g.km);
                o0 = gidx(g, 0, j, k);
                int un = 0, ok = 1;
                for(int q = i0 + gl; q <= i1; q += G){
                    const size_t o = o0 + (size_t)q * pl;
                    const unsigned char f = a.flag[o];
                    const double w = a.w[o];
                    C.flag[q] = f; C.w[q] = w;
                    un |= f;
                    if(!(w > 0.0)) ok = 0;
                }
                un = __any_sync(gm, un);
                ok = __all_sync(gm, ok);
                if(!un) continue;
                if(!ok){                                  // the column keeps its state
                    for(int q = i0 + gl; q <= i1; q += G) a.flag[o0 + (size_t)q * pl] = 0;
                    continue;
                }
                __syncwarp(gm);
                have = true;
                i = i0;
            }
            // the first pair at or above i that was unstable at the start
            while(i < i1){
                const bool u = i + gl < i1 && C.flag[i + gl] == 1;
                const unsigned m = __ballot_sync(gm, u) & gm;
                if(m){ i += __ffs(m >> (grp * G)) - 1; break; }
                i += G;
            }
            if(i < i1){ active = true; lo = i; hi = i + 1; ml = hi; mh = lo; break; }
            // the column is finished: its flags back
            for(int q = i0 + gl; q <= i1; q += G) a.flag[o0 + (size_t)q * pl] = C.flag[q] == 2 ? 2 : 0;
            __syncwarp(gm);
            have = false;
        }
        if(__all_sync(0xffffffffu, done)) return;
        bool task = false, below = false, above = false;
        int lb = lo;
        double m_h = 0.0, m_r = 0.0, m_q[MCA_NG] = {0.0, 0.0, 0.0, 0.0};
        double h = 0.0, qr = 0.0, x[MCA_NG];             // the cell this lane solves for
        if(active){
            // the segment's mass-weighted means, each sum by one lane in the reference's order: the cell it
            // grew to below, the cells that hold the last means, the cell it grew to above
            if(gl < 4){
                const size_t ol = o0 + (size_t)lo * pl, oh = o0 + (size_t)hi * pl;
                const double b0 = lo < ml ? x0[ol] : 0.0, b1 = lo < ml ? x1[ol] : 0.0;
                const double e0 = hi > mh ? x0[oh] : 0.0, e1 = hi > mh ? x1[oh] : 0.0;
                double sw = 0.0, t0 = 0.0, t1 = 0.0;
                for(int q = lo; q <= hi; q++){
                    const double w = C.w[q];
                    const double v0 = q < ml ? b0 : q > mh ? e0 : s0, v1 = q < ml ? b1 : q > mh ? e1 : s1;
                    sw += w;
                    t0 += w * v0;
                    t1 += w * v1;
                }
                s0 = t0 / sw;
                s1 = t1 / sw;
            }
            ml = lo; mh = hi;
            m_h = __shfl_sync(gm, s0, 0, G); m_r = __shfl_sync(gm, s0, 3, G);
            m_q[0] = __shfl_sync(gm, s0, 1, G); m_q[1] = __shfl_sync(gm, s1, 1, G);
            m_q[2] = __shfl_sync(gm, s0, 2, G); m_q[3] = __shfl_sync(gm, s1, 2, G);
            // a settle of one of its cells would fail (mca_equil): the column keeps its state
            const double h_top = m_h + mca_trE(A, m_r) - A.grav * mca_z(A, hi);
            if(A.cp_dyn ? !isfinite(h_top) : !(h_top / A.cp_mix > 0.0)){
                for(int q = i0 + gl; q <= i1; q += G) a.flag[o0 + (size_t)q * pl] = 0;
                __syncwarp(gm);
                active = have = false;
            } else {
                below = lo > i0; above = hi < i1;
                h = m_h; qr = m_r;
#pragma unroll
                for(int s = 0; s < MCA_NG; s++) x[s] = m_q[s];
                if(gl == 0){ task = below; }                                       // cell lo's own equilibrium
                else if(gl == 1){                                                  // cell lo - 1 lifted to lo
                    task = below;
                    if(below){
                        const size_t oa = o0 + (size_t)(lo - 1) * pl;
                        h = a.hL[oa]; qr = a.qr[oa];
#pragma unroll
                        for(int s = 0; s < MCA_NG; s++) x[s] = a.qt[s][oa];
                    }
                }
                else if(gl == 2){ task = above; lb = hi + 1; }                     // the mixed cell hi lifted to hi + 1
            }
        }
        __syncwarp();
        double T = 0.0, c[MCA_NG] = {0.0, 0.0, 0.0, 0.0};
        bool ok = false;
        if(task) ok = mca_equil(A, h + mca_trE(A, qr), x, (double)a.ps[o0 + (size_t)lb * pl], mca_z(A, lb), T, c);
        __syncwarp();
        if(!active) continue;
        // lane 0 tests the pair (lo - 1, lo) with lane 1's parcel and its own equilibrium, lane 2 the pair
        // (hi, hi + 1) with its parcel and cell hi + 1's equilibrium of the start
        double Tp = __shfl_sync(gm, T, 1, G), pc[MCA_NG], qa[MCA_NG], qb[MCA_NG];
#pragma unroll
        for(int s = 0; s < MCA_NG; s++){ pc[s] = __shfl_sync(gm, c[s], 1, G); qa[s] = __shfl_sync(gm, x[s], 1, G); }
        double ra = __shfl_sync(gm, qr, 1, G), rb = m_r;
        bool okp = __shfl_sync(gm, (int)ok, 1, G) != 0;
        bool grow = false;
        if((gl == 0 && below) || (gl == 2 && above)){
            double Tb = T, ec[MCA_NG];
            bool okb = ok;
#pragma unroll
            for(int s = 0; s < MCA_NG; s++){ ec[s] = c[s]; qb[s] = m_q[s]; }
            if(gl == 2){
                const size_t ob = o0 + (size_t)(hi + 1) * pl;
                Tp = T; okp = ok;
                Tb = a.Teq[ob]; okb = Tb > 0.0;
                ra = m_r; rb = a.qr[ob];
#pragma unroll
                for(int s = 0; s < MCA_NG; s++){ pc[s] = c[s]; ec[s] = a.ceq[s][ob]; qa[s] = m_q[s]; qb[s] = a.qt[s][ob]; }
            }
            grow = okp && okb && mca_decide(A, Tp, pc, qa, ra, Tb, ec, qb, rb);
        }
        const unsigned gr = __ballot_sync(gm, grow) >> (grp * G);
        if(gr & 1u) lo--;
        if(gr & 4u) hi++;
        if(!(gr & 5u)){
            // the segment has stopped growing: its cells hold the means
            for(int q = lo + gl; q <= hi; q += G){
                const size_t o = o0 + (size_t)q * pl;
                C.flag[q] = 2;
                a.hL[o] = m_h; a.qr[o] = m_r;
#pragma unroll
                for(int s = 0; s < MCA_NG; s++) a.qt[s][o] = m_q[s];
            }
            active = false; i = hi + 1;
        }
        __syncwarp(gm);
    }
}

// Per mixed cell: its equilibrium at the final means and the write-back (:645-661, :800-849).
template <typename S>
__global__ void __launch_bounds__(128) mca_finish_kernel(const __grid_constant__ McaArgs<S> a){
    chain_wait();
    const Grid& g = a.g;
    const McaConst& A = a.c;
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, i = 1 + blockIdx.z;
    if(k >= g.km) return;
    const size_t o = gidx(g, i, j, k);
    if(a.flag[o] != 2) return;
    double qt[MCA_NG], ce[MCA_NG], T = 0.0;
#pragma unroll
    for(int s = 0; s < MCA_NG; s++) qt[s] = a.qt[s][o];
    const double qr = a.qr[o];
    if(!mca_equil(A, a.hL[o] + mca_trE(A, qr), qt, (double)a.ps[o], mca_z(A, i), T, ce)) return;
    const double rho = mca_rho(A, A.local_rho ? (double)a.rho[o] : 0.0);
    t_st(a.t, a.tlo, o, T / A.t_ref);
#pragma unroll
    for(int s = 0; s < MCA_NG; s++){
        const double qv = qt[s] - ce[s];
        const bool liq = T >= A.G[s].t_0;
        a.sp[s][0][o] = (S)(qv * rho);
        a.sp[s][1][o] = (S)((liq ? ce[s] : 0.0) * rho);
        a.sp[s][2][o] = (S)((liq ? 0.0 : ce[s]) * rho);
    }
    a.nh4sh[o] = (S)(qr * rho);
}

// CpH2.h:66-75: the running integral of the cp table, in the table's order (one thread).
static __global__ void mca_H_kernel(const double* cp, double* H){
    if(threadIdx.x != 0 || blockIdx.x != 0) return;
    H[0] = cp[0] * CP_T_LO_D;
    for(int i = 1; i < CP_TABLE_N; i++) H[i] = H[i - 1] + 0.5 * CP_DT_D * (cp[i] + cp[i - 1]);
}

}  // namespace aturan
