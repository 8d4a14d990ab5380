// Hand-written adjoint of one RK4 step of the dry dynamics (t, u, v, w), FP64.
//
// Forward (rk4.cuh, RungeKutta_Uran_Turb.cpp:18-403): level means ref(T), p_hydro = H(T, v, w, ref),
// then four stages k_s = RHS(X_s, p_hydro) with X_0 = y, X_{s+1} = y + c_s k_s on the interior
// (boundary rows of every X_s are y's), and y' = y + dt/6 sum_s w_s k_s, T' clamped. The inputs y
// are the state and its start-of-step copies together; p_dyn, p_stat, the forcing and every
// other field are held fixed (the tendencies of t, u, v, w do not read the scalars).
//
// Reverse: with g = ybar' masked by the clamp, ybar = g, kbar_3 = dt/6 w_3 g, and for s = 3..0
//   Xbar_s = J_s^T kbar_s (+ p_hydro part), ybar += Xbar_s, kbar_{s-1} = dt/6 w_{s-1} g + c_{s-1} Xbar_s,
// then the hydrostatic integral's and the level means' adjoints add into ybar (T, v, w).
//
// J_s^T is a scatter of every interior cell's local partial derivatives onto its 7-point stencil. It
// runs as gather, without atomics and in a fixed order: what a cell sends along one direction is a
// product of its tendency adjoints and of values at the cell alone (its wind, viscosity and metric),
// so adj_stage_kernel re-forms, for each cell, what its six neighbours send it; only the centre's own
// part needs the stage input's differences. One launch per stage, no intermediate fields. Written out
// as contributions per stencil point (38 fields dry, 122 moist, written by one launch and read by the
// next) the same sums took 3.3x the memory traffic.
// The partial derivatives are those of the forward's formulas (RHS_Uran_Turb.cpp:92-788), derived
// term by term; cp(T) is the piecewise-linear table, differentiated within its interval (a kink
// convention: the derivative of the interval the value falls in).
#pragma once
#include "common.cuh"
#include "rk4.cuh"
#include "satadj.cuh"

namespace aturan {

constexpr int ADJ_NF = 4;                          // t, u, v, w (state fields 0..3)
// The moist form: the twelve condensable species (state fields 4..15, ATURAN_CH4 .. ATURAN_NH3_ICE)
// join the dry four.
constexpr int ADJ_NF_MOIST = 16;

struct AdjArgs {
    Grid g;
    const double* X;            // stage input, field q at X + q * fstride
    const double* X0;           // the step's input (boundary rows of every stage input)
    const double* Xprev;        // the previous stage's input, or null at stage 0
    const double* kbar;         // adjoint of the stage's tendencies, field q at kbar + q * fstride (0 off the interior)
    const double* pe;           // ce_sp cp_mix / cp(T) kbar_t: the p_dyn gradients' factor (0 off the interior)
    double* kbar_out;           // the previous stage's kbar and pe
    double* pe_out;
    const double* auxbar;       // stage 3 only, else null: adjoint of aux_u, aux_v, aux_w (the tendencies
                                // of u, v, w without the p_dyn gradient, RHS_Uran_Turb.cpp:1020-1022), used on
                                // the interior alone
    const double* pdyn;
    const double* nt;           // the eddy viscosity as the tendencies use it (adj_nue)
    const GeoIJ<double>* geo;
    const double* cp_tab;
    RhsConst<double> k;
    const double* g0;
    double *ybar, *phbar, *pdbar;
    double w_prev, c_prev;      // kbar_{s-1} = w_prev g0 + c_prev Xbar_s
    double* hacc;               // null, or the T tendencies' adjoint summed over the stages (heating)
};

// cp_lapse (rk4.cuh) and its derivative in T (K), the table's slope inside its 0.5 K interval.
__device__ __forceinline__ void cp_lapse_d(const RhsConst<double>& k, const double* tab, double T,
                                           double* cp, double* dcp){
    double ch, dch;
    if(k.cp_mode <= 0){ ch = k.cp_h2_const; dch = 0.0; }
    else {
        const double Tc = T < 5.0 ? 5.0 : T;
        const double x = ((Tc > 1500.0 ? 1500.0 : Tc) - 5.0) / 0.5;
        int i = (int)x; if(i > CP_TABLE_N - 2) i = CP_TABLE_N - 2;
        const double f = x - (double)i;
        const double a = __ldg(tab + i), b = __ldg(tab + i + 1);
        ch = a + f * (b - a);
        dch = (T > 5.0 && T < 1500.0) ? (b - a) / 0.5 : 0.0;
    }
    if(k.cp_gas){ *cp = (k.cp_rh2 * ch + k.cp_he_term + k.cp_ch4_term) / k.cp_rsum; *dcp = k.cp_rh2 * dch / k.cp_rsum; }
    else        { *cp = k.cp_mix + k.cp_rh2 * (ch - k.cp_h2_const);               *dcp = k.cp_rh2 * dch; }
}

// cp(T) factor of the pressure work at T (nondimensional): cp_mix / cp(T), 1 without it.
__device__ __forceinline__ double adj_cpf(const RhsConst<double>& K, const double* tab, double t){
    if(!(K.cp_dyn && t > 0.0)) return 1.0;
    double cp, dcp;
    cp_lapse_d(K, tab, t * K.t_ref, &cp, &dcp);
    return K.cp_mix / cp;
}
// The eddy viscosity the tendencies use, from the stored one.
__device__ __forceinline__ double adj_nue(const RhsConst<double>& K, double nue_c){
    return (K.turb_coupling != 0.0 && isfinite(nue_c)) ? K.turb_coupling * cmax(0.0, nue_c) : 0.0;
}
// The weights of one (i, j) row with which its cells send along r, theta and phi: of the transport (r1, t1,
// p1, times the wind), of the first-order (t2; r2, for u twice) and second-order (t3, p3, inv_dr2) parts of
// the diffusion, and of the metric cross terms (t4; p4, p5).
struct AdjRow { double r2, t1, t2, t3, t4, p1, p3, p4, p5; };

// One reverse stage of the NF fields (RHS_Uran_Turb.cpp:92-850): per cell (every row, every distinct
// meridian; the seam copy k = km-1 is read by no stencil and receives nothing) the sum of what the cells
// whose stencils contain it send; added into ybar, phbar and pdbar; and the previous stage's kbar and pe on
// the interior. A neighbour off the interior sends nothing: the cell (0, 0, 0), where every kbar and pe is 0,
// is read in its place, so that every load is unconditional and issued before the first use (branches made
// each neighbour's loads wait for the one before; one around the species' sums, 40 us a moist stage). What
// else is read there counts as 0 by a select, not by a zero weight: it may be a NaN (the boundary rows of a
// stage input are never written, those of the aux adjoint are the caller's). A cell sends its tendency
// adjoint times
//   transport: -wind * (r1, t1 or p1);  diffusion: D * (first- and second-order weights of its row),
// the same weight for every field but its D (and u's own radial term), so a neighbour costs one weight per
// D and one multiply-add per field. The rows' weights are formed once per block in shared memory.
// Bound by the latency of its ~85 loads per cell at the registers they hold, then by their L2 traffic: it
// reads the stage input, kbar, g0, nue, p_dyn and pe, and updates ybar, phbar and pdbar, ~33 words per cell
// dry and ~105 moist. Whatever a cell adds to is loaded before its first store: a load behind a store
// waits for it, and ten of them in a row cost more than the sums. At 41x91x181: 77 us a stage dry and 180
// moist at 4 and 2 resident blocks (128 and 255 registers; 79 at 3 and 87 at 5 blocks dry, 203 at 3 moist),
// against 108 and 374 as the two or three launches that wrote and gathered the contributions, and 103 and
// 254 with those loads between the stores.
template <int NF>
__global__ void __launch_bounds__(128, NF == ADJ_NF ? 4 : 2) adj_stage_kernel(const __grid_constant__ AdjArgs a){
    chain_wait();
    const Grid& g = a.g;
    const RhsConst<double>& K = a.k;
    __shared__ AdjRow rows[14];          // of this block's four j: (i, j0 - 1 .. j0 + 4), then (i - 1, j), then (i + 1, j)
    const int tj = threadIdx.y, j0 = blockIdx.y * 4, i = blockIdx.z;
    {
        const int r = tj * 32 + threadIdx.x;
        if(r < 14){
            const int ri = r < 6 ? i : (r < 10 ? i - 1 : i + 1), rj = r < 6 ? j0 - 1 + r : j0 + (r - 6) % 4;
            const GeoIJ<double>& G = a.geo[min(max(ri, 0), g.im - 1) * g.jm + min(max(rj, 0), g.jm - 1)];
            AdjRow w;
            w.r2 = G.two_inv_rm * K.inv_2dr;
            w.t1 = G.inv_rm * K.inv_2dthe; w.t2 = G.costhe_inv_rm2sinthe * K.inv_2dthe;
            w.t3 = G.inv_rm2 * K.inv_dthe2; w.t4 = 2.0 * G.inv_rm2 * K.inv_2dthe;
            w.p1 = G.inv_rmsinthe * K.inv_2dphi; w.p3 = G.inv_rm2sinthe2 * K.inv_dphi2;
            w.p4 = 2.0 * G.inv_rm2sinthe * K.inv_2dphi; w.p5 = 2.0 * G.costhe * G.inv_rm2sinthe2 * K.inv_2dphi;
            // no cell of a row off the interior sends anything, and a pole's metric may be infinite
            if(ri < 1 || ri > g.im - 2 || rj < 1 || rj > g.jm - 2) w = AdjRow{};
            rows[r] = w;
        }
        __syncthreads();
    }
    const int k = blockIdx.x * 32 + threadIdx.x;
    const int j = j0 + tj;
    if(k > g.km - 2 || j > g.jm - 1) return;
    // 32-bit offsets: a field has < 2^31 values and the tape's groups are reached field by field
    const int fs = (int)g.fstride, si = g.jm * g.kp, sj = g.kp;
    const int o = (int)gidx(g, i, j, k);
    const bool ini = i >= 1 && i <= g.im - 2, inj = j >= 1 && j <= g.jm - 2;
    const bool in = ini && inj;
    const bool nb[6] = {inj && i >= 2, inj && i <= g.im - 3, ini && j >= 2, ini && j <= g.jm - 3, in, in};
    const int on[6] = {nb[0] ? o - si : 0, nb[1] ? o + si : 0, nb[2] ? o - sj : 0, nb[3] ? o + sj : 0,
                       in ? o - k + phi_wrap(k - 1, g.km) : 0, in ? o - k + phi_wrap(k + 1, g.km) : 0};
    // the stencil's own places (boundary rows from the step's input)
    const int oc[4] = {in ? o - si : o, in ? o + si : o, in ? o - sj : o, in ? o + sj : o};
    const double* const kb[ADJ_NF] = {a.kbar, a.kbar + (size_t)fs, a.kbar + 2 * (size_t)fs, a.kbar + 3 * (size_t)fs};
    const double* const xsrc[4] = {i == 1 ? a.X0 : a.X, i == g.im - 2 ? a.X0 : a.X, j == 1 ? a.X0 : a.X, j == g.jm - 2 ? a.X0 : a.X};
    double at[7], au[7], av[7], aw[7], a0[6], wn[6], pe[6], nt[7];
#pragma unroll
    for(int d = 0; d < 7; d++){
        const int q = d < 6 ? on[d] : o;
        at[d] = ldr(kb[0] + q); au[d] = ldr(kb[1] + q); av[d] = ldr(kb[2] + q); aw[d] = ldr(kb[3] + q);
        nt[d] = ldr(a.nt + q);
        if(d < 6){
            const double wx = ldr(a.X + (size_t)(1 + d / 2) * fs + q);
            wn[d] = nb[d] ? wx : 0.0;
            pe[d] = ldr(a.pe + q);
            a0[d] = d < 2 ? au[d] : (d < 4 ? av[d] : aw[d]);
        }
    }
    auto stencil = [&](int q) -> R7<double> {
        const size_t f = (size_t)q * fs;
        R7<double> r;
        r.c  = ldr(a.X + f + o);
        r.rm = ldr(xsrc[0] + f + oc[0]); r.rp = ldr(xsrc[1] + f + oc[1]);
        r.tm = ldr(xsrc[2] + f + oc[2]); r.tp = ldr(xsrc[3] + f + oc[3]);
        r.pw = ldr(a.X + f + on[4]);     r.pe = ldr(a.X + f + on[5]);
        return r;
    };
    const R7<double> rT = stencil(0), rU = stencil(1), rV = stencil(2), rW = stencil(3);
    const double* P = a.pdyn;
    const double p_im = ldr(P + oc[0]), p_ip = ldr(P + oc[1]), p_jm = ldr(P + oc[2]), p_jp = ldr(P + oc[3]);
    const double p_kw = ldr(P + on[4]), p_ke = ldr(P + on[5]);
    if(a.auxbar){                                       // the aux adjoint joins every partial but those in p_dyn
#pragma unroll
        for(int d = 0; d < 7; d++){
            const int q = d < 6 ? on[d] : o;
            const double bu = ldr(a.auxbar + q), bv = ldr(a.auxbar + (size_t)fs + q), bw = ldr(a.auxbar + 2 * (size_t)fs + q);
            const bool use = d < 6 ? nb[d] : in;
            au[d] += use ? bu : 0.0; av[d] += use ? bv : 0.0; aw[d] += use ? bw : 0.0;
        }
    }
    const double ire = K.inv_re_eff, irp = K.inv_re_pr, i09 = 1.0 / 0.9;
    double xt = 0.0, xu = 0.0, xv = 0.0, xw = 0.0, h = 0.0, pd = 0.0;
    double lap = 0.0, inv_rm = 0.0, inv_rs = 0.0;
    if(in){                                             // the centre's own part
        const GeoIJ<double>& geo = a.geo[i * g.jm + j];
        const AdjRow& R = rows[1 + tj];
        const D6<double> T = diff6(K, rT), U = diff6(K, rU), V = diff6(K, rV), W = diff6(K, rW);
        const double u = U.c, v = V.c, w = W.c, t0 = T.c;
        inv_rm = geo.inv_rm; inv_rs = geo.inv_rmsinthe;
        const double dpdr = (p_ip - p_im) * K.inv_2dr, dpdthe = (p_jp - p_jm) * K.inv_2dthe * inv_rm, dpdphi = (p_ke - p_kw) * K.inv_2dphi * inv_rs;
        const double costhe = geo.costhe, cot = geo.cotanthe, c_t = at[6], c_u = au[6], c_v = av[6], c_w = aw[6];
        const double D = ire + nt[6], Dt = irp + nt[6] * i09, vm = geo.v_metric * D;
        if(a.hacc) a.hacc[o] += c_t;                    // rhs_t += heat_scale H(j,k) (aturan_set_heating)
        // pressure work and its cp(T) factor
        double cpf = 1.0, dcpf = 0.0;
        if(K.cp_dyn && t0 > 0.0){
            double cp, dcp;
            cp_lapse_d(K, a.cp_tab, t0 * K.t_ref, &cp, &dcp);
            cpf = K.cp_mix / cp;
            dcpf = -cpf / cp * dcp * K.t_ref;
        }
        const double P0 = K.ce_sp * (u * dpdr + v * dpdthe + w * dpdphi), cec = K.ce_sp * cpf;
        const double ut = inv_rm * U.d1t, vt = inv_rm * V.d1t, wt = inv_rm * W.d1t, tt = inv_rm * T.d1t;
        const double up = inv_rs * U.d1p, vp = inv_rs * V.d1p, wp = inv_rs * W.d1p, tp = inv_rs * T.d1p;
        lap = 2.0 * (K.inv_dr2 + R.t3 + R.p3);
        xu = c_u * (-U.d1r + D * (2.0 * geo.inv_rm2 - lap) - geo.sponge)
           + c_v * (-V.d1r - v * inv_rm)
           + c_w * (-W.d1r - w * inv_rm - K.cor_sc * K.p2om * geo.sinthe_bf)
           + c_t * (cec * dpdr - T.d1r);
        xv = c_u * -ut
           + c_v * (-vt - u * inv_rm - vm - D * lap)
           + c_w * (-wt - w * cot * inv_rm - K.cor_sc * K.p2om * costhe)
           + c_t * (cec * dpdthe - tt);
        xw = c_u * (-up - K.cor_rad_f * K.m2om * geo.sinthe_bf)
           + c_v * (-vp + 2.0 * w * cot * inv_rm - K.cor_sc * K.m2om * costhe)
           + c_w * (-wp - (u + v * cot) * inv_rm - vm - D * lap)
           + c_t * (cec * dpdphi - tp);
        xt = c_t * (P0 * dcpf - Dt * lap);
    }
    double cw[6], cd[6];                                // transport and diffusion weights of the neighbours
#pragma unroll
    for(int d = 0; d < 6; d++){
        const AdjRow& R = rows[d == 0 ? 6 + tj : (d == 1 ? 10 + tj : (d == 2 ? tj : (d == 3 ? 2 + tj : 1 + tj)))];
        const double sg = (d & 1) ? -1.0 : 1.0;         // the first differences' sign: + from the lower neighbour
        const double D = ire + nt[d], Dt = irp + nt[d] * i09;
        const double c = sg * (d < 2 ? K.inv_2dr : (d < 4 ? R.t1 : R.p1));
        cw[d] = -wn[d] * c;
        cd[d] = d < 2 ? sg * R.r2 + K.inv_dr2 : (d < 4 ? sg * R.t2 + R.t3 : R.p3);
        const double WT = cw[d] + Dt * cd[d], WD = cw[d] + D * cd[d];
        xt += at[d] * WT; xv += av[d] * WD; xw += aw[d] * WD;
        if(d < 2) xu += au[d] * (WD + D * (sg * R.r2));
        else {
            xu += au[d] * WD;
            if(d < 4){ xu += av[d] * (sg * R.t4 * D); h -= av[d] * c; }
            else {
                const double c5 = sg * R.p5 * D;
                xu += aw[d] * (sg * R.p4 * D); xv += aw[d] * c5; xw -= av[d] * c5;
                h -= aw[d] * c;
            }
        }
        pd += (wn[d] * pe[d] - K.scale_p * a0[d]) * c;
    }
    if(NF == ADJ_NF_MOIST){
        // The twelve condensable species (:790-850, scalar_rhs in rk4.cuh): rhs_q = -(u d1r + v/r d1t +
        // w/(r sin) d1p)(q) + D_q lap(q) + forcing, D_q = 1/(Sc_g Re) + nue_t/0.9, the forcing held fixed.
        double bw[6];
#pragma unroll
        for(int d = 0; d < 6; d++) bw[d] = cw[d] + (nt[d] * i09) * cd[d];
        const double b0 = -(nt[6] * i09) * lap;
#pragma unroll 1
        for(int gi = 0; gi < (NF - ADJ_NF) / 3; gi++){
            const double isc = K.inv_sc_re[gi];
            double W[6];
#pragma unroll
            for(int d = 0; d < 6; d++) W[d] = bw[d] + isc * cd[d];
            const double W0 = b0 - isc * lap;
            // every load of the gas's three fields before the first store, which the compiler must assume
            // to alias them
            double an[3][6], aq[3], yb[3], g0[3];
            R7<double> rq[3];
#pragma unroll
            for(int n = 0; n < 3; n++){
                const size_t f = (size_t)(ADJ_NF + 3 * gi + n) * fs;
                const double* kq = a.kbar + f;
#pragma unroll
                for(int d = 0; d < 6; d++) an[n][d] = ldr(kq + on[d]);
                rq[n] = stencil(ADJ_NF + 3 * gi + n);
                aq[n] = ldr(kq + o); yb[n] = a.ybar[f + o]; g0[n] = ldr(a.g0 + f + o);
            }
#pragma unroll
            for(int n = 0; n < 3; n++){
                const size_t f = (size_t)(ADJ_NF + 3 * gi + n) * fs;
                double x = aq[n] * W0;
                const double sr = rq[n].rp - rq[n].rm, st = rq[n].tp - rq[n].tm, sp = rq[n].pe - rq[n].pw;
                xu -= aq[n] * ((in ? sr : 0.0) * K.inv_2dr);
                xv -= aq[n] * inv_rm * ((in ? st : 0.0) * K.inv_2dthe);
                xw -= aq[n] * inv_rs * ((in ? sp : 0.0) * K.inv_2dphi);
#pragma unroll
                for(int d = 0; d < 6; d++) x += an[n][d] * W[d];
                a.ybar[f + o] = yb[n] + x;
                if(in && a.Xprev) a.kbar_out[f + o] = a.w_prev * g0[n] + a.c_prev * x;
            }
        }
    }
    // what the cell adds to, all of it loaded before the first store
    const double x[ADJ_NF] = {xt, xu, xv, xw};
    const bool prev = in && a.Xprev;
    double yb[ADJ_NF], gb[ADJ_NF] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
    for(int q = 0; q < ADJ_NF; q++) yb[q] = a.ybar[(size_t)q * fs + o];
    const double ph = a.phbar[o], pdb = a.pdbar[o];
    double tp = 0.0;
    if(prev){
#pragma unroll
        for(int q = 0; q < ADJ_NF; q++) gb[q] = ldr(a.g0 + (size_t)q * fs + o);
        tp = ldr(a.Xprev + o);
    }
#pragma unroll
    for(int q = 0; q < ADJ_NF; q++) a.ybar[(size_t)q * fs + o] = yb[q] + x[q];
    a.phbar[o] = ph + h;
    a.pdbar[o] = pdb + pd;
    if(prev){
        double kt = 0.0;
#pragma unroll
        for(int q = 0; q < ADJ_NF; q++){
            const double kn = a.w_prev * gb[q] + a.c_prev * x[q];
            if(q == 0) kt = kn;
            a.kbar_out[(size_t)q * fs + o] = kn;
        }
        a.pe_out[o] = K.ce_sp * adj_cpf(K, a.cp_tab, tp) * kt;
    }
}

// ---- the saturation adjustment's implicit adjoint ----
// Per cell the forward (satadj_kernel, SaturationAdjustment.h:255-746) runs the four gases in the
// loop's order H2O, H2S, NH3, CH4, the temperature carried from one to the next. For one gas every
// step it takes -- the entry melt (:365-385) and freeze (:388-399), the Newton passes with their
// Bergeron conversion and in-pass melt (:450-590) -- moves mass between vapour q_v, cloud q_c and
// ice q_i and heat by the latent heats (L_f = L_s - L_v), so the total W = q_v + q_c + q_i and the
// moist enthalpy E = h T - L_v q_c - L_s q_i (h = cp_mix rho) are invariant. The converged state
// is the root of the closure q_v = H(T, q_c, q_i) on that invariant set, with the phases present
// at convergence frozen (the branch of the forward):
//   ice only      q_v = q_I(T), q_i = W - q_v              h dT = dE + L_s dW - L_s q_I'(T) dT
//   liquid only   q_v = q_R(T), q_c = W - q_v              (L_v, q_R likewise)
//   both          H = r q_R + (1 - r) q_I with the condensate split r = q_c / (q_c + q_i) frozen,
//                 L = r L_v + (1 - r) L_s
//   none          q_v = W, T = E / h (everything evaporated)
// so dT = (dE + L dW) / (h + L H'(T)) and the rest follows; this is the derivative of the exact
// root, which the forward approaches to its 1e-3 stopping test. A gas the forward leaves alone
// (no adjustment needed) contributes the derivative of its entry melt / freeze, each linear on its
// frozen branch (full, or capped at the phase temperature), and of the entry clamps.
// The temperature entering each gas is reconstructed from the invariants: the gas's entry state
// (the taped input, then each earlier gas's own entry and result) gives E, and its result gives
// T = (E + L_v q_c + L_s q_i) / h. The entry logic deciding whether a gas adjusts is the forward's
// FP64 path restated.
struct SatEntry {
    bool skip, go, cneg, clneg, ineg;
    int melt, freeze;            // 0 none, 1 whole amount, 2 capped at the phase temperature,
                                 // 3 mass only (L_f <= 0), 4 ice dropped (no conservation: melt only)
    double t_u, c, cloud, ice;   // after the entry steps and clamps
};

__device__ __forceinline__ double sat_q_d(const GasConst& G, bool ice, double rho_c, double p_u, double T, double* dq){
    const double C = ice ? G.C_i : G.C, L0 = ice ? G.L0_i : G.L0;
    const double al = ice ? G.del_alf_i : G.del_alf, be = ice ? G.del_bet_i : G.del_bet;
    const double q = rho_c * G.ep * svp(T, C, L0, G.den, al, be) / p_u;
    if(dq) *dq = q * (L0 / (T * T) + al / T + be) / G.den;
    return q;
}

// :358-448 on the FP64 path: the entry steps and the decision to adjust.
__device__ SatEntry sat_entry(const SatConst& K, const GasConst& G, double rho_c, double p_u, double t_u,
                              double c, double cloud, double ice){
    SatEntry e;
    e.skip = !((t_u > 0.0) && (p_u > 0.0));
    e.go = false; e.melt = 0; e.freeze = 0; e.cneg = e.clneg = e.ineg = false;
    e.t_u = t_u; e.c = c; e.cloud = cloud; e.ice = ice;
    if(e.skip) return e;
    const double t_0 = G.t_0, t_00 = G.t_00, Lf = G.Lf, hc = K.cp_mix * rho_c;
    if(t_u > t_0){
        if(K.conserve){
            if(ice > 0.0){
                double dm = ice;
                if(Lf > 0.0){
                    const double cap = hc * (t_u - t_0) / Lf;
                    e.melt = 1;
                    if(dm > cap){ dm = cap; e.melt = 2; }
                    t_u -= Lf * dm / hc;
                } else e.melt = 3;
                ice -= dm;
                cloud += dm;
            }
        } else { e.melt = 4; ice = 0.0; }
    }
    if(G.freeze_on && t_u < t_00 && cloud > 0.0){
        double dm = cloud;
        if(Lf > 0.0){
            const double cap = hc * (t_00 - t_u) / Lf;
            e.freeze = 1;
            if(dm > cap){ dm = cap; e.freeze = 2; }
            t_u += Lf * dm / hc;
        } else e.freeze = 3;
        cloud -= dm;
        ice += dm;
    }
    if(c < 0.0){ c = 0.0; e.cneg = true; }
    if(cloud < 0.0){ cloud = 0.0; e.clneg = true; }
    if(ice < 0.0){ ice = 0.0; e.ineg = true; }
    e.t_u = t_u; e.c = c; e.cloud = cloud; e.ice = ice;
    const double q_Rain_0 = sat_q_d(G, false, rho_c, p_u, t_u, nullptr);
    bool go = q_Rain_0 > 0.0;
    if(go){
        double q_entry = q_Rain_0;
        if(K.ice_entry && cloud <= 0.0 && ice <= 0.0){
            const double cnd0 = t_u <= t_00 ? 0.0 : (t_u >= t_0 ? 1.0 : (t_u - t_00) * G.t_range_inv);
            if(cnd0 < 1.0) q_entry = cnd0 * q_Rain_0 + (1.0 - cnd0) * sat_q_d(G, true, rho_c, p_u, t_u, nullptr);
        }
        if(K.bergeron >= 2 && cloud <= 0.0 && ice <= 0.0 && t_u < t_0) q_entry = sat_q_d(G, true, rho_c, p_u, t_u, nullptr);
        if(c <= q_entry){
            if(!K.evap || !K.conserve || (cloud <= 0.0 && ice <= 0.0)) go = false;
            else {
                const double q_Ice_0 = sat_q_d(G, true, rho_c, p_u, t_u, nullptr);
                double q_t0;
                if(cloud > 0.0 && ice > 0.0) q_t0 = (cloud * q_Rain_0 + ice * q_Ice_0) / (cloud + ice);
                else if(ice <= 0.0)          q_t0 = q_Rain_0;
                else                         q_t0 = q_Ice_0;
                if(fabs(c - q_t0) <= K.entry_tol * q_t0) go = false;
            }
        }
    }
    e.go = go;
    return e;
}

// The entry steps' adjoint: cotangents of (t_u, c, cloud, ice) after them -> before them.
__device__ void sat_entry_adj(const GasConst& G, double hc, const SatEntry& e, double& Tb, double& cb, double& clb, double& ib){
    const double Lf = G.Lf;
    if(e.cneg) cb = 0.0;
    if(e.clneg) clb = 0.0;
    if(e.ineg) ib = 0.0;
    if(e.freeze == 1){ clb = Tb * Lf / hc + ib; }
    else if(e.freeze == 2){ Tb = (clb - ib) * hc / Lf; }
    else if(e.freeze == 3){ clb = ib; }
    if(e.melt == 1){ ib = -Tb * Lf / hc + clb; }
    else if(e.melt == 2){ Tb = (clb - ib) * hc / Lf; }
    else if(e.melt == 3){ ib = clb; }
    else if(e.melt == 4){ ib = 0.0; }
}

// One cell: ybar (fields 0..15 of the step's RK4 input, i.e. after the adjustment) -> the same
// before it. pre: the taped state before the adjustment; post: after it (ADJ_NF_MOIST fields each).
__global__ void __launch_bounds__(128) adj_satadj_kernel(Grid g, const double* pre, const double* post, const double* ps,
                                                         const double* rho_mix, SatConst K, double* ybar){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y, i = blockIdx.z;
    if(k >= g.km) return;
    const size_t fs = g.fstride, q = gidx(g, i, j, k);
    const double p_u = ps[q];
    double rho_c = K.r_mix;                               // rho_at, cUranusModel.h:526-531
    if(K.local_rho){ const double r_ = rho_mix[q]; rho_c = (r_ > 0.0 && isfinite(r_)) ? r_ : K.r_mix; }
    const double hc = K.cp_mix * rho_c, t_ref = K.t_ref;
    const int base[4] = {ATURAN_H2O, ATURAN_H2S, ATURAN_NH3, ATURAN_CH4};
    // every value of the cell up front (the loops over the gases would load a gas's behind the work, and the
    // stores, of the one before it): state on entry, cloud and ice after, adjoints
    double pv[4][3], qv[4][2], yv[4][3];
#pragma unroll
    for(int gi = 0; gi < 4; gi++){
        const size_t f = (size_t)base[gi] * fs + q;
#pragma unroll
        for(int n = 0; n < 3; n++){ pv[gi][n] = ld(pre + f + n * fs); yv[gi][n] = ybar[f + n * fs]; }
        qv[gi][0] = ld(post + f + fs); qv[gi][1] = ld(post + f + 2 * fs);
    }
    const double yt = ybar[q];
    // forward replay: each gas's entry record and the temperature after it
    SatEntry ent[4];
    double Tout[4];
    double T = pre[q] * t_ref;
    for(int gi = 0; gi < 4; gi++){
        const GasConst& G = K.gas[gi];
        ent[gi] = sat_entry(K, G, rho_c, p_u, T, pv[gi][0], pv[gi][1], pv[gi][2]);
        const SatEntry& e = ent[gi];
        if(e.skip){ Tout[gi] = T; continue; }
        if(e.go){
            const double E = hc * e.t_u - G.lv * e.cloud - G.ls * e.ice;
            T = (E + G.lv * qv[gi][0] + G.ls * qv[gi][1]) / hc;
        } else T = e.t_u;
        Tout[gi] = T;
    }
    // reverse
    double Tb = yt / t_ref;
    for(int gi = 3; gi >= 0; gi--){
        const GasConst& G = K.gas[gi];
        const size_t f = (size_t)base[gi] * fs + q;
        const SatEntry& e = ent[gi];
        if(e.skip) continue;
        double cb = yv[gi][0], clb = yv[gi][1], ib = yv[gi][2];
        if(e.go){
            const double qc = qv[gi][0], qi = qv[gi][1], Tp = Tout[gi];
            double Eb, Wb;
            if(qc > 0.0 && qi > 0.0){
                const double r = qc / (qc + qi), L = r * G.lv + (1.0 - r) * G.ls;
                double dR, dI;
                sat_q_d(G, false, rho_c, p_u, Tp, &dR);
                sat_q_d(G, true, rho_c, p_u, Tp, &dI);
                const double dH = r * dR + (1.0 - r) * dI, Cb = r * clb + (1.0 - r) * ib;
                const double a = (Tb + (cb - Cb) * dH) / (hc + L * dH);
                Eb = a; Wb = a * L + Cb;
            } else if(qi > 0.0){
                double dI;
                sat_q_d(G, true, rho_c, p_u, Tp, &dI);
                const double a = (Tb + (cb - ib) * dI) / (hc + G.ls * dI);
                Eb = a; Wb = a * G.ls + ib;
            } else if(qc > 0.0){
                double dR;
                sat_q_d(G, false, rho_c, p_u, Tp, &dR);
                const double a = (Tb + (cb - clb) * dR) / (hc + G.lv * dR);
                Eb = a; Wb = a * G.lv + clb;
            } else {
                Eb = Tb / hc; Wb = cb;
            }
            Tb = Eb * hc; cb = Wb; clb = Wb - G.lv * Eb; ib = Wb - G.ls * Eb;
        }
        sat_entry_adj(G, hc, e, Tb, cb, clb, ib);
        ybar[f] = cb; ybar[f + fs] = clb; ybar[f + 2 * fs] = ib;
    }
    ybar[q] = Tb * t_ref;
}

// The final update's adjoint: g = ybar' (times 0 where T' was clamped), ybar = g, kbar_3 =
// dt/6 w_3 g on the interior. ybar_in is the caller's adjoint of the step's output; pe of stage 3 is
// formed from its input t3, nt from nue.
__global__ void __launch_bounds__(128) adj_init_kernel(Grid g, const double* ybar_in, const double* t_out, double t_min, double t_max,
                                double w3, double* g0, double* ybar, double* kbar, double* phbar, double* pdbar, int nf,
                                RhsConst<double> K, const double* cp_tab, const double* t3, const double* nue, double* pe, double* nt){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    const int i = blockIdx.z;
    if(k >= g.km) return;
    const size_t fs = g.fstride;
    const size_t o = gidx(g, i, j, k);
    const bool interior = i >= 1 && i <= g.im - 2 && j >= 1 && j <= g.jm - 2 && k <= g.km - 2;
    const double to = t_out[o], t3o = t3[o], nu = nue[o];
    // four fields at a time (nf is 4 or 16), their loads before their stores
    for(int q0 = 0; q0 < nf; q0 += 4){
        double v[4];
#pragma unroll
        for(int c = 0; c < 4; c++) v[c] = ybar_in[(q0 + c) * fs + o];
        if(q0 == 0 && interior && !(to > t_min && to < t_max)) v[0] = 0.0;
#pragma unroll
        for(int c = 0; c < 4; c++){
            const size_t p = (q0 + c) * fs + o;
            g0[p] = interior ? v[c] : 0.0;
            ybar[p] = v[c];
            kbar[p] = interior ? w3 * v[c] : 0.0;
        }
        if(q0 == 0) pe[o] = interior ? K.ce_sp * adj_cpf(K, cp_tab, t3o) * (w3 * v[0]) : 0.0;
    }
    phbar[o] = 0.0;
    pdbar[o] = 0.0;
    nt[o] = adj_nue(K, nu);
}

// Hydrostatic integral's adjoint, per column (RungeKutta_Uran_Turb.cpp:62-177): p_hydro(i) =
// sum_{n=1..i} (F(n-1) + F(n)) dr / 2 + const, F = cB buoy + met (cB = 1 - 1/follow_tau when the
// follow filter advances, else 1). Fbar(m) = dr/2 (S(m+1) + [m >= 1] S(m)), S the suffix sums of
// phbar. Adds the met part into vbar, wbar and the local buoy part into Tbar; leaves, per cell,
// the contribution to its level mean's adjoint in rbar.
//
// A block owns 32 consecutive columns. All its threads bring a chunk of phbar (top down) into shared
// memory, one warp turns it into suffix sums in order (only those adds are serial), all threads do the
// per-cell work. One thread per column walking the levels, the divisions in its chain, left 65 blocks
// for the chip at 41x91x181 and took 151 us.
constexpr int ADJ_HCH = 48;                        // levels per chunk
__global__ void __launch_bounds__(256) adj_hydro_kernel(Grid g, const double* t, const double* ps, const double* v,
                                                        const double* w, const double* ref, const double* rm_i,
                                                        const double* cor_j, const double* phbar, double* ybar,
                                                        double* rbar, HydroConst h){
    chain_wait();
    __shared__ double sS[ADJ_HCH + 1][32];         // S(m) of the chunk's levels; the last row S of the level above it
    const int tx = threadIdx.x, ty = threadIdx.y;
    const int c = blockIdx.x * 32 + tx;
    const bool col = c < g.jm * g.km;
    const int j = col ? c / g.km : 0, k = col ? c - j * g.km : 0;
    const size_t fs = g.fstride;
    const double cB = h.follow_on ? 1.0 - 1.0 / h.follow_tau : 1.0;
    const double cor = cor_j[j];
    double S = 0.0;                                // the serial lane's running suffix sum
    for(int m1 = g.im; m1 > 0; m1 -= ADJ_HCH){     // levels m0 .. m1 - 1
        const int m0 = max(0, m1 - ADJ_HCH), n = m1 - m0;
        for(int r = ty; r < n; r += 8) sS[r][tx] = col ? phbar[gidx(g, m0 + r, j, k)] : 0.0;
        __syncthreads();
        if(ty == 0){
            sS[n][tx] = S;
            for(int r = n - 1; r >= 0; r--){ S += sS[r][tx]; sS[r][tx] = S; }
        }
        __syncthreads();
        if(col)
            for(int r = ty; r < n; r += 8){
                const int m = m0 + r;
                const size_t o = gidx(g, m, j, k);
                const double Fb = 0.5 * h.dr * (sS[r + 1][tx] + (m >= 1 ? sS[r][tx] : 0.0));
                const double vv = v[o], ww = w[o], T = t[o], p = ps[o];
                const double yv = ybar[2 * fs + o], yw = ybar[3 * fs + o], yt = ybar[o];
                ybar[2 * fs + o] = yv + Fb * 2.0 * vv / rm_i[m];
                ybar[3 * fs + o] = yw + Fb * (2.0 * ww / rm_i[m] + cor);
                double rb = 0.0;
                if(T > 0.0){
                    const double b = h.g * p / (h.rR * T * h.t_ref);
                    const double f = h.m_nd_rel_b * (b - ref[m]) / ref[m];
                    if(isfinite(f)){
                        const double FbB = cB * Fb;
                        ybar[o] = yt + FbB * h.m_nd_rel_b / ref[m] * (-b / T);
                        rb = FbB * (-h.m_nd_rel_b * b / (ref[m] * ref[m]));
                    }
                }
                rbar[o] = rb;
            }
        __syncthreads();
    }
}

// Level mean's adjoint (RungeKutta_Uran_Turb.cpp:18-37): per level, Rbar = sum rbar and the weight sum W
// over the valid cells, in a fixed tree order (ADJ_LB blocks per level, their partials added in block
// order by the apply kernel); then per valid cell Tbar += Rbar / W * wsin_j * db/dT, db/dT = -b / T.
constexpr int ADJ_LB = 16;
__global__ void __launch_bounds__(256) adj_level_sum_kernel(Grid g, const double* t, const double* ps,
                                                            const double* wsin, const double* rbar,
                                                            HydroConst h, double* lev){
    chain_wait();
    const int m = blockIdx.y;
    double s = 0.0, ws = 0.0;
    for(int c = blockIdx.x * 256 + threadIdx.x; c < g.jm * g.km; c += ADJ_LB * 256){
        const int j = c / g.km, k = c - j * g.km;
        const size_t o = gidx(g, m, j, k);
        const double T = t[o];
        if(!(T > 0.0)) continue;
        const double b = h.g * ps[o] / (h.rR * T * h.t_ref);
        if(!isfinite(b)) continue;
        s += rbar[o];
        ws += wsin[j];
    }
    __shared__ double ss[256], sw[256];
    ss[threadIdx.x] = s; sw[threadIdx.x] = ws;
    __syncthreads();
    for(int st = 128; st > 0; st >>= 1){
        if(threadIdx.x < st){ ss[threadIdx.x] += ss[threadIdx.x + st]; sw[threadIdx.x] += sw[threadIdx.x + st]; }
        __syncthreads();
    }
    if(threadIdx.x == 0){ double* q = lev + 2 * ((size_t)m * ADJ_LB + blockIdx.x); q[0] = ss[0]; q[1] = sw[0]; }
}

__global__ void __launch_bounds__(128) adj_level_apply_kernel(Grid g, const double* t, const double* ps, const double* wsin,
                                                              const double* lev, HydroConst h, double* ybar){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    const int m = blockIdx.z;
    double R = 0.0, W = 0.0;
#pragma unroll
    for(int b = 0; b < ADJ_LB; b++){ R += ld(lev + 2 * (m * ADJ_LB + b)); W += ld(lev + 2 * (m * ADJ_LB + b) + 1); }
    if(k >= g.km) return;
    const size_t o = gidx(g, m, j, k);
    const double T = t[o];
    if(!(T > 0.0) || !(W > 0.0)) return;
    const double b = h.g * ps[o] / (h.rR * T * h.t_ref);
    if(!isfinite(b)) return;
    ybar[o] += R / W * wsin[j] * (-b / T);
}

// The heating field's adjoint: heat_scale times the T tendencies' adjoint summed over the stages and
// the interior levels, per (j,k); 0 on the polar rows and the seam column, which no stage reads.
__global__ void adj_heat_reduce_kernel(Grid g, const double* hacc, double scale, double* out){
    chain_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if(c >= g.jm * g.km) return;
    const int j = c / g.km, k = c - j * g.km;
    double s = 0.0;
    if(j >= 1 && j <= g.jm - 2 && k <= g.km - 2)
        for(int i = 1; i < g.im - 1; i++) s += hacc[gidx(g, i, j, k)];
    out[c] = scale * s;
}

// ---- The pressure step's adjoint (RB_SOR / RB_LINE path): p_dyn = F(solve(compat(clamp(div aux))))
// with F the boundary passes. Reverse: F^T, the transposed solve, compat^T, the clamp mask, div^T. ----

// F^T in reverse order of launch_pdyn_bcs: seam copy, theta folds (every level), radial folds.
__global__ void adj_pbc_p_kernel(Grid g, double* B){
    chain_wait();
    const int c = blockIdx.x * blockDim.x + threadIdx.x;
    if(c >= g.im * g.jm) return;
    const int i = c / g.jm, j = c - i * g.jm;
    B[gidx(g, i, j, 0)] += B[gidx(g, i, j, g.km - 1)];
    B[gidx(g, i, j, g.km - 1)] = 0.0;
}
__global__ void adj_pbc_t_kernel(Grid g, double* B){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int i = blockIdx.y;
    if(k >= g.km) return;
    const double b0 = B[gidx(g, i, 0, k)], bn = B[gidx(g, i, g.jm - 1, k)];
    B[gidx(g, i, 0, k)] = 0.0; B[gidx(g, i, g.jm - 1, k)] = 0.0;
    B[gidx(g, i, 1, k)] += C43 * b0;        B[gidx(g, i, 2, k)] -= C13 * b0;
    B[gidx(g, i, g.jm - 2, k)] += C43 * bn; B[gidx(g, i, g.jm - 3, k)] -= C13 * bn;
}
__global__ void adj_pbc_r_kernel(Grid g, double* B){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    if(k >= g.km) return;
    const double b0 = B[gidx(g, 0, j, k)], bn = B[gidx(g, g.im - 1, j, k)];
    B[gidx(g, 0, j, k)] = 0.0; B[gidx(g, g.im - 1, j, k)] = 0.0;
    B[gidx(g, 1, j, k)] += C43 * b0;        B[gidx(g, 2, j, k)] -= C13 * b0;
    B[gidx(g, g.im - 2, j, k)] += C43 * bn; B[gidx(g, g.im - 3, j, k)] -= C13 * bn;
}

// compat^T: the forward subtracts the constant (sum w src) / (sum w) from the interior source
// (w = y_i y_j), so its transpose maps lam to lam - w (sum lam) / (sum w); `mean` holds
// sum lam / n_interior and ratio = n_interior / sum w. Then the clamp mask from the forward's
// clamped source.
__global__ void adj_compat_mask_kernel(Grid g, const double* lam, const double* mean, double ratio,
                                       const double* src_fwd, const RBW* w, double* sbar){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = 1 + blockIdx.y;
    const int i = 1 + blockIdx.z;
    if(k > g.km - 2) return;
    const size_t o = gidx(g, i, j, k);
    const double wy = ywt(i, 1, g.im - 2) * ywt(j, 1, g.jm - 2);
    const double v = lam[o] - wy * ratio * (*mean);
    const double s = src_fwd[o];
    const bool free_ = fabs(s) < w[i * g.jm + j].src_max;   // not clamped (clamped values sit at the bound)
    sbar[o] = free_ ? v : 0.0;
}

// div^T (rb_src_kernel): src(i,j,k) = (au[i+1] - au[i-1]) inv_2dr + (av[j+1] - av[j-1]) inv_2dthe inv_rm
// + (aw[k+1] - aw[k-1]) inv_2dphi inv_rmsinthe, with au = 0 on the radial boundary rows (rigid lid)
// or cubically extrapolated from the interior, and av = 0 on the polar rows (Pressure_Uran.cpp:30-146).
__global__ void adj_div_kernel(Grid g, const double* sbar, const RBW* w, PressConst c, int rigid_lid,
                               double* aub, double* avb, double* awb){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x;
    const int j = blockIdx.y;
    const int i = blockIdx.z;
    if(k >= g.km) return;
    const size_t o = gidx(g, i, j, k);
    const bool inner = i >= 1 && i <= g.im - 2 && j >= 1 && j <= g.jm - 2 && k <= g.km - 2;
    double u = 0.0, v = 0.0, ww = 0.0;
    if(inner){
        const size_t si = (size_t)g.jm * g.kp, sj = g.kp;
        if(i - 1 >= 1)        u += sbar[o - si] * c.inv_2dr;
        if(i + 1 <= g.im - 2) u -= sbar[o + si] * c.inv_2dr;
        if(!rigid_lid){       // au[0] = au[3] - 3 au[2] + 3 au[1], au[im-1] likewise (reads of the rows 1, im-2)
            const double b0 = -sbar[gidx(g, 1, j, k)] * c.inv_2dr;        // adjoint of au[0]
            const double bn =  sbar[gidx(g, g.im - 2, j, k)] * c.inv_2dr; // adjoint of au[im-1]
            if(i == 1) u += 3.0 * b0;
            if(i == 2) u -= 3.0 * b0;
            if(i == 3) u += b0;
            if(i == g.im - 2) u += 3.0 * bn;
            if(i == g.im - 3) u -= 3.0 * bn;
            if(i == g.im - 4) u += bn;
        }
        if(j - 1 >= 1)        v += sbar[o - sj] * c.inv_2dthe * w[i * g.jm + j - 1].inv_rm;
        if(j + 1 <= g.jm - 2) v -= sbar[o + sj] * c.inv_2dthe * w[i * g.jm + j + 1].inv_rm;
        const int kw = phi_wrap(k - 1, g.km), ke = phi_wrap(k + 1, g.km);
        ww = (sbar[o - k + kw] - sbar[o - k + ke]) * c.inv_2dphi * w[i * g.jm + j].inv_rmsinthe;
    }
    aub[o] = u; avb[o] = v; awb[o] = ww;
}

}  // namespace aturan
