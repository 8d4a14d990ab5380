// The passes that follow RungeKuttaUran in one iteration (planet/cUranusModel.cpp:1218-1248): the
// 1-2-1 filters of lib/Utils.cpp:224-317 (damp_wiggles), the boundary passes of
// BoundaryConditions.h:152-518 as BC_Uran.h:140-173 runs them for Uranus (margin 0, Neumann
// default, no turbulence fields, no pole fill rows), the species floor of the radial planes and
// the species clamp (BC_Uran.h:91-128).
//
// All of it is streaming work on a few planes of the state, bound by HBM. The filters update a
// field in place: along k one warp holds a row in shared memory; along j and i one thread walks
// a column, keeping the old values of the cell and its lower neighbour in registers, so every old
// value is read before it is overwritten, as the reference's copy of the field guarantees. The
// boundary passes are column-local (radius: per (j,k), theta: per (i,k), phi: per (i,j)) and
// field-local, so a thread applies every step of one field's column in the reference's order,
// and one launch per pass keeps the reference's order between passes. Arithmetic is FP64 on the stored values (FP32
// storage in the mixed form is widened, computed in FP64 and rounded back).
#pragma once
#include "common.cuh"
#include "pressure.cuh"

namespace aturan {

// Field tables: the reference's lists (BC_Uran.cpp:21-88) restricted to the fields the context
// holds. The phi list is the radius list's first POST_NPHI fields: all but difflux_nh4sh.
constexpr int POST_NRAD = 25, POST_NPHI = 24, POST_NTHX = 16, POST_NTHZ = 9, POST_NSP = 13;

// Which filter passes run and the clamp's scratch: part holds 2 nb doubles per species, out 2 x 13.
struct PostPlan {
    double damp_t_horiz, damp_t_vert, vel_shapiro;
    int damp_t_j, species_clamp, nb;
    double *part, *out;
};

template <typename S>
struct PostArgs {
    Grid g;
    S* rad[POST_NRAD];           // radius and phi passes: t, u, v, w, the species (4..16), the fluxes, difflux
    S* thx[POST_NTHX];           // theta pass, extrapolated to the poles
    S* thz[POST_NTHZ];           // theta pass, zeroed at the poles (v, w first)
    S* sp[POST_NSP];             // species for the clamp, in BC_Uran.h:83-89's order
    S *u, *v, *w;
    float* tlo;                  // the mixed form's temperature pair (common.cuh): t's low part, else null
    int radius_form, bottom_form, pole_form, lid_u, top_taper, lid_vw, positive, phi_periodic;
};

// BCForm::apply with the model default NEUMANN (BoundaryConditions.h, cUranusModel.h:397)
__device__ __forceinline__ double post_form(int form, double a, double b, double c){
    const int f = (form == 0) ? 2 : form;
    if(f == 1) return a;
    if(f == 2) return C43 * a - C13 * b;
    return c - 3.0 * b + 3.0 * a;
}
__device__ __forceinline__ double post_max0(double x){ return (0.0 < x) ? x : 0.0; }   // std::max(0.0, x)

// ---- damp_wiggles (lib/Utils.cpp:224-317), one axis per launch ----

// Along k: one warp per (i, j) row (blockDim.y rows per block), the row's old values in the warp's
// own slice of shared memory, ~km/32 loads in flight per lane. With the periodic seam the ring is
// k = 0..km-2 and k = km-1 takes the new k = 0; otherwise k wraps over all km. lo: the low part of
// the mixed form's temperature pair when x is its t (common.cuh), else null.
template <typename S>
__global__ void __launch_bounds__(128) post_filter_k_kernel(Grid g, S* x, float* lo, double coeff, int seam, int rows){
    chain_wait();
    extern __shared__ double sm[];
    const int r = blockIdx.x * blockDim.y + threadIdx.y;
    if(r >= rows) return;                          // a whole warp: only warp-level syncs below
    const int km = g.km;
    double* row = sm + (size_t)threadIdx.y * km;
    const size_t o = (size_t)r * g.kp;
    for(int k = threadIdx.x; k < km; k += 32) row[k] = t_ld(x, lo, o + k);
    __syncwarp();
    const int k_end = seam ? km - 1 : km;
    for(int k = threadIdx.x; k < k_end; k += 32){
        const int km1 = seam ? (k == 0 ? km - 2 : k - 1) : (k - 1 + km) % km;
        const int kp1 = seam ? (k == km - 2 ? 0 : k + 1) : (k + 1) % km;
        const double c = row[k];
        const double y = c + coeff * (row[km1] - 2.0 * c + row[kp1]);
        t_st(x, lo, o + k, y);
        if(seam && k == 0) t_st(x, lo, o + km - 1, y);
    }
}

// Along a column of n cells at stride st from x0 (j: clamped at the poles; i: at the ends).
template <typename S>
__device__ __forceinline__ void post_walk(S* x0, float* lo0, size_t st, int n, double coeff){
    double pm = t_ld(x0, lo0, 0), c = pm;
    for(int q = 0; q < n; q++){
        const double nx = (q + 1 < n) ? t_ld(x0, lo0, (size_t)(q + 1) * st) : c;
        t_st(x0, lo0, (size_t)q * st, c + coeff * (pm - 2.0 * c + nx));
        pm = c;
        c = nx;
    }
}
template <typename S>
__global__ void __launch_bounds__(128) post_filter_j_kernel(Grid g, S* x, float* lo, double coeff){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y;
    if(k >= g.km) return;
    const size_t o = gidx(g, i, 0, k);
    post_walk(x + o, lo ? lo + o : nullptr, (size_t)g.kp, g.jm, coeff);
}
template <typename S>
__global__ void __launch_bounds__(128) post_filter_i_kernel(Grid g, S* x, float* lo, double coeff){
    chain_wait();
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y;
    if(k >= g.km) return;
    const size_t o = gidx(g, 0, j, k);
    post_walk(x + o, lo ? lo + o : nullptr, (size_t)g.jm * g.kp, g.im, coeff);
}

// ---- damp_wiggles along k, j and i in one pass, out of place (x -> y) ----
// The three 1-2-1 passes of damp_wiggles with all axes on, fused over li levels of FT_J x FT_K
// outputs: the k pass of the tile and its one-cell i and j halo is formed from global memory (the
// k neighbours are the row's own, L1 hits), the j pass of the tile and its i halo from that, the i
// pass from that. The halo rows and planes are the clamped ones the passes use at the poles and
// the ends (j - 1 of j = 0 is j = 0, and likewise), so every output is formed from exactly the
// values, and by exactly the arithmetic, of the three passes in turn. With the periodic seam the
// k pass of k = km-1 is that of k = 0 (the pass's copy), and so the j and i passes there too. It is
// out of place (a tile that wrote in place could overwrite what its neighbour tile has yet to read):
// whoever forms the fields writes them unfiltered to scratch, and the filter puts them where they
// belong. FT_N fields to a launch: the chemistry's 4 + 4 filtered fields took eight launches of 22 us
// and eight copies back of 10 us at 41 x 181 x 361 (FP64).
constexpr int FT_N = 4;
template <typename S> struct Filter3 { const S* x[FT_N]; S* y[FT_N]; };
// A block takes FT_K meridians x FT_J rows and walks up li levels: the k pass of a level's rows
// (and the halo row on each side) goes to shared memory, double-buffered so that a level costs one
// barrier; the thread of a column forms the j pass from it and keeps the last three levels' j passes
// in registers for the i pass. The next level is in flight in registers meanwhile (two or four ahead
// cost warps and were slower). Four FP64 fields of 41 x 181 x 361: 83 us with tiles of 4 levels staged
// whole, 58 so (172 MB: 26 us).
// li: 21 levels a block, so that the halo levels cost a tenth, while that still makes a wave of blocks
// (58 us there, 66 with 7 levels), else 7 (21 x 37 x 73: 5.6 us against 10).
constexpr int FT_K = 32, FT_J = 8;
inline int filter3_levels(int km, int jm, int im){
    const long cols = (long)((km + FT_K - 1) / FT_K) * ((jm + FT_J - 1) / FT_J) * FT_N;
    return cols * ((im + 20) / 21) >= 148 * 8 ? 21 : 7;
}
template <typename S>
__global__ void __launch_bounds__(FT_K * FT_J) post_filter3_kernel(Grid g, const __grid_constant__ Filter3<S> f, int ni, int li, double coeff, int seam){
    chain_wait();
    __shared__ double YK[2][FT_J + 2][FT_K];
    const int n = blockIdx.z / ni;
    const S* x = f.x[n];
    const int tk = threadIdx.x, ty = threadIdx.y;              // 32 x 8
    const int k = blockIdx.x * FT_K + tk, j = blockIdx.y * FT_J + ty, i0 = (blockIdx.z - n * ni) * li;
    const int km = g.km;
    const int i1 = min(i0 + li, g.im);
    // the k pass's own index and neighbours (damp_wiggles, lib/Utils.cpp:250-265); off the row, those of
    // its first cell
    const int kq = k < km ? k : 0;
    const int kc = seam && kq == km - 1 ? 0 : kq;
    const int km1 = seam ? (kc == 0 ? km - 2 : kc - 1) : (kc - 1 + km) % km;
    const int kp1 = seam ? (kc == km - 2 ? 0 : kc + 1) : (kc + 1) % km;
    // this thread's rows: its own, and for the first and last row of the block the halo row
    const size_t pl = (size_t)g.jm * g.kp;
    const bool edge = ty == 0 || ty == FT_J - 1;
    const S* const row = x + (size_t)min(j, g.jm - 1) * g.kp;
    const S* const halo = x + (size_t)min(max(ty == 0 ? j - 1 : j + 1, 0), g.jm - 1) * g.kp;
    const int slot = ty == 0 ? 0 : FT_J + 1;
    S* const y = f.y[n] + (size_t)min(j, g.jm - 1) * g.kp + k;
    const bool on = k < km && j < g.jm;
    S c, w, e, hc = S(0), hw = S(0), he = S(0);
    auto fetch = [&](int i){
        const size_t o = (size_t)min(max(i, 0), g.im - 1) * pl;
        c = ld(row + o + kc); w = ld(row + o + km1); e = ld(row + o + kp1);
        if(edge){ hc = ld(halo + o + kc); hw = ld(halo + o + km1); he = ld(halo + o + kp1); }
    };
    double ym = 0.0, y0 = 0.0;                                  // j passes of levels i - 2 and i - 1
    fetch(i0 - 1);
    for(int i = i0 - 1; i <= i1; i++){
        double (*b)[FT_K] = YK[i & 1];
        b[ty + 1][tk] = (double)c + coeff * ((double)w - 2.0 * (double)c + (double)e);
        if(edge) b[slot][tk] = (double)hc + coeff * ((double)hw - 2.0 * (double)hc + (double)he);
        if(i < i1) fetch(i + 1);
        __syncthreads();
        const double v = b[ty + 1][tk];
        const double yp = v + coeff * (b[ty][tk] - 2.0 * v + b[ty + 2][tk]);
        if(on && i > i0) y[(size_t)(i - 1) * pl] = (S)(y0 + coeff * (ym - 2.0 * y0 + yp));
        ym = y0; y0 = yp;
    }
}

// ---- bcRadius (BoundaryConditions.h:152-286), floorRadialSpecies and the lid v, w (BC_Uran.h:91-170) ----
// One thread per (j, k) column of one field (blockIdx.z = the field's place in rad): the field's
// two end values, then what the reference does afterwards to that same column -- u = 0 at the
// ends (lid_u), the top taper and the lid form of v and w, the species floor. Every later step
// reads and writes only its own field's column, so the fields run side by side.
template <typename S>
__global__ void __launch_bounds__(128) post_bc_radius_kernel(PostArgs<S> a){
    chain_wait();
    const Grid& g = a.g;
    const int k = blockIdx.x * blockDim.x + threadIdx.x, j = blockIdx.y, n = blockIdx.z;
    if(k >= g.km) return;
    const int im = g.im;
    const size_t pl = (size_t)g.jm * g.kp;
    S* F = a.rad[n] + gidx(g, 0, j, k);
    auto at = [&](int i) -> S& { return F[(size_t)i * pl]; };
    const int fb = (a.bottom_form != 0 && n != 1) ? a.bottom_form : a.radius_form;
    if(n == 0 && a.tlo){                            // t as the mixed form's pair: its two end values, in order
        float* L = a.tlo + gidx(g, 0, j, k);
        auto get = [&](int i) -> double { return t_ld(F, L, (size_t)i * pl); };
        t_st(F, L, 0, post_form(fb, get(1), get(2), get(3)));
        t_st(F, L, (size_t)(im - 1) * pl, post_form(a.radius_form, get(im - 2), get(im - 3), get(im - 4)));
        return;
    }
    const bool species = n >= 4 && n <= 16;        // the twelve condensables and nh4sh
    if(im >= 8){
        // planes 1..3 and im-4..im-2 are disjoint from each other and from 0 and im-1: every
        // value is loaded up front (the third plane only for the cubic form), one round trip
        auto cubic = [](int f){ return f != 0 && f != 1 && f != 2; };
        const double b1 = (double)at(1), b2 = (double)at(2), b3 = cubic(fb) ? (double)at(3) : 0.0;
        const double t1 = (double)at(im - 2), t2 = (double)at(im - 3);
        const double t3 = cubic(a.radius_form) ? (double)at(im - 4) : 0.0;
        S y0 = (S)post_form(fb, b1, b2, b3), yl = (S)post_form(a.radius_form, t1, t2, t3);
        if(n == 1 && a.lid_u != 0){ y0 = (S)0.0; yl = (S)0.0; }
        if(species && a.positive != 0){          // the floor reads planes 1 and im-2, unchanged
            if((double)y0 < 0.0) y0 = (S)((a.positive == 2) ? post_max0(b1) : 0.0);
            if((double)yl < 0.0) yl = (S)((a.positive == 2) ? post_max0(t1) : 0.0);
        }
        at(0) = y0;
        at(im - 1) = yl;
        if(n != 2 && n != 3) return;
    } else {
        // in the reference's order, through memory (the planes overlap when im < 8)
        at(0) = (S)post_form(fb, (double)at(1), (double)at(2), (double)at(3));
        at(im - 1) = (S)post_form(a.radius_form, (double)at(im - 2), (double)at(im - 3), (double)at(im - 4));
        if(n == 1 && a.lid_u != 0){ at(0) = (S)0.0; at(im - 1) = (S)0.0; }
    }
    if(n == 2 || n == 3){                         // v, w
        const int l = im - 1;
        if(a.top_taper != 0){
            at(l) = (S)0.0;
            if(a.top_taper == 2){
                at(l - 1) = (S)((1.0 / 3.0) * (double)at(l - 3));
                at(l - 2) = (S)((2.0 / 3.0) * (double)at(l - 3));
            } else {
                at(l - 1) = (S)((double)at(l - 1) * (1.0 / 3.0));
                at(l - 2) = (S)((double)at(l - 2) * (2.0 / 3.0));
            }
        }
        if(a.lid_vw == 2)
            at(l) = (S)(2.0 * (double)at(l - 1) - (double)at(l - 2));
        else if(a.lid_vw == 3)
            at(l) = (S)((double)at(l - 3) - 3.0 * (double)at(l - 2) + 3.0 * (double)at(l - 1));
    } else if(species && a.positive != 0){
        if((double)at(0) < 0.0) at(0) = (S)((a.positive == 2) ? post_max0((double)at(1)) : 0.0);
        if((double)at(im - 1) < 0.0) at(im - 1) = (S)((a.positive == 2) ? post_max0((double)at(im - 2)) : 0.0);
    }
}

// ---- bcTheta (BoundaryConditions.h:293-391): one thread per (i, k) column of one field; fields
// 0..POST_NTHZ-1 are zeroed at the poles, the others extrapolated. ----
template <typename S>
__global__ void __launch_bounds__(128) post_bc_theta_kernel(PostArgs<S> a){
    chain_wait();
    const Grid& g = a.g;
    const int k = blockIdx.x * blockDim.x + threadIdx.x, i = blockIdx.y, n = blockIdx.z;
    if(k >= g.km) return;
    const int jm = g.jm;
    const size_t kp = (size_t)g.kp, o = gidx(g, i, 0, k);
    if(n < POST_NTHZ){
        S* F = a.thz[n] + o;
        F[0] = (S)0.0;
        F[(size_t)(jm - 1) * kp] = (S)0.0;
        return;
    }
    S* F = a.thx[n - POST_NTHZ] + o;
    if(n == POST_NTHZ && a.tlo){                    // t as the mixed form's pair
        float* L = a.tlo + o;
        auto get = [&](int j) -> double { return t_ld(F, L, (size_t)j * kp); };
        t_st(F, L, 0, post_form(a.pole_form, get(1), get(2), get(3)));
        t_st(F, L, (size_t)(jm - 1) * kp, post_form(a.pole_form, get(jm - 2), get(jm - 3), get(jm - 4)));
        return;
    }
    auto at = [&](int j) -> S& { return F[(size_t)j * kp]; };
    at(0) = (S)post_form(a.pole_form, (double)at(1), (double)at(2), (double)at(3));     // in order (jm < 5 overlaps)
    at(jm - 1) = (S)post_form(a.pole_form, (double)at(jm - 2), (double)at(jm - 3), (double)at(jm - 4));
}

// ---- bcPhi (BoundaryConditions.h:398-455, without the seam damping): one thread per (i, j) row
// of one field ----
template <typename S>
__global__ void __launch_bounds__(128) post_bc_phi_kernel(PostArgs<S> a){
    chain_wait();
    const Grid& g = a.g;
    const int r = blockIdx.x * blockDim.x + threadIdx.x;      // row (i, j)
    if(r >= g.im * g.jm) return;
    const int km = g.km;
    S* F = a.rad[blockIdx.y] + (size_t)r * g.kp;
    if(blockIdx.y == 0 && a.tlo){                   // t as the mixed form's pair
        float* L = a.tlo + (size_t)r * g.kp;
        if(a.phi_periodic){ F[km - 1] = F[0]; L[km - 1] = L[0]; }
        else {
            const double y = 0.5 * ((C43 * t_ld(F, L, 1) - C13 * t_ld(F, L, 2)) + (C43 * t_ld(F, L, km - 2) - C13 * t_ld(F, L, km - 3)));
            t_st(F, L, 0, y);
            t_st(F, L, km - 1, y);
        }
        return;
    }
    if(a.phi_periodic) F[km - 1] = F[0];
    else {
        const double lo = C43 * (double)F[1] - C13 * (double)F[2];
        const double hi = C43 * (double)F[km - 2] - C13 * (double)F[km - 3];
        const S y = (S)(0.5 * (lo + hi));
        F[0] = y;
        F[km - 1] = y;
    }
}

// ---- clampNegativeSpecies (BC_Uran.h:110-128) ----
// Block (b, n) clamps a block-stride share of species n's padded field, read as 16-byte vectors
// (a vector never straddles a row: the row pitch is a multiple of 32 values), four vectors in
// flight per thread; values in the row padding are skipped. It writes its clipped sum and count
// (as doubles, exact for any count below 2^53) to part[2 (n nb + b)] in a fixed tree order, and
// post_clamp_finish_kernel adds a species' nb partials in a fixed order. Deterministic run to
// run; the reference's OpenMP reduction order differs, so the sum agrees to its rounding.
constexpr int POST_CLAMP_NT = 256;
template <typename S> struct Vec16;
template <> struct Vec16<float>  { using T = float4;  static constexpr int N = 4; };
template <> struct Vec16<double> { using T = double2; static constexpr int N = 2; };

template <typename S>
__device__ __forceinline__ void post_clamp_one(S* R, int k, int km, double x, double& s, double& c){
    if(k < km && !(x >= 0.0)){                     // catches a NaN too
        if(isfinite(x)){ s -= x; c += 1.0; }
        R[k] = (S)0.0;
    }
}

template <typename S>
__global__ void __launch_bounds__(POST_CLAMP_NT) post_clamp_kernel(PostArgs<S> a, double* part){
    chain_wait();
    using V = typename Vec16<S>::T;
    constexpr int NV = Vec16<S>::N, U = 4;
    const Grid& g = a.g;
    const int n = blockIdx.y, nb = gridDim.x;
    S* F = a.sp[n];
    const int vpr = g.kp / NV;                                    // vectors per row
    const long long nvec = (long long)g.im * g.jm * vpr;
    const long long step = (long long)nb * POST_CLAMP_NT;
    double s = 0.0, c = 0.0;
    for(long long q0 = (long long)blockIdx.x * POST_CLAMP_NT + threadIdx.x; q0 < nvec; q0 += U * step){
        V v[U];
#pragma unroll
        for(int u = 0; u < U; u++){
            const long long q = q0 + u * step;
            if(q < nvec) v[u] = reinterpret_cast<const V*>(F)[q];
        }
#pragma unroll
        for(int u = 0; u < U; u++){
            const long long q = q0 + u * step;
            if(q >= nvec) break;
            const long long r = q / vpr;
            const int k0 = (int)(q - r * vpr) * NV;
            S* R = F + r * g.kp;
            const S* e = reinterpret_cast<const S*>(&v[u]);
#pragma unroll
            for(int m = 0; m < NV; m++) post_clamp_one(R, k0 + m, g.km, (double)e[m], s, c);
        }
    }
    __shared__ double ss[POST_CLAMP_NT], sc[POST_CLAMP_NT];
    ss[threadIdx.x] = s; sc[threadIdx.x] = c;
    __syncthreads();
    for(int st = POST_CLAMP_NT / 2; st > 0; st >>= 1){
        if((int)threadIdx.x < st){ ss[threadIdx.x] += ss[threadIdx.x + st]; sc[threadIdx.x] += sc[threadIdx.x + st]; }
        __syncthreads();
    }
    if(threadIdx.x == 0){ part[2 * ((size_t)n * nb + blockIdx.x)] = ss[0]; part[2 * ((size_t)n * nb + blockIdx.x) + 1] = sc[0]; }
}

// One block per species: thread t adds partials t, t + 256, ... in order, then a fixed tree.
static __global__ void __launch_bounds__(POST_CLAMP_NT) post_clamp_finish_kernel(const double* part, int nb, double* out){
    chain_wait();
    const int n = blockIdx.x;
    double s = 0.0, c = 0.0;
    for(int b = threadIdx.x; b < nb; b += POST_CLAMP_NT){ s += part[2 * ((size_t)n * nb + b)]; c += part[2 * ((size_t)n * nb + b) + 1]; }
    __shared__ double ss[POST_CLAMP_NT], sc[POST_CLAMP_NT];
    ss[threadIdx.x] = s; sc[threadIdx.x] = c;
    __syncthreads();
    for(int st = POST_CLAMP_NT / 2; st > 0; st >>= 1){
        if((int)threadIdx.x < st){ ss[threadIdx.x] += ss[threadIdx.x + st]; sc[threadIdx.x] += sc[threadIdx.x + st]; }
        __syncthreads();
    }
    if(threadIdx.x == 0){ out[n] = ss[0]; out[POST_NSP + n] = sc[0]; }
}

}  // namespace aturan
