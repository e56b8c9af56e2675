// fwd_kernel.cu -- B200 forward model + analytic Jacobian of the correlated-k
// thermal-emission path (radtran/cirsradg/cirsradg_wave.f, IMOD 0/1/3) fused
// with map2pro/map2xvec (radtran/cirsradg/map2pro.f, map2xvec.f).
//
// One CTA (8 warps; 16, or several CTAs of a cluster, where SMs would be idle) owns
// one (spectrum, wavenumber) work item at a time and loops over items, grid-stride or
// pulled from a counter (persistent grid, one scratch slot per CTA or cluster).
//   A  per layer (one warp each): k-table interpolation of every gas
//      (get_kg.f:306-378), continuum optical depth and its derivatives
//      (nciacon.f, dust, Rayleigh: cirsradg_wave.f:510-691) and the random
//      overlap of the gas k-distributions (noverlapg.f/rankg.f; overlap.cuh).
//      tau and dtau/dq per g go to the CTA's scratch slot (L2-resident).
//   B  per path (one warp, one lane per g): Planck, transmissions, radiance
//      and dR/dtau of every layer by a suffix sum, which replaces the O(L^2)
//      recurrence of cirsradg_wave.f:954-978 by O(L) exact algebra.
//   C  g-quadrature of the layer Jacobian (cirsradg_wave.f:1240-1286).
//   D  layer -> state vector through a precomputed sparse map
//      (map2pro o map2xvec), packed as cirsrtfg_wave.f:425-446.
//
// Bit-exactness of the g-bin assignment: every operation that feeds a sort
// key or a bin boundary is an explicitly rounded IEEE operation in the
// reference's order (no FMA contraction); the cumulative weights are FP64
// sums of FP32 products >= 2^-28, exact in any order; a pass whose bin
// boundaries fall inside a run of tied keys (where the reference's unstable
// heapsort order decides the bins) takes that heapsort (sort2g.f) in-kernel.
#include <cuda_runtime.h>
#include <stdint.h>

#include "detexp.cuh"
#include "overlap.cuh"
#include "rtb_common.h"

#ifndef FWD_PART
#error "FWD_PART: 0, the host side, or 1 to 13, a part of the instances"
#endif

namespace rtb {

namespace {

// NR heapsort of radtran/cirsradg/sort2g.f:1-52 on shared memory (one thread);
// ra/ib hold RA(1..n)/IB(1..n) at ra[0..n-1].
static __device__ __noinline__ void heapsort_sort2g(int n, float* ra0, unsigned short* ib0) {
    if (n < 2) return;
    float* RA = ra0 - 1;
    unsigned short* IB = ib0 - 1;
    int L = n / 2 + 1, IR = n;
    float RRA;
    unsigned short IRB;
    for (;;) {
        if (L > 1) {
            L = L - 1;
            RRA = RA[L];
            IRB = IB[L];
        } else {
            RRA = RA[IR];
            IRB = IB[IR];
            RA[IR] = RA[1];
            IB[IR] = IB[1];
            IR = IR - 1;
            if (IR == 1) {
                RA[1] = RRA;
                IB[1] = IRB;
                return;
            }
        }
        int I = L, J = L + L;
        while (J <= IR) {
            if (J < IR) {
                if (RA[J] < RA[J + 1]) J = J + 1;
            }
            if (RRA < RA[J]) {
                RA[I] = RA[J];
                IB[I] = IB[J];
                I = J;
                J = J + J;
            } else {
                J = IR + 1;
            }
        }
        RA[I] = RRA;
        IB[I] = IRB;
    }
}

__host__ __device__ inline int align16(int x) { return (x + 15) & ~15; }

// per-path sub-offsets (stages B-D)
struct PathOff {
    int drdt, trd, bb, dbdt, dq, rad, gts, total;
};
__host__ __device__ inline PathOff path_off(int nlmax, int ng, int nsw) {
    PathOff p;
    int o = 0;
    p.drdt = o; o += 4 * nlmax * ng;
    p.trd = o; o += 4 * nlmax * ng;
    p.bb = o; o += 4 * nlmax;
    p.dbdt = o; o += 4 * nlmax;
    p.dq = o; o += 4 * nlmax * (nsw > 0 ? nsw : 1);
    p.rad = o; o += 4 * kMaxNg;
    p.gts = o; o += 4 * kMaxNg;
    p.total = align16(o);
    return p;
}

struct Layout {
    int warp_bytes, path_bytes, off_delg, off_mtab, off_region, total;
};
__host__ __device__ inline Layout make_layout(int ng, int nsw, int ncol, int ngk, int nlmax, int npath, int warps) {
    Layout Lo;
    Lo.warp_bytes = pass_scratch_bytes(ng, ncol, ngk);
    Lo.path_bytes = path_off(nlmax, ng, nsw).total;
    int o = 0;
    Lo.off_delg = o; o += 4 * kMaxNg;
    o = align16(o);
    Lo.off_mtab = o; o += (int)sizeof(MergeLane) * kMergeLevels * 32;
    Lo.off_region = o;
    const int a = warps * Lo.warp_bytes, b = npath * Lo.path_bytes;
    o += a > b ? a : b;
    Lo.total = o;
    return Lo;
}

// RANKK (radtran/cirsradg/rankk.f:34-117) on one thread: REAL cumulative
// ordinates and distribution summed in the reference's order, the `<=` test,
// the split fraction and the ig <= ng guards.  cont/dcont/weight are sorted
// and permuted in place (sort2g heapsort); ico is scratch.
static __device__ void rankk_lane(int ng, const float* gw, int nloop, float* cont, float* dcont, float* weight,
                                        unsigned short* ico, float* tmp, float* k_g, float* dkdt) {
    float g_ord[kMaxNg + 1];
    g_ord[0] = 0.0f;
    for (int i = 0; i < ng; ++i) g_ord[i + 1] = __fadd_rn(g_ord[i], gw[i]);
    if (g_ord[ng] < 1.0f) g_ord[ng] = 1.0f;
    for (int i = 0; i < nloop; ++i) ico[i] = (unsigned short)i;
    heapsort_sort2g(nloop, cont, ico);
    for (int i = 0; i < nloop; ++i) tmp[i] = weight[ico[i]];
    for (int i = 0; i < nloop; ++i) weight[i] = tmp[i];
    for (int i = 0; i < nloop; ++i) tmp[i] = dcont[ico[i]];
    for (int i = 0; i < nloop; ++i) dcont[i] = tmp[i];
    // gdist(I) in tmp[I], I = 0..nloop
    tmp[0] = 0.0f;
    tmp[1] = weight[0];
    for (int i = 2; i <= nloop; ++i) tmp[i] = __fadd_rn(weight[i - 1], tmp[i - 1]);
    for (int i = 0; i < ng; ++i) {
        k_g[i] = 0.0f;
        dkdt[i] = 0.0f;
    }
    int ig = 1;
    float sum = 0.0f;
    for (int I = 1; I <= nloop; ++I) {
        const float c = cont[I - 1], dc = dcont[I - 1], w = weight[I - 1];
        if (ig <= ng && tmp[I] <= g_ord[ig]) {
            k_g[ig - 1] = __fadd_rn(k_g[ig - 1], __fmul_rn(c, w));
            dkdt[ig - 1] = __fadd_rn(dkdt[ig - 1], __fmul_rn(dc, w));
            sum = __fadd_rn(sum, w);
        } else {
            if (ig > ng) continue;      // the reference writes past NG here; those slots are never read
            const float frac = __fdiv_rn(__fsub_rn(g_ord[ig], tmp[I - 1]), __fsub_rn(tmp[I], tmp[I - 1]));
            k_g[ig - 1] = __fadd_rn(k_g[ig - 1], __fmul_rn(__fmul_rn(frac, c), w));
            dkdt[ig - 1] = __fadd_rn(dkdt[ig - 1], __fmul_rn(__fmul_rn(frac, dc), w));
            sum = __fadd_rn(sum, __fmul_rn(frac, w));
            k_g[ig - 1] = __fdiv_rn(k_g[ig - 1], sum);
            dkdt[ig - 1] = __fdiv_rn(dkdt[ig - 1], sum);
            ig = ig + 1;
            if (ig <= ng) {
                const float rest = __fsub_rn(1.0f, frac);
                sum = __fmul_rn(rest, w);
                k_g[ig - 1] = __fmul_rn(__fmul_rn(rest, c), w);
                dkdt[ig - 1] = __fmul_rn(__fmul_rn(rest, dc), w);
            }
        }
    }
    if (ig == ng) {
        k_g[ig - 1] = __fdiv_rn(k_g[ig - 1], sum);
        dkdt[ig - 1] = __fdiv_rn(dkdt[ig - 1], sum);
    }
}

// a layer's place in the (P, T) grid of the tables, as get_kg takes it
struct KgPos {
    int ioff[4];
    float u, v, dudt, u2, dudt2;
};
template <bool t2>
__device__ __forceinline__ KgPos kg_pos(const LayerDev& L) {
    const int4 o = __ldg((const int4*)L.ioff);
    const float4 w = __ldg((const float4*)&L.u);
    return KgPos{{o.x, o.y, o.z, o.w}, w.x, w.y, w.z, t2 ? L.u2 : 0.0f, t2 ? L.dudt2 : 0.0f};
}

// X and dX/dT of the four (P, T) corners of one g (get_kg.f:355-365 and
// 413-423): bilinear in (ln p, T) for a table with one temperature grid; for
// TEMP2 tables (NT < 0) linear in T along each pressure row with its own
// weight, then linear in ln p
template <bool t2>
__device__ __forceinline__ void corners(const KgPos& L, float Y1, float Y2, float Y3, float Y4, float& X,
                                        float& DXDT) {
    const float U = L.u, V = L.v;
    const float a = __fsub_rn(1.0f, V), b = __fsub_rn(1.0f, U);
    if (t2) {
        const float X1 = __fadd_rn(__fmul_rn(b, Y1), __fmul_rn(U, Y4));
        const float X2 = __fadd_rn(__fmul_rn(__fsub_rn(1.0f, L.u2), Y2), __fmul_rn(L.u2, Y3));
        X = __fadd_rn(__fmul_rn(a, X1), __fmul_rn(V, X2));
        DXDT = __fadd_rn(__fmul_rn(__fmul_rn(a, __fadd_rn(-Y1, Y4)), L.dudt),
                         __fmul_rn(__fmul_rn(V, __fadd_rn(-Y2, Y3)), L.dudt2));
        return;
    }
    X = __fmul_rn(__fmul_rn(a, b), Y1);
    X = __fadd_rn(X, __fmul_rn(__fmul_rn(V, b), Y2));
    X = __fadd_rn(X, __fmul_rn(__fmul_rn(V, U), Y3));
    X = __fadd_rn(X, __fmul_rn(__fmul_rn(a, U), Y4));
    float D = -__fmul_rn(a, Y1);
    D = __fsub_rn(D, __fmul_rn(V, Y2));
    D = __fadd_rn(D, __fmul_rn(V, Y3));
    D = __fadd_rn(D, __fmul_rn(a, Y4));
    DXDT = __fmul_rn(D, L.dudt);
}

// linear interpolation of one g of one table slice (no logarithms: the
// non-coincident branch of get_kg.f:396-420)
template <bool t2>
__device__ __forceinline__ void interp_lin(const float* t, const KgPos& L, int g, float& X, float& DXDT) {
    const float Y1 = __ldg(t + L.ioff[0] + g), Y2 = __ldg(t + L.ioff[1] + g);
    const float Y3 = __ldg(t + L.ioff[2] + g), Y4 = __ldg(t + L.ioff[3] + g);
    corners<t2>(L, Y1, Y2, Y3, Y4, X, DXDT);
}

// get_kg for a wavenumber between two table points (get_kg.f:380-438):
// 2 NG linearly interpolated values, weighted (1 - w2) delg and w2 delg,
// rank-rebinned by rankk on lane 0.  scr: per-warp shared scratch (RankkOff).
// Called by the whole warp.
template <bool t2>
__device__ void get_kg_lane_nc(const BatchDev& B, int64_t slice, float w1, float w2, const KgPos& L, int lane,
                               float* scr,
                               float& k, float& dk) {
    const int ng = B.ng;
    using Off = RankkOff;
    float *cont = scr + Off::cont, *dcont = scr + Off::dcont, *fac = scr + Off::fac, *tmp = scr + Off::tmp;
    float *kg = scr + Off::kg, *dkg = scr + Off::dkg;
    unsigned short* ico = (unsigned short*)(scr + Off::ico);
    k = 0.0f;
    dk = 0.0f;
    if (slice < 0) return;
    if (lane < ng) {
        const int64_t step = (int64_t)B.np * B.nt * ng;
        for (int loop = 0; loop < 2; ++loop) {
            float X, D;
            interp_lin<t2>(B.ktab_raw + slice + loop * step, L, lane, X, D);
            cont[loop * ng + lane] = X;
            dcont[loop * ng + lane] = D;
            fac[loop * ng + lane] = __fmul_rn(B.delg[lane], loop ? w2 : w1);
        }
    }
    __syncwarp();
    if (lane == 0) rankk_lane(ng, B.delg, 2 * ng, cont, dcont, fac, ico, tmp, kg, dkg);
    __syncwarp();
    if (lane < ng) {
        k = kg[lane];
        dk = dkg[lane];
        if (k != k) k = 1e-37f;
        if (dk != dk) dk = 1e-37f;
    }
    __syncwarp();
}

// get_kg for one g-ordinate of one gas at one layer (get_kg.f:320-378
// coincident branch, NaN -> 1e-37 at :443-471)
template <bool t2>
__device__ __forceinline__ void get_kg_g(const BatchDev& B, int64_t slice, const KgPos& L, int g, float& k, float& dk) {
    bool klog = (slice & kSliceLog) != 0;
    slice &= ~kSliceLog;
    if (!klog) {
        const float* raw = B.ktab_raw + slice;
        const float y10 = __ldg(raw + L.ioff[0]), y20 = __ldg(raw + L.ioff[1]);
        const float y30 = __ldg(raw + L.ioff[2]), y40 = __ldg(raw + L.ioff[3]);
        klog = !((y10 <= 0.0f) || (y20 <= 0.0f) || (y30 <= 0.0f) || (y40 <= 0.0f));
    }
    const float* t = (klog ? B.ktab_log : B.ktab_raw) + slice + g;
    const float Y1 = __ldg(t + L.ioff[0]), Y2 = __ldg(t + L.ioff[1]);
    const float Y3 = __ldg(t + L.ioff[2]), Y4 = __ldg(t + L.ioff[3]);
    float X, DXDT;
    corners<t2>(L, Y1, Y2, Y3, Y4, X, DXDT);
    if (klog) {
        const float e = det_expf(X);
        k = e;
        dk = __fmul_rn(e, DXDT);
    } else {
        k = X;
        dk = DXDT;
    }
    if (k != k) k = 1e-37f;
    if (dk != dk) dk = 1e-37f;
}

// E3INTERP (radtran/radtran/e3interp.f:42-75) on the table tabtran | tabe3 |
// egrad (1001 points each): E3 and dE3/dtrans of a transmission, DOUBLE
__device__ __forceinline__ void e3interp_dev(const double* tab, double x, double& e3, double& de3) {
    constexpr int mtab = 1001;
    if (x < 0.0 || x != x) {
        e3 = 0.0;
        de3 = 0.0;
        return;
    }
    const double dtrans = (double)(1.0f / 1000.0f);
    int j = 1 + (int)(x / dtrans);
    if (j >= mtab) j = mtab - 1;
    double f = (x - tab[j - 1]) / dtrans;
    if (f > 1.0) f = 1.0;
    const double* te3 = tab + mtab;
    const double* eg = tab + 2 * mtab;
    e3 = __dadd_rn(__dmul_rn(1.0 - f, te3[j - 1]), __dmul_rn(f, te3[j]));
    de3 = __dadd_rn(__dmul_rn(1.0 - f, eg[j - 1]), __dmul_rn(f, eg[j]));
}

// calc_nlte_t.f:1-45, the emission temperature of a layer at pressure p (atm)
// outside LTE: B(T_nlte) = f B(T) with f = k1 N / (A + k1 N), N the number
// density (inlte = 1), or f = 1e6 p / (1 + 1e6 p) (inlte = 2).  Its IWAVE is
// the wavenumber index in cirsradg_wave.f:933-935, never 0, so planck_wave
// and invplanck_wave take their wavelength branch (y = 1e4 / v) there.
// DOUBLE inside as those two are; REAL factors as calc_nlte_t forms them.
static __device__ __noinline__ float nlte_temp(int inlte, float T, float p, float v, float k1, float A) {
    float f;
    if (inlte == 1) {
        const float ntot = __fmul_rn(__fdiv_rn(__fmul_rn(p, 101325.0f), __fmul_rn(1.380658e-23f, T)), 1.0e-6f);
        f = __fdiv_rn(__fmul_rn(k1, ntot), __fadd_rn(A, __fmul_rn(k1, ntot)));
    } else if (inlte == 2) {
        const float x = __fmul_rn(p, 1.0e6f);
        f = __fdiv_rn(x, __fadd_rn(1.0f, x));
    } else {
        return T;
    }
    const double c1 = (double)1.1911e-12f, c2 = (double)1.439f;
    const float y = __fdiv_rn(1e4f, v);
    if (y == 0.0f) return 0.0f;                  // planck_wave = 0, then invplanck_wave(B = 0) = 0
    const float y2 = __fmul_rn(y, y), y4 = __fmul_rn(y2, y2);
    const double a = c1 * (double)__fmul_rn(y4, y) / 1e4;
    const float Bt = __double2float_rn(a / (exp(c2 * (double)y / (double)T) - 1.0));
    const float Bf = __fmul_rn(Bt, f);
    if (Bf == 0.0f || v == 0.0f) return 0.0f;
    const double dv = (double)v, v2 = dv * dv, v4 = v2 * v2;
    return __double2float_rn(c2 * (double)1.0e4f / dv / log((c1 * (double)1.0e16f) / ((double)Bf * (v4 * dv)) + 1.0));
}

// iform = 3 on an IMOD 3 path (cirsradg_wave.f:913-929): the total flux of the
// planet, every term of lane g's radiance and derivatives times x.  Out of
// line, as is path_imod18: the common paths' code stays as compact as it was.
static __device__ __noinline__ void scale_path(float x, int nlays, int ng, int g, float* drdt, float* trd, float* rad,
                                        float* gts) {
    rad[g] *= x;
    gts[g] *= x;
    for (int j = 0; j < nlays; ++j) {
        drdt[j * ng + g] *= x;
        trd[j * ng + g] *= x;
    }
}

// IMOD 18, hemispherically integrated emission (cirsradg_wave.f:1116-1225), on
// g-ordinate g of one path:
// R = c sum_j B_j (E3(T_{j-1}) - E3(T_j)) + c E3(T_N) e_s B_s with the vertical
// transmissions T_j in DOUBLE and E3 from e3interp's table, c = 2 pi xfac;
// dR/dtau_j = c (B_j G_j + sum_{m>j} B_m (G_m - G_{m-1})), G_m = E3'(T_m) T_m
// (the reference leaves the surface term out of the derivative).  drdt
// receives dR/dtau_j, trd the factor of dB/dT in the temperature column.
static __device__ __noinline__ void path_imod18(const double* e3tab, float xfac18, int nlays, int ng, int g,
                                         const int* layinc, const float* scale, const float* tau_s,
                                         const float* bb, float radground_s, float gradground_s, float* drdt,
                                         float* trd, float* rad, float* gts) {
    const float c = __fmul_rn(__fmul_rn(xfac18, 2.0f), 3.1415927f);
    double tr = 1.0, e3o = 0.5;
    float R = 0.0f;
    for (int j = 0; j < nlays; ++j) {
        const float tau = tau_s[layinc[j] * ng + g] * scale[j];
        tr = tr * exp(-(double)tau);
        double e3n, e3g;
        e3interp_dev(e3tab, tr, e3n, e3g);
        const float d = __double2float_rn(e3o - e3n);
        R = __fadd_rn(R, __fmul_rn(__fmul_rn(c, d), bb[j]));
        trd[j * ng + g] = __fmul_rn(c, d);
        drdt[j * ng + g] = __double2float_rn(e3g) * __double2float_rn(tr);   // G_j
        e3o = e3n;
    }
    const float e3l = __double2float_rn(e3o);
    R = __fadd_rn(R, __fmul_rn(__fmul_rn(c, e3l), radground_s));
    float Ssum = 0.0f;
    for (int j = nlays - 1; j >= 0; --j) {
        const float Gj = drdt[j * ng + g];
        drdt[j * ng + g] = c * fmaf(bb[j], Gj, Ssum);
        if (j > 0) Ssum = fmaf(bb[j], Gj - drdt[(j - 1) * ng + g], Ssum);
    }
    rad[g] = R;
    gts[g] = __fmul_rn(__fmul_rn(c, e3l), gradground_s);
}

// bilinear (wavenumber, temperature) value of one CIA table entry and its
// d/dT (ciaread.f:178-196, fpread_all.f:220-266): REAL, in the reference's
// order; the four corners are at b + stride * (ct + 25 cv) and neighbours
__device__ __forceinline__ void cia_bilinear(const float* kc, int64_t e, int64_t stride, int ct, int cv, float t,
                                             float u, float dudt, float& x, float& dx) {
    const float omt = __fsub_rn(1.0f, t), omu = __fsub_rn(1.0f, u);
    const float a11 = __ldg(kc + e + stride * ((int64_t)ct + 25 * (int64_t)cv));
    const float a12 = __ldg(kc + e + stride * ((int64_t)ct + 25 * ((int64_t)cv + 1)));
    const float a22 = __ldg(kc + e + stride * ((int64_t)ct + 1 + 25 * ((int64_t)cv + 1)));
    const float a21 = __ldg(kc + e + stride * ((int64_t)ct + 1 + 25 * (int64_t)cv));
    x = __fmul_rn(__fmul_rn(omt, omu), a11);
    x = __fadd_rn(x, __fmul_rn(__fmul_rn(t, omu), a12));
    x = __fadd_rn(x, __fmul_rn(__fmul_rn(t, u), a22));
    x = __fadd_rn(x, __fmul_rn(__fmul_rn(omt, u), a21));
    float d = -__fmul_rn(omt, a11);
    d = __fsub_rn(d, __fmul_rn(t, a12));
    d = __fadd_rn(d, __fmul_rn(t, a22));
    d = __fadd_rn(d, __fmul_rn(omt, a21));
    dx = __fmul_rn(d, dudt);
}

// RAYLEIGHA (radtran/scatter/rayleigha.f:1-38): the Rayleigh cross section of
// air at pressure P (atm) and temperature T, REAL arithmetic in its order
static __device__ __noinline__ float rayleigha_dev(float v, float P, float T) {
    const float c1 = 8342.12f, c2 = 2406030.0f, c3 = 15997.0f, delta = 0.035f, pi = 3.1415927f, k = 1.37971e-23f;
    float lambda = __fdiv_rn(1e4f, v);
    const float nu2 = __fdiv_rn(1.0f, __fmul_rn(lambda, lambda));
    float m1 = __fadd_rn(__fadd_rn(c1, __fdiv_rn(c2, __fsub_rn(130.0f, nu2))), __fdiv_rn(c3, __fsub_rn(38.9f, nu2)));
    m1 = __fmul_rn(m1, 1e-8f);
    const float P1 = __fmul_rn(P, 1.013e5f), T1 = __fsub_rn(T, 273.15f);
    const float num = __fmul_rn(P1, __fadd_rn(1.0f, __fmul_rn(__fmul_rn(P1, __fsub_rn(61.3f, T1)), 1E-10f)));
    const float xcorr = __fdiv_rn(num, __fmul_rn(96095.4f, __fadd_rn(1.0f, __fmul_rn(0.003661f, T1))));
    m1 = __fmul_rn(m1, xcorr);
    const float Ns = __fdiv_rn(P1, __fmul_rn(k, T));
    lambda = __fmul_rn(lambda, 1e-6f);
    const float x = __fmul_rn(__fmul_rn(Ns, lambda), lambda);
    const float mm = __fmul_rn(m1, __fadd_rn(m1, 2.0f));
    const float temp = __fmul_rn(__fmul_rn(8.0f, __fmul_rn(__fmul_rn(pi, pi), pi)), __fmul_rn(mm, mm));
    const float faniso = __fdiv_rn(__fadd_rn(6.0f, __fmul_rn(3.0f, delta)), __fsub_rn(6.0f, __fmul_rn(7.0f, delta)));
    return __fdiv_rn(__fmul_rn(__fmul_rn(temp, 1e4f), faniso), __fmul_rn(3.0f, __fmul_rn(x, x)));
}

// continuum optical depth of one layer and its active derivatives
// (cirsradg_wave.f:526-691 with nciacon.f:84-310 / ciaread.f:108-198, or for
// flagh2p = 1 nparacon_all.f:160-336 / fpread_all.f:195-266).  Lanes 0..8
// interpolate one CIA table entry each; the sums run on every lane.  Lane s
// takes the derivative with active parameter s (dtc).
template <bool para>
__device__ __forceinline__ float continuum(const BatchDev& B, const SpecDev& S, const LayerDev& L, const WaveDev& W,
                                           int64_t iw_glob, int64_t il_glob, int lane, float& dtc) {
    const int mine = lane < S.nsw ? S.isw[lane] : -1;   // this lane's parameter
    dtc = 0.0f;
    float taucon = 0.0f;
    for (int k = 0; k < S.ncont; ++k) {
        // this spectrum's [nwave][ncont] and [nlayer][ncont] blocks: the
        // batch's spectra need not share ncont
        const float tau = B.xsec[S.wc_off + (iw_glob - S.wave_off) * S.ncont + k];
        taucon = __fadd_rn(taucon, __fmul_rn(tau, B.cont[S.lc_off + (il_glob - S.lay_off) * S.ncont + k]));
        if (mine == S.ngas + 1 + k) dtc = tau;
    }
    float absorb = 0.0f, dab[7] = {0, 0, 0, 0, 0, 0, 0};
    if (para && S.para) {
        // lanes 0, 1: H2-H2 at the para entries j0, j0+1; 2, 3: H2-He; 4..8: the
        // five further pairs of kcia5
        const ParaLayDev PL = B.para_lay[S.para_off + (il_glob - S.lay_off)];
        const ParaWaveDev PW = B.para_wave[S.paraw_off + (iw_glob - S.wave_off)];
        float my_a = 0.0f, my_d = 0.0f;
        if (lane < 9) {
            if (lane < 4) {
                const int e = PL.j0 + ((lane & 1) && !PL.neg ? 1 : 0);
                cia_bilinear(lane < 2 ? B.kh2h2 : B.kh2he, e, B.ipara, PL.ct, PW.cv, PW.t, PL.u, PL.dudt, my_a, my_d);
            } else {
                cia_bilinear(B.kcia5, lane - 4, 5, PL.ct, PW.cv, PW.t, PL.u, PL.dudt, my_a, my_d);
            }
        }
        auto v = [&](int p) { return __shfl_sync(kFull, my_a, p); };
        auto dv = [&](int p) { return __shfl_sync(kFull, my_d, p); };
        float ah2h2, ah2he, dh2dt, dhedt, dh2dfp = 0.0f, dhedfp = 0.0f;
        if (PL.neg) {
            ah2h2 = v(0);
            ah2he = v(2);
            dh2dt = dv(0);
            dhedt = dv(2);
        } else {
            const float f = PL.f, omf = __fsub_rn(1.0f, PL.f);
            ah2h2 = __fadd_rn(__fmul_rn(omf, v(0)), __fmul_rn(f, v(1)));
            ah2he = __fadd_rn(__fmul_rn(omf, v(2)), __fmul_rn(f, v(3)));
            dh2dt = __fadd_rn(__fmul_rn(omf, dv(0)), __fmul_rn(f, dv(1)));
            dhedt = __fadd_rn(__fmul_rn(omf, dv(2)), __fmul_rn(f, dv(3)));
            dh2dfp = __fdiv_rn(__fsub_rn(v(1), v(0)), B.para_deltaf);
            dhedfp = __fdiv_rn(__fsub_rn(v(3), v(2)), B.para_deltaf);
        }
        const float qh2 = L.q[0], qhe = L.q[1], qn2 = L.q[2], qch4 = L.q[3], qco2 = L.q[4];
        float sum = __fadd_rn(__fmul_rn(__fmul_rn(ah2h2, qh2), qh2), __fmul_rn(__fmul_rn(ah2he, qh2), qhe));
        dab[0] = __fadd_rn(__fmul_rn(__fmul_rn(2.0f, qh2), ah2h2), __fmul_rn(qhe, ah2he));
        dab[1] = __fmul_rn(qh2, ah2he);
        dab[5] = __fadd_rn(__fmul_rn(__fmul_rn(dh2dt, qh2), qh2), __fmul_rn(__fmul_rn(dhedt, qh2), qhe));
        dab[6] = __fadd_rn(__fmul_rn(__fmul_rn(dh2dfp, qh2), qh2), __fmul_rn(__fmul_rn(dhedfp, qh2), qhe));
        // H2-N2, N2-CH4, N2-N2, CH4-CH4, H2-CH4 (nparacon_all.f:262-318)
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(v(4), qh2), qn2));
        dab[0] = __fadd_rn(dab[0], __fmul_rn(qn2, v(4)));
        dab[2] = __fadd_rn(dab[2], __fmul_rn(qh2, v(4)));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qh2, qn2), dv(4)));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(v(5), qn2), qch4));
        dab[2] = __fadd_rn(dab[2], __fmul_rn(qch4, v(5)));
        dab[3] = __fadd_rn(dab[3], __fmul_rn(qn2, v(5)));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qn2, qch4), dv(5)));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(v(6), qn2), qn2));
        dab[2] = __fadd_rn(dab[2], __fmul_rn(__fmul_rn(2.0f, qn2), v(6)));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qn2, qn2), dv(6)));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(v(7), qch4), qch4));
        dab[3] = __fadd_rn(dab[3], __fmul_rn(__fmul_rn(2.0f, qch4), v(7)));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qch4, qch4), dv(7)));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(v(8), qh2), qch4));
        dab[0] = __fadd_rn(dab[0], __fmul_rn(qch4, v(8)));
        dab[3] = __fadd_rn(dab[3], __fmul_rn(qh2, v(8)));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qh2, qch4), dv(8)));
        // co2cia / n2n2cia / n2h2cia are zero below 3900 cm-1 (host-checked)
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(0.0f, qco2), qco2));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(0.0f, qn2), qn2));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(0.0f, qn2), qh2));
        absorb = __fmul_rn(sum, L.cia_tau);
#pragma unroll
        for (int i = 0; i < 7; ++i) dab[i] = __fmul_rn(dab[i], L.cia_tau);
    } else if (S.has_cia) {
        float my_a = 0.0f, my_d = 0.0f;
        if (W.cia_cv >= 0 && lane < 9) {
            const int p = lane;
            const float t = W.cia_t, u = L.cia_u;
            const float omt = __fsub_rn(1.0f, t), omu = __fsub_rn(1.0f, u);
            const float* kc = B.kcia;
            const int64_t b11 = 9 * ((int64_t)L.cia_ct + 25 * (int64_t)W.cia_cv);
            const int64_t b12 = 9 * ((int64_t)L.cia_ct + 25 * ((int64_t)W.cia_cv + 1));
            const int64_t b22 = 9 * ((int64_t)L.cia_ct + 1 + 25 * ((int64_t)W.cia_cv + 1));
            const int64_t b21 = 9 * ((int64_t)L.cia_ct + 1 + 25 * (int64_t)W.cia_cv);
            const float a11 = __ldg(kc + b11 + p), a12 = __ldg(kc + b12 + p);
            const float a22 = __ldg(kc + b22 + p), a21 = __ldg(kc + b21 + p);
            float x = __fmul_rn(__fmul_rn(omt, omu), a11);
            x = __fadd_rn(x, __fmul_rn(__fmul_rn(t, omu), a12));
            x = __fadd_rn(x, __fmul_rn(__fmul_rn(t, u), a22));
            x = __fadd_rn(x, __fmul_rn(__fmul_rn(omt, u), a21));
            float d = -__fmul_rn(omt, a11);
            d = __fsub_rn(d, __fmul_rn(t, a12));
            d = __fadd_rn(d, __fmul_rn(t, a22));
            d = __fadd_rn(d, __fmul_rn(omt, a21));
            my_a = x;
            my_d = __fmul_rn(d, L.cia_dudt);
        }
        // pair p's coefficient and its d/dT, from the lane that interpolated it
        auto alpha = [&](int p) { return __shfl_sync(kFull, my_a, p); };
        auto da = [&](int p) { return __shfl_sync(kFull, my_d, p); };
        const float qh2 = L.q[0], qhe = L.q[1], qn2 = L.q[2], qch4 = L.q[3], qco2 = L.q[4];
        float sum = 0.0f;
        const int eq = S.inormal == 0 ? 0 : 2;
        const float ao = alpha(eq), ao1 = alpha(eq + 1), dao = da(eq), dao1 = da(eq + 1);
        sum = __fadd_rn(__fadd_rn(sum, __fmul_rn(__fmul_rn(ao, qh2), qh2)), __fmul_rn(__fmul_rn(ao1, qh2), qhe));
        dab[0] = __fadd_rn(__fadd_rn(dab[0], __fmul_rn(__fmul_rn(2.0f, qh2), ao)), __fmul_rn(qhe, ao1));
        dab[1] = __fadd_rn(dab[1], __fmul_rn(qh2, ao1));
        dab[5] = __fadd_rn(__fadd_rn(dab[5], __fmul_rn(__fmul_rn(qh2, qh2), dao)), __fmul_rn(__fmul_rn(qh2, qhe), dao1));
        float al = alpha(4), d = da(4);          // H2-N2
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(al, qh2), qn2));
        dab[0] = __fadd_rn(dab[0], __fmul_rn(qn2, al));
        dab[2] = __fadd_rn(dab[2], __fmul_rn(qh2, al));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qh2, qn2), d));
        al = alpha(5), d = da(5);                // N2-CH4
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(al, qn2), qch4));
        dab[2] = __fadd_rn(dab[2], __fmul_rn(qch4, al));
        dab[3] = __fadd_rn(dab[3], __fmul_rn(qn2, al));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qn2, qch4), d));
        al = alpha(6), d = da(6);                // N2-N2
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(al, qn2), qn2));
        dab[2] = __fadd_rn(dab[2], __fmul_rn(__fmul_rn(2.0f, qn2), al));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qn2, qn2), d));
        al = alpha(7), d = da(7);                // CH4-CH4
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(al, qch4), qch4));
        dab[3] = __fadd_rn(dab[3], __fmul_rn(__fmul_rn(2.0f, qch4), al));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qch4, qch4), d));
        al = alpha(8), d = da(8);                // H2-CH4
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(al, qh2), qch4));
        dab[0] = __fadd_rn(dab[0], __fmul_rn(qch4, al));
        dab[3] = __fadd_rn(dab[3], __fmul_rn(qh2, al));
        dab[5] = __fadd_rn(dab[5], __fmul_rn(__fmul_rn(qh2, qch4), d));
        // co2cia / n2n2cia / n2h2cia are zero below 3900 cm-1 (host-checked)
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(0.0f, qco2), qco2));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(0.0f, qn2), qn2));
        sum = __fadd_rn(sum, __fmul_rn(__fmul_rn(0.0f, qn2), qh2));
        absorb = __fmul_rn(sum, L.cia_tau);
#pragma unroll
        for (int i = 0; i < 7; ++i) dab[i] = __fmul_rn(dab[i], L.cia_tau);
    }
    taucon = __fadd_rn(taucon, absorb);
    const float den = __fmul_rn(L.utotl, 1.0e20f);
    float dmine = 0.0f;                        // the CIA derivative with this lane's gas, if it has one
    bool cia_gas = false;
#pragma unroll
    for (int ii = 0; ii < 5; ++ii)
        if (mine >= 0 && L.iabs[ii] == mine) {
            dmine = dab[ii];
            cia_gas = true;
        }
    if (cia_gas) dtc = __fadd_rn(dtc, __fdiv_rn(dmine, den));
    if (lane == S.sw_T) dtc = __fadd_rn(dtc, dab[5]);
    if (para && lane == S.sw_para) dtc = __fadd_rn(dtc, dab[6]);   // the para-H2 fraction (cirsradg_wave.f:659-661)
    if (S.iray) {
        float xr = W.xray;
        if (para && S.iray == 3) {   // air: rayleigha at this layer's P and T (cirsradg_wave.f:668-669)
            const int64_t l = il_glob - S.lay_off;
            const float vv = S.ispace ? __fdiv_rn(1e4f, W.vwave) : W.vwave;
            xr = __fmul_rn(rayleigha_dev(vv, B.lay_press[S.lp_off + l], B.lay_temp[S.lt_off + l]), 1E20f);
        }
        const float av = __fmul_rn(L.utotl, xr);
        taucon = __fadd_rn(taucon, av);
        if (mine >= 0 && mine < S.ngas) dtc = __fadd_rn(dtc, __fmul_rn(xr, 1.0e-20f));
    }
    return taucon;
}

// Planck function and its temperature derivative in FP32
// (planck_wave.f / planckg_wave.f; c1, c2 as the reference's REAL literals).
__device__ __forceinline__ void planck_fp32(int ispace, float vwave, float T, float& B, float& dBdT) {
    const float c1 = 1.1911e-12f, c2 = 1.439f;
    float y, a;
    if (ispace == 0) { y = vwave; a = c1 * y * y * y; }
    else { y = 1e4f / vwave; a = c1 * y * y * y * y * y / 1e4f; }
    if (y == 0.0f) { B = 0.0f; dBdT = 0.0f; return; }
    const float x = c2 * y / T;
    const float em1 = expm1f(x);
    B = a / em1;
    dBdT = B * (x / T) * ((em1 + 1.0f) / em1);
}

}  // namespace

// all threads of the cluster, with the global memory they wrote before visible to all after
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}

// ---------------------------------------------------------------------------
// t2: the run's k-tables carry one temperature grid per pressure (NT < 0);
// ext: some spectrum takes the para-H2 CIA (flagh2p = 1), an IMOD 18 path or
// iform = 3.  Template arguments, so that the usual kernel carries no trace
// of either.  WARPS: warps per CTA, the layers of one (spectrum, wavenumber)
// item worked on at once -- the tile shape the autotuner chooses.  CL = 2: two CTAs
// of a cluster share an item's layers (the wide tile: B.cluster of them).  The
// residency bound keeps 24 warps per SM at 80 registers: the passes wait on
// shuffles and fixed-latency chains, and 16 warps at 128 registers take 3.83 ms
// where 24 take 3.27 ms (120 layers, 20-point tables, 4 absorbers, 2000
// wavenumbers; 60 layers, 10-point tables, 4 absorbers, 1400 wavenumbers 0.78 and
// 0.71 ms, though 73 layers, 3 absorbers, 515 wavenumbers 0.26 and 0.27).  NGC > 0:
// NG as a compile-time constant (the overlap's sizes, offsets and loop bounds
// fold); otherwise NG is read at run time, and -4 or -8 sort the elements of a
// pass in that many registers per lane, 0 by merging rows
template <bool t2, bool ext, int WARPS, int NGC, int CL = 1>
__global__ void __launch_bounds__(WARPS * 32, WARPS <= 8 ? 24 / WARPS : 1)
fwd_kernel(BatchDev B, int nsw_max, int ncol_max, int ngk_max, int nlmax_max, int npath_max) {
    constexpr int kThreads = WARPS * 32;
    extern __shared__ __align__(16) char smem[];
    __shared__ SpecDev S_sh;
    const Layout Lo = make_layout(B.ng, nsw_max, ncol_max, ngk_max, nlmax_max, npath_max, WARPS);
    const PathOff po = path_off(nlmax_max, B.ng, nsw_max);
    float* delg = (float*)(smem + Lo.off_delg);
    char* region = smem + Lo.off_region;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    constexpr int NG = NGC > 0 ? NGC : 0;
    // the wide tile, whose calls wait on latency, sorts in registers at any NG: 2700
    // cycles a sort of 400 on one warp, the merge 8100
    constexpr int E = NGC < 0 ? -NGC : WARPS > kTileDefault || CL > 1 ? 16 : 0;
    const int ng = NG ? NG : B.ng;     // NGC > 0: the instance for NG = NGC (== B.ng)
    // per-CTA scratch slot in global memory (L2-resident): tau[l][g], dtau[l][s][g]
    // and per cluster, where several blocks share an item
    const int csize = WARPS > kTileDefault ? B.cluster : CL, crank = csize > 1 ? (int)(blockIdx.x % csize) : 0;
    auto slot = [&]() { return B.cell_scratch + (int64_t)(blockIdx.x / csize) * B.cell_slot; };
    auto slot_dtau = [&]() { return slot() + (int64_t)B.cell_Lmax * ng; };
    for (int i = tid; i < ng; i += kThreads) delg[i] = B.delg[i];
    const float dg = lane < ng ? B.delg[lane] : 0.0f;                // this lane's g-ordinate weight
    const double gb = lane < ng ? B.g_ord[lane + 1] : 0.0;          // and upper bin boundary
    MergeLane* mtab = (MergeLane*)(smem + Lo.off_mtab);
    if (E == 0)
        for (int i = tid; i < kMergeLevels * 32; i += kThreads) ((uint4*)mtab)[i] = ((const uint4*)B.merge_table)[i];
    __shared__ unsigned long long s_count[5];
    if (tid < 5) s_count[tid] = 0;
    __syncthreads();

    char* wsm = region + warp * Lo.warp_bytes;
    PassScratch ps;
    ps.gd = (double*)wsm;
    ps.rec = (uint2*)(wsm + pass_gd_bytes(ng));
    ps.mtab = mtab;
    ps.kg = (float2*)(wsm + pass_kg_offset(ng));
    ps.col = (float*)(ps.kg + ngk_max * ng);

    __shared__ int s_next;
    __shared__ int s_layer;
    __shared__ int64_t s_slice[kMaxGasDev];
    __shared__ unsigned char s_gas[kMaxGasDev];
    __shared__ unsigned s_gmask;
    int k_static = blockIdx.x / csize;      // items are numbered in 32 bits (item_order)
    for (;;) {
        // next work item: grid-stride, or pulled from the launch's counter
        // (dynamic schedule); item_order maps the issue order to items
        int k;
        if (B.work_next) {
            if (tid == 0) s_next = (int)atomicAdd(B.work_next, 1ull);
            __syncthreads();
            k = s_next;
        } else {
            k = k_static;
            k_static += gridDim.x / csize;
        }
        if (k >= B.nitems) break;
        const int item = B.item_order ? B.item_order[k] : k;
        // locate the spectrum of this item
        int lo = 0, hi = B.nspec - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (B.item_start[mid] <= item) lo = mid; else hi = mid - 1;
        }
        const int sidx = lo;
        {
            const int* src = (const int*)(B.spec + sidx);
            int* dst = (int*)&S_sh;
            for (int i = tid; i < (int)(sizeof(SpecDev) / sizeof(int)); i += kThreads) dst[i] = src[i];
            if (tid == 0) s_layer = WARPS;
        }
        __syncthreads();
        const SpecDev& S = S_sh;
        const int iw = (int)(item - B.item_start[sidx]);

        // the gases with a table at this wavenumber
        if (warp == 0) {
            const int64_t sl = lane < S.ngas ? B.wg_slice[S.wg_off + (int64_t)iw * S.ngas + lane] : -1;
            const unsigned m = __ballot_sync(kFull, sl >= 0);
            if (sl >= 0) {
                const int r = __popc(m & ((1u << lane) - 1u));
                s_slice[r] = sl;
                s_gas[r] = (unsigned char)lane;
            }
            if (lane == 0) s_gmask = m;
        }
        __syncthreads();
        // ---------------- stage A0: non-coincident gases -----------------
        // k-distributions of gases whose wavenumber falls between two table
        // points (rankk on lane 0), parked per (layer, gas) in the slot for
        // stage A
        if (B.wg_w2) {
            const float* w2s = B.wg_w2 + S.wg_off + (int64_t)iw * S.ngas;
            const int64_t* slices = B.wg_slice + S.wg_off + (int64_t)iw * S.ngas;
            for (int l = warp * csize + crank; l < S.nlayer; l += WARPS * csize) {
                const KgPos L = kg_pos<t2>(B.lay[S.lay_off + l]);
                float* ncw = slot() + B.nc_off + ((int64_t)l * S.ngas) * kMaxNg * 2;
                for (int g = 0; g < S.ngas; ++g)
                    if (w2s[g] >= 0.0f) {
                        float kv, dv;
                        const float w1 = B.wg_w1 ? B.wg_w1[S.wg_off + (int64_t)iw * S.ngas + g]
                                                 : __fsub_rn(1.0f, w2s[g]);
                        get_kg_lane_nc<t2>(B, slices[g] < 0 ? -1 : slices[g] & ~kSliceLog, w1, w2s[g], L, lane, (float*)wsm, kv, dv);
                        if (lane < ng) {
                            ncw[(g * kMaxNg + lane) * 2] = kv;
                            ncw[(g * kMaxNg + lane) * 2 + 1] = dv;
                        }
                    }
            }
            __syncthreads();
        }
        // ---------------- stage A: layers --------------------------------
        Diag dgn{0, 0, 0};
        // the layers' overlap passes differ in length: a warp takes the next layer when it is done with one
        // (in a cluster, whose warps have a layer or two each, the next in turn)
        auto next_layer = [&](int l) {
            if (csize > 1) return l + WARPS * csize;
            l = 0;
            if (lane == 0) l = atomicAdd(&s_layer, 1);
            return __shfl_sync(kFull, l, 0);
        };
        for (int l = warp * csize + crank; l < S.nlayer; l = next_layer(l)) {
            // addresses are formed where they are used: what lives across the
            // overlap passes costs registers, and those bound the resident warps
            const float amo_lane = lane < S.ngas ? B.amo[S.lg_off + (int64_t)l * S.ngas + lane] : 0.0f;
            auto amo = [&](int g) { return __shfl_sync(kFull, amo_lane, g); };
            // k and dk/dT of every gas with a table, (gas, g) spread over the lanes
            {
                const KgPos L = kg_pos<t2>(B.lay[S.lay_off + l]);
                const int ntask = __popc(s_gmask) * ng;
#pragma unroll 1
                for (int t = lane; t < ntask; t += 32) {
                    const int r = t / ng, g = t - r * ng;
                    float kv, dv;
                    const int64_t at = S.wg_off + (int64_t)iw * S.ngas + s_gas[r];
                    if (B.wg_w2 && B.wg_w2[at] >= 0.0f) {
                        const float* ncw = slot() + B.nc_off + (((int64_t)l * S.ngas + s_gas[r]) * kMaxNg + g) * 2;
                        kv = ncw[0];
                        dv = ncw[1];
                    } else {
                        get_kg_g<t2>(B, s_slice[r], L, g, kv, dv);
                    }
                    ps.kg[t] = make_float2(kv, dv);
                }
                __syncwarp();
            }
            auto get_kg = [&](int g, float& kv, float& dv) {
                const unsigned m = s_gmask;
                float2 v = make_float2(0.0f, 0.0f);
                if ((m >> g & 1u) && lane < ng) v = ps.kg[__popc(m & ((1u << g) - 1u)) * ng + lane];
                kv = v.x;
                dv = v.y;
            };
            // k(g) of the mix so far, its d/dT and its tracked gas columns (zero
            // until the gas is added), ordinate `lane` of each
            float kgv, cT;
            auto zero_columns = [&]() {
                if (lane < ng)
                    for (int c = 0; c < ncol_max; ++c) ps.col[c * ng + lane] = 0.0f;
            };
            zero_columns();
            float k1v, d1v;
            get_kg(0, k1v, d1v);
            const float a1 = amo(0);
            kgv = __fmul_rn(k1v, a1);
            cT = __fmul_rn(d1v, a1);
            int nE = 0;                         // tracked gases added so far
            if (S.col_gas[0] == 0) {
                if (lane < ng) ps.col[lane] = k1v;
                nE = 1;
            }
            for (int ig = 1; ig < S.ngas; ++ig) {
                float k2v, d2v;
                get_kg(ig, k2v, d2v);
                const float a2 = amo(ig);
                const bool z1 = __shfl_sync(kFull, ig == 1 ? k1v : kgv, ng - 1) == 0.0f;
                const bool z2 = __shfl_sync(kFull, k2v, ng - 1) == 0.0f;
                float cAdd;
                if (z1) {                       // noverlapg.f:88-97 / :152-162
                    zero_columns();
                    cT = __fmul_rn(d2v, a2);
                    cAdd = k2v;
                    kgv = __fmul_rn(k2v, a2);
                } else if (z2) {                // noverlapg.f:99-108 / :164-173
                    cAdd = 0.0f;
                } else {
                    bool mono = a2 >= 0.0f && (ig > 1 || a1 >= 0.0f);
                    const float kn = __shfl_down_sync(kFull, k2v, 1);
                    mono = __all_sync(kFull, mono && (lane + 1 >= ng || k2v <= kn));
                    const float b = __fmul_rn(k2v, a2), vT = __fmul_rn(d2v, a2);
                    const int dbg_rec = B.dbg_perm && sidx == 0 ? (iw * S.nlayer + l) * (S.ngas - 1) + (ig - 1) : -1;
                    sort_pass<E, NG>(B, ps, ng, mono, kgv, b, dg, gb, cT, nE, vT, k2v, kgv, cAdd, lane, dgn, dbg_rec);
                }
                // the added gas's column, where it is tracked
                if (nE < kMaxCols && S.col_gas[nE] == ig) {
                    if (lane < ng) ps.col[nE * ng + lane] = cAdd;
                    ++nE;
                }
            }
            // tau and dtau/dq per g (cirsradg_wave.f:744-790)
            const int64_t il_glob = S.lay_off + l, iw_glob = S.wave_off + iw;
            float dtc;
            const float taucon = continuum<ext>(B, S, B.lay[il_glob], B.wave[iw_glob], iw_glob, il_glob, lane, dtc);
            float* tau_l = slot() + l * ng;
            float* dtau_l = slot_dtau() + (size_t)l * S.nsw * ng;
            if (lane < ng) tau_l[lane] = __fadd_rn(taucon, kgv);
            for (int s = 0; s < S.nsw; ++s) {
                // the tracked columns are the first active parameters, gases then T
                float v = __shfl_sync(kFull, dtc, s);
                if (s < S.ncol) v = __fadd_rn(v, s == S.sw_T ? cT : __fmul_rn(ps.col[s * ng + min(lane, ng - 1)], 1.0e-20f));
                if (lane < ng) dtau_l[s * ng + lane] = v;
            }
            __syncwarp();
        }
        if (lane == 0 && dgn.sort_tie) {
            atomicAdd(s_count + 0, (unsigned long long)(dgn.sort_tie & 0xffffu));
            atomicAdd(s_count + 1, (unsigned long long)(dgn.sort_tie >> 16));
            atomicAdd(s_count + 2, (unsigned long long)(dgn.block_exact >> 16));
            atomicAdd(s_count + 3, (unsigned long long)dgn.irregular);
            atomicAdd(s_count + 4, (unsigned long long)(dgn.block_exact & 0xffffu));
        }
        if (csize > 1) {
            // every block's layers are in the slot before the first block runs the paths
            cluster_sync();
            if (crank > 0) {
                cluster_sync();
                continue;
            }
        }
        __syncthreads();

        // ---------------- stage B: paths ---------------------------------
        const WaveDev& W = B.wave[S.wave_off + iw];
        const float* tau_s = slot();
        const float* dtau_s = slot_dtau();
        const int nsw = S.nsw;
        // the emission of every layer of the emission paths, and for IMOD 3 its
        // transmission and absorption per g, spread over the block: a path's own
        // warp then only runs the products along it
        for (int p = 0; p < S.npath; ++p) {
            const int im = S.imod[p], nlays = S.nlayin[p];
            if (!(im == 3 || (ext && im == 18))) continue;
            char* ps = region + p * Lo.path_bytes;
            float* drdt = (float*)(ps + po.drdt);
            float* trd = (float*)(ps + po.trd);
            float* bb = (float*)(ps + po.bb);
            float* dbdt = (float*)(ps + po.dbdt);
            const int* layinc = B.p_layinc + S.path_off + (int64_t)p * S.nlmax;
            const float* scale = B.p_scale + S.path_off + (int64_t)p * S.nlmax;
            const float* emt = B.p_emtemp + S.path_off + (int64_t)p * S.nlmax;
            for (int j = tid; j < nlays; j += kThreads) {
                float Tn = emt[j];
                if (ext && S.inlte)
                    Tn = nlte_temp(S.inlte, Tn, B.lay_press[S.lp_off + layinc[j]], W.vwave, S.nlte_k1, S.nlte_A);
                planck_fp32(S.ispace, W.vwave, Tn, bb[j], dbdt[j]);
            }
            if (im == 3)
                for (int t = tid; t < nlays * ng; t += kThreads) {
                    const int j = t / ng, g = t - j * ng;
                    const float tau = tau_s[layinc[j] * ng + g] * scale[j];
                    drdt[t] = expf(-tau);
                    trd[t] = -expm1f(-tau);
                }
        }
        __syncthreads();
        for (int p = warp; p < S.npath; p += WARPS) {
            char* ps = region + p * Lo.path_bytes;
            float* drdt = (float*)(ps + po.drdt);
            float* trd = (float*)(ps + po.trd);
            float* bb = (float*)(ps + po.bb);
            float* dbdt = (float*)(ps + po.dbdt);
            float* rad = (float*)(ps + po.rad);
            float* gts = (float*)(ps + po.gts);
            const int nlays = S.nlayin[p], im = S.imod[p];
            const int* layinc = B.p_layinc + S.path_off + (int64_t)p * S.nlmax;
            const float* scale = B.p_scale + S.path_off + (int64_t)p * S.nlmax;
            if (lane < ng) {
                const int g = lane;
                if (im == 3) {
                    float tr = 1.0f, R = 0.0f;
#pragma unroll 4
                    for (int j = 0; j < nlays; ++j) {
                        const float td = trd[j * ng + g] * tr;
                        const float trn = tr * drdt[j * ng + g];
                        R = fmaf(bb[j], td, R);
                        drdt[j * ng + g] = trn;
                        trd[j * ng + g] = td;
                        tr = trn;
                    }
                    // surface term unless the path is a limb path (cirsradg_wave.f:991-1025)
                    float Ssum = 0.0f, gt = 0.0f;
                    if ((S.nonlimb_mask >> p) & 1) {
                        const float rg = S.tsurf_pos ? W.radground_s : bb[nlays - 1];
                        const float gg = S.tsurf_pos ? W.gradground_s : dbdt[nlays - 1];
                        R = fmaf(rg, tr, R);
                        gt = tr * gg;
                        Ssum = rg * tr;
                    }
#pragma unroll 4
                    for (int j = nlays - 1; j >= 0; --j) {
                        const float trj = drdt[j * ng + g];
                        drdt[j * ng + g] = bb[j] * trj - Ssum;   // dR/dtau_j
                        Ssum = fmaf(bb[j], trd[j * ng + g], Ssum);
                    }
                    rad[g] = R;
                    gts[g] = gt;
                    if (ext) {   // iform 1 (over the star's flux at v) and 3 (cirsradg_wave.f:913-929)
                        float x = S.xfac3;
                        if (S.wmode == 1) x = __fdiv_rn(x, B.wave_fac[S.wf_off + iw]);
                        if (x != 1.0f) scale_path(x, nlays, ng, g, drdt, trd, rad, gts);
                    }
                } else if (ext && im == 18) {
                    const float x18 = S.wmode == 1 ? __fdiv_rn(S.xfac18, B.wave_fac[S.wf_off + iw]) : S.xfac18;
                    path_imod18(B.e3tab, x18, nlays, ng, g, layinc, scale, tau_s, bb, W.radground_s,
                                W.gradground_s, drdt, trd, rad, gts);
                } else {
                    float tsum = 0.0f;
                    for (int j = 0; j < nlays; ++j) tsum = tsum + tau_s[layinc[j] * ng + g] * scale[j];
                    float y = fmaxf(-tsum, -500.0f);
                    if (y >= 88.7f) y = 88.7f;
                    const float e = (float)exp((double)y);
                    // IMOD 0: dcoutdq = -tau*T*dtau/dq; IMOD 1: tau*(1-A)*dtau/dq with
                    // 1-A formed as T itself (no cancellation when T < 2^-25)
                    float out, dr;
                    if (im == 0) { out = e; dr = -tsum * e; }
                    else { out = 1.0f - e; dr = tsum * e; }
                    if (ext && im == 0 && S.wmode == 2) {   // iform 4: times the star's flux (cirsradg_wave.f:861-879)
                        const float x = B.wave_fac[S.wf_off + iw];
                        out = out * x;
                        dr = dr * x;
                    }
                    for (int j = 0; j < nlays; ++j) { drdt[j * ng + g] = dr; trd[j * ng + g] = 0.0f; }
                    rad[g] = out;
                    gts[g] = 0.0f;
                }
            }
        }
        __syncthreads();

        // ---------------- stage C: g-quadrature of dR/dq -----------------
        for (int p = 0; p < S.npath; ++p) {
            char* ps = region + p * Lo.path_bytes;
            const float* drdt = (const float*)(ps + po.drdt);
            const float* trd = (const float*)(ps + po.trd);
            const float* dbdt = (const float*)(ps + po.dbdt);
            float* dq = (float*)(ps + po.dq);
            const int nlays = S.nlayin[p];
            const int* layinc = B.p_layinc + S.path_off + (int64_t)p * S.nlmax;
            const float* scale = B.p_scale + S.path_off + (int64_t)p * S.nlmax;
            const bool em = S.imod[p] == 3 || (ext && S.imod[p] == 18);
            for (int t = tid; t < nlays * nsw; t += kThreads) {
                const int j = t / nsw, s = t - (t / nsw) * nsw;
                const int l = layinc[j];
                const float sc = scale[j];
                const float* dt = dtau_s + ((size_t)l * nsw + s) * ng;
                const float* dr = drdt + j * ng;
                float acc = 0.0f;
                if (em && s == S.sw_T) {
                    const float dB = dbdt[j];
                    const float* td = trd + j * ng;
                    for (int g = 0; g < ng; ++g) acc = fmaf(delg[g], fmaf(dr[g], dt[g] * sc, td[g] * dB), acc);
                } else {
                    for (int g = 0; g < ng; ++g) acc = fmaf(delg[g], dr[g] * (dt[g] * sc), acc);
                }
                dq[j * nsw + s] = acc;
            }
        }
        __syncthreads();

        // ---------------- stage D: map to the state vector ---------------
        for (int p = 0; p < S.npath; ++p) {
            char* ps = region + p * Lo.path_bytes;
            const float* dq = (const float*)(ps + po.dq);
            if (B.dq_out) {
                float* o = B.dq_out + ((S.wave_off + iw) * B.dq_npath + p) * B.dq_stride;
                for (int t = tid; t < S.nlayin[p] * nsw; t += kThreads) o[t] = dq[t];
            }
            const int* cp = B.map_colptr + S.map_off + (int64_t)p * (S.nv + 1);
            for (int iv = tid; iv < S.nv; iv += kThreads) {
                float acc = 0.0f;
                for (int e = cp[iv]; e < cp[iv + 1]; ++e) acc = fmaf(dq[B.map_row[e]], B.map_val[e], acc);
                B.gradients[S.jac_off + ((int64_t)p * S.nv + iv) * S.nwave + iw] = acc;
            }
            if (tid == 0) {
                const float* rad = (const float*)(ps + po.rad);
                const float* gts = (const float*)(ps + po.gts);
                float o = 0.0f, gt = 0.0f;
                for (int g = 0; g < ng; ++g) {
                    o = fmaf(rad[g], delg[g], o);
                    gt = fmaf(gts[g], delg[g], gt);
                }
                B.calcout[S.out_off + (int64_t)p * S.nwave + iw] = o;
                if (B.gradtsurf) B.gradtsurf[S.out_off + (int64_t)p * S.nwave + iw] = gt;
            }
        }
        __syncthreads();
        if (csize > 1) cluster_sync();      // the slot is free for the next item
    }
    if (tid < 5 && s_count[tid]) atomicAdd(B.counters + tid, s_count[tid]);
}

// The instances are compiled in parts, this file with FWD_PART = 1 .. 13: each part
// is a module of its own, which CUDA loads at the first use of one of its kernels.
// In one module of all 47 a process's first call took 37 ms, 31 of them for loading
// it.  The host side is FWD_PART = 0.  Parts 1-4, 5-8 and 9-12: 8 warps, 16 warps and
// pairs, by t2 + 2 ext; part 13: 2 and 4 warps.
using FwdKern = void (*)(BatchDev, int, int, int, int, int);
#define RTB_FWD_PARTS(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13)
#define RTB_FWD_PART_DECL(p) FwdKern fwd_part_##p(int warps, int ng);
RTB_FWD_PARTS(RTB_FWD_PART_DECL)

#if FWD_PART > 0
namespace {
// the instance of a part for an NG: tiles of 2 and 4 warps, and NG = 20 as a
// constant, exist for the usual options only (one temperature grid, no extended
// options).  Up to 256 elements a pass are sorted in registers, more are merged in
// shared memory.  By the first and the second: 16-point tables, 80 layers, 2
// absorbers, 515 wavenumbers 0.33 and 0.37 ms; 10-point tables, 73 layers, 3
// absorbers, 515 wavenumbers 0.27 and 0.30 ms; 20-point tables, 120 layers, 4
// absorbers, 2000 wavenumbers 3.69 and 3.27 ms.  With TEMP2 tables and the extended
// options (80 layers, 3 absorbers, 1500 wavenumbers) 1.24-1.26 and 1.32-1.36 ms at
// 16 points, 1.23-1.27 and 1.17-1.23 ms at 20.
constexpr int kNgConst = 20;
template <bool t2, bool ext, int WARPS, int CL = 1>
FwdKern fwd_by_ng(int ng) {
    if (!t2 && !ext && ng == kNgConst) return fwd_kernel<t2, ext, WARPS, t2 || ext ? 0 : kNgConst, CL>;
    if (ng * ng > 256) return fwd_kernel<t2, ext, WARPS, 0, CL>;
    if (ng * ng > 128) return fwd_kernel<t2, ext, WARPS, -8, CL>;
    return fwd_kernel<t2, ext, WARPS, -4, CL>;
}
template <int part>
FwdKern fwd_of_part(int warps, int ng) {
    constexpr bool t2 = (part - 1) & 1, ext = (part - 1) & 2;
    if constexpr (part <= 4) return fwd_by_ng<t2, ext, kTileDefault>(ng);
    if constexpr (part > 4 && part <= 8) return fwd_by_ng<t2, ext, kTileWide>(ng);
    if constexpr (part > 8 && part <= 12) return fwd_by_ng<t2, ext, kTileDefault, 2>(ng);
    if constexpr (part == 13) return warps == 2 ? fwd_by_ng<false, false, 2>(ng) : fwd_by_ng<false, false, 4>(ng);
}
}  // namespace
#define RTB_FWD_PART_NAME2(p) fwd_part_##p
#define RTB_FWD_PART_NAME(p) RTB_FWD_PART_NAME2(p)
FwdKern RTB_FWD_PART_NAME(FWD_PART)(int warps, int ng) { return fwd_of_part<FWD_PART>(warps, ng); }

#else
// host-side helpers exported to host.cu
size_t fwd_merge_table_bytes() { return sizeof(MergeLane) * kMergeLevels * 32; }
void fwd_merge_table(int ng, void* table) {
    for (int i = 0; i < kMergeLevels * 32; ++i) ((MergeLane*)table)[i] = merge_lane(ng, i / 32, i % 32);
}

int fwd_smem_bytes(int ng, int nsw, int ncol, int ngk, int nlmax, int npath, int warps) {
    return make_layout(ng, nsw, ncol, ngk, nlmax, npath, warps).total;
}

namespace {
// the instance of a launch: t2 and ext as the batch needs them
FwdKern fwd_instance(bool t2, bool ext, int warps, int ng, bool pair) {
    static constexpr FwdKern (*parts[])(int, int) = {
#define RTB_FWD_PART_PTR(p) fwd_part_##p,
        RTB_FWD_PARTS(RTB_FWD_PART_PTR)};
    const int options = (t2 ? 1 : 0) + (ext ? 2 : 0);
    if (warps == kTileWide) return parts[4 + options](warps, ng);
    if (pair) return parts[8 + options](warps, ng);
    if ((warps == 2 || warps == 4) && !options) return parts[12](warps, ng);
    return parts[options](warps, ng);
}
}  // namespace

int fwd_tile_warps(bool t2, bool ext, int warps) {
    if (warps == kTileWide) return warps;
    return (ext || t2 || (warps != 2 && warps != 4)) ? kTileDefault : warps;
}

int fwd_blocks_per_sm(int smem, bool t2, bool ext, int warps, int ng, bool pair) {
    const int w = fwd_tile_warps(t2, ext, warps);
    const FwdKern k = fwd_instance(t2, ext, w, ng, pair);
    int n = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, w * 32, smem) != cudaSuccess)
        return 0;
    return n;
}

int fwd_max_clusters(int smem, bool t2, bool ext, int warps, int ng, int size) {
    const int w = fwd_tile_warps(t2, ext, warps);
    const FwdKern k = fwd_instance(t2, ext, w, ng, false);
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = size;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(size);
    cfg.blockDim = dim3(w * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int n = 0;
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, smem) != cudaSuccess ||
        cudaOccupancyMaxActiveClusters(&n, k, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

cudaError_t launch_fwd(const BatchDev& B, int nsw, int ncol, int ngk, int nlmax, int npath, int grid, int warps,
                       cudaStream_t st) {
    const int w = fwd_tile_warps(B.t2, B.ext, warps);
    const int smem = fwd_smem_bytes(B.ng, nsw, ncol, ngk, nlmax, npath, w);
    const FwdKern kern = fwd_instance(B.t2, B.ext, w, B.ng, w == kTileDefault && B.cluster == 2);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return e;
    if (B.cluster <= 1) {
        kern<<<grid, w * 32, smem, st>>>(B, nsw, ncol, ngk, nlmax, npath);
        return cudaGetLastError();
    }
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = B.cluster;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid * B.cluster);
    cfg.blockDim = dim3(w * 32);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, B, nsw, ncol, ngk, nlmax, npath);
}

#endif  // FWD_PART

}  // namespace rtb
