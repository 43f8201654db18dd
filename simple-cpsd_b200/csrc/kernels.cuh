// kernels.cuh -- pointwise, reduction, GEMM and Lagrange kernels of one SD step.
//
// Every routine cites the reference lines (ccpsdv3/, Simple-CPSD) whose
// arithmetic it carries.  Complex arrays are cx<double>; packed arrays run
// over the cutoff sphere (see fft.cuh), real grids over n^3 points.
#pragma once

#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

// ------------------------------------------------------------ reductions
template <int NT>
CPSD_D double block_sum(double v, double *sh)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) sh[w] = v;
    __syncthreads();
    double r = 0.0;
    if (threadIdx.x == 0)
        for (int i = 0; i < NT / 32; ++i) r += sh[i];
    return r;  // valid in thread 0
}

// ------------------------------------------------------------ phase factors
// ccpsdv3/strfac.c:10-77: ex_d[k] = e^{-i k (b_d . r + pi)} by recurrence,
// negative k mirrored as conjugates (ex2, ex3), Nyquist entry zeroed.
// ex1: [nion][nh], ex2/ex3: [nion][n]
__global__ void phase_tables_kernel(int nion, int n, const double *__restrict__ unitg,
                                    const double *__restrict__ r1, cx<double> *ex1,
                                    cx<double> *ex2, cx<double> *ex3)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= 3 * nion) return;
    const int ii = id / 3, d = id % 3;
    const double pi = 3.14159265358979323846;  // 4 atan(1), strfac's pi argument
    const double sw = unitg[3 * d] * r1[3 * ii] + unitg[3 * d + 1] * r1[3 * ii + 1] +
                      unitg[3 * d + 2] * r1[3 * ii + 2] + pi;
    const double cr = cos(sw), ci = -sin(sw);
    const int h = n / 2;
    cx<double> *e = (d == 0) ? ex1 + (long)ii * (h + 1) : ((d == 1) ? ex2 : ex3) + (long)ii * n;
    e[0] = cx<double>{1.0, 0.0};
    cx<double> p{1.0, 0.0};
    for (int k = 1; k <= h; ++k) {
        cx<double> q{p.x * cr - p.y * ci, p.x * ci + p.y * cr};
        e[k] = q;
        if (d > 0) e[n - k] = cx<double>{q.x, -q.y};
        p = q;
    }
    e[h] = cx<double>{0.0, 0.0};
}

// exi(G) = ex1[i] (ex2[j] ex3[k]) in the reference's multiplication order, strfac.c:112-115
CPSD_D cx<double> strfac_point(cx<double> e1, cx<double> e2, cx<double> e3)
{
    double tr = e2.x * e3.x - e2.y * e3.y;
    double ti = e2.x * e3.y + e2.y * e3.x;
    return cx<double>{e1.x * tr - e1.y * ti, e1.y * tr + e1.x * ti};
}

// ------------------------------------------------------------ local psp, projectors
// ccpsdv3/cpsd.c:224-245 (s, vall), :260-286 (projectors)
struct VlocArgs {
    int npw, npw_pad, n, nh, nion;
    const int *pt_i, *pt_j, *pt_k;
    const int *katm;
    const double *zv;
    const cx<double> *ex1, *ex2, *ex3;
    const double *vl;   // [nkatm][npw]
    const double *vnl;  // [nkatm][9][npw]
    const int *lmmax;   // [nkatm]
    const int *proj_off;  // [nion] first projector row of each ion
    cx<double> *s, *vall;
    cx<double> *proj;   // [nproj][npw_pad]
};

__global__ void vloc_proj_kernel(VlocArgs a)
{
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= a.npw_pad) return;
    if (p >= a.npw) {  // keep the GEMM padding at zero
        for (int ii = 0; ii < a.nion; ++ii) {
            const int nl = a.lmmax[a.katm[ii]];
            for (int l = 0; l < nl; ++l) a.proj[(long)(a.proj_off[ii] + l) * a.npw_pad + p] = cx<double>{0, 0};
        }
        return;
    }
    const int i = a.pt_i[p], j = a.pt_j[p], k = a.pt_k[p];
    cx<double> s{0, 0}, vall{0, 0};
    for (int ii = 0; ii < a.nion; ++ii) {
        const int ia = a.katm[ii];
        cx<double> exi = strfac_point(a.ex1[(long)ii * a.nh + i], a.ex2[(long)ii * a.n + j],
                                      a.ex3[(long)ii * a.n + k]);
        const double z = a.zv[ia];
        s.x += z * exi.x;
        s.y += z * exi.y;
        const double v = a.vl[(long)ia * a.npw + p];
        vall.x += exi.x * v;
        vall.y += exi.y * v;
        const int nl = a.lmmax[ia];
        for (int l = 0; l < nl; ++l) {
            const double w = a.vnl[((long)ia * 9 + l) * a.npw + p];
            cx<double> chi = (l == 0 || l >= 4) ? cx<double>{exi.x * w, exi.y * w}
                                                : cx<double>{-exi.y * w, exi.x * w};
            a.proj[(long)(a.proj_off[ii] + l) * a.npw_pad + p] = chi;
        }
    }
    a.s[p] = s;
    a.vall[p] = vall;
}

// ------------------------------------------------------------ ion forces
// move = 1 (cpsd.c:246-257, 291-304, 310-364).  All Gamma-point sums use the
// weight w (1 on kx = 0, 2 elsewhere: gsdot of ccpsdv3/gsdot.c) over the
// sphere; G_d is the d-th Cartesian component of G per sphere point.
constexpr int kForceChunks = 16;  // point chunks of the local + k-space Ewald sums

struct ForceArgs {
    int npw, n, nh, nion;
    const int *pt_i, *pt_j, *pt_k, *katm;
    const cx<double> *ex1, *ex2, *ex3;  // phase tables of r1
    const double *w, *G;                // G: [3][npw]
    const double *vl, *vg, *zv;
    const cx<double> *dng, *s;
    double scal2;
    double *fpart;  // [chunk][ion][3]
};

// Local force (cpsd.c:246-257: sum_G G_d (Im dng Re exi - Re dng Im exi) vl)
// and k-space Ewald force (cpsd.c:318-328: sum_G G_d (exi x s) vg zv scal2)
// of ion blockIdx.y over point chunk blockIdx.x, fixed-order block sums.
__global__ void __launch_bounds__(256) force_local_ewald_kernel(ForceArgs a)
{
    __shared__ double sh[32];
    const int ii = blockIdx.y, ch = blockIdx.x;
    const int per = (a.npw + kForceChunks - 1) / kForceChunks;
    const int p0 = ch * per, p1 = min(a.npw, p0 + per);
    const int ia = a.katm[ii];
    const double zs = a.zv[ia] * a.scal2;
    double f[3] = {0.0, 0.0, 0.0};
    for (int p = p0 + threadIdx.x; p < p1; p += 256) {
        const cx<double> e = strfac_point(a.ex1[(long)ii * a.nh + a.pt_i[p]], a.ex2[(long)ii * a.n + a.pt_j[p]],
                                          a.ex3[(long)ii * a.n + a.pt_k[p]]);
        const cx<double> d = a.dng[p], sp = a.s[p];
        const double vl = a.vl[(long)ia * a.npw + p];
        const double loc = vl * (d.y * e.x - d.x * e.y);
        const double ewk = (e.x * sp.y - e.y * sp.x) * a.vg[p] * zs;
        const double t = a.w[p] * (loc + ewk);
        for (int k = 0; k < 3; ++k) f[k] += t * a.G[(long)k * a.npw + p];
    }
    for (int k = 0; k < 3; ++k) {
        const double v = block_sum<256>(f[k], sh);
        if (threadIdx.x == 0) a.fpart[((long)ch * a.nion + ii) * 3 + k] = v;
    }
}

// Nonlocal force per projector P (cpsd.c:291-304): with Y_P = sum_b sw1(P, b)
// c1_b, fnl[P][d] = sum_G w G_d Im(conj(chi_P) Y_P).
__global__ void __launch_bounds__(256) force_nonlocal_kernel(int npw, long ld, const double *__restrict__ w,
                                                             const double *__restrict__ G,
                                                             const cx<double> *__restrict__ proj,
                                                             const cx<double> *__restrict__ Y,
                                                             double *__restrict__ fnl)
{
    __shared__ double sh[32];
    const int P = blockIdx.x;
    const cx<double> *chi = proj + (long)P * ld, *y = Y + (long)P * ld;
    double f[3] = {0.0, 0.0, 0.0};
    for (int p = threadIdx.x; p < npw; p += 256) {
        const cx<double> c = chi[p], v = y[p];
        const double t = w[p] * (c.x * v.y - c.y * v.x);
        for (int k = 0; k < 3; ++k) f[k] += t * G[(long)k * npw + p];
    }
    for (int k = 0; k < 3; ++k) {
        const double v = block_sum<256>(f[k], sh);
        if (threadIdx.x == 0) fnl[3 * P + k] = v;
    }
}

// Real-space Ewald force of each pair ii < jj (cpsd.c:331-362), summed over
// the image cells: ewp[pair][3], pair = ii (2 nion - ii - 1) / 2 + jj - ii - 1.
__global__ void __launch_bounds__(256) force_ewald_pairs_kernel(int nion, int nsh, const double *__restrict__ r1,
                                                                const double *__restrict__ rcell,
                                                                const double *__restrict__ zv,
                                                                const int *__restrict__ katm, double rcut,
                                                                double *__restrict__ ewp)
{
    const double B1 = 0.0705230784, B2 = 0.0422820123, B3 = 0.0092705272;
    const double B4 = 0.0001520143, B5 = 0.0002765672, B6 = 0.0000430638;
    const double CERFC = 1.128379167;  // 2 / sqrt(pi), as cpsd.c rounds it
    const int ii = blockIdx.x;
    const long off = (long)ii * (2L * nion - ii - 1) / 2;
    for (int jj = ii + 1 + threadIdx.x; jj < nion; jj += 256) {
        const double dx = r1[3 * ii] - r1[3 * jj];
        const double dy = r1[3 * ii + 1] - r1[3 * jj + 1];
        const double dz = r1[3 * ii + 2] - r1[3 * jj + 2];
        const double zz = zv[katm[ii]] * zv[katm[jj]];
        double s1 = 0.0, s2 = 0.0, s3 = 0.0;
        for (int l = 0; l < nsh; ++l) {
            const double x = rcell[l] + dx, y = rcell[l + nsh] + dy, z = rcell[l + 2 * nsh] + dz;
            const double r = sqrt(x * x + y * y + z * z);
            const double wr = r / rcut;
            double aa = (1.0 + wr * (B1 + wr * (B2 + wr * (B3 + wr * (B4 + wr * (B5 + wr * B6))))));
            aa *= aa * aa * aa;
            const double erfc = 1.0 / (aa * aa * aa * aa);
            const double ad = zz * (erfc + CERFC * wr * exp(-wr * wr)) / (r * r * r);
            s1 += x * ad;
            s2 += y * ad;
            s3 += z * ad;
        }
        const long pr = off + (jj - ii - 1);
        ewp[3 * pr] = s1;
        ewp[3 * pr + 1] = s2;
        ewp[3 * pr + 2] = s3;
    }
}

// fion = local + k-space Ewald - nonlocal + real-space Ewald, and the ion SD
// step r2 = r1 + dti fion (cpsd.c:401-411); one thread per ion, fixed order.
__global__ void force_total_kernel(int nion, double nl_factor, const int *__restrict__ proj_off,
                                   const int *__restrict__ lmmax, const int *__restrict__ katm,
                                   const double *__restrict__ fpart, const double *__restrict__ fnl,
                                   const double *__restrict__ ewp, const double *__restrict__ dti,
                                   const double *__restrict__ r1, double *__restrict__ fion,
                                   double *__restrict__ r2)
{
    const int ii = blockIdx.x * blockDim.x + threadIdx.x;
    if (ii >= nion) return;
    double f[3] = {0.0, 0.0, 0.0};
    for (int ch = 0; ch < kForceChunks; ++ch)
        for (int k = 0; k < 3; ++k) f[k] += fpart[((long)ch * nion + ii) * 3 + k];
    const int nl = lmmax[katm[ii]];
    for (int l = 0; l < nl; ++l)
        for (int k = 0; k < 3; ++k) f[k] -= nl_factor * fnl[3 * (proj_off[ii] + l) + k];
    for (int a = 0; a < ii; ++a) {  // pairs (a, ii) enter with a minus sign (cpsd.c:359-361)
        const long pr = (long)a * (2L * nion - a - 1) / 2 + (ii - a - 1);
        for (int k = 0; k < 3; ++k) f[k] -= ewp[3 * pr + k];
    }
    const long off = (long)ii * (2L * nion - ii - 1) / 2;
    for (int b = ii + 1; b < nion; ++b)  // pairs (ii, b): plus (cpsd.c:356-358)
        for (int k = 0; k < 3; ++k) f[k] += ewp[3 * (off + b - ii - 1) + k];
    for (int k = 0; k < 3; ++k) {
        fion[3 * ii + k] = f[k];
        r2[3 * ii + k] = r1[3 * ii + k] + dti[ii] * f[k];
    }
}

// coefficients of the KB back-projection, ccpsdv3/cpsd.c:289:
// coefT[b][P] = -beta[P][b] * scal2 / vnlnrm[P]
// (and, for the nonlocal force, the same in [P][b] order when coefP is given)
__global__ void kb_coef_kernel(int nproj, int nb, const double *__restrict__ beta,
                               const double *__restrict__ vnlnrm_p, double scal2,
                               double *__restrict__ coefT, double *__restrict__ coefP)
{
    const int id = blockIdx.x * blockDim.x + threadIdx.x;
    if (id >= nproj * nb) return;
    const int P = id / nb, b = id % nb;
    const double v = -beta[id] * scal2 / vnlnrm_p[P];
    coefT[(long)b * nproj + P] = v;
    if (coefP) coefP[id] = v;
}

// ------------------------------------------------------------ density + xc
// dn_ms = scal2 * sum_b psi_b^2 (cpsd.c:185-194); Dirac exchange then Vosko
// correlation (dirac_exchange.c:64-126, vosko.c:99-167); the forward-FFT
// input (dn_0 + dn_{ispin-1}) * scal1 (cpsd.c:198-199).
struct XcArgs {
    long n3;
    int ispin;
    int nchunk0, nchunk1;  // chunks of spin 0, then of spin 1
    const double *part;    // [nchunk][n3]
    double scal1, scal2;
    double *dn, *xcp, *xce, *rfwd;
};

// Closed shell: the same functions with one cube root (the densities of the
// two parts differ by 2e-30, which a density above ~1e-14 does not hold) and
// one division for the reciprocals of the correlation.  The evaluation is bound
// by the FP64 pipe: 128^3 64 -> 47 us, 64^3 14.4 -> 10.5 us against two cube
// roots and nine divisions, with the same error against 64 bits.
CPSD_D void dirac_vosko_closed(double nup_in, double &vx, double &ex)
{
    const double nd = nup_in + nup_in;                // dirac_exchange.c's density
    const double n = 2.0 * (nup_in + 1.0e-30);        // vosko.c's
    const double c = cbrt(n);
    // cbrt(3 / pi) cbrt(n) = cbrt(3 n / pi)
    const double n13 = (n == nd) ? 0.98474502184269654115 * c : cbrt(3.0 * nd / 3.14159265358979311600);
    const double alpha = 0.6666666666666666667;
    const double bp = 3.727440e+00, cp = 1.293520e+01, cp1 = 3.109070e-02, cp2 = 9.690228e-04, cp3 = 1.049800e-01;
    const double cp4 = 3.878329e-02, cp5 = 3.075995e+00, cp6 = 1.863720e+00;
    const double dp1 = 6.218140e-02, dp2 = 1.938045e-03, dp4 = -3.205972e-02, dp5 = -1.192972e-01, dp7 = 9.461748e+00;
    const double onesixth = 0.166666666666667;
    const double rs = 0.620350490899400 / c;
    const double x = sqrt(rs);
    const double xx = rs + bp * x + cp, dxx = 2.0 * x + bp;
    const double a = x + cp3, s = x + cp6, b = s * s + dp7;  // dp6 = cp6
    const double p1 = xx * a, p2 = b * s, ip = 1.0 / (p1 * p2);
    const double i1 = ip * p2, i2 = ip * p1;  // 1 / (xx a), 1 / (b s)
    const double ixx = i1 * a, ia = i1 * xx, ib = i2 * s, is = i2 * b;
    const double ec = cp1 * log(rs * ixx) + cp2 * log(a * a * ixx) + cp4 * atan(cp5 * is);
    ex = -(9.0 / 8.0) * alpha * n13 + ec;
    vx = -(3.0 / 2.0) * alpha * n13 + (ec - onesixth * (dp1 + x * (dp2 * ia + dp4 * dxx * ixx + dp5 * ib)));
}

CPSD_D void dirac_vosko(int ispin, double nup_in, double ndn_in, double rho0, double rho1,
                        double &vx0, double &vx1, double &ex)
{
    if (ispin == 1) {
        dirac_vosko_closed(nup_in, vx0, ex);
        vx1 = vx0;
        return;
    }
    // --- Dirac exchange, alpha = 2/3 (dirac_exchange.c:14-24, 84-122)
    const double alpha = 0.6666666666666666667;
    const double onethird_d = 0.33333333333333333333;
    const double fourthird_d = 1.33333333333333333333;
    const double two_to_onethird_d = 1.25992104989487319067;
    const double A_d = 0.25992104989487319067;
    const double pi_d = 3.14159265358979311600;
    // cube roots of the (non-negative) density by cbrt: the reference's
    // pow(x, 1/3) to within an ulp
    {
        const double n = nup_in + ndn_in;
        const double n13 = cbrt(3.0 * n / pi_d);
        // the reference's xi here uses the first two density values (dirac_exchange.c:101)
        const double xi = (n > 0.0) ? (rho0 - rho1) / n : 1.0;
        const double ex_p = -(9.0 / 8.0) * alpha * n13;
        const double ux_p = -(3.0 / 2.0) * alpha * n13;
        const double ex_f = two_to_onethird_d * ex_p;
        const double ux_f = fourthird_d * ex_f;
        const double f = (pow(1.0 + xi, fourthird_d) + pow(1.0 - xi, fourthird_d) - 2.0) / (2.0 * A_d);
        const double df = fourthird_d * (pow(1.0 + xi, onethird_d) - pow(1.0 - xi, onethird_d)) / (2.0 * A_d);
        ex = ex_p + f * (ex_f - ex_p);
        vx0 = ux_p + f * (ux_f - ux_p) + (+1.0 - xi) * (df * (ex_f - ex_p));
        vx1 = ux_p + f * (ux_f - ux_p) + (-1.0 - xi) * (df * (ex_f - ex_p));
    }
    // --- Vosko-Wilk-Nusair, the reference's parameter table (vosko.c:22-57)
    const double bp = 3.727440e+00, bf = 7.060420e+00;
    const double cp = 1.293520e+01, cf = 1.805780e+01;
    const double cp1 = 3.109070e-02, cf1 = 1.554530e-02;
    const double cp2 = 9.690228e-04, cf2 = 2.247860e-03;
    const double cp3 = 1.049800e-01, cf3 = 3.250000e-01;
    const double cp4 = 3.878329e-02, cf4 = 5.249122e-02;
    const double cp5 = 3.075995e+00, cf5 = 2.365463e+00;
    const double cp6 = 1.863720e+00, cf6 = 3.530210e+00;
    const double dp1 = 6.218140e-02, df1 = 3.109060e-02;
    const double dp2 = 1.938045e-03, df2 = 4.495720e-03;
    const double dp4 = -3.205972e-02, df4 = -1.779316e-02;
    const double dp5 = -1.192972e-01, df5 = -1.241661e-01;
    const double dp6 = 1.863720e+00, df6 = 3.530210e+00;
    const double dp7 = 9.461748e+00, df7 = 5.595417e+00;
    const double small_number = 1.0e-30;
    const double onesixth = 0.166666666666667;
    const double onethird = 0.333333333333333;
    const double fourthird = 1.333333333333333;
    const double A = 0.259921049894873;
    const double rs_scale = 0.620350490899400;
    const double nup = nup_in + small_number;
    const double ndown = ndn_in + small_number;
    const double n = nup + ndown;
    const double rs = rs_scale / cbrt(n);
    const double xi = (nup - ndown) / n;
    const double x = sqrt(rs);
    const double xxp = rs + bp * x + cp;
    const double dxxp = 2.0 * x + bp;
    const double ec_p = cp1 * log(rs / xxp) + cp2 * log((x + cp3) * (x + cp3) / xxp) + cp4 * atan(cp5 / (x + cp6));
    const double uc_p = ec_p - onesixth * x * (dp1 / x + dp2 / (x + cp3) + dp4 * dxxp / xxp +
                                               dp5 / ((x + dp6) * (x + dp6) + dp7));
    const double xxf = rs + bf * x + cf;
    const double dxxf = 2.0 * x + bf;
    const double ec_f = cf1 * log(rs / xxf) + cf2 * log((x + cf3) * (x + cf3) / xxf) + cf4 * atan(cf5 / (x + cf6));
    const double uc_f = ec_f - onesixth * x * (df1 / x + df2 / (x + cf3) + df4 * dxxf / xxf +
                                               df5 / ((x + df6) * (x + df6) + df7));
    const double f = (pow(1.0 + xi, fourthird) + pow(1.0 - xi, fourthird) - 2.0) / (2.0 * A);
    const double df = fourthird * (pow(1.0 + xi, onethird) - pow(1.0 - xi, onethird)) / (2.0 * A);
    ex += ec_p + f * (ec_f - ec_p);
    vx0 += uc_p + f * (uc_f - uc_p) + (+1.0 - xi) * (df * (ec_f - ec_p));
    vx1 += uc_p + f * (uc_f - uc_p) + (-1.0 - xi) * (df * (ec_f - ec_p));
}

__global__ void density_xc_kernel(XcArgs a)
{
    chain_wait();
    chain_start();
    const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n3) return;
    double d[2] = {0.0, 0.0}, r0 = 0.0, r1 = 0.0;
    for (int c = 0; c < a.nchunk0; ++c) {
        d[0] += a.part[(long)c * a.n3 + r];
        if (a.ispin == 2) {
            r0 += a.part[(long)c * a.n3 + 0];
            r1 += a.part[(long)c * a.n3 + 1];
        }
    }
    for (int c = a.nchunk0; c < a.nchunk0 + a.nchunk1; ++c) d[1] += a.part[(long)c * a.n3 + r];
    d[0] *= a.scal2;
    d[1] *= a.scal2;
    r0 *= a.scal2;
    r1 *= a.scal2;
    double vx0, vx1, ex;
    dirac_vosko(a.ispin, d[0], d[1], r0, r1, vx0, vx1, ex);
    a.dn[r] = d[0];
    a.xcp[r] = vx0;
    a.xce[r] = ex;
    if (a.ispin == 2) {
        a.dn[a.n3 + r] = d[1];
        a.xcp[a.n3 + r] = vx1;
    }
    a.rfwd[r] = (d[0] + d[a.ispin - 1]) * a.scal1;
}

// Band-parallel steps split density_xc_kernel at the exchange: this rank's
// chunk sums (its bands only) -> dn_part, summed over the ranks into dn,
// then the xc potential from dn.  The arithmetic per point is that of
// density_xc_kernel, so one rank owning every band gets the same bits.
__global__ void density_sum_kernel(XcArgs a, double *dn_part)
{
    const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n3) return;
    double d0 = 0.0, d1 = 0.0;
    for (int c = 0; c < a.nchunk0; ++c) d0 += a.part[(long)c * a.n3 + r];
    for (int c = a.nchunk0; c < a.nchunk0 + a.nchunk1; ++c) d1 += a.part[(long)c * a.n3 + r];
    dn_part[r] = d0 * a.scal2;
    if (a.ispin == 2) dn_part[a.n3 + r] = d1 * a.scal2;
}

__global__ void xc_from_density_kernel(XcArgs a)
{
    const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= a.n3) return;
    const double d0 = a.dn[r], d1 = (a.ispin == 2) ? a.dn[a.n3 + r] : 0.0;
    // the reference's xi of the spin-polarised exchange reads the first two
    // spin-0 density values (dirac_exchange.c:101)
    const double r0 = (a.ispin == 2) ? a.dn[0] : 0.0, r1 = (a.ispin == 2) ? a.dn[1] : 0.0;
    double vx0, vx1, ex;
    dirac_vosko(a.ispin, d0, d1, r0, r1, vx0, vx1, ex);
    a.xcp[r] = vx0;
    a.xce[r] = ex;
    if (a.ispin == 2) a.xcp[a.n3 + r] = vx1;
    a.rfwd[r] = (d0 + (a.ispin == 2 ? d1 : d0)) * a.scal1;
}

// dn = sum over the parts in their order (the ranks' spin densities of a
// band-parallel step on one device)
constexpr int kMaxGroupRanks = 8;
struct PartSum {
    const double *part[kMaxGroupRanks];
    int nparts;
};
__global__ void sum_parts_kernel(PartSum p, long n, double *out)
{
    const long r = (long)blockIdx.x * blockDim.x + threadIdx.x;
    if (r >= n) return;
    double acc = p.part[0][r];
    for (int q = 1; q < p.nparts; ++q) acc += p.part[q][r];
    out[r] = acc;
}

// ------------------------------------------------------------ FP64 GEMMs
// part[prod][split][i][j] = sum_{k in chunk} w(k) A_prod[i*lda+k] B_prod[j*ldb+k];
// K counts reals, the weight is per complex pair (w[k/2]): the Gamma-point
// dot of ccpsdv3/gcdotc.c as a matrix product.  Up to kTnMaxProd products of
// the same shape share one launch (blockIdx.z = prod * splits + split).
constexpr int kTnMaxProd = 4;

struct TnBatch {
    const double *A[kTnMaxProd];
    const double *B[kTnMaxProd];
    double *C[kTnMaxProd];
    int nprod, splits;
    unsigned sym;  // products read by their upper triangle only (bit per product)
};

// C_prod[i*ldc+j] = alpha * sum_s part[prod][s][i][j] (+ beta C): a block takes
// 32 neighbouring outputs (256-byte reads of every split's partials) and eight
// interleaved groups of splits, then adds the groups in order: the order of
// the additions (and the bits of the result) never changes.  128 bands, three
// products of 59 splits: 24 us as a warp per output with lanes over the splits
// (an 8-byte read per 32-byte sector), 9 us here.
constexpr int kRedOut = 32, kRedGroups = 8;
__global__ void __launch_bounds__(kRedOut * kRedGroups)
splitk_reduce_kernel(int M, int N, long ldc, const double *__restrict__ part, double alpha,
                     double beta, const __grid_constant__ TnBatch bt)
{
    __shared__ double sh[kRedGroups][kRedOut];
    const long MN = (long)M * N, nblk = (MN + kRedOut - 1) / kRedOut;
    const int x = threadIdx.x % kRedOut, y = threadIdx.x / kRedOut;
    const int prod = (int)(blockIdx.x / nblk);
    const long e = (blockIdx.x % nblk) * kRedOut + x;
    const bool ok = e < MN && !(((bt.sym >> prod) & 1) && e / N > e % N);  // below the diagonal: not formed
    double s = 0.0;
    if (ok) {
        const double *p = part + (long)prod * bt.splits * MN + e;
#pragma unroll 4
        for (int q = y; q < bt.splits; q += kRedGroups) s += p[(long)q * MN];
    }
    sh[y][x] = s;
    __syncthreads();
    if (y == 0 && ok) {
#pragma unroll
        for (int k = 1; k < kRedGroups; ++k) s += sh[k][x];
        const int i = (int)(e / N), j = (int)(e % N);
        double *c = bt.C[prod] + (long)i * ldc + j;
        *c = alpha * s + (beta == 0.0 ? 0.0 : beta * *c);
    }
}

// ------------------------------------------------------------ FP64 tensor-core GEMMs
// Two products on the FP64 tensor cores (mma.sync m8n8k4 f64: exact FP64
// products, FP64 sums): the split-K weighted TN partials above and the
// back-projection NN product (the reference's dgemm('N','N') on
// column-major psi blocks, cpsd.c:483-488).  A CTA of four warps owns a 64x64 output
// tile, each warp a 32x32 quadrant of 4x4 fragments of 8x8, and walks the
// contraction in slabs of 16 that arrive by cp.async, kDmStages - 1 slabs
// ahead, with one barrier per slab.
//
// Bound: the FP64 pipe (an m8n8k4 occupies its quarter of the SM for 16 cycles,
// the rate of 8 DFMAs; 27 cycles latency).  The former kernels fetched the next
// slab through registers and multiplied the weights into it as it arrived, so
// every slab waited for its loads (42-49 % of the pipe); here the weights
// multiply the fragments.
constexpr int kDmT = 64, kDmK = 16, kDmThreads = 128, kDmStages = 3;
// TN: rows of 16 reals, 18 apart: consecutive rows sit 9 16-byte units apart, a
// lane's pair of k-slots (tile columns 4q + 2h, +1) is one 16-byte load, free
// of bank conflicts.
constexpr int kDmS = 18;
// NN: matrix rows 24 apart with k-slot q = tile columns 2q, 2q + 1 of each half,
// operand rows of 64 columns 66 apart: both free of conflicts
constexpr int kDmSA = 24, kDmSB = 66;
constexpr size_t kDmTnSmem = sizeof(double) * kDmStages * (2 * kDmT * kDmS + kDmK / 2);
constexpr size_t kDmNnSmem = sizeof(double) * kDmStages * (kDmT * kDmSA + kDmK * kDmSB);

CPSD_D void dmma(double &d0, double &d1, double a, double b)
{
    asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
                 : "+d"(d0), "+d"(d1)
                 : "d"(a), "d"(b));
}

// n (0, 1 or 2) doubles to a pair in shared memory, the rest zero.  V2: the
// source is 16-byte aligned (one 16-byte copy), else two 8-byte copies.
template <bool V2>
CPSD_D void cp_async_pair(double *dst, const double *src, int n)
{
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (V2) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(8 * n) : "memory");
    } else {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(src), "r"(n > 0 ? 8 : 0) : "memory");
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d + 8), "l"(n > 1 ? src + 1 : src),
                     "r"(n > 1 ? 8 : 0) : "memory");
    }
}
CPSD_D void dm_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
CPSD_D void dm_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// part[prod][split][i][j] as above; grid (M tiles, N tiles, nprod * splits).
// Products whose bit in bt.sym is set are read by their upper triangle only
// (i <= j): their tiles below the diagonal are not formed.
template <bool V2>
__global__ void __launch_bounds__(kDmThreads, 4)
gemm_tn_dmma_kernel(int M, int N, int K, long lda, long ldb, const double *__restrict__ w, int kchunk,
                    const __grid_constant__ TnBatch bt, double *__restrict__ part)
{
    extern __shared__ __align__(16) double dm_sm[];
    const int prod = blockIdx.z / bt.splits, split = blockIdx.z % bt.splits;
    if (((bt.sym >> prod) & 1) && blockIdx.x > blockIdx.y) return;
    double *As = dm_sm, *Bs = As + kDmStages * kDmT * kDmS, *Ws = Bs + kDmStages * kDmT * kDmS;
    const double *__restrict__ A = bt.A[prod];
    const double *__restrict__ B = bt.B[prod];
    const int i0 = blockIdx.x * kDmT, j0 = blockIdx.y * kDmT;
    const int k0 = split * kchunk, k1 = min(K, k0 + kchunk);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32, fr = lane >> 2, fq = lane & 3;
    const int ns = k1 > k0 ? (k1 - k0 + kDmK - 1) / kDmK : 0;
    // slab it: thread -> reals (2p, 2p+1) of rows row, row + 16, .. (p = tid & 7, row = tid >> 3)
    auto issue = [&](int it) {
        const int st = it % kDmStages, k = k0 + it * kDmK + 2 * (tid & 7);
        const int n = min(2, max(0, k1 - k));
        double *a = As + st * kDmT * kDmS + 2 * (tid & 7), *b = Bs + st * kDmT * kDmS + 2 * (tid & 7);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int row = (tid >> 3) + 16 * q, i = i0 + row, j = j0 + row;
            cp_async_pair<V2>(a + row * kDmS, n > 0 && i < M ? A + (long)i * lda + k : A, i < M ? n : 0);
            cp_async_pair<V2>(b + row * kDmS, n > 0 && j < N ? B + (long)j * ldb + k : B, j < N ? n : 0);
        }
        if (w != nullptr && tid < kDmK / 2) {  // one weight per pair (k0 is even)
            const int kw = k0 + it * kDmK + 2 * tid;
            const uint32_t d = (uint32_t)__cvta_generic_to_shared(Ws + st * (kDmK / 2) + tid);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;" ::"r"(d), "l"(w + (kw < k1 ? kw >> 1 : 0)),
                         "r"(kw < k1 ? 8 : 0) : "memory");
        }
    };
    if (w == nullptr && tid < kDmStages * kDmK / 2) Ws[tid] = 1.0;
#pragma unroll
    for (int it = 0; it < kDmStages - 1; ++it) {
        if (it < ns) issue(it);
        dm_commit();
    }
    double acc[4][4][2] = {};
    for (int it = 0; it < ns; ++it) {
        dm_wait<kDmStages - 2>();
        __syncthreads();  // slab it has landed for every thread; the slot of slab it - 1 is free
        if (it + kDmStages - 1 < ns) issue(it + kDmStages - 1);
        dm_commit();
        const int st = it % kDmStages;
        const double *as = As + st * kDmT * kDmS, *bs = Bs + st * kDmT * kDmS;
        const double2 ww = *reinterpret_cast<const double2 *>(Ws + st * (kDmK / 2) + 2 * fq);
        // two halves of two k-steps each: one 16-byte fragment load per
        // operand row per half keeps the fragments in 32 registers
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {
            double2 a[4], b[4];
            const double wk = hh ? ww.y : ww.x;
#pragma unroll
            for (int f = 0; f < 4; ++f) {
                a[f] = *reinterpret_cast<const double2 *>(as + (wr + 8 * f + fr) * kDmS + 4 * fq + 2 * hh);
                b[f] = *reinterpret_cast<const double2 *>(bs + (wc + 8 * f + fr) * kDmS + 4 * fq + 2 * hh);
                a[f].x *= wk;
                a[f].y *= wk;
            }
#pragma unroll
            for (int fi = 0; fi < 4; ++fi)
#pragma unroll
                for (int fj = 0; fj < 4; ++fj) dmma(acc[fi][fj][0], acc[fi][fj][1], a[fi].x, b[fj].x);
#pragma unroll
            for (int fi = 0; fi < 4; ++fi)
#pragma unroll
                for (int fj = 0; fj < 4; ++fj) dmma(acc[fi][fj][0], acc[fi][fj][1], a[fi].y, b[fj].y);
        }
    }
    dm_wait<0>();
    double *out = part + ((long)prod * bt.splits + split) * M * N;
#pragma unroll
    for (int fi = 0; fi < 4; ++fi) {
        const int i = i0 + wr + 8 * fi + fr;
        if (i >= M) continue;
#pragma unroll
        for (int fj = 0; fj < 4; ++fj)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = j0 + wc + 8 * fj + 2 * fq + h;
                if (j < N) out[(long)i * N + j] = acc[fi][fj][h];
            }
    }
}

// Out[j*ldo+k] = beta*Out + alpha * sum_l
// Mat[l + j*ldm] * B[l*ldb + k]; grid x over 64-wide k tiles, y over j tiles.
// V2: Mat, B and their strides are 16-byte aligned.
template <bool V2>
__global__ void __launch_bounds__(kDmThreads, 3)
gemm_nn_dmma_kernel(int NJ, int K, int L, double alpha, const double *__restrict__ Mat, long ldm,
                    const double *__restrict__ B, long ldb, double beta, double *Out, long ldo)
{
    extern __shared__ __align__(16) double dm_sm[];
    double *Ms = dm_sm, *Bs = Ms + kDmStages * kDmT * kDmSA;
    const int k0 = blockIdx.x * kDmT, j0 = blockIdx.y * kDmT;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wr = (warp >> 1) * 32, wc = (warp & 1) * 32, fr = lane >> 2, fq = lane & 3;
    const int ns = (L + kDmK - 1) / kDmK;
    auto issue = [&](int it) {
        const int st = it % kDmStages, l0 = it * kDmK;
        double *m = Ms + st * kDmT * kDmSA + 2 * (tid & 7), *b = Bs + st * kDmK * kDmSB + 2 * (tid & 31);
        const int l = l0 + 2 * (tid & 7), n = min(2, max(0, L - l));
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // Mat: row j, reals l, l + 1
            const int row = (tid >> 3) + 16 * q, j = j0 + row;
            cp_async_pair<V2>(m + row * kDmSA, n > 0 && j < NJ ? Mat + (long)j * ldm + l : Mat, j < NJ ? n : 0);
        }
        const int k = k0 + 2 * (tid & 31), nk = min(2, max(0, K - k));
#pragma unroll
        for (int q = 0; q < 4; ++q) {  // B: row l, reals k, k + 1
            const int row = (tid >> 5) + 4 * q, lb = l0 + row;
            cp_async_pair<V2>(b + row * kDmSB, nk > 0 && lb < L ? B + (long)lb * ldb + k : B, lb < L ? nk : 0);
        }
    };
#pragma unroll
    for (int it = 0; it < kDmStages - 1; ++it) {
        if (it < ns) issue(it);
        dm_commit();
    }
    double acc[4][4][2] = {};
    for (int it = 0; it < ns; ++it) {
        dm_wait<kDmStages - 2>();
        __syncthreads();
        if (it + kDmStages - 1 < ns) issue(it + kDmStages - 1);
        dm_commit();
        const int st = it % kDmStages;
        const double *ms = Ms + st * kDmT * kDmSA, *bt = Bs + st * kDmK * kDmSB;
#pragma unroll
        for (int hh = 0; hh < 2; ++hh) {  // two k-steps per half: tile columns 8 hh + 2q, + 1
            double2 a[4];
#pragma unroll
            for (int f = 0; f < 4; ++f)
                a[f] = *reinterpret_cast<const double2 *>(ms + (wr + 8 * f + fr) * kDmSA + 8 * hh + 2 * fq);
#pragma unroll
            for (int s2 = 0; s2 < 2; ++s2) {
                const double *bs = bt + (8 * hh + 2 * fq + s2) * kDmSB + wc + fr;
                double b[4];
#pragma unroll
                for (int fj = 0; fj < 4; ++fj) b[fj] = bs[8 * fj];
#pragma unroll
                for (int fi = 0; fi < 4; ++fi)
#pragma unroll
                    for (int fj = 0; fj < 4; ++fj)
                        dmma(acc[fi][fj][0], acc[fi][fj][1], s2 ? a[fi].y : a[fi].x, b[fj]);
            }
        }
    }
    dm_wait<0>();
    // every old value is read before any new one is stored (a row's stores
    // would keep the next row's loads back)
    const bool pairs = V2 && (ldo % 2) == 0 && ((uintptr_t)Out % 16) == 0;
    double2 old[4][4];
#pragma unroll
    for (int fi = 0; fi < 4; ++fi)
#pragma unroll
        for (int fj = 0; fj < 4; ++fj) {
            const int j = j0 + wr + 8 * fi + fr, k = k0 + wc + 8 * fj + 2 * fq;
            old[fi][fj] = make_double2(0.0, 0.0);
            if (beta != 0.0 && j < NJ) {
                const double *o = Out + (long)j * ldo + k;
                if (pairs && k + 1 < K) {
                    old[fi][fj] = *reinterpret_cast<const double2 *>(o);
                } else {
                    if (k < K) old[fi][fj].x = o[0];
                    if (k + 1 < K) old[fi][fj].y = o[1];
                }
            }
        }
#pragma unroll
    for (int fi = 0; fi < 4; ++fi)
#pragma unroll
        for (int fj = 0; fj < 4; ++fj) {
            const int j = j0 + wr + 8 * fi + fr, k = k0 + wc + 8 * fj + 2 * fq;
            if (j >= NJ) continue;
            double *o = Out + (long)j * ldo + k;
            const double2 v = make_double2(alpha * acc[fi][fj][0] + (beta == 0.0 ? 0.0 : beta * old[fi][fj].x),
                                           alpha * acc[fi][fj][1] + (beta == 0.0 ? 0.0 : beta * old[fi][fj].y));
            if (pairs && k + 1 < K) {
                *reinterpret_cast<double2 *>(o) = v;
            } else {
                if (k < K) o[0] = v.x;
                if (k + 1 < K) o[1] = v.y;
            }
        }
}

// ------------------------------------------------------------ Lagrange multipliers
// ccpsdv3/cpsd.c:415-479.  One cluster of kLagCluster CTAs per launch; CTA r
// owns a contiguous range of columns.  Overlaps come in row-major from the
// GEMMs: M22[i][j] = <c2_i|c2_j>, M21[i][j] = <c2_i|c1_j>, M11[i][j] = <c1_i|c1_j>.
constexpr int kLagCluster = 8;
constexpr int kLagThreads = 256;

struct LagArgs {
    int ispin, ne0, ne1;
    double dte;
    const double *M22[2], *M21[2], *M11[2];
    double *s11, *s12, *s21, *s22, *st1, *X0, *X1;  // ne0^2 each, column-major
    double *lmd;                                     // [ms*ne0^2 + i + j*m]
    double *red;                                     // [cluster CTAs][2]
    int *fail;                                       // steps whose iteration did not converge
    int lb;                                          // l-chunk of the cluster kernel's row tiles
};

// Cluster of kLagClusterMax (or kLagCluster where 16 cannot be scheduled)
// CTAs; CTA r owns a block of columns.  Thread layout: row i = tid % RT
// (RT = min(m, 256)) and a block of this CTA's columns.  Per iteration the
// rows of s21, s11 and X stream through shared memory in chunks of LB
// columns l; the CTA's columns of X, s12 and st1 stay in shared memory.
constexpr int kLagClusterMax = 16;
constexpr int kLagCols = 16;

CPSD_HD size_t lagrange_cluster_smem(int m, int cl, int lb)
{
    const int per = (m + cl - 1) / cl;
    return sizeof(double) * (3 * (size_t)m * per + 3 * (size_t)m * lb);
}

// widest l-chunk (32, 16, 8 or 4) whose tiles fit in `limit` bytes; 0 if none
inline int lagrange_lb(int m, int cl, size_t limit)
{
    for (int lb = 32; lb >= 4; lb /= 2)
        if (lagrange_cluster_smem(m, cl, lb) <= limit) return lb;
    return 0;
}

__global__ void __launch_bounds__(kLagThreads) lagrange_kernel(LagArgs a)
{
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int ncta = (int)cl.num_blocks();
    const int tid = threadIdx.x;
    extern __shared__ double lsm[];
    __shared__ double shv[kLagThreads / 32];
    __shared__ int shi[kLagThreads / 32];
    const long ne02 = (long)a.ne0 * a.ne0;
    for (int ms = 0; ms < a.ispin; ++ms) {
        const int m = ms ? a.ne1 : a.ne0;
        const long kk = (long)m * m;
        if (m == 0) continue;
        const double *M22 = a.M22[ms], *M21 = a.M21[ms], *M11 = a.M11[ms];
        const double dte = a.dte;
        // s matrices, cpsd.c:420-437 (upper triangles mirrored as the reference does)
        for (long e = (long)rank * kLagThreads + tid; e < kk; e += (long)ncta * kLagThreads) {
            const int i = (int)(e % m), j = (int)(e / m);
            double v22, v21, v12, v11;
            if (i == j) {
                v22 = (1.0 - M22[(long)i * m + i]) * 0.5 / dte;
                v21 = (1.0 - M21[(long)i * m + i]) * 0.5;
                v12 = v21;
                v11 = -M11[(long)i * m + i] * 0.5 * dte;
            } else {
                const int lo = i < j ? i : j, hi = i < j ? j : i;
                v22 = -M22[(long)lo * m + hi] * 0.5 / dte;
                v21 = -M21[(long)lo * m + hi] * 0.5;   // <c2_lo|c1_hi>
                v12 = -M21[(long)hi * m + lo] * 0.5;   // <c1_lo|c2_hi>
                v11 = -M11[(long)lo * m + hi] * 0.5 * dte;
            }
            a.s22[e] = v22;
            a.s21[e] = v21;
            a.s12[e] = v12;
            a.s11[e] = v11;
            a.X0[e] = v22;  // sa0 = s22, cpsd.c:441
        }
        cl.sync();
        const int per = (m + ncta - 1) / ncta;  // columns per CTA
        const int jb = rank * per, je = min(m, jb + per);
        const int ncl = max(0, je - jb);
        const int RT = min(m, kLagThreads);
        const int nsub = kLagThreads / RT;
        const int csub = (ncl + nsub - 1) / max(nsub, 1);  // columns per thread
        const int i = tid % RT, sub = tid / RT;
        const int j0 = sub * csub;
        const bool active = (sub < nsub) && (i < m);
        const int LB = a.lb;
        double *Xs = lsm, *S12s = lsm + (long)m * per, *ST = lsm + 2L * m * per;
        double *T21 = lsm + 3L * m * per, *T11 = T21 + (long)m * LB, *TX = T11 + (long)m * LB;
        for (int e = tid; e < m * ncl; e += kLagThreads) {
            const int l = e % m, jl = e / m;
            S12s[jl * m + l] = a.s12[l + (long)(jb + jl) * m];
        }
        double *cur = a.X0, *nxt = a.X1;
        bool done = false;
        int iter = 0;
        while (!done && iter < 30) {
            ++iter;
            for (int e = tid; e < m * ncl; e += kLagThreads) {
                const int l = e % m, jl = e / m;
                Xs[jl * m + l] = cur[l + (long)(jb + jl) * m];
            }
            // sa1 = s22 + s21 sa0 + sa0 s12 ; st1 = s11 sa0   (cpsd.c:444-462);
            // the partial sa1 waits in nxt for the second product
            for (int cb = 0; cb < csub; cb += kLagCols) {
                double t1[kLagCols], t2[kLagCols], t3[kLagCols];
#pragma unroll
                for (int q = 0; q < kLagCols; ++q) t1[q] = t2[q] = t3[q] = 0.0;
                for (int l0 = 0; l0 < m; l0 += LB) {
                    const int lw = min(LB, m - l0);
                    __syncthreads();  // previous tile consumed (and Xs written)
                    for (int e = tid; e < m * lw; e += kLagThreads) {
                        const int ii = e % m, ll = e / m;
                        const long g = ii + (long)(l0 + ll) * m;
                        T21[ll * m + ii] = a.s21[g];
                        T11[ll * m + ii] = a.s11[g];
                        TX[ll * m + ii] = cur[g];
                    }
                    __syncthreads();
                    if (active) {
                        for (int ll = 0; ll < lw; ++ll) {
                            const int l = l0 + ll;
                            const double a21 = T21[ll * m + i], a11 = T11[ll * m + i], xil = TX[ll * m + i];
#pragma unroll
                            for (int q = 0; q < kLagCols; ++q) {
                                const int jl = j0 + cb + q;
                                if (cb + q < csub && jl < ncl) {
                                    const double xlj = Xs[jl * m + l];
                                    t1[q] = fma(a21, xlj, t1[q]);
                                    t2[q] = fma(xil, S12s[jl * m + l], t2[q]);
                                    t3[q] = fma(a11, xlj, t3[q]);
                                }
                            }
                        }
                    }
                }
                if (active) {
#pragma unroll
                    for (int q = 0; q < kLagCols; ++q) {
                        const int jl = j0 + cb + q;
                        if (cb + q < csub && jl < ncl) {
                            const int j = jb + jl;
                            nxt[i + (long)j * m] = t2[q] + (t1[q] + a.s22[i + (long)j * m]);
                            ST[jl * m + i] = t3[q];
                        }
                    }
                }
            }
            // sa1 += sa0 st1 (cpsd.c:463-468); st1 = sa1 - sa0 (:469-470)
            double bestv = -1.0;
            int besti = 0x7fffffff;
            for (int cb = 0; cb < csub; cb += kLagCols) {
                double t4[kLagCols];
#pragma unroll
                for (int q = 0; q < kLagCols; ++q) t4[q] = 0.0;
                for (int l0 = 0; l0 < m; l0 += LB) {
                    const int lw = min(LB, m - l0);
                    __syncthreads();
                    for (int e = tid; e < m * lw; e += kLagThreads) {
                        const int ii = e % m, ll = e / m;
                        TX[ll * m + ii] = cur[ii + (long)(l0 + ll) * m];
                    }
                    __syncthreads();
                    if (active) {
                        for (int ll = 0; ll < lw; ++ll) {
                            const int l = l0 + ll;
                            const double xil = TX[ll * m + i];
#pragma unroll
                            for (int q = 0; q < kLagCols; ++q) {
                                const int jl = j0 + cb + q;
                                if (cb + q < csub && jl < ncl) t4[q] = fma(xil, ST[jl * m + l], t4[q]);
                            }
                        }
                    }
                }
                if (active) {
#pragma unroll
                    for (int q = 0; q < kLagCols; ++q) {
                        const int jl = j0 + cb + q;
                        if (cb + q < csub && jl < ncl) {
                            const long f = i + (long)(jb + jl) * m;
                            const double sa1 = t4[q] + nxt[f];
                            nxt[f] = sa1;
                            const double d = sa1 - cur[f];
                            a.st1[f] = d;
                            const double ad = fabs(d);
                            if (ad > bestv || (ad == bestv && f < besti)) {
                                bestv = ad;
                                besti = (int)f;
                            }
                        }
                    }
                }
            }
            // block argmax (first index of the largest |st1|, as idamax)
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                double ov = __shfl_xor_sync(0xffffffffu, bestv, o);
                int oi = __shfl_xor_sync(0xffffffffu, besti, o);
                if (ov > bestv || (ov == bestv && oi < besti)) {
                    bestv = ov;
                    besti = oi;
                }
            }
            if ((tid & 31) == 0) {
                shv[tid >> 5] = bestv;
                shi[tid >> 5] = besti;
            }
            __syncthreads();
            if (tid == 0) {
                for (int w = 1; w < kLagThreads / 32; ++w)
                    if (shv[w] > bestv || (shv[w] == bestv && shi[w] < besti)) {
                        bestv = shv[w];
                        besti = shi[w];
                    }
                a.red[2 * rank] = bestv;
                a.red[2 * rank + 1] = (double)besti;
            }
            cl.sync();
            // every CTA reduces the cluster's candidates in the same order
            double gv = -1.0;
            long gi = 0x7fffffff;
            for (int r = 0; r < ncta; ++r) {
                const double v = a.red[2 * r];
                const long ix = (long)a.red[2 * r + 1];
                if (v > gv || (v == gv && ix < gi)) {
                    gv = v;
                    gi = ix;
                }
            }
            // idamax returns an index in 1..kk even when every entry is NaN
            // (then no comparison succeeds and it returns 1); the sentinel
            // must never reach the read below
            if (gi < 0 || gi >= kk) gi = 0;
            // the reference reads st1 at idamax's 1-based result (cpsd.c:471):
            // the element after the largest; past the end of st1 lies sa1
            const long nx = gi + 1;
            const double adiff = fabs(nx < ne02 ? a.st1[nx] : nxt[nx - ne02]);
            done = adiff < 1e-15;
            cl.sync();
            if (!done) {
                double *t = cur;
                cur = nxt;
                nxt = t;
            }
        }
        if (!done && rank == 0 && tid == 0) atomicAdd(a.fail, 1);
        // lmd = sa1, cpsd.c:478 (after 30 unconverged iterations sa1 was swapped into cur)
        const double *fin = done ? nxt : cur;
        for (int e = tid; e < m * ncl; e += kLagThreads) {
            const int ii = e % m, j = jb + e / m;
            a.lmd[ms * ne02 + ii + (long)j * m] = fin[ii + (long)j * m];
        }
        cl.sync();
    }
}

// up to this many bands per spin: small.cuh
constexpr int kLagSmallMax = 32;

// largest |d| over a warp with the smallest index among equals, as idamax
// (NaN never wins; 0x7fffffff where every entry was NaN); all lanes get the result
CPSD_D void combine_argmax(unsigned h, unsigned l, unsigned idx, unsigned &hi, unsigned &lo, int &at)
{
    hi = __reduce_max_sync(0xffffffffu, h);
    lo = __reduce_max_sync(0xffffffffu, h == hi ? l : 0u);
    at = (int)__reduce_min_sync(0xffffffffu, (h == hi && l == lo) ? idx : 0x7fffffffu);
}
CPSD_D void warp_argmax(double ad, int idx, unsigned &hi, unsigned &lo, int &at)
{
    const bool ok = ad >= 0.0;  // false for NaN and for "no entry" (-1)
    const unsigned long long k = ok ? (unsigned long long)__double_as_longlong(ad) : 0ull;
    combine_argmax((unsigned)(k >> 32), (unsigned)k, ok ? (unsigned)idx : 0x7fffffffu, hi, lo, at);
}

// ------------------------------------------------- Lagrange, 2-D tiles
// lagrange_tile_kernel: the same fixed point as lagrange_kernel (cpsd.c:
// 439-478, including the idamax read and the 30-iteration limit) for 33 to
// 128 bands per spin, on a cluster of 4 x 4 CTAs.  CTA (p, q) owns the tile
// rows I_p x columns J_q (T = 8 MT of each, zero padded) of sa0 and sa1, keeps
// its constant panels s21[I_p, :], s11[I_p, :] and s12[:, J_q]' in shared
// memory and forms its products on the FP64 tensor cores (8 x 8 tiles, a warp
// has up to two of one row).  The CTAs push what the others need into their
// shared memory: st1 = s11 sa0 to the CTAs of its column after the first
// phase, the new sa0 to those of its row and its column after the second, so
// every operand is read from local memory:
//   phase 1: t = s22 + s21 sa0 + sa0 s12, st1 = s11 sa0;   cluster barrier;
//   phase 2: sa1 = t + sa0 st1 (sa0's rows still in registers), st1 = sa1 -
//            sa0, the tile's argmax of |st1|;              cluster barrier;
// then every CTA reduces the 16 candidates and reads the element after the
// maximum, as the reference does.  All panels are stored with k along the row
// (the column panels transposed), 8 mod 16 reals apart: fragment loads of two
// k-steps are 16 bytes and free of bank conflicts.
//
// Bound at 128 bands: the FP64 pipe of 16 SMs, 8,192 cycles (4.2 us) an
// iteration; a solve takes 131 us with CUDA-core products and panels gathered
// from the peers, 70 us here (40 bands at 32^3: ten steps 1.26 -> 1.10 ms).
constexpr int kLagTileGrid = 4;  // 4 x 4 CTAs
constexpr int kLagTileMax = 128;
constexpr int lag_tile_ld(int mt) { return 32 * mt + 8; }

inline int lag_tile_mt(int m) { return (m + 31) / 32; }  // tiles of 8 along a CTA's edge
inline size_t lagrange_tile_smem(int m)
{
    const int mt = lag_tile_mt(m);
    // S21r, S11r, S12c, Xr, Xc, STc
    return sizeof(double) * 6 * (size_t)(8 * mt) * lag_tile_ld(mt);
}

template <int MT>
__global__ void __launch_bounds__(kLagThreads) lagrange_tile_kernel(LagArgs a)
{
    constexpr int T = 8 * MT, MP = 4 * T, LD = lag_tile_ld(MT), KB = MP / 8, CPW = (MT + 1) / 2, G = kLagTileGrid;
    cg::cluster_group cl = cg::this_cluster();
    const int rank = (int)cl.block_rank();
    const int p = rank / G, q = rank % G;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, fr = lane >> 2, fq = lane & 3;
    extern __shared__ __align__(16) double tsm[];
    __shared__ unsigned slot[G * G][4];  // every CTA's candidate
    __shared__ unsigned wslot[kLagThreads / 32][4];
    const long ne02 = (long)a.ne0 * a.ne0;
    double *S21r = tsm, *S11r = S21r + T * LD, *S12c = S11r + T * LD, *Xr = S12c + T * LD, *Xc = Xr + T * LD,
           *STc = Xc + T * LD;
    // this warp's tiles: row tile wi, column tiles wj .. wj + CPW - 1
    const int wi = warp >> 1, wj = (warp & 1) * CPW;
    const bool wact = wi < MT;
    const int i = 8 * wi + fr;  // this lane's row of the CTA's tile
    double *xr_to[G], *xc_to[G], *st_to[G];
#pragma unroll
    for (int g = 0; g < G; ++g) {
        xr_to[g] = cl.map_shared_rank(Xr, p * G + g);
        xc_to[g] = cl.map_shared_rank(Xc, g * G + q);
        st_to[g] = cl.map_shared_rank(STc, g * G + q);
    }
    for (int ms = 0; ms < a.ispin; ++ms) {
        const int m = ms ? a.ne1 : a.ne0;
        const long kk = (long)m * m;
        if (m == 0) continue;
        const int i0 = p * T, j0 = q * T;
        const double *M22 = a.M22[ms], *M21 = a.M21[ms], *M11 = a.M11[ms];
        const double dte = a.dte;
        // s matrices, cpsd.c:420-437 (upper triangles mirrored as the reference does)
        auto s22 = [&](int r, int c) {
            if (r >= m || c >= m) return 0.0;
            return r == c ? (1.0 - M22[(long)r * m + r]) * 0.5 / dte : -M22[(long)min(r, c) * m + max(r, c)] * 0.5 / dte;
        };
        for (int e = tid; e < T * MP; e += kLagThreads) {
            const int r = e / MP, l = e % MP, ri = i0 + r, cj = j0 + r;
            double v21 = 0.0, v11 = 0.0, v12 = 0.0;
            if (l < m && ri < m) {
                const int lo = min(ri, l), hi = max(ri, l);
                v21 = ri == l ? (1.0 - M21[(long)ri * m + ri]) * 0.5 : -M21[(long)lo * m + hi] * 0.5;  // <c2_lo|c1_hi>
                v11 = -M11[(long)lo * m + hi] * 0.5 * dte;
            }
            if (l < m && cj < m) {
                const int lo = min(cj, l), hi = max(cj, l);
                v12 = cj == l ? (1.0 - M21[(long)cj * m + cj]) * 0.5 : -M21[(long)hi * m + lo] * 0.5;  // <c1_lo|c2_hi>
            }
            S21r[r * LD + l] = v21;
            S11r[r * LD + l] = v11;
            S12c[r * LD + l] = v12;
            Xr[r * LD + l] = s22(ri, l);  // sa0 = s22, cpsd.c:441
            Xc[r * LD + l] = s22(l, cj);
        }
        double c22[CPW][2], x[CPW][2];
#pragma unroll
        for (int u = 0; u < CPW; ++u)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const bool ok = wact && wj + u < MT;
                x[u][e] = c22[u][e] = ok ? s22(i0 + i, j0 + 8 * (wj + u) + 2 * fq + e) : 0.0;
            }
        bool done = false;
        int iter = 0;
        cl.sync();  // every CTA's panels are in place (and, for spin 1, spin 0's reads done)
        while (!done && iter < 30) {
            ++iter;
            double2 xa[KB];
            double part[CPW][2];
            if (wact) {
                const double *xrow = Xr + i * LD + 2 * fq, *s21 = S21r + i * LD + 2 * fq, *s11 = S11r + i * LD + 2 * fq;
                double t1[CPW][2] = {}, t2[CPW][2] = {}, st[CPW][2] = {};
#pragma unroll
                for (int k = 0; k < KB; ++k) {
                    xa[k] = *reinterpret_cast<const double2 *>(xrow + 8 * k);
                    const double2 a21 = *reinterpret_cast<const double2 *>(s21 + 8 * k);
                    const double2 a11 = *reinterpret_cast<const double2 *>(s11 + 8 * k);
#pragma unroll
                    for (int u = 0; u < CPW; ++u) {
                        if (wj + u >= MT) break;
                        const int o = (8 * (wj + u) + fr) * LD + 8 * k + 2 * fq;
                        const double2 xb = *reinterpret_cast<const double2 *>(Xc + o);
                        const double2 b12 = *reinterpret_cast<const double2 *>(S12c + o);
                        dmma(st[u][0], st[u][1], a11.x, xb.x);
                        dmma(t1[u][0], t1[u][1], a21.x, xb.x);
                        dmma(t2[u][0], t2[u][1], xa[k].x, b12.x);
                        dmma(st[u][0], st[u][1], a11.y, xb.y);
                        dmma(t1[u][0], t1[u][1], a21.y, xb.y);
                        dmma(t2[u][0], t2[u][1], xa[k].y, b12.y);
                    }
                }
#pragma unroll
                for (int u = 0; u < CPW; ++u) {
                    if (wj + u >= MT) break;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        part[u][e] = t2[u][e] + (t1[u][e] + c22[u][e]);
                        const int o = (8 * (wj + u) + 2 * fq + e) * LD + i0 + i;
#pragma unroll
                        for (int g = 0; g < G; ++g) st_to[g][o] = st[u][e];
                    }
                }
            }
            cl.sync();  // every st1 = s11 sa0 has arrived; nobody reads Xr or Xc any more
            double bestv = -1.0;
            int besti = 0x7fffffff;
            if (wact) {
#pragma unroll
                for (int u = 0; u < CPW; ++u) {
                    if (wj + u >= MT) break;
                    double t4[2] = {0.0, 0.0};
#pragma unroll
                    for (int k = 0; k < KB; ++k) {
                        const double2 sb =
                            *reinterpret_cast<const double2 *>(STc + (8 * (wj + u) + fr) * LD + 8 * k + 2 * fq);
                        dmma(t4[0], t4[1], xa[k].x, sb.x);
                        dmma(t4[0], t4[1], xa[k].y, sb.y);
                    }
                    const int jl = 8 * (wj + u) + 2 * fq;
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        // sa1 = s22, += s21 sa0, += sa0 s12, += sa0 st1 (cpsd.c:463-470)
                        const double v = t4[e] + part[u][e];
                        const int ri = i0 + i, cj = j0 + jl + e;
                        if (ri < m && cj < m) {
                            const double d = v - x[u][e], ad = fabs(d);
                            const int f = ri + cj * m;
                            a.st1[f] = d;
                            if (f == 0) a.X1[0] = v;
                            if (ad > bestv || (ad == bestv && f < besti)) {
                                bestv = ad;
                                besti = f;
                            }
                        }
                        x[u][e] = v;
#pragma unroll
                        for (int g = 0; g < G; ++g) xc_to[g][(jl + e) * LD + i0 + i] = v;
                    }
#pragma unroll
                    for (int g = 0; g < G; ++g)
                        *reinterpret_cast<double2 *>(xr_to[g] + i * LD + j0 + jl) = make_double2(x[u][0], x[u][1]);
                }
            }
            // tile argmax (first column-major index of the largest |st1|, as idamax)
            unsigned hi, lo;
            int at;
            warp_argmax(bestv, besti, hi, lo, at);
            if (lane == 0) {
                wslot[warp][0] = hi;
                wslot[warp][1] = lo;
                wslot[warp][2] = (unsigned)at;
            }
            __syncthreads();
            if (warp == 0) {
                constexpr int NW = kLagThreads / 32;
                combine_argmax(lane < NW ? wslot[lane][0] : 0u, lane < NW ? wslot[lane][1] : 0u,
                               lane < NW ? wslot[lane][2] : 0x7fffffffu, hi, lo, at);
                if (lane < G * G) {  // to every CTA
                    unsigned *to = cl.map_shared_rank(&slot[0][0], lane) + 4 * rank;
                    to[0] = hi;
                    to[1] = lo;
                    to[2] = (unsigned)at;
                }
            }
            cl.sync();  // every candidate, difference and new sa0 is in place
            combine_argmax(lane < G * G ? slot[lane][0] : 0u, lane < G * G ? slot[lane][1] : 0u,
                           lane < G * G ? slot[lane][2] : 0x7fffffffu, hi, lo, at);
            // idamax returns an index in 1..kk even when every entry is NaN
            if (at < 0 || at >= kk) at = 0;
            // the reference reads st1 at idamax's 1-based result (cpsd.c:471):
            // the element after the largest; past the end of st1 lies sa1
            const long nx = (long)at + 1;
            const double adiff = fabs(__ldcg(nx < ne02 ? a.st1 + nx : a.X1 + (nx - ne02)));
            done = adiff < 1e-15;
            // the candidates and differences are written again only after the
            // next iteration's first barrier
        }
        if (!done && rank == 0 && tid == 0) atomicAdd(a.fail, 1);
        // lmd = the last sa1 (cpsd.c:478)
        if (wact)
#pragma unroll
            for (int u = 0; u < CPW; ++u)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int ri = i0 + i, cj = j0 + 8 * (wj + u) + 2 * fq + e;
                    if (wj + u < MT && ri < m && cj < m) a.lmd[ms * ne02 + ri + (long)cj * m] = x[u][e];
                }
        cl.sync();  // the panels and slots are reused by the next spin; no CTA leaves before its peers' stores
    }
}

// ------------------------------------------------------------ energies
// Every partial sum of the energies in one launch (five before; they are
// independent and each a few microseconds): block ranges in the order of
// EnergyArgs' counts, every block a fixed-order sum.
struct EnergyArgs {
    int pblocks, bblocks, gblocks, eblocks, nblocks;  // packed, per band, grid, Ewald (ions - 1), nonlocal
    int npw, nb, ispin, nion, nsh, nproj;
    long ldc, n3;
    const double *w, *tg, *vg, *vc, *dn, *xce, *xcp, *r1, *rcell, *zv, *beta, *vnlnrm_p;
    const int *katm;
    const cx<double> *s, *dng, *vall, *c1, *c2;
    double rcut, scal2;
    double *ppart;  // [3][pblocks]: k-space Ewald, Hartree, local (cpsd.c:520-526, 548-554, 590)
    double *bpart;  // [2][nb][bblocks]: eke_b (cpsd.c:574-586), dc_b (:650-659)
    double *gpart;  // [2][gblocks]: exc, pxc (cpsd.c:557-570)
    double *epart;  // [nion - 1]: real-space Ewald of the pairs (ii, jj > ii)
    double *npart;  // [nblocks]: nonlocal energy of the last step's projections (cpsd.c:593-634)
};

__global__ void __launch_bounds__(256) energy_terms_kernel(const __grid_constant__ EnergyArgs a)
{
    __shared__ double sh[32];
    const int tid = threadIdx.x;
    int blk = blockIdx.x;
    if (blk < a.pblocks) {
        double e0 = 0, e1 = 0, e2 = 0;
        for (int p = blk * 256 + tid; p < a.npw; p += a.pblocks * 256) {
            const double ww = a.w[p];
            const cx<double> sv = a.s[p], d = a.dng[p], va = a.vall[p];
            e0 += ww * (sv.x * sv.x + sv.y * sv.y) * a.vg[p];
            e1 += ww * (d.x * d.x + d.y * d.y) * a.vc[p];
            e2 += ww * (va.x * d.x + va.y * d.y);
        }
        const double r0 = block_sum<256>(e0, sh), r1 = block_sum<256>(e1, sh), r2 = block_sum<256>(e2, sh);
        if (tid == 0) {
            a.ppart[blk] = r0;
            a.ppart[a.pblocks + blk] = r1;
            a.ppart[2 * a.pblocks + blk] = r2;
        }
        return;
    }
    blk -= a.pblocks;
    if (blk < a.bblocks * a.nb) {
        const int b = blk / a.bblocks, x = blk % a.bblocks;
        const cx<double> *c1 = a.c1 + (long)b * a.ldc, *c2 = a.c2 + (long)b * a.ldc;
        double ek = 0, dc = 0;
        for (int p = x * 256 + tid; p < a.npw; p += a.bblocks * 256) {
            const double ww = a.w[p];
            const cx<double> u = c1[p], v = c2[p];
            ek += ww * a.tg[p] * (u.x * u.x + u.y * u.y);
            const double dx = v.x - u.x, dy = v.y - u.y;
            dc += ww * (dx * dx + dy * dy);
        }
        const double r0 = block_sum<256>(ek, sh), r1 = block_sum<256>(dc, sh);
        if (tid == 0) {
            a.bpart[(long)b * a.bblocks + x] = r0;
            a.bpart[((long)a.nb + b) * a.bblocks + x] = r1;
        }
        return;
    }
    blk -= a.bblocks * a.nb;
    if (blk < a.gblocks) {
        double ex = 0, px = 0;
        for (long r = (long)blk * 256 + tid; r < a.n3; r += (long)a.gblocks * 256) {
            const double d0 = a.dn[r], e = a.xce[r];
            ex += d0 * e;
            px += d0 * a.xcp[r];
            if (a.ispin == 2) {
                const double d1 = a.dn[a.n3 + r];
                ex += d1 * e;
                px += d1 * a.xcp[a.n3 + r];
            }
        }
        const double r0 = block_sum<256>(ex, sh), r1 = block_sum<256>(px, sh);
        if (tid == 0) {
            a.gpart[blk] = r0;
            a.gpart[a.gblocks + blk] = r1;
        }
        return;
    }
    blk -= a.gblocks;
    if (blk < a.eblocks) {
        // real-space Ewald, cpsd.c:527-545 (A&S 7.1.28 erfc, cpsd.c:11-17): the
        // pairs (ii, jj > ii) over the nsh image cells, a (pair, image) per thread
        const double B1 = 0.0705230784, B2 = 0.0422820123, B3 = 0.0092705272;
        const double B4 = 0.0001520143, B5 = 0.0002765672, B6 = 0.0000430638;
        const int ii = blk;
        const long cnt = (long)(a.nion - 1 - ii) * a.nsh;
        double ew = 0.0;
        for (long e = tid; e < cnt; e += 256) {
            const int jj = ii + 1 + (int)(e / a.nsh);
            const int l = (int)(e % a.nsh);
            const double dx = a.r1[3 * ii] - a.r1[3 * jj];
            const double dy = a.r1[1 + 3 * ii] - a.r1[1 + 3 * jj];
            const double dz = a.r1[2 + 3 * ii] - a.r1[2 + 3 * jj];
            const double zz = a.zv[a.katm[ii]] * a.zv[a.katm[jj]];
            const double x = a.rcell[l] + dx, y = a.rcell[l + a.nsh] + dy, z = a.rcell[l + 2 * a.nsh] + dz;
            const double r = sqrt(x * x + y * y + z * z);
            const double w = r / a.rcut;
            const double aa = (1.0 + w * (B1 + w * (B2 + w * (B3 + w * (B4 + w * (B5 + w * B6))))));
            const double erfc = 1.0 / (aa * aa * aa * aa);
            ew += zz * (erfc * erfc * erfc * erfc) / r;
        }
        const double t = block_sum<256>(ew, sh);
        if (tid == 0) a.epart[ii] = t;
        return;
    }
    blk -= a.eblocks;
    {
        double en = 0.0;
        const long cnt = (long)a.nproj * a.nb;
        for (long e = (long)blk * 256 + tid; e < cnt; e += (long)a.nblocks * 256) {
            const double sw = a.beta[e];
            en += sw * sw * a.scal2 / a.vnlnrm_p[e / a.nb];
        }
        const double t = block_sum<256>(en, sh);
        if (tid == 0) a.npart[blk] = t;
    }
}

// hml from M[i][j] = <c1_i|cpsi_j> (row-major per spin), with the reference's
// mirroring and eorbit reads (cpsd.c:497-515); one thread.
struct FinalArgs {
    int ispin, ne0, ne1, nion, nb, inner;
    int pblocks, bblocks, gblocks, nblocks;
    const double *ppart, *bpart, *gpart, *npart;
    const double *Mh[2];
    double *hml;
    const double *ewald_part;  // real-space Ewald sum per ion
    double scal2, omega, dv, cewald, dt, dte;
    double *E;  // in: E[0] previous energy; out: E[0..9], E[10] deltae, E[11] deltac
};

// One block of kFinalThreads: every sum is a fixed-order block reduction, so
// the energies are bitwise reproducible run to run.
constexpr int kFinalThreads = 256;

__global__ void __launch_bounds__(kFinalThreads) final_energy_kernel(FinalArgs a)
{
    __shared__ double sh[32];
    const int tid = threadIdx.x;
    const long ne02 = (long)a.ne0 * a.ne0;
    // hml (cpsd.c:497-513): the upper triangle is -<c1_i|cpsi_j>, mirrored; the
    // mirror and eorbit read hml at the spin-0 offset for both spins
    double eo = 0.0;
    for (int ms = 0; ms < a.ispin; ++ms) {
        const int m = ms ? a.ne1 : a.ne0;
        double *H = a.hml + ms * ne02;
        const double *M = a.Mh[ms];
        for (int e = tid; e < m * m; e += kFinalThreads) {
            const int i = e % m, j = e / m;
            if (i <= j) H[i + j * m] = -M[(long)i * m + j];
        }
        __syncthreads();
        for (int e = tid; e < m * m; e += kFinalThreads) {
            const int i = e % m, j = e / m;
            if (i < j) H[j + i * m] = a.hml[i + j * m];
        }
        for (int i = tid; i < m; i += kFinalThreads) eo += a.hml[i + i * m];
        __syncthreads();
    }
    double eorbit = block_sum<kFinalThreads>(eo, sh);
    // single-field packed terms
    double t[3];
    for (int q = 0; q < 3; ++q) {
        double v = 0.0;
        for (int k = tid; k < a.pblocks; k += kFinalThreads) v += a.ppart[q * a.pblocks + k];
        t[q] = block_sum<kFinalThreads>(v, sh);
    }
    // real-space Ewald: per-ion partials, summed in ion order
    double eion_real = 0.0;
    if (tid == 0)
        for (int ii = 0; ii < a.nion; ++ii) eion_real += a.ewald_part[ii];
    // xc
    double ex = 0.0, px = 0.0;
    for (int k = tid; k < a.gblocks; k += kFinalThreads) {
        ex += a.gpart[k];
        px += a.gpart[a.gblocks + k];
    }
    double exc = block_sum<kFinalThreads>(ex, sh);
    double pxc = block_sum<kFinalThreads>(px, sh);
    // kinetic and deltac per band
    double ek = 0.0, dcmax = 0.0;
    for (int b = tid; b < a.nb; b += kFinalThreads) {
        double s1 = 0.0, s2 = 0.0;
        for (int k = 0; k < a.bblocks; ++k) {
            s1 += a.bpart[(long)b * a.bblocks + k];
            s2 += a.bpart[((long)a.nb + b) * a.bblocks + k];
        }
        ek += s1;
        dcmax = fmax(dcmax, s2);
    }
    double eke = block_sum<kFinalThreads>(ek, sh);
    // max over threads (order-independent)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) dcmax = fmax(dcmax, __shfl_xor_sync(0xffffffffu, dcmax, o));
    __syncthreads();
    if ((tid & 31) == 0) sh[tid >> 5] = dcmax;
    __syncthreads();
    double dc = 0.0;
    if (tid == 0)
        for (int i = 0; i < kFinalThreads / 32; ++i) dc = fmax(dc, sh[i]);
    __syncthreads();
    // nonlocal energy from the last step's projections, cpsd.c:593-634
    double en = 0.0;
    for (int k = tid; k < a.nblocks; k += kFinalThreads) en += a.npart[k];
    double enl = block_sum<kFinalThreads>(en, sh);
    if (tid != 0) return;
    if (a.ispin == 1) eorbit *= 2;
    const double eion = t[0] * 0.5 * a.scal2 + a.cewald + eion_real;
    const double ehartr = t[1] * a.omega * 0.5;
    const double elocal = t[2];
    if (a.ispin == 1) {
        exc += exc;
        pxc += pxc;
    }
    exc *= a.dv;
    pxc *= a.dv;
    if (a.ispin == 1) eke = 2 * eke;
    if (a.ispin == 1) enl = 2 * enl;
    const double eold = a.E[0];
    a.E[0] = eorbit + eion + exc - ehartr - pxc;
    a.E[1] = eorbit;
    a.E[2] = ehartr;
    a.E[3] = exc;
    a.E[4] = eion;
    a.E[5] = eke;
    a.E[6] = elocal;
    a.E[7] = enl;
    a.E[8] = 2.0 * ehartr;
    a.E[9] = pxc;
    a.E[10] = (a.E[0] - eold) / (a.dt * a.inner);
    a.E[11] = dc / a.dte;
}

// ------------------------------------------------------------ epilogue eigenpairs
// ccpsdv3/main.c:470-481: per spin, dsyev('V','U') of hml, then eigsrt
// (ccpsdv3/eigsrt.c:9-36: selection sort into descending order, ties to the
// later index, eigenvector columns moved with their values).  Here: cyclic
// Jacobi, rounds of the round-robin pair order (n/2 disjoint pairs per
// round, n padded to even with an idle index), so one round's rotations run
// in parallel: rows of A, then columns of A and V.  Rotation and thresholds
// follow the classical scheme (Rutishauser; as in Numerical Recipes
// "jacobi"): t = sgn(theta) / (|theta| + sqrt(theta^2 + 1)), theta =
// (a_qq - a_pp) / (2 a_pq); in the first sweeps only |a_pq| above 0.2 S / n^2
// (S = sum of |a_ij|, i < j) rotate; from the fifth sweep on an a_pq that
// no longer changes a_pp or a_qq (|a_pp| + 100 |a_pq| == |a_pp|, the same
// for a_qq) is set to zero.  The sweeps end when S is zero.  One CTA per
// spin.  A round is two dependent phases (the rotations, then every 2 x 2 block
// of A by a row and a column rotation), so its time is latency: A and V
// (column-major) live in shared memory where they fit (both up to 110 bands, A
// alone up to 157), columns an odd stride apart, and up to 32 bands take 256
// threads (a barrier of 8 warps instead of 32).
constexpr int kEigMaxSweeps = 60;

struct EigArgs {
    const double *hml;   // per spin ms at hml + ms*ne0*ne0, column-major, ld ne[ms]; upper triangle read
    int ne[2], ne0;
    double *A, *V;       // workspace: per spin ne0*ne0 each
    double *eig;         // eig[ms*ne0 + i], descending
    double *vec;         // eigenvectors in hml's layout, columns in eig's order
    int *sweeps;         // per spin: sweeps run (kEigMaxSweeps + 1: not converged)
};

constexpr size_t kEigSmemMax = 200 << 10;
CPSD_HD int eig_ld(int n) { return n | 1; }
// matrices held in shared memory: 2 (A and V), 1 (A) or 0
inline int eig_in_smem(int n)
{
    const size_t one = sizeof(double) * (size_t)n * eig_ld(n);
    return 2 * one <= kEigSmemMax ? 2 : (one <= kEigSmemMax ? 1 : 0);
}

template <int kEigThreads>
__global__ void __launch_bounds__(kEigThreads) jacobi_eig_kernel(EigArgs a, int in_smem)
{
    extern __shared__ double eig_sm[];
    __shared__ double rc[128], rs[128], rd0[128], rd1[128], red[32];
    __shared__ int rp[128], rq[128], rk[128], perm[256];
    __shared__ double sum_off;
    const int ms = blockIdx.x, n = a.ne[ms], tid = threadIdx.x;
    if (n <= 0) return;
    const long off = (long)ms * a.ne0 * a.ne0;
    const double *H = a.hml + off;
    const int la = in_smem >= 1 ? eig_ld(n) : n, lv = in_smem == 2 ? eig_ld(n) : n;  // column strides
    double *A = in_smem >= 1 ? eig_sm : a.A + off;
    double *V = in_smem == 2 ? eig_sm + (long)n * la : a.V + off;
    for (long e = tid; e < (long)n * n; e += kEigThreads) {
        const int i = (int)(e % n), j = (int)(e / n);
        A[i + (long)j * la] = (i <= j) ? H[i + (long)j * n] : H[j + (long)i * n];
        V[i + (long)j * lv] = (i == j) ? 1.0 : 0.0;
    }
    __syncthreads();
    const int np = n + (n & 1), half = np / 2, m1 = np - 1;
    // a thread's first block (k, l) and V entry (l, i), and its strides
    const int k0 = tid / half, l0 = tid % half, dk = kEigThreads / half, dl = kEigThreads % half;
    const int l1 = tid / n, i1 = tid % n, dv = kEigThreads / n, di = kEigThreads % n;
    int sweep = 1;
    for (; sweep <= kEigMaxSweeps; ++sweep) {
        // S = sum_{i<j} |a_ij|
        double v = 0.0;
        for (long e = tid; e < (long)n * n; e += kEigThreads) {
            const int i = (int)(e % n), j = (int)(e / n);
            if (i < j) v += fabs(A[i + (long)j * la]);
        }
        v = block_sum<kEigThreads>(v, red);
        if (tid == 0) sum_off = v;
        __syncthreads();
        const double S = sum_off;
        if (S == 0.0) break;
        const double tresh = (sweep < 4) ? 0.2 * S / ((double)n * n) : 0.0;
        for (int r = 0; r < m1; ++r) {
            if (tid < half) {
                int p, q;
                if (tid == 0) {
                    p = 0;
                    q = 1 + r;
                } else {
                    p = 1 + (r + tid < m1 ? r + tid : r + tid - m1);
                    q = 1 + (r >= tid ? r - tid : r - tid + m1);
                }
                if (p > q) {
                    const int x = p;
                    p = q;
                    q = x;
                }
                double c = 1.0, s = 0.0, d0 = 0.0, d1 = 0.0;
                int kind = 0;  // 0: identity, 1: rotated, 2: a_pq set to zero
                if (q < n) {
                    const double app = A[p + (long)p * la], aqq = A[q + (long)q * la], apq = A[p + (long)q * la];
                    const double g = 100.0 * fabs(apq);
                    if (sweep > 4 && fabs(app) + g == fabs(app) && fabs(aqq) + g == fabs(aqq)) {
                        kind = 2;
                    } else if (fabs(apq) > tresh && apq != 0.0) {
                        const double h = aqq - app;
                        double t;
                        if (fabs(h) + g == fabs(h)) {
                            t = apq / h;
                        } else {
                            const double theta = 0.5 * h / apq;
                            t = 1.0 / (fabs(theta) + sqrt(1.0 + theta * theta));
                            if (theta < 0.0) t = -t;
                        }
                        c = rsqrt(1.0 + t * t);
                        s = t * c;
                        kind = 1;
                        d0 = app - t * apq;
                        d1 = aqq + t * apq;
                    }
                }
                rp[tid] = p;
                rq[tid] = q;  // n: the idle index of an odd n
                rk[tid] = kind;
                rc[tid] = c;
                rs[tid] = s;
                rd0[tid] = d0;
                rd1[tid] = d1;
            }
            __syncthreads();
            // A <- P^T A P, one 2 x 2 block (rows of pair k, columns of pair l)
            // per thread: the rows' rotation, then the columns'.  A rotation's
            // own block gets a_pp - t a_pq, a_qq + t a_pq and exact zeros.
            for (int e = tid, k = k0, l = l0; e < half * half; e += kEigThreads) {
                const int p = rp[k], q = rq[k], u = rp[l], w = rq[l];
                double *Au = A + (long)u * la, *Aw = A + (long)w * la;
                if (k == l) {
                    if (rk[k] == 1) {
                        Au[p] = rd0[k];
                        Aw[q] = rd1[k];
                    }
                    if (rk[k] != 0) {
                        Aw[p] = 0.0;
                        Au[q] = 0.0;
                    }
                } else if (rk[k] == 1 || rk[l] == 1) {
                    const double c = rc[k], sn = rs[k], c2 = rc[l], s2 = rs[l];
                    const bool hq = q < n, hw = w < n;
                    const double pu = Au[p], qu = hq ? Au[q] : 0.0, pw = hw ? Aw[p] : 0.0, qw = (hq && hw) ? Aw[q] : 0.0;
                    const double x0 = c * pu - sn * qu, x1 = sn * pu + c * qu;  // column u
                    const double y0 = c * pw - sn * qw, y1 = sn * pw + c * qw;  // column w
                    Au[p] = c2 * x0 - s2 * y0;
                    if (hq) Au[q] = c2 * x1 - s2 * y1;
                    if (hw) Aw[p] = s2 * x0 + c2 * y0;
                    if (hq && hw) Aw[q] = s2 * x1 + c2 * y1;
                }
                k += dk;
                l += dl;
                if (l >= half) {
                    l -= half;
                    ++k;
                }
            }
            // V <- V P
            for (int e = tid, l = l1, i = i1; e < half * n; e += kEigThreads) {
                if (rk[l] == 1) {
                    double *cp = V + (long)rp[l] * lv, *cq = V + (long)rq[l] * lv;
                    const double c = rc[l], sn = rs[l], x = cp[i], y = cq[i];
                    cp[i] = c * x - sn * y;
                    cq[i] = sn * x + c * y;
                }
                l += dv;
                i += di;
                if (i >= n) {
                    i -= n;
                    ++l;
                }
            }
            __syncthreads();
        }
        // restore exact symmetry from the upper triangle
        for (long e = tid; e < (long)n * n; e += kEigThreads) {
            const int i = (int)(e % n), j = (int)(e / n);
            if (i > j) A[i + (long)j * la] = A[j + (long)i * la];
        }
        __syncthreads();
    }
    // eigsrt: descending selection sort, ties to the later index
    if (tid == 0) {
        for (int i = 0; i < n; ++i) perm[i] = i;
        for (int i = 0; i < n - 1; ++i) {
            int k = i;
            double p = A[perm[i] + (long)perm[i] * la];
            for (int j = i + 1; j < n; ++j) {
                const double d = A[perm[j] + (long)perm[j] * la];
                if (d >= p) {
                    k = j;
                    p = d;
                }
            }
            if (k != i) {
                const int x = perm[i];
                perm[i] = perm[k];
                perm[k] = x;
            }
        }
        a.sweeps[ms] = sweep;
    }
    __syncthreads();
    for (int i = tid; i < n; i += kEigThreads) a.eig[(long)ms * a.ne0 + i] = A[perm[i] + (long)perm[i] * la];
    for (long e = tid; e < (long)n * n; e += kEigThreads) {
        const int i = (int)(e % n), j = (int)(e / n);
        a.vec[off + i + (long)j * n] = V[i + (long)perm[j] * lv];
    }
}
