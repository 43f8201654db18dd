// pair.cuh -- the band passes of an SD step (density, V psi): two bands of a
// z plane transformed as one complex field.
//
// Along x the orbitals are real, so two bands A, B of the same plane make one
// complex row psi_A + i psi_B: its line transform has the full length n, takes
// Z(k) = a + i b and Z(-k) = conj(a) + i conj(b) straight from the kx lines a,
// b of the two bands, and needs none of the half-length transform's pre- and
// post-processing (fft.cuh: reads of k and n/2 - k, a twiddle per value, a
// round trip through shared memory after the forward transform).  V(r) is
// read once for both bands, and |Z|^2 is the two bands' density.  At k = 0 and
// k = n/2 only the real parts of a and b enter, as the reference's c2r drops
// the imaginary ones (fftpack3d/fftpack3d.f:86-89).
//
// Measured on a B200 against one band a CTA (plane_kernel, the twiddles in
// shared memory too): 128 bands at 128^3 FP64 V psi 1.04 -> 0.81 ms, density
// 0.70 -> 0.52 ms; FP32 0.74 -> 0.52 and 0.47 -> 0.32 ms; 16 bands at 64^3
// FP64 26.6 -> 22.5 us and 20.5 -> 14.2 us.
//
// The sphere keeps kx < KX and |ky| < KZ P lines, so an inverse line starts
// with 2 KZ of the Q values a lane holds, the others zero, and a forward line
// ends with them: the register DFTs skip the zeros (DFTM) and the unused
// outputs (never stored, so the compiler drops them).
#pragma once

#include "fft.cuh"
#include "lines.cuh"

// Twiddles of the pair passes, one allocation: the inverse lines' table in
// line_fft's order (q P + t), and the forward (transposed) lines' table,
// W^-(t U + u) t' at (t' U + u) P + t: the P lanes of a line read P
// consecutive entries in both.
template <int NF>
struct PairTw {
    static constexpr int inv = 0, dif = NF, total = 2 * NF;
};

// How a pair pass is built: threads per CTA (a group of P lanes per x row),
// the CTAs per SM its registers are capped for, and whether a line exchanges
// its real and imaginary parts one after the other (half the exchange buffer).
//
// n = 128, FP64: the kx lines of two bands take 97 KB at KX = 21, so one CTA
// per SM; 512 threads fit beside them (64 rows at once) because the parts are
// exchanged in turn.  Measured, 128 bands, V psi / density: 512 threads 0.81 /
// 0.52 ms, 384 with whole exchanges 0.87 / 0.53, 256 with 255 registers 0.92 /
// 0.55 (density: 32 sums per lane, 104 bytes of spills, still the fastest).
// FP32: V psi with two CTAs of 256 threads 0.52 ms, one of 256 0.75; density
// with 512 threads 0.32 ms, 384 0.35, 256 0.37.
// n <= 64: a thread per lane of every row of the plane (n P threads, 256 at
// n = 64, which take the rows in two turns).
template <typename T, int NF, int MODE>
struct PairCfg {
    static constexpr bool wide = NF == 128 && sizeof(T) == 8;
    static constexpr int P = Line<NF>::P;
    static constexpr int NT = (NF == 128) ? ((wide || MODE == PM_DENSITY) ? 512 : 256)
                                          : (NF * P <= 256 ? (NF * P + 31) / 32 * 32 : 256);
    static constexpr int MINB = 512 / NT;
    static constexpr bool SPLIT = wide;
    static constexpr int NG = NT / P;
    // exchange buffer stride of a group, in reals when SPLIT, else in complex values
    static constexpr int GS = SPLIT ? pad_to(Line<NF>::XB, 16, 8) : group_stride<T, NF>();
};

// Y lines of the two bands: the row layout of the single-field passes for the
// full-length x lines
template <typename T, int NF>
struct PairShape {
    using L = Line<NF>;
    static constexpr bool YSWZ = sizeof(cx<T>) == 16 && L::P >= 8 && L::U >= 2;  // see PlaneShape
    static constexpr int YW = NF + (YSWZ ? NF / 8 : 0);
    CPSD_HD static int ymap(int p) { return YSWZ ? p + (p >> 3) : p; }
    static constexpr int YS = (L::P >= kSlots<T>) ? pad_to(YW + 1, kSlots<T>, 1)
                                                  : pad_to(YW + 1, kSlots<T>, kSlots<T> / L::P);
};

template <typename T>
constexpr size_t pair_stage_elems(int ncol)
{
    return ((size_t)2 * ncol * sizeof(cx<T>) + 15) / 16 * 16 / sizeof(cx<T>);
}

template <typename T, int NF, int MODE>
size_t pair_smem_bytes(int KX, int ncol, bool stage)
{
    using C = PairCfg<T, NF, MODE>;
    const size_t ex = C::SPLIT ? sizeof(T) * C::NG * C::GS : sizeof(cx<T>) * C::NG * C::GS;
    const size_t b = sizeof(cx<T>) * (PairTw<NF>::total + (stage ? pair_stage_elems<T>(ncol) : 0) +
                                      (size_t)2 * KX * PairShape<T, NF>::YS) + ex;
    return (b + 15) / 16 * 16;
}

// line_fft_dif with the pair passes' table: x[(t U + u) + Q s] in v[u P + s]
// -> X[t + P m] in v[m], sign -1.
template <int N, typename T, bool SPLIT>
CPSD_D void pair_forward(cx<T> *v, int t, void *xb, const cx<T> *__restrict__ tw)
{
    using L = Line<N>;
    constexpr int P = L::P, Q = L::Q, U = L::U;
    if constexpr (U == 2) {  // u = 1: the entry of u = 0 times the constant W^-t'
        DFT<P, -1, T>::run(v);
        DFT<P, -1, T>::run(v + P);
        SFor<1, P>::run([&](auto tc) {
            constexpr int tp = decltype(tc)::value;
            const cx<T> w = tw[(tp * U) * P + t];
            v[tp] = cmul(v[tp], w);
            v[P + tp] = cmul(v[P + tp], twmul<N, -1, tp>(w));
        });
    } else {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            DFT<P, -1, T>::run(v + u * P);
#pragma unroll
            for (int tp = 1; tp < P; ++tp) v[u * P + tp] = cmul(v[u * P + tp], tw[(tp * U + u) * P + t]);
        }
    }
    line_exchange<Q, SPLIT>(v, xb, [t](int i) { return L::xb_index(t * U + i / P, i % P); },
                            [t](int q) { return L::xb_index(q, t); });
    DFT<Q, -1, T>::run(v);
}

struct PairArgs {
    const int *chunk_b0;  // bands of blockIdx.y: [chunk_b0[y], chunk_b0[y+1])
    double *rho_part;     // DENSITY: [chunk][z][y][x] sums of psi^2
    const double *V;      // APPLYV: see PlaneArgs::V
    int ne0;              // bands b >= ne0 are spin 1's (V of spin 1; never paired with spin 0's)
    int stage;            // the next pair's columns are copied ahead into shared memory
};

// KZ: values on each end of a lane's line inputs that can be nonzero (Q / 2: all)
template <typename T, int NF, int MODE, int KZ>
__global__ void __launch_bounds__(PairCfg<T, NF, MODE>::NT, PairCfg<T, NF, MODE>::MINB)
pair_kernel(Geom g, cx<T> *__restrict__ Tb, PairArgs a, const cx<T> *__restrict__ twg)
{
    using C = PairCfg<T, NF, MODE>;
    using S = PairShape<T, NF>;
    using L = Line<NF>;
    constexpr int P = L::P, Q = L::Q, U = L::U, H = NF / 2;
    constexpr int NT = C::NT, NG = C::NG, YS = S::YS;
    constexpr bool ALL = 2 * KZ >= Q;
    constexpr unsigned MASK = line_mask<Q, KZ>();
    constexpr int NIT = (NF + NG - 1) / NG;  // x rows per group
    extern __shared__ unsigned char smem_raw[];
    const int KX = g.KX, ncol = g.ncol;
    cx<T> *tws = reinterpret_cast<cx<T> *>(smem_raw);
    cx<T> *stage = tws + PairTw<NF>::total;                         // [2][ncol] when staged
    cx<T> *Y = stage + (a.stage ? pair_stage_elems<T>(ncol) : 0);   // [2][KX][YS]
    const int gr = threadIdx.x / P, t = threadIdx.x % P;            // line group and lane
    void *xb = C::SPLIT ? (void *)(reinterpret_cast<T *>(Y + 2 * KX * YS) + gr * C::GS)
                        : (void *)(Y + 2 * KX * YS + gr * C::GS);
    for (int i = threadIdx.x; i < PairTw<NF>::total; i += NT) tws[i] = twg[i];
    chain_wait();
    chain_start();
    const cx<T> *twi = tws + PairTw<NF>::inv, *twd = tws + PairTw<NF>::dif;

    const int z = blockIdx.x;
    const int b0 = a.chunk_b0[blockIdx.y], b1 = a.chunk_b0[blockIdx.y + 1];
    constexpr long plane = (long)NF * NF;
    const long bstride = (long)NF * ncol;
    double rho[(MODE == PM_DENSITY) ? NIT : 1][(MODE == PM_DENSITY) ? Q : 1];
    if constexpr (MODE == PM_DENSITY) {
#pragma unroll
        for (int it = 0; it < NIT; ++it)
#pragma unroll
            for (int q = 0; q < Q; ++q) rho[it][q] = 0.0;
    }
    // bands taken together from b on: two of one spin, or the last one alone
    auto two = [&](int b) { return b + 1 < b1 && (b + 1 != a.ne0); };
    auto prefetch = [&](int b) {
        const int nb = two(b) ? 2 : 1;
        for (int h = 0; h < nb; ++h) {
            const cx<T> *src = Tb + (b + h) * bstride + (long)z * ncol;
            for (int c = threadIdx.x; c < ncol; c += NT) cp_async_cx(stage + h * ncol + c, src + c);
        }
        cp_async_commit_all();
    };
    if (a.stage && b0 < b1) prefetch(b0);
    // column of (line i, y), -1 outside the sphere
    auto column = [&](int i, int c0, int ra, int rb, int y) {
        if (g.yrun) return y < ra ? c0 + y : (y >= rb ? c0 + ra + (y - rb) : -1);
        return i >= 0 ? g.colidx[i * NF + y] : -1;
    };
    if (!a.stage) __syncthreads();  // the twiddles

    for (int b = b0; b < b1;) {
        const bool has2 = two(b);
        const int nl = has2 ? 2 * KX : KX;
        if (a.stage) {
            cp_async_wait_all();
            __syncthreads();
        }
        // ---- inverse along y: columns -> the lines kx < KX of each band
        for (int base = 0; base < nl; base += NG) {
            if (base + (gr & ~(32 / P - 1)) >= nl) break;  // whole warps without a line
            const int li = base + gr;
            const bool act = li < nl;
            const int h = act && li >= KX ? 1 : 0, i = act ? li - h * KX : -1;
            int c0 = 0, ra = 0, rb = NF;
            if (act && g.yrun) {
                c0 = g.yrun[3 * i];
                ra = g.yrun[3 * i + 1];
                rb = g.yrun[3 * i + 2];
            }
            cx<T> v[Q];
            const cx<T> *src = Tb + (b + h) * bstride + (long)z * ncol;
            const cx<T> *sst = stage + h * ncol;
            SFor<0, Q>::run([&](auto mc) {
                constexpr int m = decltype(mc)::value;
                if constexpr ((MASK >> m) & 1u) {
                    const int c = column(i, c0, ra, rb, t + P * m);
                    v[m] = (c < 0) ? cx<T>{0, 0} : (a.stage ? sst[c] : src[c]);
                }
            });
            line_masked<NF, +1, T, MASK, C::SPLIT>(v, t, xb, twi);
            if (act) {
                cx<T> *Yl = Y + li * YS;
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int s = 0; s < P; ++s) Yl[S::ymap(L::out_index(t, u, s))] = v[u * P + s];
            }
        }
        const int bn = b + (has2 ? 2 : 1);
        __syncthreads();
        if (a.stage && bn < b1) prefetch(bn);
        // ---- x rows of both bands
        const cx<T> *Ya = Y, *Yb = Y + KX * YS;
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int j = it * NG + gr;
            const bool act = j < NF;
            const int jm = S::ymap(act ? j : 0);
            cx<T> v[Q];
            SFor<0, Q>::run([&](auto mc) {
                constexpr int m = decltype(mc)::value;
                if constexpr ((MASK >> m) & 1u) {
                    const int k = t + P * m;
                    // k <= n/2: line k; above: line n - k, conjugated
                    const bool up = (m < Q / 2) || (m == Q / 2 && t == 0);
                    const int kk = up ? k : NF - k;
                    cx<T> xa{0, 0}, xc{0, 0};
                    if (kk < KX) {
                        xa = Ya[kk * YS + jm];
                        if (has2) xc = Yb[kk * YS + jm];
                    }
                    if (m < Q / 2 && !(m == 0 && t == 0))
                        v[m] = cx<T>{xa.x - xc.y, xa.y + xc.x};
                    else if (up)  // k = 0, n/2: the real parts alone
                        v[m] = cx<T>{xa.x, xc.x};
                    else
                        v[m] = cx<T>{xa.x + xc.y, xc.x - xa.y};
                }
            });
            line_masked<NF, +1, T, MASK, C::SPLIT>(v, t, xb, twi);
            // v[u P + s] = (psi_A(x), psi_B(x)), x = (t U + u) + Q s
            if constexpr (MODE == PM_DENSITY) {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    rho[it][q] += (double)v[q].x * (double)v[q].x;
                    rho[it][q] += (double)v[q].y * (double)v[q].y;
                }
            } else {
                // FP32: psi V = psi V_hi + psi V_lo in FP32 (one rounding of the
                // sum; V_hi + V_lo holds 48 bits of V): the products in FP64 took
                // two conversions and a multiplication of the FP64 pipe each
                // (128 bands at 128^3: 0.516 ms, 0.479 this way).
                const double *V = a.V + ((b >= a.ne0) ? NF * plane : 0) + (long)z * plane + (long)(act ? j : 0) * NF;
                auto times = [](cx<T> w, double v) {
                    if constexpr (sizeof(T) == 4) {
                        const float hi = __int_as_float(__double2loint(v)), lo = __int_as_float(__double2hiint(v));
                        return cx<T>{fmaf(w.x, hi, w.x * lo), fmaf(w.y, hi, w.y * lo)};
                    } else {
                        return cx<T>{w.x * v, w.y * v};
                    }
                };
#pragma unroll
                for (int s = 0; s < P; ++s) {
                    if constexpr (U % 2 == 0) {
#pragma unroll
                        for (int u = 0; u < U; u += 2) {
                            const double2 vv = *reinterpret_cast<const double2 *>(V + L::out_index(t, u, s));
                            cx<T> &w0 = v[u * P + s], &w1 = v[(u + 1) * P + s];
                            w0 = times(w0, vv.x);
                            w1 = times(w1, vv.y);
                        }
                    } else {
#pragma unroll
                        for (int u = 0; u < U; ++u) {
                            v[u * P + s] = times(v[u * P + s], V[L::out_index(t, u, s)]);
                        }
                    }
                }
                pair_forward<NF, T, C::SPLIT>(v, t, xb, twd);
                // the bands' kx lines from Z(k) and Z(n - k), which lane (P - t) % P holds
                const int src = (P - t) & (P - 1);
                SFor<0, Q / 2 + 1>::run([&](auto mc) {
                    constexpr int m = decltype(mc)::value;
                    if constexpr (ALL || m < KZ) {
                        const cx<T> mine = v[m];
                        const cx<T> give = (t == 0) ? v[(Q - m) % Q] : v[Q - 1 - m];
                        cx<T> o;
                        o.x = __shfl_sync(0xffffffffu, give.x, src, P);
                        o.y = __shfl_sync(0xffffffffu, give.y, src, P);
                        const int k = t + P * m;
                        if (act && k < KX && (m < Q / 2 || t == 0)) {
                            cx<T> A{(T)0.5 * (mine.x + o.x), (T)0.5 * (mine.y - o.y)};
                            cx<T> B{(T)0.5 * (mine.y + o.y), (T)0.5 * (o.x - mine.x)};
                            if (k == 0 || k == H) A.y = B.y = 0;
                            Y[k * YS + jm] = A;
                            if (has2) Y[(KX + k) * YS + jm] = B;
                        }
                    }
                });
            }
        }
        __syncthreads();
        // ---- forward along y, straight to the columns
        if constexpr (MODE == PM_APPLYV) {
            for (int base = 0; base < nl; base += NG) {
                if (base + (gr & ~(32 / P - 1)) >= nl) break;
                const int li = base + gr;
                const bool act = li < nl;
                const int h = act && li >= KX ? 1 : 0, i = act ? li - h * KX : -1;
                const cx<T> *Yl = Y + (act ? li : 0) * YS;  // (read only: the columns take the result)
                cx<T> v[Q];
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int s = 0; s < P; ++s) v[u * P + s] = Yl[S::ymap(L::out_index(t, u, s))];
                pair_forward<NF, T, C::SPLIT>(v, t, xb, twd);
                if (act) {
                    int c0 = 0, ra = 0, rb = NF;
                    if (g.yrun) {
                        c0 = g.yrun[3 * i];
                        ra = g.yrun[3 * i + 1];
                        rb = g.yrun[3 * i + 2];
                    }
                    cx<T> *dst = Tb + (b + h) * bstride + (long)z * ncol;
                    SFor<0, Q>::run([&](auto mc) {
                        constexpr int m = decltype(mc)::value;
                        if constexpr ((MASK >> m) & 1u) {
                            const int c = column(i, c0, ra, rb, t + P * m);
                            if (c >= 0) dst[c] = v[m];
                        }
                    });
                }
            }
        }
        b = bn;
    }

    if constexpr (MODE == PM_DENSITY) {
        double *dst = a.rho_part + ((long)blockIdx.y * NF + z) * plane;
#pragma unroll
        for (int it = 0; it < NIT; ++it) {
            const int j = it * NG + gr;
            if (j < NF) {
#pragma unroll
                for (int u = 0; u < U; ++u)
#pragma unroll
                    for (int s = 0; s < P; ++s) dst[(long)j * NF + L::out_index(t, u, s)] = rho[it][u * P + s];
            }
        }
    }
}
