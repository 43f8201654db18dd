// small.cuh -- the end of an SD step for at most 32 bands per spin: the three
// overlaps, their split-K sum and the Lagrange fixed point in one launch, and
// the constraint correction; also the single overlap of the energies.
//
// What bounds these at 1 to 32 bands is launches and serial latency, not
// bandwidth (16 bands at 64^3: 1.3 MB of orbitals, 0.2 us of HBM): as separate
// kernels (64 x 64 tiles padded from 16 bands, a reduction launch, a solver)
// they took 45 us of a 116 us step, 86 us with one band at 32^3.  Here the
// tiles are 8 x 8 (mma.sync m8n8k4, FP64), a warp holds all of them for its
// slice of k, the eight warps of a CTA and the eight CTAs of a cluster sum
// their tiles through shared memory, and the last CTA to finish adds the
// clusters' sums and runs the solver.  Every sum has a fixed order.
#pragma once

#include "kernels.cuh"

constexpr int kSmThreads = 256, kSmWarps = kSmThreads / 32, kSmCluster = 8;
constexpr int kSmMaxClusters = 18;  // 144 CTAs: one per SM

// products of one launch: the three overlaps (C2'WC2 and C1'WC1 by their upper
// tiles, C2'WC1 whole), or one plain product A'WB
enum { SM_LAGRANGE = 0, SM_ONE = 1 };
template <int MODE, int MT>
constexpr int sm_tiles()
{
    return MODE == SM_LAGRANGE ? MT * (MT + 1) + MT * MT : MT * MT;
}

struct SmallArgs {
    int K, splits;               // reals per row; CTAs along k (a multiple of kSmCluster)
    long ld;                     // reals between rows
    int m[2];                    // bands per spin (spins = gridDim.y)
    const double *A[2], *B[2];   // LAGRANGE: C2 and C1 of a spin; ONE: the two operands
    const double *w;             // weight per pair of reals
    double *part;                // [spin][cluster][tiles * 64]
    unsigned *ticket;            // zero before the launch, zero after it
    double *C[2];                // ONE: C[i * m + j]
    LagArgs lag;                 // LAGRANGE
};

template <int MODE, int MT>
size_t small_smem_bytes(int ne0)
{
    const size_t red = (size_t)(kSmWarps / 2) * sm_tiles<MODE, MT>() * 64;
    constexpr int mp = 8 * MT, ld = (mp % 16 == 8) ? mp : mp + 8;
    const size_t solve = MODE == SM_LAGRANGE ? (size_t)sm_tiles<MODE, MT>() * 64 + 3 * mp * ld + (size_t)ne0 * ne0 : 0;
    return sizeof(double) * (red > solve ? red : solve);
}

// largest |d| over a warp with the smallest index among equals, as idamax
// (NaN never wins; -1 where every entry was NaN); all lanes get the result
CPSD_D void warp_argmax(double ad, int idx, unsigned &hi, unsigned &lo, int &at)
{
    const bool ok = ad >= 0.0;  // false for NaN and for "no entry" (-1)
    const unsigned long long k = ok ? (unsigned long long)__double_as_longlong(ad) : 0ull;
    const unsigned h = (unsigned)(k >> 32), l = (unsigned)k;
    hi = __reduce_max_sync(0xffffffffu, h);
    lo = __reduce_max_sync(0xffffffffu, h == hi ? l : 0u);
    at = (int)__reduce_min_sync(0xffffffffu, (ok && h == hi && l == lo) ? (unsigned)idx : 0x7fffffffu);
}

// cpsd.c:439-478 on the summed overlaps S (tiles in the order they were
// accumulated).  Tile (I, J) of X belongs to one warp.  A fragment of the
// product register layout (row lane / 4, columns 2 (lane % 4) + e) is an A
// fragment of k-step e as it stands, and a B fragment of the transposed
// matrix, so X and its transpose are kept in shared memory and every operand
// is one 16-byte load; the constant matrices stay in registers.  Two barriers
// an iteration (one warp alone, and no barrier, for up to 8 bands).
template <int MT>
CPSD_D void small_lagrange(const LagArgs &a, int ms, int m, const double *S, double *sm, unsigned (*slot)[4])
{
    constexpr int mp = 8 * MT, LD = (mp % 16 == 8) ? mp : mp + 8;
    constexpr int TPW = (MT * MT + kSmWarps - 1) / kSmWarps;
    constexpr int NTRI = MT * (MT + 1) / 2;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, q = lane & 3;
    const long ne02 = (long)a.ne0 * a.ne0;
    const int kk = m * m;
    double *X = sm, *XT = sm + mp * LD, *STT = sm + 2 * mp * LD, *dif = sm + 3 * mp * LD;
    const double dte = a.dte;
    auto sync = [] {
        if constexpr (MT == 1) __syncwarp();
        else __syncthreads();
    };
    // s matrices, cpsd.c:420-437, from one triangle of each overlap
    auto tri = [](int I, int J) { return I * MT - I * (I - 1) / 2 + (J - I); };
    auto up = [&](const double *base, int i, int j) {  // i <= j
        return base[tri(i >> 3, j >> 3) * 64 + (i & 7) * 8 + (j & 7)];
    };
    auto m21 = [&](int i, int j) { return S[(NTRI + (i >> 3) * MT + (j >> 3)) * 64 + (i & 7) * 8 + (j & 7)]; };
    const double *S22 = S, *S11 = S + (NTRI + MT * MT) * 64;
    auto s22 = [&](int i, int j) {
        if (i >= m || j >= m) return 0.0;
        return i == j ? (1.0 - up(S22, i, i)) * 0.5 / dte : -up(S22, min(i, j), max(i, j)) * 0.5 / dte;
    };
    auto s11 = [&](int i, int j) {
        if (i >= m || j >= m) return 0.0;
        return -up(S11, min(i, j), max(i, j)) * 0.5 * dte;
    };
    auto s21 = [&](int i, int j) {  // <c2_lo|c1_hi>
        if (i >= m || j >= m) return 0.0;
        return i == j ? (1.0 - m21(i, i)) * 0.5 : -m21(min(i, j), max(i, j)) * 0.5;
    };
    auto s12 = [&](int i, int j) {  // <c1_lo|c2_hi>
        if (i >= m || j >= m) return 0.0;
        return i == j ? (1.0 - m21(i, i)) * 0.5 : -m21(max(i, j), min(i, j)) * 0.5;
    };
    double c21[TPW][MT][2], c11[TPW][MT][2], c12[TPW][MT][2], c22[TPW][2], x[TPW][2];
#pragma unroll
    for (int u = 0; u < TPW; ++u) {
        const int t = warp + u * kSmWarps;
        if (t >= MT * MT) break;
        const int I = t / MT, J = t % MT;
#pragma unroll
        for (int k = 0; k < MT; ++k)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                c21[u][k][e] = s21(8 * I + r, 8 * k + 2 * q + e);
                c11[u][k][e] = s11(8 * I + r, 8 * k + 2 * q + e);
                c12[u][k][e] = s12(8 * k + 2 * q + e, 8 * J + r);
            }
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 8 * I + r, j = 8 * J + 2 * q + e;
            x[u][e] = c22[u][e] = s22(i, j);  // sa0 = s22, cpsd.c:441
            X[i * LD + j] = c22[u][e];
            XT[j * LD + i] = c22[u][e];
        }
    }
    sync();
    bool done = false;
    for (int iter = 0; iter < 30 && !done; ++iter) {
        double2 xa[TPW][MT];
        double part[TPW][2];
        // s22 + s21 X + X s12 and st1 = s11 X (cpsd.c:444-462)
#pragma unroll
        for (int u = 0; u < TPW; ++u) {
            const int t = warp + u * kSmWarps;
            if (t >= MT * MT) break;
            const int I = t / MT, J = t % MT;
            double t1[2] = {0.0, 0.0}, t2[2] = {0.0, 0.0}, st[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < MT; ++k) {
                xa[u][k] = *reinterpret_cast<const double2 *>(X + (8 * I + r) * LD + 8 * k + 2 * q);
                const double2 xb = *reinterpret_cast<const double2 *>(XT + (8 * J + r) * LD + 8 * k + 2 * q);
                dmma(st[0], st[1], c11[u][k][0], xb.x);
                dmma(t1[0], t1[1], c21[u][k][0], xb.x);
                dmma(t2[0], t2[1], xa[u][k].x, c12[u][k][0]);
                dmma(st[0], st[1], c11[u][k][1], xb.y);
                dmma(t1[0], t1[1], c21[u][k][1], xb.y);
                dmma(t2[0], t2[1], xa[u][k].y, c12[u][k][1]);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                part[u][e] = t2[e] + (t1[e] + c22[u][e]);
                STT[(8 * J + 2 * q + e) * LD + 8 * I + r] = st[e];
            }
        }
        sync();
        // sa1 = that + X st1, the differences and their largest entry (cpsd.c:463-470)
        double bestv = -1.0;
        int besti = 0x7fffffff;
#pragma unroll
        for (int u = 0; u < TPW; ++u) {
            const int t = warp + u * kSmWarps;
            if (t >= MT * MT) break;
            const int I = t / MT, J = t % MT;
            double t4[2] = {0.0, 0.0};
#pragma unroll
            for (int k = 0; k < MT; ++k) {
                const double2 sb = *reinterpret_cast<const double2 *>(STT + (8 * J + r) * LD + 8 * k + 2 * q);
                dmma(t4[0], t4[1], xa[u][k].x, sb.x);
                dmma(t4[0], t4[1], xa[u][k].y, sb.y);
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int i = 8 * I + r, j = 8 * J + 2 * q + e;
                const double v = t4[e] + part[u][e];
                if (i < m && j < m) {
                    const double d = v - x[u][e], ad = fabs(d);
                    const int f = i + j * m;
                    dif[f] = d;
                    if (ad > bestv || (ad == bestv && f < besti)) {
                        bestv = ad;
                        besti = f;
                    }
                }
                x[u][e] = v;
                X[i * LD + j] = v;
                XT[j * LD + i] = v;
            }
        }
        unsigned hi, lo;
        int at;
        warp_argmax(bestv, besti, hi, lo, at);
        if constexpr (MT > 1) {
            if (lane == 0) {
                slot[warp][0] = hi;
                slot[warp][1] = lo;
                slot[warp][2] = (unsigned)at;
            }
        }
        sync();
        if constexpr (MT > 1) {  // every warp combines the warps' candidates and takes the same decision
            const unsigned h = lane < kSmWarps ? slot[lane][0] : 0u, l = lane < kSmWarps ? slot[lane][1] : 0u;
            const unsigned s = lane < kSmWarps ? slot[lane][2] : 0x7fffffffu;
            hi = __reduce_max_sync(0xffffffffu, h);
            lo = __reduce_max_sync(0xffffffffu, h == hi ? l : 0u);
            at = (int)__reduce_min_sync(0xffffffffu, (h == hi && l == lo) ? s : 0x7fffffffu);
        }
        // idamax returns an index in 1..kk even when every entry is NaN: the
        // sentinel must never reach the read below
        if (at < 0 || at >= kk) at = 0;
        // idamax's 1-based index used as 0-based (cpsd.c:471); past st1 lies
        // sa1, whose first entry is element (0, 0); entries of dif past m^2
        // keep the other spin's, as st1's do there
        const long nx = (long)at + 1;
        const double adiff = fabs(nx < ne02 ? dif[nx] : X[nx - ne02]);
        done = adiff < 1e-15;
        // the next iteration writes STT alone before its first barrier
    }
    if (!done && tid == 0) atomicAdd(a.fail, 1);
#pragma unroll
    for (int u = 0; u < TPW; ++u) {
        const int t = warp + u * kSmWarps;
        if (t >= MT * MT) break;
        const int I = t / MT, J = t % MT;
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = 8 * I + r, j = 8 * J + 2 * q + e;
            if (i < m && j < m) a.lmd[ms * ne02 + i + j * m] = x[u][e];
        }
    }
}

template <int MODE, int MT>
__global__ void __launch_bounds__(kSmThreads, 1) small_overlap_kernel(const __grid_constant__ SmallArgs a)
{
    constexpr int NT = sm_tiles<MODE, MT>(), NTRI = MT * (MT + 1) / 2, E = NT * 64;
    cg::cluster_group cl = cg::this_cluster();
    extern __shared__ __align__(16) double sm_raw[];
    __shared__ unsigned slot[kSmWarps][4];
    __shared__ int last;
    chain_wait();
    chain_start();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, q = lane & 3;
    const int ms = blockIdx.y, m = a.m[ms];
    const double *__restrict__ A = a.A[ms], *__restrict__ B = a.B[ms];
    // this warp's slice of k, in steps of 8 reals (a lane's 16 bytes of a row
    // feed two MMA k-steps: reals 2q of the step, then 2q + 1)
    const int n8 = a.K / 8, nw = a.splits * kSmWarps, wid = blockIdx.x * kSmWarps + warp;
    const int per = (n8 + nw - 1) / nw, s0 = min(n8, wid * per), s1 = min(n8, s0 + per);
    double acc[NT][2] = {};
    const double2 *pa[MT], *pb[MT];
    bool ok[MT];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        ok[i] = 8 * i + r < m;
        pa[i] = reinterpret_cast<const double2 *>(A + (long)(ok[i] ? 8 * i + r : 0) * a.ld + 2 * q);
        pb[i] = reinterpret_cast<const double2 *>(B + (long)(ok[i] ? 8 * i + r : 0) * a.ld + 2 * q);
    }
    double2 na[MT], nb[MT];
    double nw8 = 0.0;
    auto fetch = [&](int s) {
        nw8 = a.w[4 * s + q];
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            na[i] = ok[i] ? pa[i][4 * s] : make_double2(0.0, 0.0);
            nb[i] = ok[i] ? pb[i][4 * s] : make_double2(0.0, 0.0);
        }
    };
    if (s0 < s1) fetch(s0);
    for (int s = s0; s < s1; ++s) {
        double2 xa[MT], xb[MT];
        const double ww = nw8;
#pragma unroll
        for (int i = 0; i < MT; ++i) {
            xa[i] = na[i];
            xb[i] = nb[i];
        }
        if (s + 1 < s1) fetch(s + 1);
        int t = 0;
        if constexpr (MODE == SM_LAGRANGE) {
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const double2 wa = make_double2(xa[i].x * ww, xa[i].y * ww);
#pragma unroll
                for (int j = i; j < MT; ++j) {  // C2'WC2
                    const int k = i * MT - i * (i - 1) / 2 + (j - i);
                    dmma(acc[k][0], acc[k][1], wa.x, xa[j].x);
                    dmma(acc[k][0], acc[k][1], wa.y, xa[j].y);
                }
#pragma unroll
                for (int j = 0; j < MT; ++j) {  // C2'WC1
                    const int k = NTRI + i * MT + j;
                    dmma(acc[k][0], acc[k][1], wa.x, xb[j].x);
                    dmma(acc[k][0], acc[k][1], wa.y, xb[j].y);
                }
                const double2 wb = make_double2(xb[i].x * ww, xb[i].y * ww);
#pragma unroll
                for (int j = i; j < MT; ++j) {  // C1'WC1
                    const int k = NTRI + MT * MT + i * MT - i * (i - 1) / 2 + (j - i);
                    dmma(acc[k][0], acc[k][1], wb.x, xb[j].x);
                    dmma(acc[k][0], acc[k][1], wb.y, xb[j].y);
                }
            }
        } else {
#pragma unroll
            for (int i = 0; i < MT; ++i) {
                const double2 wa = make_double2(xa[i].x * ww, xa[i].y * ww);
#pragma unroll
                for (int j = 0; j < MT; ++j, ++t) {
                    dmma(acc[t][0], acc[t][1], wa.x, xb[j].x);
                    dmma(acc[t][0], acc[t][1], wa.y, xb[j].y);
                }
            }
        }
    }
    // the warps' tiles: halves of the warps add in turn (warp w takes w + h)
    double *red = sm_raw;
#pragma unroll
    for (int h = kSmWarps / 2; h >= 1; h /= 2) {
        if (warp >= h && warp < 2 * h) {
#pragma unroll
            for (int t = 0; t < NT; ++t)
                *reinterpret_cast<double2 *>(red + (size_t)(warp - h) * E + t * 64 + 2 * lane) =
                    make_double2(acc[t][0], acc[t][1]);
        }
        __syncthreads();
        if (warp < h) {
#pragma unroll
            for (int t = 0; t < NT; ++t) {
                const double2 v = *reinterpret_cast<const double2 *>(red + (size_t)warp * E + t * 64 + 2 * lane);
                acc[t][0] += v.x;
                acc[t][1] += v.y;
            }
        }
        __syncthreads();
    }
    if (warp == 0) {
#pragma unroll
        for (int t = 0; t < NT; ++t)
            *reinterpret_cast<double2 *>(red + t * 64 + 2 * lane) = make_double2(acc[t][0], acc[t][1]);
    }
    // entry t * 64 + 8 r + 2 q + e: row r, column 2 q + e of tile t
    cl.sync();
    const int rank = (int)cl.block_rank(), ncl = a.splits / kSmCluster, cid = blockIdx.x / kSmCluster;
    double *part = a.part + (size_t)ms * kSmMaxClusters * E;
    {
        const double *src[kSmCluster];
#pragma unroll
        for (int c = 0; c < kSmCluster; ++c) src[c] = cl.map_shared_rank(red, c);
        for (int e = rank * kSmThreads + tid; e < E; e += kSmCluster * kSmThreads) {
            double v[kSmCluster], s = 0.0;
#pragma unroll
            for (int c = 0; c < kSmCluster; ++c) v[c] = src[c][e];
#pragma unroll
            for (int c = 0; c < kSmCluster; ++c) s += v[c];
            part[(size_t)cid * E + e] = s;
        }
    }
    cl.sync();  // the peers have read this CTA's tiles
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        const unsigned total = gridDim.x * gridDim.y;
        last = atomicAdd(a.ticket, 1u) == total - 1;
        if (last) *a.ticket = 0;  // for the next launch
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    for (int sp = 0; sp < (int)gridDim.y; ++sp) {
        const int mm = a.m[sp];
        const double *ps = a.part + (size_t)sp * kSmMaxClusters * E;
        double *S = sm_raw;
        for (int e = tid; e < E; e += kSmThreads) {
            double v[kSmMaxClusters], s = 0.0;
#pragma unroll
            for (int c = 0; c < kSmMaxClusters; ++c) v[c] = c < ncl ? __ldcg(ps + (size_t)c * E + e) : 0.0;
#pragma unroll
            for (int c = 0; c < kSmMaxClusters; ++c) s += v[c];
            if constexpr (MODE == SM_LAGRANGE) {
                S[e] = s;
            } else {
                const int t = e / 64, i = 8 * (t / MT) + (e % 64) / 8, j = 8 * (t % MT) + e % 8;
                if (i < mm && j < mm) a.C[sp][i * mm + j] = s;
            }
        }
        if constexpr (MODE == SM_LAGRANGE) {
            __syncthreads();
            if (mm > 0 && (MT > 1 || warp == 0)) small_lagrange<MT>(a.lag, sp, mm, S, sm_raw + E, slot);
            __syncthreads();
        }
    }
}

// c2 += dte C1 lmd (cpsd.c:482-488) for at most 32 bands per spin, both spins
// in one launch: out_j = c2_j + alpha sum_l mat[l + j m] c1_l.  A warp takes
// 16 reals of every row (a lane's 16 bytes of row l feed two MMAs: the even
// and the odd reals), the matrix stays in registers.
struct SmallNNArgs {
    int K;
    long ld;
    int m[2];
    const double *mat[2], *in[2];
    double *out[2];
    double alpha, beta;
};

template <int MT>
__global__ void __launch_bounds__(kSmThreads) small_nn_kernel(const __grid_constant__ SmallNNArgs a)
{
    chain_wait();
    chain_start();
    const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int ms = blockIdx.y, m = a.m[ms];
    const double *__restrict__ mat = a.mat[ms], *__restrict__ in = a.in[ms];
    double *__restrict__ out = a.out[ms];
    double c[MT][2 * MT];
#pragma unroll
    for (int j = 0; j < MT; ++j)
#pragma unroll
        for (int s = 0; s < 2 * MT; ++s) {
            const int jj = 8 * j + r, l = 4 * s + q;
            c[j][s] = (jj < m && l < m) ? mat[l + jj * m] : 0.0;
        }
    const int nblk = a.K / 16, nw = gridDim.x * kSmWarps;
    for (int b = blockIdx.x * kSmWarps + (threadIdx.x >> 5); b < nblk; b += nw) {
        double2 x[2 * MT];
#pragma unroll
        for (int s = 0; s < 2 * MT; ++s) {
            const int l = 4 * s + q;
            x[s] = l < m ? *reinterpret_cast<const double2 *>(in + (long)l * a.ld + 16 * b + 2 * r) : make_double2(0.0, 0.0);
        }
#pragma unroll
        for (int j = 0; j < MT; ++j) {
            double e0[2] = {0.0, 0.0}, e1[2] = {0.0, 0.0};
#pragma unroll
            for (int s = 0; s < 2 * MT; ++s) {
                dmma(e0[0], e0[1], c[j][s], x[s].x);
                dmma(e1[0], e1[1], c[j][s], x[s].y);
            }
            // column n = 2 q + h of the product of the even reals is real 2 n, of the odd ones 2 n + 1
            const int jj = 8 * j + r;
            if (jj < m) {
                double2 *o = reinterpret_cast<double2 *>(out + (long)jj * a.ld + 16 * b + 4 * q);
                double2 v0 = make_double2(0.0, 0.0), v1 = v0;
                if (a.beta != 0.0) {
                    v0 = o[0];
                    v1 = o[1];
                }
                o[0] = make_double2(a.alpha * e0[0] + a.beta * v0.x, a.alpha * e1[0] + a.beta * v0.y);
                o[1] = make_double2(a.alpha * e0[1] + a.beta * v1.x, a.alpha * e1[1] + a.beta * v1.y);
            }
        }
    }
}
