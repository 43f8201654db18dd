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
// Rows of up to this many steps of 8 reals are split over at most 18 CTAs whose
// sums the last one adds: the cluster's two barriers cost more there than they
// save (six steps a warp; 64^3, 16 bands, ten steps: 765 us with clusters, 751
// without).
constexpr int kSmNoClusterSteps = kSmMaxClusters * kSmWarps * 6;

// products of one launch: the three overlaps (C2'WC2 and C1'WC1 by their upper
// tiles, C2'WC1 whole; MT tiles of 8 bands), or plain products A'WB in blocks
// of up to MT x NB tiles
enum { SM_LAGRANGE = 0, SM_ONE = 1 };
template <int MODE, int MT, int NB>
constexpr int sm_tiles()
{
    return MODE == SM_LAGRANGE ? MT * (MT + 1) + MT * MT : MT * NB;
}

struct SmallArgs {
    int K, splits;               // reals per row; CTAs along k (a multiple of the cluster size)
    long ld;                     // reals between rows
    int m[2], n[2];              // rows of A and of B, per spin or problem (gridDim.y)
    const double *A[2], *B[2];   // LAGRANGE: C2 and C1 of a spin; ONE: the two operands
    const double *w;             // weight per pair of reals
    double *part;                // [block][cluster][tiles * 64]
    unsigned *ticket;            // one per block (LAGRANGE: one), zero before the launch and after it
    double *C[2];                // ONE: C[i * ldc + j]
    long ldc;
    int nblk;                    // ONE: gridDim.z = blocks of 8 MT rows of A x nblk blocks of 8 NB rows of B
    // ONE, projector coefficients: coefT[j][i] = -C scal2 / norm[i] (cpsd.c:289;
    // and coefP[i][j], for the nonlocal force) beside C; null otherwise
    const double *norm;
    double *coefT, *coefP;
    long ldt, ldp;
    double scal2;
    LagArgs lag;                 // LAGRANGE
};

template <int MODE, int MT, int NB>
size_t small_smem_bytes(int ne0)
{
    const size_t red = (size_t)(kSmWarps / 2) * sm_tiles<MODE, MT, NB>() * 64;
    constexpr int mp = 8 * MT, ld = (mp % 16 == 8) ? mp : mp + 8;
    const size_t solve = MODE == SM_LAGRANGE ? (size_t)sm_tiles<MODE, MT, NB>() * 64 + 3 * mp * ld + (size_t)ne0 * ne0 : 0;
    return sizeof(double) * (red > solve ? red : solve);
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
            combine_argmax(lane < kSmWarps ? slot[lane][0] : 0u, lane < kSmWarps ? slot[lane][1] : 0u,
                           lane < kSmWarps ? slot[lane][2] : 0x7fffffffu, hi, lo, at);
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

// CL: CTAs of a cluster (kSmCluster, or 1: no cluster)
template <int MODE, int MT, int NB, int CL>
__global__ void __launch_bounds__(kSmThreads, 1) small_overlap_kernel(const __grid_constant__ SmallArgs a)
{
    static_assert(MODE == SM_ONE || MT == NB, "square");
    constexpr int NT = sm_tiles<MODE, MT, NB>(), NTRI = MT * (MT + 1) / 2, E = NT * 64;
    extern __shared__ __align__(16) double sm_raw[];
    __shared__ unsigned slot[kSmWarps][4];
    __shared__ int last;
    chain_wait();
    chain_start();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, r = lane >> 2, q = lane & 3;
    const int ms = blockIdx.y;
    const int ia = MODE == SM_ONE ? (int)blockIdx.z / a.nblk * (8 * MT) : 0;  // first rows of this block
    const int ib = MODE == SM_ONE ? (int)blockIdx.z % a.nblk * (8 * NB) : 0;
    const int ma = a.m[ms] - ia, mb = (MODE == SM_ONE ? a.n[ms] : a.m[ms]) - ib;
    const double *__restrict__ A = a.A[ms] + ia * a.ld, *__restrict__ B = a.B[ms] + ib * a.ld;
    // this warp's slice of k, in steps of 8 reals (a lane's 16 bytes of a row
    // feed two MMA k-steps: reals 2q of the step, then 2q + 1)
    const int n8 = a.K / 8, nw = a.splits * kSmWarps, wid = blockIdx.x * kSmWarps + warp;
    const int per = (n8 + nw - 1) / nw, s0 = min(n8, wid * per), s1 = min(n8, s0 + per);
    double acc[NT][2] = {};
    const double2 *pa[MT], *pb[NB];
    bool oka[MT], okb[NB];
#pragma unroll
    for (int i = 0; i < MT; ++i) {
        oka[i] = 8 * i + r < ma;
        pa[i] = reinterpret_cast<const double2 *>(A + (long)(oka[i] ? 8 * i + r : 0) * a.ld + 2 * q);
    }
#pragma unroll
    for (int i = 0; i < NB; ++i) {
        okb[i] = 8 * i + r < mb;
        pb[i] = reinterpret_cast<const double2 *>(B + (long)(okb[i] ? 8 * i + r : 0) * a.ld + 2 * q);
    }
    double2 na[MT], nb[NB];
    double nw8 = 0.0;
    auto fetch = [&](int s) {
        nw8 = a.w[4 * s + q];
#pragma unroll
        for (int i = 0; i < MT; ++i) na[i] = oka[i] ? pa[i][4 * s] : make_double2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < NB; ++i) nb[i] = okb[i] ? pb[i][4 * s] : make_double2(0.0, 0.0);
    };
    if (s0 < s1) fetch(s0);
    for (int s = s0; s < s1; ++s) {
        double2 xa[MT], xb[NB];
        const double ww = nw8;
#pragma unroll
        for (int i = 0; i < MT; ++i) xa[i] = na[i];
#pragma unroll
        for (int i = 0; i < NB; ++i) xb[i] = nb[i];
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
                for (int j = 0; j < NB; ++j, ++t) {
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
    const int ncl = a.splits / CL, cid = blockIdx.x / CL;
    const int blk = blockIdx.y * gridDim.z + blockIdx.z;
    double *part = a.part + (size_t)blk * kSmMaxClusters * E;
    if constexpr (CL > 1) {
        cg::cluster_group cl = cg::this_cluster();
        cl.sync();
        const int rank = (int)cl.block_rank();
        const double *src[CL];
#pragma unroll
        for (int c = 0; c < CL; ++c) src[c] = cl.map_shared_rank(red, c);
        for (int e = rank * kSmThreads + tid; e < E; e += CL * kSmThreads) {
            double v[CL], s = 0.0;
#pragma unroll
            for (int c = 0; c < CL; ++c) v[c] = src[c][e];
#pragma unroll
            for (int c = 0; c < CL; ++c) s += v[c];
            part[(size_t)cid * E + e] = s;
        }
        cl.sync();  // the peers have read this CTA's tiles
    } else {
        __syncthreads();
        for (int e = tid; e < E; e += kSmThreads) part[(size_t)cid * E + e] = red[e];
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        // the last CTA of a block (of the launch, for the solver)
        const unsigned total = MODE == SM_ONE ? gridDim.x : gridDim.x * gridDim.y;
        unsigned *tk = a.ticket + (MODE == SM_ONE ? blk : 0);
        last = atomicAdd(tk, 1u) == total - 1;
        if (last) *tk = 0;  // for the next launch
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    const int sp0 = MODE == SM_ONE ? ms : 0, sp1 = MODE == SM_ONE ? ms + 1 : (int)gridDim.y;
    for (int sp = sp0; sp < sp1; ++sp) {
        const double *ps = a.part + (size_t)(MODE == SM_ONE ? blk : sp) * kSmMaxClusters * E;
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
                const int t = e / 64, i = 8 * (t / NB) + (e % 64) / 8, j = 8 * (t % NB) + e % 8;
                if (i < ma && j < mb) {
                    a.C[sp][(long)(ia + i) * a.ldc + ib + j] = s;
                    if (a.norm) {
                        const double v = -s * a.scal2 / a.norm[ia + i];
                        a.coefT[(long)(ib + j) * a.ldt + ia + i] = v;
                        if (a.coefP) a.coefP[(long)(ia + i) * a.ldp + ib + j] = v;
                    }
                }
            }
        }
        if constexpr (MODE == SM_LAGRANGE) {
            __syncthreads();
            const int mm = a.m[sp];
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

// out_j = sum_l mat[j * ldm + l] in_l for up to 8 MT rows
// j per blockIdx.y and any number of l (the KB back-projection of a small cell:
// l over the projectors).  As small_nn_kernel, with the matrix rows in shared
// memory, LD = 4 mod 16 apart (a 16-lane phase then hits 16 banks).
CPSD_HD int small_proj_ld(int L) { return (L + 7) / 8 * 8 + ((L + 7) / 8 % 2 ? 12 : 4); }
struct SmallProjArgs {
    int K, L, nj;
    long ld, ldm;   // reals between the rows of in / out; of mat
    const double *mat, *in;
    double *out;
};

template <int MT>
__global__ void __launch_bounds__(kSmThreads) small_proj_kernel(const __grid_constant__ SmallProjArgs a)
{
    extern __shared__ __align__(16) double sp_mat[];
    const int lane = threadIdx.x & 31, r = lane >> 2, q = lane & 3;
    const int j0 = blockIdx.y * 8 * MT, LD = small_proj_ld(a.L), Lp = (a.L + 7) / 8 * 8;
    for (int e = threadIdx.x; e < 8 * MT * Lp; e += kSmThreads) {
        const int j = e / Lp, l = e % Lp;
        sp_mat[j * LD + l] = (j0 + j < a.nj && l < a.L) ? a.mat[(long)(j0 + j) * a.ldm + l] : 0.0;
    }
    __syncthreads();
    const int nblk = a.K / 16, nw = gridDim.x * kSmWarps;
    for (int b = blockIdx.x * kSmWarps + (threadIdx.x >> 5); b < nblk; b += nw) {
        double e0[MT][2] = {}, e1[MT][2] = {};
        const double *src = a.in + 16 * b + 2 * r;
#pragma unroll 4
        for (int l0 = 0; l0 < Lp; l0 += 4) {
            const int l = l0 + q;
            const double2 x = l < a.L ? *reinterpret_cast<const double2 *>(src + (long)l * a.ld) : make_double2(0.0, 0.0);
#pragma unroll
            for (int j = 0; j < MT; ++j) {
                const double c = sp_mat[(8 * j + r) * LD + l];
                dmma(e0[j][0], e0[j][1], c, x.x);
                dmma(e1[j][0], e1[j][1], c, x.y);
            }
        }
#pragma unroll
        for (int j = 0; j < MT; ++j) {
            const int jj = j0 + 8 * j + r;
            if (jj < a.nj) {
                double2 *o = reinterpret_cast<double2 *>(a.out + (long)jj * a.ld + 16 * b + 4 * q);
                o[0] = make_double2(e0[j][0], e1[j][0]);
                o[1] = make_double2(e0[j][1], e1[j][1]);
            }
        }
    }
}
