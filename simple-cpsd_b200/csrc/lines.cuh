// lines.cuh -- line transforms of the band passes: register DFTs that skip
// inputs known to be zero, and the exchange between a line's lanes.
//
// A sphere keeps the lines near k = 0: of the Q values a lane holds of a line,
// KZ at either end can be nonzero (kx < KZ P, |ky|, |kz| < KZ P), the others
// are zero in an inverse line and unused in a forward one.
#pragma once

#include "common.cuh"

// values at the ends of a lane's Q line inputs, as a mask (KZ = Q / 2: all)
template <int Q, int KZ>
constexpr unsigned line_mask()
{
    return 2 * KZ >= Q ? (1u << Q) - 1u : ((1u << KZ) - 1u) | (((1u << KZ) - 1u) << (Q - KZ));
}

// In-register DFT of size N whose inputs outside MASK are zero (not read).
template <int N, int SIGN, typename T, unsigned MASK>
struct DFTM;

template <bool A, bool B, typename T>
CPSD_D cx<T> addz(cx<T> a, cx<T> b)
{
    if constexpr (A && B) return a + b;
    else if constexpr (A) return a;
    else if constexpr (B) return b;
    else return cx<T>{0, 0};
}
template <bool A, bool B, typename T>
CPSD_D cx<T> subz(cx<T> a, cx<T> b)
{
    if constexpr (A && B) return a - b;
    else if constexpr (A) return a;
    else if constexpr (B) return cx<T>{-b.x, -b.y};
    else return cx<T>{0, 0};
}

template <int SIGN, typename T, unsigned MASK>
struct DFTM<2, SIGN, T, MASK> {
    CPSD_D static void run(cx<T> *v)
    {
        constexpr bool A = MASK & 1, B = MASK & 2;
        cx<T> a = v[0], b = v[1];
        v[0] = addz<A, B>(a, b);
        v[1] = subz<A, B>(a, b);
    }
};
template <int SIGN, typename T, unsigned MASK>
struct DFTM<4, SIGN, T, MASK> {
    CPSD_D static void run(cx<T> *v)
    {
        constexpr bool A = MASK & 1, B = MASK & 2, C = MASK & 4, D = MASK & 8;
        cx<T> a = v[0], b = v[1], c = v[2], d = v[3];
        const cx<T> s0 = addz<A, C>(a, c), s1 = subz<A, C>(a, c), s2 = addz<B, D>(b, d);
        const cx<T> s3 = mul_is<SIGN>(subz<B, D>(b, d));
        v[0] = addz<A || C, B || D>(s0, s2);
        v[1] = addz<A || C, B || D>(s1, s3);
        v[2] = subz<A || C, B || D>(s0, s2);
        v[3] = subz<A || C, B || D>(s1, s3);
    }
};
// inputs r, r + R, r + 2 R, ... of the size-N mask
template <int N, int R>
constexpr unsigned dft_sub_mask(unsigned mask, int r)
{
    unsigned s = 0;
    for (int m = 0; m < N / R; ++m) s |= ((mask >> (r + R * m)) & 1u) << m;
    return s;
}
template <int N, int SIGN, typename T, unsigned MASK>
struct DFTM {
    CPSD_D static void run(cx<T> *v)
    {
        if constexpr (MASK == (N >= 32 ? ~0u : (1u << N) - 1u)) {
            DFT<N, SIGN, T>::run(v);
        } else {
            constexpr int R = 4, M = N / 4;  // 8 = 4 x 2, 16 = 4 x 4
            static_assert(N == 8 || N == 16, "masked DFT size");
            cx<T> sub[R][M];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int m = 0; m < M; ++m) sub[r][m] = v[r + R * m];
            SFor<0, R>::run([&](auto rc) {
                constexpr int r = decltype(rc)::value;
                constexpr unsigned sm = dft_sub_mask<N, R>(MASK, r);
                if constexpr (sm != 0) DFTM<M, SIGN, T, sm>::run(sub[r]);
            });
            constexpr unsigned top = (dft_sub_mask<N, R>(MASK, 0) ? 1u : 0u) | (dft_sub_mask<N, R>(MASK, 1) ? 2u : 0u) |
                                     (dft_sub_mask<N, R>(MASK, 2) ? 4u : 0u) | (dft_sub_mask<N, R>(MASK, 3) ? 8u : 0u);
            SFor<0, M>::run([&](auto kc) {
                constexpr int k = decltype(kc)::value;
                cx<T> t[R];
                SFor<0, R>::run([&](auto rc) {
                    constexpr int r = decltype(rc)::value;
                    if constexpr ((top >> r) & 1u) t[r] = twmul<N, SIGN, r * k>(sub[r][k]);
                });
                DFTM<R, SIGN, T, top>::run(t);
#pragma unroll
                for (int q = 0; q < R; ++q) v[k + M * q] = t[q];
            });
        }
    }
};

// One exchange of a line: lane t stores its Q values at the slots sidx(i) and
// loads Q values from lidx(i); real and imaginary parts in turn when SPLIT.
template <int Q, bool SPLIT, typename T, typename SI, typename LI>
CPSD_D void line_exchange(cx<T> *v, void *buf, SI sidx, LI lidx)
{
    if constexpr (SPLIT) {
        T *b = static_cast<T *>(buf);
#pragma unroll
        for (int i = 0; i < Q; ++i) b[sidx(i)] = v[i].x;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < Q; ++i) v[i].x = b[lidx(i)];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < Q; ++i) b[sidx(i)] = v[i].y;
        __syncwarp();
#pragma unroll
        for (int i = 0; i < Q; ++i) v[i].y = b[lidx(i)];
        __syncwarp();
    } else {
        cx<T> *b = static_cast<cx<T> *>(buf);
#pragma unroll
        for (int i = 0; i < Q; ++i) b[sidx(i)] = v[i];
        __syncwarp();
#pragma unroll
        for (int i = 0; i < Q; ++i) v[i] = b[lidx(i)];
        __syncwarp();
    }
}

// The passes at n = 128 are bound by shared memory (70 % of its wavefronts
// busy in V psi, FP64 pipe 43 %), so half of a lane's twiddles are formed by a
// product instead of read: V psi 0.856 -> 0.813 ms, density 0.537 -> 0.524 ms
// (FP64), 0.340 -> 0.323 ms (FP32 density); the error against 64 bits stays.

// line_fft (common.cuh) with masked inputs: x[t + P m] in v[m] -> X[(t U + u)
// + Q s] in v[u P + s].  tw: line_fft's table of the sign +1 (its conjugate is
// the other sign's).
template <int N, int SIGN, typename T, unsigned MASK, bool SPLIT>
CPSD_D void line_masked(cx<T> *v, int t, void *xb, const cx<T> *__restrict__ tw)
{
    auto turn = [](cx<T> a, cx<T> w) { return SIGN > 0 ? cmul(a, w) : cx<T>{a.x * w.x + a.y * w.y, a.y * w.x - a.x * w.y}; };
    using L = Line<N>;
    constexpr int P = L::P, Q = L::Q, U = L::U;
    DFTM<Q, SIGN, T, MASK>::run(v);
    if constexpr (Q == 16) {  // W^(q + 8) t from two table entries (see above)
        const cx<T> w8 = tw[8 * P + t];
        v[8] = turn(v[8], w8);
#pragma unroll
        for (int q = 1; q < 8; ++q) {
            const cx<T> w = tw[q * P + t];
            v[q] = turn(v[q], w);
            v[q + 8] = turn(v[q + 8], cmul(w, w8));
        }
    } else {
#pragma unroll
        for (int q = 1; q < Q; ++q) v[q] = turn(v[q], tw[q * P + t]);
    }
    line_exchange<Q, SPLIT>(v, xb, [t](int q) { return L::xb_index(q, t); },
                            [t](int i) { return L::xb_index(t * U + i / P, i % P); });
#pragma unroll
    for (int u = 0; u < U; ++u) DFT<P, SIGN, T>::run(v + u * P);
}
