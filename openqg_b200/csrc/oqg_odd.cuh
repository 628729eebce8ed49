// oqg_odd.cuh -- the closed box's x-transform: DST-I of row pairs.
//
// The DST-I of n = N - 1 values (inhomog.F90:170-212; FFTW RODFT00) is the FFT
// of their odd extension to M = 2N points, and two real rows share one complex
// transform.  The odd extension makes almost half of that FFT redundant.  With
// the decimation x[r + R0 j] (r < R0, L = M / R0, R0 an even divisor of M up to
// 16) the length-L transform S_r of subsequence r satisfies
//     S_{R0-r}(k) = -W_L^{-k} S_r(L - k),
// so only the R0/2 + 1 subsequences r <= R0/2 are transformed (9 of 16), and
// the last radix-R0 stage runs for k <= L/2 only: its outputs X(k + L k1) give
// every coefficient or its mirror X(M - i) = -X(i).  Each output is the same
// sum as in the full FFT; nothing is accumulated along a row, so the rounding
// stays that of an FFT (the usual half-length sine-transform constructions
// carry a running sum).
//
// Bound by shared memory and latency: a transform moves 16-byte complex values
// through shared memory between stages.  Here the rows go straight from global
// memory into the first stage's input (no extended copy), the pruned stages
// move 9/16 of the values, and the last stage writes its outputs to global
// memory from registers.
#pragma once

#include "oqg_fft.cuh"

namespace oqg {

template <class T> struct Dft<T, 1> {
    typedef typename C2<T>::t T2;
    static __device__ __forceinline__ void run(T2 *) {}
};

// The outer (last) radix of a box length M = 2 (nxp - 1): the one that leaves
// the smallest part, (R0/2 + 1) / R0, of the extension to transform.  (M is even,
// at least 8 and has no prime factor above 5: one of these divides it.)
__host__ __device__ constexpr int odd_r0(int M) {
    return M % 16 == 0 ? 16 : M % 12 == 0 ? 12 : M % 10 == 0 ? 10 : M % 8 == 0 ? 8 : 6;
}
// Lengths with a compile-time plan: R0 = 16 and L = RA RB in two stages.
__host__ __device__ constexpr bool odd_ct_len(int M) {
    return M == 128 || M == 192 || M == 256 || M == 384 || M == 512 || M == 1024 || M == 2048 || M == 4096;
}
__host__ __device__ constexpr int odd_ra(int L) {
    return L == 256 || L == 128 || L == 16 ? 16 : L == 12 ? 4 : 8;     // 64, 32, 24, 8: 8
}
// Threads of one transform: at most 16 complex values (one radix-16 or two
// radix-8 butterflies) per thread and stage, and the L/2 + 1 last butterflies.
__host__ __device__ constexpr int odd_tt(int M) {
    const int r0 = odd_r0(M), L = M / r0, B = r0 / 2 + 1;
    if (odd_ct_len(M)) return L == 8 ? 9 : L == 12 ? 9 : L == 24 ? 18 : B * L / 16;
    const int a = (B * L + 15) / 16, c = L / 2 + 1;
    return r0 >= 10 && c > a ? c : a;
}
// Padding of the staged rows (one slot per 16 values) and of the subsequences
// (one per first radix), so that strided butterfly accesses spread over the
// banks.
__host__ __device__ constexpr int odd_sh(int M) { return odd_ct_len(M) && odd_ra(M / 16) == 16 ? 4 : 3; }
template <int SH> __host__ __device__ constexpr int zpad(int i) { return i + (i >> SH); }
// zpad(i + t S) for a compile-time stride S.
template <int SH, int S> __device__ __forceinline__ int zstep(int i, int t) {
    if constexpr (S % (1 << SH) == 0) return zpad<SH>(i) + t * (S + (S >> SH));
    else return zpad<SH>(i + t * S);
}
// Complex values of one transform's buffer: the staged row pair, then the
// subsequences in the same place; an even number, so that each buffer starts
// on 16 bytes in both types.  Lengths without a compile-time plan use two.
__host__ __device__ constexpr int odd_buf_len(int M) {
    const int n = M / 2 + (M / 2 >> 4) + 1, bl = (odd_r0(M) / 2 + 1) * (M / odd_r0(M));
    const int z = bl + (bl >> odd_sh(M)) + 1;
    return ((n > z ? n : z) + 1) & ~1;
}
__host__ __device__ constexpr int odd_smem_len(int M) { return odd_ct_len(M) ? odd_buf_len(M) : 2 * odd_buf_len(M); }

// The last stage: radix R0 over the subsequences, for k <= L/2.  get(r, k)
// reads S_r(k); out(i, X) takes the coefficient X(i), 1 <= i < M/2, once each.
template <class T, int R0, class Get, class Out>
__device__ __forceinline__ void odd_last(int M, int L, int k, const typename C2<T>::t *__restrict__ twl, Get get,
                                         Out out) {
    typedef typename C2<T>::t T2;
    constexpr int H = R0 / 2;
    const int km = k == 0 ? 0 : L - k;
    T2 v[R0];
    v[0] = get(0, k);
    if (k == 0) {
#pragma unroll
        for (int r = 1; r <= H; ++r) v[r] = get(r, 0);
#pragma unroll
        for (int r = 1; r < H; ++r) { v[R0 - r].x = -v[r].x; v[R0 - r].y = -v[r].y; }
    } else {
#pragma unroll
        for (int r = 1; r < H; ++r) {
            const T2 w = __ldg(twl + (r - 1) * L + k);
            const T2 a = get(r, k), b = get(r, km);
            v[r] = c_mul(a, w);
            // -conj(w) b
            v[R0 - r].x = -(b.x * w.x + b.y * w.y);
            v[R0 - r].y = b.x * w.y - b.y * w.x;
        }
        v[H] = c_mul(get(H, k), __ldg(twl + (H - 1) * L + k));
    }
    Dft<T, R0>::run(v);
    if (k != 0) out(k, v[0]);
#pragma unroll
    for (int k1 = 1; k1 < H; ++k1) out(k + L * k1, v[k1]);
    if (k != 0 && 2 * k != L) {
#pragma unroll
        for (int k1 = H; k1 < R0; ++k1) {
            T2 x;
            x.x = -v[k1].x;
            x.y = -v[k1].y;
            out(M - k - L * k1, x);
        }
    }
}

// The compile-time transform, in place.  z: this transform's buffer with the
// row pair staged (value i at zpad<4>(i), i = 0 .. N, zero at 0 and N) and a
// barrier taken since; t: thread of the transform (odd_tt(M) threads); the nbar
// threads that synchronise on barrier 1 (0: the CTA's) call it.
template <class T, int M, class Out>
__device__ __forceinline__ void odd_fft_ct(typename C2<T>::t *z, const typename C2<T>::t *__restrict__ tw, int t,
                                           bool live, Out out, int nbar) {
    typedef typename C2<T>::t T2;
    constexpr int L = M / 16, B = 9, TT = odd_tt(M), SH = odd_sh(M), RA = odd_ra(L), RB = L / RA, NA = L / RA;
    static_assert(RA % 2 == 0, "the first radix splits the extension in halves");
    {
        // first stage: the extension's second half is the mirrored, negated first
        constexpr int NB = B * NA, U = (NB + TT - 1) / TT, S = M / RA;
        T2 v[U][RA];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int bf = t + u * TT;
            if (live && (NB % TT == 0 || bf < NB)) {
                const int r = bf / NA, j = bf - r * NA, i0 = r + 16 * j, i1 = S - i0;
#pragma unroll
                for (int q = 0; q < RA / 2; ++q) {
                    v[u][q] = z[zstep<4, S>(i0, q)];
                    const T2 m = z[zstep<4, S>(i1, q)];
                    v[u][RA - 1 - q].x = -m.x;
                    v[u][RA - 1 - q].y = -m.y;
                }
            }
        }
        bar_sync(1, nbar);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int bf = t + u * TT;
            if (live && (NB % TT == 0 || bf < NB)) {
                const int r = bf / NA, j = bf - r * NA;
                Dft<T, RA>::run(v[u]);
#pragma unroll
                for (int q = 0; q < RA; ++q) z[zstep<SH, 1>(r * L + j * RA, q)] = v[u][q];
            }
        }
        bar_sync(1, nbar);
    }
    if constexpr (RB > 1) {
        constexpr int NB1 = L / RB, NB = B * NB1, U = (NB + TT - 1) / TT;
        static_assert(NB1 == RA, "two stages");
        T2 v[U][RB];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int bf = t + u * TT;
            if (live && (NB % TT == 0 || bf < NB)) {
                const int r = bf / NB1, j = bf - r * NB1;
#pragma unroll
                for (int q = 0; q < RB; ++q) v[u][q] = z[zstep<SH, NB1>(r * L + j, q)];
                if (j != 0) {
#pragma unroll
                    for (int q = 1; q < RB; ++q) v[u][q] = c_mul(v[u][q], __ldg(tw + (RA - 1) + (q - 1) * RA + j));
                }
            }
        }
        bar_sync(1, nbar);
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int bf = t + u * TT;
            if (live && (NB % TT == 0 || bf < NB)) {
                const int r = bf / NB1, j = bf - r * NB1;
                Dft<T, RB>::run(v[u]);
#pragma unroll
                for (int q = 0; q < RB; ++q) z[zstep<SH, RA>(r * L + j, q)] = v[u][q];
            }
        }
        bar_sync(1, nbar);
    }
    static_assert(TT >= L / 2 + 1, "one last butterfly per thread");
    if (live && t <= L / 2)
        odd_last<T, 16>(M, L, t, tw + (L - 1), [&](int r, int k) { return z[zpad<SH>(r * L + k)]; }, out);
}

// ---- any length: the same plan at run time, between two buffers, with radices
// up to 16 so that most subsequences take two stages (a barrier and a pass over
// shared memory each).  The stages are out of line: a length runs two or three
// of them, and inlined they spilled the kernel's registers.
template <class T, int R>
__device__ __noinline__ void odd_first_rt(const typename C2<T>::t *src, typename C2<T>::t *dst, int M, int R0, int L,
                                          FastDiv fd, int t, int TT) {
    typedef typename C2<T>::t T2;
    const int nA = L / R, S = M / R, N = M / 2, nb = (R0 / 2 + 1) * nA;
    for (int bf = t; bf < nb; bf += TT) {
        const int r = fd.div(bf), j = bf - r * nA, i0 = r + R0 * j;
        T2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) {
            const int i = i0 + q * S;
            const bool hi = i > N;
            T2 x = src[zpad<4>(hi ? M - i : i)];
            if (hi) { x.x = -x.x; x.y = -x.y; }
            v[q] = x;
        }
        Dft<T, R>::run(v);
#pragma unroll
        for (int q = 0; q < R; ++q) dst[zpad<3>(r * L + j * R + q)] = v[q];
    }
}
template <class T, int R>
__device__ __noinline__ void odd_mid_rt(const typename C2<T>::t *src, typename C2<T>::t *dst, int R0, int L, int Ns,
                                        FastDiv fd, FastDiv fn, const typename C2<T>::t *__restrict__ tws, int t, int TT) {
    typedef typename C2<T>::t T2;
    const int nb1 = L / R, nb = (R0 / 2 + 1) * nb1;
    for (int bf = t; bf < nb; bf += TT) {
        const int r = fd.div(bf), j = bf - r * nb1, q0 = fn.div(j), jm = j - q0 * Ns;
        T2 v[R];
#pragma unroll
        for (int q = 0; q < R; ++q) v[q] = src[zpad<3>(r * L + j + q * nb1)];
        if (jm != 0) {
#pragma unroll
            for (int q = 1; q < R; ++q) v[q] = c_mul(v[q], __ldg(tws + (q - 1) * Ns + jm));
        }
        Dft<T, R>::run(v);
        const int d = r * L + q0 * Ns * R + jm;
#pragma unroll
        for (int q = 0; q < R; ++q) dst[zpad<3>(d + q * Ns)] = v[q];
    }
}
// The radices of a subsequence, largest first; those of later stages (2 and 16
// never are: a plan has the fewest stages, of those the least sum).
#define OQG_ODD_RADICES(X) X(16) X(15) X(12) X(10) X(9) X(8) X(6) X(5) X(4) X(3) X(2)
#define OQG_ODD_LATER(X) X(15) X(12) X(10) X(9) X(8) X(6) X(5) X(4) X(3)
template <class T, class Out>
__device__ __forceinline__ void odd_fft_rt(typename C2<T>::t *a, int M, const BasinDev &b,
                                           const typename C2<T>::t *__restrict__ tw, int t, int TT, bool live, Out out,
                                           int nbar) {
    typedef typename C2<T>::t T2;
    const int R0 = odd_r0(M), L = M / R0, nrad = b.norad;
    T2 *src = a, *dst = a + odd_buf_len(M);
    int Ns = 1;
    // the length's radices, the last of which is R0's own stage below
    for (int s = 0; s < nrad - 1 || s == 0; ++s) {
        const int R = nrad == 1 ? 1 : b.orad[s];
        if (live) {
            const FastDiv fd = b.fd_obf[s], fn = b.fd_ons[s];
            if (s == 0) {
                switch (R) {
#define OQG_ODD_F(RR) case RR: odd_first_rt<T, RR>(src, dst, M, R0, L, fd, t, TT); break;
                    OQG_ODD_RADICES(OQG_ODD_F)
#undef OQG_ODD_F
                    default: odd_first_rt<T, 1>(src, dst, M, R0, L, fd, t, TT); break;
                }
            } else {
                const T2 *tws = tw + (Ns - 1);
                switch (R) {
#define OQG_ODD_M(RR) case RR: odd_mid_rt<T, RR>(src, dst, R0, L, Ns, fd, fn, tws, t, TT); break;
                    OQG_ODD_LATER(OQG_ODD_M)
#undef OQG_ODD_M
                }
            }
        }
        bar_sync(1, nbar);
        T2 *x = src; src = dst; dst = x;
        Ns *= R;
    }
    if (!live) return;
    auto get = [&](int r, int k) { return src[zpad<3>(r * L + k)]; };
    const T2 *twl = tw + (L - 1);
    for (int k = t; k <= L / 2; k += TT) {
        switch (R0) {
            case 16: odd_last<T, 16>(M, L, k, twl, get, out); break;
            case 12: odd_last<T, 12>(M, L, k, twl, get, out); break;
            case 10: odd_last<T, 10>(M, L, k, twl, get, out); break;
            case 8: odd_last<T, 8>(M, L, k, twl, get, out); break;
            default: odd_last<T, 6>(M, L, k, twl, get, out);
        }
    }
}

// MC > 0: an instance of that one length; MC = 0: the compile-time plans
// chosen by the member's length (ensembles); MC < 0: any other length.
#define OQG_ODD_CASE(MM) case MM: odd_fft_ct<T, MM>(z, tw, t, live, out, nbar); return;
template <class T, int MC, class Out>
__device__ __forceinline__ void odd_fft(typename C2<T>::t *z, int M, const BasinDev &b,
                                        const typename C2<T>::t *__restrict__ tw, int t, int TT, bool live, Out out,
                                        int nbar = 0) {
    if constexpr (MC > 0) {
        odd_fft_ct<T, MC>(z, tw, t, live, out, nbar);
    } else if constexpr (MC < 0) {
        odd_fft_rt<T>(z, M, b, tw, t, TT, live, out, nbar);
    } else {
        switch (M) {
            OQG_ODD_CASE(128)
            OQG_ODD_CASE(192)
            OQG_ODD_CASE(256)
            OQG_ODD_CASE(384)
            OQG_ODD_CASE(512)
            OQG_ODD_CASE(1024)
            OQG_ODD_CASE(2048)
            OQG_ODD_CASE(4096)
            default: odd_fft_rt<T>(z, M, b, tw, t, TT, live, out, nbar);
        }
    }
}
#undef OQG_ODD_CASE

}  // namespace oqg
