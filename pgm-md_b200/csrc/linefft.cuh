// Line transforms of length K = A B as two butterfly passes (A <= B, radices up to 10), and the three phases of a
// plane-per-block 3D real transform pair with the influence product built from them.
//
// Why two passes: a plane block holds only K/2 .. K lines, so a pass is bound by its latency (a shared-memory round
// trip and a block barrier), not by its arithmetic.  Radices up to 10 make every grid size up to 64 two passes
// instead of three or four, the loads and the stores of global memory, the separation of the row pairs, the influence
// product and the inverse's first pass all fold into a pass, and a transform pair takes 11 passes with 8 block
// barriers (the radix-4/2/3/5 passes it replaces took 27 at 48^3).  Measured at 48^3 (one B200, k_fft_grid back to
// back): float 16.5 -> 11.3 us; double 12.7 us, where cuFFT's D2Z and Z2D with the product kernel take 30.1.
#pragma once

#include "common.cuh"

#include <type_traits>

namespace pgmb200 {

constexpr int FFT_MAXK = 64;

// K = A B with A <= B <= 10: 0 when K has no such split (every K <= 64 with the prime factors 2, 3, 5 has one).
__host__ __device__ constexpr int fftSplitA(int K) {
    for (int A = 8; A >= 1; A--)
        if (A != 7 && K % A == 0) {
            const int B = K / A;
            if (A <= B && B <= 10 && B != 7)
                return A;
        }
    return 0;
}

// In-register transforms of length N, sign DIR (-1 forward, +1 inverse), unnormalised.
template <typename R, int N, int DIR> struct Dft;
template <typename R, int DIR> struct Dft<R, 1, DIR> {
    static __device__ __forceinline__ void run(R*, R*) {}
};
template <typename R, int DIR> struct Dft<R, 2, DIR> {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        const R ar = xr[0] + xr[1], ai = xi[0] + xi[1];
        xr[1] = xr[0] - xr[1];
        xi[1] = xi[0] - xi[1];
        xr[0] = ar;
        xi[0] = ai;
    }
};
template <typename R, int DIR> struct Dft<R, 3, DIR> {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        const R s = (R) (DIR * 0.86602540378443864676);   // DIR sin(2 pi / 3)
        const R tr = xr[1] + xr[2], ti = xi[1] + xi[2];
        const R ur = xr[0] - (R) 0.5 * tr, ui = xi[0] - (R) 0.5 * ti;
        const R dr = s * (xr[1] - xr[2]), di = s * (xi[1] - xi[2]);   // i s (x1 - x2) = (-di, dr)
        xr[0] += tr;
        xi[0] += ti;
        xr[1] = ur - di;
        xi[1] = ui + dr;
        xr[2] = ur + di;
        xi[2] = ui - dr;
    }
};
template <typename R, int DIR> struct Dft<R, 4, DIR> {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        const R ar = xr[0] + xr[2], ai = xi[0] + xi[2], br = xr[0] - xr[2], bi = xi[0] - xi[2];
        const R cr = xr[1] + xr[3], ci = xi[1] + xi[3], er = xr[1] - xr[3], ei = xi[1] - xi[3];
        const R dr = (R) (-DIR) * ei, di = (R) DIR * er;   // (x1 - x3) DIR i
        xr[0] = ar + cr;
        xi[0] = ai + ci;
        xr[1] = br + dr;
        xi[1] = bi + di;
        xr[2] = ar - cr;
        xi[2] = ai - ci;
        xr[3] = br - dr;
        xi[3] = bi - di;
    }
};
template <typename R, int DIR> struct Dft<R, 5, DIR> {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        const R c1 = (R) 0.30901699437494742410, c2 = (R) -0.80901699437494742410;   // cos(2 pi/5), cos(4 pi/5)
        const R s1 = (R) (DIR * 0.95105651629515357212), s2 = (R) (DIR * 0.58778525229247312917);
        const R ar = xr[1] + xr[4], ai = xi[1] + xi[4], br = xr[2] + xr[3], bi = xi[2] + xi[3];
        const R cr = xr[1] - xr[4], ci = xi[1] - xi[4], dr = xr[2] - xr[3], di = xi[2] - xi[3];
        const R pr = xr[0] + c1 * ar + c2 * br, pi = xi[0] + c1 * ai + c2 * bi;
        const R qr = xr[0] + c2 * ar + c1 * br, qi = xi[0] + c2 * ai + c1 * bi;
        const R ur = s1 * cr + s2 * dr, ui = s1 * ci + s2 * di;   // y1 = p + i u, y4 = p - i u
        const R vr = s2 * cr - s1 * dr, vi = s2 * ci - s1 * di;   // y2 = q + i v, y3 = q - i v
        xr[0] += ar + br;
        xi[0] += ai + bi;
        xr[1] = pr - ui;
        xi[1] = pi + ur;
        xr[4] = pr + ui;
        xi[4] = pi - ur;
        xr[2] = qr - vi;
        xi[2] = qi + vr;
        xr[3] = qr + vi;
        xi[3] = qi - vr;
    }
};
// N = 2 M, M odd, by the prime-factor map: n = M a + 2 b, k = M c + (M + 1) d (mod N) leave no twiddles.
template <typename R, int M, int DIR> struct DftTwiceOdd {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        constexpr int N = 2 * M;
        R yr[2][M], yi[2][M];
#pragma unroll
        for (int a = 0; a < 2; a++) {
#pragma unroll
            for (int b = 0; b < M; b++) {
                yr[a][b] = xr[(M * a + 2 * b) % N];
                yi[a][b] = xi[(M * a + 2 * b) % N];
            }
            Dft<R, M, DIR>::run(yr[a], yi[a]);
        }
#pragma unroll
        for (int d = 0; d < M; d++) {
            xr[((M + 1) * d) % N] = yr[0][d] + yr[1][d];
            xi[((M + 1) * d) % N] = yi[0][d] + yi[1][d];
            xr[(M + (M + 1) * d) % N] = yr[0][d] - yr[1][d];
            xi[(M + (M + 1) * d) % N] = yi[0][d] - yi[1][d];
        }
    }
};
template <typename R, int DIR> struct Dft<R, 6, DIR> : DftTwiceOdd<R, 3, DIR> {};
template <typename R, int DIR> struct Dft<R, 10, DIR> : DftTwiceOdd<R, 5, DIR> {};
template <typename R, int DIR> struct Dft<R, 8, DIR> {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        R er[4], ei[4], orr[4], oi[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            er[k] = xr[2 * k];
            ei[k] = xi[2 * k];
            orr[k] = xr[2 * k + 1];
            oi[k] = xi[2 * k + 1];
        }
        Dft<R, 4, DIR>::run(er, ei);
        Dft<R, 4, DIR>::run(orr, oi);
        const R h = (R) 0.70710678118654752440;
        // odd part times exp(DIR 2 pi i k / 8)
        const R t1r = h * (orr[1] - DIR * oi[1]), t1i = h * (oi[1] + DIR * orr[1]);
        const R t2r = -DIR * oi[2], t2i = DIR * orr[2];
        const R t3r = -h * (orr[3] + DIR * oi[3]), t3i = h * (DIR * orr[3] - oi[3]);
        orr[1] = t1r;
        oi[1] = t1i;
        orr[2] = t2r;
        oi[2] = t2i;
        orr[3] = t3r;
        oi[3] = t3i;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            xr[k] = er[k] + orr[k];
            xi[k] = ei[k] + oi[k];
            xr[k + 4] = er[k] - orr[k];
            xi[k + 4] = ei[k] - oi[k];
        }
    }
};
template <typename R, int DIR> struct Dft<R, 9, DIR> {
    static __device__ __forceinline__ void run(R* xr, R* xi) {
        // cos and sin of 2 pi m / 9, m = 1, 2, 4
        constexpr double cs[5] = {1.0, 0.76604444311897803520, 0.17364817766693034885, 0.0, -0.93969262078590838405};
        constexpr double sn[5] = {0.0, 0.64278760968653932632, 0.98480775301220805937, 0.0, 0.34202014332566873304};
        R yr[3][3], yi[3][3];
#pragma unroll
        for (int b = 0; b < 3; b++) {   // n = 3 a + b
#pragma unroll
            for (int a = 0; a < 3; a++) {
                yr[b][a] = xr[3 * a + b];
                yi[b][a] = xi[3 * a + b];
            }
            Dft<R, 3, DIR>::run(yr[b], yi[b]);
        }
#pragma unroll
        for (int c = 0; c < 3; c++) {   // k = c + 3 d
            R zr[3] = {yr[0][c], 0, 0}, zi[3] = {yi[0][c], 0, 0};
#pragma unroll
            for (int b = 1; b < 3; b++) {
                const R wr = (R) cs[b * c], wi = (R) (DIR * sn[b * c]);
                zr[b] = yr[b][c] * wr - yi[b][c] * wi;
                zi[b] = yr[b][c] * wi + yi[b][c] * wr;
            }
            Dft<R, 3, DIR>::run(zr, zi);
#pragma unroll
            for (int d = 0; d < 3; d++) {
                xr[c + 3 * d] = zr[d];
                xi[c + 3 * d] = zi[d];
            }
        }
    }
};

// e / K for 0 <= e < 2^20, K >= 1 without an integer division: (e + 1/2) / K lies at least 1/(2K) from an
// integer and the float product errs by at most about 2^-23 (e + 1/2) / K < 1/(8K), so truncation gives the
// exact quotient.
__device__ __forceinline__ int fdiv(int e, float invK) { return __float2int_rz(((float) e + 0.5f) * invK); }

// The length K of one dimension and its split into the two passes' radices, compile-time (KC > 0, K = KC) or not; first and
// second call f with a pass's radix as a constant (a switch where it is a run-time one).
template <int KC> struct Split {
    static constexpr int K = KC, A = fftSplitA(KC), B = KC / (fftSplitA(KC) > 0 ? fftSplitA(KC) : 1);
    __device__ __forceinline__ explicit Split(int) {}
    // f(radix) for the first / second pass's radix
    template <typename F> __device__ __forceinline__ void first(F&& f) const { f(std::integral_constant<int, A>()); }
    template <typename F> __device__ __forceinline__ void second(F&& f) const { f(std::integral_constant<int, B>()); }
};
template <> struct Split<0> {
    int K, A, B;
    __device__ __forceinline__ explicit Split(int k) : K(k), A(fftSplitA(k)) { B = k / A; }
    template <typename F> static __device__ __forceinline__ void pick(int r, F&& f) {
        switch (r) {
        case 1: f(std::integral_constant<int, 1>()); break;
        case 2: f(std::integral_constant<int, 2>()); break;
        case 3: f(std::integral_constant<int, 3>()); break;
        case 4: f(std::integral_constant<int, 4>()); break;
        case 5: f(std::integral_constant<int, 5>()); break;
        case 6: f(std::integral_constant<int, 6>()); break;
        case 8: f(std::integral_constant<int, 8>()); break;
        case 9: f(std::integral_constant<int, 9>()); break;
        default: f(std::integral_constant<int, 10>());
        }
    }
    template <typename F> __device__ __forceinline__ void first(F&& f) const { pick(A, f); }
    template <typename F> __device__ __forceinline__ void second(F&& f) const { pick(B, f); }
};

// One item of a pass: RAD values loaded by load(m), transformed, multiplied by the twiddles exp(DIR 2 pi i m t / K)
// (tw: the table exp(-2 pi i j / K); null: none) and stored by store(m, value).
template <typename R, int RAD, int DIR, typename L, typename St>
__device__ __forceinline__ void fftItem(L&& load, const typename CplxT<R>::T* tw, int t, St&& store) {
    typedef typename CplxT<R>::T C;
    R xr[RAD], xi[RAD];
#pragma unroll
    for (int m = 0; m < RAD; m++) {
        const C v = load(m);
        xr[m] = v.x;
        xi[m] = v.y;
    }
    Dft<R, RAD, DIR>::run(xr, xi);
#pragma unroll
    for (int m = 0; m < RAD; m++) {
        C o;
        if (tw && m > 0) {
            const C w = tw[m * t];
            const R wy = DIR < 0 ? w.y : -w.y;
            o.x = xr[m] * w.x - xi[m] * wy;
            o.y = xr[m] * wy + xi[m] * w.x;
        } else {
            o.x = xr[m];
            o.y = xi[m];
        }
        store(m, o);
    }
}

// Complex elements of each of the two transform buffers of a plane block for grid K (the plane's rows and columns and
// its x-lines, each padded to an odd stride).
__host__ __device__ inline int fftgBufferElems(const int* K) {
    const int K2h = K[2] / 2 + 1, P = (K[1] + 1) / 2;
    const int lpb = (K[1] * K2h + K[0] - 1) / K[0];
    int m = P * (K[2] | 1);
    m = m > K2h * (K[1] | 1) ? m : K2h * (K[1] | 1);
    m = m > K[1] * (K2h | 1) ? m : K[1] * (K2h | 1);
    m = m > lpb * (K[0] | 1) ? m : lpb * (K[0] | 1);
    return (m + 1) / 2 * 2;   // 16-byte multiples
}

// The phases of one plane block (every thread of the block calls them; KC > 0: the grid is KC^3).  b0 and b1 are the
// block's two buffers, W0 .. W2 the twiddle tables exp(-2 pi i m / K) of the three dimensions in shared memory.
template <typename R, int KC> struct PlaneFft {
    typedef typename CplxT<R>::T C;
    const Split<KC> s0, s1, s2;
    const int K2h, P, nline, lpb, lz, ly, lx, lh, tid, nT;
    C *const b0, *const b1;
    const C *const W0, *const W1, *const W2;

    __device__ __forceinline__ PlaneFft(int K0, int K1, int K2, C* b0_, C* b1_, const C* w0, const C* w1, const C* w2)
        : s0(K0), s1(K1), s2(K2), K2h(s2.K / 2 + 1), P((s1.K + 1) / 2), nline(s1.K * (s2.K / 2 + 1)),
          lpb((s1.K * (s2.K / 2 + 1) + s0.K - 1) / s0.K), lz(s2.K | 1), ly(s1.K | 1), lx(s0.K | 1),
          lh((s2.K / 2 + 1) | 1), tid(threadIdx.x), nT(blockDim.x), b0(b0_), b1(b1_), W0(w0), W1(w1), W2(w2) {}

    // e / d: by a constant when the grid is one (the compiler multiplies), else through the float reciprocal
    static __device__ __forceinline__ int quot(int e, int d) {
        if constexpr (KC > 0)
            return e / d;
        else
            return fdiv(e, __frcp_rn((float) d));
    }

    // The plane's real rows, take(index in the plane), two at a time as one complex row, forward along z; separated
    // (X = (Z_k + conj Z_-k) / 2, Y = (Z_k - conj Z_-k) / 2i) and forward along y; plane[ky K2h + kz].
    template <typename T> __device__ __forceinline__ void forward(T&& take, C* plane) const {
        const int K1 = s1.K, K2 = s2.K;
        s2.first([&](auto rad) {
            constexpr int A = decltype(rad)::value;
            const int B = s2.B;
            for (int t = tid; t < P * B; t += nT) {
                const int pr = quot(t, B), n2 = t - pr * B;
                fftItem<R, A, -1>(
                    [&](int m) {
                        const int z = B * m + n2;
                        C v;
                        v.x = take(2 * pr * K2 + z);
                        v.y = (2 * pr + 1 < K1) ? take((2 * pr + 1) * K2 + z) : (R) 0;
                        return v;
                    },
                    W2, n2, [&](int m, C v) { b0[pr * lz + m * B + n2] = v; });
            }
        });
        __syncthreads();
        s2.second([&](auto rad) {
            constexpr int B = decltype(rad)::value;
            const int A = s2.A;
            for (int t = tid; t < P * A; t += nT) {
                const int pr = quot(t, A), k1 = t - pr * A;
                fftItem<R, B, -1>([&](int m) { return b0[pr * lz + k1 * B + m]; }, nullptr, 0,
                                  [&](int m, C v) { b1[pr * lz + k1 + A * m] = v; });
            }
        });
        __syncthreads();
        s1.first([&](auto rad) {
            constexpr int A = decltype(rad)::value;
            const int B = s1.B;
            for (int t = tid; t < K2h * B; t += nT) {
                const int n2 = quot(t, K2h), kz = t - n2 * K2h, km = kz == 0 ? 0 : K2 - kz;
                fftItem<R, A, -1>(
                    [&](int m) {
                        const int y = B * m + n2;
                        const C zk = b1[(y >> 1) * lz + kz], zm = b1[(y >> 1) * lz + km];
                        C v;
                        if (y & 1) {
                            v.x = (R) 0.5 * (zk.y + zm.y);
                            v.y = (R) 0.5 * (zm.x - zk.x);
                        } else {
                            v.x = (R) 0.5 * (zk.x + zm.x);
                            v.y = (R) 0.5 * (zk.y - zm.y);
                        }
                        return v;
                    },
                    W1, n2, [&](int m, C v) { b0[kz * ly + m * B + n2] = v; });
            }
        });
        __syncthreads();
        s1.second([&](auto rad) {
            constexpr int B = decltype(rad)::value;
            const int A = s1.A;
            for (int t = tid; t < K2h * A; t += nT) {
                const int k1 = quot(t, K2h), kz = t - k1 * K2h;
                fftItem<R, B, -1>([&](int m) { return b0[kz * ly + k1 * B + m]; }, nullptr, 0,
                                  [&](int m, C v) { plane[(k1 + A * m) * K2h + kz] = v; });
            }
        });
    }

    // The x-lines l0 .. l0 + nl - 1 of the spectrum spec[x nline + l] (other blocks' planes: read past L1): forward
    // along x, product(x, line in the plane, value) in place of each value, back along x.
    template <typename Pr> __device__ __forceinline__ void lines(C* spec, int l0, int nl, Pr&& product) const {
        if (nl <= 0)
            return;
        s0.first([&](auto rad) {
            constexpr int A = decltype(rad)::value;
            const int B = s0.B;
            for (int t = tid; t < nl * B; t += nT) {
                const int n2 = fdiv(t, __frcp_rn((float) nl)), li = t - n2 * nl;
                const C* src = spec + l0 + li;
                fftItem<R, A, -1>([&](int m) { return __ldcg(src + (size_t) (B * m + n2) * nline); }, W0, n2,
                                  [&](int m, C v) { b0[li * lx + m * B + n2] = v; });
            }
        });
        __syncthreads();
        s0.second([&](auto rad) {
            constexpr int B = decltype(rad)::value;
            const int A = s0.A;
            for (int t = tid; t < nl * A; t += nT) {
                const int k1 = fdiv(t, __frcp_rn((float) nl)), li = t - k1 * nl;
                C* row = b0 + li * lx + k1 * B;
                R xr[B], xi[B];
#pragma unroll
                for (int m = 0; m < B; m++) {
                    xr[m] = row[m].x;
                    xi[m] = row[m].y;
                }
                Dft<R, B, -1>::run(xr, xi);
#pragma unroll
                for (int m = 0; m < B; m++) {
                    C v;
                    v.x = xr[m];
                    v.y = xi[m];
                    v = product(k1 + A * m, l0 + li, v);
                    xr[m] = v.x;
                    xi[m] = v.y;
                }
                Dft<R, B, 1>::run(xr, xi);
#pragma unroll
                for (int m = 0; m < B; m++) {   // conjugate twiddles: the inverse's first half
                    const C w = W0[k1 * m];
                    C o;
                    o.x = xr[m] * w.x + xi[m] * w.y;
                    o.y = xi[m] * w.x - xr[m] * w.y;
                    row[m] = o;
                }
            }
        });
        __syncthreads();
        s0.first([&](auto rad) {
            constexpr int A = decltype(rad)::value;
            const int B = s0.B;
            for (int t = tid; t < nl * B; t += nT) {
                const int n2 = fdiv(t, __frcp_rn((float) nl)), li = t - n2 * nl;
                C* dst = spec + l0 + li;
                fftItem<R, A, 1>([&](int m) { return b0[li * lx + m * B + n2]; }, nullptr, 0,
                                 [&](int m, C v) { dst[(size_t) (B * m + n2) * nline] = v; });
            }
        });
    }

    // The plane back along y and z (imaginary parts at kz = 0 and the Nyquist index dropped, as a C2R transform does),
    // its rows two at a time, put(index in the plane, value).
    template <typename T> __device__ __forceinline__ void inverse(const C* plane, T&& put) const {
        const int K1 = s1.K, K2 = s2.K;
        s1.second([&](auto rad) {
            constexpr int B = decltype(rad)::value;
            const int A = s1.A;
            for (int t = tid; t < K2h * A; t += nT) {
                const int k1 = quot(t, K2h), kz = t - k1 * K2h;
                fftItem<R, B, 1>([&](int m) { return __ldcg(plane + (k1 + A * m) * K2h + kz); }, W1, k1,
                                 [&](int m, C v) { b0[kz * ly + k1 * B + m] = v; });
            }
        });
        __syncthreads();
        s1.first([&](auto rad) {
            constexpr int A = decltype(rad)::value;
            const int B = s1.B;
            for (int t = tid; t < K2h * B; t += nT) {
                const int n2 = quot(t, K2h), kz = t - n2 * K2h;
                fftItem<R, A, 1>([&](int m) { return b0[kz * ly + m * B + n2]; }, nullptr, 0,
                                 [&](int m, C v) { b1[(B * m + n2) * lh + kz] = v; });
            }
        });
        __syncthreads();
        s2.second([&](auto rad) {
            constexpr int B = decltype(rad)::value;
            const int A = s2.A;
            for (int t = tid; t < P * A; t += nT) {
                const int pr = quot(t, A), k1 = t - pr * A;
                const C* row = b1 + 2 * pr * lh;
                const bool two = 2 * pr + 1 < K1;
                fftItem<R, B, 1>(
                    [&](int m) {   // X + i Y of the two rows' half spectra, the upper half by conjugation
                        const int k = k1 + A * m;
                        const bool upper = k >= K2h, realOnly = (k == 0) || ((K2 & 1) == 0 && k == K2 / 2);
                        const int kk = upper ? K2 - k : k;
                        C X = row[kk], Y;
                        Y.x = 0;
                        Y.y = 0;
                        if (two)
                            Y = row[lh + kk];
                        const R sg = realOnly ? (R) 0 : upper ? (R) -1 : (R) 1;
                        C z;
                        z.x = X.x - sg * Y.y;
                        z.y = sg * X.y + Y.x;
                        return z;
                    },
                    W2, k1, [&](int m, C v) { b0[pr * lz + k1 * B + m] = v; });
            }
        });
        __syncthreads();
        s2.first([&](auto rad) {
            constexpr int A = decltype(rad)::value;
            const int B = s2.B;
            for (int t = tid; t < P * B; t += nT) {
                const int pr = quot(t, B), n2 = t - pr * B;
                fftItem<R, A, 1>([&](int m) { return b0[pr * lz + m * B + n2]; }, nullptr, 0,
                                 [&](int m, C v) {
                                     const int z = B * m + n2;
                                     put(2 * pr * K2 + z, v.x);
                                     if (2 * pr + 1 < K1)
                                         put((2 * pr + 1) * K2 + z, v.y);
                                 });
            }
        });
    }
};

}  // namespace pgmb200
