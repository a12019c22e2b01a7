// The grid transforms: the transform pair with the influence product of a field pass as one cooperative kernel, and
// the bounded barrier of its blocks.
#pragma once

#include "linefft.cuh"

namespace pgmb200 {

// The transform pair with the influence product of a field pass as ONE cooperative kernel: block x of system s
// (blockIdx.y; K0 blocks per system) owns x-plane x and, between two barriers of the system's blocks, a run of
// the x-lines, by the two-pass line transforms of linefft.cuh:
//   1. plane x: its real rows two at a time as one complex row (x + i y), forward along z (real to half
//      spectrum, separated by Hermitian symmetry) and along y, stored to the spectrum F[(x K1 + ky) (K2/2 + 1) + kz];
//   2. (barrier) lines l = ky (K2/2 + 1) + kz in [x lpb, x lpb + lpb): forward along x, the influence product,
//      back along x, in place in the spectrum;
//   3. (barrier) plane x back along y and z into the real grid.
// The exchange goes through L2, so a 48^3 grid spreads over 48 SMs; loads of what other blocks wrote bypass L1
// (__ldcg).  Each barrier waits at most FFTG_SPIN_LIMIT polls; a block that gives up sets flags[11] and returns, and
// the host reports the evaluation as failed.
// Threads per block: a pass of a cubic grid has at most 31 x 10 items (K = 60) or 33 x 8 (K = 64), so 320 threads take any of
// them in one round; 256 in double, so that three blocks fit an SM as many-system launches need them (two rounds at 60 and
// 64).  Other grids can have more, in more rounds: few planes of many lines take their x-lines so (8 x 64 x 64: 264 lines x 4).
template <typename R> struct FftgThreads { static constexpr int n = 256, perSm = 3; };
template <> struct FftgThreads<float> { static constexpr int n = 320, perSm = 2; };
constexpr unsigned FFTG_SPIN_LIMIT = 1u << 22;   // polls of an L2 word (a few hundred ns each): about 1 s

__device__ __forceinline__ unsigned ldAcquireGpu(const unsigned* p) {
    unsigned v;
    asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}

// Barrier of nb blocks over an arrival counter that only grows between resets (the flags and barrier words are
// cleared at the start of every call): the blocks of barrier k arrive as numbers k nb .. k nb + nb - 1 and leave
// once the counter has reached (k + 1) nb.  The wait is bounded: false, with flags[11] set, when it gave up.
__device__ __forceinline__ unsigned atomAddAcqRelGpu(unsigned* p, unsigned v) {
    unsigned old;
    asm volatile("atom.add.acq_rel.gpu.global.u32 %0, [%1], %2;" : "=r"(old) : "l"(p), "r"(v) : "memory");
    return old;
}

// The arrival is a release (it orders the block's writes before it, made the thread's own by the block barrier
// ahead of it) and an acquire (the last block to arrive does not wait), the wait an acquire load, so no separate
// fences are needed and the block's later plain loads see what the other blocks wrote before they arrived.
__device__ __forceinline__ bool fftgBarrier(unsigned* bar, unsigned nb, int* flags) {
    __shared__ int ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        ok = 1;
        const unsigned old = atomAddAcqRelGpu(bar, 1u);
        const unsigned target = (old / nb + 1) * nb;
        if (old + 1 != target)
            for (unsigned it = 0; (int) (ldAcquireGpu(bar) - target) < 0; it++)
                if (it >= FFTG_SPIN_LIMIT) {
                    ok = 0;
                    atomicExch(flags + 11, 1);
                    break;
                }
    }
    __syncthreads();
    return ok != 0;
}

// KC > 0: every grid of the launch is KC^3 (compile-time passes and index maps); 0: any grid.
// ENERGY (the final pass): also the reciprocal energy (1/2) sum w G |F|^2 and its strain derivative, as k_conv
// sums them, from the x-lines' spectrum before the product; block x writes conv partial x of its system and clears
// partials x + K0, x + 2 K0, ... up to the system's convBlocks (the host requires K0 <= convBlocks).
template <typename R, int KC, bool ENERGY = false>
__global__ void __launch_bounds__(FftgThreads<R>::n, FftgThreads<R>::perSm) k_fft_grid(Dev dv, int gateDone) {
    typedef typename CplxT<R>::T C;
    const int s = blockIdx.y;
    if ((gateDone & 1) && dv.scal[s * NSCAL + SC_DONE] != 0.0)
        return;   // every block of the system
    // gateDone & 2: the spread went to the fixed-point grid; its plane is converted (and cleared) on the load
    long long* const fx = (gateDone & 2) ? dv.gridFix : nullptr;
    const SysDev& S = dv.sys[s];
    const int K0 = KC > 0 ? KC : S.K[0], K1 = KC > 0 ? KC : S.K[1], K2 = KC > 0 ? KC : S.K[2];
    const int x = blockIdx.x;
    if (x >= K0)
        return;   // (a smaller grid than the launch's largest)
    const int nT = blockDim.x, tid = threadIdx.x;
    const int gaveUp = tid == 0 ? dv.flags[11] : 0;   // (its load beside the tables')
    extern __shared__ __align__(16) unsigned char smraw[];
    C* W0 = (C*) smraw;
    C* W1 = W0 + FFT_MAXK;
    C* W2 = W1 + FFT_MAXK;
    C* const b0 = W2 + FFT_MAXK;
    C* const b1 = b0 + dv.fftgBuf;
    const C* tw = (const C*) dv.twiddle;
    for (int m = tid; m < K0; m += nT)
        W0[m] = tw[S.twOff[0] + m];
    for (int m = tid; m < K1; m += nT)
        W1[m] = tw[S.twOff[1] + m];
    for (int m = tid; m < K2; m += nT)
        W2[m] = tw[S.twOff[2] + m];
    // A barrier of an earlier launch of this call gave up: its counter is out of step, so every wait here would run out too,
    // a second each in every iteration still enqueued.  The results are undefined already; the host reports the flag.
    if (__syncthreads_or(gaveUp))
        return;
    const PlaneFft<R, KC> fft(K0, K1, K2, b0, b1, W0, W1, W2);
    const int nline = fft.nline, l0 = x * fft.lpb, nl = min(nline, l0 + fft.lpb) - l0;
    R* const gx = (R*) dv.grid + S.gridOff + (size_t) x * K1 * K2;
    C* const spec = (C*) dv.spec + S.specOff;
    C* const plane = spec + (size_t) x * nline;
    unsigned* const bar = dv.fftgBar + 2 * s;
    if (fx) {
        long long* const fxx = fx + S.gridOff + (size_t) x * K1 * K2;
        fft.forward([&](int e) { return (R) gridFixTake(fxx + e); }, plane);
    } else {
        fft.forward([&](int e) { return gx[e]; }, plane);
    }
    if (!fftgBarrier(bar, (unsigned) K0, dv.flags))
        return;
    const R* infl = (const R*) dv.infl + S.specOff;
    double acc[ENERGY ? NCONV : 1];
#pragma unroll
    for (int k = 0; k < (ENERGY ? NCONV : 1); k++)
        acc[k] = 0.0;
    const double fac = PI_D * PI_D / (S.beta * S.beta);
    fft.lines(spec, l0, nl, [&](int m1, int l, C v) {
        const R gk = infl[(size_t) m1 * nline + l];
        if (ENERGY && (m1 != 0 || l != 0)) {   // (the k = 0 term is left out, as k_conv does)
            const int K2h = K2 / 2 + 1, m3 = l % K2h, m2 = l / K2h;
            const double w = (m3 == 0 || ((K2 & 1) == 0 && m3 == K2 / 2)) ? 1.0 : 2.0;
            const double nrm = (double) v.x * v.x + (double) v.y * v.y;
            const double en = 0.5 * w * (double) gk * nrm;
            acc[0] += en;
            const double mm1 = (m1 <= K0 / 2) ? m1 : m1 - K0, mm2 = (m2 <= K1 / 2) ? m2 : m2 - K1, mm3 = m3;
            double ms[3];
#pragma unroll
            for (int k = 0; k < 3; k++)
                ms[k] = mm1 * S.recip[3 * k] + mm2 * S.recip[3 * k + 1] + mm3 * S.recip[3 * k + 2];
            const double m2s = ms[0] * ms[0] + ms[1] * ms[1] + ms[2] * ms[2];
            const double c2 = 2.0 * (fac + 1.0 / m2s);
#pragma unroll
            for (int a = 0; a < 3; a++)
#pragma unroll
                for (int b = 0; b < 3; b++)
                    acc[ENERGY ? 1 + 3 * a + b : 0] += en * ((a == b ? -1.0 : 0.0) + c2 * ms[a] * ms[b]);
        }
        v.x *= gk;
        v.y *= gk;
        return v;
    });
    if (ENERGY) {
        blockReduce<NCONV>(acc, 0u);
        if (tid == 0)
            for (int k = 0; k < NCONV; k++)
                dv.convPartial[(size_t) (dv.convPartialOff[s] + x) * NCONV + k] = acc[k];
        if (tid < NCONV * 16)
            for (int b = x + K0 * (1 + tid / NCONV); b < S.convBlocks; b += 16 * K0)
                dv.convPartial[(size_t) (dv.convPartialOff[s] + b) * NCONV + tid % NCONV] = 0.0;
    }
    if (!fftgBarrier(bar, (unsigned) K0, dv.flags))
        return;
    fft.inverse(plane, [&](int e, R v) { gx[e] = v; });
}

}  // namespace pgmb200
