// The CG solve of one system in mixed precision as ONE persistent cooperative kernel (one block per SM), for
// grids whose dimensions have at most FFT_MAXK points and the prime factors 2, 3, 5: the right-hand side, the initial
// guess, A x0, every iteration of core/pgm_core.cpp:297-385 (A v = v/alpha - T v; T v = pair + reciprocal + self field)
// and the convergence test, with barriers of the launch's blocks in place of kernel boundaries and graph nodes.
//
// A block owns a run of slots.  Their x, r, p, A p, alpha and spline coefficients stay in its shared memory from the
// first pass to the last, so an iteration meets global memory only where blocks exchange data:
//
//   S  (every block, 16 lanes per slot) the direction's float copy for the pair pass, its PME weights (q, e_a = K_a p .
//      recip[:, a]) and the spread into the 64-bit fixed-point grid (global atomics, the points and arithmetic of
//      k_spread; integer sums do not depend on their order, so the solve repeats bit for bit);      grid barrier
//   F  blocks 0 .. K0-1 own the x-planes of the PME grid: the plane is read from the fixed-point grid (and cleared for
//      the next spread), transformed, its share of the x-lines multiplied by the influence function (two barriers of
//      the plane blocks; linefft.cuh) and transformed back into the potential grid.  The others run the
//      direct-space field pass of the direction over the pair records (the plane blocks join in when there are many).
//      grid barrier
//   G  (every block, 16 lanes per slot) E_rec at the atom from the potential grid, the atom's row of A p and the block's
//      shares of p . A p, z . A p and A p . alpha A p;                                                grid barrier
//   U  (every block, its own slots) alph = rz / p.Ap, r' = r - alph A p, z' = alpha r'.  The next direction's beta
//      follows from the same sums, z'.(r' - r) = -alph (z.Ap - alph Ap.alpha Ap), so it needs no exchange of its own
//      and U runs into the next S.  r'.z', which the next alph needs, and max |z'|, which the convergence test needs,
//      go around with the next S's barrier (a recurrence for r'.z' would keep the rounding of the first one); the
//      spread of the iteration after the last is then dropped (the plane blocks clear it).
//
// What bounds it (8550 atoms, 48^3, one B200): the chain of phases and barriers, in us an iteration S 4.7, F 13.5 (the pair
// pass's 61 MB of records through L2 on 100 SMs; the plane blocks take 10), G 3.2, U with its sums 2.7, barriers 9.  With
// p, x, r in global memory, a barrier more, the pair pass's sources read past L1 and 512 threads, an evaluation of ten
// iterations took 691 us against 593.
//
// Every reduction sums in a fixed order.  The barriers' acquire makes what other blocks wrote visible to plain loads, so
// the pair pass's gathers and the stencil's reads share lines through L1.
// Barrier waits are bounded (about a second); a block that gives up sets flags[11] and returns, and the host
// reports the evaluation as failed.
#pragma once

#include "gridfft.cuh"

namespace pgmb200 {

// 1024 threads (64 registers): the pair pass keeps 98 KB of records in flight per SM; with 512 threads it took 17.2 us
// (8550 atoms) where 1024 take 13.
constexpr int PCG_THREADS = 1024;
constexpr int PCG_MAX_BLOCKS = 160;          // the totals' loads are unrolled for at most this many blocks
constexpr int PCG_MIN_PAIR_BLOCKS = 16;      // blocks left for the pair pass beside the plane blocks
constexpr int PCG_SLOT_LANES = 16;           // lanes per slot in the spread and gather phases
// The rule (selectTransforms) takes the kernel up to this much dynamic shared memory a block: with its static part and the
// 1 KB that the system keeps it still fits the 196 KB split of an SM, and the pair pass has 60 KB of L1; beyond, the split is
// 228 KB and the gathers of the pair pass miss (an evaluation of 85500 atoms at 64^3 takes 3062 us, of 87000 3453).
constexpr size_t PCG_RULE_SMEM = 198000;
// Directed pairs that a block sums while a plane block transforms its plane (9.9 us at 48^3): the plane blocks take
// that many fewer of the pair pass's rows, if any.  Measured at 48^3 and used for every grid; what a third / three times as
// many would give, us an evaluation: 648 atoms (20^3) 271 / 271 for 271, 12288 (50^3) 679 / 667 for 668, 26244 (64^3) 1073 /
// 1146 for 1073, 60000 (64^3) 2154 / 2243 for 2173; coarse grids of many atoms would take the lower one, 12288 (32^3) 618 /
// 631 for 630, 26244 (32^3) 1111 / 1147 for 1127.
constexpr int PCG_PLANE_PAIRS = 32000;
constexpr int PCG_SPL = 40;                  // floats per slot of the spline rows: theta, dtheta [3][6], padded so that
                                             // the four slots of a warp read different banks

// The spline record of one atom of the plane-owner kernels' bins (order P): its slot, b1, b2 and b0 mod K0, and
// theta and dtheta of the three dimensions, c[dim 2P + kind P + j].
template <int P> struct PmeRec {
    int4 idx;
    float c[6 * P];
};

// Shared memory of a block for the transforms' tables and buffers (fftgBuf complex elements each), and the state of its
// `per` slots (a multiple of 16 bytes).
__host__ __device__ inline size_t pcgTransformBytes(int fftgBuf) {
    return (3 * (size_t) FFT_MAXK + 2 * (size_t) fftgBuf) * sizeof(float2);
}
__host__ __device__ inline size_t pcgStateBytes(int per) {
    return ((size_t) per * (13 * 8 + PCG_SPL * 4 + 4 * 4) + 15) / 16 * 16;
}

// A load that leaves no line behind in L1 (the pair records, read once per pass).
__device__ __forceinline__ float4 loadStreaming(const float4* p) {
    float4 v;
    asm("ld.global.L1::no_allocate.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p));
    return v;
}
__device__ __forceinline__ float2 loadStreaming(const float2* p) {
    float2 v;
    asm("ld.global.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

// Direct-space field of the dipoles dS (mixed pair records) at slots s0 .. s1 - 1, a warp per slot: E_i = sum_j -p_j G1 +
// (p_j . x) x G2 (core/pgm_core.cpp:274-284), products in float, sums across lanes in double, written to E (slot order).
__device__ __forceinline__ void pcgPairField(const Dev& dv, double* E, int s0, int s1) {
    const int lane = threadIdx.x & 31;
    const float4* dS = (const float4*) dv.dS;
    for (int slot = s0 + (threadIdx.x >> 5); slot < s1; slot += PCG_THREADS / 32) {
        const float4* arow = (const float4*) dv.pairA + (size_t) slot * dv.cap;
        const float2* brow = (const float2*) dv.pairB + (size_t) slot * dv.cap;
        const int cnt = dv.listCount[slot];
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
#pragma unroll 4
        for (int t = lane; t < cnt; t += 32) {
            const float4 xg = loadStreaming(arow + t);
            const float2 gb = loadStreaming(brow + t);
            const float4 dj = dS[realAsSlot(gb.y)];
            const float c = (dj.x * xg.x + dj.y * xg.y + dj.z * xg.z) * gb.x;
            a0 += c * xg.x - dj.x * xg.w;
            a1 += c * xg.y - dj.y * xg.w;
            a2 += c * xg.z - dj.z * xg.w;
        }
        double E0 = a0, E1 = a1, E2 = a2;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            E0 += __shfl_xor_sync(0xffffffffu, E0, o);
            E1 += __shfl_xor_sync(0xffffffffu, E1, o);
            E2 += __shfl_xor_sync(0xffffffffu, E2, o);
        }
        if (lane < 3)
            E[3 * (size_t) slot + lane] = lane == 0 ? E0 : lane == 1 ? E1 : E2;
    }
}

// Sums over a warp (or the largest, where the bit of maxMask is set), in every lane.
template <int NV> __device__ __forceinline__ void pcgWarpSums(double* v, unsigned maxMask) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < NV; k++) {
            const double y = __shfl_xor_sync(0xffffffffu, v[k], o);
            v[k] = ((maxMask >> k) & 1u) ? fmax(v[k], y) : v[k] + y;
        }
}

// The block's share of NV values into part[k * nb + x] (thread 0), in a fixed order; one block barrier.
template <int NV>
__device__ __forceinline__ void pcgShare(double* v, unsigned maxMask, double* part, int nb) {
    __shared__ double red[NV][PCG_THREADS / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    pcgWarpSums<NV>(v, maxMask);
    if (lane < NV)
        red[lane][wid] = NV == 1 || lane == 0 ? v[0] : lane == 1 ? v[NV > 1 ? 1 : 0] : v[NV > 2 ? 2 : 0];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int k = 0; k < NV; k++)
            v[k] = red[k][lane];
        pcgWarpSums<NV>(v, maxMask);
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < NV; k++)
                part[(size_t) k * nb + blockIdx.x] = v[k];
    }
}

// The blocks' shares part[k * nb + b] of NV values, summed (or the largest) in a fixed order by every warp for itself:
// after a barrier of the blocks, without one of the block's own.
template <int NV>
__device__ __forceinline__ void pcgTotals(const double* part, int nb, unsigned maxMask, double* tot) {
    const int lane = threadIdx.x & 31;
    double x[NV][PCG_MAX_BLOCKS / 32];
#pragma unroll
    for (int k = 0; k < NV; k++)
#pragma unroll
        for (int m = 0; m < PCG_MAX_BLOCKS / 32; m++)
            x[k][m] = lane + 32 * m < nb ? part[(size_t) k * nb + lane + 32 * m] : 0.0;
#pragma unroll
    for (int k = 0; k < NV; k++) {
        tot[k] = x[k][0];
#pragma unroll
        for (int m = 1; m < PCG_MAX_BLOCKS / 32; m++)
            tot[k] = ((maxMask >> k) & 1u) ? fmax(tot[k], x[k][m]) : tot[k] + x[k][m];
    }
    pcgWarpSums<NV>(tot, maxMask);
}

// KC > 0: the grid is KC^3 (compile-time line transforms); 0: any grid the plane blocks handle.  The right-hand side is
// E_perm = E_pair + E_rec + self field of the permanent dipoles (written to b), or, with the control's customRhs, b.
// planeSlots: the rows of the pair pass that a plane block's transforms are worth.
// SHARED: the slots' state in shared memory; else, for more atoms than that holds, in the block's part of dv.pcgState.
// finish: also the final pass's preparation (k_final_prep: mu = x + peek alpha r, the total dipoles, the self and
// polarization energies, the history) and its spread of (q, d), from the state that the blocks hold: two launches
// and their loads less (480 -> 468 us an evaluation at 4104 atoms, 412 -> 395 at 1900; even at 8550).
template <int P, int KC, bool SHARED = true>
__global__ void __launch_bounds__(PCG_THREADS, 1) k_cg_persistent(Dev dv, int planeSlots, int finish) {
    typedef cufftComplex C;
    constexpr int SL = PCG_SLOT_LANES;
    const SysDev& S = dv.sys[0];
    double* sc = dv.scal;
    const int n = dv.nAtoms, nb = gridDim.x, tid = threadIdx.x, nT = blockDim.x;
    const int K0 = KC > 0 ? KC : S.K[0], K1 = KC > 0 ? KC : S.K[1], K2 = KC > 0 ? KC : S.K[2];
    const int x = blockIdx.x;
    const bool planeBlock = x < K0;
    unsigned* const gbar = dv.pcgBar;        // every block
    unsigned* const pbar = dv.pcgBar + 1;    // the plane blocks
    const int per = (n + nb - 1) / nb, s0 = min(n, x * per), ns = min(n, s0 + per) - s0;
    extern __shared__ __align__(16) unsigned char smraw[];
    C* W0 = (C*) smraw;
    C* W1 = W0 + FFT_MAXK;
    C* W2 = W1 + FFT_MAXK;
    C* const b0 = W2 + FFT_MAXK;
    C* const b1 = b0 + dv.fftgBuf;
    double* const sx = SHARED ? (double*) (b1 + dv.fftgBuf)   // the slots' x, r, p, A p (3 per slot), alpha
                              : (double*) (dv.pcgState + (size_t) x * pcgStateBytes(per));
    double* const sr = sx + 3 * per;
    double* const sp = sr + 3 * per;
    double* const sAp = sp + 3 * per;
    double* const sal = sAp + 3 * per;
    float* const spl = (float*) (sal + per);
    int* const satom = (int*) (spl + PCG_SPL * per);
    int* const sbase = satom + per;
    const C* tw = (const C*) dv.twiddle;
    if (planeBlock) {
        for (int m = tid; m < K0; m += nT)
            W0[m] = tw[S.twOff[0] + m];
        for (int m = tid; m < K1; m += nT)
            W1[m] = tw[S.twOff[1] + m];
        for (int m = tid; m < K2; m += nT)
            W2[m] = tw[S.twOff[2] + m];
    }
    for (int s = tid; s < ns; s += nT) {
        const int i = dv.slotAtom[s0 + s];
        satom[s] = i;
        sal[s] = dv.alpha[i];
        for (int k = 0; k < 3; k++)
            sbase[3 * s + k] = dv.pmeBase[3 * i + k];
    }
    for (int t = tid; t < ns * 6 * P; t += nT) {   // (the evaluation's coefficients, rows of MAXP)
        const int s = t / (6 * P), k = t - s * 6 * P;
        spl[s * PCG_SPL + k] = ((const float*) dv.spl)[(size_t) (s0 + s) * 9 * MAXP + (k / P) * MAXP + k % P];
    }
    __syncthreads();
    const PlaneFft<float, KC> fft(K0, K1, K2, b0, b1, W0, W1, W2);
    const int nline = fft.nline, l0 = x * fft.lpb, nl = min(nline, l0 + fft.lpb) - l0;
    C* const spec = (C*) dv.spec + S.specOff;
    const float* const infl = (const float*) dv.infl + S.specOff;
    long long* const gfix = dv.gridFix + S.gridOff;
    float* const gpot = (float*) dv.grid + S.gridOff;
    double* const Eslot = dv.Fpair;          // (the pair field in slot order; the final pass writes Fpair later)
    double* const partA = dv.pcgPartial;     // shares of three sums, and of the two around the next spread
    double* const partB = partA + 3 * nb;
    const int hrow = tid / SL, hl = tid % SL, rows = nT / SL;
    const unsigned hmask = groupMask<SL>();
    // the pair pass's rows: q for a plane block, planeSlots more for the others
    const int q = max(0, (n - (nb - K0) * planeSlots + nb - 1) / nb);
    const int rest = (max(0, n - K0 * q) + nb - K0 - 1) / (nb - K0);
    const int g0 = min(n, planeBlock ? x * q : K0 * q + (x - K0) * rest), g1 = min(n, g0 + (planeBlock ? q : rest));
    const size_t plane = (size_t) K1 * K2;
    const double cs = 4.0 * S.beta * S.beta * S.beta / (3.0 * SQRT_PI);
    const bool custom = dv.ctl->customRhs != 0;
    const int guess = dv.ctl->guess;

    // S: the vector v (3 per slot) as sources, with the charges in the final pass's
    auto spread = [&](const double* v, bool charges) {
        for (int s = hrow; s < ns; s += rows) {
            const double d0 = v[3 * s], d1 = v[3 * s + 1], d2 = v[3 * s + 2];
            const float qf = charges ? (float) dv.q[satom[s]] : 0.f;
            if (hl == 0)
                ((float4*) dv.dS)[s0 + s] = make_float4((float) d0, (float) d1, (float) d2, qf);
            const float e0 = (float) (S.K[0] * (d0 * S.recip[0] + d1 * S.recip[3] + d2 * S.recip[6])),
                        e1 = (float) (S.K[1] * (d0 * S.recip[1] + d1 * S.recip[4] + d2 * S.recip[7])),
                        e2 = (float) (S.K[2] * (d0 * S.recip[2] + d1 * S.recip[5] + d2 * S.recip[8]));
            const float* th = spl + s * PCG_SPL;
            const int bs0 = sbase[3 * s], bs1 = sbase[3 * s + 1], bs2 = sbase[3 * s + 2];
            int off[P];
#pragma unroll
            for (int j1 = 0; j1 < P; j1++)
                off[j1] = wrapIndex(bs0 - j1, K0) * (int) plane;
            for (int c = hl; c < P * P; c += SL) {
                const int j2 = c / P, j3 = c % P;
                const float t2 = th[P + j2], u2 = th[4 * P + j2], t3 = th[2 * P + j3], u3 = th[5 * P + j3];
                const float c23 = t2 * t3;
                const float a = qf * c23 + e1 * u2 * t3 + e2 * t2 * u3, b = e0 * c23;
                long long* col = gfix + wrapIndex(bs1 - j2, K1) * K2 + wrapIndex(bs2 - j3, K2);
#pragma unroll
                for (int j1 = 0; j1 < P; j1++)
                    gridFixAdd(col + off[j1], a * th[j1] + b * th[3 * P + j1]);
            }
        }
    };
    // F and G: T v = pair + reciprocal + self field; the rows of A v = v / alpha - T v (0 where not polarizable) in
    // sAp.  The caller's barrier came after the spread; false: a barrier gave up.
    auto apply = [&](const double* v) -> bool {
        if (planeBlock) {
            long long* const fxx = gfix + (size_t) x * plane;
            fft.forward(
                [&](int e) {
                    const long long w = __ldcg(fxx + e);
                    __stcg(fxx + e, 0ll);
                    return gridFixValue(w);
                },
                spec + (size_t) x * nline);
            if (!fftgBarrier(pbar, (unsigned) K0, dv.flags))
                return false;
            fft.lines(spec, l0, nl, [&](int m1, int l, C w) {
                const float gk = infl[(size_t) m1 * nline + l];
                w.x *= gk;
                w.y *= gk;
                return w;
            });
            if (!fftgBarrier(pbar, (unsigned) K0, dv.flags))
                return false;
            float* const gx = gpot + (size_t) x * plane;
            fft.inverse(spec + (size_t) x * nline, [&](int e, float w) { gx[e] = w; });
        }
        pcgPairField(dv, Eslot, g0, g1);
        if (!fftgBarrier(gbar, (unsigned) nb, dv.flags))
            return false;
        for (int s = hrow; s < ns; s += rows) {
            double eP = 0.0;
            if (hl < 3)
                eP = Eslot[3 * (size_t) (s0 + s) + hl];
            const float* th = spl + s * PCG_SPL;
            const int bs0 = sbase[3 * s], bs1 = sbase[3 * s + 1], bs2 = sbase[3 * s + 2];
            int off[P];
#pragma unroll
            for (int j1 = 0; j1 < P; j1++)
                off[j1] = wrapIndex(bs0 - j1, K0) * (int) plane;
            float f0 = 0.f, f1 = 0.f, f2 = 0.f;
#pragma unroll
            for (int c = hl; c < P * P; c += SL) {
                const int j2 = c / P, j3 = c % P;
                const float* col = gpot + wrapIndex(bs1 - j2, K1) * K2 + wrapIndex(bs2 - j3, K2);
                float St = 0.f, Su = 0.f;
#pragma unroll
                for (int j1 = 0; j1 < P; j1++) {
                    const float ph = col[off[j1]];
                    St += th[j1] * ph;
                    Su += th[3 * P + j1] * ph;
                }
                const float t2 = th[P + j2], u2 = th[4 * P + j2], t3 = th[2 * P + j3], u3 = th[5 * P + j3];
                f0 += Su * t2 * t3;
                f1 += St * u2 * t3;
                f2 += St * t2 * u3;
            }
            double F0 = f0, F1 = f1, F2 = f2;
#pragma unroll
            for (int o = SL / 2; o > 0; o >>= 1) {
                F0 += __shfl_xor_sync(hmask, F0, o, SL);
                F1 += __shfl_xor_sync(hmask, F1, o, SL);
                F2 += __shfl_xor_sync(hmask, F2, o, SL);
            }
            if (hl < 3) {
                const double E = -(S.K[0] * S.recip[3 * hl] * F0 + S.K[1] * S.recip[3 * hl + 1] * F1 +
                                   S.K[2] * S.recip[3 * hl + 2] * F2);
                const double al = sal[s], vk = v[3 * s + hl], T = eP + E + cs * vk;
                sAp[3 * s + hl] = (al > 0) ? vk / al - T : 0.0;
            }
        }
        __syncthreads();
        return true;
    };

    // b, x0 and the share of sum |alpha b|
    {
        const size_t hs = (size_t) 3 * dv.numGlobal;
        double v[1] = {0.0};
        for (int t = tid; t < 3 * ns; t += nT) {
            const int s = t / 3, k = t - 3 * s, i = satom[s];
            const int gi = dv.globalIndex ? dv.globalIndex[i] : i;
            const double al = sal[s];
            const double bk = custom ? dv.b[3 * i + k] : dv.Epair[3 * i + k] + dv.Erec[3 * i + k] + cs * dv.perm[3 * i + k];
            if (!custom)
                dv.b[3 * i + k] = bk;
            v[0] += fabs(al * bk);
            const double x0 = guess == 0 ? al * bk : historyGuess(dv, guess, (size_t) 3 * gi + k, hs);
            sx[t] = (guess >= 2 && !(al > 0)) ? 0.0 : x0;
            sr[t] = bk;
        }
        pcgShare<1>(v, 0u, partA, nb);   // (its barrier also publishes sx)
    }
    // The first round forms r = b - A x0 (from the zero guess r = b, without a pass), every later one is an iteration.
    // (One call of spread and of apply in the code: a second would put what they capture into local memory.)
    double norm = 0.0, rz = 0.0, err = 0.0, it = 0.0;
    for (bool first = true, last = false;; first = false) {
        if (!first || guess != 1) {
            const double* const src = last ? sAp : first ? sx : sp;
            spread(src, last);
            if (last)
                break;
            if (!fftgBarrier(gbar, (unsigned) nb, dv.flags))
                return;
            if (!first) {   // r.z, and the convergence test on max |z|: they went around with this barrier
                double tot[2];
                if (it == 0.0) {
                    pcgTotals<1>(partA, nb, 0u, tot);
                    norm = tot[0] / (3.0 * n) + 1e-300;
                }
                pcgTotals<2>(partB, nb, 2u, tot);
                rz = tot[0];
                err = tot[1] / norm;
                if (!(err > dv.tol && it < dv.maxIter)) {
                    if (planeBlock)   // the dropped direction's spread
                        for (int e = tid; e < (int) plane; e += nT)
                            __stcg(gfix + (size_t) x * plane + e, 0ll);
                    if (!finish)
                        break;
                    const int histSlot = dv.ctl->histSlot;
                    for (int s = tid; s < ns; s += nT) {   // (as k_final_prep)
                        const int i = satom[s], gi = dv.globalIndex ? dv.globalIndex[i] : i;
                        const double al = sal[s], qi = dv.q[i];
                        double m2 = 0.0, d2 = 0.0;
                        for (int k = 0; k < 3; k++) {
                            const double m = sx[3 * s + k] + dv.peek * al * sr[3 * s + k];
                            const double d = dv.perm[3 * i + k] + m;
                            dv.mu[3 * i + k] = m;
                            dv.dtot[3 * i + k] = d;
                            sAp[3 * s + k] = d;
                            m2 += m * m;
                            d2 += d * d;
                            if (histSlot >= 0)
                                dv.hist[(size_t) histSlot * 3 * dv.numGlobal + 3 * gi + k] = m;
                        }
                        dv.fin[(size_t) i * NFIN + 1] = -(S.beta / SQRT_PI) * qi * qi - 0.5 * cs * d2;
                        dv.fin[(size_t) i * NFIN + 2] = (al > 0) ? m2 / (2.0 * al) : 0.0;
                    }
                    if (!fftgBarrier(gbar, (unsigned) nb, dv.flags))   // (the planes are clear)
                        return;
                    last = true;
                    continue;
                }
            }
            if (!apply(src))
                return;
        }
        double w[2] = {0.0, 0.0};
        if (first) {   // r = b - A x0 (rows of polarizable atoms); the first direction is z
            for (int t = tid; t < 3 * ns; t += nT) {
                const double al = sal[t / 3];
                const double rk = (al > 0) ? (guess != 1 ? sr[t] - sAp[t] : sr[t]) : 0.0, zk = al * rk;
                sr[t] = rk;
                sp[t] = zk;
                w[0] += rk * zk;
                w[1] = fmax(w[1], fabs(zk));
            }
        } else {
            double v[3] = {0.0, 0.0, 0.0};
            for (int t = tid; t < 3 * ns; t += nT) {
                const double al = sal[t / 3], a = sAp[t], za = al * a;
                v[0] += sp[t] * a;
                v[1] += sr[t] * za;
                v[2] += a * za;
            }
            pcgShare<3>(v, 0u, partA, nb);
            if (!fftgBarrier(gbar, (unsigned) nb, dv.flags))
                return;
            double tot[3];
            pcgTotals<3>(partA, nb, 0u, tot);
            const double alph = rz / fmax(tot[0], 1e-300);
            const double beta = -alph * (tot[1] - alph * tot[2]) / fmax(rz, 1e-300);
            it += 1.0;
            for (int t = tid; t < 3 * ns; t += nT) {
                const double pk = sp[t], rn = sr[t] - alph * sAp[t], zn = sal[t / 3] * rn;
                sx[t] += alph * pk;
                sr[t] = rn;
                sp[t] = zn + beta * pk;
                w[0] += rn * zn;
                w[1] = fmax(w[1], fabs(zn));
            }
        }
        pcgShare<2>(w, 2u, partB, nb);
    }
    for (int t = tid; t < 3 * ns; t += nT) {
        const int i = satom[t / 3], k = t % 3;
        dv.x[3 * i + k] = sx[t];
        dv.r[3 * i + k] = sr[t];
    }
    if (x == 0 && tid == 0) {
        sc[SC_NORM] = norm;
        sc[SC_RZ] = rz;
        sc[SC_ERR] = err;
        sc[SC_IT] = it;
        sc[SC_DONE] = 1.0;
        atomicAdd(&dv.flags[2], 1);
    }
}

}  // namespace pgmb200
