// FP32 3-D r2c of the GW sources for lattices whose planes fit on chip (N a
// multiple of 16 up to 160), fused with the TT projection and h/l update: two
// passes over HBM instead of the three of fftt.cuh.
//
// The reference transforms each source array with one 3-D r2c FFT
// (fft_stresstensor, g2evolutionpert.cpp:183-195) and then updates h and l
// per k-point (evolve_perts, :343-455).
//
//   plane pass  (plane_kernel)  S[q][i][j][k] -> T[q][i][x], in place
//       rows along k (two real rows as one complex sequence), then columns
//       along j of a whole (j, k) plane in shared memory, both as four-step
//       FFTs N = L1 L2; the plane's half spectrum has the flat index
//       x = ky (N/2+1) + kz and takes the N (N + 2) reals that the plane's
//       N rows of N begin (SRC_PLANES);
//   lines pass  (lines_kernel)  T, G[p][x / 8][kx][x % 8]
//       takes the lines along i of eight neighbouring x (64-byte pieces) of
//       the ten arrays: it transforms the 80 lines, and each k-point's update
//       (kspace_update_vals) reads its ten sources from shared memory; only
//       the amplitudes return to HBM, as contiguous runs.
// The first step of each transform reads its points straight from global
// memory into registers, so shared memory holds one work buffer per CTA and
// several CTAs share an SM.
//
// The amplitudes are kept in the order of the lines pass (g_index, gt = 2)
// for the life of the handle.  q runs over the ten source arrays of each
// lattice; forward sign e^{-i}, unnormalised, times 2 (the row pairs are
// separated without their factor 1/2, which kspace_apply's source
// coefficients take in, an exact power of two).
//
// The plane pass is bound by the load/store unit's data path (ncu at 128^3:
// 53 % of its wavefronts over the whole launch, issue 28 %, HBM 14 %: the
// sources come from the L2), so the work layout is chosen for conflict-free
// accesses (place) and the pass writes its planes as they lie; the lines pass
// by the latency of its loads behind three barriers (two CTAs of 82 KB per SM
// at 128^3).
// Measured on B200, GW transforms + k-space update of one step: 96^3 53 us
// against 107 for cuFFT's plan and the separate pass, 128^3 110 against 148
// (116 for the three passes of fftt.cuh), 160^3 240 against 339; the
// ensemble of 256 lattices of 32^3 .. 128^3 580 ms per 50 steps against 922.
// Planes landed by one bulk copy, with the first row step reading them from
// shared memory, ran the same (75.6 us of planes at 128^3 against 73.5);
// planes written as 64-byte pieces in the lines pass's order 73.5 against
// 69.5; two row tasks' loads in flight per thread of the lines pass spilled
// (58 us against 45).
#pragma once

#include "dft.cuh"
#include "kspace.cuh"
#include "stencil.cuh"

namespace gabe {
namespace f2p {

// Per size: the four-step split, planes per tile, threads and CTAs per SM of
// the plane pass (TP covers one task per thread in its first phase) and of
// the lines pass.
template <int N>
struct Cfg;
#define GABE_F2P_CFG(n, l1, l2, pb, tp, mbp, tl, mbl)                                           \
    template <>                                                                                 \
    struct Cfg<n> {                                                                             \
        static constexpr int L1 = l1, L2 = l2, PB = pb, TP = tp, MBP = mbp, TL = tl, MBL = mbl; \
    };
GABE_F2P_CFG(16, 4, 4, 4, 160, 5, 128, 4)
GABE_F2P_CFG(32, 8, 4, 2, 160, 5, 256, 3)
GABE_F2P_CFG(48, 8, 6, 1, 160, 5, 192, 4)
GABE_F2P_CFG(64, 8, 8, 1, 160, 5, 256, 3)
GABE_F2P_CFG(80, 10, 8, 1, 224, 4, 320, 2)
GABE_F2P_CFG(96, 12, 8, 1, 224, 4, 256, 2)
GABE_F2P_CFG(112, 14, 8, 1, 256, 3, 320, 2)
GABE_F2P_CFG(128, 16, 8, 1, 288, 3, 320, 2)
GABE_F2P_CFG(144, 12, 12, 1, 224, 2, 288, 2)
GABE_F2P_CFG(160, 16, 10, 1, 416, 2, 320, 2)
#undef GABE_F2P_CFG

constexpr int kX = 8;  // x per tile of the lines pass: 64-byte pieces

// W_N^(n1 k2), stored [k2][n1], correctly rounded at compile time.
template <int N>
struct Roots {
    float2 w[N];
    constexpr Roots() : w{} {
        for (int m = 0; m < N; m++) {
            const int a = (m % Cfg<N>::L1) * (m / Cfg<N>::L1);
            w[m].x = (float)dft::cos_turn(a, N);
            w[m].y = (float)-dft::sin_turn(a, N);
        }
    }
};
template <int N>
static __device__ const Roots<N> kRoots = Roots<N>();

template <int N>
__device__ __forceinline__ void twiddles(float2 *tw) {
    for (int m = threadIdx.x; m < N; m += blockDim.x) tw[m] = kRoots<N>.w[m];
}

template <int N>
struct PlaneGeom {
    using C = Cfg<N>;
    static constexpr int NH = N / 2 + 1, RP = N, PR = N + 4;  // row pitch as stored, and in the work layout
    static constexpr int ROWS = C::PB * N, PAIRS = ROWS / 2;
    static constexpr size_t SMEM_BYTES = N * sizeof(float2) + (size_t)ROWS * PR * sizeof(float);
    static_assert(N % 16 == 0 && C::L1 * C::L2 == N && C::L1 % 2 == 0 && C::L2 % 2 == 0, "four-step split");
    static_assert(N % C::PB == 0, "a tile's planes belong to one source array");
};

// Work layout of a row pair (2p, 2p+1): pitch PR (pairs 8 banks apart), the
// real parts of the pair's complex sequence in row 2p, the imaginary parts in
// row 2p+1.  After the rows phase, column kz of the half spectrum of row j
// lives at (j, kz) and (j, im_at(kz)): the pair's Z[kz] and Z[N-kz] hold
// exactly the two rows' values, and the two padding columns take the
// imaginary parts that kz = 0 and kz = N/2 gain along j.
template <int N>
__device__ __forceinline__ int im_at(int kz) {
    return kz == 0 ? N : (kz == N / 2 ? N + 1 : N - kz);
}
// Place of element e of a row.  With L2 = 8 the chunks of eight elements are
// permuted in pairs and their halves swapped, so that the first step's
// 16-byte stores of neighbouring n1 (16 elements apart) fall on distinct
// banks; lanes over consecutive elements stay conflict-free.
template <int N>
__device__ __forceinline__ int place(int e) {
    if constexpr (Cfg<N>::L2 != 8) return e;
    if (e >= N) return e;
    const int c = e >> 3;
    return 8 * (c ^ ((c >> 3) & 1)) + ((e & 7) ^ (c & 4));
}

template <int N>
__global__ void __launch_bounds__(Cfg<N>::TP, Cfg<N>::MBP)
    plane_kernel(float *S, int ntiles) {
    using G = PlaneGeom<N>;
    using C = Cfg<N>;
    constexpr int L1 = C::L1, L2 = C::L2, NH = G::NH, RP = G::RP, PR = G::PR, TP = C::TP, PB = C::PB;
    constexpr int PP = N * (N + 2);  // reals from plane to plane
    extern __shared__ __align__(128) unsigned char sm[];
    float2 *tw = reinterpret_cast<float2 *>(sm);
    float *W = reinterpret_cast<float *>(sm + N * sizeof(float2));
    const int tid = threadIdx.x;
    twiddles<N>(tw);
    __syncthreads();
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        // rows, first step: L2-point DFTs over n2 (stride L1) of two neighbouring n1, twiddled,
        // from global memory to element k2 + L2 n1 of the work layout
        float *src = S + (size_t)tile * (PB * PP);
        for (int t = tid; t < G::PAIRS * (L1 / 2); t += TP) {
            const int p = t / (L1 / 2), n1 = 2 * (t % (L1 / 2));
            const float *re = src + (2 * p / N) * PP + (2 * p % N) * RP + n1, *im = re + RP;
            float2 xa[L2], xb[L2];
#pragma unroll
            for (int n2 = 0; n2 < L2; n2++) {
                const float2 a = __ldcs(reinterpret_cast<const float2 *>(re + L1 * n2));
                const float2 b = __ldcs(reinterpret_cast<const float2 *>(im + L1 * n2));
                xa[n2] = make_float2(a.x, b.x);
                xb[n2] = make_float2(a.y, b.y);
            }
            // one column of the row pair after the other: half the live registers
            auto put = [&](float2 (&x)[L2], int n) {
                dft::points<L2>(x);
#pragma unroll
                for (int k2 = 1; k2 < L2; k2++) x[k2] = dft::cmul(x[k2], tw[k2 * L1 + n]);
                float *wr = W + 2 * p * PR, *wi = wr + PR;
                if constexpr (L2 % 4 == 0) {
#pragma unroll
                    for (int u = 0; u < L2; u += 4) {
                        const int e = place<N>(L2 * n + u);
                        *reinterpret_cast<float4 *>(wr + e) = make_float4(x[u].x, x[u + 1].x, x[u + 2].x, x[u + 3].x);
                        *reinterpret_cast<float4 *>(wi + e) = make_float4(x[u].y, x[u + 1].y, x[u + 2].y, x[u + 3].y);
                    }
                } else {
#pragma unroll
                    for (int u = 0; u < L2; u += 2) {
                        const int e = L2 * n + u;
                        *reinterpret_cast<float2 *>(wr + e) = make_float2(x[u].x, x[u + 1].x);
                        *reinterpret_cast<float2 *>(wi + e) = make_float2(x[u].y, x[u + 1].y);
                    }
                }
            };
            put(xa, n1);
            put(xb, n1 + 1);
        }
        __syncthreads();
        // rows, second step, in place: element k2 + L2 n1 becomes Z[k2 + L2 k1]
        for (int t = tid; t < G::PAIRS * L2; t += TP) {
            const int p = t / L2, k2 = t % L2;
            float *re = W + 2 * p * PR, *im = re + PR;
            float2 y[L1];
#pragma unroll
            for (int n = 0; n < L1; n++) {
                const int e = place<N>(L2 * n + k2);
                y[n] = make_float2(re[e], im[e]);
            }
            dft::points<L1>(y);
#pragma unroll
            for (int n = 0; n < L1; n++) {
                const int e = place<N>(L2 * n + k2);
                re[e] = y[n].x;
                im[e] = y[n].y;
            }
        }
        __syncthreads();
        // columns, first step: separates rows (2p, 2p+1) (times 2), L2-point DFTs over j = n1 + L1 n2, in place
        for (int t = tid; t < PB * NH * (L1 / 2); t += TP) {
            const int kz = t % NH, m = t / NH, n1 = 2 * (m % (L1 / 2)), b = m / (L1 / 2);
            const int kr = place<N>(kz), rd = place<N>(kz ? N - kz : 0), wr = place<N>(im_at<N>(kz));
            float *row = W + (b * N + n1) * PR;
            float2 xa[L2], xb[L2];
#pragma unroll
            for (int n2 = 0; n2 < L2; n2++) {
                const float *r = row + L1 * n2 * PR;
                const float zr = r[kr], zi = r[PR + kr], mr = r[rd], mi = r[PR + rd];
                xa[n2] = make_float2(zr + mr, zi - mi);
                xb[n2] = make_float2(zi + mi, mr - zr);
            }
            auto put = [&](float2 (&x)[L2], int n, float *r) {
                dft::points<L2>(x);
#pragma unroll
                for (int k2 = 0; k2 < L2; k2++, r += L1 * PR) {
                    const float2 y = k2 ? dft::cmul(x[k2], tw[k2 * L1 + n]) : x[k2];
                    r[kr] = y.x;
                    r[wr] = y.y;
                }
            };
            put(xa, n1, row);
            put(xb, n1 + 1, row + PR);
        }
        __syncthreads();
        // columns, second step, over the planes: ky = k2 + L2 k1, x = ky NH + kz
        {
            float2 *To = reinterpret_cast<float2 *>(src);  // every read of the tile's rows lies behind three barriers
            for (int t = tid; t < PB * NH * L2; t += TP) {
                const int kz = t % NH, m = t / NH, k2 = m % L2, b = m / L2;
                const int re = place<N>(kz), im = place<N>(im_at<N>(kz));
                const float *row = W + (b * N + L1 * k2) * PR;
                float2 y[L1];
#pragma unroll
                for (int n = 0; n < L1; n++) y[n] = make_float2(row[n * PR + re], row[n * PR + im]);
                dft::points<L1>(y);
#pragma unroll
                for (int k1 = 0; k1 < L1; k1++) To[(b * N + k2 + L2 * k1) * NH + kz] = y[k1];
            }
        }
        __syncthreads();  // W is free
    }
}

// ---------------------------------------------------------------------------
// lines along i + TT projection and both RK2 stages of h, l
// ---------------------------------------------------------------------------
struct LineArgs {
    const float2 *T;      // [lattices][10][N][x]
    float2 *G;            // [lattices][4][x / 8][N][8]
    const DevScalars *sc; // scalars of lattice l: sc[ids ? ids[l] : l]
    const int *ids;
    LatticeConsts c;
    int slot, nlat;
};

template <int N>
struct LineGeom {
    using C = Cfg<N>;
    static constexpr int NH = N / 2 + 1, XT = N * NH / kX, NQ = 2 * kSrc;
    static constexpr int QS = N * kX + kX;  // complex values between two arrays: odd multiple of 64 bytes
    static constexpr size_t HEAD = 128;  // coefficients
    static constexpr size_t SMEM_BYTES = HEAD + N * sizeof(float2) + (size_t)NQ * QS * sizeof(float2);
    static_assert(N * NH % kX == 0 && sizeof(KsCoef<float>) <= HEAD, "tiles of eight x");
};

template <int N>
__global__ void __launch_bounds__(Cfg<N>::TL, Cfg<N>::MBL) lines_kernel(LineArgs a) {
    using G = LineGeom<N>;
    using C = Cfg<N>;
    constexpr int L1 = C::L1, L2 = C::L2, NH = G::NH, XT = G::XT, NQ = G::NQ, QS = G::QS, T = C::TL;
    constexpr int KP = (N * kX + T - 1) / T;  // k-points per thread
    constexpr size_t M = (size_t)N * N * NH;
    extern __shared__ __align__(128) unsigned char sm[];
    KsCoef<float> *kcs = reinterpret_cast<KsCoef<float> *>(sm);
    float2 *tw = reinterpret_cast<float2 *>(sm + G::HEAD);
    float2 *B = tw + N;
    const int tid = threadIdx.x;
    twiddles<N>(tw);
    __syncthreads();
    const int ntiles = a.nlat * XT;
    int have = -1;
    for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
        const int lat = tile / XT, xt = tile % XT;
        if (tid == 0 && lat != have) {  // the loop's last barrier ended every use of the last lattice's
            KsCoef<float> kc = ks_coef<float>(a.c, a.sc[a.ids ? a.ids[lat] : lat].gw[a.slot]);
            kc.src0 *= 0.5f;  // the transforms carry a factor 2
            kc.src1 *= 0.5f;
            *kcs = kc;
        }
        have = lat;
        // first step, from global memory to element k2 + L2 n1: lanes over the eight x and neighbouring n1
        const float2 *src = a.T + (size_t)lat * NQ * M + xt * kX;
        for (int t = tid; t < NQ * kX * L1; t += T) {
            const int r = t % kX, n1 = (t / kX) % L1, q = t / (kX * L1);
            const float2 *ln = src + q * M + n1 * (N * NH) + r;
            float2 x[L2];
#pragma unroll
            for (int n = 0; n < L2; n++) x[n] = __ldcs(ln + L1 * n * (N * NH));
            dft::points<L2>(x);
            float2 *o = B + q * QS + L2 * n1 * kX + r;
#pragma unroll
            for (int k = 0; k < L2; k++) o[k * kX] = k ? dft::cmul(x[k], tw[k * L1 + n1]) : x[k];
        }
        __syncthreads();
        // second step in place, natural order: lanes over the eight x and neighbouring arrays
        for (int t = tid; t < NQ * kX * L2; t += T) {
            const int r = t % kX, q = (t / kX) % NQ, k2 = t / (kX * NQ);
            float2 *ln = B + q * QS + k2 * kX + r;
            float2 y[L1];
#pragma unroll
            for (int n = 0; n < L1; n++) y[n] = ln[L2 * n * kX];
            dft::points<L1>(y);
#pragma unroll
            for (int n = 0; n < L1; n++) ln[L2 * n * kX] = y[n];
        }
        // the amplitudes of this thread's k-points arrive while the others finish
        float2 *gl = a.G + (size_t)lat * 4 * M + (size_t)xt * (N * kX);
        float2 gv[KP][4];
#pragma unroll
        for (int u = 0; u < KP; u++) {
            const int t = tid + u * T;
#pragma unroll
            for (int p = 0; p < 4; p++) gv[u][p] = t < N * kX ? __ldcs(gl + p * M + t) : make_float2(0.f, 0.f);
        }
        __syncthreads();
        const KsCoef<float> kc = *kcs;
#pragma unroll
        for (int u = 0; u < KP; u++) {
            const int t = tid + u * T;
            if (t >= N * kX) break;
            const int kx = t / kX, x = xt * kX + t % kX, ky = x / NH, kz = x % NH;
            Cplx<float> s[10], g[4];
#pragma unroll
            for (int p = 0; p < 4; p++) g[p] = {gv[u][p].x, gv[u][p].y};
#pragma unroll
            for (int q = 0; q < NQ; q++) {
                const float2 v = B[q * QS + t];
                s[q] = {v.x, v.y};
            }
            kspace_update_vals<float, POL_RATIONAL>(kc, kx <= N / 2 ? kx : kx - N, ky <= N / 2 ? ky : ky - N, kz, s, g);
#pragma unroll
            for (int p = 0; p < 4; p++) __stcs(gl + p * M + t, make_float2(g[p].re, g[p].im));
        }
        __syncthreads();  // B is free
    }
}

}  // namespace f2p
}  // namespace gabe
