// Spectra emulator: MLP forward, backward and AdamW as hand-written kernels
// (include/gabe_mlp.h).  No counterpart in the reference.
//
// One tiled GEMM kernel serves the three products of every layer
// (activations X [B][K], weights W [K][N], pre-activations Z [B][N]):
//
//   forward       Z  = X W + b          M=B, N=N, K=K      epilogue: bias, SiLU, store Z and H
//   data grad     dX = (dZ W^T) * SiLU'(Z_prev)            M=B, N=K, K=N
//   weight grad   dW = X^T dZ                              M=K, N=N, K=B
//
// Operands are addressed through (row, column) strides, so transposes cost
// nothing but coalescing.  64x64 output tiles, 16-deep k slices in shared
// memory, 4x4 outputs per thread, FP32 FMA accumulation.  Activations are
// read as BF16 (or FP32) and widened on the way into shared memory; weights
// are FP32.  With BF16 activations the forward of every layer after the
// first runs on tensor cores instead (tc::gemm_tc_kernel, BF16 weight
// copies); the first layer (a handful of inputs) and the backward products
// stay on this kernel.
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <cmath>
#include <cstdint>
#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <vector>

#include "../../include/gabe.h"
#include "../../include/gabe_mlp.h"
#include "umma.cuh"

namespace {

using bf16 = __nv_bfloat16;

template <typename T>
__device__ __forceinline__ float ldf(const T *p, long long i);
template <>
__device__ __forceinline__ float ldf<float>(const float *p, long long i) { return p[i]; }
template <>
__device__ __forceinline__ float ldf<bf16>(const bf16 *p, long long i) { return __bfloat162float(p[i]); }

template <typename T>
__device__ __forceinline__ T cvt(float v);
template <>
__device__ __forceinline__ float cvt<float>(float v) { return v; }
template <>
__device__ __forceinline__ bf16 cvt<bf16>(float v) { return __float2bfloat16_rn(v); }

__device__ __forceinline__ float sigmoid(float z) { return 1.f / (1.f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigmoid(z); }
// SiLU of the forward epilogues of the first-layer and tcgen05 kernels, from
// the identity exp(-z) = 2^(-z log2 e): z / (1 + 2^(-z log2 e)) on the
// special-function unit's base-2 exponential and reciprocal (PTX ex2.approx
// and rcp.approx, relative errors of at most 2^-22 and 2^-23), since expf and
// an IEEE division bounded those epilogues (608 against 185 us per 1M-row
// hidden layer).  Relative error at most 1.5 |z| 2^-24 (the rounded exponent)
// + 2^-21, far below the BF16 rounding of the stored activations; a value
// below |z| 2^-126 (z < -87) may be flushed to zero.  A reciprocal by
// Newton-Raphson steps on the FMA pipe instead of the second special-function
// operation measured slower (225 us): the epilogue is bound by issue as much
// as by that pipe.
__device__ __forceinline__ float silu_fast(float z) {
    float e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(1.f + e));
    return z * r;
}
__device__ __forceinline__ float dsilu(float z) {
    const float s = sigmoid(z);
    return s * (1.f + z * (1.f - s));
}

enum Epi { EPI_HIDDEN = 0, EPI_OUT = 1, EPI_BWD_DATA = 2, EPI_BWD_WEIGHT = 3 };

struct GemmArgs {
    int M, N, K;
    const void *A;
    long long sam, sak;  // A(m, k) = A[m * sam + k * sak]
    const float *B;
    long long sbk, sbn;  // B(k, n) = B[k * sbk + n * sbn]
    const float *bias;   // EPI_HIDDEN, EPI_OUT
    void *Z;             // EPI_HIDDEN: pre-activation out (may be null); EPI_BWD_DATA: pre-activation in
    void *C;             // H (activation type), Y, dX or dW (FP32)
    long long ldc;
    int kchunk;          // EPI_BWD_WEIGHT: k range of split blockIdx.z (a multiple of BK)
    float *dbp;          // EPI_BWD_WEIGHT: column sums of B per split ([splits][N])
};

constexpr int BM = 64, BN = 64, BK = 16, kThreads = 256;

// TA: type of A; TACT: activation storage type (Z/H of the epilogues).
// Tile (bx, by) of the output, split bz of k (EPI_BWD_WEIGHT).
template <typename TA, typename TACT, int EPI>
__device__ __forceinline__ void gemm_tile(const GemmArgs &g, int bx, int by, int bz) {
    __shared__ __align__(16) float As[BK][BM];
    __shared__ __align__(16) float Bs[BK][BN];
    const int tid = threadIdx.x, tx = tid % 16, ty = tid / 16;
    const int m0 = by * BM, n0 = bx * BN;
    const TA *A = static_cast<const TA *>(g.A);
    float acc[4][4] = {};
    // split-K (weight gradient): this block sums k in [kb, ke) and writes
    // its partial product to slice bz of the output
    const int kb = EPI == EPI_BWD_WEIGHT ? bz * g.kchunk : 0;
    const int ke = EPI == EPI_BWD_WEIGHT ? min(g.K, kb + g.kchunk) : g.K;
    float csum = 0.f;  // EPI_BWD_WEIGHT, first row of tiles: column sums of B (the bias gradient)
    for (int k0 = kb; k0 < ke; k0 += BK) {
        // A tile: 64 (m) x 16 (k); each thread 4 elements along the
        // operand's contiguous direction
        if (g.sak == 1) {
            const int m = tid / 4, kk = (tid % 4) * 4;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int gm = m0 + m, gk = k0 + kk + q;
                As[kk + q][m] = (gm < g.M && gk < ke) ? ldf(A, gm * g.sam + gk) : 0.f;
            }
        } else {
            const int kk = tid / 16, m = (tid % 16) * 4;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int gm = m0 + m + q, gk = k0 + kk;
                As[kk][m + q] = (gm < g.M && gk < ke) ? ldf(A, gm * g.sam + gk * g.sak) : 0.f;
            }
        }
        // B tile: 16 (k) x 64 (n)
        if (g.sbn == 1) {
            const int kk = tid / 16, n = (tid % 16) * 4;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int gk = k0 + kk, gn = n0 + n + q;
                Bs[kk][n + q] = (gk < ke && gn < g.N) ? g.B[gk * g.sbk + gn] : 0.f;
            }
        } else {
            const int n = tid / 4, kk = (tid % 4) * 4;
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int gk = k0 + kk + q, gn = n0 + n;
                Bs[kk + q][n] = (gk < ke && gn < g.N) ? g.B[gk + gn * g.sbn] : 0.f;
            }
        }
        __syncthreads();
        if (EPI == EPI_BWD_WEIGHT && by == 0 && tid < BN) {
#pragma unroll
            for (int kk = 0; kk < BK; kk++) csum += Bs[kk][tid];
        }
#pragma unroll
        for (int kk = 0; kk < BK; kk++) {
            const float4 a = *reinterpret_cast<const float4 *>(&As[kk][ty * 4]);
            const float4 b = *reinterpret_cast<const float4 *>(&Bs[kk][tx * 4]);
            const float av[4] = {a.x, a.y, a.z, a.w}, bv[4] = {b.x, b.y, b.z, b.w};
#pragma unroll
            for (int i = 0; i < 4; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
        }
        __syncthreads();
    }
    if (EPI == EPI_BWD_WEIGHT && by == 0 && tid < BN && n0 + tid < g.N)
        g.dbp[(long long)bz * g.N + n0 + tid] = csum;
    float *Cz = static_cast<float *>(g.C) + (EPI == EPI_BWD_WEIGHT ? (long long)bz * g.M * g.ldc : 0);
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const int m = m0 + ty * 4 + i;
        if (m >= g.M) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int n = n0 + tx * 4 + j;
            if (n >= g.N) continue;
            const long long o = (long long)m * g.ldc + n;
            const float v = acc[i][j];
            if (EPI == EPI_HIDDEN) {
                const float z = v + g.bias[n];
                if (g.Z) static_cast<TACT *>(g.Z)[o] = cvt<TACT>(z);
                static_cast<TACT *>(g.C)[o] = cvt<TACT>(silu(z));
            } else if (EPI == EPI_OUT) {
                static_cast<float *>(g.C)[o] = v + g.bias[n];
            } else if (EPI == EPI_BWD_DATA) {
                static_cast<float *>(g.C)[o] = v * dsilu(ldf(static_cast<const TACT *>(g.Z), o));
            } else {
                Cz[o] = v;
            }
        }
    }
}

template <typename TA, typename TACT, int EPI>
__global__ void __launch_bounds__(kThreads) gemm_kernel(GemmArgs g) {
    gemm_tile<TA, TACT, EPI>(g, blockIdx.x, blockIdx.y, blockIdx.z);
}

// Weight gradients of every layer in one launch (batches of at most
// kSmallRows): block b takes tile and split b - first[l] of layer l.
constexpr int kMaxGradLayers = 17;
struct WeightGradArgs {
    int nl, first[kMaxGradLayers + 1];
    GemmArgs g[kMaxGradLayers];
};
template <typename TACT>
__global__ void __launch_bounds__(kThreads) weight_grad_kernel(const __grid_constant__ WeightGradArgs a) {
    int l = 0;
    while (l + 1 < a.nl && (int)blockIdx.x >= a.first[l + 1]) l++;
    const GemmArgs &g = a.g[l];
    const int b = blockIdx.x - a.first[l], nx = (g.N + BN - 1) / BN, ny = (g.M + BM - 1) / BM;
    const int bx = b % nx, by = (b / nx) % ny, bz = b / (nx * ny);
    if (l == 0) gemm_tile<float, TACT, EPI_BWD_WEIGHT>(g, bx, by, bz);
    else gemm_tile<TACT, TACT, EPI_BWD_WEIGHT>(g, bx, by, bz);
}

// Data gradient of a small batch: C[m][n] = (sum_k A[m][k] W[n][k])
// SiLU'(Z[m][n]), both operands contiguous along k.  32 x 32 outputs per
// block (four per thread), so that a 512 x 256 product makes 128 blocks
// instead of the tiled kernel's 32 of 64 x 64, whose 16 latency-bound k slices
// took 28 us; here the operands of 128 k at a time land by cp.async, one slice
// ahead.  Every output sums its k in order on one FP32 accumulator, as the
// tiled kernel does: the same bits.  Needs K % 4 == 0.
constexpr int kDgT = 256, kDgTile = 32, kDgK = 128, kDgPitch = kDgK + 4;
constexpr size_t kDgSmem = (size_t)2 * 2 * kDgTile * kDgPitch * sizeof(float);
template <typename TACT>
__global__ void __launch_bounds__(kDgT) data_grad_kernel(const float *A, const float *W, const TACT *Z, float *C, int M,
                                                         int N, int K) {
    extern __shared__ __align__(16) float dg[];  // [2 stages][A, W][32][pitch]
    const int tid = threadIdx.x, m0 = blockIdx.y * kDgTile, n0 = blockIdx.x * kDgTile;
    auto stage = [&](int st, int op) { return dg + (st * 2 + op) * kDgTile * kDgPitch; };
    auto load = [&](int st, int k0) {
        for (int t = tid; t < 2 * kDgTile * (kDgK / 4); t += kDgT) {
            const int op = t / (kDgTile * (kDgK / 4)), r = (t / (kDgK / 4)) % kDgTile, c = 4 * (t % (kDgK / 4));
            const int row = (op ? n0 : m0) + r, k = k0 + c;
            float *dst = stage(st, op) + r * kDgPitch + c;
            if (row < (op ? N : M) && k < K) {
                const float *src = (op ? W : A) + (long long)row * K + k;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)),
                             "l"(src)
                             : "memory");
            } else {
                *reinterpret_cast<float4 *>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    const int tx = tid % 16, ty = tid / 16;  // rows ty, ty + 16; columns tx, tx + 16
    float acc[2][2] = {};
    load(0, 0);
    for (int k0 = 0, st = 0; k0 < K; k0 += kDgK, st ^= 1) {
        if (k0 + kDgK < K) {
            load(st ^ 1, k0 + kDgK);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const float *a = stage(st, 0) + ty * kDgPitch, *w = stage(st, 1) + tx * kDgPitch;
        const int kn = min(kDgK, K - k0);
#pragma unroll 8
        for (int k = 0; k < kn; k += 4) {
            float4 av[2], wv[2];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                av[i] = *reinterpret_cast<const float4 *>(a + i * 16 * kDgPitch + k);
                wv[i] = *reinterpret_cast<const float4 *>(w + i * 16 * kDgPitch + k);
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int j = 0; j < 2; j++) {
                    acc[i][j] = fmaf(av[i].x, wv[j].x, acc[i][j]);
                    acc[i][j] = fmaf(av[i].y, wv[j].y, acc[i][j]);
                    acc[i][j] = fmaf(av[i].z, wv[j].z, acc[i][j]);
                    acc[i][j] = fmaf(av[i].w, wv[j].w, acc[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
            const int m = m0 + ty + 16 * i, n = n0 + tx + 16 * j;
            if (m >= M || n >= N) continue;
            const long long o = (long long)m * N + n;
            C[o] = acc[i][j] * dsilu(ldf(Z, o));
        }
}

// Forward of the first layer (NIN <= 8 inputs): z = x W0 + b0, h = SiLU(z),
// the sum over k in order as the tiled kernel forms it.  A row is made by
// G = N / 8 consecutive threads (G divides the block), 8 consecutive
// outputs each, so every store is a whole 16-byte (BF16) or 32-byte (FP32)
// piece of a coalesced row.  Each thread keeps its 8 columns of W0 and b0
// in registers for all its rows (a reload per row held the loads' queue
// full) and makes RPT rows per pass, their inputs loaded together, so that
// RPT loads are in flight instead of one (one row per pass left the kernel
// bound by the inputs' load latency).
constexpr int kFirstMaxIn = 8, kFirstRows = 4;

template <typename TACT, int NIN>
__global__ void __launch_bounds__(256) first_layer_kernel(const float *x, int rows, const float *W, const float *b,
                                                          int N, TACT *H, TACT *Z) {
    constexpr int RPT = kFirstRows;
    const int G = N / 8, rpb = 256 / G;  // threads per row, rows per block pass
    const int n0 = (threadIdx.x % G) * 8;
    float w[NIN][8], bias[8];
#pragma unroll
    for (int k = 0; k < NIN; k++)
#pragma unroll
        for (int j = 0; j < 8; j++) w[k][j] = W[(long long)k * N + n0 + j];
#pragma unroll
    for (int j = 0; j < 8; j++) bias[j] = b[n0 + j];
    const long long stride = (long long)gridDim.x * rpb;
    for (long long r0 = (long long)blockIdx.x * rpb + threadIdx.x / G; r0 < rows; r0 += RPT * stride) {
        float xv[RPT][NIN];
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const long long r = r0 + q * stride;
#pragma unroll
            for (int k = 0; k < NIN; k++) xv[q][k] = r < rows ? x[r * NIN + k] : 0.f;
        }
#pragma unroll
        for (int q = 0; q < RPT; q++) {
            const long long r = r0 + q * stride;
            if (r >= rows) break;
            float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int k = 0; k < NIN; k++)
#pragma unroll
                for (int j = 0; j < 8; j++) acc[j] = fmaf(xv[q][k], w[k][j], acc[j]);
            TACT hv[8], zv[8];
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const float z = acc[j] + bias[j];
                hv[j] = cvt<TACT>(silu_fast(z));
                zv[j] = cvt<TACT>(z);
            }
            constexpr int V = 8 * sizeof(TACT) / 16;  // 16-byte pieces per thread
            const uint4 *hs = reinterpret_cast<const uint4 *>(hv), *zs = reinterpret_cast<const uint4 *>(zv);
            uint4 *ho = reinterpret_cast<uint4 *>(H + r * N + n0);
#pragma unroll
            for (int u = 0; u < V; u++) ho[u] = hs[u];
            if (Z) {
                uint4 *zo = reinterpret_cast<uint4 *>(Z + r * N + n0);
#pragma unroll
                for (int u = 0; u < V; u++) zo[u] = zs[u];
            }
        }
    }
}

template <typename TACT, int NIN>
void launch_first(const float *x, int rows, const float *W, const float *b, int N, TACT *H, TACT *Z,
                  cudaStream_t s) {
    const int rpb = 256 / (N / 8);
    const long long blocks = ((long long)rows + (long long)rpb * kFirstRows - 1) / ((long long)rpb * kFirstRows);
    const int grid = (int)(blocks < 148 * 8 ? blocks : 148 * 8);
    first_layer_kernel<TACT, NIN><<<grid, 256, 0, s>>>(x, rows, W, b, N, H, Z);
}

template <typename TACT>
void launch_first_n(int n_in, const float *x, int rows, const float *W, const float *b, int N, TACT *H, TACT *Z,
                    cudaStream_t s) {
    switch (n_in) {
        case 1: return launch_first<TACT, 1>(x, rows, W, b, N, H, Z, s);
        case 2: return launch_first<TACT, 2>(x, rows, W, b, N, H, Z, s);
        case 3: return launch_first<TACT, 3>(x, rows, W, b, N, H, Z, s);
        case 4: return launch_first<TACT, 4>(x, rows, W, b, N, H, Z, s);
        case 5: return launch_first<TACT, 5>(x, rows, W, b, N, H, Z, s);
        case 6: return launch_first<TACT, 6>(x, rows, W, b, N, H, Z, s);
        case 7: return launch_first<TACT, 7>(x, rows, W, b, N, H, Z, s);
        default: return launch_first<TACT, 8>(x, rows, W, b, N, H, Z, s);
    }
}

// ---------------------------------------------------------------------------
// Tensor-core forward of the layers fed by BF16 activations (all but the
// first): Z = H W + b with H [M][K] BF16 and the layer's weights as a BF16
// copy kept transposed, Wt [N][K] (k contiguous), multiplied by
// mma.sync.m16n8k16 (BF16 x BF16, FP32 accumulation).  128 x 128 output
// tiles, 8 warps of 64 x 32, 32-deep k slices in a 4-stage cp.async ring,
// fragments by ldmatrix; rows padded to 40 BF16 so that the eight 16-byte
// rows of each ldmatrix hit distinct banks.
// Epilogue as the SIMT kernel's: bias and SiLU into Z and H (BF16), or bias
// into the FP32 output.
// ---------------------------------------------------------------------------
namespace tc {

constexpr int BM = 128, BN = 128, BK = 32, LDS = BK + 8, T = 256;

struct Args {
    int M, N, K;
    const bf16 *A;    // [M][K]
    const bf16 *Wt;   // [N][K]
    const float *bias;
    bf16 *Z;          // EPI_HIDDEN: pre-activation (may be null)
    void *C;          // EPI_HIDDEN: H (BF16); EPI_OUT: y (FP32), [M][N]
};

__device__ __forceinline__ uint32_t saddr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cp16(void *s, const void *g) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(saddr(s)), "l"(g) : "memory");
}

__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void *p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(saddr(p)));
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, "
        "{%0, %1, %2, %3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// Shared memory: STAGES ring slots of one 128 x 32 A tile and one 128 x 32
// Wt tile; slices k0 + BK (STAGES - 1) ahead are in flight while slice k0
// is multiplied, so global latency hides behind three slices of MMAs.
constexpr int STAGES = 4;
constexpr size_t SMEM_BYTES = (size_t)STAGES * 2 * BM * LDS * sizeof(bf16);

template <int EPI>
__global__ void __launch_bounds__(T, 2) gemm_tc_kernel(Args g) {
    extern __shared__ __align__(16) unsigned char smraw[];
    auto As = reinterpret_cast<bf16(*)[BM][LDS]>(smraw);                                   // [STAGES][BM][LDS]
    auto Bs = reinterpret_cast<bf16(*)[BN][LDS]>(smraw + (size_t)STAGES * BM * LDS * sizeof(bf16));
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int wm = warp & 1, wn = warp >> 1;  // 2 x 4 warps: 64 rows x 32 columns each
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int nk = g.K / BK;
    // one 16-byte piece (8 BF16) of a 128 x 32 tile per thread and round
    auto load = [&](int st, int k0) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const int idx = tid + r * T, row = idx >> 2, c8 = (idx & 3) * 8;
            const int gm = m0 + row, gn = n0 + row;
            if (gm < g.M) cp16(&As[st][row][c8], g.A + (long long)gm * g.K + k0 + c8);
            else *reinterpret_cast<uint4 *>(&As[st][row][c8]) = make_uint4(0, 0, 0, 0);
            if (gn < g.N) cp16(&Bs[st][row][c8], g.Wt + (long long)gn * g.K + k0 + c8);
            else *reinterpret_cast<uint4 *>(&Bs[st][row][c8]) = make_uint4(0, 0, 0, 0);
        }
    };
    float acc[4][4][4];
#pragma unroll
    for (int i = 0; i < 4; i++)
#pragma unroll
        for (int j = 0; j < 4; j++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][j][q] = 0.f;
#pragma unroll
    for (int q = 0; q < STAGES - 1; q++) {  // prologue: slices 0 .. STAGES-2, one commit group each
        if (q < nk) load(q, q * BK);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int kc = 0; kc < nk; kc++) {
        const int st = kc % STAGES;
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");  // slice kc has landed
        __syncthreads();  // ... for every thread; every warp is done with slice kc-1
        if (kc + STAGES - 1 < nk) load((kc + STAGES - 1) % STAGES, (kc + STAGES - 1) * BK);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
#pragma unroll
        for (int ks = 0; ks < BK / 16; ks++) {
            uint32_t a[4][4], b[2][4];
#pragma unroll
            for (int mf = 0; mf < 4; mf++)
                ldsm4(a[mf], &As[st][wm * 64 + mf * 16 + (lane & 7) + ((lane >> 3) & 1) * 8][ks * 16 + (lane >> 4) * 8]);
#pragma unroll
            for (int nb = 0; nb < 2; nb++)
                ldsm4(b[nb], &Bs[st][wn * 32 + nb * 16 + (lane & 7) + (lane >> 4) * 8][ks * 16 + ((lane >> 3) & 1) * 8]);
#pragma unroll
            for (int mf = 0; mf < 4; mf++)
#pragma unroll
                for (int nf = 0; nf < 4; nf++)
                    mma_bf16(acc[mf][nf], a[mf], b[nf >> 1][(nf & 1) * 2], b[nf >> 1][(nf & 1) * 2 + 1]);
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    const int gr = lane >> 2, gc = (lane & 3) * 2;
#pragma unroll
    for (int mf = 0; mf < 4; mf++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int m = m0 + wm * 64 + mf * 16 + gr + 8 * h;
            if (m >= g.M) continue;
#pragma unroll
            for (int nf = 0; nf < 4; nf++) {
                const int n = n0 + wn * 32 + nf * 8 + gc;
                if (n >= g.N) continue;
                const bool pair = n + 1 < g.N;  // an odd number of outputs ends in a single column
                const float z0 = acc[mf][nf][2 * h] + g.bias[n], z1 = acc[mf][nf][2 * h + 1] + (pair ? g.bias[n + 1] : 0.f);
                const long long o = (long long)m * g.N + n;
                if constexpr (EPI == EPI_HIDDEN) {
                    if (g.Z) *reinterpret_cast<__nv_bfloat162 *>(g.Z + o) = __floats2bfloat162_rn(z0, z1);
                    *reinterpret_cast<__nv_bfloat162 *>(static_cast<bf16 *>(g.C) + o) =
                        __floats2bfloat162_rn(silu(z0), silu(z1));
                } else {
                    float *c = static_cast<float *>(g.C) + o;
                    if (pair && (reinterpret_cast<uintptr_t>(c) & 7) == 0) {
                        *reinterpret_cast<float2 *>(c) = make_float2(z0, z1);
                    } else {
                        c[0] = z0;
                        if (pair) c[1] = z1;
                    }
                }
            }
        }
}

// BF16 transposed copies Wt_l [N][K] of the weights W_l [K][N] of layers
// 1 .. nl-1 (the layers the tensor-core forward runs).
struct WtTable {
    int nl;
    long long offW[17], offWt[17];
    int K[17], N[17];
};

__global__ void weights_bf16t_kernel(const float *params, bf16 *wt, WtTable t) {
    for (int l = 1; l < t.nl; l++) {
        const long long n = (long long)t.K[l] * t.N[l];
        const float *W = params + t.offW[l];
        bf16 *Wt = wt + t.offWt[l];
        for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
             i += (long long)gridDim.x * blockDim.x) {
            const int nn = (int)(i / t.K[l]), k = (int)(i % t.K[l]);
            Wt[i] = __float2bfloat16_rn(W[(long long)k * t.N[l] + nn]);
        }
    }
}

}  // namespace tc

// ---------------------------------------------------------------------------
// Fifth-generation tensor-core (tcgen05) forward of the layers fed by BF16
// activations whose BF16 weights fit in shared memory (K <= 256 and
// N <= 256, K a multiple of 64, N of 32): Z = H W + b with H [M][K] and
// Wt [N][K] (k contiguous).  A persistent CTA per SM keeps the layer's
// weights resident (one tiled TMA load of K/64 slices of N x 64) and
// streams 128-row tiles of H through a ring of 128 x 64 stages:
//   warp 0 (one thread)  tiled TMA loads of H into the ring,
//   warp 1 (one thread)  tcgen05.mma 128 x N x 16 into a TMEM accumulator,
//                        two accumulators of N columns alternating by tile,
//                        tcgen05.commit releasing ring stages and
//                        signalling finished accumulators,
//   warps 2-17           TMEM -> registers (tcgen05.ld), bias and SiLU;
//                        warp w reads TMEM lanes 32 (w % 4) .. + 31 (its
//                        sub-partition's rows) and every fourth 32-column
//                        chunk, so the epilogue of tile t overlaps the MMAs
//                        of tile t + 1.  Each 32 x 32 block goes through a
//                        swizzled shared-memory buffer (one per warp) and
//                        out by a tiled TMA store, so HBM sees whole lines
//                        (a thread storing its own row touched 32 lines per
//                        warp store, each 32-byte sector in two halves).
// Every mbarrier wait is bounded (tma::mbar_wait); a wait that gives up
// raises ST_TIMEOUT in the status word, the loader waits for the loads it
// issued, the MMA thread for its MMAs, and the block frees its TMEM.
// ---------------------------------------------------------------------------
namespace t5 {

using gabe::tma::mbar_wait;

constexpr int BM = 128, BK = 64, NEPI = 16, NT = 64 + 32 * NEPI;  // NEPI epilogue warps
constexpr int kMaxStages = 8;
constexpr int kTmemCols = 512;                 // two accumulators of up to 256 columns
constexpr int kStageBytes = BM * BK * 2;        // one 128 x 64 BF16 tile of H
constexpr size_t kFixedBytes = 1024 + 1024 + 256;  // alignment slack, bias, barriers

struct Args {
    int M, N, K, stages;
    const float *bias;
    bf16 *Z;                // EPI_HIDDEN: pre-activation (may be null)
    unsigned int *status;
};

// Output element size of the epilogue (BF16 hidden activations, FP32 output).
template <int EPI>
__host__ __device__ constexpr int out_bytes() {
    return EPI == EPI_HIDDEN ? 2 : 4;
}

// Shared memory: weights, ring stages, a staging buffer of 32 x 32 output
// elements per epilogue warp, bias, barriers.
__host__ __device__ inline size_t smem_bytes(int N, int K, int stages, int esize) {
    return kFixedBytes + (size_t)N * K * 2 + (size_t)stages * kStageBytes + (size_t)NEPI * 32 * 32 * esize;
}

__device__ __forceinline__ uint32_t pack_bf16(float a, float b) {
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t *>(&h);
}

template <int EPI>
__global__ void __launch_bounds__(NT, 1)
    gemm_umma_kernel(const __grid_constant__ CUtensorMap mapA, const __grid_constant__ CUtensorMap mapB,
                     const __grid_constant__ CUtensorMap mapC, Args g) {
    namespace tma = gabe::tma;
    namespace umma = gabe::umma;
    extern __shared__ unsigned char smraw[];
    const uint32_t s0 = tma::saddr(smraw);
    unsigned char *sm = smraw + (((s0 + 1023u) & ~1023u) - s0);  // 1024-byte aligned for the swizzle
    const int N = g.N, K = g.K, KB = K / BK, S = g.stages;
    unsigned char *Bs = sm;                                   // K/64 slices of N x 128 bytes
    unsigned char *As = sm + (size_t)N * K * 2;               // S stages of 128 x 128 bytes
    constexpr int ES = out_bytes<EPI>(), SBUF = 32 * 32 * ES;  // one staging buffer
    unsigned char *Cs = As + (size_t)S * kStageBytes;         // [NEPI][SBUF]
    float *bias_s = reinterpret_cast<float *>(Cs + (size_t)NEPI * SBUF);  // 256 floats
    uint64_t *full = reinterpret_cast<uint64_t *>(bias_s + 256);
    uint64_t *empty = full + kMaxStages, *bfull = empty + kMaxStages, *tfull = bfull + 1, *tempty = tfull + 2,
             *done = tempty + 2;
    uint32_t *tbase_s = reinterpret_cast<uint32_t *>(done + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int ntiles = (g.M + BM - 1) / BM;

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            tma::mbar_init(&full[s], 1);
            tma::mbar_init(&empty[s], 1);
        }
        tma::mbar_init(bfull, 1);
        for (int b = 0; b < 2; b++) {
            tma::mbar_init(&tfull[b], 1);
            tma::mbar_init(&tempty[b], 32 * NEPI);  // every epilogue thread
        }
        tma::mbar_init(done, 1);
        tma::fence_barrier_init();
    }
    for (int n = tid; n < N; n += NT) bias_s[n] = g.bias[n];
    if (warp == 1) umma::tmem_alloc(tbase_s, kTmemCols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tbase = *tbase_s;

    if (warp == 0) {
        if (lane == 0) {
            int fills[kMaxStages];
            for (int s = 0; s < kMaxStages; s++) fills[s] = 0;
            tma::mbar_arrive_expect(bfull, (uint32_t)(N * K * 2));
            for (int kb = 0; kb < KB; kb++) umma::load_2d(Bs + (size_t)kb * N * 128, &mapB, kb * BK, 0, bfull);
            int it = 0;
            bool ok = true;
            for (int tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x)
                for (int kb = 0; kb < KB; kb++, it++) {
                    const int s = it % S;
                    if (!mbar_wait(&empty[s], (uint32_t)(((it / S) & 1) ^ 1), g.status)) {
                        ok = false;
                        break;
                    }
                    fills[s]++;
                    tma::mbar_arrive_expect(&full[s], (uint32_t)kStageBytes);
                    umma::load_2d(As + (size_t)s * kStageBytes, &mapA, kb * BK, tile * BM, &full[s]);
                }
            // every load issued has landed before the block may exit
            tma::drain(full, fills, S, g.status);
            mbar_wait(bfull, 0, g.status);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            const uint32_t idesc = umma::idesc_bf16(BM, N);
            bool ok = mbar_wait(bfull, 0, g.status);
            int it = 0, local = 0;
            for (int tile = blockIdx.x; ok && tile < ntiles; tile += gridDim.x, local++) {
                const int b = local & 1;
                if (!mbar_wait(&tempty[b], (uint32_t)(((local >> 1) & 1) ^ 1), g.status)) break;
                umma::fence_after();
                const uint32_t d = tbase + (uint32_t)(b * 256);
                for (int kb = 0; kb < KB; kb++, it++) {
                    const int s = it % S;
                    if (!mbar_wait(&full[s], (uint32_t)((it / S) & 1), g.status)) {
                        ok = false;
                        break;
                    }
                    umma::fence_after();
                    const uint32_t sa = tma::saddr(As + (size_t)s * kStageBytes);
                    const uint32_t sb = tma::saddr(Bs + (size_t)kb * N * 128);
#pragma unroll
                    for (int k = 0; k < BK / 16; k++)
                        umma::mma_bf16(d, umma::desc_k128(sa + 32 * k), umma::desc_k128(sb + 32 * k), idesc,
                                       (uint32_t)((kb | k) != 0));
                    umma::commit(&empty[s]);  // the stage is free once these MMAs have read it
                }
                if (ok) umma::commit(&tfull[b]);
            }
            umma::commit(done);  // arrives once every MMA issued above has completed
            mbar_wait(done, 0, g.status);
        }
    } else {
        constexpr int NH = NEPI / 4;  // epilogue warps per TMEM lane quarter
        const int q = warp & 3, h = (warp - 2) >> 2, nch = N / 32;
        unsigned char *sb = Cs + (size_t)(warp - 2) * SBUF;
        int local = 0, cnt = 0;  // tiles and staged blocks of this warp
        for (int tile = blockIdx.x; tile < ntiles; tile += gridDim.x, local++) {
            const int b = local & 1;
            const bool mine = mbar_wait(&tfull[b], (uint32_t)((local >> 1) & 1), g.status);
            if (!__all_sync(0xffffffffu, mine)) break;
            umma::fence_after();
            const int r0 = tile * BM + q * 32, row = r0 + lane;
            // (a warp whose rows all lie past M stages nothing: every staged
            // block is stored, so the buffer accounting below holds)
            for (int c = h; r0 < g.M && c < nch; c += NH, cnt++) {
                float v[32];
                umma::tmem_ld32(tbase + ((uint32_t)(q * 32) << 16) + (uint32_t)(b * 256 + c * 32), v);
                const int n0 = c * 32;
                const float4 *bq = reinterpret_cast<const float4 *>(bias_s + n0);
#pragma unroll
                for (int u = 0; u < 8; u++) {
                    const float4 bb = bq[u];
                    v[4 * u] += bb.x;
                    v[4 * u + 1] += bb.y;
                    v[4 * u + 2] += bb.z;
                    v[4 * u + 3] += bb.w;
                }
                // the previous block's store must have read the buffer
                if (cnt >= 1) {
                    if (lane == 0) umma::store_wait_read<0>();
                    __syncwarp();
                }
                if constexpr (EPI == EPI_HIDDEN) {
                    // row `lane` of the block: 64 bytes, 16-byte unit u at u ^ ((lane / 2) % 4) (64-byte swizzle)
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        *reinterpret_cast<uint4 *>(sb + lane * 64 + ((u ^ ((lane >> 1) & 3)) << 4)) =
                            make_uint4(pack_bf16(silu_fast(v[8 * u]), silu_fast(v[8 * u + 1])),
                                       pack_bf16(silu_fast(v[8 * u + 2]), silu_fast(v[8 * u + 3])),
                                       pack_bf16(silu_fast(v[8 * u + 4]), silu_fast(v[8 * u + 5])),
                                       pack_bf16(silu_fast(v[8 * u + 6]), silu_fast(v[8 * u + 7])));
                    if (g.Z && row < g.M) {
                        uint4 *zo = reinterpret_cast<uint4 *>(g.Z + (long long)row * N + n0);
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            zo[u] = make_uint4(pack_bf16(v[8 * u], v[8 * u + 1]), pack_bf16(v[8 * u + 2], v[8 * u + 3]),
                                               pack_bf16(v[8 * u + 4], v[8 * u + 5]),
                                               pack_bf16(v[8 * u + 6], v[8 * u + 7]));
                    }
                } else {
                    // row `lane`: 128 bytes, 16-byte unit u at u ^ (lane % 8) (128-byte swizzle)
#pragma unroll
                    for (int u = 0; u < 8; u++)
                        *reinterpret_cast<float4 *>(sb + lane * 128 + ((u ^ (lane & 7)) << 4)) =
                            make_float4(v[4 * u], v[4 * u + 1], v[4 * u + 2], v[4 * u + 3]);
                }
                tma::fence_proxy_async();  // the block's shared writes precede the store's reads
                __syncwarp();
                if (lane == 0) umma::store_2d(&mapC, n0, r0, sb);
            }
            umma::fence_before();
            umma::mbar_arrive(&tempty[b]);
        }
        if (lane == 0) umma::store_wait_all();
    }
    umma::fence_before();
    __syncthreads();
    if (warp == 1) {
        umma::fence_after();
        umma::tmem_free(tbase, kTmemCols);
    }
}

}  // namespace t5

// ---------------------------------------------------------------------------
// The whole forward in one launch, for networks whose layers all take the
// tcgen05 form above and the first-layer kernel: the activations of a tile of
// 128 rows stay in shared memory from the first layer to the last, so HBM
// sees the inputs and the outputs only (layer by layer, each hidden
// activation crosses it twice: 4.3 GB of 5.1 at 1M rows).
//
// One persistent CTA per SM takes groups of two tiles (one where there are
// fewer tiles than SMs): per tile its activations (K/64 slices of 128 x 64
// BF16, 128-byte swizzle, as the MMA reads them) and a 256-column TMEM
// accumulator, and one ring of 32 KB weight slots (up to 256 output columns x
// 64 inputs) that streams each layer's weights from L2 once per tile.
//   warp 0 (one thread)  tiled TMA loads of the weight slots, as far ahead
//                        as the ring allows,
//   warp 1 (one thread)  per layer and tile: the MMAs,
//   warps 2-17           first layer on FMA, then per layer and tile bias +
//                        SiLU of 32 x 32 blocks, in the old activations'
//                        place (the tile's MMAs have completed), then the
//                        output layer's blocks staged there and stored by TMA.
// One tile's MMAs and weight loads run under the other's SiLU, which needs the
// special-function pipe twice per value: 0.48 ms for 1M rows x 4 x 256
// values at 1.9 GHz, four times what the tensor pipe needs.  A tile's output
// layer is followed by the first layer of the next group's tile, so that the
// other tile's MMAs have SiLU to run under there too.
// Results are those of the layer-by-layer kernels bit for bit: the same
// products in the same K order, the same epilogue arithmetic.
// Measured at 1965 MHz: 1M rows through the default network 0.86 ms a call
// (calls queued one behind another) against 1.02 for the five launches, 41
// rows 27 us a call waited for against 47.  What set the pace on the way
// there, read from clock stamps: divisions and remainders in the two issuing
// threads (1000 cycles per weight slot beside 16 busy warps; 1.2 ms), 16 KB
// slots (twice the waits and commits of 32 KB ones), a first layer by a lane
// per row.  What is left: a hidden layer's SiLU takes 4.2-4.9k cycles per tile
// (4.1k by the special-function pipe), the first layer's 8-9k.
// Waits are bounded as in the kernel above.
// ---------------------------------------------------------------------------
namespace t6 {

using gabe::tma::mbar_wait;
using t5::BK;
using t5::BM;
using t5::pack_bf16;

constexpr int kEpiWarps = 16, kThreadsPerCta = 64 + 32 * kEpiWarps;
constexpr int kSlotBytes = 256 * BK * 2;  // up to 256 output columns x 64 inputs
constexpr int kMaxSlots = 8;
constexpr int kMaxLayers = 17;
constexpr int kBlockBytes = 32 * 32 * 4;  // one staged FP32 output block
constexpr uint32_t kCols = 256;           // TMEM columns per tile

struct Args {
    int M, width, n_in, n_out, nl, slots, tiles, box;  // tiles per group (1 or 2), rows per weight load
    const float *x, *W0;
    const float *bias[kMaxLayers];
    int rowoff[kMaxLayers];  // first row of layer l in the stacked transposed weights
    bf16 *H, *Z;             // KEEP: activations of hidden layer l at + l * keep_stride
    long long keep_stride;
    unsigned int *status;
};

// one tile's activations (also the staging area of its output blocks)
__host__ __device__ inline size_t act_bytes(int width) {
    const size_t a = (size_t)(width / BK) * BM * BK * 2, stage = (size_t)kEpiWarps * kBlockBytes;
    return a < stage ? stage : a;
}
__host__ __device__ inline size_t smem_bytes(int width, int slots) {
    return 1024 + 2 * act_bytes(width) + (size_t)slots * kSlotBytes + 256;
}

// Row `row` of the activations: 16-byte unit u of the 32 columns from col0 (a multiple of 32).
__device__ __forceinline__ uint4 *act_unit(unsigned char *act, int row, int col0, int u) {
    const int kb = col0 / BK, unit = (col0 % BK) / 8 + u;
    return reinterpret_cast<uint4 *>(act + (size_t)kb * BM * BK * 2 + (row >> 3) * 1024 + (row & 7) * 128 +
                                     ((unit ^ (row & 7)) << 4));
}

// Packed FP32 pairs: one issue slot for two values, each rounded as the scalar operation rounds it.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<uint64_t &>(r))
        : "l"(reinterpret_cast<uint64_t &>(a)), "l"(reinterpret_cast<uint64_t &>(b)),
          "l"(reinterpret_cast<uint64_t &>(c)));
    return r;
}
__device__ __forceinline__ float2 add2(float2 a, float2 b) {
    float2 r;
    asm("add.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<uint64_t &>(r))
        : "l"(reinterpret_cast<uint64_t &>(a)), "l"(reinterpret_cast<uint64_t &>(b)));
    return r;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 r;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<uint64_t &>(r))
        : "l"(reinterpret_cast<uint64_t &>(a)), "l"(reinterpret_cast<uint64_t &>(b)));
    return r;
}
// silu_fast of a pair
__device__ __forceinline__ float2 silu2(float2 z) {
    const float2 t = mul2(z, make_float2(-1.4426950408889634f, -1.4426950408889634f));
    float2 e, r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.x) : "f"(t.x));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e.y) : "f"(t.y));
    e = add2(e, make_float2(1.f, 1.f));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.x) : "f"(e.x));
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r.y) : "f"(e.y));
    return mul2(z, r);
}

// v += b, 32 values read by every lane (cached in L1)
__device__ __forceinline__ void add_bias(float2 (&v)[16], const float *b) {
    const float4 *bq = reinterpret_cast<const float4 *>(b);
#pragma unroll
    for (int u = 0; u < 8; u++) {
        const float4 bb = __ldg(bq + u);
        v[2 * u] = add2(v[2 * u], make_float2(bb.x, bb.y));
        v[2 * u + 1] = add2(v[2 * u + 1], make_float2(bb.z, bb.w));
    }
}
// 32 bytes in one store (32-byte aligned): half the line touches of two 16-byte ones where each lane writes a row.
__device__ __forceinline__ void store32(void *p, const uint4 &a, const uint4 &b) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w),
                 "r"(b.x), "r"(b.y), "r"(b.z), "r"(b.w)
                 : "memory");
}
// This lane's row of 32 accumulator columns.
__device__ __forceinline__ void load_block(uint32_t taddr, float2 (&v)[16]) {
    float f[32];
    gabe::umma::tmem_ld32(taddr, f);
#pragma unroll
    for (int j = 0; j < 16; j++) v[j] = make_float2(f[2 * j], f[2 * j + 1]);
}

// KEEP: also store the hidden layers' activations and pre-activations (training).
// NIN: at least the number of inputs (4 or 8: weights a lane holds in the first layer).
template <bool KEEP, int NIN>
__global__ void __launch_bounds__(kThreadsPerCta, 1)
    mlp_kernel(const __grid_constant__ CUtensorMap mapW, const __grid_constant__ CUtensorMap mapY,
               const __grid_constant__ Args g) {
    namespace tma = gabe::tma;
    namespace umma = gabe::umma;
    extern __shared__ unsigned char smraw[];
    const uint32_t s0 = tma::saddr(smraw);
    unsigned char *sm = smraw + (((s0 + 1023u) & ~1023u) - s0);
    const int W = g.width, KB = W / BK, S = g.slots, nl = g.nl;
    unsigned char *acts = sm;
    const size_t AB = act_bytes(W);
    unsigned char *ring = sm + 2 * AB;
    uint64_t *wfull = reinterpret_cast<uint64_t *>(ring + (size_t)S * kSlotBytes);
    uint64_t *wempty = wfull + kMaxSlots, *act = wempty + kMaxSlots, *dfull = act + 2, *sfree = dfull + 2,
             *done = sfree + 2;  // act, dfull, sfree: one per tile
    uint32_t *tbase_s = reinterpret_cast<uint32_t *>(done + 1);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int rows_per_group = g.tiles * BM, ngroups = (g.M + rows_per_group - 1) / rows_per_group;
    // tiles of group grp that hold rows
    auto tiles_of = [&](int grp) { return g.tiles == 2 && (long long)grp * rows_per_group + BM < g.M ? 2 : 1; };
    auto width_of = [&](int l) { return l + 1 == nl ? g.n_out : W; };

    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            tma::mbar_init(&wfull[s], 1);
            tma::mbar_init(&wempty[s], 1);
        }
        for (int t = 0; t < 2; t++) {
            tma::mbar_init(&act[t], 32 * kEpiWarps);
            tma::mbar_init(&dfull[t], 1);
            tma::mbar_init(&sfree[t], kEpiWarps);
        }
        tma::mbar_init(done, 1);
        tma::fence_barrier_init();
    }
    if (warp == 1) umma::tmem_alloc(tbase_s, 2 * kCols);
    umma::fence_before();
    __syncthreads();
    umma::fence_after();
    const uint32_t tbase = *tbase_s;

    if (warp == 0) {
        if (lane == 0) {
            int fills[kMaxSlots];
            for (int s = 0; s < kMaxSlots; s++) fills[s] = 0;
            int s = 0;
            uint32_t phase = 1;  // parity of wempty[s] to wait for; flips as the ring wraps
            bool ok = true;
            for (int grp = blockIdx.x; ok && grp < ngroups; grp += gridDim.x) {
                const int nt = tiles_of(grp);
                for (int l = 1; ok && l < nl; l++) {
                    const int y0 = g.rowoff[l], rows = width_of(l);
                    for (int t = 0; ok && t < nt; t++)
                        for (int x = 0; x < W; x += BK) {
                            if (!mbar_wait(&wempty[s], phase, g.status)) {
                                ok = false;
                                break;
                            }
                            fills[s]++;
                            tma::mbar_arrive_expect(&wfull[s], (uint32_t)rows * 128);
                            unsigned char *dst = ring + (size_t)s * kSlotBytes;
                            for (int r = 0; r < rows; r += g.box) umma::load_2d(dst + r * 128, &mapW, x, y0 + r, &wfull[s]);
                            if (++s == S) {
                                s = 0;
                                phase ^= 1;
                            }
                        }
                }
            }
            // every load issued has landed before the block may exit
            tma::drain(wfull, fills, S, g.status);
        }
    } else if (warp == 1) {
        if (lane == 0) {
            bool ok = true;
            // one thread issues everything, beside 16 busy warps: no divisions, descriptors by addition
            int s = 0;
            uint32_t phase = 0, pact = 0;  // parities of wfull[s], and of act[t] in bit t
            const uint64_t da0 = umma::desc_k128(tma::saddr(acts)), db0 = umma::desc_k128(tma::saddr(ring));
            const uint64_t da_tile = AB >> 4, da_kb = (BM * BK * 2) >> 4, db_slot = kSlotBytes >> 4;  // in 16-byte units
            for (int grp = blockIdx.x; ok && grp < ngroups; grp += gridDim.x) {
                const int nt = tiles_of(grp);
                for (int l = 1; ok && l < nl; l++) {
                    const uint32_t idesc = umma::idesc_bf16(BM, width_of(l));
                    for (int t = 0; ok && t < nt; t++) {
                        if (!(ok = mbar_wait(&act[t], (pact >> t) & 1u, g.status))) break;
                        pact ^= 1u << t;
                        umma::fence_after();
                        const uint32_t d = tbase + (uint32_t)t * kCols;
                        uint64_t da = da0 + (t ? da_tile : 0);
                        for (int kb = 0; kb < KB; kb++, da += da_kb) {
                            if (!(ok = mbar_wait(&wfull[s], phase, g.status))) break;
                            umma::fence_after();
                            const uint64_t db = db0 + (uint64_t)s * db_slot;
#pragma unroll
                            for (int k = 0; k < BK / 16; k++)
                                umma::mma_bf16(d, da + 2 * k, db + 2 * k, idesc, (uint32_t)((kb | k) != 0));
                            umma::commit(&wempty[s]);
                            if (++s == S) {
                                s = 0;
                                phase ^= 1;
                            }
                        }
                        if (ok) umma::commit(&dfull[t]);
                    }
                }
            }
            umma::commit(done);  // arrives once every MMA issued above has completed
            mbar_wait(done, 0, g.status);
        }
    } else {
        constexpr int NH = kEpiWarps / 4;  // epilogue warps per TMEM lane quarter
        const int q = warp & 3, hg = (warp - 2) >> 2, ew = warp - 2;
        const uint32_t tq = tbase + ((uint32_t)(q * 32) << 16);
        int nd[2] = {0, 0}, nfree[2] = {0, 0};
        // SiLU of this lane's 32 values of hidden layer l, into the activations (and kept)
        auto finish = [&](int t, int l, long long row, int col0, const float2 (&v)[16]) {
#pragma unroll
            for (int u = 0; u < 4; u += 2) {
                uint4 pv[2], zv[2];
#pragma unroll
                for (int o = 0; o < 2; o++) {
                    uint32_t p[4];
                    const float2 *z = v + 4 * (u + o);
#pragma unroll
                    for (int j = 0; j < 4; j++) {
                        const float2 y = silu2(z[j]);
                        p[j] = pack_bf16(y.x, y.y);
                    }
                    pv[o] = make_uint4(p[0], p[1], p[2], p[3]);
                    if (KEEP)
                        zv[o] = make_uint4(pack_bf16(z[0].x, z[0].y), pack_bf16(z[1].x, z[1].y),
                                           pack_bf16(z[2].x, z[2].y), pack_bf16(z[3].x, z[3].y));
                    *act_unit(acts + t * AB, q * 32 + lane, col0, u + o) = pv[o];
                }
                if (KEEP && row < g.M) {
                    const long long o = l * g.keep_stride + row * W + col0 + 8 * u;
                    store32(g.H + o, pv[0], pv[1]);
                    store32(g.Z + o, zv[0], zv[1]);
                }
            }
        };
        auto ready = [&](int t) {  // this thread's part of tile t's new activations stands
            umma::fence_before();
            tma::fence_proxy_async();
            umma::mbar_arrive(&act[t]);
        };
        auto wait_all = [&](uint64_t *bar, int n) {
            const bool r = mbar_wait(bar, (uint32_t)(n & 1), g.status);
            return (bool)__all_sync(0xffffffffu, r);
        };
        // First layer of rows base .. base + 127 into tile t.  A warp makes eight rows, a row by W / 8 lanes with
        // eight columns each, whose weights stay in registers (a lane per row instead reads every weight in every
        // lane: four data-path cycles per 16 bytes, 8-9k cycles per tile against the 4.1k of its SiLU).  xs: the
        // eight rows' inputs, lane i holding values i and i + 32.
        auto load_x = [&](long long base, float (&xs)[NIN / 4]) {
            const long long n = (g.M - base - ew * 8) * g.n_in;  // values from the warp's first row on
#pragma unroll
            for (int u = 0; u < NIN / 4; u++) {
                const int at = lane + 32 * u;
                xs[u] = at < 8 * g.n_in && at < n ? __ldg(g.x + (base + ew * 8) * g.n_in + at) : 0.f;
            }
        };
        auto first = [&](int t, long long base, const float (&xs)[NIN / 4]) {
            const int G = W / 8, rpp = 32 / G, col0 = (lane % G) * 8;  // rows per pass
            float2 w[NIN][4], bb[4];
#pragma unroll
            for (int k = 0; k < NIN; k++)
#pragma unroll
                for (int u = 0; u < 2; u++) {
                    const float4 ww = k < g.n_in ? __ldg(reinterpret_cast<const float4 *>(g.W0 + k * W + col0) + u)
                                                 : make_float4(0.f, 0.f, 0.f, 0.f);
                    w[k][2 * u] = make_float2(ww.x, ww.y);
                    w[k][2 * u + 1] = make_float2(ww.z, ww.w);
                }
#pragma unroll
            for (int u = 0; u < 2; u++) {
                const float4 ww = __ldg(reinterpret_cast<const float4 *>(g.bias[0] + col0) + u);
                bb[2 * u] = make_float2(ww.x, ww.y);
                bb[2 * u + 1] = make_float2(ww.z, ww.w);
            }
            for (int j0 = 0; j0 < 8 && base + ew * 8 + j0 < g.M; j0 += 2 * rpp) {  // two passes at a time
                float2 v[2][4];
#pragma unroll
                for (int o = 0; o < 2; o++)
#pragma unroll
                    for (int c = 0; c < 4; c++) v[o][c] = make_float2(0.f, 0.f);
#pragma unroll
                for (int k = 0; k < NIN; k++) {
                    if (k >= g.n_in) break;
#pragma unroll
                    for (int o = 0; o < 2; o++) {
                        const int at = (j0 + o * rpp + lane / G) * g.n_in + k;
                        float xk = __shfl_sync(0xffffffffu, xs[0], at & 31);
                        if constexpr (NIN > 4) {
                            const float hi = __shfl_sync(0xffffffffu, xs[1], at & 31);
                            if (at >= 32) xk = hi;
                        }
#pragma unroll
                        for (int c = 0; c < 4; c++) v[o][c] = fma2(make_float2(xk, xk), w[k][c], v[o][c]);
                    }
                }
                uint32_t p[2][4];
#pragma unroll
                for (int o = 0; o < 2; o++)
#pragma unroll
                    for (int c = 0; c < 4; c++) {
                        v[o][c] = add2(v[o][c], bb[c]);
                        const float2 y = silu2(v[o][c]);
                        p[o][c] = pack_bf16(y.x, y.y);
                    }
#pragma unroll
                for (int o = 0; o < 2; o++) {
                    const int r = ew * 8 + j0 + o * rpp + lane / G;
                    const uint4 pv = make_uint4(p[o][0], p[o][1], p[o][2], p[o][3]);
                    *act_unit(acts + t * AB, r, col0 & ~31, (col0 & 31) / 8) = pv;
                    if (KEEP && base + r < g.M) {
                        const long long at = (base + r) * W + col0;
                        *reinterpret_cast<uint4 *>(g.H + at) = pv;
                        *reinterpret_cast<uint4 *>(g.Z + at) =
                            make_uint4(pack_bf16(v[o][0].x, v[o][0].y), pack_bf16(v[o][1].x, v[o][1].y),
                                       pack_bf16(v[o][2].x, v[o][2].y), pack_bf16(v[o][3].x, v[o][3].y));
                    }
                }
            }
            ready(t);
        };
        bool ok = true;
        // rows of this warp in tile t of group grp; a warp without rows of a tile only arrives (its accumulator
        // rows are never read)
        auto row_of = [&](int grp, int t) { return (long long)grp * rows_per_group + t * BM + q * 32; };
        for (int t = 0; t < ((int)blockIdx.x < ngroups ? tiles_of(blockIdx.x) : 0); t++) {
            float xs[NIN / 4];
            load_x(row_of(blockIdx.x, t) - q * 32, xs);
            first(t, row_of(blockIdx.x, t) - q * 32, xs);
        }
        for (int grp = blockIdx.x; ok && grp < ngroups; grp += gridDim.x) {
            const int nt = tiles_of(grp);
            for (int l = 1, t = 0; ok && l + 1 < nl; t + 1 < nt ? t++ : (t = 0, l++)) {  // hidden layers
                const long long wr = row_of(grp, t);
                if (!(ok = wait_all(&dfull[t], t ? nd[1]++ : nd[0]++))) break;
                umma::fence_after();
                for (int col0 = hg * 32; wr < g.M && col0 < W; col0 += 32 * NH) {
                    float2 v[16];
                    load_block(tq + (uint32_t)(t * kCols + col0), v);
                    add_bias(v, g.bias[l] + col0);
                    finish(t, l, wr + lane, col0, v);
                }
                ready(t);
            }
            // per tile: output layer, its blocks staged in the activations' place (the tile's MMAs have completed)
            // and stored by TMA, then the first layer of the next group's tile, under the other tile's MMAs
            const int next = grp + gridDim.x, nt_next = next < ngroups ? tiles_of(next) : 0;
            for (int t = 0; ok && t < nt; t++) {
                const long long wr = row_of(grp, t);
                float xs[NIN / 4];
                if (t < nt_next) load_x(row_of(next, t) - q * 32, xs);
                if (!(ok = wait_all(&dfull[t], t ? nd[1]++ : nd[0]++))) break;
                umma::fence_after();
                unsigned char *sb = acts + t * AB + (size_t)ew * kBlockBytes;
                for (int col0 = hg * 32; wr < g.M && col0 < g.n_out; col0 += 32 * NH) {
                    float2 v[16];
                    load_block(tq + (uint32_t)(t * kCols + col0), v);
                    add_bias(v, g.bias[nl - 1] + col0);
                    if (col0 >= 32 * NH) {  // the last block's store must have read the buffer
                        if (lane == 0) umma::store_wait_read<0>();
                        __syncwarp();
                    }
#pragma unroll
                    for (int u = 0; u < 8; u++)  // row `lane`: 128 bytes, 16-byte unit u at u ^ (lane % 8)
                        *reinterpret_cast<float4 *>(sb + lane * 128 + ((u ^ (lane & 7)) << 4)) =
                            make_float4(v[2 * u].x, v[2 * u].y, v[2 * u + 1].x, v[2 * u + 1].y);
                    tma::fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) umma::store_2d(&mapY, col0, (int)wr, sb);
                }
                umma::fence_before();
                if (t >= nt_next) continue;
                if (lane == 0) {
                    umma::store_wait_read<0>();
                    umma::mbar_arrive(&sfree[t]);
                }
                if (!(ok = wait_all(&sfree[t], t ? nfree[1]++ : nfree[0]++))) break;
                first(t, row_of(next, t) - q * 32, xs);
            }
        }
        if (lane == 0) umma::store_wait_all();
    }
    umma::fence_before();
    __syncthreads();
    if (warp == 1) {
        umma::fence_after();
        umma::tmem_free(tbase, 2 * kCols);
    }
}

}  // namespace t6

// dW = sum over splits of the partial products, db = sum of the partial
// column sums; fixed order, so the result does not depend on scheduling.
__global__ void __launch_bounds__(256) splitk_reduce_kernel(const float *ws, const float *dbp, int splits,
                                                            long long mn, int N, float *dW, float *db) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < mn + N;
         i += (long long)gridDim.x * blockDim.x) {
        float s = 0.f;
        if (i < mn)
            for (int z = 0; z < splits; z++) s += ws[z * mn + i];
        else
            for (int z = 0; z < splits; z++) s += dbp[(long long)z * N + (i - mn)];
        (i < mn ? dW[i] : db[i - mn]) = s;
    }
}

struct TrainScalars {
    double loss_last;
    double loss_sum;  // sum of batch losses since the last read
    long long loss_n;
    long long step;       // Adam steps taken
    long long batch_idx;  // batches taken since the last reset
    float inv_count;
    unsigned int counter;
};

constexpr int kLossBlocks = 148;

// Rows perm[batch_idx * B + i] of x and t into the batch buffers.
__global__ void gather_kernel(const float *x, const float *t, const int32_t *perm, const TrainScalars *ts, int B,
                              int nin, int nout, float *xb, float *tb) {
    const long long base = ts->batch_idx * (long long)B;
    const int w = nin + nout;
    for (long long q = blockIdx.x * (long long)blockDim.x + threadIdx.x; q < (long long)B * w;
         q += (long long)gridDim.x * blockDim.x) {
        const int i = (int)(q / w), c = (int)(q % w);
        const long long r = perm[base + i];
        if (c < nin) xb[(long long)i * nin + c] = x[r * nin + c];
        else tb[(long long)i * nout + (c - nin)] = t[r * nout + (c - nin)];
    }
}

// dY = 2 (y - t) on finite targets (0 elsewhere), unnormalised; the loss
// sum/count and 1/count (applied in the Adam step) from fixed-order block
// partials.  The last block also advances the step and batch counters.
__global__ void __launch_bounds__(256) loss_kernel(const float *y, const float *t, long long n, float *dy,
                                                   double2 *part, TrainScalars *ts, int count_batch) {
    double s = 0., c = 0.;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
        const float tv = t[i];
        if (isfinite(tv)) {
            const float d = y[i] - tv;
            dy[i] = 2.f * d;
            s += (double)d * d;
            c += 1.;
        } else {
            dy[i] = 0.f;
        }
    }
    __shared__ double rs[256], rc[256];
    rs[threadIdx.x] = s;
    rc[threadIdx.x] = c;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            rs[threadIdx.x] += rs[threadIdx.x + w];
            rc[threadIdx.x] += rc[threadIdx.x + w];
        }
        __syncthreads();
    }
    __shared__ bool last;
    if (threadIdx.x == 0) {
        part[blockIdx.x] = make_double2(rs[0], rc[0]);
        __threadfence();
        last = atomicAdd(&ts->counter, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // the block partials arrive together, and are added in block order
    __threadfence();
    static_assert(kLossBlocks <= 256, "one partial per thread");
    if (threadIdx.x < gridDim.x) {
        const double2 p = __ldcg(&part[threadIdx.x]);
        rs[threadIdx.x] = p.x;
        rc[threadIdx.x] = p.y;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        double S = 0., C = 0.;
        for (unsigned b = 0; b < gridDim.x; b++) {
            S += rs[b];
            C += rc[b];
        }
        const double L = C > 0. ? S / C : 0.;
        ts->loss_last = L;
        ts->inv_count = C > 0. ? (float)(1. / C) : 0.f;
        if (count_batch) {
            ts->loss_sum += L;
            ts->loss_n += 1;
            ts->step += 1;
            ts->batch_idx += 1;
        }
        ts->counter = 0u;
    }
}

// grad *= 1/count (for gabe_mlp_loss_grad)
__global__ void scale_kernel(float *g, long long n, const TrainScalars *ts) {
    const float s = ts->inv_count;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        g[i] *= s;
}

struct AdamHyper {
    float lr, b1, b2, eps, wd, lr_min;
    long long decay_steps;  // cosine from lr to lr_min over this many steps (0 = constant lr)
};

// The step's scalars: 1/count, bias corrections, learning rate.
struct AdamStep {
    float inv, bc1, bc2, lr;
};
__device__ __forceinline__ float adam_correction(float beta, const TrainScalars *ts) {
    return (float)(1. - pow((double)beta, (double)ts->step));
}
__device__ __forceinline__ float adam_rate(const AdamHyper &h, const TrainScalars *ts) {
    if (h.decay_steps <= 0) return h.lr;
    const double t = (double)ts->step, f = fmin(t - 1., (double)h.decay_steps) / (double)h.decay_steps;
    return (float)(h.lr_min + 0.5 * (h.lr - h.lr_min) * (1. + cos(M_PI * f)));
}
__device__ __forceinline__ AdamStep adam_step(const AdamHyper &h, const TrainScalars *ts) {
    return AdamStep{ts->inv_count, adam_correction(h.b1, ts), adam_correction(h.b2, ts), adam_rate(h, ts)};
}

// AdamW with bias correction of parameter i; g is the unnormalised batch
// gradient.  Returns the new value.
__device__ __forceinline__ float adam_update(float *p, float *m, float *v, long long i, float g, const AdamHyper &h,
                                             const AdamStep &a) {
    // the roundings are spelled out, so that every kernel that takes this step gives the same bits
    const float gi = __fmul_rn(g, a.inv);
    float pi = p[i];
    pi = __fmaf_rn(-__fmul_rn(a.lr, h.wd), pi, pi);
    const float mi = __fmaf_rn(1.f - h.b1, gi, __fmul_rn(h.b1, m[i]));
    const float vi = __fmaf_rn(__fmul_rn(1.f - h.b2, gi), gi, __fmul_rn(h.b2, v[i]));
    m[i] = mi;
    v[i] = vi;
    return p[i] = __fsub_rn(pi, __fdiv_rn(__fmul_rn(a.lr, __fdiv_rn(mi, a.bc1)),
                                          __fadd_rn(__fsqrt_rn(__fdiv_rn(vi, a.bc2)), h.eps)));
}

__global__ void adam_kernel(float *p, const float *g, float *m, float *v, long long n, AdamHyper h,
                            const TrainScalars *ts) {
    const AdamStep a = adam_step(h, ts);
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        adam_update(p, m, v, i, g[i], h, a);
}

// End of a small batch's step in one launch: adds the split-K partials of
// every gradient in order, takes the AdamW step and writes the BF16
// transposed copy of the new weight (GRAD: stores the normalised gradient
// instead).  A block takes a 32 x 32 tile of one layer's weights, transposed
// through shared memory, or 256 biases.
struct UpdateArgs {
    int nl, first[kMaxGradLayers + 1];  // first block of layer l: its weight tiles, then its biases
    int K[kMaxGradLayers], N[kMaxGradLayers], splits[kMaxGradLayers];
    long long offW[kMaxGradLayers], offb[kMaxGradLayers], offWt[kMaxGradLayers];
    const float *ws[kMaxGradLayers], *dbp[kMaxGradLayers];
    float *p, *m, *v, *grads;
    bf16 *wt;  // null: no BF16 copy
    AdamHyper h;
    const TrainScalars *ts;
};
__device__ __forceinline__ float sum_splits(const float *ws, long long stride, int splits) {
    float s = 0.f;
    for (int z0 = 0; z0 < splits; z0 += 8) {  // eight loads in flight, added in order
        float v[8];
#pragma unroll
        for (int u = 0; u < 8; u++) v[u] = z0 + u < splits ? ws[(z0 + u) * stride] : 0.f;
#pragma unroll
        for (int u = 0; u < 8; u++)
            if (z0 + u < splits) s += v[u];
    }
    return s;
}
template <bool GRAD>
__global__ void __launch_bounds__(256) update_kernel(const __grid_constant__ UpdateArgs a) {
    __shared__ AdamStep step;
    __shared__ bf16 tile[32][33];
    // the scalars by one warp each (FP64 powers), while the gradients are summed
    if (threadIdx.x == 0) step.inv = a.ts->inv_count;
    if (!GRAD && threadIdx.x == 32) step.bc1 = adam_correction(a.h.b1, a.ts);
    if (!GRAD && threadIdx.x == 64) step.bc2 = adam_correction(a.h.b2, a.ts);
    if (!GRAD && threadIdx.x == 96) step.lr = adam_rate(a.h, a.ts);
    int l = 0;
    while (l + 1 < a.nl && (int)blockIdx.x >= a.first[l + 1]) l++;
    const int b = blockIdx.x - a.first[l], K = a.K[l], N = a.N[l];
    const int nx = (N + 31) / 32, tiles = nx * ((K + 31) / 32);
    auto put = [&](long long i, float g) {
        if constexpr (GRAD) return a.grads[i] = g * step.inv;
        else return adam_update(a.p, a.m, a.v, i, g, a.h, step);
    };
    if (b >= tiles) {
        const int n = (b - tiles) * 256 + threadIdx.x;
        const float g = n < N ? sum_splits(a.dbp[l] + n, N, a.splits[l]) : 0.f;
        __syncthreads();
        if (n < N) put(a.offb[l] + n, g);
        return;
    }
    const int k0 = (b / nx) * 32, n0 = (b % nx) * 32, x = threadIdx.x % 32, y = threadIdx.x / 32;
    float g[4];
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int k = k0 + y + 8 * r, n = n0 + x;
        g[r] = k < K && n < N ? sum_splits(a.ws[l] + (long long)k * N + n, (long long)K * N, a.splits[l]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 4; r++) {
        const int k = k0 + y + 8 * r, n = n0 + x;
        if (k < K && n < N) {
            const float w = put(a.offW[l] + (long long)k * N + n, g[r]);
            if (!GRAD) tile[x][y + 8 * r] = __float2bfloat16_rn(w);
        }
    }
    if (GRAD || !a.wt || l == 0) return;
    __syncthreads();
#pragma unroll
    for (int r = 0; r < 32; r += 8) {
        const int n = n0 + y + r, k = k0 + x;
        if (k < K && n < N) a.wt[a.offWt[l] + (long long)n * K + k] = tile[y + r][x];
    }
}

}  // namespace

struct gabe_mlp {
    gabe_mlp_params p{};
    int dev = 0;
    bool f32act = false;
    cudaStream_t stream = nullptr;
    int nl = 0;                      // layers (depth + 1)
    std::vector<int> K, N;           // per layer
    std::vector<long long> offW, offb;
    long long P = 0;
    float *params = nullptr, *grads = nullptr, *mom = nullptr, *vel = nullptr;
    float *xb = nullptr, *tb = nullptr, *y = nullptr, *dy = nullptr, *d0 = nullptr, *d1 = nullptr;
    float *ws = nullptr, *dbp = nullptr;  // split-K partials of the weight gradient
    // batches of at most small_rows rows: every layer's gradient of the pre-activations and split-K partials
    float *small_delta = nullptr, *small_ws = nullptr;
    int small_rows = 0;
    int batch = 1;  // of the last gabe_mlp_train call
    std::vector<long long> small_off;  // floats: per layer, weight partials then bias partials
    bf16 *wt = nullptr;              // BF16 transposed weights of layers >= 1 (tensor-core forward)
    tc::WtTable wtab{};
    unsigned int *status = nullptr;  // device word: a bounded wait of the tcgen05 forward gave up
    int umma_stages[17] = {};        // per layer: ring stages of the tcgen05 forward, 0 = mma.sync kernel
    int fused_box = 0;               // rows per weight load of it
    int fused_slots = 0;             // weight slots of the one-launch forward (t6), 0 = layer by layer
    CUtensorMap map_wt{};            // the stacked BF16 weights, for it
    void *Z = nullptr, *H = nullptr;  // [depth][max_rows][width] activation type
    double2 *part = nullptr;
    TrainScalars *ts = nullptr;
    cudaGraph_t graph = nullptr;
    cudaGraphExec_t gexec = nullptr;
    const void *g_x = nullptr, *g_t = nullptr, *g_perm = nullptr;
    int g_batch = 0;
    std::string err;
};

namespace {

thread_local std::string g_mlp_create_error;

int mset(gabe_mlp *m, int code, const char *fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof(buf), fmt, ap);
    va_end(ap);
    if (m) m->err = buf;
    else g_mlp_create_error = buf;
    return code;
}

#define MCK(m, call)                                                                                   \
    do {                                                                                               \
        cudaError_t _e = (call);                                                                       \
        if (_e != cudaSuccess) return mset((m), GABE_ERR_CUDA, "%s: %s", #call, cudaGetErrorString(_e)); \
    } while (0)

size_t act_size(const gabe_mlp *m) { return m->f32act ? sizeof(float) : sizeof(bf16); }

void *act_at(const gabe_mlp *m, void *base, int layer) {
    return static_cast<char *>(base) + (size_t)layer * m->p.max_rows * m->p.width * act_size(m);
}

constexpr int kMaxSplits = 16;
// Batches up to here take the one-launch weight gradients and update, which keep every layer's deltas and
// partials at once; larger ones are long enough per launch.  So are those of wide networks: the two buffers take
// no more than kSmallBytes (the default network's 34 MB), with fewer rows or none, and a handle does without them
// where the memory is not there.
constexpr int kSmallRows = 4096;
constexpr long long kSmallBytes = 256ll << 20;

// Splits of the batch for the weight gradient of a K x N layer, enough for about two blocks per SM, and the
// rows of one split.
int most_splits(int K, int N) {
    const int tiles = ((K + BM - 1) / BM) * ((N + BN - 1) / BN), splits = (296 + tiles - 1) / tiles;
    return splits < 1 ? 1 : (splits > kMaxSplits ? kMaxSplits : splits);
}
int weight_grad_splits(int K, int N, int rows, int *chunk) {
    const int splits = most_splits(K, N);
    int c = (rows + splits - 1) / splits;
    c = (c + BK - 1) / BK * BK;
    *chunk = c;
    return (rows + c - 1) / c;
}

template <typename TA, typename TACT, int EPI>
int launch_gemm(gabe_mlp *m, const GemmArgs &g, int splits = 1) {
    const dim3 grid((g.N + BN - 1) / BN, (g.M + BM - 1) / BM, splits);
    gemm_kernel<TA, TACT, EPI><<<grid, kThreads, 0, m->stream>>>(g);
    MCK(m, cudaGetLastError());
    return GABE_OK;
}

// Refreshes the BF16 transposed weight copies after the FP32 weights changed.
int refresh_wt(gabe_mlp *m) {
    if (m->f32act) return GABE_OK;
    tc::weights_bf16t_kernel<<<148, 256, 0, m->stream>>>(m->params, m->wt, m->wtab);
    MCK(m, cudaGetLastError());
    return GABE_OK;
}

template <int EPI>
int launch_tc(gabe_mlp *m, const tc::Args &a) {
    const dim3 grid((a.N + tc::BN - 1) / tc::BN, (a.M + tc::BM - 1) / tc::BM);
    MCK(m, cudaFuncSetAttribute(tc::gemm_tc_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)tc::SMEM_BYTES));
    tc::gemm_tc_kernel<EPI><<<grid, tc::T, tc::SMEM_BYTES, m->stream>>>(a);
    MCK(m, cudaGetLastError());
    return GABE_OK;
}

// cuTensorMapEncodeTiled, looked up once through the runtime (no link
// dependency on the driver library).
using EncodeTiledFn = CUresult (*)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *,
                                   const cuuint64_t *, const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q{};
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
            q != cudaDriverEntryPointSuccess) {
            cudaGetLastError();
            return (EncodeTiledFn) nullptr;
        }
        return reinterpret_cast<EncodeTiledFn>(p);
    }();
    return fn;
}

// 2-D BF16 tensor map of a row-major [rows][K] matrix, boxes of box_rows x 64
// with the 128-byte swizzle; rows beyond `rows` read as zeros.
bool encode_k_major(CUtensorMap *map, const bf16 *base, int K, int rows, int box_rows) {
    const EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)K * 2};
    const cuuint32_t box[2] = {(cuuint32_t)t5::BK, (cuuint32_t)box_rows};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<bf16 *>(base), dims, strides, box, estr,
              CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map of a row-major [rows][N] output (BF16 or FP32, esize bytes),
// boxes of 32 x 32 with the swizzle whose span is one box row (64 or 128
// bytes), as the epilogue lays its staging buffers out.
bool encode_out(CUtensorMap *map, void *base, int esize, int N, int rows) {
    const EncodeTiledFn fn = encode_fn();
    if (!fn) return false;
    const cuuint64_t dims[2] = {(cuuint64_t)N, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)N * esize};
    const cuuint32_t box[2] = {32, 32};
    const cuuint32_t estr[2] = {1, 1};
    return fn(map, esize == 2 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims,
              strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
              esize == 2 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_NONE,
              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Ring stages of the tcgen05 forward for a K x N layer on this device, 0 if
// the layer does not take it (shape, resident weights too large, no tensor
// map encoder).
int umma_stages_for(int dev, int K, int N, int esize) {
    if (K % t5::BK || K > 256 || N % 32 || N > 256 || !encode_fn()) return 0;
    int optin = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    const long long room = (long long)optin - (long long)t5::smem_bytes(N, K, 0, esize);
    const long long st = room / t5::kStageBytes;
    return st < 2 ? 0 : (int)(st > t5::kMaxStages ? t5::kMaxStages : st);
}

constexpr int kNoTensorMap = -1;  // launch_umma: no tensor map for these operands; use the mma.sync kernel

template <int EPI>
int launch_umma(gabe_mlp *m, const tc::Args &a, int stages) {
    CUtensorMap ma, mb, mc;
    if (!encode_k_major(&ma, a.A, a.K, a.M, t5::BM) || !encode_k_major(&mb, a.Wt, a.K, a.N, a.N) ||
        !encode_out(&mc, a.C, t5::out_bytes<EPI>(), a.N, a.M))
        return kNoTensorMap;  // e.g. an output pointer off a 16-byte boundary
    t5::Args g{a.M, a.N, a.K, stages, a.bias, a.Z, m->status};
    const size_t smem = t5::smem_bytes(a.N, a.K, stages, t5::out_bytes<EPI>());
    MCK(m, cudaFuncSetAttribute(t5::gemm_umma_kernel<EPI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int nsm = 0;
    MCK(m, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, m->dev));
    const int tiles = (a.M + t5::BM - 1) / t5::BM;
    const int grid = tiles < nsm ? tiles : nsm;
    t5::gemm_umma_kernel<EPI><<<grid, t5::NT, smem, m->stream>>>(ma, mb, mc, g);
    MCK(m, cudaGetLastError());
    return GABE_OK;
}

// The one-launch forward takes a network whose layers after the first all run on tcgen05 and whose first
// layer has the coalesced kernel's form; slots = weight slots that fit beside the activations (0: not taken).
int fused_slots_for(gabe_mlp *m) {
    const int W = m->p.width;
    if (m->nl < 2 || m->nl > t6::kMaxLayers || m->K[0] > kFirstMaxIn || W > 256 || 256 % (W / 8) != 0) return 0;
    for (int l = 1; l < m->nl; l++)
        if (!m->umma_stages[l]) return 0;
    int optin = 0;
    if (cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, m->dev) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    const long long s = ((long long)optin - (long long)t6::smem_bytes(W, 0)) / t6::kSlotBytes;
    if (s < 2) return 0;
    int rows = 0;
    for (int l = 1; l < m->nl; l++) rows += m->N[l];
    m->fused_box = m->p.n_out % 64 ? 32 : 64;  // divides every layer's columns
    if (!encode_k_major(&m->map_wt, m->wt, W, rows, m->fused_box)) return 0;
    return (int)(s > t6::kMaxSlots ? t6::kMaxSlots : s);
}

int launch_fused(gabe_mlp *m, const float *x, int rows, float *y, bool keep) {
    CUtensorMap my;
    if (!encode_out(&my, y, 4, m->p.n_out, rows)) return kNoTensorMap;
    t6::Args g{};
    g.M = rows;
    g.width = m->p.width;
    g.n_in = m->K[0];
    g.n_out = m->p.n_out;
    g.nl = m->nl;
    g.slots = m->fused_slots;
    g.box = m->fused_box;
    g.x = x;
    g.W0 = m->params + m->offW[0];
    for (int l = 0; l < m->nl; l++) {
        g.bias[l] = m->params + m->offb[l];
        g.rowoff[l] = l ? (int)(m->wtab.offWt[l] / m->p.width) : 0;
    }
    if (keep) {
        g.H = static_cast<bf16 *>(m->H);
        g.Z = static_cast<bf16 *>(m->Z);
        g.keep_stride = (long long)m->p.max_rows * m->p.width;
    }
    g.status = m->status;
    int nsm = 0;
    MCK(m, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, m->dev));
    const int tiles = (rows + t6::BM - 1) / t6::BM;
    g.tiles = tiles > nsm ? 2 : 1;
    const int groups = (tiles + g.tiles - 1) / g.tiles;
    const size_t smem = t6::smem_bytes(g.width, g.slots);
    auto kernel = g.n_in <= 4 ? (keep ? t6::mlp_kernel<true, 4> : t6::mlp_kernel<false, 4>)
                              : (keep ? t6::mlp_kernel<true, 8> : t6::mlp_kernel<false, 8>);
    MCK(m, cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    kernel<<<groups < nsm ? groups : nsm, t6::kThreadsPerCta, smem, m->stream>>>(m->map_wt, my, g);
    MCK(m, cudaGetLastError());
    return GABE_OK;
}

// Input activations of layer l: x (FP32) for l = 0, H[l-1] otherwise.
// With BF16 activations every layer after the first runs on tensor cores.
template <typename TACT>
int forward_rows(gabe_mlp *m, const float *x, int rows, float *y, bool keep_z) {
    // The one-launch form stores a tile's outputs while other tiles' inputs are still to be read: an output that
    // overlaps the inputs takes the layers, the first of which reads them all.
    const float *xe = x + (long long)rows * m->p.n_in, *ye = y + (long long)rows * m->p.n_out;
    if (m->fused_slots && (xe <= y || ye <= x)) {
        const int rc = launch_fused(m, x, rows, y, keep_z);
        if (rc != kNoTensorMap) return rc;  // else: e.g. an output pointer off a 16-byte boundary
    }
    for (int l = 0; l < m->nl; l++) {
        if (l == 0 && m->nl > 1 && m->K[0] <= kFirstMaxIn && 256 % (m->N[0] / 8) == 0) {
            launch_first_n<TACT>(m->K[0], x, rows, m->params + m->offW[0], m->params + m->offb[0], m->N[0],
                                 static_cast<TACT *>(act_at(m, m->H, 0)),
                                 keep_z ? static_cast<TACT *>(act_at(m, m->Z, 0)) : nullptr, m->stream);
            MCK(m, cudaGetLastError());
            continue;
        }
        if constexpr (sizeof(TACT) == 2) {
            if (l > 0) {
                tc::Args a{};
                a.M = rows;
                a.N = m->N[l];
                a.K = m->K[l];
                a.A = static_cast<const bf16 *>(act_at(m, m->H, l - 1));
                a.Wt = m->wt + m->wtab.offWt[l];
                a.bias = m->params + m->offb[l];
                const bool last = l + 1 == m->nl;
                a.Z = (!last && keep_z) ? static_cast<bf16 *>(act_at(m, m->Z, l)) : nullptr;
                a.C = last ? static_cast<void *>(y) : act_at(m, m->H, l);
                const int st = m->umma_stages[l];
                int rc = st ? (last ? launch_umma<EPI_OUT>(m, a, st) : launch_umma<EPI_HIDDEN>(m, a, st))
                            : kNoTensorMap;
                if (rc == kNoTensorMap) rc = last ? launch_tc<EPI_OUT>(m, a) : launch_tc<EPI_HIDDEN>(m, a);
                if (rc) return rc;
                continue;
            }
        }
        GemmArgs g{};
        g.M = rows;
        g.N = m->N[l];
        g.K = m->K[l];
        g.A = l == 0 ? static_cast<const void *>(x) : act_at(m, m->H, l - 1);
        g.sam = m->K[l];
        g.sak = 1;
        g.B = m->params + m->offW[l];
        g.sbk = m->N[l];
        g.sbn = 1;
        g.bias = m->params + m->offb[l];
        g.ldc = m->N[l];
        int rc;
        if (l + 1 < m->nl) {
            g.Z = keep_z ? act_at(m, m->Z, l) : nullptr;
            g.C = act_at(m, m->H, l);
            rc = l == 0 ? launch_gemm<float, TACT, EPI_HIDDEN>(m, g) : launch_gemm<TACT, TACT, EPI_HIDDEN>(m, g);
        } else {
            g.C = y;
            rc = l == 0 ? launch_gemm<float, TACT, EPI_OUT>(m, g) : launch_gemm<TACT, TACT, EPI_OUT>(m, g);
        }
        if (rc) return rc;
    }
    return GABE_OK;
}

// Gradients of the unnormalised loss sum (dy holds 2 (y - t) on finite
// targets) into m->grads.
template <typename TACT>
int backward_rows(gabe_mlp *m, const float *x, int rows) {
    float *delta = m->dy, *other = m->d0;
    for (int l = m->nl - 1; l >= 0; l--) {
        const int K = m->K[l], N = m->N[l];
        // dW_l = input^T delta
        GemmArgs w{};
        w.M = K;
        w.N = N;
        w.K = rows;
        w.A = l == 0 ? static_cast<const void *>(x) : act_at(m, m->H, l - 1);
        w.sam = 1;
        w.sak = K;
        w.B = delta;
        w.sbk = N;
        w.sbn = 1;
        w.C = m->ws;
        w.ldc = N;
        w.dbp = m->dbp;
        const int splits = weight_grad_splits(K, N, rows, &w.kchunk);
        int rc = l == 0 ? launch_gemm<float, TACT, EPI_BWD_WEIGHT>(m, w, splits)
                        : launch_gemm<TACT, TACT, EPI_BWD_WEIGHT>(m, w, splits);
        if (rc) return rc;
        splitk_reduce_kernel<<<148, 256, 0, m->stream>>>(m->ws, m->dbp, splits, (long long)K * N, N,
                                                         m->grads + m->offW[l], m->grads + m->offb[l]);
        MCK(m, cudaGetLastError());
        if (l == 0) break;
        // delta_{l-1} = (delta W_l^T) * SiLU'(Z_{l-1})
        GemmArgs d{};
        d.M = rows;
        d.N = K;
        d.K = N;
        d.A = delta;
        d.sam = N;
        d.sak = 1;
        d.B = m->params + m->offW[l];
        d.sbk = 1;
        d.sbn = N;
        d.Z = act_at(m, m->Z, l - 1);
        d.C = other;
        d.ldc = K;
        if ((rc = launch_gemm<float, TACT, EPI_BWD_DATA>(m, d))) return rc;
        delta = other;
        other = (other == m->d0) ? m->d1 : m->d0;
    }
    return GABE_OK;
}

// A small batch's backward: the data gradients layer by layer, then every weight gradient in one launch, then
// (step) the AdamW step and the BF16 weights, or (!step) the normalised gradients, in another.
template <typename TACT>
int backward_small(gabe_mlp *m, const float *x, int rows, bool step) {
    const int nl = m->nl;
    std::vector<const float *> delta(nl);
    delta[nl - 1] = m->dy;
    for (int l = nl - 1; l > 0; l--) {
        const int K = m->K[l], N = m->N[l];
        float *out = m->small_delta + (size_t)(l - 1) * m->small_rows * m->p.width;
        if (N % 4 == 0) {
            const dim3 grid((K + kDgTile - 1) / kDgTile, (rows + kDgTile - 1) / kDgTile);
            MCK(m, cudaFuncSetAttribute(data_grad_kernel<TACT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kDgSmem));
            data_grad_kernel<TACT><<<grid, kDgT, kDgSmem, m->stream>>>(
                delta[l], m->params + m->offW[l], static_cast<const TACT *>(act_at(m, m->Z, l - 1)), out, rows, K, N);
            MCK(m, cudaGetLastError());
        } else {
            GemmArgs d{};
            d.M = rows;
            d.N = K;
            d.K = N;
            d.A = delta[l];
            d.sam = N;
            d.sak = 1;
            d.B = m->params + m->offW[l];
            d.sbk = 1;
            d.sbn = N;
            d.Z = act_at(m, m->Z, l - 1);
            d.C = out;
            d.ldc = K;
            const int rc = launch_gemm<float, TACT, EPI_BWD_DATA>(m, d);
            if (rc) return rc;
        }
        delta[l - 1] = out;
    }
    WeightGradArgs w{};
    UpdateArgs u{};
    w.nl = u.nl = nl;
    int wb = 0, ub = 0;
    for (int l = 0; l < nl; l++) {
        const int K = m->K[l], N = m->N[l];
        GemmArgs &g = w.g[l];
        g.M = K;
        g.N = N;
        g.K = rows;
        g.A = l == 0 ? static_cast<const void *>(x) : act_at(m, m->H, l - 1);
        g.sam = 1;
        g.sak = K;
        g.B = delta[l];
        g.sbk = N;
        g.sbn = 1;
        u.splits[l] = weight_grad_splits(K, N, rows, &g.kchunk);
        g.C = m->small_ws + m->small_off[2 * l];
        g.ldc = N;
        g.dbp = m->small_ws + m->small_off[2 * l + 1];
        w.first[l] = wb;
        wb += ((K + BM - 1) / BM) * ((N + BN - 1) / BN) * u.splits[l];
        u.K[l] = K;
        u.N[l] = N;
        u.offW[l] = m->offW[l];
        u.offb[l] = m->offb[l];
        u.offWt[l] = m->wtab.offWt[l];
        u.ws[l] = static_cast<const float *>(g.C);
        u.dbp[l] = g.dbp;
        u.first[l] = ub;
        ub += ((K + 31) / 32) * ((N + 31) / 32) + (N + 255) / 256;
    }
    weight_grad_kernel<TACT><<<wb, kThreads, 0, m->stream>>>(w);
    MCK(m, cudaGetLastError());
    u.p = m->params;
    u.m = m->mom;
    u.v = m->vel;
    u.grads = m->grads;
    u.wt = m->f32act ? nullptr : m->wt;
    u.h = AdamHyper{m->p.lr, m->p.beta1, m->p.beta2, m->p.eps, m->p.weight_decay, m->p.lr_min, m->p.decay_steps};
    u.ts = m->ts;
    if (step) update_kernel<false><<<ub, 256, 0, m->stream>>>(u);
    else update_kernel<true><<<ub, 256, 0, m->stream>>>(u);
    MCK(m, cudaGetLastError());
    return GABE_OK;
}

int bwd_small(gabe_mlp *m, const float *x, int rows, bool step) {
    return m->f32act ? backward_small<float>(m, x, rows, step) : backward_small<bf16>(m, x, rows, step);
}

int fwd(gabe_mlp *m, const float *x, int rows, float *y, bool keep_z) {
    return m->f32act ? forward_rows<float>(m, x, rows, y, keep_z) : forward_rows<bf16>(m, x, rows, y, keep_z);
}

int bwd(gabe_mlp *m, const float *x, int rows) {
    return m->f32act ? backward_rows<float>(m, x, rows) : backward_rows<bf16>(m, x, rows);
}

int train_step(gabe_mlp *m, const float *x, const float *t, const int32_t *perm, int B) {
    const int nin = m->p.n_in, nout = m->p.n_out;
    gather_kernel<<<148, 256, 0, m->stream>>>(x, t, perm, m->ts, B, nin, nout, m->xb, m->tb);
    MCK(m, cudaGetLastError());
    int rc = fwd(m, m->xb, B, m->y, true);
    if (rc) return rc;
    loss_kernel<<<kLossBlocks, 256, 0, m->stream>>>(m->y, m->tb, (long long)B * nout, m->dy, m->part, m->ts, 1);
    MCK(m, cudaGetLastError());
    if (B <= m->small_rows) return bwd_small(m, m->xb, B, true);
    if ((rc = bwd(m, m->xb, B))) return rc;
    AdamHyper h{m->p.lr, m->p.beta1, m->p.beta2, m->p.eps, m->p.weight_decay, m->p.lr_min, m->p.decay_steps};
    adam_kernel<<<148 * 4, 256, 0, m->stream>>>(m->params, m->grads, m->mom, m->vel, m->P, h, m->ts);
    MCK(m, cudaGetLastError());
    return refresh_wt(m);
}

uint64_t splitmix(uint64_t &s) {
    uint64_t z = (s += 0x9E3779B97F4A7C15ull);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    return z ^ (z >> 31);
}

void free_all(gabe_mlp *m) {
    if (m->gexec) cudaGraphExecDestroy(m->gexec);
    if (m->graph) cudaGraphDestroy(m->graph);
    void *bufs[] = {m->params, m->grads, m->mom, m->vel, m->xb, m->tb, m->y, m->dy, m->d0, m->d1, m->Z, m->H,
                    m->part, m->ts, m->ws, m->dbp, m->wt, m->status, m->small_delta, m->small_ws};
    for (void *b : bufs)
        if (b) cudaFree(b);
    if (m->stream) cudaStreamDestroy(m->stream);
}

}  // namespace

extern "C" {

void gabe_mlp_default_params(gabe_mlp_params *p) {
    if (!p) return;
    std::memset(p, 0, sizeof(*p));
    p->struct_size = sizeof(gabe_mlp_params);
    p->n_in = 3;
    p->width = 256;
    p->depth = 4;
    p->n_out = 192;
    p->max_rows = 65536;
    p->lr = 1e-3f;
    p->beta1 = 0.9f;
    p->beta2 = 0.999f;
    p->eps = 1e-8f;
    p->weight_decay = 0.f;
    p->lr_min = 0.f;
    p->decay_steps = 0;
    p->seed = 1;
    p->device = -1;
}

int gabe_mlp_create(const gabe_mlp_params *p, gabe_mlp **out) {
    if (!out) return mset(nullptr, GABE_ERR_PARAM, "out is NULL");
    *out = nullptr;
    if (!p || p->struct_size != (int32_t)sizeof(gabe_mlp_params)) return mset(nullptr, GABE_ERR_PARAM, "bad gabe_mlp_params");
    if (p->n_in < 1 || p->n_in > 64 || p->width < 64 || p->width > 4096 || p->width % 64 || p->depth < 1 ||
        p->depth > 16 || p->n_out < 1 || p->n_out > 4096 || p->max_rows < 1 || p->max_rows > (1 << 21))
        return mset(nullptr, GABE_ERR_PARAM, "invalid MLP shape");
    if (!(p->lr >= 0) || !(p->beta1 >= 0 && p->beta1 < 1) || !(p->beta2 >= 0 && p->beta2 < 1) || !(p->eps > 0) ||
        !(p->weight_decay >= 0) || !(p->lr_min >= 0) || p->decay_steps < 0)
        return mset(nullptr, GABE_ERR_PARAM, "invalid optimiser parameters");
    gabe_mlp *m = new (std::nothrow) gabe_mlp();
    if (!m) return mset(nullptr, GABE_ERR_NOMEM, "host allocation failed");
    m->p = *p;
    m->f32act = (p->flags & GABE_MLP_FP32_ACT) != 0;
    m->nl = p->depth + 1;
    long long nwt = 0;
    m->wtab.nl = m->nl;
    for (int l = 0; l < m->nl; l++) {
        m->K.push_back(l == 0 ? p->n_in : p->width);
        m->N.push_back(l + 1 == m->nl ? p->n_out : p->width);
        m->offW.push_back(m->P);
        m->wtab.offW[l] = m->P;
        m->wtab.K[l] = m->K[l];
        m->wtab.N[l] = m->N[l];
        m->wtab.offWt[l] = nwt;
        if (l > 0) nwt += (long long)m->K[l] * m->N[l];
        m->P += (long long)m->K[l] * m->N[l];
        m->offb.push_back(m->P);
        m->P += m->N[l];
    }
    auto fail = [&](int code) {
        g_mlp_create_error = m->err;
        free_all(m);
        delete m;
        return code;
    };
    if (p->device >= 0 && cudaSetDevice(p->device) != cudaSuccess) {
        cudaGetLastError();
        mset(m, GABE_ERR_CUDA, "cudaSetDevice(%d) failed", p->device);
        return fail(GABE_ERR_CUDA);
    }
    if (cudaGetDevice(&m->dev) != cudaSuccess || cudaStreamCreateWithFlags(&m->stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        mset(m, GABE_ERR_CUDA, "no CUDA device");
        return fail(GABE_ERR_CUDA);
    }
    const size_t R = p->max_rows, W = p->width, A = act_size(m);
    const size_t wide = (size_t)(p->n_out > p->width ? p->n_out : p->width);
    long long small_ws = 0;
    for (int l = 0; l < m->nl; l++) {
        const long long splits = most_splits(m->K[l], m->N[l]);
        m->small_off.push_back(small_ws);
        small_ws += splits * m->K[l] * m->N[l];
        m->small_off.push_back(small_ws);
        small_ws += splits * m->N[l];
    }
    struct {
        void **ptr;
        size_t bytes;
    } allocs[] = {
        {(void **)&m->params, (size_t)m->P * 4}, {(void **)&m->grads, (size_t)m->P * 4},
        {(void **)&m->mom, (size_t)m->P * 4},    {(void **)&m->vel, (size_t)m->P * 4},    {(void **)&m->xb, R * p->n_in * 4}, {(void **)&m->tb, R * p->n_out * 4},
        {(void **)&m->y, R * p->n_out * 4}, {(void **)&m->dy, R * p->n_out * 4}, {(void **)&m->d0, R * wide * 4},
        {(void **)&m->d1, R * wide * 4}, {&m->Z, (size_t)p->depth * R * W * A}, {&m->H, (size_t)p->depth * R * W * A},
        {(void **)&m->part, kLossBlocks * sizeof(double2)}, {(void **)&m->ts, sizeof(TrainScalars)},
        {(void **)&m->ws, (size_t)kMaxSplits * wide * wide * 4}, {(void **)&m->dbp, (size_t)kMaxSplits * wide * 4},
        {(void **)&m->wt, (size_t)(nwt > 0 ? nwt : 1) * sizeof(bf16)}, {(void **)&m->status, sizeof(unsigned int)},
    };
    for (auto &a : allocs) {
        if (cudaMalloc(a.ptr, a.bytes) != cudaSuccess) {
            cudaGetLastError();
            mset(m, GABE_ERR_NOMEM, "cudaMalloc(%zu bytes) failed", a.bytes);
            return fail(GABE_ERR_NOMEM);
        }
    }
    const long long row_bytes = (long long)p->depth * p->width * 4, fit = (kSmallBytes - small_ws * 4) / row_bytes;
    long long small_rows = p->max_rows < kSmallRows ? p->max_rows : kSmallRows;
    if (small_rows > fit) small_rows = fit;
    if (small_rows > 0) {
        if (cudaMalloc((void **)&m->small_delta, (size_t)(small_rows * row_bytes)) == cudaSuccess &&
            cudaMalloc((void **)&m->small_ws, (size_t)small_ws * 4) == cudaSuccess) {
            m->small_rows = (int)small_rows;
        } else {  // every batch takes the kernels of the large ones
            cudaGetLastError();
            if (m->small_delta) cudaFree(m->small_delta);
            m->small_delta = m->small_ws = nullptr;
        }
    }
    // Glorot-uniform weights, zero biases, from the seed
    std::vector<float> h(m->P, 0.f);
    uint64_t s = p->seed;
    for (int l = 0; l < m->nl; l++) {
        const double a = std::sqrt(6.0 / (m->K[l] + m->N[l]));
        for (long long i = 0; i < (long long)m->K[l] * m->N[l]; i++) {
            const double u = (double)(splitmix(s) >> 11) * (1.0 / 9007199254740992.0);
            h[m->offW[l] + i] = (float)((2. * u - 1.) * a);
        }
    }
    TrainScalars ts{};
    if (cudaMemcpyAsync(m->params, h.data(), m->P * 4, cudaMemcpyHostToDevice, m->stream) != cudaSuccess ||
        cudaMemsetAsync(m->mom, 0, m->P * 4, m->stream) != cudaSuccess ||
        cudaMemsetAsync(m->vel, 0, m->P * 4, m->stream) != cudaSuccess ||
        cudaMemcpyAsync(m->ts, &ts, sizeof(ts), cudaMemcpyHostToDevice, m->stream) != cudaSuccess ||
        cudaMemsetAsync(m->status, 0, sizeof(unsigned int), m->stream) != cudaSuccess ||
        refresh_wt(m) != GABE_OK || cudaStreamSynchronize(m->stream) != cudaSuccess) {
        cudaGetLastError();
        mset(m, GABE_ERR_CUDA, "initialisation copies failed");
        return fail(GABE_ERR_CUDA);
    }
    // tcgen05 forward for the BF16 layers whose weights fit in shared memory
    if (!m->f32act && !(p->flags & GABE_MLP_MMA_SYNC))
        for (int l = 1; l < m->nl; l++)
            m->umma_stages[l] = umma_stages_for(m->dev, m->K[l], m->N[l], l + 1 == m->nl ? 4 : 2);
    m->fused_slots = fused_slots_for(m);
    *out = m;
    return GABE_OK;
}

int gabe_mlp_destroy(gabe_mlp *m) {
    if (!m) return GABE_OK;
    cudaSetDevice(m->dev);
    if (m->stream) cudaStreamSynchronize(m->stream);
    free_all(m);
    delete m;
    return GABE_OK;
}

int64_t gabe_mlp_num_params(const gabe_mlp *m) { return m ? m->P : 0; }

int gabe_mlp_set_params(gabe_mlp *m, const float *h_params) {
    if (!m || !h_params) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    MCK(m, cudaMemcpyAsync(m->params, h_params, m->P * 4, cudaMemcpyHostToDevice, m->stream));
    int rc = refresh_wt(m);
    if (rc) return rc;
    MCK(m, cudaStreamSynchronize(m->stream));
    return GABE_OK;
}

int gabe_mlp_get_params(gabe_mlp *m, float *h_params) {
    if (!m || !h_params) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    MCK(m, cudaMemcpyAsync(h_params, m->params, m->P * 4, cudaMemcpyDeviceToHost, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    return GABE_OK;
}

int gabe_mlp_forward(gabe_mlp *m, const float *x, int64_t n, float *y) {
    if (!m || n < 0 || (n > 0 && (!x || !y))) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    for (int64_t r0 = 0; r0 < n; r0 += m->p.max_rows) {
        const int rows = (int)((n - r0) < m->p.max_rows ? (n - r0) : m->p.max_rows);
        int rc = fwd(m, x + r0 * m->p.n_in, rows, y + r0 * m->p.n_out, false);
        if (rc) return rc;
    }
    return GABE_OK;
}

int gabe_mlp_loss_grad(gabe_mlp *m, const float *x, const float *t, int64_t n, double *h_loss, float *h_grad) {
    if (!m || !x || !t || n < 1 || n > m->p.max_rows || !h_loss) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    const int rows = (int)n;
    int rc = fwd(m, x, rows, m->y, true);
    if (rc) return rc;
    loss_kernel<<<kLossBlocks, 256, 0, m->stream>>>(m->y, t, (long long)rows * m->p.n_out, m->dy, m->part, m->ts, 0);
    MCK(m, cudaGetLastError());
    if (h_grad) {
        if (rows <= m->small_rows) {
            if ((rc = bwd_small(m, x, rows, false))) return rc;
        } else {
            if ((rc = bwd(m, x, rows))) return rc;
            scale_kernel<<<148, 256, 0, m->stream>>>(m->grads, m->P, m->ts);
            MCK(m, cudaGetLastError());
        }
        MCK(m, cudaMemcpyAsync(h_grad, m->grads, m->P * 4, cudaMemcpyDeviceToHost, m->stream));
    }
    TrainScalars ts;
    MCK(m, cudaMemcpyAsync(&ts, m->ts, sizeof(ts), cudaMemcpyDeviceToHost, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    *h_loss = ts.loss_last;
    return GABE_OK;
}

int gabe_mlp_train(gabe_mlp *m, const float *x, const float *t, const int32_t *perm, int32_t batch, int32_t nbatch) {
    if (!m || !x || !t || !perm || batch < 1 || batch > m->p.max_rows || nbatch < 0) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    m->batch = batch;
    if (!(m->p.flags & GABE_MLP_NO_GRAPH) &&
        (!m->gexec || m->g_x != x || m->g_t != t || m->g_perm != perm || m->g_batch != batch)) {
        if (m->gexec) cudaGraphExecDestroy(m->gexec);
        if (m->graph) cudaGraphDestroy(m->graph);
        m->gexec = nullptr;
        m->graph = nullptr;
        MCK(m, cudaStreamBeginCapture(m->stream, cudaStreamCaptureModeThreadLocal));
        int rc = train_step(m, x, t, perm, batch);
        cudaGraph_t g = nullptr;
        cudaError_t e = cudaStreamEndCapture(m->stream, &g);
        if (rc || e != cudaSuccess) {
            if (g) cudaGraphDestroy(g);
            cudaGetLastError();
            return rc ? rc : mset(m, GABE_ERR_CUDA, "capture of the training step failed: %s", cudaGetErrorString(e));
        }
        m->graph = g;
        MCK(m, cudaGraphInstantiate(&m->gexec, g, 0));
        m->g_x = x;
        m->g_t = t;
        m->g_perm = perm;
        m->g_batch = batch;
    }
    for (int s = 0; s < nbatch; s++) {
        if (m->gexec) MCK(m, cudaGraphLaunch(m->gexec, m->stream));
        else {
            int rc = train_step(m, x, t, perm, batch);
            if (rc) return rc;
        }
    }
    return GABE_OK;
}

int gabe_mlp_set_schedule(gabe_mlp *m, float lr, float lr_min, int32_t decay_steps) {
    if (!m || !(lr >= 0) || !(lr_min >= 0) || decay_steps < 0) return GABE_ERR_PARAM;
    m->p.lr = lr;
    m->p.lr_min = lr_min;
    m->p.decay_steps = decay_steps;
    // the captured step holds the hyper-parameters by value
    if (m->gexec) cudaGraphExecDestroy(m->gexec);
    if (m->graph) cudaGraphDestroy(m->graph);
    m->gexec = nullptr;
    m->graph = nullptr;
    return GABE_OK;
}

int gabe_mlp_reset_batches(gabe_mlp *m) {
    if (!m) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    MCK(m, cudaMemsetAsync(&m->ts->batch_idx, 0, sizeof(long long), m->stream));
    return GABE_OK;
}

int gabe_mlp_train_loss(gabe_mlp *m, double *h_mean_loss, int64_t *h_steps) {
    if (!m) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    TrainScalars ts;
    MCK(m, cudaMemcpyAsync(&ts, m->ts, sizeof(ts), cudaMemcpyDeviceToHost, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    if (h_mean_loss) *h_mean_loss = ts.loss_n ? ts.loss_sum / (double)ts.loss_n : 0.;
    if (h_steps) *h_steps = ts.step;
    const double zero = 0.;
    const long long zn = 0;
    MCK(m, cudaMemcpyAsync(&m->ts->loss_sum, &zero, sizeof(zero), cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaMemcpyAsync(&m->ts->loss_n, &zn, sizeof(zn), cudaMemcpyHostToDevice, m->stream));
    MCK(m, cudaStreamSynchronize(m->stream));
    return GABE_OK;
}

int gabe_mlp_sync(gabe_mlp *m) {
    if (!m) return GABE_ERR_PARAM;
    MCK(m, cudaSetDevice(m->dev));
    MCK(m, cudaStreamSynchronize(m->stream));
    unsigned int st = 0;
    MCK(m, cudaMemcpy(&st, m->status, sizeof(st), cudaMemcpyDeviceToHost));
    if (st) return mset(m, GABE_ERR_TIMEOUT, "a bounded wait of the tensor-core forward gave up (status %u)", st);
    return GABE_OK;
}

int gabe_mlp_forward_form(const gabe_mlp *m, int32_t layer) {
    if (!m || layer < 0 || layer >= m->nl) return -1;
    if (layer == 0 || m->f32act) return 0;
    return m->umma_stages[layer] ? 2 : 1;
}

void *gabe_mlp_stream(const gabe_mlp *m) { return m ? (void *)m->stream : nullptr; }

int gabe_mlp_launches_per_train_step(const gabe_mlp *m) {
    if (!m) return 0;
    const int n = 2 + (m->fused_slots ? 1 : m->nl) + (m->nl - 1);  // gather, forward, loss, data gradients
    if (m->batch <= m->small_rows) return n + 2;                   // weight gradients, update
    return n + 2 * m->nl + 1 + (m->f32act ? 0 : 1);                // ... and reductions, update, BF16 weights
}


int gabe_mlp_launches_per_forward(const gabe_mlp *m) {
    return m ? (m->fused_slots ? 1 : m->nl) : 0;
}

const char *gabe_mlp_last_error(const gabe_mlp *m) { return m ? m->err.c_str() : g_mlp_create_error.c_str(); }

}  // extern "C"
