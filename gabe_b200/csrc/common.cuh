// Shared device-side definitions for the GABE sm_100a kernels.
//
// State layout in HBM (per handle):
//   fields   X[buf][fld][i][j][k]     (k fastest; two ping-pong buffers)
//   momenta  D[buf][fld][i][j][k]
//   GW       h[12][i][j][kz], l[12][i][j][kz]   planar, kz < N/2+1
//   sources  S[10][i][j][row]  real: 11,12,13,22,23 of stage 0, then of
//            stage 1; rows of N + 2 (an in-place r2c then leaves the half
//            spectra S^[10][i][j][kz] in the same bytes) or, FP32, of N
//            (SrcLayout in stencil.cuh)
//   scalars  DevScalars (a, adot, energies per stage, homogeneous
//            trajectory of the FP32 path, status word)
//   partials per-block FP64 sums of the energy reductions
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace gabe {

// Status bits raised on the device and read by the host at sync points.
enum : uint32_t {
    ST_NONFINITE = 1u,
    ST_TIMEOUT = 2u,  // a bounded wait on a bulk copy gave up (tma.cuh)
};

// Per-stage scalars, laid out like the reference's globals
// a[2], adot[2], edkin[2], edpot[2], edgrad[2], edrho[2] (g2header.h:58-63).
struct DevScalars {
    double a[2], adot[2], edkin[2], edpot[2], edgrad[2], edrho[2];
    // FP32 path: homogeneous trajectory (fields and momenta) at stage 0.
    double fbar[2], dfbar[2];
    long long step;
    unsigned int status;
    unsigned int adot_given;  // adot[0] came from the caller (after an upload), not from adf(0)
    // a[0], adot[0], a[1], adot[1] of the step whose GW sources sit in source
    // buffer s, for the k-space update (which may run while the fields are
    // already one step further on)
    double gw[2][4];
};

enum Model : int { MODEL_QUADRATIC = 0, MODEL_LPHI4 = 1 };

// Constants of one lattice, computed on the host with the same sequence of
// IEEE operations the reference's compiler folds (so FP64 results agree
// bit for bit where the reference's operation order is kept).
struct LatticeConsts {
    int N;
    int model;
    int expansion;          // expansion_type: 0 none, 1 Friedmann, 2 Friedmann without tensor modes
    double dt, half_dt;     // dt, .5*dt
    double dx;              // L/((double)N) (g2parameters.h:93)
    double inv_dx2_div;     // dx*dx (the reference divides by it)
    double dn, c13, c23;    // 1/(dx*dx), (1./3.)*dn, (2./3.)*dn  (g2evolutionpert.cpp:53-116)
    double mc[5];           // model constants (see model_consts on the host)
    double gridsize;        // N^3
    double eight_pi_3;      // 8.*M_PI/3.
    double k2norm_c;        // 4.*M_PI*M_PI/L/L
    double eight_pi;        // 8.*M_PI
    double normmm;          // pow(dx,3)
};

__host__ __device__ inline int wrapi(int x, int N) { return x < 0 ? x + N : (x >= N ? x - N : x); }

// ---------------------------------------------------------------------------
// FP64 model, reference operation order (g2model.cpp:66-87 for the shipped
// model; oracle/ref_cfg/g2model_lphi4.cpp order for lambda phi^4).
// ---------------------------------------------------------------------------
__device__ __forceinline__ double pot64(const LatticeConsts &c, double P, double C) {
    if (c.model == MODEL_QUADRATIC) return (0.5 * P * P + c.mc[1] * P * P * C * C);
    return c.mc[2] * P * P * P * P + c.mc[3] * P * P * C * C;
}
__device__ __forceinline__ double dv64(const LatticeConsts &c, int fld, double P, double C) {
    if (c.model == MODEL_QUADRATIC) {
        if (fld == 0) return (P + c.mc[0] * C * C * P);
        return (c.mc[0] * P * P * C);
    }
    if (fld == 0) return c.mc[0] * P * P * P + c.mc[1] * C * C * P;
    return c.mc[1] * P * P * C;
}

// ---------------------------------------------------------------------------
// FP32 fluctuation model: differences V(fbar+d) - V(fbar) and
// V'(fbar+d) - V'(fbar) expanded so that no term cancels (pb, cb = homogeneous
// phi, chi; a, b = their fluctuations).
// ---------------------------------------------------------------------------
// Two FP32 values in one register pair, worked on by the packed FP32 units of
// sm_100 (one instruction for both halves, each half rounded as the scalar
// instruction rounds).  Multiply-adds are written out: nothing is contracted
// across the packed instructions.
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 f2(float x, float y) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ F2 f2(float x) { return f2(x, x); }
__device__ __forceinline__ float2 unpack(F2 a) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a.v));
    return r;
}
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator*(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) { return fma2(b, f2(-1.f), a); }
__device__ __forceinline__ double sum2(F2 a) {
    const float2 r = unpack(a);
    return (double)r.x + (double)r.y;
}

// The homogeneous values and model constants as pairs, as the site functions
// use them.
struct alignas(16) MeanP {
    F2 pb, cb, cb2, pb2, pbsq, pbcb;    // phi, chi, 2 chi, 2 phi, phi^2, phi chi
    F2 pbt, pb3sq;                      // 3 phi, 3 phi^2
    F2 pb4, pb6sq, pb4cu, pad;          // 4 phi, 6 phi^2, 4 phi^3
};
struct alignas(16) ModelP {
    F2 n0, n1, q1, q2, q3, half;        // -mc[0], -mc[1], mc[1], mc[2], mc[3], 1/2
};
__device__ __forceinline__ MeanP mean_p(const double *fb) {
    const double p = fb[0], c = fb[1];
    auto k = [](double x) { return f2((float)x); };
    return MeanP{k(p),      k(c),          k(2. * c),      k(2. * p),          k(p * p), k(p * c), k(3. * p),
                 k(3. * p * p), k(4. * p), k(6. * p * p), k(4. * p * p * p), f2(0.f)};
}
__device__ __forceinline__ ModelP model_p(const LatticeConsts &c) {
    auto k = [](double x) { return f2((float)x); };
    return ModelP{k(-c.mc[0]), k(-c.mc[1]), k(c.mc[1]), k(c.mc[2]), k(c.mc[3]), f2(0.5f)};
}

// Takes V'(fbar+d) - V'(fbar) of both fields off t (SET: off zero).
template <bool SET>
__device__ __forceinline__ void sub_dv_diff32(const MeanP &m, const ModelP &q, int model, F2 a, F2 b, F2 (&t)[2]) {
    const F2 C = m.cb + b;
    const F2 u = fma2(a, C * C, (m.pb * b) * (m.cb2 + b));  // pb b (2 cb + b) + a C^2
    const F2 w = fma2(a * (m.pb2 + a), C, m.pbsq * b);
    if (model == MODEL_QUADRATIC) {
        // V' = phi + C1 chi^2 phi ; V'_chi = C1 phi^2 chi
        t[0] = (SET ? q.n0 * u : fma2(q.n0, u, t[0])) - a;
        t[1] = SET ? q.n0 * w : fma2(q.n0, w, t[1]);
    } else {
        // V' = lam phi^3 + g chi^2 phi ; V'_chi = g phi^2 chi
        t[0] = fma2(q.n0 * a, fma2(a, m.pbt + a, m.pb3sq), SET ? q.n1 * u : fma2(q.n1, u, t[0]));
        t[1] = SET ? q.n1 * w : fma2(q.n1, w, t[1]);
    }
}

// V(fbar+d) - V(fbar).
__device__ __forceinline__ F2 v_diff32(const MeanP &m, const ModelP &q, int model, F2 a, F2 b) {
    const F2 cross = fma2(a, b, fma2(m.cb, a, m.pb * b)) * fma2(m.pb + a, m.cb + b, m.pbcb);
    if (model == MODEL_QUADRATIC) return fma2(q.q1, cross, a * fma2(q.half, a, m.pb));
    const F2 quart = fma2(a, fma2(a, m.pb4 + a, m.pb6sq), m.pb4cu);
    return fma2(q.q2 * a, quart, q.q3 * cross);
}

// Homogeneous potential and force in FP64 (for the FP32 path's mean).
__host__ __device__ inline double pot_h(int model, const double *mc, double P, double C) {
    if (model == MODEL_QUADRATIC) return 0.5 * P * P + mc[1] * P * P * C * C;
    return mc[2] * P * P * P * P + mc[3] * P * P * C * C;
}
__host__ __device__ inline double dv_h(int model, const double *mc, int fld, double P, double C) {
    if (model == MODEL_QUADRATIC) return fld == 0 ? P + mc[0] * C * C * P : mc[0] * P * P * C;
    return fld == 0 ? mc[0] * P * P * P + mc[1] * C * C * P : mc[1] * P * P * C;
}

// ---------------------------------------------------------------------------
// block reduction of NV doubles; result valid in thread 0
// ---------------------------------------------------------------------------
// Sum over the lanes of this warp that exist (blocks need not be a multiple
// of 32 threads); the total lands in lane 0.
__device__ __forceinline__ double warp_sum(double x, int nlanes) {
    const unsigned mask = nlanes >= 32 ? 0xffffffffu : ((1u << nlanes) - 1u);
    const int lane = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double y = __shfl_down_sync(mask, x, o);
        if ((lane & 31) + o < nlanes) x += y;
    }
    return x;
}

template <int NV>
__device__ __forceinline__ void block_reduce(double (&v)[NV], double *sred) {
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    const int lane = tid & 31, warp = tid >> 5, nwarp = (nthr + 31) >> 5;
    const int my_lanes = (warp == nwarp - 1) ? nthr - 32 * warp : 32;
#pragma unroll
    for (int q = 0; q < NV; q++) v[q] = warp_sum(v[q], my_lanes);
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < NV; q++) sred[warp * NV + q] = v[q];
    __syncthreads();
    if (warp == 0) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            double x = lane < nwarp ? sred[lane * NV + q] : 0.0;
            v[q] = warp_sum(x, my_lanes);
        }
    }
    __syncthreads();
}

// Deterministic sum of nblk partial vectors (stride NV) by one block, with
// compensated accumulation per thread; result valid in thread 0.
template <int NV>
__device__ __forceinline__ void sum_partials(const double *partials, int nblk, double (&out)[NV], double *sred) {
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const int nthr = blockDim.x * blockDim.y * blockDim.z;
    double s[NV], comp[NV];
#pragma unroll
    for (int q = 0; q < NV; q++) { s[q] = 0.0; comp[q] = 0.0; }
    for (int b = tid; b < nblk; b += nthr) {
#pragma unroll
        for (int q = 0; q < NV; q++) {
            double y = __ldcg(partials + (size_t)b * NV + q) - comp[q];
            double t = s[q] + y;
            comp[q] = (t - s[q]) - y;
            s[q] = t;
        }
    }
    block_reduce<NV>(s, sred);
#pragma unroll
    for (int q = 0; q < NV; q++) out[q] = s[q];
}

// Returns true in every thread of the block that finished last.
__device__ __forceinline__ bool last_block_done(unsigned int *counter, int *sflag) {
    const int tid = threadIdx.x + blockDim.x * (threadIdx.y + blockDim.y * threadIdx.z);
    const unsigned int total = gridDim.x * gridDim.y * gridDim.z;
    __threadfence();
    __syncthreads();
    if (tid == 0) {
        unsigned int prev = atomicAdd(counter, 1u);
        *sflag = (prev == total - 1) ? 1 : 0;
    }
    __syncthreads();
    bool last = *sflag != 0;
    if (last) __threadfence();
    return last;
}

}  // namespace gabe
