// |k|-binned power spectra (specOut, g2spectra.cpp:23-234).
//
// One pass over the half spectrum accumulates, per native bin
// b = (int)|n| (g2spectra.cpp:74-89), the weighted power of both fields
// (weight 2 for 0 < kz < N/2, 1 on the kz = 0 and kz = N/2 planes) and of
// the GW momenta l with the reference's component weights (:133-144).  With
// gw_spec_quirk the kz = 0 plane reads l at kz = N/2, as the reference's
// loop does (:149-164, k is left at N/2 by the preceding loop).  Sums are
// FP64: per-block shared-memory histograms, then a fixed-order reduction
// over blocks.  Normalisation to the file columns happens on the host.
//
// What bounds it is the update of the histograms, not the read of the
// spectrum: neighbouring points of a line fall into the same bin, so one
// shared FP64 atomic per point serialises the lanes of a warp.  A lane first
// adds up the points that differ only in the signs of kx and ky, a warp then
// sums the runs of equal bins of its 32 lanes by shuffles, and only the first
// lane of a run updates the histogram.  Each array is read in its
// own storage order: amplitudes kept transposed ([kz][ky][kx]) have their
// own loop instead of a strided read per point of the fields' loop.
// Measured (B200, both fields and l): 512^3 FP32 0.73 ms against 3.04 with an
// atomic per point, 256^3 FP64 0.108 against 0.315 (its 0.54 GB take 0.083 at
// the copy rate); 512^3 with one point per lane and 16 warps per SM 2.1.
#pragma once

#include "common.cuh"
#include "kspace.cuh"

namespace gabe {

struct BinArgs {
    const void *F;          // complex field spectra, 2 slots [2][N][N][N/2+1]
    const void *G;          // GW amplitudes [4][N][N][N/2+1] complex (h+, hx, l+, lx) or null
    double *part_sum;       // [nblocks][nseries][nbins]
    unsigned int *part_cnt; // [nblocks][nbins]
    int N, nbins, nseries, quirk;
    double zero_re[2];      // FP32 path: N^3 fbar per field, added to F(k=0) of the fluctuations
    int fix_zero;
    // a slab's k-points (slab.cu): F and G hold [..][N][m][N/2+1] with ky = y0 + y; m = 0: all of them
    int m, y0;
    int gt;                 // order of G (g_index); 1 and 2 for whole lattices only
};

// |n| of an integer wave vector, rounded down.  n2 <= 3 (N/2)^2 < 2^24 is
// exact in FP32, and the rounding of sqrtf cannot reach the next integer
// (sqrt(m^2 - 1) lies 1 / 2m below m, above half a spacing for m < 2048).
__device__ __forceinline__ int native_bin(int px, int py, int pz) {
    return (int)sqrtf((float)(px * px + py * py + pz * pz));
}

// The run of equal bins that starts at or contains this lane.
struct BinRun {
    int bin, len, longest;  // lanes from this one to the run's end; longest run of the warp
    bool head;
};
__device__ __forceinline__ BinRun bin_run(int bin) {
    const int lane = threadIdx.x & 31;
    BinRun r;
    r.bin = bin;
    const int before = __shfl_up_sync(0xffffffffu, bin, 1);
    r.head = lane == 0 || before != bin;
    const unsigned heads = __ballot_sync(0xffffffffu, r.head);
    const unsigned above = lane == 31 ? 0u : heads >> (lane + 1);
    r.len = above ? __ffs(above) : 32 - lane;
    r.longest = __reduce_max_sync(0xffffffffu, r.len);
    return r;
}
// Adds the run's sum of v to hist[bin] (bin < 0: lanes without a point).
__device__ __forceinline__ void bin_add(const BinRun &r, double v, double *hist) {
    for (int o = 1; o < r.longest; o <<= 1) {
        const double y = __shfl_down_sync(0xffffffffu, v, o);
        if (o < r.len) v += y;
    }
    if (r.head && r.bin >= 0) atomicAdd(&hist[r.bin], v);
}

// The points [first, first + count) of the flat index (a n1 + b) n0 + c, 32
// consecutive ones per step of a warp: coordinates of this lane's point.
struct WarpWalk {
    int a, b, c, n0, n1;
    size_t idx, end;
    __device__ __forceinline__ WarpWalk(size_t first, size_t count, int n0_, int n1_) : n0(n0_), n1(n1_) {
        idx = first + (threadIdx.x & 31);
        end = first + count;
        const unsigned t = (unsigned)idx / (unsigned)n0;  // < 2^31 for N <= 1290
        c = (int)((unsigned)idx - t * (unsigned)n0);
        a = (int)(t / (unsigned)n1);
        b = (int)(t - (unsigned)a * (unsigned)n1);
    }
    __device__ __forceinline__ bool any() const { return idx - (threadIdx.x & 31) < end; }
    __device__ __forceinline__ bool valid() const { return idx < end; }
    __device__ __forceinline__ void next() {
        idx += 32;
        c += 32;
        while (c >= n0) {
            c -= n0;
            if (++b == n1) { b = 0; a++; }
        }
    }
};

template <typename T>
__device__ __forceinline__ double l_power(const Cplx<T> p, const Cplx<T> x) {
    // sum_ij |l_ij|^2 with the reference's weights (diagonal 1, off-diagonal
    // 2) = 2 (|l+|^2 + |lx|^2) for a TT tensor
    const double pr = (double)p.re, pi = (double)p.im, xr = (double)x.re, xi = (double)x.im;
    return 2. * ((pr * pr + pi * pi) + (xr * xr + xi * xi));
}

// One lattice's share `part` of `parts` (warps) into the histograms hs
// [nseries][nb] and hc [nb] in shared memory.  F: field spectra [2] of
// N ny (N/2+1) points each, G: amplitudes [4] likewise (null: none).  Points
// that differ only in the signs of kx and ky share a bin and a weight: each
// lane reads the up to four of them (two when only part of the ky rows is
// held), so that a bin update serves four points and their loads overlap.
template <typename T>
__device__ __forceinline__ void bin_points(const Cplx<T> *F, const Cplx<T> *G, int N, int ny, int y0, int gt, int quirk,
                                           const double (&zero_re)[2], int nb, double *hs, unsigned int *hc,
                                           unsigned part, unsigned parts) {
    const int nz = N / 2 + 1;
    const bool fold_j = ny == N;
    const int nj = fold_j ? nz : ny;
    const size_t M = (size_t)N * ny * nz;
    const size_t folded = (size_t)nz * nj * nz;
    // whole steps of 32 points per warp
    const size_t per = ((folded + 32 * (size_t)parts - 1) / (32 * (size_t)parts)) * 32, first = part * per;
    const size_t count = first >= folded ? 0 : (folded - first < per ? folded - first : per);
    if (count == 0) return;
    for (WarpWalk w(first, count, nz, nj); w.any(); w.next()) {
        const bool ok = w.valid();
        const int i = w.a, y = w.b, j = fold_j ? y : y0 + y, kz = w.c;
        const bool edge = kz == 0 || kz == N / 2;
        const double wt = edge ? 1.0 : 2.0;
        const int mi = i > 0 && i < N / 2 ? 2 : 1, mj = fold_j && y > 0 && y < N / 2 ? 2 : 1;
        double p[2] = {0., 0.}, g = 0.;
        if (ok) {
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const int si = s >> 1, sj = s & 1;
                if (si < mi && sj < mj) {
                    const size_t at = ((size_t)(si ? N - i : i) * ny + (sj ? N - y : y)) * nz + kz;
#pragma unroll
                    for (int f = 0; f < 2; f++) {
                        const Cplx<T> v = F[(size_t)f * M + at];
                        double re = (double)v.re;
                        const double im = (double)v.im;
                        if (at == 0 && y0 == 0) re += zero_re[f];  // k = 0
                        p[f] += re * re + im * im;
                    }
                    if (G && gt != 1) {
                        const int lz = (quirk && kz == 0) ? N / 2 : kz;
                        const size_t src = gt == 2 ? g_index(si ? N - i : i, sj ? N - y : y, lz, N, 2) : at + (lz - kz);
                        g += l_power(G[2 * M + src], G[3 * M + src]);
                    }
                }
            }
        }
        const BinRun r = bin_run(ok ? native_bin(i, j <= N / 2 ? j : j - N, kz) : -1);
        // each point counts 2, on the kz = 0 and kz = N/2 planes 1
        unsigned c = ok ? (unsigned)(mi * mj) * (edge ? 1u : 2u) : 0u;
        for (int o = 1; o < r.longest; o <<= 1) {
            const unsigned z = __shfl_down_sync(0xffffffffu, c, o);
            if (o < r.len) c += z;
        }
        if (r.head && ok) atomicAdd(&hc[r.bin], c);
        bin_add(r, wt * p[0], hs);
        bin_add(r, wt * p[1], hs + nb);
        if (G && gt != 1) bin_add(r, wt * g, hs + 2 * nb);
    }
    if (!G || gt != 1) return;
    // amplitudes [kz][ky][kx] in their own order
    for (WarpWalk w(first, count, nz, nz); w.any(); w.next()) {
        const bool ok = w.valid();
        const int kz = w.a, j = w.b, i = w.c;
        // quirk: the kz = 0 plane is not read; the kz = N/2 plane is counted in its place too
        const bool use = ok && !(quirk && kz == 0), twice = ok && quirk && kz == N / 2;
        if (!__any_sync(0xffffffffu, use)) continue;
        const int mi = i > 0 && i < N / 2 ? 2 : 1, mj = j > 0 && j < N / 2 ? 2 : 1;
        double g = 0.;
        if (use) {
#pragma unroll
            for (int s = 0; s < 4; s++) {
                const int si = s >> 1, sj = s & 1;
                if (si < mi && sj < mj) {
                    const size_t at = ((size_t)kz * N + (sj ? N - j : j)) * N + (si ? N - i : i);
                    g += l_power(G[2 * M + at], G[3 * M + at]);
                }
            }
        }
        bin_add(bin_run(use ? native_bin(i, j, kz) : -1), (kz == 0 || kz == N / 2) ? g : 2. * g, hs + 2 * nb);
        if (__any_sync(0xffffffffu, twice)) bin_add(bin_run(twice ? native_bin(i, j, 0) : -1), g, hs + 2 * nb);
    }
}

constexpr int kBinThreads = 512;  // two blocks of 16 warps per SM

template <typename T>
__global__ void __launch_bounds__(kBinThreads, 2) bin_kernel(BinArgs a) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double *hs = reinterpret_cast<double *>(smem_raw);                      // [nseries][nbins]
    unsigned int *hc = reinterpret_cast<unsigned int *>(hs + a.nseries * a.nbins);  // [nbins]
    const int N = a.N, nb = a.nbins, ns = a.nseries;
    for (int q = threadIdx.x; q < ns * nb; q += blockDim.x) hs[q] = 0.0;
    for (int q = threadIdx.x; q < nb; q += blockDim.x) hc[q] = 0u;
    __syncthreads();
    const double zero[2] = {a.fix_zero ? a.zero_re[0] : 0., a.fix_zero ? a.zero_re[1] : 0.};
    bin_points<T>(static_cast<const Cplx<T> *>(a.F), ns > 2 ? static_cast<const Cplx<T> *>(a.G) : nullptr, N,
                  a.m ? a.m : N, a.y0, a.gt, a.quirk, zero, nb, hs, hc,
                  blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32, gridDim.x * (blockDim.x / 32));
    __syncthreads();
    double *ps = a.part_sum + (size_t)blockIdx.x * ns * nb;
    unsigned int *pc = a.part_cnt + (size_t)blockIdx.x * nb;
    for (int q = threadIdx.x; q < ns * nb; q += blockDim.x) ps[q] = hs[q];
    for (int q = threadIdx.x; q < nb; q += blockDim.x) pc[q] = hc[q];
}

// Fixed-order sum of the block histograms: 32 (series, bin) entries per block
// of 32 x kBinWays threads, each way summing every kBinWays-th histogram
// and the ways added in order.  A thread that summed all histograms of its
// entry alone waited for 296 loads in turn (63-68 us at any size).
constexpr int kBinWays = 32;
static __global__ void __launch_bounds__(32 * kBinWays)
    bin_reduce_kernel(const double *part_sum, const unsigned int *part_cnt, int nblocks, int nseries, int nbins, double *sum,
                      double *cnt) {
    __shared__ double s_sum[kBinWays][32];
    __shared__ unsigned long long s_cnt[kBinWays][32];
    const int x = threadIdx.x % 32, way = threadIdx.x / 32, q = blockIdx.x * 32 + x;
    double s = 0.0;
    unsigned long long n = 0;
#pragma unroll 4
    for (int b = way; b < nblocks; b += kBinWays) {
        if (q < nseries * nbins) s += part_sum[(size_t)b * nseries * nbins + q];
        if (q < nbins) n += part_cnt[(size_t)b * nbins + q];
    }
    s_sum[way][x] = s;
    s_cnt[way][x] = n;
    __syncthreads();
    if (way) return;
    for (int v = 1; v < kBinWays; v++) {
        s += s_sum[v][x];
        n += s_cnt[v][x];
    }
    if (q < nseries * nbins) sum[q] = s;
    if (q < nbins) cnt[q] = (double)n;
}

}  // namespace gabe
