// Host side of the plane transform (fftp.cuh): persistent grids sized from
// each kernel's occupancy.
#include "fftp.cuh"
#include "launch.h"

namespace gabe {

namespace {

template <typename K>
cudaError_t grid_of(K kernel, int threads, size_t smem, int ntiles, int *grid) {
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, per_sm = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem)) != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    *grid = nsm * per_sm < ntiles ? nsm * per_sm : ntiles;
    return cudaSuccess;
}

template <int N>
cudaError_t planes_n(float *S, int nplanes, cudaStream_t s) {
    constexpr size_t smem = f2p::PlaneGeom<N>::SMEM_BYTES;
    auto k = f2p::plane_kernel<N>;
    const int ntiles = nplanes / f2p::Cfg<N>::PB;
    int g = 0;
    cudaError_t e = grid_of(k, f2p::Cfg<N>::TP, smem, ntiles, &g);
    if (e != cudaSuccess) return e;
    k<<<g, f2p::Cfg<N>::TP, smem, s>>>(S, ntiles);
    return cudaGetLastError();
}

template <int N>
cudaError_t lines_n(const f2p::LineArgs &a, cudaStream_t s) {
    constexpr size_t smem = f2p::LineGeom<N>::SMEM_BYTES;
    auto k = f2p::lines_kernel<N>;
    int g = 0;
    cudaError_t e = grid_of(k, f2p::Cfg<N>::TL, smem, a.nlat * f2p::LineGeom<N>::XT, &g);
    if (e != cudaSuccess) return e;
    k<<<g, f2p::Cfg<N>::TL, smem, s>>>(a);
    return cudaGetLastError();
}

}  // namespace

#define GABE_F2P_SIZES(X) X(16) X(32) X(48) X(64) X(80) X(96) X(112) X(128) X(144) X(160)

bool fftp_supported(int N) {
#define X(n) || N == n
    return false GABE_F2P_SIZES(X);
#undef X
}

cudaError_t fftp_planes_f32(int N, float *S, int nplanes, cudaStream_t s) {
    switch (N) {
#define X(n) \
    case n: return planes_n<n>(S, nplanes, s);
        GABE_F2P_SIZES(X)
#undef X
        default: return cudaErrorInvalidValue;
    }
}

cudaError_t fftp_lines_f32(int N, const void *T, void *G, const DevScalars *sc, const int *ids, int nlat,
                           const LatticeConsts &c, int slot, cudaStream_t s) {
    const f2p::LineArgs a{static_cast<const float2 *>(T), static_cast<float2 *>(G), sc, ids, c, slot, nlat};
    switch (N) {
#define X(n) \
    case n: return lines_n<n>(a, s);
        GABE_F2P_SIZES(X)
#undef X
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gabe
