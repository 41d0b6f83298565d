// FP32 stencil sweeps with a cp.async plane pipeline.
//
// Same sweeps as sweep_kernel (stencil.cuh: sweep A with the GW sources,
// sweep B, mode E0) and the same per-site arithmetic, with a data path built
// for HBM bandwidth rather than registers:
//
//   * a block owns a TK x TJ column tile (TK = 2 TK2 along k, two sites per
//     thread, 8-byte accesses) and marches along i over `ci` planes;
//   * every plane of the four input arrays (f phi, f chi, fdot phi, fdot chi)
//     -- the tile plus the one-point j/k halo -- is copied global -> shared
//     with cp.async, one 16-byte chunk per thread and array, into a ring of S
//     plane slots, S-3 planes ahead of the plane being computed;
//   * one barrier per plane: the slot of plane i-2 is refilled (plane i+S-2)
//     only after every thread has left plane i-1;
//   * a thread's two sites are one packed value (F2): sm_100's packed FP32
//     units take both with one instruction;
//   * the planes are walked three at a turn, so that the own pairs of planes
//     i-1, i, i+1 change roles instead of registers, and the constants lie in
//     shared memory.
// The sweeps were bound by instruction issue, not by HBM: with one site per
// instruction, the neighbours' stage-1 values formed one by one, separate own
// and halo copies and the constants in registers a warp took 424 instructions
// per plane of sweep A (370 sweep B), now 211 (191).  At 256^3, fields only:
// sweep A 118 against 152 us, B 111 against 119 (its 537 MB take 82 at the
// measured copy rate), energies alone 107 against 118.  With GW sources the
// stores bound sweep A.
// Each input value crosses HBM once per sweep (halo points are re-read from
// L2 by the neighbouring tiles).
#pragma once

#include "stencil.cuh"

namespace gabe {
namespace s32 {

__device__ __forceinline__ void cp_async8(void *smem, const void *gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
// 16 bytes, cached in L2 only.
__device__ __forceinline__ void cp_async16(unsigned s, const void *gmem) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int NPEND>
__device__ __forceinline__ void cp_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(NPEND) : "memory");
}

// Shared-memory plane slot: [4 arrays][TJ + 2 rows][PK columns]; column C0-1
// is the k0-1 halo, columns C0 .. C0+TK-1 the tile, column C0+TK the k0+TK
// halo.  C0 = 4, PK = TK + 8: rows are 16-byte multiples, so every copy is one
// of 16 bytes (L2 only): the pairs of threads 2m and 2m+1, four points of a
// halo row, and a halo column's point with the three beside it, which nothing
// reads.
template <int TK2, int TJ>
struct Ring {
    static constexpr int TK = 2 * TK2, PK = TK + 8, ROWS = TJ + 2, C0 = 4;
    static constexpr int ARR = ROWS * PK, SLOT = 4 * ARR;
};

// Per-launch constants of the FP32 site update (stage scalars as pairs,
// homogeneous trajectory).  They lie in shared memory: read again at each
// plane by a few broadcast loads, they leave the registers to the march.
struct alignas(16) Site32 {
    MeanP m0, m1;
    ModelP q;
    F2 h, dt, k0, k1, n3H0, n3H1, qs, third, m6, pad;  // k = 1 / (a dx)^2, n3H = -3 H of the stages, qs = dn / 4
    MeanTraj mt;
    double inv_dx2, q3;
};

template <int MODE>
__device__ __forceinline__ void site32_consts(const LatticeConsts &c, const DevScalars *scp, Site32 &s) {
    const double h = c.half_dt, a0 = scp->a[0];
    auto k = [](double x) { return f2((float)x); };
    s.mt = mean_traj(c, scp);
    s.m0 = mean_p(s.mt.fb0);
    s.m1 = mean_p(s.mt.fb1);
    s.q = model_p(c);
    s.inv_dx2 = 1.0 / c.inv_dx2_div;
    s.q3 = (double)(float)(-h * 3. / a0);
    s.h = k(h);
    s.dt = k(c.dt);
    s.k0 = k(s.inv_dx2 / (a0 * a0));
    s.qs = k(0.25 * c.dn);
    s.third = f2(1.f / 3.f);
    s.m6 = f2(-6.f);
    if constexpr (MODE == MODE_B) {
        const double ad0 = scp->adot[0], a1 = scp->a[1], ad1 = scp->adot[1];
        s.k1 = k(s.inv_dx2 / (a1 * a1));
        s.n3H0 = k(-(3. * ad0) / a0);
        s.n3H1 = k(-(3. * ad1) / a1);
    }
}

// Potential of the site functions: MODEL >= 0 fixes it at compile time (the
// single-lattice sweeps, one instantiation per model, no branch per site),
// -1 reads it from the lattice constants (the ensemble's mixed batches).
template <int MODEL>
__device__ __forceinline__ int site_model(const LatticeConsts &c) {
    return MODEL >= 0 ? MODEL : c.model;
}

// What the site functions take of one array at the thread's pair of sites:
// the values, dx^2 times the Laplacian and the undivided central differences.
// The stage-1 fields are f + h fdot, so these of stage 1 follow from f's and
// fdot's without forming the neighbours' stage-1 values.
struct Pair {
    F2 v, lap, e[3];
};
// own pairs of planes i, i+1, i-1 and rows j+1, j-1; the points left and right of the pair
template <bool GRAD>
__device__ __forceinline__ Pair pair_of(F2 m6, F2 cu, F2 nx, F2 pr, F2 up, F2 dn, float lm, float rp) {
    Pair p;
    p.v = cu;
    const float2 c = unpack(cu);
    p.lap = fma2(m6, cu, ((nx + pr) + (up + dn)) + f2(c.y + lm, rp + c.x));
    if constexpr (GRAD) {
        p.e[0] = nx - pr;
        p.e[1] = up - dn;
        p.e[2] = f2(c.y - lm, rp - c.x);
    }
    return p;
}

// In the force, lap / a^2 - V' - 3 H d, the Laplacian is the largest term by far, but the mean of V' over the lattice is
// what drives the mean field.  So V' and the drag are summed first and the Laplacian's product enters last and
// unrounded: one rounding at its size, and one that is as often up as down.  Added to a rounded Laplacian, the part of V'
// below half an ulp of it was lost, always in the same direction (potential energy off by 1.7e-13 instead of 1e-15 after
// 150 steps at 128^3, lambda phi^4; by 3.9e-11 instead of 1e-14 after 1000 at 512^3).

// The thread's pair of sites in sweep A / E0: adds to the moments, fills the sources.
template <int MODE, int MODEL = -1>
__device__ __forceinline__ void site_a32(const LatticeConsts &c, const Site32 &s, const Pair (&p)[4], Moments &m,
                                         F2 (&s0)[kSrc], F2 (&s1)[kSrc]) {
    const int model = site_model<MODEL>(c);
    const F2 h = s.h;
    F2 t0[2], f1[2];
    if constexpr (MODE != MODE_E0) sub_dv_diff32<true>(s.m0, s.q, model, p[0].v, p[1].v, t0);
    F2 P0[6], P1[6];
    if constexpr (MODE == MODE_A_GW) {
#pragma unroll
        for (int q = 0; q < 6; q++) P0[q] = P1[q] = f2(0.f);
    }
#pragma unroll
    for (int f = 0; f < 2; f++) {
        const Pair &ff = p[f], &dd = p[2 + f];
        const F2 d = dd.v;
        m.a[f] = m.a[f] + d;
        m.b = fma2(d, d, m.b);
        m.g0 = fma2(ff.v, ff.lap, m.g0);
        if constexpr (MODE != MODE_E0) {
            f1[f] = fma2(h, d, ff.v);
            const F2 Pd = fma2(h, fma2(s.k0, ff.lap, t0[f]), d);  // stage-0 force without the drag
            m.c[f] = m.c[f] + Pd;
            m.e = fma2(Pd, Pd, m.e);
            m.f = fma2(Pd, d, m.f);
            m.g1 = fma2(f1[f], fma2(h, dd.lap, ff.lap), m.g1);
            if constexpr (MODE == MODE_A_GW) {
                grad_prod_add(ff.e[0], ff.e[1], ff.e[2], P0);
                grad_prod_add(fma2(h, dd.e[0], ff.e[0]), fma2(h, dd.e[1], ff.e[1]), fma2(h, dd.e[2], ff.e[2]), P1);
            }
        }
    }
    if constexpr (MODE == MODE_A_GW) {
        source_from_prod(s.qs, s.third, P0, s0);
        source_from_prod(s.qs, s.third, P1, s1);
    }
    m.v0 = m.v0 + v_diff32(s.m0, s.q, model, p[0].v, p[1].v);
    if constexpr (MODE != MODE_E0) m.v1 = m.v1 + v_diff32(s.m1, s.q, model, f1[0], f1[1]);
}

// The pair in sweep B: the new field and momentum of both fields.
template <int MODEL = -1>
__device__ __forceinline__ void site_b32(const LatticeConsts &c, const Site32 &s, const Pair (&p)[4], F2 (&xo)[2],
                                         F2 (&dout)[2]) {
    const int model = site_model<MODEL>(c);
    const F2 h = s.h, dt = s.dt;
    F2 t0[2], t1[2], f1[2], d1[2];
#pragma unroll
    for (int f = 0; f < 2; f++) {
        t0[f] = s.n3H0 * p[2 + f].v;
        f1[f] = fma2(h, p[2 + f].v, p[f].v);
    }
    sub_dv_diff32<false>(s.m0, s.q, model, p[0].v, p[1].v, t0);
#pragma unroll
    for (int f = 0; f < 2; f++) {
        d1[f] = fma2(h, fma2(s.k0, p[f].lap, t0[f]), p[2 + f].v);
        xo[f] = fma2(dt, d1[f], p[f].v);
        t1[f] = s.n3H1 * d1[f];
    }
    sub_dv_diff32<false>(s.m1, s.q, model, f1[0], f1[1], t1);
#pragma unroll
    for (int f = 0; f < 2; f++)
        dout[f] = fma2(dt, fma2(s.k1, fma2(h, p[2 + f].lap, p[f].lap), t1[f]), p[2 + f].v);
}

// Threads per SM the register budget is sized for: sweep A with sources holds
// the most live values and runs two 256-thread blocks per SM without spills;
// the others fit three.
template <int MODE>
constexpr int sweep32_threads_per_sm() {
    return (MODE == MODE_A_GW || MODE == MODE_A) ? 512 : 768;
}

// Pointers and bounds of one column tile of one lattice.
struct Tile32 {
    const float *X, *D;  // fields and momenta of the current state, [2][N^3]
    float *Xo, *Do;      // new fields and momenta (sweep B)
    float *S;            // GW sources (sweep A with sources; a slab: its own planes)
    SrcLayout src;       // ... in this layout
    int k0, j0, i0, i1;
    int planes;          // planes per field in X, D, Xo, Do (slab, no wrap along i); 0 = N, periodic
};

// The plane march of one TK x TJ tile over planes i0 .. i1-1 by a block of NT
// threads (NT >= TK2 TJ; threads beyond TK2 TJ only take part in the
// barriers).  Sweep A / E0 add the tile's folded sums to acc (per-thread
// partials, zero on idle threads); sweep B writes the new state.
template <int TK2, int TJ, int MODE, int S, int NT, int MODEL = -1>
__device__ __forceinline__ void march32(const LatticeConsts &c, const Site32 &s, const Tile32 &t, float *ring,
                                        double (&acc)[kNV]) {
    using Rg = Ring<TK2, TJ>;
    constexpr int TK = Rg::TK, PK = Rg::PK, C0 = Rg::C0;
    static_assert(S >= 4, "ring needs planes i-1, i, i+1 and one in flight");
    // chunks of 16 bytes of a plane's tile with its halo, one per thread and array
    constexpr int CQ = TK / 4 + 2, CHUNKS = (TJ + 2) * CQ;
    static_assert(TK % 4 == 0 && CHUNKS <= NT, "one chunk per thread");
    static_assert(NT >= TK2 * TJ, "block smaller than the tile");
    const int N = c.N;
    const int n3 = (t.planes ? t.planes : N) * N * N;  // < 2^31 for N <= 1024
    const int tid = threadIdx.x;
    const bool act = NT == TK2 * TJ || tid < TK2 * TJ;
    const int tx = tid % TK2, ty = tid / TK2;
    const int k0 = t.k0, j0 = t.j0, i0 = t.i0, i1 = t.i1;
    const int j = j0 + ty, k = k0 + 2 * tx;

    // the thread's own pair and the chunk that it copies (row cr, chunk cq; the
    // corners are not read), as offsets within a plane; planes are p N^2
    const int NN = N * N;
    const int o_own = j * N + k;
    const int so_own = (ty + 1) * PK + C0 + 2 * tx;  // shared offset of the own pair within an array
    const int cr = tid / CQ, cq = tid % CQ;
    const bool inner_r = cr > 0 && cr <= TJ, inner_q = cq > 0 && cq < CQ - 1;
    const bool inner = tid < CHUNKS && inner_r && inner_q, copies = tid < CHUNKS && (inner_r || inner_q);
    int ck = k0 - 4 + 4 * cq;
    ck += ck < 0 ? N : (ck >= N ? -N : 0);
    const int c_go = wrapi(j0 - 1 + cr, N) * N + ck;
    const unsigned c_so = (unsigned)__cvta_generic_to_shared(ring + cr * PK + 4 * cq);
    auto issue = [&](int p, int sl) {  // plane p (wrapped) into slot sl
        if (!copies) return;
        const unsigned d = c_so + sl * (unsigned)(Rg::SLOT * sizeof(float));
        const int g = (t.planes ? p : wrapi(p, N)) * NN + c_go;
        cp_async16(d, t.X + g);
        cp_async16(d + Rg::ARR * 4, t.X + n3 + g);
        // the energies-only sweep reads the momenta at the own sites only
        if (MODE == MODE_E0 && !inner) return;
        cp_async16(d + Rg::ARR * 8, t.D + g);
        cp_async16(d + Rg::ARR * 12, t.D + n3 + g);
    };
    auto next_slot = [](int sl) { return sl + 1 == S ? 0 : sl + 1; };

    Moments mom;
    zero(mom);
    int ngroup = 0;  // planes in the current moment group

    // prologue: planes i0-1 .. i0+S-3 (one commit group each) into slots 0 .. S-2
#pragma unroll
    for (int q = 0; q < S - 1; q++) {
        const int p = i0 - 1 + q;
        if (p <= i1) issue(p, q);
        cp_commit();
    }
    // sources of the whole lattice, or of a slab's own planes (plane i at i - 1)
    const int splanes = t.planes ? t.planes - 2 : N, sfirst = t.planes ? 1 : 0;
    const int srow = t.src == SRC_PADDED ? N + 2 : N, splane = N * (t.src == SRC_ROWS ? N : N + 2);
    const int sstride = splanes * splane;  // one source component
    const int so_row = j * srow + k;
    using Own = F2[4];  // the own pair of the four arrays in one plane
    auto own = [&](int sl, int a) {
        return *reinterpret_cast<const F2 *>(ring + sl * Rg::SLOT + a * Rg::ARR + so_own);
    };
    int i = i0, s_cu = 1, s_nx = 2, s_is = S - 1;  // slots of planes i, i+1 and of the plane issued next (i+S-2)
    // one plane: pr, cu are the own pairs of planes i-1 and i, nx becomes that of i+1
    auto plane = [&](Own &pr, Own &cu, Own &nx) {
        cp_wait<S - 4>();  // planes up to i+1 have landed (this thread's copies)
        __syncthreads();   // ... and everybody's; every thread has left plane i-1
        if (i + S - 2 <= i1) issue(i + S - 2, s_is);  // into the slot of plane i-2
        cp_commit();
        if (act) {
            const float *sc = ring + s_cu * Rg::SLOT + so_own;
            Pair p[4];
#pragma unroll
            for (int a = 0; a < 4; a++) {
                nx[a] = own(s_nx, a);
                if (MODE == MODE_E0 && a >= 2) {  // own momenta only
                    p[a].v = cu[a];
                    continue;
                }
                const float *q = sc + a * Rg::ARR;
                p[a] = pair_of<MODE == MODE_A_GW>(s.m6, cu[a], nx[a], pr[a], *reinterpret_cast<const F2 *>(q + PK),
                                                  *reinterpret_cast<const F2 *>(q - PK), q[-1], q[2]);
            }
            if constexpr (MODE == MODE_B) {
                F2 xo[2], dout[2];
                site_b32<MODEL>(c, s, p, xo, dout);
                const int gx = i * NN + o_own;
                __stcs(reinterpret_cast<float2 *>(t.Xo + gx), unpack(xo[0]));
                __stcs(reinterpret_cast<float2 *>(t.Xo + n3 + gx), unpack(xo[1]));
                __stcs(reinterpret_cast<float2 *>(t.Do + gx), unpack(dout[0]));
                __stcs(reinterpret_cast<float2 *>(t.Do + n3 + gx), unpack(dout[1]));
            } else {
                F2 s0[kSrc], s1[kSrc];
                site_a32<MODE, MODEL>(c, s, p, mom, s0, s1);
                if (++ngroup == kGroup || i == i1 - 1) {
                    fold<MODE>(s.mt, s.q3, s.inv_dx2, 2 * ngroup, mom, acc);
                    ngroup = 0;
                }
                if constexpr (MODE == MODE_A_GW) {
                    float *g = t.S + ((i - sfirst) * splane + so_row);
#pragma unroll
                    for (int q = 0; q < kSrc; q++, g += sstride) __stcs(reinterpret_cast<float2 *>(g), unpack(s0[q]));
#pragma unroll
                    for (int q = 0; q < kSrc; q++, g += sstride) __stcs(reinterpret_cast<float2 *>(g), unpack(s1[q]));
                }
            }
        }
        s_cu = s_nx;
        s_nx = next_slot(s_nx);
        s_is = next_slot(s_is);
        return ++i < i1;
    };
    cp_wait<S - 3>();  // planes i0-1 and i0
    __syncthreads();
    Own x[3];
    if (act) {
#pragma unroll
        for (int a = 0; a < 4; a++) x[0][a] = own(0, a), x[1][a] = own(1, a);
    }
    // three planes a turn, so that no pair moves from register to register
    while (plane(x[0], x[1], x[2]) && plane(x[1], x[2], x[0]) && plane(x[2], x[0], x[1])) {
    }
    cp_wait<0>();
    __syncthreads();  // the ring may be refilled by the block's next tile
}

template <int TK2, int TJ, int MODE, int S, int MODEL = -1>
__global__ void __launch_bounds__(TK2 *TJ, (sweep32_threads_per_sm<MODE>() + TK2 * TJ - 1) / (TK2 * TJ))
    sweep32_kernel(StencilArgs args) {
    extern __shared__ __align__(16) float ring[];  // S slots
    __shared__ double sred[((TK2 * TJ + 31) / 32) * kNV];
    __shared__ int sflag;

    const LatticeConsts &c = args.c;
    const int N = c.N;
    const int tid = threadIdx.x;
    Tile32 t;
    t.X = static_cast<const float *>(args.X);
    t.D = static_cast<const float *>(args.D);
    t.Xo = static_cast<float *>(args.Xo);
    t.Do = static_cast<float *>(args.Do);
    t.S = static_cast<float *>(args.S);
    t.k0 = blockIdx.x * 2 * TK2;
    t.j0 = blockIdx.y * TJ;
    t.planes = args.planes;
    t.src = args.src;
    const int first = args.planes ? 1 : 0, end = args.planes ? args.planes - 1 : N;  // own planes
    t.i0 = first + blockIdx.z * args.ci;
    t.i1 = min(t.i0 + args.ci, end);

    __shared__ Site32 s;
    // by the last thread, which copies nothing; the march waits for the block before it reads them
    if (tid == (int)blockDim.x - 1) site32_consts<MODE>(c, args.sc, s);
    double acc[kNV];
#pragma unroll
    for (int q = 0; q < kNV; q++) acc[q] = 0.;
    march32<TK2, TJ, MODE, S, TK2 * TJ, MODEL>(c, s, t, ring, acc);

    const int bid = blockIdx.x + gridDim.x * (blockIdx.y + gridDim.y * blockIdx.z);
    if constexpr (MODE != MODE_B) {
        block_reduce<kNV>(acc, sred);
        if (tid == 0)
            for (int q = 0; q < kNV; q++) args.partials[(size_t)bid * kNV + q] = acc[q];
    }
    if (!last_block_done(args.counter, &sflag)) return;
    if constexpr (MODE != MODE_B) {
        double tot[kNV];
        sum_partials<kNV>(args.partials, gridDim.x * gridDim.y * gridDim.z, tot, sred);
        if (tid == 0) {
            if (args.sums_out)
                for (int q = 0; q < kNV; q++) args.sums_out[q] = tot[q];
            else
                finish_a<float, MODE>(c, args.sc, tot, args.slot);
            if (args.mirror) *args.mirror = *args.sc;
            *args.counter = 0u;
        }
    } else if (tid == 0) {
        finish_b<float>(c, args.sc);
        *args.counter = 0u;
    }
}

}  // namespace s32
}  // namespace gabe
