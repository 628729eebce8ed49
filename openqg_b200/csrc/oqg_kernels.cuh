// oqg_kernels.cuh -- the per-step kernels of the QG core (sm_100a).
//
// One step_qg (qg/core.F90:16-33) is a chain of launches, one per dependent
// phase:
//   k_vort   vort_step (qg/vorticity.F90:14-103) + p_modes_rhs (qg/modes.F90:248-266)
//            2-D tiles staged in shared memory; the layer loop runs inside the
//            CTA so the modal right-hand side is formed in registers.
//   k_bfwd   forward x-transform of solve_inhomog_box (qg/inhomog.F90:170-212),
//            DST-I; k_xfwd, of solve_inhomog_cyclic (inhomog.F90:214-255), r2c FFT.
//   k_ysolve Thomas solve in y per (mode, wavenumber) (inhomog.F90:187-199),
//            chunks of rows in registers, their affine maps scanned.
//   k_xinv   inverse x-transform + homogeneous correction + modes_to_layers
//            (modes.F90:268-284) + ocqbdy (vorsubs.F90:58-114) +
//            suppress_comp_mode (driver.F90:174-189).  One warp of each CTA
//            runs the scalar phase meanwhile: update_mass_constr
//            (constraint.F90:167-179), box_homog's 2x2 solve (homog.F90:331-366)
//            or step_constraints + cyclic_homog (constraint.F90:182-215,
//            homog.F90:280-329), and the suppress_comp_mode schedule
//            (openqg.F90:485-487).
//   or, as two launches (the default for boxes, measured for channels):
//   k_binv, k_xinv_rows  the inverse x-transforms alone (a box's, a channel's),
//            shaped like the forward ones, with one extra CTA per basin for the
//            scalar phase;
//   k_xinv_asm   the homogeneous correction, modes_to_layers, ocqbdy and the
//            suppression averages, one thread per point.
// Every launch takes a work list, so one launch serves one basin or an
// ensemble of basins of uneven size.
#pragma once

#include "oqg_dev.cuh"
#include "oqg_fft.cuh"
#include "oqg_odd.cuh"
#include "oqg_tma.cuh"

#include <type_traits>

namespace oqg {

// ------------------------------------------------------------------ helpers
template <class T> __device__ __forceinline__ T ldg(const T *p) { return __ldg(p); }

// Programmatic dependent launch: the next kernel of the step may be scheduled
// now; and wait until the previous kernel's results are visible.  Without the
// launch attribute both are no-ops.
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ double shfl_up_d(double v, int o) { return __shfl_up_sync(0xffffffffu, v, o); }
__device__ __forceinline__ double shfl_dn_d(double v, int o) { return __shfl_down_sync(0xffffffffu, v, o); }

__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    return v;
}

// Deterministic CTA sum (result valid in every thread). red: >= 32 doubles.
__device__ __forceinline__ double block_sum(double v, double *red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = warp_sum(v);
    __syncthreads();
    if (lane == 0) red[wid] = v;
    __syncthreads();
    double s = 0.0;
    if (wid == 0) {
        s = lane < nw ? red[lane] : 0.0;
        s = warp_sum(s);
        if (lane == 0) red[0] = s;
    }
    __syncthreads();
    s = red[0];
    __syncthreads();
    return s;
}

// ------------------------------------------------------------------ compensated sums
// The mass-constraint and area integrals (int_P_dA, numerics.F90:165-204;
// box_homog's modal integrals, homog.F90:331-366) are summed with a running
// compensation: every addition is Knuth's error-free TwoSum, s + e = a + b
// exactly, and the rounding errors are summed beside the sum (Neumaier's
// scheme), so the result is correct to about one rounding of the total
// whatever the cancellation among the terms.  Nothing here is contracted
// into FMAs (no products).
__device__ __forceinline__ void two_sum(double a, double b, double &s, double &e) {
    s = a + b;
    const double bb = s - a;
    e = (a - (s - bb)) + (b - bb);
}
struct CSum {
    double s = 0.0, c = 0.0;
    __device__ __forceinline__ void add(double x) {
        double t, e;
        two_sum(s, x, t, e);
        s = t;
        c += e;
    }
    // another compensated sum (its sum and its compensation)
    __device__ __forceinline__ void merge(double os, double oc) {
        add(os);
        c += oc;
    }
    // the exact product w * x of a weight and a term, added (the product's
    // rounding error comes from an FMA)
    __device__ __forceinline__ void add_prod(double w, double x) {
        const double p = w * x;
        add(p);
        c += fma(w, x, -p);
    }
    __device__ __forceinline__ double value() const { return s + c; }
};
// Warp reduction of compensated sums; the total is in lane 0 (all lanes
// with full=true).
__device__ __forceinline__ CSum csum_warp(CSum v, bool full = false) {
    for (int o = 16; o > 0; o >>= 1) {
        const double os = full ? __shfl_xor_sync(0xffffffffu, v.s, o) : __shfl_down_sync(0xffffffffu, v.s, o);
        const double oc = full ? __shfl_xor_sync(0xffffffffu, v.c, o) : __shfl_down_sync(0xffffffffu, v.c, o);
        v.merge(os, oc);
    }
    return v;
}
// CTA reduction of compensated sums: the total as a compensated pair, valid
// in every thread.  red: >= 64 doubles of shared memory.
__device__ __forceinline__ CSum csum_block_pair(CSum v, double *red) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    v = csum_warp(v);
    __syncthreads();
    if (lane == 0) { red[wid] = v.s; red[32 + wid] = v.c; }
    __syncthreads();
    if (wid == 0) {
        CSum t;
        if (lane < nw) { t.s = red[lane]; t.c = red[32 + lane]; }
        t = csum_warp(t);
        if (lane == 0) { red[0] = t.s; red[1] = t.c; }
    }
    __syncthreads();
    CSum r;
    r.s = red[0];
    r.c = red[1];
    __syncthreads();
    return r;
}
__device__ __forceinline__ double csum_block(CSum v, double *red) { return csum_block_pair(v, red).value(); }
// K of these reductions at once, each in csum_block_pair's order: the K chains
// of shuffles and additions overlap and two barriers serve them all.  The
// totals are valid in thread 0.
template <int K> __device__ __forceinline__ void csum_block_n(CSum (&v)[K], double (&total)[K]) {
    __shared__ double rs[K][32], rc[K][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
    auto warp = [&](CSum (&x)[K]) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < K; ++q) {
                const double os = __shfl_down_sync(0xffffffffu, x[q].s, o), oc = __shfl_down_sync(0xffffffffu, x[q].c, o);
                x[q].merge(os, oc);
            }
    };
    warp(v);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < K; ++q) { rs[q][wid] = v[q].s; rc[q][wid] = v[q].c; }
    __syncthreads();
    if (wid == 0) {
        CSum t[K];
#pragma unroll
        for (int q = 0; q < K; ++q)
            if (lane < nw) { t[q].s = rs[q][lane]; t[q].c = rc[q][lane]; }
        warp(t);
#pragma unroll
        for (int q = 0; q < K; ++q) total[q] = t[q].value();
    }
}

// Barrier of the CTAs of a cluster (release and acquire), and a value of CTA
// rank's shared memory at the place of this CTA's p.
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.aligned;\nbarrier.cluster.wait.aligned;\n" ::: "memory");
}
__device__ __forceinline__ double ld_cluster(const double *p, int rank) {
    double v;
    asm volatile("{\n\t.reg .b32 a;\n\tmapa.shared::cluster.u32 a, %1, %2;\n\tld.shared::cluster.f64 %0, [a];\n\t}\n"
                 : "=d"(v) : "r"(smem_u32(p)), "r"(rank) : "memory");
    return v;
}

// ------------------------------------------------------------------ k_vort
#define VTX 60          // output columns of a vorticity tile
#define VTYMAX 17       // output rows of a vorticity tile (at most)
#define VSTRIPS 4        // row strips of a tile (64 column lanes each)
#define VWIDE 8          // the same where every SM has at most one tile
#define XINV_E 16           // complex values per transform thread of a channel

// Storage of q: FP64 handles keep q itself; FP32 handles keep the anomaly
// q - beta yprel (the planetary vorticity is most of q, and in FP32 its
// rounding would swamp the relative and stretching vorticity that the
// Helmholtz inversion recovers from q - beta y).  Every kernel that reads or
// writes q applies this; the host converts at the boundary (oqg_get_state,
// oqg_set_state_full).
template <class T> __host__ __device__ constexpr bool q_anom_stored() { return sizeof(T) == 4; }

// Geometry of a basin for the stencils; the coefficients sit in a shared
// table (K = fx, fy, fxb, fyb, jac) that the kernel fills once.
template <class T> struct GeoS {
    int nxp, nyp, cyclic;
    const T *K;
};
template <class T> __device__ __forceinline__ T gfx(const GeoS<T> &g) { return g.K[0]; }
template <class T> __device__ __forceinline__ T gfy(const GeoS<T> &g) { return g.K[1]; }
template <class T> __device__ __forceinline__ T gfxb(const GeoS<T> &g) { return g.K[2]; }
template <class T> __device__ __forceinline__ T gfyb(const GeoS<T> &g) { return g.K[3]; }
template <class T> __device__ __forceinline__ T gjac(const GeoS<T> &g) { return g.K[4]; }

// Laplacian with the mixed wall condition (del2_P_bc, numerics.F90:410-468)
// from the five stencil values (W, E, S, N, C): the interior formula, or on
// a wall the one-sided mixed-BC terms, chosen by selects (no divergent
// branches).  fx, fy: 1/dx^2, 1/dy^2; fxb, fyb: their mixed-BC factors.
template <class T>
__device__ __forceinline__ T lap5_sel(T wv, T ev, T sv, T nv, T c, bool zrow, bool wl, bool wr, bool jlo,
                                      bool jhi, T fx, T fy, T fxb, T fyb) {
    T xp = fx * (wv + ev - (T)2 * c);
    if (wl) xp = fxb * (ev - c);
    if (wr) xp = -(fxb * (c - wv));
    if (zrow) xp = (T)0;
    T yp = fy * (sv + nv - (T)2 * c);
    if (jlo) yp = fyb * (nv - c);
    if (jhi) yp = -(fyb * (c - sv));
    if (wl || wr) yp = (T)0;
    return xp + yp;
}

// cp.async copy of one element into shared memory; zero-filled when !valid
// (the source is then not read).
template <class T>
__device__ __forceinline__ void cp_async_el(T *dst, const T *src, bool valid) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(dst);
    const int n = valid ? (int)sizeof(T) : 0;
    if (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8, %2;\n" ::"r"(sa), "l"(src), "r"(n) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(sa), "l"(src), "r"(n) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Queues the copy of rows [jlo, jlo+nr) x cols [ilo, ilo+nc) of layer k of f
// into s (leading dimension nc); outside the basin -> 0.  A channel's columns
// of a halo tile wrap with period nxp-1 as far as the last output column's
// halo; an `own` tile (the CTA's output columns only) reads columns < nxp as
// stored, including the duplicate column nxp-1, and zeros beyond, so it never
// reads a column that another CTA writes.  A box (whose tiles come so when
// there are no tensor maps) has no column outside 0 .. nxp-1.
// Thread layout: 64 columns x blockDim / 64 rows.
template <class T, class G>
__device__ __forceinline__ void load_tile_async(T *s, const T *__restrict__ f, const G &g, int px,
                                                int k, int jlo, int nr, int ilo, int nc,
                                                bool own = false) {
    const int N = g.nxp - 1;
    const bool wrap = g.cyclic && !own;
    const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
    const T *fk = f + (size_t)k * g.nyp * px;
    for (int c = tx; c < nc; c += 64) {
        const int gi = ilo + c;
        const bool cv = wrap ? gi < g.nxp + 3 : gi >= 0 && gi < g.nxp;
        const int i = !cv ? 0 : !wrap ? gi : gi < 0 ? gi + N : gi >= N ? gi - N : gi;
        for (int r = ty; r < nr; r += blockDim.x >> 6) {
            const int j = jlo + r;
            const bool v = cv && j >= 0 && j < g.nyp;
            cp_async_el(s + r * nc + c, fk + (size_t)(v ? j : 0) * px + i, v);
        }
    }
}

// Tiles are VTX columns by b.vty rows (b.vty <= VTYMAX, chosen per basin so
// that the tiles fill whole waves); tile rows start at row 1 (the walls are not
// stepped).  Shared tiles per layer (origin, pitch):
//   pm     rows j0-3 .. j0+vty+2, cols from i0-4   (LPQ = VTX+8 = 68)
//   p, q   rows j0-1 .. j0+vty,   cols from i0-4   (LPQ)
//   qm     rows j0 .. j0+vty-1,   cols from i0     (LO = VTX)
//   d2     rows j0-2 .. j0+vty+1, cols from i0-2   (L2 = VTX+4 = 64), computed
//   d4     rows j0-1 .. j0+vty,   cols from i0-1   (L1 = VTX+2), computed
// The x-origins are multiples of 4 elements (16 bytes), as tensor loads need.
// Tiles arrive by TMA (one thread issues, an mbarrier counts the bytes), but
// for a channel's at the seam, which wrap and come by cp.async.  Thread
// (lane x, strip y) owns column x of each phase and marches down a strip of
// rows with a rolling window of the stencil in registers.
struct VortLayout {
    int HPM, H2, H1, VT;
    int pm, p, q, qm, nbuf;     // offsets within a layer buffer (elements)
    int d2, d4, wk, by, total;  // offsets after the two layer buffers
};
__host__ __device__ __forceinline__ int vort_round(int n, int esz) {
    const int a = 128 / esz;
    return (n + a - 1) / a * a;
}
__host__ __device__ __forceinline__ VortLayout vort_layout(int vt, int esz) {
    constexpr int LPQ = VTX + 8, L2 = VTX + 4, L1 = VTX + 2, LO = VTX;
    VortLayout L;
    L.VT = vt;
    L.HPM = vt + 6;
    L.H2 = vt + 4;
    L.H1 = vt + 2;
    L.pm = 0;
    L.p = L.pm + vort_round(L.HPM * LPQ, esz);
    L.q = L.p + vort_round(L.H1 * LPQ, esz);
    L.qm = L.q + vort_round(L.H1 * LPQ, esz);
    L.nbuf = L.qm + vort_round(vt * LO, esz);
    L.d2 = 2 * L.nbuf;
    L.d4 = L.d2 + vort_round(L.H2 * L2, esz);
    L.wk = L.d4 + vort_round(L.H1 * L1, esz);
    L.by = L.wk + vort_round(vt * LO, esz);
    L.total = L.by + vort_round(vt * 8 / esz + 1, esz);   // vt doubles
    return L;
}
// Rows of vorticity tiles (of the interior rows) and CTAs of a basin: a
// channel's strip integrals first (one CTA per wall and layer), then the tiles.
__host__ __device__ __forceinline__ int vort_tile_rows(int nyp, int vt) { return (nyp - 2 + vt - 1) / vt; }
__host__ __device__ __forceinline__ int vort_strips(int nl, int cyclic) { return cyclic ? 2 * nl : 0; }
// Dynamic shared bytes of k_vort (plus slack to align the base to 128 bytes).
__host__ __device__ __forceinline__ size_t vort_smem_bytes(int vt, int esz) {
    return (size_t)vort_layout(vt, esz).total * esz + 128;
}

// Tensor maps of a basin, in this order: p/q-shaped boxes of F[0..3],
// pm-shaped boxes of F[0], F[1], qm-shaped boxes of F[2], F[3], wekp.
#define OQG_TMAP_PQ 0
#define OQG_TMAP_PM 4
#define OQG_TMAP_QM 6
#define OQG_TMAP_WK 8
#define OQG_NTMAP 9
#define OQG_TMAP_BYTES 128

// The channel's strip integrands (vorticity.F90:84-101, numerics.F90:374-386)
// along one wall of layer k, summed over x by one CTA: with rows counted from
// the wall, q(0) dp(1), q(1) dp(1) (dp the zonal difference of p), the steps
// of del2(pm), del4(pm) and (drag layer) pm from row 0 to row 1, signed
// northward.  part: [2 walls][nl][OQG_NSTRIP].
template <class T>
__device__ __forceinline__ void vort_strip(const BasinDev &b, int side, int k, int par) {
    const int N = b.nxp - 1, px = b.px;
    const size_t lay = (size_t)k * b.nyp * px;
    auto row = [&](const void *f, int d) { return (const T *)f + lay + (size_t)(side ? b.nyp - 1 - d : d) * px; };
    const T *p1 = row(b.F[par], 1), *q0 = row(b.F[2 + par], 0), *q1 = row(b.F[2 + par], 1);
    const T *m0 = row(b.F[1 - par], 0), *m1 = row(b.F[1 - par], 1), *m2 = row(b.F[1 - par], 2), *m3 = row(b.F[1 - par], 3);
    const T fx = (T)b.fx, fy = (T)b.fy, fyb = (T)b.fy_bc;
    const bool qa = q_anom_stored<T>();
    const double by0 = qa ? b.beta * b.yprel[side ? b.nyp - 1 : 0] : 0.0;
    const double by1 = qa ? b.beta * b.yprel[side ? b.nyp - 2 : 1] : 0.0;
    double s[OQG_NSTRIP];
#pragma unroll
    for (int x = 0; x < OQG_NSTRIP; ++x) s[x] = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        auto wrap = [&](int c) { return c < 0 ? c + N : c >= N ? c - N : c; };
        const int w2 = wrap(i - 2), w1 = wrap(i - 1), e1 = wrap(i + 1), e2 = wrap(i + 2);
        const double dp = (double)(p1[e1] - p1[w1]);
        s[0] += ((double)q0[i] + by0) * dp;
        s[1] += ((double)q1[i] + by1) * dp;
        auto lap = [&](T w, T e, T sv, T nv, T c) { return fx * (w + e - (T)2 * c) + fy * (sv + nv - (T)2 * c); };
        const T d20 = fyb * (m1[i] - m0[i]);
        const T d21 = lap(m1[w1], m1[e1], m0[i], m2[i], m1[i]);
        const T d21w = lap(m1[w2], m1[i], m0[w1], m2[w1], m1[w1]), d21e = lap(m1[i], m1[e2], m0[e1], m2[e1], m1[e1]);
        const T d22 = lap(m2[w1], m2[e1], m1[i], m3[i], m2[i]);
        const T d40 = fyb * (d21 - d20), d41 = lap(d21w, d21e, d20, d22, d21);
        s[2] += (double)(d21 - d20);
        s[3] += (double)(d41 - d40);
        if (k == b.kt) s[4] += (double)(m1[i] - m0[i]);
    }
    __shared__ double red[OQG_NSTRIP][2 * VWIDE];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int x = 0; x < OQG_NSTRIP; ++x) s[x] += __shfl_down_sync(0xffffffffu, s[x], o);
    if ((threadIdx.x & 31) == 0)
#pragma unroll
        for (int x = 0; x < OQG_NSTRIP; ++x) red[x][threadIdx.x >> 5] = s[x];
    __syncthreads();
    if (threadIdx.x < OQG_NSTRIP) {
        const int x = threadIdx.x;
        double v = red[x][0];
        for (int u = 1; u < (int)blockDim.x / 32; ++u) v += red[x][u];
        if (side && x >= 2) v = -v;
        b.part_tile[((size_t)side * b.nl + k) * OQG_NSTRIP + x] = v;
    }
}

// tdt = 0: each member steps with its own b.tdt_m (ensemble launches).
// VT: the tile's rows (b.vty), a compile-time multiple of 4 (vort_tile_rows),
// so every strip's row loop has a fixed trip count: the loops unroll with no
// predicates and the rolling windows live in renamed registers.
// NS row strips of 64 threads: VSTRIPS, or VWIDE where the tiles are no more
// than the SMs, so that a CTA has its SM to itself: the rows a thread marches
// in each phase halve.
// SPLIT: a tile is shared by a cluster of NL CTAs, one per layer; they exchange
// the stepped q through distributed shared memory, and CTA m forms mode m's
// right-hand side.  For single basins with few tiles, where the time is one
// CTA's chain of NL layers.
template <class T, int NL, int VT, int NS, bool SPLIT>
__global__ void __launch_bounds__(64 * NS, NS == VSTRIPS ? 2 : 1)
k_vort(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int par, double tdt) {
    static_assert(VT % NS == 0 && VT >= 8 && VT <= VTYMAX, "tile rows: a multiple of the strips in [8, VTYMAX]");
    constexpr int LPQ = VTX + 8, L2 = VTX + 4, L1 = VTX + 2, LO = VTX;
    constexpr int HPM = VT + 6, H2 = VT + 4, H1 = VT + 2;
    // rows per strip of each phase; the last strips of d2 and d4 start early
    // and recompute a row or two of their neighbours (the same values)
    constexpr int RMAX = VT / NS, R2MAX = (H2 + NS - 1) / NS, R1MAX = (H1 + NS - 1) / NS;
    Work w;
    if constexpr (SPLIT) w = Work{0, (int)blockIdx.x};
    else w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    const int strips = vort_strips(NL, b.cyclic);
    if (w.block < strips) {
        // (a whole number of clusters: 2 NL)
        pdl_trigger();
        pdl_wait();
        vort_strip<T>(b, w.block / NL, w.block % NL, par);
        return;
    }
    // uniform constants in shared memory: fx fy fxb fyb jac | c_ent1 c_wind
    // c_ent2 c_drag tdt | c2[k] | c4[k]; FP64 ctl2m
    __shared__ T sK[11 + 2 * OQG_NLMAX];
    __shared__ double sCtl[NL * NL];
    // FP32 storage keeps q as its anomaly q - beta yprel (q_anom_stored): the
    // planetary term's Jacobian then comes from p alone (its coefficient,
    // jac_fac beta dy, is sK[10 + 2 NL])
    constexpr bool QA = q_anom_stored<T>();
    if (QA && threadIdx.x == 10 + 2 * NL) sK[10 + 2 * NL] = (T)(b.jac_fac * b.beta * b.dy);
    if (threadIdx.x < 10 + 2 * NL) {
        const int i = threadIdx.x;
        T v;
        if (i == 0) v = (T)b.fx; else if (i == 1) v = (T)b.fy; else if (i == 2) v = (T)b.fx_bc;
        else if (i == 3) v = (T)b.fy_bc; else if (i == 4) v = (T)b.jac_fac; else if (i == 5) v = (T)b.c_ent1;
        else if (i == 6) v = (T)b.c_wind; else if (i == 7) v = (T)b.c_ent2; else if (i == 8) v = (T)b.c_drag;
        else if (i == 9) v = (T)(tdt != 0.0 ? tdt : b.tdt_m); else if (i < 10 + NL) v = (T)b.c2[i - 10]; else v = (T)b.c4[i - 10 - NL];
        sK[i] = v;
    }
    if (threadIdx.x < NL * NL) sCtl[threadIdx.x] = b.ctl2m[threadIdx.x];
    GeoS<T> g;
    g.nxp = b.nxp; g.nyp = b.nyp; g.cyclic = b.cyclic; g.K = sK;
    const VortLayout LY = vort_layout(VT, (int)sizeof(T));
    const int tile = (w.block - strips) / (SPLIT ? NL : 1), tile_y = tile / b.tiles_x, tile_x = tile - tile_y * b.tiles_x;
    // the layers of this CTA
    const int kb = SPLIT ? (w.block - strips) % NL : 0, ke = SPLIT ? kb + 1 : NL;
    const int i0 = tile_x * VTX, j0 = tile_y * VT + 1;

    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *sm = reinterpret_cast<T *>(((uintptr_t)smem_raw + 127) & ~(uintptr_t)127);
    T *sD2 = sm + LY.d2;
    T *sD4 = sm + LY.d4;
    T *sWK = sm + LY.wk;
    double *sBY = reinterpret_cast<double *>(sm + LY.by);
    __shared__ __align__(8) unsigned long long bars[2];

    T *QM = (T *)b.F[3 - par];
    const T *ENT = (const T *)b.ent;
    const double *__restrict__ DD = b.ddyn;
    const int nyp = g.nyp, nxp = g.nxp, px = b.px, kt = b.kt;
    const int tx = threadIdx.x & 63, ty = threadIdx.x >> 6;
    // a channel's halo tile must lie in its N = nxp - 1 distinct columns as stored
    const bool tma = b.tmaps != nullptr && (!g.cyclic || (i0 >= 4 && i0 + VTX + 4 <= nxp - 1));
    const unsigned char *tm = (const unsigned char *)b.tmaps;

    if (tma && threadIdx.x == 0) {
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        mbar_init_fence();
    }
    // beta * yprel of the tile's rows (constant)
    for (int r = threadIdx.x; r < VT; r += blockDim.x) {
        const int gj = j0 + r;
        sBY[r] = gj < nyp ? b.beta * b.yprel[gj] : 0.0;
    }
    __syncthreads();
    pdl_trigger();
    pdl_wait();

    auto issue = [&](int k) {
        T *bf = sm + ((k - kb) & 1) * LY.nbuf;
        if (tma) {
            if (threadIdx.x == 0) {
                fence_proxy_async();
                unsigned bytes = (unsigned)((HPM * LPQ + 2 * H1 * LPQ + VT * LO) * sizeof(T));
                if (k == 0) bytes += (unsigned)(VT * LO * sizeof(T));
                unsigned long long *bar = &bars[(k - kb) & 1];
                mbar_expect_tx(bar, bytes);
                tma_load_3d(bf + LY.pm, tm + (OQG_TMAP_PM + 1 - par) * OQG_TMAP_BYTES, i0 - 4, j0 - 3, k, bar);
                tma_load_3d(bf + LY.p, tm + (OQG_TMAP_PQ + par) * OQG_TMAP_BYTES, i0 - 4, j0 - 1, k, bar);
                tma_load_3d(bf + LY.q, tm + (OQG_TMAP_PQ + 2 + par) * OQG_TMAP_BYTES, i0 - 4, j0 - 1, k, bar);
                tma_load_3d(bf + LY.qm, tm + (OQG_TMAP_QM + 1 - par) * OQG_TMAP_BYTES, i0, j0, k, bar);
                if (k == 0) tma_load_2d(sWK, tm + OQG_TMAP_WK * OQG_TMAP_BYTES, i0, j0, bar);
            }
        } else {
            load_tile_async(bf + LY.pm, (const T *)b.F[1 - par], g, px, k, j0 - 3, HPM, i0 - 4, LPQ);
            load_tile_async(bf + LY.p, (const T *)b.F[par], g, px, k, j0 - 1, H1, i0 - 4, LPQ);
            load_tile_async(bf + LY.q, (const T *)b.F[2 + par], g, px, k, j0 - 1, H1, i0 - 4, LPQ);
            load_tile_async(bf + LY.qm, (const T *)QM, g, px, k, j0, VT, i0, LO, true);
            if (k == 0) load_tile_async(sWK, (const T *)b.wekp, g, px, 0, j0, VT, i0, LO, true);
            cp_async_commit();
        }
    };
    issue(kb);

    // strips of rows: [ty*R, ty*R + R) of each region
    constexpr int R2 = R2MAX, R1 = R1MAX, R0 = RMAX;
    const int r0 = ty * R0;
    double acc[RMAX][NL];
#pragma unroll
    for (int u = 0; u < RMAX; ++u)
#pragma unroll
        for (int m = 0; m < NL; ++m) acc[u][m] = 0.0;
    const bool topo = b.topo_active != 0;
    // in-domain test of a column (a channel has none outside)
    auto colok = [&](int gi) { return g.cyclic || (gi >= 0 && gi < nxp); };
    // the del2 region (rows j0-2 .. j0+VT+1, columns i0-2 .. i0+VTX+1) lies
    // strictly inside the walls, and every output column exists
    const bool interior = (j0 - 2 >= 1 && j0 + VT + 1 <= nyp - 2) &&
                          (g.cyclic ? (i0 + VTX <= nxp) : (i0 - 2 >= 1 && i0 + VTX + 1 <= nxp - 2));

    // SPLIT: the stepped q less the planetary and topographic parts, for the
    // cluster; otherwise summed over the layers in registers
    __shared__ double sQL[SPLIT ? VT * LO : 1];
    bool lost = false;
#pragma unroll 1
    for (int k = kb; k < ke; ++k) {
        if (k + 1 < ke) issue(k + 1);
        if (tma) {
            // one thread polls the barrier; the CTA barrier then publishes
            // the tile to the others without spinning warps taking issue slots
            bool ok = true;
            if (threadIdx.x == 0) ok = mbar_wait_bounded(&bars[(k - kb) & 1], ((k - kb) >> 1) & 1, b.wait_limit);
            if (__syncthreads_or(!ok)) {
                // a tile never arrived: report, drain what is in flight, stop
                if (threadIdx.x == 0) {
                    atomicOr(b.err, OQG_DERR_TIMEOUT);
                    mbar_wait_bounded(&bars[(k - kb) & 1], ((k - kb) >> 1) & 1, OQG_WAIT_LIMIT);
                    if (k + 1 < ke) mbar_wait_bounded(&bars[(k + 1 - kb) & 1], ((k + 1 - kb) >> 1) & 1, OQG_WAIT_LIMIT);
                }
                __syncthreads();
                // (a cluster's other CTAs wait at its barriers below)
                if constexpr (!SPLIT) return;
                lost = true;
                break;
            }
        } else {
            if (k + 1 < ke) cp_async_wait<1>();
            else cp_async_wait<0>();
            __syncthreads();
        }
        const T *sPM = sm + ((k - kb) & 1) * LY.nbuf + LY.pm;
        const T *sP = sm + ((k - kb) & 1) * LY.nbuf + LY.p;
        const T *sQ = sm + ((k - kb) & 1) * LY.nbuf + LY.q;
        const T *sQM = sm + ((k - kb) & 1) * LY.nbuf + LY.qm;
        // The layer's stencils; I: every point of the tile and its halo is
        // off the walls, so the wall rules and range tests drop out.
        auto layer = [&](auto inner) {
            constexpr bool I = decltype(inner)::value;
            const T fx = gfx(g), fy = gfy(g), fxb = gfxb(g), fyb = gfyb(g);
            // ---- del2(pm) on rows j0-2.., cols i0-2.. (column tx of L2 = 64)
            {
                const int gi = i0 - 2 + tx, cs = tx + 2;          // column in the pm tile
                const bool cv = colok(gi);
                const bool wl = !g.cyclic && gi == 0, wr = !g.cyclic && gi == nxp - 1;
                const int rb = min(ty * R2, H2 - R2);
                const T *col = sPM + rb * LPQ + cs;
                T sv = col[0], cv_ = col[LPQ];
    #pragma unroll
                for (int u = 0; u < R2MAX; ++u) {
                    const int r = rb + u;
                    {
                        const T nv = col[(u + 2) * LPQ];
                        const T wv = col[(u + 1) * LPQ - 1], ev = col[(u + 1) * LPQ + 1];
                        const int gj = j0 - 2 + r;
                        T v = (T)0;
                        if (I) v = fx * (wv + ev - (T)2 * cv_) + fy * (sv + nv - (T)2 * cv_);
                        else if (cv && gj >= 0 && gj < nyp)
                            v = lap5_sel(wv, ev, sv, nv, cv_, gj == 0 || gj == nyp - 1, wl, wr, gj == 0,
                                         gj == nyp - 1, fx, fy, fxb, fyb);
                        sD2[r * L2 + tx] = v;
                        sv = cv_;
                        cv_ = nv;
                    }
                }
            }
            __syncthreads();
            // ---- del4 on rows j0-1.., cols i0-1.. (column tx < L1 = 62)
            if (tx < L1) {
                const int gi = i0 - 1 + tx, cs = tx + 1;          // column in the d2 tile
                const bool cv = colok(gi);
                const bool wl = !g.cyclic && gi == 0, wr = !g.cyclic && gi == nxp - 1;
                const int rb = min(ty * R1, H1 - R1);
                const T *col = sD2 + rb * L2 + cs;
                T sv = col[0], cv_ = col[L2];
    #pragma unroll
                for (int u = 0; u < R1MAX; ++u) {
                    const int r = rb + u;
                    {
                        const T nv = col[(u + 2) * L2];
                        const T wv = col[(u + 1) * L2 - 1], ev = col[(u + 1) * L2 + 1];
                        const int gj = j0 - 1 + r;
                        T v = (T)0;
                        if (I) v = fx * (wv + ev - (T)2 * cv_) + fy * (sv + nv - (T)2 * cv_);
                        else if (cv && gj >= 0 && gj < nyp)
                            v = lap5_sel(wv, ev, sv, nv, cv_, gj == 0 || gj == nyp - 1, wl, wr, gj == 0,
                                         gj == nyp - 1, fx, fy, fxb, fyb);
                        sD4[r * L1 + tx] = v;
                        sv = cv_;
                        cv_ = nv;
                    }
                }
            }
            __syncthreads();

            // ---- outputs: column tx < VTX, rows r0 .. r0+R0-1 of the tile.
            // Only points off the solid walls are stepped: on a wall the Arakawa
            // Jacobian is zero and the stepped q is replaced by ocqbdy
            // (vorsubs.F90:58-114) in the assembly kernel, so the interior
            // stencils are the whole computation here.
            if (tx < VTX) {
                const int gi = i0 + tx;
                const bool xin = g.cyclic ? (gi < nxp) : (gi >= 1 && gi <= nxp - 2);
                const T *d4col = sD4 + r0 * L1 + tx + 1;       // column in the d4 tile
                const T *pcol = sP + r0 * LPQ + tx + 4;         // column in the p/q tiles
                const T *qcol = sQ + r0 * LPQ + tx + 4;
                // rolling windows: d4 (column), p and q (3 x 3)
                T d4s = d4col[0], d4c = d4col[L1];
                T pw[3][3], qw[3][3];
    #pragma unroll
                for (int a = 0; a < 2; ++a)
    #pragma unroll
                    for (int cc = 0; cc < 3; ++cc) {
                        pw[a + 1][cc] = pcol[a * LPQ - 1 + cc];
                        qw[a + 1][cc] = qcol[a * LPQ - 1 + cc];
                    }
    #pragma unroll
                for (int u = 0; u < RMAX; ++u) {
                    const int r = r0 + u;
                    const int gj = j0 + r;
                    {
                        // shift the windows down one row and load the new bottom row
                        const T d4n = d4col[(u + 2) * L1];
                        const T d4w = d4col[(u + 1) * L1 - 1], d4e = d4col[(u + 1) * L1 + 1];
    #pragma unroll
                        for (int cc = 0; cc < 3; ++cc) {
                            pw[0][cc] = pw[1][cc]; pw[1][cc] = pw[2][cc];
                            qw[0][cc] = qw[1][cc]; qw[1][cc] = qw[2][cc];
                            pw[2][cc] = pcol[(u + 2) * LPQ - 1 + cc];
                            qw[2][cc] = qcol[(u + 2) * LPQ - 1 + cc];
                        }
                        if (I || (xin && gj >= 1 && gj <= nyp - 2)) {
                            const T d6 = fx * (d4w + d4e - (T)2 * d4c) + fy * (d4s + d4n - (T)2 * d4c);
                            // Arakawa J(q, p), numerics.F90:370-372
                            const T pxc = pw[1][2] - pw[1][0], pyc = pw[2][1] - pw[0][1];
                            const T qxc = qw[1][2] - qw[1][0], qyc = qw[2][1] - qw[0][1];
                            const T A = qw[1][2] * (pw[2][2] - pw[0][2]) - qw[1][0] * (pw[2][0] - pw[0][0]);
                            const T Dd = pw[1][2] * (qw[2][2] - qw[0][2]) - pw[1][0] * (qw[2][0] - qw[0][0]);
                            const T Bv = qw[2][1] * (pw[2][2] - pw[2][0]) - qw[0][1] * (pw[0][2] - pw[0][0]);
                            const T Cc = pw[2][1] * (qw[2][2] - qw[2][0]) - pw[0][1] * (qw[0][2] - qw[0][0]);
                            T jac = gjac(g) * (qxc * pyc - qyc * pxc + A - Bv + Cc - Dd);
                            if (QA) {
                                // + J(beta y, p): the Arakawa sum of a field linear in y is
                                // -dy (4 (pE - pW) + (pNE - pNW) + (pSE - pSW)); explicit FMAs
                                // fix this part's rounding
                                const T py = fma((T)4, pxc, (pw[2][2] - pw[2][0]) + (pw[0][2] - pw[0][0]));
                                jac = fma(-sK[10 + 2 * NL], py, jac);
                            }
                            T dq = jac + sK[10 + k] * d4c - sK[10 + NL + k] * d6;
                            const size_t o2 = (size_t)gj * px + gi;
                            if (k == 0) {
                                const T e1 = ENT ? ldg(ENT + o2) : (T)0;
                                dq = dq + sK[5] * e1 + sK[6] * sWK[r * LO + tx];
                            }
                            if (k == 1 && ENT) dq = dq - sK[7] * ldg(ENT + o2);
                            if (k == kt) dq = dq - sK[8] * sD2[(r + 2) * L2 + tx + 2];
                            const T qn = sQM[r * LO + tx] + sK[9] * dq;
                            QM[((size_t)k * nyp + gj) * px + gi] = qn;
                            // modal right-hand side, FP64 (p_modes_rhs)
                            double ql = QA ? (double)qn : (double)qn - sBY[r];
                            if (k == kt && topo) ql -= DD[o2];
                            if constexpr (SPLIT) sQL[r * LO + tx] = ql;
                            else
    #pragma unroll
                                for (int m = 0; m < NL; ++m) acc[u][m] += ql * sCtl[k + NL * m];
                        }
                        d4s = d4c;
                        d4c = d4n;
                    }
                }
            }
        };
        if (interior) layer(std::true_type{});
        else layer(std::false_type{});
        __syncthreads();
    }

    // write the modal right-hand side of the interior points
    T *RHS = (T *)b.rhs;
    const int ioff = g.cyclic ? 0 : 1;
    const double f0 = b.fnot;
    if constexpr (SPLIT) {
        cluster_sync();
        if (tx < VTX && !lost) {
            double v[RMAX][NL];
#pragma unroll
            for (int l = 0; l < NL; ++l)
#pragma unroll
                for (int u = 0; u < RMAX; ++u) v[u][l] = ld_cluster(&sQL[(r0 + u) * LO + tx], l);
#pragma unroll
            for (int u = 0; u < RMAX; ++u) {
                const int r = r0 + u, gj = j0 + r, xi = i0 + tx - ioff;
                if (gj < 1 || gj > nyp - 2 || xi < 0 || xi >= b.nxin) continue;
                double s = 0.0;
#pragma unroll
                for (int l = 0; l < NL; ++l) s += v[u][l] * sCtl[l + NL * kb];
                RHS[((size_t)kb * b.ny + (gj - 1)) * b.pr + xi] = (T)(f0 * s);
            }
        }
        cluster_sync();               // no CTA leaves while its tile may be read
        return;
    }
    if (tx < VTX) {
#pragma unroll
        for (int u = 0; u < RMAX; ++u) {
            const int r = r0 + u;
            const int gj = j0 + r, gi = i0 + tx;
            if (gj < 1 || gj > nyp - 2) continue;
            const int xi = gi - ioff;
            if (xi < 0 || xi >= b.nxin) continue;
#pragma unroll
            for (int m = 0; m < NL; ++m)
                RHS[((size_t)m * b.ny + (gj - 1)) * b.pr + xi] = (T)(f0 * acc[u][m]);
        }
    }
}

// ------------------------------------------------------------------ k_xfwd
// Threads per transform TT = ceil(M/E); G = blockDim/TT transforms per CTA.
// Shared memory: per group two padded buffers of fft_buf_len(M) complex
// values; the input rows are staged by cp.async into the second buffer and
// expanded into the first.  The stage twiddles are read from global memory.
__host__ __device__ __forceinline__ int round16(int bytes) { return (bytes + 15) & ~15; }

// A channel's forward transform (r2c of two rows by one complex FFT).  MC > 0:
// an instance for transforms of length MC only (the host picks it for a basin
// of that length); MC = 0 serves any length (ensembles).  G: transforms per
// CTA (<= 0: an ensemble, as many as the CTA's threads serve).
template <class T, int E, int MC = 0>
__global__ void __launch_bounds__(256, 2)
k_xfwd(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int G) {
    typedef typename C2<T>::t T2;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int M = MC > 0 ? MC : b.M, TT = (M + E - 1) / E;
    if (G <= 0) G = blockDim.x / TT;
    const int g = threadIdx.x / TT, t = threadIdx.x - g * TT;
    const int LB = fft_buf_len(M);
    T2 *zs = reinterpret_cast<T2 *>(smem_raw);
    const int npm = (b.ny + 1) >> 1;          // row pairs per mode
    const int pair = w.block * G + g;
    const bool live = g < G && pair < b.nl * npm;
    const int m = live ? pair / npm : 0;
    const int j = live ? 2 * (pair - m * npm) : 0;
    const bool two = live && (j + 1 < b.ny);
    const int n = b.nxin;
    const int RO = (n + 3) & ~3;              // offset of the second row (16-byte aligned)
    // the input rows are staged in the second buffer
    T2 *za = zs + (size_t)(g < G ? g : 0) * 2 * LB;
    T2 *zb = za + LB;
    T *raw = reinterpret_cast<T *>(zb);
    const T *x = (const T *)b.rhs + ((size_t)m * b.ny + j) * b.pr;
    pdl_trigger();
    pdl_wait();
    if (live) {
        cp_async_16(raw, x, round16(n * (int)sizeof(T)), t, TT);
        if (two) cp_async_16(raw + RO, x + b.pr, round16(n * (int)sizeof(T)), t, TT);
    }
    cp_async_commit_wait_all();
    __syncthreads();
    if (live) {
        for (int jj = t; jj < M; jj += TT) {
            T2 v;
            v.x = raw[jj];
            v.y = two ? raw[RO + jj] : (T)0;
            za[fpad(jj)] = v;
        }
    }
    __syncthreads();
    const T2 *z = fft_run<T, E, MC>(za, zb, M, b.rad, b.nrad, b.fd_ns, (const T2 *)b.tw, live ? t : TT, TT, 0, 0);
    if (!live) return;
    T2 *S = (T2 *)b.spec;
    T2 *sx = S + ((size_t)m * b.ny + j) * b.pk;
    T2 *sy = sx + b.pk;
    for (int kk = t; kk < b.nk; kk += TT) {
        const T2 a = z[fpad(kk)], c = z[fpad((M - kk) % M)];
        T2 X, Y;
        X.x = (T)0.5 * (a.x + c.x);
        X.y = (T)0.5 * (a.y - c.y);
        // (a - conj(c)) / (2i)
        const T dx_ = (T)0.5 * (a.x - c.x), dy_ = (T)0.5 * (a.y + c.y);
        Y.x = dy_;
        Y.y = -dx_;
        sx[kk] = X;
        if (two) sy[kk] = Y;
    }
}

// ------------------------------------------------------------------ k_bfwd
// Stages a row pair x, y (n values each, times f) as the complex input of one
// box transform (oqg_odd.cuh): value i at zpad<4>(i + 1), zero at both ends.
// Eight loads of each row are in flight per thread; they bypass L1 (every
// value is read once).
template <class T>
__device__ __forceinline__ void odd_stage_rows(typename C2<T>::t *z, const T *__restrict__ x, const T *__restrict__ y,
                                               bool two, int n, T f, int t, int TT) {
    constexpr int U = 8;
    typename C2<T>::t zero;
    zero.x = zero.y = (T)0;
    if (t == 0) { z[0] = zero; z[zpad<4>(n + 1)] = zero; }
    for (int i0 = t; i0 < n; i0 += U * TT) {
        T a[U], c[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * TT;
            a[u] = i < n ? __ldcg(x + i) : (T)0;
            c[u] = two && i < n ? __ldcg(y + i) : (T)0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = i0 + u * TT;
            typename C2<T>::t v;
            v.x = f * a[u];
            v.y = f * c[u];
            if (i < n) z[zpad<4>(i + 1)] = v;
        }
    }
}

// A box's forward transform: DST-I of the modal right-hand side's row pairs
// (oqg_odd.cuh).  A CTA holds G transforms (G <= 0, an ensemble: as many as
// its threads serve), numbered with the mode fastest.
template <class T, int MC = 0>
__global__ void __launch_bounds__(256, 2)
k_bfwd(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int G) {
    typedef typename C2<T>::t T2;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int M = MC > 0 ? MC : b.M, TT = odd_tt(M);
    if (G <= 0) G = blockDim.x / TT;
    const int g = threadIdx.x / TT, t = threadIdx.x - g * TT;
    const int npm = (b.ny + 1) >> 1;          // row pairs per mode
    const int tr = w.block * G + g;
    const bool live = g < G && tr < b.nl * npm;
    const int pair = live ? tr / b.nl : 0, m = live ? tr - pair * b.nl : 0, j = 2 * pair;
    const bool two = j + 1 < b.ny;
    T2 *z = reinterpret_cast<T2 *>(smem_raw) + (size_t)(g < G ? g : 0) * odd_smem_len(M);
    const T *x = (const T *)b.rhs + ((size_t)m * b.ny + j) * b.pr;
    T *sx = (T *)b.spec + ((size_t)m * b.ny + j) * b.pk, *sy = sx + b.pk;
    pdl_trigger();
    pdl_wait();
    if (live) odd_stage_rows<T>(z, x, x + b.pr, two, b.nxin, (T)1, t, TT);
    __syncthreads();
    odd_fft<T, MC>(z, M, b, (const T2 *)b.otw, t, TT, live, [&](int i, T2 v) {
        sx[i - 1] = -v.y;
        if (two) sy[i - 1] = v.x;
    });
}

// ------------------------------------------------------------------ k_ysolve
// Thomas solves in y (inhomog.F90:187-199), one column per (mode, wavenumber).
// The lanes of a warp lie along the wavenumber: KB adjacent columns times 32 / KB
// chunks of R rows, and a column's values stay in the registers of its threads
// from load to store.  A row's access is KB values: 64 bytes of FP64 (32 of FP32)
// up to 1024 rows of a box, half of that up to 2048, where an FP32 row is then
// half of its 32-byte sector, a quarter up to 4096, and one value above; a
// channel's complex values are 64 bytes (32) up to 2048 rows, half above.  Both substitutions are affine recurrences with the same
// coefficients e_j = -a beta_j:
//   down   u_j = beta_j f_j + e_j u_{j-1},   up   w_j = u_j + e_j w_{j+1}.
// A thread runs its R rows from a zero input (v_j) and keeps the products
// P_j = e_s .. e_j; then u_j = v_j + P_j u_in, and the chunk's map of the up
// sweep is known at once: w_s = sum P_{j-1} v_j + u_in sum P_{j-1} P_j + P w_in.
// The chunk maps are scanned across the lanes by shuffles and across the warps
// of a column group through shared memory (two barriers in all).
//
// Bound by latency: a thread's two serial passes over its rows and the scans;
// above 1024 rows one CTA of 512 threads fills an SM, and no load overlaps
// another group's passes.  Per launch 11.2 us at 513^2 and 93 us at 2049^2 FP64
// (91 in FP32 storage); staging four columns per CTA in shared memory with the
// lanes along y took 14.5 and 147 us (132).
template <class T, bool CPLX> struct YT;
template <class T> struct YT<T, false> { typedef double v; typedef T g; };
template <class T> struct YT<T, true> { typedef double2 v; typedef typename C2<T>::t g; };

__device__ __forceinline__ double yt_zero(double) { return 0.0; }
__device__ __forceinline__ double2 yt_zero(double2) { return make_double2(0.0, 0.0); }
// c + d x
__device__ __forceinline__ double yt_axpy(double c, double d, double x) { return fma(d, x, c); }
__device__ __forceinline__ double2 yt_axpy(double2 c, double d, double2 x) {
    return make_double2(fma(d, x.x, c.x), fma(d, x.y, c.y));
}
__device__ __forceinline__ double yt_scale(double f, double s) { return f * s; }
__device__ __forceinline__ double2 yt_scale(double2 f, double s) { return make_double2(f.x * s, f.y * s); }
__device__ __forceinline__ double yt_up(double v, int o) { return shfl_up_d(v, o); }
__device__ __forceinline__ double2 yt_up(double2 v, int o) { return make_double2(shfl_up_d(v.x, o), shfl_up_d(v.y, o)); }
__device__ __forceinline__ double yt_dn(double v, int o) { return shfl_dn_d(v, o); }
__device__ __forceinline__ double2 yt_dn(double2 v, int o) { return make_double2(shfl_dn_d(v.x, o), shfl_dn_d(v.y, o)); }
__device__ __forceinline__ double yt_load(float v) { return (double)v; }
__device__ __forceinline__ double yt_load(double v) { return v; }
__device__ __forceinline__ double2 yt_load(float2 v) { return make_double2(v.x, v.y); }
__device__ __forceinline__ double2 yt_load(double2 v) { return v; }
template <class G> __device__ __forceinline__ G yt_store(double v) { return (G)v; }
template <class G> __device__ __forceinline__ G yt_store(double2 v) {
    G g;
    g.x = v.x;
    g.y = v.y;
    return g;
}

#define YS_THREADS 512      // most threads of a CTA
#define YS_PIVB 8           // columns of a pivot-table block
#define YS_ROWS 16          // most rows per thread (values and pivots in registers)
// Columns per group: 64 bytes of FP64, fewer when the rows need more threads.
__host__ __device__ __forceinline__ int ysolve_kb(int ny, int cplx) {
    for (int k = cplx ? 4 : 8; k > 1; k /= 2)
        if ((ny + YS_ROWS - 1) / YS_ROWS * k <= YS_THREADS) return k;
    return 1;
}
// Rows per thread of a column spread over about 25 W chunks: W = 1, 2, 4 trade
// the length of a thread's chain for threads.  At W = 2 a step took (us, rows
// 4 / 8 / 16): 257^2 29.8 / 30.0 / 30.6, 361 x 287 - / 42.7 / 43.7, 513^2
// - / 51.4 / 50.2; 32 rows do not fit the registers (1025^2: 168 against 147
// with 16).  A channel's complex values spill 160-224 bytes per thread at 16
// rows: 8 against 16 rows 67.2 / 72.1 at 769 x 481 (FP32 storage 53.3 / 56.4),
// 81.2 / 83.9 at 641^2, but 123.9 / 121.9 at 1025 x 801 (93.5 / 95.3), so the
// boxes' rule serves both, and oqg_autotune_ysolve finds the 8 rows of spread 4.
__host__ __device__ __forceinline__ int ysolve_rows(int ny, int cplx, int W) {
    const int kb = ysolve_kb(ny, cplx);
    int R = 4;
    while (R < YS_ROWS && (R * 25 * W < ny || (ny + R - 1) / R * kb > YS_THREADS)) R *= 2;
    return R;
}
// Warps of a group of kb columns.
__host__ __device__ __forceinline__ int ysolve_group_warps(int ny, int R, int kb) {
    return ((ny + R - 1) / R * kb + 31) / 32;
}

template <class T, bool CPLX, int R, int KB>
__global__ void __launch_bounds__(YS_THREADS, 1)
k_ysolve(const BasinDev *__restrict__ bas, const Work *__restrict__ work) {
    typedef typename YT<T, CPLX>::v V;
    typedef typename YT<T, CPLX>::g Gm;
    constexpr int MAXW = YS_THREADS / 32;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int nk = b.nk, ny = b.ny, pk = b.pk, nl = b.nl;
    const int WG = ysolve_group_warps(ny, R, KB), G = max(1, (int)(blockDim.x >> 5) / WG);
    const int g = wid / WG, wg = wid - g * WG;  // group of the CTA, warp within it
    const int ncb = (nk + KB - 1) / KB, cb = w.block * G + g;
    const bool live = g < G && cb < nl * ncb;
    const int m = live ? cb / ncb : 0, k0 = live ? (cb - m * ncb) * KB : 0;
    const int col = lane % KB, rc = lane / KB, k = k0 + col;
    const int s = (wg * (32 / KB) + rc) * R;    // this thread's first row
    const bool on = live && k < nk;
    __shared__ V sC[2][MAXW][KB];
    __shared__ double sD[2][MAXW][KB];
    __shared__ double part[2][MAXW];
    // pivots of the table block's columns, [plen][YS_PIVB]; beyond the stored
    // length a pivot repeats its fixed point
    const int pb = m * ((nk + YS_PIVB - 1) / YS_PIVB) + k0 / YS_PIVB;
    const int plen = b.piv_len[pb];
    const double *__restrict__ piv = b.piv_tab + b.piv_off[pb] + k0 % YS_PIVB + col;
    const double a = b.a_tri;
    const bool flat = s >= plen - 1;            // every row of the thread has the fixed point
    const double bt0 = __ldg(piv + (size_t)min(s, plen - 1) * YS_PIVB);
    double bt[R];                               // zero, as the value, in rows at or beyond ny
#pragma unroll
    for (int t = 0; t < R; ++t)
        bt[t] = s + t >= ny ? 0.0 : flat ? bt0 : __ldg(piv + (size_t)min(s + t, plen - 1) * YS_PIVB);
    Gm *S = (Gm *)b.spec + ((size_t)m * ny + s) * pk + k;
    pdl_trigger();
    pdl_wait();
    V x[R];
    {
        Gm raw[R];
#pragma unroll
        for (int t = 0; t < R; ++t)
            if (on && s + t < ny) raw[t] = __ldcg(S + (size_t)t * pk);
#pragma unroll
        for (int t = 0; t < R; ++t) x[t] = on && s + t < ny ? yt_load(raw[t]) : yt_zero(V());
    }
    // the chunk from a zero input, and its map of the up sweep
    V v = yt_zero(V()), A = yt_zero(V());
    double P = 1.0, S2 = 0.0;
#pragma unroll
    for (int t = 0; t < R; ++t) {
        const double be = bt[t], e = -a * be;
        v = yt_axpy(yt_scale(x[t], be), e, v);
        x[t] = v;
        A = yt_axpy(A, P, v);
        const double Pn = P * e;
        S2 = fma(P, Pn, S2);
        P = Pn;
    }
    // scan down: C + D u over the chunks above
    V u;
    {
        V C = v;
        double D = P;
#pragma unroll
        for (int o = KB; o < 32; o <<= 1) {
            const V Co = yt_up(C, o);
            const double Do = shfl_up_d(D, o);
            if (lane >= o) { C = yt_axpy(C, D, Co); D *= Do; }
        }
        V Ce = yt_up(C, KB);
        double De = shfl_up_d(D, KB);
        if (rc == 0) { Ce = yt_zero(V()); De = 1.0; }
        if (lane >= 32 - KB) { sC[0][wid][col] = C; sD[0][wid][col] = D; }
        __syncthreads();
        u = yt_zero(V());
        const int w0 = wid - wg;
        for (int y = 0; y < wg; ++y) u = yt_axpy(sC[0][w0 + y][col], sD[0][w0 + y][col], u);
        u = yt_axpy(Ce, De, u);
    }
    // scan up: the chunks below
    V win;
    {
        V C = yt_axpy(A, S2, u);
        double D = P;
#pragma unroll
        for (int o = KB; o < 32; o <<= 1) {
            const V Co = yt_dn(C, o);
            const double Do = shfl_dn_d(D, o);
            if (lane + o < 32) { C = yt_axpy(C, D, Co); D *= Do; }
        }
        V Ce = yt_dn(C, KB);
        double De = shfl_dn_d(D, KB);
        if (rc == 32 / KB - 1) { Ce = yt_zero(V()); De = 1.0; }
        if (lane < KB) { sC[1][wid][col] = C; sD[1][wid][col] = D; }
        __syncthreads();
        win = yt_zero(V());
        const int w0 = wid - wg;
        for (int y = WG - 1; y > wg; --y)
            if (w0 + y < MAXW) win = yt_axpy(sC[1][w0 + y][col], sD[1][w0 + y][col], win);
        win = yt_axpy(Ce, De, win);
    }
    P = 1.0;
#pragma unroll
    for (int t = 0; t < R; ++t) {
        P *= -a * bt[t];
        x[t] = yt_axpy(x[t], P, u);
    }
    CSum sum;
#pragma unroll
    for (int t = R - 1; t >= 0; --t) {
        win = yt_axpy(x[t], -a * bt[t], win);
        if (on && s + t < ny) __stcg(S + (size_t)t * pk, yt_store<Gm>(win));
        // the box's dst_w-weighted column sum (a channel has none)
        if constexpr (!CPLX) sum.add(win);
    }
    if constexpr (!CPLX) {
        // the group's partial (sum, compensation), merged in a fixed order
        CSum ws;
        if (on) {
            const double wk = b.dst_w[k];
            ws.add_prod(wk, sum.s);
            ws.add_prod(wk, sum.c);
        }
        ws = csum_warp(ws);
        if (lane == 0) { part[0][wid] = ws.s; part[1][wid] = ws.c; }
        __syncthreads();
        if (live && wg == 0 && lane == 0) {
            CSum t;
            for (int y = 0; y < WG; ++y) t.merge(part[0][wid + y], part[1][wid + y]);
            b.part_col[2 * cb] = t.s;
            b.part_col[2 * cb + 1] = t.c;
        }
    }
}

// LU solve with the pivots of DGETRF (column-major n x n) -- DGETRS 'N'.
template <int N>
__device__ __forceinline__ void lu_solve_dev(const double (&lu)[N * N], const int (&piv)[N], double (&x)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) {
        // row interchange i <-> piv[i]
#pragma unroll
        for (int r = 0; r < N; ++r)
            if (r > i && piv[i] == r) { double t = x[i]; x[i] = x[r]; x[r] = t; }
    }
#pragma unroll
    for (int c = 0; c < N; ++c)
#pragma unroll
        for (int r = c + 1; r < N; ++r) x[r] -= x[c] * lu[r + N * c];
#pragma unroll
    for (int c = N - 1; c >= 0; --c) {
        x[c] /= lu[c + N * c];
#pragma unroll
        for (int r = 0; r < c; ++r) x[r] -= x[c] * lu[r + N * c];
    }
}

// solve_Ax_b (util/linalg.F90:57-93): DGETRS then the DGERFS refinement loop
// (at most 5 refinements), in registers.
template <int N>
__device__ __forceinline__ void solve_ax_b_dev(const double (&A)[N * N], const double (&lu)[N * N],
                                               const int (&piv)[N], const double (&rhs)[N], double (&x)[N]) {
#pragma unroll
    for (int i = 0; i < N; ++i) x[i] = rhs[i];
    lu_solve_dev<N>(lu, piv, x);
    const double eps = 1.1102230246251565e-16;
    const double safe1 = (N + 1) * 2.2250738585072014e-308, safe2 = safe1 / eps;
    double lstres = 3.0;
#pragma unroll 1
    for (int count = 1; count <= 6; ++count) {
        double r[N], wv[N];
#pragma unroll
        for (int i = 0; i < N; ++i) { r[i] = rhs[i]; wv[i] = fabs(rhs[i]); }
#pragma unroll
        for (int j = 0; j < N; ++j) {
            const double t = -x[j], xk = fabs(x[j]);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                r[i] += t * A[i + N * j];
                wv[i] += fabs(A[i + N * j]) * xk;
            }
        }
        double sm = 0.0;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const double q = (wv[i] > safe2) ? fabs(r[i]) / wv[i] : (fabs(r[i]) + safe1) / (wv[i] + safe1);
            sm = fmax(sm, q);
        }
        if (!(sm > eps && 2.0 * sm <= lstres && count <= 5)) break;
        lu_solve_dev<N>(lu, piv, r);
#pragma unroll
        for (int i = 0; i < N; ++i) x[i] += r[i];
        lstres = sm;
    }
}

// Per-step scalars the assembly needs: the homogeneous-correction
// coefficients and the suppress_comp_mode flag of this step.
struct XinvScal {
    double alpha[OQG_NLMAX];                             // box
    double c_bt, c_bc1[OQG_NLMAX], c_bc2[OQG_NLMAX];     // channel
    int supp;
};

// Brings a basin's descriptor into L1 ahead of the dependency wait (a full
// warp calls it): the scalar phase's loads of constants then hit.
__device__ __forceinline__ void prefetch_basin(const BasinDev &b) {
    for (int o = (threadIdx.x & 31) * 128; o < (int)sizeof(BasinDev); o += 32 * 128)
        asm volatile("prefetch.global.L1 [%0];" ::"l"((const char *)&b + o));
}

// The scalar phase of one step, run by one warp from the current state st[par]
// (every caller computes the same values); the writer also writes the next
// state st[1-par].
//   update_mass_constr (constraint.F90:167-179);
//   box_homog's area integrals and 2x2 solve (homog.F90:331-366), from the
//     dst_w-weighted spectral column sums of the y-solve (the inverse DST is
//     linear, so the area integral of the modal solution is known before it);
//   or, for a channel, the strip integrals of the vorticity kernel,
//     step_constraints (constraint.F90:182-215) and cyclic_homog
//     (homog.F90:280-329), lane k holding layer k, then mode k;
//   the suppress_comp_mode schedule and its scalar part (openqg.F90:485-487,
//     driver.F90:183-188).
// Bound by the latency of its loads and divisions: the assembly of a channel
// waits for it, and with one lane looping over the layers it took two thirds
// of the one-kernel inverse (k_xinv 18.8 us per launch on a 193 x 97 channel).
template <class T, int NL>
__device__ __noinline__ void scalar_phase(const BasinDev &b, double tdt, int par, bool writer,
                                          XinvScal *out) {
    constexpr unsigned ALL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const DevState *st = b.st + par;
    DevState *nx = b.st + (1 - par);
    const DevForcing *fr = b.frc;
    const long long nt = st->nt;
    const double ent_xn = fr->ent_xn;
    // update_mass_constr (constraint.F90:167-179)
    double dpi[NL], dpip[NL];
#pragma unroll
    for (int l = 0; l < NL - 1; ++l) {
        dpi[l] = st->dpip[l] - tdt * b.gp[l] * (l == 0 ? ent_xn : 0.0);
        dpip[l] = st->dpi[l];
    }
    const int per = b.suppress_period;
    const bool supp = per > 0 && (nt >> 31 ? nt % per : (long long)((unsigned)nt % (unsigned)per)) == 0;
    if (!b.cyclic) {
        const int nkb = (b.nk + b.ykb - 1) / b.ykb;       // y-solve column groups per mode
        double imode[NL];
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            CSum s;
#pragma unroll 4
            for (int x = lane; x < nkb; x += 32) s.merge(b.part_col[2 * (m * nkb + x)], b.part_col[2 * (m * nkb + x) + 1]);
            s = csum_warp(s, true);
            imode[m] = s.value() * b.ftnorm * b.dx * b.dy;
        }
        // box_homog (homog.F90:331-366)
        double ik[NL];
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            double s = 0.0;
#pragma unroll
            for (int m = 0; m < NL; ++m) s += b.ctm2l[m + NL * k] * imode[m];
            ik[k] = s;
        }
        constexpr int N = (NL > 1) ? NL - 1 : 1;
        double A[N * N], LU[N * N], rhs[N], al[N];
        int pv[N];
#pragma unroll
        for (int x = 0; x < N * N; ++x) { A[x] = b.cdhoc[x]; LU[x] = b.lu[x]; }
#pragma unroll
        for (int x = 0; x < N; ++x) { pv[x] = b.piv[x]; rhs[x] = dpi[x] - (ik[x + 1] - ik[x]); }
        solve_ax_b_dev<N>(A, LU, pv, rhs, al);
        if (lane == 0)
#pragma unroll
            for (int l = 0; l < N; ++l) out->alpha[l] = al[l];
    } else {
        const int k = lane < NL ? lane : NL - 1;
        const double dx = b.dx, dy = b.dy, f0 = b.fnot;
        double cs = st->cs[k], cn = st->cn[k];
        const double csp = st->csp[k], cnp = st->cnp[k];
        double S[OQG_NSTRIP], R[OQG_NSTRIP];              // the south's and north's strip integrals
#pragma unroll
        for (int q = 0; q < OQG_NSTRIP; ++q) {
            S[q] = b.part_tile[k * OQG_NSTRIP + q];
            R[q] = b.part_tile[(NL + k) * OQG_NSTRIP + q];
        }
        double rhss = -0.5 * dy * f0 * fr->int_Be_s[k], rhsn = -0.5 * dy * f0 * fr->int_Be_n[k];
        // step_constraints (constraint.F90:182-215)
        if (k == 0) {
            rhss = rhss + b.tau_sign * (f0 / b.h[0]) * fr->txis;
            rhsn = rhsn - b.tau_sign * (f0 / b.h[0]) * fr->txin;
        }
        const double bs = __shfl_sync(ALL, S[4], b.kt), bn = __shfl_sync(ALL, R[4], b.kt);
        if (k == NL - 1) {
            const double dfac = f0 * b.delek / (2.0 * fabs(f0)), fh = f0 / b.h[NL - 1];
            rhss = rhss + fh * (dfac * ((bs * dx) / dy));
            rhsn = rhsn - fh * (dfac * ((bn * dx) / dy));
        }
        const double a5s = (S[0] * dx) / (2.0 * dx), a9s = (S[1] * dx) / (2.0 * dx);
        const double a5n = (R[0] * dx) / (2.0 * dx), a9n = (R[1] * dx) / (2.0 * dx);
        const double ajis = (a5s + 2.0 * a9s) / 6.0, ajin = -(a5n + 2.0 * a9n) / 6.0;
        const double ap3s = b.ah2[k] * (S[2] * dx) / dy, ap3n = b.ah2[k] * (R[2] * dx) / dy;
        const double ap5s = b.ah4[k] * (S[3] * dx) / dy, ap5n = b.ah4[k] * (R[3] * dx) / dy;
        rhss = rhss + ajis - ap3s + ap5s;
        rhsn = rhsn + ajin + ap3n - ap5n;
        const double csn = csp + tdt * rhss, cnn = cnp + tdt * rhsn;
        // cyclic_homog (homog.F90:280-329), lane m.  The x-integral of row j of the
        // modal solution is dx times its zero wavenumber (before the 1/N of the
        // inverse transform, which the N-term row sum cancels).
        typedef typename C2<T>::t T2;
        const T2 *Sp = (const T2 *)b.spec + (size_t)k * b.ny * b.pk;
        const double u0s = (double)Sp[0].x, u0n = (double)Sp[(size_t)(b.ny - 1) * b.pk].x;
        double ss = 0.0, sn = 0.0;
#pragma unroll
        for (int l = 0; l < NL; ++l) {
            const double c = b.ctl2m[l + NL * k];
            ss += c * __shfl_sync(ALL, csn, l);
            sn += c * __shfl_sync(ALL, cnn, l);
        }
        const double clhss = ss + (u0s * dx) / dy, clhsn = sn + (u0n * dx) / dy;
        if (lane == 0) out->c_bt = clhss * b.hbsi;
        else if (lane < NL) {
            out->c_bc1[k] = b.hc2n[k] * clhss - b.hc2s[k] * clhsn;
            out->c_bc2[k] = b.hc1s[k] * clhsn - b.hc1n[k] * clhss;
        }
        if (writer && lane < NL) {
            // suppress_comp_mode's channel scalars (driver.F90:185-188)
            nx->cs[k] = supp ? 0.5 * (csn + cs) : csn;
            nx->cn[k] = supp ? 0.5 * (cnn + cn) : cnn;
            nx->csp[k] = cs;
            nx->cnp[k] = cn;
        }
    }
    if (lane != 0) return;
    out->supp = supp ? 1 : 0;
    if (!writer) return;
#pragma unroll
    for (int l = 0; l < NL - 1; ++l) {
        nx->dpi[l] = supp ? 0.5 * (dpi[l] + dpip[l]) : dpi[l];
        nx->dpip[l] = dpip[l];
    }
    nx->nt = nt + 1;
}

// ------------------------------------------------------------------ k_binv, k_xinv_rows
// The inverse x-transforms of the y-solved spectral rows as a launch of
// their own, shaped like the forward one, into the modal rows b.inh_g, which
// k_xinv_asm assembles (into out instead when out != null: the solve-only
// mode).  The first and last row pairs of a mode clear the wall rows 0 and
// nyp - 1.  The last scal CTAs run the scalar phase of member 0, 1, ... once
// into its b.scal_g (the assembly reads it there) and write the member's next
// scalar state (scal = 0: none).
template <class T>
__device__ __forceinline__ bool xinv_scalar_cta(const BasinDev *__restrict__ bas, int scal, int par, double tdt) {
    if (scal <= 0 || (int)blockIdx.x < (int)gridDim.x - scal) return false;
    const BasinDev &b = bas[blockIdx.x - (gridDim.x - scal)];
    pdl_trigger();
    if (threadIdx.x < 32) prefetch_basin(b);
    pdl_wait();
    if (threadIdx.x < 32) {
        const double dt = tdt != 0.0 ? tdt : b.tdt_m;
        XinvScal *sc = (XinvScal *)b.scal_g;
        if (b.nl == 2) scalar_phase<T, 2>(b, dt, par, true, sc);
        else if (b.nl == 3) scalar_phase<T, 3>(b, dt, par, true, sc);
        else scalar_phase<T, 4>(b, dt, par, true, sc);
    }
    return true;
}
template <class T>
__device__ __forceinline__ void xinv_wall_rows(const BasinDev &b, T *inh, int m, int j, int t, int TT) {
    const int nxp = b.nxp, px = b.px;
    if (j == 0) {
        T *first = inh + (size_t)m * b.nyp * px;
        for (int i = t; i < nxp; i += TT) first[i] = (T)0;
    }
    if (j + 2 >= b.ny) {
        T *last = inh + ((size_t)m * b.nyp + b.nyp - 1) * px;
        for (int i = t; i < nxp; i += TT) last[i] = (T)0;
    }
}

// A box: the inverse DST-I is the forward transform scaled by ftnorm
// (inhomog.F90:200-211); the modal row j + 1 gets the n interior values and
// zeros on both walls.  G: transforms per CTA as in k_bfwd; the scalar CTAs
// need a full warp, so blockDim is a multiple of 32.
template <class T, int MC = 0>
__global__ void __launch_bounds__(256, 2)
k_binv(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int G, int scal, int par, double tdt, T *out) {
    typedef typename C2<T>::t T2;
    if (xinv_scalar_cta<T>(bas, scal, par, tdt)) return;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int M = MC > 0 ? MC : b.M, TT = odd_tt(M);
    if (G <= 0) G = blockDim.x / TT;
    const int g = threadIdx.x / TT, t = threadIdx.x - g * TT;
    const int npm = (b.ny + 1) >> 1;
    const int tr = w.block * G + g;
    const bool live = g < G && tr < b.nl * npm;
    const int pair = live ? tr / b.nl : 0, m = live ? tr - pair * b.nl : 0, j = 2 * pair;
    const bool two = j + 1 < b.ny;
    T2 *z = reinterpret_cast<T2 *>(smem_raw) + (size_t)(g < G ? g : 0) * odd_smem_len(M);
    const T *x = (const T *)b.spec + ((size_t)m * b.ny + j) * b.pk;
    T *inh = out ? out : (T *)b.inh_g;
    const int n = b.nxin, px = b.px;
    T *ox = inh + ((size_t)m * b.nyp + j + 1) * px, *oy = ox + px;
    pdl_trigger();
    pdl_wait();
    if (live) odd_stage_rows<T>(z, x, x + b.pk, two, n, (T)b.ftnorm, t, TT);
    __syncthreads();
    odd_fft<T, MC>(z, M, b, (const T2 *)b.otw, t, TT, live, [&](int i, T2 v) {
        ox[i] = -v.y;
        if (two) oy[i] = v.x;
    });
    if (!live) return;
    if (t == 0) {
        ox[0] = ox[n + 1] = (T)0;
        if (two) oy[0] = oy[n + 1] = (T)0;
    }
    xinv_wall_rows(b, inh, m, j, t, TT);
}

// A channel: the c2r (inhomog.F90:214-255) of two rows by one complex
// transform fills every column, the last repeating the first.  G <= 0:
// blockDim / TT, per member of an ensemble.
template <class T, int E, int MC = 0>
__global__ void __launch_bounds__(256, 2)
k_xinv_rows(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int G, int scal, int par,
            double tdt, T *out) {
    typedef typename C2<T>::t T2;
    if (xinv_scalar_cta<T>(bas, scal, par, tdt)) return;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int M = MC > 0 ? MC : b.M, TT = (M + E - 1) / E;
    if (G <= 0) G = blockDim.x / TT;            // an ensemble: per member, as k_xfwd
    const int g = threadIdx.x / TT, t = threadIdx.x - g * TT;
    const int LB = fft_buf_len(M);
    T2 *zs = reinterpret_cast<T2 *>(smem_raw);
    const int npm = (b.ny + 1) >> 1;          // row pairs per mode
    const int pair = w.block * G + g;
    const bool live = g < G && pair < b.nl * npm;
    const int m = live ? pair / npm : 0;
    const int j = live ? 2 * (pair - m * npm) : 0;
    const bool two = live && (j + 1 < b.ny);
    const int px = b.px;
    // a spectral row: nk complex values, staged in the second buffer
    const int rowbytes = b.nk * (int)sizeof(T2);
    const int RO = round16(rowbytes) / (int)sizeof(T);   // offset of the second row (16-byte aligned)
    T2 *za = zs + (size_t)(g < G ? g : 0) * 2 * LB;
    T2 *zb = za + LB;
    T *raw = reinterpret_cast<T *>(zb);
    const size_t pitchb = (size_t)b.pk * sizeof(T2);
    const char *x = (const char *)b.spec + ((size_t)m * b.ny + j) * pitchb;
    T *inh = out ? out : (T *)b.inh_g;
    const T ftn = (T)b.ftnorm;
    pdl_trigger();
    pdl_wait();
    if (live) {
        cp_async_16(raw, x, round16(rowbytes), t, TT);
        if (two) cp_async_16(raw + RO, x + pitchb, round16(rowbytes), t, TT);
    }
    cp_async_commit_wait_all();
    __syncthreads();
    if (live) {
        // the Hermitian extension of X + iY, conjugated
        const T2 *xr = reinterpret_cast<const T2 *>(raw), *yr = reinterpret_cast<const T2 *>(raw + RO);
        for (int kk = t; kk < M; kk += TT) {
            T2 X, Y;
            const bool lo = kk <= M / 2;
            const int ks = lo ? kk : M - kk;
            X = xr[ks];
            if (two) Y = yr[ks]; else { Y.x = (T)0; Y.y = (T)0; }
            if (!lo) { X.y = -X.y; Y.y = -Y.y; }
            if (kk == 0 || 2 * kk == M) { X.y = (T)0; Y.y = (T)0; }
            T2 v;
            v.x = ftn * X.x - ftn * Y.y;
            v.y = -(ftn * X.y + ftn * Y.x);
            za[fpad(kk)] = v;
        }
    }
    __syncthreads();
    const T2 *z = fft_run<T, E, MC>(za, zb, M, b.rad, b.nrad, b.fd_ns, (const T2 *)b.tw, live ? t : TT, TT, 0, 0);
    if (!live) return;
    T *ox = inh + ((size_t)m * b.nyp + j + 1) * px;
    T *oy = ox + px;
    // every column; column nxp-1 = M repeats column 0 (inhomog.F90:250)
    for (int i = t; i < M; i += TT) {
        const T2 v = z[fpad(i)];
        ox[i] = v.x;
        if (two) oy[i] = -v.y;
    }
    if (t == 0) {
        const T2 v = z[fpad(0)];
        ox[M] = v.x;
        if (two) oy[M] = -v.y;
    }
    xinv_wall_rows(b, inh, m, j, t, TT);
}

// ------------------------------------------------------------------ k_xinv
// The inverse x-transforms and the assembly as one launch: a CTA transforms
// one row pair of every mode, then forms the layers of those rows (the first
// and last CTA the wall rows too).  The last warp runs the scalar phase of the
// step while the others transform; every CTA computes the same scalars, the
// first writes the next state.  Threads: NL transforms' (at least 128), and
// the scalar warp.  Bound by latency: on a 193 x 97 channel the 48 CTAs run one
// transform and 400 points each.  The launch takes 15 us there (5 of them the
// launch's own) with the transform's length compiled in, 128 threads and the
// scalars lane by layer; with an any-length transform, the modal rows cleared
// and rewritten in place and the scalars in one lane it took 27.
__host__ __device__ __forceinline__ int xinv_tt(int M, int cyclic) { return cyclic ? (M + XINV_E - 1) / XINV_E : odd_tt(M); }
__host__ __device__ __forceinline__ int xinv_threads(int M, int cyclic, int nl) {
    const int t = (nl * xinv_tt(M, cyclic) + 31) / 32 * 32;
    return t > 128 ? t : 128;
}
// Dynamic shared bytes: the transforms' buffers; the modal rows take the
// buffer that the last stage leaves free, or follow an in-place transform's.
__host__ __device__ __forceinline__ size_t xinv_bytes(int M, int cyclic, int nl, int nxp, int esz) {
    const size_t buf = (size_t)nl * 2 * esz * (cyclic ? 2 * fft_buf_len(M) : odd_smem_len(M));
    return buf + (!cyclic && odd_ct_len(M) ? (size_t)nl * 2 * nxp * esz : 0);
}

// The assembly of rows jfirst .. jlast of a basin (see k_xinv_asm): inh(m, j, i)
// is the modal solution at a point.
template <class T, int NL, class Inh>
__device__ __forceinline__ void xinv_assemble(const BasinDev &b, int par, const XinvScal *sc, int jfirst, int jlast, Inh inh) {
    const int nxp = b.nxp, nyp = b.nyp, px = b.px;
    const size_t ms = (size_t)nyp * px;
    const T *__restrict__ H = (const T *)b.hsb;
    const T *__restrict__ Pold = (const T *)b.F[par];
    T *__restrict__ Pnew = (T *)b.F[1 - par];
    T *__restrict__ Qc = (T *)b.F[3 - par];          // q after this step
    const T *__restrict__ Qm = (const T *)b.F[2 + par];
    const bool cyc = b.cyclic != 0, supp = sc->supp != 0;
    double ctm[NL * NL], hc[2 * NL];
#pragma unroll
    for (int x = 0; x < NL * NL; ++x) ctm[x] = b.ctm2l[x];
#pragma unroll
    for (int m = 0; m < NL; ++m) {
        hc[m] = !cyc ? (m ? sc->alpha[m - 1] : 0.0) : m ? sc->c_bc1[m] : sc->c_bt;
        hc[NL + m] = cyc && m ? sc->c_bc2[m] : 0.0;
    }
    auto layers = [&](int j, int i, T *pn) {
        const size_t o2 = (size_t)j * px + i;
        double pm_[NL];
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            double h = 0.0;
            if (!cyc) { if (m) h = hc[m] * (double)H[(m - 1) * ms + o2]; }
            else h = m ? hc[m] * b.hbc1[m * nyp + j] + hc[NL + m] * b.hbc2[m * nyp + j] : hc[0] * b.hbt[j];
            pm_[m] = inh(m, j, i) + h;
        }
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            double s2 = 0.0;
#pragma unroll
            for (int m = 0; m < NL; ++m) s2 += pm_[m] * ctm[m + NL * k];
            pn[k] = (T)s2;
        }
    };
    const T fac = (T)b.qb_fac;
    const FastDiv fdx = b.fd_nxp;
    const int npts = (jlast - jfirst + 1) * nxp;
    for (int idx = threadIdx.x; idx < npts; idx += blockDim.x) {
        const int jr = fdx.div(idx), i = idx - jr * nxp, j = jfirst + jr;
        const size_t o2 = (size_t)j * px + i;
        T pn[NL];
        layers(j, i, pn);
#pragma unroll
        for (int k = 0; k < NL; ++k)
            Pnew[k * ms + o2] = supp ? (T)((T)0.5 * (pn[k] + Pold[k * ms + o2])) : pn[k];
        const bool zon = (j == 0 || j == nyp - 1), mer = !cyc && (i == 0 || i == nxp - 1);
        if (!zon && !mer) {
            if (supp)
#pragma unroll
                for (int k = 0; k < NL; ++k) Qc[k * ms + o2] = (T)0.5 * (Qc[k * ms + o2] + Qm[k * ms + o2]);
            continue;
        }
        // ocqbdy (vorsubs.F90:58-114): the inner neighbour across the meridional
        // wall (a corner takes that one), else across the zonal wall
        T pnb[NL];
        layers(mer ? j : (j == 0 ? 1 : nyp - 2), mer ? (i == 0 ? 1 : nxp - 2) : i, pnb);
        const int cnt = (zon ? 1 : 0) + (mer ? 1 : 0);
        const T by = (T)(b.beta * b.yprel[j]);
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            T qv = fac * (pnb[k] - pn[k]);
            double mv = 0.0;
#pragma unroll
            for (int l = 0; l < NL; ++l) mv += b.amat[k + NL * l] * (double)pn[l];
            const T fmv = (T)(b.fnot * mv);
            for (int c = 0; c < cnt; ++c) qv = qv - fmv;
            // (FP32 storage holds q - beta y: one beta y fewer)
            for (int c = q_anom_stored<T>() ? 1 : 0; c < cnt; ++c) qv = qv + by;
            if (k == b.kt && b.topo_active) {
                const T dd = (T)b.ddyn[o2];
                for (int c = 0; c < cnt; ++c) qv = qv + dd;
            }
            Qc[k * ms + o2] = supp ? (T)((T)0.5 * (qv + Qm[k * ms + o2])) : qv;
        }
    }
}

// MC: as in k_xfwd (channels) and odd_fft (boxes).
template <class T, bool CYC, int MC>
__global__ void __maxnreg__(112)
k_xinv(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int par, double tdt) {
    typedef typename C2<T>::t T2;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    const int nfft = blockDim.x - 32, M = MC > 0 ? MC : b.M, TT = xinv_tt(M, CYC), nl = b.nl;
    const int g = threadIdx.x / TT, t = threadIdx.x - g * TT;
    const bool live = (int)threadIdx.x < nfft && g < nl;
    const int j = 2 * w.block, n = b.nxin, nxp = b.nxp;
    const bool two = j + 1 < b.ny;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __shared__ XinvScal sS;
    const int lz = CYC ? 2 * fft_buf_len(M) : odd_smem_len(M);
    T2 *z0 = reinterpret_cast<T2 *>(smem_raw), *z = z0 + (size_t)(live ? g : 0) * lz;
    // transform m's two modal rows
    T *inh0;
    size_t li;
    if (!CYC && odd_ct_len(M)) { inh0 = reinterpret_cast<T *>(z0 + (size_t)nl * lz); li = 2 * (size_t)nxp; }
    else {
        const int stages = CYC ? b.nrad : max(b.norad - 1, 1);
        inh0 = reinterpret_cast<T *>(z0 + ((stages & 1) ? 0 : lz / 2));
        li = 2 * (size_t)lz;
    }
    T *ox = inh0 + (live ? g : 0) * li, *oy = ox + nxp;
    const T ftn = (T)b.ftnorm;
    pdl_trigger();
    if ((int)threadIdx.x >= nfft) prefetch_basin(b);
    pdl_wait();
    if ((int)threadIdx.x >= nfft) {
        const double dt = tdt != 0.0 ? tdt : b.tdt_m;
        if (nl == 2) scalar_phase<T, 2>(b, dt, par, w.block == 0, &sS);
        else if (nl == 3) scalar_phase<T, 3>(b, dt, par, w.block == 0, &sS);
        else scalar_phase<T, 4>(b, dt, par, w.block == 0, &sS);
    } else if constexpr (CYC) {
        // the Hermitian extension of X + iY, conjugated (inhomog.F90:214-255)
        constexpr int U = 4;
        const int nk = b.nk;
        const FastDiv fd = b.fd_nk;
        for (int x0 = threadIdx.x; x0 < nl * nk; x0 += U * nfft) {
            T2 X[U], Y[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int x = x0 + u * nfft;
                X[u].x = X[u].y = Y[u].x = Y[u].y = (T)0;
                if (x < nl * nk) {
                    const int m = fd.div(x), kk = x - m * nk;
                    const T2 *r = (const T2 *)b.spec + ((size_t)m * b.ny + j) * b.pk + kk;
                    X[u] = __ldcg(r);
                    if (two) Y[u] = __ldcg(r + b.pk);
                }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
                const int x = x0 + u * nfft;
                if (x >= nl * nk) break;
                const int m = fd.div(x), kk = x - m * nk;
                T2 *zm = z0 + (size_t)m * lz;
                if (kk == 0 || 2 * kk == M) X[u].y = Y[u].y = (T)0;
                T2 v;
                v.x = ftn * X[u].x - ftn * Y[u].y;
                v.y = -(ftn * X[u].y + ftn * Y[u].x);
                zm[fpad(kk)] = v;
                if (kk > 0 && 2 * kk < M) {
                    v.x = ftn * X[u].x + ftn * Y[u].y;
                    v.y = -(ftn * Y[u].x - ftn * X[u].y);
                    zm[fpad(M - kk)] = v;
                }
            }
        }
        bar_sync(1, nfft);
        const T2 *r = fft_run<T, XINV_E, MC>(z, z + lz / 2, M, b.rad, b.nrad, b.fd_ns, (const T2 *)b.tw, live ? t : TT, TT, 1, nfft);
        if (live) {
            // every column; column nxp-1 = M repeats column 0 (inhomog.F90:250)
            for (int i = t; i <= M; i += TT) {
                const T2 v = r[fpad(i == M ? 0 : i)];
                ox[i] = v.x;
                oy[i] = -v.y;
            }
        }
    } else {
        if (live && t == 0) {
            T2 zero;
            zero.x = zero.y = (T)0;
            z[0] = z[zpad<4>(n + 1)] = zero;
        }
        const FastDiv fd = b.fd_nxin;
#pragma unroll 4
        for (int x = threadIdx.x; x < nl * n; x += nfft) {
            const int m = fd.div(x), i = x - m * n;
            const T *r = (const T *)b.spec + ((size_t)m * b.ny + j) * b.pk + i;
            T2 v;
            v.x = ftn * __ldcg(r);
            v.y = two ? ftn * __ldcg(r + b.pk) : (T)0;
            z0[(size_t)m * lz + zpad<4>(i + 1)] = v;
        }
        bar_sync(1, nfft);
        odd_fft<T, MC>(z, M, b, (const T2 *)b.otw, t, TT, live, [&](int i, T2 v) {
            ox[i] = -v.y;
            oy[i] = v.x;
        }, nfft);
        if (live && t == 0) ox[0] = ox[n + 1] = oy[0] = oy[n + 1] = (T)0;
    }
    __syncthreads();
    const int jfirst = j == 0 ? 0 : j + 1, jlast = j + 2 >= b.ny ? b.nyp - 1 : j + 2;
    auto inh = [&](int m, int jj, int i) {
        const int lr = jj - j - 1;
        return lr >= 0 && lr < (two ? 2 : 1) ? (double)inh0[m * li + lr * nxp + i] : 0.0;
    };
    if (nl == 2) xinv_assemble<T, 2>(b, par, &sS, jfirst, jlast, inh);
    else if (nl == 3) xinv_assemble<T, 3>(b, par, &sS, jfirst, jlast, inh);
    else xinv_assemble<T, 4>(b, par, &sS, jfirst, jlast, inh);
}

// ------------------------------------------------------------------ k_xinv_asm
#define XASM_ENS_POINTS 1024   // points per assembly work item of an ensemble's member
// The assembly of a basin whose inverse transforms ran as a launch of their own: the
// homogeneous correction and modes_to_layers (modes.F90:268-284) of every
// point from the modal rows in b.inh_g, ocqbdy (vorsubs.F90:58-114) on the
// walls and the suppress_comp_mode averages (driver.F90:174-189), with the
// step's scalars from b.scal_g.  The work items of a basin (the work list
// spans an ensemble's members) take interleaved runs of 256 vectors of a row's
// points, one per thread; a wall point also forms the layer values of its
// inner neighbour (the same arithmetic as the neighbour's own thread), so no
// point waits for another.  Bound by the loads in flight: with one FP32 point
// per thread 24 warps kept 15 KB in flight on an SM, and a 2049^2 launch of
// FP32 storage ran at 2.3 TB/s (58.6 us; 40.8 with four).
// hc: the box's alpha (nl-1), or the channel's c_bt, c_bc1[1..], c_bc2[1..]
// (homog.F90:280-366, by that launch's scalar CTA).
template <class T, int NL>
__device__ __forceinline__ void xinv_layers(const BasinDev &b, const T *__restrict__ inh, const T *__restrict__ H,
                                            const double *ctm, const double *hc, size_t o2, int j, T *pn) {
    const size_t ms = (size_t)b.nyp * b.px;
    double pm_[NL];
#pragma unroll
    for (int m = 0; m < NL; ++m) pm_[m] = (double)inh[m * ms + o2];
    if (!b.cyclic) {
#pragma unroll
        for (int m = 1; m < NL; ++m) pm_[m] = pm_[m] + hc[m - 1] * (double)H[(m - 1) * ms + o2];
    } else {
        const int nyp = b.nyp;
        pm_[0] = pm_[0] + hc[0] * b.hbt[j];
#pragma unroll
        for (int m = 1; m < NL; ++m)
            pm_[m] = pm_[m] + (hc[m] * b.hbc1[m * nyp + j] + hc[NL + m] * b.hbc2[m * nyp + j]);
    }
#pragma unroll
    for (int k = 0; k < NL; ++k) {
        double s2 = 0.0;
#pragma unroll
        for (int m = 0; m < NL; ++m) s2 += pm_[m] * ctm[m + NL * k];
        pn[k] = (T)s2;
    }
}

template <class T, int NL>
__global__ void __launch_bounds__(256)
k_xinv_asm(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int par) {
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    __shared__ double sCtm[NL * NL], sAmat[NL * NL], sHc[2 * NL];
    __shared__ int sSupp;
    pdl_trigger();
    // the basin's constant tables before the wait for the previous launch
    if (threadIdx.x < NL * NL) {
        sCtm[threadIdx.x] = b.ctm2l[threadIdx.x];
        sAmat[threadIdx.x] = b.amat[threadIdx.x];
    }
    pdl_wait();
    const XinvScal *sc = (const XinvScal *)b.scal_g;
    if (!b.cyclic) {
        if (threadIdx.x < NL - 1) sHc[threadIdx.x] = sc->alpha[threadIdx.x];
    } else if (threadIdx.x < 2 * NL) {
        // c_bt, c_bc1[1..NL), then c_bc2 at NL + m
        const int x = threadIdx.x;
        sHc[x] = x == 0 ? sc->c_bt : (x < NL ? sc->c_bc1[x] : (x == NL ? 0.0 : sc->c_bc2[x - NL]));
    }
    if (threadIdx.x == 0) sSupp = sc->supp;
    __syncthreads();
    double ctm[NL * NL], hc[2 * NL];
#pragma unroll
    for (int x = 0; x < NL * NL; ++x) ctm[x] = sCtm[x];
#pragma unroll
    for (int m = 0; m < 2 * NL; ++m) hc[m] = sHc[m];
    const bool supp = sSupp != 0;
    const int nxp = b.nxp, nyp = b.nyp, px = b.px;
    const size_t ms = (size_t)nyp * px;
    const T *__restrict__ inh = (const T *)b.inh_g;
    const T *__restrict__ H = (const T *)b.hsb;
    const T *__restrict__ Pold = (const T *)b.F[par];
    T *__restrict__ Pnew = (T *)b.F[1 - par];
    T *__restrict__ Qc = (T *)b.F[3 - par];          // q after this step
    const T *__restrict__ Qm = (const T *)b.F[2 + par];
    const T fac = (T)b.qb_fac;
    const FastDiv fdx = b.fd_nxp;
    const int npts = nxp * nyp;
    // the basin's b.asm_items work items interleave: item w.block takes the
    // points w.block * 256 + t, then every b.asm_items * 256 further
    const int stride = b.asm_items * 256;
    for (int idx = w.block * 256 + threadIdx.x; idx < npts; idx += stride) {
        const int j = fdx.div(idx), i = idx - j * nxp;
        const size_t o2 = (size_t)j * px + i;
        T pn[NL];
        xinv_layers<T, NL>(b, inh, H, ctm, hc, o2, j, pn);
#pragma unroll
        for (int k = 0; k < NL; ++k)
            Pnew[k * ms + o2] = supp ? (T)((T)0.5 * (pn[k] + Pold[k * ms + o2])) : pn[k];
        const bool zon = (j == 0 || j == nyp - 1);
        const bool mer = !b.cyclic && (i == 0 || i == nxp - 1);
        if (!zon && !mer) {
            if (supp)
#pragma unroll
                for (int k = 0; k < NL; ++k) Qc[k * ms + o2] = (T)0.5 * (Qc[k * ms + o2] + Qm[k * ms + o2]);
            continue;
        }
        // ocqbdy: the inner neighbour across the meridional wall (a corner
        // takes that one), else across the zonal wall
        const int jn = mer ? j : (j == 0 ? 1 : nyp - 2);
        const size_t on = mer ? (size_t)j * px + (i == 0 ? 1 : nxp - 2) : (size_t)jn * px + i;
        T pnb[NL];
        xinv_layers<T, NL>(b, inh, H, ctm, hc, on, jn, pnb);
        const int cnt = (zon ? 1 : 0) + (mer ? 1 : 0);
        const T by = (T)(b.beta * b.yprel[j]);
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            T qv = fac * (pnb[k] - pn[k]);
            double mv = 0.0;
#pragma unroll
            for (int l = 0; l < NL; ++l) mv += sAmat[k + NL * l] * (double)pn[l];
            const T fmv = (T)(b.fnot * mv);
            for (int c = 0; c < cnt; ++c) qv = qv - fmv;
            // (FP32 storage holds q - beta y: one beta y fewer)
            for (int c = q_anom_stored<T>() ? 1 : 0; c < cnt; ++c) qv = qv + by;
            if (k == b.kt && b.topo_active) {
                const T dd = (T)b.ddyn[o2];
                for (int c = 0; c < cnt; ++c) qv = qv + dd;
            }
            Qc[k * ms + o2] = supp ? (T)((T)0.5 * (qv + Qm[k * ms + o2])) : qv;
        }
    }
}

// The same with four points of a row per thread, for FP32 storage.  (In FP64 two
// points per thread took 62 us against 75 at 2049^2 but left the whole step as
// it was, 529 us, and cost the smaller grids their threads, 257^2 29.3 -> 31.9.)
#define XASM_V 4
template <class T> struct alignas(sizeof(T) * XASM_V) XasmVec { T v[XASM_V]; };
template <class T, int NL>
__global__ void __launch_bounds__(256, 3)
k_xinv_asm4(const BasinDev *__restrict__ bas, const Work *__restrict__ work, int par) {
    constexpr int V = XASM_V;
    typedef XasmVec<T> Vec;
    const Work w = work[blockIdx.x];
    const BasinDev &b = bas[w.member];
    __shared__ double sCtm[NL * NL], sAmat[NL * NL], sHc[2 * NL];
    __shared__ int sSupp;
    pdl_trigger();
    // the basin's constant tables before the wait for the previous launch
    if (threadIdx.x < NL * NL) {
        sCtm[threadIdx.x] = b.ctm2l[threadIdx.x];
        sAmat[threadIdx.x] = b.amat[threadIdx.x];
    }
    const int nxp = b.nxp, nyp = b.nyp, px = b.px;
    const bool cyc = b.cyclic != 0;
    const size_t ms = (size_t)nyp * px;
    const T *__restrict__ inh = (const T *)b.inh_g;
    const T *__restrict__ H = (const T *)b.hsb;
    const T *__restrict__ Pold = (const T *)b.F[par];
    T *__restrict__ Pnew = (T *)b.F[1 - par];
    T *__restrict__ Qc = (T *)b.F[3 - par];          // q after this step
    const T *__restrict__ Qm = (const T *)b.F[2 + par];
    const T fac = (T)b.qb_fac;
    const int rv = (nxp + V - 1) / V;                // vectors of a row
    const FastDiv fdx(rv);                           // (formed while the previous launch drains)
    const int nvec = rv * nyp;
    pdl_wait();
    const XinvScal *sc = (const XinvScal *)b.scal_g;
    if (!cyc) {
        if (threadIdx.x < NL - 1) sHc[threadIdx.x] = sc->alpha[threadIdx.x];
    } else if (threadIdx.x < 2 * NL) {
        // c_bt, c_bc1[1..NL), then c_bc2 at NL + m
        const int x = threadIdx.x;
        sHc[x] = x == 0 ? sc->c_bt : (x < NL ? sc->c_bc1[x] : (x == NL ? 0.0 : sc->c_bc2[x - NL]));
    }
    if (threadIdx.x == 0) sSupp = sc->supp;
    __syncthreads();
    double ctm[NL * NL], hc[2 * NL];
#pragma unroll
    for (int x = 0; x < NL * NL; ++x) ctm[x] = sCtm[x];
#pragma unroll
    for (int m = 0; m < 2 * NL; ++m) hc[m] = sHc[m];
    const bool supp = sSupp != 0;
    // ocqbdy and the suppression average of q at a wall point with layer
    // values pn: its inner neighbour across the meridional wall (a corner takes
    // that one), else across the zonal wall
    auto wall = [&](int j, int i, const T *pn) {
        const bool zon = (j == 0 || j == nyp - 1), mer = !cyc && (i == 0 || i == nxp - 1);
        const size_t o2 = (size_t)j * px + i;
        const int jn = mer ? j : (j == 0 ? 1 : nyp - 2);
        const size_t on = mer ? (size_t)j * px + (i == 0 ? 1 : nxp - 2) : (size_t)jn * px + i;
        T pnb[NL];
        xinv_layers<T, NL>(b, inh, H, ctm, hc, on, jn, pnb);
        const int cnt = (zon ? 1 : 0) + (mer ? 1 : 0);
        const T by = (T)(b.beta * b.yprel[j]);
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            T qv = fac * (pnb[k] - pn[k]);
            double mv = 0.0;
#pragma unroll
            for (int l = 0; l < NL; ++l) mv += sAmat[k + NL * l] * (double)pn[l];
            const T fmv = (T)(b.fnot * mv);
            for (int c = 0; c < cnt; ++c) qv = qv - fmv;
            // (FP32 storage holds q - beta y: one beta y fewer)
            for (int c = q_anom_stored<T>() ? 1 : 0; c < cnt; ++c) qv = qv + by;
            if (k == b.kt && b.topo_active) {
                const T dd = (T)b.ddyn[o2];
                for (int c = 0; c < cnt; ++c) qv = qv + dd;
            }
            Qc[k * ms + o2] = supp ? (T)((T)0.5 * (qv + Qm[k * ms + o2])) : qv;
        }
    };
    // the basin's b.asm_items work items interleave: item w.block takes the
    // vectors w.block * 256 + t, then every b.asm_items * 256 further
    const int stride = b.asm_items * 256;
    for (int idx = w.block * 256 + threadIdx.x; idx < nvec; idx += stride) {
        const int j = fdx.div(idx), i0 = (idx - j * rv) * V;
        const size_t o2 = (size_t)j * px + i0;
        Vec x[NL], h[NL];
#pragma unroll
        for (int m = 0; m < NL; ++m) {
            x[m] = *(const Vec *)(inh + m * ms + o2);
            if (!cyc && m) h[m] = *(const Vec *)(H + (m - 1) * ms + o2);
        }
        double hr[NL];                               // a channel's corrections of the row
        if (cyc) {
            hr[0] = hc[0] * b.hbt[j];
#pragma unroll
            for (int m = 1; m < NL; ++m) hr[m] = hc[m] * b.hbc1[m * nyp + j] + hc[NL + m] * b.hbc2[m * nyp + j];
        }
        Vec pn[NL];
#pragma unroll
        for (int e = 0; e < V; ++e) {
            double pm_[NL];
#pragma unroll
            for (int m = 0; m < NL; ++m) {
                pm_[m] = (double)x[m].v[e];
                if (cyc) pm_[m] = pm_[m] + hr[m];
                else if (m) pm_[m] = pm_[m] + hc[m - 1] * (double)h[m].v[e];
            }
#pragma unroll
            for (int k = 0; k < NL; ++k) {
                double s2 = 0.0;
#pragma unroll
                for (int m = 0; m < NL; ++m) s2 += pm_[m] * ctm[m + NL * k];
                pn[k].v[e] = (T)s2;
            }
        }
        const bool whole = i0 + V <= nxp;
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            Vec r = pn[k];
            if (supp) {
                const Vec old = *(const Vec *)(Pold + k * ms + o2);
#pragma unroll
                for (int e = 0; e < V; ++e) r.v[e] = (T)0.5 * (r.v[e] + old.v[e]);
            }
            if (whole) *(Vec *)(Pnew + k * ms + o2) = r;
            else
#pragma unroll
                for (int e = 0; e < V; ++e)
                    if (i0 + e < nxp) Pnew[k * ms + o2 + e] = r.v[e];
        }
        const bool zon = (j == 0 || j == nyp - 1);
        if (!supp && !zon && (cyc || (i0 > 0 && i0 + V < nxp))) continue;
#pragma unroll 1
        for (int e = 0; e < V && i0 + e < nxp; ++e) {
            const int i = i0 + e;
            if (zon || (!cyc && (i == 0 || i == nxp - 1))) {
                T q[NL];
#pragma unroll
                for (int k = 0; k < NL; ++k) {
                    q[k] = pn[k].v[0];
#pragma unroll
                    for (int f = 1; f < V; ++f)
                        if (f == e) q[k] = pn[k].v[f];
                }
                wall(j, i, q);
            } else if (supp) {
                for (int k = 0; k < NL; ++k) {
                    const size_t o3 = k * ms + o2 + e;
                    Qc[o3] = (T)0.5 * (Qc[o3] + Qm[o3]);
                }
            }
        }
    }
}

// ------------------------------------------------------------------ init / aux
// Laplacian with the wall condition on a global FP64 field (one layer),
// numerics.F90:410-468; the channel's column nxp-1 repeats column 0.
__device__ __forceinline__ double lap_bc_g(const double *f, const BasinDev &b, int i, int j, double alpha_fac) {
    const int px = b.px, nxp = b.nxp, nyp = b.nyp;
    if (b.cyclic && i == nxp - 1) i = 0;
    const double v = f[(size_t)j * px + i];
    double xp, yp;
    const bool wall_x = !b.cyclic && (i == 0 || i == nxp - 1);
    if (j == 0 || j == nyp - 1) xp = 0.0;
    else if (!b.cyclic && i == 0) xp = b.fx * alpha_fac * (f[(size_t)j * px + 1] - v);
    else if (!b.cyclic && i == nxp - 1) xp = -(b.fx * alpha_fac * (v - f[(size_t)j * px + i - 1]));
    else {
        int il = (i == 0) ? nxp - 2 : i - 1;
        xp = b.fx * (f[(size_t)j * px + il] + f[(size_t)j * px + i + 1] - 2.0 * v);
    }
    if (wall_x) yp = 0.0;
    else if (j == 0) yp = b.fy * alpha_fac * (f[(size_t)px + i] - v);
    else if (j == nyp - 1) yp = -(b.fy * alpha_fac * (v - f[(size_t)(j - 1) * px + i]));
    else yp = b.fy * (f[(size_t)(j - 1) * px + i] + f[(size_t)(j + 1) * px + i] - 2.0 * v);
    return xp + yp;
}

// qcomp (vorsubs.F90:27-56): q = del2(p)/f0 + ddyn[kt] + beta y - f0 A p.
// p: FP64 staging [nl][nyp][px]; q: field of type T.
template <class T, int NL>
__global__ void k_qcomp(const BasinDev *__restrict__ bas, int member, const double *p, T *q) {
    const BasinDev &b = bas[member];
    const size_t n2 = (size_t)b.nyp * b.px;
    const double afac = b.fx_bc / b.fx;   // alpha/(alpha/2+1)
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (size_t)b.nyp * b.nxp;
         idx += (size_t)gridDim.x * blockDim.x) {
        const int j = b.fd_nxp.div((int)idx), i = (int)idx - j * b.nxp;
        const size_t o2 = (size_t)j * b.px + i;
        double pv[NL];
#pragma unroll
        for (int l = 0; l < NL; ++l) pv[l] = p[l * n2 + o2];
#pragma unroll
        for (int k = 0; k < NL; ++k) {
            double v = lap_bc_g(p + k * n2, b, i, j, afac) / b.fnot;
            if (k == b.kt && b.topo_active) v += b.ddyn[o2];
            if (!q_anom_stored<T>()) v += b.beta * b.yprel[j];
            double mv = 0.0;
#pragma unroll
            for (int l = 0; l < NL; ++l) mv += b.amat[k + NL * l] * pv[l];
            v -= b.fnot * mv;
            q[k * n2 + o2] = (T)v;
        }
    }
}

template <class T>
__global__ void k_cvt_in(const double *src, T *dst, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = (T)src[i];
}
template <class T>
__global__ void k_cvt_out(const T *src, double *dst, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x)
        dst[i] = (double)src[i];
}

// q fields [nl][nyp][px] <-> FP64 staging, with the storage's anomaly
// (q_anom_stored) removed on the way out and applied on the way in.
template <class T>
__global__ void k_q_out(const BasinDev *__restrict__ bas, int member, const T *src, double *dst, size_t n) {
    const BasinDev &b = bas[member];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)((i / b.px) % b.nyp);
        dst[i] = (double)src[i] + (q_anom_stored<T>() ? b.beta * b.yprel[j] : 0.0);
    }
}
template <class T>
__global__ void k_q_in(const BasinDev *__restrict__ bas, int member, const double *src, T *dst, size_t n) {
    const BasinDev &b = bas[member];
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)((i / b.px) % b.nyp);
        dst[i] = (T)(q_anom_stored<T>() ? src[i] - b.beta * b.yprel[j] : src[i]);
    }
}

// Host-order rows (nxp contiguous FP64 values per row) <-> pitched field rows
// of type T: the unpacking and packing of contiguous host copies.
template <class T>
__global__ void k_rows_in(const double *src, T *dst, int nxp, int px, size_t nrows) {
    const size_t n = nrows * (size_t)nxp;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = (unsigned)i / (unsigned)nxp, c = i - r * nxp;    // n < 2^31
        dst[r * px + c] = (T)src[i];
    }
}
template <class T>
__global__ void k_rows_out(const T *src, double *dst, int nxp, int px, size_t nrows) {
    const size_t n = nrows * (size_t)nxp;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        const size_t r = (unsigned)i / (unsigned)nxp, c = i - r * nxp;    // n < 2^31
        dst[i] = (double)src[r * px + c];
    }
}

// Trapezoid weight of int_P_dA (numerics.F90:188-204) at (i, j).
__device__ __forceinline__ double trap_w(const BasinDev &b, int i, int j) {
    double w = 1.0;
    if (i == 0 || i == b.nxp - 1) w *= 0.5;
    if (j == 0 || j == b.nyp - 1) w *= 0.5;
    return w;
}
// int_P_dx (numerics.F90:206-212) weight.
__device__ __forceinline__ double trap_x(const BasinDev &b, int i) {
    return (i == 0 || i == b.nxp - 1) ? 0.5 : 1.0;
}

// int_P_dA (numerics.F90:165-204), compensated; red: >= 64 doubles.
template <class T>
__device__ double area_integral(const BasinDev &b, const T *f, double *red) {
    // eight loads in flight per thread (one at a time, a 257^2 field took 39 us)
    constexpr int U = 8;
    const FastDiv fd = b.fd_nxp;
    const int n = b.nyp * b.nxp;
    CSum s;
    for (int x0 = threadIdx.x; x0 < n; x0 += U * blockDim.x) {
        double v[U];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int idx = x0 + u * blockDim.x, j = fd.div(idx < n ? idx : 0), i = idx - j * b.nxp;
            v[u] = idx < n ? trap_w(b, i, j) * (double)f[(size_t)j * b.px + i] : 0.0;
        }
#pragma unroll
        for (int u = 0; u < U; ++u) s.add(v[u]);
    }
    return csum_block(s, red) * b.dx * b.dy;
}
// int_P_dx of row ja of f minus row jb (jb < 0: no subtraction), compensated
template <class T>
__device__ double row_integral(const BasinDev &b, const T *f, int ja, int jb, double *red) {
    CSum s;
    for (int i = threadIdx.x; i < b.nxp; i += blockDim.x) {
        double v = (double)f[(size_t)ja * b.px + i];
        if (jb >= 0) v -= (double)f[(size_t)jb * b.px + i];
        s.add(trap_x(b, i) * v);
    }
    return csum_block(s, red) * b.dx;
}

// int_P_dA of one FP64 field [nyp][px] into out[0] (one CTA): the integral
// the mass constraint uses, exposed for tests of its compensation.
__global__ void k_area_integral(const BasinDev *__restrict__ bas, int member, const double *f, double *out) {
    __shared__ double red[64];
    const double v = area_integral(bas[member], f, red);
    if (threadIdx.x == 0) out[0] = v;
}

// init_mass_constr (constraint.F90:145-165) and, for a channel,
// init_constraint (constraint.F90:80-143).  One CTA.
template <class T, int NL>
__global__ void k_init_constraints(const BasinDev *__restrict__ bas, int member, int par) {
    const BasinDev &b = bas[member];
    __shared__ double red[64];
    __shared__ double ip[OQG_NLMAX], ipm[OQG_NLMAX], pins[OQG_NLMAX], pinn[OQG_NLMAX],
        pinsp[OQG_NLMAX], pinnp[OQG_NLMAX], cs[OQG_NLMAX], cn[OQG_NLMAX], csp[OQG_NLMAX],
        cnp[OQG_NLMAX];
    const T *P = (const T *)b.F[par];
    const T *PM = (const T *)b.F[1 - par];
    const size_t n2 = (size_t)b.nyp * b.px;
    const int ny1 = b.nyp - 1;
    for (int k = 0; k < NL; ++k) {
        double a = area_integral(b, P + k * n2, red);
        double am = area_integral(b, PM + k * n2, red);
        if (threadIdx.x == 0) { ip[k] = a; ipm[k] = am; }
        if (b.cyclic) {
            double v0 = row_integral(b, PM + k * n2, 0, -1, red);
            double v1 = row_integral(b, P + k * n2, 0, -1, red);
            double v2 = row_integral(b, PM + k * n2, ny1, -1, red);
            double v3 = row_integral(b, P + k * n2, ny1, -1, red);
            double v4 = row_integral(b, PM + k * n2, 1, 0, red) / b.dy;
            double v5 = row_integral(b, PM + k * n2, ny1, ny1 - 1, red) / b.dy;
            double v6 = row_integral(b, P + k * n2, 1, 0, red) / b.dy;
            double v7 = row_integral(b, P + k * n2, ny1, ny1 - 1, red) / b.dy;
            if (threadIdx.x == 0) {
                pinsp[k] = v0; pins[k] = v1; pinnp[k] = v2; pinn[k] = v3;
                csp[k] = v4; cnp[k] = v5; cs[k] = v6; cn[k] = v7;
            }
        }
    }
    __syncthreads();
    if (threadIdx.x != 0) return;
    DevState *sc = b.st + par;
    for (int k = 0; k < NL - 1; ++k) {
        sc->dpip[k] = b.dz_sign * (ipm[k] - ipm[k + 1]);
        sc->dpi[k] = b.dz_sign * (ip[k] - ip[k + 1]);
    }
    if (b.cyclic) {
        const double f2 = 0.5 * b.dy * b.fnot * b.fnot;
        for (int k = 0; k < NL; ++k) {
            double apsp = 0, apnp = 0, aps = 0, apn = 0;
            for (int l = 0; l < NL; ++l) {
                double a = b.amat[k + NL * l];
                apsp += a * pinsp[l]; apnp += a * pinnp[l]; aps += a * pins[l]; apn += a * pinn[l];
            }
            sc->csp[k] = -csp[k] + f2 * apsp;
            sc->cnp[k] = cnp[k] + f2 * apnp;
            sc->cs[k] = -cs[k] + f2 * aps;
            sc->cn[k] = cn[k] + f2 * apn;
        }
    }
}

// Row sums of the ent area integral (int_P_dA, numerics.F90:165-204): one
// CTA per row j writes sum_i trap_x(i) ent(i, j, 1) to ent_rows[2j] with its
// compensation in ent_rows[2j+1].
template <class T>
__global__ void __launch_bounds__(128) k_ent_rows(const BasinDev *__restrict__ bas, int member) {
    const BasinDev &b = bas[member];
    __shared__ double red[64];
    const T *E = (const T *)b.ent + (size_t)blockIdx.x * b.px;
    CSum s;
    for (int i = threadIdx.x; i < b.nxp; i += blockDim.x) s.add(trap_x(b, i) * (double)E[i]);
    const CSum t = csum_block_pair(s, red);
    if (threadIdx.x == 0) { b.ent_rows[2 * blockIdx.x] = t.s; b.ent_rows[2 * blockIdx.x + 1] = t.c; }
}

// Forcing integrals that depend only on ent: ent_xn = int_P_dA(ent(:,:,1))
// (pressure.F90:52-54) from the row sums of k_ent_rows, in a fixed order,
// and the channel strip integrals int_Be_s/n (vorticity.F90:122-128).  One CTA.
// K CTA sums in one pass: the warps' shuffles of the K values interleave and
// three barriers serve them all.  The result is valid in every thread.
template <int K>
__device__ __forceinline__ void block_sum_n(double (&v)[K]) {
    __shared__ double r[K][32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1)
#pragma unroll
        for (int q = 0; q < K; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
    __syncthreads();
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < K; ++q) r[q][wid] = v[q];
    __syncthreads();
    if (wid == 0) {
#pragma unroll
        for (int q = 0; q < K; ++q) v[q] = lane < nw ? r[q][lane] : 0.0;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
#pragma unroll
            for (int q = 0; q < K; ++q) v[q] += __shfl_down_sync(0xffffffffu, v[q], o);
        if (lane == 0)
#pragma unroll
            for (int q = 0; q < K; ++q) r[q][0] = v[q];
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < K; ++q) v[q] = r[q][0];
}

template <class T>
__device__ void forcing_integrals_cta(const BasinDev &b, const T *E) {
    DevForcing *sc = b.frc;
    const size_t n2 = (size_t)b.nyp * b.px;
    // ent_rows' trapezoidal sum, and for a channel the trapezoidal x-sums of
    // ent's rows 0 and nyp-1 in layers 1 and 2 (row_integral), together
    // (compensated: the mass constraint's area integral, numerics.F90:165-204)
    CSum cv[5];
    if (E) {
        for (int j = threadIdx.x; j < b.nyp; j += blockDim.x) {
            const double wj = (j == 0 || j == b.nyp - 1) ? 0.5 : 1.0;   // exact scaling
            cv[0].merge(wj * b.ent_rows[2 * j], wj * b.ent_rows[2 * j + 1]);
        }
        if (b.cyclic) {
            const size_t last = (size_t)(b.nyp - 1) * b.px;
            const bool two = b.nl - 1 >= 2;
            for (int i = threadIdx.x; i < b.nxp; i += blockDim.x) {
                const double t = trap_x(b, i);
                cv[1].add(t * (double)E[i]);
                cv[2].add(t * (double)E[last + i]);
                if (two) {
                    cv[3].add(t * (double)E[n2 + i]);
                    cv[4].add(t * (double)E[n2 + last + i]);
                }
            }
        }
    }
    // (the five reductions one after the other were 5 of the 13 us of a
    // channel's k_aml_post, whose last CTA ends with them)
    double v[5] = {};
    csum_block_n<5>(cv, v);
    const double exn = v[0] * b.dx * b.dy;
    const double s1 = v[1] * b.dx, n1 = v[2] * b.dx, s2 = v[3] * b.dx, n2v = v[4] * b.dx;
    if (threadIdx.x != 0) return;
    sc->ent_xn = exn;
    for (int k = 0; k < OQG_NLMAX; ++k) { sc->int_Be_s[k] = 0.0; sc->int_Be_n[k] = 0.0; }
    const double f1 = b.fnot / b.h[0], f2 = b.fnot / b.h[1];
    sc->int_Be_s[0] = b.dz_sign * f1 * s1;
    sc->int_Be_s[1] = b.dz_sign * f1 * s2;
    sc->int_Be_n[0] = -b.dz_sign * f2 * n1;
    sc->int_Be_n[1] = -b.dz_sign * f2 * n2v;
}

// The forcing's integrals (ent_xn; a channel's ent strip integrals) from the
// descriptor's entrainment, one CTA.
template <class T>
__global__ void k_forcing_integrals(const BasinDev *__restrict__ bas, int member) {
    const BasinDev &b = bas[member];
    forcing_integrals_cta<T>(b, (const T *)b.ent);
}

// Whether this CTA is the last of its grid to arrive (a ticket counter that
// the last one resets): every CTA's global writes before the call are then
// visible to it.  No CTA waits.
__device__ __forceinline__ bool last_cta(unsigned *ticket) {
    __shared__ bool is_last;
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) is_last = atomicAdd(ticket, 1u) == gridDim.x - 1;
    __syncthreads();
    if (!is_last) return false;
    __threadfence();
    if (threadIdx.x == 0) *ticket = 0u;
    return true;
}

// Solve-only input: the same (nxp, nyp) right-hand side for every mode.
template <class T>
__global__ void k_rhs_from_field(const BasinDev *__restrict__ bas, int member, const double *f, T *rhs) {
    const BasinDev &b = bas[member];
    const int ioff = b.cyclic ? 0 : 1;
    for (int idx = blockIdx.x * blockDim.x + threadIdx.x; idx < b.nl * b.ny * b.nxin;
         idx += gridDim.x * blockDim.x) {
        int m = idx / (b.ny * b.nxin), rem = idx - m * b.ny * b.nxin;
        int jj = rem / b.nxin, xi = rem - jj * b.nxin;
        rhs[((size_t)m * b.ny + jj) * b.pr + xi] = (T)f[(size_t)(jj + 1) * b.px + xi + ioff];
    }
}

// suppress_comp_mode now (driver.F90:174-189).
template <class T>
__global__ void k_suppress(const BasinDev *__restrict__ bas, int member, int par) {
    const BasinDev &b = bas[member];
    T *P = (T *)b.F[par];
    const T *PM = (const T *)b.F[1 - par];
    T *Q = (T *)b.F[2 + par];
    const T *QM = (const T *)b.F[3 - par];
    const size_t n = (size_t)b.nl * b.nyp * b.px;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        Q[i] = (T)0.5 * (Q[i] + QM[i]);
        P[i] = (T)0.5 * (P[i] + PM[i]);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        DevState *sc = b.st + par;
        for (int l = 0; l < b.nl - 1; ++l) sc->dpi[l] = 0.5 * (sc->dpi[l] + sc->dpip[l]);
        if (b.cyclic)
            for (int k = 0; k < b.nl; ++k) {
                sc->cs[k] = 0.5 * (sc->cs[k] + sc->csp[k]);
                sc->cn[k] = 0.5 * (sc->cn[k] + sc->cnp[k]);
            }
    }
}

// Count of non-finite values of p and q (the role of valids).
template <class T>
__global__ void k_check_finite(const BasinDev *__restrict__ bas, int member, int par,
                               unsigned long long *bad) {
    const BasinDev &b = bas[member];
    const T *P = (const T *)b.F[par];
    const T *Q = (const T *)b.F[2 + par];
    unsigned long long c = 0;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (size_t)b.nl * b.nyp * b.nxp;
         idx += (size_t)gridDim.x * blockDim.x) {
        size_t k = idx / ((size_t)b.nyp * b.nxp), rem = idx - k * b.nyp * b.nxp;
        size_t j = rem / b.nxp, i = rem - j * b.nxp;
        size_t o = (k * b.nyp + j) * b.px + i;
        if (!isfinite((double)P[o])) ++c;
        if (!isfinite((double)Q[o])) ++c;
    }
    if (c) atomicAdd(bad, c);
}

// qg_diagno energetics and extrema (qg_monitor.F90:289-376): one CTA per layer.
// out[k*4 + 0..3] = ekei, sfmin, sfmax, circ.
template <class T>
__global__ void k_diag(const BasinDev *__restrict__ bas, int member, int par, double rho, double *out) {
    const BasinDev &b = bas[member];
    const int k = blockIdx.x;
    __shared__ double red[32];
    const T *P = (const T *)b.F[par] + (size_t)k * b.nyp * b.px;
    double uke = 0.0, vke = 0.0, pmin = 1e308, pmax = -1e308;
    const int nxp = b.nxp, nyp = b.nyp, px = b.px;
    // (alpha/2 + 1) of dPdx_2bc/dPdy_2bc, recovered from the mixed-BC factor
    const double ah = b.bc_half1;
    for (int idx = threadIdx.x; idx < nxp * nyp; idx += blockDim.x) {
        int j = idx / nxp, i = idx - j * nxp;
        double pv = (double)P[(size_t)j * px + i];
        pmin = fmin(pmin, pv);
        pmax = fmax(pmax, pv);
        // dPdx_2bc / dPdy_2bc (numerics.F90:470-513)
        double dpx, dpy;
        if (j == 0 || j == nyp - 1) dpx = 0.0;
        else if (b.cyclic && (i == 0 || i == nxp - 1))
            dpx = ((double)P[(size_t)j * px + 1] - (double)P[(size_t)j * px + nxp - 2]) / (2.0 * b.dx);
        else if (i == 0) dpx = ((double)P[(size_t)j * px + 1] - pv) / (b.dx * ah);
        else if (i == nxp - 1) dpx = (pv - (double)P[(size_t)j * px + i - 1]) / (b.dx * ah);
        else dpx = ((double)P[(size_t)j * px + i + 1] - (double)P[(size_t)j * px + i - 1]) / (2.0 * b.dx);
        if (!b.cyclic && (i == 0 || i == nxp - 1)) dpy = 0.0;
        else if (j == 0) dpy = ((double)P[(size_t)px + i] - pv) / (b.dy * ah);
        else if (j == nyp - 1) dpy = (pv - (double)P[(size_t)(j - 1) * px + i]) / (b.dy * ah);
        else dpy = ((double)P[(size_t)(j + 1) * px + i] - (double)P[(size_t)(j - 1) * px + i]) / (2.0 * b.dy);
        double u = -dpy / b.fnot, v = dpx / b.fnot;
        double w = trap_w(b, i, j);
        uke += w * (u * u);
        vke += w * (v * v);
    }
    uke = block_sum(uke, red) * b.dx * b.dy;
    vke = block_sum(vke, red) * b.dx * b.dy;
    // min / max
    __shared__ double mn[32], mx[32];
    for (int o = 16; o > 0; o >>= 1) {
        pmin = fmin(pmin, __shfl_down_sync(0xffffffffu, pmin, o));
        pmax = fmax(pmax, __shfl_down_sync(0xffffffffu, pmax, o));
    }
    if ((threadIdx.x & 31) == 0) { mn[threadIdx.x >> 5] = pmin; mx[threadIdx.x >> 5] = pmax; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int wv = 1; wv < (int)(blockDim.x >> 5); ++wv) { pmin = fmin(pmin, mn[wv]); pmax = fmax(pmax, mx[wv]); }
        const double p00 = (double)P[0], p0n = (double)P[(size_t)(nyp - 1) * px];
        const double poref = b.fnot > 0 ? p00 : p0n;
        const double e1 = fmin(pmin / b.fnot, pmax / b.fnot), e2 = fmax(pmin / b.fnot, pmax / b.fnot);
        out[k * 4 + 0] = 0.5 * rho * b.h[k] * (uke + vke);
        out[k * 4 + 1] = 1.0e-6 * (b.h[k] * (e1 - poref / b.fnot));
        out[k * 4 + 2] = 1.0e-6 * (b.h[k] * (e2 - poref / b.fnot));
        out[k * 4 + 3] = 1.0e-6 * ((p00 - p0n) / b.fnot);
    }
}

// ------------------------------------------------------------------ valids
// Extremes of p, q (all layers) and wekp for the validity scan (valsubs.F90:
// 46-139), and the count of non-finite values among them: per CTA into
// out[blockIdx.x * 7 + (pmin, pmax, qmin, qmax, wmin, wmax, nonfinite)].
template <class T>
__global__ void __launch_bounds__(256) k_valids(const BasinDev *__restrict__ bas, int member, int par, double *out) {
    const BasinDev &b = bas[member];
    const T *P = (const T *)b.F[par], *Q = (const T *)b.F[2 + par], *W = (const T *)b.wekp;
    const size_t n2 = (size_t)b.nyp * b.px;
    double v[6] = {1e308, -1e308, 1e308, -1e308, 1e308, -1e308};
    double bad = 0.0;
    const size_t tot = (size_t)b.nl * b.nyp * b.nxp;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < tot; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t k = idx / ((size_t)b.nyp * b.nxp), rem = idx - k * b.nyp * b.nxp;
        const size_t j = rem / b.nxp, i = rem - j * b.nxp;
        const size_t o = k * n2 + j * b.px + i;
        const double pv = (double)P[o], qv = (double)Q[o] + (q_anom_stored<T>() ? b.beta * b.yprel[j] : 0.0);
        if (!isfinite(pv)) bad += 1.0; else { v[0] = fmin(v[0], pv); v[1] = fmax(v[1], pv); }
        if (!isfinite(qv)) bad += 1.0; else { v[2] = fmin(v[2], qv); v[3] = fmax(v[3], qv); }
        if (k == 0) {
            const double wv = (double)W[j * b.px + i];
            if (!isfinite(wv)) bad += 1.0; else { v[4] = fmin(v[4], wv); v[5] = fmax(v[5], wv); }
        }
    }
    __shared__ double red[7][8];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    for (int q = 0; q < 6; ++q) {
        double x = v[q];
        for (int o = 16; o > 0; o >>= 1) {
            const double y = __shfl_down_sync(0xffffffffu, x, o);
            x = (q & 1) ? fmax(x, y) : fmin(x, y);
        }
        if (lane == 0) red[q][wid] = x;
    }
    for (int o = 16; o > 0; o >>= 1) bad += __shfl_down_sync(0xffffffffu, bad, o);
    if (lane == 0) red[6][wid] = bad;
    __syncthreads();
    if (threadIdx.x < 7) {
        const int q = threadIdx.x;
        double x = red[q][0];
        for (int w = 1; w < (int)(blockDim.x >> 5); ++w)
            x = q == 6 ? x + red[q][w] : ((q & 1) ? fmax(x, red[q][w]) : fmin(x, red[q][w]));
        out[blockIdx.x * 7 + q] = x;
    }
}

// ------------------------------------------------------------------ qg_diagno
// The monitor record of qg_diagno (qg_monitor.F90:219-383) on the device:
// velocity fields, their wall Laplacians, then per-row sums of every
// integrand; the host adds the rows in a fixed order.

// dPdx_2bc / dPdy_2bc (numerics.F90:470-513) of layer field P at (i, j).
template <class T>
__device__ __forceinline__ void dpdxy_bc(const T *P, const BasinDev &b, int i, int j, double &dpx, double &dpy) {
    const int nxp = b.nxp, nyp = b.nyp, px = b.px;
    const double ah = b.bc_half1;
    const double pv = (double)P[(size_t)j * px + i];
    if (j == 0 || j == nyp - 1) dpx = 0.0;
    else if (b.cyclic && (i == 0 || i == nxp - 1))
        dpx = ((double)P[(size_t)j * px + 1] - (double)P[(size_t)j * px + nxp - 2]) / (2.0 * b.dx);
    else if (i == 0) dpx = ((double)P[(size_t)j * px + 1] - pv) / (b.dx * ah);
    else if (i == nxp - 1) dpx = (pv - (double)P[(size_t)j * px + i - 1]) / (b.dx * ah);
    else dpx = ((double)P[(size_t)j * px + i + 1] - (double)P[(size_t)j * px + i - 1]) / (2.0 * b.dx);
    if (!b.cyclic && (i == 0 || i == nxp - 1)) dpy = 0.0;
    else if (j == 0) dpy = ((double)P[(size_t)px + i] - pv) / (b.dy * ah);
    else if (j == nyp - 1) dpy = (pv - (double)P[(size_t)(j - 1) * px + i]) / (b.dy * ah);
    else dpy = ((double)P[(size_t)(j + 1) * px + i] - (double)P[(size_t)(j - 1) * px + i]) / (2.0 * b.dy);
}

// Lagged (from pm) and current (from p) geostrophic velocities, FP64:
// V[0..3] = ug, vg, uc, vc, each [nl][nyp][px].
template <class T>
__global__ void k_dg_vel(const BasinDev *__restrict__ bas, int member, int par, double *V) {
    const BasinDev &b = bas[member];
    const size_t n2 = (size_t)b.nyp * b.px, n3 = n2 * b.nl;
    const T *P = (const T *)b.F[par], *PM = (const T *)b.F[1 - par];
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < (size_t)b.nl * b.nyp * b.nxp;
         idx += (size_t)gridDim.x * blockDim.x) {
        const size_t k = idx / ((size_t)b.nyp * b.nxp), rem = idx - k * b.nyp * b.nxp;
        const int j = (int)(rem / b.nxp), i = (int)(rem - (size_t)j * b.nxp);
        const size_t o = k * n2 + (size_t)j * b.px + i;
        double dx, dy;
        dpdxy_bc(PM + k * n2, b, i, j, dx, dy);
        V[o] = -dy / b.fnot;
        V[n3 + o] = dx / b.fnot;
        dpdxy_bc(P + k * n2, b, i, j, dx, dy);
        V[2 * n3 + o] = -dy / b.fnot;
        V[3 * n3 + o] = dx / b.fnot;
    }
}

// del2_P_bc (numerics.F90:410-425) of nf FP64 fields [nl][nyp][px] each.
__global__ void k_dg_del2(const BasinDev *__restrict__ bas, int member, const double *in, double *out, int nf) {
    const BasinDev &b = bas[member];
    const size_t n2 = (size_t)b.nyp * b.px;
    const double afac = b.fx_bc / b.fx;   // alpha/(alpha/2+1)
    const size_t tot = (size_t)nf * b.nl * b.nyp * b.nxp;
    for (size_t idx = blockIdx.x * (size_t)blockDim.x + threadIdx.x; idx < tot; idx += (size_t)gridDim.x * blockDim.x) {
        const size_t f = idx / ((size_t)b.nyp * b.nxp), rem = idx - f * b.nyp * b.nxp;
        const int j = (int)(rem / b.nxp), i = (int)(rem - (size_t)j * b.nxp);
        out[f * n2 + (size_t)j * b.px + i] = lap_bc_g(in + f * n2, b, i, j, afac);
    }
}

#define OQG_DGQ 22   // row sums per (layer, row) of k_dg_rows

// One CTA per (row j, layer k): trapezoid-in-x row sums (int_P_dx / dx) of
// the qg_diagno integrands, into R[(q nl + k) nyp + j]; q 20 and 21 are the
// row minimum and maximum of p.  V: ug, vg, uc, vc, del2 u, del4 u, del2 v,
// del4 v (FP64 [nl][nyp][px] each); tau: taux, tauy rows (or null).
template <class T>
__global__ void __launch_bounds__(128) k_dg_rows(const BasinDev *__restrict__ bas, int member, int par,
                                                 const double *V, const double *tau, double *R) {
    const BasinDev &b = bas[member];
    const int j = blockIdx.x, k = blockIdx.y, nl = b.nl, nxp = b.nxp, nyp = b.nyp;
    const size_t n2 = (size_t)nyp * b.px, n3 = n2 * nl, o0 = (size_t)k * n2 + (size_t)j * b.px;
    const T *P = (const T *)b.F[par], *Q = (const T *)b.F[2 + par];
    const T *WK = (const T *)b.wekp, *EN = (const T *)b.ent;
    __shared__ double red[32];
    double s[OQG_DGQ];
#pragma unroll
    for (int q = 0; q < OQG_DGQ; ++q) s[q] = 0.0;
    double pmin = 1e308, pmax = -1e308;
    const double gpk = k < nl - 1 ? b.gp[k] : 1.0;
    for (int i = threadIdx.x; i < nxp; i += blockDim.x) {
        const double w = trap_x(b, i);
        const size_t o = o0 + i, oj = (size_t)j * b.px + i;
        const double pv = (double)P[o];
        const double ug = V[o], vg = V[n3 + o], uc = V[2 * n3 + o], vc = V[3 * n3 + o];
        s[0] += w * pv;
        s[1] += w * ((double)Q[o] + (q_anom_stored<T>() ? b.beta * b.yprel[j] : 0.0));
        s[2] += w * (uc * V[4 * n3 + o]);
        s[3] += w * (vc * V[6 * n3 + o]);
        s[4] += w * (uc * V[5 * n3 + o]);
        s[5] += w * (vc * V[7 * n3 + o]);
        s[6] += w * (uc * uc);
        s[7] += w * (vc * vc);
        s[8] += w * uc;
        s[9] += w * (ug * ug);
        s[10] += w * (vg * vg);
        if (k < nl - 1) {
            const double eta = b.dz_sign * (pv - (double)P[o + n2]) / gpk;
            s[11] += w * eta;
            s[12] += w * (eta * eta);
            if (k == 0) s[13] += w * (eta * (EN ? (double)EN[oj] : 0.0));
        }
        if (k == 0) {
            const double wk = (double)WK[oj], e1 = EN ? (double)EN[oj] : 0.0;
            s[14] += w * wk;
            s[15] += w * fabs(wk);
            s[16] += w * e1;
            s[17] += w * fabs(e1);
            if (tau) {
                s[18] += w * (tau[oj] * uc);
                s[19] += w * (tau[n2 + oj] * vc);
            }
        }
        pmin = fmin(pmin, pv);
        pmax = fmax(pmax, pv);
    }
    for (int q = 0; q < 20; ++q) {
        const double v = block_sum(s[q], red);
        if (threadIdx.x == 0) R[((size_t)q * nl + k) * nyp + j] = v;
    }
    __shared__ double mn[32], mx[32];
    for (int o = 16; o > 0; o >>= 1) {
        pmin = fmin(pmin, __shfl_down_sync(0xffffffffu, pmin, o));
        pmax = fmax(pmax, __shfl_down_sync(0xffffffffu, pmax, o));
    }
    if ((threadIdx.x & 31) == 0) { mn[threadIdx.x >> 5] = pmin; mx[threadIdx.x >> 5] = pmax; }
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int wv = 1; wv < (int)(blockDim.x >> 5); ++wv) { pmin = fmin(pmin, mn[wv]); pmax = fmax(pmax, mx[wv]); }
        R[((size_t)20 * nl + k) * nyp + j] = pmin;
        R[((size_t)21 * nl + k) * nyp + j] = pmax;
    }
}

}  // namespace oqg
