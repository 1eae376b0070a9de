// Whole Yee/CPML step in one plane march over the whole grid (sm_100a).
//
// Every cell's H^{n+1/2} and E^{n+1}, CPML slabs included, come from one
// kernel that reads E, H, ce (ca) once and writes E_next, H_next once:
// 60 B per FP32 lossless cell plus the ψ stripes, in place of an interior
// march with separate shell kernels (84 B per shell cell in three more,
// partly serial launches joined over two streams).
//
// Each CTA owns a (TJ x TK) tile of (j, k) and marches along i over a chunk of
// planes.  The planes of E^n (one-cell halo) and H^{n-1/2} move through an
// NSTAGE-deep shared-memory ring by TMA (cp.async.bulk.tensor 3-D tiled maps, no
// multicast, mbarrier transaction counts), with ce (ca) beside them.  Cell
// threads own V = 16 B / elem consecutive k cells each; a further warp evaluates
// H^{n+1/2} of the row j0-1 and of the vectors left of the tile, which the E
// stencil needs.  E^{n+1}(p) uses H^{n+1/2}(p) from shared memory and
// H^{n+1/2}(p-1) carried in registers.  The new-H plane is double-buffered, so one
// CTA barrier per plane suffices.  ψ is loaded one plane ahead into registers and
// prefetched into L2 PD planes earlier.
//
// CPML: a tile is compiled for the axes whose slabs it (or its halo) touches:
// AX bit 0 = x, bit 1 = y, bit 2 = z, bit 3 = a vector may straddle a z slab's
// edge; CTA-uniform choice.  Interior tiles carry no CPML code.  The planes
// [0, npml] and [nx-npml, nx) are chunks of their own; only they need x (the
// plane npml rides with the low slab, since its E needs the x-CPML H of the
// plane below).  A halo H cell needs the ψ_H of a cell that another CTA
// advances, so ψ_H is read from psi_h and written to psi_h_next; ψ_E is owned by
// one thread and advanced in place.
//
// Arithmetic: the expressions and operand order of h_cell / e_cell
// (yee_cell.cuh, reference yee_update.cl:30-39, 75-117, 145-154, 195-237), so
// that every cell rounds as in the per-cell kernels (the ψ terms of an axis whose
// slab no cell of the tile touches, exact zeros there, are left out).
//
// Every mbarrier wait is bounded (MarchBox::wait_polls); on timeout the kernel
// raises a device error flag, drains the copies it issued and returns.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <cstring>

#include "launch_chain.cuh"
#include "launch_count.cuh"
#include "tma.cuh"
#include "yee_launch.cuh"

namespace fdtd {

__device__ int g_march_error = 0;

namespace {

constexpr int MARCH_MAX_PLANES = 64;  // planes of a chunk (x profiles kept in shared memory)
constexpr unsigned MARCH_DRAIN_LIMIT = 1u << 20;

struct alignas(64) MarchMaps {
    CUtensorMap m[12];  // E, H, ce, then ca when lossy
};

// Tile columns (rows) 0 .. lo-1 and n-hi .. n-1 along k (j) touch a z (y) slab.
struct TileSpan {
    int n, lo, hi;
};

struct MarchBox {
    TileSpan tj, tk;
    int tiles;             // tiles of a plane
    int nlo, nhi, xchunk;  // chunks of the planes [0, npml] and [nx - npml, nx), their planes
    int nmid, chunk;       // chunks of the planes between, their planes
    unsigned wait_polls;
    int zmix;  // a vector may hold cells on both sides of a z slab's edge
};

// Tile of TJ rows x TK cells, V consecutive cells a thread, G threads a row.
// Two CTAs an SM: a ring of four stages fits without ca, of three with it.
template <typename T, int TKK, int TJJ, bool LOSSY>
struct MTile {
    static constexpr int V = 16 / (int)sizeof(T);
    static constexpr int TK = TKK, TJ = TJJ;
    static constexpr int NSTAGE = LOSSY ? 3 : 4, NCO = LOSSY ? 6 : 3;
    static constexpr int G = TK / V;
    static constexpr int CELLTHR = G * TJ;
    static constexpr int THREADS = CELLTHR + 32;
    static_assert(G + TJ <= 32 && 32 % G == 0, "one halo warp; whole rows in a warp");
    static constexpr int EW = TK + 2 * V, EH = TJ + 2, HW = TK + V, HH = TJ + 1;
    __host__ __device__ static constexpr int pad128(int b) { return (b + 127) / 128 * 128; }
    static constexpr int EB = pad128(EW * EH * (int)sizeof(T));
    static constexpr int HB = pad128(HW * HH * (int)sizeof(T));
    static constexpr int CB = pad128(TK * TJ * (int)sizeof(T));
    static constexpr int STAGE = 3 * (EB + HB) + NCO * CB;
    static constexpr int NEW_OFF = NSTAGE * STAGE;   // two new-H planes in the H box layout
    static constexpr int PROF_OFF = NEW_OFF + 6 * HB;
    static constexpr int PM = MARCH_MAX_PLANES + 1;
    static constexpr int BAR_OFF = (PROF_OFF + 6 * PM * (int)sizeof(T) + 63) / 64 * 64;
    static constexpr int SMEM = BAR_OFF + 64 + 128;
    static_assert(2 * (SMEM + 1024) <= 228 * 1024, "two CTAs must fit an SM");
    static constexpr uint32_t TX_E = 3u * EW * EH * sizeof(T);
    static constexpr uint32_t TX_REST = (3u * HW * HH + (uint32_t)NCO * TK * TJ) * sizeof(T);
};

// The cells of mask m of a vector at p.  ALL: the mask is all or nothing.
template <typename T, int V, bool ALL>
__device__ __forceinline__ void ld_mask(const T *p, unsigned m, T (&o)[V]) {
    if (ALL) {
        if (m) ld_vec<T, V>(p, o);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (m >> v & 1u) o[v] = p[v];
    }
}
template <typename T, int V, bool ALL>
__device__ __forceinline__ void st_mask(T *p, unsigned m, const T (&in)[V]) {
    if (ALL) {
        if (m) st_vec<T, V>(p, in);
    } else {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (m >> v & 1u) p[v] = in[v];
    }
}

__device__ __forceinline__ bool march_wait(uint64_t *bar, uint32_t parity, unsigned limit) {
    if (limit == 0) {
        if (mbar_test_wait(bar, parity)) return true;
    } else {
        for (unsigned it = 0; it < limit; ++it)
            if (mbar_try_wait(bar, parity)) return true;
    }
    atomicOr(&g_march_error, 1);
    return false;
}

template <typename T, typename L, bool LOSSY, int AX>
__device__ __forceinline__ void march_tile(const MarchMaps &maps, const YeeArgs<T> &a,
                                           const MarchBox &bx, const SourceList &src,
                                           unsigned char *smem, int i0, int i1, int j0, int k0) {
    constexpr int V = L::V, G = L::G, TJ = L::TJ, EW = L::EW, HW = L::HW, PM = L::PM;
    constexpr int NSTAGE = L::NSTAGE;
    constexpr bool AXX = (AX & 1) != 0, AXY = (AX & 2) != 0, AXZ = (AX & 4) != 0;
    constexpr bool ZALL = (AX & 8) == 0;  // a vector lies all or not at all in a z slab
    const int nx = a.nx, ny = a.ny, nz = a.nz, P = a.npml;
    uint64_t *bar = reinterpret_cast<uint64_t *>(smem + L::BAR_OFF);
    const int pfirst = (i0 > 0) ? i0 - 1 : i0;  // pre-plane: H(i0-1) only
    const int tid = threadIdx.x;

    // x profiles of the chunk's planes [pfirst, i1): H ik, b, c then E ik, b, c
    T *const prof = reinterpret_cast<T *>(smem + L::PROF_OFF);
    if (AX != 0) {
        for (int q = tid; q < i1 - pfirst; q += L::THREADS) {
            prof[q] = a.cph.ik[0][pfirst + q];
            prof[3 * PM + q] = a.cpe.ik[0][pfirst + q];
            if (AXX) {
                prof[PM + q] = a.cph.b[0][pfirst + q];
                prof[2 * PM + q] = a.cph.c[0][pfirst + q];
                prof[4 * PM + q] = a.cpe.b[0][pfirst + q];
                prof[5 * PM + q] = a.cpe.c[0][pfirst + q];
            }
        }
    }
    if (tid == 0) {
        for (int s = 0; s < NSTAGE; ++s) mbar_init(&bar[s], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();

    // The warp after the cell threads, idle in the E phase, issues the copies of a
    // plane (E only for plane i1): lane c copies array c, so the boxes' addresses
    // are formed side by side.  (One cell thread issuing them all held its warp, and
    // with it the CTA's next barrier, for several hundred cycles a plane.)
    const int hl = tid - L::CELLTHR;
    const int il = hl < 3 ? 0 : (hl < 6 ? 1 : 2);  // lane's array: E, H or coefficient
    const int ioff = il == 0 ? hl * L::EB
                             : (il == 1 ? 3 * L::EB + (hl - 3) * L::HB
                                        : 3 * (L::EB + L::HB) + (hl - 6) * L::CB);
    const int ik = il == 2 ? k0 : k0 - V, ij = il == 2 ? j0 : j0 - 1;
    int last_issued = pfirst - 1;
    auto issue = [&](int p) {  // by the whole warp
        const int s = (p - pfirst) % NSTAGE;
        last_issued = p;
        if (hl == 0) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            mbar_expect_tx(&bar[s], L::TX_E + (p < i1 ? L::TX_REST : 0u));
        }
        __syncwarp();
        if (hl < (p < i1 ? 6 + L::NCO : 3))
            tma_load_3d(smem + s * L::STAGE + ioff, &maps.m[hl], &bar[s], ik, ij, p);
    };
    if (hl >= 0)
        for (int p = pfirst; p <= i1 && p < pfirst + NSTAGE; ++p) issue(p);
    // a zero budget gives up here, before the first plane can have landed
    bool w = bx.wait_polls != 0 || march_wait(&bar[0], 0, 0);

    // this thread's vector: row r, group g of the tile; the warp after the cell
    // threads takes row -1 (lanes 0 .. G-1) and group -1 (lanes G .. G+TJ-1)
    const bool own = tid < L::CELLTHR;
    const int r = own ? tid / G : (hl < G ? -1 : (hl < G + TJ ? hl - G : 0));
    const int g = own ? tid % G : (hl < G ? hl : -1);
    const int j = j0 + r, kb = k0 + V * g;
    // rows are multiples of a vector, so it lies in the grid whole or not at all
    const bool work = (own || hl < G + TJ) && j >= 0 && j < ny && kb >= 0 && kb < nz;
    const bool iny = AXY && work && (j < P || j >= ny - P);
    unsigned zm = 0;  // its cells in a z slab
    if (AXZ && work) {
#pragma unroll
        for (int v = 0; v < V; ++v)
            if (kb + v < P || kb + v >= nz - P) zm |= 1u << v;
    }
    const bool jlast = AXY && j == ny - 1, klast = AXZ && kb + V == nz;
    const bool jzero = AXY && j == 0, kzero = AXZ && kb == 0;
    // k+1 of the last cell: the next lane's first cell, or from shared memory at
    // the row's end and for group -1; k-1 of the first likewise
    const bool edge = own ? g == G - 1 : hl >= G - 1;
    const int e0 = (r + 1) * EW + V + V * g, h0 = (r + 1) * HW + V + V * g;

    // CPML coefficients of the cells' y and z coordinates (H and E staggers)
    T iky_h = T(0), by_h = T(0), cy_h = T(0), iky_e = T(0), by_e = T(0), cy_e = T(0);
    T ikz_h[V], bz_h[V], cz_h[V], ikz_e[V], bz_e[V], cz_e[V];
    if (AX != 0) {
        if (work) {
            iky_h = a.cph.ik[1][j];
            iky_e = a.cpe.ik[1][j];
            if (AXY) {
                by_h = a.cph.b[1][j];
                cy_h = a.cph.c[1][j];
                by_e = a.cpe.b[1][j];
                cy_e = a.cpe.c[1][j];
            }
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            ikz_h[v] = work ? a.cph.ik[2][kb + v] : T(0);
            ikz_e[v] = work ? a.cpe.ik[2][kb + v] : T(0);
            bz_h[v] = (AXZ && work) ? a.cph.b[2][kb + v] : T(0);
            cz_h[v] = (AXZ && work) ? a.cph.c[2][kb + v] : T(0);
            bz_e[v] = (AXZ && work) ? a.cpe.b[2][kb + v] : T(0);
            cz_e[v] = (AXZ && work) ? a.cpe.c[2][kb + v] : T(0);
        }
    }

    // offsets of the first cell at the loop's plane: grid, x, y and z stripes;
    // consecutive planes of a chunk are consecutive x layers, and the slab cells of
    // a vector consecutive z layers of one slab (the slabs are V or more apart)
    const int64_t plane = (int64_t)ny * nz, dy = (int64_t)(2 * P) * nz, dz = (int64_t)ny * (2 * P);
    const int yl = j < P ? j : P + j - (ny - P), zl = kb < P ? kb : P + kb - (nz - P);
    int64_t gi = pfirst * plane + (int64_t)j * nz + kb;
    int64_t ox = AXX ? ((int64_t)(i0 <= P ? pfirst : P + pfirst - (nx - P)) * ny + j) * nz + kb : 0;
    int64_t oy = AXY ? pfirst * dy + (int64_t)yl * nz + kb : 0;
    int64_t oz = AXZ ? pfirst * dz + (int64_t)j * (2 * P) + zl : 0;
    auto inx = [&](int p) { return AXX && (p < P || p >= nx - P); };

    // ψ of the coming plane: H (own and halo cells), E (own cells)
    T hxa[V], hxb[V], hya[V], hyb[V], hza[V], hzb[V];
    T fxa[V], fxb[V], fya[V], fyb[V], fza[V], fzb[V];
    auto load_psi = [&](T *const *psi, int xa, int xb, int ya, int yb, int za, int zb, int p,
                        int ahead, T(&qxa)[V], T(&qxb)[V], T(&qya)[V], T(&qyb)[V], T(&qza)[V],
                        T(&qzb)[V]) {
        if (AXX && work && inx(p)) {
            ld_vec<T, V>(psi[xa] + ox + ahead * plane, qxa);
            ld_vec<T, V>(psi[xb] + ox + ahead * plane, qxb);
        }
        if (AXY && iny) {
            ld_vec<T, V>(psi[ya] + oy + ahead * dy, qya);
            ld_vec<T, V>(psi[yb] + oy + ahead * dy, qyb);
        }
        if (AXZ && zm) {
            ld_mask<T, V, ZALL>(psi[za] + oz + ahead * dz, zm, qza);
            ld_mask<T, V, ZALL>(psi[zb] + oz + ahead * dz, zm, qzb);
        }
    };
    auto store_psi = [&](T *const *psi, int xa, int xb, int ya, int yb, int za, int zb, bool px,
                         const T(&qxa)[V], const T(&qxb)[V], const T(&qya)[V], const T(&qyb)[V],
                         const T(&qza)[V], const T(&qzb)[V]) {
        if (AXX && px && work) {
            st_vec<T, V>(psi[xa] + ox, qxa);
            st_vec<T, V>(psi[xb] + ox, qxb);
        }
        if (AXY && iny) {
            st_vec<T, V>(psi[ya] + oy, qya);
            st_vec<T, V>(psi[yb] + oy, qyb);
        }
        if (AXZ && zm) {
            st_mask<T, V, ZALL>(psi[za] + oz, zm, qza);
            st_mask<T, V, ZALL>(psi[zb] + oz, zm, qzb);
        }
    };
    auto load_h = [&](int p, int ahead) {
        load_psi(a.psi_h, 2, 4, 0, 5, 1, 3, p, ahead, hxa, hxb, hya, hyb, hza, hzb);
    };
    auto load_e = [&](int p, int ahead) {
        if (own) load_psi(a.psi_e, 2, 4, 0, 5, 1, 3, p, ahead, fxa, fxb, fya, fyb, fza, fzb);
    };
    // L2 prefetch of the own cells' ψ, PD planes before their loads: at 512³ the
    // loads issued one plane ahead still waited for a busy DRAM (1.92 against
    // 1.71 ms a step with it)
    constexpr int PD = 3;
    auto pf = [&](const T *q) { asm volatile("prefetch.global.L2 [%0];" ::"l"(q)); };
    auto prefetch_psi = [&](int p, int ahead) {
        if (AX == 0 || p >= i1 || !own) return;
        if (AXX && work && inx(p)) {
            const int64_t o = ox + ahead * plane;
            pf(a.psi_h[2] + o);
            pf(a.psi_h[4] + o);
            pf(a.psi_e[2] + o);
            pf(a.psi_e[4] + o);
        }
        if (AXY && iny) {
            const int64_t o = oy + ahead * dy;
            pf(a.psi_h[0] + o);
            pf(a.psi_h[5] + o);
            pf(a.psi_e[0] + o);
            pf(a.psi_e[5] + o);
        }
        if (AXZ && zm) {
            const int64_t o = oz + ahead * dz;
            pf(a.psi_h[1] + o);
            pf(a.psi_h[3] + o);
            pf(a.psi_e[1] + o);
            pf(a.psi_e[3] + o);
        }
    };
#pragma unroll
    for (int v = 0; v < V; ++v) {
        hxa[v] = hxb[v] = hya[v] = hyb[v] = hza[v] = hzb[v] = T(0);
        fxa[v] = fxb[v] = fya[v] = fyb[v] = fza[v] = fzb[v] = T(0);
    }
    for (int q = 1; q <= PD; ++q) prefetch_psi(pfirst + q, q);
    load_h(pfirst, 0);
    load_e(i0, i0 - pfirst);
    // sheet injections that can reach the cells (row and k range)
    bool src_row = false;
    for (int q = 0; q < src.n; ++q) {
        const fdtd_source &sq = src.s[q];
        src_row |= own && work && j >= sq.j0 && j < sq.j1 && sq.z >= kb && sq.z < kb + V;
    }

    const T dtm = a.dtm, dtm_dl = a.dtm_dl, inv_dl = a.inv_dl;
    T hyc[V], hzc[V];  // H^{n+1/2}(p-1) at own cells
#pragma unroll
    for (int v = 0; v < V; ++v) hyc[v] = hzc[v] = T(0);

    // stage of the loop's plane, and of the next: its index and parity
    const unsigned char *cur = smem;
    int sn = 1;
    uint32_t par = 0;
    w = w && march_wait(&bar[0], 0, bx.wait_polls);
    T *nh = reinterpret_cast<T *>(smem + L::NEW_OFF) + h0;  // new-H buffer of the plane
    constexpr int NE = L::HB / (int)sizeof(T), EE = L::EB / (int)sizeof(T);
    int nflip = 3 * NE;
    bool ok = true;
    for (int p = pfirst; p < i1; ++p) {
        w = w && march_wait(&bar[sn], par, bx.wait_polls);
        const unsigned char *nxt = smem + sn * L::STAGE;
        const T *E0 = reinterpret_cast<const T *>(cur) + e0;
        const T *E1 = reinterpret_cast<const T *>(nxt) + e0;
        const T *H0 = reinterpret_cast<const T *>(cur + 3 * L::EB) + h0;
        const bool main = p >= i0;  // else the pre-plane: H of the own cells only
        const bool px = inx(p);
        T ex0[V], ey0[V], ez0[V], hx[V], hy[V], hz[V];
        {
            T ezj[V], exj[V], ez1[V], ey1[V], exk[V], eyk[V];
            ld_vec<T, V>(E0, ex0);
            ld_vec<T, V>(E0 + EE, ey0);
            ld_vec<T, V>(E0 + 2 * EE, ez0);
            ld_vec<T, V>(E0 + 2 * EE + EW, ezj);
            ld_vec<T, V>(E0 + EW, exj);
            ld_vec<T, V>(E1 + 2 * EE, ez1);
            ld_vec<T, V>(E1 + EE, ey1);
            ld_vec<T, V>(H0, hx);
            ld_vec<T, V>(H0 + NE, hy);
            ld_vec<T, V>(H0 + 2 * NE, hz);
            T xn = __shfl_down_sync(0xffffffffu, ex0[0], 1);
            T yn = __shfl_down_sync(0xffffffffu, ey0[0], 1);
            if (edge) {
                xn = E0[V];
                yn = E0[EE + V];
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                exk[v] = v < V - 1 ? ex0[v < V - 1 ? v + 1 : v] : xn;
                eyk[v] = v < V - 1 ? ey0[v < V - 1 ? v + 1 : v] : yn;
            }
            const T ikx = AX != 0 ? prof[p - pfirst] : T(0);
            const T bx_ = AXX ? prof[PM + p - pfirst] : T(0);
            const T cx_ = AXX ? prof[2 * PM + p - pfirst] : T(0);
            const bool plast = AXX && p == nx - 1;
            auto cell = [&](int v, bool pml) {
                // the reference's zero differences at the last index of an axis,
                // which lies in that axis' slab
                const bool kl = AXZ && v == V - 1 && klast;
                const T d_zy = jlast ? T(0) : ezj[v] - ez0[v], d_xy = jlast ? T(0) : exj[v] - ex0[v];
                const T d_yz = kl ? T(0) : eyk[v] - ey0[v], d_xz = kl ? T(0) : exk[v] - ex0[v];
                const T d_zx = plast ? T(0) : ez1[v] - ez0[v], d_yx = plast ? T(0) : ey1[v] - ey0[v];
                if (!pml) {
                    hx[v] = hx[v] - dtm_dl * (d_zy - d_yz);
                    hy[v] = hy[v] - dtm_dl * (d_xz - d_zx);
                    hz[v] = hz[v] - dtm_dl * (d_yx - d_xy);
                    return;
                }
                const bool inz = AXZ && (ZALL ? zm != 0 : (zm >> v & 1u) != 0);
                T sxy = d_zy * iky_h, sxz = d_xz * ikz_h[v], syx = d_yx * ikx;
                if (AXY) {
                    const T q = iny ? by_h * hya[v] + cy_h * d_zy : T(0);
                    hya[v] = q;
                    sxy = sxy + q;
                }
                if (AXZ) {
                    const T q = inz ? bz_h[v] * hzb[v] + cz_h[v] * d_xz : T(0);
                    hzb[v] = q;
                    sxz = sxz + q;
                }
                if (AXX) {
                    const T q = px ? bx_ * hxb[v] + cx_ * d_yx : T(0);
                    hxb[v] = q;
                    syx = syx + q;
                }
                sxy = sxy - d_yz * ikz_h[v];
                sxz = sxz - d_zx * ikx;
                syx = syx - d_xy * iky_h;
                if (AXZ) {
                    const T q = inz ? bz_h[v] * hza[v] + cz_h[v] * d_yz : T(0);
                    hza[v] = q;
                    sxy = sxy - q;
                }
                if (AXX) {
                    const T q = px ? bx_ * hxa[v] + cx_ * d_zx : T(0);
                    hxa[v] = q;
                    sxz = sxz - q;
                }
                if (AXY) {
                    const T q = iny ? by_h * hyb[v] + cy_h * d_xy : T(0);
                    hyb[v] = q;
                    syx = syx - q;
                }
                hx[v] = hx[v] - dtm * sxy;
                hy[v] = hy[v] - dtm * sxz;
                hz[v] = hz[v] - dtm * syx;
            };
            if (AX == 0) {
#pragma unroll
                for (int v = 0; v < V; ++v) cell(v, false);
            } else if (ZALL) {
                if (px || iny || zm != 0) {
#pragma unroll
                    for (int v = 0; v < V; ++v) cell(v, true);
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) cell(v, false);
                }
            } else {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if (px || iny || (zm >> v & 1u))
                        cell(v, true);
                    else
                        cell(v, false);
                }
            }
            if (work) {
                st_vec<T, V>(nh, hx);
                st_vec<T, V>(nh + NE, hy);
                st_vec<T, V>(nh + 2 * NE, hz);
                if (own && main) {
                    st_vec<T, V>(a.H_next[0] + gi, hx);
                    st_vec<T, V>(a.H_next[1] + gi, hy);
                    st_vec<T, V>(a.H_next[2] + gi, hz);
                }
            }
            if (own && main)
                store_psi(a.psi_h_next, 2, 4, 0, 5, 1, 3, px, hxa, hxb, hya, hyb, hza, hzb);
            prefetch_psi(p + 1 + PD, 1 + PD);
            if (AX != 0 && p + 1 < i1) load_h(p + 1, 1);
        }
        // new H complete; everyone is past plane p-1
        if (!__syncthreads_and(w)) {  // CTA-uniform exit on a timed-out copy
            ok = false;
            break;
        }
        if (hl >= 0 && p > pfirst && p - 1 + NSTAGE <= i1) issue(p - 1 + NSTAGE);
        if (own && main) {
            T hzj[V], hxj[V], hxk[V], hyk[V], cex[V], cey[V], cez[V], cax[V], cay[V], caz[V];
            ld_vec<T, V>(nh + 2 * NE - HW, hzj);
            ld_vec<T, V>(nh - HW, hxj);
            T xn = __shfl_up_sync(0xffffffffu, hx[V - 1], 1);
            T yn = __shfl_up_sync(0xffffffffu, hy[V - 1], 1);
            if (g == 0) {
                xn = nh[-1];
                yn = nh[NE - 1];
            }
#pragma unroll
            for (int v = 0; v < V; ++v) {
                hxk[v] = v ? hx[v ? v - 1 : 0] : xn;
                hyk[v] = v ? hy[v ? v - 1 : 0] : yn;
            }
            const T *C0 = reinterpret_cast<const T *>(cur + 3 * (L::EB + L::HB)) + r * L::TK + V * g;
            constexpr int CE = L::CB / (int)sizeof(T);
            ld_vec<T, V>(C0, cex);
            ld_vec<T, V>(C0 + CE, cey);
            ld_vec<T, V>(C0 + 2 * CE, cez);
            if (LOSSY) {
                ld_vec<T, V>(C0 + 3 * CE, cax);
                ld_vec<T, V>(C0 + 4 * CE, cay);
                ld_vec<T, V>(C0 + 5 * CE, caz);
            } else {
#pragma unroll
                for (int v = 0; v < V; ++v) cax[v] = cay[v] = caz[v] = T(1);
            }
            if (src_row) {
#pragma unroll
                for (int v = 0; v < V; ++v)
                    ex0[v] = apply_sources<T>(src, p, j, kb + v, ex0[v], cex[v]);
            }
            const T ikx = AX != 0 ? prof[3 * PM + p - pfirst] : T(0);
            const T bx_ = AXX ? prof[4 * PM + p - pfirst] : T(0);
            const T cx_ = AXX ? prof[5 * PM + p - pfirst] : T(0);
            const bool pzero = AXX && p == 0;
            auto cell = [&](int v, bool pml) {
                // zero differences at index 0 of an axis
                const bool kz = AXZ && v == 0 && kzero;
                DH<T> d;
                d.zy = jzero ? T(0) : hz[v] - hzj[v];
                d.xy = jzero ? T(0) : hx[v] - hxj[v];
                d.yz = kz ? T(0) : hy[v] - hyk[v];
                d.xz = kz ? T(0) : hx[v] - hxk[v];
                d.zx = pzero ? T(0) : hz[v] - hzc[v];
                d.yx = pzero ? T(0) : hy[v] - hyc[v];
                if (!pml) {
                    e_interior<T, LOSSY>(d, inv_dl, cax[v], cay[v], caz[v], cex[v], cey[v], cez[v],
                                         ex0[v], ey0[v], ez0[v]);
                    return;
                }
                const bool inz = AXZ && (ZALL ? zm != 0 : (zm >> v & 1u) != 0);
                T sxy = d.zy * iky_e, sxz = d.xz * ikz_e[v], syx = d.yx * ikx;
                if (AXY) {
                    const T q = iny ? by_e * fya[v] + cy_e * d.zy : T(0);
                    fya[v] = q;
                    sxy = sxy + q;
                }
                if (AXZ) {
                    const T q = inz ? bz_e[v] * fzb[v] + cz_e[v] * d.xz : T(0);
                    fzb[v] = q;
                    sxz = sxz + q;
                }
                if (AXX) {
                    const T q = px ? bx_ * fxb[v] + cx_ * d.yx : T(0);
                    fxb[v] = q;
                    syx = syx + q;
                }
                sxy = sxy - d.yz * ikz_e[v];
                sxz = sxz - d.zx * ikx;
                syx = syx - d.xy * iky_e;
                if (AXZ) {
                    const T q = inz ? bz_e[v] * fza[v] + cz_e[v] * d.yz : T(0);
                    fza[v] = q;
                    sxy = sxy - q;
                }
                if (AXX) {
                    const T q = px ? bx_ * fxa[v] + cx_ * d.zx : T(0);
                    fxa[v] = q;
                    sxz = sxz - q;
                }
                if (AXY) {
                    const T q = iny ? by_e * fyb[v] + cy_e * d.xy : T(0);
                    fyb[v] = q;
                    syx = syx - q;
                }
                ex0[v] = (LOSSY ? cax[v] * ex0[v] : ex0[v]) + cex[v] * sxy;
                ey0[v] = (LOSSY ? cay[v] * ey0[v] : ey0[v]) + cey[v] * sxz;
                ez0[v] = (LOSSY ? caz[v] * ez0[v] : ez0[v]) + cez[v] * syx;
            };
            if (AX == 0) {
#pragma unroll
                for (int v = 0; v < V; ++v) cell(v, false);
            } else if (ZALL) {
                if (px || iny || zm != 0) {
#pragma unroll
                    for (int v = 0; v < V; ++v) cell(v, true);
                } else {
#pragma unroll
                    for (int v = 0; v < V; ++v) cell(v, false);
                }
            } else {
#pragma unroll
                for (int v = 0; v < V; ++v) {
                    if (px || iny || (zm >> v & 1u))
                        cell(v, true);
                    else
                        cell(v, false);
                }
            }
            if (work) {
                st_vec<T, V>(a.E_next[0] + gi, ex0);
                st_vec<T, V>(a.E_next[1] + gi, ey0);
                st_vec<T, V>(a.E_next[2] + gi, ez0);
            }
            store_psi(a.psi_e, 2, 4, 0, 5, 1, 3, px, fxa, fxb, fya, fyb, fza, fzb);
            if (AX != 0 && p + 1 < i1) load_e(p + 1, 1);
        }
#pragma unroll
        for (int v = 0; v < V; ++v) {
            hyc[v] = hy[v];
            hzc[v] = hz[v];
        }
        gi += plane;
        if (AXX) ox += plane;
        if (AXY) oy += dy;
        if (AXZ) oz += dz;
        cur = nxt;
        nh += nflip;
        nflip = -nflip;
        if (++sn == NSTAGE) {
            sn = 0;
            par ^= 1;
        }
    }
    if (!ok) {
        // drain: every copy issued must land before the CTA exits; only the
        // last NSTAGE issued planes can still be in flight
        __syncthreads();
        if (hl == 0) {
            const int from = max(pfirst, last_issued - NSTAGE + 1);
            for (int p = from; p <= last_issued; ++p) {
                const int s = (p - pfirst) % NSTAGE;
                const uint32_t q = ((p - pfirst) / NSTAGE) & 1;
                for (unsigned it = 0; it < MARCH_DRAIN_LIMIT; ++it)
                    if (mbar_try_wait(&bar[s], q)) break;
            }
        }
        __syncthreads();
    }
}

// The q-th tile row or column that touches a slab (edge) or does not.
__device__ __forceinline__ int span_edge(const TileSpan &s, int q) {
    return q < s.lo ? q : s.n - s.hi + (q - s.lo);
}

// CTAs in the order of their variant, the costliest first: the x chunks
// (planes [0, npml] and [nx - npml, nx)), then the middle chunks of the tiles
// that touch y and z slabs, y, z, none.  CTAs that share an SM then mostly run
// the same code: in tile order, warps waited for instructions a third of the
// time (the variants' loops together exceed the instruction caches; 386 against
// 329 us a step at 256³).
//
// Bound by DRAM at large grids.  Measured (FP32 lossless, whole step without
// DFT, against the interior march with shell kernels): 512³ npml 16 1.60 against
// 1.87 ms (8.9 GB: 5.5 TB/s), 256³ npml 12 0.25 against 0.32 ms; FP64 384³ 1.36
// against 1.56 ms.  Two CTAs of four stages an SM: three of three stages (ce by
// plain loads, the ring holds no more) took 1.83 ms at 512³, five stages without ce
// in the ring 1.71, two cells a thread instead of four the same time.
template <typename T, typename L, bool LOSSY>
__global__ void __launch_bounds__(L::THREADS, 2)
    k_march(const __grid_constant__ MarchMaps maps, const __grid_constant__ YeeArgs<T> a,
            const __grid_constant__ MarchBox bx, const __grid_constant__ SourceList src) {
    chain_next();
    chain_wait();
    extern __shared__ __align__(128) unsigned char smem_raw[];
    unsigned char *smem = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 127) & ~uintptr_t(127));
    const TileSpan &tj = bx.tj, &tk = bx.tk;
    const int je = tj.lo + tj.hi, ke = tk.lo + tk.hi, jm = tj.n - je, km = tk.n - ke;
    const int n_yz = je * ke, n_y = je * km, n_z = jm * ke, n_0 = jm * km;
    // position b among the x (or middle) CTAs of a class of n tiles, chunk-major
    const int nxc = bx.nlo + bx.nhi;
    int b = blockIdx.x, n = n_yz, cls = 0;
    const bool xs = b < nxc * bx.tiles;
    if (!xs) b -= nxc * bx.tiles;
    const int per = xs ? nxc : bx.nmid;
    if (b >= n * per) {
        b -= n * per;
        n = n_y;
        cls = 1;
        if (b >= n * per) {
            b -= n * per;
            n = n_z;
            cls = 2;
            if (b >= n * per) {
                b -= n * per;
                n = n_0;
                cls = 3;
            }
        }
    }
    const int c = b / n;
    b -= c * n;
    const bool y = cls < 2, z = cls == 0 || cls == 2;
    const int w = z ? ke : km;
    const int tr = b / w, tc = b % w;
    const int j0 = (y ? span_edge(tj, tr) : tj.lo + tr) * L::TJ;
    const int k0 = (z ? span_edge(tk, tc) : tk.lo + tc) * L::TK;
    const int nx = a.nx, P = a.npml;
    int i0, i1;
    if (!xs) {
        i0 = P + 1 + c * bx.chunk;
        i1 = min(nx - P, i0 + bx.chunk);
    } else if (c < bx.nlo) {
        i0 = c * bx.xchunk;
        i1 = min(P + 1, i0 + bx.xchunk);
    } else {
        i0 = nx - P + (c - bx.nlo) * bx.xchunk;
        i1 = min(nx, i0 + bx.xchunk);
    }
    if (i0 >= i1) return;  // CTA-uniform, before any barrier
#define FDTD_TILE(AX) \
    march_tile<T, L, LOSSY, AX>(maps, a, bx, src, smem, i0, i1, j0, k0)
    const bool mix = bx.zmix != 0;
    if (xs) {
        if (!y && !z)
            FDTD_TILE(1);
        else if (mix)
            FDTD_TILE(15);
        else
            FDTD_TILE(7);
    } else if (cls == 0) {
        if (mix)
            FDTD_TILE(14);
        else
            FDTD_TILE(6);
    } else if (cls == 1) {
        FDTD_TILE(2);
    } else if (cls == 2) {
        if (mix)
            FDTD_TILE(12);
        else
            FDTD_TILE(4);
    } else {
        FDTD_TILE(0);
    }
#undef FDTD_TILE
}

// Tiles of w cells over n cells whose own cells or halo (one cell below) lie in
// a CPML slab of P layers.
TileSpan tile_span(int n, int w, int P) {
    TileSpan s;
    s.n = (n + w - 1) / w;
    s.lo = s.hi = 0;
    for (int t = 0; t < s.n; ++t) {
        const int first = t * w > 0 ? t * w - 1 : 0, last = ((t + 1) * w < n ? (t + 1) * w : n) - 1;
        if (first < P)
            ++s.lo;
        else if (last >= n - P)
            ++s.hi;
    }
    return s;
}

template <typename T, typename L, bool LOSSY>
bool build_march_maps(const YeeArgs<T> &a, MarchMaps &m) {
    const int elem = (int)sizeof(T);
    static KeyedCache<MarchMaps, 15> cache;  // the maps of the last few buffer sets
    uint64_t key[15];
    for (int c = 0; c < 3; ++c) {
        key[c] = (uint64_t)(uintptr_t)a.E[c];
        key[3 + c] = (uint64_t)(uintptr_t)a.H[c];
    }
    key[6] = (uint64_t)a.nx;
    key[7] = (uint64_t)a.ny;
    key[8] = (uint64_t)a.nz;
    const T *coef[6];
    for (int c = 0; c < 6; ++c) {
        coef[c] = c < 3 ? a.ce[c] : (LOSSY ? a.ca[c - 3] : nullptr);
        key[9 + c] = (uint64_t)(uintptr_t)coef[c];
    }
    if (cache.get(key, m)) return true;
    memset(&m, 0, sizeof(m));
    for (int c = 0; c < 3; ++c)
        if (!make_tensor_map(&m.m[c], a.E[c], a.nx, a.ny, a.nz, elem, L::EW, L::EH) ||
            !make_tensor_map(&m.m[3 + c], a.H[c], a.nx, a.ny, a.nz, elem, L::HW, L::HH))
            return false;
    for (int c = 0; c < L::NCO; ++c)
        if (!make_tensor_map(&m.m[6 + c], coef[c], a.nx, a.ny, a.nz, elem, L::TK, L::TJ))
            return false;
    cache.put(key, m);
    return true;
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

// Chunks along x.  A CTA costs its planes plus about two and a half (pipeline
// fill, the H-only plane before and the E-only plane after), an x-CPML plane
// about 1.6 middle ones.  CTAs that fit the slots (two per SM) run as one wave of
// the longest, which lies in a y or z slab and takes about 1.6 middle ones a plane
// too; more, the costliest first, run at the mean load plus about half a chunk of
// tail.  (Without the 1.6, grids of 1 to 4 M cells got one wave of long chunks, slower
// than the schedules that the march replaces: FP64 112³ npml 8 74.2 us a step against
// 54.5 now, 56 by two whole-grid launches and 53 by the interior march; 314x56x144 npml 4
// 108 / 82 / 90 / 88; FP32 252x197x56 npml 3 85 / 62 / 61 / 72, 404x62x184 npml 4 98 / 82 /
// 88 / 82, 270x46x392 npml 4 116 / 89 / 89 / 84.)
void march_chunks(MarchBox &bx, int P, int mid) {
    const int slots = 2 * device_sm_count();
    double best = 1e30;
    for (int n = 1; n <= mid; ++n) {
        const int len = ceil_div(mid, n);
        if (len > MARCH_MAX_PLANES) continue;
        if (len < 2 && n > 1) break;
        const int nlo = ceil_div(P + 1, len), xlen = ceil_div(P + 1, nlo);
        const int nx2 = nlo + ceil_div(P, xlen);
        const int nm = ceil_div(mid, len);
        const double cx = 1.6 * (xlen + 2.5), cm = len + 2.5;
        const double load = bx.tiles * (nm * cm + nx2 * cx) / slots;
        const double longest = cx > cm ? cx : cm;
        const double est = bx.tiles * (nm + nx2) <= slots ? 1.6 * longest : load + 0.5 * longest;
        if (est < best - 1e-9) {
            best = est;
            bx.chunk = len;
            bx.nmid = nm;
            bx.xchunk = xlen;
            bx.nlo = nlo;
            bx.nhi = nx2 - nlo;
        }
    }
}

template <typename T, int TK, int TJ, bool LOSSY>
cudaError_t launch_march_t(const YeeArgs<T> &a, const SourceList &src, cudaStream_t st) {
    using L = MTile<T, TK, TJ, LOSSY>;
    MarchMaps maps;
    if (!build_march_maps<T, L, LOSSY>(a, maps)) return cudaErrorNotSupported;
    MarchBox bx;
    memset(&bx, 0, sizeof(bx));
    bx.tk = tile_span(a.nz, TK, a.npml);
    bx.tj = tile_span(a.ny, TJ, a.npml);
    bx.tiles = bx.tk.n * bx.tj.n;
    march_chunks(bx, a.npml, a.nx - 2 * a.npml - 1);
    bx.wait_polls = interior_wait_polls();
    bx.zmix = a.npml % L::V != 0;
    cudaError_t e = ensure_max_dynamic_smem((const void *)k_march<T, L, LOSSY>, L::SMEM);
    if (e != cudaSuccess) return e;
    const unsigned ctas = (unsigned)(bx.tiles * (bx.nmid + bx.nlo + bx.nhi));
    e = launch_chained(k_march<T, L, LOSSY>, ctas, L::THREADS, L::SMEM, st, maps, a, bx, src);
    count_launches(1);
    return e;
}

bool aligned16(const void *p) { return reinterpret_cast<uintptr_t>(p) % 16 == 0; }

}  // namespace

template <typename T>
bool march_path_ok(const YeeArgs<T> &a) {
    constexpr int V = 16 / (int)sizeof(T);
    const int P = a.npml;
    // TMA: rows of 16-byte multiples
    if (P < 1 || a.nz % V != 0) return false;
    if (a.xb.pml_lo != P || a.xb.pml_hi != P || a.ghost_lo != 0 || a.ghost_hi != 0) return false;
    // the two slabs of an axis apart, on z by a whole vector
    if (a.nx - 2 * P < 2 || a.ny - 2 * P < 2 || a.nz - 2 * P < V) return false;
    for (int q = 0; q < 6; ++q) {
        if (!a.psi_h_next[q] || a.psi_h_next[q] == a.psi_h[q]) return false;
        if (!aligned16(a.psi_h[q]) || !aligned16(a.psi_h_next[q]) || !aligned16(a.psi_e[q]))
            return false;
    }
    for (int c = 0; c < 3; ++c)
        if (!aligned16(a.E[c]) || !aligned16(a.H[c]) || !aligned16(a.E_next[c]) ||
            !aligned16(a.H_next[c]) || !aligned16(a.ce[c]) || (a.lossy && !aligned16(a.ca[c])))
            return false;
    if (!march_size<T>((int64_t)a.nx * a.ny * a.nz)) return false;
    return march_pays<T>(a.nx, a.ny, a.nz, P, a.lossy != 0, march_narrow<T>(a.nz),
                         march_pad<T>(a.ny, a.nz));
}

// cudaErrorNotSupported, with nothing launched, when the tensor maps cannot be built.
template <typename T>
cudaError_t launch_march(const YeeArgs<T> &a, const SourceList &src, cudaStream_t st) {
    constexpr int W = 256 / (int)sizeof(T), N = W / 2;
    // march_pays: lossy grids in FP32 and the wide tile only
    if (march_narrow<T>(a.nz)) return launch_march_t<T, N, 16, false>(a, src, st);
    if constexpr (sizeof(T) == 4)
        if (a.lossy) return launch_march_t<T, W, 8, true>(a, src, st);
    return launch_march_t<T, W, 8, false>(a, src, st);
}

template bool march_path_ok<float>(const YeeArgs<float> &);
template bool march_path_ok<double>(const YeeArgs<double> &);
template cudaError_t launch_march<float>(const YeeArgs<float> &, const SourceList &, cudaStream_t);
template cudaError_t launch_march<double>(const YeeArgs<double> &, const SourceList &,
                                          cudaStream_t);

int read_march_error(int reset) {
    int v = 0;
    cudaMemcpyFromSymbol(&v, g_march_error, sizeof(int));
    if (reset) {
        int z = 0;
        cudaMemcpyToSymbol(g_march_error, &z, sizeof(int));
    }
    return v;
}

}  // namespace fdtd
