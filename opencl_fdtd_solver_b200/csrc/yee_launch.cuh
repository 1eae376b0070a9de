// Typed kernel arguments and launcher declarations for the Yee kernels.
#pragma once
#include <cuda_runtime.h>

#include "yee_cell.cuh"

namespace fdtd {

// Everything a Yee kernel needs, by value (device pointers + scalars already
// rounded to T).  E/H are read (and, for the split kernels, written in place);
// E_next/H_next are the fused step's outputs, psi_h_next its advanced psi_H
// (== psi_h: in place).
template <typename T>
struct YeeArgs {
    int nx, ny, nz, npml, lossy;
    XBounds xb;        // x CPML layers per face and interior x bounds (slabs)
    int ghost_lo, ghost_hi;  // ghost planes at x = 0 / nx-1 (slabs only)
    T dtm, dtm_dl, inv_dl;
    T *E[3];
    T *H[3];
    T *E_next[3];
    T *H_next[3];
    const T *ce[3];
    const T *ca[3];
    Cpml1D<T> cph, cpe;
    T *psi_h[6];
    T *psi_h_next[6];
    T *psi_e[6];
};

// Box [lo, hi) per axis; lo == hi == 0 on every axis means "no box".
struct ShellBox {
    int lo[3], hi[3];
};

template <typename T>
cudaError_t launch_shell_H(const YeeArgs<T> &a, const ShellBox &b, cudaStream_t st);
template <typename T>
cudaError_t launch_shell_E(const YeeArgs<T> &a, const ShellBox &b, const SourceList &src,
                           const PlaneList &pl, cudaStream_t st);
// E^{n+1} of the cells of box o outside box b (b empty: all of o).
template <typename T>
cudaError_t launch_shell_E_region(const YeeArgs<T> &a, const ShellBox &o, const ShellBox &b,
                                  const SourceList &src, const PlaneList &pl, cudaStream_t st);

// Plane-DFT accumulation for the monitored planes' cells inside box b (read
// back from E_next / H_next after the interior update).
template <typename T>
cudaError_t launch_plane_dft_box(const YeeArgs<T> &a, const ShellBox &b, const PlaneList &pl,
                                 cudaStream_t st);

struct SideStream;

// Shell E of the fused step through the CPML face kernels (yee_face.cu): the
// six face slabs as TMA plane marches on st, the remaining shell cells by the
// per-cell kernel on the side stream, joined back to st; no plane DFTs (the
// caller accumulates the monitored planes afterwards); cudaErrorNotSupported,
// with nothing launched, when the tensor maps cannot be built.  face_path_ok:
// the grid qualifies (whole grid, npml a multiple of 16 bytes of elements,
// aligned stripes).
int face_mode();  // FDTD_B200_FACE_E: 1 forced on, 0 off, -1 unset
template <typename T>
bool face_path_ok(const YeeArgs<T> &a);
template <typename T>
cudaError_t launch_shell_E_faces(const YeeArgs<T> &a, const SourceList &src, cudaStream_t st,
                                 SideStream *side);
int read_face_error(int reset);

// Fraction of a grid's cells in a CPML slab.
inline double pml_fraction(int nx, int ny, int nz, int npml) {
    auto in = [&](int n) { return n > 2 * npml ? (double)(n - 2 * npml) / n : 0.0; };
    return 1.0 - in(nx) * in(ny) * in(nz);
}

// The march takes grids whose step (15 arrays: six fields read, six written,
// three coefficients) clearly exceeds the 126 MB L2.  Below, more threads beat
// fewer bytes: the march's planes follow one another, about 1.7 us each.
// Measured per step with a source and a plane DFT, march against one whole-grid H
// and one E launch: FP32 64³ 20.6 / 16.4 us, 96³ 29.8 / 28.0, 128³ 64.4 / 59.7,
// 160x160x96 69.1 / 69.8, 192³ 141.9 / 174.5; FP64 96³ 62.3 / 44.2, 128³ 85.5 / 95.9.
constexpr int64_t MARCH_MIN_BYTES = 140000000;
template <typename T>
inline bool march_size(int64_t cells) {
    return 15 * cells * (int64_t)sizeof(T) >= MARCH_MIN_BYTES;
}

// And whose CPML is not most of the grid: its CPML tiles evaluate their cells in
// fewer, longer threads.  In ps per FP32 cell the march costs about (11 + 20 f)
// per cell of its (padded) tiles, f the CPML fraction, 1.17 times that with ca; the
// two whole-grid launches 21 + 4 f, 1.08 times with ca.  Measured, march / whole-grid
// launches in us: 256³ npml 20 lossy (f 0.40) 349.9 / 363.9, 192³ npml 20 lossy
// (0.50) 161 / 171, 100x300x200 npml 20 (0.58) 154.4 / 137.5, 160³ npml 20 lossy
// (0.58) 124.2 / 108.6, 34x483x224 npml 13 (0.80) 117.8 / 94.6.
inline bool march_pays(int nx, int ny, int nz, int npml, bool lossy, int tk, int tj) {
    const double pad = (double)((nz + tk - 1) / tk * tk) / nz * ((ny + tj - 1) / tj * tj) / ny;
    const double f = pml_fraction(nx, ny, nz, npml);
    return pad * (11.0 + 20.0 * f) * (lossy ? 1.17 : 1.0) < (21.0 + 4.0 * f) * (lossy ? 1.08 : 1.0);
}

// The whole step but the plane DFTs as one plane march over the grid, CPML
// included (yee_march.cu): reads E/H/psi_h, writes E_next/H_next/psi_h_next,
// psi_e in place.  march_path_ok: the grid and buffers qualify.
template <typename T>
bool march_path_ok(const YeeArgs<T> &a);
template <typename T>
cudaError_t launch_march(const YeeArgs<T> &a, const SourceList &src, cudaStream_t st);
int read_march_error(int reset);
unsigned interior_wait_polls();

template <typename T>
cudaError_t launch_update_H(const YeeArgs<T> &a, cudaStream_t st);
template <typename T>
cudaError_t launch_update_E(const YeeArgs<T> &a, const SourceList &src, const PlaneList &pl,
                            cudaStream_t st);
template <typename T>
cudaError_t launch_add_source(int nx, int ny, int nz, const fdtd_source &s, T *Ex,
                              const T *ce_x, cudaStream_t st);
// Fused step: shell H, interior single-pass kernel, shell E.  Reads E/H/psi,
// writes E_next/H_next (psi in place).  Falls back to the shell kernels over
// the whole grid when the interior kernel's TMA alignment does not hold.
template <typename T>
cudaError_t launch_step_fused(const YeeArgs<T> &a, const SourceList &src, const PlaneList &pl,
                              cudaStream_t st);

}  // namespace fdtd
