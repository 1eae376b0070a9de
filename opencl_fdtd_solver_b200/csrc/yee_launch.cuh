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
// Measured per step with a z-plane DFT, march against one whole-grid H and one E
// launch: FP32 64³ 18.4 / 13.0 us, 96³ 28.3 / 22.6, 128³ 55.4 / 50.0, 160³ 89.7 / 89.6,
// 192³ 124.1 / 143.5; FP64 96³ 44.6 / 35.8, 112³ 62.2 / 58.2, 128³ 79.2 / 81.2.
constexpr int64_t MARCH_MIN_BYTES = 140000000;
template <typename T>
inline bool march_size(int64_t cells) {
    return 15 * cells * (int64_t)sizeof(T) >= MARCH_MIN_BYTES;
}

// Padding of a grid's (j, k) plane to whole tiles.
inline double tile_pad(int ny, int nz, int tk, int tj) {
    return (double)((nz + tk - 1) / tk * tk) / nz * ((ny + tj - 1) / tj * tj) / ny;
}

// Lossless grids that the march's tiles pad and whose z slabs are a tenth of the rows
// at most stay with the interior march and its shell kernels, if the planes are few.
// Per step in us, interior march / march / two whole-grid launches: FP32 72x224x328
// npml 4 81.8 / 96.0 / 94.3, 200³ npml 4 127.8 / 140.8 / 139.1, 328x224x208 npml 8 232 /
// 243 / 265, but 368x224x272 npml 4 344 / 316 / 369; FP64 48x292x104 npml 4 52.9 / 61.8 /
// 55.0, 120x239x136 npml 4 114 / 126 / 128, but 355x136x52 npml 6 118.8 / 90.5 / 94.8.
// (Just above the line of 1.05 the march can win: FP32 256x168x304 npml 6, padded by
// 1.053, 206.8 / 200.4 / 221.5.)
inline bool interior_pays(int nx, int nz, int npml, double pad) {
    return pad > 1.05 && nz >= 20 * npml && (nx <= 256 || pad > 1.2);
}

// Padding of the interior box's (j, k) extent to the interior march's 64 x 8 (FP64: 32 x
// 8) tiles, which start on a 16-byte boundary.
template <typename T>
inline double interior_pad(int ny, int nz, int npml) {
    constexpr int V = 16 / (int)sizeof(T);
    return tile_pad(ny - 2 * npml, nz - npml - npml / V * V, 256 / (int)sizeof(T), 8);
}

// And those, not for the march, with long rows, enough cells and little CPML, or whose
// interior box fits the tiles: FP32, interior march / two whole-grid launches, 84x296x264
// npml 10 119.7 / 128.0, 62x200x352 npml 8 82.0 / 86.1, 328x224x208 npml 8 232 / 265, 144³
// npml 8 58.2 / 63.7, 192x162x144 npml 10 91.3 / 93.4; but 280x216x80 npml
// 6 126 / 99, 160x160x96 npml 12 64.5 / 57.7.
template <typename T>
inline bool interior_beats_grid(int nx, int ny, int nz, int npml) {
    const int64_t cells = (int64_t)nx * ny * nz;
    const double f = pml_fraction(nx, ny, nz, npml);
    const int row = nz * (int)sizeof(T);
    return (row >= 768 && cells * (int)sizeof(T) >= 16000000 && f <= 0.42) ||
           (row >= 512 && f <= 0.4 && interior_pad<T>(ny, nz, npml) < 1.1);
}

// Where the march beats the two whole-grid launches.  Its CPML tiles evaluate their
// cells in fewer, longer threads, its padding is work, and the narrower tile streams
// less well in FP32.  In ps per cell, f the CPML fraction, lossless FP32 grids below
// 10 M cells take about pad (11 + 20 f), 1.45 times that in narrow tiles, against 18 +
// 7 f; measured, march / whole-grid launches in us: 192³ npml 20 132 / 148, 280x216x80 npml
// 6 (narrow) 108 / 98, 240x48x280 npml 10 79 / 71, but 160x160x96 npml 12 (narrow) 53.1 /
// 57.7 goes to the launches and 150x136x176 npml 10 82.4 / 74.0 to the march: chunks are
// whole planes, and the estimate is good to a tenth.  Above, the bytes count: 344x136x272
// npml 16 214 / 241, 398x160x336 npml 20 350 / 405.  FP64: 192³ npml 8 193 / 227,
// 34x483x224 npml 13 170 / 156, 384³ npml 16 1366 / 1737.  Lossy (a deeper read per cell,
// one stage less in the ring): 192³ npml 20 159 / 163, 256³ npml 12 326 / 336, but padded
// 200³ npml 4 194 / 157 and FP64 192³ npml 8 (interior march) 300 / 240.
// Of 1460 random grids of 0.4 M to 200 M cells with npml 3 to 20, 18 run more than 5 %
// (one 17 %) slower by all these rules than by the interior march; their mean is 13 % faster.
template <typename T>
inline bool march_pays(int nx, int ny, int nz, int npml, bool lossy, bool narrow, double pad) {
    const int64_t cells = (int64_t)nx * ny * nz;
    if (lossy) return sizeof(T) == 4 && !narrow && pad < 1.05 && cells >= 7000000;
    if (interior_pays(nx, nz, npml, pad)) return false;
    const double f = pml_fraction(nx, ny, nz, npml), march = pad * (11.0 + 20.0 * f);
    if (sizeof(T) == 8) return march < 21.0 + 4.0 * f;
    if (!narrow && cells >= 10000000) return f < 0.6;
    return (narrow ? 1.45 : 1.0) * march < 18.0 + 7.0 * f;
}

// Tile of a grid's march: 64 x 8 (FP64: 32 x 8) cells streams better; the narrower one
// is taken where it saves a fifth of the padded k extent.
template <typename T>
inline bool march_narrow(int nz) {
    constexpr int W = 256 / (int)sizeof(T), N = W / 2;
    return 5 * ((nz + W - 1) / W * W) > 6 * ((nz + N - 1) / N * N);
}
template <typename T>
inline double march_pad(int ny, int nz) {
    const bool narrow = march_narrow<T>(nz);
    return tile_pad(ny, nz, (narrow ? 128 : 256) / (int)sizeof(T), narrow ? 16 : 8);
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
// Which of the FDTD_SCHEDULE_* it takes for the arguments' grid and buffers.
// march: the march may be taken; it may not once its tensor maps could not be built.
template <typename T>
int step_schedule(const YeeArgs<T> &a, bool march = true);

}  // namespace fdtd
