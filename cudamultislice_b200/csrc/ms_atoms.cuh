// ms_atoms.cuh -- atom index (bit-exact binning) and projected-potential build.
#pragma once
#include <cuda_runtime.h>
#include "ms_common.cuh"

namespace ms {

// Box as computed by LoadAtomFile (U.cu:1350-1355).
struct Box {
  float MaxX, MinX, MaxY, MinY, MaxZ, MinZ;
};

// Device atom index: atoms sorted slice -> y-bin -> x-bin, stable in input
// order, positions shifted by the box minimum (U.cu:1444-1525).
struct AtomIndex {
  float4* atoms;   // (x, y, z, Z as int bits), shifted frame
  int* off;        // CSR offsets, nz * 2500 + 1
  int n;           // atoms
  int nz;          // 1-A z-bins
};

// Scratch for building the index (all sized by n or by the bin count).
struct BinScratch {
  int* key;      // n
  int* idx;      // n
  int* cursor;   // nbins
  int* blocksum; // scan partials
};

size_t bin_scratch_blocks(int nbins);
// First sorted atom of every z-bin (and the atom count) of nb indices whose
// offsets lie off_stride apart: out[k * (nz + 1) + z].
cudaError_t zbin_starts(const int* off, long long off_stride, int nz, int nb, int* out, cudaStream_t s);
// The Gaussians of every element at the radial bins' centres (PotArgs::gbin)
// from the expansions (PotArgs::gauss).
cudaError_t build_gauss_bins(const float* gauss, float* gbin, cudaStream_t s);
cudaError_t build_atom_index(const int* dZ, const float* dx, const float* dy, const float* dz, int n,
                             const Box& box, int nz, AtomIndex& out, BinScratch& scr, cudaStream_t s);

// Per-Z coefficients of vatom / vzatom2 derived from one fparams row on the
// host in FP64: 12 floats for vatom, then 12 for vzatom2 (see engine).
constexpr int kCoefPerZ = 24;

enum PotKind : int { POT_CONVENTIONAL = 0, POT_FD = 1, POT_PROJECTED = 2, POT_RS = 3 };

struct PotArgs {
  const float4* atoms;
  const int* off;
  const float* coef;     // [103][kCoefPerZ]
  float* V;              // [ny][nx] output (V*A, not yet exponentiated)
  int nx, ny, nz;
  float ps, xoff, yoff;  // pixel (x,y) sits at (xoff + x*ps, yoff + y*ps) in the shifted frame
  float bw_x, bw_y;      // bin widths (MaxX-MinX)/50, (MaxY-MinY)/50
  int kt, kb;            // inclusive z-bin window
  int nsub;              // sub-planes (20 conventional, 1 finite difference)
  float zsub[20];        // sub-plane z (shifted frame), FP32 as the reference
  float zsub_lo[20];     // exact height minus zsub (values only; the cut-off
                         // decisions use zsub as the reference rounds it)
  float wsub;            // weight per sub-plane
  // projected mode: atoms with floorf((top - z)/dz) == slab
  float top, slab_dz;
  int slab;
  long long batch_stride_V;
  // separable conventional kernel: per-atom tables of the slice (written by
  // the table kernel, kTabStride floats per atom of the z-window, in CSR
  // order) and the Gaussian expansions [103][2][kGaussJ] (alpha_j log2(e),
  // then w_j)
  float* tab;
  const float* gauss;
  const float* gbin;     // exp(-alpha_j s) at the radial bins' centres [103][kRadBins][kGaussJ]
  // batched separable builds (one instance per blockIdx.z of the pixel kernel,
  // blockIdx.y of the table kernel): element strides of atoms, off, tab and V
  // between instances (0 for one instance)
  long long b_atoms, b_off, b_tab, b_V;
};

// Gaussian expansion of vatom per element: v(r) ~= sum_j w_j exp(-alpha_j r^2)
// for 0.25 A <= r <= 2.2365 A (positive weights).
constexpr int kGaussJ = 12;
// The radial function of an atom in one slice, G(rho^2) = sum over the planes
// that pass the cut-off of wsub v(rho^2 + dz_k^2), as polynomials in rho^2 for
// the pixel kernels.  With s = fadd(rho^2, dz_0^2) (dz_0: the nearest plane;
// s < 5 is the cut-off test of that plane), s >= 1/16 falls into bins of 1/16
// octave (the float's exponent and top four mantissa bits), and inside a bin
// the thresholds t_k ("plane k passes exactly when rho^2 < t_k") separate
// segments of constant plane count.  Each segment holds a polynomial of degree
// four in s - (bin centre).  Degree four over 1/16 octave: at most 5e-8 of G
// off the Gaussian sum for every element (1.3e-7 of its derivative); eight bins
// per octave or degree three would cost 2e-6.
constexpr int kRadBin0 = 0x3D800000 >> 19;  // bin key of s = 1/16
constexpr int kRadBins = 100;               // up to s = 5
// Per-atom table (floats): header {dz_0^2 as the cut-off rounds it, at the
// exact height, first bin (int), planes n (int)}; thresholds ascending, +inf
// padded; exact-height dz_k^2 ascending; rows k = 0..19 of
// wsub sum_{k' <= k} w_j exp(-alpha_j (dzv_k'^2 - dzv_0^2)); per bin -1 .. 100
// the next three thresholds and the first segment (int, + kRadMore when the
// pixel needs more than these: more than three thresholds, or bin -1, the
// clamp region); per segment (bin - first bin + thresholds passed, below
// kRadSegs; segment kRadSegs is zero, for bins -1 and 100, out of reach) c_4,
// then c_0..c_3.
constexpr int kRadSegs = 120, kRadMore = 1024;
constexpr int kTabHead = 0, kTabAsc = 4, kTabQV = 28, kTabT = 48, kTabBin = 288,
              kTabC4 = kTabBin + 4 * (kRadBins + 2), kTabSeg = kTabC4 + kRadSegs + 4,
              kTabStride = kTabSeg + 4 * (kRadSegs + 4);

// The separable kernels' launch: up to kSepGroup consecutive slices and nb
// instances at once (tables: blockIdx.y = instance, blockIdx.z = slice; pixels:
// blockIdx.z = slice * nb + instance), the slices' planes and z-bin windows in
// parameter space, s_tab and s_V the strides of the tables and the output
// between slices.
struct SlicePlanes {
  float zsub[20], zsub_lo[20];
  int kt, kb;
};
constexpr int kSepGroup = 16;
struct SepArgs {
  PotArgs p;
  int ns, nb;
  int rows;  // atoms of the fullest window (bounds the table launch)
  float zero;  // 0, unknown to the compiler (mul2_rn)
  long long s_tab, s_V;
  SlicePlanes pl[kSepGroup];
  void set_slice(int i, const PotArgs& a) {
    for (int m = 0; m < 20; ++m) {
      pl[i].zsub[m] = a.zsub[m];
      pl[i].zsub_lo[m] = a.zsub_lo[m];
    }
    pl[i].kt = a.kt;
    pl[i].kb = a.kb;
  }
};
// One slice, one instance.
inline SepArgs sep_args(const PotArgs& a, int rows) {
  SepArgs s{};
  s.p = a;
  s.rows = rows;
  s.ns = s.nb = 1;
  s.set_slice(0, a);
  return s;
}


// tile: the per-sub-plane conventional kernel's tile shape (0: 32 x 8, 1:
// 16 x 16, 2: 64 x 4 pixels; other kinds take 32 x 8).
cudaError_t launch_potential(const PotArgs& a, int kind, cudaStream_t s, int tile = 0);
int potential_tiles();
int potential_tiles_separable();
// The separable conventional kernel's two launches: the per-atom tables of the
// slices into a.p.tab (derivative: dG/d(rho^2) for the position adjoint), then
// the potentials from them.  tile: 0..3 = 16 x 16,
// 16 x 32, 32 x 16, 32 x 32 pixels (two, four, four and eight per thread), -1 =
// by grid and pixel size.
cudaError_t launch_atom_tables(const SepArgs& a, cudaStream_t s, bool derivative = false);
cudaError_t launch_potential_from_tables(const SepArgs& a, cudaStream_t s, int tile);

// Adjoint of the conventional potential of one slice with respect to atom x, y:
// dxy[2 perm[l] + {0,1}] += dL/d{x,y} of sorted atoms l in [a0, a1) (the CSR
// range of the slice's z-window), G = dL/dV of the slice [ny][nx].
// separable: through the derivative tables of the slice's atoms in a.tab (a0
// must be the first atom of the slice's z-window, as there).
cudaError_t launch_potential_adjoint(const PotArgs& a, const float* G, const int* perm, int a0, int a1, double* dxy,
                                     cudaStream_t s, bool separable = false);

}  // namespace ms
