// Host-callable launchers of the CCD kernels (implemented in kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

#include "common.cuh"
#include "devlayout.hpp"

namespace ccx {

// ---- grouped GEMM (FP64 / complex FP64) ------------------------------------
// C(m,n) = [C0 or 0] + alpha sum_s sum_k A_s(m,k) B_s(k,n), element strides per operand.
template <typename S>
struct GemmSeg {
  const S *A, *B;
  int64_t sAm, sAk, sBk, sBn;
  int K;
};
template <typename S>
struct GemmProb {
  GemmSeg<S> seg[2];
  int nseg;
  int M, N;
  double alpha;
  S *C;
  const S *C0;  // null: zero
  int64_t sCm, sCn;
};
// The work of one warp: nm row tiles from m0 on, columns n0 .. n0 + nj - 1 (nj <= kGemmCols).
struct GemmTile {
  int prob, m0, n0;
  int16_t nj, nm;
};
constexpr int kGemmCols = 8;
// two warp tiles: 8 rows with K over 4 lanes each, 4 rows with K over 8 lanes each
enum GemmShape { kShape8 = 0, kShape4 = 1 };
inline int gemm_rows(int shape) { return shape == kShape8 ? 8 : 4; }

// tiles of shape 0 first (n8 of them), then n4 of shape 1
template <typename S>
void launch_gemm(const GemmProb<S> *probs, const GemmTile *tiles, int n8, int n4, cudaStream_t st);

// ---- potentials -----------------------------------------------------------
struct DevPotential {
  int kind;            // 0 Minnesota, 1 chiral-like
  int f32_literals;
  double lec[9];       // CS, CT, C1..C7 (MeV units)
  const double *lat;   // element tables of a lattice (launch_lattice_tables), or null
};
// doubles of the element tables of a potential kind on a lattice (O.nq2 entries each)
int lattice_table_doubles(const DevOrbits &O, int kind);
// fills them; every element is then evaluated from its orbitals' integers and the tables
void launch_lattice_tables(const DevOrbits &O, const DevPotential &pot, double *lat, cudaStream_t st);

// ---- residual pieces --------------------------------------------------------
template <typename S> void launch_gather_tph(const DevLayout &L, const S *T, S *Tph, cudaStream_t st);
// where each T_ph entry comes from: +/-(packed T' index + 1), 0 for a zero entry
void launch_tph_map(const DevLayout &L, int32_t *map, cudaStream_t st);
template <typename S> void launch_i7(const DevLayout &L, const S *X, const S *fdiag, const S *f7, S *d2ij, S *i7off, cudaStream_t st);
template <typename S> void launch_i9(const DevLayout &L, int64_t n, const S *Vhh, const S *X, S *I9, cudaStream_t st);
// I7 without X: the X entries it reads as 2 A^2 column dots of V_hhpp' and T' into xd
// (2 A^2 scalars), then summed as launch_i7 does
template <typename S>
void launch_i7_direct(const DevLayout &L, const S *V, const S *T, S *xd, const S *fdiag, const S *f7, S *d2ij, S *i7off,
                      cudaStream_t st);
// I9 = Vhh + (Xb + dX), n entries
template <typename S> void launch_i9b(int64_t n, const S *Vhh, const S *Xb, const S *dX, S *I9, cudaStream_t st);
// I6 in two passes; rowtile: (channel, first packed pp row) per block of kI6Rows rows;
// D: 3 values per packed row, at 3 * (t_off[ch] + row)
constexpr int kI6Rows = 128;
constexpr int kI6Parts = 4;  // threads per row: interleaved slices of the hole-pair sum
template <typename S> void launch_i6(const DevLayout &L, const int2 *rowtile, int nrowtile, S *D, const S *T, const S *Vhp,
                                     const S *fdiag, const S *f6, S *d2ab, S *i6off, cudaStream_t st);
// R' initialisation; omap / rmap (int4 per packed amplitude) from launch_rinit_maps.
// The ring term gathered from Rph is stored per amplitude into ring_out when given, and
// ring_base (per amplitude) is added to it when given: a ring split as R_ph,b + dR_ph.
// add: R' += the terms (R' holds the ladders already) instead of R' = the terms.
void launch_rinit_maps(const DevLayout &L, int4 *omap, int4 *rmap, cudaStream_t st);
template <typename S>
void launch_rinit(const DevLayout &L, const int4 *omap, const int4 *rmap, const S *T, const S *Vhp, const S *Rph,
                  const S *i6off, const S *i7off, const S *ring_base, S *ring_out, bool add, S *R, cudaStream_t st);

// ---- update / energy / norms (per-block partial sums, then a fixed-order finish) --
// mode 0: reference update T <- 0.75 T + 0.25 R/D, history column written
// mode 1: Jacobi T_jac = R/D into hist_t, step into hist_e, T untouched
// mode 2: energy only (no update); mode 3: residual norm + energy, no update
// the DIIS step vectors of the standard mode: the step is computed to FP32 accuracy and
// stored in FP32 (real engines) or as FP32 (re, im) pairs (complex engines)
struct __align__(8) cplxf {
  float re, im;
};
template <typename S> struct StepOf;
template <> struct StepOf<double> { using type = float; };
template <> struct StepOf<cplx> { using type = cplxf; };
template <typename S>
void launch_update(const DevLayout &L, int mode, S *T, const S *R, const S *Vhp, const S *d2ij, const S *d2ab,
                   S *hist_t, typename StepOf<S>::type *hist_e, double *partial, double *out4, cudaStream_t st);
// dot products: out[j] = sum_x w(a[x]) * b_j[x] for j < nb; conj on a when conj_a
template <typename S>
void launch_dots(int64_t n, const S *a, const S *const *bs, int nb, int conj_a, double *partial, double *out, cudaStream_t st);
// mode-1 update and the Gram row of its step in one pass:
// out[0] = E (re), out[1] = E (im, 0 for real engines), out[2] = |R - D T|^2, out[3] = *err (0 when err is null),
// out[4 + j] = Re(conj(step) . es[j]) for j < nb (1 <= nb <= 16); es[self] is hist_e, the step
// this pass writes.  partial holds 20 doubles for each of up to 760 blocks.
template <typename S>
void launch_update_std(const DevLayout &L, const S *T, const S *R, const S *Vhp, const S *d2ij, const S *d2ab, S *hist_t,
                       typename StepOf<S>::type *hist_e, const typename StepOf<S>::type *const *es, int nb, int self,
                       const int *err, double *partial, double *out, cudaStream_t st);
// reference DIIS Gram matrix of differences of nstep history columns (no conjugation)
template <typename S>
void launch_diis_gram(int64_t n, const S *const *cols, int nstep, double *partial, double *out, cudaStream_t st);
// y = sum_i c_i x_i
template <typename S>
void launch_combine(int64_t n, const S *const *xs, const double *coef /* host, 2 per term */, int m, S *y, cudaStream_t st);

// ---- interaction -----------------------------------------------------------
template <typename S>
void launch_pack_vblock(const DevLayout &L, int kind, int ch, int n_rows, const double *stage, S *dst, int *flag, cudaStream_t st);
// The same packing of many blocks of one kind in one launch, read straight from host
// memory the device can address (pinned and mapped): reads follow each block's
// column-major order (consecutive rows), through a shared-memory transpose where the packed
// layout is row-major (kind 3).  first: units of work (pack_units) in the jobs before this
// one; a channel occurs once in a list.  jobs null: the one job given by value (a list on the
// device costs a copy and a wait, 5 of the 24 us of a call with one block).
struct PackJob {
  const double *src;
  int ch, n_rows;
  int rows, cols;  // packed extents (kind 3: H, P; 6: P, P; 1: H, H)
  int first;
};
int pack_units(int kind, int rows, int cols);
template <typename S>
void launch_pack_jobs(const DevLayout &L, int kind, const PackJob *jobs, const PackJob &one, int njobs, int units, S *dst,
                      int *flag, cudaStream_t st);
// Copies of many blocks in one launch (n doubles from src to dst per job); src may be
// mapped host memory.
struct CopyJob {
  const double *src;
  double *dst;
  int64_t n;
};
void launch_copy_jobs(const CopyJob *jobs, int njobs, cudaStream_t st);
template <typename S>
void launch_build_w(const DevLayout &L, const int2 *hp4_slot, const int64_t *v4_off, const int *n4, const double *v4,
                    S *W, int *flag, cudaStream_t st);
template <typename S> void launch_build_vph(const DevLayout &L, const S *Vhp, S *Vph, cudaStream_t st);
template <typename S>
// pairf: npp + nhh + A (ns - A) doubles of scratch for the per-pair factors of the
// chiral-like kind (complex engines; null: every element evaluated in full)
void launch_generate(const DevLayout &L, const DevOrbits &O, const DevPotential &pot, S *Vhp, S *Vpp, S *Vhh, S *W,
                     S *fdiag, S *f6, S *f7, double *e0, double *pairf, int npp, int nhh, cudaStream_t st);
// ordered block of <row|V|col> (or <col|V|row> when swap) into interleaved doubles
template <typename S>
void launch_gen_ordered(const DevOrbits &O, const DevPotential &pot, const int2 *rows, const int2 *cols, int nr, int nc,
                        int swap, double *out, cudaStream_t st);
// packed V' -> ordered reference block (kind 3 V_hhpp, 6 V_pppp, 1 V_hhhh of hhpp channel ch)
template <typename S>
void launch_unpack_vblock(const DevLayout &L, int kind, int ch, int n_rows, int n_cols, const int *row_sgn,
                          const int *col_sgn, const S *src, double *out, cudaStream_t st);
double measure_fp64_peak(int device);
// y += x (n elements)
template <typename S> void launch_axpy(int64_t n, const S *x, S *y, cudaStream_t st);
template <typename S> void launch_mp2(const DevLayout &L, const S *Vhp, const S *fdiag, S *T, cudaStream_t st);
template <typename S> void launch_pack_t(const DevLayout &L, int ch, int n_pp, const double *stage, S *T, int *flag, cudaStream_t st);
// the packed amplitudes of channels [c0, c1) into their ordered blocks, one after the other
// from out (ntiles: their tiles); vec: out is 16-byte aligned
template <typename S>
void launch_unpack_t(const DevLayout &L, const DevOrdered &O, int c0, int c1, int ntiles, bool vec, const S *T, double *out,
                     cudaStream_t st);

}  // namespace ccx
