// Device image of the layout: plain structs of device pointers passed to kernels.
#pragma once

#include <cstdint>
#include <vector_types.h>

namespace ccx {

// Packed (a<b, i<j) hhpp channel tables and the particle-hole ring tables.
struct DevLayout {
  int ns, A, NP;  // states, holes, particles
  int nch;        // hhpp channels
  const int *P, *H;             // packed sizes per channel
  const int64_t *t_off;         // T/R block offsets (P*H, column-major, pp fastest)
  const int64_t *vpp_off;       // V_pppp' offsets (P*P, row ab' major: [ab'*P + cd'])
  const int64_t *hh2_off;       // X / I9 / V_hhhh' offsets (H*H column-major)
  const int *pp_off, *hh_off;   // offsets into the packed pair arrays
  const int2 *pp_orb, *hh_orb;  // packed pair orbitals
  const int *pp_row, *hh_row;   // packed pair -> ordered row of the reference block
  const int2 *pp_slot;          // [(a-A)*NP + (b-A)] -> (channel, signed packed index)
  const int2 *hh_slot;          // [i*A + j]          -> (channel, signed packed index)
  const int *partner;           // [ns] other-spin orbital with the same n and tz, or -1
  // ring (phhp) channels
  int nph;
  const int *n_ph, *n_hp;
  const int64_t *tph_off;       // T_ph / R_ph offsets (n_ph*n_hp column-major)
  const int64_t *i4_off;        // I4 / W offsets (n_hp*n_hp)
  const int64_t *vph_off;       // V_ph offsets (n_hp*n_ph)
  const int *ph_off, *hp_off;
  const int2 *ph_orb;           // (a particle, i hole) rows
  const int2 *hp_orb;           // (j hole, b particle) columns
  const int2 *ph_slot;          // [(a-A)*A + i] -> (channel, row)
  const int2 *hp_slot;          // [j*NP + (b-A)] -> (channel, column)
  // element tiles: {channel, start}
  const int2 *ttile;
  int nttile;
  const int2 *phtile;
  int nphtile;
  // 32 x 32 tiles on and above the diagonal of each V_pppp' block: vt_off[c] of them in
  // the channels before c, column by column within a channel
  const int *vt_off;
  int nvtile;
};

constexpr int kTileElems = 1024;

// The caller's ordered T2 blocks (n_pp x n_hh, one after the other from amp_off), for
// unpacking: signed packed index + 1 of every ordered pair (0 for a = b), and tiles of
// kTileElems ordered elements, tile_off[c] of them in the channels before c.
struct DevOrdered {
  const int *n_pp, *n_hh;
  const int64_t *amp_off, *pp_sgn_off, *hh_sgn_off;
  const int *pp_sgn, *hh_sgn;
  const int *tile_off;
};

// Orbital data used by the device potentials.
struct DevOrbits {
  int ns;
  const int *nx, *ny, *nz, *sz, *tz;
  const double *kx, *ky, *kz, *e;
  double volume;
  // Momenta on one cubic lattice (k_p - k_q = step (n_p - n_q) to rounding): per orbital
  // (nx, ny, nz) in the signed low bytes, and spin up (bit 0) and isospin +1 (bit 1); null
  // for any other set of momenta.  nq2: one more than the largest |n_p - n_q|^2.
  const int2 *lat;
  double step;
  int nq2;
};

}  // namespace ccx
