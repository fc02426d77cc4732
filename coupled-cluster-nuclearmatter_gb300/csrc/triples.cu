// Perturbative triples (T): pert_triples2 (ccm_triples.f90:528-735) with its two
// helpers three_body_oneparticle_1 (:174-232) and three_body_onehole_1 (:238-294),
// over the triples of setup_t3_channel_structures (ccm_t3full_channels.f90:4-284): all
// i < j < k and a < b < c of equal momentum and isospin.  The FP64 sum of conj(W) W / D is
// reduced per block and finished in a fixed order.
#include <cuda_runtime.h>

#include <algorithm>
#include <array>
#include <cmath>
#include <stdexcept>
#include <type_traits>
#include <utility>
#include <vector>

#include "common.cuh"
#include "engine.hpp"
#include "potential.cuh"
#include "triples.hpp"

namespace ccx {

namespace {

void tck(cudaError_t e, const char *what) {
  if (e != cudaSuccess) throw EngineError(2, std::string(what) + ": " + cudaGetErrorString(e));
}

constexpr int kQBias = 64;

struct TriplesDev {
  int A, NP;
  // Momenta of the lattice, split into those with hole states and those with particle
  // states: their packed integers (nx, ny, nz biased by kQBias, one per byte) and the orbitals
  // of their states, state 2 t + s (G = 4: isospin and spin) or s (G = 2: one isospin), -1
  // where a state is absent or on the other side of the Fermi level.
  int nhm, npm;
  const unsigned *hmom, *pmom;
  const int4 *horb, *porb;
  unsigned qlo, qspan;                 // per byte: smallest allowed value, allowed span
  int ey, ez;
  const int2 *mom_of;                  // momentum -> (hole momentum, particle momentum) or -1
  int nbra;
  const int3 *bra;                     // hole momenta of every block of hole triples
  // Where the blocks hold an element: the first entry of a column and the row in it.  Momentum
  // and isospin put the column's pair and the row's pair of a term in the same channel.  For T'
  // both are signed and one more than the index (0: no such pair).
  const int64_t *t_col;                // T'(., ij) of hole pair (i, j)
  const int *t_row;                    // T'(ab, .) of particle pair (a, b)
  const int64_t *v5_col;               // V_hppp(., cb) of particle pair (c, b), -1: none
  const int *v5_row;                   // V_hppp(kd, .) of (k, d), -1: none
  const int64_t *v2_col;               // V_hhhp(., lc) of (l, c), -1: none
  const int *v2_row;                   // V_hhhp(jk, .) of hole pair (j, k), -1: none
};

// Bytewise q_i + q_j - q_a of packed momenta: the momentum of the orbital that closes a pair
// (each byte stays in 0 .. 255 for |n| <= 21 per axis).
__device__ __forceinline__ unsigned qsum(unsigned qi, unsigned qj, unsigned qa) { return __vsub4(__vadd4(qi, qj), qa); }

// (hole momentum, particle momentum) of a packed momentum, -1 where there is none
__device__ __forceinline__ int2 t_momentum(const TriplesDev &D, unsigned q) {
  const unsigned d = __vsub4(q, D.qlo);  // per byte: n + nk
  if (__vcmpgtu4(d, D.qspan)) return make_int2(-1, -1);
  return D.mom_of[((d & 0xffu) * D.ey + ((d >> 8) & 0xffu)) * D.ez + ((d >> 16) & 0xffu)];
}

// The 18 gather-contractions of a pair run in the contraction type W: the engine's
// scalar S (FP64), or its FP32 counterpart (float, or cplxf for complex engines) on
// FP32 copies of T, V_hppp and V_hhhp.  GB300's FP64 pipe retires 2 FMA per clock per SM
// against 128 for FP32, so the FP32 form takes the contractions off the narrow pipe; the
// |W|^2 / D accumulation stays FP64 in both.
template <typename S> struct LowOf;
template <> struct LowOf<double> { using type = float; };
template <> struct LowOf<cplx> { using type = cplxf; };

template <typename W> __device__ __forceinline__ W wzero();
template <> __device__ __forceinline__ double wzero<double>() { return 0.0; }
template <> __device__ __forceinline__ float wzero<float>() { return 0.0f; }
template <> __device__ __forceinline__ cplx wzero<cplx>() { return cplx(0.0, 0.0); }
template <> __device__ __forceinline__ cplxf wzero<cplxf>() { return cplxf{0.0f, 0.0f}; }

// x with its sign flipped when s is 1: a sign-bit flip on the integer pipe
__device__ __forceinline__ double flip(double x, unsigned s) {
  return __longlong_as_double((long long)((unsigned long long)__double_as_longlong(x) ^ ((unsigned long long)s << 63)));
}
__device__ __forceinline__ float flip(float x, unsigned s) { return __int_as_float(__float_as_int(x) ^ (int)(s << 31)); }
__device__ __forceinline__ cplx flip(cplx x, unsigned s) { return cplx(flip(x.re, s), flip(x.im, s)); }
__device__ __forceinline__ cplxf flip(cplxf x, unsigned s) { return cplxf{flip(x.re, s), flip(x.im, s)}; }

__device__ __forceinline__ double madd_conj(double v, double t, double acc) { return fma(v, t, acc); }
__device__ __forceinline__ cplx madd_conj(cplx v, cplx t, cplx acc) {
  return cplx(fma(v.re, t.re, fma(v.im, t.im, acc.re)), fma(v.re, t.im, fma(-v.im, t.re, acc.im)));
}
__device__ __forceinline__ float madd_conj(float v, float t, float acc) { return fmaf(v, t, acc); }
__device__ __forceinline__ cplxf madd_conj(cplxf v, cplxf t, cplxf acc) {
  return cplxf{fmaf(v.re, t.re, fmaf(v.im, t.im, acc.re)), fmaf(v.re, t.im, fmaf(-v.im, t.re, acc.im))};
}
// |W|^2 in FP64 as the engine's scalar
__device__ __forceinline__ double wnorm2(double w) { return w * w; }
__device__ __forceinline__ double wnorm2(cplx w) { return w.re * w.re + w.im * w.im; }

// Sum of |W|^2 / D, in FP64 term by term, and the denominators it needs.  With FP64 contractions the
// ratio is FP64 as well, with FP32 ones FP32 (its rounding, 6e-8 of the term, is far below the
// contractions' own), from FP64 denominators in real engines.  Complex ones, with two FP64
// differences a pair beside the two additions of the sum, take the denominators' differences from
// pairs of FP32 numbers, which hold the Fock sums to 2^-49: an FP64 operation costs 64 FP32 ones on
// this GPU (SNM 76 nmax=2 16.1 ms with FP64 differences, 11.6 so; PNM 54 nmax=2 1.97 with FP64, 2.00
// with pairs).  The sum in pairs, added to an FP64 one every 64 terms, would save another tenth of
// the complex time (10.4 ms), but holds 48 bits and turns an infinite term into a NaN.
template <typename S, typename W> struct TripleSum;
// n1 / d1 + n2 / d2 as one fraction: an FP64 division costs some ten operations of the FP64
// pipe, three multiplications and an addition are cheaper
__device__ __forceinline__ void add_fractions(double n1, double d1, double n2, double d2, double &n, double &d) {
  n = fma(n1, d2, n2 * d1);
  d = d1 * d2;
}
template <> struct TripleSum<double, double> {
  using Fock = double;
  double re = 0.0;
  static __device__ __forceinline__ Fock fock(double f) { return f; }
  // the four pairs of a thread; live: which of them count
  __device__ __forceinline__ void add(const double (&w)[4], const Fock (&h)[4], const Fock (&p)[4], const bool (&live)[4]) {
    double n[4], d[4], n2[2], d2[2], nn, dd;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      n[q] = live[q] ? wnorm2(w[q]) : 0.0;
      d[q] = live[q] ? h[q] - p[q] : 1.0;
    }
    add_fractions(n[0], d[0], n[1], d[1], n2[0], d2[0]);
    add_fractions(n[2], d[2], n[3], d[3], n2[1], d2[1]);
    add_fractions(n2[0], d2[0], n2[1], d2[1], nn, dd);
    re += nn / dd;
  }
  __device__ __forceinline__ void total(double (&v)[2]) const { v[0] = re; v[1] = 0.0; }
};
template <> struct TripleSum<cplx, cplx> {
  using Fock = cplx;
  cplx s = cplx(0.0, 0.0);
  static __device__ __forceinline__ Fock fock(cplx f) { return f; }
  __device__ __forceinline__ void add(const cplx (&w)[4], const Fock (&h)[4], const Fock (&p)[4], const bool (&live)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (live[q]) {  // |W|^2 / D = |W|^2 conj(D) / |D|^2
        const cplx d = h[q] - p[q];
        const double r = wnorm2(w[q]) / fma(d.re, d.re, d.im * d.im);
        s.re = fma(r, d.re, s.re);
        s.im = fma(-r, d.im, s.im);
      }
  }
  __device__ __forceinline__ void total(double (&v)[2]) const { v[0] = s.re; v[1] = s.im; }
};
__device__ __forceinline__ float2 two_floats(double x) {
  const float h = __double2float_rn(x);
  return make_float2(h, __double2float_rn(x - (double)h));
}
// (h - p) of two pairs, to FP32: Knuth's two-sum of the high parts, and what it leaves
__device__ __forceinline__ float two_sub(float2 h, float2 p) {
  const float s = __fsub_rn(h.x, p.x), bb = __fsub_rn(s, h.x);
  const float rest = __fsub_rn(__fsub_rn(h.x, __fsub_rn(s, bb)), __fadd_rn(p.x, bb));
  return __fadd_rn(s, __fadd_rn(rest, __fsub_rn(h.y, p.y)));
}
template <> struct TripleSum<double, float> {
  using Fock = double;
  double re = 0.0;
  static __device__ __forceinline__ Fock fock(double f) { return f; }
  __device__ __forceinline__ void add(const float (&w)[4], const Fock (&h)[4], const Fock (&p)[4], const bool (&live)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (live[q]) re += (double)((w[q] * w[q]) / (float)(h[q] - p[q]));
  }
  __device__ __forceinline__ void total(double (&v)[2]) const { v[0] = re; v[1] = 0.0; }
};
template <> struct TripleSum<cplx, cplxf> {
  using Fock = float4;
  double re = 0.0, im = 0.0;
  static __device__ __forceinline__ Fock fock(cplx f) {
    const float2 a = two_floats(f.re), b = two_floats(f.im);
    return make_float4(a.x, a.y, b.x, b.y);
  }
  __device__ __forceinline__ void add(const cplxf (&w)[4], const Fock (&h)[4], const Fock (&p)[4], const bool (&live)[4]) {
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (live[q]) {
        // |W|^2, written out as rounded (lattices of a few thousand pairs show the other order of
        // the two squares at 1e-9 of the sum)
        const float n = fmaf(w[q].im, w[q].im, __fmul_rn(w[q].re, w[q].re));
        const float dr = two_sub(make_float2(h[q].x, h[q].y), make_float2(p[q].x, p[q].y));
        const float di = two_sub(make_float2(h[q].z, h[q].w), make_float2(p[q].z, p[q].w));
        const float s = n / (dr * dr + di * di);  // |W|^2 / D = |W|^2 conj(D) / |D|^2
        re += (double)(s * dr);
        im += (double)(-s * di);
      }
  }
  __device__ __forceinline__ void total(double (&v)[2]) const { v[0] = re; v[1] = im; }
};

// FP32 copy of an FP64 array
__device__ __forceinline__ float to_low(double x) { return __double2float_rn(x); }
__device__ __forceinline__ cplxf to_low(cplx x) { return cplxf{__double2float_rn(x.re), __double2float_rn(x.im)}; }
template <typename S>
__global__ void k_to_low(const S *__restrict__ src, int64_t n, typename LowOf<S>::type *__restrict__ dst) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    dst[e] = to_low(src[e]);
}

template <int NV>
__device__ void block_sum(double (&v)[NV], double *partial) {
  __shared__ double red[NV][32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5, nw = blockDim.x >> 5;
  for (int k = 0; k < NV; ++k) {
    double x = warp_sum(v[k]);
    if (lane == 0) red[k][wid] = x;
  }
  __syncthreads();
  if (wid == 0)
    for (int k = 0; k < NV; ++k) {
      double x = lane < nw ? red[k][lane] : 0.0;
      x = warp_sum(x);
      if (lane == 0) partial[(int64_t)blockIdx.x * NV + k] = x;
    }
}

// (permutation of the particles, permutation of the holes) of the nine terms of each
// kind, 2 + 2 bits per term: (0,0) (1,0) (2,0) (0,1) (0,2) (2,2) (2,1) (1,2) (1,1)
constexpr unsigned long long kTermOrder = 0x596A84210ull;

// A momentum block: every i j k on three hole momenta with every a b c on three particle
// momenta of the same total.  W of its pairs is a sum of 18 products, each over the two spins of
// the one orbital that momentum and isospin leave:
//   particle terms  T(A d, I J) conj(<C B|V|K d>),  hole terms  T(A B, I l) conj(<J K|V|l C>)
// with (A, B, C) and (I, J, K) permutations of the triples.  A factor depends on three of the six
// states only, so a block's 1280 pairs (20 isospin patterns x 64 spins; 64 pairs of one
// isospin) read 36 tables of 64 (8) entries: they are gathered once into shared memory, and each
// thread then forms four pairs (both spins of k and c), which share half of their reads.
// Gathering the factors pair by pair through slot tables, 36 gathers of some ten dependent
// loads each, kept the integer pipe and L1 busy and the FP32 pipe idle.  ms before and now, FP32
// / FP64 contractions: PNM 14 nmax=2 0.33 to 0.22 / 0.37 to 0.35, PNM 54 nmax=2 8.4 to 2.0 / 9.0
// to 4.2, SNM 28 nmax=2 6.8 to 1.6 / 12.9 to 9.8, SNM 76 nmax=2 (6.3e8 pairs) 89.8 to 11.6 /
// 170 to 82.1.  FP32 contractions of complex engines issue in 45% of the cycles beside an FP64 pipe
// that is 47% busy with the sum (FMA pipe 19%, shared memory 24%); the rest is the latency of the
// gathers and barriers.  FP64 contractions are bound by their pipe.
template <typename W> struct alignas(2 * sizeof(W)) SpinPair {
  W v[2];  // the two spins of the closing orbital
};
template <typename W, int G> struct TripleShape {
  // ket blocks a thread block holds at once and the (a, b, i, j) of one (with both isospins
  // times the 20 isospin patterns)
  static constexpr int kKets = G == 4 ? 1 : (sizeof(W) == 16 ? 4 : 8);
  static constexpr int kItems = G == 4 ? 320 : 16;
  // Two sets of tables where a ket fills the block (both isospins: the gathers of one ket run
  // beside the pairs of the other, a tenth of SNM 76 nmax=2), one set and
  // twice the resident blocks otherwise (PNM 54 nmax=2 2.0 ms against 2.5).  Complex FP64 with
  // both isospins takes one set and two rounds of half as many threads, so that three blocks fit.
  static constexpr int kBuffers = sizeof(W) == 16 || G == 2 ? 1 : 2;
  static constexpr int kRounds = G == 4 && sizeof(W) == 16 ? 2 : 1;
  static constexpr int kThreads = kKets * kItems / kRounds;
  static constexpr int kCube = G * G * G;
  // blocks an SM holds (shared memory allows no more): the registers are cut for them
  static constexpr int kMinBlocks = G == 4 ? (sizeof(W) == 16 ? 3 : 2) : sizeof(W) == 4 ? 7 : 5;
  static constexpr size_t table_bytes() { return (size_t)kBuffers * kKets * 36 * kCube * sizeof(SpinPair<W>); }
};
// isospin patterns (a b c i j k, one bit each) of equal sums
__constant__ const unsigned char kIso[20] = {0x00, 0x09, 0x0a, 0x0c, 0x11, 0x12, 0x14, 0x21, 0x22, 0x24,
                                             0x1b, 0x1d, 0x1e, 0x2b, 0x2d, 0x2e, 0x33, 0x35, 0x36, 0x3f};

template <typename S, typename W, int G>
__global__ void __launch_bounds__(TripleShape<W, G>::kThreads, TripleShape<W, G>::kMinBlocks)
    k_triples(TriplesDev D, const W *__restrict__ T, const W *__restrict__ V5, const W *__restrict__ V2,
              const S *__restrict__ fd, int seg, int nseg, int stride, double *partial) {
  using Sh = TripleShape<W, G>;
  using Sum = TripleSum<S, W>;
  using Fock = typename Sum::Fock;
  constexpr int NT = Sh::kThreads, KB = Sh::kKets, CU = Sh::kCube, CAP = 2 * NT;
  constexpr bool kSort = std::is_same<S, W>::value, kOne = kSort && G == 4;
  extern __shared__ __align__(32) unsigned char tsm[];
  SpinPair<W> *tab = reinterpret_cast<SpinPair<W> *>(tsm);  // [buffer][ket][table U, Q, X, Y][term][states]
  __shared__ Fock eh[CU], ep[3][KB][CU];
  __shared__ int oh[3][4], op[3][KB][3][4];    // orbitals of the momenta's states
  // closing momentum of each term, particle (terms 0 .. 8) or hole (9 .. 17), -1 where there is
  // none (most hole terms, and the particle terms that leave the lattice: nothing of such a term
  // is gathered or added); and the terms that have one, as ket * 32 + term
  __shared__ int close[4][KB][18];
  __shared__ unsigned short live[3][KB * 18];
  __shared__ int nlive[3];
  __shared__ int2 kets[CAP];                   // (p1 | p2 << 16, p3)
  __shared__ int nkets_warp[NT / 32 + 1];
  __shared__ unsigned short items[Sh::kItems];  // the (a, b, i, j) whose i, j exist and are in order
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  Sum sum;
  // this thread's ket of a step and its states of it: bit s of spin (and 2 t of isospin)
  struct Item {
    int kb, iso, sa, sb, si, sj;
    bool bc;     // a state of c in order behind b's
    int cs, ks;  // the one spin of c and k of a single pair
  };
  Item mine[Sh::kRounds];
  auto state = [](int iso, int pos, int s) { return G == 4 ? ((iso >> (5 - pos)) & 1) * 2 + s : s; };
  int last_bra = -1, nket = 0;
  bool one = false;
  int3 hm = make_int3(0, 0, 0);
  unsigned qn = 0;
  // closing momenta of the kets of step st
  auto closing = [&](int st) {
    const int k0 = st * KB, n = min(KB, nket - k0) * 18;
    for (int x = tid; x < n; x += NT) {
      const int b = x / 18, u = x - b * 18, t = u < 9 ? u : u - 9, pp = t / 3, hp = t - 3 * pp;
      const int2 kt = kets[k0 + b];
      const unsigned m1 = D.pmom[kt.x & 0xffff], m2 = D.pmom[(unsigned)kt.x >> 16], m3 = D.pmom[kt.y];
      const unsigned n1 = D.hmom[hm.x], n2 = D.hmom[hm.y], n3 = D.hmom[hm.z];
      // d = I + J - A with A the particle pp and (I, J) = (i,j), (k,j), (i,k);
      // l = J + K - C with C = c, b, a and (J, K) = (j,k), (j,i), (i,k)
      const unsigned q = u < 9 ? qsum(hp == 1 ? n3 : n1, hp == 2 ? n3 : n2, pp == 0 ? m1 : pp == 1 ? m2 : m3)
                               : qsum(hp == 2 ? n1 : n2, hp == 1 ? n1 : n3, pp == 0 ? m3 : pp == 1 ? m2 : m1);
      const int2 c = t_momentum(D, q);
      close[st & 3][b][u] = u < 9 ? c.y : c.x;
    }
  };
  // live terms, orbitals and denominators of the kets of step st, into buffer m
  auto meta = [&](int st, int m) {
    const int k0 = st * KB, nk = min(KB, nket - k0);
    if (wid == 0) {
      int n = 0;
      for (int x0 = 0; x0 < nk * 18; x0 += 32) {
        const int x = x0 + lane, b = x / 18;
        const bool on = x < nk * 18 && close[st & 3][b][x - b * 18] >= 0;
        const unsigned vote = __ballot_sync(0xffffffffu, on);
        if (on) live[m][n + __popc(vote & ((1u << lane) - 1u))] = (unsigned short)(b * 32 + x - b * 18);
        n += __popc(vote);
      }
      if (lane == 0) nlive[m] = n;
    }
    for (int x = NT - 1 - tid; x < nk * 12; x += NT) {
      const int b = x / 12, y = x - b * 12;
      const int2 kt = kets[k0 + b];
      op[m][b][y >> 2][y & 3] =
          reinterpret_cast<const int *>(D.porb + (y < 4 ? kt.x & 0xffff : y < 8 ? (unsigned)kt.x >> 16 : kt.y))[y & 3];
    }
    for (int x = NT - 1 - tid; x < nk * CU; x += NT) {
      const int b = x / CU, y = x - b * CU, y0 = y / (G * G), y1 = y / G % G, y2 = y % G;
      const int2 kt = kets[k0 + b];
      const int a = reinterpret_cast<const int *>(D.porb + (kt.x & 0xffff))[y0];
      const int c = reinterpret_cast<const int *>(D.porb + ((unsigned)kt.x >> 16))[y1];
      const int e = reinterpret_cast<const int *>(D.porb + kt.y)[y2];
      ep[m][b][y] = Sum::fock(a >= 0 && c >= 0 && e >= 0 ? fd[a] + fd[c] + fd[e] : S(0.0));
    }
  };
  // The tables of the live terms of step st, entry by entry; signs of the permutations in Q, Y.
  auto build = [&](int st, int m, SpinPair<W> *to) {
    const int n = nlive[m] * CU;
    for (int x = tid; x < n; x += NT) {
      const int e = x % CU, w = live[m][x / CU], b = w >> 5, u = w & 31, t = u < 9 ? u : u - 9, pp = t / 3, hp = t - 3 * pp;
      const int s0 = e / (G * G), s1 = e / G % G, s2 = e % G;
      const int(*o)[4] = op[m][b];
      // isospin bit of the closing orbital: of (s0, s1 | s2) in Q and X, of (s1, s2 | s0) in U and Y
      const int ta = G == 4 ? (s0 >> 1) + (s1 >> 1) - (s2 >> 1) : 0, tb = G == 4 ? (s1 >> 1) + (s2 >> 1) - (s0 >> 1) : 0;
      const bool oka = ta == 0 || ta == 1, okb = tb == 0 || tb == 1;
      SpinPair<W> first, second;
#pragma unroll
      for (int s = 0; s < 2; ++s) first.v[s] = second.v[s] = wzero<W>();
      if (u < 9) {
        const int *dorb = reinterpret_cast<const int *>(D.porb + close[st & 3][b][u]);
        const int A1 = o[pp][s0], I1 = oh[hp == 1 ? 2 : 0][s1], J1 = oh[hp == 2 ? 2 : 1][s2];
        const int B1 = o[pp == 1 ? 0 : 1][s0], C1 = o[pp == 2 ? 0 : 2][s1], K1 = oh[hp == 0 ? 2 : hp == 1 ? 0 : 1][s2];
        if (okb && (A1 | I1 | J1) >= 0) {  // U: T(A d, I J), states (A, I, J)
          const int64_t c = D.t_col[I1 * D.A + J1];
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const int d = dorb[2 * tb + s];
            const int r = d >= 0 ? D.t_row[(int64_t)(A1 - D.A) * D.NP + (d - D.A)] : 0;
            if (r != 0 && c != 0) first.v[s] = flip(T[llabs(c) - 1 + (abs(r) - 1)], (unsigned)((c < 0) != (r < 0)));
          }
        }
        if (oka && (B1 | C1 | K1) >= 0) {  // Q: <C B|V|K d>, states (B, C, K)
          const int64_t c = D.v5_col[(int64_t)(C1 - D.A) * D.NP + (B1 - D.A)];
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const int d = dorb[2 * ta + s];
            const int r = d >= 0 ? D.v5_row[(int64_t)K1 * D.NP + (d - D.A)] : -1;
            if (r >= 0 && c >= 0) second.v[s] = flip(V5[c + r], (unsigned)((pp != 0) != (hp != 0)));
          }
        }
      } else {
        const int *lorb = reinterpret_cast<const int *>(D.horb + close[st & 3][b][u]);
        const int A1 = o[pp == 2 ? 2 : 0][s0], B1 = o[pp == 1 ? 2 : 1][s1], I1 = oh[hp == 0 ? 0 : hp == 1 ? 2 : 1][s2];
        const int C1 = o[2 - pp][s0], J1 = oh[hp == 2 ? 0 : 1][s1], K1 = oh[hp == 1 ? 0 : 2][s2];
        if (oka && (A1 | B1 | I1) >= 0) {  // X: T(A B, I l), states (A, B, I)
          const int r = D.t_row[(int64_t)(A1 - D.A) * D.NP + (B1 - D.A)];
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const int l = lorb[2 * ta + s];
            const int64_t c = l >= 0 ? D.t_col[I1 * D.A + l] : 0;
            if (r != 0 && c != 0) first.v[s] = flip(T[llabs(c) - 1 + (abs(r) - 1)], (unsigned)((c < 0) != (r < 0)));
          }
        }
        if (okb && (C1 | J1 | K1) >= 0) {  // Y: <J K|V|l C>, states (C, J, K)
          const int r = D.v2_row[J1 * D.A + K1];
#pragma unroll
          for (int s = 0; s < 2; ++s) {
            const int l = lorb[2 * tb + s];
            const int64_t c = l >= 0 ? D.v2_col[(int64_t)l * D.NP + (C1 - D.A)] : -1;
            if (r >= 0 && c >= 0) second.v[s] = flip(V2[c + r], (unsigned)((pp != 0) == (hp != 0)));
          }
        }
      }
      SpinPair<W> *out = to + (size_t)b * 36 * CU + (u < 9 ? t : 18 + t) * CU + e;
      out[0] = first;
      out[9 * CU] = second;
    }
  };
  // the pairs of the kets of step st
  auto pairs = [&](const Item &I, int st, int m, const SpinPair<W> *from, auto single) {
    constexpr int NS = decltype(single)::value ? 1 : 2;  // spins of c and of k
    const int kb = I.kb, sa = I.sa, sb = I.sb, si = I.si, sj = I.sj;
    if (kb >= KB || st * KB + kb >= nket) return;
    const SpinPair<W> *tb = from + (size_t)kb * 36 * CU;
    const int2 kt = kets[st * KB + kb];
    const int pa = kt.x & 0xffff, pb = (int)((unsigned)kt.x >> 16), pc = kt.y;
    // each triple once: states in order where momenta coincide, and all of them present
    const int(*o)[4] = op[m][kb];
    if ((pa == pb && sa >= sb) || (kSort && pb == pc && !I.bc) || (o[0][sa] | o[1][sb]) < 0) return;
    W w[NS][NS];
#pragma unroll
    for (int cs = 0; cs < NS; ++cs)
#pragma unroll
      for (int ks = 0; ks < NS; ++ks) w[cs][ks] = wzero<W>();
    auto cube = [](int p, int q, int r) { return (p * G + q) * G + r; };
#pragma unroll
    for (int half = 0; half < 2; ++half)  // the terms in pert_triples2's order
#pragma unroll
      for (int t = 0; t < 9; ++t) {
        const int pp = (int)(kTermOrder >> (4 * t)) & 3, hp = (int)(kTermOrder >> (4 * t + 2)) & 3;
        if (close[st & 3][kb][9 * half + 3 * pp + hp] < 0) continue;
        const SpinPair<W> *first = tb + (18 * half + 3 * pp + hp) * CU, *second = first + 9 * CU;
#pragma unroll
        for (int cs = 0; cs < NS; ++cs)
#pragma unroll
          for (int ks = 0; ks < NS; ++ks) {
            const int sc = state(I.iso, 2, NS == 1 ? I.cs : cs), sk = state(I.iso, 5, NS == 1 ? I.ks : ks);
            int f, g;
            if (half == 0) {
              f = cube(pp == 0 ? sa : pp == 1 ? sb : sc, hp == 1 ? sk : si, hp == 2 ? sk : sj);
              g = cube(pp == 1 ? sa : sb, pp == 2 ? sa : sc, hp == 0 ? sk : hp == 1 ? si : sj);
            } else {
              f = cube(pp == 2 ? sc : sa, pp == 1 ? sc : sb, hp == 0 ? si : hp == 1 ? sk : sj);
              g = cube(pp == 0 ? sc : pp == 1 ? sb : sa, hp == 2 ? si : sj, hp == 1 ? si : sk);
            }
            const SpinPair<W> x = first[f], y = second[g];
            w[cs][ks] = madd_conj(y.v[0], x.v[0], w[cs][ks]);
            w[cs][ks] = madd_conj(y.v[1], x.v[1], w[cs][ks]);
          }
      }
    W wv[4];
    Fock hv[4], pv[4];
    bool on[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      on[q] = q < NS * NS;
      wv[q] = wzero<W>();
      hv[q] = pv[q] = Fock{};
      if (!on[q]) continue;
      const int sc = state(I.iso, 2, NS == 1 ? I.cs : q >> 1), sk = state(I.iso, 5, NS == 1 ? I.ks : q & 1);
      wv[q] = w[NS == 1 ? 0 : q >> 1][NS == 1 ? 0 : q & 1];
      hv[q] = eh[cube(si, sj, sk)];
      pv[q] = ep[m][kb][cube(sa, sb, sc)];
      on[q] = (o[2][sc] | oh[2][sk]) >= 0 && (pb != pc || sb < sc) && (hm.y != hm.z || sj < sk);
    }
    sum.add(wv, hv, pv, on);
  };
  const int64_t nitems = (int64_t)D.nbra * nseg;
  const int tests = D.npm * D.npm;
  for (int64_t wave = 0; wave * gridDim.x < nitems; ++wave) {
    // the order of the blocks turns round from one wave of items to the next: early segments
    // hold more kets than later ones
    const int64_t it = wave * gridDim.x + ((wave & 1) ? gridDim.x - 1 - blockIdx.x : blockIdx.x);
    if (it >= nitems) continue;
    const int sg = (int)(it / D.nbra), bra = (int)(it - (int64_t)sg * D.nbra);
    if (bra != last_bra) {
      last_bra = bra;
      hm = D.bra[bra];
      qn = __vadd4(__vadd4(__vsub4(D.hmom[hm.x], kQBias * 0x010101u), __vsub4(D.hmom[hm.y], kQBias * 0x010101u)),
                   D.hmom[hm.z]);  // total + bias
      if (tid < 12) oh[tid >> 2][tid & 3] = reinterpret_cast<const int *>(D.horb + (tid < 4 ? hm.x : tid < 8 ? hm.y : hm.z))[tid & 3];
      __syncthreads();
      for (int x = tid; x < CU; x += NT) {
        const int i = oh[0][x / (G * G)], j = oh[1][x / G % G], k = oh[2][x % G];
        eh[x] = Sum::fock(i >= 0 && j >= 0 && k >= 0 ? fd[i] + fd[j] + fd[k] : S(0.0));
      }
      // The states (a, b, i, j) of this block whose i and j exist and come in order, with a k behind
      // them, spread over the threads without gaps.  FP64 contractions, which are bound by their pipe,
      // take those first that kets of coinciding momenta need (a < b, and a c behind b), so that
      // whole warps have nothing to do there; and single pairs where all of i, j, k share a momentum
      // (96 pairs, in 36 of the 320 states).  FP32 ones keep neighbouring states in neighbouring
      // lanes, which the shared-memory reads want.
      one = kOne && hm.x == hm.z;
      if (wid == 0) {
        int n = 0;
        for (int y = 0; y < (kSort ? 4 : 1) * (one ? 4 : 1); ++y)
          for (int x0 = 0; x0 < Sh::kItems; x0 += 32) {
            const int x = x0 + lane, order = one ? y >> 2 : y, cs = one ? y >> 1 & 1 : 1;
            bool ok = false;
            if (x < Sh::kItems) {
              const int iso = G == 4 ? kIso[x >> 4] : 0;
              const int a = state(iso, 0, (x >> 3) & 1), b = state(iso, 1, (x >> 2) & 1);
              const int i = state(iso, 3, (x >> 1) & 1), j = state(iso, 4, x & 1);
              bool k = false;
              for (int s = one ? y & 1 : 0; s < (one ? (y & 1) + 1 : 2); ++s)
                k |= oh[2][state(iso, 5, s)] >= 0 && (hm.y != hm.z || j < state(iso, 5, s));
              ok = (oh[0][i] | oh[1][j]) >= 0 && (hm.x != hm.y || i < j) && k &&
                   (!kSort || (a < b ? 0 : 2) + (b < state(iso, 2, cs) ? 0 : 1) == order);
            }
            const unsigned vote = __ballot_sync(0xffffffffu, ok);
            if (ok) items[n + __popc(vote & ((1u << lane) - 1u))] = (unsigned short)(x | (y & 3) << 9);
            n += __popc(vote);
          }
        if (lane == 0) nkets_warp[NT / 32] = n;
      }
      __syncthreads();
      const int nitem = nkets_warp[NT / 32];
#pragma unroll
      for (int r = 0; r < Sh::kRounds; ++r) {
        const int y = tid + r * NT, z = nitem > 0 ? items[y % nitem] : 0, x = z & 511, iso = G == 4 ? kIso[x >> 4] : 0;
        mine[r] = Item{nitem > 0 ? y / nitem : KB, iso, state(iso, 0, (x >> 3) & 1), state(iso, 1, (x >> 2) & 1),
                       state(iso, 3, (x >> 1) & 1), state(iso, 4, x & 1), false, z >> 10 & 1, z >> 9 & 1};
        mine[r].bc = mine[r].sb < state(iso, 2, one ? mine[r].cs : 1);
      }
    }
    // test x of the segment: (p1, p2) number first + x * stride
    const int first = stride == 1 ? sg * seg : sg;
    const int t1 = min(seg, (tests - first + stride - 1) / stride);
    int t0 = 0;
    while (t0 < t1) {
      // the ket momenta p1 <= p2 <= p3 of this total, in the order of (p1, p2)
      nket = 0;
      for (; t0 < t1 && nket + NT <= CAP; t0 += NT) {
        const int x = t0 + tid, t = x < t1 ? first + x * stride : 0, p1 = t / D.npm, p2 = t - p1 * D.npm;
        int p3 = -1;
        if (x < t1 && p2 >= p1)
          p3 = t_momentum(D, __vsub4(__vadd4(__vsub4(qn, D.pmom[p1]), 2 * kQBias * 0x010101u), D.pmom[p2])).y;
        const bool live = p3 >= 0 && p3 >= p2;
        const unsigned vote = __ballot_sync(0xffffffffu, live);
        if (lane == 0) nkets_warp[wid] = __popc(vote);
        __syncthreads();
        int before = nket, all = 0;
        for (int w = 0; w < NT / 32; ++w) {
          if (w < wid) before += nkets_warp[w];
          all += nkets_warp[w];
        }
        // (FP64: two that coincide first, as in the order of the bras)
        const bool turn = kSort && p2 == p3;
        if (live)
          kets[before + __popc(vote & ((1u << lane) - 1u))] =
              turn ? make_int2(p2 | p3 << 16, p1) : make_int2(p1 | p2 << 16, p3);
        nket += all;
        __syncthreads();
      }
      // Four stages, one barrier a step (two with one set of tables): closing momenta of the
      // kets three steps on, what else belongs to those two steps on, the tables one step on,
      // the pairs of this step.
      const int steps = (nket + KB - 1) / KB;
      for (int q = 0; q < min(3, steps); ++q) closing(q);
      __syncthreads();
      for (int q = 0; q < min(2, steps); ++q) meta(q, q);
      __syncthreads();
      if (steps > 0) build(0, 0, tab);
      __syncthreads();
      for (int st = 0; st < steps; ++st) {
        if (st + 3 < steps) closing(st + 3);
        if (st + 2 < steps) meta(st + 2, (st + 2) % 3);
        if (Sh::kBuffers == 2 && st + 1 < steps) build(st + 1, (st + 1) % 3, tab + (size_t)((st + 1) & 1) * KB * 36 * CU);
        const SpinPair<W> *from = tab + (Sh::kBuffers == 2 ? (size_t)(st & 1) * KB * 36 * CU : 0);
        if (kOne && one) {
#pragma unroll
          for (int r = 0; r < Sh::kRounds; ++r) pairs(mine[r], st, st % 3, from, std::true_type{});
        } else {
#pragma unroll
          for (int r = 0; r < Sh::kRounds; ++r) pairs(mine[r], st, st % 3, from, std::false_type{});
        }
        __syncthreads();
        if (Sh::kBuffers == 1 && st + 1 < steps) {
          build(st + 1, (st + 1) % 3, tab);
          __syncthreads();
        }
      }
    }
  }
  double acc[2];
  sum.total(acc);
  block_sum<2>(acc, partial);
}

__global__ void k_finish2(const double *partial, int nb, double *out) {
  const int k = blockIdx.x;
  double s = 0.0;
  for (int b = threadIdx.x; b < nb; b += blockDim.x) s += partial[(int64_t)b * 2 + k];
  __shared__ double red[32];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double x = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    x = warp_sum(x);
    if (threadIdx.x == 0) out[k] = x;
  }
}

// generation of the V_hppp / V_hhhp blocks (setup_vnn_hppp_block NN part, ccm_iter.f90:1720-1760;
// V_hhhp as ccm_iter.f90:885-930): vnn_hppp(kl, ij) = <ij|V|kl>, vnn_hhhp(ij, kd) = <ij|V|kd>
template <typename S, bool LAT>
__global__ void k_gen_block(DevOrbits O, DevPotential P, const int2 *__restrict__ rows, const int2 *__restrict__ cols,
                            const int64_t *__restrict__ off, const int *__restrict__ nr, const int *__restrict__ nc,
                            const int *__restrict__ roff, const int *__restrict__ coff, int nchan, int rows_are_ket,
                            S *__restrict__ V) {
  for (int ch = blockIdx.x; ch < nchan; ch += gridDim.x) {
    const int r = nr[ch], c = nc[ch];
    for (int64_t e = threadIdx.x; e < (int64_t)r * c; e += blockDim.x) {
      const int ri = (int)(e % r), ci = (int)(e / r);
      const int2 x = rows[roff[ch] + ri], y = cols[coff[ch] + ci];
      V[off[ch] + e] =
          rows_are_ket ? pot::anti_of<S, LAT>(O, P, y.x, y.y, x.x, x.y) : pot::anti_of<S, LAT>(O, P, x.x, x.y, y.x, y.y);
    }
  }
}

template <typename S> __device__ inline S in_cvt(const double *p);
template <> __device__ inline double in_cvt<double>(const double *p) { return p[0]; }
template <> __device__ inline cplx in_cvt<cplx>(const double *p) { return cplx(p[0], p[1]); }
template <typename S>
__global__ void k_copy_in(const double *__restrict__ src, int64_t n, S *__restrict__ dst) {
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    dst[e] = in_cvt<S>(src + 2 * e);
}

// Device buffer.  What it is filled with is in place when put and zeros return: both run on the
// legacy stream, which the engine's streams do not wait for.
struct DB {
  void *p = nullptr;
  size_t n = 0;
  ~DB() { release(); }
  void release() {
    if (p) cudaFree(p);
    p = nullptr;
    n = 0;
  }
  template <typename T> void put(const std::vector<T> &h) {
    n = std::max<size_t>(h.size(), 1) * sizeof(T);
    tck(cudaMalloc(&p, n), "cudaMalloc (T)");
    if (!h.empty()) tck(cudaMemcpy(p, h.data(), h.size() * sizeof(T), cudaMemcpyHostToDevice), "upload (T)");
    tck(cudaStreamSynchronize(cudaStreamLegacy), "upload (T)");
  }
  void zeros(size_t bytes) {
    n = std::max<size_t>(bytes, 1);
    tck(cudaMalloc(&p, n), "cudaMalloc (T)");
    tck(cudaMemset(p, 0, n), "memset (T)");
    tck(cudaStreamSynchronize(cudaStreamLegacy), "memset (T)");
  }
  template <typename T> T *as() const { return (T *)p; }
};

}  // namespace

template <typename S>
class Triples final : public ITriples<S> {
 public:
  Triples(const Layout &L, const DevOrbits &O, int device) : O_(O) {
    tck(cudaSetDevice(device), "cudaSetDevice");
    const Basis &B = L.b;
    const int A = B.A, NP = B.ns - A;
    TD_.A = A; TD_.NP = NP;
    if (std::max(B.nkmax[0], std::max(B.nkmax[1], B.nkmax[2])) > 21)
      throw EngineError(1, "(T): momentum range too large for packed quantum numbers");
    build_momenta(B);
    // hppp (kind 5) and hhhp (kind 2) blocks in the reference's ordered layout
    auto blocks = [&](int kind, std::vector<int2> &s1slot, std::vector<int2> &s2slot, bool s1_is_hh, DB &off, DB &nrow,
                      std::vector<int64_t> &offh, std::vector<int2> &rows, std::vector<int2> &cols, std::vector<int> &nr,
                      std::vector<int> &nc, std::vector<int> &roff, std::vector<int> &coff) {
      const ChannelFamily &F = L.fam[kind];
      int64_t acc = 0;
      for (int c = 0; c < F.count(); ++c) {
        const PairList &a = F.side1[c], &b = F.side2[c];
        offh.push_back(acc);
        nr.push_back(a.size());
        nc.push_back(b.size());
        roff.push_back((int)rows.size());
        coff.push_back((int)cols.size());
        acc += (int64_t)a.size() * b.size();
        for (int r = 0; r < a.size(); ++r) {
          rows.push_back(make_int2(a.p[r], a.q[r]));
          if (s1_is_hh) s1slot[(size_t)a.p[r] * A + a.q[r]] = make_int2(c, r);
          else s1slot[(size_t)a.p[r] * NP + (a.q[r] - A)] = make_int2(c, r);
        }
        for (int r = 0; r < b.size(); ++r) {
          cols.push_back(make_int2(b.p[r], b.q[r]));
          if (kind == 5) s2slot[(size_t)(b.p[r] - A) * NP + (b.q[r] - A)] = make_int2(c, r);
          else s2slot[(size_t)b.p[r] * NP + (b.q[r] - A)] = make_int2(c, r);
        }
      }
      off.put(offh);
      nrow.put(nr);
      return acc;
    };
    std::vector<int2> hp5((size_t)A * NP, make_int2(-1, 0)), pp5((size_t)NP * NP, make_int2(-1, 0));
    std::vector<int2> hh2((size_t)A * A, make_int2(-1, 0)), hp2((size_t)A * NP, make_int2(-1, 0));
    std::vector<int64_t> o5, o2;
    std::vector<int2> r5, c5, r2, c2;
    std::vector<int> nr5, nc5, ro5, co5, nr2, nc2, ro2, co2;
    n_v5_ = blocks(5, hp5, pp5, false, v5_off_, n5_, o5, r5, c5, nr5, nc5, ro5, co5);
    n_v2_ = blocks(2, hh2, hp2, true, v2_off_, n2_, o2, r2, c2, nr2, nc2, ro2, co2);
    off5_h_ = o5; off2_h_ = o2; nr5_h_ = nr5; nc5_h_ = nc5; nr2_h_ = nr2; nc2_h_ = nc2;
    rows5_.put(r5); cols5_.put(c5); rows2_.put(r2); cols2_.put(c2);
    nc5_.put(nc5); ro5_.put(ro5); co5_.put(co5); nc2_.put(nc2); ro2_.put(ro2); co2_.put(co2);
    {  // columns and rows of the blocks
      auto col = [](const std::vector<int2> &slot, const std::vector<int64_t> &off, const std::vector<int> &rows) {
        std::vector<int64_t> v(slot.size(), -1);
        for (size_t x = 0; x < slot.size(); ++x)
          if (slot[x].x >= 0) v[x] = off[slot[x].x] + (int64_t)rows[slot[x].x] * slot[x].y;
        return v;
      };
      auto row = [](const std::vector<int2> &slot) {
        std::vector<int> v(slot.size(), -1);
        for (size_t x = 0; x < slot.size(); ++x)
          if (slot[x].x >= 0) v[x] = slot[x].y;
        return v;
      };
      v5_col_.put(col(pp5, o5, nr5)); v5_row_.put(row(hp5));
      v2_col_.put(col(hp2, o2, nr2)); v2_row_.put(row(hh2));
      std::vector<int64_t> tc((size_t)A * A, 0);
      std::vector<int> tr((size_t)NP * NP, 0);
      for (int i = 0; i < A; ++i)
        for (int j = 0; j < A; ++j) {
          const int pos = L.hh_hhpp[(size_t)i * B.ns + j];
          if (!pos) continue;
          const PackedChannel &pk = L.pk[L.chan3_of_pair(i, j)];
          const int sl = pk.hh_packed[pos - 1];
          const int64_t c = pk.t_off + (int64_t)pk.P * sidx(sl) + 1;
          tc[(size_t)i * A + j] = sl > 0 ? c : sl < 0 ? -c : 0;
        }
      for (int a = 0; a < NP; ++a)
        for (int b = 0; b < NP; ++b) {
          const int pos = L.pp_hhpp[(size_t)(a + A) * B.ns + (b + A)];
          if (pos) tr[(size_t)a * NP + b] = L.pk[L.chan3_of_pair(a + A, b + A)].pp_packed[pos - 1];
        }
      t_col_.put(tc); t_row_.put(tr);
    }
    TD_.t_col = t_col_.as<int64_t>(); TD_.t_row = t_row_.as<int>();
    TD_.v5_col = v5_col_.as<int64_t>(); TD_.v5_row = v5_row_.as<int>();
    TD_.v2_col = v2_col_.as<int64_t>(); TD_.v2_row = v2_row_.as<int>();
    V5_.zeros((size_t)n_v5_ * sizeof(S));
    V2_.zeros((size_t)n_v2_ * sizeof(S));
    partial_.zeros((size_t)kMaxBlocks * 2 * sizeof(double));
    res_.zeros(4 * sizeof(double));
  }

  bool has_v() const override { return have5_ && have2_; }
  bool generated() const override { return generated_; }
  int64_t launches() const override { return launches_; }

  void set_hhhp(int ch, const double *v, cudaStream_t st) override {
    if (ch < 0 || ch >= (int)off2_h_.size()) throw EngineError(1, "hhhp channel out of range");
    stage(v, (int64_t)nr2_h_[ch] * nc2_h_[ch], V2_.as<S>() + off2_h_[ch], st);
    have2_ = true;
    low_ready_ = false;
  }
  void set_hppp(int ch, const double *v, cudaStream_t st) override {
    if (ch < 0 || ch >= (int)off5_h_.size()) throw EngineError(1, "hppp channel out of range");
    stage(v, (int64_t)nr5_h_[ch] * nc5_h_[ch], V5_.as<S>() + off5_h_[ch], st);
    have5_ = true;
    low_ready_ = false;
  }
  void generate_v(const DevPotential &pot, cudaStream_t st) override {
    const int n5 = (int)off5_h_.size(), n2 = (int)off2_h_.size();
    auto gen = [&](auto kernel) {
      if (n5) kernel<<<std::min(n5, 8192), 256, 0, st>>>(O_, pot, rows5_.as<int2>(), cols5_.as<int2>(), v5_off_.as<int64_t>(),
                                                         n5_.as<int>(), nc5_.as<int>(), ro5_.as<int>(), co5_.as<int>(), n5,
                                                         1, V5_.as<S>());
      if (n2) kernel<<<std::min(n2, 8192), 256, 0, st>>>(O_, pot, rows2_.as<int2>(), cols2_.as<int2>(), v2_off_.as<int64_t>(),
                                                         n2_.as<int>(), nc2_.as<int>(), ro2_.as<int>(), co2_.as<int>(), n2,
                                                         0, V2_.as<S>());
    };
    if (pot.lat) gen(k_gen_block<S, true>);
    else gen(k_gen_block<S, false>);
    launches_ += 2;
    tck(cudaGetLastError(), "V_hppp/V_hhhp generation");
    have5_ = have2_ = generated_ = true;
    low_ready_ = false;
  }
  void energy(const S *T, int64_t n_t, const S *fdiag, double et[2], cudaStream_t st, bool fp32) override {
    if (!has_v()) throw EngineError(4, "(T): V_hppp and V_hhhp blocks are not set");
    if (TD_.nbra > 0 && TD_.npm > 0) {
      int blocks = 0;
      if (fp32) {
        using Wt = typename LowOf<S>::type;
        if (!low_ready_) {  // FP32 copies of the interaction, once per interaction
          if (!V5l_.p) V5l_.zeros((size_t)std::max<int64_t>(n_v5_, 1) * sizeof(Wt));
          if (!V2l_.p) V2l_.zeros((size_t)std::max<int64_t>(n_v2_, 1) * sizeof(Wt));
          k_to_low<S><<<1216, 256, 0, st>>>(V5_.as<S>(), n_v5_, V5l_.as<Wt>());
          k_to_low<S><<<1216, 256, 0, st>>>(V2_.as<S>(), n_v2_, V2l_.as<Wt>());
          launches_ += 2;
          low_ready_ = true;
        }
        if (Tl_.n < (size_t)std::max<int64_t>(n_t, 1) * sizeof(Wt)) {
          Tl_.release();
          Tl_.zeros((size_t)std::max<int64_t>(n_t, 1) * sizeof(Wt));
        }
        k_to_low<S><<<1216, 256, 0, st>>>(T, n_t, Tl_.as<Wt>());
        ++launches_;
        blocks = two_isospins_ ? run<Wt, 4>(Tl_.as<Wt>(), V5l_.as<Wt>(), V2l_.as<Wt>(), fdiag, st)
                               : run<Wt, 2>(Tl_.as<Wt>(), V5l_.as<Wt>(), V2l_.as<Wt>(), fdiag, st);
      } else {
        blocks = two_isospins_ ? run<S, 4>(T, V5_.as<S>(), V2_.as<S>(), fdiag, st)
                               : run<S, 2>(T, V5_.as<S>(), V2_.as<S>(), fdiag, st);
      }
      k_finish2<<<2, 256, 0, st>>>(partial_.as<double>(), blocks, res_.as<double>());
      launches_ += 2;
      tck(cudaGetLastError(), "(T) kernel");
      double h[2];
      tck(cudaMemcpyAsync(h, res_.p, 2 * sizeof(double), cudaMemcpyDeviceToHost, st), "(T) result");
      tck(cudaStreamSynchronize(st), "(T) sync");
      et[0] = h[0];
      et[1] = h[1];
    } else {
      et[0] = et[1] = 0.0;
    }
  }

 private:
  static constexpr int kMaxBlocks = 152 * 32;

  // the contractions in type W with G states per momentum, as many blocks as fit the device
  template <typename W, int G>
  int run(const W *T, const W *V5, const W *V2, const S *fdiag, cudaStream_t st) {
    using Sh = TripleShape<W, G>;
    const auto kernel = k_triples<S, W, G>;
    TD_.bra = std::is_same<S, W>::value ? bra64_.as<int3>() : bra_.as<int3>();
    int64_t &want = want_[std::is_same<S, W>::value];  // blocks that the device holds at once
    if (!want) {
      tck(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)Sh::table_bytes()), "(T) attribute");
      int per_sm = 0, sms = 0, dev = 0;
      tck(cudaGetDevice(&dev), "(T) device");
      tck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "(T) attribute");
      tck(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, Sh::kThreads, Sh::table_bytes()), "(T) occupancy");
      want = std::min<int64_t>(kMaxBlocks, std::max(1, per_sm * sms));
    }
    // Items of work: a block of hole triples and a segment of its (p1, p2) tests, some 64 a thread
    // block where the lattice has enough for a few steps of kets in each.  Thread blocks take them in
    // strides, segment by segment: the first segments hold most of the kets, so each block must get
    // some of all.  A lattice with fewer than two such items a block (a step of kets takes some 5 us,
    // and an item three to get going) gives every block one, every nseg-th test of its triples: SNM 4
    // nmax=2 1280 to 139 us with FP64 contractions and 563 to 78 with FP32, SNM 28 nmax=1 503 to 326
    // and 118 to 90, with the states and their order above.
    const int64_t tests = (int64_t)TD_.npm * TD_.npm;
    int64_t seg = std::max<int64_t>(48 * Sh::kKets, (int64_t)TD_.nbra * tests / (64 * want));
    seg = std::min(tests, (seg + Sh::kThreads - 1) / Sh::kThreads * Sh::kThreads);
    int64_t nseg = (tests + seg - 1) / seg, stride = 1;
    if (nseg * TD_.nbra < 2 * want) {
      nseg = std::min(tests, std::max<int64_t>(1, want / TD_.nbra));
      seg = (tests + nseg - 1) / nseg;
      stride = nseg;
    }
    const int blocks = (int)std::min<int64_t>((int64_t)TD_.nbra * nseg, want);
    kernel<<<blocks, Sh::kThreads, Sh::table_bytes(), st>>>(TD_, T, V5, V2, fdiag, (int)seg, (int)nseg, (int)stride,
                                                            partial_.as<double>());
    return blocks;
  }

  void stage(const double *v, int64_t n, S *dst, cudaStream_t st) {
    if (!v) throw EngineError(1, "null V block");
    DB tmp;
    tmp.zeros((size_t)n * 2 * sizeof(double));
    tck(cudaMemcpyAsync(tmp.p, v, (size_t)n * 2 * sizeof(double), cudaMemcpyHostToDevice, st), "V block upload");
    k_copy_in<S><<<608, 256, 0, st>>>(tmp.as<double>(), n, dst);
    ++launches_;
    tck(cudaStreamSynchronize(st), "V block sync");
    if (!ScalarOf<S>::complex) {
      std::vector<double> h((size_t)n * 2);
      std::copy(v, v + 2 * n, h.begin());
      for (int64_t e = 0; e < n; ++e)
        if (h[2 * e + 1] != 0.0) throw EngineError(1, "complex V block given to a real engine");
    }
  }

  // The lattice's momenta with their hole and particle states, and the blocks of hole triples;
  // the particle momenta of a block's kets follow from the total.
  void build_momenta(const Basis &B) {
    two_isospins_ = B.tzmin != B.tzmax;
    const int ex = 2 * B.nkmax[0] + 1, ey = 2 * B.nkmax[1] + 1, ez = 2 * B.nkmax[2] + 1;
    TD_.ey = ey; TD_.ez = ez;
    TD_.qlo = (unsigned)(kQBias - B.nkmax[0]) | (unsigned)(kQBias - B.nkmax[1]) << 8 | (unsigned)(kQBias - B.nkmax[2]) << 16;
    TD_.qspan = (unsigned)(2 * B.nkmax[0]) | (unsigned)(2 * B.nkmax[1]) << 8 | (unsigned)(2 * B.nkmax[2]) << 16;
    std::vector<int2> mom((size_t)ex * ey * ez, make_int2(-1, -1));
    std::vector<unsigned> q[2];
    std::vector<std::array<int, 4>> orb[2];
    for (int p = 0; p < B.ns; ++p) {  // momenta in the order of their first orbital
      const size_t key = ((size_t)(B.nx[p] + B.nkmax[0]) * ey + (B.ny[p] + B.nkmax[1])) * ez + (B.nz[p] + B.nkmax[2]);
      const int part = p >= B.A;
      int &at = part ? mom[key].y : mom[key].x;
      if (at < 0) {
        at = (int)q[part].size();
        q[part].push_back((unsigned)(B.nx[p] + kQBias) | (unsigned)(B.ny[p] + kQBias) << 8 |
                          (unsigned)(B.nz[p] + kQBias) << 16);
        orb[part].push_back({-1, -1, -1, -1});
      }
      orb[part][at][(two_isospins_ && B.tz[p] > 0 ? 2 : 0) + (B.sz[p] > 0 ? 1 : 0)] = p;
    }
    TD_.nhm = (int)q[0].size();
    TD_.npm = (int)q[1].size();
    if (TD_.npm > 46340) throw EngineError(1, "(T): momentum range too large for packed quantum numbers");
    // Every three hole momenta with a triple of hole states among them.  For FP64 contractions
    // two that coincide come first, where the kernel leaves the states out of order out (items);
    // FP32 ones keep the orbitals' order, in which W is rounded.
    std::vector<int3> bra, bra64;
    auto states = [&](int m) {
      int n = 0;
      for (int o : orb[0][m]) n += o >= 0;
      return n;
    };
    for (int a = 0; a < TD_.nhm; ++a)
      for (int b = a; b < TD_.nhm; ++b)
        for (int c = b; c < TD_.nhm; ++c) {
          if (a == c ? states(a) < 3 : (a == b && states(a) < 2) || (b == c && states(b) < 2)) continue;
          bra.push_back(make_int3(a, b, c));
          bra64.push_back(b == c && a != b ? make_int3(b, c, a) : make_int3(a, b, c));
        }
    // The longest first (distinct momenta, two that coincide, three), but for FP64 contractions only
    // where thread blocks get one item each: SNM 28 nmax=1 361 to 327 us, nmax=2 9.8 to 10.3 ms (FP32
    // 1.50 to 1.45).
    auto spread = [](const int3 &b) { return (b.x != b.y) + (b.y != b.z) + (b.x != b.z); };
    auto longest = [&](std::vector<int3> &v) {
      std::stable_sort(v.begin(), v.end(), [&](const int3 &x, const int3 &y) { return spread(x) > spread(y); });
    };
    longest(bra);
    if ((int64_t)bra.size() * TD_.npm * TD_.npm < 1 << 18) longest(bra64);
    TD_.nbra = (int)bra.size();
    hmom_.put(q[0]); pmom_.put(q[1]); mom_of_.put(mom); bra_.put(bra); bra64_.put(bra64);
    horb_.put(orb[0]); porb_.put(orb[1]);
    TD_.hmom = hmom_.as<unsigned>(); TD_.pmom = pmom_.as<unsigned>();
    TD_.horb = horb_.as<int4>(); TD_.porb = porb_.as<int4>();
    TD_.mom_of = mom_of_.as<int2>();
  }

  DevOrbits O_;
  TriplesDev TD_{};
  DB hmom_, pmom_, horb_, porb_, mom_of_, bra_, bra64_;
  bool two_isospins_ = false;
  DB t_col_, t_row_, v5_col_, v5_row_, v2_col_, v2_row_, v5_off_, n5_, v2_off_, n2_;
  DB rows5_, cols5_, rows2_, cols2_, nc5_, ro5_, co5_, nc2_, ro2_, co2_;
  DB V5l_, V2l_, Tl_;  // FP32 copies for the FP32 contractions
  bool low_ready_ = false;
  DB V5_, V2_, partial_, res_;
  std::vector<int64_t> off5_h_, off2_h_;
  std::vector<int> nr5_h_, nc5_h_, nr2_h_, nc2_h_;
  int64_t n_v5_ = 0, n_v2_ = 0, launches_ = 0;
  int64_t want_[2] = {0, 0};  // thread blocks of a launch with FP32 and FP64 contractions
  bool have5_ = false, have2_ = false, generated_ = false;
};

template <typename S>
std::unique_ptr<ITriples<S>> make_triples(const Layout &L, const DevOrbits &O, int device) {
  return std::unique_ptr<ITriples<S>>(new Triples<S>(L, O, device));
}

template std::unique_ptr<ITriples<double>> make_triples<double>(const Layout &, const DevOrbits &, int);
template std::unique_ptr<ITriples<cplx>> make_triples<cplx>(const Layout &, const DevOrbits &, int);

}  // namespace ccx
