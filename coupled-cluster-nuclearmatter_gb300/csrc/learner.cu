// Learned warm start (see learner.hpp): feature extraction, FP32 training kernels (a tile of
// samples through all layers and back in one kernel, sliced weight gradients reduced in a fixed
// order, Adam) and the fused BF16 tensor-core inference kernel.
#include <cuda_pipeline.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <random>
#include <string>
#include <vector>

#include "common.cuh"
#include "engine.hpp"
#include "learner.hpp"
#include "tc_ptx.cuh"

namespace ccx {

namespace {

using namespace tcptx;

void lck(cudaError_t e, const char *what) {
  if (e != cudaSuccess) throw EngineError(2, std::string(what) + ": " + cudaGetErrorString(e));
}

struct LBuf {
  void *p = nullptr;
  size_t bytes = 0;
  LBuf() = default;
  LBuf(const LBuf &) = delete;
  LBuf &operator=(const LBuf &) = delete;
  LBuf(LBuf &&o) noexcept : p(o.p), bytes(o.bytes) { o.p = nullptr; o.bytes = 0; }
  ~LBuf() { if (p) cudaFree(p); }
  void alloc(size_t b) {
    if (p) cudaFree(p);
    p = nullptr;
    bytes = std::max<size_t>(b, 16);
    lck(cudaMalloc(&p, bytes), "cudaMalloc (learner)");
  }
  template <typename T> T *as() const { return (T *)p; }
};

// ---------------------------------------------------------------- features
constexpr float kMlPriorUnit = 100.0f;  // the prior feature in units of 0.01, a typical correction
struct MLCtx {
  DevLayout L;
  DevOrbits O;
  const double *fd, *V;
  const float *prior;  // per packed amplitude, or null
  float rho, kF, eF, vol, th[3];
};

__device__ __forceinline__ float norm3(float x, float y, float z) { return sqrtf(x * x + y * y + z * z); }

// Features of packed amplitude e of hhpp channel ch (a<b particles, i<j holes), and
// its MP2 value V/D in FP64.  Momenta in units of kF and energies in units of eF make
// the features comparable across densities.
__device__ void ml_feat(const MLCtx &c, int ch, int e, float (&f)[kMlIn], double &tmp2) {
  const int P = c.L.P[ch];
  const int ij = e / P, ab = e - ij * P;
  const int2 po = c.L.pp_orb[c.L.pp_off[ch] + ab], ho = c.L.hh_orb[c.L.hh_off[ch] + ij];
  const int a = po.x, b = po.y, i = ho.x, j = ho.y;
  const double D = ((0.0 - c.fd[a]) - c.fd[b] + c.fd[i]) + c.fd[j];
  const double v = c.V[c.L.t_off[ch] + e];
  tmp2 = D == 0.0 ? 0.0 : v / D;
  const float ik = 1.0f / c.kF;
  const float ax = (float)c.O.kx[a] * ik, ay = (float)c.O.ky[a] * ik, az = (float)c.O.kz[a] * ik;
  const float bx = (float)c.O.kx[b] * ik, by = (float)c.O.ky[b] * ik, bz = (float)c.O.kz[b] * ik;
  const float ix = (float)c.O.kx[i] * ik, iy = (float)c.O.ky[i] * ik, iz = (float)c.O.kz[i] * ik;
  const float jx = (float)c.O.kx[j] * ik, jy = (float)c.O.ky[j] * ik, jz = (float)c.O.kz[j] * ik;
  f[0] = (c.rho - 0.12f) / 0.08f;
  f[1] = c.th[0];
  f[2] = c.th[1];
  f[3] = c.th[2];
  f[4] = (float)D / c.eF;
  f[5] = (float)v * c.vol / 500.0f;
  f[6] = (float)tmp2 * c.vol / 10.0f;
  f[7] = norm3(ax - ix, ay - iy, az - iz);
  f[8] = norm3(ax - jx, ay - jy, az - jz);
  f[9] = norm3(ax + bx, ay + by, az + bz);
  f[10] = (ax * ax + ay * ay + az * az) + (bx * bx + by * by + bz * bz) - 2.0f;
  f[11] = (ix * ix + iy * iy + iz * iz) + (jx * jx + jy * jy + jz * jz);
  f[12] = (float)(c.O.sz[a] * c.O.sz[b]);
  f[13] = (float)(c.O.sz[a] * c.O.sz[i]);
  f[14] = (float)(c.O.tz[a] * c.O.tz[b]);
  f[15] = (float)(c.O.tz[a] * c.O.tz[i]);
  // the prior: the correction interpolated from neighbouring converged solutions
  f[16] = c.prior ? c.prior[c.L.t_off[ch] + e] * kMlPriorUnit : 0.0f;
  f[17] = c.prior ? 1.0f : 0.0f;
}

// Target: the correction of the amplitude numerator, y = (T - T_MP2) D vol / kMlNum, with
// D the bare denominator.  The residual weights an amplitude error by D, so a uniform
// error in y is a uniform error in the residual of the start.
constexpr double kMlNum = 1000.0;  // MeV fm^3

// training samples of a converged solution, every stride-th packed amplitude g:
// X[g / stride] features, y[g / stride] the numerator correction
__global__ void k_ml_extract(MLCtx c, const double *__restrict__ T, int stride, float *__restrict__ X,
                             float *__restrict__ y) {
  const int2 tl = c.L.ttile[blockIdx.x];
  const int ch = tl.x;
  const int n = c.L.P[ch] * c.L.H[ch];
  const int end = min(tl.y + kTileElems, n);
  for (int e = tl.y + threadIdx.x; e < end; e += blockDim.x) {
    const int64_t g = c.L.t_off[ch] + e;
    if (g % stride) continue;
    float f[kMlIn];
    double tmp2;
    ml_feat(c, ch, e, f, tmp2);
    const int64_t o = g / stride;
#pragma unroll
    for (int q = 0; q < kMlIn; ++q) X[o * kMlIn + q] = f[q];
    const double D = (double)f[4] * (double)c.eF;
    // with a prior the network learns what the prior leaves over (a skip connection):
    // the BF16 inference then perturbs only that small remainder
    y[o] = (float)((T[g] - tmp2) * D * (double)c.vol / kMlNum) - (c.prior ? c.prior[g] : 0.0f);
  }
}
// A solution the prior is taken from (another density of the same lattice and twist)
struct PriorSrc {
  DevLayout L;
  const double *fd, *V, *T;
  const int *oof;
  double vol;
};
// prior += w * (the numerator correction of src's T), per packed amplitude g of the target
// layout Lt: the target's orbitals a, b, i, j are mapped to src's by quantum numbers
// (okey of the target, oof of src), and src's packed amplitude is read with the product of
// its two pair-slot signs.  The correction (T - V/D) D vol / 1000 is src's own, which
// makes it comparable across densities.
__global__ void k_ml_prior(DevLayout Lt, const int *__restrict__ okey, PriorSrc src, float w, int first,
                           float *__restrict__ prior) {
  const int2 tl = Lt.ttile[blockIdx.x];
  const int ch = tl.x;
  const int P = Lt.P[ch];
  const int end = min(tl.y + kTileElems, P * Lt.H[ch]);
  const DevLayout &L = src.L;
  for (int e = tl.y + threadIdx.x; e < end; e += blockDim.x) {
    const int ij = e / P, ab = e - ij * P;
    const int2 po = Lt.pp_orb[Lt.pp_off[ch] + ab], ho = Lt.hh_orb[Lt.hh_off[ch] + ij];
    const int a = src.oof[okey[po.x]], b = src.oof[okey[po.y]];
    const int i = src.oof[okey[ho.x]], j = src.oof[okey[ho.y]];
    float y = 0.0f;
    if (a >= L.A && b >= L.A && i >= 0 && i < L.A && j >= 0 && j < L.A) {
      const int2 sab = L.pp_slot[(int64_t)(a - L.A) * L.NP + (b - L.A)];
      const int2 sij = L.hh_slot[i * L.A + j];
      if (sab.y != 0 && sij.y != 0 && sab.x == sij.x) {
        const int64_t gs = L.t_off[sab.x] + sidx(sab.y) + (int64_t)L.P[sab.x] * sidx(sij.y);
        const double sg = ssign(sab.y) * ssign(sij.y);
        const double D = ((0.0 - src.fd[a]) - src.fd[b] + src.fd[i]) + src.fd[j];
        if (D != 0.0) y = (float)(sg * (src.T[gs] - src.V[gs] / D) * D * src.vol / kMlNum);
      }
    }
    const int64_t g = Lt.t_off[ch] + e;
    prior[g] = first ? w * y : fmaf(w, y, prior[g]);
  }
}

__global__ void k_ml_gather(const float *__restrict__ Xs, const float *__restrict__ ys, const int64_t *__restrict__ perm,
                            int64_t n, float *__restrict__ X, float *__restrict__ y) {
  for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < n; r += (int64_t)gridDim.x * blockDim.x) {
    const int64_t s = perm[r];
#pragma unroll
    for (int q = 0; q < kMlIn; ++q) X[r * kMlIn + q] = Xs[s * kMlIn + q];
    y[r] = ys[s];
  }
}

// ---------------------------------------------------------------- FP32 training
__device__ __forceinline__ float sigm(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float silu(float z) { return z * sigm(z); }

// A training pass is three kernels: k_ml_pass runs a tile of samples through all layers,
// forward and back, k_ml_wgrad forms the weight gradients from the activations and
// differences it left, k_ml_grad adds the partial sums up.
//
// k_ml_pass: 256 threads take a tile of 16 R samples; thread (tm, tn) owns samples
// R tm .. R tm + R - 1 and the columns 4 tn .. 4 tn + 3 and 64 + 4 tn .. 64 + 4 tn + 3 of every
// layer, so silu'(Z1), silu'(Z2), silu'(Z3) stay in its registers for the way back, and only the
// 128-wide operand of the next product goes through shared memory (k-major).  The weights of a
// product are copied while the one before it runs.  The FMAs (1.7 GFLOP for 8192 samples) keep
// their pipe 40% busy and the issue slots 51%: one block of eight warps an SM waits for its
// shared-memory reads and barriers.  The layers as 25 separate launches of a 64 x 64 tile GEMM, the gradients and column
// sums among them on a few dozen blocks, took 966 us with the copies to and from the host; now 125,
// of which this kernel 48, the weight gradients 26 and their sum 6.
constexpr int kPassThreads = 256;
constexpr int kWRow = kMlW;  // floats of one k of a weight operand in shared memory
template <int R>
struct PassTile {
  static constexpr int kSamples = 16 * R;
  static constexpr int kActRow = kSamples + 4;
  static constexpr size_t kSmem = (2 * kMlW * kWRow + kMlW * kActRow + 16 * kMlW) * sizeof(float);
};
struct PassArgs {
  const float *X, *y;     // samples (n x kMlIn) and targets; y null: forward only
  int n;
  const float *p, *pT;    // parameters, and W1, W2, W3 transposed ([in][out], at the same order)
  float *out;             // forward only: the outputs
  float *H1, *H2, *D1, *D2, *D3;  // activations and pre-activation differences (n x kMlW)
  float *part;            // per tile: db1, db2, db3, dw4 (kMlW each), db4
  double *loss;           // per tile: sum of squared differences
};
constexpr int kPartLen = 4 * kMlW + 1;
constexpr int kPT1 = 0, kPT2 = kPT1 + kMlIn * kMlW, kPT3 = kPT2 + kMlW * kMlW, kPTLen = kPT3 + kMlW * kMlW;

__device__ __forceinline__ void copy_weights(float *dst, const float *src, int floats) {
  for (int x = 4 * threadIdx.x; x < floats; x += 4 * kPassThreads) __pipeline_memcpy_async(dst + x, src + x, 16);
  __pipeline_commit();
}
// acc(m, c) = sum_k act[k][m] w[k][c] over the thread's samples and columns
template <int R>
__device__ __forceinline__ void pass_product(const float *act, const float *w, int K, int tm, int tn, float (&acc)[R][8]) {
  constexpr int AR = PassTile<R>::kActRow;
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
#pragma unroll 4
  for (int k = 0; k < K; ++k) {
    float a[R], b[8];
    if constexpr (R == 4) *reinterpret_cast<float4 *>(a) = *reinterpret_cast<const float4 *>(act + k * AR + 4 * tm);
    else *reinterpret_cast<float2 *>(a) = *reinterpret_cast<const float2 *>(act + k * AR + 2 * tm);
    *reinterpret_cast<float4 *>(b) = *reinterpret_cast<const float4 *>(w + k * kWRow + 4 * tn);
    *reinterpret_cast<float4 *>(b + 4) = *reinterpret_cast<const float4 *>(w + k * kWRow + 64 + 4 * tn);
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
  }
}
__device__ __forceinline__ int pass_col(int tn, int j) { return j < 4 ? 4 * tn + j : 60 + 4 * tn + j; }
// the thread's values as the next product's operand, and to global memory when g is given
template <int R>
__device__ __forceinline__ void pass_store(const float (&v)[R][8], float *act, float *g, int m0, int n, int tm, int tn) {
  constexpr int AR = PassTile<R>::kActRow;
#pragma unroll
  for (int j = 0; j < 8; ++j)
#pragma unroll
    for (int i = 0; i < R; ++i) act[pass_col(tn, j) * AR + R * tm + i] = v[i][j];
  if (!g) return;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    const int m = m0 + R * tm + i;
    if (m >= n) continue;
    float *row = g + (int64_t)m * kMlW;
    *reinterpret_cast<float4 *>(row + 4 * tn) = make_float4(v[i][0], v[i][1], v[i][2], v[i][3]);
    *reinterpret_cast<float4 *>(row + 64 + 4 * tn) = make_float4(v[i][4], v[i][5], v[i][6], v[i][7]);
  }
}
// column sums over the tile's samples of the thread sums s, to dst (kMlW); red: 16 x kMlW
__device__ __forceinline__ void pass_colsum(const float (&s)[8], float *red, float *dst, int tm, int tn) {
#pragma unroll
  for (int j = 0; j < 8; ++j) red[tm * kMlW + pass_col(tn, j)] = s[j];
  __syncthreads();
  if (threadIdx.x < kMlW) {
    float t = 0.0f;
#pragma unroll
    for (int q = 0; q < 16; ++q) t += red[q * kMlW + threadIdx.x];
    dst[threadIdx.x] = t;
  }
  __syncthreads();
}

template <int R>
__global__ void __launch_bounds__(kPassThreads, 1) k_ml_pass(PassArgs g) {
  extern __shared__ __align__(16) float psm[];
  constexpr int AR = PassTile<R>::kActRow;
  float *w0 = psm, *w1 = psm + kMlW * kWRow, *act = w1 + kMlW * kWRow, *red = act + kMlW * AR;
  const int tid = threadIdx.x, tm = tid >> 4, tn = tid & 15;
  const int m0 = blockIdx.x * PassTile<R>::kSamples;
  const bool back = g.y != nullptr;
  copy_weights(w0, g.pT + kPT1, kMlIn * kMlW);
  copy_weights(w1, g.pT + kPT2, kMlW * kMlW);
  for (int x = tid; x < PassTile<R>::kSamples * kMlIn; x += kPassThreads) {
    const int m = x / kMlIn, k = x - m * kMlIn;
    act[k * AR + m] = m0 + m < g.n ? g.X[(int64_t)m0 * kMlIn + x] : 0.0f;
  }
  float b[8];
  auto bias = [&](int off) {
#pragma unroll
    for (int j = 0; j < 8; ++j) b[j] = g.p[off + pass_col(tn, j)];
  };
  float z1[R][8], z2[R][8], z3[R][8], v[R][8];
  // pre-activations z to v = silu(z), and z replaced by silu'(z), which is all the way back needs
  auto activate = [&](float (&z)[R][8]) {
#pragma unroll
    for (int i = 0; i < R; ++i)
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const float x = z[i][j] + b[j], sg = sigm(x);
        v[i][j] = x * sg;
        z[i][j] = sg * (1.0f + x * (1.0f - sg));
      }
  };
  // layer 1
  bias(kMlOffB1);
  __pipeline_wait_prior(1);
  __syncthreads();
  pass_product<R>(act, w0, kMlIn, tm, tn, z1);
  activate(z1);
  __syncthreads();  // act and w0 are read
  copy_weights(w0, g.pT + kPT3, kMlW * kMlW);
  pass_store<R>(v, act, back ? g.H1 : nullptr, m0, g.n, tm, tn);
  // layer 2
  bias(kMlOffB2);
  __pipeline_wait_prior(1);
  __syncthreads();
  pass_product<R>(act, w1, kMlW, tm, tn, z2);
  activate(z2);
  __syncthreads();
  if (back) copy_weights(w1, g.p + kMlOffW3, kMlW * kMlW);
  pass_store<R>(v, act, back ? g.H2 : nullptr, m0, g.n, tm, tn);
  // layer 3 and the output
  bias(kMlOffB3);
  if (back) __pipeline_wait_prior(1);
  else __pipeline_wait_prior(0);
  __syncthreads();
  pass_product<R>(act, w0, kMlW, tm, tn, z3);
  activate(z3);
  __syncthreads();
  if (back) copy_weights(w0, g.p + kMlOffW2, kMlW * kMlW);
  float w4[8], dout[R];
#pragma unroll
  for (int j = 0; j < 8; ++j) w4[j] = g.p[kMlOffW4 + pass_col(tn, j)];
  const float b4 = g.p[kMlOffB4];
  double sq = 0.0;
  float db4 = 0.0f;
#pragma unroll
  for (int i = 0; i < R; ++i) {
    float o = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) o = fmaf(v[i][j], w4[j], o);
#pragma unroll
    for (int q = 8; q > 0; q >>= 1) o += __shfl_xor_sync(0xffffffffu, o, q);  // the 16 threads of these samples
    o += b4;
    const int m = m0 + R * tm + i;
    dout[i] = 0.0f;
    if (m < g.n) {
      if (back) {
        const float d = o - g.y[m];
        dout[i] = 2.0f * d / (float)g.n;
        sq += (double)d * d;
        db4 += dout[i];
      } else if (tn == 0) {
        g.out[m] = o;
      }
    }
  }
  if (!back) return;
  float *part = g.part + (int64_t)blockIdx.x * kPartLen;
  // output layer: dw4 = H3^T dout, db4 = sum dout, and the loss; dZ3 = dout w4^T silu'(Z3)
  float s[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) {
    s[j] = 0.0f;
#pragma unroll
    for (int i = 0; i < R; ++i) s[j] = fmaf(v[i][j], dout[i], s[j]);
  }
  pass_colsum(s, red, part + 3 * kMlW, tm, tn);
  if (tn == 0) {  // one thread per sample group
    red[tm] = db4;
    reinterpret_cast<double *>(red + 32)[tm] = sq;
  }
  __syncthreads();
  if (tid == 0) {
    float t = 0.0f;
    double l = 0.0;
    for (int q = 0; q < 16; ++q) {
      t += red[q];
      l += reinterpret_cast<double *>(red + 32)[q];
    }
    part[4 * kMlW] = t;
    g.loss[blockIdx.x] = l;
  }
  __syncthreads();
  auto difference = [&](const float (&dz)[R][8], float *dst, float *db) {  // v * silu': to dst, its column sums to db
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s[j] = 0.0f;
#pragma unroll
      for (int i = 0; i < R; ++i) {
        v[i][j] *= dz[i][j];
        s[j] += v[i][j];
      }
    }
    pass_store<R>(v, act, dst, m0, g.n, tm, tn);
    pass_colsum(s, red, db, tm, tn);
  };
#pragma unroll
  for (int i = 0; i < R; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) v[i][j] = dout[i] * w4[j];
  difference(z3, g.D3, part + 2 * kMlW);
  // dZ2 = (dZ3 W3) silu'(Z2), dZ1 = (dZ2 W2) silu'(Z1)
  __pipeline_wait_prior(1);
  __syncthreads();
  pass_product<R>(act, w1, kMlW, tm, tn, v);
  __syncthreads();
  difference(z2, g.D2, part + kMlW);
  __pipeline_wait_prior(0);
  __syncthreads();
  pass_product<R>(act, w0, kMlW, tm, tn, v);
  __syncthreads();
  difference(z1, g.D1, part);
}

// Weight gradients dW(o, k) = sum_m D(m, o) H(m, k), one slice of the samples a block
// (blockIdx.y: W3, W2, W1), 8 x 8 outputs a thread (W1: 8 x 2 of its 18 columns, padded), to
// the slice's partial sums in the parameters' order.
constexpr int kGradK = 16;      // samples staged at a time
constexpr int kGradStages = 3;  // stages in flight: a stage's FMAs take about as long as its loads
struct WgradArgs {
  const float *X, *H1, *H2, *D1, *D2, *D3;
  int n, per;              // samples, samples of a slice (a multiple of kGradK)
  float *part;             // per slice: W1, W2, W3
};
constexpr int kGradLen = kMlIn * kMlW + 2 * kMlW * kMlW;
__global__ void __launch_bounds__(256) k_ml_wgrad(WgradArgs g) {
  __shared__ __align__(16) float As[kGradStages][kGradK][kMlW], Bs[kGradStages][kGradK][kMlW];
  const int which = blockIdx.y;  // 0: W3, 1: W2, 2: W1
  const float *A = which == 0 ? g.D3 : which == 1 ? g.D2 : g.D1;
  const float *B = which == 0 ? g.H2 : which == 1 ? g.H1 : g.X;
  const int nb = which == 2 ? kMlIn : kMlW;
  const int tid = threadIdx.x, tm = tid >> 4, tn = tid & 15;
  const int beg = blockIdx.x * g.per, end = min(g.n, beg + g.per);
  auto stage = [&](int s, int m) {
    for (int x = 4 * tid; x < kGradK * kMlW; x += 4 * 256) {
      const int r = x / kMlW, c = x % kMlW;
      if (m + r < end) {
        __pipeline_memcpy_async(&As[s][r][c], A + (int64_t)(m + r) * kMlW + c, 16);
        if (which != 2) __pipeline_memcpy_async(&Bs[s][r][c], B + (int64_t)(m + r) * kMlW + c, 16);
      } else {
        *reinterpret_cast<float4 *>(&As[s][r][c]) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (which != 2) *reinterpret_cast<float4 *>(&Bs[s][r][c]) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      }
    }
    if (which == 2)
      for (int x = tid; x < kGradK * 32; x += 256) {
        const int r = x >> 5, c = x & 31;
        Bs[s][r][c] = m + r < end && c < kMlIn ? B[(int64_t)(m + r) * kMlIn + c] : 0.0f;
      }
    __pipeline_commit();
  };
  float acc[8][8];
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int j = 0; j < 8; ++j) acc[i][j] = 0.0f;
  // every iteration commits a group (an empty one past the end), so that the groups count stages
  for (int q = 0; q < kGradStages - 1; ++q) {
    if (beg + q * kGradK < end) stage(q, beg + q * kGradK);
    else __pipeline_commit();
  }
  int s = 0;
  for (int m = beg; m < end; m += kGradK, s = s + 1 == kGradStages ? 0 : s + 1) {
    __pipeline_wait_prior(kGradStages - 2);
    __syncthreads();  // this stage is in place, and the one before it is read
    const int mn = m + (kGradStages - 1) * kGradK, sn = s == 0 ? kGradStages - 1 : s - 1;
    if (mn < end) stage(sn, mn);
    else __pipeline_commit();
#pragma unroll
    for (int k = 0; k < kGradK; ++k) {
      float a[8], b[8];
      *reinterpret_cast<float4 *>(a) = *reinterpret_cast<const float4 *>(&As[s][k][4 * tm]);
      *reinterpret_cast<float4 *>(a + 4) = *reinterpret_cast<const float4 *>(&As[s][k][64 + 4 * tm]);
      if (which != 2) {
        *reinterpret_cast<float4 *>(b) = *reinterpret_cast<const float4 *>(&Bs[s][k][4 * tn]);
        *reinterpret_cast<float4 *>(b + 4) = *reinterpret_cast<const float4 *>(&Bs[s][k][64 + 4 * tn]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 8; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      } else {
        *reinterpret_cast<float2 *>(b) = *reinterpret_cast<const float2 *>(&Bs[s][k][2 * tn]);
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
          for (int j = 0; j < 2; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
      }
    }
  }
  float *out = g.part + (int64_t)blockIdx.x * kGradLen +
               (which == 2 ? 0 : kMlIn * kMlW + (which == 1 ? 0 : kMlW * kMlW));
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    float *row = out + pass_col(tm, i) * nb;
    if (which != 2) {
      *reinterpret_cast<float4 *>(row + 4 * tn) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
      *reinterpret_cast<float4 *>(row + 64 + 4 * tn) = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
    } else if (2 * tn < kMlIn) {
      *reinterpret_cast<float2 *>(row + 2 * tn) = make_float2(acc[i][0], acc[i][1]);
    }
  }
}

// the gradient in the parameters' order from the partial sums of the slices (weights) and of
// the tiles (biases, output layer), each in order; the last block finishes the loss
__global__ void __launch_bounds__(256) k_ml_grad(const float *__restrict__ wpart, int slices, const float *__restrict__ bpart,
                                                 const double *__restrict__ lpart, int tiles, int n, float *__restrict__ grad,
                                                 double *__restrict__ loss) {
  if (blockIdx.x == gridDim.x - 1) {
    __shared__ double sh[256];
    double s = 0.0;
    for (int t = threadIdx.x; t < tiles; t += 256) s += lpart[t];
    sh[threadIdx.x] = s;
    __syncthreads();
    for (int o = 128; o > 0; o >>= 1) {
      if (threadIdx.x < o) sh[threadIdx.x] += sh[threadIdx.x + o];
      __syncthreads();
    }
    if (threadIdx.x == 0) *loss = sh[0] / n;
    return;
  }
  // 32 parameters a block, eight threads each: short chains of loads, and the rounding of a
  // few dozen additions in a row instead of a few hundred
  __shared__ float red[8][32];
  const int q = threadIdx.x >> 5, i = blockIdx.x * 32 + (threadIdx.x & 31);
  const float *src = bpart;
  int64_t step = kPartLen;
  int cnt = i < kMlParams ? tiles : 0;
  if (i < kMlOffB1) { src = wpart + i; step = kGradLen; cnt = slices; }
  else if (i < kMlOffW2) src += i - kMlOffB1;
  else if (i < kMlOffB2) { src = wpart + kMlIn * kMlW + (i - kMlOffW2); step = kGradLen; cnt = slices; }
  else if (i < kMlOffW3) src += kMlW + (i - kMlOffB2);
  else if (i < kMlOffB3) { src = wpart + kMlIn * kMlW + kMlW * kMlW + (i - kMlOffW3); step = kGradLen; cnt = slices; }
  else if (i < kMlOffW4) src += 2 * kMlW + (i - kMlOffB3);
  else src += 3 * kMlW + (i - kMlOffW4);
  float s = 0.0f;
#pragma unroll 8
  for (int z = q; z < cnt; z += 8) s += src[z * step];
  red[q][threadIdx.x & 31] = s;
  __syncthreads();
  if (q == 0 && i < kMlParams) {
    const int l = threadIdx.x;
    grad[i] = ((red[0][l] + red[1][l]) + (red[2][l] + red[3][l])) + ((red[4][l] + red[5][l]) + (red[6][l] + red[7][l]));
  }
}

// index of parameter i in the transposed weights, or -1 (biases, output layer)
__device__ __forceinline__ int transposed_index(int i) {
  if (i < kMlOffB1) return kPT1 + (i % kMlIn) * kMlW + i / kMlIn;
  if (i >= kMlOffW2 && i < kMlOffB2) { const int x = i - kMlOffW2; return kPT2 + (x % kMlW) * kMlW + x / kMlW; }
  if (i >= kMlOffW3 && i < kMlOffB3) { const int x = i - kMlOffW3; return kPT3 + (x % kMlW) * kMlW + x / kMlW; }
  return -1;
}
// New parameters from page-locked host memory, their transposed copy, and Adam's moments from zero,
// in one launch (a copy, two memsets and a transposition took 38 us a call, now 26).
__global__ void k_ml_new_params(const float *__restrict__ host, float *__restrict__ p, float *__restrict__ pT,
                                float *__restrict__ m, float *__restrict__ v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= kMlParams) return;
  const float x = host[i];
  p[i] = x;
  const int t = transposed_index(i);
  if (t >= 0) pT[t] = x;
  m[i] = v[i] = 0.0f;
}

__global__ void k_ml_adam(float *__restrict__ p, float *__restrict__ pT, float *__restrict__ m, float *__restrict__ v,
                          const float *__restrict__ g, int n, float lr, float b1t, float b2t) {
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.0f - b1) * gi;
    const float vi = b2 * v[i] + (1.0f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float x = p[i] - lr * (mi / (1.0f - b1t)) / (sqrtf(vi / (1.0f - b2t)) + eps);
    p[i] = x;
    const int t = transposed_index(i);
    if (t >= 0) pT[t] = x;
  }
}

__global__ void k_ml_scale(float *__restrict__ x, int64_t n, float s) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) x[i] *= s;
}

// ---------------------------------------------------------------- BF16 tensor-core inference
// One persistent CTA of 128 threads per SM, one sample per thread and TMEM lane.  The
// three hidden layers are 128 x 128 x K tcgen05 MMAs with BF16 operands in shared
// memory (weights loaded once per CTA) and the FP32 accumulator in tensor memory; each
// thread turns its accumulator row into the next layer's BF16 operand row (bias, SiLU),
// and the 128 -> 1 output layer is a per-thread FP32 dot product.
constexpr uint32_t kWTile = 128u * 128u;           // one 128-row x 64-BF16 K tile
constexpr uint32_t kWBytes = 5u * kWTile;          // W1 (1 K tile), W2, W3 (2 each)
constexpr uint32_t kFeatOff = kWBytes;             // features: 1 K tile
constexpr uint32_t kActOff = kFeatOff + kWTile;    // activations: 2 K tiles
constexpr uint32_t kParOff = kActOff + 2 * kWTile; // b1, b2, b3, w4 (FP32) and b4
constexpr uint32_t kBarOff2 = kParOff + (4 * kMlW + 4) * 4;
constexpr size_t kInferSmem = kBarOff2 + 32;

struct InferArgs {
  MLCtx c;
  int use_view;
  double *T;                // view: T' written here
  const float *X;           // external features (n x 16)
  float *out;               // external outputs
  int n;
  const uint8_t *wt;        // BF16 weight tiles (kWBytes)
  const float *par;         // FP32 parameter vector
  int ntiles;
  int *err;
};

__device__ __forceinline__ uint32_t bf16_bits(float x) {
  // round to nearest even on the bit pattern (finite inputs)
  const uint32_t u = __float_as_uint(x);
  return (u + 0x7FFFu + ((u >> 16) & 1u)) >> 16;
}
// byte offset of element (row, k) inside a canonical no-swizzle K-major tile set
__device__ __forceinline__ uint32_t cm_off(int row, int k) {
  return (uint32_t)(k >> 6) * kWTile + (uint32_t)((((row >> 3) << 3) + ((k & 63) >> 3)) << 7) + (uint32_t)((row & 7) << 4) +
         (uint32_t)((k & 7) << 1);
}

__global__ void __launch_bounds__(128, 1) k_ml_infer(InferArgs g) {
  extern __shared__ __align__(1024) uint8_t smem[];
  const int tid = threadIdx.x, warp = tid >> 5;
  uint64_t *bar = (uint64_t *)(smem + kBarOff2);
  uint64_t *wbar = bar + 1;
  uint32_t *tslot = (uint32_t *)(bar + 2);
  volatile int *abort_flag = (volatile int *)(tslot + 1);
  float *sp = (float *)(smem + kParOff);
  if (warp == 0) {
    tmem_alloc(smem_u32(tslot), 128);
    tmem_relinquish();
  }
  if (tid == 0) {
    mbar_init(smem_u32(bar), 1);
    mbar_init(smem_u32(wbar), 1);
    *abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // biases and output weights; zero feature padding (K columns 32..63 are never rewritten)
  for (int x = tid; x < kMlW; x += 128) {
    sp[x] = g.par[kMlOffB1 + x];
    sp[kMlW + x] = g.par[kMlOffB2 + x];
    sp[2 * kMlW + x] = g.par[kMlOffB3 + x];
    sp[3 * kMlW + x] = g.par[kMlOffW4 + x];
  }
  if (tid == 0) sp[4 * kMlW] = g.par[kMlOffB4];
  for (int x = tid; x < (int)(kWTile / 16); x += 128) ((uint4 *)(smem + kFeatOff))[x] = make_uint4(0, 0, 0, 0);
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tslot;
  if (tid == 0) {
    mbar_expect_tx(smem_u32(wbar), kWBytes);
    bulk_g2s(smem_u32(smem), g.wt, kWBytes, smem_u32(wbar));
  }
  bool ok = mbar_wait(smem_u32(wbar), 0);
  if (!ok) *abort_flag = 1;
  __syncthreads();
  const uint32_t idesc16 = instr_desc<kTcBF16>(128, 128);
  const uint32_t lane_base = tmem + ((uint32_t)(warp * 32) << 16);
  uint32_t phase = 0;
  for (int t = blockIdx.x; t < g.ntiles && !*abort_flag; t += gridDim.x) {
    // ---- features of this thread's sample
    bool live = false;
    int ch = 0;
    int64_t gidx = 0;
    double tmp2 = 0.0;
    float f[kMlIn];
    if (g.use_view) {
      const int2 tt = g.c.L.ttile[t >> 3];
      ch = tt.x;
      const int e = tt.y + (t & 7) * 128 + tid;
      const int n = g.c.L.P[ch] * g.c.L.H[ch];
      live = e < min(tt.y + kTileElems, n);
      if (live) {
        ml_feat(g.c, ch, e, f, tmp2);
        gidx = g.c.L.t_off[ch] + e;
      }
    } else {
      const int r = t * 128 + tid;
      live = r < g.n;
      if (live)
        for (int q = 0; q < kMlIn; ++q) f[q] = g.X[(int64_t)r * kMlIn + q];
    }
    if (!live)
      for (int q = 0; q < kMlIn; ++q) f[q] = 0.0f;
    {  // features into K columns 0 .. kMlIn - 1 of the tile, zeros up to column 31
      uint32_t w[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const float lo = 2 * q < kMlIn ? f[2 * q] : 0.0f, hi = 2 * q + 1 < kMlIn ? f[2 * q + 1] : 0.0f;
        w[q] = bf16_bits(lo) | (bf16_bits(hi) << 16);
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
        *(uint4 *)(smem + kFeatOff + cm_off(tid, 8 * q)) = make_uint4(w[4 * q], w[4 * q + 1], w[4 * q + 2], w[4 * q + 3]);
    }
    float o = 0.0f;
    for (int layer = 0; layer < 3; ++layer) {
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      tc_fence_before();
      __syncthreads();
      if (tid == 0) {
        tc_fence_after();
        if (layer == 0) {  // K = 32: the features and their zero padding
#pragma unroll
          for (int ks = 0; ks < 2; ++ks)
            tc_mma<kTcBF16>(tmem, smem_desc(smem_u32(smem + kFeatOff) + ks * 256), smem_desc(smem_u32(smem) + ks * 256),
                            idesc16, ks ? 1u : 0u);
        } else {
          const uint32_t wb = smem_u32(smem + (layer == 1 ? kWTile : 3 * kWTile));
#pragma unroll
          for (int kt = 0; kt < 2; ++kt)
#pragma unroll
            for (int ks = 0; ks < 4; ++ks)
              tc_mma<kTcBF16>(tmem, smem_desc(smem_u32(smem + kActOff) + kt * kWTile + ks * 256),
                              smem_desc(wb + kt * kWTile + ks * 256), idesc16, (kt | ks) ? 1u : 0u);
        }
        tc_commit(smem_u32(bar));
      }
      const bool got = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), phase & 1u));
      ++phase;
      if (!got) {
        *abort_flag = 1;
        break;
      }
      tc_fence_after();
      const float *bias = sp + layer * kMlW;
      for (int c0 = 0; c0 < kMlW; c0 += 32) {
        uint32_t r[32];
        tmem_ld32(lane_base + (uint32_t)c0, r);
        tmem_ld_wait();
        if (layer < 2) {
#pragma unroll
          for (int q = 0; q < 32; q += 8) {
            uint32_t w[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
              const float z0 = __uint_as_float(r[q + 2 * h]) + bias[c0 + q + 2 * h];
              const float z1 = __uint_as_float(r[q + 2 * h + 1]) + bias[c0 + q + 2 * h + 1];
              w[h] = bf16_bits(silu(z0)) | (bf16_bits(silu(z1)) << 16);
            }
            *(uint4 *)(smem + kActOff + cm_off(tid, c0 + q)) = make_uint4(w[0], w[1], w[2], w[3]);
          }
        } else {
#pragma unroll
          for (int q = 0; q < 32; ++q) o = fmaf(silu(__uint_as_float(r[q]) + bias[c0 + q]), sp[3 * kMlW + c0 + q], o);
        }
      }
    }
    if (*abort_flag) break;
    o += sp[4 * kMlW];
    if (live) {
      if (g.use_view) {
        if (g.c.prior) o += g.c.prior[gidx];  // the skip connection of the prior, in FP32
        const double D = (double)f[4] * (double)g.c.eF;
        g.T[gidx] = D == 0.0 ? tmp2 : tmp2 + (double)o * kMlNum / (D * (double)g.c.vol);
      }
      else g.out[t * 128 + tid] = o;
    }
  }
  if (*abort_flag && tid == 0) atomicExch(g.err, 1);
  tc_fence_before();
  __syncthreads();
  if (warp == 0) {
    tc_fence_after();
    tmem_dealloc(tmem, 128);
  }
}

// ---------------------------------------------------------------- host side
uint16_t host_bf16(float x) {
  uint32_t u;
  std::memcpy(&u, &x, 4);
  return (uint16_t)((u + 0x7FFFu + ((u >> 16) & 1u)) >> 16);
}
size_t host_cm_off(int row, int k) {
  return (size_t)(k >> 6) * kWTile + (size_t)((((row >> 3) << 3) + ((k & 63) >> 3)) << 7) + (size_t)((row & 7) << 4) +
         (size_t)((k & 7) << 1);
}

MLCtx make_ctx(const MLView &v) {
  MLCtx c{};
  c.L = v.L;
  c.O = v.O;
  c.fd = v.fdiag;
  c.V = v.Vhp;
  c.rho = (float)v.rho;
  c.kF = (float)v.kF;
  c.eF = (float)v.eF;
  c.vol = (float)v.vol;
  for (int q = 0; q < 3; ++q) c.th[q] = (float)(v.theta[q] / 3.14159265358979323846);
  return c;
}

class Learner final : public ILearner {
 public:
  Learner(int device, uint64_t seed) : device_(device) {
    lck(cudaSetDevice(device), "cudaSetDevice");
    lck(cudaStreamCreateWithFlags(&st_, cudaStreamNonBlocking), "cudaStreamCreate");
    params_.alloc(kMlParams * 4);
    m_.alloc(kMlParams * 4);
    v_.alloc(kMlParams * 4);
    grad_.alloc(kGradLoss + 8);
    pT_.alloc(kPTLen * 4);
    lck(cudaMallocHost(&host_grad_, kGradLoss + 8), "cudaMallocHost (learner)");
    wt_.alloc(kWBytes);
    err_.alloc(4);
    lck(cudaMemsetAsync(err_.p, 0, 4, st_), "memset");
    // Kaiming-uniform initial weights from splitmix64, zero biases, small output layer
    std::vector<float> p(kMlParams, 0.0f);
    uint64_t s = seed;
    auto uni = [&]() {
      uint64_t z = (s += 0x9e3779b97f4a7c15ULL);
      z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ULL;
      z = (z ^ (z >> 27)) * 0x94d049bb133111ebULL;
      z ^= z >> 31;
      return (double)(z >> 11) * (1.0 / 9007199254740992.0) * 2.0 - 1.0;
    };
    auto fill = [&](int off, int n, int fan_in, double gain) {
      const double a = gain * std::sqrt(6.0 / fan_in);
      for (int i = 0; i < n; ++i) p[off + i] = (float)(a * uni());
    };
    fill(kMlOffW1, kMlW * kMlIn, kMlIn, 1.0);
    fill(kMlOffW2, kMlW * kMlW, kMlW, 1.0);
    fill(kMlOffW3, kMlW * kMlW, kMlW, 1.0);
    fill(kMlOffW4, kMlW, kMlW, 0.1);
    set_params(p.data());
    folded_ = false;  // the initial output layer is in the standardised units of training
  }
  ~Learner() override {
    if (st_) cudaStreamDestroy(st_);
    if (host_grad_) cudaFreeHost(host_grad_);
  }

  void add_solution(const MLView &v, int stride) override {
    lck(cudaSetDevice(device_), "cudaSetDevice");
    if (stride < 1) throw EngineError(1, "learner: sample stride must be >= 1");
    Chunk c;
    c.n = (v.n_t + stride - 1) / stride;
    c.X.alloc((size_t)c.n * kMlIn * 4);
    c.y.alloc((size_t)c.n * 4);
    const MLCtx ctx = ctx_of(v);
    if (v.L.nttile) k_ml_extract<<<v.L.nttile, 256, 0, v.st>>>(ctx, v.T, stride, c.X.as<float>(), c.y.as<float>());
    lck(cudaGetLastError(), "feature extraction");
    lck(cudaStreamSynchronize(v.st), "feature extraction");
    data_.push_back(std::move(c));
  }
  void set_prior(const MLView &target, const MLView *views, const double *w, int n) override {
    lck(cudaSetDevice(device_), "cudaSetDevice");
    has_prior_ = false;
    if (n <= 0) return;
    const int64_t nt = target.n_t;
    for (int i = 0; i < n; ++i)
      if (views[i].nkeys != target.nkeys || views[i].L.ns != target.L.ns || views[i].L.A != target.L.A)
        throw EngineError(1, "learner: the prior's engines are not the target's lattice at another density");
    if (prior_.bytes < (size_t)std::max<int64_t>(nt, 1) * 4) prior_.alloc((size_t)std::max<int64_t>(nt, 1) * 4);
    lck(cudaStreamSynchronize(target.st), "prior");
    for (int i = 0; i < n; ++i) {
      const MLView &v = views[i];
      lck(cudaStreamSynchronize(v.st), "prior");  // the source's amplitudes are final
      const PriorSrc src{v.L, v.fdiag, v.Vhp, v.T, v.oof, v.vol};
      if (target.L.nttile)
        k_ml_prior<<<target.L.nttile, 256, 0, target.st>>>(target.L, target.okey, src, (float)w[i], i == 0,
                                                            prior_.as<float>());
      lck(cudaGetLastError(), "prior");
    }
    lck(cudaStreamSynchronize(target.st), "prior");
    prior_n_ = nt;
    has_prior_ = true;
  }
  void clear() override { data_.clear(); }
  int64_t samples() const override {
    int64_t n = 0;
    for (const auto &c : data_) n += c.n;
    return n;
  }

  double train(int steps, int batch, double lr, uint64_t seed) override {
    lck(cudaSetDevice(device_), "cudaSetDevice");
    const int64_t N = samples();
    if (N < 1) throw EngineError(4, "learner: no training samples");
    if (batch < 1 || steps < 1) throw EngineError(1, "learner: steps and batch must be positive");
    batch = (int)std::min<int64_t>(batch, N);
    // one concatenated copy, shuffled once per pass with a host permutation
    LBuf Xa, ya, Xs, ys, perm;
    Xa.alloc((size_t)N * kMlIn * 4);
    ya.alloc((size_t)N * 4);
    int64_t o = 0;
    for (const auto &c : data_) {
      lck(cudaMemcpyAsync(Xa.as<float>() + o * kMlIn, c.X.p, (size_t)c.n * kMlIn * 4, cudaMemcpyDeviceToDevice, st_), "copy");
      lck(cudaMemcpyAsync(ya.as<float>() + o, c.y.p, (size_t)c.n * 4, cudaMemcpyDeviceToDevice, st_), "copy");
      o += c.n;
    }
    // The network trains on targets divided by their RMS (fixed at the first training)
    // and the output layer is scaled back afterwards, so that the loss is relative to the
    // size of what is learned (with a prior, a small remainder)
    if (yscale_ <= 0.0f) {
      std::vector<float> yh(N);
      lck(cudaMemcpyAsync(yh.data(), ya.p, (size_t)N * 4, cudaMemcpyDeviceToHost, st_), "targets");
      lck(cudaStreamSynchronize(st_), "targets");
      double ss = 0.0;
      for (float v : yh) ss += (double)v * v;
      yscale_ = (float)std::max(std::sqrt(ss / (double)N), 1e-12);
    }
    k_ml_scale<<<1216, 256, 0, st_>>>(ya.as<float>(), N, 1.0f / yscale_);
    if (folded_) k_ml_scale<<<1, 256, 0, st_>>>(params_.as<float>() + kMlOffW4, kMlW + 1, 1.0f / yscale_);
    Xs.alloc((size_t)N * kMlIn * 4);
    ys.alloc((size_t)N * 4);
    perm.alloc((size_t)N * 8);
    std::vector<int64_t> pv(N);
    std::mt19937_64 rng(seed);
    const int64_t passes_steps = std::max<int64_t>(1, N / batch);
    std::vector<double> losses(steps);
    LBuf lossd;
    lossd.alloc((size_t)steps * 8);
    ensure_batch(batch);
    for (int s = 0; s < steps; ++s) {
      if (s % passes_steps == 0) {
        for (int64_t i = 0; i < N; ++i) pv[i] = i;
        std::shuffle(pv.begin(), pv.end(), rng);
        lck(cudaMemcpyAsync(perm.p, pv.data(), (size_t)N * 8, cudaMemcpyHostToDevice, st_), "perm");
        k_ml_gather<<<1216, 256, 0, st_>>>(Xa.as<float>(), ya.as<float>(), perm.as<int64_t>(), N, Xs.as<float>(),
                                           ys.as<float>());
        lck(cudaStreamSynchronize(st_), "shuffle");
      }
      const int64_t off = (int64_t)(s % passes_steps) * batch;
      forward_backward(Xs.as<float>() + off * kMlIn, ys.as<float>() + off, batch, lossd.as<double>() + s);
      ++t_;
      const float b1t = (float)std::pow(0.9, (double)t_), b2t = (float)std::pow(0.999, (double)t_);
      k_ml_adam<<<(kMlParams + 255) / 256, 256, 0, st_>>>(params_.as<float>(), pT_.as<float>(), m_.as<float>(),
                                                           v_.as<float>(), grad_.as<float>(), kMlParams, (float)lr, b1t,
                                                           b2t);
    }
    // the output layer back in the targets' units (the Adam moments stay with the
    // standardised units of the next training)
    k_ml_scale<<<1, 256, 0, st_>>>(params_.as<float>() + kMlOffW4, kMlW + 1, yscale_);
    folded_ = true;
    lck(cudaGetLastError(), "training");
    lck(cudaMemcpyAsync(losses.data(), lossd.p, (size_t)steps * 8, cudaMemcpyDeviceToHost, st_), "loss");
    lck(cudaStreamSynchronize(st_), "training");
    double tail = 0.0;
    const int k0 = std::max(0, steps - 10);
    for (int s = k0; s < steps; ++s) tail += losses[s];
    weights_dirty_ = true;
    return tail / (steps - k0) * (double)yscale_ * (double)yscale_;
  }

  void warm_start(const MLView &v) override {
    lck(cudaSetDevice(device_), "cudaSetDevice");
    upload_weight_tiles();
    InferArgs a{};
    a.c = ctx_of(v);
    a.use_view = 1;
    a.T = v.T;
    a.wt = wt_.as<uint8_t>();
    a.par = params_.as<float>();
    a.ntiles = v.L.nttile * 8;
    a.err = err_.as<int>();
    run_infer(a, v.st);
  }

  void get_params(float *p) const override {
    lck(cudaMemcpy(p, params_.p, kMlParams * 4, cudaMemcpyDeviceToHost), "params");
  }
  void set_params(const float *p) override {
    // on the learner's own stream, as all that reads them; waited for, since the engines' streams
    // read them too.  Marked first: a failure half-way leaves no inference tiles of the old ones.
    lck(cudaSetDevice(device_), "cudaSetDevice");
    std::lock_guard<std::mutex> hold(io_mutex_);
    weights_dirty_ = true;
    std::memcpy(host_grad_, p, kMlParams * 4);
    k_ml_new_params<<<(kMlParams + 255) / 256, 256, 0, st_>>>((const float *)host_grad_, params_.as<float>(),
                                                               pT_.as<float>(), m_.as<float>(), v_.as<float>());
    lck(cudaGetLastError(), "params");
    lck(cudaStreamSynchronize(st_), "params");
    folded_ = true;  // parameters from get_params: output layer in the targets' units
    t_ = 0;
  }

  void loss_grad(const float *X, const float *y, int n, double *loss, float *grad) override {
    lck(cudaSetDevice(device_), "cudaSetDevice");
    std::lock_guard<std::mutex> hold(io_mutex_);
    if (n < 1) throw EngineError(1, "learner: empty batch");
    ensure_batch(n);
    ensure_io(n);
    lck(cudaMemcpyAsync(ioX_.p, X, (size_t)n * kMlIn * 4, cudaMemcpyHostToDevice, st_), "copy");
    lck(cudaMemcpyAsync(ioy_.p, y, (size_t)n * 4, cudaMemcpyHostToDevice, st_), "copy");
    // the gradient and the loss behind it in one copy
    forward_backward(ioX_.as<float>(), ioy_.as<float>(), n, (double *)(grad_.as<char>() + kGradLoss));
    lck(cudaMemcpyAsync(host_grad_, grad_.p, kGradLoss + 8, cudaMemcpyDeviceToHost, st_), "copy");
    lck(cudaStreamSynchronize(st_), "loss_grad");
    std::memcpy(grad, host_grad_, kMlParams * 4);
    std::memcpy(loss, host_grad_ + kGradLoss, 8);
  }

  void infer(const float *X, int n, float *out, int tensor_cores) override {
    lck(cudaSetDevice(device_), "cudaSetDevice");
    std::lock_guard<std::mutex> hold(io_mutex_);
    if (n < 1) return;
    ensure_io(n);
    lck(cudaMemcpyAsync(ioX_.p, X, (size_t)n * kMlIn * 4, cudaMemcpyHostToDevice, st_), "copy");
    if (tensor_cores) {
      upload_weight_tiles();
      InferArgs a{};
      a.use_view = 0;
      a.X = ioX_.as<float>();
      a.out = ioy_.as<float>();
      a.n = n;
      a.wt = wt_.as<uint8_t>();
      a.par = params_.as<float>();
      a.ntiles = (n + 127) / 128;
      a.err = err_.as<int>();
      run_infer(a, st_);
    } else {
      PassArgs a{};
      a.X = ioX_.as<float>();
      a.n = n;
      a.p = params_.as<float>();
      a.pT = pT_.as<float>();
      a.out = ioy_.as<float>();
      run_pass(a);
    }
    lck(cudaGetLastError(), "infer");
    lck(cudaMemcpyAsync(out, ioy_.p, (size_t)n * 4, cudaMemcpyDeviceToHost, st_), "copy");
    lck(cudaStreamSynchronize(st_), "infer");
  }

 private:
  struct Chunk {
    LBuf X, y;
    int64_t n = 0;
  };

  // the feature context of a view, with the prior when one is set
  MLCtx ctx_of(const MLView &v) const {
    MLCtx c = make_ctx(v);
    if (has_prior_) {
      if (v.n_t != prior_n_) throw EngineError(1, "learner: the prior was set for another layout");
      c.prior = prior_.as<float>();
    }
    return c;
  }

  // Workspaces grow to the largest batch seen and are freed with the learner.
  void ensure_batch(int b) {
    if (b <= cap_) return;
    cap_ = 0;
    for (LBuf *x : {&H1_, &H2_, &D1_, &D2_, &D3_}) x->alloc((size_t)b * kMlW * 4);
    const int tiles = (b + PassTile<2>::kSamples - 1) / PassTile<2>::kSamples;
    bpart_.alloc((size_t)tiles * kPartLen * 4);
    lpart_.alloc((size_t)tiles * 8);
    wpart_.alloc((size_t)kGradSlices * kGradLen * 4);
    cap_ = b;
  }
  void ensure_io(int n) {
    if (n <= io_cap_) return;
    io_cap_ = 0;
    ioX_.alloc((size_t)n * kMlIn * 4);
    ioy_.alloc((size_t)n * 4);
    io_cap_ = n;
  }

  // Tiles of 64 samples, or of 32 while that many leave SMs without one (a tile's time is
  // latency and FMAs of one SM, so half the samples take half of it): 8192 samples 125 us a call in
  // tiles of 64 and 141 of 32, 4096 samples 111 and 98.
  int run_pass(const PassArgs &a) {
    return a.n <= 152 * PassTile<2>::kSamples ? run_tiles<2>(a) : run_tiles<4>(a);
  }
  template <int R>
  int run_tiles(const PassArgs &a) {
    const int tiles = (a.n + PassTile<R>::kSamples - 1) / PassTile<R>::kSamples;
    lck(cudaFuncSetAttribute(k_ml_pass<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)PassTile<R>::kSmem),
        "attribute");
    k_ml_pass<R><<<tiles, kPassThreads, PassTile<R>::kSmem, st_>>>(a);
    return tiles;
  }

  void forward_backward(const float *X, const float *y, int n, double *loss) {
    PassArgs a{};
    a.X = X;
    a.y = y;
    a.n = n;
    a.p = params_.as<float>();
    a.pT = pT_.as<float>();
    a.H1 = H1_.as<float>(); a.H2 = H2_.as<float>();
    a.D1 = D1_.as<float>(); a.D2 = D2_.as<float>(); a.D3 = D3_.as<float>();
    a.part = bpart_.as<float>();
    a.loss = lpart_.as<double>();
    const int tiles = run_pass(a);
    // as many slices as fill the SMs with the two large gradients, of at least 64 samples
    const int want = std::max(1, std::min(kGradSlices, n / 64));
    const int per = ((n + want - 1) / want + kGradK - 1) / kGradK * kGradK, slices = (n + per - 1) / per;
    const WgradArgs w{X, a.H1, a.H2, a.D1, a.D2, a.D3, n, per, wpart_.as<float>()};
    k_ml_wgrad<<<dim3(slices, 3), 256, 0, st_>>>(w);
    k_ml_grad<<<(kMlParams + 31) / 32 + 1, 256, 0, st_>>>(wpart_.as<float>(), slices, bpart_.as<float>(),
                                                            lpart_.as<double>(), tiles, n, grad_.as<float>(), loss);
    lck(cudaGetLastError(), "training pass");
  }

  void upload_weight_tiles() {
    if (!weights_dirty_) return;
    std::vector<float> p(kMlParams);
    get_params(p.data());
    std::vector<uint8_t> w(kWBytes, 0);
    auto put = [&](size_t base, int o, int k, float x) {
      const uint16_t b = host_bf16(x);
      std::memcpy(&w[base + host_cm_off(o, k)], &b, 2);
    };
    for (int o = 0; o < kMlW; ++o) {
      for (int k = 0; k < kMlIn; ++k) put(0, o, k, p[kMlOffW1 + o * kMlIn + k]);
      for (int k = 0; k < kMlW; ++k) {
        put(kWTile, o, k, p[kMlOffW2 + o * kMlW + k]);
        put(3 * kWTile, o, k, p[kMlOffW3 + o * kMlW + k]);
      }
    }
    lck(cudaMemcpyAsync(wt_.p, w.data(), kWBytes, cudaMemcpyHostToDevice, st_), "weight tiles");
    lck(cudaStreamSynchronize(st_), "weight tiles");  // read on the engine's stream
    weights_dirty_ = false;
  }

  void run_infer(const InferArgs &a, cudaStream_t st) {
    if (a.ntiles <= 0) return;
    int sms = 0;
    lck(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device_), "attribute");
    lck(cudaFuncSetAttribute(k_ml_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInferSmem), "attribute");
    k_ml_infer<<<std::min(a.ntiles, std::max(sms, 1)), 128, kInferSmem, st>>>(a);
    lck(cudaGetLastError(), "inference launch");
    int err = 0;
    lck(cudaMemcpyAsync(&err, err_.p, 4, cudaMemcpyDeviceToHost, st), "copy");
    lck(cudaStreamSynchronize(st), "inference");
    if (err) {
      cudaMemset(err_.p, 0, 4);
      throw EngineError(2, "tensor-core inference timed out on an mbarrier wait");
    }
  }

  static constexpr int kGradSlices = 76;
  static constexpr size_t kGradLoss = (kMlParams * 4 + 7) / 8 * 8;  // byte offset of the loss behind the gradient
  int device_ = 0;
  cudaStream_t st_ = nullptr;
  LBuf params_, pT_, m_, v_, grad_, wt_, err_;
  LBuf H1_, H2_, D1_, D2_, D3_, bpart_, wpart_, lpart_, ioX_, ioy_;
  char *host_grad_ = nullptr;  // page-locked: gradient and loss of loss_grad, parameters of set_params
  int cap_ = 0, io_cap_ = 0;
  std::mutex io_mutex_;  // calls that share ioX_, ioy_ and host_grad_, one at a time
  int64_t t_ = 0;
  bool weights_dirty_ = true;
  std::vector<Chunk> data_;
  LBuf prior_;
  int64_t prior_n_ = 0;
  bool has_prior_ = false;
  float yscale_ = 0.0f;  // RMS of the training targets (0: not measured yet)
  bool folded_ = false;  // the output layer is in the targets' units
};

}  // namespace

std::unique_ptr<ILearner> make_learner(int device, uint64_t seed) { return std::make_unique<Learner>(device, seed); }

}  // namespace ccx
