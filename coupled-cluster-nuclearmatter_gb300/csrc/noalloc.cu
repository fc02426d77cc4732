// ccd_energy_save on caller-owned device buffers, with no allocation at all.
//
// Some callers cannot allocate device memory: a host program that owns every device
// buffer through its own pool (the Fortran host keeps t2_ccm and vnn_hhpp in arrays it
// manages), or code running where an allocation would be an error.  For them this
// entry point evaluates E = 1/4 sum_ch sum_{ab,ij} T(ab,ij) V(ij,ab) directly on their
// buffers, in the reference's layout (ccm_energy.f90:4-71).  Its scratch -- one partial sum
// per block, some 5 KiB -- is the file-scope array g_energy_slots below, held by every GPU that
// loads the library until the process exits.
//
// Set-up: the first call in a CUDA context (with that context's device current) looks
// up the device address of g_energy_slots with cudaGetSymbolAddress; make that first
// call before any stream capture.  The address is cached with the context's unique id
// (cuCtxGetId), so a context that is destroyed and created again (cudaDeviceReset, a
// reset primary context, a caller's own context) is seen as new and its address is
// looked up again on its first call.  Every call in a context shares the one array and
// it keeps the last call's contents: each call rewrites every slot it reads, and calls
// whose work overlaps on the GPU race on it.
#include <cuda.h>
#include <cuda_runtime.h>

#include <mutex>

#include "ccx.h"
#include "engine.hpp"

namespace {

constexpr int kMaxChannels = 16384;  // of the interface; the kernel's work per channel is a scan entry
constexpr int kMaxDevices = 64;
constexpr int kEnergyBlocks = 304, kEnergyThreads = 256, kScan = 4 * kEnergyThreads;

struct __align__(16) EnergySlot {
  double re, im;  // partial sum of a block
};

static __device__ __align__(256) EnergySlot g_energy_slots[kEnergyBlocks];

// per device: the context the cached address belongs to, and the address
struct SlotCache {
  unsigned long long ctx_id = 0;
  EnergySlot *addr = nullptr;
};
SlotCache g_slot_cache[kMaxDevices];
std::mutex g_setup_mutex;

using CtxGetCurrentFn = CUresult (*)(CUcontext *);
using CtxGetIdFn = CUresult (*)(CUcontext, unsigned long long *);

// Unique id of the calling thread's current context, 0 if there is none yet.  The two
// driver functions are reached through the runtime, so the library needs no libcuda
// at link time.
unsigned long long current_context_id() {
  static CtxGetCurrentFn get_current = nullptr;
  static CtxGetIdFn get_id = nullptr;
  if (!get_current || !get_id) {
    void *f0 = nullptr, *f1 = nullptr;
    cudaDriverEntryPointQueryResult q0 = cudaDriverEntryPointSymbolNotFound, q1 = q0;
    if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &f0, 12000, cudaEnableDefault, &q0) != cudaSuccess ||
        cudaGetDriverEntryPointByVersion("cuCtxGetId", &f1, 12000, cudaEnableDefault, &q1) != cudaSuccess ||
        q0 != cudaDriverEntryPointSuccess || q1 != cudaDriverEntryPointSuccess || !f0 || !f1)
      return 0;
    get_current = (CtxGetCurrentFn)f0;
    get_id = (CtxGetIdFn)f1;
  }
  CUcontext ctx = nullptr;
  unsigned long long id = 0;
  if (get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
  return id;
}

// Partial sums of T(ab,ij) V(ij,ab), T (n_pp x n_hh) and V (n_hh x n_pp) of every channel.
//
// The sizes are on the device only, so the grid is fixed and every block finds the work by a
// scan of dims, kScan channels at a time.  A warp's task is 32 ab by up to 8 ij of a channel:
// its lanes read T along ab, and each its own 128-byte run of V, all sixteen loads in flight
// at once.  One block per channel behind a scan kernel of its own left 25 blocks with a strided
// V for a small lattice: 58 us a call at PNM 14 nmax=2 (1 MB of each), now 10.2; PNM 66 nmax=4
// (129 MB of each) 1212 to 75 us.
// blocks of the call in progress that have written their partial sum: every launch counts it
// round to 0 again
static __device__ unsigned g_energy_done;
__device__ __forceinline__ double2 energy_load(const double *p, bool vec) {
  if (vec) return *reinterpret_cast<const double2 *>(p);
  return make_double2(p[0], p[1]);
}
__global__ void __launch_bounds__(kEnergyThreads) k_noalloc_energy(int nch, const int *__restrict__ dims,
                                                                   const double *__restrict__ t2,
                                                                   const double *__restrict__ v, bool vec,
                                                                   EnergySlot *slots, double *__restrict__ energy) {
  __shared__ long long off[kScan];  // first element of each channel of the chunk
  __shared__ int task[kScan + 1];   // first task of each
  __shared__ long long wsum[kEnergyThreads / 32];
  __shared__ int wtask[kEnergyThreads / 32];
  const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
  const int w = wid * kEnergyBlocks + blockIdx.x;  // few tasks go to as many SMs
  constexpr int stride = kEnergyBlocks * (kEnergyThreads / 32);
  long long off0 = 0;  // elements of the chunks before
  int task0 = 0;       // and their tasks, modulo stride
  double re = 0.0, im = 0.0, re1 = 0.0, im1 = 0.0;  // two chains of each: even and odd ij
  for (int c0 = 0; c0 < nch; c0 += kScan) {
    long long ne[4], es = 0;
    int nt[4], ts = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int c = c0 + 4 * tid + q;
      const int nh = c < nch ? dims[2 * c] : 0, np = c < nch ? dims[2 * c + 1] : 0;
      ne[q] = es;
      nt[q] = ts;
      es += (long long)nh * np;
      ts += ((np + 31) / 32) * ((nh + 7) / 8);
    }
    // exclusive scan of the threads' totals
    long long ei = es;
    int ti = ts;
    for (int o = 1; o < 32; o <<= 1) {
      const long long a = __shfl_up_sync(0xffffffffu, ei, o);
      const int b = __shfl_up_sync(0xffffffffu, ti, o);
      if (lane >= o) { ei += a; ti += b; }
    }
    __syncthreads();  // the previous chunk's tables are no longer read
    if (lane == 31) { wsum[wid] = ei; wtask[wid] = ti; }
    __syncthreads();
    long long eb = 0, et = 0;
    int tb = 0, tt = 0;
#pragma unroll
    for (int k = 0; k < kEnergyThreads / 32; ++k) {
      if (k < wid) { eb += wsum[k]; tb += wtask[k]; }
      et += wsum[k];
      tt += wtask[k];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      off[4 * tid + q] = off0 + eb + ei - es + ne[q];
      task[4 * tid + q] = tb + ti - ts + nt[q];
    }
    if (tid == 0) task[kScan] = tt;
    __syncthreads();
    // the warp's tasks of this chunk: global task numbers w, w + stride, ...
    for (int g = w >= task0 ? w - task0 : w - task0 + stride; g < tt; g += stride) {
      int lo = 0, hi = min(kScan, nch - c0);  // task[lo] <= g < task[lo + 1]
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (task[mid] <= g) lo = mid;
        else hi = mid;
      }
      const long long nh = dims[2 * (c0 + lo)], np = dims[2 * (c0 + lo) + 1];
      const int njb = (int)((nh + 7) / 8), loc = g - task[lo];
      const long long ab = (long long)(loc / njb) * 32 + lane, ij0 = (long long)(loc % njb) * 8;
      const int nj = (int)min(8ll, nh - ij0);
      if (ab >= np) continue;
      const double *t = t2 + 2 * (off[lo] + ab + np * ij0), *x = v + 2 * (off[lo] + ij0 + nh * ab);
      double2 a[8], b[8];
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const bool live = j < nj;
        a[j] = live ? energy_load(t + 2 * np * j, vec) : make_double2(0.0, 0.0);
        b[j] = live ? energy_load(x + 2 * j, vec) : make_double2(0.0, 0.0);
      }
#pragma unroll
      for (int j = 0; j < 8; j += 2) {
        re = fma(a[j].x, b[j].x, fma(-a[j].y, b[j].y, re));
        im = fma(a[j].x, b[j].y, fma(a[j].y, b[j].x, im));
        re1 = fma(a[j + 1].x, b[j + 1].x, fma(-a[j + 1].y, b[j + 1].y, re1));
        im1 = fma(a[j + 1].x, b[j + 1].y, fma(a[j + 1].y, b[j + 1].x, im1));
      }
    }
    off0 += et;
    task0 = (int)(((long long)task0 + tt) % stride);
  }
  // The block's sum, halving the warps that add in each step: shuffles in every warp would
  // be five FP64 additions a value on all eight, on a pipe of two a clock.
  __shared__ double2 part[kEnergyThreads];
  part[tid] = make_double2(re + re1, im + im1);
  __syncthreads();
#pragma unroll
  for (int o = kEnergyThreads / 2; o >= 32; o >>= 1) {
    if (tid < o) {
      part[tid].x += part[tid + o].x;
      part[tid].y += part[tid + o].y;
    }
    __syncthreads();
  }
  if (wid == 0) {
    re = part[lane].x;
    im = part[lane].y;
    for (int o = 16; o > 0; o >>= 1) {
      re += __shfl_xor_sync(0xffffffffu, re, o);
      im += __shfl_xor_sync(0xffffffffu, im, o);
    }
  }
  __shared__ bool last;
  if (tid == 0) {
    __stcg(&slots[blockIdx.x].re, re);
    __stcg(&slots[blockIdx.x].im, im);
    __threadfence();
    last = atomicInc(&g_energy_done, kEnergyBlocks - 1) == kEnergyBlocks - 1;
  }
  __syncthreads();
  if (!last || wid) return;
  // the block that finished last: 1/4 of the partials' sum, in a fixed order
  __threadfence();
  re = im = 0.0;
  double2 got[(kEnergyBlocks + 31) / 32];  // every load in flight before the first addition
#pragma unroll
  for (int k = 0; k < (kEnergyBlocks + 31) / 32; ++k) {
    const int c = lane + 32 * k;
    got[k] = c < kEnergyBlocks ? __ldcg(reinterpret_cast<const double2 *>(&slots[c].re)) : make_double2(0.0, 0.0);
  }
#pragma unroll
  for (int k = 0; k < (kEnergyBlocks + 31) / 32; ++k) {
    re += got[k].x;
    im += got[k].y;
  }
  for (int o = 16; o > 0; o >>= 1) {
    re += __shfl_xor_sync(0xffffffffu, re, o);
    im += __shfl_xor_sync(0xffffffffu, im, o);
  }
  if (lane == 0) {
    energy[0] = 0.25 * re;
    energy[1] = 0.25 * im;
  }
}

}  // namespace

extern "C" int ccx_ccd_energy_noalloc(int32_t nch, const int32_t *dims, const double *t2, const double *vhhpp,
                                      double *energy, void *stream) {
  if (nch < 1 || !dims || !t2 || !vhhpp || !energy) {
    ccx::set_last_error("ccx_ccd_energy_noalloc: null pointer or nch < 1");
    return CCX_EINVAL;
  }
  if (nch > kMaxChannels) {
    ccx::set_last_error("ccx_ccd_energy_noalloc: more than 16384 channels");
    return CCX_EINVAL;
  }
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) {
    ccx::set_last_error("ccx_ccd_energy_noalloc: no current CUDA device");
    return CCX_ENOGPU;
  }
  EnergySlot *slots = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_setup_mutex);
    SlotCache &c = g_slot_cache[dev];
    const unsigned long long id = current_context_id();
    if (id == 0 || id != c.ctx_id || !c.addr) {
      // first call in this context (or no context yet): look the address up; the
      // lookup creates the device's primary context if the thread has none
      void *p = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&p, g_energy_slots);
      if (e != cudaSuccess || !p) {
        ccx::set_last_error(cudaGetErrorString(e));
        return CCX_ECUDA;
      }
      c.addr = (EnergySlot *)p;
      c.ctx_id = current_context_id();
    }
    slots = c.addr;
  }
  cudaStream_t st = (cudaStream_t)stream;
  const bool vec = ((reinterpret_cast<uintptr_t>(t2) | reinterpret_cast<uintptr_t>(vhhpp)) & 15) == 0;
  k_noalloc_energy<<<kEnergyBlocks, kEnergyThreads, 0, st>>>(nch, dims, t2, vhhpp, vec, slots, energy);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    ccx::set_last_error(cudaGetErrorString(e));
    return CCX_ECUDA;
  }
  return CCX_OK;
}
