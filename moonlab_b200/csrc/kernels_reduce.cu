// kernels_reduce.cu -- FP64 reductions in one HBM pass.
//
// probs_z: the norm and P(qubit=1) for every qubit from a single read of the
// state (the reference makes one full pass per qubit, measurement.c:73).
// A CTA walks chunks of 2^13 contiguous amplitudes; in a chunk thread t
// reads amplitudes t + 256 k (k < 32), so the low 8 index bits are the
// thread's own (constant), bits 8..12 are the loop counter (compile-time
// after unrolling) and bits >= 13 are the chunk index (constant per chunk).
// Per amplitude that costs one |a|^2 and ~2.5 FP64 adds; lane b of a CTA's
// first warp adds a chunk's total to the sum of bit 13 + b.  A second kernel
// folds the CTAs' sums.
// All reductions use a fixed order, so results are identical run to run.
#include <algorithm>
#include <atomic>
#include <mutex>

#include "kernels_common.cuh"
#include "hypot_glibc.cuh"
#include "mlb_internal.h"

namespace mlb {

namespace {

constexpr int kRT = 256;        // threads per CTA
constexpr int kRK = 32;         // amplitudes per thread per chunk
constexpr int kChunkBits = 13;  // 2^13 amplitudes per chunk
constexpr int kSums = 1 + 34;    // a CTA's sums: the total, then every bit's

template <typename A> __device__ __forceinline__ double norm2(const A& a) {
  const double x = (double)a.x, y = (double)a.y;
  return x * x + y * y;
}

__device__ __forceinline__ double block_sum(double v, double* red) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  double r = 0.0;
  if (threadIdx.x == 0)
    for (int i = 0; i < (int)(blockDim.x >> 5); i++) r += red[i];
  return r;  // valid in thread 0
}

// Pass 1: every CTA's total and its sum for every bit.
template <typename Real>
__global__ void __launch_bounds__(kRT) k_probs_z_pass1(const typename Cplx<Real>::T* __restrict__ amp,
                                                       uint64_t num_chunks, uint32_t chunk_amps,
                                                       double* __restrict__ partials) {
  __shared__ double red[kRT / 32];
  double low_tot = 0.0;                 // this thread's total (its low bits are fixed)
  double mid[kChunkBits - 8] = {0, 0, 0, 0, 0};
  double high = 0.0;                    // first warp: the sum of bit 13 + lane
  for (uint64_t c = blockIdx.x; c < num_chunks; c += gridDim.x) {
    const uint64_t base = c << kChunkBits;
    double ctot = 0.0;
    if (chunk_amps == (1u << kChunkBits)) {
      double p[kRK];
#pragma unroll
      for (int k = 0; k < kRK; k++) p[k] = norm2(amp[base + threadIdx.x + (uint32_t)k * kRT]);
#pragma unroll
      for (int k = 0; k < kRK; k++) {
        ctot += p[k];
#pragma unroll
        for (int b = 0; b < kChunkBits - 8; b++)
          if (k >> b & 1) mid[b] += p[k];
      }
    } else {  // small state: a single partial chunk
      for (uint32_t e = threadIdx.x; e < chunk_amps; e += kRT) {
        const double p = norm2(amp[e]);
        ctot += p;
        const uint32_t k = e / kRT;
#pragma unroll
        for (int b = 0; b < kChunkBits - 8; b++)
          if (k >> b & 1) mid[b] += p;
      }
    }
    low_tot += ctot;
    double t = ctot;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o);
    __syncthreads();
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x < 32 && (c >> threadIdx.x & 1ull))
      for (int w = 0; w < kRT / 32; w++) high += red[w];
  }
  double* out = partials + (size_t)blockIdx.x * kSums;
  double v = block_sum(low_tot, red);
  if (threadIdx.x == 0) out[0] = v;
  for (int b = 0; b < 8; b++) {
    v = block_sum((threadIdx.x >> b & 1) ? low_tot : 0.0, red);
    if (threadIdx.x == 0) out[1 + b] = v;
  }
  for (int b = 0; b < kChunkBits - 8; b++) {
    v = block_sum(mid[b], red);
    if (threadIdx.x == 0) out[1 + 8 + b] = v;
  }
  if (threadIdx.x < kSums - 1 - kChunkBits) out[1 + kChunkBits + threadIdx.x] = high;
}

// Pass 2 (one CTA, a warp per sum): out[0..n) = P1, out[n] = norm.
__global__ void __launch_bounds__(kRT) k_probs_z_pass2(const double* __restrict__ partials, int num_parts, int n,
                                                       double* __restrict__ out) {
  for (int j = threadIdx.x >> 5; j <= n; j += kRT / 32) {
    double v = 0.0;
    for (int i = threadIdx.x & 31; i < num_parts; i += 32) v += partials[(size_t)i * kSums + j];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) out[j == 0 ? n : j - 1] = v;
  }
}

template <typename Real>
__global__ void k_probabilities(const typename Cplx<Real>::T* __restrict__ amp, uint64_t dim,
                                int rule, double* __restrict__ out) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += stride) {
    const auto a = amp[i];
    const double x = (double)a.x, y = (double)a.y;
    if (rule == 0) {
      const double h = glibc_cabs(x, y);
      out[i] = __dmul_rn(h, h);
    } else {
      out[i] = __fma_rn(x, x, __dmul_rn(y, y));  // fma(re, re, im*im), as the reference build
    }
  }
}

// amp *= factor where (i & zero_mask) == zero_val, else amp = 0.
// zero_mask = 0 scales everything.  Division mode (factor < 0 encodes
// "divide by -factor") reproduces quantum_measure's amp /= norm.
template <typename Real>
__global__ void k_scale(typename Cplx<Real>::T* __restrict__ amp, uint64_t dim, double factor,
                        uint64_t keep_mask, uint64_t keep_val) {
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  const bool divide = factor < 0.0;
  const double f = divide ? -factor : factor;
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < dim; i += stride) {
    auto a = amp[i];
    if ((i & keep_mask) != keep_val) {
      a.x = 0;
      a.y = 0;
    } else if (divide) {
      a.x = (Real)__ddiv_rn((double)a.x, f);
      a.y = (Real)__ddiv_rn((double)a.y, f);
    } else {
      a.x = (Real)__dmul_rn((double)a.x, f);
      a.y = (Real)__dmul_rn((double)a.y, f);
    }
    amp[i] = a;
  }
}

int rgrid(uint64_t items, int num_sms) {
  uint64_t g = (items + kRT - 1) / kRT;
  const uint64_t cap = (uint64_t)num_sms * 8;
  if (g > cap) g = cap;
  if (g < 1) g = 1;
  return (int)g;
}

}  // namespace

int launch_reduce_probs_z(int dtype, const void* amp, int n, double* d_out, double* d_partials,
                          int num_sms, cudaStream_t stream) {
  const uint64_t dim = 1ull << n;
  const uint64_t num_chunks = n >= kChunkBits ? dim >> kChunkBits : 1;
  const uint32_t chunk_amps = n >= kChunkBits ? (1u << kChunkBits) : (uint32_t)dim;
  int grid = (int)std::min<uint64_t>(num_chunks, (uint64_t)num_sms * 4);
  if (dtype == MLB_C128)
    k_probs_z_pass1<double><<<grid, kRT, 0, stream>>>((const double2*)amp, num_chunks, chunk_amps, d_partials);
  else
    k_probs_z_pass1<float><<<grid, kRT, 0, stream>>>((const float2*)amp, num_chunks, chunk_amps, d_partials);
  k_probs_z_pass2<<<1, kRT, 0, stream>>>(d_partials, grid, n, d_out);
  count_launch(2);
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_probabilities(int dtype, const void* amp, int n, int rule, double* d_out,
                         cudaStream_t stream) {
  const uint64_t dim = 1ull << n;
  const int grid = rgrid(dim, 148 * 4);
  if (dtype == MLB_C128)
    k_probabilities<double><<<grid, kRT, 0, stream>>>((const double2*)amp, dim, rule, d_out);
  else
    k_probabilities<float><<<grid, kRT, 0, stream>>>((const float2*)amp, dim, rule, d_out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_scale(int dtype, void* amp, int n, double factor, uint64_t keep_mask, uint64_t keep_val,
                 cudaStream_t stream) {
  const uint64_t dim = 1ull << n;
  const int grid = rgrid(dim, 148 * 4);
  if (dtype == MLB_C128)
    k_scale<double><<<grid, kRT, 0, stream>>>((double2*)amp, dim, factor, keep_mask, keep_val);
  else
    k_scale<float><<<grid, kRT, 0, stream>>>((float2*)amp, dim, factor, keep_mask, keep_val);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

}  // namespace mlb

// ---- probs_z without device allocation -------------------------------------
// mlb_prob_one_all_noalloc runs the probs_z reduction above on caller-owned
// buffers, with its scratch in one fixed array per device instead of a
// cudaMalloc'd buffer.  Scratch use: pass-1 partials ([grid x 35] doubles,
// grid <= kNoAllocMaxParts).  Pass 1 writes every entry pass 2 reads, so
// nothing is cleared between calls.
namespace {

constexpr uint32_t kNoAllocMaxQubits = 30;
constexpr int kNoAllocMaxParts = 1024;  // pass-1 CTAs; the grid is min(chunks, 4 * SMs)
constexpr size_t kNoAllocScratchDoubles = (size_t)kNoAllocMaxParts * mlb::kSums;  // 35,840
constexpr int kNoAllocMaxDevices = 64;

static __device__ __align__(256) double g_probs_z_scratch[kNoAllocScratchDoubles];

struct NoAllocDevice {
  std::atomic<double*> scratch{nullptr};
  int num_sms = 0;
};
NoAllocDevice g_noalloc_dev[kNoAllocMaxDevices];
std::mutex g_noalloc_mu;

// Set-up, once per device, with that device current: the array's address and
// the SM count.
int noalloc_setup(int dev, double** scratch, int* num_sms) {
  NoAllocDevice& d = g_noalloc_dev[dev];
  double* p = d.scratch.load(std::memory_order_acquire);
  if (!p) {
    std::lock_guard<std::mutex> lk(g_noalloc_mu);
    p = d.scratch.load(std::memory_order_relaxed);
    if (!p) {
      int sms = 0;
      cudaError_t e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      if (e != cudaSuccess || sms <= 0)
        return mlb::record_error(MLB_ERR_DRIVER, "mlb_prob_one_all_noalloc: SM count query failed");
      void* addr = nullptr;
      e = cudaGetSymbolAddress(&addr, g_probs_z_scratch);
      if (e != cudaSuccess || !addr)
        return mlb::record_error(MLB_ERR_DRIVER, "mlb_prob_one_all_noalloc: scratch address lookup failed");
      d.num_sms = sms;
      p = (double*)addr;
      d.scratch.store(p, std::memory_order_release);
    }
  }
  *scratch = p;
  *num_sms = d.num_sms;
  return MLB_OK;
}

// True when ptr is device (or managed) memory of device dev.
bool on_device(const void* ptr, int dev) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, ptr) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return (a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged) && a.device == dev;
}

}  // namespace

extern "C" int mlb_prob_one_all_noalloc(const void* amp_device, int dtype, uint32_t num_qubits,
                                        double* out_device, void* stream) {
  if (!amp_device || !out_device)
    return mlb::record_error(MLB_ERR_INVALID_ARG, "mlb_prob_one_all_noalloc: null buffer");
  if (dtype != MLB_C128 && dtype != MLB_C64)
    return mlb::record_error(MLB_ERR_INVALID_ARG, "mlb_prob_one_all_noalloc: dtype must be MLB_C128 or MLB_C64");
  if (num_qubits < 1 || num_qubits > kNoAllocMaxQubits)
    return mlb::record_error(MLB_ERR_NUM_QUBITS,
                             "mlb_prob_one_all_noalloc: num_qubits must be 1..30 (fixed scratch size)");
  const uintptr_t align = dtype == MLB_C128 ? 16 : 8;
  if ((uintptr_t)amp_device % align || (uintptr_t)out_device % 8)
    return mlb::record_error(MLB_ERR_INVALID_ARG, "mlb_prob_one_all_noalloc: misaligned buffer");
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess) {
    cudaGetLastError();
    return mlb::record_error(MLB_ERR_NO_DEVICE, "mlb_prob_one_all_noalloc: no current device");
  }
  if (dev < 0 || dev >= kNoAllocMaxDevices)
    return mlb::record_error(MLB_ERR_NOT_SUPPORTED, "mlb_prob_one_all_noalloc: device ordinal above 63");
  if (!on_device(amp_device, dev) || !on_device(out_device, dev))
    return mlb::record_error(MLB_ERR_INVALID_ARG,
                             "mlb_prob_one_all_noalloc: buffers must be device memory of the current device");
  double* scratch = nullptr;
  int num_sms = 0;
  int rc = noalloc_setup(dev, &scratch, &num_sms);
  if (rc) return rc;
  // grid = min(chunks, 4 * SMs) stays within the array's kNoAllocMaxParts CTAs.
  const int sms = std::min(num_sms, kNoAllocMaxParts / 4);
  rc = mlb::launch_reduce_probs_z(dtype, amp_device, (int)num_qubits, out_device, scratch, sms,
                                  (cudaStream_t)stream);
  if (rc) return mlb::record_error(rc, "mlb_prob_one_all_noalloc: launch failed");
  return MLB_OK;
}
