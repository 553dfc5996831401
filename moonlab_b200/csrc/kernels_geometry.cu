// kernels_geometry.cu -- Gram matrix of a batch of complex128 states in FP64,
// G[a][b] = sum_x conj(S_a[x]) S_b[x] for a <= b: the inner products the
// quantum geometric tensor is assembled from (adjoint.cpp,
// mlb_hea_geometry).
//
// The B x B upper triangle is cut into 32 x 32 tile pairs (ta <= tb); the
// amplitude axis into K chunks.  One CTA of four warps takes one (pair,
// chunk): 16 amplitudes of the pair's 32 + 32 rows at a time come to shared
// memory by cp.async, the next 16 during the products.  A warp forms a
// 16 x 16 block with mma.sync m8n8k4 f64: a row of complex numbers is a row of
// twice as many reals, Re conj(x) y = (xr, xi) . (yr, yi) and
// Im = (xr, xi) . (yi, -yr), so of three fragments of doubles (x, y and y with
// its pairs swapped) eight products of 256 multiply-adds are made; the row
// pitch of 36 doubles puts a fragment's four rows on distinct banks.
// Per-chunk partials are then summed in chunk order by a second kernel, so
// the result does not depend on scheduling.
// Bound: FP64.  With 2 x 2 blocks a thread on the CUDA cores, four 16-byte
// shared loads fed 16 multiply-adds and bound the kernel: 373 us for 181
// states of 15 qubits; the geometry call around it went from 966 to 810 us.
#include <vector>

#include "kernels_common.cuh"
#include "mlb_internal.h"

namespace mlb {

namespace {

constexpr int kGT = 32;           // rows per tile
constexpr int kGK = 16;           // amplitudes per shared-memory step
constexpr int kGP = 2 * kGK + 4;  // doubles a row in shared memory

__device__ __forceinline__ void dmma(double (&d)[2], double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d[0]), "+d"(d[1])
               : "d"(a), "d"(b));
}

__global__ void __launch_bounds__(128) k_gram_partial(const double2* __restrict__ S, uint64_t dim, int B,
                                                         const int2* __restrict__ pairs, int npairs,
                                                         uint64_t kchunk, double2* __restrict__ part) {
  __shared__ __align__(16) double buf[2][2 * kGT][kGP];  // [step parity][x rows, y rows]
  const int2 pr = pairs[blockIdx.x];
  const int a0 = pr.x * kGT, b0 = pr.y * kGT;
  const uint64_t k0 = (uint64_t)blockIdx.y * kchunk;
  const uint64_t k1 = k0 + kchunk < dim ? k0 + kchunk : dim;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int c = threadIdx.x % kGK, r0 = threadIdx.x / kGK;  // copies amplitude c of rows r0, r0 + 8, ...
  auto fetch = [&](uint64_t k, int to) {
#pragma unroll
    for (int r = r0; r < 2 * kGT; r += 128 / kGK) {
      const int row = r < kGT ? a0 + r : b0 + r - kGT;
      const bool in = row < B && k + c < k1;  // else zeros
      const double2* src = S + (in ? (uint64_t)row * dim + k + c : 0);
      asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(
                       static_cast<uint32_t>(__cvta_generic_to_shared(&buf[to][r][2 * c]))),
                   "l"(src), "r"(in ? 16 : 0)
                   : "memory");
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
  };
  // fragments: lane l holds x[l >> 2][l & 3], y[l & 3][l >> 2] and out[l >> 2][2 (l & 3) + {0, 1}]
  const int fr = lane >> 2, fk = lane & 3;
  const int xr = 16 * (warp >> 1) + fr, yr = kGT + 16 * (warp & 1) + fr;
  const int flip = (fk & 1) << 31;
  double re[2][2][2] = {}, im[2][2][2] = {};
  fetch(k0, 0);
  int at = 0;
  for (uint64_t k = k0; k < k1; k += kGK, at ^= 1) {
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if (k + kGK < k1) fetch(k + kGK, at ^ 1);
#pragma unroll
    for (int t = 0; t < 2 * kGK; t += 4) {
      double x[2], y[2], z[2];
#pragma unroll
      for (int i = 0; i < 2; i++) {
        x[i] = buf[at][xr + 8 * i][t + fk];
        y[i] = buf[at][yr + 8 * i][t + fk];
        const double w = buf[at][yr + 8 * i][t + (fk ^ 1)];
        z[i] = __hiloint2double(__double2hiint(w) ^ flip, __double2loint(w));
      }
#pragma unroll
      for (int i = 0; i < 2; i++)
#pragma unroll
        for (int j = 0; j < 2; j++) {
          dmma(re[i][j], x[i], y[j]);
          dmma(im[i][j], x[i], z[j]);
        }
    }
  }
  double2* out = part + ((size_t)blockIdx.y * npairs + blockIdx.x) * (kGT * kGT);
#pragma unroll
  for (int i = 0; i < 2; i++)
#pragma unroll
    for (int j = 0; j < 2; j++)
#pragma unroll
      for (int q = 0; q < 2; q++)
        out[(xr + 8 * i) * kGT + yr - kGT - fr + 8 * j + 2 * fk + q] = make_double2(re[i][j][q], im[i][j][q]);
}

// G[a][b] (a <= b, both < B) = sum over chunks, in chunk order.
__global__ void __launch_bounds__(128) k_gram_reduce(const double2* __restrict__ part, const int2* __restrict__ pairs,
                                                     int npairs, int nchunks, int B, double2* __restrict__ G) {
  const int p = blockIdx.x, e = blockIdx.y * 128 + threadIdx.x;
  const int2 pr = pairs[p];
  const int a = pr.x * kGT + e / kGT, b = pr.y * kGT + e % kGT;
  if (a >= B || b >= B || a > b) return;
  double2 s = make_double2(0.0, 0.0);
#pragma unroll 8
  for (int c = 0; c < nchunks; c++) {
    const double2 v = part[((size_t)c * npairs + p) * (kGT * kGT) + e];
    s.x += v.x;
    s.y += v.y;
  }
  G[(size_t)a * B + b] = s;
}

// Launch geometry of one Gram computation: tile pairs, K chunks (about four
// CTAs per SM in all) and the chunk length in amplitudes (a multiple of kGK).
struct GramGeo {
  int npairs;
  uint64_t nchunks, kchunk;
  size_t pairs_bytes;  // the pair table, padded to 256 bytes
};
GramGeo gram_geo(int B, uint64_t dim, int num_sms) {
  GramGeo g;
  const int T = (B + kGT - 1) / kGT;
  g.npairs = T * (T + 1) / 2;
  const uint64_t steps = (dim + kGK - 1) / kGK;
  uint64_t nchunks = (uint64_t)(4 * num_sms + g.npairs - 1) / (uint64_t)g.npairs;
  if (nchunks < 1) nchunks = 1;
  if (nchunks > steps) nchunks = steps;
  g.kchunk = ((steps + nchunks - 1) / nchunks) * kGK;
  g.nchunks = (dim + g.kchunk - 1) / g.kchunk;
  g.pairs_bytes = (sizeof(int2) * (size_t)g.npairs + 255) / 256 * 256;
  return g;
}

}  // namespace

size_t gram_scratch_bytes(int B, uint64_t dim, int num_sms) {
  const GramGeo g = gram_geo(B, dim, num_sms);
  return g.pairs_bytes + sizeof(double2) * (size_t)g.nchunks * g.npairs * kGT * kGT;
}

int launch_gram(const void* states, uint64_t dim, int B, double2* d_G, void* d_scratch, int num_sms,
                cudaStream_t stream) {
  if (B < 1 || dim < 1) return MLB_ERR_INVALID_ARG;
  const GramGeo g = gram_geo(B, dim, num_sms);
  const int T = (B + kGT - 1) / kGT;
  const int npairs = g.npairs;
  const uint64_t kchunk = g.kchunk, nchunks = g.nchunks;
  // tile-pair table at the start of the scratch (256-byte padded), partials after it
  int2* d_pairs = static_cast<int2*>(d_scratch);
  double2* d_part = reinterpret_cast<double2*>(static_cast<unsigned char*>(d_scratch) + g.pairs_bytes);
  std::vector<int2> pairs;
  pairs.reserve(npairs);
  for (int a = 0; a < T; a++)
    for (int b = a; b < T; b++) pairs.push_back(make_int2(a, b));
  if (cudaMemcpyAsync(d_pairs, pairs.data(), sizeof(int2) * pairs.size(), cudaMemcpyHostToDevice, stream) !=
      cudaSuccess)
    return MLB_ERR_DRIVER;
  dim3 grid((unsigned)npairs, (unsigned)nchunks);
  k_gram_partial<<<grid, 128, 0, stream>>>(static_cast<const double2*>(states), dim, B, d_pairs, npairs, kchunk,
                                           d_part);
  k_gram_reduce<<<dim3((unsigned)npairs, kGT * kGT / 128), 128, 0, stream>>>(d_part, d_pairs, npairs, (int)nchunks, B, d_G);
  count_launch(2);
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

}  // namespace mlb
