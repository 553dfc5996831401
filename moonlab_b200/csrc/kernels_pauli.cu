// kernels_pauli.cu -- sums of Pauli strings in tile passes over linear
// subspaces of the index space (planned by pauli_plan.h).
//
//   k_pauli_sum   : partials of sum_k c_k <psi|P_k|psi>, one per CTA; the last
//                   CTA of the last pass adds them up.
//   k_pauli_apply : lambda (+)= sum_k c_k P_k psi for a batch of states; the
//                   last pass also emits the per-tile partial of
//                   Re<psi|lambda> (the energy).
//
// A tile holds both amplitudes of every pair of its strings, whatever qubits
// they touch: its basis is the strings' X masks beside the low unit vectors.
// The 16-byte units of a tile come by cp.async, all in flight at once.  A
// thread keeps 8 amplitudes per segment in registers along three masks, so
// one shared-memory read serves up to 7 masks, and the strings' signs are
// one bit pattern over the register index, one functional of the group
// index and one sign per tile (folded into the coefficient table).
// Bound: HBM for few strings; the FP64 products (two or three multiply-adds
// per pair and string) and their issue for many.  Two CTAs per SM overlap
// one's copies with the other's sums.
// Measured: norm, <Z>, 58 random one- and two-local strings and 4096 samples
// of a 29-qubit complex128 state 68.1 -> 28.6 ms (one pass over the state per
// distinct X mask before, three passes for all of them now), 22.1 ms with two
// groups per thread and a routine per kind of string; lambda = H psi
// of 80 strings on 256 states of 20 qubits: the whole gradient 134 -> 107 ms.
#include "kernels_common.cuh"
#include "mlb_internal.h"

namespace mlb {

namespace {

constexpr int kThreads = 256;       // two CTAs per SM: 16 warps at 128 registers
constexpr int kMaxUnitSteps = 64;  // units of a tile per thread

__device__ __forceinline__ double flip_sign(double c, uint32_t bit) {  // bit in 0/1
  return __hiloint2double(__double2hiint(c) ^ (int)(bit << 31), __double2loint(c));
}

// A tile's index offsets: unit tid + j NT adds toff ^ joff[j] to the base.
template <int NT, int UB>
struct UnitOffsets {
  static_assert(NT == 256, "eight thread bits");
  uint64_t toff;
  __device__ __forceinline__ void init(const PauliPass& P, uint64_t* joff) {
    constexpr int TB = 8;
    for (uint32_t j = threadIdx.x; j < kMaxUnitSteps; j += NT) {
      uint64_t off = 0;
#pragma unroll
      for (int b = TB; b < kMaxPauliBits - UB; b++)
        if (b + UB < P.m && (j >> (b - TB) & 1u)) off ^= P.basis[b + UB];
      joff[j] = off;
    }
    toff = 0;
#pragma unroll
    for (int b = 0; b < TB; b++)
      if (b + UB < P.m && (threadIdx.x >> b & 1u)) toff ^= P.basis[b + UB];
  }
};

// Byte offset of group gi in the tile: tid's bits here, the loop's by the caller.
template <int TB>
__device__ __forceinline__ uint32_t group_lane_offset(const PauliSeg& s) {
  uint32_t off = 0;
#pragma unroll
  for (int q = 0; q < TB; q++)
    if (threadIdx.x >> q & 1u) off ^= s.kappa[q];
  return off;
}
template <int TB>
__device__ __forceinline__ uint32_t group_step_offset(const PauliSeg& s, uint32_t g0) {
  uint32_t off = 0;
#pragma unroll
  for (int q = TB; q < kMaxPauliBits - 3; q++)
    if (g0 >> q & 1u) off ^= s.kappa[q];
  return off;
}

// Keeps products of the amplitudes inside the loop over strings: they are the
// same for every string of a mask, and hoisted ones would spill.
__device__ __forceinline__ void opaque(double2 (&v)[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) asm volatile("" : "+d"(v[k].x), "+d"(v[k].y));
}
__device__ __forceinline__ void opaque(float2 (&v)[8]) {
#pragma unroll
  for (int k = 0; k < 8; k++) asm volatile("" : "+f"(v[k].x), "+f"(v[k].y));
}

// One string on two groups of 8 amplitudes: acc += sum over its pairs of
// +-c times the real (ODD: imaginary) part.  KAP: its X mask among the
// segment's directions, 0: its diagonal.
template <typename A, int KAP, bool ODD>
__device__ __forceinline__ void pairs(const A (&v)[2][8], const double (&c)[2], uint32_t pat, double (&acc)[2]) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (k & (KAP & -KAP)) continue;  // the member without the lowest mask bit
#pragma unroll
    for (int g = 0; g < 2; g++) {
      const double ix = v[g][k].x, iy = v[g][k].y, px = v[g][k ^ KAP].x, py = v[g][k ^ KAP].y;
      const double x = ODD ? px * iy - py * ix : px * ix + py * iy;
      acc[g] = fma(flip_sign(c[g], pat >> k & 1u), x, acc[g]);
    }
  }
}

template <typename Real>
__global__ void __launch_bounds__(kThreads, 2)
    k_pauli_sum(const typename Cplx<Real>::T* __restrict__ amp, const __grid_constant__ PauliPass P,
                const PauliSeg* __restrict__ segs, const PauliTerm* __restrict__ terms,
                double* partials, int before, unsigned* done, double* __restrict__ out) {
  using A = typename Cplx<Real>::T;
  constexpr int NT = kThreads, UB = sizeof(A) == 16 ? 0 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t joff[kMaxUnitSteps];
  __shared__ double red[NT / 32];
  __shared__ bool last;
  const uint32_t tile_bytes = (uint32_t)sizeof(A) << P.m;
  double* coef = reinterpret_cast<double*>(smem + tile_bytes);       // [term] with the tile's sign
  PauliTerm* st = reinterpret_cast<PauliTerm*>(coef + P.num_terms);
  PauliSeg* ss = reinterpret_cast<PauliSeg*>(st + P.num_terms);
  const int tid = threadIdx.x;
  for (int i = tid; i < P.num_terms * (int)(sizeof(PauliTerm) / 4); i += NT)
    reinterpret_cast<uint32_t*>(st)[i] = reinterpret_cast<const uint32_t*>(terms)[i];
  for (int i = tid; i < P.num_segs * (int)(sizeof(PauliSeg) / 4); i += NT)
    reinterpret_cast<uint32_t*>(ss)[i] = reinterpret_cast<const uint32_t*>(segs)[i];
  UnitOffsets<NT, UB> uo;
  uo.init(P, joff);
  const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const uint32_t units = 1u << (P.m - UB), groups = 1u << (P.m - 3);
  __syncthreads();
  double acc[2] = {0.0, 0.0};
  for (uint64_t tile = blockIdx.x; tile < P.tiles_per_state; tile += gridDim.x) {
    const uint64_t base = pdep64(tile, P.free_mask);
    for (uint32_t u = tid, j = 0; u < units; u += NT, j++)
      cp_async16(sm0 + tile_swz16(u) * 16u, amp + (base ^ uo.toff ^ joff[j]));
    for (int t = tid; t < P.num_terms; t += NT) coef[t] = flip_sign(st[t].c, __popcll(st[t].z & base) & 1);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    for (int s = 0; s < P.num_segs; s++) {
      const PauliSeg& sg = ss[s];
      const uint32_t a0 = sg.alpha[0], a1 = sg.alpha[1], a2 = sg.alpha[2];
      const uint32_t lane_off = group_lane_offset<8>(sg);
      for (uint32_t g0 = 0; g0 + tid < groups; g0 += 2 * NT) {
        const bool two = g0 + NT + tid < groups;
        const uint32_t off = lane_off ^ group_step_offset<8>(sg, g0);
        const uint32_t off1 = two ? lane_off ^ group_step_offset<8>(sg, g0 + NT) : off;
        A v[2][8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint32_t ak = (k & 1 ? a0 : 0u) ^ (k & 2 ? a1 : 0u) ^ (k & 4 ? a2 : 0u);
          v[0][k] = *reinterpret_cast<const A*>(smem + (off ^ ak));
          v[1][k] = *reinterpret_cast<const A*>(smem + (off1 ^ ak));
        }
        uint32_t wn = *reinterpret_cast<const uint32_t*>(&st[sg.term_begin].zg);  // zg, kap, pat
        double cn = coef[sg.term_begin];
        for (int t = sg.term_begin; t < sg.term_end; t++) {
          const uint32_t w = wn, pat = w >> 24;
          const double ct = cn;
          const int tn = t + 1 < sg.term_end ? t + 1 : t;  // the next string's, while this one is summed
          wn = *reinterpret_cast<const uint32_t*>(&st[tn].zg);
          cn = coef[tn];
          const double c[2] = {flip_sign(ct, __popc(w & 0xffffu & (g0 + tid)) & 1),
                               two ? flip_sign(ct, __popc(w & 0xffffu & (g0 + NT + tid)) & 1) : 0.0};
          opaque(v[0]);
          opaque(v[1]);
          switch (w >> 16 & 15u) {
#define MLB_P(k) \
  case k: pairs<A, k & 7, (k > 7)>(v, c, pat, acc); break;
            MLB_P(0) MLB_P(1) MLB_P(2) MLB_P(3) MLB_P(4) MLB_P(5) MLB_P(6) MLB_P(7)
            MLB_P(9) MLB_P(10) MLB_P(11) MLB_P(12) MLB_P(13) MLB_P(14) MLB_P(15)
#undef MLB_P
          }
        }
      }
    }
    __syncthreads();
  }
  double sum = acc[0] + acc[1];
  for (int o = 16; o > 0; o >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, o);
  if ((tid & 31) == 0) red[tid >> 5] = sum;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int w = 0; w < NT / 32; w++) s += red[w];
    partials[before + blockIdx.x] = s;
    __threadfence();
    last = out && atomicAdd(done, 1u) == gridDim.x - 1;
  }
  if (!out) return;
  __syncthreads();
  if (!last) return;
  // the last pass's last CTA: all passes' partials, in a fixed order
  double v = 0.0;
  for (int i = tid; i < before + (int)gridDim.x; i += NT) v += __ldcg(partials + i);
  for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
  if ((tid & 31) == 0) red[tid >> 5] = v;
  __syncthreads();
  if (tid == 0) {
    double s = 0.0;
    for (int w = 0; w < NT / 32; w++) s += red[w];
    *out = s;
  }
}

// States of fewer than 8 amplitudes: a thread for every 32nd string, over the amplitudes in turn.
template <typename Real>
__global__ void k_pauli_tiny(const typename Cplx<Real>::T* __restrict__ amp, int n, int num_terms,
                             const uint64_t* __restrict__ xm, const uint64_t* __restrict__ zm,
                             const double* __restrict__ coeff, double* __restrict__ out) {
  double acc = 0.0;
  for (int t = threadIdx.x; t < num_terms; t += 32) {
    const int ny = __popcll(xm[t] & zm[t]) & 3;
    double v = 0.0;
    for (uint32_t i = 0; i < (1u << n); i++) {
      const auto a = amp[i], b = amp[i ^ (uint32_t)xm[t]];
      const double re = (double)b.x * a.x + (double)b.y * a.y, im = (double)b.x * a.y - (double)b.y * a.x;
      const double x = ny == 0 ? re : ny == 1 ? -im : ny == 2 ? -re : im;  // Re(i^ny conj(b) a)
      v += __popcll(i & zm[t]) & 1 ? -x : x;
    }
    acc += coeff[t] * v;
  }
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_down_sync(0xffffffffu, acc, o);
  if (threadIdx.x == 0) *out = acc;
}

// lambda[k] += +-c (ODD: times i) psi[k ^ KAP]; the sign is that of the source.
template <typename A, int KAP, bool ODD>
__device__ __forceinline__ void apply_string(const A (&v)[8], double2 (&l)[8], double c, uint32_t pat) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    const double cs = flip_sign(c, pat >> (k ^ KAP) & 1u);
    const double x = v[k ^ KAP].x, y = v[k ^ KAP].y;
    l[k].x = ODD ? fma(-cs, y, l[k].x) : fma(cs, x, l[k].x);
    l[k].y = ODD ? fma(cs, x, l[k].y) : fma(cs, y, l[k].y);
  }
}

// The tile of lambda is held in FP64 for both types and rounded to the
// state's type once, at its store.
template <typename Real>
__global__ void __launch_bounds__(kThreads, 2)
    k_pauli_apply(const typename Cplx<Real>::T* __restrict__ psi, typename Cplx<Real>::T* __restrict__ lam,
                  const __grid_constant__ PauliPass P, const PauliSeg* __restrict__ segs,
                  const PauliTerm* __restrict__ terms, int accumulate, double* __restrict__ energy_partials) {
  using A = typename Cplx<Real>::T;
  constexpr int NT = kThreads, UB = sizeof(A) == 16 ? 0 : 1;
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t joff[kMaxUnitSteps];
  __shared__ double red[NT / 32];
  const uint32_t tile_bytes = (uint32_t)sizeof(A) << P.m;
  unsigned char* ltile = smem + tile_bytes;  // [2^m] double2, at twice psi's offsets for complex64
  double* coef = reinterpret_cast<double*>(ltile + (16u << P.m));
  PauliTerm* st = reinterpret_cast<PauliTerm*>(coef + P.num_terms);
  PauliSeg* ss = reinterpret_cast<PauliSeg*>(st + P.num_terms);
  const int tid = threadIdx.x;
  for (int i = tid; i < P.num_terms * (int)(sizeof(PauliTerm) / 4); i += NT)
    reinterpret_cast<uint32_t*>(st)[i] = reinterpret_cast<const uint32_t*>(terms)[i];
  for (int i = tid; i < P.num_segs * (int)(sizeof(PauliSeg) / 4); i += NT)
    reinterpret_cast<uint32_t*>(ss)[i] = reinterpret_cast<const uint32_t*>(segs)[i];
  UnitOffsets<NT, UB> uo;
  uo.init(P, joff);
  const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  const uint32_t units = 1u << (P.m - UB), groups = 1u << (P.m - 3);
  __syncthreads();
  for (uint64_t tile = blockIdx.x; tile < P.num_tiles; tile += gridDim.x) {
    const uint64_t b = tile / P.tiles_per_state;
    const uint64_t base = pdep64(tile % P.tiles_per_state, P.free_mask);
    const A* gs = psi + (b << P.n);
    A* gl = lam + (b << P.n);
    for (uint32_t u = tid, j = 0; u < units; u += NT, j++) {
      const uint64_t off = base ^ uo.toff ^ joff[j];
      const uint32_t dst = tile_swz16(u) * 16u;
      cp_async16(sm0 + dst, gs + off);
      if constexpr (UB == 0) {
        if (accumulate) cp_async16(sm0 + tile_bytes + dst, gl + off);
        else *reinterpret_cast<double2*>(ltile + dst) = make_double2(0.0, 0.0);
      } else {
        float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
        if (accumulate) o = *reinterpret_cast<const float4*>(gl + off);
        *reinterpret_cast<double2*>(ltile + 2 * dst) = make_double2(o.x, o.y);
        *reinterpret_cast<double2*>(ltile + 2 * dst + 16) = make_double2(o.z, o.w);
      }
    }
    for (int t = tid; t < P.num_terms; t += NT) coef[t] = flip_sign(st[t].c, __popcll(st[t].z & base) & 1);
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    for (int s = 0; s < P.num_segs; s++) {
      const PauliSeg& sg = ss[s];
      const uint32_t a0 = sg.alpha[0], a1 = sg.alpha[1], a2 = sg.alpha[2];
      const uint32_t lane_off = group_lane_offset<8>(sg);
      for (uint32_t g0 = 0; g0 + tid < groups; g0 += NT) {
        const uint32_t off = lane_off ^ group_step_offset<8>(sg, g0);
        A v[8];
        double2 l[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
          const uint32_t at = off ^ (k & 1 ? a0 : 0u) ^ (k & 2 ? a1 : 0u) ^ (k & 4 ? a2 : 0u);
          v[k] = *reinterpret_cast<const A*>(smem + at);
          l[k] = *reinterpret_cast<const double2*>(ltile + (at << UB));
        }
        uint32_t wn = *reinterpret_cast<const uint32_t*>(&st[sg.term_begin].zg);  // zg, kap, pat
        double cn = coef[sg.term_begin];
        for (int t = sg.term_begin; t < sg.term_end; t++) {
          const uint32_t w = wn, pat = w >> 24;
          const double c = flip_sign(cn, __popc(w & 0xffffu & (g0 + tid)) & 1);
          const int tn = t + 1 < sg.term_end ? t + 1 : t;
          wn = *reinterpret_cast<const uint32_t*>(&st[tn].zg);
          cn = coef[tn];
          switch (w >> 16 & 15u) {
#define MLB_A(k) \
  case k: apply_string<A, k & 7, (k > 7)>(v, l, c, pat); break;
            MLB_A(0) MLB_A(1) MLB_A(2) MLB_A(3) MLB_A(4) MLB_A(5) MLB_A(6) MLB_A(7)
            MLB_A(9) MLB_A(10) MLB_A(11) MLB_A(12) MLB_A(13) MLB_A(14) MLB_A(15)
#undef MLB_A
          }
        }
#pragma unroll
        for (int k = 0; k < 8; k++)
          *reinterpret_cast<double2*>(ltile + ((off ^ (k & 1 ? a0 : 0u) ^ (k & 2 ? a1 : 0u) ^ (k & 4 ? a2 : 0u)) << UB)) = l[k];
      }
      __syncthreads();
    }
    double e_acc = 0.0;
    for (uint32_t u = tid, j = 0; u < units; u += NT, j++) {
      const uint64_t off = base ^ uo.toff ^ joff[j];
      const uint32_t at = tile_swz16(u) * 16u;
      if constexpr (UB == 0) {
        const double2 x = *reinterpret_cast<const double2*>(ltile + at);
        const double2 p = *reinterpret_cast<const double2*>(smem + at);
        gl[off] = x;
        e_acc += p.x * x.x + p.y * x.y;  // Re(conj(psi) lambda)
      } else {
        const double2 x = *reinterpret_cast<const double2*>(ltile + 2 * at);
        const double2 y = *reinterpret_cast<const double2*>(ltile + 2 * at + 16);
        const float4 p = *reinterpret_cast<const float4*>(smem + at);
        const float4 o = make_float4((float)x.x, (float)x.y, (float)y.x, (float)y.y);
        *reinterpret_cast<float4*>(gl + off) = o;
        e_acc += (double)p.x * o.x + (double)p.y * o.y;
        e_acc += (double)p.z * o.z + (double)p.w * o.w;
      }
    }
    if (energy_partials) {
      for (int o = 16; o > 0; o >>= 1) e_acc += __shfl_down_sync(0xffffffffu, e_acc, o);
      if ((tid & 31) == 0) red[tid >> 5] = e_acc;
      __syncthreads();
      if (tid == 0) {
        double s = 0.0;
        for (int w = 0; w < NT / 32; w++) s += red[w];
        energy_partials[tile] = s;
      }
    }
    __syncthreads();
  }
}

template <typename Real>
constexpr int tile_bits(bool apply) {
  return (sizeof(Real) == 8 ? 12 : 13) - (apply ? 1 : 0);
}

constexpr size_t tables_bytes(size_t terms, size_t segs) {
  return terms * (sizeof(double) + sizeof(PauliTerm)) + segs * sizeof(PauliSeg);
}
// every segment takes a string at least
constexpr size_t kMaxTables = tables_bytes(kMaxPauliTerms, kMaxPauliTerms);

template <typename Real>
int launch_sum_t(const void* amp, const PauliPass& P, const PauliSeg* d_segs, const PauliTerm* d_terms,
                 double* d_partials, int* parts, unsigned* d_done, double* d_out, int num_sms,
                 cudaStream_t stream) {
  using A = typename Cplx<Real>::T;
  const size_t smem = (sizeof(A) << P.m) + tables_bytes(P.num_terms, P.num_segs);
  auto kern = k_pauli_sum<Real>;
  static std::atomic<uint64_t> allowed{0};
  allow_shared(allowed, kern, (sizeof(A) << tile_bits<Real>(false)) + kMaxTables);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem);
  uint64_t grid = (uint64_t)num_sms * (per_sm < 1 ? 1 : per_sm > kPauliCtasPerSm ? kPauliCtasPerSm : per_sm);
  if (grid > P.tiles_per_state) grid = P.tiles_per_state;
  kern<<<(unsigned)grid, kThreads, smem, stream>>>((const A*)amp, P, d_segs, d_terms, d_partials, *parts, d_done, d_out);
  count_launch();
  *parts += (int)grid;
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

template <typename Real>
int launch_apply_t(const void* psi, void* lam, const PauliPass& P, const PauliSeg* d_segs, const PauliTerm* d_terms,
                   bool accumulate, double* d_epart, int num_sms, cudaStream_t stream) {
  using A = typename Cplx<Real>::T;
  const size_t smem = ((sizeof(A) + 16) << P.m) + tables_bytes(P.num_terms, P.num_segs);
  auto kern = k_pauli_apply<Real>;
  static std::atomic<uint64_t> allowed{0};
  allow_shared(allowed, kern, ((sizeof(A) + 16) << tile_bits<Real>(true)) + kMaxTables);
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kThreads, smem);
  uint64_t grid = (uint64_t)num_sms * (per_sm < 1 ? 1 : per_sm);
  if (grid > P.num_tiles) grid = P.num_tiles;
  kern<<<(unsigned)grid, kThreads, smem, stream>>>((const A*)psi, (A*)lam, P, d_segs, d_terms,
                                                        accumulate ? 1 : 0, d_epart);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

}  // namespace

int pauli_tile_bits(int dtype, bool apply) {
  return dtype == MLB_C128 ? tile_bits<double>(apply) : tile_bits<float>(apply);
}

int launch_pauli_sum(int dtype, const void* amp, const PauliPass& P, const PauliSeg* d_segs,
                     const PauliTerm* d_terms, double* d_partials, int* parts, unsigned* d_done, double* d_out,
                     int num_sms, cudaStream_t stream) {
  if (P.m < 3 || P.m > pauli_tile_bits(dtype, false) || P.num_terms < 1 || P.num_terms > kMaxPauliTerms ||
      P.num_segs > P.num_terms)
    return MLB_ERR_INVALID_ARG;
  return dtype == MLB_C128 ? launch_sum_t<double>(amp, P, d_segs, d_terms, d_partials, parts, d_done, d_out, num_sms, stream)
                           : launch_sum_t<float>(amp, P, d_segs, d_terms, d_partials, parts, d_done, d_out, num_sms, stream);
}

int launch_pauli_tiny(int dtype, const void* amp, int n, int num_terms, const uint64_t* d_xm, const uint64_t* d_zm,
                      const double* d_coeff, double* d_out, cudaStream_t stream) {
  if (n > 2) return MLB_ERR_INVALID_ARG;
  if (dtype == MLB_C128)
    k_pauli_tiny<double><<<1, 32, 0, stream>>>((const double2*)amp, n, num_terms, d_xm, d_zm, d_coeff, d_out);
  else
    k_pauli_tiny<float><<<1, 32, 0, stream>>>((const float2*)amp, n, num_terms, d_xm, d_zm, d_coeff, d_out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_pauli_apply(int dtype, const void* psi, void* lam, const PauliPass& P, const PauliSeg* d_segs,
                       const PauliTerm* d_terms, bool accumulate, double* d_epart, int num_sms,
                       cudaStream_t stream) {
  if (P.m < 3 || P.m > pauli_tile_bits(dtype, true) || P.num_terms < 1 || P.num_terms > kMaxPauliTerms ||
      P.num_segs > P.num_terms)
    return MLB_ERR_INVALID_ARG;
  return dtype == MLB_C128
             ? launch_apply_t<double>(psi, lam, P, d_segs, d_terms, accumulate, d_epart, num_sms, stream)
             : launch_apply_t<float>(psi, lam, P, d_segs, d_terms, accumulate, d_epart, num_sms, stream);
}

}  // namespace mlb
