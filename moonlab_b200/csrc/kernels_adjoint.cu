// kernels_adjoint.cu -- batched adjoint gradient of a hardware-efficient
// ansatz energy E(theta) = <psi(theta)|H|psi(theta)>, H a sum of Pauli strings.
//
// The reference (differentiable.c:438-491, per Hamiltonian term) walks the
// gate tape backwards once per term, cloning states and taking one inner
// product per parameter.  The gradient is linear in the observable, so here
// lambda = H psi is formed once and a single backward sweep carries (psi,
// lambda) through the inverse gates:  dE/dtheta_p = Im<lambda|G_p|psi> at the
// point where both states stand just after gate p (G = Y for RY, Z for RZ).
//
// Batch layout: B parameter vectors give B states stored back to back,
// [B][2^N]; a tile never spans two batch elements, so every tile reads the
// cos/sin of its own theta (table cs[b][p], computed once per call).
//
// Kernels (all tile passes, one HBM read + write of each array per pass):
//   k_hea       : rotations on psi (forward) or on psi and lambda together
//                 with the per-parameter partial inner products (backward).
//   k_pauli_apply (kernels_pauli.cu): lambda = H psi and the per-tile
//                 partials of the energy.
//   k_hea_reduce, k_adj_energy: fixed-order sums of the partials
//                 (deterministic, and the same for every batch size).
//   k_unladder  : a complex64 batch from the index order of a layer boundary
//                 to the order after the last layer (hea_plan.h).
// Tiles come into shared memory by asynchronous copies, all in flight at
// once.
#include <vector>

#include "hea_plan.h"
#include "kernels_common.cuh"
#include "mlb_internal.h"

namespace mlb {

namespace {

constexpr int kUnladderBits = 11, kUnladderLow = 4;  // tile of k_unladder, contiguous bits of its rows

// ---------------------------------------------------------------------------
// rotation passes
// ---------------------------------------------------------------------------
// One tile per step and CTA: 2^m amplitudes base ^ span(basis), whose local
// index bits 0.. are contiguous amplitudes.  The 16-byte units of
// a tile (one complex128 or two complex64 amplitudes) come by cp.async, all
// in flight at once.  A segment's thread holds groups of 8 amplitudes whose
// register index is the segment's three target bits, so every rotation is
// compile-time code: no per-gate dispatch, no CNOTs (they are relabelling,
// hea_plan.h).  RZ's of a segment are one phase per register index, from a
// table per state; RY [[c, -s], [s, c]] is applied as c [[1, -t], [t, 1]]
// (t = s / c; c and s swap roles where |c| < |s|), two multiply-adds per
// component pair instead of four operations, and the product of the three
// scales is folded into the phases.
// Bound: shared memory (64 bytes per complex128 psi + lambda pair and segment,
// 0.5 clk per SM) and FP64 (about 30 operations, 0.47 clk) together; 64 KiB
// tiles, so three CTAs per SM overlap one's copies with the others' work.
// Measured, 20 qubits, 8 layers, 256 vectors with gradients: 616 ms by
// gate-by-gate passes with the CNOTs carried out (19 forward, 17 backward),
// 134 ms by these (6 and 9); complex64 326 -> 116 ms, and of 100 ms after
// lambda's passes 90 ms with values converted to FP64 once a segment.
template <typename Real, bool BACK> struct HeaCfg;
// Three CTAs of four warps, at 168 registers.  Two of eight warps at 128
// registers measured 8 % slower forward and 20 % slower backward in complex64.
template <> struct HeaCfg<double, false> { static constexpr int BITS = 12, NT = 128, CTAS = 3; };
template <> struct HeaCfg<double, true> { static constexpr int BITS = 11, NT = 128, CTAS = 3; };
template <> struct HeaCfg<float, false> { static constexpr int BITS = 13, NT = 128, CTAS = 3; };
template <> struct HeaCfg<float, true> { static constexpr int BITS = 12, NT = 128, CTAS = 3; };

// Per-state tables of a segment.
template <typename Real>
struct HeaTab {
  typename Cplx<Real>::T ph[4];  // scale * exp(-+ i ...) for register indexes 0 .. 3; 7 - k has the conjugate of k's
  Real t[3];                     // tangent, or cotangent where `flip`
  uint32_t flip;                 // bit i: rotation i uses the cotangent form
  double unscale;                // 1 / scale^2 (the gradients are taken on scaled states)
};

// v[k], v[k1] <- RY (forward) or its inverse (BACK), up to the scale.
template <typename A, typename Real, int RT, bool BACK>
__device__ __forceinline__ void hea_ry(A (&v)[8], Real t, bool flip) {
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (k & (1 << RT)) continue;
    const A a = v[k], b = v[k | (1 << RT)];
    const Real tt = BACK ? t : -t;
    if (!flip) {
      v[k] = {a.x + tt * b.x, a.y + tt * b.y};
      v[k | (1 << RT)] = {b.x - tt * a.x, b.y - tt * a.y};
    } else if (BACK) {
      v[k] = {t * a.x + b.x, t * a.y + b.y};
      v[k | (1 << RT)] = {t * b.x - a.x, t * b.y - a.y};
    } else {
      v[k] = {t * a.x - b.x, t * a.y - b.y};
      v[k | (1 << RT)] = {t * b.x + a.x, t * b.y + a.y};
    }
  }
}

// Im<lambda|Y|psi> over the pairs of register bit RT.
template <int RT>
__device__ __forceinline__ double hea_grad_y(const double2 (&v)[8], const double2 (&w)[8]) {
  double acc = 0.0;
#pragma unroll
  for (int k = 0; k < 8; k++) {
    if (k & (1 << RT)) continue;
    const double2 p0 = v[k], p1 = v[k | (1 << RT)], l0 = w[k], l1 = w[k | (1 << RT)];
    acc -= l0.x * p1.x + l0.y * p1.y;
    acc += l1.x * p0.x + l1.y * p0.y;
  }
  return acc;
}

// x times the phase of register index k (a constant): conj(ph[7 - k]) from 4 on.
template <typename A>
__device__ __forceinline__ A turn(const A (&ph)[4], int k, A x) {
  const A p = k < 4 ? ph[k] : ph[7 - k];
  return k < 4 ? A{p.x * x.x - p.y * x.y, p.x * x.y + p.y * x.x} : A{p.x * x.x + p.y * x.y, p.x * x.y - p.y * x.x};
}

// The arithmetic of a table's entries.  An entry multiplies 1/8 of all
// amplitudes, so its rounding does not average out over them: a complex128
// product is kept as hi + lo (lo the rounding of hi and first-order terms) and
// rounded once.  |psi|^2 - 1 after 8 layers on 12 qubits, rms of 64 vectors:
// 1.7e-15 with products of plain doubles, 6.9e-16 now (gate by gate 8.2e-16);
// the sweep takes as long.
struct Two {
  double hi, lo;
};
__device__ __forceinline__ Two times(Two a, Two b) {
  const double p = a.hi * b.hi;
  return {p, fma(a.hi, b.hi, -p) + (a.hi * b.lo + a.lo * b.hi)};
}
__device__ __forceinline__ Two plus(Two a, Two b) {
  const double s = a.hi + b.hi, t = s - a.hi;
  return {s, ((a.hi - (s - t)) + (b.hi - t)) + (a.lo + b.lo)};
}
__device__ __forceinline__ Two minus(Two a) { return {-a.hi, -a.lo}; }
__device__ __forceinline__ double rounded(Two a) { return a.hi + a.lo; }
__device__ __forceinline__ double times(double a, double b) { return a * b; }
__device__ __forceinline__ double plus(double a, double b) { return a + b; }
__device__ __forceinline__ double minus(double a) { return -a; }
__device__ __forceinline__ double rounded(double a) { return a; }
__device__ __forceinline__ double from_lane(uint32_t four, double a, int g) { return __shfl_sync(four, a, g, 4); }
__device__ __forceinline__ Two from_lane(uint32_t four, Two a, int g) {
  return {from_lane(four, a.hi, g), from_lane(four, a.lo, g)};
}
template <typename Real> struct Wide { using T = double; };
template <> struct Wide<double> { using T = Two; };
// 1 / sqrt(1 + t t)
__device__ __forceinline__ void inverse_norm(double t, double& h) { h = 1.0 / sqrt(1.0 + t * t); }
__device__ __forceinline__ void inverse_norm(double t, Two& h) {
  const double p = t * t, q = 1.0 + p, ql = (p - (q - 1.0)) + fma(t, t, -p);  // q + ql, p <= 1
  const double g = rsqrt(q), g2 = g * g, x = q * g2;
  // one Newton step on the residual 1 - (q + ql) g g: g's own error goes with it
  const double r = ((1.0 - x) - fma(q, g2, -x)) - (q * fma(g, g, -g2) + ql * g2);
  h = {g, 0.5 * g * r};
}

template <typename Real, bool BACK>
__global__ void __launch_bounds__(HeaCfg<Real, BACK>::NT, HeaCfg<Real, BACK>::CTAS)
    k_hea(const typename Cplx<Real>::T* src, typename Cplx<Real>::T* psi, typename Cplx<Real>::T* lam,
          const __grid_constant__ HeaPass P, const HeaSeg* __restrict__ segs, const double2* __restrict__ cs,
          double* __restrict__ partials, int part_stride) {
  using A = typename Cplx<Real>::T;
  constexpr int NT = HeaCfg<Real, BACK>::NT, TB = 7, kWarps = NT / 32;
  static_assert(NT == 1 << TB);
  constexpr int UB = sizeof(A) == 16 ? 0 : 1;  // log2 of the amplitudes of a 16-byte unit
  extern __shared__ __align__(128) unsigned char smem[];
  const uint32_t tile_bytes = (uint32_t)sizeof(A) << P.m;
  unsigned char* tables = smem + (BACK ? 2u : 1u) * tile_bytes;
  HeaTab<Real>* tab = reinterpret_cast<HeaTab<Real>*>(tables);
  double* red = reinterpret_cast<double*>(tab + P.num_segs);  // [warp][slot], backward only
  __shared__ uint32_t joff[1 << (kMaxHeaBits - TB)];            // index offset of unit j * NT
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int nslots = P.num_segs * kHeaSlots;
  HeaSeg* sseg = reinterpret_cast<HeaSeg*>(red + (BACK ? kWarps * nslots : 0));
  const uint32_t units = 1u << (P.m - UB), groups = 1u << (P.m - 3);

  for (uint32_t j = tid; j < (1u << (kMaxHeaBits - TB)); j += NT) {
    uint32_t off = 0;
#pragma unroll
    for (int b = TB; b < kMaxHeaBits - UB; b++)
      if (b + UB < P.m && (j >> (b - TB) & 1u)) off ^= P.basis[b + UB];
    joff[j] = off;
  }
  for (int i = tid; i < P.num_segs * (int)(sizeof(HeaSeg) / 4); i += NT)
    reinterpret_cast<uint32_t*>(sseg)[i] = reinterpret_cast<const uint32_t*>(segs)[i];
  uint32_t toff = 0;  // this thread's part of a unit's index
#pragma unroll
  for (int b = 0; b < TB; b++)
    if (b + UB < P.m && (tid >> b & 1)) toff ^= P.basis[b + UB];
  const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  __syncthreads();

  for (uint64_t item = blockIdx.x; item < P.num_items; item += gridDim.x) {
    const uint64_t b = item / P.items_per_state;
    const uint32_t tile0 = (uint32_t)(item % P.items_per_state) * P.tiles_per_item;
    const A* gs = src + (b << P.n);
    A* gp = psi + (b << P.n);
    A* gl = BACK ? lam + (b << P.n) : nullptr;
    for (uint32_t ti = 0; ti < P.tiles_per_item; ti++) {
      const uint32_t base = (uint32_t)pdep64(tile0 + ti, P.free_mask);
      bool work = true;
      if (!BACK && P.init) {
        work = base == P.init_base;
        for (uint32_t u = tid; u < units; u += NT) reinterpret_cast<double2*>(smem)[u] = make_double2(0.0, 0.0);
        if (work) {
          __syncthreads();
          if (tid == 0)
            *reinterpret_cast<A*>(smem + (UB ? tile_swz16(P.init_local >> 1) * 16u + (P.init_local & 1u) * 8u
                                             : tile_swz16(P.init_local) * 16u)) = A{1, 0};
        }
      } else {
        for (uint32_t u = tid, j = 0; u < units; u += NT, j++) {
          const uint32_t off = base ^ toff ^ joff[j];
          const uint32_t dst = sm0 + tile_swz16(u) * 16u;
          cp_async16(dst, gs + off);
          if (BACK) cp_async16(dst + tile_bytes, gl + off);
        }
      }
      if (ti == 0) {  // this state's tables, while the tile is on its way
        for (int i = tid; i < P.num_segs * 4; i += NT) {
          const HeaSeg& sg = sseg[i >> 2];
          HeaTab<Real>& tb = tab[i >> 2];
          const int k = i & 3;
          using W = typename Wide<Real>::T;
          W pr{1.0}, pi{0.0}, scale{1.0};
#pragma unroll
          for (int g = 0; g < 3; g++) {
            const int p = sg.param[g];
            const double2 z = p >= 0 ? cs[b * P.num_params + p + 1] : make_double2(1.0, 0.0);
            // RZ: bit 0 -> c - i s, bit 1 -> c + i s; undone: the conjugate
            const W zr{z.x}, zi{((k >> g & 1) != 0) != BACK ? z.y : -z.y};
            const W nr = plus(times(pr, zr), minus(times(pi, zi))), ni = plus(times(pr, zi), times(pi, zr));
            pr = nr;
            pi = ni;
          }
          // lane k of the segment's four has rotation k's tangent and scale
          // (of the rounded t, so that |scale [[1, t], [-t, 1]]| is 1)
          const int p = k < 3 ? sg.param[k] : -1;
          const double2 y = p >= 0 ? cs[b * P.num_params + p] : make_double2(1.0, 0.0);
          const bool flip = fabs(y.x) < fabs(y.y);
          const Real t = (Real)(flip ? y.x / y.y : y.y / y.x);
          W h;
          inverse_norm((double)t, h);
          if ((flip ? y.y : y.x) < 0.0) h = minus(h);
          const uint32_t four = 0xfu << (lane & 28);
#pragma unroll
          for (int g = 0; g < 3; g++) scale = times(scale, from_lane(four, h, g));
          const uint32_t flips = __ballot_sync(four, flip) >> (lane & 28) & 7u;
          if (k < 3) tb.t[k] = t;
          tb.ph[k] = A{(Real)rounded(times(scale, pr)), (Real)rounded(times(scale, pi))};
          if (k == 3) {
            tb.flip = flips;
            tb.unscale = 1.0 / (rounded(scale) * rounded(scale));
          }
        }
        if (BACK)
          for (int i = tid; i < kWarps * nslots; i += NT) red[i] = 0.0;
      }
      asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
      __syncthreads();
      for (int s = 0; s < (work ? P.num_segs : 0); s++) {
        const HeaSeg& sg = sseg[s];
        const HeaTab<Real>& tb = tab[s];
        const uint32_t a0 = sg.alpha[0], a1 = sg.alpha[1], a2 = sg.alpha[2];
        uint32_t off0 = 0;
        if (__popc(sg.fun[0] & base) & 1) off0 ^= a0;
        if (__popc(sg.fun[1] & base) & 1) off0 ^= a1;
        if (__popc(sg.fun[2] & base) & 1) off0 ^= a2;
#pragma unroll
        for (int q = 0; q < TB; q++)
          if (tid >> q & 1) off0 ^= sg.kappa[q];
        const uint32_t flip = tb.flip;
        const Real t0 = tb.t[0], t1 = tb.t[1], t2 = tb.t[2];
        A ph[4];  // read once: a broadcast 16-byte load takes four wavefronts
#pragma unroll
        for (int k = 0; k < 4; k++) ph[k] = tb.ph[k];
        double acc[8];
        if (BACK) {
#pragma unroll
          for (int i = 0; i < 8; i++) acc[i] = 0.0;
        }
        for (uint32_t g0 = 0; g0 < groups; g0 += NT) {
          const bool active = g0 + tid < groups;
          uint32_t off = off0;
#pragma unroll
          for (int q = TB; q < kMaxHeaBits - 3; q++)
            if (g0 >> q & 1u) off ^= sg.kappa[q];
          A v[8], w[8];
          if (active) {
#pragma unroll
            for (int k = 0; k < 8; k++) {
              const unsigned char* at = smem + (off ^ (k & 1 ? a0 : 0u) ^ (k & 2 ? a1 : 0u) ^ (k & 4 ? a2 : 0u));
              v[k] = *reinterpret_cast<const A*>(at);
              if (BACK) w[k] = *reinterpret_cast<const A*>(at + tile_bytes);
            }
            if (BACK) {
#pragma unroll
              for (int k = 0; k < 8; k++) {
                v[k] = turn(ph, k, v[k]);
                w[k] = turn(ph, k, w[k]);
              }
              // On the scaled states (the phases cancel): Im(conj(lambda) psi)
              // per amplitude, summed with the sign of each target bit, and
              // Im<lambda|Y|psi> of each: (Y psi)_0 = -i psi_1, (Y psi)_1 = i psi_0.
              // complex64 values are converted once: conversions run at a
              // quarter of the FP64 rate.
              double2 V[8], L[8];
#pragma unroll
              for (int k = 0; k < 8; k++) {
                V[k] = make_double2(v[k].x, v[k].y);
                L[k] = make_double2(w[k].x, w[k].y);
              }
              double d[8];
#pragma unroll
              for (int k = 0; k < 8; k++) d[k] = L[k].x * V[k].y - L[k].y * V[k].x;
              const double s0 = d[0] + d[1], s1 = d[2] + d[3], s2 = d[4] + d[5], s3 = d[6] + d[7];
              acc[0] += ((d[0] - d[1]) + (d[2] - d[3])) + ((d[4] - d[5]) + (d[6] - d[7]));
              acc[1] += (s0 - s1) + (s2 - s3);
              acc[2] += (s0 + s1) - (s2 + s3);
              acc[3] += hea_grad_y<0>(V, L);
              acc[4] += hea_grad_y<1>(V, L);
              acc[5] += hea_grad_y<2>(V, L);
              hea_ry<A, Real, 0, true>(v, t0, flip & 1u);
              hea_ry<A, Real, 0, true>(w, t0, flip & 1u);
              hea_ry<A, Real, 1, true>(v, t1, flip & 2u);
              hea_ry<A, Real, 1, true>(w, t1, flip & 2u);
              hea_ry<A, Real, 2, true>(v, t2, flip & 4u);
              hea_ry<A, Real, 2, true>(w, t2, flip & 4u);
            } else {
              hea_ry<A, Real, 0, false>(v, t0, flip & 1u);
              hea_ry<A, Real, 1, false>(v, t1, flip & 2u);
              hea_ry<A, Real, 2, false>(v, t2, flip & 4u);
#pragma unroll
              for (int k = 0; k < 8; k++) v[k] = turn(ph, k, v[k]);
            }
#pragma unroll
            for (int k = 0; k < 8; k++) {
              unsigned char* at = smem + (off ^ (k & 1 ? a0 : 0u) ^ (k & 2 ? a1 : 0u) ^ (k & 4 ? a2 : 0u));
              *reinterpret_cast<A*>(at) = v[k];
              if (BACK) *reinterpret_cast<A*>(at + tile_bytes) = w[k];
            }
          }
        }
        if (BACK) {
          // 8 sums over 32 lanes: halve the values with each of the first
          // three exchanges, then two full ones; lane 4 i ends with value i
          double h4[4], h2[2], h1;
          const bool b4 = lane & 16, b3 = lane & 8, b2 = lane & 4;
#pragma unroll
          for (int i = 0; i < 4; i++) {
            const double give = b4 ? acc[i] : acc[4 + i], keep = b4 ? acc[4 + i] : acc[i];
            h4[i] = keep + __shfl_xor_sync(0xffffffffu, give, 16);
          }
#pragma unroll
          for (int i = 0; i < 2; i++) {
            const double give = b3 ? h4[i] : h4[2 + i], keep = b3 ? h4[2 + i] : h4[i];
            h2[i] = keep + __shfl_xor_sync(0xffffffffu, give, 8);
          }
          const double give = b2 ? h2[0] : h2[1], keep = b2 ? h2[1] : h2[0];
          h1 = keep + __shfl_xor_sync(0xffffffffu, give, 4);
          h1 += __shfl_xor_sync(0xffffffffu, h1, 2);
          h1 += __shfl_xor_sync(0xffffffffu, h1, 1);
          if ((lane & 3) == 0 && lane < 4 * kHeaSlots) red[warp * nslots + s * kHeaSlots + (lane >> 2)] += h1;
        }
        __syncthreads();
      }
      for (uint32_t u = tid, j = 0; u < units; u += NT, j++) {
        const uint32_t off = base ^ toff ^ joff[j];
        const double2* at = reinterpret_cast<const double2*>(smem + tile_swz16(u) * 16u);
        __stcs(reinterpret_cast<double2*>(gp + off), *at);
        if (BACK) __stcs(reinterpret_cast<double2*>(gl + off), at[tile_bytes / 16]);
      }
      __syncthreads();
    }
    if (BACK) {
      for (int j = tid; j < nslots; j += NT) {
        double t = 0.0;
        for (int wp = 0; wp < kWarps; wp++) t += red[wp * nslots + j];
        partials[item * (uint64_t)part_stride + j] = t * tab[j / kHeaSlots].unscale;
      }
      __syncthreads();
    }
  }
}

// grads[b][p] = sum over state b's items for the parameter p of each of
// `slots` slots (-1: none).  A CTA takes 32 slots of one state, its warps an
// eighth of the items each, in order; then the eight sums in order.  (One
// thread a slot took 25 us for 256 items of two states, by the loads' latency.)
constexpr int kReduceWarps = 8;
__global__ void __launch_bounds__(32 * kReduceWarps) k_hea_reduce(const double* __restrict__ partials, uint32_t items,
                                                                  int slots, const int* __restrict__ param_of_slot,
                                                                  int num_params, double* __restrict__ grads) {
  __shared__ double sums[kReduceWarps][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int slot = blockIdx.x * 32 + lane;
  const uint64_t b = blockIdx.y;
  const double* p = partials + b * items * (uint64_t)slots + slot;
  const uint32_t each = (items + kReduceWarps - 1) / kReduceWarps, t0 = warp * each;
  const uint32_t t1 = t0 + each < items ? t0 + each : items;
  double sum = 0.0;
  if (slot < slots) {
#pragma unroll 32
    for (uint32_t t = t0; t < t1; t++) sum += p[t * (uint64_t)slots];
  }
  sums[warp][lane] = sum;
  __syncthreads();
  if (warp > 0 || slot >= slots) return;
  const int param = param_of_slot[slot];
  if (param < 0) return;
  for (int w = 1; w < kReduceWarps; w++) sum += sums[w][lane];
  grads[b * (uint64_t)num_params + param] = sum;
}

// out[b] = sum over state b's tiles, in order.
__global__ void k_adj_energy(const double* __restrict__ partials, uint64_t tiles_per_state, uint64_t batch,
                             double* __restrict__ out) {
  for (uint64_t b = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; b < batch; b += (uint64_t)gridDim.x * blockDim.x) {
    double s = 0.0;
    for (uint64_t t = 0; t < tiles_per_state; t++) s += partials[b * tiles_per_state + t];
    out[b] = s;
  }
}

// dst[p] = src[C^-k p] on n-bit indices, C^-1 x = x ^ (x << 1): (1 + S)^k
// over GF(2) is the product of 1 + S^(2^j) over the set bits j of k.
__host__ __device__ inline uint32_t unladder_index(uint32_t x, int n, int k) {
  for (int j = 0; (1 << j) < n; j++)
    if (k >> j & 1) x ^= (x << (1 << j)) & (uint32_t)((1ull << n) - 1ull);
  return x;
}
struct UnladderPass {
  int32_t n, k, m;
  uint32_t dst[kUnladderBits];       // dst index part of local bit b
  uint32_t src[kUnladderBits];       // src index part of load bit b
  uint32_t src_local[kUnladderBits]; // and its local index part
  uint64_t free_mask, num_tiles, tiles_per_state;
};
// Tiles hold whole rows of both orders: 2^kUnladderLow contiguous amplitudes
// of src on the way in, of dst on the way out.
__global__ void __launch_bounds__(256) k_unladder(const float2* __restrict__ src, float2* __restrict__ dst,
                                                  const __grid_constant__ UnladderPass P) {
  __shared__ float2 sm[1 << kUnladderBits];
  const uint32_t amps = 1u << P.m;
  for (uint64_t tile = blockIdx.x; tile < P.num_tiles; tile += gridDim.x) {
    const uint64_t b = tile / P.tiles_per_state;
    const uint32_t base = (uint32_t)pdep64(tile % P.tiles_per_state, P.free_mask);
    const uint32_t sbase = unladder_index(base, P.n, P.k);
    for (uint32_t e = threadIdx.x; e < amps; e += 256) {
      uint32_t off = sbase, t = 0;
#pragma unroll
      for (int q = 0; q < kUnladderBits; q++)
        if (e >> q & 1u) {
          off ^= P.src[q];
          t ^= P.src_local[q];
        }
      sm[t ^ (t >> 4 & 15u)] = src[(b << P.n) + off];
    }
    __syncthreads();
    for (uint32_t e = threadIdx.x; e < amps; e += 256) {
      uint32_t off = base;
#pragma unroll
      for (int q = 0; q < kUnladderBits; q++)
        if (e >> q & 1u) off ^= P.dst[q];
      dst[(b << P.n) + off] = sm[e ^ (e >> 4 & 15u)];
    }
    __syncthreads();
  }
}

// |0...0> in every state, for the tensor-core forward sweep (complex64).
__global__ void k_adj_init(float2* __restrict__ psi, uint64_t dim, uint64_t total) {
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x)
    psi[i] = (i & (dim - 1)) == 0 ? make_float2(1.f, 0.f) : make_float2(0.f, 0.f);
}

template <typename Real, bool BACK>
int launch_hea_t(const void* src, void* psi, void* lam, const HeaPass& P, const HeaSeg* d_segs, const double2* d_cs,
                 double* d_partials, int part_stride, int num_sms, cudaStream_t stream) {
  using A = typename Cplx<Real>::T;
  auto shared = [](int bits, int segs) {
    const size_t red = BACK ? sizeof(double) * (HeaCfg<Real, BACK>::NT / 32) * kHeaSlots : 0;
    return ((BACK ? 2 : 1) * sizeof(A) << bits) + segs * (sizeof(HeaTab<Real>) + red + sizeof(HeaSeg));
  };
  const size_t smem = shared(P.m, P.num_segs);
  auto kern = k_hea<Real, BACK>;
  static std::atomic<uint64_t> allowed{0};
  allow_shared(allowed, kern, shared(HeaCfg<Real, BACK>::BITS, kMaxHeaSegs));
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, HeaCfg<Real, BACK>::NT, smem);
  uint64_t grid = (uint64_t)num_sms * (per_sm < 1 ? 1 : per_sm);
  if (grid > P.num_items) grid = P.num_items;
  kern<<<(unsigned)grid, HeaCfg<Real, BACK>::NT, smem, stream>>>((const A*)src, (A*)psi, (A*)lam, P, d_segs, d_cs, d_partials,
                                                      part_stride);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

}  // namespace

int hea_tile_bits(int dtype, bool backward) {
  if (dtype == MLB_C128) return backward ? HeaCfg<double, true>::BITS : HeaCfg<double, false>::BITS;
  return backward ? HeaCfg<float, true>::BITS : HeaCfg<float, false>::BITS;
}

int launch_adj_init(void* psi, int n, uint64_t batch, cudaStream_t stream) {
  const uint64_t dim = 1ull << n, total = dim * batch;
  uint64_t grid = (total + 255) / 256;
  if (grid > 148ull * 32) grid = 148ull * 32;
  k_adj_init<<<(unsigned)grid, 256, 0, stream>>>((float2*)psi, dim, total);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_hea_pass(int dtype, const void* psi_src, void* psi, void* lam, const HeaPass& P, const HeaSeg* d_segs,
                    const double2* d_cs, double* d_partials, int part_stride, bool backward, int num_sms,
                    cudaStream_t stream) {
  if (P.num_segs < 1 || P.num_segs > kMaxHeaSegs || P.m < 3 || P.m > hea_tile_bits(dtype, backward) || P.n > 30)
    return MLB_ERR_INVALID_ARG;
  auto run = [&](auto f) {
    return f(psi_src, psi, lam, P, d_segs, d_cs, d_partials, part_stride, num_sms, stream);
  };
  if (dtype == MLB_C128) return backward ? run(launch_hea_t<double, true>) : run(launch_hea_t<double, false>);
  return backward ? run(launch_hea_t<float, true>) : run(launch_hea_t<float, false>);
}

int launch_hea_reduce(const double* d_partials, uint32_t items, int slots, uint64_t batch, const int* d_param_of_slot,
                      int num_params, double* d_grads, cudaStream_t stream) {
  if (slots < 1) return MLB_ERR_INVALID_ARG;
  for (uint64_t b0 = 0; b0 < batch; b0 += 65535) {  // grid.y's limit
    const uint64_t nb = batch - b0 < 65535 ? batch - b0 : 65535;
    k_hea_reduce<<<dim3((unsigned)((slots + 31) / 32), (unsigned)nb), 32 * kReduceWarps, 0, stream>>>(
        d_partials + b0 * items * (uint64_t)slots, items, slots, d_param_of_slot, num_params,
        d_grads + b0 * (uint64_t)num_params);
    count_launch();
  }
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_adj_energy(const double* d_partials, uint64_t tiles_per_state, uint64_t batch, double* d_out,
                      cudaStream_t stream) {
  uint64_t grid = (batch + 31) / 32;
  if (grid > 148ull * 16) grid = 148ull * 16;
  k_adj_energy<<<(unsigned)grid, 32, 0, stream>>>(d_partials, tiles_per_state, batch, d_out);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_unladder(const void* src, void* dst, int n, int k, uint64_t batch, int num_sms, cudaStream_t stream) {
  if (n < 3 || n > 30 || batch < 1 || k < 0) return MLB_ERR_INVALID_ARG;
  UnladderPass P{};
  P.n = n;
  P.k = k;
  P.m = n < kUnladderBits ? n : kUnladderBits;
  // the tile: rows of dst (low unit vectors), rows of src (C^k e_i), then
  // low unit vectors; load order: src's rows first
  hea::Basis B, S;
  std::vector<uint64_t> load;
  const int low = P.m < 2 * kUnladderLow ? P.m / 2 : kUnladderLow;
  for (int i = 0; i < low; i++) B.add(1ull << i);
  for (int i = 0; i < low; i++) {
    uint64_t v = 1ull << i;
    for (int j = 0; j < k; j++) v = hea::ladder(v, n);
    B.add(v);
    S.add(v);
    load.push_back(v);
  }
  for (int b = 0; b < n && (int)B.v.size() < P.m; b++) B.add(1ull << b);
  for (uint64_t v : B.v)
    if (S.add(v)) load.push_back(v);
  uint64_t pivots = 0;
  for (int b = 0; b < P.m; b++) {
    P.dst[b] = (uint32_t)B.v[b];
    P.src[b] = unladder_index((uint32_t)load[b], n, k);
    P.src_local[b] = B.coords(load[b]);
    pivots |= 1ull << B.piv[b];
  }
  P.free_mask = ((1ull << n) - 1ull) & ~pivots;
  P.tiles_per_state = 1ull << (n - P.m);
  P.num_tiles = P.tiles_per_state * batch;
  uint64_t grid = (uint64_t)num_sms * 8;
  if (grid > P.num_tiles) grid = P.num_tiles;
  k_unladder<<<(unsigned)grid, 256, 0, stream>>>((const float2*)src, (float2*)dst, P);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

// ---------------------------------------------------------------------------
// Per-vector squared norms of a batch of complex64 states and the division
// of energies and gradients by them (the tensor-core forward sweep's norm
// drift cancels: E and dE/dtheta both carry |psi|^2).  One CTA per vector,
// a fixed-order tree: the result does not depend on scheduling.
// ---------------------------------------------------------------------------
namespace {
__global__ void __launch_bounds__(256) k_batch_norm(const float2* __restrict__ psi, uint64_t dim,
                                                    double* __restrict__ out) {
  __shared__ double red[256];
  const float2* v = psi + (uint64_t)blockIdx.x * dim;
  double acc = 0.0;
  for (uint64_t i = threadIdx.x; i < dim; i += 256) {
    const float2 a = v[i];
    acc += (double)a.x * a.x + (double)a.y * a.y;
  }
  red[threadIdx.x] = acc;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) out[blockIdx.x] = red[0];
}

// out = [B] energies, then [B][P] gradients
__global__ void k_divide_by_norm(double* __restrict__ out, uint64_t batch, int num_params,
                                 const double* __restrict__ nrm) {
  const uint64_t total = batch * (uint64_t)(1 + num_params);
  for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < total; i += (uint64_t)gridDim.x * blockDim.x) {
    const uint64_t b = i < batch ? i : (i - batch) / (uint64_t)num_params;
    out[i] /= nrm[b];
  }
}
}  // namespace

int launch_batch_norm(const void* psi_c64, uint64_t dim, uint64_t batch, double* d_norm, cudaStream_t stream) {
  if (batch == 0 || batch > 65535) return MLB_ERR_INVALID_ARG;
  k_batch_norm<<<(unsigned)batch, 256, 0, stream>>>(static_cast<const float2*>(psi_c64), dim, d_norm);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

int launch_divide_by_norm(double* d_out, uint64_t batch, int num_params, const double* d_norm,
                          cudaStream_t stream) {
  const uint64_t total = batch * (uint64_t)(1 + num_params);
  uint64_t grid = (total + 255) / 256;
  if (grid < 1) grid = 1;
  if (grid > 148ull * 8) grid = 148ull * 8;
  k_divide_by_norm<<<(unsigned)grid, 256, 0, stream>>>(d_out, batch, num_params, d_norm);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

}  // namespace mlb
