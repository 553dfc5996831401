// kernels_rotate.cu -- tile passes as programs of plane rotations and
// diagonal tables (planned by rotate_plan.h).
//
// One pass reads and writes the state once, in the tiles of the qubit planner
// (64 KiB: 12 bits of complex128, 13 of complex64).  The 16-byte units of a
// tile come by cp.async, all in flight at once.  In a segment a thread keeps
// the 16 amplitudes of a group in registers along the segment's four
// directions and runs the segment's rounds: a table of 16 complex factors and
// four plane rotations along the register bits, two multiply-adds per
// component each, as one block of straight code.  (A switch per rotation over
// its direction took three times the instructions: every case has to leave
// the 16 amplitudes in the same registers, so each moved half of them.)  A
// CNOT between register bits permutes the registers; others, X and SWAP cost
// nothing: the store reads each output's slot through the labels' directions.
// The program's ops, with this tile's signs, and its tables lie in shared
// memory; a round's table is read ahead of its use (a broadcast load of 16
// bytes takes four wavefronts, a table of complex128 half as many as the
// amplitudes' own round trip).  Read from global memory as it is used, or
// from the constant bank, the tables took twice as long.
// Bound: of a 30-qubit, depth-40 circuit's 62 complex128 passes, 682 ms,
// 155 ms are the segments' shared-memory round trips, 143 ms the tables,
// 192 ms the rotations (FP64), and about 190 ms the part of the memory phases
// that other CTAs' work does not cover; the same circuit in complex64 takes
// 457 ms (1197 ms gate by gate).  engine.cpp states where each form runs.
#include "kernels_common.cuh"
#include "mlb_internal.h"

namespace mlb {

namespace {

template <typename Real> struct RotCfg;
template <> struct RotCfg<double> { static constexpr int BITS = kTileBitsC128, NT = 128, CTAS = 3; };
template <> struct RotCfg<float> { static constexpr int BITS = 13, NT = 256, CTAS = 2; };

template <typename Real>
struct TileOp {  // an op with this tile's outside functionals applied
  Real t[4];
  uint32_t tzg[2];  // two group functionals each
  uint32_t vzg[2];
  uint32_t table;   // first entry, the tile's part of the variant included
  uint32_t perm;
  uint32_t flags;   // flags | nv << 8
  uint32_t variant; // the tile's part
};

__device__ __forceinline__ double signed_by(double t, uint32_t bit) {  // bit in bit 0
  return __hiloint2double(__double2hiint(t) ^ (int)(bit << 31), __double2loint(t));
}
__device__ __forceinline__ float signed_by(float t, uint32_t bit) {
  return __uint_as_float(__float_as_uint(t) ^ (bit << 31));
}

template <typename A, typename Real, int BIT>
__device__ __forceinline__ void rotate(A (&v)[16], Real t) {
#pragma unroll
  for (int k = 0; k < 16; k++) {
    if (k & (1 << BIT)) continue;
    const A a = v[k], b = v[k | 1 << BIT];
    v[k] = {a.x - t * b.x, a.y - t * b.y};
    v[k | 1 << BIT] = {b.x + t * a.x, b.y + t * a.y};
  }
}

// Register index bit J ^= bit I.
template <typename A, int I, int J>
__device__ __forceinline__ void permute(A (&v)[16]) {
#pragma unroll
  for (int k = 0; k < 16; k++)
    if ((k >> I & 1) && !(k >> J & 1)) {
      const A x = v[k];
      v[k] = v[k | 1 << J];
      v[k | 1 << J] = x;
    }
}

__device__ __forceinline__ uint32_t slot_of(uint32_t off, const uint16_t (&a)[4], int k) {
  return off ^ (k & 1 ? a[0] : 0u) ^ (k & 2 ? a[1] : 0u) ^ (k & 4 ? a[2] : 0u) ^ (k & 8 ? a[3] : 0u);
}

template <typename Real>
__global__ void __launch_bounds__(RotCfg<Real>::NT, RotCfg<Real>::CTAS)
    k_rotate(typename Cplx<Real>::T* __restrict__ amp, const __grid_constant__ RotPass P,
             const RotSeg* __restrict__ segs, const RotOp* __restrict__ ops,
             const typename Cplx<Real>::T* __restrict__ d_table) {
  using A = typename Cplx<Real>::T;
  constexpr int NT = RotCfg<Real>::NT, TB = NT == 256 ? 8 : 7;
  constexpr int UB = sizeof(A) == 16 ? 0 : 1;              // log2 of the amplitudes of a 16-byte unit
  constexpr int kSteps = 1 << (RotCfg<Real>::BITS - UB - TB);  // units of a full tile per thread
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ uint64_t joff[kSteps];   // index offset of unit j NT
  __shared__ uint16_t jslot[kSteps];  // and its outputs' slot offset
  __shared__ uint32_t s_flip;         // slot offset of this tile's label constants
  constexpr int m = RotCfg<Real>::BITS;
  const int num_ops = P.num_ops, num_segs = P.num_segs;
  A* table = reinterpret_cast<A*>(smem + (sizeof(A) << m));
  TileOp<Real>* tops = reinterpret_cast<TileOp<Real>*>(table + P.entries);
  const int tid = threadIdx.x;
  for (uint32_t i = tid; i < P.entries; i += NT) table[i] = d_table[i];
  for (int j = tid; j < kSteps; j += NT) {
    uint64_t off = 0;
    uint32_t slot = 0;
    for (int b = TB; b + UB < m; b++)
      if (j >> (b - TB) & 1) {
        off |= P.basis[b + UB];
        slot ^= P.dir_slot[b + UB];
      }
    joff[j] = off;
    jslot[j] = (uint16_t)slot;
  }
  uint64_t toff = 0;   // this thread's part of a unit's index
  uint32_t tslot = 0;  // and of its outputs' slot
  for (int b = 0; b < TB && b + UB < m; b++)
    if (tid >> b & 1) {
      toff |= P.basis[b + UB];
      tslot ^= P.dir_slot[b + UB];
    }
  const uint32_t slot1 = UB ? P.dir_slot[0] : 0u;  // the unit's second amplitude
  const uint32_t sm0 = static_cast<uint32_t>(__cvta_generic_to_shared(smem));
  constexpr uint32_t units = 1u << (m - UB), groups = 1u << (m - 4);
  __syncthreads();

  for (uint64_t tile = blockIdx.x; tile < P.num_tiles; tile += gridDim.x) {
    const uint64_t base = pdep64(tile, P.free_mask);
    for (uint32_t u = tid, j = 0; u < units; u += NT, j++)
      cp_async16(sm0 + tile_swz16(u) * 16u, amp + (base | toff | joff[j]));
    for (int o = tid; o < num_ops; o += NT) {
      const RotOp& op = ops[o];
      TileOp<Real> w;
#pragma unroll
      for (int i = 0; i < 4; i++) w.t[i] = (Real)signed_by(op.t[i], (uint32_t)(__popcll(op.tout[i] & base) & 1));
      w.tzg[0] = op.tzg[0] | (uint32_t)op.tzg[1] << 16;
      w.tzg[1] = op.tzg[2] | (uint32_t)op.tzg[3] << 16;
      w.vzg[0] = op.vzg[0] | (uint32_t)op.vzg[1] << 16;
      w.vzg[1] = op.vzg[2] | (uint32_t)op.vzg[3] << 16;
      w.variant = 0;
      for (int j = 0; j < op.nv; j++) w.variant |= (uint32_t)(__popcll(op.vout[j] & base) & 1) << j;
      w.table = op.table;
      w.perm = op.perm;
      w.flags = op.flags;
      tops[o] = w;
    }
    if (tid < 32) {
      uint32_t f = 0;
      if (tid < m && (((P.label_const >> tid) ^ (uint32_t)__popcll(P.label_out[tid] & base)) & 1u))
        f = P.dir_slot[tid];
      f = __reduce_xor_sync(0xffffffffu, f);
      if (tid == 0) s_flip = f;
    }
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    for (int s = 0; s < num_segs; s++) {
      const RotSeg& sg = segs[s];
      uint32_t off0 = 0;
#pragma unroll
      for (int q = 0; q < TB; q++)
        if (tid >> q & 1) off0 ^= sg.kappa[q];
      for (uint32_t g0 = 0; g0 < groups; g0 += NT) {
        uint32_t off = off0;
#pragma unroll
        for (int q = TB; q < kRotBits - 4; q++)
          if (g0 >> q & 1u) off ^= sg.kappa[q];
        const uint32_t gi = g0 + tid;
        A v[16];
#pragma unroll
        for (int k = 0; k < 16; k++) v[k] = *reinterpret_cast<const A*>(smem + slot_of(off, sg.alpha, k));
        for (int o = sg.op_begin; o < sg.op_end; o++) {
          const TileOp<Real>& w = tops[o];
          const uint32_t flags = w.flags;
          // the table's first entries, on their way while the registers move
          constexpr int kAhead = sizeof(Real) == 8 ? 4 : 16;
          const A* T = table;
          A ahead[kAhead];
          if (flags & kRotTable) {
            const uint32_t z0 = w.vzg[0], z1 = w.vzg[1];
            uint32_t x = w.variant;
            x ^= (uint32_t)(__popc(z0 & 0xffffu & gi) & 1) | (uint32_t)(__popc(z0 >> 16 & gi) & 1) << 1 |
                 (uint32_t)(__popc(z1 & 0xffffu & gi) & 1) << 2 | (uint32_t)(__popc(z1 >> 16 & gi) & 1) << 3;
            T = table + (w.table + 16 * x);
#pragma unroll
            for (int k = 0; k < kAhead; k++) ahead[k] = T[k];
          }
          for (uint32_t p = w.perm; p; p >>= 4)
            switch (p & 15u) {
#define MLB_P(i, j) \
  case 4 * i + j: permute<A, i, j>(v); break;
              MLB_P(0, 1) MLB_P(0, 2) MLB_P(0, 3) MLB_P(1, 0) MLB_P(1, 2) MLB_P(1, 3)
              MLB_P(2, 0) MLB_P(2, 1) MLB_P(2, 3) MLB_P(3, 0) MLB_P(3, 1) MLB_P(3, 2)
#undef MLB_P
            }
          if (flags & kRotTable) {
#pragma unroll
            for (int k0 = 0; k0 < 16; k0 += kAhead) {
              A next[kAhead];
#pragma unroll
              for (int k = 0; k < kAhead; k++)
                if (k0 + kAhead < 16) next[k] = T[k0 + kAhead + k];
#pragma unroll
              for (int k = 0; k < kAhead; k++) v[k0 + k] = cmul(ahead[k], v[k0 + k]);
#pragma unroll
              for (int k = 0; k < kAhead; k++) ahead[k] = next[k];
            }
          }
          if (flags & kRotTurn) {
            const uint32_t z0 = w.tzg[0], z1 = w.tzg[1];
            rotate<A, Real, 0>(v, signed_by(w.t[0], (uint32_t)__popc(z0 & 0xffffu & gi)));
            rotate<A, Real, 1>(v, signed_by(w.t[1], (uint32_t)__popc(z0 >> 16 & gi)));
            rotate<A, Real, 2>(v, signed_by(w.t[2], (uint32_t)__popc(z1 & 0xffffu & gi)));
            rotate<A, Real, 3>(v, signed_by(w.t[3], (uint32_t)__popc(z1 >> 16 & gi)));
          }
        }
#pragma unroll
        for (int k = 0; k < 16; k++) *reinterpret_cast<A*>(smem + slot_of(off, sg.alpha_out, k)) = v[k];
      }
      __syncthreads();
    }
    const uint32_t flip = s_flip;
    for (uint32_t u = tid, j = 0; u < units; u += NT, j++) {
      const uint32_t slot = tslot ^ jslot[j] ^ flip;
      A* to = amp + (base | toff | joff[j]);
      if constexpr (UB == 0) {
        __stcs(to, *reinterpret_cast<const A*>(smem + slot));
      } else {
        const A a = *reinterpret_cast<const A*>(smem + slot), b = *reinterpret_cast<const A*>(smem + (slot ^ slot1));
        __stcs(reinterpret_cast<float4*>(to), make_float4(a.x, a.y, b.x, b.y));
      }
    }
    __syncthreads();
  }
}

template <typename Real>
int launch_rot_t(void* amp, const RotPass& P, const RotSeg* d_segs, const RotOp* d_ops, const void* d_table,
                 int num_sms, cudaStream_t stream) {
  using A = typename Cplx<Real>::T;
  const size_t prog = P.num_ops * sizeof(TileOp<Real>) + P.entries * sizeof(A);
  if (P.m != RotCfg<Real>::BITS || prog > kRotMaxShared) return MLB_ERR_INVALID_ARG;  // whole tiles: every lane has a group
  static std::atomic<uint64_t> allowed{0};
  allow_shared(allowed, k_rotate<Real>, (sizeof(A) << RotCfg<Real>::BITS) + kRotMaxShared);
  const size_t smem = (sizeof(A) << P.m) + prog;
  int per_sm = 1;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_rotate<Real>, RotCfg<Real>::NT, smem);
  uint64_t grid = (uint64_t)num_sms * (per_sm < 1 ? 1 : per_sm);
  if (grid > P.num_tiles) grid = P.num_tiles;
  k_rotate<Real><<<(unsigned)grid, RotCfg<Real>::NT, smem, stream>>>((A*)amp, P, d_segs, d_ops, (const A*)d_table);
  count_launch();
  return cudaGetLastError() == cudaSuccess ? MLB_OK : MLB_ERR_DRIVER;
}

}  // namespace

size_t rot_shared_bytes(int dtype, size_t num_ops, size_t entries) {
  return dtype == MLB_C128 ? num_ops * sizeof(TileOp<double>) + entries * 16
                           : num_ops * sizeof(TileOp<float>) + entries * 8;
}

int launch_rot_pass(int dtype, void* amp, const RotPass& pass, const RotSeg* d_segs, const RotOp* d_ops,
                    const void* d_table, int num_sms, cudaStream_t stream) {
  return dtype == MLB_C128 ? launch_rot_t<double>(amp, pass, d_segs, d_ops, d_table, num_sms, stream)
                           : launch_rot_t<float>(amp, pass, d_segs, d_ops, d_table, num_sms, stream);
}

}  // namespace mlb
