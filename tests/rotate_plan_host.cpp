// Host harness of tests/test_rotate_plan.py: one tile pass lowered to a
// rotation program (rotate_plan.h) and run on the host as kernels_rotate.cu
// runs it, in double.
#include <complex>
#include <map>
#include <vector>

#include "rotate_plan.h"

using namespace mlb;
using cd = std::complex<double>;

size_t mlb::rot_shared_bytes(int dtype, size_t num_ops, size_t entries) {
  return dtype == MLB_C128 ? num_ops * 64 + entries * 16 : num_ops * 48 + entries * 8;
}

namespace {

uint64_t deposit(uint64_t x, uint64_t mask) {
  uint64_t r = 0;
  for (uint64_t b = 1; mask; b <<= 1, mask &= mask - 1)
    if (x & b) r |= mask & -mask;
  return r;
}

int odd(uint64_t x) { return __builtin_parityll(x); }

bool run(const DevPass& P, const rot::Program& pr, int dtype, std::vector<cd>& amp) {
  const RotPass& D = pr.dev;
  const uint32_t size = 1u << D.m;
  std::map<uint32_t, uint32_t> local;  // local index at a byte offset of the tile
  for (uint32_t t = 0; t < size; t++) local[hea::slot_bytes(t, dtype)] = t;
  auto combine = [](uint32_t bits, const uint16_t* v, int n) {
    uint32_t x = 0;
    for (int i = 0; i < n; i++)
      if (bits >> i & 1) x ^= v[i];
    return x;
  };
  for (uint64_t tile = 0; tile < P.num_tiles; tile++) {
    const uint64_t base = deposit(tile, P.tile_free_mask);
    auto index = [&](uint32_t t) {
      uint64_t x = base;
      for (int b = 0; b < D.m; b++)
        if (t >> b & 1) x ^= D.basis[b];
      return x;
    };
    std::vector<cd> s(size);
    for (uint32_t t = 0; t < size; t++) s[t] = amp[index(t)];
    for (const RotSeg& sg : pr.segs) {
      std::vector<cd> next(size);
      std::vector<char> written(size, 0);
      for (uint32_t g = 0; g < size >> 4; g++) {
        const uint32_t off = combine(g, sg.kappa, D.m - 4);
        cd v[16];
        for (uint32_t k = 0; k < 16; k++) v[k] = s[local.at(off ^ combine(k, sg.alpha, 4))];
        for (int o = sg.op_begin; o < sg.op_end; o++) {
          const RotOp& op = pr.ops[o];
          for (uint32_t p = op.perm; p; p >>= 4) {
            const int i = (p & 15u) >> 2, j = p & 3u;
            for (int k = 0; k < 16; k++)
              if ((k >> i & 1) && !(k >> j & 1)) std::swap(v[k], v[k | 1 << j]);
          }
          if (op.flags & kRotTable) {
            uint32_t x = 0;
            for (int j = 0; j < op.nv; j++) x |= (uint32_t)(odd(op.vzg[j] & g) ^ odd(op.vout[j] & base)) << j;
            for (int k = 0; k < 16; k++) v[k] *= pr.table[op.table + 16 * x + k];
          }
          if (op.flags & kRotTurn)
            for (int b = 0; b < 4; b++) {
              const double t = odd(op.tzg[b] & g) ^ odd(op.tout[b] & base) ? -op.t[b] : op.t[b];
              for (int k = 0; k < 16; k++)
                if (!(k >> b & 1)) {
                  const cd lo = v[k], hi = v[k | 1 << b];
                  v[k] = lo - t * hi;
                  v[k | 1 << b] = hi + t * lo;
                }
            }
        }
        for (uint32_t k = 0; k < 16; k++) {
          const uint32_t t = local.at(off ^ combine(k, sg.alpha_out, 4));
          if (written[t]++) return false;
          next[t] = v[k];
        }
      }
      s.swap(next);
    }
    uint32_t flip = 0;
    for (int i = 0; i < D.m; i++)
      if ((D.label_const >> i & 1u) ^ (uint32_t)odd(D.label_out[i] & base)) flip ^= D.dir_slot[i];
    for (uint32_t t = 0; t < size; t++) amp[index(t)] = s[local.at(flip ^ combine(t, D.dir_slot, D.m))];
  }
  return true;
}

}  // namespace

extern "C" {

int host_covers(const mlb_op_t* op) { return rot::covers(*op); }

// The pushed matrices, rounded, in place.
void host_push_forward(mlb_op_t* ops, size_t num, uint32_t n) {
  const std::vector<rot::Unitary> u = rot::push_forward(std::vector<mlb_op_t>(ops, ops + num), n);
  for (size_t i = 0; i < num; i++)
    for (int k = 0; k < 4 && ops[i].kind == MLB_OP_1Q; k++) {
      ops[i].m[2 * k] = (double)u[i].m[k].real();
      ops[i].m[2 * k + 1] = (double)u[i].m[k].imag();
    }
}

// The ops on n qubits as one pass whose tile holds the qubits of `tile`
// (qubits 0 and 1 among them), on amp in place, pushed forward first if
// `push`.  1: an op is not covered, 2: the program does not fit, 3: an
// amplitude is written twice.
int host_run(const mlb_op_t* ops, size_t num, int n, uint64_t tile, int dtype, int push, double* amp) {
  DevPass P{};
  P.n = n;
  P.L = 2;
  for (int q = 2; q < n; q++)
    if (tile >> q & 1) P.high[P.H++] = q;
  P.tile_free_mask = ((1ull << n) - 1) & ~tile;
  P.num_tiles = 1ull << (n - P.L - P.H);
  std::vector<rot::Unitary> units;
  if (push) units = rot::push_forward(std::vector<mlb_op_t>(ops, ops + num), n);
  std::vector<rot::Gate> list;
  for (size_t i = 0; i < num; i++) {
    if (!rot::covers(ops[i])) return 1;
    list.push_back({ops + i, push ? &units[i] : nullptr});
  }
  rot::Program pr;
  if (!rot::Lower::lower(P, dtype, list, pr)) return 2;
  std::vector<cd> a(1ull << n);
  for (size_t i = 0; i < a.size(); i++) a[i] = cd(amp[2 * i], amp[2 * i + 1]);
  if (!run(P, pr, dtype, a)) return 3;
  for (size_t i = 0; i < a.size(); i++) {
    amp[2 * i] = a[i].real();
    amp[2 * i + 1] = a[i].imag();
  }
  return 0;
}

}  // extern "C"
