// rotate_plan.h -- lowers the ops of one tile pass into a program of plane
// rotations and diagonal tables (run by kernels_rotate.cu).  Host-only.
//
// The ops of most circuits are one-qubit unitaries, CNOTs, SWAPs and
// diagonals.  Inside a tile:
//   * X, CNOT and SWAP are not carried out.  They relabel: logical bit i of
//     an amplitude at local index t is an affine functional of t and of the
//     tile's outside bits, and flipping logical bit i moves along a direction
//     (an XOR mask of t).  The store at the end of the pass writes every
//     amplitude to the index its labels spell, a permutation of the tile.
//   * A one-qubit unitary is diag(u1, u2) s [[1, -t], [t, 1]] diag(1, w),
//     0 <= t <= 1 (the columns swapped first, an X, where |U00| < |U10|).  The
//     rotation costs two multiply-adds per component pair; s is folded into
//     the next table.
//     Factors and their products are long double until a table's entry is
//     rounded: 20 qubits, depth 16: the norm drifts 5e-16, with doubles
//     4.8e-15, as 16x16 matrices 2.8e-15.
//   * Diagonals (those factors, RZ, phases, ZZ, controlled phases) are
//     products over the functionals they read.  All that are due are merged
//     into one table of a complex factor per register index, in up to 16
//     variants for the parities of functionals that the registers do not hold.
// A segment keeps 16 amplitudes of a group in registers along four
// directions and runs every rotation whose direction lies in their span, in
// rounds: a permutation of the registers, a table and up to four commuting
// rotations, each along one register bit that it alone reads.  Program order
// is kept between rotations and diagonals that do not commute (a functional
// of one that changes along the other's direction).
#pragma once

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdint>
#include <vector>

#include "hea_plan.h"
#include "mlb_internal.h"
#include "planner.h"

namespace mlb {
namespace rot {

using cd = std::complex<double>;
using cl = std::complex<long double>;  // products of many factors, rounded once

struct Fun {  // parity(row & t) ^ parity(out & tile base) ^ c
  uint32_t row = 0;
  uint64_t out = 0;
  bool c = false;
  void add(const Fun& o) { row ^= o.row; out ^= o.out; c ^= o.c; }
  bool same(const Fun& o) const { return row == o.row && out == o.out; }
};

constexpr int kMaxItems = 512, kWords = kMaxItems / 64;  // a pass's ops give at most three items each
static_assert(3 * kMaxPassOps <= kMaxItems, "items of a pass");

struct Set {
  uint64_t w[kWords] = {};
  void add(int i) { w[i >> 6] |= 1ull << (i & 63); }
  bool has(int i) const { return w[i >> 6] >> (i & 63) & 1ull; }
};

struct Item {
  bool rotation = false;
  // rotation: direction, its target bit and its tangent; scale owed
  uint32_t dir = 0;
  Fun fun;
  double t = 0;
  long double s = 1;
  // diagonal: where every condition holds, d[0] or d[1] by the key (no key: d[1])
  Fun cond[3];
  int nc = 0;
  bool keyed = false;
  Fun key;
  cl d[2] = {1.0L, 1.0L};
  Set pred, succ;
  int height = 0;
};

inline cl mul(cl a, cl b) {
  const long double br = b.real(), bi = b.imag();
  return {a.real() * br - a.imag() * bi, a.real() * bi + a.imag() * br};
}
struct Program {
  RotPass dev{};
  std::vector<RotSeg> segs;
  std::vector<RotOp> ops;
  std::vector<cd> table;  // 16 << nv entries a table op: [variant][register index]
};

// Whether the rotation program covers an op (matrix values aside from
// unitarity included): what it does not cover runs as before.
inline bool covers(const mlb_op_t& o) {
  switch (o.kind) {
    case MLB_OP_1Q: {
      if (o.cmask) return false;
      // columns of length one and orthogonal, to rounding
      const double* m = o.m;
      const double p = m[0] * m[0] + m[1] * m[1] + m[4] * m[4] + m[5] * m[5] - 1.0;
      const double q = m[2] * m[2] + m[3] * m[3] + m[6] * m[6] + m[7] * m[7] - 1.0;
      const double x = m[0] * m[2] + m[1] * m[3] + m[4] * m[6] + m[5] * m[7];  // conj(a) b + conj(c) d
      const double y = m[0] * m[3] - m[1] * m[2] + m[4] * m[7] - m[5] * m[6];
      return std::abs(p) < 2e-14 && std::abs(q) < 2e-14 && x * x + y * y < 4e-28;
    }
    case MLB_OP_X: return plan::popc(o.cmask) <= 1;
    case MLB_OP_SWAP: return o.cmask == 0;
    case MLB_OP_DIAG1: return plan::popc(o.cmask) <= 2;
    case MLB_OP_ZZ: return plan::popc(o.cmask) <= 3;
    case MLB_OP_PHASE: return plan::popc(o.cmask) <= 3;
    default: return false;
  }
}

// A one-qubit op's matrix as the programs take it: products of several are
// rounded only where a table's entry or a tangent is.
struct Unitary {
  cl m[4] = {};
};
inline Unitary unitary(const mlb_op_t& o) {
  Unitary u;
  for (int k = 0; k < 4; k++) u.m[k] = cl(o.m[2 * k], o.m[2 * k + 1]);
  return u;
}
inline cl conj(cl a) { return {a.real(), -a.imag()}; }
inline long double norm(cl a) { return a.real() * a.real() + a.imag() * a.imag(); }
inline long double size(cl a) { return std::sqrt(norm(a)); }

// The ops' matrices (of one-qubit unitaries) once what each ends with has
// moved past the ops that it commutes with and into the next unitary of its
// qubit, so that most need no diagonal after their rotation: a phase past
// controls and diagonals, an X rotation past CNOTs that have the qubit as
// target (U = RX(alpha) V with V's first column real up to a phase).  The
// 20-qubit, depth-20 brickwork lowers to a third fewer tables, and its 24-qubit
// one runs in 5.5 ms, not 6.7.
inline std::vector<Unitary> push_forward(const std::vector<mlb_op_t>& ops, uint32_t n) {
  struct Open {
    int op = -1;      // the qubit's last one-qubit unitary
    int between = 0;  // ops since: 1 diagonal on it, 2 X on it, 3 neither way
  };
  std::vector<Open> open(n);
  std::vector<Unitary> out(ops.size());
  for (size_t i = 0; i < ops.size(); i++) {
    const mlb_op_t& o = ops[i];
    const uint64_t T = plan::op_targets(o);
    for (uint64_t b = plan::op_qubits(o) & ~T; b; b &= b - 1) open[__builtin_ctzll(b)].between |= 1;
    if (o.kind == MLB_OP_X) {
      open[o.target].between |= 2;
      continue;
    }
    if (o.kind != MLB_OP_1Q || o.cmask) {
      for (uint64_t b = T; b; b &= b - 1) open[__builtin_ctzll(b)].op = -1;
      continue;
    }
    out[i] = unitary(o);
    Open& e = open[o.target];
    if (e.op >= 0 && (e.between == 1 || e.between == 2)) {
      cl* p = out[e.op].m;  // = f V: V stays, f goes to o
      cl* q = out[i].m;
      if (e.between == 1) {
        // f = diag(1, x / |x|), the second row's phase beside the first's, of
        // the larger column (an entry of rounding's size or less has none
        // that matters)
        const cl x = norm(p[0]) >= norm(p[2]) ? mul(p[2], conj(p[0])) : mul(p[3], conj(p[1]));
        const long double r = size(x);
        if (r > 1e-150L) {
          const cl f = x / r;
          p[2] = mul(p[2], conj(f));
          p[3] = mul(p[3], conj(f));
          q[1] = mul(q[1], f);
          q[3] = mul(q[3], f);
        }
      } else {
        // f = [[co, -i si], [-i si, co]], half the angle of (z, y)
        const long double y = -2 * mul(conj(p[0]), p[2]).imag(), z = norm(p[0]) - norm(p[2]),
                          r = std::sqrt(y * y + z * z);
        long double co = 1.0L, si = 0.0L;
        if (z >= 0 && r > 0) {
          co = std::sqrt((r + z) / (2 * r));
          si = y / (2 * r * co);
        } else if (r > 0) {
          si = std::copysign(std::sqrt((r - z) / (2 * r)), y);
          co = y / (2 * r * si);
        }
        auto turn = [&](cl& u, cl& v, long double t) {  // u, v <- co u + i t v, i t u + co v
          const cl a = u, b = v;
          u = {co * a.real() - t * b.imag(), co * a.imag() + t * b.real()};
          v = {co * b.real() - t * a.imag(), co * b.imag() + t * a.real()};
        };
        turn(p[0], p[2], si);
        turn(p[1], p[3], si);
        turn(q[0], q[1], -si);
        turn(q[2], q[3], -si);
      }
    }
    e.op = (int)i;
    e.between = 0;
  }
  return out;
}

// An op of a pass, with its matrix where it is a one-qubit unitary's.
struct Gate {
  const mlb_op_t* op;
  const Unitary* u;
};

// The pass with its tile filled to `bits` by the lowest qubits outside it.
inline DevPass filled(DevPass p, int bits) {
  for (int q = 0; q < p.n && p.L + p.H < bits; q++)
    if (p.tile_free_mask >> q & 1ull) {
      p.high[p.H++] = q;
      p.tile_free_mask &= ~(1ull << q);
      p.num_tiles >>= 1;
    }
  return p;
}

struct Lower {
  const DevPass& P;
  int dtype, m;
  int local_of[64];
  std::vector<Item> items;
  Fun label[kRotBits];
  uint32_t dir[kRotBits];
  bool full = false;  // the program outgrew shared memory: the rest is not planned

  Lower(const DevPass& pass, int dt) : P(pass), dtype(dt), m(pass.L + pass.H) {
    for (int& x : local_of) x = -1;
    for (int q = 0; q < P.L; q++) local_of[q] = q;
    for (int h = 0; h < P.H; h++) local_of[P.high[h]] = P.L + h;
    for (int i = 0; i < m; i++) {
      label[i].row = 1u << i;
      dir[i] = 1u << i;
    }
  }

  Fun fun(int q) const {
    if (local_of[q] >= 0) return label[local_of[q]];
    Fun f;
    f.out = 1ull << q;
    return f;
  }

  void diag(const std::vector<Fun>& cond, bool keyed, const Fun& key, cl d0, cl d1) {
    if (keyed && cond.empty())  // one on the same functional, with no rotation between that changes it: merged
      for (int i = (int)items.size(); i-- > 0;) {
        Item& it = items[i];
        if (it.rotation) {
          if (hea::parity(key.row & it.dir)) break;
        } else if (it.keyed && it.nc == 0 && it.key.same(key)) {
          const bool x = it.key.c != key.c;
          it.d[0] = mul(it.d[0], x ? d1 : d0);
          it.d[1] = mul(it.d[1], x ? d0 : d1);
          return;
        }
      }
    Item it;
    for (const Fun& f : cond) it.cond[it.nc++] = f;
    it.keyed = keyed;
    it.key = key;
    it.d[0] = d0;
    it.d[1] = d1;
    items.push_back(it);
  }

  void add(const mlb_op_t& o, const Unitary* given) {
    std::vector<Fun> cond;
    for (uint64_t c = o.cmask; c; c &= c - 1) cond.push_back(fun(__builtin_ctzll(c)));
    switch (o.kind) {
      case MLB_OP_X: {
        Fun& f = label[local_of[o.target]];
        if (cond.empty()) {
          f.c = !f.c;
        } else {
          const int c = __builtin_ctzll(o.cmask);
          f.add(cond[0]);
          if (local_of[c] >= 0) dir[local_of[c]] ^= dir[local_of[o.target]];
        }
        return;
      }
      case MLB_OP_SWAP: {
        const int a = local_of[o.target], b = local_of[o.target2];
        std::swap(label[a], label[b]);
        std::swap(dir[a], dir[b]);
        return;
      }
      case MLB_OP_DIAG1: diag(cond, true, fun(o.target), cd(o.m[0], o.m[1]), cd(o.m[2], o.m[3])); return;
      case MLB_OP_PHASE: diag(cond, false, Fun(), 1.0, cd(o.m[0], o.m[1])); return;
      case MLB_OP_ZZ: {
        Fun f = fun(o.target);
        f.add(fun(o.target2));
        diag(cond, true, f, cd(o.m[0], o.m[1]), cd(o.m[2], o.m[3]));
        return;
      }
      default: break;
    }
    const int q = local_of[o.target];
    const Unitary U = given ? *given : unitary(o);
    cl a = U.m[0], b = U.m[1], c = U.m[2], d = U.m[3];
    if (norm(a) < norm(c)) {  // the columns swapped: an X first
      label[q].c = !label[q].c;
      std::swap(a, b);
      std::swap(c, d);
    }
    // a = s u, c = s u t v, d = s u w v: diag(1, v) s [[1, -t], [t, 1]] diag(u, u w).
    // A real c / a needs no diag(1, v) (t takes the sign).
    const long double s = size(a);
    const cl u = a / s, r = mul(c, conj(u)) / s;  // t v
    double t = (double)size(r);
    cl v = 1.0L;
    if (std::abs(r.imag()) <= 2e-17L) t = (double)r.real();
    else v = r / size(r);
    const cl w = mul(mul(d, conj(u)), conj(v)) / size(d);
    diag({}, true, label[q], u, mul(u, w));
    Item it;
    it.rotation = true;
    it.dir = dir[q];
    it.fun = label[q];
    it.t = dtype == MLB_C128 ? t : (double)(float)t;  // as the kernel holds it
    it.s = 1.0L / std::sqrt(1.0L + (long double)it.t * it.t);  // of the rounded t: the rotation keeps norms
    items.push_back(it);
    if (v != cl(1.0L)) diag({}, true, label[q], 1.0L, v);
  }

  // The pass's program, with fewer variants a table where its tables would
  // outgrow shared memory.  False: it does not fit.
  static bool lower(const DevPass& pass, int dtype, const std::vector<Gate>& ops, Program& out) {
    for (int max_var = kRotMaxVar; max_var >= 1; max_var--) {
      Program p;
      if (!Lower(pass, dtype).build(ops, p, max_var)) continue;
      p.dev.entries = (uint32_t)p.table.size();
      out = std::move(p);
      return true;
    }
    return false;
  }

  void order() {
    const int N = (int)items.size();
    struct Turn {
      uint32_t dir, row;
      int i;
    };
    struct Read {  // a functional that diagonal i reads
      uint32_t row;
      int i;
    };
    std::vector<Turn> turns;
    std::vector<Read> reads;
    turns.reserve(N);
    reads.reserve(2 * N);
    auto edge = [&](int i, int j) {
      items[i].succ.add(j);
      items[j].pred.add(i);
    };
    for (int j = 0; j < N; j++) {
      const Item& y = items[j];
      if (y.rotation) {
        const uint32_t dir = y.dir, row = y.fun.row;
        for (const Turn& x : turns)
          if (hea::parity(x.row & dir) || hea::parity(row & x.dir)) edge(x.i, j);
        for (const Read& x : reads)
          if (hea::parity(x.row & dir)) edge(x.i, j);
        turns.push_back({dir, row, j});
      } else {
        const size_t first = reads.size();
        if (y.keyed) reads.push_back({y.key.row, j});
        for (int c = 0; c < y.nc; c++) reads.push_back({y.cond[c].row, j});
        for (const Turn& x : turns)
          for (size_t k = first; k < reads.size(); k++)
            if (hea::parity(reads[k].row & x.dir)) edge(x.i, j);
      }
    }
    for (int i = N; i-- > 0;)
      for (int k = 0; k < kWords; k++)
        for (uint64_t b = items[i].succ.w[k]; b; b &= b - 1) {
          const Item& y = items[64 * k + __builtin_ctzll(b)];
          items[i].height = std::max(items[i].height, y.height + (y.rotation ? 1 : 0));
        }
  }

  // A functional in a segment's coordinates: its value over the register
  // index, and what is left (group index and tile).
  struct Split {
    uint32_t reg = 0, zg = 0;
    uint64_t out = 0;
    bool c = false;
  };

  using Rest = std::pair<uint32_t, uint64_t>;  // (group functional, outside functional)

  // The program of `ops`; a table has up to 2^max_var variants where its ops
  // allow.  False: it does not fit shared memory.
  bool build(const std::vector<Gate>& ops, Program& out, int max_var) {
    long double scale = 1.0L;  // owed by rotations so far
    // what a table's rounding took from the norm, given back by the next one: a
    // table of one scale for all its entries rounds them all alike
    long double owed = 1.0L;
    items.reserve(3 * ops.size());
    for (const Gate& g : ops) add(*g.op, g.u);
    order();
    const int N = (int)items.size(), words = (N + 63) / 64;
    int left = 0;
    for (const Item& it : items) left += it.rotation;
    int diags = N - left;
    RotPass& D = out.dev;
    D.n = P.n;
    D.m = m;
    for (int i = 0; i < m; i++) D.basis[i] = i < P.L ? 1ull << i : 1ull << P.high[i - P.L];
    Set done, turns, reads;  // the rotations and the diagonals
    for (int i = 0; i < N; i++) (items[i].rotation ? turns : reads).add(i);
    auto each_left = [&](const Set& of, auto&& f) {  // in program order
      for (int k = 0; k < words; k++)
        for (uint64_t b = of.w[k] & ~done.w[k]; b; b &= b - 1) f(64 * k + __builtin_ctzll(b));
    };
    auto after = [&](const Item& it, const Set& before) {  // its predecessors lie in `before`
      for (int k = 0; k < words; k++)
        if (it.pred.w[k] & ~before.w[k]) return false;
      return true;
    };
    while (left || diags || scale != 1.0L || out.segs.empty()) {
      if (full) return false;
      // 1. the segment's directions and its rounds; a round's diagonals are
      // those its rotations wait for, `free` the others that could join
      hea::Basis W;
      std::vector<uint32_t> al, rows;
      struct Round {
        std::vector<int> diag, rot, free;
      };
      std::vector<Round> rounds;
      Set marked;
      while (left) {
        std::vector<int> cand;
        Round r;
        Set open = done;  // and the diagonals that can run now
        each_left(reads, [&](int i) {
          if (!after(items[i], done)) return;
          open.add(i);
          r.free.push_back(i);
        });
        each_left(turns, [&](int i) {
          if (after(items[i], open)) cand.push_back(i);
        });
        // a new direction: the rotation that shares the most later ones with
        // the directions so far, then the one that the longest chain waits for
        while ((int)al.size() < 4) {
          int best = -1;
          long most = -1;
          for (int i : cand) {
            if (!W.reduce(items[i].dir)) continue;
            long common = 0;
            for (int k = 0; k < words; k++) common += __builtin_popcountll(items[i].succ.w[k] & marked.w[k]);
            const long score = common * 4096 + items[i].height;
            if (score > most) {
              most = score;
              best = i;
            }
          }
          if (best < 0) break;
          W.add(items[best].dir);
          al.push_back(items[best].dir);
          rows.push_back(items[best].fun.row);
          for (int k = 0; k < words; k++) marked.w[k] |= items[best].succ.w[k];
        }
        for (int i : cand)
          if (!W.reduce(items[i].dir)) r.rot.push_back(i);
        if (r.rot.empty()) break;
        for (int i : r.free)
          for (int j : r.rot)
            if (items[j].pred.has(i)) {
              done.add(i);
              diags--;
              r.diag.push_back(i);
              break;
            }
        for (int i : r.rot) {
          done.add(i);
          left--;
        }
        rounds.push_back(std::move(r));
      }
      for (int b = 0; b < m && (int)al.size() < 4; b++)
        if (W.add(1u << b)) al.push_back(1u << b);
      // 2. the groups: the common kernel of four functionals that are
      // independent on the directions, the rotations' own first
      uint32_t fn[4], mat[4], comb[16];
      int nf = 0;
      {
        hea::Basis rank;
        auto take = [&](uint32_t f) {
          uint32_t v = 0;
          for (int i = 0; i < 4; i++) v |= (uint32_t)hea::parity(f & al[i]) << i;
          if (nf < 4 && rank.add(v)) {
            fn[nf] = f;
            mat[nf++] = v;
          }
        };
        for (uint32_t f : rows) take(f);
        for (int b = 0; b < m; b++) take(1u << b);
      }
      for (uint32_t k = 0; k < 16; k++) {  // combinations of the directions
        comb[k] = 0;
        for (int i = 0; i < 4; i++)
          if (k >> i & 1) comb[k] ^= al[i];
      }
      hea::Basis span;
      std::vector<uint32_t> ker;
      for (int b = 0; b < m; b++)
        for (uint32_t k = 0; k < 16; k++) {  // the unit vector, corrected along the directions
          const uint32_t t = (1u << b) ^ comb[k];
          bool in = true;
          for (int i = 0; i < 4; i++) in = in && !hea::parity(fn[i] & t);
          if (!in) continue;  // one combination of the directions corrects it
          if (span.add(t)) ker.push_back(t);
          break;
        }
      // lanes (the first five group bits) where the tables' variants do not
      // depend on them, so that a warp reads one variant: the common kernel of
      // the rounds' functionals, the commonest first, while it has five dimensions
      std::vector<uint32_t> lanes = ker;
      {
        std::vector<std::pair<int, uint32_t>> seen;
        auto see = [&](const Fun& f) {
          bool rest = false;
          for (uint32_t t : ker) rest = rest || hea::parity(f.row & t);
          if (!rest) return;
          for (auto& x : seen)
            if (x.second == f.row) {
              x.first--;
              return;
            }
          seen.push_back({-1, f.row});
        };
        for (const Round& r : rounds)
          for (int i : r.diag) {
            if (items[i].keyed) see(items[i].key);
            for (int c = 0; c < items[i].nc; c++) see(items[i].cond[c]);
          }
        std::stable_sort(seen.begin(), seen.end(), [](const auto& a, const auto& b) { return a.first < b.first; });
        for (auto& x : seen) {
          std::vector<uint32_t> in;
          uint32_t odd = 0;
          for (uint32_t t : lanes)
            if (!hea::parity(x.second & t)) in.push_back(t);
            else if (!odd) odd = t;
            else in.push_back(t ^ odd);
          if (in.size() >= 5) lanes = in;
        }
      }
      std::vector<uint32_t> kap = hea::bank_order(lanes, dtype);
      {
        hea::Basis have;
        for (uint32_t t : kap) have.add(t);
        for (uint32_t t : ker)
          if (have.add(t)) kap.push_back(t);
      }
      RotSeg sg{};
      for (int i = 0; i < 4; i++) sg.alpha[i] = (uint16_t)hea::slot_bytes(al[i], dtype);
      for (size_t i = 0; i < kap.size(); i++) sg.kappa[i] = (uint16_t)hea::slot_bytes(kap[i], dtype);
      sg.op_begin = (int)out.ops.size();
      // the directions of the register index bits; a round first adds
      // directions to one another (a permutation of the registers) until its
      // rotations move along single bits and read them alone
      uint32_t cur[4] = {al[0], al[1], al[2], al[3]};
      std::vector<uint32_t> steps;  // 4 i + j: direction i += direction j
      auto step = [&](int i, int j) {
        cur[i] ^= cur[j];
        steps.push_back((uint32_t)(4 * i + j));
      };
      auto emit = [&](RotOp op) {  // with the steps before it, up to 8 an op
        while (steps.size() > 8) {
          RotOp more{};
          for (int k = 0; k < 8; k++) more.perm |= steps[k] << (4 * k);
          steps.erase(steps.begin(), steps.begin() + 8);
          out.ops.push_back(more);
        }
        for (size_t k = 0; k < steps.size(); k++) op.perm |= steps[k] << (4 * k);
        steps.clear();
        out.ops.push_back(op);
      };
      auto split = [&](const Fun& f) {
        Split s;
        for (int i = 0; i < 4; i++) s.reg |= (uint32_t)hea::parity(f.row & cur[i]) << i;
        for (size_t j = 0; j < kap.size(); j++) s.zg |= (uint32_t)hea::parity(f.row & kap[j]) << j;
        s.out = f.out;
        s.c = f.c;
        return s;
      };
      // 3. emit: tables of the diagonals, and the rotations
      hea::Basis held;  // functionals that the registers hold alone
      for (int i = 0; i < 4; i++) held.add(fn[i]);
      std::vector<Rest> var;  // the open table's variant functionals
      std::vector<int> open;
      auto combo = [&](const Rest& r) {  // r as a sum of variant functionals, -1: none
        for (uint32_t v = 0; v < (1u << var.size()); v++) {
          Rest x{0, 0};
          for (size_t j = 0; j < var.size(); j++)
            if (v >> j & 1u) {
              x.first ^= var[j].first;
              x.second ^= var[j].second;
            }
          if (x == r) return (int)v;
        }
        return -1;
      };
      auto plain = [&](const Item& d) {
        if (d.keyed && (d.key.out || held.reduce(d.key.row))) return false;
        for (int i = 0; i < d.nc; i++)
          if (d.cond[i].out || held.reduce(d.cond[i].row)) return false;
        return true;
      };
      auto known = [&](const Item& d) {  // read by the registers and the open table's variants
        auto in = [&](const Fun& f) {
          const Split s = split(f);
          return combo({s.zg, s.out}) >= 0;
        };
        bool k = !d.keyed || in(d.key);
        for (int i = 0; i < d.nc && k; i++) k = in(d.cond[i]);
        return k;
      };
      auto put = [&](int i) {  // false: no room for its functionals
        const size_t before = var.size();
        auto need = [&](const Fun& f) {
          const Split s = split(f);
          if (combo({s.zg, s.out}) < 0) var.push_back({s.zg, s.out});
        };
        if (items[i].keyed) need(items[i].key);
        for (int c = 0; c < items[i].nc; c++) need(items[i].cond[c]);
        if (var.size() > (size_t)max_var && !open.empty()) {
          var.resize(before);
          return false;
        }
        open.push_back(i);
        return true;
      };
      auto close = [&](RotOp op) {  // emits op with the open table
        const uint32_t nv = (uint32_t)var.size();
        const size_t at = out.table.size();
        full = full || rot_shared_bytes(dtype, out.ops.size() + 1, at + ((size_t)16 << nv)) > kRotMaxShared;
        if (full) {
          var.clear();
          open.clear();
          scale = 1.0L;
          return;
        }
        out.table.resize(at + ((size_t)16 << nv));
        std::vector<cl> wide((size_t)16 << nv, cl(scale * owed, 0.0L));
        scale = 1.0;
        struct Bit {
          uint32_t reg, v, c;  // patterns over the register index and the variant
          uint32_t row(uint32_t x) const { return (reg ^ (((v >> x) ^ c) & 1u ? 0xffffu : 0u)) & 0xffffu; }  // of variant x
        };
        auto pattern = [](uint32_t f) {
          uint32_t p = 0;
          for (uint32_t k = 0; k < 16; k++) p |= (uint32_t)hea::parity(f & k) << k;
          return p;
        };
        for (int i : open) {
          const Item& d = items[i];
          auto bit = [&](const Fun& f) {
            const Split s = split(f);
            return Bit{pattern(s.reg), pattern((uint32_t)combo({s.zg, s.out})), s.c ? 1u : 0u};
          };
          Bit cond[3];
          for (int c = 0; c < d.nc; c++) cond[c] = bit(d.cond[c]);
          const Bit key = d.keyed ? bit(d.key) : Bit{0, 0, 1};
          for (uint32_t x = 0; x < (1u << nv); x++) {
            uint32_t on = 0xffffu;
            for (int c = 0; c < d.nc; c++) on &= cond[c].row(x);
            for (int b = 0; b < 2; b++)
              if (d.d[b] != cl(1.0L))
                for (uint32_t m = on & (b ? key.row(x) : ~key.row(x)); m; m &= m - 1) {
                  cl& e = wide[16 * x + (uint32_t)__builtin_ctz(m)];
                  e = mul(e, d.d[b]);
                }
          }
        }
        long double off = 0.0L, sum = 0.0L;  // of the rounded entries' squares, halved; of the squares
        for (size_t k = 0; k < wide.size(); k++) {
          const cl w = wide[k];
          const cd e = dtype == MLB_C128 ? cd((double)w.real(), (double)w.imag()) : cd((float)w.real(), (float)w.imag());
          out.table[at + k] = e;
          off += w.real() * (e.real() - w.real()) + w.imag() * (e.imag() - w.imag());
          sum += norm(w);
        }
        owed = std::abs(off / sum) < 1e-6L ? 1.0L - off / sum : 1.0L;
        op.table = (uint32_t)at;
        op.nv = (uint8_t)nv;
        op.flags |= kRotTable;
        for (uint32_t j = 0; j < nv; j++) {
          op.vzg[j] = (uint16_t)var[j].first;
          op.vout[j] = var[j].second;
        }
        emit(op);
        var.clear();
        open.clear();
      };
      // a diagonal on the very functional of a later rotation joins that one's table
      auto later_same = [&](const Item& d) {
        if (d.keyed && d.nc == 0)
          for (int k = 0; k < words; k++)
            for (uint64_t b = d.succ.w[k] & ~done.w[k]; b; b &= b - 1)
              if (items[64 * k + __builtin_ctzll(b)].fun.same(d.key)) return true;
        return false;
      };
      auto join = [&](int i) {
        if (put(i)) {
          done.add(i);
          diags--;
        }
      };
      for (const Round& r : rounds) {
        RotOp op{};
        int place[4] = {-1, -1, -1, -1};  // rotation at each register bit
        for (int i : r.rot)
          for (int b = 0; b < 4; b++)
            if (place[b] < 0 && cur[b] == items[i].dir) {
              place[b] = i;
              break;
            }
        for (int i : r.rot) {
          if (place[0] == i || place[1] == i || place[2] == i || place[3] == i) continue;
          uint32_t x = 0;  // its direction in the current ones
          for (uint32_t k = 1; k < 16; k++) {
            uint32_t v = 0;
            for (int b = 0; b < 4; b++)
              if (k >> b & 1u) v ^= cur[b];
            if (v == items[i].dir) x = k;
          }
          int b = 0;
          while (place[b] >= 0 || !(x >> b & 1u)) b++;
          for (int j = 0; j < 4; j++)
            if (j != b && (x >> j & 1u)) step(b, j);
          place[b] = i;
        }
        for (int b = 0; b < 4; b++)
          for (int j = 0; j < 4; j++)
            if (place[b] < 0 && place[j] >= 0 && hea::parity(items[place[j]].fun.row & cur[b])) step(b, j);
        for (int b = 0; b < 4; b++)
          if (place[b] >= 0) {
            const Item& it = items[place[b]];
            const Split sp = split(it.fun);
            op.t[b] = sp.c ? -it.t : it.t;
            op.tzg[b] = (uint16_t)sp.zg;
            op.tout[b] = sp.out;
            op.flags |= kRotTurn;
          }
        for (int i : r.diag)
          if (!put(i)) {
            close(RotOp{});
            put(i);
          }
        for (int i : r.rot) scale *= items[i].s;
        if (!open.empty())  // the table is paid for: others that may run now, with no variant more
          for (int i : r.free)
            if (!done.has(i) && !later_same(items[i]) && known(items[i])) join(i);
        if (!open.empty() || scale != 1.0L) close(op);
        else emit(op);
      }
      // what the registers hold now goes here; with no rotation left, all of it
      do {
        std::vector<int> now;
        each_left(reads, [&](int i) {
          if (after(items[i], done) && !later_same(items[i])) now.push_back(i);
        });
        for (int form = 0; form < 2; form++)
          for (int i : now)
            if (!done.has(i) && plain(items[i]) == (form == 0) && (form == 0 || left == 0 || (!open.empty() && known(items[i]))))
              join(i);
        if (!open.empty()) close(RotOp{});
      } while (!left && diags);
      for (int i = 0; i < 4; i++) sg.alpha_out[i] = (uint16_t)hea::slot_bytes(cur[i], dtype);
      sg.op_end = (int)out.ops.size();
      out.segs.push_back(sg);
    }
    if (full || rot_shared_bytes(dtype, out.ops.size(), out.table.size()) > kRotMaxShared) return false;
    D.num_ops = (int)out.ops.size();
    D.num_segs = (int)out.segs.size();
    for (int i = 0; i < m; i++) {
      D.dir_slot[i] = (uint16_t)hea::slot_bytes(dir[i], dtype);
      D.label_out[i] = label[i].out;
      if (label[i].c) D.label_const |= 1u << i;
    }
    return true;
  }
};

}  // namespace rot
}  // namespace mlb
