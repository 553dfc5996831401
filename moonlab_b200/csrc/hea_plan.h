// hea_plan.h -- plans the rotation sweeps of the hardware-efficient ansatz
// (kernels_adjoint.cu, k_hea) as tile passes over linear subspaces of the
// index space.  Host-only.
//
// A layer is RY, RZ on every qubit and a CNOT ladder.  The ladder permutes
// amplitudes by a linear map of the index over GF(2), y = C x with
// y_q = x_0 ^ ... ^ x_q, so it is never carried out: an amplitude stays where
// it is and the rotations of layer l act in relabelled coordinates.  With p
// the index after the last layer, the index at layer l is x = C^-k p, where
// k ladders follow; a rotation of qubit q there
//   * pairs p with p ^ a, a = C^k e_q (its direction), and
//   * has its target bit at parity(r & p), r = row q of C^-k (its functional).
// Two rotations commute when neither's direction changes the other's bit.
//
// A pass takes tiles p = base ^ span(u_0 .. u_{m-1}): the first L basis
// vectors are the low unit vectors (rows of 2^L contiguous amplitudes), the
// others are chosen so that as many rotations as possible have their
// direction in the span.  Rotations of neighbouring qubits in successive
// layers share directions (layer l + 1's differ from layer l's by one
// neighbour), so a pass takes a band of several layers: s layers on n qubits
// need about (n + s) / (m - L - s + 1) passes instead of two per layer.
//
// Inside a pass, segments of three rotations that commute with each other
// run on groups of 8 amplitudes, whose register index is the three target
// bits (unused places hold idle directions).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "mlb_internal.h"

namespace mlb {
namespace hea {

inline int parity(uint64_t x) { return __builtin_parityll(x); }

// y = C x on the low `nr` bits (the register's real qubits), others unchanged
inline uint64_t ladder(uint64_t x, int nr) {
  const uint64_t real = (1ull << nr) - 1ull;
  uint64_t z = x & real;
  for (int s = 1; s < nr; s <<= 1) z ^= z << s;
  return (z & real) | (x & ~real);
}
// functional of C^-1 composed with r: x_q = y_q ^ y_{q-1}
inline uint64_t unladder_functional(uint64_t r, int nr) {
  const uint64_t real = (1ull << nr) - 1ull;
  return r ^ ((r & real & ~1ull) >> 1);
}

struct Rot {
  int layer, q;
  int p;            // parameter of its RY; its RZ is p + 1
  uint64_t dir;     // direction a
  uint64_t fun;     // functional r
};

inline bool conflict(const Rot& x, const Rot& y) { return parity(x.fun & y.dir) || parity(y.fun & x.dir); }

// A list of at most 64 entries in place.
template <typename T>
struct Few {
  T at[64];
  size_t count = 0;
  size_t size() const { return count; }
  void push_back(T x) { at[count++] = x; }
  T& operator[](size_t i) { return at[i]; }
  const T& operator[](size_t i) const { return at[i]; }
  T* begin() { return at; }
  T* end() { return at + count; }
  const T* begin() const { return at; }
  const T* end() const { return at + count; }
};

// Reduced basis of a subspace: basis[i] has pivot bit piv[i] and zeros at
// every other pivot.
struct Basis {
  Few<uint64_t> v;
  Few<int> piv;
  uint64_t reduce(uint64_t x) const {
    for (size_t i = 0; i < v.size(); i++)
      if (x >> piv[i] & 1ull) x ^= v[i];
    return x;
  }
  bool add(uint64_t x) {  // false: already inside
    x = reduce(x);
    if (!x) return false;
    const int b = __builtin_ctzll(x);
    for (auto& w : v)
      if (w >> b & 1ull) w ^= x;
    v.push_back(x);
    piv.push_back(b);
    return true;
  }
  uint32_t coords(uint64_t x) const {  // of a vector inside the span
    uint32_t t = 0;
    for (size_t i = 0; i < v.size(); i++)
      if (x >> piv[i] & 1ull) t |= 1u << i;
    return t;
  }
};

struct Pass {
  HeaPass dev{};
  std::vector<HeaSeg> segs;
  Basis basis;
  size_t segs_off = 0;  // in the problem's device array
  size_t slots_off = 0; // backward: first gradient slot of the pass in its group
};

// Byte offset in the tile's shared memory of local index t: 16-byte units
// (one complex128 or two complex64 amplitudes) under the tile swizzle.
inline uint32_t slot_bytes(uint32_t t, int dtype) {
  return dtype == MLB_C128 ? tile_swz16(t) * 16u : tile_swz16(t >> 1) * 16u + (t & 1u) * 8u;
}
// The bits of that offset that choose the shared-memory bank group of one
// lane's access (8 groups of 16 bytes, or 16 of 8 bytes).
inline uint32_t bank_of(uint32_t t, int dtype) {
  const uint32_t b = slot_bytes(t, dtype);
  return dtype == MLB_C128 ? (b >> 4) & 7u : (b >> 3) & 15u;
}

// A basis of span(vecs) whose first vectors (the lanes of one access phase)
// reach distinct bank groups where the span allows.
inline std::vector<uint32_t> bank_order(const std::vector<uint32_t>& vecs, int dtype) {
  const size_t want = dtype == MLB_C128 ? 3 : 4;
  std::vector<uint32_t> order;
  uint32_t bank[32], reached = 1;  // bit b: bank group b is a sum of the chosen vectors' (linear in them)
  for (size_t i = 0; i < vecs.size(); i++) bank[i] = bank_of(vecs[i], dtype);
  auto consider = [&](uint32_t t, uint32_t b) {
    if (order.size() == want || (reached >> b & 1u)) return;
    uint32_t more = reached;
    for (uint32_t x = 0; x < 16; x++)
      if (reached >> x & 1u) more |= 1u << (x ^ b);
    reached = more;
    order.push_back(t);
  };
  // single vectors and sums of two and three, in the order of their sets as binary numbers
  for (size_t i = 0; i < vecs.size() && order.size() < want; i++) {
    consider(vecs[i], bank[i]);
    for (size_t j = 0; j < i; j++) {
      consider(vecs[i] ^ vecs[j], bank[i] ^ bank[j]);
      for (size_t k = 0; k < j; k++) consider(vecs[i] ^ vecs[j] ^ vecs[k], bank[i] ^ bank[j] ^ bank[k]);
    }
  }
  Basis chosen;
  for (uint32_t t : order) chosen.add(t);
  for (uint32_t t : vecs)
    if (chosen.add(t)) order.push_back(t);
  return order;
}

// One segment: the rotations `rot` (at most 3, mutually commuting) in the
// pass's local coordinates.
inline HeaSeg lower_segment(const std::vector<const Rot*>& rot, const Basis& B, int m, int dtype) {
  HeaSeg s{};
  uint32_t al[3], rho[3];
  for (int i = 0; i < 3; i++) s.param[i] = -1;
  int k = 0;
  for (const Rot* g : rot) {
    al[k] = B.coords(g->dir);
    rho[k] = 0;
    for (int b = 0; b < m; b++)
      if (parity(g->fun & B.v[b])) rho[k] |= 1u << b;
    s.fun[k] = (uint32_t)g->fun;
    s.param[k] = g->p;
    k++;
  }
  for (; k < 3; k++) {
    // an idle place: a direction in the kernel of the functionals so far, and
    // a functional that is 1 on it and 0 on the directions so far.  Its sign
    // over the tile's base is free (fun = 0: register index 0 at parity 0).
    for (int b = 0; b < m; b++) {
      uint32_t a = 1u << b;
      for (int i = 0; i < k; i++)
        if (parity(rho[i] & (1u << b))) a ^= al[i];
      if (!a) continue;
      const int c = __builtin_ctz(a);
      uint32_t r = 1u << c;
      for (int i = 0; i < k; i++)
        if (al[i] >> c & 1u) r ^= rho[i];
      if (!parity(r & a)) continue;
      al[k] = a;
      rho[k] = r;
      break;
    }
  }
  for (int i = 0; i < 3; i++) s.alpha[i] = (uint16_t)slot_bytes(al[i], dtype);
  // a basis of the common kernel of the three functionals: the groups'
  // representatives.  Unit vectors projected onto it span it; the lanes' bits
  // come first, chosen so that one access phase hits distinct banks.
  std::vector<uint32_t> ker;
  Basis kb;
  for (int b = 0; b < m; b++) {
    uint32_t t = 1u << b;
    for (int i = 0; i < 3; i++)
      if (rho[i] >> b & 1u) t ^= al[i];
    if (kb.add(t)) ker.push_back(t);
  }
  const std::vector<uint32_t> order = bank_order(ker, dtype);
  for (size_t i = 0; i < order.size(); i++) s.kappa[i] = (uint16_t)slot_bytes(order[i], dtype);
  return s;
}

// Plans `rots` (program order of the sweep) as passes of 2^min(n, TB)
// amplitudes.  L: contiguous low bits of a tile.
inline void plan(const std::vector<Rot>& rots, int n, int TB, int L, int dtype, std::vector<Pass>& out) {
  const int m = std::min(n, TB);
  L = std::min(L, m);
  // two candidate orders, both topological: as given, and by bands of
  // q + layer (a band is what a later band's rotations wait for)
  std::vector<int> rem[2];
  for (size_t i = 0; i < rots.size(); i++) rem[0].push_back((int)i);
  rem[1] = rem[0];
  {
    const bool descending = !rots.empty() && rots.front().layer > rots.back().layer;
    auto key = [&](int i) { return rots[i].q + rots[i].layer; };
    std::stable_sort(rem[1].begin(), rem[1].end(),
                     [&](int a, int b) { return descending ? key(a) > key(b) : key(a) < key(b); });
  }
  while (!rem[0].empty()) {
    std::vector<int> best_take;
    Basis best_basis;
    for (const std::vector<int>& order : rem) {
      Basis V;
      for (int b = 0; b < L; b++) V.add(1ull << b);
      // a rotation waits for the skipped ones that it does not commute with:
      // it commutes with all where its functional vanishes on the span of
      // their directions and theirs on its direction (both orders are
      // topological, so that none of them comes after it in the sweep)
      std::vector<int> take;
      Basis dirs, funs;
      for (int i : order) {
        if ((int)take.size() == 3 * kMaxHeaSegs || dirs.v.size() == (size_t)n || funs.v.size() == (size_t)n) break;
        bool ok = true;
        for (size_t j = 0; ok && j < dirs.v.size(); j++) ok = !parity(rots[i].fun & dirs.v[j]);
        for (size_t j = 0; ok && j < funs.v.size(); j++) ok = !parity(funs.v[j] & rots[i].dir);
        if (ok && V.reduce(rots[i].dir)) {
          if ((int)V.v.size() < m) V.add(rots[i].dir);
          else ok = false;
        }
        if (ok) {
          take.push_back(i);
        } else {
          dirs.add(rots[i].dir);
          funs.add(rots[i].fun);
        }
      }
      if (take.size() > best_take.size()) {
        best_take = take;
        best_basis = V;
      }
    }
    for (int b = 0; b < n && (int)best_basis.v.size() < m; b++) best_basis.add(1ull << b);
    Pass P;
    P.basis = best_basis;
    P.dev.n = n;
    P.dev.m = m;
    uint64_t pivots = 0;
    for (int b = 0; b < m; b++) {
      P.dev.basis[b] = (uint32_t)P.basis.v[b];
      pivots |= 1ull << P.basis.piv[b];
    }
    P.dev.free_mask = ((1ull << n) - 1ull) & ~pivots;
    P.dev.tiles_per_state = 1ull << (n - m);
    // segments by list scheduling: any rotations that wait for none are
    // mutually commuting; those that the most others wait for go first
    std::sort(best_take.begin(), best_take.end());
    const size_t N = best_take.size();
    std::vector<int> waits(N, 0), height(N, 0);
    std::vector<std::vector<int>> after(N);
    for (size_t i = 0; i < N; i++)
      for (size_t j = i + 1; j < N; j++)
        if (conflict(rots[best_take[i]], rots[best_take[j]])) {
          after[i].push_back((int)j);
          waits[j]++;
        }
    for (size_t i = N; i-- > 0;)
      for (int j : after[i]) height[i] = std::max(height[i], height[j] + 1);
    std::vector<char> done(N, 0);
    size_t left = N;
    while (left && (int)P.segs.size() < kMaxHeaSegs) {
      std::vector<int> ready;
      for (size_t i = 0; i < N; i++)
        if (!done[i] && !waits[i]) ready.push_back((int)i);
      std::stable_sort(ready.begin(), ready.end(), [&](int a, int b) { return height[a] > height[b]; });
      if (ready.size() > 3) ready.resize(3);
      std::vector<const Rot*> seg;
      for (int i : ready) {
        seg.push_back(&rots[best_take[i]]);
        done[i] = 1;
        left--;
        for (int j : after[i]) waits[j]--;
      }
      P.segs.push_back(lower_segment(seg, P.basis, m, dtype));
    }
    P.dev.num_segs = (int)P.segs.size();
    std::vector<char> gone(rots.size(), 0);
    for (size_t i = 0; i < N; i++)
      if (done[i]) gone[best_take[i]] = 1;
    for (std::vector<int>& r : rem) r.erase(std::remove_if(r.begin(), r.end(), [&](int i) { return gone[i]; }), r.end());
    out.push_back(std::move(P));
  }
}

}  // namespace hea
}  // namespace mlb
