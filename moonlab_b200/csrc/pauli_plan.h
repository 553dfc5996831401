// pauli_plan.h -- plans a sum of Pauli strings as tile passes over linear
// subspaces of the index space (kernels_pauli.cu).  Host-only.
//
// P_k |i> = i^{ny} (-1)^{|i & z|} |i ^ x>: a string pairs i with i ^ x, so a
// tile base ^ span(u_0 .. u_{m-1}) holds both amplitudes of every string
// whose X mask lies in the span.  The first L basis vectors are the low unit
// vectors (rows of 2^L contiguous amplitudes); the others are X masks, chosen
// to cover as many of the remaining strings as possible, whatever qubits
// they touch.  Inside a pass, a segment holds groups of 8 amplitudes in
// registers along three directions and takes the strings whose mask is one
// of their 8 combinations, so a tile is read once per ~3 masks.
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "hea_plan.h"
#include "mlb_internal.h"

namespace mlb {
namespace pauli {

struct Pass {
  PauliPass dev{};
  std::vector<PauliSeg> segs;
  std::vector<PauliTerm> terms;
  size_t segs_off = 0, terms_off = 0;  // in the caller's device arrays
};

// Greedy: masks added to V (up to `dims` vectors), each the one that brings
// the most strings into the span with it; among equals, the one whose qubits
// the most masks touch.  masks: sorted, with their numbers of strings.
inline void grow(hea::Basis& V, const std::vector<uint64_t>& masks, const std::vector<int>& weight, int dims) {
  int degree[64] = {};
  for (uint64_t x : masks)
    for (uint64_t y = x; y; y &= y - 1) degree[__builtin_ctzll(y)]++;
  // the masks modulo the span: equal residues come in together
  std::vector<uint64_t> res;
  std::vector<int> strings;
  for (size_t i = 0; i < masks.size(); i++)
    if (const uint64_t r = V.reduce(masks[i])) {
      res.push_back(r);
      strings.push_back(weight[i]);
    }
  struct Class {
    uint64_t r;
    long gain;
  };
  std::vector<Class> classes;
  int log = 4;
  while ((size_t)1 << log < 2 * res.size()) log++;
  std::vector<uint32_t> slot((size_t)1 << log);  // hash table: 1 + index of a class
  while ((int)V.v.size() < dims && !res.empty()) {
    classes.clear();
    std::fill(slot.begin(), slot.end(), 0u);
    for (size_t i = 0; i < res.size(); i++) {
      size_t h = (res[i] * 0x9E3779B97F4A7C15ull) >> (64 - log);
      while (slot[h] && classes[slot[h] - 1].r != res[i]) h = (h + 1) & (slot.size() - 1);
      if (!slot[h]) {
        classes.push_back({res[i], 0});
        slot[h] = (uint32_t)classes.size();
      }
      classes[slot[h] - 1].gain += strings[i];
    }
    uint64_t best = 0;
    long most = 0, score = -1;
    for (const Class& c : classes) {
      if (c.gain < most) continue;
      long touch = 0;
      for (uint64_t y = c.r; y; y &= y - 1) touch += degree[__builtin_ctzll(y)];
      const long t = (touch << 8) / __builtin_popcountll(c.r);
      if (c.gain > most || t > score || (t == score && c.r < best)) {
        most = c.gain;
        score = t;
        best = c.r;
      }
    }
    V.add(best);
    const int pivot = __builtin_ctzll(best);
    size_t left = 0;
    for (size_t i = 0; i < res.size(); i++) {
      const uint64_t r = res[i] >> pivot & 1ull ? res[i] ^ best : res[i];
      if (!r) continue;
      res[left] = r;
      strings[left++] = strings[i];
    }
    res.resize(left);
    strings.resize(left);
  }
}

constexpr int kTilesLog = 9, kSmallTile = 6;  // of a small state: tiles (log2), a tile's least bits

// `lambda`: the strings of a lambda pass (out[i ^ x] += c i^{ny} ... in[i]),
// else of an expectation value.
inline void plan(int n, int TB, int L, int dtype, size_t num, const uint64_t* xm, const uint64_t* zm,
                 const double* coeff, bool lambda, std::vector<Pass>& out) {
  const int most = std::min(n, TB);
  L = std::min(L, most);
  std::vector<size_t> rem(num);
  for (size_t i = 0; i < num; i++) rem[i] = i;
  std::stable_sort(rem.begin(), rem.end(), [&](size_t a, size_t b) { return xm[a] < xm[b]; });
  while (!rem.empty()) {
    std::vector<uint64_t> masks;
    std::vector<int> weight;
    for (size_t i : rem)
      if (xm[i]) {
        if (masks.empty() || masks.back() != xm[i]) {
          masks.push_back(xm[i]);
          weight.push_back(0);
        }
        weight.back()++;
      }
    hea::Basis V;
    for (int b = 0; b < L; b++) V.add(1ull << b);
    // An expectation value of a small state takes smaller tiles where its
    // strings' masks leave room, up to 512 of them, so that more than a few
    // CTAs share them (one string on 12 to 18 qubits: 39 us, 42 with full tiles).
    int fill = most;
    if (!lambda && most > kSmallTile && n - kTilesLog < most && masks.size() < (size_t)most)
      fill = std::max(n - kTilesLog, kSmallTile);
    if (n > most || fill < most) grow(V, masks, weight, most);
    for (int b = 0; b < n && (int)V.v.size() < fill; b++) V.add(1ull << b);
    const int m = (int)V.v.size();
    std::vector<size_t> take, left;
    for (size_t i : rem) (take.size() < (size_t)kMaxPauliTerms && !V.reduce(xm[i]) ? take : left).push_back(i);
    Pass P;
    P.dev.n = n;
    P.dev.m = m;
    uint64_t pivots = 0;
    for (int b = 0; b < m; b++) {
      P.dev.basis[b] = V.v[b];
      pivots |= 1ull << V.piv[b];
    }
    P.dev.free_mask = ((1ull << n) - 1ull) & ~pivots;
    P.dev.tiles_per_state = 1ull << (n - m);
    while (!take.empty()) {
      // three directions of this segment, in the tile's local coordinates
      std::vector<uint64_t> loc;
      std::vector<int> w;
      for (size_t i : take)
        if (xm[i]) {
          const uint64_t t = V.coords(xm[i]);
          if (loc.empty() || loc.back() != t) {
            loc.push_back(t);
            w.push_back(0);
          }
          w.back()++;
        }
      hea::Basis R;
      grow(R, loc, w, 3);
      for (int b = m; b-- > 0 && (int)R.v.size() < 3;) R.add(1ull << b);
      PauliSeg s{};
      for (int i = 0; i < 3; i++) s.alpha[i] = (uint16_t)hea::slot_bytes((uint32_t)R.v[i], dtype);
      // groups: a complement of the three directions, lanes on distinct banks first
      std::vector<uint32_t> comp;
      {
        hea::Basis full = R;
        for (int b = 0; b < m; b++)
          if (full.add(1ull << b)) comp.push_back(1u << b);
      }
      const std::vector<uint32_t> order = hea::bank_order(comp, dtype);
      for (size_t i = 0; i < order.size(); i++) s.kappa[i] = (uint16_t)hea::slot_bytes(order[i], dtype);
      auto global = [&](uint64_t t) {
        uint64_t g = 0;
        for (int b = 0; b < m; b++)
          if (t >> b & 1ull) g ^= V.v[b];
        return g;
      };
      s.term_begin = (int)P.terms.size();
      std::vector<size_t> later;
      for (size_t i : take) {
        const uint64_t t = V.coords(xm[i]);
        if (R.reduce(t)) {
          later.push_back(i);
          continue;
        }
        PauliTerm d{};
        d.z = zm[i];
        d.kap = (uint8_t)R.coords(t);
        for (int k = 0; k < 8; k++) {
          uint64_t g = 0;
          for (int j = 0; j < 3; j++)
            if (k >> j & 1) g ^= global(R.v[j]);
          if (hea::parity(g & zm[i])) d.pat |= (uint8_t)(1u << k);
        }
        for (size_t j = 0; j < order.size(); j++)
          if (hea::parity(global(order[j]) & zm[i])) d.zg |= (uint16_t)(1u << j);
        const int ny = __builtin_popcountll(xm[i] & zm[i]) & 3;
        const double c = coeff ? coeff[i] : 1.0;
        if (ny & 1) d.kap |= 8;
        if (lambda) {
          d.c = ny >= 2 ? -c : c;  // i^{ny}: 1, i, -1, -i
        } else {
          // both members of a pair, i the one kept: 2 s(i) {re, -im, -re, im}
          d.c = (xm[i] ? 2.0 : 1.0) * (ny == 1 || ny == 2 ? -c : c);
        }
        P.terms.push_back(d);
      }
      s.term_end = (int)P.terms.size();
      P.segs.push_back(s);
      take.swap(later);
    }
    P.dev.num_segs = (int)P.segs.size();
    P.dev.num_terms = (int)P.terms.size();
    out.push_back(std::move(P));
    rem.swap(left);
  }
}

}  // namespace pauli
}  // namespace mlb
