// QAOA passes over two register groups (complex64 and float-float): device
// bodies shared by the single-instance kernels (qpair.cu) and the batch's
// multi-instance passes (waves.cu), and the pass lists.
//
// The arithmetic is that of the warp-tile kernels (qaoa.cu k_qaoaw,
// adjoint.cu k_adjw) operation for operation: a warp holds 32 lanes (global
// bits 0..4) x 2^RB registers (a group of high bits) and applies the mixer
// bit by bit in the same order, with the gradient terms of one warp sub-tile
// and group summed together.  Here the 2^RB warps of a CTA hold the sub-tiles
// that differ in a second group's bits, so after the first group the CTA
// exchanges registers with warps through shared memory and goes on with the
// second: a pass over two groups reads and writes the state once.  At a layer
// boundary it runs both groups, the cost layer, and both groups of the next
// layer in reverse.
#pragma once
#include <cstdint>
#include <vector>

#include "engine.cuh"

namespace qf {

constexpr int PAIR_MAX_RB = 4;

// One pass.  Register set X is worked on first before the cost layer and last
// after it, Y in between; without `pair` only Y is.
struct PairPass {
  int32_t inst, block_begin, prow;       // batch: instance, first block, first partial row
  int8_t pair, init, cost, hasA, hasB;
  int8_t lanesA;                         // mixer A starts with the lane bits
  int8_t nx, ny;                         // bits acted on in X and Y
  int16_t layerA, layerB;
  uint8_t x[PAIR_MAX_RB], y[PAIR_MAX_RB];  // global bit of each register index bit
  uint8_t s[2 * PAIR_MAX_RB];              // both, ascending
};

// sets used by the pass lists: groups of RB high bits as the warp-tile
// kernels form them, the last one padded with the lowest bits outside it
struct PairGroups {
  std::vector<std::vector<int>> bits;  // padded to RB
  std::vector<int> nact;
};
inline PairGroups pair_groups(int n, int RB) {
  PairGroups g;
  for (int b = 5; b < n; b += RB) {
    std::vector<int> v;
    for (int k = b; k < std::min(n, b + RB); ++k) v.push_back(k);
    g.nact.push_back((int)v.size());
    for (int k = 5; k < n && (int)v.size() < RB; ++k)
      if (std::find(v.begin(), v.end(), k) == v.end()) v.push_back(k);
    g.bits.push_back(v);
  }
  return g;
}
// runs of one or two consecutive groups with disjoint registers
inline std::vector<std::vector<int>> pair_runs(const PairGroups& g) {
  std::vector<std::vector<int>> runs;
  const int m = (int)g.bits.size();
  for (int i = 0; i < m;) {
    bool two = i + 1 < m;
    if (two)
      for (int b : g.bits[i]) two = two && std::find(g.bits[i + 1].begin(), g.bits[i + 1].end(), b) == g.bits[i + 1].end();
    runs.push_back(two ? std::vector<int>{i, i + 1} : std::vector<int>{i});
    i += two ? 2 : 1;
  }
  return runs;
}
// a pass over `run` in the order first, second (second -1: one group)
inline PairPass pair_pass(int n, int RB, const PairGroups& g, int first, int second) {
  PairPass P{};
  P.pair = second >= 0;
  const int y = second >= 0 ? second : first;
  std::vector<int> yb = g.bits[y], xb;
  P.ny = (int8_t)g.nact[y];
  if (P.pair) {
    xb = g.bits[first];
    P.nx = (int8_t)g.nact[first];
  } else {  // the warps' sub-tiles differ in the lowest other bits
    for (int k = 5; k < n && (int)xb.size() < RB; ++k)
      if (std::find(yb.begin(), yb.end(), k) == yb.end()) xb.push_back(k);
  }
  std::vector<int> all = xb;
  all.insert(all.end(), yb.begin(), yb.end());
  std::sort(all.begin(), all.end());
  for (int j = 0; j < RB; ++j) {
    P.x[j] = (uint8_t)xb[j];
    P.y[j] = (uint8_t)yb[j];
  }
  for (int j = 0; j < 2 * RB; ++j) P.s[j] = (uint8_t)all[j];
  return P;
}
// smallest n of the forward passes (a whole tile); the adjoint ones want two
// runs of groups, one qubit more
inline int pair_min_qubits(int RB) { return 5 + 2 * RB; }

// forward passes: |+>^n and p layers
inline std::vector<PairPass> pair_fwd_passes(int n, int p, int RB) {
  const PairGroups g = pair_groups(n, RB);
  const auto runs = pair_runs(g);
  const int m = (int)runs.size();
  std::vector<PairPass> out;
  auto make = [&](int run, bool up) {
    const auto& r = runs[run];
    if (r.size() == 1) return pair_pass(n, RB, g, r[0], -1);
    return up ? pair_pass(n, RB, g, r[0], r[1]) : pair_pass(n, RB, g, r[1], r[0]);
  };
  PairPass f = make(0, false);  // layer 0 starts upwards: its first group is Y
  f.init = f.cost = f.hasB = 1;
  out.push_back(f);
  for (int l = 1; m == 1 && l < p; ++l) {  // the tile is the state: a pass per layer
    PairPass a = make(0, (l & 1) != 0);
    a.cost = a.hasB = 1;
    a.layerB = (int16_t)l;
    out.push_back(a);
  }
  for (int l = 0; l < p; ++l)
    for (int k = 1; k < m; ++k) {
      const bool up = (l & 1) == 0;
      PairPass a = make(up ? k : m - 1 - k, up);
      a.hasA = 1;
      a.layerA = (int16_t)l;
      if (k == m - 1 && l + 1 < p) {
        a.cost = a.hasB = 1;
        a.layerB = (int16_t)(l + 1);
      }
      out.push_back(a);
    }
  return out;
}
// adjoint passes; layerA's cost layer is undone in its last one
inline std::vector<PairPass> pair_adj_passes(int n, int p, int RB) {
  const PairGroups g = pair_groups(n, RB);
  const auto runs = pair_runs(g);
  const int m = (int)runs.size();
  std::vector<PairPass> out;
  for (int l = p - 1; l >= 0; --l) {
    const bool up = ((p - 1 - l) & 1) == 0;
    for (int k = l == p - 1 ? 0 : 1; k < m; ++k) {
      const auto& r = runs[up ? k : m - 1 - k];
      PairPass a = r.size() == 1 ? pair_pass(n, RB, g, r[0], -1)
                   : up          ? pair_pass(n, RB, g, r[0], r[1])
                                 : pair_pass(n, RB, g, r[1], r[0]);
      a.hasA = 1;
      a.init = out.empty();
      a.lanesA = out.empty();
      a.layerA = (int16_t)l;
      a.cost = k == m - 1;
      a.hasB = k == m - 1 && l > 0;
      a.layerB = (int16_t)(l - 1);
      out.push_back(a);
    }
  }
  return out;
}

#ifdef __CUDACC__
template <int LAY, int RB>
struct PairShape {
  using E = typename Types<LAY>::E;
  static constexpr int R = 1 << RB, NT = 32 * R;
  static constexpr size_t VEC = (size_t)NT * R * sizeof(E);  // one vector's tile
};

// geometry of a pass for one thread
template <int RB>
struct PairTile {
  uint32_t bx[RB], by[RB];  // global offset of each register index bit
  uint32_t wx, wy;          // this warp's index in X (while Y is in registers) and in Y
  const PairPass& F;
  QF_D PairTile(const PairPass& f, int warp) : wx(0), wy(0), F(f) {
#pragma unroll
    for (int j = 0; j < RB; ++j) {
      bx[j] = 1u << F.x[j];
      by[j] = 1u << F.y[j];
      if ((warp >> j) & 1) {
        wx |= bx[j];
        wy |= by[j];
      }
    }
  }
  static QF_D uint32_t off(const uint32_t (&b)[RB], int r) {  // r is a constant after unrolling
    uint32_t o = 0;
#pragma unroll
    for (int j = 0; j < RB; ++j)
      if ((r >> j) & 1) o |= b[j];
    return o;
  }
  QF_D uint32_t offx(int r) const { return off(bx, r); }
  QF_D uint32_t offy(int r) const { return off(by, r); }
  QF_D uint32_t base(uint32_t tile, int lane) const {
    uint32_t b = tile << 5;
#pragma unroll
    for (int j = 0; j < 2 * RB; ++j) b = insert0(b, (int)F.s[j]);
    return b | lane;
  }
};

// swap the roles of registers and warps (both are indices 0..R-1)
template <int LAY, int RB>
QF_D void pair_exchange(typename Types<LAY>::E (&a)[1 << RB], typename Types<LAY>::E* work, int lane, int warp) {
  constexpr int R = 1 << RB;
  __syncthreads();  // the buffer's previous readers are done
#pragma unroll
  for (int r = 0; r < R; ++r) work[(warp * R + r) * 32 + lane] = a[r];
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r) a[r] = work[(r * R + warp) * 32 + lane];
}

template <int RB, typename E>
QF_D void pair_rx(const Coef& c, const Coef& s, bool lanes, int nact, E (&a)[1 << RB]) {
  constexpr int R = 1 << RB;
  if (lanes) {
    for (int b = 0; b < 5; ++b) {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = rx_one(c, s, a[r], shfl_xor(a[r], 1 << b));
    }
  }
#pragma unroll
  for (int j = 0; j < RB; ++j) {
    if (j < nact) {
#pragma unroll
      for (int i = 0; i < R / 2; ++i) {
        const int i0 = ((i >> j) << (j + 1)) | (i & ((1 << j) - 1));
        const int i1 = i0 | (1 << j);
        const E a0 = a[i0];
        a[i0] = rx_one(c, s, a0, a[i1]);
        a[i1] = rx_one(c, s, a[i1], a0);
      }
    }
  }
}

// mixer on both vectors with its gradient terms: each bit's reduction
// precedes its own RX(-beta); complex64 sums a sub-tile's terms in FP32 and
// adds that partial to the compensated accumulator once
template <int LAY, int RB, typename E>
QF_D void pair_mix(const Coef& c, const Coef& s, bool lanes, int nact, E (&a)[1 << RB], E (&l)[1 << RB], FFAcc& acc) {
  constexpr int R = 1 << RB;
  constexpr bool F32 = LAY == C64;
  float part = 0.f;
  auto redx = [&](const E& lv, const E& pv) {
    if constexpr (F32) {
      part = fmaf(lv.x, pv.y, part);
      part = fmaf(-lv.y, pv.x, part);
    } else {
      redx_acc(acc, lv, pv);
    }
  };
  if (lanes) {
    for (int b = 0; b < 5; ++b) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const E pa = shfl_xor(a[r], 1 << b);
        const E pl = shfl_xor(l[r], 1 << b);
        redx(l[r], pa);
        a[r] = rx_one(c, s, a[r], pa);
        l[r] = rx_one(c, s, l[r], pl);
      }
    }
  }
#pragma unroll
  for (int j = 0; j < RB; ++j) {
    if (j < nact) {
#pragma unroll
      for (int i = 0; i < R / 2; ++i) {
        const int i0 = ((i >> j) << (j + 1)) | (i & ((1 << j) - 1));
        const int i1 = i0 | (1 << j);
        redx(l[i0], a[i1]);
        redx(l[i1], a[i0]);
        const E a0 = a[i0], l0 = l[i0];
        a[i0] = rx_one(c, s, a0, a[i1]);
        a[i1] = rx_one(c, s, a[i1], a0);
        l[i0] = rx_one(c, s, l0, l[i1]);
        l[i1] = rx_one(c, s, l[i1], l0);
      }
    }
  }
  if constexpr (F32) acc.add(part, 0.f);
}

// PREF: the next tile's amplitudes are fetched into thread-private slots while
// a tile is worked on; else two CTAs per SM overlap each other's loads, which
// the tile of 2^13 complex64 amplitudes leaves room for only without the
// slots (32 graphs of 20 qubits, p = 6: 3474 us an evaluation with them, 2961
// without; float-float, whose tiles are smaller, the other way round).
// Forward pass over the tiles first, first + stride, ... < ntiles.  ac .. bs:
// RX of mixer A and B; tab: the cost layer's phases (shared memory).
template <int LAY, int RB, bool PREF>
QF_D void pair_forward(const PairPass& F, typename Types<LAY>::E* psi, const uint16_t* cuts, const Coef* tab, int ncut,
                       typename Types<LAY>::E amp0, const Coef& ac, const Coef& as, const Coef& bc, const Coef& bs,
                       uint32_t first, uint32_t stride, uint32_t ntiles, unsigned char* smem) {
  using S = PairShape<LAY, RB>;
  using E = typename S::E;
  constexpr int R = S::R;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const PairTile<RB> G(F, warp);
  E* work = reinterpret_cast<E*>(smem);
  E* next = reinterpret_cast<E*>(smem + S::VEC) + threadIdx.x;  // this thread's slots: register * NT
  const bool xfirst = F.pair && F.hasA;  // arrangement at load: X in registers, else Y
  auto fetch = [&](uint32_t tile) {
    if constexpr (!PREF) return;
    if (tile < ntiles && !F.init) {
      const uint32_t b = G.base(tile, lane) | (xfirst ? G.wy : G.wx);
#pragma unroll
      for (int r = 0; r < R; ++r) cp_async_amp(next + r * S::NT, psi + (b | (xfirst ? G.offx(r) : G.offy(r))));
    }
    cp_async_commit();
  };
  fetch(first);
  for (uint32_t tile = first; tile < ntiles; tile += stride) {
    const uint32_t b = G.base(tile, lane);
    const uint32_t by = b | G.wx;  // Y in registers
    int cv[R];
    if constexpr (PREF) {
      if (F.cost) {  // on their way while the tile is awaited
#pragma unroll
        for (int r = 0; r < R; ++r) cv[r] = cuts[by | G.offy(r)];
      }
      cp_async_wait<0>();
    }
    E a[R];
    if (F.init) {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = amp0;
    } else if constexpr (PREF) {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = next[r * S::NT];
    } else if (xfirst) {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = psi[b | G.wy | G.offx(r)];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = psi[by | G.offy(r)];
    }
    bool xnow = xfirst;
    if (F.hasA) {
      if (F.pair) {
        pair_rx<RB>(ac, as, F.lanesA != 0, F.nx, a);
        pair_exchange<LAY, RB>(a, work, lane, warp);
        xnow = false;
        fetch(tile + stride);  // the slots were read: their values went through the exchange
        pair_rx<RB>(ac, as, false, F.ny, a);
      } else {
        pair_rx<RB>(ac, as, F.lanesA != 0, F.ny, a);
      }
    }
    if (F.cost) {
#pragma unroll
      for (int r = 0; r < R; ++r) a[r] = cmul_v(tab[min(PREF ? cv[r] : (int)cuts[by | G.offy(r)], ncut - 1)], a[r]);
    }
    if (F.hasB) {
      pair_rx<RB>(bc, bs, true, F.ny, a);
      if (F.pair) {
        pair_exchange<LAY, RB>(a, work, lane, warp);
        xnow = true;
        pair_rx<RB>(bc, bs, false, F.nx, a);
      }
    }
    if (xnow) {
#pragma unroll
      for (int r = 0; r < R; ++r) psi[b | G.wy | G.offx(r)] = a[r];
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) psi[by | G.offy(r)] = a[r];
    }
    // (not fetched above: without an exchange the mixer consumed the slots'
    // values, or the pass generates them)
    if (!(F.hasA && F.pair)) fetch(tile + stride);
  }
  cp_async_wait<0>();
}

// sums of an adjoint pass, per thread
struct PairSums {
  FFAcc a, cut, e, b;
};

// Adjoint pass: psi and lambda together.
template <int LAY, int RB, bool F32_INIT>
QF_D void pair_adjoint(const PairPass& F, typename Types<LAY>::E* psi, typename Types<LAY>::E* lam,
                       const uint16_t* cuts, const Coef* tab, int ncut, float wref, const Coef& ac, const Coef& as,
                       const Coef& bc, const Coef& bs, uint32_t first, uint32_t stride, uint32_t ntiles,
                       unsigned char* smem, PairSums& S_) {
  using S = PairShape<LAY, RB>;
  using E = typename S::E;
  constexpr int R = S::R;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const PairTile<RB> G(F, warp);
  E* work = reinterpret_cast<E*>(smem);
  E* next = reinterpret_cast<E*>(smem + S::VEC) + threadIdx.x;
  const bool xfirst = F.pair != 0;
  auto fetch = [&](uint32_t tile) {
    if (tile < ntiles) {
      const uint32_t b = G.base(tile, lane) | (xfirst ? G.wy : G.wx);
#pragma unroll
      for (int r = 0; r < R; ++r) cp_async_amp(next + r * S::NT, psi + (b | (xfirst ? G.offx(r) : G.offy(r))));
      if (!F.init) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          cp_async_amp(next + (R + r) * S::NT, lam + (b | (xfirst ? G.offx(r) : G.offy(r))));
      }
    }
    cp_async_commit();
  };
  fetch(first);
  for (uint32_t tile = first; tile < ntiles; tile += stride) {
    const uint32_t b = G.base(tile, lane);
    const uint32_t by = b | G.wx;
    int cv[R];
    if (F.cost) {
#pragma unroll
      for (int r = 0; r < R; ++r) cv[r] = cuts[by | G.offy(r)];
    }
    int ci[R];
    if (F.init) {
#pragma unroll
      for (int r = 0; r < R; ++r) ci[r] = cuts[xfirst ? b | G.wy | G.offx(r) : by | G.offy(r)];
    }
    cp_async_wait<0>();
    E a[R], l[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      a[r] = next[r * S::NT];
      if (!F.init) l[r] = next[(R + r) * S::NT];
    }
    if (F.init) {
      float part = 0.f;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float c = (float)ci[r];
        if constexpr (F32_INIT) {
          part = fmaf(c, fmaf(a[r].x, a[r].x, a[r].y * a[r].y), part);
        } else {
          FFAcc t;
          t.zero();
          acc_norm2(t, a[r]);
          S_.e.add_prod(c, 0.f, t.s, t.e);
        }
        l[r] = scale_ff(a[r], c);
      }
      if constexpr (F32_INIT) S_.e.add(part, 0.f);
    }
    bool xnow = xfirst;
    if (F.pair) {
      pair_mix<LAY, RB>(ac, as, F.lanesA != 0, F.nx, a, l, S_.a);
      pair_exchange<LAY, RB>(a, work, lane, warp);
      pair_exchange<LAY, RB>(l, work, lane, warp);
      xnow = false;
      fetch(tile + stride);  // the slots were read: their values went through the exchange
      pair_mix<LAY, RB>(ac, as, false, F.ny, a, l, S_.a);
    } else {
      pair_mix<LAY, RB>(ac, as, F.lanesA != 0, F.ny, a, l, S_.a);
    }
    if (F.cost) {
      if constexpr (LAY == C64) {
        float part = 0.f;
#pragma unroll
        for (int r = 0; r < R; ++r)
          part = fmaf(wref - (float)cv[r], fmaf(l[r].x, a[r].y, -l[r].y * a[r].x), part);
        S_.cut.add(part, 0.f);
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) acc_imconj(S_.cut, to_ff(l[r]), to_ff(a[r]), wref - (float)cv[r]);
      }
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const Coef& c = tab[min(cv[r], ncut - 1)];
        a[r] = cmul_v(c, a[r]);
        l[r] = cmul_v(c, l[r]);
      }
    }
    if (F.hasB) {
      pair_mix<LAY, RB>(bc, bs, true, F.ny, a, l, S_.b);
      if (F.pair) {
        pair_exchange<LAY, RB>(a, work, lane, warp);
        pair_exchange<LAY, RB>(l, work, lane, warp);
        xnow = true;
        pair_mix<LAY, RB>(bc, bs, false, F.nx, a, l, S_.b);
      }
    }
    if (xnow) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t x = b | G.wy | G.offx(r);
        psi[x] = a[r];
        lam[x] = l[r];
      }
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const uint32_t x = by | G.offy(r);
        psi[x] = a[r];
        lam[x] = l[r];
      }
    }
    if (!F.pair) fetch(tile + stride);
  }
  cp_async_wait<0>();
}
#endif

}  // namespace qf
