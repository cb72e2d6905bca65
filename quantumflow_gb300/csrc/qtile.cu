// QAOA forward state and adjoint gradient of float-float states on wide
// tiles.
//
// Reference semantics: the circuit of quantumflow/qaoa.py:22-64 (|+>^n, then
// per layer the cost phase exp(i gamma (E/2 - C)) and RX(beta) on every
// node) and the gradient of <C> the reference takes by automatic
// differentiation (examples/qaoa_maxcut.py:56-64); the adjoint method and the
// outputs are those of adjoint.cu.
//
// A CTA holds a tile of 2^T amplitudes, 2^RB per thread, so a pass applies
// the mixer on up to T bits where a warp tile takes 7 or 8.  With the qubits
// in m groups a pass finishes one layer's mixer on its group, applies the
// cost layer and starts the next layer's mixer on the same group: p layers
// take 1 + p (m - 1) passes, and m = 2 up to 23 qubits.  Within a tile the
// register bits move through the tile's bits in stages, exchanged through
// shared memory (swizzled: conflict-free at every stage), downwards before
// the cost layer and upwards after it, so a pass loads and stores runs of
// contiguous amplitudes.  The next tile's amplitudes are on their way
// (cp.async into thread-private slots) while a tile is worked on.  The stages
// are a loop over one body per register bit: with every stage unrolled the
// code outgrew the instruction caches and warps waited on fetches two thirds
// of the time (a backward pass at n = 22: 467 -> 333 us).
//
// Arithmetic per bit:
//  * amplitudes are kept as phi_x = i^|x| psi_x.  RX(beta) is then the real
//    rotation phi0' = c phi0 - s phi1, phi1' = c phi1 + s phi0 (c, s of
//    beta / 2), the same on real and imaginary parts;
//  * where the pass has a cost layer and |tan(beta / 2)| <= 1, the rotation
//    runs as phi0 - t phi1, phi1 + t phi0 with t = s / c: 15 operations a
//    part instead of 20; the factors c go into the cost layer's phase table;
//  * the gradient term of a bit is Re(conj(lam1) psi0 - conj(lam0) psi1) over
//    pairs, weighted with the square of the factors c not yet applied.
// Bound: FP32 issue (about 70% of its rate at n = 22); below n = 18 the latency
// of a pass.  A gradient evaluation against the warp-tile kernels: n = 22,
// p = 8 5570 -> 4090 us; n = 18, p = 6 739 -> 319 us; n = 12, p = 5 292 ->
// 140 us.
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "engine.cuh"
#include "qtile.cuh"
#include "state.cuh"

namespace qf {

namespace {

constexpr int QT_MAX_COEF = 1024;
constexpr int QT_MAX_T = 12;
constexpr int QT_MAX_R = 8;
constexpr int QT_LEAD = 1;  // lowest bits every tile carries (32-byte runs)

struct QTileParams {
  float4* psi;
  float4* lam;
  const uint16_t* cuts;
  double* rows;
  int32_t n, nslots;
  uint32_t active;      // local bits the mixer acts on
  int32_t fwd_init;     // generate |+>^n
  int32_t adj_init;     // lambda = C psi; <C> accumulator
  int32_t cost;
  int32_t has[2];       // mixer before / after the cost layer
  int32_t tan[2];       // ... its rotations leave out their factors c
  int32_t conv_out;     // store psi, not phi
  int32_t ncut;
  int32_t slot[2], slot_cut, slot_e;
  float wref;           // E/2
  uint8_t tb[QT_MAX_T + 4];    // global bit of each local bit, ascending
  uint32_t off0[QT_MAX_R];     // global offset of register index r, first arrangement
  uint32_t off1[QT_MAX_R];     // ... last arrangement
  float2 amp0;                 // 2^(-n/2)
  float2 c[2], s[2];           // phi0' = c phi0 + s phi1, phi1' = c phi1 - s phi0
  float2 w[2][QT_MAX_T];       // weight of the k-th bit's gradient term
  float2 wcut;                 // weight of the cost gradient
  Coef coef[QT_MAX_COEF];      // phase per cut value
};

// y + s x in float-float: the product to 2^-48, one TwoSum, one renormalisation
QF_D void ff_axpy(float2 s, float xh, float xl, float yh, float yl, float& rh, float& rl) {
  float p, c, u, t;
  ff_term(s.x, s.y, xh, xl, p, c);
  two_sum(yh, p, u, t);
  fast_two_sum(u, __fadd_rn(__fadd_rn(t, c), yl), rh, rl);
}
// c a + s b (TAN: a + s b) on both parts
template <bool TAN>
QF_D float4 rot_one(float4 a, float4 b, float2 c, float2 s) {
  float4 r;
  if (TAN) {
    ff_axpy(s, b.x, b.y, a.x, a.y, r.x, r.y);
    ff_axpy(s, b.z, b.w, a.z, a.w, r.z, r.w);
  } else {
    ff_dot2(c.x, c.y, a.x, a.y, s.x, s.y, b.x, b.y, r.x, r.y);
    ff_dot2(c.x, c.y, a.z, a.w, s.x, s.y, b.z, b.w, r.z, r.w);
  }
  return r;
}
template <bool TAN>
QF_D void rot_pair(float4& x0, float4& x1, float2 c, float2 s) {
  const float4 y0 = rot_one<TAN>(x0, x1, c, s);
  x1 = rot_one<TAN>(x1, x0, c, make_float2(-s.x, -s.y));
  x0 = y0;
}
// (-i)^k v
QF_D float4 turn(float4 v, int k) {
  if (k & 1) v = make_float4(v.z, v.w, -v.x, -v.y);
  return (k & 2) ? make_float4(-v.x, -v.y, -v.z, -v.w) : v;
}

template <int T, int RB>
struct QTile {
  static constexpr int R = 1 << RB, NT = 1 << (T - RB), NST = T / RB;
  static constexpr int LO0 = T - RB;  // register position of the first arrangement; the last one's is 0
  static constexpr size_t BYTES = (size_t(1) << T) * sizeof(float4);
  static_assert((RB == 2 || RB == 3) && T % RB == 0 && NT >= 32 && R <= QT_MAX_R, "tile shape");

  // local index of register 0 of thread t, registers at position lo
  static QF_D int tpart(int t, int lo) { return ((t >> lo) << (lo + RB)) | (t & ((1 << lo) - 1)); }
  // 16-byte units of a 128-byte row, permuted by the bits above them so that
  // eight lanes hit eight banks at every register position
  static QF_D int swz(int i) {
    return RB == 3 ? i ^ ((i >> 3) & 7) : i ^ ((i >> 3) & 3) ^ ((i >> 2) & 4);
  }
  // move the registers from position `from` to position `to`
  static QF_D void exchange(float4 (&a)[R], float4* work, int t, int from, int to) {
    __syncthreads();  // the buffer's previous readers are done
    const int f = swz(tpart(t, from)), g = swz(tpart(t, to));
#pragma unroll
    for (int r = 0; r < R; ++r) work[f ^ swz(r << from)] = a[r];
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) a[r] = work[g ^ swz(r << to)];
  }
};

// the mixer on register bit J: the bit's gradient term, then both rotations
template <int RB, int J, bool ADJ, bool TAN>
QF_D void mix_bit(float4 (&a)[1 << RB], float4 (&l)[1 << RB], float2 c, float2 s, float2 w, FFAcc& acc) {
  FFAcc t{0.f, 0.f};
#pragma unroll
  for (int i = 0; i < (1 << RB) / 2; ++i) {
    const int i0 = ((i >> J) << (J + 1)) | (i & ((1 << J) - 1)), i1 = i0 | (1 << J);
    if (ADJ) {
      t.add_prod(l[i1].x, l[i1].y, a[i0].x, a[i0].y);
      t.add_prod(l[i1].z, l[i1].w, a[i0].z, a[i0].w);
      t.add_prod(-l[i0].x, -l[i0].y, a[i1].x, a[i1].y);
      t.add_prod(-l[i0].z, -l[i0].w, a[i1].z, a[i1].w);
    }
    rot_pair<TAN>(a[i0], a[i1], c, s);
    if (ADJ) rot_pair<TAN>(l[i0], l[i1], c, s);
  }
  if (ADJ) acc.add_prod(w.x, w.y, t.s, t.e);
}
template <int RB, bool ADJ, bool TAN>
QF_D void mix_stage(float4 (&a)[1 << RB], float4 (&l)[1 << RB], uint32_t bits, float2 c, float2 s, const float2* w,
                    int& k, FFAcc& acc) {
  if (bits & 1u) mix_bit<RB, 0, ADJ, TAN>(a, l, c, s, w[k++], acc);
  if constexpr (RB > 1)
    if (bits & 2u) mix_bit<RB, 1, ADJ, TAN>(a, l, c, s, w[k++], acc);
  if constexpr (RB > 2)
    if (bits & 4u) mix_bit<RB, 2, ADJ, TAN>(a, l, c, s, w[k++], acc);
}

template <int T, int RB, bool ADJ>
__global__ void __launch_bounds__(QTile<T, RB>::NT, T >= 12 ? 1 : 2) k_qtile(const __grid_constant__ QTileParams P) {
  using Q = QTile<T, RB>;
  constexpr int R = Q::R, NT = Q::NT;
  extern __shared__ __align__(128) unsigned char qt_smem[];
  __shared__ double red[4][NT / 32];
  // per-thread sums (two mixers, cost, <C>) between tiles; in registers they
  // would be live throughout
  __shared__ FFAcc sums[ADJ ? 4 : 1][NT];
  float4* work = reinterpret_cast<float4*>(qt_smem);
  float4* next = reinterpret_cast<float4*>(qt_smem + Q::BYTES);  // [vector][register][thread]
  Coef* scoef = reinterpret_cast<Coef*>(qt_smem + (ADJ ? 3 : 2) * Q::BYTES);
  const int t = threadIdx.x;
  if (P.cost)
    for (int i = t; i < P.ncut; i += NT) scoef[i] = P.coef[i];
  if (ADJ)
    for (int k = 0; k < 4; ++k) sums[k][t] = FFAcc{0.f, 0.f};
  auto add_sum = [&](int k, FFAcc v) {
    FFAcc s = sums[ADJ ? k : 0][t];
    s.add(v.s, v.e);
    sums[ADJ ? k : 0][t] = s;
  };
  auto spread = [&](int i) {  // local index -> global offset
    uint32_t o = 0;
#pragma unroll
    for (int j = 0; j < T; ++j) o |= static_cast<uint32_t>((i >> j) & 1) << P.tb[j];
    return o;
  };
  const uint32_t t0 = spread(Q::tpart(t, Q::LO0)), t1 = spread(Q::tpart(t, 0));
  const uint32_t ntiles = 1u << (P.n - T);
  auto base_of = [&](uint32_t tile) {
#pragma unroll
    for (int j = 0; j < T; ++j) tile = insert0(tile, (int)P.tb[j]);
    return tile;
  };
  auto fetch = [&](uint32_t tile) {
    if (tile < ntiles && !P.fwd_init) {
      const uint32_t b = base_of(tile) | t0;
#pragma unroll
      for (int r = 0; r < R; ++r) cp_async_amp(next + r * NT + t, P.psi + (b | P.off0[r]));
      if (ADJ && !P.adj_init) {
#pragma unroll
        for (int r = 0; r < R; ++r) cp_async_amp(next + (R + r) * NT + t, P.lam + (b | P.off0[r]));
      }
    }
    cp_async_commit();
  };
  __syncthreads();
  // so far only parameters were read: this may have run while the previous
  // pass drained (programmatic dependent launch)
  pdl_wait();
  uint32_t tile = blockIdx.x;
  fetch(tile);
  for (; tile < ntiles; tile += gridDim.x) {
    const uint32_t base = base_of(tile);
    cp_async_wait<0>();
    float4 a[R], l[R];
    int lo = Q::LO0;  // register position
    if (!P.fwd_init) {
      FFAcc e{0.f, 0.f};
#pragma unroll
      for (int r = 0; r < R; ++r) {
        a[r] = next[r * NT + t];
        if (ADJ) {
          if (!P.adj_init) {
            l[r] = next[(R + r) * NT + t];
          } else {
            const float c = (float)P.cuts[base | t0 | P.off0[r]];
            FFAcc nrm{0.f, 0.f};
            acc_norm2(nrm, a[r]);
            e.add_prod(c, 0.f, nrm.s, nrm.e);
            l[r] = scale_ff(a[r], c);
          }
        }
      }
      if (ADJ && P.adj_init) add_sum(3, e);
    } else {
      lo = 0;
#pragma unroll
      for (int r = 0; r < R; ++r)  // i^|x| = (-i)^(-|x|)
        a[r] = turn(make_float4(P.amp0.x, P.amp0.y, 0.f, 0.f), (-__popc(base | t1 | P.off1[r])) & 3);
    }
    bool fetched = false;
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int end = half == 0 ? 0 : Q::LO0;  // register position after this half
      if (P.has[half]) {
        const float2 c = P.c[half], s = P.s[half];
        const bool tan_form = P.tan[half];
        FFAcc acc{0.f, 0.f};
        int k = 0;
#pragma unroll 1
        for (;;) {
          const uint32_t bits = P.active >> lo;
          if (tan_form) mix_stage<RB, ADJ, true>(a, l, bits, c, s, P.w[half], k, acc);
          else mix_stage<RB, ADJ, false>(a, l, bits, c, s, P.w[half], k, acc);
          if (lo == end) break;
          const int to = half == 0 ? lo - RB : lo + RB;
          Q::exchange(a, work, t, lo, to);
          if (ADJ) Q::exchange(l, work, t, lo, to);
          lo = to;
          // the slots have been read: their values are in shared memory
          if (!fetched) fetch(tile + gridDim.x);
          fetched = true;
        }
        if (ADJ) add_sum(half, acc);
      } else if (lo != end) {
        Q::exchange(a, work, t, lo, end);
        if (ADJ) Q::exchange(l, work, t, lo, end);
        lo = end;
        if (!fetched) fetch(tile + gridDim.x);
        fetched = true;
      }
      if (half == 0 && P.cost) {
        FFAcc cut{0.f, 0.f};
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int cv = P.cuts[base | t1 | P.off1[r]];
          if (ADJ) acc_imconj(cut, l[r], a[r], P.wref - (float)cv);
          const Coef& c = scoef[min(cv, P.ncut - 1)];
          a[r] = cmul_v(c, a[r]);
          if (ADJ) l[r] = cmul_v(c, l[r]);
        }
        if (ADJ) {
          FFAcc v{0.f, 0.f};
          v.add_prod(P.wcut.x, P.wcut.y, cut.s, cut.e);
          add_sum(2, v);
        }
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const uint32_t x = base | t0 | P.off0[r];
      P.psi[x] = P.conv_out ? turn(a[r], __popc(x) & 3) : a[r];
      if (ADJ) P.lam[x] = l[r];
    }
  }
  cp_async_wait<0>();
  if constexpr (ADJ) {
    const int lane = t & 31, warp = t >> 5;
    for (int k = 0; k < 4; ++k) {
      const double v = warp_sum((double)sums[k][t].s + (double)sums[k][t].e);
      if (lane == 0) red[k][warp] = v;
    }
    __syncthreads();
    if (t < 4) {
      const int slot = t < 2 ? P.slot[t] : t == 2 ? P.slot_cut : P.slot_e;
      if (slot >= 0) {
        double s = 0.0;
        for (int w = 0; w < NT / 32; ++w) s += red[t][w];
        P.rows[(size_t)blockIdx.x * P.nslots + slot] += (t == 2 ? -2.0 : 1.0) * s;
      }
    }
  }
}

// ------------------------------------------------------------------ host ----
// Tile width by size: the narrowest that keeps two groups of qubits, since its
// CTAs spread over more of the chip (gradient, p = 6: n = 16 256 us on 10
// bits, 500 on 12; n = 18 319 on 10, 499 on 12), while the chip is not full
// (n = 19: 538 on 10, 512 on 12).  Indices are 32-bit.
int tile_bits(int n) { return n < 8 || n > 31 ? 0 : n <= 15 ? 8 : n <= 18 ? 10 : 12; }

template <int T>
int grid_of(int n) {
  const int64_t tiles = int64_t(1) << (n - T);
  const int64_t cap = (int64_t)device_sm_count() * (T >= 12 ? 1 : T >= 10 ? 2 : 4);
  return (int)(tiles < cap ? tiles : cap);
}
int grid_of(int n) { return tile_bits(n) == 12 ? grid_of<12>(n) : tile_bits(n) == 10 ? grid_of<10>(n) : grid_of<8>(n); }

template <int T, int RB, bool ADJ>
int launch_t(QTileParams& P, cudaStream_t stream) {
  using Q = QTile<T, RB>;
  const size_t bytes = (ADJ ? 3 : 2) * Q::BYTES;
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr[dev].load()) {
    int rc = check_cuda(cudaFuncSetAttribute(k_qtile<T, RB, ADJ>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)(bytes + QT_MAX_COEF * sizeof(Coef))));
    if (rc) return rc;
    attr[dev].store(true);
  }
  const size_t smem = bytes + (P.cost ? (size_t)P.ncut * sizeof(Coef) : 0);
  for (int r = 0; r < Q::R; ++r) {
    P.off0[r] = P.off1[r] = 0;
    for (int j = 0; j < RB; ++j)
      if ((r >> j) & 1) {
        P.off0[r] |= 1u << P.tb[Q::LO0 + j];
        P.off1[r] |= 1u << P.tb[j];
      }
  }
  return pdl_launch(k_qtile<T, RB, ADJ>, grid_of<T>(P.n), Q::NT, smem, stream, P);
}
template <bool ADJ>
int launch(QTileParams& P, int T, cudaStream_t stream) {
  return T == 12   ? launch_t<12, 3, ADJ>(P, stream)
         : T == 10 ? launch_t<10, 2, ADJ>(P, stream)
                   : launch_t<8, 2, ADJ>(P, stream);
}

float2 ff_of(double v) {
  const float h = static_cast<float>(v);
  return make_float2(h, static_cast<float>(v - static_cast<double>(h)));
}

// what the passes of both sweeps share
struct Sweep {
  int n, T, m, nedges;
  std::vector<std::vector<int>> groups;  // mixer bits of each group
  QTileParams P;

  void init(void* psi, int n_, const uint16_t* cuts, int nedges_) {
    n = n_;
    nedges = nedges_;
    T = tile_bits(n);
    std::memset(&P, 0, sizeof(P));
    groups.assign(1, {});
    for (int b = 0; b < T; ++b) groups[0].push_back(b);
    for (int b = T; b < n;) {  // the other bits, shared out evenly
      const int left = n - b, cap = T - QT_LEAD, parts = (left + cap - 1) / cap, take = (left + parts - 1) / parts;
      groups.push_back({});
      for (int k = 0; k < take; ++k) groups.back().push_back(b++);
    }
    m = (int)groups.size();
    P.psi = static_cast<float4*>(psi);
    P.cuts = cuts;
    P.n = n;
    P.ncut = nedges + 1;
    P.wref = (float)(0.5 * nedges);
    P.slot[0] = P.slot[1] = P.slot_cut = P.slot_e = -1;
  }
  // tile bits of group g: its bits and the lowest others
  int use_group(int g) {
    const std::vector<int>& act = groups[g];
    std::vector<int> bits = act;
    for (int b = 0; b < n && (int)bits.size() < T; ++b)
      if (std::find(act.begin(), act.end(), b) == act.end()) bits.push_back(b);
    std::sort(bits.begin(), bits.end());
    P.active = 0;
    for (int j = 0; j < T; ++j) {
      P.tb[j] = (uint8_t)bits[j];
      if (std::find(act.begin(), act.end(), bits[j]) != act.end()) P.active |= 1u << j;
    }
    return (int)act.size();
  }
  // Mixer `half` rotates by the angle `by` (phi0' = c phi0 - s phi1, c and s
  // of `by`).  Returns the factor left out per bit: cos(by) when `may` allows
  // the tangent form and |tan| <= 1 (the factors then stay within a few
  // binades), else 1.
  double rotation(int half, double by, bool may) {
    const double ch = std::cos(by), sh = std::sin(by);
    P.has[half] = 1;
    P.tan[half] = may && std::abs(ch) >= std::abs(sh);
    P.c[half] = ff_of(ch);
    P.s[half] = ff_of(P.tan[half] ? -sh / ch : -sh);
    if (!P.tan[half]) return 1.0;
    // of the rounded tangent: the norm then drifts by its rounding in no layer
    const double t = static_cast<double>(P.s[half].x) + static_cast<double>(P.s[half].y);
    return std::copysign(1.0 / std::sqrt(1.0 + t * t), ch);
  }
  void cut_table(double gamma, double factor) {
    P.cost = 1;
    for (int cv = 0; cv <= nedges; ++cv)
      P.coef[cv] = make_coef(factor * std::polar(1.0, gamma * (0.5 * nedges - cv)), FF);
  }
  void weights(int half, double first, double ratio) {
    for (int k = 0; k < QT_MAX_T; ++k, first *= ratio) P.w[half][k] = ff_of(first);
  }
};

}  // namespace

// (Complex64 keeps the warp-tile kernels, whose FP32 sums callers read as
// float64 gradients and may compare at that precision; node phases do too:
// their loop over the nodes keeps every amplitude and a table entry of each
// in registers, and spilled.)
bool qtile_fits(int n, int layout, int nedges, int p, const double* node_theta) {
  if (node_theta != nullptr)
    for (int q = 0; q < n; ++q)
      if (!std::isnan(node_theta[q])) return false;
  return layout == FF && p > 0 && tile_bits(n) > 0 && nedges + 1 <= QT_MAX_COEF;
}
size_t qtile_grad_rows(int n, int layout) { return layout == FF && tile_bits(n) > 0 ? (size_t)grid_of(n) : 0; }

// |+>^n, then p layers; psi ends as amplitudes, or as phi (i^|x| psi_x) when
// `keep_phi` (the gradient sweep goes on from there).
int qtile_state(void* psi, int n, const uint16_t* cuts, int nedges, int p, const double* beta, const double* gamma,
                bool keep_phi, cudaStream_t stream) {
  static thread_local Sweep S;
  S.init(psi, n, cuts, nedges);
  QTileParams& P = S.P;
  const int m = S.m;
  P.amp0 = ff_of(std::ldexp(1.0, -n / 2) / ((n & 1) ? std::sqrt(2.0) : 1.0));
  auto order = [&](int l, int k) { return (l & 1) ? m - 1 - k : k; };
  auto start_layer = [&](int l, int nact, double factor) {
    S.cut_table(gamma[l], factor * std::pow(S.rotation(1, 0.5 * beta[l], true), nact));
  };
  P.fwd_init = 1;
  start_layer(0, S.use_group(order(0, 0)), 1.0);
  P.conv_out = !keep_phi && p == 1 && m == 1;
  int rc = launch<false>(P, S.T, stream);
  P.fwd_init = 0;
  for (int l = 0; l < p && !rc; ++l) {
    if (m == 1) {
      if (l == 0) continue;
      start_layer(l, S.use_group(0), 1.0);
      P.conv_out = !keep_phi && l == p - 1;
      rc = launch<false>(P, S.T, stream);
      continue;
    }
    for (int k = 1; k < m && !rc; ++k) {
      const int nact = S.use_group(order(l, k));
      const bool boundary = k == m - 1 && l + 1 < p;
      const double f = S.rotation(0, 0.5 * beta[l], boundary);
      P.cost = P.has[1] = 0;
      if (boundary) start_layer(l + 1, nact, std::pow(f, nact));  // order(l + 1, 0) == order(l, m - 1)
      P.conv_out = !keep_phi && l == p - 1 && k == m - 1;
      rc = launch<false>(P, S.T, stream);
    }
  }
  return rc;
}

// The adjoint sweep from psi = phi of the final state; rows: qtile_grad_rows
// x nslots doubles, zeroed by the caller.  psi ends at |+>^n.
int qtile_grad(void* psi, void* lam, int n, const uint16_t* cuts, int nedges, int p, const double* beta,
               const double* gamma, double* rows, int nslots, cudaStream_t stream) {
  static thread_local Sweep S;
  S.init(psi, n, cuts, nedges);
  QTileParams& P = S.P;
  const int m = S.m;
  P.lam = static_cast<float4*>(lam);
  P.rows = rows;
  P.nslots = nslots;
  auto order = [&](int l, int k) { return ((p - 1 - l) & 1) ? m - 1 - k : k; };
  bool started = false;  // the layer's first group was undone by the previous pass
  P.adj_init = 1;
  for (int l = p - 1; l >= 0; --l) {
    for (int k = started ? 1 : 0; k < m; ++k) {
      const int nact = S.use_group(order(l, k));
      const bool last = k == m - 1;
      const bool next = last && l > 0 && m > 1;  // order(l - 1, 0) == order(l, m - 1)
      const double fa = S.rotation(0, -0.5 * beta[l], last);
      double fb = 1.0;
      P.cost = P.has[1] = 0;
      if (next) fb = S.rotation(1, -0.5 * beta[l - 1], true);
      const double na = std::pow(fa, nact), nb = std::pow(fb, nact);
      if (last) S.cut_table(-gamma[l], na * nb);
      S.weights(0, 1.0, fa * fa);
      S.weights(1, 1.0 / (nb * nb), fb * fb);
      P.wcut = ff_of(na * na);
      P.slot[0] = p + l;
      P.slot[1] = next ? p + l - 1 : -1;
      P.slot_cut = last ? l : -1;
      P.slot_e = P.adj_init ? 2 * p : -1;
      P.conv_out = l == 0 && last;
      const int rc = launch<true>(P, S.T, stream);
      if (rc) return rc;
      P.adj_init = 0;
    }
    started = m > 1;
  }
  return QF_OK;
}

}  // namespace qf
