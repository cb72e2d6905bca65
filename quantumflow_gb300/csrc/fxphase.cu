// Element-wise phase passes and qubit-exchange passes on complex128 states
// (QF_LAYOUT_FX).
//
// Reference semantics: quantumflow/backend/numpybk.py:159-214 tensormul with
// diagonal gates (CPHASE, ZZ, RZ, T, ..., quantumflow/stdgates.py) and SWAPs,
// applied in list order (quantumflow/circuits.py:87-99).
//
// k_fxphase applies a run of diagonal gates on one or two qubits (and signs)
// in one pass.  A thread holds the 2^G amplitudes of G <= 4 window bits; the
// planner picks the window so that every two-qubit gate has a bit in it.
// What the gates do to an amplitude is then a product of at most G + 1
// functions of the other bits, one per set window bit and one common, and
// each function is a product over single bits: table lookups, one by the
// thread's index in its block and one per further eight bits.  So the cost
// per amplitude (about 1.7 complex products to form the 2^G phases from the
// functions and apply them) does not depend on the number of gates, where
// the interpreted group pass spends a complex product and the decoding on
// every gate and amplitude.
//
// Arithmetic: an amplitude's two parts share one exponent (57-bit integers,
// fx.cuh), phases are 2^58 integers multiplied with 2^-57 relative error, and
// each part is rounded to FP64 once by the exactly rounding convert.
// Bound: 160 to 220 instructions an amplitude (n = 24: issue 50 to 58%, integer
// ALU 58 to 60%), then HBM (32 bytes an amplitude).  QFT, n = 23: 70 us a pass (0.27 GB
// moved; 40 us at the copy rate); the interpreted group passes took 950 to
// 1570 us.
#include <atomic>

#include "fx.cuh"
#include "fxphase.cuh"

namespace qf {

namespace {

constexpr int FXP_THREADS = 256;
constexpr int FXP_LOW = 8;  // bits of t looked up by thread, and per further table

struct Phase {
  int64_t r, i;  // 2^58 units
};
QF_D FxC fxp_coef(const Phase& p) {
  FxC c;
  const int64_t s = p.r + p.i;
  c.rh = static_cast<int32_t>(p.r >> FX_L);
  c.rl = static_cast<int32_t>(static_cast<uint32_t>(p.r) & FX_LMASK);
  c.ih = static_cast<int32_t>(p.i >> FX_L);
  c.il = static_cast<int32_t>(static_cast<uint32_t>(p.i) & FX_LMASK);
  c.sh = static_cast<int32_t>(s >> FX_L);
  c.sl = static_cast<int32_t>(static_cast<uint32_t>(s) & FX_LMASK);
  return c;
}
// products in T units of a 2^56 amplitude are 2^58 integers again
QF_D Phase fxp_mul(const Phase& a, const FxC& c) {
  const FxAmp x = fx_amp_from_t(a.r, a.i);
  Phase p;
  fx_cdot<1>(&c, &x, p.r, p.i);
  return p;
}
QF_D Phase fxp_mul(const Phase& a, const Phase& b) { return fxp_mul(a, fxp_coef(b)); }
QF_D Phase fxp_of(longlong2 v) { return Phase{v.x, v.y}; }

// v * p, rounded once; `flip` is 0 or the sign bit
QF_D double2 fxp_apply(double2 v, const FxC& c, uint32_t flip) {
  constexpr int M = 57;
  const uint32_t m = max(fx_hiword(v.x) & 0x7fffffffu, fx_hiword(v.y) & 0x7fffffffu);
  int E = static_cast<int>(m >> 20);
  if (E < FX_EMIN) E = 4095;  // parts below 2^-959 become 0, as in every fixed-point pass
  FxAmp a;
  fx_in<M>(v.x, E, a.rh, a.rl);
  fx_in<M>(v.y, E, a.ih, a.il);
  int64_t tr, ti;
  fx_cdot<1>(&c, &a, tr, ti);
  // value T * 2^(E - 1024 - M): the convert rounds to nearest even, the
  // power of two is an add on the exponent field (T = 0 stays 0)
  const uint32_t scale = (static_cast<uint32_t>(E - 1024 - M) << 20) ^ flip;
  const double dr = __ll2double_rn(tr), di = __ll2double_rn(ti);
  return make_double2(fx_double(fx_hiword(dr) + min(fx_hiword(dr), 1u) * scale, fx_loword(dr)),
                      fx_double(fx_hiword(di) + min(fx_hiword(di), 1u) * scale, fx_loword(di)));
}
QF_D double2 fxp_flip(double2 v, uint32_t flip) {
  return make_double2(fx_double(fx_hiword(v.x) ^ flip, fx_loword(v.x)),
                      fx_double(fx_hiword(v.y) ^ flip, fx_loword(v.y)));
}

// CTAS of them share an SM: two load eight amplitudes of a thread at a time;
// three, at fewer registers, load four.
template <int G, typename IT, int CTAS>
__global__ void __launch_bounds__(FXP_THREADS, CTAS) k_fxphase(const __grid_constant__ FxPhaseParams P, int nch) {
  extern __shared__ __align__(16) longlong2 tab[];  // [1 + nch][G + 1][256]
  constexpr int F = G + 1, TS = 1 << FXP_LOW;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int tbits = P.n - G;
  // tables by doubling, one warp per (table, function)
  for (int k = warp; k < (1 + nch) * F; k += FXP_THREADS / 32) {
    const int ch = k / F, f = k % F;
    longlong2* T = tab + k * TS;
    if (lane == 0) T[0] = ch == 0 ? P.one[f] : make_longlong2(int64_t(1) << 58, 0);
    __syncwarp();
    const int bits = min(FXP_LOW, tbits - FXP_LOW * ch);
    for (int b = 0; b < bits; ++b) {
      const FxC c = fxp_coef(fxp_of(P.ratio[f][FXP_LOW * ch + b]));
      for (int x = lane; x < (1 << b); x += 32) {
        const Phase p = fxp_mul(fxp_of(T[x]), c);
        T[x | (1 << b)] = make_longlong2(p.r, p.i);
      }
      __syncwarp();
    }
  }
  __syncthreads();
  pdl_wait();  // QFT, launches overlapped: n = 16 72 -> 61 us, n = 20 147 -> 135, n = 23 847 -> 823
  const IT ngroups = IT(1) << tbits;
  const IT ntiles = (ngroups + FXP_THREADS - 1) / FXP_THREADS;
  for (IT tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    // the functions at the tile's bits, one lane per function
    Phase uni{int64_t(1) << 58, 0};
    if (nch > 0) {
      const int f = lane < F ? lane : 0;
      uni = fxp_of(tab[(F + f) * TS + static_cast<int>(tile & (TS - 1))]);
      for (int ch = 2; ch <= nch; ++ch)
        uni = fxp_mul(uni, fxp_of(tab[(ch * F + f) * TS + static_cast<int>((tile >> (FXP_LOW * (ch - 1))) & (TS - 1))]));
    }
    const IT t = tile * FXP_THREADS + threadIdx.x;
    Phase fn[F];
#pragma unroll
    for (int f = 0; f < F; ++f) {
      if (f == G && !P.has_c) continue;
      fn[f] = fxp_of(tab[f * TS + threadIdx.x]);  // entries above 2^tbits are never used
      if (nch > 0) {
        const Phase u{__shfl_sync(0xffffffffu, uni.r, f), __shfl_sync(0xffffffffu, uni.i, f)};
        fn[f] = fxp_mul(fn[f], u);
      }
    }
    if (t >= ngroups) continue;
    IT xb = t;
#pragma unroll
    for (int j = 0; j < G; ++j) xb = insert0(xb, (int)P.sbits[j]);
    uint32_t neg = 0;
    for (int s = 0; s < P.nsign; ++s)
      if ((xb & (IT)P.mout[s]) == (IT)P.mout[s]) neg ^= P.rmask[s];
    // phases of the low two window bits, then the others outermost
    constexpr int GI = G < 2 ? G : 2, NI = 1 << GI, NO = 1 << (G - GI);
    Phase inner[NI];
    inner[1] = fn[0];
    if constexpr (GI >= 2) {
      inner[2] = fn[1];
      inner[3] = fxp_mul(fn[0], fn[1]);
    }
#pragma unroll
    for (int o0 = 0; o0 < NO; o0 += CTAS > 2 ? 1 : 2) {
      constexpr int STEP = NO < 2 || CTAS > 2 ? 1 : 2;
      double2 x[STEP * NI];
#pragma unroll
      for (int k = 0; k < STEP * NI; ++k) x[k] = P.in[xb | (IT)P.off[o0 * NI + k]];
#pragma unroll
      for (int oo = 0; oo < STEP; ++oo) {
        const int o = o0 + oo;
        Phase q;
        bool one = false;  // q is exactly 1
        if (o == 0) {
          one = !P.has_c;
          if (P.has_c) q = fn[G];
        } else {
          if constexpr (G >= 3) q = (o & 1) ? fn[2] : fn[G > 3 ? 3 : 2];
          if constexpr (G >= 4)
            if (o == 3) q = fxp_mul(fn[2], fn[3]);
          if (P.has_c) q = fxp_mul(q, fn[G]);
        }
        const FxC qc = fxp_coef(one ? Phase{0, 0} : q);
#pragma unroll
        for (int i = 0; i < NI; ++i) {
          const int c = o * NI + i;
          const uint32_t flip = ((neg >> c) & 1u) << 31;
          double2 y = x[oo * NI + i];
          if (i == 0 && o == 0 && one && !P.has_kc) {
            y = fxp_flip(y, flip);
          } else {
            Phase p;
            if (i == 0) p = one ? Phase{int64_t(1) << 58, 0} : q;
            else p = one ? inner[i] : fxp_mul(inner[i], qc);
            if (P.has_kc) p = fxp_mul(p, fxp_of(P.kc[c]));
            y = fxp_apply(y, fxp_coef(p), flip);
          }
          P.out[xb | (IT)P.off[c]] = y;
        }
      }
    }
  }
}

// tables beyond the thread's own, and the bytes of all of them
constexpr int fxp_chunks(int n, int G) { return n - G <= FXP_LOW ? 0 : (n - G - 1) / FXP_LOW; }
constexpr int fxp_smem(int n, int G) { return (1 + fxp_chunks(n, G)) * (G + 1) * (16 << FXP_LOW); }
constexpr int SM_SMEM = 228 << 10;  // of an SM, 1 KiB of it reserved per CTA

template <int G, typename IT, int CTAS>
int phase_launch_t(const FxPhaseParams& P, cudaStream_t stream) {
  const int hbits = P.n - G - FXP_LOW;
  const int nch = fxp_chunks(P.n, G);
  const size_t smem = (size_t)fxp_smem(P.n, G);
  static std::atomic<int> attr_set[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) dev = 0;
  if (!attr_set[dev].load()) {  // up to four tables (n <= 34): 100 KiB
    int rc = check_cuda(cudaFuncSetAttribute(k_fxphase<G, IT, CTAS>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             5 * (G + 1) * (16 << FXP_LOW)));
    if (rc) return rc;
    attr_set[dev].store(1);
  }
  int64_t grid = hbits <= 0 ? 1 : int64_t(1) << hbits;
  const int64_t cap = (int64_t)device_sm_count() * CTAS;
  if (grid > cap) grid = cap;
  return pdl_launch(k_fxphase<G, IT, CTAS>, grid, FXP_THREADS, smem, stream, P, nch);
}

// A CTA exchanges the tiles at base b and pi(b) (the tile bits include the
// lowest five and their partners, so reads and writes are runs of 32
// amplitudes, and the state may be permuted in place).  Rows of 32 are
// padded by one amplitude: a permuted read steps through 32 of them.
// Bound: HBM.  n = 23, 11 exchanges: 70 us; six passes of two as 4x4
// gates on the tensor cores took 412 (354 with today's pass).
constexpr int FXSW_THREADS = 256;
QF_D int fxsw_slot(int i) { return i + (i >> 5); }

__global__ void __launch_bounds__(FXSW_THREADS) k_fxswap(const __grid_constant__ FxSwapParams P) {
  constexpr int N = 1 << FXSW_TILE_BITS, PER = N / FXSW_THREADS;
  __shared__ double2 ta[N + N / 32], tb[N + N / 32];
  const int namp = 1 << P.nt;
  int64_t off[PER];
  int from[PER];
#pragma unroll
  for (int k = 0; k < PER; ++k) {
    const int i = threadIdx.x + k * FXSW_THREADS;
    off[k] = 0;
    from[k] = 0;
    for (int j = 0; j < P.nt; ++j)
      if ((i >> j) & 1) {
        off[k] |= int64_t(1) << P.tb[j];
        from[k] |= 1 << P.lp[j];
      }
  }
  const int64_t nbase = int64_t(1) << (P.n - P.nt);
  pdl_wait();
  for (int64_t u = blockIdx.x; u < nbase; u += gridDim.x) {
    int64_t b = u;
    for (int j = 0; j < P.nt; ++j) b = insert0(b, (int)P.tb[j]);
    int64_t pb = b;
    for (int j = 0; j < P.npair; ++j) {
      const int64_t d = ((b >> P.pa[j]) ^ (b >> P.pb[j])) & 1;
      pb ^= (d << P.pa[j]) | (d << P.pb[j]);
    }
    if (pb < b) continue;  // the block of pi(b) takes both
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x + k * FXSW_THREADS;
      if (i < namp) {
        ta[fxsw_slot(i)] = P.in[b | off[k]];
        if (pb != b) tb[fxsw_slot(i)] = P.in[pb | off[k]];
      }
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      const int i = threadIdx.x + k * FXSW_THREADS;
      if (i < namp) {
        P.out[pb | off[k]] = ta[fxsw_slot(from[k])];
        if (pb != b) P.out[b | off[k]] = tb[fxsw_slot(from[k])];
      }
    }
    __syncthreads();
  }
}

}  // namespace

// Three CTAs an SM from 2^11 tiles of 256 threads (five rounds of them) on,
// where they hide more of each other's latency: QFT, n = 24 1595 -> 1560 us,
// n = 26 6731 -> 6530; below, the last round is emptier than with two: n = 21
// 249 with two, 265 with three.  Only while the tables of three fit an SM
// (four window bits: up to n = 28): four CPHASEs, n = 29, 5223 us with a grid
// for three of which two fit, 4000 with two.
constexpr int phase_ctas(int n, int G) {
  return n - G - FXP_LOW >= 11 && 3 * (fxp_smem(n, G) + 1024) <= SM_SMEM ? 3 : 2;
}
constexpr bool phase_ctas_fit() {
  for (int n = 11; n <= QF_MAX_QUBITS; ++n)
    for (int G = 1; G <= 4; ++G)
      if (phase_ctas(n, G) * (fxp_smem(n, G) + 1024) > SM_SMEM) return false;
  return true;
}
static_assert(phase_ctas_fit(), "a grid of CTAs that are all resident");

template <int G>
static int phase_launch(const FxPhaseParams& P, cudaStream_t stream) {
  const bool three = phase_ctas(P.n, G) == 3;
  if (P.n > 31)
    return three ? phase_launch_t<G, int64_t, 3>(P, stream) : phase_launch_t<G, int64_t, 2>(P, stream);
  return three ? phase_launch_t<G, uint32_t, 3>(P, stream) : phase_launch_t<G, uint32_t, 2>(P, stream);
}

int fx_phase_launch(const FxPhaseParams& P, cudaStream_t stream) {
  switch (P.G) {
    case 1: return phase_launch<1>(P, stream);
    case 2: return phase_launch<2>(P, stream);
    case 3: return phase_launch<3>(P, stream);
    case 4: return phase_launch<4>(P, stream);
  }
  return QF_ERR_NOT_SUPPORTED;
}

int fx_swap_launch(const FxSwapParams& P, cudaStream_t stream) {
  int64_t grid = int64_t(1) << (P.n - P.nt);
  const int64_t cap = (int64_t)device_sm_count() * 6;
  if (grid > cap) grid = cap;
  return pdl_launch(k_fxswap, grid, FXSW_THREADS, 0, stream, P);
}

}  // namespace qf
