// Parameters of the complex128 phase and qubit-exchange passes (fxphase.cu).
#pragma once
#include <cstdint>

#include "engine.cuh"

namespace qf {

constexpr int FXP_MAX_SIGNS = 48;

// A phase pass multiplies amplitude x by
//   kc[c] * F_C(t) * prod_{j in c} F_j(t),
// c = the window index of x (the G window bits) and t = the index of its
// other bits (the compact index: window bits removed).  Function f = 0..G-1
// belongs to a window bit, f = G to no bit; each is a product over the bits
// of t: F_f(t) = one[f] * prod_{b in t} ratio[f][b].  All factors have unit
// modulus and are integers round(v * 2^58).
struct FxPhaseParams {
  const double2* in;
  double2* out;
  int32_t n, G, nsign, has_c, has_kc, pad;
  uint8_t sbits[8];           // window bits, ascending (the first G)
  int64_t off[16];            // global offset of window index c
  longlong2 one[5];
  longlong2 ratio[5][QF_MAX_QUBITS];
  longlong2 kc[16];
  uint64_t mout[FXP_MAX_SIGNS];   // sign ops: their bits outside the window
  uint16_t rmask[FXP_MAX_SIGNS];  // window indices that carry all of the op's window bits
};
int fx_phase_launch(const FxPhaseParams& P, cudaStream_t stream);

// Exchange of disjoint pairs of qubits: out[x] = in[pi(x)].
constexpr int FXSW_TILE_BITS = 10;
struct FxSwapParams {
  const double2* in;
  double2* out;
  int32_t n, nt, npair;
  uint8_t tb[FXSW_TILE_BITS];   // tile bits, ascending; closed under the exchange
  uint8_t lp[FXSW_TILE_BITS];   // local bit j of a tile goes to local bit lp[j]
  uint8_t pa[16], pb[16];       // exchanged pairs outside the tile
};
int fx_swap_launch(const FxSwapParams& P, cudaStream_t stream);

}  // namespace qf
