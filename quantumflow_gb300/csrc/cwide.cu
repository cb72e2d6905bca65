// Complex64 gate passes on wide tiles.
//
// Reference semantics: quantumflow/backend/numpybk.py:159-214 tensormul in
// list order (quantumflow/circuits.py:87-99), for runs of 2x2 and 4x4 gates
// and CZ-like signs.
//
// A shape pass (group.cu) reads and writes the state for at most two gates on
// four bits and runs at the copy rate, so only fewer passes are faster.  Here
// a CTA holds a tile of 2^13 amplitudes, 16 per thread, and works through up
// to three stages: the gates of a stage act on four tile bits that sit in the
// register index, and between stages the tile is re-arranged through shared
// memory.  Two CTAs per SM overlap each other's loads and exchanges: with the
// next tile prefetched into slots of its own instead, one CTA fits and the
// same passes took a third longer.  Complex products are packed
// (fma.rn.f32x2): the products with the real and with the imaginary parts of
// a row's coefficients are summed apart and combined at the end.
// Bound: FP32 and issue (55%) before HBM.  Random layers, n = 26: a shape pass
// of two gates 168 us, a wide pass of six 370 us; 10 layers 6630 -> 4480 us.
#include <algorithm>
#include <atomic>
#include <cstring>

#include "cwide.cuh"

namespace qf {

namespace {

constexpr int CW_R = 1 << CW_RB, CW_NT = 1 << (CW_T - CW_RB);
constexpr size_t CW_TILE = (size_t(1) << CW_T) * sizeof(float2);
constexpr size_t CW_SMEM = CW_TILE + CW_MAX_STAGES * CW_NT * sizeof(uint2);

// gate kinds: 2x2 on register bit j, 4x4 on register bits (hi, lo), matrix
// MSB on hi
enum CWKind : uint8_t { CWK_D1 = 0, CWK_D2 = 4 };  // D1 + j; D2 + pair index
struct CWGate {
  float4 c[16];  // (re, re, im, im)
};
struct CWStage {
  uint32_t roff[CW_RB];  // global offset of each register index bit
  uint32_t rloc[CW_RB];  // swizzled local index of each register index bit
  uint8_t tpos[CW_T - CW_RB];  // local bit of each thread index bit
  uint8_t ngates;
  uint8_t kind[CW_MAX_GATES];
  uint8_t gate[CW_MAX_GATES];      // index into gates
  uint8_t sign_end[CW_MAX_GATES + 1];  // signs before gate g end here; [ngates]: after the last
  uint8_t sign_begin;
};
struct CWParams {
  const float2* in;
  float2* out;
  int32_t n, nstages;
  uint8_t tb[CW_T + 3];  // global bit of each local bit, ascending
  CWStage st[CW_MAX_STAGES];
  CWGate gates[CW_MAX_GATES];
  uint32_t mout[CW_MAX_SIGNS];   // sign ops: their bits outside the stage's registers
  uint16_t rmask[CW_MAX_SIGNS];  // register indices that carry all of the op's register bits
};

using V2 = unsigned long long;
QF_D V2 pk(float x, float y) { return (static_cast<V2>(__float_as_uint(y)) << 32) | __float_as_uint(x); }
QF_D float lo_of(V2 v) { return __uint_as_float(static_cast<uint32_t>(v)); }
QF_D float hi_of(V2 v) { return __uint_as_float(static_cast<uint32_t>(v >> 32)); }
QF_D V2 fma2(V2 a, V2 b, V2 c) {
  V2 d;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
  return d;
}
QF_D V2 mul2(V2 a, V2 b) {
  V2 d;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
  return d;
}
// a gate's coefficients as (re, re), (im, im)
template <int N>
QF_D void load_coefs(const CWGate& g, V2 (&re)[N], V2 (&im)[N]) {
#pragma unroll
  for (int e = 0; e < N; ++e) {
    const float4 c = g.c[e];
    re[e] = pk(c.x, c.y);
    im[e] = pk(c.z, c.w);
  }
}
// sum_c u_c x_c: the products with re and with im are summed apart, then
// (p.re - q.im, p.im + q.re)
template <int D>
QF_D V2 row(const V2* re, const V2* im, const V2 (&x)[D]) {
  V2 p = mul2(re[0], x[0]), q = mul2(im[0], x[0]);
#pragma unroll
  for (int c = 1; c < D; ++c) {
    p = fma2(re[c], x[c], p);
    q = fma2(im[c], x[c], q);
  }
  return pk(lo_of(p) - hi_of(q), hi_of(p) + lo_of(q));
}
template <int J>
QF_D void gate1(const CWGate& g, V2 (&a)[CW_R]) {
  V2 re[4], im[4];
  load_coefs<4>(g, re, im);
#pragma unroll
  for (int i = 0; i < CW_R / 2; ++i) {
    const int i0 = ((i >> J) << (J + 1)) | (i & ((1 << J) - 1)), i1 = i0 | (1 << J);
    const V2 x[2] = {a[i0], a[i1]};
    a[i0] = row<2>(re, im, x);
    a[i1] = row<2>(re + 2, im + 2, x);
  }
}
template <int HI, int LO>
QF_D void gate2(const CWGate& g, V2 (&a)[CW_R]) {
  V2 re[16], im[16];
  load_coefs<16>(g, re, im);
#pragma unroll
  for (int i = 0; i < CW_R / 4; ++i) {
    int b = ((i >> LO) << (LO + 1)) | (i & ((1 << LO) - 1));
    b = ((b >> HI) << (HI + 1)) | (b & ((1 << HI) - 1));
    const int k[4] = {b, b | (1 << LO), b | (1 << HI), b | (1 << LO) | (1 << HI)};
    const V2 x[4] = {a[k[0]], a[k[1]], a[k[2]], a[k[3]]};
#pragma unroll
    for (int r = 0; r < 4; ++r) a[k[r]] = row<4>(re + 4 * r, im + 4 * r, x);
  }
}

// Swizzle: the bank (low four bits) of a local index is linear in its low
// eight bits with the columns of the extended Hamming code [8, 4, 4], so the
// 16 lanes of a half-warp, which differ in the four lowest bits outside the
// registers, meet at most two to a bank whatever those are.
QF_HD uint32_t cw_swz(uint32_t i) {
  const uint32_t h = (i >> 4) & 15u;
  const uint32_t parity = (0x6996u >> h) & 1u;
  return i ^ h ^ (parity ? 15u : 0u);
}
// base combined with the contributions of register index r, for all r (both
// the offsets and the swizzle are linear over XOR)
QF_D void cw_spread(uint32_t base, const uint32_t (&bit)[CW_RB], uint32_t (&at)[CW_R]) {
  at[0] = base;
#pragma unroll
  for (int j = 0; j < CW_RB; ++j)
#pragma unroll
    for (int r = 0; r < (1 << j); ++r) at[(1 << j) | r] = at[r] ^ bit[j];
}

__global__ void __launch_bounds__(CW_NT, 2) k_cwide(const __grid_constant__ CWParams P) {
  extern __shared__ __align__(128) unsigned char cw_smem[];
  V2* work = reinterpret_cast<V2*>(cw_smem);
  const uint32_t ntiles = 1u << (P.n - CW_T);
  auto base_of = [&](uint32_t tile) {
#pragma unroll
    for (int j = 0; j < CW_T; ++j) tile = insert0(tile, (int)P.tb[j]);
    return tile;
  };
  // this thread's global offset and swizzled local index in every stage
  uint2* mine = reinterpret_cast<uint2*>(cw_smem + CW_TILE) + threadIdx.x;
  for (int k = 0; k < P.nstages; ++k) {
    uint32_t l = 0, o = 0;
    for (int j = 0; j < CW_T - CW_RB; ++j)
      if ((threadIdx.x >> j) & 1) {
        l |= 1u << P.st[k].tpos[j];
        o |= 1u << P.tb[P.st[k].tpos[j]];
      }
    mine[k * CW_NT] = make_uint2(o, cw_swz(l));
  }
  const uint2 first = mine[0];
  for (uint32_t tile = blockIdx.x; tile < ntiles; tile += gridDim.x) {
    const uint32_t base = base_of(tile);
    V2 a[CW_R];
    uint32_t at[CW_R];
    cw_spread(base | first.x, P.st[0].roff, at);
#pragma unroll
    for (int r = 0; r < CW_R; ++r) a[r] = *reinterpret_cast<const V2*>(P.in + at[r]);
    uint2 me = first;
#pragma unroll 1
    for (int s = 0;; ++s) {
      const CWStage& S = P.st[s];
      const uint32_t xb = base | me.x;
      int sg = S.sign_begin;
#pragma unroll 1
      for (int g = 0;; ++g) {
        const int end = S.sign_end[g];
        if (sg < end) {
          uint32_t m = 0;
          for (; sg < end; ++sg)
            if ((xb & P.mout[sg]) == P.mout[sg]) m ^= P.rmask[sg];
#pragma unroll
          for (int r = 0; r < CW_R; ++r)
            if ((m >> r) & 1u) a[r] ^= 0x8000000080000000ull;
        }
        if (g == S.ngates) break;
        const CWGate& G = P.gates[S.gate[g]];
        switch (S.kind[g]) {
          case CWK_D1 + 0: gate1<0>(G, a); break;
          case CWK_D1 + 1: gate1<1>(G, a); break;
          case CWK_D1 + 2: gate1<2>(G, a); break;
          case CWK_D1 + 3: gate1<3>(G, a); break;
          case CWK_D2 + 0: gate2<1, 0>(G, a); break;
          case CWK_D2 + 1: gate2<2, 0>(G, a); break;
          case CWK_D2 + 2: gate2<2, 1>(G, a); break;
          case CWK_D2 + 3: gate2<3, 0>(G, a); break;
          case CWK_D2 + 4: gate2<3, 1>(G, a); break;
          default: gate2<3, 2>(G, a); break;
        }
      }
      if (s == P.nstages - 1) break;
      const CWStage& N = P.st[s + 1];
      __syncthreads();  // the buffer's previous readers are done
      cw_spread(me.y, S.rloc, at);
#pragma unroll
      for (int r = 0; r < CW_R; ++r) work[at[r]] = a[r];
      __syncthreads();
      me = mine[(s + 1) * CW_NT];
      cw_spread(me.y, N.rloc, at);
#pragma unroll
      for (int r = 0; r < CW_R; ++r) a[r] = work[at[r]];
    }
    cw_spread(base | me.x, P.st[P.nstages - 1].roff, at);
#pragma unroll
    for (int r = 0; r < CW_R; ++r) *reinterpret_cast<V2*>(P.out + at[r]) = a[r];
  }
}

uint64_t bits_of(const HostOp& op) {
  uint64_t m = 0;
  for (int j = 0; j < op.k; ++j) m |= uint64_t(1) << op.gb[j];
  return m;
}

}  // namespace

bool cwide_op(const HostOp& op) {
  return op.type == OP_DENSE1 || op.type == OP_DENSE2 || op.type == OP_SIGN;
}
// From two or more tiles on: n = 15, 10 random layers, 171 us against 212 on
// shape passes; n = 18 191 / 241; n = 21 215 / 333.  Indices are 32-bit.
bool cwide_fits(int n) { return n >= 15 && n <= 31; }

std::vector<CWidePass> cwide_plan(const std::vector<HostOp>& ops, const std::vector<int>& idx, int n) {
  std::vector<CWidePass> out;
  CWidePass cur;
  std::vector<int> stage;
  uint64_t all = 0, sb = 0;  // bits of the pass's gates, of the stage's
  int gates = 0, signs = 0;
  // the pass's bits with the lowest qubits must fit the tile
  auto tile_bits = [&](uint64_t b) { return __builtin_popcountll(b | ((1u << CW_LEAD) - 1)); };
  auto end_stage = [&]() {
    if (!stage.empty()) cur.stages.push_back(stage);
    stage.clear();
    sb = 0;
  };
  auto end_pass = [&]() {
    end_stage();
    if (!cur.stages.empty()) out.push_back(cur);
    cur = CWidePass();
    all = 0;
    gates = signs = 0;
  };
  for (int i : idx) {
    const HostOp& op = ops[i];
    if (op.type == OP_SIGN) {
      if (signs == CW_MAX_SIGNS) end_pass();
      ++signs;
      stage.push_back(i);
      continue;
    }
    const uint64_t b = bits_of(op);
    const bool fits_stage = __builtin_popcountll(sb | b) <= CW_RB;
    const bool fits_pass = tile_bits(all | b) <= CW_T && gates < CW_MAX_GATES &&
                           (fits_stage || (int)cur.stages.size() < 2);
    if (!fits_pass) end_pass();
    else if (!fits_stage) end_stage();
    sb |= b;
    all |= b;
    ++gates;
    stage.push_back(i);
  }
  end_pass();
  return out;
}

int cwide_run(const void* in, void* out, int n, const std::vector<HostOp>& ops, const CWidePass& pass,
              cudaStream_t stream) {
  static thread_local CWParams P;
  std::memset(&P, 0, sizeof(P));
  P.in = static_cast<const float2*>(in);
  P.out = static_cast<float2*>(out);
  P.n = n;
  uint64_t all = 0;
  for (const auto& st : pass.stages)
    for (int i : st)
      if (ops[i].type != OP_SIGN) all |= bits_of(ops[i]);
  std::vector<int> tile;
  for (int b = 0; b < n; ++b)
    if ((all >> b) & 1) tile.push_back(b);
  for (int b = 0; b < n && (int)tile.size() < CW_T; ++b)
    if (!((all >> b) & 1)) tile.push_back(b);
  if ((int)tile.size() != CW_T) return QF_ERR_NOT_SUPPORTED;
  std::sort(tile.begin(), tile.end());
  for (int j = 0; j < CW_T; ++j) P.tb[j] = (uint8_t)tile[j];
  auto local = [&](int bit) { return (int)(std::find(tile.begin(), tile.end(), bit) - tile.begin()); };
  int ng = 0, ns = 0;
  // arrangement with register bits reg[0..3] (local bits, ascending)
  auto arrange = [&](const int* reg) -> CWStage& {
    CWStage& S = P.st[P.nstages++];
    uint32_t used = 0;
    for (int j = 0; j < CW_RB; ++j) used |= 1u << reg[j];
    int t = 0;
    for (int j = 0; j < CW_T; ++j)
      if (!((used >> j) & 1)) S.tpos[t++] = (uint8_t)j;
    for (int j = 0; j < CW_RB; ++j) {
      const uint32_t l = 1u << reg[j];
      S.roff[j] = 1u << tile[reg[j]];
      S.rloc[j] = cw_swz(l);
    }
    S.sign_begin = (uint8_t)ns;
    S.sign_end[0] = (uint8_t)ns;
    return S;
  };
  static const int top[CW_RB] = {CW_T - 4, CW_T - 3, CW_T - 2, CW_T - 1};
  for (size_t s = 0; s < pass.stages.size(); ++s) {
    uint64_t sb = 0;
    for (int i : pass.stages[s])
      if (ops[i].type != OP_SIGN) sb |= bits_of(ops[i]);
    int reg[CW_RB], nr = 0;
    for (int j = 0; j < CW_T; ++j)
      if ((sb >> tile[j]) & 1) reg[nr++] = j;
    for (int j = CW_T - 1; nr < CW_RB && j >= 0; --j)  // the rest: the highest tile bits
      if (std::find(reg, reg + nr, j) == reg + nr) reg[nr++] = j;
    std::sort(reg, reg + CW_RB);
    // registers on the lowest bits would scatter the loads and stores: the
    // tile is then loaded (stored) by its top bits and re-arranged
    if (s == 0 && reg[0] < CW_LEAD) arrange(top);
    CWStage& S = arrange(reg);
    auto reg_of = [&](int bit) {
      const int l = local(bit);
      for (int j = 0; j < CW_RB; ++j)
        if (reg[j] == l) return j;
      return -1;
    };
    uint32_t rbits = 0;
    for (int j = 0; j < CW_RB; ++j) rbits |= 1u << tile[reg[j]];
    for (int i : pass.stages[s]) {
      const HostOp& op = ops[i];
      if (op.type == OP_SIGN) {
        if (ns == CW_MAX_SIGNS) return QF_ERR_NOT_SUPPORTED;
        uint32_t m = 0;
        int jm = 0;
        for (int j = 0; j < op.k; ++j) {
          m |= 1u << op.gb[j];
          if (reg_of(op.gb[j]) >= 0) jm |= 1 << reg_of(op.gb[j]);
        }
        P.mout[ns] = m & ~rbits;
        P.rmask[ns] = 0;
        for (int r = 0; r < CW_R; ++r)
          if ((r & jm) == jm) P.rmask[ns] |= (uint16_t)(1u << r);
        S.sign_end[S.ngates] = (uint8_t)++ns;
        continue;
      }
      if (ng == CW_MAX_GATES) return QF_ERR_NOT_SUPPORTED;
      CWGate& G = P.gates[ng];
      auto put = [&](int e, cplx v) {
        const float re = static_cast<float>(v.real()), im = static_cast<float>(v.imag());
        G.c[e] = make_float4(re, re, im, im);
      };
      if (op.k == 1) {
        S.kind[S.ngates] = (uint8_t)(CWK_D1 + reg_of(op.gb[0]));
        for (int e = 0; e < 4; ++e) put(e, op.m[e]);
      } else {
        const int ja = reg_of(op.gb[0]), jb = reg_of(op.gb[1]);
        const int hi = std::max(ja, jb), lo = std::min(ja, jb);
        S.kind[S.ngates] = (uint8_t)(CWK_D2 + hi * (hi - 1) / 2 + lo);
        auto sw = [&](int x) { return ja > jb ? x : ((x & 1) << 1) | (x >> 1); };  // matrix MSB on hi
        for (int r = 0; r < 4; ++r)
          for (int c = 0; c < 4; ++c) put(4 * r + c, op.m[sw(r) * 4 + sw(c)]);
      }
      S.gate[S.ngates++] = (uint8_t)ng++;
      S.sign_end[S.ngates] = (uint8_t)ns;
    }
    if (s + 1 == pass.stages.size() && reg[0] < CW_LEAD) arrange(top);
  }
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < 64 && !attr[dev].load()) {
    int rc = check_cuda(cudaFuncSetAttribute(k_cwide, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CW_SMEM));
    if (rc) return rc;
    attr[dev].store(true);
  }
  int64_t grid = int64_t(1) << (n - CW_T);
  const int64_t cap = 2 * device_sm_count();
  if (grid > cap) grid = cap;
  k_cwide<<<(int)grid, CW_NT, CW_SMEM, stream>>>(P);
  return check_cuda(cudaGetLastError());
}

}  // namespace qf
