// QAOA forward state and adjoint gradient of one complex64 instance, two
// register groups a pass (device bodies and pass lists: qpair.cuh).
//
// Reference semantics: quantumflow/qaoa.py:22-64 and
// examples/qaoa_maxcut.py:56-64, as in qaoa.cu and adjoint.cu, whose
// warp-tile passes these replace from 13 qubits on: the same operations in
// the same order, half of the passes over the state.
// Bound: HBM (adjoint passes, 106 us at n = 24 of 80 at the copy rate); the
// forward passes, 66 us of 40, FP32 issue and shuffles at the layer
// boundaries.  n = 24, p = 6: 4967 -> 2960 us a gradient evaluation
// (forward 25 passes -> 13, adjoint 37 -> 19).
#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstring>
#include <vector>

#include "engine.cuh"
#include "qpair.cuh"
#include "state.cuh"

namespace qf {

namespace {

constexpr int QP_MAX_COEF = 1024;
constexpr int QP_RBF = 4, QP_RBA = 3;  // register bits, those of the complex64 warp tiles

struct QPairParams {
  PairPass F;
  float2* psi;
  float2* lam;
  const uint16_t* cuts;
  double* rows;
  int32_t n, nslots, ncut;
  int32_t slot_a, slot_cut, slot_e, slot_b;
  float wref;
  Coef amp0, ac, as, bc, bs;
  Coef coef[QP_MAX_COEF];
};

QF_D unsigned char* qp_table(const QPairParams& P, unsigned char* smem) {
  Coef* tab = reinterpret_cast<Coef*>(smem);
  if (P.F.cost)
    for (int i = threadIdx.x; i < P.ncut; i += blockDim.x) tab[i] = P.coef[i];
  __syncthreads();
  pdl_wait();
  return smem + ((P.ncut * sizeof(Coef) + 127) & ~size_t(127));
}

__global__ void __launch_bounds__(PairShape<C64, QP_RBF>::NT, 2) k_qpair_fwd(const __grid_constant__ QPairParams P) {
  extern __shared__ __align__(128) unsigned char qp_smem[];
  unsigned char* buf = qp_table(P, qp_smem);
  pair_forward<C64, QP_RBF, false>(P.F, P.psi, P.cuts, reinterpret_cast<const Coef*>(qp_smem), P.ncut,
                            make_float2(P.amp0.f[0], P.amp0.f[2]), P.ac, P.as, P.bc, P.bs, blockIdx.x, gridDim.x,
                            1u << (P.n - 5 - 2 * QP_RBF), buf);
}

__global__ void __launch_bounds__(PairShape<C64, QP_RBA>::NT, 3) k_qpair_adj(const __grid_constant__ QPairParams P) {
  extern __shared__ __align__(128) unsigned char qp_smem[];
  __shared__ double red[8][4];
  unsigned char* buf = qp_table(P, qp_smem);
  PairSums S{};
  pair_adjoint<C64, QP_RBA, false>(P.F, P.psi, P.lam, P.cuts, reinterpret_cast<const Coef*>(qp_smem), P.ncut, P.wref,
                                   P.ac, P.as, P.bc, P.bs, blockIdx.x, gridDim.x, 1u << (P.n - 5 - 2 * QP_RBA), buf,
                                   S);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double v[4] = {warp_sum((double)S.a.s + (double)S.a.e), warp_sum((double)S.cut.s + (double)S.cut.e),
                       warp_sum((double)S.e.s + (double)S.e.e), warp_sum((double)S.b.s + (double)S.b.e)};
  if (lane == 0)
    for (int k = 0; k < 4; ++k) red[warp][k] = v[k];
  __syncthreads();
  if (threadIdx.x < 4) {
    const int k = threadIdx.x;
    const int slot = k == 0 ? P.slot_a : k == 1 ? P.slot_cut : k == 2 ? P.slot_e : P.slot_b;
    if (slot >= 0) {
      double t = 0.0;
      for (int w = 0; w < 8; ++w) t += red[w][k];
      P.rows[(size_t)blockIdx.x * P.nslots + slot] += (k == 1 ? -2.f : 1.f) * t;
    }
  }
}

template <int RB>
size_t qp_smem(int vectors, int ncut) {
  return ((ncut * sizeof(Coef) + 127) & ~size_t(127)) + (1 + vectors) * PairShape<C64, RB>::VEC;
}
int qp_grid(int n, int RB, int per_sm) {
  const int64_t tiles = int64_t(1) << (n - 5 - 2 * RB), cap = (int64_t)device_sm_count() * per_sm;
  return (int)(tiles < cap ? tiles : cap);
}
int qp_attr() {
  static std::atomic<bool> attr[64];
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64 || attr[dev].load()) return QF_OK;
  int rc = check_cuda(cudaFuncSetAttribute(k_qpair_fwd, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                           (int)qp_smem<QP_RBF>(0, QP_MAX_COEF)));
  if (rc) return rc;
  rc = check_cuda(cudaFuncSetAttribute(k_qpair_adj, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                       (int)qp_smem<QP_RBA>(2, QP_MAX_COEF)));
  if (rc) return rc;
  attr[dev].store(true);
  return QF_OK;
}

}  // namespace

bool qpair_fits(int n, int layout, int nedges, int p, const double* node_theta) {
  if (node_theta != nullptr)
    for (int q = 0; q < n; ++q)
      if (!std::isnan(node_theta[q])) return false;
  return layout == C64 && p > 0 && n >= pair_min_qubits(QP_RBF) && n <= 31 && nedges + 1 <= QP_MAX_COEF;
}

int qpair_state(void* psi, int n, const uint16_t* cuts, int nedges, int p, const double* beta, const double* gamma,
                cudaStream_t stream) {
  int rc = qp_attr();
  if (rc) return rc;
  static thread_local QPairParams P;
  std::memset(&P, 0, sizeof(P));
  P.psi = static_cast<float2*>(psi);
  P.cuts = cuts;
  P.n = n;
  P.ncut = nedges + 1;
  P.amp0 = make_coef(cplx(std::ldexp(1.0, -n / 2) / ((n & 1) ? std::sqrt(2.0) : 1.0), 0.0), C64);
  auto rx = [&](int l, Coef& c, Coef& s) {
    c = make_coef(cplx(std::cos(0.5 * beta[l]), 0.0), C64);
    s = make_coef(cplx(-std::sin(0.5 * beta[l]), 0.0), C64);
  };
  const int grid = qp_grid(n, QP_RBF, 2);
  for (const PairPass& F : pair_fwd_passes(n, p, QP_RBF)) {
    P.F = F;
    if (F.hasA) rx(F.layerA, P.ac, P.as);
    if (F.hasB) {
      rx(F.layerB, P.bc, P.bs);
      for (int cv = 0; cv <= nedges; ++cv)
        P.coef[cv] = make_coef(std::polar(1.0, gamma[F.layerB] * (0.5 * nedges - cv)), C64);
    }
    rc = pdl_launch(k_qpair_fwd, grid, PairShape<C64, QP_RBF>::NT, qp_smem<QP_RBF>(0, P.ncut), stream, P);
    if (rc) return rc;
  }
  return QF_OK;
}

// adjoint sweep from the final state in psi (left at |+>^n); returns the
// number of rows of partial sums (nslots doubles each, zeroed by the caller)
int qpair_grad(void* psi, void* lam, int n, const uint16_t* cuts, int nedges, int p, const double* beta,
               const double* gamma, double* rows, int nslots, int* nrows, cudaStream_t stream) {
  int rc = qp_attr();
  if (rc) return rc;
  static thread_local QPairParams P;
  std::memset(&P, 0, sizeof(P));
  P.psi = static_cast<float2*>(psi);
  P.lam = static_cast<float2*>(lam);
  P.cuts = cuts;
  P.rows = rows;
  P.n = n;
  P.nslots = nslots;
  P.ncut = nedges + 1;
  const double half_e = 0.5 * nedges;
  P.wref = (float)half_e;
  auto rx = [&](int l, Coef& c, Coef& s) {  // RX(-beta)
    c = make_coef(cplx(std::cos(0.5 * beta[l]), 0.0), C64);
    s = make_coef(cplx(std::sin(0.5 * beta[l]), 0.0), C64);
  };
  const int grid = *nrows = qp_grid(n, QP_RBA, 3);
  for (const PairPass& F : pair_adj_passes(n, p, QP_RBA)) {
    const int l = F.layerA;
    P.F = F;
    rx(l, P.ac, P.as);
    if (F.hasB) rx(F.layerB, P.bc, P.bs);
    if (F.cost)
      for (int cv = 0; cv <= nedges; ++cv) P.coef[cv] = make_coef(std::polar(1.0, -gamma[l] * (half_e - cv)), C64);
    P.slot_a = p + l;
    P.slot_cut = F.cost ? l : -1;
    P.slot_e = F.init ? 2 * p : -1;
    P.slot_b = F.hasB ? p + l - 1 : -1;
    rc = pdl_launch(k_qpair_adj, grid, PairShape<C64, QP_RBA>::NT, qp_smem<QP_RBA>(2, P.ncut), stream, P);
    if (rc) return rc;
  }
  return QF_OK;
}

}  // namespace qf
