// QAOA on wide tiles (qtile.cu): forward state and adjoint gradient of
// float-float states.
#pragma once
#include <cstddef>
#include <cstdint>
#include <cuda_runtime.h>

namespace qf {

bool qtile_fits(int n, int layout, int nedges, int p, const double* node_theta);
size_t qtile_grad_rows(int n, int layout);
int qtile_state(void* psi, int n, const uint16_t* cuts, int nedges, int p, const double* beta, const double* gamma,
                bool keep_phi, cudaStream_t stream);
int qtile_grad(void* psi, void* lam, int n, const uint16_t* cuts, int nedges, int p, const double* beta,
               const double* gamma, double* rows, int nslots, cudaStream_t stream);

// Two register groups a pass (qpair.cu): one complex64 instance.  The number
// of rows of partial sums is at most that of the warp-tile sweep.
bool qpair_fits(int n, int layout, int nedges, int p, const double* node_theta);
int qpair_state(void* psi, int n, const uint16_t* cuts, int nedges, int p, const double* beta, const double* gamma,
                cudaStream_t stream);
int qpair_grad(void* psi, void* lam, int n, const uint16_t* cuts, int nedges, int p, const double* beta,
               const double* gamma, double* rows, int nslots, int* nrows, cudaStream_t stream);

}  // namespace qf
