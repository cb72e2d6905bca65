// Complex64 gate passes on tiles of 2^13 amplitudes (cwide.cu).
#pragma once
#include <cstdint>
#include <vector>

#include "engine.cuh"

namespace qf {

constexpr int CW_T = 13;           // tile bits
constexpr int CW_RB = 4;           // register bits
constexpr int CW_MAX_STAGES = 5;   // arrangements of a pass (load and store among them)
constexpr int CW_MAX_GATES = 12;
constexpr int CW_MAX_SIGNS = 64;
constexpr int CW_LEAD = 3;         // lowest qubits every tile holds (64-byte runs)

// A pass: stages of gates on at most four bits each, over at most
// CW_T - CW_LEAD bits in all.
struct CWidePass {
  std::vector<std::vector<int>> stages;  // op indices in order
};
// Cut the ops `idx` (2x2 and 4x4 gates and signs only) into passes.
std::vector<CWidePass> cwide_plan(const std::vector<HostOp>& ops, const std::vector<int>& idx, int n);
int cwide_run(const void* in, void* out, int n, const std::vector<HostOp>& ops, const CWidePass& pass,
              cudaStream_t stream);
bool cwide_op(const HostOp& op);
// smallest and largest state the passes are used for
bool cwide_fits(int n);

}  // namespace qf
