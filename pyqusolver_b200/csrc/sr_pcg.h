// Internal interface of the persistent CG kernel (sr_pcg.cu) used by sr.cu.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>
#include <stdint.h>

#include "sr_tc.h"

struct PcgDims {
  int ns, nh;
  int Mh;            // hidden units padded to 8 (complex) / 16 (real): rows of one operand half
  int NZ;            // operand rows / accumulator columns: 2 Mh (complex) or Mh (real)
  int Kz;            // sites + the ones column, padded to 16 (K of O v)
  int R;             // samples per CTA (multiple of 16, at most 128)
  int n_chunks;      // CTAs that hold samples
  int G;             // CTAs of the grid (all resident): n_chunks, or more where the vectors need them
  int S;             // operand stages in shared memory
  int vpc, groups;   // 16-byte vectors of the parameter vector per CTA, split groups of the reduction
  int64_t nvec;      // 16-byte vectors of one partial (W rows and g_b, then g_a)
  int nc;            // collectors of a grid-wide sum
  int tmem_cols, smem;
};

// test hook: the wait that runs out (in pass -2, -1, 0, ...; DIRECTION and COPY from pass 0 on) and the polls before it does
struct PcgWaitTest {
  enum { NONE = 0, PARTIALS = 1, SUM = 2, DIRECTION = 3, COPY = 4 };
  int which, pass;
  uint32_t polls;
};

// whether the shapes admit the persistent kernel, and its tiling
bool pcg_plan(int dtype, int ns, int nh, int64_t n_samples, PcgDims* d);
size_t pcg_partial_bytes(const PcgDims& d);
size_t pcg_operand_bytes(const PcgDims& d);        // direction operand tiles and v_a
size_t pcg_slot_bytes(const PcgDims& d);

struct PcgArgs {
  const uint32_t* bits; const void* tt; const float2* eloc; const float* wts;
  double shift, rtol, atol, prefactor; int maxiter;
  void *x, *b, *x_out;                              // [P]: x, the force, prefactor * x
  double* scal;                                     // solver state, as the kernel chain leaves it
  void* partial; void* operand; double* slots; int* status; int* err;
};
int pcg_solve(int dtype, const PcgDims& d, int64_t n_samples, const PcgArgs& a, cudaStream_t st);
