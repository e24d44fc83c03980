// gd_oz.cuh -- FP64 Legendre GEMMs on the tensor cores by exact splitting
// (gd_oz.cu).  Declarations.
#pragma once
#include <cuda.h>

#include <vector>

#include "gd_kernels.h"

namespace gd {

// Tables and operand buffers of the FP64 tensor-core Legendre path for one
// grid, orders m >= 1.  An FP64 operand row (a batch column over the degrees or
// latitudes, a table row) is a power of two times a 62-bit integer, its eight
// signed base-256 digits kept as BF16 slices.
struct OzPlan {
  int T = 0, nh = 0, nlat = 0;
  int nhpad = 0;   // padded latitudes of the analysis operands
  int nsyn = 0, nana = 0;  // N tiles: latitudes, degrees per parity
  int ncap = 0;    // column capacity
  long nlm = 0;
  int nsm = 0;
  long xlen = 0;
  // start of order m along the degrees of the synthesis operand and tables
  // (both parities, each padded to the chunk)
  long* d_xbase = nullptr;
  // digits: synthesis tables [8][nh][xlen], analysis tables [8][nlm][nhpad] (an
  // order's even degrees, then its odd ones); operands X [8][ncap][xlen] and, per
  // parity, G [8][(T+1) ncap][nhpad], in the same memory.  A tile that reaches past its own rows reads
  // other rows' digits into outputs that are not stored.
  void *tsyn[2] = {nullptr, nullptr}, *tana[2] = {nullptr, nullptr};
  void *x = nullptr, *g[2] = {nullptr, nullptr};
  // binary exponents of the rows
  int *esyn[2] = {nullptr, nullptr}, *eana[2] = {nullptr, nullptr}, *ex = nullptr, *eg[2] = {nullptr, nullptr};
  CUtensorMap m_tsyn[2], m_tana[2], m_x, m_g[2];
  // work lists by the legs' column tiles and the direction (0 synthesis, 1 analysis)
  struct Items {
    int ct[2], mode, n;
    int4* d;
  };
  std::vector<Items> items;
  // error flag, nonzero: a bounded wait gave up.  Page-locked host memory of the
  // caller's, set before init; kernels write it in that case alone
  int* err = nullptr;
  void* mem = nullptr;  // all of the above but the work lists
};

// false, and nothing kept, where the digits of the tables and of ncap operand
// columns take more than `limit` bytes or than the device has left, or where
// there is no order m >= 1
bool oz_init(OzPlan& p, int T, int nh, int nlat, int ncap, size_t limit, const long* d_moff, const long* d_toff,
             const double* P, const double* H, cudaStream_t s);
void oz_free(OzPlan& p);
// Legendre transform of `ncols` real columns through the P or the dP/dphi table, orders m >= 1
struct OzLeg {
  bool useH;
  const double* in;
  long ldin;
  int ncols;
  double* out;
  long ldout;
};
// syntheses F[m][j][c] of B[nlm][c], analyses A[nlm][c] of G[m][j][c]: one or two
// legs in a launch, within the capacity; a synthesis' second leg reads columns of the first
void oz_synth(OzPlan& p, const long* d_moff, const OzLeg& a, const OzLeg* b, cudaStream_t s);
void oz_anal(OzPlan& p, const long* d_moff, const OzLeg& a, const OzLeg* b, cudaStream_t s);

}  // namespace gd
