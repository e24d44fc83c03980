// gd_tc.cuh -- split-precision (TF32x3 / BF16x3) Legendre GEMMs on the
// sm_103a tensor cores (tcgen05 + TMEM + TMA).  Declarations.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>

#include <array>

#include "gd_kernels.h"

namespace gd {

// the driver's cuTensorMapEncodeTiled
PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder();

enum TcKind { TC_TF32 = 0, TC_BF16 = 1 };

// Tables and staging buffers of the tensor-core Legendre path for one grid.
struct TcPlan {
  int kind = TC_TF32;
  int T = 0, nh = 0, nlat = 0;
  int esize = 4;    // bytes per operand element (4 tf32, 2 bf16)
  int kc = 32;      // K elements per 128-byte swizzle row
  int kepad = 0;    // padded even/odd K extent of the synthesis tables
  int nhpad = 0;    // padded latitude extent of the analysis operands
  int nsyn = 0;     // N tile (latitudes) of the synthesis GEMM
  int nana = 0;     // N tile (degrees per parity) of the analysis GEMM
  int kirows = 0;   // rows per parity of the analysis tables
  int ncap = 0;     // real-column capacity of the staging buffers
  bool persistent = true;  // persistent warp-specialised GEMM (N <= 128)
  // fused TF32x3 GEMM: the hi*lo and lo*hi products in their own accumulator
  // (a third of the truncating accumulation steps in the main one); set by
  // the FP64-state modes (and GD_TC_SEPX) before tc_init (it bounds the N
  // tile)
  bool sepx = false;
  // fused TF32x3 GEMM: K segments of cps chunks per parity, accumulated afresh
  // and folded in FP32 (round to nearest) by the epilogue; 0 = none; set
  // before tc_init (it bounds the N tile)
  int cps = 0;
  // fused TF32x3 GEMM: A-operand slots in tensor memory requested (2..4; a
  // launch gets as many as fit beside its accumulators)
  int aslots = 2;
  // widest N tile tc_init chooses for the fused TF32x3 GEMM, as far as tensor
  // memory holds it (tiles above 96 are single-buffered).  A chunk's operand tile
  // is read from L2 once per N tile, and that traffic bounds the GEMM: cap 96 ->
  // 192, one step's syntheses and analyses T574L64 8.22 -> 6.89 and 5.12 -> 4.72
  // ms, T382L64 3.19 -> 2.90 and (capped at 160) the same, T254L64 1.32 -> 1.20 and
  // 1.17 -> 1.07, T170L64 0.63 -> 0.54 ms; T126 and below need no wider tile
  int tile_cap = 192;
  // fused TF32x3 analysis: the latitude sum in aseg segments, each written as
  // FP32 partial sums to its own copy of the output (nlm x ldA floats apart),
  // to be added in the caller's precision; set by the FP64-state modes
  int aseg = 1;
  int nsm = 0;             // SMs of the device (persistent grid size)
  long xlen = 0;    // padded spectral length of the synthesis operand
  std::vector<long> xbase;  // [T+1] start of order m in the padded layout
  long* d_xbase = nullptr;
  // tables: synthesis [m][j][2*kepad], analysis [m][2*kirows][nhpad]; hi/lo
  void* tsyn[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};  // [P/H][hi/lo]
  void* tana[2][2] = {{nullptr, nullptr}, {nullptr, nullptr}};
  // staging: X [ncap][xlen] hi/lo; G+- [T+1][ncap][nhpad] hi/lo
  void* x[2] = {nullptr, nullptr};
  void* gp[2] = {nullptr, nullptr};
  void* gm[2] = {nullptr, nullptr};
  CUtensorMap m_tsyn[2][2], m_tana[2][2], m_x[2], m_gp[2], m_gm[2];
  std::vector<std::pair<long, int4*>> item_cache;  // work lists by (ncols, direction)
  std::vector<std::pair<std::array<uint64_t, 9>, CUtensorMap>> raw_maps;  // fused-path maps by geometry
  int* d_xmap = nullptr;  // padded synthesis position -> spectral index (or -1)
  // error flag, nonzero: a bounded wait gave up.  Page-locked host memory of the
  // caller's, set before init; kernels write it in that case alone
  int* err = nullptr;
  std::vector<void*> allocs;
};

// Builds tables (from the FP64 tables), staging buffers and tensor maps.
void tc_init(TcPlan& p, int kind, int T, int nh, int nlat, int ncap, const long* d_toff, const double* P64,
             const double* H64, cudaStream_t s);
void tc_free(TcPlan& p);
// the balanced tile at most cap wide over n rows (a multiple of 16)
int tc_tile_n(int n, int cap);
// largest N tile the plan's GEMM kernel takes (TMEM budget)
int tc_max_n(const TcPlan& p);
// A slots a fused launch at N tile n gets (the request, as far as TMEM holds)
int tc_slots(const TcPlan& p, int n);
// switches the synthesis GEMM to latitude tile nsyn (autotuning)
void tc_set_nsyn(TcPlan& p, int nsyn);

// One transform's columns through a table (useH: dP/dphi); the fused kernel
// takes one or two (both tables, any arrays) in a launch.
struct TcLeg {
  bool useH;
  const float* in;
  long ldin;
  int ncols;
  float* out;
  long ldout;
};
// Legendre synthesis out[m][j][c] of each leg's real columns [0, ncols) of
// in[idx][.] (nrowsB rows allocated).  The fused path reads the input in pairs of
// rows, so it needs 2 floor(nrowsB / 2) >= nlm; otherwise the split path runs.
void tc_synth(TcPlan& p, const long* d_moff, const TcLeg* legs, int n, long nrowsB, cudaStream_t s);
// Legendre analysis out[idx][c] of each leg's in[m][j][c], real columns [0, ncols)
void tc_anal(TcPlan& p, const long* d_moff, const TcLeg* legs, int n, cudaStream_t s);
// the K segments tc_anal uses (the plan's aseg, at most one per latitude chunk)
int tc_anal_segments(const TcPlan& p);

// A chain of dense layers of the closure network on the tensor cores, one
// launch: layer l takes the rows of the layer before it (the first x [M][ldx])
// to acc[m][n] = sum_k A[m][k] W[n][k] (+ bias[n]), W in BF16, A carried as BF16
// hi + mid + lo (the FP32 value), FP32 accumulation in TMEM, then
//   act 0: acc; 1: GELU(acc); 2: acc GELU'(zin[m][n]) (the backward chain).
// Optional copies in FP32, row pitch ldz: z (acc), out (the layer's result).
// The last layer's result goes to y.  N <= 256 (every layer), K <= 256 but for
// the first.  wrow: the layer's first row in the packed weights, rows of
// kpitch BF16 zero-padded past K, each layer's block a multiple of 64 rows.
struct TcChainLayer {
  int N, K, wrow, act;
  const float* bias;
  float* z;
  float* out;
  const float* zin;
  int ldz;
};
void tc_chain_map(CUtensorMap* m, const void* w, int kpitch, long rows);
// layers: device array
void tc_chain(const CUtensorMap& w, const TcChainLayer* layers, int nl, const float* x, int ldx, int M, float* y,
              int ldy, int* err, cudaStream_t s);

// Weight gradients of the closure's layers, one launch: item i, slice q:
// part[q][poff + m Np + n] = sum over the slice's K chunks of A(arow + m, k)
// B(brow + n, k), m < 128, n < Np; both operands TF32 hi + lo rows with the
// batch (K) contiguous: A the layers' dZ^T stacked (blocks of 128 rows), B
// their inputs transposed (Np <= 256, blocks of 64 rows).  Three products per K
// step (hi hi, hi lo, lo hi), FP32 accumulation in TMEM; the slices' partial
// tiles are summed afterwards in a fixed order.
struct TcWgradItem {
  int arow, brow, Np;
  long poff;
};
struct TcWgrad {
  CUtensorMap ah, al, bh, bl;
  const TcWgradItem* items = nullptr;  // device array
  int nitems = 0;
  float* part = nullptr;
  long pstride = 0;
  int* err = nullptr;
};
// maps over the stacked transposed operands; kpitch = their row length (a
// multiple of 32)
void tc_wgrad_maps(TcWgrad& W, const uint32_t* ah, const uint32_t* al, const uint32_t* bh, const uint32_t* bl,
                   long arows, long brows, int kpitch);
// nk = K chunks of 32 in use, split over nsplit slices of cps chunks each
// (every slice non-empty), the partial tiles from slice0 on
void tc_wgrad(const TcWgrad& W, int nk, int cps, int nsplit, int slice0, cudaStream_t s);

}  // namespace gd
