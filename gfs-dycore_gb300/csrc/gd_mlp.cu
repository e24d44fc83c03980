// gd_mlp.cu -- the learned per-column closure's network: a fully connected
// net nin -> nh (GELU) -> ... -> nh (GELU) -> nout with BF16 weights and FP32
// accumulation.  Forward and backward passes, the mean-squared-error loss and
// Adam run as CUDA kernels on the net's stream; the dycore applies a trained
// net to its grid columns once per step (gd_set_closure, gd_dycore.cu).
//
// Parameters are one FP32 master array, layer after layer: W_l [fout][fin]
// row-major, then b_l [fout].  The forward and backward passes read the
// weights from a BF16 copy made after every update (biases stay FP32), so a
// trained net is exactly the BF16 net it is evaluated as.
//
// The products with the batch (the grid's columns) as rows, X W^T and dZ W,
// run on the tensor cores when every layer is at most 256 wide: one launch
// (k_tc_chain in gd_tc.cu) takes 128 rows through all layers with the
// activations on chip, as BF16 hi + mid + lo slices against the BF16 weights,
// so three MMAs per K step give the FP32 products of the BF16 net.  That
// covers inference (gd_mlp_forward and the closure in the step), the training
// forward pass (which also stores each hidden layer's Z and A) and the chain
// of backward products dZ_l W_l with the GELU derivative fused.  The weights
// it reads are packed (padded, and transposed for the backward chain) once
// per update.  The weight gradients dZ^T A, reductions over the batch, run on
// the tensor cores too (k_tc_wgrad, all layers in one launch): the operands
// transposed with the batch contiguous and split hi + lo (k_tsplit), the batch
// in slices whose partial tiles k_wsum adds in order.  Nets wider than 256
// (and GD_MLP_TRAIN_TC=0) train on a tiled SIMT GEMM: 64 x 64 output tiles, K
// in steps of 16 through shared memory, 4 x 4 outputs per thread, operands
// addressed through (row, column) strides, split K for the weight gradient.
#include <cuda_bf16.h>

#include <cmath>
#include <cstdlib>
#include <cstdint>
#include <memory>
#include <random>
#include <stdexcept>
#include <string>
#include <vector>

#include "gd_api.h"
#include "gd_common.cuh"
#include "gd_mlp.cuh"
#include "gd_tc.cuh"

namespace gd {
// a packed weight row: cnt entries of the BF16 copy from off on, stride apart
struct PackRow {
  long off;
  int stride, cnt;
};
// transposing split: src [n][w] (null: the batch's inputs) to rows of dh, dl;
// boff >= 0: also the column sums, into the bias partials from boff on
struct TsplitJob {
  const float* src;
  int w, boff;
  uint32_t *dh, *dl;
};
// where a layer's gradient entries are: in the packed gradient (offw, offb),
// the partial tiles and the bias partials
struct WgradLayer {
  long offw, offb, poff;
  int fo, fi, Np, boff;
};
constexpr int kSlab = 32768;  // columns of the batch transposed at a time
constexpr int kTrows = 128;   // columns of the batch per k_tsplit CTA
}  // namespace gd

struct gd_mlp {
  int device = 0;
  int nin = 0, nh = 0, nl = 0, nout = 0;  // nl hidden layers
  int nlayer = 0;                          // nl + 1 linear layers
  std::vector<int> fin, fout;
  std::vector<long> offw, offb;  // offsets of W_l and b_l in the parameter array
  long np = 0;
  float* p32 = nullptr;          // master parameters
  __nv_bfloat16* w16 = nullptr;  // BF16 copy (all np entries; the bias slots are unused)
  float* grad = nullptr;
  float* am = nullptr;  // Adam moments
  float* av = nullptr;
  long adam_t = 0;
  // normalisation of the closure's inputs and outputs (device, nin / nout)
  float *in_mu = nullptr, *in_sd = nullptr, *out_mu = nullptr, *out_sd = nullptr;
  bool has_norm = false;
  // activations: Z_l (pre-activation) and A_l (GELU) of each hidden layer,
  // the output and its gradient, two gradient buffers for the backward pass
  int bcap = 0;
  float *zb = nullptr, *ab = nullptr, *yb = nullptr, *gy = nullptr, *g0 = nullptr, *g1 = nullptr;  // g0, g1: SIMT
  float* partial = nullptr;  // loss partial sums
  float* kpart = nullptr;    // split-K partial weight gradients
  float* lossd = nullptr;
  // tensor-core chains (gd_tc.cu): the weights packed as rows of kpf BF16
  // (wpf, every layer's W_l) and of kpb (wpb, the transposed W_l of l >= 1),
  // each layer's block padded to 64 rows; pack = where each packed row comes
  // from.  Layer tables (device): inference, training forward, backward.
  bool tc = false, tcb = false;
  int kpf = 0, kpb = 0;
  long rowsf = 0, rowsb = 0;
  std::vector<int> wrowf, wrowb;
  __nv_bfloat16 *wpf = nullptr, *wpb = nullptr;
  gd::PackRow* pack = nullptr;
  CUtensorMap mapf, mapb;
  gd::TcChainLayer *inf_layers = nullptr, *trn_layers = nullptr, *bwd_layers = nullptr;
  float* dzb = nullptr;  // dZ of the hidden layers, [nl][bcap][nh]
  // weight gradients: dZ^T and the layers' inputs transposed, stacked and
  // split over a slab of the batch (kSlab columns at most), the slices'
  // partial tiles, the bias gradients' partial sums
  gd::TcWgrad wg;
  uint32_t *zth = nullptr, *ztl = nullptr, *ath = nullptr, *atl = nullptr;
  gd::WgradLayer* wlay = nullptr;  // device, one per layer
  gd::TsplitJob* jobs = nullptr;   // device, two per layer
  float *wpart = nullptr, *bpart = nullptr;
  int nbias = 0, opcols = 0;  // columns of the transposed operands (slab capacity)
  int tcap = 0;               // batch capacity of the training buffers
  int nsm = 0;
  int* terr = nullptr;
  float* hres = nullptr;  // page-locked: error flag and loss on their way out
  cudaStream_t stream = nullptr;  // the stream the net's work runs on
  cudaStream_t own = nullptr;     // the net's own stream (destroyed with it)
  std::string err;
  std::vector<void*> allocs;
  void* alloc(size_t bytes) {
    void* p = nullptr;
    GD_CUDA(cudaMalloc(&p, std::max<size_t>(bytes, 16)));
    allocs.push_back(p);
    return p;
  }
  // Gives back what was allocated since it was made, unless kept: a growth of
  // the net's buffers that fails leaves the net as it was.
  struct Growth {
    gd_mlp* p;
    size_t n;
    bool kept = false;
    explicit Growth(gd_mlp* q) : p(q), n(q->allocs.size()) {}
    ~Growth() {
      if (kept) return;
      cudaStreamSynchronize(p->stream);
      for (; p->allocs.size() > n; p->allocs.pop_back()) cudaFree(p->allocs.back());
    }
  };
  ~gd_mlp() {
    int cur = 0;
    if (cudaGetDevice(&cur) == cudaSuccess && cur != device) cudaSetDevice(device);
    if (stream) cudaStreamSynchronize(stream);
    for (void* p : allocs)
      if (p) cudaFree(p);
    if (hres) cudaFreeHost(hres);
    if (own) cudaStreamDestroy(own);
    if (cur != device) cudaSetDevice(cur);
  }
};

namespace gd {
namespace {

constexpr int GM = 64, GN = 64, GK = 16;
constexpr int KPART = 256;  // loss partial sums

__device__ __forceinline__ float tofloat(float x) { return x; }
__device__ __forceinline__ float tofloat(__nv_bfloat16 x) { return __bfloat162float(x); }

// GELU with the exact normal CDF, and its derivative
__device__ __forceinline__ float gelu(float z) { return 0.5f * z * (1.f + erff(z * 0.70710678118654752f)); }
__device__ __forceinline__ float gelu_d(float z) {
  return 0.5f * (1.f + erff(z * 0.70710678118654752f)) + z * 0.39894228040143268f * expf(-0.5f * z * z);
}

// C(m, n) = sum_k A(m, k) B(k, n) with A(m, k) = A[m sam + k sak], B(k, n) =
// B[k sbk + n sbn]; epi(m, n, c) takes each output
template <typename TA, typename TB, typename Epi>
__global__ void __launch_bounds__(256) k_gemm(int M, int N, int K, int kchunk, const TA* __restrict__ A, long sam,
                                              long sak, const TB* __restrict__ B, long sbk, long sbn, Epi epi) {
  __shared__ float As[GK][GM + 4];
  __shared__ float Bs[GK][GN + 4];
  const int tid = threadIdx.x;
  const int m0 = blockIdx.y * GM, n0 = blockIdx.x * GN;
  const int tm = (tid >> 4) * 4, tn = (tid & 15) * 4;
  float acc[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  const bool a_kfast = sak == 1, b_nfast = sbn == 1;
  // split K: this CTA sums k in [kb, ke) (blockIdx.z-th chunk)
  const int kb = blockIdx.z * kchunk, ke = min(K, kb + kchunk);
  for (int k0 = kb; k0 < ke; k0 += GK) {
    for (int e = tid; e < GM * GK; e += 256) {  // the unit-stride index fastest over the threads
      const int mm = a_kfast ? e / GK : e % GM, kk = a_kfast ? e % GK : e / GM;
      const int m = m0 + mm, k = k0 + kk;
      As[kk][mm] = (m < M && k < ke) ? tofloat(A[(long)m * sam + (long)k * sak]) : 0.f;
    }
    for (int e = tid; e < GK * GN; e += 256) {
      const int nn = b_nfast ? e % GN : e / GK, kk = b_nfast ? e / GN : e % GK;
      const int n = n0 + nn, k = k0 + kk;
      Bs[kk][nn] = (n < N && k < ke) ? tofloat(B[(long)k * sbk + (long)n * sbn]) : 0.f;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < GK; ++kk) {
      float a[4], b[4];
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        a[i] = As[kk][tm + i];
        b[i] = Bs[kk][tn + i];
      }
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int m = m0 + tm + i, n = n0 + tn + j;
      if (m < M && n < N) epi(m + blockIdx.z * M, n, acc[i][j]);  // split K: partial z at rows zM..
    }
}

struct EpiHidden {  // Z = acc + b, A = GELU(Z)
  const float* b;
  float* Z;
  float* Aout;
  int N;
  __device__ void operator()(int m, int n, float c) const {
    const float z = c + b[n];
    Z[(long)m * N + n] = z;
    Aout[(long)m * N + n] = gelu(z);
  }
};
struct EpiLinear {  // Y = acc + b
  const float* b;
  float* Y;
  int N;
  __device__ void operator()(int m, int n, float c) const { Y[(long)m * N + n] = c + b[n]; }
};
struct EpiStore {  // G = acc
  float* G;
  int N;
  __device__ void operator()(int m, int n, float c) const { G[(long)m * N + n] = c; }
};
struct EpiGeluD {  // dZ = acc * GELU'(Z)
  const float* Z;
  float* G;
  int N;
  __device__ void operator()(int m, int n, float c) const {
    const long i = (long)m * N + n;
    G[i] = c * gelu_d(Z[i]);
  }
};

template <typename TA, typename TB, typename Epi>
void gemm(int M, int N, int K, const TA* A, long sam, long sak, const TB* B, long sbk, long sbn, Epi epi,
          cudaStream_t s) {
  if (M <= 0 || N <= 0) return;
  dim3 grid((unsigned)ceil_div(N, GN), (unsigned)ceil_div(M, GM));
  k_gemm<TA, TB, Epi><<<grid, 256, 0, s>>>(M, N, K, K, A, sam, sak, B, sbk, sbn, epi);
  count_launch();
  GD_LAUNCH_CHECK();
}
// C = A B with K split into nsplit chunks: partial z goes to part[z][M][N],
// then the partials are summed in order (deterministic) into out [M][N]
constexpr int KSPLIT = 16;
__global__ void k_sum_parts(const float* __restrict__ part, int nsplit, long count, float* __restrict__ out) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < count; i += (long)gridDim.x * blockDim.x) {
    float t = 0.f;
    for (int z = 0; z < nsplit; ++z) t += part[z * count + i];
    out[i] = t;
  }
}
template <typename TA, typename TB>
void gemm_splitk(int M, int N, int K, const TA* A, long sam, long sak, const TB* B, long sbk, long sbn, float* part,
                 float* out, cudaStream_t s) {
  if (M <= 0 || N <= 0) return;
  const int nsplit = std::max(1, std::min(KSPLIT, K / 256));
  const int kchunk = (ceil_div(K, nsplit) + GK - 1) / GK * GK;
  const int ns = ceil_div(K, kchunk);
  dim3 grid((unsigned)ceil_div(N, GN), (unsigned)ceil_div(M, GM), (unsigned)ns);
  k_gemm<TA, TB, EpiStore><<<grid, 256, 0, s>>>(M, N, K, kchunk, A, sam, sak, B, sbk, sbn, EpiStore{part, N});
  const long cnt = (long)M * N;
  k_sum_parts<<<std::min(ceil_div(cnt, 256), 1024), 256, 0, s>>>(part, ns, cnt, out);
  count_launch(2);
  GD_LAUNCH_CHECK();
}

// db[n] = sum_m G[m][n] (fixed order: 8 strided partial sums, then a tree)
__global__ void k_colsum(const float* __restrict__ G, int M, int N, float* db) {
  __shared__ float red[8][33];
  const int n = blockIdx.x * 32 + threadIdx.x;
  float s = 0.f;
  if (n < N)
    for (int m = threadIdx.y; m < M; m += 8) s += G[(long)m * N + n];
  red[threadIdx.y][threadIdx.x] = s;
  __syncthreads();
  if (threadIdx.y == 0 && n < N) {
    float t = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) t += red[y][threadIdx.x];
    db[n] = t;
  }
}

// squared error: gy = 2 (y - t) / count, partial[block] = sum (y - t)^2
__global__ void k_mse(const float* __restrict__ y, const float* __restrict__ t, long count, float* gy,
                      float* partial) {
  __shared__ float red[256];
  float s = 0.f;
  const float sc = 2.f / (float)count;
  for (long i = (long)blockIdx.x * 256 + threadIdx.x; i < count; i += (long)gridDim.x * 256) {
    const float d = y[i] - t[i];
    s += d * d;
    if (gy) gy[i] = sc * d;
  }
  red[threadIdx.x] = s;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) partial[blockIdx.x] = red[0];
}
__global__ void k_mse_final(const float* partial, int n, long count, float* loss) {
  __shared__ float red[KPART];
  red[threadIdx.x] = threadIdx.x < n ? partial[threadIdx.x] : 0.f;
  __syncthreads();
  for (int o = KPART / 2; o > 0; o >>= 1) {
    if (threadIdx.x < o) red[threadIdx.x] += red[threadIdx.x + o];
    __syncthreads();
  }
  if (threadIdx.x == 0) *loss = red[0] / (float)count;
}

__global__ void k_adam(float* p, const float* g, float* m, float* v, __nv_bfloat16* w16, long n, float lr, float b1,
                       float b2, float eps, float c1, float c2) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x) {
    const float gi = g[i];
    const float mi = b1 * m[i] + (1.f - b1) * gi, vi = b2 * v[i] + (1.f - b2) * gi * gi;
    m[i] = mi;
    v[i] = vi;
    const float pi = p[i] - lr * (mi / c1) / (sqrtf(vi / c2) + eps);
    p[i] = pi;
    w16[i] = __float2bfloat16_rn(pi);
  }
}
__global__ void k_to_bf16(const float* p, __nv_bfloat16* w16, long n) {
  for (long i = (long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long)gridDim.x * blockDim.x)
    w16[i] = __float2bfloat16_rn(p[i]);
}

// packed weight rows: row r < rowsf of the forward pack, then the backward
// pack's, zero past the row's entries; one CTA per row
__global__ void k_pack(const __nv_bfloat16* __restrict__ w, const PackRow* __restrict__ rows, long rowsf, int kpf,
                       int kpb, __nv_bfloat16* __restrict__ wpf, __nv_bfloat16* __restrict__ wpb) {
  const long r = blockIdx.x;
  const PackRow pr = rows[r];
  const int kp = r < rowsf ? kpf : kpb;
  __nv_bfloat16* o = r < rowsf ? wpf + r * kpf : wpb + (r - rowsf) * kpb;
  for (int k = threadIdx.x; k < kp; k += blockDim.x)
    o[k] = k < pr.cnt ? w[pr.off + (long)k * pr.stride] : __float2bfloat16_rn(0.f);
}
// Operands of the weight gradients, every layer in one launch (blockIdx.z the
// job): rows r0 + [0, nbc) of src [n][w] (rows past n read as zero) transposed
// and split to TF32 hi + lo, dh / dl [c][r], row pitch kp, the batch
// contiguous.  A CTA takes kTrows rows x 32 columns; for a dZ job it also adds
// up its rows for the bias gradient (fixed order: eight strided sums, then
// those in order), one partial per CTA.
__global__ void __launch_bounds__(256) k_tsplit(const TsplitJob* __restrict__ jobs, const float* __restrict__ x,
                                                long r0, int n, int nbc, int kp, float* __restrict__ bpart, int nbias) {
  __shared__ float t[32][33];
  const TsplitJob j = jobs[blockIdx.z];
  const int c0 = blockIdx.y * 32, w = j.w;
  if (c0 >= w) return;
  const float* __restrict__ src = (j.src ? j.src : x) + r0 * w;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  float s = 0.f;
  for (int b = 0; b < kTrows && blockIdx.x * kTrows + b < nbc; b += 32) {
    const int rb = blockIdx.x * kTrows + b;
#pragma unroll
    for (int i = ty; i < 32; i += 8) {
      const int r = rb + i, c = c0 + tx;
      const float v = (r < n && c < w) ? src[(long)r * w + c] : 0.f;
      t[i][tx] = v;
      s += v;
    }
    __syncthreads();
#pragma unroll
    for (int i = ty; i < 32; i += 8) {
      const int c = c0 + i, r = rb + tx;
      if (c < w && r < nbc) {
        const float v = t[tx][i];
        const uint32_t h = (__float_as_uint(v) + 0x1000u) & 0xFFFFE000u;  // nearest TF32, ties away
        j.dh[(long)c * kp + r] = h;
        j.dl[(long)c * kp + r] = __float_as_uint(v - __uint_as_float(h));
      }
    }
    __syncthreads();
  }
  if (j.boff < 0) return;  // uniform over the CTA
  t[ty][tx] = s;
  __syncthreads();
  if (ty == 0 && c0 + tx < w) {
    float v = 0.f;
#pragma unroll
    for (int y = 0; y < 8; ++y) v += t[y][tx];
    bpart[(r0 / kTrows + blockIdx.x) * nbias + j.boff + c0 + tx] = v;
  }
}
// the packed gradient: weights from the slices' partial tiles, biases from
// their partial sums, each added in order
__global__ void k_wsum(const WgradLayer* __restrict__ lay, int nlayer, long np, const float* __restrict__ part,
                       long pstride, int nsplit, const float* __restrict__ bpart, int nbias, int nblk,
                       float* __restrict__ grad) {
  for (long e = (long)blockIdx.x * blockDim.x + threadIdx.x; e < np; e += (long)gridDim.x * blockDim.x) {
    int l = 0;
    while (l + 1 < nlayer && e >= lay[l + 1].offw) ++l;
    const WgradLayer L = lay[l];
    float s = 0.f;
    if (e < L.offb) {
      const int m = (int)((e - L.offw) / L.fi), c = (int)((e - L.offw) % L.fi);
      const float* p = part + L.poff + (long)m * L.Np + c;
#pragma unroll 4
      for (int q = 0; q < nsplit; ++q) s += p[q * pstride];
    } else {
      const float* p = bpart + L.boff + (e - L.offb);
#pragma unroll 4
      for (int q = 0; q < nblk; ++q) s += p[(long)q * nbias];
    }
    grad[e] = s;
  }
}

template <typename F>
int mguard(gd_mlp* p, F f) {
  if (!p) return GD_ERR_ARG;
  try {
    int cur = 0;
    GD_CUDA(cudaGetDevice(&cur));
    if (cur != p->device) GD_CUDA(cudaSetDevice(p->device));
    f();
    if (cur != p->device) GD_CUDA(cudaSetDevice(cur));
    return GD_OK;
  } catch (const CudaError& e) {
    p->err = e.what();
    return GD_ERR_CUDA;
  } catch (const std::invalid_argument& e) {
    p->err = e.what();
    return GD_ERR_ARG;
  } catch (const std::exception& e) {
    p->err = e.what();
    return GD_ERR_CUDA;
  }
}
std::string g_mlp_init_error;

// x, t and y of the batch entry points must be device memory of the net's
// device (a host pointer would fault the kernels)
void need_device(const gd_mlp* p, const void* ptr, const char* what) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, ptr) != cudaSuccess) {
    cudaGetLastError();
    throw std::invalid_argument(std::string("gd_mlp: ") + what + " is not a device pointer");
  }
  if ((a.type != cudaMemoryTypeDevice && a.type != cudaMemoryTypeManaged) || a.device != p->device)
    throw std::invalid_argument(std::string("gd_mlp: ") + what + " is not device memory of the net's device");
}

void to_bf16(gd_mlp* p) {
  k_to_bf16<<<std::min(ceil_div(p->np, 256), 4096), 256, 0, p->stream>>>(p->p32, p->w16, p->np);
  count_launch();
  GD_LAUNCH_CHECK();
}
// after every change of the BF16 weights, on the stream that changed them
void pack_weights(gd_mlp* p) {
  if (!p->tc) return;
  k_pack<<<(unsigned)(p->rowsf + p->rowsb), 64, 0, p->stream>>>(p->w16, p->pack, p->rowsf, p->kpf, p->kpb, p->wpf,
                                                               p->wpb);
  count_launch();
  GD_LAUNCH_CHECK();
}

}  // namespace

// --------------------------------------------------- shared with the dycore
// Buffers of a forward pass over ncols columns: none on the tensor cores
// (activations stay on chip), the activations on the SIMT path.  Old buffers
// are kept until the net is destroyed: a context's captured step may still
// address them.
struct Acts {
  int cap;
  float *zb, *ab;
};
Acts act_buffers(gd_mlp* p, int ncols) {
  if (ncols <= p->bcap) return Acts{p->bcap, p->zb, p->ab};
  GD_CUDA(cudaStreamSynchronize(p->stream));
  const size_t bytes = sizeof(float) * (size_t)p->nl * ncols * p->nh;
  float* zb = (float*)p->alloc(bytes);
  return Acts{ncols, zb, (float*)p->alloc(bytes)};
}
void act_set(gd_mlp* p, const Acts& a) { p->bcap = a.cap, p->zb = a.zb, p->ab = a.ab; }
void mlp_reserve(gd_mlp* p, int ncols) {
  if (p->tc) return;
  gd_mlp::Growth g(p);
  act_set(p, act_buffers(p, ncols));
  g.kept = true;
}

namespace {
void forward_simt(gd_mlp* p, const float* x, int n, float* y, cudaStream_t s);
template <typename X>
X* to_device(gd_mlp* p, const std::vector<X>& h) {
  X* d = (X*)p->alloc(sizeof(X) * h.size());
  upload_on(d, h.data(), sizeof(X) * h.size(), p->stream);
  return d;
}
}  // namespace

// Training buffers for batches of up to ncols columns, and on the tensor
// cores the layer tables over them: all of them first, then the net takes them
// over together, since a batch within the capacity uses every one.
void train_reserve(gd_mlp* p, int ncols) {
  if (ncols <= p->tcap) return;
  if (p->tcb && p->nin > 256)
    throw std::invalid_argument("gd_mlp: training on the tensor cores takes at most 256 inputs");
  gd_mlp::Growth grown(p);
  const Acts a = act_buffers(p, ncols);
  GD_CUDA(cudaStreamSynchronize(p->stream));
  const int cap = a.cap;
  float* yb = (float*)p->alloc(sizeof(float) * (size_t)cap * p->nout);
  float* gy = (float*)p->alloc(sizeof(float) * (size_t)cap * p->nout);
  if (!p->tcb) {
    const long w = std::max(p->nh, std::max(p->nin, p->nout));
    float* g0 = (float*)p->alloc(sizeof(float) * (size_t)cap * w);
    float* g1 = (float*)p->alloc(sizeof(float) * (size_t)cap * w);
    act_set(p, a);
    p->yb = yb, p->gy = gy, p->g0 = g0, p->g1 = g1;
    p->tcap = cap;
    grown.kept = true;
    return;
  }
  const size_t act = (size_t)cap * p->nh;
  float* dzb = (float*)p->alloc(sizeof(float) * (size_t)p->nl * act);
  std::vector<TcChainLayer> f, b;
  for (int l = 0; l < p->nlayer; ++l) {
    TcChainLayer L{};
    L.N = p->fout[l], L.K = p->fin[l], L.wrow = p->wrowf[l], L.bias = p->p32 + p->offb[l];
    if (l < p->nl) L.act = 1, L.z = a.zb + l * act, L.out = a.ab + l * act, L.ldz = p->nh;
    f.push_back(L);
  }
  for (int l = p->nlayer - 1; l >= 1; --l) {  // dZ_{l-1} = (dZ_l W_l) GELU'(Z_{l-1})
    TcChainLayer L{};
    L.N = p->fin[l], L.K = p->fout[l], L.wrow = p->wrowb[l], L.act = 2;
    L.zin = a.zb + (l - 1) * act, L.out = dzb + (l - 1) * act, L.ldz = p->nh;
    b.push_back(L);
  }
  TcChainLayer* trn_layers = to_device(p, f);
  TcChainLayer* bwd_layers = to_device(p, b);
  // weight gradients: stacked transposed operands over a slab of the batch
  const int cols = std::max(p->opcols, std::min((cap + 31) / 32 * 32, kSlab));
  long ar = 0, br = 0, po = 0;
  int bo = 0;
  std::vector<TcWgradItem> items;
  std::vector<WgradLayer> lay;
  std::vector<long> arow, brow;
  for (int l = 0; l < p->nlayer; ++l) {
    const int Mp = (p->fout[l] + 127) / 128 * 128, Np = (p->fin[l] + 15) / 16 * 16;
    arow.push_back(ar), brow.push_back(br);
    for (int m = 0; m < Mp; m += 128) items.push_back({(int)ar + m, (int)br, Np, po + (long)m * Np});
    lay.push_back({p->offw[l], p->offb[l], po, p->fout[l], p->fin[l], Np, bo});
    ar += Mp, br += (p->fin[l] + 63) / 64 * 64, po += (long)Mp * Np, bo += p->fout[l];
  }
  uint32_t *zth = p->zth, *ztl = p->ztl, *ath = p->ath, *atl = p->atl;
  if (cols > p->opcols) {  // rows past a layer's outputs or inputs stay zero
    auto z = [&](size_t words) {
      uint32_t* q = (uint32_t*)p->alloc(sizeof(uint32_t) * words);
      GD_CUDA(cudaMemsetAsync(q, 0, sizeof(uint32_t) * words, p->stream));
      return q;
    };
    zth = z((size_t)ar * cols), ztl = z((size_t)ar * cols);
    ath = z((size_t)br * cols), atl = z((size_t)br * cols);
    GD_CUDA(cudaStreamSynchronize(p->stream));
  }
  std::vector<TsplitJob> jobs;
  for (int l = 0; l < p->nlayer; ++l) {
    const size_t za = (size_t)arow[l] * cols, ba = (size_t)brow[l] * cols;
    jobs.push_back({l == p->nlayer - 1 ? gy : dzb + l * act, p->fout[l], lay[l].boff, zth + za, ztl + za});
    jobs.push_back({l == 0 ? nullptr : a.ab + (l - 1) * act, p->fin[l], -1, ath + ba, atl + ba});
  }
  TsplitJob* djobs = to_device(p, jobs);
  WgradLayer* wlay = to_device(p, lay);
  TcWgrad wg;
  wg.items = to_device(p, items);
  wg.nitems = (int)items.size();
  wg.pstride = po;
  wg.err = p->terr;
  const int nslab = ceil_div(cap, kSlab);
  wg.part = (float*)p->alloc(sizeof(float) * (size_t)nslab * std::max(1, p->nsm / wg.nitems) * po);
  float* bpart = (float*)p->alloc(sizeof(float) * (size_t)ceil_div(cap, kTrows) * bo);
  tc_wgrad_maps(wg, zth, ztl, ath, atl, ar, br, cols);
  act_set(p, a);
  p->yb = yb, p->gy = gy, p->dzb = dzb;
  p->trn_layers = trn_layers, p->bwd_layers = bwd_layers;
  p->zth = zth, p->ztl = ztl, p->ath = ath, p->atl = atl, p->opcols = cols;
  p->jobs = djobs, p->wlay = wlay, p->nbias = bo;
  p->wg = wg, p->wpart = wg.part, p->bpart = bpart;
  p->tcap = cap;
  grown.kept = true;
}

// y [n][nout] = net(x [n][nin]) on stream s, on the tensor cores when the
// shape allows (every layer at most 256 wide).  No allocation.
void mlp_forward_on(gd_mlp* p, const float* x, int n, float* y, cudaStream_t s) {
  if (!p->tc && n > p->bcap) throw std::invalid_argument("gd_mlp: batch above the reserved capacity");
  if (n <= 0) return;
  if (p->tc)
    tc_chain(p->mapf, p->inf_layers, p->nlayer, x, p->nin, n, y, p->nout, p->terr, s);
  else
    forward_simt(p, x, n, y, s);
}

namespace {
// the SIMT forward; the hidden pre-activations and activations stay in the
// net's buffers for a backward pass
void forward_simt(gd_mlp* p, const float* x, int n, float* y, cudaStream_t s) {
  const float* in = x;
  for (int l = 0; l < p->nlayer; ++l) {
    const int fi = p->fin[l], fo = p->fout[l];
    const __nv_bfloat16* W = p->w16 + p->offw[l];
    const float* b = p->p32 + p->offb[l];
    if (l < p->nl) {
      float* Z = p->zb + (size_t)l * p->bcap * p->nh;
      float* A = p->ab + (size_t)l * p->bcap * p->nh;
      gemm(n, fo, fi, in, (long)fi, 1L, W, 1L, (long)fi, EpiHidden{b, Z, A, fo}, s);
      in = A;
    } else {
      gemm(n, fo, fi, in, (long)fi, 1L, W, 1L, (long)fi, EpiLinear{b, y, fo}, s);
    }
  }
}
}  // namespace

// a bounded wait of a tensor-core kernel gave up: clears the flag and raises it
[[noreturn]] static void mlp_timeout(gd_mlp* p, cudaStream_t s, int code) {
  GD_CUDA(cudaMemsetAsync(p->terr, 0, sizeof(int), s));
  GD_CUDA(cudaStreamSynchronize(s));
  throw CudaError("closure net: a tensor-core wait timed out (code " + std::to_string(code) + ")");
}
// the end of an entry point of the net itself: copies the error flag and the
// loss through page-locked memory, the gradient straight to the caller (a
// second host copy of 0.9 MB costs more than it saves), waits once, and
// raises a timeout
void mlp_results(gd_mlp* p, cudaStream_t s, float* loss, float* grad) {
  int* e = reinterpret_cast<int*>(p->hres);
  *e = 0;
  if (p->terr) GD_CUDA(cudaMemcpyAsync(e, p->terr, sizeof(int), cudaMemcpyDeviceToHost, s));
  if (loss) GD_CUDA(cudaMemcpyAsync(p->hres + 1, p->lossd, sizeof(float), cudaMemcpyDeviceToHost, s));
  if (grad) GD_CUDA(cudaMemcpyAsync(grad, p->grad, sizeof(float) * p->np, cudaMemcpyDeviceToHost, s));
  GD_CUDA(cudaStreamSynchronize(s));
  if (*e) mlp_timeout(p, s, *e);
  if (loss) *loss = p->hres[1];
}
// for a context the net is attached to: another thread may be using the net's
// own page-locked results
void mlp_check(gd_mlp* p, cudaStream_t s) {
  if (!p->terr) return;
  int e = 0;
  GD_CUDA(cudaMemcpyAsync(&e, p->terr, sizeof(int), cudaMemcpyDeviceToHost, s));
  GD_CUDA(cudaStreamSynchronize(s));
  if (e) mlp_timeout(p, s, e);
}

int mlp_nin(const gd_mlp* p) { return p->nin; }
int mlp_nout(const gd_mlp* p) { return p->nout; }
int mlp_device(const gd_mlp* p) { return p->device; }
bool mlp_norm(const gd_mlp* p, const float** in_mu, const float** in_sd, const float** out_mu,
              const float** out_sd) {
  *in_mu = p->in_mu;
  *in_sd = p->in_sd;
  *out_mu = p->out_mu;
  *out_sd = p->out_sd;
  return p->has_norm;
}

namespace {
// loss and gradient of a batch into p->grad; the loss lands in p->lossd
void loss_grad(gd_mlp* p, const float* x, const float* t, int n) {
  cudaStream_t s = p->stream;
  if (p->tcb)
    tc_chain(p->mapf, p->trn_layers, p->nlayer, x, p->nin, n, p->yb, p->nout, p->terr, s);
  else
    forward_simt(p, x, n, p->yb, s);
  const long cnt = (long)n * p->nout;
  const int nb = std::min(KPART, ceil_div(cnt, 256));
  k_mse<<<nb, 256, 0, s>>>(p->yb, t, cnt, p->gy, p->partial);
  k_mse_final<<<1, KPART, 0, s>>>(p->partial, nb, cnt, p->lossd);
  count_launch(2);
  GD_LAUNCH_CHECK();
  if (p->tcb) {
    // dZ of every hidden layer, then all weight gradients, slab by slab of
    // the batch: operands transposed and split (with the bias gradients'
    // partial sums), partial tiles of slices of at least four chunks, as many
    // as one wave of CTAs takes; last the sums over slices
    tc_chain(p->mapb, p->bwd_layers, p->nl, p->gy, p->nout, n, p->dzb, p->nh, p->terr, s);
    int wmax = 0, slices = 0;
    for (int l = 0; l < p->nlayer; ++l) wmax = std::max(wmax, std::max(p->fout[l], p->fin[l]));
    for (int r0 = 0; r0 < n; r0 += kSlab) {
      const int m = std::min(kSlab, n - r0), nbc = (m + 31) / 32 * 32, nk = nbc / 32;
      k_tsplit<<<dim3(ceil_div(nbc, kTrows), ceil_div(wmax, 32), 2 * p->nlayer), 256, 0, s>>>(
          p->jobs, x, (long)r0, m, nbc, p->opcols, p->bpart, p->nbias);
      count_launch();
      GD_LAUNCH_CHECK();
      int ns = std::max(1, std::min(nk / 4, std::max(1, p->nsm / p->wg.nitems)));
      const int cps = (nk + ns - 1) / ns;
      ns = (nk + cps - 1) / cps;  // every slice non-empty
      tc_wgrad(p->wg, nk, cps, ns, slices, s);
      slices += ns;
    }
    k_wsum<<<std::min(ceil_div(p->np, 256), 1024), 256, 0, s>>>(p->wlay, p->nlayer, p->np, p->wpart, p->wg.pstride,
                                                               slices, p->bpart, p->nbias, ceil_div(n, kTrows),
                                                               p->grad);
    count_launch();
    GD_LAUNCH_CHECK();
    return;
  }
  // backward: dZ of layer l in cur; dW_l = dZ^T A_{l-1}, db_l = colsum dZ,
  // dZ_{l-1} = (dZ W_l) * GELU'(Z_{l-1})
  const float* cur = p->gy;
  for (int l = p->nlayer - 1; l >= 0; --l) {
    const int fi = p->fin[l], fo = p->fout[l];
    const float* Ain = l == 0 ? x : p->ab + (size_t)(l - 1) * p->bcap * p->nh;
    gemm_splitk(fo, fi, n, cur, 1L, (long)fo, Ain, (long)fi, 1L, p->kpart, p->grad + p->offw[l], s);
    k_colsum<<<ceil_div(fo, 32), dim3(32, 8), 0, s>>>(cur, n, fo, p->grad + p->offb[l]);
    count_launch();
    GD_LAUNCH_CHECK();
    if (l > 0) {
      float* nxt = (cur == p->g0) ? p->g1 : p->g0;
      const float* Zp = p->zb + (size_t)(l - 1) * p->bcap * p->nh;
      gemm(n, fi, fo, cur, (long)fo, 1L, p->w16 + p->offw[l], (long)fi, 1L, EpiGeluD{Zp, nxt, fi}, s);
      cur = nxt;
    }
  }
}
}  // namespace

}  // namespace gd

using namespace gd;

extern "C" {

int gd_mlp_init(int nin, int nhidden, int nlayers, int nout, unsigned long long seed, int device, gd_mlp** out) {
  if (!out) return GD_ERR_ARG;
  *out = nullptr;
  if (nin < 1 || nhidden < 1 || nlayers < 1 || nout < 1) {
    g_mlp_init_error = "gd_mlp_init: need nin, nhidden, nlayers, nout >= 1";
    return GD_ERR_ARG;
  }
  std::unique_ptr<gd_mlp> p(new gd_mlp());
  p->device = device;
  p->nin = nin;
  p->nh = nhidden;
  p->nl = nlayers;
  p->nout = nout;
  p->nlayer = nlayers + 1;
  long off = 0;
  for (int l = 0; l < p->nlayer; ++l) {
    const int fi = l == 0 ? nin : nhidden, fo = l == nlayers ? nout : nhidden;
    p->fin.push_back(fi);
    p->fout.push_back(fo);
    p->offw.push_back(off);
    off += (long)fi * fo;
    p->offb.push_back(off);
    off += fo;
  }
  p->np = off;
  // tensor cores when every layer is at most 256 wide (training too: the
  // backward products' outputs are the hidden widths); GD_MLP_TRAIN_TC=0
  // keeps training on the SIMT kernels (a comparison knob)
  p->tc = nhidden <= 256 && nout <= 256;
  {
    const char* e = getenv("GD_MLP_TRAIN_TC");
    p->tcb = p->tc && !(e && e[0] == '0');
  }
  std::vector<PackRow> pack;
  auto block = [&](std::vector<int>& first, long& rows, int n, long off0, long offn, int stride, int cnt) {
    first.push_back((int)rows);
    for (int i = 0; i < (n + 63) / 64 * 64; ++i, ++rows)
      pack.push_back(i < n ? PackRow{off0 + i * offn, stride, cnt} : PackRow{0, 0, 0});
  };
  for (int l = 0; l < p->nlayer; ++l) {
    p->kpf = std::max(p->kpf, (p->fin[l] + 63) / 64 * 64);
    block(p->wrowf, p->rowsf, p->fout[l], p->offw[l], p->fin[l], 1, p->fin[l]);
  }
  p->kpb = 64;
  for (int l = 0; l < p->nlayer; ++l) {
    p->kpb = std::max(p->kpb, (p->fout[l] + 63) / 64 * 64);
    if (l == 0 || !p->tcb)
      p->wrowb.push_back(0);
    else
      block(p->wrowb, p->rowsb, p->fin[l], p->offw[l], 1, p->fin[l], p->fout[l]);
  }
  // He-normal hidden weights, the output layer scaled by 0.1 (the net starts
  // close to no correction), zero biases
  std::vector<float> h(off, 0.f);
  std::mt19937_64 rng(seed);
  std::normal_distribution<double> nd(0.0, 1.0);
  for (int l = 0; l < p->nlayer; ++l) {
    const double sd = std::sqrt(2.0 / p->fin[l]) * (l == nlayers ? 0.1 : 1.0);
    for (long i = 0; i < (long)p->fin[l] * p->fout[l]; ++i) h[p->offw[l] + i] = (float)(sd * nd(rng));
  }
  const int rc = mguard(p.get(), [&] {
    GD_CUDA(cudaStreamCreateWithFlags(&p->own, cudaStreamNonBlocking));
    p->stream = p->own;
    GD_CUDA(cudaMallocHost(&p->hres, sizeof(float) * 2));
    long wmax = 0;
    for (int l = 0; l < p->nlayer; ++l) wmax = std::max(wmax, (long)p->fin[l] * p->fout[l]);
    // one allocation: the sizes first, then the addresses
    char* base = nullptr;
    size_t used = 0;
    auto take = [&](auto** q, size_t n) {
      *q = reinterpret_cast<std::remove_reference_t<decltype(*q)>>(base ? base + used : nullptr);
      used += (n * sizeof(**q) + 255) / 256 * 256;
    };
    auto carve = [&]() {
      for (float** q : {&p->p32, &p->grad, &p->am, &p->av}) take(q, off);
      take(&p->w16, off);
      take(&p->partial, KPART);
      if (!p->tcb) take(&p->kpart, KSPLIT * wmax);  // SIMT training
      take(&p->lossd, 1);
      for (float** q : {&p->in_mu, &p->in_sd}) take(q, nin);
      for (float** q : {&p->out_mu, &p->out_sd}) take(q, nout);
      if (!p->tc) return;
      take(&p->wpf, (size_t)p->rowsf * p->kpf);
      if (p->rowsb > 0) take(&p->wpb, (size_t)p->rowsb * p->kpb);
      take(&p->terr, 1);
    };
    carve();
    base = (char*)p->alloc(used);
    used = 0;
    carve();
    if (p->tc) {
      tc_chain_map(&p->mapf, p->wpf, p->kpf, p->rowsf);
      if (p->rowsb > 0) tc_chain_map(&p->mapb, p->wpb, p->kpb, p->rowsb);
      p->pack = to_device(p.get(), pack);
      std::vector<TcChainLayer> inf;
      for (int l = 0; l < p->nlayer; ++l) {
        TcChainLayer L{};
        L.N = p->fout[l], L.K = p->fin[l], L.wrow = p->wrowf[l], L.act = l < p->nl ? 1 : 0;
        L.bias = p->p32 + p->offb[l];
        inf.push_back(L);
      }
      p->inf_layers = to_device(p.get(), inf);
      GD_CUDA(cudaMemsetAsync(p->terr, 0, sizeof(int), p->stream));
      GD_CUDA(cudaDeviceGetAttribute(&p->nsm, cudaDevAttrMultiProcessorCount, p->device));
    }
    upload_on(p->p32, h.data(), sizeof(float) * off, p->stream);
    for (float* q : {p->am, p->av, p->grad}) GD_CUDA(cudaMemsetAsync(q, 0, sizeof(float) * off, p->stream));
    to_bf16(p.get());
    pack_weights(p.get());
    GD_CUDA(cudaStreamSynchronize(p->stream));
  });
  if (rc != GD_OK) {
    g_mlp_init_error = p->err;
    return rc;
  }
  *out = p.release();
  return GD_OK;
}

int gd_mlp_destroy(gd_mlp* p) {
  if (!p) return GD_ERR_ARG;
  delete p;
  return GD_OK;
}

int gd_mlp_nparams(gd_mlp* p, long long* n) {
  if (!p || !n) return GD_ERR_ARG;
  *n = p->np;
  return GD_OK;
}

int gd_mlp_get_params(gd_mlp* p, float* params) {
  if (!params) return GD_ERR_ARG;
  return mguard(p, [&] {
    GD_CUDA(cudaStreamSynchronize(p->stream));
    GD_CUDA(cudaMemcpy(params, p->p32, sizeof(float) * p->np, cudaMemcpyDeviceToHost));
  });
}

int gd_mlp_set_params(gd_mlp* p, const float* params) {
  if (!params) return GD_ERR_ARG;
  return mguard(p, [&] {
    GD_CUDA(cudaStreamSynchronize(p->stream));
    upload_on(p->p32, params, sizeof(float) * p->np, p->stream);
    to_bf16(p);
    pack_weights(p);
    GD_CUDA(cudaStreamSynchronize(p->stream));
  });
}

int gd_mlp_set_norm(gd_mlp* p, const float* in_mu, const float* in_sd, const float* out_mu, const float* out_sd) {
  if (!in_mu || !in_sd || !out_mu || !out_sd) return GD_ERR_ARG;
  return mguard(p, [&] {
    for (int i = 0; i < p->nin; ++i)
      if (!(in_sd[i] > 0)) throw std::invalid_argument("gd_mlp_set_norm: input scales must be > 0");
    GD_CUDA(cudaStreamSynchronize(p->stream));
    upload_on(p->in_mu, in_mu, sizeof(float) * p->nin, p->stream);
    upload_on(p->in_sd, in_sd, sizeof(float) * p->nin, p->stream);
    upload_on(p->out_mu, out_mu, sizeof(float) * p->nout, p->stream);
    upload_on(p->out_sd, out_sd, sizeof(float) * p->nout, p->stream);
    p->has_norm = true;
  });
}

int gd_mlp_forward(gd_mlp* p, const float* x, int ncols, float* y) {
  if (!x || !y || ncols < 0) return GD_ERR_ARG;
  return mguard(p, [&] {
    if (ncols == 0) return;
    need_device(p, x, "x");
    need_device(p, y, "y");
    mlp_reserve(p, ncols);
    mlp_forward_on(p, x, ncols, y, p->stream);
    mlp_results(p, p->stream, nullptr, nullptr);
  });
}

int gd_mlp_loss_grad(gd_mlp* p, const float* x, const float* t, int ncols, float* loss, float* grad) {
  if (!x || !t || ncols < 1) return GD_ERR_ARG;
  return mguard(p, [&] {
    need_device(p, x, "x");
    need_device(p, t, "t");
    train_reserve(p, ncols);
    loss_grad(p, x, t, ncols);
    mlp_results(p, p->stream, loss, grad);
  });
}

int gd_mlp_train_step(gd_mlp* p, const float* x, const float* t, int ncols, float lr, float* loss) {
  if (!x || !t || ncols < 1 || !(lr > 0)) return GD_ERR_ARG;
  return mguard(p, [&] {
    need_device(p, x, "x");
    need_device(p, t, "t");
    train_reserve(p, ncols);
    loss_grad(p, x, t, ncols);
    ++p->adam_t;
    const float b1 = 0.9f, b2 = 0.999f;
    const float c1 = 1.f - std::pow(b1, (float)p->adam_t), c2 = 1.f - std::pow(b2, (float)p->adam_t);
    k_adam<<<std::min(ceil_div(p->np, 256), 4096), 256, 0, p->stream>>>(p->p32, p->grad, p->am, p->av, p->w16, p->np,
                                                                         lr, b1, b2, 1e-8f, c1, c2);
    count_launch();
    GD_LAUNCH_CHECK();
    pack_weights(p);
    if (loss) mlp_results(p, p->stream, loss, nullptr);  // waits; raises a tensor-core wait that gave up
  });
}

int gd_mlp_set_stream(gd_mlp* p, void* stream) {
  return mguard(p, [&] {
    GD_CUDA(cudaStreamSynchronize(p->stream));
    p->stream = stream ? (cudaStream_t)stream : p->own;
  });
}

int gd_mlp_sync(gd_mlp* p) {
  return mguard(p, [&] { mlp_results(p, p->stream, nullptr, nullptr); });
}

const char* gd_mlp_last_error(gd_mlp* p) { return p ? p->err.c_str() : g_mlp_init_error.c_str(); }

}  // extern "C"

// ------------------------------------------------------ closure columns --
namespace gd {
namespace {
constexpr int CT = 32;  // grid columns per CTA of the transposes
}

// rows of gS (column index fastest) -> x [column][feature] through a shared
// tile: the reads and the writes both run along contiguous memory
template <typename R>
__global__ void k_closure_in(const R* __restrict__ gS, SynthRows s, int L, long ng, const float* __restrict__ mu,
                             const float* __restrict__ sd, float* __restrict__ x) {
  extern __shared__ float tile[];  // [nf][CT + 1]
  const int nf = 3 * L + 1;
  const long p0 = (long)blockIdx.x * CT;
  for (int e = threadIdx.x; e < nf * CT; e += blockDim.x) {
    const int f = e / CT, c = e % CT;
    const long p = p0 + c;
    float v = 0.f;
    if (p < ng) {
      if (f < L)
        v = (float)gS[(long)(s.u + f) * ng + p];
      else if (f < 2 * L)
        v = (float)gS[(long)(s.v + f - L) * ng + p];
      else if (f < 3 * L)
        v = (float)gS[(long)(s.tv + f - 2 * L) * ng + p];
      else
        v = (float)exp(gS[(long)s.lnps * ng + p]);
      if (mu) v = (v - mu[f]) / sd[f];
    }
    tile[f * (CT + 1) + c] = v;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < nf * CT; e += blockDim.x) {
    const int c = e / nf, f = e % nf;
    const long p = p0 + c;
    if (p < ng) x[p * nf + f] = tile[f * (CT + 1) + c];
  }
}

template <typename R>
__global__ void k_closure_out(const float* __restrict__ y, int L, long ng, const float* __restrict__ mu,
                              const float* __restrict__ sd, R dt, R* __restrict__ gA) {
  extern __shared__ float tile[];  // [3L][CT + 1]
  const int no = 3 * L;
  const long p0 = (long)blockIdx.x * CT;
  for (int e = threadIdx.x; e < no * CT; e += blockDim.x) {
    const int c = e / no, f = e % no;
    const long p = p0 + c;
    tile[f * (CT + 1) + c] = p < ng ? y[p * no + f] * sd[f] + mu[f] : 0.f;
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 4 * L * CT; e += blockDim.x) {
    const int r = e / CT, c = e % CT;
    const long p = p0 + c;
    if (p >= ng) continue;
    // grid row r: Tv [0,L) <- y[2L, 3L); q [L,2L) <- 0; u [2L,3L) <- y[0,L); v [3L,4L) <- y[L,2L)
    const int f = r < L ? 2 * L + r : r < 2 * L ? -1 : r - 2 * L;
    gA[(long)r * ng + p] = f < 0 ? R(0) : dt * (R)tile[f * (CT + 1) + c];
  }
}

template <typename R>
void launch_closure_in(const R* gS, const SynthRows& s, int L, long ng, const float* mu, const float* sd, float* x,
                       cudaStream_t st) {
  const size_t sm = sizeof(float) * (size_t)(3 * L + 1) * (CT + 1);
  if (sm > 48 * 1024) GD_CUDA(cudaFuncSetAttribute(k_closure_in<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  k_closure_in<R><<<ceil_div(ng, CT), 256, sm, st>>>(gS, s, L, ng, mu, sd, x);
  count_launch();
  GD_LAUNCH_CHECK();
}
template <typename R>
void launch_closure_out(const float* y, int L, long ng, const float* mu, const float* sd, R dt, R* gA,
                        cudaStream_t st) {
  const size_t sm = sizeof(float) * (size_t)(3 * L) * (CT + 1);
  if (sm > 48 * 1024)
    GD_CUDA(cudaFuncSetAttribute(k_closure_out<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm));
  k_closure_out<R><<<ceil_div(ng, CT), 256, sm, st>>>(y, L, ng, mu, sd, dt, gA);
  count_launch();
  GD_LAUNCH_CHECK();
}
template void launch_closure_in<double>(const double*, const SynthRows&, int, long, const float*, const float*,
                                        float*, cudaStream_t);
template void launch_closure_in<float>(const float*, const SynthRows&, int, long, const float*, const float*, float*,
                                       cudaStream_t);
template void launch_closure_out<double>(const float*, int, long, const float*, const float*, double, double*,
                                         cudaStream_t);
template void launch_closure_out<float>(const float*, int, long, const float*, const float*, float, float*,
                                        cudaStream_t);

}  // namespace gd
