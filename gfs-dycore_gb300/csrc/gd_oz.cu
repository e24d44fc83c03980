// gd_oz.cu -- the plain FP64 Legendre GEMMs on the sm_103a tensor cores.
//
// The FP64 pipe of this part does two multiply-adds per clock and SM, the BF16
// tensor pipe 4096: an FP64 product is cheaper as integer products of short
// slices (Ozaki, Ogita, Oishi and Rump 2012, error-free splitting of a matrix
// product).  Each operand row is scaled by a power of two to 62-bit integers
// q = sum_b d_b 256^b, b = 0..7, with balanced digits |d_b| <= 128, exact in
// BF16.  The products of digit pairs with b1 + b2 = g + 7 share accumulator g
// (0..7, 36 pairs).  What is dropped is at most 2^-57 of the product of the two
// rows' largest entries per term (every dropped digit -128 against row maxima of
// a power of two: 2^-57.2; digits of both signs, as operands have, 2^-60 and
// less), an FP64 rounding of it is 2^-53.  An accumulator sums at most 8
// x 128 products of at most 2^14 between drains, so every FP32 accumulation
// in tensor memory is an exact integer below 2^24, and the epilogue adds the
// eight of them as 64-bit integers and rounds once to FP64.
//
// Orientation as in gd_tc.cu: M = 128 batch columns on the TMEM lanes, N <= 32
// latitudes or degrees, K degrees or latitudes of one hemispheric parity.
// TMEM: two sets of 8 accumulators x 32 columns.  A work item (order, column
// tile, N tile) runs its parities, in K segments of 128, one after the other
// through the sets.  The synthesis forms E +- O as integers, before the one
// rounding; sums over several segments are added in FP64 at the outputs.
//
// A launch takes both tables' work (P and dP/dphi), after one split of their
// operand columns.
//
// One step of T126 with 64 levels and 3 tracers (1026 columns; 152 SMs): all its
// Legendre transforms 18.8 ms on the FP64 pipe (70% of its rate), 3.92 ms here.
// With 4 tracers (1154 columns) a synthesis through P reads 0.9 GB of operands from L2 and
// needs 0.13 ms for it, 0.11 ms of tensor-core issue and 0.13 ms of FP64
// additions; the three overlap in part (0.29 ms).  T42 with 20 levels: 0.57 -> 0.35 ms; with a launch
// per table 0.47 ms (and 4.35 ms at T126).
#include <algorithm>
#include <stdexcept>

#include "gd_oz.cuh"
#include "gd_ptx.cuh"
#include "gd_tc.cuh"

namespace gd {

namespace {
constexpr int OZ_S = 8;         // digits of an operand
constexpr int OZ_M = 128;       // batch columns per item
constexpr int OZ_N = 32;        // widest N tile: TMEM columns per accumulator
constexpr int OZ_NBUF = 2;      // sets of the eight accumulators in TMEM
constexpr int OZ_KC = 32;       // K per ring stage (64-byte rows, 64-byte swizzle)
constexpr int OZ_SEG = 128;     // K per drain: 8 x 128 x 2^14 = 2^24
constexpr int OZ_NS = 2;        // ring stages
constexpr int OZ_EPI = 16;      // epilogue warps
constexpr int OZ_THREADS = 64 + 32 * OZ_EPI;
constexpr int OZ_BAD = 1 << 20;  // exponent of a row with an infinity or NaN
constexpr uint32_t OZ_ABYTES = OZ_S * OZ_M * OZ_KC * 2;

int round_to(int x, int a) { return (x + a - 1) / a * a; }
// N tile of n latitudes or degrees: the multiple of 16 up to `widest` with the least
// padded work, a tile counted as 16 columns wider than it is (its fixed costs)
int oz_tile(int n, int widest) {
  int best = 16;
  for (int t = 32; t <= widest; t += 16)
    if (((n + t - 1) / t) * (t + 16) <= ((n + best - 1) / best) * (best + 16)) best = t;
  return best;
}

// ---------------------------------------------------------------- digits --
// biased exponent field of |x|; a NaN or infinity has 0x7ff
__device__ __forceinline__ int oz_field(double x) { return (__double2hiint(x) >> 20) & 0x7ff; }
// 62-bit integer q with x = q 2^(fm - 1084) up to 2^-62 of the row's largest
// entry, fm the row's largest exponent field (at least 1)
__device__ __forceinline__ long long oz_fixed(double x, int fm) {
  const long long b = __double_as_longlong(x);
  const int f = (int)((b >> 52) & 0x7ff), sh = fm - max(f, 1);
  if (sh > 61) return 0;
  const long long m = (long long)(((unsigned long long)((b & 0xfffffffffffffLL) | (f ? 1LL << 52 : 0)) << 9) >> sh);
  return b < 0 ? -m : m;
}
// The balanced digits of q: with 128 added at every digit but the top one, byte
// b of the sum is digit b + 128 (the carries are the balancing).  Digit b of
// q0 and of q1 in BF16, q1's in the high half; biased: q + OZ_BIAS.
constexpr long long OZ_BIAS = 0x0080808080808080LL;
__device__ __forceinline__ uint32_t oz_digits(long long t0, long long t1, int b) {
  float f0, f1;
  if (b == OZ_S - 1) {  // signed
    f0 = __int_as_float(0x4B400000 + (int)(t0 >> 56)) - 12582912.f;
    f1 = __int_as_float(0x4B400000 + (int)(t1 >> 56)) - 12582912.f;
  } else {
    const uint32_t w0 = b < 4 ? (uint32_t)t0 : (uint32_t)(t0 >> 32), w1 = b < 4 ? (uint32_t)t1 : (uint32_t)(t1 >> 32);
    f0 = __uint_as_float(__byte_perm(w0, 0x4B000000u, 0x7440 + (b & 3))) - 8388736.f;  // 2^23 + 128
    f1 = __uint_as_float(__byte_perm(w1, 0x4B000000u, 0x7440 + (b & 3))) - 8388736.f;
  }
  return __byte_perm(__float_as_uint(f0), __float_as_uint(f1), 0x7632);
}
__device__ __forceinline__ int oz_exponent(int fm) { return fm == 0x7ff ? OZ_BAD : fm - 1084; }

// tables, one warp per row of order m = blockIdx.y + 1.  Synthesis rows: the
// latitudes, K = the degrees (even ones, then odd ones); analysis rows: the
// degrees in that order, K = the latitudes.
__global__ void __launch_bounds__(256) k_oz_table(int mode, int T, int nh, int nhpad, const long* __restrict__ moff,
                                                  const long* __restrict__ xbase, long xlen,
                                                  const long* __restrict__ toff, const double* __restrict__ tab,
                                                  uint16_t* __restrict__ out, int* __restrict__ ex) {
  const int lane = threadIdx.x & 31, m = blockIdx.y + 1, K = T - m + 1, ke = (K + 1) / 2;
  const int rows = mode == 0 ? nh : K, kpad = mode == 0 ? (ke + 31) / 32 * 32 : nhpad;
  const long slice = mode == 0 ? nh * xlen : moff[T + 1] * nhpad;
  for (int r = blockIdx.x * 8 + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8) {
    const double* src = tab + toff[m] + (mode == 0 ? (long)r * K : r < ke ? 2 * r : 2 * (r - ke) + 1);
    const int n = mode == 0 ? K : nh;
    const long stride = mode == 0 ? 1 : K;
    int fm = 1;
    for (int k = lane; k < n; k += 32) fm = max(fm, oz_field(src[k * stride]));
    fm = __reduce_max_sync(0xffffffffu, fm);
    if (lane == 0) ex[mode == 0 ? (long)m * nh + r : moff[m] + r] = oz_exponent(fm);
    uint16_t* o = out + (mode == 0 ? r * xlen + xbase[m] : (moff[m] + r) * nhpad);
    for (int k = lane; k < (mode == 0 ? 2 * kpad : kpad); k += 32) {
      const int i = mode == 0 ? (k < kpad ? 2 * k : 2 * (k - kpad) + 1) : k;  // its entry
      const long long t = (i < n ? oz_fixed(src[i * stride], fm) : 0) + OZ_BIAS;
#pragma unroll
      for (int b = 0; b < OZ_S; ++b) o[b * slice + k] = (uint16_t)oz_digits(t, t, b);
    }
  }
}

// Operand columns to digits, K contiguous: one CTA per (order, 32 columns),
// lane = column, a thread takes adjacent K entries in pairs.  mode 0: the
// degrees of each parity of order m, rows of B; mode 1: the latitude pairs of
// G, north + south for the parity that pairs with the even degrees of P (north
// - south for dP/dphi), and the other.  The values of up to 128 K entries stay
// in registers between the search for the column's largest exponent and the
// digits, more are read again.  Bound by integer issue.
struct OzSplit {
  int T, nh, nlat, ncap, nhpad;
  const long* moff;
  const long* xbase;
  long xlen;
  // up to two sources side by side in the operand (blockIdx.z), from column coff
  const double* src[2];
  long ld[2];
  int ncols[2], coff[2], parityH[2];
  uint16_t* out[2];  // mode 0: X (both parities in one row); mode 1: G of each parity
  int* ex[2];        // [(T+1)][ncap]: mode 0 one for both parities, mode 1 per parity
};
template <int MODE>
__global__ void __launch_bounds__(256) k_oz_split(const __grid_constant__ OzSplit a) {
  __shared__ uint32_t t[OZ_S][32][33];
  __shared__ int red[2][8][32];
  constexpr int NU = 8;  // pairs per thread and register block of 128 K entries
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int z = blockIdx.z, ncols = a.ncols[z], parityH = a.parityH[z];
  const int m = blockIdx.x + 1, c0 = blockIdx.y * 32, c = c0 + lane;
  if (c0 >= ncols) return;  // the grid covers the wider source
  const long ld = a.ld[z], d0 = a.coff[z] + c0;  // first operand column of the CTA
  const int K = a.T - m + 1, ke = (K + 1) / 2, kp = MODE == 0 ? (ke + 31) / 32 * 32 : a.nhpad;
  const int n0 = MODE == 0 ? ke : a.nh, n1 = MODE == 0 ? K / 2 : a.nh;  // entries of each parity
  const bool live = c < ncols;
  const double* src = a.src[z] + (MODE == 0 ? a.moff[m] : (long)m * a.nlat) * ld + c;
  double v[2][NU][2];
  // entries k0 + 2 (w + 8 u) + {0, 1} of both parities
  auto load = [&](int k0) {
#pragma unroll
    for (int u = 0; u < NU; ++u)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        const int k = k0 + 2 * (w + 8 * u) + i;
        double x = 0.0, y = 0.0;
        if (MODE == 0) {
          if (live && k < n0) x = src[(long)(2 * k) * ld];
          if (live && k < n1) y = src[(long)(2 * k + 1) * ld];
        } else if (live && k < n0) {
          x = src[(long)k * ld];
          y = src[(long)(a.nlat - 1 - k) * ld];
        }
        v[0][u][i] = x;
        v[1][u][i] = y;
      }
    if (MODE == 1) {
#pragma unroll
      for (int u = 0; u < NU; ++u)
#pragma unroll
        for (int i = 0; i < 2; ++i) {
          const double p = v[0][u][i] + v[1][u][i], d = v[0][u][i] - v[1][u][i];
          v[0][u][i] = parityH ? d : p;
          v[1][u][i] = parityH ? p : d;
        }
    }
  };
  int fm[2] = {1, 1};
  for (int k0 = 0; k0 < n0; k0 += 128) {
    load(k0);
#pragma unroll
    for (int par = 0; par < 2; ++par)
#pragma unroll
      for (int u = 0; u < NU; ++u) fm[par] = max(fm[par], max(oz_field(v[par][u][0]), oz_field(v[par][u][1])));
  }
#pragma unroll
  for (int par = 0; par < 2; ++par) red[par][w][lane] = fm[par];
  __syncthreads();
#pragma unroll
  for (int par = 0; par < 2; ++par)
#pragma unroll
    for (int i = 0; i < 8; ++i) fm[par] = max(fm[par], red[par][i][lane]);
  if (MODE == 0) fm[0] = fm[1] = max(fm[0], fm[1]);
  if (w == 0 && live) {
    a.ex[0][(long)m * a.ncap + d0 + lane] = oz_exponent(fm[0]);
    if (MODE == 1) a.ex[1][(long)m * a.ncap + d0 + lane] = oz_exponent(fm[1]);
  }
  const long pitch = MODE == 0 ? a.xlen : a.nhpad;
  const long slice = MODE == 0 ? (long)a.ncap * a.xlen : (long)(a.T + 1) * a.ncap * a.nhpad;
  for (int k0 = 0; k0 < kp; k0 += 128) {
    if (n0 > 128) load(k0);
#pragma unroll
    for (int par = 0; par < 2; ++par) {
      uint16_t* out = MODE == 0 ? a.out[0] + a.xbase[m] + (long)par * kp + d0 * a.xlen
                                : a.out[par] + ((long)m * a.ncap + d0) * a.nhpad;
#pragma unroll
      for (int h = 0; h < 2; ++h) {  // 64 K entries through shared memory
        if (k0 + 64 * h >= kp) break;
#pragma unroll
        for (int u = 0; u < NU / 2; ++u) {
          const long long q0 = oz_fixed(v[par][4 * h + u][0], fm[par]) + OZ_BIAS,
                          q1 = oz_fixed(v[par][4 * h + u][1], fm[par]) + OZ_BIAS;
#pragma unroll
          for (int b = 0; b < OZ_S; ++b) t[b][lane][w + 8 * u] = oz_digits(q0, q1, b);
        }
        __syncthreads();
        if (k0 + 64 * h + 2 * lane < kp)
          for (int r = w; r < OZ_S * 32; r += 8) {
            const int b = r >> 5, cc = r & 31;
            if (c0 + cc < ncols)
              *reinterpret_cast<uint32_t*>(out + b * slice + cc * pitch + k0 + 64 * h + 2 * lane) = t[b][cc][lane];
          }
        __syncthreads();
      }
    }
  }
}

// -------------------------------------------------------------- the GEMM --
struct OzArgs {
  const int4* items;
  int nitems;
  int mode;  // 0 synthesis, 1 analysis
  int T, nh, nlat, N, ncap;
  const long* xbase;
  const long* moff;
  const int* ea[2];  // operand exponents [m][ncap] of each parity (synthesis: the same)
  // up to two tables' jobs on columns [coff, coff + ncols) of the operand
  struct Job {
    int parityH, ncols, coff;
    const int* eb;  // table exponents (synthesis [m nh + j], analysis [spectral row, even degrees first])
    double* out;
    long ldout;
  } job[2];
  int* err;
};
// A work item's passes, each through one set of accumulators: a K segment of 128
// of one parity; in the synthesis a segment's even degrees, then its odd ones (if
// it has any), in the analysis all segments of the even degrees, then the others'.
struct OzItem {
  int m, c0, n0, K, segs, passes, job;
  __device__ OzItem(const OzArgs& a, int idx) {
    const int4 it = a.items[idx];
    m = it.x;
    c0 = it.y * OZ_M;
    n0 = it.z * a.N;
    job = it.w;
    K = a.T - m + 1;
    segs = ((a.mode ? a.nh : degrees(0)) + OZ_SEG - 1) / OZ_SEG;
    passes = a.mode == 0 ? segs + (degrees(1) + OZ_SEG - 1) / OZ_SEG : ncount(a, 1) > 0 ? 2 * segs : segs;
  }
  __device__ int degrees(int par) const { return par ? K / 2 : (K + 1) / 2; }
  // valid N columns
  __device__ int ncount(const OzArgs& a, int par) const { return min(a.N, (a.mode ? degrees(par) : a.nh) - n0); }
};
struct OzPass {
  int par, k0, kn;  // first K entry, number of entries
  __device__ OzPass(const OzArgs& a, const OzItem& t, int p) {
    par = a.mode ? (p >= t.segs) : (p & 1);
    k0 = (a.mode ? p - par * t.segs : p >> 1) * OZ_SEG;
    kn = min(OZ_SEG, (a.mode ? a.nh : t.degrees(par)) - k0);
  }
};

__device__ __forceinline__ uint64_t oz_desc(uint32_t saddr) {  // K-major, 64-byte swizzle, 8-row groups of 512 bytes
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (uint64_t)1 << 16 | (uint64_t)(512 >> 4) << 32 | (uint64_t)1 << 46 |
         (uint64_t)4 << 61;
}
__device__ __forceinline__ void oz_mma(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, uint32_t acc) {
  asm volatile(
      "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(d),
      "l"(a), "l"(b), "r"(idesc), "r"(acc));
}
__device__ __forceinline__ void oz_ld4(uint32_t taddr, uint32_t* r) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(taddr));
}
// accumulators b..b+3 of one output as an integer (each below 2^24 in size)
template <int NC>
__device__ __forceinline__ long long oz_int(const uint32_t (&r)[OZ_S][NC], int b, int q) {
  long long v = __float2int_rn(__uint_as_float(r[b][q]));
#pragma unroll
  for (int g = 1; g < 4; ++g) v += (long long)__float2int_rn(__uint_as_float(r[b + g][q])) * (1 << (8 * g));
  return v;
}
__device__ __noinline__ double oz_scale(double v, int k) {
  return k >= OZ_BAD / 2 ? __longlong_as_double(0x7ff8000000000000LL) : scalbn(v, k);
}
// (hi 2^32 + lo) 2^k rounded once to FP64, |hi|, |lo| < 2^51.  The integers
// become FP64 numbers by their place in a mantissa (1.5 2^52 + lo, and the same
// 32 binary digits higher), the scale goes into these numbers' exponents, and
// two additions remain for the slow FP64 pipe, the first of them exact.
__device__ __forceinline__ double oz_join(long long hi, long long lo, int k) {
  const bool plain = k >= -900 && k <= 900;  // else scaled afterwards
  const int kk = plain ? k << 20 : 0;
  const double xl = __hiloint2double((int)(lo >> 32) + (0x43380000 + kk), (int)lo);
  const double xh = __hiloint2double((int)(hi >> 32) + (0x45380000 + kk), (int)hi);
  double v = (xh - __hiloint2double(0x45380000 + kk, 0x00180000)) + xl;
  if (!plain && ((hi | lo) != 0 || k >= OZ_BAD / 2)) v = oz_scale(v, k);  // a zero column's k is out of range too
  return v;
}

__global__ void __launch_bounds__(OZ_THREADS, 1)
    k_oz_gemm(const __grid_constant__ CUtensorMap mA0, const __grid_constant__ CUtensorMap mA1,
              const __grid_constant__ CUtensorMap mB0, const __grid_constant__ CUtensorMap mB1,
              const __grid_constant__ OzArgs a) {
  extern __shared__ __align__(1024) unsigned char smraw[];
  unsigned char* sm = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smraw) + 1023) & ~(uintptr_t)1023);
  const uint32_t bbytes = (uint32_t)(OZ_S * a.N * OZ_KC * 2), stage = OZ_ABYTES + bbytes;
  uint64_t* full = reinterpret_cast<uint64_t*>(sm + OZ_NS * stage);
  uint64_t* empty = full + OZ_NS;
  uint64_t* tfull = empty + OZ_NS;     // a pass's accumulators are complete
  uint64_t* tempty = tfull + OZ_NBUF;  // and drained
  uint64_t* done = tempty + OZ_NBUF;
  uint32_t* tslot = reinterpret_cast<uint32_t*>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tslot)), "r"(512u));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  if (tid == 0) {
    for (int s = 0; s < OZ_NS; ++s) {
      mbar_init(smem_u32(&full[s]), 1);
      mbar_init(smem_u32(&empty[s]), 1);
    }
    for (int s = 0; s < OZ_NBUF; ++s) {
      mbar_init(smem_u32(&tfull[s]), 1);
      mbar_init(smem_u32(&tempty[s]), OZ_EPI);
    }
    mbar_init(smem_u32(done), 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tbase = *tslot;

  if (tid == 0) {  // ------------------------------------------- producer
    int fills[OZ_NS] = {};
    long g = 0;
    TcRing rs;
    bool bad = false;
    for (int idx = blockIdx.x; idx < a.nitems && !bad; idx += gridDim.x) {
      const OzItem t(a, idx);
      const int kpx = (t.degrees(0) + 31) / 32 * 32, row = a.job[t.job].coff + t.c0;
      for (int p = 0; p < t.passes && !bad; ++p) {
        const OzPass ps(a, t, p);
        for (int k = ps.k0; k < ps.k0 + ps.kn; k += OZ_KC, ++g) {
          const int s = rs.slot;
          if (g >= OZ_NS && !mbar_wait(smem_u32(&empty[s]), rs.ph ^ 1u, a.err, 51)) {
            bad = true;
            break;
          }
          const uint32_t st = smem_u32(sm + s * stage), fb = smem_u32(&full[s]);
          mbar_expect_tx(fb, stage);
          if (a.mode == 0) {
            const int x = (int)a.xbase[t.m] + ps.par * kpx + k;
            tma_3d(st, &mA0, x, row, 0, fb);
            if (t.job)
              tma_3d(st + OZ_ABYTES, &mB1, x, t.n0, 0, fb);
            else
              tma_3d(st + OZ_ABYTES, &mB0, x, t.n0, 0, fb);
          } else {
            if (ps.par)
              tma_3d(st, &mA1, k, t.m * a.ncap + row, 0, fb);
            else
              tma_3d(st, &mA0, k, t.m * a.ncap + row, 0, fb);
            const int y = (int)a.moff[t.m] + ps.par * t.degrees(0) + t.n0;
            if (t.job)
              tma_3d(st + OZ_ABYTES, &mB1, k, y, 0, fb);
            else
              tma_3d(st + OZ_ABYTES, &mB0, k, y, 0, fb);
          }
          ++fills[s];
          rs.next(OZ_NS);
        }
      }
    }
    for (int s = 0; s < OZ_NS; ++s)  // no copies left in flight at exit
      if (fills[s] > 0) mbar_wait(smem_u32(&full[s]), (fills[s] - 1) & 1, a.err, 52);
  } else if (tid == 32) {  // ------------------------------------ MMA issuer
    TcRing rs, tb;  // stages, accumulator buffers
    uint32_t pass = 0;
    bool bad = false;
    for (int idx = blockIdx.x; idx < a.nitems && !bad; idx += gridDim.x) {
      const OzItem t(a, idx);
      for (int p = 0; p < t.passes && !bad; ++p, ++pass, tb.next(OZ_NBUF)) {
        const OzPass ps(a, t, p);
        if (pass >= OZ_NBUF && !mbar_wait(smem_u32(&tempty[tb.slot]), tb.ph ^ 1u, a.err, 53)) {
          bad = true;
          break;
        }
        tc_fence_after();
        const int nn = (t.ncount(a, ps.par) + 15) & ~15;
        const uint32_t idesc =
            (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(nn >> 3) << 17) | ((uint32_t)(OZ_M >> 4) << 24);
        const uint32_t acc = tbase + tb.slot * OZ_S * OZ_N;
        for (int k = 0; k < ps.kn; k += OZ_KC) {
          const int s = rs.slot;
          if (!mbar_wait(smem_u32(&full[s]), rs.ph, a.err, 54)) {
            bad = true;
            break;
          }
          tc_fence_after();
          const uint32_t st = smem_u32(sm + s * stage);
          const uint64_t da = oz_desc(st), db = oz_desc(st + OZ_ABYTES);
          const uint64_t sa = (OZ_M * OZ_KC * 2) >> 4, sb = (uint64_t)(a.N * OZ_KC * 2) >> 4;
          for (int h = 0; h < 2 && k + 16 * h < ps.kn; ++h) {  // K = 16: 32 bytes
            const uint64_t ah = da + 2 * h, bh = db + 2 * h;
#pragma unroll
            for (int d = 0; d < OZ_S; ++d)  // neighbours in time go to different accumulators
#pragma unroll
              for (int g = 0; g + d < OZ_S; ++g)
                oz_mma(acc + (uint32_t)(g * OZ_N), ah + (g + d) * sa, bh + (7 - d) * sb, idesc,
                       (k > 0 || h > 0 || d > 0) ? 1u : 0u);
          }
          mma_commit(smem_u32(&empty[s]));
          rs.next(OZ_NS);
        }
        if (!bad) mma_commit(smem_u32(&tfull[tb.slot]));
      }
    }
    mma_commit(smem_u32(done));
  } else if (warp >= 2) {  // ------------------------------------- epilogue
    const int q4 = warp & 3, grp = (warp - 2) >> 2;
    TcRing tb;
    // waits for a pass; its accumulators' address for this warp
    auto begin = [&](uint32_t* lw) {
      const bool ok = mbar_wait(smem_u32(&tfull[tb.slot]), tb.ph, a.err, 55);
      if (!__all_sync(0xffffffffu, ok)) return false;
      tc_fence_after();
      *lw = tbase + ((uint32_t)(q4 * 32) << 16) + tb.slot * OZ_S * OZ_N;
      return true;
    };
    // the set of accumulators is free
    auto release = [&]() {
      tc_fence_before();
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&tempty[tb.slot]));
      tb.next(OZ_NBUF);
    };
    auto load4 = [&](uint32_t lw, int n, uint32_t (&r)[OZ_S][4]) {
#pragma unroll
      for (int g = 0; g < OZ_S; ++g) oz_ld4(lw + (uint32_t)(g * OZ_N + n), r[g]);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    };
    bool bad = false;
    uint32_t lw = 0;
    for (int idx = blockIdx.x; idx < a.nitems && !bad; idx += gridDim.x) {
      const OzItem t(a, idx);
      const OzArgs::Job& job = a.job[t.job];
      const int c = t.c0 + q4 * 32 + lane;
      const bool live = c < job.ncols;
      const long ldout = job.ldout;
      if (a.mode == 0) {
        // north E + O, south E - O (dP/dphi: O - E), a quarter of the latitudes
        // per warp; E waits in registers as integers, so that the next item's
        // even degrees are multiplied while this one's sums are formed and stored
        const int ng = grp * (a.N / 4), nv = t.ncount(a, 0);
        const int ea = live ? a.ea[0][(long)t.m * a.ncap + job.coff + c] + 56 : 0;
        const int* eb = job.eb + (long)t.m * a.nh + t.n0;
        const int flip = job.parityH ? (int)0x80000000 : 0;
        double* north = job.out + ((long)t.m * a.nlat + t.n0) * ldout + c;
        double* south = job.out + ((long)t.m * a.nlat + (a.nlat - 1 - t.n0)) * ldout + c;
        for (int k0 = 0, p = 0; p < t.passes; k0 += OZ_SEG, p += 2) {
          const bool odd = k0 < t.degrees(1), more = k0 > 0;
          if (!begin(&lw)) {
            bad = true;
            break;
          }
          long long eh[OZ_N / 4], el[OZ_N / 4];
#pragma unroll
          for (int i = 0; i < OZ_N / 4; i += 4)
            if (i < a.N / 4) {
              uint32_t r[OZ_S][4];
              load4(lw, ng + i, r);
#pragma unroll
              for (int q = 0; q < 4; ++q) eh[i + q] = oz_int(r, 4, q), el[i + q] = oz_int(r, 0, q);
            }
          release();
          if (odd && !begin(&lw)) {
            bad = true;
            break;
          }
#pragma unroll
          for (int i = 0; i < OZ_N / 4; i += 4)
            if (i < a.N / 4) {
              uint32_t r[OZ_S][4];
              if (odd) {
                load4(lw, ng + i, r);
              } else {
#pragma unroll
                for (int g = 0; g < OZ_S; ++g) r[g][0] = r[g][1] = r[g][2] = r[g][3] = 0u;
              }
#pragma unroll
              for (int q = 0; q < 4; ++q) {
                const int n = ng + i + q;
                if (live && n < nv) {
                  const int k = ea + __ldg(eb + n);
                  const long long oh = oz_int(r, 4, q), ol = oz_int(r, 0, q);
                  double vn = oz_join(eh[i + q] + oh, el[i + q] + ol, k);
                  double vs = oz_join(eh[i + q] - oh, el[i + q] - ol, k);
                  vs = __hiloint2double(__double2hiint(vs) ^ flip, __double2loint(vs));
                  double* const on = north + n * ldout;
                  double* const os = south - n * ldout;
                  if (more) vn += *on, vs += *os;
                  *on = vn;
                  *os = vs;
                }
              }
              __syncwarp();
            }
          if (odd) release();
        }
      } else {  // four degrees a time
        for (int p = 0; p < t.passes; ++p) {
          const OzPass ps(a, t, p);
          const int nv = t.ncount(a, ps.par);
          const int ea = live ? (ps.par ? a.ea[1] : a.ea[0])[(long)t.m * a.ncap + job.coff + c] + 56 : 0;
          const bool more = ps.k0 > 0;
          const int* eb = job.eb + a.moff[t.m] + ps.par * t.degrees(0) + t.n0;
          double* out = job.out + (a.moff[t.m] + 2 * t.n0 + ps.par) * ldout + c;
          if (!begin(&lw)) {
            bad = true;
            break;
          }
          for (int n4 = grp * 4; n4 < nv; n4 += OZ_EPI) {
            uint32_t r[OZ_S][4];
            load4(lw, n4, r);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
              if (live && n4 + q < nv) {
                double v = oz_join(oz_int(r, 4, q), oz_int(r, 0, q), ea + __ldg(eb + n4 + q));
                double* const o = out + 2 * (n4 + q) * ldout;
                if (more) v += *o;
                *o = v;
              }
            }
            __syncwarp();
          }
          release();
        }
      }
    }
  }
  __syncwarp();
  mbar_wait(smem_u32(done), 0, a.err, 56);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tbase), "r"(512u));
}

// ------------------------------------------------------------ host side --
// [8][rows][k] BF16 slices, boxes of 32 k x boxrows x 8
void oz_map(CUtensorMap* m, void* base, long k, long rows, int boxrows) {
  cuuint64_t gd[3] = {(cuuint64_t)k, (cuuint64_t)rows, OZ_S}, gs[2] = {(cuuint64_t)k * 2, (cuuint64_t)k * rows * 2};
  cuuint32_t bx[3] = {OZ_KC, (cuuint32_t)boxrows, OZ_S}, es[3] = {1, 1, 1};
  const CUresult r = tensor_map_encoder()(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, base, gd, gs, bx, es,
                                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_64B,
                                          CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) throw CudaError("cuTensorMapEncodeTiled (digits) failed: " + std::to_string((int)r));
}
const int4* oz_items(OzPlan& p, const OzLeg* legs, int nlegs, int mode, int* n, cudaStream_t s) {
  int ct[2] = {0, 0};
  for (int i = 0; i < nlegs; ++i) ct[i] = (legs[i].ncols + OZ_M - 1) / OZ_M;
  for (const auto& l : p.items)
    if (l.ct[0] == ct[0] && l.ct[1] == ct[1] && l.mode == mode) {
      *n = l.n;
      return l.d;
    }
  std::vector<int4> it;
  for (int m = 1; m <= p.T; ++m) {
    const int nn = mode == 0 ? p.nh : (p.T - m + 2) / 2, N = mode == 0 ? p.nsyn : p.nana;
    for (int i = 0; i < nlegs; ++i)
      for (int c = 0; c < ct[i]; ++c)
        for (int b = 0; b * N < nn; ++b) it.push_back(make_int4(m, c, b, i));
  }
  OzPlan::Items l{{ct[0], ct[1]}, mode, (int)it.size(), nullptr};
  GD_CUDA(cudaMalloc(&l.d, sizeof(int4) * it.size()));
  upload_on(l.d, it.data(), sizeof(int4) * it.size(), s);
  p.items.push_back(l);
  *n = l.n;
  return l.d;
}
// the operand's columns of the legs, from `src` if given (analyses: the legs side by side)
OzSplit oz_split_args(const OzPlan& p, const long* d_moff, const OzLeg* legs, int nlegs, int* widest) {
  OzSplit a{};
  a.T = p.T, a.nh = p.nh, a.nlat = p.nlat, a.ncap = p.ncap, a.nhpad = p.nhpad;
  a.moff = d_moff, a.xbase = p.d_xbase, a.xlen = p.xlen;
  *widest = 0;
  int at = 0;
  for (int i = 0; i < nlegs; ++i) {
    a.src[i] = legs[i].in, a.ld[i] = legs[i].ldin, a.ncols[i] = legs[i].ncols, a.coff[i] = at;
    a.parityH[i] = legs[i].useH ? 1 : 0;
    at += legs[i].ncols;
    *widest = std::max(*widest, legs[i].ncols);
  }
  if (at > p.ncap) throw std::runtime_error("FP64 tensor-core Legendre path: too many columns");
  return a;
}
void oz_gemm(OzPlan& p, const long* d_moff, int mode, const OzLeg* legs, const int* coff, int nlegs, cudaStream_t s) {
  OzArgs a{};
  a.mode = mode, a.T = p.T, a.nh = p.nh, a.nlat = p.nlat, a.ncap = p.ncap, a.N = mode ? p.nana : p.nsyn;
  a.xbase = p.d_xbase, a.moff = d_moff, a.err = p.err;
  for (int t = 0; t < 2; ++t) a.ea[t] = mode ? p.eg[t] : p.ex;
  const CUtensorMap* mb[2];
  for (int i = 0; i < 2; ++i) {
    const OzLeg& l = legs[i < nlegs ? i : 0];
    const int t = l.useH ? 1 : 0, at = coff[i < nlegs ? i : 0];
    if (at < 0 || at + l.ncols > p.ncap) throw std::runtime_error("FP64 tensor-core Legendre path: too many columns");
    a.job[i] = {t, l.ncols, at, mode ? p.eana[t] : p.esyn[t], l.out, l.ldout};
    mb[i] = mode ? &p.m_tana[t] : &p.m_tsyn[t];
  }
  a.items = oz_items(p, legs, nlegs, mode, &a.nitems, s);
  const size_t sm = (size_t)OZ_NS * (OZ_ABYTES + (size_t)OZ_S * a.N * OZ_KC * 2) + 1024 + 128;
  k_oz_gemm<<<std::min(a.nitems, p.nsm), OZ_THREADS, sm, s>>>(mode ? p.m_g[0] : p.m_x, mode ? p.m_g[1] : p.m_x, *mb[0],
                                                             *mb[1], a);
  count_launch();
  GD_LAUNCH_CHECK();
}
}  // namespace

bool oz_init(OzPlan& p, int T, int nh, int nlat, int ncap, size_t limit, const long* d_moff, const long* d_toff,
             const double* P, const double* H, cudaStream_t s) {
  if (T < 1) return false;  // no order m >= 1
  int dev = 0;
  GD_CUDA(cudaGetDevice(&dev));
  GD_CUDA(cudaDeviceGetAttribute(&p.nsm, cudaDevAttrMultiProcessorCount, dev));
  p.T = T;
  p.nh = nh;
  p.nlat = nlat;
  p.nlm = (long)(T + 1) * (T + 2) / 2;
  p.nhpad = round_to(nh, OZ_KC);
  p.ncap = round_to(ncap, OZ_M);
  // narrow tiles where wide ones leave SMs without a second item (T42 step 0.960 -> 0.934 ms)
  const int widest = (long)T * (p.ncap / OZ_M) * ((nh + OZ_N - 1) / OZ_N) < 2 * p.nsm ? 16 : OZ_N;
  p.nsyn = oz_tile(nh, widest);
  p.nana = oz_tile((T + 1) / 2, widest);
  std::vector<long> xb(T + 1);
  for (int m = 1; m <= T; ++m) {
    xb[m] = p.xlen;
    p.xlen += 2L * round_to((T - m + 2) / 2, OZ_KC);
  }
  // one allocation: offsets first
  size_t bytes = 0;
  auto part = [&](size_t n) {
    const size_t at = bytes;
    bytes += (n + 255) / 256 * 256;
    return at;
  };
  const long rsyn = (long)(T + 1) * nh, rg = (long)(T + 1) * p.ncap;
  const size_t dig = 2 * OZ_S;  // bytes of an operand's digits
  // a synthesis and an analysis of a context never overlap (one stream), and
  // each writes its operand's digits before it reads them: one place for both
  const size_t gbytes = (dig * rg * p.nhpad + 255) / 256 * 256;
  const size_t ox = part(std::max(dig * p.ncap * p.xlen, 2 * gbytes)), oex = part(sizeof(int) * rg), oxb = part(sizeof(long) * (T + 1));
  size_t ots[2], ota[2], oes[2], oea[2], oeg[2];
  for (int t = 0; t < 2; ++t) {
    ots[t] = part(dig * nh * p.xlen);
    ota[t] = part(dig * p.nlm * p.nhpad);
    oes[t] = part(sizeof(int) * rsyn);
    oea[t] = part(sizeof(int) * p.nlm);
    oeg[t] = part(sizeof(int) * rg);
  }
  if (bytes > limit) return false;
  void* mem = nullptr;
  const cudaError_t e = cudaMalloc(&mem, bytes);
  if (e == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return false;
  }
  GD_CUDA(e);
  p.mem = mem;
  auto at = [&](size_t o) { return (void*)((char*)mem + o); };
  p.x = at(ox);
  p.ex = (int*)at(oex);
  p.d_xbase = (long*)at(oxb);
  GD_CUDA(cudaFuncSetAttribute(k_oz_gemm, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024));
  GD_CUDA(cudaMemcpyAsync(p.d_xbase, xb.data(), sizeof(long) * (T + 1), cudaMemcpyHostToDevice, s));
  oz_map(&p.m_x, p.x, p.xlen, p.ncap, OZ_M);
  for (int t = 0; t < 2; ++t) {
    const double* tab = t ? H : P;
    p.tsyn[t] = at(ots[t]);
    p.tana[t] = at(ota[t]);
    p.g[t] = at(ox + t * gbytes);
    p.esyn[t] = (int*)at(oes[t]);
    p.eana[t] = (int*)at(oea[t]);
    p.eg[t] = (int*)at(oeg[t]);
    for (int mode = 0; mode < 2; ++mode) {
      k_oz_table<<<dim3(mode == 0 ? (nh + 7) / 8 : (T + 7) / 8, T), 256, 0, s>>>(
          mode, T, nh, p.nhpad, d_moff, p.d_xbase, p.xlen, d_toff, tab, (uint16_t*)(mode == 0 ? p.tsyn[t] : p.tana[t]),
          mode == 0 ? p.esyn[t] : p.eana[t]);
      count_launch();
      GD_LAUNCH_CHECK();
    }
    oz_map(&p.m_tsyn[t], p.tsyn[t], p.xlen, nh, p.nsyn);
    oz_map(&p.m_tana[t], p.tana[t], p.nhpad, p.nlm, p.nana);
    oz_map(&p.m_g[t], p.g[t], p.nhpad, rg, OZ_M);
  }
  GD_CUDA(cudaStreamSynchronize(s));  // xb
  return true;
}

void oz_free(OzPlan& p) {
  for (auto& l : p.items) cudaFree(l.d);
  p.items.clear();
  if (p.mem) cudaFree(p.mem);
  p.mem = nullptr;
}

void oz_synth(OzPlan& p, const long* d_moff, const OzLeg& a, const OzLeg* b, cudaStream_t s) {
  if (a.ncols <= 0) return;
  // both tables read the same columns: one split serves them
  const long off = b ? b->in - a.in : 0;
  if (b && (b->ldin != a.ldin || off < 0 || off + b->ncols > a.ncols))
    throw std::runtime_error("FP64 tensor-core Legendre path: legs of different arrays");
  int n = 0;
  OzSplit sp = oz_split_args(p, d_moff, &a, 1, &n);
  sp.out[0] = (uint16_t*)p.x;
  sp.ex[0] = p.ex;
  k_oz_split<0><<<dim3(p.T, (n + 31) / 32), 256, 0, s>>>(sp);
  count_launch();
  GD_LAUNCH_CHECK();
  const OzLeg legs[2] = {a, b ? *b : a};
  const int coff[2] = {0, (int)off};
  oz_gemm(p, d_moff, 0, legs, coff, b && b->ncols > 0 ? 2 : 1, s);
}

void oz_anal(OzPlan& p, const long* d_moff, const OzLeg& a, const OzLeg* b, cudaStream_t s) {
  if (b && b->ncols <= 0) b = nullptr;
  if (a.ncols <= 0) return;
  const OzLeg legs[2] = {a, b ? *b : a};
  const int nl = b ? 2 : 1;
  int n = 0;
  OzSplit sp = oz_split_args(p, d_moff, legs, nl, &n);
  for (int t = 0; t < 2; ++t) sp.out[t] = (uint16_t*)p.g[t], sp.ex[t] = p.eg[t];
  k_oz_split<1><<<dim3(p.T, (n + 31) / 32, nl), 256, 0, s>>>(sp);
  count_launch();
  GD_LAUNCH_CHECK();
  const int coff[2] = {0, a.ncols};
  oz_gemm(p, d_moff, 1, legs, coff, nl, s);
}

}  // namespace gd
