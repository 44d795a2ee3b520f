// smoothn for the two displacement fields of each pair, as PIVGPU uses it
// (SmoothnGPU(f_shape, mask, s)(u, v), gpu_smoothn.py:123-231: non-robust,
// order 2, equal weights): z = IDCT2(gamma * DCT2(f)), gamma = 1/(1 + s lambda^2),
// lambda = 2 (2 - cos(pi i/m) - cos(pi j/n)) (gpu_smoothn.py:340-351), one s
// shared by u and v. With s unset, p = log10(s) minimises the GCV score
// (gpu_smoothn.py:353-372) over [p_min, p_max] (gpu_smoothn.py:320-338): a
// 10-point scan (gpu_smoothn.py:182-188) followed by a bounded local search
// from the best scan point that keeps the scan point when its projected
// finite-difference gradient is below 1e-5 (the stopping test of the
// reference's L-BFGS-B call, gpu_smoothn.py:191-193).
//
// The orthonormal DCT-II/III pairs are matrix products with cosine matrices
// built on the device. The GCV search and the weighted iteration of one pair
// run on one CTA or, when the pairs leave SMs idle, on a cluster of up to
// eight (cluster_size): float64 has 1/64 of the float32 rate here, so a
// search on one SM is bound by that SM's float64 pipe. The sums are formed by
// kVT virtual threads in the same order whatever the cluster size, so the
// results do not depend on it, bit for bit.
#include <math.h>

#include <algorithm>
#include <mutex>

#include "piv_common.cuh"
#include "piv_internal.h"
#include "piv_lbfgsb1.cuh"

namespace piv {

// Constant tables of an m x n field.
struct SmoothTables {
  double* cm;    // [m][m] DCT-II matrix (lines too long for the staged kernels)
  double* cn;    // [n][n]
  float* cmf;    // [2][m][m] cm as hi/lo floats
  float* cnf;    // [2][n][n]
  float2* cm2;   // weighted path: [m][m] cm as (hi, lo)
  float2* cn2;   // [n][n]
  float2* cnt2;  // [n][n] the transpose of cn2
  double* lam2;  // [mn] lambda^2
  float* lam2f;  // [mn] lambda^2 in float32 (the GCV scan's fast score)
};

struct SmoothScratch {
  double* fd;    // [pairs][2][mn] DCT coefficients of u and v
  double* tmp;   // [pairs][2][mn]
  double* f2;    // [pairs][mn] fd_u^2 + fd_v^2
  double* s;     // [pairs] 10^p
  float* f2f;    // [pairs][mn] f2 in float32 (the GCV search's fast score)
  SmoothTables t;
};

// A square field has one cosine matrix.
static void share_square(int m, int n, SmoothTables& t) {
  if (m != n) return;
  t.cn = t.cm;
  t.cnf = t.cmf;
  t.cn2 = t.cm2;
}

static size_t align_up(size_t v) { return (v + 255) / 256 * 256; }

// Per-pair block of the weighted path: f, z, z', fd, tmp (2 mn doubles each),
// w (mn doubles), the column-nearest table (mn ints) and 2 mn spare floats.
static size_t weighted_pair_bytes(size_t mn) { return align_up(11 * mn * 8 + mn * 4 + 2 * mn * 4); }
// The DCT matrices of the weighted path as hi/lo float pairs (2 (m^2 + n^2) floats).
static size_t weighted_matrix_bytes(int m, int n) { return align_up(2 * ((size_t)m * m + (size_t)n * n) * 4); }

// Scratch of the unweighted path (no field mask) and of the weighted path.
static size_t smoothn_scratch_bytes_path(int m, int n, int n_pairs, bool weighted_path) {
  const size_t mn = (size_t)m * n;
  const size_t shared = align_up((size_t)m * m * 8) + align_up((size_t)n * n * 8) + align_up(mn * 8) +
                        align_up((size_t)n_pairs * 8);
  if (weighted_path) return shared + weighted_matrix_bytes(m, n) + weighted_pair_bytes(mn) * n_pairs;
  return align_up(2 * mn * n_pairs * 8) * 2 + align_up(mn * n_pairs * 8) + shared + align_up(mn * n_pairs * 4) +
         align_up(mn * 4) + align_up((size_t)m * m * 8) + align_up((size_t)n * n * 8);
}

size_t smoothn_scratch_bytes(int m, int n, int n_pairs) {
  const size_t plain = smoothn_scratch_bytes_path(m, n, n_pairs, false);
  const size_t weighted = smoothn_scratch_bytes_path(m, n, n_pairs, true);
  return plain > weighted ? plain : weighted;
}

static SmoothScratch carve(void* base, int m, int n, int n_pairs) {
  const size_t mn = (size_t)m * n;
  char* p = (char*)base;
  SmoothScratch s;
  s.fd = (double*)p; p += align_up(2 * mn * n_pairs * 8);
  s.tmp = (double*)p; p += align_up(2 * mn * n_pairs * 8);
  s.f2 = (double*)p; p += align_up(mn * n_pairs * 8);
  s.t.cm = (double*)p; p += align_up((size_t)m * m * 8);
  s.t.cn = (double*)p; p += align_up((size_t)n * n * 8);
  s.t.lam2 = (double*)p; p += align_up(mn * 8);
  s.s = (double*)p; p += align_up((size_t)n_pairs * 8);
  s.f2f = (float*)p; p += align_up(mn * n_pairs * 4);
  s.t.lam2f = (float*)p; p += align_up(mn * 4);
  s.t.cmf = (float*)p; p += align_up((size_t)m * m * 8);
  s.t.cnf = (float*)p;
  s.t.cm2 = s.t.cn2 = s.t.cnt2 = nullptr;
  share_square(m, n, s.t);
  return s;
}

// The constant tables: the orthonormal DCT-II matrices C[k][i] = s_k cos(pi
// (2i+1) k / (2 len)), one thread per entry, and lambda^2 with lambda = 2 (2 -
// (cos(pi i/m) + cos(pi j/n))), kLamRows rows per CTA; NULL tables are left
// out. sc: s_0 and s_k of the two lengths. One launch where five small ones
// (two matrices, their splits, lambda^2) took 32 us for 253 x 253, this takes
// 11 us; bound by the float64 cosines.
static constexpr int kTabThreads = 128, kLamRows = 16;
struct TableScale {
  double m0, mk, n0, nk;
};
__global__ void __launch_bounds__(kTabThreads) k_smooth_tables(int m, int n, SmoothTables t, TableScale sc,
                                                               int mat_blocks, int lam_cols) {
  __shared__ double row_cos[kLamRows];
  if ((int)blockIdx.x < mat_blocks) {
    const long long id = (long long)blockIdx.x * kTabThreads + threadIdx.x;
    const long long mm = (long long)m * m, nn = (long long)n * n;
    const bool same = t.cn == t.cm && t.cnf == t.cmf && t.cn2 == t.cm2;  // one matrix for a square field
    if (id >= mm + (same ? 0 : nn)) return;
    const bool rows = id >= mm;  // the matrix of the transform along the rows
    const int len = rows ? n : m;
    const long long e = rows ? id - mm : id;
    const int k = (int)(e / len), i = (int)(e % len);
    const double sk = k == 0 ? (rows ? sc.n0 : sc.m0) : (rows ? sc.nk : sc.mk);
    const double c = sk * cospi((double)((2 * i + 1) * k) / (2.0 * len));
    double* cd = rows ? t.cn : t.cm;
    float* cf = rows ? t.cnf : t.cmf;
    float2* c2 = rows ? t.cn2 : t.cm2;
    const long long ll = rows ? nn : mm;
    const float h = (float)c, l = (float)(c - (double)h);
    if (cd) cd[e] = c;
    if (cf) {
      cf[e] = h;
      cf[ll + e] = l;
    }
    if (c2) c2[e] = make_float2(h, l);
    if ((rows || same) && t.cnt2) t.cnt2[(long long)i * n + k] = make_float2(h, l);
    return;
  }
  const int q = blockIdx.x - mat_blocks, i0 = (q / lam_cols) * kLamRows;
  const int j = (q % lam_cols) * kTabThreads + threadIdx.x;
  if (threadIdx.x < kLamRows) row_cos[threadIdx.x] = cos(M_PI * (i0 + (int)threadIdx.x) / m);
  const double col_cos = cos(M_PI * j / n);
  __syncthreads();
  if (j >= n) return;
  for (int i = i0; i < min(i0 + kLamRows, m); ++i) {
    const double l = 2.0 * (2.0 - (row_cos[i - i0] + col_cos));
    t.lam2[(long long)i * n + j] = l * l;
    if (t.lam2f) t.lam2f[(long long)i * n + j] = (float)(l * l);
  }
}

static int check(const char* what) {
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, what);
}

#define PIV_RC(expr)               \
  do {                             \
    const int rc_ = (expr);        \
    if (rc_ != PIV_OK) return rc_; \
  } while (0)

static int build_tables(int m, int n, const SmoothTables& t, cudaStream_t stream) {
  const TableScale sc{sqrt(1.0 / m), sqrt(2.0 / m), sqrt(1.0 / n), sqrt(2.0 / n)};
  const long long entries = (long long)m * m + (long long)n * n;
  const long long mat = (entries + kTabThreads - 1) / kTabThreads;
  const long long lam_cols = (n + kTabThreads - 1) / kTabThreads, lam_rows = (m + kLamRows - 1) / kLamRows;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(mat + lam_cols * lam_rows));
  cfg.blockDim = dim3(kTabThreads);
  cfg.stream = stream;
  // The launch's own status: an error that the caller has left behind is not the tables'.
  const cudaError_t e = cudaLaunchKernelEx(&cfg, k_smooth_tables, m, n, t, sc, (int)mat, (int)lam_cols);
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_smooth_tables");
}

// Tables that a plan keeps (every table, whichever path its runs take).
size_t smooth_tables_bytes(int m, int n) {
  const size_t mm = (size_t)m * m * 8, nn = (size_t)n * n * 8, mn = (size_t)m * n;
  return 3 * align_up(mm) + 4 * align_up(nn) + align_up(mn * 8) + align_up(mn * 4);
}

static SmoothTables kept_tables(const void* base, int m, int n) {
  const size_t mm = (size_t)m * m * 8, nn = (size_t)n * n * 8, mn = (size_t)m * n;
  char* p = (char*)const_cast<void*>(base);
  SmoothTables t;
  t.cm = (double*)p; p += align_up(mm);
  t.cn = (double*)p; p += align_up(nn);
  t.cmf = (float*)p; p += align_up(mm);
  t.cnf = (float*)p; p += align_up(nn);
  t.cm2 = (float2*)p; p += align_up(mm);
  t.cn2 = (float2*)p; p += align_up(nn);
  t.cnt2 = (float2*)p; p += align_up(nn);
  t.lam2 = (double*)p; p += align_up(mn * 8);
  t.lam2f = (float*)p;
  share_square(m, n, t);
  return t;
}

int smooth_tables_build(int m, int n, void* base, cudaStream_t stream) {
  return build_tables(m, n, kept_tables(base, m, n), stream);
}

// ---------------------------------------------------------------------------
// Clusters of CTAs that share one pair's sums.
// ---------------------------------------------------------------------------
static constexpr int kVT = 512;         // virtual threads of a pair's sums
static constexpr int kVW = kVT / 32;    // virtual warps

PIV_D unsigned cluster_rank() {
  unsigned r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
// Barrier of every thread of the cluster; orders shared and global memory. A
// kernel passes one before its first st_cluster: until then a CTA of the
// cluster may not have started, and its shared memory is not there to write.
PIV_D void cluster_barrier(int c) {
  if (c == 1) {
    __syncthreads();
  } else {
    asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
  }
}
// Stores v at *p (this CTA's shared memory) of CTA `rank` of the cluster.
PIV_D void st_cluster(double* p, unsigned rank, double v) {
  asm volatile(
      "{\n.reg .u32 a;\nmapa.shared::cluster.u32 a, %0, %1;\nst.shared::cluster.f64 [a], %2;\n}\n" ::"r"(
          (unsigned)__cvta_generic_to_shared(p)),
      "r"(rank), "d"(v)
      : "memory");
}

// CTAs per pair: the largest power of two up to 8 (the portable cluster size)
// that keeps every CTA on an SM of its own (with more pairs than that the
// float64 pipes are busy anyway). Measured: one pair's two GCV searches of a
// three-pass 1024 x 1024 run 396 -> 139 us with 8 CTAs, those of 64 pairs
// 230 -> 86 us with 2.
static int cluster_size(int n_pairs) {
  int c = 1;
  while (c < 8 && (long long)n_pairs * c * 2 <= sm_count()) c *= 2;
  return c;
}

template <typename... P, typename... A>
static int launch_cluster(void (*kernel)(P...), int n_pairs, int c, int threads, cudaStream_t stream, const char* what,
                          A... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)n_pairs * (unsigned)c);
  cfg.blockDim = dim3((unsigned)threads);
  cfg.stream = stream;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim.x = (unsigned)c;
  at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, static_cast<P>(args)...);
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, what);
}

// Sums over the warp of K values per lane, the sum of x[l] left in lane l: the
// xor tree (16, 8, 4, 2, 1) of a full warp sum per value, but each level
// halves the values a lane still carries (31 additions for up to 32 values
// instead of 5 per value; the additions pair the same lanes, so the sums are
// the same bit for bit).
template <int K, typename T>
PIV_D double warp_sums(const T (&x)[K]) {
  static_assert(K <= 32, "one value per lane");
  const int lane = threadIdx.x & 31;
  double v[16];
  {
    const bool up = lane & 16;
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      const T lo = i < K ? x[i] : (T)0, hi = i + 16 < K ? x[i + 16] : (T)0;
      const T other = __shfl_xor_sync(~0u, up ? lo : hi, 16);
      v[i] = (double)(up ? hi : lo) + (double)other;
    }
  }
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < o; ++i) {
      const double other = __shfl_xor_sync(~0u, up ? v[i] : v[i + o], o);
      v[i] = (up ? v[i + o] : v[i]) + other;
    }
  }
  return v[0];
}

// warp_sums of two values: one level that halves them, then the tree; the sum
// of x0 is in lanes 0 .. 15, that of x1 in lanes 16 .. 31.
PIV_D double warp_sums2(double x0, double x1) {
  const bool up = threadIdx.x & 16;
  double v = (up ? x1 : x0) + __shfl_xor_sync(~0u, up ? x0 : x1, 16);
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
  return v;
}

// warp_sums of four values: the sum of x[k] is in the lanes whose bits 4 and 3
// are k's bits 1 and 0.
PIV_D double warp_sums4(double x0, double x1, double x2, double x3) {
  const int lane = threadIdx.x & 31;
  const bool u16 = lane & 16, u8 = lane & 8;
  double a = (u16 ? x2 : x0) + __shfl_xor_sync(~0u, u16 ? x0 : x2, 16);
  double b = (u16 ? x3 : x1) + __shfl_xor_sync(~0u, u16 ? x1 : x3, 16);
  double v = (u8 ? b : a) + __shfl_xor_sync(~0u, u8 ? a : b, 8);
  for (int o = 4; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
  return v;
}

// x / c for a constant c with rc = 1 / c rounded: the correctly rounded
// quotient (Markstein 1990: the product's remainder is exact in one FMA, and
// one correction rounds as the division), a third of the division's chain of
// float64 instructions. Outside the range where that holds, the division.
PIV_D double div_const(double x, double c, double rc) {
  if (!(fabs(x) > 1e-280 && fabs(x) < 1e300)) return x / c;
  const double q = x * rc;
  return fma(fma(-q, c, x), rc, q);
}

// Fields of a DCT pass: component c of pair k at (c ? v : u) + k * stride.
struct DctIo {
  double* u;
  double* v;
  long long stride;
  PIV_D double* field(long long f) const { return ((f & 1) ? v : u) + (f >> 1) * stride; }
};
// The factor 1 / (1 + s lambda^2) on the inputs of the inverse row pass (lam2
// NULL: none): s of pair k is s[k], or `given` for every pair.
struct DctGamma {
  const double* lam2;
  const double* s;
  double given;
  PIV_D double of(long long pair) const { return s ? s[pair] : given; }
};

// out[b][i][l] = sum_j in[b][i][j] * c[l][j]       (transform along rows, mode 0)
// out[b][i][l] = sum_j in[b][i][j] * c[j][l]       (inverse along rows, mode 1)
// out[b][k][j] = sum_i c[k][i] * in[b][i][j]       (transform along columns, mode 2)
// out[b][k][j] = sum_i c[i][k] * in[b][i][j]       (inverse along columns, mode 3)
// Lines beyond the staged kernels' shared memory (kDctLongLen) only.
__global__ void k_dct_apply(int m, int n, int batch, int mode, const double* __restrict__ c, DctIo in, DctIo out) {
  const long long mn = (long long)m * n;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= mn * batch) return;
  const long long b = t / mn;
  const int e = (int)(t % mn);
  const int r = e / n, col = e % n;
  const double* x = in.field(b);
  double acc = 0.0;
  if (mode == 0) {
    for (int j = 0; j < n; ++j) acc = fma(x[r * n + j], c[col * n + j], acc);
  } else if (mode == 1) {
    for (int j = 0; j < n; ++j) acc = fma(x[r * n + j], c[j * n + col], acc);
  } else if (mode == 2) {
    for (int i = 0; i < m; ++i) acc = fma(c[r * m + i], x[i * n + col], acc);
  } else {
    for (int i = 0; i < m; ++i) acc = fma(c[i * m + r], x[i * n + col], acc);
  }
  out.field(b)[e] = acc;
}

// Dot product of two hi/lo float vectors in float32 with error-free
// transformations: every product's rounding error is kept (fma), the cross
// terms a_hi b_lo + a_lo b_hi join a small-term sum, and the main sum is
// compensated (TwoSum). The result, (hi, lo), is within ~1e-13 of the float64
// dot product here (orthonormal cosine matrices, smooth fields), at a fraction
// of the cost of float64 FMAs on this GPU.
struct DfAcc {
  float s = 0.f, c = 0.f;
  PIV_D void add(float ah, float al, float bh, float bl) {
    const float p = ah * bh;
    c += fmaf(ah, bh, -p) + fmaf(ah, bl, al * bh);
    const float t = s + p, bp = t - s;
    c += (s - (t - bp)) + (p - bp);
    s = t;
  }
  PIV_D void result(float& hi, float& lo) const {
    hi = s + c;
    lo = c - (hi - s);
  }
};

// 1/d for d >= 1 from the float32 reciprocal and two Newton steps in float64:
// within an ulp or two of the rounded quotient, at a fraction of the cost of
// a float64 division (float64 throughput on this GPU is low).
PIV_D double rcp_fast(double d) {
  double r = (double)__frcp_rn((float)d);
  double e = fma(-d, r, 1.0);
  r = fma(r, e, r);
  e = fma(-d, r, 1.0);
  return fma(r, e, r);
}

static constexpr int kDctLines = 32, kDctThreads = 256, kDctMaxLen = 90;
static constexpr int kDctLongLen = 860;  // 33 doubles per position: 227 KB

// DCT-II (or, INV, DCT-III) of kDctLines lines per CTA with the symmetric
// split of the cosine matrix: C[k][L-1-i] = (-1)^k C[k][i], so the forward
// transform needs only the sums x[i] + x[L-1-i] (even k) or differences (odd
// k) of the first L/2 positions, and the inverse gives x[i] and x[L-1-i] from
// one pass over the even and the odd k: half the products. The lines are
// staged in shared memory as [position][line]; `cols` selects lines along the
// columns of the [m][n] fields instead of along the rows. blockIdx.y takes a
// share of the outputs, so that a few lines still fill the SMs (one pair of
// 63 x 63 has 126 lines, 4 CTAs).
// DF: double-float products (DfAcc: hi/lo float pairs with error-free
// transformations, within ~1e-13 of float64) with cf the matrix as [2][L][L]
// hi/lo floats; else float64 products with cd, which the float64 pipe bounds.
template <bool INV, bool DF>
__global__ void __launch_bounds__(kDctThreads) k_dct_lines(int m, int n, int batch, int cols, const float* __restrict__ cf,
                                                           const double* __restrict__ cd, DctIo in, DctIo out,
                                                           DctGamma gam) {
  extern __shared__ double dsm[];
  const int nt = blockDim.x;
  const int L = cols ? m : n;
  const long long n_lines = (long long)batch * (cols ? n : m);
  const long long l0 = (long long)blockIdx.x * kDctLines;
  constexpr int S = kDctLines + 1;           // odd stride: conflict-free rows of 32 lines
  double* xs = dsm;                          // [L][S] doubles
  const int h = L / 2, hc = (L + 1) / 2;
  float* fs = reinterpret_cast<float*>(dsm + L * S);  // DF: 4 hc S floats after xs
  const float* ch = cf;
  const float* cl = cf + (size_t)L * L;
  // The lines' places, found once per line: first elements of input and
  // output, of the line in lambda^2, and s of its pair.
  __shared__ const double* src_s[kDctLines];
  __shared__ double* dst_s[kDctLines];
  __shared__ int at_s[kDctLines];
  __shared__ double s_s[kDctLines];
  const int step = cols ? n : 1;  // between the elements of a line
  if (threadIdx.x < kDctLines) {
    const long long line = l0 + threadIdx.x, per = cols ? n : m;
    const long long f = line < n_lines ? line / per : 0;
    const int q = line < n_lines ? (int)(line - f * per) : 0, at = cols ? q : q * n;
    src_s[threadIdx.x] = line < n_lines ? in.field(f) + at : nullptr;
    dst_s[threadIdx.x] = line < n_lines ? out.field(f) + at : nullptr;
    at_s[threadIdx.x] = at;
    s_s[threadIdx.x] = INV && gam.lam2 ? gam.of(f >> 1) : 0.0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = nt / 32;
  // Staging, coalesced along the line for rows and across lines for columns:
  // kBatch loads of a thread are in flight together (64 pairs of 63 x 63, four
  // passes: 139 us with four at a time, 126 us with eight).
  constexpr int kBatch = DF ? 8 : 16;
  const unsigned n_el = (unsigned)(kDctLines * L);
  for (unsigned b0 = threadIdx.x; b0 < n_el; b0 += kBatch * nt) {
    double v[kBatch];
    int l[kBatch], e[kBatch];
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      const unsigned id = b0 + k * nt;
      const bool ok = id < n_el;
      l[k] = !ok ? 0 : (int)(cols ? id % kDctLines : id / (unsigned)L);
      e[k] = !ok ? 0 : (int)(cols ? id / kDctLines : id % (unsigned)L);
      const double* p = ok ? src_s[l[k]] : nullptr;
      v[k] = p ? p[(long long)e[k] * step] : 0.0;
    }
#pragma unroll
    for (int k = 0; k < kBatch; ++k) {
      if (b0 + k * nt >= n_el) break;
      if (INV && gam.lam2) v[k] = rcp_fast(1.0 + s_s[l[k]] * gam.lam2[at_s[l[k]] + e[k] * step]) * v[k];
      xs[e[k] * S + l[k]] = v[k];
    }
  }
  __syncthreads();
  const int split_n = gridDim.y, share = blockIdx.y;
  double* dst = dst_s[lane];  // this lane's output line
  const bool mine = dst != nullptr;
  auto split = [](double x, float& hi, float& lo) {
    hi = (float)x;
    lo = (float)(x - (double)hi);
  };
  // Outputs go back through the staging buffer where one CTA holds all of
  // them (coalesced stores); a share of them is stored directly.
  auto put = [&](int e, double v) {
    if (split_n == 1) xs[e * S + lane] = v;
    else if (mine) dst[(long long)e * step] = v;
  };
  if (!INV) {
    // Sums and differences of mirrored inputs.
    float* esh = fs;
    float* esl = fs + hc * S;
    float* osh = fs + 2 * hc * S;
    float* osl = fs + 3 * hc * S;
    for (int i = warp; i < h; i += nw) {
      const double a = xs[i * S + lane], b = xs[(L - 1 - i) * S + lane];
      if (DF) {
        split(a + b, esh[i * S + lane], esl[i * S + lane]);
        split(a - b, osh[i * S + lane], osl[i * S + lane]);
      } else {
        xs[i * S + lane] = a + b;
        xs[(L - 1 - i) * S + lane] = a - b;
      }
    }
    float mid_h = 0.f, mid_l = 0.f;
    double mid = 0.0;
    if (L & 1) {
      mid = xs[h * S + lane];
      split(mid, mid_h, mid_l);
    }
    __syncthreads();
    if (DF) {
      // y[k] (into xs: the inputs are no longer needed).
      for (int k = share * nw + warp; k < L; k += nw * split_n) {
        const float* sh = (k & 1) ? osh : esh;
        const float* sl = (k & 1) ? osl : esl;
        const float* ckh = ch + (long long)k * L;
        const float* ckl = cl + (long long)k * L;
        DfAcc acc;
        if (L & 1) acc.add(ckh[h], ckl[h], mid_h, mid_l);
#pragma unroll 8
        for (int i = 0; i < h; ++i) acc.add(ckh[i], ckl[i], sh[i * S + lane], sl[i * S + lane]);
        float rh, rl;
        acc.result(rh, rl);
        put(k, (double)rh + (double)rl);
      }
    } else {
      // Two outputs of one parity per turn share the loaded sums.
      for (int g = share * nw + warp; 2 * g < L + 2; g += nw * split_n) {
        const int par = g & 1, k0 = 4 * (g >> 1) + par, k1 = k0 + 2;
        if (k0 >= L) continue;
        const double* c0 = cd + (long long)k0 * L;
        const double* c1 = cd + (long long)min(k1, L - 1) * L;
        double a0 = (L & 1) ? c0[h] * mid : 0.0, a1 = (L & 1) ? c1[h] * mid : 0.0;
        const double* x = par ? xs + (L - 1) * S + lane : xs + lane;
        const int xstep = par ? -S : S;
#pragma unroll 8
        for (int i = 0; i < h; ++i, x += xstep) {
          a0 = fma(__ldg(c0 + i), *x, a0);
          a1 = fma(__ldg(c1 + i), *x, a1);
        }
        if (mine) dst[(long long)k0 * step] = a0;
        if (mine && k1 < L) dst[(long long)k1 * step] = a1;
      }
    }
  } else if (DF) {
    // The inputs as hi/lo floats.
    float* xh = fs;
    float* xl = fs + L * S;
    for (int idx = threadIdx.x; idx < L * kDctLines; idx += nt) {
      const int q = (idx / kDctLines) * S + idx % kDctLines;
      split(xs[q], xh[q], xl[q]);
    }
    __syncthreads();
    for (int i = share * nw + warp; i < hc; i += nw * split_n) {
      DfAcc ev, od;
#pragma unroll 8
      for (int k = 0; k < L; k += 2) ev.add(ch[(long long)k * L + i], cl[(long long)k * L + i], xh[k * S + lane], xl[k * S + lane]);
#pragma unroll 8
      for (int k = 1; k < L; k += 2) od.add(ch[(long long)k * L + i], cl[(long long)k * L + i], xh[k * S + lane], xl[k * S + lane]);
      float eh, el, oh, ol;
      ev.result(eh, el);
      od.result(oh, ol);
      const double e = (double)eh + (double)el, o = (double)oh + (double)ol;
      put(i, e + o);                          // x[i]
      if (L - 1 - i != i) put(L - 1 - i, e - o);  // x[L-1-i]
    }
  } else {
    for (int g = share * nw + warp; 2 * g < hc; g += nw * split_n) {
      const int i0 = 2 * g, i1 = min(i0 + 1, hc - 1);
      double e0 = 0.0, e1 = 0.0, o0 = 0.0, o1 = 0.0;
#pragma unroll 4
      for (int k = 0; k + 1 < L; k += 2) {
        const double x = xs[k * S + lane], y = xs[(k + 1) * S + lane];
        const double* c = cd + (long long)k * L;
        e0 = fma(__ldg(c + i0), x, e0);
        e1 = fma(__ldg(c + i1), x, e1);
        o0 = fma(__ldg(c + L + i0), y, o0);
        o1 = fma(__ldg(c + L + i1), y, o1);
      }
      if (L & 1) {
        const double x = xs[(L - 1) * S + lane];
        const double* c = cd + (long long)(L - 1) * L;
        e0 = fma(__ldg(c + i0), x, e0);
        e1 = fma(__ldg(c + i1), x, e1);
      }
      if (!mine) continue;
      dst[(long long)i0 * step] = e0 + o0;
      if (L - 1 - i0 != i0) dst[(long long)(L - 1 - i0) * step] = e0 - o0;
      if (i1 == i0) continue;
      dst[(long long)i1 * step] = e1 + o1;
      if (L - 1 - i1 != i1) dst[(long long)(L - 1 - i1) * step] = e1 - o1;
    }
  }
  if (!DF || split_n > 1) return;
  __syncthreads();
  if (cols) {
    for (int e = warp; e < L; e += nw)
      if (mine) dst[(long long)e * step] = xs[e * S + lane];
  } else {
#pragma unroll 4
    for (unsigned idx = threadIdx.x; idx < (unsigned)(kDctLines * L); idx += nt) {
      const int l = (int)(idx / (unsigned)L), e = (int)(idx % (unsigned)L);
      if (dst_s[l]) dst_s[l][e] = xs[e * S + l];
    }
  }
}

// Both fields of every pair times 1 / (1 + s lambda^2).
__global__ void k_apply_gamma(long long mn, DctGamma gam, DctIo io) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x, pair = blockIdx.y;
  if (e >= mn) return;
  const double g = rcp_fast(1.0 + gam.of(pair) * gam.lam2[e]);
  double* u = io.field(2 * pair) + e;
  double* v = io.field(2 * pair + 1) + e;
  *u = g * *u;
  *v = g * *v;
}

// One DCT pass over `batch` fields: forward (DCT-II) or inverse (DCT-III)
// along rows (cols = 0, tables of size n) or columns (cols = 1, size m). Lines
// of up to kDctMaxLen positions take the double-float products, longer ones
// the float64 products (the double-float error grows with the length), both
// staged with the symmetric split. Measured, the four passes of one pair: 31 x
// 31 30 us, 253 x 253 174 us (plain float64 dot products 283 us), 170 x 137
// 89 us (87 us, plus 5 us for gamma and 6 us for the copies, which are part
// of these passes); 16 pairs of 253 x 253 2.13 ms (3.36 ms), of which 1.65 ms
// at the float64 rate. The staging's loads in flight matter as much as the
// products for a few lines: four of a thread at a time 200 / 106 us.
template <bool INV>
static int dct_pass(int m, int n, int batch, int cols, const SmoothTables& t, DctIo in, DctIo out, DctGamma gam,
                    cudaStream_t stream) {
  const int L = cols ? m : n;
  const long long n_lines = (long long)batch * (cols ? n : m);
  const bool df = L <= kDctMaxLen;
  const long long blocks = (n_lines + kDctLines - 1) / kDctLines;
  // Shares of the outputs: as many as the SMs take, each warp of a share
  // with at least one turn (fewer warps per CTA stage the lines too slowly).
  const int turns = df ? (INV ? (L + 1) / 2 : L) : (INV ? (L + 3) / 4 : (L + 1) / 2);
  const long long room = blocks < sm_count() ? sm_count() / blocks : 1;
  const int shares = (int)std::min<long long>((turns + kDctThreads / 32 - 1) / (kDctThreads / 32), room);
  // Every share of the staged kernels scales all of its lines' inputs, nine
  // float64 instructions each: from three shares on, one launch that scales
  // them once costs less (253 x 253, nine shares: both inverse passes 105 us,
  // now 82 us and a launch of 3 us).
  if (gam.lam2 && (L > kDctLongLen || (!df && shares >= 3))) {
    const long long mn = (long long)m * n;
    k_apply_gamma<<<dim3((unsigned)((mn + 127) / 128), (unsigned)(batch / 2)), 128, 0, stream>>>(mn, gam, in);
    gam = DctGamma{nullptr, nullptr, 0.0};
  }
  if (L > kDctLongLen) {
    const long long tot = (long long)m * n * batch;
    const int mode = cols ? (INV ? 3 : 2) : (INV ? 1 : 0);
    k_dct_apply<<<(unsigned)((tot + 255) / 256), 256, 0, stream>>>(m, n, batch, mode, cols ? t.cm : t.cn, in, out);
    return check("k_dct_apply");
  }
  const float* cf = cols ? t.cmf : t.cnf;
  const double* cd = cols ? t.cm : t.cn;
  const int threads = kDctThreads;
  const dim3 grid((unsigned)blocks, (unsigned)shares);
  if (df) {
    const size_t smem = (size_t)(L + 2 * ((L + 1) / 2)) * (kDctLines + 1) * sizeof(double);
    k_dct_lines<INV, true><<<grid, threads, smem, stream>>>(m, n, batch, cols, cf, cd, in, out, gam);
  } else {
    const size_t smem = (size_t)L * (kDctLines + 1) * sizeof(double);
    cudaError_t e = cudaFuncSetAttribute(k_dct_lines<INV, false>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         kDctLongLen * (kDctLines + 1) * (int)sizeof(double));
    if (e != cudaSuccess) return set_cuda_error(e, "cudaFuncSetAttribute(k_dct_lines)");
    k_dct_lines<INV, false><<<grid, threads, smem, stream>>>(m, n, batch, cols, cf, cd, in, out, gam);
  }
  return check("k_dct_lines");
}

// Flags of SmoothnGPU's log messages (gpu_smoothn.py:218-222, 429-439): with
// GCV, the smoothing parameter within 0.1 (in log10) of its lower or else its
// upper bound; the iteration reaching its last allowed step.
PIV_D int smooth_flags(bool is_auto, double p, double pmin, double pmax, bool last_iter) {
  int f = 0;
  if (is_auto) {
    if (fabs(p - pmin) < 0.1) f |= PIV_SMOOTH_S_LOWER;
    else if (fabs(p - pmax) < 0.1) f |= PIV_SMOOTH_S_UPPER;
  }
  if (last_iter) f |= PIV_SMOOTH_MAX_ITERS;
  return f;
}

// The GCV search of one pair, by the c CTAs of a cluster. The sums of each
// score are formed by the kVT virtual threads (each CTA runs kVT / c of them);
// the warps' partial sums go to every CTA of the cluster through distributed
// shared memory, and warp 0 of every CTA adds them in warp order and runs the
// search (scan bookkeeping and the L-BFGS-B steps: scalar float64 work) for
// itself, so one cluster barrier per evaluation suffices. The fast score
// (float32 terms, float64 sums: 1 - gamma = s l / (1 + s l) formed without
// cancellation, each term within a few float32 ulps, the score within ~1e-9)
// only ranks the scan points, all ten in one pass over the field; the
// L-BFGS-B evaluations, whose difference quotients divide score differences
// by 1e-8, use the float64 score, the point and its neighbour together. SETS
// = 2 (clusters of eight, whose CTAs hold two virtual warps): a second set of
// the virtual threads sums the scores of the odd points, so that all four
// float64 units of an SM work.
// Bound by the float64 pipe and by the latency of the search's steps. One
// score at a time on one CTA, with the scan in ten passes, took 396 us for
// the 31 x 31 and 63 x 63 fields of one 1024 x 1024 pair; this takes 139 us.
template <int SETS>
__global__ void __launch_bounds__(kVT)
k_gcv(int m, int n, int c, double rmn, const double* __restrict__ fd, double* __restrict__ f2, float* __restrict__ f2f,
      const double* __restrict__ lam2, const float* __restrict__ lam2f, double pmin, double pmax,
      double* __restrict__ p_out, double* __restrict__ s_out, int* __restrict__ flags) {
  __shared__ double part[2][kVW][20];  // by parity of the evaluation: the virtual warps' partial sums
  __shared__ double sh_s[10];          // 10^p of the next scores
  __shared__ int sh_go;                // warp 0's decision for the next step
  const int pair = blockIdx.x / c;
  const int rank = c > 1 ? (int)cluster_rank() : 0;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int vtn = kVT / c, set = SETS == 2 && (int)threadIdx.x >= vtn;
  const int vt = rank * vtn + (threadIdx.x - set * vtn), vw = vt >> 5;
  const bool w0 = warp == 0;
  const long long mn = (long long)m * n;
  const double* fu = fd + 2 * pair * mn;
  double* f2p = f2 + pair * mn;
  float* f2fp = f2f + pair * mn;
  const double n_finite = (double)mn;
  // fd_u^2 + fd_v^2, by the first set.
  for (long long e = vt; !set && e < mn; e += kVT) {
    const double a = fu[e], b = fu[mn + e];
    const double q = a * a + b * b;
    f2p[e] = q;
    f2fp[e] = (float)q;
  }
  int par = 0;
  // Leaves v as the virtual warp's partial sum `slot` in CTA r of the cluster.
  auto put = [&](int slot, double v, int r) {
    if (c == 1) part[par][vw][slot] = v;
    else st_cluster(&part[par][vw][slot], (unsigned)r, v);
  };
  // 10-point scan (gpu_smoothn.py:182-188), ranked with the fast score; when
  // other points score within 1e-6 of the best, those points are scored
  // again in float64 and the first minimum among them is kept (np.argmin).
  auto scan_point = [&](int k) { return fma((double)k * (1.0 / 9.0), pmax - pmin, pmin); };
  if (threadIdx.x < 10) sh_s[threadIdx.x] = pow(10.0, scan_point(threadIdx.x));
  cluster_barrier(c);  // sh_s is complete, and every CTA of the cluster runs
  {
    // Points SETS k + set: sums of the residuals in acc[k], of 1 - gamma in
    // acc[PER + k].
    constexpr int PER = 10 / SETS;
    float acc[2 * PER], s[PER];
#pragma unroll
    for (int k = 0; k < PER; ++k) {
      s[k] = (float)sh_s[SETS * k + set];
      acc[k] = acc[PER + k] = 0.f;
    }
    for (long long e = vt; e < mn; e += kVT) {
      const float l = lam2f[e], f = f2fp[e];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        const float sl = s[k] * l;
        const float d = sl * __frcp_rn(1.0f + sl);  // 1 - gamma
        acc[k] = fmaf(f * d, d, acc[k]);
        acc[PER + k] += d;
      }
    }
    const double v = warp_sums(acc);
    if (lane < 2 * PER)
      for (int r = 0; r < c; ++r) put((lane < PER ? 0 : 10) + SETS * (lane % PER) + set, v, r);
    cluster_barrier(c);
  }
  double p0 = pmin;
  unsigned rescore = 0;  // scan points within 1e-6 of the best fast score, when there are several
  if (w0) {
    const int q = lane < 10 ? lane : 0;
    double trss = 0.0, ttr = 0.0;
    for (int k = 0; k < kVW; ++k) {
      trss += part[par][k][q];
      ttr += part[par][k][10 + q];
    }
    const double w = div_const(ttr, n_finite, rmn);
    const double f = div_const(trss, n_finite, rmn) / (w * w) / 2;
    double best_f = INFINITY;
    double fast[10];
#pragma unroll
    for (int k = 0; k < 10; ++k) {
      fast[k] = __shfl_sync(~0u, f, k);
      if (fast[k] < best_f) best_f = fast[k];
    }
    unsigned near_best = 0;
#pragma unroll
    for (int k = 9; k >= 0; --k) {
      if (fast[k] <= best_f + 1e-6 * fabs(best_f)) near_best |= 1u << k;
      if (fast[k] == best_f) p0 = scan_point(k);
    }
    if (lane == 0) sh_go = __popc(near_best) > 1 ? (int)near_best : 0;
  }
  par ^= 1;
  // Announces two points (warp 0) and whether the search goes on, and makes
  // both visible to the CTA.
  auto announce = [&](double pa, double pb, bool go) {
    if (w0) {
      if (lane < 2) sh_s[lane] = pow(10.0, lane ? pb : pa);
      if (lane == 0) sh_go = go;
    }
    __syncthreads();
  };
  // Float64 scores at the two announced points (valid in warp 0).
  auto score2 = [&](double& fa, double& fb) {
    if constexpr (SETS == 2) {
      const double s = sh_s[set];
      double rss = 0.0, tr = 0.0;
      for (long long e = vt; e < mn; e += kVT) {
        const double gm = rcp_fast(1.0 + s * lam2[e]);
        const double d = gm - 1.0;
        rss += f2p[e] * d * d;
        tr += gm;
      }
      // Lane l holds sum l / 16, for CTA l % 16.
      const double v = warp_sums2(rss, tr);
      if ((lane & 15) < c) put(2 * set + (lane >> 4), v, lane & 15);
    } else {
      const double sa = sh_s[0], sb = sh_s[1];
      double ra = 0.0, ta = 0.0, rb = 0.0, tb = 0.0;
      for (long long e = vt; e < mn; e += kVT) {
        const double l = lam2[e], f = f2p[e];
        const double ga = rcp_fast(1.0 + sa * l), gb = rcp_fast(1.0 + sb * l);
        const double da = ga - 1.0, db = gb - 1.0;
        ra += f * da * da;
        ta += ga;
        rb += f * db * db;
        tb += gb;
      }
      // Lane l holds sum l / 8, for CTA l % 8.
      const double v = warp_sums4(ra, ta, rb, tb);
      if ((lane & 7) < c) put(lane >> 3, v, lane & 7);
    }
    cluster_barrier(c);
    if (w0) {
      double t = 0.0;
      for (int k = 0; k < kVW; ++k) t += part[par][k][lane & 3];
      const double trss = __shfl_sync(~0u, t, (lane & 1) * 2), ttr = __shfl_sync(~0u, t, (lane & 1) * 2 + 1);
      const double q = 1.0 - div_const(ttr, n_finite, rmn);
      const double f = div_const(trss, n_finite, rmn) / (q * q) / 2;
      fa = __shfl_sync(~0u, f, 0);
      fb = __shfl_sync(~0u, f, 1);
    }
    par ^= 1;
  };
  __syncthreads();
  rescore = (unsigned)sh_go;
  if (rescore) {
    double best64 = INFINITY;
    p0 = pmin;
    while (rescore) {
      const int ka = __ffs(rescore) - 1;
      rescore &= rescore - 1;
      const int kb = rescore ? __ffs(rescore) - 1 : ka;
      rescore &= rescore - 1;
      const double pa = scan_point(ka), pb = scan_point(kb);
      __syncthreads();  // every read of sh_go and sh_s is done
      announce(pa, pb, true);
      double fa = 0.0, fb = 0.0;
      score2(fa, fb);
      if (fa < best64) { best64 = fa; p0 = pa; }
      if (fb < best64) { best64 = fb; p0 = pb; }
    }
  }
  // L-BFGS-B from the scan point (gpu_smoothn.py:191-193), its scalar state
  // in warp 0.
  Lb1 lb;
  lb.done = false;
  if (w0) lb_init(lb, p0, pmin, pmax);
  for (int ev = 0; ev < kLbMaxEvals; ++ev) {
    double xt = 0.0, xs = 0.0;
    if (w0) {
      xt = lb.xt;
      xs = lb_fd_point(xt, pmin, pmax);
    }
    __syncthreads();  // every read of sh_go and sh_s is done
    announce(xt, xs, !lb.done);
    if (!sh_go) break;
    double f = 0.0, fh = 0.0;
    score2(f, fh);
    if (w0) lb_feed(lb, f, (fh - f) / (xs - xt));
  }
  if (rank == 0 && threadIdx.x == 0) {
    const double p = lb.x;
    s_out[pair] = pow(10.0, p);
    if (p_out) p_out[pair] = p;
    if (flags) flags[pair] = smooth_flags(true, p, pmin, pmax, false);
  }
}

__global__ void k_fill(int count, double value, double* out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t < count) out[t] = value;
}

// Bounds of p = log10(s) for order 2 (gpu_smoothn.py:320-338), on the host.
static void gcv_bounds(int m, int n, double* pmin, double* pmax) {
  const double h_min = 1e-3, h_max = 1.0 - h_min;
  const int rank = (m != 1) + (n != 1);
  const double a_max = pow(h_max, 2.0 / rank), a_min = pow(h_min, 2.0 / rank);
  *pmin = log10((pow((1.0 + sqrt(1.0 + 8.0 * a_max)) / 4.0 / a_max, 2.0) - 1.0) / 16.0);
  *pmax = log10((pow((1.0 + sqrt(1.0 + 8.0 * a_min)) / 4.0 / a_min, 2.0) - 1.0) / 16.0);
}

// ---------------------------------------------------------------------------
// Weighted smoothn (a field mask, or fields with non-finite values): Garcia's
// iteration as SmoothnGPU runs it with weights (gpu_smoothn.py:123-231):
// missing values take the value of their nearest finite neighbour
// (replace_non_finite, gpu_smoothn.py:233-251, with scipy's feature-transform
// choice among equidistant neighbours: per column the nearest finite row, the
// lower one on a tie, then the nearest column, the lower one on a tie), the
// start z keeps the low DCT coefficients (get_init_z, gpu_smoothn.py:284-297),
// then z <- rf IDCT2(gamma DCT2(w (f - z) + z)) + (1 - rf) z with rf = 1.75
// until ||z_old - z|| / (||z|| + 1e-6) <= 1e-3 or 100 iterations; with s unset
// the GCV search runs at iterations 1, 2, 4, 8, ... (gpu_smoothn.py:176-193),
// with the w_mean <= 0.9 score refitting the field for every candidate s
// (gpu_smoothn.py:359-368). Output zero inside the mask (gpu_smoothn.py:224-225).
// Float64 throughout but for the DCTs' double-float products (DfAcc).
//
// A cluster of c CTAs runs each pair (cluster_size). CTA r owns the rows [r
// R, (r + 1) R) of the 2 m rows of the two fields: it transforms its rows and
// forms its rows of the column passes, whose inputs (all rows) come through
// global memory (L2) with one cluster barrier in between; the forward column
// pass leaves the rows that the inverse row pass of the same CTA starts from.
// The sums run over virtual threads as in k_gcv, so the result does not
// depend on c. Sums of two products have their roundings written out (the
// search stops where its curve is flat: a last bit of a score moves p by
// 1e-4). Bound by the DCTs' dot products and the barriers between
// passes: one pair of 63 x 63 around a masked disc takes 0.84 to 0.89 ms with 8 CTAs.
// On one CTA, with strided matrix reads and 10^p formed by every thread, it
// took 6.4 ms.
// ---------------------------------------------------------------------------
static constexpr int kSwThreads = 512;

struct SwShared {
  double red[2][20][kVW];  // by parity of the sums: the virtual warps' partial sums
  double sums[20];
  double s[10];
  int go;
};

struct SwCtx {
  int m, n, mn, c, rank, par;
  int e0, e1;  // this CTA's rows as flat elements of the two fields
  const double* lam2;
  const float2 *cm, *cn, *cnt;  // DCT matrices as (hi, lo): [m][m], [n][n] and its transpose
  double *f, *z, *zo, *fd, *tmp, *w;
  double n_finite, w_mean;
  SwShared* sh;
};

// Row pass over this CTA's rows, in the double-float arithmetic of DfAcc: the
// inputs load(e) are split into xs (this CTA's rows of it), the results go to
// out as (hi, lo). out may be the array that load reads.
template <class Load>
PIV_D void sw_row_pass(const SwCtx& x, bool inv, Load load, float2* xs, float2* out) {
  for (int e = x.e0 + threadIdx.x; e < x.e1; e += kSwThreads) {
    const double v = load(e);
    const float h = (float)v;
    xs[e] = make_float2(h, (float)(v - (double)h));
  }
  __syncthreads();
  const float2* mat = inv ? x.cn : x.cnt;
  const int n = x.n;
  for (int e = x.e0 + threadIdx.x; e < x.e1; e += kSwThreads) {
    const int l = e % n;
    const float2* xr = xs + (e - l);
    const float2* mc = mat + l;
    DfAcc acc;
#pragma unroll 8
    for (int j = 0; j < n; ++j) {
      const float2 a = xr[j], b = __ldg(mc + (long long)j * n);
      acc.add(a.x, a.y, b.x, b.y);
    }
    float2 r;
    acc.result(r.x, r.y);
    out[e] = r;
  }
}

// Column pass: this CTA's rows of the result from all rows of `in`.
template <class Store>
PIV_D void sw_col_pass(const SwCtx& x, bool inv, const float2* in, Store store) {
  const int m = x.m, n = x.n, mn = x.mn;
  for (int e = x.e0 + threadIdx.x; e < x.e1; e += kSwThreads) {
    const int fi = e >= mn ? 1 : 0, q = e - fi * mn, k = q / n, j = q - k * n;
    const float2* col = in + fi * mn + j;
    const float2* mr = inv ? x.cm + k : x.cm + k * m;
    const int ms = inv ? m : 1;
    DfAcc acc;
#pragma unroll 8
    for (int i = 0; i < m; ++i) {
      const float2 a = __ldg(mr + i * ms), b = col[i * n];
      acc.add(a.x, a.y, b.x, b.y);
    }
    float h, l;
    acc.result(h, l);
    store(e, (double)h + (double)l);
  }
}

// Leaves v as partial sum `slot` of virtual warp vw in CTA r of the cluster.
PIV_D void sw_put(SwCtx& x, int slot, int vw, double v, int r) {
  if (x.c == 1) x.sh->red[x.par][slot][vw] = v;
  else st_cluster(&x.sh->red[x.par][slot][vw], (unsigned)r, v);
}

// After every virtual warp's sw_put: the sums of `count` values into sh->sums
// (every thread of the cluster calls it; it ends with a barrier).
PIV_D void sw_take(SwCtx& x, int count) {
  const int lane = threadIdx.x & 31, q = (threadIdx.x >> 5) * 2 + (lane >> 4);
  cluster_barrier(x.c);
  if (q < ((count + 1) & ~1)) {  // whole warps: two values each
    double t = x.sh->red[x.par][q][lane & 15];
    for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(~0u, t, o);
    if ((lane & 15) == 0) x.sh->sums[q] = t;
  }
  __syncthreads();
  x.par ^= 1;
}

// Sums over the pair's virtual threads of two values, into sh->sums[0 .. 1].
PIV_D void sw_sums(SwCtx& x, double a, double b) {
  const int lane = threadIdx.x & 31, vtn = kVT / x.c;
  if ((int)threadIdx.x < vtn) {
    const double v = warp_sums2(a, b);
    if ((lane & 15) < x.c) sw_put(x, lane >> 4, (x.rank * vtn + threadIdx.x) >> 5, v, lane & 15);
  }
  sw_take(x, 2);
}

// GCV scores of the first `count` (2 or 10) announced points (gpu_smoothn.py:
// 353-372; s in sh->s), score k in lane k of warp 0. fd: DCT of both fields.
// The points are shared between two sets of the virtual threads (the even ones
// and the odd ones) where the CTA has room for both.
template <int COUNT>
PIV_D double sw_scores(SwCtx& x) {
  constexpr int PER = COUNT / 2;
  const int mn = x.mn, vtn = kVT / x.c, lane = threadIdx.x & 31;
  const int sets = 2 * vtn <= kSwThreads ? 2 : 1, set = (int)threadIdx.x / vtn;
  const int vt = set < sets ? x.rank * vtn + (int)threadIdx.x % vtn : 0x7fffffff;
  const int vw = vt >> 5;
  if (x.w_mean > 0.9) {
    for (int g = set; g < 2 && set < sets; g += sets) {  // points 2 k + g
      double s[PER], acc[2 * PER];
#pragma unroll
      for (int k = 0; k < PER; ++k) {
        s[k] = x.sh->s[2 * k + g];
        acc[k] = acc[PER + k] = 0.0;
      }
      for (int e = vt; e < mn; e += kVT) {
        const double l = x.lam2[e], fu = x.fd[e], fv = x.fd[mn + e];
        const double f2 = fma(fu, fu, __dmul_rn(fv, fv));
#pragma unroll
        for (int k = 0; k < PER; ++k) {
          const double gm = rcp_fast(1.0 + s[k] * l);
          const double d = gm - 1.0;
          acc[k] = fma(f2 * d, d, acc[k]);
          acc[PER + k] += gm;
        }
      }
      if constexpr (PER == 1) {
        const double v = warp_sums2(acc[0], acc[1]);
        if ((lane & 15) < x.c) sw_put(x, 2 * (lane >> 4) + g, vw, v, lane & 15);
      } else {
        const double v = warp_sums(acc);
        if (lane < 2 * PER)
          for (int r = 0; r < x.c; ++r) sw_put(x, (lane < PER ? 0 : COUNT) + 2 * (lane % PER) + g, vw, v, r);
      }
    }
  } else {
    const int vt1 = (int)threadIdx.x < vtn ? vt : 0x7fffffff;  // one set: the refit takes every thread
    for (int k = 0; k < COUNT; ++k) {
      const double s = x.sh->s[k];
      double rss = 0.0, tr = 0.0;
      for (int e = vt1; e < mn; e += kVT) tr += rcp_fast(1.0 + s * x.lam2[e]);
      // f_hat = IDCT2(gamma fd), into the spare z buffer.
      sw_row_pass(x, true, [&](int e) { return __dmul_rn(x.fd[e], rcp_fast(1.0 + s * x.lam2[e >= mn ? e - mn : e])); },
                  reinterpret_cast<float2*>(x.zo), reinterpret_cast<float2*>(x.tmp));
      cluster_barrier(x.c);
      sw_col_pass(x, true, reinterpret_cast<const float2*>(x.tmp), [&](int e, double v) { x.zo[e] = v; });
      cluster_barrier(x.c);
      for (int fi = 0; fi < 2; ++fi)
        for (int e = vt1; e < mn; e += kVT) {
          const double fv = x.f[fi * mn + e];
          if (isfinite(fv) || x.w[e] > 0) {
            const double d = fv - x.zo[fi * mn + e];
            rss += x.w[e] * d * d;
          }
        }
      if ((int)threadIdx.x < vtn) {
        const double v = warp_sums2(rss, tr);
        if ((lane & 15) < x.c) sw_put(x, COUNT * (lane >> 4) + k, vw, v, lane & 15);
      }
      cluster_barrier(x.c);  // the next refit rewrites the buffers
    }
  }
  sw_take(x, 2 * COUNT);
  double f = 0.0;
  if (threadIdx.x < 32) {
    const int k = lane < COUNT ? lane : 0;
    const double q = 1.0 - x.sh->sums[COUNT + k] / (double)mn;
    f = x.sh->sums[k] / x.n_finite / (q * q) / 2.0;
  }
  return f;
}

// Announces 10^p of a point per lane (count lanes of warp 0) and whether the
// search goes on.
PIV_D void sw_announce(SwCtx& x, int count, double p, bool go) {
  __syncthreads();  // every read of the previous announcement is done
  if ((int)threadIdx.x < count) x.sh->s[threadIdx.x] = pow(10.0, p);
  if (threadIdx.x == 0) x.sh->go = go;
  __syncthreads();
}

// The search of k_gcv: the 10-point scan on the first call (float64 scores,
// np.argmin's first minimum), then L-BFGS-B from the start point
// (gpu_smoothn.py:179-193), its scalar steps in warp 0 of every CTA.
PIV_D double sw_search(SwCtx& x, double p, bool have_p, double pmin, double pmax) {
  const bool w0 = threadIdx.x < 32;
  const int lane = threadIdx.x & 31;
  auto scan_point = [&](int k) { return fma((double)k * (1.0 / 9.0), pmax - pmin, pmin); };
  if (!have_p) {
    sw_announce(x, 10, scan_point(lane), true);
    const double f = sw_scores<10>(x);
    if (w0) {
      double best_f = INFINITY;
#pragma unroll
      for (int k = 0; k < 10; ++k) {
        const double fk = __shfl_sync(~0u, f, k);
        if (k == 0 || fk < best_f) { best_f = fk; p = scan_point(k); }
      }
    }
  }
  Lb1 lb;
  lb.done = false;
  if (w0) lb_init(lb, p, pmin, pmax);
  for (int ev = 0; ev < kLbMaxEvals; ++ev) {
    double xt = 0.0, xs = 0.0;
    if (w0) {
      xt = lb.xt;
      xs = lb_fd_point(xt, pmin, pmax);
    }
    sw_announce(x, 2, lane == 0 ? xt : xs, !lb.done);
    if (!x.sh->go) break;
    const double f2 = sw_scores<2>(x);
    if (w0) {
      const double f = __shfl_sync(~0u, f2, 0), fh = __shfl_sync(~0u, f2, 1);
      lb_feed(lb, f, (fh - f) / (xs - xt));
    }
  }
  return w0 ? lb.x : p;
}

__global__ void __launch_bounds__(kSwThreads)
k_smoothn_weighted(int m, int n, int c, const double* u_in, const double* v_in, double* u_out, double* v_out,
                   const uint8_t* __restrict__ mask, double fixed_p, int is_auto, double pmin, double pmax,
                   const float2* cm2, const float2* cn2, const float2* cnt2, const double* __restrict__ lam2,
                   unsigned char* scratch, size_t pair_bytes, double* p_out, int* flags) {
  __shared__ SwShared sh;
  const int pair = blockIdx.x / c, mn = m * n, tid = threadIdx.x;
  double* base = reinterpret_cast<double*>(scratch + pair_bytes * pair);
  SwCtx x;
  x.m = m; x.n = n; x.mn = mn; x.c = c; x.rank = c > 1 ? (int)cluster_rank() : 0; x.par = 0;
  x.cm = cm2; x.cn = cn2; x.cnt = cnt2; x.lam2 = lam2;
  x.f = base; x.z = base + 2 * mn; x.zo = base + 4 * mn; x.fd = base + 6 * mn; x.tmp = base + 8 * mn;
  x.w = base + 10 * mn; x.sh = &sh;
  int* near = reinterpret_cast<int*>(base + 11 * mn);
  const int rows = (2 * m + c - 1) / c;
  x.e0 = min(x.rank * rows, 2 * m) * n;
  x.e1 = min((x.rank + 1) * rows, 2 * m) * n;
  const int vtn = kVT / c;
  const int vt = tid < vtn ? x.rank * vtn + tid : 0x7fffffff;
  const int gt = x.rank * kSwThreads + tid, gn = c * kSwThreads;  // thread of the cluster
  const long long off = (long long)pair * mn;
  // Fields, finite mask and weights.
  double nf = 0.0, ws = 0.0;
  for (int e = vt; e < mn; e += kVT) {
    const double a = u_in[off + e], b = v_in[off + e];
    const bool fin = isfinite(a) && isfinite(b);
    x.f[e] = a;
    x.f[mn + e] = b;
    const double wv = (fin && !(mask && mask[e])) ? 1.0 : 0.0;
    x.w[e] = wv;
    nf += fin ? 1.0 : 0.0;
    ws += wv;
  }
  cluster_barrier(c);  // every CTA of the cluster runs
  sw_sums(x, nf, ws);
  nf = sh.sums[0];
  ws = sh.sums[1];
  x.n_finite = nf;
  x.w_mean = ws / (double)mn;
  const bool weighted = ws != (double)mn;
  // Nearest finite neighbour of the missing points: first the nearest finite
  // row in every column (ties: the lower row), then the nearest column.
  if (nf < (double)mn && nf > 0) {
    for (int col = gt; col < n; col += gn) {
      int last = -1;
      for (int y = 0; y < m; ++y) {
        if (isfinite(x.f[y * n + col]) && isfinite(x.f[mn + y * n + col])) last = y;
        near[y * n + col] = last;
      }
      int next = -1;
      for (int y = m - 1; y >= 0; --y) {
        if (isfinite(x.f[y * n + col]) && isfinite(x.f[mn + y * n + col])) next = y;
        const int up = near[y * n + col];
        int r = up;
        if (up < 0 || (next >= 0 && next - y < y - up)) r = next;
        near[y * n + col] = r;
      }
    }
    cluster_barrier(c);
    for (int e = gt; e < mn; e += gn) {
      if (isfinite(x.f[e]) && isfinite(x.f[mn + e])) continue;
      const int y = e / n, xx = e % n;
      long long best = -1;
      int br = 0, bc = 0;
      for (int col = 0; col < n; ++col) {
        const int r = near[y * n + col];
        if (r < 0) continue;
        const long long d = (long long)(col - xx) * (col - xx) + (long long)(r - y) * (r - y);
        if (best < 0 || d < best) { best = d; br = r; bc = col; }
      }
      x.zo[e] = x.f[br * n + bc];
      x.zo[mn + e] = x.f[mn + br * n + bc];
    }
    cluster_barrier(c);
    for (int e = gt; e < mn; e += gn) {
      if (isfinite(x.f[e]) && isfinite(x.f[mn + e])) continue;
      x.f[e] = x.zo[e];
      x.f[mn + e] = x.zo[mn + e];
    }
    cluster_barrier(c);
  }
  // Start: the low DCT coefficients of f (one trailing block cleared), or 0.
  const int n0 = (m + 9) / 10 + 1, n1 = (n + 9) / 10 + 1;
  if (weighted) {
    sw_row_pass(x, false, [&](int e) { return x.f[e]; }, reinterpret_cast<float2*>(x.zo),
                reinterpret_cast<float2*>(x.tmp));
    cluster_barrier(c);
    sw_col_pass(x, false, reinterpret_cast<const float2*>(x.tmp), [&](int e, double v) {
      const int q = e >= mn ? e - mn : e;
      x.z[e] = (q / n >= n0 && q % n >= n1) ? 0.0 : v;
    });
    sw_row_pass(x, true, [&](int e) { return x.z[e]; }, reinterpret_cast<float2*>(x.zo),
                reinterpret_cast<float2*>(x.fd));
    cluster_barrier(c);
    sw_col_pass(x, true, reinterpret_cast<const float2*>(x.fd), [&](int e, double v) { x.z[e] = v; });
  } else {
    for (int e = x.e0 + tid; e < x.e1; e += kSwThreads) x.z[e] = 0.0;
  }
  const double rf = weighted ? 1.75 : 1.0;
  double p = fixed_p;
  bool have_p = !is_auto;
  if (have_p) sw_announce(x, 1, p, true);
  int k_last = 0;  // index of the last iteration run
  for (int k = 0; k < 100; ++k) {
    k_last = k;
    sw_row_pass(x, false,
                [&](int e) {
                  const double wv = x.w[e >= mn ? e - mn : e];
                  return wv * (x.f[e] - x.z[e]) + x.z[e];
                },
                reinterpret_cast<float2*>(x.zo), reinterpret_cast<float2*>(x.tmp));
    cluster_barrier(c);
    sw_col_pass(x, false, reinterpret_cast<const float2*>(x.tmp), [&](int e, double v) { x.fd[e] = v; });
    if (is_auto && ((k + 1) & k) == 0) {
      cluster_barrier(c);  // the scores read every row of fd
      p = sw_search(x, p, have_p, pmin, pmax);
      have_p = true;
      sw_announce(x, 1, p, true);
      cluster_barrier(c);  // fd is rewritten below
    }
    const double s = sh.s[0];
    // The inverse row pass takes the rows of fd that this CTA just wrote and
    // leaves its (hi, lo) results in their place.
    sw_row_pass(x, true, [&](int e) { return __dmul_rn(x.fd[e], rcp_fast(1.0 + s * lam2[e >= mn ? e - mn : e])); },
                reinterpret_cast<float2*>(x.zo), reinterpret_cast<float2*>(x.fd));
    cluster_barrier(c);
    sw_col_pass(x, true, reinterpret_cast<const float2*>(x.fd),
                [&](int e, double v) { x.zo[e] = fma(1.0 - rf, x.z[e], __dmul_rn(rf, v)); });
    cluster_barrier(c);
    double num = 0.0, den = 0.0;
    for (int fi = 0; fi < 2; ++fi)
      for (int e = vt; e < mn; e += kVT) {
        const double z0 = x.z[fi * mn + e], z1 = x.zo[fi * mn + e];
        num += (z0 - z1) * (z0 - z1);
        den += z1 * z1;
      }
    sw_sums(x, num, den);
    double* t = x.z;
    x.z = x.zo;
    x.zo = t;
    if (tid == 0) {
      const double tol = weighted ? sqrt(sh.sums[0]) / (sqrt(sh.sums[1]) + 1e-6) : 0.0;
      sh.go = tol > 1e-3 || isnan(tol);
    }
    __syncthreads();
    if (!sh.go) break;
  }
  for (int e = x.e0 + tid; e < x.e1; e += kSwThreads) {
    const int fi = e >= mn ? 1 : 0, q = e - fi * mn;
    (fi ? v_out : u_out)[off + q] = (mask && mask[q]) ? 0.0 : x.z[e];
  }
  if (x.rank == 0 && tid == 0) {
    if (p_out) p_out[pair] = p;
    if (flags) flags[pair] = smooth_flags(is_auto != 0, p, pmin, pmax, k_last == 99);
  }
}

static int smoothn_weighted(int m, int n, int n_pairs, const double* u_in, const double* v_in, double* u_out,
                            double* v_out, const uint8_t* field_mask, double s, double* p_out, void* scratch,
                            cudaStream_t stream, int* flags, const void* tables) {
  const size_t mn = (size_t)m * n;
  // Scratch: room of m^2 and n^2 doubles, lambda^2, n_pairs doubles, the
  // matrices as float pairs, then the pairs' blocks.
  char* p = (char*)scratch;
  p += align_up((size_t)m * m * 8);
  float2* cnt2 = (float2*)p; p += align_up((size_t)n * n * 8);
  double* lam2 = (double*)p; p += align_up(mn * 8);
  p += align_up((size_t)n_pairs * 8);
  float2* cm2 = (float2*)p;
  float2* cn2 = cm2 + (size_t)m * m;
  p += weighted_matrix_bytes(m, n);
  SmoothTables t{};
  if (tables) {
    t = kept_tables(tables, m, n);
  } else {
    t.cm2 = cm2; t.cn2 = cn2; t.cnt2 = cnt2; t.lam2 = lam2;
    share_square(m, n, t);
    const int rc = build_tables(m, n, t, stream);
    if (rc) return rc;
  }
  const bool is_auto = !(s > 0);
  double pmin = 0, pmax = 0;
  if (is_auto) gcv_bounds(m, n, &pmin, &pmax);
  const int c = cluster_size(n_pairs);
  return launch_cluster(k_smoothn_weighted, n_pairs, c, kSwThreads, stream, "k_smoothn_weighted", m, n, c, u_in, v_in,
                        u_out, v_out, field_mask, is_auto ? 0.0 : log10(s), is_auto ? 1 : 0, pmin, pmax, t.cm2, t.cn2,
                        t.cnt2, t.lam2, (unsigned char*)p, weighted_pair_bytes(mn), p_out, flags);
}

int smoothn(int m, int n, int n_pairs, const double* u_in, const double* v_in, double* u_out, double* v_out,
            const uint8_t* field_mask, double s, double* p_out, void* scratch, cudaStream_t stream, int* flags,
            const void* tables) {
  const long long mn = (long long)m * n;
  if (n_pairs == 0 || mn == 0) return PIV_OK;
  if (flags && (mn < 2 || (!field_mask && s > 0))) cudaMemsetAsync(flags, 0, sizeof(int) * n_pairs, stream);
  if (mn < 2) {
    cudaMemcpyAsync(u_out, u_in, mn * n_pairs * 8, cudaMemcpyDeviceToDevice, stream);
    cudaMemcpyAsync(v_out, v_in, mn * n_pairs * 8, cudaMemcpyDeviceToDevice, stream);
    return check("smoothn copy");
  }
  if (field_mask)
    return smoothn_weighted(m, n, n_pairs, u_in, v_in, u_out, v_out, field_mask, s, p_out, scratch, stream, flags,
                            tables);
  if (n_pairs > 65535) return set_error(PIV_E_UNSUPPORTED, "smoothn: more than 65535 pairs in one call");
  SmoothScratch sc = carve(scratch, m, n, n_pairs);
  if (tables) {
    sc.t = kept_tables(tables, m, n);
  } else {
    PIV_RC(build_tables(m, n, sc.t, stream));
  }
  const DctIo in{const_cast<double*>(u_in), const_cast<double*>(v_in), mn}, result{u_out, v_out, mn};
  const DctIo fd{sc.fd, sc.fd + mn, 2 * mn}, tmp{sc.tmp, sc.tmp + mn, 2 * mn};
  const DctGamma none{nullptr, nullptr, 0.0};
  DctGamma gam{sc.t.lam2, sc.s, 0.0};
  // Forward DCT-II: rows, then columns.
  PIV_RC(dct_pass<false>(m, n, 2 * n_pairs, 0, sc.t, in, tmp, none, stream));
  PIV_RC(dct_pass<false>(m, n, 2 * n_pairs, 1, sc.t, tmp, fd, none, stream));
  if (!(s > 0)) {
    double pmin = 0, pmax = 0;
    gcv_bounds(m, n, &pmin, &pmax);
    const int c = cluster_size(n_pairs);
    auto search = c == 8 ? k_gcv<2> : k_gcv<1>;
    PIV_RC(launch_cluster(search, n_pairs, c, c == 8 ? 2 * kVT / c : kVT / c, stream, "k_gcv", m, n, c,
                          1.0 / (double)mn, sc.fd, sc.f2, sc.f2f, sc.t.lam2, sc.t.lam2f, pmin, pmax, p_out, sc.s,
                          flags));
  } else {
    gam.s = nullptr;
    gam.given = pow(10.0, log10(s));
    if (p_out) k_fill<<<(n_pairs + 127) / 128, 128, 0, stream>>>(n_pairs, log10(s), p_out);
    PIV_RC(check("k_fill"));
  }
  // Inverse DCT (DCT-III): rows, their inputs scaled by 1 / (1 + s lambda^2),
  // then columns.
  PIV_RC(dct_pass<true>(m, n, 2 * n_pairs, 0, sc.t, fd, tmp, gam, stream));
  return dct_pass<true>(m, n, 2 * n_pairs, 1, sc.t, tmp, result, none, stream);
}

}  // namespace piv

namespace piv {

// ---------------------------------------------------------------------------
// smoothn without device allocation.
//
// Some callers cannot allocate device memory while they run: a host that
// hands this library a fixed memory budget at start-up, a real-time loop that
// must not stall in the allocator, or a framework that owns every device
// allocation itself. piv_smoothn_noalloc serves them with scratch that lives
// in a fixed device array of this file, sized for modest fields. Every GPU
// that loads the library holds the array until the process exits.
// ---------------------------------------------------------------------------
// 4 MiB: e.g. 4 pairs of 128 x 128 fields, or with a field mask 2 pairs of
// 127 x 127 (the weighted path keeps more per pair).
static constexpr size_t kNoAllocScratchBytes = 4u << 20;
static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

// Device address of g_noalloc_scratch in the current context. In host code
// the array's name is only a host-side stand-in, never a device address. The
// address is looked up on every call made outside stream capture (so a call
// after a device reset, which reloads the module at a new address, gets the
// new one) and remembered per device for calls made while `stream` is being
// captured, which reuse the address of the device's last uncaptured call.
static void* noalloc_scratch_address(cudaStream_t stream, int* rc) {
  static std::mutex mu;
  static void* addr[64] = {nullptr};
  int dev = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess) {
    *rc = set_cuda_error(e, "cudaGetDevice");
    return nullptr;
  }
  if (dev < 0 || dev >= 64) {
    *rc = set_error(PIV_E_UNSUPPORTED, "device index %d out of range", dev);
    return nullptr;
  }
  cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
  e = cudaStreamIsCapturing(stream, &cap);
  if (e != cudaSuccess) {
    *rc = set_cuda_error(e, "cudaStreamIsCapturing");
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (cap != cudaStreamCaptureStatusNone) {
    if (!addr[dev]) {
      *rc = set_error(PIV_E_ARG,
                      "piv_smoothn_noalloc: the first call on device %d must come before any stream capture", dev);
      return nullptr;
    }
  } else {
    void* p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      *rc = set_cuda_error(e, "cudaGetSymbolAddress(g_noalloc_scratch)");
      return nullptr;
    }
    addr[dev] = p;
  }
  *rc = PIV_OK;
  return addr[dev];
}

}  // namespace piv

extern "C" int piv_smoothn_noalloc(int m, int n, int n_pairs, double* u, double* v, const uint8_t* field_mask,
                                   double s, double* p_out, void* stream) {
  using namespace piv;
  if (!u || !v) return set_error(PIV_E_ARG, "NULL argument");
  if (m <= 0 || n <= 0 || n_pairs <= 0) return set_error(PIV_E_ARG, "empty field (m=%d, n=%d, pairs=%d)", m, n, n_pairs);
  // The kernels index with 32-bit products m n, m m and n n and launch one
  // block row per pair: refuse shapes beyond those before sizing the scratch
  // (whose 64-bit byte counts then cannot wrap).
  const long long lim = 1LL << 31;
  if ((long long)m * n >= lim || (long long)m * m >= lim || (long long)n * n >= lim || n_pairs > 65535)
    return set_error(PIV_E_ARG, "piv_smoothn_noalloc: field %d x %d with %d pair(s) is beyond the kernels' limits",
                     m, n, n_pairs);
  const bool weighted = field_mask != nullptr && (long long)m * n >= 2;
  const size_t need = smoothn_scratch_bytes_path(m, n, n_pairs, weighted);
  if (need > kNoAllocScratchBytes)
    return set_error(PIV_E_ARG,
                     "piv_smoothn_noalloc: %d pair(s) of %d x %d %sfields need %zu bytes of scratch, more than its "
                     "fixed %zu bytes; use piv_smoothn or fewer/smaller fields",
                     n_pairs, m, n, weighted ? "masked " : "", need, kNoAllocScratchBytes);
  int rc = PIV_OK;
  void* scratch = noalloc_scratch_address((cudaStream_t)stream, &rc);
  if (!scratch) return rc;
  return smoothn(m, n, n_pairs, u, v, u, v, field_mask, s, p_out, scratch, (cudaStream_t)stream);
}
