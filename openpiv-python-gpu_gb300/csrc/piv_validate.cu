// Outlier validation and replacement on the device.
//
// Validation restates ValidationGPU (gpu_validation.py:80-243): local median,
// MAD and mean of the (2s+1)^2 neighbourhood without its centre (NaN padding
// and NaN values skipped), global mean/std for the RMS test, S2N threshold;
// the selected tests are OR-ed, then points excluded by the mask are cleared.
// Comparisons use strict '>' (or '<' for S2N) like the reference.
//
// Replacement restates PIVGPU.replace_outliers (gpu_process.py:788-834) and
// ReplacementGPU (gpu_validation.py:245-415) with one CTA per field pair:
// spring (the reference builds a sparse linear system and calls spsolve; here
// the same system, scaled to its symmetric form, is solved by conjugate
// gradients in float64), local median or local mean replacement, optional
// revalidation of the replaced points, and reset of unresolved points.
//
// `fp32` selects float32 arithmetic, which the reference uses for fields that
// have not been through smoothn yet (dtype_f float32, first iteration); the
// field arrays are float64 throughout and hold float32 values in that mode.
#include <math.h>

#include "piv_common.cuh"
#include "piv_internal.h"

namespace piv {

static constexpr int kMaxKernel = 7;                       // validation/replacement size <= 3
static constexpr int kMaxNbrs = kMaxKernel * kMaxKernel;   // values incl. centre

template <typename T>
PIV_D void sort_small(T* a, int n) {
  for (int i = 1; i < n; ++i) {
    T v = a[i];
    int j = i - 1;
    while (j >= 0 && a[j] > v) { a[j + 1] = a[j]; --j; }
    a[j + 1] = v;
  }
}

// nanmedian of n finite values (sorted in place): middle value, or the mean of
// the two middle values as (lo + hi) / 2 (numpy.ma.median); NaN when n == 0.
template <typename T>
PIV_D T median_of(T* a, int n) {
  if (n == 0) return (T)NAN;
  sort_small(a, n);
  const T lo = a[(n - 1) / 2], hi = a[n / 2];
  return mul_rn(add_rn(lo, hi), (T)0.5);  // exact: the same value as the division by 2
}

// numpy's pairwise summation (n <= 128 branch) of n values.
template <typename T>
PIV_D T pairwise_sum(const T* a, int n) {
  if (n < 8) {
    T r = (T)0;
    for (int i = 0; i < n; ++i) r = add_rn(r, a[i]);
    return r;
  }
  T r[8];
#pragma unroll
  for (int j = 0; j < 8; ++j) r[j] = a[j];
  int i = 8;
  for (; i < n - (n % 8); i += 8) {
#pragma unroll
    for (int j = 0; j < 8; ++j) r[j] = add_rn(r[j], a[i + j]);
  }
  T res = add_rn(add_rn(add_rn(r[0], r[1]), add_rn(r[2], r[3])), add_rn(add_rn(r[4], r[5]), add_rn(r[6], r[7])));
  for (; i < n; ++i) res = add_rn(res, a[i]);
  return res;
}

template <typename T>
PIV_D T as_t(double v) { return (T)v; }

// Field value at (i, j) with NaN outside the field; `sub` replaces the value at
// points flagged in `subst` (outliers) by `sub_val` when non-null.
struct FieldView {
  const double* f;
  int m, n;
  const uint8_t* subst;  // may be null
  double sub_val;        // NaN or 0
};

template <typename T>
PIV_D T fv_at(const FieldView& v, int i, int j) {
  if (i < 0 || i >= v.m || j < 0 || j >= v.n) return (T)NAN;
  const int p = i * v.n + j;
  if (v.subst && v.subst[p]) return (T)v.sub_val;
  return (T)v.f[p];
}

// Order-preserving integer keys: signed comparison of the keys orders the
// values like the floating-point comparison (-0 sorts below +0). The sorting
// network then runs on the integer ALUs; float64 min/max are slow here.
PIV_D int sort_key(float v) {
  const int b = __float_as_int(v);
  return b ^ ((b >> 31) & 0x7fffffff);
}
PIV_D long long sort_key(double v) {
  const long long b = __double_as_longlong(v);
  return b ^ ((b >> 63) & 0x7fffffffffffffffLL);
}
PIV_D float key_value(int k) { return __int_as_float(k ^ ((k >> 31) & 0x7fffffff)); }
PIV_D double key_value(long long k) { return __longlong_as_double(k ^ ((k >> 63) & 0x7fffffffffffffffLL)); }

// Median (kind 0) or MAD (kind 2, |v - med|) of the eight neighbours of (i, j)
// in registers: missing values sort last as +inf, a 19-comparator network
// (Batcher's odd-even merge) sorts their keys, and the middle pair of the cnt
// valid values is picked by selects. Same result as median_of on the valid
// values.
template <typename T>
PIV_D T median8(const FieldView& fv, int i, int j, int kind, T med) {
  using K = decltype(sort_key(T(0)));
  K a[8];
  int cnt = 0, k = 0;
#pragma unroll
  for (int di = -1; di <= 1; ++di)
#pragma unroll
    for (int dj = -1; dj <= 1; ++dj) {
      if (di == 0 && dj == 0) continue;
      T v = fv_at<T>(fv, i + di, j + dj);
      const bool ok = !is_nan(v);
      if (kind == 2) v = fabs(sub_rn(v, med));
      a[k++] = sort_key(ok ? v : (T)INFINITY);
      cnt += ok ? 1 : 0;
    }
  auto cx = [&](int x, int y) {
    const K lo = min(a[x], a[y]), hi = max(a[x], a[y]);
    a[x] = lo;
    a[y] = hi;
  };
  cx(0, 1); cx(2, 3); cx(4, 5); cx(6, 7);
  cx(0, 2); cx(1, 3); cx(4, 6); cx(5, 7);
  cx(1, 2); cx(5, 6);
  cx(0, 4); cx(1, 5); cx(2, 6); cx(3, 7);
  cx(2, 4); cx(3, 5);
  cx(1, 2); cx(3, 4); cx(5, 6);
  if (cnt == 0) return (T)NAN;
  const int il = (cnt - 1) / 2, ih = cnt / 2;
  K lo = a[0], hi = a[0];
#pragma unroll
  for (int q = 1; q < 8; ++q) {
    lo = il == q ? a[q] : lo;
    hi = ih == q ? a[q] : hi;
  }
  return mul_rn(add_rn(key_value(lo), key_value(hi)), (T)0.5);  // exact: the same value as the division by 2
}

// Neighbourhood statistics at (i, j): kind 0 median, 1 mean, 2 MAD (needs med).
template <typename T>
PIV_D T nbr_stat(const FieldView& fv, int i, int j, int s, int kind, T med) {
  if (s == 1 && kind != 1) return median8<T>(fv, i, j, kind, med);
  T vals[kMaxNbrs];
  const int k = 2 * s + 1;
  if (kind == 1) {
    // nanmean over the whole (2s+1)^2 kernel with the centre NaN: pairwise sum
    // of the kernel in row-major order with NaN -> 0, divided by the count.
    int cnt = 0;
    for (int di = 0; di < k; ++di)
      for (int dj = 0; dj < k; ++dj) {
        T v = (di == s && dj == s) ? (T)NAN : fv_at<T>(fv, i + di - s, j + dj - s);
        if (is_nan(v)) v = (T)0; else ++cnt;
        vals[di * k + dj] = v;
      }
    const T sum = pairwise_sum(vals, k * k);
    return cnt ? div_rn(sum, (T)cnt) : (T)NAN;
  }
  int cnt = 0;
  for (int di = -s; di <= s; ++di)
    for (int dj = -s; dj <= s; ++dj) {
      if (di == 0 && dj == 0) continue;
      T v = fv_at<T>(fv, i + di, j + dj);
      if (is_nan(v)) continue;
      vals[cnt++] = kind == 2 ? fabs(sub_rn(v, med)) : v;
    }
  return median_of(vals, cnt);
}

struct ValSettings {
  int size;
  double s2n_tol, median_tol, mad_tol, mean_tol, rms_tol;
  int fp32;
  const void* s2n;
  int s2n_dtype;
};

// Outlier test of point p of one pair. rms: {mean_u, std_u, mean_v, std_v}.
template <typename T>
PIV_D bool point_invalid(const ValSettings& s, const FieldView& fu, const FieldView& fv, long long s2n_index, int i,
                         int j, const double* rms) {
  const int p = i * fu.n + j;
  const T u = (T)fu.f[p], v = (T)fv.f[p];
  bool out = false;
  if (!isnan(s.s2n_tol) && s.s2n) {
    if (s.s2n_dtype == PIV_DTYPE_F64) out |= ((const double*)s.s2n)[s2n_index] < s.s2n_tol;
    else out |= ((const float*)s.s2n)[s2n_index] < (float)s.s2n_tol;
  }
  T mu = (T)NAN, mv = (T)NAN;
  const bool need_med = !isnan(s.median_tol) || !isnan(s.mad_tol);
  if (need_med) {
    mu = nbr_stat<T>(fu, i, j, s.size, 0, (T)0);
    mv = nbr_stat<T>(fv, i, j, s.size, 0, (T)0);
  }
  if (!isnan(s.median_tol)) {
    const T tol = (T)s.median_tol;
    out |= fabs(sub_rn(u, mu)) > tol || fabs(sub_rn(v, mv)) > tol;
  }
  if (!isnan(s.mad_tol)) {
    const T tol = (T)s.mad_tol;
    const T du = nbr_stat<T>(fu, i, j, s.size, 2, mu), dv = nbr_stat<T>(fv, i, j, s.size, 2, mv);
    out |= fabs(sub_rn(u, mu)) > mul_rn(tol, du) || fabs(sub_rn(v, mv)) > mul_rn(tol, dv);
  }
  if (!isnan(s.mean_tol)) {
    const T tol = (T)s.mean_tol;
    const T au = nbr_stat<T>(fu, i, j, s.size, 1, (T)0), av = nbr_stat<T>(fv, i, j, s.size, 1, (T)0);
    out |= fabs(sub_rn(u, au)) > tol || fabs(sub_rn(v, av)) > tol;
  }
  if (!isnan(s.rms_tol) && rms) {
    const T tol = (T)s.rms_tol;
    out |= fabs(sub_rn(u, (T)rms[0])) > mul_rn(tol, (T)rms[1]) || fabs(sub_rn(v, (T)rms[2])) > mul_rn(tol, (T)rms[3]);
  }
  return out;
}

// Per-pair nanmean / nanstd of u and v (RMS test), one CTA per pair.
template <typename T>
__global__ void k_field_stats(int m, int n, const double* __restrict__ u, const double* __restrict__ v, double* out) {
  __shared__ double red[3][32];
  const int pair = blockIdx.x;
  const long long off = (long long)pair * m * n;
  for (int f = 0; f < 2; ++f) {
    const double* x = (f == 0 ? u : v) + off;
    T s = 0;
    int c = 0;
    for (int p = threadIdx.x; p < m * n; p += blockDim.x) {
      const T val = (T)x[p];
      if (!is_nan(val)) { s += val; ++c; }
    }
    for (int o = 16; o > 0; o >>= 1) { s += __shfl_xor_sync(~0u, s, o); c += __shfl_xor_sync(~0u, c, o); }
    if ((threadIdx.x & 31) == 0) { red[0][threadIdx.x >> 5] = (double)s; red[1][threadIdx.x >> 5] = c; }
    __syncthreads();
    __shared__ double mean_s, cnt_s;
    if (threadIdx.x == 0) {
      T ts = 0;
      double tc = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) { ts += (T)red[0][w]; tc += red[1][w]; }
      mean_s = tc > 0 ? (double)(ts / (T)tc) : NAN;
      cnt_s = tc;
    }
    __syncthreads();
    const T mean = (T)mean_s;
    T q = 0;
    for (int p = threadIdx.x; p < m * n; p += blockDim.x) {
      const T val = (T)x[p];
      if (!is_nan(val)) { const T d = val - mean; q += d * d; }
    }
    for (int o = 16; o > 0; o >>= 1) q += __shfl_xor_sync(~0u, q, o);
    if ((threadIdx.x & 31) == 0) red[2][threadIdx.x >> 5] = (double)q;
    __syncthreads();
    if (threadIdx.x == 0) {
      T tq = 0;
      for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tq += (T)red[2][w];
      out[pair * 4 + 2 * f] = mean_s;
      out[pair * 4 + 2 * f + 1] = cnt_s > 0 ? (double)sqrt(tq / (T)cnt_s) : NAN;
    }
    __syncthreads();
  }
}

// val2 (may be NULL) receives a copy of val.
template <typename T>
__global__ void k_validate(ValArgs a, uint8_t* __restrict__ val, uint8_t* __restrict__ val2,
                           const double* __restrict__ rms) {
  const long long npts = (long long)a.m * a.n;
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= npts * a.n_pairs) return;
  const int pair = (int)(t / npts);
  const int p = (int)(t % npts);
  if ((a.field_mask && a.field_mask[p]) || (a.exclude && a.exclude[t])) {
    val[t] = 0;
    if (val2) val2[t] = 0;
    return;
  }
  const long long off = (long long)pair * npts;
  FieldView fu{a.u + off, a.m, a.n, nullptr, 0.0}, fv{a.v + off, a.m, a.n, nullptr, 0.0};
  ValSettings s{a.size, a.s2n_tol, a.median_tol, a.mad_tol, a.mean_tol, a.rms_tol, a.fp32, a.s2n, a.s2n_dtype};
  const uint8_t bad = point_invalid<T>(s, fu, fv, t, p / a.n, p % a.n, rms ? rms + pair * 4 : nullptr) ? 1 : 0;
  val[t] = bad;
  if (val2) val2[t] = bad;
}

int validate(const ValArgs& a, uint8_t* val, double* rms_stats, cudaStream_t stream, uint8_t* val2) {
  if (a.size > 3 || a.size < 1) return set_error(PIV_E_UNSUPPORTED, "validation_size %d (supported: 1..3)", a.size);
  const long long total = (long long)a.m * a.n * a.n_pairs;
  if (total == 0) return PIV_OK;
  const double* rms = nullptr;
  if (!isnan(a.rms_tol)) {
    if (!rms_stats) return set_error(PIV_E_ARG, "RMS validation needs a statistics buffer");
    if (a.fp32) k_field_stats<float><<<a.n_pairs, 256, 0, stream>>>(a.m, a.n, a.u, a.v, rms_stats);
    else k_field_stats<double><<<a.n_pairs, 256, 0, stream>>>(a.m, a.n, a.u, a.v, rms_stats);
    rms = rms_stats;
  }
  const int bs = 128;
  const unsigned grid = (unsigned)((total + bs - 1) / bs);
  if (a.fp32) k_validate<float><<<grid, bs, 0, stream>>>(a, val, val2, rms);
  else k_validate<double><<<grid, bs, 0, stream>>>(a, val, val2, rms);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_validate launch");
}

// ---------------------------------------------------------------------------
// Field combination u = u_corr (+ up).
// ---------------------------------------------------------------------------
__global__ void k_combine(long long count, const void* uc, const void* vc, int corr_dtype, const double* up,
                          const double* vp, double* u, double* v) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  double a, b;
  if (corr_dtype == PIV_DTYPE_F64) { a = ((const double*)uc)[t]; b = ((const double*)vc)[t]; }
  else { a = (double)((const float*)uc)[t]; b = (double)((const float*)vc)[t]; }
  if (up) { a = __dadd_rn(a, up[t]); b = __dadd_rn(b, vp[t]); }
  u[t] = a;
  v[t] = b;
}

int combine_fields(int count, const void* u_corr, const void* v_corr, int corr_dtype, const double* up,
                   const double* vp, int fp32, double* u, double* v, cudaStream_t stream) {
  (void)fp32;
  if (count == 0) return PIV_OK;
  k_combine<<<(count + 255) / 256, 256, 0, stream>>>(count, u_corr, v_corr, corr_dtype, up, vp, u, v);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_combine launch");
}

// (u * scaling) / dt in the field's float type.
__global__ void k_scale(long long count, const double* u, const double* v, double scaling, double dt, int fp32,
                        double* uo, double* vo) {
  const long long t = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= count) return;
  if (fp32) {
    uo[t] = (double)__fdiv_rn(__fmul_rn((float)u[t], (float)scaling), (float)dt);
    vo[t] = (double)__fdiv_rn(__fmul_rn((float)v[t], (float)scaling), (float)dt);
  } else {
    uo[t] = __ddiv_rn(__dmul_rn(u[t], scaling), dt);
    vo[t] = __ddiv_rn(__dmul_rn(v[t], scaling), dt);
  }
}

int scale_fields(int count, const double* u, const double* v, double scaling, double dt, int fp32, double* uo,
                 double* vo, cudaStream_t stream) {
  if (count == 0) return PIV_OK;
  k_scale<<<(count + 255) / 256, 256, 0, stream>>>(count, u, v, scaling, dt, fp32, uo, vo);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_scale launch");
}

// ---------------------------------------------------------------------------
// Replacement: one CTA per pair, bound by the float64 units of its SM and by
// latency; work per flagged point, and one read of the mask per iteration to
// list them. Measured: 64 pairs of a three-pass 1024 x 1024 run (3 to 80
// outliers per pair and pass) 335 -> 190 us for the three passes, one 253 x
// 253 field with 2,560 outliers 900 -> 184 us.
// ---------------------------------------------------------------------------
static constexpr int kRepThreads = 512;
static constexpr int kCgMaxIters = 20000;
// Up to kCgSmall outliers per pair, the conjugate-gradient vectors stay in
// registers (kCgPer per thread) and the search direction in shared memory.
static constexpr int kCgPer = 4;
static constexpr int kCgSmall = kRepThreads * kCgPer;

struct RepScratch {
  double* init_u;   // [mn]
  double* init_v;
  double* new_u;    // [mn] replacement values by outlier rank
  double* new_v;
  double* cg;       // 8 * [mn]: x_u, x_v, r_u, r_v, p_u, p_v, q_u, q_v
  double* dinv;     // [mn] spring row scale 1/c_r by outlier rank
  int* nbr;         // 4 * [mn] outlier ranks of the linked neighbours (-1: none)
  int* list;        // [mn] outlier positions
  int* rank;        // [mn] position -> outlier rank or -1
  uint8_t* flag;    // [mn] anchored / scratch flags
};

// Bytes of one pair's replacement scratch, rounded up to 256 so that every
// pair's block (and the doubles at its start) stays aligned.
PIV_HD size_t rep_scratch_stride(size_t mn) {
  return ((mn * (13 * sizeof(double) + 6 * sizeof(int) + 1) + 255) / 256) * 256;
}

size_t replace_scratch_bytes(int m, int n, int n_pairs) {
  return rep_scratch_stride((size_t)m * n) * (size_t)n_pairs;
}

static __device__ RepScratch rep_scratch(void* base, int mn, int pair) {
  char* p = (char*)base + rep_scratch_stride((size_t)mn) * pair;
  RepScratch s;
  s.init_u = (double*)p; p += mn * sizeof(double);
  s.init_v = (double*)p; p += mn * sizeof(double);
  s.new_u = (double*)p; p += mn * sizeof(double);
  s.new_v = (double*)p; p += mn * sizeof(double);
  s.cg = (double*)p; p += 8 * (size_t)mn * sizeof(double);
  s.dinv = (double*)p; p += mn * sizeof(double);
  s.nbr = (int*)p; p += 4 * (size_t)mn * sizeof(int);
  s.list = (int*)p; p += mn * sizeof(int);
  s.rank = (int*)p; p += mn * sizeof(int);
  s.flag = (uint8_t*)p;
  return s;
}

// Block-wide sums of two doubles in one reduction (all threads get both). The
// warps' partial sums are combined by a shuffle tree rather than a serial
// chain: the conjugate-gradient loop waits on this twice per iteration.
PIV_D double2 block_sum2(double a, double b, double* red) {
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(~0u, a, o);
    b += __shfl_xor_sync(~0u, b, o);
  }
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31, nw = blockDim.x >> 5;
  __syncthreads();
  if (l == 0) { red[w] = a; red[32 + w] = b; }
  __syncthreads();
  double ta = l < nw ? red[l] : 0.0, tb = l < nw ? red[32 + l] : 0.0;
  for (int o = 16; o > 0; o >>= 1) {
    ta += __shfl_xor_sync(~0u, ta, o);
    tb += __shfl_xor_sync(~0u, tb, o);
  }
  return make_double2(ta, tb);
}

// The first nwa warps of the block: a named barrier (id 1) among them, and
// sums of two doubles over them (every thread of the group gets both). With
// one warp the shuffle tree alone suffices. Float64 throughput on this GPU is
// a small fraction of float32, so work that only the warps holding data need
// is kept off the others.
PIV_D void group_bar(int nwa) {
  if (nwa == 1) __syncwarp();
  else asm volatile("bar.sync 1, %0;" ::"r"(nwa * 32) : "memory");
}

// Warp sums of a (in lanes 0 .. 15) and b (lanes 16 .. 31): the xor tree of a
// full warp sum of each, but one level exchanges the halves, so that one
// instruction stream adds for both. A float64 instruction holds its unit for
// 64 cycles here, whatever the number of lanes.
PIV_D double warp_sum2(double a, double b) {
  const bool up = threadIdx.x & 16;
  double v = (up ? b : a) + __shfl_xor_sync(~0u, up ? a : b, 16);
  for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(~0u, v, o);
  return v;
}

// Publishes a warp's sums of two values in red for warp 0 of the group.
PIV_D void group_put2(double a, double b, double* red, int nwa) {
  const double v = warp_sum2(a, b);
  if ((threadIdx.x & 15) == 0) red[((threadIdx.x & 16) ? 32 : 0) + (threadIdx.x >> 5)] = v;
  group_bar(nwa);
}
// In warp 0: the group's sum of a (lanes 0 .. 15) and of b (lanes 16 .. 31).
PIV_D double group_take2(const double* red, int nwa) {
  const int l = threadIdx.x & 15;
  double t = l < nwa ? red[((threadIdx.x & 16) ? 32 : 0) + l] : 0.0;
  for (int o = 8; o > 0; o >>= 1) t += __shfl_xor_sync(~0u, t, o);
  return t;
}

// Stable compaction of the flagged positions into list (ascending), returns
// their count; rank[p] = place of p in list (flagged positions only). Each
// warp takes a contiguous part of the field, 32 positions at a time, counts
// its flags, and after one scan over the warps places them.
PIV_D int block_compact(const uint8_t* flags, int mn, int* list, int* rank, int* red) {
  const int tid = threadIdx.x, lane = tid & 31, w = tid >> 5, nw = blockDim.x >> 5;
  const int per = ((mn + nw - 1) / nw + 31) / 32 * 32, p0 = w * per, p1 = min(mn, p0 + per);
  int c = 0;
#pragma unroll 8
  for (int p = p0 + lane; p < p1; p += 32) c += flags[p] ? 1 : 0;
  c = __reduce_add_sync(~0u, c);
  if (lane == 0) red[w] = c;
  __syncthreads();
  int pos = 0, total = 0;
  for (int k = 0; k < nw; ++k) {
    if (k < w) pos += red[k];
    total += red[k];
  }
  if (c > 0)
    for (int q = p0; q < p1; q += 32 * 8) {
      unsigned bal[8];
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        const int p = q + 32 * k + lane;
        bal[k] = __ballot_sync(~0u, p < p1 && flags[p]);
      }
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        if ((bal[k] >> lane) & 1u) {
          const int p = q + 32 * k + lane, at = pos + __popc(bal[k] & ((1u << lane) - 1u));
          list[at] = p;
          rank[p] = at;
        }
        pos += __popc(bal[k]);
      }
    }
  __syncthreads();  // list and rank are complete, red is reused by the caller
  return total;
}

// Row scale n_r of the spring link (gpu_validation.py:365-371): the reciprocal
// of the link coefficient 1/2, 1/3 or 1/4 in the link matrix's type. third:
// that of 1/3, formed once (the other coefficients are powers of two).
PIV_D double spring_scale(int i, int j, int m, int n, int s, double third) {
  const bool ei = i < s || i >= m - s, ej = j < s || j >= n - s;
  return (ei && ej) ? 2.0 : ((ei || ej) ? third : 4.0);
}

// Spring right-hand side: mean over the four linked neighbours at distance s,
// outliers counted as 0, NaN and out-of-field ignored (gpu_validation.py:381-394).
template <typename T>
PIV_D T spring_rhs(const FieldView& fv, int i, int j, int s) {
  const int k = 2 * s + 1;
  int cnt = 0;
  T sum;
  if (s == 1) {
    // The pairwise sum of the 3 x 3 kernel, whose other entries are zeros.
    T t = fv_at<T>(fv, i - 1, j), l = fv_at<T>(fv, i, j - 1), r = fv_at<T>(fv, i, j + 1), b = fv_at<T>(fv, i + 1, j);
    cnt = (is_nan(t) ? 0 : 1) + (is_nan(l) ? 0 : 1) + (is_nan(r) ? 0 : 1) + (is_nan(b) ? 0 : 1);
    t = is_nan(t) ? (T)0 : t;
    l = is_nan(l) ? (T)0 : l;
    r = is_nan(r) ? (T)0 : r;
    b = is_nan(b) ? (T)0 : b;
    sum = add_rn(add_rn(add_rn(t, l), add_rn(r, b)), (T)0);
  } else {
    T vals[kMaxNbrs];
    for (int q = 0; q < k * k; ++q) vals[q] = (T)0;
    const int di[4] = {0, s, s, 2 * s}, dj[4] = {s, 0, 2 * s, s};  // top, left, right, bottom (row-major)
    for (int e = 0; e < 4; ++e) {
      T v = fv_at<T>(fv, i + di[e] - s, j + dj[e] - s);
      if (!is_nan(v)) { vals[di[e] * k + dj[e]] = v; ++cnt; }
    }
    sum = pairwise_sum(vals, k * k);
  }
  if (cnt == 3) return div_rn(sum, (T)3);
  return cnt ? mul_rn(sum, cnt == 4 ? (T)0.25 : (cnt == 2 ? (T)0.5 : (T)1)) : (T)NAN;  // exact
}

// Shared memory of cg_small.
struct CgShared {
  double pu[kCgSmall], pv[kCgSmall];  // search direction
  double red[2][64];
  double step[4];  // alpha of u and v, beta of u and v
  int done;        // bit 0: u has converged, bit 1: v
};

// Conjugate gradients on (D - Adj) x = b for both fields, up to kCgSmall rows:
// row tid + k nt in registers (scale dd, right-hand sides in ru and rv,
// neighbour rows nb or -1), the search direction in shared memory. Run by the
// nwa warps that hold rows; warp 0 forms the sums and the scalars (u in lanes
// 0 .. 15, v in lanes 16 .. 31) for all: bound by the float64 units, whose
// work the other warps would repeat. tol: stop where |r|^2 is at most this
// (per half warp as the scalars); negative: 1e-28 of the start's.
PIV_D void cg_small(int nv, int nwa, const double (&dd)[kCgPer], const int (&nb)[kCgPer][4], double (&ru)[kCgPer],
                    double (&rv)[kCgPer], double (&xu)[kCgPer], double (&xv)[kCgPer], CgShared& sh, double tol,
                    int* status) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const bool w0 = tid < 32;
  double rr_u = 0, rr_v = 0;
#pragma unroll
  for (int k = 0; k < kCgPer; ++k) {
    const int r = tid + k * nt;
    xu[k] = xv[k] = 0;
    if (r < nv) {
      sh.pu[r] = ru[k];
      sh.pv[r] = rv[k];
      rr_u += ru[k] * ru[k];
      rr_v += rv[k] * rv[k];
    }
  }
  group_put2(rr_u, rr_v, sh.red[0], nwa);
  double rr = 0;  // warp 0
  bool done = false;
  auto publish_done = [&]() {
    const unsigned d = __ballot_sync(~0u, done);
    if (tid == 0) sh.done = (d & 1u) | ((d >> 15) & 2u);
  };
  if (w0) {
    rr = group_take2(sh.red[0], nwa);
    if (tol < 0) tol = rr * 1e-28;
    done = rr <= tol || rr == 0;
    publish_done();
  }
  group_bar(nwa);
  int iter = 0;
  for (; iter < kCgMaxIters; ++iter) {
    const int d = sh.done;
    if (d == 3) break;
    double qu[kCgPer], qv[kCgPer], pq_u = 0, pq_v = 0;
#pragma unroll
    for (int k = 0; k < kCgPer; ++k) {
      const int r = tid + k * nt;
      qu[k] = qv[k] = 0;
      if (r < nv) {
        // The first neighbour's subtraction is fused with the product.
        const int q0 = nb[k][0];
        double au = q0 >= 0 ? fma(dd[k], sh.pu[r], -sh.pu[q0]) : dd[k] * sh.pu[r];
        double av = q0 >= 0 ? fma(dd[k], sh.pv[r], -sh.pv[q0]) : dd[k] * sh.pv[r];
#pragma unroll
        for (int e = 1; e < 4; ++e) {
          const int q = nb[k][e];
          if (q >= 0) { au = __dsub_rn(au, sh.pu[q]); av = __dsub_rn(av, sh.pv[q]); }
        }
        qu[k] = au; qv[k] = av;
        pq_u += sh.pu[r] * au; pq_v += sh.pv[r] * av;
      }
    }
    group_put2(pq_u, pq_v, sh.red[0], nwa);
    if (w0) {
      const double pq = group_take2(sh.red[0], nwa);
      const double al = done ? 0.0 : rr / pq;
      if ((tid & 15) == 0) sh.step[tid >> 4] = al;
    }
    group_bar(nwa);
    const double al_u = sh.step[0], al_v = sh.step[1];
    double nr_u = 0, nr_v = 0;
#pragma unroll
    for (int k = 0; k < kCgPer; ++k) {
      const int r = tid + k * nt;
      if (r < nv) {
        xu[k] += al_u * sh.pu[r]; xv[k] += al_v * sh.pv[r];
        ru[k] -= al_u * qu[k]; rv[k] -= al_v * qv[k];
        nr_u += ru[k] * ru[k]; nr_v += rv[k] * rv[k];
      }
    }
    group_put2(nr_u, nr_v, sh.red[1], nwa);
    if (w0) {
      const double nr = group_take2(sh.red[1], nwa);
      const double be = done ? 0.0 : nr / rr;
      if ((tid & 15) == 0) sh.step[2 + (tid >> 4)] = be;
      rr = nr;
      done = done || rr <= tol;
      publish_done();
    }
    group_bar(nwa);
    const double be_u = sh.step[2], be_v = sh.step[3];
#pragma unroll
    for (int k = 0; k < kCgPer; ++k) {
      const int r = tid + k * nt;
      if (r < nv) {
        if (!(d & 1)) sh.pu[r] = ru[k] + be_u * sh.pu[r];
        if (!(d & 2)) sh.pv[r] = rv[k] + be_v * sh.pv[r];
      }
    }
    group_bar(nwa);  // the new search direction is visible to the next product
  }
  if (iter >= kCgMaxIters && tid == 0 && status) atomicExch(status, PIV_E_TIMEOUT);
}

template <typename T>
__global__ void __launch_bounds__(kRepThreads) k_replace(RepArgs a, int* status) {
  __shared__ double red_d[64];
  __shared__ CgShared cg;
  __shared__ int red_i[40];
  const int pair = blockIdx.x;
  const int m = a.val.m, n = a.val.n, mn = m * n;
  const long long off = (long long)pair * mn;
  double* u = a.u + off;
  double* v = a.v + off;
  uint8_t* val = a.val_mask + off;
  const uint8_t* fmask = a.val.field_mask;
  RepScratch sc = rep_scratch(a.scratch, mn, pair);
  const int tid = threadIdx.x, nt = blockDim.x;
  const int s = a.size;

  if (a.n_iters == 0) return;
  int nv = block_compact(val, mn, sc.list, sc.rank, red_i);
  if (nv == 0) return;
  // The input values of the flagged points (the only ones that change).
  for (int r = tid; r < nv; r += nt) {
    const int p = sc.list[r];
    sc.init_u[p] = u[p];
    sc.init_v[p] = v[p];
  }

  // 1 / c of a link coefficient 1/3 in the link matrix's type.
  const double third = 1.0 / (a.dtype == PIV_DTYPE_F32 ? (double)(float)(1.0 / 3.0) : 1.0 / 3.0);
  bool fill_nan = true;
  ValSettings vs{a.val.size, a.val.s2n_tol, a.val.median_tol, a.val.mad_tol, a.val.mean_tol, a.val.rms_tol,
                 a.val.fp32, a.val.s2n, a.val.s2n_dtype};
  for (int it = 0; it < a.n_iters; ++it) {
    if (it > 0) nv = block_compact(val, mn, sc.list, sc.rank, red_i);
    if (nv == 0) break;
    // 1. Replacement values from the current fields.
    if (a.method == PIV_REPLACE_SPRING && nv <= kCgSmall) {
      // Every outlier is a row; the warps without rows wait at the block
      // barrier below.
      const int nwa = min(nt >> 5, (nv + 31) >> 5);
      if ((tid >> 5) < nwa) {
        FieldView fu{u, m, n, val, 0.0}, fv{v, m, n, val, 0.0};
        double xu[kCgPer], xv[kCgPer], ru[kCgPer], rv[kCgPer], dd[kCgPer];
        int nb[kCgPer][4];
#pragma unroll
        for (int k = 0; k < kCgPer; ++k) {
          const int r = tid + k * nt;
          ru[k] = rv[k] = dd[k] = 0;
          nb[k][0] = nb[k][1] = nb[k][2] = nb[k][3] = -1;
          if (r < nv) {
            const int p = sc.list[r], i = p / n, j = p % n;
            dd[k] = spring_scale(i, j, m, n, s, third);
            ru[k] = dd[k] * (double)spring_rhs<T>(fu, i, j, s);
            rv[k] = dd[k] * (double)spring_rhs<T>(fv, i, j, s);
            const int oi[4] = {-s, 0, 0, s}, oj[4] = {0, -s, s, 0};
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int ii = i + oi[e], jj = j + oj[e];
              nb[k][e] = (ii < 0 || ii >= m || jj < 0 || jj >= n || !val[ii * n + jj]) ? -1 : sc.rank[ii * n + jj];
            }
          }
        }
        cg_small(nv, nwa, dd, nb, ru, rv, xu, xv, cg, -1.0, status);
#pragma unroll
        for (int k = 0; k < kCgPer; ++k) {
          const int r = tid + k * nt;
          if (r < nv) { sc.new_u[r] = xu[k]; sc.new_v[r] = xv[k]; }
        }
      }
    } else if (a.method == PIV_REPLACE_SPRING) {
      FieldView fu{u, m, n, val, 0.0}, fv{v, m, n, val, 0.0};
      double* xu = sc.cg;
      double* xv = sc.cg + mn;
      double* ru = sc.cg + 2 * mn;
      double* rv = sc.cg + 3 * mn;
      double* pu = sc.cg + 4 * mn;
      double* pv = sc.cg + 5 * mn;
      double* qu = sc.cg + 6 * mn;
      double* qv = sc.cg + 7 * mn;
      // Row scale d_r = 1/c_r. A cluster of outliers with no other neighbour
      // (only possible when every point is an outlier) has a zero right-hand
      // side; CG leaves it at zero, the minimum-norm solution that the
      // reference's direct solve returns for this singular case.
      // Rows that no other row links to are solved at once, x = b / d = rhs;
      // the others (coupled rows: 15% of 4% scattered outliers) are numbered
      // in order for the iterations.
      int* cidx = reinterpret_cast<int*>(qu);   // row -> coupled row or -1
      int* crow = reinterpret_cast<int*>(qv);   // coupled row -> row
      double rr_u = 0, rr_v = 0;
      int nc = 0;
      for (int r0 = 0; r0 < nv; r0 += nt) {
        const int r = r0 + tid;
        bool coupled = false;
        if (r < nv) {
          const int p = sc.list[r], i = p / n, j = p % n;
          const double d = spring_scale(i, j, m, n, s, third);
          const double bu = (double)spring_rhs<T>(fu, i, j, s), bv = (double)spring_rhs<T>(fv, i, j, s);
          const double b1 = d * bu, b2 = d * bv;
          xu[r] = 0; xv[r] = 0;
          ru[r] = b1; rv[r] = b2;
          pu[r] = b1; pv[r] = b2;
          sc.new_u[r] = bu; sc.new_v[r] = bv;
          rr_u += b1 * b1; rr_v += b2 * b2;
          // The row's coupling to the other outliers, resolved once for the
          // iterations: scale and neighbour ranks.
          sc.dinv[r] = d;
          const int oi[4] = {-s, 0, 0, s}, oj[4] = {0, -s, s, 0};
#pragma unroll
          for (int e = 0; e < 4; ++e) {
            const int ii = i + oi[e], jj = j + oj[e];
            const int q = (ii < 0 || ii >= m || jj < 0 || jj >= n || !val[ii * n + jj]) ? -1 : sc.rank[ii * n + jj];
            sc.nbr[e * mn + r] = q;
            coupled = coupled || q >= 0;
          }
        }
        const unsigned bal = __ballot_sync(~0u, coupled);
        if ((tid & 31) == 0) red_i[tid >> 5] = __popc(bal);
        __syncthreads();
        int at = nc;
        for (int w = 0; w < (nt >> 5); ++w) {
          if (w < (tid >> 5)) at += red_i[w];
          nc += red_i[w];
        }
        at += __popc(bal & ((1u << (tid & 31)) - 1u));
        if (r < nv) cidx[r] = coupled ? at : -1;
        if (coupled) crow[at] = r;
        __syncthreads();
      }
      const double2 rr0 = block_sum2(rr_u, rr_v, red_d);
      __syncthreads();
      // The iterations stop where the residual is 1e-14 of the whole right-hand
      // side's norm; right-hand sides that are not finite keep the general
      // iteration.
      if (nc <= kCgSmall && isfinite(rr0.x) && isfinite(rr0.y)) {
        const int nwa = min(nt >> 5, (nc + 31) >> 5);
        if ((tid >> 5) < nwa) {
          double yu[kCgPer], yv[kCgPer], su[kCgPer], sv[kCgPer], dd[kCgPer];
          int nb[kCgPer][4];
#pragma unroll
          for (int k = 0; k < kCgPer; ++k) {
            const int c = tid + k * nt;
            su[k] = sv[k] = dd[k] = 0;
            nb[k][0] = nb[k][1] = nb[k][2] = nb[k][3] = -1;
            if (c < nc) {
              const int r = crow[c];
              dd[k] = sc.dinv[r];
              su[k] = ru[r];
              sv[k] = rv[r];
#pragma unroll
              for (int e = 0; e < 4; ++e) {
                const int q = sc.nbr[e * mn + r];
                nb[k][e] = q < 0 ? -1 : cidx[q];
              }
            }
          }
          cg_small(nc, nwa, dd, nb, su, sv, yu, yv, cg,
                   1e-28 * ((threadIdx.x & 16) ? rr0.y : rr0.x), status);
#pragma unroll
          for (int k = 0; k < kCgPer; ++k) {
            const int c = tid + k * nt;
            if (c < nc) { sc.new_u[crow[c]] = yu[k]; sc.new_v[crow[c]] = yv[k]; }
          }
        }
      } else {
        // Conjugate gradients on (D - Adj) x = D rhs for both fields at once.
        rr_u = rr0.x;
        rr_v = rr0.y;
        const double tol_u = rr_u * 1e-28, tol_v = rr_v * 1e-28;
        bool done_u = rr_u <= tol_u || rr_u == 0, done_v = rr_v <= tol_v || rr_v == 0;
        int iter = 0;
        for (; iter < kCgMaxIters && !(done_u && done_v); ++iter) {
          // q = A p
          double pq_u = 0, pq_v = 0;
          for (int r = tid; r < nv; r += nt) {
            const double d = sc.dinv[r];
            double au = d * pu[r], av = d * pv[r];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
              const int k = sc.nbr[e * mn + r];
              if (k >= 0) { au -= pu[k]; av -= pv[k]; }
            }
            qu[r] = au; qv[r] = av;
            pq_u += pu[r] * au; pq_v += pv[r] * av;
          }
          const double2 pq = block_sum2(pq_u, pq_v, red_d);
          const double al_u = done_u ? 0.0 : rr_u / pq.x, al_v = done_v ? 0.0 : rr_v / pq.y;
          double nr_u = 0, nr_v = 0;
          for (int r = tid; r < nv; r += nt) {
            xu[r] += al_u * pu[r]; xv[r] += al_v * pv[r];
            ru[r] -= al_u * qu[r]; rv[r] -= al_v * qv[r];
            nr_u += ru[r] * ru[r]; nr_v += rv[r] * rv[r];
          }
          const double2 nr = block_sum2(nr_u, nr_v, red_d);
          const double be_u = done_u ? 0.0 : nr.x / rr_u, be_v = done_v ? 0.0 : nr.y / rr_v;
          for (int r = tid; r < nv; r += nt) {
            if (!done_u) pu[r] = ru[r] + be_u * pu[r];
            if (!done_v) pv[r] = rv[r] + be_v * pv[r];
          }
          rr_u = nr.x; rr_v = nr.y;
          done_u = done_u || rr_u <= tol_u;
          done_v = done_v || rr_v <= tol_v;
          __syncthreads();
        }
        if (iter >= kCgMaxIters && tid == 0 && status) atomicExch(status, PIV_E_TIMEOUT);
        for (int r = tid; r < nv; r += nt) { sc.new_u[r] = xu[r]; sc.new_v[r] = xv[r]; }
      }
    } else {
      const double fill = fill_nan ? NAN : 0.0;
      FieldView fu{u, m, n, fill_nan ? val : nullptr, fill}, fv{v, m, n, fill_nan ? val : nullptr, fill};
      const int kind = a.method == PIV_REPLACE_MEDIAN ? 0 : 1;
      for (int r = tid; r < nv; r += nt) {
        const int p = sc.list[r], i = p / n, j = p % n;
        sc.new_u[r] = (double)nbr_stat<T>(fu, i, j, s, kind, (T)0);
        sc.new_v[r] = (double)nbr_stat<T>(fv, i, j, s, kind, (T)0);
      }
    }
    __syncthreads();
    // 2. Write the replacements (rounded to the field type).
    for (int r = tid; r < nv; r += nt) {
      const int p = sc.list[r];
      u[p] = (double)(T)sc.new_u[r];
      v[p] = (double)(T)sc.new_v[r];
    }
    __syncthreads();
    if (a.revalidate) {
      // Reset unresolved points, then revalidate the replaced points only.
      for (int r = tid; r < nv; r += nt) {
        const int p = sc.list[r];
        const bool unres = isnan(u[p]) || isnan(v[p]);
        sc.flag[p] = unres ? 1 : 0;
        if (unres) { u[p] = sc.init_u[p]; v[p] = sc.init_v[p]; }
      }
      __syncthreads();
      FieldView fu{u, m, n, nullptr, 0.0}, fv{v, m, n, nullptr, 0.0};
      for (int r = tid; r < nv; r += nt) {
        const int p = sc.list[r];
        uint8_t nvl = sc.flag[p];
        if (!(fmask && fmask[p])) nvl |= point_invalid<T>(vs, fu, fv, off + p, p / n, p % n, nullptr) ? 1 : 0;
        val[p] = nvl;
      }
      __syncthreads();
    } else {
      fill_nan = false;
    }
  }
  if (!a.revalidate) {
    for (int r = tid; r < nv; r += nt) {
      const int p = sc.list[r];
      if (isnan(u[p]) || isnan(v[p])) { u[p] = sc.init_u[p]; v[p] = sc.init_v[p]; }
    }
  }
}

int replace(const RepArgs& a, cudaStream_t stream) {
  if (a.size > 3 || a.size < 1) return set_error(PIV_E_UNSUPPORTED, "replacing_size %d (supported: 1..3)", a.size);
  if (a.val.size > 3 || a.val.size < 1)
    return set_error(PIV_E_UNSUPPORTED, "validation_size %d (supported: 1..3)", a.val.size);
  if (!isnan(a.val.rms_tol) && a.revalidate)
    return set_error(PIV_E_UNSUPPORTED, "revalidation with rms_tol is not implemented");
  if (a.val.n_pairs == 0 || a.val.m * a.val.n == 0 || a.n_iters == 0) return PIV_OK;
  if (a.val.fp32) k_replace<float><<<a.val.n_pairs, kRepThreads, 0, stream>>>(a, a.status);
  else k_replace<double><<<a.val.n_pairs, kRepThreads, 0, stream>>>(a, a.status);
  cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_replace launch");
}

}  // namespace piv
