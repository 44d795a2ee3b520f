// Plain-form correlation in float64: the double launch configurations (the
// kernel is in piv_corr_fft.cuh) and the searched form of the common passes.
#include <type_traits>

#include "piv_corr_fft.cuh"
#include "piv_corr_fft_half.cuh"

namespace piv {

static const FftVariant kFft8d[] = {PIV_FFT_VAR(8, double, 1, 8, 16, 128)};
static const FftVariant kFft16d[] = {PIV_FFT_VAR(16, double, 1, 16, 8, 128), PIV_FFT_VAR(16, double, 4, 4, 8, 128)};
static const FftVariant kFft32d[] = {PIV_FFT_VAR(32, double, 4, 8, 4, 128), PIV_FFT_VAR(32, double, 8, 4, 4, 128),
                                     PIV_FFT_VAR(32, double, 4, 8, 2, 128)};
static const FftVariant kFft64d[] = {PIV_FFT_VAR(64, double, 8, 8, 1, 256), PIV_FFT_VAR(64, double, 4, 16, 1, 256),
                                     PIV_FFT_VAR(64, double, 8, 8, 1, 512)};
static const FftVariant kFft128d[] = {PIV_FFT_VAR(128, double, 8, 16, 1, 512),
                                      PIV_FFT_VAR(128, double, 16, 8, 1, 512)};
static const FftVariant kFft256d[] = {PIV_FFT_VAR(256, double, 16, 16, 1, 1024)};

const FftVariant* fft_variants_f64(int fft_size, int* count) {
  *count = 0;
  switch (fft_size) {
    case 8: return table(kFft8d, count);
    case 16: return table(kFft16d, count);
    case 32: return table(kFft32d, count);
    case 64: return table(kFft64d, count);
    case 128: return table(kFft128d, count);
    case 256: return table(kFft256d, count);
    default: return nullptr;
  }
}

// ---------------------------------------------------------------------------
// The searched form. Float64 has 1/64 of the float32 rate here, and the
// transforms of a window cost about 300,000 float64 instructions (N = 64): the
// kernel was bound by the float64 pipe, 2.49 ms for the 3,871 windows of an
// 800 x 1280 pair, where this form takes 0.11 ms (search 68 us, fits 33 us,
// open windows 8 us). What is read from the map is its first maximum and five
// values around it, so a float32 map finds the maximum wherever its two
// largest values are further apart than the float32 errors of both
// (search_settled), the five values are formed as direct sums in float64 (five
// products per pixel; exact sums of whole numbers for 8- and 16-bit frames).
// Where the search leaves a few candidates, float64 sums at their lags decide;
// windows with many, or tied in float64 too, take the float64 transforms, as
// do maps and S2N, which read more of the map.
// ---------------------------------------------------------------------------
static constexpr int kFitWarps = 16;

// Sums of a window over K lags as one warp leaves them. Whole-number pixels: a
// - mean a = (a - A) - f_a with A a whole number next to the mean; the sums of
// the pixels, and over each lag's overlap of (a - A)(b - B), a - A and b - B,
// are exact, and value() brings in the fractions. Other pixels: the float64
// values.
template <typename P, int K>
struct LagSums {
  static constexpr bool whole = sizeof(P) <= 2;
  using Acc = std::conditional_t<sizeof(P) == 1, int, std::conditional_t<whole, long long, double>>;
  Acc s[K];
  int ta[whole ? K : 1], tb[whole ? K : 1], sum_a, sum_b;
  PIV_D static int pivot(int sum, int ss) { return (sum + ss * ss / 2) / (ss * ss); }
  PIV_D double value(int k, int ss, int di, int dj) const {
    if constexpr (whole) {
      // With n = ss^2 pixels, A n = sum_a - ra: the value times n^2 is a whole
      // number. 8-bit frames: below 2^53, so the value is exact.
      const int n = ss * ss, ra = sum_a - pivot(sum_a, ss) * n, rb = sum_b - pivot(sum_b, ss) * n;
      const int hy = ss - abs(di), hx = ss - abs(dj), cnt = hy > 0 && hx > 0 ? hy * hx : 0;
      if constexpr (sizeof(P) == 1) {
        const long long v = ((long long)n * s[k] - ((long long)ra * tb[k] + (long long)rb * ta[k])) * n +
                            (long long)cnt * ra * rb;
        return (double)v / ((double)n * n);  // a power of two
      } else {
        const double fa = (double)ra / n, fb = (double)rb / n;
        return (double)s[k] - (fa * (double)tb[k] + fb * (double)ta[k]) + (double)cnt * fa * fb;
      }
    } else {
      return s[k];
    }
  }
};

// The sums at lags (di[k], dj[k]), in every lane. Every load is issued (at a
// clamped position where the lag leaves b's window), so that the loads of
// several pixels are in flight together.
template <typename P, int K>
PIV_D void lag_sums(const P* fa, const P* fb, int width, int ss, const int (&di)[K], const int (&dj)[K],
                    LagSums<P, K>& o) {
  constexpr bool whole = LagSums<P, K>::whole;
  using T = std::conditional_t<whole, int, double>;  // a pixel less its mean
  using Acc = typename LagSums<P, K>::Acc;
  const int lane = threadIdx.x & 31, sh = 31 - __clz(ss), n = ss * ss;
  T sa = 0, sb = 0;
#pragma unroll 8
  for (int e = lane; e < n; e += 32) {
    const long long at = (long long)(e >> sh) * width + (e & (ss - 1));
    sa += (T)__ldg(fa + at);
    sb += (T)__ldg(fb + at);
  }
  T A, B;
  if constexpr (whole) {
    o.sum_a = __reduce_add_sync(~0u, sa);
    o.sum_b = __reduce_add_sync(~0u, sb);
    A = o.pivot(o.sum_a, ss);
    B = o.pivot(o.sum_b, ss);
  } else {
    A = warp_sum(sa) / n;
    B = warp_sum(sb) / n;
  }
  Acc s[K];
  int ta[K], tb[K];
#pragma unroll
  for (int k = 0; k < K; ++k) s[k] = 0, ta[k] = tb[k] = 0;
#pragma unroll 4
  for (int e = lane; e < n; e += 32) {
    const int y = e >> sh, x = e & (ss - 1);
    const T va = (T)__ldg(fa + (long long)y * width + x) - A;
#pragma unroll
    for (int k = 0; k < K; ++k) {
      const int r = y + di[k], q = x + dj[k];
      const bool in = (unsigned)r < (unsigned)ss && (unsigned)q < (unsigned)ss;
      const int rc = min(max(r, 0), ss - 1), qc = min(max(q, 0), ss - 1);
      const T px = (T)__ldg(fb + (long long)rc * width + qc);
      if constexpr (whole) {
        const int vb = in ? px - B : 0;
        s[k] += (Acc)va * vb;
        ta[k] += in ? va : 0;
        tb[k] += vb;
      } else if (in) {
        s[k] = fma(va, px - B, s[k]);
      }
    }
  }
#pragma unroll
  for (int k = 0; k < K; ++k) {
    if constexpr (whole) {
      if constexpr (sizeof(Acc) == 4) {
        s[k] = __reduce_add_sync(~0u, s[k]);
      } else {
        for (int d = 16; d > 0; d >>= 1) s[k] += __shfl_xor_sync(~0u, s[k], d);
      }
      o.s[k] = s[k];
      o.ta[k] = __reduce_add_sync(~0u, ta[k]);
      o.tb[k] = __reduce_add_sync(~0u, tb[k]);
    } else {
      o.s[k] = warp_sum(s[k]);
    }
  }
}

// The windows whose float32 map left a few candidates: their float64 values
// decide, one warp per window; a window whose two largest are within the
// float64 tie tolerance goes to the float64 transforms' list.
template <typename P>
__global__ void __launch_bounds__(32 * kFitWarps) k_resolve64(CorrArgs a) {
  const int count = min(*a.cand_count, a.cand_cap), n = a.fft_size, lane = threadIdx.x & 31;
  for (int q = blockIdx.x * kFitWarps + (threadIdx.x >> 5); q < count; q += gridDim.x * kFitWarps) {
    const int* rec = a.cand + (long long)q * kCandInts;
    const int g = rec[0], cnt = rec[1];
    long long base;
    window_corner(a, g, base);
    double best = -INFINITY, second = -INFINITY;
    int at = 0;
    for (int k0 = 0; k0 < cnt; k0 += 2) {
      const int p0 = rec[2 + k0], p1 = rec[2 + min(k0 + 1, cnt - 1)];
      const int di[2] = {p0 / n - n / 2, p1 / n - n / 2}, dj[2] = {p0 % n - n / 2, p1 % n - n / 2};
      LagSums<P, 2> sums;
      lag_sums<P, 2>(reinterpret_cast<const P*>(a.frame_a) + base, reinterpret_cast<const P*>(a.frame_b) + base,
                     a.width, a.ss, di, dj, sums);
#pragma unroll
      for (int k = 0; k < 2; ++k) {
        if (k0 + k >= cnt) break;
        const double c = sums.value(k, a.ss, di[k], dj[k]);
        second = fmax(second, fmin(best, c));
        if (c > best) {
          best = c;
          at = k == 0 ? p0 : p1;
        }
      }
    }
    if (lane != 0) continue;
    if (best - second > (double)kTieTolF64 * fabs(best)) {
      a.peak_i[g] = at / n;
      a.peak_j[g] = at % n;
    } else {
      a.tie_list[atomicAdd(a.tie_list_count, 1)] = g;
    }
  }
}

// Fit and displacement of every window (none is masked) from its peak: each
// warp sums kFitPerWarp windows, then one warp fits all of the CTA's, a window
// per lane (a fit is some 500 float64 instructions, whose cost does not depend
// on how many lanes take part: with one fit per warp the kernel took 81 us for
// 3,871 windows of 32 px, so it takes 33 us).
static constexpr int kFitPerWarp = 2;
static_assert(kFitWarps * kFitPerWarp == 32, "one window per lane of the fitting warp");
template <typename P>
__global__ void __launch_bounds__(32 * kFitWarps) k_fit64(CorrArgs a) {
  __shared__ LagSums<P, 5> sums_s[32];
  const long long total = (long long)a.n_pairs * a.m * a.n;
  const int n = a.fft_size, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  auto lags = [&](long long g, int (&di)[5], int (&dj)[5]) {  // false: a peak on the map's border
    const int pi = a.peak_i[g], pj = a.peak_j[g], i = pi - n / 2, j = pj - n / 2;
    // Centre, rows above and below, columns left and right.
    di[0] = di[3] = di[4] = i;
    dj[0] = dj[1] = dj[2] = j;
    di[1] = i - 1, di[2] = i + 1, dj[3] = j - 1, dj[4] = j + 1;
    return pi > 0 && pi < n - 1 && pj > 0 && pj < n - 1;
  };
  int di[5], dj[5];
  for (long long g0 = (long long)blockIdx.x * 32; g0 < total; g0 += (long long)gridDim.x * 32) {
    for (int k = 0; k < kFitPerWarp; ++k) {
      const int slot = warp * kFitPerWarp + k;
      const long long g = g0 + slot;
      if (g >= total || !lags(g, di, dj)) continue;
      long long base;
      window_corner(a, g, base);
      LagSums<P, 5> sums;
      lag_sums<P, 5>(reinterpret_cast<const P*>(a.frame_a) + base, reinterpret_cast<const P*>(a.frame_b) + base,
                     a.width, a.ss, di, dj, sums);
      if (lane == 0) sums_s[slot] = sums;
    }
    __syncthreads();
    const long long g = g0 + lane;
    if (warp == 0 && g < total) {
      const bool inner = lags(g, di, dj);
      const int pi = a.peak_i[g], pj = a.peak_j[g];
      double isp = (double)pi, jsp = (double)pj, c[5];
      if (inner) {
#pragma unroll
        for (int k = 0; k < 5; ++k) c[k] = sums_s[lane].value(k, a.ss, di[k], dj[k]);
        subpixel_fit<double>(a.subpixel, pi, pj, c[0], c[1], c[2], c[3], c[4], isp, jsp);
      }
      reinterpret_cast<double*>(a.u)[g] = sub_rn(jsp, (double)(n / 2));
      reinterpret_cast<double*>(a.v)[g] = sub_rn(isp, (double)(n / 2));
    }
    __syncthreads();
  }
}

template <typename P>
static int launch_fit64(const CorrArgs& a, cudaStream_t stream) {
  const long long total = (long long)a.n_pairs * a.m * a.n;
  k_resolve64<P><<<(unsigned)std::min<long long>((a.cand_cap + kFitWarps - 1) / kFitWarps, sm_count() * 4),
                   32 * kFitWarps, 0, stream>>>(a);
  const long long blocks = std::min((total + 31) / 32, (long long)sm_count() * 8);
  k_fit64<P><<<(unsigned)blocks, 32 * kFitWarps, 0, stream>>>(a);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_fit64 launch");
}

// Windows of a float64 pass with n_fft 2 and no shrink, when the caller gives
// a list buffer and peak arrays and reads neither maps nor S2N. Masked passes
// keep the transforms: their fields enter the weighted smoothing, whose search
// for the parameter stops where its curve is flat, and a last bit of a
// displacement moves the smoothed field there by up to 2e-3 px.
static bool correlate_f64_searched(const CorrArgs& a) {
  return a.dtype == PIV_DTYPE_F64 && corr_fft_half_windows(a) && !a.win_mask && !a.maps && !a.s2n && !a.win_list && a.tie_list &&
         a.tie_list_count && a.peak_i && a.peak_j && a.cand && a.cand_count == a.tie_list_count + 1 &&
         a.cand_cap > 0;
}

int correlate_f64(const CorrArgs& a, const FftVariant& t, cudaStream_t stream) {
  const long long total = (long long)a.n_pairs * a.m * a.n;
  if (!correlate_f64_searched(a) || total == 0 || total > 2147483647LL) return t.launch(a, stream);
  cudaError_t e = cudaMemsetAsync(a.tie_list_count, 0, 2 * sizeof(int), stream);  // and cand_count (set_f64_lists)
  if (e != cudaSuccess) return set_cuda_error(e, "window list counts");
  const bool whole = a.pixel_type == PIV_PIXEL_U8 || a.pixel_type == PIV_PIXEL_U16;
  int rc = whole ? correlate_fft_half<true, float>(a, stream) : correlate_fft_half<true, double>(a, stream);
  if (rc != PIV_OK) return rc;
  switch (a.pixel_type) {
    case PIV_PIXEL_U8: rc = launch_fit64<uint8_t>(a, stream); break;
    case PIV_PIXEL_U16: rc = launch_fit64<uint16_t>(a, stream); break;
    case PIV_PIXEL_F32: rc = launch_fit64<float>(a, stream); break;
    default: rc = launch_fit64<double>(a, stream); break;
  }
  if (rc != PIV_OK) return rc;
  CorrArgs f = a;
  f.win_list = a.tie_list;
  f.win_count = a.tie_list_count;
  return t.launch(f, stream);
}

}  // namespace piv
