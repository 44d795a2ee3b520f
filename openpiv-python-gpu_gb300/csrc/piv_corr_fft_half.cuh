// Plain-form correlation for the common passes: float32, windows of ss = N / 2
// (n_fft 2, no shrink), N = 32, 64 and 128. The same transforms, product and
// search as k_corr_fft (piv_corr_fft.cuh), term by term, with fewer sweeps
// over shared memory:
//   * only the ss x ss window is stored; the zero pad is never written, and
//     the forward passes leave its terms out (half the inputs of the first
//     radix stage along both axes are zero);
//   * N = 64, 128: the last forward pass along the columns, the conjugate
//     product and the first inverse pass run on one pair of eight-point groups
//     (the group of frequencies k2 + R2 k1 and that of the negated
//     frequencies), in registers;
//   * N = 32: one warp per window, one line per lane, no block barriers;
//   * the last inverse pass forms only the real parts, scales them and finds
//     each line's two largest values on the way;
//   * the twiddles inside the register DFTs are constants.
// Shared-memory traffic and instruction issue bound the kernel. Measured (one
// 1024 x 1024 pair at 50% overlap, 8-bit frames; the general kernel, then
// this): N = 32 136 -> 57 us, N = 64 139 -> 68 us, N = 128 174 -> 90 us.
#pragma once

#include "piv_corr_fft.cuh"

namespace piv {

// W_32^j = exp(-2 pi i j / 32), j < 16 (every eighth entry of c_tw256_f).
struct TwPair {
  float x, y;
};
PIV_HD constexpr TwPair tw32(int j) {
  switch (j) {
    case 0: return {1.0f, -0.0f};
    case 1: return {0.9807852506637573f, -0.19509032368659973f};
    case 2: return {0.9238795042037964f, -0.3826834261417389f};
    case 3: return {0.8314695954322815f, -0.5555702447891235f};
    case 4: return {0.7071067690849304f, -0.7071067690849304f};
    case 5: return {0.5555702447891235f, -0.8314695954322815f};
    case 6: return {0.3826834261417389f, -0.9238795042037964f};
    case 7: return {0.19509032368659973f, -0.9807852506637573f};
    case 8: return {-0.0f, -1.0f};
    case 9: return {-0.19509032368659973f, -0.9807852506637573f};
    case 10: return {-0.3826834261417389f, -0.9238795042037964f};
    case 11: return {-0.5555702447891235f, -0.8314695954322815f};
    case 12: return {-0.7071067690849304f, -0.7071067690849304f};
    case 13: return {-0.8314695954322815f, -0.5555702447891235f};
    case 14: return {-0.9238795042037964f, -0.3826834261417389f};
    default: return {-0.9807852506637573f, -0.19509032368659973f};
  }
}

// a w and the product's terms with the roundings written out (one product of
// each sum rounded, the other fused), as the compiler contracts the general
// kernel's expressions: the maps of both kernels are the same bit for bit.
PIV_D Cplx<float> cmul_k(Cplx<float> a, float wx, float wy) {
  return cmake<float>(__fmaf_rn(a.x, wx, -__fmul_rn(a.y, wy)), __fmaf_rn(a.y, wx, __fmul_rn(a.x, wy)));
}
PIV_D Cplx<float> cmul_k(Cplx<float> a, Cplx<float> w) { return cmul_k(a, w.x, w.y); }

// a + b and a - b of both parts in one packed float32 pair instruction each
// (rounded as the scalar ones; half the issue slots): N = 32 64.2 -> 56.5 us,
// N = 64 68.4 -> 67.6 us, N = 128 92.2 -> 90.4 us on the pair above. A rotated
// operand (W = -+i) takes scalar sums instead: packing its swapped parts would
// cost the moves that the pair saves.
PIV_D void butterfly(Cplx<float> a, Cplx<float> b, Cplx<float>& sum, Cplx<float>& dif) {
  asm("{\n.reg .b64 a, b, s, d;\nmov.b64 a, {%4, %5};\nmov.b64 b, {%6, %7};\nadd.rn.f32x2 s, a, b;\nsub.rn.f32x2 d, a, b;\n"
      "mov.b64 {%0, %1}, s;\nmov.b64 {%2, %3}, d;\n}\n"
      : "=f"(sum.x), "=f"(sum.y), "=f"(dif.x), "=f"(dif.y)
      : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
}

// Radix-2 stages from span LEN up of the R-point register DFT (dft_stage with
// constant twiddles).
template <int R, int LEN, bool INV>
PIV_D void dft_stage_k(Cplx<float> (&y)[R]) {
#pragma unroll
  for (int i = 0; i < R; i += LEN) {
#pragma unroll
    for (int j = 0; j < LEN / 2; ++j) {
      const Cplx<float> a = y[i + j];
      Cplx<float> b = y[i + j + LEN / 2];
      if (LEN >= 4 && j == LEN / 4) {
        // W = -i (forward) or +i (inverse): a +- (b.y, -b.x) or its negative.
        const Cplx<float> lo = cmake<float>(a.x + b.y, a.y - b.x), hi = cmake<float>(a.x - b.y, a.y + b.x);
        y[i + j] = INV ? hi : lo;
        y[i + j + LEN / 2] = INV ? lo : hi;
        continue;
      }
      if (j != 0) {
        const TwPair w = tw32(j * (32 / LEN));  // constant once unrolled
        b = cmul_k(b, w.x, INV ? -w.y : w.y);
      }
      butterfly(a, b, y[i + j], y[i + j + LEN / 2]);
    }
  }
  if constexpr (LEN < R) dft_stage_k<R, 2 * LEN, INV>(y);
}

template <int R, bool INV>
PIV_D void dft_k(Cplx<float> (&x)[R]) {
  Cplx<float> y[R];
  bitrev_permute<R, float>(y, x, std::make_integer_sequence<int, R>{});
  dft_stage_k<R, 2, INV>(y);
#pragma unroll
  for (int i = 0; i < R; ++i) x[i] = y[i];
}

// Forward DFT of R points of which only x[R/4 .. 3R/4) are non-zero (the
// others are not read): of each pair (k, k + R/2) of the first stage one is
// zero.
template <int R>
PIV_D void dft_half(Cplx<float> (&x)[R]) {
  Cplx<float> y[R];
#pragma unroll
  for (int i = 0; i < R; i += 2) {
    const int k = bitrev<R>(i);  // y[i] = x[k] + x[k + R/2], y[i + 1] = x[k] - x[k + R/2]
    if (k >= R / 4) {
      y[i] = x[k];
      y[i + 1] = x[k];
    } else {
      y[i] = x[k + R / 2];
      y[i + 1] = cmake<float>(-x[k + R / 2].x, -x[k + R / 2].y);
    }
  }
  if constexpr (R > 2) dft_stage_k<R, 4, false>(y);
#pragma unroll
  for (int i = 0; i < R; ++i) x[i] = y[i];
}

// P = conj(A) B at frequency k from Z(k) and Z(-k) of z = a + i b.
PIV_D Cplx<float> conj_product(Cplx<float> zk, Cplx<float> zm) {
  const float ar = zk.x + zm.x, ai = zk.y - zm.y;
  const float br = zk.y + zm.y, bi = zm.x - zk.x;
  return cmake<float>(__fmul_rn(__fmaf_rn(ar, br, __fmul_rn(ai, bi)), 0.25f),
                      __fmul_rn(__fmaf_rn(ar, bi, -__fmul_rn(ai, br)), 0.25f));
}

// Corner of window g (element offset in a frame batch); false when masked.
PIV_D bool window_corner(const CorrArgs& a, long long g, long long& base) {
  const int n_wins = a.m * a.n;
  const int pair = (int)(g / n_wins), k = (int)(g - (long long)pair * n_wins);
  const int wr = k / a.n, wc = k - wr * a.n;
  base = pair * ((long long)a.height * a.width) + (long long)(wr * a.spacing + a.y_offset) * a.width +
         wc * a.spacing + a.x_offset;
  return !(a.win_mask && a.win_mask[k]);
}

// Two largest of a line's values in ascending shifted order: v enters with
// index f.
struct Top2 {
  float best, second;
  int at;
  PIV_D void init() {
    best = second = -INFINITY;
    at = 0x7fffffff;
  }
  PIV_D void next(float v, int f) {  // f above every earlier index
    second = fmaxf(second, fminf(v, best));
    const bool up = v > best;
    best = up ? v : best;
    at = up ? f : at;
  }
  PIV_D void merge(const Top2& o) {
    second = fmaxf(fmaxf(second, o.second), fminf(best, o.best));
    const bool up = o.best > best || (o.best == best && o.at < at);
    best = up ? o.best : best;
    at = up ? o.at : at;
  }
};

// Search mode (float64 passes, correlate_f64): the float32 map only finds the
// integer peak. The window means are removed in a way that leaves rounding of
// the differences alone: whole-number pixels less the nearest whole number of
// the mean and then its fraction, other pixels in float64. Both mean-removed
// windows are then scaled by powers of two to 2-norms in [1, 2) (search_scale):
// they share one transform z = a + i b, whose rounding follows |z|, so that the
// spectrum of the smaller window would carry the larger one's error (frames 1e4
// apart in contrast: map errors above the gap below, wrong peaks settled).
// A window is settled when its two largest values are further apart than
// kSearchTol |a| |b|; the others go to the list. With norms within a factor of
// two, the forward transforms' errors move a map value by at most 3.4 eta |a|
// |b|, eta = 6.7 u log2(N^2) the transform's norm-wise bound (Higham, Accuracy
// and Stability of Numerical Algorithms, section 24.1; u = 2^-24): 1.9e-5 |a|
// |b| for N = 128, under a third of the gap of 6.1e-5 |a| |b|. The inverse's
// error is bounded by eta |c|_2 only, and the map's norm |c|_2 exceeds |a| |b|
// for smooth windows, so there the margin is a measured one: 2.7e-7 |a| |b| in
// all, the largest error of 12,600 noisy, matched and smooth windows of 16 to
// 64 px with contrasts up to 1e9 apart.
constexpr float kSearchTol = 1.0f / 16384.0f;
// The power of two that brings a window of squared 2-norm `norm` to [1, 2).
PIV_D float search_scale(float norm) {
  const int e = (__float_as_int(norm) >> 23) - 127;  // floor of log2
  return __int_as_float((127 - (e >> 1)) << 23);
}
// Gap that settles a window of squared norms norm_a and norm_b, scaled by sa
// and sb; infinite where the sums of squares leave the float32 range (nothing
// is settled then).
PIV_D float search_gap(float norm_a, float norm_b, float sa, float sb) {
  const bool in_range = norm_a > 1e-30f && norm_a < 1e30f && norm_b > 1e-30f && norm_b < 1e30f;
  return in_range ? kSearchTol * (sqrtf(norm_a) * sa) * (sqrtf(norm_b) * sb) : INFINITY;
}
// The open window g: a record of its candidates (values within `gap` of the
// largest; count may exceed kCandMax), or its place in the window list.
PIV_D void search_open(const CorrArgs& a, long long g, int count, const int* at) {
  if (count >= 2 && count <= kCandMax) {
    const int q = atomicAdd(a.cand_count, 1);
    if (q < a.cand_cap) {
      int* rec = a.cand + (long long)q * kCandInts;
      rec[0] = (int)g;
      rec[1] = count;
      for (int k = 0; k < count; ++k) rec[2 + k] = at[k];
      return;
    }
  }
  a.tie_list[atomicAdd(a.tie_list_count, 1)] = (int)g;
}

// Loads CNT pixels of each frame (element k at offset of(k) from the window's
// corner) as X: float for the plain form (any pixel type) and for whole-number
// pixels, double for the search of float pixels.
template <typename X, bool SEARCH, int CNT, class Of>
PIV_D void load_window(const CorrArgs& a, long long base, bool ok, Of of, X (&xa)[CNT], X (&xb)[CNT]) {
  auto load = [&](auto tag) {
    using P = decltype(tag);
    const P* fa = reinterpret_cast<const P*>(a.frame_a) + base;
    const P* fb = reinterpret_cast<const P*>(a.frame_b) + base;
#pragma unroll
    for (int k = 0; k < CNT; ++k) {
      const long long at = of(k);
      xa[k] = ok ? (X)__ldg(fa + at) : (X)0;
      xb[k] = ok ? (X)__ldg(fb + at) : (X)0;
    }
  };
  constexpr bool whole = !SEARCH || sizeof(X) == 4, other = !SEARCH || sizeof(X) == 8;
  if (whole && a.pixel_type == PIV_PIXEL_U8) load(uint8_t{});
  else if (whole && a.pixel_type == PIV_PIXEL_U16) load(uint16_t{});
  else if (other && a.pixel_type == PIV_PIXEL_F32) load(float{});
  else if (other) load(double{});
}

// x less the window mean.
template <bool SEARCH>
PIV_D float less_mean(float x, float mean, float frac) {
  return SEARCH ? (x - mean) - frac : x - mean;
}

// ---------------------------------------------------------------------------
// N = 64 and 128: one window per CTA, lines split as N = 8 R2.
// ---------------------------------------------------------------------------
template <int N_, int NT_, int MIN_CTAS_>
struct HalfCfg {
  static constexpr int N = N_, NT = NT_, MIN_CTAS = MIN_CTAS_;
  using Fft = FftCfg<N, float, 8, N / 8, 1, NT>;  // layout and search of the general kernel
};

template <class H, bool SEARCH = false, typename X = float>
__global__ void __launch_bounds__(H::NT, H::MIN_CTAS) k_corr_fft_half(CorrArgs a) {
  using C = typename H::Fft;
  using L = FftLayout<C>;
  constexpr int N = H::N, NT = H::NT, SS = N / 2, PAD = N / 4, R1 = 8, R2 = N / 8, LD = L::LD, NW = NT / 32;
  // The window means are summed by the general kernel's threads (NT0 of them,
  // then its warps in order), so that both give the same bits.
  constexpr int NT0 = N == 128 ? 1024 : 128, NV = NT0 / NT, PER = SS * SS / NT0, NW0 = NT0 / 32;
  static_assert(NV >= 1 && NT % 64 == 0, "whole virtual warps per warp");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  Cplx<float>* tw = reinterpret_cast<Cplx<float>*>(smem_raw);
  CorrShared<C> S(smem_raw + L::TW_BYTES);
  Cplx<float>* buf = reinterpret_cast<Cplx<float>*>(smem_raw + L::SMEM_SMALL);
  __shared__ float sum_part[2][NW0];
  __shared__ Top2 top_part[NW];
  __shared__ float second_part[NW];
  __shared__ double dsum_part[2][SEARCH ? NW : 1], dmean[2];  // search
  __shared__ float norm_part[2][SEARCH ? NW : 1], cand_from;
  __shared__ int cand_n, cand_at[kCandMax];
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  for (int k = tid; k < 256; k += NT) {
    const float2 w = c_tw256_f[k];
    tw[k] = cmake<float>(w.x, w.y);
  }
  const long long total = a.win_list ? (long long)*a.win_count : (long long)a.n_pairs * a.m * a.n;
  auto tw_n = [&](int e) { return tw[(e & (N - 1)) * (256 / N)]; };

  for (long long slot = blockIdx.x; slot < total; slot += gridDim.x) {
    const long long g = a.win_list ? (long long)a.win_list[slot] : slot;
    long long base;
    const bool ok = window_corner(a, g, base) || SEARCH;  // the search's passes have no mask
    // The window's pixels, PER per virtual thread, and the means.
    X xa[NV * PER], xb[NV * PER];
    auto elem = [&](int k) { return tid + (k / PER) * NT + (k % PER) * NT0; };
    load_window<X, SEARCH>(a, base, ok,
                           [&](int k) { return (long long)(elem(k) / SS) * a.width + elem(k) % SS; }, xa, xb);
    if constexpr (!SEARCH) {
#pragma unroll
      for (int v = 0; v < NV; ++v) {
        float sa = 0.f, sb = 0.f;
#pragma unroll
        for (int q = 0; q < PER; ++q) {
          sa += xa[v * PER + q];
          sb += xb[v * PER + q];
        }
        sa = warp_sum(sa);
        sb = warp_sum(sb);
        if (lane == 0) {
          sum_part[0][warp + v * NW] = sa;
          sum_part[1][warp + v * NW] = sb;
        }
      }
    } else if constexpr (sizeof(X) == 4) {
      int sa = 0, sb = 0;  // whole numbers: at most 4096 x 65535
#pragma unroll
      for (int k = 0; k < NV * PER; ++k) {
        sa += (int)xa[k];
        sb += (int)xb[k];
      }
      sa = __reduce_add_sync(~0u, sa);
      sb = __reduce_add_sync(~0u, sb);
      if (lane == 0) {
        dsum_part[0][warp] = (double)sa;
        dsum_part[1][warp] = (double)sb;
      }
    } else {
      double sa = 0.0, sb = 0.0;
#pragma unroll
      for (int k = 0; k < NV * PER; ++k) {
        sa += xa[k];
        sb += xb[k];
      }
      sa = warp_sum(sa);
      sb = warp_sum(sb);
      if (lane == 0) {
        dsum_part[0][warp] = sa;
        dsum_part[1][warp] = sb;
      }
    }
    __syncthreads();
    if (lane == 0 && warp < 2) {
      if constexpr (!SEARCH) {
        float t = 0.f;
        for (int q = 0; q < NW0; ++q) t += sum_part[warp][q];
        S.means[warp] = t / (float)(SS * SS);
      } else {
        double t = 0.0;
        for (int q = 0; q < NW; ++q) t += dsum_part[warp][q];
        dmean[warp] = t / (double)(SS * SS);
      }
    }
    __syncthreads();
    float na = 0.f, nb = 0.f;  // search: sums of squares
    {
      float ma = 0.f, mb = 0.f, fa = 0.f, fb = 0.f;
      double da = 0.0, db = 0.0;
      if constexpr (!SEARCH) {
        ma = S.means[0];
        mb = S.means[1];
      } else {
        da = dmean[0];
        db = dmean[1];
        ma = (float)rint(da);
        mb = (float)rint(db);
        fa = (float)(da - rint(da));
        fb = (float)(db - rint(db));
      }
#pragma unroll
      for (int k = 0; k < NV * PER; ++k) {
        const int e = elem(k), r = e / SS, c = e % SS;
        float va, vb;
        if constexpr (sizeof(X) == 8) {
          va = (float)(xa[k] - da);
          vb = (float)(xb[k] - db);
        } else {
          va = less_mean<SEARCH>(xa[k], ma, fa);
          vb = less_mean<SEARCH>(xb[k], mb, fb);
        }
        if (!ok) va = vb = 0.f;
        if (SEARCH) {
          na = fmaf(va, va, na);
          nb = fmaf(vb, vb, nb);
        }
        buf[(PAD + r) * LD + PAD + c] = cmake<float>(va, vb);
      }
    }
    if (SEARCH) {
      na = warp_sum(na);
      nb = warp_sum(nb);
      if (lane == 0) {
        norm_part[0][warp] = na;
        norm_part[1][warp] = nb;
      }
    }
    __syncthreads();
    // Search: the windows' scales, applied as the rows are read, and the gap.
    float scale_a = 1.f, scale_b = 1.f, gap = 0.f;
    if constexpr (SEARCH) {
      na = warp_sum(lane < NW ? norm_part[0][lane] : 0.f);
      nb = warp_sum(lane < NW ? norm_part[1][lane] : 0.f);
      scale_a = search_scale(na);
      scale_b = search_scale(nb);
      gap = search_gap(na, nb, scale_a, scale_b);
    }

    // Rows of the window: R2-point DFTs, then eight-point ones. Lanes take
    // adjacent rows (bank-conflict free), the in-line index is the warp's.
#pragma unroll 1
    for (int it0 = 0; it0 < SS * R1; it0 += NT) {
      const int it = it0 + tid, l = it % SS, n1 = it / SS;
      Cplx<float>* p = buf + (PAD + l) * LD + n1;
      Cplx<float> x[R2];
#pragma unroll
      for (int k = R2 / 4; k < 3 * R2 / 4; ++k) {
        x[k] = p[k * R1];
        if (SEARCH) x[k] = cmake<float>(x[k].x * scale_a, x[k].y * scale_b);
      }
      dft_half<R2>(x);
      if (n1 != 0) {
#pragma unroll
        for (int k = 1; k < R2; ++k) x[k] = cmul_k(x[k], tw_n(n1 * k));
      }
#pragma unroll
      for (int k = 0; k < R2; ++k) p[k * R1] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int it0 = 0; it0 < SS * R2; it0 += NT) {
      const int it = it0 + tid, l = it % SS, k2 = it / SS;
      Cplx<float>* p = buf + (PAD + l) * LD + R1 * k2;
      Cplx<float> x[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) x[k] = p[k];
      dft_k<R1, false>(x);
#pragma unroll
      for (int k = 0; k < R1; ++k) p[k] = x[k];
    }
    __syncthreads();
    // Columns: R2-point DFTs over the window's rows.
#pragma unroll 1
    for (int it0 = 0; it0 < N * R1; it0 += NT) {
      const int it = it0 + tid, l = it % N, n1 = it / N;
      Cplx<float>* p = buf + n1 * LD + l;
      Cplx<float> x[R2];
#pragma unroll
      for (int k = R2 / 4; k < 3 * R2 / 4; ++k) x[k] = p[k * R1 * LD];
      dft_half<R2>(x);
      if (n1 != 0) {
#pragma unroll
        for (int k = 1; k < R2; ++k) x[k] = cmul_k(x[k], tw_n(n1 * k));
      }
#pragma unroll
      for (int k = 0; k < R2; ++k) p[k * R1 * LD] = x[k];
    }
    __syncthreads();
    // Column frequencies: position p holds frequency p / 8 + R2 (p % 8). The
    // group (column c, rows 8 k2 .. 8 k2 + 7) holds the row frequencies k2 +
    // R2 k1; the negated frequencies form the group (c', rows 8 (R2 - k2) % N
    // ..), k1 -> 7 - k1 (k2 > 0) or -k1 mod 8 (k2 = 0). One item takes both
    // groups: eight-point DFTs, product, eight-point inverse DFTs.
#pragma unroll 1
    for (int it = tid; it < N * R2 / 2; it += NT) {
      int c, cm, k2;
      bool self = false;  // both groups are their own negatives
      auto negated = [](int q) {
        const int ca = q >> 3, cb = q & 7;
        return ca ? 8 * (R2 - ca) + 7 - cb : ((8 - cb) & 7);
      };
      if (it < (R2 / 2 - 1) * N) {
        k2 = 1 + it / N;
        c = it % N;
        cm = negated(c);
      } else {
        // k2 = 0 and R2 / 2 pair with themselves: half of the columns each.
        const int j = it - (R2 / 2 - 1) * N, jj = j % (N / 2);
        k2 = j < N / 2 ? 0 : R2 / 2;
        constexpr int M = 8 * (R2 / 2 - 1);
        const int q = jj - M;
        c = jj < M ? 8 + jj : (q < 3 ? q + 1 : (q == 3 ? 0 : 8 * (R2 / 2) + q - 4));
        cm = q == 3 ? 4 : negated(c);
        self = q == 3;
      }
      Cplx<float>* pg = buf + 8 * k2 * LD + c;
      Cplx<float>* ph = buf + 8 * ((R2 - k2) % R2) * LD + cm;
      Cplx<float> x[R1], y[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        x[k] = pg[k * LD];
        y[k] = ph[k * LD];
      }
      dft_k<R1, false>(x);
      dft_k<R1, false>(y);
      if (!self) {
        if (k2 == 0) {
#pragma unroll
          for (int k = 0; k < R1; ++k) {
            const Cplx<float> q = conj_product(x[k], y[(8 - k) & 7]);
            x[k] = q;
            y[(8 - k) & 7] = cconj(q);
          }
        } else {
#pragma unroll
          for (int k = 0; k < R1; ++k) {
            const Cplx<float> q = conj_product(x[k], y[7 - k]);
            x[k] = q;
            y[7 - k] = cconj(q);
          }
        }
      } else {
        Cplx<float> u[R1], w[R1];
#pragma unroll
        for (int k = 0; k < R1; ++k) {
          u[k] = k2 == 0 ? conj_product(x[k], x[(8 - k) & 7]) : conj_product(x[k], x[7 - k]);
          w[k] = k2 == 0 ? conj_product(y[k], y[(8 - k) & 7]) : conj_product(y[k], y[7 - k]);
        }
#pragma unroll
        for (int k = 0; k < R1; ++k) {
          x[k] = u[k];
          y[k] = w[k];
        }
      }
      dft_k<R1, true>(x);
      dft_k<R1, true>(y);
#pragma unroll
      for (int k = 0; k < R1; ++k) {
        pg[k * LD] = x[k];
        ph[k * LD] = y[k];
      }
    }
    __syncthreads();
    // Inverse along the columns (R2-point part), then the rows.
#pragma unroll 1
    for (int it0 = 0; it0 < N * R1; it0 += NT) {
      const int it = it0 + tid, l = it % N, n1 = it / N;
      Cplx<float>* p = buf + n1 * LD + l;
      Cplx<float> x[R2];
#pragma unroll
      for (int k = 0; k < R2; ++k) x[k] = p[k * R1 * LD];
      if (n1 != 0) {
#pragma unroll
        for (int k = 1; k < R2; ++k) x[k] = cmul_k(x[k], cconj(tw_n(n1 * k)));
      }
      dft_k<R2, true>(x);
#pragma unroll
      for (int k = 0; k < R2; ++k) p[k * R1 * LD] = x[k];
    }
    __syncthreads();
#pragma unroll 1
    for (int it0 = 0; it0 < N * R2; it0 += NT) {
      const int it = it0 + tid, l = it % N, k2 = it / N;
      Cplx<float>* p = buf + l * LD + R1 * k2;
      Cplx<float> x[R1];
#pragma unroll
      for (int k = 0; k < R1; ++k) x[k] = p[k];
      dft_k<R1, true>(x);
#pragma unroll
      for (int k = 0; k < R1; ++k) p[k] = x[k];
    }
    __syncthreads();
    Top2 top;
    top.init();
    float sum = 0.f;  // not a number if any value is
    const float inv_nn = 1.0f / (float)(N * N);
#pragma unroll 1
    for (int it0 = 0; it0 < N * R1; it0 += NT) {
      const int it = it0 + tid, l = it % N, n1 = it / N;
      Cplx<float>* p = buf + l * LD + n1;
      Cplx<float> x[R2];
#pragma unroll
      for (int k = 0; k < R2; ++k) x[k] = p[k * R1];
      if (n1 != 0) {
#pragma unroll
        for (int k = 1; k < R2; ++k) x[k] = cmul_k(x[k], cconj(tw_n(n1 * k)));
      }
      dft_k<R2, true>(x);
      const int i = l ^ (N / 2);
      Top2 line;
      line.init();
#pragma unroll
      for (int q = 0; q < R2; ++q) {
        const int k = q ^ (R2 / 2);  // ascending shifted columns j = n1 + 8 q
        float v = x[k].x * inv_nn;
        p[k * R1].x = v;
        sum += v;
        if (i == 0 || (q == 0 && n1 == 0)) v = 0.f;  // no window overlap
        line.next(v, i * N + n1 + R1 * q);
      }
      top.merge(line);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      Top2 t;
      t.best = __shfl_xor_sync(~0u, top.best, o);
      t.second = __shfl_xor_sync(~0u, top.second, o);
      t.at = __shfl_xor_sync(~0u, top.at, o);
      top.merge(t);
    }
    if (lane == 0) top_part[warp] = top;
    const bool bad = __syncthreads_or(is_nan(sum));
    if (bad) {
      // Values that are not numbers: the general search's order.
      window_argmax<C>(buf, SS, -1, nullptr, nullptr, S.part_v, S.part_i, S.pval, S.peak, S.part_v + NW, S.means);
      if (tid == 0) {
        S.pi[0] = S.peak[0] / N;
        S.pj[0] = S.peak[0] % N;
      }
    } else if (tid == 0) {
      Top2 t = top_part[0];
      for (int w = 1; w < NW; ++w) t.merge(top_part[w]);
      S.pval[0] = t.best;
      S.means[0] = t.second;
      S.peak[0] = t.at;
      S.pi[0] = t.at / N;
      S.pj[0] = t.at % N;
    }
    if constexpr (SEARCH) {
      if (tid == 0) {
        const float best = S.pval[0];
        a.peak_i[g] = S.pi[0];
        a.peak_j[g] = S.pj[0];
        if (a.near_tie) a.near_tie[g] = 0;
        // The values that the window's candidates reach (open windows only).
        cand_from = !bad && best - S.means[0] > gap ? INFINITY : (bad ? -INFINITY : best - gap);
        cand_n = 0;
      }
      __syncthreads();
      const float from = cand_from;
      if (from == INFINITY) continue;
      if (from > -INFINITY) {
        for (int f = tid; f < N * N; f += NT)
          if (corr_at<N, float>(buf, f / N, f % N, SS) >= from) {
            const int q = atomicAdd(&cand_n, 1);
            if (q < kCandMax) cand_at[q] = f;
          }
      }
      __syncthreads();
      if (tid == 0) search_open(a, g, cand_n, cand_at);
      continue;
    }
    if (tid == 0) S.valid[0] = ok ? 1 : 0;
    if (a.maps || a.s2n) __syncthreads();
    if (a.maps) {
      float* mo = reinterpret_cast<float*>(a.maps) + g * N * N;
      for (int f = tid; f < N * N; f += NT) mo[f] = corr_at<N, float>(buf, f / N, f % N, SS);
      __syncthreads();
    }
    if (a.s2n && a.s2n_method == PIV_S2N_PEAK2PEAK && !bad) {
      // The largest value outside the box (wrapped) around the peak: a column
      // per thread, whose test against the box is made once; -inf where the
      // box leaves nothing, as the reference's masked map reads there. Against
      // the general search, with its position and box at every value: one
      // 1080 x 1920 pair, N = 128, 266 -> 208 us (164 us without the ratio).
      const int box = min(a.s2n_size, N), j = tid % N;
      auto in_box = [&](int at, int peak) { return box >= 0 && ((at - peak + box) & (N - 1)) <= 2 * box; };
      const bool col_in = in_box(j, S.pj[0]);
      float second = -INFINITY;
#pragma unroll 8
      for (int i = tid / N; i < N; i += NT / N) {
        const float v = corr_at<N, float>(buf, i, j, SS);
        if (!(col_in && in_box(i, S.pi[0]))) second = fmaxf(second, v);
      }
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) second = fmaxf(second, __shfl_xor_sync(~0u, second, o));
      if (lane == 0) second_part[warp] = second;
      __syncthreads();
      if (tid == 0)
        for (int w = 1; w < NW; ++w) second_part[0] = fmaxf(second_part[0], second_part[w]);
      corr_outputs<C>(a, buf, S, slot, total, second_part);
    } else {
      corr_outputs<C>(a, buf, S, slot, total);
      if (a.s2n) __syncthreads();
    }
    // The next window's means need two barriers before its pixels replace
    // this window's map, so the fit above is done by then.
  }
}

// ---------------------------------------------------------------------------
// N = 32: one warp per window, line l in lane l.
// ---------------------------------------------------------------------------
static constexpr int kWarpFftWarps = 4, kWarpFftCtas = 4;

template <bool SEARCH = false, typename X = float>
__global__ void __launch_bounds__(32 * kWarpFftWarps, kWarpFftCtas) k_corr_fft_warp32(CorrArgs a) {
  constexpr int N = 32, SS = 16, PAD = 8, LD = N + 1;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Cplx<float>* buf = reinterpret_cast<Cplx<float>*>(smem_raw) + warp * N * LD;
  const long long total = a.win_list ? (long long)*a.win_count : (long long)a.n_pairs * a.m * a.n;
  const float inv_nn = 1.0f / (float)(N * N);
  const bool ties = a.near_tie || a.tie_count;
  for (long long slot = (long long)blockIdx.x * kWarpFftWarps + warp; slot < total;
       slot += (long long)gridDim.x * kWarpFftWarps) {
    const long long g = a.win_list ? (long long)a.win_list[slot] : slot;
    long long base;
    const bool ok = window_corner(a, g, base) || SEARCH;  // the search's passes have no mask
    // Pixels e = lane + 32 v + 128 q: the sums of the general kernel's 128
    // threads (pairs e, e + 128), then its four warps in order.
    X xa[8], xb[8];
    load_window<X, SEARCH>(
        a, base, ok, [&](int k) { return (long long)((lane + 32 * k) / SS) * a.width + (lane + 32 * k) % SS; }, xa, xb);
    float ma = 0.f, mb = 0.f, fa = 0.f, fb = 0.f;
    double da = 0.0, db = 0.0;
    if constexpr (!SEARCH) {
      float ta = 0.f, tb = 0.f;
#pragma unroll
      for (int v = 0; v < 4; ++v) {
        ta += warp_sum(xa[v] + xa[v + 4]);
        tb += warp_sum(xb[v] + xb[v + 4]);
      }
      ma = ta / (float)(SS * SS);
      mb = tb / (float)(SS * SS);
    } else {
      if constexpr (sizeof(X) == 4) {
        int sa = 0, sb = 0;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          sa += (int)xa[k];
          sb += (int)xb[k];
        }
        da = (double)__reduce_add_sync(~0u, sa);
        db = (double)__reduce_add_sync(~0u, sb);
      } else {
#pragma unroll
        for (int k = 0; k < 8; ++k) {
          da += xa[k];
          db += xb[k];
        }
        da = warp_sum(da);
        db = warp_sum(db);
      }
      da /= (double)(SS * SS);
      db /= (double)(SS * SS);
      ma = (float)rint(da);
      mb = (float)rint(db);
      fa = (float)(da - rint(da));
      fb = (float)(db - rint(db));
    }
    float va[8], vb[8], na = 0.f, nb = 0.f;  // search: sums of squares
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      if constexpr (sizeof(X) == 8) {
        va[k] = (float)(xa[k] - da);
        vb[k] = (float)(xb[k] - db);
      } else {
        va[k] = less_mean<SEARCH>(xa[k], ma, fa);
        vb[k] = less_mean<SEARCH>(xb[k], mb, fb);
      }
      if (!ok) va[k] = vb[k] = 0.f;
      if (SEARCH) {
        na = fmaf(va[k], va[k], na);
        nb = fmaf(vb[k], vb[k], nb);
      }
    }
    float scale_a = 1.f, scale_b = 1.f, gap = 0.f;
    if constexpr (SEARCH) {
      na = warp_sum(na);
      nb = warp_sum(nb);
      scale_a = search_scale(na);
      scale_b = search_scale(nb);
      gap = search_gap(na, nb, scale_a, scale_b);
    }
    __syncwarp();  // the previous window's map has been read
#pragma unroll
    for (int k = 0; k < 8; ++k) {
      const int e = lane + 32 * k, r = e / SS, c = e % SS;
      if (SEARCH) {
        va[k] *= scale_a;
        vb[k] *= scale_b;
      }
      buf[(PAD + r) * LD + PAD + c] = cmake<float>(va[k], vb[k]);
    }
    __syncwarp();
    Cplx<float> x[N];
    // Rows of the window (lanes 0 .. 15).
    if (lane < SS) {
      Cplx<float>* p = buf + (PAD + lane) * LD;
#pragma unroll
      for (int k = PAD; k < PAD + SS; ++k) x[k] = p[k];
      dft_half<N>(x);
#pragma unroll
      for (int k = 0; k < N; ++k) p[k] = x[k];
    }
    __syncwarp();
    // Columns.
#pragma unroll
    for (int k = PAD; k < PAD + SS; ++k) x[k] = buf[k * LD + lane];
    dft_half<N>(x);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < N; ++k) buf[k * LD + lane] = x[k];
    __syncwarp();
    // Product with the column of the negated frequency (read in place), then
    // the inverse along the columns.
    const int cm = (N - lane) & (N - 1);
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = conj_product(x[k], buf[((N - k) & (N - 1)) * LD + cm]);
    dft_k<N, true>(x);
    __syncwarp();
#pragma unroll
    for (int k = 0; k < N; ++k) buf[k * LD + lane] = x[k];
    __syncwarp();
    // Rows: real parts, scaled, with the line's two largest values.
#pragma unroll
    for (int k = 0; k < N; ++k) x[k] = buf[lane * LD + k];
    dft_k<N, true>(x);
    const int i = lane ^ (N / 2);
    Top2 top;
    top.init();
    float sum = 0.f;
#pragma unroll
    for (int q = 0; q < N; ++q) {
      float v = x[q ^ (N / 2)].x * inv_nn;
      buf[lane * LD + (q ^ (N / 2))].x = v;
      sum += v;
      if (i == 0 || q == 0) v = 0.f;  // no window overlap
      top.next(v, i * N + q);
    }
    const bool bad = __any_sync(~0u, is_nan(sum));
    __syncwarp();
    if (bad) {
      // Values that are not numbers: the general search's order.
      float bv = -INFINITY, sv = -INFINITY;
      int bi = 0x7fffffff;
      for (int f = lane; f < N * N; f += 32) {
        const float v = corr_at<N, float>(buf, f / N, f % N, SS);
        if (argmax_better(v, f, bv, bi)) { sv = bv; bv = v; bi = f; }
        else if (v > sv) sv = v;
      }
      warp_argmax2(bv, bi, sv);
      top.best = bv;
      top.second = sv;
      top.at = bi;
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        Top2 t;
        t.best = __shfl_xor_sync(~0u, top.best, o);
        t.second = __shfl_xor_sync(~0u, top.second, o);
        t.at = __shfl_xor_sync(~0u, top.at, o);
        top.merge(t);
      }
    }
    if constexpr (SEARCH) {
      if (lane == 0) {
        a.peak_i[g] = top.at / N;
        a.peak_j[g] = top.at % N;
        if (a.near_tie) a.near_tie[g] = 0;
      }
      if (bad || !(top.best - top.second > gap)) {
        const float from = bad ? INFINITY : top.best - gap;
        int count = 0, at[kCandMax];
        // Candidates in map order, counted by every lane.
        for (int f0 = 0; f0 < N * N && from > -INFINITY; f0 += 32) {
          const int f = f0 + lane;
          unsigned hit = __ballot_sync(~0u, corr_at<N, float>(buf, f / N, f % N, SS) >= from);
          while (hit) {
            const int k = __ffs(hit) - 1;
            hit &= hit - 1;
#pragma unroll
            for (int q = 0; q < kCandMax; ++q)
              if (q == count) at[q] = f0 + k;
            ++count;
          }
        }
        if (lane == 0) search_open(a, g, count, at);
      }
      continue;
    }
    if (a.maps) {
      float* mo = reinterpret_cast<float*>(a.maps) + g * N * N;
      for (int f = lane; f < N * N; f += 32) mo[f] = corr_at<N, float>(buf, f / N, f % N, SS);
    }
    const int pi = top.at / N, pj = top.at % N;
    const bool inner = pi > 0 && pi < N - 1 && pj > 0 && pj < N - 1;
    if (lane == 0) {
      float isp = (float)pi, jsp = (float)pj;
      if (inner)
        subpixel_fit(a.subpixel, pi, pj, corr_at<N, float>(buf, pi, pj, SS), corr_at<N, float>(buf, pi - 1, pj, SS),
                     corr_at<N, float>(buf, pi + 1, pj, SS), corr_at<N, float>(buf, pi, pj - 1, SS),
                     corr_at<N, float>(buf, pi, pj + 1, SS), isp, jsp);
      reinterpret_cast<float*>(a.u)[g] = ok ? sub_rn(jsp, (float)(N / 2)) : NAN;
      reinterpret_cast<float*>(a.v)[g] = ok ? sub_rn(isp, (float)(N / 2)) : NAN;
      if (a.peak_i) a.peak_i[g] = pi;
      if (a.peak_j) a.peak_j[g] = pj;
      if (ties) {
        const float gap = top.best - top.second;
        const bool tie = ok && !(gap > a.tie_tol * fabsf(top.best));
        if (a.near_tie) a.near_tie[g] = tie ? 1 : 0;
        if (tie && a.tie_count) atomicAdd(a.tie_count, 1);
      }
    }
  }
}

template <class H, bool SEARCH = false, typename X = float>
static int launch_corr_fft_half(const CorrArgs& a, cudaStream_t stream) {
  using L = FftLayout<typename H::Fft>;
  const long long total = (long long)a.n_pairs * a.m * a.n;
  if (total == 0) return PIV_OK;
  static thread_local int configured_dev = -1;
  static thread_local int per_sm = 1;
  int dev = 0;
  cudaGetDevice(&dev);
  if (configured_dev != dev) {
    cudaError_t e = cudaFuncSetAttribute(k_corr_fft_half<H, SEARCH, X>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)L::SMEM);
    if (e != cudaSuccess) return set_cuda_error(e, "cudaFuncSetAttribute(k_corr_fft_half)");
    per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_corr_fft_half<H, SEARCH, X>, H::NT, L::SMEM);
    if (per_sm < 1) per_sm = 1;
    configured_dev = dev;
  }
  const long long room = (long long)sm_count() * per_sm;
  CorrArgs b = a;
  b.tie_tol = kTieTolF32;
  k_corr_fft_half<H, SEARCH, X><<<(unsigned)std::min(total, room), H::NT, L::SMEM, stream>>>(b);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_corr_fft_half launch");
}

template <bool SEARCH = false, typename X = float>
static int launch_corr_fft_warp32(const CorrArgs& a, cudaStream_t stream) {
  const long long total = (long long)a.n_pairs * a.m * a.n;
  if (total == 0) return PIV_OK;
  constexpr int smem = kWarpFftWarps * 32 * 33 * (int)sizeof(Cplx<float>);
  static_assert(smem <= 48 * 1024, "fits the default shared memory");
  const long long blocks = (total + kWarpFftWarps - 1) / kWarpFftWarps;
  const long long room = (long long)sm_count() * kWarpFftCtas;
  CorrArgs b = a;
  b.tie_tol = kTieTolF32;
  k_corr_fft_warp32<SEARCH, X><<<(unsigned)std::min(blocks, room), 32 * kWarpFftWarps, smem, stream>>>(b);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? PIV_OK : set_cuda_error(e, "k_corr_fft_warp32 launch");
}

// Passes that the kernels above take (float32 passes; the search of float64
// passes on the same windows).
static bool corr_fft_half_windows(const CorrArgs& a) {
  return (a.fft_size == 32 || a.fft_size == 64 || a.fft_size == 128) &&
         a.fft_size == 2 * a.ss && a.ws == a.ss;
}

// Threads per CTA: N = 64 six CTAs of 128 per SM (four or five: 72, 70 us); N
// = 128, whose map takes most of an SM's shared memory, 512 (256 threads 95
// us, 1024 with 64 registers each 133 us).
template <bool SEARCH, typename X>
static int correlate_fft_half(const CorrArgs& a, cudaStream_t stream) {
  if (a.fft_size == 32) return launch_corr_fft_warp32<SEARCH, X>(a, stream);
  if (a.fft_size == 64) return launch_corr_fft_half<HalfCfg<64, 128, sizeof(X) == 8 ? 4 : 6>, SEARCH, X>(a, stream);
  return launch_corr_fft_half<HalfCfg<128, 512, 1>, SEARCH, X>(a, stream);
}

}  // namespace piv
