// dg_adjoint.cuh -- reverse-mode derivative of the subset objective.
//
// For each subset the forward map is the path of the correlation engine:
// warp of the subset pixels by the shape function (affine or quadratic,
// DICe_LocalShapeFunction.cpp:220-248, 509-520), Keys fourth-order
// interpolation of the deformed image (DICe_Image.cpp:834-883) and the
// objective over the active pixels, either
//   objective 0: gamma = sum (G~/|G~| - F~/|F~|)^2 = 2 - 2 S / (|G~| |F~|)
//                (Objective::gamma, DICe_Objective.cpp:58-76, with
//                G~ = G - mean G, F~ = F - mean F, S = sum G~ F~), or
//   objective 1: C = sum (G~ - F~)^2, the least-squares objective whose
//                Gauss-Newton right-hand side q (DICe_Objective.cpp:523-546)
//                is dC/dp / 2.
// Both are functions of G only through dObj/dG_i = a F~_i + b G~_i (the
// derivatives of the means cancel because sum G~ = sum F~ = 0):
//   gamma: a = -2 / (|G~| |F~|), b = 2 S / (|G~|^3 |F~|);   C: a = -2, b = 2.
// One warp per subset, two passes: the moments give the objective and (a, b);
// the second pass forms lambda_i = seed * (a F~_i + b G~_i), accumulates
// dObj/dp = sum lambda_i dG_i/dp (dG/dp = the shape-function Jacobian applied
// to the interpolant's spatial derivative) and scatters lambda_i times the 36
// interpolation weights into dObj/dI for the deformed image.
//
// The spatial derivative is either the exact derivative of the Keys
// interpolant (grad_source 0: what finite differences of the forward map
// measure) or the Keys interpolation of the gradient images (grad_source 1:
// the Gauss-Newton residual's approximation, DICe_LocalShapeFunction.cpp:
// 350-396, which makes dC/dp equal 2 q exactly).  The 4-pixel border
// deactivation (DICe_Subset.cpp:408) is piecewise constant in the
// parameters and contributes no derivative.
#pragma once

#include "dg_device.cuh"

namespace dg {

struct AdjointArgs {
  DevParams P;
  DevImage ref;
  DevImage def;            // I plane; gx / gy planes for grad_source 1
  DevGeometry geo;
  const double* fields;    // n x DICEGPU_FIELD_STRIDE: parameters per subset
  const double* seed;      // dL/dObj per subset (nullptr: 1)
  int n;
  int objective;           // 0 gamma, 1 least squares
  int grad_source;         // 0 interpolant derivative, 1 interpolated gradient images
  double* value_out;       // n objective values (nullptr: skip)
  double* dparams_out;     // n x 12 derivatives in slot order (nullptr: skip)
  float* ddef;             // W x H accumulated derivative (nullptr: skip)
};

// Derivatives of the Keys kernel pieces (DICe_Image.cpp:114-122): for
// s in [0,1) 4 s^2 - 14/3 s; [1,2) -7/4 s^2 + 6 s - 59/12; [2,3) 1/4 s^2 - 4/3 s + 7/4.
__device__ __forceinline__ float dkeys0(float s) { return fmaf(4.0f, s, -14.0f / 3.0f) * s; }
__device__ __forceinline__ float dkeys1(float s) { return fmaf(fmaf(-1.75f, s, 6.0f), s, -59.0f / 12.0f); }
__device__ __forceinline__ float dkeys2(float s) { return fmaf(fmaf(0.25f, s, -4.0f / 3.0f), s, 1.75f); }
// d/dt of keys_weights(t, w)
__device__ __forceinline__ void dkeys_weights(float t, float d[6]) {
  d[0] = dkeys2(t + 2.0f);
  d[1] = dkeys1(t + 1.0f);
  d[2] = dkeys0(t);
  d[3] = -dkeys0(1.0f - t);
  d[4] = -dkeys1(2.0f - t);
  d[5] = -dkeys2(3.0f - t);
}

template <int SHAPE>
__device__ __forceinline__ void adjoint_slots(const double* f, float* slots) {
#pragma unroll
  for (int i = 0; i < 12; ++i) slots[i] = 0.0f;
  if (SHAPE == DICEGPU_QUADRATIC_SF) {
#pragma unroll
    for (int i = 0; i < 12; ++i) slots[i] = (float)f[DICEGPU_F_QUAD_A + i];
  } else {
#pragma unroll
    for (int i = 0; i < 6; ++i) slots[i] = (float)f[DICEGPU_F_DISP_X + i];
  }
}

// The objective's value and the weights of dObj/dG_i from the lanes' moments.
struct AdjointWeights {
  double value, a, b, mF, mG;
  bool valid;
};
__device__ __forceinline__ AdjointWeights adjoint_weights(const AdjointArgs& A, int idx, double n, double sF, double sF2,
                                                          double sG, double sG2, double sGF) {
  n = warp_sum(n);
  sF = warp_sum(sF);
  sF2 = warp_sum(sF2);
  sG = warp_sum(sG);
  sG2 = warp_sum(sG2);
  sGF = warp_sum(sGF);
  AdjointWeights w;
  w.mF = n > 0.0 ? sF / n : 0.0;
  w.mG = n > 0.0 ? sG / n : 0.0;
  const double ff = sF2 - n * w.mF * w.mF, gg = sG2 - n * w.mG * w.mG, S = sGF - n * w.mG * w.mF;
  w.valid = n > 0.0;
  w.a = w.b = 0.0;
  if (A.objective == 0) {
    w.valid = w.valid && ff > 0.0 && gg > 0.0;
    const double nf = sqrt(ff), ng = sqrt(gg);
    w.value = w.valid ? 2.0 - 2.0 * S / (ng * nf) : -1.0;
    if (w.valid) {
      w.a = -2.0 / (ng * nf);
      w.b = 2.0 * S / (gg * ng * nf);
    }
  } else {
    w.value = w.valid ? gg + ff - 2.0 * S : -1.0;
    w.a = -2.0;
    w.b = 2.0;
  }
  const double sd = A.seed ? A.seed[idx] : 1.0;
  w.a *= sd;
  w.b *= sd;
  return w;
}
__device__ __forceinline__ void adjoint_store(const AdjointArgs& A, int idx, const AdjointWeights& w, double* dp) {
  const int lane = threadIdx.x & 31;
  if (A.dparams_out) {
#pragma unroll
    for (int i = 0; i < 12; ++i) dp[i] = warp_sum(dp[i]);
    if (lane == 0) {
#pragma unroll
      for (int i = 0; i < 12; ++i) A.dparams_out[(size_t)idx * 12 + i] = dp[i];
    }
  }
  if (A.value_out && lane == 0) A.value_out[idx] = w.value;
}

template <int SHAPE>
__device__ void adjoint_subset(const AdjointArgs& A, int idx) {
  const int lane = threadIdx.x & 31;
  const double* f = A.fields + (size_t)idx * DICEGPU_FIELD_STRIDE;
  const int cx = (int)f[DICEGPU_F_COORD_X], cy = (int)f[DICEGPU_F_COORD_Y];
  const float fcx = (float)cx, fcy = (float)cy;
  float slots[12];
  adjoint_slots<SHAPE>(f, slots);
  MapConst k;
  make_mapconst<SHAPE>(slots, false, fcx, fcy, k);
  int npix, off;
  if (A.geo.half >= 0) {
    const int side = 2 * A.geo.half + 1;
    npix = side * side;
    off = -1;
  } else {
    off = A.geo.offsets[idx];
    npix = A.geo.offsets[idx + 1] - off;
  }
  const int W = A.def.w, H = A.def.h;
  const long rlim = (long)A.ref.w * A.ref.h;
  auto pixel = [&](int p, int& x, int& y) {
    if (off < 0) {
      const int side = 2 * A.geo.half + 1;
      const int row = p / side;
      x = cx - A.geo.half + (p - row * side);
      y = cy - A.geo.half + row;
    } else {
      x = __ldg(A.geo.px + off + p);
      y = __ldg(A.geo.py + off + p);
    }
    x = max(x, 0);
    y = max(y, 0);
  };
  // pass 1: moments over the active pixels
  double n = 0.0, sF = 0.0, sF2 = 0.0, sG = 0.0, sG2 = 0.0, sGF = 0.0;
  for (int p = lane; p < npix; p += 32) {
    int x, y;
    pixel(p, x, y);
    float mx, my, Dx, Dy;
    map_offset<SHAPE>(k, __fsub_rn((float)x, fcx), __fsub_rn((float)y, fcy), fcx, fcy, mx, my, Dx, Dy);
    const int px = round_pixel(mx), py = round_pixel(my);
    if (px < 4 || px >= W - 4 || py < 4 || py >= H - 4) continue;
    const long ri = (long)y * A.ref.w + x;
    const double F = ri < rlim ? (double)__ldg(A.ref.I + ri) : 0.0;
    float G, gdum, hdum;
    keys_fast_interior<false>(A.def, mx, my, G, gdum, hdum);
    n += 1.0;
    sF += F;
    sF2 += F * F;
    sG += (double)G;
    sG2 += (double)G * (double)G;
    sGF += (double)G * F;
  }
  const AdjointWeights w = adjoint_weights(A, idx, n, sF, sF2, sG, sG2, sGF);
  const bool valid = w.valid;
  const double a = w.a, b = w.b, mF = w.mF, mG = w.mG;
  double dp[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) dp[i] = 0.0;
  if (valid && (A.dparams_out || A.ddef)) {
    // pass 2: lambda_i, dObj/dp and the scatter into dObj/dI
    for (int p = lane; p < npix; p += 32) {
      int x, y;
      pixel(p, x, y);
      const float dxf = __fsub_rn((float)x, fcx), dyf = __fsub_rn((float)y, fcy);
      float mx, my, Dx, Dy;
      map_offset<SHAPE>(k, dxf, dyf, fcx, fcy, mx, my, Dx, Dy);
      const int px = round_pixel(mx), py = round_pixel(my);
      if (px < 4 || px >= W - 4 || py < 4 || py >= H - 4) continue;
      const long ri = (long)y * A.ref.w + x;
      const double F = ri < rlim ? (double)__ldg(A.ref.I + ri) : 0.0;
      const int ix = (int)mx, iy = (int)my;
      float wx[6], wy[6], dwx[6], dwy[6];
      keys_weights(mx - (float)ix, wx);
      keys_weights(my - (float)iy, wy);
      dkeys_weights(mx - (float)ix, dwx);
      dkeys_weights(my - (float)iy, dwy);
      const size_t base = (size_t)(iy - 2) * W + (ix - 2);
      float G = 0.0f, gx = 0.0f, gy = 0.0f;
#pragma unroll
      for (int m = 0; m < 6; ++m) {
        float rI = 0.0f, rdx = 0.0f, rgx = 0.0f, rgy = 0.0f;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
          const size_t t = base + (size_t)m * W + q;
          const float v = __ldg(A.def.I + t);
          rI = fmaf(wx[q], v, rI);
          if (A.grad_source == 0) {
            rdx = fmaf(dwx[q], v, rdx);
          } else {
            rgx = fmaf(wx[q], __ldg(A.def.gx + t), rgx);
            rgy = fmaf(wx[q], __ldg(A.def.gy + t), rgy);
          }
        }
        G = fmaf(wy[m], rI, G);
        if (A.grad_source == 0) {
          gx = fmaf(wy[m], rdx, gx);
          gy = fmaf(dwy[m], rI, gy);
        } else {
          gx = fmaf(wy[m], rgx, gx);
          gy = fmaf(wy[m], rgy, gy);
        }
      }
      const double lam = a * (F - mF) + b * ((double)G - mG);
      if (A.dparams_out) {
        float r[12];
        residuals_D<SHAPE>(k, dxf, dyf, Dx, Dy, gx, gy, false, r);
        constexpr int NS = SHAPE == DICEGPU_QUADRATIC_SF ? 12 : 6;
#pragma unroll
        for (int i = 0; i < NS; ++i) dp[i] = fma(lam, (double)r[i], dp[i]);
      }
      if (A.ddef) {
        const float lf = (float)lam;
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          const float lm = lf * wy[m];
#pragma unroll
          for (int q = 0; q < 6; ++q) atomicAdd(A.ddef + base + (size_t)m * W + q, lm * wx[q]);
        }
      }
    }
  }
  adjoint_store(A, idx, w, dp);
}

// Square subsets with the image derivative: a lane walks down one column of the subset (narrow subsets:
// of one of several bands of rows), a row per step, and keeps in registers the
// 6 x 6 window of taps and the 36 sums of the scatter that the window's pixels
// are due.  From one row to the next both slide by one row as long as no lane
// crosses a pixel boundary sideways or skips a row (a few steps of a
// subset): 6 taps are loaded and 6 sums go to the image per pixel instead of
// 36 and 36.  (A pixel per lane in reading order, 36 loads and 36 atomics: 657 us
// for 19,600 25 x 25 subsets, bound by the L1's wavefronts; the operations
// per value are the same.)  Subsets far from a translation, whose windows seldom
// slide, are left to adjoint_distorted_kernel.
template <int SHAPE>
struct AdjointColumn {
  const AdjointArgs& A;
  const MapConst& k;
  const int cx, cy, side, lane, W, H;
  int rows, band;      // steps, and this lane's first row
  bool has;            // the lane has a column in this chunk
  int col;
  // the pixel of the step
  bool live;
  float dxf, dyf, Dx, Dy, mx, my;
  int x, y, ix, iy;
  // the window: valid for base (pix, piy) when had
  bool had;
  int pix, piy;
  float v[6][6];

  __device__ __forceinline__ AdjointColumn(const AdjointArgs& a, const MapConst& mk, int cx_, int cy_)
      : A(a), k(mk), cx(cx_), cy(cy_), side(2 * a.geo.half + 1), lane(threadIdx.x & 31), W(a.def.w), H(a.def.h) {}
  __device__ __forceinline__ int chunks() const { return (side + 31) / 32; }
  __device__ __forceinline__ void start(int chunk) {
    const int bands = side >= 32 ? 1 : 32 / side;
    rows = (side + bands - 1) / bands;
    const int b = side >= 32 ? 0 : lane / side;
    col = chunk * 32 + lane - b * side;
    band = b * rows;
    has = b < bands && col < side;
    had = false;
  }
  // the step's pixel; uniform across the warp but for has / live
  __device__ __forceinline__ void place(int r) {
    live = has && r < rows && band + r < side;
    x = max(cx - A.geo.half + col, 0);
    y = max(cy - A.geo.half + band + r, 0);
    dxf = __fsub_rn((float)x, (float)cx);
    dyf = __fsub_rn((float)y, (float)cy);
    map_offset<SHAPE>(k, dxf, dyf, (float)cx, (float)cy, mx, my, Dx, Dy);
    const int px = round_pixel(mx), py = round_pixel(my);
    live = live && !(px < 4 || px >= W - 4 || py < 4 || py >= H - 4);
    ix = (int)mx;
    iy = (int)my;
  }
  // whether every lane's window (and scatter sums) slide by one row
  __device__ __forceinline__ bool slides() const {
    return __all_sync(FULL, live ? had && ix == pix && iy == piy + 1 : !had);
  }
  __device__ __forceinline__ void window(bool slide) {
    if (live) {
      const float* q = A.def.I + (size_t)(iy - 2) * W + (ix - 2);
      if (slide) {
#pragma unroll
        for (int m = 0; m < 5; ++m)
#pragma unroll
          for (int t = 0; t < 6; ++t) v[m][t] = v[m + 1][t];
#pragma unroll
        for (int t = 0; t < 6; ++t) v[5][t] = __ldg(q + 5 * (size_t)W + t);
      } else {
#pragma unroll
        for (int m = 0; m < 6; ++m)
#pragma unroll
          for (int t = 0; t < 6; ++t) v[m][t] = __ldg(q + (size_t)m * W + t);
      }
    }
  }
  __device__ __forceinline__ void done() {
    had = live;
    pix = ix;
    piy = iy;
  }
};

// Whether the magnitudes of the displacement's gradients (at the centre) add
// up to more than 0.34.  Columns and pixels, us for 19,600 25 px subsets: sum 0.
// 597 and 670; 0.23 962 and 980; 0.33 815 and 815; 0.35 1,035 and 940; 0.46 1,362
// and 1,160; rotations of 0.4, 0.79 and 1.57 rad 1,718 and 1,435, 2,625 and
// 2,180, 4,940 and 4,030.  (15 px, 0.79 rad: 1,370 and 930.)
template <int SHAPE>
__device__ __forceinline__ bool adjoint_distorted(const float* s) {
  const float sum = SHAPE == DICEGPU_QUADRATIC_SF ? fabsf(s[0] - 1.0f) + fabsf(s[1]) + fabsf(s[6]) + fabsf(s[7] - 1.0f)
                                                  : 2.0f * fmaxf(fabsf(s[2]), fabsf(s[5])) + fabsf(s[3]) + fabsf(s[4]);
  return !(sum <= 0.34f);
}

template <int SHAPE>
__device__ void adjoint_square(const AdjointArgs& A, int idx) {
  const double* f = A.fields + (size_t)idx * DICEGPU_FIELD_STRIDE;
  const int cx = (int)f[DICEGPU_F_COORD_X], cy = (int)f[DICEGPU_F_COORD_Y];
  const float fcx = (float)cx, fcy = (float)cy;
  float slots[12];
  adjoint_slots<SHAPE>(f, slots);
  MapConst k;
  make_mapconst<SHAPE>(slots, false, fcx, fcy, k);
  const bool distorted = adjoint_distorted<SHAPE>(slots);
  AdjointColumn<SHAPE> c(A, k, cx, cy);
  const long rlim = (long)A.ref.w * A.ref.h;
  // pass 1: moments over the active pixels
  double n = 0.0, sF = 0.0, sF2 = 0.0, sG = 0.0, sG2 = 0.0, sGF = 0.0;
  // (left here, after the map's constants: before them it costs 4 us of 598,
  // the field row's loads no longer overlapping)
  if (distorted) return;
#pragma unroll 1
  for (int chunk = 0; chunk < c.chunks(); ++chunk) {
    c.start(chunk);
#pragma unroll 1
    for (int r = 0; r < c.rows; ++r) {
      c.place(r);
      c.window(c.slides());
      if (c.live) {
        const long ri = (long)c.y * A.ref.w + c.x;
        const double F = ri < rlim ? (double)__ldg(A.ref.I + ri) : 0.0;
        float wx[6], wy[6], G = 0.0f;
        keys_weights(c.mx - (float)c.ix, wx);
        keys_weights(c.my - (float)c.iy, wy);
#pragma unroll
        for (int m = 0; m < 6; ++m) {
          float row = 0.0f;
#pragma unroll
          for (int t = 0; t < 6; ++t) row = fmaf(wx[t], c.v[m][t], row);
          G = fmaf(wy[m], row, G);
        }
        n += 1.0;
        sF += F;
        sF2 += F * F;
        sG += (double)G;
        sG2 += (double)G * (double)G;
        sGF += (double)G * F;
      }
      c.done();
    }
  }
  AdjointWeights w = adjoint_weights(A, idx, n, sF, sF2, sG, sG2, sGF);
  double dp[12];
#pragma unroll
  for (int i = 0; i < 12; ++i) dp[i] = 0.0;
  if (w.valid) {
    // pass 2: lambda_i, dObj/dp and the scatter into dObj/dI
#pragma unroll 1
    for (int chunk = 0; chunk < c.chunks(); ++chunk) {
      c.start(chunk);
      float acc[6][6];
#pragma unroll
      for (int m = 0; m < 6; ++m)
#pragma unroll
        for (int t = 0; t < 6; ++t) acc[m][t] = 0.0f;
      // one step more than rows: it finds no lane live and empties the sums
#pragma unroll 1
      for (int r = 0; r <= c.rows; ++r) {
        c.place(r);
        const bool slide = c.slides();
        if (c.had) {
          float* o = A.ddef + (size_t)(c.piy - 2) * c.W + (c.pix - 2);
#pragma unroll
          for (int t = 0; t < 6; ++t) atomicAdd(o + t, acc[0][t]);
          if (slide) {
#pragma unroll
            for (int m = 0; m < 5; ++m)
#pragma unroll
              for (int t = 0; t < 6; ++t) acc[m][t] = acc[m + 1][t];
#pragma unroll
            for (int t = 0; t < 6; ++t) acc[5][t] = 0.0f;
          } else {
#pragma unroll
            for (int m = 1; m < 6; ++m)
#pragma unroll
              for (int t = 0; t < 6; ++t) atomicAdd(o + (size_t)m * c.W + t, acc[m][t]);
#pragma unroll
            for (int m = 0; m < 6; ++m)
#pragma unroll
              for (int t = 0; t < 6; ++t) acc[m][t] = 0.0f;
          }
        }
        c.window(slide);
        if (c.live) {
          const long ri = (long)c.y * A.ref.w + c.x;
          const double F = ri < rlim ? (double)__ldg(A.ref.I + ri) : 0.0;
          float wx[6], wy[6], dwx[6], dwy[6];
          keys_weights(c.mx - (float)c.ix, wx);
          keys_weights(c.my - (float)c.iy, wy);
          dkeys_weights(c.mx - (float)c.ix, dwx);
          dkeys_weights(c.my - (float)c.iy, dwy);
          float G = 0.0f, gx = 0.0f, gy = 0.0f;
          const size_t base = (size_t)(c.iy - 2) * c.W + (c.ix - 2);
#pragma unroll
          for (int m = 0; m < 6; ++m) {
            float rI = 0.0f, rdx = 0.0f;
#pragma unroll
            for (int t = 0; t < 6; ++t) {
              rI = fmaf(wx[t], c.v[m][t], rI);
              rdx = fmaf(dwx[t], c.v[m][t], rdx);
            }
            G = fmaf(wy[m], rI, G);
            gx = fmaf(wy[m], rdx, gx);
            gy = fmaf(dwy[m], rI, gy);
          }
          if (A.grad_source != 0) {
            gx = gy = 0.0f;
#pragma unroll 1
            for (int m = 0; m < 6; ++m) {
              float rgx = 0.0f, rgy = 0.0f, wm = 0.0f;
#pragma unroll
              for (int t = 0; t < 6; ++t) {
                rgx = fmaf(wx[t], __ldg(A.def.gx + base + (size_t)m * c.W + t), rgx);
                rgy = fmaf(wx[t], __ldg(A.def.gy + base + (size_t)m * c.W + t), rgy);
                if (t == m) wm = wy[t];
              }
              gx = fmaf(wm, rgx, gx);
              gy = fmaf(wm, rgy, gy);
            }
          }
          const double lam = w.a * (F - w.mF) + w.b * ((double)G - w.mG);
          if (A.dparams_out) {
            float rr[12];
            residuals_D<SHAPE>(k, c.dxf, c.dyf, c.Dx, c.Dy, gx, gy, false, rr);
            constexpr int NS = SHAPE == DICEGPU_QUADRATIC_SF ? 12 : 6;
#pragma unroll
            for (int i = 0; i < NS; ++i) dp[i] = fma(lam, (double)rr[i], dp[i]);
          }
          const float lf = (float)lam;
#pragma unroll
          for (int m = 0; m < 6; ++m) {
            const float lm = lf * wy[m];
#pragma unroll
            for (int t = 0; t < 6; ++t) acc[m][t] = fmaf(lm, wx[t], acc[m][t]);
          }
        }
        c.done();
      }
    }
  }
  adjoint_store(A, idx, w, dp);
}

// Launch bounds: three CTAs of four warps per SM, for the registers of the two
// windows.
template <int SHAPE>
__global__ void __launch_bounds__(128, 3) adjoint_square_kernel(const __grid_constant__ AdjointArgs a) {
  const int warps = (gridDim.x * blockDim.x) >> 5;
#pragma unroll 1
  for (int idx = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; idx < a.n; idx += warps) adjoint_square<SHAPE>(a, idx);
}

template <int SHAPE>
__global__ void __launch_bounds__(256) adjoint_kernel(const __grid_constant__ AdjointArgs a) {
  const int warps = (gridDim.x * blockDim.x) >> 5;
  for (int idx = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; idx < a.n; idx += warps)
    adjoint_subset<SHAPE>(a, idx);
}

// The squares that adjoint_square leaves, a pixel per lane: lane l of a warp
// looks at the warp's l-th next subset, and the warp takes those found.  A
// launch of its own (3 us when there are none): with both paths in one kernel,
// the columns lose 10 us of 598.
template <int SHAPE>
__global__ void __launch_bounds__(256) adjoint_distorted_kernel(const __grid_constant__ AdjointArgs a) {
  const int warps = (gridDim.x * blockDim.x) >> 5, lane = threadIdx.x & 31;
#pragma unroll 1
  for (long long first = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; first < a.n; first += 32LL * warps) {
    const long long mine = first + (long long)lane * warps;
    bool distorted = false;
    if (mine < a.n) {
      float slots[12];
      adjoint_slots<SHAPE>(a.fields + (size_t)mine * DICEGPU_FIELD_STRIDE, slots);
      distorted = adjoint_distorted<SHAPE>(slots);
    }
#pragma unroll 1
    for (unsigned left = __ballot_sync(FULL, distorted); left; left &= left - 1)
      adjoint_subset<SHAPE>(a, (int)first + (__ffs(left) - 1) * warps);
  }
}

}  // namespace dg
