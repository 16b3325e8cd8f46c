// k_loss.cu — SSIM loss and gradient on the device (loss.rs:22-375; the
// reference computes it on the CPU after reading the image back,
// train.rs:180-196).
//
// SSIM (Wang et al. 2004) over an 11-tap separable Gaussian window (sigma 1.5)
// with reflect-101 padding, C1 = 1e-4, C2 = 9e-4, per rgb channel; the loss is
// 1 - mean SSIM and its gradient is the reference's analytic form: coefficient
// planes P = dSSIM/dmu_x, Q = dSSIM/dsigma_x^2, R = dSSIM/dsigma_xy pulled back
// through the adjoint of the blur.  The reference pulls mu_x Q and mu_y R back
// too and adds P~ - 2 (mu_x Q)~ - (mu_y R)~; the adjoint is linear, so the
// plane P - 2 mu_x Q - mu_y R is formed per pixel and three planes per channel
// are stored and pulled back instead of five.
//
// Two kernels per call, each one CTA per 32x32 pixel tile of one view:
//   k_ssim_terms  stage the tile plus a 5-pixel reflected halo of prediction and
//                 target in shared memory, blur (horizontal then vertical, the
//                 reference's order and f32 rounding: no contraction) the five
//                 moments of the three channels, write the 9 coefficient planes
//                 and add the tile's SSIM-map sum to the view's f64 total;
//   k_ssim_grad   stage the coefficient planes with a 5-pixel halo (zero outside
//                 the image), apply the transposed blur as a gather (vertical
//                 then horizontal; near the border the reflected taps add their
//                 mirrored sources), combine with the prediction and target and
//                 add scale * dL/dC into dl_dc.
// Both are bound by instructions: a 32x32 tile computes 1.3 halo rows per row
// (2.25 with 8 rows), a thread slides over 12 or 14 staged values for 2 or 4
// outputs (8 or 4 in the adjoint) instead of 11 loads each, and the moments of
// x and y go as packed pairs.  2 views of 1237x822: terms 158 -> 79 us, gradient 422 ->
// 113 us.  The gradient's planes come by cp.async, the next channel's during the
// horizontal pass of this one, the prediction and target ahead of both passes, and the
// reflected taps are at most five, unrolled: 113 -> 98 us (103 without the last;
// two buffers of planes, with 3 CTAs per SM instead of 4, 111 us).
// Reflect-101 with a 5-pixel radius folds at most once for images of 6 or more
// pixels per side, which the host requires.
#include "sc_internal.cuh"

#include <cmath>

namespace sck {

namespace {

constexpr int SS_W = 11, SS_R = 5;
constexpr int SS_T = 32;               // tile side
constexpr int SS_H = SS_T + 2 * SS_R;  // staged side: 42
constexpr int SS_PLANES = 9;           // 3 per channel
constexpr float SS_C1 = 0.0001f, SS_C2 = 0.0009f;

struct SsimArgs {
  float g[SS_W];
  uint32_t w, h;
  uint64_t P;
  float scale;
  float inv_n;  // 1 / (w h) in f32
};

__device__ __forceinline__ int reflect101(int i, int n) {
  // single fold: i in [-(n-1), 2(n-1)]
  if (i < 0) i = -i;
  if (i >= n) i = 2 * (n - 1) - i;
  return i;
}

// reference rounding: every product and sum rounded separately
__device__ __forceinline__ float mul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float add(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float sub(float a, float b) { return __fsub_rn(a, b); }

struct TermsSmem {
  float2 xy[3][SS_H][SS_H];   // (prediction, target) per channel
  float2 h0[SS_H][SS_T];      // one channel's horizontally blurred (x, y),
  float2 h1[SS_H][SS_T];      // (x^2, y^2)
  float h2[SS_H][SS_T];       // and x y
};

__global__ void __launch_bounds__(256, 3) k_ssim_terms(const float4* __restrict__ pred,
                                                       const float* __restrict__ target, SsimArgs a,
                                                       float* __restrict__ terms, double* __restrict__ ssim_sum) {
  sc_after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TermsSmem& sm = *reinterpret_cast<TermsSmem*>(smem_raw);
  __shared__ double red[8];
  const uint32_t v = blockIdx.z;
  const int x0 = blockIdx.x * SS_T, y0 = blockIdx.y * SS_T;
  const int W = (int)a.w, H = (int)a.h;
  const float4* pv = pred + (uint64_t)v * a.P;
  const float* tv = target + (uint64_t)v * a.P * 3;
  const int tx = threadIdx.x & 31, ts = threadIdx.x >> 5;  // vertical pass: column, strip of 4 rows
  // a warp stages whole rows, 32 columns and then 10; clamped to the blur
  // footprint of the image first (columns past it feed no output pixel)
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int rx = tx + 32 * h;
    if (rx >= SS_H) break;
    const int gx = reflect101(min(x0 - SS_R + rx, W - 1 + SS_R), W);
#pragma unroll 3
    for (int ry = ts; ry < SS_H; ry += 8) {
      const int gy = reflect101(min(y0 - SS_R + ry, H - 1 + SS_R), H);
      const uint64_t p = (uint64_t)gy * W + gx;
      const float4 c = pv[p];
      const float* t = tv + 3 * p;
      sm.xy[0][ry][rx] = make_float2(c.x, t[0]);
      sm.xy[1][ry][rx] = make_float2(c.y, t[1]);
      sm.xy[2][ry][rx] = make_float2(c.z, t[2]);
    }
  }
  // the window's taps as pairs (it is symmetric)
  float2 g[SS_R + 1];
#pragma unroll
  for (int k = 0; k <= SS_R; ++k) g[k] = make_float2(a.g[k], a.g[k]);
  double local = 0.0;
  __syncthreads();
  for (int c = 0; c < 3; ++c) {
    // horizontal pass over every staged row: two output columns per task
    for (int t = threadIdx.x; t < SS_H * (SS_T / 2); t += 256) {
      const int ry = t / (SS_T / 2), x = 2 * (t - ry * (SS_T / 2));
      const float4* src = reinterpret_cast<const float4*>(&sm.xy[c][ry][x]);
      float2 s0[2], s1[2];
      float s2[2];
#pragma unroll
      for (int o = 0; o < 2; ++o) { s0[o] = s1[o] = make_float2(0.f, 0.f); s2[o] = 0.f; }
#pragma unroll
      for (int q = 0; q < SS_W / 2 + 1; ++q) {
        const float4 two = src[q];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
          const float2 p = e ? make_float2(two.z, two.w) : make_float2(two.x, two.y);
          const float2 pp = __fmul2_rn(p, p);
          const float pxy = mul(p.x, p.y);
#pragma unroll
          for (int o = 0; o < 2; ++o) {
            const int k = 2 * q + e - o;
            if (k < 0 || k >= SS_W) continue;
            const float2 gk = g[k <= SS_R ? k : SS_W - 1 - k];
            s0[o] = __fadd2_rn(s0[o], __fmul2_rn(p, gk));
            s1[o] = __fadd2_rn(s1[o], __fmul2_rn(pp, gk));
            s2[o] = add(s2[o], mul(pxy, gk.x));
          }
        }
      }
      *reinterpret_cast<float4*>(&sm.h0[ry][x]) = make_float4(s0[0].x, s0[0].y, s0[1].x, s0[1].y);
      *reinterpret_cast<float4*>(&sm.h1[ry][x]) = make_float4(s1[0].x, s1[0].y, s1[1].x, s1[1].y);
      *reinterpret_cast<float2*>(&sm.h2[ry][x]) = make_float2(s2[0], s2[1]);
    }
    __syncthreads();
    // vertical pass, SSIM map and coefficient planes: 4 rows of a column per thread
    float2 m0[4], m1[4];
    float m2[4];
#pragma unroll
    for (int o = 0; o < 4; ++o) { m0[o] = m1[o] = make_float2(0.f, 0.f); m2[o] = 0.f; }
#pragma unroll
    for (int r = 0; r < SS_W + 3; ++r) {
      const float2 a0 = sm.h0[4 * ts + r][tx], a1 = sm.h1[4 * ts + r][tx];
      const float a2 = sm.h2[4 * ts + r][tx];
#pragma unroll
      for (int o = 0; o < 4; ++o) {
        const int k = r - o;
        if (k < 0 || k >= SS_W) continue;
        const float2 gk = g[k <= SS_R ? k : SS_W - 1 - k];
        m0[o] = __fadd2_rn(m0[o], __fmul2_rn(a0, gk));
        m1[o] = __fadd2_rn(m1[o], __fmul2_rn(a1, gk));
        m2[o] = add(m2[o], mul(a2, gk.x));
      }
    }
#pragma unroll
    for (int o = 0; o < 4; ++o) {
      const int x = x0 + tx, y = y0 + 4 * ts + o;
      if (x < W && y < H) {
        const float mux = m0[o].x, muy = m0[o].y;
        const float mux2 = mul(mux, mux), muy2 = mul(muy, muy);
        const float sxx = sub(m1[o].x, mux2), syy = sub(m1[o].y, muy2), sxy = sub(m2[o], mul(mux, muy));
        const float av = add(mul(mul(2.0f, mux), muy), SS_C1);
        const float bv = add(mul(2.0f, sxy), SS_C2);
        const float cv = add(add(mux2, muy2), SS_C1);
        const float dv = add(add(sxx, syy), SS_C2);
        const float cd = mul(cv, dv);
        local += (double)__fdiv_rn(mul(av, bv), cd);
        const float pp = __fdiv_rn(mul(mul(2.0f, bv), sub(mul(muy, cv), mul(mux, av))), mul(cv, cd));
        const float qq = __fdiv_rn(mul(-av, bv), mul(cd, dv));
        const float rr = __fdiv_rn(mul(2.0f, av), cd);
        float* t = terms + ((uint64_t)v * SS_PLANES + c * 3) * a.P + (uint64_t)y * W + x;
        t[0] = sub(sub(pp, mul(2.0f, mul(mux, qq))), mul(muy, rr));
        t[a.P] = qq;
        t[2 * a.P] = rr;
      }
    }
    __syncthreads();
  }
  // block sum of the SSIM map -> one f64 atomic per block
  for (int o = 16; o > 0; o >>= 1) local += __shfl_xor_sync(0xffffffffu, local, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = local;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    atomicAdd(ssim_sum + v, s);
  }
}

constexpr int SS_S = 43;  // row stride: 4 rows' groups of 4 columns fall on different banks
struct GradSmem {
  float f[3][SS_H][SS_S];   // one channel's planes
  float vt[3][SS_T][SS_S];  // their vertical adjoint
};

// The taps of the transposed 1-D blur at index i along an axis of length n whose
// source index was reflected onto i (src[j - base] is source j): those below 0
// come back to 1..5, those beyond n - 1 to n - 6..n - 2.
template <int STRIDE>
__device__ __forceinline__ float reflected_taps(const float* src, int i, int n, int base, const float* g) {
  float acc = 0.f;
  if (i <= SS_R && i >= 1) {
#pragma unroll
    for (int k = 0; k < SS_R; ++k)
      if (k <= SS_R - i) acc += g[k] * src[(SS_R - i - k - base) * STRIDE];
  }
  if (i >= n - 1 - SS_R && i <= n - 2) {
#pragma unroll
    for (int k = SS_R + 1; k < SS_W; ++k) {
      const int j = 2 * (n - 1) - i - k + SS_R;
      if (j <= n - 1) acc += g[k] * src[(j - base) * STRIDE];
    }
  }
  return acc;
}

// Copies one channel's planes to shared memory (cp.async, zeros outside the image): a
// warp takes whole rows, 32 columns and then 10.
__device__ __forceinline__ void stage_planes(float (*f)[SS_H][SS_S], const float* __restrict__ tc, uint64_t P, int x0,
                                             int y0, int W, int H) {
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int rx = (threadIdx.x & 31) + 32 * h, gx = x0 - SS_R + rx;
    if (rx >= SS_H) break;
    const bool in_x = gx >= 0 && gx < W;
#pragma unroll 3
    for (int ry = threadIdx.x >> 5; ry < SS_H; ry += 8) {
      const int gy = y0 - SS_R + ry;
      const bool in = in_x && gy >= 0 && gy < H;
      const float* t = in ? tc + ((int64_t)gy * W + gx) : tc;  // nothing is read with a size of 0
#pragma unroll
      for (int pl = 0; pl < 3; ++pl)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(
                         (uint32_t)__cvta_generic_to_shared(&f[pl][ry][rx])),
                     "l"(t + pl * P), "r"(in ? 4 : 0)
                     : "memory");
    }
  }
}

__global__ void __launch_bounds__(256, 4) k_ssim_grad(const float4* __restrict__ pred,
                                                      const float* __restrict__ target, SsimArgs a,
                                                      const float* __restrict__ terms, float4* __restrict__ dl_dc) {
  sc_after_previous();
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradSmem& sm = *reinterpret_cast<GradSmem*>(smem_raw);
  const uint32_t v = blockIdx.z;
  const int x0 = blockIdx.x * SS_T, y0 = blockIdx.y * SS_T;
  const int W = (int)a.w, H = (int)a.h;
  const float* tv = terms + (uint64_t)v * SS_PLANES * a.P;
  const bool y_edge = y0 == 0 || y0 + SS_T + SS_R >= H, x_edge = x0 == 0 || x0 + SS_T + SS_R >= W;
  const int ty = threadIdx.x >> 3, tx = 4 * (threadIdx.x & 7);  // horizontal pass: row, 4 columns
  const int y = y0 + ty;
  stage_planes(sm.f, tv, a.P, x0, y0, W, H);
  float gout[3][4];
#pragma unroll
  for (int c = 0; c < 3; ++c) {
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    float xs[4], tg[4];  // this channel's prediction and target, on their way during both passes
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const bool in = x0 + tx + q < W && y < H;
      const uint64_t p = (uint64_t)v * a.P + (uint64_t)y * W + x0 + tx + q;
      xs[q] = in ? reinterpret_cast<const float*>(pred + p)[c] : 0.f;
      tg[q] = in ? target[3 * p + c] : 0.f;
    }
    // vertical adjoint: 8 rows of a staged column per task (sources outside the image are staged as zeros)
    for (int t = threadIdx.x; t < (SS_T / 8) * 3 * SS_H; t += 256) {
      const int strip = t / (3 * SS_H), rem = t - strip * (3 * SS_H);
      const int pl = rem / SS_H, rx = rem - pl * SS_H;
      float o[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) o[q] = 0.f;
#pragma unroll
      for (int r = 0; r < 8 + 2 * SS_R; ++r) {
        const float f = sm.f[pl][8 * strip + r][rx];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const int k = q - r + 2 * SS_R;  // output row q takes source row r of its staged 18 by tap k
          if (k >= 0 && k < SS_W) o[q] = fmaf(a.g[k], f, o[q]);
        }
      }
      if (y_edge) {
#pragma unroll
        for (int q = 0; q < 8; ++q)
          if (y0 + 8 * strip + q < H)
            o[q] += reflected_taps<SS_S>(&sm.f[pl][0][rx], y0 + 8 * strip + q, H, y0 - SS_R, a.g);
      }
#pragma unroll
      for (int q = 0; q < 8; ++q) sm.vt[pl][8 * strip + q][rx] = o[q];
    }
    __syncthreads();
    // the next channel's planes travel during the horizontal pass
    if (c < 2) stage_planes(sm.f, tv + (uint64_t)(3 * (c + 1)) * a.P, a.P, x0, y0, W, H);
    // horizontal adjoint of this channel's planes at 4 pixels
    float s[3][4];
#pragma unroll
    for (int pl = 0; pl < 3; ++pl) {
#pragma unroll
      for (int q = 0; q < 4; ++q) s[pl][q] = 0.f;
#pragma unroll
      for (int r = 0; r < 4 + 2 * SS_R; ++r) {
        const float f = sm.vt[pl][ty][tx + r];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int k = q - r + 2 * SS_R;
          if (k >= 0 && k < SS_W) s[pl][q] = fmaf(a.g[k], f, s[pl][q]);
        }
      }
      if (x_edge) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (x0 + tx + q < W) s[pl][q] += reflected_taps<1>(&sm.vt[pl][ty][0], x0 + tx + q, W, x0 - SS_R, a.g);
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float dssim = s[0][q] + 2.0f * (xs[q] * s[1][q]) + tg[q] * s[2][q];
      gout[c][q] = (-a.inv_n * dssim) / 3.0f * a.scale;
    }
  }
  if (y >= H) return;
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const int x = x0 + tx + q;
    if (x >= W) break;
    const uint64_t p = (uint64_t)v * a.P + (uint64_t)y * W + x;
    float4 d = dl_dc[p];
    d.x += gout[0][q]; d.y += gout[1][q]; d.z += gout[2][q];
    dl_dc[p] = d;
  }
}

__global__ void k_loss_parts(const double* __restrict__ mse, const double* __restrict__ ssim_sum, uint32_t n_views,
                             double inv_3p, float lambda, double* __restrict__ out) {
  const uint32_t v = blockIdx.x * blockDim.x + threadIdx.x;
  if (v >= n_views) return;
  const double m = mse ? mse[v] * inv_3p : 0.0;
  const double s = ssim_sum ? 1.0 - ssim_sum[v] * inv_3p : 0.0;
  const double l = (double)lambda;
  out[3 * v] = lambda == 0.0f ? m : (lambda == 1.0f ? s : (1.0 - l) * m + l * s);
  out[3 * v + 1] = lambda == 1.0f ? 0.0 : m;
  out[3 * v + 2] = lambda == 0.0f ? 0.0 : s;
}

}  // namespace

sc_status launch_loss_parts(sc_ctx* ctx, const double* mse, const double* ssim_sum, uint32_t n_views, uint64_t P,
                            float lambda, double* out) {
  if (n_views == 0) return SC_OK;
  k_loss_parts<<<(n_views + 63) / 64, 64, 0, ctx->stream>>>(mse, ssim_sum, n_views, 1.0 / (3.0 * (double)P), lambda,
                                                             out);
  return sc_check_launch(ctx, "k_loss_parts");
}

void ssim_window(float g[11]) {
  // loss.rs:36-51, in f32 like the reference
  const float centre = 5.0f, two_sigma_sq = 2.0f * 1.5f * 1.5f;
  float sum = 0.0f;
  for (int i = 0; i < SS_W; ++i) {
    const float d = (float)i - centre;
    g[i] = std::exp(-d * d / two_sigma_sq);
    sum += g[i];
  }
  for (int i = 0; i < SS_W; ++i) g[i] /= sum;
}

size_t ssim_terms_bytes(uint64_t pixels_per_view, uint32_t n_views) {
  return (size_t)n_views * SS_PLANES * pixels_per_view * sizeof(float);
}

sc_status launch_ssim(sc_ctx* ctx, const float4* pred, const float* target, uint32_t w, uint32_t h, uint32_t n_views,
                      float scale, float4* dl_dc, double* ssim_sum, float* terms) {
  if (n_views == 0) return SC_OK;
  if (w < 6 || h < 6) return sc_fail(ctx, SC_ERR_INVALID_ARG, "SSIM needs images of at least 6x6 pixels");
  SsimArgs a;
  ssim_window(a.g);
  a.w = w; a.h = h; a.P = (uint64_t)w * h; a.scale = scale;
  a.inv_n = 1.0f / (float)a.P;
  static bool attr_set[64] = {};
  const int dev = ctx->device & 63;
  if (!attr_set[dev]) {
    SC_CUDA_TRY(ctx, cudaFuncSetAttribute(k_ssim_terms, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)sizeof(TermsSmem)), "ssim smem");
    SC_CUDA_TRY(ctx, cudaFuncSetAttribute(k_ssim_grad, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                          (int)sizeof(GradSmem)), "ssim smem");
    attr_set[dev] = true;
  }
  const dim3 grid((w + SS_T - 1) / SS_T, (h + SS_T - 1) / SS_T, n_views);
  sc_launch(ctx, k_ssim_terms, grid, 256, sizeof(TermsSmem), pred, target, a, terms, ssim_sum);
  SC_TRY(sc_check_launch(ctx, "k_ssim_terms"));
  sc_launch(ctx, k_ssim_grad, grid, 256, sizeof(GradSmem), pred, target, a, terms, dl_dc);
  return sc_check_launch(ctx, "k_ssim_grad");
}

}  // namespace sck
