// Conv2d layers (NCHW activations, OIHW weights, groups = 1, dilation = 1):
// interval propagation in centre/radius form and the CROWN backward transformer
// (ReLU backward + transposed convolution of the coefficient rows).
#include <cooperative_groups.h>

#include <float.h>
#include <stdlib.h>

#include "conv_tc.cuh"

namespace bf {

// ---------------------------------------------------------------------------
// Forward convolutions (interval propagation, and plain rows) as implicit GEMMs on FP32 FFMA tiles
// ---------------------------------------------------------------------------

struct IbpConvArgs {
  const float* in_a; const float* in_b; int in_mode; int relu_in;
  const float* W; const float* bias;
  const int8_t* split; int split_stride;
  const float* cons_l; const float* cons_u;
  float* out_l; float* out_u; int* infeasible;
  int B, Ci, Hi, Wi, Co, Ho, Wo, kh, kw, sh, sw, ph, pw;
};

// A CTA computes TN output channels x TM = 4096 / TN output pixels (pixels of all images in one line), a thread 4 x 4 of them,
// over slabs of CBK input taps in (channel, kernel row, kernel column) order.  The gather positions of a slab's taps are
// decoded once per CTA into `tab`, two slabs ahead.  INTERVAL: centre and radius accumulators; otherwise one convolution of
// plain rows (in_a).  A sum runs over its taps in ascending order; above CONV_SERIAL_K taps it is cut in four, whatever the
// batch (so that an image's bounds are the same bits in every one), and a cluster of four CTAs takes the parts, which meet in
// distributed shared memory in rank order: 16 images, 128 -> 128 channels, 3x3 on 8 x 8: 31 us, in one part 113.  (Cutting shorter
// sums too was 10-20 us faster per layer at 16 images, but a pre-activation bound within an ulp of zero then changes sides
// against the serial sum and takes the relaxation of its ReLU with it.)
// Bound by FFMA issue and the slab's shared-memory reads (three 128-bit reads for 32 FMAs; issue slots 66 %, shared memory 51 %, FMA
// pipe 44 % busy): 200 images, 32 -> 32 channels, 4x4 / 2
// kernel on 32 x 32: 138 us = 24 TFLOP/s (one thread per output, weights and pixels read through L1 for every tap, before: 1.1 ms);
// plain rows, 432 x 16 x 14 x 14 -> 32, 4x4 / 2: 27 us (164).
// Plain rows of few tiles are cut too (conv_row_parts): one tile an SM is bound by the latency of its slabs (copy, barrier, 16 taps: 1.4 us).  They are
// points of a gradient, not bounds: the order of their sums follows the tile count.  (One order for every batch, the parts of a tile added one by one
// by one, two or four CTAs: 1.02 to 1.07 of the time where the tiles are many.)
// TC channels a thread: eight for plain rows of more than 32 channels and more than two tiles an SM (three 128-bit reads per 32 FMAs instead of four; 128 threads): 1152 x 64 x 8 x 8 ->
// 64, 3x3: 195 -> 179 us, 4608 rows 755 -> 672.  Not for intervals (128 registers: 30 -> 36 us and 92 -> 142 us at 16 images, 0.92 of the time at best) nor
// for few tiles (9 x 128 x 8 x 8 -> 128, 3x3: 26 -> 33; 72 x 16 x 14 x 14 -> 48, 3x3, 221 tiles: 19 -> 21) or channels (32: 11 -> 13 us at 36 rows, 148 -> 134 at 4608).
constexpr int CONV_SERIAL_K = 1024, CONV_PARTS = 4, CONV_ROWS_CUT_4 = 128, CONV_ROWS_CUT_2 = 256;

template <int TN>
struct ConvTile {
  static constexpr int TM = 4096 / TN, SLAB = (TN == 16) ? 8 : 16;
};

// Parts that a sum of K taps of plain rows is cut into, a CTA each: four while the CTAs are two an SM at most, else two.  16 -> 32 channels, 14 x 14, 4x4 / 2
// (256 taps), one / two / four parts: 36 rows 22 / 17 / 11 us, 144 rows (56 tiles) 22 / 17 / 14, 288 rows (111) 22 / 21 / 21, 432 rows (166) 31 / 27 / 29,
// 576 rows (221) 32 / 27 / 33, 1152 rows (441) 44 / 49 / 54; 32 -> 32, 16 x 16, 4x4 / 2 (512 taps): 38 / 25 / 19 at 36 tiles, 39 / 33 / 38 at 144, 56 / 53 / 62
// at 288.  128 taps: 12 / 9 in four parts, 12.3 -> 13.1 in two (144 tiles); 135 taps 13 / 12 in four (55 tiles), 13.2 -> 14.7 in two (110).
static int conv_row_parts(long long tiles, int K) {
  if (K > CONV_SERIAL_K) return CONV_PARTS;
  if (tiles * 4 <= 2 * 148) return K >= CONV_ROWS_CUT_4 ? 4 : 1;
  return tiles <= 2 * 148 && K >= CONV_ROWS_CUT_2 ? 2 : 1;
}

// Sums of one output (pixel of all images, channel) over the taps inside the image: centre, radius
template <bool INTERVAL>
__device__ __forceinline__ float2 taps_inside(const IbpConvArgs& g, long long pix, int co) {
  const int howo = g.Ho * g.Wo, b = (int)(pix / howo), q = (int)(pix - (long long)b * howo);
  const int h0 = q / g.Wo * g.sh - g.ph, w0 = q % g.Wo * g.sw - g.pw;
  float2 t = make_float2(0.f, 0.f);
  for (int ci = 0; ci < g.Ci; ++ci)
    for (int r = max(0, -h0); r < g.kh && h0 + r < g.Hi; ++r)
      for (int s = max(0, -w0); s < g.kw && w0 + s < g.Wi; ++s) {
        const size_t i = (((size_t)b * g.Ci + ci) * g.Hi + h0 + r) * g.Wi + w0 + s;
        const float w = g.W[(((size_t)co * g.Ci + ci) * g.kh + r) * g.kw + s];
        float c = g.in_a[i];
        if (INTERVAL) {
          float d = g.in_b[i];
          if (g.in_mode == BF_IN_LOWER_UPPER) {
            if (g.relu_in) { c = fmaxf(c, 0.f); d = fmaxf(d, 0.f); }
            const float mid = (c + d) * 0.5f;
            d = (d - c) * 0.5f;
            c = mid;
          }
          t.y = fmaf(d, fabsf(w), t.y);
        }
        t.x = fmaf(c, w, t.x);
      }
  return t;
}

template <bool INTERVAL, int TN, int TC>
__global__ void __launch_bounds__(1024 / TC) conv_tile_kernel(IbpConvArgs g, int kper, int vec) {
  grid_wait();
  constexpr int TM = ConvTile<TN>::TM, CBK = ConvTile<TN>::SLAB, ACCS = INTERVAL ? 2 : 1;
  constexpr int T = 1024 / TC, NA = TM * CBK / T, KSTEP = T / TM, WLD = TN + 4, NW = (TN * CBK + T - 1) / T;
  constexpr int STAGE = ACCS * CBK * TM + CBK * WLD, PART = ACCS * TM * TN;
  __shared__ __align__(16) float smem[2 * STAGE > PART ? 2 * STAGE : PART];
  __shared__ int4 tab[2][CBK];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int tid = threadIdx.x, tx = tid % (TM / 4), ty = tid / (TM / 4);
  const int taps = g.kh * g.kw, K = g.Ci * taps, howo = g.Ho * g.Wo, hw = g.Hi * g.Wi;
  const long long npix = (long long)g.B * howo;
  const long long p0 = (long long)blockIdx.x * TM;
  const int c0 = blockIdx.y * TN;
  const int k0 = blockIdx.z * kper, k1 = min(K, k0 + kper);
  const int nk = (k1 > k0) ? (k1 - k0 + CBK - 1) / CBK : 0;

  // this thread's pixel as a loader
  const long long lp = p0 + tid % TM;
  const int lk = tid / TM;
  const bool live = lp < npix;
  int h0 = 0, w0 = 0;
  const float *base_a = g.in_a, *base_b = g.in_b;
  if (live) {
    const int b = (int)(lp / howo), q = (int)(lp - (long long)b * howo);
    h0 = (q / g.Wo) * g.sh - g.ph;
    w0 = (q % g.Wo) * g.sw - g.pw;
    const long long off = (long long)b * g.Ci * hw;
    base_a += off;
    if (INTERVAL) base_b += off;
  }
  auto decode = [&](int kt) {  // x: offset of the tap in the image, y / z: kernel row / column (far outside past the end of K)
    if (tid < CBK) {
      const int k = k0 + kt * CBK + tid;
      const int ci = k / taps, t = k - ci * taps, r = t / g.kw, s = t - r * g.kw;
      tab[kt & 1][tid] = (k < k1) ? make_int4(ci * hw + r * g.Wi + s, r, s, 0) : make_int4(0, 1 << 29, 0, 0);
    }
  };
  const int pix_off = h0 * g.Wi + w0;
  float ra[NA], rb[INTERVAL ? NA : 1], rw[NW];
  auto load_slab = [&](int kt) {
#pragma unroll
    for (int j = 0; j < NA; ++j) {
      const int4 t = tab[kt & 1][lk + j * KSTEP];
      const int hi = h0 + t.y, wi = w0 + t.z;
      const bool ok = live && (unsigned)hi < (unsigned)g.Hi && (unsigned)wi < (unsigned)g.Wi;
      ra[j] = ok ? base_a[pix_off + t.x] : 0.f;
      if (INTERVAL) rb[j] = ok ? base_b[pix_off + t.x] : 0.f;
    }
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      const int e = tid + j * T, co = c0 + e / CBK, k = k0 + kt * CBK + e % CBK;
      rw[j] = (e < TN * CBK && co < g.Co && k < k1) ? g.W[(size_t)co * K + k] : 0.f;
    }
  };
  auto store_slab = [&](int stage) {
    float* as = smem + stage * STAGE;
    float* ws = as + ACCS * CBK * TM;
#pragma unroll
    for (int j = 0; j < NA; ++j) {
      float a = ra[j];
      const int at = (lk + j * KSTEP) * TM + tid % TM;
      if (INTERVAL) {
        float b = rb[j];
        if (g.in_mode == BF_IN_LOWER_UPPER) {
          if (g.relu_in) { a = fmaxf(a, 0.f); b = fmaxf(b, 0.f); }
          const float c = (a + b) * 0.5f;
          b = (b - a) * 0.5f;
          a = c;
        }
        as[CBK * TM + at] = b;
      }
      as[at] = a;
    }
#pragma unroll
    for (int j = 0; j < NW; ++j) {
      const int e = tid + j * T;
      if (e < TN * CBK) ws[(e % CBK) * WLD + e / CBK] = rw[j];
    }
  };

  float accC[TC][4], accR[INTERVAL ? TC : 1][4];  // [channel][pixel]
#pragma unroll
  for (int i = 0; i < TC; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      accC[i][j] = 0.f;
      if (INTERVAL) accR[i][j] = 0.f;
    }
  decode(0);
  decode(1);
  __syncthreads();
  if (nk > 0) {
    load_slab(0);
    store_slab(0);
  }
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    const int stage = kt & 1;
    if (kt + 1 < nk) load_slab(kt + 1);
    if (kt + 2 < nk) decode(kt + 2);  // its slot was last read before the previous barrier
    const float* as = smem + stage * STAGE;
    const float* ws = as + ACCS * CBK * TM;
#pragma unroll
    for (int kk = 0; kk < CBK; ++kk) {
      const float4 c4 = *reinterpret_cast<const float4*>(as + kk * TM + tx * 4);
      float w[TC];
#pragma unroll
      for (int q = 0; q < TC; q += 4) {
        const float4 w4 = *reinterpret_cast<const float4*>(ws + kk * WLD + ty * TC + q);
        w[q] = w4.x; w[q + 1] = w4.y; w[q + 2] = w4.z; w[q + 3] = w4.w;
      }
      float4 r4 = c4;
      if (INTERVAL) r4 = *reinterpret_cast<const float4*>(as + CBK * TM + kk * TM + tx * 4);
      const float c[4] = {c4.x, c4.y, c4.z, c4.w}, r[4] = {r4.x, r4.y, r4.z, r4.w};
#pragma unroll
      for (int i = 0; i < TC; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          accC[i][j] = fmaf(c[j], w[i], accC[i][j]);
          if (INTERVAL) accR[i][j] = fmaf(r[j], fabsf(w[i]), accR[i][j]);
        }
    }
    if (kt + 1 < nk) store_slab(stage ^ 1);
    __syncthreads();
  }

  grid_release();

  const int ranks = gridDim.z;
  if (ranks > 1) {
    const int at = ty * TC * TM + tx * 4;  // part[acc][channel][pixel]
#pragma unroll
    for (int i = 0; i < TC; ++i) {
      *reinterpret_cast<float4*>(smem + at + i * TM) = make_float4(accC[i][0], accC[i][1], accC[i][2], accC[i][3]);
      if (INTERVAL) *reinterpret_cast<float4*>(smem + TM * TN + at + i * TM) = make_float4(accR[i][0], accR[i][1], accR[i][2], accR[i][3]);
    }
    cluster.sync();
#pragma unroll
    for (int i = 0; i < TC; ++i) {
      if (i % ranks != (int)blockIdx.z) continue;  // rank z finishes channels z, z + ranks, ... of every thread
      float4 c = make_float4(0.f, 0.f, 0.f, 0.f), r = c;
      for (int q = 0; q < ranks; ++q) {
        const float* p = cluster.map_shared_rank(smem, q);
        const float4 a = *reinterpret_cast<const float4*>(p + at + i * TM);
        c.x += a.x; c.y += a.y; c.z += a.z; c.w += a.w;
        if (INTERVAL) {
          const float4 b = *reinterpret_cast<const float4*>(p + TM * TN + at + i * TM);
          r.x += b.x; r.y += b.y; r.z += b.z; r.w += b.w;
        }
      }
      accC[i][0] = c.x; accC[i][1] = c.y; accC[i][2] = c.z; accC[i][3] = c.w;
      if (INTERVAL) { accR[i][0] = r.x; accR[i][1] = r.y; accR[i][2] = r.z; accR[i][3] = r.w; }
    }
    cluster.sync();
  }

  const long long pt = p0 + tx * 4;
  if (pt >= npix) return;
  // A tap outside the image has multiplied its weight by 0, which is NaN for an infinite weight: sums that are not finite are
  // formed again from the taps inside.
  bool finite = true;
#pragma unroll
  for (int i = 0; i < TC; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      finite &= fabsf(accC[i][j]) <= FLT_MAX;
      if (INTERVAL) finite &= fabsf(accR[i][j]) <= FLT_MAX;
    }
  if (!finite) {
    for (int e = 0; e < 4 * TC; ++e) {
      const int i = e >> 2, j = e & 3;
      if (pt + j >= npix || c0 + ty * TC + i >= g.Co) continue;
      const float2 t = taps_inside<INTERVAL>(g, pt + j, c0 + ty * TC + i);
      smem[e * T + tid] = t.x;  // the slabs are read no more; a thread has words of its own
      if (INTERVAL) smem[4096 + e * T + tid] = t.y;
    }
#pragma unroll
    for (int e = 0; e < 4 * TC; ++e) {
      accC[e >> 2][e & 3] = smem[e * T + tid];
      if (INTERVAL) accR[e >> 2][e & 3] = smem[4096 + e * T + tid];
    }
  }
  int b4[4], q4[4];
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    b4[j] = (int)((pt + j) / howo);
    q4[j] = (int)((pt + j) - (long long)b4[j] * howo);
  }
#pragma unroll
  for (int i = 0; i < TC; ++i) {
    const int co = c0 + ty * TC + i;
    if (co >= g.Co || (ranks > 1 && i % ranks != (int)blockIdx.z)) continue;
    const float bias = g.bias ? g.bias[co] : 0.f;
    float lo[4], up[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      if (!INTERVAL) {
        lo[j] = accC[i][j] + bias;
        continue;
      }
      lo[j] = (accC[i][j] - accR[i][j]) + bias;
      up[j] = (accC[i][j] + accR[i][j]) + bias;
      if (pt + j < npix && (g.cons_l || g.split)) {
        const size_t idx = ((size_t)b4[j] * g.Co + co) * howo + q4[j];
        bool bad = false;
        if (g.cons_l) {
          lo[j] = fmaxf(lo[j], g.cons_l[idx]);
          up[j] = fminf(up[j], g.cons_u[idx]);
          bad |= lo[j] > up[j];
        }
        if (g.split) {
          const int s = g.split[(size_t)b4[j] * g.split_stride + (size_t)co * howo + q4[j]];
          if (s > 0) lo[j] = fmaxf(lo[j], 0.f);
          if (s < 0) up[j] = fminf(up[j], 0.f);
          bad |= lo[j] > up[j];
        }
        if (bad && g.infeasible) g.infeasible[b4[j]] = 1;
      }
    }
    if (vec) {  // Ho * Wo % 4 == 0: a thread's four pixels lie in one image, and 16-byte aligned outputs
      const size_t idx = ((size_t)b4[0] * g.Co + co) * howo + q4[0];
      *reinterpret_cast<float4*>(g.out_l + idx) = make_float4(lo[0], lo[1], lo[2], lo[3]);
      if (INTERVAL) *reinterpret_cast<float4*>(g.out_u + idx) = make_float4(up[0], up[1], up[2], up[3]);
    } else {
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (pt + j >= npix) continue;
        const size_t idx = ((size_t)b4[j] * g.Co + co) * howo + q4[j];
        g.out_l[idx] = lo[j];
        if (INTERVAL) g.out_u[idx] = up[j];
      }
    }
  }
}

template <bool INTERVAL, int TN, int TC>
static int launch_conv_tile_n(const IbpConvArgs& g, int vec, cudaStream_t stream) {
  const long long npix = (long long)g.B * g.Ho * g.Wo;
  const long long tiles = (npix + ConvTile<TN>::TM - 1) / ConvTile<TN>::TM;
  const int K = g.Ci * g.kh * g.kw, slabs = ceil_div(K, ConvTile<TN>::SLAB), ctas_y = ceil_div(g.Co, TN);
  BF_REQUIRE(ctas_y <= 65535 && tiles <= 2147483647LL, BF_E_UNSUPPORTED, "conv2d: too many output channels or pixels");
  const int ks = !INTERVAL ? conv_row_parts(tiles * ctas_y, K) : K > CONV_SERIAL_K ? CONV_PARTS : 1;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)tiles, ctas_y, ks);
  cfg.blockDim = dim3(1024 / TC);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = ks;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  // Fewer blocks than the chip holds, or clusters, are not placed early, unless they are short or one to an SM: bunched on the SMs that are
  // free first, 400 of them took 88 us for 71 (200 x 32 x 32 x 32 -> 32, 4x4 / 2), 128 in clusters of four 37 for 30 (16 x 128 x 8 x 8 -> 128, 3x3,
  // intervals); 110 of 16 taps (144 x 1 x 28 x 28 -> 16) 4.0 for 4.6.  One to an SM: 10 steps of alpha on a CNN of 48 inputs 2.03 -> 2.00 ms.
  const bool one_each = ks == 1 && tiles * ctas_y <= 148;
  cfg.numAttrs = one_each || (ks == 1 && (K <= 64 || tiles * ctas_y >= 4 * 148)) ? 2 : 1;
  if (one_each) {
    static SmemOptIn opt_in;
    if (int rc = ensure_dynamic_smem(conv_tile_kernel<INTERVAL, TN, TC>, ONE_PER_SM, opt_in, "conv_tile_kernel")) return rc;
    cfg.dynamicSmemBytes = ONE_PER_SM;
  }
  cudaLaunchKernelEx(&cfg, conv_tile_kernel<INTERVAL, TN, TC>, g, ceil_div(slabs, ks) * ConvTile<TN>::SLAB, vec);
  BF_CHECK_LAUNCH("conv_tile_kernel");
  return BF_OK;
}

// tile width by the output channels: a wider one wastes accumulators on channels that do not exist
template <bool INTERVAL>
static int launch_conv_tile(const IbpConvArgs& g, cudaStream_t stream) {
  int vec = (g.Ho * g.Wo) % 4 == 0 && ((reinterpret_cast<uintptr_t>(g.out_l) | reinterpret_cast<uintptr_t>(g.out_u)) & 15u) == 0;
  if (g.Co <= 16) return launch_conv_tile_n<INTERVAL, 16, 4>(g, vec, stream);
  if (g.Co <= 32) return launch_conv_tile_n<INTERVAL, 32, 4>(g, vec, stream);
  const long long tiles = ((long long)g.B * g.Ho * g.Wo + 63) / 64 * ceil_div(g.Co, 64);
  if (INTERVAL || tiles <= 2 * 148) return launch_conv_tile_n<INTERVAL, 64, 4>(g, vec, stream);
  return launch_conv_tile_n<false, 64, 8>(g, vec, stream);
}

int launch_ibp_conv2d(const float* in_a, const float* in_b, int in_mode, int relu_in, const float* W, const float* bias,
                      const int8_t* split, int split_stride, const float* cons_l, const float* cons_u, float* out_l,
                      float* out_u, int* infeasible, int B, const bf_layer_desc& L, cudaStream_t stream) {
  IbpConvArgs g{in_a, in_b, in_mode, relu_in, W, bias, split, split_stride, cons_l, cons_u, out_l, out_u, infeasible,
                B, L.Ci, L.Hi, L.Wi, L.Co, L.Ho, L.Wo, L.kh, L.kw, L.sh, L.sw, L.ph, L.pw};
  timing_begin(T_IBP_CONV, stream);
  const int rc = launch_conv_tile<true>(g, stream);
  timing_end(T_IBP_CONV, stream, 4.0 * ((double)L.Co * L.Ci * L.kh * L.kw + L.Co) + 8.0 * (double)B * (L.n_in + L.n_out),
             4.0 * (double)B * L.n_out * L.Ci * L.kh * L.kw);
  return rc;
}

// Forward convolution of rows: out[m] = conv2d(in[m], W) + bias (the gradient sweep of the alpha optimiser pushes its
// adjoint points through the layers in forward direction).
int launch_conv_forward_rows(const float* in, const float* W, const float* bias, float* out, int M, const bf_layer_desc& L,
                             cudaStream_t stream) {
  IbpConvArgs g{in, nullptr, BF_IN_MID_RAD, 0, W, bias, nullptr, 0, nullptr, nullptr, out, nullptr, nullptr,
                M, L.Ci, L.Hi, L.Wi, L.Co, L.Ho, L.Wo, L.kh, L.kw, L.sh, L.sw, L.ph, L.pw};
  return launch_conv_tile<false>(g, stream);
}

// ---------------------------------------------------------------------------
// ReLU backward on coefficient rows, in front of the transposed convolution:
//   Lam = A * slope_sel (+ add, the split term of beta-CROWN) ;  delta (+)= sum_k A*icpt_sel + Lam*bias[channel]
// grid (row, column chunk): a block streams RELU_ROWS_CHUNK columns of one row
// and leaves one partial sum (fixed summation order); sum_partials_kernel adds
// the chunks of a row.
// ---------------------------------------------------------------------------
constexpr int RELU_ROWS_CHUNK = 4096;

__global__ void __launch_bounds__(256) relu_bwd_rows_kernel(const float* A, const float* dpos, const float* dneg, const float* epos, const float* eneg,
                                                            const float* add, const float* bias, int chan_size, float* Lam, float* partial,
                                                            float* delta, int accumulate, int chunk, int S, int n, int vec) {
  grid_wait();
  const int m = blockIdx.x;
  const int k0 = blockIdx.y * chunk;
  const int k1 = min(n, k0 + chunk);
  const float* a = A + (size_t)m * n;
  const size_t off = (size_t)(m / S) * n;
  float acc = 0.f;
  if (vec) {  // n % 4 == 0 and 16-byte aligned rows: four columns per access
    for (int k = k0 + 4 * (int)threadIdx.x; k < k1; k += 4 * 256) {
      const float4 v4 = *reinterpret_cast<const float4*>(a + k);
      float v[4] = {v4.x, v4.y, v4.z, v4.w};
      float lam[4] = {v4.x, v4.y, v4.z, v4.w};
      if (dpos) {
        const float4 p4 = *reinterpret_cast<const float4*>(dpos + off + k), n4 = *reinterpret_cast<const float4*>(dneg + off + k);
        const float p[4] = {p4.x, p4.y, p4.z, p4.w}, q[4] = {n4.x, n4.y, n4.z, n4.w};
        float ep[4] = {0.f, 0.f, 0.f, 0.f}, en[4] = {0.f, 0.f, 0.f, 0.f};
        if (epos) { const float4 e4 = *reinterpret_cast<const float4*>(epos + off + k); ep[0] = e4.x; ep[1] = e4.y; ep[2] = e4.z; ep[3] = e4.w; }
        if (eneg) { const float4 e4 = *reinterpret_cast<const float4*>(eneg + off + k); en[0] = e4.x; en[1] = e4.y; en[2] = e4.z; en[3] = e4.w; }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          const bool sel = v[c] >= 0.f;
          lam[c] = v[c] * (sel ? p[c] : q[c]);
          acc = fmaf(v[c], sel ? ep[c] : en[c], acc);
        }
        if (add) {
          const float4 a4 = *reinterpret_cast<const float4*>(add + off + k);
          lam[0] += a4.x; lam[1] += a4.y; lam[2] += a4.z; lam[3] += a4.w;
        }
      }
      if (bias) {
        int ch = k / chan_size, rem = k - ch * chan_size;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          acc = fmaf(lam[c], bias[ch], acc);
          if (++rem == chan_size) { rem = 0; ++ch; }
        }
      }
      if (Lam) *reinterpret_cast<float4*>(Lam + (size_t)m * n + k) = make_float4(lam[0], lam[1], lam[2], lam[3]);
    }
  } else {
    for (int k = k0 + (int)threadIdx.x; k < k1; k += 256) {
      const float v = a[k];
      float lam = v;
      if (dpos) {
        const bool sel = v >= 0.f;
        lam = v * (sel ? dpos[off + k] : dneg[off + k]);
        const float e = sel ? (epos ? epos[off + k] : 0.f) : (eneg ? eneg[off + k] : 0.f);
        acc = fmaf(v, e, acc);
        if (add) lam += add[off + k];
      }
      if (bias) acc = fmaf(lam, bias[k / chan_size], acc);
      if (Lam) Lam[(size_t)m * n + k] = lam;
    }
  }
  grid_release();
  if (!partial && !delta) return;
  __shared__ float red[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += red[w];
    if (partial) partial[(size_t)m * gridDim.y + blockIdx.y] = t;   // several chunks per row: summed by sum_partials_kernel
    else delta[m] = accumulate ? (delta[m] + t) : t;                // one block per row
  }
}

// ---------------------------------------------------------------------------
// Transposed convolution of coefficient rows (gather form): one thread per
// (row, input pixel) accumulating ACC input channels in registers; the weight
// slice W[co0:co0+CO_CHUNK, ci0:ci0+ACC, :, :] is staged in shared memory with
// the input channel innermost so that one 128-bit read feeds four FMAs.
// ---------------------------------------------------------------------------
struct ConvTArgs {
  const float* Lam;  // [M, Co, Ho, Wo]
  const float* W;    // [Co, Ci, kh, kw]
  float* out;        // [M, Ci, Hi, Wi]
  int M, Ci, Hi, Wi, Co, Ho, Wo, kh, kw, sh, sw, ph, pw;
  int co_chunk;
};

template <int ACC>
__global__ void __launch_bounds__(256) conv_transpose_rows_kernel(ConvTArgs g) {
  extern __shared__ __align__(16) float wsm[];  // [co_chunk][kh][kw][ACC]
  const int m = blockIdx.x;
  const int pix = blockIdx.y * blockDim.x + threadIdx.x;
  const int ci0 = blockIdx.z * ACC;
  const int npix = g.Hi * g.Wi;
  const bool active = pix < npix;
  const int hi = active ? pix / g.Wi : 0, wi = active ? pix % g.Wi : 0;
  float acc[ACC];
#pragma unroll
  for (int c = 0; c < ACC; ++c) acc[c] = 0.f;
  const int taps = g.kh * g.kw;
  const float* lam_m = g.Lam + (size_t)m * g.Co * g.Ho * g.Wo;

  for (int co0 = 0; co0 < g.Co; co0 += g.co_chunk) {
    const int nco = min(g.co_chunk, g.Co - co0);
    __syncthreads();
    for (int e = threadIdx.x; e < nco * taps * ACC; e += blockDim.x) {
      const int c = e % ACC;
      const int t = (e / ACC) % taps;
      const int co = e / (ACC * taps);
      const int ci = ci0 + c;
      wsm[e] = (ci < g.Ci) ? __ldg(g.W + ((size_t)(co0 + co) * g.Ci + ci) * taps + t) : 0.f;
    }
    __syncthreads();
    if (!active) continue;
    for (int r = 0; r < g.kh; ++r) {
      const int hn = hi + g.ph - r;
      if (hn < 0 || hn % g.sh != 0) continue;
      const int ho = hn / g.sh;
      if (ho >= g.Ho) continue;
      for (int s = 0; s < g.kw; ++s) {
        const int wn = wi + g.pw - s;
        if (wn < 0 || wn % g.sw != 0) continue;
        const int wo = wn / g.sw;
        if (wo >= g.Wo) continue;
        const float* lp = lam_m + ((size_t)co0 * g.Ho + ho) * g.Wo + wo;
        const float* wp = wsm + (r * g.kw + s) * ACC;
        for (int co = 0; co < nco; ++co) {
          const float v = lp[(size_t)co * g.Ho * g.Wo];
          const float4* w4 = reinterpret_cast<const float4*>(wp + (size_t)co * taps * ACC);
#pragma unroll
          for (int c = 0; c < ACC / 4; ++c) {
            const float4 w = w4[c];
            acc[4 * c + 0] = fmaf(v, w.x, acc[4 * c + 0]);
            acc[4 * c + 1] = fmaf(v, w.y, acc[4 * c + 1]);
            acc[4 * c + 2] = fmaf(v, w.z, acc[4 * c + 2]);
            acc[4 * c + 3] = fmaf(v, w.w, acc[4 * c + 3]);
          }
        }
      }
    }
  }
  if (!active) return;
#pragma unroll
  for (int c = 0; c < ACC; ++c) {
    const int ci = ci0 + c;
    if (ci < g.Ci) g.out[((size_t)m * g.Ci + ci) * npix + pix] = acc[c];
  }
}

// ---------------------------------------------------------------------------
// Transposed convolution, row-segment form, for square kernels with equal stride and padding
// in both directions (KS, ST, PD compile-time).  A thread owns a segment of 16 consecutive
// input-image pixels of one image row for TCI input channels (16*TCI accumulators).  The lanes
// of a warp are 32 different segments (image rows, or rows of further coefficient rows when the
// image is small) of the same channel group: a coefficient read is one conflict-free 16-byte
// word per lane, a weight read is a broadcast.  Per output channel and kernel row a thread loads
// the NL coefficient words its segment can touch and the KS*TCI weights, and does
// 16*KS*TCI/ST multiply-adds on registers (all indices compile-time).  The block stages, per
// chunk of cc output channels, the zero-padded coefficient tiles [MR][cc][LH][NLT] and the weights
// [cc][KS*KS][CIB] with cp.async into one of two buffers while it computes on the other.
// ---------------------------------------------------------------------------
// VEC: the coefficient tile starts on a 16-byte boundary of the image row (SH extra columns on the
// left) so that it can be staged with 16-byte copies; needs Wo % 4 == 0.
template <int KS, int ST, int PD, bool VEC, int TWP = 16>
struct RowSeg {
  static constexpr int TW = TWP;                              // pixels per thread (16, or 8 for narrow windows)
  static constexpr int C0 = (KS - 1 - PD + ST - 1) / ST;       // coefficient columns left of the segment's first pixel
  static constexpr int SH = VEC ? ((C0 + 3) / 4 * 4 - C0) : 0;
  static constexpr int C0E = C0 + SH;
  static constexpr int NL = (((TW - 1 + PD) / ST + C0E + 1) + 3) / 4 * 4;
  static constexpr int Q0 = SH / 4;                           // first 16-byte word of a row that holds a needed column
  static_assert(PD <= KS - 1 && TW % ST == 0 && (TW / ST) % 4 == 0, "unsupported geometry");
  // row pitch: a multiple of 4 words whose count of 16-byte words is odd, so that the 16-byte reads of
  // eight consecutive tile rows (a quarter warp) fall into different bank groups
  __host__ __device__ static int tile_w(int sx) {
    const int w4 = (((TW * sx - 1 + PD) / ST + C0E + 1) + 3) / 4;
    return 4 * (w4 | 1);
  }
  __host__ __device__ static int tile_h(int th) { return (th - 1 + PD) / ST + C0 + 1; }
};

struct RowSegArgs {
  ConvTArgs c;
  int sxl;      // log2 of the 16-pixel segments per image row in a block
  int thl;      // log2 of the image rows per block
  int mrl;      // log2 of the coefficient rows per block  (2^(sxl+thl+mrl) segments = 256 / channel groups)
  int cigl;     // log2 of the channel groups per block (TCI channels each)
  int cc;       // output channels staged per chunk (divides Co)
  int tiles_x, tiles_y;
  int rowl;     // log2 of the threads that copy one coefficient-tile row while staging
};

// Asynchronous global->shared copies; `ok == false` writes zeros instead (src is not read).
__device__ __forceinline__ void cp_async_f32(float* smem_dst, const float* gsrc, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  const int bytes = ok ? 4 : 0;
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(gsrc), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_f32x4(float* smem_dst, const float* gsrc, bool ok) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(smem_dst);
  const int bytes = ok ? 16 : 0;
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(gsrc), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// A plain launch unless its blocks are one to an SM: placed early, behind the short ReLU pass, the blocks of a sweep of a few hundred rows bunched on
// half of the SMs (256 rows, 64 -> 32 channels, 3x3 on 8 x 8, with the pass: 113 us, 48 plain; 856 sizes: 0.97 of the time, 78 of them under 0.95).
// RT = 2 (8-pixel segments): a thread owns two image rows that meet the same kernel rows, and each weight read feeds twice the
// multiply-adds.  Same order of sums.
template <int KS, int ST, int PD, int TCI, bool VEC, int TWP, int RT>
__global__ void __launch_bounds__(256, (TCI > 1 && TWP * RT > 8 ? 2 : 3)) conv_transpose_rowseg_kernel(RowSegArgs a) {
  grid_wait();
  using G = RowSeg<KS, ST, PD, VEC, TWP>;
  extern __shared__ __align__(16) float rs_smem[];
  const ConvTArgs& g = a.c;
  const int sx = 1 << a.sxl, th = 1 << a.thl, MR = 1 << a.mrl;
  const int cibl = a.cigl + (TCI == 4 ? 2 : 0);
  const int cib = 1 << cibl;                             // input channels per block
  const int cc = a.cc;
  const int LH = G::tile_h(th), NLT = G::tile_w(sx);
  const int tile = LH * NLT;
  const int nrows = MR * cc * LH;                        // coefficient-tile rows per chunk
  const int lam_words = nrows * NLT;                     // [MR][cc][LH][NLT]
  const int w_row = KS * cib + 4;                        // one kernel row of weights + 16 bytes: rows r and r+1 (image rows of
                                                         // different parity read them in one instruction) fall into different banks
  const int w_words = (cc * KS * w_row + 3) & ~3;        // [cc][KS][KS*cib + 4], padded so that the second buffer stays 16-byte aligned
  const int buf_words = lam_words + w_words;
  constexpr int ROW_ZERO = -2147483647 - 1;
  int* row_off = reinterpret_cast<int*>(rs_smem + 2 * buf_words);  // [nrows] source offset of each tile row, ROW_ZERO: all zeros
  const int m0 = blockIdx.x << a.mrl;
  const int h0 = (blockIdx.y / a.tiles_x) << a.thl;
  const int w0 = (blockIdx.y % a.tiles_x) * (G::TW * sx);
  const int ci0 = blockIdx.z << cibl;
  const int hrowl = a.thl - (RT - 1);                    // log2 of the lanes that share a block's image rows
  const int nsegl = a.sxl + hrowl + a.mrl;
  const int seg = threadIdx.x & ((1 << nsegl) - 1);
  const int cig = threadIdx.x >> nsegl;
  const int hrow = seg & ((1 << hrowl) - 1);
  const int hi = h0 + (RT == 1 ? hrow : hrow / ST * (2 * ST) + hrow % ST);  // lanes of a warp: consecutive image rows (pairs of rows)
  const int colseg = (seg >> hrowl) & (sx - 1);
  const int mr = seg >> (a.sxl + hrowl);
  const int ho_lo = h0 / ST - G::C0;
  const int wo_lo = w0 / ST - G::C0E;
  const int howo = g.Ho * g.Wo;
  const size_t lam_row = (size_t)g.Co * howo;
  const bool row_ok = hi < g.Hi && (w0 + colseg * G::TW) < g.Wi && (m0 + mr) < g.M;

  // source offset (floats, relative to the block's first coefficient row and the chunk's first output channel)
  for (int row = threadIdx.x; row < nrows; row += 256) {
    const int hl = row % LH, cm = row / LH;
    const int co = cm % cc, smr = cm / cc;
    const int ho = ho_lo + hl;
    const bool ok = (m0 + smr < g.M) && ho >= 0 && ho < g.Ho;
    row_off[row] = ok ? (int)(smr * lam_row) + co * howo + ho * g.Wo + wo_lo : ROW_ZERO;
  }
  __syncthreads();

  // staging: 2^rowl threads copy one tile row (16-byte words when VEC), 256 >> rowl rows per step
  const int rsub = threadIdx.x & ((1 << a.rowl) - 1);
  const int rrow = threadIdx.x >> a.rowl;
  const int rstep = 256 >> a.rowl;
  const int jcol = VEC ? 4 * rsub : rsub;
  const bool col_in = jcol < NLT;
  const bool col_ok = col_in && (wo_lo + jcol) >= 0 && (wo_lo + jcol) < g.Wo;  // VEC: words are all-in or all-out (Wo % 4 == 0)
  const float* lam_base = g.Lam + (size_t)m0 * lam_row;
  // weights: thread -> fixed input channel, walks (output channel, tap)
  const int wci = threadIdx.x & (cib - 1);
  const int wq0 = threadIdx.x >> cibl;
  const int wqstep = 256 >> cibl;
  const bool wci_ok = ci0 + wci < g.Ci;
  const float* w_base = g.W + (size_t)(ci0 + wci) * (KS * KS);
  auto stage = [&](int buf, int co0) {
    float* lamS = rs_smem + buf * buf_words;
    float* wS = lamS + lam_words;
    if (col_in) {
      const float* src0 = lam_base + (size_t)co0 * howo + jcol;
      for (int row = rrow; row < nrows; row += rstep) {
        const int off = row_off[row];
        const bool ok = col_ok && off != ROW_ZERO;
        if (VEC) cp_async_f32x4(lamS + row * NLT + jcol, ok ? src0 + off : g.Lam, ok);
        else cp_async_f32(lamS + row * NLT + jcol, ok ? src0 + off : g.Lam, ok);
      }
    }
    for (int q = wq0; q < cc * KS * KS; q += wqstep) {
      const int co = q / (KS * KS);
      const int t = q - co * (KS * KS), r = t / KS;
      cp_async_f32(wS + (co * KS + r) * w_row + (t - r * KS) * cib + wci, wci_ok ? w_base + (size_t)((co0 + co) * g.Ci) * (KS * KS) + (q - co * (KS * KS)) : g.W, wci_ok);
    }
    cp_async_commit();
  };

  float acc[RT][TCI][G::TW];
#pragma unroll
  for (int rt = 0; rt < RT; ++rt)
#pragma unroll
    for (int c = 0; c < TCI; ++c)
#pragma unroll
      for (int i = 0; i < G::TW; ++i) acc[rt][c][i] = 0.f;

  // kernel rows this image row meets: r = r_first + ST * jr (jr < JR, r < KS); they map to tile rows hl_top - jr
  constexpr int JR = (KS + ST - 1) / ST;
  const int r_first = (hi + PD) % ST;
  const int hl_top = (hi + PD - r_first) / ST - ho_lo;
  const int lam_thread = (mr * cc * LH + hl_top) * NLT + colseg * (G::TW / ST);
  const int w_thread = r_first * w_row + cig * TCI;

  stage(0, 0);
  int buf = 0;
  for (int co0 = 0; co0 < g.Co; co0 += cc, buf ^= 1) {
    const bool more = co0 + cc < g.Co;
    if (more) {
      stage(buf ^ 1, co0 + cc);  // the other buffer was released by the barrier that ended the previous iteration
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    if (row_ok) {
      const float* lam_t = rs_smem + buf * buf_words + lam_thread;
      const float* w_t = rs_smem + buf * buf_words + lam_words + w_thread;
      for (int co = 0; co < cc; ++co) {
        const float* lam_co = lam_t + co * tile;
        const float* w_co = w_t + co * KS * w_row;
#pragma unroll
        for (int jr = 0; jr < JR; ++jr) {
          if (KS % ST != 0 && r_first + ST * jr >= KS) break;
          float w[KS][TCI];
#pragma unroll
          for (int sct = 0; sct < KS; ++sct) {
            if (TCI == 4) {
              const float4 w4 = *reinterpret_cast<const float4*>(w_co + jr * ST * w_row + sct * cib);
              w[sct][0] = w4.x; w[sct][1 % TCI] = w4.y; w[sct][2 % TCI] = w4.z; w[sct][3 % TCI] = w4.w;
            } else {
#pragma unroll
              for (int c = 0; c < TCI; ++c) w[sct][c] = w_co[jr * ST * w_row + sct * cib + c];
            }
          }
#pragma unroll
          for (int rt = 0; rt < RT; ++rt) {
            const float4* lp = reinterpret_cast<const float4*>(lam_co + (rt - jr) * NLT);
            float L[G::NL];
#pragma unroll
            for (int q = G::Q0; q < G::NL / 4; ++q) {
              const float4 t4 = lp[q];
              L[4 * q + 0] = t4.x; L[4 * q + 1] = t4.y; L[4 * q + 2] = t4.z; L[4 * q + 3] = t4.w;
            }
#pragma unroll
            for (int sct = 0; sct < KS; ++sct) {
#pragma unroll
              for (int i = 0; i < G::TW; ++i) {
                if ((i + PD - sct) % ST == 0) {
#pragma unroll
                  for (int c = 0; c < TCI; ++c) acc[rt][c][i] = fmaf(L[(i + PD - sct) / ST + G::C0E], w[sct][c], acc[rt][c][i]);
                }
              }
            }
          }
        }
      }
    }
    __syncthreads();
  }
  grid_release();
  if (!row_ok) return;
  const int wleft = g.Wi - (w0 + colseg * G::TW);
#pragma unroll
  for (int rt = 0; rt < RT; ++rt) {
    if (hi + rt * ST >= g.Hi) break;
#pragma unroll
    for (int c = 0; c < TCI; ++c) {
      const int ci = ci0 + cig * TCI + c;
      if (ci >= g.Ci) break;
      float* op = g.out + (((size_t)(m0 + mr) * g.Ci + ci) * g.Hi + hi + rt * ST) * g.Wi + w0 + colseg * G::TW;
      if (wleft >= G::TW && (reinterpret_cast<uintptr_t>(op) & 15u) == 0) {
#pragma unroll
        for (int q = 0; q < G::TW / 4; ++q)
          reinterpret_cast<float4*>(op)[q] = make_float4(acc[rt][c][4 * q], acc[rt][c][4 * q + 1], acc[rt][c][4 * q + 2], acc[rt][c][4 * q + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < G::TW; ++i)
          if (i < wleft) op[i] = acc[rt][c][i];
      }
    }
  }
}

static int ilog2_ceil(int v) {
  int l = 0;
  while ((1 << l) < v) ++l;
  return l;
}

// A launch's expected time without its start, its blocks, and the share of the sums it forms that are results (not padding)
struct RowSegCost {
  double us;
  long long blocks;
  double used;
};
// cost: only that (nothing is launched)
template <int KS, int ST, int PD, int TCI, bool VEC, int TWP, int RT = 1>
static int launch_rowseg_tci(const ConvTArgs& g, RowSegCost* cost, cudaStream_t stream) {
  using G = RowSeg<KS, ST, PD, VEC, TWP>;
  RowSegArgs a{};
  a.c = g;
  // channel groups per block: up to 32 input channels side by side
  int cig = ceil_div(g.Ci, TCI);
  if (cig > 32 / TCI) cig = 32 / TCI;
  a.cigl = ilog2_ceil(cig);
  const int nsegl = 8 - a.cigl;  // 256 threads
  const int segs_row = ceil_div(g.Wi, G::TW);
  a.sxl = ilog2_ceil(segs_row);
  if (a.sxl > nsegl - 1) a.sxl = nsegl - 1;  // leave at least two image rows per block
  a.thl = ilog2_ceil(g.Hi);
  if (a.thl > nsegl - a.sxl + RT - 1) a.thl = nsegl - a.sxl + RT - 1;
  if ((1 << a.thl) % (ST * RT) != 0) return BF_E_UNSUPPORTED;
  a.mrl = nsegl - a.sxl - (a.thl - (RT - 1));
  a.tiles_x = ceil_div(segs_row, 1 << a.sxl);
  a.tiles_y = ceil_div(g.Hi, 1 << a.thl);
  const int nlt = G::tile_w(1 << a.sxl);
  a.rowl = ilog2_ceil(VEC ? nlt / 4 : nlt);
  if (a.rowl > 8) return BF_E_UNSUPPORTED;
  const int cib = TCI << a.cigl;
  const size_t per_co = ((size_t)(1 << a.mrl) * G::tile_h(1 << a.thl) * nlt + (size_t)KS * (KS * cib + 4)) * sizeof(float);
  const size_t budget = (TCI > 1 ? 48 : 32) * 1024;  // per buffer; two buffers per block, two or three blocks per SM
  int cc = (int)(budget / per_co);
  if (cc > 16) cc = 16;
  if (cc > g.Co) cc = g.Co;
  if (cc < 1) return BF_E_UNSUPPORTED;
  while (g.Co % cc != 0) --cc;  // a divisor of Co: every chunk is full
  a.cc = cc;
  const size_t lam_words = (size_t)(1 << a.mrl) * cc * G::tile_h(1 << a.thl) * nlt;
  const size_t w_words = ((size_t)cc * KS * (KS * cib + 4) + 3) & ~(size_t)3;
  const size_t smem = 2 * (lam_words + w_words) * sizeof(float) + (size_t)(1 << a.mrl) * cc * G::tile_h(1 << a.thl) * sizeof(int);
  dim3 grid(ceil_div(g.M, 1 << a.mrl), a.tiles_x * a.tiles_y, ceil_div(g.Ci, cib));
  if (grid.y > 65535 || grid.z > 65535) return BF_E_UNSUPPORTED;
  if (cost) {
    // multiply-adds of a block at a rate per kernel shape, and its chunks; blocks share an SM up to its shared memory
    const double blocks = (double)grid.x * grid.y * grid.z / 148.0;
    double room = (TCI > 1 && TWP * RT > 8) ? 2 : 3;
    if (room > 227 * 1024 / (double)(smem + 1024)) room = (double)(int)(227 * 1024 / (smem + 1024));
    const double waves = blocks > room ? blocks / room : 1.0, side = blocks > room ? room : (blocks > 1.0 ? blocks : 1.0);
    const double rate = KS == 5 ? 1.17e-3 : (KS == 4 ? 2.4e-3 : (ST == 1 ? 1.67e-3 : 3.3e-3));
    cost->us = waves * (side * rate * g.Co * KS * KS * TCI * TWP * RT / (ST * ST) + 0.4 * g.Co / cc) * (TWP == 8 ? 1.35 : 1.0);
    cost->blocks = (long long)grid.x * grid.y * grid.z;
    cost->used = (double)g.Ci * g.Hi * g.Wi / ((double)grid.z * cib * ((long long)a.tiles_y << a.thl) * ((long long)a.tiles_x << a.sxl) * G::TW);
    return BF_OK;
  }
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(conv_transpose_rowseg_kernel<KS, ST, PD, TCI, VEC, TWP, RT>, ONE_PER_SM, opt_in, "conv_transpose_rowseg_kernel")) return rc;
  if ((long long)grid.x * grid.y * grid.z <= 148)
    launch_dependent(conv_transpose_rowseg_kernel<KS, ST, PD, TCI, VEC, TWP, RT>, grid, 256, ONE_PER_SM, stream, a);
  else
    conv_transpose_rowseg_kernel<KS, ST, PD, TCI, VEC, TWP, RT><<<grid, 256, smem, stream>>>(a);
  BF_CHECK_LAUNCH("conv_transpose_rowseg_kernel");
  return BF_OK;
}

template <int KS, int ST, int PD>
static int launch_rowseg(const ConvTArgs& g, RowSegCost* cost, cudaStream_t stream) {
  const bool vec = (g.Wo % 4 == 0) && ((reinterpret_cast<uintptr_t>(g.Lam) & 15u) == 0);
  if (g.Ci <= 2) return vec ? launch_rowseg_tci<KS, ST, PD, 1, true, 16>(g, cost, stream) : launch_rowseg_tci<KS, ST, PD, 1, false, 16>(g, cost, stream);
  // 8-pixel segments when they waste fewer lanes than 16-pixel ones (narrow windows of the windowed sweeps)
  const bool narrow = ((g.Wi + 7) / 8) * 8 < ((g.Wi + 15) / 16) * 16;
  if constexpr (KS == 4) {
    // Two image rows per thread, measured against one over seven kernels, 8 to 64 channels and 4 to 24 rows: faster for 4x4 / 2
    // kernels on five to eight rows from 24 -> 32 channels on (1.03 to 1.18 of the speed), elsewhere mostly slower (4x4 / 2 on 17 to
    // 24 rows 0.90 to 0.98, 3x3 / 1 0.66 to 1.02, 5x5 / 1 0.8 to 1.05), and with few channels its tile can outgrow shared memory.
    if (narrow && g.Ci >= 24 && g.Co >= 32 && g.Hi >= 5 && g.Hi <= 8)
      return vec ? launch_rowseg_tci<KS, ST, PD, 4, true, 8, 2>(g, cost, stream) : launch_rowseg_tci<KS, ST, PD, 4, false, 8, 2>(g, cost, stream);
  }
  if (narrow) return vec ? launch_rowseg_tci<KS, ST, PD, 4, true, 8>(g, cost, stream) : launch_rowseg_tci<KS, ST, PD, 4, false, 8>(g, cost, stream);
  return vec ? launch_rowseg_tci<KS, ST, PD, 4, true, 16>(g, cost, stream) : launch_rowseg_tci<KS, ST, PD, 4, false, 16>(g, cost, stream);
}

// Row-segment kernel for the geometries it is instantiated for; BF_E_UNSUPPORTED otherwise.
static int launch_convT_rowseg(const ConvTArgs& g, RowSegCost* cost, cudaStream_t stream) {
  if (g.kh != g.kw || g.sh != g.sw || g.ph != g.pw) return BF_E_UNSUPPORTED;
  if (g.kh == 3 && g.sh == 1 && g.ph == 1) return launch_rowseg<3, 1, 1>(g, cost, stream);
  if (g.kh == 4 && g.sh == 2 && g.ph == 1) return launch_rowseg<4, 2, 1>(g, cost, stream);
  if (g.kh == 3 && g.sh == 2 && g.ph == 1) return launch_rowseg<3, 2, 1>(g, cost, stream);
  // zero padding: the windowed sweeps below run every transposed convolution in window coordinates
  if (g.kh == 3 && g.sh == 1 && g.ph == 0) return launch_rowseg<3, 1, 0>(g, cost, stream);
  if (g.kh == 4 && g.sh == 2 && g.ph == 0) return launch_rowseg<4, 2, 0>(g, cost, stream);
  if (g.kh == 3 && g.sh == 2 && g.ph == 0) return launch_rowseg<3, 2, 0>(g, cost, stream);
  if (g.kh == 5 && g.sh == 1 && g.ph == 2) return launch_rowseg<5, 1, 2>(g, cost, stream);
  return BF_E_UNSUPPORTED;
}

// Where full coefficient rows take the tensor-core kernel (conv_tc.cu): from one 128-position tile per SM on, and where the
// expected time (conv_tc_supports) is below that of the ReLU pass and the FP32 kernel.  Of 2791 layers of 148 tiles and more (1x1 to
// 5x5 kernels, 8 to 256 channels, 7 to 32 pixels) it takes 2211, 33 of them at less than 0.9 of the FP32 speed (worst 0.72), and leaves
// 44 that would gain 1.3 and more.  (All layers of 148 tiles, 8 channels and up to 9 taps: 266 below 0.9, worst 0.39, namely 8 to 16
// input channels at stride 1, 8 output channels, and weights of so many blocks that the rows are staged four and eight times.)
// The FP32 time is that of the row-segment kernel, also for unpadded square maps, which conv_window.cu takes: of 378 such layers that
// this rule sends here (3x3 / 1, 4x4 / 2, 3x3 / 2 on 3 to 14 pixels, 8 to 128 channels, 256 to 16,384 rows) the time is 0.76 of the FP32 kernels' on
// average, but 97 are slower than them, 39 by more than 1.25 (worst 1.72, 8 and 16 channels).  They stay: their sums are nearer to float64.
// Kernels without a row-segment form take it unless a staged element feeds few multiply-adds: 1x1 / 1 from 32 -> 32 channels on (0.9 to
// 1.4 of the gather kernel's speed; 16 -> 32: 0.7 to 1.1), 2x2 / 1 from 8 -> 32 or 16 -> 16 (0.8 to 1.6), strided ones from 12 -> 32 at
// 1x1 (0.8 to 1.8) and 12 -> 8 at 2x2 (0.8 to 2.0).
// Rows that bound the neurons of a conv layer stay on the FP32 kernels, as windows and as full rows (Lp balls, windows that
// have grown to the map), although the tensor cores took a third of their time (64,000 windows, 32 -> 32 channels: 0.33
// against 1.5 ms): they are millions of values whose last bit differs, and a few of those lie within that bit of zero, where
// the relaxation of their ReLU changes sides: 2 of 8 networks moved by 6e-5.  Rows that bound the neurons of Linear layers or
// the specs are some ten thousand values: no change of sides in 8 networks.
constexpr int CONV_TC_MIN_TILES = 148, CONV_TC_MIN_CI = 8, CONV_TC_MAX_TAPS = 9;

// scaled coefficients [M, n_out] followed by the per-chunk partial sums of the intercept term [M, chunks]
static size_t relu_rows_lam_bytes(int M, int n_out) { return ((size_t)M * n_out * sizeof(float) + 255) & ~(size_t)255; }
size_t crown_bwd_conv2d_scratch_bytes(int M, const bf_layer_desc& L) {
  return relu_rows_lam_bytes(M, L.n_out) + (size_t)M * ceil_div(L.n_out, RELU_ROWS_CHUNK) * sizeof(float);
}

template <int ACC>
static int launch_convT(const ConvTArgs& g0, cudaStream_t stream) {
  ConvTArgs g = g0;
  const int taps = g.kh * g.kw;
  int co_chunk = (64 * 1024) / (taps * ACC * (int)sizeof(float));
  if (co_chunk < 1) co_chunk = 1;
  if (co_chunk > g.Co) co_chunk = g.Co;
  g.co_chunk = co_chunk;
  const int smem = co_chunk * taps * ACC * (int)sizeof(float);
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(conv_transpose_rows_kernel<ACC>, 96 * 1024, opt_in, "conv_transpose_rows_kernel")) return rc;
  BF_REQUIRE(smem <= 96 * 1024, BF_E_UNSUPPORTED, "conv backward: kernel window of %d taps is too large", taps);
  const int npix = g.Hi * g.Wi;
  const int threads = npix >= 256 ? 256 : ((npix + 31) / 32) * 32;
  dim3 grid(g.M, ceil_div(npix, threads), ceil_div(g.Ci, ACC));
  BF_REQUIRE(grid.y <= 65535 && grid.z <= 65535, BF_E_UNSUPPORTED, "conv backward: feature map too large");
  conv_transpose_rows_kernel<ACC><<<grid, threads, smem, stream>>>(g);
  BF_CHECK_LAUNCH("conv_transpose_rows_kernel");
  return BF_OK;
}

static ConvTcProblem conv_tc_geometry(int M, int S, const bf_layer_desc& L) {
  ConvTcProblem c{};
  c.M = M; c.S = S; c.Co = L.Co; c.Ci = L.Ci; c.WH = L.Ho; c.WW = L.Wo; c.Hi = L.Hi; c.Wi = L.Wi;
  c.kh = L.kh; c.kw = L.kw; c.sh = L.sh; c.sw = L.sw; c.ph = L.ph; c.pw = L.pw;
  return c;
}
static bool conv_tc_rule(const ConvTcProblem& c, int* slots) {
  int tiles = 0;
  double tc = 0.0;
  RowSegCost fp32{};
  const int taps = ceil_div(c.kh, c.sh) * ceil_div(c.kw, c.sw);
  if (c.Ci < CONV_TC_MIN_CI || taps > CONV_TC_MAX_TAPS || !conv_tc_supports(c, slots, &tiles, &tc) || tiles < CONV_TC_MIN_TILES) return false;
  ConvTArgs g{nullptr, nullptr, nullptr, c.M, c.Ci, c.Hi, c.Wi, c.Co, c.WH, c.WW, c.kh, c.kw, c.sh, c.sw, c.ph, c.pw, 0};
  if (launch_convT_rowseg(g, &fp32, nullptr) != BF_OK) {
    const int npix = c.Hi * c.Wi, idle = npix < 32 ? 32 : npix;  // the gather kernel's threads of a small map
    return (long long)c.kh * c.kw * c.Ci * (c.Co < 32 ? c.Co : 32) * idle / npix >= (c.sh * c.sw > 1 ? 384 : 1024);
  }
  return tc < fp32.us + 13.0 + 2.5e-6 * c.M * c.Co * c.WH * c.WW;  // and the ReLU pass
}
bool conv_rows_on_tensor_cores(int M, const bf_layer_desc& L) {
  int slots = 0;
  return conv_tc_rule(conv_tc_geometry(M, 1, L), &slots);
}

// The tensor-core kernel takes ReLU scaling, row sums and transposed convolution of full rows in one pass.
// BF_E_UNSUPPORTED: the caller takes the FP32 kernels.
static int launch_conv_tc_bwd(const float* A, const float* dpos, const float* dneg, const float* epos, const float* eneg, const float* add,
                              const float* W, const float* bias, float* A_prev, float* delta, int accumulate, int M, int S,
                              const bf_layer_desc& L, void* scratch, int* status, cudaStream_t stream, int sides) {
  const char* ffma = getenv("BF_B200_FORCE_FFMA");
  if ((ffma && ffma[0] == '1') || !A_prev) return BF_E_UNSUPPORTED;
  ConvTcProblem c = conv_tc_geometry(M / sides, S, L);
  int slots = 0, tiles = 0;
  double us = 0.0;
  if (!conv_tc_rule(c, &slots)) return BF_E_UNSUPPORTED;
  c.M = M;
  c.A = A; c.dpos = dpos; c.dneg = dneg; c.epos = epos; c.eneg = eneg; c.add = dpos ? add : nullptr;
  c.bias = bias; c.W = W; c.out = A_prev; c.status = status;
  if (!conv_tc_supports(c, &slots, &tiles, &us)) return BF_E_UNSUPPORTED;
  const bool sums = delta && (dpos || bias || !accumulate);
  if (sums) {  // the row sums take the place that the scaled coefficients have on the FP32 path
    if (!scratch || slots > L.Co * L.Ho * L.Wo) return BF_E_UNSUPPORTED;
    c.partial = static_cast<float*>(scratch);
  }
  timing_begin(T_CONV_T, stream);
  int rc = launch_conv_tc(c, stream);
  timing_end(T_CONV_T, stream, 4.0 * (double)M * (L.n_out + L.n_in) + 4.0 * (double)L.Co * L.Ci * L.kh * L.kw,
             2.0 * (double)M * L.n_out * L.Ci * L.kh * L.kw);
  if (rc == BF_OK && sums) rc = launch_sum_partials(accumulate ? delta : nullptr, c.partial, slots, delta, M, stream);
  return rc;
}

// Windows that the row-segment kernel keeps: results of 14 and 16 pixels (windows of 12 and 14 under 3x3 / 1, of 7 under 4x4 / 2) fill
// its segments, and its blocks cut a row finer, so it is the faster one where few of its lanes idle (from the channels
// rounded up to a block's) or its blocks fit the SMs at once.  Window kernel against it, time ratios over 8 to 64 output, 1 to 64 input
// channels, 32 to 8192 rows, where this rule takes the one or the other:
//   3x3 / 1, 12 -> 14: 0.43 to 0.88 | 1.02 to 1.25 (16 channels, few rows, also 0.98)
//            14 -> 16: 0.38 to 1.00 | 1.02 to 1.43 (16 channels 0.94 to 1.25)
//   4x4 / 2,  7 -> 16: 0.73 to 0.95 | 1.05 to 1.57 (1 and 8 channels, few rows, 0.92 to 0.99)
static bool rowseg_keeps(const ConvTArgs& g) {
  const bool s1 = g.kh == 3 && g.sh == 1 && g.Wi >= 14, s2 = g.kh == 4 && g.sh == 2 && g.Wi == 16;
  if (g.Hi != g.Wi || g.kh != g.kw || g.sh != g.sw || g.ph != 0 || g.pw != 0 || (!s1 && !s2)) return false;
  RowSegCost cost{};
  if (launch_convT_rowseg(g, &cost, nullptr) != BF_OK) return false;
  const bool full = cost.used >= 0.8, one_wave = cost.blocks <= 148;
  if (s2) return full || (one_wave && g.Ci > 8);
  if (g.Ci > 8) return full || one_wave;
  return g.Wi == 14 && g.Ci <= 2 && one_wave;
}

int launch_crown_bwd_conv2d(const float* A, const float* dpos, const float* dneg, const float* epos, const float* eneg,
                            const float* W, const float* bias, float* A_prev, float* delta, int accumulate, int M, int S,
                            const bf_layer_desc& L, void* scratch, cudaStream_t stream, const float* add, bool tensor_cores, int* status, int sides) {
  const int tc = tensor_cores ? launch_conv_tc_bwd(A, dpos, dneg, epos, eneg, add, W, bias, A_prev, delta, accumulate, M, S, L, scratch, status, stream, sides)
                              : BF_E_UNSUPPORTED;
  if (tc != BF_E_UNSUPPORTED) return tc;
  const float* lam = A;
  const bool need_pro = (dpos != nullptr) || (bias != nullptr) || (delta != nullptr && !accumulate);
  if (need_pro) {
    BF_REQUIRE(!dpos || scratch, BF_E_WORKSPACE, "conv backward: scratch missing");
    float* lam_out = dpos ? static_cast<float*>(scratch) : nullptr;
    // without scratch (no ReLU) a block streams a whole row
    const int chunk = scratch ? RELU_ROWS_CHUNK : L.n_out;
    const int nchunks = ceil_div(L.n_out, chunk);
    float* partial = (delta && nchunks > 1) ? reinterpret_cast<float*>(static_cast<char*>(scratch) + relu_rows_lam_bytes(M, L.n_out)) : nullptr;
    BF_REQUIRE(nchunks <= 65535, BF_E_UNSUPPORTED, "conv backward: layer too wide");
    const void* ptrs[] = {A, dpos, dneg, epos, eneg, add, lam_out};
    int vec = (L.n_out % 4 == 0) ? 1 : 0;
    for (const void* q : ptrs) if (reinterpret_cast<uintptr_t>(q) & 15u) vec = 0;
    dim3 grid(M, nchunks);
    timing_begin(T_RELU_ROWS, stream);
    launch_dependent(relu_bwd_rows_kernel, grid, 256, 0, stream, A, dpos, dneg, epos, eneg, dpos ? add : nullptr, bias, L.Ho * L.Wo, lam_out, partial, delta, accumulate,
                                                  chunk, S, L.n_out, vec);
    // rows in (+ out when a ReLU scales them) and the slope / intercept vectors of every domain
    timing_end(T_RELU_ROWS, stream, (lam_out ? 8.0 : 4.0) * (double)M * L.n_out + (dpos ? 12.0 * (double)(M / S) * L.n_out : 0.0),
               4.0 * (double)M * L.n_out);
    BF_CHECK_LAUNCH("relu_bwd_rows_kernel");
    if (partial) {
      int rc = launch_sum_partials(accumulate ? delta : nullptr, partial, nchunks, delta, M, stream);
      if (rc != BF_OK) return rc;
    }
    if (dpos) lam = lam_out;
  }
  if (!A_prev) return BF_OK;
  ConvTArgs g{lam, W, A_prev, M, L.Ci, L.Hi, L.Wi, L.Co, L.Ho, L.Wo, L.kh, L.kw, L.sh, L.sw, L.ph, L.pw, 0};
  static const bool gather_only = getenv("BF_B200_CONV_GATHER") != nullptr;  // A/B switch, read once per process
  const double conv_bytes = 4.0 * (double)M * (L.n_out + L.n_in) + 4.0 * (double)L.Co * L.Ci * L.kh * L.kw;
  const double conv_flops = 2.0 * (double)M * L.n_out * L.Ci * L.kh * L.kw;
  timing_begin(T_CONV_T, stream);
  int rc = BF_E_UNSUPPORTED;
  if (!gather_only && L.Hi == (L.Ho - 1) * L.sh + L.kh - 2 * L.ph && L.Wi == (L.Wo - 1) * L.sw + L.kw - 2 * L.pw && !rowseg_keeps(g))
    rc = launch_conv_window(lam, W, A_prev, M, L.Ci, L.Co, L.Ho, L.Wo, L.kh, L.kw, L.sh, L.sw, L.ph, L.pw, stream);
  if (rc == BF_E_UNSUPPORTED && !gather_only) rc = launch_convT_rowseg(g, nullptr, stream);
  if (rc == BF_E_UNSUPPORTED) {
    if (L.Ci <= 4) rc = launch_convT<4>(g, stream);
    else if (L.Ci <= 16) rc = launch_convT<16>(g, stream);
    else rc = launch_convT<32>(g, stream);
  }
  timing_end(T_CONV_T, stream, conv_bytes, conv_flops);
  return rc;
}

// ---------------------------------------------------------------------------
// Backward step of a conv2d layer for coefficient rows that are rows first..first+S-1 of the
// identity (the start of an intermediate-bound sweep): row j = (co, ho, wo) maps to the kernel
// patch W[co, :, :, :] placed at (ho*sh - ph, wo*sw - pw), the same for every domain, and its
// bias term is bias[co].  One thread per output element; nothing is multiplied.
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) onehot_conv_rows_kernel(const float* __restrict__ W, const float* __restrict__ bias,
                                                               float* __restrict__ out, float* __restrict__ delta, int first,
                                                               int S, int vec, ConvTArgs g) {
  // grid (coefficient row, group of input channels): the row's output position is decoded once per block
  const int m = blockIdx.x;
  const int j = first + m % S;
  const int co = j / (g.Ho * g.Wo), rem = j - co * (g.Ho * g.Wo);
  const int ho = rem / g.Wo, wo = rem - ho * g.Wo;
  const int h_top = ho * g.sh - g.ph, w_left = wo * g.sw - g.pw;  // image position of kernel tap (0, 0)
  if (blockIdx.y == 0 && threadIdx.x == 0 && delta) delta[m] = bias ? __ldg(bias + co) : 0.f;
  const int ci_per_block = (g.Ci + gridDim.y - 1) / gridDim.y;
  const int ci_end = min(g.Ci, (int)(blockIdx.y + 1) * ci_per_block);
  for (int ci = blockIdx.y * ci_per_block; ci < ci_end; ++ci) {
  const float* wp = W + ((size_t)co * g.Ci + ci) * g.kh * g.kw;
  float* op = out + ((size_t)m * g.Ci + ci) * g.Hi * g.Wi;
  if (vec) {  // Wi % 4 == 0 and 16-byte aligned rows
    const int w4 = g.Wi >> 2;
    for (int p = threadIdx.x; p < g.Hi * w4; p += 256) {
      const int hi = p / w4, wi = (p - hi * w4) << 2;
      const int r = hi - h_top;
      float v[4] = {0.f, 0.f, 0.f, 0.f};
      if (r >= 0 && r < g.kh) {
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int sc = wi + q - w_left;
          if (sc >= 0 && sc < g.kw) v[q] = __ldg(wp + r * g.kw + sc);
        }
      }
      *reinterpret_cast<float4*>(op + (size_t)hi * g.Wi + wi) = make_float4(v[0], v[1], v[2], v[3]);
    }
  } else {
    for (int p = threadIdx.x; p < g.Hi * g.Wi; p += 256) {
      const int hi = p / g.Wi, wi = p - hi * g.Wi;
      const int r = hi - h_top, sc = wi - w_left;
      op[p] = (r >= 0 && r < g.kh && sc >= 0 && sc < g.kw) ? __ldg(wp + r * g.kw + sc) : 0.f;
    }
  }
  }
}

int launch_onehot_conv_rows(int first, const float* W, const float* bias, float* A_prev, float* delta, int M, int S,
                            const bf_layer_desc& L, cudaStream_t stream) {
  ConvTArgs g{nullptr, W, A_prev, M, L.Ci, L.Hi, L.Wi, L.Co, L.Ho, L.Wo, L.kh, L.kw, L.sh, L.sw, L.ph, L.pw, 0};
  BF_REQUIRE(L.Ci <= 65535, BF_E_UNSUPPORTED, "conv backward: too many input channels");
  const int vec = (L.Wi % 4 == 0 && (reinterpret_cast<uintptr_t>(A_prev) & 15u) == 0) ? 1 : 0;
  // about 16 KB of output per block once there are enough rows to fill the machine
  int groups = L.Ci;
  const int per_block = 16384 / (L.Hi * L.Wi * 4);
  if (M >= 148 * 8 && per_block > 1) groups = ceil_div(L.Ci, per_block);
  dim3 grid(M, groups);
  onehot_conv_rows_kernel<<<grid, 256, 0, stream>>>(W, bias, A_prev, delta, first, S, vec, g);
  BF_CHECK_LAUNCH("onehot_conv_rows_kernel");
  return BF_OK;
}

// ---------------------------------------------------------------------------
// Windowed coefficient rows.  A row that started as a row of the identity on a conv layer's output is zero
// outside a small window of every feature map below it: kh x kw after the first backward step, and
// (WH-1)*stride + k after each further transposed convolution.  While the window is smaller than the
// feature map the sweep keeps only the window, [M, C, WH, WW] per row, whose image position follows from
// the row's output pixel (ho, wo):  top = ho*sy + ty, left = wo*sx + tx.  A transposed convolution in
// window coordinates is the ordinary one with zero padding (the kernels above, geometry Ho=WH, Wo=WW);
// what falls outside the feature map is cleared by the next ReLU pass or ignored by the concretisation.
// ---------------------------------------------------------------------------

// Division by a run-time constant: a handful of instructions instead of some twenty.  Rows of 100 to 300 elements are a warp each, and
// the nine divisions of a warp (row, pixel, position) took longer than the elements.  Exact for 0 <= n < 2^31 (the quotient from the
// rounded-down reciprocal is at most one too small).
struct FastDiv {
  unsigned d, magic;
};
static FastDiv fast_div(int d) { return FastDiv{(unsigned)d, 0xffffffffu / (unsigned)d}; }
__device__ __forceinline__ int fast_quot(int n, FastDiv f, int* rem) {
  unsigned q = __umulhi((unsigned)n, f.magic), r = (unsigned)n - q * f.d;
  if (r >= f.d) { ++q; r -= f.d; }
  *rem = (int)r;
  return (int)q;
}
// divisors of the kernels on windows: spec rows per domain, pixels and row length of the bounded value, window plane and row length
struct WindowDiv {
  FastDiv S, pixels, wo, plane, ww;
};
static WindowDiv window_div(const WindowGeom& w) {
  return WindowDiv{fast_div(w.S), fast_div(w.HoB * w.WoB), fast_div(w.WoB), fast_div(w.WH * w.WW), fast_div(w.WW)};
}
// the domain of row m, the output channel that it bounds and its window's origin
__device__ __forceinline__ void window_row(const WindowGeom& w, const WindowDiv& dv, int m, int* domain, int* channel, int* top, int* left) {
  int s, pixel, wo;
  *domain = fast_quot(m, dv.S, &s);
  *channel = fast_quot(w.first + s, dv.pixels, &pixel);
  *top = fast_quot(pixel, dv.wo, &wo) * w.sy + w.ty;
  *left = wo * w.sx + w.tx;
}

// first backward step: the window is the kernel itself (one warp per row)
__global__ void __launch_bounds__(256) onehot_conv_window_kernel(const float* __restrict__ W, const float* __restrict__ bias,
                                                                 float* __restrict__ out, float* __restrict__ delta, WindowGeom w,
                                                                 int per) {
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= w.M) return;
  const int cb = (w.first + m % w.S) / (w.HoB * w.WoB);
  const float* src = W + (size_t)cb * per;
  float* dst = out + (size_t)m * per;
  for (int r = lane; r < per; r += 32) dst[r] = __ldg(src + r);
  if (lane == 0 && delta) delta[m] = bias ? __ldg(bias + cb) : 0.f;
}

// ReLU backward on windows: Lam = A * slope_sel inside the feature map, 0 outside;
// delta += sum A * icpt_sel + Lam * bias[channel].  T threads per row (T = 32 ... 256, by window size), 256 / T
// rows per block.  A thread owns positions of the WH x WW window plane and walks the channels: the image pixel of a
// position, whether it lies inside the feature map and both offsets are computed once per position.  The kernel is bound
// by the latency of its reads (the window value, then the slope and intercept that value selects, gathered from the
// feature map), so the channel loop handles eight channels at a time: eight window values in flight, then eight slopes.
// When the plane is smaller than T the threads split into T / plane channel groups (thread = group * plane + position).
// wstart: the rows are those of the identity on a conv layer's output, whose windows are that layer's kernels: they are read in
// place (wstart, bias wbias), no window is copied first, and delta starts here.
template <int T>
__global__ void __launch_bounds__(256) relu_bwd_window_kernel(const float* __restrict__ A, const float* __restrict__ dpos,
                                                              const float* __restrict__ dneg, const float* __restrict__ epos,
                                                              const float* __restrict__ eneg, const float* __restrict__ bias,
                                                              const float* __restrict__ wstart, const float* __restrict__ wbias,
                                                              float* __restrict__ Lam, float* __restrict__ delta, WindowGeom w, WindowDiv dv) {
  __shared__ float red[8];
  const int m = blockIdx.x * (256 / T) + threadIdx.x / T;
  const int t = threadIdx.x % T;
  const bool live = m < w.M;  // whole warps: T is a multiple of 32
  float acc = 0.f;
  int domain, cb, top, left;   // cb: output channel that the row bounds
  window_row(w, dv, live ? m : 0, &domain, &cb, &top, &left);
  if (live) {
    const int plane = w.WH * w.WW;
    const int HW = w.H * w.W;
    const size_t dom = (size_t)domain * w.C * HW;
    const float* a_row = wstart ? wstart + (size_t)cb * w.C * plane : A + (size_t)m * w.C * plane;
    float* lo_row = Lam + (size_t)m * w.C * plane;
    int p0 = t, rest;                                        // this thread's first position
    const int c0 = (plane < T) ? fast_quot(t, dv.plane, &p0) : 0;        // and its first channel
    const int groups = (plane < T) ? fast_quot(T, dv.plane, &rest) : 1;  // channel groups when the plane is smaller than T
    const int pstep = (plane < T) ? plane : T;               // plane < T: a single position per thread
    if (c0 < groups) {
      const size_t astep = (size_t)groups * plane, kstep = (size_t)groups * HW;
      for (int pos = p0; pos < plane; pos += pstep) {
        int x;
        const int Y = top + fast_quot(pos, dv.ww, &x), X = left + x;
        const bool inside = Y >= 0 && Y < w.H && X >= 0 && X < w.W;
        const float* a = a_row + (size_t)c0 * plane + pos;
        float* lo = lo_row + (size_t)c0 * plane + pos;
        if (!inside) {
          for (int c = c0; c < w.C; c += groups, lo += astep) *lo = 0.f;
          continue;
        }
        size_t k = dom + (size_t)c0 * HW + (size_t)Y * w.W + X;
        int c = c0;
        constexpr int U = 8;   // channels in flight
        for (; c + (U - 1) * groups < w.C; c += U * groups, a += U * astep, lo += U * astep, k += U * kstep) {
          float v[U], sl[U], ic[U];
#pragma unroll
          for (int q = 0; q < U; ++q) v[q] = a[q * astep];
#pragma unroll
          for (int q = 0; q < U; ++q) {
            const size_t kq = k + q * kstep;
            const bool sel = v[q] >= 0.f;
            sl[q] = sel ? dpos[kq] : dneg[kq];
            ic[q] = sel ? (epos ? epos[kq] : 0.f) : (eneg ? eneg[kq] : 0.f);
          }
#pragma unroll
          for (int q = 0; q < U; ++q) {
            const float lam = v[q] * sl[q];
            acc = fmaf(v[q], ic[q], acc);
            if (bias) acc = fmaf(lam, __ldg(bias + c + q * groups), acc);
            lo[q * astep] = lam;
          }
        }
        for (; c < w.C; c += groups, a += astep, lo += astep, k += kstep) {
          const float v = *a;
          const bool sel = v >= 0.f;
          const float lam = v * (sel ? dpos[k] : dneg[k]);
          acc = fmaf(v, sel ? (epos ? epos[k] : 0.f) : (eneg ? eneg[k] : 0.f), acc);
          if (bias) acc = fmaf(lam, __ldg(bias + c), acc);
          *lo = lam;
        }
      }
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  auto finish = [&](float sum) { delta[m] = (wstart ? (wbias ? __ldg(wbias + cb) : 0.f) : delta[m]) + sum; };
  if (T == 32) {
    if (live && t == 0) finish(acc);
  } else {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (live && t == 0) {
      float sum = 0.f;
#pragma unroll
      for (int i = 0; i < T / 32; ++i) sum += red[(threadIdx.x >> 5) + i];
      finish(sum);
    }
  }
}

// window -> full feature map (zeros elsewhere, what falls outside the map is dropped)
__global__ void __launch_bounds__(256) window_to_dense_kernel(const float* __restrict__ Awin, float* __restrict__ dense, WindowGeom w) {
  const int m = blockIdx.x;
  const int j = w.first + m % w.S;
  const int rem = j % (w.HoB * w.WoB);
  const int top = (rem / w.WoB) * w.sy + w.ty, left = (rem % w.WoB) * w.sx + w.tx;
  const int n = w.C * w.H * w.W, n_win = w.C * w.WH * w.WW;
  for (int k = threadIdx.x; k < n; k += 256) {
    const int c = k / (w.H * w.W), r2 = k - c * (w.H * w.W);
    const int y = r2 / w.W - top, x = r2 % w.W - left;
    dense[(size_t)m * n + k] = (y >= 0 && y < w.WH && x >= 0 && x < w.WW) ? Awin[(size_t)m * n_win + (c * w.WH + y) * w.WW + x] : 0.f;
  }
}

// box concretisation of windows on the network input: out[m] = sum A*mid -/+ |A|*rad over the window inside the image + delta
__global__ void __launch_bounds__(256) concretize_window_kernel(const float* __restrict__ Awin, const float* __restrict__ mid,
                                                                const float* __restrict__ rad, const float* __restrict__ delta,
                                                                float* __restrict__ out, float sgn, WindowGeom w, WindowDiv dv) {
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= w.M) return;
  int domain, channel, top, left;
  window_row(w, dv, m, &domain, &channel, &top, &left);
  const int n_win = w.C * w.WH * w.WW;
  const size_t dom = (size_t)domain * w.C * w.H * w.W;
  float acc = 0.f;
  // four elements of a lane per iteration: their index arithmetic first, then all loads, then the sums in element order
  // (the loop is bound by the latency of its gathered reads, like the ReLU pass on windows)
  for (int e0 = lane; e0 < n_win; e0 += 128) {
    float v[4], cm[4], cr[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int e = e0 + 32 * q;
      v[q] = cm[q] = cr[q] = 0.f;
      if (e < n_win) {
        int r2, x;
        const int c = fast_quot(e, dv.plane, &r2);
        const int Y = top + fast_quot(r2, dv.ww, &x), X = left + x;
        if (Y >= 0 && Y < w.H && X >= 0 && X < w.W) {
          const size_t k = dom + ((size_t)c * w.H + Y) * w.W + X;
          v[q] = Awin[(size_t)m * n_win + e];
          cm[q] = mid[k];
          cr[q] = rad[k];
        }
      }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {   // an element outside the window or the image contributes exact zeros
      acc = fmaf(v[q], cm[q], acc);
      acc = fmaf(sgn * fabsf(v[q]), cr[q], acc);
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if (lane == 0) out[m] = acc + (delta ? delta[m] : 0.f);
}

int launch_onehot_conv_window(const float* W, const float* bias, float* out, float* delta, const WindowGeom& w, int M, int Ci, int kk,
                              cudaStream_t stream) {
  onehot_conv_window_kernel<<<ceil_div((long long)M * 32, 256), 256, 0, stream>>>(W, bias, out, delta, w, Ci * kk);
  BF_CHECK_LAUNCH("onehot_conv_window_kernel");
  return BF_OK;
}

int launch_relu_bwd_window(const float* A, const float* dpos, const float* dneg, const float* epos, const float* eneg,
                           const float* bias, const float* wstart, const float* wbias, float* Lam, float* delta, const WindowGeom& w, int M,
                           cudaStream_t stream) {
  const int n_win = w.C * w.WH * w.WW;
  timing_begin(T_RELU_WINDOW, stream);
  if (n_win <= 512)
    relu_bwd_window_kernel<32><<<ceil_div(M, 8), 256, 0, stream>>>(A, dpos, dneg, epos, eneg, bias, wstart, wbias, Lam, delta, w, window_div(w));
  else if (n_win <= 1536)
    relu_bwd_window_kernel<64><<<ceil_div(M, 4), 256, 0, stream>>>(A, dpos, dneg, epos, eneg, bias, wstart, wbias, Lam, delta, w, window_div(w));
  else if (n_win <= 4096)
    relu_bwd_window_kernel<128><<<ceil_div(M, 2), 256, 0, stream>>>(A, dpos, dneg, epos, eneg, bias, wstart, wbias, Lam, delta, w, window_div(w));
  else
    relu_bwd_window_kernel<256><<<M, 256, 0, stream>>>(A, dpos, dneg, epos, eneg, bias, wstart, wbias, Lam, delta, w, window_div(w));
  // window rows in and out; the slopes and intercepts are gathered per element (three values of the row's domain)
  timing_end(T_RELU_WINDOW, stream, 8.0 * (double)M * n_win + 12.0 * (double)M * n_win, 4.0 * (double)M * n_win);
  BF_CHECK_LAUNCH("relu_bwd_window_kernel");
  return BF_OK;
}

int launch_window_to_dense(const float* Awin, float* dense, const WindowGeom& w, int M, cudaStream_t stream) {
  window_to_dense_kernel<<<M, 256, 0, stream>>>(Awin, dense, w);
  BF_CHECK_LAUNCH("window_to_dense_kernel");
  return BF_OK;
}

int launch_concretize_window(const float* Awin, const float* mid, const float* rad, const float* delta, float* out, int side,
                             const WindowGeom& w, int M, cudaStream_t stream) {
  concretize_window_kernel<<<ceil_div((long long)M * 32, 256), 256, 0, stream>>>(Awin, mid, rad, delta, out,
                                                                               side == BF_SIDE_LOWER ? -1.f : 1.f, w, window_div(w));
  BF_CHECK_LAUNCH("concretize_window_kernel");
  return BF_OK;
}

// Same for a linear layer: coefficient row j is row j of W, its bias term bias[j].  2^tl threads copy a row, as many as its words need.  25,600 rows
// of 16, 100, 784 and 1568: 2.1, 4.6, 21 and 28 us; with a division per element 4.4, 10.9, 61 and 117, a block per row 17.6, 17.7, 22 and 27.
__global__ void __launch_bounds__(256) onehot_linear_rows_kernel(const float* __restrict__ W, const float* __restrict__ bias,
                                                                 float* __restrict__ out, float* __restrict__ delta, int first,
                                                                 int M, int S, int n_in, int vec, int tl) {
  const int m = blockIdx.x * (256 >> tl) + (threadIdx.x >> tl), t = threadIdx.x & ((1 << tl) - 1);
  if ((unsigned)m >= (unsigned)M) return;
  const int j = first + m % S;
  const float* src = W + (size_t)j * n_in;
  float* dst = out + (size_t)m * n_in;
  if (vec) {
    for (int k = 4 * t; k < n_in; k += 4 << tl) *reinterpret_cast<float4*>(dst + k) = __ldg(reinterpret_cast<const float4*>(src + k));
  } else {
    for (int k = t; k < n_in; k += 1 << tl) dst[k] = __ldg(src + k);
  }
  if (t == 0 && delta) delta[m] = bias ? __ldg(bias + j) : 0.f;
}

int launch_onehot_linear_rows(int first, const float* W, const float* bias, float* A_prev, float* delta, int M, int S, int n_in,
                              cudaStream_t stream) {
  const int vec = n_in % 4 == 0 && ((reinterpret_cast<uintptr_t>(W) | reinterpret_cast<uintptr_t>(A_prev)) & 15u) == 0;
  int tl = 0;
  while (tl < 8 && (1 << tl) < (vec ? n_in / 4 : n_in)) ++tl;
  onehot_linear_rows_kernel<<<ceil_div(M, 256 >> tl), 256, 0, stream>>>(W, bias, A_prev, delta, first, M, S, n_in, vec, tl);
  BF_CHECK_LAUNCH("onehot_linear_rows_kernel");
  return BF_OK;
}

}  // namespace bf

extern "C" int bf_ibp_conv2d(const float* in_a, const float* in_b, int in_mode, int relu_in, const float* W,
                             const float* bias, const int8_t* split, int split_stride, const float* cons_l,
                             const float* cons_u, float* out_l, float* out_u, int* infeasible, int B, int Ci, int Hi,
                             int Wi, int Co, int kh, int kw, int sh, int sw, int ph, int pw, bf_stream_t stream) {
  BF_REQUIRE(in_a && in_b && W && out_l && out_u, BF_E_INVALID, "bf_ibp_conv2d: null tensor");
  BF_REQUIRE(B > 0 && Ci > 0 && Hi > 0 && Wi > 0 && Co > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0 && ph >= 0 && pw >= 0,
             BF_E_INVALID, "bf_ibp_conv2d: bad geometry");
  BF_REQUIRE(!(relu_in && in_mode == BF_IN_MID_RAD), BF_E_INVALID, "bf_ibp_conv2d: relu_in needs lower/upper inputs");
  BF_REQUIRE((cons_l == nullptr) == (cons_u == nullptr), BF_E_INVALID, "bf_ibp_conv2d: give both constraint tensors or none");
  bf_layer_desc L{};
  L.op = BF_OP_CONV2D; L.Ci = Ci; L.Hi = Hi; L.Wi = Wi; L.Co = Co; L.kh = kh; L.kw = kw; L.sh = sh; L.sw = sw; L.ph = ph; L.pw = pw;
  L.Ho = (Hi + 2 * ph - kh) / sh + 1;
  L.Wo = (Wi + 2 * pw - kw) / sw + 1;
  BF_REQUIRE(L.Ho > 0 && L.Wo > 0, BF_E_INVALID, "bf_ibp_conv2d: empty output");
  L.n_in = Ci * Hi * Wi; L.n_out = Co * L.Ho * L.Wo;
  BF_REQUIRE(!split || split_stride == 0 || split_stride == L.n_out, BF_E_INVALID, "bf_ibp_conv2d: split_stride must be 0 or Co*Ho*Wo");
  return bf::launch_ibp_conv2d(in_a, in_b, in_mode, relu_in, W, bias, split, split_stride, cons_l, cons_u, out_l, out_u,
                               infeasible, B, L, bf::as_stream(stream));
}

// Bytes of scratch the fused ReLU + Conv2d backward needs for the scaled coefficients.
extern "C" size_t bf_crown_relu_conv2d_bwd_scratch_bytes(int B, int S, int Co, int Ho, int Wo) {
  bf_layer_desc L{};
  L.n_out = Co * Ho * Wo;
  return bf::crown_bwd_conv2d_scratch_bytes(B * S, L);
}

// sides: 0 the FP32 kernels; 1, 2: the kernel that M / sides rows take
static int conv2d_bwd(int sides, const float* A, int side, const float* alpha_u, const float* alpha_l,
                      const float* beta_u, const float* beta_l, const float* W, const float* bias, float* A_prev, float* delta,
                      int accumulate, void* scratch, size_t scratch_bytes, int B, int S, int Ci, int Hi, int Wi, int Co, int Ho,
                      int Wo, int kh, int kw, int sh, int sw, int ph, int pw, bf_stream_t stream) {
  BF_REQUIRE(A && W, BF_E_INVALID, "bf_crown_relu_conv2d_bwd: A and W must be non-null");
  BF_REQUIRE(B > 0 && S > 0 && Ci > 0 && Co > 0 && Hi > 0 && Wi > 0 && Ho > 0 && Wo > 0 && kh > 0 && kw > 0 && sh > 0 && sw > 0,
             BF_E_INVALID, "bf_crown_relu_conv2d_bwd: bad geometry");
  BF_REQUIRE(side == BF_SIDE_LOWER || side == BF_SIDE_UPPER, BF_E_INVALID, "bf_crown_relu_conv2d_bwd: bad side");
  BF_REQUIRE(Ho == (Hi + 2 * ph - kh) / sh + 1 && Wo == (Wi + 2 * pw - kw) / sw + 1, BF_E_INVALID,
             "bf_crown_relu_conv2d_bwd: output size does not match the convolution geometry");
  BF_REQUIRE((long long)B * S < 2147483647LL, BF_E_INVALID, "bf_crown_relu_conv2d_bwd: B*S overflows int");
  const bool relu = alpha_u || alpha_l || beta_u || beta_l;
  BF_REQUIRE(!relu || (alpha_u && alpha_l), BF_E_INVALID, "bf_crown_relu_conv2d_bwd: alpha_u and alpha_l must both be given");
  BF_REQUIRE(!relu || (scratch && scratch_bytes >= bf_crown_relu_conv2d_bwd_scratch_bytes(B, S, Co, Ho, Wo)), BF_E_WORKSPACE,
             "bf_crown_relu_conv2d_bwd: scratch of %zu bytes needed", bf_crown_relu_conv2d_bwd_scratch_bytes(B, S, Co, Ho, Wo));
  const float *dpos = nullptr, *dneg = nullptr, *epos = nullptr, *eneg = nullptr;
  if (relu) {
    if (side == BF_SIDE_LOWER) { dpos = alpha_l; dneg = alpha_u; epos = beta_l; eneg = beta_u; }
    else { dpos = alpha_u; dneg = alpha_l; epos = beta_u; eneg = beta_l; }
  }
  bf_layer_desc L{};
  L.op = BF_OP_CONV2D; L.Ci = Ci; L.Hi = Hi; L.Wi = Wi; L.Co = Co; L.Ho = Ho; L.Wo = Wo; L.kh = kh; L.kw = kw;
  L.sh = sh; L.sw = sw; L.ph = ph; L.pw = pw; L.n_in = Ci * Hi * Wi; L.n_out = Co * Ho * Wo;
  // without slopes the scratch is optional; one that is too small for the chunked intercept sums is not used at all
  // (a block then streams a whole coefficient row)
  if (!relu && scratch_bytes < bf_crown_relu_conv2d_bwd_scratch_bytes(B, S, Co, Ho, Wo)) scratch = nullptr;
  return bf::launch_crown_bwd_conv2d(A, dpos, dneg, epos, eneg, W, bias, A_prev, delta, accumulate, B * S, S, L, scratch,
                                     bf::as_stream(stream), nullptr, sides > 0, nullptr, sides);
}

extern "C" int bf_crown_relu_conv2d_bwd(const float* A, int side, const float* alpha_u, const float* alpha_l,
                                        const float* beta_u, const float* beta_l, const float* W, const float* bias,
                                        float* A_prev, float* delta, int accumulate, void* scratch, size_t scratch_bytes,
                                        int B, int S, int Ci, int Hi, int Wi, int Co, int Ho, int Wo, int kh, int kw, int sh,
                                        int sw, int ph, int pw, bf_stream_t stream) {
  return conv2d_bwd(1, A, side, alpha_u, alpha_l, beta_u, beta_l, W, bias, A_prev, delta, accumulate, scratch, scratch_bytes, B, S,
                    Ci, Hi, Wi, Co, Ho, Wo, kh, kw, sh, sw, ph, pw, stream);
}

extern "C" int bf_crown_relu_conv2d_bwd_sides(const float* A, int side, const float* alpha_u, const float* alpha_l,
                                              const float* beta_u, const float* beta_l, const float* W, const float* bias,
                                              float* A_prev, float* delta, int accumulate, void* scratch, size_t scratch_bytes,
                                              int B, int S, int Ci, int Hi, int Wi, int Co, int Ho, int Wo, int kh, int kw, int sh,
                                              int sw, int ph, int pw, bf_stream_t stream) {
  return conv2d_bwd(2, A, side, alpha_u, alpha_l, beta_u, beta_l, W, bias, A_prev, delta, accumulate, scratch, scratch_bytes, B, S,
                    Ci, Hi, Wi, Co, Ho, Wo, kh, kw, sh, sw, ph, pw, stream);
}

extern "C" int bf_crown_relu_conv2d_bwd_fp32(const float* A, int side, const float* alpha_u, const float* alpha_l,
                                             const float* beta_u, const float* beta_l, const float* W, const float* bias,
                                             float* A_prev, float* delta, int accumulate, void* scratch, size_t scratch_bytes,
                                             int B, int S, int Ci, int Hi, int Wi, int Co, int Ho, int Wo, int kh, int kw, int sh,
                                             int sw, int ph, int pw, bf_stream_t stream) {
  return conv2d_bwd(0, A, side, alpha_u, alpha_l, beta_u, beta_l, W, bias, A_prev, delta, accumulate, scratch, scratch_bytes, B, S,
                    Ci, Hi, Wi, Co, Ho, Wo, kh, kw, sh, sw, ph, pw, stream);
}

// ReLU backward alone (graphs where the ReLU's producer is not a single affine layer, e.g. after an add):
// A_prev = A * slope_sel, delta (+)= sum A * icpt_sel (+ add term on the lower side is not needed here).
extern "C" size_t bf_crown_relu_bwd_scratch_bytes(int B, int S, int n) {
  return (size_t)B * S * bf::ceil_div(n, bf::RELU_ROWS_CHUNK) * sizeof(float);
}

extern "C" int bf_crown_relu_bwd(const float* A, int side, const float* alpha_u, const float* alpha_l, const float* beta_u,
                                 const float* beta_l, float* A_prev, float* delta, int accumulate, void* scratch,
                                 size_t scratch_bytes, int B, int S, int n, bf_stream_t stream_) {
  BF_REQUIRE(A && alpha_u && alpha_l && A_prev, BF_E_INVALID, "bf_crown_relu_bwd: null tensor");
  BF_REQUIRE(B > 0 && S > 0 && n > 0 && (long long)B * S < 2147483647LL, BF_E_INVALID, "bf_crown_relu_bwd: bad sizes");
  BF_REQUIRE(side == BF_SIDE_LOWER || side == BF_SIDE_UPPER, BF_E_INVALID, "bf_crown_relu_bwd: bad side");
  const float *dpos, *dneg, *epos, *eneg;
  if (side == BF_SIDE_LOWER) { dpos = alpha_l; dneg = alpha_u; epos = beta_l; eneg = beta_u; }
  else { dpos = alpha_u; dneg = alpha_l; epos = beta_u; eneg = beta_l; }
  const int M = B * S;
  const int nchunks = bf::ceil_div(n, bf::RELU_ROWS_CHUNK);
  float* partial = nullptr;
  if (delta && nchunks > 1) {
    BF_REQUIRE(scratch && scratch_bytes >= bf_crown_relu_bwd_scratch_bytes(B, S, n), BF_E_WORKSPACE,
               "bf_crown_relu_bwd: scratch of %zu bytes needed", bf_crown_relu_bwd_scratch_bytes(B, S, n));
    partial = static_cast<float*>(scratch);
  }
  BF_REQUIRE(nchunks <= 65535, BF_E_UNSUPPORTED, "bf_crown_relu_bwd: layer too wide");
  const void* ptrs[] = {A, dpos, dneg, epos, eneg, A_prev};
  int vec = (n % 4 == 0) ? 1 : 0;
  for (const void* q : ptrs) if (reinterpret_cast<uintptr_t>(q) & 15u) vec = 0;
  cudaStream_t stream = bf::as_stream(stream_);
  dim3 grid(M, nchunks);
  bf::launch_dependent(bf::relu_bwd_rows_kernel, grid, 256, 0, stream, A, dpos, dneg, epos, eneg, nullptr, nullptr, 1, A_prev, partial, delta, accumulate,
                                                    bf::RELU_ROWS_CHUNK, S, n, vec);
  BF_CHECK_LAUNCH("relu_bwd_rows_kernel");
  if (partial) return bf::launch_sum_partials(accumulate ? delta : nullptr, partial, nchunks, delta, M, stream);
  return BF_OK;
}

// ---------------------------------------------------------------------------
// Allocation-free variant of the fused ReLU + Conv2d backward.
//
// Some callers cannot obtain device memory at the moment they need this kernel:
// a verification service whose device pool is sized at start-up and then
// frozen, a plugin loaded into a process that already owns all device memory,
// or a host runtime that forbids cudaMalloc / cudaFree on its request path
// because those calls synchronise the whole device.
// For them the scratch that holds the ReLU-scaled coefficients lives in a
// fixed-size array inside the library image instead of a caller buffer.
// ---------------------------------------------------------------------------
#define BF_NOALLOC_SCRATCH_BYTES (16u * 1024u * 1024u)
static __device__ __align__(256) unsigned char g_noalloc_scratch[BF_NOALLOC_SCRATCH_BYTES];

// In host code the array's name is only a handle; the device address is resolved
// once per device (with that device current) and cached here.
static void* g_noalloc_scratch_addr[64] = {nullptr};

extern "C" size_t bf_crown_relu_conv2d_bwd_noalloc_max_bytes(void) { return (size_t)BF_NOALLOC_SCRATCH_BYTES; }

extern "C" int bf_crown_relu_conv2d_bwd_noalloc(const float* A, int side, const float* alpha_u, const float* alpha_l,
                                                const float* beta_u, const float* beta_l, const float* W, const float* bias,
                                                float* A_prev, float* delta, int accumulate, int B, int S, int Ci, int Hi,
                                                int Wi, int Co, int Ho, int Wo, int kh, int kw, int sh, int sw, int ph, int pw,
                                                bf_stream_t stream) {
  BF_REQUIRE(B > 0 && S > 0 && Co > 0 && Ho > 0 && Wo > 0, BF_E_INVALID, "bf_crown_relu_conv2d_bwd_noalloc: bad geometry");
  const size_t need = bf_crown_relu_conv2d_bwd_scratch_bytes(B, S, Co, Ho, Wo);
  BF_REQUIRE(need <= (size_t)BF_NOALLOC_SCRATCH_BYTES, BF_E_WORKSPACE,
             "bf_crown_relu_conv2d_bwd_noalloc: B*S*Co*Ho*Wo*4 = %zu bytes exceeds the built-in scratch of %u bytes; "
             "use bf_crown_relu_conv2d_bwd with a caller buffer",
             need, BF_NOALLOC_SCRATCH_BYTES);
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) {
    bf::set_error("bf_crown_relu_conv2d_bwd_noalloc: cannot identify the current device");
    return BF_E_CUDA;
  }
  void* scratch = g_noalloc_scratch_addr[dev];
  if (scratch == nullptr) {
    // first call on this device: resolve the symbol's device address (do this before any stream capture)
    cudaError_t e = cudaGetSymbolAddress(&scratch, g_noalloc_scratch);
    if (e != cudaSuccess || scratch == nullptr) {
      bf::set_error("bf_crown_relu_conv2d_bwd_noalloc: cudaGetSymbolAddress failed: %s", cudaGetErrorString(e));
      return BF_E_CUDA;
    }
    g_noalloc_scratch_addr[dev] = scratch;
  }
  return bf_crown_relu_conv2d_bwd(A, side, alpha_u, alpha_l, beta_u, beta_l, W, bias, A_prev, delta, accumulate, scratch,
                                  (size_t)BF_NOALLOC_SCRATCH_BYTES, B, S, Ci, Hi, Wi, Co, Ho, Wo, kh, kw, sh, sw, ph, pw, stream);
}
