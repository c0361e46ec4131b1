// Interval bound propagation through a Linear layer in centre/radius form:
//   c = (relu(l)+relu(u))/2, r = (relu(u)-relu(l))/2
//   y_l = W c - |W| r + b,  y_u = W c + |W| r + b
// fused with the preceding interval ReLU, the pre-activation constraint
// intersection and the ReLU split clamp.  One CTA owns a 64x64 output tile and
// keeps two accumulators per output (centre and radius); |W| costs nothing
// (absolute value is an operand modifier of FFMA).
#include <cooperative_groups.h>

#include "kernels.cuh"

namespace bf {

constexpr int IBM = 64, IBN = 64, IBK = 16, ILD = 68, ISLAB = IBK * ILD;

// Up to IBP_SERIAL_K terms a sum is one chain over k.  Above (the layer behind a flatten: K = 1568, 4096, 8192) it is four
// chains, one behind the other, per segment of ibp_segment(K) columns; a segment adds its chains in order, the sum its segments.
// That is the order of every kernel here, so that an input's bounds are the same bits in every batch.  Widths of hidden layers
// stay with the single chain: their bounds feed optimisation loops whose trajectories follow the last bit, and cutting it
// saves a few microseconds there; above it saves most of the time (16 x 8192 x 10: 27 us with eight segments, 113 in one chain).
constexpr int IBP_SERIAL_K = 1024, IBP_CHAINS = 4;
static int ibp_segments(int K) { return K <= 2 * IBP_SERIAL_K ? 4 : 8; }
static int ibp_segment(int K) { return ceil_div(ceil_div(K, 64), ibp_segments(K)) * 64; }

struct IbpArgs {
  const float* in_a; const float* in_b; int in_mode; int relu_in;
  const float* W; const float* bias;
  const int8_t* split; int split_stride;
  const float* cons_l; const float* cons_u;
  float* out_l; float* out_u; int* infeasible;
  int B, K, N; int vecK, vecN;
  const float* row_dev;  // [N] or null: per-output deviation (eps * dual norm of the weight row), Lp-ball first layer
};

// Two CTAs per SM (95 registers).  Forcing three (80 registers) was measured at +2 % on 8192 x 512 x 512, +10 % on the
// 784-wide first layer and -7 % on 1024 rows and fewer; four CTAs spill and lose everywhere: occupancy is not the limit.  A 64 x 128 tile (4 x 8 outputs per thread, 1.0 instead of
// 1.5 shared-memory bytes per FFMA, 128 registers) was measured at 233 against 226 us on 8192 x 512 x 512 (512 CTAs are 1.7
// waves of 296), 364 against 391 us on the 784-wide layer and 137 against 105 us on a ragged 260-wide one: not kept.
// CHAINS: sums in chains of `chain` slabs (see IBP_SERIAL_K); those of finished segments wait in shared memory.
template <bool CHAINS>
__global__ void __launch_bounds__(256) ibp_linear_kernel(IbpArgs g, int chain) {
  __shared__ __align__(16) float smem[2 * 3 * ISLAB];
  extern __shared__ __align__(16) float seg_smem[];  // CHAINS: segments before this one, [centre, radius][16][thread]
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * IBM, n0 = blockIdx.y * IBN;
  const int lrow = tid >> 2, lkc = (tid & 3) * 4;
  const bool vK = g.vecK != 0, vN = g.vecN != 0;

  float accC[4][4], accR[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) accC[i][j] = accR[i][j] = 0.f;

  float4 creg, rreg, wreg;
  auto load_slab = [&](int kt) {
    const int k = kt * IBK + lkc;
    const int m = m0 + lrow, n = n0 + lrow;
    creg = rreg = wreg = make_float4(0.f, 0.f, 0.f, 0.f);
    if (m < g.B && k < g.K) {
      float4 a = load4_guard(g.in_a + (size_t)m * g.K, k, g.K, vK);
      float4 b = g.in_b ? load4_guard(g.in_b + (size_t)m * g.K, k, g.K, vK) : make_float4(0.f, 0.f, 0.f, 0.f);
      if (g.in_mode == BF_IN_LOWER_UPPER) {
        if (g.relu_in) {
          a.x = fmaxf(a.x, 0.f); a.y = fmaxf(a.y, 0.f); a.z = fmaxf(a.z, 0.f); a.w = fmaxf(a.w, 0.f);
          b.x = fmaxf(b.x, 0.f); b.y = fmaxf(b.y, 0.f); b.z = fmaxf(b.z, 0.f); b.w = fmaxf(b.w, 0.f);
        }
        creg = make_float4((a.x + b.x) * 0.5f, (a.y + b.y) * 0.5f, (a.z + b.z) * 0.5f, (a.w + b.w) * 0.5f);
        rreg = make_float4((b.x - a.x) * 0.5f, (b.y - a.y) * 0.5f, (b.z - a.z) * 0.5f, (b.w - a.w) * 0.5f);
      } else {
        creg = a;
        rreg = b;
      }
    }
    if (n < g.N && k < g.K) wreg = load4_guard(g.W + (size_t)n * g.K, k, g.K, vK);
  };
  auto store_slab = [&](int stage) {
    float* cs = smem + stage * 3 * ISLAB;
    float* rs = cs + ISLAB;
    float* ws = rs + ISLAB;
    cs[(lkc + 0) * ILD + lrow] = creg.x; cs[(lkc + 1) * ILD + lrow] = creg.y;
    cs[(lkc + 2) * ILD + lrow] = creg.z; cs[(lkc + 3) * ILD + lrow] = creg.w;
    rs[(lkc + 0) * ILD + lrow] = rreg.x; rs[(lkc + 1) * ILD + lrow] = rreg.y;
    rs[(lkc + 2) * ILD + lrow] = rreg.z; rs[(lkc + 3) * ILD + lrow] = rreg.w;
    ws[(lkc + 0) * ILD + lrow] = wreg.x; ws[(lkc + 1) * ILD + lrow] = wreg.y;
    ws[(lkc + 2) * ILD + lrow] = wreg.z; ws[(lkc + 3) * ILD + lrow] = wreg.w;
  };

  const int nk = (g.K + IBK - 1) / IBK;
  int left = chain, chains = IBP_CHAINS;
  float segment[CHAINS ? 32 : 1];                     // of the segment's finished chains
  if (CHAINS) {
#pragma unroll
    for (int e = 0; e < 32; ++e) segment[e] = seg_smem[e * 256 + tid] = 0.f;
  }
  load_slab(0);
  store_slab(0);
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    const int stage = kt & 1;
    if (kt + 1 < nk) load_slab(kt + 1);
    const float* cs = smem + stage * 3 * ISLAB;
    const float* rs = cs + ISLAB;
    const float* ws = rs + ISLAB;
#pragma unroll
    for (int kk = 0; kk < IBK; ++kk) {
      const float4 c4 = *reinterpret_cast<const float4*>(&cs[kk * ILD + ty * 4]);
      const float4 r4 = *reinterpret_cast<const float4*>(&rs[kk * ILD + ty * 4]);
      const float4 w4 = *reinterpret_cast<const float4*>(&ws[kk * ILD + tx * 4]);
      const float c[4] = {c4.x, c4.y, c4.z, c4.w};
      const float r[4] = {r4.x, r4.y, r4.z, r4.w};
      const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          accC[i][j] = fmaf(c[i], w[j], accC[i][j]);
          accR[i][j] = fmaf(r[i], fabsf(w[j]), accR[i][j]);
        }
    }
    if (CHAINS && (--left == 0 || kt + 1 == nk)) {
      left = chain;
      const bool ends = --chains == 0 || kt + 1 == nk;
      if (ends) chains = IBP_CHAINS;
#pragma unroll
      for (int e = 0; e < 32; ++e) {
        float& acc = e < 16 ? accC[(e & 15) >> 2][e & 3] : accR[(e & 15) >> 2][e & 3];
        segment[CHAINS ? e : 0] += acc;
        acc = 0.f;
        if (ends) {
          seg_smem[e * 256 + tid] += segment[CHAINS ? e : 0];
          segment[CHAINS ? e : 0] = 0.f;
        }
      }
    }
    if (kt + 1 < nk) store_slab(stage ^ 1);
    __syncthreads();
  }
  if (CHAINS) {
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      accC[e >> 2][e & 3] = seg_smem[e * 256 + tid];
      accR[e >> 2][e & 3] = seg_smem[(16 + e) * 256 + tid];
    }
  }

  const int col = n0 + tx * 4;
  if (col >= g.N) return;
  float4 bv = make_float4(0.f, 0.f, 0.f, 0.f);
  if (g.bias) bv = load4_guard(g.bias, col, g.N, vN);
  const float bb[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int row = m0 + ty * 4 + i;
    if (row >= g.B) continue;
    float lo[4], up[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      lo[j] = (accC[i][j] - accR[i][j]) + bb[j];
      up[j] = (accC[i][j] + accR[i][j]) + bb[j];
    }
    if (g.row_dev) {  // Lp-ball first layer: deviation eps * ||W_row||_q instead of |W| * radius
      const float4 dv = load4_guard(g.row_dev, col, g.N, vN);
      const float d4[4] = {dv.x, dv.y, dv.z, dv.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        lo[j] -= d4[j];
        up[j] += d4[j];
      }
    }
    bool bad = false;
    if (g.cons_l) {
      const float4 cl = load4_guard(g.cons_l + (size_t)row * g.N, col, g.N, vN);
      const float4 cu = load4_guard(g.cons_u + (size_t)row * g.N, col, g.N, vN);
      const float cl4[4] = {cl.x, cl.y, cl.z, cl.w}, cu4[4] = {cu.x, cu.y, cu.z, cu.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (col + j < g.N) {
          lo[j] = fmaxf(lo[j], cl4[j]);
          up[j] = fminf(up[j], cu4[j]);
          bad |= lo[j] > up[j];
        }
      }
    }
    if (g.split) {
      const int8_t* sp = g.split + (size_t)row * g.split_stride;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        if (col + j < g.N) {
          const int s = sp[col + j];
          if (s > 0) lo[j] = fmaxf(lo[j], 0.f);
          if (s < 0) up[j] = fminf(up[j], 0.f);
          bad |= lo[j] > up[j];
        }
      }
    }
    store4_guard(g.out_l + (size_t)row * g.N, col, g.N, vN, make_float4(lo[0], lo[1], lo[2], lo[3]));
    store4_guard(g.out_u + (size_t)row * g.N, col, g.N, vN, make_float4(up[0], up[1], up[2], up[3]));
    if (bad && g.infeasible) g.infeasible[row] = 1;
  }
}

// bounds of one output from its centre and radius sums: bias, Lp deviation, constraint intersection, split clamp, store
__device__ __forceinline__ void ibp_finish(const IbpArgs& g, int row, int col, float c, float r) {
  const float bb = g.bias ? __ldg(g.bias + col) : 0.f;
  float lo = (c - r) + bb, up = (c + r) + bb;
  if (g.row_dev) {
    const float d = __ldg(g.row_dev + col);
    lo -= d;
    up += d;
  }
  const size_t idx = (size_t)row * g.N + col;
  bool bad = false;
  if (g.cons_l) {
    lo = fmaxf(lo, g.cons_l[idx]);
    up = fminf(up, g.cons_u[idx]);
    bad |= lo > up;
  }
  if (g.split) {
    const int s = g.split[(size_t)row * g.split_stride + col];
    if (s > 0) lo = fmaxf(lo, 0.f);
    if (s < 0) up = fminf(up, 0.f);
    bad |= lo > up;
  }
  g.out_l[idx] = lo;
  g.out_u[idx] = up;
  if (bad && g.infeasible) g.infeasible[row] = 1;
}
__device__ __forceinline__ void centre_radius(const IbpArgs& g, float& a, float& b) {
  if (g.in_mode != BF_IN_LOWER_UPPER) return;
  if (g.relu_in) { a = fmaxf(a, 0.f); b = fmaxf(b, 0.f); }
  const float c = (a + b) * 0.5f;
  b = (b - a) * 0.5f;
  a = c;
}
__device__ __forceinline__ void centre_radius4(const IbpArgs& g, float4& a, float4& b) {
  centre_radius(g, a.x, b.x); centre_radius(g, a.y, b.y); centre_radius(g, a.z, b.z); centre_radius(g, a.w, b.w);
}

// Few outputs: 64 x 64 tiles leave most SMs idle and each walks K with one 16-deep slab in flight, so the time is K / 16
// memory latencies.  Here a tile is 16 rows x 16 CPT columns, one thread per row and CPT columns, a slab 64 deep.  Every sum runs over k
// in ascending order like the 64 x 64 tiles', so both give the same bits.
// Shared slabs are [row][k] with a pitch of 68: 128-bit stores and reads without bank conflicts.
constexpr int QM = 16, QBK = 64, QLD = QBK + 4;
template <int CPT>
__global__ void __launch_bounds__(256) ibp_linear_small_kernel(IbpArgs g) {
  constexpr int QN = 16 * CPT, ROWS = 2 * QM + QN;  // centre, radius, weight rows of a slab
  __shared__ __align__(16) float smem[2 * ROWS * QLD];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int m0 = blockIdx.x * QM, n0 = blockIdx.y * QN;
  const int lk = tx * 4;
  const bool vK = g.vecK != 0;
  const bool row_ok = m0 + ty < g.B;
  const float* pa = g.in_a + (size_t)(m0 + ty) * g.K;
  const float* pb = g.in_b ? g.in_b + (size_t)(m0 + ty) * g.K : nullptr;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  float4 a4, b4, w4[CPT];
  auto load_slab = [&](int k) {
    a4 = row_ok ? load4_guard(pa, k + lk, g.K, vK) : z4;
    b4 = (row_ok && pb) ? load4_guard(pb, k + lk, g.K, vK) : z4;
#pragma unroll
    for (int j = 0; j < CPT; ++j) {
      const int n = n0 + ty + 16 * j;
      w4[j] = (n < g.N) ? load4_guard(g.W + (size_t)n * g.K, k + lk, g.K, vK) : z4;
    }
  };
  auto store_slab = [&](int stage) {
    float* s = smem + stage * ROWS * QLD;
    centre_radius4(g, a4, b4);
    *reinterpret_cast<float4*>(s + ty * QLD + lk) = a4;
    *reinterpret_cast<float4*>(s + (QM + ty) * QLD + lk) = b4;
#pragma unroll
    for (int j = 0; j < CPT; ++j) *reinterpret_cast<float4*>(s + (2 * QM + ty + 16 * j) * QLD + lk) = w4[j];
  };
  float accC[CPT], accR[CPT];
#pragma unroll
  for (int j = 0; j < CPT; ++j) accC[j] = accR[j] = 0.f;
  const int nk = (g.K + QBK - 1) / QBK;
  load_slab(0);
  store_slab(0);
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    if (kt + 1 < nk) load_slab((kt + 1) * QBK);
    const float* s = smem + (kt & 1) * ROWS * QLD;
#pragma unroll
    for (int q = 0; q < QBK; q += 4) {
      const float4 c = *reinterpret_cast<const float4*>(s + ty * QLD + q);
      const float4 r = *reinterpret_cast<const float4*>(s + (QM + ty) * QLD + q);
#pragma unroll
      for (int j = 0; j < CPT; ++j) {
        const float4 w = *reinterpret_cast<const float4*>(s + (2 * QM + tx + 16 * j) * QLD + q);
        accC[j] = fmaf(c.x, w.x, accC[j]); accR[j] = fmaf(r.x, fabsf(w.x), accR[j]);
        accC[j] = fmaf(c.y, w.y, accC[j]); accR[j] = fmaf(r.y, fabsf(w.y), accR[j]);
        accC[j] = fmaf(c.z, w.z, accC[j]); accR[j] = fmaf(r.z, fabsf(w.z), accR[j]);
        accC[j] = fmaf(c.w, w.w, accC[j]); accR[j] = fmaf(r.w, fabsf(w.w), accR[j]);
      }
    }
    if (kt + 1 < nk) store_slab((kt + 1) & 1);
    __syncthreads();
  }
  if (!row_ok) return;
#pragma unroll
  for (int j = 0; j < CPT; ++j) {
    const int col = n0 + tx + 16 * j;
    if (col < g.N) ibp_finish(g, m0 + ty, col, accC[j], accR[j]);
  }
}

// Long sums in chains (see IBP_SERIAL_K): a tile is 32 x 32; a CTA takes one segment, each of its four thread groups one chain, 16
// columns of every chain per slab (six 128-bit loads in flight per thread); the CTAs of a cluster take the segments, whose sums
// meet in distributed shared memory in rank order, without a workspace or atomics.  Measured, against one chain on 64 x 64
// tiles: 200 x 4096 x 512: 91 us (320), 256 x 1568 x 100: 17 (124), 16 x 8192 x 10: 27 (541), 600 x 6144 x 249: 162 (476).
// Issue slots 61 %, shared memory 40 %, FMA pipe 38 % busy on the first.
// Shared slabs are [k][row] with rows XOR-ed by ((k >> 2) & 7) << 2: transposed stores conflict two-way, 128-bit reads not at all.
constexpr int STM = 32, STN = 32, SBK = 64, SSLAB = SBK * 32, SGROUPS = IBP_CHAINS, SCOLS = SBK / SGROUPS;
__device__ __forceinline__ int swz(int k, int row) { return k * 32 + (row ^ (((k >> 2) & 7) << 2)); }

__global__ void __launch_bounds__(256) ibp_linear_chains_kernel(IbpArgs g, int chain) {  // chain: slabs of a chain
  __shared__ __align__(16) float smem[2 * 3 * SSLAB];
  static_assert(SGROUPS * 2 * STM * STN + 2 * STM * STN <= 2 * 3 * SSLAB, "the reduction reuses the slabs");
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int tid = threadIdx.x, kg = tid >> 6, tx = tid & 7, ty = (tid & 63) >> 3;
  const int m0 = blockIdx.x * STM, n0 = blockIdx.y * STN;
  const int k0 = blockIdx.z * SGROUPS * chain * SCOLS;
  const int lrow = tid >> 4, lk = (tid & 15) * 4;
  const int column = k0 + lk / SCOLS * chain * SCOLS + lk % SCOLS;  // this thread's in the first slab
  const bool vK = g.vecK != 0;
  float accC[4][4], accR[4][4];
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) accC[i][j] = accR[i][j] = 0.f;

  float4 creg[2], rreg[2], wreg[2];
  auto load_slab = [&](int kt) {
    const int k = column + kt * SCOLS;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int m = m0 + lrow + 16 * i, n = n0 + lrow + 16 * i;
      creg[i] = rreg[i] = wreg[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (m < g.B) {
        creg[i] = load4_guard(g.in_a + (size_t)m * g.K, k, g.K, vK);
        if (g.in_b) rreg[i] = load4_guard(g.in_b + (size_t)m * g.K, k, g.K, vK);
      }
      if (n < g.N) wreg[i] = load4_guard(g.W + (size_t)n * g.K, k, g.K, vK);
    }
  };
  auto store_slab = [&](int stage) {
    float* cs = smem + stage * 3 * SSLAB;
    float* rs = cs + SSLAB;
    float* ws = rs + SSLAB;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float4 a = creg[i], b = rreg[i];
      centre_radius4(g, a, b);
      const int r = lrow + 16 * i;
      cs[swz(lk, r)] = a.x; cs[swz(lk + 1, r)] = a.y; cs[swz(lk + 2, r)] = a.z; cs[swz(lk + 3, r)] = a.w;
      rs[swz(lk, r)] = b.x; rs[swz(lk + 1, r)] = b.y; rs[swz(lk + 2, r)] = b.z; rs[swz(lk + 3, r)] = b.w;
      ws[swz(lk, r)] = wreg[i].x; ws[swz(lk + 1, r)] = wreg[i].y; ws[swz(lk + 2, r)] = wreg[i].z; ws[swz(lk + 3, r)] = wreg[i].w;
    }
  };

  const int nk = max(0, min(chain, (g.K - k0 + SCOLS - 1) / SCOLS));
  if (nk > 0) {
    load_slab(0);
    store_slab(0);
  }
  __syncthreads();
  for (int kt = 0; kt < nk; ++kt) {
    const int stage = kt & 1;
    if (kt + 1 < nk) load_slab(kt + 1);
    const float* cs = smem + stage * 3 * SSLAB;
    const float* rs = cs + SSLAB;
    const float* ws = rs + SSLAB;
#pragma unroll
    for (int q = 0; q < SCOLS; ++q) {
      const int kk = kg * SCOLS + q;
      const float4 c4 = *reinterpret_cast<const float4*>(&cs[swz(kk, ty * 4)]);
      const float4 r4 = *reinterpret_cast<const float4*>(&rs[swz(kk, ty * 4)]);
      const float4 w4 = *reinterpret_cast<const float4*>(&ws[swz(kk, tx * 4)]);
      const float c[4] = {c4.x, c4.y, c4.z, c4.w};
      const float r[4] = {r4.x, r4.y, r4.z, r4.w};
      const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          accC[i][j] = fmaf(c[i], w[j], accC[i][j]);
          accR[i][j] = fmaf(r[i], fabsf(w[j]), accR[i][j]);
        }
    }
    if (kt + 1 < nk) store_slab(stage ^ 1);
    __syncthreads();
  }

  // chains of the segment, then segments
  float* red = smem;                                  // [SGROUPS][2][32][32]
  float* part = smem + SGROUPS * 2 * STM * STN;       // [2][32][32]
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float* d = red + kg * 2 * STM * STN + (ty * 4 + i) * STN + tx * 4;
    *reinterpret_cast<float4*>(d) = make_float4(accC[i][0], accC[i][1], accC[i][2], accC[i][3]);
    *reinterpret_cast<float4*>(d + STM * STN) = make_float4(accR[i][0], accR[i][1], accR[i][2], accR[i][3]);
  }
  __syncthreads();
  for (int e = tid; e < 2 * STM * STN; e += 256) {
    float t = red[e];
#pragma unroll
    for (int q = 1; q < SGROUPS; ++q) t += red[q * 2 * STM * STN + e];
    part[e] = t;
  }
  cluster.sync();
  const int ranks = gridDim.z;
  for (int e = blockIdx.z * 256 + tid; e < STM * STN; e += ranks * 256) {
    const int row = m0 + (e >> 5), col = n0 + (e & 31);
    if (row >= g.B || col >= g.N) continue;
    float c = 0.f, r = 0.f;
    for (int j = 0; j < ranks; ++j) {
      const float* p = cluster.map_shared_rank(part, j);
      c += p[e];
      r += p[STM * STN + e];
    }
    ibp_finish(g, row, col, c, r);
  }
  cluster.sync();  // the peers read this CTA's shared memory
}

int launch_ibp_linear(const float* in_a, const float* in_b, int in_mode, int relu_in, const float* W, const float* bias,
                      const int8_t* split, int split_stride, const float* cons_l, const float* cons_u, float* out_l,
                      float* out_u, int* infeasible, int B, int K, int N, const float* row_dev, cudaStream_t stream) {
  IbpArgs g{in_a, in_b, in_mode, relu_in, W, bias, split, split_stride, cons_l, cons_u, out_l, out_u, infeasible, B, K, N, 0, 0, row_dev};
  g.vecK = (K % 4 == 0);
  const void* kptrs[] = {in_a, in_b, W};
  for (const void* p : kptrs) if (p && (reinterpret_cast<uintptr_t>(p) & 15u)) g.vecK = 0;
  g.vecN = (N % 4 == 0);
  const void* nptrs[] = {bias, cons_l, cons_u, out_l, out_u, row_dev};
  for (const void* p : nptrs) if (p && (reinterpret_cast<uintptr_t>(p) & 15u)) g.vecN = 0;
  timing_begin(T_IBP_LINEAR, stream);
  // Measured around the lines (64 x 64 tiles; K = 100 to 1024): the small kernel takes 0.8 of the other's time at 64 tiles, 1.2 at
  // 95 (512 wide: 35 and 50 against 44 us).  Above IBP_SERIAL_K one tile per SM: 1000 x 8192 x 300
  // (80 tiles) 416 us on 32 x 32 tiles, 742 on 64 x 64; 1000 x 4096 x 512 (128) 349 and 320; 2300 x 2048 x 512 (288) 365 and 254.
  const long long tiles = (long long)ceil_div(B, IBM) * ceil_div(N, IBN);
  const dim3 grid(ceil_div(B, IBM), ceil_div(N, IBN));
  int rc = BF_OK;
  if (K <= IBP_SERIAL_K) {
    const int gx = ceil_div(B, QM);
    if (2 * tiles > 148) ibp_linear_kernel<false><<<grid, 256, 0, stream>>>(g, 0);
    else if ((long long)gx * ceil_div(N, 32) < 148) ibp_linear_small_kernel<1><<<dim3(gx, ceil_div(N, 16)), 256, 0, stream>>>(g);
    else ibp_linear_small_kernel<2><<<dim3(gx, ceil_div(N, 32)), 256, 0, stream>>>(g);
  } else {
    const int chain = ibp_segment(K) / (IBP_CHAINS * IBK);
    if (tiles < 148) {
      cudaLaunchConfig_t cfg = {};
      cfg.gridDim = dim3(ceil_div(B, STM), ceil_div(N, STN), ibp_segments(K));
      cfg.blockDim = dim3(256);
      cfg.stream = stream;
      cudaLaunchAttribute attr[1];
      attr[0].id = cudaLaunchAttributeClusterDimension;
      attr[0].val.clusterDim.x = 1; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = ibp_segments(K);
      cfg.attrs = attr;
      cfg.numAttrs = 1;
      cudaLaunchKernelEx(&cfg, ibp_linear_chains_kernel, g, chain);
    } else {
      constexpr int bytes = 32 * 256 * sizeof(float);
      static SmemOptIn opt_in;
      rc = ensure_dynamic_smem(ibp_linear_kernel<true>, bytes, opt_in, "ibp_linear_kernel");
      if (rc == BF_OK) ibp_linear_kernel<true><<<grid, 256, bytes, stream>>>(g, chain);
    }
  }
  // weights and bias once, the input interval once, both output bounds once (+ the split bytes)
  timing_end(T_IBP_LINEAR, stream, 4.0 * ((double)K * N + N) + 8.0 * (double)B * (K + N) + (split ? (double)B * N : 0.0),
             4.0 * (double)B * K * N);
  if (rc != BF_OK) return rc;
  BF_CHECK_LAUNCH("ibp_linear_kernel");
  return BF_OK;
}

}  // namespace bf

extern "C" int bf_ibp_linear(const float* in_a, const float* in_b, int in_mode, int relu_in, const float* W,
                             const float* bias, const int8_t* split, int split_stride, const float* cons_l,
                             const float* cons_u, float* out_l, float* out_u, int* infeasible, int B, int n_in,
                             int n_out, bf_stream_t stream) {
  BF_REQUIRE(in_a && in_b && W && out_l && out_u, BF_E_INVALID, "bf_ibp_linear: null tensor");
  BF_REQUIRE(B > 0 && n_in > 0 && n_out > 0, BF_E_INVALID, "bf_ibp_linear: sizes must be positive");
  BF_REQUIRE(in_mode == BF_IN_LOWER_UPPER || in_mode == BF_IN_MID_RAD, BF_E_INVALID, "bf_ibp_linear: bad in_mode");
  BF_REQUIRE(!(relu_in && in_mode == BF_IN_MID_RAD), BF_E_INVALID, "bf_ibp_linear: relu_in needs lower/upper inputs");
  BF_REQUIRE((cons_l == nullptr) == (cons_u == nullptr), BF_E_INVALID, "bf_ibp_linear: give both constraint tensors or none");
  BF_REQUIRE(!split || split_stride == 0 || split_stride == n_out, BF_E_INVALID, "bf_ibp_linear: split_stride must be 0 or n_out");
  return bf::launch_ibp_linear(in_a, in_b, in_mode, relu_in, W, bias, split, split_stride, cons_l, cons_u, out_l, out_u,
                               infeasible, B, n_in, n_out, nullptr, bf::as_stream(stream));
}

// ---------------------------------------------------------------------------
// Lp-ball (p = 1, 2, inf) support: dual-norm row reductions
// ---------------------------------------------------------------------------
namespace bf {

// out[r] = scale * ||rows[r, :]||_q with q the dual of p: p=inf -> sum |x|, p=2 -> sqrt(sum x^2), p=1 -> max |x|.
// One warp per row.
__global__ void __launch_bounds__(256) row_dual_norm_kernel(const float* __restrict__ rows, int n_rows, int n, int p, float scale,
                                                            float* __restrict__ out) {
  const int r = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= n_rows) return;
  float acc = 0.f;
  for (int k = lane; k < n; k += 32) {
    const float x = rows[(size_t)r * n + k];
    if (p == 2) acc = fmaf(x, x, acc);
    else if (p == 1) acc = fmaxf(acc, fabsf(x));
    else acc += fabsf(x);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, acc, o);
    acc = (p == 1) ? fmaxf(acc, other) : (acc + other);
  }
  if (lane == 0) out[r] = scale * ((p == 2) ? sqrtf(acc) : acc);
}

int launch_row_dual_norm(const float* rows, int n_rows, int n, int p, float scale, float* out, cudaStream_t stream) {
  row_dual_norm_kernel<<<ceil_div((long long)n_rows * 32, 256), 256, 0, stream>>>(rows, n_rows, n, p, scale, out);
  BF_CHECK_LAUNCH("row_dual_norm_kernel");
  return BF_OK;
}

// out[m] = A[m,:].center[d,:] -/+ eps * ||A[m,:]||_q + bias_in[m]
__global__ void __launch_bounds__(256) concretize_lp_kernel(const float* __restrict__ A, const float* __restrict__ center,
                                                            const float* __restrict__ bias_in, float* __restrict__ out, float sgn,
                                                            float eps, int p, int M, int S, int n0) {
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= M) return;
  const float* a = A + (size_t)m * n0;
  const float* c = center + (size_t)(m / S) * n0;
  float dot = 0.f, acc = 0.f;
  for (int k = lane; k < n0; k += 32) {
    const float x = a[k];
    dot = fmaf(x, c[k], dot);
    if (p == 2) acc = fmaf(x, x, acc);
    else if (p == 1) acc = fmaxf(acc, fabsf(x));
    else acc += fabsf(x);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    dot += __shfl_xor_sync(0xffffffffu, dot, o);
    const float other = __shfl_xor_sync(0xffffffffu, acc, o);
    acc = (p == 1) ? fmaxf(acc, other) : (acc + other);
  }
  if (lane == 0) out[m] = dot + sgn * eps * ((p == 2) ? sqrtf(acc) : acc) + (bias_in ? bias_in[m] : 0.f);
}

int launch_concretize_lp(const float* A, const float* center, const float* bias_in, float* out, int side, float eps, int p, int B,
                         int S, int n0, cudaStream_t stream) {
  const int M = B * S;
  concretize_lp_kernel<<<ceil_div((long long)M * 32, 256), 256, 0, stream>>>(A, center, bias_in, out, side == BF_SIDE_LOWER ? -1.f : 1.f,
                                                                           eps, p, M, S, n0);
  BF_CHECK_LAUNCH("concretize_lp_kernel");
  return BF_OK;
}

// Derivative of the Lp-ball lower bound  A.center - eps * ||A||_q  with respect to the coefficient row,
// written over the row itself:  H[m,k] = center[d,k] - eps * d||A[m,:]||_q / dA[m,k]
//   q = 2: A_k / ||A||_2 (0 for a zero row);  q = inf (p = 1): sign(A_k) / #maxima at the maxima of |A|, else 0;
//   q = 1 (p = inf): sign(A_k).   This is the start vector of the adjoint (gradient) sweep.
__global__ void __launch_bounds__(256) h0_lp_kernel(float* __restrict__ A, const float* __restrict__ center, float eps, int p, int M,
                                                    int S, int n0) {
  const int m = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (m >= M) return;
  float* a = A + (size_t)m * n0;
  const float* c = center + (size_t)(m / S) * n0;
  float acc = 0.f;
  for (int k = lane; k < n0; k += 32) {
    const float x = a[k];
    if (p == 2) acc = fmaf(x, x, acc);
    else if (p == 1) acc = fmaxf(acc, fabsf(x));
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, acc, o);
    acc = (p == 1) ? fmaxf(acc, other) : (acc + other);
  }
  float cnt = 0.f;
  if (p == 1) {
    for (int k = lane; k < n0; k += 32) cnt += (fabsf(a[k]) == acc) ? 1.f : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
  }
  const float nrm = (p == 2) ? sqrtf(acc) : acc;
  for (int k = lane; k < n0; k += 32) {
    const float x = a[k];
    const float sg = (x > 0.f) ? 1.f : ((x < 0.f) ? -1.f : 0.f);
    float g;
    if (p == 2) g = (nrm > 0.f) ? x / nrm : 0.f;
    else if (p == 1) g = (fabsf(x) == nrm && nrm > 0.f) ? sg / cnt : 0.f;
    else g = sg;
    a[k] = c[k] - eps * g;
  }
}

int launch_h0_lp(float* A, const float* center, float eps, int p, int B, int S, int n0, cudaStream_t stream) {
  const int M = B * S;
  h0_lp_kernel<<<ceil_div((long long)M * 32, 256), 256, 0, stream>>>(A, center, eps, p, M, S, n0);
  BF_CHECK_LAUNCH("h0_lp_kernel");
  return BF_OK;
}

}  // namespace bf

static bool lp_ok(int p) { return p == BF_NORM_INF || p == BF_NORM_L2 || p == BF_NORM_L1; }

extern "C" int bf_row_dual_norms(const float* W, int n_rows, int n_cols, int p, float scale, float* out, bf_stream_t stream) {
  BF_REQUIRE(W && out && n_rows > 0 && n_cols > 0, BF_E_INVALID, "bf_row_dual_norms: bad argument");
  BF_REQUIRE(lp_ok(p), BF_E_INVALID, "bf_row_dual_norms: p must be BF_NORM_INF, BF_NORM_L2 or BF_NORM_L1");
  return bf::launch_row_dual_norm(W, n_rows, n_cols, p, scale, out, bf::as_stream(stream));
}

extern "C" int bf_ibp_linear_lp(const float* center, const float* row_dev, const float* W, const float* bias, const int8_t* split,
                                int split_stride, const float* cons_l, const float* cons_u, float* out_l, float* out_u,
                                int* infeasible, int B, int n_in, int n_out, bf_stream_t stream) {
  BF_REQUIRE(center && row_dev && W && out_l && out_u, BF_E_INVALID, "bf_ibp_linear_lp: null tensor");
  BF_REQUIRE(B > 0 && n_in > 0 && n_out > 0, BF_E_INVALID, "bf_ibp_linear_lp: sizes must be positive");
  BF_REQUIRE((cons_l == nullptr) == (cons_u == nullptr), BF_E_INVALID, "bf_ibp_linear_lp: give both constraint tensors or none");
  return bf::launch_ibp_linear(center, nullptr, BF_IN_MID_RAD, 0, W, bias, split, split_stride, cons_l, cons_u, out_l, out_u,
                               infeasible, B, n_in, n_out, row_dev, bf::as_stream(stream));
}

// ---------------------------------------------------------------------------
// IBP linear layer whose weight differs per batch element (the output spec merged into the last
// layer: W' = C @ W, b' = C @ b): one warp per (batch element, output row), midpoint/radius form.
// HBM-bound: every weight is read once.
// ---------------------------------------------------------------------------
namespace bf {
__global__ void __launch_bounds__(256) ibp_linear_batched_kernel(const float* __restrict__ in_l, const float* __restrict__ in_u,
                                                                 int relu_in, const float* __restrict__ W,
                                                                 const float* __restrict__ bias, float* __restrict__ out_l,
                                                                 float* __restrict__ out_u, int B, int S, int n_in) {
  const long long row = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (row >= (long long)B * S) return;
  const int b = (int)(row / S);
  const float* w = W + (size_t)row * n_in;
  const float* xl = in_l + (size_t)b * n_in;
  const float* xu = in_u + (size_t)b * n_in;
  float c = 0.f, d = 0.f;
  for (int i = lane; i < n_in; i += 32) {
    float lo = xl[i], up = xu[i];
    if (relu_in) { lo = fmaxf(lo, 0.f); up = fmaxf(up, 0.f); }
    const float wv = w[i];
    c = fmaf(0.5f * (lo + up), wv, c);
    d = fmaf(0.5f * (up - lo), fabsf(wv), d);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    c += __shfl_xor_sync(0xffffffffu, c, o);
    d += __shfl_xor_sync(0xffffffffu, d, o);
  }
  if (lane == 0) {
    const float bb = bias ? bias[row] : 0.f;
    out_l[row] = c - d + bb;
    out_u[row] = c + d + bb;
  }
}
}  // namespace bf

extern "C" int bf_ibp_linear_batched(const float* in_l, const float* in_u, int relu_in, const float* W, const float* bias,
                                     float* out_l, float* out_u, int B, int S, int n_in, bf_stream_t stream) {
  BF_REQUIRE(in_l && in_u && W && out_l && out_u, BF_E_INVALID, "bf_ibp_linear_batched: null tensor");
  BF_REQUIRE(B > 0 && S > 0 && n_in > 0 && (long long)B * S < 2147483647LL, BF_E_INVALID, "bf_ibp_linear_batched: bad sizes");
  const long long warps = (long long)B * S;
  bf::ibp_linear_batched_kernel<<<(int)((warps + 7) / 8), 256, 0, bf::as_stream(stream)>>>(in_l, in_u, relu_in, W, bias, out_l, out_u,
                                                                                          B, S, n_in);
  BF_CHECK_LAUNCH("ibp_linear_batched_kernel");
  return BF_OK;
}

extern "C" int bf_concretize_lp(const float* A, const float* center, float eps, int p, const float* bias_in, float* out, int side,
                                int B, int S, int n0, bf_stream_t stream) {
  BF_REQUIRE(A && center && out, BF_E_INVALID, "bf_concretize_lp: null tensor");
  BF_REQUIRE(B > 0 && S > 0 && n0 > 0 && (long long)B * S < 2147483647LL, BF_E_INVALID, "bf_concretize_lp: bad sizes");
  BF_REQUIRE(lp_ok(p) && eps >= 0.f, BF_E_INVALID, "bf_concretize_lp: bad norm or eps");
  BF_REQUIRE(side == BF_SIDE_LOWER || side == BF_SIDE_UPPER, BF_E_INVALID, "bf_concretize_lp: bad side");
  return bf::launch_concretize_lp(A, center, bias_in, out, side, eps, p, B, S, n0, bf::as_stream(stream));
}
