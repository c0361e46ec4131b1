// FP32 contraction of small problems (too few 64 x 64 tiles to fill the GPU): 32 x 64 tiles, C[M,N] = f(A)[M,K] * B, the operands,
// prologues and order of sums of gemm_ffma.cuh.
//
// Such a launch is a serial chain: its time is the first loads, K / 32 slabs, and the epilogue.  Four warps compute, a thread
// 4 x 4 sums (two 128-bit shared-memory reads for 16 multiply-adds: 32 clocks a term; 2 x 4 sums per thread of eight warps take 48; with
// one CTA on an SM shared memory is 42 to 56 % busy, issue 43 to 52 %, the FFMA pipe 27 to 36 %), and four warps fill a ring of four slabs: weights by cp.async one slab ahead, coefficients and slopes through
// registers two slabs ahead, scaled and transposed on the way (16-byte groups of four rows, XOR-swizzled by k / 4: no conflicts).  So
// no load, conversion or barrier of the copying side sits between two slabs of the computing one, and the computing
// warps load what their epilogue needs before the first slab.
#pragma once
#include "gemm_ffma.cuh"

namespace bf {

constexpr int GS_ROWS = 32, GS_COLS = 64, GS_K = 32, GS_STAGES = 4, GS_KP = GS_K + 4;
constexpr int GS_COMPUTE = 128, GS_THREADS = 256;
constexpr int GS_A_WORDS = GS_K * GS_ROWS;
template <bool B_NT>
constexpr int GS_B_WORDS = B_NT ? GS_COLS * GS_KP : GS_K * GS_COLS;  // B_NT: [column][GS_KP], else [k][column]

__device__ __forceinline__ void gs_copy16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void gs_copy4(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
// Named barriers: 1 + s: slab s is there; 1 + GS_STAGES + s: slab s has been read
__device__ __forceinline__ void gs_sync(int id) { asm volatile("bar.sync %0, %1;" ::"r"(id), "n"(GS_THREADS) : "memory"); }
__device__ __forceinline__ void gs_arrive(int id) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "n"(GS_THREADS) : "memory"); }

struct GsRegs {
  float4 a[2], p[2], n[2], d[2];  // PRO_RELU: coefficients, slopes, split term; PRO_H0: coefficients, mid, rad
  bool got[2];
};

// The copying warps; t = 0 .. 127.
template <int PRO, bool B_NT>
__device__ __forceinline__ void gs_fill(const GemmArgs& g, const int m0, const int n0, float* As, float* Bs, const int t) {
  const bool vK = g.vecK != 0;
  const bool vB = B_NT ? g.vecK != 0 : g.vecN != 0;
  const int slabs = (g.K + GS_K - 1) / GS_K;
  const int lrow = t >> 3, lk = (t & 7) * 4;  // coefficients: rows lrow, lrow + 16, four k from lk
  const float* pa[2];
  size_t off[2];
  bool live[2];
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int m = m0 + lrow + 16 * h;
    live[h] = m < g.M;
    pa[h] = g.A + (size_t)(live[h] ? m : 0) * g.K;
    off[h] = (size_t)((live[h] ? m : 0) / g.S) * g.K;
  }
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  auto copy_b = [&](int i) {
    const int k0 = i * GS_K;
    float* dst = Bs + i % GS_STAGES * GS_B_WORDS<B_NT>;
    if (B_NT) {
      const int c0 = vB ? t >> 3 : t >> 5, kk = vB ? lk : t & 31, step = vB ? 16 : 4;
      const bool in = k0 + kk < g.K;
      const float* src = g.Bm + (size_t)(n0 + c0) * g.K + k0 + kk;
#pragma unroll 4
      for (int c = c0; c < GS_COLS; c += step, src += (size_t)step * g.K) {
        const bool ok = in && n0 + c < g.N;
        if (vB) gs_copy16(dst + c * GS_KP + kk, ok ? src : g.Bm, ok);
        else gs_copy4(dst + c * GS_KP + kk, ok ? src : g.Bm, ok);
      }
    } else {
      const int kk0 = vB ? t >> 4 : t >> 6, c = vB ? (t & 15) * 4 : t & 63, step = vB ? 8 : 2;
      const bool in = n0 + c < g.N;
      const float* src = g.Bm + (size_t)(k0 + kk0) * g.N + n0 + c;
#pragma unroll 4
      for (int kk = kk0; kk < GS_K; kk += step, src += (size_t)step * g.N) {
        const bool ok = in && k0 + kk < g.K;
        if (vB) gs_copy16(dst + kk * GS_COLS + c, ok ? src : g.Bm, ok);
        else gs_copy4(dst + kk * GS_COLS + c, ok ? src : g.Bm, ok);
      }
    }
  };
  auto load_a = [&](int i, GsRegs& r) {
    const int k = i * GS_K + lk;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      r.got[h] = live[h] && k < g.K;
      r.a[h] = r.p[h] = r.n[h] = r.d[h] = z4;
      if (r.got[h]) {
        r.a[h] = load4_plain(pa[h], k, g.K, vK);
        if (PRO == PRO_RELU && g.dpos) {
          r.p[h] = load4_plain(g.dpos + off[h], k, g.K, vK);
          r.n[h] = load4_plain(g.dneg + off[h], k, g.K, vK);
          if (g.add) r.d[h] = load4_plain(g.add + off[h], k, g.K, vK);
        } else if (PRO == PRO_H0) {
          r.p[h] = load4_plain(g.mid + off[h], k, g.K, vK);
          r.n[h] = load4_plain(g.rad + off[h], k, g.K, vK);
        }
      }
    }
  };
  auto store_a = [&](int i, const GsRegs& r) {
    float* as = As + i % GS_STAGES * GS_A_WORDS + lk * GS_ROWS;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      float4 a = r.a[h];
      if (r.got[h]) {
        if (PRO == PRO_RELU && g.dpos) {
          a.x = a.x * (a.x >= 0.f ? r.p[h].x : r.n[h].x) + r.d[h].x;
          a.y = a.y * (a.y >= 0.f ? r.p[h].y : r.n[h].y) + r.d[h].y;
          a.z = a.z * (a.z >= 0.f ? r.p[h].z : r.n[h].z) + r.d[h].z;
          a.w = a.w * (a.w >= 0.f ? r.p[h].w : r.n[h].w) + r.d[h].w;
        } else if (PRO == PRO_H0) {
          a.x = r.p[h].x - sgnf(a.x) * r.n[h].x;
          a.y = r.p[h].y - sgnf(a.y) * r.n[h].y;
          a.z = r.p[h].z - sgnf(a.z) * r.n[h].z;
          a.w = r.p[h].w - sgnf(a.w) * r.n[h].w;
        }
      }
      const int row = lrow + 16 * h;
      float* d = as + (((row >> 2) ^ (lk >> 2)) << 2) + (row & 3);
      d[0] = a.x; d[GS_ROWS] = a.y; d[2 * GS_ROWS] = a.z; d[3 * GS_ROWS] = a.w;
    }
  };
  GsRegs r0, r1;
  copy_b(0);
  asm volatile("cp.async.commit_group;" ::: "memory");
  load_a(0, r0);
  if (slabs > 1) load_a(1, r1);
  auto slab = [&](int i, GsRegs& r) {
    if (i + 1 < slabs) {
      if (i + 1 >= GS_STAGES) gs_sync(1 + GS_STAGES + (i + 1) % GS_STAGES);
      copy_b(i + 1);
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
    store_a(i, r);
    if (i + 2 < slabs) load_a(i + 2, r);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    gs_arrive(1 + i % GS_STAGES);
  };
  for (int i = 0; i < slabs; i += 2) {
    slab(i, r0);
    if (i + 1 < slabs) slab(i + 1, r1);
  }
}

// The computing warps: rows r0 .. r0 + 3 of the tile; columns c0 .. c0 + 3, or c0, c0 + 8, + 16, + 24 (B_NT).
template <bool B_NT>
__device__ __forceinline__ void gs_compute(const int K, const float* As, const float* Bs, const int r0, const int c0, float (&acc)[4][4]) {
  const int slabs = (K + GS_K - 1) / GS_K, chunk = r0 >> 2;
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
  for (int i = 0; i < slabs; ++i) {
    const int s = i % GS_STAGES;
    gs_sync(1 + s);
    const float* as = As + s * GS_A_WORDS;
    const float* bs = Bs + s * GS_B_WORDS<B_NT> + (B_NT ? c0 * GS_KP : c0);
    auto terms = [&](int kk) {  // four; past the end of K both operands are zero
      const float* ap = as + kk * GS_ROWS + ((chunk ^ (kk >> 2)) << 2);
      float a[4][4], b[4][4];   // a[term][row], b[term][column]
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const float4 x = *reinterpret_cast<const float4*>(ap + q * GS_ROWS);
        const float4 y = *reinterpret_cast<const float4*>(B_NT ? bs + 8 * q * GS_KP + kk : bs + (kk + q) * GS_COLS);
        a[q][0] = x.x; a[q][1] = x.y; a[q][2] = x.z; a[q][3] = x.w;
        if (B_NT) { b[0][q] = y.x; b[1][q] = y.y; b[2][q] = y.z; b[3][q] = y.w; }
        else { b[q][0] = y.x; b[q][1] = y.y; b[q][2] = y.z; b[q][3] = y.w; }
      }
#pragma unroll
      for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int m = 0; m < 4; ++m)
#pragma unroll
          for (int n = 0; n < 4; ++n) acc[m][n] = fmaf(a[q][m], b[q][n], acc[m][n]);
    };
    const int left = K - i * GS_K;
    if (left >= GS_K) {
#pragma unroll
      for (int kk = 0; kk < GS_K; kk += 4) terms(kk);
    } else {
#pragma unroll 1
      for (int kk = 0; kk < left; kk += 4) terms(kk);
    }
    if (i + GS_STAGES < slabs) gs_arrive(1 + GS_STAGES + s);
  }
}

// delta[m] (+)= sum_k a * intercept + lam * kbias of 32 rows, in gemm_mainloop's order: four threads per row, thread p the
// columns 16 t + 4 p .. + 3 of every t, then their sums pairwise.
__device__ __forceinline__ void prologue_row_sums(const GemmArgs& g, const int m0) {
  const int row = m0 + ((int)threadIdx.x >> 2), lkc = ((int)threadIdx.x & 3) * 4;
  if (threadIdx.x >= 128) return;
  const bool vK = g.vecK != 0, live = row < g.M;
  const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
  const float* pa = g.A + (size_t)(live ? row : 0) * g.K;
  const size_t off = live ? (size_t)(row / g.S) * g.K : 0;
  float r = 0.f;
  constexpr int U = 4;                              // column groups in flight
  for (int k0 = lkc; k0 < g.K && live; k0 += 16 * U) {
    float4 a[U], kb[U], dp[U], dn[U], ep[U], en[U], ad[U];
#pragma unroll
    for (int u = 0; u < U; ++u) {
      const int k = k0 + 16 * u;
      a[u] = kb[u] = dp[u] = dn[u] = ep[u] = en[u] = ad[u] = z4;
      if (k < g.K) {
        a[u] = load4_plain(pa, k, g.K, vK);
        if (g.kbias) kb[u] = load4_plain(g.kbias, k, g.K, vK);
        if (g.dpos) {
          dp[u] = load4_plain(g.dpos + off, k, g.K, vK);
          dn[u] = load4_plain(g.dneg + off, k, g.K, vK);
          if (g.epos) ep[u] = load4_plain(g.epos + off, k, g.K, vK);
          if (g.eneg) en[u] = load4_plain(g.eneg + off, k, g.K, vK);
          if (g.add) ad[u] = load4_plain(g.add + off, k, g.K, vK);
        }
      }
    }
#pragma unroll
    for (int u = 0; u < U; ++u) {
      if (k0 + 16 * u >= g.K) break;
      if (g.dpos) {
#define BF_ROW_SUM(c)                                                          \
  {                                                                            \
    const bool sel = a[u].c >= 0.f;                                            \
    const float lam = a[u].c * (sel ? dp[u].c : dn[u].c) + ad[u].c;            \
    r += a[u].c * (sel ? ep[u].c : en[u].c);                                   \
    r = fmaf(lam, kb[u].c, r);                                                 \
  }
        BF_ROW_SUM(x) BF_ROW_SUM(y) BF_ROW_SUM(z) BF_ROW_SUM(w)
#undef BF_ROW_SUM
      } else {
        r += a[u].x * kb[u].x + a[u].y * kb[u].y + a[u].z * kb[u].z + a[u].w * kb[u].w;
      }
    }
  }
  r += __shfl_xor_sync(0xffffffffu, r, 1);
  r += __shfl_xor_sync(0xffffffffu, r, 2);
  if (lkc == 0 && live) g.delta[row] = g.accumulate ? (g.delta[row] + r) : r;
}

}  // namespace bf
