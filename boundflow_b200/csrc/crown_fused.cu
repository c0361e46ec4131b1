// CROWN sweeps of small batches through Linear layers, one launch per sweep: a cluster of CTAs takes 32 coefficient rows through
// all layers.
//
// A row's coefficients in one layer depend on the same row's in the layer above only, so 32 rows need no other rows: the CTAs of a
// cluster share the columns of every layer in tiles of 64 and write their results, with the next layer's ReLU scaling applied, into
// every CTA's shared memory; a cluster barrier per layer is the only synchronisation.  Weights do not depend on the
// sweep, so their slabs stream ahead across tiles and layers.  One launch per layer spends half its time on the launch, the first
// slabs and the epilogue's loads (1152 rows, 256 x 256: 12 us and a gap of 2 to 3 us, the multiply-adds of it 2 us).
// A thread of the four computing warps holds 4 x 4 sums: two 128-bit shared-memory reads for 16 multiply-adds, which is what bounds
// a layer (4 us at 32 x 64 sums per SM and 256 terms).
// Every sum keeps the order of the layer-by-layer kernels (terms ascending; row sums, concretisation and gradient sums as there), so
// the results are the same bits.
#include <cooperative_groups.h>

#include "gemm_ffma.cuh"
#include "kernels.cuh"

namespace bf {

constexpr int FS_ROWS = 32, FS_COLS = 64, FS_K = 32, FS_STAGES = 3, FS_COMPUTE = 128;
constexpr int FS_KP = FS_K + 4;  // adjoint: pitch of a weight row's slab

__device__ __forceinline__ void fs_copy16(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void fs_copy4(float* dst, const float* src, bool ok) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 4 : 0) : "memory");
}
__device__ __forceinline__ void fs_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void fs_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
__device__ __forceinline__ void fs_bar() { asm volatile("bar.sync 1, 128;" ::: "memory"); }  // the computing warps

// position in the stream of weight slabs: layer, tile of this CTA, slab
struct FsCursor {
  int layer, tile, k0;
};

// ---------------------------------------------------------------------------
// backward sweep
// ---------------------------------------------------------------------------
__device__ __forceinline__ void fs_advance(const FusedSweepArgs& a, FsCursor& c, int ranks, int rank) {
  while (c.layer < a.layers) {
    const FusedSweepLayer& L = a.L[c.layer];
    if (c.tile * FS_COLS < L.N && c.k0 < L.K) return;
    if (c.tile * FS_COLS < L.N) { c.tile += ranks; c.k0 = 0; }
    if (c.tile * FS_COLS >= L.N) { ++c.layer; c.tile = rank; c.k0 = 0; }
  }
}

__global__ void __launch_bounds__(256, 2) crown_fused_bwd_kernel(FusedSweepArgs a) {
  extern __shared__ __align__(16) float fs_smem[];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int m0 = (int)(blockIdx.x / ranks) * FS_ROWS;
  float* As[2] = {fs_smem, fs_smem + a.kmax * FS_ROWS};     // [k][row], coefficients after the ReLU scaling
  float* Bs = fs_smem + 2 * a.kmax * FS_ROWS;               // [stage][k][column]
  float* pbuf = Bs + FS_STAGES * FS_K * FS_COLS;            // [row]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const bool computing = tid < FS_COMPUTE;

  // spec rows
  for (int k = warp; k < a.L[0].K; k += 8) As[0][k * FS_ROWS + lane] = (m0 + lane < a.M) ? a.C[(size_t)(m0 + lane) * a.L[0].K + k] : 0.f;

  FsCursor next{0, rank, 0};
  int fetched = 0, used = 0;
  auto fetch = [&]() {
    fs_advance(a, next, ranks, rank);
    if (next.layer < a.layers) {
      const FusedSweepLayer& L = a.L[next.layer];
      float* dst = Bs + fetched % FS_STAGES * (FS_K * FS_COLS);
      const int n0 = next.tile * FS_COLS;
      if (L.vec) {
#pragma unroll
        for (int j = 0; j < FS_K * FS_COLS / 4 / FS_COMPUTE; ++j) {
          const int e = tid + j * FS_COMPUTE, kk = e / (FS_COLS / 4), c = e % (FS_COLS / 4) * 4;
          const bool ok = next.k0 + kk < L.K && n0 + c < L.N;
          fs_copy16(dst + kk * FS_COLS + c, ok ? L.W + (size_t)(next.k0 + kk) * L.N + n0 + c : L.W, ok);
        }
      } else {
#pragma unroll 4
        for (int j = 0; j < FS_K * FS_COLS / FS_COMPUTE; ++j) {
          const int e = tid + j * FS_COMPUTE, kk = e / FS_COLS, c = e % FS_COLS;
          const bool ok = next.k0 + kk < L.K && n0 + c < L.N;
          fs_copy4(dst + kk * FS_COLS + c, ok ? L.W + (size_t)(next.k0 + kk) * L.N + n0 + c : L.W, ok);
        }
      }
      next.k0 += FS_K;
    }
    ++fetched;
    fs_commit();
  };
  if (computing)
    for (int i = 0; i < FS_STAGES - 1; ++i) fetch();
  cluster.sync();  // every CTA of the cluster runs, and its spec rows are in place

  // computing warps: rows r0 .. r0 + 3, columns c0 .. c0 + 3 of a tile
  const int tx = lane & 7, ty = lane >> 3;
  const int r0 = (warp >> 1) * 16 + ty * 4, c0 = (warp & 1) * 32 + tx * 4;
  const float sgn = (a.side == BF_SIDE_LOWER) ? -1.f : 1.f;
  float delta = 0.f;  // row-sum warps of the last rank
  for (int l = 0; l < a.layers; ++l) {
    const FusedSweepLayer& L = a.L[l];
    const bool last = l + 1 == a.layers;
    if (computing) {
      const float* A = As[l & 1];
      for (int tile = rank; tile * FS_COLS < L.N; tile += ranks) {
        const int col = tile * FS_COLS + c0;
        // what the epilogue needs: the next layer's slopes and split terms, or the input box
        float4 x[4], y[4], z[4];
        const float* px = last ? a.mid : a.L[l + 1].dpos;
        const float* py = last ? a.rad : a.L[l + 1].dneg;
        const float* pz = last ? nullptr : a.L[l + 1].add;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          x[i] = y[i] = z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
          const int row = m0 + r0 + i;
          if (row < a.M && col < L.N) {
            const size_t off = (size_t)(row / a.S) * L.N;
            if (px) x[i] = load4_guard(px + off, col, L.N, L.vec);
            if (py) y[i] = load4_guard(py + off, col, L.N, L.vec);
            if (pz) z[i] = load4_guard(pz + off, col, L.N, L.vec);
          }
        }
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
          for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
        for (int k0 = 0; k0 < L.K; k0 += FS_K, ++used) {
          fs_wait<FS_STAGES - 2>();
          fs_bar();                                   // this slab is there, and nobody reads the one before it any more
          fetch();
          const float* as = A + k0 * FS_ROWS + r0;
          const float* bs = Bs + used % FS_STAGES * (FS_K * FS_COLS) + c0;
          const int left = min(FS_K, L.K - k0);
          auto step = [&](int kk) {
            const float4 p = *reinterpret_cast<const float4*>(as + kk * FS_ROWS);
            const float4 q = *reinterpret_cast<const float4*>(bs + kk * FS_COLS);
            const float av[4] = {p.x, p.y, p.z, p.w}, bv[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], bv[j], acc[i][j]);
          };
          if (left == FS_K) {
#pragma unroll
            for (int kk = 0; kk < FS_K; ++kk) step(kk);
          } else {
#pragma unroll 1
            for (int kk = 0; kk < left; ++kk) step(kk);
          }
        }
        // raw coefficients
        if (L.out && col < L.N) {
#pragma unroll
          for (int i = 0; i < 4; ++i)
            if (m0 + r0 + i < a.M)
              store4_guard(L.out + (size_t)(m0 + r0 + i) * L.N, col, L.N, L.vec, make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]));
        }
        if (!last) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float xs[4] = {x[i].x, x[i].y, x[i].z, x[i].w}, ys[4] = {y[i].x, y[i].y, y[i].z, y[i].w}, zs[4] = {z[i].x, z[i].y, z[i].z, z[i].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(acc[i][j], acc[i][j] >= 0.f ? xs[j] : ys[j], zs[j]);
          }
          float* to = As[(l + 1) & 1] + r0;
          for (int q = 0; q < ranks; ++q) {
            float* p = cluster.map_shared_rank(to, (rank + q) % ranks);
#pragma unroll
            for (int j = 0; j < 4; ++j)
              if (col + j < L.N) *reinterpret_cast<float4*>(p + (size_t)(col + j) * FS_ROWS) = make_float4(acc[0][j], acc[1][j], acc[2][j], acc[3][j]);
          }
        } else if (a.partial) {
          float p4[4];
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            float p = 0.f;
            const float4 v = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]), md = x[i], rd = y[i];
            p += v.x * md.x + sgn * fabsf(v.x) * rd.x;
            p += v.y * md.y + sgn * fabsf(v.y) * rd.y;
            p += v.z * md.z + sgn * fabsf(v.z) * rd.z;
            p += v.w * md.w + sgn * fabsf(v.w) * rd.w;
            p += __shfl_xor_sync(0xffffffffu, p, 1);
            p += __shfl_xor_sync(0xffffffffu, p, 2);
            p += __shfl_xor_sync(0xffffffffu, p, 4);
            p4[i] = p;
            if ((warp & 1) && tx == 0) pbuf[r0 + i] = p;
          }
          fs_bar();
          if (!(warp & 1) && tx == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
              if (m0 + r0 + i < a.M) a.partial[(size_t)(m0 + r0 + i) * a.ptiles + tile] = p4[i] + pbuf[r0 + i];
          }
          fs_bar();
        }
      }
    } else if (rank == ranks - 1) {
      // row sums of this layer's prologue: four threads per row (gemm_mainloop's order)
      const int t = tid - FS_COMPUTE, row = m0 + (t >> 2), lkc = (t & 3) * 4;
      if (row < a.M) {
        const float* pa = (l == 0) ? a.C + (size_t)row * L.K : a.L[l - 1].out + (size_t)row * L.K;
        const size_t off = (size_t)(row / a.S) * L.K;
        float r = 0.f;
        if (l == 0 && a.thin_top) {
          if (lkc == 0 && L.kbias)
            for (int k = 0; k < L.K; ++k) r = fmaf(pa[k], __ldg(L.kbias + k), r);
        } else {
          constexpr int U = 4;
          const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
          for (int k0 = lkc; k0 < L.K; k0 += 16 * U) {
            float4 v[U], kb[U], dp[U], dn[U], ep[U], en[U], ad[U];
#pragma unroll
            for (int u = 0; u < U; ++u) {
              const int k = k0 + 16 * u;
              v[u] = kb[u] = dp[u] = dn[u] = ep[u] = en[u] = ad[u] = z4;
              if (k < L.K) {
                v[u] = load4_plain(pa, k, L.K, L.veck);  // written by other CTAs of the cluster during this launch
                if (L.kbias) kb[u] = load4_guard(L.kbias, k, L.K, L.veck);
                if (L.dpos) {
                  dp[u] = load4_guard(L.dpos + off, k, L.K, L.veck);
                  dn[u] = load4_guard(L.dneg + off, k, L.K, L.veck);
                  if (L.epos) ep[u] = load4_guard(L.epos + off, k, L.K, L.veck);
                  if (L.eneg) en[u] = load4_guard(L.eneg + off, k, L.K, L.veck);
                  if (L.add) ad[u] = load4_guard(L.add + off, k, L.K, L.veck);
                }
              }
            }
#pragma unroll
            for (int u = 0; u < U; ++u) {
              if (k0 + 16 * u >= L.K) break;
              if (L.dpos) {
#define BF_ROW_SUM(c)                                                          \
  {                                                                            \
    const bool sel = v[u].c >= 0.f;                                            \
    const float lam = v[u].c * (sel ? dp[u].c : dn[u].c) + ad[u].c;            \
    r += v[u].c * (sel ? ep[u].c : en[u].c);                                   \
    r = fmaf(lam, kb[u].c, r);                                                 \
  }
                BF_ROW_SUM(x) BF_ROW_SUM(y) BF_ROW_SUM(z) BF_ROW_SUM(w)
#undef BF_ROW_SUM
              } else {
                r += v[u].x * kb[u].x + v[u].y * kb[u].y + v[u].z * kb[u].z + v[u].w * kb[u].w;
              }
            }
          }
        }
        const unsigned quad = 0xfu << (lane & ~3);
        if (!(l == 0 && a.thin_top)) {
          r += __shfl_xor_sync(quad, r, 1);
          r += __shfl_xor_sync(quad, r, 2);
        }
        delta = (l == 0) ? r : delta + r;
        if (last && lkc == 0) a.delta[row] = delta;
      }
    }
    cluster.sync();  // the next layer's coefficients are complete in every CTA; nobody leaves before the others' last stores to it
  }
}

// ---------------------------------------------------------------------------
// adjoint (gradient) sweep
// ---------------------------------------------------------------------------
__device__ __forceinline__ void fs_advance(const FusedAdjointArgs& a, FsCursor& c, int ranks, int rank) {
  while (c.layer < a.layers) {
    const FusedAdjointLayer& L = a.L[c.layer];
    if (c.tile * FS_COLS < L.N && c.k0 < L.K) return;
    if (c.tile * FS_COLS < L.N) { c.tile += ranks; c.k0 = 0; }
    if (c.tile * FS_COLS >= L.N) { ++c.layer; c.tile = rank; c.k0 = 0; }
  }
}

__global__ void __launch_bounds__(FS_COMPUTE, 2) crown_fused_adjoint_kernel(FusedAdjointArgs a) {
  extern __shared__ __align__(16) float fs_smem[];
  cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int ranks = (int)cluster.num_blocks(), rank = (int)cluster.block_rank();
  const int m0 = (int)(blockIdx.x / ranks) * FS_ROWS;
  float* As[2] = {fs_smem, fs_smem + a.kmax * FS_ROWS};      // [k][row], adjoint points between layers
  float* Bs = fs_smem + 2 * a.kmax * FS_ROWS;                // [stage][column][FS_KP]
  float* A0s = Bs + FS_STAGES * FS_COLS * FS_KP;             // [2][k][row], slabs of the points at the network input
  float* red = A0s + 2 * FS_K * FS_ROWS;                     // [row][FS_COLS + 1]
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  FsCursor next{0, rank, 0};
  int fetched = 0, used = 0;
  auto fetch = [&]() {
    fs_advance(a, next, ranks, rank);
    if (next.layer < a.layers) {
      const FusedAdjointLayer& L = a.L[next.layer];
      float* dst = Bs + fetched % FS_STAGES * (FS_COLS * FS_KP);
      const int n0 = next.tile * FS_COLS;
      if (L.veck) {
#pragma unroll
        for (int j = 0; j < FS_K * FS_COLS / 4 / FS_COMPUTE; ++j) {
          const int e = tid + j * FS_COMPUTE, c = e / (FS_K / 4), kk = e % (FS_K / 4) * 4;
          const bool ok = next.k0 + kk < L.K && n0 + c < L.N;
          fs_copy16(dst + c * FS_KP + kk, ok ? L.W + (size_t)(n0 + c) * L.K + next.k0 + kk : L.W, ok);
        }
      } else {
#pragma unroll 4
        for (int j = 0; j < FS_K * FS_COLS / FS_COMPUTE; ++j) {
          const int e = tid + j * FS_COMPUTE, c = e / FS_K, kk = e % FS_K;
          const bool ok = next.k0 + kk < L.K && n0 + c < L.N;
          fs_copy4(dst + c * FS_KP + kk, ok ? L.W + (size_t)(n0 + c) * L.K + next.k0 + kk : L.W, ok);
        }
      }
      next.k0 += FS_K;
    }
    ++fetched;
    fs_commit();
  };
  for (int i = 0; i < FS_STAGES - 1; ++i) fetch();

  // points at the network input, one slab ahead in registers: row = lane, k = 8 * warp .. + 7
  const int arow = m0 + lane;
  float4 ha[2], hm[2], hr[2];
  auto load_h0 = [&](int k0) {
    const int K = a.L[0].K;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const int k = k0 + warp * 8 + i * 4;
      ha[i] = hm[i] = hr[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      if (arow < a.M && k < K) {
        ha[i] = load4_guard(a.A0 + (size_t)arow * K, k, K, a.L[0].veck);
        if (a.mid) {
          const size_t off = (size_t)(arow / a.S) * K;
          hm[i] = load4_guard(a.mid + off, k, K, a.L[0].veck);
          hr[i] = load4_guard(a.rad + off, k, K, a.L[0].veck);
        }
      }
    }
  };
  auto store_h0 = [&](float* to) {
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      float4 v = ha[i];
      if (a.mid) {
        v.x = hm[i].x - sgnf(v.x) * hr[i].x;
        v.y = hm[i].y - sgnf(v.y) * hr[i].y;
        v.z = hm[i].z - sgnf(v.z) * hr[i].z;
        v.w = hm[i].w - sgnf(v.w) * hr[i].w;
      }
      float* d = to + (warp * 8 + i * 4) * FS_ROWS + lane;
      d[0] = v.x; d[FS_ROWS] = v.y; d[2 * FS_ROWS] = v.z; d[3 * FS_ROWS] = v.w;
    }
  };
  cluster.sync();  // every CTA of the cluster runs

  const int tx = lane & 7, ty = lane >> 3;
  const int r0 = (warp >> 1) * 16 + ty * 4, c0 = (warp & 1) * 32 + tx;  // columns c0, c0 + 8, + 16, + 24
  for (int l = 0; l < a.layers; ++l) {
    const FusedAdjointLayer& L = a.L[l];
    for (int tile = rank; tile * FS_COLS < L.N; tile += ranks) {
      const int n0 = tile * FS_COLS;
      float ah[4][4], dp[4][4], dn[4][4], ep[4][4], en[4][4];
      bool amb[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          ah[i][j] = dp[i][j] = dn[i][j] = ep[i][j] = en[i][j] = 0.f;
          amb[i][j] = false;
          const int row = m0 + r0 + i, col = n0 + c0 + 8 * j;
          if (row < a.M && col < L.N) {
            const size_t off = (size_t)(row / a.S) * L.N + col;
            ah[i][j] = __ldg(L.Ahat + (size_t)row * L.N + col);
            dp[i][j] = __ldg(L.dpos + off);
            dn[i][j] = __ldg(L.dneg + off);
            if (L.epos) ep[i][j] = __ldg(L.epos + off);
            if (L.eneg) en[i][j] = __ldg(L.eneg + off);
            amb[i][j] = __ldg(L.pre_l + off) < 0.f && __ldg(L.pre_u + off) > 0.f;
          }
        }
      float acc[4][4];
#pragma unroll
      for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;
      if (l == 0) load_h0(0);
      for (int k0 = 0; k0 < L.K; k0 += FS_K, ++used) {
        if (l == 0) store_h0(A0s + (k0 / FS_K & 1) * (FS_K * FS_ROWS));
        fs_wait<FS_STAGES - 2>();
        __syncthreads();                              // this slab is there, and nobody reads the one before it any more
        fetch();
        if (l == 0 && k0 + FS_K < L.K) load_h0(k0 + FS_K);
        const float* as = (l == 0 ? A0s + (k0 / FS_K & 1) * (FS_K * FS_ROWS) : As[l & 1] + k0 * FS_ROWS) + r0;
        const float* bs = Bs + used % FS_STAGES * (FS_COLS * FS_KP) + c0 * FS_KP;
        const int left = min(FS_K, L.K - k0);
        auto step = [&](int kk) {                     // four terms; past the end of K both operands are zero
          float av[4][4], bv[4][4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const float4 p = *reinterpret_cast<const float4*>(as + (kk + q) * FS_ROWS);
            const float4 b = *reinterpret_cast<const float4*>(bs + 8 * q * FS_KP + kk);
            av[q][0] = p.x; av[q][1] = p.y; av[q][2] = p.z; av[q][3] = p.w;
            bv[q][0] = b.x; bv[q][1] = b.y; bv[q][2] = b.z; bv[q][3] = b.w;
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
              for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[q][i], bv[j][q], acc[i][j]);
        };
        if (left == FS_K) {
#pragma unroll
          for (int kk = 0; kk < FS_K; kk += 4) step(kk);
        } else {
#pragma unroll 1
          for (int kk = 0; kk < left; kk += 4) step(kk);
        }
      }
      __syncthreads();                                // `red` of the tile before is read, A0s too
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const int col = n0 + c0 + 8 * j;
        const float nb = (L.nbias && col < L.N) ? __ldg(L.nbias + col) : 0.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float gg = acc[i][j] + nb;
          const bool sel = ah[i][j] >= 0.f;
          red[(r0 + i) * (FS_COLS + 1) + c0 + 8 * j] = (sel && amb[i][j]) ? ah[i][j] * gg : 0.f;
          dp[i][j] = (sel ? dp[i][j] : dn[i][j]) * gg + (sel ? ep[i][j] : en[i][j]);
          acc[i][j] = (m0 + r0 + i < a.M) ? gg : 0.f;
        }
      }
      if (l + 1 < a.layers) {
        float* to = As[(l + 1) & 1] + r0;
        const int np = (L.N + 3) & ~3;                // columns past the end carry zeros
        for (int q = 0; q < ranks; ++q) {
          float* p = cluster.map_shared_rank(to, (rank + q) % ranks);
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            const int col = n0 + c0 + 8 * j;
            if (col < np)
              *reinterpret_cast<float4*>(p + (size_t)col * FS_ROWS) = col < L.N ? make_float4(dp[0][j], dp[1][j], dp[2][j], dp[3][j]) : make_float4(0.f, 0.f, 0.f, 0.f);
          }
        }
      }
      // per-domain sums over the rows of this tile
      const int m_end = min(m0 + FS_ROWS, a.M), d_first = m0 / a.S, d_last = (m_end - 1) / a.S;
      const int c = tid % FS_COLS, half = tid / FS_COLS, col = n0 + c;
      auto reduce = [&](float* to) {
        __syncthreads();
        for (int d = d_first + half; d <= d_last; d += FS_COMPUTE / FS_COLS) {
          const int lo = max(d * a.S, m0) - m0, hi = min((d + 1) * a.S, m_end) - m0;
          float s = 0.f;
          for (int r = lo; r < hi; ++r) s += red[r * (FS_COLS + 1) + c];
          if (col < L.N) atomicAdd(to + (size_t)d * L.N + col, s);
        }
      };
      reduce(L.grad);
      if (L.gsum) {
        __syncthreads();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const float w = (a.gw && m0 + r0 + i < a.M) ? __ldg(a.gw + m0 + r0 + i) : 1.f;
#pragma unroll
          for (int j = 0; j < 4; ++j) red[(r0 + i) * (FS_COLS + 1) + c0 + 8 * j] = a.gw ? acc[i][j] * w : acc[i][j];
        }
        reduce(L.gsum);
      }
    }
    cluster.sync();
  }
}

// ---------------------------------------------------------------------------
// launchers
// ---------------------------------------------------------------------------
static size_t fused_bwd_smem(int kmax) { return ((size_t)2 * kmax * FS_ROWS + FS_STAGES * FS_K * FS_COLS + FS_ROWS) * sizeof(float); }
static size_t fused_adjoint_smem(int kmax) {
  return ((size_t)2 * kmax * FS_ROWS + FS_STAGES * FS_COLS * FS_KP + 2 * FS_K * FS_ROWS + FS_ROWS * (FS_COLS + 1)) * sizeof(float);
}
constexpr int FUSED_SMEM = 220 * 1024;

// Clusters of cs CTAs that run at once, for kernels of up to HALF_SM or FUSED_SMEM bytes of shared memory (a property of the device)
constexpr size_t HALF_SM = 112 * 1024;
struct ClusterRoom {
  std::atomic<int> active[MAX_DEVICES][2][4];  // [device][half an SM or more][log2 cs], plus one; 0: not asked yet
};
template <typename Kernel>
static int clusters_at_once(Kernel kernel, int threads, size_t smem, int csl, ClusterRoom& room) {
  int dev = -1;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= MAX_DEVICES) return 0;
  std::atomic<int>& slot = room.active[dev][smem > HALF_SM][csl];
  int known = slot.load(std::memory_order_relaxed);
  if (known == 0) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(148 << csl);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem > HALF_SM ? FUSED_SMEM : HALF_SM;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1 << csl; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    int active = 0;
    if (cudaOccupancyMaxActiveClusters(&active, kernel, &cfg) != cudaSuccess) { (void)cudaGetLastError(); active = 0; }
    known = active + 1;
    slot.store(known, std::memory_order_relaxed);
  }
  return known - 1;
}

// CTAs per cluster for M rows: as many as have a tile in the widest layer, and as let every cluster run at once (0: none do)
template <typename Kernel>
static int fused_cluster(Kernel kernel, int threads, size_t smem, int M, int widest, ClusterRoom& room) {
  const int clusters = ceil_div(M, FS_ROWS), tiles = ceil_div(widest, FS_COLS);
  for (int csl = 3; csl >= 1; --csl)
    if ((1 << (csl - 1)) < tiles && clusters <= clusters_at_once(kernel, threads, smem, csl, room)) return 1 << csl;
  return 0;
}

template <typename Kernel, typename Args>
static int fused_launch(Kernel kernel, const Args& a, int threads, size_t smem, int cs, cudaStream_t stream, const char* name) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(ceil_div(a.M, FS_ROWS) * cs);
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = cs; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  cudaLaunchKernelEx(&cfg, kernel, a);
  BF_CHECK_LAUNCH(name);
  return BF_OK;
}

static bool al16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

int launch_crown_fused_bwd(FusedSweepArgs a, cudaStream_t stream) {
  a.kmax = 0;
  int widest = 0;
  double flops = 0.0, bytes = 0.0;
  for (int l = 0; l < a.layers; ++l) {
    FusedSweepLayer& L = a.L[l];
    if (L.K > a.kmax) a.kmax = L.K;
    if (L.N > widest) widest = L.N;
    const bool last = l + 1 == a.layers;
    const FusedSweepLayer* below = last ? nullptr : &a.L[l + 1];
    const void* n_side[] = {L.W, L.out, last ? a.mid : below->dpos, last ? a.rad : below->dneg, last ? nullptr : below->add};
    L.vec = L.N % 4 == 0;
    for (const void* p : n_side) if (p && !al16(p)) L.vec = 0;
    const void* k_side[] = {l == 0 ? a.C : a.L[l - 1].out, L.kbias, L.dpos, L.dneg, L.epos, L.eneg, L.add};
    L.veck = L.K % 4 == 0;
    for (const void* p : k_side) if (p && !al16(p)) L.veck = 0;
    if (!last && !L.out) return BF_E_UNSUPPORTED;
    flops += 2.0 * (double)a.M * L.K * L.N;
    bytes += 4.0 * (double)a.M * L.K + (L.out ? 4.0 * (double)a.M * L.N : 0.0);
  }
  const size_t smem = fused_bwd_smem(a.kmax);
  if (smem > FUSED_SMEM) return BF_E_UNSUPPORTED;
  static SmemOptIn opt_in;
  static ClusterRoom room;
  if (int rc = ensure_dynamic_smem(crown_fused_bwd_kernel, FUSED_SMEM, opt_in, "crown_fused_bwd_kernel")) return rc;
  const int cs = fused_cluster(crown_fused_bwd_kernel, 256, smem, a.M, widest, room);
  if (cs == 0) return BF_E_UNSUPPORTED;
  timing_begin(T_BWD, stream);
  const int rc = fused_launch(crown_fused_bwd_kernel, a, 256, smem, cs, stream, "crown_fused_bwd_kernel");
  timing_end(T_BWD, stream, bytes, flops);
  return rc;
}

int launch_crown_fused_adjoint(FusedAdjointArgs a, cudaStream_t stream) {
  a.kmax = 4;
  int widest = 0;
  double flops = 0.0, bytes = 0.0;
  for (int l = 0; l < a.layers; ++l) {
    FusedAdjointLayer& L = a.L[l];
    if (l + 1 < a.layers && ((L.N + 3) & ~3) > a.kmax) a.kmax = (L.N + 3) & ~3;
    if (L.N > widest) widest = L.N;
    const void* k_side[] = {L.W, l == 0 ? a.A0 : nullptr, l == 0 ? a.mid : nullptr, l == 0 ? a.rad : nullptr};
    L.veck = L.K % 4 == 0;
    for (const void* p : k_side) if (p && !al16(p)) L.veck = 0;
    flops += 2.0 * (double)a.M * L.K * L.N;
    bytes += 4.0 * (double)a.M * (L.K + L.N);
  }
  const size_t smem = fused_adjoint_smem(a.kmax);
  if (smem > FUSED_SMEM) return BF_E_UNSUPPORTED;
  static SmemOptIn opt_in;
  static ClusterRoom room;
  if (int rc = ensure_dynamic_smem(crown_fused_adjoint_kernel, FUSED_SMEM, opt_in, "crown_fused_adjoint_kernel")) return rc;
  const int cs = fused_cluster(crown_fused_adjoint_kernel, FS_COMPUTE, smem, a.M, widest, room);
  if (cs == 0) return BF_E_UNSUPPORTED;
  timing_begin(T_ADJ, stream);
  const int rc = fused_launch(crown_fused_adjoint_kernel, a, FS_COMPUTE, smem, cs, stream, "crown_fused_adjoint_kernel");
  timing_end(T_ADJ, stream, bytes, flops);
  return rc;
}

}  // namespace bf
