// Linear layers of small CROWN sweeps on the 5th-generation tensor cores: backward step (ReLU scaling, contraction, row sums,
// concretisation of the first layer) and adjoint step (contraction, next adjoint point, alpha / beta gradients) of sweeps whose
// coefficient rows are too few for the 128-row tiles of crown_tc.cu.
//
// Such a launch is a chain of latencies: operands, contraction, epilogue, next launch.  On FP32 units the contraction alone is 40 clocks a
// term (gemm_small.cuh: shared-memory reads).  Here a CTA owns 128 output features x 32 coefficient rows:
//   * features are the MMA's M side: weights are packed at the start of a call (pack_small_weights_kernel) as the shared-memory images that the MMA reads, per
//     (feature tile, 16 terms), and come by bulk copies, 32 terms (24 KB) a stage of a ring of seven;
//   * rows are its N side: sixteen warps load, scale and split them, and read the accumulators back afterwards.
// Where there are fewer tiles than SMs a cluster of two or four CTAs shares a tile: each takes a part of the terms, leaves its sums in shared memory
// and finishes a part of the features.
// An FP32 value is split into three bfloat16 parts without a remainder, x = x0 + x1 + x2; all nine
// products are formed, by four MMAs per 16 terms (an MMA takes max(N / 2, 32 + N / 4) clocks whatever the layout: it reads 4 KB of weights).
// Tensor-memory accumulators truncate: the error of a sum grows with its MMA steps, and always towards zero, so the leading
// products of every stage, of short sums of every step, have an accumulator of their own; they are added in FP32.
// Error against float64 (2-norm) of bounds and gradients of 3 to 6 layers of 64 to 800 inputs: 6.3e-8 to 9e-8 and 8e-8 to 2.1e-7 (FP32 kernels 9e-8 to
// 1e-7 and 4e-7 to 1.2e-6, TF32 kernels 1.8e-6 to 3.4e-6 and 8e-6 to 4e-4), and fewer signs of small coefficients on the wrong side.
// Layouts are K-major; weights without swizzle (8-row x 16-byte core matrices), [16 terms][part][8-term chunk][128 features][16 bytes], rows
// [part][32 rows][64 bytes] with the 64-byte swizzle: four lanes read 128 bytes of a row and a warp's stores meet different banks.
// From the end of one launch to the end of the next, FP32 kernels -> here: 1152 x 256 x 256 backward 12.5 -> 6.8 us, adjoint 9.3 -> 6.5; 1152 rows, 256 -> 784
// 28.4 -> 17.3; 784 -> 256 adjoint 28 -> 12.5; 333 x 512 x 512 20 -> 9.9 and 15 -> 7.8; 432 rows, 1568 -> 100 adjoint 39 -> 9.9.
// Of some 6.6 us (13 thousand clocks) 1.5 are the loads of the rows, 4 the MMAs (480 to 700 a stage: shared memory is busy with their operands), 2.5 the epilogue.
// Every wait is bounded; on expiry the status word is raised, whose reader replaces the call's results by NaN.
#include <float.h>

#include <algorithm>
#include <initializer_list>
#include <type_traits>

#include "kernels.cuh"
#include "tc_primitives.cuh"

namespace bf {
namespace stc {

using namespace tc;

constexpr int TF = 128;                     // output features of a CTA
constexpr int KS = 32;                      // terms of a stage
constexpr int NR = 32;                      // coefficient rows of a CTA
constexpr int W_STAGE = TF * KS * 3 * 2, STAGE = W_STAGE + NR * KS * 3 * 2;  // bytes: weights, and with the rows behind them
constexpr int WORKERS = 16, MMA_WARP = WORKERS, COPY_WARP = WORKERS + 1, THREADS = 32 * (WORKERS + 2);
constexpr int RING = 7;                     // stages in shared memory: 210 KB
constexpr int AHEAD = 2;                    // stages whose loads a thread has in flight

// Tensor memory of a CTA: accumulators of the leading products w0 r0 of every stage (GROUP stages are read back together, GROUPS groups by turns), one of
// w0 [r1 | r2] and one of w1 and w2 with [r0 | r1 | r2].
constexpr int GROUP = 5, GROUPS = 2, COL_E = GROUP * GROUPS * NR, COL_L = COL_E + 2 * NR;
static_assert(COL_L + 3 * NR <= 512, "tensor memory");
static_assert(RING > (GROUPS - 1) * GROUP, "a place of the ring is filled again behind the read-back of its stage's group");

struct Div {  // n / d for n < 2^31 by one multiplication (round-up reciprocal: Granlund and Montgomery)
  uint32_t mul, sh;
  void set(uint32_t d) {
    sh = 0;
    while ((1ull << sh) < d) ++sh;
    mul = (uint32_t)(((1ull << (31 + sh)) + d - 1) / d);
  }
  __device__ __forceinline__ int operator()(int n) const { return (int)(((unsigned long long)(uint32_t)n * mul) >> (31 + sh)); }
};

enum { RELU = 0, PLAIN = 1, BOX = 2 };      // what happens to a row on the way in: ReLU backward, nothing, mid - sign(a) * rad

struct Args {
  const float* A;                           // [M, K]
  const unsigned char* Wpk;
  const float* W;                           // the layer's weight [n_out, n_in]
  int M, N, K, S;
  Div dS;                                   // row -> domain
  int vec;                                  // 128-bit accesses along K are legal for every operand
  const float *dpos, *dneg, *epos, *eneg, *add, *kbias;  // RELU: [D, K], kbias [K]; dpos null: no ReLU
  const float *mid, *rad;                   // BOX: [D, K]
  int stages;                               // ring
  int* status;
  // backward
  float* delta;                             // [M] or null: row sums of a * intercept + lam * kbias
  int accumulate;
  float* out;                               // [M, N] or null
  const float *cmid, *crad;                 // [D, N], with `partial`
  float* partial;                           // [M, feature tiles] or null
  int side;
  // adjoint (see AdjEpilogue in crown_linear.cu)
  const float *nbias, *Ahat, *adpos, *adneg, *aepos, *aeneg, *pre_l, *pre_u, *gw;
  float *hout, *grad, *gsum;
};

struct Control {
  unsigned long long full[RING], summed[RING], drained[GROUPS], drain;
  uint32_t tmem_base;
  int abort_flag;
};

// The upper halves of two FP32 values, the first one's below: two bfloat16 values, cut off
__device__ __forceinline__ uint32_t upper_halves(float a, float b) { return __byte_perm(__float_as_uint(a), __float_as_uint(b), 0x7632); }
// x = x0 + x1 + x2: each part takes the next eight bits as they are (differences are exact), which is a third of the instructions of rounding
__device__ __forceinline__ void split2(float a, float b, uint32_t (&p)[3]) {
  p[0] = upper_halves(a, b);
  a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
  p[1] = upper_halves(a, b);
  a -= __uint_as_float(__float_as_uint(a) & 0xffff0000u);
  b -= __uint_as_float(__float_as_uint(b) & 0xffff0000u);
  p[2] = upper_halves(a, b);
}
__device__ __forceinline__ void split_store(const float (&v)[8], unsigned char* at, int part) {
  uint32_t p[4][3];
#pragma unroll
  for (int q = 0; q < 4; ++q) split2(v[2 * q], v[2 * q + 1], p[q]);
#pragma unroll
  for (int i = 0; i < 3; ++i) *reinterpret_cast<uint4*>(at + i * part) = make_uint4(p[0][i], p[1][i], p[2][i], p[3][i]);
}
__device__ __forceinline__ uint64_t plain_desc(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | (8ull << 32) | (1ull << 46);
}
// K-major, 64-byte swizzle: rows of 64 bytes (32 terms), groups of eight rows 512 bytes apart; 16 terms further are 32 bytes
__device__ __forceinline__ uint64_t rows_desc(uint32_t saddr) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | (1ull << 16) | (32ull << 32) | (1ull << 46) | (4ull << 61);
}
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}
// The MMAs of 16 terms.  w, r: low words of the descriptors, high, high_r: their high words; PART: from part to part of the weights.  The second MMA takes
// w0 from the collector, where the first has left it.
template <int PART>
__device__ __forceinline__ void mma_step(uint32_t d, uint32_t e, uint32_t l, uint32_t w, uint32_t r, uint32_t high, uint32_t high_r, uint32_t id1,
                                         uint32_t id2, uint32_t id3, uint32_t more_d, uint32_t more) {
  const uint32_t w1 = w + PART, w2 = w + 2 * PART, r1 = r + NR * 64 / 16;
  asm volatile(
      "{\n\t.reg .pred pd, pm, pone;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 pd, %8, 0;\n\tsetp.ne.b32 pm, %9, 0;\n\tsetp.eq.b32 pone, %10, %10;\n\t"
      "mov.b64 da, {%2, %6};\n\tmov.b64 db, {%5, %15};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16.collector::a::fill [%0], da, db, %11, {%10, %10, %10, %10}, pd;\n\t"
      "mov.b64 db, {%14, %15};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16.collector::a::lastuse [%13], da, db, %12, {%10, %10, %10, %10}, pm;\n\t"
      "mov.b64 da, {%3, %6};\n\tmov.b64 db, {%5, %15};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, pm;\n\t"
      "mov.b64 da, {%4, %6};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, pone;\n\t}"
      ::"r"(d), "r"(l), "r"(w), "r"(w1), "r"(w2), "r"(r), "r"(high), "r"(id3), "r"(more_d), "r"(more), "r"(0u), "r"(id1), "r"(id2), "r"(e), "r"(r1), "r"(high_r)
      : "memory");
}
// The MMA thread's wait.  The loop is hidden from the compiler: where the issuing loop depends on a value of this one thread, descriptors and
// addresses leave the uniform registers that the MMA reads, and a stage takes twice the time.
__device__ __forceinline__ uint32_t wait_spinning(uint32_t bar, uint32_t parity, uint32_t limit) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p, q;\n\t.reg .u32 i;\n\tmov.u32 i, 0;\n\t"
      "AGAIN:\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
      "@p bra DONE;\n\tadd.u32 i, i, 1;\n\tsetp.lt.u32 q, i, %3;\n\t@q bra AGAIN;\n\t"
      "DONE:\n\tselp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(limit)
      : "memory");
  return ok;
}
// Bounded waits that sleep in the barrier unit: sixteen warps polling as fast as they can take issue slots and shared-memory cycles from
// the thread that issues the MMAs.
__device__ __forceinline__ bool try_wait_asleep(uint32_t bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, 20000;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ bool wait_asleep(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  if (try_wait_asleep(bar, parity)) return true;
  const long long t0 = clock64();
  while (!try_wait_asleep(bar, parity)) {
    if (*abort_flag) return false;
    if (clock64() - t0 > WAIT_LIMIT) {
      *abort_flag = 1;
      return false;
    }
  }
  return true;
}
__device__ __forceinline__ bool wait_warp(uint32_t bar, uint32_t parity, volatile int* abort_flag) {
  int ok = 1;
  if ((threadIdx.x & 31) == 0) ok = wait_asleep(bar, parity, abort_flag) ? 1 : 0;
  ok = __shfl_sync(0xffffffffu, ok, 0);
  __syncwarp();  // what lane 0 has acquired is visible to the warp
  return ok != 0;
}
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
               : "r"(taddr));
}
// t += eight columns of each of the accumulators at the given columns, in order
template <int N>
__device__ __forceinline__ void add_columns(const uint32_t (&col)[N], float (&t)[8]) {
  uint32_t r[N][8];
#pragma unroll
  for (int u = 0; u < N; ++u) tmem_ld8_async(col[u], r[u]);
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
  for (int i = 0; i < 8; ++i)
#pragma unroll
    for (int u = 0; u < N; ++u) t[i] += __uint_as_float(r[u][i]);
}
__device__ __forceinline__ float ld_cluster(uint32_t addr) {
  float v;
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(addr) : "memory");
  return v;
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }
__device__ __forceinline__ void workers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * WORKERS) : "memory"); }

struct Eight {
  float v[8];
};
// Eight consecutive floats of a row of n, from k on.  VEC: n is a multiple of four and everything is aligned; what lies past the end is read from
// its last four elements, without a branch (behind guards, loads go out one after the other).  Otherwise zeros past the end.
template <bool VEC>
__device__ __forceinline__ Eight load8(const float* p, int k, int n) {
  if constexpr (VEC) {
    const float4 a = *reinterpret_cast<const float4*>(p + min(k, n - 4)), b = *reinterpret_cast<const float4*>(p + min(k + 4, n - 4));
    return Eight{{a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w}};
  } else {
    Eight e;
#pragma unroll
    for (int q = 0; q < 8; ++q) e.v[q] = k + q < n ? p[k + q] : 0.f;
    return e;
  }
}
__device__ __forceinline__ Eight zero8() { return Eight{{0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f}}; }

// what becomes of one element of a row
template <int PRO>
__device__ __forceinline__ float prologue(float a, float x, float y, float ad, bool relu) {
  if (PRO == RELU) return relu ? a * (a >= 0.f ? x : y) + ad : a;
  if (PRO == BOX) return x - tc::sgnf(a) * y;
  return a;
}

// One output on the FP32 units: splitting an infinity leaves NaN (inf - inf), so outputs that are not finite are formed again.
template <int MODE, int PRO>
__device__ __noinline__ float scalar_output(const Args& g, int m, int n) {
  const float* a = g.A + (size_t)m * g.K;
  const size_t dom = (size_t)(m / g.S) * g.K;
  const bool relu = PRO == RELU && g.dpos != nullptr;
  float t = 0.f;
  for (int k = 0; k < g.K; ++k) {
    float x = 0.f, y = 0.f, ad = 0.f;
    if (relu) {
      x = g.dpos[dom + k];
      y = g.dneg[dom + k];
      if (g.add) ad = g.add[dom + k];
    } else if (PRO == BOX) {
      x = g.mid[dom + k];
      y = g.rad[dom + k];
    }
    t = fmaf(prologue<PRO>(a[k], x, y, ad, relu), MODE == 0 ? g.W[(size_t)k * g.N + n] : g.W[(size_t)n * g.K + k], t);
  }
  return t;
}

// A cluster of CS CTAs shares one tile: each takes a part of the terms, leaves its sums in shared memory and finishes TF / CS features of all rows.
template <int MODE, int PRO, int CS>
__global__ void __launch_bounds__(THREADS, 1) crown_small_tc_kernel(const __grid_constant__ Args g) {
  extern __shared__ __align__(1024) unsigned char st_smem[];
  __shared__ Control ctl;
  constexpr int RGROUPS = NR / 8, SUBS = WORKERS / RGROUPS;  // a warp takes eight rows of every SUBS-th stage
  constexpr int FS = TF / CS;                      // features this CTA finishes
  __shared__ float row_part[SUBS][NR];             // row sums of the stages of a warp
  __shared__ float con_part[FS / 32][NR];          // concretisation sums of 32 features
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = tid & 31;
  const int rank = CS > 1 ? (int)cluster_ctarank() : 0, tile = blockIdx.x / CS, m0 = blockIdx.y * NR;
  const int all = (g.K + KS - 1) / KS, s_begin = rank * all / CS, nst = (rank + 1) * all / CS - s_begin, k_begin = s_begin * KS;
  const int steps = (g.K + 15) / 16 - 2 * s_begin;
  // Short sums have an accumulator of leading products per step
  const bool fine = 2 * nst <= GROUP * GROUPS;
  volatile int* abort_flag = &ctl.abort_flag;

  // Before the wait for the kernel in front: barriers, tensor memory, indices
  if (warp == COPY_WARP) {
    if (lane == 0) {
      for (int s = 0; s < g.stages; ++s) {
        mbar_init(smem_u32(&ctl.full[s]), RGROUPS + 1);
        mbar_init(smem_u32(&ctl.summed[s]), 1);
      }
      for (int b = 0; b < GROUPS; ++b) mbar_init(smem_u32(&ctl.drained[b]), WORKERS);
      mbar_init(smem_u32(&ctl.drain), 1);
      ctl.abort_flag = 0;
      asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
  } else if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // rows of this thread on the way in
  const int grp = warp % RGROUPS, sub = warp / RGROUPS, r8 = lane >> 2, chunk = lane & 3;
  const int row = m0 + grp * 8 + r8;
  const bool live = row < g.M, relu = PRO == RELU && g.dpos != nullptr;
  const float* pa = g.A + (size_t)(live ? row : 0) * g.K;
  const size_t dom = live ? (size_t)g.dS(row) * g.K : 0;
  const float* px = relu ? g.dpos + dom : (PRO == BOX ? g.mid + dom : nullptr);
  const float* py = relu ? g.dneg + dom : (PRO == BOX ? g.rad + dom : nullptr);
  const float* pz = (relu && g.add) ? g.add + dom : nullptr;
  unsigned char* to = st_smem + W_STAGE + (grp * 8 + r8) * 64 + ((chunk ^ (r8 >> 1)) << 4);
  // results of this thread: one feature, BR rows
  constexpr int BR = NR * FS / (32 * WORKERS);
  const int fl = tid % FS, ql = tid / FS * BR, n = tile * TF + rank * FS + fl, nc = min(n, g.N - 1);
  const bool n_ok = n < g.N;
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  grid_wait_after_setup();
  const uint32_t tmem = __shfl_sync(0xffffffffu, ctl.tmem_base, 0);  // in a uniform register: descriptors and addresses of the MMAs are

  constexpr int V = MODE == 0 ? 2 : 6;
  float dv[2][V], ah[BR], nb = 0.f;        // what the epilogue needs: of the two domains that BR rows can touch where S >= 8
  const bool few = g.S >= 8, wants = MODE == 1 || g.partial != nullptr;
  const int last_dom = g.dS(g.M - 1), first = m0 + ql, d0 = g.dS(first), rows = min(BR, g.M - first);
  const int split = few ? (d0 + 1) * g.S - first : 0;  // rows from here on belong to the next domain
  // an intercept that is not there is read from another table and counts as zero: no branch between the loads
  const float *aepos = g.aepos ? g.aepos : g.pre_l, *aeneg = g.aeneg ? g.aeneg : g.pre_l;
  auto load_domain = [&](int d, float (&v)[V]) {
    const size_t at = (size_t)min(d, last_dom) * g.N + nc;
    if (MODE == 0) {
      v[0] = g.cmid[at];
      v[1] = g.crad[at];
    } else {
      v[0] = g.adpos[at];
      v[1] = g.adneg[at];
      v[2 % V] = aepos[at];
      v[3 % V] = aeneg[at];
      v[4 % V] = g.pre_l[at];
      v[5 % V] = g.pre_u[at];
    }
  };
  float* red = reinterpret_cast<float*>(st_smem);   // [row][TF] sums of this CTA's terms: the ring is done with then
  float* gr = red + NR * TF;                        // [row][FS] contributions to the gradients of alpha, then those of beta

  if (warp < WORKERS) {
    // ------------------------------------------------------------------ rows
    const int quarter = warp & 3, r0 = (warp >> 2) * 8;   // 32 features and eight rows of the accumulators
    const uint32_t lanes = tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)r0;
    float t[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) t[i] = 0.f;
    bool alive = true;
    // Waits until the MMAs of stage s are complete.  One warp asks and the others are held by the barrier: MMAs this narrow take all cycles of shared memory,
    // and sixteen polling warps double their time.
    auto await_stage = [&](int s) {
      if (warp == 0) wait_warp(smem_u32(&ctl.summed[s % g.stages]), (uint32_t)(s / g.stages) & 1u, abort_flag);
      workers_sync();
      alive = alive && *abort_flag == 0;
      tc_fence_after();
    };
    // (Stage s + ring is not complete before everybody has seen stage s: its accumulators are those of a group behind that of s.)
    int next = 0;
    // adds the leading products of the groups of stages up to `last` to t
    auto drain = [&](int last) {
      for (; next <= last; ++next) {
        const int stages = min(fine ? nst : GROUP, nst - next * GROUP), accs = fine ? min(2 * nst, steps) : stages;
        await_stage(next * GROUP + stages - 1);
        const uint32_t at = lanes + (uint32_t)(next % GROUPS * GROUP * NR);
        int q = accs;
        for (; q >= 4; q -= 4)
          add_columns<4>({at + (uint32_t)((q - 1) * NR), at + (uint32_t)((q - 2) * NR), at + (uint32_t)((q - 3) * NR), at + (uint32_t)((q - 4) * NR)}, t);
        for (; q > 0; --q) add_columns<1>({at + (uint32_t)((q - 1) * NR)}, t);
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl.drained[next % GROUPS]));
      }
    };
    auto produce = [&](auto vector) {
      constexpr bool VEC = decltype(vector)::value;
      for (int b0 = 0; b0 < nst; b0 += AHEAD * SUBS) {
        const int k0 = k_begin + (b0 + sub) * KS + chunk * 8;
        Eight a[AHEAD], x[AHEAD], y[AHEAD], z[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) a[u] = load8<VEC>(pa, k0 + u * SUBS * KS, g.K);
        if (px) {
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) {
            x[u] = load8<VEC>(px, k0 + u * SUBS * KS, g.K);
            y[u] = load8<VEC>(py, k0 + u * SUBS * KS, g.K);
          }
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) z[u] = zero8();
        if (PRO == RELU && pz) {
#pragma unroll
          for (int u = 0; u < AHEAD; ++u) z[u] = load8<VEC>(pz, k0 + u * SUBS * KS, g.K);
        }
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const int s = b0 + sub + u * SUBS, slot = s % g.stages, k = k0 + u * SUBS * KS;
          // the ring's places of these SUBS stages are free again when the MMAs of the stages before them are complete; those wait for accumulators
          const int before = min(b0 + u * SUBS + SUBS, nst) - 1 - g.stages;
          if (before >= 0 && b0 + u * SUBS < nst) {
            drain(before / GROUP - GROUPS);
            await_stage(before);
          }
          if (s < nst && alive) {
            float v[8];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
              v[q] = prologue<PRO>(a[u].v[q], x[u].v[q], y[u].v[q], z[u].v[q], relu);
              if (!live || k + (VEC ? q / 4 * 4 : q) >= g.K) v[q] = 0.f;
            }
            split_store(v, to + slot * STAGE, NR * 64);
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(smem_u32(&ctl.full[slot]));
          }
        }
      }
    };
    if (g.vec) produce(std::true_type{});
    else produce(std::false_type{});
    if (MODE == 0 && g.delta && tile == 0) {
      // Row sums, from a second read of the rows (the first level of cache has them): the MMAs of the last stages are still at work.
      const float* pe = (relu && g.epos) ? g.epos + dom : nullptr;
      const float* pn = (relu && g.eneg) ? g.eneg + dom : nullptr;
      float r = 0.f;
      auto sums = [&](auto vector) {
        constexpr bool VEC = decltype(vector)::value;
        for (int s = sub; s < nst; s += SUBS) {
          const int k = k_begin + s * KS + chunk * 8;
          const Eight a = load8<VEC>(pa, k, g.K);
          Eight x = zero8(), y = x, z = x, e = x, f = x, b = x;
          if (px) {
            x = load8<VEC>(px, k, g.K);
            y = load8<VEC>(py, k, g.K);
          }
          if (PRO == RELU && pz) z = load8<VEC>(pz, k, g.K);
          if (pe) e = load8<VEC>(pe, k, g.K);
          if (pn) f = load8<VEC>(pn, k, g.K);
          if (g.kbias) b = load8<VEC>(g.kbias, k, g.K);
#pragma unroll
          for (int q = 0; q < 8; ++q) {
            if (k + (VEC ? q / 4 * 4 : q) < g.K) {
              if (relu) r += a.v[q] * (a.v[q] >= 0.f ? e.v[q] : f.v[q]);
              r = fmaf(prologue<PRO>(a.v[q], x.v[q], y.v[q], z.v[q], relu), b.v[q], r);
            }
          }
        }
      };
      if (g.vec) sums(std::true_type{});
      else sums(std::false_type{});
      r += __shfl_xor_sync(0xffffffffu, r, 1);
      r += __shfl_xor_sync(0xffffffffu, r, 2);
      if (chunk == 0) row_part[sub][grp * 8 + r8] = r;
    }
    // what the epilogue needs is loaded while the MMAs are at work
    if (MODE == 1 && g.nbias) nb = g.nbias[nc];
    if (wants && few) {
      load_domain(d0, dv[0]);
      load_domain(d0 + 1, dv[1]);
    }
    if (MODE == 1) {
#pragma unroll
      for (int i = 0; i < BR; ++i) ah[i] = g.Ahat[(size_t)min(first + i, g.M - 1) * g.N + nc];
    }
    drain(fine ? 0 : (nst - 1) / GROUP);
    add_columns<5>({lanes + COL_L + 2 * NR, lanes + COL_L + NR, lanes + COL_L, lanes + COL_E + NR, lanes + COL_E}, t);
#pragma unroll
    for (int i = 0; i < 8; ++i) red[(r0 + i) * TF + quarter * 32 + lane] = t[i];
  } else if (warp == MMA_WARP) {
    // ------------------------------------------------------------------ MMA issue
    if (elect_one()) {
      uint32_t limit = 1u << 24;
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(TF >> 4) << 24);
      const uint32_t id1 = idesc | ((uint32_t)(NR >> 3) << 17), id2 = idesc | ((uint32_t)(2 * NR >> 3) << 17), id3 = idesc | ((uint32_t)(3 * NR >> 3) << 17);
      const uint64_t wd = plain_desc(smem_u32(st_smem), TF * 16), rd = rows_desc(smem_u32(st_smem) + W_STAGE);
      const uint32_t high = (uint32_t)(wd >> 32), high_r = (uint32_t)(rd >> 32);
      constexpr int PART = (TF * 32) >> 4, W_STEP = 3 * PART, R_STEP = 32 >> 4;
      int slot = 0, place = 0, group = 0;    // ring; stage of the group; accumulators of the group
      uint32_t phase = 0, group_phase = 1, d = tmem;
      for (int s = 0; s < nst; ++s) {
        uint32_t ok = wait_spinning(smem_u32(&ctl.full[slot]), phase, limit);
        if (place == 0 && s >= GROUP * GROUPS) ok &= wait_spinning(smem_u32(&ctl.drained[group]), group_phase, limit);
        if (!ok) {  // the rest of the MMAs work on what is there; the results are not used
          limit = 1;
          *abort_flag = 1;
        }
        tc_fence_after();
        const uint32_t w = (uint32_t)wd + (uint32_t)(slot * (STAGE >> 4)), r = (uint32_t)rd + (uint32_t)(slot * (STAGE >> 4));
        mma_step<PART>(d, tmem + COL_E, tmem + COL_L, w, r, high, high_r, id1, id2, id3, 0u, s > 0);
        if (fine) d += NR;
        if (2 * s + 1 < steps) mma_step<PART>(d, tmem + COL_E, tmem + COL_L, w + W_STEP, r + R_STEP, high, high_r, id1, id2, id3, !fine, 1u);
        mma_commit(smem_u32(&ctl.summed[slot]));
        if (++slot == g.stages) {
          slot = 0;
          phase ^= 1u;
        }
        d += NR;
        if (++place == GROUP) {
          place = 0;
          if (++group == GROUPS) {
            group = 0;
            group_phase ^= 1u;
            d = tmem;
          }
        }
      }
      if (limit == 1) {  // MMAs in flight still read shared memory
        mma_commit(smem_u32(&ctl.drain));
        wait_spinning(smem_u32(&ctl.drain), 0, 1u << 20);
      }
    }
    __syncwarp();
  } else {
    // ------------------------------------------------------------------ weight copies
    if (lane == 0) {
      const unsigned char* src = g.Wpk + ((size_t)tile * all + s_begin) * W_STAGE;
      int copied = 0;
      for (; copied < nst; ++copied) {
        const int slot = copied % g.stages;
        if (copied >= g.stages && !wait_asleep(smem_u32(&ctl.summed[slot]), (uint32_t)(copied / g.stages - 1) & 1u, abort_flag)) break;
        mbar_arrive_expect_tx(smem_u32(&ctl.full[slot]), W_STAGE);
        bulk_copy_g2s(smem_u32(st_smem) + (uint32_t)(slot * STAGE), src + (size_t)copied * W_STAGE, W_STAGE, smem_u32(&ctl.full[slot]));
      }
      if (copied < nst) drain_bulk_copies(ctl.full, g.stages, copied);
    }
    __syncwarp();
  }
  // ------------------------------------------------------------------ results
  // The next launch is placed while these are written.  (Placed at the wait, with its weights' copies next to this launch's loads, a gradient evaluation of
  // five 256-wide layers, 128 inputs, takes 144.4 us instead of 141.5, two 512-wide ones, 60 inputs, 75.4 instead of 73.1, four, 37 inputs, 127.0 and 126.8.)
  grid_release();
  tc_fence_before();
  if (CS > 1) cluster_sync_all();
  else __syncthreads();
  tc_fence_after();
  float v[BR];
  if (warp < WORKERS) {
#pragma unroll
    for (int i = 0; i < BR; ++i) {
      const float* at = red + (ql + i) * TF + rank * FS + fl;
      v[i] = CS == 1 ? *at : ld_cluster(map_to_cta(smem_u32(at), 0));
#pragma unroll
      for (int r = 1; r < CS; ++r) v[i] += ld_cluster(map_to_cta(smem_u32(at), r));
    }
    if (MODE == 0 && g.delta && blockIdx.x == 0 && tid < NR && m0 + tid < g.M) {
      float r = 0.f;
      for (int q = 0; q < CS; ++q)
#pragma unroll
        for (int s = 0; s < SUBS; ++s) r += CS == 1 ? row_part[s][tid] : ld_cluster(map_to_cta(smem_u32(&row_part[s][tid]), q));
      g.delta[m0 + tid] = g.accumulate ? g.delta[m0 + tid] + r : r;
    }
  }
  if (CS > 1) cluster_arrive();  // the others' sums have been read
  if (warp < WORKERS) {
    bool finite = true;
#pragma unroll
    for (int i = 0; i < BR; ++i) finite &= fabsf(v[i]) <= FLT_MAX;
    if (!finite && n_ok) {
#pragma unroll
      for (int i = 0; i < BR; ++i)
        if (!(fabsf(v[i]) <= FLT_MAX) && i < rows) v[i] = scalar_output<MODE, PRO>(g, first + i, n);
    }
    __syncwarp();
    if (MODE == 0) {
      if (g.out && n_ok) {
        float* to_out = g.out + (size_t)first * g.N + n;
#pragma unroll
        for (int i = 0; i < BR; ++i)
          if (i < rows) to_out[(size_t)i * g.N] = v[i];
      }
      if (g.partial) {
        float p[BR];
        const float sgn = g.side == BF_SIDE_LOWER ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < BR; ++i) {
          if (!few) load_domain(g.dS(first + i), dv[1]);
          const float md = i < split ? dv[0][0] : dv[1][0], rd = i < split ? dv[0][1] : dv[1][1];
          p[i] = (n_ok && i < rows) ? v[i] * md + sgn * fabsf(v[i]) * rd : 0.f;
        }
        // sums over the 32 features of the warp: the lanes of row i end with its sum
        int mask = 16;
#pragma unroll
        for (int w = BR / 2; w >= 1; w /= 2, mask /= 2) {
          const bool up = lane & mask;
#pragma unroll
          for (int i = 0; i < w; ++i) p[i] = (up ? p[i + w] : p[i]) + __shfl_xor_sync(0xffffffffu, up ? p[i] : p[i + w], mask);
        }
#pragma unroll
        for (int w = 32 / BR / 2; w >= 1; w /= 2) p[0] += __shfl_xor_sync(0xffffffffu, p[0], w);
        if (lane % (32 / BR) == 0) con_part[fl >> 5][ql + lane / (32 / BR)] = p[0];
      }
    } else {
      float* to_h = g.hout ? g.hout + (size_t)first * g.N + n : nullptr;
      const float *gw = g.gw, *ep = g.aepos, *en = g.aeneg;
      auto element = [&](int i, float gg, float a, const float (&x)[V]) {
        const bool sel = a >= 0.f;
        if (to_h && n_ok && i < rows) to_h[(size_t)i * g.N] = (sel ? x[0] : x[1]) * gg + (sel ? (ep ? x[2 % V] : 0.f) : (en ? x[3 % V] : 0.f));
        gr[(ql + i) * FS + fl] = (sel && x[4 % V] < 0.f && x[5 % V] > 0.f) ? a * gg : 0.f;
        if (g.gsum) gr[(NR + ql + i) * FS + fl] = gw ? gg * gw[min(first + i, g.M - 1)] : gg;
      };
      if (few) {
#pragma unroll
        for (int i = 0; i < BR; ++i) {
          float x[V];
#pragma unroll
          for (int j = 0; j < V; ++j) x[j] = i < split ? dv[0][j] : dv[1][j];
          element(i, v[i] + nb, ah[i], x);
        }
      } else {
        // more than two domains in a block: by way of shared memory, a row at a time
#pragma unroll
        for (int i = 0; i < BR; ++i) gr[(ql + i) * FS + fl] = v[i] + nb;
#pragma unroll 1
        for (int i = 0; i < BR; ++i) {
          float x[V];
          load_domain(g.dS(first + i), x);
          element(i, gr[(ql + i) * FS + fl], g.Ahat[(size_t)min(first + i, g.M - 1) * g.N + nc], x);
        }
      }
    }
    workers_sync();
    if (MODE == 0) {
      if (g.partial && tid < NR && m0 + tid < g.M) {
        float p = con_part[0][tid];
#pragma unroll
        for (int q = 1; q < FS / 32; ++q) p += con_part[q][tid];
        g.partial[(size_t)(m0 + tid) * gridDim.x + blockIdx.x] = p;
      }
    } else {
      // sums over the rows of every domain that fall into this tile; at most two tiles add to an entry (S <= NR)
      const int m_end = min(m0 + NR, g.M), d_first = g.dS(m0), d_last = g.dS(m_end - 1);
      for (int d = d_first + tid / FS; d <= d_last; d += 32 * WORKERS / FS) {
        const int lo = max(d * g.S, m0) - m0, hi = min((d + 1) * g.S, m_end) - m0;
        float s = 0.f, s2 = 0.f;
#pragma unroll 4
        for (int r = lo; r < hi; ++r) s += gr[r * FS + fl];
        if (n_ok) atomicAdd(g.grad + (size_t)d * g.N + n, s);
        if (g.gsum) {
#pragma unroll 4
          for (int r = lo; r < hi; ++r) s2 += gr[(NR + r) * FS + fl];
          if (n_ok) atomicAdd(g.gsum + (size_t)d * g.N + n, s2);
        }
      }
    }
  }
  if (tid == 0 && ctl.abort_flag && g.status) atomicExch(g.status, 1);
  if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
  if (CS > 1) cluster_wait();
}

// Images of up to PACK_JOBS weights in one launch: a block takes 256 (feature, eight terms) items of a job.  The blocks behind those form the input set and
// the negated spec rows of a query (a launch of its own in front of it cost 784-100-100-10, 64 inputs, 3.8 us of 61).
constexpr int PACK_JOBS = 16;
struct PackJob {
  const float* W;
  unsigned char* out;
  int ldw, transposed, vec, N, K, nst, first_block;  // vec: 128-bit loads along a row of W are legal
};
struct PackJobs {
  PackJob job[PACK_JOBS];
  int count;
};
struct QueryStart {
  const float *a, *b, *C;
  float *mid, *rad, *C2;
  float eps;
  long long n, per, total;
  int set_blocks;  // blocks for the input set; the rest of the grid is for the spec rows
};
__device__ __forceinline__ void query_start_block(const QueryStart& q, int block, int blocks) {
  if (block >= q.set_blocks) {  // C2[b] = (C[b], -C[b])
    for (long long i = (block - q.set_blocks) * 256ll + threadIdx.x; i < q.total; i += (blocks - q.set_blocks) * 256ll) {
      const long long o = i + i / q.per * q.per;
      const float c = q.C[i];
      q.C2[o] = c;
      q.C2[o + q.per] = -c;
    }
    return;
  }
  for (long long i = block * 256ll + threadIdx.x; i < q.n; i += q.set_blocks * 256ll) {
    if (q.b) {
      const float lo = q.a[i], up = q.b[i];
      q.mid[i] = (lo + up) / 2.f;
      q.rad[i] = (up - lo) / 2.f;
    } else {
      q.rad[i] = q.eps;
    }
  }
}
__global__ void __launch_bounds__(256) pack_small_weights_kernel(const __grid_constant__ PackJobs jobs, int pack_blocks, const __grid_constant__ QueryStart q) {
  if ((int)blockIdx.x >= pack_blocks) {
    query_start_block(q, (int)blockIdx.x - pack_blocks, (int)gridDim.x - pack_blocks);
    return;
  }
  int j = 0;
  while (j + 1 < jobs.count && (int)blockIdx.x >= jobs.job[j + 1].first_block) ++j;
  const PackJob& p = jobs.job[j];
  const long long i = (long long)((int)blockIdx.x - p.first_block) * 256 + threadIdx.x;  // chunks of a tile are whole blocks: 4 * nst * 128 items
  const int f = (int)(i % TF), chunk = (int)(i / TF % (p.nst * 4)), tile = (int)(i / TF / (p.nst * 4));
  const int n = tile * TF + f;
  float v[8];
  if (!p.transposed && p.vec && n < p.N && chunk * 8 + 8 <= p.K) {
    const float4* w = reinterpret_cast<const float4*>(p.W + (size_t)n * p.ldw + chunk * 8);
    const float4 a = w[0], b = w[1];
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
    v[4] = b.x; v[5] = b.y; v[6] = b.z; v[7] = b.w;
  } else
#pragma unroll
  for (int q = 0; q < 8; ++q) {
    const int k = chunk * 8 + q;
    v[q] = (n < p.N && k < p.K) ? (p.transposed ? p.W[(size_t)k * p.ldw + n] : p.W[(size_t)n * p.ldw + k]) : 0.f;
  }
  split_store(v, p.out + ((size_t)tile * p.nst * 2 + chunk / 2) * (3 * TF * 32) + (size_t)((chunk & 1) * TF + f) * 16, TF * 32);
}

}  // namespace stc

// CTAs that share the terms of a tile; 0: the problem is not small.
// Gradient evaluations (one sweep down, one up, images packed) of 784-input networks, other kernels -> here, us: three 256-wide layers, 300 inputs (gradient
// sweep only, see few_rows_call) 241 -> 187, 500 inputs 245 -> 195, three 128-wide ones, 1000 inputs 201 -> 162; three tiles an SM 256-wide, 530 inputs
// 227 -> 209, 785 inputs 243 -> 232, five such layers 359 -> 313 and 369 -> 344, 512-wide, 300 inputs 366 -> 283, two 800-wide, 200 inputs 306 -> 250, but
// (without the packing) 128-wide, 1200 inputs 203 -> 210 and 100-wide 204 -> 208; four an SM 256-wide, 900 inputs 250 -> 271.
// Sums of up to 64 terms are short on the FP32 units, too: three 33-, 48- and 64-wide layers, 1 to 128 inputs 50 to 69 there and, without the packing, 52 to 72 here.
// Clusters while all CTAs find an SM: four 512-wide layers, 37 inputs 150 us with one CTA a tile, 121 with two, 784-100-100-10, 64 inputs 63 and 56.  Four CTAs
// share sums above 1024 terms (1568-1568-100-10, 48 inputs: 199 with one CTA a tile, 182).  Shorter sums would mostly gain from four, too (one, two, four: 500-wide,
// 9 inputs 118, 89, 77 us, five 256-wide layers, 20 inputs 134, 115, 107, two 784-wide, 16 inputs 107, 77, 87; errors alike), but tests follow loops of a
// 784-input network step by step, two of whose steps have objectives that are equal up to rounding, and with four such a loop keeps another step.
static int small_tc_cluster(int M, int N, int K) {
  const long long tiles = (long long)ceil_div(N, stc::TF) * ceil_div(M, stc::NR);
  if (K <= 64 || tiles > (K >= 256 ? 3 : 2) * 148) return 0;
  int cs = K > 1024 ? 4 : (K > 96 ? 2 : 1);
  while (tiles * cs > 148 && cs > 1) cs /= 2;
  return cs;
}

bool small_tc_supports(int M, int N, int K, int S, bool adjoint) { return small_tc_cluster(M, N, K) > 0 && (!adjoint || S <= stc::NR); }
int small_tc_tiles(int M, int N, int K) { return ceil_div(N, stc::TF) * small_tc_cluster(M, N, K); }
int small_tc_max_tiles(int N) { return ceil_div(N, stc::TF) * 4; }
size_t small_tc_packed_bytes(int N, int K) { return (size_t)ceil_div(N, stc::TF) * ceil_div(K, stc::KS) * stc::W_STAGE; }

static int pack_images(const SmallPack* packs, int count, const stc::QueryStart* start, int start_blocks, cudaStream_t stream) {
  int first = 0;
  do {
    stc::PackJobs jobs{};
    int blocks = 0;
    for (; first < count && jobs.count < stc::PACK_JOBS; ++first) {
      const SmallPack& p = packs[first];
      const int N = p.transposed ? p.cols : p.rows, K = p.transposed ? p.rows : p.cols, nst = ceil_div(K, stc::KS);
      jobs.job[jobs.count++] = {p.W, p.out, p.cols, p.transposed, p.cols % 4 == 0 && (reinterpret_cast<uintptr_t>(p.W) & 15u) == 0, N, K, nst, blocks};
      blocks += ceil_div(N, stc::TF) * nst * 4 * stc::TF / 256;
    }
    stc::pack_small_weights_kernel<<<blocks + start_blocks, 256, 0, stream>>>(jobs, blocks, start ? *start : stc::QueryStart{});
    BF_CHECK_LAUNCH("pack_small_weights_kernel");
    start_blocks = 0;
  } while (first < count);
  return BF_OK;
}
int launch_query_start(const float* a, const float* b, float eps, float* mid, float* rad, long long n, const float* C, float* C2, long long per, int B,
                       const SmallPack* packs, int count, cudaStream_t stream) {
  auto blocks = [](long long items) { return (int)std::min((items + 255) / 256, 148ll * 16); };
  const stc::QueryStart q{a, b, C, mid, rad, C2, eps, n, per, B * per, blocks(n)};
  return pack_images(packs, count, &q, q.set_blocks + (C2 ? blocks(q.total) : 0), stream);
}

int small_tc_pack(const SmallPack* packs, int count, cudaStream_t stream) { return count ? pack_images(packs, count, nullptr, 0, stream) : BF_OK; }
template <int MODE, int PRO, int CS>
static int launch_small_n(stc::Args g, cudaStream_t stream) {
  g.dS.set((uint32_t)g.S);
  g.stages = std::min(ceil_div(ceil_div(g.K, stc::KS), CS), stc::RING);
  const int smem = std::max(std::max(g.stages * stc::STAGE, stc::NR * (stc::TF + 2 * stc::TF / CS) * 4), ONE_PER_SM);
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(stc::crown_small_tc_kernel<MODE, PRO, CS>, stc::RING * stc::STAGE, opt_in, "crown_small_tc_kernel")) return rc;
  const dim3 grid(ceil_div(g.N, stc::TF) * CS, ceil_div(g.M, stc::NR));
  launch_after_setup(stc::crown_small_tc_kernel<MODE, PRO, CS>, grid, stc::THREADS, smem, CS, stream, g);
  BF_CHECK_LAUNCH("crown_small_tc_kernel");
  g_tc_launches.fetch_add(1, std::memory_order_relaxed);
  return BF_OK;
}
template <int MODE, int PRO>
static int launch_small(const stc::Args& g, cudaStream_t stream) {
  switch (small_tc_cluster(g.M, g.N, g.K)) {
    case 4: return launch_small_n<MODE, PRO, 4>(g, stream);
    case 2: return launch_small_n<MODE, PRO, 2>(g, stream);
    default: return launch_small_n<MODE, PRO, 1>(g, stream);
  }
}

static int all_aligned(std::initializer_list<const void*> ptrs) {
  for (const void* p : ptrs)
    if (reinterpret_cast<uintptr_t>(p) & 15u) return 0;
  return 1;
}

int launch_crown_bwd_small_tc(const float* A, const float* dpos, const float* dneg, const float* epos, const float* eneg, const float* add,
                              const unsigned char* Wpk, const float* W, const float* kbias, float* A_prev, float* delta, int accumulate, const float* mid,
                              const float* rad, float* partial, int side, int M, int S, int K, int N, int* status, cudaStream_t stream) {
  stc::Args g{};
  g.A = A; g.Wpk = Wpk; g.W = W; g.M = M; g.N = N; g.K = K; g.S = S;
  g.vec = K % 4 == 0 && all_aligned({A, dpos, dneg, epos, eneg, add, kbias});
  g.dpos = dpos; g.dneg = dneg; g.epos = epos; g.eneg = eneg; g.add = add; g.kbias = kbias;
  g.delta = delta; g.accumulate = accumulate; g.out = A_prev; g.cmid = mid; g.crad = rad; g.partial = partial; g.side = side;
  g.status = status;
  timing_begin(T_BWD, stream);
  const int rc = launch_small<0, stc::RELU>(g, stream);
  timing_end(T_BWD, stream, 4.0 * (double)M * K + (A_prev ? 4.0 * (double)M * N : 0.0), 2.0 * (double)M * K * N);
  return rc;
}

int launch_crown_adjoint_small_tc(const float* Hprev, int first_layer, const float* mid, const float* rad, const unsigned char* Wpk, const float* W,
                                  const float* nbias, const float* Ahat, const float* dpos, const float* dneg, const float* epos, const float* eneg,
                                  const float* pre_l, const float* pre_u, float* hout, float* grad, float* gsum, int M, int S, int K, int N, int* status,
                                  cudaStream_t stream, const float* gw) {
  stc::Args g{};
  g.A = Hprev; g.Wpk = Wpk; g.W = W; g.M = M; g.N = N; g.K = K; g.S = S;
  g.mid = mid; g.rad = rad;
  g.vec = K % 4 == 0 && all_aligned({Hprev, mid, rad});
  g.nbias = nbias; g.Ahat = Ahat; g.adpos = dpos; g.adneg = dneg; g.aepos = epos; g.aeneg = eneg; g.pre_l = pre_l; g.pre_u = pre_u;
  g.gw = gw; g.hout = hout; g.grad = grad; g.gsum = gsum; g.status = status;
  timing_begin(T_ADJ, stream);
  const int rc = first_layer ? launch_small<1, stc::BOX>(g, stream) : launch_small<1, stc::PLAIN>(g, stream);
  timing_end(T_ADJ, stream, 4.0 * (double)M * K + 8.0 * (double)M * N, 2.0 * (double)M * K * N);
  return rc;
}

}  // namespace bf
