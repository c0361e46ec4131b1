// CROWN backward through ReLU + Conv2d on the 5th-generation tensor cores: the ReLU scaling of coefficient rows
// (sign-selected slope, intercept and bias sums) and the transposed convolution in one pass over the rows.
//
// With u = h_in + padding = stride * q + phase and kernel row r = phase + stride * j, input row u receives output row q - j:
//   out[m, ci, phase, q] = sum_{j, co} Lam[m, co, q - j] * W[co, ci, phase + stride * j]        (the same for columns)
// so a row's coefficient plane, padded with zeros behind each line and behind the plane, becomes one line of positions per
// coefficient row, and every tap (jy, jx) is the same line read jy * Wp + jx positions earlier.  A GEMM tile is 128
// consecutive positions x all (phase, input channel) pairs of a block:
//   * A: the tile's positions and the halo in front of them are scaled, split and staged ONCE per 16 channels in the
//     unswizzled K-major layout, [part][8-channel chunk][position][16 bytes]; positions are 16 bytes apart, so a tap is a
//     descriptor whose start address lies that many positions earlier.  No im2col copy exists.
//   * B: the weights of all taps are split and stay in shared memory; the CTAs are persistent.
// An FP32 value is split into three bfloat16 parts of eight bits each, without a remainder: x = x0 + x1 + x2.  Of the nine
// products all but x1 y2, x2 y1 and x2 y2 are formed (narrow blocks: all nine); those three are below 2^-24 of x y together.
// Tensor-memory accumulators truncate: the error of a sum grows with its number of MMA steps (16 products each), in one
// direction, by half a unit in the last place of the running sum per step that adds anything.  So every tile has several
// accumulators for the leading products x0 y0, of at most CHUNK_STEPS steps where tensor memory has the room, and separate
// ones for the other products; the epilogue adds them in FP32.  A sum of few non-zero products truncates next to nothing: a
// row with one non-zero coefficient 1 gives the weights back exactly.
// Error against float64 (2-norm, random rows): 7e-8 and 1.3e-7 for the two layers below, the FP32 kernels' 2.0e-7 and 4.2e-7.
// 512 rows without a ReLU, 32 -> 32 channels, 16 x 16 -> 32 x 32, 4x4 / 2: 59 us (FP32 kernel 161); 64 -> 32 channels 16 x 16,
// 3x3: 71 us (143); with one 70 and 89 us (ReLU pass and FP32 kernel 170 and 153).  (Two TF32 parts a value, which leave a remainder,
// and twice as many steps: 63 and 91 us without a ReLU, 2.0e-7 and 4.9e-7.)  Bound by the instructions of its producers and of the
// read-back: issue slots 56 and 65 % busy at 31 % of the warps, tensor pipe 23 and 34 %, DRAM 11 and 6 %.
// Warps 0-10 stage A, 11-18 read the accumulators back, 19 issues the MMAs.  Every wait is bounded; on expiry the CTA
// writes NaN to all rows it owns and to their sums, so that no bound can be taken from them, and raises the status word.
#include <float.h>

#include "conv_tc.cuh"
#include "tc_primitives.cuh"

namespace bf {
namespace ctc {

using namespace tc;

constexpr int PROD_WARPS = 11, EPI_WARPS = 8, PRODUCERS = PROD_WARPS * 32;
constexpr int MMA_WARP = PROD_WARPS + EPI_WARPS, THREADS = (MMA_WARP + 1) * 32;
constexpr int TILE = 128;          // positions of a tile = MMA rows
constexpr int KC = 16;             // channels of a stage
constexpr int MAX_STAGES = 4;
constexpr int SMEM_LIMIT = 221 * 1024;  // dynamic; 5.6 KB of tables are static
constexpr int CHUNK_STEPS = 6;     // MMA steps (of 16 products each) summed in one accumulator, where tensor memory has the room
constexpr int PARTS = 3;           // bfloat16 parts of an FP32 value
constexpr int MAX_COLS = 512;
constexpr int MAX_NB = 128;
constexpr int MAX_CO = 512;

struct Control {
  unsigned long long a_full[MAX_STAGES], a_empty[MAX_STAGES], acc_full[2], acc_empty[2], sum_full[2], sum_empty[2], drain;
  uint32_t tmem_base;
  int abort_flag;
};

struct Div {  // n / d for n < 2^31 by one multiplication (round-up reciprocal: Granlund and Montgomery)
  uint32_t d, mul, sh;
  void set(uint32_t div) {
    d = div;
    sh = 0;
    while ((1ull << sh) < div) ++sh;
    mul = (uint32_t)(((1ull << (31 + sh)) + div - 1) / div);
  }
  __device__ __forceinline__ int operator()(int n) const { return (int)(((unsigned long long)(uint32_t)n * mul) >> (31 + sh)); }
};

struct Plan {  // everything the kernel derives from the geometry, computed on the host
  int JY, JX, Wp, P, halo, npos, pstr, groups;
  int cib, nblk, NB, merged, nchunk, bufs, units, cpad, stages, slots, tiles, pairs;
  Div dP, dWp, dS;   // positions per row, per line; rows per domain
  Div dNB, dChunks, dCib, dJX;
  int b_bytes, stage_bytes, smem;
};

struct Args {
  ConvTcProblem c;
  Plan p;
};

// x = x0 + x1 + x2 for two neighbouring channels (the differences are exact; each part holds the next eight bits)
__device__ __forceinline__ void split2(float a, float b, uint32_t (&p)[PARTS]) {
#pragma unroll
  for (int i = 0; i < PARTS; ++i) {
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(p[i]) : "f"(b), "f"(a));
    a -= __uint_as_float(p[i] << 16);
    b -= __uint_as_float(p[i] & 0xffff0000u);
  }
}
// stores the eight channels (16 bytes) of one position in the three images, `part` bytes apart
__device__ __forceinline__ void split_store(const float (&v)[8], unsigned char* at, size_t part) {
  uint32_t p[4][PARTS];
#pragma unroll
  for (int q = 0; q < 4; ++q) split2(v[2 * q], v[2 * q + 1], p[q]);
#pragma unroll
  for (int i = 0; i < PARTS; ++i) *reinterpret_cast<uint4*>(at + i * part) = make_uint4(p[0][i], p[1][i], p[2][i], p[3][i]);
}

// K-major without swizzle: 8-row x 16-byte core matrices, rows 16 bytes apart, row groups 128 bytes apart (SBO), 8-channel
// chunks `lbo` bytes apart
__device__ __forceinline__ uint64_t plain_desc(uint32_t saddr, uint32_t lbo) {
  return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(lbo >> 4) << 16) | (8ull << 32) | (1ull << 46);
}

__device__ __forceinline__ void tmem_ld_async(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
        "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr));
}
__device__ __forceinline__ void tmem_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }

// Bounded waits that sleep in the barrier unit: twenty warps polling as fast as they can take issue slots and
// shared-memory cycles from the one thread that issues the MMAs.
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

// One thread of a converged warp.  The compiler knows the predicate: it keeps descriptors in uniform registers, where
// behind `lane == 0` every tcgen05.mma costs a loop over the warp to find a uniform value (84 against 58 clocks per MMA in a
// bare loop over nine taps).
__device__ __forceinline__ bool elect_one() {
  uint32_t p;
  asm volatile("{\n\t.reg .pred q;\n\telect.sync _|q, 0xffffffff;\n\tselp.u32 %0, 1, 0, q;\n\t}" : "=r"(p));
  return p != 0;
}

// The MMAs of one tap and 16 channels as one sequence.  a, b: low words of the first descriptors (all share the high word),
// advanced by plain adds: a_part / b_part from one part's image to the next.
// MMAs on one accumulator are ordered among themselves only while they have one shape and one address.
// merged (the three parts' columns side by side): [D | D1 | D2] += a0 * [b0 | b1 | b2], [L0 | L1 | L2] += (a1, a2) * [b0 | b1 | b2]
__device__ __forceinline__ void mma_tap_merged(uint32_t d, uint32_t d_lo, uint32_t a, uint32_t b, uint32_t high, uint32_t a_part, uint32_t idesc,
                                               uint32_t accumulate, uint32_t accumulate_lo) {
  asm volatile(
      "{\n\t.reg .pred pacc, plo, pone;\n\t.reg .b32 u, v;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 pacc, %7, 0;\n\tsetp.ne.b32 plo, %8, 0;\n\tsetp.eq.b32 pone, %9, %9;\n\t"
      "add.u32 u, %2, %5;\n\tadd.u32 v, u, %5;\n\t"
      "mov.b64 da, {%2, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %6, {%9, %9, %9, %9}, pacc;\n\t"
      "mov.b64 da, {u, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %6, {%9, %9, %9, %9}, plo;\n\t"
      "mov.b64 da, {v, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %6, {%9, %9, %9, %9}, pone;\n\t}"
      ::"r"(d), "r"(d_lo), "r"(a), "r"(b), "r"(high), "r"(a_part), "r"(idesc), "r"(accumulate), "r"(accumulate_lo), "r"(0u)
      : "memory");
}
// D += a0 b0, D_lo += a0 b1 + a0 b2 + a1 b0 + a1 b1 + a2 b0, six MMAs
__device__ __forceinline__ void mma_tap(uint32_t d, uint32_t d_lo, uint32_t a, uint32_t b, uint32_t high, uint32_t a_part, uint32_t b_part,
                                        uint32_t idesc, uint32_t accumulate, uint32_t accumulate_lo) {
  asm volatile(
      "{\n\t.reg .pred pacc, plo, pone;\n\t.reg .b32 u, v, x, y;\n\t.reg .b64 da, db;\n\t"
      "setp.ne.b32 pacc, %8, 0;\n\tsetp.ne.b32 plo, %9, 0;\n\tsetp.eq.b32 pone, %10, %10;\n\t"
      "add.u32 u, %2, %5;\n\tadd.u32 v, u, %5;\n\tadd.u32 x, %3, %6;\n\tadd.u32 y, x, %6;\n\t"
      "mov.b64 da, {%2, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %7, {%10, %10, %10, %10}, pacc;\n\t"
      "mov.b64 db, {x, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, plo;\n\t"
      "mov.b64 db, {y, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, pone;\n\t"
      "mov.b64 da, {u, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, pone;\n\t"
      "mov.b64 db, {x, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, pone;\n\t"
      "mov.b64 da, {v, %4};\n\tmov.b64 db, {%3, %4};\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%1], da, db, %7, {%10, %10, %10, %10}, pone;\n\t}"
      ::"r"(d), "r"(d_lo), "r"(a), "r"(b), "r"(high), "r"(a_part), "r"(b_part), "r"(idesc), "r"(accumulate), "r"(accumulate_lo), "r"(0u)
      : "memory");
}

// predicated accesses: a branch per element costs more than the element
__device__ __forceinline__ float ldg_if(const float* p, bool ok) {
  float v;
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\tmov.f32 %0, 0f00000000;\n\t@p ld.global.nc.f32 %0, [%1];\n\t}"
               : "=f"(v) : "l"(p), "r"((uint32_t)ok));
  return v;
}
__device__ __forceinline__ void stg_if(float* p, float v, uint32_t ok) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.global.f32 [%0], %1;\n\t}" ::"l"(p), "f"(v), "r"(ok) : "memory");
}
__device__ __forceinline__ void stg2_if(float* p, float v, float w, uint32_t ok) {
  asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p st.global.v2.f32 [%0], {%1, %2};\n\t}" ::"l"(p), "f"(v), "f"(w), "r"(ok) : "memory");
}

// t (+)= W columns of N accumulators, added in order
constexpr int W = 16;
template <int N>
__device__ __forceinline__ void sum_accumulators(uint32_t at, const int* col, bool first, float (&t)[W]) {
  uint32_t r[N][W];
#pragma unroll
  for (int u = 0; u < N; ++u) tmem_ld_async(at + (uint32_t)col[u], r[u]);
  tmem_wait();
#pragma unroll
  for (int i = 0; i < W; ++i) {
    float v = first ? 0.f : t[i];
#pragma unroll
    for (int u = 0; u < N; ++u) v += __uint_as_float(r[u][i]);
    t[i] = v;
  }
}

// One output on the FP32 units, over the taps that exist.  Splitting an infinity leaves NaN (inf - inf), and a zero that only
// fills a tile (a tap past the kernel, a channel past Co) times an infinity is NaN too, so outputs that are not finite
// are formed again from the coefficients and weights they are made of.
__device__ __forceinline__ float scalar_output(const ConvTcProblem& c, long long at) {
  const int w = (int)(at % c.Wi), h = (int)(at / c.Wi % c.Hi), ci = (int)(at / ((long long)c.Wi * c.Hi) % c.Ci);
  const int m = (int)(at / ((long long)c.Wi * c.Hi * c.Ci)), plane = c.WH * c.WW;
  const float* a = c.A + (size_t)m * c.Co * plane;
  const size_t dom = (size_t)(m / c.S) * c.Co * plane;
  float t = 0.f;
  for (int r = 0; r < c.kh; ++r) {
    const int u = h + c.ph - r, y = u / c.sh;
    if (u < 0 || u % c.sh != 0 || y >= c.WH) continue;
    for (int s = 0; s < c.kw; ++s) {
      const int v = w + c.pw - s, x = v / c.sw;
      if (v < 0 || v % c.sw != 0 || x >= c.WW) continue;
      for (int co = 0; co < c.Co; ++co) {
        const int i = co * plane + y * c.WW + x;
        float lam = a[i];
        if (c.dpos) lam = lam * (lam >= 0.f ? c.dpos : c.dneg)[dom + i] + (c.add ? c.add[dom + i] : 0.f);
        t = fmaf(lam, c.W[((size_t)co * c.Ci + ci) * c.kh * c.kw + r * c.kw + s], t);
      }
    }
  }
  return t;
}

// Column groups g, g + 1, ... end - 1 (W columns each) of a warp's 32 positions: sums the accumulators and stores; the
// accumulators are handed back before the last group's stores.
__device__ __forceinline__ void read_and_store(uint32_t base, int g, int end, int naccs, const int* acc_col, const int2* col_tab,
                                               const ConvTcProblem& c, long long off, uint32_t ok, bool pairs, uint32_t empty_bar) {
  constexpr int N = 4;  // accumulators in flight
  float* out = c.out + off;
  for (; g < end; ++g) {
    float t[W];
    const uint32_t at = base + (uint32_t)(g * W);
    int x = 0;
    for (; x + N <= naccs; x += N) sum_accumulators<N>(at, acc_col + x, x == 0, t);
    for (; x + 2 <= naccs; x += 2) sum_accumulators<2>(at, acc_col + x, x == 0, t);
    if (x < naccs) sum_accumulators<1>(at, acc_col + x, x == 0, t);
    if (g + 1 == end) {
      tc_fence_before();
      __syncwarp();
      if ((threadIdx.x & 31) == 0) mbar_arrive(empty_bar);
    }
    const int4* tab = reinterpret_cast<const int4*>(col_tab + g * W);
    if (pairs) {
#pragma unroll
      for (int q = 0; q < W; q += 2) {
        const int4 ct = tab[q / 2];
        stg2_if(out + ct.x, t[q], t[q + 1], (ok >> ct.y) & 1u);
      }
    } else {
#pragma unroll
      for (int q = 0; q < W; q += 2) {
        const int4 ct = tab[q / 2];
        stg_if(out + ct.x, t[q], (ok >> ct.y) & 1u);
        stg_if(out + ct.z, t[q + 1], (ok >> ct.w) & 1u);
      }
    }
    bool finite = true;
#pragma unroll
    for (int i = 0; i < W; ++i) finite &= fabsf(t[i]) <= FLT_MAX;
    if (!finite) {
      for (int q = g * W; q < (g + 1) * W; ++q) {
        const int2 ct = col_tab[q];
        if (((ok >> ct.y) & 1u) && !(fabsf(out[ct.x]) <= FLT_MAX)) out[ct.x] = scalar_output(c, off + ct.x);
      }
    }
    __syncwarp();  // the next tensor-memory loads take the whole warp
  }
}

// Output side of position g: pointer offset of phase (0, 0) and one bit per phase that lands inside the image.
__device__ __forceinline__ uint32_t output_phases(const Args& a, int g, long long& off) {
  const ConvTcProblem& c = a.c;
  const Plan& p = a.p;
  const int m = p.dP(g);
  if (m >= c.M) return 0;
  const int rem = g - m * p.P, y = p.dWp(rem), x = rem - y * p.Wp;
  const int u0 = y * c.sh - c.ph, v0 = x * c.sw - c.pw;
  uint32_t ok = 0;
  for (int py = 0; py < c.sh; ++py)
    for (int px = 0; px < c.sw; ++px)
      if ((unsigned)(u0 + py) < (unsigned)c.Hi && (unsigned)(v0 + px) < (unsigned)c.Wi) ok |= 1u << (py * c.sw + px);
  off = (long long)m * c.Ci * c.Hi * c.Wi + u0 * c.Wi + v0;  // may lie in front of the row when only a later phase is inside
  return ok;
}

template <bool RELU>
__global__ void __launch_bounds__(THREADS, 1) conv_tc_kernel(const __grid_constant__ Args a) {
  extern __shared__ __align__(128) unsigned char smem[];
  const ConvTcProblem& c = a.c;
  const Plan& p = a.p;
  const int tid = threadIdx.x, warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = tid & 31;
  __shared__ Control ctl;
  __shared__ __align__(16) int2 col_tab[MAX_NB];   // per accumulator column (phase row, channel, phase column): output offset, phase (31: none)
  __shared__ float psum[2][2][TILE];               // [tile parity][channel group][position] row-sum contributions
  __shared__ float bias_s[MAX_CO];
  __shared__ int acc_col[MAX_COLS / 8];            // first column of every accumulator, the small products' before the others
  unsigned char* b_sm = smem + p.stages * p.stage_bytes;
  const int blk = blockIdx.x % p.nblk, ci0 = blk * p.cib;
  const int tile0 = blockIdx.x / p.nblk, tile_step = gridDim.x / p.nblk;
  const int phases = c.sh * c.sw, taps = p.JY * p.JX;
  volatile int* abort_flag = &ctl.abort_flag;

  if (tid == 0) {
    for (int s = 0; s < p.stages; ++s) {
      mbar_init(smem_u32(&ctl.a_full[s]), PROD_WARPS);
      mbar_init(smem_u32(&ctl.a_empty[s]), 1);
    }
    for (int s = 0; s < 2; ++s) {
      mbar_init(smem_u32(&ctl.acc_full[s]), 1);
      mbar_init(smem_u32(&ctl.acc_empty[s]), EPI_WARPS);
      mbar_init(smem_u32(&ctl.sum_full[s]), PROD_WARPS);
      mbar_init(smem_u32(&ctl.sum_empty[s]), EPI_WARPS);
    }
    mbar_init(smem_u32(&ctl.drain), 1);
    ctl.abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&ctl.tmem_base)), "r"(512u) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  // column n: phase row py, channel ci0 + i, phase column px
  auto column = [&](int n, int& py, int& i, int& px) {
    const int rest = n / c.sw;
    px = n - rest * c.sw;
    py = p.dCib(rest);
    i = rest - py * p.cib;
  };
  for (int n = tid; n < p.NB; n += THREADS) {
    int py, i, px;
    column(n, py, i, px);
    col_tab[n] = (py < c.sh && ci0 + i < c.Ci) ? make_int2((ci0 + i) * c.Hi * c.Wi + py * c.Wi + px, py * c.sw + px) : make_int2(0, 31);
  }
  if (tid < MAX_COLS / 8) {
    // merged: parts 2, 1 and 0 of the small products' accumulator, parts 2 and 1 of the others, then their leading products
    if (!p.merged) acc_col[tid] = (tid == 0) ? p.nchunk * p.NB : (tid - 1) * p.NB;
    else if (tid < PARTS) acc_col[tid] = (p.nchunk * PARTS + PARTS - 1 - tid) * p.NB;
    else if (tid < PARTS + 2 * p.nchunk) acc_col[tid] = ((tid - PARTS) / 2 * PARTS + 2 - (tid - PARTS) % 2) * p.NB;
    else acc_col[tid] = (tid - PARTS - 2 * p.nchunk) * PARTS * p.NB;
  }
  for (int co = tid; co < MAX_CO; co += THREADS) bias_s[co] = (c.bias && co < c.Co) ? c.bias[co] : 0.f;
  // B: [tap][part][8-channel chunk][column][8]   (merged: [tap][chunk][part][column][8])
  {
    const int chunks = p.cpad / 8, total = taps * chunks * p.NB;
    const size_t step = (size_t)c.Ci * c.kh * c.kw;
    for (int e = tid; e < total; e += THREADS) {
      const int tk = p.dNB(e), n = e - tk * p.NB, t = p.dChunks(tk), kc = tk - t * chunks, jy = p.dJX(t);
      int py, i, px;
      column(n, py, i, px);
      const int r = py + c.sh * jy, s = px + c.sw * (t - jy * p.JX);
      const bool in = py < c.sh && ci0 + i < c.Ci && r < c.kh && s < c.kw;
      const float* w = c.W + (in ? ((size_t)(kc * 8) * c.Ci + ci0 + i) * c.kh * c.kw + r * c.kw + s : 0);
      float v[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) v[q] = ldg_if(w + q * step, in && kc * 8 + q < c.Co);
      const size_t part = (size_t)(p.merged ? 1 : chunks) * p.NB * 16;
      split_store(v, b_sm + ((size_t)(p.merged ? tk * PARTS : t * PARTS * chunks + kc) * p.NB + n) * 16, part);
    }
  }
  fence_proxy_async();
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctl.tmem_base;
  const int kchunks = p.cpad / KC;  // stages per tile
  bool alive = true;

  if (warp < PROD_WARPS) {
    // ------------------------------------------------------------------ A producers: thread = position, eight channels at a time
    // Three items of a thread are in flight: coefficients of the next but one, slopes and intercepts (chosen by the
    // coefficients' signs) of the next, and the one being split and stored.  Loads are predicated, not branched around.
    const int pos = tid % p.pstr, grp = tid / p.pstr;
    const bool worker = grp < p.groups && pos < p.npos;
    const int per_tile = kchunks * (2 / p.groups);  // items of this thread per tile
    const int plane = c.WH * c.WW;
    const bool want_delta = c.partial != nullptr && blk == 0;
    const bool has_pos = c.epos != nullptr && want_delta, has_neg = c.eneg != nullptr && want_delta;

    // position of the item stream that loads coefficients
    int f_tile = tile0, f_item = 0;
    bool f_live = false;
    const float* f_a = c.A;
    size_t f_dom = 0;
    auto seek = [&]() {                             // decodes this thread's position in tile f_tile
      f_live = false;
      if (!worker || f_tile >= p.tiles) return;
      // the stage's first entry may lie (at most a halo, less than a row) in front of row 0
      const int idx = f_tile * TILE - p.halo + pos + p.P;
      const int row1 = p.dP(idx), row = row1 - 1;
      const int rem = idx - row1 * p.P, y = p.dWp(rem), x = rem - y * p.Wp;
      if (row < 0 || row >= c.M || y >= c.WH || x >= c.WW) return;
      const int d = p.dS(row);
      f_live = true;
      f_a = c.A + ((size_t)row * c.Co * plane + y * c.WW + x);
      f_dom = (size_t)d * c.Co * plane + y * c.WW + x;
    };
    auto channel = [&](int item) { return (p.groups == 2) ? item * KC + grp * 8 : item * 8; };

    float va[8];                                    // coefficients in flight
    bool a_live = false;
    size_t a_dom = 0;
    auto fetch = [&]() {                            // issues the loads of the next item
      const int ch = channel(f_item);
#pragma unroll
      for (int q = 0; q < 8; ++q) va[q] = ldg_if(f_a + (size_t)(ch + q) * plane, f_live && ch + q < c.Co);
      a_live = f_live;
      a_dom = f_dom + (size_t)ch * plane;
      if (++f_item == per_tile) {
        f_item = 0;
        f_tile += tile_step;
        seek();
      }
    };
    float vs[8], sl[8], ic[8];                      // coefficients with their slopes and intercepts in flight
    bool s_live = false;
    size_t s_dom = 0;
    auto select = [&](int ch) {                     // va has arrived: issues the loads that depend on its signs
      s_live = a_live;
      s_dom = a_dom;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const float x = va[q];
        vs[q] = x;
        if (RELU) {
          const bool sel = x >= 0.f, ok = a_live && ch + q < c.Co;
          sl[q] = ldg_if((sel ? c.dpos : c.dneg) + a_dom + (size_t)q * plane, ok);
          ic[q] = ldg_if((sel ? c.epos : c.eneg) + a_dom + (size_t)q * plane, ok && (sel ? has_pos : has_neg));
        }
      }
    };

    seek();
    fetch();
    select(channel(0));
    fetch();
    int s = 0, nt = 0;
    uint32_t phase = 1;
    for (int tile = tile0; tile < p.tiles && alive; tile += tile_step, ++nt) {
      float acc = 0.f;
      for (int item = 0; item < per_tile; ++item) {
        const int ch = channel(item);
        float lam[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) {
          const float x = vs[q];
          float l = x;
          if (RELU) {
            l = x * sl[q];
            acc = fmaf(x, ic[q], acc);
            if (c.add) l += ldg_if(c.add + s_dom + (size_t)q * plane, s_live && ch + q < c.Co);
          }
          if (want_delta) acc = fmaf(l, bias_s[ch + q], acc);
          lam[q] = l;
        }
        select(channel(item + 1 < per_tile ? item + 1 : 0));
        fetch();
        const bool opens = p.groups == 2 || (item & 1) == 0, closes = p.groups == 2 || (item & 1) == 1;
        if (opens && !wait_warp(smem_u32(&ctl.a_empty[s]), phase, abort_flag)) { alive = false; break; }
        if (worker) {
          split_store(lam, smem + s * p.stage_bytes + ((ch >> 3) & 1) * p.npos * 16 + pos * 16, (size_t)2 * p.npos * 16);
        }
        if (closes) {
          fence_proxy_async();
          __syncwarp();
          if (lane == 0) mbar_arrive(smem_u32(&ctl.a_full[s]));
          if (++s == p.stages) { s = 0; phase ^= 1u; }
        }
      }
      if (want_delta && alive) {  // this position's share of its row's sum goes to the epilogue warps
        const int sb = nt & 1;
        if (!wait_warp(smem_u32(&ctl.sum_empty[sb]), ((uint32_t)(nt >> 1) & 1u) ^ 1u, abort_flag)) { alive = false; break; }
        if (worker && pos >= p.halo) psum[sb][grp][pos - p.halo] = acc;
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl.sum_full[sb]));
      }
    }
  } else if (warp < MMA_WARP) {
    // ------------------------------------------------------------------ epilogue: thread = position, half of the column groups
    const int q = warp & 3, half = (warp - PROD_WARPS) >> 2;   // a warp may read the tensor-memory lanes of its index mod 4
    const int naccs = (p.merged ? PARTS : 1) * (p.nchunk + 1);
    const int groups = p.NB / W, from = half ? (groups + 1) / 2 : 0, to = half ? groups : (groups + 1) / 2;
    const uint32_t row = tmem + ((uint32_t)(q * 32) << 16);
    const bool want_delta = c.partial != nullptr && blk == 0;
    int it = 0;
    for (int tile = tile0; tile < p.tiles; tile += tile_step, ++it) {
      if (want_delta) {
        // row sums of the tile's positions, rows dealt to the warps; a row cut by tile edges has one slot per tile
        const int sb = it & 1;
        if (!wait_warp(smem_u32(&ctl.sum_full[sb]), (uint32_t)(it >> 1) & 1u, abort_flag)) break;
        const int lo = tile * TILE, hi = min(lo + TILE, c.M * p.P);
        const int r1 = p.dP(hi - 1);
        for (int r = p.dP(lo) + (warp - PROD_WARPS); r <= r1; r += EPI_WARPS) {
          const int first = r * p.P, last = first + p.P;
          const int from = max(first, lo) - lo, to = min(last, hi) - lo;
          float t = 0.f;
          for (int i = from + lane; i < to; i += 32) {
            t += psum[sb][0][i];
            if (p.groups == 2) t += psum[sb][1][i];
          }
#pragma unroll
          for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
          const int slot = tile - first / TILE, last_slot = (last - 1) / TILE - first / TILE;
          if (lane == 0) c.partial[(size_t)r * p.slots + slot] = t;
          if (slot == last_slot && lane > slot && lane < p.slots) c.partial[(size_t)r * p.slots + lane] = 0.f;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctl.sum_empty[sb]));
      }
      long long off = 0;
      const uint32_t ok = output_phases(a, tile * TILE + q * 32 + lane, off);
      const int buf = it % p.bufs;
      if (!wait_warp(smem_u32(&ctl.acc_full[buf]), (uint32_t)(it / p.bufs) & 1u, abort_flag)) break;
      tc_fence_after();
      const uint32_t base = row + (uint32_t)(buf * (MAX_COLS / 2));
      const uint32_t empty_bar = smem_u32(&ctl.acc_empty[buf]);
      read_and_store(base, from, to, naccs, acc_col, col_tab, c, off, ok, p.pairs, empty_bar);
      if (from >= to && lane == 0) mbar_arrive(empty_bar);
    }
  } else {
    // ------------------------------------------------------------------ MMA issue
    if (elect_one()) {
      const uint32_t n_mma = p.merged ? PARTS * p.NB : p.NB;
      // FP32 accumulators, bfloat16 operands
      const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((n_mma >> 3) << 17) | ((uint32_t)(TILE >> 4) << 24);
      const uint32_t a_lbo = (uint32_t)p.npos * 16, b_lbo = n_mma * 16;
      const int chunks = p.cpad / 8;
      // descriptor distances: from part to part, 16 channels, one tap's weights
      const uint32_t a_part = (2 * a_lbo) >> 4, b_k = (2 * b_lbo) >> 4;
      const uint32_t b_part = (uint32_t)(chunks * p.NB), b_tap = (uint32_t)(chunks * PARTS * p.NB);
      const uint64_t a_desc = plain_desc(smem_u32(smem) + (uint32_t)p.halo * 16, a_lbo), b_desc = plain_desc(smem_u32(b_sm), b_lbo);
      const uint32_t a_first = (uint32_t)a_desc, b_first = (uint32_t)b_desc, high = (uint32_t)(a_desc >> 32);
      const uint32_t a_stage = (uint32_t)(p.stage_bytes >> 4);
      const int per_chunk = (p.units + p.nchunk - 1) / p.nchunk;   // taps x 16 channels per accumulator
      int s = 0, tcount = 0;
      uint32_t phase = 0;
      for (int tile = tile0; tile < p.tiles && alive; tile += tile_step, ++tcount) {
        const int buf = tcount % p.bufs;
        if (!wait_asleep(smem_u32(&ctl.acc_empty[buf]), ((uint32_t)(tcount / p.bufs) & 1u) ^ 1u, abort_flag)) { alive = false; break; }
        tc_fence_after();
        uint32_t d = tmem + (uint32_t)(buf * (MAX_COLS / 2)) - n_mma;
        const uint32_t d_lo = tmem + (uint32_t)(buf * (MAX_COLS / 2)) + p.nchunk * n_mma;
        int left = 0;
        uint32_t started = 0;
        for (int kc = 0; kc < kchunks; ++kc) {
          if (!wait_asleep(smem_u32(&ctl.a_full[s]), phase, abort_flag)) { alive = false; break; }
          tc_fence_after();
          uint32_t ad = a_first + (uint32_t)s * a_stage, bd = b_first + (uint32_t)kc * b_k;
          int jx = 0;
          for (int t = 0; t < taps; ++t, bd += b_tap) {
            uint32_t acc = 1;
            if (left == 0) {
              d += n_mma;
              left = per_chunk;
              acc = 0;
            }
            --left;
            if (p.merged) mma_tap_merged(d, d_lo, ad, bd, high, a_part, idesc, acc, started);
            else mma_tap(d, d_lo, ad, bd, high, a_part, b_part, idesc, acc, started);
            started = 1;
            --ad;                                   // the next tap reads one position earlier, or one line
            if (++jx == p.JX) {
              jx = 0;
              ad -= (uint32_t)(p.Wp - p.JX);
            }
          }
          mma_commit(smem_u32(&ctl.a_empty[s]));
          if (++s == p.stages) { s = 0; phase ^= 1u; }
        }
        if (alive) mma_commit(smem_u32(&ctl.acc_full[buf]));
      }
      if (!alive) {  // MMAs in flight still read shared memory
        mma_commit(smem_u32(&ctl.drain));
        const long long t0 = clock64();
        while (!mbar_try_wait(smem_u32(&ctl.drain), 0) && clock64() - t0 < 200000000LL) {
        }
      }
    }
    __syncwarp();
  }

  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  if (ctl.abort_flag) {  // a wait ran out: no row of this CTA may pass as a result
    for (int tile = tile0; tile < p.tiles; tile += tile_step)
      for (int i = tid; i < TILE; i += THREADS) {
        long long off = 0;
        const uint32_t ok = output_phases(a, tile * TILE + i, off);
        for (int n = 0; n < p.NB; ++n) {
          const int2 ct = col_tab[n];
          if ((ok >> ct.y) & 1u) c.out[off + ct.x] = __int_as_float(0x7fffffff);
        }
      }
    if (c.partial != nullptr && blk == 0)
      for (int tile = tile0; tile < p.tiles; tile += tile_step) {
        const int lo = tile * TILE, hi = min(lo + TILE, c.M * p.P);
        for (int r = p.dP(lo) + tid; r <= p.dP(hi - 1); r += THREADS) c.partial[(size_t)r * p.slots + tile - r * p.P / TILE] = __int_as_float(0x7fffffff);
      }
    if (tid == 0 && c.status) atomicExch(c.status, 1);
  }
  if (warp == MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u) : "memory");
}

static bool make_plan(const ConvTcProblem& c, Plan& p) {
  if (c.Co > MAX_CO || c.sh * c.sw > 16 || c.ph < 0 || c.pw < 0) return false;  // a negative padding leaves input rows that no position stands for
  p.JY = ceil_div(c.kh, c.sh);
  p.JX = ceil_div(c.kw, c.sw);
  // lines and columns of positions: all outputs, and at least JY - 1 / JX - 1 zero ones behind the plane
  const int ny = (c.Hi - 1 + c.ph) / c.sh + 1, nx = (c.Wi - 1 + c.pw) / c.sw + 1;
  const int Hp = ny > c.WH + p.JY - 1 ? ny : c.WH + p.JY - 1;
  p.Wp = nx > c.WW + p.JX - 1 ? nx : c.WW + p.JX - 1;
  const long long P = (long long)Hp * p.Wp;
  const long long halo = (long long)(p.JY - 1) * p.Wp + p.JX - 1;
  if (halo > PRODUCERS - TILE || P > (1 << 24)) return false;
  p.halo = (int)halo;
  p.npos = TILE + p.halo;
  p.P = (int)P;
  const long long line = (long long)c.M * P;
  if (line > (1ll << 31) - (1 << 25)) return false;  // positions are 32-bit
  p.tiles = (int)((line + TILE - 1) / TILE);
  p.dP.set(p.P);
  p.dWp.set(p.Wp);
  p.dS.set(c.S);
  p.pstr = (p.npos <= PRODUCERS / 2) ? PRODUCERS / 2 : PRODUCERS;
  p.groups = PRODUCERS / p.pstr;
  p.slots = (int)((P - 1) / TILE + 2);
  if (p.slots > 32) return false;
  p.cpad = ceil_div(c.Co, KC) * KC;
  p.units = p.JY * p.JX * p.cpad / 16;  // MMA steps of a sum
  p.stage_bytes = ((PARTS * 2 * p.npos * 16) + 127) / 128 * 128;
  const int phases = c.sh * c.sw;
  // input channels per block: as many as the accumulator columns and shared memory hold (each block stages A again)
  for (p.nblk = 1; p.nblk <= 8; ++p.nblk) {
    p.cib = ceil_div(c.Ci, p.nblk);
    while ((phases * p.cib) % 16 != 0) ++p.cib;
    const int NB = phases * p.cib;
    p.merged = NB <= 32;   // narrow MMAs are bound by their issue: three wider ones instead of six
    p.NB = NB;
    if (NB > MAX_NB) continue;
    p.b_bytes = p.JY * p.JX * p.cpad * NB * 2 * PARTS;
    if (p.b_bytes + 2 * p.stage_bytes > SMEM_LIMIT) continue;
    p.stages = (SMEM_LIMIT - p.b_bytes) / p.stage_bytes;
    if (p.stages > MAX_STAGES) p.stages = MAX_STAGES;
    p.smem = p.b_bytes + p.stages * p.stage_bytes;
    // accumulators: as many as the steps ask for; two tiles in tensor memory when they fit side by side
    const int want = ceil_div(p.units, p.units / 2 < 1 ? 1 : (p.units / 2 < CHUNK_STEPS ? p.units / 2 : CHUNK_STEPS));
    const int one = p.merged ? PARTS * NB : NB;
    const int room = MAX_COLS / one - 1, room2 = MAX_COLS / 2 / one - 1;  // next to the small products'
    p.bufs = (want <= room2) ? 2 : 1;
    const int most = want < room ? want : room;
    p.nchunk = ceil_div(p.units, ceil_div(p.units, most));  // of equal length, all used
    p.pairs = c.sw == 2 && c.pw % 2 == 0 && c.Wi % 2 == 0 && (reinterpret_cast<uintptr_t>(c.out) & 7u) == 0;
    p.dNB.set(NB);
    p.dChunks.set(p.cpad / 8);
    p.dCib.set(p.cib);
    p.dJX.set(p.JX);
    return true;
  }
  return false;
}

}  // namespace ctc

bool conv_tc_supports(const ConvTcProblem& c, int* slots, int* tiles, double* us) {
  ctc::Plan p{};
  if (!ctc::make_plan(c, p)) return false;
  *slots = p.slots;
  *tiles = p.tiles;
  // launch and set-up, splitting the weights, and per tile of a CTA: hand-over, staging (two passes where the halo takes all
  // producers), read-back, MMAs.  Fitted to 3279 layers (1x1 to 7x7 kernels, 8 to 256 channels, 7 to 32 pixels, 160 to 2400
  // tiles): 7 % from the measured time in the 2-norm, 15 % at the 95th percentile.
  const int per = p.tiles < 148 / p.nblk ? p.tiles : 148 / p.nblk;
  const double split = 1.0 * p.JY * p.JX * p.cpad / 8 * p.NB / ctc::THREADS;
  const double stage = 1.25 * p.cpad / ctc::KC * (p.groups == 2 ? 1 : 2), read = 0.207 * p.NB / ctc::W;
  const double mma = p.units * ((p.merged ? 0.012 : 0.008) + 0.00133 * p.NB);
  *us = 14.2 + split + ceil_div(p.tiles, per) * (0.91 + stage + read + mma);
  return true;
}

int launch_conv_tc(const ConvTcProblem& c, cudaStream_t stream) {
  ctc::Args a{};
  a.c = c;
  BF_REQUIRE(ctc::make_plan(c, a.p), BF_E_UNSUPPORTED, "conv_tc: unsupported geometry");
  static SmemOptIn opt[2];
  const int per = a.p.tiles < 148 / a.p.nblk ? a.p.tiles : 148 / a.p.nblk;
  const int grid = per * a.p.nblk;
  if (c.dpos) {
    if (int rc = ensure_dynamic_smem(ctc::conv_tc_kernel<true>, ctc::SMEM_LIMIT, opt[0], "conv_tc_kernel")) return rc;
    ctc::conv_tc_kernel<true><<<grid, ctc::THREADS, a.p.smem, stream>>>(a);
  } else {
    if (int rc = ensure_dynamic_smem(ctc::conv_tc_kernel<false>, ctc::SMEM_LIMIT, opt[1], "conv_tc_kernel")) return rc;
    ctc::conv_tc_kernel<false><<<grid, ctc::THREADS, a.p.smem, stream>>>(a);
  }
  BF_CHECK_LAUNCH("conv_tc_kernel");
  g_tc_launches.fetch_add(1, std::memory_order_relaxed);
  return BF_OK;
}

}  // namespace bf
