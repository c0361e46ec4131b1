// Transposed convolution of narrow windows of coefficient rows (the identity-row sweeps on conv layers) and of small maps: square
// windows, kernels and strides, lanes = coefficient rows.
#include <math.h>

#include "common.cuh"
#include "kernels.cuh"

namespace bf {

// A row's window is WW x WW pixels of Co channels, its result OW x OW pixels (OW = (WW - 1) * ST + KS) of Ci channels.  Every
// row has the same geometry, so a warp takes 32 rows, a lane one of them: the window values are 16-byte words per lane, the
// weights are the same for the whole warp, and every tap that exists is a compile-time index, so no work is done for the zeros
// around a window (gathered from a padded tile, 3 x 3 -> 8 x 8 pixels of a 4x4 / 2 kernel is 256 multiply-adds per channel pair
// for 144 that exist).  A thread holds a band of TH image rows of TCI input channels (up to 72 sums, so that 16 warps share an SM):
// per output channel it reads its KS * KS * TCI weights once and its part of the window row by row, about one shared-memory word
// per six multiply-adds.  Window rows come in descending, kernel columns in ascending order: for each sum that is channel,
// kernel row, kernel column ascending, the order of conv_transpose_rowseg_kernel, whose bits it returns.
// Blocks stay: a block keeps the weights of its channel groups and walks tiles of 32 * R rows, whose windows come in chunks of
// cc output channels with 16-byte cp.async (4-byte copies took eight clocks of the SM for 128 bytes and bound the kernel), one
// chunk ahead.  Results leave through a 32 x 33 tile per warp, 128 bytes of a row at a time.
// Bound by instruction issue (slots 62 to 79 % busy with 12 to 16 warps an SM, FFMA pipe 46 to 67 %, shared memory 29 to 43 %): 15 to 23 of the
// 31 T multiply-adds/s that the chip reaches where a block's channels are many; with one to three channels the chunks' copies and the
// results' stores count too (DRAM 35 %).  65,536 rows, against the row-segment kernels: 32 -> 32 channels, 3 x 3 -> 8 x 8 of 4x4 / 2:
// 1291 -> 471 us; 64 -> 32, 4 x 4 -> 6 x 6 of 3x3: 3672 -> 838; 32 -> 32, 6 x 6 -> 14 x 14 of 4x4 / 2: 5486 -> 2514; 32 -> 3, 8 x 8 -> 10 x 10 of
// 3x3: 1124 -> 201; 32 -> 1, 4 x 4 -> 10 x 10 of 4x4 / 2: 221 -> 53.  Few rows: no slower (32 rows of 220 shapes: 0.1 to 1.0 of the time),
// except where rowseg_keeps (conv.cu) says so.
struct ConvWindowArgs {
  const float* Lam;  // [M, Co, WW, WW]
  const float* W;    // [Co, Ci, KS, KS]
  float* out;        // [M, Ci, OW, OW]
  int M, Co, Ci;
  int cgb;           // channel groups (of TCI) per block
  int R;             // groups of 32 rows per block
  int cc;            // output channels per chunk, a multiple of ConvWindow::CU
  int lprl;          // log2 of the lanes that copy one row's chunk
};

constexpr int CONV_WINDOW_SUMS = 72;

template <int KS, int ST, int PD, int WW>
struct ConvWindow {
  static constexpr int OW = (WW - 1) * ST + KS - 2 * PD;
  static constexpr int TH0 = (CONV_WINDOW_SUMS / OW) / ST * ST;                  // whole image rows that fit
  static constexpr bool FULL = OW * OW <= CONV_WINDOW_SUMS;
  static constexpr int NB0 = FULL ? 1 : (OW + TH0 - 1) / TH0;
  static constexpr int TH = FULL ? OW : ((OW + NB0 - 1) / NB0 + ST - 1) / ST * ST;
  static constexpr int NB = (OW + TH - 1) / TH;                                  // bands of TH image rows
  static constexpr int TCI = FULL ? (CONV_WINDOW_SUMS / (OW * OW) > 4 ? 4 : CONV_WINDOW_SUMS / (OW * OW)) : 1;
  static constexpr int CU = WW % 2 ? 4 : 1;                                      // channels whose windows end on 16 bytes
  static constexpr int WARPS = NB > 2 ? 12 : 8, BLOCKS = NB > 2 ? 1 : 2;         // three channels of four bands in one block
};

// One output channel (number U of CU) of a band: acc += window * weights.  lam: the channels' windows, in 16-byte words.
template <int KS, int ST, int PD, int WW, int TCI, int BAND, int U>
__device__ __forceinline__ void window_band(const float4* lam, const float* w, float (&acc)[TCI][ConvWindow<KS, ST, PD, WW>::TH][ConvWindow<KS, ST, PD, WW>::OW]) {
  using G = ConvWindow<KS, ST, PD, WW>;
  constexpr int H0 = BAND * G::TH;
  constexpr int HI = (H0 + G::TH - 1 + PD) / ST < WW - 1 ? (H0 + G::TH - 1 + PD) / ST : WW - 1;
  constexpr int LO = H0 + PD > KS - 1 ? (H0 + PD - KS + ST) / ST : 0;   // window rows LO to HI reach the band
  float l[G::CU * WW * WW + 4];
#pragma unroll
  for (int iy = HI; iy >= LO; --iy) {
    const int first = U * WW * WW + iy * WW, last = first + WW - 1;
#pragma unroll
    for (int k = first / 4; k <= last / 4; ++k) {
      if (iy < HI && k == (last + 1) / 4) continue;  // came with the row below
      const float4 t = lam[k];
      l[4 * k] = t.x; l[4 * k + 1] = t.y; l[4 * k + 2] = t.z; l[4 * k + 3] = t.w;
    }
#pragma unroll
    for (int r = 0; r < KS; ++r) {
      const int oy = iy * ST + r - PD - H0;
      if (oy < 0 || oy >= G::TH) continue;
#pragma unroll
      for (int s = 0; s < KS; ++s)
#pragma unroll
        for (int x = 0; x < WW; ++x) {
          const int ox = x * ST + s - PD;
          if (ox < 0 || ox >= G::OW) continue;
#pragma unroll
          for (int c = 0; c < TCI; ++c) acc[c][oy][ox] = fmaf(l[first + x], w[(r * KS + s) * TCI + c], acc[c][oy][ox]);
        }
    }
  }
}

template <int KS, int ST, int PD, int WW, int TCI, int BAND, int U>
__device__ __forceinline__ void window_channels(const float4* lam, const float4* wp, int w_step,
                                                float (&acc)[TCI][ConvWindow<KS, ST, PD, WW>::TH][ConvWindow<KS, ST, PD, WW>::OW]) {
  constexpr int NWP = (KS * KS * TCI + 3) / 4 * 4;
  float w[NWP];
#pragma unroll
  for (int k = 0; k < NWP / 4; ++k) {
    const float4 t = wp[k];
    w[4 * k] = t.x; w[4 * k + 1] = t.y; w[4 * k + 2] = t.z; w[4 * k + 3] = t.w;
  }
  window_band<KS, ST, PD, WW, TCI, BAND, U>(lam, w, acc);
  if constexpr (U + 1 < ConvWindow<KS, ST, PD, WW>::CU) window_channels<KS, ST, PD, WW, TCI, BAND, U + 1>(lam, wp + w_step, w_step, acc);
}

// ncc channels of a chunk for the warp's band
template <int KS, int ST, int PD, int WW, int TCI, int BAND>
__device__ __forceinline__ void window_chunk(int band, const float4* lam, const float4* wp, int w_step, int ncc,
                                             float (&acc)[TCI][ConvWindow<KS, ST, PD, WW>::TH][ConvWindow<KS, ST, PD, WW>::OW]) {
  using G = ConvWindow<KS, ST, PD, WW>;
  if (band == BAND) {
#pragma unroll 1
    for (int co = 0; co < ncc; co += G::CU, lam += G::CU * WW * WW / 4, wp += G::CU * w_step)
      window_channels<KS, ST, PD, WW, TCI, BAND, 0>(lam, wp, w_step, acc);
  } else if constexpr (BAND + 1 < G::NB) {
    window_chunk<KS, ST, PD, WW, TCI, BAND + 1>(band, lam, wp, w_step, ncc, acc);
  }
}

template <int KS, int ST, int PD, int WW, int TCI>
__global__ void __launch_bounds__(32 * ConvWindow<KS, ST, PD, WW>::WARPS, ConvWindow<KS, ST, PD, WW>::BLOCKS) conv_window_kernel(ConvWindowArgs a) {
  using G = ConvWindow<KS, ST, PD, WW>;
  constexpr int OW = G::OW, TH = G::TH, NB = G::NB, PLANE = WW * WW;
  constexpr int NW = KS * KS * TCI, NWP = (NW + 3) / 4 * 4;
  constexpr int N = TCI * TH * OW;
  static_assert(NB == 1 || (TCI == 1 && TH % ST == 0), "bands start at a window row");
  extern __shared__ __align__(16) float cw_smem[];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int combos = a.cgb * NB, rg = warp / combos, q = warp - rg * combos;
  const int cgl = q / NB, band = (q % NB + cgl + rg) % NB;        // bands of unequal work meet different schedulers
  const int pitch4 = (a.cc * PLANE / 4) | 1, buf4 = 32 * a.R * pitch4;
  float* wS = cw_smem;                                            // [Co][cgb][NWP]: kernel row, kernel column, channel
  float4* lamS = reinterpret_cast<float4*>(wS + a.Co * a.cgb * NWP);  // two buffers [32 * R][pitch4]
  float* epi = reinterpret_cast<float*>(lamS + 2 * buf4) + warp * (32 * 33);
  const int cg0 = blockIdx.y * a.cgb, ci0 = (cg0 + cgl) * TCI;

  for (int e = threadIdx.x; e < a.Co * a.cgb * NWP; e += blockDim.x) {
    const int k = e % NWP, g = e / NWP, co = g / a.cgb, ci = (cg0 + g - co * a.cgb) * TCI + k % TCI;
    wS[e] = (k < NW && ci < a.Ci) ? __ldg(a.W + ((size_t)co * a.Ci + ci) * (KS * KS) + k / TCI) : 0.f;
  }

  const int rows = 32 * a.R, nch = (a.Co + a.cc - 1) / a.cc;
  const size_t row4 = (size_t)a.Co * PLANE / 4;
  const int lpr = 1 << a.lprl, sub = threadIdx.x & (lpr - 1), row0 = threadIdx.x >> a.lprl, row_step = blockDim.x >> a.lprl;
  auto stage = [&](int buf, int m0, int co0) {
    const int n4 = min(a.cc, a.Co - co0) * PLANE / 4;
    const float4* base = reinterpret_cast<const float4*>(a.Lam) + co0 * PLANE / 4;
    for (int i = row0; i < rows; i += row_step) {
      const float4* src = base + (size_t)min(m0 + i, a.M - 1) * row4;
      const unsigned dst = (unsigned)__cvta_generic_to_shared(lamS + buf * buf4 + i * pitch4);
      for (int e = sub; e < n4; e += lpr) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + 16 * e), "l"(src + e) : "memory");
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  };

  const int tiles = (a.M + rows - 1) / rows;
  int tile = blockIdx.x, ch = 0, buf = 0;
  if (tile < tiles) stage(0, tile * rows, 0);
  float acc[TCI][TH][OW];
#pragma unroll
  for (int k = 0; k < N; ++k) acc[k / (TH * OW)][k / OW % TH][k % OW] = 0.f;
  while (tile < tiles) {
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    __syncthreads();                       // this chunk is there, and nobody reads the other buffer any more
    int next_tile = tile, next_ch = ch + 1;
    if (next_ch == nch) { next_ch = 0; next_tile += gridDim.x; }
    if (next_tile < tiles) stage(buf ^ 1, next_tile * rows, next_ch * a.cc);
    window_chunk<KS, ST, PD, WW, TCI, 0>(band, lamS + buf * buf4 + (rg * 32 + lane) * pitch4,
                                     reinterpret_cast<const float4*>(wS) + (ch * a.cc * a.cgb + cgl) * (NWP / 4), a.cgb * (NWP / 4),
                                     min(a.cc, a.Co - ch * a.cc), acc);
    if (next_ch == 0) {
      const int m0 = tile * rows + rg * 32, mrows = min(32, a.M - m0);
      const int h0 = band * TH;
      const int valid = G::FULL ? max(0, min(TCI, a.Ci - ci0)) * OW * OW : (ci0 < a.Ci ? min(TH, OW - h0) * OW : 0);
      const size_t m_step = (size_t)a.Ci * OW * OW;
      float* out = a.out + (size_t)m0 * m_step + ((size_t)ci0 * OW + h0) * OW + lane;
#pragma unroll
      for (int k0 = 0; k0 < N; k0 += 32) {
        __syncwarp();
#pragma unroll
        for (int j = 0; j < 32; ++j)
          if (k0 + j < N) epi[lane * 33 + j] = acc[(k0 + j) / (TH * OW)][(k0 + j) / OW % TH][(k0 + j) % OW];
        __syncwarp();
        if (k0 + lane < valid) {
#pragma unroll 8
          for (int i = 0; i < mrows; ++i) out[(size_t)i * m_step + k0] = epi[i * 33 + lane];
        }
      }
#pragma unroll
      for (int k = 0; k < N; ++k) acc[k / (TH * OW)][k / OW % TH][k % OW] = 0.f;
    }
    tile = next_tile;
    ch = next_ch;
    buf ^= 1;
  }
}

template <int KS, int ST, int PD, int WW, int TCI>
static int launch_window(ConvWindowArgs a, cudaStream_t stream) {
  using G = ConvWindow<KS, ST, PD, WW>;
  constexpr int NWP = (KS * KS * TCI + 3) / 4 * 4, LIMIT = (G::BLOCKS == 1 ? 224 : 112) * 1024, EPI = 32 * 33 * 4, PLANE = WW * WW;
  const int ncg = ceil_div(a.Ci, TCI);
  // Channel groups per block: few of them idle, few blocks that read the same rows (a tenth for each), and no idle warps where a block has an
  // SM.  Over 198 shapes (11 windows, 6 pairs of channels, 512 to 16,384 rows) the best other count is 5 % faster on average, more than 6 % on 46 of
  // them, 38 of these at 512 rows, where fewer groups in more blocks would take down to 0.68 of the time.
  double best = 0.0;
  int gy = 0;
  for (int c = G::WARPS / G::NB; c >= 1; --c) {
    if (c > ncg) continue;
    const int y = ceil_div(ncg, c);
    int r = G::WARPS / (c * G::NB);
    const double used = (double)ncg / (y * c) / (1.0 + 0.1 * y) * (G::BLOCKS == 1 ? sqrt((double)(c * G::NB * r) / G::WARPS) : 1.0);
    if (G::BLOCKS == 1) {
      // Row groups for the least rounds of blocks times a block's time, as its warps and a start that four more would take: 188 blocks of four
      // warps are two rounds on 148 SMs, 94 of eight one (4x4 / 2, padding 1, 8 -> 16 pixels, 16 -> 2 channels: 3000 rows 19.1 -> 15.4 us, 8192
      // rows 39.1 -> 28.6; row segments 17.8 and 38.1).
      const int gx = y < 148 ? 148 / y : 1;
      long long least = -1;
      for (int t = r; t >= 1; --t) {
        const long long time = (long long)ceil_div(ceil_div(a.M, 32 * t), gx) * (c * G::NB * t + 4);
        if (least < 0 || time < least) { least = time; r = t; }
      }
    } else {
      while (r > 1 && (long long)ceil_div(a.M, 32 * r) * y < 148) --r;    // few rows: more blocks with longer chunks
    }
    const long long left = LIMIT - (long long)a.Co * c * NWP * 4 - c * G::NB * r * EPI;
    const long long room = left / (2 * 32 * r * 16) - 1;                  // 16-byte words of a row's chunk
    if (room < G::CU * PLANE / 4 || used <= best + 1e-9) continue;
    // Chunks of up to 40 KB: 24 KB were one output channel of 10-pixel windows (3x3 / 1, 64 -> 32 channels, 64 rows: 85 us, 71 with 40 KB, row
    // segments 82).  Time of all shapes against 24 KB: 8 KB 1.10, 16 KB 1.02, 32 KB 0.96, 40 KB 0.95, 56 KB 0.96.
    long long cc = room * 4 / PLANE, want = 40 * 1024 / (32 * r * 4 * PLANE);
    if (want < G::CU) want = G::CU;
    if (cc > want) cc = want;
    if (cc > 16) cc = 16;
    if (cc > a.Co) cc = a.Co;
    best = used;
    a.cgb = c; a.R = r; a.cc = (int)cc / G::CU * G::CU; gy = y;
  }
  if (gy == 0 || gy > 65535) return BF_E_UNSUPPORTED;  // weights beyond an SM's shared memory
  const int threads = 32 * a.cgb * G::NB * a.R;
  a.lprl = 0;
  while (a.lprl < 5 && (1 << a.lprl) < a.cc * PLANE / 4) ++a.lprl;
  const size_t smem = (size_t)a.Co * a.cgb * NWP * 4 + 2 * (size_t)32 * a.R * ((a.cc * PLANE / 4) | 1) * 16 + threads / 32 * EPI;
  const int tiles = ceil_div(a.M, 32 * a.R);
  int gx = G::BLOCKS * 148 / gy;
  if (gx > tiles) gx = tiles;
  if (gx < 1) gx = 1;
  static SmemOptIn opt_in;
  if (int rc = ensure_dynamic_smem(conv_window_kernel<KS, ST, PD, WW, TCI>, LIMIT, opt_in, "conv_window_kernel")) return rc;
  conv_window_kernel<KS, ST, PD, WW, TCI><<<dim3(gx, gy), threads, smem, stream>>>(a);
  BF_CHECK_LAUNCH("conv_window_kernel");
  return BF_OK;
}

template <int KS, int ST, int PD, int WW, int MAXW>
static int launch_window_side(const ConvWindowArgs& a, int ww, cudaStream_t stream) {
  if constexpr (WW > MAXW) {
    return BF_E_UNSUPPORTED;
  } else {
    if (ww != WW) return launch_window_side<KS, ST, PD, WW + 1, MAXW>(a, ww, stream);
    if constexpr (WW % 2 == 0 || (PD == 0 && WW <= 7)) {
      constexpr int TCI = ConvWindow<KS, ST, PD, WW>::TCI;
      if (a.Co % ConvWindow<KS, ST, PD, WW>::CU != 0) return BF_E_UNSUPPORTED;
      // single channels where groups would be mostly padding (three channels in groups of four or two), and while the warps of single
      // channels are no more than the chip holds at once: TCI times the warps, each with 1 / TCI of the multiply-adds in series.
      // 3x3 / 1, 4 -> 6 pixels, groups and single channels (row segments): 64 -> 32 channels, 512 rows 44.5 and 25.4 us (42.3), 2048 rows 45.1
      // and 39.3, 4096 rows (twice the line) 71.5 and 69.8; 16 -> 16, 512 rows 14.0 and 9.0 (13.3), 8192 rows (twice the line) 22.5 and 23.3.
      if (TCI > 1 && (5 * (ceil_div(a.Ci, TCI) * TCI) > 6 * a.Ci || (long long)ceil_div(a.M, 32) * a.Ci <= 16 * 148))
        return launch_window<KS, ST, PD, WW, 1>(a, stream);
      return launch_window<KS, ST, PD, WW, TCI>(a, stream);
    }
    return BF_E_UNSUPPORTED;
  }
}

// Transposed convolution of M rows of WH x WW maps: windows (no padding), and full maps of 6 to 10 pixels under a 4x4 / 2 kernel with padding
// 1 and one or two channels below, from 2048 rows on (row segments -> here, us):
//   pixels, channels   2048 rows      8192 rows     25,600 rows
//    6, 16 -> 1 | 2    15 -> 11 | 15 -> 9     38 -> 12 | 45 -> 13     93 -> 35 | 130 -> 34
//    8, 16 -> 1 | 2    12 -> 11 | 13 -> 11    31 -> 16 | 38 -> 29     74 -> 45 | 112 -> 81
//   10, 16 -> 1 | 2    32 -> 19 | 36 -> 25    97 -> 50 | 132 -> 92    294 -> 124 | 401 -> 243
// Fewer rows are 0.83 to 1.02 of the row-segment kernel's speed, and larger maps stay there: their ten and more bands are as many copies
// of the loop in the instruction cache (16 -> 1 channels, 14 x 14: 333 us there, 419 here).
// BF_E_UNSUPPORTED for geometries without an instance.
int launch_conv_window(const float* Lam, const float* W, float* out, int M, int Ci, int Co, int WH, int WW, int kh, int kw, int sh, int sw,
                       int ph, int pw, cudaStream_t stream) {
  if (WH != WW || kh != kw || sh != sw || ph != pw || (reinterpret_cast<uintptr_t>(Lam) & 15u) != 0) return BF_E_UNSUPPORTED;
  const ConvWindowArgs a{Lam, W, out, M, Co, Ci, 0, 0, 0, 0};
  if (kh == 3 && sh == 1 && ph == 0) return launch_window_side<3, 1, 0, 2, 14>(a, WW, stream);
  if (kh == 4 && sh == 2 && ph == 0) return launch_window_side<4, 2, 0, 2, 7>(a, WW, stream);
  if (kh == 3 && sh == 2 && ph == 0) return launch_window_side<3, 2, 0, 2, 7>(a, WW, stream);
  if (kh == 4 && sh == 2 && ph == 1 && Ci <= 2 && M >= 2048) return launch_window_side<4, 2, 1, 6, 10>(a, WW, stream);
  return BF_E_UNSUPPORTED;
}

}  // namespace bf
