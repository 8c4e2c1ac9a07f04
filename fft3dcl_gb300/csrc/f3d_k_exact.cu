// f3d_k_exact.cu -- exact-form kernels: the reference's radix-2 transforms in
// its own operation order, no fused multiply-add, so the engine's output has
// the same bits as the reference CPU backend.
//
// Compiled once per block width (-DF3D_BW=4|8|16|32|64) with --fmad=false;
// each object holds the kernels for every block height of that width.
//
// Thread mapping: TPB = max(bw, bh) threads own one block. The forward
// transform gives one thread per block row (row FFT held in registers), then
// one thread per kept column; the inverse one thread per column (Hermitian
// completion on the fly), then one thread per row. Shared memory carries the
// transposes; a CTA of 128 threads works on 128/TPB blocks.
// 64 x 64 blocks run their 64-point transforms on lane pairs and groups of four
// instead (k_forward_exact64, 128 threads per block; k_inverse_lanes, 256), the
// inverse of 32 x 32 blocks on pairs (k_inverse_lanes, 64).
#include "f3d_device.cuh"

#ifndef F3D_BW
#error "F3D_BW must be defined"
#endif

namespace f3d {
namespace {

template <int BW, int BH>
struct Cfg {
  static constexpr int FBW = BW / 2 + 1;
  static constexpr int PS = FBW * BH;                 // bins per block
  static constexpr int TPB = BW > BH ? BW : BH;       // threads per block
  static constexpr int THREADS = TPB > 128 ? TPB : 128;
  static constexpr int BPC = THREADS / TPB;           // blocks per CTA
  static constexpr int TS = BW + 1;                   // padded row stride
  // Shared memory of a block (a multiple of 4 floats): the input tile, then
  // the row spectra; the filtered spectrum, then the column results.
  static constexpr int even4(int n) { return (n + 3) / 4 * 4; }
  static constexpr int FWD_FLOATS = even4(BH * TS > 2 * PS ? BH * TS : 2 * PS);
  static constexpr int INV_FLOATS = even4(2 * PS > 2 * BH * TS ? 2 * PS : 2 * BH * TS);
  // Loads in flight per thread: the gather takes GB samples (and window
  // values) per round, the Kalman filter KB bins (spectrum, state, tables)
  // before any of their results is stored.
  static constexpr int GB = BW * BH / TPB < 16 ? BW * BH / TPB : 16;
  static constexpr int NJ = (PS + TPB - 1) / TPB;
  static constexpr int KB = NJ < 8 ? NJ : 8;
  // Resident CTAs per SM the register budget is set for (a transform of TPB
  // values holds 2 TPB registers).
  static constexpr int FWD_CTAS = TPB == 64 ? 3 : 6;
  static constexpr int INV_CTAS = TPB == 64 ? 3 : 5;  // Kalman: one fewer at TPB < 64
};

// Threads of one block: a block of up to 32 threads lives in one warp.
template <int TPB>
__device__ __forceinline__ void block_sync() {
  if constexpr (TPB <= 32) __syncwarp();
  else __syncthreads();
}

// Gather of a block with mirror addressing, sample conversion, chroma
// centering and analysis window (src/cpu/reference.cpp:140-159) into
// tile[BH][TS]. Thread t of TPB (a multiple of BW) keeps one column and takes
// every (TPB / BW)-th row, GB rows in flight. The sample format is fixed
// outside the loops and blocks inside the plane need no mirroring: with the
// format switch and the mirror inside the unrolled loop the code was large
// enough for instruction fetch to stall the kernels (forward, 1080p 10-bit
// with 32x32 blocks: 53 -> 20 us; 720p float with 64x64 blocks: 30 -> 18 us).
template <int BW, int BH, int TPB, int GB, int TS, int FMT>
__device__ __forceinline__ void gather_fmt(const FwdArgs& a, int bx, int by, int t, float* tile) {
  constexpr int RS = TPB / BW, NR = BH / RS;  // rows per round, rounds
  static_assert(TPB % BW == 0 && BH % RS == 0 && NR % GB == 0, "row split");
  const int lx = t % BW, ly0 = t / BW;
  const float* win = a.win + t;
  float* dst = tile + ly0 * TS + lx;
  if (bx >= 0 && by >= 0 && bx + BW <= a.g.W && by + BH <= a.g.H) {
    const uint8_t* row = a.src + (long long)(by + ly0) * a.pitch;
    for (int k0 = 0; k0 < NR; k0 += GB) {
      float v[GB], w[GB];
#pragma unroll
      for (int u = 0; u < GB; u++) {
        v[u] = load_sample(row + (long long)((k0 + u) * RS) * a.pitch, bx + lx, FMT, a.norm);
        w[u] = win[(k0 + u) * TPB];
      }
#pragma unroll
      for (int u = 0; u < GB; u++) {
        const float c = v[u] - a.chroma_norm;
        dst[(k0 + u) * RS * TS] = c * w[u];
      }
    }
  } else {
    const int x = mirror_i(bx + lx, a.g.W);
#pragma unroll 4
    for (int k = 0; k < NR; k++) {
      const int y = mirror_i(by + ly0 + k * RS, a.g.H);
      const float c = load_sample(a.src + (long long)y * a.pitch, x, FMT, a.norm) - a.chroma_norm;
      dst[k * RS * TS] = c * win[k * TPB];
    }
  }
}
template <int BW, int BH, int TPB, int GB, int TS>
__device__ __forceinline__ void gather_block(const FwdArgs& a, int b, int t, float* tile) {
  int bx, by, par;
  block_origin(a.g, b, bx, by, par);
  if (a.fmt == FMT_U8) gather_fmt<BW, BH, TPB, GB, TS, FMT_U8>(a, bx, by, t, tile);
  else if (a.fmt == FMT_U16) gather_fmt<BW, BH, TPB, GB, TS, FMT_U16>(a, bx, by, t, tile);
  else gather_fmt<BW, BH, TPB, GB, TS, FMT_F32>(a, bx, by, t, tile);
}

// One block: gather, row FFTs, then the fbw kept column FFTs
// (src/cpu/fft.cpp:68-86); store the half spectrum. The row spectra take the
// input tile's place: every row is in registers before any is written.
template <int BW, int BH>
__global__ void __launch_bounds__(Cfg<BW, BH>::THREADS, Cfg<BW, BH>::FWD_CTAS)
    k_forward_exact(const __grid_constant__ FwdArgs a) {
  using C = Cfg<BW, BH>;
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const int slot = threadIdx.x / C::TPB, t = threadIdx.x - slot * C::TPB;
  const int b = blockIdx.x * C::BPC + slot;
  const bool valid = b < a.g.nb;
  float* tile = smem + slot * C::FWD_FLOATS;
  float2* rows = reinterpret_cast<float2*>(tile);
  float2* out = a.spec + (size_t)b * C::PS;

  grid_go();
  grid_wait();
  stamp_start(a.clk);
  if (valid) gather_block<BW, BH, C::TPB, C::GB, C::TS>(a, b, t, tile);
  block_sync<C::TPB>();
  static_assert(C::TPB >= BH && C::TPB >= C::FBW, "one row, one column per thread");
  {
    float2 v[BW];
    if (t < BH) {
#pragma unroll
      for (int c = 0; c < BW; c++) v[c] = make_float2(tile[t * C::TS + c], 0.0f);
    }
    block_sync<C::TPB>();
    if (t < BH) {
      fft_r2<BW, false>(v, a.tw.row);
#pragma unroll
      for (int c = 0; c < C::FBW; c++) rows[t * C::FBW + c] = v[c];
    }
  }
  block_sync<C::TPB>();
  if (valid && t < C::FBW) {
    float2 v[BH];
#pragma unroll
    for (int r = 0; r < BH; r++) v[r] = rows[r * C::FBW + t];
    fft_r2<BH, false>(v, a.tw.col);
#pragma unroll
    for (int r = 0; r < BH; r++) out[r * C::FBW + t] = v[r];
  }
  stamp_end(a.clk);
}

// The filtered half spectrum of block b (temporal filter + sharpen per bin,
// src/cpu/reference.cpp:246-409) into F[PS]. NB bins' window spectra (Kalman:
// and state and tables) are loaded before any of them is filtered: the
// compiler cannot move a bin's loads above the previous bin's state stores,
// and the loads of one bin alone leave the memory system idle.
template <int BM, int PS, int TPB, int NB>
__device__ __forceinline__ void filter_block(const InvArgs& a, int b, int t, float2* F) {
  constexpr int NJ = (PS + TPB - 1) / TPB;
  const size_t base = (size_t)b * PS;
  const float dc = block_dc(a, b);
  for (int j0 = 0; j0 < NJ; j0 += NB) {
    float2 sv[NB][4];
    KState ks[NB];
    BinTables tb[NB];
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int i = t + (j0 + u) * TPB;
      if (j0 + u >= NJ || i >= PS) continue;
      load_window<BM>(a, base + i, sv[u]);
      if (BM == 0) ks[u] = load_kstate(a, base + i);
      if (BM == 0) tb[u] = bin_tables(a, i);
    }
#pragma unroll
    for (int u = 0; u < NB; u++) {
      const int i = t + (j0 + u) * TPB;
      if (j0 + u >= NJ || i >= PS) continue;
      F[i] = filter_vals_ks<BM>(a, dc, BM == 0 ? tb[u] : bin_tables(a, i), base + i, sv[u], ks[u]);
    }
  }
}

// Blocks four wide or high (PS bins, TPB threads): at most three bins a thread,
// all loaded together, and no prefetch of runs as short as 96 bytes (inverse, 4K
// 10-bit bt=4, both / one bin at a time and prefetched / neither prefetched: 4 x 8
// 225, 285, 260 us, 8 x 4 223, 272, 235, 4 x 32 410, 455, 466).
constexpr bool small_block(int ps, int tpb) { return ps <= 3 * tpb; }

// The temporal mode as a template argument (square blocks: one copy of the
// filter for each mode, of which a launch runs one) or read per bin.
template <bool KALMAN, bool BY_MODE, int PS, int TPB, int KB>
__device__ __forceinline__ void filter_block_any(const InvArgs& a, int b, int t, float2* F) {
  // Bins in flight, temporal modes (the block's spectra are on their way into
  // L2): with more, the code outgrows the instruction cache (1080p 10-bit, pass
  // with 1, 2, 3, 4 in flight: 32x32 bt=4 97.4, 97.6, 97.6, 104 us, bt=1 78, 76,
  // 75, 76; bt=3 64x64 on pairs 129.5, 129.6, 132, 137, 16x16 79, 81, 84, 86, 8x8 85, 86,
  // 89, 95).
  constexpr int KN = TPB == 64 ? 3 : (small_block(PS, TPB) ? 4 : 1);
  if constexpr (KALMAN) {
    filter_block<0, PS, TPB, KB>(a, b, t, F);
  } else if constexpr (BY_MODE) {
    switch (a.bm) {
    case 4: filter_block<4, PS, TPB, KN>(a, b, t, F); break;
    case 3: filter_block<3, PS, TPB, KN>(a, b, t, F); break;
    case 2: filter_block<2, PS, TPB, KN>(a, b, t, F); break;
    case 1: filter_block<1, PS, TPB, KN>(a, b, t, F); break;
    default: filter_block<-1, PS, TPB, KN>(a, b, t, F);
    }
  } else {
    filter_block<kRuntimeBm, PS, TPB, KN>(a, b, t, F);
  }
}

// Starts the window spectra of block b moving into L2 (one thread's call).
template <int PS>
__device__ __forceinline__ void prefetch_window(const InvArgs& a, int b) {
  const int nf = a.bm >= 2 ? a.bm : 1;
  for (int k = 0; k < nf; k++)
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(a.s[k] + (size_t)b * PS), "r"(PS * 8) : "memory");
}

// Rows of a block's windowed inverse: sample pair j of row r (its two values
// before the window) at S[at(r, j)], written by the threads of the row
// transforms, read back here in plane order, so that the window is read and
// the block written in whole lines. Stored straight from the row transforms
// each thread walks its own row: 16 to 32 lines per request, and the loads
// and stores of the block took half of the kernel (inverse, 1080p 10-bit bt=4
// with 32x32 blocks: 180 -> 99 us; 720p Kalman with 64x64 blocks: 60 -> 35 us).
template <int BW, int BH, int TPB, class At>
__device__ __forceinline__ void store_block(const InvArgs& a, int b, int t, const float2* S, At&& at) {
  int bx, by, par;
  block_origin(a.g, b, bx, by, par);
  const float2* win = reinterpret_cast<const float2*>(par ? a.win_b : a.win_a);
  float2* out = reinterpret_cast<float2*>(a.blocks + (size_t)b * BW * BH);
#pragma unroll 8
  for (int i = t; i < BW * BH / 2; i += TPB) {
    const float2 v = S[at(i / (BW / 2), i % (BW / 2))], w = win[i];
    out[i] = make_float2(v.x * w.x, v.y * w.y);
  }
}

// One block: temporal filter + sharpen per bin, Hermitian completion and
// column inverse FFTs, row inverse FFTs, real part times the synthesis
// window (src/cpu/reference.cpp:246-430, src/cpu/fft.cpp:88-119). G takes
// F's place: every column is in registers before any is written.
template <int BW, int BH, bool KALMAN>
__global__ void __launch_bounds__(Cfg<BW, BH>::THREADS, Cfg<BW, BH>::INV_CTAS - (KALMAN && Cfg<BW, BH>::TPB < 64))
    k_inverse_exact(const __grid_constant__ InvArgs a) {
  using C = Cfg<BW, BH>;
  extern __shared__ float4 smem4[];
  float* smem = reinterpret_cast<float*>(smem4);
  const int slot = threadIdx.x / C::TPB, t = threadIdx.x - slot * C::TPB;
  const int b = blockIdx.x * C::BPC + slot;
  const bool valid = b < a.g.nb;
  float2* F = reinterpret_cast<float2*>(smem + slot * C::INV_FLOATS);
  float2* G = F;

  grid_go();
  grid_wait();
  stamp_start(a.clk);
  if (!KALMAN && !small_block(C::PS, C::TPB) && valid && t == 0) prefetch_window<C::PS>(a, b);
  if (valid) filter_block_any<KALMAN, BW == BH, C::PS, C::TPB, C::KB>(a, b, t, F);
  block_sync<C::TPB>();
  {
    float2 v[BH];
    if (t < C::FBW) {  // column t, kept or completed
#pragma unroll
      for (int r = 0; r < BH; r++) v[r] = F[r * C::FBW + t];
    } else if (t < BW) {
#pragma unroll
      for (int r = 0; r < BH; r++) {
        const float2 m = F[((BH - r) % BH) * C::FBW + (BW - t)];
        v[r] = make_float2(m.x, -m.y);
      }
    }
    block_sync<C::TPB>();
    if (t < BW) {
      fft_r2<BH, true>(v, a.tw.col);
#pragma unroll
      for (int r = 0; r < BH; r++) G[r * C::TS + t] = v[r];
    }
  }
  block_sync<C::TPB>();
  if (t < BH) {
    float2 v[BW];
#pragma unroll
    for (int c = 0; c < BW; c++) v[c] = G[t * C::TS + c];
    fft_r2<BW, true>(v, a.tw.row);
#pragma unroll
    for (int c = 0; c < BW / 2; c++) G[t * C::TS + c] = make_float2(v[2 * c].x, v[2 * c + 1].x);
  }
  block_sync<C::TPB>();
  if (valid) store_block<BW, BH, C::TPB>(a, b, t, G, [](int r, int j) { return r * C::TS + j; });
  stamp_end(a.clk);
}

// ---- 64 x 64 blocks, inverse of 32 x 32: each transform on 2 or 4 lanes -----
//
// One thread per 64-point transform holds 128 registers of data and leaves
// 504 CTAs of two 720p blocks in two waves; a lane pair (lanes 2i, 2i+1)
// halves both. The bit-reversed array is split in halves: the even lane
// holds positions 0..N/2-1, the odd lane the others. Stages len = 2..N/2 stay
// inside a half (twiddles tw[j * N / len], as in the whole transform); the last
// stage pairs position j with j + N/2: the odd lane forms t = w_j * a[j + N/2],
// the lanes swap t and u = a[j] by one shuffle, and each forms its output,
// u + t or u - t. On four lanes the last two stages are formed so. Every value
// is computed by the same operations as in fft_r2<N> (src/cpu/fft.cpp:28-58),
// so the bits are the same.
//
// The inverse takes 16 values of a transform per lane: 64 registers a thread
// and 32 warps an SM. 32 x 32 blocks, pairs (k_inverse_exact: 24 warps of twice
// the work, half of their issue slots idle on loads, divides and instruction
// fetch): pass of 1080p 10-bit bt=4 124 -> 98 us, bt=1 90 -> 75, Kalman
// 89 -> 74, 360p bt=3 38 -> 27. 64 x 64 blocks, four lanes (pairs: 20 warps, and
// the latency of one block counted twice where 720p has 1,008 of them for 760
// places): 720p Kalman 56 -> 51, bt=3 72 -> 59, 1080p bt=3 130 -> 116.
// The forward of 32 x 32 blocks lost by pairs (98 -> 103 us): 17 columns take
// a second warp.

template <int N, int LEN, bool INV, int M>
__device__ __forceinline__ void half_stage(float2 (&a)[M], const float2* tw) {
  constexpr int half = LEN / 2, step = N / LEN;
#pragma unroll
  for (int i = 0; i < M; i += LEN) {
#pragma unroll
    for (int j = 0; j < half; j++) {
      const float2 b = a[i + j + half];
      float2 t;
      if (j == 0) {
        t = b;
      } else {
        const float2 w = tw[j * step];
        const float wy = INV ? -w.y : w.y;
        t.x = w.x * b.x - wy * b.y;
        t.y = w.x * b.y + wy * b.x;
      }
      const float2 u = a[i + j];
      a[i + j] = make_float2(u.x + t.x, u.y + t.y);
      a[i + j + half] = make_float2(u.x - t.x, u.y - t.y);
    }
  }
  if constexpr (LEN < M) half_stage<N, LEN * 2, INV, M>(a, tw);
}

// a: positions N/2 * odd + p (p < N/2) of the bit-reversed input; out: the
// transform's values N/2 * odd + p. Every lane of the warp takes part.
template <int N, bool INV>
__device__ __forceinline__ void fft_pair(float2 (&a)[N / 2], const float2* tw, bool odd) {
  half_stage<N, 2, INV, N / 2>(a, tw);
#pragma unroll
  for (int j = 0; j < N / 2; j++) {
    const float2 x = a[j];
    float2 t = x;
    if (j > 0) {
      const float2 w = tw[j];
      const float wy = INV ? -w.y : w.y;
      t.x = w.x * x.x - wy * x.y;
      t.y = w.x * x.y + wy * x.x;
    }
    const float2 send = odd ? t : x;
    const float rx = __shfl_xor_sync(0xffffffffu, send.x, 1), ry = __shfl_xor_sync(0xffffffffu, send.y, 1);
    a[j] = odd ? make_float2(rx - t.x, ry - t.y) : make_float2(x.x + rx, x.y + ry);
  }
  if (INV) {
    const float invn = 1.0f / N;
#pragma unroll
    for (int i = 0; i < N / 2; i++) a[i] = make_float2(a[i].x * invn, a[i].y * invn);
  }
}

constexpr int kPairThreads = 128;  // one 64 x 64 block per CTA
constexpr int kPairTS = 65;        // padded row stride (float or float2)

// Forward of one 64 x 64 block per CTA: gather, row transforms (pair p =
// row p), then the 33 kept columns (pair p = column p). The input tile and
// the row spectra share shared memory: every row is in registers before any
// row spectrum is written.
__global__ void __launch_bounds__(kPairThreads, 6) k_forward_exact64(const __grid_constant__ FwdArgs a) {
  constexpr int FBW = 33;
  extern __shared__ float4 smem4[];
  float* tile = reinterpret_cast<float*>(smem4);    // [64][kPairTS]
  float2* rows = reinterpret_cast<float2*>(smem4);  // [64][FBW], after the row transforms
  const int t = threadIdx.x, p = t >> 1;
  const bool odd = t & 1;
  const int b = blockIdx.x;
  grid_go();
  grid_wait();
  stamp_start(a.clk);
  gather_block<64, 64, kPairThreads, 16, kPairTS>(a, b, t, tile);
  __syncthreads();
  float2 r[32];
#pragma unroll
  for (int q = 0; q < 32; q++) r[q] = make_float2(tile[p * kPairTS + bit_reverse(q, 6) + odd], 0.0f);
  __syncthreads();  // the tile is read: the row spectra may overwrite it
  fft_pair<64, false>(r, a.tw.row, odd);
  if (!odd) {
#pragma unroll
    for (int c = 0; c < 32; c++) rows[p * FBW + c] = r[c];
  } else {
    rows[p * FBW + 32] = r[0];
  }
  __syncthreads();
  if (t < 2 * 48) {  // warps holding columns 0..32 (lanes of columns 33.. run along, store nothing)
    const int c = p < FBW ? p : 0;
#pragma unroll
    for (int q = 0; q < 32; q++) r[q] = rows[(bit_reverse(q, 6) + odd) * FBW + c];
    fft_pair<64, false>(r, a.tw.col, odd);
    if (p < FBW) {
      float2* out = a.spec + (size_t)b * 64 * FBW + c;
#pragma unroll
      for (int q = 0; q < 32; q++) out[(32 * odd + q) * FBW] = r[q];
      stamp_end(a.clk);  // in here: behind the branches it made the registers spill
    }
  }
}

// One stage between lanes: u + t on the lane with the lower half (hi false),
// u - t on the other, t = w_j * its value; w_0 = 1 (first: of a[0]) takes no
// product, which would change zeros' signs and infinities.
template <bool INV, int M, class W>
__device__ __forceinline__ void lane_stage(float2 (&a)[M], int lane_mask, bool hi, bool first, W&& tw) {
#pragma unroll
  for (int j = 0; j < M; j++) {
    const float2 x = a[j], w = tw(j);
    const float wy = INV ? -w.y : w.y;
    float2 t = make_float2(w.x * x.x - wy * x.y, w.x * x.y + wy * x.x);
    if (j == 0 && first) t = x;
    const float2 send = hi ? t : x;
    const float rx = __shfl_xor_sync(0xffffffffu, send.x, lane_mask), ry = __shfl_xor_sync(0xffffffffu, send.y, lane_mask);
    a[j] = hi ? make_float2(rx - t.x, ry - t.y) : make_float2(x.x + rx, x.y + ry);
  }
}

// The inverse transform of N values on a group of G lanes, lane l holding
// positions N/G * l + q of the bit-reversed input, then of the output.
template <int N, int G>
__device__ __forceinline__ void ifft_group(float2 (&a)[N / G], const float2* tw, int l) {
  if constexpr (G == 2) {
    fft_pair<N, true>(a, tw, l);
  } else {
    constexpr int M = N / 4;
    static_assert(G == 4, "two or four lanes");
    half_stage<N, 2, true, M>(a, tw);
    lane_stage<true>(a, 1, l & 1, true, [&](int j) { return tw[2 * j]; });
    lane_stage<true>(a, 2, l & 2, !(l & 1), [&](int j) {
      const float2 w0 = tw[j], w1 = tw[j + M];
      return l & 1 ? w1 : w0;
    });
    const float invn = 1.0f / N;
#pragma unroll
    for (int i = 0; i < M; i++) a[i] = make_float2(a[i].x * invn, a[i].y * invn);
  }
}

template <int N>
struct InvLanes {
  static constexpr int LN = N == 64 ? 4 : 2;
  static constexpr int THREADS = LN * N, M = N / LN;
  // Row stride of G, and how far each further M rows are moved along: a
  // half-warp's columns, or rows, lie in different banks.
  static constexpr int TS = LN == 4 ? N + 4 : N + 1, SKEW = LN == 4 ? 4 : 0;
  static __device__ __forceinline__ int at(int row, int col) { return row * TS + row / M * SKEW + col; }
  // A row's lanes put their M/2 sample pairs kAt entries apart (banks again).
  static constexpr int kAt = LN == 4 ? 12 : 8;
  static constexpr size_t SMEM = sizeof(float2) * (N * TS + LN * SKEW);
};

// Filter + inverse of one N x N block per CTA, each transform on LN lanes: the
// filtered half spectrum F, column transforms (group p = column p, Hermitian
// completion on the fly) into G, which shares F's space once every column is in
// registers, then row transforms (group p = row p) and the windowed rows in
// plane order.
template <int N, bool KALMAN>
__global__ void __launch_bounds__(InvLanes<N>::THREADS, 1024 / InvLanes<N>::THREADS)
    k_inverse_lanes(const __grid_constant__ InvArgs a) {
  using C = InvLanes<N>;
  constexpr int FBW = N / 2 + 1, PS = N * FBW, LN = C::LN, M = C::M, L = Log2<N>::v;
  extern __shared__ float4 smem4[];
  float2* F = reinterpret_cast<float2*>(smem4);  // [N][FBW]
  float2* G = F;                                 // [N][TS], after the column reads
  const int t = threadIdx.x, p = t / LN, l = t % LN;
  const int rl = LN == 4 ? bit_reverse(l, 2) : l;
  const int b = blockIdx.x;
  grid_go();
  grid_wait();
  stamp_start(a.clk);
  if (!KALMAN && t == 0) prefetch_window<PS>(a, b);
  filter_block_any<KALMAN, true, PS, C::THREADS, 3>(a, b, t, F);
  __syncthreads();
  float2 r[M];
#pragma unroll
  for (int q = 0; q < M; q++) {
    const int row = bit_reverse(q, L) + rl;  // bit_reverse(M * l + q)
    if (p < FBW) {
      r[q] = F[row * FBW + p];
    } else {
      const float2 m = F[((N - row) & (N - 1)) * FBW + (N - p)];
      r[q] = make_float2(m.x, -m.y);
    }
  }
  __syncthreads();  // F is read: G may overwrite it
  ifft_group<N, LN>(r, a.tw.col, l);
#pragma unroll
  for (int q = 0; q < M; q++) G[C::at(M * l + q, p)] = r[q];
  __syncthreads();
#pragma unroll
  for (int q = 0; q < M; q++) r[q] = G[C::at(p, bit_reverse(q, L) + rl)];
  ifft_group<N, LN>(r, a.tw.row, l);
  __syncwarp();  // the group has read its row
#pragma unroll
  for (int q = 0; q < M / 2; q++) G[C::at(p, C::kAt * l + q)] = make_float2(r[2 * q].x, r[2 * q + 1].x);
  __syncthreads();
  store_block<N, N, C::THREADS>(a, b, t, G, [](int row, int j) {
    return C::at(row, j / (M / 2) * C::kAt + j % (M / 2));
  });
  stamp_end(a.clk);
}

cudaError_t launch_fwd64(const FwdArgs& a, cudaStream_t st) {
  const size_t smem = sizeof(float2) * 64 * 33 > sizeof(float) * 64 * kPairTS ? sizeof(float2) * 64 * 33
                                                                               : sizeof(float) * 64 * kPairTS;
  if (a.g.nb == 0) return cudaSuccess;
  return launch_kernel(k_forward_exact64, a.g.nb, kPairThreads, smem, st, a);
}

template <int N, bool KALMAN>
cudaError_t launch_inv_lanes(const InvArgs& a, cudaStream_t st) {
  using C = InvLanes<N>;
  static_assert(C::SMEM <= 48 * 1024, "shared memory without opting in");
  static_assert(C::SMEM >= sizeof(float2) * N * (N / 2 + 1), "G covers F");
  if (a.g.nb == 0) return cudaSuccess;
  return launch_kernel(k_inverse_lanes<N, KALMAN>, a.g.nb, C::THREADS, C::SMEM, st, a);
}

template <int BW, int BH>
cudaError_t launch_fwd(const FwdArgs& a, cudaStream_t st) {
  if constexpr (BW == 64 && BH == 64) {
    return launch_fwd64(a, st);
  } else {
    using C = Cfg<BW, BH>;
    const size_t smem = sizeof(float) * C::FWD_FLOATS * C::BPC;
    auto k = k_forward_exact<BW, BH>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    const int grid = (a.g.nb + C::BPC - 1) / C::BPC;
    if (grid == 0) return cudaSuccess;
    return launch_kernel(k, grid, C::THREADS, smem, st, a);
  }
}

template <int BW, int BH>
cudaError_t launch_inv(const InvArgs& a, cudaStream_t st) {
  if constexpr (BW == BH && BW >= 32) {
    return a.bm == 0 ? launch_inv_lanes<BW, true>(a, st) : launch_inv_lanes<BW, false>(a, st);
  } else {
    using C = Cfg<BW, BH>;
    const size_t smem = sizeof(float) * C::INV_FLOATS * C::BPC;
    auto k = a.bm == 0 ? k_inverse_exact<BW, BH, true> : k_inverse_exact<BW, BH, false>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    const int grid = (a.g.nb + C::BPC - 1) / C::BPC;
    if (grid == 0) return cudaSuccess;
    return launch_kernel(k, grid, C::THREADS, smem, st, a);
  }
}

}  // namespace

#define F3D_CAT2(a, b) a##b
#define F3D_CAT(a, b) F3D_CAT2(a, b)

cudaError_t F3D_CAT(launch_forward_exact_bw, F3D_BW)(const FwdArgs& a, cudaStream_t st) {
  switch (a.g.bh) {
  case 4: return launch_fwd<F3D_BW, 4>(a, st);
  case 8: return launch_fwd<F3D_BW, 8>(a, st);
  case 16: return launch_fwd<F3D_BW, 16>(a, st);
  case 32: return launch_fwd<F3D_BW, 32>(a, st);
  case 64: return launch_fwd<F3D_BW, 64>(a, st);
  default: return cudaErrorInvalidValue;
  }
}

cudaError_t F3D_CAT(launch_inverse_exact_bw, F3D_BW)(const InvArgs& a, cudaStream_t st) {
  switch (a.g.bh) {
  case 4: return launch_inv<F3D_BW, 4>(a, st);
  case 8: return launch_inv<F3D_BW, 8>(a, st);
  case 16: return launch_inv<F3D_BW, 16>(a, st);
  case 32: return launch_inv<F3D_BW, 32>(a, st);
  case 64: return launch_inv<F3D_BW, 64>(a, st);
  default: return cudaErrorInvalidValue;
  }
}

}  // namespace f3d
