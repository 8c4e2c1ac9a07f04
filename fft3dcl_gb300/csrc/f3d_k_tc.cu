// f3d_k_tc.cu -- the tensor-core form: 2D block DFTs as dense DFT-matrix
// products on the fifth-generation tensor cores (tcgen05), fp16 operands
// split into hi + lo parts with fp32 accumulation in tensor memory.
//
// Forward transform of an n x n real block X (n = 32) with separable
// analysis window wx[x] * wy[y] (src/cpu/tables.cpp:21-105), folded into the
// DFT matrices:
//   step 1 (rows):    Z[y][j] = sum_x X[y][x] * B1[j][x], the n real outputs
//                     j = (Re Z0, Re Z(n/2), Re Z1, Im Z1, .., Im Z(n/2-1)) of
//                     each row's real DFT;
//   step 2 (columns): for each packed column k' = 0..n/2-1 (k' = 0 carries
//                     Z0 + i Z(n/2)), Y[ky][k'] = sum_y e^(-2 pi i ky y/n)
//                     wy[y] Z[y][k'] as a real 2n x 2n matrix B2 acting on
//                     interleaved (re, im) pairs;
//   unpacking:        Y0 = (P + conj P(-ky))/2, Y(n/2) = (P - conj P(-ky))/2i
//                     for the packed column P.
// This equals fft2dRealForward of the windowed block (src/cpu/fft.cpp:68-86,
// src/cpu/reference.cpp:140-170) up to fp32 rounding. The chroma offset is
// removed in the spectrum (c * DFT(window)), the sample scale (1/255,
// 2^(16-bits)/65535) applied to the output.
//
// Tiling: a group of G = 8 blocks; step 1 runs as two M = 128 tiles (rows =
// 4 blocks x 32 rows, N = 32, K = 32), step 2 as one M = 128 tile (rows = 8
// blocks x 16 packed columns, N = 64, K = 64). Operands hi/lo: step 1 uses
// X exactly (integer samples of up to 11 bits are exact in fp16) times
// B1hi + B1lo, or Xhi*B1hi + Xhi*B1lo + Xlo*B1hi; step 2 Ahi*Bhi + Ahi*Blo +
// Alo*Bhi. The spectra of a group (8 x 4352 bytes, contiguous in HBM) leave
// shared memory by one bulk copy.
#include "f3d_batch_plan.hpp"
#include "f3d_device.cuh"
#include "f3d_tc.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>

namespace f3d {
namespace {

constexpr double kPiD = 3.14159265358979323846;

// Byte offsets of the table sections for n x n blocks.
template <int N>
struct TcTab {
  static constexpr int FBW = N / 2 + 1;
  static constexpr uint32_t B1HI = 0, B1LO = B1HI + N * N * 2;
  static constexpr uint32_t B2HI = B1LO + N * N * 2, B2LO = B2HI + 8 * N * N;
  static constexpr uint32_t WSPEC = B2LO + 8 * N * N;  // float2 [N][FBW]
  static constexpr uint32_t C2HI = WSPEC + N * FBW * 8, C2LO = C2HI + 8 * N * N;
  // Row inverses with the even (A) and odd (B) synthesis x-windows.
  static constexpr uint32_t C1AHI = C2LO + 8 * N * N, C1ALO = C1AHI + N * N * 2;
  static constexpr uint32_t C1BHI = C1ALO + N * N * 2, C1BLO = C1BHI + N * N * 2;
  static constexpr uint32_t TOTAL = C1BLO + N * N * 2;
  static_assert(WSPEC % 16 == 0 && C2HI % 16 == 0 && C1AHI % 16 == 0, "16-byte sections");
};

// Scale of the filtered spectrum before its hi/lo split in the inverse
// (keeps the column sums inside fp16 range), undone with the inverse's
// 1/n^2 when the blocks are added up.
constexpr float kInvPre = 1.0f / 16.0f;

// Kernel configuration for n x n blocks.
template <int N>
struct TcCfg {
  static constexpr int NY = N / 2, FBW = NY + 1, PS = N * FBW;
  static constexpr int G = 128 / NY;       // blocks per group (step-2 tile rows: G x NY)
  static constexpr int BPT1 = 128 / N;     // blocks per step-1 tile (rows: BPT1 x N)
  static constexpr int T1 = G / BPT1;      // step-1 tiles per group
  static constexpr int K1 = N, N1 = N;     // step 1: K = x, N = packed outputs
  static constexpr int K2 = 2 * N, N2 = 2 * N;
  static constexpr uint32_t A1_BYTES = 128 * K1 * 2, A2_BYTES = 128 * K2 * 2;
  static constexpr uint32_t B1_BYTES = N1 * K1 * 2, B2_BYTES = N2 * K2 * 2;
  static constexpr uint32_t TMEM_COLS = 128;
  static constexpr uint32_t D1_COL = 0, D2_COL = 64;
  static_assert(N == 16 || N == 32, "the tensor-core form is built for 16 x 16 and 32 x 32 blocks");
  static_assert(T1 * N1 <= (int)D2_COL && D2_COL + N2 <= (int)TMEM_COLS, "tensor memory columns");
};

// The step-2 operand (128 rows, K2 = 2N fp16 columns; the column inverse's
// operand tile too): SWIZZLE_128B for N = 32 (rows of 128 bytes), the
// interleaved core-matrix layout for N = 16 (rows of 64 bytes).
template <int N>
__host__ __device__ constexpr uint32_t a2_off(int row, int k) {
  return N == 32 ? tc::off_sw128(row, k) : tc::off_il(row, k, 2 * N);
}
// Descriptor of K-step ks (16 columns) of a step-2 operand at base.
template <int N>
__device__ __forceinline__ uint64_t a2_desc(uint32_t base, int ks) {
  if constexpr (N == 32) return tc::sdesc(base + ks * 32, 16, 1024, tc::LAYOUT_SW128);
  else return tc::sdesc(base + ks * 256, 128, (2 * N / 8) * 128, tc::LAYOUT_INTERLEAVE);
}

constexpr int kTcThreads = 256;
constexpr uint64_t kWaitNs = 1000000000ull;  // one second

// ---- forward ---------------------------------------------------------------

// Shared memory of the forward kernel (offsets from a 1024-aligned base).
// A1 and A2 are live at the same time (the next group's step-1 operand is
// deposited while step 2 of the current group runs). The staging area of a
// group's spectra shares A2's space: it is written once step 2 has read A2,
// and its bulk store has drained before the next group writes A2. Without the
// split (integer samples of up to 11 bits) A1 holds only the hi parts: 73 KB,
// three CTAs per SM; with the split 88 KB, two.
template <int N, bool SPLIT>
struct FwdSmem {
  using C = TcCfg<N>;
  // Step-1 operand: core matrices of 8 rows x 16 bytes, those of 8 columns of
  // all rows together (SBO 128), LBO apart. LBO is 32 or 64 bytes over a
  // multiple of 128: the chunks of a row that neighbouring lanes deposit then
  // fall in different banks (in the same four before: 512 of the 1214
  // shared-memory wavefronts of a 10-bit group).
  static constexpr uint32_t A1_LBO = 128 * 16 + (N == 32 ? 32 : 64), A1_SBO = 128;
  static constexpr uint32_t A1_PART = C::K1 / 8 * A1_LBO;
  static constexpr uint32_t A1_TILE = (SPLIT ? 2 : 1) * A1_PART;      // hi[, lo] of one step-1 tile
  static constexpr uint32_t a1_off(int row, int k) {
    return (k >> 3) * A1_LBO + (row >> 3) * A1_SBO + (row & 7) * 16 + (k & 7) * 2;
  }
  static constexpr uint32_t STAGE_BYTES = C::G * C::PS * 8;           // float2 [G][N][FBW]
  static constexpr uint32_t B2 = 0;                       // hi, lo
  static constexpr uint32_t B1 = B2 + 2 * C::B2_BYTES;    // hi, lo
  static constexpr uint32_t A2 = (B1 + 2 * C::B1_BYTES + 1023) / 1024 * 1024;  // hi, lo (SWIZZLE_128B)
  static constexpr uint32_t STAGE = A2;
  static constexpr uint32_t A1 = A2 + (2 * C::A2_BYTES > STAGE_BYTES ? 2 * C::A2_BYTES : STAGE_BYTES);
  static constexpr uint32_t BAR = A1 + C::T1 * A1_TILE;   // [tile][hi, lo]
  static constexpr uint32_t TSLOT = BAR + 16;
  static constexpr uint32_t BYTES = TSLOT + 16 + 1024;    // + alignment slack
  static_assert(STAGE % 16 == 0 && A1 % 128 == 0 && BAR % 16 == 0, "bulk-copy and operand alignment");
};
// CTAs per SM of the forward kernel: three fit in shared memory without the
// split, two with it; the words of unaligned rows do not fit in the registers
// of three (30 bytes spilled per thread cost more than the third CTA gave: 4K
// 10-bit 52 -> 60 us). Aligned 16-bit rows of 32 x 32 blocks spill 16 bytes at
// three, the other kernels none.
constexpr int kFwdMaxCtasPerSm = 3;
constexpr int fwd_ctas(bool split, bool aligned, int bps) { return split || (!aligned && bps == 2) ? 2 : kFwdMaxCtasPerSm; }

// Gather of a group's samples: a task covers 16 source bytes (16/BPS samples)
// of a row of a block. The raw bytes are fetched into registers one group
// ahead, so that their loads are in flight while the tensor cores work on the
// current group, and deposited into the step-1 operand as fp16. A thread's
// tasks are one chunk of one row of every BSTEP-th block; neighbouring lanes
// take the chunks of a row. (Eight rows of a chunk for neighbouring lanes would
// store without bank conflicts in any layout, but touch 8 lines in every
// quarter of a load: 4K 10-bit 52 -> 57 us.)
template <int N, int BPS>
struct Gather {
  static constexpr int S = 16 / BPS;                   // samples per task
  static constexpr int TPR = N / S;                    // tasks per block row
  static constexpr int TASKS = TcCfg<N>::G * N * TPR;
  static constexpr int TPT = TASKS / kTcThreads;       // tasks per thread
  static constexpr int BSTEP = kTcThreads / TPR / N;
  static_assert(TASKS % kTcThreads == 0 && S >= 4, "task split");
  static_assert(BSTEP * TPR * N == kTcThreads, "a thread keeps its row");
  static __device__ __forceinline__ int chunk() { return threadIdx.x % TPR; }
  static __device__ __forceinline__ int row() { return threadIdx.x / TPR % N; }
  static __device__ __forceinline__ int block() { return threadIdx.x / TPR / N; }
};

// mirror_i; within one plane width of the plane one reflection does it,
// without the division.
__device__ __forceinline__ int mirror_near(int x, int w) {
  if (x >= -w && x < 2 * w) return x < 0 ? -1 - x : (x < w ? x : 2 * w - 1 - x);
  return mirror_i(x, w);
}

// 16 bytes at p: one load where they are aligned, else the words that hold
// them. (A word read here holds at least one of the 16 bytes.)
__device__ __forceinline__ uint4 load16(const uint8_t* p) {
  const uintptr_t at = reinterpret_cast<uintptr_t>(p);
  if ((at & 15) == 0) return *reinterpret_cast<const uint4*>(p);
  const uint32_t* w = reinterpret_cast<const uint32_t*>(at & ~static_cast<uintptr_t>(3));
  const uint32_t sh = (at & 3) * 8;
  uint4 r = make_uint4(w[0], w[1], w[2], w[3]);
  if (sh) {
    const uint32_t e = w[4];
    r = make_uint4(__funnelshift_r(r.x, r.y, sh), __funnelshift_r(r.y, r.z, sh), __funnelshift_r(r.z, r.w, sh),
                   __funnelshift_r(r.w, e, sh));
  }
  return r;
}
// r = the 16 bytes (word) at p where `on`, else unchanged.
__device__ __forceinline__ void load16_if(bool on, const uint8_t* p, uint4& r) {
  asm volatile(
      "{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %4, 0;\n\t@q ld.global.v4.u32 {%0, %1, %2, %3}, [%5];\n\t}"
      : "+r"(r.x), "+r"(r.y), "+r"(r.z), "+r"(r.w)
      : "r"((int)on), "l"(p));
}
__device__ __forceinline__ void load4_if(bool on, const uint8_t* p, uint32_t& r) {
  asm volatile("{\n\t.reg .pred q;\n\tsetp.ne.b32 q, %1, 0;\n\t@q ld.global.u32 %0, [%2];\n\t}"
               : "+r"(r)
               : "r"((int)on), "l"(p));
}

// Raw bytes of a thread's tasks, one group ahead. ALIGNED: rows whose blocks
// start on 16 bytes (of every plane of the launch); else the words that hold
// the 16 bytes, shifted into place when they are used. plain: the group lies in
// one block row, inside the plane, and its loads have been issued; other groups
// (mirrored blocks, the ends of block rows) are read when they are used. The
// loads are predicated: behind a branch they were waited for where the paths
// join, one group early (4K 10-bit 50 -> 59 us).
template <int N, int BPS, bool ALIGNED>
struct RawGroup {
  using Gt = Gather<N, BPS>;
  static constexpr bool EXTRA = !ALIGNED && BPS < 4;  // a fifth word where rows start inside words
  uint4 r[Gt::TPT];
  uint32_t e[EXTRA ? Gt::TPT : 1];
  uint32_t sh;
  bool plain;

  __device__ __forceinline__ void fetch(const TcFwdArgs& a, int b0, int nvalid) {
    const int m0 = b0 / a.g.ncols, n0 = b0 - m0 * a.g.ncols;
    const int bx0 = a.g.xoff + n0 * a.g.xstep, by0 = a.g.yoff + m0 * a.g.ystep;
    plain = nvalid == TcCfg<N>::G && n0 + TcCfg<N>::G <= a.g.ncols && by0 >= 0 && by0 + N <= a.g.H && bx0 >= 0 &&
            bx0 + (TcCfg<N>::G - 1) * a.g.xstep + N <= a.g.W;
    const uint8_t* p = a.src + (long long)(by0 + Gt::row()) * a.pitch + (bx0 + Gt::block() * a.g.xstep) * BPS + 16 * Gt::chunk();
    const int step = Gt::BSTEP * a.g.xstep * BPS;  // a multiple of 4
    sh = ALIGNED ? 0u : (uint32_t)(reinterpret_cast<uintptr_t>(p) & 3) * 8;
    if constexpr (!ALIGNED) p -= sh / 8;
#pragma unroll
    for (int i = 0; i < Gt::TPT; i++) {
      r[i] = make_uint4(0u, 0u, 0u, 0u);
      if constexpr (ALIGNED) {
        load16_if(plain, p + i * step, r[i]);
      } else {
        load4_if(plain, p + i * step, r[i].x);
        load4_if(plain, p + i * step + 4, r[i].y);
        load4_if(plain, p + i * step + 8, r[i].z);
        load4_if(plain, p + i * step + 12, r[i].w);
        if constexpr (EXTRA) {
          e[i] = 0u;
          load4_if(plain && sh, p + i * step + 16, e[i]);
        }
      }
    }
  }

  // The bytes of the group that fetch() was called for, in r.
  __device__ __forceinline__ void finish(const TcFwdArgs& a, int b0, int nvalid) {
    if (plain) {
      if constexpr (EXTRA) {
#pragma unroll
        for (int i = 0; i < Gt::TPT; i++)
          r[i] = make_uint4(__funnelshift_r(r[i].x, r[i].y, sh), __funnelshift_r(r[i].y, r[i].z, sh),
                            __funnelshift_r(r[i].z, r[i].w, sh), __funnelshift_r(r[i].w, e[i], sh));
      }
      return;
    }
    // The group's blocks are consecutive in the mode-1 grid (the only mode of
    // this form): one division for the first, a carry into the next block row
    // for the others.
    const int m0 = b0 / a.g.ncols, n0 = b0 - m0 * a.g.ncols;
#pragma unroll
    for (int i = 0; i < Gt::TPT; i++) {
      const int bl = Gt::block() + i * Gt::BSTEP, y = Gt::row(), c = Gt::chunk();
      if (bl >= nvalid) continue;
      int n = n0 + bl, m = m0;
      while (n >= a.g.ncols) {
        n -= a.g.ncols;
        m++;
      }
      const int bx = a.g.xoff + n * a.g.xstep, by = a.g.yoff + m * a.g.ystep;
      if (bx >= 0 && by >= 0 && bx + N <= a.g.W && by + N <= a.g.H) {
        r[i] = load16(a.src + (long long)(by + y) * a.pitch + (long long)bx * BPS + 16 * c);
        continue;
      }
      // Mirrored: one sample at a time (src/cpu/reference.cpp:10-17).
      const uint8_t* line = a.src + (long long)mirror_near(by + y, a.g.H) * a.pitch;
      uint32_t w[4] = {0u, 0u, 0u, 0u};
#pragma unroll
      for (int k = 0; k < Gt::S; k++) {
        const int x = mirror_near(bx + c * Gt::S + k, a.g.W);
        uint32_t v;
        if (BPS == 1) v = line[x];
        else if (BPS == 2) v = reinterpret_cast<const uint16_t*>(line)[x];
        else v = reinterpret_cast<const uint32_t*>(line)[x];
        w[(k * BPS) / 4] |= v << (8 * ((k * BPS) % 4));
      }
      r[i] = make_uint4(w[0], w[1], w[2], w[3]);
    }
  }
};

// Raw bytes -> fp16 (hi, and lo on the split path) in A1[tile][part]: rows
// (block % BPT1, y), K = x.
template <int N, int BPS, bool SPLIT>
__device__ __forceinline__ void deposit(const TcFwdArgs& a, uint8_t* a1, const uint4 (&r)[Gather<N, BPS>::TPT]) {
  using Gt = Gather<N, BPS>;
  using C = TcCfg<N>;
  using L = FwdSmem<N, SPLIT>;
  const bool split = SPLIT && a.split;
  // Integer samples below 1024 become fp16 exactly by exponent bias: 0x6400
  // is 1024.0, and its ten mantissa bits hold the sample, so (0x6400 | v) -
  // 1024 = v, two instructions per pair. Samples of 1024 and above (11-bit
  // clips) take the conversion through fp32.
  bool small = BPS == 1;
  if (BPS == 2 && !split) {
    uint32_t hi_bits = 0u;
#pragma unroll
    for (int i = 0; i < Gt::TPT; i++) hi_bits |= r[i].x | r[i].y | r[i].z | r[i].w;
    small = (hi_bits & 0xFC00FC00u) == 0u;
  }
  const __half2 k1024 = __halves2half2(__ushort_as_half(0x6400), __ushort_as_half(0x6400));
#pragma unroll
  for (int i = 0; i < Gt::TPT; i++) {
    const int c = Gt::chunk(), bl = Gt::block() + i * Gt::BSTEP, y = Gt::row();
    const int tile = bl / C::BPT1, row = (bl % C::BPT1) * N + y;
    const uint32_t w[4] = {r[i].x, r[i].y, r[i].z, r[i].w};
    uint32_t h[Gt::S / 2], l[Gt::S / 2];
    if (BPS <= 2 && small) {
#pragma unroll
      for (int k = 0; k < Gt::S / 2; k++) {
        // The pair (sample 2k, sample 2k+1) with 0x64 as each one's high byte.
        const uint32_t biased = BPS == 1 ? __byte_perm(w[k >> 1], 0x64646464u, (k & 1) ? 0x4342u : 0x4140u)
                                         : (w[k] | 0x64006400u);
        const __half2 hv = __hsub2(*reinterpret_cast<const __half2*>(&biased), k1024);
        h[k] = *reinterpret_cast<const uint32_t*>(&hv);
        l[k] = 0u;
      }
    } else {
      float v[Gt::S];
#pragma unroll
      for (int k = 0; k < Gt::S; k++) {
        if (BPS == 1) v[k] = (float)((w[k >> 2] >> (8 * (k & 3))) & 0xffu);
        else if (BPS == 2) v[k] = (float)((w[k >> 1] >> (16 * (k & 1))) & 0xffffu) * (split ? a.norm : 1.0f);
        else v[k] = __uint_as_float(w[k]);
      }
#pragma unroll
      for (int k = 0; k < Gt::S / 2; k++) tc::split_pair(v[2 * k], v[2 * k + 1], h[k], l[k]);
    }
    uint8_t* t0 = a1 + tile * L::A1_TILE;
    const int x0 = c * Gt::S;
    if (Gt::S >= 8) {
#pragma unroll
      for (int j = 0; j < Gt::S / 8; j++) {
        const uint32_t o = L::a1_off(row, x0 + 8 * j);
        *reinterpret_cast<uint4*>(t0 + o) = make_uint4(h[4 * j], h[4 * j + 1], h[4 * j + 2], h[4 * j + 3]);
        if (split)
          *reinterpret_cast<uint4*>(t0 + L::A1_PART + o) = make_uint4(l[4 * j], l[4 * j + 1], l[4 * j + 2], l[4 * j + 3]);
      }
    } else {
      const uint32_t o = L::a1_off(row, x0);
      *reinterpret_cast<uint2*>(t0 + o) = make_uint2(h[0], h[1]);
      if (split) *reinterpret_cast<uint2*>(t0 + L::A1_PART + o) = make_uint2(l[0], l[1]);
    }
  }
}

// Plane of a batch that item idx (a CTA, or a forward block group) belongs to.
template <class Batch>
__device__ __forceinline__ int plane_of(const Batch& b, const int (&prefix)[kMaxBatch + 1], int idx) {
  int p = 0;
  while (p + 1 < b.n && idx >= prefix[p + 1]) p++;
  return p;
}

// Forward kernel: bound by the latency of a group's barrier-separated phases
// (tensor memory -> registers -> shared memory -> tensor cores), which three
// CTAs per SM overlap, and by shared-memory wavefronts. Without the address
// work and the bank conflicts of the gather (829 -> 590 instructions per block)
// ten 4K 10-bit outputs' step takes 1422 -> 1387 us; one 4K frame stays at 49
// us (cold), 1919x1079 float with 16x16 blocks goes 38 -> 30 us with word
// loads for its unaligned rows.
template <int N, int BPS, bool SPLIT, bool ALIGNED>
__global__ void __launch_bounds__(kTcThreads, fwd_ctas(SPLIT, ALIGNED, BPS)) k_forward_tc(const __grid_constant__ TcFwdBatch B) {
  using C = TcCfg<N>;
  using L = FwdSmem<N, SPLIT>;
  using T = TcTab<N>;
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sm = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  const uint32_t sbase = tc::smem_u32(sm);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + L::BAR);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + L::TSLOT);
  float2* stage = reinterpret_cast<float2*>(sm + L::STAGE);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;

  const int ngroups = B.grp0[B.n];
  uint32_t phase = 0;
  RawGroup<N, BPS, ALIGNED> raw;
  // The CTA's groups ascend, and so do their planes: pl is that of the group
  // whose spectra leave next, at or before any later group's.
  int pl = 0;
  auto plane_from = [&](int g) {
    int p = pl;
    while (g >= B.grp0[p + 1]) p++;
    return p;
  };
  // Raw samples of batch group g (the block group g - grp0[p] of plane p).
  auto fetch_group = [&](int g) {
    const int p = plane_from(g);
    const TcFwdArgs& ap = B.p[p];
    const int b = (g - B.grp0[p]) * C::G;
    raw.fetch(ap, b, min(C::G, ap.g.nb - b));
  };
  // Constant operands (the same for every plane of a batch): B2 (hi, lo) and
  // B1 (hi, lo) are contiguous in the table.
  {
    const uint4* src2 = reinterpret_cast<const uint4*>(B.p[0].tab + T::B2HI);
    uint4* dst2 = reinterpret_cast<uint4*>(sm + L::B2);
    for (int i = tid; i < (int)(2 * C::B2_BYTES / 16); i += kTcThreads) dst2[i] = src2[i];
    const uint4* src1 = reinterpret_cast<const uint4*>(B.p[0].tab + T::B1HI);
    uint4* dst1 = reinterpret_cast<uint4*>(sm + L::B1);
    for (int i = tid; i < (int)(2 * C::B1_BYTES / 16); i += kTcThreads) dst1[i] = src1[i];
  }
  if (warp == 0) {
    tc::tmem_alloc(tslot, C::TMEM_COLS);
    tc::tmem_relinquish();
  }
  if (tid == 0) {
    tc::mbar_init(&bar[0], 1);
    tc::mbar_init(&bar[1], 1);
    tc::fence_mbar_init();
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  const uint32_t tmem = *tslot;
  grid_go();
  grid_wait();
  stamp_start(B.p[0].clk);
  // Group g (its samples in raw) into A1, the loads of the CTA's group after
  // it started, then step 1 on the tensor cores: D1[tile] = A1 * B1^T, two or
  // three passes, committed to bar[0]. A1 and D1 must be free: no step 1 in
  // flight, D1 read out.
  auto begin_group = [&](int g) {
    const int p = plane_from(g);
    const TcFwdArgs& ap = B.p[p];
    const int b = (g - B.grp0[p]) * C::G;
    raw.finish(ap, b, min(C::G, ap.g.nb - b));
    deposit<N, BPS, SPLIT>(ap, sm + L::A1, raw.r);
    if (g + (int)gridDim.x < ngroups) fetch_group(g + gridDim.x);
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();
    if (tid == 0) {
      tc::fence_after_sync();
      constexpr uint32_t id1 = tc::idesc_f16(128, C::N1);
      const uint32_t sbo = (C::K1 / 8) * 128;
      for (int t = 0; t < C::T1; t++) {
        const uint32_t a_hi = sbase + L::A1 + t * L::A1_TILE, a_lo = a_hi + L::A1_PART;
        const uint32_t d = tmem + C::D1_COL + t * C::N1;
        for (int ks = 0; ks < C::K1 / 16; ks++) {
          const uint64_t ah = tc::sdesc(a_hi + ks * 2 * L::A1_LBO, L::A1_LBO, L::A1_SBO, tc::LAYOUT_INTERLEAVE);
          const uint64_t bh = tc::sdesc(sbase + L::B1 + ks * 256, 128, sbo, tc::LAYOUT_INTERLEAVE);
          const uint64_t bl = tc::sdesc(sbase + L::B1 + C::B1_BYTES + ks * 256, 128, sbo, tc::LAYOUT_INTERLEAVE);
          tc::mma_f16(d, ah, bh, id1, ks > 0);
          tc::mma_f16(d, ah, bl, id1, 1);
          if (SPLIT && ap.split)
            tc::mma_f16(d, tc::sdesc(a_lo + ks * 2 * L::A1_LBO, L::A1_LBO, L::A1_SBO, tc::LAYOUT_INTERLEAVE), bh, id1, 1);
        }
      }
      tc::mma_commit(&bar[0]);
    }
  };
  if ((int)blockIdx.x < ngroups) {
    fetch_group(blockIdx.x);
    begin_group(blockIdx.x);
  }

  // Per group: step 1 was issued one iteration earlier; step 2 runs while
  // the next group's samples are deposited and its step 1 issued; the
  // spectra are staged and leave by one bulk copy, which drains while the
  // next group goes through steps 1 to 5.
  for (int grp = blockIdx.x; grp < ngroups; grp += gridDim.x) {
    pl = plane_from(grp);
    const TcFwdArgs& a = B.p[pl];
    const int b0 = (grp - B.grp0[pl]) * C::G;
    const int nvalid = min(C::G, a.g.nb - b0);
    // The previous group's bulk store must have read the staging area, which
    // shares A2's space (written next). Every thread takes the same branch: a
    // wait that gave up anywhere ends the sweep of groups for the whole CTA.
    if (tid == 0) tc::bulk_wait_read();
    if (!__syncthreads_and(tc::mbar_wait(&bar[0], phase, kWaitNs))) {
      if (tid == 0) atomicOr(a.err, kErrWaitForward);
      break;
    }
    tc::fence_after_sync();

    // 3. D1 -> A2 (hi, lo): row (block, k'), K = 2y + (re, im).
    {
      const int t = warp >> 2, s = warp & 3;
      const int r1 = 32 * s + lane;
      const int bl = t * C::BPT1 + r1 / N, y = r1 % N;
      // 16 columns at a time: the next group's samples are in registers too.
#pragma unroll
      for (int k0 = 0; k0 < C::NY; k0 += 8) {
        float v[16];
        tc::tmem_ld<16>(tmem + ((uint32_t)(32 * s) << 16) + C::D1_COL + t * C::N1 + 2 * k0, v);
#pragma unroll
        for (int k = 0; k < 8; k++) {
          uint32_t hi, lo;
          tc::split_pair(v[2 * k], v[2 * k + 1], hi, lo);
          const uint32_t o = a2_off<N>(bl * C::NY + k0 + k, 2 * y);
          *reinterpret_cast<uint32_t*>(sm + L::A2 + o) = hi;
          *reinterpret_cast<uint32_t*>(sm + L::A2 + C::A2_BYTES + o) = lo;
        }
      }
    }
    tc::fence_async_smem();
    tc::fence_before_sync();
    __syncthreads();

    // 4. Step 2: D2 = A2 * B2^T, three passes.
    if (tid == 0) {
      tc::fence_after_sync();
      constexpr uint32_t id2 = tc::idesc_f16(128, C::N2);
      const uint32_t sbo_b = (C::K2 / 8) * 128;
      const uint32_t d = tmem + C::D2_COL;
      for (int ks = 0; ks < C::K2 / 16; ks++) {
        const uint64_t ah = a2_desc<N>(sbase + L::A2, ks);
        const uint64_t al = a2_desc<N>(sbase + L::A2 + C::A2_BYTES, ks);
        const uint64_t bh = tc::sdesc(sbase + L::B2 + ks * 256, 128, sbo_b, tc::LAYOUT_INTERLEAVE);
        const uint64_t bl = tc::sdesc(sbase + L::B2 + C::B2_BYTES + ks * 256, 128, sbo_b, tc::LAYOUT_INTERLEAVE);
        tc::mma_f16(d, ah, bh, id2, ks > 0);
        tc::mma_f16(d, ah, bl, id2, 1);
        tc::mma_f16(d, al, bh, id2, 1);
      }
      tc::mma_commit(&bar[1]);
    }

    // 5. The next group's operand and step 1 (every warp has read D1 above).
    if (grp + (int)gridDim.x < ngroups) begin_group(grp + gridDim.x);

    // Step 2 done: A2's space is free for the staging area.
    if (!__syncthreads_and(tc::mbar_wait(&bar[1], phase, kWaitNs))) {
      if (tid == 0) atomicOr(a.err, kErrWaitForward);
      break;
    }
    phase ^= 1;
    tc::fence_after_sync();

    // 6. D2 -> staging [block][ky][kx], scaled; column 0 holds the packed P.
    {
      const int s = warp & 3, h = warp >> 2;
      const int r2 = 32 * s + lane;
      const int bl = r2 / C::NY, kp = r2 % C::NY;
      float v[N];  // half of the N2 = 2N columns: NY values of ky, (re, im)
      tc::tmem_ld<N>(tmem + ((uint32_t)(32 * s) << 16) + C::D2_COL + N * h, v);
      float2* o = stage + bl * C::PS + kp;
#pragma unroll
      for (int j = 0; j < C::NY; j++) {
        const int ky = C::NY * h + j;
        o[ky * C::FBW] = make_float2(v[2 * j] * a.out_scale, v[2 * j + 1] * a.out_scale);
      }
    }
    __syncthreads();

    // 7. Unpack columns 0 and n/2; chroma offset.
    {
      const int bl = tid / N, ky = tid % N;
      float2* blk = stage + bl * C::PS;
      const float2 P = blk[ky * C::FBW], Q = blk[((N - ky) % N) * C::FBW];
      __syncwarp();
      // Both halves of a pair (ky, n-ky) sit in the same warp (N <= 32).
      blk[ky * C::FBW] = make_float2(0.5f * (P.x + Q.x), 0.5f * (P.y - Q.y));
      blk[ky * C::FBW + C::NY] = make_float2(0.5f * (P.y + Q.y), 0.5f * (Q.x - P.x));
      if (a.chroma_norm != 0.0f) {
        const float2* ws = reinterpret_cast<const float2*>(a.tab + T::WSPEC) + ky * C::FBW;
        for (int kx = 0; kx < C::FBW; kx++) {
          const float2 w = ws[kx];
          float2& z = blk[ky * C::FBW + kx];
          z.x -= a.chroma_norm * w.x;
          z.y -= a.chroma_norm * w.y;
        }
      }
    }
    // Half storage: the staged spectra narrowed to fp16 pairs in place (all
    // values read before any is written).
    if (a.half) {
      constexpr int PER = C::G * C::PS / kTcThreads;
      static_assert(C::G * C::PS % kTcThreads == 0, "staged values per thread");
      float2 r[PER];
      __syncthreads();
#pragma unroll
      for (int i = 0; i < PER; i++) r[i] = stage[tid + kTcThreads * i];
      __syncthreads();
      __half2* hs = reinterpret_cast<__half2*>(stage);
#pragma unroll
      for (int i = 0; i < PER; i++) hs[tid + kTcThreads * i] = __float22half2_rn(r[i]);
    }
    tc::fence_async_smem();
    __syncthreads();

    // 8. One bulk copy of the group's spectra to HBM.
    if (tid == 0 && nvalid > 0) {
      if (a.half)
        tc::bulk_store(reinterpret_cast<__half2*>(a.spec) + (size_t)b0 * C::PS, stage, (uint32_t)(nvalid * C::PS * 4));
      else
        tc::bulk_store(a.spec + (size_t)b0 * C::PS, stage, (uint32_t)(nvalid * C::PS * 8));
      tc::bulk_commit();
    }
  }
  if (tid == 0) tc::bulk_wait_read();  // the shared memory outlives the copies out of it
  stamp_end(B.p[0].clk);
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(tmem, C::TMEM_COLS);
}

// ---- sweep: filter, then inverse + overlap-add -------------------------------
//
// The tensor-core counterpart of the fast-form sweep (f3d_k_sweep.cu).
//
// k_filter_tc: the temporal filter (filter_vals, fast form) of every block's
// bins; the block's part of the column-inverse operand, rows k' (k' = 0
// packing the Hermitian parts of columns 0 and n/2 as H0 + i H(n/2)), scaled
// by kInvPre and split hi/lo, leaves as the block's image (BlkImg): the exact
// shared-memory bytes, so that the images of consecutive blocks are an operand
// tile.
//
// k_sweep_tc: the plane is cut into strips of TJ = 7 cells, covered by block
// columns J0..J0+7 (the last one the strip's right neighbour). One CTA per
// (strip, segment of block rows), per row:
//   the images of the row's 8 blocks arrive by one bulk copy (issued while the
//   previous row's transforms ran);
//   step 2': V[y][k'] = sum_ky e^(2 pi i ky y/n) sy[y] F[ky][k'] (tensor cores);
//   V: V into the row-inverse operand, rows (y, block slot) of two tiles
//      that hold the even and the odd block columns;
//   step 1': out[y][x] = sum_j V'[y][j] C1[x][j] with the even or odd
//      synthesis x-window (tensor cores), i.e. fft2dRealInverseHalf
//      (src/cpu/fft.cpp:88-119) times the synthesis window;
//   O: overlap-add from tensor memory into the cell partial sums in the
//      reference's block order (src/cpu/reference.cpp:415-436), finished cell
//      rows packed straight to the output plane; segment seams as in the
//      fast-form sweep.

// A block's operand image: rows k' = 0..n/2-1, K = 2 ky + (re, im), in 8-row
// atoms, each atom's hi part followed by its lo part, so that the atoms of
// consecutive blocks are evenly spaced. n = 32: two SWIZZLE_128B atoms of
// 1024 bytes; n = 16: one interleaved atom of 512.
template <int N>
struct BlkImg {
  static constexpr uint32_t BYTES = 4 * N * N;
  static constexpr uint32_t LO = N == 32 ? 1024 : 512;  // from a hi part to its lo part
  static constexpr uint32_t SBO = 2 * LO;               // from atom to atom
};
template <int N>
__host__ __device__ constexpr uint32_t img_off(int kp, int ky) {
  return (kp >> 3) * BlkImg<N>::SBO + (N == 32 ? tc::off_sw128(kp & 7, 2 * ky) : tc::off_il(kp & 7, 2 * ky, 2 * N));
}
// Descriptor of K-step ks (16 columns) of the hi parts of a tile of images at base.
template <int N>
__device__ __forceinline__ uint64_t img_desc(uint32_t base, int ks) {
  if constexpr (N == 32) return tc::sdesc(base + ks * 32, 16, BlkImg<N>::SBO, tc::LAYOUT_SW128);
  else return tc::sdesc(base + ks * 256, 128, BlkImg<N>::SBO, tc::LAYOUT_INTERLEAVE);
}

template <int N>
struct SwpCfg {
  using C = TcCfg<N>;
  static constexpr int TJ = C::G - 1;        // cells per strip
  static constexpr int CH = N / 2, CW = N / 2;
  static constexpr int PR = CW + 4;          // partial-sum row stride (floats), padded
  static constexpr int PC = CH * PR + 4;     // partial-sum cell stride (floats), padded
  static constexpr uint32_t TILE = C::G * BlkImg<N>::BYTES;          // operand tile: the images of a row's blocks
  // Inverse kernel shared memory.
  static constexpr uint32_t C2 = 0;                                  // hi, lo
  static constexpr uint32_t C1 = C2 + 2 * C::B2_BYTES;               // A hi, A lo, B hi, B lo
  static constexpr uint32_t A2 = (C1 + 4 * C::B1_BYTES + 1023) / 1024 * 1024;  // the operand tile
  // A1 shares A2's space: step 2' has read the operand tile before V writes
  // A1, and the next tile is loaded once step 1' has read A1. Three CTAs fit
  // on an SM.
  static constexpr uint32_t A1 = A2;                                 // [tile][hi, lo] (SWIZZLE_64B / 32B)
  static constexpr uint32_t A1_STRIDE = 2 * C::A1_BYTES;
  // The row of (y, slot) in the second tile, against the first: in V half the
  // lanes store to each tile, whose rows then fall in different banks.
  static constexpr int FLIP = N == 32 ? 1 : 2;
  static constexpr uint32_t P = A2 + TILE;                           // [2][TJ][PC] floats
  static constexpr uint32_t BAR = P + 2 * TJ * PC * 4;               // operand load, step 2', step 1'
  static constexpr uint32_t TSLOT = BAR + 24;
  static constexpr uint32_t BYTES = TSLOT + 8 + 1024;
  static_assert(C::T1 == 2, "one tile per block-column parity");
  static_assert(A1_STRIDE * C::T1 <= TILE, "the row-inverse operand fits in the operand tile's space");
  static_assert(A1_STRIDE % 512 == 0 && C::A1_BYTES % 512 == 0, "swizzle atoms");
  static_assert(BAR % 8 == 0 && P % 16 == 0, "alignment");
};

// Scale of a block sample after step 1': the inverse's 1/n^2 and kInvPre.
template <int N>
__host__ __device__ constexpr float out_scale() {
  return 1.0f / (kInvPre * N * N);
}

// Packs and stores samples x0 .. x0+W-1 (W = 8 or 16) of plane row y
// (bounds-checked), with 8- and 16-byte stores where the run is inside the
// plane and aligned.
template <int W>
__device__ __forceinline__ void emit_run(const SweepArgs& sa, int y, int x0, const float (&v)[W]) {
  static_assert(W == 8 || W == 16, "run width");
  if (y >= sa.inv.g.H) return;
  uint8_t* row = sa.dst + (long long)y * sa.pitch;
  const bool full = x0 + W <= sa.inv.g.W;
  if (full && sa.fmt == FMT_U16 && ((reinterpret_cast<uintptr_t>(row) + 2 * x0) & 15) == 0) {
    uint32_t w[W / 2];
#pragma unroll
    for (int k = 0; k < W / 2; k++)
      w[k] = pack_u16(v[2 * k] + sa.chroma_norm, sa.inv_norm, sa.max_pix) |
             (pack_u16(v[2 * k + 1] + sa.chroma_norm, sa.inv_norm, sa.max_pix) << 16);
    uint4* p = reinterpret_cast<uint4*>(row + 2 * x0);
#pragma unroll
    for (int k = 0; k < W / 8; k++) p[k] = make_uint4(w[4 * k], w[4 * k + 1], w[4 * k + 2], w[4 * k + 3]);
    return;
  }
  if (full && sa.fmt == FMT_U8 && ((reinterpret_cast<uintptr_t>(row) + x0) & (W - 1)) == 0) {
    uint32_t w[W / 4];
#pragma unroll
    for (int k = 0; k < W / 4; k++)
      w[k] = pack_u8(v[4 * k] + sa.chroma_norm) | (pack_u8(v[4 * k + 1] + sa.chroma_norm) << 8) |
             (pack_u8(v[4 * k + 2] + sa.chroma_norm) << 16) | (pack_u8(v[4 * k + 3] + sa.chroma_norm) << 24);
    if constexpr (W == 16) *reinterpret_cast<uint4*>(row + x0) = make_uint4(w[0], w[1], w[2], w[3]);
    else *reinterpret_cast<uint2*>(row + x0) = make_uint2(w[0], w[1]);
    return;
  }
#pragma unroll
  for (int k = 0; k < W; k++) {
    if (x0 + k >= sa.inv.g.W) break;
    float s = v[k];
    if (sa.chroma_norm != 0.0f) s += sa.chroma_norm;
    store_sample(row, x0 + k, s, sa.fmt, sa.inv_norm, sa.max_pix);
  }
}

// Bin j of a spectrum stored as float2 or, with half storage, as __half2.
template <bool HALF>
__device__ __forceinline__ float2 spec_at(const float2* s, size_t j) {
  if constexpr (HALF) return __half22float2(reinterpret_cast<const __half2*>(s)[j]);
  else return s[j];
}

// Filter kernel: one CTA per group of G consecutive blocks (8 of 32 x 32, 16
// of 16 x 16), whose spectra and images are contiguous. It is bound by the
// instructions per bin (75 % of the issue slots with ten outputs in a launch)
// and, with one output, by HBM (5.3 TB/s of reads and image writes). Each
// result goes straight to its place in the group's images, which leave by one
// bulk copy; the results of columns 0 and n/2 pass through `side`. Figures,
// 1080p 10-bit bt=4 with sharpen, ten outputs / one: 251 / 42.8 us with the
// switches read per bin and the results transposed through a buffer of
// filtered bins (131 instructions per bin), 173 / 36.1 us now (108).
template <int N>
struct FltCfg {
  using C = TcCfg<N>;
  static constexpr uint32_t IMG = BlkImg<N>::BYTES;
  static constexpr uint32_t SIDE = C::G * IMG;                   // float2 [G][2][N]: columns 0 and n/2
  static constexpr uint32_t DC = SIDE + C::G * 2 * N * 8;        // float [G]
  static constexpr uint32_t BYTES = DC + C::G * 4;
};

// One bin's result into the image at img (offset `at` of its hi part), or,
// of columns 0 and n/2, into side.
template <int N>
__device__ __forceinline__ void put_bin(uint8_t* img, float2* side, bool packed, uint32_t at, int side_at, float2 f) {
  if (packed) {
    side[side_at] = f;
  } else {
    uint32_t hi, lo;
    tc::split_pair(f.x * kInvPre, f.y * kInvPre, hi, lo);
    *reinterpret_cast<uint32_t*>(img + at) = hi;
    *reinterpret_cast<uint32_t*>(img + at + BlkImg<N>::LO) = lo;
  }
}

// The temporal filter (filter_vals, fast form) of a group's nvb blocks.
// Thread t filters bin li = t + 256 r (r < NL) of every block of the group,
// the bin's tables read once for all blocks, then tail item q: bin NL * 256 +
// e % TAIL of block e / TAIL, e = t + 256 q. The spectra loads of BATCH blocks
// are issued together; every index is the thread's base plus a constant.
template <int N, int BM, int BATCH, bool HALF>
__device__ __forceinline__ void filter_group(const FilterArgs& a, size_t gb0, int nvb, const float* dcs, uint8_t* img,
                                             float2* side, int tid) {
  using C = TcCfg<N>;
  constexpr int NF = BM >= 2 ? BM : 1;
  constexpr int NL = C::PS / kTcThreads;
  constexpr int TAIL = C::PS - NL * kTcThreads;
  constexpr int NT = TAIL * C::G / kTcThreads;
  static_assert((TAIL * C::G) % kTcThreads == 0, "tail bins per thread");
  static_assert(C::G % BATCH == 0, "load batches");
  const size_t gt = gb0 + tid;
  if constexpr (NL > 0) {
    BinTables tb[NL];
    uint32_t at[NL];
    int side_at[NL];
    bool packed[NL];
#pragma unroll
    for (int r = 0; r < NL; r++) {
      const int li = tid + kTcThreads * r, ky = li / C::FBW, kx = li - ky * C::FBW;
      tb[r] = bin_tables(a, li);
      at[r] = img_off<N>(kx & (C::NY - 1), ky);
      side_at[r] = (kx ? N : 0) + ky;
      packed[r] = kx == 0 || kx == C::NY;
    }
#pragma unroll
    for (int b0 = 0; b0 < C::G; b0 += BATCH) {
      float2 sv[BATCH][NL][4];
#pragma unroll
      for (int u = 0; u < BATCH; u++) {
        if (b0 + u >= nvb) continue;
#pragma unroll
        for (int r = 0; r < NL; r++)
#pragma unroll
          for (int k = 0; k < NF; k++)
            sv[u][r][k] = spec_at<HALF>(a.s[k], gt + (size_t)(b0 + u) * C::PS + kTcThreads * r);
      }
#pragma unroll
      for (int u = 0; u < BATCH; u++) {
        const int b = b0 + u;
        if (b >= nvb) continue;
        const float dc = dcs[b];
#pragma unroll
        for (int r = 0; r < NL; r++)
          put_bin<N>(img + b * BlkImg<N>::BYTES, side + b * 2 * N, packed[r], at[r], side_at[r],
                     filter_vals_t<BM, true>(a, dc, tb[r], 0, sv[u][r]));
      }
    }
  }
#pragma unroll
  for (int q = 0; q < NT; q++) {
    const int e = tid + kTcThreads * q;
    const int b = e / TAIL, li = NL * kTcThreads + e % TAIL;
    if (b >= nvb) continue;
    const int ky = li / C::FBW, kx = li - ky * C::FBW;
    float2 sv[4];
#pragma unroll
    for (int k = 0; k < NF; k++) sv[k] = spec_at<HALF>(a.s[k], gb0 + (size_t)b * C::PS + li);
    put_bin<N>(img + b * BlkImg<N>::BYTES, side + b * 2 * N, kx == 0 || kx == C::NY, img_off<N>(kx & (C::NY - 1), ky),
               (kx ? N : 0) + ky, filter_vals_t<BM, true>(a, dcs[b], bin_tables(a, li), 0, sv));
  }
}

template <int N, int BM, int MINB, int SW, bool HALF>
__global__ void __launch_bounds__(kTcThreads, MINB) k_filter_tc(const __grid_constant__ FilterBatch B) {
  using C = TcCfg<N>;
  using K = FltCfg<N>;
  constexpr int NF = BM >= 2 ? BM : 1;  // window frames read
  constexpr uint32_t BLK = C::PS * (HALF ? 4 : 8);
  // A run of planes of one geometry (e.g. consecutive frames of a plane)
  // runs the same group of each of its planes back to back, so that the
  // window spectra they share are read from L2 the second time.
  const int r0 = B.run[plane_of(B, B.cta0, blockIdx.x)];
  const int rl = B.rlen[r0];
  const int local = (int)blockIdx.x - B.cta0[r0];
  const int pl = r0 + local % rl;
  const FilterPlane& P = B.p[pl];
  // One plane: the sweep starts as this kernel's CTAs end. At once, its CTAs
  // take the first places that come free, crowded on few SMs (360p 8-bit bt=3
  // 29.1 us, else 27.9; 4K 10-bit bt=4 249, else 237). In a batch the planes'
  // CTAs spread by themselves and the early start pays (three 1080p planes
  // 110 -> 106 us, sixteen at 360p 97 -> 94).
  const bool late = B.n == 1;
  if (!late) grid_go();
  grid_wait();
  stamp_start(B.clk);
  FilterArgs a = P.f;
  fix_switches<SW>(a);
  extern __shared__ __align__(128) uint8_t smem_f[];
  float2* side = reinterpret_cast<float2*>(smem_f + K::SIDE);
  float* dcs = reinterpret_cast<float*>(smem_f + K::DC);
  const int tid = threadIdx.x;
  const int b0 = local / rl * C::G, nvb = min(C::G, P.nblk - b0);
  const size_t gb0 = (size_t)b0 * C::PS;
  // The window spectra begin moving into L2 as whole runs (of shifted
  // windows, only the newest frame: the others are an earlier output's). With
  // one output of a large plane a fifth is read twice (4K bt=4: 680 MB of 573),
  // probably because that is more than L2 keeps: five CTAs on 152 SMs ask for
  // 106 MB beside 25 MB of images.
  if (tid < NF && (!((B.shifted >> pl) & 1) || tid == NF - 1))
    tc::prefetch_l2(reinterpret_cast<const uint8_t*>(P.f.s[tid]) + b0 * (size_t)BLK, nvb * BLK);
  // The current frame's DC of each block (the degrid correction's scale).
  if (tid < nvb) dcs[tid] = a.dg ? spec_at<HALF>(P.f.s[P.f.cur], (size_t)(b0 + tid) * C::PS).x : 0.0f;
  __syncthreads();
  filter_group<N, BM, MINB >= 5 ? 1 : 2, HALF>(a, gb0, nvb, dcs, smem_f, side, tid);
  __syncthreads();
  {  // Row k' = 0 of block tid / N: the Hermitian parts of columns 0 and n/2, H0 + i H(n/2).
    const int ky = tid % N, kym = (N - ky) & (N - 1);
    const float2* f0 = side + tid / N * 2 * N;
    const float2* fn = f0 + N;
    const float2 p = f0[ky], pm = f0[kym], n = fn[ky], nm = fn[kym];
    const float h0x = 0.5f * (p.x + pm.x), h0y = 0.5f * (p.y - pm.y);
    const float hnx = 0.5f * (n.x + nm.x), hny = 0.5f * (n.y - nm.y);
    put_bin<N>(smem_f + tid / N * K::IMG, nullptr, false, img_off<N>(0, ky), 0, make_float2(h0x - hny, h0y + hnx));
  }
  tc::fence_async_smem();
  __syncthreads();
  if (tid == 0) {
    tc::bulk_store(P.img + (size_t)b0 * K::IMG, smem_f, nvb * K::IMG);
    tc::bulk_commit();
    tc::bulk_wait_read();
  }
  if (late) grid_go();
  stamp_end(B.clk);
}

// Shared-memory and barrier state of the inverse phases of one CTA.
struct InvState {
  uint8_t* sm;
  uint32_t sbase;
  uint64_t* bar;  // [1] column-inverse products, [2] row-inverse products
  uint32_t tmem;
  uint32_t phase;
  float* P_old;   // cell partial sums of block row m - 1 (finished by this row's top halves)
  float* P_new;   // cell partial sums of block row m
};

// The inverse of block row m once its operand tile is in shared memory (A2):
// step 2' (column inverse, tensor cores), V, step 1' (row inverse with the
// synthesis windows, tensor cores), then `after` (the tile's space is free
// again), then O (overlap-add in the reference's block order, finished cell
// rows packed to the output, segment seams). Returns false when a wait gave
// up (the error word has its bit); every thread of the CTA returns the same.
template <int N, class After>
__device__ __forceinline__ bool inverse_row(const SweepArgs& sa, InvState& st, int m, int M0, int M1, int seg, int J0,
                                            int ncell, After after) {
  using C = TcCfg<N>;
  using S = SwpCfg<N>;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint8_t* sm = st.sm;
  const uint32_t sbase = st.sbase;
  uint64_t* bar = st.bar;
  const uint32_t tmem = st.tmem;
  if (tid == 0) {
    tc::fence_after_sync();
    constexpr uint32_t id2 = tc::idesc_f16(128, C::N2);
    const uint32_t sbo_b = (C::K2 / 8) * 128;
    const uint32_t d = tmem + C::D2_COL;
    for (int ks = 0; ks < C::K2 / 16; ks++) {
      const uint64_t ah = img_desc<N>(sbase + S::A2, ks);
      const uint64_t al = img_desc<N>(sbase + S::A2 + BlkImg<N>::LO, ks);
      const uint64_t bh = tc::sdesc(sbase + S::C2 + ks * 256, 128, sbo_b, tc::LAYOUT_INTERLEAVE);
      const uint64_t bl = tc::sdesc(sbase + S::C2 + C::B2_BYTES + ks * 256, 128, sbo_b, tc::LAYOUT_INTERLEAVE);
      tc::mma_f16(d, ah, bh, id2, ks > 0);
      tc::mma_f16(d, ah, bl, id2, 1);
      tc::mma_f16(d, al, bh, id2, 1);
    }
    tc::mma_commit(&bar[1]);
  }
  if (!__syncthreads_and(tc::mbar_wait(&bar[1], st.phase, kWaitNs))) {
    if (tid == 0) atomicOr(sa.err, kErrWaitColumn);
    return false;
  }
  tc::fence_after_sync();

  // V. Row-inverse operand: tile = parity of the block column, row (y, slot).
  {
    const int s = warp & 3, h = warp >> 2;
    const int r2 = 32 * s + lane;
    const int kp = r2 % C::NY, bl = r2 / C::NY;
    const int tile = (J0 + bl) & 1, slot = (bl >> 1) ^ (tile ? S::FLIP : 0);
    uint8_t* t0 = sm + S::A1 + tile * S::A1_STRIDE;
    float v[N];  // half of the N2 = 2N columns: NY values of y, (re, im)
    tc::tmem_ld<N>(tmem + ((uint32_t)(32 * s) << 16) + C::D2_COL + N * h, v);
#pragma unroll
    for (int j = 0; j < C::NY; j++) {
      const int y = C::NY * h + j;
      uint32_t hi, lo;
      tc::split_pair(v[2 * j], v[2 * j + 1], hi, lo);
      const uint32_t o = tc::off_sw_k<C::K1>((C::G / 2) * y + slot, 2 * kp);
      *reinterpret_cast<uint32_t*>(t0 + o) = hi;
      *reinterpret_cast<uint32_t*>(t0 + C::A1_BYTES + o) = lo;
    }
  }
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();

  // Step 1' on the tensor cores: D1[tile] = A1[tile] * C1(tile)^T.
  if (tid == 0) {
    tc::fence_after_sync();
    constexpr uint32_t id1 = tc::idesc_f16(128, C::N1);
    const uint32_t sbo = (C::K1 / 8) * 128;
    for (int t = 0; t < C::T1; t++) {
      const uint32_t a_hi = sbase + S::A1 + t * S::A1_STRIDE, a_lo = a_hi + C::A1_BYTES;
      const uint32_t b_hi = sbase + S::C1 + t * 2 * C::B1_BYTES, b_lo = b_hi + C::B1_BYTES;
      const uint32_t d = tmem + C::D1_COL + t * C::N1;
      for (int ks = 0; ks < C::K1 / 16; ks++) {
        const uint64_t ah = tc::sdesc(a_hi + ks * 32, 16, 16 * N, N == 32 ? tc::LAYOUT_SW64 : tc::LAYOUT_SW32);
        const uint64_t al = tc::sdesc(a_lo + ks * 32, 16, 16 * N, N == 32 ? tc::LAYOUT_SW64 : tc::LAYOUT_SW32);
        const uint64_t bh = tc::sdesc(b_hi + ks * 256, 128, sbo, tc::LAYOUT_INTERLEAVE);
        const uint64_t bl = tc::sdesc(b_lo + ks * 256, 128, sbo, tc::LAYOUT_INTERLEAVE);
        tc::mma_f16(d, ah, bh, id1, ks > 0);
        tc::mma_f16(d, ah, bl, id1, 1);
        tc::mma_f16(d, al, bh, id1, 1);
      }
    }
    tc::mma_commit(&bar[2]);
  }
  if (!__syncthreads_and(tc::mbar_wait(&bar[2], st.phase, kWaitNs))) {
    if (tid == 0) atomicOr(sa.err, kErrWaitRow);
    return false;
  }
  st.phase ^= 1;
  tc::fence_after_sync();
  after();

  // O. Overlap-add. Thread: block row y of block bl; y < n/2 finishes cell
  // row m-1 (P_old), y >= n/2 starts cell row m (P_new).
  float* P_old = st.P_old;
  float* P_new = st.P_new;
  {
    const int t = warp >> 2, s = warp & 3;
    const int r = 32 * s + lane;
    const int y = r / (C::G / 2), slot = r % (C::G / 2);
    const int bl = 2 * (slot ^ (t ? S::FLIP : 0)) + ((t ^ J0) & 1);
    float v[N];
    tc::tmem_ld<N>(tmem + ((uint32_t)(32 * s) << 16) + C::D1_COL + t * C::N1, v);
#pragma unroll
    for (int x = 0; x < N; x++) v[x] *= out_scale<N>();
    const bool top = y < S::CH;
    const int yy = top ? y : y - S::CH;
    const bool right_ok = bl < ncell;                // right half -> cell bl
    const bool left_ok = bl >= 1 && bl - 1 < ncell;  // left half -> cell bl-1
    const bool seam_top = m == M0;                   // cell row m-1 is another segment's (or none)
    if (top) {
      if (seam_top) {
        if (M0 > 0 && right_ok) {
          float* t0 = sa.seam_t + ((size_t)((seg - 1) * 2) * S::CH + yy) * sa.seam_w + (J0 + bl) * S::CW;
#pragma unroll
          for (int x = 0; x < S::CW; x += 4)
            *reinterpret_cast<float4*>(t0 + x) = make_float4(v[S::CW + x], v[S::CW + x + 1], v[S::CW + x + 2], v[S::CW + x + 3]);
        }
      } else if (right_ok) {
        float* p = P_old + bl * S::PC + yy * S::PR;
#pragma unroll
        for (int x = 0; x < S::CW; x += 4) {
          float4 q = *reinterpret_cast<float4*>(p + x);
          q.x += v[S::CW + x], q.y += v[S::CW + x + 1], q.z += v[S::CW + x + 2], q.w += v[S::CW + x + 3];
          *reinterpret_cast<float4*>(p + x) = q;
        }
      }
    } else if (right_ok) {
      float* p = P_new + bl * S::PC + yy * S::PR;
#pragma unroll
      for (int x = 0; x < S::CW; x += 4)
        *reinterpret_cast<float4*>(p + x) = make_float4(v[S::CW + x], v[S::CW + x + 1], v[S::CW + x + 2], v[S::CW + x + 3]);
    }
    __syncthreads();
    if (top) {
      if (seam_top) {
        if (M0 > 0 && left_ok) {
          float* t1 = sa.seam_t + ((size_t)((seg - 1) * 2 + 1) * S::CH + yy) * sa.seam_w + (J0 + bl - 1) * S::CW;
#pragma unroll
          for (int x = 0; x < S::CW; x += 4)
            *reinterpret_cast<float4*>(t1 + x) = make_float4(v[x], v[x + 1], v[x + 2], v[x + 3]);
        }
      } else if (left_ok) {
        const float* p = P_old + (bl - 1) * S::PC + yy * S::PR;
        float o[S::CW];
#pragma unroll
        for (int x = 0; x < S::CW; x += 4) {
          const float4 q = *reinterpret_cast<const float4*>(p + x);
          o[x] = q.x + v[x], o[x + 1] = q.y + v[x + 1], o[x + 2] = q.z + v[x + 2], o[x + 3] = q.w + v[x + 3];
        }
        emit_run<S::CW>(sa, (m - 1) * S::CH + yy, (J0 + bl - 1) * S::CW, o);
      }
    } else if (left_ok) {
      float* p = P_new + (bl - 1) * S::PC + yy * S::PR;
      const bool seam_bot = m == M1 - 1 && seg < sa.segs - 1;
      float* sb = sa.seam_b + ((size_t)seg * S::CH + yy) * sa.seam_w + (J0 + bl - 1) * S::CW;
#pragma unroll
      for (int x = 0; x < S::CW; x += 4) {
        float4 q = *reinterpret_cast<float4*>(p + x);
        q.x += v[x], q.y += v[x + 1], q.z += v[x + 2], q.w += v[x + 3];
        if (seam_bot) *reinterpret_cast<float4*>(sb + x) = q;
        else *reinterpret_cast<float4*>(p + x) = q;
      }
    }
  }
  st.P_old = P_new;
  st.P_new = P_old;
  tc::fence_before_sync();
  __syncthreads();
  return true;
}

// Constant operands of the inverse (C2 hi, lo, then C1 A hi, lo, B hi, lo)
// into shared memory, and tensor memory.
template <int N>
__device__ __forceinline__ void inverse_setup(const SweepArgs& sa, uint8_t* sm, uint32_t* tslot) {
  using C = TcCfg<N>;
  using S = SwpCfg<N>;
  using T = TcTab<N>;
  const int tid = threadIdx.x;
  const uint4* src2 = reinterpret_cast<const uint4*>(sa.tab + T::C2HI);
  uint4* dst2 = reinterpret_cast<uint4*>(sm + S::C2);
  for (int i = tid; i < (int)(2 * C::B2_BYTES / 16); i += kTcThreads) dst2[i] = src2[i];
  const uint4* src1 = reinterpret_cast<const uint4*>(sa.tab + T::C1AHI);
  uint4* dst1 = reinterpret_cast<uint4*>(sm + S::C1);
  for (int i = tid; i < (int)(4 * C::B1_BYTES / 16); i += kTcThreads) dst1[i] = src1[i];
  if ((tid >> 5) == 0) {
    tc::tmem_alloc(tslot, C::TMEM_COLS);
    tc::tmem_relinquish();
  }
}

template <int N>
__global__ void __launch_bounds__(kTcThreads, kTcSweepCtasPerSm) k_sweep_tc(const __grid_constant__ SweepBatch B) {
  using C = TcCfg<N>;
  using S = SwpCfg<N>;
  static_assert(sizeof(B) <= 32000, "kernel parameter space");
  extern __shared__ __align__(1024) uint8_t smem_raw[];
  uint8_t* sm = smem_raw + ((1024u - (tc::smem_u32(smem_raw) & 1023u)) & 1023u);
  uint64_t* bar = reinterpret_cast<uint64_t*>(sm + S::BAR);  // [0] operand load, [1] step 2', [2] step 1'
  uint32_t* tslot = reinterpret_cast<uint32_t*>(sm + S::TSLOT);
  const int tid = threadIdx.x, warp = tid >> 5;

  const int pl = plane_of(B, B.cta0, blockIdx.x);
  const SweepArgs& sa = B.p[pl];
  const int cta = blockIdx.x - B.cta0[pl];
  const int strip = cta % sa.strips, seg = cta / sa.strips;
  const int J0 = strip * S::TJ;
  const int nrow = sa.cells_y + 1;
  const int M0 = (int)((long long)seg * nrow / sa.segs);
  const int M1 = (int)((long long)(seg + 1) * nrow / sa.segs);
  const int ncell = min(S::TJ, sa.cells_x - J0);
  // Operand tile of row m: the images of the strip's blocks (the last strip
  // may have fewer; the operand rows of the others are never looked at).
  auto tile_of = [&](int m) { return sa.img + ((size_t)m * sa.inv.g.ncols + J0) * BlkImg<N>::BYTES; };
  const uint32_t tile_bytes = (ncell + 1) * BlkImg<N>::BYTES;

  if (tid == 0) {
    for (int i = 0; i < 3; i++) tc::mbar_init(&bar[i], 1);
    tc::fence_mbar_init();
  }
  inverse_setup<N>(sa, sm, tslot);
  tc::fence_async_smem();
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  grid_go();
  grid_wait();
  stamp_start(B.p[0].clk2);
  if (tid == 0 && M0 < M1) {
    tc::mbar_expect_tx(&bar[0], tile_bytes);
    // A test of the bounded wait leaves this copy out: nothing is then in
    // flight on the barrier, the wait below gives up and the CTA leaves.
    if (!(sa.test_skip && cta == 0)) tc::bulk_load(sm + S::A2, tile_of(M0), tile_bytes, &bar[0]);
  }
  InvState st{sm, tc::smem_u32(sm), bar, *tslot, 0u, reinterpret_cast<float*>(sm + S::P),
              reinterpret_cast<float*>(sm + S::P) + S::TJ * S::PC};

  for (int m = M0; m < M1; m++) {
    // The operand tile of row m arrives by bulk copy (issued while the
    // previous row's overlap-add ran).
    if (!__syncthreads_and(tc::mbar_wait(&bar[0], st.phase, kWaitNs))) {
      if (tid == 0) atomicOr(sa.err, kErrWaitTile);
      break;
    }
    // A1 (the operand tile's space) is consumed once step 1' is done: the
    // next row's tile starts moving in while the overlap-add runs.
    const bool ok = inverse_row<N>(sa, st, m, M0, M1, seg, J0, ncell, [&] {
      if (tid == 0 && m + 1 < M1) {
        tc::mbar_expect_tx(&bar[0], tile_bytes);
        tc::bulk_load(sm + S::A2, tile_of(m + 1), tile_bytes, &bar[0]);
      }
    });
    if (!ok) break;
  }
  tc::fence_before_sync();
  __syncthreads();
  tc::fence_after_sync();
  if (warp == 0) tc::tmem_dealloc(st.tmem, C::TMEM_COLS);
  // The partial sums are done with: two ints of them for the seams.
  finish_seams<S::CH, S::CW>(sa, strip, seg, J0, ncell, reinterpret_cast<int*>(sm + S::P));
  stamp_end(B.p[0].clk2);
}

template <class K>
cudaError_t prepare(K k, size_t smem) {
  return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// Host-side fp16 hi/lo split of a double.
void split_h(double v, __half& hi, __half& lo) {
  hi = __float2half_rn((float)v);
  lo = __float2half_rn((float)(v - (double)__half2float(hi)));
}
void put_pair(std::vector<uint8_t>& t, uint32_t hi_base, uint32_t lo_base, uint32_t off, double v) {
  __half h, l;
  split_h(v, h, l);
  std::memcpy(t.data() + hi_base + off, &h, 2);
  std::memcpy(t.data() + lo_base + off, &l, 2);
}

template <int N>
std::vector<uint8_t> tables_n(const std::vector<double>& wx, const std::vector<double>& wy,
                              const std::vector<double>& sxa, const std::vector<double>& sxb,
                              const std::vector<double>& sy) {
  using T = TcTab<N>;
  constexpr int NY = N / 2, FBW = NY + 1;
  std::vector<uint8_t> t(T::TOTAL, 0);
  auto cs = [](int k, int x, double& c, double& s) {
    const double th = 2.0 * kPiD * (double)((k * x) % N) / N;
    c = std::cos(th);
    s = std::sin(th);
  };
  // Packed real row transform coefficient j at x: 1, (-1)^x, cos, -sin.
  auto row_coef = [&](int j, int x) {
    if (j == 0) return 1.0;
    if (j == 1) return (x & 1) ? -1.0 : 1.0;
    double c, s;
    cs(j / 2, x, c, s);
    return (j & 1) ? -s : c;
  };
  // B1 [j][x]: packed real row DFT, analysis x-window folded in.
  for (int j = 0; j < N; j++)
    for (int x = 0; x < N; x++) put_pair(t, T::B1HI, T::B1LO, tc::off_il(j, x, N), row_coef(j, x) * wx[x]);
  // B2 [2ky+ro][2y+ri]: complex column DFT, analysis y-window folded in.
  for (int ky = 0; ky < N; ky++)
    for (int y = 0; y < N; y++) {
      double c, s;
      cs(ky, y, c, s);
      const double w = wy[y];
      put_pair(t, T::B2HI, T::B2LO, tc::off_il(2 * ky, 2 * y, 2 * N), w * c);
      put_pair(t, T::B2HI, T::B2LO, tc::off_il(2 * ky, 2 * y + 1, 2 * N), w * s);
      put_pair(t, T::B2HI, T::B2LO, tc::off_il(2 * ky + 1, 2 * y, 2 * N), -w * s);
      put_pair(t, T::B2HI, T::B2LO, tc::off_il(2 * ky + 1, 2 * y + 1, 2 * N), w * c);
    }
  // Spectrum of the analysis window (the chroma offset's contribution): the
  // window is separable, so it is the product of the two axes' DFTs.
  std::vector<double> ayr(N), ayi(N), axr(FBW), axi(FBW);
  for (int k = 0; k < N; k++)
    for (int j = 0; j < N; j++) {
      double c, s;
      cs(k, j, c, s);
      ayr[k] += wy[j] * c;
      ayi[k] -= wy[j] * s;
      if (k < FBW) {
        axr[k] += wx[j] * c;
        axi[k] -= wx[j] * s;
      }
    }
  for (int ky = 0; ky < N; ky++)
    for (int kx = 0; kx < FBW; kx++) {
      const float f[2] = {(float)(ayr[ky] * axr[kx] - ayi[ky] * axi[kx]),
                          (float)(ayr[ky] * axi[kx] + ayi[ky] * axr[kx])};
      std::memcpy(t.data() + T::WSPEC + (ky * FBW + kx) * 8, f, 8);
    }
  // C2 [2y+ro][2ky+ri]: complex column inverse DFT (unnormalised), synthesis
  // y-window folded in.
  for (int y = 0; y < N; y++)
    for (int ky = 0; ky < N; ky++) {
      double c, s;
      cs(ky, y, c, s);
      const double w = sy[y];
      put_pair(t, T::C2HI, T::C2LO, tc::off_il(2 * y, 2 * ky, 2 * N), w * c);
      put_pair(t, T::C2HI, T::C2LO, tc::off_il(2 * y, 2 * ky + 1, 2 * N), -w * s);
      put_pair(t, T::C2HI, T::C2LO, tc::off_il(2 * y + 1, 2 * ky, 2 * N), w * s);
      put_pair(t, T::C2HI, T::C2LO, tc::off_il(2 * y + 1, 2 * ky + 1, 2 * N), w * c);
    }
  // C1 [x][j]: real row inverse from the packed half spectrum (twice the
  // cos/sin terms: the mirrored columns), synthesis x-window folded in.
  for (int x = 0; x < N; x++)
    for (int j = 0; j < N; j++) {
      const double v = j < 2 ? row_coef(j, x) : 2.0 * row_coef(j, x);
      put_pair(t, T::C1AHI, T::C1ALO, tc::off_il(x, j, N), v * sxa[x]);
      put_pair(t, T::C1BHI, T::C1BLO, tc::off_il(x, j, N), v * sxb[x]);
    }
  return t;
}

}  // namespace

bool tc_supported(int mode, int bw, int bh, int bm) {
  return mode == 1 && bw == bh && (bw == 16 || bw == 32) && bm != 0;
}

int tc_group_blocks(int n) { return 128 / (n / 2); }
int tc_sweep_cells(int n) { return tc_group_blocks(n) - 1; }

static_assert(TcCfg<32>::G == 8 && TcCfg<16>::G == 16, "forward group sizes of the batch plan");

std::vector<uint8_t> tc_tables(int n, const std::vector<double>& wx, const std::vector<double>& wy,
                               const std::vector<double>& sxa, const std::vector<double>& sxb,
                               const std::vector<double>& sy) {
  for (const auto* v : {&wx, &wy, &sxa, &sxb, &sy})
    if ((int)v->size() != n) return {};
  if (n == 32) return tables_n<32>(wx, wy, sxa, sxb, sy);
  if (n == 16) return tables_n<16>(wx, wy, sxa, sxb, sy);
  return {};
}

namespace {

template <int N, bool ALIGNED>
void (*forward_kernel(int fmt, bool split))(TcFwdBatch) {
  return fmt == FMT_U8 ? k_forward_tc<N, 1, false, ALIGNED>
         : fmt == FMT_U16 ? (split ? k_forward_tc<N, 2, true, ALIGNED> : k_forward_tc<N, 2, false, ALIGNED>)
                          : k_forward_tc<N, 4, true, ALIGNED>;
}
// Whether the blocks of a plane start on 16 bytes in every row.
bool rows_aligned(const TcFwdArgs& a, int bps) {
  return ((reinterpret_cast<uintptr_t>(a.src) | (uintptr_t)a.pitch | (uintptr_t)(a.g.xoff * bps) |
           (uintptr_t)(a.g.xstep * bps)) & 15) == 0;
}

// The forward launch of a batch of planes of one sample format: the split
// kernel (hi + lo step-1 operand) where any plane needs it; it takes the others
// too. Null where there is none.
struct FwdLaunch {
  void (*kernel)(TcFwdBatch) = nullptr;
  size_t smem = 0;
  int ctas = 0;  // per SM
};
// Shared memory of which no more than `ctas` CTAs fit on an SM (228 KB, 1 KB of
// it for each CTA).
constexpr size_t smem_for_ctas(int ctas) { return 228 * 1024 / (ctas + 1) - 1024 + 128; }

// Whether one plane's forward of 16 x 16 blocks asks for that much: its
// persistent CTAs are placed where the kernel ahead leaves room first, and where
// an SM holds more of them than the grid is meant to put there (8-bit 4 for 3,
// 16-bit at two an SM 3; 10-bit and float no more), the first SMs to come free took
// more and others were left with fewer. It pays once a CTA has a group and a
// half: queued passes, bt=4, before the kernels overlapped / overlapped / now: 4K
// 16-bit 293, 292, 266 us, 8-bit 327, 275, 256; 7680x4320 16-bit 1004, 1058, 940;
// 1080p 16-bit 111, 93, 87; 720p 8-bit 74, 49.3, 48.3 (932 groups for 456 CTAs).
// With fewer groups each has one and crowding costs nothing (960x540 8-bit, 534:
// 33.2 us, else 34.1). In a batch of several planes the forward shares the SMs
// with another kernel and takes what is there (8-bit 1080p, sixteen outputs: 769
// us, else 784).
bool spread_ctas(int n_planes, int fmt, int ctas, int groups) {
  return n_planes == 1 && (fmt == FMT_U8 || (fmt == FMT_U16 && ctas == 2)) && 2 * groups >= 3 * ctas * sm_count();
}

template <int N>
FwdLaunch forward_launch_n(const TcFwdArgs* planes, int n) {
  FwdLaunch l;
  const int fmt = planes[0].fmt;
  const bool aligned = tc_rows_aligned(planes, n);
  bool split = false;
  for (int i = 0; i < n; i++) split = split || planes[i].split;
  if (fmt == FMT_U8 && split) return l;
  l.kernel = aligned ? forward_kernel<N, true>(fmt, split) : forward_kernel<N, false>(fmt, split);
  l.smem = split ? FwdSmem<N, true>::BYTES : FwdSmem<N, false>::BYTES;
  l.ctas = fwd_ctas(split, aligned, fmt == FMT_U16 ? 2 : 1);
  if (N == 16 && spread_ctas(n, fmt, l.ctas, (planes[0].g.nb + TcCfg<N>::G - 1) / TcCfg<N>::G))
    l.smem = std::max(l.smem, smem_for_ctas(l.ctas));
  return l;
}
FwdLaunch forward_launch(const TcFwdArgs* planes, int n) {
  return planes[0].g.bw == 16 ? forward_launch_n<16>(planes, n) : forward_launch_n<32>(planes, n);
}

}  // namespace

bool tc_rows_aligned(const TcFwdArgs* planes, int n) {
  const int bps = planes[0].fmt == FMT_U8 ? 1 : (planes[0].fmt == FMT_U16 ? 2 : 4);
  for (int i = 0; i < n; i++)
    if (!rows_aligned(planes[i], bps)) return false;
  return true;
}

cudaError_t launch_forward_tc_batch(const TcFwdArgs* planes, int n, const TcTune& t, cudaStream_t st) {
  TcFwdBatch B;
  if (!forward_batch(planes, n, B)) return n < 1 || n > kMaxBatch ? cudaErrorInvalidValue : cudaErrorNotSupported;
  const FwdLaunch l = forward_launch(planes, n);
  if (!l.kernel) return cudaErrorNotSupported;
  const cudaError_t attr = prepare(l.kernel, l.smem);
  if (attr != cudaSuccess) return attr;
  const int ngroups = B.grp0[n];
  if (ngroups == 0) return cudaSuccess;
  static_assert(kFwdMaxCtasPerSm * (FwdSmem<32, false>::BYTES + 1024) <= 228 * 1024, "CTAs per SM");
  static_assert(2 * (FwdSmem<32, true>::BYTES + 1024) <= 228 * 1024, "CTAs per SM");
  const int per_sm = std::max(1, std::min(t.fwd_ctas_per_sm, l.ctas));
  const int grid = std::min(ngroups, per_sm * sm_count());
  return launch_kernel(l.kernel, grid, kTcThreads, l.smem, st, B);
}

cudaError_t launch_forward_tc(const TcFwdArgs& a, cudaStream_t st) { return launch_forward_tc_batch(&a, 1, TcTune{}, st); }

namespace {

template <int N, int BM, int MINB, int SW>
const void* filter_kernel_h(bool half) {
  return half ? (const void*)k_filter_tc<N, BM, MINB, SW, true> : (const void*)k_filter_tc<N, BM, MINB, SW, false>;
}
template <int N, int MINB, int SW>
const void* filter_kernel_bm(int bm, bool half) {
  switch (bm) {
  case -1: return filter_kernel_h<N, -1, MINB, SW>(half);
  case 1: return filter_kernel_h<N, 1, MINB, SW>(half);
  case 2: return filter_kernel_h<N, 2, MINB, SW>(half);
  case 3: return filter_kernel_h<N, 3, MINB, SW>(half);
  case 4: return filter_kernel_h<N, 4, MINB, SW>(half);
  default: return nullptr;
  }
}
template <int N, int MINB>
const void* filter_kernel_n(int sw, int bm, bool half) {
  return sw == kSwPlain     ? filter_kernel_bm<N, MINB, kSwPlain>(bm, half)
         : sw == kSwSharpen ? filter_kernel_bm<N, MINB, kSwSharpen>(bm, half)
                            : filter_kernel_bm<N, MINB, kSwAny>(bm, half);
}
template <int N>
const void* filter_kernel(int minb, int sw, int bm, bool half) {
  return minb >= 5 ? filter_kernel_n<N, 5>(sw, bm, half) : filter_kernel_n<N, 4>(sw, bm, half);
}

// The filter launch of a batch (one CTA per group of blocks).
struct FilterLaunch {
  const void* kernel = nullptr;
  int grid = 0;
  size_t smem = 0;
};
FilterLaunch filter_launch(const SweepBatch& S, int minb, FilterBatch& F) {
  const bool n16 = S.p[0].inv.g.bw == 16;
  FilterLaunch l;
  l.grid = filter_batch(S, n16 ? TcCfg<16>::G : TcCfg<32>::G, F);
  const int sw = filter_switches(S), bm = S.p[0].inv.bm;
  const bool half = S.p[0].inv.half;  // the planes store their spectra alike (sweep_batches checks)
  l.kernel = n16 ? filter_kernel<16>(minb, sw, bm, half) : filter_kernel<32>(minb, sw, bm, half);
  l.smem = n16 ? FltCfg<16>::BYTES : FltCfg<32>::BYTES;
  return l;
}

}  // namespace

namespace {

template <int N>
cudaError_t launch_sweep_n(const SweepBatch& B, int n, const TcTune& t, cudaStream_t st, cudaEvent_t after_filter) {
  using S = SwpCfg<N>;
  constexpr size_t smem = S::BYTES;
  static_assert(kTcSweepCtasPerSm * (S::BYTES + 1024) <= 228 * 1024, "CTAs per SM");
  FilterBatch F;
  const FilterLaunch l = filter_launch(B, t.filter_minb, F);
  if (!l.kernel) return cudaErrorNotSupported;
  cudaError_t e = cudaSuccess;
  if (l.grid > 0) {
    e = prepare(l.kernel, l.smem);
    if (e != cudaSuccess) return e;
    void* args[1] = {&F};
    e = launch_kernel(l.kernel, l.grid, kTcThreads, l.smem, st, args);
    if (e != cudaSuccess) return e;
  }
  if (after_filter && (e = cudaEventRecord(after_filter, st)) != cudaSuccess) return e;
  // Inverse + overlap-add: one CTA per (strip, segment) of every plane. It
  // starts within the filter but behind a batch's long one, where what is saved
  // is little and its waiting CTAs cost more (ten 10-bit 4K outputs, 41,140
  // filter CTAs: 1404 us, else 1388; three 1080p planes, 1,597: 106, else 108;
  // nothing between them was measured, so the line at eight waves is a choice).
  const bool overlap = n == 1 || l.grid <= 8 * 5 * sm_count();
  e = prepare(k_sweep_tc<N>, smem);
  if (e != cudaSuccess) return e;
  return launch_kernel(k_sweep_tc<N>, B.cta0[n], kTcThreads, smem, st, B, overlap);
}

// The inverse kernel's batch parameters, with the segments planned for one
// launch of all planes.
cudaError_t tc_sweep_batch(const SweepArgs* planes, int n, SweepBatch& B) {
  if (n < 1 || n > kMaxBatch) return cudaErrorInvalidValue;
  SweepArgs p[kMaxBatch];
  std::copy(planes, planes + n, p);
  plan_segments(p, n, kTcSweepCtasPerSm * sm_count());
  SweepBatch Bf, Bm;
  return sweep_batches(p, n, Bf, B, Bm) ? cudaSuccess : cudaErrorNotSupported;
}

}  // namespace

cudaError_t launch_sweep_tc_batch(const SweepArgs* planes, int n, const TcTune& t, cudaStream_t st,
                                  cudaEvent_t after_filter) {
  SweepBatch B;
  const cudaError_t e = tc_sweep_batch(planes, n, B);
  if (e != cudaSuccess) return e;
  static_assert(SwpCfg<32>::TJ == 7 && SwpCfg<16>::TJ == 15, "cells per strip");
  return planes[0].inv.g.bw == 16 ? launch_sweep_n<16>(B, n, t, st, after_filter)
                                  : launch_sweep_n<32>(B, n, t, st, after_filter);
}

cudaError_t launch_sweep_tc(const SweepArgs& a, cudaStream_t st) {
  return launch_sweep_tc_batch(&a, 1, TcTune{}, st);
}

cudaError_t tc_graph_update(cudaGraphExec_t exec, cudaGraph_t graph, const TcFwdArgs* fwd, int nf,
                            const SweepArgs* sw, int ns) {
  TcFwdBatch Bw{};
  SweepBatch Bs;
  FilterBatch F;
  FilterLaunch fl[2];
  cudaError_t e = cudaSuccess;
  FwdLaunch wl;
  if (nf > 0) {
    if (!forward_batch(fwd, nf, Bw)) return cudaErrorNotSupported;
    wl = forward_launch(fwd, nf);
    if (!wl.kernel) return cudaErrorNotSupported;
  }
  if (ns > 0) {
    if ((e = tc_sweep_batch(sw, ns, Bs)) != cudaSuccess) return e;
    for (int v = 0; v < 2; v++) fl[v] = filter_launch(Bs, 4 + v, F);
  }
  size_t cnt = 0;
  e = cudaGraphGetNodes(graph, nullptr, &cnt);
  if (e != cudaSuccess) return e;
  std::vector<cudaGraphNode_t> nodes(cnt);
  if ((e = cudaGraphGetNodes(graph, nodes.data(), &cnt)) != cudaSuccess) return e;
  for (cudaGraphNode_t node : nodes) {
    cudaGraphNodeType ty;
    if ((e = cudaGraphNodeGetType(node, &ty)) != cudaSuccess) return e;
    if (ty != cudaGraphNodeTypeKernel) continue;
    cudaKernelNodeParams kp{};
    if ((e = cudaGraphKernelNodeGetParams(node, &kp)) != cudaSuccess) return e;
    void* args[1] = {nullptr};
    const void* f = kp.func;
    if (nf > 0 && f == (const void*)wl.kernel) {
      args[0] = &Bw;
    } else if (ns > 0 && (f == fl[0].kernel || f == fl[1].kernel)) {
      args[0] = &F;
    } else if (f == (const void*)k_sweep_tc<32> || f == (const void*)k_sweep_tc<16>) {
      args[0] = &Bs;
    } else {
      return cudaErrorInvalidValue;
    }
    kp.kernelParams = args;
    kp.extra = nullptr;
    if ((e = cudaGraphExecKernelNodeSetParams(exec, node, &kp)) != cudaSuccess) return e;
  }
  return cudaSuccess;
}

size_t tc_image_bytes(const Geo& g) {
  const int cells_y = (g.H + g.bh / 2 - 1) / (g.bh / 2);
  return (size_t)(cells_y + 1) * g.ncols * (g.bw == 16 ? BlkImg<16>::BYTES : BlkImg<32>::BYTES);
}

}  // namespace f3d
