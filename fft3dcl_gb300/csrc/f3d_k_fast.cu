// f3d_k_fast.cu -- fast form: packed real transforms in registers with FMA.
//
// Compiled with --fmad=true -ftz=true -prec-div=false -prec-sqrt=false: the
// per-bin filter (the same source as the exact form, f3d_device.cuh) then
// uses the hardware reciprocal and square-root approximations. Results stay
// within the engine's tolerance of the reference (+-1 LSB at 8 bit, +-4 LSB
// at 10 bit, 1e-4 for float output) instead of matching it bit for bit.
//
// Layout and building blocks: f3d_fast.cuh.
//
// Square blocks have kernels of their own (further down). Other shapes, per
// block TPB = max(bw, bh)/2 threads:
//  forward  - the block is gathered cooperatively (vector loads where the
//             rows are aligned), converted and windowed into shared memory;
//             thread t transforms rows 2t and 2t+1 as one complex FFT and
//             splits the two half spectra; thread t then transforms column t,
//             thread 0 columns 0 and bw/2 together (both are real).
//  inverse  - thread t filters column t (and a share of column bw/2) and
//             inverse-transforms it; thread 0 inverts columns 0 and bw/2
//             together after taking their Hermitian parts, which is what the
//             real part of the reference's full complex inverse keeps; thread t
//             then inverts rows 2t and 2t+1 from their Hermitian halves as one
//             complex FFT whose real and imaginary parts are the two rows.
#include "f3d_fast.cuh"

#include <type_traits>

namespace f3d {
namespace {

constexpr int kThreads = 128;

// The samples of a block inside the plane whose rows are aligned, four per
// thread and load, so that samples and window are read in whole lines (with
// 16 bytes of samples per thread each window read touched up to 24 sectors).
template <int BW, int BH, int TPB, int TS, int FMT>
__device__ __forceinline__ void gather_quads(const FwdArgs& a, uintptr_t row0, int t, float* tile) {
  constexpr int BPS = FMT == FMT_U8 ? 1 : (FMT == FMT_U16 ? 2 : 4);
  using Raw = typename std::conditional<BPS == 1, uint32_t, typename std::conditional<BPS == 2, uint2, uint4>::type>::type;
  constexpr int QPR = BW / 4, RPT = TPB / QPR, NR = BH / RPT;  // quads per row, rows per round, rounds
  constexpr int NB = NR < 8 ? NR : 8;                          // loads in flight
  static_assert(TPB % QPR == 0 && BH % RPT == 0 && NR % NB == 0, "row split");
  const int lx = t % QPR * 4, ly0 = t / QPR;
  const float4* win = reinterpret_cast<const float4*>(a.win) + t;
#pragma unroll 1
  for (int i0 = 0; i0 < NR; i0 += NB) {
    Raw raw[NB];
    float4 w[NB];
#pragma unroll
    for (int i = 0; i < NB; i++) {
      raw[i] = *reinterpret_cast<const Raw*>(row0 + (long long)(ly0 + RPT * (i0 + i)) * a.pitch + lx * BPS);
      w[i] = win[(i0 + i) * TPB];
    }
#pragma unroll
    for (int i = 0; i < NB; i++) {
      float* dst = tile + (ly0 + RPT * (i0 + i)) * TS + lx;
      const float wk[4] = {w[i].x, w[i].y, w[i].z, w[i].w};
#pragma unroll
      for (int k = 0; k < 4; k++) {
        if constexpr (FMT == FMT_U8) {
          dst[k] = ((float)((raw[i] >> (8 * k)) & 0xffu) * (1.0f / 255.0f) - a.chroma_norm) * wk[k];
        } else if constexpr (FMT == FMT_U16) {
          const uint32_t v = k < 2 ? raw[i].x : raw[i].y;
          dst[k] = ((float)((v >> (16 * (k & 1))) & 0xffffu) * a.norm - a.chroma_norm) * wk[k];
        } else {
          const uint32_t v = k == 0 ? raw[i].x : (k == 1 ? raw[i].y : (k == 2 ? raw[i].z : raw[i].w));
          dst[k] = (__uint_as_float(v) - a.chroma_norm) * wk[k];
        }
      }
    }
  }
}

// The samples of block b, converted and windowed, into tile[BH][TS], by TPB
// threads.
template <int BW, int BH, int TPB, int TS>
__device__ __forceinline__ void gather_block(const FwdArgs& a, int b, int t, float* tile) {
  int bx, by, par;
  block_origin(a.g, b, bx, by, par);
  const bool inside = bx >= 0 && by >= 0 && bx + BW <= a.g.W && by + BH <= a.g.H;
  const int bps = a.fmt == FMT_U8 ? 1 : (a.fmt == FMT_U16 ? 2 : 4);
  const uintptr_t row0 = reinterpret_cast<uintptr_t>(a.src) + (long long)by * a.pitch + (long long)bx * bps;
  // Rows aligned to whole loads. With a chroma offset the sample loop below
  // rounds the scaled sample before the offset is taken off, and the quads
  // after it: they keep to the blocks that were always read that way.
  const uintptr_t low = row0 | (uintptr_t)a.pitch;
  const bool quads = inside && (a.chroma_norm == 0.0f ? (low & (4 * bps - 1)) == 0
                                                      : (low & 15) == 0 && (BW * bps) % 16 == 0);
  if (quads) {
    if (a.fmt == FMT_U8) gather_quads<BW, BH, TPB, TS, FMT_U8>(a, row0, t, tile);
    else if (a.fmt == FMT_U16) gather_quads<BW, BH, TPB, TS, FMT_U16>(a, row0, t, tile);
    else gather_quads<BW, BH, TPB, TS, FMT_F32>(a, row0, t, tile);
    return;
  }
  for (int idx = t; idx < BW * BH; idx += TPB) {
    const int ly = idx / BW, lx = idx - ly * BW;
    const int y = inside ? by + ly : mirror_i(by + ly, a.g.H);
    const int x = inside ? bx + lx : mirror_i(bx + lx, a.g.W);
    tile[ly * TS + lx] =
        (load_sample(a.src + (long long)y * a.pitch, x, a.fmt, a.norm) - a.chroma_norm) * a.win[idx];
  }
}

template <int BW, int BH>
__global__ void __launch_bounds__(128) k_forward_fast(const __grid_constant__ FwdArgs a) {
  using C = FCfg<BW, BH>;
  constexpr int BPC = kThreads / C::TPB;
  extern __shared__ float4 smem4[];
  const int slot = threadIdx.x / C::TPB, t = threadIdx.x - slot * C::TPB;
  const int b = blockIdx.x * BPC + slot;
  const bool valid = b < a.g.nb;
  float2* S = reinterpret_cast<float2*>(smem4) + slot * C::SMEM_F2;
  float* tile = reinterpret_cast<float*>(S);  // input tile [BH][TS], aliased with S

  grid_wait();
  stamp_start(a.clk);
  if (valid) gather_block<BW, BH, C::TPB, C::TS>(a, b, t, tile);
  __syncwarp();
  float2 z[BW];
  const bool rows = valid && t < BH / 2;
  if (rows) {
#pragma unroll
    for (int c = 0; c < BW; c++) z[c] = make_float2(tile[(2 * t) * C::TS + c], tile[(2 * t + 1) * C::TS + c]);
  }
  __syncwarp();  // the tile is dead from here on; S reuses its storage
  if (rows) {
    fft_fast<BW, false>(z, a.tw.row);
    // Split Z = X_2t + i X_2t+1: X_2t[k] = (Z[k] + conj Z[-k])/2,
    // X_2t+1[k] = (Z[k] - conj Z[-k])/(2i).
#pragma unroll
    for (int k = 0; k <= C::NY; k++) {
      const float2 A = z[k], B = z[(BW - k) % BW];
      tile_pair<C::SB>(S, k, 2 * t) =
          make_float4(0.5f * (A.x + B.x), 0.5f * (A.y - B.y), 0.5f * (A.y + B.y), 0.5f * (B.x - A.x));
    }
  }
  __syncwarp();
  if (valid && t < C::NY) {
    float2 y[BH];
    if (t == 0) {  // columns 0 and bw/2 are real: transform them together
#pragma unroll
      for (int r = 0; r < BH; r += 2) {
        const float4 p0 = tile_pair<C::SB>(S, 0, r), pn = tile_pair<C::SB>(S, C::NY, r);
        y[r] = make_float2(p0.x, pn.x);
        y[r + 1] = make_float2(p0.z, pn.z);
      }
    } else {
#pragma unroll
      for (int r = 0; r < BH; r += 2) {
        const float4 p = tile_pair<C::SB>(S, t, r);
        y[r] = make_float2(p.x, p.y);
        y[r + 1] = make_float2(p.z, p.w);
      }
    }
    fft_fast<BH, false>(y, a.tw.col);
    float2* out = a.spec + (size_t)b * C::PS;
    if (t == 0) {
#pragma unroll
      for (int k = 0; k < BH; k++) {
        const float2 A = y[k], B = y[(BH - k) % BH];
        out[k * C::FBW] = make_float2(0.5f * (A.x + B.x), 0.5f * (A.y - B.y));
        out[k * C::FBW + C::NY] = make_float2(0.5f * (A.y + B.y), 0.5f * (B.x - A.x));
      }
    } else {
#pragma unroll
      for (int r = 0; r < BH; r++) out[r * C::FBW + t] = y[r];
    }
  }
  grid_go();
  stamp_end(a.clk);
}

template <int BW, int BH, int BM>
__global__ void __launch_bounds__(128) k_inverse_fast(const __grid_constant__ InvArgs a) {
  using C = FCfg<BW, BH>;
  constexpr int BPC = kThreads / C::TPB;
  extern __shared__ float4 smem4[];
  const int slot = threadIdx.x / C::TPB, t = threadIdx.x - slot * C::TPB;
  const int b = blockIdx.x * BPC + slot;
  const bool valid = b < a.g.nb;
  float2* S = reinterpret_cast<float2*>(smem4) + slot * C::SMEM_F2;
  int bx = 0, by = 0, par = 0;
  if (valid) block_origin(a.g, b, bx, by, par);
  const float* win = par ? a.win_b : a.win_a;
  float* out = a.blocks + (size_t)b * BW * BH;
  constexpr float inv_n = 1.0f / (BW * BH);
  grid_go();
  grid_wait();
  stamp_start(a.clk);
  inverse_block<BW, BH, BM>(a, b, t, valid, S, [&](int y, const float2(&xy)[BW / 2]) {
#pragma unroll
    for (int n = 0; n < BW / 2; n += 2) {
      const float4 wv = *reinterpret_cast<const float4*>(win + y * BW + 2 * n);
      *reinterpret_cast<float4*>(out + y * BW + 2 * n) =
          make_float4(xy[n].x * inv_n * wv.x, xy[n].y * inv_n * wv.y, xy[n + 1].x * inv_n * wv.z,
                      xy[n + 1].y * inv_n * wv.w);
    }
  }, [] {});
  stamp_end(a.clk);
}

// ---- square blocks ---------------------------------------------------------
//
// Forward of N x N blocks with N threads per block and each transform on a
// lane pair, in CTAs of 64 threads. 1080p 10-bit with 32x32 blocks (28 warps
// per SM in all at 16 threads per block): 44 -> 35 us, 4K 86 -> 75; 8-bit with 64x64
// blocks 73 -> 50 us.
constexpr int kPairThreads = 64;
template <int N>
constexpr int kPairFwdCtas = N == 64 ? 12 : (N == 32 ? 20 : 24);

template <int N>
__device__ __forceinline__ void pair_sync() {
  if constexpr (N > 32) __syncthreads();
  else __syncwarp();
}

template <int N>
__global__ void __launch_bounds__(kPairThreads, kPairFwdCtas<N>) k_forward_fast_sq(const __grid_constant__ FwdArgs a) {
  using C = FCfg<N, N>;
  constexpr int SB = C::SB, FBW = C::FBW, NY = C::NY, H = N / 2, L = Log2<N>::v;
  constexpr int BPC = kPairThreads / N;
  extern __shared__ float4 smem4[];
  const int slot = threadIdx.x / N, t = threadIdx.x - slot * N, p = t >> 1;
  const bool odd = t & 1;
  const int b = blockIdx.x * BPC + slot;
  const bool valid = b < a.g.nb;
  float2* S = reinterpret_cast<float2*>(smem4) + slot * C::SMEM_F2;
  float* tile = reinterpret_cast<float*>(S);  // input tile [N][TS], aliased with S
  if (N == 64) grid_go();
  grid_wait();
  stamp_start(a.clk);
  if (valid) gather_block<N, N, N, C::TS>(a, b, t, tile);
  pair_sync<N>();
  float2 z[H];
  // Rows 2p and 2p + 1 as one complex transform.
#pragma unroll
  for (int q = 0; q < H; q++) {
    const int c = bit_reverse(q, L) + odd;
    z[q] = make_float2(tile[(2 * p) * C::TS + c], tile[(2 * p + 1) * C::TS + c]);
  }
  pair_sync<N>();  // the tile is dead from here on; S reuses its storage
  fft_fast_pair<N>(z, a.tw.row, odd);
  // Split Z = X_2p + i X_2p+1: X_2p[k] = (Z[k] + conj Z[-k])/2, X_2p+1[k] =
  // (Z[k] - conj Z[-k])/(2i); columns 0..N/4 on the even lane, N/2..N/4+1 on
  // the odd one. Z[N - k] of the even lane's k is the odd lane's entry N/2 - k,
  // and the other way round.
  tile_pair<SB>(S, odd ? NY : 0, 2 * p) =
      make_float4(0.5f * (z[0].x + z[0].x), 0.5f * (z[0].y - z[0].y), 0.5f * (z[0].y + z[0].y), 0.5f * (z[0].x - z[0].x));
#pragma unroll
  for (int i = 1; i <= N / 4; i++) {
    const float2 r = shfl_pair(z[H - i]);
    const float2 A = odd ? r : z[i], B = odd ? z[i] : r;
    if (i < N / 4 || !odd)
      tile_pair<SB>(S, odd ? NY - i : i, 2 * p) =
          make_float4(0.5f * (A.x + B.x), 0.5f * (A.y - B.y), 0.5f * (A.y + B.y), 0.5f * (B.x - A.x));
  }
  pair_sync<N>();
  // Column p; pair 0: columns 0 and N/2, which are real, together.
#pragma unroll
  for (int q = 0; q < H; q++) {
    const int r = bit_reverse(q, L) + odd;
    z[q] = p ? S[p * SB + r] : make_float2(S[r].x, S[NY * SB + r].x);
  }
  fft_fast_pair<N>(z, a.tw.col, odd);
  float2* out = a.spec + (size_t)b * C::PS + (odd ? H * FBW : 0);
  if (N <= 32 || t < 32) {  // the warp of pair 0
#pragma unroll
    for (int i = 0; i < H; i++) {
      const float2 A = z[i], B = i ? shfl_pair(z[H - i]) : z[0];
      if (p == 0 && valid) {
        out[i * FBW] = make_float2(0.5f * (A.x + B.x), 0.5f * (A.y - B.y));
        out[i * FBW + NY] = make_float2(0.5f * (A.y + B.y), 0.5f * (B.x - A.x));
      }
    }
  }
  if (p && valid) {
#pragma unroll
    for (int i = 0; i < H; i++) out[i * FBW + p] = z[i];
  }
  // The sweep takes these blocks' spectra: as the filter's in the tensor-core
  // form, its CTAs start as this kernel's end (4K 10-bit bt=4: 261 us; started
  // at once, 352). 64 x 64 blocks go to k_inverse_fast64, CTAs as small as
  // these: at once (1080p 8-bit bt=3 122 us; as they end, 129).
  if (N < 64) grid_go();
  stamp_end(a.clk);
}

template <int N>
cudaError_t launch_fwd_sq(const FwdArgs& a, cudaStream_t st) {
  constexpr int BPC = kPairThreads / N;
  constexpr size_t smem = sizeof(float2) * FCfg<N, N>::SMEM_F2 * BPC;
  static_assert(smem <= 48 * 1024, "no opt-in needed");
  const int grid = (a.g.nb + BPC - 1) / BPC;
  if (grid == 0) return cudaSuccess;
  return launch_kernel(k_forward_fast_sq<N>, grid, kPairThreads, smem, st, a);
}

// ---- 64 x 64 blocks -----------------------------------------------------------
//
// The inverse, one block per CTA of 64 threads, each column transform on a
// lane pair; the windowed rows go back to shared memory and leave in plane
// order, where from the row transforms each thread would walk its own row, a
// line per lane and request. 1080p 8-bit bt=3 (2,232 blocks for 1,824 CTA
// slots: the latency of one block counts twice): 79 -> 67 us.
// inverse_block (f3d_fast.cuh) with 64 threads: thread (c, h) = (t / 2, t % 2)
// filters rows 32 h .. 32 h + 31 of column c and row t of column 32, then
// inverts column c's even (h = 0) or odd inputs, combined through a shuffle
// (as inverse_block_sq), then the row at tile position t.
template <int BM>
__global__ void __launch_bounds__(kPairThreads, 12) k_inverse_fast64(const __grid_constant__ InvArgs a) {
  using C = FCfg<64, 64>;
  constexpr int SB = C::SB, FBW = C::FBW, NY = C::NY, H = 32;
  extern __shared__ float4 smem4[];
  float2* S = reinterpret_cast<float2*>(smem4);
  const int t = threadIdx.x, c = t >> 1, h = t & 1, b = blockIdx.x;
  const size_t base = (size_t)b * C::PS;
  grid_go();
  grid_wait();
  stamp_start(a.clk);
  {
    constexpr int NF = BM >= 2 ? BM : 1;
    if (t < NF) prefetch_l2(a.s[t] + base, C::PS * sizeof(float2));
    const float dc = block_dc(a, b);
    // Four bins' spectra and tables are loaded together.
#pragma unroll 1
    for (int k = 0; k < H; k += 4) {
      const int r = h * H + k;
      float2 sv[4][4], f[4];
      BinTables tb[4];
#pragma unroll
      for (int u = 0; u < 4; u++) {
        load_window<BM>(a, base + (r + u) * FBW + c, sv[u]);
        tb[u] = bin_tables(a, (r + u) * FBW + c);
      }
#pragma unroll
      for (int u = 0; u < 4; u++) f[u] = filter_vals_t<BM, true>(a, dc, tb[u], 0, sv[u]);
      tile_pair<SB>(S, c, r) = make_float4(f[0].x, f[0].y, f[1].x, f[1].y);
      tile_pair<SB>(S, c, r + 2) = make_float4(f[2].x, f[2].y, f[3].x, f[3].y);
    }
    S[NY * SB + t] = filter_bin_t<BM, true>(a, dc, t * FBW + NY, base + t * FBW + NY);
  }
  __syncthreads();
  if (t <= 32) {  // Hermitian parts of columns 0 and 32, packed into column 0
    const int r = t, m = (64 - t) % 64;
    const float2 zr = S[r], zm = S[m];
    const float2 nr = S[NY * SB + r], nm = S[NY * SB + m];
    const float ar = 0.5f * (zr.x + zm.x), ai = 0.5f * (zr.y - zm.y);
    const float qr = 0.5f * (nr.x + nm.x), qi = 0.5f * (nr.y - nm.y);
    S[r] = make_float2(ar - qi, ai + qr);
    if (m != r) S[m] = make_float2(ar + qi, qr - ai);
  }
  __syncthreads();
  float2 e[H];
#pragma unroll
  for (int j = 0; j < H; j++) e[j] = S[c * SB + 2 * j + h];
  fft_fast<H, true, 2>(e, a.tw.col);
  __syncwarp();  // the pair has read its column
#pragma unroll
  for (int y = 0; y < H; y++) {
    const float2 w = a.tw.col[y];
    // e^{+2 pi i y/64} O[y] on h = 1
    const float2 o = make_float2(fmaf(e[y].x, w.x, e[y].y * w.y), fmaf(e[y].y, w.x, -e[y].x * w.y));
    const float2 v = h ? o : e[y], q = shfl_pair(v);
    // h = 0: x[y] = E + P at slot 2y; h = 1: x[y + 32] = E - P at slot 2y + 1
    const float2 x = h ? make_float2(q.x - v.x, q.y - v.y) : make_float2(v.x + q.x, v.y + q.y);
    if (c == 0) {  // real inverses of columns 0 and 32
      S[2 * y + h] = make_float2(x.x, 0.0f);
      S[NY * SB + 2 * y + h] = make_float2(x.y, 0.0f);
    } else {
      S[c * SB + 2 * y + h] = x;
    }
  }
  __syncthreads();
  {
#pragma unroll
    for (int k = 0; k < H; k++) {
      const float2 yk = S[k * SB + t], ym = S[(H - k) * SB + t];
      const float ax = yk.x + ym.x, ay = yk.y - ym.y;
      const float bx = yk.x - ym.x, by = yk.y + ym.y;
      const float2 w = a.tw.row[k];  // e^{-2 pi i k/64}; the conjugate is used
      const float px = fmaf(bx, w.x, by * w.y), py = fmaf(by, w.x, -bx * w.y);
      e[k] = make_float2(ax - py, ay + px);
    }
    fft_fast<H, true, 2>(e, a.tw.row);
    // Only this thread reads or writes the entries at tile position t.
#pragma unroll
    for (int k = 0; k < H; k++) S[k * SB + t] = e[k];
  }
  __syncthreads();
  int bx, by, par;
  block_origin(a.g, b, bx, by, par);
  const float2* win = reinterpret_cast<const float2*>(par ? a.win_b : a.win_a);
  float2* out = reinterpret_cast<float2*>(a.blocks + (size_t)b * 64 * 64);
  constexpr float inv_n = 1.0f / (64 * 64);
#pragma unroll 8
  for (int i = t; i < 64 * H; i += kPairThreads) {
    const float2 v = S[(i % H) * SB + yperm<64>(i / H)], w = win[i];
    out[i] = make_float2(v.x * inv_n * w.x, v.y * inv_n * w.y);
  }
  stamp_end(a.clk);
}

template <int BM>
cudaError_t launch_inv64(const InvArgs& a, cudaStream_t st) {
  if (a.g.nb == 0) return cudaSuccess;
  return launch_kernel(k_inverse_fast64<BM>, a.g.nb, kPairThreads, sizeof(float2) * FCfg<64, 64>::SMEM_F2, st, a);
}

// Square blocks up to 32 x 32: inverse_block_sq, N threads per block (one
// warp or part of one), the rows through the tile as in k_inverse_fast64.
// 1365x767 16-bit bt=2 with a quarter overlap: 16.5 -> 14.4 us (k_inverse_fast,
// half the threads per block, each storing its own rows).
template <int N, int BM>
__global__ void __launch_bounds__(kThreads) k_inverse_fast_sq(const __grid_constant__ InvArgs a) {
  using C = FCfg<N, N>;
  constexpr int BPC = kThreads / N, SB = C::SB;
  extern __shared__ float4 smem4[];
  const int slot = threadIdx.x / N, t = threadIdx.x - slot * N;
  const int b = blockIdx.x * BPC + slot;
  const bool valid = b < a.g.nb;
  float2* S = reinterpret_cast<float2*>(smem4) + slot * C::SMEM_F2;
  grid_go();
  grid_wait();
  stamp_start(a.clk);
  inverse_block_sq<N, BM, 4>(a, a, b, t, valid, S, [&](int y, const float2(&xy)[N / 2]) {
#pragma unroll
    for (int k = 0; k < N / 2; k++) S[k * SB + yperm<N>(y)] = xy[k];
  }, [] {});
  if (!valid) return;  // not thread 0
  int bx, by, par;
  block_origin(a.g, b, bx, by, par);
  const float2* win = reinterpret_cast<const float2*>(par ? a.win_b : a.win_a);
  float2* out = reinterpret_cast<float2*>(a.blocks + (size_t)b * N * N);
  constexpr float inv_n = 1.0f / (N * N);
#pragma unroll 8
  for (int i = t; i < N * N / 2; i += N) {
    const float2 v = S[(i % (N / 2)) * SB + yperm<N>(i / (N / 2))], w = win[i];
    out[i] = make_float2(v.x * inv_n * w.x, v.y * inv_n * w.y);
  }
  stamp_end(a.clk);
}

template <int N, int BM>
cudaError_t launch_inv_sq(const InvArgs& a, cudaStream_t st) {
  constexpr int BPC = kThreads / N;
  constexpr size_t smem = sizeof(float2) * FCfg<N, N>::SMEM_F2 * BPC;
  static_assert(smem <= 48 * 1024, "no opt-in needed");
  const int grid = (a.g.nb + BPC - 1) / BPC;
  if (grid == 0) return cudaSuccess;
  return launch_kernel(k_inverse_fast_sq<N, BM>, grid, kThreads, smem, st, a);
}

template <int BW, int BH>
cudaError_t launch_fwd(const FwdArgs& a, cudaStream_t st) {
  if constexpr (BW == BH) {
    return launch_fwd_sq<BW>(a, st);
  } else {
    using C = FCfg<BW, BH>;
    constexpr int BPC = kThreads / C::TPB;
    const size_t smem = sizeof(float2) * C::SMEM_F2 * BPC;
    auto k = k_forward_fast<BW, BH>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    const int grid = (a.g.nb + BPC - 1) / BPC;
    if (grid == 0) return cudaSuccess;
    return launch_kernel(k, grid, kThreads, smem, st, a);
  }
}

template <int BW, int BH, int BM>
cudaError_t launch_inv_bm(const InvArgs& a, cudaStream_t st) {
  if constexpr (BW == 64 && BH == 64) {
    return launch_inv64<BM>(a, st);
  } else if constexpr (BW == BH) {
    return launch_inv_sq<BW, BM>(a, st);
  } else {
    using C = FCfg<BW, BH>;
    constexpr int BPC = kThreads / C::TPB;
    const size_t smem = sizeof(float2) * C::SMEM_F2 * BPC;
    auto k = k_inverse_fast<BW, BH, BM>;
    if (smem > 48 * 1024) {
      cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
      if (e != cudaSuccess) return e;
    }
    const int grid = (a.g.nb + BPC - 1) / BPC;
    if (grid == 0) return cudaSuccess;
    return launch_kernel(k, grid, kThreads, smem, st, a);
  }
}

template <int BW, int BH>
cudaError_t launch_inv(const InvArgs& a, cudaStream_t st) {
  switch (a.bm) {
  case -1: return launch_inv_bm<BW, BH, -1>(a, st);
  case 1: return launch_inv_bm<BW, BH, 1>(a, st);
  case 2: return launch_inv_bm<BW, BH, 2>(a, st);
  case 3: return launch_inv_bm<BW, BH, 3>(a, st);
  case 4: return launch_inv_bm<BW, BH, 4>(a, st);
  default: return cudaErrorNotSupported;  // Kalman runs the exact form
  }
}

template <int BW>
cudaError_t fwd_bh(const FwdArgs& a, cudaStream_t st) {
  switch (a.g.bh) {
  case 8: return launch_fwd<BW, 8>(a, st);
  case 16: return launch_fwd<BW, 16>(a, st);
  case 32: return launch_fwd<BW, 32>(a, st);
  case 64: return launch_fwd<BW, 64>(a, st);
  default: return cudaErrorInvalidValue;
  }
}

template <int BW>
cudaError_t inv_bh(const InvArgs& a, cudaStream_t st) {
  switch (a.g.bh) {
  case 8: return launch_inv<BW, 8>(a, st);
  case 16: return launch_inv<BW, 16>(a, st);
  case 32: return launch_inv<BW, 32>(a, st);
  case 64: return launch_inv<BW, 64>(a, st);
  default: return cudaErrorInvalidValue;
  }
}

}  // namespace

cudaError_t launch_forward_fast(const FwdArgs& a, cudaStream_t st) {
  switch (a.g.bw) {
  case 8: return fwd_bh<8>(a, st);
  case 16: return fwd_bh<16>(a, st);
  case 32: return fwd_bh<32>(a, st);
  case 64: return fwd_bh<64>(a, st);
  default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_inverse_fast(const InvArgs& a, cudaStream_t st) {
  switch (a.g.bw) {
  case 8: return inv_bh<8>(a, st);
  case 16: return inv_bh<16>(a, st);
  case 32: return inv_bh<32>(a, st);
  case 64: return inv_bh<64>(a, st);
  default: return cudaErrorInvalidValue;
  }
}

}  // namespace f3d
