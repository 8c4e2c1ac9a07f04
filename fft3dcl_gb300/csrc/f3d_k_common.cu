// f3d_k_common.cu -- overlap-add + sample packing, and the launch dispatch.
// Compiled with --fmad=false (the packing must round like the reference).
#include "f3d_device.cuh"

#include <atomic>

namespace f3d {

static std::atomic<unsigned long long> g_launch_count{0};
void count_launch() { g_launch_count.fetch_add(1, std::memory_order_relaxed); }
unsigned long long launch_count() { return g_launch_count.load(std::memory_order_relaxed); }

int sm_count() {
  int dev = 0, n = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev);
  return n > 0 ? n : 1;
}

namespace {

__device__ __forceinline__ int floor_div(int a, int b) {
  int q = a / b;
  return (a % b != 0 && ((a < 0) != (b < 0))) ? q - 1 : q;
}

// The mode-1 blocks covering a sample along one axis: first block and how
// many (the step is at least half the block, so at most two).
__device__ __forceinline__ void covering(int x, int off, int step, int b, int nblk, int& first, int& cnt) {
  int i0 = floor_div(x - off - b, step) + 1, i1 = floor_div(x - off, step);
  if (i0 < 0) i0 = 0;
  if (i1 > nblk - 1) i1 = nblk - 1;
  first = i0;
  cnt = i1 - i0 + 1;
}

// V (1 or 4) neighbouring output samples per thread: sum of the covering
// windowed blocks in ascending block order starting from 0
// (src/cpu/reference.cpp:415-430, the same order as src/cl/kernels.h:409-435),
// plus chroma centering once (:433-436), then packed to the plane's sample
// format (:107-138). One sample per thread spends its time on the divisions
// that find the blocks; four share them and move 16 bytes at a time (1080p
// from 32x32 blocks: 18 -> 8.5 us; 720p float from 64x64: 9.5 -> 5.5 us). Four
// neighbours (from a multiple of four) have the same blocks when the block
// size, offset and step are multiples of four.
template <int V>
__global__ void __launch_bounds__(256) k_ola(const __grid_constant__ OlaArgs a) {
  const int x = (blockIdx.x * 32 + (threadIdx.x & 31)) * V;
  const int y = blockIdx.y * 8 + (threadIdx.x >> 5);
  const Geo& g = a.g;
  grid_go();
  grid_wait();
  stamp_start(a.clk);
  if (x >= g.W || y >= g.H) return;  // not thread 0
  const int bsz = g.bw * g.bh;
  float sum[V];
#pragma unroll
  for (int k = 0; k < V; k++) sum[k] = 0.0f;
  if (g.mode == 1) {
    int n0, nc, m0, mc;
    covering(x, g.xoff, g.xstep, g.bw, g.ncols, n0, nc);
    covering(y, g.yoff, g.ystep, g.bh, g.nrows, m0, mc);
    // The blocks' values are loaded together, then added in block order.
    float v[2][2][V];
#pragma unroll
    for (int i = 0; i < 2; i++) {
      const int ly = y - (g.yoff + (m0 + i) * g.ystep);
#pragma unroll
      for (int j = 0; j < 2; j++) {
        if (i >= mc || j >= nc) continue;
        const int lx = x - (g.xoff + (n0 + j) * g.xstep);
        const float* p = a.blocks + (size_t)((m0 + i) * g.ncols + n0 + j) * bsz + ly * g.bw + lx;
        if constexpr (V == 4) {
          const float4 q = *reinterpret_cast<const float4*>(p);
          v[i][j][0] = q.x, v[i][j][1] = q.y, v[i][j][2] = q.z, v[i][j][3] = q.w;
        } else {
          v[i][j][0] = *p;
        }
      }
    }
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
      for (int j = 0; j < 2; j++)
        if (i < mc && j < nc)
#pragma unroll
          for (int k = 0; k < V; k++) sum[k] += v[i][j][k];
  } else {
    const int per = g.ncols * g.nrows;
    for (int grid = 0; grid < 2; grid++) {
      const int ox = grid ? g.bw / 2 : 0, oy = grid ? g.bh / 2 : 0;
      const int n = (x + ox) / g.bw, m = (y + oy) / g.bh;
      if (n < g.ncols && m < g.nrows) {
        const int lx = x + ox - n * g.bw, ly = y + oy - m * g.bh;
        sum[0] += a.blocks[(size_t)(grid * per + m * g.ncols + n) * bsz + ly * g.bw + lx];
      }
    }
  }
  if (a.chroma_norm != 0.0f)
#pragma unroll
    for (int k = 0; k < V; k++) sum[k] += a.chroma_norm;
  if constexpr (V == 4) store_quad(a.dst + (long long)y * a.pitch, x, g.W, sum, a.fmt, a.inv_norm, a.max_pix);
  else store_sample(a.dst + (long long)y * a.pitch, x, sum[0], a.fmt, a.inv_norm, a.max_pix);
  stamp_end<false>(a.clk);
}

}  // namespace

cudaError_t launch_ola(const OlaArgs& a, cudaStream_t st) {
  if (a.g.W <= 0 || a.g.H <= 0) return cudaSuccess;
  const bool quads = a.g.mode == 1 && a.g.bw % 4 == 0 && a.g.xoff % 4 == 0 && a.g.xstep % 4 == 0;
  const int v = quads ? 4 : 1;
  dim3 grid((a.g.W + 32 * v - 1) / (32 * v), (a.g.H + 7) / 8);
  return launch_kernel(quads ? k_ola<4> : k_ola<1>, grid, 256, 0, st, a);
}

static bool pow2_in(int v, int lo, int hi) { return v >= lo && v <= hi && (v & (v - 1)) == 0; }

bool form_supported(int form, int bw, int bh) {
  if (form == F3D_FORM_EXACT) return pow2_in(bw, 4, 512) && pow2_in(bh, 4, 512);
  if (form == F3D_FORM_FAST) return pow2_in(bw, 8, 64) && pow2_in(bh, 8, 64);
  if (form == F3D_FORM_TC) return bw == bh && (bw == 16 || bw == 32);
  return false;
}

cudaError_t launch_forward(int form, const FwdArgs& a, cudaStream_t st) {
  if (form == F3D_FORM_FAST) return launch_forward_fast(a, st);
  if (form != F3D_FORM_EXACT) return cudaErrorNotSupported;
  if (big_block(a.g.bw, a.g.bh)) return launch_forward_big(a, st);
  switch (a.g.bw) {
  case 4: return launch_forward_exact_bw4(a, st);
  case 8: return launch_forward_exact_bw8(a, st);
  case 16: return launch_forward_exact_bw16(a, st);
  case 32: return launch_forward_exact_bw32(a, st);
  case 64: return launch_forward_exact_bw64(a, st);
  default: return cudaErrorInvalidValue;
  }
}

cudaError_t launch_filter_inverse(int form, const InvArgs& a, cudaStream_t st) {
  if (form == F3D_FORM_FAST) return launch_inverse_fast(a, st);
  if (form != F3D_FORM_EXACT) return cudaErrorNotSupported;
  if (big_block(a.g.bw, a.g.bh)) return launch_inverse_big(a, st);
  switch (a.g.bw) {
  case 4: return launch_inverse_exact_bw4(a, st);
  case 8: return launch_inverse_exact_bw8(a, st);
  case 16: return launch_inverse_exact_bw16(a, st);
  case 32: return launch_inverse_exact_bw32(a, st);
  case 64: return launch_inverse_exact_bw64(a, st);
  default: return cudaErrorInvalidValue;
  }
}

}  // namespace f3d
