// ksj_gpu_combine.cu -- adaptive coil combination (Walsh) on coil-last images.
//
//   k_walsh<C>  one thread per pixel of a 32 x 8 tile whose coil values, with a
//               halo of half the window, sit in shared memory: the window's
//               coil covariance R = sum_q x(q) x(q)^H as sums down the
//               window's columns, shared by the pixels of a row, then across
//               them; its dominant eigenvector by power iteration started from
//               the pixel's own coil vector, phase-referenced to coil 0, and
//               the combination v^H x(p).
//
// Walsh, Gmitro and Marcellin, MRM 43:682-690, 2000 (noise covariance taken as
// the identity).  The window is clipped at the image border (samples outside
// the image contribute nothing).  No counterpart in the reference, whose
// adaptive combine is a planned interface only.
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <complex>
#include <cstdint>
#include <vector>

#include "ksj_gpu.h"
#include "ksj_gpu_internal.cuh"

namespace ksj_gpu {
namespace {

constexpr int kWalshCols = 32, kWalshRows = 8;  // pixels of a block's tile, a warp per row
constexpr int kWalshThreads = kWalshCols * kWalshRows;
constexpr int kWalshMaxHalf = 4;  // windows 1, 3, ..., 9
constexpr int kWalshSquare = 12;  // power iterations left from which R^4 is formed first
// ... where R v (v of unit length, R of trace 1/2 to 1) is at least 2^-6 long: then R^4 v is
// at least 2^-24. A vector in the space of a small eigenvalue (coils that share no pixel of the window)
// is taken to its fourth power, whose square is below FP32's range from 2e-6 of the trace
// on; there R itself goes on.
constexpr float kWalshSquareNorm = 0x1p-12f;  // its square

// Hermitian C x C matrix: real diagonal, upper triangle row by row.
template <int C>
struct Hermitian {
  float d[C];
  float2 o[C * (C - 1) / 2 + 1];  // (never empty)
};
template <int C>
__host__ __device__ constexpr int upper(int i, int j) {  // i < j
  return i * C - i * (i + 1) / 2 + j - i - 1;
}

// u = R v.
template <int C>
__device__ __forceinline__ void hermitian_apply(const Hermitian<C>& r, const float2* v, float2* u) {
#pragma unroll
  for (int i = 0; i < C; ++i) u[i] = make_float2(r.d[i] * v[i].x, r.d[i] * v[i].y);
#pragma unroll
  for (int i = 0; i < C; ++i) {
#pragma unroll
    for (int j = i + 1; j < C; ++j) {
      const float2 a = r.o[upper<C>(i, j)];
      u[i].x = fmaf(a.x, v[j].x, fmaf(-a.y, v[j].y, u[i].x));  // R_ij v_j
      u[i].y = fmaf(a.x, v[j].y, fmaf(a.y, v[j].x, u[i].y));
      u[j].x = fmaf(a.x, v[i].x, fmaf(a.y, v[i].y, u[j].x));   // conj(R_ij) v_i
      u[j].y = fmaf(a.x, v[i].y, fmaf(-a.y, v[i].x, u[j].y));
    }
  }
}

// s = R R (Hermitian: the upper triangle of it).
template <int C>
__device__ __forceinline__ void hermitian_square(const Hermitian<C>& r, Hermitian<C>& s) {
#pragma unroll
  for (int i = 0; i < C; ++i) {
    float d = r.d[i] * r.d[i];
#pragma unroll
    for (int k = 0; k < C; ++k) {
      if (k == i) continue;
      const float2 a = r.o[k < i ? upper<C>(k, i) : upper<C>(i, k)];
      d = fmaf(a.x, a.x, fmaf(a.y, a.y, d));
    }
    s.d[i] = d;
#pragma unroll
    for (int j = i + 1; j < C; ++j) {
      const float2 a = r.o[upper<C>(i, j)];
      const float both = r.d[i] + r.d[j];  // k = i and k = j
      float2 t = make_float2(both * a.x, both * a.y);
#pragma unroll
      for (int k = 0; k < C; ++k) {
        if (k == i || k == j) continue;
        // R_ik R_kj, each from the upper triangle (conjugated below it)
        const float2 p = r.o[i < k ? upper<C>(i, k) : upper<C>(k, i)];
        const float2 q = r.o[k < j ? upper<C>(k, j) : upper<C>(j, k)];
        const float py = i < k ? p.y : -p.y, qy = k < j ? q.y : -q.y;
        t.x = fmaf(p.x, q.x, fmaf(-py, qy, t.x));
        t.y = fmaf(p.x, qy, fmaf(py, q.x, t.y));
      }
      s.o[upper<C>(i, j)] = t;
    }
  }
}

template <int C>
__device__ __forceinline__ float norm2(const float2* u) {
  float n = 0.0f;
#pragma unroll
  for (int i = 0; i < C; ++i) n = fmaf(u[i].x, u[i].x, fmaf(u[i].y, u[i].y, n));
  return n;
}

template <int C>
__device__ __forceinline__ void normalise(float2* v) {
  const float inv = rsqrtf(norm2<C>(v));
#pragma unroll
  for (int i = 0; i < C; ++i) v[i] = cscale(v[i], inv);
}

// Bound by FP32 issue.  Per pixel of 8 coils and a 7 x 7 window: the sums down
// the columns are 7 outer products for each of the tile's 38 columns (1.2 a
// pixel and row of the window, instead of 49 a pixel), the sums across 7 x 64
// additions; 24 power iterations are 6 with R^4 (two squarings and six products, 3.3 k
// multiply-adds, instead of 24 products, 5.8 k: the powers of R commute, and each is
// Hermitian).  R is scaled by a power of two first, so that R^4 of any image
// stays within range.  The sums across run over the window's columns with all 64 sums of a pixel
// inside (a loop for each sum was 64 loops of code, and the kernel waited for the
// instruction cache more than for anything else).  256 x 256 pixels, 8 coils: 57 us -> 34, with
// the sums across so 24.1, and 24.6 with the look at each product's length.
template <int C>
__global__ void __launch_bounds__(kWalshThreads, 2) k_walsh(const float2* __restrict__ in, float2* out, int rows, int cols,
                                                         int half, int iterations) {
  chain_begin();
  extern __shared__ float2 walsh_smem[];
  const int span = kWalshCols + 2 * half, tall = kWalshRows + 2 * half;
  float2* tile = walsh_smem;                                        // [coil][tall][span]
  float* sums = reinterpret_cast<float*>(tile + C * tall * span);  // [C * C][kWalshRows][span]
  const int across_tiles = (cols + kWalshCols - 1) / kWalshCols;
  const int ty0 = blockIdx.x / across_tiles * kWalshRows, tx0 = blockIdx.x % across_tiles * kWalshCols;
  const int r0 = ty0 - half;
  const int c0 = tx0 - half;
  const int tid = threadIdx.x;
  for (int i = tid; i < tall * span * C; i += kWalshThreads) {
    const int pix = i / C;
    const int c = i - pix * C;
    const int y = pix / span, x = pix - y * span;
    const int r = r0 + y, cc = c0 + x;
    tile[(c * tall + y) * span + x] = (r >= 0 && r < rows && cc >= 0 && cc < cols)
                                          ? __ldg(in + (static_cast<size_t>(r) * cols + cc) * C + c)
                                          : make_float2(0.0f, 0.0f);
  }
  __syncthreads();
  const int positions = kWalshRows * span;
  for (int p = tid; p < positions; p += kWalshThreads) {
    Hermitian<C> a;
#pragma unroll
    for (int i = 0; i < C; ++i) a.d[i] = 0.0f;
#pragma unroll
    for (int k = 0; k < C * (C - 1) / 2; ++k) a.o[k] = make_float2(0.0f, 0.0f);
    for (int dy = 0; dy <= 2 * half; ++dy) {
      float2 x[C];
#pragma unroll
      for (int c = 0; c < C; ++c) x[c] = tile[c * tall * span + dy * span + p];
#pragma unroll
      for (int i = 0; i < C; ++i) {
        a.d[i] = fmaf(x[i].x, x[i].x, fmaf(x[i].y, x[i].y, a.d[i]));
#pragma unroll
        for (int j = i + 1; j < C; ++j) {  // x_i conj(x_j)
          float2& o = a.o[upper<C>(i, j)];
          o.x = fmaf(x[i].x, x[j].x, fmaf(x[i].y, x[j].y, o.x));
          o.y = fmaf(x[i].y, x[j].x, fmaf(-x[i].x, x[j].y, o.y));
        }
      }
    }
#pragma unroll
    for (int i = 0; i < C; ++i) sums[i * positions + p] = a.d[i];
#pragma unroll
    for (int k = 0; k < C * (C - 1) / 2; ++k) {
      sums[(C + 2 * k) * positions + p] = a.o[k].x;
      sums[(C + 2 * k + 1) * positions + p] = a.o[k].y;
    }
  }
  __syncthreads();
  const int ty = tid / kWalshCols, tx = tid - ty * kWalshCols;
  const int r = ty0 + ty;
  const int cc = tx0 + tx;
  if (r >= rows || cc >= cols) return;
  Hermitian<C> R;
  const float* line = sums + ty * span + tx;
#pragma unroll
  for (int i = 0; i < C; ++i) R.d[i] = 0.0f;
#pragma unroll
  for (int k = 0; k < C * (C - 1) / 2; ++k) R.o[k] = make_float2(0.0f, 0.0f);
#pragma unroll 1
  for (int dx = 0; dx <= 2 * half; ++dx) {
#pragma unroll
    for (int i = 0; i < C; ++i) R.d[i] += line[i * positions + dx];
#pragma unroll
    for (int k = 0; k < C * (C - 1) / 2; ++k) {
      R.o[k].x += line[(C + 2 * k) * positions + dx];
      R.o[k].y += line[(C + 2 * k + 1) * positions + dx];
    }
  }
  float trace = 0.0f;
#pragma unroll
  for (int i = 0; i < C; ++i) trace += R.d[i];
  float2 own[C], v[C];
#pragma unroll
  for (int c = 0; c < C; ++c) v[c] = own[c] = tile[(c * tall + ty + half) * span + tx + half];
  if (!(norm2<C>(v) > 0.0f)) {
#pragma unroll
    for (int c = 0; c < C; ++c) v[c] = make_float2(c == 0 ? 1.0f : 0.0f, 0.0f);
  }
  if (iterations > 0) {
    float2 u[C];
    if (trace > 0.0f && isfinite(trace)) {
      // times 2^-k with trace 2^-k in [1/2, 1): exact
      int k;
      frexpf(trace, &k);
      const float sc = ldexpf(1.0f, max(min(-k, 126), -126));
#pragma unroll
      for (int i = 0; i < C; ++i) R.d[i] *= sc;
#pragma unroll
      for (int i = 0; i < C * (C - 1) / 2; ++i) R.o[i] = cscale(R.o[i], sc);
    }
    // the start vector at unit length, so that its size does not reach the powers
    {
      float big = 0.0f;
#pragma unroll
      for (int c = 0; c < C; ++c) big = fmaxf(big, fmaxf(fabsf(v[c].x), fabsf(v[c].y)));
      const float inv = 1.0f / big;
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = cscale(v[c], inv);
      normalise<C>(v);
    }
    int left = iterations;
    bool fourth = false;
#pragma unroll 1
    while (left > 0 && !fourth) {
      hermitian_apply<C>(R, v, u);
      float n = norm2<C>(u);
      const bool fits = n >= kWalshSquareNorm;
      if (n < 0x1p-100f) {  // squares may have underflowed
#pragma unroll
        for (int c = 0; c < C; ++c) u[c] = cscale(u[c], 0x1p100f);
        n = norm2<C>(u);
      }
      if (!(n > 0.0f)) break;  // R takes it to nothing: it stays
      const float inv = rsqrtf(n);
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = cscale(u[c], inv);
      --left;
      fourth = left >= kWalshSquare && (left & 3) == 0 && fits;
    }
    if (left == iterations) {  // (its first product: the start vector as it came)
      const bool some = norm2<C>(own) > 0.0f;
#pragma unroll
      for (int c = 0; c < C; ++c) v[c] = some ? own[c] : make_float2(c == 0 ? 1.0f : 0.0f, 0.0f);
    }
    if (fourth) {
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        Hermitian<C> s;
        hermitian_square<C>(R, s);
        R = s;
      }
#pragma unroll 1
      for (; left > 0; left -= 4) {
        hermitian_apply<C>(R, v, u);
#pragma unroll
        for (int c = 0; c < C; ++c) v[c] = u[c];
        normalise<C>(v);
      }
    }
  }
  // phase reference: coil 0's weight real and non-negative
  const float m0 = sqrtf(v[0].x * v[0].x + v[0].y * v[0].y);
  float2 ph = m0 > 0.0f ? make_float2(v[0].x / m0, -v[0].y / m0) : make_float2(1.0f, 0.0f);
  float2 acc = make_float2(0.0f, 0.0f);
#pragma unroll
  for (int c = 0; c < C; ++c) {
    const float2 w = cmul(v[c], ph);
    // conj(w) x
    acc.x = fmaf(w.x, own[c].x, fmaf(w.y, own[c].y, acc.x));
    acc.y = fmaf(w.x, own[c].y, fmaf(-w.y, own[c].x, acc.y));
  }
  out[static_cast<size_t>(r) * cols + cc] = acc;
}

template <int C>
ksj_gpu_status launch_walsh(uint32_t rows, uint32_t cols, int half, uint32_t iterations, const void* in, void* out,
                            cudaStream_t stream) {
  const int span = kWalshCols + 2 * half, tall = kWalshRows + 2 * half;
  const size_t smem = static_cast<size_t>(span) * C * (tall * sizeof(float2) + kWalshRows * C * sizeof(float));
  KSJ_TRY(allow_smem(k_walsh<C>, smem));
  const unsigned grid = ((cols + kWalshCols - 1) / kWalshCols) * ((rows + kWalshRows - 1) / kWalshRows);
  LaunchScope scope("k_walsh", stream);
  KSJ_TRY(launch_chained(k_walsh<C>, dim3(grid), dim3(kWalshThreads), smem, stream, static_cast<const float2*>(in),
                 static_cast<float2*>(out), static_cast<int>(rows), static_cast<int>(cols), half,
                 static_cast<int>(iterations)));
  return check_launch();
}

}  // namespace
}  // namespace ksj_gpu

using namespace ksj_gpu;

extern "C" ksj_gpu_status ksj_gpu_walsh_combine(uint32_t rows, uint32_t cols, uint32_t channels, uint32_t window,
                                                uint32_t iterations, const void* d_coil_last, void* d_out,
                                                void* stream) {
  if (rows == 0 || cols == 0 || channels == 0 || d_coil_last == nullptr || d_out == nullptr)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if ((window & 1u) == 0 || window / 2 > static_cast<uint32_t>(kWalshMaxHalf) || iterations > 1000 ||
      rows > 65535u * 16 || cols > 65535u * 16)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const int half = static_cast<int>(window / 2);
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  switch (channels) {
    case 1: return launch_walsh<1>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 2: return launch_walsh<2>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 3: return launch_walsh<3>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 4: return launch_walsh<4>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 5: return launch_walsh<5>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 6: return launch_walsh<6>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 7: return launch_walsh<7>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    case 8: return launch_walsh<8>(rows, cols, half, iterations, d_coil_last, d_out, cs);
    default: return KSJ_GPU_ERROR_UNSUPPORTED;
  }
}

// ------------------------------------------------- coil covariance (tcgen05)
//
// R = (1/M) X X^H for X complex64 [C][M] (channel-major k-space), C <= 32,
// the covariance of coil_compression_basis_estimate.cpp:207-227.  As a real
// contraction: with A = [Re X; Im X] (64 x M), G = A A^T holds every term
// (R.re = G[i][j] + G[32+i][32+j], R.im = G[32+i][j] - G[i][32+j]).  Each
// element of A is split as hi + lo (both bf16, hi = bf16(a), lo = bf16(a - hi))
// and G ~= hi hi^T + lo hi^T + (lo hi^T)^T, every product accumulated in FP32
// by the tensor cores:
//   k_cov_mma     per block a range of 64-sample tiles of X: split in registers into the operand
//                 [hi(Re); hi(Im); lo(Re); lo(Im)] (128 rows of bf16) and stored to one of two
//                 shared-memory stages in the 128-byte swizzle, the next tile's samples already
//                 requested; one thread issues tcgen05.mma M=128 (the whole operand), N=64 (its hi
//                 rows, the same shared memory), K=16; the 128 x 64 FP32 accumulator lives in tensor
//                 memory and is read out once by four warps
//   k_cov_form    sums the blocks' accumulators in a fixed order; its last block forms R or the
//                 noise covariance (deterministic)

namespace ksj_gpu {
namespace {

constexpr int kCovRows = 128;
constexpr int kCovKTile = 64;  // samples per stage: 128 bytes of bf16 per operand row
constexpr int kCovStages = 2;
constexpr uint32_t kCovStageBytes = kCovRows * kCovKTile * 2;
constexpr int kCovThreads = 256;
constexpr uint32_t kCovWaitLimit = 1u << 22;
constexpr int kCovMaxBlocks = 2 * kSms;

// Four consecutive samples of one coil per thread and turn, two turns per tile
// (32 coils x 64 samples): eight 8-byte loads in flight, one 8-byte store per
// operand row and turn (a half-warp stores one row's 128 bytes).
constexpr int kCovQuad = 4;
constexpr int kCovTurns = 32 * kCovKTile / kCovQuad / kCovThreads;

// Shared-memory matrix descriptor of a K-major operand in the 128-byte swizzle
// layout (8-row x 128-byte atoms stacked 1024 bytes apart along M/N).
__device__ __forceinline__ uint64_t sw128_kmajor_desc(uint32_t saddr) {
  uint64_t d = static_cast<uint64_t>((saddr >> 4) & 0x3FFFu);  // start address
  d |= static_cast<uint64_t>(1) << 16;                          // leading byte offset (unused here): 16 B
  d |= static_cast<uint64_t>(1024 >> 4) << 32;                  // stride byte offset: 8 rows x 128 B
  d |= static_cast<uint64_t>(1) << 46;                          // descriptor version
  d |= static_cast<uint64_t>(2) << 61;                          // 128-byte swizzle
  return d;
}

// Instruction descriptor, kind::f16: FP32 accumulator, bf16 A and B, both
// K-major, N = 64, M = 128.
constexpr uint32_t kCovIdesc = (1u << 4) | (1u << 7) | (1u << 10) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                          uint32_t accumulate) {
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "setp.ne.b32 p, %4, 0;\n\t"
      "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
      ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
      : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
               : "memory");
}

__device__ __forceinline__ void tmem_ld16(uint32_t taddr, float* v) {
  uint32_t r[16];
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, "
      "[%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
#pragma unroll
  for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}

struct CovArgs {
  const float2* x;  // [channels][samples]
  float* partials;  // [blocks][128][64]
  uint32_t* flags;
  int channels, samples, ktiles;
};

// One tile's samples of this thread's quads (zero past the channels and samples).
__device__ __forceinline__ void cov_load(const CovArgs& a, int tile, float2 (&v)[kCovTurns][kCovQuad]) {
#pragma unroll
  for (int u = 0; u < kCovTurns; ++u) {
    const int q = threadIdx.x + u * kCovThreads;
    const int c = q / (kCovKTile / kCovQuad);
    const int s0 = tile * kCovKTile + (q % (kCovKTile / kCovQuad)) * kCovQuad;
    const float2* src = a.x + static_cast<size_t>(c) * a.samples + s0;
#pragma unroll
    for (int i = 0; i < kCovQuad; ++i)
      v[u][i] = c < a.channels && s0 + i < a.samples ? __ldg(src + i) : make_float2(0.0f, 0.0f);
  }
}

// Split into hi and lo and stored: operand row r at r * 128 bytes, its 16-byte
// chunk k at k ^ (r mod 8) (the 128-byte swizzle of a 1024-byte aligned stage).
__device__ __forceinline__ void cov_store(unsigned char* stage, const float2 (&v)[kCovTurns][kCovQuad]) {
#pragma unroll
  for (int u = 0; u < kCovTurns; ++u) {
    const int q = threadIdx.x + u * kCovThreads;
    const int c = q / (kCovKTile / kCovQuad), quad = q % (kCovKTile / kCovQuad);
    uint32_t h[2][2], l[2][2];  // [Re, Im][pair of samples]
#pragma unroll
    for (int i = 0; i < 2; ++i) {
      const float2 p = v[u][2 * i], n = v[u][2 * i + 1];
      const __nv_bfloat162 hr = __floats2bfloat162_rn(p.x, n.x), hi = __floats2bfloat162_rn(p.y, n.y);
      const __nv_bfloat162 lr = __floats2bfloat162_rn(p.x - __low2float(hr), n.x - __high2float(hr));
      const __nv_bfloat162 li = __floats2bfloat162_rn(p.y - __low2float(hi), n.y - __high2float(hi));
      h[0][i] = *reinterpret_cast<const uint32_t*>(&hr);
      h[1][i] = *reinterpret_cast<const uint32_t*>(&hi);
      l[0][i] = *reinterpret_cast<const uint32_t*>(&lr);
      l[1][i] = *reinterpret_cast<const uint32_t*>(&li);
    }
    // rows c, 32 + c, 64 + c and 96 + c: the same row mod 8
    unsigned char* dst = stage + c * 128 + (((quad >> 1) ^ (c & 7)) << 4) + ((quad & 1) << 3);
#pragma unroll
    for (int part = 0; part < 2; ++part) {
      *reinterpret_cast<uint2*>(dst + part * 32 * 128) = make_uint2(h[part][0], h[part][1]);
      *reinterpret_cast<uint2*>(dst + (2 + part) * 32 * 128) = make_uint2(l[part][0], l[part][1]);
    }
  }
}

// Bound by reading X once: 412160 samples x 32 coils (105 MB) in 27 us; splitting into a
// bf16 operand in memory first (another 105 MB written and read) took 58.
__global__ void __launch_bounds__(kCovThreads, 2) k_cov_mma(CovArgs a) {
  chain_begin();
  extern __shared__ __align__(16) unsigned char cov_smem[];
  // stage buffers on a 1024-byte boundary (128-byte swizzle atoms)
  unsigned char* base = cov_smem + ((1024u - (smem_addr(cov_smem) & 1023u)) & 1023u);
  __shared__ __align__(8) uint64_t empty[kCovStages], done;
  __shared__ uint32_t tmem_base;
  __shared__ int failed;
  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int t0 = static_cast<int>(static_cast<long long>(a.ktiles) * blockIdx.x / gridDim.x);
  const int t1 = static_cast<int>(static_cast<long long>(a.ktiles) * (blockIdx.x + 1) / gridDim.x);
  const int n = t1 - t0;
  if (tid == 0) {
    for (int s = 0; s < kCovStages; ++s) mbar_init(&empty[s], 1);
    mbar_init(&done, 1);
    mbar_init_fence();
    failed = 0;
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 64;" ::"r"(smem_addr(&tmem_base))
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  const uint32_t tmem = tmem_base;

  float2 v[kCovTurns][kCovQuad];
  if (n > 0) cov_load(a, t0, v);
  bool ok = true;
  for (int i = 0; i < n; ++i) {
    const int s = i & 1;
    unsigned char* stage = base + s * kCovStageBytes;
    // the stage's previous tile must have been consumed by its MMAs
    if (i >= kCovStages) ok = mbar_wait_bounded(&empty[s], ((i >> 1) - 1) & 1, kCovWaitLimit);
    if (ok) cov_store(stage, v);
    if (i + 1 < n) cov_load(a, t0 + i + 1, v);
    fence_proxy_async_shared();  // the stores, before the MMAs read them
    ok = __syncthreads_and(ok);
    if (!ok) break;
    if (tid == 0) {
      asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
      const uint32_t sa = smem_addr(stage);
#pragma unroll
      for (int k = 0; k < kCovKTile / 16; ++k) {
        const uint64_t d = sw128_kmajor_desc(sa + k * 32);
        umma_bf16(tmem, d, d, kCovIdesc, (i > 0 || k > 0) ? 1u : 0u);
      }
      umma_commit(&empty[s]);
    }
  }
  if (tid == 0) {
    // every MMA issued so far completes before `done` fires
    umma_commit(&done);
    const bool fin = mbar_wait_bounded(&done, 0, kCovWaitLimit);
    if (!ok || !fin) {
      failed = 1;
      atomicOr(a.flags, KSJ_GPU_FLAG_WAIT_TIMEOUT);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
  if (!failed && warp < 4) {
    // accumulator row 32*warp + lane, 64 FP32 columns
    const int row = warp * 32 + (tid & 31);
    float* dst = a.partials + (static_cast<size_t>(blockIdx.x) * kCovRows + row) * 64;
#pragma unroll
    for (int c = 0; c < 64; c += 16) {
      float w[16];
      tmem_ld16(tmem + (static_cast<uint32_t>(warp * 32) << 16) + c, w);
      asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
      if (n == 0) {
#pragma unroll
        for (int i = 0; i < 16; ++i) w[i] = 0.0f;
      }
#pragma unroll
      for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(dst + c + i) = make_float4(w[i], w[i + 1], w[i + 2], w[i + 3]);
    }
  }
  asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
  __syncthreads();
  if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 64;" ::"r"(tmem) : "memory");
}

// The covariance from the blocks' accumulators.  Each block sums 32
// accumulator elements, eight threads an element over an eighth of the blocks'
// copies each (in block order, the eighths then added in order: deterministic,
// and eight short chains of loads where one per element waited out all of
// them); the last block to finish forms the elements of R or of the noise covariance.
//
// G = hi hi^T + lo hi^T + (lo hi^T)^T, R = G times 1/M (in float, as the
// reference scales its sums).  The lower triangle is computed and the upper
// mirrored (conjugate), as the reference stores it, so R is Hermitian bit for bit.
//
// means non-null: the noise covariance of noise_model_estimate.cpp:161-162
// (covariance_channel_major_with_workspace, population normalisation,
// moments.hpp:99-140), C(r, c) = (1/M) sum_s conj(x_r - mu_r) (x_c - mu_c)
// = conj(R(r, c) - mu_r conj(mu_c)); lower triangle computed, upper mirrored.
constexpr int kCovSumElems = 32, kCovSumSlices = 8;
static_assert(kCovRows * 64 % kCovSumElems == 0, "whole blocks of elements");

__global__ void __launch_bounds__(kCovSumElems * kCovSumSlices) k_cov_form(const float* partials, int blocks, float* sum,
                                                                           uint32_t* finished, int channels,
                                                                           float inv_m,
                                                                           const float2* __restrict__ means,
                                                                           float2* cov) {
  chain_begin();
  __shared__ float part[kCovSumSlices][kCovSumElems];
  __shared__ bool last;
  const int el = threadIdx.x % kCovSumElems, slice = threadIdx.x / kCovSumElems;
  const int e = blockIdx.x * kCovSumElems + el;
  const int b0 = blocks * slice / kCovSumSlices, b1 = blocks * (slice + 1) / kCovSumSlices;
  float s = 0.0f;
#pragma unroll 20
  for (int b = b0; b < b1; ++b) s += __ldg(partials + static_cast<size_t>(b) * kCovRows * 64 + e);
  part[slice][el] = s;
  __syncthreads();
  if (slice == 0) {
    for (int k = 1; k < kCovSumSlices; ++k) s += part[k][el];
    sum[e] = s;
    __threadfence();
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    last = atomicAdd(finished, 1u) == gridDim.x - 1;
    __threadfence();
  }
  __syncthreads();
  if (!last) return;
  auto g = [&](int r, int c) {
    return __ldcg(sum + r * 64 + c) + __ldcg(sum + (64 + r) * 64 + c) + __ldcg(sum + (64 + c) * 64 + r);
  };
  for (int idx = threadIdx.x; idx < channels * channels; idx += blockDim.x) {
    const int i = idx / channels, j = idx - (idx / channels) * channels;
    const int r = i >= j ? i : j, c = i >= j ? j : i;
    const float re = (g(r, c) + g(32 + r, 32 + c)) * inv_m;
    const float im = r == c ? 0.0f : (g(32 + r, c) - g(r, 32 + c)) * inv_m;
    if (means == nullptr) {
      cov[idx] = make_float2(re, i >= j ? im : -im);
    } else {
      const float2 mr = means[r], mc = means[c];
      // d = R(r, c) - mu_r conj(mu_c); C(r, c) = conj(d), C(c, r) = d
      const float dre = re - (mr.x * mc.x + mr.y * mc.y);
      const float dim = r == c ? 0.0f : im - (mr.y * mc.x - mr.x * mc.y);
      cov[idx] = make_float2(dre, i >= j ? -dim : dim);
    }
  }
}

// Per-channel mean of channel-major X [channels][samples] (one block per
// channel, a fixed-order tree over the block: deterministic), as
// covariance_channel_major_with_workspace forms it (moments.hpp:117-123).
__global__ void __launch_bounds__(256) k_channel_means(const float2* __restrict__ x, int samples, float2* means) {
  __shared__ float2 part[256];
  const float2* row = x + static_cast<size_t>(blockIdx.x) * samples;
  float2 acc = make_float2(0.0f, 0.0f);
  for (int s = threadIdx.x; s < samples; s += blockDim.x) {
    const float2 v = __ldg(row + s);
    acc.x += v.x;
    acc.y += v.y;
  }
  part[threadIdx.x] = acc;
  __syncthreads();
  for (int h = blockDim.x >> 1; h > 0; h >>= 1) {
    if (threadIdx.x < h) {
      part[threadIdx.x].x += part[threadIdx.x + h].x;
      part[threadIdx.x].y += part[threadIdx.x + h].y;
    }
    __syncthreads();
  }
  if (threadIdx.x == 0) {
    const float inv = 1.0f / static_cast<float>(samples);
    means[blockIdx.x] = make_float2(part[0].x * inv, part[0].y * inv);
  }
}

struct CovLayout {
  size_t flags, partials, sum, means, total;
  int ktiles, blocks;
};

CovLayout cov_layout(uint32_t samples) {
  CovLayout l{};
  l.ktiles = static_cast<int>((samples + kCovKTile - 1) / kCovKTile);
  l.blocks = std::min(l.ktiles, kCovMaxBlocks);
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  l.flags = take(16);  // check flags, then the count of finished k_cov_form blocks
  l.partials = take(static_cast<size_t>(l.blocks) * kCovRows * 64 * sizeof(float));
  l.sum = take(static_cast<size_t>(kCovRows) * 64 * sizeof(float));
  l.means = take(32 * sizeof(float2));
  l.total = off;
  return l;
}

}  // namespace
}  // namespace ksj_gpu

extern "C" size_t ksj_gpu_coil_covariance_workspace_bytes(uint32_t channels, uint32_t samples) {
  if (channels == 0 || channels > 32 || samples == 0 || samples > (1u << 28)) return 0;
  return ksj_gpu::cov_layout(samples).total;
}

namespace ksj_gpu {
namespace {

// X [channels][samples] -> the summed split-BF16 products (tensor cores), then
// either R = (1/M) X X^H (noise = false) or the mean-removed noise covariance
// in the reference's convention (noise = true) into d_cov.
ksj_gpu_status covariance_run(uint32_t channels, uint32_t samples, const void* d_kspace, void* d_cov,
                              void* d_workspace, size_t workspace_bytes, void* stream, bool noise) {
  if (channels == 0 || channels > 32 || samples == 0 || samples > (1u << 28) || d_kspace == nullptr ||
      d_cov == nullptr || (reinterpret_cast<uintptr_t>(d_kspace) & 7u) != 0 ||
      (reinterpret_cast<uintptr_t>(d_cov) & 7u) != 0)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const CovLayout l = cov_layout(samples);
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < l.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + l.flags);
  float* partials = reinterpret_cast<float*>(ws + l.partials);
  if (cudaMemsetAsync(flags, 0, 16, cs) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  const size_t smem = 1024 + static_cast<size_t>(kCovStages) * kCovStageBytes;
  {
    const CovArgs args{static_cast<const float2*>(d_kspace), partials, flags, static_cast<int>(channels),
                       static_cast<int>(samples), l.ktiles};
    LaunchScope scope("k_cov_mma", cs);
    KSJ_TRY(launch_chained(k_cov_mma, dim3(l.blocks), dim3(kCovThreads), smem, cs, args));
  }
  float2* means = nullptr;
  if (noise) {
    means = reinterpret_cast<float2*>(ws + l.means);
    LaunchScope scope("k_channel_means", cs);
    k_channel_means<<<channels, 256, 0, cs>>>(static_cast<const float2*>(d_kspace), static_cast<int>(samples), means);
    KSJ_TRY(check_launch());
  }
  LaunchScope scope("k_cov_form", cs);
  KSJ_TRY(launch_chained(k_cov_form, dim3(kCovRows * 64 / kCovSumElems), dim3(kCovSumElems * kCovSumSlices), 0, cs, partials,
                 l.blocks, reinterpret_cast<float*>(ws + l.sum), flags + 1, static_cast<int>(channels),
                 1.0f / static_cast<float>(samples), means, static_cast<float2*>(d_cov)));
  return check_launch();
}

}  // namespace
}  // namespace ksj_gpu

extern "C" ksj_gpu_status ksj_gpu_coil_covariance(uint32_t channels, uint32_t samples, const void* d_kspace,
                                                  void* d_cov, void* d_workspace, size_t workspace_bytes,
                                                  void* stream) {
  return ksj_gpu::covariance_run(channels, samples, d_kspace, d_cov, d_workspace, workspace_bytes, stream, false);
}

extern "C" ksj_gpu_status ksj_gpu_noise_covariance(uint32_t channels, uint32_t samples, const void* d_noise,
                                                   void* d_cov, void* d_workspace, size_t workspace_bytes,
                                                   void* stream) {
  return ksj_gpu::covariance_run(channels, samples, d_noise, d_cov, d_workspace, workspace_bytes, stream, true);
}

// ------------------------------------------------- coil compression basis and apply

namespace ksj_gpu {
namespace {

// Y[v][s] = sum_c B[v][c] X[c][s] (noncartesian_coil_compress.cpp:143-148), the
// kV outputs of kS consecutive samples in a thread's registers, B in shared
// memory as [channel][output], two outputs per 16-byte load.
//
// 32 -> 8 is bound by HBM (132 MB), 32 x 32 by the FP32 pipe (1.69 G multiply-adds, 45 us at 128 per clock
// and SM): each load of B serves kS samples, and each thread has the samples of
// kAheadC channels in flight (one sample and one channel at a time measured 40
// and 114 us at 412160 samples, 150 for the two in turn; this 107 for the two).
constexpr int kAheadC = 4;

// threads of a block: fewer where the outputs take more than half the registers
__host__ __device__ constexpr int compress_threads(int v) { return v > 16 ? 128 : 256; }

template <int kV, int kS>
__global__ void __launch_bounds__(compress_threads(kV)) k_coil_compress(const float2* __restrict__ basis,
                                                                        const float2* __restrict__ x, float2* y,
                                                                        int channels, int samples) {
  chain_begin();
  constexpr int kP = (kV + 1) / 2;  // pairs of outputs
  __shared__ float4 b[32 * kP];
  for (int i = threadIdx.x; i < 32 * kP * 2; i += blockDim.x) {
    const int c = i / (2 * kP), v = i - c * (2 * kP);
    reinterpret_cast<float2*>(b)[i] = c < channels && v < kV ? basis[v * channels + c] : make_float2(0.0f, 0.0f);
  }
  __syncthreads();
  const size_t s = (static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x) * kS;
  if (s >= static_cast<size_t>(samples)) return;
  float2 acc[kV][kS];
#pragma unroll
  for (int v = 0; v < kV; ++v)
#pragma unroll
    for (int k = 0; k < kS; ++k) acc[v][k] = make_float2(0.0f, 0.0f);
  for (int c0 = 0; c0 < channels; c0 += kAheadC) {
    float2 xv[kAheadC][kS];
#pragma unroll
    for (int u = 0; u < kAheadC; ++u) {
      const float2* src = x + static_cast<size_t>(c0 + u) * samples + s;
      if constexpr (kS == 2) {
        const float4 q = c0 + u < channels ? __ldg(reinterpret_cast<const float4*>(src)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        xv[u][0] = make_float2(q.x, q.y);
        xv[u][1] = make_float2(q.z, q.w);
      } else {
        xv[u][0] = c0 + u < channels ? __ldg(src) : make_float2(0.0f, 0.0f);
      }
    }
#pragma unroll
    for (int u = 0; u < kAheadC; ++u) {
      if (c0 + u >= channels) break;
#pragma unroll
      for (int q = 0; q < kP; ++q) {
        const float4 w2 = b[(c0 + u) * kP + q];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
          if (2 * q + h >= kV) continue;
          const float2 w = h ? make_float2(w2.z, w2.w) : make_float2(w2.x, w2.y);
#pragma unroll
          for (int k = 0; k < kS; ++k) {
            float2& o = acc[2 * q + h][k];
            o.x = fmaf(w.x, xv[u][k].x, fmaf(-w.y, xv[u][k].y, o.x));
            o.y = fmaf(w.x, xv[u][k].y, fmaf(w.y, xv[u][k].x, o.y));
          }
        }
      }
    }
  }
#pragma unroll
  for (int v = 0; v < kV; ++v) {
    float2* dst = y + static_cast<size_t>(v) * samples + s;
    if constexpr (kS == 2)
      *reinterpret_cast<float4*>(dst) = make_float4(acc[v][0].x, acc[v][0].y, acc[v][1].x, acc[v][1].y);
    else
      *dst = acc[v][0];
  }
}

// Two samples per thread where every row starts on 16 bytes (an even sample
// count and aligned arrays), else one.
template <int kV>
ksj_gpu_status launch_compress(uint32_t channels, uint32_t samples, const void* basis, const void* x, void* y,
                               cudaStream_t stream) {
  const bool pairs = samples % 2 == 0 && (reinterpret_cast<uintptr_t>(x) & 15u) == 0 &&
                     (reinterpret_cast<uintptr_t>(y) & 15u) == 0;
  const auto kernel = pairs ? k_coil_compress<kV, 2> : k_coil_compress<kV, 1>;
  const uint32_t per_block = compress_threads(kV) * (pairs ? 2 : 1);
  LaunchScope scope("k_coil_compress", stream);
  KSJ_TRY(launch_chained(kernel, dim3((samples + per_block - 1) / per_block), dim3(compress_threads(kV)), 0, stream,
      static_cast<const float2*>(basis), static_cast<const float2*>(x), static_cast<float2*>(y),
      static_cast<int>(channels), static_cast<int>(samples)));
  return check_launch();
}

}  // namespace
}  // namespace ksj_gpu

// Cyclic Jacobi for a Hermitian matrix (host, double precision).  For each
// pair (p, q): a phase on index q makes a_pq real and positive, then a real
// plane rotation zeroes it (the symmetric Jacobi step).  `a` and `vec` are
// row-major n x n; on return the diagonal of `a` holds the eigenvalues and
// the columns of `vec` the eigenvectors.
static void hermitian_jacobi(int n, std::complex<double>* a, std::complex<double>* vec) {
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) vec[i * n + j] = i == j ? 1.0 : 0.0;
  double total = 0.0;
  for (int i = 0; i < n * n; ++i) total += std::norm(a[i]);
  for (int sweep = 0; sweep < 64; ++sweep) {
    double off = 0.0;
    for (int p = 0; p < n; ++p)
      for (int q = p + 1; q < n; ++q) off += std::norm(a[p * n + q]);
    if (off <= 1e-32 * total) break;
    for (int p = 0; p < n; ++p) {
      for (int q = p + 1; q < n; ++q) {
        const double r = std::abs(a[p * n + q]);
        if (r <= 1e-300) continue;
        const std::complex<double> e = a[p * n + q] / r;
        for (int k = 0; k < n; ++k) {
          a[k * n + q] *= std::conj(e);
          vec[k * n + q] *= std::conj(e);
        }
        for (int k = 0; k < n; ++k) a[q * n + k] *= e;
        const double theta = (a[q * n + q].real() - a[p * n + p].real()) / (2.0 * r);
        const double t = (theta >= 0.0 ? 1.0 : -1.0) / (std::fabs(theta) + std::sqrt(theta * theta + 1.0));
        const double c = 1.0 / std::sqrt(t * t + 1.0), s = t * c;
        for (int k = 0; k < n; ++k) {
          const std::complex<double> kp = a[k * n + p], kq = a[k * n + q];
          a[k * n + p] = c * kp - s * kq;
          a[k * n + q] = s * kp + c * kq;
        }
        for (int k = 0; k < n; ++k) {
          const std::complex<double> pk = a[p * n + k], qk = a[q * n + k];
          a[p * n + k] = c * pk - s * qk;
          a[q * n + k] = s * pk + c * qk;
        }
        for (int k = 0; k < n; ++k) {
          const std::complex<double> vp = vec[k * n + p], vq = vec[k * n + q];
          vec[k * n + p] = c * vp - s * vq;
          vec[k * n + q] = s * vp + c * vq;
        }
      }
    }
  }
}

using namespace ksj_gpu;

extern "C" ksj_gpu_status ksj_coil_compression_basis(uint32_t channels, uint32_t virtual_channels,
                                                     const void* covariance, void* basis, float* eigenvalues) {
  if (channels == 0 || channels > 64 || virtual_channels == 0 || virtual_channels > channels ||
      covariance == nullptr || basis == nullptr)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const int n = static_cast<int>(channels);
  const float* cov = static_cast<const float*>(covariance);
  std::vector<std::complex<double>> a(static_cast<size_t>(n) * n), vec(static_cast<size_t>(n) * n);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      // Hermitian part of the input (the lower triangle mirrored, as the reference stores it)
      const int lo = i >= j ? i * n + j : j * n + i;
      const std::complex<double> v(cov[2 * lo], cov[2 * lo + 1]);
      a[static_cast<size_t>(i) * n + j] = i >= j ? v : std::conj(v);
      if (!std::isfinite(v.real()) || !std::isfinite(v.imag())) return KSJ_GPU_ERROR_NONFINITE_INPUT;
    }
  hermitian_jacobi(n, a.data(), vec.data());
  std::vector<int> order(static_cast<size_t>(n));
  for (int i = 0; i < n; ++i) order[i] = i;
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
    return a[static_cast<size_t>(x) * n + x].real() > a[static_cast<size_t>(y) * n + y].real();
  });
  float* out = static_cast<float*>(basis);
  for (uint32_t v = 0; v < virtual_channels; ++v) {
    const int col = order[v];
    for (int c = 0; c < n; ++c) {
      // basis row v = conj(eigenvector), largest eigenvalue first (coil_compression_basis_estimate.cpp:233-239)
      const std::complex<double> e = std::conj(vec[static_cast<size_t>(c) * n + col]);
      out[2 * (v * n + c)] = static_cast<float>(e.real());
      out[2 * (v * n + c) + 1] = static_cast<float>(e.imag());
    }
  }
  if (eigenvalues != nullptr)
    for (int i = 0; i < n; ++i) eigenvalues[i] = static_cast<float>(a[static_cast<size_t>(order[i]) * n + order[i]].real());
  return KSJ_GPU_OK;
}

extern "C" ksj_gpu_status ksj_gpu_coil_compress(uint32_t channels, uint32_t virtual_channels, uint32_t samples,
                                                const void* d_basis, const void* d_kspace, void* d_out,
                                                void* stream) {
  if (channels == 0 || channels > 32 || virtual_channels == 0 || virtual_channels > 16 ||
      virtual_channels > channels || samples == 0 || d_basis == nullptr || d_kspace == nullptr || d_out == nullptr)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  switch (virtual_channels) {
#define KSJ_COMPRESS_CASE(V) \
  case V: return launch_compress<V>(channels, samples, d_basis, d_kspace, d_out, cs);
    KSJ_COMPRESS_CASE(1) KSJ_COMPRESS_CASE(2) KSJ_COMPRESS_CASE(3) KSJ_COMPRESS_CASE(4)
    KSJ_COMPRESS_CASE(5) KSJ_COMPRESS_CASE(6) KSJ_COMPRESS_CASE(7) KSJ_COMPRESS_CASE(8)
    KSJ_COMPRESS_CASE(9) KSJ_COMPRESS_CASE(10) KSJ_COMPRESS_CASE(11) KSJ_COMPRESS_CASE(12)
    KSJ_COMPRESS_CASE(13) KSJ_COMPRESS_CASE(14) KSJ_COMPRESS_CASE(15) KSJ_COMPRESS_CASE(16)
#undef KSJ_COMPRESS_CASE
    default: return KSJ_GPU_ERROR_UNSUPPORTED;
  }
}

// Whitening matrix of a noise covariance (noise_model_estimate.cpp:163-167,
// whitening.hpp:27-51): W = V diag(1 / sqrt(max(lambda, floor))) V^H over the
// eigenpairs of the Hermitian covariance (double-precision cyclic Jacobi),
// W(r, c) = sum_k V(r, k) / sqrt(max(lambda_k, floor)) conj(V(c, k)).
extern "C" ksj_gpu_status ksj_whitening_matrix(uint32_t channels, const void* covariance, float eigenvalue_floor,
                                               void* whitening) {
  if (channels == 0 || channels > 64 || covariance == nullptr || whitening == nullptr || !(eigenvalue_floor > 0.0f))
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const int n = static_cast<int>(channels);
  const float* cov = static_cast<const float*>(covariance);
  std::vector<std::complex<double>> a(static_cast<size_t>(n) * n), vec(static_cast<size_t>(n) * n);
  for (int i = 0; i < n; ++i)
    for (int j = 0; j < n; ++j) {
      const int lo = i >= j ? i * n + j : j * n + i;
      const std::complex<double> v(cov[2 * lo], cov[2 * lo + 1]);
      if (!std::isfinite(v.real()) || !std::isfinite(v.imag())) return KSJ_GPU_ERROR_NONFINITE_INPUT;
      a[static_cast<size_t>(i) * n + j] = i >= j ? v : std::conj(v);
    }
  hermitian_jacobi(n, a.data(), vec.data());
  std::vector<double> scale(static_cast<size_t>(n));
  for (int k = 0; k < n; ++k)
    scale[k] = 1.0 / std::sqrt(std::max(a[static_cast<size_t>(k) * n + k].real(), static_cast<double>(eigenvalue_floor)));
  float* out = static_cast<float*>(whitening);
  for (int r = 0; r < n; ++r)
    for (int c = 0; c < n; ++c) {
      std::complex<double> sum = 0.0;
      for (int k = 0; k < n; ++k)
        sum += vec[static_cast<size_t>(r) * n + k] * scale[k] * std::conj(vec[static_cast<size_t>(c) * n + k]);
      out[2 * (r * n + c)] = static_cast<float>(sum.real());
      out[2 * (r * n + c) + 1] = static_cast<float>(sum.imag());
    }
  return KSJ_GPU_OK;
}

// Y = W X (noncartesian_noise_prewhiten.cpp:140-146): the square form of the
// compression apply, W complex64 [channels][channels].
extern "C" ksj_gpu_status ksj_gpu_noise_prewhiten(uint32_t channels, uint32_t samples, const void* d_whitening,
                                                  const void* d_kspace, void* d_out, void* stream) {
  if (channels == 0 || channels > 32 || samples == 0 || d_whitening == nullptr || d_kspace == nullptr ||
      d_out == nullptr)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  switch (channels) {
#define KSJ_WHITEN_CASE(V) \
  case V: return launch_compress<V>(channels, samples, d_whitening, d_kspace, d_out, cs);
    KSJ_WHITEN_CASE(1) KSJ_WHITEN_CASE(2) KSJ_WHITEN_CASE(3) KSJ_WHITEN_CASE(4)
    KSJ_WHITEN_CASE(5) KSJ_WHITEN_CASE(6) KSJ_WHITEN_CASE(7) KSJ_WHITEN_CASE(8)
    KSJ_WHITEN_CASE(9) KSJ_WHITEN_CASE(10) KSJ_WHITEN_CASE(11) KSJ_WHITEN_CASE(12)
    KSJ_WHITEN_CASE(13) KSJ_WHITEN_CASE(14) KSJ_WHITEN_CASE(15) KSJ_WHITEN_CASE(16)
    KSJ_WHITEN_CASE(17) KSJ_WHITEN_CASE(18) KSJ_WHITEN_CASE(19) KSJ_WHITEN_CASE(20)
    KSJ_WHITEN_CASE(21) KSJ_WHITEN_CASE(22) KSJ_WHITEN_CASE(23) KSJ_WHITEN_CASE(24)
    KSJ_WHITEN_CASE(25) KSJ_WHITEN_CASE(26) KSJ_WHITEN_CASE(27) KSJ_WHITEN_CASE(28)
    KSJ_WHITEN_CASE(29) KSJ_WHITEN_CASE(30) KSJ_WHITEN_CASE(31) KSJ_WHITEN_CASE(32)
#undef KSJ_WHITEN_CASE
    default: return KSJ_GPU_ERROR_UNSUPPORTED;
  }
}
