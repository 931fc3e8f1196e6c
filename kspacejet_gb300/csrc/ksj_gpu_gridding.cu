// ksj_gpu_gridding.cu -- adjoint gridding reconstruction on sm_103a.
//
// One call reconstructs `frames` independent frames of `channels` coils:
//
//   k_prepare  per (frame, sample): error-free grid coordinate, taps and
//              weights (linear or Kaiser-Bessel), accurately reduced origin
//              phase times the DCF; per block of consecutive samples a count
//              for every binning list
//   k_bin_prefix  per list: each block's start among the list's entries, and the
//              list's length
//   k_scan     per frame: exclusive scan of the list lengths; in further blocks
//              the call's tables (quarter-turn-reduced FFT twiddles, FP64
//              Kaiser-Bessel deapodisation factors)
//   k_place    per block of samples: every sample's entries straight into their
//              places, in sample order, so every cell later accumulates in
//              sample order -- the reference's order -- and the result is
//              deterministic
//   (3-D: the same twice over, first the samples of every grid plane, then
//              each plane's samples as a frame's)
//   k_samples_coil_last  [frame][coil][sample] -> [frame][sample][coil] times
//              the sample's weight and phase, so the row pass reads one
//              sample's coils as one coalesced segment
//   k_rows     per (frame, grid row, coil group): groups of lanes (lane =
//              coil) take the row's lists, one 16-column chunk each,
//              and sum its cells in registers with no atomics (a cell is
//              only ever touched by its owning group, in list order); the block
//              then runs the row inverse FFT of every coil line in place and
//              writes only the columns the image keeps, coil-last
//              ([frame][grid row][column][channel]), so the column pass
//              reads every coil of a column as one tile
//   k_cols     per (frame, column block): one TMA tile of all grid rows x
//              columns x a group of coils, column inverse FFT in place, crop,
//              deapodise, then write coil-last images or sum |x|^2 over coils
//              in channel order (the reference RSS order and rounding)
//   k_images_coil_major  coil-last -> coil-major transpose when asked for
//
// Binning lists are (frame, grid row, 16-column chunk); a sample is listed
// once per row its stencil covers and per chunk its W columns fall into
// (one or two; three where the last chunk of a row is narrower than a stencil's inner
// columns, which then reach over it into the first).  The "reference permutation" a list must equal is the
// increasing sequence of sample indices whose stencil touches that row and
// chunk, with the lower tap index floor(k N / 2 pi) of the exact coordinate
// (the value the reference's double-precision grid_coordinate computes,
// eigen_radial_gridding.cpp:262-277).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>
#include <mutex>
#include <map>
#include <tuple>
#include <type_traits>
#include <vector>

#include "ksj_gpu.h"
#include "ksj_gpu_internal.cuh"

namespace ksj_gpu {
namespace {

constexpr int kChunk = 16;        // grid columns per binning list (<= 32 lists per row)
constexpr int kMaxWidth = 8;      // largest Kaiser-Bessel width
constexpr int kMaxGrid = 512;
constexpr int kColsThreads = 256;  // k_cols block size
constexpr int kRowsThreads = 384;  // most threads of a k_rows block (two such blocks per SM)
constexpr int kRowsBatch = 8;      // list entries a lane group stages and loads samples for at once
constexpr uint32_t kFlagBytes = 256;

// Per (frame, sample) record written by k_prepare, read by k_rows.
template <int W>
struct alignas(16) SampleRecord {
  int r0;        // first tap row (wrapped)
  int c0;        // first tap column (wrapped)
  float2 scale;  // dcf * exp(i * origin phase)
  float wr[W];
  float wc[W];
};

// Per sample record of the 3-D path: first tap plane/row/column (wrapped),
// dcf * phase, and the W tap weights along z, y and x.
template <int W>
struct alignas(16) SampleRecord3 {
  int z0, r0, c0, pad;
  float2 scale;
  float wz[W];
  float wr[W];
  float wc[W];
};

// One list entry as the row pass reads it: the first tap's column as
// seen from the list's chunk (-7 .. 15; a row length lower when the taps reaching
// the chunk wrapped past the last column), the sample index, and the W column
// weights times the list's row (and plane) weight.
__host__ __device__ constexpr int entry_bytes(int w) { return 8 + 4 * w; }
// Widths 2 and 6 are stored and loaded in 16-byte vectors (24-byte entries padded
// to 32 for the same cost the row pass 2 % more than they saved).
__host__ __device__ constexpr bool entry_vectors(int w) { return entry_bytes(w) % 16 == 0; }

// A staged entry in shared memory: the 16 weights of the chunk's columns (zero
// where no tap falls), then the sample index.  80 bytes apart, so that lanes
// writing or reading the same word of consecutive entries meet different banks.
constexpr int kSlotFloats = 20;

// Shared memory of one k_rows block: accumulators, twiddles and the staged
// entries of every lane group.  Lane groups
// are the lanes of a coil group's part: lanes = coil_group / coil_parts.
inline size_t rows_smem_for(int grid_cols, int cg, int lanes, int threads) {
  const size_t head = static_cast<size_t>(grid_cols) * (cg + 1) * 8;
  return ((head + 15) & ~size_t{15}) + static_cast<size_t>(threads / lanes) * kRowsBatch * kSlotFloats * 4;
}
// Threads of a k_rows block: enough for the transform's first step (n / 16
// times cg of them) in two rounds, but no fewer than 8 warps, so that a row's
// long lists, cut in segments, have warps to run on; narrow groups take 4, as
// each of their many lane groups stages its own entries.
inline int rows_threads_for(int grid_cols, int lanes, int cg) {
  if (lanes < 4) return 128;
  return grid_cols / 16 * cg > 512 ? kRowsThreads : 256;
}

constexpr uint32_t kWaitLimit = 1u << 22;  // polls before a bounded wait gives up

// Binning in sample order (k_prepare, k_place): a block takes bin_span
// consecutive samples, kBinThreads at a time, with a word or two of shared
// memory per binning list of the frame.
constexpr int kBinThreads = 512;
constexpr int kBinWarps = kBinThreads / 32;
constexpr size_t kPlaceListBytes = 4;  // of k_place: the list's running position
constexpr size_t kListSmem = kMaxGrid * (kMaxGrid / kChunk) * 4;  // a word of every list of the largest grid
constexpr size_t kRowsSmem = 200 * 1024;                          // of a k_rows block, at most
// A call keeps one count per list for each of its blocks: at most this many (64 MB), or one
// block a frame where that is more.
constexpr size_t kBinCounts = size_t{1} << 24;
// 3-D: most blocks of the plane stage of the binning (four per SM)
constexpr int kPlaneStageBlocks = 4 * kSms;

struct Shape {
  int frames, channels, samples;
  int rows, cols;          // image
  int grid_rows, grid_cols;
  int width;
  int nchunks;             // ceil(grid_cols / kChunk)
  int lists_per_frame;     // grid_rows * nchunks
  int lists_per_row;       // most chunks a stencil's columns fall into: 2, or 3 (see list_chunks)
  int first_of_two;        // 1: two chunks, and the first may see both ends of a stencil that wraps
  size_t entries_per_frame;
  int out_rows, out_cols;  // kept image region
  int col_group;           // coils per column-pass tile: a power of two >= 2, <= 32
  // channel pitch of the row-transformed grid: channels rounded up to a 16-byte stride (a
  // column tile's coils past it are zeros that TMA fills in; rounded up to
  // col_group, 20 coils took 1.6 times the memory, and a 300 grid of 11 coils x 7 frames 240 us a
  // call instead of 236)
  int cpitch;
  bool kb;
  float beta, inv_i0_beta;
  float row_origin, col_origin;
  float phase_row, phase_col, phase_sign;  // origin-phase coefficients
  int bin_blocks, bin_span;  // 2-D binning: blocks per frame and samples per block
  // blocks of all frames that the counts have room for: never fewer for more samples or
  // frames, where bin_blocks rises and falls, so that a workspace serves every smaller call
  size_t bin_capacity;
  int coil_group, column_block, frames_per_pass, coil_parts;
  uint32_t wait_fault;  // tests only: segment waits that cannot succeed, given up after this many polls
  int column_pass;      // 1 one CTA per tile (k_cols), 2 persistent ring (k_cols_ring)
  DifPlan plan_rows, plan_cols;
  // ragged batches (device arrays, null otherwise): valid coils and samples
  // of each frame, and the addresses of its samples [C_f][M_f] and of its
  // trajectory [M_f][2] (device memory or host memory the device reads)
  const uint32_t* frame_channels = nullptr;
  const uint32_t* frame_samples = nullptr;
  const uint64_t* frame_kspace = nullptr;
  const uint64_t* frame_traj = nullptr;
};

// Column tiles that take all the coils of a column.
inline int column_groups(const Shape& s) { return (s.cpitch + s.col_group - 1) / s.col_group; }

// TMA boxes of equal rows, at most 256 each, that take a tile of `rows` rows.
inline int tile_boxes(int rows) {
  int boxes = 1;
  while (rows / boxes > 256 || rows % boxes != 0) ++boxes;
  return boxes;
}

// Columns of a column tile, `cb` or more: each of a tile's boxes has to start on 128 bytes of
// shared memory (a TMA copy to any other address faults).  Where there are several boxes and a
// row is fewer than 16 lines (128 bytes), their size may not be a multiple of that (315 rows x 8
// lines: three of 6720 bytes); the tile then takes more columns, of which those past
// the image are filled with zeros and not written.
inline int aligned_column_block(int rows, int col_group, int cb) {
  const int boxes = tile_boxes(rows);
  if (boxes > 1)
    while (static_cast<size_t>(rows / boxes) * cb * col_group * sizeof(float2) % 128 != 0) cb <<= 1;
  return cb;
}

struct Layout {
  size_t flags, frame_flags, cleared, records, counts, totals, offsets, expanded, samples_t, inter,
      coil_last, tables, total;
};

size_t record_bytes(int width) {
  switch (width) {
    case 2: return sizeof(SampleRecord<2>);
    case 4: return sizeof(SampleRecord<4>);
    case 6: return sizeof(SampleRecord<6>);
    default: return sizeof(SampleRecord<8>);
  }
}

bool is_fft_size(uint32_t n) {
  DifPlan p;
  return n >= 2 && n <= kMaxGrid && make_dif_plan(static_cast<int>(n), &p);
}

ksj_gpu_status make_shape(const ksj_gpu_gridding_desc* d, const ksj_gpu_gridding_tuning* t, Shape* s) {
  if (d == nullptr || d->struct_size < sizeof(ksj_gpu_gridding_desc)) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (d->channels == 0 || d->samples == 0 || d->frames == 0 || d->image_rows < 2 || d->image_cols < 2)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (d->dcf_mode > KSJ_GPU_DCF_EXTERNAL || d->output > KSJ_GPU_OUTPUT_COIL_MAJOR ||
      d->sample_format > KSJ_GPU_SAMPLES_BF16)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (!std::isfinite(d->row_origin) || !std::isfinite(d->col_origin)) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (d->samples > (1u << 26) || d->channels > 4096 || d->frames > 65535) return KSJ_GPU_ERROR_UNSUPPORTED;
  s->kb = d->kernel == KSJ_GPU_KERNEL_KAISER_BESSEL;
  if (d->kernel == KSJ_GPU_KERNEL_LINEAR) {
    if (d->kernel_width != 2 || d->grid_rows != d->image_rows || d->grid_cols != d->image_cols)
      return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  } else if (s->kb) {
    if (d->kernel_width < 2 || d->kernel_width > kMaxWidth || (d->kernel_width & 1u) != 0)
      return KSJ_GPU_ERROR_INVALID_ARGUMENT;
    if (d->grid_rows < d->image_rows || d->grid_cols < d->image_cols || d->grid_rows < d->kernel_width ||
        d->grid_cols < d->kernel_width)
      return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  } else {
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  }
  if (!is_fft_size(d->grid_rows) || !is_fft_size(d->grid_cols)) return KSJ_GPU_ERROR_UNSUPPORTED;
  s->frames = static_cast<int>(d->frames);
  s->channels = static_cast<int>(d->channels);
  s->samples = static_cast<int>(d->samples);
  s->rows = static_cast<int>(d->image_rows);
  s->cols = static_cast<int>(d->image_cols);
  s->grid_rows = static_cast<int>(d->grid_rows);
  s->grid_cols = static_cast<int>(d->grid_cols);
  s->width = static_cast<int>(d->kernel_width);
  s->nchunks = (s->grid_cols + kChunk - 1) / kChunk;
  s->lists_per_frame = s->grid_rows * s->nchunks;
  {
    const int tail = s->grid_cols % kChunk;  // columns of a narrower last chunk
    const bool over = s->nchunks > 1 && tail != 0 && tail < s->width - 1;
    s->lists_per_row = over ? 3 : 2;
    s->first_of_two = over && s->nchunks == 2 ? 1 : 0;
  }
  s->entries_per_frame = static_cast<size_t>(s->samples) * s->width * s->lists_per_row;
  {
    // Samples per block of the binning, in turns of kBinThreads: the time is about
    // the turns an SM gets, with the loading of the list positions (one turn per
    // 4608 lists) for each block and half as much again where it has one block
    // alone; so the blocks of all frames should fill whole rounds of SMs (96 frames x
    // 26 turns: 3, 4, 6 blocks a frame take 108, 161, 132 us of k_place).
    const int turns = (s->samples + kBinThreads - 1) / kBinThreads;
    const double load = s->lists_per_frame / 4608.0;
    const size_t most = std::max<size_t>(s->frames, kBinCounts / s->lists_per_frame);
    double best = HUGE_VAL;
    s->bin_span = turns * kBinThreads;
    s->bin_blocks = 1;
    for (int t = 1; t <= turns; t += 1 + t / 16) {
      const int blocks = (turns + t - 1) / t;
      if (static_cast<size_t>(blocks) * s->frames > most) continue;
      const double rounds = std::ceil(static_cast<double>(blocks) * s->frames / kSms);
      const double cost = (t + load) * std::max(rounds, 1.5);
      if (cost <= best) {
        best = cost;
        s->bin_span = t * kBinThreads;
        s->bin_blocks = blocks;
      }
    }
    s->bin_capacity = std::min(static_cast<size_t>(s->frames) * turns, most);
  }
  s->out_rows = s->rows;
  s->out_cols = s->cols;
  s->col_group = 2;
  while (s->col_group < s->channels && s->col_group < 32) s->col_group <<= 1;
  s->cpitch = (s->channels + 1) / 2 * 2;
  s->row_origin = static_cast<float>(d->row_origin);
  s->col_origin = static_cast<float>(d->col_origin);
  if (s->kb) {
    const double sigma = static_cast<double>(d->grid_rows) / static_cast<double>(d->image_rows);
    double beta = d->kb_beta;
    if (!(beta > 0.0)) {
      const double a = (static_cast<double>(d->kernel_width) / sigma) * (sigma - 0.5);
      const double arg = a * a - 0.8;
      if (arg <= 0.0) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
      beta = 3.14159265358979323846 * std::sqrt(arg);
    }
    s->beta = static_cast<float>(beta);
    s->inv_i0_beta = static_cast<float>(1.0 / std::cyl_bessel_i(0.0, beta));
    // exp(i k (q + delta)), delta = n/2 - origin: the image is centred on
    // offsets q = p - n/2 so the deapodisation sees |q| <= n/2.
    s->phase_row = static_cast<float>(static_cast<double>(s->rows / 2) - d->row_origin);
    s->phase_col = static_cast<float>(static_cast<double>(s->cols / 2) - d->col_origin);
    s->phase_sign = 1.0f;
    if (static_cast<double>(s->phase_row) != static_cast<double>(s->rows / 2) - d->row_origin ||
        static_cast<double>(s->phase_col) != static_cast<double>(s->cols / 2) - d->col_origin)
      return KSJ_GPU_ERROR_UNSUPPORTED;
  } else {
    s->beta = 0.0f;
    s->inv_i0_beta = 0.0f;
    // exp(-i (k_r r0 + k_c c0)) (eigen_radial_gridding.cpp:330-334)
    s->phase_row = s->row_origin;
    s->phase_col = s->col_origin;
    s->phase_sign = -1.0f;
    if (static_cast<double>(s->row_origin) != d->row_origin || static_cast<double>(s->col_origin) != d->col_origin)
      return KSJ_GPU_ERROR_UNSUPPORTED;  // origins must be exact floats (the reference casts them, :320-321)
  }
  make_dif_plan(s->grid_rows, &s->plan_rows);
  make_dif_plan(s->grid_cols, &s->plan_cols);

  // tuning
  int cg = t && t->coil_group ? static_cast<int>(t->coil_group) : 0;
  int cb = t && t->column_block ? static_cast<int>(t->column_block) : 0;
  int cap = t && t->list_capacity ? static_cast<int>(t->list_capacity) : 0;
  if (cap == 0) cap = 512;
  if (cap < 64 || cap > 2048 || (cap & (cap - 1)) != 0) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const size_t smem_limit = kRowsSmem;
  const int parts = t && t->struct_size >= offsetof(ksj_gpu_gridding_tuning, coil_parts) + 4 && t->coil_parts
                        ? static_cast<int>(t->coil_parts)
                        : 1;
  if (parts != 1 && parts != 2) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  auto rows_smem = [&](int g) {
    const int lanes = std::max(1, g / parts);
    return rows_smem_for(s->grid_cols, g, lanes, rows_threads_for(s->grid_cols, lanes, g));
  };
  if (cg == 0) {
    int want = 1;
    while (want < s->channels && want < 32) want <<= 1;
    cg = want;
    // two row blocks per SM at least ((228 KiB - 2 x 1 KiB reserved) / 2), so
    // that one block's transform overlaps another's gridding; the whole coil
    // array where it fits (32 coils on a 384 grid, 96 frames: groups of 32, 16, 8
    // coils take 2488, 2640, 3621 us)
    while (cg > 1 && rows_smem(cg) > 115712 - 1024) cg >>= 1;
  }
  if (cg < 1 || cg > 32 || (cg & (cg - 1)) != 0 || rows_smem(cg) > smem_limit) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  // column pass: cb columns x col_group coils per tile (a power of two
  // number of lines, at most the block's threads), double-buffered when the
  // channels take more than one tile
  const int cgroups = column_groups(*s);
  auto cols_tile = [&](int b) {
    return static_cast<size_t>(s->grid_rows) * b * s->col_group * sizeof(float2) * (cgroups > 1 ? 2 : 1);
  };
  if (cb == 0) {
    cb = std::max(1, 32 / s->col_group);
    while (cb > 1 && (cols_tile(cb) > 110 * 1024 || cb > s->out_cols)) cb >>= 1;
  }
  if (cb < 1 || cb > 32 || (cb & (cb - 1)) != 0 || cb > s->out_cols || cb * s->col_group > kColsThreads ||
      cols_tile(cb) > smem_limit)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  s->coil_group = cg;
  s->column_block = aligned_column_block(s->grid_rows, s->col_group, cb);
  // frames per k_rows/k_cols pass: keep one pass's row-transformed grid
  // (channels x grid_rows x out_cols complex) within ~64 MB of L2
  // fields appended to the tuning struct are read only when the caller's
  // struct_size covers them
  auto has = [&](size_t field_end) { return t != nullptr && t->struct_size >= field_end; };
  int fpp = has(offsetof(ksj_gpu_gridding_tuning, frames_per_pass) + 4) ? static_cast<int>(t->frames_per_pass) : 0;
  // default: two passes (on two streams, so one pass's last partial wave
  // overlaps the other) once there are enough frames to split
  if (fpp <= 0) fpp = s->frames >= 4 ? (s->frames + 1) / 2 : s->frames;
  s->frames_per_pass = std::min(fpp, s->frames);
  int rb = has(offsetof(ksj_gpu_gridding_tuning, rows_blocks_per_sm) + 4) ? static_cast<int>(t->rows_blocks_per_sm) : 0;
  if (rb < 0 || rb > 2) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (parts > cg) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  s->coil_parts = parts;
  s->wait_fault = has(offsetof(ksj_gpu_gridding_tuning, wait_fault_polls) + 4) ? t->wait_fault_polls : 0u;
  int cp = has(offsetof(ksj_gpu_gridding_tuning, column_pass) + 4) ? static_cast<int>(t->column_pass) : 0;
  if (cp < 0 || cp > 2) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  s->column_pass = cp == 0 ? 1 : cp;  // one CTA per tile unless asked (measured faster on the 384 grid)
  return KSJ_GPU_OK;
}

size_t sample_bytes(uint32_t format) { return format == KSJ_GPU_SAMPLES_BF16 ? 4 : 8; }

Layout make_layout(const Shape& s, const ksj_gpu_gridding_desc* d) {
  Layout l{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t fm = static_cast<size_t>(s.frames) * s.samples;
  const size_t nl = static_cast<size_t>(s.frames) * s.lists_per_frame;
  l.flags = take(kFlagBytes);  // flags and frame flags are cleared together
  l.frame_flags = take(static_cast<size_t>(s.frames) * 4);
  l.cleared = off;
  l.records = take(fm * record_bytes(s.width));
  l.totals = take(nl * 4);
  l.offsets = take((nl + s.frames) * 4);
  l.expanded = take(static_cast<size_t>(s.frames) * s.entries_per_frame * entry_bytes(s.width));
  l.samples_t = take(fm * s.channels * sizeof(float2));
  l.inter = take(static_cast<size_t>(s.frames) * s.grid_rows * s.out_cols * s.cpitch * sizeof(float2));
  l.coil_last = d->output == KSJ_GPU_OUTPUT_COIL_MAJOR
                    ? take(static_cast<size_t>(s.frames) * s.channels * s.out_rows * s.out_cols * sizeof(float2))
                    : off;
  // tables: twiddles for rows and cols, inverse deapodisation for rows and
  // cols, and the FFT output position of every kept row and column
  l.tables = take((static_cast<size_t>(s.grid_rows) + s.grid_cols) * sizeof(float2) +
                  (static_cast<size_t>(s.out_rows) + s.out_cols) * (sizeof(float) + sizeof(int)));
  // last, as most of it may be room that this call's blocks leave empty (between the records and
  // the lists it cost a 512 grid 0.5 % of the call)
  l.counts = take(s.bin_capacity * s.lists_per_frame * 4);
  l.total = off;
  return l;
}

// ------------------------------------------------------------------ kernels

// Twiddles exp(2 pi i t / n) for both axes and the inverse deapodisation
// factors 1 / psi(q), q = p - n/2, psi the continuous Fourier transform of the
// normalised Kaiser-Bessel kernel: W sinh(z)/z / I0(beta),
// z = sqrt(beta^2 - (pi W q / g)^2) (Jackson et al. 1991).  FP64 here only.
//
// pos_rows[p] / pos_cols[p]: where the in-place DIF leaves the frequency
// index that kept image row / column p takes: p itself for the linear
// operator (no oversampling), (p - n/2) mod g for Kaiser-Bessel (the image is
// centred on q = p - n/2).
struct TablesArgs {
  float2* tw_rows;
  float2* tw_cols;
  float* inv_dr;
  float* inv_dc;
  int* pos_rows;
  int* pos_cols;
  int grid_rows, grid_cols, out_rows, out_cols;
  DifPlan plan_rows, plan_cols;
  int kb, width;
  double beta, i0_beta;
};

// Entries of all tables; one thread each, see table_entry.
__host__ __device__ inline int table_entries(const TablesArgs& t) {
  return t.out_rows + t.out_cols + t.grid_rows + t.grid_cols;
}

__device__ __forceinline__ void table_entry(const TablesArgs& t, int i) {
  auto source = [&](int p, int n, int g) { return t.kb ? (p - n / 2 + g) % g : p; };
  if (i < t.out_rows) {
    const int k = source(i, t.out_rows, t.grid_rows);
    t.pos_rows[i] = has_two_step_rows(t.grid_rows) ? two_step_slot(k, t.grid_rows) : dif_position(t.plan_rows, k);
    t.inv_dr[i] = t.kb ? kb_inv_deapod(i, t.out_rows, t.grid_rows, t.width, t.beta, t.i0_beta) : 1.0f;
    return;
  }
  i -= t.out_rows;
  if (i < t.out_cols) {
    t.pos_cols[i] = dif_position(t.plan_cols, source(i, t.out_cols, t.grid_cols));
    t.inv_dc[i] = t.kb ? kb_inv_deapod(i, t.out_cols, t.grid_cols, t.width, t.beta, t.i0_beta) : 1.0f;
    return;
  }
  i -= t.out_cols;
  if (i < t.grid_rows)
    t.tw_rows[i] = twiddle(i, t.grid_rows);
  else if (i - t.grid_rows < t.grid_cols)
    t.tw_cols[i - t.grid_rows] = twiddle(i - t.grid_rows, t.grid_cols);
}

__global__ void __launch_bounds__(256) k_fill(float* p, int n, float v) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) p[i] = v;
}

struct PrepareArgs {
  const float* traj;
  const float* dcf;
  const uint32_t* frame_samples;  // ragged batches: valid samples of each frame (null: all)
  const uint64_t* frame_traj;     // ragged batches: address of each frame's trajectory [M_f][2]
  uint32_t* frame_flags;          // per-frame copy of the check flags (null: none)
  uint32_t dcf_mode;
  uint32_t require_nyquist;
  unsigned char* records;
  uint32_t* counts;               // [frame][block][list]: entries of the block's samples in the list
  uint32_t* flags;
  int frames, samples, grid_rows, grid_cols, nchunks, lists_per_frame;
  int bin_span;                   // samples per block
  int kb;
  float beta, two_over_w, inv_i0_beta;
  float phase_row, phase_col, phase_sign;
};

// The chunks that the columns c0 .. c0 + W - 1 (wrapped) fall into: those of the first and the
// last (k[1] = k[0] where it is the same) and, for kLists 3, the row's last chunk where the columns
// begin before it, cover it and go on at column 0 (else k[2] = -1).
template <int W, int kLists>
__device__ __forceinline__ void list_chunks(int c0, int grid_cols, int (&k)[kLists]) {
  const bool wraps = c0 + W - 1 >= grid_cols;
  const int last = wraps ? c0 + W - 1 - grid_cols : c0 + W - 1;
  k[0] = c0 / kChunk;
  k[1] = last / kChunk;
  if constexpr (kLists == 3) {
    const int tail = (grid_cols - 1) / kChunk;
    k[2] = wraps && k[0] != tail ? tail : -1;
  }
}

// Whether k[h] names a list that no earlier one of k does.
template <int kLists>
__device__ __forceinline__ bool own_list(const int (&k)[kLists], int h) {
  return h == 0 || (h == 1 ? k[1] != k[0] : k[h] >= 0);
}

// A warp's samples, one per lane: how many lanes below this one join each of this
// lane's lists (rows r0 + j wrapped, chunks k), and whether one above does.
// Byte j of below[h] is the count for (row r0 + j, chunk k[h]); bit j of
// above[h].  r0 < 0: no sample.  Every lane's rows and chunks go round the warp once.
template <int W, int kLists>
struct WarpRanks {
  static constexpr int kWords = (W + 3) / 4;
  uint32_t below[kLists][kWords], above[kLists];
};

template <int W, int kLists>
__device__ __forceinline__ WarpRanks<W, kLists> warp_ranks(int r0, const int (&k)[kLists], int grid_rows) {
  constexpr uint32_t kRows = (1u << W) - 1u;
  constexpr int kWords = WarpRanks<W, kLists>::kWords;
  WarpRanks<W, kLists> out;
#pragma unroll
  for (int h = 0; h < kLists; ++h) {
    out.above[h] = 0;
#pragma unroll
    for (int q = 0; q < kWords; ++q) out.below[h][q] = 0;
  }
  const int lane = threadIdx.x & 31;
  // row, then the chunks (63: none)
  uint32_t mine = r0 < 0 ? 0u : static_cast<uint32_t>(r0);
#pragma unroll
  for (int h = 0; h < kLists; ++h) mine = mine << 6 | (r0 < 0 ? 63u : static_cast<uint32_t>(k[h]) & 63u);
#pragma unroll 4
  for (int i = 0; i < 32; ++i) {
    const uint32_t other = __shfl_sync(0xffffffffu, mine, i);
    // this lane's rows that the other sample's stencil covers: its rows start
    // d before ours, or (across the wrap) grid_rows - d after
    int d = r0 - static_cast<int>(other >> (6 * kLists));
    if (d < 0) d += grid_rows;
    const uint32_t rows = (kRows >> min(d, 31)) | ((kRows << min(grid_rows - d, 31)) & kRows);
#pragma unroll
    for (int h = 0; h < kLists; ++h) {
      const uint32_t own = static_cast<uint32_t>(k[h]);
      bool same = false;
#pragma unroll
      for (int o = 0; o < kLists; ++o) same = same || own == ((other >> (6 * o)) & 63u);
      const uint32_t m = same ? rows : 0u;
      if (i < lane) {
#pragma unroll
        for (int q = 0; q < kWords; ++q)  // bit j of a nibble to byte j
          out.below[h][q] += (((m >> (4 * q)) & 15u) * 0x00204081u) & 0x01010101u;
      } else if (i > lane) {
        out.above[h] |= m;
      }
    }
  }
  return out;
}

// Places of one sample per thread in the lists of rows r0 .. r0 + W - 1
// (wrapped) and chunks k (r0 < 0: no sample), in thread order: a list's
// entries have to stand in sample order.  at: running position of each list.  The
// ranks within the warps are found first, by all warps at once; then the warps take
// turns, passed on by named barriers: each reads its lists' positions, adds the ranks,
// and the last lane of a list moves its position on.  Called by the whole block;
// synchronises it first.
template <int W, int kLists>
__device__ __forceinline__ void place_turn(uint32_t* at, int r0, const int (&k)[kLists], int nchunks, int grid_rows,
                                           uint32_t (&pos)[W][kLists]) {
  const int warp = threadIdx.x >> 5;
  const WarpRanks<W, kLists> ranks = warp_ranks<W>(r0, k, grid_rows);
  int first[kLists];  // list of row r0 and each chunk, -1: none
#pragma unroll
  for (int h = 0; h < kLists; ++h) first[h] = r0 >= 0 && own_list(k, h) ? r0 * nchunks + k[h] : -1;
  const int wrap = grid_rows - r0;  // rows from here on wrap
  auto list_of = [&](int j, int h) { return first[h] + (j >= wrap ? j - grid_rows : j) * nchunks; };
  __syncthreads();  // the positions are loaded, and every warp's last turn is over
  if (warp > 0) asm volatile("bar.sync %0, 64;" ::"r"(warp) : "memory");
#pragma unroll
  for (int j = 0; j < W; ++j)
#pragma unroll
    for (int h = 0; h < kLists; ++h)
      if (first[h] >= 0) pos[j][h] = at[list_of(j, h)];
  __syncwarp();
#pragma unroll
  for (int j = 0; j < W; ++j) {
#pragma unroll
    for (int h = 0; h < kLists; ++h) {
      if (first[h] >= 0) {
        pos[j][h] += (ranks.below[h][j / 4] >> (8 * (j & 3))) & 255u;
        if (!((ranks.above[h] >> j) & 1u)) at[list_of(j, h)] = pos[j][h] + 1;
      }
    }
  }
  __syncwarp();
  if (warp + 1 < kBinWarps) asm volatile("bar.arrive %0, 64;" ::"r"(warp + 1) : "memory");
}

// One sample counted in its lists (shared memory).
template <int W, int kLists>
__device__ __forceinline__ void count_lists(uint32_t* counts, int r0, const int (&k)[kLists], int nchunks,
                                            int grid_rows) {
#pragma unroll
  for (int j = 0; j < W; ++j) {
    int row = r0 + j;
    if (row >= grid_rows) row -= grid_rows;
#pragma unroll
    for (int h = 0; h < kLists; ++h)
      if (own_list(k, h)) atomicAdd(counts + row * nchunks + k[h], 1u);
  }
}

// One sample's record, and its entries counted in `counts` (shared memory, per list).
template <int W, int kLists>
__device__ __forceinline__ void prepare_sample(const PrepareArgs& a, int f, int sample, uint32_t* counts) {
  const size_t idx = static_cast<size_t>(f) * a.samples + sample;
  if (a.frame_samples != nullptr && static_cast<uint32_t>(sample) >= __ldg(a.frame_samples + f)) {
    // a padding sample of a ragged batch: in no list (its trajectory is not read)
    reinterpret_cast<SampleRecord<W>*>(a.records)[idx].r0 = -1;
    return;
  }
  const float2 k =
      a.frame_traj != nullptr
          ? reinterpret_cast<const float2*>(__ldg(a.frame_traj + f))[sample]
          : __ldg(reinterpret_cast<const float2*>(a.traj) + idx);
  bool ok = isfinite(k.x) && isfinite(k.y);
  if (ok && a.require_nyquist) ok = k.x >= -kPiF && k.x <= kPiF && k.y >= -kPiF && k.y <= kPiF;
  // a coordinate far outside the grid would overflow the int tap arithmetic
  if (ok && !a.require_nyquist) ok = fabsf(k.x) < 1.0e4f && fabsf(k.y) < 1.0e4f;
  float w = 1.0f;
  if (a.dcf_mode == KSJ_GPU_DCF_ANALYTIC_RAMP) {
    w = hypotf(k.x, k.y);
  } else if (a.dcf_mode == KSJ_GPU_DCF_EXTERNAL) {
    w = __ldg(a.dcf + idx);
    if (!(isfinite(w) && w >= 0.0f)) {
      atomicOr(a.flags, KSJ_GPU_FLAG_BAD_DCF);
      if (a.frame_flags) atomicOr(a.frame_flags + f, KSJ_GPU_FLAG_BAD_DCF);
      w = 0.0f;
    }
  }
  SampleRecord<W> rec;
  if (!ok) {
    atomicOr(a.flags, KSJ_GPU_FLAG_BAD_TRAJECTORY);
    if (a.frame_flags) atomicOr(a.frame_flags + f, KSJ_GPU_FLAG_BAD_TRAJECTORY);
    rec.r0 = 0;
    rec.c0 = 0;
    rec.scale = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      rec.wr[j] = 0.0f;
      rec.wc[j] = 0.0f;
    }
  } else {
    const dfloat ur = grid_coordinate(k.x, static_cast<float>(a.grid_rows));
    const dfloat uc = grid_coordinate(k.y, static_cast<float>(a.grid_cols));
    float fr, fc;
    const int lr = dfloor(ur, &fr);
    const int lc = dfloor(uc, &fc);
    if (!a.kb) {
      // periodic 2x2 linear stencil (eigen_radial_gridding.cpp:325-342)
      rec.r0 = wrap_index(lr, a.grid_rows);
      rec.c0 = wrap_index(lc, a.grid_cols);
      rec.wr[0] = 1.0f - fr;
      rec.wr[1] = fr;
      rec.wc[0] = 1.0f - fc;
      rec.wc[1] = fc;
#pragma unroll
      for (int j = 2; j < W; ++j) {
        rec.wr[j] = 0.0f;
        rec.wc[j] = 0.0f;
      }
    } else {
      const int sr = lr - W / 2 + 1;
      const int sc = lc - W / 2 + 1;
      rec.r0 = wrap_index(sr, a.grid_rows);
      rec.c0 = wrap_index(sc, a.grid_cols);
#pragma unroll
      for (int j = 0; j < W; ++j) {
        // offset (tap - u), exact in its high part
        const float dr = __fsub_rn(__fsub_rn(static_cast<float>(sr + j), ur.hi), ur.lo);
        const float dc = __fsub_rn(__fsub_rn(static_cast<float>(sc + j), uc.hi), uc.lo);
        rec.wr[j] = kb_weight(dr, a.two_over_w, a.beta, a.inv_i0_beta);
        rec.wc[j] = kb_weight(dc, a.two_over_w, a.beta, a.inv_i0_beta);
      }
    }
    const float2 e = exp_i_dot(k.x, a.phase_row, k.y, a.phase_col, a.phase_sign);
    rec.scale = cscale(e, w);
  }
  reinterpret_cast<SampleRecord<W>*>(a.records)[idx] = rec;
  int chunks[kLists];
  list_chunks<W>(rec.c0, a.grid_cols, chunks);
  count_lists<W>(counts, rec.r0, chunks, a.nchunks, a.grid_rows);
}

// One block per (block of samples, frame).  The counts go to shared memory: as atomics on
// global memory the samples of a radial scan's centre, all in the same few
// lists, were serialised (25 us for 205824 samples on a 512 grid, this 17).
template <int W, int kLists>
__global__ void __launch_bounds__(kBinThreads) k_prepare(PrepareArgs a) {
  extern __shared__ uint32_t prepare_counts[];
  chain_begin();
  const int f = blockIdx.y;
  for (int l = threadIdx.x; l < a.lists_per_frame; l += kBinThreads) prepare_counts[l] = 0;
  __syncthreads();
  const int s0 = blockIdx.x * a.bin_span, s1 = min(s0 + a.bin_span, a.samples);
  for (int sample = s0 + threadIdx.x; sample < s1; sample += kBinThreads)
    prepare_sample<W, kLists>(a, f, sample, prepare_counts);
  __syncthreads();
  uint32_t* out = a.counts + (static_cast<size_t>(f) * gridDim.x + blockIdx.x) * a.lists_per_frame;
  for (int l = threadIdx.x; l < a.lists_per_frame; l += kBinThreads) out[l] = prepare_counts[l];
}

// Thread per list: the blocks' counts of the list become each block's start
// among the list's entries; their sum is the list's length.  Bound by
// latency: kPrefixAhead blocks' counts are in flight at once (8: 12.4 us on a 512 grid
// with 134 blocks, 16: 10.3; 32 take so many registers that the scan cannot start beside them).
constexpr int kPrefixAhead = 16;

__global__ void __launch_bounds__(128) k_bin_prefix(uint32_t* counts, uint32_t* totals, int blocks, int lists) {
  chain_begin();
  const int l = blockIdx.x * blockDim.x + threadIdx.x;
  if (l >= lists) return;
  uint32_t* c = counts + static_cast<size_t>(blockIdx.y) * blocks * lists + l;
  uint32_t run = 0;
  for (int b0 = 0; b0 < blocks; b0 += kPrefixAhead) {
    uint32_t v[kPrefixAhead];
#pragma unroll
    for (int k = 0; k < kPrefixAhead; ++k) v[k] = b0 + k < blocks ? c[static_cast<size_t>(b0 + k) * lists] : 0u;
#pragma unroll
    for (int k = 0; k < kPrefixAhead; ++k) {
      if (b0 + k < blocks) c[static_cast<size_t>(b0 + k) * lists] = run;
      run += v[k];
    }
  }
  totals[static_cast<size_t>(blockIdx.y) * lists + l] = run;
}

// [frame][channel][sample] -> [frame][sample][channel] complex64, each sample
// times its weight and phase (dcf * exp(i * origin phase), in its record), in tiles of 32 samples x 32
// channels, checking every sample on the way: a
// non-finite value (either component; bf16 exponent all ones) raises
// KSJ_GPU_FLAG_NONFINITE_SAMPLE.  The product is formed here, once, and not by
// each of the W rows (W^2 in 3-D) that read the sample.
//
// Ragged batches (frame_channels / frame_samples / frame_src non-null):
// frame f holds frame_channels[f] coils of frame_samples[f] samples, packed
// [channel][sample] at address frame_src[f] (device memory, or host memory
// the device reads in place); the padding up to the call's channels and
// samples is written as zeros.
struct CoilLastArgs {
  const void* in;
  float2* out;
  const unsigned char* scales;  // the records' scale fields, `scale_stride` bytes apart
  int scale_stride;
  int channels, samples;
  uint32_t* flags;
  const uint32_t* frame_channels;
  const uint32_t* frame_samples;
  const uint64_t* frame_src;
  int frame0;
  uint32_t* frame_flags;
};
using CoilLastTile = float2[32][33];

// One tile by 256 consecutive threads (tx, ty) of a block, (tx, 0 .. 7); every thread
// of the block takes part, with tiles of the same frame.
template <uint32_t kFormat>
__device__ __forceinline__ void coil_last_tile(const CoilLastArgs& a, int f, int s0, int c0, CoilLastTile& t, int tx,
                                               int ty) {
  using T = typename std::conditional<kFormat == KSJ_GPU_SAMPLES_BF16, uint32_t, unsigned long long>::type;
  const int channels = a.channels, samples = a.samples;
  float2* dst = a.out + static_cast<size_t>(f) * channels * samples;
  const int live_c = a.frame_channels ? min(channels, static_cast<int>(__ldg(a.frame_channels + f))) : channels;
  const int live_s = a.frame_samples ? min(samples, static_cast<int>(__ldg(a.frame_samples + f))) : samples;
  // ragged frames are packed at their own sample count
  const T* src = a.frame_src ? reinterpret_cast<const T*>(__ldg(a.frame_src + f))
                             : static_cast<const T*>(a.in) + static_cast<size_t>(f) * channels * samples;
  const int pitch = a.frame_src ? live_s : samples;
  const int sm = s0 + tx;
  float2 scale = make_float2(0.0f, 0.0f);
  if (sm < live_s)
    scale = __ldg(reinterpret_cast<const float2*>(
        a.scales + (static_cast<size_t>(f) * samples + sm) * static_cast<size_t>(a.scale_stride)));
  bool bad = false;
#pragma unroll
  for (int y = ty; y < 32; y += 8) {
    const int c = c0 + y;
    if (c < channels && sm < samples) {
      if (c >= live_c || sm >= live_s) {
        t[y][tx] = make_float2(0.0f, 0.0f);
        continue;
      }
      const T v = __ldg(src + static_cast<size_t>(c) * pitch + sm);
      float2 x;
      if constexpr (kFormat == KSJ_GPU_SAMPLES_BF16) {
        bad |= (v & 0x7f80u) == 0x7f80u || (v & 0x7f800000u) == 0x7f800000u;
        x = make_float2(bf16_to_float(static_cast<uint16_t>(v & 0xffffu)), bf16_to_float(static_cast<uint16_t>(v >> 16)));
      } else {
        bad |= (v & 0x7f800000ull) == 0x7f800000ull || (v & 0x7f80000000000000ull) == 0x7f80000000000000ull;
        x = make_float2(__uint_as_float(static_cast<uint32_t>(v)), __uint_as_float(static_cast<uint32_t>(v >> 32)));
      }
      t[y][tx] = cmul(x, scale);
    }
  }
  if (__syncthreads_or(bad) && threadIdx.x == 0 && threadIdx.y == 0) {
    atomicOr(a.flags, KSJ_GPU_FLAG_NONFINITE_SAMPLE);
    if (a.frame_flags) atomicOr(a.frame_flags + f, KSJ_GPU_FLAG_NONFINITE_SAMPLE);
  }
#pragma unroll
  for (int y = ty; y < 32; y += 8) {
    const int so = s0 + y, c = c0 + tx;
    if (c < channels && so < samples) dst[static_cast<size_t>(so) * channels + c] = t[tx][y];
  }
}

// The tiles as a launch of their own ((32, 8) threads, grid (ceil(samples/32),
// ceil(channels/32), frames)): calls of more samples than the scan's launch takes, 3-D, and
// passes whose samples arrive one by one.
template <uint32_t kFormat>
__global__ void __launch_bounds__(256) k_samples_coil_last(CoilLastArgs a) {
  __shared__ CoilLastTile t;
  chain_wait();  // (row-pass blocks waiting beside these would hold shared memory their cache uses)
  coil_last_tile<kFormat>(a, a.frame0 + blockIdx.z, blockIdx.x * 32, blockIdx.y * 32, t, threadIdx.x, threadIdx.y);
}

// Exclusive scan of one frame's list lengths, one block per frame.  Bound by latency (one block
// for a single frame), so a warp holds its whole stretch of counts in registers,
// 32 consecutive ones per load, all loads in flight at once (per-thread
// stretches, read twice one count after another, took 24 us for 16384 lists, this
// and the tables 10).
// Blocks from `frames` on fill the call's tables meanwhile, 64 entries each: their FP64
// functions run at a few lanes per clock and SM, so they are spread over many
// (a kernel of their own on one or two SMs took 7 to 20 us).
// The blocks after those bring the samples themselves into the row pass's order
// (coil_last_tile), which needs the records alone, where the launch fits the SMs in
// one round (kScanSampleBlocks): a frame's scan leaves the others idle.  One frame of 13056
// samples x 32 coils 64.1 -> 60.1 us a call.  Beyond that they are a launch of their
// own with small blocks (512 blocks here: 30 us against 9 + 16; 96 frames 317 against 10 + 153).
constexpr int kScanPer = kMaxGrid * (kMaxGrid / kChunk) / 1024;  // counts per thread, at most
constexpr int kTablesPerBlock = 64;
constexpr int kCoilLastTiles = 1024 / 256;  // tiles of a block, of consecutive samples
constexpr int kScanSampleBlocks = kSms - 8;  // with a few for the tables, one round of the SMs
struct ScanSamples {
  CoilLastArgs a;
  int first_block;  // of the launch
  int bf16, none;
};

__global__ void __launch_bounds__(1024) k_scan(const uint32_t* counts, uint32_t* offsets, int lists,
                                               int frames,
                                               const __grid_constant__ TablesArgs tables,
                                               const __grid_constant__ ScanSamples samples) {
  __shared__ CoilLastTile tiles[kCoilLastTiles];
  chain_wait();
  // (blocks of the next launch would take the places of those that move samples)
  if (samples.none) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  if (static_cast<int>(blockIdx.x) >= samples.first_block) {
    const int per_block = 32 * kCoilLastTiles;
    const int blocks = (samples.a.samples + per_block - 1) / per_block, groups = (samples.a.channels + 31) / 32;
    const int i = blockIdx.x - samples.first_block, frame = i / (blocks * groups);
    const int j = i - frame * blocks * groups, group = j / blocks, tile = threadIdx.x / 256;
    const int s0 = (j - group * blocks) * per_block + tile * 32;
    const int tx = threadIdx.x & 31, ty = (threadIdx.x >> 5) & 7;
    if (samples.bf16)
      coil_last_tile<KSJ_GPU_SAMPLES_BF16>(samples.a, frame, s0, group * 32, tiles[tile], tx, ty);
    else
      coil_last_tile<KSJ_GPU_SAMPLES_CF32>(samples.a, frame, s0, group * 32, tiles[tile], tx, ty);
    return;
  }
  if (static_cast<int>(blockIdx.x) >= frames) {
    const int i = (blockIdx.x - frames) * kTablesPerBlock + threadIdx.x;
    if (threadIdx.x < kTablesPerBlock && i < table_entries(tables)) table_entry(tables, i);
    return;
  }
  __shared__ uint32_t warp_sums[32];
  const int f = blockIdx.x;
  const uint32_t* c = counts + static_cast<size_t>(f) * lists;
  uint32_t* o = offsets + static_cast<size_t>(f) * (lists + 1);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int per = (lists + 1023) / 1024;
  const int base = warp * per * 32 + lane;
  uint32_t v[kScanPer];
  uint32_t local = 0;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) v[k] = k < per && base + 32 * k < lists ? __ldg(c + base + 32 * k) : 0u;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) local += v[k];
  local = __reduce_add_sync(0xffffffffu, local);
  if (lane == 0) warp_sums[warp] = local;
  __syncthreads();
  if (warp == 0) {
    uint32_t ws = warp_sums[lane];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, ws, d);
      if (lane >= d) ws += u;
    }
    warp_sums[lane] = ws;
  }
  __syncthreads();
  uint32_t run = warp_sums[warp] - local;
#pragma unroll
  for (int k = 0; k < kScanPer; ++k) {
    if (k >= per) break;
    uint32_t incl = v[k];
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t u = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += u;
    }
    if (base + 32 * k < lists) o[base + 32 * k] = run + incl - v[k];
    run += __shfl_sync(0xffffffffu, incl, 31);
  }
  if (threadIdx.x == 0) o[lists] = warp_sums[31];
}

// Blocks that move the samples of `frames` frames in the scan's launch.
inline size_t scan_sample_blocks(int samples, int channels, int frames) {
  return static_cast<size_t>((samples + 32 * kCoilLastTiles - 1) / (32 * kCoilLastTiles)) * ((channels + 31) / 32) *
         frames;
}

// The scan of `frames` frames, with the tables and the move of the samples where they are
// wanted.
ksj_gpu_status launch_scan(const uint32_t* counts, uint32_t* offsets, int lists, int frames,
                           const TablesArgs* tables, cudaStream_t stream, const CoilLastArgs* coil_last = nullptr,
                           bool bf16 = false) {
  const int extra = tables ? (table_entries(*tables) + kTablesPerBlock - 1) / kTablesPerBlock : 0;
  LaunchScope scope("k_scan", stream);
  ScanSamples samples{};
  samples.first_block = frames + extra;
  samples.none = coil_last == nullptr;
  size_t total = samples.first_block;
  if (coil_last != nullptr) {
    samples.a = *coil_last;
    samples.bf16 = bf16;
    total += scan_sample_blocks(coil_last->samples, coil_last->channels, frames);
  }
  return launch_chained(k_scan, dim3(static_cast<unsigned>(total)), 1024, 0, stream, counts, offsets, lists, frames,
                        tables ? *tables : TablesArgs{}, samples);
}

// One list entry (entry_bytes(W)) from its sample's record.
template <int W>
__device__ __forceinline__ void put_entry(uint32_t sidx, int c0, float wrow, const float* wc, int col_lo, int grid_cols,
                                          unsigned char* out) {
  float v[entry_bytes(W) / 4];
  v[0] = __int_as_float(c0 - col_lo >= kChunk ? c0 - col_lo - grid_cols : c0 - col_lo);
  v[1] = __uint_as_float(sidx);
#pragma unroll
  for (int j = 0; j < W; ++j) v[2 + j] = wrow * wc[j];
  if constexpr (entry_vectors(W)) {
#pragma unroll
    for (int q = 0; q < entry_bytes(W) / 16; ++q)
      reinterpret_cast<float4*>(out)[q] = make_float4(v[4 * q], v[4 * q + 1], v[4 * q + 2], v[4 * q + 3]);
  } else {
#pragma unroll
    for (int q = 0; q < entry_bytes(W) / 8; ++q) reinterpret_cast<float2*>(out)[q] = make_float2(v[2 * q], v[2 * q + 1]);
  }
}

// Density weights (2-D): a sample's double-precision taps, and one list
// entry as the grid step streams it.
template <int W>
struct PmRecord {
  int r0, c0;  // first tap row and column (wrapped)
  double wr[W];
  double wc[W];
};
template <int W>
struct alignas(16) PmEntry {
  double wr;     // the list's row weight (0: the taps miss the row)
  int t0;        // first tap's column as seen from the chunk, as in the float entries
  uint32_t sample;
  double wc[W];
};

struct PlaceArgs {
  const unsigned char* records;
  const uint32_t* offsets;  // [frame][list + 1]
  const uint32_t* starts;   // [frame][block][list]: the block's start in the list (k_bin_prefix)
  unsigned char* expanded;  // entries in their places
  const void* pm;           // density weights: the samples' PmRecords, and `expanded` takes PmEntry
  int samples, grid_rows, grid_cols, nchunks, lists_per_frame, bin_span;
  size_t entries_per_frame;
};

// One block per (block of samples, frame): kBinThreads samples at a time, their
// places in turn (place_turn), their entries written outside the turns.
//
// kPm: the entries are the density weights' (PmEntry).
//
// Bound by the chain of turns and, for one frame, by launches: appending to the
// lists with atomics and sorting each
// afterwards took three kernels (scatter, sort, long sort: 40 us of a 128-grid
// slice, 92 us of 205824 samples on a 512 grid, 219 us of 96 frames of 13056
// samples) where this and k_bin_prefix take 21, 60 and 144.  (Finding the ranks inside the
// turns, by lane masks per list in shared memory, took 203 of the 144.)
template <int W, bool kPm, int kLists>
__global__ void __launch_bounds__(kBinThreads) k_place(PlaceArgs a) {
  extern __shared__ uint32_t place_smem[];
  chain_begin();
  uint32_t* at = place_smem;  // running position of each list
  const int f = blockIdx.y;
  {
    const uint32_t* off = a.offsets + static_cast<size_t>(f) * (a.lists_per_frame + 1);
    const uint32_t* st = a.starts + (static_cast<size_t>(f) * gridDim.x + blockIdx.x) * a.lists_per_frame;
#pragma unroll 8
    for (int l = threadIdx.x; l < a.lists_per_frame; l += kBinThreads) at[l] = __ldg(off + l) + __ldg(st + l);
  }
  const SampleRecord<W>* recs = reinterpret_cast<const SampleRecord<W>*>(a.records) + static_cast<size_t>(f) * a.samples;
  const int s0 = blockIdx.x * a.bin_span, s1 = min(s0 + a.bin_span, a.samples);
  for (int base = s0; base < s1; base += kBinThreads) {
    const int sample = base + threadIdx.x;
    constexpr int kRV = static_cast<int>(sizeof(SampleRecord<W>) / 16);
    float4 q[kRV];
    if (sample < s1) {
#pragma unroll
      for (int v = 0; v < kRV; ++v) q[v] = __ldg(reinterpret_cast<const float4*>(recs + sample) + v);
    }
    const float* w = reinterpret_cast<const float*>(q);
    const int r0 = sample < s1 ? __float_as_int(w[0]) : -1;  // -1: also a padding sample of a ragged batch
    const int c0 = r0 >= 0 ? __float_as_int(w[1]) : 0;
    int chunks[kLists];
    list_chunks<W>(c0, a.grid_cols, chunks);
    uint32_t pos[W][kLists];
    place_turn<W>(at, r0, chunks, a.nchunks, a.grid_rows, pos);
    if (r0 < 0) continue;
    PmRecord<W> pm;
    if constexpr (kPm) pm = static_cast<const PmRecord<W>*>(a.pm)[static_cast<size_t>(f) * a.samples + sample];
#pragma unroll
    for (int j = 0; j < W; ++j) {
#pragma unroll
      for (int h = 0; h < kLists; ++h) {
        if (!own_list(chunks, h)) continue;
        const size_t slot = static_cast<size_t>(f) * a.entries_per_frame + pos[j][h];
        const int col_lo = chunks[h] * kChunk;
        if constexpr (kPm) {
          // the taps of the double-precision coordinate, on the list's row and chunk
          int dr = (r0 + j >= a.grid_rows ? r0 + j - a.grid_rows : r0 + j) - pm.r0;
          if (dr < 0) dr += a.grid_rows;
          PmEntry<W> e;
          e.wr = 0.0;
#pragma unroll
          for (int k = 0; k < W; ++k) {
            if (k == dr) e.wr = pm.wr[k];
            e.wc[k] = pm.wc[k];
          }
          e.t0 = pm.c0 - col_lo >= kChunk ? pm.c0 - col_lo - a.grid_cols : pm.c0 - col_lo;
          e.sample = static_cast<uint32_t>(sample);
          reinterpret_cast<PmEntry<W>*>(a.expanded)[slot] = e;
        } else {
          put_entry<W>(static_cast<uint32_t>(sample), c0, w[4 + j], w + 4 + W, col_lo, a.grid_cols,
                       a.expanded + slot * entry_bytes(W));
        }
      }
    }
  }
}

struct RowsArgs {
  int frame0;             // first frame of this pass
  const float2* samples_t;     // [frame][sample][channel], weighted
  size_t sample_frame_stride;  // elements between frames of samples_t (0: one sample set for all frames)
  const uint32_t* offsets;
  const unsigned char* expanded;  // list entries (entry_bytes(width) each)
  const float2* tw_cols;
  const int* pos_cols;    // DIF output position of each kept column
  float2* inter;          // [frame][grid_row][out_col][cpitch]
  uint32_t* flags;
  int frames, channels, samples, grid_rows, grid_cols, nchunks, lists_per_frame, width;
  size_t entries_per_frame;
  int coil_group, coil_parts;
  int both_ends;  // block x takes rows in from both ends
  int out_cols, cpitch;
  int col_shift;  // kept column of frequency k: (k + col_shift) mod grid_cols, when below out_cols
  int first_of_two;  // as in Shape
  uint32_t wait_limit;   // polls before a segment wait gives up
  int wait_beyond;       // added to every segment wait's target: 0, or unreachable in the wait-fault test mode
  DifPlan plan;
};

// Lists longer than a row's unit are gridded in segments (all but the last of
// segment_length entries) that different lane
// groups take at once, so that a row's long lists do not hold its CTA at the
// barrier after the gridding while one warp works through each; a cell is then
// the sum, in segment order, of its segments' partial sums, each partial sum
// in sample order from zero.  Shorter lists are one segment: the cell is its
// samples' sum in sample order.  The unit is kSegMin entries, or a 32nd of the
// row's where that is more (a row with that many has lists enough to share out,
// and every segment pays for putting its 16 cells in turn), but at most kSegMost: it depends on the
// lists alone, so every coil grouping gives the same cells.  Units of 32, 64, 128 entries
// and this rule measured, us of the row pass: 8 coils on a 128 grid 35, 29, 33,
// 28, on a 512 grid 131, 107, 99, 95; a 32-coil frame 35, 31, 37, 32.
// The upper bound keeps the sums short where rows are crowded (the centre of a
// kooshball: rows of 3e5 entries, lists of half of them, which without it are 16 segments of 9000).
// Mean and largest error against double precision of 24 images, 256 000 to 2 M kooshball samples on 24^3 to 96^3 grids,
// 1e-7: no bound 9.9, 29; bounds of 128, 256, 512, 1024: 7.1, 12; 6.0, 10; 5.6, 6.8; 5.6, 7.0 (the
// sum of the segments grows as they get shorter).  Row pass of 10.2 M samples x 20 coils on 384^3, ms:
// 19.46 without, 19.53, 19.29, 19.18, 19.18; of the 512 grid above, whose centre has units of 281,
// us: 82, 87, 90, 82, 82 (a few tasks more than a block takes at once are a round more).
constexpr int kSegMin = 64;
constexpr int kSegMost = 512;

__device__ __forceinline__ int segment_unit(int row_entries) {
  return min(max(kSegMin, (row_entries + 32 - 1) / 32), kSegMost);
}
__device__ __forceinline__ int list_segments(int n, int unit) { return n <= unit ? 1 : (n + unit - 1) / unit; }
__device__ __forceinline__ int segment_length(int n, int unit) {
  if (n <= unit) return n;  // one segment (most lists): no division
  const int sg = list_segments(n, unit);
  return (n + sg - 1) / sg;
}

// Up to kRowsBatch entries of one list staged by their lane group (`lanes`
// lanes, this one is `gl`): slot i gets entry i's weights spread over the
// chunk's 16 columns, so that the lanes that apply them need no column
// arithmetic and no branch per tap, and lane groups on different lists run in
// step.  Slots from cnt on get no weights.  wrap: the row's length where
// its first chunk may see both ends of a wrapped stencil, else 0.  Returns this lane's share of the
// halves its slots touch: bit 2 i the low, 2 i + 1 the high half of slot i.
__device__ __forceinline__ uint32_t stage_entries(int w, float* slots, const unsigned char* ent, int cnt, int gl,
                                                  int lanes, int wrap) {
  uint32_t halves = 0;
#pragma unroll 1
  for (int i = gl; i < kRowsBatch; i += lanes) {
    float* slot = slots + i * kSlotFloats;
    float4* s4 = reinterpret_cast<float4*>(slot);
    float2 h = make_float2(__int_as_float(-kMaxWidth), 0.0f), p0 = h, p1 = h;  // no tap, no sample
    const float2* e = reinterpret_cast<const float2*>(ent + i * entry_bytes(w));
    if (i < cnt) {
      if (entry_vectors(w)) {
        const float4 q = __ldg(reinterpret_cast<const float4*>(e));
        h = make_float2(q.x, q.y);
        p0 = make_float2(q.z, q.w);
      } else {
        h = __ldg(e);
        p0 = __ldg(e + 1);
      }
      if (w > 2) p1 = __ldg(e + 2);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) s4[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    slot[kChunk] = h.y;
    const int t0 = __float_as_int(h.x);
    auto put = [&](int t, float v) {
      if (wrap != 0 && t >= wrap) t -= wrap;
      if (static_cast<uint32_t>(t) < kChunk) slot[t] = v;
    };
    put(t0, p0.x);
    put(t0 + 1, p0.y);
    if (w > 2) {
      put(t0 + 2, p1.x);
      put(t0 + 3, p1.y);
    }
#pragma unroll 1
    for (int j = 4; j < w; j += 2) {
      const float2 p = i < cnt ? __ldg(e + 1 + j / 2) : make_float2(0.0f, 0.0f);
      put(t0 + j, p.x);
      put(t0 + j + 1, p.y);
    }
    if (i < cnt) halves |= (wrap != 0 ? 3u : (t0 < 8 ? 1u : 0u) | (t0 + w > 8 ? 2u : 0u)) << (2 * i);
  }
  return halves;
}

// A chunk's cells of one coil in registers: real and imaginary parts of columns 2 t
// and 2 t + 1 as packed pairs, so that the staged weights are operands as they lie
// (parts of one column as a pair would need every weight twice).
struct ChunkCells {
  float2 re[kChunk / 2], im[kChunk / 2];
  __device__ __forceinline__ float2 cell(int t) const {
    return t & 1 ? make_float2(re[t / 2].y, im[t / 2].y) : make_float2(re[t / 2].x, im[t / 2].x);
  }
};

// Eight columns of the chunk: the staged weights of one entry on its sample.
template <int kFirst>
__device__ __forceinline__ void half_taps(ChunkCells& r, const float* slot, float2 y) {
  const float4 a = reinterpret_cast<const float4*>(slot)[kFirst / 4];
  const float4 b = reinterpret_cast<const float4*>(slot)[kFirst / 4 + 1];
  const float2 w[4] = {{a.x, a.y}, {a.z, a.w}, {b.x, b.y}, {b.z, b.w}};
  const float2 re = make_float2(y.x, y.x), im = make_float2(y.y, y.y);
#pragma unroll
  for (int t = 0; t < 4; ++t) {
    r.re[kFirst / 2 + t] = __ffma2_rn(re, w[t], r.re[kFirst / 2 + t]);
    r.im[kFirst / 2 + t] = __ffma2_rn(im, w[t], r.im[kFirst / 2 + t]);
  }
}

// The chunk's cells from registers into the accumulator (dst: the chunk's
// first cell of this lane's coil, cells `stride` apart).  A one-segment list
// (counter null) stores them.  For a segmented list each lane works on its
// own coil's cells alone: segment 0 stores, segment seg > 0 waits until the
// list's counter shows all `lanes` lanes of segments 0 .. seg-1 in, then adds its
// partial sums; every lane then counts itself in.  Lanes wait on the counter
// each for itself (no warp-wide sync), fenced on both sides.  The wait is
// bounded: on a timeout the lane's partial sums are dropped, it still counts
// itself in (the later segments do not wait out the limit as well) and
// KSJ_GPU_FLAG_WAIT_TIMEOUT is raised.
__device__ __forceinline__ void put_chunk(const ChunkCells& r, float2* dst, int stride, int width, int seg,
                                          int lanes, int* counter, uint32_t* flags, uint32_t wait_limit,
                                          int wait_beyond) {
  if (counter == nullptr) {
    if (width == kChunk) {  // every chunk of the row but a partial last one
#pragma unroll
      for (int t = 0; t < kChunk; ++t) dst[t * stride] = r.cell(t);
    } else {
#pragma unroll
      for (int t = 0; t < kChunk; ++t)
        if (t < width) dst[t * stride] = r.cell(t);
    }
    return;
  }
  // segmented list: every lane of segments 0 .. seg-1 has counted itself in
  bool ok = true;
  if (seg > 0) {
    uint32_t polls = 0;
    while (*reinterpret_cast<volatile int*>(counter) < lanes * seg + wait_beyond) {
      if (++polls >= wait_limit) {
        ok = false;
        atomicOr(flags, KSJ_GPU_FLAG_WAIT_TIMEOUT);
        break;
      }
      __nanosleep(32);
    }
    __threadfence_block();
  }
  if (ok) {
#pragma unroll
    for (int t = 0; t < kChunk; ++t) {
      if (t < width) {
        float2 v = r.cell(t);
        if (seg > 0) {
          const float2 c = dst[t * stride];
          v = make_float2(c.x + v.x, c.y + v.y);
        }
        dst[t * stride] = v;
      }
    }
  }
  __threadfence_block();
  atomicAdd(counter, 1);
}

// One CTA per (frame, grid row, coil group): the row's cells gridded into
// shared memory [column][coil], then the row's inverse transform and the kept
// columns written coil-last.
//
// Gridding.  A task is one segment of one list (times the coil parts); a lane
// group (lane = coil, `lanes` of them) grids a task into registers, the 16
// cells of its chunk, and a warp takes as many tasks at once as it has lane
// groups, longest first, from a shared counter.  The groups of a warp run in step
// on different lists (neighbours in length), because a staged entry's weights
// are spread over the whole chunk: the same 8 or 16 multiply-adds whatever the
// columns, where a tap switch would send every group its own way.  Tasks are
// claimed in increasing order and a warp's groups are put in that order, so the
// smallest unfinished segment is always some warp's current one: a segment's
// wait for its predecessors always ends.
//
// Bound by issue slots (32 coils: two thirds of the cycles issue) and, for few
// rows, by the longest row.  A call, before (a switch on the tap column for 32 coils, cells in
// shared memory below) -> now: 96 frames x 384 rows x 32 coils 2597 -> 2488 us, one
// such frame 141 -> 119, 8 coils on a 512 grid 585 -> 330, on a 128 grid 210 -> 115,
// 11 coils, width 6, on a 300 grid 670 -> 385, 20 coils in 3-D 57.9 -> 46.7 ms.
//
// kN: the row length for the two-step transform (128 .. 512), or 0 for the
// in-place mixed-radix form of any other length; one instance per length keeps
// each kernel's code small.  kLgL (when nonzero) fixes log2 of the coil group, taken
// whole (coil_parts 1), and with it the lane groups (3 % of the row pass at 32 coils).
// kHalf: the sigma = 2 crop form of the row transform (out_cols =
// grid_cols / 2, col_shift = out_cols / 2), whose kept columns are known at
// compile time (fft_two_step_half); the same bytes as the general form.
template <int kN, int kLgL, bool kHalf>
__global__ void __launch_bounds__(kRowsThreads, 2) k_rows(RowsArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  chain_begin();
  const int row = !a.both_ends ? blockIdx.x
                  : (blockIdx.x & 1) ? a.grid_rows - 1 - static_cast<int>(blockIdx.x >> 1)
                                     : static_cast<int>(blockIdx.x >> 1);
  const int cgi = blockIdx.y;
  const int f = a.frame0 + blockIdx.z;
  const int cg = kLgL ? (1 << kLgL) : a.coil_group;
  const int tid = threadIdx.x;
  const int nthreads = blockDim.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  float2* acc = reinterpret_cast<float2*>(smem_raw);
  float2* tw = acc + static_cast<size_t>(a.grid_cols) * cg;
  // offsets from the shared array itself keep every access a shared-memory one
  const size_t slot_off = (static_cast<size_t>(a.grid_cols) * (cg + 1) * sizeof(float2) + 15) & ~static_cast<size_t>(15);

  const uint32_t* off = a.offsets + static_cast<size_t>(f) * (a.lists_per_frame + 1) + row * a.nchunks;
  // the row's task table: rank r is the r-th longest list (a bitonic sort
  // across warp 0, one key per lane: length << 8 | chunk), cut into
  // list_segments(len) segments; tasks task_base[r] .. task_base[r + 1] - 1
  // are its segments
  __shared__ int4 task_list[kMaxGrid / kChunk];  // per rank: first entry, length, segment length, chunk
  __shared__ int task_base[kMaxGrid / kChunk + 1];
  __shared__ int task_combined[2 * (kMaxGrid / kChunk)];  // per (part, chunk): lanes of finished segments
  __shared__ int task_next;
  if (warp == 0) {
    int key = -1;
    uint32_t start = 0, length = 0;
    if (lane < a.nchunks) {
      start = __ldg(off + lane);
      length = __ldg(off + lane + 1) - start;
      key = static_cast<int>(min(length, 1u << 22) << 8) | lane;
    }
#pragma unroll
    for (int k = 2; k <= 32; k <<= 1) {
#pragma unroll
      for (int j = k >> 1; j > 0; j >>= 1) {
        const int other = __shfl_xor_sync(0xffffffffu, key, j);
        const bool lower = (lane & j) == 0;
        const bool desc = (lane & k) == 0;
        key = (lower == desc) ? max(key, other) : min(key, other);
      }
    }
    const int chunk = key & 31;
    start = __shfl_sync(0xffffffffu, start, chunk);
    length = __shfl_sync(0xffffffffu, length, chunk);
    // segments per rank and their exclusive prefix (the key's length is capped for the
    // order alone)
    const int n = lane < a.nchunks ? static_cast<int>(length) : 0;
    const int unit = segment_unit(__reduce_add_sync(0xffffffffu, n));
    const int nseg = lane < a.nchunks ? list_segments(n, unit) : 0;
    int incl = nseg;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const int v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane < a.nchunks) {
      task_list[lane] = make_int4(static_cast<int>(start), n, segment_length(n, unit), chunk);
      task_base[lane] = incl - nseg;
    }
    if (lane == a.nchunks - 1) task_base[a.nchunks] = incl;
    if (lane == 0) task_next = 0;
  }
  for (int i = tid; i < 2 * (kMaxGrid / kChunk); i += nthreads) task_combined[i] = 0;
  for (int i = tid; i < a.grid_cols; i += nthreads) tw[i] = a.tw_cols[i];
  __syncthreads();

  {
    const int lg_parts = kLgL ? 0 : a.coil_parts - 1;  // coil_parts is 1 or 2
    const int lanes = cg >> lg_parts, groups = 32 / lanes;
    const int g = lane / lanes, gl = lane & (lanes - 1);
    float* slots = reinterpret_cast<float*>(smem_raw + slot_off) +
                   static_cast<size_t>(warp * groups + g) * kRowsBatch * kSlotFloats;
    const int ntasks = task_base[a.nchunks] << lg_parts;
    const bool segmented_row = task_base[a.nchunks] != a.nchunks;
    const int wrap = a.nchunks == 1 || a.first_of_two ? a.grid_cols : 0;
    const float2* samples = a.samples_t + static_cast<size_t>(f) * a.sample_frame_stride;
    const unsigned char* ents = a.expanded + static_cast<size_t>(f) * a.entries_per_frame * entry_bytes(a.width);
    for (;;) {
      int q = 0;
      if (lane == 0) q = atomicAdd(&task_next, groups);
      q = __shfl_sync(0xffffffffu, q, 0);
      if (q >= ntasks) break;
      q += g;
      const bool live = q < ntasks;
      const int part = q & lg_parts;
      q >>= lg_parts;
      // (rank, segment) of the task; a row without segmented lists has task q = rank q
      int rank = live ? q : 0, seg = 0;
      if (segmented_row) {
        rank = 0;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
          if (rank + d < a.nchunks && task_base[rank + d] <= q) rank += d;
        seg = q - task_base[rank];
      }
      const int4 list = task_list[rank];
      const int chunk = list.w;
      const int first = seg * list.z;
      const int cnt = live ? max(0, min(list.y - first, list.z)) : 0;
      const unsigned char* ent = ents + (static_cast<size_t>(static_cast<uint32_t>(list.x)) + first) * entry_bytes(a.width);
      const int coil = part * lanes + gl;
      // (lanes past the channels read the first coil: their lines are not kept)
      const SampleRows<KSJ_GPU_SAMPLES_CF32> sample_row(
          samples, cgi * cg + coil < a.channels ? cgi * cg + coil : 0, a.channels);
      ChunkCells r;
#pragma unroll
      for (int t = 0; t < kChunk / 2; ++t) r.re[t] = r.im[t] = make_float2(0.0f, 0.0f);
      const int most = __reduce_max_sync(0xffffffffu, cnt);
      for (int base = 0; base < most; base += kRowsBatch) {
        __syncwarp();  // the previous batch is read by every lane before it is replaced
        const uint32_t halves = __reduce_or_sync(
            0xffffffffu, stage_entries(a.width, slots, ent + base * entry_bytes(a.width), cnt - base, gl, lanes, wrap));
        __syncwarp();
        // every sample of the batch is requested before the first is used
        float2 y[kRowsBatch];
#pragma unroll
        for (int i = 0; i < kRowsBatch; ++i) {
          // (32 lanes: a slot past the list has no weights and is skipped as a whole)
          y[i] = make_float2(0.0f, 0.0f);
          if (kLgL == 5 || base + i < cnt)
            y[i] = sample_row(reinterpret_cast<const uint32_t*>(slots + i * kSlotFloats)[kChunk]);
        }
#pragma unroll
        for (int i = 0; i < kRowsBatch; ++i) {
          if (halves & (1u << (2 * i))) half_taps<0>(r, slots + i * kSlotFloats, y[i]);
          if (halves & (2u << (2 * i))) half_taps<8>(r, slots + i * kSlotFloats, y[i]);
        }
      }
      float2* dst = acc + chunk * kChunk * cg + coil;
      const int width = min(kChunk, a.grid_cols - chunk * kChunk);
      const bool segmented = live && list.z < list.y;
      if (!__any_sync(0xffffffffu, segmented)) {
        if (live) put_chunk(r, dst, cg, width, 0, lanes, nullptr, a.flags, a.wait_limit, a.wait_beyond);
      } else {
        // in task order: a group may wait for the segment of an earlier one
        for (int k = 0; k < groups; ++k) {
          if (k == g && live)
            put_chunk(r, dst, cg, width, seg, lanes, segmented ? task_combined + part * a.nchunks + chunk : nullptr,
                      a.flags, a.wait_limit, a.wait_beyond);
          __syncwarp();
        }
      }
    }
  }
  __syncthreads();

  // ---- row inverse FFT of every coil line; the kept columns are written
  // coil-last: [frame][grid_row][out_col][channel]
  const int lg_cg = kLgL ? kLgL : ilog2(cg);
  float2* dst_row = a.inter + (static_cast<size_t>(f) * a.grid_rows + row) * a.out_cols * a.cpitch + cgi * cg;
  const int live_lines = min(cg, a.channels - cgi * cg);
  if constexpr (kN != 0 && kHalf) {
    fft_two_step_half<16, kN / 16>(
        acc, lg_cg, tw, tid, nthreads, [&](int line) { return line < live_lines; },
        [&](int pc, int, int line, float2 v) { dst_row[static_cast<size_t>(pc) * a.cpitch + line] = v; });
  } else if constexpr (kN != 0) {
    fft_two_step<16, kN / 16>(acc, lg_cg, tw, tid, nthreads, [&](int k, int line, float2 v) {
      int pc = k + a.col_shift;
      if (pc >= a.grid_cols) pc -= a.grid_cols;
      if (pc < a.out_cols && line < live_lines) dst_row[static_cast<size_t>(pc) * a.cpitch + line] = v;
    });
  } else {
    // other lengths: in place (output digit-reversed), then the kept columns
    dif_lines(acc, lg_cg, a.plan, tw, tid, nthreads);
    const int coil = tid & (cg - 1);
    if (coil < live_lines) {
      for (int pc = tid >> lg_cg; pc < a.out_cols; pc += nthreads >> lg_cg)
        dst_row[static_cast<size_t>(pc) * a.cpitch + coil] = acc[(__ldg(a.pos_cols + pc) << lg_cg) + coil];
    }
  }
}

struct ColsArgs {
  const float2* tw_rows;
  const float* inv_dr;
  const float* inv_dc;
  const int* pos_rows;  // DIF output position of each kept row
  void* out;
  uint32_t* flags;
  int frame0;  // first frame of this pass
  int frames, channels, grid_rows, out_rows, out_cols, kb;
  int column_block, col_group, groups;  // tile: column_block columns x col_group coils; groups tiles per block
  int box_rows, boxes;                  // TMA boxes of box_rows rows cover one tile
  uint32_t output;                      // RSS or COIL_LAST (COIL_MAJOR goes through COIL_LAST + transpose)
  int out_pitch;                        // COIL_LAST: elements between pixels of the output (>= channels)
  int row_shift;                        // kept row of frequency k: (k + row_shift) mod grid_rows, when below out_rows
  DifPlan plan;
  // persistent form (k_cols_ring): tiles of tile_coils coils x (kRingLines /
  // tile_coils) columns; a unit is (frame, column block), tiles_per_unit
  // tiles of consecutive coils each; units = frames of the pass x col_blocks
  int tile_coils, tiles_per_unit, units, col_blocks;
};


// One CTA per (frame, column block).  The row-transformed grid
// [frame][grid_row][out_col][channel] is read one tile (grid_rows x
// column_block columns x col_group coils, coils contiguous) at a time by
// TMA; with more than one coil group the next tile's copy is in flight while
// the block transforms the current one.  Each tile is inverse-transformed
// along rows in place (lines = (column, coil) pairs), cropped and
// deapodised; then either written coil-last or squared in place and summed
// over coils in channel order per pixel.  The channel-order sum runs lane =
// pixel with lane j reading coil t - j at step t, so the 32 lanes read 32
// different coils (distinct banks) while each pixel still adds its coils
// 0, 1, 2, ... in order: the result is bit-identical to the RSS of the coil
// images.
//
// kN is the column length for the two-step transform (128 .. 512, see
// has_two_step_rows), or 0 for the in-place mixed-radix form of any other
// length; one instance per length keeps each kernel's code small.
// kLgL (when nonzero) fixes log2 of the line count (column_block x
// col_group) at compile time; kHalf selects the sigma = 2 crop form of the
// two-step transform (out_rows = grid_rows / 2, row_shift = out_rows / 2,
// Kaiser-Bessel deapodisation), whose kept rows are known at compile time.
// Every form gives the same bytes.
template <int kN, int kLgL = 0, bool kHalf = false>
__global__ void __launch_bounds__(kColsThreads) k_cols(const __grid_constant__ CUtensorMap inter_map, ColsArgs a) {
  extern __shared__ __align__(16) unsigned char smem_cols[];
  chain_begin();
  unsigned char* smem_raw = smem_cols;
  const int cb = a.column_block;
  const int cgc = a.col_group;
  const int lines = kLgL ? (1 << kLgL) : cb * cgc;
  const int lg_lines = kLgL ? kLgL : ilog2(lines);
  const int lg_cgc = ilog2(cgc);
  const int lg_cb = ilog2(cb);
  const int col0 = blockIdx.x * cb;
  const int fg = a.frame0 + blockIdx.y;
  const int tid = threadIdx.x;
  const int nthreads = blockDim.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  const int nbuf = a.groups > 1 ? 2 : 1;
  // each tile buffer starts on a 128-byte boundary (TMA destination)
  const size_t tile_elems = (static_cast<size_t>(a.grid_rows) * lines + 15) & ~static_cast<size_t>(15);
  float2* tiles = reinterpret_cast<float2*>(smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u));
  float2* tw = tiles + nbuf * tile_elems;
  float* rss = reinterpret_cast<float*>(tw + a.grid_rows);
  const int npix = a.out_rows * cb;
  uint64_t* bars = reinterpret_cast<uint64_t*>(rss + ((npix + 1) & ~1));
  float* inv_dr = reinterpret_cast<float*>(bars + 2);  // row deapodisation, out_rows values
  const uint32_t tile_bytes = static_cast<uint32_t>(static_cast<size_t>(a.grid_rows) * lines * sizeof(float2));
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_init_fence();
  }
  for (int i = tid; i < a.grid_rows; i += nthreads) tw[i] = a.tw_rows[i];
  for (int i = tid; i < npix; i += nthreads) rss[i] = 0.0f;
  if (a.kb)
    for (int i = tid; i < a.out_rows; i += nthreads) inv_dr[i] = __ldg(a.inv_dr + i);
  __syncthreads();
  auto issue = [&](int g, int b) {
    float2* dst = tiles + b * tile_elems;
    mbar_arrive_expect_tx(&bars[b], tile_bytes);
    for (int k = 0; k < a.boxes; ++k)
      tma_load_3d(dst + static_cast<size_t>(k) * a.box_rows * lines, &inter_map, g * cgc, col0,
                  fg * a.grid_rows + k * a.box_rows, &bars[b]);
  };
  if (tid == 0) issue(0, 0);
  const int line = tid & (lines - 1);
  const int lcol = line >> lg_cgc;   // column within the block
  const int lcoil = line & (cgc - 1);
  const bool col_ok = col0 + lcol < a.out_cols;
  bool ok = true;
  int issued = 1;
  for (int g = 0; g < a.groups; ++g) {
    const int b = nbuf > 1 ? (g & 1) : 0;
    const uint32_t parity = static_cast<uint32_t>((nbuf > 1 ? (g >> 1) : g) & 1);
    if (tid == 0 && g + 1 < a.groups) {
      fence_proxy_async_shared();  // this buffer was last written by the generic proxy
      issue(g + 1, b ^ 1);
      ++issued;
    }
    const bool mine = mbar_wait_bounded(&bars[b], parity, kWaitLimit);
    if (!__syncthreads_and(mine)) {
      ok = false;
      break;
    }
    float2* tile = tiles + b * tile_elems;
    // crop and deapodise; coil-last images are written from here, RSS
    // inputs are squared in place at pos_rows[pr]
    auto emit_pixel = [&](int pr, int ln, float2* e, float2 x) {
      const int lc = ln >> lg_cgc;
      if (a.kb) {
        const float sc = inv_dr[pr] * __ldg(a.inv_dc + col0 + lc);
        x.x *= sc;
        x.y *= sc;
      }
      if (a.output == KSJ_GPU_OUTPUT_RSS) {
        e->x = __fadd_rn(__fmul_rn(x.x, x.x), __fmul_rn(x.y, x.y));
      } else {
        float2* o = static_cast<float2*>(a.out);
        o[((static_cast<size_t>(fg) * a.out_rows + pr) * a.out_cols + col0 + lc) * a.out_pitch + g * cgc +
          (ln & (cgc - 1))] = x;
      }
    };
    const int live_coils_g = min(cgc, a.channels - g * cgc);
    auto emit = [&](int k, int ln, float2 v) {
      int pr = k + a.row_shift;
      if (pr >= a.grid_rows) pr -= a.grid_rows;
      if (pr >= a.out_rows || col0 + (ln >> lg_cgc) >= a.out_cols || (ln & (cgc - 1)) >= live_coils_g) return;
      emit_pixel(pr, ln, tile + (two_step_slot(k, a.grid_rows) << lg_lines) + ln, v);
    };
    if constexpr (kN != 0 && kHalf) {
      auto live = [&](int ln) { return col0 + (ln >> lg_cgc) < a.out_cols && (ln & (cgc - 1)) < live_coils_g; };
      auto emit_half = [&](int pr, int slot, int ln, float2 v) {
        const int lc = ln >> lg_cgc;
        const float sc = inv_dr[pr] * __ldg(a.inv_dc + col0 + lc);
        v.x *= sc;
        v.y *= sc;
        if (a.output == KSJ_GPU_OUTPUT_RSS) {
          tile[(slot << lg_lines) + ln].x = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
        } else {
          float2* o = static_cast<float2*>(a.out);
          o[((static_cast<size_t>(fg) * a.out_rows + pr) * a.out_cols + col0 + lc) * a.out_pitch + g * cgc +
            (ln & (cgc - 1))] = v;
        }
      };
      fft_two_step_half<16, kN / 16>(tile, lg_lines, tw, tid, nthreads, live, emit_half);
    } else if constexpr (kN != 0) {
      fft_two_step<16, kN / 16>(tile, lg_lines, tw, tid, nthreads, emit);
    } else {
      dif_lines(tile, lg_lines, a.plan, tw, tid, nthreads);
      if (col_ok && lcoil < live_coils_g) {
        for (int pr = tid >> lg_lines; pr < a.out_rows; pr += nthreads >> lg_lines) {
          float2* e = tile + (static_cast<size_t>(__ldg(a.pos_rows + pr)) << lg_lines) + line;
          emit_pixel(pr, line, e, *e);
        }
      }
    }
    if (a.output == KSJ_GPU_OUTPUT_RSS) {
      __syncthreads();
      // channel-order sum per pixel (reductions.hpp:972-982)
      const int live_coils = min(cgc, a.channels - g * cgc);
      for (int q0 = warp * 32; q0 < npix; q0 += nthreads) {
        const int q = q0 + lane;
        const bool live = q < npix && col0 + (q & (cb - 1)) < a.out_cols;
        const int pr = q >> lg_cb;
        const int base = live ? (__ldg(a.pos_rows + pr) << lg_lines) + ((q & (cb - 1)) << lg_cgc) : 0;
        float total = live ? rss[q] : 0.0f;
        if (live_coils == 32) {
          // fixed trip count: every load of the walk can be issued ahead of
          // the dependent adds
#pragma unroll
          for (int t = 0; t < 63; ++t) {
            const int c = t - lane;
            if (live && c >= 0 && c < 32) total = __fadd_rn(total, tile[base + c].x);
          }
        } else {
          for (int t = 0; t < live_coils + 31; ++t) {
            const int c = t - lane;
            if (live && c >= 0 && c < live_coils) total = __fadd_rn(total, tile[base + c].x);
          }
        }
        if (live) rss[q] = total;
      }
    }
    __syncthreads();
  }
  if (!ok) {
    // a copy never completed: report, then give every copy this block issued
    // a bounded chance to land before the block's shared memory is released
    if (tid == 0) {
      atomicOr(a.flags, KSJ_GPU_FLAG_WAIT_TIMEOUT);
      for (int u = 0; u < issued; ++u) {
        const int bb = nbuf > 1 ? (u & 1) : 0;
        const uint32_t par = static_cast<uint32_t>((nbuf > 1 ? (u >> 1) : u) & 1);
        mbar_wait_bounded(&bars[bb], par, kWaitLimit);
      }
    }
    return;
  }
  if (a.output == KSJ_GPU_OUTPUT_RSS) {
    float* o = static_cast<float*>(a.out);
    for (int q = tid; q < npix; q += nthreads) {
      const int pr = q >> lg_cb;
      const int l = q & (cb - 1);
      if (col0 + l < a.out_cols) o[(static_cast<size_t>(fg) * a.out_rows + pr) * a.out_cols + col0 + l] = __fsqrt_rn(rss[q]);
    }
  }
}

// Persistent column pass for the two-step column lengths.  Each CTA walks
// its share of the (frame, column block) units -- units blockIdx.x,
// blockIdx.x + gridDim.x, ... -- one tile of kRingLines lines (tile_coils
// coils x kRingLines / tile_coils columns, all grid rows) at a time, through
// a two-stage ring of shared-memory tiles: while the block transforms tile i,
// the TMA copy of tile i + 1 is in flight, and tile i + 2's copy is issued as
// soon as tile i's stage is free.  Per line the arithmetic is the one-shot
// k_cols's (the same transform, crop and deapodisation); the RSS sums a
// pixel's coils in channel order across the unit's tiles (the accumulator
// carries over from tile to tile), so the bytes equal k_cols's.
constexpr int kRingLines = 16;
constexpr int kRingLgLines = 4;

template <int kN>
struct RingCfg;  // block size (step A of the two-step transform has kN / 16 x 16 tasks) and CTAs per SM
template <>
struct RingCfg<128> { static constexpr int kThreads = 256, kBlocks = 2; };
template <>
struct RingCfg<192> { static constexpr int kThreads = 256, kBlocks = 2; };
template <>
struct RingCfg<256> { static constexpr int kThreads = 256, kBlocks = 2; };
template <>
struct RingCfg<384> { static constexpr int kThreads = 384, kBlocks = 2; };
template <>
struct RingCfg<512> { static constexpr int kThreads = 512, kBlocks = 1; };

template <int kN>
__global__ void __launch_bounds__(RingCfg<kN>::kThreads, RingCfg<kN>::kBlocks)
    k_cols_ring(const __grid_constant__ CUtensorMap inter_map, ColsArgs a) {
  constexpr int kT = RingCfg<kN>::kThreads;
  constexpr int kL = kRingLines;
  constexpr int kLgL = kRingLgLines;
  extern __shared__ __align__(16) unsigned char smem_cols[];
  unsigned char* smem_raw = smem_cols;
  chain_begin();
  const int tc = a.tile_coils;
  const int lg_tc = ilog2(tc);
  const int cb = kL / tc;  // columns per tile
  const int lg_cb = kLgL - lg_tc;
  const int tid = threadIdx.x;
  const int tpu = a.tiles_per_unit;
  constexpr size_t kTileElems = static_cast<size_t>(kN) * kL;
  float2* tiles = reinterpret_cast<float2*>(smem_raw + ((128u - (smem_addr(smem_raw) & 127u)) & 127u));
  float2* tw = tiles + 2 * kTileElems;
  float* rss = reinterpret_cast<float*>(tw + kN);
  const int npix = a.out_rows * cb;
  uint64_t* bars = reinterpret_cast<uint64_t*>(rss + ((npix + 1) & ~1));
  float* inv_dr = reinterpret_cast<float*>(bars + 2);
  constexpr uint32_t kTileBytes = static_cast<uint32_t>(kTileElems * sizeof(float2));
  if (tid == 0) {
    mbar_init(&bars[0], 1);
    mbar_init(&bars[1], 1);
    mbar_init_fence();
  }
  for (int i = tid; i < kN; i += kT) tw[i] = a.tw_rows[i];
  for (int i = tid; i < npix; i += kT) rss[i] = 0.0f;
  if (a.kb)
    for (int i = tid; i < a.out_rows; i += kT) inv_dr[i] = __ldg(a.inv_dr + i);
  __syncthreads();
  const int my_units = a.units > static_cast<int>(blockIdx.x)
                           ? (a.units - 1 - static_cast<int>(blockIdx.x)) / static_cast<int>(gridDim.x) + 1
                           : 0;
  const int ntiles = my_units * tpu;
  auto unit_of = [&](int i) { return static_cast<int>(blockIdx.x) + (i / tpu) * static_cast<int>(gridDim.x); };
  auto issue = [&](int i) {
    const int u = unit_of(i), h = i - (i / tpu) * tpu;
    const int f = a.frame0 + u / a.col_blocks;
    const int col0 = (u - (u / a.col_blocks) * a.col_blocks) * cb;
    float2* dst = tiles + (i & 1) * kTileElems;
    mbar_arrive_expect_tx(&bars[i & 1], kTileBytes);
    for (int k = 0; k < a.boxes; ++k)
      tma_load_3d(dst + static_cast<size_t>(k) * a.box_rows * kL, &inter_map, h * tc, col0,
                  f * kN + k * a.box_rows, &bars[i & 1]);
  };
  if (tid == 0)
    for (int i = 0; i < 2 && i < ntiles; ++i) issue(i);
  int i = 0;
  bool ok = true;
  for (; i < ntiles; ++i) {
    const int b = i & 1;
    const bool mine = mbar_wait_bounded(&bars[b], static_cast<uint32_t>((i >> 1) & 1), kWaitLimit);
    if (!__syncthreads_and(mine)) {
      ok = false;
      break;
    }
    const int u = unit_of(i), h = i - (i / tpu) * tpu;
    const int fg = a.frame0 + u / a.col_blocks;
    const int col0 = (u - (u / a.col_blocks) * a.col_blocks) * cb;
    const int coil0 = h * tc;
    const int live_coils = min(tc, a.channels - coil0);
    float2* tile = tiles + b * kTileElems;
    auto emit = [&](int k, int ln, float2 v) {
      int pr = k + a.row_shift;
      if (pr >= kN) pr -= kN;
      const int lc = ln >> lg_tc;
      if (pr >= a.out_rows || col0 + lc >= a.out_cols || (ln & (tc - 1)) >= live_coils) return;
      if (a.kb) {
        const float sc = inv_dr[pr] * __ldg(a.inv_dc + col0 + lc);
        v.x *= sc;
        v.y *= sc;
      }
      if (a.output == KSJ_GPU_OUTPUT_RSS) {
        float2* e = tile + (two_step_slot(k, kN) << kLgL) + ln;
        e->x = __fadd_rn(__fmul_rn(v.x, v.x), __fmul_rn(v.y, v.y));
      } else {
        float2* o = static_cast<float2*>(a.out);
        o[((static_cast<size_t>(fg) * a.out_rows + pr) * a.out_cols + col0 + lc) * a.out_pitch + coil0 +
          (ln & (tc - 1))] = v;
      }
    };
    fft_two_step<16, kN / 16>(tile, kLgL, tw, tid, kT, emit);
    if (a.output == KSJ_GPU_OUTPUT_RSS) {
      __syncthreads();
      // channel-order sum per pixel (reductions.hpp:972-982), continued from
      // the unit's previous tiles; thread q owns pixel q in both loops below
      const int lane = tid & 31;
      for (int q0 = tid - lane; q0 < npix; q0 += kT) {
        const int q = q0 + lane;
        const bool live = q < npix && col0 + (q & (cb - 1)) < a.out_cols;
        const int pr = q >> lg_cb;
        const int base = live ? (__ldg(a.pos_rows + pr) << kLgL) + ((q & (cb - 1)) << lg_tc) : 0;
        float total = live ? rss[q] : 0.0f;
        for (int t = 0; t < live_coils + 31; ++t) {
          const int c = t - lane;
          if (live && c >= 0 && c < live_coils) total = __fadd_rn(total, tile[base + c].x);
        }
        if (live) rss[q] = total;
      }
      if (h == tpu - 1) {
        float* o = static_cast<float*>(a.out);
        for (int q = tid; q < npix; q += kT) {
          const int pr = q >> lg_cb;
          const int l = q & (cb - 1);
          if (col0 + l < a.out_cols) o[(static_cast<size_t>(fg) * a.out_rows + pr) * a.out_cols + col0 + l] =
              __fsqrt_rn(rss[q]);
          rss[q] = 0.0f;
        }
      }
    }
    __syncthreads();  // every thread is done with stage b
    if (tid == 0 && i + 2 < ntiles) {
      fence_proxy_async_shared();  // the stage was last written by the generic proxy
      issue(i + 2);
    }
  }
  if (!ok && tid == 0) {
    // a copy never completed: report, then give the copies still in flight
    // (tiles i and i + 1) a bounded chance to land before the block exits
    atomicOr(a.flags, KSJ_GPU_FLAG_WAIT_TIMEOUT);
    for (int t = i; t < i + 2 && t < ntiles; ++t)
      mbar_wait_bounded(&bars[t & 1], static_cast<uint32_t>((t >> 1) & 1), kWaitLimit);
  }
}

// ------------------------------------------------------------------ driver

using RowsKernel = void (*)(RowsArgs);

template <int kN>
RowsKernel rows_kernel_two_step(int cg, bool half) {
  switch (cg) {
    case 32: return half ? k_rows<kN, 5, true> : k_rows<kN, 5, false>;
    case 16: return half ? k_rows<kN, 4, true> : k_rows<kN, 4, false>;
    case 8: return half ? k_rows<kN, 3, true> : k_rows<kN, 3, false>;
    case 4: return half ? k_rows<kN, 2, true> : k_rows<kN, 2, false>;
    default: return half ? k_rows<kN, 0, true> : k_rows<kN, 0, false>;
  }
}

// The instance for rows of n columns; cg 0: a coil group and parts known at run time.
RowsKernel rows_kernel_for(int n, int cg, bool half) {
  switch (n) {
    case 128: return rows_kernel_two_step<128>(cg, half);
    case 192: return rows_kernel_two_step<192>(cg, half);
    case 256: return rows_kernel_two_step<256>(cg, half);
    case 384: return rows_kernel_two_step<384>(cg, half);
    case 512: return rows_kernel_two_step<512>(cg, half);
    default: return k_rows<0, 0, false>;
  }
}

// The row-pass kernel a shape selects, its launch setup and launch.
struct RowsLauncher {
  RowsKernel kernel = nullptr;
  int threads = 0;
  size_t smem = 0;

  bool setup(const Shape& s) {
    const int lanes = s.coil_group / s.coil_parts;
    threads = rows_threads_for(s.grid_cols, lanes, s.coil_group);
    smem = rows_smem_for(s.grid_cols, s.coil_group, lanes, threads);
    kernel = rows_kernel_for(s.grid_cols, s.coil_parts == 1 ? s.coil_group : 0, s.kb && s.out_cols * 2 == s.grid_cols);
    return allow_smem(kernel, smem, kRowsSmem) == KSJ_GPU_OK &&
           cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
  }

  // One pass of nf frames of grid_rows rows and `groups` coil groups.
  // A launch of few waves takes the rows in from both ends: frequency 0, where radial
  // scans crowd, is at row 0, and the rows before it, at the end, should not be the
  // last to start (a 32-coil frame 72 -> 65 us; 48 frames, 61 waves, 1 % slower).
  ksj_gpu_status launch(RowsArgs r, int grid_rows, int groups, int nf, cudaStream_t stream) const {
    r.both_ends = static_cast<long long>(grid_rows) * groups * nf <= 16 * 2 * kSms;
    LaunchScope scope("k_rows", stream);
    return launch_chained(kernel, dim3(grid_rows, groups, nf), threads, smem, stream, r);
  }
};

size_t cols_smem_bytes(const Shape& s) {
  const size_t lines = static_cast<size_t>(s.column_block) * s.col_group;
  const size_t tile = (static_cast<size_t>(s.grid_rows) * lines + 15) & ~static_cast<size_t>(15);
  const int nbuf = column_groups(s) > 1 ? 2 : 1;
  const size_t npix = static_cast<size_t>(s.out_rows) * s.column_block;
  return 128 + nbuf * tile * sizeof(float2) + s.grid_rows * sizeof(float2) + ((npix + 1) & ~size_t{1}) * sizeof(float) +
         2 * sizeof(uint64_t) + static_cast<size_t>(s.out_rows) * sizeof(float);
}

using ColsKernel = void (*)(const __grid_constant__ CUtensorMap, ColsArgs);

// The k_cols instance for columns of n grid rows; half: the sigma = 2 crop
// (out_rows = n / 2, row_shift = n / 4, Kaiser-Bessel), lines32: 32 lines per
// tile (the default column block).
template <int kN>
ColsKernel cols_kernel_two_step(bool half, bool lines32) {
  if (half) return lines32 ? k_cols<kN, 5, true> : k_cols<kN, 0, true>;
  return lines32 ? k_cols<kN, 5, false> : k_cols<kN, 0, false>;
}

ColsKernel cols_kernel_for(int n, bool half = false, bool lines32 = false) {
  switch (n) {
    case 128: return cols_kernel_two_step<128>(half, lines32);
    case 192: return cols_kernel_two_step<192>(half, lines32);
    case 256: return cols_kernel_two_step<256>(half, lines32);
    case 384: return cols_kernel_two_step<384>(half, lines32);
    case 512: return cols_kernel_two_step<512>(half, lines32);
    default: return k_cols<0>;
  }
}

// Opt a k_cols instance into its dynamic shared memory.
bool cols_kernel_setup(ColsKernel k, size_t smem) {
  return allow_smem(k, smem) == KSJ_GPU_OK &&
         cudaFuncSetAttribute(k, cudaFuncAttributePreferredSharedMemoryCarveout, 100) == cudaSuccess;
}

using EncodeTiledFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiledFn encode_tiled() {
  static EncodeTiledFn fn = [] {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q{};
    if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      p = nullptr;
    return reinterpret_cast<EncodeTiledFn>(p);
  }();
  return fn;
}

// Tensor map over the row-transformed grid [frame*grid_row][out_col][cpitch]
// of 8-byte elements, box (col_group coils, column_block columns, box_rows rows).
bool make_inter_map(const Shape& s, void* inter, CUtensorMap* map, int* box_rows, int* boxes) {
  EncodeTiledFn enc = encode_tiled();
  if (enc == nullptr) return false;
  *boxes = tile_boxes(s.grid_rows);
  *box_rows = s.grid_rows / *boxes;
  const cuuint64_t dims[3] = {static_cast<cuuint64_t>(s.cpitch), static_cast<cuuint64_t>(s.out_cols),
                              static_cast<cuuint64_t>(s.frames) * s.grid_rows};
  const cuuint64_t strides[2] = {static_cast<cuuint64_t>(s.cpitch) * 8,
                                 static_cast<cuuint64_t>(s.cpitch) * s.out_cols * 8};
  const cuuint32_t box[3] = {static_cast<cuuint32_t>(s.col_group), static_cast<cuuint32_t>(s.column_block),
                             static_cast<cuuint32_t>(*box_rows)};
  const cuuint32_t estr[3] = {1, 1, 1};
  return enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT64, 3, inter, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
             CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
             CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// Tensor map for the persistent column pass: box (tile_coils coils,
// kRingLines / tile_coils columns, box_rows rows).
bool make_ring_map(const Shape& s, void* inter, int tile_coils, CUtensorMap* map, int* box_rows, int* boxes) {
  Shape t = s;
  t.col_group = tile_coils;
  t.column_block = kRingLines / tile_coils;
  return make_inter_map(t, inter, map, box_rows, boxes);
}

using RingKernel = void (*)(const __grid_constant__ CUtensorMap, ColsArgs);

// The column pass of one shape: the persistent ring kernel for the two-step
// column lengths, else one k_cols CTA per (frame, column block).  Both give
// the same bytes.
struct ColsPass {
  bool ring = false;
  ColsKernel kernel = nullptr;
  size_t smem = 0;
  int threads = kColsThreads;
  int ctas = 0;
  int column_block = 1;
  int out_cols = 0;
  CUtensorMap map;

  bool setup(const Shape& s, void* inter, ColsArgs* c) {
    const int tc = std::min(s.col_group, kRingLines);
    const int cb = kRingLines / tc;
    out_cols = s.out_cols;
    ring = s.column_pass == 2 && has_two_step_rows(s.grid_rows) && tc >= 2 && cb <= s.out_cols;
    if (!ring) {
      column_block = s.column_block;
      smem = cols_smem_bytes(s);
      const bool half = c->kb && s.out_rows * 2 == s.grid_rows && c->row_shift == s.out_rows / 2;
      kernel = cols_kernel_for(s.grid_rows, half, s.column_block * s.col_group == 32);
      return cols_kernel_setup(kernel, smem) && make_inter_map(s, inter, &map, &c->box_rows, &c->boxes);
    }
    column_block = cb;
    c->tile_coils = tc;
    c->tiles_per_unit = (s.cpitch + tc - 1) / tc;
    c->col_blocks = (s.out_cols + cb - 1) / cb;
    int blocks = 2;
    switch (s.grid_rows) {
      case 128: kernel = k_cols_ring<128>; threads = RingCfg<128>::kThreads; blocks = RingCfg<128>::kBlocks; break;
      case 192: kernel = k_cols_ring<192>; threads = RingCfg<192>::kThreads; blocks = RingCfg<192>::kBlocks; break;
      case 256: kernel = k_cols_ring<256>; threads = RingCfg<256>::kThreads; blocks = RingCfg<256>::kBlocks; break;
      case 384: kernel = k_cols_ring<384>; threads = RingCfg<384>::kThreads; blocks = RingCfg<384>::kBlocks; break;
      default: kernel = k_cols_ring<512>; threads = RingCfg<512>::kThreads; blocks = RingCfg<512>::kBlocks; break;
    }
    const size_t npix = static_cast<size_t>(s.out_rows) * cb;
    smem = 128 + 2 * static_cast<size_t>(s.grid_rows) * kRingLines * sizeof(float2) + s.grid_rows * sizeof(float2) +
           ((npix + 1) & ~size_t{1}) * sizeof(float) + 2 * sizeof(uint64_t) + static_cast<size_t>(s.out_rows) * sizeof(float);
    int device = 0, sms = 0;
    if (cudaGetDevice(&device) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
      return false;
    ctas = sms * blocks;
    return cols_kernel_setup(kernel, smem) && make_ring_map(s, inter, tc, &map, &c->box_rows, &c->boxes);
  }

  // The column pass over nf frames starting at c.frame0.
  ksj_gpu_status launch(ColsArgs c, int nf, cudaStream_t stream, const char* name) const {
    LaunchScope scope(name, stream);
    if (!ring)
      return launch_chained(kernel, dim3((out_cols + column_block - 1) / column_block, nf), kColsThreads, smem, stream,
                            map, c);
    c.units = nf * c.col_blocks;
    return launch_chained(kernel, std::min(ctas, c.units), threads, smem, stream, map, c);
  }
};

// The binning lists of one call: per-sample records, list offsets, and the lists'
// entries in sample order, as the row pass reads them or, where `pm` holds the
// density weights' records, as their grid step does; and the call's tables where
// `tables` names them, and the samples in the row pass's order where `coil_last` does.  The
// flags must already be cleared.
template <int W>
ksj_gpu_status build_lists(const Shape& s, const ksj_gpu_gridding_desc* d, const float* d_traj, const float* d_dcf,
                           uint32_t* flags, unsigned char* records, uint32_t* counts, uint32_t* totals,
                           uint32_t* offsets, unsigned char* expanded, const void* pm, cudaStream_t stream,
                           uint32_t* frame_flags = nullptr, const TablesArgs* tables = nullptr,
                           const CoilLastArgs* coil_last = nullptr) {
  const int count_smem = s.lists_per_frame * 4;
  const int place_smem = s.lists_per_frame * static_cast<int>(kPlaceListBytes);
  auto prepare = k_prepare<W, 2>;
  auto place = pm ? k_place<W, true, 2> : k_place<W, false, 2>;
  if constexpr (W > 2) {
    if (s.lists_per_row == 3) {
      prepare = k_prepare<W, 3>;
      place = pm ? k_place<W, true, 3> : k_place<W, false, 3>;
    }
  }
  KSJ_TRY(allow_smem(prepare, count_smem, kListSmem));
  KSJ_TRY(allow_smem(place, place_smem, kListSmem));
  const dim3 blocks(s.bin_blocks, s.frames);
  {
    PrepareArgs p{};
    p.traj = d_traj;
    p.dcf = d_dcf;
    p.frame_samples = s.frame_samples;
    p.frame_traj = s.frame_traj;
    p.frame_flags = frame_flags;
    p.dcf_mode = d->dcf_mode;
    p.require_nyquist = d->require_nyquist;
    p.records = records;
    p.counts = counts;
    p.flags = flags;
    p.frames = s.frames;
    p.samples = s.samples;
    p.grid_rows = s.grid_rows;
    p.grid_cols = s.grid_cols;
    p.nchunks = s.nchunks;
    p.lists_per_frame = s.lists_per_frame;
    p.bin_span = s.bin_span;
    p.kb = s.kb ? 1 : 0;
    p.beta = s.beta;
    p.two_over_w = 2.0f / static_cast<float>(s.width);
    p.inv_i0_beta = s.inv_i0_beta;
    p.phase_row = s.phase_row;
    p.phase_col = s.phase_col;
    p.phase_sign = s.phase_sign;
    LaunchScope scope("k_prepare", stream);
    KSJ_TRY(launch_chained(prepare, blocks, kBinThreads, count_smem, stream, p));
  }
  {
    LaunchScope scope("k_bin_prefix", stream);
    KSJ_TRY(launch_chained(k_bin_prefix, dim3((s.lists_per_frame + 127) / 128, s.frames), 128, 0, stream, counts, totals,
                   s.bin_blocks, s.lists_per_frame));
  }
  KSJ_TRY(launch_scan(totals, offsets, s.lists_per_frame, s.frames, tables, stream, coil_last,
                      d->sample_format == KSJ_GPU_SAMPLES_BF16));
  {
    PlaceArgs p{};
    p.records = records;
    p.offsets = offsets;
    p.starts = counts;
    p.expanded = expanded;
    p.pm = pm;
    p.samples = s.samples;
    p.grid_rows = s.grid_rows;
    p.grid_cols = s.grid_cols;
    p.nchunks = s.nchunks;
    p.lists_per_frame = s.lists_per_frame;
    p.bin_span = s.bin_span;
    p.entries_per_frame = s.entries_per_frame;
    LaunchScope scope("k_place", stream);
    KSJ_TRY(launch_chained(place, blocks, kBinThreads, place_smem, stream, p));
  }
  return KSJ_GPU_OK;
}

// Streams and events of a multi-pass call.  Odd passes run on a second
// compute stream (`alt`, joined after the binning through `ready` and back
// through `alt_done`), so a pass's last, partly filled wave overlaps the
// next pass.  With host buffers (ksj_gpu_gridding_adjoint_host, `copy` set):
// pass p's samples reach device memory on the copy stream (event in[p]); the
// pass waits for them before its transpose, and its images go back to the
// host on the copy stream once the pass is done (event done[p]).
struct HostIo {
  cudaStream_t copy, alt;
  const cudaEvent_t* in;
  const cudaEvent_t* done;
  cudaEvent_t ready, alt_done;
  void* h_out;
  size_t out_frame_bytes;
};

template <int W, uint32_t kFormat>
ksj_gpu_status launch_all(const Shape& s, const Layout& l, const ksj_gpu_gridding_desc* d, const void* d_kspace,
                          const float* d_traj, const float* d_dcf, void* d_out, unsigned char* ws,
                          cudaStream_t stream, const HostIo* io = nullptr) {
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + l.flags);
  unsigned char* records = ws + l.records;
  uint32_t* offsets = reinterpret_cast<uint32_t*>(ws + l.offsets);
  float2* inter = reinterpret_cast<float2*>(ws + l.inter);
  float2* tw_rows = reinterpret_cast<float2*>(ws + l.tables);
  float2* tw_cols = tw_rows + s.grid_rows;
  float* inv_dr = reinterpret_cast<float*>(tw_cols + s.grid_cols);
  float* inv_dc = inv_dr + s.out_rows;
  int* pos_rows = reinterpret_cast<int*>(inv_dc + s.out_cols);
  int* pos_cols = pos_rows + s.out_rows;

  if (cudaMemsetAsync(ws + l.flags, 0, l.cleared - l.flags, stream) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  const double beta = s.beta;
  const TablesArgs tables{tw_rows, tw_cols, inv_dr, inv_dc, pos_rows, pos_cols, s.grid_rows, s.grid_cols, s.out_rows,
                          s.out_cols, s.plan_rows, s.plan_cols, s.kb ? 1 : 0, s.width, beta,
                          s.kb ? std::cyl_bessel_i(0.0, beta) : 1.0};
  CoilLastArgs coil_last{d_kspace, reinterpret_cast<float2*>(ws + l.samples_t), records + offsetof(SampleRecord<W>, scale),
                         static_cast<int>(sizeof(SampleRecord<W>)), s.channels, s.samples, flags, s.frame_channels,
                         s.frame_samples, s.frame_kspace, 0, reinterpret_cast<uint32_t*>(ws + l.frame_flags)};
  const bool samples_here = io == nullptr || io->copy == nullptr;  // (else pass by pass)
  const bool with_scan =
      samples_here && s.frames + scan_sample_blocks(s.samples, s.channels, s.frames) <= kScanSampleBlocks;
  {
    const ksj_gpu_status st =
        build_lists<W>(s, d, d_traj, d_dcf, flags, records, reinterpret_cast<uint32_t*>(ws + l.counts),
                       reinterpret_cast<uint32_t*>(ws + l.totals), offsets, ws + l.expanded, nullptr, stream,
                       reinterpret_cast<uint32_t*>(ws + l.frame_flags), &tables, with_scan ? &coil_last : nullptr);
    if (st != KSJ_GPU_OK) return st;
  }
  auto to_coil_last = [&](int f0, int nf, cudaStream_t st) {
    const dim3 tg((s.samples + 31) / 32, (s.channels + 31) / 32, nf);
    LaunchScope scope("k_samples_coil_last", st);
    coil_last.frame0 = f0;
    return launch_chained(k_samples_coil_last<kFormat>, tg, dim3(32, 8), 0, st, coil_last);
  };
  if (samples_here && !with_scan) KSJ_TRY(to_coil_last(0, s.frames, stream));
  RowsArgs r{};
  r.samples_t = reinterpret_cast<const float2*>(ws + l.samples_t);
  r.sample_frame_stride = static_cast<size_t>(s.samples) * s.channels;
  r.offsets = offsets;
  r.expanded = ws + l.expanded;
  r.width = s.width;
  r.tw_cols = tw_cols;
  r.pos_cols = pos_cols;
  r.inter = inter;
  r.flags = flags;
  r.frames = s.frames;
  r.channels = s.channels;
  r.samples = s.samples;
  r.grid_rows = s.grid_rows;
  r.grid_cols = s.grid_cols;
  r.nchunks = s.nchunks;
  r.lists_per_frame = s.lists_per_frame;
  r.entries_per_frame = s.entries_per_frame;
  r.coil_group = s.coil_group;
  r.coil_parts = s.coil_parts;
  r.wait_limit = s.wait_fault ? s.wait_fault : kWaitLimit;
  r.wait_beyond = s.wait_fault ? (1 << 30) : 0;
  r.out_cols = s.out_cols;
  r.cpitch = s.cpitch;
  r.plan = s.plan_cols;
  r.col_shift = s.kb ? s.out_cols / 2 : 0;
  r.first_of_two = s.first_of_two;
  RowsLauncher rows_launch;
  if (!rows_launch.setup(s)) return KSJ_GPU_ERROR_CUDA;

  ColsArgs c{};
  c.tw_rows = tw_rows;
  c.inv_dr = inv_dr;
  c.inv_dc = inv_dc;
  c.pos_rows = pos_rows;
  c.flags = flags;
  c.frames = s.frames;
  c.channels = s.channels;
  c.grid_rows = s.grid_rows;
  c.out_rows = s.out_rows;
  c.out_cols = s.out_cols;
  c.kb = s.kb ? 1 : 0;
  c.row_shift = s.kb ? s.out_rows / 2 : 0;
  c.column_block = s.column_block;
  c.col_group = s.col_group;
  c.groups = column_groups(s);
  c.plan = s.plan_rows;
  const bool coil_major = d->output == KSJ_GPU_OUTPUT_COIL_MAJOR;
  c.output = d->output == KSJ_GPU_OUTPUT_RSS ? KSJ_GPU_OUTPUT_RSS : KSJ_GPU_OUTPUT_COIL_LAST;
  c.out = coil_major ? static_cast<void*>(ws + l.coil_last) : d_out;
  c.out_pitch = s.channels;
  ColsPass cols_pass;
  if (!cols_pass.setup(s, inter, &c)) return KSJ_GPU_ERROR_CUDA;

  // frames in passes sized so one pass's row-transformed grid stays in L2
  const int pixels = s.out_rows * s.out_cols;
  bool alt_used = false;
  if (io != nullptr && s.frames > s.frames_per_pass &&
      (cudaEventRecord(io->ready, stream) != cudaSuccess || cudaStreamWaitEvent(io->alt, io->ready, 0) != cudaSuccess))
    return KSJ_GPU_ERROR_CUDA;
  auto run_pass = [&](int f0, int pass) {
    const int nf = std::min(s.frames_per_pass, s.frames - f0);
    cudaStream_t ps = stream;
    if (io != nullptr) {
      if (pass & 1) {
        ps = io->alt;
        alt_used = true;
      }
      if (io->copy != nullptr) {
        if (cudaStreamWaitEvent(ps, io->in[pass], 0) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
        KSJ_TRY(to_coil_last(f0, nf, ps));
      }
    }
    r.frame0 = f0;
    c.frame0 = f0;
    KSJ_TRY(rows_launch.launch(r, s.grid_rows, (s.channels + s.coil_group - 1) / s.coil_group, nf, ps));
    KSJ_TRY(cols_pass.launch(c, nf, ps, "k_cols"));
    if (coil_major) {
      // [frame][pixel][channel] -> [frame][channel][pixel], this pass's frames
      const size_t fe = static_cast<size_t>(pixels) * s.channels;
      const dim3 tg((s.channels + 31) / 32, (pixels + 31) / 32, nf);
      LaunchScope scope("k_images_coil_major", ps);
      k_transpose<unsigned long long><<<tg, dim3(32, 8), 0, ps>>>(
          reinterpret_cast<const unsigned long long*>(ws + l.coil_last) + f0 * fe,
          static_cast<unsigned long long*>(d_out) + f0 * fe, pixels, s.channels);
      KSJ_TRY(check_launch());
    }
    if (io != nullptr && io->copy != nullptr) {
      const size_t off = static_cast<size_t>(f0) * io->out_frame_bytes;
      if (cudaEventRecord(io->done[pass], ps) != cudaSuccess ||
          cudaStreamWaitEvent(io->copy, io->done[pass], 0) != cudaSuccess ||
          cudaMemcpyAsync(static_cast<unsigned char*>(io->h_out) + off, static_cast<unsigned char*>(d_out) + off,
                          static_cast<size_t>(nf) * io->out_frame_bytes, cudaMemcpyDeviceToHost, io->copy) !=
              cudaSuccess)
        return KSJ_GPU_ERROR_CUDA;
    }
    return check_launch();
  };
  ksj_gpu_status result = KSJ_GPU_OK;
  for (int f0 = 0, pass = 0; f0 < s.frames && result == KSJ_GPU_OK; f0 += s.frames_per_pass, ++pass)
    result = run_pass(f0, pass);
  // the second compute stream joins back before the call's stream goes on, after a failure too
  if (alt_used &&
      (cudaEventRecord(io->alt_done, io->alt) != cudaSuccess || cudaStreamWaitEvent(stream, io->alt_done, 0) != cudaSuccess))
    return KSJ_GPU_ERROR_CUDA;
  return result;
}

// ------------------------------------------------- Pipe-Menon density weights
//
// w <- w / ((w * phi) sampled back through phi), phi the Kaiser-Bessel
// gridding kernel, 10 iterations by default, in double precision (Pipe and
// Menon, MRM 1999; grid-based form).  The binning lists of the gridding path
// give, per (row, 16-column chunk), the samples touching it in increasing
// order, so each grid cell sums its samples in that order: deterministic.

__device__ __forceinline__ double kb_weight64(double d, int width, double beta, double inv_i0_beta) {
  const double t = 2.0 * d / static_cast<double>(width);
  if (t * t > 1.0) return 0.0;
  return cyl_bessel_i0(beta * sqrt(1.0 - t * t)) * inv_i0_beta;
}

// The Kaiser-Bessel weight of tap j, at distance d = j - W/2 + 1 - f of a coordinate
// with the fraction f in [0, 1), as a polynomial in z = 2 f - 1: I0(beta sqrt(1 - (2 d /
// W)^2)) / I0(beta) is an entire function of d, so its Chebyshev coefficients fall
// off factorially.  The host interpolates each tap at kKbNodes Chebyshev points (values
// from the Maclaurin series sum (beta^2 s / 4)^k / (k!)^2, all terms positive) and
// drops the terms below 2^-52 of the peak.  Tap W - 1 - j is tap j mirrored in z, so
// its even and odd parts give both: 16 to 20 multiply-adds for two weights, where the
// square root, the division by W and the Bessel function's two ranges took about
// 70 FP64 instructions for one.  The largest error over the widths and oversamplings
// of 1 to 4 is 7e-16 of the peak.  A beta that kKbNodes points do not resolve (above 28 to
// 40, where the default for width 8 ends at 23) leaves `half` 0 and the weights to
// kb_weight64.
constexpr int kKbNodes = 32;
struct KbTaps {
  int half;               // even and odd coefficients kept of every tap, or 0
  double c[4][kKbNodes];  // monomial coefficients in z of tap j < W / 2
};

KbTaps kb_taps(int width, double beta) {
  constexpr double kPi = 3.14159265358979323846;
  double series[64];  // (beta^2 / 4)^k / (k!)^2 over I0(beta)
  int terms = 0;
  {
    long double term[64] = {1.0L}, top = 1.0L;
    while (++terms < 63 && term[terms - 1] > 1e-19L * top) {
      term[terms] = term[terms - 1] * (0.25L * beta * beta) / (static_cast<long double>(terms) * terms);
      top += term[terms];
    }
    if (terms == 63) return KbTaps{};
    for (int k = 0; k < terms; ++k) series[k] = static_cast<double>(term[k] / top);
  }
  // Horner's rule with the rounding errors carried along (Graillat, Langlois, Louvet 2005)
  auto i0 = [&](double s) {
    double sum = series[terms - 1], carry = 0.0;
    for (int k = terms - 2; k >= 0; --k) {
      const double product = sum * s, next = product + series[k], part = next - product;
      carry = std::fma(carry, s, std::fma(sum, s, -product) + ((product - (next - part)) + (series[k] - part)));
      sum = next;
    }
    return sum + carry;
  };
  double cosine[4 * kKbNodes];
  for (int i = 0; i <= kKbNodes / 2; ++i) {  // angles up to pi / 4, then by symmetry
    cosine[i] = std::cos(kPi * i / (2 * kKbNodes));
    cosine[kKbNodes - i] = std::sin(kPi * i / (2 * kKbNodes));
  }
  for (int i = 1; i <= kKbNodes; ++i) cosine[kKbNodes + i] = -cosine[kKbNodes - i];
  for (int i = 1; i < 2 * kKbNodes; ++i) cosine[2 * kKbNodes + i] = cosine[2 * kKbNodes - i];
  KbTaps p{};
  for (int tap = 0; tap < width / 2; ++tap) {
    double value[kKbNodes], cheb[kKbNodes];
    for (int j = 0; j < kKbNodes; ++j) {
      const double t = (2.0 * (tap - width / 2 + 1) - 1.0 - cosine[2 * j + 1]) / width;  // 2 d / W
      value[j] = i0(std::max(std::fma(-t, t, 1.0), 0.0));
    }
    int degree = 0;
    for (int k = 0; k < kKbNodes; ++k) {
      double sum = 0.0, carry = 0.0;
      for (int j = 0; j < kKbNodes; ++j) {
        const double product = value[j] * cosine[(k * (2 * j + 1)) % (4 * kKbNodes)], next = sum + product,
                     part = next - sum;
        carry += (sum - (next - part)) + (product - part);
        sum = next;
      }
      cheb[k] = (k == 0 ? 1.0 : 2.0) / kKbNodes * (sum + carry);
      if (std::fabs(cheb[k]) > 0x1p-52) degree = k;
    }
    if (degree > kKbNodes - 3) return KbTaps{};
    p.half = std::max(p.half, degree / 2 + 1);
    // T_k in monomials, by its recurrence
    double t0[kKbNodes] = {1.0}, t1[kKbNodes] = {0.0, 1.0};
    p.c[tap][0] = cheb[0];
    for (int k = 1; k <= degree; ++k) {
      for (int i = 0; i <= k; ++i) p.c[tap][i] += cheb[k] * t1[i];
      double t2[kKbNodes] = {};
      for (int i = 0; i < kKbNodes; ++i) t2[i] = (i > 0 ? 2.0 * t1[i - 1] : 0.0) - t0[i];
      std::copy(t1, t1 + kKbNodes, t0);
      std::copy(t2, t2 + kKbNodes, t1);
    }
  }
  return p;
}

// The W weights of each of two coordinates with fractions f.
template <int W>
__device__ __forceinline__ void kb_weights64(const KbTaps& p, const double (&f)[2], double (&out)[2][W]) {
  double x[2], z[2], even[2][W / 2], odd[2][W / 2];
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    z[i] = fma(2.0, f[i], -1.0);
    x[i] = z[i] * z[i];
#pragma unroll
    for (int j = 0; j < W / 2; ++j) even[i][j] = odd[i][j] = 0.0;
  }
  for (int k = p.half - 1; k >= 0; --k) {
#pragma unroll
    for (int j = 0; j < W / 2; ++j) {
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        even[i][j] = fma(even[i][j], x[i], p.c[j][2 * k]);
        odd[i][j] = fma(odd[i][j], x[i], p.c[j][2 * k + 1]);
      }
    }
  }
#pragma unroll
  for (int i = 0; i < 2; ++i) {
#pragma unroll
    for (int j = 0; j < W / 2; ++j) {
      out[i][j] = fma(z[i], odd[i][j], even[i][j]);
      out[i][W - 1 - j] = fma(-z[i], odd[i][j], even[i][j]);
    }
  }
}

// Per sample: the double-precision tap weights and w = 1.  The coordinate
// u = k g / (2 pi) is formed in double (an exact product, one rounded
// division); a sample the gridding checks rejected gets w = 0.
template <int W>
__global__ void __launch_bounds__(256) k_pm_prepare(const float* traj, PmRecord<W>* pm, double* w, size_t total,
                                                    int grid_rows, int grid_cols, const __grid_constant__ KbTaps taps,
                                                    double beta, double inv_i0_beta,
                                                    int require_nyquist) {
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const float2 k = __ldg(reinterpret_cast<const float2*>(traj) + idx);
  bool ok = isfinite(k.x) && isfinite(k.y);
  if (ok && require_nyquist) ok = k.x >= -kPiF && k.x <= kPiF && k.y >= -kPiF && k.y <= kPiF;
  if (ok && !require_nyquist) ok = fabsf(k.x) < 1.0e4f && fabsf(k.y) < 1.0e4f;
  PmRecord<W> r;
  constexpr double kTwoPiD = 6.283185307179586476925286766559;
  if (ok) {
    const double ur = static_cast<double>(k.x) * grid_rows / kTwoPiD;
    const double uc = static_cast<double>(k.y) * grid_cols / kTwoPiD;
    const int tr = static_cast<int>(floor(ur)) - W / 2 + 1;
    const int tc = static_cast<int>(floor(uc)) - W / 2 + 1;
    r.r0 = wrap_index(tr, grid_rows);
    r.c0 = wrap_index(tc, grid_cols);
    if (taps.half > 0) {
      const double f[2] = {ur - floor(ur), uc - floor(uc)};
      double v[2][W];
      kb_weights64<W>(taps, f, v);
#pragma unroll
      for (int j = 0; j < W; ++j) {
        r.wr[j] = v[0][j];
        r.wc[j] = v[1][j];
      }
    } else {
      for (int j = 0; j < W; ++j) {
        r.wr[j] = kb_weight64(static_cast<double>(tr + j) - ur, W, beta, inv_i0_beta);
        r.wc[j] = kb_weight64(static_cast<double>(tc + j) - uc, W, beta, inv_i0_beta);
      }
    }
  } else {
    r.r0 = 0;
    r.c0 = 0;
#pragma unroll
    for (int j = 0; j < W; ++j) {
      r.wr[j] = 0.0;
      r.wc[j] = 0.0;
    }
  }
  pm[idx] = r;
  w[idx] = ok ? 1.0 : 0.0;
}

// The grid step with kPmLanes lanes per list (3-D, and the longer lists in 2-D): lane q
// takes the list's entries q, q + kPmLanes, ... in order and, for every column tap of
// an entry that lands in the list's 16-column chunk, adds u * wc[k] (u = w times
// the entry's row, and plane, weights) to its own 16 cells in shared memory; then lane q
// sums cells 4q .. 4q+3 over the list's lanes, each cell in a fixed order
// (starting at lane q).  Every FP64 operation a lane issues is one a cell
// needs; with a lane per column instead, 12 of every 16 lanes multiplied by taps
// outside their column.  Lists are kPmLanes consecutive lanes of one warp, so a
// warp barrier orders the two phases.
constexpr int kPmLanes = 4;
constexpr int kPmThreads = 256;
constexpr int kPmCellsPerLane = kChunk / kPmLanes;
static_assert(kChunk == 16 && (kPmLanes & (kPmLanes - 1)) == 0 && 32 % kPmLanes == 0, "lanes of a list");

// Lane q of a list (its lane 0 is thread `lane0`): cells 4q .. 4q+3 summed
// over the list's lanes, starting at lane q, written to row[lo + t] inside
// the grid.
__device__ __forceinline__ void pm_reduce_store(const double* cells, int lane0, int q, double* row, int lo,
                                                int grid_cols) {
#pragma unroll
  for (int i = 0; i < kPmCellsPerLane; ++i) {
    const int t = q * kPmCellsPerLane + i;
    const double* c = cells + t * kPmThreads + lane0;
    double acc = c[q];
#pragma unroll
    for (int j = 1; j < kPmLanes; ++j) acc += c[(q + j) & (kPmLanes - 1)];
    if (lo + t < grid_cols) row[lo + t] = acc;
  }
}

// The lists of a call ordered by length, longest first (bins of up to
// kPmBins - 1 entries, longer ones in the last; any order within a bin): a warp of the
// grid step issues every FP64 instruction for all its lanes, so lists of one
// warp should end together.  bins: kPmBins counts, then kPmBins cursors, cleared before.
constexpr int kPmBins = 256;
constexpr int kPmOrderThreads = 1024;

__device__ __forceinline__ uint32_t list_length(const uint32_t* offsets, size_t list, int lists_per_frame) {
  const uint32_t* off = offsets + list + list / lists_per_frame;  // lists + 1 offsets per frame
  return off[1] - off[0];
}

__global__ void __launch_bounds__(kPmOrderThreads) k_pm_bins(const uint32_t* offsets, size_t lists, int lists_per_frame,
                                                             uint32_t* bins) {
  __shared__ uint32_t count[kPmBins];
  for (int i = threadIdx.x; i < kPmBins; i += kPmOrderThreads) count[i] = 0;
  __syncthreads();
  const size_t list = static_cast<size_t>(blockIdx.x) * kPmOrderThreads + threadIdx.x;
  if (list < lists) atomicAdd(count + min(list_length(offsets, list, lists_per_frame), kPmBins - 1u), 1u);
  __syncthreads();
  for (int i = threadIdx.x; i < kPmBins; i += kPmOrderThreads)
    if (count[i] != 0) atomicAdd(bins + i, count[i]);
}

__global__ void __launch_bounds__(kPmOrderThreads) k_pm_order(const uint32_t* offsets, size_t lists,
                                                              int lists_per_frame, uint32_t* bins, uint32_t* order) {
  __shared__ uint32_t count[kPmBins], start[kPmBins];
  for (int i = threadIdx.x; i < kPmBins; i += kPmOrderThreads) {
    count[i] = 0;
    uint32_t before = 0;  // lists of longer bins
    for (int j = i + 1; j < kPmBins; ++j) before += __ldg(bins + j);
    start[i] = before;
  }
  __syncthreads();
  const size_t list = static_cast<size_t>(blockIdx.x) * kPmOrderThreads + threadIdx.x;
  uint32_t bin = 0, rank = 0;
  if (list < lists) {
    bin = min(list_length(offsets, list, lists_per_frame), kPmBins - 1u);
    rank = atomicAdd(count + bin, 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < kPmBins; i += kPmOrderThreads)
    if (count[i] != 0) start[i] += atomicAdd(bins + kPmBins + i, count[i]);
  __syncthreads();
  if (list < lists) order[start[bin] + rank] = static_cast<uint32_t>(list);
}

// The 2-D grid step: one lane per list of up to kPmAlone entries, kPmLanes lanes for a
// longer one (which come first in `order`), each adding u * wc[k] (u = w times
// the entry's row weight) for the column taps that land in the list's chunk to its
// own 16 cells in shared memory; four lanes' cells are then added in a fixed
// order.  A half-warp writes a list's cells.  The entries are streamed (16 + 8 W
// bytes, written in list order once a call), two requested ahead and the next
// one's sample weight with them (one ahead, its weight fetched when it is used, 144 us an iteration, now 128).
//
// Bound by the FP64 pipe (two lanes per clock and SM): 5 operations an entry and,
// for the few lists of four lanes, 48 to add them.  Four lanes for every list, in grid
// order, spent 4 of 5 issues on idle lanes and as many again on adding the lanes:
// 275 us an iteration on 96 frames x 13056 samples, now 128.
constexpr uint32_t kPmAlone = 32;
constexpr int kPmPitch = kChunk + 1;  // cells of one thread, an odd number of doubles apart

template <int W>
__global__ void __launch_bounds__(kPmThreads, W <= 4 ? 4 : 2) k_pm_grid(const uint32_t* offsets, const PmEntry<W>* entries,
                                                        const uint32_t* order, const uint32_t* bins, const double* w,
                                                        double* grid, size_t lists, int samples, int grid_rows,
                                                        int grid_cols, int nchunks, int lists_per_frame,
                                                        size_t entries_per_frame, int first_of_two) {
  __shared__ double cells[kPmThreads * kPmPitch];
  __shared__ uint32_t many_shared;
  chain_begin();
  // lists of more than kPmAlone entries
  if (threadIdx.x < 32) {
    uint32_t n = 0;
    for (int i = kPmAlone + 1 + threadIdx.x; i < kPmBins; i += 32) n += __ldg(bins + i);
    n = __reduce_add_sync(0xffffffffu, n);
    if (threadIdx.x == 0) many_shared = n;
  }
  __syncthreads();
  const size_t many = many_shared;
  const size_t many_threads = (many * kPmLanes + kPmThreads - 1) / kPmThreads * kPmThreads;
  const size_t thread = static_cast<size_t>(blockIdx.x) * kPmThreads + threadIdx.x;
  const bool split = thread < many_threads;  // the same for a whole block
  const size_t rank = split ? thread / kPmLanes : many + thread - many_threads;
  const int q = split ? threadIdx.x & (kPmLanes - 1) : 0;
  const bool active = rank < (split ? many : lists);
  if (!__syncthreads_or(active)) return;
  double* cell = cells + threadIdx.x * kPmPitch;
#pragma unroll
  for (int t = 0; t < kChunk; ++t) cell[t] = 0.0;
  double* out = nullptr;  // the list's first cell in the grid
  int width = 0;
  if (active) {
    const uint32_t list = __ldg(order + rank);
    const int f = static_cast<int>(list / static_cast<uint32_t>(lists_per_frame));
    const int l = static_cast<int>(list - static_cast<uint32_t>(f) * lists_per_frame);
    const int row = l / nchunks, lo = (l - row * nchunks) * kChunk;
    out = grid + (static_cast<size_t>(f) * grid_rows + row) * grid_cols + lo;
    width = min(kChunk, grid_cols - lo);
    const uint32_t* off = offsets + static_cast<size_t>(f) * (lists_per_frame + 1);
    const PmEntry<W>* ent = entries + static_cast<size_t>(f) * entries_per_frame;
    const double* wf = w + static_cast<size_t>(f) * samples;
    // one chunk, or the first of two, may see both ends of a wrapped stencil
    const int wrap = nchunks == 1 || first_of_two ? grid_cols : 0;
    const uint32_t end = off[l + 1], step = split ? kPmLanes : 1;
    auto load = [&](uint32_t e) {
      PmEntry<W> r;
      const float4* src = reinterpret_cast<const float4*>(ent + e);
      float4* dst = reinterpret_cast<float4*>(&r);
#pragma unroll
      for (int v = 0; v < static_cast<int>(sizeof(PmEntry<W>) / 16); ++v) dst[v] = __ldg(src + v);
      return r;
    };
    uint32_t e = off[l] + q;
    if (e < end) {
      PmEntry<W> next = load(e), after = next;
      double weight = wf[next.sample];
      if (e + step < end) after = load(e + step);
      for (; e < end; e += step) {
        const PmEntry<W> r = next;
        const double u = weight * r.wr;
        next = after;
        if (e + step < end) weight = wf[next.sample];
        if (e + 2 * step < end) after = load(e + 2 * step);
#pragma unroll
        for (int k = 0; k < W; ++k) {
          int t = r.t0 + k;
          if (wrap != 0 && t >= wrap) t -= wrap;
          if (static_cast<uint32_t>(t) < kChunk) cell[t] = fma(u, r.wc[k], cell[t]);
        }
      }
    }
  }
  __syncwarp();
  const int lane = threadIdx.x & 31;
  if (split) {
    // lane q of a list: cells 4q .. 4q + 3 over its lanes, starting at lane q, left in lane 0's
    double sum[kPmCellsPerLane];
#pragma unroll
    for (int i = 0; i < kPmCellsPerLane; ++i) {
      const double* c = cells + (threadIdx.x - q) * kPmPitch + q * kPmCellsPerLane + i;
      sum[i] = c[q * kPmPitch];
#pragma unroll
      for (int j = 1; j < kPmLanes; ++j) sum[i] += c[((q + j) & (kPmLanes - 1)) * kPmPitch];
    }
    __syncwarp();
#pragma unroll
    for (int i = 0; i < kPmCellsPerLane; ++i) cells[(threadIdx.x - q) * kPmPitch + q * kPmCellsPerLane + i] = sum[i];
    __syncwarp();
  }
  // two lists at a time, a half-warp each
  for (int i = (lane >> 4) * (split ? kPmLanes : 1); i < 32; i += 2 * (split ? kPmLanes : 1)) {
    double* to = reinterpret_cast<double*>(__shfl_sync(0xffffffffu, reinterpret_cast<unsigned long long>(out), i));
    const int n = __shfl_sync(0xffffffffu, width, i);
    if ((lane & 15) < n) to[lane & 15] = cells[(threadIdx.x - lane + i) * kPmPitch + (lane & 15)];
  }
}

// Per sample: d = the grid read back through the sample's taps (row-major),
// w = w / d (0 when d is not positive); the last iteration also writes the
// float weights.
template <int W>
__global__ void __launch_bounds__(256) k_pm_update(const PmRecord<W>* pm, const double* grid, double* w, float* out,
                                                   size_t total, int samples, int grid_rows, int grid_cols) {
  chain_begin();
  const size_t idx = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (idx >= total) return;
  const size_t f = idx / samples;
  const PmRecord<W> r = pm[idx];
  const double* g = grid + f * grid_rows * grid_cols;
  // separable taps: d = sum_a wr[a] (sum_b wc[b] grid[a][b]), W + 1 FP64
  // operations per row of taps instead of 2W
  int cols[W];
#pragma unroll
  for (int b = 0; b < W; ++b) {
    cols[b] = r.c0 + b;
    if (cols[b] >= grid_cols) cols[b] -= grid_cols;
  }
  double d = 0.0;
#pragma unroll
  for (int a = 0; a < W; ++a) {
    int rr = r.r0 + a;
    if (rr >= grid_rows) rr -= grid_rows;
    const double* line = g + static_cast<size_t>(rr) * grid_cols;
    double t = 0.0;
#pragma unroll
    for (int b = 0; b < W; ++b) t = fma(line[cols[b]], r.wc[b], t);
    d = fma(r.wr[a], t, d);
  }
  const double nw = d > 0.0 ? w[idx] / d : 0.0;
  w[idx] = nw;
  if (out != nullptr) out[idx] = static_cast<float>(nw);
}

struct PmLayout {
  size_t flags, records, counts, totals, offsets, entries, bins, order, pm, w, grid, total;
};

// Frames are independent, so a call takes them in passes through one workspace: as many at
// once as keep their entries (48 bytes for a width of 4, up to 2 or 3 W of them a sample) and
// their grids within kPmPassBytes each, and at least one.
constexpr size_t kPmPassBytes = size_t{4} << 30;

// The workspace of a call, which every pass of it uses as it is: the regions hold the most
// samples and frames of any pass, of this call and of every smaller one.
ksj_gpu_status make_pm_layout(const ksj_gpu_gridding_desc* desc, PmLayout* layout, uint32_t* pass_frames) {
  Shape s{};
  ksj_gpu_gridding_desc d = *desc;
  ksj_gpu_status st = make_shape(&d, nullptr, &s);
  if (st != KSJ_GPU_OK) return st;
  const size_t grid_bytes = static_cast<size_t>(s.grid_rows) * s.grid_cols * sizeof(double);
  d.frames = static_cast<uint32_t>(std::min<size_t>(d.frames, kPmPassBytes / grid_bytes));
  st = make_shape(&d, nullptr, &s);
  if (st != KSJ_GPU_OK) return st;
  const size_t entry = 16 + 8 * static_cast<size_t>(s.width), m = static_cast<size_t>(s.samples);
  const size_t per_sample = s.entries_per_frame / m;
  const size_t held = std::max(kPmPassBytes / (per_sample * entry), m);  // samples of one pass, at most
  const size_t fm = std::min(s.frames * m, held);
  *pass_frames = static_cast<uint32_t>(fm / m);
  PmLayout& l = *layout;
  l = PmLayout{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t nl = static_cast<size_t>(s.frames) * s.lists_per_frame;
  l.flags = take(kFlagBytes);
  l.records = take(fm * record_bytes(s.width));
  l.counts = take(s.bin_capacity * s.lists_per_frame * 4);
  l.totals = take(nl * 4);
  l.offsets = take((nl + s.frames) * 4);
  l.entries = take(fm * per_sample * entry);
  l.bins = take(2 * kPmBins * 4);
  l.order = take(nl * 4);
  l.pm = take(fm * (8 + 16 * static_cast<size_t>(s.width)));
  l.w = take(fm * sizeof(double));
  l.grid = take(s.frames * grid_bytes);
  l.total = off;
  return KSJ_GPU_OK;
}

// The flags must already be cleared.
template <int W>
ksj_gpu_status launch_pipe_menon(const Shape& s, const PmLayout& l, const ksj_gpu_gridding_desc* d,
                                 uint32_t iterations, const float* d_traj, float* d_dcf, unsigned char* ws,
                                 cudaStream_t stream) {
  static_assert(sizeof(PmRecord<W>) == 8 + 16 * W, "PmRecord layout");
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + l.flags);
  ksj_gpu_gridding_desc dd = *d;
  dd.dcf_mode = KSJ_GPU_DCF_NONE;
  static_assert(sizeof(PmEntry<W>) == 16 + 8 * W, "PmEntry layout");
  const size_t fm = static_cast<size_t>(s.frames) * s.samples;
  PmRecord<W>* pm = reinterpret_cast<PmRecord<W>*>(ws + l.pm);
  double* w = reinterpret_cast<double*>(ws + l.w);
  double* grid = reinterpret_cast<double*>(ws + l.grid);
  {
    LaunchScope scope("k_pm_prepare", stream);
    k_pm_prepare<W><<<static_cast<unsigned>((fm + 255) / 256), 256, 0, stream>>>(
        d_traj, pm, w, fm, s.grid_rows, s.grid_cols, kb_taps(W, s.beta), s.beta,
        1.0 / std::cyl_bessel_i(0.0, static_cast<double>(s.beta)), d->require_nyquist);
    KSJ_TRY(check_launch());
  }
  const ksj_gpu_status st =
      build_lists<W>(s, &dd, d_traj, nullptr, flags, ws + l.records, reinterpret_cast<uint32_t*>(ws + l.counts),
                     reinterpret_cast<uint32_t*>(ws + l.totals), reinterpret_cast<uint32_t*>(ws + l.offsets),
                     ws + l.entries, pm, stream);
  if (st != KSJ_GPU_OK) return st;
  const size_t lists = static_cast<size_t>(s.frames) * s.lists_per_frame;
  const uint32_t* offsets = reinterpret_cast<const uint32_t*>(ws + l.offsets);
  uint32_t* bins = reinterpret_cast<uint32_t*>(ws + l.bins);
  uint32_t* order = reinterpret_cast<uint32_t*>(ws + l.order);
  if (cudaMemsetAsync(bins, 0, 2 * kPmBins * 4, stream) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  const unsigned order_blocks = static_cast<unsigned>((lists + kPmOrderThreads - 1) / kPmOrderThreads);
  {
    LaunchScope scope("k_pm_bins", stream);
    k_pm_bins<<<order_blocks, kPmOrderThreads, 0, stream>>>(offsets, lists, s.lists_per_frame, bins);
    KSJ_TRY(check_launch());
  }
  {
    LaunchScope scope("k_pm_order", stream);
    k_pm_order<<<order_blocks, kPmOrderThreads, 0, stream>>>(offsets, lists, s.lists_per_frame, bins, order);
    KSJ_TRY(check_launch());
  }
  for (uint32_t it = 0; it < iterations; ++it) {
    {
      LaunchScope scope("k_pm_grid", stream);
      KSJ_TRY(launch_chained(k_pm_grid<W>, dim3(static_cast<unsigned>((lists * kPmLanes + kPmThreads - 1) / kPmThreads + 1)),
                     dim3(kPmThreads), 0, stream,
          offsets, reinterpret_cast<const PmEntry<W>*>(ws + l.entries), static_cast<const uint32_t*>(order),
                     static_cast<const uint32_t*>(bins), static_cast<const double*>(w), grid, lists, s.samples,
          s.grid_rows, s.grid_cols, s.nchunks, s.lists_per_frame, s.entries_per_frame,
                     s.first_of_two));
    }
    LaunchScope scope("k_pm_update", stream);
    KSJ_TRY(launch_chained(k_pm_update<W>, dim3(static_cast<unsigned>((fm + 255) / 256)), dim3(256), 0, stream,
                   static_cast<const PmRecord<W>*>(pm), static_cast<const double*>(grid), w,
                   it + 1 == iterations ? d_dcf : nullptr, fm, s.samples, s.grid_rows, s.grid_cols));
  }
  return check_launch();
}

// ------------------------------------------------------------ 3-D gridding
//
// A g^3 grid is gridded as g z-planes of the 2-D row/column machinery: the
// binning lists are (plane, row, 16-column chunk); an entry's row weight is
// the sample's y weight times its z weight for that plane; every plane reads
// the one coil-last sample array.  After the per-plane row and column passes
// (y and x transformed, cropped, deapodised) the intermediate
// [plane][pixel][coil] takes a third pass along z, which is the column pass
// again with planes as rows and pixels as columns.

struct Prepare3Args {
  const float* traj;  // [M][3] (k_z, k_y, k_x)
  const float* dcf;
  uint32_t dcf_mode;
  unsigned char* records;
  uint32_t* counts;  // [block][plane]: samples of the block on the plane
  uint32_t* flags;
  int samples, grid, bin_span;
  float beta, two_over_w, inv_i0_beta, phase;
};

// One sample's record; its first tap plane.
template <int W>
__device__ __forceinline__ int prepare_sample3(const Prepare3Args& a, int idx) {
  const float kz = __ldg(a.traj + 3 * static_cast<size_t>(idx));
  const float ky = __ldg(a.traj + 3 * static_cast<size_t>(idx) + 1);
  const float kx = __ldg(a.traj + 3 * static_cast<size_t>(idx) + 2);
  bool ok = isfinite(kz) && isfinite(ky) && isfinite(kx) && fabsf(kz) < 1.0e4f && fabsf(ky) < 1.0e4f &&
            fabsf(kx) < 1.0e4f;
  float w = 1.0f;
  if (a.dcf_mode == KSJ_GPU_DCF_ANALYTIC_RAMP) {
    w = fmaf(kz, kz, fmaf(ky, ky, kx * kx));  // 3-D radial density ~ 1 / |k|^2
  } else if (a.dcf_mode == KSJ_GPU_DCF_EXTERNAL) {
    w = __ldg(a.dcf + idx);
    if (!(isfinite(w) && w >= 0.0f)) {
      atomicOr(a.flags, KSJ_GPU_FLAG_BAD_DCF);
      w = 0.0f;
    }
  }
  SampleRecord3<W> rec;
  rec.pad = 0;
  if (!ok) {
    atomicOr(a.flags, KSJ_GPU_FLAG_BAD_TRAJECTORY);
    rec.z0 = rec.r0 = rec.c0 = 0;
    rec.scale = make_float2(0.0f, 0.0f);
#pragma unroll
    for (int j = 0; j < W; ++j) rec.wz[j] = rec.wr[j] = rec.wc[j] = 0.0f;
  } else {
    const float gf = static_cast<float>(a.grid);
    const dfloat uz = grid_coordinate(kz, gf), uy = grid_coordinate(ky, gf), ux = grid_coordinate(kx, gf);
    float f;
    const int sz = dfloor(uz, &f) - W / 2 + 1;
    const int sy = dfloor(uy, &f) - W / 2 + 1;
    const int sx = dfloor(ux, &f) - W / 2 + 1;
    rec.z0 = wrap_index(sz, a.grid);
    rec.r0 = wrap_index(sy, a.grid);
    rec.c0 = wrap_index(sx, a.grid);
#pragma unroll
    for (int j = 0; j < W; ++j) {
      rec.wz[j] = kb_weight(__fsub_rn(__fsub_rn(static_cast<float>(sz + j), uz.hi), uz.lo), a.two_over_w, a.beta,
                            a.inv_i0_beta);
      rec.wr[j] = kb_weight(__fsub_rn(__fsub_rn(static_cast<float>(sy + j), uy.hi), uy.lo), a.two_over_w, a.beta,
                            a.inv_i0_beta);
      rec.wc[j] = kb_weight(__fsub_rn(__fsub_rn(static_cast<float>(sx + j), ux.hi), ux.lo), a.two_over_w, a.beta,
                            a.inv_i0_beta);
    }
    rec.scale = cscale(exp_i_dot3(kz, a.phase, ky, a.phase, kx, a.phase), w);
  }
  reinterpret_cast<SampleRecord3<W>*>(a.records)[idx] = rec;
  return rec.z0;
}

// Binning in 3-D, in sample order: a sample is first placed in the lists of its W
// planes (k_prepare3 counts, k_plane_place), then a plane's samples, in that
// order, in the plane's row and chunk lists as a frame's (k_count3, k_place3,
// kPlaneBlocks blocks a plane).  Appending to the (plane, row, chunk) lists with
// atomics and sorting them took 15 ms of a call on 10.24 M samples, 384^3 (the
// centre's lists hold up to 1.5e5 entries), these take 5.7.
constexpr int kPlaneBlocks = 16;

template <int W>
__global__ void __launch_bounds__(kBinThreads) k_prepare3(Prepare3Args a) {
  __shared__ uint32_t counts[kMaxGrid];
  for (int p = threadIdx.x; p < a.grid; p += kBinThreads) counts[p] = 0;
  __syncthreads();
  const int s0 = blockIdx.x * a.bin_span, s1 = min(s0 + a.bin_span, a.samples);
  for (int base = s0; base < s1; base += kBinThreads) {
    const int sample = base + threadIdx.x;
    const int one[2] = {0, 0};  // a plane is a row of one list
    if (sample < s1) count_lists<W>(counts, prepare_sample3<W>(a, sample), one, 1, a.grid);
  }
  __syncthreads();
  for (int p = threadIdx.x; p < a.grid; p += kBinThreads) a.counts[blockIdx.x * a.grid + p] = counts[p];
}

// The samples of every plane, in order.  starts: [block][plane].
template <int W>
__global__ void __launch_bounds__(kBinThreads) k_plane_place(const unsigned char* records, const uint32_t* offsets,
                                                             const uint32_t* starts, uint32_t* plane_samples,
                                                             int samples, int grid, int bin_span) {
  __shared__ uint32_t at[kMaxGrid];
  for (int p = threadIdx.x; p < grid; p += kBinThreads)
    at[p] = __ldg(offsets + p) + __ldg(starts + blockIdx.x * grid + p);
  const int s0 = blockIdx.x * bin_span, s1 = min(s0 + bin_span, samples);
  for (int base = s0; base < s1; base += kBinThreads) {
    const int sample = base + threadIdx.x;
    const int z0 = sample < s1 ? reinterpret_cast<const SampleRecord3<W>*>(records)[sample].z0 : -1;
    const int one[2] = {0, 0};
    uint32_t pos[W][2];
    place_turn<W>(at, z0, one, 1, grid, pos);
    if (z0 < 0) continue;
#pragma unroll
    for (int j = 0; j < W; ++j) plane_samples[pos[j][0]] = static_cast<uint32_t>(sample);
  }
}

// Items [*i0, *i1) of plane p's samples that block b of kPlaneBlocks takes, as
// positions in plane_samples.
__device__ __forceinline__ void plane_span(const uint32_t* plane_offsets, int p, int b, uint32_t* i0, uint32_t* i1) {
  const uint32_t begin = __ldg(plane_offsets + p), end = __ldg(plane_offsets + p + 1);
  const uint32_t turns = (end - begin + kBinThreads - 1) / kBinThreads;
  const uint32_t span = (turns + kPlaneBlocks - 1) / kPlaneBlocks * kBinThreads;
  *i0 = min(begin + b * span, end);
  *i1 = min(*i0 + span, end);
}

// One block per (block of a plane's samples, plane): their counts per list.
template <int W, int kLists>
__global__ void __launch_bounds__(kBinThreads) k_count3(const unsigned char* records, const uint32_t* plane_offsets,
                                                        const uint32_t* plane_samples, uint32_t* counts, int grid,
                                                        int nchunks, int lists_per_plane) {
  extern __shared__ uint32_t list_counts[];
  for (int l = threadIdx.x; l < lists_per_plane; l += kBinThreads) list_counts[l] = 0;
  __syncthreads();
  uint32_t i0, i1;
  plane_span(plane_offsets, blockIdx.y, blockIdx.x, &i0, &i1);
  for (uint32_t base = i0; base < i1; base += kBinThreads) {
    const uint32_t i = base + threadIdx.x;
    int r0 = -1, c0 = 0;
    if (i < i1) {
      const SampleRecord3<W>* rec = reinterpret_cast<const SampleRecord3<W>*>(records) + __ldg(plane_samples + i);
      const int4 first = __ldg(reinterpret_cast<const int4*>(rec));  // z0, r0, c0
      r0 = first.y;
      c0 = first.z;
    }
    int chunks[kLists];
    list_chunks<W>(c0, grid, chunks);
    if (r0 >= 0) count_lists<W>(list_counts, r0, chunks, nchunks, grid);
  }
  __syncthreads();
  uint32_t* out = counts + (static_cast<size_t>(blockIdx.y) * kPlaneBlocks + blockIdx.x) * lists_per_plane;
  for (int l = threadIdx.x; l < lists_per_plane; l += kBinThreads) out[l] = list_counts[l];
}

struct Place3Args {
  const unsigned char* records;
  const uint32_t* plane_offsets;
  const uint32_t* plane_samples;
  const uint32_t* offsets;  // [plane][list + 1], absolute
  const uint32_t* starts;   // [plane][block][list]
  unsigned char* expanded;  // entries in their places, or null:
  uint32_t* entries;        // the sample indices alone
  int grid, nchunks, lists_per_plane;
};

// One block per (block of a plane's samples, plane): the entries of its lists.
template <int W, int kLists>
__global__ void __launch_bounds__(kBinThreads) k_place3(Place3Args a) {
  extern __shared__ uint32_t place_smem[];
  uint32_t* at = place_smem;
  const int plane = blockIdx.y;
  uint32_t i0, i1;
  plane_span(a.plane_offsets, plane, blockIdx.x, &i0, &i1);
  if (i0 >= i1) return;
  {
    const uint32_t* off = a.offsets + static_cast<size_t>(plane) * (a.lists_per_plane + 1);
    const uint32_t* st = a.starts + (static_cast<size_t>(plane) * kPlaneBlocks + blockIdx.x) * a.lists_per_plane;
#pragma unroll 8
    for (int l = threadIdx.x; l < a.lists_per_plane; l += kBinThreads) at[l] = __ldg(off + l) + __ldg(st + l);
  }
  for (uint32_t base = i0; base < i1; base += kBinThreads) {
    const uint32_t i = base + threadIdx.x;
    constexpr int kRV = static_cast<int>(sizeof(SampleRecord3<W>) / 16);
    float4 q[kRV];
    uint32_t sample = 0;
    if (i < i1) {
      sample = __ldg(a.plane_samples + i);
      const float4* rp = reinterpret_cast<const float4*>(reinterpret_cast<const SampleRecord3<W>*>(a.records) + sample);
#pragma unroll
      for (int v = 0; v < kRV; ++v) q[v] = __ldg(rp + v);
    }
    const float* w = reinterpret_cast<const float*>(q);
    const int r0 = i < i1 ? __float_as_int(w[1]) : -1, c0 = i < i1 ? __float_as_int(w[2]) : 0;
    int chunks[kLists];
    list_chunks<W>(c0, a.grid, chunks);
    uint32_t pos[W][kLists];
    place_turn<W>(at, r0, chunks, a.nchunks, a.grid, pos);
    if (r0 < 0) continue;
    int tz = plane - __float_as_int(w[0]);
    if (tz < 0) tz += a.grid;
    float wz = 0.0f;
#pragma unroll
    for (int j = 0; j < W; ++j)
      if (j == tz) wz = w[6 + j];
#pragma unroll
    for (int j = 0; j < W; ++j) {
#pragma unroll
      for (int h = 0; h < kLists; ++h) {
        if (!own_list(chunks, h)) continue;
        if (a.expanded != nullptr)
          put_entry<W>(sample, c0, w[6 + W + j] * wz, w + 6 + 2 * W, chunks[h] * kChunk, a.grid,
                       a.expanded + static_cast<size_t>(pos[j][h]) * entry_bytes(W));
        else
          a.entries[pos[j][h]] = sample;
      }
    }
  }
}

// The per-plane scans leave offsets[p][lists] = the plane's total; turn them
// into absolute positions in one entry array (one block: planes <= 512).
__global__ void __launch_bounds__(512) k_plane_bases(uint32_t* offsets, int planes, int lists, uint32_t* bases) {
  __shared__ uint32_t tot[512];
  const int t = threadIdx.x;
  tot[t] = t < planes ? offsets[static_cast<size_t>(t) * (lists + 1) + lists] : 0u;
  __syncthreads();
  if (t == 0) {
    uint32_t run = 0;
    for (int p = 0; p < planes; ++p) {
      const uint32_t v = tot[p];
      tot[p] = run;
      run += v;
    }
  }
  __syncthreads();
  if (t < planes) bases[t] = tot[t];
}

__global__ void __launch_bounds__(256) k_offsets_add(uint32_t* offsets, int planes, int lists, const uint32_t* bases) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<size_t>(planes) * (lists + 1)) return;
  offsets[i] += bases[i / (lists + 1)];
}

// Workspace of the 3-D binning.
struct Lists3 {
  size_t plane_counts, plane_totals, plane_offsets, plane_samples, counts, totals, offsets, bases;
};

template <class Take>
Lists3 take_lists3(const Shape& s, Take&& take) {
  const size_t g = static_cast<size_t>(s.grid_rows), nl = g * s.lists_per_frame;
  Lists3 l{};
  l.plane_counts = take(s.bin_capacity * g * 4);
  l.plane_totals = take(g * 4);
  l.plane_offsets = take((g + 1) * 4);
  l.plane_samples = take(static_cast<size_t>(s.samples) * s.width * 4);
  l.counts = take(nl * kPlaneBlocks * 4);
  l.totals = take(nl * 4);
  l.offsets = take((nl + g) * 4);
  l.bases = take(g * 4);
  return l;
}

struct Layout3 {
  size_t flags, records, expanded, samples_t, inter, inter2, tables, total;
  Lists3 lists;
  size_t entries_total;
};

size_t record3_bytes(int width) {
  switch (width) {
    case 2: return sizeof(SampleRecord3<2>);
    case 4: return sizeof(SampleRecord3<4>);
    case 6: return sizeof(SampleRecord3<6>);
    default: return sizeof(SampleRecord3<8>);
  }
}

// The y pass writes coil images, so it may take a column's coils in parts, each a column of its own
// of few coils (the largest power of two that divides the pitch), where the tile of all
// of them is at least a quarter empty: 20 coils in five parts of 4, eight columns of
// them a tile, leave none of the 32 lines without a coil (kooshball: 3.65 -> 2.52 ms).
int column_parts3(const Shape& s) {
  int q = 1;
  while (q < 32 && s.cpitch % (2 * q) == 0) q *= 2;
  const bool empty = 4 * s.cpitch <= 3 * column_groups(s) * s.col_group;
  return empty && q >= 4 && s.column_pass != 2 ? s.cpitch / q : 1;
}

// s: the 2-D shape of one plane with frames = planes (see make_shape3).
Layout3 make_layout3(const Shape& s) {
  Layout3 l{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t g = static_cast<size_t>(s.grid_rows), n = static_cast<size_t>(s.rows);
  l.entries_total = static_cast<size_t>(s.samples) * s.width * s.width * s.lists_per_row;
  l.flags = take(kFlagBytes);
  l.records = take(static_cast<size_t>(s.samples) * record3_bytes(s.width));
  l.lists = take_lists3(s, take);
  l.expanded = take(l.entries_total * entry_bytes(s.width));
  l.samples_t = take(static_cast<size_t>(s.samples) * s.channels * sizeof(float2));
  l.inter = take(g * g * n * s.cpitch * sizeof(float2));
  l.inter2 = take(g * n * n * s.cpitch * sizeof(float2));
  // twiddles (rows, cols), deapodisation (rows, cols), DIF positions (rows, cols), ones for the pixel axis,
  // the column deapodisation once per part of a column's coils
  l.tables = take(2 * g * sizeof(float2) + 2 * n * sizeof(float) + 2 * n * sizeof(int) + n * n * sizeof(float) +
                  n * column_parts3(s) * sizeof(float));
  l.total = off;
  return l;
}

ksj_gpu_status make_shape3(const ksj_gpu_gridding3_desc* d, const ksj_gpu_gridding_tuning* t, Shape* s) {
  if (d == nullptr || d->struct_size < sizeof(ksj_gpu_gridding3_desc)) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (d->output != KSJ_GPU_OUTPUT_RSS && d->output != KSJ_GPU_OUTPUT_COIL_LAST) return KSJ_GPU_ERROR_UNSUPPORTED;
  if (d->image == 0 || d->grid == 0 || static_cast<uint64_t>(d->image) * d->image > (1u << 24))
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  ksj_gpu_gridding_desc d2{};
  d2.struct_size = sizeof(d2);
  d2.kernel = KSJ_GPU_KERNEL_KAISER_BESSEL;
  d2.image_rows = d2.image_cols = d->image;
  d2.grid_rows = d2.grid_cols = d->grid;
  d2.kernel_width = d->kernel_width;
  d2.kb_beta = d->kb_beta;
  d2.row_origin = d2.col_origin = (static_cast<double>(d->image) - 1.0) / 2.0;
  d2.channels = d->channels;
  d2.samples = d->samples;
  d2.frames = d->grid;  // one frame per z-plane
  d2.dcf_mode = d->dcf_mode;
  d2.output = KSJ_GPU_OUTPUT_COIL_LAST;
  d2.sample_format = d->sample_format;
  const ksj_gpu_status st = make_shape(&d2, t, s);
  if (st != KSJ_GPU_OK) return st;
  s->entries_per_frame = 0;  // absolute offsets into one entry array
  // the plane stage of the binning: one frame, planes for lists
  const int turns = (s->samples + kBinThreads - 1) / kBinThreads;
  const int blocks = std::min(turns, kPlaneStageBlocks);
  s->bin_capacity = blocks;
  s->bin_span = (turns + blocks - 1) / blocks * kBinThreads;
  s->bin_blocks = (s->samples + s->bin_span - 1) / s->bin_span;
  return KSJ_GPU_OK;
}

// The 3-D binning lists: per-sample records, the samples of every plane, the
// (plane, row, chunk) list offsets, and the lists' entries as the row pass reads them
// (`expanded`) or as sample indices alone (`entries`); and the call's tables where
// `tables` names them.  The flags must already be cleared.
template <int W>
ksj_gpu_status build_lists3(const Shape& s, uint32_t dcf_mode, const float* d_traj, const float* d_dcf,
                            uint32_t* flags, unsigned char* records, unsigned char* ws, const Lists3& l,
                            uint32_t* entries, unsigned char* expanded, cudaStream_t stream,
                            const TablesArgs* tables = nullptr) {
  const int g = s.grid_rows;
  auto at = [&](size_t offset) { return reinterpret_cast<uint32_t*>(ws + offset); };
  const int count_smem = s.lists_per_frame * 4;
  const int place_smem = s.lists_per_frame * static_cast<int>(kPlaceListBytes);
  auto count = k_count3<W, 2>;
  auto place = k_place3<W, 2>;
  if constexpr (W > 2) {
    if (s.lists_per_row == 3) {
      count = k_count3<W, 3>;
      place = k_place3<W, 3>;
    }
  }
  KSJ_TRY(allow_smem(count, count_smem, kListSmem));
  KSJ_TRY(allow_smem(place, place_smem, kListSmem));
  {
    Prepare3Args p{};
    p.traj = d_traj;
    p.dcf = d_dcf;
    p.dcf_mode = dcf_mode;
    p.records = records;
    p.counts = at(l.plane_counts);
    p.flags = flags;
    p.samples = s.samples;
    p.grid = g;
    p.bin_span = s.bin_span;
    p.beta = s.beta;
    p.two_over_w = 2.0f / static_cast<float>(s.width);
    p.inv_i0_beta = s.inv_i0_beta;
    p.phase = s.phase_row;
    LaunchScope scope("k_prepare3", stream);
    k_prepare3<W><<<s.bin_blocks, kBinThreads, 0, stream>>>(p);
    KSJ_TRY(check_launch());
  }
  {
    LaunchScope scope("k_bin_prefix", stream);
    KSJ_TRY(launch_chained(k_bin_prefix, (g + 127) / 128, 128, 0, stream, at(l.plane_counts), at(l.plane_totals), s.bin_blocks, g));
  }
  KSJ_TRY(launch_scan(at(l.plane_totals), at(l.plane_offsets), g, 1, tables, stream));
  {
    LaunchScope scope("k_plane_place", stream);
    k_plane_place<W><<<s.bin_blocks, kBinThreads, 0, stream>>>(records, at(l.plane_offsets), at(l.plane_counts),
                                                              at(l.plane_samples), s.samples, g, s.bin_span);
    KSJ_TRY(check_launch());
  }
  const dim3 blocks(kPlaneBlocks, g);
  {
    LaunchScope scope("k_count3", stream);
    count<<<blocks, kBinThreads, count_smem, stream>>>(records, at(l.plane_offsets), at(l.plane_samples),
                                                            at(l.counts), g, s.nchunks, s.lists_per_frame);
    KSJ_TRY(check_launch());
  }
  {
    LaunchScope scope("k_bin_prefix", stream);
    KSJ_TRY(launch_chained(k_bin_prefix, dim3((s.lists_per_frame + 127) / 128, g), 128, 0, stream, at(l.counts), at(l.totals),
                   kPlaneBlocks, s.lists_per_frame));
  }
  KSJ_TRY(launch_scan(at(l.totals), at(l.offsets), s.lists_per_frame, g, nullptr, stream));
  {
    LaunchScope scope("k_plane_offsets", stream);
    k_plane_bases<<<1, 512, 0, stream>>>(at(l.offsets), g, s.lists_per_frame, at(l.bases));
    KSJ_TRY(check_launch());
    const size_t total = static_cast<size_t>(g) * (s.lists_per_frame + 1);
    k_offsets_add<<<static_cast<unsigned>((total + 255) / 256), 256, 0, stream>>>(at(l.offsets), g, s.lists_per_frame,
                                                                                at(l.bases));
    KSJ_TRY(check_launch());
  }
  {
    const Place3Args p{records, at(l.plane_offsets), at(l.plane_samples), at(l.offsets), at(l.counts), expanded, entries,
                       g, s.nchunks, s.lists_per_frame};
    LaunchScope scope("k_place3", stream);
    place<<<blocks, kBinThreads, place_smem, stream>>>(p);
    KSJ_TRY(check_launch());
  }
  return KSJ_GPU_OK;
}

// out[i] = in[i / times].
__global__ void __launch_bounds__(256) k_repeat(const float* in, float* out, int times, int total) {
  const int i = blockIdx.x * 256 + threadIdx.x;
  if (i < total) out[i] = in[i / times];
}

template <int W, uint32_t kFormat>
ksj_gpu_status launch_all3(const Shape& s, const Layout3& l, const ksj_gpu_gridding3_desc* d, const void* d_kspace,
                           const float* d_traj, const float* d_dcf, void* d_out, unsigned char* ws,
                           cudaStream_t stream) {
  const int g = s.grid_rows, n = s.rows;
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + l.flags);
  uint32_t* offsets = reinterpret_cast<uint32_t*>(ws + l.lists.offsets);
  float2* inter = reinterpret_cast<float2*>(ws + l.inter);
  float2* inter2 = reinterpret_cast<float2*>(ws + l.inter2);
  float2* tw_rows = reinterpret_cast<float2*>(ws + l.tables);
  float2* tw_cols = tw_rows + g;
  float* inv_dr = reinterpret_cast<float*>(tw_cols + g);
  float* inv_dc = inv_dr + n;
  int* pos_rows = reinterpret_cast<int*>(inv_dc + n);
  int* pos_cols = pos_rows + n;
  float* ones = reinterpret_cast<float*>(pos_cols + n);
  float* inv_dc_parts = ones + static_cast<size_t>(n) * n;
  const int parts = column_parts3(s);

  if (cudaMemsetAsync(flags, 0, kFlagBytes, stream) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  const TablesArgs tables{tw_rows, tw_cols, inv_dr, inv_dc, pos_rows, pos_cols, g, g, n, n, s.plan_rows, s.plan_cols, 1,
                          s.width, s.beta, std::cyl_bessel_i(0.0, static_cast<double>(s.beta))};
  {
    LaunchScope scope("k_fill_ones", stream);
    k_fill<<<(n * n + 255) / 256, 256, 0, stream>>>(ones, n * n, 1.0f);
    KSJ_TRY(check_launch());
  }
  {
    const ksj_gpu_status st = build_lists3<W>(s, d->dcf_mode, d_traj, d_dcf, flags, ws + l.records, ws, l.lists, nullptr,
                                              ws + l.expanded, stream, &tables);
    if (st != KSJ_GPU_OK) return st;
  }
  if (parts > 1) {
    LaunchScope scope("k_repeat", stream);
    k_repeat<<<(n * parts + 255) / 256, 256, 0, stream>>>(inv_dc, inv_dc_parts, parts, n * parts);
    KSJ_TRY(check_launch());
  }
  {
    const dim3 tg((s.samples + 31) / 32, (s.channels + 31) / 32, 1);
    LaunchScope scope("k_samples_coil_last", stream);
    const CoilLastArgs a{d_kspace, reinterpret_cast<float2*>(ws + l.samples_t),
                         ws + l.records + offsetof(SampleRecord3<W>, scale), static_cast<int>(sizeof(SampleRecord3<W>)),
                         s.channels, s.samples, flags, nullptr, nullptr, nullptr, 0, nullptr};
    KSJ_TRY(launch_chained(k_samples_coil_last<kFormat>, tg, dim3(32, 8), 0, stream, a));
  }
  // rows of every plane (x transformed, kept columns, coil-last)
  RowsArgs r{};
  r.samples_t = reinterpret_cast<const float2*>(ws + l.samples_t);
  r.sample_frame_stride = 0;
  r.offsets = offsets;
  r.expanded = ws + l.expanded;
  r.width = s.width;
  r.tw_cols = tw_cols;
  r.pos_cols = pos_cols;
  r.inter = inter;
  r.flags = flags;
  r.frames = g;
  r.channels = s.channels;
  r.samples = s.samples;
  r.grid_rows = g;
  r.grid_cols = g;
  r.nchunks = s.nchunks;
  r.lists_per_frame = s.lists_per_frame;
  r.entries_per_frame = 0;
  r.coil_group = s.coil_group;
  r.coil_parts = s.coil_parts;
  r.wait_limit = s.wait_fault ? s.wait_fault : kWaitLimit;
  r.wait_beyond = s.wait_fault ? (1 << 30) : 0;
  r.out_cols = n;
  r.cpitch = s.cpitch;
  r.plan = s.plan_cols;
  r.col_shift = n / 2;
  r.first_of_two = s.first_of_two;
  RowsLauncher rows_launch;
  if (!rows_launch.setup(s)) return KSJ_GPU_ERROR_CUDA;
  // columns of every plane (y transformed, cropped, y/x deapodised): [plane][pixel][cpitch]
  ColsArgs c{};
  c.tw_rows = tw_rows;
  c.inv_dr = inv_dr;
  c.inv_dc = inv_dc;
  c.pos_rows = pos_rows;
  c.flags = flags;
  c.frames = g;
  c.channels = s.channels;
  c.grid_rows = g;
  c.out_rows = n;
  c.out_cols = n;
  c.kb = 1;
  c.row_shift = n / 2;
  c.column_block = s.column_block;
  c.col_group = s.col_group;
  c.groups = column_groups(s);
  c.plan = s.plan_rows;
  c.output = KSJ_GPU_OUTPUT_COIL_LAST;
  c.out = inter2;
  c.out_pitch = s.cpitch;
  // [plane][row][column][pitch] is also [plane][row][column, part][pitch / parts], before the
  // pass and after it
  Shape y = s;
  ColsArgs cy = c;
  if (parts > 1) {
    y.cpitch = y.col_group = y.channels = s.cpitch / parts;
    y.column_block = std::max(1, 32 / y.col_group);
    y.out_cols = n * parts;
    cy.channels = cy.col_group = cy.out_pitch = y.cpitch;
    cy.column_block = y.column_block;
    cy.groups = 1;
    cy.out_cols = y.out_cols;
    cy.inv_dc = inv_dc_parts;
  }
  ColsPass cols_pass;
  if (!cols_pass.setup(y, inter, &cy)) return KSJ_GPU_ERROR_CUDA;
  for (int f0 = 0; f0 < g; f0 += s.frames_per_pass) {
    const int nf = std::min(s.frames_per_pass, g - f0);
    r.frame0 = f0;
    cy.frame0 = f0;
    KSJ_TRY(rows_launch.launch(r, g, (s.channels + s.coil_group - 1) / s.coil_group, nf, stream));
    KSJ_TRY(cols_pass.launch(cy, nf, stream, "k_cols"));
  }
  // z: the column pass over [plane][pixel][cpitch] with planes as rows and pixels as columns
  Shape z = s;
  z.frames = 1;
  z.out_cols = n * n;
  ColsArgs cz = c;
  cz.frame0 = 0;
  cz.frames = 1;
  cz.out_cols = n * n;
  cz.inv_dc = ones;
  cz.output = d->output;
  cz.out = d_out;
  cz.out_pitch = s.channels;
  ColsPass z_pass;
  if (!z_pass.setup(z, inter2, &cz)) return KSJ_GPU_ERROR_CUDA;
  KSJ_TRY(z_pass.launch(cz, 1, stream, "k_cols_z"));
  return check_launch();
}

// ------------------------------------------- 3-D Pipe-Menon density weights

template <int W>
struct PmRecord3 {
  int z0, r0, c0, pad;
  double wz[W];
  double wr[W];
  double wc[W];
};

// The column part of a 3-D record, compact: what the grid step gathers per
// entry after the first iteration (the entry's plane and row weight product
// is kept per entry then).
template <int W>
struct PmCol3 {
  double wc[W];
  int c0, pad;
};

template <int W>
__global__ void __launch_bounds__(256) k_pm_prepare3(const float* traj, PmRecord3<W>* pm, PmCol3<W>* pmc, double* w,
                                                     int samples, int grid, double beta, double inv_i0_beta) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= samples) return;
  float k[3];
#pragma unroll
  for (int d = 0; d < 3; ++d) k[d] = __ldg(traj + 3 * static_cast<size_t>(idx) + d);
  const bool ok = isfinite(k[0]) && isfinite(k[1]) && isfinite(k[2]) && fabsf(k[0]) < 1.0e4f &&
                  fabsf(k[1]) < 1.0e4f && fabsf(k[2]) < 1.0e4f;
  PmRecord3<W> r;
  r.pad = 0;
  constexpr double kTwoPiD = 6.283185307179586476925286766559;
  int t0[3] = {0, 0, 0};
  double u[3] = {0.0, 0.0, 0.0};
  if (ok)
    for (int d = 0; d < 3; ++d) {
      u[d] = static_cast<double>(k[d]) * grid / kTwoPiD;
      t0[d] = static_cast<int>(floor(u[d])) - W / 2 + 1;
    }
  r.z0 = wrap_index(t0[0], grid);
  r.r0 = wrap_index(t0[1], grid);
  r.c0 = wrap_index(t0[2], grid);
#pragma unroll
  for (int j = 0; j < W; ++j) {
    r.wz[j] = ok ? kb_weight64(static_cast<double>(t0[0] + j) - u[0], W, beta, inv_i0_beta) : 0.0;
    r.wr[j] = ok ? kb_weight64(static_cast<double>(t0[1] + j) - u[1], W, beta, inv_i0_beta) : 0.0;
    r.wc[j] = ok ? kb_weight64(static_cast<double>(t0[2] + j) - u[2], W, beta, inv_i0_beta) : 0.0;
  }
  pm[idx] = r;
  PmCol3<W> c;
#pragma unroll
  for (int j = 0; j < W; ++j) c.wc[j] = r.wc[j];
  c.c0 = r.c0;
  c.pad = 0;
  pmc[idx] = c;
  w[idx] = ok ? 1.0 : 0.0;
}

// One lane's share of a 3-D list's entries (as pm_accumulate).  The first
// iteration (kFirst) reads each entry's whole record, forms u = w * (wz[dz] *
// wr[dr]) and keeps the product wz[dz] * wr[dr] per entry (wzr, in entry
// order); the later iterations gather only w and the compact column record
// and read the product back in entry order -- under half the bytes per
// entry, the bound of this step.  The same operations in the same order
// either way: bit-identical cells.
template <int W, bool kFirst>
__device__ __forceinline__ void pm3_accumulate(const uint32_t* entries, uint32_t e0, uint32_t e1, uint32_t step,
                                               const PmRecord3<W>* pm, const PmCol3<W>* pmc, const double* w,
                                               double* wzr, int plane, int row, int lo, int g, double* cell) {
  for (uint32_t e = e0; e < e1; e += step) {
    const uint32_t sidx = __ldg(entries + e);
    double f;
    int col;
    const double* wc;
    if constexpr (kFirst) {
      const PmRecord3<W>& r = pm[sidx];
      int dz = plane - r.z0;
      if (dz < 0) dz += g;
      int dr = row - r.r0;
      if (dr < 0) dr += g;
      f = dz < W && dr < W ? r.wz[dz] * r.wr[dr] : 0.0;
      wzr[e] = f;
      col = r.c0;
      wc = r.wc;
    } else {
      f = wzr[e];
      const PmCol3<W>& c = pmc[sidx];
      col = c.c0;
      wc = c.wc;
    }
    // taps outside the list's plane or row (f >= 0: an integer test keeps
    // the FP64 pipe, the bound of this step, for the arithmetic)
    if (__double_as_longlong(f) == 0) continue;
    const double u = w[sidx] * f;
#pragma unroll
    for (int k = 0; k < W; ++k) {
      const int t = col - lo;
      if (t >= 0 && t < kChunk) cell[t * kPmThreads] = fma(u, wc[k], cell[t * kPmThreads]);
      if (++col == g) col = 0;
    }
  }
}

// The 3-D grid step for lists of at most `capacity` entries: the
// kPmLanes lanes per list, with the entry's plane weight in u; cell t of thread i at
// cells[t * kPmThreads + i], so that the lanes of a warp always touch distinct banks.
// Longer lists (queued by k_pm_queue) are left to k_pm_long3.
template <int W, bool kFirst>
__global__ void __launch_bounds__(kPmThreads) k_pm_grid3(const uint32_t* offsets, const uint32_t* entries,
                                                         const PmRecord3<W>* pm, const PmCol3<W>* pmc, const double* w,
                                                         double* wzr, double* grid, int g, int nchunks,
                                                         int lists_per_plane, int capacity) {
  __shared__ double cells[kChunk * kPmThreads];
  const size_t list = (static_cast<size_t>(blockIdx.x) * kPmThreads + threadIdx.x) / kPmLanes;
  const int q = threadIdx.x & (kPmLanes - 1);
  double* cell = cells + threadIdx.x;
#pragma unroll
  for (int t = 0; t < kChunk; ++t) cell[t * kPmThreads] = 0.0;
  bool active = list < static_cast<size_t>(g) * lists_per_plane;
  int plane = 0, row = 0, lo = 0;
  if (active) {
    plane = static_cast<int>(list / lists_per_plane);
    const int l = static_cast<int>(list - static_cast<size_t>(plane) * lists_per_plane);
    row = l / nchunks;
    lo = (l - row * nchunks) * kChunk;
    const uint32_t* off = offsets + static_cast<size_t>(plane) * (lists_per_plane + 1);
    const uint32_t begin = off[l], end = off[l + 1];
    active = static_cast<int>(end - begin) <= capacity;
    if (active)
      pm3_accumulate<W, kFirst>(entries, begin + q, end, kPmLanes, pm, pmc, w, wzr, plane, row, lo, g, cell);
  }
  __syncwarp();
  if (active) pm_reduce_store(cells, threadIdx.x - q, q, grid + (static_cast<size_t>(plane) * g + row) * g, lo, g);
}

// The lists longer than kPmLong entries, queued: count at long_lists[0]
// (cleared before), global list ids after it.
constexpr int kPmLong = 512;

__global__ void __launch_bounds__(256) k_pm_queue(const uint32_t* offsets, int planes, int lists, uint32_t* long_lists) {
  const size_t i = static_cast<size_t>(blockIdx.x) * blockDim.x + threadIdx.x;
  if (i >= static_cast<size_t>(planes) * lists) return;
  const uint32_t* off = offsets + i + i / lists;  // lists + 1 offsets per plane
  if (off[1] - off[0] > kPmLong) long_lists[1 + atomicAdd(long_lists, 1u)] = static_cast<uint32_t>(i);
}

// The queued long lists
// are cut into parts of kPmPart entries: part_base[i] is the first part of
// queued list i (an exclusive scan, the total at part_base[count]).
constexpr uint32_t kPmPart = 512;

__global__ void __launch_bounds__(1024) k_pm_long_parts(const uint32_t* long_lists, const uint32_t* offsets,
                                                        int lists_per_plane, uint32_t* part_base) {
  __shared__ uint32_t warp_sums[32];
  __shared__ uint32_t carry;
  const uint32_t queued = long_lists[0];
  if (threadIdx.x == 0) carry = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (uint32_t i0 = 0; i0 < queued; i0 += 1024) {
    const uint32_t i = i0 + threadIdx.x;
    uint32_t parts = 0;
    if (i < queued) {
      const uint32_t gl = long_lists[1 + i];
      const uint32_t plane = gl / static_cast<uint32_t>(lists_per_plane);
      const uint32_t l = gl - plane * static_cast<uint32_t>(lists_per_plane);
      const uint32_t* off = offsets + static_cast<size_t>(plane) * (lists_per_plane + 1);
      parts = (off[l + 1] - off[l] + kPmPart - 1) / kPmPart;
    }
    uint32_t incl = parts;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
      const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
      if (lane >= d) incl += v;
    }
    if (lane == 31) warp_sums[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      uint32_t ws = warp_sums[lane];
#pragma unroll
      for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, ws, d);
        if (lane >= d) ws += v;
      }
      warp_sums[lane] = ws;  // inclusive over warps
    }
    __syncthreads();
    const uint32_t before = carry + (warp > 0 ? warp_sums[warp - 1] : 0u) + incl - parts;
    if (i < queued) part_base[i] = before;
    __syncthreads();
    if (threadIdx.x == 1023) carry = before + parts;
    __syncthreads();
  }
  if (threadIdx.x == 0) part_base[queued] = carry;
}

// The long lists' parts, kPmLanes lanes per part (as in k_pm_grid3; every
// part the same work however long its list).  Each part's sums go to
// partial[part]; the part that completes its list's count (the counters grow
// by the list's part count every iteration, zeroed once per call) adds the
// list's parts in part order and writes the cells -- deterministic, and no
// part waits for another.  Groups stride over the parts.
template <int W, bool kFirst>
__global__ void __launch_bounds__(kPmThreads) k_pm_long3(const uint32_t* long_lists, const uint32_t* part_base,
                                                         const uint32_t* offsets, const uint32_t* entries,
                                                         const PmRecord3<W>* pm, const PmCol3<W>* pmc,
                                                         const double* w, double* wzr, double* grid, int g,
                                                         int nchunks, int lists_per_plane, double* partial,
                                                         uint32_t* counters) {
  __shared__ double cells[kChunk * kPmThreads];
  const int q = threadIdx.x & (kPmLanes - 1);
  const int lane0 = (threadIdx.x & 31) & ~(kPmLanes - 1);
  const unsigned gmask = ((1u << kPmLanes) - 1u) << lane0;
  const uint32_t queued = long_lists[0];
  const uint32_t total_parts = part_base[queued];
  const uint32_t groups = gridDim.x * (kPmThreads / kPmLanes);
  double* cell = cells + threadIdx.x;
  for (uint32_t part = (blockIdx.x * kPmThreads + threadIdx.x) / kPmLanes; part < total_parts; part += groups) {
    // the queued list holding this part: the last i with part_base[i] <= part
    uint32_t lo_i = 0, hi_i = queued;  // part_base[lo_i] <= part < part_base[hi_i]
    while (hi_i - lo_i > 1) {
      const uint32_t mid = (lo_i + hi_i) / 2;
      if (__ldg(part_base + mid) <= part)
        lo_i = mid;
      else
        hi_i = mid;
    }
    const uint32_t first = __ldg(part_base + lo_i), parts = __ldg(part_base + lo_i + 1) - first;
    const uint32_t gl = __ldg(long_lists + 1 + lo_i);
    const int plane = static_cast<int>(gl / static_cast<uint32_t>(lists_per_plane));
    const int l = static_cast<int>(gl - static_cast<uint32_t>(plane) * lists_per_plane);
    const int row = l / nchunks;
    const int lo = (l - row * nchunks) * kChunk;
    const uint32_t* off = offsets + static_cast<size_t>(plane) * (lists_per_plane + 1);
    const uint32_t e0 = off[l] + (part - first) * kPmPart, e1 = min(off[l + 1], e0 + kPmPart);
#pragma unroll
    for (int t = 0; t < kChunk; ++t) cell[t * kPmThreads] = 0.0;
    pm3_accumulate<W, kFirst>(entries, e0 + q, e1, kPmLanes, pm, pmc, w, wzr, plane, row, lo, g, cell);
    __syncwarp(gmask);
    // this part's sums (cells 4q .. 4q+3 over the group's lanes)
    double* mine = partial + static_cast<size_t>(part) * kChunk + q * kPmCellsPerLane;
#pragma unroll
    for (int i = 0; i < kPmCellsPerLane; ++i) {
      const double* c = cells + (q * kPmCellsPerLane + i) * kPmThreads + (threadIdx.x - q);
      double acc = c[q];
#pragma unroll
      for (int j = 1; j < kPmLanes; ++j) acc += c[(q + j) & (kPmLanes - 1)];
      mine[i] = acc;
    }
    __threadfence();
    __syncwarp(gmask);
    uint32_t old = 0;
    if (q == 0) old = atomicAdd(counters + lo_i, 1u);
    old = __shfl_sync(gmask, old, lane0);
    if ((old + 1) % parts == 0) {
      __threadfence();
      double acc[kPmCellsPerLane];
#pragma unroll
      for (int i = 0; i < kPmCellsPerLane; ++i) acc[i] = 0.0;
      for (uint32_t p = first; p < first + parts; ++p) {
        const double* src = partial + static_cast<size_t>(p) * kChunk + q * kPmCellsPerLane;
#pragma unroll
        for (int i = 0; i < kPmCellsPerLane; ++i) acc[i] += __ldcg(src + i);
      }
      double* out_row = grid + (static_cast<size_t>(plane) * g + row) * g;
#pragma unroll
      for (int i = 0; i < kPmCellsPerLane; ++i) {
        const int col = lo + q * kPmCellsPerLane + i;
        if (col < g) out_row[col] = acc[i];
      }
    }
    __syncwarp(gmask);  // the cells are read before the next part clears them
  }
}

template <int W>
__global__ void __launch_bounds__(256) k_pm_update3(const PmRecord3<W>* pm, const double* grid, double* w, float* out,
                                                    int samples, int g) {
  const int idx = blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= samples) return;
  const PmRecord3<W> r = pm[idx];
  // separable taps: d = sum_a wz[a] sum_b wr[b] (sum_c wc[c] grid[a][b][c]):
  // W^3 + W^2 + W FP64 operations instead of 2 W^3 + W^2
  int cols[W];
#pragma unroll
  for (int c = 0; c < W; ++c) {
    cols[c] = r.c0 + c;
    if (cols[c] >= g) cols[c] -= g;
  }
  double d = 0.0;
  for (int a = 0; a < W; ++a) {
    int zz = r.z0 + a;
    if (zz >= g) zz -= g;
    double plane = 0.0;
#pragma unroll
    for (int b = 0; b < W; ++b) {
      int yy = r.r0 + b;
      if (yy >= g) yy -= g;
      const double* line = grid + (static_cast<size_t>(zz) * g + yy) * g;
      double t = 0.0;
#pragma unroll
      for (int c = 0; c < W; ++c) t = fma(line[cols[c]], r.wc[c], t);
      plane = fma(r.wr[b], t, plane);
    }
    d = fma(r.wz[a], plane, d);
  }
  const double nw = d > 0.0 ? w[idx] / d : 0.0;
  w[idx] = nw;
  if (out != nullptr) out[idx] = static_cast<float>(nw);
}

struct PmLayout3 {
  size_t flags, records, entries, long_lists, pm, pmc, wzr, w, grid, part_base, partial, counters, total, entries_total,
      max_long;
  Lists3 lists;
};

PmLayout3 make_pm_layout3(const Shape& s) {
  PmLayout3 l{};
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t g = static_cast<size_t>(s.grid_rows);
  l.entries_total = static_cast<size_t>(s.samples) * s.width * s.width * s.lists_per_row;
  l.max_long = l.entries_total / (kPmLong + 1) + 2;
  l.flags = take(kFlagBytes);
  l.records = take(static_cast<size_t>(s.samples) * record3_bytes(s.width));
  l.lists = take_lists3(s, take);
  l.entries = take(l.entries_total * 4);
  l.long_lists = take(l.max_long * 4);
  l.pm = take(static_cast<size_t>(s.samples) * (16 + 24 * static_cast<size_t>(s.width)));
  l.pmc = take(static_cast<size_t>(s.samples) * (8 + 8 * static_cast<size_t>(s.width)));
  l.wzr = take(l.entries_total * sizeof(double));
  l.w = take(static_cast<size_t>(s.samples) * sizeof(double));
  l.grid = take(g * g * g * sizeof(double));
  // the long lists' parts of kPmPart entries: first part of each list, the
  // parts' sums, one counter per list
  l.part_base = take((l.max_long + 1) * 4);
  l.partial = take((l.entries_total / kPmPart + l.max_long) * kChunk * sizeof(double));
  l.counters = take(l.max_long * 4);
  l.total = off;
  return l;
}

template <int W>
ksj_gpu_status launch_pipe_menon3(const Shape& s, const PmLayout3& l, uint32_t iterations, const float* d_traj,
                                  float* d_dcf, unsigned char* ws, cudaStream_t stream) {
  static_assert(sizeof(PmRecord3<W>) == 16 + 24 * W, "PmRecord3 layout");
  const int g = s.grid_rows;
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + l.flags);
  if (cudaMemsetAsync(flags, 0, kFlagBytes, stream) != cudaSuccess ||
      cudaMemsetAsync(ws + l.long_lists, 0, 4, stream) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  const ksj_gpu_status st =
      build_lists3<W>(s, KSJ_GPU_DCF_NONE, d_traj, nullptr, flags, ws + l.records, ws, l.lists,
                      reinterpret_cast<uint32_t*>(ws + l.entries), nullptr, stream);
  if (st != KSJ_GPU_OK) return st;
  static_assert(sizeof(PmCol3<W>) == 8 + 8 * W, "PmCol3 layout");
  PmRecord3<W>* pm = reinterpret_cast<PmRecord3<W>*>(ws + l.pm);
  PmCol3<W>* pmc = reinterpret_cast<PmCol3<W>*>(ws + l.pmc);
  double* wzr = reinterpret_cast<double*>(ws + l.wzr);
  double* w = reinterpret_cast<double*>(ws + l.w);
  double* grid = reinterpret_cast<double*>(ws + l.grid);
  {
    LaunchScope scope("k_pm_prepare3", stream);
    k_pm_prepare3<W><<<(s.samples + 255) / 256, 256, 0, stream>>>(d_traj, pm, pmc, w, s.samples, g, s.beta,
                                                                 1.0 / std::cyl_bessel_i(0.0, static_cast<double>(s.beta)));
    KSJ_TRY(check_launch());
  }
  const uint32_t* offsets = reinterpret_cast<const uint32_t*>(ws + l.lists.offsets);
  const uint32_t* entries = reinterpret_cast<const uint32_t*>(ws + l.entries);
  const uint32_t* long_lists = reinterpret_cast<const uint32_t*>(ws + l.long_lists);
  uint32_t* part_base = reinterpret_cast<uint32_t*>(ws + l.part_base);
  uint32_t* counters = reinterpret_cast<uint32_t*>(ws + l.counters);
  double* partial = reinterpret_cast<double*>(ws + l.partial);
  if (cudaMemsetAsync(counters, 0, l.max_long * 4, stream) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  {
    LaunchScope scope("k_pm_queue", stream);
    const size_t lists = static_cast<size_t>(g) * s.lists_per_frame;
    k_pm_queue<<<static_cast<unsigned>((lists + 255) / 256), 256, 0, stream>>>(
        offsets, g, s.lists_per_frame, reinterpret_cast<uint32_t*>(ws + l.long_lists));
    KSJ_TRY(check_launch());
  }
  {
    LaunchScope scope("k_pm_long_parts", stream);
    k_pm_long_parts<<<1, 1024, 0, stream>>>(long_lists, offsets, s.lists_per_frame, part_base);
    KSJ_TRY(check_launch());
  }
  const size_t lists = static_cast<size_t>(g) * s.lists_per_frame;
  const unsigned grid_blocks = static_cast<unsigned>((lists * kPmLanes + kPmThreads - 1) / kPmThreads);
  // the long-list parts: a grid-stride loop over six 256-thread blocks per SM
  int device = 0, sms = 0;
  if (cudaGetDevice(&device) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess || sms <= 0)
    return KSJ_GPU_ERROR_CUDA;
  const unsigned long_blocks = static_cast<unsigned>(sms) * 6;
  for (uint32_t it = 0; it < iterations; ++it) {
    // the first iteration keeps each entry's plane-row weight product
    {
      LaunchScope scope("k_pm_grid3", stream);
      auto kernel = it == 0 ? k_pm_grid3<W, true> : k_pm_grid3<W, false>;
      kernel<<<grid_blocks, kPmThreads, 0, stream>>>(offsets, entries, pm, pmc, w, wzr, grid, g, s.nchunks,
                                                     s.lists_per_frame, kPmLong);
      KSJ_TRY(check_launch());
    }
    {
      LaunchScope scope("k_pm_long3", stream);
      auto kernel = it == 0 ? k_pm_long3<W, true> : k_pm_long3<W, false>;
      kernel<<<long_blocks, kPmThreads, 0, stream>>>(long_lists, part_base, offsets, entries, pm, pmc, w, wzr, grid, g,
                                                 s.nchunks, s.lists_per_frame, partial, counters);
      KSJ_TRY(check_launch());
    }
    LaunchScope scope("k_pm_update3", stream);
    k_pm_update3<W><<<(s.samples + 255) / 256, 256, 0, stream>>>(pm, grid, w, it + 1 == iterations ? d_dcf : nullptr,
                                                                s.samples, g);
    KSJ_TRY(check_launch());
  }
  return check_launch();
}

template <int W>
ksj_gpu_status dispatch_format(const Shape& s, const Layout& l, const ksj_gpu_gridding_desc* d, const void* k,
                               const float* t, const float* w, void* o, unsigned char* ws, cudaStream_t st,
                               const HostIo* io = nullptr) {
  if (d->sample_format == KSJ_GPU_SAMPLES_BF16)
    return launch_all<W, KSJ_GPU_SAMPLES_BF16>(s, l, d, k, t, w, o, ws, st, io);
  return launch_all<W, KSJ_GPU_SAMPLES_CF32>(s, l, d, k, t, w, o, ws, st, io);
}

ksj_gpu_status dispatch_width(const Shape& s, const Layout& l, const ksj_gpu_gridding_desc* d, const void* k,
                              const float* t, const float* w, void* o, unsigned char* ws, cudaStream_t st,
                              const HostIo* io = nullptr) {
  switch (s.width) {
    case 2: return dispatch_format<2>(s, l, d, k, t, w, o, ws, st, io);
    case 4: return dispatch_format<4>(s, l, d, k, t, w, o, ws, st, io);
    case 6: return dispatch_format<6>(s, l, d, k, t, w, o, ws, st, io);
    case 8: return dispatch_format<8>(s, l, d, k, t, w, o, ws, st, io);
    default: return KSJ_GPU_ERROR_UNSUPPORTED;
  }
}

// ------------------------------------------------ Cartesian coil images
//
// cartesian_ifft2_coil_images (providers/kspacejet-cartesian-recon/src/
// operators/cartesian_ifft2_coil_images.cpp:372-407): per channel, the
// inverse 2-D DFT normalised by 1 / (rows cols) (fft2_inplace_with_workspace
// with Direction::inverse and Normalization::inverse: 1/cols on the row pass,
// 1/rows on the column pass, libs/numerics/kspacejet-fft/src/eigen/
// eigen_fft_transforms.cpp:148-205), no shift; channel-major k-space in,
// coil-last images out.  Here: the row transform per (frame, row, coil group)
// (k_cart_rows), which reads the channel-major rows as they are and writes
// them coil-last, then the column pass k_cols with its
// deapodisation factors set to 1/rows and 1/cols and no crop or shift.
// An axis whose length has a prime factor above 7 (no mixed-radix plan; the
// reference's transform takes every length 2..512) is transformed by a
// direct DFT instead: the row form of k_cart_rows, and k_cart_cols_direct
// for the columns (coil-last output, then k_rss for the RSS form).

constexpr int kCartThreads = 256;

// Direct inverse DFT of 2^lg lines of length n held line-contiguous in
// shared memory (element (j, line) at x[(j << lg) + line]): output k of a
// line is sum_j x[j] w^(jk), w = exp(2 pi i / n), with jk reduced mod n
// exactly in integers (tw[t] = w^t) and eight interleaved partial sums
// (rounding error ~ sqrt(n / 8) ulp instead of sqrt(n)).  emit(k, line, v).
template <class Emit>
__device__ __forceinline__ void dft_direct_lines(const float2* x, int lg, int n, const float2* tw, int tid,
                                                 int nthreads, Emit emit) {
  const int lines = 1 << lg;
  for (int o = tid; o < n * lines; o += nthreads) {
    const int k = o >> lg, line = o & (lines - 1);
    float2 s[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) s[u] = make_float2(0.0f, 0.0f);
    int e = 0, j = 0;
    for (; j + 8 <= n; j += 8) {
#pragma unroll
      for (int u = 0; u < 8; ++u) {
        const float2 v = x[((j + u) << lg) + line];
        const float2 w = tw[e];
        s[u].x = fmaf(v.x, w.x, fmaf(-v.y, w.y, s[u].x));
        s[u].y = fmaf(v.x, w.y, fmaf(v.y, w.x, s[u].y));
        e += k;
        if (e >= n) e -= n;
      }
    }
    for (int u = 0; j < n; ++j, ++u) {
      const float2 v = x[(j << lg) + line];
      const float2 w = tw[e];
      s[u].x = fmaf(v.x, w.x, fmaf(-v.y, w.y, s[u].x));
      s[u].y = fmaf(v.x, w.y, fmaf(v.y, w.x, s[u].y));
      e += k;
      if (e >= n) e -= n;
    }
    const float re = ((s[0].x + s[1].x) + (s[2].x + s[3].x)) + ((s[4].x + s[5].x) + (s[6].x + s[7].x));
    const float im = ((s[0].y + s[1].y) + (s[2].y + s[3].y)) + ((s[4].y + s[5].y) + (s[6].y + s[7].y));
    emit(k, line, make_float2(re, im));
  }
}

// Twiddles, the normalisation factors and the position of output k of each
// axis's transform (two-step slot or digit-reversed position).
__global__ void k_cart_tables(float2* tw_rows, int rows, float2* tw_cols, int cols, float* inv_dr, float* inv_dc,
                              int* pos_rows, int* pos_cols, DifPlan plan_rows, DifPlan plan_cols) {
  chain_begin();
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < rows) {
    tw_rows[i] = twiddle(i, rows);
    inv_dr[i] = 1.0f / static_cast<float>(rows);
    pos_rows[i] = has_two_step_rows(rows) ? two_step_slot(i, rows) : dif_position(plan_rows, i);
  }
  if (i < cols) {
    tw_cols[i] = twiddle(i, cols);
    inv_dc[i] = 1.0f / static_cast<float>(cols);
    pos_cols[i] = dif_position(plan_cols, i);
  }
}

// One block per (frame, row, coil group of cg): the row's cg coil lines
// transformed along the row and every column written to
// [frame][row][column][cpitch].  kN > 0: the two-step transform of that
// length, its inputs straight from the channel-major rows (a warp takes
// consecutive columns of a coil) and its steps exchanged through shared memory of an
// odd pitch, cg + 1, so that lanes on consecutive columns store to different
// banks; 0: the mixed-radix plan; -1: the direct DFT, both on a copy of the
// rows in shared memory.  Bound by HBM: a separate pass that made the k-space
// coil-last first moved it twice more (8 frames x 32 coils x 256^2: 46 + 120 us, now 57).
template <int kN>
__global__ void __launch_bounds__(kCartThreads) k_cart_rows(const float2* __restrict__ kspace, float2* inter,
                                                            const float2* __restrict__ tw_cols,
                                                            const int* __restrict__ pos_cols, DifPlan plan, int rows,
                                                            int cols, int channels, int cg, int cpitch) {
  chain_begin();
  extern __shared__ __align__(16) float2 cart_smem[];
  float2* acc = cart_smem;
  float2* tw = cart_smem + static_cast<size_t>(cols) * (kN > 0 ? cg + 1 : cg);
  const int row = blockIdx.x, cgi = blockIdx.y, f = blockIdx.z;
  const int lg = ilog2(cg);
  const size_t plane = static_cast<size_t>(rows) * cols;
  const float2* src = kspace + (static_cast<size_t>(f) * channels + cgi * cg) * plane + static_cast<size_t>(row) * cols;
  const int live = min(cg, channels - cgi * cg);
  for (int i = threadIdx.x; i < cols; i += blockDim.x) tw[i] = tw_cols[i];
  if constexpr (kN <= 0) {
    // four columns of eight coils per warp (or as many as make 32): whole
    // 32-byte sectors, and the stores meet a bank four times
    const int lg_c = min(lg, 3);
    for (int i = threadIdx.x; i < ((cols + 31) / 32 * 32) << lg; i += blockDim.x) {
      const int l = i & 31, block = i >> 5;                 // blocks: coils first, then columns
      const int coil = ((block & ((1 << (lg - lg_c)) - 1)) << lg_c) + (l >> (5 - lg_c));
      const int col = ((block >> (lg - lg_c)) << (5 - lg_c)) + (l & ((1 << (5 - lg_c)) - 1));
      if (col < cols) acc[(col << lg) + coil] = coil < live ? __ldg(src + coil * plane + col) : make_float2(0.0f, 0.0f);
    }
  }
  __syncthreads();
  float2* dst = inter + (static_cast<size_t>(f) * rows + row) * cols * cpitch + cgi * cg;
  auto emit = [&](int k, int line, float2 v) {
    if (line < live) dst[static_cast<size_t>(k) * cpitch + line] = v;
  };
  if constexpr (kN > 0) {
    fft_two_step_from<kN / 16, false, false>(
        acc, lg, cg + 1, live, tw, threadIdx.x, blockDim.x,
        [&](int col, int coil) { return __ldg(src + coil * plane + col); }, emit);
  } else if constexpr (kN < 0) {
    dft_direct_lines(acc, lg, cols, tw, threadIdx.x, blockDim.x, emit);
  } else {
    dif_lines(acc, lg, plan, tw, threadIdx.x, blockDim.x);
    const int c = threadIdx.x & (cg - 1);
    if (c < live)
      for (int k = threadIdx.x >> lg; k < cols; k += blockDim.x >> lg)
        dst[static_cast<size_t>(k) * cpitch + c] = acc[(__ldg(pos_cols + k) << lg) + c];
  }
}

using CartRowsKernel = void (*)(const float2*, float2*, const float2*, const int*, DifPlan, int, int, int, int, int);

CartRowsKernel cart_rows_for(int n) {
  if (!is_fft_size(static_cast<uint32_t>(n))) return k_cart_rows<-1>;
  switch (n) {
    case 128: return k_cart_rows<128>;
    case 192: return k_cart_rows<192>;
    case 256: return k_cart_rows<256>;
    case 384: return k_cart_rows<384>;
    case 512: return k_cart_rows<512>;
    default: return k_cart_rows<0>;
  }
}

// Columns of an axis without a mixed-radix plan: one block per (frame,
// column, coil group of cg): the column's rows x cg lines from the
// row-transformed grid [frame][row][column][cpitch] into shared memory, the
// direct DFT along the rows, each output scaled by (1/rows)(1/cols) and
// written coil-last [frame][row][column][channel].
__global__ void __launch_bounds__(kCartThreads) k_cart_cols_direct(const float2* __restrict__ inter, float2* out,
                                                                   const float2* __restrict__ tw_rows, int rows,
                                                                   int cols, int channels, int cg, int cpitch) {
  extern __shared__ __align__(16) float2 cart_smem[];
  float2* acc = cart_smem;
  float2* tw = cart_smem + static_cast<size_t>(rows) * cg;
  const int col = blockIdx.x, cgi = blockIdx.y, f = blockIdx.z;
  const int lg = ilog2(cg);
  const float2* src = inter + (static_cast<size_t>(f) * rows * cols + col) * cpitch + cgi * cg;
  for (int i = threadIdx.x; i < rows * cg; i += blockDim.x)
    acc[i] = __ldg(src + static_cast<size_t>(i >> lg) * cols * cpitch + (i & (cg - 1)));
  for (int i = threadIdx.x; i < rows; i += blockDim.x) tw[i] = tw_rows[i];
  __syncthreads();
  const float scale = (1.0f / static_cast<float>(rows)) * (1.0f / static_cast<float>(cols));
  const int live = min(cg, channels - cgi * cg);
  float2* dst = out + static_cast<size_t>(f) * rows * cols * channels + static_cast<size_t>(col) * channels + cgi * cg;
  dft_direct_lines(acc, lg, rows, tw, threadIdx.x, blockDim.x, [&](int k, int line, float2 v) {
    if (line < live)
      dst[static_cast<size_t>(k) * cols * channels + line] = make_float2(v.x * scale, v.y * scale);
  });
}

// The shape of a Cartesian call as the column pass reads it.
struct CartShape {
  Shape s;
  int cg;  // coils per row block
  size_t flags, coil_last, inter, tables, total;
};

ksj_gpu_status make_cart_shape(uint32_t rows, uint32_t cols, uint32_t channels, uint32_t frames, CartShape* c) {
  if (rows < 2 || cols < 2 || channels == 0 || channels > 64 || frames == 0) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (rows > kMaxGrid || cols > kMaxGrid) return KSJ_GPU_ERROR_UNSUPPORTED;
  Shape& s = c->s;
  s = Shape{};
  s.frames = static_cast<int>(frames);
  s.channels = static_cast<int>(channels);
  s.rows = s.grid_rows = s.out_rows = static_cast<int>(rows);
  s.cols = s.grid_cols = s.out_cols = static_cast<int>(cols);
  s.col_group = 2;
  while (s.col_group < s.channels && s.col_group < 32) s.col_group <<= 1;
  s.cpitch = (s.channels + s.col_group - 1) / s.col_group * s.col_group;
  const int cgroups = s.cpitch / s.col_group;
  auto tile = [&](int b) {
    return static_cast<size_t>(s.grid_rows) * b * s.col_group * sizeof(float2) * (cgroups > 1 ? 2 : 1);
  };
  int cb = std::max(1, 32 / s.col_group);
  if (is_fft_size(rows)) {  // the column pass k_cols and its tile
    while (cb > 1 && (tile(cb) > 110 * 1024 || cb > s.out_cols)) cb >>= 1;
    if (tile(cb) > 200 * 1024) return KSJ_GPU_ERROR_UNSUPPORTED;
    cb = aligned_column_block(s.grid_rows, s.col_group, cb);
  } else {
    cb = 1;
  }
  s.column_block = cb;
  s.frames_per_pass = s.frames;
  // an axis without a mixed-radix plan (direct DFT) keeps an empty plan
  if (!make_dif_plan(s.grid_rows, &s.plan_rows)) s.plan_rows = DifPlan{s.grid_rows, 0, {}, {}, {}, {}, {}};
  if (!make_dif_plan(s.grid_cols, &s.plan_cols)) s.plan_cols = DifPlan{s.grid_cols, 0, {}, {}, {}, {}, {}};
  c->cg = s.col_group;
  size_t off = 0;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t px = static_cast<size_t>(frames) * rows * cols;
  c->flags = take(kFlagBytes);
  // coil images on their way to the RSS of the direct-DFT column form
  c->coil_last = is_fft_size(rows) ? off : take(px * channels * sizeof(float2));
  c->inter = take(px * s.cpitch * sizeof(float2));
  c->tables = take((static_cast<size_t>(rows) + cols) * (sizeof(float2) + sizeof(float) + sizeof(int)));
  c->total = off;
  return KSJ_GPU_OK;
}

// Workspace of the host-buffer entry point: the device workspace, then the
// device copies of the samples, trajectory, density weights and images.
struct HostLayout {
  Layout dev;
  size_t kspace, traj, dcf, out, total;
};

size_t image_frame_bytes(const Shape& s, const ksj_gpu_gridding_desc* d) {
  const size_t px = static_cast<size_t>(s.out_rows) * s.out_cols;
  return d->output == KSJ_GPU_OUTPUT_RSS ? px * sizeof(float) : px * s.channels * sizeof(float2);
}

HostLayout make_host_layout(const Shape& s, const ksj_gpu_gridding_desc* d) {
  HostLayout h{};
  h.dev = make_layout(s, d);
  size_t off = h.dev.total;
  auto take = [&](size_t bytes) {
    const size_t at = off;
    off = align_up(off + bytes, 256);
    return at;
  };
  const size_t fm = static_cast<size_t>(s.frames) * s.samples;
  h.kspace = take(fm * s.channels * sample_bytes(d->sample_format));
  h.traj = take(fm * 2 * sizeof(float));
  h.dcf = d->dcf_mode == KSJ_GPU_DCF_EXTERNAL ? take(fm * sizeof(float)) : off;
  h.out = take(static_cast<size_t>(s.frames) * image_frame_bytes(s, d));
  h.total = off;
  return h;
}

// Non-blocking streams per device for the host-buffer entry point: which 0
// carries the copies, which 1 the odd frame passes.
cudaStream_t side_stream(int device, int which) {
  static std::mutex m;
  static std::map<std::pair<int, int>, cudaStream_t> streams;
  std::lock_guard<std::mutex> lock(m);
  auto it = streams.find({device, which});
  if (it != streams.end()) return it->second;
  cudaStream_t st = nullptr;
  if (cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking) != cudaSuccess) return nullptr;
  streams[{device, which}] = st;
  return st;
}

}  // namespace
}  // namespace ksj_gpu

using namespace ksj_gpu;

extern "C" size_t ksj_gpu_gridding_workspace_bytes(const ksj_gpu_gridding_desc* desc) {
  Shape s{};
  if (make_shape(desc, nullptr, &s) != KSJ_GPU_OK) return 0;
  return make_layout(s, desc).total;
}

extern "C" size_t ksj_gpu_gridding_frame_flags_offset(const ksj_gpu_gridding_desc* desc) {
  Shape s{};
  if (make_shape(desc, nullptr, &s) != KSJ_GPU_OK) return 0;
  return make_layout(s, desc).frame_flags;
}

namespace {
// The adjoint of a uniform batch (ragged null) or a ragged one (per-frame
// counts and input addresses; d_kspace and d_traj unused).
struct Ragged {
  const uint32_t* channels;
  const uint32_t* samples;
  const uint64_t* kspace;
  const uint64_t* traj;
};

ksj_gpu_status gridding_adjoint(const ksj_gpu_gridding_desc* desc, const ksj_gpu_gridding_tuning* tuning,
                                const Ragged* ragged, const void* d_kspace, const float* d_traj, const float* d_dcf,
                                void* d_out, void* d_workspace, size_t workspace_bytes, void* stream) {
  Shape s{};
  const ksj_gpu_status st = make_shape(desc, tuning, &s);
  if (st != KSJ_GPU_OK) return st;
  if (ragged != nullptr) {
    s.frame_channels = ragged->channels;
    s.frame_samples = ragged->samples;
    s.frame_kspace = ragged->kspace;
    s.frame_traj = ragged->traj;
  } else if (d_kspace == nullptr || d_traj == nullptr) {
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  }
  if (d_out == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (desc->dcf_mode == KSJ_GPU_DCF_EXTERNAL && d_dcf == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const Layout l = make_layout(s, desc);
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < l.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(d_kspace) & (sample_bytes(desc->sample_format) - 1)) != 0 ||
      (reinterpret_cast<uintptr_t>(d_traj) & 7u) != 0 || (reinterpret_cast<uintptr_t>(d_out) & 7u) != 0)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (s.frames_per_pass >= s.frames) return dispatch_width(s, l, desc, d_kspace, d_traj, d_dcf, d_out, ws, cs);
  // several passes: odd ones on the second compute stream
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  cudaStream_t alt = side_stream(device, 1);
  cudaEvent_t ready = nullptr, alt_done = nullptr;
  if (alt == nullptr || cudaEventCreateWithFlags(&ready, cudaEventDisableTiming) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  if (cudaEventCreateWithFlags(&alt_done, cudaEventDisableTiming) != cudaSuccess) {
    cudaEventDestroy(ready);
    return KSJ_GPU_ERROR_CUDA;
  }
  const HostIo io{nullptr, alt, nullptr, nullptr, ready, alt_done, nullptr, 0};
  const ksj_gpu_status result = dispatch_width(s, l, desc, d_kspace, d_traj, d_dcf, d_out, ws, cs, &io);
  cudaEventDestroy(ready);
  cudaEventDestroy(alt_done);
  return result;
}
}  // namespace

extern "C" ksj_gpu_status ksj_gpu_gridding_adjoint(const ksj_gpu_gridding_desc* desc,
                                                   const ksj_gpu_gridding_tuning* tuning, const void* d_kspace,
                                                   const float* d_traj, const float* d_dcf, void* d_out,
                                                   void* d_workspace, size_t workspace_bytes, void* stream) {
  return gridding_adjoint(desc, tuning, nullptr, d_kspace, d_traj, d_dcf, d_out, d_workspace, workspace_bytes, stream);
}

extern "C" ksj_gpu_status ksj_gpu_gridding_adjoint_ragged(const ksj_gpu_gridding_desc* desc,
                                                          const ksj_gpu_gridding_tuning* tuning,
                                                          const uint32_t* d_frame_channels,
                                                          const uint32_t* d_frame_samples,
                                                          const uint64_t* d_frame_kspace,
                                                          const uint64_t* d_frame_traj, void* d_out,
                                                          void* d_workspace, size_t workspace_bytes, void* stream) {
  if (d_frame_channels == nullptr || d_frame_samples == nullptr || d_frame_kspace == nullptr ||
      d_frame_traj == nullptr)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (desc == nullptr || desc->struct_size < sizeof(ksj_gpu_gridding_desc) ||
      desc->kernel != KSJ_GPU_KERNEL_KAISER_BESSEL || desc->dcf_mode == KSJ_GPU_DCF_EXTERNAL)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const Ragged r{d_frame_channels, d_frame_samples, d_frame_kspace, d_frame_traj};
  return gridding_adjoint(desc, tuning, &r, nullptr, nullptr, nullptr, d_out, d_workspace, workspace_bytes, stream);
}

extern "C" size_t ksj_gpu_gridding_host_workspace_bytes(const ksj_gpu_gridding_desc* desc) {
  Shape s{};
  if (make_shape(desc, nullptr, &s) != KSJ_GPU_OK) return 0;
  return make_host_layout(s, desc).total;
}

extern "C" ksj_gpu_status ksj_gpu_gridding_adjoint_host(const ksj_gpu_gridding_desc* desc,
                                                        const ksj_gpu_gridding_tuning* tuning, const void* h_kspace,
                                                        const float* h_traj, const float* h_dcf, void* h_out,
                                                        void* d_workspace, size_t workspace_bytes, void* stream) {
  Shape s{};
  const ksj_gpu_status st = make_shape(desc, tuning, &s);
  if (st != KSJ_GPU_OK) return st;
  if (h_kspace == nullptr || h_traj == nullptr || h_out == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (desc->dcf_mode == KSJ_GPU_DCF_EXTERNAL && h_dcf == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  // copies and passes overlap: at least 8 passes (fewer leave more of the
  // first copy exposed; with odd passes on a second stream, 8 measured best
  // for 96 frames); a tuning with smaller passes keeps them
  s.frames_per_pass = std::min(s.frames_per_pass, std::max(1, (s.frames + 7) / 8));
  const HostLayout h = make_host_layout(s, desc);
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < h.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  cudaStream_t copy = side_stream(device, 0), alt = side_stream(device, 1);
  if (copy == nullptr || alt == nullptr) return KSJ_GPU_ERROR_CUDA;
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  const size_t fm = static_cast<size_t>(s.frames) * s.samples;
  const size_t frame_bytes = static_cast<size_t>(s.samples) * s.channels * sample_bytes(desc->sample_format);
  const int passes = (s.frames + s.frames_per_pass - 1) / s.frames_per_pass;
  std::vector<cudaEvent_t> events(static_cast<size_t>(2 * passes + 4), nullptr);
  auto release = [&]() {
    for (cudaEvent_t e : events)
      if (e != nullptr) cudaEventDestroy(e);
  };
  for (cudaEvent_t& e : events)
    if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
      release();
      return KSJ_GPU_ERROR_CUDA;
    }
  cudaEvent_t* in = events.data();
  cudaEvent_t* done = in + passes;
  cudaEvent_t start = done[passes], end = done[passes + 1], ready = done[passes + 2], alt_done = done[passes + 3];
  ksj_gpu_status result = KSJ_GPU_OK;
  // the trajectory (and weights) first, on the stream, for the binning; the
  // copy stream starts after everything already queued on the stream (the
  // staging buffers may still be read by an earlier call)
  if (cudaMemcpyAsync(ws + h.traj, h_traj, fm * 2 * sizeof(float), cudaMemcpyHostToDevice, cs) != cudaSuccess ||
      (desc->dcf_mode == KSJ_GPU_DCF_EXTERNAL &&
       cudaMemcpyAsync(ws + h.dcf, h_dcf, fm * sizeof(float), cudaMemcpyHostToDevice, cs) != cudaSuccess) ||
      cudaEventRecord(start, cs) != cudaSuccess || cudaStreamWaitEvent(copy, start, 0) != cudaSuccess)
    result = KSJ_GPU_ERROR_CUDA;
  for (int p = 0; p < passes && result == KSJ_GPU_OK; ++p) {
    const int f0 = p * s.frames_per_pass, nf = std::min(s.frames_per_pass, s.frames - f0);
    if (cudaMemcpyAsync(ws + h.kspace + f0 * frame_bytes, static_cast<const unsigned char*>(h_kspace) + f0 * frame_bytes,
                        static_cast<size_t>(nf) * frame_bytes, cudaMemcpyHostToDevice, copy) != cudaSuccess ||
        cudaEventRecord(in[p], copy) != cudaSuccess)
      result = KSJ_GPU_ERROR_CUDA;
  }
  if (result == KSJ_GPU_OK) {
    const HostIo io{copy, alt, in, done, ready, alt_done, h_out, image_frame_bytes(s, desc)};
    result = dispatch_width(s, h.dev, desc, ws + h.kspace, reinterpret_cast<const float*>(ws + h.traj),
                            desc->dcf_mode == KSJ_GPU_DCF_EXTERNAL ? reinterpret_cast<const float*>(ws + h.dcf)
                                                                   : nullptr,
                            ws + h.out, ws, cs, &io);
  }
  // the stream completes only after the last image copy
  if (cudaEventRecord(end, copy) != cudaSuccess || cudaStreamWaitEvent(cs, end, 0) != cudaSuccess)
    if (result == KSJ_GPU_OK) result = KSJ_GPU_ERROR_CUDA;
  release();
  return result;
}

extern "C" ksj_gpu_status ksj_gpu_gridding_binning(const ksj_gpu_gridding_desc* desc,
                                                   const ksj_gpu_gridding_tuning* tuning, const void* d_workspace,
                                                   uint32_t* out_chunk_width, uint64_t* out_list_count,
                                                   uint64_t* out_entry_count, uint64_t* out_offsets,
                                                   uint32_t* out_samples) {
  Shape s{};
  const ksj_gpu_status st = make_shape(desc, tuning, &s);
  if (st != KSJ_GPU_OK) return st;
  if (d_workspace == nullptr) return KSJ_GPU_ERROR_WORKSPACE;
  const Layout l = make_layout(s, desc);
  const unsigned char* ws = static_cast<const unsigned char*>(d_workspace);
  const size_t lists = static_cast<size_t>(s.frames) * s.lists_per_frame;
  if (out_chunk_width) *out_chunk_width = kChunk;
  if (out_list_count) *out_list_count = lists;
  std::vector<uint32_t> off(static_cast<size_t>(s.frames) * (s.lists_per_frame + 1));
  if (cudaDeviceSynchronize() != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  if (cudaMemcpy(off.data(), ws + l.offsets, off.size() * 4, cudaMemcpyDeviceToHost) != cudaSuccess)
    return KSJ_GPU_ERROR_CUDA;
  uint64_t total = 0;
  for (int f = 0; f < s.frames; ++f) total += off[static_cast<size_t>(f) * (s.lists_per_frame + 1) + s.lists_per_frame];
  if (out_entry_count) *out_entry_count = total;
  if (out_offsets == nullptr || out_samples == nullptr) return KSJ_GPU_OK;
  uint64_t base = 0;
  for (int f = 0; f < s.frames; ++f) {
    const uint32_t* fo = off.data() + static_cast<size_t>(f) * (s.lists_per_frame + 1);
    for (int i = 0; i < s.lists_per_frame; ++i)
      out_offsets[static_cast<size_t>(f) * s.lists_per_frame + i] = base + fo[i];
    // the sample index of every expanded entry (its second word)
    const uint32_t n = fo[s.lists_per_frame];
    const size_t pitch = entry_bytes(s.width);
    if (n && cudaMemcpy2D(out_samples + base, 4, ws + l.expanded + static_cast<size_t>(f) * s.entries_per_frame * pitch + 4,
                          pitch, 4, n, cudaMemcpyDeviceToHost) != cudaSuccess)
      return KSJ_GPU_ERROR_CUDA;
    base += n;
  }
  out_offsets[lists] = base;
  return KSJ_GPU_OK;
}

extern "C" ksj_gpu_status ksj_gpu_read_flags(const void* d_workspace, void* stream, uint32_t* out_flags) {
  if (d_workspace == nullptr || out_flags == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (cudaStreamSynchronize(cs) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  if (cudaMemcpy(out_flags, d_workspace, sizeof(uint32_t), cudaMemcpyDeviceToHost) != cudaSuccess)
    return KSJ_GPU_ERROR_CUDA;
  return KSJ_GPU_OK;
}

namespace {
std::mutex g_tune_mutex;
// keyed by the shape and the device: a tuning is chosen against one device's
// shared-memory and SM limits
std::map<std::tuple<int, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t, uint32_t,
                    uint32_t, uint32_t>,
         ksj_gpu_gridding_tuning>
    g_tune_cache;
}  // namespace

extern "C" ksj_gpu_status ksj_gpu_gridding_tune(const ksj_gpu_gridding_desc* desc, const void* d_kspace,
                                                const float* d_traj, const float* d_dcf, void* d_out,
                                                void* d_workspace, size_t workspace_bytes, void* stream,
                                                ksj_gpu_gridding_tuning* tuning) {
  if (desc == nullptr || tuning == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  int device = 0;
  if (cudaGetDevice(&device) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  const auto key = std::make_tuple(device, desc->kernel, desc->image_rows, desc->image_cols, desc->grid_rows,
                                   desc->grid_cols, desc->kernel_width, desc->channels, desc->samples, desc->frames,
                                   desc->output, desc->sample_format);
  {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    const auto it = g_tune_cache.find(key);
    if (it != g_tune_cache.end()) {
      *tuning = it->second;
      return KSJ_GPU_OK;
    }
  }
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  cudaEvent_t e0, e1;
  if (cudaEventCreate(&e0) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  if (cudaEventCreate(&e1) != cudaSuccess) {
    cudaEventDestroy(e0);
    return KSJ_GPU_ERROR_CUDA;
  }
  ksj_gpu_gridding_tuning best{};
  float best_ms = 1e30f;
  for (uint32_t cg : {32u, 16u, 8u, 4u, 2u, 1u}) {
    if (cg > 1 && cg / 2 >= desc->channels) continue;
    if (cg * 4 < desc->channels && cg < 8) continue;
    for (uint32_t cbm : {1u, 2u})
    for (uint32_t fpp : {0u, 12u, 48u})
    for (uint32_t colp : {1u, 2u})
    for (uint32_t parts : {1u, 2u}) {
      if (fpp >= desc->frames) continue;
      if (parts > 1 && cg < 16) continue;
      ksj_gpu_gridding_tuning t{};
      t.struct_size = sizeof(t);
      uint32_t gcols = 2;
      while (gcols < desc->channels && gcols < 32) gcols <<= 1;
      t.coil_group = cg;
      t.column_block = cbm * std::max(1u, 32u / gcols);
      t.frames_per_pass = fpp;
      t.rows_blocks_per_sm = 2;
      t.coil_parts = parts;
      t.column_pass = colp;
      Shape s{};
      if (make_shape(desc, &t, &s) != KSJ_GPU_OK) continue;
      if (workspace_bytes < make_layout(s, desc).total) continue;
      if (ksj_gpu_gridding_adjoint(desc, &t, d_kspace, d_traj, d_dcf, d_out, d_workspace, workspace_bytes, stream) !=
          KSJ_GPU_OK)
        continue;
      cudaEventRecord(e0, cs);
      for (int rep = 0; rep < 2; ++rep)
        ksj_gpu_gridding_adjoint(desc, &t, d_kspace, d_traj, d_dcf, d_out, d_workspace, workspace_bytes, stream);
      cudaEventRecord(e1, cs);
      if (cudaEventSynchronize(e1) != cudaSuccess) break;
      float ms = 0.0f;
      cudaEventElapsedTime(&ms, e0, e1);
      if (ms < best_ms) {
        best_ms = ms;
        best = t;
      }
    }
  }
  cudaEventDestroy(e0);
  cudaEventDestroy(e1);
  if (best.struct_size == 0) return KSJ_GPU_ERROR_UNSUPPORTED;
  {
    std::lock_guard<std::mutex> lock(g_tune_mutex);
    g_tune_cache[key] = best;
  }
  *tuning = best;
  return KSJ_GPU_OK;
}

extern "C" size_t ksj_gpu_pipe_menon_workspace_bytes(const ksj_gpu_gridding_desc* desc) {
  PmLayout l{};
  uint32_t per_pass = 0;
  if (desc == nullptr || desc->struct_size < sizeof(ksj_gpu_gridding_desc) ||
      desc->kernel != KSJ_GPU_KERNEL_KAISER_BESSEL)
    return 0;
  return make_pm_layout(desc, &l, &per_pass) == KSJ_GPU_OK ? l.total : 0;
}

extern "C" ksj_gpu_status ksj_gpu_pipe_menon_dcf(const ksj_gpu_gridding_desc* desc, uint32_t iterations,
                                                 const float* d_traj, float* d_dcf, void* d_workspace,
                                                 size_t workspace_bytes, void* stream) {
  if (desc == nullptr || desc->struct_size < sizeof(ksj_gpu_gridding_desc) ||
      desc->kernel != KSJ_GPU_KERNEL_KAISER_BESSEL || iterations == 0 || iterations > 1000)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  PmLayout l{};
  uint32_t per_pass = 0;
  const ksj_gpu_status st = make_pm_layout(desc, &l, &per_pass);
  if (st != KSJ_GPU_OK) return st;
  if (d_traj == nullptr || d_dcf == nullptr || (reinterpret_cast<uintptr_t>(d_traj) & 7u) != 0 ||
      (reinterpret_cast<uintptr_t>(d_dcf) & 3u) != 0)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < l.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(ws, 0, kFlagBytes, cs) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  for (uint32_t f0 = 0; f0 < desc->frames; f0 += per_pass) {
    ksj_gpu_gridding_desc pass = *desc;
    pass.frames = std::min(per_pass, desc->frames - f0);
    Shape s{};
    const ksj_gpu_status ps = make_shape(&pass, nullptr, &s);
    if (ps != KSJ_GPU_OK) return ps;
    const float* traj = d_traj + static_cast<size_t>(f0) * s.samples * 2;
    float* dcf = d_dcf + static_cast<size_t>(f0) * s.samples;
    ksj_gpu_status run = KSJ_GPU_ERROR_UNSUPPORTED;
    switch (s.width) {
      case 2: run = launch_pipe_menon<2>(s, l, &pass, iterations, traj, dcf, ws, cs); break;
      case 4: run = launch_pipe_menon<4>(s, l, &pass, iterations, traj, dcf, ws, cs); break;
      case 6: run = launch_pipe_menon<6>(s, l, &pass, iterations, traj, dcf, ws, cs); break;
      case 8: run = launch_pipe_menon<8>(s, l, &pass, iterations, traj, dcf, ws, cs); break;
    }
    if (run != KSJ_GPU_OK) return run;
  }
  return KSJ_GPU_OK;
}

extern "C" size_t ksj_gpu_gridding3_workspace_bytes(const ksj_gpu_gridding3_desc* desc) {
  Shape s{};
  if (make_shape3(desc, nullptr, &s) != KSJ_GPU_OK) return 0;
  return make_layout3(s).total;
}

extern "C" ksj_gpu_status ksj_gpu_gridding3_adjoint(const ksj_gpu_gridding3_desc* desc,
                                                    const ksj_gpu_gridding_tuning* tuning, const void* d_kspace,
                                                    const float* d_traj, const float* d_dcf, void* d_out,
                                                    void* d_workspace, size_t workspace_bytes, void* stream) {
  Shape s{};
  const ksj_gpu_status st = make_shape3(desc, tuning, &s);
  if (st != KSJ_GPU_OK) return st;
  if (d_kspace == nullptr || d_traj == nullptr || d_out == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (desc->dcf_mode == KSJ_GPU_DCF_EXTERNAL && d_dcf == nullptr) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const Layout3 l = make_layout3(s);
  if (l.entries_total > 0xffffffffull) return KSJ_GPU_ERROR_UNSUPPORTED;
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < l.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  if ((reinterpret_cast<uintptr_t>(d_kspace) & (sample_bytes(desc->sample_format) - 1)) != 0 ||
      (reinterpret_cast<uintptr_t>(d_traj) & 3u) != 0 || (reinterpret_cast<uintptr_t>(d_out) & 7u) != 0)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  const bool bf16 = desc->sample_format == KSJ_GPU_SAMPLES_BF16;
  switch (s.width) {
#define KSJ_G3_CASE(W)                                                                                       \
  case W:                                                                                                    \
    return bf16 ? launch_all3<W, KSJ_GPU_SAMPLES_BF16>(s, l, desc, d_kspace, d_traj, d_dcf, d_out, ws, cs)     \
                : launch_all3<W, KSJ_GPU_SAMPLES_CF32>(s, l, desc, d_kspace, d_traj, d_dcf, d_out, ws, cs);
    KSJ_G3_CASE(2) KSJ_G3_CASE(4) KSJ_G3_CASE(6) KSJ_G3_CASE(8)
#undef KSJ_G3_CASE
    default: return KSJ_GPU_ERROR_UNSUPPORTED;
  }
}

extern "C" size_t ksj_gpu_pipe_menon3_workspace_bytes(const ksj_gpu_gridding3_desc* desc) {
  Shape s{};
  if (make_shape3(desc, nullptr, &s) != KSJ_GPU_OK) return 0;
  return make_pm_layout3(s).total;
}

extern "C" ksj_gpu_status ksj_gpu_pipe_menon_dcf3(const ksj_gpu_gridding3_desc* desc, uint32_t iterations,
                                                  const float* d_traj, float* d_dcf, void* d_workspace,
                                                  size_t workspace_bytes, void* stream) {
  if (iterations == 0 || iterations > 1000) return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  Shape s{};
  const ksj_gpu_status st = make_shape3(desc, nullptr, &s);
  if (st != KSJ_GPU_OK) return st;
  if (d_traj == nullptr || d_dcf == nullptr || (reinterpret_cast<uintptr_t>(d_traj) & 3u) != 0 ||
      (reinterpret_cast<uintptr_t>(d_dcf) & 3u) != 0)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  const PmLayout3 l = make_pm_layout3(s);
  if (l.entries_total > 0xffffffffull) return KSJ_GPU_ERROR_UNSUPPORTED;
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < l.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  cudaStream_t cs = static_cast<cudaStream_t>(stream);
  switch (s.width) {
    case 2: return launch_pipe_menon3<2>(s, l, iterations, d_traj, d_dcf, ws, cs);
    case 4: return launch_pipe_menon3<4>(s, l, iterations, d_traj, d_dcf, ws, cs);
    case 6: return launch_pipe_menon3<6>(s, l, iterations, d_traj, d_dcf, ws, cs);
    case 8: return launch_pipe_menon3<8>(s, l, iterations, d_traj, d_dcf, ws, cs);
    default: return KSJ_GPU_ERROR_UNSUPPORTED;
  }
}

extern "C" size_t ksj_gpu_cartesian_workspace_bytes(uint32_t rows, uint32_t cols, uint32_t channels,
                                                    uint32_t frames) {
  CartShape c{};
  return make_cart_shape(rows, cols, channels, frames, &c) == KSJ_GPU_OK ? c.total : 0;
}

extern "C" ksj_gpu_status ksj_gpu_cartesian_ifft2(uint32_t rows, uint32_t cols, uint32_t channels, uint32_t frames,
                                                  uint32_t output, const void* d_kspace, void* d_out,
                                                  void* d_workspace, size_t workspace_bytes, void* stream) {
  CartShape cs{};
  const ksj_gpu_status st = make_cart_shape(rows, cols, channels, frames, &cs);
  if (st != KSJ_GPU_OK) return st;
  if (d_kspace == nullptr || d_out == nullptr || (output != KSJ_GPU_OUTPUT_COIL_LAST && output != KSJ_GPU_OUTPUT_RSS) ||
      (reinterpret_cast<uintptr_t>(d_kspace) & 7u) != 0 || (reinterpret_cast<uintptr_t>(d_out) & 7u) != 0)
    return KSJ_GPU_ERROR_INVALID_ARGUMENT;
  if (d_workspace == nullptr || (reinterpret_cast<uintptr_t>(d_workspace) & 255u) != 0 || workspace_bytes < cs.total)
    return KSJ_GPU_ERROR_WORKSPACE;
  const Shape& s = cs.s;
  cudaStream_t cstream = static_cast<cudaStream_t>(stream);
  unsigned char* ws = static_cast<unsigned char*>(d_workspace);
  uint32_t* flags = reinterpret_cast<uint32_t*>(ws + cs.flags);
  float2* coil_last = reinterpret_cast<float2*>(ws + cs.coil_last);
  float2* inter = reinterpret_cast<float2*>(ws + cs.inter);
  float2* tw_rows = reinterpret_cast<float2*>(ws + cs.tables);
  float2* tw_cols = tw_rows + rows;
  float* inv_dr = reinterpret_cast<float*>(tw_cols + cols);
  float* inv_dc = inv_dr + rows;
  int* pos_rows = reinterpret_cast<int*>(inv_dc + cols);
  int* pos_cols = pos_rows + rows;
  if (cudaMemsetAsync(flags, 0, kFlagBytes, cstream) != cudaSuccess) return KSJ_GPU_ERROR_CUDA;
  {
    const int n = static_cast<int>(std::max(rows, cols));
    LaunchScope scope("k_cart_tables", cstream);
    KSJ_TRY(launch_chained(k_cart_tables, dim3((n + 255) / 256), dim3(256), 0, cstream, tw_rows, static_cast<int>(rows), tw_cols,
                   static_cast<int>(cols), inv_dr, inv_dc, pos_rows, pos_cols, s.plan_rows, s.plan_cols));
  }
  {
    const CartRowsKernel rk = cart_rows_for(static_cast<int>(cols));
    const size_t smem = (static_cast<size_t>(cols) * (cs.cg + 1) + cols) * sizeof(float2);
    KSJ_TRY(allow_smem(rk, smem));
    const dim3 grid(rows, (channels + cs.cg - 1) / cs.cg, frames);
    LaunchScope scope("k_cart_rows", cstream);
    KSJ_TRY(launch_chained(rk, grid, dim3(kCartThreads), smem, cstream, static_cast<const float2*>(d_kspace), inter, tw_cols,
                   pos_cols, s.plan_cols, static_cast<int>(rows), static_cast<int>(cols), static_cast<int>(channels),
                   cs.cg, s.cpitch));
  }
  if (!is_fft_size(rows)) {
    // direct DFT along the columns, coil-last into the output (or into the
    // workspace, then its RSS)
    float2* dst = output == KSJ_GPU_OUTPUT_COIL_LAST ? static_cast<float2*>(d_out) : coil_last;
    const size_t smem = (static_cast<size_t>(rows) * cs.cg + rows) * sizeof(float2);
    KSJ_TRY(allow_smem(k_cart_cols_direct, smem));
    {
      const dim3 grid(cols, (channels + cs.cg - 1) / cs.cg, frames);
      LaunchScope scope("k_cart_cols_direct", cstream);
      k_cart_cols_direct<<<grid, kCartThreads, smem, cstream>>>(inter, dst, tw_rows, static_cast<int>(rows),
                                                               static_cast<int>(cols), static_cast<int>(channels),
                                                               cs.cg, s.cpitch);
      KSJ_TRY(check_launch());
    }
    if (output == KSJ_GPU_OUTPUT_RSS) {
      return ksj_gpu_rss_coil_last(static_cast<uint64_t>(frames) * rows * cols, channels, coil_last,
                                   static_cast<float*>(d_out), stream);
    }
    return check_launch();
  }
  ColsArgs c{};
  c.tw_rows = tw_rows;
  c.inv_dr = inv_dr;
  c.inv_dc = inv_dc;
  c.pos_rows = pos_rows;
  c.flags = flags;
  c.frames = s.frames;
  c.channels = s.channels;
  c.grid_rows = s.grid_rows;
  c.out_rows = s.out_rows;
  c.out_cols = s.out_cols;
  c.kb = 1;  // apply the factors: here the normalisation
  c.row_shift = 0;
  c.column_block = s.column_block;
  c.col_group = s.col_group;
  c.groups = column_groups(s);
  c.plan = s.plan_rows;
  c.output = output;
  c.out = d_out;
  c.out_pitch = s.channels;
  c.frame0 = 0;
  ColsPass cols_pass;
  if (!cols_pass.setup(s, inter, &c)) return KSJ_GPU_ERROR_CUDA;
  KSJ_TRY(cols_pass.launch(c, s.frames, cstream, "k_cols"));
  return check_launch();
}
