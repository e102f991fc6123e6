// Host-side declarations shared by the translation units of the library (not part of
// the public C ABI, which is include/plenoxels_gb300.h).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "plenoxels_gb300.h"

namespace pgb {

template <typename Real> struct RenderArgs;

// Counts one kernel launch and converts the launch status into a PGB status.
int after_launch();

// Most warps the fused fp64 training kernel may use (size of its loss table).
constexpr int kMaxTrainWarps = 32768;
// Bytes behind the fp64 loss tables of a training workspace: the block counter (fp64), then
// the state of an fp32 launch (TrainState).
constexpr int kTrainStateOffset = 256, kTrainStateBytes = 1024;
// Samples per chunk are 32 * K; a ray may span at most this many chunks.
constexpr int kMaxChunks = 32;
// Largest samples-per-ray the fused kernels accept.
constexpr int kMaxSamples = kMaxChunks * 32 * 8;

// Gradient marks: bit u % 32 of word u / 32 marks unit u = cell >> kMarkCellsLog2, a unit
// some step wrote. Units of 4 cells (64 B of fp32 gradient, two whole sectors): a 256^3
// trilinear step took 0.1014 ms per step with them, 0.1011 ms with 2-cell units and
// 0.1074 ms with 1-cell units, whose clear writes half the bytes but as half sectors and
// whose marks touch twice the words.
#ifndef PGB_MARK_CELLS_LOG2
#define PGB_MARK_CELLS_LOG2 2
#endif
constexpr int kMarkCellsLog2 = PGB_MARK_CELLS_LOG2;
// Words of the mark bitmap of a gradient of num_cells cells.
inline int64_t mark_words(int64_t num_cells) {
  const int64_t units = (num_cells + (1 << kMarkCellsLog2) - 1) >> kMarkCellsLog2;
  return (units + 31) / 32;
}

int launch_render_f32(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
int launch_render_bf16(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
int launch_render_f64(const RenderArgs<double>& a, int mode, int phase, cudaStream_t s);
// Log-sum transmittance form (fp32 arithmetic over fp32 or BF16 cells).
int launch_render_logt_f32(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
int launch_render_logt_bf16(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
// fp32 and BF16 grids outside the quick index arithmetic's range (quick_grid).
int launch_render_general_f32(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
int launch_render_general_bf16(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
int launch_render_general_logt_f32(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);
int launch_render_general_logt_bf16(const RenderArgs<float>& a, int mode, int phase, cudaStream_t s);

// Slots per lane (K) of a chunk of 32 * K samples. A chunk size (32 * K for K in 1, 2, 4, 8,
// 16) is raised until a ray spans at most kMaxChunks chunks. Without a requested one: 32
// samples for trilinear lookup, 64 for nearest. Short chunks skip the most samples behind
// opaque cells where a ray may stop there, and hold fewer registers where it may not (the
// beta term, no clip). Measured on GB300, one training launch, chunks of 32 / 64 / 128 / 256
// samples: 256^3 trilinear, 8192 rays x 256 with early stop 80 / 96 / 105 / 162 us; 7500
// rays x 600 with the beta term trilinear 359 / 380 / 403 / 569 us, nearest 146 / 132 / 134
// / 189 us (256 was the choice there before); nearest without it 105 / 92 / 92 / 127 us. With
// the queue of rays, 8192 rays x 256 with the beta term, opaque, trilinear: 137 / 138 / 237 /
// 277 us (172 before it in one chunk); 200^3 without clip, 64 / 128 / 256 samples: 80 / 126 /
// 169 us in chunks of 32 and 80 / 131 / 206 us in one.
// `long_chunks` keeps whole rays up to 512 samples in one chunk: rays that may not stop early
// and have a threshold on T, which is looked at after each chunk.
inline int pick_slots(int S, int chunk_samples = 0, int mode = PGB_TRILINEAR,
                      bool long_chunks = false) {
#ifdef PGB_FORCE_SLOTS
  if (S <= 32 * kMaxChunks * PGB_FORCE_SLOTS) return PGB_FORCE_SLOTS;
#endif
  if (chunk_samples <= 0 && long_chunks) return S <= 64 ? 2 : S <= 128 ? 4 : S <= 256 || S > 512 ? 8 : 16;
  if (chunk_samples <= 0) chunk_samples = mode == PGB_NEAREST ? 64 : 32;
  int k = 1;
  while (k < 16 && 32 * k < chunk_samples) k *= 2;
  while (k < 16 && (S + 32 * k - 1) / (32 * k) > kMaxChunks) k *= 2;
  return k;
}

}  // namespace pgb
