// Compile-time dispatch of the fused render kernel over lookup mode, phase and slots per
// lane. Included once per storage type (render_f32.cu, render_bf16.cu, render_f64.cu) and
// per storage type for the log-sum transmittance form (render_logt_*.cu) so the instantiations compile
// in parallel.
#pragma once

#include <algorithm>

#include "pgb_host.h"
#include "render.cuh"

namespace pgb {

template <typename Real, typename Store, int MODE, int K, int PHASE, bool LOGT, int A>
int launch_render_k(const RenderArgs<Real>& a, cudaStream_t s) {
  constexpr int kThreads = render_threads<Real, MODE, K, PHASE>();
  constexpr int kWarpsPerBlock = kThreads / kWarp;
  constexpr int kSmem = render_smem_bytes<Real, K, PHASE, LOGT>(kWarpsPerBlock);
  // the dynamic shared-memory opt-in (dynamic + static may pass 48 KiB) is per device:
  // set it on first use of each device, and note how many blocks the device holds
  static int configured[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  int resident = dev >= 0 && dev < 64 ? configured[dev] : 0;
  if (resident == 0) {
    if (cudaFuncSetAttribute(render_kernel<Real, Store, MODE, K, PHASE, LOGT, A>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem) != cudaSuccess)
      return PGB_ERR_LAUNCH;
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(
            &per_sm, render_kernel<Real, Store, MODE, K, PHASE, LOGT, A>, kThreads, kSmem) !=
            cudaSuccess ||
        sms * per_sm < 1)
      return PGB_ERR_LAUNCH;
    resident = sms * per_sm;
    if (dev >= 0 && dev < 64) configured[dev] = resident;
  }
  // fp32: one wave, or a ray per block when there are fewer rays (and nothing to clear beside
  // them); fp64: a ray per warp
  int64_t blocks = std::max<int64_t>(a.R, a.clear_words / kWarp);
  if (sizeof(Real) == 4)
    blocks = std::min<int64_t>(blocks, resident);
  else
    blocks = std::min<int64_t>((a.R + kWarpsPerBlock - 1) / kWarpsPerBlock,
                               PHASE == kTrain ? kMaxTrainWarps / kWarpsPerBlock : (int64_t)1 << 20);
  if (blocks < 1) blocks = 1;
  // Groups of up to 8 consecutive rays as long as every block gets at least 32 groups (one more
  // or less is little then; training batches of some thousand rays keep single rays):
  // neighbouring rays of a picture share cells. One 800 x 800 picture of a 256^3 grid in
  // groups of 1 / 8 / 32 / 128: 976 / 792 / 776 / 797 us, three of 400 x 400: 678 / 648 / 677
  // / 676 us, half transparent 1913 / 1625 / 1630 / 1635 us.
  RenderArgs<Real> b = a;
  while (b.group_log2 < 3 && (a.R >> (b.group_log2 + 1)) >= 32 * blocks) ++b.group_log2;
  // From five rays per warp on, every other warp begins with the clear, up to three quarters of
  // it: the other warps' atomics leave HBM idle meanwhile, and hundreds of MB behind the last ray
  // overlap with nothing. Only behind / three quarters early / all early, us: half-transparent
  // trilinear steps, 256^3, 20,000 rays x 200 597 / 586 / 582, 400^3, 65,536 x 300 3280 / 3223 /
  // 3211; 512^3 log-sum, 65,536 x 512 337 / 323 / 327; opaque 320^3, 40,000 x 256 103.6 / 104.1 /
  // 106.6. With a round before every ray instead, inlined in the loop, every launch lost 2 %.
  b.clear_early = a.clear_words > 0 && a.R >= 5 * blocks * kWarpsPerBlock ? 1 : 0;
  render_kernel<Real, Store, MODE, K, PHASE, LOGT, A><<<(unsigned)blocks, kThreads, kSmem, s>>>(b);
  return after_launch();
}

template <typename Real, typename Store, int MODE, int PHASE, bool LOGT, int A>
int launch_render_mp(const RenderArgs<Real>& a, cudaStream_t s) {
  const bool early_stop = a.g.clip && !(PHASE == kTrain && a.beta_w != 0.0);
  RenderArgs<Real> b = a;
  b.long_ray = MODE == PGB_NEAREST && !early_stop && a.S > 128;
  const bool long_chunks = !early_stop && a.term_thr > 0.0f;
  switch (pick_slots(a.S, a.chunk_samples, MODE, long_chunks)) {
    case 1: return launch_render_k<Real, Store, MODE, 1, PHASE, LOGT, A>(b, s);
    case 2: return launch_render_k<Real, Store, MODE, 2, PHASE, LOGT, A>(b, s);
    case 4: return launch_render_k<Real, Store, MODE, 4, PHASE, LOGT, A>(b, s);
    case 8: return launch_render_k<Real, Store, MODE, 8, PHASE, LOGT, A>(b, s);
    case 16: return launch_render_k<Real, Store, MODE, 16, PHASE, LOGT, A>(b, s);
    default: return PGB_ERR_UNSUPPORTED;
  }
}

// A: kQuick for the fp32 grids of quick_grid, kGeneral for all others and for fp64. Both have
// every chunk size: chunk_samples and the threshold on T mean the same on any grid. Origin (0,
// 0, 0) against the same grid centred, us, general / quick (one general kernel of 256-sample
// chunks for all took the figure behind): 256^3, 8192 rays x 256 trilinear step 102 / 99 (198);
// 512^3 BF16 log-sum step of 65,536 rays 279 / 277 (1897); nearest, 7500 x 600 62 / 57 (102);
// 160,000 rays x 256 forward, trilinear 304 / 300 (1139), nearest 260 / 253 (332).
template <typename Real, typename Store, bool LOGT, int A>
int launch_render_t(const RenderArgs<Real>& a, int mode, int phase, cudaStream_t s) {
  if (mode == PGB_NEAREST) {
    if (phase == kForward) return launch_render_mp<Real, Store, PGB_NEAREST, kForward, LOGT, A>(a, s);
    if (phase == kBackward) return launch_render_mp<Real, Store, PGB_NEAREST, kBackward, LOGT, A>(a, s);
    if (phase == kTrain) return launch_render_mp<Real, Store, PGB_NEAREST, kTrain, LOGT, A>(a, s);
  } else if (mode == PGB_TRILINEAR) {
    if (phase == kForward) return launch_render_mp<Real, Store, PGB_TRILINEAR, kForward, LOGT, A>(a, s);
    if (phase == kBackward) return launch_render_mp<Real, Store, PGB_TRILINEAR, kBackward, LOGT, A>(a, s);
    if (phase == kTrain) return launch_render_mp<Real, Store, PGB_TRILINEAR, kTrain, LOGT, A>(a, s);
  }
  return PGB_ERR_ARG;
}

}  // namespace pgb
