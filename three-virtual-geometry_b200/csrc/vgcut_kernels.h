// Host-callable launchers of the cut engine's kernels (vgcut_kernels.cu).
#pragma once

#include <cuda_runtime.h>

#include "vgcut_internal.h"

namespace vgc {

// Resident 128-thread blocks per SM of the instance / chunk kernels (their persistent grid size); multi: the
// variants of a multi-scene launch.
cudaError_t configure_select(bool multi, int *instances_per_sm, int *chunks_per_sm);
// What the first kernel of a launch sequence reads from pinned host memory: the view constants (null: `views` on the
// device already holds them), the HZB plan (16-byte vectors) and a multi-scene launch's scene table (words).
struct LaunchInputs {
  const ViewConst *views = nullptr;
  const uint4 *plan_src = nullptr;
  uint4 *plan_dst = nullptr;
  uint32_t plan_vecs = 0, scene_words = 0;
  const uint32_t *scenes_src = nullptr;
  uint32_t *scenes_dst = nullptr;
};
// ctl: the sequence's control words (kLaunchCtlWords, cleared here): [0] visible units, [1..2] a view redoes a cut in round
// 1..2, [4..5] the work queue's 64-bit counter (spans low, chunks high), [6..7] the most spans / chunks any pass asked for,
// [8] the next chunk, [9] the next instance unit, [10] a unit's items did not fit the queue, [11] the next overflow word,
// [12] a wait of k_retry gave up, [16] k_retry's phase and from [17] the phases' counters of its two rounds
cudaError_t launch_reset(const LaunchInputs &in, ViewConst *views, uint32_t nviews, uint32_t *ctl, cudaStream_t st,
                         bool plain = false);
// plain: launched without programmatic serialization (launch_after).
// Scene arguments: a launch over one context passes its Scene and scenes = nullptr; a multi-scene launch passes
// a device table of Scene records that each view's `scene` indexes (S is then unused).
cudaError_t launch_cells(const Scene &S, const Scene *scenes, const ViewConst *views, uint32_t nviews,
                         uint32_t total_units, uint2 *units, uint32_t *unit_count, cudaStream_t st,
                         bool plain = false);
// round < 0: the triangleBudget search's histogram pass (k_instances / k_chunks), then launch_budget picks the
// threshold of each budget view.
cudaError_t launch_budget(const ViewConst *views, uint32_t nviews, uint32_t *ctl, cudaStream_t st, bool plain = false);
// lim: how the pass may be cut up (the same for a pass's instances and redo launches; default 512 meshlets per chunk).
// overflow: a bit per warp-unit (4 per unit of `units`), zero between passes: k_instances marks the units whose
// items did not fit the queue, and launch_instances_redo (after launch_chunks of the same pass) tests their items
// in place and clears the bits.
cudaError_t launch_instances(const Scene &S, const Scene *scenes, const ViewConst *views, const uint2 *units,
                             uint32_t *ctl, uint4 *queue, uint32_t capacity, int round, uint32_t grid,
                             uint32_t *overflow, cudaStream_t st, const PassLimits &lim = PassLimits(),
                             bool plain = false);
cudaError_t launch_instances_redo(const Scene &S, const Scene *scenes, const ViewConst *views, const uint2 *units,
                                  uint32_t *ctl, uint4 *queue, uint32_t capacity, int round, uint32_t *overflow,
                                  uint32_t grid, cudaStream_t st, const PassLimits &lim = PassLimits(),
                                  bool plain = false);
// The meshlet work queue (spans and chunks) lives in `queue`, `capacity` uint4 entries; ctl[4..5] counts it.
cudaError_t launch_chunks(const Scene &S, const Scene *scenes, const ViewConst *views, uint4 *queue,
                          uint32_t *ctl, uint32_t capacity, int round, uint32_t grid, cudaStream_t st,
                          bool plain = false);
// computeCell on the device for n cells from c0 of one mesh (bit-identical to the host's computation).
cudaError_t launch_cells_update(const float4 *inst, const double sphere[4], uint32_t instance_base,
                                uint32_t instance_count, uint32_t cell_base, uint32_t slot, uint32_t c0, uint32_t n,
                                CellRec *cells, cudaStream_t st);
// host_ctl (optional, pinned): receives control words 6 and 7, the peak queue demand of the sequence so far.
cudaError_t launch_finish(const ViewConst *views, uint32_t nviews, uint32_t *ctl, int round, uint32_t *host_ctl,
                          cudaStream_t st, bool plain = false);
// Rounds 1 and 2 of the cuts that overflowed in one kernel (returns at once when none did), after launch_finish.
cudaError_t launch_retry(const Scene &S, const Scene *scenes, const ViewConst *views, uint32_t nviews,
                         const uint2 *units, uint32_t *ctl, uint4 *queue, uint32_t capacity, uint32_t *overflow,
                         uint32_t *host_ctl, uint32_t grid, cudaStream_t st, const PassLimits &lim = PassLimits(),
                         bool plain = false);
struct ExpandView {  // what index expansion reads of an output slot
  const uint32_t *counters;
  const uint4 *draw_list;
  uint32_t max_drawn;
};
cudaError_t launch_expand(const Scene &S, const ExpandView &view, uint32_t cut, uint32_t *out, uint64_t capacity,
                          uint32_t grid, cudaStream_t st);
cudaError_t launch_hzb(const float *depth, const HzbDesc &H, float *out, int copy_mip0, cudaStream_t st);
// HZB builds of the views whose constants carry build_hzb (grid covers the largest depth image).
cudaError_t launch_hzb_views(const ViewConst *views, uint32_t nviews, uint32_t max_w,
                             uint32_t max_h, bool tail, cudaStream_t st);
// The same builds as one stream of strips (k_hzb_stream, levels 0..4) from the launch's HZB plan in device memory;
// `grid` blocks (hzb_stream_blocks_per_sm() per SM), then the tail kernel for levels 5+ when `tail`.
cudaError_t launch_hzb_stream(const unsigned char *plan, uint32_t grid, const ViewConst *views, uint32_t nviews,
                              bool tail, cudaStream_t st);
// k_retry of one view in the last phase of round 1, whose one piece is taken already: it waits for `limit_ns` and leaves a
// fault in the view's counters. ctl (kLaunchCtlWords) is overwritten first.
cudaError_t launch_retry_probe(const ViewConst *view, uint32_t *ctl, uint32_t *overflow, uint32_t *host_ctl,
                               uint64_t limit_ns, cudaStream_t st);
// The bounded mbarrier wait of the strip stream on a barrier nothing completes (out[0]: completed, out[1]: ns waited).
cudaError_t launch_wait_probe(uint64_t limit_ns, unsigned long long *out, cudaStream_t st);
// Blocks of k_hzb_stream resident per SM (sets its shared-memory limit on the first call for the current device).
uint32_t hzb_stream_blocks_per_sm();
cudaError_t launch_select_cut(const Scene &S, uint32_t slot, uint32_t mcount, uint32_t count, const float *vm16,
                              const float *params, float threshold, float blend, uint8_t *lo, uint8_t *hi, cudaStream_t st);

}  // namespace vgc
