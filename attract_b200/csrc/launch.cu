// Launches of the scoring kernels (score.cu): the kernel of a launch, its
// shared memory and occupancy, and the kernels' error words.
#include <mutex>

#include "score_parts.h"

namespace att {

static const void* kernel_of(int mode, int S, int K, bool one_grid, bool chunked) {
  switch (mode) {
    case MODE_EVAL:
    case MODE_EVAL_MAT: return score_part_kernel<0>(mode, S, K, one_grid, chunked);
    case MODE_MIN: return score_part_kernel<1>(mode, S, K, one_grid, chunked);
    case MODE_BWD: return score_part_kernel<2>(mode, S, K, one_grid, chunked);
    case MODE_QUAT: return score_part_kernel<3>(mode, S, K, one_grid, chunked);
  }
  return nullptr;
}

int beads_per_lane(int S, int max_beads) {
  const int need = (max_beads + S - 1) / S;
  int K = 1;
  while (K < need) K <<= 1;
  return K <= ATT_MAX_BEADS_PER_LANE ? K : ATT_MAX_BEADS_PER_LANE;  // larger ligands run in chunks
}

// A minimiser keeps every bead's brick and record in shared memory from step to
// step, so its lanes hold all of a ligand's beads.  A single evaluation copies each
// once whatever its chunk: one bead per lane leaves room for 24 warps per SM at 32 lanes, 20 at
// 8 and 16 (5 blocks; at 32 lanes too with 128-byte records) where 2, 4 and 8 beads per lane
// left 16, 8 and 4, to cover the copies' latency.  energrad, before and now: 32 lanes: 40 beads,
// 20 000 poses 78 -> 69 us; 100 beads, 8000 poses 97 -> 65; 200 beads, 5000 poses
// 191 -> 76; 301 beads, 3000 matrices 184 -> 64; the adjoint of 100 beads, 8000 poses
// 129 -> 105.  16 lanes, 30 000 poses: 24 beads 91 -> 60 us, 60 beads 224 -> 112; 8 lanes: 24 beads
// 108 -> 55, 60 beads 345 -> 116, 100 beads 503 -> 175.  (Few poses: split_poses.)  One rule for all
// sizes keeps a pose's energy the same to the bit in any batch.
int mode_beads_per_lane(int mode, int S, int max_beads) {
  return mode == MODE_MIN || mode == MODE_QUAT ? beads_per_lane(S, max_beads) : 1;
}

// Whether the four warps of a block share each tile of poses, a quarter of the chunks each:
// from three chunks on, while the blocks are at most two waves (6 blocks per SM at 32 lanes, 5 at 8 and
// 16), where a warp's chunks one after another are the launch's time.  energrad, one warp per
// tile against four, without the host's time: 32 lanes: 301 beads, 300 poses 34.3 -> 14.4 us, 1500
// 44.7 -> 36.7, 3000 60.2 -> 62.2; 100 beads, 300 poses 15.8 -> 7.8, 2000 22.8 -> 22.1.  16 lanes (two poses
// per tile): 100 beads, 600 poses 25.7 -> 11.6, 2400 28.7 -> 24.8, 3000 32.1 -> 31.6; 40 beads, 3000 16.7 -> 18.6.
// 8 lanes (four poses): 40 beads, 1200 poses 21.0 -> 11.5, 4800 23.9 -> 24.0, 6000 26.5 -> 29.5; 301 beads,
// 1200 130 -> 42.  Two chunks leave two warps idle (32 lanes: 40 beads, 2200 poses 17.0 -> 20.5).
// The sums are the same to the bit.
bool split_poses(int mode, int S, int threads, int max_beads, int n_tiles) {
  if (mode == MODE_MIN || mode == MODE_QUAT || threads != 128 || max_beads <= 2 * S) return false;
  int dev = 0, sms = 148;
  if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  return n_tiles <= sms * (S == 32 ? 6 : 5) * 2;
}

size_t score_smem_bytes(int K, int threads, int rec_slot) {
  return warp_smem_bytes(K, rec_slot) * (size_t)(threads / 32);
}

// the shared memory of one block of `mode` (without bead arms unless the mode
// accumulates dE/dmat)
static size_t mode_smem_bytes(int mode, int K, int threads, int rec_slot) {
  const bool arms = mode == MODE_EVAL_MAT || mode == MODE_QUAT;
  return warp_smem_bytes(K, rec_slot, arms) * (size_t)(threads / 32);
}

// lets a kernel use `bytes` of dynamic shared memory; 48 KB need no leave (a
// driver call less for small launches)
static cudaError_t allow_smem(const void* k, size_t bytes) {
  return bytes <= 48 * 1024 ? cudaSuccess
                            : cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
}

static cudaError_t launch_one(const KParams& p, int mode, int S, int K, bool one_grid, int blocks, int threads,
                              cudaStream_t st) {
  const void* k = kernel_of(mode, S, K, one_grid, p.max_beads > S * K);
  if (k == nullptr) return cudaErrorInvalidValue;
  const size_t smem = mode_smem_bytes(mode, K, threads, p.rec_slot);
  cudaError_t e = allow_smem(k, smem);
  if (e == cudaSuccess && p.counter != nullptr) e = cudaMemsetAsync(p.counter, 0, sizeof(int), st);
  if (e != cudaSuccess) return e;
  void* args[] = {const_cast<KParams*>(&p)};
  return cudaLaunchKernel(k, dim3(blocks), dim3(threads), args, smem, st);
}

// Side streams of launch_side_by_side.  To make and destroy one costs the host 110 us, so up to
// KEPT of them stay for later calls (in any thread).  A call takes one only when its work is done and makes
// another otherwise: no caller's stream ever waits for another's.  They belong to a context; its id is never
// used twice, so streams of one that was reset are not touched again.
struct SideStream {
  cudaStream_t stream;
  unsigned long long ctx;
  int priority;
};
struct SideStreams {
  static constexpr int KEPT = 8;
  std::mutex mutex;
  SideStream kept[KEPT];
  int n = 0;
};
static SideStreams g_side_streams;  // (for the process: no CUDA call at its exit)

static unsigned long long context_id() {  // 0: not to be had
  typedef int (*CtxGetId)(void*, unsigned long long*);
  static const CtxGetId fn = [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) != cudaSuccess ||
        q != cudaDriverEntryPointSuccess)
      f = nullptr;
    return reinterpret_cast<CtxGetId>(f);
  }();
  unsigned long long id = 0;
  return fn != nullptr && fn(nullptr, &id) == 0 ? id : 0;
}

static cudaError_t take_side_stream(unsigned long long ctx, int priority, cudaStream_t* out) {
  if (ctx != 0) {
    SideStreams& s = g_side_streams;
    std::lock_guard<std::mutex> lock(s.mutex);
    for (int i = 0; i < s.n; ++i)
      if (s.kept[i].ctx == ctx && s.kept[i].priority == priority) {
        const cudaError_t e = cudaStreamQuery(s.kept[i].stream);
        if (e == cudaErrorNotReady) {
          cudaGetLastError();
        } else {
          *out = s.kept[i].stream;
          s.kept[i] = s.kept[--s.n];
          return e;
        }
      }
  }
  return cudaStreamCreateWithPriority(out, cudaStreamNonBlocking, priority);
}
static void give_side_stream(unsigned long long ctx, int priority, cudaStream_t stream) {
  if (ctx != 0) {
    SideStreams& s = g_side_streams;
    std::lock_guard<std::mutex> lock(s.mutex);
    if (s.n < SideStreams::KEPT) {
      s.kept[s.n++] = {stream, ctx, priority};
      return;
    }
  }
  cudaStreamDestroy(stream);  // (freed when its work is done)
}

// The launches of one call, one per grid, side by side: each skips the other grids'
// segments and takes its tiles statically, so that blocks without a tile of its grid end at once.
// One after another each would end with a tail of its own.  Up to SIDE_STREAMS side streams,
// between two events of the caller's stream, take the grids in turn with it.  In a stream that is
// being captured the launches become branches of the graph.  50 steps of 40 beads, one after
// another and now: 2 grids x 500 poses 0.56 -> 0.29 ms, 8 x 500 2.41 -> 0.70, 4 x 4000 2.37 -> 2.05, 8 x 4000
// 4.75 -> 3.94; 1 step of 4 poses on each of 8 grids 0.18 -> 0.06 (0.35 with streams made for the call).
// (On an easier case 8 x 500 took 1.58 -> 0.72, 0.54 in the reference mode's one launch; 1, 2 and 7 side
// streams 0.92, 0.80 and 0.87.)
constexpr int SIDE_STREAMS = 3;
static cudaError_t launch_side_by_side(const KParams& p, int mode, int S, int K, int blocks, int threads,
                                       cudaStream_t st) {
  constexpr size_t MAX_DEPS = 64;
  KParams q = p;
  q.counter = nullptr;
  auto launch = [&](int g, cudaStream_t s) {
    q.grid[0] = p.grid[g];
    q.grid_sel = g;
    return launch_one(q, mode, S, K, true, blocks, threads, s);
  };
  cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
  const cudaGraphNode_t* deps = nullptr;
  size_t n_deps = 0;
  cudaError_t e = cudaStreamGetCaptureInfo_v2(st, &capture, nullptr, nullptr, &deps, &n_deps);
  if (e != cudaSuccess) return e;

  if (capture == cudaStreamCaptureStatusActive) {
    cudaGraphNode_t start[MAX_DEPS], ends[MAX_DEPS];
    const size_t n_start = n_deps;
    const bool branches = n_deps <= MAX_DEPS;  // (else one after another)
    for (size_t i = 0; branches && i < n_start; ++i) start[i] = deps[i];
    size_t n_ends = 0;
    for (int g = 0; g < p.n_grids; ++g) {
      if (branches && g > 0) {
        e = cudaStreamUpdateCaptureDependencies(st, start, n_start, cudaStreamSetCaptureDependencies);
        if (e != cudaSuccess) return e;
      }
      e = launch(g, st);
      if (e != cudaSuccess) return e;
      if (branches) {  // the branch's node
        e = cudaStreamGetCaptureInfo_v2(st, &capture, nullptr, nullptr, &deps, &n_deps);
        if (e != cudaSuccess) return e;
        for (size_t i = 0; i < n_deps && n_ends < MAX_DEPS; ++i) ends[n_ends++] = deps[i];
      }
    }
    return branches ? cudaStreamUpdateCaptureDependencies(st, ends, n_ends, cudaStreamSetCaptureDependencies)
                    : cudaSuccess;
  }

  cudaStream_t side[SIDE_STREAMS] = {};
  cudaEvent_t event = nullptr;
  int priority = 0, n_side = 0;
  const unsigned long long ctx = context_id();
  // (another thread may be capturing: nothing here touches its stream)
  cudaStreamCaptureMode mode_before = cudaStreamCaptureModeRelaxed;
  e = cudaThreadExchangeStreamCaptureMode(&mode_before);
  if (e != cudaSuccess) return e;
  e = cudaStreamGetPriority(st, &priority);
  if (e == cudaSuccess) e = cudaEventCreateWithFlags(&event, cudaEventDisableTiming);
  if (e == cudaSuccess) e = cudaEventRecord(event, st);
  for (int g = 0; g < p.n_grids && e == cudaSuccess; ++g) {
    const int lane = g % (SIDE_STREAMS + 1);  // 0: the caller's stream
    if (lane == n_side + 1) {
      if (take_side_stream(ctx, priority, &side[n_side]) == cudaSuccess) {
        e = cudaStreamWaitEvent(side[n_side], event, 0);
        ++n_side;
      } else {
        cudaGetLastError();  // none to be had: behind the others
      }
    }
    if (e == cudaSuccess) e = launch(g, lane > 0 && lane <= n_side ? side[lane - 1] : st);
  }
  for (int i = 0; i < n_side; ++i) {  // the caller's stream waits for them, whatever became of a launch
    const cudaError_t e1 = cudaEventRecord(event, side[i]), e2 = cudaStreamWaitEvent(st, event, 0);
    if (e == cudaSuccess) e = e1 != cudaSuccess ? e1 : e2;
  }
  for (int i = 0; i < n_side; ++i) give_side_stream(ctx, priority, side[i]);
  if (event != nullptr) cudaEventDestroy(event);
  cudaThreadExchangeStreamCaptureMode(&mode_before);
  return e;
}

// One launch, but for the analytic gradient of a minimiser over several grids with
// several beads per lane: one per grid over the same tiles.  (Those kernels hold the
// reference mode only.  Compiled with both, a 32-lane, two-beads-per-lane evaluation over
// two grids reported a misaligned address in the analytic mode, where the bounds-checked
// build of the same source found every index and alignment right.)
cudaError_t launch_score(const KParams& p, int mode, int S, int K, int blocks, int threads, cudaStream_t st) {
  if (p.n_grids == 1 || K == 1 || p.grad_mode == ATT_GRAD_REFERENCE)
    return launch_one(p, mode, S, K, p.n_grids == 1, blocks, threads, st);
  // Many tiles: one after another, tiles from the counter.  Static tiles end about a wave unevenly,
  // each tail saved is worth part of one: even at 3 waves of a grid for 2 grids, 6 to 8 for 4 (50 steps of 40 beads:
  // 2 x 6000 poses 1.61 -> 1.65 ms, 2 x 20 000 4.52 -> 4.70, 4 x 10 000 4.96 -> 4.80, 4 x 20 000 9.10 -> 9.19, 8 x 10 000
  // 10.03 -> 9.36; a wave is 2368 poses here).
  if (2LL * p.n_tiles > 3LL * p.n_grids * p.n_grids * blocks * (threads / 32)) {
    KParams q = p;
    cudaError_t e = cudaSuccess;
    for (int g = 0; g < p.n_grids && e == cudaSuccess; ++g) {
      q.grid[0] = p.grid[g];
      q.grid_sel = g;
      e = launch_one(q, mode, S, K, true, blocks, threads, st);
    }
    return e;
  }
  return launch_side_by_side(p, mode, S, K, blocks, threads, st);
}

// the bits of every part's error word
cudaError_t kernel_status(int* out, int clear, cudaStream_t st) {
  int w[SCORE_PARTS] = {0};
  cudaError_t e = score_part_status<0>(&w[0], clear, st);
  if (e == cudaSuccess) e = score_part_status<1>(&w[1], clear, st);
  if (e == cudaSuccess) e = score_part_status<2>(&w[2], clear, st);
  if (e == cudaSuccess) e = score_part_status<3>(&w[3], clear, st);
  *out = 0;
  for (int i = 0; i < SCORE_PARTS; ++i) *out |= w[i];
  return e;
}

// the first failed check of the lowest part that has one
cudaError_t kernel_debug_info(unsigned long long* out3, int clear, cudaStream_t st) {
  unsigned long long w[SCORE_PARTS][3] = {};
  cudaError_t e = score_part_debug<0>(w[0], clear, st);
  if (e == cudaSuccess) e = score_part_debug<1>(w[1], clear, st);
  if (e == cudaSuccess) e = score_part_debug<2>(w[2], clear, st);
  if (e == cudaSuccess) e = score_part_debug<3>(w[3], clear, st);
  int hit = 0;
  while (hit < SCORE_PARTS - 1 && w[hit][0] == 0ull) ++hit;
  for (int k = 0; k < 3; ++k) out3[k] = w[hit][k];
  return e;
}

cudaError_t occupancy_blocks(int mode, int S, int K, int threads, int rec_slot, bool one_grid, int* blocks_per_sm) {
  const void* k = kernel_of(mode, S, K, one_grid, true);  // (the minimisers')
  if (k == nullptr) return cudaErrorInvalidValue;
  const size_t smem = mode_smem_bytes(mode, K, threads, rec_slot);
  const cudaError_t e = allow_smem(k, smem);
  if (e != cudaSuccess) return e;
  return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks_per_sm, k, threads, smem);
}

}  // namespace att
