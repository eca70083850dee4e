// Device side of the engine: context, device buffers and the launchers of
// the linking-number kernels (direct sum: direct.cu; Barnes–Hut: bh.cu).
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <functional>
#include <map>
#include <mutex>
#include <utility>
#include <string>
#include <vector>

#include "host.hpp"

namespace fln {

#define FLN_CUDA(call)                                                                      \
  do {                                                                                      \
    cudaError_t e_ = (call);                                                                \
    if (e_ != cudaSuccess)                                                                  \
      throw ::fln::Error(e_ == cudaErrorMemoryAllocation ? FLN_ERR_OUT_OF_MEMORY : FLN_ERR_CUDA, \
                         std::string(#call) + ": " + cudaGetErrorString(e_));              \
  } while (0)

// Grow-only device buffer. It grows with some room to spare (an eighth, at
// most 256 MB, where there is memory for it), so that calls of about the same
// size do not each free and allocate it again.
struct DevBuf {
  void *ptr = nullptr;
  size_t bytes = 0;
  void *need(size_t n) {
    if (n > bytes) {
      if (ptr) cudaFree(ptr);
      ptr = nullptr;
      bytes = 0;
      size_t want = n + std::min(n / 8, size_t(256) << 20);
      if (cudaMalloc(&ptr, want) != cudaSuccess) {
        cudaGetLastError();
        ptr = nullptr;
        want = n;
        FLN_CUDA(cudaMalloc(&ptr, want));
      }
      bytes = want;
    }
    return ptr;
  }
  template <class T>
  T *as(size_t count) {
    return static_cast<T *>(need(count * sizeof(T) + 16));
  }
  void release() {
    if (ptr) cudaFree(ptr);
    ptr = nullptr;
    bytes = 0;
  }
};

// Grow-only pinned host buffer (for the host-array entry points).
struct HostBuf {
  void *ptr = nullptr;
  size_t bytes = 0;
  void *need(size_t n) {
    if (n > bytes) {
      if (ptr) cudaFreeHost(ptr);
      ptr = nullptr;
      bytes = 0;
      FLN_CUDA(cudaMallocHost(&ptr, n));
      bytes = n;
    }
    return ptr;
  }
  ~HostBuf() {
    if (ptr) cudaFreeHost(ptr);
  }
};

// Learned opening criterion of the Barnes–Hut traversal (learned.cuh has the
// weight layout; frag == nullptr: off).
struct MlpFrag;
struct LearnedCfg {
  const MlpFrag *frag;  // device copy of the packed BF16 weights
  float s_min;          // candidates: separation |dr| / (r1 + r2) at least this
  float log10_tau;      // accept when the predicted log10 error is below this (at beta0)
  int32_t min_cand;     // run the MLP only when a warp step has at least this many candidates
  int32_t min_seg;      // candidates: the smaller node holds at least this many segments
};

// Sampling of node pairs for training, during the first Barnes–Hut pass
// (rec == nullptr: off). Pairs are (slot, node 1, node 2, 0).
struct Recording {
  int4 *rec = nullptr;
  unsigned long long *count = nullptr;
  int64_t cap = 0;
  float s_min = 0.f;
  uint32_t keep = 0;  // keep a candidate when its 32-bit hash is below this
};

struct Context {
  int device = 0;
  cudaStream_t stream = nullptr;
  bool own_stream = false;
  int num_sms = 0;
  cudaEvent_t ev0 = nullptr, ev1 = nullptr, ev2 = nullptr, ev3 = nullptr;
  fln_stats stats{};
  // Device buffers.
  DevBuf d_xyz, d_off, d_pairs, d_loops, d_items, d_partial, d_counter, d_lk, d_err, d_flags, d_near, d_redo;
  DevBuf d_bh[28];
  size_t bh_front_guess = 0;  // the most records a call's size has asked for
  int64_t bh_front_hint = 0;  // frontier records of the largest Barnes–Hut first pass so far
  // CTAs per SM of the traversal kernels (per occupancy set), of the learned
  // traversal and of bh_classify; 0 until first queried.
  int bh_per_sm[3] = {0, 0, 0};
  int bh_per_sm_learned = 0, bh_per_sm_classify = 0;
  bool bh_build_smem = false;  // the tree build's shared memory size is set
  HostBuf h_in, h_out;  // pinned staging of copy_h2d / copy_d2h
  HostBuf h_call, h_head;  // pinned: a small call's inputs and results; the head of a direct sum's plan
  int64_t direct_items = 0;  // room for a direct sum's items (the largest call so far)
  cudaEvent_t ev_stage[2] = {nullptr, nullptr};
  // The exact-list launches of the fused Barnes–Hut rounds run on their own
  // stream, beside the next round's traversal; ev_round holds an event pair
  // around each (grown on demand, kept for later calls).
  cudaStream_t exact_stream = nullptr;
  std::vector<cudaEvent_t> ev_round;
  // Vertices from host arrays arrive in pieces on a copy stream (split at
  // loop boundaries); the Barnes–Hut tree build of each piece's loops waits
  // only for its piece. xyz_pieces = 0: the vertices are resident.
  static constexpr int kXyzPieces = 8;
  cudaStream_t copy_stream = nullptr;
  cudaEvent_t ev_piece[kXyzPieces] = {};
  cudaEvent_t ev_before_copy = nullptr;
  int64_t xyz_piece_end[kXyzPieces] = {};  // vertex index at which each piece ends
  int xyz_pieces = 0;
  // Learned criterion in use on this context, and training buffers.
  DevBuf d_mlp, d_learn[8];
  // Device Discretize (discretize.cu).
  DevBuf d_disc[37];
  LearnedCfg learned{nullptr, 0.f, 0.f, 0};
  Recording recording;

  explicit Context(int dev, void *user_stream);
  // Device time between two events recorded around launches on `stream`.
  float elapsed(cudaEvent_t a, cudaEvent_t b) {
    float ms = 0.f;
    cudaEventSynchronize(b);
    cudaEventElapsedTime(&ms, a, b);
    return ms;
  }
  ~Context();
};

// The context's stream waits for every piece of the vertices still on its
// way (Context::xyz_pieces); afterwards they are resident.
inline void wait_xyz_pieces(Context &c) {
  for (int i = 0; i < c.xyz_pieces; ++i) cudaStreamWaitEvent(c.stream, c.ev_piece[i], 0);
  c.xyz_pieces = 0;
}

// Resident CTAs per SM of `kernel` at `block` threads (at least 1), asked of
// the driver once per kernel and block size: the library is built for one
// architecture, and a driver query on every call costs host time while the
// GPU waits.
inline int occupancy_of(const void *kernel, int block) {
  static std::mutex mu;
  static std::map<std::pair<const void *, int>, int> cache;
  std::lock_guard<std::mutex> lock(mu);
  const auto key = std::make_pair(kernel, block);
  auto it = cache.find(key);
  if (it != cache.end()) return it->second;
  int n = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, block, 0) != cudaSuccess) {
    cudaGetLastError();
    return 1;
  }
  return cache[key] = std::max(n, 1);
}

// Mixed direct sum: a segment pair whose closest endpoint distance is below
// this multiple of the longer segment's length is evaluated in FP64 (the
// default of fln_params.near_factor, and the factor of the allocation-free
// entry point).
constexpr double kDefaultNearFactor = 4.0;
// Barnes–Hut round budget (traversal steps a warp spends on a batch per
// launch) when fln_params.bh_budget is 0: on the polymer step with the exact
// list, 128 ran the traversal in 48.0 ms against 49.6 ms at 256.
constexpr int kDefaultBhBudget = 128;
constexpr int kDefaultBhCtas = 6;  // fln_params.bh_occupancy 0

// Plans (on the device) and runs the direct sum over `npairs` pairs of the
// loops in device memory; everything but the returned counts stays there.
// Checks the offsets and pairs; throws FLN_ERR_INVALID_ARGUMENT before any sum
// is written when they are bad. margin >= 0: pairs whose distance to the
// rounding boundary is below it, or which are not finite, are recomputed in
// FP64 (FLN_PAIR_FP64_RECOMPUTED). Of an FP64 sum, pairs whose products leave
// the kernel's range are summed again by the wide kernel (wide: all pairs are,
// at once). d_err and d_flags may be null; they get 0
// otherwise. tile_shape: index into the direct sum's tile shapes
// (fln_params.direct_tile).
struct DirectResult {
  int launches = 0;
  double near_terms = 0;  // mixed: segment pairs evaluated in FP64
  double work = 0;        // sum over pairs of n_i n_j
  int64_t redone = 0;     // pairs recomputed in FP64
  bool complete = false;  // the tail's event and copy are done (no pair was recomputed)
};
// What a caller wants at the end of a call without recomputed pairs, before
// the call's one host wait: an event, and the results copied to the host.
struct DirectTail {
  cudaEvent_t end;
  void *h_dst = nullptr;  // pinned
  const void *d_src = nullptr;
  size_t bytes = 0;
  int64_t known_longest = 0;  // of one pair: segments of its longer loop where the host knows it
};
constexpr int kDirectTileShapes = 6;
DirectResult direct_sum_device(Context &ctx, const double *d_xyz, const int64_t *d_off, int32_t nloops,
                               const int32_t *d_pairs, int64_t npairs, int precision, double near_factor,
                               double margin, double *d_lk, double *d_err, int32_t *d_flags, int tile_shape = 0,
                               const DirectTail *tail = nullptr, bool wide = false);

// FP64 direct sums of the n pairs in d_list (indices into d_pairs), written
// back to d_lk; d_flags (may be null) gets FLN_PAIR_FP64_RECOMPUTED there.
int recompute_pairs(Context &ctx, const double *d_xyz, const int64_t *d_off, int32_t nloops, const int32_t *d_pairs,
                    const int32_t *d_list, int64_t n, double *d_lk, int32_t *d_flags);

// Barnes–Hut over the same inputs; err per pair after ERROR_EST_SCALE and the
// reference's beta retry; flags (may be null) gets FLN_PAIR_BETA_RETRIED and
// FLN_PAIR_BETA_ESCALATED. Pairs that fail the margin check (prm.fp64_margin)
// or whose estimate stays above prm.bh_err_limit are recomputed in FP64 direct
// sum. d_pairs: the pairs on the device. Returns launches.
int barnes_hut_device(Context &ctx, const double *d_xyz, const int64_t *d_off, const std::vector<int64_t> &h_off,
                      const std::vector<int32_t> &h_pairs, const int32_t *d_pairs, const fln_params &prm,
                      double *d_lk_out, double *d_err_out, int32_t *d_flags_out);

// Runs the Barnes–Hut stage (curve-order trees, beta0, learned criterion off)
// while sampling node pairs with separation in [s_min, 1.25 beta0] (opened
// pairs and far-field pairs near the threshold; a fraction `keep` of them by
// a hash of (pair, node, node), lowered and rerun until at most `cap` are
// recorded), then computes for each sample its features (learned.cuh) and
// the log10 of the true far-field error: |multipole value - FP64 exact sum
// over the two nodes' segment ranges| + 1e-14. Samples whose ranges hold more
// than max_terms segment pairs are dropped. X gets 8 floats per sample, T the
// target, S the separation, E log10 of the Eq. 14 estimate x err_scale (the
// reference's error measure for the same pair).
void learned_collect(Context &ctx, const double *d_xyz, const int64_t *d_off, const std::vector<int64_t> &h_off,
                     const std::vector<int32_t> &h_pairs, const fln_params &prm, float s_min, double keep,
                     int64_t cap, int64_t max_terms, std::vector<float> &X, std::vector<float> &T,
                     std::vector<float> &S, std::vector<float> &E, int64_t *recorded);

// Training of the MLP on (X, T): pinball loss at quantile q, Adam, our own
// kernels (learned.cu), on the rows idx_train. params holds kMlpParams FP32
// values (initialised by the caller) and is updated; returns the mean loss of
// the last epoch.
struct TrainOptions {
  int epochs = 40;
  int batch = 4096;
  float lr = 2e-3f;
  float quantile = 0.9f;
  uint64_t seed = 1;
};
double learned_train(Context &ctx, const std::vector<float> &X, const std::vector<float> &T,
                     const std::vector<int32_t> &idx_train, const TrainOptions &opt, std::vector<float> &params);
// FP32 (mma = 0) or BF16 warp-MMA (mma = 1, the traversal's path) predictions.
void learned_predict(Context &ctx, const float *params, const float *X, int64_t n, int mma, float *Y);
// Mean pinball loss and its gradient (d loss / d params) at params.
double learned_gradients(Context &ctx, const float *params, const float *X, const float *T, int64_t n, float q,
                         float *grad);
// Discretize (discretize.cpp:103-281) and the potential-link searches before
// and after it, on the GPU: the same closed polylines (CSR offsets, xyz) and
// sorted unique pairs (i < j) as the host path, bit for bit; rounds = the
// refinement rounds run. Throws Error on the reference's failure conditions.
// bcc_f32: the same control points as float32 (curves in order, 3 per
// point), or nullptr; when given they are uploaded as such and widened on the
// device (the same doubles, half the copy).
//
// The polylines stay on the device (DiscretizedOnDevice) until the next call
// or release_discretized; copy_polylines brings them to the host.
struct DiscretizedOnDevice {
  const double *d_xyz = nullptr;
  const int64_t *d_off = nullptr;
};
DiscretizedOnDevice discretize_device(Context &ctx, const std::vector<CurveData> &curves, const float *bcc_f32,
                                      std::vector<int64_t> &offsets, std::vector<int32_t> &pairs, int32_t &rounds);
// Copies n doubles to `xyz` on `stream` (see copy_d2h).
void copy_polylines(Context &ctx, cudaStream_t stream, const double *d_xyz, size_t n, DoubleArray &xyz,
                    bool all_threads);
// Gives the polylines' buffers back when they are large.
void release_discretized(Context &ctx);

// Host<->device copies on ctx.stream that return when the data has arrived.
// Pinned host memory is copied directly; pageable memory goes in 64 MB
// chunks through two pinned buffers, the host side by all threads (a single
// pageable DMA copy runs at a few GB/s, slower still into fresh pages).
void copy_h2d(Context &ctx, void *d_dst, const void *h_src, size_t bytes);
void copy_d2h(Context &ctx, cudaStream_t stream, void *h_dst, const void *d_src, size_t bytes, bool all_threads);
// The same for data that is formed on the way: fill(dst, offset, len) writes
// bytes [offset, offset + len) of it.
void fill_h2d(Context &ctx, void *d_dst, size_t bytes, const std::function<void(char *, size_t, size_t)> &fill);
// memcpy by all host threads.
void parallel_memcpy(void *dst, const void *src, size_t bytes);

// Packs params into the context's device weights and enables the criterion.
void learned_enable(Context &ctx, const float *params, float s_min, float log10_tau, int32_t min_cand,
                    int32_t min_seg);

}  // namespace fln
