// Direct summation of the Gauss linking integral on B200 (sm_100a).
//
// Work: every potential loop pair (i, j) is split into items: kBlockSegs
// consecutive segments of its longer loop ("curve 1") against a span of the
// other; a CTA takes items from a device work queue (an atomic counter) until it
// runs dry, so all pairs — 16-segment rings to 2^18-segment loops — run in one
// persistent launch. The items are planned on the device (plan_items), so that a
// call has one host wait. Each thread owns one or two curve-1 segments and walks
// curve-2 segments, which the CTA stages tile by tile in shared memory (coalesced
// loads, broadcast reads). Per segment pair it evaluates the
// closed-form solid-angle term of Arai 2013 as the reference does
// (src/compute_link.cpp:126-178, :200-280): with a = q_k - p_i,
// b = q_k - p_{i+1}, c = q_{k+1} - p_{i+1}, d = q_{k+1} - p_i,
//   det  = a . (b x c)
//   div1 = |a||b||c| + (a.b)|c| + (c.a)|b| + (c.b)|a|
//   div2 = |a||d||c| + (a.d)|c| + (c.a)|d| + (c.d)|a|
//   term = atan2(det (div1 + div2), div1 div2 - det^2) / 2pi
//          + [det (div1 + div2) det < 0] sign(det)          (in full turns).
// Consecutive steps share vertices: step k+1's a, b are step k's d, c, so
// each step computes two new difference vectors and two norms.
//
// Two precisions:
//  * FP64 ("plain FP64 GPU direct sum"): every operation in FP64; the per-
//    thread terms are combined by the arctangent-addition recurrence of
//    ComputeLinkingNumberDirectFast (Bertolazzi et al. 2019) — a running
//    complex product with a count of negative-x-axis crossings — and one
//    atan2 per thread per item. The product is rescaled by an exact power of
//    two every second step instead of the reference's division (range: see
//    kLeastScale).
//  * MIXED: coordinates relative to the tile's first vertex in FP32, one FP32
//    arctangent per segment pair (a series for small angles, else atan2f), FP32
//    sums over runs of 32 terms and FP64 sums above that. det uses the identity
//    det = a . (f x e) with e = p_{i+1} - p_i and f = q_{k+1} - q_k, which keeps
//    its relative accuracy for distant pairs. A segment pair whose closest
//    endpoint distance is below near_factor x (longer segment length), or below
//    kNearLeast, is evaluated in FP64 (near-singular and too small terms). FP32
//    holds a term, 64 d^6, up to distances d of 9e5 from the tile's segments.
// Item results go to one FP64 partial per item; a second kernel sums them
// per pair in a fixed order, so results are deterministic.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <mutex>
#include <numeric>
#include <string>

#include "engine.hpp"
#include "root.cuh"

namespace fln {
namespace {

constexpr int kBlockSegs = 128;  // default: threads per CTA = curve-1 segments per item
constexpr int kTile = 256;       // default: curve-2 vertices per shared-memory tile
constexpr double kInvTwoPi = 0.15915494309189533576888376337251436;

// What a call's plan and its kernels tell each other and the host.
struct PlanHead {
  unsigned long long queue;  // work queue head
  unsigned long long near;   // mixed: segment pairs evaluated in FP64
  unsigned long long items;
  unsigned long long redo;   // pairs that failed the margin check
  unsigned long long longest;  // segments of the longest loop of a pair
  double work;               // sum over pairs of n_i n_j
  int32_t status;            // kBad* bits
  int32_t pad;
};
constexpr int kSmRanks = 256;  // sm_turn: CTAs per SM that asked, and one counter for all, behind the head
constexpr int kBadStart = 1, kBadOrder = 2, kBadPair = 4, kBadSize = 8, kBadSame = 16;

struct DirectArgs {
  const double *xyz;          // 3 doubles per vertex
  const int64_t *off;         // loop offsets
  const int32_t *pairs;       // (i, j) per pair
  int64_t *start;             // per pair: its first item
  int32_t *item_pair;         // per item: its pair; null: searched in start (npairs + 1 entries)
  int32_t npairs;
  int64_t cap;                // room for items
  int64_t target;             // items a call should have at least (plan_span)
  double least;               // calls of less work (PlanHead::work) take the whole of curve 2 per item
  int block;                  // curve-1 segments per item
  int64_t few;                // mixed: most items of a call for direct_mixed_few_kernel (few_items); 0: none
  int64_t lone;               // one pair in FP64: the longest loop for direct_fp64_lone_kernel; 0: none
  PlanHead *head;
  unsigned *sm_rank;          // kSmRanks + 1 counters, 0 at first; null: the grid has no more CTAs than items
  int sms;
  double *partial;            // per item
  float near_factor;
  bool wide;                  // FP64: the kernel that forms shares out of range again (host)
};

// Curve-2 segments per item. A call whose pairs give few items of kBlockSegs
// segments is cut along curve 2 as well, so that it fills the chip and ends
// evenly: `target` items (eight per resident CTA) of about the same work, down
// to 32 segments, below which a CTA's start costs more than its terms. The
// mixed precision does so only from kMixedSpans segment pairs. That line is no
// measured one: cutting a walk regroups its FP64 sum, and below it the sums stay
// bit for bit those of one walk per segment (all there is to see when no loops
// are linked).
constexpr double kMixedSpans = 1 << 30;
// A lone pair goes to direct_fp64_lone_kernel, 32 curve-1 segments an item, when
// its items are resident at once, two CTAs per SM. The kernel is for loops that
// fill few CTAs; longer ones it takes a wave at a time. Calls by this kernel /
// the general one (one thread per segment before both): 300 x 211 segments 79 /
// 70 us (135), 5,000 x 4,286 397 / 258 (1,285), 10,000 x 8,572 1,112 / 454
// (2,487), 30,000 x 20 115 / 77 (89), 200,000 x 300 845 / 416 (536), 200,000 x 2,000
// 3,572 / 1,645 (2,914). (Below the line it stays for its sums, see there.)
constexpr int kLoneSegs = 32;
constexpr int64_t kLonePerSm = 2;
__device__ __forceinline__ bool plan_lone(const DirectArgs &A) {
  return A.lone > 0 && (int64_t)A.head->longest <= A.lone;
}
__device__ __forceinline__ int plan_block(const DirectArgs &A) { return plan_lone(A) ? kLoneSegs : A.block; }
__device__ __forceinline__ int64_t plan_span(const DirectArgs &A, double work) {
  if (work < A.least || plan_lone(A)) return int64_t(1) << 62;
  const double want = work / ((double)A.block * (double)A.target);
  int64_t span = 32;
  while ((double)span < want) span *= 2;
  return span;
}

// The pair of an item, its longer loop first, and the item's share of it.
struct Item {
  int64_t o1, n1, o2, n2;  // vertex offsets and segment counts
  int64_t first;           // first curve-1 segment
  int64_t k0, k1;          // curve-2 segments
};

__device__ __forceinline__ int find_slot(const int64_t *start, int n, int64_t item) {
  int lo = 0, hi = n;  // start[lo] <= item < start[hi]
  while (hi - lo > 1) {
    const int mid = (lo + hi) >> 1;
    if (__ldg(start + mid) <= item) lo = mid;
    else hi = mid;
  }
  return lo;
}

__device__ __forceinline__ Item item_of(const DirectArgs &A, int64_t item, int block, int64_t span) {
  const int p = A.item_pair ? A.item_pair[item] : find_slot(A.start, A.npairs, item);
  int a = A.pairs[2 * p], b = A.pairs[2 * p + 1];
  Item it;
  it.o1 = A.off[a];
  it.n1 = A.off[a + 1] - it.o1;
  it.o2 = A.off[b];
  it.n2 = A.off[b + 1] - it.o2;
  if (it.n2 > it.n1) {
    const int64_t o = it.o1, n = it.n1;
    it.o1 = it.o2;
    it.n1 = it.n2;
    it.o2 = o;
    it.n2 = n;
  }
  const int64_t x = item - A.start[p], spans = (it.n2 + span - 1) / span;
  it.first = x / spans * block;
  it.k0 = x % spans * span;
  it.k1 = min(it.n2, it.k0 + span);
  return it;
}

// The items of a valid plan that fits; 0 otherwise.
__device__ __forceinline__ int64_t plan_ready(const DirectArgs &A) {
  const int64_t n = (int64_t)A.head->items;
  return A.head->status == 0 && n <= A.cap ? n : 0;
}
// A mixed plan of few items (direct_mixed_few_kernel). Calls by the packed kernel
// / by this one:
//  - at most `most` items, the CTAs of this kernel that fit the chip at once; it
//    needs a second wave beyond (9 walks of 2,000 steps, 576 items of 592: 1.97 /
//    1.74 ms; 10 of 2,000, 720 items: 1.57 / 1.95);
//  - loops longer than those of which the packed kernel gives the runs to two
//    groups of threads (200 linked rings of 64 segments: 79 / 91 us, but 20 walks
//    of 30 steps, all pairs near: 120 / 92; 20 of 72 steps: 228 / 139);
//  - walks of curve 2 of at most 3,500 segments: longer ones meet enough near
//    pairs for the packed kernel's warps to evaluate them together (4 of 500
//    steps 0.80 / 0.49 ms; 2 of 3,000 1.15 to 1.97 / 1.42 to 1.69;
//    6 of 4,000 1.57 to 2.35 / 1.78 to 2.27; 10,000 2.08 to 2.21 / 2.48 to 2.73; two
//    stretches of 10,000 of one walk 4.26 / 8.69).
constexpr double kFewWork = 64 * 64;  // segment pairs per item, more than
constexpr double kFewMost = 128 * 3500.0;
__host__ __device__ __forceinline__ bool few_items(int64_t items, double work, int64_t most) {
  return items <= most && work < kMixedSpans && work > kFewWork * (double)items && work < kFewMost * (double)items;
}
__device__ __forceinline__ bool plan_few(const DirectArgs &A) {
  return A.few > 0 && few_items((int64_t)A.head->items, A.head->work, A.few);
}

// Whether this CTA takes items of a plan with fewer items than CTAs (thread 0
// asks): items / SMs CTAs on each SM do, and one more on as many as the
// remainder. All CTAs at the queue at once, two items often met on one SM while
// others had none (3 walks of 5,000 steps far apart, 120 items: 1.19 ms by CTA
// number, 1.01 this way). The queue hands out every item as long as one CTA takes
// part, and the first to ask does.
__device__ __forceinline__ bool sm_turn(const DirectArgs &A, int64_t items) {
  if (!A.sm_rank || items >= (int64_t)gridDim.x) return true;
  unsigned sm;
  asm volatile("mov.u32 %0, %%smid;" : "=r"(sm));
  const int64_t each = items / A.sms, rank = atomicAdd(&A.sm_rank[sm % kSmRanks], 1u);
  return rank < each || (rank == each && atomicAdd(&A.sm_rank[kSmRanks], 1u) < items % A.sms);
}

__device__ __forceinline__ double3 load_v(const double *xyz, int64_t v) {
  return make_double3(__ldg(xyz + 3 * v), __ldg(xyz + 3 * v + 1), __ldg(xyz + 3 * v + 2));
}

// Sum over the CTA of kB threads; the result is valid in thread 0.
template <int kB>
__device__ __forceinline__ double block_sum(double v, double *s_red) {
  for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0) s_red[warp] = v;
  __syncthreads();
  double r = 0;
  if (threadIdx.x == 0)
    for (int w = 0; w < kB / 32; ++w) r += s_red[w];
  return r;
}

// One segment pair in FP64, in full turns (OneArctanPerPair form,
// compute_link.cpp:151-175 divided by 4 pi).
__device__ __noinline__ double term_fp64(double3 p0, double3 p1, double3 q0, double3 q1) {
  const double ax = q0.x - p0.x, ay = q0.y - p0.y, az = q0.z - p0.z;
  const double bx = q0.x - p1.x, by = q0.y - p1.y, bz = q0.z - p1.z;
  const double cx = q1.x - p1.x, cy = q1.y - p1.y, cz = q1.z - p1.z;
  const double dx = q1.x - p0.x, dy = q1.y - p0.y, dz = q1.z - p0.z;
  const double la = sqrt(ax * ax + ay * ay + az * az), lb = sqrt(bx * bx + by * by + bz * bz);
  const double lc = sqrt(cx * cx + cy * cy + cz * cz), ld = sqrt(dx * dx + dy * dy + dz * dz);
  const double ca = cx * ax + cy * ay + cz * az;
  const double div1 = la * lb * lc + (ax * bx + ay * by + az * bz) * lc + ca * lb + (cx * bx + cy * by + cz * bz) * la;
  const double div2 = la * ld * lc + (ax * dx + ay * dy + az * dz) * lc + ca * ld + (cx * dx + cy * dy + cz * dz) * la;
  const double det = ax * (by * cz - bz * cy) + az * (bx * cy - by * cx) + ay * (bz * cx - bx * cz);
  const double xp = div1 * div2 - det * det, yp = det * (div1 + div2);
  double r = atan2(yp, xp) * kInvTwoPi;
  if (yp * det < 0) r += (det > 0) ? 1.0 : -1.0;
  return r;
}

// The term of segment q.x of curve 1 and q.y of curve 2.
__device__ __forceinline__ double near_term(const double *xyz, int64_t o1, int64_t n1, int64_t o2, int64_t n2, int2 q) {
  return term_fp64(load_v(xyz, o1 + q.x), load_v(xyz, o1 + (q.x + 1 == n1 ? 0 : q.x + 1)), load_v(xyz, o2 + q.y),
                   load_v(xyz, o2 + (q.y + 1 == n2 ? 0 : q.y + 1)));
}

// Rescales (x, y) by the power of two that brings max(|x|, |y|) into [1, 2),
// with the exponent from the integer pipe. Returns that exponent (the biased
// one, in bits 20 to 30).
__device__ __forceinline__ int renorm(double &x, double &y) {
  const int e = max(__double2hiint(x) & 0x7ff00000, __double2hiint(y) & 0x7ff00000);
  const double s = __hiloint2double(0x7fe00000 - min(e, 0x7fd00000), 0);
  x *= s;
  y *= s;
  return e;
}

// A sum of angles as a complex product (x, y) and a count of full turns (the
// arctangent addition of compute_link.cpp:245-269).
struct AngleSum {
  double x = 1.0, y = 0.0;
  int turns = 0;
  // Above the real axis or on its negative half.
  static __device__ __forceinline__ bool upper(double x, double y) { return y > 0.0 || (y == 0.0 && x < 0.0); }
  // Adds the angle of the segment-pair term (px + i py), where py = det x sum:
  // its arctangent's principal value, a turn more or less when sum < 0.
  // The product crosses the negative real axis when it changes sides while the
  // added angle has the sign of the old side (or is zero); since that angle is
  // at most half a turn, the old or the new product then lies left of the
  // imaginary axis, which is rare, so the crossing test sits in a branch.
  __device__ __forceinline__ void add(double px, double py, double det, double sum) {
    const double ny = x * py + px * y;
    const double nx = x * px - y * py;
    if (__builtin_expect((__double2hiint(x) | __double2hiint(nx) | __double2hiint(sum)) < 0, 0)) {
      if (sum < 0.0 && det != 0.0) turns += det > 0.0 ? 1 : -1;
      const bool was = upper(x, y);
      if (upper(nx, ny) != was && (was ? py >= 0.0 : py <= 0.0)) turns += was ? 1 : -1;
    }
    x = nx;
    y = ny;
  }
};

// The walk of two neighbouring segments p0 p1, p1 p2 along curve 2, at q_k:
// v_j = q_k - p_j, their norms, and the dot products of neighbours.
struct Walk2 {
  double v0x, v0y, v0z, v1x, v1y, v1z, v2x, v2y, v2z;
  double L0, L1, L2, ab0, ab1;
};
struct __align__(16) TileVertex {  // a curve-2 vertex q and f = next vertex - q: three 16-byte loads
  double2 q01, q2f0, f12;
};
struct Segs2 {
  double3 p0, p1, p2, e0, e1;  // e_j = p_{j+1} - p_j
};

constexpr double kTiny = 1e-300;  // keeps root() away from 0 when two vertices coincide
__device__ __forceinline__ void walk_to(const Segs2 &S, const TileVertex &t, Walk2 &w) {
  const double qx = t.q01.x, qy = t.q01.y, qz = t.q2f0.x;
  w.v0x = qx - S.p0.x; w.v0y = qy - S.p0.y; w.v0z = qz - S.p0.z;
  w.v1x = qx - S.p1.x; w.v1y = qy - S.p1.y; w.v1z = qz - S.p1.z;
  w.v2x = qx - S.p2.x; w.v2y = qy - S.p2.y; w.v2z = qz - S.p2.z;
  w.L0 = root(fma(w.v0x, w.v0x, fma(w.v0y, w.v0y, fma(w.v0z, w.v0z, kTiny))));
  w.L1 = root(fma(w.v1x, w.v1x, fma(w.v1y, w.v1y, fma(w.v1z, w.v1z, kTiny))));
  w.L2 = root(fma(w.v2x, w.v2x, fma(w.v2y, w.v2y, fma(w.v2z, w.v2z, kTiny))));
  w.ab0 = w.v0x * w.v1x + w.v0y * w.v1y + w.v0z * w.v1z;
  w.ab1 = w.v1x * w.v2x + w.v1y * w.v2y + w.v1z * w.v2z;
}

// One step q_k -> q_{k+1} (f = q_{k+1} - q_k): the walk goes from a to w, and
// the two segments' terms are added to s0 and s1.
__device__ __forceinline__ void walk_step(const Segs2 &S, const Walk2 &a, Walk2 &w, const TileVertex &at,
                                          const TileVertex &to, AngleSum &s0, AngleSum &s1) {
  walk_to(S, to, w);
  const double fx = at.q2f0.y, fy = at.f12.x, fz = at.f12.y;
  const double cx = a.v1y * fz - a.v1z * fy, cy = a.v1z * fx - a.v1x * fz, cz = a.v1x * fy - a.v1y * fx;
  const double g0 = a.v0x * w.v0x + a.v0y * w.v0y + a.v0z * w.v0z;
  const double g1 = a.v1x * w.v1x + a.v1y * w.v1y + a.v1z * w.v1z;
  const double g2 = a.v2x * w.v2x + a.v2y * w.v2y + a.v2z * w.v2z;
  {
    const double det = S.e0.x * cx + S.e0.y * cy + S.e0.z * cz;
    const double u = a.L0 * w.L1 + (w.v1x * a.v0x + w.v1y * a.v0y + w.v1z * a.v0z);
    const double div1 = a.L1 * u + (a.ab0 * w.L1 + g1 * a.L0);
    const double div2 = w.L0 * u + (g0 * w.L1 + w.ab0 * a.L0);
    const double sum = div1 + div2;
    s0.add(div1 * div2 - det * det, det * sum, det, sum);
  }
  {
    const double det = S.e1.x * cx + S.e1.y * cy + S.e1.z * cz;
    const double u = a.L1 * w.L2 + (w.v2x * a.v1x + w.v2y * a.v1y + w.v2z * a.v1z);
    const double div1 = a.L2 * u + (a.ab1 * w.L2 + g2 * a.L1);
    const double div2 = w.L1 * u + (g1 * w.L2 + w.ab1 * a.L1);
    const double sum = div1 + div2;
    s1.add(div1 * div2 - det * det, det * sum, det, sum);
  }
}

// A thread's share of an item term by term: `segs` segments of curve 1 from
// segment i on, against its group's part of every tile. For shares whose
// product left the range of kLeastScale.
__device__ __noinline__ double sum_terms(const double *xyz, int64_t o1, int64_t n1, int64_t i, int segs, int64_t o2,
                                         int64_t n2, int64_t k0, int64_t k1, int tile, int grp, int groups) {
  double v = 0.0;
  for (; k0 < k1; k0 += tile) {
    const int kt = (int)min(k1 - k0, (int64_t)tile);
    const int64_t ka = k0 + kt * grp / groups, kb = k0 + kt * (grp + 1) / groups;
    for (int64_t k = ka; k < kb; ++k)
      for (int j = 0; j < segs; ++j) v += near_term(xyz, o1, n1, o2, n2, make_int2((int)(i + j), (int)k));
  }
  return v;
}

// ------------------------------------------------------------------ FP64
// Tile shape: kB threads per CTA, kB curve-1 segments per item, kT curve-2
// vertices per shared-memory tile.
//
// A thread owns two neighbouring curve-1 segments (p0 p1, p1 p2), so that the
// CTA's threads are two or more groups; the groups take a share of each
// tile's steps each. Short loops (fewer than kB segments) make more groups,
// so that the CTA stays full. With v_j = q_k - p_j, w_j = q_{k+1} - p_j and
// f = q_{k+1} - q_k, a step of the segment p_j p_{j+1} needs
//   det = e_j . (v_1 x f)  (e_j = p_{j+1} - p_j; one cross product for both
//         segments, with the relative accuracy of the segment vectors),
//   the norms of w, v_j . w_j, w_{j+1} . v_j and w_j . w_{j+1}
// of which the two segments share p1's: 50 FP64 operations per segment pair,
// where one segment per thread with library square roots and FP64 sign tests
// took about 80.
//
// Bound: the schedulers. An FP64 instruction holds a scheduler's issue port
// for two cycles (16 lanes), so a step of 64 segment pairs costs 200 cycles
// plus one for every other instruction; hence the sign tests in a rare branch,
// the tile in 16-byte loads, the rescaling once per two steps and the
// two-state walk. 12 walks of 4,001 steps (1.84e9 segment pairs), B200: 12.6 ms
// with one segment per thread, 8.0 with two, 7.6 with the two-state walk, 6.8
// with the rest (269 G segment pairs/s; 372 G at 200 cycles a step). Twelve
// warps of 152 registers per SM; sixteen of 128 took 7.1 ms.
//
// Range: a term is at most 64 d^6 at a distance d, and two terms are multiplied
// between rescalings, so the product overflows above d = 1e25 and loses digits
// below 1e-23 (a single term below 1e-50), or when two vertices meet. The
// smallest product before a rescaling is kept (one integer minimum per two
// steps and segment); the share of a thread that saw one below kLeastScale, or
// whose product is not finite, is not a number, which its pair's sum shows to
// the reduction. kWide forms such a share again term by term (sum_terms); that
// code costs the others 1.5 %, so a call runs the kernel without it and has the
// pairs concerned summed again. The 12 walks: 6.01 ms a call without any of
// this, 6.02 with the check, 6.13 with kWide.
constexpr int kLeastScale = (1023 - 900) << 20;  // exponent bits of 2^-900: two terms at d = 1e-23
template <int kB, int kT, bool kWide = false>
__global__ void __launch_bounds__(kB, 384 / kB > 0 ? 384 / kB : 1) direct_fp64_kernel(DirectArgs A) {
  __shared__ TileVertex tile[kT + 1];
  __shared__ double s_red[kB / 32];
  __shared__ long long s_item;
  const int64_t items = plan_lone(A) ? 0 : plan_ready(A), span = plan_span(A, A.head->work);
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s_item = (long long)atomicAdd(&A.head->queue, 1ULL);
    __syncthreads();
    const int64_t item = s_item;
    if (item >= items) break;
    const Item it = item_of(A, item, kB, span);
    const int64_t o1 = it.o1, n1 = it.n1, o2 = it.o2, n2 = it.n2;
    // Threads: `width` segment pairs x `groups` shares of every tile.
    const int segs = (int)min((int64_t)kB, n1 - it.first);
    const int width = (segs + 1) / 2, groups = kB / width;
    const int grp = threadIdx.x / width, at = 2 * (threadIdx.x - grp * width);
    const bool active = grp < groups, second = at + 1 < segs;
    Segs2 S;
    S.p0 = S.p1 = S.p2 = make_double3(0, 0, 0);
    if (active) {
      const int64_t i = it.first + at;
      S.p0 = load_v(A.xyz, o1 + i);
      S.p1 = load_v(A.xyz, o1 + (i + 1 == n1 ? 0 : i + 1));
      S.p2 = second ? load_v(A.xyz, o1 + (i + 2 == n1 ? 0 : i + 2)) : S.p1;
    }
    S.e0 = make_double3(S.p1.x - S.p0.x, S.p1.y - S.p0.y, S.p1.z - S.p0.z);
    S.e1 = make_double3(S.p2.x - S.p1.x, S.p2.y - S.p1.y, S.p2.z - S.p1.z);
    AngleSum s0, s1;
    int least = INT_MAX;
    for (int64_t k0 = it.k0; k0 < it.k1; k0 += kT) {
      const int kt = (int)min(it.k1 - k0, (int64_t)kT);
      __syncthreads();
      for (int t = threadIdx.x; t <= kt; t += kB) {
        const int64_t kk = k0 + t;
        const double3 v = load_v(A.xyz, o2 + (kk == n2 ? 0 : kk));
        tile[t].q01 = make_double2(v.x, v.y);
        tile[t].q2f0.x = v.z;
      }
      __syncthreads();
      for (int t = threadIdx.x; t < kt; t += kB) {
        tile[t].q2f0.y = tile[t + 1].q01.x - tile[t].q01.x;
        tile[t].f12 = make_double2(tile[t + 1].q01.y - tile[t].q01.y, tile[t + 1].q2f0.x - tile[t].q2f0.x);
      }
      __syncthreads();
      if (!active) continue;
      const int ka = kt * grp / groups, kb = kt * (grp + 1) / groups;
      // Two steps per pass, the walk going a -> b -> a (no copies of its state).
      Walk2 a, b;
      walk_to(S, tile[ka], a);
      int k = ka;
      for (; k + 2 <= kb; k += 2) {
        walk_step(S, a, b, tile[k], tile[k + 1], s0, s1);
        walk_step(S, b, a, tile[k + 1], tile[k + 2], s0, s1);
        least = min(least, min(renorm(s0.x, s0.y), renorm(s1.x, s1.y)));
      }
      if (k < kb) {
        walk_step(S, a, b, tile[k], tile[k + 1], s0, s1);
        least = min(least, min(renorm(s0.x, s0.y), renorm(s1.x, s1.y)));
      }
    }
    double v = 0.0;
    if (active && (least < kLeastScale || !(fabs(s0.x) + fabs(s0.y) + fabs(s1.x) + fabs(s1.y) < 1e300))) {
      if constexpr (kWide)
        v = sum_terms(A.xyz, o1, n1, it.first + at, second ? 2 : 1, o2, n2, it.k0, it.k1, kT, grp, groups);
      else
        v = __longlong_as_double(0x7ff8000000000000ll);
    } else if (active) {
      if (second) {
        s0.add(s1.x, s1.y, 0.0, 0.0);
        s0.turns += s1.turns;
      }
      v = atan2(s0.y, s0.x) * kInvTwoPi + (double)s0.turns;
    }
    const double s = block_sum<kB>(v, s_red);
    if (threadIdx.x == 0) A.partial[item] = s;
  }
}

// A lone pair. The sum of one unlinked pair is nothing but the rounding of its
// terms, so the per-pair functions (fln_direct_pair) keep the operations and
// the order of one thread per segment, bit for bit: a segment's terms are
// multiplied in order, 32 segments summed by a butterfly, four such sums in
// order, then the next four. But a walk of n steps is n times the latency of
// a whole term, and a small pair has few segments; so an item is 32 segments,
// seven warps form the terms of 42 steps (lanes = segments, six steps each)
// while the eighth multiplies those of the 42 before, a chain of two FP64
// operations per step. The terms are stored scaled by a power of two, which
// changes no digit of their product. 300 x 211 segments, one call: 131 us with
// one thread per segment, 75 us now (with the launches and copies around it).
constexpr int kLoneSteps = 6, kLoneTile = 7 * kLoneSteps, kLoneChunk = 4 * kLoneTile;
__global__ void __launch_bounds__(256) direct_fp64_lone_kernel(DirectArgs A) {
  __shared__ double2 s_z[2][kLoneTile][32];
  __shared__ double s_q[3 * (kLoneChunk + 1)];
  __shared__ int s_turns[7][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const double work = A.head->work;
  const int64_t items = plan_lone(A) ? plan_ready(A) : 0;
  for (int64_t item = blockIdx.x; item < items; item += gridDim.x) {
    const Item it = item_of(A, item, kLoneSegs, plan_span(A, work));
    const int64_t o1 = it.o1, n1 = it.n1, o2 = it.o2, n2 = it.n2;
    const int64_t i = it.first + lane;
    const bool active = i < n1;
    double3 p0 = make_double3(0, 0, 0), p1 = p0;
    if (active) {
      p0 = load_v(A.xyz, o1 + i);
      p1 = load_v(A.xyz, o1 + (i + 1 == n1 ? 0 : i + 1));
    }
    double xs = 1.0, ys = 0.0, S = -1.0, turns = 0.0;
    int whole = 0;  // turns of the terms themselves
    const int64_t tiles = (n2 + kLoneTile - 1) / kLoneTile;
    for (int64_t t = 0; t <= tiles; ++t) {
      const int64_t k0 = t * kLoneTile;
      if (t < tiles && t % 4 == 0) {
        for (int x = threadIdx.x; x < 3 * (kLoneChunk + 1); x += 256) {
          int64_t v = 3 * k0 + x;
          if (v >= 3 * n2) v -= 3 * n2;
          if (v < 3 * n2) s_q[x] = __ldg(A.xyz + 3 * o2 + v);
        }
        __syncthreads();
      }
      if (warp < 7) {
        const int j0 = warp * kLoneSteps;
        const int steps = (int)min((int64_t)kLoneSteps, n2 - k0 - j0);
        if (t < tiles && steps > 0 && active) {
          const double *q = s_q + 3 * ((int)(t % 4) * kLoneTile + j0);
          double ax = q[0] - p0.x, ay = q[1] - p0.y, az = q[2] - p0.z;
          double bx = q[0] - p1.x, by = q[1] - p1.y, bz = q[2] - p1.z;
          double la = sqrt(ax * ax + ay * ay + az * az), lb = sqrt(bx * bx + by * by + bz * bz);
          double ab = ax * bx + ay * by + az * bz;
          for (int j = 0; j < steps; ++j) {
            const double qx = q[3 * j + 3], qy = q[3 * j + 4], qz = q[3 * j + 5];
            const double cx = qx - p1.x, cy = qy - p1.y, cz = qz - p1.z;
            const double dx = qx - p0.x, dy = qy - p0.y, dz = qz - p0.z;
            const double lc = sqrt(cx * cx + cy * cy + cz * cz), ld = sqrt(dx * dx + dy * dy + dz * dz);
            const double ca = cx * ax + cy * ay + cz * az;
            const double cb = cx * bx + cy * by + cz * bz;
            const double ad = ax * dx + ay * dy + az * dz;
            const double cd = cx * dx + cy * dy + cz * dz;
            const double det = ax * (by * cz - bz * cy) + az * (bx * cy - by * cx) + ay * (bz * cx - bx * cz);
            const double tt = la * lc;
            const double div1 = tt * lb + ab * lc + ca * lb + cb * la;
            const double div2 = tt * ld + ad * lc + ca * ld + cd * la;
            double xp = __fma_rn(div1, div2, -__dmul_rn(det, det));
            double yp = det * (div1 + div2);
            if (yp * det < 0) whole += det > 0 ? 1 : -1;
            renorm(xp, yp);
            s_z[t & 1][j0 + j][lane] = make_double2(xp, yp);
            ax = dx; ay = dy; az = dz;
            bx = cx; by = cy; bz = cz;
            la = ld; lb = lc; ab = cd;
          }
        }
      } else if (t > 0) {
        // Arctangent addition: (xs + i ys) *= (xp + i yp), tracking crossings
        // of the negative real axis (compute_link.cpp:245-269).
        const int n = (int)min((int64_t)kLoneTile, n2 - (k0 - kLoneTile));
        for (int j = 0; j < n; ++j) {
          const double2 z = s_z[(t - 1) & 1][j][lane];
          const double xp = z.x, yp = z.y;
          // (Fused as the compiler fuses the two sums in one loop.)
          const double ny = __fma_rn(xs, yp, __dmul_rn(xp, ys));
          const double nx = __fma_rn(xs, xp, -__dmul_rn(ys, yp));
          const double s3 = (ny > 0.0 || (ny == 0.0 && nx < 0.0)) ? 1.0 : -1.0;
          if (s3 * S < 0 && yp * S >= 0) turns += S;
          xs = nx;
          ys = ny;
          S = s3;
        }
        renorm(xs, ys);
      }
      __syncthreads();
    }
    if (warp < 7) s_turns[warp][lane] = whole;
    __syncthreads();
    if (warp == 7) {
      for (int w = 0; w < 7; ++w) turns += (double)s_turns[w][lane];
      double v = active ? atan2(ys, xs) * kInvTwoPi + turns : 0.0;
      for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) A.partial[item] = v;
    }
    __syncthreads();
  }
}

// ------------------------------------------------------------------ mixed
// Two FP32 values in a 64-bit register pair: one instruction does two adds,
// multiplies or fused multiply-adds (add/mul/fma.rn.f32x2), each rounded as
// the scalar one. They take the FMA pipe as long as two scalar instructions,
// but one issue slot.
using F2 = unsigned long long;
__device__ __forceinline__ F2 pack2(float lo, float hi) {
  F2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
  return r;
}
__device__ __forceinline__ float lo2(F2 v) { return __uint_as_float((unsigned)v); }
__device__ __forceinline__ float hi2(F2 v) { return __uint_as_float((unsigned)(v >> 32)); }
__device__ __forceinline__ F2 neg2(F2 v) { return v ^ 0x8000000080000000ull; }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
  F2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
  F2 r;
  asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
  F2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}
// 1 / sqrt(x) and y / x by the hardware's approximations, as rsqrtf and
// __fdividef but for subnormal numbers (treated as 0): of a squared distance
// (below 1e-19: the pair's other distances are about a segment's length, and
// it is a near one), and of a term's y beside an x of 2^-88 and more (kSmallX),
// where the flushed y changes the angle by less than 2^-38.
__device__ __forceinline__ float rsqrt_normal(float x) {
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
  return r;
}
__device__ __forceinline__ float div_normal(float y, float x) {
  float r;
  asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(y), "f"(x));
  return r;
}
struct F2x3 {
  F2 x, y, z;
};
__device__ __forceinline__ F2 dot2(const F2x3 &a, const F2x3 &b) {
  return fma2(a.z, b.z, fma2(a.x, b.x, mul2(a.y, b.y)));
}
// Small terms. A term (x, y) is 64 d^6 at a distance d. A pair with an endpoint
// distance below kNearLeast counts as near whatever its segments' lengths: its x
// and y would be subnormal, too short of digits for an angle (d of 2e-7), or 0
// (1e-8). The series for small angles takes x above 4 kSmallX (d of about 2e-5),
// where a flushed y does no harm; the comparison has that bound in the addend
// of x / 4, which changes nothing for larger x. Between the two a term takes the
// full arctangent. (Tests of x and y themselves cost 1 to 3 %.)
constexpr float kSmallX = 0x1p-90f, kNearLeast = 1e-6f;
// The segment length whose near distance is kNearLeast, taken in place of
// shorter ones (near_factor 0: not a number, and no pair is near).
__device__ __forceinline__ float least_length(float near_factor) { return kNearLeast / near_factor; }

__device__ __forceinline__ float dot_f(float ax, float ay, float az, float bx, float by, float bz) {
  return __fmaf_rn(az, bz, __fmaf_rn(ax, bx, __fmul_rn(ay, by)));
}

// arctan(t) for |t| <= 1/4 from its Maclaurin series t - t^3/3 + t^5/5 - t^7/7
// + t^9/9; the first omitted term, t^11/11, is below 8.7e-8 |t| (2.2e-8 at 1/4),
// about one rounding of FP32 there and less for smaller angles.
__device__ __forceinline__ F2 atan_small2(F2 t) {
  auto c = [](float v) { return pack2(v, v); };
  const F2 u = mul2(t, t);
  F2 p = fma2(u, c(1.0f / 9.0f), c(-1.0f / 7.0f));
  p = fma2(p, u, c(1.0f / 5.0f));
  p = fma2(p, u, c(-1.0f / 3.0f));
  p = fma2(p, u, c(1.0f));
  return mul2(p, t);
}

// Minimum and maximum over the CTA of 7 values each (a box and a length);
// the result is in out[0..6] (min) and out[7..13] (max) for every thread.
template <int kThreads>
__device__ __forceinline__ void block_minmax7(float *lo, float *hi, float (*s_box)[14], float *out) {
  for (int o = 16; o; o >>= 1)
    for (int v = 0; v < 7; ++v) {
      lo[v] = fminf(lo[v], __shfl_xor_sync(0xffffffffu, lo[v], o));
      hi[v] = fmaxf(hi[v], __shfl_xor_sync(0xffffffffu, hi[v], o));
    }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (lane == 0)
    for (int v = 0; v < 7; ++v) {
      s_box[warp][v] = lo[v];
      s_box[warp][7 + v] = hi[v];
    }
  __syncthreads();
  for (int v = 0; v < 14; ++v) {
    float r = s_box[0][v];
    for (int w = 1; w < kThreads / 32; ++w) r = v < 7 ? fminf(r, s_box[w][v]) : fmaxf(r, s_box[w][v]);
    out[v] = r;
  }
}

// Lanes of a warp with a near pair from which each evaluates its own (24 / never:
// 100 walks of 60 steps on one spot 480 / 543 us a call, 12 walks of 20,000 76.1 /
// 80.2 ms, 100 x 100 linked rings 857 / 816 us).
constexpr int kDenseNear = 24;

// A tile vertex: q relative to the tile's origin and the segment f to the next
// vertex, every value twice (the two halves of a packed operand), and
// near_factor x the segment's length.
struct __align__(16) MixVertex {
  float4 qxy, qzw, fxy, fz;
};

// The packed state of the walks of two neighbouring segments (p0 p1) and
// (p1 p2): low halves the first segment's, high halves the second's.
struct MixWalk {
  F2x3 a, b;  // q - p_j, q - p_{j+1}
  F2 la, lb;  // their norms
  F2 ab;      // a . b
  float m0, m1;  // min(la, lb) of each
};
struct MixSegs {
  F2x3 ra, rb;  // p_j, p_{j+1} relative to the tile's origin
  F2x3 e, ne;   // e = p_{j+1} - p_j and -e
  float near0, near1;  // near_factor x their lengths
};

// Vectors and norms of the walk at vertex v. The products of the shared
// vertex p1 are formed once (the second segment's a is the first one's b).
__device__ __forceinline__ void mix_at(const MixSegs &S, const MixVertex &v, MixWalk &w, F2 &aa, float &cc) {
  const F2 qx = pack2(v.qxy.x, v.qxy.y), qy = pack2(v.qxy.z, v.qxy.w), qz = pack2(v.qzw.x, v.qzw.y);
  w.a = F2x3{add2(qx, S.ra.x), add2(qy, S.ra.y), add2(qz, S.ra.z)};  // ra, rb hold -p
  w.b = F2x3{add2(qx, S.rb.x), add2(qy, S.rb.y), add2(qz, S.rb.z)};
  aa = dot2(w.a, w.a);
  const float x = hi2(w.b.x), y = hi2(w.b.y), z = hi2(w.b.z);
  cc = dot_f(x, y, z, x, y, z);
  w.ab = dot2(w.b, w.a);
}

// Terms of one step that are not both on the packed path: near pairs get 0 and
// their bit, the others the full arctangent with the branch turn.
__device__ __forceinline__ void mix_slow(F2 xp, F2 yp, F2 sdiv, F2 det, bool near0, bool near1, bool fast0, bool fast1,
                                         unsigned bit, float &t0, float &t1, unsigned &mask0, unsigned &mask1,
                                         int &turns0, int &turns1) {
  if (near0) {
    t0 = 0.f;
    mask0 |= bit;
  } else if (!fast0) {
    t0 = atan2f(lo2(yp), lo2(xp));
    if (lo2(sdiv) < 0.f && lo2(det) != 0.f) turns0 += lo2(det) > 0.f ? 1 : -1;
  }
  if (near1) {
    t1 = 0.f;
    mask1 |= bit;
  } else if (!fast1) {
    t1 = atan2f(hi2(yp), hi2(xp));
    if (hi2(sdiv) < 0.f && hi2(det) != 0.f) turns1 += hi2(det) > 0.f ? 1 : -1;
  }
}

// One step q_k -> q_{k+1} (step j of its run): the walk goes from a to w; the
// two terms are added to sum0 and sum1. A near pair adds 0 and sets bit j of its mask.
__device__ __forceinline__ void mix_step(const MixSegs &S, const MixWalk &a, MixWalk &w, const MixVertex &at,
                                         const MixVertex &to, bool far_tile, int j, float &sum0, float &sum1, unsigned &mask0,
                                         unsigned &mask1, int &turns0, int &turns1) {
  F2 dd;
  float cc;
  mix_at(S, to, w, dd, cc);
  w.la = mul2(dd, pack2(rsqrt_normal(lo2(dd)), rsqrt_normal(hi2(dd))));
  w.lb = pack2(hi2(w.la), cc * rsqrt_normal(cc));
  w.m0 = fminf(lo2(w.la), hi2(w.la));
  w.m1 = fminf(lo2(w.lb), hi2(w.lb));
  const F2 fx = pack2(at.fxy.x, at.fxy.y), fy = pack2(at.fxy.z, at.fxy.w), fz = pack2(at.fz.x, at.fz.y);
  const F2 ca = dot2(w.b, a.a), cb = dot2(w.b, a.b);
  const F2 ad = dot2(a.a, w.a);
  const F2 cx = fma2(fy, S.e.z, mul2(fz, S.ne.y)), cy = fma2(fz, S.e.x, mul2(fx, S.ne.z)),
           cz = fma2(fx, S.e.y, mul2(fy, S.ne.x));
  const F2 det = fma2(a.a.z, cz, fma2(a.a.x, cx, mul2(a.a.y, cy)));
  const F2 t = mul2(a.la, w.lb);
  const F2 div1 = fma2(cb, a.la, fma2(ca, a.lb, fma2(a.ab, w.lb, mul2(t, a.lb))));
  const F2 div2 = fma2(w.ab, a.la, fma2(ca, w.la, fma2(ad, w.lb, mul2(t, w.la))));
  const F2 sdiv = add2(div1, div2);
  const F2 xp = fma2(div1, div2, mul2(det, neg2(det)));
  const F2 yp = mul2(det, sdiv);
  const F2 quarter = fma2(xp, pack2(0.25f, 0.25f), pack2(-kSmallX, -kSmallX));
  const bool fast0 = lo2(sdiv) > 0.f && fabsf(lo2(yp)) < lo2(quarter);
  const bool fast1 = hi2(sdiv) > 0.f && fabsf(hi2(yp)) < hi2(quarter);
  // (fz.z: near_factor x the length of this curve-2 segment)
  const bool near0 = !far_tile && fminf(a.m0, w.m0) < fmaxf(S.near0, at.fz.z);
  const bool near1 = !far_tile && fminf(a.m1, w.m1) < fmaxf(S.near1, at.fz.z);
  // The principal branch, |angle| < 0.245.
  const F2 small = atan_small2(pack2(div_normal(lo2(yp), lo2(xp)), div_normal(hi2(yp), hi2(xp))));
  float t0 = lo2(small), t1 = hi2(small);
  if (__builtin_expect(!(fast0 && fast1) || near0 || near1, 0))
    mix_slow(xp, yp, sdiv, det, near0, near1, fast0, fast1, 1u << j, t0, t1, mask0, mask1, turns0, turns1);
  sum0 += t0;
  sum1 += t1;
}

// The mixed direct sum: kB curve-1 segments per item, two neighbouring ones
// per thread (kB / 2 threads), their FP32 arithmetic packed. A segment pair's
// term, the runs of 32 steps in which terms are summed in FP32 and the order of
// the FP64 sums are those of one thread per segment: the mixed sum of unlinked
// loops is the rounding of its terms, and it stays what it was bit for bit. So
// an item takes the whole of curve 2 (but for large calls, kMixedSpans), and
// only loops of at most kB / 2 segments make several groups of threads, a run
// of 32 steps each.
// Near pairs are noted in a bit mask per run and evaluated in FP64 by the warp
// together, 32 of a queue at a time, or by their own lanes where nearly all have
// one (kDenseNear), and added to their segment's sum in order. (A lane finds the
// queued pairs of its segments by one match of the 32 owners; looking through
// all 32 cost as much as the terms: 100 x 100 linked rings 954 us a call, 857
// now; 100 walks of 60 steps on one spot, nearly all pairs near, 849 -> 480, 786
// by one scalar segment per thread with near pairs as a divergent call. The walk
// of far pairs pays for the registers of this code, by 0 to 8 % for one form or
// another of it: one loop with a single place of evaluation took 4 % more on 12
// walks of 20,000 steps, 4 % less on the rings.)
//
// Bound: issue and the FMA pipe together. A step of 64 segment pairs needs 50
// packed and 8 scalar FMA-pipe operations (108 cycles of a scheduler's pipe, 709
// G segment pairs/s) and issues about 120 instructions; the pipe is 60 % and
// the issue slots 59 % busy. 16 walks of 5,003 steps (4.99e9 segment pairs),
// B200, whole call: 22.6 ms with one scalar segment per thread and near pairs
// as a divergent call; 16.7 packed with the near queue; 14.7 with the near and
// slow terms in one branch, subnormals flushed in the reciprocal and root, and
// cuts along curve 2. 10,000 linked rings: 1.49 -> 0.75 ms of kernel. Sixteen
// warps of 128 registers per SM: 12 of 162 take 14.9 ms, 20 of 96 16.0.
template <int kB, int kT>
__global__ void __launch_bounds__(kB / 2, 1024 / kB) direct_mixed_kernel(DirectArgs A) {
  constexpr int kThreads = kB / 2;
  __shared__ MixVertex tile[kT + 1];
  __shared__ int2 s_near[kThreads / 32][64];  // (curve-1 segment of the item x 32 + lane, curve-2 segment) left to FP64
  __shared__ double s_term[kThreads / 32][32];
  __shared__ unsigned s_mine[kThreads / 32][32];  // per lane: the flushed pairs of its segments
  __shared__ double s_red[kB / 32];
  __shared__ double s_seg[kB];  // per segment of the item
  __shared__ float s_box[kThreads / 32][14];
  __shared__ long long s_item;
  const float INF = __int_as_float(0x7f800000);
  const int lane = threadIdx.x & 31;
  const unsigned below = (1u << lane) - 1;
  int2 *queue = s_near[threadIdx.x >> 5];
  double *term = s_term[threadIdx.x >> 5];
  unsigned *mine = s_mine[threadIdx.x >> 5];
  const int64_t items = plan_few(A) ? 0 : plan_ready(A), span = plan_span(A, A.head->work);
  unsigned long long near_count = 0;
  if (threadIdx.x == 0) s_item = items > 0 && sm_turn(A, items) ? 0 : INT64_MAX;
  for (;;) {
    if (threadIdx.x == 0 && s_item < INT64_MAX) s_item = (long long)atomicAdd(&A.head->queue, 1ULL);
    __syncthreads();
    const int64_t item = s_item;
    if (item >= items) break;
    const Item it = item_of(A, item, kB, span);
    const int64_t o1 = it.o1, n1 = it.n1, o2 = it.o2, n2 = it.n2;
    const int segs = (int)min((int64_t)kB, n1 - it.first);
    // Groups: of at most as many as there are runs (more only for short loops).
    const int width = (segs + 1) / 2, groups = n1 > kB / 2 ? 1 : (int)min((int64_t)(kThreads / width), (n2 + 31) / 32);
    const int grp = threadIdx.x / width, at = 2 * (threadIdx.x - grp * width);
    const bool active = grp < groups, second = active && at + 1 < segs;
    const int64_t i0 = it.first + (active ? at : 0);
    const int64_t i1 = i0 + 1 == n1 ? 0 : i0 + 1, i2 = second ? (i1 + 1 == n1 ? 0 : i1 + 1) : i1;
    MixSegs S;
    float len0, len1;
    {
      const double3 p0 = load_v(A.xyz, o1 + i0), p1 = load_v(A.xyz, o1 + i1), p2 = load_v(A.xyz, o1 + i2);
      const float x0 = (float)(p1.x - p0.x), y0 = (float)(p1.y - p0.y), z0 = (float)(p1.z - p0.z);
      const float x1 = (float)(p2.x - p1.x), y1 = (float)(p2.y - p1.y), z1 = (float)(p2.z - p1.z);
      S.e = F2x3{pack2(x0, x1), pack2(y0, y1), pack2(z0, z1)};
      S.ne = F2x3{neg2(S.e.x), neg2(S.e.y), neg2(S.e.z)};
      len0 = fmaxf(sqrtf(dot_f(x0, y0, z0, x0, y0, z0)), least_length(A.near_factor));
      len1 = fmaxf(sqrtf(dot_f(x1, y1, z1, x1, y1, z1)), least_length(A.near_factor));
      S.near0 = A.near_factor * len0;
      S.near1 = A.near_factor * len1;
    }
    double acc0 = 0.0, acc1 = 0.0, near0 = 0.0, near1 = 0.0;
    int turns0 = 0, turns1 = 0, queued = 0;
    // Evaluates the oldest n queued pairs (n <= 32); every lane adds those of its
    // segments, oldest first.
    auto flush = [&](int n) {
      int2 q = make_int2(32 + lane, 0);  // (of no lane's segments)
      if (lane < n) {
        q = queue[lane];
        term[lane] = near_term(A.xyz, o1, n1, o2, n2, make_int2((int)(it.first + (q.x >> 5)), q.y));
      }
      mine[lane] = 0;
      __syncwarp();
      const unsigned of = __match_any_sync(0xffffffffu, lane < n ? q.x & 31 : q.x);
      if (lane < n) mine[q.x & 31] = of;
      __syncwarp();
      for (unsigned m = mine[lane]; m; m &= m - 1) {
        const int x = __ffs(m) - 1;
        if (queue[x].x >> 5 == at) near0 += term[x];
        else near1 += term[x];
      }
      __syncwarp();
      q = queue[32 + lane];
      __syncwarp();
      queue[lane] = q;
      __syncwarp();
    };
    for (int64_t k0 = it.k0; k0 < it.k1; k0 += kT) {  // a span is a multiple of kT (kMixedSpans)
      const int kt = (int)min(it.k1 - k0, (int64_t)kT);
      const double3 O = load_v(A.xyz, o2 + k0);
      __syncthreads();
      for (int t = threadIdx.x; t <= kt; t += kThreads) {
        const int64_t kk = k0 + t;
        const double3 v = load_v(A.xyz, o2 + (kk == n2 ? 0 : kk));
        const float x = (float)(v.x - O.x), y = (float)(v.y - O.y), z = (float)(v.z - O.z);
        tile[t].qxy = make_float4(x, x, y, y);
        tile[t].qzw.x = z;
        tile[t].qzw.y = z;
      }
      __syncthreads();
      // Boxes of this thread's curve-1 segments (slots 0-2) and of its
      // curve-2 tile vertices (slots 4-6), the longest segment (slot 3).
      float lo[7], hi[7];
      for (int v = 0; v < 7; ++v) {
        lo[v] = INF;
        hi[v] = -INF;
      }
      {
        const double3 p[3] = {load_v(A.xyz, o1 + i0), load_v(A.xyz, o1 + i1), load_v(A.xyz, o1 + i2)};
        float x[3], y[3], z[3];
        for (int v = 0; v < 3; ++v) {
          x[v] = (float)(p[v].x - O.x);
          y[v] = (float)(p[v].y - O.y);
          z[v] = (float)(p[v].z - O.z);
        }
        S.ra = F2x3{pack2(-x[0], -x[1]), pack2(-y[0], -y[1]), pack2(-z[0], -z[1])};
        S.rb = F2x3{pack2(-x[1], -x[2]), pack2(-y[1], -y[2]), pack2(-z[1], -z[2])};
        if (active) {
          lo[0] = fminf(x[0], fminf(x[1], x[2])); hi[0] = fmaxf(x[0], fmaxf(x[1], x[2]));
          lo[1] = fminf(y[0], fminf(y[1], y[2])); hi[1] = fmaxf(y[0], fmaxf(y[1], y[2]));
          lo[2] = fminf(z[0], fminf(z[1], z[2])); hi[2] = fmaxf(z[0], fmaxf(z[1], z[2]));
          hi[3] = fmaxf(len0, len1);
        }
      }
      for (int t = threadIdx.x; t < kt; t += kThreads) {
        const float4 axy = tile[t].qxy, bxy = tile[t + 1].qxy;
        const float az = tile[t].qzw.x, bz = tile[t + 1].qzw.x;
        const float fx = bxy.x - axy.x, fy = bxy.z - axy.z, fz = bz - az;
        const float len = sqrtf(dot_f(fx, fy, fz, fx, fy, fz));
        tile[t].fxy = make_float4(fx, fx, fy, fy);
        tile[t].fz = make_float4(fz, fz, A.near_factor * len, 0.f);
        lo[4] = fminf(lo[4], fminf(axy.x, bxy.x)); hi[4] = fmaxf(hi[4], fmaxf(axy.x, bxy.x));
        lo[5] = fminf(lo[5], fminf(axy.z, bxy.z)); hi[5] = fmaxf(hi[5], fmaxf(axy.z, bxy.z));
        lo[6] = fminf(lo[6], fminf(az, bz)); hi[6] = fmaxf(hi[6], fmaxf(az, bz));
        hi[3] = fmaxf(hi[3], len);
      }
      float bx[14];
      block_minmax7<kThreads>(lo, hi, s_box, bx);
      __syncthreads();
      // Box gap between the CTA's curve-1 segments and this tile: no segment
      // pair can be near when it exceeds near_factor x (longest segment).
      const float gx = fmaxf(0.f, fmaxf(bx[4] - bx[7], bx[0] - bx[11]));
      const float gy = fmaxf(0.f, fmaxf(bx[5] - bx[8], bx[1] - bx[12]));
      const float gz = fmaxf(0.f, fmaxf(bx[6] - bx[9], bx[2] - bx[13]));
      const float lim = A.near_factor * bx[10];
      const bool far_tile = gx * gx + gy * gy + gz * gz > 1.0001f * lim * lim;
      // The runs of 32 steps of this thread's group.
      const int runs = (kt + 31) / 32, ra = runs * grp / groups, rb = runs * (grp + 1) / groups;
      const int rounds = (runs + groups - 1) / groups;  // no group has more
      MixWalk wa, wb;
      for (int r = 0; r < rounds; ++r) {
        unsigned near_mask0 = 0, near_mask1 = 0;
        const int run = ra + r, j0 = 32 * run, steps = active && run < rb ? min(32, kt - j0) : 0;
        if (steps > 0) {
          if (r == 0) {
            F2 aa;
            float cc;
            mix_at(S, tile[j0], wa, aa, cc);
            // Norms at the start of a tile by the square root, inside one as
            // the steps form them.
            const bool inside = j0 > 0;
            const float a0 = lo2(aa), a1 = hi2(aa);
            const float l0 = inside ? a0 * rsqrt_normal(a0) : sqrtf(a0), l1 = inside ? a1 * rsqrt_normal(a1) : sqrtf(a1);
            const float l2 = inside ? cc * rsqrt_normal(cc) : sqrtf(cc);
            wa.la = pack2(l0, l1);
            wa.lb = pack2(l1, l2);
            wa.m0 = fminf(l0, l1);
            wa.m1 = fminf(l1, l2);
          }
          float sum0 = 0.f, sum1 = 0.f;
          int j = 0;
          const MixVertex *at_j = tile + j0;
          for (; j + 2 <= steps; j += 2, at_j += 2) {
            mix_step(S, wa, wb, at_j[0], at_j[1], far_tile, j, sum0, sum1, near_mask0, near_mask1, turns0, turns1);
            mix_step(S, wb, wa, at_j[1], at_j[2], far_tile, j + 1, sum0, sum1, near_mask0, near_mask1, turns0, turns1);
          }
          if (j < steps)
            mix_step(S, wa, wb, at_j[0], at_j[1], far_tile, j, sum0, sum1, near_mask0, near_mask1, turns0, turns1);
          acc0 += (double)sum0;
          acc1 += (double)sum1;
          if (!second) near_mask1 = 0;
        }
        // This run's near pairs, one per lane at a time: evaluated at once when
        // most lanes have one (after what is queued: a lane adds its segments'
        // pairs in order), else queued, and 32 of the queue evaluated together.
        while (__any_sync(0xffffffffu, (near_mask0 | near_mask1) != 0)) {
          const bool has = (near_mask0 | near_mask1) != 0;
          const unsigned m = __ballot_sync(0xffffffffu, has);
          near_count += lane == 0 ? __popc(m) : 0;
          const bool dense = __popc(m) >= kDenseNear;
          if (dense && queued > 0) {
            flush(queued);
            queued = 0;
          }
          if (has) {
            const bool first = near_mask0 != 0;
            const int k = __ffs(first ? near_mask0 : near_mask1) - 1;
            if (first) near_mask0 &= near_mask0 - 1;
            else near_mask1 &= near_mask1 - 1;
            const int seg = first ? at : at + 1, step = (int)(k0 + j0 + k);
            if (dense) {
              const double v = near_term(A.xyz, o1, n1, o2, n2, make_int2((int)it.first + seg, step));
              if (first) near0 += v;
              else near1 += v;
            } else {
              queue[queued + __popc(m & below)] = make_int2(seg << 5 | lane, step);
            }
          }
          if (dense) continue;
          queued += __popc(m);
          __syncwarp();
          if (queued >= 32) {
            flush(32);
            queued -= 32;
          }
        }
      }
    }
    if (queued > 0) flush(queued);
    // The item's sum: 32 segments at a time by a butterfly, those sums in order.
    for (int g = 0; g < groups; ++g) {
      if (grp == g) {
        const double v0 = acc0 * kInvTwoPi + (double)turns0 + near0;
        const double v1 = second ? acc1 * kInvTwoPi + (double)turns1 + near1 : 0.0;
        s_seg[at] = g ? s_seg[at] + v0 : v0;
        s_seg[at + 1] = g ? s_seg[at + 1] + v1 : v1;
      }
      __syncthreads();
    }
    double r = 0.0;
    for (int g = threadIdx.x >> 5; g < kB / 32; g += kThreads / 32) {
      double v = 32 * g + lane < segs ? s_seg[32 * g + lane] : 0.0;
      for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
      if (lane == 0) s_red[g] = v;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int g = 0; g < kB / 32; ++g) r += s_red[g];
      A.partial[item] = r;
    }
  }
  if (near_count) atomicAdd(&A.head->near, near_count);
}

// arctan(t) for |t| <= 1/4, the series of atan_small2.
__device__ __forceinline__ float atan_small(float t) {
  const float u = t * t;
  float p = fmaf(u, 1.0f / 9.0f, -1.0f / 7.0f);
  p = fmaf(p, u, 1.0f / 5.0f);
  p = fmaf(p, u, -1.0f / 3.0f);
  p = fmaf(p, u, 1.0f);
  return p * t;
}

// The mixed sum of few items, one segment per thread: with at most a few CTAs
// per SM a call lasts as long as one thread's walk, and a walk of two packed
// segments takes longer than a walk of one. Terms, runs and sums are those of
// direct_mixed_kernel, bit for bit (down to distances of 2e-5, see kSmallX).
// The times of both stand at few_items.
template <int kB, int kT>
__global__ void __launch_bounds__(kB) direct_mixed_few_kernel(DirectArgs A) {
  __shared__ float4 sq[kT + 1];  // xyz relative to the tile origin; w = length of segment t
  __shared__ double s_red[kB / 32];
  __shared__ float s_box[kB / 32][14];
  const float INF = __int_as_float(0x7f800000);
  __shared__ long long s_item;
  const int64_t items = plan_few(A) ? plan_ready(A) : 0;
  if (items == 0) return;
  if (threadIdx.x == 0) s_item = sm_turn(A, items) ? 0 : INT64_MAX;
  unsigned near_count = 0;
  for (;;) {
    if (threadIdx.x == 0 && s_item < INT64_MAX) s_item = (long long)atomicAdd(&A.head->queue, 1ULL);
    __syncthreads();
    const int64_t item = s_item;
    if (item >= items) break;
    const Item it = item_of(A, item, kB, int64_t(1) << 62);
    const int64_t o1 = it.o1, n1 = it.n1, o2 = it.o2, n2 = it.n2;
    const int64_t i = it.first + threadIdx.x;
    const bool active = i < n1;
    double3 p0 = make_double3(0, 0, 0), p1 = p0;
    if (active) {
      p0 = load_v(A.xyz, o1 + i);
      p1 = load_v(A.xyz, o1 + (i + 1 == n1 ? 0 : i + 1));
    }
    const float ex = (float)(p1.x - p0.x), ey = (float)(p1.y - p0.y), ez = (float)(p1.z - p0.z);
    const float len1 = fmaxf(sqrtf(ex * ex + ey * ey + ez * ez), least_length(A.near_factor));
    double acc = 0.0, near_turns = 0.0;
    int turns = 0;
    for (int64_t k0 = 0; k0 < n2; k0 += kT) {
      const int kt = (int)min(n2 - k0, (int64_t)kT);
      const double3 O = load_v(A.xyz, o2 + k0);
      __syncthreads();
      for (int t = threadIdx.x; t <= kt; t += kB) {
        const int64_t kk = k0 + t;
        const double3 v = load_v(A.xyz, o2 + (kk == n2 ? 0 : kk));
        sq[t] = make_float4((float)(v.x - O.x), (float)(v.y - O.y), (float)(v.z - O.z), 0.f);
      }
      __syncthreads();
      const float r0x = (float)(p0.x - O.x), r0y = (float)(p0.y - O.y), r0z = (float)(p0.z - O.z);
      const float r1x = (float)(p1.x - O.x), r1y = (float)(p1.y - O.y), r1z = (float)(p1.z - O.z);
      // Boxes of this thread's curve-1 segment (slots 0-2, length 3) and of
      // its curve-2 tile vertices (slots 4-6, length 3 of the max).
      float lo[7], hi[7];
      for (int v = 0; v < 7; ++v) {
        lo[v] = INF;
        hi[v] = -INF;
      }
      if (active) {
        lo[0] = fminf(r0x, r1x); hi[0] = fmaxf(r0x, r1x);
        lo[1] = fminf(r0y, r1y); hi[1] = fmaxf(r0y, r1y);
        lo[2] = fminf(r0z, r1z); hi[2] = fmaxf(r0z, r1z);
        hi[3] = len1;
      }
      for (int t = threadIdx.x; t < kt; t += kB) {
        const float4 a = sq[t], b = sq[t + 1];
        const float fx = b.x - a.x, fy = b.y - a.y, fz = b.z - a.z;
        const float len = sqrtf(fx * fx + fy * fy + fz * fz);
        sq[t].w = len;
        lo[4] = fminf(lo[4], fminf(a.x, b.x)); hi[4] = fmaxf(hi[4], fmaxf(a.x, b.x));
        lo[5] = fminf(lo[5], fminf(a.y, b.y)); hi[5] = fmaxf(hi[5], fmaxf(a.y, b.y));
        lo[6] = fminf(lo[6], fminf(a.z, b.z)); hi[6] = fmaxf(hi[6], fmaxf(a.z, b.z));
        hi[3] = fmaxf(hi[3], len);
      }
      float bx[14];
      block_minmax7<kB>(lo, hi, s_box, bx);
      __syncthreads();
      // Box gap between the CTA's curve-1 segments and this tile: no segment
      // pair can be near when it exceeds near_factor x (longest segment).
      const float gx = fmaxf(0.f, fmaxf(bx[4] - bx[7], bx[0] - bx[11]));
      const float gy = fmaxf(0.f, fmaxf(bx[5] - bx[8], bx[1] - bx[12]));
      const float gz = fmaxf(0.f, fmaxf(bx[6] - bx[9], bx[2] - bx[13]));
      const float lim = A.near_factor * bx[10];
      const bool far_tile = gx * gx + gy * gy + gz * gz > 1.0001f * lim * lim;
      if (!active) continue;
      float4 q = sq[0];
      float ax = q.x - r0x, ay = q.y - r0y, az = q.z - r0z;
      float bx_ = q.x - r1x, by = q.y - r1y, bz = q.z - r1z;
      const float aa = ax * ax + ay * ay + az * az, bb = bx_ * bx_ + by * by + bz * bz;
      float la = sqrtf(aa), lb = sqrtf(bb);
      float ab = ax * bx_ + ay * by + az * bz;
      float accf = 0.f;
      for (int k = 0; k < kt; ++k) {
        const float4 qn = sq[k + 1];
        const float cx = qn.x - r1x, cy = qn.y - r1y, cz = qn.z - r1z;
        const float dx = qn.x - r0x, dy = qn.y - r0y, dz = qn.z - r0z;
        const float cc = cx * cx + cy * cy + cz * cz, dd = dx * dx + dy * dy + dz * dz;
        const float lc = cc * rsqrtf(cc), ld = dd * rsqrtf(dd);
        const float cd = cx * dx + cy * dy + cz * dz;
        bool near = false;
        if (!far_tile) near = fminf(fminf(la, lb), fminf(lc, ld)) < A.near_factor * fmaxf(len1, q.w);
        if (near) {
          const int64_t kk = k0 + k, kn = kk + 1;
          near_turns += term_fp64(p0, p1, load_v(A.xyz, o2 + kk), load_v(A.xyz, o2 + (kn == n2 ? 0 : kn)));
          ++near_count;
        } else {
          const float ca = cx * ax + cy * ay + cz * az;
          const float cb = cx * bx_ + cy * by + cz * bz;
          const float ad = ax * dx + ay * dy + az * dz;
          const float fx = qn.x - q.x, fy = qn.y - q.y, fz = qn.z - q.z;
          const float det = ax * (fy * ez - fz * ey) + ay * (fz * ex - fx * ez) + az * (fx * ey - fy * ex);
          const float t = la * lc;
          const float div1 = t * lb + ab * lc + ca * lb + cb * la;
          const float div2 = t * ld + ad * lc + ca * ld + cd * la;
          const float sdiv = div1 + div2;
          const float xp = div1 * div2 - det * det;
          const float yp = det * sdiv;
          float term;
          if (sdiv > 0.f && fabsf(yp) < 0.25f * xp) {
            term = atan_small(__fdividef(yp, xp));  // principal branch, |angle| < 0.245
          } else {
            term = atan2f(yp, xp);
            if (sdiv < 0.f && det != 0.f) turns += (det > 0.f) ? 1 : -1;
          }
          accf += term;
        }
        if ((k & 31) == 31) {
          acc += (double)accf;
          accf = 0.f;
        }
        q = qn;
        ax = dx; ay = dy; az = dz;
        bx_ = cx; by = cy; bz = cz;
        la = ld; lb = lc; ab = cd;
      }
      acc += (double)accf;
    }
    const double v = active ? acc * kInvTwoPi + (double)turns + near_turns : 0.0;
    const double s = block_sum<kB>(v, s_red);
    if (threadIdx.x == 0) A.partial[item] = s;
  }
  if (near_count) atomicAdd(&A.head->near, (unsigned long long)near_count);
}

// Sums the item partials of each pair, a warp per pair, in item order, and
// checks it if there is a list `redo`: sums that are not numbers go there and,
// with a margin >= 0, those nearer than that to the rounding boundary. The
// estimate and the flags of a direct sum are 0.
__global__ void __launch_bounds__(256) reduce_items_kernel(DirectArgs A, double margin, double *lk, double *err, int32_t *flags, int32_t *redo) {
  const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (p >= A.npairs || (plan_ready(A) == 0)) return;
  const double work = A.head->work;
  const int64_t span = plan_span(A, work), block = plan_block(A);
  const int per = plan_lone(A) ? kBlockSegs / kLoneSegs : 1;  // a lone pair's items count in fours
  const int a = A.pairs[2 * p], b = A.pairs[2 * p + 1];
  const int64_t na = A.off[a + 1] - A.off[a], nb = A.off[b + 1] - A.off[b];
  const int64_t n = (max(na, nb) + block - 1) / block * ((min(na, nb) + span - 1) / span), s = A.start[p];
  double acc = 0.0, part = 0.0;
  for (int64_t x0 = 0; x0 < n; x0 += 32) {  // 32 loads at once, added one after another
    const double v = x0 + lane < n ? A.partial[s + x0 + lane] : 0.0;
    const int m = (int)min(n - x0, (int64_t)32);
    if (per == 1) {
#pragma unroll 8
      for (int j = 0; j < m; ++j) acc += __shfl_sync(0xffffffffu, v, j);
      continue;
    }
    for (int j = 0; j < m; ++j) {
      part += __shfl_sync(0xffffffffu, v, j);
      if ((j + 1) % per == 0 || j + 1 == m) {
        acc += part;
        part = 0.0;
      }
    }
  }
  if (lane) return;
  lk[p] = acc;
  if (err) err[p] = 0.0;
  if (flags) flags[p] = 0;
  if (redo && !(0.5 - fabs(acc - round(acc)) >= margin)) redo[atomicAdd(&A.head->redo, 1ULL)] = (int32_t)p;
}

// Checks the offsets and pairs, sums n_i n_j (a whole number: exact in any order
// below 2^53) and finds the longest loop, for the thread's share of them.
__device__ __forceinline__ void plan_check(const int64_t *off, int32_t nloops, const int32_t *pairs, int64_t npairs,
                                           int64_t t, int64_t nt, int &status, double &work,
                                           unsigned long long &longest) {
  if (t == 0 && off[0] != 0) status |= kBadStart;
  for (int64_t l = t; l < nloops; l += nt)
    if (off[l + 1] < off[l]) status |= kBadOrder;
  for (int64_t p = t; p < npairs; p += nt) {
    const int a = pairs[2 * p], b = pairs[2 * p + 1];
    if (a < 0 || a >= nloops || b < 0 || b >= nloops) {
      status |= kBadPair;
      continue;
    }
    const int64_t na = off[a + 1] - off[a], nb = off[b + 1] - off[b];
    if (na < 2 || nb < 2) status |= kBadSize;
    if (a == b) status |= kBadSame;
    work += (double)na * (double)nb;
    longest = max(longest, (unsigned long long)max(max(na, nb), int64_t(0)));
  }
}

// Items of the pairs [p0 + 32 w, ...) of a warp: reserved with one atomic,
// pairs in order, and written to the item list.
__device__ __forceinline__ void plan_warp(const DirectArgs &A, int64_t p, double work, int lane) {
  const int64_t span = plan_span(A, work), block = plan_block(A);
  int64_t n = 0;
  if (p < A.npairs) {
    const int a = A.pairs[2 * p], b = A.pairs[2 * p + 1];
    const int64_t na = A.off[a + 1] - A.off[a], nb = A.off[b + 1] - A.off[b];
    n = (max(na, nb) + block - 1) / block * ((min(na, nb) + span - 1) / span);
  }
  int64_t incl = n;
  for (int o = 1; o < 32; o <<= 1) {
    const int64_t y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  int64_t at = 0;
  if (lane == 31) at = (int64_t)atomicAdd(&A.head->items, (unsigned long long)incl);
  at = __shfl_sync(0xffffffffu, at, 31);
  const int64_t total = __shfl_sync(0xffffffffu, incl, 31), mine = at + incl - n;
  if (p < A.npairs) A.start[p] = mine;
  if (at + total > A.cap) return;  // the host makes room and plans again
  for (int j = 0; j < 32; ++j) {
    const int64_t s = __shfl_sync(0xffffffffu, mine, j), c = __shfl_sync(0xffffffffu, n, j);
    for (int64_t x = lane; x < c; x += 32) A.item_pair[s + x] = (int32_t)(p - lane + j);
  }
}

__global__ void __launch_bounds__(256) plan_work(DirectArgs A, int32_t nloops) {
  int status = 0;
  double work = 0.0;
  unsigned long long longest = 0;
  plan_check(A.off, nloops, A.pairs, A.npairs, (int64_t)blockIdx.x * blockDim.x + threadIdx.x,
             (int64_t)gridDim.x * blockDim.x, status, work, longest);
  if (A.lone > 0 && longest > 0) A.head->longest = longest;  // one pair: one thread has it
  status = __reduce_or_sync(0xffffffffu, status);
  for (int o = 16; o; o >>= 1) work += __shfl_xor_sync(0xffffffffu, work, o);
  if ((threadIdx.x & 31) == 0) {
    if (status) atomicOr(&A.head->status, status);
    if (work > 0) atomicAdd(&A.head->work, work);
  }
}

__global__ void __launch_bounds__(256) plan_items(DirectArgs A) {
  const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (A.head->status || p - (threadIdx.x & 31) >= A.npairs) return;
  plan_warp(A, p, A.head->work, threadIdx.x & 31);
}

// Both in one CTA, for calls of few pairs; it also clears the head.
constexpr int64_t kPlanSmall = 2048;
__global__ void __launch_bounds__(1024) plan_small(DirectArgs A, int32_t nloops) {
  __shared__ int s_status;
  __shared__ double s_work[32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_status = 0;
  __syncthreads();
  int status = 0;
  double work = 0.0;
  unsigned long long longest = 0;
  plan_check(A.off, nloops, A.pairs, A.npairs, threadIdx.x, 1024, status, work, longest);
  status = __reduce_or_sync(0xffffffffu, status);
  for (int o = 16; o; o >>= 1) work += __shfl_xor_sync(0xffffffffu, work, o);
  if (lane == 0) {
    s_work[w] = work;
    if (status) atomicOr(&s_status, status);
  }
  __syncthreads();
  work = 0.0;
  for (int x = 0; x < 32; ++x) work += s_work[x];
  // (A lone pair is thread 0's.)
  if (threadIdx.x == 0) *A.head = PlanHead{0, 0, 0, 0, A.lone > 0 ? longest : 0, work, s_status, 0};
  if (threadIdx.x <= kSmRanks) A.sm_rank[threadIdx.x] = 0;
  __syncthreads();
  if (s_status) return;
  for (int64_t p = threadIdx.x; p - lane < A.npairs; p += 1024) plan_warp(A, p, work, lane);
}

// The pairs of the redo list, and back: sums and flags of recomputed pairs.
__global__ void gather_pairs(const int32_t *list, int64_t n, const int32_t *pairs, int32_t *out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  out[2 * k] = pairs[2 * (int64_t)list[k]];
  out[2 * k + 1] = pairs[2 * (int64_t)list[k] + 1];
}
__global__ void scatter_redo(const int32_t *list, int64_t n, const double *src, double *lk, int32_t *flags) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  lk[list[k]] = src[k];
  if (flags) flags[list[k]] |= FLN_PAIR_FP64_RECOMPUTED;
}

// The tile shapes the direct sum can run with (fln_params.direct_tile), the
// default first: (curve-1 segments per item = threads per CTA, curve-2
// vertices per shared-memory tile).
struct TileShape {
  int block, tile;
};
constexpr TileShape kShapes[kDirectTileShapes] = {{128, 256}, {128, 128}, {128, 512},
                                                  {256, 256}, {256, 512}, {64, 256}};
static_assert(kShapes[0].block == kBlockSegs && kShapes[0].tile == kTile, "the default shape comes first");

// The sum kernel that a plan needs, where the host knows it; otherwise those it
// may need are all launched, and the plan fits one of them.
enum class SumKernel { kUnknown, kLone, kFew, kMany };

template <int kB, int kT>
void launch_direct_t(cudaStream_t st, int sms, int precision, int64_t most, SumKernel which, const DirectArgs &A) {
  if (A.lone > 0 && which != SumKernel::kMany)
    direct_fp64_lone_kernel<<<(int)std::min(most, kLonePerSm * sms), 256, 0, st>>>(A);
  if (A.few > 0 && which != SumKernel::kMany)
    direct_mixed_few_kernel<kB, kT><<<(int)std::min(most, A.few), kB, 0, st>>>(A);
  if (which == SumKernel::kLone || which == SumKernel::kFew) return;
  auto kernel = precision != FLN_PREC_FP64 ? direct_mixed_kernel<kB, kT> : direct_fp64_kernel<kB, kT>;
  if constexpr (kB == kBlockSegs && kT == kTile)
    if (precision == FLN_PREC_FP64 && A.wide) kernel = direct_fp64_kernel<kB, kT, true>;
  const int threads = precision == FLN_PREC_FP64 ? kB : kB / 2;
  const int64_t resident = (int64_t)sms * occupancy_of((const void *)kernel, threads);
  kernel<<<(int)std::max<int64_t>(1, std::min(most, resident)), threads, 0, st>>>(A);
}

void launch_direct(int shape, cudaStream_t st, int sms, int precision, int64_t most, SumKernel which,
                   const DirectArgs &A) {
  switch (shape) {
    case 1: launch_direct_t<128, 128>(st, sms, precision, most, which, A); break;
    case 2: launch_direct_t<128, 512>(st, sms, precision, most, which, A); break;
    case 3: launch_direct_t<256, 256>(st, sms, precision, most, which, A); break;
    case 4: launch_direct_t<256, 512>(st, sms, precision, most, which, A); break;
    case 5: launch_direct_t<64, 256>(st, sms, precision, most, which, A); break;
    default: launch_direct_t<kBlockSegs, kTile>(st, sms, precision, most, which, A); break;
  }
}

// Most items of a plan for direct_mixed_few_kernel: its resident CTAs.
int64_t few_most(int shape, int sms) {
  const void *k[kDirectTileShapes] = {
      (const void *)direct_mixed_few_kernel<128, 256>, (const void *)direct_mixed_few_kernel<128, 128>,
      (const void *)direct_mixed_few_kernel<128, 512>, (const void *)direct_mixed_few_kernel<256, 256>,
      (const void *)direct_mixed_few_kernel<256, 512>, (const void *)direct_mixed_few_kernel<64, 256>};
  return (int64_t)sms * occupancy_of(k[shape], kShapes[shape].block);
}

}  // namespace

int recompute_pairs(Context &ctx, const double *d_xyz, const int64_t *d_off, int32_t nloops, const int32_t *d_pairs,
                    const int32_t *d_list, int64_t n, double *d_lk, int32_t *d_flags) {
  if (n <= 0) return 0;
  // The list first: the direct sum uses the buffers it may lie in.
  int32_t *list = ctx.d_redo.as<int32_t>(3 * n + (n & 1) + 2 * n), *pairs = list + n;
  double *sums = reinterpret_cast<double *>(list + 3 * n + (n & 1));
  const int grid = (int)((n + 255) / 256);
  FLN_CUDA(cudaMemcpyAsync(list, d_list, n * sizeof(int32_t), cudaMemcpyDeviceToDevice, ctx.stream));
  gather_pairs<<<grid, 256, 0, ctx.stream>>>(list, n, d_pairs, pairs);
  FLN_CUDA(cudaGetLastError());
  const int launches =
      direct_sum_device(ctx, d_xyz, d_off, nloops, pairs, n, FLN_PREC_FP64, 0.0, -1.0, sums, nullptr, nullptr, 0, nullptr,
                        true).launches;
  scatter_redo<<<grid, 256, 0, ctx.stream>>>(list, n, sums, d_lk, d_flags);
  FLN_CUDA(cudaGetLastError());
  return launches + 2;
}

DirectResult direct_sum_device(Context &ctx, const double *d_xyz, const int64_t *d_off, int32_t nloops,
                               const int32_t *d_pairs, int64_t np, int precision, double near_factor, double margin,
                               double *d_lk, double *d_err, int32_t *d_flags, int tile_shape, const DirectTail *tail,
                               bool wide) {
  if (tile_shape < 0 || tile_shape >= kDirectTileShapes)
    throw Error(FLN_ERR_INVALID_ARGUMENT, "direct_tile in [0, " + std::to_string(kDirectTileShapes - 1) + "]");
  DirectResult R;
  if (np == 0) return R;
  if (np > INT32_MAX) throw Error(FLN_ERR_INVALID_ARGUMENT, "more than 2^31 - 1 pairs");
  const int kB = kShapes[tile_shape].block;
  cudaStream_t st = ctx.stream;
  constexpr size_t kHeadBytes = sizeof(PlanHead) + (kSmRanks + 1) * sizeof(unsigned);
  PlanHead *d_head = static_cast<PlanHead *>(ctx.d_counter.need(kHeadBytes));
  unsigned *d_rank = reinterpret_cast<unsigned *>(d_head + 1);
  int64_t *d_start = ctx.d_items.as<int64_t>(np);
  int32_t *d_redo = wide ? nullptr : ctx.d_near.as<int32_t>(np);
  PlanHead &head = *static_cast<PlanHead *>(ctx.h_head.need(sizeof(PlanHead)));
  const int64_t target = (int64_t)ctx.num_sms * 8 * (512 / kB);
  // FP64 sums and large mixed ones are cut along curve 2; a lone FP64 pair has
  // a kernel of its own.
  const double least = precision == FLN_PREC_MIXED ? kMixedSpans : 0.0;
  const int64_t lone = precision == FLN_PREC_FP64 && np == 1 && tile_shape == 0 ? kLonePerSm * ctx.num_sms * kLoneSegs : 0;
  int64_t few = precision == FLN_PREC_MIXED ? few_most(tile_shape, ctx.num_sms) : 0;
  if (np > few) few = 0;  // (a pair has at least one item)
  // Room for the items: of the largest call so far, or a guess; a plan that
  // does not fit runs no kernel and is made again with room.
  ctx.direct_items = std::max<int64_t>(ctx.direct_items, std::max<int64_t>(4 * target, 2 * np));
  for (int attempt = 0;; ++attempt) {
    const int64_t cap = ctx.direct_items;
    DirectArgs A{d_xyz, d_off, d_pairs, d_start, ctx.d_loops.as<int32_t>(cap), (int32_t)np, cap, target, least, kB, few, lone,
                 d_head, d_rank, ctx.num_sms, ctx.d_partial.as<double>(cap), (float)near_factor, wide};
    if (np <= kPlanSmall && nloops <= 16 * kPlanSmall) {
      plan_small<<<1, 1024, 0, st>>>(A, nloops);
    } else {
      FLN_CUDA(cudaMemsetAsync(d_head, 0, kHeadBytes, st));
      const int64_t most = std::max<int64_t>(np, nloops);
      plan_work<<<(int)std::min<int64_t>((most + 255) / 256, 8 * ctx.num_sms), 256, 0, st>>>(A, nloops);
      plan_items<<<(int)((np + 255) / 256), 256, 0, st>>>(A);
      ++R.launches;
    }
    FLN_CUDA(cudaGetLastError());
    FLN_CUDA(cudaEventRecord(ctx.ev2, st));
    SumKernel which = SumKernel::kUnknown;
    if (lone > 0 && tail && tail->known_longest > 0)
      which = tail->known_longest <= lone ? SumKernel::kLone : SumKernel::kMany;
    launch_direct(tile_shape, st, ctx.num_sms, precision, cap, which, A);
    FLN_CUDA(cudaGetLastError());
    FLN_CUDA(cudaEventRecord(ctx.ev3, st));
    reduce_items_kernel<<<(int)((np + 7) / 8), 256, 0, st>>>(A, margin, d_lk, d_err, d_flags, d_redo);
    FLN_CUDA(cudaGetLastError());
    R.launches += 3;
    if (tail) FLN_CUDA(cudaEventRecord(tail->end, st));
    if (tail && tail->bytes) FLN_CUDA(cudaMemcpyAsync(tail->h_dst, tail->d_src, tail->bytes, cudaMemcpyDeviceToHost, st));
    FLN_CUDA(cudaMemcpyAsync(&head, d_head, sizeof head, cudaMemcpyDeviceToHost, st));
    FLN_CUDA(cudaStreamSynchronize(st));
    if (head.status) {
      throw Error(FLN_ERR_INVALID_ARGUMENT,
                  head.status & kBadStart ? "loop_offsets must start at 0 and hold nloops + 1 entries."
                  : head.status & kBadOrder ? "loop_offsets must be non-decreasing."
                  : head.status & kBadPair ? "pair index out of range."
                  : head.status & kBadSize ? "every loop in a pair needs at least two vertices."
                                           : "a pair must name two different loops.");
    }
    if ((int64_t)head.items <= cap) break;
    if (attempt > 0) throw Error(FLN_ERR_INTERNAL, "direct sum: the plan does not fit its own count");
    ctx.direct_items = (int64_t)head.items;
  }
  float ms = 0;
  FLN_CUDA(cudaEventElapsedTime(&ms, ctx.ev2, ctx.ev3));
  ctx.stats.ms_main_kernel += ms;
  R.near_terms = (double)head.near;
  R.work = head.work;
  const int64_t redo = (int64_t)head.redo;
  const bool mixed = precision == FLN_PREC_MIXED;
  if (mixed) R.redone = redo;
  R.complete = tail && redo == 0;
  if (redo > 0)
    R.launches += recompute_pairs(ctx, d_xyz, d_off, nloops, d_pairs, d_redo, redo, d_lk, mixed ? d_flags : nullptr);
  return R;
}

}  // namespace fln

// ---------------------------------------------------------------------------
// Direct sum that allocates nothing (fln_linking_numbers_direct_noalloc).
//
// Some callers cannot call cudaMalloc: code that runs while another framework
// owns the device's memory pool (a renderer or simulator with its own
// allocator and a fixed budget), code that must not add allocator
// synchronisation or fragmentation to a latency-critical loop, and code on
// paths where an allocation failure cannot be handled. For them the direct
// sum runs entirely in the caller's input and output buffers plus one
// file-scope device array, g_noalloc_scratch, of kNoAllocScratchBytes
// (about 8.9 MB). Every GPU that loads libfln.so holds that array until the
// process exits. Limits: at most kNoAllocMaxPairs loop pairs per call and
// kNoAllocMaxItems work items (one item = 128 segments of the longer loop of
// a pair, summed over the pairs); larger calls are rejected with
// FLN_ERR_INVALID_ARGUMENT before any kernel runs on them. The mixed
// precision uses the default near factor (kDefaultNearFactor), so results
// equal the allocating entry point's with fln_default_params.
//
// Every call copies the plan's header (item count, status) back to the host
// and waits for it: the call blocks until the work queued earlier on the
// stream and the planning kernel have run.
//
// In host code the name g_noalloc_scratch only stands for the array: its
// device address is obtained once per device with cudaGetSymbolAddress, on
// the first call made with that device current, and cached. That first call
// therefore does the set-up and should come before any stream capture.
// All calls share the array and it keeps the previous call's contents: the
// planning kernel clears the work-queue counters at the start of every call.
// Calls whose work overlaps on the GPU (different streams, or host threads
// racing) race on the array; issue them one after another.
namespace fln {
namespace {

constexpr int64_t kNoAllocMaxPairs = 65536;
constexpr int64_t kNoAllocMaxItems = int64_t(1) << 20;
constexpr size_t kNaHeader = 256;  // PlanHead
constexpr size_t kNaStart = kNaHeader;                                       // int64 per pair + 1
constexpr size_t kNaPartial = (kNaStart + (kNoAllocMaxPairs + 1) * 8 + 255) / 256 * 256;  // double per item
constexpr size_t kNoAllocScratchBytes = kNaPartial + kNoAllocMaxItems * 8;

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocScratchBytes];

static_assert(sizeof(PlanHead) <= kNaHeader, "the header's room");
// status of the plan: bit 0: bad pair index, bit 1: loop with < 2 vertices

// One CTA plans the call inside the scratch array: counts each pair's items
// (kBlockSegs segments of its longer loop against the whole other one), scans
// them into start and clears the counters the direct-sum kernels start from.
__global__ void __launch_bounds__(1024) noalloc_plan(const int64_t *off, int32_t nloops, const int32_t *pairs,
                                                     int64_t npairs, unsigned char *scratch) {
  PlanHead *h = reinterpret_cast<PlanHead *>(scratch);
  int64_t *start = reinterpret_cast<int64_t *>(scratch + kNaStart);
  __shared__ long long s_warp[32];
  __shared__ long long s_carry;
  __shared__ double s_work[32];
  __shared__ int s_status;
  if (threadIdx.x == 0) {
    s_carry = 0;
    s_status = 0;
  }
  __syncthreads();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double work = 0.0;
  for (int64_t base = 0; base < npairs; base += 1024) {
    const int64_t p = base + threadIdx.x;
    long long items = 0;
    if (p < npairs) {
      const int a = pairs[2 * p], b = pairs[2 * p + 1];
      if (a < 0 || a >= nloops || b < 0 || b >= nloops || a == b) {
        atomicOr(&s_status, 1);
      } else {
        const int64_t na = off[a + 1] - off[a], nb = off[b + 1] - off[b];
        if (na < 2 || nb < 2) {
          atomicOr(&s_status, 2);
        } else {
          items = (max(na, nb) + kBlockSegs - 1) / kBlockSegs;
          work += (double)na * (double)nb;
        }
      }
    }
    // Exclusive block scan of `items`.
    long long incl = items;
    for (int o = 1; o < 32; o <<= 1) {
      const long long y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) s_warp[warp] = incl;
    __syncthreads();
    if (warp == 0) {
      long long v = s_warp[lane];
      for (int o = 1; o < 32; o <<= 1) {
        const long long y = __shfl_up_sync(0xffffffffu, v, o);
        if (lane >= o) v += y;
      }
      s_warp[lane] = v;  // inclusive over warps
    }
    __syncthreads();
    const long long warp_base = warp ? s_warp[warp - 1] : 0;
    if (p < npairs) start[p] = s_carry + warp_base + incl - items;
    __syncthreads();
    if (threadIdx.x == 0) s_carry += s_warp[31];
    __syncthreads();
  }
  for (int o = 16; o; o >>= 1) work += __shfl_xor_sync(0xffffffffu, work, o);
  if (lane == 0) s_work[warp] = work;
  __syncthreads();
  if (threadIdx.x == 0) {
    work = 0.0;
    for (int w = 0; w < 32; ++w) work += s_work[w];
    start[npairs] = s_carry;
    *h = PlanHead{0, 0, (unsigned long long)s_carry, 0, 0, work, s_status, 0};
  }
}

// Device address of g_noalloc_scratch per device, set up on first use.
void *noalloc_scratch_for_current_device(fln_status &st, std::string &msg) {
  static void *addr[64] = {nullptr};
  static std::mutex mu;
  int dev = -1;
  cudaError_t e = cudaGetDevice(&dev);
  if (e != cudaSuccess || dev < 0 || dev >= 64) {
    st = e == cudaSuccess ? FLN_ERR_INVALID_ARGUMENT : FLN_ERR_NO_DEVICE;
    msg = std::string("cudaGetDevice: ") + (e == cudaSuccess ? "device index >= 64" : cudaGetErrorString(e));
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void *p = nullptr;
    e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      st = FLN_ERR_CUDA;
      msg = std::string("cudaGetSymbolAddress(g_noalloc_scratch): ") + cudaGetErrorString(e);
      return nullptr;
    }
    addr[dev] = p;
  }
  return addr[dev];
}

}  // namespace

// Records the message behind a non-OK status for fln_last_error() (capi.cpp).
void set_last_error(const std::string &msg);

}  // namespace fln

extern "C" fln_status fln_linking_numbers_direct_noalloc(const double *d_xyz, const int64_t *d_loop_offsets,
                                                         int32_t nloops, const int32_t *d_pairs, int64_t npairs,
                                                         int32_t precision, double *d_lk_out, void *stream) {
  using namespace fln;
  auto fail = [](fln_status s, const std::string &m) {
    set_last_error(m);
    return s;
  };
  if (npairs < 0 || npairs > kNoAllocMaxPairs)
    return fail(FLN_ERR_INVALID_ARGUMENT, "fln_linking_numbers_direct_noalloc: npairs must be in [0, " +
                                              std::to_string(kNoAllocMaxPairs) + "], got " + std::to_string(npairs));
  if (nloops < 0 || (npairs > 0 && (!d_xyz || !d_loop_offsets || !d_pairs || !d_lk_out)))
    return fail(FLN_ERR_INVALID_ARGUMENT, "fln_linking_numbers_direct_noalloc: NULL or negative argument");
  if (precision != FLN_PREC_FP64 && precision != FLN_PREC_MIXED)
    return fail(FLN_ERR_INVALID_ARGUMENT, "fln_linking_numbers_direct_noalloc: unknown precision");
  if (npairs == 0) return FLN_OK;
  fln_status st = FLN_OK;
  std::string msg;
  unsigned char *scratch = static_cast<unsigned char *>(noalloc_scratch_for_current_device(st, msg));
  if (!scratch) return fail(st, msg);
  cudaStream_t s = static_cast<cudaStream_t>(stream);
  noalloc_plan<<<1, 1024, 0, s>>>(d_loop_offsets, nloops, d_pairs, npairs, scratch);
  PlanHead h;
  cudaError_t e = cudaGetLastError();
  if (e == cudaSuccess) e = cudaMemcpyAsync(&h, scratch, sizeof h, cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) return fail(FLN_ERR_CUDA, std::string("fln_linking_numbers_direct_noalloc: ") + cudaGetErrorString(e));
  if (h.status & 1) return fail(FLN_ERR_INVALID_ARGUMENT, "fln_linking_numbers_direct_noalloc: pair index out of range or a pair names one loop twice");
  if (h.status & 2) return fail(FLN_ERR_INVALID_ARGUMENT, "fln_linking_numbers_direct_noalloc: every loop in a pair needs at least two vertices");
  if ((int64_t)h.items > kNoAllocMaxItems)
    return fail(FLN_ERR_INVALID_ARGUMENT, "fln_linking_numbers_direct_noalloc: " + std::to_string((int64_t)h.items) +
                                              " work items exceed the limit of " + std::to_string(kNoAllocMaxItems) +
                                              " (one item = 128 segments of the longer loop of a pair)");
  int dev = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  // The default tile shape (the planning kernel cuts items of kBlockSegs), whole
  // walks of curve 2 at any amount of work.
  const int64_t most = precision == FLN_PREC_MIXED ? few_most(0, sms) : 0;
  const bool few = few_items((int64_t)h.items, h.work, most);
  const DirectArgs A{d_xyz, d_loop_offsets, d_pairs, reinterpret_cast<int64_t *>(scratch + kNaStart), nullptr,
                     (int32_t)npairs, (int64_t)h.items, 1, 1e300, kBlockSegs, few ? most : 0, 0, reinterpret_cast<PlanHead *>(scratch), nullptr, sms,
                     reinterpret_cast<double *>(scratch + kNaPartial), (float)kDefaultNearFactor, true};
  launch_direct(0, s, sms, precision, (int64_t)h.items, few ? SumKernel::kFew : SumKernel::kMany, A);
  reduce_items_kernel<<<(int)((npairs + 7) / 8), 256, 0, s>>>(A, -1.0, d_lk_out, nullptr, nullptr, nullptr);
  e = cudaGetLastError();
  if (e != cudaSuccess) return fail(FLN_ERR_CUDA, std::string("fln_linking_numbers_direct_noalloc: ") + cudaGetErrorString(e));
  return FLN_OK;
}
