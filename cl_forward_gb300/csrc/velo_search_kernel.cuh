// velo_search_kernel.cuh -- sm_103a search-by-triplet kernel (device code).
//
// Included by one translation unit per seeding width (velo_kernels_g8.cu,
// _g16.cu, _g32.cu), each of which instantiates the kernel builds for its
// width; velo_kernels.cu picks the kernel of a launch.
//
// One CTA reconstructs one event (the reference's one work-group per event,
// Kernel.cl:607, KernelInvoker.cpp:26-27), either one CTA per event or
// persistent CTAs pulling events, largest first, from a work queue.  The
// event's hits and its per-hit working state (the "arena": x, y, z,
// candidate windows, used flags) live in dynamic shared memory when the event
// fits the launch's tile, else in global scratch with the same layout, which
// L1 caches.  On GB300 the fastest launch keeps the tile tiny: shared memory
// and L1 share each SM's storage, and resident CTAs are register-bound, so L1
// serves the arenas better than staging does.  The tracks-to-follow entries,
// tracklets and working tracks are per-hit-row global scratch.
//
// Decisions are the reference's, bit for bit:
//  * every FP32 expression is written with round-to-nearest intrinsics
//    (__fadd_rn/__fsub_rn/__fmul_rn/__fdiv_rn), term by term as in
//    Kernel.cl, so no contraction into FMA can change a cut;
//  * ties resolve as in the reference: forwarding keeps the first minimum in
//    h2 order (Kernel.cl:302-305); seeding keeps the minimum of the packed
//    key (fit, Y-lane, h1 element, h2), which is the reference's per-lane
//    first minimum followed by its lowest-lane reduction (Kernel.cl:517-545);
//  * a Y-lane stops at its first h1 without an h2 window (the cumulative
//    `inside_bounds` of Kernel.cl:437,457).
// Narrowing: on a module whose hits are x-sorted, x-window searches use
// binary search and skip only hits that provably fail the reference's own
// float predicate (the predicted x is monotone in hit z, so the module's z
// range bounds it; a 0.01 mm guard covers the rounding of the bound).  On an
// unsorted module the full sequential scan runs.  Narrowing changes work, not
// results.
//
// The two parities of modules are seeded by different warps, each with its own
// tracks-to-follow entries, so a CTA meets at one barrier per two module
// iterations (Worker).
//
// Optional per launch: the x-sort of each event while it is staged, with the
// sorted hit arrays written back into the input (sort_events), and a
// per-event record published in host memory when the event is done
// (results, for a host that consumes events while the search runs).
#pragma once

#include <cuda_runtime.h>
#include <float.h>
#include <stdint.h>

#include <type_traits>

#include "velo_internal.h"
#include "velo_mlp_warp.cuh"
#include "velo_partition.cuh"

namespace velo {

__device__ __forceinline__ float fadd(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ float fsub(float a, float b) { return __fsub_rn(a, b); }
__device__ __forceinline__ float fmul(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ float fdiv(float a, float b) { return __fdiv_rn(a, b); }

constexpr unsigned kFull = 0xffffffffu;
constexpr uint32_t kNone16 = 0xffffu;
// Per-hit flag byte.  kUsed: the reference's hit_used.  kDead (set once per
// event, only where the pair seeding runs): the hit as an h1 has no h2 window.
constexpr uint8_t kUsed = 1, kDead = 2;
// Per-module flags: its hits are x-sorted; its dead h1s are its last hits.
constexpr uint8_t kSorted = 1, kDeadTail = 2;

// Seeding state per CTA: each warp's lists, and per module parity the
// occupancy map of the h2 module.  kOwn: the h0s a warp seeds at once.
constexpr int kQueue = 32;            // pairs a warp holds for the exact fits
template <int kWarps, int kOwn, int kList, int kMapRows>
struct SeedShared {
  float4 h0[kWarps][kOwn];            // x, y, z, first h1's place - first pair (int bits)
  float2 reach[kWarps][kOwn];         // the h0's y cut, and in plain geometry (z2 - z0) / (z1 - z0)
  unsigned long long best[kWarps][kOwn];   // the h0's best (fit, Y-lane, h1, h2) so far
  alignas(16) uint32_t map[2][kMapRows];   // rows of 32 cells
  std::conditional_t<(kOwn > 4), uint32_t, uint16_t> queue[kWarps][kQueue];   // h0 << 14 | h1 in its module
  uint16_t first[kWarps][kOwn];       // the h0's first h1 in its module
  // by parity: the usable h1s (unused, with an h2 window) of a module of up to
  // kList hits; per 32 hits their lanes and their number before
  uint2 usable[2][kList / 32 + 1];
  uint8_t list[2][kList];
  uint8_t active[2][32];              // by parity: unused h0s of a block of 32 hits, by rank
};

// Per-CTA shared state for events of up to kMods modules.  Launches whose
// events all have at most kCompactModules - 1 modules (every VELO geometry)
// use the compact form: 4 KB less static shared memory per CTA, which goes
// to L1 and to more resident CTAs.
template <int kMods, int kWarps>
struct SharedT {
  // h0s per warp and round: with two warps a block of 32 hits rarely leaves
  // more than 16 unused; the others keep the static state below 8 KB
  static constexpr int kOwn = kWarps <= 2 ? 16 : kMods <= kCompactModules ? 64 / kWarps : 16 / kWarps + (kWarps <= 8) * 2;
  static constexpr int kMaxWarps = kWarps;
  static constexpr int kList = kMods <= kCompactModules ? 256 : 64;
  static constexpr int kMapRows = kMods <= kCompactModules ? 256 : 64;
  SeedShared<kWarps, kOwn, kList, kMapRows> seed;
  int32_t start[kMods];       // [S] = H
  int32_t sz[kMods];
  float zmin[kMods];
  float zmax[kMods];
  uint32_t inflight[kMods];   // forwarding f: entries at its start | entries at its start and pushed << 16
  uint8_t flags[kMods];       // kSorted, kDeadTail
  uint32_t tracks[kWarps];    // tracks of each warp
  uint32_t status;
  uint32_t considered, kept;  // learned seeding: doublets scored / kept
  unsigned long long out_first;
  int32_t next_event;
  __device__ __forceinline__ int num(int m) const { return start[m + 1] - start[m]; }
};

struct EventView {
  const SearchParams* p;    // the kernel's parameters (constant memory)
  int S, H;
  int event;
  // the arena: x, y, z, windows (per hit {h1 first | h1 last << 16, h2 first
  // | h2 last << 16}) and flags at multiples of one stride P
  uint8_t* arena;
  uint32_t P;
  bool tame;                // every module x-sorted and every coordinate within kMaxCoordinate
  bool plain;               // plain geometry: tame, one z per module, ascending
  const MlpFrag* mlp;       // learned seeding: weights in shared memory
  bool sparse;              // learned seeding: only doublets that some h2 is near are scored
  __device__ __forceinline__ float* xs() const { return reinterpret_cast<float*>(arena); }
  __device__ __forceinline__ float* ys() const { return reinterpret_cast<float*>(arena + P); }
  __device__ __forceinline__ float* zs() const { return reinterpret_cast<float*>(arena + 2u * P); }
  __device__ __forceinline__ uint2* wins() const { return reinterpret_cast<uint2*>(arena + 3u * P); }
  __device__ __forceinline__ uint8_t* useds() const { return arena + 5u * P; }
  // scratch by row: tracklets {h0, h1, h2, 0}, tracks, weak list, entries
  uint4* tracklets;
  velo_track* tracks;
  uint32_t* weak;
  uint4* entry_words;
  float4* entry_lines;
  int y_lanes, narrow;
};

// Hits of a module that the general seedings look at at once: their loads and
// distances do not depend on one another.  One after another, with a branch on
// each, the walk of an unsorted module's windows waits some 100 cycles a hit: 100
// unsorted events of 1,240 hits 7.0 -> 3.3 ms with 64 threads, 2.3 -> 1.6 ms
// with 512 (two or eight at once: 4.1 ms with 64 threads).
constexpr int kAtOnce = 4;

// First index i in [lo, hi) with x[i] > c, for non-decreasing x.
__device__ __forceinline__ int first_gt(const float* x, int lo, int hi, float c) {
  while (lo < hi) {
    const int mid = (lo + hi) >> 1;
    if (x[mid] > c) hi = mid; else lo = mid + 1;
  }
  return lo;
}

// Sub-range [lo, hi) of [lo0, hi0) on a sorted module outside which no hit
// can satisfy |fl(xp - x)| < tol for any predicted xp in [xl, xh].  The upper
// end is usually a few hits past the lower one: walk, then bisect.
// x_first = x[lo0] and x_last = x[hi0 - 1] are passed in (any value when
// lo0 == hi0), so that a caller can load them early.
__device__ __forceinline__ void narrow_range_ends(const float* x, int lo0, int hi0, float x_first, float x_last,
                                                  float xl, float xh, float tol, int* lo, int* hi) {
  const float margin = fadd(0.01f, fmul(1e-5f, fadd(fabsf(xl), fabsf(xh))));
  const float lt = fsub(fsub(xl, tol), margin);
  const float ht = fadd(fadd(xh, tol), margin);
  if (isfinite(lt) && isfinite(ht)) {
    // both ends first: a prediction beyond either end of the module (a track
    // tried on the other detector half) is settled without the bisection,
    // with the bisection's own result
    if (lo0 < hi0 && (x_last <= lt || x_first > ht)) {
      *lo = *hi = x_first > ht ? lo0 : hi0;
      return;
    }
    const int l = first_gt(x, lo0, hi0, lt);
    int h = l;
    const int walk_end = min(hi0, l + 8);
    while (h < walk_end && !(x[h] > ht)) ++h;
    if (h == walk_end && h < hi0) h = first_gt(x, h, hi0, ht);
    *lo = l;
    *hi = h;
  } else {
    *lo = lo0;
    *hi = hi0;
  }
}

__device__ __forceinline__ void narrow_range(const float* x, int lo0, int hi0, float xl, float xh, float tol,
                                             int* lo, int* hi) {
  float x_first = 0.f, x_last = 0.f;
  if (lo0 < hi0) {   // two independent loads
    x_first = x[lo0];
    x_last = x[hi0 - 1];
  }
  narrow_range_ends(x, lo0, hi0, x_first, x_last, xl, xh, tol, lo, hi);
}

// ---------------------------------------------------------------------------
// Candidate windows of hit h on module f (Kernel.cl:50-178), stored relative
// to the start of module f-2 (0xffff = none).
template <class Shared>
__device__ void compute_windows(const EventView& ev, const Shared& s, int h, int f) {
  const int s2 = f - 2;
  const bool proc_h2 = f <= ev.S - 3;
  const int st2 = s.start[s2], n2 = s.num(s2);
  const float x0 = ev.xs()[h], z0 = ev.zs()[h];
  const float* x2 = ev.xs() + st2;
  const float* z2 = ev.zs() + st2;
  const bool sorted = ev.narrow && (s.flags[s2] & kSorted);
  uint32_t r1f = kNone16, r1l = kNone16, r2f = kNone16, r2l = kNone16;

  // h1 window: first hit with |x1-x0| < 0.7|z1-z0|, then the first later hit
  // that fails it (Kernel.cl:115-135,161-165).
  {
    int lo = 0, hi = n2;
    if (sorted && n2 > 0) {
      const float da = fabsf(fsub(s.zmin[s2], z0));
      const float db = fabsf(fsub(s.zmax[s2], z0));
      const float D = fmul(kMaxXSlopeCandidates, fmaxf(da, db));   // >= every hit's dxmax
      narrow_range(x2, 0, n2, x0, x0, D, &lo, &hi);
    }
    if (sorted && n2 > 0 && s.zmin[s2] == s.zmax[s2]) {
      // one z on the module: dxmax is the same for every hit, and
      // d = fl(x2 - x0) is non-decreasing in x2, so the hits passing
      // |d| < dxmax are exactly [A, B): A = first with d > -dxmax, B = first
      // with d >= dxmax -- the scan's first pass and first later failure
      const float dxmax = fmul(kMaxXSlopeCandidates, fabsf(fsub(z2[0], z0)));
      int a = lo, b = hi;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (fsub(x2[mid], x0) > -dxmax) b = mid; else a = mid + 1;
      }
      const int A = a;
      b = hi;
      while (a < b) {
        const int mid = (a + b) >> 1;
        if (!(fsub(x2[mid], x0) < dxmax)) b = mid; else a = mid + 1;
      }
      if (A < a) {
        r1f = (uint32_t)A;
        r1l = (uint32_t)a;   // a == hi: hit `hi` provably fails, or hi is the end
      }
    } else {
      bool found = false;
      for (int e = lo; e < hi; ++e) {
        const float h_dist = fabsf(fsub(z2[e], z0));
        const float dxmax = fmul(kMaxXSlopeCandidates, h_dist);
        const bool tol = fabsf(fsub(x2[e], x0)) < dxmax;
        if (!found) {
          if (tol) { found = true; r1f = (uint32_t)e; }
        } else if (!tol) {
          r1l = (uint32_t)e;
          break;
        }
      }
      if (found && r1l == kNone16) r1l = (uint32_t)hi;   // hit `hi` provably fails, or hi is the end
    }
  }

  // h2 window for h taken as the h1 of a seed on f+2 (Kernel.cl:85-102,137-150).
  if (proc_h2) {
    const float fz0 = __int2float_rn(s.sz[f + 2]);
    const float fz2 = __int2float_rn(s.sz[s2]);
    const float h_dist = fabsf(fsub(z0, fz0));
    const float dxmax = fmul(kMaxXSlopeCandidates, h_dist);
    const float x0_min = fsub(x0, dxmax);
    const float x0_max = fadd(x0, dxmax);
    const float z2_tz = fdiv(fsub(fz2, fz0), fsub(z0, fz0));
    const float xmin_h2 = fsub(fadd(x0_max, fmul(fsub(x0, x0_max), z2_tz)), kToleranceCandidates);
    const float xmax_h2 = fadd(fadd(x0_min, fmul(fsub(x0, x0_min), z2_tz)), kToleranceCandidates);
    if (sorted) {   // `x > c` is monotone on a non-decreasing module: exact
      const int a = first_gt(x2, 0, n2, xmin_h2);
      if (a < n2) {
        r2f = (uint32_t)a;
        r2l = (uint32_t)first_gt(x2, a + 1, n2, xmax_h2);
      }
    } else {
      bool found = false;
      for (int e = 0; e < n2; ++e) {
        if (!found) {
          if (x2[e] > xmin_h2) { found = true; r2f = (uint32_t)e; }
        } else if (x2[e] > xmax_h2) {
          r2l = (uint32_t)e;
          break;
        }
      }
      if (found && r2l == kNone16) r2l = (uint32_t)n2;
    }
  }
  ev.wins()[h] = make_uint2(r1f | (r1l << 16), r2f | (r2l << 16));
}

// ---------------------------------------------------------------------------
// Work split.  Seeding module f touches modules f, f-2 and f-4 only, so the
// two parities of modules are seeded by different warps: half of the CTA's
// warps seed the modules f = S-1, S-3, ..., the other half S-2, S-4, ...
// Each warp owns the tracks-to-follow entries of its own seeds, forwards them
// in every iteration (onto modules of either parity), and keeps its
// tracklets, tracks and weak list in its own rows, so none of them needs an
// atomic or a barrier.  What the warps share is the hits' used flags:
//  * an extension in the forwarding of iteration f marks a hit of f-4, first
//    read by the seeding of f-2;
//  * a tracklet's promotion marks hits of its own parity; a seeding of that
//    parity must see the promotions before it and none after it: both are
//    the warp's own (or, with more than two warps, its group's), in order.
// So the warps meet once per two iterations: when iterations f and f-1 begin,
// every forwarding down to f+1 has been done by all of them.
//
// All warps forwarding and seeding each module together takes two barriers per
// iteration, shared-memory counters, and spreads each module's 4 unused h0s
// over the warps.  With 64 threads the split runs one warp per parity: 18 %
// fewer warp instructions, 21 % less time for 10,000 events of 1,160 hits, 31 %
// for one event.
struct Worker {
  uint32_t row;        // first of its scratch rows
  uint32_t n, tracklets, tracks, weak;
  // warp in the CTA; the parity it seeds, (S-1-f) & 1 (one warp: every f); its
  // place among the `of` warps of that parity
  __device__ __forceinline__ static int warp() { return threadIdx.x >> 5; }
  __device__ __forceinline__ static bool alone() { return blockDim.x == 32; }
  __device__ __forceinline__ static int parity() { return warp() & 1; }
  __device__ __forceinline__ static int idx() { return warp() >> 1; }
  __device__ __forceinline__ static int of() { return alone() ? 1 : (int)blockDim.x >> 6; }
};

// An entry is {word, last hit | iteration it was found in << 24, z of the
// previous hit, z of the last hit} and the line through the last two hits {x
// and y of the previous hit, x and y slopes}.  Bit 31 of the word marks a
// tracklet (3 hits, number = its row among the warp's tracklets), as in the
// reference (Kernel.cl:222-225,566); otherwise bits 23-27 are the track's hit
// count and bits 0-22 its row among the warp's tracks.   The iteration says
// how many modules were skipped (the reference counts them in bits 28-30), so
// an entry that finds nothing stays as it is, where it is.  The line is
// computed when the hit is found: forwarding reads no hit, track or tracklet
// before its fit.
constexpr uint32_t kEntryNumber = 0x007FFFFFu;
constexpr uint32_t kEntryCountShift = 23;
constexpr uint32_t kEntryHit = 0x00FFFFFFu;   // 255 modules of 16,383 hits: 22 bits
constexpr uint32_t kEntryIterationShift = 24;

__device__ __forceinline__ unsigned lanemask_lt() { return (1u << (threadIdx.x & 31)) - 1u; }

// The line through hit a and then hit b (z differing), as the reference
// takes it from a track's last two hits (Kernel.cl:253-257).  td = 1 / (zb - za).
__device__ __forceinline__ float4 line_through(float xa, float ya, float xb, float yb, float td) {
  return make_float4(xa, ya, fmul(fsub(xb, xa), td), fmul(fsub(yb, ya), td));
}

// The scatter cut (dx^2 + dy^2) / dz^2 < kMaxScatter bounds |dx| and |dy| by
// sqrt(kMaxScatter) |dz| = 0.004 |dz|; 1 % more covers the rounding of the
// reference's products.  At the usual 25 mm between modules that is 0.1 mm,
// a sixth of kTolerance, so far fewer hits are tried.
constexpr float kScatterReach = 0.00404f;
// With |dz| at least this, 1 / dz squared stays far from overflow, so a fit
// outside the cuts is finite and need not be evaluated.
constexpr float kMinDz = 1e-3f;
// Plain-geometry events (EventView::plain): every module x-sorted and of one
// z, the modules' z ascending by more than kMinGap, every coordinate within
// kMaxCoordinate of the origin (mm).  A line through hits of two modules then
// predicts one point on a module, below 4e9, its fits with the module's hits
// are finite, and where the point is near a hit its sum with a reach is
// rounded by less than kRounding.
constexpr float kMaxCoordinate = 1e4f;
constexpr float kMinGap = 0.1f;
constexpr float kRounding = 0.01f;

// Appends the tracklets {h0, h1, h2} of the lanes with `win`, seeded in
// iteration f, to the warp's rows and entries (Kernel.cl:550-567).
__device__ __forceinline__ void append_tracklets(const EventView& ev, Worker& w, bool win, uint32_t h0, uint32_t h1,
                                                 uint32_t h2, int f) {
  const unsigned m = __ballot_sync(kFull, win);
  if (m == 0) return;
  if (win) {
    const uint32_t r = (uint32_t)__popc(m & lanemask_lt());
    const uint32_t tp = w.tracklets + r, i = w.row + w.n + r;
    ev.tracklets[w.row + tp] = make_uint4(h0, h1, h2, 0u);
    const float z1 = ev.zs()[h1], z2 = ev.zs()[h2];
    const float4 line =
        line_through(ev.xs()[h1], ev.ys()[h1], ev.xs()[h2], ev.ys()[h2], fdiv(1.0f, fsub(z2, z1)));
    ev.entry_words[i] = make_uint4(kTrackletFlag | tp, h2 | ((uint32_t)f << kEntryIterationShift),
                                     __float_as_uint(z1), __float_as_uint(z2));
    ev.entry_lines[i] = line;
  }
  w.tracklets += __popc(m);
  w.n += __popc(m);
}

// Barrier of the warps of one parity.
template <int kWarps>
__device__ __forceinline__ void group_sync(const Worker& w) {
  if (kWarps <= 2 || w.of() == 1)
    __syncwarp();
  else if (w.parity() == 0)   // constant names: a variable one reserves all 16 of the CTA, and 4 CTAs fill an SM
    asm volatile("bar.sync 1, %0;" ::"r"(32 * w.of()) : "memory");
  else
    asm volatile("bar.sync 2, %0;" ::"r"(32 * w.of()) : "memory");
}

// The rows of a warp: as many as it can seed h0s.  A module's hits are dealt
// by rank within blocks of 32 to the warps of its parity (see active_h0s).
template <class Shared>
__device__ __forceinline__ uint32_t first_row(const Shared& s, const Worker& w, int S) {
  if (w.alone()) return 0u;
  int rows = 0;
  const int per = 32 / w.of();
  for (int m = threadIdx.x & 31; m < S; m += 32) {
    const int n = s.num(m), rem = n & 31, parity = (S - 1 - m) & 1;
    if (parity == w.parity())
      rows += (n >> 5) * per * w.idx() + rem / w.of() * w.idx() + min(rem % w.of(), w.idx());
    else if (w.parity() == 1)
      rows += n;
  }
  return (uint32_t)__reduce_add_sync(kFull, rows);
}

// Per-warp counts of entries are summed in 16 bits: each is cut off well
// above VELO_TTF_MODULO, where the event is flagged in any case.
constexpr uint32_t kInflightMax = 2 * VELO_TTF_MODULO;

// The unused h0s of hits [block, block + 32) of module f (Kernel.cl:720-764)
// are dealt by rank to the warps of the module's parity; their number for
// this warp; its c-th is hit block + active[idx + c of].  A warp writes and
// reads its own ranks only.
__device__ __forceinline__ int active_h0s(const EventView& ev, const Worker& w, int st0, int n0, int block,
                                          uint8_t* active) {
  __syncwarp();   // the previous block's list has been read
  const int lane = threadIdx.x & 31;
  const bool unused = block + lane < n0 && !(ev.useds()[st0 + block + lane] & kUsed);
  const unsigned m = __ballot_sync(kFull, unused);
  const int rank = __popc(m & lanemask_lt()), total = __popc(m);
  if (unused && (rank & (w.of() - 1)) == w.idx()) active[rank] = (uint8_t)lane;
  __syncwarp();
  return (total + w.of() - 1 - w.idx()) / w.of();
}

// The best hit of module m4 for an entry (fitHitToTrack, Kernel.cl:15-35, first
// minimum over the module's hits), any module and any line: its place in the
// module or -1, its z, and the fit's 1 / (z2 - z1).
struct Fit {
  int k;
  float z, den;
  bool degenerate;
};

template <class Shared>
__device__ __forceinline__ Fit fit_any(const EventView& ev, const Shared& s, int m4, float4 line, float h0z,
                                       float h1z) {
  const int st4 = s.start[m4], n4 = s.num(m4);
  const float zmin4 = s.zmin[m4], zmax4 = s.zmax[m4];
  const float* x4 = ev.xs() + st4;
  const float* y4 = ev.ys() + st4;
  const float* z4 = ev.zs() + st4;
  int k = 0;
  float ht = __int_as_float(0x7f800000);   // +inf: every hit from k on is tried
  bool all_fits = true;                    // every fit is evaluated, for its finiteness
  if (ev.narrow && (s.flags[m4] & kSorted) && n4 > 0) {
    const float dza = fsub(zmin4, h0z), dzb = fsub(zmax4, h0z);
    const float xa = fadd(line.x, fmul(line.z, dza)), xb = fadd(line.x, fmul(line.z, dzb));
    const float d_lo = fsub(zmin4, h1z), d_hi = fsub(zmax4, h1z);
    const float reach = fmul(kScatterReach, fmaxf(fabsf(d_lo), fabsf(d_hi)));
    const float ymax = fadd(fabsf(line.y), fmul(fabsf(line.w), fmaxf(fabsf(dza), fabsf(dzb))));
    // the fits outside the cuts are known to be finite
    const bool tame = ev.tame && (d_lo > kMinDz || d_hi < -kMinDz) && ymax < 1e15f;
    const float tol = tame ? fminf(kTolerance, reach) : kTolerance;
    const float xl = fminf(xa, xb), xh = fmaxf(xa, xb);
    const float margin = fadd(0.01f, fmul(1e-5f, fadd(fabsf(xl), fabsf(xh))));
    const float lt = fsub(fsub(xl, tol), margin);
    const float h = fadd(fadd(xh, tol), margin);
    if (isfinite(xa) && isfinite(xb) && isfinite(lt) && isfinite(h)) {
      ht = h;
      all_fits = !tame;
      k = x4[n4 - 1] <= lt || x4[0] > ht ? n4 : first_gt(x4, 0, n4, lt);
    }
  }
  // The scatter's 1/(z2 - z1) depends only on z2 here: it is recomputed only
  // when z2's bit pattern changes (same operands, same rounded value).
  Fit fit{-1, 0.f, 0.f, false};
  float best = FLT_MAX;
  uint32_t zc = 0x7fc00001u;   // bit pattern of the z2 the cached factor belongs to (none yet)
  float den = 0.f;
  for (; k < n4; ++k) {
    const float h2x = x4[k];
    if (h2x > ht) break;
    const float h2z = z4[k];
    const float dz = fsub(h2z, h0z);
    const float dx = fabsf(fsub(fadd(line.x, fmul(line.z, dz)), h2x));
    const float dy = fabsf(fsub(fadd(line.y, fmul(line.w, dz)), y4[k]));
    const bool near = dx < kTolerance && dy < kTolerance;
    if (near || all_fits) {
      if (__float_as_uint(h2z) != zc) {
        zc = __float_as_uint(h2z);
        den = fdiv(1.f, fsub(h2z, h1z));
      }
      const float scatter = fmul(fmul(fadd(fmul(dx, dx), fmul(dy, dy)), den), den);
      if (near && scatter < kMaxScatter) {
        if (scatter < best) {
          best = scatter;
          fit.k = k;
          fit.z = h2z;
          fit.den = den;
        }
      } else if (!isfinite(scatter)) {
        fit.degenerate = true;   // the reference's `condition*scatter + !condition*MAX` is NaN here
      }
    }
  }
  return fit;
}

// Track forwarding of iteration f, onto module f-4 (Kernel.cl:210-367): the
// warp's entries, 32 at a time, kept in place or moved down over dropped ones.
// In plain geometry one factor 1 / (z2 - z1) serves all hits of the module,
// and only the hits within reach of the predicted x are fitted.
template <bool kPlainGeometry, class Shared>
__device__ __forceinline__ void forward(const EventView& ev, Shared& s, Worker& w, int f) {
  if (w.n == 0) return;   // warp-uniform
  const int lane = threadIdx.x & 31, m4 = f - 4;
  const int st4 = s.start[m4], n4 = s.num(m4);
  const float z4 = s.zmin[m4];
  const float* x4 = ev.xs() + st4;
  const float* y4 = ev.ys() + st4;
  // the ends of module m4 (same addresses in every lane)
  float x4_first = 0.f, x4_last = 0.f;
  if (kPlainGeometry && n4 > 0) {
    x4_first = x4[0];
    x4_last = x4[n4 - 1];
  }
  const uint32_t n = w.n;
  uint32_t kept = 0;
  for (uint32_t i0 = 0; i0 < n; i0 += 32) {   // warp-uniform
    const uint32_t i = i0 + lane;
    bool keep = false, changed = false, promote = false, weak = false;
    uint4 en = make_uint4(0, 0, 0, 0);
    float4 line = make_float4(0.f, 0.f, 0.f, 0.f);
    uint32_t found = 0;
    if (i < n) {
      en = ev.entry_words[w.row + i];
      line = ev.entry_lines[w.row + i];
      const bool is_tracklet = (en.x & kTrackletFlag) != 0;
      const float h0z = __uint_as_float(en.z), h1z = __uint_as_float(en.w);
      int best_k = -1;
      float best_z = z4, best_den;
      if constexpr (kPlainGeometry) {
        const float d = fsub(z4, h1z), dz = fsub(z4, h0z);
        const float xp = fadd(line.x, fmul(line.z, dz)), yp = fadd(line.y, fmul(line.w, dz));
        const float tol = fadd(fminf(kTolerance, fmul(kScatterReach, fabsf(d))), kRounding);
        const float lt = fsub(xp, tol), ht = fadd(xp, tol);
        int k = n4;
        if (n4 > 0 && x4_last > lt && x4_first <= ht) k = first_gt(x4, 0, n4, lt);
        best_den = fdiv(1.f, d);
        float best = FLT_MAX;
        for (; k < n4; ++k) {
          const float h2x = x4[k];
          if (h2x > ht) break;
          const float dx = fabsf(fsub(xp, h2x)), dy = fabsf(fsub(yp, y4[k]));
          const float scatter = fmul(fmul(fadd(fmul(dx, dx), fmul(dy, dy)), best_den), best_den);
          if (dx < kTolerance && dy < kTolerance && scatter < kMaxScatter && scatter < best) {
            best = scatter;
            best_k = k;
          }
        }
      } else {
        const Fit fit = fit_any(ev, s, m4, line, h0z, h1z);
        best_k = fit.k;
        best_z = fit.z;
        best_den = fit.den;
        if (fit.degenerate) atomicOr(&s.status, VELO_EVENT_DEGENERATE);
      }

      if (best_k >= 0) {
        const uint32_t hits = is_tracklet ? 3u : (en.x >> kEntryCountShift) & 31u;
        if (hits >= VELO_MAX_TRACK_SIZE) {   // the reference writes past hits[24] here
          atomicOr(&s.status, VELO_EVENT_TRACK_OVERFLOW);
        } else {
          found = (uint32_t)(st4 + best_k);
          ev.useds()[found] = kUsed;
          // the entry's next line: through its last hit and the one found, whose
          // 1 / (z2 - z1) is the fit's own
          const uint32_t h1 = en.y & kEntryHit;
          line = line_through(ev.xs()[h1], ev.ys()[h1], x4[best_k], y4[best_k], best_den);
          keep = changed = true;
          promote = is_tracklet;   // third -> fourth hit: a track is made below
          if (!is_tracklet) {
            velo_track& t = ev.tracks[w.row + (en.x & kEntryNumber)];
            t.hits[hits] = found;
            t.hitsNum = hits + 1;
            en.x += 1u << kEntryCountShift;
          }
          en.y = found | ((uint32_t)f << kEntryIterationShift);
          en.z = en.w;
          en.w = __float_as_uint(best_z);
        }
      } else {
        // dropped when it has skipped more than kMaxSkippedModules before this one
        keep = (en.y >> kEntryIterationShift) - 1u - (uint32_t)f <= kMaxSkippedModules;
        weak = !keep && is_tracklet;
      }
    }
    // new tracks (Kernel.cl:324-337); the words past the last hit are cleared
    // when the track is written out
    const unsigned pm = __ballot_sync(kFull, promote);
    if (promote) {
      const uint4 tl = ev.tracklets[w.row + (en.x & kEntryNumber)];
      ev.useds()[tl.x] = kUsed;
      ev.useds()[tl.y] = kUsed;
      ev.useds()[tl.z] = kUsed;
      const uint32_t tn = w.tracks + (uint32_t)__popc(pm & lanemask_lt());
      uint32_t* t = reinterpret_cast<uint32_t*>(&ev.tracks[w.row + tn]);
      t[0] = 4; t[1] = tl.x; t[2] = tl.y; t[3] = tl.z; t[4] = found;
      en.x = tn | (4u << kEntryCountShift);
    }
    w.tracks += __popc(pm);
    // three-hit tracklets that ran out of skips (Kernel.cl:359-363)
    const unsigned wm = __ballot_sync(kFull, weak);
    if (weak) ev.weak[w.row + w.weak + (uint32_t)__popc(wm & lanemask_lt())] = en.x & kEntryNumber;
    w.weak += __popc(wm);
    // entries to follow in the next iteration (Kernel.cl:344-355): every lane
    // has read its own, and slots below i0 are done with
    const unsigned km = __ballot_sync(kFull, keep);
    const uint32_t to = kept + (uint32_t)__popc(km & lanemask_lt());
    if (keep && (changed || to != i)) {
      ev.entry_words[w.row + to] = en;
      ev.entry_lines[w.row + to] = line;
    }
    kept += __popc(km);
    __syncwarp();
  }
  w.n = kept;
  if (ev.H > VELO_TTF_MODULO / 2 && lane == 0)   // smaller events cannot overrun the reference's buffer
    atomicAdd(&s.inflight[f], min(n, kInflightMax) | (min(n + kept, kInflightMax) << 16));
}

// Features of an (h0, h1) doublet seen by the learned seeding (and recorded
// as training data): slopes, h0 radius and azimuth, module, predicted x / y
// at module f-4, z gap, h2 candidates in the exact window, and the y-slope
// cut margin.  Plain FP32; the features steer pruning, not the cuts.  The
// h0 terms (radius, azimuth, module, 1 / dymax) are computed once per h0 by
// h0_features; dz_inv is the seeding's own 1 / (z1 - z0).
struct H0Features {
  float r, phi, module, inv_dymax;
};

__device__ __forceinline__ H0Features h0_features(float h0x, float h0y, int module, int n_modules, float dymax) {
  H0Features g;
  g.r = sqrtf(h0x * h0x + h0y * h0y) * (1.f / 42.f);
  g.phi = atan2f(h0y, h0x) * 0.31830988f;
  g.module = (float)module / (float)n_modules;
  g.inv_dymax = 1.f / dymax;
  return g;
}

__device__ __forceinline__ void doublet_features(float* f, const H0Features& g, float h0x, float h0y, float h0z,
                                                 float h1x, float h1y, float h1z, float dz_inv, float zmid4,
                                                 int h2_window) {
  const float tx = (h1x - h0x) * dz_inv, ty = (h1y - h0y) * dz_inv;
  f[0] = 5.f * tx;
  f[1] = 5.f * ty;
  f[2] = g.r;
  f[3] = g.phi;
  f[4] = g.module;
  f[5] = (h0x + tx * (zmid4 - h0z)) * (1.f / 42.f);
  f[6] = (h0y + ty * (zmid4 - h0z)) * (1.f / 42.f);
  f[7] = (h1z - h0z) * 0.01f;
  f[8] = (float)h2_window * (1.f / 32.f);
  f[9] = fabsf(h1y - h0y) * g.inv_dymax;
}

constexpr int kPlain = 0;    // the reference's seeding
constexpr int kDump = 1;     // plain, recording sampled doublets as training data
constexpr int kLearned = 2;  // MLP-pruned seeding

// Lane constants of the seeding ballots, per event.  With G lanes per h0 (a
// group; G = 32: the whole warp), lane j of a group takes, in chunk c, h1
// element e = G c + j of its h0, which belongs to the reference's Y-lane
// e mod Y.
struct SeedLanes {
  uint32_t below;      // lanes of my group below me whose element shares my Y-lane in a chunk
  uint32_t same_all;   // G < 32 (Y divides G): every lane of my group that shares my Y-lane
  uint32_t lane_mod;   // (lane mod G) mod Y: my Y-lane in chunk 0
};

__device__ __forceinline__ SeedLanes seed_lanes_of(int G, uint32_t Y) {
  SeedLanes sl;
  const int lane = threadIdx.x & 31;
  const int jl = lane & (G - 1), gbase = lane - jl;
  sl.below = 0;
  for (int j = jl - (int)Y; j >= 0; j -= (int)Y) sl.below |= 1u << (gbase + j);
  sl.same_all = 0;
  for (int j = (int)((uint32_t)jl % Y); j < G; j += (int)Y) sl.same_all |= 1u << (gbase + j);
  sl.lane_mod = (uint32_t)jl % Y;
  return sl;
}

// Features and MLP of the learned seeding for the warp's doublets: lanes
// with score == false pass zeros and ignore the result.  All 32 lanes call it
// together.  score_doublets keeps it out of line where the windows are walked,
// so that the loop keeps its registers wherever nothing is scored.
static __device__ __forceinline__ float2 score_batch(const MlpFrag* mlp, bool score, float h0x, float h0y, float h0z,
                                              float h1x, float h1y, float h1z, float dz_inv, float zmid4,
                                              int h2_window, int f, int n_modules, float dymax) {
  float feat[kMlpIn];
  if (score) {
    const H0Features g0 = h0_features(h0x, h0y, f, n_modules, dymax);
    doublet_features(feat, g0, h0x, h0y, h0z, h1x, h1y, h1z, dz_inv, zmid4, h2_window);
  } else {
#pragma unroll
    for (int q = 0; q < kMlpIn; ++q) feat[q] = 0.f;
  }
  float logit, width;
  mlp_eval_warp(*mlp, feat, &logit, &width);
  return make_float2(logit, width);
}

static __device__ __noinline__ float2 score_doublets(const MlpFrag* mlp, bool score, float h0x, float h0y, float h0z,
                                              float h1x, float h1y, float h1z, float dz_inv, float zmid4,
                                              int h2_window, int f, int n_modules, float dymax) {
  return score_batch(mlp, score, h0x, h0y, h0z, h1x, h1y, h1z, dz_inv, zmid4, h2_window, f, n_modules, dymax);
}

// Seeding of module f: h0 on f, h1 on f-2, h2 on f-4 (Kernel.cl:392-568
// with the unused-h0 gather of :720-764), G lanes per h0 (SeedLanes): the
// form that walks the candidate windows, for unsorted events, for learned
// seeding of several z per module, and for the training-data dump.
// G = 32: one warp per unused h0.  G = 8 or 16: a warp seeds 32 / G h0s at
// once and walks the chunks of its groups' h1 windows together, so every
// ballot and the groups' minimum reductions run with all lanes present; the
// host allows G < 32 only where Y divides G, so that a lane's Y-lane is the
// same in every chunk.
template <int kMode, int G, class Shared>
__device__ void seed_module(const EventView& ev, Shared& s, Worker& w, int f, const SeedLanes& sl) {
  constexpr int kShift = G == 8 ? 3 : G == 16 ? 4 : 5;
  constexpr int kGroups = 32 / G;
  static_assert(G == 8 || G == 16 || G == 32, "8, 16 or 32 lanes per h0");
  const int lane = threadIdx.x & 31;
  const int jl = lane & (G - 1);
  const int st0 = s.start[f], n0 = s.num(f);
  const int s1 = f - 2, m4 = f - 4;
  const int st1 = s.start[s1], st4 = s.start[m4], n4 = s.num(m4);
  const uint32_t Y = (uint32_t)ev.y_lanes;
  const uint32_t chunk_step = G == 32 ? 32u % Y : 0u;   // how far the Y-lanes turn per chunk
  const float s1_z = s.num(s1) > 0 ? ev.zs()[st1] : 0.f;   // Kernel.cl:420
  const bool narrow4 = ev.narrow && (s.flags[m4] & kSorted) && n4 > 0;
  const float zmin4 = s.zmin[m4], zmax4 = s.zmax[m4];
  const float* x4 = ev.xs() + st4;
  const float* y4 = ev.ys() + st4;
  const float* z4 = ev.zs() + st4;
  bool degenerate = false;
  // 1 / (z1 - z0) by bit patterns of (z0, z1): hits of a module share few z
  // values, so the division is rarely redone (same operands, same result)
  uint32_t zk0 = 0x7fc00001u, zk1 = 0x7fc00001u;
  float dz_inv_cached = 0.f;

  uint8_t* active = s.seed.active[w.parity()];
  for (int block = 0; block < n0; block += 32)                    // warp-uniform
  for (int c0 = 0, mine = active_h0s(ev, w, st0, n0, block, active); c0 < mine; c0 += kGroups) {
    int h0 = 0, n1 = 0;
    uint32_t f1 = 0;
    if (c0 + lane / G < mine) {
      h0 = st0 + block + active[w.idx() + (c0 + lane / G) * w.of()];
      const uint32_t w0 = ev.wins()[h0].x;
      f1 = w0 & 0xffffu;
      if (f1 != kNone16) n1 = (int)(w0 >> 16) - (int)f1;
    }
    const int c_end = G * (int)__reduce_max_sync(kFull, (uint32_t)((n1 + G - 1) >> kShift));
    if (c_end == 0) continue;                           // warp-uniform
    float h0x = 0.f, h0y = 0.f, h0z = 0.f;
    if (n1 > 0) {
      h0x = ev.xs()[h0];
      h0y = ev.ys()[h0];
      h0z = ev.zs()[h0];
    }
    const float dymax = fmul(kMaxYSlope, fabsf(fsub(s1_z, h0z)));
    H0Features g0{};
    if constexpr (kMode == kDump) g0 = h0_features(h0x, h0y, f, ev.S, dymax);
    unsigned long long best = ~0ull;
    uint32_t dead_lanes = 0;                         // G = 32: Y-lanes already stopped (bit per lane)
    bool lane_dead = false;                          // G < 32: my Y-lane has stopped
    uint32_t chunk_mod = 0;
    for (int c = 0; c < c_end; c += G) {
      const int e = c + jl;
      const bool in = e < n1;
      uint32_t ly = sl.lane_mod + chunk_mod;
      if (ly >= Y) ly -= Y;
      const int h1 = st1 + (int)f1 + e;
      // everything the cuts read about h1, loaded at once (one round trip)
      uint32_t w1 = 0;
      uint8_t u1 = 1;
      float h1x = 0.f, h1y = 0.f, h1z = 0.f;
      if (in) {
        w1 = ev.wins()[h1].y;
        u1 = ev.useds()[h1] & kUsed;
        h1x = ev.xs()[h1];
        h1y = ev.ys()[h1];
        h1z = ev.zs()[h1];
      }
      const bool dead = in && (w1 & 0xffffu) == kNone16;
      const unsigned dmask = __ballot_sync(kFull, dead);
      bool stopped;
      if constexpr (G == 32) {
        stopped = ((dmask & sl.below) != 0) || ((dead_lanes >> ly) & 1u);
        dead_lanes |= __reduce_or_sync(kFull, dead ? (1u << ly) : 0u);
        chunk_mod += chunk_step;
        if (chunk_mod >= Y) chunk_mod -= Y;
      } else {   // a lane's Y-lane is the same in every chunk
        stopped = (dmask & sl.below) != 0 || lane_dead;
        lane_dead = lane_dead || (dmask & sl.same_all) != 0;
      }
      bool cand = in && !dead && !stopped && !u1;
      if (cand) cand = fabsf(fsub(h1y, h0y)) < dymax;   // h2-independent term of Kernel.cl:509
      int a = (int)(w1 & 0xffffu), b = (int)(w1 >> 16);
      float tol = kTolerance;
      float dz_inverted = 0.f;
      if (cand) {
        if (__float_as_uint(h1z) != zk1 || __float_as_uint(h0z) != zk0) {
          zk0 = __float_as_uint(h0z);
          zk1 = __float_as_uint(h1z);
          dz_inv_cached = fdiv(1.f, fsub(h1z, h0z));
        }
        dz_inverted = dz_inv_cached;
      }
      if constexpr (kMode == kDump) {
        if (cand) {
          float feat[kMlpIn];
          doublet_features(feat, g0, h0x, h0y, h0z, h1x, h1y, h1z, dz_inverted, 0.5f * (zmin4 + zmax4), b - a);
          uint32_t hs = (uint32_t)ev.event * 0x9E3779B1u ^ (uint32_t)h0 * 0x85EBCA77u ^ (uint32_t)h1 * 0xC2B2AE3Du;
          hs ^= hs >> 15;
          hs *= 0x2C1B3C6Du;
          hs ^= hs >> 12;
          if (hs % max(ev.p->dump_keep, 1u) == 0u) {
            const unsigned long long k = atomicAdd(ev.p->dump_count, 1ull);
            if (k < ev.p->dump_capacity) {
#pragma unroll
              for (int q = 0; q < kMlpIn; ++q) ev.p->dump_features[k * kMlpIn + q] = feat[q];
              ev.p->dump_ids[3 * k + 0] = (uint32_t)ev.event;
              ev.p->dump_ids[3 * k + 1] = (uint32_t)h0;
              ev.p->dump_ids[3 * k + 2] = (uint32_t)h1;
            }
          }
        }
      }
      if constexpr (kMode == kLearned) {
        // only doublets with a wide exact h2 window are worth scoring
        const bool score = cand && b - a >= ev.p->learned_min_window;
        bool keep = true;
        if (__any_sync(kFull, score)) {             // the warp scores its doublets together
          const float2 r = score_doublets(ev.mlp, score, h0x, h0y, h0z, h1x, h1y, h1z, dz_inverted,
                                          0.5f * (zmin4 + zmax4), b - a, f, ev.S, dymax);
          if (score) {
            keep = r.x >= ev.p->keep_threshold;
            tol = fminf(kTolerance, fmaxf(r.y, 0.f) + ev.p->window_margin);
          }
        }
        // keep-rate bookkeeping for the guard: the scored doublets
        const unsigned mc = __ballot_sync(kFull, score), mk = __ballot_sync(kFull, score && keep);
        if (lane == 0 && mc) {
          atomicAdd(&s.considered, (uint32_t)__popc(mc));
          atomicAdd(&s.kept, (uint32_t)__popc(mk));
        }
        cand = cand && keep;
      }
      if (!cand) continue;
      const float ddx = fsub(h1x, h0x), ddy = fsub(h1y, h0y);
      if (narrow4) {
        const float xa = fadd(h0x, fmul(ddx, fmul(fsub(zmin4, h0z), dz_inverted)));
        const float xb = fadd(h0x, fmul(ddx, fmul(fsub(zmax4, h0z), dz_inverted)));
        if (isfinite(xa) && isfinite(xb) && a < b) {
          int lo, hi;
          narrow_range(x4, a, b, fminf(xa, xb), fmaxf(xa, xb), tol, &lo, &hi);
          a = lo;
          b = hi;
        }
      }
      float lbest = FLT_MAX;
      int lk = -1;
      uint32_t zc = 0x7fc00001u;
      float den = 0.f;
      for (int k0 = a; k0 < b; k0 += kAtOnce) {
        float dx[kAtOnce], dy[kAtOnce], z2[kAtOnce];
        uint32_t near = 0;
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
          const int k = min(k0 + q, b - 1);
          z2[q] = z4[k];
          const float z2_tz = fmul(fsub(z2[q], h0z), dz_inverted);
          dx[q] = fsub(fadd(h0x, fmul(ddx, z2_tz)), x4[k]);
          dy[q] = fsub(fadd(h0y, fmul(ddy, z2_tz)), y4[k]);
          near |= (uint32_t)(k0 + q < b && fabsf(dx[q]) < kTolerance && fabsf(dy[q]) < kTolerance) << q;
        }
        if (near == 0) continue;
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) {
          if (!((near >> q) & 1u)) continue;
          if (__float_as_uint(z2[q]) != zc) {   // the factor depends on z2 only (per h1)
            zc = __float_as_uint(z2[q]);
            den = fdiv(1.f, fsub(z2[q], h1z));
          }
          const float scatter = fmul(fmul(fadd(fmul(dx[q], dx[q]), fmul(dy[q], dy[q])), den), den);
          if (scatter < kMaxScatter) {
            if (scatter < lbest) { lbest = scatter; lk = k0 + q; }
          } else if (!isfinite(scatter)) {
            degenerate = true;
          }
        }
      }
      if (lk >= 0) {
        const unsigned long long key = ((unsigned long long)__float_as_uint(lbest) << 32) |
                                       ((unsigned long long)ly << 28) | ((unsigned long long)e << 14) |
                                       (unsigned long long)lk;
        best = key < best ? key : best;
      }
    }
    // the group's 64-bit minimum as two 32-bit minima: the high words, then
    // the low words of the lanes that hold the minimal high word
    const uint32_t hi = (uint32_t)(best >> 32);
    uint32_t hmin, lmin;
    if constexpr (G == 32) {
      hmin = __reduce_min_sync(kFull, hi);
      lmin = __reduce_min_sync(kFull, hi == hmin ? (uint32_t)best : 0xffffffffu);
    } else {   // butterflies inside each group
      hmin = hi;
#pragma unroll
      for (int o = G >> 1; o > 0; o >>= 1) hmin = min(hmin, __shfl_xor_sync(kFull, hmin, o));
      lmin = hi == hmin ? (uint32_t)best : 0xffffffffu;
#pragma unroll
      for (int o = G >> 1; o > 0; o >>= 1) lmin = min(lmin, __shfl_xor_sync(kFull, lmin, o));
    }
    best = ((unsigned long long)hmin << 32) | lmin;
    // each group's first lane appends its tracklet
    const uint32_t h1 = (uint32_t)(st1 + (int)f1) + ((uint32_t)(best >> 14) & 0x3fffu);
    append_tracklets(ev, w, jl == 0 && best != ~0ull, (uint32_t)h0, h1,
                     (uint32_t)st4 + (uint32_t)(best & 0x3fffu), f);
  }
  if (degenerate) atomicOr(&s.status, VELO_EVENT_DEGENERATE);
}

// The candidate windows of every hit (all threads of the CTA).
template <class Shared>
__device__ __noinline__ void fill_windows(const EventView ev, const Shared& s) {
  // windows of modules 0..3 stay empty (Kernel.cl:104 gates the body on f >= 4)
  const int hbeg = ev.S >= 5 ? s.start[4] : ev.H;
  for (int i = threadIdx.x; i < hbeg; i += blockDim.x) ev.wins()[i] = make_uint2(0xffffffffu, 0xffffffffu);
  for (int h = hbeg + threadIdx.x; h < ev.H; h += blockDim.x) {
    int lo = 4, hi = ev.S - 1;   // last module whose start is <= h
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (s.start[mid] <= h) lo = mid; else hi = mid - 1;
    }
    compute_windows(ev, s, h, lo);
  }
}

// ---------------------------------------------------------------------------
// Pair seeding: the seeding of module f (h0 on f, h1 on f-2, h2 on f-4;
// Kernel.cl:392-568 with the gather of :720-764) for events whose modules are
// all x-sorted and whose coordinates are tame, with the results of
// seed_module.
//
// Of a module's hits few are still unused when it is seeded (4 of 24 at the
// ordinary pile-up), each with some 35 h1 candidates, of which one pair in 20
// meets a hit of f-4.  So the unused h0s are gathered first, a warp lays the
// (h0, h1) pairs of its h0s end to end over its lanes, whatever the h0s'
// window lengths, and each pair only looks up the cell of its predicted
// (x, y) in a map of the cells that f-4's hits could be met from.  The pairs
// that pass are queued in shared memory and fitted 32 at a time.
//
// Against a group of 8 lanes per h0 walking its chunk of h1s and searching h2
// for every pair (seed_module) the kernel takes three quarters of the time for
// 10,000 events of 1,160 hits, a third for 4,000 events of 4,550.
//
// The windows need no table.  An h0's h1 window is bisected when the h0 is
// seeded (most hits never are); whether an h1 has an h2 window is the flag
// kDead; the h2 window itself is only tested on an h2 that passed the cuts.
// 32 columns of 1.3 mm span half a module's width, the rows its height.  With
// 256 rows instead of 64 half as many pairs pass that no hit is near (of 54,000
// pairs in an event of 4,400 hits 2,850 instead of 6,000, 800 of them met).
// A cell's number is the scaled coordinate rounded to an integer, taken from
// the low bits of a sum with 1.5 * 2^23 (one instruction, non-decreasing in the
// coordinate, and no conversion: those issue at a quarter of the rate).
__device__ __forceinline__ int map_cell(float v, float scale) {
  return __float_as_int(__fmaf_rn(v, scale, 12582912.f));
}
__device__ __forceinline__ int map_column(float x) { return map_cell(x, 1.f / 1.3125f); }
template <class Shared>
__device__ __forceinline__ int map_row(float y) {
  return map_cell(y, (float)Shared::kMapRows / 84.f);
}

template <class Shared>
__device__ __forceinline__ bool map_marked(const uint32_t* map, float x, float y) {
  return (map[map_row<Shared>(y) & (Shared::kMapRows - 1)] >> (map_column(x) & 31)) & 1u;
}

// Marks the cells from which hit i of module m4 could be met: a pair whose
// fit passes lies within 0.004 |z2 - z1| of it, and within kTolerance.  A
// cell index is non-decreasing in the coordinate, so the cells of both ends
// of the reach bracket the pair's; 0.01 mm covers the rounding.  Indices wrap
// around, which can only let a pair through.
template <class Shared>
__device__ __forceinline__ void mark_map(const EventView& ev, const Shared& s, uint32_t* map, int s1, int m4, int i) {
  const float dz = fabsf(fsub(s.zmin[m4], s.zmin[s1]));
  const float reach = fadd(fminf(kTolerance, fmul(kScatterReach, dz)), 0.01f);
  const float x = ev.xs()[s.start[m4] + i], y = ev.ys()[s.start[m4] + i];
  uint32_t bits = 0;
  const int c_end = map_column(fadd(x, reach)), r_end = map_row<Shared>(fadd(y, reach));
  for (int c = map_column(fsub(x, reach)); c <= c_end; ++c) bits |= 1u << (c & 31);
  for (int r = map_row<Shared>(fsub(y, reach)); r <= r_end; ++r) atomicOr(&map[r & (Shared::kMapRows - 1)], bits);
}

// The bounds of an h1's h2 window (Kernel.cl:85-102) for h1 at (x, z) on
// module s1: the window is the first hit of f-4 above *lo, up to the first
// later one above *hi.
__device__ __forceinline__ void h2_bounds(float x, float z, int sz0, int sz2, float* lo, float* hi) {
  const float fz0 = __int2float_rn(sz0), fz2 = __int2float_rn(sz2);
  const float dxmax = fmul(kMaxXSlopeCandidates, fabsf(fsub(z, fz0)));
  const float x_min = fsub(x, dxmax), x_max = fadd(x, dxmax);
  const float z2_tz = fdiv(fsub(fz2, fz0), fsub(z, fz0));
  *lo = fsub(fadd(x_max, fmul(fsub(x, x_max), z2_tz)), kToleranceCandidates);
  *hi = fadd(fadd(x_min, fmul(fsub(x, x_min), z2_tz)), kToleranceCandidates);
}

// An h1 of module m has no h2 window: no hit of module m-2 lies above its
// lower bound (modules 0-3 and the last two have no windows at all,
// Kernel.cl:104,137).
template <class Shared>
__device__ __forceinline__ bool h1_dead(const EventView& ev, const Shared& s, int m, int h) {
  if (m < 4 || m > ev.S - 3 || s.num(m - 2) == 0) return true;
  float lo, hi;
  h2_bounds(ev.xs()[h], ev.zs()[h], s.sz[m + 2], s.sz[m - 2], &lo, &hi);
  return !(ev.xs()[s.start[m - 2] + s.num(m - 2) - 1] > lo);
}

// The h1 window of an h0 at (x0, z0) on x-sorted module s1: the first hit
// with |x1 - x0| < 0.7 |z1 - z0| and the first later one that fails it
// (Kernel.cl:115-135,161-165).  With one z on the module the passing hits
// are a contiguous range, bisected at both ends at once.
template <class Shared>
__device__ __forceinline__ void h1_window(const EventView& ev, const Shared& s, int s1, float x0, float z0,
                                          int* first, int* last) {
  const int st = s.start[s1], n = s.num(s1);
  const float* x = ev.xs() + st;
  if (s.zmin[s1] == s.zmax[s1]) {
    const float dxmax = fmul(kMaxXSlopeCandidates, fabsf(fsub(s.zmin[s1], z0)));
    int a = 0, b = 0, len = n;   // a: first with x - x0 > -dxmax; b: first with x - x0 >= dxmax
    while (len > 0) {            // a and b keep ranges of one length, so both loads go out together
      const int half = len >> 1;
      const float da = fsub(x[a + half], x0), db = fsub(x[b + half], x0);
      if (!(da > -dxmax)) a += len - half;
      if (db < dxmax) b += len - half;
      len = half;
    }
    *first = a;
    *last = b;
  } else {
    int lo = 0, hi = n;
    const float D = fmul(kMaxXSlopeCandidates,
                         fmaxf(fabsf(fsub(s.zmin[s1], z0)), fabsf(fsub(s.zmax[s1], z0))));   // >= every hit's dxmax
    narrow_range(x, 0, n, x0, x0, D, &lo, &hi);
    const float* z = ev.zs() + st;
    auto passes = [&](int e) {
      return fabsf(fsub(x[e], x0)) < fmul(kMaxXSlopeCandidates, fabsf(fsub(z[e], z0)));
    };
    auto next = [&](int e, bool what) {   // the first from e on that does so
      for (; e < hi; e += kAtOnce) {
        uint32_t m = 0;
#pragma unroll
        for (int q = 0; q < kAtOnce; ++q) m |= (uint32_t)(passes(min(e + q, hi - 1)) == what) << q;
        if (m) return min(e + __ffs(m) - 1, hi);
      }
      return hi;
    };
    *first = next(lo, true);
    *last = next(*first, false);
  }
}

// h2 (hit k of module m4, at x) lies in the window of an h1 with bounds lo and
// hi: from the first hit above lo (that one even if it is above hi) up to the
// first later one above hi.
__device__ __forceinline__ bool in_h2_window(const float* x4, int k, float x, float lo, float hi) {
  return x > lo && (!(x > hi) || k == 0 || !(x4[k - 1] > lo));
}

// The best h2 of one (h0, h1) on module m4 (Kernel.cl:468-529) where the
// modules hold several z values or the fits may not be finite; h0 = {x, y, z}.
template <class Shared>
__device__ __forceinline__ Fit pair_fit_any(const EventView& ev, const Shared& s, int f, float h0x, float h0y, float h0z,
                                         int hit1, float* scatter_out) {
  const int m4 = f - 4, st4 = s.start[m4], n4 = s.num(m4);
  const float zmin4 = s.zmin[m4], zmax4 = s.zmax[m4];
  const float* x4 = ev.xs() + st4;
  const float* y4 = ev.ys() + st4;
  const float* z4 = ev.zs() + st4;
  const float h1x = ev.xs()[hit1], h1y = ev.ys()[hit1], h1z = ev.zs()[hit1];
  float lo, hi;
  h2_bounds(h1x, h1z, s.sz[f], s.sz[m4], &lo, &hi);
  const float dz_inverted = fdiv(1.f, fsub(h1z, h0z));
  const float ddx = fsub(h1x, h0x), ddy = fsub(h1y, h0y);
  const float xa = fadd(h0x, fmul(ddx, fmul(fsub(zmin4, h0z), dz_inverted)));
  const float xb = fadd(h0x, fmul(ddx, fmul(fsub(zmax4, h0z), dz_inverted)));
  const float d_lo = fsub(zmin4, h1z), d_hi = fsub(zmax4, h1z);
  const float reach = fmul(kScatterReach, fmaxf(fabsf(d_lo), fabsf(d_hi)));
  const float tol = d_lo > kMinDz || d_hi < -kMinDz ? fminf(kTolerance, reach) : kTolerance;
  const float xl = fminf(xa, xb), xh = fmaxf(xa, xb);
  const float margin = fadd(0.01f, fmul(1e-5f, fadd(fabsf(xl), fabsf(xh))));
  const float lt = fsub(fsub(xl, tol), margin);
  float ht = fadd(fadd(xh, tol), margin);
  int k = 0;
  if (isfinite(xa) && isfinite(xb) && isfinite(lt) && isfinite(ht))
    k = first_gt(x4, 0, n4, lt);
  else
    ht = __int_as_float(0x7f800000);   // +inf: every hit is tried
  Fit fit{-1, 0.f, 0.f, false};
  float best = FLT_MAX;
  uint32_t zc = 0x7fc00001u;
  float z2_tz = 0.f, den = 0.f;
  for (; k < n4; ++k) {
    const float h2x = x4[k];
    if (h2x > ht) break;
    const float h2z = z4[k];
    if (__float_as_uint(h2z) != zc) {   // both factors depend on h2z only (per h0, h1)
      zc = __float_as_uint(h2z);
      z2_tz = fmul(fsub(h2z, h0z), dz_inverted);
      den = fdiv(1.f, fsub(h2z, h1z));
    }
    const float dx = fsub(fadd(h0x, fmul(ddx, z2_tz)), h2x);
    const float dy = fsub(fadd(h0y, fmul(ddy, z2_tz)), y4[k]);
    if (fabsf(dx) < kTolerance && fabsf(dy) < kTolerance && in_h2_window(x4, k, h2x, lo, hi)) {
      const float scatter = fmul(fmul(fadd(fmul(dx, dx), fmul(dy, dy)), den), den);
      if (scatter < kMaxScatter) {
        if (scatter < best) {
          best = scatter;
          fit.k = k;
        }
      } else if (!isfinite(scatter)) {
        fit.degenerate = true;
      }
    }
  }
  *scatter_out = best;
  return fit;
}

// The usable h1s of module s1, for the seeding of its parity (one warp).  Half
// of a module's hits are used or without an h2 window by then: pairs with them
// are not formed (3,930 instead of 6,950 pairs an event of 1,160 hits, 54,000
// instead of 103,000 of 4,400: 15 % of the time of 10,000 uneven events, 8 % of
// 4,000 dense ones).  Larger modules are paired hit by hit.
template <class Shared>
__device__ __forceinline__ void list_h1s(const EventView& ev, Shared& s, const Worker& w, int s1) {
  const int lane = threadIdx.x & 31, st1 = s.start[s1], n1 = s.num(s1);
  if (n1 > Shared::kList) return;
  int before = 0;
  for (int i0 = 0; i0 <= n1; i0 += 32) {   // n1 itself has a place too: the end of a window
    const int i = i0 + lane;
    const bool usable = i < n1 && ev.useds()[st1 + i] == 0;
    const unsigned m = __ballot_sync(kFull, usable);
    if (lane == 0) s.seed.usable[w.parity()][i0 >> 5] = make_uint2(m, (unsigned)before);
    if (usable) s.seed.list[w.parity()][before + __popc(m & lanemask_lt())] = (uint8_t)i;
    before += __popc(m);
  }
}

// Learned seeding scores every doublet that passes the cuts, and one in 15 of
// them has a hit of f-4 in reach: the others yield no tracklet whatever their
// score, which only counts for the guard (too few kept: the event is searched
// by the plain method).  So a first search scores the doublets in reach only
// (`sparse`) and counts the others; where the kept ones of those are enough,
// they are enough of all.  Else the event is searched again with every doublet
// scored (process_event).  That needs the doublets to be known when their cell
// is looked up: modules whose dead h1s are their last hits, and no
// learned_min_window.  It saves a fifth of the time of 5,000 events of 1,160
// hits.
template <int kMode, bool kPlainGeometry, class Shared>
__device__ __forceinline__ void seed_pairs(const EventView& ev, Shared& s, Worker& w, int f) {
  constexpr int kOwn = Shared::kOwn;
  auto& sd = s.seed;
  const int lane = threadIdx.x & 31;
  const int s1 = f - 2, m4 = f - 4;
  const int st0 = s.start[f], n0 = s.num(f), st1 = s.start[s1], st4 = s.start[m4], n4 = s.num(m4);
  const float zmin1 = s.zmin[s1], zmin4 = s.zmin[m4];
  const uint32_t* map = sd.map[w.parity()];
  const bool listed = s.num(s1) <= Shared::kList;   // list_h1s has run
  const uint8_t* list = sd.list[w.parity()];
  float4* own_h0 = sd.h0[w.warp()];
  float2* own_reach = sd.reach[w.warp()];
  unsigned long long* own_best = sd.best[w.warp()];
  uint16_t* own_first = sd.first[w.warp()];
  // plain geometry: one factor 1 / (z2 - z1), and the reach in x
  const float d41 = fsub(zmin4, zmin1);
  const float den = fdiv(1.f, d41), tol = fadd(fminf(kTolerance, fmul(kScatterReach, fabsf(d41))), kRounding);
  const float* x4 = ev.xs() + st4;
  const float* y4 = ev.ys() + st4;
  const uint32_t Y = (uint32_t)ev.y_lanes;
  if (n0 == 0 || n4 == 0 || s.num(s1) == 0) return;
  const float s1_z = ev.zs()[st1];   // Kernel.cl:420
  const bool sparse = kMode == kLearned && ev.sparse && (s.flags[s1] & kDeadTail);

  for (int block = 0; block < n0; block += 32)   // warp-uniform
  for (int c0 = 0, mine = active_h0s(ev, w, st0, n0, block, sd.active[w.parity()]); c0 < mine; c0 += kOwn) {
    int h0 = 0, first = 0, count = 0, from = 0;
    float h0x = 0.f, h0y = 0.f, h0z = 0.f;
    if (lane < kOwn && c0 + lane < mine) {
      h0 = st0 + block + sd.active[w.parity()][w.idx() + (c0 + lane) * w.of()];
      h0x = ev.xs()[h0];
      h0y = ev.ys()[h0];
      h0z = ev.zs()[h0];
      int last;
      h1_window(ev, s, s1, h0x, h0z, &first, &last);
      count = max(last - first, 0);
      from = first;
      if (listed && count > 0) {   // the window's usable h1s
        const uint2 u = sd.usable[w.parity()][first >> 5], v = sd.usable[w.parity()][last >> 5];
        from = (int)(u.y + __popc(u.x & ((1u << (first & 31)) - 1u)));
        count = (int)(v.y + __popc(v.x & ((1u << (last & 31)) - 1u))) - from;
      }
    }
    // the pairs of the warp's h0s, end to end
    int end = count;
#pragma unroll
    for (int o = 1; o < kOwn; o <<= 1) {
      const int v = __shfl_up_sync(kFull, end, o);
      if (lane >= o) end += v;
    }
    const int total = __shfl_sync(kFull, end, kOwn - 1);
    if (total == 0) continue;
    const int begin = end - count;
    const unsigned om = __ballot_sync(kFull, count > 0);
    const int slot = __popc(om & lanemask_lt());
    __syncwarp();   // the previous round's lists have been read
    if (count > 0) {
      own_h0[slot] = make_float4(h0x, h0y, h0z, __int_as_float(from - begin));
      own_reach[slot] = make_float2(fmul(kMaxYSlope, fabsf(fsub(s1_z, h0z))),
                                   fmul(fsub(zmin4, h0z), fdiv(1.f, fsub(zmin1, h0z))));
      own_best[slot] = ~0ull;
      own_first[slot] = (uint16_t)first;
    }
    __syncwarp();

    int owners = 0, queued = 0;
    for (int base = 0;; base += 32) {
      const bool more = base < total;   // warp-uniform
      bool pass = false, scored = false;
      int h1 = 0, o = 0;
      if (more) {
        // the h0 of each lane's pair: count the h0s that begin up to it
        const uint32_t starts =
            __reduce_or_sync(kFull, count > 0 && begin >= base && begin < base + 32 ? 1u << (begin - base) : 0u);
        o = owners + __popc(starts & (2u * (1u << lane) - 1u)) - 1;
        owners += __popc(starts);
        if (base + lane < total) {
          const float4 q = own_h0[o];
          const float2 r = own_reach[o];
          const int at = __float_as_int(q.w) + base + lane;
          h1 = st1 + (listed ? (int)list[at] : at);
          const bool usable = listed || ev.useds()[h1] == 0;
          const float h1x = ev.xs()[h1], h1y = ev.ys()[h1];
          pass = usable && fabsf(fsub(h1y, q.y)) < r.x;
          scored = pass;
          if (kPlainGeometry && (kMode == kPlain || sparse) && pass) {   // the fit's own predicted point
            const float px = fadd(q.x, fmul(fsub(h1x, q.x), r.y));
            const float py = fadd(q.y, fmul(fsub(h1y, q.y), r.y));
            pass = map_marked<Shared>(map, px, py);
          }
        }
        if (kMode == kLearned && sparse) {
          const unsigned mc = __ballot_sync(kFull, scored);
          if (lane == 0 && mc) atomicAdd(&s.considered, (uint32_t)__popc(mc));
        }
      }
      const unsigned pm = __ballot_sync(kFull, pass);
      if (queued + __popc(pm) > kQueue || !more) {   // warp-uniform
        __syncwarp();
        const uint32_t entry = sd.queue[w.warp()][lane];
        const int own = (int)(entry >> 14);
        const int local1 = (int)(entry & 0x3fffu), hit1 = st1 + local1;
        // a Y-lane stops at its first dead h1: where the dead h1s are not the
        // module's last ones, look for one before this pair's
        bool reached = lane < queued;
        if (!(s.flags[s1] & kDeadTail) && reached)
          for (int e = local1 - (int)Y; e >= (int)own_first[own]; e -= (int)Y) reached &= !h1_dead(ev, s, s1, st1 + e);
        // learned: the batch is scored together, and a kept doublet's h2 lies
        // within its own tolerance, in the h1's exact window
        float learned_tol = kTolerance;
        int a = 0, b = n4;
        if constexpr (kMode == kLearned) {
          float4 q = make_float4(0.f, 0.f, 0.f, 0.f);
          float h1x = 0.f, h1y = 0.f;
          if (reached) {
            q = own_h0[own];
            h1x = ev.xs()[hit1];
            h1y = ev.ys()[hit1];
            // the h1's window, found for the scored pairs only: filling in all
            // windows per event takes 5 % more time
            float lo, hi;
            h2_bounds(h1x, zmin1, s.sz[f], s.sz[m4], &lo, &hi);
            a = first_gt(x4, 0, n4, lo);
            b = first_gt(x4, min(a + 1, n4), n4, hi);
          }
          // only doublets with a wide exact h2 window are worth scoring
          const bool score = reached && b - a >= ev.p->learned_min_window;
          bool keep = true;
          if (__any_sync(kFull, score)) {
            const float2 r = score_batch(ev.mlp, score, q.x, q.y, q.z, h1x, h1y, zmin1,
                                            fdiv(1.f, fsub(zmin1, q.z)), 0.5f * (zmin4 + zmin4), b - a, f, ev.S,
                                            reached ? own_reach[own].x : 0.f);
            if (score) {
              keep = r.x >= ev.p->keep_threshold;
              learned_tol = fminf(kTolerance, fmaxf(r.y, 0.f) + ev.p->window_margin);
            }
          }
          // keep-rate bookkeeping for the guard: the scored doublets
          const unsigned mc = __ballot_sync(kFull, score), mk = __ballot_sync(kFull, score && keep);
          if (lane == 0 && mc) {
            if (!sparse) atomicAdd(&s.considered, (uint32_t)__popc(mc));
            atomicAdd(&s.kept, (uint32_t)__popc(mk));
          }
          reached = reached && keep;
        }
        if (reached) {
          const float4 q = own_h0[own];
          float best = FLT_MAX;
          int best_k = -1;
          if constexpr (kPlainGeometry) {
            // Kernel.cl:468-529 for one (h0, h1): the fits of the h2s in reach
            const float z2_tz = own_reach[own].y;
            const float h1x = ev.xs()[hit1], h1y = ev.ys()[hit1];
            const float px = fadd(q.x, fmul(fsub(h1x, q.x), z2_tz)), py = fadd(q.y, fmul(fsub(h1y, q.y), z2_tz));
            float lt = fsub(px, tol), ht = fadd(px, tol);
            if constexpr (kMode == kLearned) {
              const float margin = fadd(0.01f, fmul(1e-5f, fadd(fabsf(px), fabsf(px))));
              const float l = fsub(fsub(px, learned_tol), margin), h = fadd(fadd(px, learned_tol), margin);
              if (isfinite(l) && isfinite(h)) {   // else the whole window is tried
                lt = fmaxf(lt, l);
                ht = fminf(ht, h);
              }
              if (!map_marked<Shared>(map, px, py)) b = a;   // no hit in reach
            }
            for (int k = first_gt(x4, a, b, lt); k < b; ++k) {
              const float h2x = x4[k];
              if (h2x > ht) break;
              const float dx = fsub(px, h2x), dy = fsub(py, y4[k]);
              const float scatter = fmul(fmul(fadd(fmul(dx, dx), fmul(dy, dy)), den), den);
              if (fabsf(dx) < kTolerance && fabsf(dy) < kTolerance && scatter < kMaxScatter && scatter < best) {
                bool in = kMode == kLearned;   // [a, b) is the window
                if constexpr (kMode == kPlain) {
                  float lo, hi;
                  h2_bounds(h1x, zmin1, s.sz[f], s.sz[m4], &lo, &hi);
                  in = in_h2_window(x4, k, h2x, lo, hi);
                }
                if (in) {
                  best = scatter;
                  best_k = k;
                }
              }
            }
          } else {
            const Fit fit = pair_fit_any(ev, s, f, q.x, q.y, q.z, hit1, &best);
            best_k = fit.k;
            if (fit.degenerate) atomicOr(&s.status, VELO_EVENT_DEGENERATE);
          }
          if (best_k >= 0) {   // smallest fit, then Y-lane, h1, h2
            const uint32_t e = (uint32_t)local1 - own_first[own];
            atomicMin(&own_best[own], ((unsigned long long)__float_as_uint(best) << 32) |
                                         ((unsigned long long)(e % Y) << 28) | ((unsigned long long)e << 14) |
                                         (unsigned long long)best_k);
          }
        }
        queued = 0;
        __syncwarp();
      }
      if (!more) break;
      if (pass) sd.queue[w.warp()][queued + __popc(pm & lanemask_lt())] = ((uint32_t)o << 14) | (uint32_t)(h1 - st1);
      queued += __popc(pm);
    }
    const unsigned long long best = count > 0 ? own_best[slot] : ~0ull;
    append_tracklets(ev, w, best != ~0ull, (uint32_t)h0, (uint32_t)(st1 + first) + ((uint32_t)(best >> 14) & 0x3fffu),
                     (uint32_t)st4 + (uint32_t)(best & 0x3fffu), f);
  }
}

// The flags of module m's hits before the search (one warp): unused, and
// kDead where the hit as an h1 has no h2 window; whether the dead hits are
// the module's last ones.
template <class Shared>
__device__ __forceinline__ bool clear_flags(const EventView& ev, const Shared& s, int m) {
  const int lane = threadIdx.x & 31;
  const int st = s.start[m], n = s.num(m);
  bool tail = true;
  unsigned before = 0;   // dead hits so far
  for (int i0 = 0; i0 < n; i0 += 32) {
    const int i = i0 + lane;
    const bool in = i < n;
    const bool dead = in && h1_dead(ev, s, m, st + i);
    if (in) ev.useds()[st + i] = dead ? kDead : 0;
    const unsigned dm = __ballot_sync(kFull, dead), im = __ballot_sync(kFull, in);
    const unsigned live = im & ~dm, from_dead = 0u - (dm & (0u - dm));   // lanes from the first dead hit on
    if ((before && live) || (live & from_dead)) tail = false;
    before |= dm;
  }
  return tail;
}

// Words a thread loads before it stores any, while an event is staged.
constexpr int kStageWords = 6;
// Words of tracks a lane loads before it stores any, while they are written out.
constexpr int kCopyWords = 4;

// Hits of a module that one warp sorts by rank in registers (4 per lane).
constexpr int kArenaRankMax = 128;

// The reference's per-module x-sort (preorder_by_x, Tools.cpp:46-66) of the
// event staged in the arena, hit IDs alongside in `ids`; one warp per
// module.  Where a module's x values are distinct the reference's quicksort
// reaches the one ascending order there is, so each hit goes to its rank;
// a module with equal x values, or more than kArenaRankMax hits not already
// in strictly increasing order, replays the reference's partition steps in
// one thread (quicksort4).  x is finite here (the staging checked it).
// Returns, in every thread, whether any hit moved.
template <class Shared>
__device__ bool sort_arena(const EventView& ev, const Shared& s, int S, uint32_t* ids) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  float* x = ev.xs();
  float* y = ev.ys();
  float* z = ev.zs();
  bool moved = false;
  for (int m = warp; m < S; m += nwarps) {   // warp-uniform
    const int s0 = s.start[m], n = s.num(m);
    if (n < 2) continue;
    if (n > kArenaRankMax) {
      bool changed = false;
      if (lane == 0) {
        bool increasing = true;
        for (int i = s0 + 1; i < s0 + n && increasing; ++i) increasing = x[i - 1] < x[i];
        if (!increasing) {
          quicksort4(x, y, z, ids, s0, s0 + n - 1);
          changed = true;
        }
      }
      moved |= __shfl_sync(kFull, changed, 0);
      __syncwarp();
      continue;
    }
    float xr[4];
    int rk[4], eq[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane + 32 * k;
      xr[k] = i < n ? x[s0 + i] : 0.f;
      rk[k] = 0;
      eq[k] = 0;
    }
    for (int j = 0; j < n; ++j) {   // the same address in every lane
      const float xj = x[s0 + j];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        rk[k] += xj < xr[k];
        eq[k] += xj == xr[k];
      }
    }
    bool tie = false, mv = false;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane + 32 * k;
      if (i < n) {
        tie |= eq[k] > 1;
        mv |= rk[k] != i;
      }
    }
    if (__any_sync(kFull, tie)) {   // equal x values: the reference's partition steps decide
      if (lane == 0) quicksort4(x, y, z, ids, s0, s0 + n - 1);
      moved = true;
      __syncwarp();
      continue;
    }
    if (!__any_sync(kFull, mv)) continue;   // strictly increasing already
    moved = true;
    float yr[4], zr[4];
    uint32_t ir[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane + 32 * k;
      if (i < n) {
        yr[k] = y[s0 + i];
        zr[k] = z[s0 + i];
        ir[k] = ids[s0 + i];
      }
    }
    __syncwarp();   // every lane has read its hits before any is overwritten
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      const int i = lane + 32 * k;
      if (i < n) {
        const int r = s0 + rk[k];
        x[r] = xr[k];
        y[r] = yr[k];
        z[r] = zr[k];
        ids[r] = ir[k];
      }
    }
    __syncwarp();
  }
  return __syncthreads_or(moved) != 0;
}

// Streaming results (velo_search_begin): thread 0 writes the event's record,
// its ready flag last, after a system-scope fence; the caller has fenced the
// CTA's track writes before.
__device__ __forceinline__ void publish_result(const SearchParams& p, int e, unsigned long long first,
                                               uint32_t count, uint32_t status) {
  velo_event_result* r = p.results + e;
  r->first = first;
  r->count = count;
  r->status = status;
  __threadfence_system();
  *reinterpret_cast<volatile uint32_t*>(&r->ready) = 1u;
}

// Per-phase cycle counters, compiled in only with -DVELO_PHASE_CLOCKS
// (diagnostic builds): thread 0 of every CTA adds the clock64() time between
// the barriers that close each phase; slot 7 counts events.
#ifdef VELO_PHASE_CLOCKS
static __device__ unsigned long long g_phase_cycles[8];   // one per translation unit
#define VELO_PHASE_BEGIN() long long ph_t = clock64(); unsigned long long ph[7] = {0, 0, 0, 0, 0, 0, 0}
#define VELO_PHASE(k)                 \
  do {                                \
    const long long t_ = clock64();   \
    ph[k] += (unsigned long long)(t_ - ph_t); \
    ph_t = t_;                        \
  } while (0)
#define VELO_PHASE_END()                                              \
  do {                                                                \
    if (threadIdx.x == 0) {                                           \
      for (int k_ = 0; k_ < 7; ++k_) atomicAdd(&g_phase_cycles[k_], ph[k_]); \
      atomicAdd(&g_phase_cycles[7], 1ull);                            \
    }                                                                 \
  } while (0)
#else
#define VELO_PHASE_BEGIN() do {} while (0)
#define VELO_PHASE(k) do {} while (0)
#define VELO_PHASE_END() do {} while (0)
#endif

// The module loop, Kernel.cl:671-767 (see Worker for the order of the warps).
// kMode: the seeding; kPlainGeometry: the event is of plain geometry; kPairs:
// it takes the pair seeding.
template <int kMode, int kLanes, bool kPlainGeometry, bool kPairs, class Shared>
__device__ __forceinline__ Worker module_loop(const EventView& ev, Shared& s, Worker w) {
  const int lane = threadIdx.x & 31, S = ev.S;
  for (int f = S - 1; f >= 4; --f) {
    forward<kPlainGeometry>(ev, s, w, f);
    const int step = (S - 1 - f) & 1;
    if (w.alone() || step == w.parity()) {
      const int gt = w.idx() * 32 + lane, gn = w.of() * 32;
      if (kPlainGeometry) {
        uint4* map = reinterpret_cast<uint4*>(s.seed.map[w.parity()]);
        for (int i = gt; i < Shared::kMapRows / 4; i += gn) map[i] = make_uint4(0, 0, 0, 0);
      }
      group_sync<Shared::kMaxWarps>(w);
      if constexpr (kPairs) {
        if (w.idx() == 0) list_h1s(ev, s, w, f - 2);
        if (kPlainGeometry)   // from the group's last warp on
          for (int i = gn - 1 - gt; i < s.num(f - 4); i += gn)
            mark_map(ev, s, s.seed.map[w.parity()], f - 2, f - 4, i);
        group_sync<Shared::kMaxWarps>(w);
        seed_pairs<kPlainGeometry ? kMode : kPlain, kPlainGeometry>(ev, s, w, f);
      } else {
        seed_module<kMode, kLanes>(ev, s, w, f, seed_lanes_of(kLanes, (uint32_t)ev.y_lanes));
      }
      group_sync<Shared::kMaxWarps>(w);
    }
    if (step == 1 || f == 4) __syncthreads();
  }
  return w;
}

// The loops of the events that the kernel's own is not made for: each of its own
// registers, and behind one call of the kernel, so that what they need is none
// of the kernel's concern (called from it directly, they moved its spills: 1.67
// -> 1.73 ms for 10,000 events that never call them).  With the two seedings in
// one loop, events of several z per module ran 5 to 10 % slower.  (The dump's
// kernel has the walked loop only, in place: 3,000 events 1.83 ms, 2.21 through
// these calls.)
template <int kMode, int kLanes, bool kPlainGeometry, bool kPairs, class Shared>
__device__ __noinline__ Worker module_loop_any(const EventView& ev, Shared& s, Worker w) {
  return module_loop<kMode, kLanes, kPlainGeometry, kPairs>(ev, s, w);
}

template <int kLanes, class Shared>
__device__ __noinline__ Worker module_loop_other(const EventView ev, Shared& s, Worker w) {
  if (!ev.tame) return module_loop_any<kPlain, kLanes, false, false>(ev, s, w);
  if (!ev.plain) return module_loop_any<kPlain, kLanes, false, true>(ev, s, w);
  // never taken; without the call the ordinary loop's registers are dealt out
  // otherwise (10,000 events 1.67 -> 1.69 ms)
  return module_loop_any<kPlain, kLanes, true, true>(ev, s, w);
}

// The same for the learned build, of plain geometry neither.
template <int kLanes, class Shared>
__device__ __noinline__ Worker module_loop_learned(const EventView ev, Shared& s, Worker w, bool learned) {
  if (learned) return module_loop_any<kLearned, kLanes, false, false>(ev, s, w);
  return ev.tame ? module_loop_any<kPlain, kLanes, false, true>(ev, s, w)
                 : module_loop_any<kPlain, kLanes, false, false>(ev, s, w);
}

// The plain search of an event that the learned one gave up, called directly
// (5,000 events that all fall back 1.10 ms, 1.15 behind the other call).
template <int kLanes, class Shared>
__device__ __noinline__ Worker module_loop_fallback(const EventView ev, Shared& s, Worker w) {
  return module_loop<kPlain, kLanes, true, true>(ev, s, w);
}

// ---------------------------------------------------------------------------
template <int kMode, int kLanes, class Shared>
__device__ void process_event(const SearchParams& p, int e, Shared& s, uint8_t* dyn, const MlpFrag* mlp_smem) {
  const int tid = threadIdx.x, nt = blockDim.x;
  const int lane = tid & 31, warp = tid >> 5, nwarps = nt >> 5;
  VELO_PHASE_BEGIN();
  if (!p.ev_valid[e]) {
    if (tid == 0) {
      p.out_counts[e] = 0;
      p.out_first[e] = 0;
      p.out_status[e] = VELO_EVENT_INVALID;
      if (p.results) publish_result(p, e, 0ull, 0u, VELO_EVENT_INVALID);
    }
    return;
  }
  const int32_t* hdr = reinterpret_cast<const int32_t*>(p.input + p.ev_offset[e]);
  EventView ev;
  ev.p = &p;
  ev.S = hdr[0];
  ev.H = hdr[1];
  const int S = ev.S, H = ev.H;
  const int32_t* gZ = hdr + 2;
  const int32_t* gstart = gZ + S;
  const int32_t* gnum = gstart + S;
  const float* gx = reinterpret_cast<const float*>(gnum + S + H);
  const float* gy = gx + H;
  const float* gz = gy + H;

  const ArenaLayout L = arena_layout((uint32_t)H, p.ev_maxmod[e], (uint32_t)p.y_lanes);
  ev.arena = p.arena_off[e] == kNoArena ? dyn : p.global_arena + p.arena_off[e];
  ev.P = L.y;
  ev.event = e;
  ev.mlp = mlp_smem;
  ev.tracklets = reinterpret_cast<uint4*>(p.tracklets);
  ev.tracks = p.tracks;
  ev.weak = p.weak;
  ev.entry_words = reinterpret_cast<uint4*>(p.entry_words);
  ev.entry_lines = reinterpret_cast<float4*>(p.entry_lines);
  ev.y_lanes = p.y_lanes;
  ev.narrow = p.narrow;

  // stage the event; the module table must tile [0, H) in order (the host
  // checked only the header and the blob's length)
  bool bad = tid == 0 && S == 0 && H != 0;
  bool wild = !ev.narrow;   // the event does not take the pair seeding
  for (int m = tid; m < S; m += nt) {
    const int32_t st = gstart[m], nm = gnum[m];
    const int64_t expect = m == 0 ? 0 : (int64_t)gstart[m - 1] + (int64_t)gnum[m - 1];
    bad |= nm < 0 || nm > VELO_MAX_MODULE_HITS || (int64_t)st != expect ||
           (m == S - 1 && (int64_t)st + (int64_t)nm != (int64_t)H);
    s.start[m] = st;
    s.sz[m] = gZ[m];
  }
  for (int m = tid; m <= S; m += nt) s.inflight[m] = 0;
  // with sort_events the IDs are staged too, in the window area (written
  // only after the sort)
  const uint32_t* gid = reinterpret_cast<const uint32_t*>(gnum + S);
  uint32_t* ids = reinterpret_cast<uint32_t*>(ev.wins());
  // x, y and z lie one after another: copied as one array, a warp to whole
  // 128-byte lines of it and several lines in flight (events read in place
  // come over the host link, where a request for part of a line costs a line)
  const int values = 3 * H;
  for (int i0 = tid - (int)((reinterpret_cast<uintptr_t>(gx) >> 2) & 31u); i0 < values; i0 += kStageWords * nt) {
    float v[kStageWords];
#pragma unroll
    for (int k = 0; k < kStageWords; ++k) {
      const int i = i0 + k * nt;
      v[k] = i >= 0 && i < values ? gx[i] : 0.f;
    }
#pragma unroll
    for (int k = 0; k < kStageWords; ++k) {
      const int i = i0 + k * nt;
      bad |= !(fabsf(v[k]) <= FLT_MAX);
      wild |= fabsf(v[k]) > kMaxCoordinate;
      if (i >= 0 && i < values) {
        const int a = (i >= H) + (i >= 2 * H);   // which array
        *reinterpret_cast<float*>(ev.arena + (uint32_t)a * ev.P + 4u * (uint32_t)(i - a * H)) = v[k];
      }
    }
  }
  if (p.sort_events)
    for (int i = tid; i < H; i += nt) ids[i] = gid[i];
  if (tid == 0) {
    s.start[S] = H;
    s.status = 0;
    s.considered = 0; s.kept = 0;
  }
  if (__syncthreads_or(bad)) {   // a bad module table, or a non-finite coordinate
    if (tid == 0) {
      p.out_counts[e] = 0;
      p.out_first[e] = 0;
      p.out_status[e] = VELO_EVENT_INVALID;
      if (p.results) publish_result(p, e, 0ull, 0u, VELO_EVENT_INVALID);
    }
    return;
  }
  if (p.sort_events && sort_arena(ev, s, S, ids)) {
    // the sorted hit arrays (IDs, x, y, z) back into the input, the
    // caller's buffer read in place: posted writes across the host link,
    // overlapped with the search of the other resident events
    uint32_t* wid = const_cast<uint32_t*>(gid);
    float* wx = reinterpret_cast<float*>(wid + H);
    float* wy = wx + H;
    float* wz = wy + H;
    for (int i = tid; i < H; i += nt) {
      wid[i] = ids[i];
      wx[i] = ev.xs()[i];
      wy[i] = ev.ys()[i];
      wz[i] = ev.zs()[i];
    }
    __syncthreads();   // the window area is written next
  }
  VELO_PHASE(0);

  // per-module z range, x-sortedness and hit flags (one warp per module)
  // The first hits of a warp's next module are loaded while it goes over one.
  float x_next = 0.f, z_next = 0.f;
  auto load_module = [&](int m) {
    if (m < S && lane < s.num(m)) {
      x_next = ev.xs()[s.start[m] + lane];
      z_next = ev.zs()[s.start[m] + lane];
    }
  };
  load_module(warp);
  for (int m = warp; m < S; m += nwarps) {
    const int st = s.start[m], n = s.num(m);
    float x = x_next, z = z_next;
    load_module(m + nwarps);
    float zmn = FLT_MAX, zmx = -FLT_MAX, x_before = -FLT_MAX;
    bool sorted = true;
    for (int i0 = 0; i0 < n; i0 += 32) {   // warp-uniform
      const int i = i0 + lane;
      if (i0 > 0 && i < n) {
        x = ev.xs()[st + i];
        z = ev.zs()[st + i];
      }
      const float left = __shfl_up_sync(kFull, x, 1);
      if (i < n) {
        sorted &= (lane > 0 ? left : x_before) <= x;
        zmn = fminf(zmn, z);
        zmx = fmaxf(zmx, z);
      }
      x_before = __shfl_sync(kFull, x, 31);
    }
    const float z0 = __shfl_sync(kFull, zmn, 0);   // lane 0 has a hit if any has
    if (__all_sync(kFull, zmn > zmx || (zmn == z0 && zmx == z0))) {
      zmn = z0;
      zmx = n > 0 ? z0 : -FLT_MAX;
    } else {
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) {
        zmn = fminf(zmn, __shfl_xor_sync(kFull, zmn, o));
        zmx = fmaxf(zmx, __shfl_xor_sync(kFull, zmx, o));
      }
    }
    sorted = __all_sync(kFull, sorted);
    wild |= !sorted;
    const bool tail = clear_flags(ev, s, m);
    if (lane == 0) {
      s.zmin[m] = zmn;
      s.zmax[m] = zmx;
      s.flags[m] = (sorted ? kSorted : 0) | (tail ? kDeadTail : 0);
    }
  }
  ev.tame = !__syncthreads_or(wild);
  // the modules' z ascend, empty modules apart
  bool odd = false;
  for (int m = tid; m < S; m += nt)
    if (s.num(m) > 0) {
      int q = m - 1;
      while (q >= 0 && s.num(q) == 0) --q;
      odd |= s.zmin[m] != s.zmax[m] || (q >= 0 && !(fsub(s.zmin[m], s.zmax[q]) > kMinGap));
    }
  ev.plain = !__syncthreads_or(odd) && ev.tame;
  VELO_PHASE(1);

  bool learned = kMode == kLearned && (p.learned_max_hits == 0 || (uint32_t)H <= p.learned_max_hits);
  // candidate windows for the seedings that read them (with several z per
  // module the learned one walks them)
  if (kMode == kDump || !ev.tame || (kMode == kLearned && !ev.plain)) {
    fill_windows(ev, s);
    __syncthreads();
  }
  VELO_PHASE(2);

  // The learned seeding runs first when enabled, scoring the doublets in reach
  // (plain geometry; seed_pairs); if those it kept are too small a fraction of
  // the doublets, the event is searched again with all of them scored, and if
  // the fraction is still too small, by the plain method (flags and lists
  // reset; windows kept).
  uint32_t fallback = (kMode == kLearned && !learned) ? VELO_EVENT_LEARNED_FALLBACK : 0u;
  Worker w{};
  w.row = (uint32_t)p.hit_base[e] + first_row(s, w, S);
  ev.sparse = learned && ev.plain && p.learned_min_window <= 0;
  for (bool again = false;; again = true) {
    if (again) {
      for (int m = warp; m < S; m += nwarps) clear_flags(ev, s, m);
      for (int m = tid; m <= S; m += nt) s.inflight[m] = 0;
      if (tid == 0) { s.status = 0; s.considered = 0; s.kept = 0; }
      w.n = w.tracklets = w.tracks = w.weak = 0;
      __syncthreads();
    }
    if constexpr (kMode == kDump)
      w = module_loop<kDump, kLanes, false, false>(ev, s, w);
    else if (kMode == kLearned && ev.plain && !learned)
      w = module_loop_fallback<kLanes>(ev, s, w);
    else if (kMode == kLearned && !ev.plain)
      w = module_loop_learned<kLanes>(ev, s, w, learned);
    else if (!ev.plain)
      w = module_loop_other<kLanes>(ev, s, w);
    else
      w = module_loop<kMode, kLanes, true, true>(ev, s, w);
    VELO_PHASE(4);

    // leftover tracklets become weak (Kernel.cl:771-792)
    if (ev.H > VELO_TTF_MODULO / 2 && lane == 0) atomicAdd(&s.inflight[3], min(w.n, kInflightMax));
    for (uint32_t i0 = 0; i0 < w.n; i0 += 32) {   // warp-uniform
      const uint32_t v = i0 + lane < w.n ? ev.entry_words[w.row + i0 + lane].x : 0u;
      const unsigned m = __ballot_sync(kFull, (v & kTrackletFlag) != 0);
      if (v & kTrackletFlag) ev.weak[w.row + w.weak + (uint32_t)__popc(m & lanemask_lt())] = v & kEntryNumber;
      w.weak += __popc(m);
    }
    __syncwarp();
    // weak tracks made of three unused hits (Kernel.cl:796-815)
    for (uint32_t i0 = 0; i0 < w.weak; i0 += 32) {
      uint4 t = make_uint4(0, 0, 0, 0);
      bool take = false;
      if (i0 + lane < w.weak) {
        t = ev.tracklets[w.row + ev.weak[w.row + i0 + lane]];
        take = ((ev.useds()[t.x] | ev.useds()[t.y] | ev.useds()[t.z]) & kUsed) == 0;
      }
      const unsigned m = __ballot_sync(kFull, take);
      if (take) {
        uint32_t* wr =
            reinterpret_cast<uint32_t*>(&ev.tracks[w.row + w.tracks + (uint32_t)__popc(m & lanemask_lt())]);
        wr[0] = 3; wr[1] = t.x; wr[2] = t.y; wr[3] = t.z;
      }
      w.tracks += __popc(m);
    }
    if (lane == 0) s.tracks[warp] = w.tracks;
    __syncthreads();
    VELO_PHASE(5);
    if (!learned) break;
    const uint32_t considered = s.considered, kept = s.kept;   // final after the barrier above
    if (considered == 0 || (float)kept >= p.min_keep_rate * (float)considered) break;
    if (ev.sparse) {
      ev.sparse = false;
    } else {
      learned = false;
      fallback = VELO_EVENT_LEARNED_FALLBACK;
    }
    __syncthreads();   // everyone has read the counters before the reset
  }

  // compacted output: one atomic per event reserves its range, the warps'
  // tracks one after another
  uint32_t count = 0, before = 0;
  for (int k = 0; k < nwarps; ++k) {
    const uint32_t c = s.tracks[k];
    if (k < warp) before += c;
    count += c;
  }
  if (H > VELO_TTF_MODULO / 2)   // Kernel.cl:344,354,565
    for (int f = 3 + tid; f < S; f += nt)
      if ((s.inflight[f] & 0xffffu) > VELO_TTF_MODULO || (s.inflight[f] >> 16) > VELO_TTF_MODULO)
        atomicOr(&s.status, VELO_EVENT_RING_OVERFLOW);
  if (tid == 0) {
    if (count > VELO_MAX_TRACKS) atomicOr(&s.status, VELO_EVENT_MAX_TRACKS);
    s.out_first = atomicAdd(p.out_cursor, (unsigned long long)count);
  }
  __syncthreads();
  if (tid == 0) {
    p.out_counts[e] = count;
    p.out_first[e] = s.out_first;
    p.out_status[e] = s.status | fallback;
  }
  {
    // rows past out_capacity stay unwritten (the host reports the shortfall)
    const unsigned long long first = s.out_first + before;
    const unsigned long long room = first < p.out_capacity ? p.out_capacity - first : 0ull;
    const uint32_t words = (uint32_t)min((unsigned long long)w.tracks, room) * 25u;
    const uint32_t* src = reinterpret_cast<const uint32_t*>(ev.tracks + w.row);
    uint32_t* dst = reinterpret_cast<uint32_t*>(p.out_tracks + first);
    // whole 128-byte lines per warp, as in the staging
    const int count_words = (int)words;
    const int skew = count_words > 0 ? (int)((reinterpret_cast<uintptr_t>(dst) >> 2) & 31u) : 0;   // none: no pass
    for (int i0 = lane - skew; i0 < count_words; i0 += 32 * kCopyWords) {
      uint32_t v[kCopyWords], hits[kCopyWords];
#pragma unroll
      for (int k = 0; k < kCopyWords; ++k) {
        const uint32_t i = (uint32_t)min(max(i0 + 32 * k, 0), count_words - 1);
        v[k] = src[i];
        hits[k] = src[i / 25u * 25u];
      }
#pragma unroll
      for (int k = 0; k < kCopyWords; ++k) {   // words past a track's last hit are zero
        const int i = i0 + 32 * k;
        if (i >= 0 && i < count_words) dst[i] = (uint32_t)i % 25u <= hits[k] ? v[k] : 0u;
      }
    }
  }
  if (p.results) {   // streaming: the tracks first, then the record
    __threadfence_system();
    __syncthreads();
    if (tid == 0) publish_result(p, e, s.out_first, count, s.status | fallback);
  }
  VELO_PHASE(6);
  VELO_PHASE_END();
}

// Builds: up to 256 threads per CTA with registers budgeted for 4 or for 5
// resident 256-thread CTAs per SM (velo_options.register_ctas 4 / 5: 64 / 48
// registers; of up to 64 threads in a build with the seeding state of two
// warps), 64-thread CTAs with 56 registers (18 CTAs per SM, register_ctas 18),
// and 512-thread CTAs; the learned mode in a build of up to 256 threads with
// 80 registers (3 resident CTAs) and one of up to 64 threads whose bound of 11
// CTAs leaves the same 80 registers, and 12 CTAs fit (5,000 events 1.43 ms, 1.44
// with a bound of 12; a bound of 16 takes an eighth more, the scorer out of line
// a fifth); each for one seeding width kLanes (lanes per h0 where the windows are
// walked).
template <int kMaxThreads, int kMinCtas, int kMode, int kMods, int kLanes>
__global__ void __launch_bounds__(kMaxThreads, kMinCtas) search_kernel(const __grid_constant__ SearchParams p) {
  extern __shared__ __align__(16) uint8_t dyn_smem_raw[];
  __shared__ SharedT<kMods, kMaxThreads / 32> s;
  // learned seeding: the MLP weights lead the dynamic shared memory
  const MlpFrag* mlp_smem = nullptr;
  uint8_t* dyn_smem = dyn_smem_raw;
  if constexpr (kMode == kLearned) {
    MlpFrag* w = reinterpret_cast<MlpFrag*>(dyn_smem_raw);
    stage_mlp_fragments(p.mlp, w);
    __syncthreads();
    mlp_smem = w;
    dyn_smem = dyn_smem_raw + kMlpSmemBytes;
  }
  if (!p.persistent) {
    if ((int)blockIdx.x < p.n_events) process_event<kMode, kLanes>(p, blockIdx.x, s, dyn_smem, mlp_smem);
    return;
  }
  for (;;) {
    __syncthreads();
    if (threadIdx.x == 0) s.next_event = atomicAdd(p.work_counter, 1);
    __syncthreads();
    const int k = s.next_event;
    if (k >= p.n_events) break;
    process_event<kMode, kLanes>(p, p.order[k], s, dyn_smem, mlp_smem);
  }
}

constexpr int kFullModules = kMaxModules + 1;

// The builds of one seeding width G: launch, dynamic shared-memory limit and
// occupancy, as launch_search / configure_search_kernel / search_occupancy
// (velo_internal.h) take them.  The dump mode exists for G = 32 only.
template <int G>
struct SearchBuilds {
  static int launch(const SearchParams& p, int grid, int block, uint32_t smem, cudaStream_t st, int reg_ctas,
                    bool compact) {
    if (p.mlp && compact && block <= 64)
      search_kernel<64, 11, kLearned, kCompactModules, G><<<grid, block, smem, st>>>(p);
    else if (p.mlp && compact)
      search_kernel<256, 3, kLearned, kCompactModules, G><<<grid, min(block, 256), smem, st>>>(p);
    else if (p.mlp)
      search_kernel<256, 3, kLearned, kFullModules, G><<<grid, min(block, 256), smem, st>>>(p);
    else if (G == 32 && p.dump_features)
      search_kernel<256, 4, kDump, kFullModules, 32><<<grid, min(block, 256), smem, st>>>(p);
    else if (block > 256)
      search_kernel<512, 1, kPlain, kFullModules, G><<<grid, block, smem, st>>>(p);
    else if (reg_ctas == 18 && compact)
      search_kernel<64, 18, kPlain, kCompactModules, G><<<grid, block, smem, st>>>(p);
    else if (reg_ctas == 18)
      search_kernel<64, 18, kPlain, kFullModules, G><<<grid, block, smem, st>>>(p);
    else if (reg_ctas == 4 && block <= 64 && compact)
      search_kernel<64, 16, kPlain, kCompactModules, G><<<grid, block, smem, st>>>(p);
    else if (reg_ctas == 4 && block <= 64)
      search_kernel<64, 16, kPlain, kFullModules, G><<<grid, block, smem, st>>>(p);
    else if (reg_ctas == 4 && compact)
      search_kernel<256, 4, kPlain, kCompactModules, G><<<grid, block, smem, st>>>(p);
    else if (reg_ctas == 4)
      search_kernel<256, 4, kPlain, kFullModules, G><<<grid, block, smem, st>>>(p);
    else if (compact)
      search_kernel<256, 5, kPlain, kCompactModules, G><<<grid, block, smem, st>>>(p);
    else
      search_kernel<256, 5, kPlain, kFullModules, G><<<grid, block, smem, st>>>(p);
    return (int)cudaGetLastError();
  }

  static int configure(uint32_t smem) {
    cudaError_t e = cudaSuccess;
#define VELO_LIMIT(...)   \
  if (e == cudaSuccess) e = cudaFuncSetAttribute(__VA_ARGS__, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem)
    VELO_LIMIT(search_kernel<256, 4, kPlain, kFullModules, G>);
    VELO_LIMIT(search_kernel<256, 5, kPlain, kFullModules, G>);
    VELO_LIMIT(search_kernel<256, 4, kPlain, kCompactModules, G>);
    VELO_LIMIT(search_kernel<256, 5, kPlain, kCompactModules, G>);
    VELO_LIMIT(search_kernel<64, 18, kPlain, kFullModules, G>);
    VELO_LIMIT(search_kernel<64, 18, kPlain, kCompactModules, G>);
    VELO_LIMIT(search_kernel<64, 16, kPlain, kFullModules, G>);
    VELO_LIMIT(search_kernel<64, 16, kPlain, kCompactModules, G>);
    VELO_LIMIT(search_kernel<512, 1, kPlain, kFullModules, G>);
    VELO_LIMIT(search_kernel<256, 3, kLearned, kFullModules, G>);
    VELO_LIMIT(search_kernel<256, 3, kLearned, kCompactModules, G>);
    VELO_LIMIT(search_kernel<64, 11, kLearned, kCompactModules, G>);
    if (G == 32) VELO_LIMIT(search_kernel<256, 4, kDump, kFullModules, 32>);
#undef VELO_LIMIT
    return (int)e;
  }

  static int occupancy(int block, uint32_t smem, int reg_ctas, int mode, bool compact, int* ctas) {
    if (mode == kModeLearned && compact && block <= 64)
      return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
          ctas, search_kernel<64, 11, kLearned, kCompactModules, G>, block, smem);
    if (mode == kModeLearned)
      return compact ? (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<256, 3, kLearned, kCompactModules, G>, min(block, 256), smem)
                     : (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<256, 3, kLearned, kFullModules, G>, min(block, 256), smem);
    if (mode == kModeDump)
      return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, search_kernel<256, 4, kDump, kFullModules, 32>,
                                                                min(block, 256), smem);
    if (block > 256)
      return (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(ctas, search_kernel<512, 1, kPlain, kFullModules, G>,
                                                                block, smem);
    if (reg_ctas == 18)
      return compact ? (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<64, 18, kPlain, kCompactModules, G>, block, smem)
                     : (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<64, 18, kPlain, kFullModules, G>, block, smem);
    if (reg_ctas == 4 && block <= 64)
      return compact ? (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<64, 16, kPlain, kCompactModules, G>, block, smem)
                     : (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<64, 16, kPlain, kFullModules, G>, block, smem);
    if (reg_ctas == 4)
      return compact ? (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<256, 4, kPlain, kCompactModules, G>, block, smem)
                     : (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                           ctas, search_kernel<256, 4, kPlain, kFullModules, G>, block, smem);
    return compact ? (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                         ctas, search_kernel<256, 5, kPlain, kCompactModules, G>, block, smem)
                   : (int)cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                         ctas, search_kernel<256, 5, kPlain, kFullModules, G>, block, smem);
  }

#ifdef VELO_PHASE_CLOCKS
  // Adds this unit's per-phase cycle counters to out[8] and clears them.
  static int phase_cycles(unsigned long long* out) {
    unsigned long long v[8] = {};
    cudaError_t e = cudaMemcpyFromSymbol(v, g_phase_cycles, sizeof v);
    unsigned long long zero[8] = {};
    if (e == cudaSuccess) e = cudaMemcpyToSymbol(g_phase_cycles, zero, sizeof zero);
    for (int k = 0; k < 8; ++k) out[k] += v[k];
    return (int)e;
  }
#endif
};

}  // namespace velo
