// How the persistent CTAs of the grouped GEMMs share the work.
//
// A unit is (token tile, 128-row weight block); it needs k_blocks K steps.  The plan word of a GEMM says how
// the units are cut along K:
//   * K split S in {1, 2, 4, 8}: every unit is cut into S equal segments, handed out one by one;
//   * stream-K (plan word 0): the units' K steps are laid end to end and every CTA takes one contiguous
//     share of that line, so all CTAs stream the same number of weight bytes whatever the unit count; a unit that
//     straddles CTA boundaries is cut there.
// With a counter (mf_gemm_args.sched) the segments of a K split go to whichever CTA asks next.  SMs do not get equal
// shares of the memory rate: with a fixed round-robin the fastest CTA of a weight-streaming GEMM was done a third
// before the slowest, and the down GEMM's CTAs that took the free SMs had a fixed share as well (8 tokens on 288 e4m3
// experts: the last 40 % of the bytes ran at two thirds of the rate).  Without a counter segments are dealt
// round-robin.  A segment's result does not depend on who computes it.
//
// Only the weight producer warp decides what comes next; it also fetches the tile's words.  It publishes each segment
// in a small ring in shared memory, about one segment ahead, and the other roles read it there: no global loads and no
// index arithmetic in them between two units.
#pragma once

#include "common.cuh"
#include "moeflow_b200.h"

namespace mf {

// One piece of work of a CTA: `nkb` K steps of unit (tt, mb) starting at K block kb0.
struct Seg {
  int unit, tt, mb;          // unit < 0: no more work
  int e, row_start, n_rows;  // the token tile: expert, first entry, entries
  int kb0, nkb;
  int nseg, seg;             // segments of this unit and this one's index in K order (nseg == 1: whole unit)
  int c_first;               // stream-K: CTA that holds segment 0 of the unit; K split: -1
  int late;                  // stream-K: 1 when that CTA's share begins before the unit
};

// Partial-sum slot of segment `sg` of the unit of `s`.  K split: slots are (unit, segment).  Stream-K: every CTA owns two
// slots, one for the segment its share starts with and one for the segment it ends with.
__device__ __forceinline__ int slot_of(const Seg& s, int sg) {
  if (s.c_first < 0) return s.unit * s.nseg + sg;
  return 2 * (s.c_first + sg) + (sg == 0 ? s.late : 0);
}

struct WorkIter {
  const mf_gemm_args* a;
  int n_max, m_blocks, KB, split, stream;
  int units;         // n_tiles * m_blocks
  int cta, G;        // this CTA, CTAs that take part
  long long W;       // stream-K: units * KB
  long long w, w1;   // stream-K: cursor and end of this CTA's share
  int u;             // K split: this CTA's next (unit, split) index

  __device__ __forceinline__ long long share_begin(int c) const { return (long long)c * W / G; }
  // CTA holding K step x of the line (the largest c with share_begin(c) <= x)
  __device__ __forceinline__ int cta_of(long long x) const { return (int)(((x + 1) * G + W - 1) / W) - 1; }

  __device__ __forceinline__ void init(const mf_gemm_args& args, int n_max_, int n_tiles, int split_, int cta_, int grid) {
    a = &args;
    n_max = n_max_;
    m_blocks = args.m_blocks;
    KB = args.k_blocks;
    split = split_ < 1 ? 1 : split_;
    stream = split_ == 0;
    units = n_tiles * m_blocks;
    cta = cta_;
    W = (long long)units * KB;
    G = stream ? (int)(W < (long long)grid ? W : (long long)grid) : grid;
    u = cta;
    w = w1 = 0;
    if (stream && cta < G) {
      w = share_begin(cta);
      w1 = share_begin(cta + 1);
    }
  }

  // The segment at the cursor, its tile words still in flight (nothing here waits for the three loads).
  __device__ __forceinline__ bool locate(Seg& s) {
    if (stream) {
      if (w >= w1) return false;
      s.unit = (int)(w / KB);
      s.kb0 = (int)(w - (long long)s.unit * KB);
      const long long left = w1 - w;
      s.nkb = (KB - s.kb0) < left ? (KB - s.kb0) : (int)left;
      w += s.nkb;
      const long long x0 = (long long)s.unit * KB;
      s.c_first = cta_of(x0);
      s.nseg = cta_of(x0 + KB - 1) - s.c_first + 1;
      s.seg = cta - s.c_first;
      s.late = share_begin(s.c_first) < x0 ? 1 : 0;
    } else {
      if (u >= units * split) return false;
      const int ks = u % split;
      s.unit = u / split;
      s.nkb = KB / split;
      s.kb0 = ks * s.nkb;
      s.nseg = split;
      s.seg = ks;
      s.c_first = -1;
      s.late = 0;
    }
    s.tt = s.unit / m_blocks;
    s.mb = s.unit - s.tt * m_blocks;
    s.e = __ldcg(a->tile_e + s.tt);
    s.row_start = __ldcg(a->tile_s + s.tt);
    s.n_rows = __ldcg(a->tile_n + s.tt);
    return true;
  }
  // Moves the cursor of a K split (stream-K moves in locate).  The counter's answer may still be in flight on return.
  __device__ __forceinline__ void step() {
    if (stream) return;
    if (a->sched != nullptr) {
      int t = 0;
      if (lane_id() == 0) t = atomicAdd(a->sched, 1);
      u = t;
    } else {
      u += G;
    }
  }
  __device__ __forceinline__ void stepped() {  // ... and is here now
    if (!stream && a->sched != nullptr) u = G + __shfl_sync(0xffffffffu, u, 0);
  }

  // Slots the plan needs (for the capacity check).
  __device__ __forceinline__ long long slots_needed() const {
    if (stream) return 2ll * G;
    return split > 1 ? (long long)units * split : 0;
  }
};

// The ring of published segments.
constexpr int kSegRing = 4;
struct SegRing {
  Seg slot[kSegRing];
  uint64_t full[kSegRing], empty[kSegRing];
  __device__ __forceinline__ void init(int consumers) {
    for (int i = 0; i < kSegRing; ++i) {
      mbar_init(&full[i], 1);
      mbar_init(&empty[i], consumers);
    }
  }
};

// Consumer side (one per warp, the whole warp calls).
struct SegReader {
  SegRing* ring;
  volatile int* abort_flag;
  unsigned long long wait_ns;
  int i = 0;
  uint32_t phase = 0;
  __device__ __forceinline__ SegReader(SegRing* r, volatile int* abort, unsigned long long ns)
      : ring(r), abort_flag(abort), wait_ns(ns) {}
  // The next segment; false at the end of the work, or with `ok` cleared when the wait ran out.
  __device__ __forceinline__ bool next(Seg& s, bool& ok) {
    ok = __all_sync(0xffffffffu, mbar_wait_bounded(&ring->full[i], phase, abort_flag, wait_ns));
    if (!ok) return false;
    const int4* p = reinterpret_cast<const int4*>(&ring->slot[i]);
    const int4 x = p[0], y = p[1], z = p[2];
    s.unit = x.x;
    s.tt = x.y;
    s.mb = x.z;
    s.e = x.w;
    s.row_start = y.x;
    s.n_rows = y.y;
    s.kb0 = y.z;
    s.nkb = y.w;
    s.nseg = z.x;
    s.seg = z.y;
    s.c_first = z.z;
    s.late = z.w;
    __syncwarp();
    if (lane_id() == 0) mbar_arrive(&ring->empty[i]);
    if (++i == kSegRing) {
      i = 0;
      phase ^= 1u;
    }
    return s.unit >= 0;
  }
};

// A CTA pair works on the same segments: CTA 0 asks the counter and leaves each answer here in CTA 1's shared memory.  An answer
// is at most one segment ahead of a K block whose stage CTA 1 has filled (CTA 0's producer waits for that stage's MMA, which
// needs both CTAs' operands), so with up to kPairMail - 2 pipeline stages no answer is overwritten before it is read.
constexpr int kPairMail = 8;
struct PairMail {
  int u[kPairMail];
  uint64_t bar[kPairMail];
  __device__ __forceinline__ void init() {
    for (int i = 0; i < kPairMail; ++i) mbar_init(&bar[i], 1);
  }
};

// Producer side (the weight producer warp, the whole warp calls).  The segment behind the current one is prepared in
// three steps spread over the current one's first K blocks: ask the counter, fetch the tile's words, publish.
// kPair: the two CTAs of a pair (rank 0 and 1) publish the same segments, each in its own ring.
template <bool kPair>
struct SegFeedOf {
  WorkIter it;
  SegRing* ring;
  volatile int* abort_flag;
  unsigned long long wait_ns;
  Seg nx;
  int i = 0, stage = 0;
  uint32_t phase = 0;
  bool have = false, bad_tile = false, ok = true;
  PairMail* mail = nullptr;
  int rank = 0, n_mail = 0;
  __device__ __forceinline__ SegFeedOf(const WorkIter& w, SegRing* r, volatile int* abort, unsigned long long ns)
      : it(w), ring(r), abort_flag(abort), wait_ns(ns) {}

  __device__ __forceinline__ void step() {
    if (!kPair || rank == 0 || it.a->sched == nullptr) it.step();
  }
  __device__ __forceinline__ void stepped() {
    if (!kPair || it.stream || it.a->sched == nullptr) {
      it.stepped();
      return;
    }
    const int i_ = n_mail % kPairMail;
    if (rank == 0) {
      it.stepped();
      if (lane_id() == 0) {
        st_cluster_s32(cluster_map(smem_u32(&mail->u[i_]), 1), it.u);
        mbar_arrive_cluster<true>(cluster_map(smem_u32(&mail->bar[i_]), 1));
      }
      __syncwarp();
    } else {
      ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded<true>(&mail->bar[i_], (uint32_t)(n_mail / kPairMail) & 1u, abort_flag, wait_ns));
      it.u = ok ? *reinterpret_cast<volatile int*>(&mail->u[i_]) : 0x7fffffff;  // (past every unit)
    }
    ++n_mail;
  }

  __device__ __forceinline__ void publish() {
    ok = ok && __all_sync(0xffffffffu, mbar_wait_bounded(&ring->empty[i], phase ^ 1u, abort_flag, wait_ns));
    if (ok && lane_id() == 0) {
      int4* p = reinterpret_cast<int4*>(&ring->slot[i]);
      p[0] = make_int4(have ? nx.unit : -1, nx.tt, nx.mb, nx.e);
      p[1] = make_int4(nx.row_start, nx.n_rows, nx.kb0, nx.nkb);
      p[2] = make_int4(nx.nseg, nx.seg, nx.c_first, nx.late);
      mbar_arrive(&ring->full[i]);
    }
    __syncwarp();
    if (++i == kSegRing) {
      i = 0;
      phase ^= 1u;
    }
  }
  // One of the three steps; after the third the next segment is in `nx` (have == false: there is none).
  __device__ __forceinline__ void advance() {
    if (stage == 0) {
      step();
    } else if (stage == 1) {
      stepped();
      have = it.locate(nx);
    } else if (stage == 2) {
      // a plan built for wider tiles than this kernel: such segments are skipped (and reported); by a pair they are worked
      // through as tiles without rows, since skipping runs ahead of the other CTA
      if (kPair && have && (unsigned)nx.n_rows > (unsigned)it.n_max) {
        bad_tile = true;
        nx.n_rows = 0;
      }
      while (!kPair && have && (unsigned)nx.n_rows > (unsigned)it.n_max) {
        bad_tile = true;
        it.step();
        it.stepped();
        have = it.locate(nx);
      }
      publish();
    }
    if (stage < 3) ++stage;
  }
  __device__ __forceinline__ bool first(Seg& s) {
    have = it.locate(nx);
    stage = 2;
    return next(s);
  }
  __device__ __forceinline__ bool next(Seg& s) {
    while (stage < 3) advance();
    s = nx;
    stage = 0;
    return have && ok;
  }
};
using SegFeed = SegFeedOf<false>;

}  // namespace mf
