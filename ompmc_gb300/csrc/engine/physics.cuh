// Photon/electron transport physics of one lane (one CUDA thread).
//
// Each routine restates the reference routine named in its comment
// (edoerner/ompMC src/ompmc.c, ucodes/omc_dosxyz/omc_dosxyz.c) with the same
// random-number consumption, so a lane processes its histories exactly as a
// thread of the reference does; R is the transport precision (double or
// float), tallies are always FP64.
//
// Two schedules share this code (WF template parameter):
//  - per-lane histories (WF = false): the top particle lives in registers
//    (p, at slot np); slots 0..np-1 live in HBM in the lane's interleaved
//    stack; a lane finishes a history before it takes the next, so a lane
//    with its stream is exactly a thread of the reference;
//  - wavefront (WF = true): p is one particle taken from a photon or
//    electron queue in HBM; every particle an event leaves behind is
//    appended to the queue of its kind (warp-aggregated), and the next
//    phase of the persistent kernel picks it up.
#pragma once

#include <type_traits>

#include "device.cuh"

namespace omcgpu {

#define RC(x) static_cast<R>(x)

template <typename R>
__device__ __forceinline__ R pwlf(const R *c1, const R *c0, int idx, R lv) {
  return lv * __ldg(c1 + idx) + __ldg(c0 + idx);
}

__device__ __forceinline__ V4<float> ld4(const V4<float> *p) {
  float4 v = __ldg(reinterpret_cast<const float4 *>(p));
  return V4<float>{v.x, v.y, v.z, v.w};
}
__device__ __forceinline__ V4<double> ld4(const V4<double> *p) {
  const double2 *q = reinterpret_cast<const double2 *>(p);
  double2 a = __ldg(q), b = __ldg(q + 1);
  return V4<double>{a.x, a.y, b.x, b.y};
}

// One vector load per voxel record.
__device__ __forceinline__ VoxelRec<float> load_voxel(const VoxelRec<float> *p) {
  float2 v = __ldg(reinterpret_cast<const float2 *>(p));
  return VoxelRec<float>{v.x, __float_as_int(v.y)};
}
__device__ __forceinline__ VoxelRec<double> load_voxel(const VoxelRec<double> *p) {
  double2 v = __ldg(reinterpret_cast<const double2 *>(p));
  return VoxelRec<double>{v.x, static_cast<int>(__double_as_longlong(v.y))};
}

// Separately rounded products and sums (never fused into an FMA), where a
// one-ulp difference from the reference's arithmetic matters.
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
// Correctly rounded quotient and square root, also in a fast-math build.
__device__ __forceinline__ float div_rn(float a, float b) { return __fdiv_rn(a, b); }
__device__ __forceinline__ double div_rn(double a, double b) { return __ddiv_rn(a, b); }
__device__ __forceinline__ float sqrt_rn(float a) { return __fsqrt_rn(a); }
__device__ __forceinline__ double sqrt_rn(double a) { return __dsqrt_rn(a); }

__device__ __forceinline__ unsigned lanemask_lt() {
  unsigned m;
  asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
  return m;
}

template <typename R, bool WF, bool MULTI = false, bool HBH = false>
struct Lane {
  const Params<R> &P;
  std::conditional_t<WF, RngPool<R>, Ranmar> rng;
  int lane;
  int slot;  // tally slot of the current history / particle (beamlet jobs;
             // multi-job launches: the job slot)
  int batch; // multi-job launches: batch of the job the particle scores in
  const JobSlot<R> *js;  // multi-job launches: P.jobs + slot
  int np;    // top slot, -1 = empty (per-lane schedule)
  Particle<R> p;
  bool alive;           // wavefront: p still needs to be queued
  bool pending_interaction = false; // wavefront: p ended its step at an interaction
  int single_passes = 1;  // wavefront: steps of one boundary event at most
  unsigned events = 0;  // wavefront: electron steps and photon flights
  R skin = 0;           // wavefront: skin depth of p's last step (0: none, or vacuum)
  R cont_mfp = -1;      // wavefront: mean free paths left of the photon emitted (-1: a new flight)
  R taken_mfp = -1;     // wavefront: mean free paths left of the photon taken (-1: a new flight)
  int flight_cap = kNoFlightCap;  // wavefront: voxel crossings of a photon flight per event
  int gen = 0;          // wavefront: generation and counter slot this phase
  int slot_out = 0;     // appends to
  int dest = QUEUE_NONE;  // wavefront: queue p goes to at the end of the event
  double ensrc;         // per-lane schedule
  double *src_e = nullptr;  // wavefront: source energy of the lane's histories, in shared memory
  unsigned err;
  int max_np;
  // howfar calls (voxel-stepping decisions) and ausgab calls (energy
  // deposits) of this lane; 32 bits on the wavefront path, where a lane has
  // its share of the events of one launch and registers bound the occupancy
  using Count = std::conditional_t<WF, unsigned, unsigned long long>;
  Count n_geom, n_dep;
  // history-by-history scoring (HBH): head block of the current particle's
  // history (-1: not tracked), particles emitted by the current take, the
  // ring entries written before this iteration began, a history this lane
  // completed and its warp is to merge (-1: none), and the warp's merge
  // table in shared memory
  int hblk = -1;
  int hbh_cur = -1;  // block of the history's chain the lane appended to last
  int emitted = 0;
  unsigned long long hbh_pop_limit = 0;
  int hbh_done = -1;
  int *hbh_tir = nullptr;
  double *hbh_tx = nullptr;
  unsigned long long hbh_merged = 0, hbh_split = 0;

  __device__ Lane(const Params<R> &prm, int ln) : P(prm), lane(ln) {
    np = -1;
    slot = 0;
    batch = 0;
    js = nullptr;
    ensrc = 0.0;
    err = 0;
    max_np = 0;
    n_geom = 0;
    n_dep = 0;
    alive = false;
  }

  __device__ __forceinline__ R rnd() {
    if constexpr (WF) {
#ifdef OMC_POOL_CHECK
      if (rng.n <= 0) err |= ERR_EVENTS;  // a need() is missing or too small
#endif
      rng.n = max(rng.n - 1, 0);
      return rng.base[32 * rng.n];
    } else {
      return static_cast<R>(rng.next_int()) * RC(1.0 / 16777216.0);
    }
  }
  // Wavefront: the next k draws find numbers on the lane's stack.
  __device__ __forceinline__ void need(int k) {
    if constexpr (WF) {
      if (rng.n < k) rng.overflow();
    }
  }
  // A number the reference draws and does not use: only where the order of
  // the stream counts.
  __device__ __forceinline__ void skip_rnd() {
    if constexpr (!WF) (void)rnd();
  }

  // Geometry and source of the current particle: the launch's, or its
  // job's in a multi-job launch.
  __device__ __forceinline__ const Geometry<R> &geo() const {
    if constexpr (MULTI) return js->G;
    else return P.G;
  }
  __device__ __forceinline__ const Source<R> &src() const {
    if constexpr (MULTI) return js->S;
    else return P.S;
  }
  __device__ __forceinline__ int tag_value() const {
    if constexpr (MULTI) return slot * kBatchTag + batch;
    else return slot;
  }
  __device__ __forceinline__ void set_tag(int t) {
    if constexpr (MULTI) {
      slot = t / kBatchTag;
      batch = t - slot * kBatchTag;
      js = P.jobs + slot;
    } else {
      slot = t;
    }
  }

  // ---- stack --------------------------------------------------------------
  __device__ __forceinline__ size_t sidx(int slot) const {
    return static_cast<size_t>(slot) * P.nlanes + lane;
  }
  __device__ __forceinline__ void store(int slot, const Particle<R> &q) {
    size_t i = sidx(slot), plane = static_cast<size_t>(P.depth) * P.nlanes;
    R *s = P.stk;
    s[i] = q.e;
    s[i + plane] = q.x;
    s[i + 2 * plane] = q.y;
    s[i + 3 * plane] = q.z;
    s[i + 4 * plane] = q.u;
    s[i + 5 * plane] = q.v;
    s[i + 6 * plane] = q.w;
    s[i + 7 * plane] = q.wt;
    P.stk_key[i] = q.ir * 4 + (q.iq + 1);
  }
  __device__ __forceinline__ void load(int slot, Particle<R> &q) const {
    size_t i = sidx(slot), plane = static_cast<size_t>(P.depth) * P.nlanes;
    const R *s = P.stk;
    q.e = s[i];
    q.x = s[i + plane];
    q.y = s[i + 2 * plane];
    q.z = s[i + 3 * plane];
    q.u = s[i + 4 * plane];
    q.v = s[i + 5 * plane];
    q.w = s[i + 6 * plane];
    q.wt = s[i + 7 * plane];
    int key = P.stk_key[i];
    q.ir = key >> 2;
    q.iq = (key & 3) - 1;
  }
  // Per-lane schedule: the top (p) goes to memory and q becomes the new top
  // (false, history dropped, error flagged, if the stack is full).
  // Wavefront: q is appended to its queue and p stays current.
  __device__ __forceinline__ bool push(const Particle<R> &q) {
    if constexpr (WF) {
      emit(q);
      return true;
    } else {
      if (np + 1 >= P.depth) {
        err |= ERR_STACK;
        np = -1;
        return false;
      }
      store(np, p);
      np += 1;
      p = q;
      if (np > max_np) max_np = np;
      return true;
    }
  }
  // Per-lane schedule: remove the top; wavefront: p is consumed.
  __device__ __forceinline__ void pop() {
    if constexpr (WF) {
      alive = false;
    } else {
      np -= 1;
      if (np >= 0) load(np, p);
    }
  }

  // ---- wavefront queues (layout in device.cuh) ------------------------------
  // The record of slot `slot` in the queue of kind `kind`, generation g.
  __device__ __forceinline__ char *record(int kind, int g, unsigned slot) const {
    const QueueLayout &q = P.q;
    const unsigned blk = kind == QUEUE_PH ? q.block_ph : q.block;
    const size_t at = kind == QUEUE_PH ? g * q.bytes_ph : 2 * q.bytes_ph + (2 * (kind - 1) + g) * q.bytes;
    return q.base + at + static_cast<size_t>(slot >> 5) * blk + (slot & 31) * sizeof(R);
  }
  // Key and tag planes are 4-byte: their lane offset from the record.
  __device__ __forceinline__ static int *int_plane(char *rec, unsigned slot, int k) {
    return reinterpret_cast<int *>(rec + 8 * 32 * sizeof(R) + 128 * k - (slot & 31) * (sizeof(R) - 4));
  }
  // Mean free paths left of a photon flight: the last plane.
  __device__ __forceinline__ R *mfp_plane(char *rec) const {
    return reinterpret_cast<R *>(rec + P.q.block);
  }
  __device__ __forceinline__ void store_slot(int kind, unsigned slot, const Particle<R> &q, R mfp) {
    char *rec = record(kind, gen, slot);
    R *f = reinterpret_cast<R *>(rec);
    __stcg(f, q.e);
    __stcg(f + 32, q.x);
    __stcg(f + 64, q.y);
    __stcg(f + 96, q.z);
    __stcg(f + 128, q.u);
    __stcg(f + 160, q.v);
    __stcg(f + 192, q.w);
    __stcg(f + 224, q.wt);
    __stcg(int_plane(rec, slot, 0), q.ir * 4 + (q.iq + 1));
    if constexpr (HBH) {
      __stcg(int_plane(rec, slot, 1), hblk);
      emitted++;
    } else if (P.q.tags) {
      __stcg(int_plane(rec, slot, 1), tag_value());
    }
    if (kind == QUEUE_PH) __stcg(mfp_plane(rec), mfp);
  }
  // Append position idx of a queue: its slot, or false (error flagged) if
  // the queue is full.  Boundary electrons share the electron queue's
  // buffer: the others fill it from slot 0 up, the boundary electrons from
  // the top down, so together they have the one queue's worst-case room.
  __device__ __forceinline__ void store_at(int kind, unsigned idx, const Particle<R> &q, R mfp) {
    if (idx >= P.q.cap) {
      err |= ERR_QUEUE;
      return;
    }
    const bool b = kind == QUEUE_EB;
    store_slot(b ? QUEUE_EL : kind, b ? P.q.cap - 1 - idx : idx, q, mfp);
  }
  // Append at once (secondaries, split photons): the lanes that are here
  // together share one atomic.
  __device__ __forceinline__ void emit_to(int kind, const Particle<R> &q) {
    unsigned m = __activemask();
    int leader = __ffs(m) - 1;
    unsigned base = 0;
    if ((threadIdx.x & 31) == leader)
      base = atomicAdd(queue_ctr(P.q.ctr, kind, slot_out), static_cast<unsigned>(__popc(m)));
    base = __shfl_sync(m, base, leader);
    store_at(kind, base + __popc(m & lanemask_lt()), q, RC(-1));
  }
  __device__ __forceinline__ void emit(const Particle<R> &q) {
    if (q.iq == 0) emit_to(QUEUE_PH, q);
    else emit_to(QUEUE_EL, q);
  }
  // A photon at its interaction point.  Its key holds iq + 1 = 1 for a
  // split whose scattered photon is dropped and 3 for the surviving one.
  __device__ __forceinline__ void emit_photon_interaction(const Particle<R> &q, bool survivor) {
    Particle<R> t = q;
    t.iq = survivor ? 2 : 0;
    emit_to(QUEUE_PI, t);
  }
  // The particle an event leaves (p, bound for queue dest) for the whole
  // warp at once: called by all 32 lanes at the end of a chunk, so that a
  // chunk costs one atomic instruction -- one lane per destination queue --
  // and its records land side by side.  Appends in the divergent code of
  // the events took about three, and a copy of the record store each.
  // Measured with the blocked record layout: 6 MV slab FP32 959 -> 942 ms,
  // 250 kVp job 7.9 -> 7.4 ms, positron field 57.7 -> 54.8 ms, nsplit 16 job
  // 44.3 -> 40.2 ms; registers 96 -> 91 (FP32) and 248 -> 210 (FP64).
  __device__ __forceinline__ void flush() {
    const unsigned full = 0xffffffffu;
    const unsigned m = __match_any_sync(full, dest);
    const int leader = __ffs(m) - 1;
    unsigned base = 0;
    if (dest >= 0 && (threadIdx.x & 31) == leader)
      base = atomicAdd(queue_ctr(P.q.ctr, dest, slot_out), static_cast<unsigned>(__popc(m)));
    base = __shfl_sync(full, base, leader);
    if (dest >= 0) store_at(dest, base + __popc(m & lanemask_lt()), p, cont_mfp);
    dest = QUEUE_NONE;
    cont_mfp = RC(-1);
  }
  // Where an electron goes after its step (or the particle left on top of
  // its take).  Electrons go to one of two queues by the kind of step they
  // will take next, so that a warp's chunk runs one of the two branches of
  // the step (ompmc.c:4963-5048).  Within the skin depth of a boundary
  // (hownear <= skindepth) the step is a single-scattering step: tustep is
  // capped at max(tperp, skindepth), so the test tustep > skindepth of the
  // condensed-history branch fails.  The skin depth is the last step's,
  // taken at the slightly higher energy before the step; on the 6 MV slab
  // the guess matches the branch taken in 99.7% of the steps.  Only the
  // order in which particles are processed changes.
  __device__ __forceinline__ int step_queue() const {
    if (p.iq == 0) return QUEUE_PH;
    return skin > RC(0) && hownear(p) <= skin ? QUEUE_EB : QUEUE_EL;
  }
  __device__ __forceinline__ void take(int kind, int g, unsigned slot) {
    char *rec = record(kind, g, slot);
    if constexpr (HBH) {
      // The tag is the history's head block; the block holds the tally slot.
      hblk = __ldcg(int_plane(rec, slot, 1));
      emitted = 0;
      hbh_cur = hblk;
      if (hblk >= 0) this->slot = __ldcg(&P.hbh.blocks[hblk].slot);
    } else if (P.q.tags) {
      set_tag(__ldcg(int_plane(rec, slot, 1)));
    }
    const R *f = reinterpret_cast<const R *>(rec);
    p.e = __ldcg(f);
    p.x = __ldcg(f + 32);
    p.y = __ldcg(f + 64);
    p.z = __ldcg(f + 96);
    p.u = __ldcg(f + 128);
    p.v = __ldcg(f + 160);
    p.w = __ldcg(f + 192);
    p.wt = __ldcg(f + 224);
    int key = __ldcg(int_plane(rec, slot, 0));
    p.ir = key >> 2;
    p.iq = (key & 3) - 1;
    if (kind == QUEUE_PH) taken_mfp = __ldcg(mfp_plane(rec));
    alive = true;
  }

  // ---- scoring: ausgab (omc_dosxyz.c:683-694) ------------------------------
  __device__ __forceinline__ void ausgab(int ir, R wt, R edep) {
    n_dep++;
    if constexpr (MULTI)
      atomicAdd(js->tally + static_cast<size_t>(batch) * js->nreg + ir, static_cast<double>(wt * edep));
    else
      atomicAdd(P.endep + static_cast<size_t>(slot) * P.tally_stride + ir, static_cast<double>(wt * edep));
    if constexpr (HBH) hbh_append(ir, wt * edep);
  }

  // ---- history-by-history scoring (HBH) --------------------------------------
  __device__ int hbh_pop() {
    const unsigned long long i = atomicAdd(P.hbh.ctr + 1, 1ull);
    if (i >= hbh_pop_limit) {
      atomicAdd(P.hbh.ctr + 1, ~0ull);  // undo: no entry written before this iteration is left
      err |= ERR_HISTORY;
      return -1;
    }
    return __ldcg(P.hbh.ring + (i & P.hbh.ring_mask));
  }
  __device__ void hbh_push(int b) {
    const unsigned long long i = atomicAdd(P.hbh.ctr, 1ull);
    __stcg(P.hbh.ring + (i & P.hbh.ring_mask), b);
  }
  // A new history: its head block, with no particle counted yet.  The
  // lanes that start histories together take their blocks with one atomic.
  __device__ void hbh_start() {
    emitted = 0;
    const unsigned am = __activemask();
    const int leader = __ffs(am) - 1;
    const unsigned cnt = __popc(am);
    unsigned long long b = 0;
    if ((threadIdx.x & 31) == leader) {
      b = atomicAdd(P.hbh.ctr + 1, static_cast<unsigned long long>(cnt));
      if (b + cnt > hbh_pop_limit) {  // undo the ids that are not there this iteration
        const unsigned long long over = b + cnt - (b > hbh_pop_limit ? b : hbh_pop_limit);
        atomicAdd(P.hbh.ctr + 1, 0ull - over);
      }
    }
    b = __shfl_sync(am, b, leader);
    const unsigned long long i = b + __popc(am & lanemask_lt());
    if (i >= hbh_pop_limit) {
      err |= ERR_HISTORY;
      hblk = hbh_cur = -1;
      return;
    }
    hblk = __ldcg(P.hbh.ring + (i & P.hbh.ring_mask));
    HbhBlock<R> *h = P.hbh.blocks + hblk;
    __stcg(&h->count, 0);
    __stcg(&h->next, -1);
    __stcg(&h->live, 0);
    __stcg(&h->slot, slot);
    __stcg(&h->tail, -1);
    hbh_cur = hblk;
  }
  // Append (region, energy) to the history's chain; a full block gets a
  // continuation block (the first lane to install one wins, the others
  // return theirs).  The search for room starts at the block the lane used
  // last, and goes from a full head block to the one the head names as near
  // the end: a track along a voxel boundary makes thousands of deposits, and
  // walking its chain from the head for each took the time of the square of
  // their number (the runs of a 6e6-history job spread from 70 to 104 ms).
  // Measured, FP32: that job 71 -> 43.5 ms, now within 2%; 6 MV slab on 2 mm
  // voxels, 2e7 histories, 570 -> 368 ms; FP64, 2e6 histories, 161 -> 118 ms.
  __device__ void hbh_append(int ir, R x) {
    int b = hbh_cur;
    for (int guard = 0; b >= 0 && guard < 1024; guard++) {
      HbhBlock<R> *blk = P.hbh.blocks + b;
      const int i = atomicAdd(&blk->count, 1);
      if (i < HbhBlock<R>::kEntries) {
        __stcg(&blk->ir[i], ir);
        __stcg(&blk->x[i], x);
        hbh_cur = b;
        return;
      }
      int nb = -1;
      if (b == hblk) nb = *static_cast<volatile int *>(&blk->tail);
      if (nb < 0) nb = *static_cast<volatile int *>(&blk->next);
      if (nb < 0) {
        const int cand = hbh_pop();
        if (cand < 0) return;  // pool empty: this deposit is missing from the history sums (flagged)
        HbhBlock<R> *c = P.hbh.blocks + cand;
        __stcg(&c->count, 0);
        __stcg(&c->next, -1);
        __threadfence();
        const int old = atomicCAS(&blk->next, -1, cand);
        if (old == -1) {
          nb = cand;
          __stcg(&P.hbh.blocks[hblk].tail, cand);
        } else {
          hbh_push(cand);
          nb = old;
        }
      }
      b = nb;
    }
    err |= ERR_HISTORY;
  }
  // End of a take (consumed = 1) or of an injection (consumed = 0): the
  // history's particle count changes by emitted - consumed; at zero the
  // history is complete, and this lane hands it to its warp's merge.
  __device__ void hbh_finish(int consumed) {
    if (hblk < 0) return;
    const int delta = emitted - consumed;
    emitted = 0;
    if (delta == 0) {
      hblk = -1;  // every lane comes here after a chunk, with or without a take
      return;
    }
    __threadfence();  // this lane's appends before the count
    const int left = atomicAdd(&P.hbh.blocks[hblk].live, delta) + delta;
    if (left == 0) {
      __threadfence();  // every other lane's appends before the merge
      hbh_done = hblk;
    }
    hblk = -1;
  }
  // The warp merges the histories its lanes completed, one after another
  // and all 32 lanes on each: the lanes load a block's entries together and
  // sum them per region in the warp's shared-memory table, then score each
  // region's total x as x (sum) and x^2 (sum2) and return the blocks.  A
  // history over the table's regions is scored in parts (counted in split).
  // Called by all 32 lanes of the warp at the same point.
  __device__ void hbh_warp_merge() {
    const unsigned full = 0xffffffffu;
    const int lane_id = threadIdx.x & 31;
    unsigned pending = __ballot_sync(full, hbh_done >= 0);
    while (pending) {
      const int src = __ffs(pending) - 1;
      pending &= pending - 1;
      const int head = __shfl_sync(full, hbh_done, src);
      for (int k = lane_id; k < kHbhRegions; k += 32) {
        hbh_tir[k] = -1;
        hbh_tx[k] = 0.0;
      }
      __syncwarp();
      bool split = false;
      int b = head;
      int mine = -1;  // block `guard` of the chain when guard == this lane
      for (int guard = 0; b >= 0 && guard < (1 << 20); guard++) {
        const HbhBlock<R> *blk = P.hbh.blocks + b;
        const int n = min(__ldcg(&blk->count), HbhBlock<R>::kEntries);
        const int nb = __ldcg(&blk->next);
        for (int i = lane_id; i < n; i += 32) {
          const int ir = __ldcg(&blk->ir[i]);
          const double x = static_cast<double>(__ldcg(&blk->x[i]));
          unsigned h = (static_cast<unsigned>(ir) * 2654435761u) >> 25;  // 7 bits: kHbhRegions = 128
          int probe = 0;
          for (; probe < kHbhRegions; probe++) {
            const int old = atomicCAS(hbh_tir + h, -1, ir);
            if (old == -1 || old == ir) {
              atomicAdd(hbh_tx + h, x);
              break;
            }
            h = (h + 1) & (kHbhRegions - 1);
          }
          if (probe == kHbhRegions) {  // table full: this deposit scores as a part of its own
            atomicAdd(P.hbh.sum + ir, x);
            atomicAdd(P.hbh.sum2 + ir, x * x);
            split = true;
          }
        }
        if (guard < 32) {
          if (lane_id == guard) mine = b;
        } else if (lane_id == 0) {
          hbh_push(b);  // chains over 32 blocks: the rest one by one
        }
        b = nb;
      }
      // Return the chain's first 32 blocks with one atomic.
      const unsigned have = __ballot_sync(full, mine >= 0);
      if (have) {
        unsigned long long base = 0;
        if (lane_id == 0) base = atomicAdd(P.hbh.ctr, static_cast<unsigned long long>(__popc(have)));
        base = __shfl_sync(full, base, 0);
        if (mine >= 0) __stcg(P.hbh.ring + ((base + __popc(have & lanemask_lt())) & P.hbh.ring_mask), mine);
      }
      __syncwarp();
      for (int k = lane_id; k < kHbhRegions; k += 32) {
        const int ir = hbh_tir[k];
        if (ir < 0) continue;
        const double x = hbh_tx[k];
        atomicAdd(P.hbh.sum + ir, x);
        atomicAdd(P.hbh.sum2 + ir, x * x);
      }
      __syncwarp();
      split = __any_sync(full, split);
      if (lane_id == src) {
        hbh_done = -1;
        hbh_merged++;
        if (split) hbh_split++;
      }
    }
  }

  // ---- geometry: region decode, howfar, hownear (omc_dosxyz.c:187-334) ----
  __device__ __forceinline__ VoxelRec<R> voxel(int ir) const { return load_voxel(geo().vox + ir); }
  __device__ __forceinline__ int med_of(int ir) const { return voxel(ir).med; }
  __device__ __forceinline__ R rhof_of(int ir) const { return voxel(ir).rhof; }
  __device__ __forceinline__ R ecut_of(int ir) const { return __ldg(geo().ecut_m + med_of(ir) + 1); }
  __device__ __forceinline__ R pcut_of(int ir) const { return __ldg(geo().pcut_m + med_of(ir) + 1); }

  // Voxel indices of region irl >= 1: irl = 1 + ix + iy*nx + iz*nx*ny.
  __device__ __forceinline__ void decode(int irl, int &ix, int &iy, int &iz) const {
    const Geometry<R> &g = geo();
    const unsigned n = static_cast<unsigned>(irl - 1);
    const unsigned z = divide(n, g.div_nxy);
    const unsigned rem = n - z * static_cast<unsigned>(g.nxy);
    const unsigned y = divide(rem, g.div_nx);
    ix = static_cast<int>(rem - y * static_cast<unsigned>(g.nx));
    iy = static_cast<int>(y);
    iz = static_cast<int>(z);
  }

  __device__ void howfar(const Particle<R> &q, int &idisc, int &irnew, R &ustep) {
    const Geometry<R> &g = geo();
    n_geom++;
    int irl = q.ir;
    if (irl == 0) {
      idisc = 1;
      return;
    }
    int irx, iry, irz;
    decode(irl, irx, iry, irz);
    R dist;
    if (q.w > RC(0)) {
      dist = (__ldg(g.zb + irz + 1) - q.z) / q.w;
      if (dist < ustep) {
        ustep = dist;
        irnew = (irz != g.nz - 1) ? irl + g.nxy : 0;
      }
    } else if (q.w < RC(0)) {
      dist = -(q.z - __ldg(g.zb + irz)) / q.w;
      if (dist < ustep) {
        ustep = dist;
        irnew = (irz != 0) ? irl - g.nxy : 0;
      }
    }
    if (q.u > RC(0)) {
      dist = (__ldg(g.xb + irx + 1) - q.x) / q.u;
      if (dist < ustep) {
        ustep = dist;
        irnew = (irx != g.nx - 1) ? irl + 1 : 0;
      }
    } else if (q.u < RC(0)) {
      dist = -(q.x - __ldg(g.xb + irx)) / q.u;
      if (dist < ustep) {
        ustep = dist;
        irnew = (irx != 0) ? irl - 1 : 0;
      }
    }
    if (q.v > RC(0)) {
      dist = (__ldg(g.yb + iry + 1) - q.y) / q.v;
      if (dist < ustep) {
        ustep = dist;
        irnew = (iry != g.ny - 1) ? irl + g.nx : 0;
      }
    } else if (q.v < RC(0)) {
      dist = -(q.y - __ldg(g.yb + iry)) / q.v;
      if (dist < ustep) {
        ustep = dist;
        irnew = (iry != 0) ? irl - g.nx : 0;
      }
    }
  }

  // a < b and min(a, b) for distances.  In FP64 on the wavefront path the
  // comparison is one of the bit patterns, on the integer pipe: an FP64
  // compare takes 16 cycles of a pipe that all warps of the SM share.  (Two
  // negative distances, which only rounding makes, compare the other way
  // round.)  6 MV slab FP64, 2 mm, 1e7 histories: 965 -> 909 ms.
  __device__ __forceinline__ static bool closer(R a, R b) {
    if constexpr (WF && sizeof(R) == 8) return __double_as_longlong(a) < __double_as_longlong(b);
    else return a < b;
  }
  __device__ __forceinline__ static R nearer(R a, R b) {
    if constexpr (WF && sizeof(R) == 8) return closer(b, a) ? b : a;
    else return fmin(a, b);
  }

  __device__ R hownear(const Particle<R> &q) const {
    const Geometry<R> &g = geo();
    int irl = q.ir;
    if (irl == 0) return RC(0);
    int irx, iry, irz;
    decode(irl, irx, iry, irz);
    R t = RC(1.0E10);
    t = nearer(t, __ldg(g.xb + irx + 1) - q.x);
    t = nearer(t, q.x - __ldg(g.xb + irx));
    t = nearer(t, __ldg(g.yb + iry + 1) - q.y);
    t = nearer(t, q.y - __ldg(g.yb + iry));
    t = nearer(t, __ldg(g.zb + irz + 1) - q.z);
    t = nearer(t, q.z - __ldg(g.zb + irz));
    return t;
  }

  // ---- packed interpolation records ---------------------------------------
  __device__ __forceinline__ size_t eidx(int qel, int m, int l) const {
    return (static_cast<size_t>(qel) * P.T.nmed + m) * MXEKE + l;
  }
  __device__ __forceinline__ V4<R> esd(int qel, int m, int l) const { return ld4(P.T.el_sd + eidx(qel, m, l)); }
  __device__ __forceinline__ V4<R> ete(int qel, int m, int l) const { return ld4(P.T.el_te + eidx(qel, m, l)); }
  __device__ __forceinline__ V4<R> erg(int qel, int m, int l) const { return ld4(P.T.el_rg + eidx(qel, m, l)); }
  __device__ __forceinline__ V4<R> eq(int qel, int m, int l) const { return ld4(P.T.el_q + eidx(qel, m, l)); }

  // ---- interpolation indices, clamped to the table --------------------------
  __device__ __forceinline__ int photon_bin(int imed, R gle) {
    int l = static_cast<int>(gle * __ldg(P.T.ge1 + imed) + __ldg(P.T.ge0 + imed)) - 1;
    if (l < 0 || l >= MXGE) {
      err |= ERR_TABLE;
      l = l < 0 ? 0 : MXGE - 1;
    }
    return l;
  }
  __device__ __forceinline__ int electron_bin(int imed, R elke) {
    int l = static_cast<int>(elke * __ldg(P.T.eke1 + imed) + __ldg(P.T.eke0 + imed)) - 1;
    int top = __ldg(P.T.meke + imed) - 1;
    if (l < 0 || l > top) {
      err |= ERR_TABLE;
      l = l < 0 ? 0 : top;
    }
    return l;
  }

  // ---- rotations (ompmc.c:101-201) ------------------------------------------
  struct Uphi {
    R A, B, C, cosphi, sinphi;
  };

  // cos and sin of a uniform azimuth.  The reference's box method accepts
  // pi/4 of its pairs, so a warp runs on until the unluckiest of its lanes
  // is through (3.3 rounds of two draws on average, 1.3 for a lane).  In
  // FP32 the wavefront path takes the angle itself from one draw; in FP64
  // sincospi would cost 2.5 times the FP64 instructions of the rounds.
  __device__ void azimuth(R &cphi, R &sphi) {
    if constexpr (WF && sizeof(R) == 4) {
      sincospif(RC(2) * rnd(), &sphi, &cphi);
      return;
    }
    R xphi, xphi2, yphi, yphi2, rhophi2;
    int guard = 0;
    do {
      need(2);
      xphi = rnd();
      xphi = RC(2) * xphi - RC(1);
      xphi2 = xphi * xphi;
      yphi = rnd();
      yphi2 = yphi * yphi;
      rhophi2 = xphi2 + yphi2;
      if (++guard > kRejectCap) {
        err |= ERR_LOOP;
        break;
      }
    } while (rhophi2 > RC(1));
    rhophi2 = RC(1) / rhophi2;
    cphi = (xphi2 - yphi2) * rhophi2;
    sphi = RC(2) * xphi * yphi * rhophi2;
  }

  __device__ __forceinline__ static void rotate(Particle<R> &q, const Uphi &up, R costhe, R sinthe) {
    R sinps2 = up.A * up.A + up.B * up.B;
    if (sinps2 < RC(1.0E-20)) {
      q.u = sinthe * up.cosphi;
      q.v = sinthe * up.sinphi;
      q.w = up.C * costhe;
    } else {
      R sinpsi = sqrt(sinps2);
      R us = sinthe * up.cosphi;
      R vs = sinthe * up.sinphi;
      R sindel = up.B / sinpsi;
      R cosdel = up.A / sinpsi;
      q.u = up.C * cosdel * us - sindel * vs + up.A * costhe;
      q.v = up.C * sindel * us + cosdel * vs + up.B * costhe;
      q.w = -sinpsi * us + up.C * costhe;
    }
  }

  // uphi21: new direction of q itself, azimuth sampled here.
  __device__ void uphi21(Particle<R> &q, Uphi &up, R costhe, R sinthe) {
    azimuth(up.cosphi, up.sinphi);
    up.A = q.u;
    up.B = q.v;
    up.C = q.w;
    rotate(q, up, costhe, sinthe);
  }
  // uphi32: a second particle at the position of `from`, rotated from the
  // direction saved in up (transferProperties + rotation, ompmc.c:166-201).
  __device__ static void uphi32(Particle<R> &q, const Particle<R> &from, const Uphi &up, R costhe, R sinthe) {
    q.x = from.x;
    q.y = from.y;
    q.z = from.z;
    q.ir = from.ir;
    q.wt = from.wt;
    rotate(q, up, costhe, sinthe);
  }

#include "photon.inc"
#include "electron.inc"
#include "wf_electron.inc"

  // ---- source -------------------------------------------------------------
  // Energy and charge of a new history (initHistory's first part, the same
  // in omc_dosxyz.c:970-996 and omc_matrad.c:1092-1123).
  __device__ __forceinline__ void source_energy(Particle<R> &q) {
    const Source<R> &s = src();
    q.iq = s.charge;
    R ein;
    if (s.spectrum) {
      R rnno1 = rnd();
      R rnno2 = rnd();
      int k = static_cast<int>(fmin(s.deltak * rnno1, s.deltak - RC(1)));
      ein = __ldg(s.cdfinv1 + k) + rnno2 * __ldg(s.cdfinv2 + k);
    } else {
      ein = s.energy;
    }
    q.e = (q.iq != 0) ? ein + RC(0.5109989461) : ein;
    if constexpr (MULTI) atomicAdd(js->ensrc, static_cast<double>(ein));
    else if constexpr (WF) *src_e += static_cast<double>(ein);
    else ensrc += static_cast<double>(ein);
  }

  // History h of the launch: its tally slot (beamlet jobs), then the
  // source particle.
  __device__ void init_history(long long h) {
    if (P.nslots > 0) {
      int lo = 0, hi = P.nslots - 1;
      while (lo < hi) {  // last slot whose first history is <= h
        int mid = (lo + hi + 1) >> 1;
        if (__ldg(P.slot_first + mid) <= h) lo = mid;
        else hi = mid - 1;
      }
      slot = lo;
    }
    if constexpr (MULTI) {
      js = P.jobs + slot;
      const long long hj = js->h0 + (h - __ldg(P.slot_first + slot));
      if (js->nbl > 0) {
        int lo = 0, hi = js->nbl - 1;
        while (lo < hi) {  // last beamlet whose first history is <= hj
          int mid = (lo + hi + 1) >> 1;
          if (__ldg(js->bl_first + mid) <= hj) lo = mid;
          else hi = mid - 1;
        }
        batch = lo;
        init_beamlet_history(lo);
      } else {
        batch = static_cast<int>(hj / js->nperbatch);
        init_point_history();
      }
    } else {
      if (P.S.beamlets) init_beamlet_history(__ldg(P.slot_beamlet + slot));
      else init_point_history();
    }
  }

  // initHistory(ibeamlet) (omc_matrad.c:1084-1254): a uniform point of the
  // bixel, moved back along the line to the beam's source point onto the
  // phantom surface, heading into the phantom.  The reference clamps z
  // against ybounds[0] (:1225); that is kept.  A point that lands a
  // rounding error below zbounds[0] is moved by that clamp, so the
  // arithmetic here is rounded operation by operation like the
  // reference's: no fused multiply-adds, and correctly rounded division
  // and square root.
  __device__ void init_beamlet_history(int ib) {
    const Source<R> &s = src();
    const Geometry<R> &g = geo();
    Particle<R> q;
    source_energy(q);
    R rnno1 = rnd();
    R rnno2 = rnd();
    const R *b = s.bixel + static_cast<size_t>(ib) * 9;
    R xiso = add_rn(add_rn(mul_rn(rnno1, __ldg(b + 3)), mul_rn(rnno2, __ldg(b + 6))), __ldg(b + 0));
    R yiso = add_rn(add_rn(mul_rn(rnno1, __ldg(b + 4)), mul_rn(rnno2, __ldg(b + 7))), __ldg(b + 1));
    R ziso = add_rn(add_rn(mul_rn(rnno1, __ldg(b + 5)), mul_rn(rnno2, __ldg(b + 8))), __ldg(b + 2));
    const R *src = s.beam_src + 3 * __ldg(s.ibeam + ib);
    R dx = xiso - __ldg(src + 0), dy = yiso - __ldg(src + 1), dz = ziso - __ldg(src + 2);
    R vnorm = sqrt_rn(add_rn(add_rn(mul_rn(dx, dx), mul_rn(dy, dy)), mul_rn(dz, dz)));
    R u = div_rn(-dx, vnorm), v = div_rn(-dy, vnorm), w = div_rn(-dz, vnorm);
    R ustep = RC(1.0E5), dist;
    const R x0 = __ldg(g.xb), x1 = __ldg(g.xb + g.nx);
    const R y0 = __ldg(g.yb), y1 = __ldg(g.yb + g.ny);
    const R z0 = __ldg(g.zb), z1 = __ldg(g.zb + g.nz);
    if (u > RC(0)) {
      dist = div_rn(x1 - xiso, u);
      if (dist < ustep) ustep = dist;
    }
    if (u < RC(0)) {
      dist = div_rn(-(xiso - x0), u);
      if (dist < ustep) ustep = dist;
    }
    if (v > RC(0)) {
      dist = div_rn(y1 - yiso, v);
      if (dist < ustep) ustep = dist;
    }
    if (v < RC(0)) {
      dist = div_rn(-(yiso - y0), v);
      if (dist < ustep) ustep = dist;
    }
    if (w > RC(0)) {
      dist = div_rn(z1 - ziso, w);
      if (dist < ustep) ustep = dist;
    }
    if (w < RC(0)) {
      dist = div_rn(-(ziso - z0), w);
      if (dist < ustep) ustep = dist;
    }
    R x = add_rn(xiso, mul_rn(ustep, u)), y = add_rn(yiso, mul_rn(ustep, v)), z = add_rn(ziso, mul_rn(ustep, w));
    q.u = -u;
    q.v = -v;
    q.w = -w;
    const R tiny = RC(2.0 * 2.2250738585072014e-308);  // 2*DBL_MIN
    if (x < x0) x = x0 + tiny;
    if (x > x1) x = x1 - tiny;
    if (y < y0) y = y0 + tiny;
    if (y > y1) y = y1 - tiny;
    if (z < z0) z = y0 + tiny;
    if (z > z1) z = z1 - tiny;
    q.x = x;
    q.y = y;
    q.z = z;
    int ix = 0, iy = 0, iz = 0;
    while (ix < g.nx - 1 && __ldg(g.xb + ix + 1) < x) ix++;
    while (iy < g.ny - 1 && __ldg(g.yb + iy + 1) < y) iy++;
    while (iz < g.nz - 1 && __ldg(g.zb + iz + 1) < z) iz++;
    q.ir = 1 + ix + iy * g.nx + iz * g.nxy;
    q.wt = RC(1);
    p = q;
    np = 0;
  }

  // initHistory (omc_dosxyz.c:964-1068): collimated point source.
  __device__ void init_point_history() {
    const Source<R> &s = src();
    const Geometry<R> &g = geo();
    Particle<R> q;
    source_energy(q);
    R rxyz;
    if (s.xsize == RC(0) || s.ysize == RC(0)) {
      q.x = s.xinl;
      q.y = s.yinl;
      rxyz = sqrt(s.ssd * s.ssd + q.x * q.x + q.y * q.y);
      q.w = s.ssd / rxyz;
    } else {
      R fw, rnno3;
      int guard = 0;
      do {
        need(3);
        rnno3 = rnd();
        q.x = rnno3 * s.xsize + s.xinl;
        rnno3 = rnd();
        q.y = rnno3 * s.ysize + s.yinl;
        rnno3 = rnd();
        rxyz = sqrt(s.ssd * s.ssd + q.x * q.x + q.y * q.y);
        q.w = s.ssd / rxyz;
        fw = q.w * q.w * q.w;
        if (++guard > kRejectCap) {
          err |= ERR_LOOP;
          break;
        }
      } while (rnno3 >= fw);
    }
    q.z = __ldg(g.zb + 0);
    q.u = q.x / rxyz;
    q.v = q.y / rxyz;
    int ix, iy;
    if (s.xsize == RC(0)) {
      ix = s.ixinl;
    } else {
      ix = s.ixinl - 1;
      while ((__ldg(g.xb + ix + 1) < q.x) && ix < g.nx - 1) ix++;
    }
    if (s.ysize == RC(0)) {
      iy = s.iyinl;
    } else {
      iy = s.iyinl - 1;
      while ((__ldg(g.yb + iy + 1) < q.y) && iy < g.ny - 1) iy++;
    }
    q.ir = 1 + ix + iy * g.nx;
    q.wt = RC(1);
    p = q;
    np = 0;
  }
};

#undef RC

}  // namespace omcgpu
