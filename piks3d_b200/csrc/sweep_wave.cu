// Octant sweeps (solver.F90:176-526) over the hyperplane-column schedule (WaveJobs).
//
// A work item is one column of an octant (a cross-section of A x B cells of the octant's
// frame over the whole z extent) for one chunk of V velocities. A persistent CTA takes items
// in dependency order and marches each along the hyperplanes u + v + w: batch k holds the
// column's tasks of one hyperplane, which are independent of one another, and the rows they
// read. Rows live in a ring in shared memory: a batch's rows are read by its own tasks and
// by the next two batches (the scheme reaches two cells upwind), so a row is staged once per
// column and only the two upwind layers of the neighbouring columns are staged twice.
//   request warp    takes items and, four batches at a time, requests their row lists and task
//                   records by bulk asynchronous copies on the group's `meta` mbarrier;
//   go warp         lets a batch's rows in once the ring has room for them;
//   dep warp        lets in the rows of upwind columns once those have published the hyperplane;
//   copy warps      gather a batch's rows and moments together by 16-byte cp.async that arrive
//                   on its `full` mbarrier, two rows per warp instruction;
//   consumer warps  update the batch's tasks, LPT lanes per task, 16 bytes of velocities per
//                   lane; each result goes to the row's ring slot and to HBM; a warp arrives
//                   on the batch's `done` mbarrier;
//   publish warp    follows `done` and tells the downwind columns (a release store of the
//                   column's progress, which takes a thousand cycles and holds up nothing here).
// One warp that did requests, room, progress and copies took 7000 cycles a batch (in a warp by
// itself each instruction waits for the one before), five times what eight consumer warps take
// for its tasks; the roles are separate warps so that none takes longer than the consumers.
// Items are claimed in an order in which every upwind column comes first, by CTAs that are
// running, so the earliest unfinished item can always proceed. Every wait is bounded
// (kWaitNs): a progress wait that gives up sets the error flag and goes on with stale rows;
// an mbarrier wait that gives up sets the error flag and the CTA's abort flag, on which every
// warp leaves, the copying ones after their own copies are complete. Warps leave one by one, so
// after the first of these waits they meet on mbarriers only, never on a counted barrier.
//
// What bounds it and why this shape: the tile-diagonal kernel staged 2.4 (FP64) to 2.6
// (FP32) rows per swept row, each CTA as one chain of metadata, rows, ten to fourteen local
// hyperplanes with a few tasks each, and write-back. Here a hyperplane of a column holds
// tens of tasks, the loads of the next ones run meanwhile, and about 1.5 rows are staged. What is
// left is some 930 cycles a batch for the hand-over to the next hyperplane, and 30 (FP64) to 32 (FP32)
// a task, whose shared-memory accesses are 35 and 33 wavefronts (fitted over packs of five porosities
// with 7 x 7 and 8 x 8 columns; wider ones take 4 to 25 % more, as the ring no longer holds the next
// batches' rows); short columns wait for the chain of upwind columns. Sweep per iteration, tile
// diagonals / this: 128^3 pack, 512 velocities, FP64 5.31 / 2.70 ms, FP32 2.66 / 1.43; 100^3 quarter
// sphere FP64 5.58 / 2.43; 48^3 pack FP64 0.598 / 0.256; 256^3 field of porosity 0.20, FP32, 8.98 /
// 6.55; 96^3 pack, 64 velocities, FP32 0.72 / 0.316; 75 x 53 x 37, 216 velocities an octant, FP64 2.28 /
// 0.95.
#include <cuda_runtime.h>

#include <algorithm>

#include "kernels.h"
#include "piks_internal.h"
#include "sweep_core.cuh"

namespace piks {

namespace {

using namespace sweep;

constexpr int kStages = 16;      // batches between request and completion (mbarrier stages)
constexpr int kGroup = kWaveGroup;  // batches of one request
constexpr int kGroups = kStages / kGroup;
constexpr int kLists = 3;        // groups whose row lists are held
constexpr int kDone = 1 << 30;   // progress of a finished column
// Warps of a CTA (one per SM): consumers, the copy warps in teams that take batches in turn,
// then the request, go, dep and publish warps; whole warpgroups of either kind.
constexpr int kConsumers = 16, kTeam = 4, kTeams = 2, kOthers = kTeam * kTeams + 4;
constexpr int kThreads = (kConsumers + kOthers) * 32;
// Registers: launched with 72 a thread; the consumer warpgroups take 96 and the others give
// theirs up to 40.
constexpr int kLaunchRegs = 72, kConsumerRegs = 96, kOtherRegs = 40;
static_assert(kConsumers % 4 == 0 && kOthers % 4 == 0 &&
              kConsumers * kConsumerRegs + kOthers * kOtherRegs <= (kConsumers + kOthers) * kLaunchRegs, "register split");

struct WaveLayout {
  int rb;                        // bytes per row
  int task_ring;                 // task records
  int max_rows;                  // rows of a group's list
  unsigned off_rec, off_mom, off_lists, off_ctab, off_info, off_bar, total;
};

// A batch in flight.
struct WaveInfo {
  int ntask, slot0, t0, flags;       // own rows, ring slot of the first row, its records' place; flags: 1 first
                                     // batch of an item, 2 last, 4 end of work
  int nrows, nstat, octant, l0;      // rows, own and static rows
  int progress, step, upx, upy;      // the column's progress entry, its hyperplane, upwind columns' entries or -1
  int member, list, item, pad;       // place of its row list; member and first velocity as one number
};

__device__ __forceinline__ void cp16(unsigned dst, const void *src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_arrive(unsigned bar) {
  asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ int ld_acquire(const int *p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(int *p, int v) {
  asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ int ld_acquire_sm(unsigned a) {
  int v;
  asm volatile("ld.acquire.cta.shared::cta.s32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void st_release_sm(unsigned a, int v) {
  asm volatile("st.release.cta.shared::cta.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Waits (suspended by the hardware, at most about 20 us) for the phase of `parity`.
__device__ __forceinline__ bool mbar_sleep(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity), "r"(20000u)
      : "memory");
  return ok != 0;
}
// Whether the phase of `parity` is complete, without waiting.
__device__ __forceinline__ bool mbar_test(unsigned bar, unsigned parity) {
  unsigned ok;
  asm volatile(
      "{\n .reg .pred p;\n mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
      : "=r"(ok)
      : "r"(bar), "r"(parity)
      : "memory");
  return ok != 0;
}

// A CTA's barriers and control words.
struct WavePipe {
  // shared addresses: kStages mbarriers each; the batches that the publish warp has followed
  unsigned meta, go, dep, full, done, seen;
  __device__ static unsigned parity(int k) { return (unsigned)(k / kStages) & 1u; }
  __device__ static unsigned at(unsigned bars, int k) { return bars + 8u * (unsigned)(k % kStages); }
  __device__ bool wait_for(unsigned bars, int k) const { return wait(at(bars, k), parity(k)); }
  // the group of batch k (its mbarriers are the first kGroups of `meta`)
  __device__ unsigned meta_at(int k) const { return meta + 8u * (unsigned)(k / kGroup % kGroups); }
  __device__ bool wait_meta(int k) const { return wait(meta_at(k), parity(k)); }
  volatile int *abort;
  int *err;
  // Waits for the phase of `parity`; false when it gave up or the CTA has aborted.
  __device__ bool wait(unsigned bar, unsigned parity) const {
    if (mbar_sleep(bar, parity)) return true;
    const unsigned long long t0 = gtimer();
    while (!mbar_sleep(bar, parity)) {
      if (*abort) return false;
      if (gtimer() - t0 > kWaitNs) {
        *abort = 1;
        atomicExch(err, 1);
        return false;
      }
    }
    return true;
  }
  // Waits until `n` batches are complete. (Batch n - 1 + kStages is not requested yet.)
  __device__ bool wait_done(int n) const { return n <= 0 || wait_for(done, n - 1); }
  // Waits until the publish warp has followed n batches.
  __device__ bool wait_seen(int n) const {
    if (ld_acquire_sm(seen) >= n) return true;
    const unsigned long long t0 = gtimer();
    for (int it = 1;; ++it) {
      if (ld_acquire_sm(seen) >= n) return true;
      if ((it & 31) == 0) {
        if (*abort) return false;
        if (gtimer() - t0 > kWaitNs) {
          *abort = 1;
          atomicExch(err, 1);
          return false;
        }
      }
    }
  }
};

// Waits until *p >= need and returns it; gives up (returns need, *err set) after kWaitNs or
// once *err is set.
__device__ int wait_progress(const int *p, int need, int *err) {
  int v = ld_acquire(p);
  if (v >= need) return v;
  const unsigned long long t0 = gtimer();
  for (int it = 1;; ++it) {
    v = ld_acquire(p);
    if (v >= need) return v;
    if ((it & 63) == 0) {
      if (ld_acquire(err) != 0) return need;
      if (gtimer() - t0 > kWaitNs) {
        atomicExch(err, 1);
        return need;
      }
    }
    __nanosleep(32);
  }
}

// The state of batch item `member`: the launch's own, or one of a batch's.
template <bool BATCH>
__device__ __forceinline__ const DevState &member_state(const DevState &a, const DevState *states, int m) {
  if constexpr (BATCH) return states[m];
  else return a;
}

// Items and batches in order; row lists and task records. Columns have a multiple of kGroup
// batches, whose lists and records lie together; lanes 0 .. kGroup - 1 hold a batch each.
template <int V, bool BATCH>
__device__ void wave_request(const DevState &a0, const DevState *states, const int4 *items, int nitems, int *counter,
                             const WaveLayout &L, unsigned char *smem, const WavePipe &P, WaveInfo *info) {
  const int lane = threadIdx.x & 31;
  const unsigned rec = smem_u32(smem + L.off_rec), lists = smem_u32(smem + L.off_lists);
  int bi = 0, bn = 0, claimed = -1;
  int b0 = 0, octant = 0, step0 = 0, upx = -1, upy = -1, chunk = 0, member = 0, progress = 0;  // the item
  int4 recs = make_int4(0, 0, 0, 0);           // 32 batch records, one per lane
  int done = 0;                                // batches known to be complete
  int tpos = 0, tmod = 0, tstart = 0;          // records placed, modulo their ring; lane i: before group = i (mod 32)
  int k = 0;
  for (;; k += kGroup) {
    int flags = 0;
    if (bi >= bn) {
      if (claimed < 0) {
        if (lane == 0) claimed = atomicAdd(counter, 1);
        claimed = __shfl_sync(0xffffffffu, claimed, 0);
      }
      if (claimed >= nitems) {
        flags = 4;
      } else {
        const int4 it = __ldg(items + claimed);
        claimed = -1;
        const DevState &a = member_state<BATCH>(a0, states, it.x);
        const int4 h0 = __ldg(a.wv.cols + 2 * (size_t)it.y), h1 = __ldg(a.wv.cols + 2 * (size_t)it.y + 1);
        const int nchunk = a.wv.nchunk;
        chunk = it.z;
        member = it.x;
        progress = it.y * nchunk + chunk;
        b0 = h0.x; bn = h0.y; octant = h0.z; step0 = h0.w;
        upx = h1.x < 0 ? -1 : h1.x * nchunk + chunk;
        upy = h1.y < 0 ? -1 : h1.y * nchunk + chunk;
        bi = 0;
        flags = 1;
      }
    }
    const DevState &a = member_state<BATCH>(a0, states, member);
    if (!(flags & 4) && (bi & 31) == 0)
      recs = bi + lane < bn ? __ldg(a.wv.batch + (size_t)b0 + bi + lane) : make_int4(0, 0, 0, 0);
    // each lane its batch of the group; the group's first and last give its lists and records
    const int src = (bi + (lane & (kGroup - 1))) & 31;
    int4 b;
    b.x = __shfl_sync(0xffffffffu, recs.x, src);
    b.y = __shfl_sync(0xffffffffu, recs.y, src);
    b.z = __shfl_sync(0xffffffffu, recs.z, src);
    b.w = __shfl_sync(0xffffffffu, recs.w, src);
    const int nrows = b.z & 0xffff, nt = (int)((unsigned)b.z >> 16);
    const int x0 = __shfl_sync(0xffffffffu, b.x, 0), y0 = __shfl_sync(0xffffffffu, b.y, 0);
    const int gl = __shfl_sync(0xffffffffu, b.x + (nrows + 3) / 4, kGroup - 1) - x0;   // list, in groups of 4 rows
    const int gt = (flags & 4) ? 0 : __shfl_sync(0xffffffffu, b.y + nt, kGroup - 1) - y0;
    // a group's records lie together: the rest of their ring is skipped when it is too short
    if (tmod + gt > L.task_ring) { tpos += L.task_ring - tmod; tmod = 0; }
    // room: stages, the records of the groups that are not complete, and a free row list
    bool ok = true;
    for (;;) {
      const int dg = done / kGroup;
      int need = k + kGroup - kStages;
      if (done >= need && dg * kGroup < k && tpos + gt - __shfl_sync(0xffffffffu, tstart, dg & 31) > L.task_ring)
        need = (dg + 1) * kGroup;
      if (done >= need) break;
      if (!(ok = __all_sync(0xffffffffu, P.wait_done(need)))) break;
      done = need;
    }
    if (ok) ok = __all_sync(0xffffffffu, P.wait_seen(k + kGroup - kStages));
    if (ok && k >= kLists * kGroup && !(flags & 4)) {
      const int old = k - kLists * kGroup + (lane & (kGroup - 1));
      ok = __all_sync(0xffffffffu, P.wait_for(P.full, old));
    }
    if (!ok) break;
    if (lane == (k / kGroup & 31)) tstart = tpos;
    const int list = (k / kGroup % kLists) * L.max_rows;
    if (lane < kGroup) {
      WaveInfo &d = info[(k + lane) % kStages];
      const int f = flags & 4 ? 4 : (lane == 0 ? flags : 0) | (bi + lane == bn - 1 ? 2 : 0);
      *reinterpret_cast<int4 *>(&d.ntask) = make_int4(nt, (int)((unsigned)b.w >> 16), tmod + b.y - y0, f);
      *reinterpret_cast<int4 *>(&d.nrows) = make_int4(nrows, b.w & 0xffff, octant, chunk * V);
      *reinterpret_cast<int4 *>(&d.progress) = make_int4(progress, step0 + bi + lane, upx, upy);
      *reinterpret_cast<int4 *>(&d.member) = make_int4(member, list + 4 * (b.x - x0), member << 16 | chunk, 0);
    }
    __syncwarp();
    if (lane == 0) {
      const unsigned bar = P.meta_at(k);
      if (flags & 4) {
        mbar_arrive(bar);
      } else {
        const unsigned cb = (unsigned)gl * 16u, tb = (unsigned)gt * 16u;
        mbar_expect_arrive(bar, cb + tb);
        if (cb) bulk_g2s(lists + (unsigned)list * 4u, a.wv.rows + (size_t)(unsigned)x0 * 4, cb, bar);
        if (tb) bulk_g2s(rec + (unsigned)tmod * 16u, a.wv.tasks + y0, tb, bar);
      }
    }
    tpos += gt;
    tmod += gt;
    __syncwarp();
    if (flags & 4) { k += kGroup; break; }
    bi += kGroup;
    // the next item is claimed shortly before this one runs out of batches: an item claimed
    // early would be held back by the rest of this column
    if (claimed < 0 && bn - bi <= kGroup) {
      if (lane == 0) claimed = atomicAdd(counter, 1);
      claimed = __shfl_sync(0xffffffffu, claimed, 0);
    }
  }
  // the copies that were requested finish before the warp leaves, aborted or not
  for (int m = max(0, k - kStages); m < k; m += kGroup) {
    const unsigned long long t0 = gtimer();
    while (!mbar_test(P.meta_at(m), P.parity(m)) && gtimer() - t0 < kWaitNs) {
    }
  }
}

// When a batch's rows may enter the ring.
template <bool BATCH>
__device__ void wave_go(const DevState &a0, const DevState *states, const WavePipe &P, const WaveInfo *info) {
  const int lane = threadIdx.x & 31;
  int done = 0;
  int rpos = 0, rmod = 0, rstart = 0;          // ring position, modulo the ring; lane i: the start of batch = i (mod 32)
  int first_k = 0, R = 0;                      // the item's first batch; the ring of its member
  for (int k = 0;; ++k) {
    if (k % kGroup == 0 && !__all_sync(0xffffffffu, P.wait_meta(k))) return;
    const WaveInfo &d = info[k % kStages];
    const int nrows = d.nrows, slot0 = d.slot0, flags = d.flags;
    if (flags & 4) {
      if (lane == 0) mbar_arrive(P.at(P.go, k));
      if (k % kGroup == kGroup - 1) return;
      continue;
    }
    if (flags & 1) {
      first_k = k;
      const int ring = member_state<BATCH>(a0, states, d.member).wv.ring;
      if (BATCH && R != ring) {                // another member's ring: once the previous item is done
        if (!__all_sync(0xffffffffu, P.wait_done(k))) return;
        done = k;
        rpos = rmod = 0;
      }
      R = ring;
      // a column's slots count from the ring's start
      if (rmod) rpos += R - rmod;
    }
    // batches known to be complete: at least the one whose stage batch k has taken (`rstart`
    // then still holds the starts of the batches from done - 2 on)
    done = max(done, k - kStages + 1);
    while (done < k && __all_sync(0xffffffffu, mbar_test(P.at(P.done, done), P.parity(done)))) ++done;
    // room: the batch overwrites nothing that a batch still to be completed reads (a complete
    // batch's rows are read by the two after it, of the same item)
    for (;;) {
      int live = done - 2;
      if (live < first_k && done >= first_k) live = first_k;
      if (live < 0) live = 0;
      if (live >= k || rpos + nrows - __shfl_sync(0xffffffffu, rstart, live & 31) <= R) break;
      if (!__all_sync(0xffffffffu, P.wait_done(done + 1))) return;
      ++done;
    }
    if (lane == 0) mbar_arrive(P.at(P.go, k));
    if (lane == (k & 31)) rstart = rpos;
    rpos += nrows;
    rmod = slot0 - 1 + nrows;
    if (rmod >= R) rmod -= R;
  }
}

// When the rows of the upwind columns may be read: the tasks of hyperplane `step` read
// hyperplanes up to step - 1, which are hyperplanes up to A + step - 1 of the column upwind in
// x (B in y). Lane 0 follows the column upwind in x, lane 1 the one in y.
template <bool BATCH>
__device__ void wave_dep(const DevState &a0, const DevState *states, const WavePipe &P, const WaveInfo *info) {
  const int lane = threadIdx.x & 31;
  int know = 0, ahead = 0;
  const int *up = nullptr;
  for (int k = 0;; ++k) {
    if (k % kGroup == 0 && !__all_sync(0xffffffffu, P.wait_meta(k))) return;
    const WaveInfo &d = info[k % kStages];
    const int flags = d.flags, step = d.step;
    const bool any = d.nstat < d.nrows;
    if (flags & 1) {
      const WaveView &w = member_state<BATCH>(a0, states, d.member).wv;
      const int e = lane == 0 ? d.upx : lane == 1 ? d.upy : -1;
      up = e < 0 ? nullptr : w.progress + e;
      ahead = lane ? w.B : w.A;
      know = 0;
    }
    if (any && up && know < step + ahead) know = wait_progress(up, step + ahead, P.err);
    __syncwarp();
    if (lane == 0) { mbar_arrive(P.at(P.dep, k)); mbar_arrive(P.at(P.full, k)); }
    if ((flags & 4) && k % kGroup == kGroup - 1) return;
  }
}

// The rows and moments of batches team, team + kTeams, ...: warp `cw` of a team.
template <typename T, int V, bool BATCH>
__device__ void wave_copy(const DevState &a0, const DevState *states, const WaveLayout &L, unsigned char *smem,
                          const WavePipe &P, const WaveInfo *info, int team, int cw) {
  constexpr int EPP = 16 / (int)sizeof(T);     // velocities per 16-byte piece
  constexpr int PIECES = V / EPP;              // pieces per row (a power of two, at most 32)
  constexpr int RPI = 32 / PIECES;             // rows per warp instruction
  constexpr int STEP = 2 * RPI * kTeam;      // a lane group takes two neighbouring rows of every STEP
  constexpr unsigned RB = V * sizeof(T);
  const int lane = threadIdx.x & 31, sub = lane % PIECES, first = 2 * (cw * RPI + lane / PIECES);
  const unsigned dst0 = smem_u32(smem) + 16u * sub, mom0 = smem_u32(smem + L.off_mom) + 16u * (lane & 1);
  const int *lists = reinterpret_cast<const int *>(smem + L.off_lists);
  int item = -1;                               // of the item:
  const char *base = nullptr, *moments = nullptr;
  unsigned stride = 0;
  int R = 0;
  bool lv = true;
  for (int k = team;; k += kTeams) {
    if (!P.wait_meta(k)) break;
    const WaveInfo &d = info[k % kStages];
    const int4 d0 = *reinterpret_cast<const int4 *>(&d.ntask);
    const int4 d1 = *reinterpret_cast<const int4 *>(&d.nrows);
    const int4 d3 = *reinterpret_cast<const int4 *>(&d.member);
    if (d0.w & 4) {
      cp_async_arrive(P.at(P.full, k));
      break;
    }
    if (d3.z != item) {
      item = d3.z;
      const DevState &a = member_state<BATCH>(a0, states, d3.x);
      stride = (unsigned)a.Nc8 * (unsigned)sizeof(T);
      base = reinterpret_cast<const char *>(state_h<T>(a)) + (size_t)d1.w * sizeof(T) + 16 * sub;
      moments = reinterpret_cast<const char *>(a.mom) + 16 * (lane & 1);
      lv = d1.w + sub * EPP < a.Nc8;           // the last chunk may be short
      R = a.wv.ring;
    }
    const int *rows = lists + d3.y;
    const unsigned dst = dst0 + (unsigned)d0.y * RB;
    const int wrap = R + 1 - d0.y;             // rows before the ring's end
    auto copy_rows = [&](int r0, int r1) {     // [r0, r1), r0 even
      for (int q = r0 + first; q < r1; q += STEP) {
        const int2 c = *reinterpret_cast<const int2 *>(rows + q);
        const unsigned at0 = dst + (unsigned)(q - (q >= wrap ? R : 0)) * RB;
        const unsigned at1 = dst + (unsigned)(q + 1 - (q + 1 >= wrap ? R : 0)) * RB;
        if (lv) {
          cp16(at0, base + (unsigned long long)(unsigned)c.x * stride);
          if (q + 1 < r1) cp16(at1, base + (unsigned long long)(unsigned)c.y * stride);
        }
      }
    };
    if (!P.wait_for(P.go, k)) break;
    // own and static rows; an odd last one goes with the dependent rows
    const int nrows = d1.x, nstat = d1.y < nrows ? d1.y & ~1 : nrows;
    copy_rows(0, nstat);
    // the moments of the tasks' nodes, by ring slot
    for (int t = cw * 16 + (lane >> 1); t < d0.x; t += 16 * kTeam)
      cp16(mom0 + 32u * (unsigned)(d0.y + t - (t >= wrap ? R : 0)), moments + (size_t)((unsigned)rows[t] >> 3) * 32);
    if (nstat < nrows) {
      if (!P.wait_for(P.dep, k)) break;
      copy_rows(nstat, nrows);
    }
    cp_async_arrive(P.at(P.full, k));
  }
  asm volatile("cp.async.wait_all;" ::: "memory");
}

// Follows the completed batches: the CTA's count, then the columns' progress.
template <bool BATCH>
__device__ void wave_publish(const DevState &a0, const DevState *states, const WavePipe &P, const WaveInfo *info) {
  for (int k = 0;;) {
    if (!P.wait_for(P.done, k)) return;
    // read before `seen` frees the stage
    const WaveInfo &d = info[k % kStages];
    const int flags = d.flags, progress = d.progress, step = d.step, member = d.member;
    if (flags & 4) return;
    ++k;
    st_release_sm(P.seen, k);
    // a batch that the next one of its column has already followed needs no store of its own
    if (!(flags & 2) && mbar_test(P.at(P.done, k), P.parity(k))) continue;
    const DevState &a = member_state<BATCH>(a0, states, member);
    st_release(a.wv.progress + progress, (flags & 2) ? kDone : step + 1);
  }
}

// The 7 per-velocity constants a consumer lane keeps for its velocities: the signed velocity
// components, the weight and the products c / ds. The second-order coefficients are those
// products times 2 and -1/2, made by exponent arithmetic (exact: the reference's products
// c * (2/ds) and c * (-0.5/ds) are the same powers of two apart).
template <typename T, int VPL>
struct WaveConsts {
  T c[3][VPL], w[VPL], k[3][VPL];
};
__device__ __forceinline__ double twice(double x, int one) { return __hiloint2double(__double2hiint(x) + (one << 20), __double2loint(x)); }
__device__ __forceinline__ double minus_half(double x) { return __hiloint2double(__double2hiint(x) + 0x7FF00000, __double2loint(x)); }
__device__ __forceinline__ float twice(float x, int one) { return __int_as_float(__float_as_int(x) + (one << 23)); }
__device__ __forceinline__ float minus_half(float x) { return __int_as_float(__float_as_int(x) + 0x7F800000); }

// A lane's VPL velocities of a row: NP pieces of up to 16 bytes, `span` bytes apart (the task's
// lanes read neighbouring pieces, so a row's reads meet no bank conflicts).
template <typename T, int VPL>
struct Lane {
  static constexpr int kPiece = VPL * sizeof(T) < 16 ? VPL : 16 / (int)sizeof(T);  // velocities per piece
  static constexpr int NP = VPL / kPiece;
};
template <typename T, int VPL>
__device__ __forceinline__ void ld_row(unsigned addr, unsigned span, T (&v)[VPL]) {
  constexpr int E = Lane<T, VPL>::kPiece;
#pragma unroll
  for (int p = 0; p < Lane<T, VPL>::NP; ++p) {
    const unsigned a = addr + p * span;
    if constexpr (sizeof(T) == 8) asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v[p * E]), "=d"(v[p * E + 1]) : "r"(a) : "memory");
    else if constexpr (E == 4)
      asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[p * E]), "=f"(v[p * E + 1]), "=f"(v[p * E + 2]), "=f"(v[p * E + 3]) : "r"(a) : "memory");
    else asm volatile("ld.shared.v2.f32 {%0, %1}, [%2];" : "=f"(v[p * E]), "=f"(v[p * E + 1]) : "r"(a) : "memory");
  }
}
// The same from the class table, which other warps may be writing (see wave_consume).
template <typename T, int VPL>
__device__ __forceinline__ void ld_table(unsigned addr, unsigned span, T (&v)[VPL]) {
  constexpr int E = Lane<T, VPL>::kPiece;
#pragma unroll
  for (int p = 0; p < Lane<T, VPL>::NP; ++p) {
    const unsigned a = addr + p * span;
    if constexpr (sizeof(T) == 8) asm volatile("ld.relaxed.cta.shared::cta.v2.f64 {%0, %1}, [%2];" : "=d"(v[p * E]), "=d"(v[p * E + 1]) : "r"(a) : "memory");
    else if constexpr (E == 4)
      asm volatile("ld.relaxed.cta.shared::cta.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v[p * E]), "=f"(v[p * E + 1]), "=f"(v[p * E + 2]), "=f"(v[p * E + 3]) : "r"(a) : "memory");
    else asm volatile("ld.relaxed.cta.shared::cta.v2.f32 {%0, %1}, [%2];" : "=f"(v[p * E]), "=f"(v[p * E + 1]) : "r"(a) : "memory");
  }
}
__device__ __forceinline__ void st_table(unsigned addr, double v) { asm volatile("st.relaxed.cta.shared::cta.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory"); }
__device__ __forceinline__ void st_table(unsigned addr, float v) { asm volatile("st.relaxed.cta.shared::cta.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
template <typename T, int VPL>
__device__ __forceinline__ void st_row(unsigned addr, unsigned span, const T (&v)[VPL]) {
  constexpr int E = Lane<T, VPL>::kPiece;
#pragma unroll
  for (int p = 0; p < Lane<T, VPL>::NP; ++p) {
    const unsigned a = addr + p * span;
    if constexpr (sizeof(T) == 8) asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v[p * E]), "d"(v[p * E + 1]) : "memory");
    else if constexpr (E == 4)
      asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(a), "f"(v[p * E]), "f"(v[p * E + 1]), "f"(v[p * E + 2]), "f"(v[p * E + 3]) : "memory");
    else asm volatile("st.shared.v2.f32 [%0], {%1, %2};" ::"r"(a), "f"(v[p * E]), "f"(v[p * E + 1]) : "memory");
  }
}

// One task: solver.F90:205-214 in the reference's order. FP64 through mul / add (no
// contraction) and the corrected reciprocal (sweep_core.cuh), FP32 as base32 / update32. In
// two parts: what the batch before has no say in (the equilibrium part, the far upwind rows,
// two hyperplanes back, and the divisor), and the rest, which needs the near upwind rows.
template <typename T, int VPL>
struct WaveTask {
  T num[VPL], x2[VPL], y2[VPL], z2[VPL], rc[VPL], den[sizeof(T) == 8 ? VPL : 1];
  unsigned x1, y1, z1, own;        // shared addresses
  int flags, node;
};
template <typename T, int V, int VPL>
__device__ __forceinline__ void wave_begin(const WaveConsts<T, VPL> &K, double mu, unsigned lane_ring, unsigned ctab,
                                           unsigned own, const int4 rec, const double2 m01, const double2 m23,
                                           WaveTask<T, VPL> &w) {
  constexpr unsigned RB = V * sizeof(T), SPAN = RB / Lane<T, VPL>::NP;
  T f[VPL];
  ld_row<T, VPL>(own, SPAN, f);
  ld_row<T, VPL>(lane_ring + ((unsigned)rec.y >> 16) * RB, SPAN, w.x2);
  ld_row<T, VPL>(lane_ring + ((unsigned)rec.z >> 16) * RB, SPAN, w.y2);
  ld_row<T, VPL>(lane_ring + ((unsigned)rec.w >> 16) * RB, SPAN, w.z2);
  const int fl = (unsigned)rec.x >> 27;
  ld_table<T, VPL>(ctab + (unsigned)(fl & 7) * RB, SPAN, w.rc);
  w.flags = fl;
  w.node = rec.x & ((1 << 27) - 1);
  w.own = own;
  w.x1 = lane_ring + (rec.y & 0xffff) * RB;
  w.y1 = lane_ring + (rec.z & 0xffff) * RB;
  w.z1 = lane_ring + (rec.w & 0xffff) * RB;
  if constexpr (sizeof(T) == 8) {
    ld_table<T, VPL>(ctab + (unsigned)(8 + (fl & 7)) * RB, SPAN, w.den);
    const double rho = m01.x, ux = m01.y, uy = m23.x, uz = m23.y;
#pragma unroll
    for (int q = 0; q < VPL; ++q) {
      const double ex = dmul(K.c[0][q], ux), ey = dmul(K.c[1][q], uy), ez = dmul(K.c[2][q], uz);
      const double feq = dmul(K.w[q], dadd(rho, dadd(dadd(ex, ey), ez)));
      w.num[q] = dmul(mu, dsub(feq, dmul(0.5, f[q])));
      // the far point of a first-order axis is the zero row, whose term (-0) leaves the sum
      // unchanged
      w.x2[q] = dmul(minus_half(K.k[0][q]), w.x2[q]);
      w.y2[q] = dmul(minus_half(K.k[1][q]), w.y2[q]);
      w.z2[q] = dmul(minus_half(K.k[2][q]), w.z2[q]);
    }
  } else {
    const float rho = (float)m01.x, ux = (float)m01.y, uy = (float)m23.x, uz = (float)m23.y;
    const float mu32 = (float)mu;
#pragma unroll
    for (int q = 0; q < VPL; ++q) {
      float cu = __fmul_rn(K.c[0][q], ux);
      cu = __fmaf_rn(K.c[1][q], uy, cu);
      cu = __fmaf_rn(K.c[2][q], uz, cu);
      const float feq = __fmul_rn(K.w[q], __fadd_rn(rho, cu));
      w.num[q] = __fmul_rn(mu32, __fmaf_rn(-0.5f, f[q], feq));
    }
  }
}
template <typename T, int V, int VPL>
__device__ __forceinline__ void wave_end(const WaveConsts<T, VPL> &K, const WaveTask<T, VPL> &w, T (&out)[VPL]) {
  constexpr unsigned SPAN = V * sizeof(T) / Lane<T, VPL>::NP;
  T x1[VPL], y1[VPL], z1[VPL];
  ld_row<T, VPL>(w.x1, SPAN, x1);
  ld_row<T, VPL>(w.y1, SPAN, y1);
  ld_row<T, VPL>(w.z1, SPAN, z1);
  // second order along an axis: the first coefficient is 2 c / ds instead of c / ds
  const int ox = (w.flags & 1) ^ 1, oy = ((w.flags >> 1) & 1) ^ 1, oz = ((w.flags >> 2) & 1) ^ 1;
#pragma unroll
  for (int q = 0; q < VPL; ++q) {
    T num = w.num[q];
    if constexpr (sizeof(T) == 8) {
      num = dadd(num, dmul(twice(K.k[0][q], ox), x1[q]));
      num = dadd(num, w.x2[q]);
      num = dadd(num, dmul(twice(K.k[1][q], oy), y1[q]));
      num = dadd(num, w.y2[q]);
      num = dadd(num, dmul(twice(K.k[2][q], oz), z1[q]));
      num = dadd(num, w.z2[q]);
      out[q] = markstein_div(num, w.den[q], w.rc[q]);
    } else {
      num = __fmaf_rn(twice(K.k[0][q], ox), x1[q], num);
      num = __fmaf_rn(minus_half(K.k[0][q]), w.x2[q], num);
      num = __fmaf_rn(twice(K.k[1][q], oy), y1[q], num);
      num = __fmaf_rn(minus_half(K.k[1][q]), w.y2[q], num);
      num = __fmaf_rn(twice(K.k[2][q], oz), z1[q], num);
      num = __fmaf_rn(minus_half(K.k[2][q]), w.z2[q], num);
      out[q] = __fmul_rn(num, w.rc[q]);
    }
  }
}

template <typename T, int V, int VPL, bool BATCH>
__device__ void wave_consume(const DevState &a0, const DevState *states, const WaveLayout &L, unsigned char *smem,
                             const WavePipe &P, const WaveInfo *info) {
  constexpr int LPT = V / VPL, THREADS = kConsumers * 32, GROUPS = THREADS / LPT;
  constexpr int E = Lane<T, VPL>::kPiece, NP = Lane<T, VPL>::NP;
  constexpr unsigned RB = V * sizeof(T), SPAN = RB / NP;
  static_assert(LPT * VPL == V && 32 % LPT == 0, "whole task groups per warp");
  const int ct = threadIdx.x, lane = ct & 31;
  const int grp = ct / LPT, sub = ct % LPT;
  const unsigned lane_bytes = (unsigned)(sub * E * sizeof(T));
  const unsigned lane_ring = smem_u32(smem) + lane_bytes;
  const unsigned ctab = smem_u32(smem + L.off_ctab) + lane_bytes;
  const int4 *rec = reinterpret_cast<const int4 *>(smem + L.off_rec);
  const double2 *mom = reinterpret_cast<const double2 *>(smem + L.off_mom);
  WaveConsts<T, VPL> K{};
  double mu = 0.0;
  int table_of = -1;               // member and chunk of the class table
  T *h = nullptr;                  // the lane's velocities of the octant of node 0
  unsigned stride = 0;             // values per node
  int R = 0;
  bool lv[NP] = {};                // the last chunk may be short
  for (int k = 0;; ++k) {
    if (!P.wait_for(P.full, k)) return;        // the batch's rows have landed
    const WaveInfo &d = info[k % kStages];
    const int4 d0 = *reinterpret_cast<const int4 *>(&d.ntask);
    const int nt = d0.x, slot0 = d0.y, t0 = d0.z, flags = d0.w;
    if (flags & 4) {
      if (lane == 0) mbar_arrive(P.at(P.done, k));
      return;
    }
    if (flags & 1) {
      const int m = d.member, l0 = d.l0, oct = d.octant;
      const DevState &a = member_state<BATCH>(a0, states, m);
      mu = a.mu;
      stride = 8u * (unsigned)a.Nc8;
      R = a.wv.ring;
      h = const_cast<T *>(state_h<T>(a)) + (size_t)oct * a.Nc8 + l0 + sub * E;
#pragma unroll
      for (int p = 0; p < NP; ++p) lv[p] = l0 + (sub + p * LPT) * E < a.Nc8;
      const bool neg[3] = {neg_x(oct), neg_y(oct), neg_z(oct)};
#pragma unroll
      for (int q = 0; q < VPL; ++q) {
        const int l = min(l0 + (sub + q / E * LPT) * E + q % E, a.Nc8 - 1);
        const T *vt;
        if constexpr (sizeof(T) == 8) vt = a.vtab + (size_t)l * kVtab;
        else vt = a.vtab32 + (size_t)l * kVtab;
#pragma unroll
        for (int x = 0; x < 3; ++x) {
          const T c = __ldg(vt + x);
          K.c[x][q] = neg[x] ? -c : c;
          K.k[x][q] = __ldg(vt + 5 + 3 * x);
        }
        K.w[q] = __ldg(vt + 3);
      }
      const int key = m * 4096 + l0 / V;
      if (key != table_of) {
        // the class table of the chunk: reciprocals, and for FP64 denominators, once every
        // warp has finished the previous batch (none reads the old one). Each warp writes the
        // whole table, the same values into the same places (relaxed accesses), and reads it
        // after its own writes: no warp waits for another, where filling it together would take
        // a barrier that a warp which has left never reaches. Sweep with a barrier of all
        // consumers / this: 96^3 pack, 64 velocities, FP32 0.321 / 0.315, FP64 0.420 / 0.411 ms;
        // 48^3 pack, 512 velocities, FP64 0.263 / 0.260, FP32 0.233 / 0.232.
        table_of = key;
        if (k > 0 && !P.wait_for(P.done, k - 1)) return;
        const unsigned tab = smem_u32(smem + L.off_ctab);
        constexpr int NT = sizeof(T) == 8 ? 16 : 8;
        for (int i = lane; i < NT * V; i += 32) {
          const int cls = i / V, l = min(l0 + i % V, a.Nc8 - 1);
          if constexpr (sizeof(T) == 8) st_table(tab + 8u * i, __ldg(a.vtab + (size_t)l * kVtab + (cls < 8 ? 21 + cls : 5 + cls)));
          else st_table(tab + 4u * i, __ldg(a.vtab32 + (size_t)l * kVtab + 21 + cls));
        }
        __syncwarp();
      }
    }
    WaveTask<T, VPL> w;
    auto begin = [&](int t) {
      int slot = slot0 + t;
      if (slot > R) slot -= R;
      wave_begin<T, V, VPL>(K, mu, lane_ring, ctab, lane_ring + (unsigned)slot * RB, rec[t0 + t], mom[2 * slot],
                            mom[2 * slot + 1], w);
    };
    auto end = [&]() {
      T out[VPL];
      wave_end<T, V, VPL>(K, w, out);
      st_row<T, VPL>(w.own, SPAN, out);
      T *hp = h + (size_t)((unsigned long long)(unsigned)w.node * stride);
#pragma unroll
      for (int p = 0; p < NP; ++p) {
        if (!lv[p]) continue;
        if constexpr (sizeof(T) == 8) *reinterpret_cast<double2 *>(hp + p * LPT * E) = make_double2(out[p * E], out[p * E + 1]);
        else if constexpr (E == 4) *reinterpret_cast<float4 *>(hp + p * LPT * E) = make_float4(out[p * E], out[p * E + 1], out[p * E + 2], out[p * E + 3]);
        else *reinterpret_cast<float2 *>(hp + p * LPT * E) = make_float2(out[p * E], out[p * E + 1]);
      }
    };
    // odd batches start with the other half of the warps: a half that the previous batch had no
    // tasks for does the first part of this one meanwhile (sweep of the 128^3 pack FP64 2.91 -> 2.79,
    // FP32 1.48 -> 1.45 ms; 256^3 field 6.82 -> 6.69)
    const int first = grp ^ ((k & 1) * (GROUPS / 2));
    if (first < nt) begin(first);
    // every warp has finished the previous batch: its results are in the ring
    if (k > 0 && !P.wait_for(P.done, k - 1)) return;
    for (int t = first; t < nt;) {
      end();
      t += GROUPS;
      if (t < nt) begin(t);
    }
    __syncwarp();
    if (lane == 0) mbar_arrive(P.at(P.done, k));
  }
}

template <typename T, int V, int VPL, bool BATCH>
__global__ void __launch_bounds__(kThreads, 1)
k_wave_sweep(const DevState a, const DevState *states, const int4 *items, int nitems, int *counter, int *err,
             const WaveLayout L) {
  extern __shared__ __align__(128) unsigned char smem[];
  const int warp = threadIdx.x >> 5;
  WaveInfo *info = reinterpret_cast<WaveInfo *>(smem + L.off_info);
  WavePipe P;
  const unsigned bars = smem_u32(smem + L.off_bar);
  P.meta = bars;
  P.go = bars + 8u * kStages;
  P.dep = bars + 16u * kStages;
  P.full = bars + 24u * kStages;
  P.done = bars + 32u * kStages;
  P.seen = bars + 40u * kStages;
  P.abort = reinterpret_cast<volatile int *>(smem + L.off_bar + 40 * kStages + 4);
  P.err = err;
  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages; ++s) {
      mbar_init(P.meta + 8u * s, 1);
      mbar_init(P.go + 8u * s, 1);
      mbar_init(P.dep + 8u * s, 1);
      mbar_init(P.full + 8u * s, kTeam * 32 + 1);  // the copy team's lanes, and the dep warp
      mbar_init(P.done + 8u * s, kConsumers);
    }
    *reinterpret_cast<int2 *>(smem + L.off_bar + 40 * kStages) = make_int2(0, 0);  // seen, abort
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (threadIdx.x < V * (int)sizeof(T) / 16) reinterpret_cast<int4 *>(smem)[threadIdx.x] = make_int4(0, 0, 0, 0);
  __syncthreads();
  if (warp < kConsumers) {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(kConsumerRegs));
    wave_consume<T, V, VPL, BATCH>(a, states, L, smem, P, info);
    return;
  }
  asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(kOtherRegs));
  const int w = warp - kConsumers - kTeam * kTeams;
  if (w < 0) wave_copy<T, V, BATCH>(a, states, L, smem, P, info, (warp - kConsumers) / kTeam, (warp - kConsumers) % kTeam);
  else if (w == 0) wave_request<V, BATCH>(a, states, items, nitems, counter, L, smem, P, info);
  else if (w == 1) wave_go<BATCH>(a, states, P, info);
  else if (w == 2) wave_dep<BATCH>(a, states, P, info);
  else if ((threadIdx.x & 31) == 0) wave_publish<BATCH>(a, states, P, info);
}

constexpr unsigned kSmemCap = 227u * 1024u;

WaveLayout wave_layout(int rb, int ring, int task_ring, int max_rows, bool fp32) {
  WaveLayout L{};
  auto up16 = [](unsigned x) { return (x + 15u) / 16u * 16u; };
  L.rb = rb;
  L.task_ring = task_ring;
  L.max_rows = max_rows;
  unsigned off = (unsigned)(ring + 1) * (unsigned)rb;
  L.off_rec = off; off += (unsigned)task_ring * 16u;
  L.off_mom = off; off += (unsigned)(ring + 1) * 32u;
  L.off_lists = off; off += (unsigned)kLists * (unsigned)max_rows * 4u;
  L.off_ctab = off; off += (unsigned)(fp32 ? 8 : 16) * (unsigned)rb;
  L.off_info = off; off += (unsigned)sizeof(WaveInfo) * kStages;
  off = up16(off);
  L.off_bar = off; off += 40u * kStages + 16u;
  L.total = up16(off);
  return L;
}

template <typename T, int V, int VPL, bool BATCH>
void launch_wave_v(const DevState &s, const DevState *states, const int4 *items, int nitems, const WaveRings &r,
                   int *counter, int *err, cudaStream_t st) {
  const WaveLayout L = wave_layout(V * (int)sizeof(T), r.ring, r.task_ring, r.max_rows, sizeof(T) == 4);
  const void *fn = reinterpret_cast<const void *>(k_wave_sweep<T, V, VPL, BATCH>);
  once_per_device(fn, [](int) {
    cudaFuncSetAttribute(reinterpret_cast<const void *>(k_wave_sweep<T, V, VPL, BATCH>),
                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemCap);
  });
  const int threads = kThreads;
  long grid = resident_blocks(fn, threads, L.total);
  if (grid > nitems) grid = nitems;
  if (grid < 1) return;
  k_wave_sweep<T, V, VPL, BATCH><<<(unsigned)grid, threads, L.total, st>>>(s, states, items, nitems, counter, err, L);
}

template <bool BATCH>
void launch_wave_any(const DevState &s, const DevState *states, const int4 *items, int nitems, bool fp32, int V,
                     const WaveRings &r, int *counter, int *err, cudaStream_t st) {
  if (nitems <= 0) return;
  if (fp32) {
    if (V == 64) launch_wave_v<float, 64, 4, BATCH>(s, states, items, nitems, r, counter, err, st);
    else launch_wave_v<float, 8, 2, BATCH>(s, states, items, nitems, r, counter, err, st);
  } else {
    if (V == 32) launch_wave_v<double, 32, 2, BATCH>(s, states, items, nitems, r, counter, err, st);
    else launch_wave_v<double, 8, 2, BATCH>(s, states, items, nitems, r, counter, err, st);
  }
}

}  // namespace

int wave_velocities(int Nc8, bool fp32) { return Nc8 < 32 ? 8 : fp32 ? 64 : 32; }

int wave_max_ring(int Nc8, bool fp32, int task_ring, int max_rows) {
  const int rb = wave_velocities(Nc8, fp32) * (fp32 ? 4 : 8);
  const unsigned fixed = wave_layout(rb, 0, task_ring, max_rows, fp32).total;
  return fixed >= kSmemCap ? 0 : (int)((kSmemCap - fixed) / (unsigned)(rb + 32));  // a row and its moments
}

void launch_wave_sweep(const DevState &s, bool fp32, cudaStream_t st) {
  const WaveView &w = s.wv;
  cudaMemsetAsync(w.counter, 0, ((size_t)(w.ncol + 1) * w.nchunk + 4) * sizeof(int), st);
  launch_wave_any<false>(s, nullptr, w.items, w.ncol * w.nchunk, fp32, wave_velocities(s.Nc8, fp32),
                         {w.ring, w.task_ring, w.max_rows}, w.counter, w.err, st);
}

void launch_wave_sweep_batch(const DevState *states, const int4 *items, int nitems, bool fp32, int V, const WaveRings &r,
                             int *counter, int *err, cudaStream_t st) {
  launch_wave_any<true>(DevState{}, states, items, nitems, fp32, V, r, counter, err, st);
}

}  // namespace piks
