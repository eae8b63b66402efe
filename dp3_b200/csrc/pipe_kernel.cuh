#pragma once

#include <type_traits>

#include "pass_device.cuh"

namespace {

// ---------------------------------------------------------------------------
// pipe_kernel: the Blackwell streaming path. Per CTA one producer thread
// moves the (time, channel) rows of each tile from HBM into a ring of
// shared-memory stages, one 1-D bulk copy per row (cp.async.bulk, completion
// on an mbarrier, no multicast; the tile-packed slab layout makes a row of a
// tile, data and every direction, contiguous). The consumer warps compute the
// residual and the per-direction P/Q sums from shared memory, 1, 2, 4 or 8
// lanes per run, and stage a tile's sums in shared memory; then a thread per
// (antenna of the tile, group of directions) gathers that antenna's runs, in
// the order of the tile's entry list, and updates the CTA's accumulators. Two
// barriers per staging round, no shared-memory float atomics.
//
// One launch runs several passes, up to a solve's stop. The finalisation is
// part of it: after a grid-wide arrival count, every CTA finalises a share of
// the (channel block, antenna, sub-solution) items (merge of the partial slots,
// FP64 update, step, norm, gain tables, non-finite detection for the lazy
// MakeSolutionsFinite); after a second one, the last CTA of the grid runs the
// iteration control of every interval still going. Meanwhile the ring fills
// with the next pass's rows, and the pass itself begins where its start cannot
// depend on the verdict; it is given up before its finalisation when the solve
// has stopped. Every wait is bounded by a device timer (4 s); when one runs out,
// an error flag that the host reports as DDSOLVE_E_TIMEOUT ends the launch.
// ---------------------------------------------------------------------------
// Consumer warps of a CTA, beside one producer warp: kWarps (168 registers a
// thread), or kWideWarps (255) for 13 directions and more (FindPipeKernel).
constexpr int kWarps = 11, kWideWarps = 7;
// Directions per lane at most (2 and 4 correlations): gains, sums and the
// model row of that many fit a thread's 168 registers; with kWideWarps, gains
// and sums fit 255.
constexpr uint32_t kPipeDirs2 = 5, kPipeDirs4 = 3, kPipeDirsWide = 12;
constexpr int kPipeMaxStages = 8;
constexpr uint64_t kWaitNs = 4000000000ull;  // limit of a device wait

// Device counters of pipe_kernel, each polled word on a cache line of its
// own. The error flag (a bounded wait ran out). Arrivals of CTAs whose partial
// slots are written, and (64 bits) of CTAs that have finalised the pass, with
// the arrivals that saw non-finite solutions in the high half: both count on
// through the passes and launches, a multiple of the grid between launches.
// The number of passes whose control step is done and, beside it, its verdict.
constexpr uint32_t kCntError = 1, kCntArrive = 32, kCntEpoch = 64, kCntVerdict = 65,
                   kCntFinal = 96;
constexpr uint32_t kCounterWords = 128;
constexpr size_t kCounterBytes = kCounterWords * 4;
constexpr uint32_t kVerdictStop = 1u;  // the solve ends with this pass
constexpr uint32_t kVerdictNear = 2u;  // it may end with the next one
// Passes per launch at most, and the visibilities that its passes read (1.5 ms):
// a launch holds every SM, and another context's kernels get the GPU between
// two. 62 stations, 10 directions, 50 passes of 637 MB: a launch more adds 16 us
// to a solve of 5.36 ms; with the next interval's upload and predict on a second
// context an interval takes 8.7 to 9.5 ms with one launch a solve, 7.9 to 8.1
// with 9 GB, 7.7 with 6 or 4 GB. At least ten passes, so that the
// launches cost no more than half a percent of a large array's solve.
constexpr uint32_t kItersPerLaunch = 64, kItersAtLeast = 10;
constexpr double kLaunchBytes = 9e9;

// The partial slots of one (channel block, sub-solution) in the finalisation:
// a range of visits, or a list in fin_visits; its direction; and its gain-table
// entry (table * 256 + direction) when it has just one, else kManyEntries.
struct FinList {
  uint32_t first;  // first visit, or first index in fin_visits
  uint32_t count;  // | kFinRange
  uint32_t dir, entry;
};
constexpr uint32_t kFinRange = 0x80000000u, kManyEntries = 0xFFFFFFFFu;

struct PipeParams {
  const SlabDesc* slabs;
  const Frag* frags;
  const uint32_t* cta_frag_off;
  double2* solutions;
  float* partials;
  float2* tables;         // gain tables [n_tables][table_f2]
  uint32_t table_f2;      // float2 per table (n_ant * gain_stride, even)
  const uint32_t* tab_off;  // finalisation: (cb, s) -> [tab_off, tab_off+1)
  const uint32_t* tab_ent;  //   entries table * 256 + direction
  uint32_t n_ant, n_dir, n_sub, n_cb;
  uint32_t acc_stride;    // floats per antenna in the accumulator table (PipeAccStride)
  uint32_t gain_stride;   // float2 per antenna in a gain table (PipeGainStride)
  uint32_t stages;
  uint32_t acc_floats;    // n_ant * acc_stride = one partial slot
  const uint32_t* metas;  // TileMeta blocks
  uint32_t meta_words;    // words of a TileMeta buffer in shared memory
  uint32_t n_gbuf;        // gain table buffers in shared memory (1 or 2)
  const float* powers;    // model powers per tile [tile][dir][runs of a tile][corr],
                          // or null: accumulated in the row loop
  uint32_t power_floats;  // floats per tile in `powers`
  // shared-memory layout (byte offsets)
  uint32_t off_acc, off_gtab, off_stg, off_q, off_meta, off_stages;
  uint32_t hold;  // no staging area (PipeLayout::hold)
  const FinList* fin_lists;    // [n_cb * n_sub]
  const uint32_t* fin_visits;
  uint32_t* cb_flag;     // channel block holds non-finite solutions
  double* cb_avg;        // replacement value for them (MakeSolutionsFinite)
  uint32_t* cb_newflag;  // set during the finalisation that produced them
  double* block_sum;     // per-CTA norm partials
  uint32_t* block_cnt;
  uint32_t* counters;    // kCounterWords words, see there
  double2* next_out;
  // Passes of this launch: a solve's iterations until it stops, or (host
  // mode) a chain of next-solutions passes, pass k + 1 starting from the
  // output of pass k, which goes to next_out + k * out_stride.
  uint32_t n_iters;
  size_t out_stride;
  volatile uint32_t* host_stopped;  // pinned host memory: set when a solve ends, or null
  int32_t host_mode;
  int32_t fin_mode;      // FinFused / FinStepOnly / FinAssignOnly
  const DevSettings* settings;
  LoopState* state;
  double* step_magnitudes;
  cudaGraphConditionalHandle handle;
  int32_t use_handle;
  // Independent intervals (batched solve): interval g owns the channel blocks
  // with cb_group[cb] = g, its loop state state[g] and step magnitudes
  // step_magnitudes[g * mags_stride]. One interval: n_groups = 1, and a norm
  // partial per CTA.
  uint32_t n_groups;
  const uint32_t* cb_group;
  uint32_t mags_stride;
  // Several intervals: their finalisation items in runs of at most 32 of one
  // interval, a warp's round each: first item, count << 24 | interval. The
  // norm partials are per chunk then, interval g's at [group_chunk[g],
  // group_chunk[g + 1]).
  uint32_t n_chunks;
  const uint2* chunks;
  const uint32_t* group_chunk;
  // The limit of every device wait, and arrivals that the grid barrier expects
  // beyond those of its CTAs (none but in ddsolve_check_wait_limit).
  uint64_t wait_ns;
  uint32_t arrive_extra;
};

// The head of pipe_kernel's shared memory.
struct PipeShared {
  uint64_t full[kPipeMaxStages], empty[kPipeMaxStages];  // ring
  uint64_t gfull[2], gfree[2];  // gain table buffer loaded / released
  uint64_t mfree[2];            // antenna buffer released
  // Thread 0 polls the grid's counters for its CTA and passes the news on to
  // the consumers: every partial slot of the pass is written; every CTA has
  // finalised it (in the CTA of the control step only); the pass is finished
  // (with `stop`: so is the launch). One phase per pass each. The producer,
  // which no barrier keeps within a phase of the consumers, reads the number
  // of finished passes instead.
  uint64_t flushed, finalised, ready;
  double sum[16];  // the warps' norm partials
  uint32_t cnt[32];
  uint32_t flag[2];
  uint32_t skip;  // the launch does nothing
  volatile uint32_t stop, passes;
  volatile int err;
  // thread 0: the counters before the launch, non-finite arrivals so far, the
  // verdict on the pass before
  uint32_t epoch0, final0, arrive0, bad_seen, verdict;
  PipeParams params;
};

// A fragment of an interval that has stopped: skipped by the producer and the
// consumers alike: with several intervals no pass begins before the control
// step of the one before it, and none runs while a CTA is in its rows.
__device__ __forceinline__ bool FragFrozen(const PipeParams& p, uint32_t slab) {
  if (p.n_groups <= 1 || p.host_mode) return false;
  const uint32_t g = p.cb_group[p.slabs[slab].cb];
  return static_cast<volatile const LoopState*>(p.state)[g].done != 0;
}

__device__ __forceinline__ uint32_t SmemAddr(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
// A pointer to shared memory from its 32-bit address: passed so to functions
// kept out of line, whose pointer arguments would be read as generic memory.
template <typename T>
__device__ __forceinline__ T* SharedPtr(uint32_t at) {
  return static_cast<T*>(__cvta_shared_to_generic(at));
}
// The thread index, read anew: what is computed from it is not carried through
// (or hoisted out of) the loops around.
__device__ __forceinline__ int FreshTid() {
  int t;
  asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
  return t;
}
__device__ __forceinline__ void MbarInit(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(SmemAddr(bar)),
               "r"(count)
               : "memory");
}
__device__ __forceinline__ void MbarArriveExpectTx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(
                   SmemAddr(bar)),
               "r"(bytes)
               : "memory");
}
__device__ __forceinline__ void MbarArrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(SmemAddr(bar))
               : "memory");
}
__device__ __forceinline__ bool MbarTryWait(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n .reg .pred p;\n"
      " mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
      " selp.u32 %0, 1, 0, p;\n}"
      : "=r"(ok)
      : "r"(SmemAddr(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
__device__ __forceinline__ void BulkCopyG2S(void* dst, const void* src,
                                            uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes "
      "[%0], [%1], %2, [%3];" ::"r"(SmemAddr(dst)),
      "l"(src), "r"(bytes), "r"(SmemAddr(bar))
      : "memory");
}
// Orders this thread's generic accesses to global memory (its own writes, or
// writes it has acquired) against bulk copies of the same memory.
__device__ __forceinline__ void FenceProxyAsync() {
  asm volatile("fence.proxy.async.global;" ::: "memory");
}
__device__ __forceinline__ uint32_t LoadAcquire(const uint32_t* p) {
  uint32_t v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void StoreRelease(uint32_t* p, uint32_t v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ uint64_t GlobalTimerNs() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}
// Named barrier of the consumer warps: the warp-aligned form, entered by
// whole warps (__syncwarp first, so lane-divergent code before it is
// reconverged), at the same place by every consumer warp. Measured on B200:
// the non-aligned `barrier.sync 1, 224` let six waiting warps through while
// the seventh was still busy, and so did `bar.sync` after a loop that only
// one warp ran; waits of that kind are done by every warp instead.
template <int W>
__device__ __forceinline__ void ConsumerBarrier() {
  __syncwarp();
  asm volatile("bar.sync 1, %0;" ::"n"(W * 32) : "memory");
}

// Bounded wait on an mbarrier phase. Returns false on timeout (or when the CTA
// is already in error), after recording the error.
__device__ __forceinline__ bool PipeWaitSlow(uint64_t* bar, uint32_t parity, PipeShared& sh) {
  uint64_t t0 = 0;
  for (uint32_t n = 1;; ++n) {
    if (MbarTryWait(bar, parity)) return true;
    if ((n & 15u) == 0) {  // (reading the timer is slow)
      if (sh.err) return false;
      const uint64_t t = GlobalTimerNs();
      if (t0 == 0) t0 = t;
      if (t - t0 > sh.params.wait_ns) {
        sh.err = 1;
        atomicExch(&sh.params.counters[kCntError], 1u);
        return false;
      }
    }
  }
}
__device__ __forceinline__ bool PipeWait(uint64_t* bar, uint32_t parity, PipeShared& sh) {
  if (MbarTryWait(bar, parity)) return true;
  return PipeWaitSlow(bar, parity, sh);
}

// The consumers' wait for thread 0's news of the grid. What they do next
// depends on it, and a warp that gave up by itself would miss named barriers at
// which the others wait for good. Thread 0 always passes the news on: between
// two of them it waits at most twice, each time within the limit, so the limit
// here, four times that, is not reached.
__device__ __forceinline__ void NewsWait(uint64_t* bar, uint32_t parity, PipeShared& sh) {
  uint64_t t0 = 0;
  for (uint32_t n = 1; !MbarTryWait(bar, parity); ++n) {
    if ((n & 15u) != 0) continue;
    const uint64_t t = GlobalTimerNs();
    if (t0 == 0) t0 = t;
    if (t - t0 > 4 * sh.params.wait_ns) {
      sh.err = 1;
      atomicExch(&sh.params.counters[kCntError], 1u);
      return;
    }
  }
}

__device__ __forceinline__ uint64_t LoadAcquire64(const uint64_t* p) {
  uint64_t v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
// Thread 0's bounded wait until reached() holds; false when it ran out or an
// error is flagged.
template <typename Reached>
__device__ __forceinline__ bool GridWait(const PipeParams& p, const Reached& reached) {
  const uint64_t t0 = GlobalTimerNs();
  for (uint32_t n = 1;; ++n) {
    if (reached()) return true;
    if ((n & 63u) == 0) {
      if (static_cast<volatile uint32_t*>(p.counters)[kCntError]) return false;
      if (GlobalTimerNs() - t0 > p.wait_ns) {
        atomicExch(&p.counters[kCntError], 1u);
        return false;
      }
    }
  }
}

template <int NCORR>
__device__ __forceinline__ void LoadVisShared(const char* base, uint32_t idx,
                                              float2 (&v)[NCORR]) {
  if constexpr (NCORR == 2) {
    const float4 x = reinterpret_cast<const float4*>(base)[idx];
    v[0] = make_float2(x.x, x.y);
    v[1] = make_float2(x.z, x.w);
  } else {
    const float4 x = reinterpret_cast<const float4*>(base)[2 * idx];
    const float4 y = reinterpret_cast<const float4*>(base)[2 * idx + 1];
    v[0] = make_float2(x.x, x.y);
    v[1] = make_float2(x.z, x.w);
    v[2] = make_float2(y.x, y.y);
    v[3] = make_float2(y.z, y.w);
  }
}

// Accumulator table of pipe_kernel, per antenna `stride` floats: the
// numerators of every direction (NPOL complex values each), then the
// denominators (NPOL real values each), so that one direction's update is
// one vector read-modify-write of each (stride = 4 mod 8: distinct
// shared-memory banks for consecutive antennas).
template <int NPOL, bool HAS_DEN>
__device__ __forceinline__ void AccAdd(float* row, uint32_t n_dir, uint32_t d,
                                       const float2 (&num)[NPOL], const float (&den)[NPOL]) {
  if constexpr (NPOL == 2) {
    float4* pn = reinterpret_cast<float4*>(row) + d;
    float2* pd = reinterpret_cast<float2*>(row + 4 * n_dir) + d;
    float4 v = *pn;
    float2 w = HAS_DEN ? *pd : make_float2(0.f, 0.f);
    v.x += num[0].x;
    v.y += num[0].y;
    v.z += num[1].x;
    v.w += num[1].y;
    *pn = v;
    if constexpr (HAS_DEN) {
      w.x += den[0];
      w.y += den[1];
      *pd = w;
    }
  } else {
    float2* pn = reinterpret_cast<float2*>(row) + d;
    float2 v = *pn;
    v.x += num[0].x;
    v.y += num[0].y;
    *pn = v;
    if constexpr (HAS_DEN) row[2 * n_dir + d] += den[0];
  }
}
__host__ __device__ constexpr uint32_t AccNumOffset(uint32_t npol, uint32_t d, uint32_t q) {
  return (d * npol + q) * 2;
}
__host__ __device__ constexpr uint32_t AccDenOffset(uint32_t npol, uint32_t n_dir, uint32_t d,
                                                    uint32_t q) {
  return 2 * npol * n_dir + d * npol + q;
}

// Gains of antenna `ant`, direction d from a gain table (NPOL float2 per
// direction; for two polarizations one 16-byte load: stride = 2 mod 4).
template <int NPOL>
__device__ __forceinline__ void LoadGains(const float2* gtab, uint32_t ant, uint32_t stride,
                                          uint32_t d, float2 (&g)[NPOL]) {
  if constexpr (NPOL == 2) {
    const float4 v = *reinterpret_cast<const float4*>(gtab + size_t(ant) * stride + 2 * d);
    g[0] = make_float2(v.x, v.y);
    g[1] = make_float2(v.z, v.w);
  } else {
    g[0] = gtab[size_t(ant) * stride + d];
  }
}

// Writes the FP32 gain-table entries of solution (cb, ant, s): one entry per
// gain table of that channel block whose slab uses sub-solution s.
template <int NPOL>
__device__ __forceinline__ void WriteTables(const PipeParams& p, uint32_t cb, uint32_t ant,
                                            uint32_t s, uint32_t entry,
                                            const double2 (&v)[NPOL]) {
  auto put = [&](uint32_t e) {
    float2* t = p.tables + size_t(e >> 8) * p.table_f2 + size_t(ant) * p.gain_stride +
                (e & 255u) * NPOL;
#pragma unroll
    for (int q = 0; q < NPOL; ++q) t[q] = make_float2(float(v[q].x), float(v[q].y));
  };
  if (entry != kManyEntries) {
    put(entry);
    return;
  }
  const uint32_t k1 = p.tab_off[cb * p.n_sub + s + 1];
  for (uint32_t k = p.tab_off[cb * p.n_sub + s]; k < k1; ++k) put(p.tab_ent[k]);
}

// |diff / old| of the AssignSolutions norm; false where the quotient by the
// inverse of `old` would not be finite. Within the range where neither square
// can over- or underflow it is one division and one square root.
__device__ __noinline__ bool StepNormSlow(double2 old, double2 diff, double& r) {
  const double2 inv = dinv(old);
  if (!dfinite(inv)) return false;
  const double2 q = dmul(diff, inv);
  r = hypot(q.x, q.y);
  return true;
}
__device__ __forceinline__ bool StepNorm(double2 old, double2 diff, double& r) {
  const double o2 = old.x * old.x + old.y * old.y, d2 = diff.x * diff.x + diff.y * diff.y;
  if (o2 > 1e-200 && o2 < 1e200 && d2 < 1e200 && (d2 > 1e-200 || d2 == 0.0)) {
    r = sqrt(d2 / o2);
    return true;
  }
  return StepNormSlow(old, diff, r);
}

// One item's sums in a partial slot: NPOL complex numerators and NPOL real
// denominators (AccAdd), as one vector load of each.
template <int NPOL>
__device__ __forceinline__ void LoadSlot(const float* num, const float* den,
                                         float (&v)[NPOL * 3]) {
  if constexpr (NPOL == 2) {
    const float4 n = __ldcg(reinterpret_cast<const float4*>(num));
    const float2 d = __ldcg(reinterpret_cast<const float2*>(den));
    v[0] = n.x;
    v[1] = n.y;
    v[2] = n.z;
    v[3] = n.w;
    v[4] = d.x;
    v[5] = d.y;
  } else {
    const float2 n = __ldcg(reinterpret_cast<const float2*>(num));
    v[0] = n.x;
    v[1] = n.y;
    v[2] = __ldcg(den);
  }
}

// Sums (and the or of `flag`) over the consumer threads of a CTA in a fixed
// order; valid in thread 0. s_cnt: two words per warp.
template <int W>
__device__ __forceinline__ void BlockNorm(int ctid, double& sum, uint32_t& cnt, bool& flag,
                                          double* s_sum, uint32_t* s_cnt) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
    cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
  }
  flag = __any_sync(0xFFFFFFFFu, flag);
  if ((ctid & 31) == 0) {
    s_sum[ctid >> 5] = sum;
    s_cnt[2 * (ctid >> 5)] = cnt;
    s_cnt[2 * (ctid >> 5) + 1] = flag ? 1u : 0u;
  }
  ConsumerBarrier<W>();
  if (ctid == 0)
    for (int w = 1; w < W; ++w) {
      sum += s_sum[w];
      cnt += s_cnt[2 * w];
      flag = flag || s_cnt[2 * w + 1] != 0;
    }
}

// An interval's loop state, read and written past L1: within one launch one
// CTA changes it, pass by pass, and every CTA reads it.
__device__ __forceinline__ LoopState LoadState(const LoopState* s) {
  static_assert(sizeof(LoopState) % 8 == 0, "copied in 8-byte words");
  LoopState r;
  const uint2* src = reinterpret_cast<const uint2*>(s);
  uint2* dst = reinterpret_cast<uint2*>(&r);
#pragma unroll
  for (size_t i = 0; i < sizeof(LoopState) / 8; ++i) dst[i] = __ldcg(src + i);
  return r;
}
__device__ __forceinline__ void StoreState(LoopState* s, const LoopState& v) {
  uint2* dst = reinterpret_cast<uint2*>(s);
  const uint2* src = reinterpret_cast<const uint2*>(&v);
#pragma unroll
  for (size_t i = 0; i < sizeof(LoopState) / 8; ++i) __stcg(dst + i, src[i]);
}

// The control step of a pass, run by one CTA after all have finalised it:
// sums each interval's per-CTA norms in a fixed order, runs
// ReachedStoppingCriterion / DetectStall (SolverBase.h:274-285,
// SolverBase.cc:63-86), and (`bad`) prepares the next iteration's
// MakeSolutionsFinite{1,2}Pol (SolverBase.cc:316-371) of the channel blocks
// that got non-finite solutions. Returns the verdict (in thread 0). All
// consumer threads of the CTA take part; s_flag: two words.
template <int W, int NPOL>
__device__ __forceinline__ uint32_t ControlPass(const PipeParams& p, int ctid, bool bad,
                                                double* s_sum, uint32_t* s_cnt,
                                                uint32_t* s_flag) {
  const DevSettings st = *p.settings;
  const bool error = static_cast<volatile uint32_t*>(p.counters)[kCntError] != 0;
  if (bad) {
    // Replacement values for channel blocks with new non-finite solutions:
    // mean |pol 0| over finite pairs; the gain tables take the replacement
    // now, the solutions when the next finalisation reads them.
    const uint32_t n_items_cb = p.n_ant * p.n_sub;
    for (uint32_t cb = 0; cb < p.n_cb; ++cb) {
      if (static_cast<volatile uint32_t*>(p.cb_newflag)[cb] == 0) continue;
      double asum = 0.0;
      uint32_t acnt = 0;
      for (uint32_t i = ctid; i < n_items_cb; i += (W * 32)) {
        const double2* sol = p.solutions + (size_t(cb) * n_items_cb + i) * NPOL;
        bool ok = true;
        double2 v[NPOL];
#pragma unroll
        for (int q = 0; q < NPOL; ++q) {
          v[q] = __ldcg(sol + q);
          ok = ok && dfinite(v[q]);
        }
        if (ok) {
          asum += hypot(v[0].x, v[0].y);
          ++acnt;
        }
      }
      bool unused = false;
      BlockNorm<W>(ctid, asum, acnt, unused, s_sum, s_cnt);
      if (ctid == 0) s_sum[0] = acnt == 0 ? 1.0 : asum / double(acnt);
      ConsumerBarrier<W>();
      const double avg = s_sum[0];
      for (uint32_t i = ctid; i < n_items_cb; i += (W * 32)) {
        const double2* sol = p.solutions + (size_t(cb) * n_items_cb + i) * NPOL;
        bool ok = true;
#pragma unroll
        for (int q = 0; q < NPOL; ++q) ok = ok && dfinite(__ldcg(sol + q));
        if (!ok) {
          double2 r[NPOL];
#pragma unroll
          for (int q = 0; q < NPOL; ++q) r[q] = make_double2(avg, 0.0);
          WriteTables<NPOL>(p, cb, i / p.n_sub, i % p.n_sub, kManyEntries, r);
        }
      }
      ConsumerBarrier<W>();
      if (ctid == 0) {
        __stcg(p.cb_avg + cb, avg);
        __stcg(p.cb_flag + cb, 1u);
        p.cb_newflag[cb] = 0u;
      }
      ConsumerBarrier<W>();
    }
    FenceProxyAsync();
    ConsumerBarrier<W>();
  }
  uint32_t verdict = 0;
  if (p.n_groups == 1) {
    if (ctid >= 32) return 0u;
    LoopState ls = LoadState(p.state);  // (issued with the norms' loads)
    double sum = 0.0;
    uint32_t cnt = 0;
    constexpr int kLoads = 5;  // 160 CTAs per round
    for (uint32_t b0 = ctid; b0 < gridDim.x; b0 += 32 * kLoads) {
      double v[kLoads];
      uint32_t c[kLoads];
#pragma unroll
      for (int k = 0; k < kLoads; ++k) {
        const uint32_t b = min(b0 + 32 * k, gridDim.x - 1);
        v[k] = __ldcg(p.block_sum + b);
        c[k] = __ldcg(p.block_cnt + b);
      }
#pragma unroll
      for (int k = 0; k < kLoads; ++k)
        if (b0 + 32 * k < gridDim.x) {
          sum += v[k];
          cnt += c[k];
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
      cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
    }
    if (ctid == 0) {
      bool stop = ControlStep(ls, st, sum, cnt, p.step_magnitudes);
      if (error) {
        ls.done = 1;
        stop = true;
      }
      StoreState(p.state, ls);
      // within a factor of two of a criterion (or not comparable with it)
      const double mag = cnt == 0 ? 0.0 : sum / st.step_size / double(cnt);
      const bool near_end = !(mag > 2.0 * st.accuracy) ||
                            (st.detect_stalling &&
                             !(ls.step_mean > 2.0 * st.step_diff_sigma *
                                                  sqrt(ls.step_var / double(ls.n_var_count))));
      verdict = (stop ? kVerdictStop : 0u) | (near_end ? kVerdictNear : 0u);
    }
    return verdict;
  }
  // Several intervals: one warp per interval still going sums its norm
  // partials (in chunk order per lane) and runs its control step; the loop
  // goes on while any interval does.
  ConsumerBarrier<W>();
  if (ctid == 0) s_flag[0] = 0u;
  ConsumerBarrier<W>();
  const int lane = ctid & 31;
  for (uint32_t g = uint32_t(ctid >> 5); g < p.n_groups; g += W) {
    LoopState ls = LoadState(p.state + g);
    if (ls.done) continue;
    double sum = 0.0;
    uint32_t cnt = 0;
    const uint32_t c1 = p.group_chunk[g + 1];
#pragma unroll 4
    for (uint32_t c = p.group_chunk[g] + lane; c < c1; c += 32) {
      sum += __ldcg(p.block_sum + c);
      cnt += __ldcg(p.block_cnt + c);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      sum += __shfl_xor_sync(0xFFFFFFFFu, sum, o);
      cnt += __shfl_xor_sync(0xFFFFFFFFu, cnt, o);
    }
    if (lane == 0) {
      bool stop = ControlStep(ls, st, sum, cnt, p.step_magnitudes + size_t(g) * p.mags_stride);
      if (error) {
        ls.done = 1;
        stop = true;
      }
      StoreState(p.state + g, ls);
      __threadfence();
      if (!stop) atomicOr(&s_flag[0], 1u);
    }
    __syncwarp();
  }
  ConsumerBarrier<W>();
  return s_flag[0] ? kVerdictNear : kVerdictStop | kVerdictNear;
}

// Grid-wide finalisation of a pass of pipe_kernel, after the grid barrier:
// the consumer threads of all CTAs take (channel block, antenna,
// sub-solution) items, warp by warp over the CTAs (with several intervals, at
// most 32 items of one interval a warp): fixed-order compensated merge
// of the item's partial slots, FP64 add-back and division
// (IterativeDiagonalSolver.cc:206-221, IterativeScalarSolver.cc:184-194),
// SolverBase::Step (SolverBase.cc:88-158), the AssignSolutions norm
// (SolverBase.cc:234-285), and the FP32 gain tables of the next iteration.
// With device constraints the work is split by p.fin_mode: kFinStepOnly
// (pipe_kernel) stops after the step, writing the stepped solutions to
// next_out; kFinAssignOnly (assign_kernel) starts from the constrained ones
// in next_out. `it` is the pass of the launch. Solutions change between the
// passes of a launch, so they are read past L1. wait_slots() is the grid
// barrier, false when the launch ends there; what an item needs besides its
// slots is read before it. Returns false with it, else sets `bad` (in thread
// 0) when the CTA's items got non-finite solutions.
// Bound by latency (7440 items of a 62-station, 12-block, 10-direction
// interval are one item per thread of a quarter of the grid; a dependent read
// of L2 costs 0.7 us): the items are spread over all CTAs and an item's slots
// are loaded together, numerators and denominators as one vector each.
template <int W, int NPOL, typename WaitSlots>
__device__ __forceinline__ bool FinalizeDistributed(const PipeParams& p, uint32_t it, int ctid,
                                                    double* s_sum, uint32_t* s_cnt, bool& bad,
                                                    const WaitSlots& wait_slots) {
  const DevSettings st = *p.settings;
  const uint32_t n_items_cb = p.n_ant * p.n_sub;
  const uint32_t n_items = p.n_cb * n_items_cb;
  const bool chained = p.host_mode && it > 0;
  const double2* sol_in =
      chained ? p.next_out + size_t(it - 1) * p.out_stride : p.solutions;
  double2* nxt_out = p.next_out + size_t(p.host_mode ? it : 0u) * p.out_stride;
  double nsum = 0.0;
  uint32_t ncnt = 0;
  bad = false;
  // One item: the merged sums and the old solutions in, the next solutions,
  // their norm terms, the gain tables and the non-finite flag out.
  auto finish = [&](uint32_t item, uint32_t cb, uint32_t ant, uint32_t s, uint32_t entry,
                    const double2 (&old_in)[NPOL], const NeumaierSum (&nr)[NPOL],
                    const NeumaierSum (&ni)[NPOL], const NeumaierSum (&dn)[NPOL]) {
    double2* sol = p.solutions + size_t(item) * NPOL;
    double2 old[NPOL], nxt[NPOL];
    bool pair_ok = true;
#pragma unroll
    for (int q = 0; q < NPOL; ++q) {
      old[q] = old_in[q];
      pair_ok = pair_ok && dfinite(old[q]);
    }
    // the lazy MakeSolutionsFinite of a solve (next-solutions passes use the
    // solutions they are given, as PerformIteration does)
    if (!pair_ok && !p.host_mode && __ldcg(p.cb_flag + cb)) {
      const double rv = __ldcg(p.cb_avg + cb);
#pragma unroll
      for (int q = 0; q < NPOL; ++q) old[q] = make_double2(rv, 0.0);
    }
#pragma unroll
    for (int q = 0; q < NPOL; ++q) {
      const float den = dn[q].Value();
      if (den == 0.f) {
        nxt[q] = make_double2(nan(""), 0.0);
      } else {
        nxt[q] = make_double2(
            double(float(old[q].x)) + double(nr[q].Value()) / double(den),
            double(float(old[q].y)) + double(ni[q].Value()) / double(den));
      }
    }
    double2* out = nxt_out + size_t(item) * NPOL;
    if (p.host_mode) {
#pragma unroll
      for (int q = 0; q < NPOL; ++q) out[q] = nxt[q];
      // the gain tables of a chained next pass, which starts from `nxt`
      // (every other launch rebuilds them from its own solutions first)
      WriteTables<NPOL>(p, cb, ant, s, entry, nxt);
      return;
    }
    if (p.fin_mode == kFinAssignOnly) {
      // the stepped and constrained next solutions of this iteration
#pragma unroll
      for (int q = 0; q < NPOL; ++q) nxt[q] = out[q];
    } else {
#pragma unroll
      for (int q = 0; q < NPOL; ++q) {
        if (!st.phase_only) {
          nxt[q] = make_double2(old[q].x * (1.0 - st.step_size) + nxt[q].x * st.step_size,
                                old[q].y * (1.0 - st.step_size) + nxt[q].y * st.step_size);
        } else {
          const double from = atan2(old[q].y, old[q].x);
          double dist = atan2(nxt[q].y, nxt[q].x) - from;
          if (dist > M_PI)
            dist -= 2.0 * M_PI;
          else if (dist < -M_PI)
            dist += 2.0 * M_PI;
          double sn, cs;
          sincos(from + st.step_size * dist, &sn, &cs);
          nxt[q] = make_double2(cs, sn);
        }
      }
      if (p.fin_mode == kFinStepOnly) {
#pragma unroll
        for (int q = 0; q < NPOL; ++q) out[q] = nxt[q];
        return;
      }
    }
    {  // (a polarization pair counts when both do; a zero solution does not)
      double r = 0.0;
      bool ok = true;
#pragma unroll
      for (int q = 0; q < NPOL; ++q) {
        double rq = 0.0;
        ok = StepNorm(old[q], make_double2(nxt[q].x - old[q].x, nxt[q].y - old[q].y), rq) && ok;
        r += rq;
      }
      if (ok && isfinite(r)) {
        nsum += r;
        ncnt += NPOL;
      }
    }
    bool all_finite = true;
#pragma unroll
    for (int q = 0; q < NPOL; ++q) {
      sol[q] = nxt[q];
      all_finite = all_finite && dfinite(nxt[q]);
    }
    WriteTables<NPOL>(p, cb, ant, s, entry, nxt);
    if (!all_finite) {
      p.cb_newflag[cb] = 1u;
      bad = true;
    }
  };
  const uint32_t item_step = gridDim.x * (W * 32);
  const uint32_t item_first =
      (uint32_t(ctid >> 5) * gridDim.x + blockIdx.x) * 32u + uint32_t(ctid & 31);
  struct Item {
    uint32_t cb, ant, s;
    uint4 list;  // FinList
    double2 old[NPOL];
  };
  auto fetch = [&](uint32_t item, Item& x) {
    x.cb = item / n_items_cb;
    const uint32_t rem = item - x.cb * n_items_cb;
    x.ant = rem / p.n_sub;
    x.s = rem - x.ant * p.n_sub;
    x.list = *reinterpret_cast<const uint4*>(p.fin_lists + x.cb * p.n_sub + x.s);
#pragma unroll
    for (int q = 0; q < NPOL; ++q) x.old[q] = __ldcg(sol_in + size_t(item) * NPOL + q);
  };
  Item x{};
  const bool single = p.n_groups == 1;
  // Four lanes share an item, a few slots each, where the grid has them: one
  // round trip for 16 slots, and registers for 4 of them only.
  const uint32_t share = single && n_items <= item_step / 4 ? 2u : 0u;
  if (single && (item_first >> share) < n_items) fetch(item_first >> share, x);
  if (!wait_slots()) return false;
  // The items, warp by warp over the CTAs; a lane reads its slots of an item
  // kR at a time and adds them in slot order, and the lanes of the item then
  // add up theirs.
  auto merge = [&](uint32_t item, const Item& x, uint32_t part) {
    const bool range = (x.list.y & kFinRange) != 0;
    // no partial slots to merge after the constraints
    const uint32_t count = p.fin_mode == kFinAssignOnly ? 0u : x.list.y & ~kFinRange;
    // the item's numerators and denominators in a partial slot (AccAdd)
    const float* num = p.partials + size_t(x.ant) * p.acc_stride + AccNumOffset(NPOL, x.list.z, 0);
    const float* den =
        p.partials + size_t(x.ant) * p.acc_stride + AccDenOffset(NPOL, p.n_dir, x.list.z, 0);
    NeumaierSum nr[NPOL], ni[NPOL], dn[NPOL];
    // slots per round (8 at once spill the row loop of kWarps warps)
    constexpr uint32_t kR = W == kWideWarps ? 6 : 4;
    for (uint32_t k = part * kR; k < count; k += kR << share) {
      float v[kR][NPOL * 3];
#pragma unroll
      for (uint32_t u = 0; u < kR; ++u) {
        if (k + u >= count) break;
        const size_t at =
            size_t(range ? x.list.x + k + u : p.fin_visits[x.list.x + k + u]) * p.acc_floats;
        LoadSlot<NPOL>(num + at, den + at, v[u]);
      }
#pragma unroll
      for (uint32_t u = 0; u < kR; ++u) {
        if (k + u >= count) break;
#pragma unroll
        for (int q = 0; q < NPOL; ++q) {
          nr[q].Add(v[u][q * 2 + 0]);
          ni[q].Add(v[u][q * 2 + 1]);
          dn[q].Add(v[u][NPOL * 2 + q]);
        }
      }
    }
    if (share) {
      const uint32_t lanes = 15u << (ctid & 28);
#pragma unroll
      for (int o = 1; o < 4; o <<= 1)
#pragma unroll
        for (int q = 0; q < NPOL; ++q) {
          nr[q].Join(lanes, o);
          ni[q].Join(lanes, o);
          dn[q].Join(lanes, o);
        }
      if (part) return;
    }
    finish(item, x.cb, x.ant, x.s, x.list.w, x.old, nr, ni, dn);
  };
  if (single) {
    for (uint32_t i = item_first; (i >> share) < n_items; i += item_step) {
      const Item now = x;
      if (((i + item_step) >> share) < n_items) fetch((i + item_step) >> share, x);
      merge(i >> share, now, i & ((1u << share) - 1u));
    }
    FenceProxyAsync();  // the gain tables, before the next pass's bulk copies
    BlockNorm<W>(ctid, nsum, ncnt, bad, s_sum, s_cnt);
    if (ctid == 0) {
      __stcg(p.block_sum + blockIdx.x, nsum);
      __stcg(p.block_cnt + blockIdx.x, ncnt);
    }
    return true;
  }
  // Several intervals: an interval that has stopped keeps its solutions.
  for (uint32_t c = uint32_t(ctid >> 5) * gridDim.x + blockIdx.x; c < p.n_chunks;
       c += gridDim.x * W) {
    const uint2 chunk = p.chunks[c];
    if (!p.host_mode &&
        static_cast<volatile const LoopState*>(p.state)[chunk.y & 0xFFFFFFu].done != 0)
      continue;
    nsum = 0.0;
    ncnt = 0;
    if (uint32_t(ctid & 31) < chunk.y >> 24) {
      const uint32_t item = chunk.x + uint32_t(ctid & 31);
      fetch(item, x);
      merge(item, x, 0);
    }
    __syncwarp();
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      nsum += __shfl_xor_sync(0xFFFFFFFFu, nsum, o);
      ncnt += __shfl_xor_sync(0xFFFFFFFFu, ncnt, o);
    }
    if ((ctid & 31) == 0) {
      __stcg(p.block_sum + c, nsum);
      __stcg(p.block_cnt + c, ncnt);
    }
  }
  FenceProxyAsync();
  nsum = 0.0;
  ncnt = 0;
  BlockNorm<W>(ctid, nsum, ncnt, bad, s_sum, s_cnt);
  return true;
}

// Builds the FP32 gain tables from the FP64 solutions: one thread per
// (table, antenna, direction). tab_cb / tab_sol give each table's channel
// block and per-direction sub-solution.
template <int NPOL>
__global__ void build_tables_kernel(const double2* __restrict__ solutions,
                                    float2* __restrict__ tables,
                                    const uint32_t* __restrict__ tab_cb,
                                    const uint32_t* __restrict__ tab_sol,
                                    uint32_t n_tables, uint32_t n_ant, uint32_t n_dir,
                                    uint32_t n_sub, uint32_t gain_stride,
                                    uint32_t table_f2) {
  const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n_tables * n_ant * n_dir) return;
  const uint32_t tab = i / (n_ant * n_dir);
  const uint32_t rem = i - tab * n_ant * n_dir;
  const uint32_t ant = rem / n_dir;
  const uint32_t d = rem - ant * n_dir;
  const uint32_t s = tab_sol[tab * n_dir + d];
  const double2* src = solutions + (size_t(tab_cb[tab] * n_ant + ant) * n_sub + s) * NPOL;
  float2* dst = tables + size_t(tab) * table_f2 + size_t(ant) * gain_stride + d * NPOL;
#pragma unroll
  for (int q = 0; q < NPOL; ++q) dst[q] = make_float2(float(src[q].x), float(src[q].y));
}

// Model powers of the pipelined path: for every tile of runs, direction and
// correlation, sum over the tile's (time, channel) rows of |M|^2. They depend
// on the model alone, so they are computed once per upload instead of in
// every iteration's row loop. One block per (tile, direction), one thread per
// run; FP64 sums, stored as FP32.
struct PowerTile {
  uint32_t slab, r0, n, pad;
};

template <int NCORR>
__global__ void __launch_bounds__(kWarps * 32)
    power_kernel(const SlabDesc* __restrict__ slabs, const PowerTile* __restrict__ tiles,
                 uint32_t n_dir, uint32_t power_floats, float* __restrict__ powers) {
  const uint32_t tile = blockIdx.x / n_dir;
  const uint32_t k = blockIdx.x - tile * n_dir;
  const PowerTile t = tiles[tile];
  const SlabDesc sl = slabs[t.slab];
  const uint32_t r = threadIdx.x;  // blockDim.x: the runs of a full tile
  double q[NCORR];
#pragma unroll
  for (int c = 0; c < NCORR; ++c) q[c] = 0.0;
  if (r < t.n) {
    const size_t rows = size_t(sl.T) * sl.L;
    const uint32_t nd1 = 1 + n_dir;
    const float2* m = static_cast<const float2*>(sl.vis) +
                      SlabElem(sl.R, sl.W, nd1, 0, 1 + k, t.r0 + r) * NCORR;
    for (size_t row = 0; row < rows; ++row, m += size_t(sl.R) * nd1 * NCORR) {
#pragma unroll
      for (int c = 0; c < NCORR; ++c) {
        const float2 v = __ldcs(m + c);
        q[c] += double(v.x) * v.x + double(v.y) * v.y;
      }
    }
  }
  float* out = powers + size_t(tile) * power_floats + (size_t(k) * blockDim.x + r) * NCORR;
#pragma unroll
  for (int c = 0; c < NCORR; ++c) out[c] = float(q[c]);
}

// The end of a pass of pipe_kernel, from the partial slots of this CTA on;
// false when the launch ends with it.
template <int W, int NPOL>
__device__ __forceinline__ bool EndPass(uint32_t smem_at, uint32_t it) {
  const int ctid = FreshTid();
  PipeShared& sh = *SharedPtr<PipeShared>(smem_at);
  const PipeParams& p = sh.params;
  const bool control = !p.host_mode && p.fin_mode == kFinFused;
  const bool is_control = blockIdx.x == gridDim.x - 1;
  // Grid barrier: every CTA has flushed every partial slot (the launch is
  // cooperative, so all CTAs are resident). Thread 0 polls the arrival count
  // and passes it on through an mbarrier (a named barrier after one warp's
  // polling loop was measured to let the other warps through early). Bounded:
  // a timeout flags an error and the finalisation goes ahead on whatever is
  // there; an error anywhere ends every wait.
  // A pass may have begun before the verdict on the one before it was known
  // (see below): if that ends the solve, the pass ends here, with nothing but
  // partial slots written.
  ConsumerBarrier<W>();  // this CTA's slots are written
  if (ctid == 0) {
    __threadfence();
    atomicAdd(&p.counters[kCntArrive], 1u);
  }
  bool bad;
  const bool go = FinalizeDistributed<W, NPOL>(p, it, ctid, sh.sum, sh.cnt, bad, [&]() {
    if (ctid == 0) {
      const uint32_t target = (it + 1) * gridDim.x + p.arrive_extra;
      GridWait(p,
               [&]() { return LoadAcquire(&p.counters[kCntArrive]) - sh.arrive0 >= target; });
      if (control && it > 0) {
        const bool known = GridWait(
            p, [&]() { return LoadAcquire(&p.counters[kCntEpoch]) - sh.epoch0 >= it; });
        uint32_t v = kVerdictStop;
        if (known) v = static_cast<volatile uint32_t*>(p.counters)[kCntVerdict];
        sh.verdict = v;
        if (v & kVerdictStop) {
          sh.stop = 1u;
          __threadfence_block();
          sh.passes = 0xFFFFFFFFu;
        }
      }
      MbarArrive(&sh.flushed);
    }
    NewsWait(&sh.flushed, it & 1u, sh);
    return sh.stop == 0u;
  });
  if (!go) return false;
  // The solutions and gain tables of every CTA are final when all have
  // arrived; the last CTA (with the fewest rows) runs the control step. The
  // next pass begins at once where the solve is not about to end (or its
  // verdict could change what the pass reads: several intervals, non-finite
  // solutions); the verdict is looked at before its finalisation, the first
  // step that could not be undone.
  bool all_bad = false;
  if (ctid == 0) {
    __threadfence();
    atomicAdd(reinterpret_cast<unsigned long long*>(p.counters + kCntFinal),
              1ull | (bad ? 1ull << 32 : 0ull));
    uint64_t count = 0;
    const uint32_t target = (it + 1) * gridDim.x;
    const bool done = GridWait(p, [&]() {
      count = LoadAcquire64(reinterpret_cast<const uint64_t*>(p.counters + kCntFinal));
      return uint32_t(count) - sh.final0 >= target;
    });
    all_bad = uint32_t(count >> 32) != sh.bad_seen;
    sh.bad_seen = uint32_t(count >> 32);
    if (!done) sh.stop = 1u;
    sh.flag[1] = !done ? 2u : all_bad ? 1u : 0u;
    if (control && is_control) MbarArrive(&sh.finalised);
  }
  if (control && is_control) {
    // (every warp waits for the news itself: no named barrier right after
    // thread 0's polling, see ConsumerBarrier)
    NewsWait(&sh.finalised, it & 1u, sh);
    // Where the wait ran out there is no control step: another CTA may still be
    // in the rows of the pass, whose fragments depend on which intervals go on.
    const uint32_t news = sh.flag[1];
    const uint32_t v =
        news == 2u ? kVerdictStop
                   : ControlPass<W, NPOL>(p, ctid, news != 0u, sh.sum, sh.cnt, sh.flag);
    if (ctid == 0) {
      if ((v & kVerdictStop) && p.host_stopped) *p.host_stopped = 1u;
      p.counters[kCntVerdict] = v;
      StoreRelease(&p.counters[kCntEpoch], sh.epoch0 + it + 1);
    }
  }
  if (it + 1 == p.n_iters) return false;
  if (ctid == 0) {
    if (control && (it == 0 || all_bad || p.n_groups > 1 || (sh.verdict & kVerdictNear))) {
      const bool known = GridWait(
          p, [&]() { return LoadAcquire(&p.counters[kCntEpoch]) - sh.epoch0 >= it + 1; });
      uint32_t v = kVerdictStop;
      if (known) v = static_cast<volatile uint32_t*>(p.counters)[kCntVerdict];
      sh.verdict = v;
      if (v & kVerdictStop) sh.stop = 1u;
    }
    __threadfence_block();
    sh.passes = it + 1;
    MbarArrive(&sh.ready);
  }
  NewsWait(&sh.ready, it & 1u, sh);
  return sh.stop == 0u;
}

// What a tile's fragments need of its runs besides the visibilities, one
// block of 32-bit words per tile (equal tiles of different channel blocks
// share one), copied to shared memory with a fragment's first row:
//   [0] antennas of the tile, [1] first word of their list, [2] of the entries
//   [4 ..) antenna1 | antenna2 << 16 of each run
//   list: antenna | first entry << 16, ascending, and one end mark
//   entries: run | side << 15 | other antenna << 16, by antenna, runs ascending
//   (side 1: the antenna is the run's antenna 2)
constexpr uint32_t kMetaRuns = 4;
__host__ __device__ constexpr uint32_t MetaWords(uint32_t runs, uint32_t n_ant) {
  const uint32_t present = n_ant < 2 * runs ? n_ant : 2 * runs;
  return kMetaRuns + ((runs + 3u) & ~3u) + ((present + 1u + 3u) & ~3u) + ((2 * runs + 3u) & ~3u);
}

// The second half of a tile's reduction (GatherTile): one antenna's sums over
// `n` of its entries in a tile (at most kGather) for the staged directions
// j, j + step, ...
constexpr uint32_t kGather = 4;
template <int NCORR, int NPOL, int RUNS, bool HAS_Q>
__device__ __forceinline__ void GatherEntries(const uint32_t (&en)[kGather], uint32_t n,
                                              uint32_t gtab_at, uint32_t gain_bytes,
                                              uint32_t stg_at, uint32_t q_at, float* row,
                                              uint32_t n_dir, uint32_t d0, uint32_t j,
                                              uint32_t step, uint32_t n_staged) {
  uint32_t gains[kGather], run[kGather];
#pragma unroll
  for (uint32_t u = 0; u < kGather; ++u) {
    run[u] = en[u] & 0x7FFFu;
    gains[u] = gtab_at + (en[u] >> 16) * gain_bytes + d0 * NPOL * 8;
  }
#pragma unroll 2
  for (; j < n_staged; j += step) {
    float2 num[NPOL];
    float den[NPOL];
#pragma unroll
    for (int q = 0; q < NPOL; ++q) {
      num[q] = make_float2(0.f, 0.f);
      den[q] = 0.f;
    }
    if constexpr (NPOL == 1) {
      // one gain for every correlation: their sums are staged
      const float2* const v_at = SharedPtr<const float2>(stg_at + j * (RUNS * 8));
      const float* const z_at = SharedPtr<const float>(q_at + j * (RUNS * 4));
#pragma unroll
      for (uint32_t u = 0; u < kGather; ++u) {
        if (u >= n) break;
        const float2 gc = *SharedPtr<const float2>(gains[u] + j * 8);
        const float2 v = v_at[run[u]];
        const float vy = __uint_as_float(__float_as_uint(v.y) ^ ((en[u] << 16) & 0x80000000u));
        num[0].x = fmaf(gc.x, v.x, fmaf(-gc.y, vy, num[0].x));
        num[0].y = fmaf(gc.x, vy, fmaf(gc.y, v.x, num[0].y));
        den[0] = fmaf(cnorm(gc), z_at[run[u]], den[0]);
      }
    } else {
      const uint32_t p_at = stg_at + j * (RUNS * NCORR * 8);
      const uint32_t qj_at = q_at + j * (RUNS * NCORR * 4);
#pragma unroll
      for (uint32_t u = 0; u < kGather; ++u) {
        if (u >= n) break;
        const uint32_t flip = (en[u] << 16) & 0x80000000u;  // side 1: the Hermitian transpose
        float2 gb[NPOL];
        LoadGains<NPOL>(SharedPtr<const float2>(gains[u] + j * NPOL * 8), 0, 0, 0, gb);
        float2 Pc[NCORR];
        LoadVisShared<NCORR>(SharedPtr<const char>(p_at), run[u], Pc);
#pragma unroll
        for (int c = 0; c < NCORR; ++c)
          Pc[c].y = __uint_as_float(__float_as_uint(Pc[c].y) ^ flip);
        float Qc[NCORR];
        if constexpr (HAS_Q) {
          if constexpr (NCORR == 2) {
            const float2 w = SharedPtr<const float2>(qj_at)[run[u]];
            Qc[0] = w.x;
            Qc[NCORR - 1] = w.y;
          } else {
            const float4 w = SharedPtr<const float4>(qj_at)[run[u]];
            Qc[0] = w.x;
            Qc[1] = flip ? w.z : w.y;
            Qc[2] = flip ? w.y : w.z;
            Qc[NCORR - 1] = w.w;
          }
        }
        if constexpr (NCORR == 4) {
          const float2 t = Pc[1];
          Pc[1] = flip ? Pc[2] : Pc[1];
          Pc[2] = flip ? t : Pc[2];
        }
#pragma unroll
        for (int c = 0; c < NCORR; ++c) {  // num += g_b P, den += |g_b|^2 Q
          const int q = RowPol<NCORR, NPOL>(c);
          const float2 gc = gb[ColPol<NCORR, NPOL>(c)];
          num[q].x = fmaf(gc.x, Pc[c].x, fmaf(-gc.y, Pc[c].y, num[q].x));
          num[q].y = fmaf(gc.x, Pc[c].y, fmaf(gc.y, Pc[c].x, num[q].y));
          if constexpr (HAS_Q) den[q] = fmaf(cnorm(gc), Qc[c], den[q]);
        }
      }
    }
    AccAdd<NPOL, HAS_Q>(row, n_dir, d0 + j, num, den);
  }
}

// The second half of a tile's reduction: the antennas' sums over the staged
// directions d0 .. d0 + n_staged - 1, P at stg[j][run][corr] and the model
// powers at q[j][run][corr] (0: none in this fragment); for one polarization
// their sums over the correlations, P at stg[j][run] and Q at q[j][run]. Thread (i, j0) adds up
// antenna i (and i + (W * 32), ...) for the staged directions j0, j0 +
// step, ..., over the antenna's entries in their order, kGather entries per
// update of an accumulator: few barriers and read-modify-write chains,
// whatever the order of the runs. Consecutive threads take consecutive
// antennas, mostly of consecutive runs: distinct shared-memory banks.
template <int W, int NCORR, int NPOL, int RUNS>
__device__ __forceinline__ void GatherTile(uint32_t meta_at, uint32_t gtab_at, uint32_t stg_at,
                                        uint32_t q_at, uint32_t acc_at, uint32_t ctid,
                                        uint32_t n_dir, uint32_t d0, uint32_t n_staged,
                                        uint32_t acc_stride, uint32_t gain_stride) {
  const uint32_t* const meta = SharedPtr<const uint32_t>(meta_at);
  float* const acc = SharedPtr<float>(acc_at);
  const uint32_t n_present = meta[0];
  const uint32_t* const list = meta + meta[1];
  const uint32_t* const ent = meta + meta[2];
  const uint32_t step = n_present < (W * 32) ? (W * 32) / n_present : 1u;
  const uint32_t j = step > 1 ? ctid / n_present : 0u;
  if (j >= step || j >= n_staged) return;
  for (uint32_t i = ctid - j * n_present; i < n_present; i += (W * 32)) {
    const uint32_t w0 = list[i], e1 = list[i + 1] >> 16;
    float* const row = acc + (w0 & 0xFFFFu) * acc_stride;
    for (uint32_t e = w0 >> 16; e < e1; e += kGather) {
      uint32_t en[kGather];
#pragma unroll
      for (uint32_t u = 0; u < kGather; ++u) en[u] = ent[min(e + u, e1 - 1)];
      if (NPOL == 1 || q_at)
        GatherEntries<NCORR, NPOL, RUNS, true>(en, e1 - e, gtab_at, gain_stride * 8, stg_at, q_at,
                                               row, n_dir, d0, j, step, n_staged);
      else
        GatherEntries<NCORR, NPOL, RUNS, false>(en, e1 - e, gtab_at, gain_stride * 8, stg_at, 0,
                                                row, n_dir, d0, j, step, n_staged);
    }
  }
}

// NG lanes per run (1, 2, 4 or 8): a tile has (W * 32) / NG runs and
// lane g of a run owns directions g, g + NG, ... (DPL of them); the residual
// is the sum over the run's lanes (warp shuffles). NG = 1: one run per lane,
// exactly DPL directions.
// Launched cooperatively (all CTAs co-resident), one CTA per SM.
// Bound: HBM while rows stream, and latency in the end of a pass. 11 consumer
// warps of at most DPL = 5 directions a lane, in 168 registers, cover each
// other's latencies: a 30 KB row (62 stations, 10 directions) takes 0.66 us, the
// time of its copy, a tile's reduction 2.7 us; 7 warps of up to 10 directions a
// lane took 6.8 us for the reduction. Several passes in one launch, the ring
// filling while the grid finalises: 50 passes over 24 channel blocks of 80 rows
// (240 channels, 8 times) 6.27 -> 5.41 ms, over 12 blocks of 20 rows 2.13 -> 1.05.
// SUMQ: the model powers are summed in the row loop (else precomputed).
constexpr int kPairValues = 6;  // model values per lane up to which two rows fit its registers
// Of a lane's directions, staged at a time: all; in the wide variant of more
// than kPipeDirs2 three (40 directions take 101 KB of accumulators and gains), and
// of up to five with P and Q of two polarizations half of them. 512 stations, 16
// directions, one polarization, 8 rows a tile: 214 us a pass in two rounds, 202
// in one.
__host__ __device__ constexpr int StageDirs(int warps, int dpl, int npol, bool sumq) {
  if (warps != kWideWarps) return 8;
  return dpl > int(kPipeDirs2) ? 3 : npol == 1 || !sumq ? dpl : (dpl + 1) / 2;
}
// Where a staging area of their own would leave a ring of fewer than three
// stages, the sums are staged in the ring stage of the tile's last row
// (PipeLayout::hold), as many directions at a time as it holds: on the variants
// whose large arrays come to that and gain by it, all with two correlations (one
// polarization and one lane per run: 900 stations, 5 directions 162 us a pass,
// 159 on two lanes).
__host__ __device__ constexpr bool MayHold(int warps, int ncorr, int npol, int ng) {
  return warps == kWideWarps || (ncorr == 2 && npol == 2 && ng == 1);
}
__host__ __device__ constexpr int HeldDirs(int dpl, int npol, bool sumq) {
  if (dpl > int(kPipeDirs2)) return 3;
  return npol == 1 || !sumq || dpl == 1 ? dpl : dpl == 2 ? 1 : (dpl + 1) / 2;
}
__host__ __device__ constexpr uint32_t StagedBytes(uint32_t staged, uint32_t runs, uint32_t ncorr,
                                                   uint32_t npol) {  // of P
  return staged * runs * (npol == 1 ? 1u : ncorr) * 8u;
}
template <int NCORR, int NPOL, int DPL, int NG, bool SUMQ, int W>
__global__ void __launch_bounds__(W * 32 + 32, 1) pipe_kernel(const PipeParams p) {
  static_assert(32 % NG == 0, "lanes per run must divide a warp");
  constexpr int RUNS = (W * 32) / NG;  // runs per tile
  extern __shared__ __align__(128) unsigned char smem[];
  PipeShared& sh = *reinterpret_cast<PipeShared*>(smem);
  uint64_t* full = sh.full;
  uint64_t* empty = sh.empty;
  uint64_t* gfull = sh.gfull;
  uint64_t* gfree = sh.gfree;
  uint64_t* mfree = sh.mfree;
  float* acc = reinterpret_cast<float*>(smem + p.off_acc);
  float2* gtab_buf = reinterpret_cast<float2*>(smem + p.off_gtab);
  constexpr int kStage = StageDirs(W, DPL, NPOL, SUMQ);
  constexpr int kHeldStage = HeldDirs(DPL, NPOL, SUMQ);
  constexpr bool kMayHold = MayHold(W, NCORR, NPOL, NG);
  const bool hold = kMayHold && p.hold != 0;
  uint32_t* metas = reinterpret_cast<uint32_t*>(smem + p.off_meta);
  char* stages = reinterpret_cast<char*>(smem + p.off_stages);
  constexpr uint32_t E = NCORR * 8;  // bytes per visibility
  const uint32_t acc_n = p.acc_floats;
  const uint32_t n_dir = NG == 1 ? uint32_t(DPL) : p.n_dir;
  const uint32_t stage_bytes = (1 + n_dir) * RUNS * E;  // data, model 0, ...
  const uint32_t table_bytes = p.table_f2 * 8;
  const uint32_t S = p.stages;

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  if (tid == 0) {
    for (uint32_t s = 0; s < S; ++s) {
      MbarInit(&full[s], 1);
      MbarInit(&empty[s], W);
    }
    for (int b = 0; b < 2; ++b) {
      MbarInit(&gfull[b], 1);
      MbarInit(&gfree[b], W);
      MbarInit(&mfree[b], W);
    }
    MbarInit(&sh.flushed, 1);
    MbarInit(&sh.finalised, 1);
    MbarInit(&sh.ready, 1);
    sh.err = 0;
    sh.stop = 0;
    sh.passes = 0;
    sh.params = p;
    // A solve may be several launches (of so many iterations, or the
    // unrolled body of a constrained solve's graph): a launch after the solve
    // has stopped, or after an error, does nothing. One thread looks: the
    // error may be flagged while it does, and the warps have to agree.
    bool skip = static_cast<volatile uint32_t*>(p.counters)[kCntError] != 0;
    if (!p.host_mode && !skip) {
      skip = true;
      for (uint32_t g = 0; g < p.n_groups && skip; ++g)
        skip = static_cast<volatile const LoopState*>(p.state)[g].done != 0;
    }
    sh.skip = skip ? 1u : 0u;
    // The counters before this launch. Those of finished passes and control
    // steps cannot move before this CTA has arrived at its first grid barrier;
    // other CTAs may have arrived there once each already.
    sh.epoch0 = LoadAcquire(&p.counters[kCntEpoch]);
    const uint64_t final_now =
        LoadAcquire64(reinterpret_cast<const uint64_t*>(p.counters + kCntFinal));
    sh.final0 = uint32_t(final_now);
    sh.bad_seen = uint32_t(final_now >> 32);
    const uint32_t arrived = LoadAcquire(&p.counters[kCntArrive]);
    sh.arrive0 = arrived - arrived % gridDim.x;
    sh.verdict = kVerdictNear;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    if (!skip && p.use_handle && blockIdx.x == 0) cudaGraphSetConditional(p.handle, 0);
  }
  __syncthreads();
  if (sh.skip) return;

  const uint32_t f_begin = p.cta_frag_off[blockIdx.x];
  const uint32_t f_end = p.cta_frag_off[blockIdx.x + 1];

  if (warp == W) {
    // ---------------- producer warp: one thread issues all bulk copies ----
    // The visibilities do not depend on the solutions, so the next pass's
    // first rows are fetched while the grid finalises this one, into the ring
    // as its stages fall free. Only the gain tables (one per visit) wait for
    // the pass to be finished.
    if (lane != 0) return;
    uint32_t row = 0, nvis = 0, nfrag = 0;
    uint32_t st = 0, ph = 0;  // stage of `row` and the parity of its use
    bool ok = true;
    for (uint32_t it = 0; it < p.n_iters && ok; ++it) {
      bool tables_ready = it == 0;
      const uint32_t row0 = row, nfrag0 = nfrag;  // first row and fragment of the pass
      uint32_t cur_visit = 0xFFFFFFFFu;
      uint32_t pending = 0xFFFFFFFFu;  // gain table not asked for yet
      // The pending gain table, once the solutions of the pass are final;
      // false when the launch ends instead (or a wait gave up).
      auto fetch_table = [&]() {
        if (!tables_ready) {
          const uint64_t t0 = GlobalTimerNs();
          for (uint32_t n = 1; sh.passes < it; ++n) {
            if (sh.err) return false;
            if ((n & 63u) == 0 && GlobalTimerNs() - t0 > p.wait_ns) {
              sh.err = 1;
              atomicExch(&p.counters[kCntError], 1u);
              return false;
            }
          }
          if (sh.stop) return false;
          __threadfence();
          FenceProxyAsync();
          tables_ready = true;
        }
        if (pending == 0xFFFFFFFFu) return true;
        const uint32_t b = nvis % p.n_gbuf;
        const uint32_t use = nvis / p.n_gbuf;  // earlier uses of buffer b
        if (use >= 1 && !PipeWait(&gfree[b], (use - 1) & 1u, sh))
          return false;
        MbarArriveExpectTx(&gfull[b], table_bytes);
        BulkCopyG2S(gtab_buf + size_t(b) * p.table_f2, p.tables + size_t(pending) * p.table_f2,
                    table_bytes, &gfull[b]);
        pending = 0xFFFFFFFFu;
        ++nvis;
        return true;
      };
      // With several intervals the fragments of the pass depend on which
      // intervals go on: nothing is fetched before that is known.
      if (p.n_groups > 1 && !fetch_table()) break;
      for (uint32_t fi = f_begin; fi < f_end && ok; ++fi) {
        const Frag f = p.frags[fi];
        if (FragFrozen(p, f.slab)) continue;
        const SlabDesc sl = p.slabs[f.slab];
        if (f.visit != cur_visit) {  // new visit: its gain table first
          if (pending != 0xFFFFFFFFu && !fetch_table()) {
            ok = false;
            break;
          }
          pending = sl.table;
          cur_visit = f.visit;
          if (tables_ready && !fetch_table()) {
            ok = false;
            break;
          }
        }
        // The fragment's tile is one tile of the packed slab: a row of it,
        // data and all directions, is one contiguous block.
        const uint32_t seg = (1 + n_dir) * f.n_runs * E;
        const size_t row_step = size_t(sl.R) * (1 + n_dir) * E;
        const char* src = static_cast<const char*>(sl.vis) + size_t(f.row_lo) * row_step +
                          size_t(f.r0) * (1 + n_dir) * E;
        // The next stage, free: a ring full of rows whose gain table is
        // still pending cannot move before it.
        auto take_stage = [&]() {
          if (pending != 0xFFFFFFFFu && row - row0 >= S && !fetch_table()) return false;
          return row < S || PipeWait(&empty[st], ph ^ 1u, sh);
        };
        // The antenna buffer of the fragment before the last, which (like the
        // ring) is not released before its gain table has arrived.
        if (pending != 0xFFFFFFFFu && nfrag - nfrag0 >= 2 && !fetch_table()) {
          ok = false;
          break;
        }
        if (nfrag >= 2 && !PipeWait(&mfree[nfrag & 1u], (nfrag / 2 - 1) & 1u, sh)) {
          ok = false;
          break;
        }
        for (uint32_t rr = f.row_lo; rr < f.row_hi; ++rr, ++row) {
          if (!take_stage()) {
            ok = false;
            break;
          }
          // The tile's antennas travel with the fragment's first row.
          const uint32_t mb = rr == f.row_lo ? f.meta_bytes : 0u;
          MbarArriveExpectTx(&full[st], seg + mb);
          if (mb) {
            BulkCopyG2S(metas + (nfrag & 1u) * p.meta_words, p.metas + size_t(f.meta) * 4, mb,
                        &full[st]);
            ++nfrag;
          }
          BulkCopyG2S(stages + size_t(st) * stage_bytes, src, seg, &full[st]);
          src += row_step;
          if (++st == S) {
            st = 0;
            ph ^= 1u;
          }
        }
        if (ok && (f.flags & kFragPower)) {
          // one more stage: the tile's model powers [dir][run][corr]
          if (!take_stage()) {
            ok = false;
            break;
          }
          const uint32_t pb = n_dir * NCORR * RUNS * 4;
          MbarArriveExpectTx(&full[st], pb);
          BulkCopyG2S(stages + size_t(st) * stage_bytes,
                      p.powers + size_t(f.tile) * p.power_floats, pb, &full[st]);
          ++row;
          if (++st == S) {
            st = 0;
            ph ^= 1u;
          }
        }
      }
      if (ok && pending != 0xFFFFFFFFu) ok = fetch_table();
      // a CTA without fragments still follows the passes
      if (ok && !tables_ready) ok = fetch_table();
    }
    // Wait for the last copies, so none is in flight when the CTA ends.
    for (uint32_t k = 0; k < S && k < row; ++k) {
      const uint32_t r = row - 1 - k;
      PipeWait(&full[r % S], (r / S) & 1u, sh);
    }
    for (uint32_t k = 0; k < p.n_gbuf && k < nvis; ++k) {
      const uint32_t v = nvis - 1 - k;
      PipeWait(&gfull[v % p.n_gbuf], (v / p.n_gbuf) & 1u, sh);
    }
    return;
  }

  // ---------------- consumer warps ----------------
  uint32_t nvis = 0, cur_visit = 0xFFFFFFFFu, nfrag = 0;
  uint32_t st = 0, ph = 0;  // stage of the next row and the parity of its use
  const float2* gtab = gtab_buf;
  for (uint32_t it = 0; it < p.n_iters; ++it) {
    // (the lane's constants, recomputed every pass: carried through the end of
    // the pass they would spill the row loop, 0.6 us a row became 1.1 us)
    const int ctid = FreshTid();  // 0 .. W * 32 - 1
    const int warp = ctid >> 5, lane = ctid & 31;
    // A warp holds 32 / NG runs; lane g * (32 / NG) + i serves run i of the
    // warp for directions g, g + NG, ...: the 8 lanes of a quarter warp read 8
    // consecutive runs of one direction row (NG = 8: 4 runs of two rows), in
    // distinct shared-memory banks.
    constexpr int kRunsPerWarp = 32 / NG;
    const int run = warp * kRunsPerWarp + lane % kRunsPerWarp;  // run within the tile
    const int g = lane / kRunsPerWarp;  // the lane's first direction
    // Every lane has its first DPL - 1 directions; the last one of some lanes
    // is past the end (n_dir > (DPL - 1) NG): they read the last direction with
    // zero gains and drop its sums.
    const bool last_mine = uint32_t(g + (DPL - 1) * NG) < n_dir;
    const uint32_t last_row = min(uint32_t(g + (DPL - 1) * NG), n_dir - 1) - uint32_t(g);
    auto end_visit = [&]() {
      // all consumers are done with the visit: release its gain table buffer
      // and flush the accumulators into the visit's partial slot
      ConsumerBarrier<W>();
      if (lane == 0) MbarArrive(&gfree[(nvis - 1) % p.n_gbuf]);
      float4* out = reinterpret_cast<float4*>(p.partials + size_t(cur_visit) * acc_n);
      const float4* src = reinterpret_cast<const float4*>(acc);
      for (uint32_t i = ctid; i < acc_n / 4; i += (W * 32)) __stcg(out + i, src[i]);
    };
    cur_visit = 0xFFFFFFFFu;
    for (uint32_t fi = f_begin; fi < f_end; ++fi) {
      // (what is needed of the descriptor, read when it is: it is in L1 after
      // the first pass, and a register held through the row loop costs more)
      const Frag& f = p.frags[fi];
      if (FragFrozen(p, f.slab)) continue;
      if (f.visit != cur_visit) {
        if (cur_visit != 0xFFFFFFFFu) {
          end_visit();
          ConsumerBarrier<W>();  // the accumulators are flushed
        }
        float4* z = reinterpret_cast<float4*>(acc);
        for (uint32_t i = ctid; i < acc_n / 4; i += (W * 32))
          z[i] = make_float4(0.f, 0.f, 0.f, 0.f);
        const uint32_t b = nvis % p.n_gbuf;
        PipeWait(&gfull[b], (nvis / p.n_gbuf) & 1u, sh);
        gtab = gtab_buf + size_t(b) * p.table_f2;
        cur_visit = f.visit;
        ++nvis;
      }
      const uint32_t* meta = metas + (nfrag & 1u) * p.meta_words;
      const uint32_t n_runs = f.n_runs, flags = f.flags;
      const bool active = uint32_t(run) < n_runs;
      const bool warp_busy = uint32_t(warp) * kRunsPerWarp < n_runs;
      // the run's data in a stage, its first direction's model, and the step
      // to the lane's next one and to its last one
      const uint32_t off_d = uint32_t(run) * E, pitch = n_runs * E;
      const uint32_t off_m = off_d + (1 + g) * pitch, step_m = NG * pitch;
      const uint32_t off_l = off_m + last_row * pitch;
      float2 G[DPL][NCORR];
      float2 P[DPL][NCORR];
      float Q[SUMQ ? DPL : 1][NCORR];
#pragma unroll
      for (int k = 0; k < DPL; ++k)
#pragma unroll
        for (int c = 0; c < NCORR; ++c) {
          P[k][c] = make_float2(0.f, 0.f);
          if constexpr (SUMQ) Q[k][c] = 0.f;
        }
      const uint32_t n_rows = f.row_hi - f.row_lo;
      PipeWait(&full[st], ph, sh);
      if (warp_busy) {  // with the first row: the run's antennas, gain products
        const uint32_t ap = active ? meta[kMetaRuns + run] : 0u;
        const uint32_t a1 = ap & 0xFFFFu, a2 = ap >> 16;
#pragma unroll
        for (int k = 0; k < DPL; ++k) {
          float2 ga[NPOL], gb[NPOL];
#pragma unroll
          for (int q = 0; q < NPOL; ++q) {
            ga[q] = make_float2(0.f, 0.f);
            gb[q] = make_float2(0.f, 0.f);
          }
          if (k < DPL - 1 || last_mine) {
            LoadGains<NPOL>(gtab, a1, p.gain_stride, g + k * NG, ga);
            LoadGains<NPOL>(gtab, a2, p.gain_stride, g + k * NG, gb);
          }
#pragma unroll
          for (int c = 0; c < NCORR; ++c)
            G[k][c] = cmul_conj(ga[RowPol<NCORR, NPOL>(c)], gb[ColPol<NCORR, NPOL>(c)]);
        }
      }
      uint32_t rr = 0;
      // NR rows at once: the dependent steps of one row (load, residual,
      // shuffles, sums) fill the latencies of the other's.
      auto rows = [&](auto nr) {
        constexpr int NR = decltype(nr)::value;
        // the model row stays in registers between the residual and the sums,
        // or is read twice where it does not fit beside them
        constexpr bool kKeep = DPL <= int(kPipeDirs2);
        uint32_t stage[NR];
#pragma unroll
        for (int i = 0; i < NR; ++i) {
          PipeWait(&full[st], ph, sh);
          stage[i] = st;
          if (++st == S) {
            st = 0;
            ph ^= 1u;
          }
        }
        // Warps without runs in this tile only release the stages.
        if (warp_busy) {
          // Residual R = D - sum_d G_d M_d, then P_d += R conj(M_d) and
          // (SUMQ) Q_d += |M_d|^2. With NG > 1 each lane sums its own
          // directions' terms and the run's lanes then add theirs up
          // (shuffles) before D is added.
          float2 R[NR][NCORR], M[NR][kKeep ? DPL : 1][NCORR], D[NR][NCORR];
          auto model = [&](int i, int k, float2 (&m)[NCORR]) {
            LoadVisShared<NCORR>(stages + stage[i] * stage_bytes +
                                     (k < DPL - 1 ? off_m + k * step_m : off_l),
                                 0, m);
          };
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            if constexpr (kKeep) {
#pragma unroll
              for (int k = 0; k < DPL; ++k) model(i, k, M[i][k]);
            }
            LoadVisShared<NCORR>(stages + stage[i] * stage_bytes + off_d, 0, D[i]);
          }
#pragma unroll
          for (int i = 0; i < NR; ++i) {
            // (in two halves, to halve the chain of dependent multiply-adds)
            float2 h[2][NCORR];
#pragma unroll
            for (int c = 0; c < NCORR; ++c) {
              h[0][c] = NG == 1 ? D[i][c] : make_float2(0.f, 0.f);
              h[1][c] = make_float2(0.f, 0.f);
            }
#pragma unroll
            for (int k = 0; k < DPL; ++k) {
              float2 m[NCORR];
              if constexpr (kKeep) {
#pragma unroll
                for (int c = 0; c < NCORR; ++c) m[c] = M[i][k][c];
              } else {
                model(i, k, m);
              }
#pragma unroll
              for (int c = 0; c < NCORR; ++c) {
                float2& r = h[k & 1][c];
                r.x = fmaf(-G[k][c].x, m[c].x, r.x);
                r.x = fmaf(G[k][c].y, m[c].y, r.x);
                r.y = fmaf(-G[k][c].x, m[c].y, r.y);
                r.y = fmaf(-G[k][c].y, m[c].x, r.y);
              }
            }
#pragma unroll
            for (int c = 0; c < NCORR; ++c)
              R[i][c] =
                  DPL > 1 ? make_float2(h[0][c].x + h[1][c].x, h[0][c].y + h[1][c].y) : h[0][c];
          }
          if constexpr (NG > 1) {
#pragma unroll
            for (int m = kRunsPerWarp; m < 32; m <<= 1)
#pragma unroll
              for (int i = 0; i < NR; ++i)
#pragma unroll
                for (int c = 0; c < NCORR; ++c) {
                  R[i][c].x += __shfl_xor_sync(0xFFFFFFFFu, R[i][c].x, m);
                  R[i][c].y += __shfl_xor_sync(0xFFFFFFFFu, R[i][c].y, m);
                }
#pragma unroll
            for (int i = 0; i < NR; ++i)
#pragma unroll
              for (int c = 0; c < NCORR; ++c) {
                R[i][c].x += D[i][c].x;
                R[i][c].y += D[i][c].y;
              }
          }
#pragma unroll
          for (int k = 0; k < DPL; ++k)
#pragma unroll
            for (int i = 0; i < NR; ++i) {
              float2 mk[NCORR];
              if constexpr (kKeep) {
#pragma unroll
                for (int c = 0; c < NCORR; ++c) mk[c] = M[i][k][c];
              } else {
                model(i, k, mk);
              }
#pragma unroll
              for (int c = 0; c < NCORR; ++c) {
                const float2 m = mk[c], r = R[i][c];
                P[k][c].x = fmaf(r.x, m.x, P[k][c].x);
                P[k][c].x = fmaf(r.y, m.y, P[k][c].x);
                P[k][c].y = fmaf(r.y, m.x, P[k][c].y);
                P[k][c].y = fmaf(-r.x, m.y, P[k][c].y);
                if constexpr (SUMQ) {
                  Q[k][c] = fmaf(m.x, m.x, Q[k][c]);
                  Q[k][c] = fmaf(m.y, m.y, Q[k][c]);
                }
              }
            }
        }
        __syncwarp();
        // (a held last row's stage is released after the reduction)
        if (lane == 0 && !(hold && rr + NR == n_rows)) {
#pragma unroll
          for (int i = 0; i < NR; ++i) MbarArrive(&empty[stage[i]]);
        }
      };
      if constexpr (DPL * NCORR <= kPairValues)
        if (S >= 4)  // (a shorter ring would run dry)
          for (; rr + 2 <= n_rows; rr += 2) rows(std::integral_constant<int, 2>{});
      for (; rr < n_rows; ++rr) rows(std::integral_constant<int, 1>{});

      // ---- tile reduction into the visit's antenna accumulators ----
      // The lanes stage their runs' sums; then one thread per (direction,
      // antenna of the tile) adds up that antenna's runs, in the fixed order
      // of the tile's entry list, and updates the accumulator once. Two
      // barriers and no read-modify-write chains, whatever the runs' order.
      uint32_t q_src = 0;  // none, or at [dir][run][corr] (SUMQ: of the staged ones)
      uint32_t q_stage = 0;
      const uint32_t held = st == 0 ? S - 1 : st - 1;  // the last row's stage
      constexpr int kFewest = (DPL - 1) * NG + 1;  // directions of this variant
      static_assert(!kMayHold || (kHeldStage < DPL ? kHeldStage * NG : kFewest) *
                            (NPOL == 1 ? 12 : SUMQ ? 12 * NCORR : 8 * NCORR) <=
                        (1 + kFewest) * int(E),
                    "the staged sums must fit in a held stage");
      const uint32_t stg_at =
          hold ? SmemAddr(stages + held * stage_bytes) : SmemAddr(smem) + p.off_stg;
      const uint32_t stg_q_at =
          hold ? stg_at + StagedBytes(min(uint32_t(kHeldStage * NG), n_dir), RUNS, NCORR, NPOL)
               : SmemAddr(smem) + p.off_q;
      if (flags & kFragPower) {
        // the tile's precomputed model powers, in the stage after its rows
        q_stage = st;
        PipeWait(&full[st], ph, sh);
        if (++st == S) {
          st = 0;
          ph ^= 1u;
        }
        q_src = SmemAddr(stages + q_stage * stage_bytes);
      } else if (SUMQ) {
        q_src = stg_q_at;
      }
      float4* const stg = SharedPtr<float4>(stg_at);
      float2* const stg_q = SharedPtr<float2>(stg_q_at);
      auto reduce = [&](auto at_a_time) {
        constexpr int KS = decltype(at_a_time)::value;
#pragma unroll
        for (int k0 = 0; k0 < DPL; k0 += KS) {
          ConsumerBarrier<W>();  // the previous reduction is complete everywhere
          if (active) {
#pragma unroll
            for (int k = k0; k < DPL && k < k0 + KS; ++k) {
              const uint32_t j = g + (k - k0) * NG;  // staged direction k0 * NG + j
              if (k < DPL - 1 || last_mine) {
                if constexpr (NPOL == 1) {
                  float3 v = make_float3(0.f, 0.f, 0.f);
#pragma unroll
                  for (int c = 0; c < NCORR; ++c) {
                    v.x += P[k][c].x;
                    v.y += P[k][c].y;
                    if constexpr (SUMQ) v.z += Q[k][c];
                  }
                  if (!SUMQ && q_src) {
                    const float* q =
                        SharedPtr<const float>(q_src) + ((g + k * NG) * RUNS + run) * NCORR;
#pragma unroll
                    for (int c = 0; c < NCORR; ++c) v.z += q[c];
                  }
                  reinterpret_cast<float2*>(stg)[j * RUNS + run] = make_float2(v.x, v.y);
                  reinterpret_cast<float*>(stg_q)[j * RUNS + run] = v.z;
                } else {
#pragma unroll
                  for (int h = 0; h < NCORR / 2; ++h)
                    stg[(j * RUNS + run) * (NCORR / 2) + h] = make_float4(
                        P[k][2 * h].x, P[k][2 * h].y, P[k][2 * h + 1].x, P[k][2 * h + 1].y);
                  if constexpr (SUMQ) {
#pragma unroll
                    for (int h = 0; h < NCORR / 2; ++h)
                      stg_q[(j * RUNS + run) * (NCORR / 2) + h] =
                          make_float2(Q[k][2 * h], Q[k][2 * h + 1]);
                  }
                }
              }
            }
          }
          ConsumerBarrier<W>();
          const uint32_t d0 = k0 * NG;
          const uint32_t n_staged = min(uint32_t(KS * NG), n_dir - d0);
          const uint32_t q_from = NPOL == 1          ? stg_q_at
                                  : q_src && !SUMQ ? q_src + d0 * NCORR * RUNS * 4
                                                   : q_src;
          GatherTile<W, NCORR, NPOL, RUNS>(SmemAddr(meta), SmemAddr(gtab), stg_at, q_from,
                                        SmemAddr(acc), ctid, n_dir, d0, n_staged, p.acc_stride,
                                        p.gain_stride);
        }
      };
      if constexpr (kMayHold && kHeldStage < DPL && kHeldStage < kStage) {
        if (hold)
          reduce(std::integral_constant<int, kHeldStage>{});
        else
          reduce(std::integral_constant<int, kStage>{});
      } else {
        reduce(std::integral_constant<int, kStage>{});
      }
      // (this thread's sums in the held stage, before a copy overwrites them)
      if (hold) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      __syncwarp();
      if (lane == 0) {
        if (hold) MbarArrive(&empty[held]);
        if (flags & kFragPower) MbarArrive(&empty[q_stage]);
        MbarArrive(&mfree[nfrag & 1u]);
      }
      ++nfrag;
    }
    if (cur_visit != 0xFFFFFFFFu) end_visit();
    if (!EndPass<W, NPOL>(SmemAddr(smem), it)) break;
  }
}

// The assignment pass of a constrained iteration on the pipelined path
// (fin_mode = kFinAssignOnly): FinalizeDistributed over the constrained next
// solutions, with kWarps warps per CTA (its barriers span them) and
// the CTA count of pipe_kernel (its norm partials); the last CTA to arrive
// runs the control step.
template <int NPOL>
__global__ void __launch_bounds__(kWarps * 32) assign_kernel(const PipeParams p) {
  constexpr int W = kWarps;
  if (p.use_handle && static_cast<volatile const LoopState*>(p.state)->done) return;
  __shared__ double s_sum[W];
  __shared__ uint32_t s_cnt[2 * W];
  __shared__ uint32_t s_flag[2];
  const int ctid = int(threadIdx.x);
  bool bad;
  FinalizeDistributed<W, NPOL>(p, 0, ctid, s_sum, s_cnt, bad, []() { return true; });
  auto* final = reinterpret_cast<unsigned long long*>(p.counters + kCntFinal);
  if (ctid == 0) {
    __threadfence();
    const unsigned long long one = 1ull | (bad ? 1ull << 32 : 0ull);
    const unsigned long long count = atomicAdd(final, one) + one;
    // (a multiple of the grid between launches; the high half starts at zero)
    s_flag[0] = uint32_t(count) % gridDim.x == 0 ? 1u : 0u;
    s_flag[1] = uint32_t(count >> 32);
  }
  ConsumerBarrier<W>();
  if (!s_flag[0]) return;
  __threadfence();
  const bool any_bad = s_flag[1] != 0;
  const uint32_t v = ControlPass<W, NPOL>(p, ctid, any_bad, s_sum, s_cnt, s_flag);
  if (ctid == 0) {
    if (any_bad) atomicAnd(final, 0xFFFFFFFFull);
    if (p.use_handle) cudaGraphSetConditional(p.handle, v & kVerdictStop ? 0u : 1u);
  }
}

}  // namespace
