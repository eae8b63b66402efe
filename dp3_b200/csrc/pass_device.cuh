// Device code that every streaming pass shares: plan structures, loop state,
// complex helpers, compensated sums, the control step of an iteration.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

namespace {

constexpr int kThreads = 256;
constexpr uint32_t kInvalidKey = 0xFFFFFFFFu;
constexpr uint32_t kMaxAntennas = 65535;
constexpr size_t kB200BlockSmem = 227 * 1024;  // shared memory a block may ask for

// ---------------------------------------------------------------------------
// Device-side plan structures
// ---------------------------------------------------------------------------
// A slab's visibilities, packed tile by tile: for every (time, channel) row,
// its runs are cut into tiles of W runs (the last one shorter), and a tile
// holds the data and then every direction's model for its runs,
//   [T][L][tile][1 + n_dir][runs of the tile],
// so that one row of one tile, with all its directions, is one contiguous
// block (one bulk copy of the pipelined kernel).
struct SlabDesc {
  const void* vis;          // data and model, packed as above
  const uint32_t* run_ant;  // [R] antenna1 | antenna2 << 16
  uint32_t cb, T, L, R;
  uint32_t W;        // runs per tile (a multiple of 4)
  uint32_t sol_off;  // first of n_dir entries in slab_sol
  uint32_t table;    // gain table of the slab (pipe_kernel)
};

// Element index in a packed slab of run r, row (t * L + l), and j = 0 for the
// data or 1 + d for direction d's model; nd1 = 1 + n_dir.
__host__ __device__ __forceinline__ uint64_t SlabElem(uint32_t R, uint32_t W, uint32_t nd1,
                                                      uint64_t row, uint32_t j, uint32_t r) {
  const uint32_t k = r / W;
  const uint32_t base = k * W;
  const uint32_t w = R - base < W ? R - base : W;
  return row * R * nd1 + uint64_t(base) * nd1 + uint64_t(j) * w + (r - base);
}

// pipe_kernel work item: rows [row_lo, row_hi) of the (t, channel) rows of
// the tile of runs [r0, r0 + n_runs) of a slab; fragments of one CTA that
// share a slab form a visit (one partial slot). meta: the tile's antennas
// (TileMeta), first word / 4 and bytes.
struct Frag {
  uint32_t slab, r0, n_runs, flags, row_lo, row_hi, visit, tile, meta, meta_bytes, pad[2];
};
constexpr uint32_t kFragPower = 1u;  // the fragment adds its tile's precomputed
                                     // model powers sum |M|^2 (one per tile)

struct Visit {
  uint32_t slab, run_lo, run_hi, pad;
};

struct DevSettings {
  uint32_t max_iterations;
  uint32_t min_iterations;
  double accuracy;
  double constraint_accuracy;
  double step_size;
  int32_t detect_stalling;
  int32_t phase_only;
  double step_diff_sigma;
  uint32_t hard_cap;
  uint32_t pad;
};

struct LoopState {
  uint32_t iteration;
  int32_t done;
  int32_t has_converged;
  int32_t has_stalled;
  uint32_t n_var_count;
  uint32_t blocks_done;
  double step_mean;
  double step_var;
};

struct StreamParams {
  const SlabDesc* slabs;
  const Visit* visits;
  const uint32_t* cta_visit_off;
  const uint32_t* slab_sol;
  const double2* solutions;
  float* partials;
  uint32_t n_ant, n_dir, n_sub, ng;
};

// Finalisation modes of a solve iteration. Fused: merge, FP64 division,
// SolverBase::Step, AssignSolutions and the iteration control in one pass.
// With device constraints the iteration is split around them
// (IterativeDiagonalSolver.cc:77-83: Step, ApplyConstraints, AssignSolutions):
// StepOnly writes the stepped next solutions to next_out and stops there;
// AssignOnly reads the constrained next solutions from next_out and does the
// rest (norm, solutions, gain tables, non-finite flags, control).
constexpr int32_t kFinFused = 0;
constexpr int32_t kFinStepOnly = 1;
constexpr int32_t kFinAssignOnly = 2;

struct FinParams {
  const float* partials;
  const uint32_t* fin_off;     // [n_cb * n_sub + 1]
  const uint32_t* fin_visits;  // visit indices
  const uint32_t* dir_of_sub;  // [n_sub]
  double2* solutions;          // [n_cb][n_ant][n_sub][NPOL]
  double2* next_out;           // host mode output; the constrained passes' buffer
  uint32_t n_cb, n_ant, n_dir, n_sub;
  int32_t host_mode;
  int32_t fin_mode;            // FinFused / FinStepOnly / FinAssignOnly
  const DevSettings* settings;
  double* block_sum;
  uint32_t* block_cnt;
  LoopState* state;
  uint32_t* nonfinite;  // [n_cb]
  double* step_magnitudes;
  cudaGraphConditionalHandle handle;
  int32_t use_handle;
  // independent solution intervals (groups of channel blocks): finalisation
  // block b covers items [block_item0[b], block_item_end[b]) of interval
  // block_group[b]; interval g owns blocks [group_blocks[g], group_blocks[g+1])
  // and its loop state state[g] and step magnitudes step_magnitudes[g * mags_stride]
  const uint32_t* block_group;
  const uint32_t* block_item0;
  const uint32_t* block_item_end;
  const uint32_t* group_blocks;
  uint32_t n_groups;
  uint32_t mags_stride;
};

// ---------------------------------------------------------------------------
// Complex helpers (float2 / double2)
// ---------------------------------------------------------------------------
__device__ __forceinline__ float2 cmul(float2 a, float2 b) {
  return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 cmul_conj(float2 a, float2 b) {  // a*conj(b)
  return make_float2(fmaf(a.x, b.x, a.y * b.y), fmaf(a.y, b.x, -a.x * b.y));
}
__device__ __forceinline__ float2 cconj(float2 a) {
  return make_float2(a.x, -a.y);
}
__device__ __forceinline__ float cnorm(float2 a) {
  return fmaf(a.x, a.x, a.y * a.y);
}

// Polarization of the row (left gain) and column (right gain) of correlation
// c. NCORR = 4 is the row-major 2x2 [XX XY; YX YY]; NCORR = 2 is XX/YY; a
// scalar solution (NPOL = 1) applies one gain to every correlation.
template <int NCORR, int NPOL>
__device__ __forceinline__ constexpr int RowPol(int c) {
  return NPOL == 1 ? 0 : (NCORR == 4 ? (c >> 1) : c);
}
template <int NCORR, int NPOL>
__device__ __forceinline__ constexpr int ColPol(int c) {
  return NPOL == 1 ? 0 : (NCORR == 4 ? (c & 1) : c);
}

template <int NCORR>
__device__ __forceinline__ void LoadVis(const void* base, size_t idx,
                                        float2 (&v)[NCORR]) {
  if constexpr (NCORR == 1) {
    v[0] = __ldg(reinterpret_cast<const float2*>(base) + idx);
  } else if constexpr (NCORR == 2) {
    const float4 x = __ldg(reinterpret_cast<const float4*>(base) + idx);
    v[0] = make_float2(x.x, x.y);
    v[1] = make_float2(x.z, x.w);
  } else {
    const float4* p = reinterpret_cast<const float4*>(base) + 2 * idx;
    const float4 x = __ldg(p);
    const float4 y = __ldg(p + 1);
    v[0] = make_float2(x.x, x.y);
    v[1] = make_float2(x.z, x.w);
    v[2] = make_float2(y.x, y.y);
    v[3] = make_float2(y.z, y.w);
  }
}

// Sums and FP64 complex helpers of the finalisation; one iteration's control.
struct NeumaierSum {  // compensated FP32 summation (two-sum)
  float s = 0.f, c = 0.f;
  __device__ __forceinline__ void Add(float x) {
    const float t = s + x;
    if (fabsf(s) >= fabsf(x))
      c += (s - t) + x;
    else
      c += (x - t) + s;
    s = t;
  }
  // Adds the sum of the lane `o` away (which adds this one).
  __device__ __forceinline__ void Join(uint32_t lanes, int o) {
    const float xs = __shfl_xor_sync(lanes, s, o), xc = __shfl_xor_sync(lanes, c, o);
    Add(xs);
    c += xc;
  }
  __device__ __forceinline__ float Value() const { return s + c; }
};

__device__ __forceinline__ double2 dmul(double2 a, double2 b) {
  return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ bool dfinite(double2 a) {
  return isfinite(a.x) && isfinite(a.y);
}
// 1 / s (Smith's algorithm), as std::complex<double> division does for
// finite operands.
__device__ __forceinline__ double2 dinv(double2 s) {
  if (fabs(s.x) >= fabs(s.y)) {
    const double r = s.y / s.x;
    const double den = s.x + s.y * r;
    return make_double2(1.0 / den, -r / den);
  } else {
    const double r = s.x / s.y;
    const double den = s.x * r + s.y;
    return make_double2(r / den, -1.0 / den);
  }
}

// One interval's AssignSolutions norm, stopping criterion and stall
// detection after an iteration whose norm sum / count are given; returns
// whether the interval stops.
__device__ bool ControlStep(LoopState& ls, const DevSettings& st, double sum, uint64_t cnt,
                            double* step_magnitudes) {
  // AssignSolutions (SolverBase.cc:297-306), no constraints: accuracy.
  const double mag = cnt == 0 ? 0.0 : sum / st.step_size / double(cnt);
  const uint32_t it = ls.iteration + 1;
  ls.iteration = it;
  if (it <= st.hard_cap) step_magnitudes[it - 1] = mag;
  const bool converged = mag <= st.accuracy;
  // ReachedStoppingCriterion / DetectStall (SolverBase.h:274-285,
  // SolverBase.cc:63-86)
  bool stalled = false;
  if (st.detect_stalling) {
    if (it == 1) {
      ls.n_var_count = 1;
      ls.step_mean = mag;
      ls.step_var = 0.0;
    } else {
      ls.n_var_count += 1;
      const double delta_1 = mag - ls.step_mean;
      ls.step_mean += delta_1 / double(ls.n_var_count);
      const double delta_2 = mag - ls.step_mean;
      ls.step_var += delta_1 * delta_2;
    }
    if (it >= 30)
      stalled = ls.step_mean <
                st.step_diff_sigma * sqrt(ls.step_var / double(ls.n_var_count));
  }
  const bool ready = it >= st.max_iterations || converged || stalled;
  const bool stop = (it >= st.min_iterations && ready) || it >= st.hard_cap;
  ls.has_converged = converged;
  ls.has_stalled = stalled;
  ls.done = stop;
  return stop;
}

}  // namespace
