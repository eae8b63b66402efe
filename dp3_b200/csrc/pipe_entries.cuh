// Registers variants of pipe_kernel (included by the pipe_*.cu files).
#pragma once

#include <utility>

#include "pipe_kernel.cuh"
#include "pipe_registry.h"

namespace {

using ddsolve_impl::KernelEntry;

template <int NC, int NP, int DM, int NG, int W = kWarps>
KernelEntry PipeEntry() {
  return KernelEntry{NC, NP, DM,
                     reinterpret_cast<const void*>(&pipe_kernel<NC, NP, DM, NG, true, W>), NG,
                     reinterpret_cast<const void*>(&pipe_kernel<NC, NP, DM, NG, false, W>), W};
}
template <int NC, int NP, int NG, int... DM>
void AddDirections(std::vector<KernelEntry>& k, std::integer_sequence<int, DM...>) {
  (k.push_back(PipeEntry<NC, NP, DM + 1, NG>()), ...);
}
// 1 to 5 directions a lane for two correlations, to 3 for four, on each count
// of lanes per run.
template <int NC, int NP, int... NG>
void AddLanes(std::vector<KernelEntry>& k) {
  using D = std::make_integer_sequence<int, int(NC == 2 ? kPipeDirs2 : kPipeDirs4)>;
  (AddDirections<NC, NP, NG>(k, D{}), ...);
}
// Four lanes per run of 4 directions (13 in all) to 12 each, fewer warps.
constexpr int kWideFrom = 4;
template <int NP, int... DM>
void AddWide(std::vector<KernelEntry>& k, std::integer_sequence<int, DM...>) {
  (k.push_back(PipeEntry<2, NP, kWideFrom + DM, 4, kWideWarps>()), ...);
}
using WideDirections = std::make_integer_sequence<int, kPipeDirsWide - kWideFrom + 1>;

}  // namespace
