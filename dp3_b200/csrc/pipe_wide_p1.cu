// pipe_kernel, wide variant, 2 correlations, 1 solution polarization.
#include "pipe_entries.cuh"

void ddsolve_impl::AddWide21(std::vector<KernelEntry>& k) { AddWide<1>(k, WideDirections{}); }
