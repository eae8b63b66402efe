// pipe_kernel, wide variant, 2 correlations, 2 solution polarizations.
#include "pipe_entries.cuh"

void ddsolve_impl::AddWide22(std::vector<KernelEntry>& k) { AddWide<2>(k, WideDirections{}); }
