// pipe_kernel, 4 correlations, 2 solution polarizations.
#include "pipe_entries.cuh"

void ddsolve_impl::AddPipe42(std::vector<KernelEntry>& k) { AddLanes<4, 2, 1, 2, 4, 8>(k); }
