// pipe_kernel, 2 correlations, 2 solution polarizations.
#include "pipe_entries.cuh"

void ddsolve_impl::AddPipe22(std::vector<KernelEntry>& k) { AddLanes<2, 2, 1, 2, 4>(k); }
