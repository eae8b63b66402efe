// pipe_kernel, 2 correlations, 1 solution polarization.
#include "pipe_entries.cuh"

void ddsolve_impl::AddPipe21(std::vector<KernelEntry>& k) { AddLanes<2, 1, 1, 2, 4>(k); }
