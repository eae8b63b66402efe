// pipe_kernel, 4 correlations, 1 solution polarization.
#include "pipe_entries.cuh"

void ddsolve_impl::AddPipe41(std::vector<KernelEntry>& k) { AddLanes<4, 1, 1, 2, 4, 8>(k); }
