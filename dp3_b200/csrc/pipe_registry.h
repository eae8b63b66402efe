// The compiled variants of pipe_kernel. They are compiled apart from the other
// kernels, one source file (pipe_*.cu) per group: the code of a kernel does not
// depend on which variants exist, and a process loads the groups that it uses
// (one module of all kernels, optimised in parts on every core, changed the
// register allocation of unrelated kernels: the full-Jones solve of 62 stations
// and 4 directions took 15.67 ms against 15.39).
#pragma once

#include <vector>

namespace ddsolve_impl {

struct KernelEntry {
  int ncorr, npol, dmax;  // dmax: directions per lane (or thread)
  const void* fn;
  int ng = 1;  // pipe_kernel: lanes per run
  const void* fn_powers = nullptr;  // pipe_kernel: with precomputed model powers
  int warps = 0;                    // pipe_kernel: consumer warps
  const void* fn_alone = nullptr;   // stream_kernel: for one block per SM
};

// Correlations and solution polarizations; Wide: 13 directions and more, with
// kWideWarps.
void AddPipe22(std::vector<KernelEntry>& k);
void AddPipe21(std::vector<KernelEntry>& k);
void AddPipe42(std::vector<KernelEntry>& k);
void AddPipe41(std::vector<KernelEntry>& k);
void AddWide22(std::vector<KernelEntry>& k);
void AddWide21(std::vector<KernelEntry>& k);

}  // namespace ddsolve_impl
