// Test harness: the similarity bins of the row top-K.  Not part of the library.
#include "../../rabbitbin_b200/csrc/sim_bins.cuh"

extern "C" int host_bins() { return rbg::kBins; }
extern "C" int host_sim_bin(uint32_t bits) { return rbg::sim_bin(bits); }
