// Entries of the node-indexed kappa array (khat: kappa of the element whose upper corner is the node).  The marched
// operator reads, past the last node, a plane of kappa above the last plane and, with two x-lines per lane, up
// to two lines more (rg_march.cuh); the gathering kernels a plane, a line and a node.  kCoefPad on top is for
// reads rounded up to whole groups.  No CUDA in here: a test enumerates the reads on the host.
#pragma once
#include <cstdint>

namespace rg {

constexpr int64_t kCoefPad = 1024;

inline int64_t khat_reach(int64_t n, int64_t nn0, int64_t nn1) { return n + nn0 * nn1 + 2 * nn0; }

}  // namespace rg
