// Direct solver for K_AA of Beam_1 chains (elements e = 0..m-1 on nodes
// 2e, 2e+1, 2e+2; node-major DOF numbering), FP64, no pivoting.
//
// A midside node couples only to the two corner nodes of its element, so the
// solve eliminates
//   1. the midside node of every element (condensation): the element becomes a
//      "part", a stiffness between two corners and the forces it leaves on them;
//   2. corners, by merging pairs of neighbouring parts level by level, the last
//      levels of a chain in one CTA;
//   3. the last part with the chain's end nodes;
// and substitutes back in reverse.  The critical path is O(log m) small dense
// solves instead of the O(n) column recurrence of a banded LU, which on a GPU
// with slow FP64 latency (~64 cycles per dependent FP64 operation) dominates
// long chains.  The solver never reads an assembled K_AA: it takes each
// element's tangent K_e from the element scratch (plus the nodal load
// stiffness), which is the same K_AA term by term.  Corners may have fixed DOFs
// (a pinned end): their rows and columns are those of the identity.  Equations
// follow from block Gaussian elimination on the assembled matrix; the
// reference solves the same K_AA with PARDISO (reference
// src/SparseMatrix.cpp:74-166).
#pragma once
#include <cuda_runtime.h>

#include "gf_types.h"

namespace gf {

// Doubles per part and per kept elimination of the two kinds.
constexpr int CHAIN_SYM_PART = 57, CHAIN_SYM_KEEP = 81, CHAIN_GEN_PART = 156, CHAIN_GEN_KEEP = 78;

// Items below which an item per warp (half warp) is the faster form.  General: it
// takes 8 us for as many as there are sub-partitions (608), then 5.3 ns an item, an
// item per thread 98 us for anything up to 19,456 (its chain of 1,550 operations of
// 64 cycles).  Symmetric: 7 us for 1,216, then 3.1 ns, against 41 us for 16,000 and
// 55 us for 33,000.
constexpr int CHAIN_GEN_SMALL = 152 * 4 * 28, CHAIN_SYM_SMALL = 152 * 4 * 20;

// The chains of b.chain_gen (gf_chain.cu) and of b.chain_sym (gf_chain_sym.cu).
void launch_gen_chains(const Batch& b, const ChainParts& c, cudaStream_t st);
void launch_sym_chains(const Batch& b, const ChainParts& c, cudaStream_t st);
// Kernel launches of one solve.
inline int chain_launches(const ChainParts& c) { return c.n_elem ? 3 + 2 * c.n_levels : 0; }

}  // namespace gf
