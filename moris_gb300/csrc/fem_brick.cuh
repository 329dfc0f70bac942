// fem_brick.cuh -- what the brick-cell kernels (fem_brick.cu) and the set-up of
// their sets share.
#pragma once

#include <cstdint>
#include <vector>

#include "fem_internal.hpp"

namespace fem {

// Equation objects the brick kernels take, decided once per set (SetData::fast):
//   0        none of the below: the general cluster kernel
//   1        bulk cell or cluster
//   2 + face ghost on a whole cell face; face = 2 axis + (leader side up)
//   8        interface inside one cell (both sides the same brick)
//   10 + ord boundary facet of ordinal ord (Neumann, Nitsche Dirichlet)
constexpr uint8_t kFastBulk = 1, kFastGhost = 2, kFastInterface = 8, kFastSide = 10;

// ghost tables: per face 7 matrices over (b, lane), lane = (side, node, other side)
constexpr int kGhostMats = 7, kGhostTab = kGhostMats * 256;
// boundary tables: per ordinal the face integrals N_a dN_b (3) and N_a N_b over (b, a)
constexpr int kSideTab = 4 * 64;

void brick_classify(const fem_gpu_ctx* c, SetData& s);
fem_gpu_status brick_upload(fem_gpu_ctx* c, SetData& s);
void brick_release(SetData& s);
// the equation objects of a set in [first, first + count) that are fast
int64_t brick_count(const SetData& s, int64_t first, int64_t count);
fem_gpu_status brick_launch(fem_gpu_ctx* c, const SetData& s, int64_t first, int64_t count, const double* u,
                            double* vals, double* rhs, void* stream);

}  // namespace fem
