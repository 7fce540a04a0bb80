// The team walk on 64-bit states (qb_team.cuh).
#include "qb_team.cuh"

namespace qb {
void launch_walk_team64(int shape, bool in32, bool out32, const qb_sector* row, const qb_sector* col, const qb_program* P,
                        const void* in, void* out, int k, cudaStream_t st) {
    launch_walk_team<u64, kLists>(shape, in32, out32, row, col, P, in, out, k, st);
}
}  // namespace qb
