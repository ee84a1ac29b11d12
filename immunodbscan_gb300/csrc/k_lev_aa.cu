// k_lev_aa.cu -- edit distances up to 3 on 5-plane records (up to 32 residue values).
#include "lev_diag.cuh"

namespace idb {
void launch_lev_diag_5(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    launch_lev_diag<5>(P, a, grid, s);
}
}  // namespace idb
