// k_lev_nt.cu -- edit distances up to 3 on 2-plane records (up to 4 residue values).
#include "lev_diag.cuh"

namespace idb {
void launch_lev_diag_2(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    launch_lev_diag<2>(P, a, grid, s);
}
}  // namespace idb
