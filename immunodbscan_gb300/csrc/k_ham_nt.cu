// k_ham_nt.cu -- Hamming distances on 2-plane records (up to 4 residue values).
#include "hamming.cuh"

namespace idb {
void launch_hamming_2(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    launch_hamming<2>(P, a, grid, s);
}
}  // namespace idb
