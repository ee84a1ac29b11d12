// k_ham_aa.cu -- Hamming distances on 5-plane records (up to 32 residue values).
#include "hamming.cuh"

namespace idb {
void launch_hamming_5(const Plan &P, const DistArgs &a, int grid, cudaStream_t s) {
    launch_hamming<5>(P, a, grid, s);
}
}  // namespace idb
