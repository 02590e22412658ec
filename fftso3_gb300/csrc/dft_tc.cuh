// The direct DFT of the SO(3) grid transforms on the tensor cores (dft_tc.cu).
#pragma once
#include <cuda_runtime.h>

#include <vector>

namespace fftso3 {

// Even N from 80 to 222 (at most 56 folded terms).
bool dft_tc_supported(int N);
// The passes over nf grids of N^3, with the work grid [nf][p][j2][k]:
//   pass 1: grid [nf][k][j1][j2] -> DFT over j1 -> work;  2: work -> DFT over j2 -> pencils [nf][p][q][k];
//   pass -2: pencils -> DFT over q -> work;               -1: work -> DFT over p -> grid.
// real: real samples in / real part out (the pencils then Hermitian); the work grid, dft_tc_work_elems complex64 a function, then
// holds p <= N/2 only.  The
// inverse passes take the Nyquist bins p = N/2, q = N/2 as zero without reading them.  err: device error word (a bounded
// wait that gave up).
size_t dft_tc_work_elems(int N, bool real);
cudaError_t launch_dft_tc_grid_pass(const void* in, void* out, long long nf, int N, int pass, bool real,
                                    const void* table, int* err, cudaStream_t st);
// The DFT matrices of length N as the kernel's shared-memory operand, made once per plan from its twiddle table.
size_t dft_tc_table_bytes(int N);
cudaError_t dft_tc_build_table(void* table, int N, const void* tw, cudaStream_t st);

// Both passes of a direction of the plans (buckets) of a batch in one cooperative launch with a barrier between the passes:
// forward grids -> pencils, inverse pencils -> grids (Nyquist bins taken as zero).  Any even N up to 222.
bool dft_tc_batch_supported(int N);
struct DftTcBucket {
    int N;
    long long nf;        // functions
    float2* pencil;      // [fn][p][q][k]
    float2* work;        // [fn][p][j2][k]
    const void* table;   // dft_tc_build_table of N
    long long g0;        // first element of its grids in the caller's buffer
};
struct DftTcBatch {
    void* segs = nullptr;    // device: segments of (direction, pass), nseg each
    unsigned* bar = nullptr; // device: two counters, zero between launches
    int nseg = 0, KCmax = 0;
    bool real = false;
    unsigned ntiles[2][2] = {{0, 0}, {0, 0}};
};
// buckets: ascending in N.  Allocates segs and bar (dft_tc_batch_destroy frees them).
cudaError_t dft_tc_batch_create(DftTcBatch& b, const std::vector<DftTcBucket>& buckets, bool real);
void dft_tc_batch_destroy(DftTcBatch& b);
cudaError_t launch_dft_tc_batch(const DftTcBatch& b, bool fwd, const void* in, void* out, int* err, cudaStream_t st);

}  // namespace fftso3
