// The direct DFT of the SO(3) grid transforms on the tensor cores (dft_tc.cu).
#pragma once
#include <cuda_runtime.h>

namespace fftso3 {

// Even N from 80 to 222 (at most 56 folded terms).
bool dft_tc_supported(int N);
// The passes over nf grids of N^3, with the work grid [nf][p][j2][k]:
//   pass 1: grid [nf][k][j1][j2] -> DFT over j1 -> work;  2: work -> DFT over j2 -> pencils [nf][p][q][k];
//   pass -2: pencils -> DFT over q -> work;               -1: work -> DFT over p -> grid.
// real: real samples in / real part out (the pencils then Hermitian); the work grid then holds p <= N/2 only.  The
// inverse passes take the Nyquist bins p = N/2, q = N/2 as zero without reading them.  err: device error word (a bounded
// wait that gave up).
cudaError_t launch_dft_tc_grid_pass(const void* in, void* out, long long nf, int N, int pass, bool real,
                                    const void* table, int* err, cudaStream_t st);
// The DFT matrices of length N as the kernel's shared-memory operand, made once per plan from its twiddle table.
size_t dft_tc_table_bytes(int N);
cudaError_t dft_tc_build_table(void* table, int N, const void* tw, cudaStream_t st);

}  // namespace fftso3
