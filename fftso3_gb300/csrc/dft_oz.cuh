// The direct DFT in double-float by exact digit sums on the tensor cores (dft_oz.cu).
#pragma once
#include <cuda_runtime.h>

namespace fftso3 {

// Even N up to 222.
bool dft_oz_supported(int N);
// The DFT matrices of length N as digits, made once per plan from its twiddle table (N double2).
size_t dft_oz_table_bytes(int N);
cudaError_t dft_oz_build_table(void* table, int N, const void* tw, cudaStream_t st);
// The passes over nf grids of N^3; double-float elements are (re.h, re.l, im.h, im.l).
//   pass 1: sample grid [nf][k][j1][j2] (complex64, or float32 when real) -> DFT over j1 -> out [nf][p][j2][k] double-float
//   pass 2: that -> DFT over j2 -> pencils [nf][p][q][k] as hi (out: complex64) + lo (lo: the remainder)
//   pass -2: double-float pencils [nf][p][q][k] -> DFT over q -> out [nf][p][j2][k] double-float (out may be in)
//   pass -1: that -> DFT over p -> grids [nf][k][j1][j2], rounded once to complex64 or to the real part as float32
// real: the arrays between the passes hold p <= N/2 only.  The inverse passes take the Nyquist bins as zero without reading
// them.  err: device error word (a bounded wait that gave up).
cudaError_t launch_dft_oz_grid_pass(const void* in, void* out, float2* lo, long long nf, int N, int pass, bool real,
                                    const void* table, int* err, cudaStream_t st);

}  // namespace fftso3
