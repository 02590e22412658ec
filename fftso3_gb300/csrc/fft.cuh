// Batched strided 1-D FFT launcher (see fft.cu).
#pragma once
#include <cuda_runtime.h>

namespace fftso3 {

struct FFTFactors {
    int N;
    int n;
    int r[24];
};

struct FFTLaunch {
    const void* in;       // complex (or real when real_in) input
    void* out;            // complex (or real part only when real_out) output; may equal in
    FFTFactors fac;
    long long nlines;     // number of transforms
    int lpb;              // lines per CTA
    long long inner, ostride, istride, es;  // line i base = (i/inner)*ostride + (i%inner)*istride; element stride es
    const void* tw;       // device double2 table, W[i] = exp(-2 pi i i / N)
    bool fp64;
    bool df32 = false;    // double-float complex data (dfc32, 16 bytes: re.h, re.l, im.h, im.l); complex only
    bool real_in;
    bool real_out;
    bool lines_fastest;   // consecutive lines adjacent in memory (column pass)
    int threads = 256;    // threads per CTA (<= 256)
    // FP64 synthesis passes (dft64.cu, and the line FFT with real_out): element N/2 is taken as zero (nyq); elements past
    // N/2 as the conjugates of their mirrors, without reading them (herm, with real_out and nyq); lines i with
    // i % inner == skip are not written (dft64 only)
    int nyq = 0, herm = 0, skip = -1;
};

void make_fft_factors(int N, FFTFactors& f);
// Same factors with the prime radices above 8 first (largest first): the
// first stage is then a plain DFT whose twiddles every lane of a warp shares.
void make_fft_factors_prime_first(int N, FFTFactors& f);
size_t fft_smem_bytes(int N, int lpb, bool fp64);
cudaError_t launch_fft_lines(const FFTLaunch& L, cudaStream_t st);
// FP64 passes of short lines as direct DFTs (dft64.cu); one line's arithmetic depends on N only.
bool dft64_supported(int N);
cudaError_t launch_dft64(const FFTLaunch& L, cudaStream_t st);

// Double-float (dfc32) FFTs of N = 64..512, powers of two, along a strided axis of arrays whose innermost index k (N values)
// is contiguous (fft.cu).  table: the stage twiddles in double-float, made once per plan from its twiddle table tw.
bool fft_df32_k_supported(int N);
size_t fft_df32_k_table_bytes(int N);
cudaError_t fft_df32_k_build_table(void* table, int N, const void* tw, cudaStream_t st);
// Double-float forward FFT of nb sample grids f [fn][k][j1][j2] (complex64, or float32 when real) into the
// k-contiguous pencils [fn][p][q][k], written renormalised as hi (complex64, the FP32 rounding) + lo (the
// remainder); buf: nb double-float grids of work space.
cudaError_t launch_fft_df32_k_forward(void* buf, int N, long long nb, const void* f, bool real, float2* hi,
                                      float2* lo, const void* table, cudaStream_t st);
// One pass (1: along p, in place; 2: along q into out) of the double-float FFT of nb synthesis pencils buf [fn][p][q][k]
// (dfc32; overwritten) into the grids out [fn][k][j1][j2], rounded once to complex64, or to the real part as float32 when real.
cudaError_t launch_fft_df32_k_synth_pass(int pass, void* buf, int N, long long nb, void* out, bool real,
                                         const void* table, cudaStream_t st);

// Register-resident FP32 kernels for N = 64..1024, powers of two (fft_fast.cu).
bool fft_fast_supported(int N);
// Tiled transposing passes over nf grids of N^3 complex64 (in != out):
//   pass  1: grid [nf][k][j1][j2] -> FFT over j2 -> T1 [nf][k][q][j1]
//   pass  2: T1 [nf][k][q][j1]    -> FFT over j1 -> pencils [nf][p][q][k]
//   pass -2: pencils [nf][p][q][k] -> FFT over p -> T1 [nf][k][q][j1]
//   pass -1: T1 [nf][k][q][j1]     -> FFT over q -> grid [nf][k][j1][j2]
// real_io: pass 1 reads real samples (float), pass -1 writes the real part only.  half (real grids, all four passes): T1 and
// the pencils hold q < N / 2 alone, as in launch_fft_grid_fused.  nyq (pass -2): the Nyquist bins p = N / 2 and q = N / 2 are
// taken as zero without being read (no coefficient maps to them).
cudaError_t launch_fft_grid_pass(const void* in, void* out, long long nf, int N, int pass, const void* tw,
                                 cudaStream_t st, bool real_io = false, bool half = false, bool nyq = false);
// Both passes of one direction in one persistent launch (N = 64..512): dir 1
// grid -> pencils (passes 1, 2), dir -1 pencils -> grid (passes -2, -1), the
// intermediate held in a ring of ring_elems >= fft_grid_fused_ring_elems(N)
// complex64 (sized for the current device) that stays in L2, instead of a
// full-size work grid.  ctl: fft_grid_fused_ctl_ints device ints (zeroed by
// the launch, on st); err: device error word (9 when a wait on another tile
// timed out).  Same arithmetic as the two-pass form: bit-identical results.
// half (with real_io): the pencils of q < N / 2 alone are written or read (a real function's others are their conjugates, its
// Nyquist bins q = N / 2 are taken as zero).
bool fft_grid_fused_supported(int N);
size_t fft_grid_fused_ring_elems(int N, bool half = false);
size_t fft_grid_fused_ctl_ints(long long nf, int N);
cudaError_t launch_fft_grid_fused(const void* in, void* out, void* ring, size_t ring_elems, int* ctl, int* err,
                                  long long nf, int N, int dir, const void* tw, cudaStream_t st,
                                  bool real_io = false, bool half = false, bool nyq = false);
// Tiled pass over nf S^2 grids of N^2 complex64 (in != out):
//   dir  1: grid [nf][k][j]     -> FFT over j -> pencils [nf][p][k]
//   dir -1: pencils [nf][p][k]  -> FFT over p -> grid [nf][k][j]
// real_io: dir 1 reads real samples, dir -1 writes the real part only.  half (with real_io): the pencils of p < N / 2
// alone are written or read (a real function's others are their conjugates, its Nyquist bin is taken as zero).
cudaError_t launch_fft_s2_pass(const void* in, void* out, long long nf, int N, int dir, const void* tw,
                               cudaStream_t st, bool real_io = false, bool half = false, bool nyq = false);

}  // namespace fftso3
