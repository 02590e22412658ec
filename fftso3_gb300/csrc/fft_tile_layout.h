// Layout of the tile FFT (fft_fast.cu): the two steps of a line and their exchange in shared memory.  No CUDA in it, so that the
// bank conflicts can be checked on the host.
#pragma once

#ifdef __CUDACC__
#define FFTSO3_HD __host__ __device__ __forceinline__
#else
#define FFTSO3_HD inline
#endif

namespace fftso3 {
namespace ffast {

constexpr int TL = 16;               // lines per CTA tile
// The tile kernels' line FFT in two steps, N = A B, n = j2 + B j1, K = k1 + A k2:
//   X[K] = sum_j2 w_B^{j2 k2} w_N^{j2 k1} sum_j1 w_A^{j1 k1} x[n],
// an A-point DFT in a thread's registers per (line, j2), one exchange through shared memory, a B-point DFT per (line, k1).
// Each step's threads run along whichever index makes its global accesses whole 128-byte runs, so the transposition of the
// tile costs nothing beyond that exchange.
template <int R, bool C2T>
constexpr int rad_a() { return R == 2 ? 8 : R == 4 ? (C2T ? 8 : 16) : R == 32 ? 32 : 16; }
template <int R, bool C2T>
constexpr int rad_b() { return 32 * R / rad_a<R, C2T>(); }
// The exchange: element (line, k1, j2) at line LS + k1 KS + j2, both strides odd: lanes along the line or along k1 hit
// distinct banks.
template <int R, bool C2T>
constexpr int tile_ks() { return rad_b<R, C2T>() + 1; }
template <int R, bool C2T>
constexpr int tile_ls() { return (rad_a<R, C2T>() * tile_ks<R, C2T>()) | 1; }
// Places of 0 .. n - 1 in which x and n - x are neighbours (0 and n / 2 the first two).
FFTSO3_HD int paired(int pos, int n)
{
    const int u = pos >> 1;
    return (pos & 1) ? (u ? n - u : n / 2) : u;
}

// What thread u of a step works on: its line l (pairs of real lines: row) and column x, j2 of step 1 or k1 of step 2.
struct TilePlace {
    int l, x;
};
template <int R, bool C2T, bool REAL_IO>
FFTSO3_HD TilePlace step1_place(int u)
{
    constexpr int B = rad_b<R, C2T>(), ROWS = REAL_IO ? TL / 2 : TL;
    return {C2T ? u / B : u % ROWS, C2T ? u % B : REAL_IO ? paired(u / ROWS, B) : u / ROWS};
}
template <int R, bool C2T, bool REAL_IO>
FFTSO3_HD TilePlace step2_place(int u)
{
    constexpr int A = rad_a<R, C2T>(), ROWS = REAL_IO ? TL / 2 : TL;
    return {C2T ? u % ROWS : u / A, !C2T ? u % A : REAL_IO ? paired(u / ROWS, A) : u / ROWS};
}
// Places in shared memory (float2): what step 1 stores as its k1-th, step 2 loads as its j-th value.
template <int R, bool C2T>
FFTSO3_HD int step1_slot(TilePlace p, int k1) { return p.l * tile_ls<R, C2T>() + p.x + k1 * tile_ks<R, C2T>(); }
template <int R, bool C2T>
FFTSO3_HD int step2_slot(TilePlace p, int j) { return p.l * tile_ls<R, C2T>() + p.x * tile_ks<R, C2T>() + j; }

}  // namespace ffast
}  // namespace fftso3
