// The direct DFT of even length N = 2P as four small real matrix products in packed FP32 (fma.rn.f32x2), the
// arithmetic of the FP32 FFT passes for every N that the register FFT (fft_fast.cu) does not serve.
//
// A line x folds twice.  With a_t = x_t + x_{N-t}, b_t = x_t - x_{N-t} (a_0 = x_0, a_P = x_P, b_0 = b_P = 0)
//   X[q], X[N-q] = C[q] -/+ i S[q],  C[q] = sum_{t<=P} a_t cos(2 pi t q / N),  S[q] = sum_{t<P} b_t sin(2 pi t q / N),
// and cos / sin of P - t and t differ by the sign (-1)^q only, so for q even / odd
//   C[q] = sum_{t<=P/2} (a_t +/- a_{P-t}) cos,   S[q] = sum_{t<=P/2} (b_t -/+ b_{P-t}) sin:
// N^2 / 2 FMAs a complex line (P / 2 a real one) whatever N's factors are, all of them independent register-tile work
// with every operand in shared memory.  A mixed-radix Stockham FFT has fewer operations, but its stages each cross
// shared memory and a barrier, and a prime factor R costs it R FMAs an element anyway.  Measured on one GB300 (all four
// passes, 64 complex functions, N = 194): 38.9 ms with the separate transposes as a mixed-radix FFT, 18.2 ms here.
//
// A unit is a complex line, or two real lines x, y.  Its folded terms are held as the pairs (a.x, b.y), (a.y, b.x) (real
// lines: (a.x, b.x), (a.y, b.y)) and the matrices as the pairs (cos, sin), so that one packed FMA advances a cosine sum
// and a sine sum with no operand to duplicate, and the two halves of an accumulator are what the outputs add and subtract.
#pragma once
#include <cuda_runtime.h>

namespace fftso3 {
namespace ddft {

typedef unsigned long long u64;

__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(u64 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}

// Sizes of the folded problem of length N.
struct Fold {
    int N, P;
    int H;       // folded terms: t = 0 .. P/2
    int nbE, nb; // blocks of four outputs: of the even q = 0, 2, .. <= P, and of even and odd q together
    int QS;      // row stride of a matrix (a multiple of four)
};
__host__ __device__ inline Fold fold_of(int N)
{
    Fold f;
    f.N = N;
    f.P = N / 2;
    f.H = f.P / 2 + 1;
    f.nbE = (f.P / 2 + 1 + 3) / 4;
    f.nb = f.nbE + ((f.P + 1) / 2 + 3) / 4;
    f.QS = 4 * f.nbE;  // the odd q are never more than the even ones
    return f;
}
// the matrices [t][parity of q][q index] as (cos, sin)
__host__ __device__ inline int mat_elems(const Fold& f) { return 2 * f.H * f.QS; }

// Entry e of the matrices: (cos, sin) of 2 pi t q / N from the plan's table W[i] = e^{-2 pi i i / N}, q = 2 i (even) or
// 2 i + 1; zero past P.
__device__ __forceinline__ float2 mat_entry(const Fold& f, int e, const double2* __restrict__ tw)
{
    const int row = 2 * f.QS, t = e / row, r = e - t * row, odd = r >= f.QS, q = 2 * (r - odd * f.QS) + odd;
    if (q > f.P) return make_float2(0.f, 0.f);
    const double2 w = __ldg(tw + (t * q) % f.N);
    return make_float2((float)w.x, (float)(-w.y));
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// Folded terms of t from x_t, x_{N-t}, x_{P-t}, x_{P+t} (t = 0: x_N counts as 0 and x_P once; t = P/2 for even P: the
// two pairs coincide), for the even and the odd q, as the pairs described above (REAL: of two real lines).
struct Folded {
    float4 even, odd;
};
template <bool REAL>
__device__ __forceinline__ Folded fold_ab(int t, int P, float2 a, float2 b, float2 ap, float2 bp)
{
    const float2 z = make_float2(0.f, 0.f);
    const bool mid = 2 * t == P;
    const float2 ae = mid ? a : add2(a, ap), be = mid ? z : sub2(b, bp);
    const float2 ao = mid ? z : sub2(a, ap), bo = mid ? b : add2(b, bp);
    Folded r;
    r.even = REAL ? make_float4(ae.x, be.x, ae.y, be.y) : make_float4(ae.x, be.y, ae.y, be.x);
    r.odd = REAL ? make_float4(ao.x, bo.x, ao.y, bo.y) : make_float4(ao.x, bo.y, ao.y, bo.x);
    return r;
}
template <bool REAL>
__device__ __forceinline__ Folded fold_line(int t, int P, float2 x, float2 xn, float2 xp, float2 xq)
{
    const float2 z = make_float2(0.f, 0.f);
    if (t == 0) return fold_ab<REAL>(t, P, x, z, xp, z);
    return fold_ab<REAL>(t, P, add2(x, xn), sub2(x, xn), add2(xp, xq), sub2(xp, xq));
}

// A thread's register tile: four outputs q of one parity of four units.  Lanes: QL blocks of outputs fastest, then 32 / QL
// units.  Adjacent lanes then read the same units: a 16-byte shared-memory read costs max(2, distinct bytes / 128) cycles
// (measured: 2 for a warp-uniform one, 4 for 32 lanes side by side or for eight lanes' addresses repeated in each quarter
// warp), so reads are shared by as many lanes as possible.
struct Tile {
    u64 A[4][4], B[4][4];  // [output][unit]: the accumulators of the unit's two pairs
};
// A sum goes in chunks of at most CHUNK terms that are added up apart, each an even sample of the line (every C-th term, C
// chunks), from its last term to its first: one accumulator over all terms rounds at the size of its partial sums, which
// spectra (largest at t = 0) reach with their first term and smooth samples grow through and beyond
// (inverse of l_max 135 and 143, one function: off by 2.70e-7 and 2.79e-7 of the 2-norm, now 1.86e-7 and 1.94e-7; S^2 l_max 99
// 2.17e-7 and 1.63e-7).
// The chunks' totals take the registers of two units' accumulators, so a tile's units go two by two: 16 cycles of the
// shared-memory pipe a step instead of 12 (64 against the 64 of the FMAs).
constexpr int CHUNK = 12;
// m: the block's pairs at t = 0 (next t 2 QS further on); v: the thread's first unit of the parity at t = 0 (next t TS
// further on), the others HU, 32 / QL, HU + 32 / QL further on.
template <int QL>
__device__ __forceinline__ void product(const float2* m, const float4* v, int H, int QS, int HU, int TS, Tile& a)
{
    constexpr int G = 32 / QL;
    const int C = (H + CHUNK - 1) / CHUNK, sm = 2 * QS * C, sv = TS * C;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) a.A[i][2 * h + j] = a.B[i][2 * h + j] = 0;
        for (int c0 = C - 1; c0 >= 0; --c0) {
            u64 A[4][2], B[4][2];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) A[i][j] = B[i][j] = 0;
            const int t0 = H - 1 - (H - 1 - c0) % C;  // the chunk's last term
            const float2* mt = m + t0 * 2 * QS;
            const float4* vt = v + t0 * TS + h * G;
#pragma unroll 2
            for (int t = t0; t >= 0; t -= C) {
                const ulonglong2 m0 = *reinterpret_cast<const ulonglong2*>(mt);
                const ulonglong2 m1 = *reinterpret_cast<const ulonglong2*>(mt + 2);
                const u64 c[4] = {m0.x, m0.y, m1.x, m1.y};
                const ulonglong2 x[2] = {*reinterpret_cast<const ulonglong2*>(vt), *reinterpret_cast<const ulonglong2*>(vt + HU)};
                mt -= sm;
                vt -= sv;
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        A[i][j] = fma2(c[i], x[j].x, A[i][j]);
                        B[i][j] = fma2(c[i], x[j].y, B[i][j]);
                    }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    a.A[i][2 * h + j] = add2(a.A[i][2 * h + j], A[i][j]);
                    a.B[i][2 * h + j] = add2(a.B[i][2 * h + j], B[i][j]);
                }
        }
    }
}

}  // namespace ddft

// ---- per-plan passes (direct_dft.cu)

// One pass of nf functions: units U = (f no + o) ni + u (f < nf, o < no, u < ni); element j of unit u at
// in + f i_f + o i_o + u i_u + j i_e, output p at out + f o_f + o o_o + u o_u + p o_e (elements of the side's type).
// One of (i_u, i_e) and one of (o_u, o_e) is 1 (real kinds: the unit's step of 1 is a pair of lines, 2).
enum DirectKind {
    DIRECT_COMPLEX,   // unit = a complex64 line
    DIRECT_REAL_IN,   // unit = two float32 lines (i_l apart): complex spectra at p <= N/2 (full: all p), o_u = 2
    DIRECT_REAL_OUT   // unit = the spectra p <= N/2 of two real lines, i_u = 2: two float32 lines (o_l apart)
};
struct DirectPass {
    const void* in;
    void* out;
    int N, kind;
    long long nf;
    int no, ni;
    long long i_f, i_o, i_u, i_e, i_l;
    long long o_f, o_o, o_u, o_e, o_l;
    bool nyq;     // element N/2 of every line is taken as zero (the Nyquist bins of the synthesis)
    bool mirror;  // DIRECT_COMPLEX: outputs of o = 1 .. N/2 - 1 also go, conjugated, to (N - o, N - p)
    bool full;    // DIRECT_REAL_IN: also the outputs p > N/2
};
// Even N whose matrices and one tile fit a CTA's shared memory (N <= 400 or so).
bool direct_dft_supported(int N);
// Share of the SMs' CTAs that a pass of so many units keeps busy in its waves of tiles.
double direct_dft_fill(int N, long long units);
// The matrices of length N in device memory, made once per plan from its twiddle table tw (N double2): built by every CTA
// of every pass, the FP64 loads and conversions took 10 to 25 us of small passes.
size_t direct_dft_table_bytes(int N);
cudaError_t direct_dft_build_table(void* table, int N, const void* tw, cudaStream_t st);
cudaError_t launch_direct_dft(const DirectPass& p, const void* table, cudaStream_t st);
// The passes of the SO(3) grid transforms over nf grids of N^3, as launch_fft_grid_pass but with its own layout of
// the work grid: pass 1 grid [nf][k][j1][j2] -> work [nf][k][q][j1]; 2 work -> pencils [nf][p][q][k]; -2 pencils ->
// work [nf][j1][q][k]; -1 work -> grid.  real: real samples in / real part out; the work grid then holds q <= N/2
// only, and with half the pencils too (else pass 2 writes the others' conjugates as well).  The inverse passes take the Nyquist bins p = N/2, q = N/2 as zero without reading them.
cudaError_t launch_direct_grid_pass(const void* in, void* out, long long nf, int N, int pass, bool real, bool half,
                                    const void* table, cudaStream_t st);
// ... and of nf S^2 grids of N^2: dir 1 grid [nf][k][j] -> pencils [nf][p][k], dir -1 pencils -> grid (bin N/2 zero).
// half (real): the pencils p <= N/2 alone are written (the inverse reads those in any case).
cudaError_t launch_direct_s2_pass(const void* in, void* out, long long nf, int N, int dir, bool real, bool half,
                                  const void* table, cudaStream_t st);

}  // namespace fftso3
