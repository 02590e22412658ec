// The direct DFT of even length N = 2P as four small real matrix products in packed FP32 (fma.rn.f32x2), the
// arithmetic of the FP32 FFT passes for every N that the register FFT (fft_fast.cu) does not serve.
//
// A line x folds twice.  With a_t = x_t + x_{N-t}, b_t = x_t - x_{N-t} (a_0 = x_0, a_P = x_P, b_0 = b_P = 0)
//   X[q], X[N-q] = C[q] -/+ i S[q],  C[q] = sum_{t<=P} a_t cos(2 pi t q / N),  S[q] = sum_{t<P} b_t sin(2 pi t q / N),
// and cos / sin of P - t and t differ by the sign (-1)^q only, so for q even / odd
//   C[q] = sum_{t<=P/2} (a_t +/- a_{P-t}) cos,   S[q] = sum_{t<=P/2} (b_t -/+ b_{P-t}) sin:
// N^2 / 2 FMAs a complex line (P / 2 a real one) whatever N's factors are, all of them independent register-tile work
// with every operand in shared memory.  A mixed-radix Stockham FFT has fewer operations, but its stages each cross
// shared memory and a barrier, and a prime factor R costs it R FMAs an element anyway.  Measured on one GB300
// (DFT stages of both directions, l_max 96, 64 functions, N = 194): see direct_dft.cu.
//
// Data are held as units of two floats that go through the same products (one packed FMA): the real and imaginary
// part of a complex line, or the same element of two real lines.
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
__device__ __forceinline__ u64 dup2(float a)
{
    u64 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
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
// the matrices [t][cos even, sin even, cos odd, sin odd][q index]
__host__ __device__ inline int mat_floats(const Fold& f) { return 4 * f.H * f.QS; }

// cos / sin of 2 pi t q / N from the plan's table W[i] = e^{-2 pi i i / N}, q = 2 i (even) or 2 i + 1; zero past P.
__device__ __forceinline__ void build_mats(float* M, const Fold& f, const double2* __restrict__ tw)
{
    const int row = 2 * f.QS;
    for (int e = threadIdx.x; e < f.H * row; e += blockDim.x) {
        const int t = e / row, r = e - t * row, odd = r >= f.QS, i = r - odd * f.QS, q = 2 * i + odd;
        float c = 0.f, s = 0.f;
        if (q <= f.P) {
            const double2 v = __ldg(tw + (t * q) % f.N);
            c = (float)v.x;
            s = (float)(-v.y);
        }
        float* m = M + (4 * t + 2 * odd) * f.QS + i;
        m[0] = c;
        m[f.QS] = s;
    }
}

__device__ __forceinline__ float2 add2(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }

// Folded values of t from x_t, x_{N-t}, x_{P-t}, x_{P+t} (t = 0: x_N counts as 0 and x_P once; t = P/2 for even P:
// the two pairs coincide), in the order of the matrices: even-q cosine and sine terms, odd-q ones.
struct Folded {
    float2 v[4];
};
__device__ __forceinline__ Folded fold_ab(int t, int P, float2 a, float2 b, float2 ap, float2 bp)
{
    const float2 z = make_float2(0.f, 0.f);
    Folded r;
    if (2 * t == P) {
        r.v[0] = a;
        r.v[1] = z;
        r.v[2] = z;
        r.v[3] = b;
    } else {
        r.v[0] = add2(a, ap);
        r.v[1] = sub2(b, bp);
        r.v[2] = sub2(a, ap);
        r.v[3] = add2(b, bp);
    }
    return r;
}
__device__ __forceinline__ Folded fold_line(int t, int P, float2 x, float2 xn, float2 xp, float2 xq)
{
    const float2 z = make_float2(0.f, 0.f);
    if (t == 0) return fold_ab(t, P, x, z, xp, z);
    return fold_ab(t, P, add2(x, xn), sub2(x, xn), add2(xp, xq), sub2(xp, xq));
}

// A thread's register tile: four outputs q of one parity of four units.  Lanes: QL blocks of outputs fastest, then 32 / QL
// pairs of units; a thread's units are 2 ug, 2 ug + 1 and the same 64 / QL further on.  Adjacent lanes then read the same
// units: a 16-byte shared-memory read costs max(2, distinct bytes / 128) cycles (measured: 2 for a warp-uniform one, 4 for 32
// lanes side by side or for eight lanes' addresses repeated in each quarter warp), so a step t costs 12 cycles of the
// shared-memory pipe for 32 packed FMAs, 48 against the 64 that four warps' FMAs take.
struct Tile {
    u64 C[4][4], S[4][4];
};
// m: the block's cosines at t = 0 (sines QS further on, next t 4 QS); v: the thread's first unit of the parity's
// cosine terms at t = 0 (sine terms US further on, next t TS).
template <int QL>
__device__ __forceinline__ void product(const float* m, const float2* v, int H, int QS, int US, int TS, Tile& a)
{
    constexpr int UO = 64 / QL;
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) a.C[i][j] = a.S[i][j] = 0;
#pragma unroll 1
    for (int t = 0; t < H; ++t) {
        const float4 c = *reinterpret_cast<const float4*>(m);
        const float4 s = *reinterpret_cast<const float4*>(m + QS);
        const ulonglong2 a0 = *reinterpret_cast<const ulonglong2*>(v);
        const ulonglong2 a1 = *reinterpret_cast<const ulonglong2*>(v + UO);
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(v + US);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(v + US + UO);
        m += 4 * QS;
        v += TS;
        const u64 cd[4] = {dup2(c.x), dup2(c.y), dup2(c.z), dup2(c.w)};
        const u64 sd[4] = {dup2(s.x), dup2(s.y), dup2(s.z), dup2(s.w)};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            a.C[i][0] = fma2(cd[i], a0.x, a.C[i][0]);
            a.C[i][1] = fma2(cd[i], a0.y, a.C[i][1]);
            a.C[i][2] = fma2(cd[i], a1.x, a.C[i][2]);
            a.C[i][3] = fma2(cd[i], a1.y, a.C[i][3]);
            a.S[i][0] = fma2(sd[i], b0.x, a.S[i][0]);
            a.S[i][1] = fma2(sd[i], b0.y, a.S[i][1]);
            a.S[i][2] = fma2(sd[i], b1.x, a.S[i][2]);
            a.S[i][3] = fma2(sd[i], b1.y, a.S[i][3]);
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
cudaError_t launch_direct_dft(const DirectPass& p, const void* tw, cudaStream_t st);
// The passes of the SO(3) grid transforms over nf grids of N^3, as launch_fft_grid_pass but with its own layout of
// the work grid: pass 1 grid [nf][k][j1][j2] -> work [nf][k][q][j1]; 2 work -> pencils [nf][p][q][k]; -2 pencils ->
// work [nf][j1][q][k]; -1 work -> grid.  real: real samples in / real part out; the work grid then holds q <= N/2
// only.  The inverse passes take the Nyquist bins p = N/2, q = N/2 as zero without reading them.
cudaError_t launch_direct_grid_pass(const void* in, void* out, long long nf, int N, int pass, bool real,
                                    const void* tw, cudaStream_t st);
// ... and of nf S^2 grids of N^2: dir 1 grid [nf][k][j] -> pencils [nf][p][k], dir -1 pencils -> grid (bin N/2 zero).
cudaError_t launch_direct_s2_pass(const void* in, void* out, long long nf, int N, int dir, bool real, const void* tw,
                                  cudaStream_t st);

}  // namespace fftso3
