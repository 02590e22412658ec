// The direct DFT of even length N = 2P on the tcgen05 tensor cores, for the passes of the SO(3) grid transforms whose N
// the register FFT does not serve.
//
// A line folds twice into four real problems of H = P/2 + 1 terms (direct_dft.cuh has the identities):
//   C[q] = sum_t u_t cos(2 pi t q / N), S[q] = sum_t v_t sin(2 pi t q / N), for the even and the odd q <= P,
//   X[q], X[N - q] = C[q] -/+ i S[q].
// Each is a product of 128 rows (64 complex lines x re / im, or 128 real lines) with a constant matrix of the plan's N: the
// lines' folded terms are the A operand (128 x H, K-major), the matrix the B operand, both as three BF16 terms with the six
// products of weight >= 2^-16 accumulated in FP32 (the leading one apart from the five small ones), as the beta-sum does it.
//
// The leading terms are in fixed point, 8 bits under the line's largest folded value and 8 under 1 for the matrix, so that
// their products are whole multiples of one unit, at most 56 2^16 of it, and their sums exact.  The tensor cores cut a sum
// off where they cannot hold it; with floating-point leading terms that shrank every bin by the same 1e-8 to 2e-8 of itself,
// which the beta-sum, unlike rounding, does not average (forward of l_max 96, one complex function: off by 1.79e-7 of its
// 2-norm, now 1.53e-7, of which the beta-sum alone makes most; inverse 1.82e-7 and 1.28e-7; 0 to 7 % more time a
// direction).  The two other terms hold the remainder to 2^-26 of the line's largest value.
//
// Why: as FP32 register tiles (direct_dft.cu) the products and the loads take turns on the same warps: 1.0 to 1.2 ms a pass
// at N = 194 (16 complex functions).  Here one thread issues them and the warps only move data: 0.39 ms (0.49 and 0.63 the
// transposing passes), 0.21 to 0.29 ms real.  Roles of the one CTA an SM holds:
//   warps 0-13   producers: load a line's elements t, N - t, P - t, P + t for eight t, fold, split, store the K-major
//                swizzled rows, one problem at a time into a ring of two 48 KB slots (the folded values wait in registers);
//   warps 14-17  epilogue, one TMEM lane quarter each: C and S -> X[q], X[N - q] -> global memory;
//   warp 18      MMA issuer (and TMEM owner).
// The matrices (at most 96 KB) stay in shared memory.  Accumulators: two buffers (even and odd q) of C and S, hi and lo.
// Bound: a 64-line tile takes 12 k cycles at N = 194, of which its bytes need 8.6 k (16 a complex sample and pass at
// 6.8 TB/s) and its 80 MMAs 6 k; the rest is the producers' load latency, which 96 registers a thread cannot cover further
// (64 hold the folded values), and instruction issue (45 to 55% of the slots).  Eight epilogue warps with a register split
// (setmaxnreg 88 / 64) measured the same.

// Layouts: both sides of a pass are contiguous along a line index, never along the transformed one, so every global access
// is a run of 64 bytes or more.  A transposing pass (the grid's j2 on one side, k on the other) takes tiles of 8 x 8
// lines (real data 16 x 8).  Eight consecutive accumulator rows are the eight lines of one output run, permuted by an
// exclusive or with the input index so that the producers' stores meet distinct bank groups.
#include <algorithm>

#include <cuda_bf16.h>

#include "common.cuh"
#include "dft_tc.cuh"
#include "tc_ptx.cuh"

namespace fftso3 {

namespace dtc {

using namespace ptx;

constexpr int NPROD = 14, NEPI = 4, MMAW = 18;  // 19 warps: five a scheduler, 96 registers a thread
constexpr int THREADS = 32 * (MMAW + 1);
constexpr int PLANE = 128 * 128;      // 128 rows x 64 BF16
constexpr int SLOT = 3 * PLANE;
constexpr int MAXH = 56;              // folded terms: 7 chunks of 8 (a 64-line tile is 14 items, one a producer warp)
constexpr int MX = 3 * 128 * 4;       // bytes of the lines' largest values (a ring of three tiles)

// Below, the FP32 kernel: with few terms a tile's fixed latencies outweigh its products (all four passes, complex / real, ms:
// N = 66, 64 functions 0.51 / 0.28 here, 0.42 / 0.26 there; N = 160, 16 functions 0.92 / 0.52 here, 2.32 / 1.24 there).
constexpr int MINN = 80;

enum { COMPLEX = 0, REAL_IN = 1, REAL_OUT = 2 };

// One pass over the functions of one N.
struct Geo {
    const void* in;
    void* out;
    const unsigned char* table;
    int N, H, KC;        // folded terms, 16-wide K steps (also 16-wide blocks of outputs)
    unsigned tile0, ntiles;  // its tiles among the launch's
    // straight passes: lines (f, o, u), u < N contiguous on both sides, o < no (skipping o == skip)
    // transposing: lines (f, x, y), x contiguous in the input, y in the output
    int no, skip;
    unsigned tx, ty;     // transposing: tiles along x and y
    unsigned nlines;     // straight: nf no N
    long long i_f, i_a, i_e;  // input: function, o (or y), element strides
    long long o_f, o_a, o_e;  // output: function, o (or x), element strides
    int nyq;             // element P is taken as zero
    int ext;             // batches: in (1) or out (2) is a byte offset into the caller's buffer
};
// A launch: one pass of one plan, or both passes of a direction of several plans (segments ascending in N and tile0).
struct Args {
    Geo g;
    const Geo* segs[2];
    int nseg;
    unsigned ntiles[2];
    int KCmax;
    char* ext;           // batches: the caller's samples (forward) or grids (inverse)
    unsigned* bar;       // batches: arrivals and departures of the barrier between the passes
    int* err;
};

__host__ __device__ constexpr size_t smem_bytes(int KC) { return 2 * SLOT + 12 * 16 * KC * 128 + 128 + MX + 1024; }

// Loads: data of an earlier launch through the read-only path; the work grid of the same launch's first pass at L2.
template <bool COH, typename T>
__device__ __forceinline__ T ld(const T* p)
{
    if constexpr (COH) return __ldcg(p);
    else return __ldg(p);
}

__device__ __forceinline__ void l2_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint32_t bf2(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// The unit of a line's leading terms, 2^(e - 8) for its largest folded value m < 2^e (as bits; not finite: any), and its
// inverse.
struct Unit {
    float u, inv;
};
__device__ __forceinline__ Unit unit_of(unsigned m)
{
    const int e = min(max((int)(m >> 23) - 126, -118), 128);
    return {__uint_as_float((unsigned)(127 + e - 8) << 23), __uint_as_float((unsigned)(127 + 8 - e) << 23)};
}

// Packed FP32 pairs: half the instructions of the splits (19 warps' producers are short of issue slots).
typedef unsigned long long u64;
__device__ __forceinline__ u64 pack2(float a, float b)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float2 unpack2(u64 a)
{
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(a));
    return r;
}
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
__device__ __forceinline__ u64 mul2(u64 a, u64 b)
{
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// eight values into one 16-byte chunk of each of the three BF16 planes
__device__ __forceinline__ void store_split(uint32_t dst, const float* x, Unit s)
{
    const u64 magic = pack2(12582912.f, 12582912.f), minus = pack2(-12582912.f, -12582912.f);  // 1.5 2^23
    const u64 inv = pack2(s.inv, s.inv), u = pack2(s.u, s.u), nu = pack2(-s.u, -s.u), n1 = pack2(-1.f, -1.f);
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const u64 v = pack2(x[2 * j], x[2 * j + 1]);
        const u64 q = add2(fma2(v, inv, magic), minus);  // |q| <= 256
        const u64 r = fma2(q, nu, v);                    // exact
        const float2 lead = unpack2(mul2(q, u)), rest = unpack2(r);
        w[0][j] = bf2(lead.x, lead.y);
        w[1][j] = bf2(rest.x, rest.y);
        const u64 t = pack2(__uint_as_float(w[1][j] << 16), __uint_as_float(w[1][j] & 0xffff0000u));
        const float2 last = unpack2(fma2(t, n1, r));
        w[2][j] = bf2(last.x, last.y);
    }
#pragma unroll
    for (int p = 0; p < 3; ++p)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + p * PLANE), "r"(w[p][0]), "r"(w[p][1]),
                     "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
}
// A line's warps: those of the same parity (their items' blocks of 32 lines have it).
__device__ __forceinline__ void producers_sync(int warp)
{
    asm volatile("bar.sync %0, %1;" ::"r"(1 + (warp & 1)), "n"(16 * NPROD) : "memory");
}

// A line of a tile: its place in the input and the output (elements of the side's type), and whether it exists.
struct Line {
    long long in, out;
    int o;       // straight: the outer index
    bool ok;
};
// Straight tile: line number l of 64 (complex).  Transposing: l = (x, y) of the tile.
template <int KIND, bool TR>
__device__ __forceinline__ Line line_of(const Geo& a, unsigned tile, int x, int y)
{
    Line r;
    tile -= a.tile0;
    if (TR) {
        constexpr int XB = KIND == REAL_IN ? 16 : 8, YB = KIND == REAL_OUT ? 16 : 8;
        const unsigned per = a.tx * a.ty, f = tile / per, rem = tile - f * per, by = rem / a.tx, bx = rem - by * a.tx;
        const int gx = bx * XB + x, gy = by * YB + y;
        r.ok = gx < a.N && gy < a.N;
        r.in = f * a.i_f + gy * a.i_a + gx;
        r.out = f * a.o_f + gx * a.o_a + gy;
        r.o = 0;
    } else {
        const unsigned U = tile * 64u + 8u * x + y;
        const unsigned fo = U / (unsigned)a.N, u = U - fo * a.N, f = fo / (unsigned)a.no;
        int o = (int)(fo - f * a.no);
        if (a.skip >= 0 && o >= a.skip) ++o;
        r.ok = U < a.nlines;
        r.in = f * a.i_f + o * a.i_a + u;
        r.out = f * a.o_f + o * a.o_a + u;
        r.o = o;
    }
    return r;
}

// Loads and folds eight terms t = t0 .. t0 + 7 of a line: x[problem][t - t0 (re row), 8 + t - t0 (im row)].  The sine
// problems of a complex line take (im, -re) in the (re, im) rows, so that both parts of X[q], X[N - q] are C +/- S of
// one row; those of real samples are negated (the spectrum is C - i S).  EDGE: the chunk may
// hold t = 0 (x_N counts as 0, x_P once), t = P / 2 (the two pairs coincide) or t >= H (zero).
template <int KIND, bool EDGE, bool COH, int VPL>
__device__ __forceinline__ void load_fold(const Geo& a, const void* src, long long in, int t0, int H, int N, float (&x)[4][VPL])
{
    const int P = N / 2;
    if (KIND == COMPLEX) {
        const float2* g = reinterpret_cast<const float2*>(src) + in;
        const float2* p0 = g + t0 * a.i_e;
        const float2* p1 = g + (N - t0) * a.i_e;
        const float2* p2 = g + (P - t0) * a.i_e;
        const float2* p3 = g + (P + t0) * a.i_e;
        const float2 z = make_float2(0.f, 0.f);
        float2 y[4][8];
#pragma unroll
        for (int k = 0; k < 8; ++k, p0 += a.i_e, p1 -= a.i_e, p2 -= a.i_e, p3 += a.i_e) {
            const int t = t0 + k;
            const bool in0 = !EDGE || t < H, two = !EDGE || 2 * t != P, pos = !EDGE || t > 0;
            y[0][k] = in0 ? ld<COH>(p0) : z;
            y[1][k] = in0 && pos ? ld<COH>(p1) : z;
            y[2][k] = in0 && two && (pos || !a.nyq) ? ld<COH>(p2) : z;
            y[3][k] = in0 && two && pos ? ld<COH>(p3) : z;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const bool pos = !EDGE || t0 + k > 0, mid = EDGE && 2 * (t0 + k) == P;
            const float2 a0 = make_float2(y[0][k].x + y[1][k].x, y[0][k].y + y[1][k].y);
            const float2 a1 = make_float2(y[2][k].x + y[3][k].x, y[2][k].y + y[3][k].y);
            const float2 b0 = pos ? make_float2(y[0][k].x - y[1][k].x, y[0][k].y - y[1][k].y) : z;
            const float2 b1 = pos ? make_float2(y[2][k].x - y[3][k].x, y[2][k].y - y[3][k].y) : z;
            x[0][k] = a0.x + a1.x;
            x[0][k + 8] = a0.y + a1.y;
            x[1][k] = mid ? 0.f : b0.y - b1.y;
            x[1][k + 8] = mid ? 0.f : b1.x - b0.x;
            x[2][k] = mid ? 0.f : a0.x - a1.x;
            x[2][k + 8] = mid ? 0.f : a0.y - a1.y;
            x[3][k] = b0.y + b1.y;
            x[3][k + 8] = -b0.x - b1.x;
        }
    } else if (KIND == REAL_IN) {
        const float* g = reinterpret_cast<const float*>(src) + in;
        const float* p0 = g + t0 * a.i_e;
        const float* p1 = g + (N - t0) * a.i_e;
        const float* p2 = g + (P - t0) * a.i_e;
        const float* p3 = g + (P + t0) * a.i_e;
#pragma unroll
        for (int k = 0; k < 8; ++k, p0 += a.i_e, p1 -= a.i_e, p2 -= a.i_e, p3 += a.i_e) {
            const int t = t0 + k;
            const bool in0 = !EDGE || t < H, two = !EDGE || 2 * t != P, pos = !EDGE || t > 0;
            x[0][k] = in0 ? ld<COH>(p0) : 0.f;
            x[1][k] = in0 && pos ? ld<COH>(p1) : 0.f;
            x[2][k] = in0 && two ? ld<COH>(p2) : 0.f;
            x[3][k] = in0 && two && pos ? ld<COH>(p3) : 0.f;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const bool pos = !EDGE || t0 + k > 0, mid = EDGE && 2 * (t0 + k) == P;
            const float a0 = x[0][k] + x[1][k], a1 = x[2][k] + x[3][k];
            const float b0 = pos ? x[0][k] - x[1][k] : 0.f, b1 = pos ? x[2][k] - x[3][k] : 0.f;
            x[0][k] = a0 + a1;
            x[1][k] = mid ? 0.f : b1 - b0;
            x[2][k] = mid ? 0.f : a0 - a1;
            x[3][k] = -b0 - b1;
        }
    } else {
        // a_t = 2 Re X_t, b_t = 2 Im X_t (t = 0: Re X_0 and 0); X_P = 0
        const float2* g = reinterpret_cast<const float2*>(src) + in;
        const float2* p0 = g + t0 * a.i_e;
        const float2* p2 = g + (P - t0) * a.i_e;
        const float2 z = make_float2(0.f, 0.f);
        float2 y[2][8];
#pragma unroll
        for (int k = 0; k < 8; ++k, p0 += a.i_e, p2 -= a.i_e) {
            const int t = t0 + k;
            y[0][k] = !EDGE || t < H ? ld<COH>(p0) : z;
            y[1][k] = !EDGE || (t < H && t > 0 && 2 * t != P) ? ld<COH>(p2) : z;
        }
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            const bool pos = !EDGE || t0 + k > 0, mid = EDGE && 2 * (t0 + k) == P;
            const float sa = pos ? 2.f : 1.f, sb = pos ? 2.f : 0.f;
            x[0][k] = sa * y[0][k].x + 2.f * y[1][k].x;
            x[1][k] = mid ? 0.f : sb * y[0][k].y - 2.f * y[1][k].y;
            x[2][k] = mid ? 0.f : sa * y[0][k].x - 2.f * y[1][k].x;
            x[3][k] = sb * y[0][k].y + 2.f * y[1][k].y;
        }
    }
}

// Finishes the outputs q = q0, q0 + 2, .. (the first nv of sixteen; FULL: all of them, and 0 < q < P) of an accumulator row
// in TMEM at c (cosine sums: hi, NQ columns on lo) and c + 128 (sine sums).
template <int KIND, bool TR, bool FULL>
__device__ __forceinline__ void finish(const Geo& a, void* dst, const Line& L, uint32_t c, int q0, int nv, int part)
{
    const int N = a.N, P = N / 2, NQ = 16 * a.KC;
    float C[16], S[16];
    {
        uint32_t t[4][16];
        tmem_ld16_nowait(c, t[0]);
        tmem_ld16_nowait(c + NQ, t[1]);
        tmem_ld16_nowait(c + 128, t[2]);
        tmem_ld16_nowait(c + 128 + NQ, t[3]);
        tmem_wait_ld();
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            C[i] = __uint_as_float(t[0][i]) + __uint_as_float(t[1][i]);
            S[i] = __uint_as_float(t[2][i]) + __uint_as_float(t[3][i]);
        }
    }
    // addresses as base + i step in one multiply-add each
    if (KIND == REAL_IN) {
        const unsigned step = (unsigned)(16 * a.o_e);
        char* o = reinterpret_cast<char*>(reinterpret_cast<float2*>(dst) + L.out + q0 * a.o_e);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (FULL || i < nv) *reinterpret_cast<float2*>(o + (unsigned long long)i * step) = make_float2(C[i], S[i]);
        return;
    }
    constexpr int W = KIND == COMPLEX ? 2 : 1;  // floats: complex elements are two apart
    char* lo = reinterpret_cast<char*>(reinterpret_cast<float*>(dst) + W * (L.out + q0 * a.o_e) + part);
    // the sixteenth output's mirror, from where the others ascend
    char* hi = reinterpret_cast<char*>(reinterpret_cast<float*>(dst) + W * (L.out + (N - q0 - 30) * a.o_e) + part);
    const unsigned step = (unsigned)(8 * W * a.o_e);
    const int h0 = q0 == 0 ? 1 : 0, h1 = min(nv, (P - q0 + 1) >> 1);  // 0 < q < P
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (FULL || i < nv) *reinterpret_cast<float*>(lo + (unsigned long long)i * step) = C[i] + S[i];
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (FULL || (i >= h0 && i < h1)) *reinterpret_cast<float*>(hi + (unsigned long long)(15 - i) * step) = C[i] - S[i];
}

// What the roles of a CTA share.
struct Ctx {
    unsigned char* smem;  // two slots, then the matrices [problem][plane][q][t] (K-major swizzled rows of 128 bytes)
    unsigned char* bmat;
    uint64_t *full, *empty, *accf, *acce, *bfull;
    volatile int* abort_flag;
    unsigned* mx;  // [tile mod 3][line]: bits of the largest folded value
    uint32_t tmem;
    int warp, lane;
};
// Counts that run on over the passes of a launch.
struct Counts {
    unsigned s = 0;   // problems produced / issued, or accumulator buffers finished
    unsigned nb = 0;  // matrices loaded
    int tp = 0;       // producers: tiles mod 3
};

// The segment a role's next tile is in (tiles ascend).
template <bool BATCH>
__device__ __forceinline__ const Geo& seek(const Args& a, int pass, unsigned tile, int& seg)
{
    if (!BATCH) return a.g;
    const Geo* s = a.segs[pass];
    while (seg + 1 < a.nseg && tile >= s[seg + 1].tile0) ++seg;
    return s[seg];
}

// producers: an item is 32 lines x 8 folded terms
template <int KIND, bool TR, bool BATCH, bool COH>
__device__ __forceinline__ void produce(const Args& a, int pass, const Ctx& c, Counts& n)
{
    constexpr int VPL = KIND == COMPLEX ? 16 : 8;  // values of a problem held by an item's thread (8 t, re and im)
    constexpr int IPW = KIND == COMPLEX ? 1 : 2;   // items of a warp
    constexpr int LB = KIND == COMPLEX ? 2 : 4;    // blocks of 32 lines in a tile
    const int lane = c.lane;
    int lx[IPW], ly[IPW], ch[IPW], row[IPW], ln[IPW];
#pragma unroll
    for (int w = 0; w < IPW; ++w) {
        const int it = c.warp + w * NPROD, lb = it % LB;
        ch[w] = it / LB;
        if (KIND == COMPLEX) {
            // x = lane & 7 in the input's order; straight tiles number their lines 8 x + y
            lx[w] = TR ? (lane & 7) : (lane >> 3) + 4 * lb;
            ly[w] = TR ? (lane >> 3) + 4 * lb : (lane & 7);
            row[w] = lx[w] * 16 + (ly[w] ^ (lx[w] & 7));
        } else if (KIND == REAL_IN) {
            lx[w] = lane & 15;
            ly[w] = (lane >> 4) + 2 * lb;
            row[w] = lx[w] * 8 + (ly[w] ^ (lx[w] & 7));
        } else {
            lx[w] = lane & 7;
            ly[w] = (lane >> 3) + 4 * lb;
            row[w] = lx[w] * 16 + (ly[w] ^ lx[w]);
        }
        ln[w] = lane + 32 * lb;
    }
    int seg = 0;
    const unsigned ntiles = a.ntiles[pass];
    // a failed wait (every producer meets it in its turn) ends the stores; the tiles' barriers go on, so that no warp waits
    // for one that left
    for (unsigned tile = blockIdx.x; tile < ntiles; tile += gridDim.x, n.tp = n.tp == 2 ? 0 : n.tp + 1) {
        const Geo& g = seek<BATCH>(a, pass, tile, seg);
        const int H = g.H, N = g.N, P = N / 2;
        const void* src = BATCH && g.ext == 1 ? a.ext + (size_t)g.in : g.in;
        float v[IPW][4][VPL];  // [problem][t (re row), then t (im row)]
#pragma unroll
        for (int w = 0; w < IPW; ++w) {
            const int t0 = 8 * ch[w];
            if (t0 >= H) continue;
            const Line L = line_of<KIND, TR>(g, tile, lx[w], ly[w]);
            float (&x)[4][VPL] = v[w];
            if (!L.ok) {
#pragma unroll
                for (int k = 0; k < VPL; ++k) x[0][k] = x[1][k] = x[2][k] = x[3][k] = 0.f;
            } else if (t0 > 0 && t0 + 8 <= H && 2 * (t0 + 7) != P) {
                load_fold<KIND, false, COH>(g, src, L.in, t0, H, N, x);
            } else {
                load_fold<KIND, true, COH>(g, src, L.in, t0, H, N, x);
            }
            unsigned m = 0;
#pragma unroll
            for (int k = 0; k < VPL; ++k)
#pragma unroll
                for (int pr = 0; pr < 4; ++pr) m = max(m, __float_as_uint(x[pr][k]) & 0x7fffffffu);
            atomicMax(&c.mx[n.tp * 128 + ln[w]], m);
        }
        // the next tile's elements into L2 while this one's problems are stored and multiplied: lane k of a run of
        // eight lines requests the run's element t0 + k (and its three images)
        if (tile + gridDim.x < g.tile0 + g.ntiles) {
#pragma unroll
            for (int w = 0; w < IPW; ++w) {
                const int k = 8 * ch[w] + (lane & 7);
                if (k >= H) continue;
                const Line L = line_of<KIND, TR>(g, tile + gridDim.x, lx[w], ly[w]);
                if (!L.ok) continue;
                constexpr int E = KIND == REAL_IN ? 4 : 8;
                const char* p = reinterpret_cast<const char*>(src) + E * (L.in - (lane & (KIND == REAL_IN ? 15 : 7)));
                const long long e = E * g.i_e;
                l2_prefetch(p + k * e);
                l2_prefetch(p + (P - k) * e);
                if (KIND != REAL_OUT && k > 0) {
                    l2_prefetch(p + (N - k) * e);
                    l2_prefetch(p + (P + k) * e);
                }
            }
        }
        // the next tile's maxima (of this parity's lines): last read before the last tile's barrier
        if (c.warp < 2) {
            unsigned* next = c.mx + (n.tp == 2 ? 0 : n.tp + 1) * 128 + 32 * c.warp + lane;
            next[0] = 0;
            if (LB == 4) next[64] = 0;
        }
        producers_sync(c.warp);
        bool dead = __any_sync(0xffffffffu, *c.abort_flag);
        Unit un[IPW];
#pragma unroll
        for (int w = 0; w < IPW; ++w) un[w] = unit_of(c.mx[n.tp * 128 + ln[w]]);
#pragma unroll
        for (int pr = 0; pr < 4; ++pr, ++n.s) {
            const int sl = n.s & 1;
            if (dead) continue;
            if (__any_sync(0xffffffffu, n.s >= 2 && !mbar_wait(&c.empty[sl], ((n.s >> 1) - 1) & 1, a.err, 31))) {
                *c.abort_flag = 1;
                dead = true;
                continue;
            }
#pragma unroll
            for (int w = 0; w < IPW; ++w) {
                if (8 * ch[w] >= H) continue;
                const uint32_t d = smem_u32(c.smem + sl * SLOT) + row[w] * 128 + ((ch[w] ^ (row[w] & 7)) << 4);
                store_split(d, v[w][pr], un[w]);
                if (KIND == COMPLEX) store_split(d + 8 * 128, v[w][pr] + 8, un[w]);
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) mbar_arrive(&c.full[sl]);
        }
    }
}

// MMA issuer (one elected thread)
template <bool BATCH>
__device__ __forceinline__ void issue(const Args& a, int pass, const Ctx& c, Counts& n)
{
    const uint32_t sa = smem_u32(c.smem), sb = smem_u32(c.bmat);
    int seg = 0, held = -1;  // the segment whose matrices are in shared memory
    bool ok = true;
    const unsigned ntiles = a.ntiles[pass];
    for (unsigned tile = blockIdx.x; tile < ntiles && ok && !*c.abort_flag; tile += gridDim.x) {
        const Geo& g = seek<BATCH>(a, pass, tile, seg);
        const int KC = g.KC, NQ = 16 * KC, BPLANE = NQ * 128;
        if (seg != held) {
            // the matrices of this N, once the MMAs that read the last ones are done (both accumulator buffers committed)
            for (int b = 0; b < 2 && ok; ++b) {
                const unsigned k = (n.s + 2 - 2 * b) / 4;
                if (k > 0) ok = mbar_wait(&c.accf[b], (k - 1) & 1, a.err, 37);
            }
            if (ok) {
                mbar_expect_tx(c.bfull, 12 * BPLANE);
                bulk_load(c.bmat, g.table, 12 * BPLANE, c.bfull);
                ok = mbar_wait(c.bfull, n.nb & 1, a.err, 34);
                ++n.nb;
            }
            if (!ok) break;
            held = seg;
        }
        const uint32_t id1 = idesc_bf16_mn(false, NQ, 128), id2 = idesc_bf16_mn(false, 2 * NQ, 128);
        for (int pr = 0; pr < 4; ++pr, ++n.s) {
            const unsigned s = n.s;
            const int sl = s & 1, ab = (s >> 1) & 1;  // accumulator buffer: alternates with the parity of q
            if ((pr & 1) == 0 && s >= 4 && !mbar_wait(&c.acce[ab], ((s >> 2) - 1) & 1, a.err, 32)) {
                ok = false;
                break;
            }
            if (!mbar_wait(&c.full[sl], (s >> 1) & 1, a.err, 33)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t hi = c.tmem + ab * 256 + (pr & 1) * 128, lo = hi + NQ;
            // descriptors: 16-byte units in the low bits, 32 bytes of K a step
            uint64_t ad = smem_desc(sa + sl * SLOT, 16, 1024), bd = smem_desc(sb + pr * 3 * BPLANE, 16, 1024);
            const uint64_t bp = (uint64_t)(BPLANE >> 4);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk, ad += 2, bd += 2) {
                if (kk >= KC) break;
                mma_bf16(hi, ad, bd, id2, kk > 0);  // x0 [y0 | y1] -> [hi | lo]
                mma_bf16(lo, ad + (PLANE >> 4), bd, id1, 1);
                mma_bf16(lo, ad, bd + 2 * bp, id1, 1);
                mma_bf16(lo, ad + (PLANE >> 4), bd + bp, id1, 1);
                mma_bf16(lo, ad + 2 * (PLANE >> 4), bd, id1, 1);
            }
            mma_commit(&c.empty[sl]);
            if (pr & 1) mma_commit(&c.accf[ab]);
        }
    }
    if (!ok) *c.abort_flag = 1;
    // the last commits must land before the next pass or before TMEM is freed: buffer b was committed (s + 2 - 2 b) / 4 times
    for (int b = 0; b < 2; ++b) {
        const unsigned k = (n.s + 2 - 2 * b) / 4;
        if (k > 0) mbar_wait(&c.accf[b], (k - 1) & 1, a.err, 36);
    }
}

template <int KIND, bool TR, bool BATCH>
__device__ __forceinline__ void drain(const Args& a, int pass, const Ctx& c, Counts& n)
{
    const int quarter = c.warp & 3, r = quarter * 32 + c.lane;
    int x, y, part = 0;
    if (KIND == COMPLEX) {
        x = r >> 4;
        y = (r & 7) ^ (x & 7);
        part = (r >> 3) & 1;
    } else if (KIND == REAL_IN) {
        x = r >> 3;
        y = (r & 7) ^ (x & 7);
    } else {
        x = r >> 4;
        y = (r & 15) ^ x;
    }
    int seg = 0;
    const unsigned ntiles = a.ntiles[pass];
    for (unsigned tile = blockIdx.x; tile < ntiles && !*c.abort_flag; tile += gridDim.x) {
        const Geo& g = seek<BATCH>(a, pass, tile, seg);
        const int P = g.N / 2;
        void* dst = BATCH && g.ext == 2 ? a.ext + (size_t)g.out : g.out;
        const Line L = line_of<KIND, TR>(g, tile, x, y);
        const bool all = __all_sync(0xffffffffu, L.ok);
        for (int par = 0; par < 2; ++par, ++n.s) {
            const int ab = n.s & 1;
            if (!mbar_wait(&c.accf[ab], (n.s >> 1) & 1, a.err, 35)) {
                *c.abort_flag = 1;
                return;
            }
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            const uint32_t base = c.tmem + ((uint32_t)(quarter * 32) << 16) + ab * 256;
            const int nq = (P - par) / 2 + 1;  // outputs of this parity
            for (int b = 0; 16 * b < nq; ++b) {
                const int q0 = 32 * b + par;
                if (all && q0 > 0 && q0 + 30 < P)
                    finish<KIND, TR, true>(g, dst, L, base + 16 * b, q0, 16, part);
                else
                    finish<KIND, TR, false>(g, dst, L, base + 16 * b, q0, L.ok ? nq - 16 * b : 0, part);
            }
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (c.lane == 0) mbar_arrive(&c.acce[ab]);
        }
    }
}

template <int KIND, bool TR, bool BATCH, bool COH>
__device__ __forceinline__ void run_pass(const Args& a, int pass, const Ctx& c, Counts& n)
{
    if (c.warp < NPROD) {
        produce<KIND, TR, BATCH, COH>(a, pass, c, n);
    } else if (c.warp == MMAW) {
        if (elect_one()) issue<BATCH>(a, pass, c, n);
        __syncwarp();
    } else {
        drain<KIND, TR, BATCH>(a, pass, c, n);
    }
}

// Every CTA of the launch (all resident: a cooperative launch) has finished the first pass.  bar[0] counts arrivals, bar[1]
// departures; the last to leave clears both for the next launch.  The wait is bounded (about a second); a CTA that gave up
// or aborted still arrives.
__device__ __forceinline__ void grid_barrier(const Args& a, volatile int* abort_flag)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(&a.bar[0], 1u);
        const long long t0 = clock64();
        while (*(volatile unsigned*)&a.bar[0] < gridDim.x) {
            if (clock64() - t0 > WAIT_CYCLES) {
                atomicCAS(a.err, 0, 38);
                *abort_flag = 1;
                break;
            }
        }
        __threadfence();
        if (atomicAdd(&a.bar[1], 1u) == gridDim.x - 1) {
            a.bar[0] = 0;
            a.bar[1] = 0;
        }
    }
    __syncthreads();
}

__device__ __forceinline__ void clear_slots(unsigned char* smem)
{
    for (int i = threadIdx.x; i < 2 * SLOT / 16; i += THREADS) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
    fence_proxy_async();
}

// MODE: a single pass (KIND, TR), or (BATCH) both passes of a direction of real or complex plans.
enum { SINGLE = 0, BATCH_FWD = 1, BATCH_INV = 2 };
template <int MODE, int KIND, bool TR>
__global__ void __launch_bounds__(THREADS, 1) dft_tc_kernel(const __grid_constant__ Args a)
{
    extern __shared__ unsigned char smem_raw[];
    Ctx c;
    c.smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    c.bmat = c.smem + 2 * SLOT;
    c.full = (uint64_t*)(c.bmat + 12 * 16 * a.KCmax * 128);
    c.empty = c.full + 2;
    c.accf = c.empty + 2;
    c.acce = c.accf + 2;
    c.bfull = c.acce + 2;
    uint32_t* tmem_slot = (uint32_t*)(c.bfull + 1);
    c.abort_flag = (volatile int*)(tmem_slot + 1);
    c.mx = (unsigned*)((unsigned char*)c.full + 128);
    c.warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0);
    c.lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&c.full[s], NPROD);
            mbar_init(&c.empty[s], 1);
            mbar_init(&c.accf[s], 1);
            mbar_init(&c.acce[s], NEPI);
        }
        mbar_init(c.bfull, 1);
        *c.abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (c.warp == MMAW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    for (int i = threadIdx.x; i < MX / 4; i += THREADS) c.mx[i] = 0;
    // the slots' columns past the folded terms stay zero (segments ascend in N, so a pass never leaves longer rows behind)
    clear_slots(c.smem);
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    c.tmem = *tmem_slot;

    Counts n;
    if (MODE == SINGLE) {
        run_pass<KIND, TR, false, false>(a, 0, c, n);
    } else {
        constexpr bool REAL = KIND != COMPLEX;
        if (MODE == BATCH_FWD) run_pass<REAL ? REAL_IN : COMPLEX, true, true, false>(a, 0, c, n);
        else run_pass<COMPLEX, false, true, false>(a, 0, c, n);
        grid_barrier(a, c.abort_flag);
        clear_slots(c.smem);
        __syncthreads();
        if (MODE == BATCH_FWD) run_pass<COMPLEX, false, true, true>(a, 1, c, n);
        else run_pass<REAL ? REAL_OUT : COMPLEX, true, true, true>(a, 1, c, n);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (c.warp == MMAW) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(c.tmem), "r"(512));
    }
}

// [problem: cos even, sin even, cos odd, sin odd][plane][q][t] BF16, rows of 128 bytes, their 16-byte chunks swizzled; one
// thread a chunk (eight t of the three planes).  The terms are split from the FP64 values, the first to multiples of 2^-8.
__global__ void build_table_kernel(unsigned char* table, int N, int H, int NQ, const double2* __restrict__ tw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 4 * NQ * 8) return;
    const int c = i & 7, qi = (i >> 3) % NQ, pr = (i >> 3) / NQ, q = 2 * qi + (pr >> 1);
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        double v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int t = 8 * c + 2 * j + h;
            v[h] = 0.0;
            if (t < H && q <= N / 2) {
                const double2 x = __ldg(tw + (t * q) % N);
                v[h] = (pr & 1) ? -x.y : x.x;
            }
        }
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            w[p][j] = p ? bf2((float)v[0], (float)v[1]) : bf2((float)(rint(v[0] * 256.) / 256.), (float)(rint(v[1] * 256.) / 256.));
            v[0] -= (double)__uint_as_float(w[p][j] << 16);
            v[1] -= (double)__uint_as_float(w[p][j] & 0xffff0000u);
        }
    }
    unsigned char* d = table + (size_t)pr * 3 * NQ * 128 + qi * 128 + ((c ^ (qi & 7)) << 4);
#pragma unroll
    for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(d + (size_t)p * NQ * 128) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

static cudaError_t device_sms(int& nsm)
{
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    return e == cudaSuccess ? cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) : e;
}

template <int KIND, bool TR>
static cudaError_t run(const Geo& g, int* err, cudaStream_t st)
{
    auto kern = dft_tc_kernel<SINGLE, KIND, TR>;
    int nsm = 0;
    cudaError_t e = device_sms(nsm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(4));
    if (e != cudaSuccess) return e;
    Args a = {};
    a.g = g;
    a.nseg = 1;
    a.ntiles[0] = g.ntiles;
    a.KCmax = g.KC;
    a.err = err;
    kern<<<std::min(g.ntiles, (unsigned)nsm), THREADS, smem_bytes(g.KC), st>>>(a);
    return cudaGetLastError();
}

static int folded_terms(int N) { return N / 4 + 1; }

// Geometry of a pass (numbered as in launch_dft_tc_grid_pass).
static bool geometry(Geo& a, const void* in, void* out, long long nf, int N, int pass, bool real, const void* table)
{
    const long long n = N, NN = n * n;
    const int P = N / 2;
    if (nf < 1 || nf * NN > 0x7fffffffLL) return false;
    a = Geo{};
    a.in = in;
    a.out = out;
    a.table = (const unsigned char*)table;
    a.N = N;
    a.H = folded_terms(N);
    a.KC = (a.H + 15) / 16;
    a.i_f = a.o_f = NN * n;
    (pass == 1 || pass == -2 ? a.o_f : a.i_f) = (long long)dft_tc_work_elems(N, real);
    a.skip = -1;
    auto blocks = [&](int b) { return (unsigned)((N + b - 1) / b); };
    switch (pass) {
        case 1:  // x = j2, y = k
            a.tx = blocks(real ? 16 : 8);
            a.ty = blocks(8);
            a.i_a = NN;
            a.i_e = n;
            a.o_a = n;
            a.o_e = NN;
            break;
        case 2:
        case -2:  // o = p, lines along k
            a.i_a = a.o_a = NN;
            a.i_e = a.o_e = n;
            a.nyq = pass < 0;
            if (pass > 0) {
                a.no = real ? P + 1 : N;
            } else {
                a.no = real ? P : N - 1;  // without the Nyquist row p = P
                a.skip = real ? -1 : P;
            }
            a.nlines = (unsigned)(nf * a.no * n);
            break;
        case -1:  // x = k, y = j2
            a.tx = blocks(8);
            a.ty = blocks(real ? 16 : 8);
            a.nyq = 1;
            a.i_a = n;
            a.i_e = NN;
            a.o_a = NN;
            a.o_e = n;
            break;
        default: return false;
    }
    a.ntiles = a.nlines ? (a.nlines + 63) / 64 : (unsigned)nf * a.tx * a.ty;
    return true;
}

}  // namespace dtc

using namespace dtc;

bool dft_tc_supported(int N) { return N >= MINN && dft_tc_batch_supported(N); }
bool dft_tc_batch_supported(int N) { return N >= 2 && N % 2 == 0 && folded_terms(N) <= MAXH; }

size_t dft_tc_work_elems(int N, bool real) { return (size_t)(real ? N / 2 + 1 : N) * N * N; }

size_t dft_tc_table_bytes(int N) { return (size_t)12 * 16 * ((folded_terms(N) + 15) / 16) * 128; }

cudaError_t dft_tc_build_table(void* table, int N, const void* tw, cudaStream_t st)
{
    const int H = folded_terms(N), NQ = 16 * ((H + 15) / 16), n = 4 * NQ * 8;
    build_table_kernel<<<(n + 127) / 128, 128, 0, st>>>((unsigned char*)table, N, H, NQ, (const double2*)tw);
    return cudaGetLastError();
}

cudaError_t launch_dft_tc_grid_pass(const void* in, void* out, long long nf, int N, int pass, bool real,
                                    const void* table, int* err, cudaStream_t st)
{
    Geo g;
    if (!dft_tc_supported(N) || !geometry(g, in, out, nf, N, pass, real, table)) return cudaErrorInvalidValue;
    if (pass == 2 || pass == -2) return run<COMPLEX, false>(g, err, st);
    if (!real) return run<COMPLEX, true>(g, err, st);
    return pass == 1 ? run<REAL_IN, true>(g, err, st) : run<REAL_OUT, true>(g, err, st);
}

cudaError_t dft_tc_batch_create(DftTcBatch& b, const std::vector<DftTcBucket>& buckets, bool real)
{
    const size_t n = buckets.size();
    std::vector<Geo> segs(4 * n);
    b.real = real;
    b.nseg = (int)n;
    for (int d = 0; d < 2; ++d)
        for (int pass = 0; pass < 2; ++pass) {
            unsigned long long tiles = 0;
            for (size_t i = 0; i < n; ++i) {
                const DftTcBucket& k = buckets[i];
                Geo& g = segs[(2 * d + pass) * n + i];
                const size_t off = (size_t)k.g0 * (real ? 4 : 8);
                const int which = d == 0 ? pass + 1 : pass - 2;
                if (!dft_tc_batch_supported(k.N) ||
                    !geometry(g, which == 1 ? (const void*)off : which == -1 || which == 2 ? (const void*)k.work : k.pencil,
                              which == -1 ? (void*)off : which == 2 ? (void*)k.pencil : (void*)k.work, k.nf, k.N, which, real,
                              k.table))
                    return cudaErrorInvalidValue;
                g.ext = which == 1 ? 1 : which == -1 ? 2 : 0;
                g.tile0 = (unsigned)tiles;
                tiles += g.ntiles;
                b.KCmax = std::max(b.KCmax, g.KC);
            }
            if (tiles > 0x7fffffffULL) return cudaErrorInvalidValue;
            b.ntiles[d][pass] = (unsigned)tiles;
        }
    cudaError_t e = cudaMalloc(&b.segs, sizeof(Geo) * segs.size());
    if (e == cudaSuccess) e = cudaMemcpy(b.segs, segs.data(), sizeof(Geo) * segs.size(), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&b.bar, 2 * sizeof(unsigned));
    if (e == cudaSuccess) e = cudaMemset(b.bar, 0, 2 * sizeof(unsigned));
    return e;
}

void dft_tc_batch_destroy(DftTcBatch& b)
{
    if (b.segs) cudaFree(b.segs);
    if (b.bar) cudaFree(b.bar);
    b = DftTcBatch();
}

cudaError_t launch_dft_tc_batch(const DftTcBatch& b, bool fwd, const void* in, void* out, int* err, cudaStream_t st)
{
    auto kern = fwd ? (b.real ? dft_tc_kernel<BATCH_FWD, REAL_IN, true> : dft_tc_kernel<BATCH_FWD, COMPLEX, true>)
                    : (b.real ? dft_tc_kernel<BATCH_INV, REAL_OUT, true> : dft_tc_kernel<BATCH_INV, COMPLEX, true>);
    int nsm = 0;
    cudaError_t e = device_sms(nsm);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(4));
    if (e != cudaSuccess) return e;
    const int d = fwd ? 0 : 1;
    Args a = {};
    for (int p = 0; p < 2; ++p) {
        a.segs[p] = reinterpret_cast<const Geo*>(b.segs) + (size_t)(2 * d + p) * b.nseg;
        a.ntiles[p] = b.ntiles[d][p];
    }
    a.nseg = b.nseg;
    a.KCmax = b.KCmax;
    a.ext = fwd ? (char*)const_cast<void*>(in) : (char*)out;
    a.bar = b.bar;
    a.err = err;
    // one CTA an SM (shared memory), all of them resident: they wait for one another between the passes
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.gridDim = dim3(std::min(std::max(a.ntiles[0], a.ntiles[1]), (unsigned)nsm));
    cfg.blockDim = dim3(THREADS);
    cfg.dynamicSmemBytes = smem_bytes(b.KCmax);
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, a);
}

}  // namespace fftso3
