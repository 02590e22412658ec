// The direct DFT of even length N = 2P on the tcgen05 tensor cores, for the passes of the SO(3) grid transforms whose N
// the register FFT does not serve.
//
// A line folds twice into four real problems of H = P/2 + 1 terms (direct_dft.cuh has the identities):
//   C[q] = sum_t u_t cos(2 pi t q / N), S[q] = sum_t v_t sin(2 pi t q / N), for the even and the odd q <= P,
//   X[q], X[N - q] = C[q] -/+ i S[q].
// Each is a product of 128 rows (64 complex lines x re / im, or 128 real lines) with a constant matrix of the plan's N: the
// lines' folded terms are the A operand (128 x H, K-major), the matrix the B operand, both as three BF16 terms (24
// significant bits) with the six products of weight >= 2^-16 accumulated in FP32 (the leading one apart from the five
// small ones), as the beta-sum does it.
//
// Why: as FP32 register tiles (direct_dft.cu) the products and the loads take turns on the same warps: 1.1 to 1.2 ms a pass
// at N = 194 (16 complex functions).  Here one thread issues them and the warps only move data: 0.43 ms (0.55 ms the
// transposing passes), 0.24 to 0.38 ms real.  Roles of the one CTA an SM holds:
//   warps 0-13   producers: load a line's elements t, N - t, P - t, P + t for eight t, fold, split, store the K-major
//                swizzled rows, one problem at a time into a ring of two 48 KB slots (the folded values wait in registers);
//   warps 14-17  epilogue, one TMEM lane quarter each: C and S -> X[q], X[N - q] -> global memory;
//   warp 18      MMA issuer (and TMEM owner).
// The matrices (at most 96 KB) stay in shared memory.  Accumulators: two buffers (even and odd q) of C and S, hi and lo.
// Bound: a 64-line tile takes 12 k cycles at N = 194, of which its bytes need 8.6 k (16 a complex sample and pass at
// 6.8 TB/s) and its 80 MMAs 6 k; the rest is the producers' load latency, which 96 registers a thread cannot cover further
// (64 hold the folded values), and instruction issue (53% of the slots).  Eight epilogue warps with a register split
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

// Below, the FP32 kernel: with few terms a tile's fixed latencies outweigh its products (all four passes, complex / real, ms:
// N = 66, 64 functions 0.52 / 0.40 here, 0.53 / 0.32 there; N = 160, 16 functions 1.00 / 0.70 here, 2.44 / 1.33 there).
constexpr int MINN = 80;

enum { COMPLEX = 0, REAL_IN = 1, REAL_OUT = 2 };

struct Args {
    const void* in;
    void* out;
    const unsigned char* table;
    int* err;
    int N, H, KC;        // folded terms, 16-wide K steps (also 16-wide blocks of outputs)
    unsigned ntiles;
    // straight passes: lines (f, o, u), u < N contiguous on both sides, o < no (skipping o == skip)
    // transposing: lines (f, x, y), x contiguous in the input, y in the output
    int no, skip;
    unsigned tx, ty;     // transposing: tiles along x and y
    unsigned nlines;     // straight: nf no N
    long long i_f, i_a, i_e;  // input: function, o (or y), element strides
    long long o_f, o_a, o_e;  // output: function, o (or x), element strides
    int nyq;             // element P is taken as zero
    int mirror;          // COMPLEX, straight: outputs of 0 < o < P also go conjugated to (N - o, N - q)
};

__host__ __device__ constexpr size_t smem_bytes(int KC) { return 2 * SLOT + 12 * 16 * KC * 128 + 128 + 1024; }

__device__ __forceinline__ void l2_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

__device__ __forceinline__ uint32_t bf2(float a, float b)
{
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
// eight values into one 16-byte chunk of each of the three BF16 planes
__device__ __forceinline__ void store_split(uint32_t dst, const float* x)
{
    uint32_t w[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        float a = x[2 * j], b = x[2 * j + 1];
#pragma unroll
        for (int p = 0; p < 3; ++p) {
            w[p][j] = bf2(a, b);
            a -= __uint_as_float(w[p][j] << 16);
            b -= __uint_as_float(w[p][j] & 0xffff0000u);
        }
    }
#pragma unroll
    for (int p = 0; p < 3; ++p)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + p * PLANE), "r"(w[p][0]), "r"(w[p][1]),
                     "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
}

// A line of a tile: its place in the input and the output (elements of the side's type), and whether it exists.
struct Line {
    long long in, out;
    int o;       // straight: the outer index
    bool ok;
};
// Straight tile: line number l of 64 (complex).  Transposing: l = (x, y) of the tile.
template <int KIND, bool TR>
__device__ __forceinline__ Line line_of(const Args& a, unsigned tile, int x, int y)
{
    Line r;
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
template <int KIND, bool EDGE, int VPL>
__device__ __forceinline__ void load_fold(const Args& a, long long in, int t0, int H, int N, float (&x)[4][VPL])
{
    const int P = N / 2;
    if (KIND == COMPLEX) {
        const float2* g = reinterpret_cast<const float2*>(a.in) + in;
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
            y[0][k] = in0 ? __ldg(p0) : z;
            y[1][k] = in0 && pos ? __ldg(p1) : z;
            y[2][k] = in0 && two && (pos || !a.nyq) ? __ldg(p2) : z;
            y[3][k] = in0 && two && pos ? __ldg(p3) : z;
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
        const float* g = reinterpret_cast<const float*>(a.in) + in;
        const float* p0 = g + t0 * a.i_e;
        const float* p1 = g + (N - t0) * a.i_e;
        const float* p2 = g + (P - t0) * a.i_e;
        const float* p3 = g + (P + t0) * a.i_e;
#pragma unroll
        for (int k = 0; k < 8; ++k, p0 += a.i_e, p1 -= a.i_e, p2 -= a.i_e, p3 += a.i_e) {
            const int t = t0 + k;
            const bool in0 = !EDGE || t < H, two = !EDGE || 2 * t != P, pos = !EDGE || t > 0;
            x[0][k] = in0 ? __ldg(p0) : 0.f;
            x[1][k] = in0 && pos ? __ldg(p1) : 0.f;
            x[2][k] = in0 && two ? __ldg(p2) : 0.f;
            x[3][k] = in0 && two && pos ? __ldg(p3) : 0.f;
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
        const float2* g = reinterpret_cast<const float2*>(a.in) + in;
        const float2* p0 = g + t0 * a.i_e;
        const float2* p2 = g + (P - t0) * a.i_e;
        const float2 z = make_float2(0.f, 0.f);
        float2 y[2][8];
#pragma unroll
        for (int k = 0; k < 8; ++k, p0 += a.i_e, p2 -= a.i_e) {
            const int t = t0 + k;
            y[0][k] = !EDGE || t < H ? __ldg(p0) : z;
            y[1][k] = !EDGE || (t < H && t > 0 && 2 * t != P) ? __ldg(p2) : z;
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
__device__ __forceinline__ void finish(const Args& a, const Line& L, uint32_t c, int q0, int nv, int part)
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
        char* o = reinterpret_cast<char*>(reinterpret_cast<float2*>(a.out) + L.out + q0 * a.o_e);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (FULL || i < nv) *reinterpret_cast<float2*>(o + (unsigned long long)i * step) = make_float2(C[i], S[i]);
        return;
    }
    constexpr int W = KIND == COMPLEX ? 2 : 1;  // floats: complex elements are two apart
    char* lo = reinterpret_cast<char*>(reinterpret_cast<float*>(a.out) + W * (L.out + q0 * a.o_e) + part);
    // the sixteenth output's mirror, from where the others ascend
    char* hi = reinterpret_cast<char*>(reinterpret_cast<float*>(a.out) + W * (L.out + (N - q0 - 30) * a.o_e) + part);
    const unsigned step = (unsigned)(8 * W * a.o_e);
    const int h0 = q0 == 0 ? 1 : 0, h1 = min(nv, (P - q0 + 1) >> 1);  // 0 < q < P
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (FULL || i < nv) *reinterpret_cast<float*>(lo + (unsigned long long)i * step) = C[i] + S[i];
#pragma unroll
    for (int i = 0; i < 16; ++i)
        if (FULL || (i >= h0 && i < h1)) *reinterpret_cast<float*>(hi + (unsigned long long)(15 - i) * step) = C[i] - S[i];
    if (KIND == COMPLEX && !TR && a.mirror && L.o > 0 && L.o < P) {
        // (o, q) -> (N - o, N - q) and (o, N - q) -> (N - o, q), conjugated
        const long long mo = 8 * (long long)(N - 2 * L.o) * a.o_a;
        const float sg = part ? -1.f : 1.f;
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (FULL || (i >= h0 && i < nv))
                *reinterpret_cast<float*>(hi + mo + (unsigned long long)(15 - i) * step) = sg * (C[i] + S[i]);
#pragma unroll
        for (int i = 0; i < 16; ++i)
            if (FULL || i < h1) *reinterpret_cast<float*>(lo + mo + (unsigned long long)i * step) = sg * (C[i] - S[i]);
    }
}

template <int KIND, bool TR>
__global__ void __launch_bounds__(THREADS, 1) dft_tc_kernel(const __grid_constant__ Args a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int KC = a.KC, NQ = 16 * KC, H = a.H, N = a.N, P = N / 2;
    unsigned char* bmat = smem + 2 * SLOT;  // [problem][plane][q][t], K-major swizzled rows of 128 bytes
    const int BPLANE = NQ * 128;
    uint64_t* full = (uint64_t*)(bmat + 12 * BPLANE);
    uint64_t* empty = full + 2;
    uint64_t* accf = empty + 2;
    uint64_t* acce = accf + 2;
    uint64_t* bfull = acce + 2;  // the matrices have arrived
    uint32_t* tmem_slot = (uint32_t*)(bfull + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], NPROD);
            mbar_init(&empty[s], 1);
            mbar_init(&accf[s], 1);
            mbar_init(&acce[s], NEPI);
        }
        mbar_init(bfull, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMAW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // the slots' columns past the folded terms stay zero
    for (int i = threadIdx.x; i < 2 * SLOT / 16; i += THREADS) reinterpret_cast<uint4*>(smem)[i] = make_uint4(0, 0, 0, 0);
    if (threadIdx.x == 0) {
        mbar_expect_tx(bfull, 12 * BPLANE);
        bulk_load(bmat, a.table, 12 * BPLANE, bfull);
    }
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp < NPROD) {
        // ---------------- producers: an item is 32 lines x 8 folded terms
        constexpr int VPL = KIND == COMPLEX ? 16 : 8;  // values of a problem held by an item's thread (8 t, re and im)
        constexpr int IPW = KIND == COMPLEX ? 1 : 2;   // items of a warp
        constexpr int LB = KIND == COMPLEX ? 2 : 4;    // blocks of 32 lines in a tile
        const int nitems = LB * ((H + 7) / 8);
        int lx[IPW], ly[IPW], ch[IPW], row[IPW];
#pragma unroll
        for (int w = 0; w < IPW; ++w) {
            const int it = warp + w * NPROD, lb = it % LB;
            ch[w] = it < nitems ? it / LB : -1;
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
        }
        unsigned s = 0;  // problems produced so far
        for (unsigned tile = blockIdx.x; tile < a.ntiles && !*abort_flag; tile += gridDim.x) {
            float v[IPW][4][VPL];  // [problem][t (re), then t (im)]
#pragma unroll
            for (int w = 0; w < IPW; ++w) {
                if (ch[w] < 0) continue;
                const Line L = line_of<KIND, TR>(a, tile, lx[w], ly[w]);
                const int t0 = 8 * ch[w];
                float (&x)[4][VPL] = v[w];
                if (!L.ok) {
#pragma unroll
                    for (int k = 0; k < VPL; ++k) x[0][k] = x[1][k] = x[2][k] = x[3][k] = 0.f;
                } else if (t0 > 0 && t0 + 8 <= H && 2 * (t0 + 7) != P) {
                    load_fold<KIND, false>(a, L.in, t0, H, N, x);
                } else {
                    load_fold<KIND, true>(a, L.in, t0, H, N, x);
                }
            }
            // the next tile's elements into L2 while this one's problems are stored and multiplied: lane k of a run of
            // eight lines requests the run's element t0 + k (and its three images)
            if (tile + gridDim.x < a.ntiles) {
#pragma unroll
                for (int w = 0; w < IPW; ++w) {
                    const int k = 8 * ch[w] + (lane & 7);
                    if (ch[w] < 0 || k >= H) continue;
                    const Line L = line_of<KIND, TR>(a, tile + gridDim.x, lx[w], ly[w]);
                    if (!L.ok) continue;
                    constexpr int E = KIND == REAL_IN ? 4 : 8;
                    const char* g = reinterpret_cast<const char*>(a.in) + E * (L.in - (lane & (KIND == REAL_IN ? 15 : 7)));
                    const long long e = E * a.i_e;
                    l2_prefetch(g + k * e);
                    l2_prefetch(g + (P - k) * e);
                    if (KIND != REAL_OUT && k > 0) {
                        l2_prefetch(g + (N - k) * e);
                        l2_prefetch(g + (P + k) * e);
                    }
                }
            }
            bool ok = true;
#pragma unroll
            for (int pr = 0; pr < 4; ++pr, ++s) {
                const int sl = s & 1;
                if (s >= 2 && !mbar_wait(&empty[sl], ((s >> 1) - 1) & 1, a.err, 31)) {
                    ok = false;
                    break;
                }
#pragma unroll
                for (int w = 0; w < IPW; ++w) {
                    if (ch[w] < 0) continue;
                    const uint32_t d = smem_u32(smem + sl * SLOT) + row[w] * 128 + ((ch[w] ^ (row[w] & 7)) << 4);
                    store_split(d, v[w][pr]);
                    if (KIND == COMPLEX) store_split(d + 8 * 128, v[w][pr] + 8);
                }
                fence_proxy_async();
                __syncwarp();
                if (lane == 0) mbar_arrive(&full[sl]);
            }
            if (!ok) {
                *abort_flag = 1;
                break;
            }
        }
    } else if (warp == MMAW) {
        if (elect_one()) {
            // ---------------- MMA issuer
            const uint32_t id1 = idesc_bf16_mn(false, NQ, 128), id2 = idesc_bf16_mn(false, 2 * NQ, 128);
            const uint32_t sa = smem_u32(smem), sb = smem_u32(bmat);
            unsigned s = 0;
            bool ok = mbar_wait(bfull, 0, a.err, 34);
            for (unsigned tile = blockIdx.x; tile < a.ntiles && ok && !*abort_flag; tile += gridDim.x) {
                for (int pr = 0; pr < 4; ++pr, ++s) {
                    const int sl = s & 1, ab = (s >> 1) & 1;  // accumulator buffer: alternates with the parity of q
                    if ((pr & 1) == 0 && s >= 4 && !mbar_wait(&acce[ab], ((s >> 2) - 1) & 1, a.err, 32)) {
                        ok = false;
                        break;
                    }
                    if (!mbar_wait(&full[sl], (s >> 1) & 1, a.err, 33)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t hi = tmem + ab * 256 + (pr & 1) * 128, lo = hi + NQ;
                    const uint32_t A = sa + sl * SLOT, B = sb + pr * 3 * BPLANE;
                    // descriptors: 16-byte units in the low bits, 32 bytes of K a step
                    uint64_t ad = smem_desc(A, 16, 1024), bd = smem_desc(B, 16, 1024);
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
                    mma_commit(&empty[sl]);
                    if (pr & 1) mma_commit(&accf[ab]);
                }
            }
            if (!ok) *abort_flag = 1;
            // the last commits must land before TMEM is freed: buffer b was committed (s + 2 - 2 b) / 4 times
            for (int b = 0; b < 2; ++b) {
                const unsigned n = (s + 2 - 2 * b) / 4;
                if (n > 0) mbar_wait(&accf[b], (n - 1) & 1, a.err, 36);
            }
        }
    } else {
        // ---------------- epilogue
        const int quarter = warp & 3, r = quarter * 32 + lane;
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
        unsigned s = 0;  // accumulator buffers consumed so far
        bool ok = true;
        for (unsigned tile = blockIdx.x; tile < a.ntiles && ok && !*abort_flag; tile += gridDim.x) {
            const Line L = line_of<KIND, TR>(a, tile, x, y);
            const bool all = __all_sync(0xffffffffu, L.ok);
            for (int par = 0; par < 2; ++par, ++s) {
                const int ab = s & 1;
                if (!mbar_wait(&accf[ab], (s >> 1) & 1, a.err, 35)) {
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16) + ab * 256;
                const int nq = (P - par) / 2 + 1;  // outputs of this parity
                for (int b = 0; 16 * b < nq; ++b) {
                    const int q0 = 32 * b + par;
                    if (all && q0 > 0 && q0 + 30 < P)
                        finish<KIND, TR, true>(a, L, base + 16 * b, q0, 16, part);
                    else
                        finish<KIND, TR, false>(a, L, base + 16 * b, q0, L.ok ? nq - 16 * b : 0, part);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(&acce[ab]);
            }
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == MMAW) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
    }
}

// [problem: cos even, sin even, cos odd, sin odd][plane][q][t] BF16, rows of 128 bytes, their 16-byte chunks swizzled; one
// thread a chunk (eight t of the three planes).  The terms are split from the FP64 values.
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
            w[p][j] = bf2((float)v[0], (float)v[1]);
            v[0] -= (double)__uint_as_float(w[p][j] << 16);
            v[1] -= (double)__uint_as_float(w[p][j] & 0xffff0000u);
        }
    }
    unsigned char* d = table + (size_t)pr * 3 * NQ * 128 + qi * 128 + ((c ^ (qi & 7)) << 4);
#pragma unroll
    for (int p = 0; p < 3; ++p)
        *reinterpret_cast<uint4*>(d + (size_t)p * NQ * 128) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

template <int KIND, bool TR>
static cudaError_t run(const Args& a, cudaStream_t st)
{
    auto kern = dft_tc_kernel<KIND, TR>;
    const size_t smem = smem_bytes(a.KC);
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes(4));
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    kern<<<std::min(a.ntiles, (unsigned)nsm), THREADS, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace dtc

using namespace dtc;

bool dft_tc_supported(int N) { return N >= MINN && N % 2 == 0 && N / 4 + 1 <= MAXH; }

static int folded_terms(int N) { return N / 4 + 1; }
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
    if (!dft_tc_supported(N) || nf < 1) return cudaErrorInvalidValue;
    const long long n = N, NN = n * n;
    const int P = N / 2;
    Args a = {};
    a.in = in;
    a.out = out;
    a.table = (const unsigned char*)table;
    a.err = err;
    a.N = N;
    a.H = folded_terms(N);
    a.KC = (a.H + 15) / 16;
    a.i_f = a.o_f = NN * n;
    a.skip = -1;
    if (nf * NN > 0x7fffffffLL) return cudaErrorInvalidValue;
    auto blocks = [&](int b) { return (unsigned)((N + b - 1) / b); };
    switch (pass) {
        case 1:  // x = j2, y = k
            a.tx = blocks(real ? 16 : 8);
            a.ty = blocks(8);
            a.i_a = NN;
            a.i_e = n;
            a.o_a = n;
            a.o_e = NN;
            a.ntiles = (unsigned)nf * a.tx * a.ty;
            return real ? run<REAL_IN, true>(a, st) : run<COMPLEX, true>(a, st);
        case 2:
        case -2:  // o = p, lines along k
            a.i_a = a.o_a = NN;
            a.i_e = a.o_e = n;
            a.nyq = pass < 0;
            a.mirror = pass > 0 && real;
            if (pass > 0) {
                a.no = real ? P + 1 : N;
            } else {
                a.no = real ? P : N - 1;  // without the Nyquist row p = P
                a.skip = real ? -1 : P;
            }
            a.nlines = (unsigned)(nf * a.no * n);
            a.ntiles = (a.nlines + 63) / 64;
            return run<COMPLEX, false>(a, st);
        case -1:  // x = k, y = j2
            a.tx = blocks(8);
            a.ty = blocks(real ? 16 : 8);
            a.nyq = 1;
            a.i_a = n;
            a.i_e = NN;
            a.o_a = NN;
            a.o_e = n;
            a.ntiles = (unsigned)nf * a.tx * a.ty;
            return real ? run<REAL_OUT, true>(a, st) : run<COMPLEX, true>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace fftso3
