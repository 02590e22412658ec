// Register-resident FP32 FFT kernels for the tensor-core path, N = 32 R
// (R = 2..32, i.e. N = 64..1024, powers of two).
//
// Kernels:
//   fft_tile      a tile of 16 lines with one side contiguous and the other transposed, so a 2-D transform of
//                 the Euler grid is two passes that both read and write whole 128-byte runs, the second one
//                 producing the k-contiguous pencils [fn][p][q][k] the beta-sum GEMM consumes (and the reverse
//                 for the inverse); each line in two in-register DFTs around one exchange through shared memory,
//                 which also transposes the tile;
//   fft_grid2d    both passes of the Euler grid in one persistent launch, through an L2-resident ring.
// Bound: latency and the loads in flight (N = 256: 55 % of the L1's and 50 % of DRAM's rate).  With the line FFT over a warp's
// lanes (radix-2 butterflies with loaded twiddles, two exchanges and a shuffle stage, the tile staged in shared memory besides)
// a sample took 75 instructions a pass and the L1 was at 71 to 86 %: l_max 127, 16 functions, 1.61 and 1.72 ms a direction
// against 1.05 and 1.04 (268 M samples; DRAM's floor 0.63), l_max 63, 64 real functions 0.65 and 0.71 against 0.33 and 0.37,
// S^2 l_max 511, 512 real functions 0.94 and 0.97 against 0.84 and 0.82.
#include <algorithm>
#include <cstdlib>

#include "common.cuh"
#include "fft.cuh"
#include "fft_tile_layout.h"

namespace fftso3 {

namespace ffast {

constexpr unsigned FULL = 0xffffffffu;

__host__ __device__ constexpr int brev(int x, int bits)
{
    int r = 0;
    for (int b = 0; b < bits; ++b) r |= ((x >> b) & 1) << (bits - 1 - b);
    return r;
}

__host__ __device__ constexpr int ilog2(int x) { return x <= 1 ? 0 : 1 + ilog2(x >> 1); }

__device__ __forceinline__ float2 cmulf(float2 a, float2 b)
{
    return make_float2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}

// cos(2 pi k / 32)
__host__ __device__ constexpr float cos32(int k)
{
    constexpr double c[9] = {1.0, 0.98078528040323044913, 0.92387953251128675613, 0.83146961230254523708,
                             0.70710678118654752440, 0.55557023301960222474, 0.38268343236508977173,
                             0.19509032201612826785, 0.0};
    k &= 31;
    if (k > 16) k = 32 - k;
    return k <= 8 ? (float)c[k] : -(float)c[16 - k];
}

// d w, w = e^{-2 pi i e / 32} a literal
__device__ __forceinline__ float2 twiddle32(float2 d, int e)
{
    if (e == 0) return d;
    if (e == 8) return make_float2(d.y, -d.x);
    return cmulf(d, make_float2(cos32(e), -cos32(e - 8)));
}

// P-point DIF in registers with literal twiddles (P <= 32; natural input, bit-reversed output): radix-4 stages, which round
// once less between twiddles than pairs of radix-2 ones, and a last radix-2 one for P = 8, 32.
template <int P>
__device__ __forceinline__ void reg_dft(float2 (&v)[P])
{
#pragma unroll
    for (int n = P; n >= 4; n >>= 2) {
        const int q = n / 4;
#pragma unroll
        for (int j = 0; j < P; j += n) {
#pragma unroll
            for (int k = 0; k < q; ++k) {
                const float2 a = v[j + k], b = v[j + k + q], c = v[j + k + 2 * q], d = v[j + k + 3 * q];
                const float2 s = make_float2(a.x + c.x, a.y + c.y), t = make_float2(b.x + d.x, b.y + d.y);
                const float2 m = make_float2(a.x - c.x, a.y - c.y), u = make_float2(b.x - d.x, b.y - d.y);
                const int e = 32 * k / n;
                v[j + k] = make_float2(s.x + t.x, s.y + t.y);
                v[j + k + q] = twiddle32(make_float2(s.x - t.x, s.y - t.y), 2 * e);
                v[j + k + 2 * q] = twiddle32(make_float2(m.x + u.y, m.y - u.x), e);
                v[j + k + 3 * q] = twiddle32(make_float2(m.x - u.y, m.y + u.x), 3 * e);
            }
        }
    }
    if (P == 8 || P == 32 || P == 2) {
#pragma unroll
        for (int j = 0; j < P; j += 2) {
            const float2 a = v[j], b = v[j + 1];
            v[j] = make_float2(a.x + b.x, a.y + b.y);
            v[j + 1] = make_float2(a.x - b.x, a.y - b.y);
        }
    }
}

// Threads of a tile's CTA and CTAs an SM (a thread has 8 to 16 values of N <= 256 a step, one or two 32-point DFTs, 64
// registers of values, of N >= 512).  Both directions, ms: N = 128, 64 real functions, 256 threads x 3 CTAs 1.19, 128 x 6 0.74;
// N = 256, 16 real functions, 256 x 3 1.48, 128 x 5 1.18, 128 x 6 1.20 (complex 2.20, 2.11); N = 1024 (S^2, 512 real
// functions) 256 x 2 1.65, 256 x 3 2.28, 128 x 3 1.94.
__host__ __device__ constexpr int tile_threads(int R) { return R <= 8 ? 128 : 256; }
__host__ __device__ constexpr int tile_ctas(int R) { return R <= 2 ? 8 : R <= 4 ? 6 : R <= 8 ? 5 : 2; }

// Twiddles in shared memory: W[k1 B + j2] = w_N^{j2 k1}.
template <int R, bool C2T>
__device__ __forceinline__ void load_tile_twiddles(float2* W, const double2* __restrict__ tw)
{
    constexpr int N = 32 * R, B = rad_b<R, C2T>();
    for (int i = threadIdx.x; i < N; i += blockDim.x) {
        const int j = (i % B) * (i / B);
        W[i] = make_float2((float)tw[j].x, (float)tw[j].y);
    }
}
// Geometry of a tiled pass (element offsets).
struct TileGeo {
    long long FS;  // per function (N^3 for SO(3) grids, N^2 for S^2 grids)
    int NO;        // outer index range (N for SO(3), 1 for S^2)
    long long Oc, Ls, Ot, Js;
};

// Global-memory access modes of a tile's two sides.
//   IO_PLAIN:   read-only loads through the texture path, plain stores (one pass per launch);
//   IO_STREAM:  data touched once (grid, pencils): loads and stores marked first for L2 eviction;
//   IO_SCRATCH: the L2-resident ring between the two passes of a fused launch: stores marked last
//               for eviction, loads coherent at L2 (other CTAs of the same launch wrote them).
enum { IO_PLAIN = 0, IO_STREAM = 1, IO_SCRATCH = 2 };

__device__ __forceinline__ uint64_t l2_policy_first()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_last()
{
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}

template <int M>
__device__ __forceinline__ float ld1(const float* p, uint64_t pol)
{
    if constexpr (M == IO_PLAIN) return __ldg(p);
    else if constexpr (M == IO_SCRATCH) return __ldcg(p);
    else {
        float v;
        asm volatile("ld.global.nc.L2::cache_hint.f32 %0, [%1], %2;" : "=f"(v) : "l"(p), "l"(pol));
        return v;
    }
}
template <int M>
__device__ __forceinline__ float2 ld2(const float2* p, uint64_t pol)
{
    if constexpr (M == IO_PLAIN) return __ldg(p);
    else if constexpr (M == IO_SCRATCH) return __ldcg(p);
    else {
        float2 v;
        asm volatile("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;" : "=f"(v.x), "=f"(v.y) : "l"(p), "l"(pol));
        return v;
    }
}
template <int M>
__device__ __forceinline__ float4 ld4(const float4* p, uint64_t pol)
{
    if constexpr (M == IO_PLAIN) return __ldg(p);
    else if constexpr (M == IO_SCRATCH) return __ldcg(p);
    else {
        float4 v;
        asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;"
                     : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                     : "l"(p), "l"(pol));
        return v;
    }
}
template <int M>
__device__ __forceinline__ void st1(float* p, float v, uint64_t pol)
{
    if constexpr (M == IO_PLAIN) *p = v;
    else asm volatile("st.global.L2::cache_hint.f32 [%0], %1, %2;" ::"l"(p), "f"(v), "l"(pol) : "memory");
}
template <int M>
__device__ __forceinline__ void st2(float2* p, float2 v, uint64_t pol)
{
    if constexpr (M == IO_PLAIN) *p = v;
    else asm volatile("st.global.L2::cache_hint.v2.f32 [%0], {%1, %2}, %3;" ::"l"(p), "f"(v.x), "f"(v.y), "l"(pol)
                      : "memory");
}
template <int M>
__device__ __forceinline__ void st4(float4* p, float4 v, uint64_t pol)
{
    if constexpr (M == IO_PLAIN) *p = v;
    else asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;" ::"l"(p), "f"(v.x), "f"(v.y),
                      "f"(v.z), "f"(v.w), "l"(pol)
                      : "memory");
}
// Drop one 128-byte line from L2 without writing it back (its data is dead).
__device__ __forceinline__ void l2_discard(const void* p)
{
    asm volatile("discard.global.L2 [%0], 128;" ::"l"(p) : "memory");
}

// A tile of TL lines with one side contiguous and the other transposed.
//   contiguous side: line l, element j at  cbase + l * Ls + j
//   transposed side: line l, element j at  tbase + j * Js + l    (TL consecutive l)
// C2T = true reads the contiguous side and writes the transposed one; C2T =
// false the reverse.  Both sides move TL * 8 = 128-byte runs.
// REAL_IO: the contiguous side holds real values (pass 1 reads real samples,
// pass -1 writes the real part only).  IN / OUT: access modes (IO_*) of the
// side read and the side written; an IO_SCRATCH input is dropped from L2
// once the tile holds it (every line of the ring is read by exactly one tile).
// HALF (with REAL_IO): the transposed side holds the elements j < N / 2 alone; those past N / 2 are the conjugates of
// N - j, and j = N / 2 is zero (the Nyquist bin, which no coefficient maps to).
// nyq (transposed input): the elements j = N / 2 are taken as zero without being read; zero: all of them (complex lines).
// T: the exchange in shared memory; Ws: twiddles (staged, synchronised).
// mid(): run by every thread right after the barrier between the two halves of
// the tile (the input is consumed, no output written yet).
template <int R, bool C2T, bool REAL_IO, bool HALF, int IN, int OUT, typename MID>
__device__ __forceinline__ void tile_body(const float2* __restrict__ in, float2* __restrict__ out, long long cbase,
                                          long long tbase, long long Ls, long long Js, float2* T,
                                          const float2* Ws, uint64_t pol_in, uint64_t pol_out, MID mid, bool nyq = false,
                                          bool zero = false)
{
    constexpr int N = 32 * R, A = rad_a<R, C2T>(), B = rad_b<R, C2T>(), KS = tile_ks<R, C2T>();
    constexpr int LA = ilog2(A), LB = ilog2(B), NT = tile_threads(R);
    static_assert(!(REAL_IO && IN == IO_SCRATCH && C2T), "the ring holds complex lines");
    static_assert(!HALF || REAL_IO, "half of a real line's spectrum");
    // REAL_IO: real lines 2p and 2p+1 share one complex transform (row p):
    // forward z = x_{2p} + i x_{2p+1}, X = (Z[k] + conj Z[-k]) / 2, Y = (Z[k] - conj Z[-k]) / 2i;
    // inverse z = X_{2p} + i X_{2p+1} (spectra of real lines), lines = Re, Im of its transform.
    constexpr int ROWS = REAL_IO ? TL / 2 : TL;
#pragma unroll 1
    for (int u = threadIdx.x; u < ROWS * B; u += NT) {  // whole warps
        const TilePlace at = step1_place<R, C2T, REAL_IO>(u);
        const int l = at.l, j2 = at.x;
        float2 v[A];
        if (C2T && REAL_IO) {
            const float* s0 = reinterpret_cast<const float*>(in) + cbase + (2 * l) * Ls + j2;
            const float* s1 = s0 + Ls;
#pragma unroll
            for (int i = 0; i < A; ++i) v[i] = make_float2(ld1<IN>(s0 + B * i, pol_in), ld1<IN>(s1 + B * i, pol_in));
        } else if (C2T) {
            const float2* src = in + cbase + l * Ls + j2;
#pragma unroll
            for (int i = 0; i < A; ++i) v[i] = ld2<IN>(src + B * i, pol_in);
        } else if (!REAL_IO) {
            const float2* src = in + tbase + j2 * Js + l;
#pragma unroll
            for (int i = 0; i < A; ++i)
                v[i] = zero || (i == A / 2 && nyq && j2 == 0) ? make_float2(0.f, 0.f)
                                                              : ld2<IN>(src + (long long)(B * i) * Js, pol_in);
        } else {
            constexpr int AL = HALF ? A / 2 : A;
            const float4* src = reinterpret_cast<const float4*>(in) + (tbase + j2 * Js + 2 * l) / 2;
            float4 x[AL];
#pragma unroll
            for (int i = 0; i < AL; ++i)
                x[i] = i == A / 2 && nyq && j2 == 0 ? make_float4(0.f, 0.f, 0.f, 0.f)
                                                    : ld4<IN>(src + (long long)(B * i) * Js / 2, pol_in);
#pragma unroll
            for (int i = 0; i < AL; ++i) v[i] = make_float2(x[i].x - x[i].w, x[i].y + x[i].z);
            if (HALF) {
                // elements past N / 2: those of N - j with conjugate spectra, held by the neighbour B - j2
                if (j2 == 0) v[0] = make_float2(x[0].x, x[0].z);
#pragma unroll
                for (int i = A / 2; i < A; ++i) {
                    const float4 o = x[A - 1 - i], q = i > A / 2 ? x[A - i] : make_float4(0.f, 0.f, 0.f, 0.f);
                    const float2 own = make_float2(o.x + o.w, o.z - o.y);
                    const float2 oth = make_float2(__shfl_xor_sync(FULL, own.x, ROWS), __shfl_xor_sync(FULL, own.y, ROWS));
                    v[i] = j2 == 0 ? make_float2(q.x + q.w, q.z - q.y) : 2 * j2 == B ? own : oth;
                }
            }
        }
        reg_dft<A>(v);
        float2* S = T + step1_slot<R, C2T>(at, 0);
#pragma unroll
        for (int r = 0; r < A; ++r) {
            const int k1 = brev(r, LA);
            S[k1 * KS] = r == 0 ? v[r] : cmulf(v[r], Ws[k1 * B + j2]);
        }
    }
    __syncthreads();
    mid();
    if (IN == IO_SCRATCH && C2T)
        for (int i = threadIdx.x; i < TL * (N / 16); i += NT)
            l2_discard(in + cbase + (long long)(i / (N / 16)) * Ls + (i % (N / 16)) * 16);
    if (IN == IO_SCRATCH && !C2T)
        for (int j = threadIdx.x; j < (HALF ? N / 2 : N); j += NT) l2_discard(in + tbase + (long long)j * Js);
#pragma unroll 1
    for (int u = threadIdx.x; u < ROWS * A; u += NT) {
        const TilePlace at = step2_place<R, C2T, REAL_IO>(u);
        const int l = at.l, k1 = at.x;
        float2 v[B];
        const float2* S = T + step2_slot<R, C2T>(at, 0);
#pragma unroll
        for (int j = 0; j < B; ++j) v[j] = S[j];
        reg_dft<B>(v);
        if (C2T && REAL_IO) {
            float4* dst = reinterpret_cast<float4*>(out) + (tbase + k1 * Js + 2 * l) / 2;
#pragma unroll
            for (int k2 = 0; k2 < (HALF ? B / 2 : B); ++k2) {
                // Z[N - K]: the neighbour A - k1's B - 1 - k2
                const float2 z = v[brev(k2, LB)], own = v[brev(B - 1 - k2, LB)], own0 = v[brev((B - k2) % B, LB)];
                const float2 oth = make_float2(__shfl_xor_sync(FULL, own.x, ROWS), __shfl_xor_sync(FULL, own.y, ROWS));
                const float2 zm = k1 == 0 ? own0 : 2 * k1 == A ? own : oth;
                st4<OUT>(dst + (long long)(A * k2) * Js / 2,
                         make_float4(0.5f * (z.x + zm.x), 0.5f * (z.y - zm.y), 0.5f * (z.y + zm.y), -0.5f * (z.x - zm.x)),
                         pol_out);
            }
        } else if (C2T) {
            float2* dst = out + tbase + k1 * Js + l;
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) st2<OUT>(dst + (long long)(A * k2) * Js, v[brev(k2, LB)], pol_out);
        } else if (REAL_IO) {
            float* d0 = reinterpret_cast<float*>(out) + cbase + (2 * l) * Ls + k1;
            float* d1 = d0 + Ls;
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) {
                st1<OUT>(d0 + A * k2, v[brev(k2, LB)].x, pol_out);
                st1<OUT>(d1 + A * k2, v[brev(k2, LB)].y, pol_out);
            }
        } else {
            float2* dst = out + cbase + l * Ls + k1;
#pragma unroll
            for (int k2 = 0; k2 < B; ++k2) st2<OUT>(dst + A * k2, v[brev(k2, LB)], pol_out);
        }
    }
}

// One pass over nf functions: the CTA index splits into (f, o < NO, bb < N / TL),
// cbase = f FS + o Oc + bb TL Ls, tbase = f FS + o Ot + bb TL.
template <int R, bool C2T, bool REAL_IO, bool HALF>
__global__ void __launch_bounds__(tile_threads(R), tile_ctas(R)) fft_tile(const float2* __restrict__ in, float2* __restrict__ out,
                                                        const TileGeo g, bool nyq, const double2* __restrict__ tw)
{
    constexpr int N = 32 * R;
    extern __shared__ float2 smem_f2[];
    float2* Ws = smem_f2;
    float2* T = smem_f2 + 32 * R;
    load_tile_twiddles<R, C2T>(Ws, tw);
    constexpr int NB = N / TL;
    const long long b = blockIdx.x;
    const long long f = b / ((long long)g.NO * NB);
    const long long o = (b / NB) % g.NO;
    const long long bb = b % NB;
    const long long cbase = f * g.FS + o * g.Oc + bb * TL * g.Ls;
    const long long tbase = f * g.FS + o * g.Ot + bb * TL;
    __syncthreads();  // twiddles staged
    tile_body<R, C2T, REAL_IO, HALF, IO_PLAIN, IO_PLAIN>(in, out, cbase, tbase, g.Ls, g.Js, T, Ws, 0, 0, [] {}, nyq,
                                                          nyq && g.NO > 1 && o == N / 2);
}

// ---------------------------------------------------------------------------
// Both passes of one direction of the SO(3) grid transform in one persistent
// launch, with the intermediate held in an L2-resident ring instead of a
// full-size work grid.
//
// The batch splits into chunks c = (f, kb): the TL consecutive beta slices
// k = kb TL + kl of function f.  Phase A of a chunk is the first pass over
// those slices into ring slot c mod S (N tiles), phase B the second pass out
// of the slot (N tiles):
//   forward  A: grid slice rows  -> FFT over j2 -> slot [kl][q][j1]       (tile = (kl, bb))
//            B: slot rows (kl, q) -> FFT over j1 -> pencils [f][p][q][kb TL + kl] (tile = q)
//   inverse  A: pencils            -> FFT over p  -> slot [kl][q][j1]     (tile = q)
//            B: slot              -> FFT over q  -> grid slice rows       (tile = (kl, bb))
// Every phase-B tile needs every phase-A tile of its chunk (a transpose), and
// phase A of chunk c reuses the slot of chunk c - S.  CTAs claim tiles from
// one atomic counter in the order (blocks of N tiles, lookahead D)
//   A(0), ..., A(D-1), A(D), B(0), A(D+1), B(1), ..., B(C-1)
// so a phase-B tile's producers were claimed at least D + 1 blocks earlier
// and a slot is reused 2 (S - D) - 1 blocks after its last reader was claimed;
// D and S are chosen from the number of resident CTAs (several tiles per CTA
// are claimed but not yet published at any time) so that dependencies are
// normally complete when checked, while only about D + 1 slots hold live data
// (the rest were dropped from L2 as they were read).  At N = 512 D stays 1 so
// that the live 32 MB slots fit in L2; about a third of the tiles then find
// their dependency incomplete at the first check (a larger D was measured
// slower).  Every tile waits only on tiles claimed before it, by CTAs that are
// running or done, so the launch cannot deadlock and needs no co-residency;
// waits are bounded, and on timeout the launch records an error and every CTA
// stops at its next wait.
//
// Control (thread 0 of each CTA), kept off the critical path where it can be:
// the claim of the tile after next is issued when a tile starts and the next
// tile's dependency counter is read then too, with an acquire load; at the
// tile's middle barrier (its input consumed) one release reduction publishes
// the previous tile, so a tile costs two barriers and no fence (the form with
// one fence.acq_rel for both, and relaxed operations, measured 0.3% slower).
// A dependency still incomplete at that point is read again at the end of the
// tile (one fence if it has completed); only if it is still incomplete is the
// current tile published first, then waited for.
constexpr long long WAIT_LIMIT = 4000000000LL;  // clock64 cycles (~2 s)

struct Grid2DArgs {
    const float2* in;
    float2* out;
    float2* ring;    // nslots slots of TL N^2 complex64
    int* ctl;        // [0] next tile, [1] abort, [2, 2 + C) phase-A done per chunk, [2 + C, 2 + 2C) phase-B done
    int* err;        // first error code (9: dependency wait timed out)
    int nchunks;     // C = nf * N / TL
    int look;        // D
    int nslots;      // S
    int nyq;         // inverse: the Nyquist bins p = N / 2 and q = N / 2 are zero, not read
    int prefetch;    // 1: prefetch the next claimed phase-A tile's input into L2 at each middle barrier
};

__device__ __forceinline__ int ld_relaxed(const int* p)
{
    int v;
    asm volatile("ld.relaxed.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ int ld_acquire(const int* p)
{
    int v;
    asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
    return v;
}
__device__ __forceinline__ void red_add_release(int* p, int v)
{
    asm volatile("red.release.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void fence_gpu() { asm volatile("fence.acq_rel.gpu;" ::: "memory"); }
__device__ __forceinline__ void red_add(int* p, int v)
{
    asm volatile("red.relaxed.gpu.global.add.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void prefetch_l2(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// Claim order -> (phase, chunk, tile within the phase); NA, NB: tiles of a chunk's phases.
template <int NA, int NB>
__device__ __forceinline__ void decode_task(int t, int C, int D, bool& phaseA, int& c, int& u)
{
    const int P = D < C ? D : C, Q = C > D ? C - D : 0;
    if (t < P * NA) {
        phaseA = true;
        c = t / NA;
        u = t - c * NA;
        return;
    }
    t -= P * NA;
    const int j = t / (NA + NB);
    if (j < Q) {
        u = t - j * (NA + NB);
        phaseA = u < NA;
        c = j + (phaseA ? D : 0);
        if (!phaseA) u -= NA;
        return;
    }
    t -= Q * (NA + NB);
    phaseA = false;
    c = Q + t / NB;
    u = t - (c - Q) * NB;
}

template <int R, bool FWD, bool REAL_IO, bool HALF>
__global__ void __launch_bounds__(tile_threads(R), tile_ctas(R)) fft_grid2d(const Grid2DArgs a, const double2* __restrict__ tw)
{
    constexpr int N = 32 * R;
    constexpr int NB = N / TL;
    constexpr long long N2 = (long long)N * N, N3 = N2 * N;
    extern __shared__ float2 smem_f2[];
    float2* Ws = smem_f2;
    float2* T = smem_f2 + 32 * R;
    __shared__ int s_cur[2], s_slow;
    __shared__ const char* s_pf;  // input of the next tile to prefetch into L2 (null: none)
    load_tile_twiddles<R, FWD>(Ws, tw);
    const uint64_t pol_stream = l2_policy_first(), pol_keep = l2_policy_last();
    const int C = a.nchunks, D = a.look, S = a.nslots;
    // HALF: phase B forward / phase A inverse has the tiles q < N / 2 alone
    constexpr int TA = !FWD && HALF ? N / 2 : N, TB = FWD && HALF ? N / 2 : N;
    const int total = C * (TA + TB);
    int* const abort_flag = a.ctl + 1;
    int* const doneA = a.ctl + 2;
    int* const doneB = a.ctl + 2 + C;

    // thread-0 control state
    int nxt = -1, pend = -1, prev = -1, dv = 0;
    const int* dptr = nullptr;  // dependency counter of nxt (null: none) ..
    int need = 0;               // .. and the count it waits for
    bool ready = true;
    // raw claim (checked against total where it is used, so the atomic's latency hides behind a tile)
    auto claim = [&]() -> int { return atomicAdd(a.ctl, 1); };
    auto valid = [&](int t) { return t < total ? t : -1; };
    auto dep_of = [&](int t) -> const int* {
        bool pa;
        int c, u;
        decode_task<TA, TB>(t, C, D, pa, c, u);
        need = pa ? TB : TA;
        if (pa) return c >= S ? doneB + (c - S) : nullptr;
        return doneA + c;
    };
    auto signal = [&](int t) {  // after a fence (release pattern)
        bool pa;
        int c, u;
        decode_task<TA, TB>(t, C, D, pa, c, u);
        red_add(pa ? doneA + c : doneB + c, 1);
    };
    auto signal_release = [&](int t) {  // one release reduction
        bool pa;
        int c, u;
        decode_task<TA, TB>(t, C, D, pa, c, u);
        red_add_release(pa ? doneA + c : doneB + c, 1);
    };
    // bounded wait for *p >= need (relaxed reads; the caller fences)
    auto spin = [&](const int* p) -> bool {
        const long long t0 = clock64();
        while (ld_relaxed(p) < need) {
            if (*(volatile int*)abort_flag) return false;
            if (clock64() - t0 > WAIT_LIMIT) {
                atomicCAS(a.err, 0, 9);
                atomicExch(abort_flag, 1);
                return false;
            }
            __nanosleep(64);
        }
        return true;
    };
    if (threadIdx.x == 0) {
        int t0 = valid(claim());
        nxt = t0 >= 0 ? valid(claim()) : -1;
        if (t0 >= 0) {
            const int* p = dep_of(t0);
            if (p && !spin(p)) t0 = nxt = -1;
            fence_gpu();
        }
        s_cur[0] = t0;
        dptr = nxt >= 0 ? dep_of(nxt) : nullptr;
    }
    __syncthreads();
    for (int it = 0;; ++it) {
        const int t = s_cur[it & 1];
        if (t < 0) break;
        if (threadIdx.x == 0) {
            pend = nxt >= 0 ? claim() : -1;  // the tile after next
            dv = dptr ? ld_acquire(dptr) : need;  // acquire: the next tile's reads are ordered after it
            // The next tile's input, if it comes from HBM (phase A), is prefetched into L2 by every
            // thread after the middle barrier, a half tile ahead: its loads then wait on L2 instead of
            // HBM.  Phase-B inputs (the ring) are in L2 already.
            const char* pf = nullptr;
            if (a.prefetch && nxt >= 0) {
                bool pa;
                int cn, un;
                decode_task<TA, TB>(nxt, C, D, pa, cn, un);
                const long long fb = (long long)(cn / NB) * N3, kbn = cn % NB;
                if (pa && FWD)  // TL contiguous grid rows of slice kbn TL + un / NB (as tile_body reads them)
                    pf = reinterpret_cast<const char*>(a.in) +
                         (fb + (kbn * TL + un / NB) * N2 + (long long)(un % NB) * TL * N) * (REAL_IO ? 4 : 8);
                else if (pa)    // N runs of TL pencil entries (128 bytes each, N^2 apart), one per p
                    pf = reinterpret_cast<const char*>(a.in + fb + (long long)un * N + kbn * TL);
            }
            s_pf = pf;
        }
        auto mid = [&] {
            if (threadIdx.x == 0) {
                // publish the previous tile: its stores (every thread's, ordered before this point by the
                // barriers) are released by the reduction
                if (prev >= 0) signal_release(prev);
                prev = -1;
                ready = nxt < 0 || dv >= need;
                s_cur[(it + 1) & 1] = nxt;
                s_slow = !ready;
            }
            // next-tile prefetch (thread 0 after publishing: measured faster than before it, a release
            // would also wait for its prefetches)
            if (const char* pf = s_pf) {
                constexpr int NL = FWD ? TL * N * (REAL_IO ? 4 : 8) / 128 : N;
                constexpr long long STEP = FWD ? 128 : 8 * N2;
#pragma unroll
                for (int i = threadIdx.x; i < NL; i += tile_threads(R)) prefetch_l2(pf + STEP * i);
            }
        };
        bool phaseA;
        int c, u;
        decode_task<TA, TB>(t, C, D, phaseA, c, u);
        const long long f = c / NB, kb = c % NB;
        float2* slot = a.ring + (long long)(c % S) * TL * N2;
        const long long fbase = f * N3;
        const int kl = u / NB, bb = u % NB, q = u;  // slice-type tile (kl, bb), q-type tile q
        if (FWD) {
            if (phaseA)
                tile_body<R, true, REAL_IO, HALF, IO_STREAM, IO_SCRATCH>(
                    a.in, slot, fbase + (kb * TL + kl) * N2 + (long long)bb * TL * N, kl * N2 + bb * TL, N, N, T,
                    Ws, pol_stream, pol_keep, mid);
            else
                tile_body<R, true, false, false, IO_SCRATCH, IO_STREAM>(slot, a.out, (long long)q * N,
                                                                  fbase + (long long)q * N + kb * TL, N2, N2, T, Ws,
                                                                  0, pol_stream, mid);
        } else {
            if (phaseA)
                tile_body<R, false, false, false, IO_STREAM, IO_SCRATCH>(a.in, slot, (long long)q * N,
                                                                   fbase + (long long)q * N + kb * TL, N2, N2, T,
                                                                   Ws, pol_stream, pol_keep, mid, a.nyq,
                                                                   a.nyq && q == N / 2);
            else
                tile_body<R, false, REAL_IO, HALF, IO_SCRATCH, IO_STREAM>(
                    slot, a.out, fbase + (kb * TL + kl) * N2 + (long long)bb * TL * N, kl * N2 + bb * TL, N, N, T,
                    Ws, 0, pol_stream, mid);
        }
        __syncthreads();  // every thread's stores (and discards) of tile t issued; shared memory free
        if (s_slow) {
            // the next tile's dependency was incomplete at the middle barrier.  Usually it has completed
            // since: re-read it and, if so, one fence (acquire) suffices and t stays unpublished until the
            // next tile's middle barrier.  Otherwise publish t first (it may be one of them) and wait.
            if (threadIdx.x == 0) {
                bool published = false, ok = true;
                if (ld_relaxed(dptr) < need) {
                    fence_gpu();
                    signal(t);
                    published = true;
                    ok = spin(dptr);
                }
                fence_gpu();
                s_cur[(it + 1) & 1] = ok ? nxt : -1;
                if (!ok) pend = -1;
                prev = published ? -1 : t;
            }
            __syncthreads();
        } else if (threadIdx.x == 0) {
            prev = t;
        }
        if (threadIdx.x == 0) {
            nxt = pend >= 0 ? valid(pend) : -1;
            dptr = nxt >= 0 ? dep_of(nxt) : nullptr;
        }
    }
    if (threadIdx.x == 0 && prev >= 0) {
        fence_gpu();
        signal(prev);
    }
}

template <int R, bool C2T, bool REAL_IO, bool HALF>
static cudaError_t tile_r(const void* in, void* out, long long nf, const TileGeo& g, bool nyq, const void* tw, cudaStream_t st)
{
    constexpr int N = 32 * R;
    constexpr int ROWS = REAL_IO ? TL / 2 : TL;  // real lines go in pairs
    const size_t smem = sizeof(float2) * (N + (size_t)ROWS * tile_ls<R, C2T>());
    auto k = fft_tile<R, C2T, REAL_IO, HALF>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    const long long nblk = nf * (long long)g.NO * (N / TL);
    k<<<(unsigned)nblk, tile_threads(R), smem, st>>>((const float2*)in, (float2*)out, g, nyq, (const double2*)tw);
    return cudaGetLastError();
}

template <bool C2T, bool REAL_IO, bool HALF>
static cudaError_t tile_dispatch(const void* in, void* out, long long nf, int N, const TileGeo& g, bool nyq, const void* tw,
                                 cudaStream_t st)
{
    switch (N) {
        case 64: return tile_r<2, C2T, REAL_IO, HALF>(in, out, nf, g, nyq, tw, st);
        case 128: return tile_r<4, C2T, REAL_IO, HALF>(in, out, nf, g, nyq, tw, st);
        case 256: return tile_r<8, C2T, REAL_IO, HALF>(in, out, nf, g, nyq, tw, st);
        case 512: return tile_r<16, C2T, REAL_IO, HALF>(in, out, nf, g, nyq, tw, st);
        case 1024: return tile_r<32, C2T, REAL_IO, HALF>(in, out, nf, g, nyq, tw, st);
        default: return cudaErrorNotSupported;
    }
}

template <bool C2T>
static cudaError_t tile_any(const void* in, void* out, long long nf, int N, const TileGeo& g, const void* tw,
                            cudaStream_t st, bool real_io, bool half, bool nyq)
{
    if (real_io && half) return tile_dispatch<C2T, true, true>(in, out, nf, N, g, nyq, tw, st);
    return real_io ? tile_dispatch<C2T, true, false>(in, out, nf, N, g, nyq, tw, st)
                   : tile_dispatch<C2T, false, false>(in, out, nf, N, g, nyq, tw, st);
}

// Lookahead D and ring slots S for N on a device of nsm SMs: about 4 nsm tile_ctas
// tiles are claimed and not yet published at any time (the resident CTAs, each
// holding up to three claims and one unpublished tile); D and S put every
// dependency at least W = twice that many tiles back (a chunk is `pair` tiles),
// where the live slots (D + 1) stay below 42 MB, a third of the L2.  Both bounds
// measured (both directions, ms): N = 128, 64 functions 1.10 with W once, 1.08
// twice, 1.08 three times; N = 64, 256 functions 0.83, 0.68, 0.68; N = 256, 16
// functions D = 3 2.26, 4 2.11 (42 MB), 6 2.26, 10 2.53; N = 512 D = 1 2.58, 2
// 2.91; the rare incomplete dependency takes the slow path.
static void fused_geometry(int N, int nsm, bool half, int& D, int& S)
{
    const int W = 8 * tile_ctas(N / 32) * nsm, pair = half ? N + N / 2 : 2 * N;  // tiles of a chunk
    const long long slot = (long long)TL * N * N * sizeof(float2) / (half ? 2 : 1);  // its live bytes
    D = std::max(1, (W - N + pair - 1) / pair);
    D = std::max(1, std::min(D, (int)((42LL << 20) / slot) - 1));
    if (const char* ev = getenv("FFTSO3_FFT_LOOKAHEAD")) {  // tuning override of D (1..16)
        const int d = atoi(ev);
        if (d >= 1 && d <= 16) D = d;
    }
    S = D + std::max(2, (W + N + pair - 1) / pair);
}

static int device_sms()
{
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess)
        return 0;
    return nsm;
}

template <int R, bool FWD, bool REAL_IO, bool HALF>
static cudaError_t grid2d_r(const Grid2DArgs& a, long long tiles, const void* tw, cudaStream_t st)
{
    const size_t smem = sizeof(float2) * (32 * R + (size_t)TL * tile_ls<R, FWD>());
    auto k = fft_grid2d<R, FWD, REAL_IO, HALF>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    int dev = 0, nsm = 0, occ = 0;
    if ((e = cudaGetDevice(&dev)) != cudaSuccess) return e;
    if ((e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev)) != cudaSuccess) return e;
    if ((e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&occ, k, tile_threads(R), smem)) != cudaSuccess) return e;
    const long long ctas = std::min<long long>(tiles, (long long)nsm * std::max(occ, 1));
    k<<<(unsigned)ctas, tile_threads(R), smem, st>>>(a, (const double2*)tw);
    return cudaGetLastError();
}

template <bool FWD, bool REAL_IO, bool HALF>
static cudaError_t grid2d_dispatch(const Grid2DArgs& a, long long tiles, int N, const void* tw, cudaStream_t st)
{
    switch (N) {
        case 64: return grid2d_r<2, FWD, REAL_IO, HALF>(a, tiles, tw, st);
        case 128: return grid2d_r<4, FWD, REAL_IO, HALF>(a, tiles, tw, st);
        case 256: return grid2d_r<8, FWD, REAL_IO, HALF>(a, tiles, tw, st);
        case 512: return grid2d_r<16, FWD, REAL_IO, HALF>(a, tiles, tw, st);
        default: return cudaErrorNotSupported;
    }
}

}  // namespace ffast

bool fft_fast_supported(int N) { return N == 64 || N == 128 || N == 256 || N == 512 || N == 1024; }

// Forward passes of one batch of N^3 grids (see fft.cuh):
//   pass 1: grid [f][k][j1][j2] -> FFT over j2 -> T1 [f][k][q][j1]
//   pass 2: T1 [f][k][q][j1]    -> FFT over j1 -> pencils [f][p][q][k]
// Inverse passes:
//   pass 2': pencils [f][p][q][k] -> FFT over p  -> T1 [f][k][q][j1]
//   pass 1': T1 [f][k][q][j1]     -> FFT over q  -> grid [f][k][j1][j2]
cudaError_t launch_fft_grid_pass(const void* in, void* out, long long nf, int N, int pass, const void* tw,
                                 cudaStream_t st, bool real_io, bool half, bool nyq)
{
    const long long N1 = N, N2 = (long long)N * N, N3 = N2 * N;
    if (real_io && pass != 1 && pass != -1) return cudaErrorInvalidValue;
    const ffast::TileGeo g1{N3, N, N2, N1, N2, N1};  // lines along j2 / q, transposed (q, j1)
    const ffast::TileGeo g2{N3, half ? N / 2 : N, N1, N2, N1, N2};  // lines along j1 / p of each q, transposed (p.., k)
    switch (pass) {
        case 1: return ffast::tile_any<true>(in, out, nf, N, g1, tw, st, real_io, half, false);
        case 2: return ffast::tile_any<true>(in, out, nf, N, g2, tw, st, false, false, false);
        case -2: return ffast::tile_any<false>(in, out, nf, N, g2, tw, st, false, false, nyq);
        case -1: return ffast::tile_any<false>(in, out, nf, N, g1, tw, st, real_io, half, false);
        default: return cudaErrorInvalidValue;
    }
}

bool fft_grid_fused_supported(int N) { return N == 64 || N == 128 || N == 256 || N == 512; }
size_t fft_grid_fused_ring_elems(int N, bool half)
{
    int D, S;
    ffast::fused_geometry(N, ffast::device_sms(), half, D, S);
    return (size_t)S * ffast::TL * N * N;
}
size_t fft_grid_fused_ctl_ints(long long nf, int N) { return 2 + 2 * (size_t)nf * (N / ffast::TL); }

// Both passes of one direction (dir 1: grid -> pencils, dir -1: pencils ->
// grid) in one persistent launch through the L2-resident ring (fft_grid2d).
cudaError_t launch_fft_grid_fused(const void* in, void* out, void* ring, size_t ring_elems, int* ctl, int* err,
                                  long long nf, int N, int dir, const void* tw, cudaStream_t st, bool real_io, bool half, bool nyq)
{
    if (half && !real_io) return cudaErrorInvalidValue;
    if (!fft_grid_fused_supported(N) || (dir != 1 && dir != -1) || nf < 1) return cudaErrorInvalidValue;
    const long long C = nf * (N / ffast::TL);
    if (C > (1LL << 29) / N) return cudaErrorInvalidValue;  // tile indices stay in int
    cudaError_t e = cudaMemsetAsync(ctl, 0, sizeof(int) * fft_grid_fused_ctl_ints(nf, N), st);
    if (e != cudaSuccess) return e;
    int D, S;
    ffast::fused_geometry(N, ffast::device_sms(), half, D, S);
    if ((size_t)S * ffast::TL * N * N > ring_elems) return cudaErrorInvalidValue;  // ring sized for another device
    const char* pf = getenv("FFTSO3_FFT_PREFETCH");  // 0 turns the next-tile L2 prefetch off (tuning)
    ffast::Grid2DArgs a{(const float2*)in, (float2*)out, (float2*)ring, ctl, err, (int)C, D, S, nyq,
                        pf && atoi(pf) == 0 ? 0 : 1};
    const long long tiles = C * (half ? N + N / 2 : 2 * N);
    if (half)
        return dir == 1 ? ffast::grid2d_dispatch<true, true, true>(a, tiles, N, tw, st)
                        : ffast::grid2d_dispatch<false, true, true>(a, tiles, N, tw, st);
    if (dir == 1)
        return real_io ? ffast::grid2d_dispatch<true, true, false>(a, tiles, N, tw, st)
                       : ffast::grid2d_dispatch<true, false, false>(a, tiles, N, tw, st);
    return real_io ? ffast::grid2d_dispatch<false, true, false>(a, tiles, N, tw, st)
                   : ffast::grid2d_dispatch<false, false, false>(a, tiles, N, tw, st);
}

cudaError_t launch_fft_s2_pass(const void* in, void* out, long long nf, int N, int dir, const void* tw,
                               cudaStream_t st, bool real_io, bool half, bool nyq)
{
    const long long N1 = N, N2 = (long long)N * N;
    const ffast::TileGeo g{N2, 1, 0, N1, 0, N1};  // lines along j (contiguous), transposed [p][k]
    if (dir == 1) return ffast::tile_any<true>(in, out, nf, N, g, tw, st, real_io, half, nyq);
    if (dir == -1) return ffast::tile_any<false>(in, out, nf, N, g, tw, st, real_io, half, nyq);
    return cudaErrorInvalidValue;
}

}  // namespace fftso3
