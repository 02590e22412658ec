// The direct DFT of even length N = 2P in double-float on the tcgen05 tensor cores, for the refinement and the exact inverse of
// plans whose N the double-float FFT (fft.cu, powers of two from 64 to 512) does not serve.
//
// The folding, the four problems, the row and line layouts and the roles are those of dft_tc.cu.  The arithmetic is exact:
//  * every line is written in fixed point, X = x 2^(35 - E), 2^E above 1.01 times its largest folded value (found in FP32
//    first), as two limbs of 18 bits: the upper ones are folded as integers, the remainders in FP32;
//  * a folded value is four balanced base-512 digits, a matrix entry sum_j s_j 2^(-8 - 9 j), |s_j| <= 256, both exact in
//    FP16; the digit products d_i s_j with i + j = v accumulate in FP32 accumulator v (v = 0..3) as integers below 2^24
//    (4 pairs x 56 terms x 2^16), so without rounding;
//  * the epilogue adds or subtracts the cosine and sine sums level by level, combines the levels to a double-float and
//    scales by 2^(E - 16).
// A value is exact to about 2^-33 of its line's largest folded input (the fixed point and the dropped products i + j >= 4).
// Not-a-number and infinite inputs make their line's outputs not-a-number.
//
// Bound: the producers' instructions (about 30 a value read: two sweeps' fixed-point splits, folds, carries and digit fields)
// and the epilogue's 20 a level sum, with 19 warps to hide their latency (0.38 to 0.50 issued a scheduler and cycle), not the
// MMAs or memory (DRAM 12 to 27 %).  In double-float arithmetic on the CUDA cores the mixed-radix line kernels
// took 5.9 ms for the forward passes of 16 real functions of N = 160 and 6.1 ms for the inverse ones; these take 1.13 and
// 0.98 (65.5 M samples).  Powers of two from 64 keep the line FFT along k runs, which is faster still: N = 126 30 G complex
// samples/s here, N = 128 76 there (two passes).  Folding in 32-bit words instead (four base-256 digits, one sweep) took 0.80 ms,
// but its rounding at 2^-30 showed in the outputs (2.5485e-8 of the rms against 2.5355e-8, where the output rounding alone is
// 2.5261e-8); with the two limbs the errors are those of the line kernels.
//
// Roles of the one CTA an SM holds: warps 0-13 producers, 14-17 epilogue, 18 MMA issuer, which also streams the matrices' digits
// (32 KB a problem) next to the operand they meet.  A tile's inputs are read three times, the second and third time from L2:
// for the largest folded values, and for the digits of the even and of the odd q's problems, whose two words a value take
// the producers' registers.  The four levels of C and of S fill TMEM, so the products of the odd q wait for the epilogue
// of the even ones.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "df32.cuh"
#include "dft_oz.cuh"
#include "tc_ptx.cuh"

namespace fftso3 {

namespace doz {

using namespace ptx;

constexpr int NPROD = 14, NEPI = 4, MMAW = 18;  // 19 warps: five a scheduler, 96 registers a thread
constexpr int THREADS = 32 * (MMAW + 1);
constexpr int ND = 4;                 // digits
constexpr int PLANE = 128 * 128;      // 128 rows x 64 FP16
constexpr int SLOT_A = ND * PLANE, SLOT_B = ND * 64 * 128, SLOT = SLOT_A + SLOT_B;
constexpr int MAXH = 56;
constexpr int SMEM = 2 * SLOT + 256 + 6 * 128 * 4 + 1024;
constexpr int EMIN = -109, EMAX = 129;

enum { COMPLEX = 0, REAL_IN = 1, REAL_OUT = 2 };
enum { DF = 0, HILO = 1, F32 = 2 };

struct Args {
    const void* in;
    void* out;
    float2* lo;
    const unsigned char* table;
    int* err;
    int N, H, KC;
    unsigned ntiles;
    int no, skip;
    unsigned tx, ty, nlines;
    long long i_f, i_a, i_e, o_f, o_a, o_e;
    int nyq, mirror;
};

struct Line {
    long long in, out;
    int o;
    bool ok;
};
// as in dft_tc.cu
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

__device__ __forceinline__ float pow2f(int e) { return __int_as_float((127 + e) << 23); }
__device__ __forceinline__ unsigned absbits(float x) { return __float_as_uint(x) & 0x7fffffffu; }

// |a| + |b| is the larger of |a + b| and |a - b|.
__device__ __forceinline__ float larger(float a, float b) { return fabsf(a) + fabsf(b); }
// Largest folded value of x_t, x_{N-t}, x_{P-t}, x_{P+t}, as bits (NaN compares largest).
__device__ __forceinline__ unsigned folded_max(float x, float xn, float xp, float xq)
{
    return max(absbits(larger(x + xn, xp + xq)), absbits(larger(x - xn, xp - xq)));
}

__device__ __forceinline__ int exponent_of(unsigned m)
{
    const int e = (int)(__float_as_uint(__uint_as_float(m) * 1.01f) >> 23) - 126;
    return e < EMIN ? EMIN : e > EMAX ? EMAX : e;
}
// A value in fixed point: its upper limb as the bits of an FP32 number 1.5 2^23 + limb (conversions run at a quarter of the
// rate), the remainder in units of the upper limb.
constexpr float MAGIC = 12582912.f;
constexpr uint32_t MAGIC_BITS = 0x4B400000u;
struct Fixed {
    uint32_t i;
    float r;
};
__device__ __forceinline__ Fixed fixed(float h, float s)
{
    const float q = h * s, f = __fadd_rn(q, MAGIC);
    return {__float_as_uint(f), __fsub_rn(q, __fsub_rn(f, MAGIC))};
}
__device__ __forceinline__ Fixed fixed(float h, float l, float s)
{
    const Fixed x = fixed(h, s);
    return {x.i, __fmaf_rn(l, s, x.r)};
}
// The limbs of a folded value, each offset by 256 * 512 + 256, so that its two digits are bit fields offset by 256 (the upper
// one of the first limb from 3 to 509, as |X| < 2^35 / 1.01; the others from 0 to 512).  magics: the MAGIC_BITS in x.i.
struct Limbs {
    uint32_t w1, w0;
};
__device__ __forceinline__ Limbs limbs(uint32_t i, float r, int magics)
{
    const float c = __fadd_rn(r, MAGIC);
    return {i + __float_as_uint(c) + (131328u - MAGIC_BITS * (uint32_t)(magics + 1)),
            __float_as_uint(__fmaf_rn(__fsub_rn(r, __fsub_rn(c, MAGIC)), 262144.f, MAGIC + 131328.f))};
}

// Eight values' digits into one 16-byte chunk of each digit plane.
__device__ __forceinline__ void store_digits(uint32_t dst, const Limbs* x)
{
    // a field u in FP16's low bits under 0x6400 is 1024 + u
    const __half2 off = __floats2half2_rn(-1280.f, -1280.f), half = __floats2half2_rn(0.5f, 0.5f),
                  off2 = __floats2half2_rn(-768.f, -768.f);
    uint32_t w[ND][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const Limbs a = x[2 * j], b = x[2 * j + 1];
        auto h2 = [](uint32_t u) { return *reinterpret_cast<const __half2*>(&u); };
        // bits 8-23: twice the upper field and a bit of the lower
        const __half2 d[ND] = {
            __hfma2(h2((__byte_perm(a.w1, b.w1, 0x6521) & 0x07fe07feu) | 0x64006400u), half, off2),
            __hadd2(h2((__byte_perm(a.w1, b.w1, 0x5410) & 0x01ff01ffu) | 0x64006400u), off),
            __hadd2(h2(((__byte_perm(a.w0, b.w0, 0x6521) >> 1) & 0x03ff03ffu) | 0x64006400u), off),
            __hadd2(h2((__byte_perm(a.w0, b.w0, 0x5410) & 0x01ff01ffu) | 0x64006400u), off)};
#pragma unroll
        for (int p = 0; p < ND; ++p) w[p][j] = *reinterpret_cast<const uint32_t*>(&d[p]);
    }
#pragma unroll
    for (int p = 0; p < ND; ++p)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + p * PLANE), "r"(w[p][0]), "r"(w[p][1]),
                     "r"(w[p][2]), "r"(w[p][3])
                     : "memory");
}

// level sums (integers, units 2^-9v) -> double-float, scaled
__device__ __forceinline__ float2 combine(float a0, float a1, float a2, float a3, float sc)
{
    const df32 s = df_two_sum(a0, a1 * 0.001953125f);
    const df32 r = df_quick_two_sum(s.h, s.l + __fmaf_rn(a3, 7.450580596923828e-09f, a2 * 3.814697265625e-06f));
    return make_float2(r.h * sc, r.l * sc);
}

__device__ __forceinline__ void producers_sync() { asm volatile("bar.sync 1, %0;" ::"n"(32 * NPROD) : "memory"); }

// Folds x_t, x_{N-t}, x_{P-t}, x_{P+t} for the even (ODD = false) or odd q: the cosine problem's value and the sine problem's,
// NEG: negated.  (Terms whose sine or cosine is zero for all those q need no zeroing: the matrix has zeros there.)
template <bool ODD>
__device__ __forceinline__ Limbs fold_cos(Fixed x, Fixed xn, Fixed xp, Fixed xq)
{
    return ODD ? limbs(x.i + xn.i - xp.i - xq.i, (x.r + xn.r) - (xp.r + xq.r), 0)
               : limbs(x.i + xn.i + xp.i + xq.i, (x.r + xn.r) + (xp.r + xq.r), 4);
}
template <bool ODD, bool NEG>
__device__ __forceinline__ Limbs fold_sin(Fixed x, Fixed xn, Fixed xp, Fixed xq)
{
    if (NEG) return fold_sin<ODD, false>(xn, x, xq, xp);
    return ODD ? limbs(x.i - xn.i + xp.i - xq.i, (x.r - xn.r) + (xp.r - xq.r), 0)
               : limbs(x.i - xn.i - xp.i + xq.i, (x.r - xn.r) - (xp.r - xq.r), 0);
}

// The digits' limbs of eight terms t0.. of a line at `in`, for the cosine (v[0]) and the sine problem (v[1]).  As in dft_tc.cu,
// the sine problem of a complex line takes (im, -re) in the (re, im) rows, that of real samples is negated.
template <int KIND, bool INDF, bool ODD, int VPL>
__device__ __forceinline__ void load_fold(const Args& a, long long in, bool ok, int t0, float s, Limbs (&v)[2][VPL])
{
    const int N = a.N, P = N / 2;
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int t = t0 + k;
        const bool use = ok && t < a.H, pos = t > 0, two = 2 * t != P;
        if (KIND == REAL_IN) {
            const float* g = reinterpret_cast<const float*>(a.in) + in;
            auto at = [&](int j, bool u) { return fixed(u ? __ldg(g + j * a.i_e) : 0.f, s); };
            const Fixed x0 = at(t, use), x1 = at(N - t, use && pos), x2 = at(P - t, use && two), x3 = at(P + t, use && two && pos);
            v[0][k] = fold_cos<ODD>(x0, x1, x2, x3);
            v[1][k] = fold_sin<ODD, true>(x0, x1, x2, x3);
        } else {
            Fixed x[4], y[4];  // re, im
            auto at = [&](int n, int j, bool u, float s) {
                if (INDF) {
                    float4 z = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (u) z = __ldcg(reinterpret_cast<const float4*>(a.in) + in + j * a.i_e);
                    x[n] = fixed(z.x, z.y, s);
                    y[n] = fixed(z.z, z.w, s);
                } else {
                    float2 z = make_float2(0.f, 0.f);
                    if (u) z = __ldg(reinterpret_cast<const float2*>(a.in) + in + j * a.i_e);
                    x[n] = fixed(z.x, s);
                    y[n] = fixed(z.y, s);
                }
            };
            if constexpr (KIND == COMPLEX) {
                at(0, t, use, s);
                at(1, N - t, use && pos, s);
                at(2, P - t, use && two && (pos || !a.nyq), s);
                at(3, P + t, use && two && pos, s);
                v[0][k] = fold_cos<ODD>(x[0], x[1], x[2], x[3]);
                v[0][k + 8] = fold_cos<ODD>(y[0], y[1], y[2], y[3]);
                v[1][k] = fold_sin<ODD, false>(y[0], y[1], y[2], y[3]);
                v[1][k + 8] = fold_sin<ODD, true>(x[0], x[1], x[2], x[3]);
            } else {
                // a_t = 2 Re X_t, b_t = 2 Im X_t (a_0 = Re X_0); X_P = 0
                at(0, t, use, pos ? 2.f * s : s);
                at(2, P - t, use && two && pos, 2.f * s);
                v[0][k] = ODD ? limbs(x[0].i - x[2].i, x[0].r - x[2].r, 0) : limbs(x[0].i + x[2].i, x[0].r + x[2].r, 2);
                v[1][k] = ODD ? limbs(y[0].i + y[2].i, y[0].r + y[2].r, 2) : limbs(y[0].i - y[2].i, y[0].r - y[2].r, 0);
            }
        }
    }
}

// The largest folded value of those terms, as bits.
template <int KIND, bool INDF>
__device__ __forceinline__ unsigned line_max(const Args& a, long long in, int t0)
{
    const int N = a.N, P = N / 2;
    unsigned m = 0;
#pragma unroll 4
    for (int k = 0; k < 8; ++k) {
        const int t = t0 + k;
        if (t >= a.H) break;
        const bool pos = t > 0, two = 2 * t != P;
        if (KIND == REAL_IN) {
            const float* g = reinterpret_cast<const float*>(a.in) + in;
            auto at = [&](int j, bool u) { return u ? __ldg(g + j * a.i_e) : 0.f; };
            m = max(m, folded_max(at(t, true), at(N - t, pos), at(P - t, two), at(P + t, two && pos)));
        } else {
            auto at = [&](int j, bool u) {
                if (!u) return make_float2(0.f, 0.f);
                if (!INDF) return __ldg(reinterpret_cast<const float2*>(a.in) + in + j * a.i_e);
                const float4 z = __ldcg(reinterpret_cast<const float4*>(a.in) + in + j * a.i_e);
                return make_float2(z.x, z.z);
            };
            const float2 x0 = at(t, true), x2 = at(P - t, two && (pos || !a.nyq));
            if (KIND == COMPLEX) {
                const float2 x1 = at(N - t, pos), x3 = at(P + t, two && pos);
                m = max(m, folded_max(x0.x, x1.x, x2.x, x3.x));
                m = max(m, folded_max(x0.y, x1.y, x2.y, x3.y));
            } else {
                m = max(m, absbits(2.f * larger(x0.x, x2.x)));
                m = max(m, absbits(2.f * larger(x0.y, x2.y)));
            }
        }
    }
    return m;
}

// KIND, TR: as in dft_tc.cu.  INDF: double-float input.  OUT: DF, HILO or F32.
template <int KIND, bool TR, bool INDF, int OUT>
__global__ void __launch_bounds__(THREADS, 1) dft_oz_kernel(const __grid_constant__ Args a)
{
    extern __shared__ unsigned char smem_raw[];
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(smem + 2 * SLOT);  // operand written (producers) ..
    uint64_t* bful = full + 2;                      // .. and the matrix's digits arrived
    uint64_t* empty = bful + 2;
    uint64_t* accf = empty + 2;
    uint64_t* acce = accf + 1;
    uint32_t* tmem_slot = (uint32_t*)(acce + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    unsigned* mx = (unsigned*)(smem + 2 * SLOT + 256);  // [tile mod 3][line]: bits of the largest component
    int* ex = (int*)(mx + 384);                         // [tile mod 3][line]: exponent, or 1 << 20 (not finite)
    const int warp = __shfl_sync(0xffffffffu, (int)threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int KC = a.KC, NQ = 16 * KC, H = a.H, N = a.N, P = N / 2, BPLANE = NQ * 128;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2; ++s) {
            mbar_init(&full[s], NPROD);
            mbar_init(&bful[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(accf, 1);
        mbar_init(acce, NEPI);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == MMAW) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    // operand columns past the folded terms stay zero
    for (int i = threadIdx.x; i < 2 * SLOT_A / 16; i += THREADS)
        reinterpret_cast<uint4*>(smem + (i / (SLOT_A / 16)) * SLOT)[i % (SLOT_A / 16)] = make_uint4(0, 0, 0, 0);
    for (int i = threadIdx.x; i < 384; i += THREADS) mx[i] = 0;
    fence_proxy_async();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp < NPROD) {
        // ---------------- producers: an item is 32 lines x 8 folded terms
        constexpr int VPL = KIND == COMPLEX ? 16 : 8;
        constexpr int IPW = KIND == COMPLEX ? 1 : 2;
        constexpr int LB = KIND == COMPLEX ? 2 : 4;
        int lx[IPW], ly[IPW], ch[IPW], row[IPW], ln[IPW];
#pragma unroll
        for (int w = 0; w < IPW; ++w) {
            const int it = warp + w * NPROD, lb = it % LB;
            ch[w] = it / LB;
            if (KIND == COMPLEX) {
                lx[w] = TR ? (lane & 7) : (lane >> 3) + 4 * lb;
                ly[w] = TR ? (lane >> 3) + 4 * lb : (lane & 7);
                row[w] = lx[w] * 16 + (ly[w] ^ (lx[w] & 7));
                ln[w] = lx[w] * 8 + ly[w];
            } else if (KIND == REAL_IN) {
                lx[w] = lane & 15;
                ly[w] = (lane >> 4) + 2 * lb;
                row[w] = lx[w] * 8 + (ly[w] ^ (lx[w] & 7));
                ln[w] = lx[w] * 8 + ly[w];
            } else {
                lx[w] = lane & 7;
                ly[w] = (lane >> 3) + 4 * lb;
                row[w] = lx[w] * 16 + (ly[w] ^ lx[w]);
                ln[w] = lx[w] * 16 + ly[w];
            }
        }
        // a failed wait (every producer meets it in its turn) ends the stores; the tiles' barriers go on, so that no warp
        // waits for one that left
        unsigned s = 0;
        int tp = 0;
        for (unsigned tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, tp = tp == 2 ? 0 : tp + 1) {
            long long in[IPW];
            bool ok[IPW];
            float scale[IPW];
#pragma unroll
            for (int w = 0; w < IPW; ++w) {
                const Line L = line_of<KIND, TR>(a, tile, lx[w], ly[w]);
                ok[w] = L.ok && 8 * ch[w] < H;
                in[w] = L.in;
                if (ok[w]) atomicMax(&mx[tp * 128 + ln[w]], line_max<KIND, INDF>(a, in[w], 8 * ch[w]));
            }
            // the next tile's maxima: last read before the last tile's barrier
            if (threadIdx.x < 128) mx[(tp == 2 ? 0 : tp + 1) * 128 + threadIdx.x] = 0;
            producers_sync();
#pragma unroll
            for (int w = 0; w < IPW; ++w) {
                const unsigned m = mx[tp * 128 + ln[w]];
                const int E = exponent_of(m);
                if (ch[w] == 0) ex[tp * 128 + ln[w]] = m >= 0x7f7fffffu - (1u << 18) ? 1 << 20 : E;
                scale[w] = pow2f(17 - E);
            }
#pragma unroll
            for (int par = 0; par < 2; ++par) {
                Limbs v[IPW][2][VPL];
#pragma unroll
                for (int w = 0; w < IPW; ++w) {
                    if (8 * ch[w] >= H) continue;
                    if (par == 0)
                        load_fold<KIND, INDF, false>(a, in[w], ok[w], 8 * ch[w], scale[w], v[w]);
                    else
                        load_fold<KIND, INDF, true>(a, in[w], ok[w], 8 * ch[w], scale[w], v[w]);
                }
#pragma unroll
                for (int pr = 0; pr < 2; ++pr, ++s) {
                    const int sl = s & 1;
                    const bool stop = *abort_flag || (s >= 2 && !mbar_wait(&empty[sl], ((s >> 1) - 1) & 1, a.err, 41));
                    if (__any_sync(0xffffffffu, stop)) {
                        *abort_flag = 1;
                        continue;
                    }
#pragma unroll
                    for (int w = 0; w < IPW; ++w) {
                        if (8 * ch[w] >= H) continue;
                        const uint32_t d = smem_u32(smem + sl * SLOT) + row[w] * 128 + ((ch[w] ^ (row[w] & 7)) << 4);
                        store_digits(d, v[w][pr]);
                        if (KIND == COMPLEX) store_digits(d + 8 * 128, v[w][pr] + (VPL - 8));
                    }
                    fence_proxy_async();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&full[sl]);
                }
            }
        }
    } else if (warp == MMAW) {
        if (elect_one()) {
            // ---------------- MMA issuer; A_j x [B_0 .. B_{3-j}] -> levels j .. 3
            uint32_t id[ND];
#pragma unroll
            for (int j = 0; j < ND; ++j) id[j] = idesc_f16_mn((ND - j) * NQ, 128);
            const unsigned T = blockIdx.x < a.ntiles ? 4 * ((a.ntiles - 1 - blockIdx.x) / gridDim.x + 1) : 0;  // problems
            unsigned loaded = 0;
            auto load_b = [&](unsigned s) {
                const int sl = s & 1;
                ++loaded;
                mbar_expect_tx(&bful[sl], ND * BPLANE);
                bulk_load(smem + sl * SLOT + SLOT_A, a.table + (size_t)(s & 3) * ND * BPLANE, ND * BPLANE, &bful[sl]);
            };
            if (T > 0) load_b(0);
            unsigned s = 0;  // issued
            bool ok = true;
            for (; s < T && ok && !*abort_flag; ++s) {
                const int sl = s & 1, pr = s & 3;
                // C and S of one parity fill TMEM: the last parity's must have been read
                if ((pr & 1) == 0 && s >= 2 && !mbar_wait(acce, ((s >> 1) - 1) & 1, a.err, 42)) {
                    ok = false;
                    break;
                }
                if (!mbar_wait(&bful[sl], (s >> 1) & 1, a.err, 43) || !mbar_wait(&full[sl], (s >> 1) & 1, a.err, 44)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t d = tmem + (pr & 1) * 256;
                uint64_t ad = smem_desc(smem_u32(smem + sl * SLOT), 16, 1024);
                uint64_t bd = smem_desc(smem_u32(smem + sl * SLOT + SLOT_A), 16, 1024);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk, ad += 2, bd += 2) {
                    if (kk >= KC) break;
#pragma unroll
                    for (int j = 0; j < ND; ++j)
                        mma_bf16(d + j * NQ, ad + j * (PLANE >> 4), bd, id[j], kk > 0 || j > 0);
                }
                mma_commit(&empty[sl]);
                if (pr & 1) mma_commit(accf);
                if (s + 1 < T) {
                    // the next problem's matrix, where the last problem's was (its MMAs were committed before these)
                    if (s >= 1 && !mbar_wait(&empty[(s + 1) & 1], ((s - 1) >> 1) & 1, a.err, 45)) {
                        ok = false;
                        ++s;
                        break;
                    }
                    load_b(s + 1);
                }
            }
            if (!ok) *abort_flag = 1;
            // copies in flight land and the last MMAs end before the shared memory and TMEM are freed
            if (loaded) mbar_wait(&bful[(loaded - 1) & 1], ((loaded - 1) >> 1) & 1, a.err, 46);
            if (s) mbar_wait(&empty[(s - 1) & 1], ((s - 1) >> 1) & 1, a.err, 46);
        }
    } else {
        // ---------------- epilogue
        const int quarter = warp & 3, r = quarter * 32 + lane;
        int x, y, part = 0, ln;
        if (KIND == COMPLEX) {
            x = r >> 4;
            y = (r & 7) ^ (x & 7);
            part = (r >> 3) & 1;
            ln = x * 8 + y;
        } else if (KIND == REAL_IN) {
            x = r >> 3;
            y = (r & 7) ^ (x & 7);
            ln = x * 8 + y;
        } else {
            x = r >> 4;
            y = (r & 15) ^ x;
            ln = x * 16 + y;
        }
        unsigned s = 0;
        int tp = 0;
        bool ok = true;
        for (unsigned tile = blockIdx.x; tile < a.ntiles && ok && !*abort_flag; tile += gridDim.x, tp = tp == 2 ? 0 : tp + 1) {
            const Line L = line_of<KIND, TR>(a, tile, x, y);
            float sc = 0.f;
            for (int par = 0; par < 2; ++par, ++s) {
                // in place: the odd q's producers must have read the lines too (the third problem written: the second phase of
                // its slot, which the next cannot complete before these accumulators are read)
                if (!mbar_wait(accf, s & 1, a.err, 47) || (par == 0 && a.in == a.out && !mbar_wait(&full[0], 1, a.err, 48))) {
                    *abort_flag = 1;
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (par == 0) {
                    const int E = *(volatile int*)&ex[tp * 128 + ln];
                    sc = E == (1 << 20) ? __int_as_float(0x7fffffff) : pow2f(E - 16);
                }
                const uint32_t base = tmem + ((uint32_t)(quarter * 32) << 16);
                const int nq = (P - par) / 2 + 1;
                for (int b = 0; 8 * b < nq; ++b) {
                    const int q0 = 16 * b + par, nv = L.ok ? nq - 8 * b : 0;
                    uint32_t t[2][ND][8];
#pragma unroll
                    for (int c = 0; c < 2; ++c)
#pragma unroll
                        for (int j = 0; j < ND; ++j) tmem_ld8_nowait(base + c * 256 + j * NQ + b * 8, t[c][j]);
                    tmem_wait_ld();
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        const int q = q0 + 2 * i;
                        float C[ND], S[ND];
#pragma unroll
                        for (int j = 0; j < ND; ++j) {
                            C[j] = __uint_as_float(t[0][j][i]);
                            S[j] = __uint_as_float(t[1][j][i]);
                        }
                        if (KIND == REAL_IN) {
                            const float2 re = combine(C[0], C[1], C[2], C[3], sc), im = combine(S[0], S[1], S[2], S[3], sc);
                            if (i < nv)
                                reinterpret_cast<float4*>(a.out)[L.out + q * a.o_e] = make_float4(re.x, re.y, im.x, im.y);
                            continue;
                        }
                        const float2 u = combine(C[0] + S[0], C[1] + S[1], C[2] + S[2], C[3] + S[3], sc);
                        const float2 w = combine(C[0] - S[0], C[1] - S[1], C[2] - S[2], C[3] - S[3], sc);
                        const bool v0 = i < nv, v1 = v0 && q > 0 && q < P;
                        const long long i0 = L.out + q * a.o_e, i1 = L.out + (N - q) * a.o_e;
                        if (OUT == DF) {
                            float2* o = reinterpret_cast<float2*>(a.out);
                            if (v0) o[2 * i0 + part] = u;
                            if (v1) o[2 * i1 + part] = w;
                        } else if (OUT == HILO) {
                            float* hi = reinterpret_cast<float*>(a.out) + part;
                            float* lo = reinterpret_cast<float*>(a.lo) + part;
                            if (v0) {
                                hi[2 * i0] = u.x;
                                lo[2 * i0] = u.y;
                            }
                            if (v1) {
                                hi[2 * i1] = w.x;
                                lo[2 * i1] = w.y;
                            }
                            if (a.mirror && L.o > 0 && L.o < P && v0) {
                                // (o, q) -> (N - o, N - q) and (o, N - q) -> (N - o, q), conjugated
                                const long long mo = (long long)(N - 2 * L.o) * a.o_a;
                                const float sg = part ? -1.f : 1.f;
                                if (q > 0) {
                                    hi[2 * (i1 + mo)] = sg * u.x;
                                    lo[2 * (i1 + mo)] = sg * u.y;
                                }
                                if (q < P) {
                                    hi[2 * (i0 + mo)] = sg * w.x;
                                    lo[2 * (i0 + mo)] = sg * w.y;
                                }
                            }
                        } else {
                            constexpr int W = KIND == COMPLEX ? 2 : 1;
                            float* o = reinterpret_cast<float*>(a.out) + part;
                            if (v0) o[W * i0] = u.x + u.y;
                            if (v1) o[W * i1] = w.x + w.y;
                        }
                    }
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncwarp();
                if (lane == 0) mbar_arrive(acce);
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

// [problem: cos even, sin even, cos odd, sin odd][digit][q][t] FP16, rows of 128 bytes, their 16-byte chunks swizzled
__global__ void build_table_kernel(unsigned char* table, int N, int H, int NQ, const double2* __restrict__ tw)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 4 * NQ * 64) return;
    const int t = i & 63, qi = (i >> 6) % NQ, pr = (i >> 6) / NQ, q = 2 * qi + (pr >> 1);
    double v = 0.0;
    if (t < H && q <= N / 2) {
        const double2 x = __ldg(tw + (t * q) % N);
        v = (pr & 1) ? -x.y : x.x;
    }
    unsigned char* d = table + (size_t)pr * ND * NQ * 128 + qi * 128 + (((t >> 3) ^ (qi & 7)) << 4) + 2 * (t & 7);
    v *= 256.0;
    for (int p = 0; p < ND; ++p) {
        const double s = rint(v);
        *reinterpret_cast<__half*>(d + (size_t)p * NQ * 128) = __double2half(s);
        v = (v - s) * 512.0;
    }
}

template <int KIND, bool TR, bool INDF, int OUT>
static cudaError_t run(const Args& a, cudaStream_t st)
{
    auto kern = dft_oz_kernel<KIND, TR, INDF, OUT>;
    int dev = 0, nsm = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) e = cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
    if (e != cudaSuccess) return e;
    kern<<<std::min(a.ntiles, (unsigned)nsm), THREADS, SMEM, st>>>(a);
    return cudaGetLastError();
}

static int folded_terms(int N) { return N / 4 + 1; }

}  // namespace doz

using namespace doz;

bool dft_oz_supported(int N) { return N >= 2 && N % 2 == 0 && folded_terms(N) <= MAXH; }

size_t dft_oz_table_bytes(int N) { return (size_t)4 * ND * 16 * ((folded_terms(N) + 15) / 16) * 128; }

cudaError_t dft_oz_build_table(void* table, int N, const void* tw, cudaStream_t st)
{
    const int H = folded_terms(N), NQ = 16 * ((H + 15) / 16), n = 4 * NQ * 64;
    build_table_kernel<<<(n + 127) / 128, 128, 0, st>>>((unsigned char*)table, N, H, NQ, (const double2*)tw);
    return cudaGetLastError();
}

cudaError_t launch_dft_oz_grid_pass(const void* in, void* out, float2* lo, long long nf, int N, int pass, bool real,
                                    const void* table, int* err, cudaStream_t st)
{
    const long long n = N, NN = n * n;
    if (!dft_oz_supported(N) || nf < 1 || nf * NN > 0x7fffffffLL) return cudaErrorInvalidValue;
    const int P = N / 2;
    Args a = {};
    a.in = in;
    a.out = out;
    a.lo = lo;
    a.table = (const unsigned char*)table;
    a.err = err;
    a.N = N;
    a.H = folded_terms(N);
    a.KC = (a.H + 15) / 16;
    a.i_f = a.o_f = NN * n;
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
            a.ntiles = (unsigned)nf * a.tx * a.ty;
            return real ? run<REAL_IN, true, false, DF>(a, st) : run<COMPLEX, true, false, DF>(a, st);
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
            return pass > 0 ? run<COMPLEX, false, true, HILO>(a, st) : run<COMPLEX, false, true, DF>(a, st);
        case -1:  // x = k, y = j2
            a.tx = blocks(8);
            a.ty = blocks(real ? 16 : 8);
            a.nyq = 1;
            a.i_a = n;
            a.i_e = NN;
            a.o_a = NN;
            a.o_e = n;
            a.ntiles = (unsigned)nf * a.tx * a.ty;
            return real ? run<REAL_OUT, true, true, F32>(a, st) : run<COMPLEX, true, true, F32>(a, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace fftso3
