// Strided passes of the direct DFT (direct_dft.cuh) for the SO(3) and S^2 grid transforms of FP32-data plans whose N
// the register FFT does not serve (any even N up to about 400): each pass reads and writes every sample once and
// leaves the transposition to its addressing, so a direction is two launches and no separate transpose.
//
// A persistent CTA holds the four matrices and walks tiles of LT units: load and fold into shared memory, one
// register tile of products per thread, outputs straight from registers (unit-contiguous side: 128-byte runs) or
// through the folded buffer (line-contiguous side).  The next tile's lines are requested into L2 while the products
// run, and two CTAs share an SM where the shared memory allows, so one loads while the other multiplies.
// What bounds it: N / 2 packed FMAs a complex sample (35 T FMA/s measured with fma.rn.f32x2; 25 T with scalar fma, whose
// three register operands meet in the register banks), and that a CTA's loads and products take turns: at N = 194, 16
// functions, a pass takes 1.0 to 1.2 ms, 0.3 of it the bytes, 0.5 the products (0.35 at the FMA rate), the rest loading and
// folding.  SO(3) passes of N = 80 to 222 run on the tensor cores instead (dft_tc.cu).
#include <algorithm>
#include <type_traits>

#include "common.cuh"
#include "direct_dft.cuh"

namespace fftso3 {

namespace ddft {

constexpr int MAXT = 512;  // threads of a CTA: one register tile each, at most 128 registers

// Tile of a pass: warps of QL blocks of four outputs x 128 / QL units; UB unit blocks a tile.
struct Shape {
    Fold f;
    int QL, UB, LT, threads;
    size_t smem;
};
static size_t smem_bytes(const Fold& f, int LT)
{
    return sizeof(float2) * mat_elems(f) + sizeof(float4) * f.H * (2 * LT + 1) + 3 * 2 * sizeof(long long) * LT + 16;
}
__global__ void build_table_kernel(float2* M, int N, const double2* tw)
{
    const Fold f = fold_of(N);
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e < mat_elems(f)) M[e] = mat_entry(f, e, tw);
}

// The shape with the fewest idle lanes among those of at least four warps; two CTAs of up to eight warps an SM (one loads while the other
// multiplies) before one, and (few units) tiles for every SM.
static Shape shape_of(int N, unsigned nu = 0x7fffffffu, int nsm = 1)
{
    Shape s = {};
    s.f = fold_of(N);
    double best = 0;
    for (int ql = 2; ql <= 4; ql *= 2)
        for (int ub = 1; ub <= 4; ++ub) {
            const int qw = (s.f.nb + ql - 1) / ql, warps = qw * ub, lt = ub * 128 / ql;
            const size_t b = smem_bytes(s.f, lt);
            if (32 * warps > MAXT || b > 227 * 1024) continue;
            const double sc = (double)s.f.nb / (ql * qw) * (b <= 113 * 1024 && warps <= 8 ? 1.0 : 0.6) * (warps >= 4 ? 1.0 : warps / 4.0) *
                                  std::min(1.0, (double)((nu + lt - 1) / lt) / nsm) +
                              0.01 * warps;
            if (sc > best) {
                best = sc;
                s.QL = ql;
                s.UB = ub;
                s.LT = lt;
                s.threads = 32 * warps;
                s.smem = b;
            }
        }
    return s;
}

// CTAs an SM holds (the runtime's occupancy query costs more than a small pass): shared memory, and 128 registers a thread
static int ctas_per_sm(const Shape& s)
{
    return std::max(1, std::min((int)(228 * 1024 / (s.smem + 1024)), 512 / s.threads));
}
static int device_sms()
{
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    return nsm;
}

struct Args {
    DirectPass p;
    const float4* table;
    int LT, UB;
    unsigned nu, ntiles;
    int nsm;
};

__device__ __forceinline__ void l2_prefetch(const void* p) { asm volatile("prefetch.global.L2 [%0];" ::"l"(p)); }

// LC: the input's lines are contiguous (else its units are); SC: the output's.  MIR: p.mirror.
template <int KIND, bool LC, bool SC, bool MIR, int QL>
__global__ void __launch_bounds__(MAXT, 1) direct_dft_kernel(const __grid_constant__ Args a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const DirectPass& p = a.p;
    const Fold f = fold_of(p.N);
    const int N = f.N, P = f.P, H = f.H, LT = a.LT, HU = LT / 2;
    // odd, so that the folding stores of consecutive t meet distinct banks
    const int TS = 2 * LT + 1;
    float2* M = reinterpret_cast<float2*>(smem_raw);
    // folded units [t] (TS apart) [parity][even units, then odd ones]: a pair of units is HU apart, so that a thread
    // owns adjacent units (16-byte global accesses) and reads them without bank conflicts
    float4* V = reinterpret_cast<float4*>(M + mat_elems(f));
    long long* tab = reinterpret_cast<long long*>(V + H * TS);  // [2 buffers][in, out, mirror][LT]
    constexpr bool REAL = KIND != DIRECT_COMPLEX;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;

    // offsets of a tile's units: input (-1: past the last unit), output, mirrored output (-1: none)
    auto tables = [&](unsigned tile, int buf) {
        long long* tb = tab + buf * 3 * LT;
        for (int i = tid; i < LT; i += blockDim.x) {
            const unsigned U = tile * LT + i;
            long long bi = -1, bo = 0, bm = -1;
            if (U < a.nu) {
                const unsigned fo = U / (unsigned)p.ni, u = U - fo * p.ni;
                const unsigned fn = fo / (unsigned)p.no, o = fo - fn * p.no;
                bi = fn * p.i_f + o * p.i_o + u * p.i_u;
                bo = fn * p.o_f + o * p.o_o + u * p.o_u;
                if (MIR && o > 0 && o < (unsigned)P) bm = fn * p.o_f + (N - (int)o) * p.o_o + u * p.o_u;
            }
            tb[i] = bi;
            tb[LT + i] = bo;
            tb[2 * LT + i] = bm;
        }
    };
    auto put = [&](int t, int u, const Folded& r) {
        float4* d = V + t * TS + (u >> 1) + (u & 1) * HU;
        d[0] = r.even;
        d[LT] = r.odd;
    };

    for (int e = tid; e < mat_elems(f) / 2; e += blockDim.x) reinterpret_cast<float4*>(M)[e] = __ldg(a.table + e);
    int buf = 0;
    if (blockIdx.x < a.ntiles) tables(blockIdx.x, 0);
    __syncthreads();
    // this thread's register tile
    const int qw = (f.nb + QL - 1) / QL, ub = warp / qw;
    const int qb = (warp - ub * qw) * QL + lane % QL;
    const bool active = ub < a.UB && qb < f.nb;
    const int par = qb >= f.nbE, qi = active ? (par ? qb - f.nbE : qb) : 0;
    constexpr int G = 32 / QL;
    const int pr = ub * 2 * G + lane / QL;  // first pair of units; the second G further on
    const float2 z = make_float2(0.f, 0.f);
    for (unsigned tile = blockIdx.x; tile < a.ntiles; tile += gridDim.x, buf ^= 1) {
        const long long* ib = tab + buf * 3 * LT;
        const long long* ob = ib + LT;
        const long long* mb = ob + LT;
        // ---- load and fold
        if (LC) {
            // consecutive threads take consecutive terms, then the next unit (a warp a unit left most lanes idle: forward of
            // l_max 9, 500 functions, 217 us, now 112; l_max 30, 134 functions, 720 and 461)
            const int ui = blockDim.x / H, ti = blockDim.x - ui * H;
            int u = tid / H, t = tid - u * H;
            const float2 z2 = make_float2(0.f, 0.f);
#pragma unroll 2
            while (u < LT) {
                const long long b = ib[u];
                const float* g0 = reinterpret_cast<const float*>(p.in) + (KIND == DIRECT_REAL_IN ? b : 2 * b);
                const float* g1 = g0 + p.i_l;
                auto at = [&](int j) {
                    return b < 0                    ? z2
                           : KIND == DIRECT_REAL_IN ? make_float2(__ldg(g0 + j), __ldg(g1 + j))
                                                    : __ldg(reinterpret_cast<const float2*>(g0) + j);
                };
                put(t, u, fold_line<REAL>(t, P, at(t), at(t ? N - t : 0), at(P - t), at(t ? P + t : P)));
                t += ti;
                u += ui;
                if (t >= H) {
                    t -= H;
                    ++u;
                }
            }
        } else {
            // 16 bytes a lane: a pair of complex units, or one unit of two real lines' spectra
            constexpr int UPL = KIND == DIRECT_REAL_OUT ? 1 : 2;
            const int np = LT / UPL, ti = blockDim.x / np, ui = blockDim.x - ti * np;
            int t = tid / np, u = tid - t * np;
            const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 2
            while (t < H) {
                const long long b = ib[u * UPL];
                const float2* g = reinterpret_cast<const float2*>(p.in) + b;
                auto at = [&](int j) { return b < 0 ? z4 : __ldg(reinterpret_cast<const float4*>(g + j * p.i_e)); };
                if (KIND == DIRECT_REAL_OUT) {
                    // f_j = X_0 + (-1)^j X_P + sum 2 Re X_t cos + 2 Im X_t sin: a_t = 2 Re X_t, b_t = 2 Im X_t; X_P = 0
                    const float4 x = at(t), y = t ? at(P - t) : z4;
                    const float c = t ? 2.f : 1.f, s = t ? 2.f : 0.f;
                    put(t, u, fold_ab<true>(t, P, make_float2(c * x.x, c * x.z), make_float2(s * x.y, s * x.w),
                                            make_float2(c * y.x, c * y.z), make_float2(s * y.y, s * y.w)));
                } else {
                    const float4 x = at(t), xn = at(t ? N - t : 0);
                    const float4 xp = p.nyq && t == 0 ? z4 : at(P - t), xq = t ? at(P + t) : xp;
                    put(t, 2 * u, fold_line<false>(t, P, make_float2(x.x, x.y), make_float2(xn.x, xn.y),
                                                   make_float2(xp.x, xp.y), make_float2(xq.x, xq.y)));
                    put(t, 2 * u + 1, fold_line<false>(t, P, make_float2(x.z, x.w), make_float2(xn.z, xn.w),
                                                       make_float2(xp.z, xp.w), make_float2(xq.z, xq.w)));
                }
                t += ti;
                u += ui;
                if (u >= np) {
                    u -= np;
                    ++t;
                }
            }
        }
        const unsigned next = tile + gridDim.x;
        if (next < a.ntiles) tables(next, buf ^ 1);
        __syncthreads();
        // ---- the next tile's input into L2 under this tile's products
        if (next < a.ntiles) {
            const long long* nb = tab + (buf ^ 1) * 3 * LT;
            if (LC) {
                const int bytes = N * (KIND == DIRECT_REAL_IN ? 4 : 8);
                const int lines = KIND == DIRECT_REAL_IN ? 2 * LT : LT;
                const int per = (bytes + 124 + 127) / 128;  // a line's 128-byte runs, wherever it begins
                for (int k = tid; k < lines * per; k += blockDim.x) {
                    const int i = k / per, c = 128 * (k - i * per);
                    const long long b = nb[KIND == DIRECT_REAL_IN ? i >> 1 : i];
                    if (b < 0) continue;
                    const char* g = reinterpret_cast<const char*>(p.in) +
                                    (KIND == DIRECT_REAL_IN ? 4 * (b + (i & 1) * p.i_l) : 8 * b);
                    l2_prefetch(g + min(c, bytes - 4));
                }
            } else {
                const int per = (LT * (KIND == DIRECT_REAL_OUT ? 16 : 8) + 127) / 128;
                const int last = KIND == DIRECT_REAL_OUT ? P : N;
                // units of one (f, o) are adjacent; a tile that crosses into the next leaves the rest to the loads
                if (lane < per && nb[0] >= 0) {
                    const int u = min(lane * (KIND == DIRECT_REAL_OUT ? 8 : 16), LT - 1);
                    if (nb[u] == nb[0] + u * p.i_u) {
                        const float2* g = reinterpret_cast<const float2*>(p.in) + nb[u];
                        for (int j = warp; j < last; j += nw) l2_prefetch(g + j * p.i_e);
                    }
                }
            }
        }
        // ---- products
        Tile acc;
        if (active) product<QL>(M + par * f.QS + 4 * qi, V + par * LT + pr, H, f.QS, HU, TS, acc);
        const int q0 = 8 * qi + par;  // outputs q0, q0 + 2, q0 + 4, q0 + 6 (<= P)
        if (!SC) {
            if (active) {
                const long long step = 2 * p.o_e;
                if (KIND == DIRECT_REAL_IN) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int u = 2 * (pr + (j >> 1) * G) + (j & 1);
                        if (ib[u] < 0) continue;
                        float2* o = reinterpret_cast<float2*>(p.out) + ob[u];
                        float2* lo = o + q0 * p.o_e;
                        float2* hi = o + (N - q0) * p.o_e;
#pragma unroll
                        for (int i = 0; i < 4; ++i, lo += step, hi -= step) {
                            const int q = q0 + 2 * i;
                            if (q > P) break;
                            const float2 A = unpack2(acc.A[i][j]), B = unpack2(acc.B[i][j]);
                            *reinterpret_cast<float4*>(lo) = make_float4(A.x, -A.y, B.x, -B.y);
                            if (p.full && q > 0 && q < P)
                                *reinterpret_cast<float4*>(hi) = make_float4(A.x, A.y, B.x, B.y);
                        }
                    }
                } else {
#pragma unroll
                    for (int h = 0; h < 2; ++h) {
                        const int u = 2 * (pr + h * G);
                        if (ib[u] < 0) continue;  // the units come in pairs (nu and ni are even)
                        float2* o = reinterpret_cast<float2*>(p.out) + ob[u];
                        float2* lo = o + q0 * p.o_e;
                        float2* hi = o + (N - q0) * p.o_e;
                        const long long mo = MIR ? mb[u] - ob[u] : 0;
                        const bool mir = MIR && mb[u] >= 0;
#pragma unroll
                        for (int i = 0; i < 4; ++i, lo += step, hi -= step) {
                            const int q = q0 + 2 * i;
                            if (q > P) break;
                            const float2 A0 = unpack2(acc.A[i][2 * h]), B0 = unpack2(acc.B[i][2 * h]);
                            const float2 A1 = unpack2(acc.A[i][2 * h + 1]), B1 = unpack2(acc.B[i][2 * h + 1]);
                            const float4 x = make_float4(A0.x + A0.y, B0.x - B0.y, A1.x + A1.y, B1.x - B1.y);
                            const float4 y = make_float4(A0.x - A0.y, B0.x + B0.y, A1.x - A1.y, B1.x + B1.y);
                            *reinterpret_cast<float4*>(lo) = x;
                            if (q > 0 && q < P) *reinterpret_cast<float4*>(hi) = y;
                            if (MIR && mir) {
                                // (o, q) -> (N - o, N - q) and (o, N - q) -> (N - o, q), conjugated
                                if (q > 0) *reinterpret_cast<float4*>(hi + mo) = make_float4(x.x, -x.y, x.z, -x.w);
                                if (q < P) *reinterpret_cast<float4*>(lo + mo) = make_float4(y.x, -y.y, y.z, -y.w);
                            }
                        }
                    }
                }
            }
            __syncthreads();
        } else {
            // through shared memory (over the folded units): rows of N + 1 elements
            __syncthreads();
            if (active) {
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const int u = 2 * (pr + (j >> 1) * G) + (j & 1);
                    float2* r = reinterpret_cast<float2*>(V) + u * (N + 1);
                    float* r0 = reinterpret_cast<float*>(V) + 2 * u * (N + 1);
                    float* r1 = r0 + N + 1;
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const int q = q0 + 2 * i;
                        if (q > P) break;
                        const float2 A = unpack2(acc.A[i][j]), B = unpack2(acc.B[i][j]);
                        if (KIND == DIRECT_REAL_OUT) {
                            r0[q] = A.x + A.y;
                            r1[q] = B.x + B.y;
                            if (q > 0 && q < P) {
                                r0[N - q] = A.x - A.y;
                                r1[N - q] = B.x - B.y;
                            }
                        } else {
                            r[q] = make_float2(A.x + A.y, B.x - B.y);
                            if (q > 0 && q < P) r[N - q] = make_float2(A.x - A.y, B.x + B.y);
                        }
                    }
                }
            }
            __syncthreads();
            using E = std::conditional_t<KIND == DIRECT_REAL_OUT, float, float2>;
            const E* r = reinterpret_cast<const E*>(V);
            const int rows = KIND == DIRECT_REAL_OUT ? 2 * LT : LT;
            auto row = [&](int i) {  // its place, or null: past the last unit
                const int u = KIND == DIRECT_REAL_OUT ? i >> 1 : i;
                return ib[u] < 0 ? nullptr : reinterpret_cast<E*>(p.out) + ob[u] + (KIND == DIRECT_REAL_OUT ? (i & 1) * p.o_l : 0);
            };
            if (N < 64) {
                // threads over all rows (a warp a row left most lanes idle: inverse of l_max 6, 200 real functions, 62 us, now
                // 44; from N = 78 on the rows are up to 8 % faster)
                const int ri = blockDim.x / N, ji = blockDim.x - ri * N;
                int i = tid / N, j = tid - i * N;
#pragma unroll 4
                while (i < rows) {
                    if (E* o = row(i)) o[j] = r[i * (N + 1) + j];
                    j += ji;
                    i += ri;
                    if (j >= N) {
                        j -= N;
                        ++i;
                    }
                }
            } else {
                for (int i = warp; i < rows; i += nw) {
                    E* o = row(i);
                    if (!o) continue;
#pragma unroll 4
                    for (int j = lane; j < N; j += 32) o[j] = r[i * (N + 1) + j];
                }
            }
            __syncthreads();
        }
    }
}

template <int KIND, bool LC, bool SC, bool MIR, int QL>
static cudaError_t run_ql(const Args& a, const Shape& s, cudaStream_t st)
{
    auto kern = direct_dft_kernel<KIND, LC, SC, MIR, QL>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)s.smem);
    if (e != cudaSuccess) return e;
    const unsigned nblk = std::min(a.ntiles, (unsigned)(a.nsm * ctas_per_sm(s)));
    kern<<<nblk, s.threads, s.smem, st>>>(a);
    return cudaGetLastError();
}

template <int KIND, bool LC, bool SC, bool MIR = false>
static cudaError_t run(const Args& a, const Shape& s, cudaStream_t st)
{
    return s.QL == 4 ? run_ql<KIND, LC, SC, MIR, 4>(a, s, st) : run_ql<KIND, LC, SC, MIR, 2>(a, s, st);
}

}  // namespace ddft

using namespace ddft;

size_t direct_dft_table_bytes(int N) { return sizeof(float2) * mat_elems(fold_of(N)); }

cudaError_t direct_dft_build_table(void* table, int N, const void* tw, cudaStream_t st)
{
    build_table_kernel<<<(mat_elems(fold_of(N)) + 255) / 256, 256, 0, st>>>((float2*)table, N, (const double2*)tw);
    return cudaGetLastError();
}

bool direct_dft_supported(int N)
{
    if (N < 2 || N % 2) return false;
    const Shape s = shape_of(N);
    return s.QL > 0;
}

double direct_dft_fill(int N, long long units)
{
    const int nsm = device_sms();
    const Shape s = shape_of(N, (unsigned)std::min(units, 0x7fffffffLL), nsm);
    if (!s.QL || nsm < 1) return 0;
    const long long tiles = (units + s.LT - 1) / s.LT, slots = (long long)nsm * ctas_per_sm(s);
    return (double)tiles / (double)((tiles + slots - 1) / slots * slots);
}

cudaError_t launch_direct_dft(const DirectPass& p, const void* table, cudaStream_t st)
{
    if (!direct_dft_supported(p.N) || p.nf < 1 || p.no < 1 || p.ni < 1) return cudaErrorInvalidValue;
    if (p.nf > (0x7fffffffLL / p.no) / p.ni) return cudaErrorInvalidValue;
    Args a;
    a.p = p;
    a.nu = (unsigned)(p.nf * p.no * p.ni);
    const int nsm = device_sms();
    const Shape s = shape_of(p.N, a.nu, nsm);
    a.table = (const float4*)table;
    a.LT = s.LT;
    a.UB = s.UB;
    a.nsm = nsm;
    a.ntiles = (a.nu + s.LT - 1) / s.LT;
    const bool lc = p.i_e == 1, sc = p.o_e == 1;
    if (p.kind == DIRECT_REAL_IN && lc && !sc) return run<DIRECT_REAL_IN, true, false>(a, s, st);
    if (p.kind == DIRECT_REAL_OUT && !lc && sc && p.nyq) return run<DIRECT_REAL_OUT, false, true>(a, s, st);
    if (p.kind != DIRECT_COMPLEX || p.ni % 2) return cudaErrorInvalidValue;
    if (lc && !sc) return p.mirror ? run<DIRECT_COMPLEX, true, false, true>(a, s, st) : run<DIRECT_COMPLEX, true, false>(a, s, st);
    if (!lc && !sc) return run<DIRECT_COMPLEX, false, false>(a, s, st);
    if (!lc && sc) return run<DIRECT_COMPLEX, false, true>(a, s, st);
    return cudaErrorInvalidValue;
}

cudaError_t launch_direct_grid_pass(const void* in, void* out, long long nf, int N, int pass, bool real, bool half,
                                    const void* table, cudaStream_t st)
{
    const long long n = N, NN = n * n, NNN = NN * n;
    const int B = N / 2;
    DirectPass p = {in, out, N, DIRECT_COMPLEX, nf, 0, 0, NNN, 0, 0, 0, 0, NNN, 0, 0, 0, 0, false, false, false};
    auto side_in = [&](long long o, long long u, long long e) { p.i_o = o; p.i_u = u; p.i_e = e; };
    auto side_out = [&](long long o, long long u, long long e) { p.o_o = o; p.o_u = u; p.o_e = e; };
    switch (pass) {
        case 1:  // o = k, units j1
            p.no = N;
            if (real) {
                p.kind = DIRECT_REAL_IN;
                p.ni = B;
                p.i_l = n;
                side_in(NN, 2 * n, 1);
                side_out(NN, 2, n);
            } else {
                p.ni = N;
                side_in(NN, n, 1);
                side_out(NN, 1, n);
            }
            break;
        case 2:  // o = q, units k
            p.no = real ? B + 1 : N;
            p.ni = N;
            p.mirror = real && !half;
            side_in(n, NN, 1);
            side_out(n, 1, NN);
            break;
        case -2:  // o = q, units k; q = B holds only Nyquist bins, which the next pass takes as zero
            p.no = real ? B : N;
            p.ni = N;
            p.nyq = true;
            side_in(n, 1, NN);
            side_out(n, 1, NN);
            break;
        case -1:  // o = j1, units k
            p.no = N;
            p.nyq = true;
            if (real) {
                p.kind = DIRECT_REAL_OUT;
                p.ni = B;
                p.o_l = NN;
                side_in(NN, 2, n);
                side_out(n, 2 * NN, 1);
            } else {
                p.ni = N;
                side_in(NN, 1, n);
                side_out(n, NN, 1);
            }
            break;
        default: return cudaErrorInvalidValue;
    }
    return launch_direct_dft(p, table, st);
}

cudaError_t launch_direct_s2_pass(const void* in, void* out, long long nf, int N, int dir, bool real, bool half,
                                  const void* table, cudaStream_t st)
{
    const long long n = N, NN = n * n;
    DirectPass p = {in, out, N, DIRECT_COMPLEX, nf, 1, N, NN, 0, 0, 0, 0, NN, 0, 0, 0, 0, false, false, false};
    if (dir == 1) {  // units k
        p.i_e = 1;
        p.o_e = n;
        p.i_u = n;
        p.o_u = 1;
        if (real) {
            p.kind = DIRECT_REAL_IN;
            p.full = !half;
            p.ni = N / 2;
            p.i_l = n;
            p.i_u = 2 * n;
            p.o_u = 2;
        }
    } else {
        p.nyq = true;
        p.i_e = n;
        p.o_e = 1;
        p.i_u = 1;
        p.o_u = n;
        if (real) {
            p.kind = DIRECT_REAL_OUT;
            p.ni = N / 2;
            p.i_u = 2;
            p.o_u = 2 * n;
            p.o_l = n;
        }
    }
    return launch_direct_dft(p, table, st);
}

}  // namespace fftso3
