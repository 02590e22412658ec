// Direct FP64 DFT of short lines (the FP64 plans' FFT passes where the mixed-radix kernel of fft.cu is the slower one).
//
// The folding of direct_dft.cuh in FP64: N^2 / 2 FMAs a complex line, and one thread an output pair X[q], X[N - q] of one
// line with four independent sums.  For short lines the mixed-radix kernel is bound by its stages' latencies (a barrier, a
// round through shared memory and FP64 index twiddles each) and, at N = 2p, by the prime stage's 8p operations an element:
// one pass over a 34^3 grid took 23 to 29 us, of which the FP64 units need 1.4.  Here a CTA holds a few lines only, so that
// the sums of a small grid spread over every SM's FP64 units (1.6 FMAs a clock and SM, measured).
#include <algorithm>

#include "common.cuh"
#include "fft.cuh"

namespace fftso3 {

namespace {

constexpr int T64 = 128;

struct D64 {
    const void* in;
    void* out;
    const double2* tw;
    long long nlines, inner, ostride, istride, es;
    int N, lpb, nyq, herm, skip;
};

__device__ __forceinline__ double2 dadd(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
__device__ __forceinline__ double2 dsub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }

// RI: real samples in; RO: the real part out.
template <bool RI, bool RO>
__global__ void __launch_bounds__(T64) dft64_kernel(const D64 a)
{
    extern __shared__ double2 sm64[];
    const int N = a.N, P = N / 2, H = P / 2 + 1, LB = a.lpb;
    double2* W = sm64;           // e^{-2 pi i j / N}
    double2* V = W + N;          // [four folded terms][t][line]
    const int tid = threadIdx.x;
    for (int j = tid; j < N; j += T64) W[j] = __ldg(a.tw + j);
    const long long line0 = (long long)blockIdx.x * LB;
    const int nl = (int)min((long long)LB, a.nlines - line0);
    auto base = [&](int l) {
        const long long i = line0 + l;
        return (i / a.inner) * a.ostride + (i % a.inner) * a.istride;
    };
    const double2 z = make_double2(0., 0.);
    for (int e = tid; e < H * LB; e += T64) {
        const int t = e / LB, l = e - t * LB;
        double2 v[4] = {z, z, z, z};
        if (l < nl) {
            const long long b = base(l);
            auto at = [&](int j) {
                if (a.nyq && j == P) return z;
                if (RI) return make_double2(reinterpret_cast<const double*>(a.in)[b + j * a.es], 0.);
                const bool c = a.herm && j > P;
                double2 x = reinterpret_cast<const double2*>(a.in)[b + (c ? N - j : j) * a.es];
                if (c) x.y = -x.y;
                return x;
            };
            const double2 x0 = at(t), x1 = t ? at(N - t) : z;
            const double2 a0 = dadd(x0, x1), b0 = t ? dsub(x0, x1) : z;
            if (2 * t == P) {
                v[0] = a0;
                v[3] = b0;
            } else {
                const double2 x2 = at(P - t), x3 = t ? at(P + t) : z;
                const double2 a1 = dadd(x2, x3), b1 = t ? dsub(x2, x3) : z;
                v[0] = dadd(a0, a1);
                v[1] = dsub(b0, b1);
                v[2] = dsub(a0, a1);
                v[3] = dadd(b0, b1);
            }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) V[(j * H + t) * LB + l] = v[j];
    }
    __syncthreads();
    for (int e = tid; e < (P + 1) * LB; e += T64) {
        const int q = e / LB, l = e - q * LB;
        // lines of the Nyquist row (skip): not read by the next pass
        if (l >= nl || (a.skip >= 0 && (line0 + l) % a.inner == a.skip)) continue;
        const double2* vc = V + 2 * (q & 1) * H * LB + l;
        const double2* vs = vc + H * LB;
        double cr = 0., ci = 0., sr = 0., si = 0.;
        int i = 0;  // t q mod N
        for (int t = 0; t < H; ++t) {
            const double2 w = W[i], c = vc[t * LB], s = vs[t * LB];
            cr = __fma_rn(c.x, w.x, cr);
            if (!RI && !RO) ci = __fma_rn(c.y, w.x, ci);
            if (!RO) sr = __fma_rn(s.x, w.y, sr);  // -S
            if (!RI) si = __fma_rn(s.y, w.y, si);
            i += q;
            if (i >= N) i -= N;
        }
        // X[q], X[N - q] = C -/+ i S
        const long long b = base(l);
        const bool two = q > 0 && q < P;
        if (RO) {
            double* o = reinterpret_cast<double*>(a.out) + b;
            o[q * a.es] = cr - si;
            if (two) o[(N - q) * a.es] = cr + si;
        } else {
            double2* o = reinterpret_cast<double2*>(a.out) + b;
            o[q * a.es] = make_double2(cr - si, ci + sr);
            if (two) o[(N - q) * a.es] = make_double2(cr + si, ci - sr);
        }
    }
}

}  // namespace

// The direct form below N = 64 and where it takes less than 0.72 of the mixed radices' FP64 operations.  Both directions of
// complex functions, direct over mixed radices (ratio of the operations): N = 56 (0.77) 0.82, 60 (0.79) 0.92, 62 (0.12) 0.26; 64
// (1.33) 1.12; 70 (0.71) 0.86, 154 (0.64) 0.97, 238 (0.71) 0.79, 286 (0.719) 0.93; 266 (0.725) 1.04, 176 (0.82) 1.14, 198
// (0.85) 1.15, 98 (0.88) 1.20, 84 (0.93) 1.15, 90 (0.99) 1.22, 260 (0.99) 1.25.  By N alone: batches keep a single plan's bits.
bool dft64_supported(int N)
{
    if (N < 2 || N % 2) return false;
    if (N < 64) return true;
    if (N > 512) return false;
    FFTFactors f;
    make_fft_factors(N, f);
    double cost = 0;
    for (int i = 0; i < f.n; ++i) cost += f.r[i] > 8 ? 8.0 * f.r[i] : f.r[i] == 8 ? 12 : f.r[i] == 4 ? 10 : f.r[i] == 2 ? 7 : 3.5 * f.r[i];
    return 0.5 * N < 0.72 * cost;
}

cudaError_t launch_dft64(const FFTLaunch& L, cudaStream_t st)
{
    const int N = L.fac.N, P = N / 2, H = P / 2 + 1;
    if (!dft64_supported(N) || (L.real_in && L.real_out)) return cudaErrorInvalidValue;
    int dev = 0, nsm = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    // lines a CTA: about two outputs a thread, fewer while some SMs would have none
    int lpb = std::max(1, std::min(16, 2 * T64 / (P + 1)));
    while (lpb > 1 && L.nlines / lpb < 2 * nsm) --lpb;
    D64 a = {L.in, L.out, (const double2*)L.tw, L.nlines, L.inner, L.ostride, L.istride, L.es, N, lpb, L.nyq, L.herm, L.skip};
    const size_t smem = sizeof(double2) * (N + 4 * H * lpb);
    const long long nblk = (L.nlines + lpb - 1) / lpb;
    if (nblk > 0x7fffffffLL) return cudaErrorInvalidValue;
    auto kern = L.real_in ? dft64_kernel<true, false> : L.real_out ? dft64_kernel<false, true> : dft64_kernel<false, false>;
    kern<<<(unsigned)nblk, T64, smem, st>>>(a);
    return cudaGetLastError();
}

}  // namespace fftso3
