// FP64 beta-sum contractions (the plain method) and the coefficient-basis
// conversions of the real transforms.
//
// SO(3) forward (fdcl_FFTSO3.cpp:704-740):
//   F(l,m,n) = sum_k w_k d^l_mn(beta_k) G_k(-m mod N, -n mod N),
// where G_k is the unscaled 2-D DFT of the beta_k slice.  One CTA per
// (symmetry group, function): the group's <= 4 (m,n) pairs share one table
// block d_g[l][k], so X[p][k] = w_k G_k(pair p) is staged in shared memory and
// each warp takes four rows l at a time, eight lanes a row over k, finishing
// with a shuffle reduction over the eight.
//
// SO(3) inverse (grid form of fdcl_FFTSO3.cpp:498-531):
//   H_k(m,n) = sum_l (2l+1) F(l,m,n) d^l_mn(beta_k), placed at bin
//   (m mod N, n mod N) of slice k; a forward 2-D DFT of the slice then gives
//   f(alpha_j1, beta_k, gamma_j2) = sum_mn H_k(m,n) e^{-i m alpha_j1} e^{-i n gamma_j2}.
//   Threads over k (coalesced table reads), (2l+1) F staged in shared memory.
//
// S^2 is the same pattern with the Legendre table and groups m >= 0 serving
// the pairs (m, -m) (fdcl_FFTS2.cpp:157-173 forward, :194-230 inverse), its
// sums folded by parity.
#include "common.cuh"
#include "contract.cuh"
#include "rsph.cuh"

namespace fftso3 {

__device__ __forceinline__ int mod_n(int a, int N) { int r = a % N; return r < 0 ? r + N : r; }

// Reduce-scatter of 8 (4) per-lane partial sums over eight neighbouring lanes: lane `sub` of them gets the full sum of value
// sub (sub >> 1); each level halves the values a lane carries.  The forward sums take eight lanes a degree, four degrees a
// warp: 7 (4) FP64 additions for all four.  Over a whole warp a degree it took 9 (7) for each, a third to as many as the
// products of N < 100, so the forward sums of l_max 127, real, went from 1.63 to 1.36 ms.
__device__ __forceinline__ double reduce_scatter(const double (&v)[8], int sub)
{
    const bool b2 = sub & 4, b1 = sub & 2, b0 = sub & 1;
    double w[4], x[2];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = (b2 ? v[j + 4] : v[j]) + __shfl_xor_sync(0xffffffffu, b2 ? v[j] : v[j + 4], 4);
#pragma unroll
    for (int j = 0; j < 2; ++j) x[j] = (b1 ? w[j + 2] : w[j]) + __shfl_xor_sync(0xffffffffu, b1 ? w[j] : w[j + 2], 2);
    return (b0 ? x[1] : x[0]) + __shfl_xor_sync(0xffffffffu, b0 ? x[0] : x[1], 1);
}
__device__ __forceinline__ double reduce_scatter(const double (&v)[4], int sub)
{
    const bool b2 = sub & 4, b1 = sub & 2;
    double w[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) w[j] = (b2 ? v[j + 2] : v[j]) + __shfl_xor_sync(0xffffffffu, b2 ? v[j] : v[j + 2], 4);
    double y = (b1 ? w[1] : w[0]) + __shfl_xor_sync(0xffffffffu, b1 ? w[0] : w[1], 2);
    y += __shfl_xor_sync(0xffffffffu, y, 1);
    return y;
}

// ------------------------------------------------------------------ SO(3)

// REAL: the pairs 0 and 2 only; the transform of real samples is Hermitian, so the others are (-1)^(m+n) times their
// conjugates (half of the sums).
template <int NT, bool REAL>
__global__ void __launch_bounds__(NT) so3_fwd_fp64_kernel(const double* __restrict__ table,
                                                          const long long* __restrict__ goff,
                                                          const double2* __restrict__ G, const double* __restrict__ w,
                                                          double2* __restrict__ F, int L, int N, long long gstride,
                                                          long long cstride)
{
    constexpr int S = REAL ? 2 : 1, NP = 4 / S;  // pair of slot p: S p
    extern __shared__ double2 X[];  // [NP][N]
    const int g = blockIdx.x, b = blockIdx.y;
    int m0, n0;
    group_mn(g, m0, n0);
    const GroupPairs P = group_pairs(m0, n0);
    const int np = (P.np + S - 1) / S;
    const double2* Gb = G + (long long)b * gstride;
    const long long NN = (long long)N * N;
    for (int i = threadIdx.x; i < np * N; i += NT) {
        int p = i / N, k = i - p * N;
        int pi = mod_n(-P.m[S * p], N), qi = mod_n(-P.n[S * p], N);
        const bool c = REAL && qi > N / 2;  // read as the conjugate of the mirrored bin
        if (c) {
            pi = pi ? N - pi : 0;
            qi = N - qi;
        }
        double2 v = Gb[(long long)k * NN + (long long)pi * N + qi];
        double wk = w[k];
        X[p * N + k] = make_double2(wk * v.x, c ? -(wk * v.y) : wk * v.y);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 7;
    const double* tg = table + goff[g];
    double* Fb = reinterpret_cast<double*>(F + (long long)b * cstride);
    // after the reduce-scatter lane `sub` of a degree holds value vi = 2 p + (re, im) of slot p (REAL: two lanes each)
    const int vi = REAL ? sub >> 1 : sub;
    const int wp = vi >> 1, wq = S * wp;
    const bool writer = !(REAL && (sub & 1)) && wp < np;
    const int wm = wp < np ? P.m[wq] : 0, wn = wp < np ? P.n[wq] : 0;
    const double wsign = wp < np ? (double)P.sign[wq] : 0.;
    // the conjugate partner (-m, -n): (-1)^(m+n) conj
    const double csign = (((wm + wn) & 1) ? -1. : 1.) * ((vi & 1) ? -1. : 1.);
    for (int l0 = m0 + 4 * warp; l0 <= L; l0 += NT / 8) {
        const int l = l0 + (lane >> 3);
        const double* drow = tg + (long long)(min(l, L) - m0) * N;
        double v[2 * NP];
#pragma unroll
        for (int j = 0; j < 2 * NP; ++j) v[j] = 0.;
        for (int k = sub; k < N; k += 8) {
            double d = drow[k];
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (p < np) {
                    double2 x = X[p * N + k];
                    v[2 * p] += d * x.x;
                    v[2 * p + 1] += d * x.y;
                }
        }
        const double y = reduce_scatter(v, sub);
        if (writer && l <= L) {
            Fb[2 * so3_idx(l, wm, wn) + (vi & 1)] = wsign * y;
            if (REAL && m0 > 0) Fb[2 * so3_idx(l, -wm, -wn) + (vi & 1)] = csign * (wsign * y);
        }
    }
}

// REAL: the pairs 0 and 2 only; H(-m, -n) = conj H(m, n) for the coefficients of a real function.
template <int NT, bool REAL>
__global__ void __launch_bounds__(NT) so3_inv_fp64_kernel(const double* __restrict__ table,
                                                          const long long* __restrict__ goff,
                                                          const double2* __restrict__ F, double2* __restrict__ H,
                                                          int L, int N, long long gstride, long long cstride)
{
    constexpr int S = REAL ? 2 : 1, NP = 4 / S;
    extern __shared__ double2 Y[];  // [NP][B]
    const int g = blockIdx.x, b = blockIdx.y;
    const int B = L + 1;
    int m0, n0;
    group_mn(g, m0, n0);
    const GroupPairs P = group_pairs(m0, n0);
    const int nl = B - m0, np = (P.np + S - 1) / S;
    const double2* Fb = F + (long long)b * cstride;
    for (int i = threadIdx.x; i < np * nl; i += NT) {
        int p = i / nl, l = m0 + (i - p * nl);
        double2 c = Fb[so3_idx(l, P.m[S * p], P.n[S * p])];
        double s = (double)(2 * l + 1) * P.sign[S * p];
        Y[p * B + (l - m0)] = make_double2(s * c.x, s * c.y);
    }
    __syncthreads();
    const double* tg = table + goff[g];
    double2* Hb = H + (long long)b * gstride;
    const long long NN = (long long)N * N;
    for (int k = threadIdx.x; k < N; k += NT) {
        double ar[NP], ai[NP];
#pragma unroll
        for (int p = 0; p < NP; ++p) ar[p] = ai[p] = 0.;
        for (int j = 0; j < nl; ++j) {
            double d = tg[(long long)j * N + k];
#pragma unroll
            for (int p = 0; p < NP; ++p)
                if (p < np) {
                    double2 y = Y[p * B + j];
                    ar[p] += d * y.x;
                    ai[p] += d * y.y;
                }
        }
#pragma unroll
        for (int p = 0; p < NP; ++p)
            if (p < np) {
                const int m = P.m[S * p], n = P.n[S * p];
                Hb[(long long)k * NN + (long long)mod_n(m, N) * N + mod_n(n, N)] = make_double2(ar[p], ai[p]);
                if (REAL && m0 > 0)
                    Hb[(long long)k * NN + (long long)mod_n(-m, N) * N + mod_n(-n, N)] = make_double2(ar[p], -ai[p]);
            }
    }
}

// Zero the Nyquist row p = B and column q = B of every N x N slice (the bins
// no (m, n) with |m|, |n| <= L maps to).
template <typename C>
__global__ void zero_nyquist_so3_kernel(C* __restrict__ H, int N, long long nslices)
{
    long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nslices * 2 * N) return;
    long long s = idx / (2 * N);
    int r = (int)(idx % (2 * N));
    int B = N / 2;
    C z;
    z.x = 0;
    z.y = 0;
    C* slice = H + s * N * N;
    if (r < N)
        slice[(long long)B * N + r] = z;
    else
        slice[(long long)(r - N) * N + B] = z;
}

// The basis changes, F_r = Re(T F_c T^H) per l (fdcl_FFTSO3.cpp:1169-1181) and back, F_c = T^H F_r T (the complex
// coefficients whose synthesis equals the real synthesis of F_r).  One thread a quadruple (l, +-mu, +-nu), which is closed
// under both: every coefficient is read and written once.  (One CTA a degree read each four times and left most SMs idle at
// a batch of one: 0.56 and 0.43 ms at l_max 127 in FP64, now 0.04 and 0.05.)  HERM: the FP64 forward writes exact conjugate pairs.
__device__ __forceinline__ int quad_off(int l) { return l * (l + 1) * (2 * l + 1) / 6; }
__device__ __forceinline__ void quad_of(int e, int& l, int& mu, int& nu)
{
    l = (int)cbrtf(3.f * (float)e);
    while (l > 0 && quad_off(l) > e) --l;
    while (quad_off(l + 1) <= e) ++l;
    const int r = e - quad_off(l);
    nu = r / (l + 1);
    mu = r - nu * (l + 1);
}

template <typename CIN, typename ROUT, typename A, bool HERM>
__global__ void so3_c2r_kernel(const CIN* __restrict__ Fc, ROUT* __restrict__ Fr, int nquad, long long C)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nquad) return;
    int l, mu, nu;
    quad_of(e, l, mu, nu);
    const CIN* fc = Fc + (long long)blockIdx.y * C;
    ROUT* fr = Fr + (long long)blockIdx.y * C;
    c2t<A> v[2][2];  // [a < 0][b < 0]
#pragma unroll
    for (int i = 0; i < (HERM ? 1 : 2); ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const CIN x = fc[so3_idx(l, i ? -mu : mu, j ? -nu : nu)];
            v[i][j] = {(A)x.x, (A)x.y};
        }
    auto at = [&](int a, int b) { return a < 0 ? (b < 0 ? v[1][1] : v[1][0]) : (b < 0 ? v[0][1] : v[0][0]); };
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int m = i ? -mu : mu, n = j ? -nu : nu;
            if ((i && mu == 0) || (j && nu == 0)) continue;
            fr[so3_idx(l, m, n)] = (ROUT)real_coefficient<A, HERM>(m, n, at);
        }
}

template <typename RIN, typename COUT, typename A>
__global__ void so3_r2c_kernel(const RIN* __restrict__ Fr, COUT* __restrict__ Fc, int nquad, long long C)
{
    const int e = blockIdx.x * blockDim.x + threadIdx.x;
    if (e >= nquad) return;
    int l, mu, nu;
    quad_of(e, l, mu, nu);
    const RIN* fr = Fr + (long long)blockIdx.y * C;
    COUT* fc = Fc + (long long)blockIdx.y * C;
    A v[2][2];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) v[i][j] = (A)fr[so3_idx(l, i ? -mu : mu, j ? -nu : nu)];
    auto at = [&](int a, int b) { return a < 0 ? (b < 0 ? v[1][1] : v[1][0]) : (b < 0 ? v[0][1] : v[0][0]); };
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const int m = i ? -mu : mu, n = j ? -nu : nu;
            if ((i && mu == 0) || (j && nu == 0)) continue;
            const c2t<A> x = complex_coefficient<A>(m, n, at);
            COUT o;
            o.x = x.x;
            o.y = x.y;
            fc[so3_idx(l, m, n)] = o;
        }
}

// ------------------------------------------------------------------- S^2

// P_l^m(pi - beta) = (-1)^(l - m) P_l^m(beta), and beta_{N-1-k} = pi - beta_k: both directions take the samples k < N / 2 alone,
// the forward against sums (l - m even) and differences (odd) of the two halves, the inverse with the even and the odd degrees'
// sums E and O, H(k) = E + O, H(N-1-k) = E - O.  Half of the FP64 operations (which bound large l_max) and of the table reads;
// l_max 47, 8 functions: 26.5 and 19.1 us, now 14.5 and 15.0.
template <int NT>
__global__ void __launch_bounds__(NT) s2_fwd_fp64_kernel(const double* __restrict__ table,
                                                         const long long* __restrict__ moff,
                                                         const double2* __restrict__ G, const double* __restrict__ w,
                                                         double2* __restrict__ F, int L, int N, long long gstride,
                                                         long long cstride, int is_real)
{
    extern __shared__ double2 X[];  // [l - m odd][pair][N / 2]
    const int m = blockIdx.x, b = blockIdx.y, P = N / 2;
    const int np = (m > 0 && !is_real) ? 2 : 1;
    const double2* Gb = G + (long long)b * gstride;
    for (int i = threadIdx.x; i < np * P; i += NT) {
        const int p = i / P, k = i - p * P, kn = N - 1 - k;
        const int bin = (p == 0) ? m : N - m;  // F_k(m) and F_k(2B + (-m)), fdcl_FFTS2.cpp:162,165
        const double2 v = Gb[(long long)k * N + bin], u = Gb[(long long)kn * N + bin];
        const double wv = w[k], wu = w[kn];
        const double2 a = make_double2(wv * v.x, wv * v.y), c = make_double2(wu * u.x, wu * u.y);
        X[p * P + k] = make_double2(a.x + c.x, a.y + c.y);
        X[N + p * P + k] = make_double2(a.x - c.x, a.y - c.y);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, sub = lane & 7;
    const double* tg = table + moff[m];
    double* Fd = reinterpret_cast<double*>(F + (long long)b * cstride);
    const double sg = (m & 1) ? -1. : 1.;
    // eight lanes a degree, four degrees of one parity a warp; lane sub ends with value sub >> 1 = 2 p + (re, im) of pair p
    // (p = 1: -m)
    const int wp = sub >> 2, wc = (sub >> 1) & 1;
    for (int g = warp; m + (g & 1) + 8 * (g >> 1) <= L; g += NT / 32) {
        const int l = m + (g & 1) + 8 * (g >> 1) + 2 * (lane >> 3);
        const bool in = l <= L;
        const double* prow = tg + (long long)(in ? l - m : 0) * N;
        const double2* Xl = X + (g & 1 ? N : 0);
        double v[4] = {0., 0., 0., 0.};
        for (int k = sub; k < P; k += 8) {
            const double d = prow[k];
            const double2 x0 = Xl[k];
            v[0] += d * x0.x;
            v[1] += d * x0.y;
            if (np == 2) {
                const double2 x1 = Xl[P + k];
                v[2] += d * x1.x;
                v[3] += d * x1.y;
            }
        }
        const double y = reduce_scatter(v, sub);
        if (!in || (sub & 1) || wp >= np) continue;
        if (wp == 0) {
            Fd[2 * s2_idx(l, m) + wc] = y;
            if (m > 0 && is_real)  // Hermitian fill, fdcl_FFTS2.cpp:182-188
                Fd[2 * s2_idx(l, -m) + wc] = sg * (wc ? -y : y);
        } else {
            Fd[2 * s2_idx(l, -m) + wc] = sg * y;
        }
    }
}

template <int NT>
__global__ void __launch_bounds__(NT) s2_inv_fp64_kernel(const double* __restrict__ table,
                                                         const long long* __restrict__ moff,
                                                         const double2* __restrict__ F, double2* __restrict__ H,
                                                         int L, int N, long long gstride, long long cstride)
{
    extern __shared__ double2 Y[];  // [2][B]
    const int m = blockIdx.x, b = blockIdx.y;
    const int B = L + 1;
    const int nl = B - m;
    const int np = (m > 0) ? 2 : 1;
    const double sg = (m & 1) ? -1. : 1.;
    const double2* Fb = F + (long long)b * cstride;
    for (int i = threadIdx.x; i < np * nl; i += NT) {
        int p = i / nl, l = m + (i - p * nl);
        double2 c = Fb[s2_idx(l, p == 0 ? m : -m)];
        double s = (p == 0) ? 1. : sg;
        Y[p * B + (l - m)] = make_double2(s * c.x, s * c.y);
    }
    __syncthreads();
    const double* tg = table + moff[m];
    double2* Hb = H + (long long)b * gstride;
    // the Nyquist bin, which no coefficient maps to
    if (m == 0)
        for (int k = threadIdx.x; k < N; k += NT) Hb[(long long)k * N + N / 2] = make_double2(0., 0.);
    // neighbouring threads take the even and the odd degrees of one k; whole warps run for the exchange
    const int odd = threadIdx.x & 1;
    for (int k0 = 0; k0 < N / 2; k0 += NT / 2) {
        const int k = k0 + (threadIdx.x >> 1);
        const bool in = k < N / 2;
        double ar[2] = {0., 0.}, ai[2] = {0., 0.};
        for (int j = in ? odd : nl; j < nl; j += 2) {
            double d = tg[(long long)j * N + k];
            double2 y0 = Y[j];
            ar[0] += d * y0.x;
            ai[0] += d * y0.y;
            if (np == 2) {
                double2 y1 = Y[B + j];
                ar[1] += d * y1.x;
                ai[1] += d * y1.y;
            }
        }
        // even: E + O at k; odd: E - O at N - 1 - k
#pragma unroll
        for (int p = 0; p < 2; ++p) {
            const double r = __shfl_xor_sync(0xffffffffu, ar[p], 1), i = __shfl_xor_sync(0xffffffffu, ai[p], 1);
            ar[p] = odd ? r - ar[p] : ar[p] + r;
            ai[p] = odd ? i - ai[p] : ai[p] + i;
        }
        if (!in) continue;
        const long long row = (long long)(odd ? N - 1 - k : k) * N;
        // f = sum_m H(m) e^{+i m phi}: H(m) goes to bin -m mod N of a forward DFT
        Hb[row + mod_n(-m, N)] = make_double2(ar[0], ai[0]);
        if (np == 2) Hb[row + mod_n(m, N)] = make_double2(ar[1], ai[1]);
    }
}

// degree l of packed S^2 index i = l^2 + l + m (integer fix-up of a float square root)
__device__ __forceinline__ int s2_degree(long long i)
{
    int l = (int)sqrtf((float)i);
    while ((long long)l * l > i) --l;
    while ((long long)(l + 1) * (l + 1) <= i) ++l;
    return l;
}

// F_r(l) = Re(conj(T(l)) F_c(l)) (fdcl_FFTS2.cpp:424-436), arithmetic in A
// (double for the FP64 path, float for the tensor-core path).
template <typename CIN, typename ROUT, typename A>
__global__ void s2_c2r_kernel(const CIN* __restrict__ Fc, ROUT* __restrict__ Fr, int L, long long cstride)
{
    const int b = blockIdx.y;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long C = (long long)(L + 1) * (L + 1);
    if (i >= C) return;
    const int l = s2_degree(i);
    const int m = (int)(i - (long long)l * l) - l;
    const CIN* fc = Fc + (long long)b * cstride;
    int cs[2] = {-m, m};
    if (m > 0) { cs[0] = -m; cs[1] = m; } else if (m < 0) { cs[0] = m; cs[1] = -m; }
    const int nc = (m == 0) ? 1 : 2;
    A acc = 0;
    for (int j = 0; j < nc; ++j) {
        const c2t<A> t = conj_t(tmat_t<A>(m, cs[j]));
        const CIN v = fc[s2_idx(l, cs[j])];
        acc += t.x * (A)v.x - t.y * (A)v.y;
    }
    Fr[(long long)b * cstride + i] = (ROUT)acc;
}

// F_c = T^T F_r: the complex coefficients whose synthesis is the real-basis
// synthesis sum F_r(l,m) y(l,m), y = T Y (fdcl_FFTS2.cpp:383-422).
template <typename RIN, typename COUT, typename A>
__global__ void s2_r2c_kernel(const RIN* __restrict__ Fr, COUT* __restrict__ Fc, int L, long long cstride)
{
    const int b = blockIdx.y;
    long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    const long long C = (long long)(L + 1) * (L + 1);
    if (i >= C) return;
    const int l = s2_degree(i);
    const int c = (int)(i - (long long)l * l) - l;
    const RIN* fr = Fr + (long long)b * cstride;
    const int as[2] = {c, -c};
    const int na = (c == 0) ? 1 : 2;
    c2t<A> acc = {(A)0, (A)0};
    for (int j = 0; j < na; ++j) {
        const c2t<A> t = tmat_t<A>(as[j], c);
        const A v = (A)fr[s2_idx(l, as[j])];
        acc.x += t.x * v;
        acc.y += t.y * v;
    }
    COUT o;
    o.x = acc.x;
    o.y = acc.y;
    Fc[(long long)b * cstride + i] = o;
}

// S^2 real coefficients straight from the tensor-core group-major layout
// (Fg[f][goff2[g] + p (B - g) + (l - g)] = F_c(l, m) for g = |m|, p = (m < 0)):
// the gather to the packed complex layout and s2_c2r_kernel in one pass, with
// the same arithmetic.  A CTA stages a 32 (l) x 32 (m) tile of F_c(l, +-m) in
// shared memory, so the group-major side is read along l and the packed real
// side written along m, both in runs of 32.
constexpr int S2T = 32;

__global__ void __launch_bounds__(256) s2_group_to_real_kernel(const float2* __restrict__ Fg, float* __restrict__ Fr,
                                                              const long long* __restrict__ goff2, int L,
                                                              long long cstride, bool half)
{
    __shared__ float2 tp[S2T][S2T + 1];  // F_c(l0 + li, +(mb + mi)) as [mi][li]
    __shared__ float2 tn[S2T][S2T + 1];  // F_c(l0 + li, -(mb + mi))
    const int B = L + 1;
    const int l0 = blockIdx.x * S2T, mb = (int)blockIdx.y * S2T, b = blockIdx.z;  // |m| tile [mb, mb + 32)
    if (mb > l0 + S2T - 1 || mb > L) return;  // every |m| of the tile exceeds every l
    const float2* fg = Fg + (long long)b * cstride;
    for (int e = threadIdx.x; e < S2T * S2T; e += 256) {
        const int mi = e / S2T, li = e % S2T, g = mb + mi, l = l0 + li;
        if (g > L || l > L || l < g) continue;
        const long long o = goff2[g] + (l - g);
        const float2 v = fg[o];
        tp[mi][li] = v;
        if (half)
            tn[mi][li] = g > 0 ? (g & 1 ? make_float2(-v.x, v.y) : make_float2(v.x, -v.y)) : v;
        else
            tn[mi][li] = g > 0 ? fg[o + (B - g)] : v;
    }
    __syncthreads();
    float* fr = Fr + (long long)b * cstride;
    // outputs (l, m) for |m| in the tile, m = +g and m = -g: runs along m (packed l^2 + l + m)
    for (int e = threadIdx.x; e < 2 * S2T * S2T; e += 256) {
        const int li = e / (2 * S2T), r = e % (2 * S2T), neg = r < S2T, mi = neg ? S2T - 1 - r : r - S2T;
        const int g = mb + mi, l = l0 + li;
        if (g > L || l > L || l < g || (neg && g == 0)) continue;
        const int m = neg ? -g : g;
        int cs[2] = {-m, m};
        if (m > 0) { cs[0] = -m; cs[1] = m; } else if (m < 0) { cs[0] = m; cs[1] = -m; }
        const int nc = (m == 0) ? 1 : 2;
        float acc = 0.f;
        for (int j = 0; j < nc; ++j) {
            const c2t<float> t = conj_t(tmat_t<float>(m, cs[j]));
            const float2 v = cs[j] < 0 ? tn[mi][li] : tp[mi][li];
            acc += t.x * v.x - t.y * v.y;
        }
        fr[(long long)l * l + l + m] = acc;
    }
}

// (half, in both: of the pairs of m > 0 the GEMM writes pair 0 alone, and reads pair 1 alone: the others are their conjugates.)
// S^2 real coefficients straight into the scaled group-major layout of the
// inverse GEMM (pair 0: F_c(l, m), pair 1: (-1)^m F_c(l, -m), m >= 0):
// s2_r2c_kernel and the packed -> group-major permutation in one pass, with
// the same arithmetic.  A CTA stages F_r(l, +-m) for a 32 (l) x 32 (m) tile,
// read along m (packed) and written along l (group-major).
__global__ void __launch_bounds__(256) s2_real_to_group_kernel(const float* __restrict__ Fr, float2* __restrict__ Y,
                                                              const long long* __restrict__ goff2, int L,
                                                              long long cstride, bool half)
{
    __shared__ float tp[S2T][S2T + 1];  // F_r(l0 + li, +(mb + mi)) as [li][mi]
    __shared__ float tn[S2T][S2T + 1];  // F_r(l0 + li, -(mb + mi))
    const int B = L + 1;
    const int l0 = blockIdx.x * S2T, mb = (int)blockIdx.y * S2T, b = blockIdx.z;
    if (mb > l0 + S2T - 1 || mb > L) return;
    const float* fr = Fr + (long long)b * cstride;
    for (int e = threadIdx.x; e < 2 * S2T * S2T; e += 256) {
        const int li = e / (2 * S2T), r = e % (2 * S2T), neg = r < S2T, mi = neg ? S2T - 1 - r : r - S2T;
        const int g = mb + mi, l = l0 + li;
        if (g > L || l > L || l < g) continue;
        const float v = fr[(long long)l * l + l + (neg ? -g : g)];
        if (neg) tn[li][mi] = v; else tp[li][mi] = v;
    }
    __syncthreads();
    float2* y = Y + (long long)b * cstride;
    for (int e = threadIdx.x; e < 2 * S2T * S2T; e += 256) {
        const int p = e / (S2T * S2T), r = e % (S2T * S2T), mi = r / S2T, li = r % S2T;
        const int m = mb + mi, l = l0 + li;
        if (m > L || l > L || l < m || (p == 1 && m == 0) || (half && p == 0 && m > 0)) continue;
        const int c = p == 0 ? m : -m;
        const int as[2] = {c, -c};
        const int na = (c == 0) ? 1 : 2;
        c2t<float> acc = {0.f, 0.f};
        for (int j = 0; j < na; ++j) {
            const c2t<float> t = tmat_t<float>(as[j], c);
            const float v = as[j] < 0 ? tn[li][mi] : tp[li][mi];
            acc.x += t.x * v;
            acc.y += t.y * v;
        }
        const float sc = (p == 0 || !(m & 1)) ? 1.f : -1.f;
        y[goff2[m] + (long long)p * (B - m) + (l - m)] = make_float2(sc * acc.x, sc * acc.y);
    }
}

// ---------------------------------------------------------------- launchers

cudaError_t launch_so3_fwd_fp64(const double* table, const long long* goff, const double2* G, const double* w,
                                double2* F, int L, int N, int batch, bool real, cudaStream_t st)
{
    const int B = L + 1;
    size_t smem = sizeof(double2) * (real ? 2 : 4) * N;
    auto k = real ? so3_fwd_fp64_kernel<256, true> : so3_fwd_fp64_kernel<256, false>;
    cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    dim3 grid(B * B, batch);
    k<<<grid, 256, smem, st>>>(table, goff, G, w, F, L, N, (long long)N * N * N, so3_off(B));
    return cudaGetLastError();
}

cudaError_t launch_so3_inv_fp64(const double* table, const long long* goff, const double2* F, double2* H, int L,
                                int N, int batch, bool real, cudaStream_t st)
{
    const int B = L + 1;
    size_t smem = sizeof(double2) * (real ? 2 : 4) * B;
    dim3 grid(B * B, batch);
    auto k = real ? so3_inv_fp64_kernel<256, true> : so3_inv_fp64_kernel<256, false>;
    k<<<grid, 256, smem, st>>>(table, goff, F, H, L, N, (long long)N * N * N, so3_off(B));
    return cudaGetLastError();
}

cudaError_t launch_zero_nyquist_so3(void* H, bool fp64, int N, long long nslices, cudaStream_t st)
{
    long long tot = nslices * 2 * N;
    unsigned nb = (unsigned)((tot + 255) / 256);
    if (fp64)
        zero_nyquist_so3_kernel<double2><<<nb, 256, 0, st>>>((double2*)H, N, nslices);
    else
        zero_nyquist_so3_kernel<float2><<<nb, 256, 0, st>>>((float2*)H, N, nslices);
    return cudaGetLastError();
}

cudaError_t launch_so3_c2r(const void* Fc, void* Fr, bool fp64, int L, int batch, cudaStream_t st)
{
    const long long C = so3_off(L + 1);
    const int nq = (L + 1) * (L + 2) * (2 * L + 3) / 6;
    const dim3 grid((unsigned)((nq + 127) / 128), batch);
    if (fp64)
        so3_c2r_kernel<double2, double, double, true><<<grid, 128, 0, st>>>((const double2*)Fc, (double*)Fr, nq, C);
    else
        so3_c2r_kernel<float2, float, float, false><<<grid, 128, 0, st>>>((const float2*)Fc, (float*)Fr, nq, C);
    return cudaGetLastError();
}

cudaError_t launch_so3_r2c(const void* Fr, void* Fc, bool fp64, int L, int batch, cudaStream_t st)
{
    const long long C = so3_off(L + 1);
    const int nq = (L + 1) * (L + 2) * (2 * L + 3) / 6;
    const dim3 grid((unsigned)((nq + 127) / 128), batch);
    if (fp64)
        so3_r2c_kernel<double, double2, double><<<grid, 128, 0, st>>>((const double*)Fr, (double2*)Fc, nq, C);
    else
        so3_r2c_kernel<float, float2, float><<<grid, 128, 0, st>>>((const float*)Fr, (float2*)Fc, nq, C);
    return cudaGetLastError();
}

cudaError_t launch_s2_fwd_fp64(const double* table, const long long* moff, const double2* G, const double* w,
                               double2* F, int L, int N, int batch, bool is_real, cudaStream_t st)
{
    size_t smem = sizeof(double2) * 2 * N;
    dim3 grid(L + 1, batch);
    s2_fwd_fp64_kernel<256><<<grid, 256, smem, st>>>(table, moff, G, w, F, L, N, (long long)N * N,
                                                     (long long)(L + 1) * (L + 1), is_real ? 1 : 0);
    return cudaGetLastError();
}

cudaError_t launch_s2_inv_fp64(const double* table, const long long* moff, const double2* F, double2* H, int L,
                               int N, int batch, cudaStream_t st)
{
    size_t smem = sizeof(double2) * 2 * (L + 1);
    dim3 grid(L + 1, batch);
    s2_inv_fp64_kernel<256><<<grid, 256, smem, st>>>(table, moff, F, H, L, N, (long long)N * N,
                                                     (long long)(L + 1) * (L + 1));
    return cudaGetLastError();
}

cudaError_t launch_s2_c2r(const void* Fc, void* Fr, bool fp64, int L, int batch, cudaStream_t st)
{
    long long C = (long long)(L + 1) * (L + 1);
    dim3 grid((unsigned)((C + 255) / 256), batch);
    if (fp64)
        s2_c2r_kernel<double2, double, double><<<grid, 256, 0, st>>>((const double2*)Fc, (double*)Fr, L, C);
    else
        s2_c2r_kernel<float2, float, float><<<grid, 256, 0, st>>>((const float2*)Fc, (float*)Fr, L, C);
    return cudaGetLastError();
}

cudaError_t launch_s2_group_to_real(const void* Fg, void* Fr, const long long* goff2, int L, int batch, bool half,
                                   cudaStream_t st)
{
    const long long C = (long long)(L + 1) * (L + 1);
    const unsigned nt = (unsigned)((L + 1 + S2T - 1) / S2T);
    s2_group_to_real_kernel<<<dim3(nt, nt, batch), 256, 0, st>>>((const float2*)Fg, (float*)Fr, goff2, L, C, half);
    return cudaGetLastError();
}

cudaError_t launch_s2_real_to_group(const void* Fr, void* Y, const long long* goff2, int L, int batch, bool half,
                                   cudaStream_t st)
{
    const long long C = (long long)(L + 1) * (L + 1);
    const unsigned nt = (unsigned)((L + 1 + S2T - 1) / S2T);
    s2_real_to_group_kernel<<<dim3(nt, nt, batch), 256, 0, st>>>((const float*)Fr, (float2*)Y, goff2, L, C, half);
    return cudaGetLastError();
}

cudaError_t launch_s2_r2c(const void* Fr, void* Fc, bool fp64, int L, int batch, cudaStream_t st)
{
    long long C = (long long)(L + 1) * (L + 1);
    dim3 grid((unsigned)((C + 255) / 256), batch);
    if (fp64)
        s2_r2c_kernel<double, double2, double><<<grid, 256, 0, st>>>((const double*)Fr, (double2*)Fc, L, C);
    else
        s2_r2c_kernel<float, float2, float><<<grid, 256, 0, st>>>((const float*)Fr, (float2*)Fc, L, C);
    return cudaGetLastError();
}

// ---- residual refinement of the FP32-data plans (F += forward(f - inverse(F)), the inverse in FP64)

__global__ void widen_kernel(const float* __restrict__ in, double* __restrict__ out, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (double)in[i];
}

// r = f - g with f the FP32 samples the forward transformed and g the FP64
// synthesis of its first result: the subtraction is done in FP64 (f is exact
// there), only the small difference is rounded to FP32.  f may be r itself.
__global__ void resid_fp64_kernel(const float* f, const double* __restrict__ g, float* r, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) r[i] = (float)((double)f[i] - g[i]);
}

__global__ void add_real_kernel(float* __restrict__ F, const float* __restrict__ d, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) F[i] += d[i];
}

cudaError_t launch_widen(const float* in, double* out, long long n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    widen_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}

__global__ void narrow_kernel(const double* __restrict__ in, float* __restrict__ out, long long n)
{
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) out[i] = (float)in[i];
}

cudaError_t launch_narrow(const double* in, float* out, long long n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    narrow_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(in, out, n);
    return cudaGetLastError();
}

cudaError_t launch_resid_fp64(const float* f, const double* g, float* r, long long n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    resid_fp64_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(f, g, r, n);
    return cudaGetLastError();
}

cudaError_t launch_add_real(float* F, const float* d, long long n, cudaStream_t st)
{
    if (n <= 0) return cudaSuccess;
    add_real_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(F, d, n);
    return cudaGetLastError();
}

}  // namespace fftso3
