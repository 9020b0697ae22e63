// Latitudinal (Legendre / spin-weighted Wigner-d) stage, SIMT kernels for sm_100a.
//
// For each order m the rows lambda^{s'}_lm(theta) = sqrt((2l+1)/4pi) d^l_{m,s'}(theta)
// are generated on the fly in double precision with an explicit binary exponent per lane
// (values below 2^-300 are carried exactly and emitted as zero), and contracted against the
// ring spectra.  With r_l = 1 / alpha_l the normalised three-term recurrence
//     v_{l+1} = alpha_{l+1} (x - c_{l+1}) v_l - (alpha_{l+1} / alpha_l) v_{l-1}
// is carried through the differences v_l - v_{l-1} = alpha_l d_l:
//     d_{l+1} = d_l + ((x - 1) + e_{l+1}) v_l,   e_l = 1 - r_{l-1} - r_l - c_l,
//     v_{l+1} = v_l + alpha_{l+1} d_{l+1},
// three operations with two coefficients per row (legendre_rows.cu has the same form in single
// precision).  Only northern lanes are marched: the hemisphere fold
//   lambda^{s'}_lm(pi - theta) = (-1)^{l+m} lambda^{-s'}_lm(theta)
// turns the two hemispheres into the Sum / Diff right-hand sides of `rhs`.
//
// The contraction is carried in T (double for GM_FP64, float for GM_MIXED); the
// recurrence is always double.  These kernels are the plain-FP64 path, and the mixed path of
// a few maps where no checkpoint tables exist (spins other than 0 and 2, Nside above 2048;
// with tables: legendre_rows.cu); the tensor-core path (legendre_ck.cu, legendre_tc.cu) takes
// wide batches.
//
// A CTA is up to four warps of one order; the rows go in segments of up to 128 whose
// coefficients its threads compute once, then in blocks of eight without barriers: a warp whose
// lanes are all below 2^-300 only steps.  Spin s takes the sum F and the difference G of the two
// variants' rows, formed in double precision, against Q and U (four values a row, E and B: at m = 0,
// where G = 0, E takes Q alone and B takes U alone).  Small sizes are bound by the chain of rows
// (m = 0) and the reduction trees, large ones by the FP64 pipe: (3 + 2 NC) operations per row and
// lane (spin 0), 16 (spin s).  Against windows of 32 rows with coefficients by square roots and
// divisions in each, and eight sums a row: FP64 analysis / synthesis at Nside 128 58 / 44 -> 33 / 23
// us, at Nside 1024 10.0 / 8.1 -> 5.2 / 4.0 ms (spin 0) and 26.8 / 21.5 -> 13.3 / 10.9 ms (spin 2);
// mixed spin 1 at Nside 1024 20.1 / 18.3 -> 10.9 / 9.7 ms.
//
// Replaces gmaster/_native/cuda/march_v2.cu:155-407 (march_analysis /
// march_synthesis: float32 difference-form recurrence, SIMT FMA contraction).
#include <math.h>

#include "gm_common.cuh"

namespace gm {

constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
// Spins 1..kMaxSpin share the polarised kernels (template SPIN = 2) with the spin passed at
// run time; the seed table holds 2 kMaxSpin + 1 variants.
constexpr int kMaxSpin = 8;

// First seed-table variant of spin s >= 1 (s' = -s; the next one is s' = +s): spin 2 keeps
// variants 1 and 2 (the tensor-core kernels read them), spin 1 takes 3 and 4, spin s >= 3
// takes 2s - 1 and 2s.
__host__ __device__ __forceinline__ int seed_variant(int s)
{
    return s == 2 ? 1 : (s == 1 ? 3 : 2 * s - 1);
}
constexpr double kBig = 2.037035976334486e90;     // 2^300
constexpr double kShrink = 2.409919865102884e-181;  // 2^-600

// Seed of one lane: value = sign * 2^f carried as v * 2^(600 k), k <= 0.
__device__ __forceinline__ void seed_lane(const double *__restrict__ sd, double lsin, double lcos,
                                          double &v, int &k)
{
    double f = sd[0];
    if (sd[2] != 0.0) f += sd[2] * lcos;
    if (sd[3] != 0.0) f += sd[3] * lsin;
    if (!(f > -1.0e300)) {
        v = 0.0;
        k = 0;
        return;
    }
    int kk = 0;
    if (f < -300.0) kk = (int)floor((f + 300.0) / 600.0);
    v = sd[1] * exp2(f - 600.0 * (double)kk);
    k = kk;
}

// Coefficients of the step from row l to row l + 1 (see the head of the file): e of s' = -s, e of
// s' = +s, alpha_{l+1}.
struct Coef {
    double ea, eb, alpha;
};

// r_l = 1 / alpha_l, zero at l = max(m, s), and h = 1/2 - r_l without its cancellation, from
//   1/4 - r_l^2 = (l^2 (4 m^2 + 4 s^2 - 1) - 4 m^2 s^2) / (4 l^2 (4 l^2 - 1)).
__device__ __forceinline__ double inv_alpha(int l, int m, int s, double &h)
{
    const double l2 = (double)l * l, m2 = (double)m * m, s2 = (double)s * s, q = 4.0 * l2 - 1.0;
    double r, num, den;
    if (s == 0) {
        r = sqrt((l2 - m2) / q);
        num = 4.0 * m2 - 1.0;
        den = 4.0 * q;
    } else {
        r = sqrt((l2 - m2) * (l2 - s2) / q) / (double)l;
        num = fma(l2, 4.0 * (m2 + s2) - 1.0, -4.0 * m2 * s2);
        den = 4.0 * l2 * q;
    }
    h = num / (den * (0.5 + r));
    return r;
}

__device__ __forceinline__ Coef step_coef(int l, int m, int s)
{
    double h0, h1;
    inv_alpha(l, m, s, h0);
    const double r1 = inv_alpha(l + 1, m, s, h1);
    const double e = h0 + h1;
    const double c = s != 0 ? (double)s * m / ((double)l * (l + 1)) : 0.0;
    return Coef{e + c, e - c, 1.0 / r1};
}

// Sum of each of the V values of all 32 threads: thread t returns value t % V.  The last LD of the
// five levels add in double precision.
template <int LD, typename T, int V>
__device__ __forceinline__ double warp_reduce_scatter(T (&v)[V], int lane)
{
    double w[V];
#pragma unroll
    for (int h = V / 2, level = 5; h >= 1; h >>= 1, --level) {
        const bool upper = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            if (level > LD) {
                const T send = upper ? v[i] : v[i + h], keep = upper ? v[i + h] : v[i];
                v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
                w[i] = (double)v[i];
            } else {
                const double send = upper ? w[i] : w[i + h], keep = upper ? w[i + h] : w[i];
                w[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
            }
        }
    }
#pragma unroll
    for (int h = V, level = V == 16 ? 1 : 0; h < 32; h <<= 1, --level) {
        if (level > LD) {
            v[0] += __shfl_xor_sync(0xffffffffu, v[0], h);
            w[0] = (double)v[0];
        } else {
            w[0] += __shfl_xor_sync(0xffffffffu, w[0], h);
        }
    }
    return w[0];
}

__device__ __forceinline__ int64_t alm_index(int64_t lmax, int64_t l, int64_t m)
{
    return m * (2 * lmax + 1 - m) / 2 + l;
}

// x - 1 of lane j, rounded once (HEALPix rings): cos(theta) less one would keep the rounding of
// cos(theta), relative to x - 1 a large error near the poles, and add another for x < 1/2.  With it
// and the e of inv_alpha below, the error of a pass at Nside 128, lmax 300, against sums in 80 bits
// is 1.1e-14 (spin 0) and 1.3e-14 (spin 2); from cos(theta) - 1 and 1 - r_{l-1} - r_l it was
// 7.8e-14 to 1.1e-13.
__device__ __forceinline__ double lane_xm1(int64_t nside, int64_t j)
{
    const double i = (double)(j + 1), n = (double)nside;
    return i < n ? -(i * i) / (3.0 * n * n) : (n - 2.0 * i) / (3.0 * n);
}

// The rows of a thread's R lanes, NVAR variants each: value v 2^(600 k), scaled difference d.
template <int NVAR, int R> struct RowState {
    double y[R], v[NVAR][R], d[NVAR][R];
    int k[NVAR][R];

    // Seeds at row l0.
    __device__ __forceinline__ void start(const double *__restrict__ geom, const double *__restrict__ seeds,
                                          int64_t nlanes, int64_t L, int64_t jw, int lane, int m, int var, bool any)
    {
#pragma unroll
        for (int r = 0; r < R; ++r) {
            const int64_t j = jw + r * 32 + lane;
            const bool ok = any && j < nlanes;
            y[r] = ok ? lane_xm1(nlanes / 2, j) : 0.0;
            const double ls = ok ? geom[nlanes + j] : 0.0, lc = ok ? geom[2 * nlanes + j] : 0.0;
#pragma unroll
            for (int q = 0; q < NVAR; ++q) {
                v[q][r] = d[q][r] = 0.0;
                k[q][r] = 0;
                if (ok) seed_lane(seeds + ((int64_t)(var + q) * L + m) * 4, ls, lc, v[q][r], k[q][r]);
            }
        }
    }

    __device__ __forceinline__ void step(const Coef &c, int r)
    {
#pragma unroll
        for (int q = 0; q < NVAR; ++q) {
            const double C = y[r] + (q == 0 ? c.ea : c.eb);
            d[q][r] = fma(C, v[q][r], d[q][r]);
            v[q][r] = fma(c.alpha, d[q][r], v[q][r]);
        }
    }

    // Lanes below 2^-300 that grew past it: once per eight rows (a row grows a value by at most
    // 2^8, alpha <= sqrt(2m) + 1).
    __device__ __forceinline__ void rescale()
    {
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < NVAR; ++q)
                if (k[q][r] < 0 && fabs(v[q][r]) > kBig) {
                    v[q][r] *= kShrink;
                    d[q][r] *= kShrink;
                    ++k[q][r];
                }
    }

    // 0: every lane of the warp emits its rows, 1: some do, 2: none does (all below 2^-300).
    __device__ __forceinline__ int emission() const
    {
        bool all = true, none = true;
#pragma unroll
        for (int r = 0; r < R; ++r)
#pragma unroll
            for (int q = 0; q < NVAR; ++q) {
                all = all && k[q][r] == 0;
                none = none && (k[q][r] < 0 || (v[q][r] == 0.0 && d[q][r] == 0.0));
            }
        if (__all_sync(0xffffffffu, all)) return 0;
        return __all_sync(0xffffffffu, none) ? 2 : 1;
    }
};

// ---------------------------------------------------------------- analysis

// NC components per CTA (spin 0: NC maps; spin s: NC = 2, one (Q, U) pair), NV sums per degree.
template <int SPIN, int NC> struct Shape {
    static constexpr int NVAR = SPIN == 0 ? 1 : 2;
    static constexpr int NV = SPIN == 0 ? 2 * NC : 4;
    static constexpr int kRows = 512 / NV < 128 ? 512 / NV : 128;   // rows per staged segment
};

// Eight rows of one warp into red[8 NV].  rh: spin 0, per map Sum re, im, Diff re, im; spin s,
// Q Sum, Q Diff, U Sum, U Diff (re, im).
template <typename T, int SPIN, int NC, int R, bool PART>
__device__ __forceinline__ void ana8(RowState<Shape<SPIN, NC>::NVAR, R> &w, const T (&rh)[R][4 * NC],
                                     const Coef *__restrict__ cf, double *__restrict__ red, int lane)
{
    constexpr int NV = Shape<SPIN, NC>::NV, NVAR = Shape<SPIN, NC>::NVAR;
    // values per reduction tree: 32 where the registers allow (half the trees, of one more level)
    constexpr int V = (NV * 8 >= 32 && R <= 2) || NV == 16 ? 32 : 16;
    constexpr int RB = V / NV;
    // Spin s adds the F and the G terms in one chain of 2 R products; the last levels of the tree in
    // double precision take off as much rounding as that adds over two chains and trees of R
    // products each (in units of a product's: 3, 10, 36, 136 and 5 x 2 R less 2 R a level against 2,
    // 6, 20, 72 and 5 x 2 R).
    constexpr int LD = SPIN == 0 || sizeof(T) == 8 ? 0 : (R <= 2 ? 1 : (R == 4 ? 2 : 4));
    static_assert(V == 16 || V == 32, "levels of the tree");
    static_assert(RB % 2 == 0 && 8 % RB == 0, "row parity is fixed by the row index");
#pragma unroll 1
    for (int i = 0; i < 8; i += RB) {
        T acc[V];
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] = (T)0;
#pragma unroll
        for (int s = 0; s < RB; ++s) {
            const Coef c = cf[i + s];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                double lam[NVAR];
#pragma unroll
                for (int q = 0; q < NVAR; ++q) lam[q] = !PART || w.k[q][r] == 0 ? w.v[q][r] : 0.0;
                if (SPIN == 0) {
                    const T val = (T)lam[0];
#pragma unroll
                    for (int e = 0; e < NC; ++e) {
                        acc[s * NV + 2 * e] += val * rh[r][4 * e + 2 * (s & 1)];
                        acc[s * NV + 2 * e + 1] += val * rh[r][4 * e + 2 * (s & 1) + 1];
                    }
                } else {
                    // E += F Q_p + i G U_d, B += F U_p - i G Q_d
                    const T f = (T)(lam[0] + lam[NVAR - 1]), g = (T)(lam[0] - lam[NVAR - 1]);
                    const T *qp = rh[r] + 2 * (s & 1), *qd = rh[r] + 2 - 2 * (s & 1), *up = qp + 4, *ud = qd + 4;
                    T *a = acc + s * NV;
                    a[0] += f * qp[0];
                    a[0] -= g * ud[1];
                    a[1] += f * qp[1];
                    a[1] += g * ud[0];
                    a[2] += f * up[0];
                    a[2] += g * qd[1];
                    a[3] += f * up[1];
                    a[3] -= g * qd[0];
                }
                w.step(c, r);
            }
        }
        const double tot = warp_reduce_scatter<LD>(acc, lane);
        if (lane < V) red[i * NV + lane] = tot;
    }
    w.rescale();
}

template <typename T, int SPIN, int NC, int R>
__global__ void __launch_bounds__(kThreads) k_legendre_ana(
    int64_t nside, int64_t lmax, int64_t ncomp, const double *__restrict__ geom,
    const double *__restrict__ seeds, const T *__restrict__ rhs, double *__restrict__ alm,
    double scale, int spin)
{
    using S = Shape<SPIN, NC>;
    constexpr int NV = S::NV, NVAR = S::NVAR, kRows = S::kRows;
    __shared__ Coef cf[kRows];
    __shared__ double red[kWarps][kRows * NV];
    const int64_t L = lmax + 1, nlanes = 2 * nside, nelem = L * (L + 1) / 2;
    const int m = blockIdx.y;
    const int64_t c0 = (int64_t)blockIdx.z * NC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int sv = SPIN == 0 ? 0 : spin;   // the field's spin (SPIN = 2: any spin >= 1)
    const int l0 = m > sv ? m : sv;
    if (l0 > lmax) return;
    const int64_t jw = ((int64_t)blockIdx.x * nw + warp) * 32 * R;

    RowState<NVAR, R> w;
    w.start(geom, seeds, nlanes, L, jw, lane, m, SPIN == 0 ? 0 : seed_variant(sv), true);
    T rh[R][4 * NC];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t j = jw + r * 32 + lane;
        T g[NC][4];
#pragma unroll
        for (int c = 0; c < NC; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                g[c][e] = j < nlanes && c0 + c < ncomp ? rhs[(((int64_t)m * nlanes + j) * ncomp + c0 + c) * 4 + e] : (T)0;
        if (SPIN == 0) {
            // l + m of a segment's even rows is even: row s takes half s & 1
#pragma unroll
            for (int q = 0; q < 4 * NC; ++q) rh[r][q] = g[q / 4][q % 4];
        } else {
            // the southern rows are the northern ones of the other variant times (-1)^(l + m + s):
            // where a segment's even rows have it odd, Sum and Diff change places
            const int p = (l0 + m + sv) & 1;
#pragma unroll
            for (int q = 0; q < 8; ++q) rh[r][q] = p ? g[q / 4][(q + 2) % 4] : g[q / 4][q % 4];
        }
    }

    for (int64_t lb = l0; lb < L; lb += kRows) {
        const int nrow = (int)(L - lb < kRows ? L - lb : kRows);
        __syncthreads();   // the previous segment's sums are read
        for (int i = threadIdx.x; i < kRows; i += blockDim.x)
            cf[i] = i < nrow ? step_coef((int)lb + i, m, sv) : Coef{0.0, 0.0, 0.0};
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < nrow; i += 8) {
            double *out = red[warp] + i * NV;
            const int mode = w.emission();
            if (mode == 0) {
                ana8<T, SPIN, NC, R, false>(w, rh, cf + i, out, lane);
            } else if (mode == 1) {
                ana8<T, SPIN, NC, R, true>(w, rh, cf + i, out, lane);
            } else {
                for (int q = lane; q < 8 * NV; q += 32) out[q] = 0.0;
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const Coef c = cf[i + s];
#pragma unroll
                    for (int r = 0; r < R; ++r) w.step(c, r);
                }
                w.rescale();
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nrow; i += blockDim.x) {
            double sum[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) {
                double t = 0.0;
                for (int g = 0; g < nw; ++g) t += red[g][i * NV + q];
                sum[q] = t;
            }
            const int64_t idx = alm_index(lmax, lb + i, m);
            if (SPIN == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (c0 + c < ncomp) {
                        double *a = alm + 2 * ((c0 + c) * nelem + idx);
                        atomicAdd(a, scale * sum[2 * c]);
                        atomicAdd(a + 1, scale * sum[2 * c + 1]);
                    }
                }
            } else {
                double *e = alm + 2 * (c0 * nelem + idx), *b = e + 2 * nelem;
                const double hs = -0.5 * scale;
                atomicAdd(e, hs * sum[0]);
                atomicAdd(e + 1, hs * sum[1]);
                atomicAdd(b, hs * sum[2]);
                atomicAdd(b + 1, hs * sum[3]);
            }
        }
    }
}

// ---------------------------------------------------------------- synthesis

// Eight rows of one warp added to the accumulators.  aw[row][.]: spin 0, (re, im) per map; spin s,
// E and B (re, im).  acc: spin 0, per map the even and odd rows (re, im); spin s, Q Sum, Q Diff,
// U Sum, U Diff (re, im): F of an even row and G of an odd one go to the hemispheres' sum.
template <typename T, int SPIN, int NC, int R, bool PART>
__device__ __forceinline__ void syn8(RowState<Shape<SPIN, NC>::NVAR, R> &w, T (&acc)[R][4 * NC],
                                     const Coef *__restrict__ cf, const T *__restrict__ aw)
{
    constexpr int NVAR = Shape<SPIN, NC>::NVAR, NA = SPIN == 0 ? NC : 2;
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        const Coef c = cf[s];
        T a[2 * NA];
#pragma unroll
        for (int q = 0; q < 2 * NA; ++q) a[q] = aw[s * 2 * NA + q];
#pragma unroll
        for (int r = 0; r < R; ++r) {
            double lam[NVAR];
#pragma unroll
            for (int q = 0; q < NVAR; ++q) lam[q] = !PART || w.k[q][r] == 0 ? w.v[q][r] : 0.0;
            T *o = acc[r];
            if (SPIN == 0) {
                const T val = (T)lam[0];
#pragma unroll
                for (int e = 0; e < NC; ++e) {
                    o[4 * e + 2 * (s & 1)] += val * a[2 * e];
                    o[4 * e + 2 * (s & 1) + 1] += val * a[2 * e + 1];
                }
            } else {
                // -2 Q = F E + i G B, -2 U = F B - i G E
                const T f = (T)(lam[0] + lam[NVAR - 1]), g = (T)(lam[0] - lam[NVAR - 1]);
                T *qp = o + 2 * (s & 1), *qd = o + 2 - 2 * (s & 1), *up = qp + 4, *ud = qd + 4;
                qp[0] += f * a[0];
                qp[1] += f * a[1];
                up[0] += f * a[2];
                up[1] += f * a[3];
                qd[0] -= g * a[3];
                qd[1] += g * a[2];
                ud[0] += g * a[1];
                ud[1] -= g * a[0];
            }
            w.step(c, r);
        }
    }
    w.rescale();
}

template <typename T, int SPIN, int NC, int R>
__global__ void __launch_bounds__(kThreads) k_legendre_syn(
    int64_t nside, int64_t lmax, int64_t ncomp, const double *__restrict__ geom,
    const double *__restrict__ seeds, const double *__restrict__ alm, T *__restrict__ syn,
    int spin)
{
    using S = Shape<SPIN, NC>;
    constexpr int NVAR = S::NVAR, kRows = 128;
    constexpr int NA = SPIN == 0 ? NC : 2;  // complex alm rows per degree (maps, or E and B)
    // Spin s in single precision: the sums of the rows done, kept apart from the running one of 32
    // rows (even rows' F and odd rows' G terms share an accumulator: one over all rows would add
    // twice as many terms as sums of F and G apart).  Spin 1, Nside 512: relative error of a pass
    // 1.5e-7; one accumulator over all rows 5.7e-7, F and G apart 4.1e-7.
    constexpr bool kTwoLevel = SPIN != 0 && sizeof(T) == 4;
    __shared__ Coef cf[kRows];
    __shared__ T aw[kRows * 2 * NA];
    __shared__ T done[kTwoLevel ? R * 4 * NC : 1][kTwoLevel ? kThreads : 1];
    const int64_t L = lmax + 1, nlanes = 2 * nside, nelem = L * (L + 1) / 2;
    const int m = blockIdx.y;
    const int64_t c0 = (int64_t)blockIdx.z * NC;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int sv = SPIN == 0 ? 0 : spin;
    const int l0 = m > sv ? m : sv;
    const int64_t jw = ((int64_t)blockIdx.x * nw + warp) * 32 * R;

    RowState<NVAR, R> w;
    w.start(geom, seeds, nlanes, L, jw, lane, m, SPIN == 0 ? 0 : seed_variant(sv), l0 <= lmax);
    T acc[R][4 * NC];
#pragma unroll
    for (int r = 0; r < R; ++r)
#pragma unroll
        for (int q = 0; q < 4 * NC; ++q) {
            acc[r][q] = (T)0;
            if (kTwoLevel) done[r * 4 * NC + q][threadIdx.x] = (T)0;
        }

    for (int64_t lb = l0; lb < L; lb += kRows) {
        const int nrow = (int)(L - lb < kRows ? L - lb : kRows);
        __syncthreads();   // the previous segment's rows are done with
        for (int i = threadIdx.x; i < kRows; i += blockDim.x) {
            const bool in = i < nrow;
            cf[i] = in ? step_coef((int)lb + i, m, sv) : Coef{0.0, 0.0, 0.0};
            const double *src = alm + 2 * (c0 * nelem + (in ? alm_index(lmax, lb + i, m) : 0));   // 8-byte aligned
            T *o = aw + i * 2 * NA;
            if (SPIN == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const bool have = in && c0 + c < ncomp;
                    o[2 * c] = have ? (T)src[2 * c * nelem] : (T)0;
                    o[2 * c + 1] = have ? (T)src[2 * c * nelem + 1] : (T)0;
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) o[q] = in ? (T)src[2 * (q / 2) * nelem + q % 2] : (T)0;
            }
        }
        __syncthreads();
#pragma unroll 1
        for (int i = 0; i < nrow; i += 8) {
            const int mode = w.emission();
            if (mode == 0) {
                syn8<T, SPIN, NC, R, false>(w, acc, cf + i, aw + i * 2 * NA);
            } else if (mode == 1) {
                syn8<T, SPIN, NC, R, true>(w, acc, cf + i, aw + i * 2 * NA);
            } else {
#pragma unroll
                for (int s = 0; s < 8; ++s) {
                    const Coef c = cf[i + s];
#pragma unroll
                    for (int r = 0; r < R; ++r) w.step(c, r);
                }
                w.rescale();
            }
            if (kTwoLevel && ((i & 24) == 24 || i + 8 >= nrow)) {
#pragma unroll
                for (int q = 0; q < R * 4 * NC; ++q) {
                    T &d = done[q][threadIdx.x];
                    d += acc[q / (4 * NC)][q % (4 * NC)];
                    acc[q / (4 * NC)][q % (4 * NC)] = (T)0;
                }
            }
        }
    }
    if (kTwoLevel) {
#pragma unroll
        for (int q = 0; q < R * 4 * NC; ++q) acc[q / (4 * NC)][q % (4 * NC)] = done[q][threadIdx.x];
    }

    // Sum and Diff change places where even rows have odd l + m + s
    const T h = (T)-0.5, hs = (l0 + m + sv) & 1 ? (T)0.5 : (T)-0.5;
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int64_t j = jw + r * 32 + lane;
        if (j >= nlanes) continue;
        const T *a = acc[r];
        if (SPIN == 0) {
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (c0 + c >= ncomp) continue;
                T *o = syn + (((int64_t)m * nlanes + j) * ncomp + c0 + c) * 4;
                o[0] = a[4 * c] + a[4 * c + 2];
                o[1] = a[4 * c + 1] + a[4 * c + 3];
                o[2] = a[4 * c] - a[4 * c + 2];
                o[3] = a[4 * c + 1] - a[4 * c + 3];
            }
        } else {
            T *o = syn + (((int64_t)m * nlanes + j) * ncomp + c0) * 4;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const T *q = a + 4 * c;   // north = Sum + Diff, south = Sum - Diff
                o[4 * c] = h * (q[0] + q[2]);
                o[4 * c + 1] = h * (q[1] + q[3]);
                o[4 * c + 2] = hs * (q[0] - q[2]);
                o[4 * c + 3] = hs * (q[1] - q[3]);
            }
        }
    }
}

}  // namespace gm

using namespace gm;

extern "C" int64_t gm_seed_table_len(int64_t L) { return (2 * kMaxSpin + 1) * 4 * L; }

// Warps of a CTA: as many as the lanes fill, up to kWarps.
static int cta_warps(int64_t nlanes, int R)
{
    const int64_t need = (nlanes + 32 * R - 1) / (32 * R);
    return (int)(need < kWarps ? need : kWarps);
}

template <typename T, int SPIN, int NC, int R>
static int launch_ana(int spin, int64_t nside, int64_t lmax, int64_t ncomp, const double *geom,
                      const double *seeds, const void *rhs, double *alm, double scale,
                      cudaStream_t s)
{
    const int64_t nlanes = 2 * nside;
    const int nw = cta_warps(nlanes, R), per = 32 * R * nw;
    dim3 grid((unsigned)((nlanes + per - 1) / per), (unsigned)(lmax + 1), (unsigned)((ncomp + NC - 1) / NC));
    k_legendre_ana<T, SPIN, NC, R><<<grid, 32 * nw, 0, s>>>(nside, lmax, ncomp, geom, seeds, (const T *)rhs,
                                                             alm, scale, spin);
    return check_launch("gm_legendre_analysis");
}

template <typename T, int SPIN, int NC, int R>
static int launch_syn(int spin, int64_t nside, int64_t lmax, int64_t ncomp, const double *geom,
                      const double *seeds, const double *alm, void *syn, cudaStream_t s)
{
    const int64_t nlanes = 2 * nside;
    const int nw = cta_warps(nlanes, R), per = 32 * R * nw;
    dim3 grid((unsigned)((nlanes + per - 1) / per), (unsigned)(lmax + 1), (unsigned)((ncomp + NC - 1) / NC));
    k_legendre_syn<T, SPIN, NC, R><<<grid, 32 * nw, 0, s>>>(nside, lmax, ncomp, geom, seeds, alm, (T *)syn,
                                                             spin);
    return check_launch("gm_legendre_synthesis");
}

template <typename T>
static int dispatch_ana(int spin, int64_t nside, int64_t lmax, int64_t ncomp, const double *geom,
                        const double *seeds, const void *rhs, double *alm, double scale,
                        cudaStream_t s)
{
    if (spin == 0) {
        if (ncomp == 1)
            return launch_ana<T, 0, 1, 4>(spin, nside, lmax, ncomp, geom, seeds, rhs, alm, scale, s);
        if (ncomp == 2)
            return launch_ana<T, 0, 2, 4>(spin, nside, lmax, ncomp, geom, seeds, rhs, alm, scale, s);
        return launch_ana<T, 0, 4, 2>(spin, nside, lmax, ncomp, geom, seeds, rhs, alm, scale, s);
    }
    return launch_ana<T, 2, 2, 2>(spin, nside, lmax, ncomp, geom, seeds, rhs, alm, scale, s);
}

template <typename T>
static int dispatch_syn(int spin, int64_t nside, int64_t lmax, int64_t ncomp, const double *geom,
                        const double *seeds, const double *alm, void *syn, cudaStream_t s)
{
    if (spin == 0) {
        if (ncomp == 1) return launch_syn<T, 0, 1, 2>(spin, nside, lmax, ncomp, geom, seeds, alm, syn, s);
        if (ncomp == 2) return launch_syn<T, 0, 2, 2>(spin, nside, lmax, ncomp, geom, seeds, alm, syn, s);
        return launch_syn<T, 0, 4, 1>(spin, nside, lmax, ncomp, geom, seeds, alm, syn, s);
    }
    return launch_syn<T, 2, 2, 2>(spin, nside, lmax, ncomp, geom, seeds, alm, syn, s);
}

// Tile shapes the autotuner chooses from: (NC, R) = (components per CTA, lanes per thread).
// Spin 0 takes NC in {1, 2, 4, 8} (the reduce-scatter needs 2 NC to divide 32); spin 2
// handles one (Q, U) pair per CTA (NC = 2).  Index -1 selects the built-in heuristic.
// The last tile of each list (8 lanes per thread: a reduce-scatter tree per 8 rows shared by
// 64 elements of a thread instead of 32) is compiled for single precision only; the FP64
// kernels run it as the tile with 4 lanes per thread.  The checkpointed single-precision
// passes (legendre_rows.cu) read R as the pairs of lanes (spin 0) or lanes (spin 2) of a thread.
static const int kTiles0[][2] = {{1, 1}, {1, 2}, {1, 4}, {2, 1}, {2, 2}, {2, 4}, {4, 1}, {4, 2}, {8, 1}, {2, 8}};
static const int kTiles2[][2] = {{2, 1}, {2, 2}, {2, 4}, {2, 8}};
constexpr int kNTiles0 = sizeof(kTiles0) / sizeof(kTiles0[0]);
constexpr int kNTiles2 = sizeof(kTiles2) / sizeof(kTiles2[0]);

template <typename T>
static int tile_ana(int spin, int tile, int64_t nside, int64_t lmax, int64_t ncomp,
                    const double *geom, const double *seeds, const void *rhs, double *alm,
                    double scale, cudaStream_t s)
{
#define GM_ANA(SP, NC, R) return launch_ana<T, SP, NC, R>(spin, nside, lmax, ncomp, geom, seeds, rhs, alm, scale, s)
    if (spin == 0) {
        switch (tile) {
        case 0: GM_ANA(0, 1, 1);
        case 1: GM_ANA(0, 1, 2);
        case 2: GM_ANA(0, 1, 4);
        case 3: GM_ANA(0, 2, 1);
        case 4: GM_ANA(0, 2, 2);
        case 5: GM_ANA(0, 2, 4);
        case 6: GM_ANA(0, 4, 1);
        case 7: GM_ANA(0, 4, 2);
        case 8: GM_ANA(0, 8, 1);
        case 9:
            if constexpr (sizeof(T) == 8) { GM_ANA(0, 2, 4); } else { GM_ANA(0, 2, 8); }
        default: return GM_ERR_BAD_SHAPE;
        }
    }
    switch (tile) {
    case 0: GM_ANA(2, 2, 1);
    case 1: GM_ANA(2, 2, 2);
    case 2: GM_ANA(2, 2, 4);
    case 3:
        if constexpr (sizeof(T) == 8) { GM_ANA(2, 2, 4); } else { GM_ANA(2, 2, 8); }
    default: return GM_ERR_BAD_SHAPE;
    }
#undef GM_ANA
}

template <typename T>
static int tile_syn(int spin, int tile, int64_t nside, int64_t lmax, int64_t ncomp,
                    const double *geom, const double *seeds, const double *alm, void *syn,
                    cudaStream_t s)
{
#define GM_SYN(SP, NC, R) return launch_syn<T, SP, NC, R>(spin, nside, lmax, ncomp, geom, seeds, alm, syn, s)
    if (spin == 0) {
        switch (tile) {
        case 0: GM_SYN(0, 1, 1);
        case 1: GM_SYN(0, 1, 2);
        case 2: GM_SYN(0, 1, 4);
        case 3: GM_SYN(0, 2, 1);
        case 4: GM_SYN(0, 2, 2);
        case 5: GM_SYN(0, 2, 4);
        case 6: GM_SYN(0, 4, 1);
        case 7: GM_SYN(0, 4, 2);
        case 8: GM_SYN(0, 8, 1);
        case 9:
            if constexpr (sizeof(T) == 8) { GM_SYN(0, 2, 4); } else { GM_SYN(0, 2, 8); }
        default: return GM_ERR_BAD_SHAPE;
        }
    }
    switch (tile) {
    case 0: GM_SYN(2, 2, 1);
    case 1: GM_SYN(2, 2, 2);
    case 2: GM_SYN(2, 2, 4);
    case 3:
        if constexpr (sizeof(T) == 8) { GM_SYN(2, 2, 4); } else { GM_SYN(2, 2, 8); }
    default: return GM_ERR_BAD_SHAPE;
    }
#undef GM_SYN
}

extern "C" int gm_legendre_tiles(int spin, int32_t *nc_r, int capacity)
{
    if (spin < 0 || spin > kMaxSpin) return -1;
    const int n = spin == 0 ? kNTiles0 : kNTiles2;
    for (int i = 0; i < n && i < capacity; ++i) {
        nc_r[2 * i] = spin == 0 ? kTiles0[i][0] : kTiles2[i][0];
        nc_r[2 * i + 1] = spin == 0 ? kTiles0[i][1] : kTiles2[i][1];
    }
    return n;
}

extern "C" int gm_legendre_analysis_tile(int precision, int spin, int64_t nside, int64_t lmax,
                                         int64_t ncomp, const double *lane_geom, const double *seeds,
                                         const void *rhs, double *alm, double scale, int tile,
                                         void *stream)
{
    if (nside < 1 || lmax < 0 || lmax + 1 > 65535 || ncomp < 1 || ncomp > 65535)
        return GM_ERR_BAD_SHAPE;
    if (spin < 0 || spin > kMaxSpin) return GM_ERR_UNSUPPORTED;
    if (spin != 0 && (ncomp % 2)) return GM_ERR_BAD_SHAPE;
    if (tile < -1 || tile >= (spin == 0 ? kNTiles0 : kNTiles2)) return GM_ERR_BAD_SHAPE;
    if (!lane_geom || !seeds || !rhs || !alm) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    if (precision == GM_FP64)
        return tile < 0 ? dispatch_ana<double>(spin, nside, lmax, ncomp, lane_geom, seeds, rhs, alm, scale, s)
                        : tile_ana<double>(spin, tile, nside, lmax, ncomp, lane_geom, seeds, rhs, alm, scale, s);
    if (precision == GM_MIXED)
        return tile < 0 ? dispatch_ana<float>(spin, nside, lmax, ncomp, lane_geom, seeds, rhs, alm, scale, s)
                        : tile_ana<float>(spin, tile, nside, lmax, ncomp, lane_geom, seeds, rhs, alm, scale, s);
    return GM_ERR_UNSUPPORTED;
}

extern "C" int gm_legendre_synthesis_tile(int precision, int spin, int64_t nside, int64_t lmax,
                                          int64_t ncomp, const double *lane_geom, const double *seeds,
                                          const double *alm, void *syn, int tile, void *stream)
{
    if (nside < 1 || lmax < 0 || lmax + 1 > 65535 || ncomp < 1 || ncomp > 65535)
        return GM_ERR_BAD_SHAPE;
    if (spin < 0 || spin > kMaxSpin) return GM_ERR_UNSUPPORTED;
    if (spin != 0 && (ncomp % 2)) return GM_ERR_BAD_SHAPE;
    if (tile < -1 || tile >= (spin == 0 ? kNTiles0 : kNTiles2)) return GM_ERR_BAD_SHAPE;
    if (!lane_geom || !seeds || !alm || !syn) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    if (precision == GM_FP64)
        return tile < 0 ? dispatch_syn<double>(spin, nside, lmax, ncomp, lane_geom, seeds, alm, syn, s)
                        : tile_syn<double>(spin, tile, nside, lmax, ncomp, lane_geom, seeds, alm, syn, s);
    if (precision == GM_MIXED)
        return tile < 0 ? dispatch_syn<float>(spin, nside, lmax, ncomp, lane_geom, seeds, alm, syn, s)
                        : tile_syn<float>(spin, tile, nside, lmax, ncomp, lane_geom, seeds, alm, syn, s);
    return GM_ERR_UNSUPPORTED;
}

extern "C" int gm_legendre_analysis(int precision, int spin, int64_t nside, int64_t lmax,
                                    int64_t ncomp, const double *lane_geom, const double *seeds,
                                    const void *rhs, double *alm, double scale, void *stream)
{
    if (nside < 1 || lmax < 0 || lmax + 1 > 65535 || ncomp < 1 || ncomp > 65535)
        return GM_ERR_BAD_SHAPE;
    if (spin < 0 || spin > kMaxSpin) return GM_ERR_UNSUPPORTED;
    if (spin != 0 && (ncomp % 2)) return GM_ERR_BAD_SHAPE;
    if (!lane_geom || !seeds || !rhs || !alm) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    if (precision == GM_FP64)
        return dispatch_ana<double>(spin, nside, lmax, ncomp, lane_geom, seeds, rhs, alm, scale, s);
    if (precision == GM_MIXED)
        return dispatch_ana<float>(spin, nside, lmax, ncomp, lane_geom, seeds, rhs, alm, scale, s);
    return GM_ERR_UNSUPPORTED;
}

extern "C" int gm_legendre_synthesis(int precision, int spin, int64_t nside, int64_t lmax,
                                     int64_t ncomp, const double *lane_geom, const double *seeds,
                                     const double *alm, void *syn, void *stream)
{
    if (nside < 1 || lmax < 0 || lmax + 1 > 65535 || ncomp < 1 || ncomp > 65535)
        return GM_ERR_BAD_SHAPE;
    if (spin < 0 || spin > kMaxSpin) return GM_ERR_UNSUPPORTED;
    if (spin != 0 && (ncomp % 2)) return GM_ERR_BAD_SHAPE;
    if (!lane_geom || !seeds || !alm || !syn) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    if (precision == GM_FP64)
        return dispatch_syn<double>(spin, nside, lmax, ncomp, lane_geom, seeds, alm, syn, s);
    if (precision == GM_MIXED)
        return dispatch_syn<float>(spin, nside, lmax, ncomp, lane_geom, seeds, alm, syn, s);
    return GM_ERR_UNSUPPORTED;
}

// The Jacobi refinement of one field's analysis, n_iter times synthesis, ring-fold residual and
// analysis, issued by one call.  segoff: checkpointed rows (legendre_rows.cu); NULL: the FP64
// recurrence.
extern "C" int gm_refine(int precision, int spin, int64_t nside, int64_t lmax, int64_t ncomp, int64_t n_iter,
                         const double *lane_geom, const double *seeds, const void *rhs_map, const uint8_t *shifted,
                         void *syn, void *res, double *alm, int tile_syn, int tile_ana, const int64_t *segoff,
                         const void *ck_a, const uint8_t *cn_a, const void *ck_b, const uint8_t *cn_b,
                         const uint64_t *mask_a, const uint64_t *mask_b, void *stream)
{
    if (segoff && precision != GM_MIXED) return GM_ERR_UNSUPPORTED;
    for (int64_t it = 0; it < n_iter; ++it) {
        int st = segoff ? gm_legendre_synthesis_ck(spin, nside, lmax, ncomp, lane_geom, alm, syn, segoff, ck_a, cn_a,
                                                   ck_b, cn_b, mask_a, mask_b, tile_syn, stream)
                        : gm_legendre_synthesis_tile(precision, spin, nside, lmax, ncomp, lane_geom, seeds, alm, syn,
                                                     tile_syn, stream);
        if (st == GM_OK) st = gm_fold_residual(precision, nside, lmax + 1, ncomp, syn, rhs_map, shifted, res, stream);
        if (st == GM_OK)
            st = segoff ? gm_legendre_analysis_ck(spin, nside, lmax, ncomp, lane_geom, res, alm, -1.0, segoff, ck_a, cn_a,
                                                  ck_b, cn_b, mask_a, mask_b, tile_ana, stream)
                        : gm_legendre_analysis_tile(precision, spin, nside, lmax, ncomp, lane_geom, seeds, res, alm, -1.0,
                                                    tile_ana, stream);
        if (st != GM_OK) return st;
    }
    return GM_OK;
}
