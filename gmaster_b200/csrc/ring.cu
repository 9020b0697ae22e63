// Azimuthal (ring) stage of the HEALPix spherical-harmonic transforms, sm_100a.
//
// One CTA transforms one ring of one map component entirely in shared memory:
// a real ring of nphi = 4i samples is packed into a complex sequence of length
// h = nphi/2 (even samples real, odd samples imaginary), transformed by a
// self-sorting Stockham FFT of mixed radix (4, 2, then odd primes; a generic
// radix-p stage for large prime factors), and unpacked.  Loads and stores of
// pixels and spectra are coalesced along the ring / along m.
//
// Replaces the reference's XLA-lowered ring stage (gmaster/_sht/rings.py:251-299
// forward, :477-524 inverse: a cuFFT of the equatorial belt plus Bluestein chirp-Z
// convolutions for the polar caps) and its ring-fold residual kernel
// (gmaster/_native/cuda/march_v2.cu:426-493).
#include <math.h>

#include <type_traits>

#include "gm_common.cuh"

namespace gm {

// ---------------------------------------------------------------- twiddles

// tw64[i(i-1) + k] = exp(-2 pi i k / (4 i)), k < 2 i, followed by the float copy.
__global__ void k_twiddles(int64_t nside, double2 *tw64, float2 *tw32)
{
    int64_t i = blockIdx.y + 1;
    int64_t half = 2 * i;
    for (int64_t k = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; k < half;
         k += (int64_t)gridDim.x * blockDim.x) {
        double s, c;
        sincospi(-(double)k / (double)half, &s, &c);  // -2 pi k / (4 i) = -pi k / (2 i)
        int64_t idx = i * (i - 1) + k;
        tw64[idx] = make_double2(c, s);
        tw32[idx] = make_float2((float)c, (float)s);
    }
}

template <typename T2> struct TwTable;
template <> struct TwTable<double2> {
    static __device__ __forceinline__ const double2 *get(const void *tw, int64_t cnt)
    {
        return reinterpret_cast<const double2 *>(tw);
    }
};
template <> struct TwTable<float2> {
    static __device__ __forceinline__ const float2 *get(const void *tw, int64_t cnt)
    {
        return reinterpret_cast<const float2 *>(reinterpret_cast<const double2 *>(tw) + cnt);
    }
};

// omega_h^e for an FFT of length h and 0 <= e < h, from the table of n = TM h: tw holds
// omega_n^k for k < n / 2, and omega_n^{k + n/2} = -omega_n^k.  TM = 2 is the ring
// transform (n = 2h, the ring's own table); TM = 1 a length-h FFT with its own table
// (h = n).  `sign` > 0 conjugates (inverse transform).
template <int TM = 2, typename T2>
__device__ __forceinline__ T2 twiddle(const T2 *__restrict__ tw, int h, int e, int sign)
{
    const int k = TM * e, half = TM * h / 2;
    T2 w;
    if (k < half) {
        w = __ldg(tw + k);
    } else {
        w = __ldg(tw + (k - half));
        w.x = -w.x;
        w.y = -w.y;
    }
    if (sign > 0) w.y = -w.y;
    return w;
}

// omega_n^k for k < n (n = 2h).
template <typename T2>
__device__ __forceinline__ T2 twiddle_n(const T2 *__restrict__ tw, int h, int k, int sign)
{
    T2 w;
    if (k < h) {
        w = __ldg(tw + k);
    } else {
        w = __ldg(tw + (k - h));
        w.x = -w.x;
        w.y = -w.y;
    }
    if (sign > 0) w.y = -w.y;
    return w;
}

// e^{sign i pi q2 / n} for 0 <= q2 < 2n from the table: omega_n^{q2/2} (times e^{-i pi / n}
// for odd q2), conjugated for sign > 0.  c1 = e^{-i pi / n}.
template <typename T2>
__device__ __forceinline__ T2 phase_pi(const T2 *__restrict__ tw, int h, int q2, T2 c1, int sign)
{
    T2 w = twiddle_n(tw, h, q2 >> 1, -1);
    if (q2 & 1) w = cmul(w, c1);
    if (sign > 0) w.y = -w.y;
    return w;
}

// ---------------------------------------------------------------- FFT core

// Radices of h into rad (4s, a 2, then odd primes ascending), written by one warp of 32
// threads that test 32 odd divisors at a time; returns their number.
__device__ int factorize(int h, int *rad)
{
    const int lane = threadIdx.x & 31;
    int n = 0;
    auto put = [&](int p) {
        if (lane == 0) rad[n] = p;
        ++n;
    };
    while (h % 4 == 0) { put(4); h /= 4; }
    if (h % 2 == 0) { put(2); h /= 2; }
    for (int base = 3; base * base <= h; base += 64) {
        const int d = base + 2 * lane;
        unsigned hit = __ballot_sync(0xffffffffu, d <= h && h % d == 0);
        while (hit) {   // ascending: a composite divisor no longer divides
            const int p = base + 2 * (__ffs(hit) - 1);
            hit &= hit - 1;
            while (p * p <= h && h % p == 0) { put(p); h /= p; }
        }
    }
    if (h > 1) put(h);
    return n;
}

// Multiply by sign * i.
template <typename T2>
__device__ __forceinline__ T2 mul_i(T2 z, int sign)
{
    T2 r;
    r.x = -sign * z.y;
    r.y = sign * z.x;
    return r;
}

// One Stockham stage: out[k' Lp + j + Ls v] = sum_q omega_p^{q v} omega_Lp^{q j} in[(k' + r q) Ls + j]
// with Lp = Ls p and r = h / Lp.  Butterflies (k', j) are spread over the CTA.
template <int TM, typename T2>
__device__ void stockham_stage(const T2 *__restrict__ in, T2 *__restrict__ out, int h, int p,
                               int Ls, const T2 *__restrict__ tw, int sign)
{
    const int Lp = Ls * p;
    const int r = h / Lp;
    const int nb = h / p;
    if (p == 4) {
        // the radix-4 and radix-2 stages come first: Ls is a power of two
        const int lg = 31 - __clz(Ls);
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            const int kk = b >> lg, j = b & (Ls - 1);
            T2 x0 = in[kk * Ls + j];
            T2 x1 = in[(kk + r) * Ls + j];
            T2 x2 = in[(kk + 2 * r) * Ls + j];
            T2 x3 = in[(kk + 3 * r) * Ls + j];
            if (Ls > 1) {
                const int e = j * r;   // < h / 4
                x1 = cmul(x1, twiddle<TM>(tw, h, e, sign));
                x2 = cmul(x2, twiddle<TM>(tw, h, 2 * e, sign));
                x3 = cmul(x3, twiddle<TM>(tw, h, 3 * e, sign));
            }
            T2 a = cadd(x0, x2), bq = csub(x0, x2);
            T2 c = cadd(x1, x3), d = mul_i(csub(x1, x3), sign);
            T2 *o = out + kk * Lp + j;
            o[0] = cadd(a, c);
            o[Ls] = cadd(bq, d);
            o[2 * Ls] = csub(a, c);
            o[3 * Ls] = csub(bq, d);
        }
    } else if (p == 2) {
        const int lg = 31 - __clz(Ls);
        for (int b = threadIdx.x; b < nb; b += blockDim.x) {
            const int kk = b >> lg, j = b & (Ls - 1);
            T2 x0 = in[kk * Ls + j];
            T2 x1 = in[(kk + r) * Ls + j];
            if (Ls > 1) x1 = cmul(x1, twiddle<TM>(tw, h, j * r, sign));   // j r < h / 2
            T2 *o = out + kk * Lp + j;
            o[0] = cadd(x0, x1);
            o[Ls] = csub(x0, x1);
        }
    } else {
        // generic radix: one output (k', j, v) per thread iteration, p terms each
        for (int o = threadIdx.x; o < h; o += blockDim.x) {
            int kk = o / Lp, jp = o - kk * Lp;
            int j = jp % Ls;
            T2 acc;
            acc.x = 0;
            acc.y = 0;
            // term q: omega_Lp^{q jp} in[(kk + r q) Ls + j];  omega_Lp = omega_h^r, with
            // the exponent q jp mod Lp stepped incrementally
            int eq = 0;
            for (int q = 0; q < p; ++q) {
                T2 x = in[(kk + r * q) * Ls + j];
                T2 w = twiddle<TM>(tw, h, eq * r, sign);
                acc.x += x.x * w.x - x.y * w.y;
                acc.y += x.x * w.y + x.y * w.x;
                eq += jp;
                if (eq >= Lp) eq -= Lp;
            }
            out[o] = acc;
        }
    }
}

// In-shared-memory FFT of length h (ping-pong between a and b); returns the buffer
// holding the result.  Ends with a __syncthreads().
template <int TM = 2, typename T2>
__device__ T2 *fft_shared(T2 *a, T2 *b, int h, const T2 *__restrict__ tw, int sign)
{
    __shared__ int rad[40];
    __shared__ int nst;
    if (threadIdx.x < 32) {
        const int k = factorize(h, rad);
        if (threadIdx.x == 0) nst = k;
    }
    __syncthreads();
    int Ls = 1;
    for (int s = 0; s < nst; ++s) {
        int p = rad[s];
        stockham_stage<TM>(a, b, h, p, Ls, tw, sign);
        __syncthreads();
        T2 *t = a;
        a = b;
        b = t;
        Ls *= p;
    }
    return a;
}

// ---------------------------------------------------------------- analysis

// Rings whose half-length h has a prime factor above 64 are transformed by Bluestein's
// chirp-z method (three power-of-two FFTs of length M = nextpow2(2h - 1) <= mcap), instead of a
// generic radix-p stage costing h p.
__host__ __device__ __forceinline__ int largest_prime_factor(int h)
{
    int p = 1;
    for (int q = 2; q * q <= h; ++q)
        while (h % q == 0) {
            p = q;
            h /= q;
        }
    return h > p ? h : p;
}

__host__ __device__ __forceinline__ int next_pow2(int x)
{
    int m = 1;
    while (m < x) m <<= 1;
    return m;
}

// Largest prime factor transformed by a direct stage.
constexpr int kDirectPrime = 64;

__host__ __device__ __forceinline__ bool use_bluestein(int h, int mcap)
{
    return largest_prime_factor(h) > kDirectPrime && next_pow2(2 * h - 1) <= mcap;
}

// Largest power-of-two FFT length of the Bluestein path: its table must exist (a ring
// length 4i with i <= nside) and three buffers of it must fit in shared memory.
static inline int bluestein_mcap(int64_t nside)
{
    int64_t m = 1;
    while (2 * m <= 4 * nside && 2 * m <= 8192) m *= 2;
    return (int)m;
}

// Rings beyond the shared-memory kernels: half-length above `hcap` (the ping-pong buffers
// would not fit), or, in single precision, a prime factor above 64 with a Bluestein length
// 2h - 1 < M above `bsmin` (8192, the shared-memory Bluestein length; 0: none) for which the
// M-point table exists (M <= 4 nside).  They are transformed by the persistent *_big kernels
// in global scratch.
__host__ __device__ __forceinline__ bool bluestein_big(int h, int nside, int bsmin)
{
    const int M = next_pow2(2 * h - 1);
    return bsmin > 0 && largest_prime_factor(h) > 64 && M > bsmin && M <= 4 * nside;
}

__host__ __device__ __forceinline__ bool ring_big(int h, int hcap, int nside, int bsmin)
{
    return h > hcap || bluestein_big(h, nside, bsmin);
}

// ---- Bluestein's method: the DFT of length h as a circular convolution of length M

template <typename T2>
__device__ __forceinline__ T2 bs_chirp(const T2 *__restrict__ tw, int h, int n, int j, int sign)
{
    const unsigned q = ((unsigned)j * (unsigned)j) % (unsigned)n;
    return twiddle_n(tw, h, (int)q, sign);   // e^{sign i pi j^2 / h}
}

// Bluestein filter: the transform of the wrapped conjugate chirp of length M; returns the
// buffer holding it (b0 or b1).
template <typename T2>
__device__ T2 *bs_filter(int h, int n, int M, const T2 *__restrict__ tw, const T2 *__restrict__ twM, int sign,
                         T2 *b0, T2 *b1)
{
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        T2 v{};
        int j = -1;
        if (m < h) j = m;
        else if (m > M - h) j = M - m;
        if (j >= 0) {
            v = bs_chirp(tw, h, n, j, sign);
            v.y = -v.y;
        }
        b0[m] = v;
    }
    __syncthreads();
    return fft_shared<1>(b0, b1, M, twM, -1);
}

// X[0, h) holds z_j c_j; zero-pads to M, convolves with the filter FB and returns the buffer
// holding the DFT sum_j z_j e^{sign 2 pi i jk / h}, k < h.
template <typename T2>
__device__ T2 *bs_apply(T2 *X, T2 *Y, const T2 *FB, int h, int n, int M, const T2 *__restrict__ tw,
                        const T2 *__restrict__ twM, int sign)
{
    for (int j = h + threadIdx.x; j < M; j += blockDim.x) X[j] = T2{};
    __syncthreads();
    T2 *FA = fft_shared<1>(X, Y, M, twM, -1);
    T2 *G = (FA == X) ? Y : X;
    const auto invM = (decltype(X->x))1 / (decltype(X->x))M;
    for (int m = threadIdx.x; m < M; m += blockDim.x) {
        T2 v = cmul(FA[m], FB[m]);
        v.x *= invM;
        v.y *= invM;
        FA[m] = v;
    }
    __syncthreads();
    T2 *R = fft_shared<1>(FA, G, M, twM, +1);
    T2 *Z = (R == FA) ? G : FA;
    for (int k = threadIdx.x; k < h; k += blockDim.x) Z[k] = cmul(R[k], bs_chirp(tw, h, n, k, sign));
    __syncthreads();
    return Z;
}

// Load one ring of one map (times the mask) as h complex z_t = x_2t + i x_2t+1, each
// multiplied by f(t) (the Bluestein chirp, or 1).  vec: x and mask are aligned to two elements
// (every ring starts at an even pixel), so a pair is one load.
template <typename T, typename Tin, typename T2, typename F>
__device__ __forceinline__ void load_ring(const Tin *__restrict__ x, const double *__restrict__ mask, bool vec,
                                          int h, T2 *__restrict__ dst, F f)
{
    using Tin2 = typename vec2<Tin>::type;
    for (int t = threadIdx.x; t < h; t += blockDim.x) {
        Tin2 p;
        if (vec) {
            p = reinterpret_cast<const Tin2 *>(x)[t];
        } else {
            p.x = x[2 * t];
            p.y = x[2 * t + 1];
        }
        T2 z;
        if (mask) {
            // masked field: the FP64 product map * mask, rounded once to T
            double2 w;
            if (vec) {
                w = reinterpret_cast<const double2 *>(mask)[t];
            } else {
                w.x = mask[2 * t];
                w.y = mask[2 * t + 1];
            }
            z.x = (T)((double)p.x * w.x);
            z.y = (T)((double)p.y * w.y);
        } else {
            z.x = (T)p.x;
            z.y = (T)p.y;
        }
        dst[t] = f(t, z);
    }
}

// Unpack the half-length transform Z of one real ring into its spectrum for m < L, with
// the quadrature weight and the ring phase e^{-i m phi0}: dst[m] = w e^{-i m phi0} X[m mod n].
template <typename T, typename T2>
__device__ __forceinline__ void ring_outputs(const T2 *__restrict__ Z, int n, int64_t L,
                                             const T2 *__restrict__ tw, bool sh, T w,
                                             T2 *__restrict__ dst)
{
    const int h = n / 2;
    T2 c1;   // e^{-i pi / n}
    {
        double s1, c1d;
        sincospi(-1.0 / (double)n, &s1, &c1d);
        c1.x = (T)c1d;
        c1.y = (T)s1;
    }
    const unsigned n2 = 2u * (unsigned)n;
    for (int m = threadIdx.x; m < (int)L; m += blockDim.x) {
        const unsigned m2 = (unsigned)m % n2;           // m mod 2n
        const int k = (int)(m2 < (unsigned)n ? m2 : m2 - (unsigned)n);
        const bool conj = k > h;
        const int kk = conj ? n - k : k;                // 0..h
        // X[kk] = E + omega_n^kk O, E = (Z[kk] + conj Z[h-kk]) / 2, O = (Z[kk] - conj Z[h-kk]) / 2i
        const T2 za = Z[kk == h ? 0 : kk], zb = Z[kk == 0 ? 0 : h - kk];
        T er = (za.x + zb.x) * (T)0.5, ei = (za.y - zb.y) * (T)0.5;
        T orr = (za.y + zb.y) * (T)0.5, oi = -(za.x - zb.x) * (T)0.5;
        T2 wn = twiddle_n(tw, h, kk, -1);
        T xr = er + wn.x * orr - wn.y * oi;
        T xi = ei + wn.x * oi + wn.y * orr;
        if (conj) xi = -xi;
        T pr = 1, pi = 0;
        if (sh) {
            // e^{-i m phi0}, phi0 = pi / n
            const T2 ph = phase_pi(tw, h, (int)m2, c1, -1);
            pr = ph.x;
            pi = ph.y;
        }
        T2 g;
        g.x = w * (xr * pr - xi * pi);
        g.y = w * (xr * pi + xi * pr);
        dst[m] = g;
    }
}

// Ring of row b of a launch (forward and inverse): the cap rings of length 4 i, i0 <= i < i0 + cnt,
// longest first (the north and the south one), then the belt.
__device__ __forceinline__ int64_t launch_ring(int64_t nside, int64_t i0, int64_t cnt, int64_t b)
{
    if (b >= 2 * cnt) return nside - 1 + b - 2 * cnt;
    const int64_t i = i0 + cnt - 1 - (b >> 1);
    return b & 1 ? 4 * nside - 1 - i : i - 1;
}

// Forward ring transform: one CTA per (ring, block of cpc components), the component block the
// fast grid index so that the CTAs of one ring run together and read its mask once from DRAM.
// Rings whose half-length has a prime factor above 64 go through Bluestein's method (M <= mcap:
// three buffers of M; the transform of the chirp once per CTA), the others through the
// mixed-radix FFT.  Bound by the passes over shared memory (one per radix) and their barriers:
// an eighth of the points as threads, two radix-4 butterflies each, fills an SM with CTAs.
template <typename T, typename Tin, bool BS>
__global__ void __launch_bounds__(512) k_ring_forward(int64_t nside, int64_t L, int64_t ncomp, int cpc,
                                                      const Tin *__restrict__ maps,
                                                      const double *__restrict__ mask, bool vec,
                                                      const void *__restrict__ twall, int64_t twcnt,
                                                      const uint8_t *__restrict__ shifted,
                                                      typename vec2<T>::type *__restrict__ out, int64_t i0,
                                                      int64_t cnt, int mcap, int hcap, int bsmin, int buf)
{
    using T2 = typename vec2<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int64_t r = launch_ring(nside, i0, cnt, blockIdx.y), nring = 4 * nside - 1, npix = 12 * nside * nside;
    const int n = (int)ring_nphi(nside, r), h = n / 2;
    const bool bs = BS && use_bluestein(h, mcap);
    if (hcap > 0 && ring_big(h, hcap, (int)nside, bsmin)) return;   // left to k_ring_analysis_big
    const int64_t off = ring_offset(nside, r);
    const bool sh = shifted[r] != 0;
    T2 *b0 = reinterpret_cast<T2 *>(smem_raw), *b1 = b0 + buf, *b2 = b1 + buf;
    const T2 *twT = TwTable<T2>::get(twall, twcnt);
    const T2 *tw = twT + twiddle_offset(n);
    const int M = bs ? next_pow2(2 * h - 1) : 0;
    const T2 *twM = bs ? twT + twiddle_offset(M) : nullptr;
    T2 *FB = nullptr, *X = b0, *Y = b1;
    if (bs) {
        FB = bs_filter(h, n, M, tw, twM, -1, b0, b1);
        X = FB == b0 ? b1 : b0;
        Y = b2;
    }
    const T w = (T)(4.0 * M_PI / (double)npix);
    const int64_t cend = (int64_t)(blockIdx.x + 1) * cpc < ncomp ? (int64_t)(blockIdx.x + 1) * cpc : ncomp;
    for (int64_t c = (int64_t)blockIdx.x * cpc; c < cend; ++c) {
        const double *mk = mask ? mask + off : nullptr;
        const T2 *Z;
        if (bs) {
            load_ring<T>(maps + c * npix + off, mk, vec, h, X,
                         [&](int t, T2 z) { return cmul(z, bs_chirp(tw, h, n, t, -1)); });
            __syncthreads();
            Z = bs_apply(X, Y, FB, h, n, M, tw, twM, -1);
        } else {
            load_ring<T>(maps + c * npix + off, mk, vec, h, X, [](int, T2 z) { return z; });
            __syncthreads();
            Z = fft_shared(X, Y, h, tw, -1);
        }
        ring_outputs<T>(Z, n, L, tw, sh, w, out + (c * nring + r) * L);
        __syncthreads();
    }
}

// ---------------------------------------------------------------- hemisphere pack

template <typename T>
__global__ void k_pack_rhs(int64_t nside, int64_t L, int64_t ncomp,
                           const typename vec2<T>::type *__restrict__ spec, T *__restrict__ rhs)
{
    using T2 = typename vec2<T>::type;
    __shared__ T tile[32][33][4];
    const int64_t nlanes = 2 * nside, nring = 4 * nside - 1;
    const int64_t m0 = (int64_t)blockIdx.x * 32, j0 = (int64_t)blockIdx.y * 32, c = blockIdx.z;
    const int tx = threadIdx.x, ty = threadIdx.y;
    for (int jj = ty; jj < 32; jj += 8) {
        int64_t j = j0 + jj, m = m0 + tx;
        T v[4] = {0, 0, 0, 0};
        if (j < nlanes && m < L) {
            T2 gn = spec[(c * nring + north_ring(j)) * L + m];
            T2 gs;
            gs.x = 0;
            gs.y = 0;
            if (j != nlanes - 1) gs = spec[(c * nring + south_ring(nside, j)) * L + m];
            v[0] = gn.x + gs.x;
            v[1] = gn.y + gs.y;
            v[2] = gn.x - gs.x;
            v[3] = gn.y - gs.y;
        }
        for (int q = 0; q < 4; ++q) tile[jj][tx][q] = v[q];
    }
    __syncthreads();
    for (int mm = ty; mm < 32; mm += 8) {
        int64_t m = m0 + mm, j = j0 + tx;
        if (j < nlanes && m < L) {
            T *o = rhs + ((m * nlanes + j) * ncomp + c) * 4;
            for (int q = 0; q < 4; ++q) o[q] = tile[tx][mm][q];
        }
    }
}

// ---------------------------------------------------------------- fold residual

// Sum over the residue class k (mod n) of the synthesised coefficients of one ring
// side (`part` 0 north, 2 south) with the alternating sign (-1)^{s t} of the ring
// shift: P_k = sum_t (-1)^{s t} c(k + t n), |k + t n| < L, c(-m) = conj c(m).
template <typename T>
__device__ __forceinline__ void residue_sums(const T *__restrict__ syn, int64_t L, int64_t nlanes,
                                             int64_t ncomp, int64_t j, int64_t c, int k, int n,
                                             bool sh, bool two_sides, T *pn, T *ps)
{
    T nr = 0, ni = 0, sr = 0, si = 0;
    // t >= 0 : m = k + t n in [0, L)
    int t = 0;
    for (int64_t m = k; m < L; m += n, ++t) {
        const T *e = syn + ((m * nlanes + j) * ncomp + c) * 4;
        T sg = (sh && (t & 1)) ? (T)-1 : (T)1;
        nr += sg * e[0];
        ni += sg * e[1];
        if (two_sides) {
            sr += sg * e[2];
            si += sg * e[3];
        }
    }
    // t < 0 : m = k - t' n (t' >= 1), order m < 0 with -m = t' n - k in (0, L)
    t = -1;
    for (int64_t mm = (int64_t)n - k; mm < L; mm += n, --t) {
        if (mm == 0) continue;
        const T *e = syn + ((mm * nlanes + j) * ncomp + c) * 4;
        T sg = (sh && (t & 1)) ? (T)-1 : (T)1;
        nr += sg * e[0];
        ni -= sg * e[1];
        if (two_sides) {
            sr += sg * e[2];
            si -= sg * e[3];
        }
    }
    pn[0] = nr;
    pn[1] = ni;
    ps[0] = sr;
    ps[1] = si;
}

// Both hemispheres' coefficients of one order: (north re, im, south re, im), of 16-byte aligned
// arrays or (not WIDE) of arrays aligned to their elements only.
template <typename T, bool WIDE> struct alignas(WIDE ? 16 : sizeof(T)) Quad {
    T x, y, z, w;
};

// Ring fold of J consecutive (lane, component) columns of syn (L, nlanes, ncomp, 4): for every
// residue k of the ring length n,
//   P_k = sum_t sigma^t c(k + t n) + sum_{t >= 1} sigma^t conj c(t n - k),  sigma = -1 if shifted,
// from A_k = sum_{t >= 0} sigma^t c(k + t n) as P_k = A_k + sigma conj A_{n-k}: residues k and
// n - k are summed together, so every coefficient is read once.  A CTA's threads run along
// the J columns first (J x 16 or 32 contiguous bytes a row), then over the residue pairs; on
// short rings (pairs fewer than half the slots) several slots share a pair, each summing every
// s-th alias, and their sums are added in a fixed order.
//   RESIDUAL: out(m) = sigma^t w n P_k - rhs_map(m) for m = k + t n, as Sum / Diff halves;
//   otherwise spec[comp][ring][k] = P_k, k <= n / 2, of the north and the south ring.
// Bound by memory: reads syn (and rhs_map) once, writes once.  One thread block per lane with
// the threads along m read 16 bytes per 32-byte sector 128 lanes apart and summed the aliases
// of the polar rings (n = 4, 8, ...) in a few threads: 2.2 -> 0.45 ms a pass at Nside 2048 with
// one map (1.2 GB: 2.7 TB/s), 370 -> 78 us at Nside 512 with a (Q, U) pair.
__host__ __device__ constexpr int fold_threads(int J) { return J == 8 ? 512 : 256; }

template <typename T, int J, bool RESIDUAL, bool WIDE>
__global__ void __launch_bounds__(fold_threads(J)) k_fold_lanes(int64_t nside, int64_t L, int64_t ncomp, int64_t cbeg, int64_t cw,
                                                    const Quad<T, WIDE> *__restrict__ syn,
                                                    const Quad<T, WIDE> *__restrict__ rhs_map,
                                                    const uint8_t *__restrict__ shifted, Quad<T, WIDE> *__restrict__ out,
                                                    typename vec2<T>::type *__restrict__ spec, int64_t sstride)
{
    using T2 = typename vec2<T>::type;
    using Q4 = Quad<T, WIDE>;
    constexpr int NT = fold_threads(J), Q = NT / J;
    __shared__ Q4 pa[NT], pb[NT];
    const int64_t nlanes = 2 * nside, stride = nlanes * ncomp;
    const int q = threadIdx.x / J;
    const int64_t item = (int64_t)blockIdx.x * J + threadIdx.x % J;
    const bool ok = item < nlanes * cw;
    const int64_t j = ok ? item / cw : 0, c = cbeg + (ok ? item % cw : 0);
    const int64_t col = j * ncomp + c;
    const int n = (int)ring_nphi(nside, north_ring(j)), np = n / 2 + 1;
    const bool sh = shifted[north_ring(j)] != 0, two = j != nlanes - 1;
    const T sigma = sh ? (T)-1 : (T)1;
    const T wn = (T)(4.0 * M_PI / (double)(12 * nside * nside) * (double)n);
    const Q4 *src = syn + col;
    int s = 1;
    while (2 * s * np <= Q) s *= 2;
    const int part = q & (s - 1);

    // aliases k + t n, t = t0, t0 + s, ...
    auto sum = [&](int k, int t0) {
        Q4 a{0, 0, 0, 0};
        const int64_t dm = (int64_t)s * n;
        int t = t0;
#pragma unroll 4
        for (int64_t m = k + (int64_t)t0 * n; m < L; m += dm, t += s) {
            const Q4 v = src[m * stride];
            const T sg = (sh && (t & 1)) ? (T)-1 : (T)1;
            a.x += sg * v.x;
            a.y += sg * v.y;
            a.z += sg * v.z;
            a.w += sg * v.w;
        }
        return a;
    };
    auto pair_sums = [&](int p, Q4 &A, Q4 &B) {
        // residue 0 leaves order 0 to the caller
        A = sum(p, p == 0 && part == 0 ? s : part);
        B = (p > 0 && 2 * p < n) ? sum(n - p, part) : Q4{0, 0, 0, 0};
    };
    auto emit = [&](int k, const Q4 &P) {
        if (RESIDUAL) {
            const int64_t dm = (int64_t)s * n;
            int t = part;
#pragma unroll 4
            for (int64_t m = k + (int64_t)part * n; m < L; m += dm, t += s) {
                const T f = (sh && (t & 1)) ? -wn : wn;
                const T nr = f * P.x, ni = f * P.y, sr = two ? f * P.z : (T)0, si = two ? f * P.w : (T)0;
                const int64_t idx = m * stride + col;
                const Q4 b = rhs_map[idx];
                out[idx] = Q4{nr + sr - b.x, ni + si - b.y, nr - sr - b.z, ni - si - b.w};
            }
        } else if (part == 0 && 2 * k <= n) {
            const int64_t base = (c - cbeg) * (4 * nside - 1);
            spec[(base + north_ring(j)) * sstride + k] = make2<T2, T>(P.x, P.y);
            if (two) spec[(base + south_ring(nside, j)) * sstride + k] = make2<T2, T>(P.z, P.w);
        }
    };
    auto finish = [&](int p, const Q4 &A, const Q4 &B) {
        if (p == 0) {
            const Q4 z = src[0];
            emit(0, Q4{z.x + 2 * A.x, z.y, z.z + 2 * A.z, z.w});
        } else if (2 * p == n) {
            emit(p, Q4{A.x + sigma * A.x, A.y - sigma * A.y, A.z + sigma * A.z, A.w - sigma * A.w});
        } else {
            emit(p, Q4{A.x + sigma * B.x, A.y - sigma * B.y, A.z + sigma * B.z, A.w - sigma * B.w});
            if (RESIDUAL)
                emit(n - p, Q4{B.x + sigma * A.x, B.y - sigma * A.y, B.z + sigma * A.z, B.w - sigma * A.w});
        }
    };

    const int p0 = q / s;
    if (s > 1 && ok && p0 < np) {
        Q4 A, B;
        pair_sums(p0, A, B);
        pa[threadIdx.x] = A;
        pb[threadIdx.x] = B;
    }
    __syncthreads();
    if (!ok) return;
    if (s > 1) {
        if (p0 >= np) return;
        Q4 A{0, 0, 0, 0}, B{0, 0, 0, 0};
        for (int u = 0; u < s; ++u) {
            const int e = (p0 * s + u) * J + (int)(threadIdx.x % J);
            const Q4 a = pa[e], b = pb[e];
            A.x += a.x; A.y += a.y; A.z += a.z; A.w += a.w;
            B.x += b.x; B.y += b.y; B.z += b.z; B.w += b.w;
        }
        finish(p0, A, B);
    } else {
        for (int p = p0; p < np; p += Q) {
            Q4 A, B;
            pair_sums(p, A, B);
            finish(p, A, B);
        }
    }
}

// ---------------------------------------------------------------- synthesis

template <typename T>
__global__ void __launch_bounds__(512) k_ring_synthesis(int64_t nside, int64_t L, int64_t ncomp,
                                                        const T *__restrict__ syn,
                                                        const void *__restrict__ twall,
                                                        int64_t twcnt,
                                                        const uint8_t *__restrict__ shifted,
                                                        double *__restrict__ maps, int hcap,
                                                        int bsmin)
{
    using T2 = typename vec2<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int64_t r = blockIdx.x, c = blockIdx.y;
    const int64_t npix = 12 * nside * nside, nlanes = 2 * nside;
    const int n = (int)ring_nphi(nside, r), h = n / 2;
    if (ring_big(h, hcap, (int)nside, bsmin)) return;   // left to k_ring_synthesis_big
    const int64_t off = ring_offset(nside, r);
    const bool south = r >= nlanes;
    const int64_t j = south ? 4 * nside - 2 - r : r;
    const bool sh = shifted[r] != 0;
    T2 *A = reinterpret_cast<T2 *>(smem_raw);
    T2 *B = A + hcap;
    const T2 *tw = TwTable<T2>::get(twall, twcnt) + twiddle_offset(n);
    T2 cpi;   // e^{-i pi / n}
    {
        double s1, c1d;
        sincospi(-1.0 / (double)n, &s1, &c1d);
        cpi.x = (T)c1d;
        cpi.y = (T)s1;
    }
    // Fold into the n-periodic spectrum C_k = e^{i pi s k / n} P_k and build
    // Z'[k] = (C_k + C_{k+h}) + i (C_k - C_{k+h}) omega_n^{-k}, k < h.
    const T *base = syn + (south ? 2 : 0);
    for (int k = threadIdx.x; k < h; k += blockDim.x) {
        T c0[2], c1[2], dummy[2];
        residue_sums(base, L, nlanes, ncomp, j, c, k, n, sh, false, c0, dummy);
        residue_sums(base, L, nlanes, ncomp, j, c, k + h, n, sh, false, c1, dummy);
        T2 ck = make2<T2, T>(c0[0], c0[1]);
        T2 ckh = make2<T2, T>(c1[0], c1[1]);
        if (sh) {
            // e^{i pi k / n} and e^{i pi (k + h) / n}
            ck = cmul(ck, phase_pi(tw, h, k, cpi, +1));
            ckh = cmul(ckh, phase_pi(tw, h, k + h, cpi, +1));
        }
        T2 sum = cadd(ck, ckh);
        T2 dif = cmul(csub(ck, ckh), twiddle_n(tw, h, k, +1));
        T2 z;
        z.x = sum.x - dif.y;
        z.y = sum.y + dif.x;
        A[k] = z;
    }
    __syncthreads();
    T2 *Z = fft_shared(A, B, h, tw, +1);
    double *dst = maps + c * npix + off;
    for (int t = threadIdx.x; t < h; t += blockDim.x) {
        T2 z = Z[t];
        dst[2 * t] = (double)z.x;
        dst[2 * t + 1] = (double)z.y;
    }
}


// Inverse ring transform from the folded spectra of k_fold_lanes: one CTA per (ring, block of
// cpc components), with the rings and buffers of k_ring_forward.
// With the fold before it: 2.22 -> 0.75 ms for a (Q, U) pair at Nside 1024 (a ring per CTA reading
// its coefficients 128 lanes apart and taking prime factors up to 1021 as one radix), 180 -> 65
// us for one FP64 map at Nside 256.
template <typename T, bool BS>
__global__ void __launch_bounds__(512) k_ring_inverse(int64_t nside, int64_t ncomp, int cpc, int64_t sstride,
                                                      const typename vec2<T>::type *__restrict__ spec,
                                                      const void *__restrict__ twall, int64_t twcnt,
                                                      const uint8_t *__restrict__ shifted, double *__restrict__ maps,
                                                      int64_t cbeg, int64_t i0, int64_t cnt, int mcap, int hcap,
                                                      int bsmin, int buf)
{
    using T2 = typename vec2<T>::type;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int64_t nring = 4 * nside - 1, npix = 12 * nside * nside;
    const int64_t r = launch_ring(nside, i0, cnt, blockIdx.y);
    const int n = (int)ring_nphi(nside, r), h = n / 2;
    const bool bs = BS && use_bluestein(h, mcap);
    if (hcap > 0 && ring_big(h, hcap, (int)nside, bsmin)) return;   // left to k_ring_synthesis_big
    const int64_t off = ring_offset(nside, r);
    const bool sh = shifted[r] != 0;
    T2 *b0 = reinterpret_cast<T2 *>(smem_raw), *b1 = b0 + buf, *b2 = b1 + buf;
    const T2 *twT = TwTable<T2>::get(twall, twcnt);
    const T2 *tw = twT + twiddle_offset(n);
    const int M = bs ? next_pow2(2 * h - 1) : 0;
    const T2 *twM = bs ? twT + twiddle_offset(M) : nullptr;
    T2 *FB = nullptr, *X = b0, *Y = b1;
    if (bs) {
        FB = bs_filter(h, n, M, tw, twM, +1, b0, b1);
        X = FB == b0 ? b1 : b0;
        Y = b2;
    }
    T2 cpi;   // e^{-i pi / n}
    {
        double s1, c1d;
        sincospi(-1.0 / (double)n, &s1, &c1d);
        cpi = make2<T2, T>((T)c1d, (T)s1);
    }
    const int64_t cend = (int64_t)(blockIdx.x + 1) * cpc < ncomp ? (int64_t)(blockIdx.x + 1) * cpc : ncomp;
    for (int64_t c = (int64_t)blockIdx.x * cpc; c < cend; ++c) {
        const T2 *P = spec + (c * nring + r) * sstride;
        // Z'[k] = (C_k + C_{k+h}) + i (C_k - C_{k+h}) omega_n^{-k}, C_k = e^{i pi s k / n} P_k and
        // C_{k+h} = conj C_{h-k} for k > 0
        for (int k = threadIdx.x; k < h; k += blockDim.x) {
            T2 ck = P[k], ch = P[h - k];
            if (sh) {
                ck = cmul(ck, phase_pi(tw, h, k, cpi, +1));
                ch = cmul(ch, phase_pi(tw, h, h - k, cpi, +1));
            }
            if (k > 0) ch = cconj(ch);
            const T2 sum = cadd(ck, ch);
            const T2 dif = cmul(csub(ck, ch), twiddle_n(tw, h, k, +1));
            T2 z = make2<T2, T>(sum.x - dif.y, sum.y + dif.x);
            if (bs) z = cmul(z, bs_chirp(tw, h, n, k, +1));
            X[k] = z;
        }
        __syncthreads();
        const T2 *Z = bs ? bs_apply(X, Y, FB, h, n, M, tw, twM, +1) : fft_shared(X, Y, h, tw, +1);
        double2 *dst = reinterpret_cast<double2 *>(maps + (cbeg + c) * npix + off);
        for (int t = threadIdx.x; t < h; t += blockDim.x) {
            const T2 z = Z[t];
            dst[t] = make_double2((double)z.x, (double)z.y);
        }
        __syncthreads();
    }
}

// ---------------------------------------------------------------- rings beyond shared memory
//
// One persistent CTA per slot of the global scratch (three buffers of Mmax complex floats
// each) walks the rings; only the rings of ring_big are transformed, with the arithmetic of
// the shared-memory kernels: a Stockham FFT of length h, or Bluestein's method with a
// power-of-two length M.  __syncthreads orders the CTA's global-memory accesses.

// T = float: three buffers of Mmax complex floats per slot (Bluestein rings included).
// T = double: no Bluestein path here (the FP64 shared-memory kernels have one up to M = 4096; the
// mixed-radix FFT takes every ring that is too long for them); two buffers of 2 nside complex
// doubles per slot, which fit the same slot bytes (64 nside <= 96 nside).
template <typename T, typename Tin>
__global__ void __launch_bounds__(512) k_ring_analysis_big(int64_t nside, int64_t L, int64_t ncomp,
                                                           const Tin *__restrict__ maps,
                                                           const double *__restrict__ mask,
                                                           const void *__restrict__ twall,
                                                           int64_t twcnt,
                                                           const uint8_t *__restrict__ shifted,
                                                           typename vec2<T>::type *__restrict__ out,
                                                           int hcap, int bsmin, void *__restrict__ gscratch,
                                                           int64_t slot_bytes)
{
    using T2 = typename vec2<T>::type;
    constexpr bool kSingle = std::is_same<T, float>::value;
    const int64_t nring = 4 * nside - 1, npix = 12 * nside * nside;
    T2 *b0 = reinterpret_cast<T2 *>(static_cast<unsigned char *>(gscratch) + blockIdx.x * slot_bytes);
    const int64_t bstride = kSingle ? 4 * nside : 2 * nside;
    T2 *b1 = b0 + bstride, *b2 = b1 + bstride;
    const T2 *twT = TwTable<T2>::get(twall, twcnt);
    const T w = (T)(4.0 * M_PI / (double)npix);
    for (int64_t r = blockIdx.x; r < nring; r += gridDim.x) {
        const int n = (int)ring_nphi(nside, r), h = n / 2;
        if (!ring_big(h, hcap, (int)nside, bsmin)) continue;
        const int64_t off = ring_offset(nside, r);
        const T2 *tw = twT + twiddle_offset(n);
        const bool sh = shifted[r] != 0;
        if constexpr (kSingle) {
            const bool bs = bluestein_big(h, (int)nside, bsmin);
            const int M = bs ? next_pow2(2 * h - 1) : 0;
            const float2 *twM = bs ? twT + twiddle_offset(M) : nullptr;
            float2 *FB = nullptr, *X = b0, *Y = b1;
            if (bs) {
                FB = bs_filter(h, n, M, tw, twM, -1, b0, b1);
                X = (FB == b0) ? b1 : b0;
                Y = b2;
            }
            for (int64_t c = 0; c < ncomp; ++c) {
                float2 *Z;
                if (bs) {
                    load_ring<float>(maps + c * npix + off, mask ? mask + off : nullptr, false, h, X,
                                     [&](int t, float2 z) { return cmul(z, bs_chirp(tw, h, n, t, -1)); });
                    __syncthreads();
                    Z = bs_apply(X, Y, FB, h, n, M, tw, twM, -1);
                } else {
                    load_ring<float>(maps + c * npix + off, mask ? mask + off : nullptr, false, h, X,
                                     [](int, float2 z) { return z; });
                    __syncthreads();
                    Z = fft_shared(X, Y, h, tw, -1);
                }
                ring_outputs<float>(Z, n, L, tw, sh, w, out + (c * nring + r) * L);
                __syncthreads();
            }
        } else {
            for (int64_t c = 0; c < ncomp; ++c) {
                load_ring<T>(maps + c * npix + off, mask ? mask + off : nullptr, false, h, b0,
                             [](int, T2 z) { return z; });
                __syncthreads();
                T2 *Z = fft_shared(b0, b1, h, tw, -1);
                ring_outputs<T>(Z, n, L, tw, sh, w, out + (c * nring + r) * L);
                __syncthreads();
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(512) k_ring_synthesis_big(int64_t nside, int64_t L, int64_t ncomp,
                                                            const T *__restrict__ syn,
                                                            const void *__restrict__ twall,
                                                            int64_t twcnt,
                                                            const uint8_t *__restrict__ shifted,
                                                            double *__restrict__ maps, int hcap,
                                                            int bsmin, void *__restrict__ gscratch,
                                                            int64_t slot_bytes)
{
    using T2 = typename vec2<T>::type;
    constexpr bool kSingle = std::is_same<T, float>::value;
    const int64_t nring = 4 * nside - 1, npix = 12 * nside * nside, nlanes = 2 * nside;
    T2 *b0 = reinterpret_cast<T2 *>(static_cast<unsigned char *>(gscratch) + blockIdx.x * slot_bytes);
    const int64_t bstride = kSingle ? 4 * nside : 2 * nside;
    T2 *b1 = b0 + bstride, *b2 = b1 + bstride;
    const T2 *twT = TwTable<T2>::get(twall, twcnt);
    for (int64_t r = blockIdx.x; r < nring; r += gridDim.x) {
        const int n = (int)ring_nphi(nside, r), h = n / 2;
        if (!ring_big(h, hcap, (int)nside, bsmin)) continue;
        const int64_t off = ring_offset(nside, r);
        const bool south = r >= nlanes;
        const int64_t j = south ? 4 * nside - 2 - r : r;
        const bool sh = shifted[r] != 0;
        const T2 *tw = twT + twiddle_offset(n);
        T2 cpi;
        {
            double s1, c1d;
            sincospi(-1.0 / (double)n, &s1, &c1d);
            cpi = make2<T2, T>((T)c1d, (T)s1);
        }
        bool bs = false;
        int M = 0;
        const T2 *twM = nullptr;
        T2 *FB = nullptr, *X = b0, *Y = b1;
        if constexpr (kSingle) {
            bs = bluestein_big(h, (int)nside, bsmin);
            M = bs ? next_pow2(2 * h - 1) : 0;
            twM = bs ? twT + twiddle_offset(M) : nullptr;
            if (bs) {
                FB = bs_filter(h, n, M, tw, twM, +1, b0, b1);
                X = (FB == b0) ? b1 : b0;
                Y = b2;
            }
        }
        const T *base = syn + (south ? 2 : 0);
        for (int64_t c = 0; c < ncomp; ++c) {
            for (int k = threadIdx.x; k < h; k += blockDim.x) {
                T c0[2], c1[2], dummy[2];
                residue_sums(base, L, nlanes, ncomp, j, c, k, n, sh, false, c0, dummy);
                residue_sums(base, L, nlanes, ncomp, j, c, k + h, n, sh, false, c1, dummy);
                T2 ck = make2<T2, T>(c0[0], c0[1]);
                T2 ckh = make2<T2, T>(c1[0], c1[1]);
                if (sh) {
                    ck = cmul(ck, phase_pi(tw, h, k, cpi, +1));
                    ckh = cmul(ckh, phase_pi(tw, h, k + h, cpi, +1));
                }
                const T2 sum = cadd(ck, ckh);
                const T2 dif = cmul(csub(ck, ckh), twiddle_n(tw, h, k, +1));
                T2 z = make2<T2, T>(sum.x - dif.y, sum.y + dif.x);
                if constexpr (kSingle) {
                    if (bs) z = cmul(z, bs_chirp(tw, h, n, k, +1));
                }
                X[k] = z;
            }
            __syncthreads();
            T2 *Z;
            if constexpr (kSingle) Z = bs ? bs_apply(X, Y, FB, h, n, M, tw, twM, +1) : fft_shared(X, Y, h, tw, +1);
            else Z = fft_shared(X, Y, h, tw, +1);
            double *dst = maps + c * npix + off;
            for (int t = threadIdx.x; t < h; t += blockDim.x) {
                const T2 z = Z[t];
                dst[2 * t] = (double)z.x;
                dst[2 * t + 1] = (double)z.y;
            }
            __syncthreads();
        }
    }
}

}  // namespace gm

using namespace gm;

extern "C" int64_t gm_ring_twiddle_count(int64_t nside) { return nside * (nside + 1); }

extern "C" int gm_ring_twiddles(int64_t nside, void *tw, void *stream)
{
    if (nside < 1 || nside > 8192) return GM_ERR_BAD_SHAPE;
    if (!tw) return GM_ERR_BAD_PTR;
    int64_t cnt = gm_ring_twiddle_count(nside);
    double2 *t64 = reinterpret_cast<double2 *>(tw);
    float2 *t32 = reinterpret_cast<float2 *>(t64 + cnt);
    int64_t gx = (2 * nside + 255) / 256;
    if (gx > 64) gx = 64;
    k_twiddles<<<dim3((unsigned)gx, (unsigned)nside), 256, 0, as_stream(stream)>>>(nside, t64, t32);
    return check_launch("gm_ring_twiddles");
}

static size_t ring_smem_bytes(int precision, int64_t nside)
{
    size_t elem = precision == GM_FP64 ? sizeof(double2) : sizeof(float2);
    return 2 * (size_t)(2 * nside) * elem;
}

static int ring_shape_ok(int precision, int64_t nside, int64_t L, int64_t ncomp)
{
    if (nside < 1 || L < 1 || ncomp < 1 || ncomp > 65535) return 0;
    if (ring_smem_bytes(precision, nside) > 227 * 1024) return 0;
    return 1;
}

// Most dynamic shared memory of the ring kernels: 227 KB less their static arrays.
constexpr int kRingSmem = 227 * 1024 - 336;

// Shared memory of the ring kernels: ping-pong buffers of hcap complex values.
static int ring_hcap(int precision, int64_t nside, bool big)
{
    const size_t elem = precision == GM_FP64 ? sizeof(double2) : sizeof(float2);
    // 227 KB of dynamic shared memory per block, less 1 KB left to the kernels' static arrays
    const int64_t fit = (int64_t)((227 * 1024 - 1024) / (2 * elem));
    const int64_t h = 2 * nside;
    return (int)(big && h > fit ? fit : h);
}

extern "C" int64_t gm_ring_big_scratch_bytes(int64_t nside, int64_t nslots)
{
    return nside < 1 || nslots < 1 ? 0 : nslots * 3 * 4 * nside * (int64_t)sizeof(float2);
}

// Whether some ring goes to the *_big kernels (ring_big of the longest ring).
static bool any_ring_big(int64_t nside, int hcap, int bsmin)
{
    return 2 * nside > hcap || (bsmin > 0 && next_pow2((int)(4 * nside - 1)) > bsmin);
}

// The launches of the ring kernels: the belt (length 4 nside) and the caps by powers of two of their
// length; all rings up to Nside 128 in one.  run(i0, cnt, rows, buf, buffers, threads, cpc, mcap):
// cap rings i0 .. i0 + cnt - 1 of both hemispheres, then the belt where rows says so; buf complex
// values in each of 2 buffers (3 with Bluestein rings, whose M fits buf).  The longest caps, where
// none takes Bluestein, share the belt's launch: longest first, the belt fills up behind their
// direct sums over primes (one FP64 map at Nside 2048: 8.6 -> 6.8 ms).  Threads: an eighth of the
// points where the rings of all components fill the chip many times over (64 maps at Nside 512:
// 5.5 -> 3.6 ms), else two to four times as many, for the latency of a ring (one FP64 map at Nside
// 256: 66 us with an eighth, 53 us).  cpc components of a CTA share the transform of the chirp
// where that leaves two rounds of CTAs (eight everywhere: 16 maps at Nside 64 78 us, 21 here).
template <typename T, typename Run>
static int for_ring_classes(int64_t nside, int64_t ncomp, int hcap, bool big, Run run)
{
    int mcap = bluestein_mcap(nside);
    if (sizeof(T) == 8 && mcap > 4096) mcap = 4096;   // three buffers of M in 227 KB
    auto one = [&](int64_t i0, int64_t cnt, bool belt, int hmax, int M) {
        if (big && hmax > hcap) hmax = hcap;          // longer rings go to the *_big kernels
        const int buf = M > hmax ? M : hmax;
        const int64_t rows = 2 * cnt + (belt ? 2 * nside + 1 : 0);
        int threads = rows * ncomp >= 148 * 64 ? buf / 8 : (M ? buf / 4 : buf / 2);
        threads = threads >= 512 ? 512 : (threads >= 256 ? 256 : (threads >= 128 ? 128 : 64));
        int cpc = 1;
        if (M) {
            const int64_t room = kRingSmem / (3 * (int64_t)buf * 2 * sizeof(T)), cap = 2048 / threads;
            const int64_t fill = rows * ncomp / (2 * 148 * (room < cap ? room : cap));
            cpc = fill < 1 ? 1 : (fill < 8 ? (int)fill : 8);
        }
        return run(i0, cnt, rows, buf, M ? 3 : 2, threads, cpc, M ? mcap : 0);
    };
    // M of the caps lo .. top (one power of two above the first class), 0 without Bluestein rings
    auto caps_M = [&](int64_t lo, int64_t top) {
        // rings of up to 512 pixels on a full chip: direct FP64 sums over primes up to 127 cost less
        // than three transforms of 512 points (64 maps at Nside 128: 380 -> 279 us)
        if (sizeof(T) == 8 && top <= 128 && (4 * nside - 1) * ncomp >= 148 * 64) return 0;
        const int64_t first = lo > kDirectPrime ? lo : kDirectPrime + 1;
        if (first > top || next_pow2((int)(4 * first - 1)) > mcap) return 0;
        const int M = next_pow2((int)(4 * top - 1));
        return M < mcap ? M : mcap;
    };
    const int hb = (int)(2 * nside), Mb = use_bluestein(hb, mcap) ? next_pow2(2 * hb - 1) : 0;
    if (nside <= 128) {
        const int M = caps_M(1, nside - 1);
        return one(1, nside - 1, true, hb, M > Mb ? M : Mb);
    }
    int64_t hi = 128;
    while (2 * hi < nside - 1) hi *= 2;
    const bool joint = Mb == 0 && caps_M(hi + 1, nside - 1) == 0;   // the last class and the belt
    int st = joint ? GM_OK : one(1, 0, true, hb, Mb);
    for (int64_t lo = 1, h = 128; st == GM_OK && lo < nside; lo = h + 1, h *= 2) {
        const int64_t top = h < nside - 1 ? h : nside - 1;
        const bool last = joint && top == nside - 1;
        st = one(lo, top - lo + 1, last, last ? hb : (int)(2 * top), caps_M(lo, top));
    }
    return st;
}

template <typename T, typename Tin>
static int ring_analysis(int64_t nside, int64_t L, int64_t ncomp, const void *maps, const double *mask, const void *tw,
                         const uint8_t *shifted, void *ringspec, int hcap, int bsmin, bool big, void *scratch,
                         int64_t slot, int64_t nslots, cudaStream_t s)
{
    using T2 = typename vec2<T>::type;
    const int64_t twcnt = gm_ring_twiddle_count(nside), nring = 4 * nside - 1;
    const bool vec = reinterpret_cast<uintptr_t>(maps) % (2 * sizeof(Tin)) == 0 && reinterpret_cast<uintptr_t>(mask) % 16 == 0;
    int st = for_ring_classes<T>(nside, ncomp, hcap, big, [&](int64_t i0, int64_t cnt, int64_t rows, int buf, int nbuf,
                                                              int threads, int cpc, int mcap) {
        const size_t bytes = (size_t)nbuf * buf * sizeof(T2);
        auto kernel = nbuf == 3 ? k_ring_forward<T, Tin, true> : k_ring_forward<T, Tin, false>;
        const int e = allow_smem(kernel, kRingSmem, "gm_ring_analysis attr");
        if (e) return e;
        dim3 grid((unsigned)((ncomp + cpc - 1) / cpc), (unsigned)rows);
        kernel<<<grid, threads, bytes, s>>>(nside, L, ncomp, cpc, (const Tin *)maps, mask, vec, tw, twcnt,
                                                            shifted, (T2 *)ringspec, i0, cnt, mcap, big ? hcap : 0, bsmin,
                                                            buf);
        return check_launch("gm_ring_analysis");
    });
    if (st || !big) return st;
    const unsigned gbig = (unsigned)(nslots < nring ? nslots : nring);
    k_ring_analysis_big<T, Tin><<<gbig, 512, 0, s>>>(nside, L, ncomp, (const Tin *)maps, mask, tw, twcnt, shifted,
                                                     (T2 *)ringspec, hcap, bsmin, scratch, slot);
    return check_launch("gm_ring_analysis");
}

extern "C" int gm_ring_analysis_ws(int precision, int64_t nside, int64_t L, int64_t ncomp,
                                   const void *maps, int map_dtype_bytes, const double *mask,
                                   const void *tw, const uint8_t *shifted, void *ringspec,
                                   void *scratch, int64_t scratch_bytes, int64_t hcap_max,
                                   int64_t bs_min, void *stream)
{
    const bool ws = scratch != nullptr;
    if (nside < 1 || nside > 8192 || L < 1 || ncomp < 1 || ncomp > 65535) return GM_ERR_BAD_SHAPE;
    if (!ws && !ring_shape_ok(precision, nside, L, ncomp)) return GM_ERR_BAD_SHAPE;
    if (!maps || !tw || !shifted || !ringspec) return GM_ERR_BAD_PTR;
    if (map_dtype_bytes != 8 && map_dtype_bytes != 4) return GM_ERR_UNSUPPORTED;
    if (precision != GM_FP64 && precision != GM_MIXED) return GM_ERR_UNSUPPORTED;
    const int64_t slot = gm_ring_big_scratch_bytes(nside, 1), nslots = ws ? scratch_bytes / slot : 0;
    if (ws && nslots < 1) return GM_ERR_BAD_SHAPE;
    int hcap = ring_hcap(precision, nside, ws);
    if (ws && hcap_max > 0 && hcap_max < hcap) hcap = (int)hcap_max;
    // single precision only: FP64 has no Bluestein path in global memory
    const int bsmin = ws && precision == GM_MIXED ? (bs_min > 0 ? (int)bs_min : 8192) : 0;
    const bool big = ws && any_ring_big(nside, hcap, bsmin);
    cudaStream_t s = as_stream(stream);
#define GM_RING(T, TIN)                                                                                           \
    return ring_analysis<T, TIN>(nside, L, ncomp, maps, mask, tw, shifted, ringspec, hcap, bsmin, big, scratch,   \
                                 slot, nslots, s)
    if (precision == GM_FP64) {
        if (map_dtype_bytes == 8) GM_RING(double, double);
        GM_RING(double, float);
    }
    if (map_dtype_bytes == 8) GM_RING(float, double);
    GM_RING(float, float);
#undef GM_RING
}

extern "C" int gm_ring_analysis(int precision, int64_t nside, int64_t L, int64_t ncomp,
                                const void *maps, int map_dtype_bytes, const double *mask,
                                const void *tw, const uint8_t *shifted, void *ringspec,
                                void *stream)
{
    return gm_ring_analysis_ws(precision, nside, L, ncomp, maps, map_dtype_bytes, mask, tw, shifted,
                               ringspec, nullptr, 0, 0, 0, stream);
}

extern "C" int gm_pack_rhs(int precision, int64_t nside, int64_t L, int64_t ncomp,
                           const void *ringspec, void *rhs, void *stream)
{
    if (nside < 1 || L < 1 || ncomp < 1 || ncomp > 65535) return GM_ERR_BAD_SHAPE;
    if (!ringspec || !rhs) return GM_ERR_BAD_PTR;
    const int64_t nlanes = 2 * nside;
    dim3 grid((unsigned)((L + 31) / 32), (unsigned)((nlanes + 31) / 32), (unsigned)ncomp);
    dim3 block(32, 8);
    cudaStream_t s = as_stream(stream);
    if (precision == GM_FP64)
        k_pack_rhs<double><<<grid, block, 0, s>>>(nside, L, ncomp, (const double2 *)ringspec,
                                                  (double *)rhs);
    else if (precision == GM_MIXED)
        k_pack_rhs<float><<<grid, block, 0, s>>>(nside, L, ncomp, (const float2 *)ringspec,
                                                 (float *)rhs);
    else
        return GM_ERR_UNSUPPORTED;
    return check_launch("gm_pack_rhs");
}

// Columns per CTA: eight (a full 128-byte line a row in single precision) where that leaves two
// CTAs per SM, else two.
template <typename T, bool RESIDUAL, bool WIDE = true>
static void fold_lanes(int64_t nside, int64_t L, int64_t ncomp, int64_t cbeg, int64_t cw, const void *syn,
                       const void *rhs_map, const uint8_t *shifted, void *out, void *spec, int64_t sstride,
                       cudaStream_t s)
{
    using T2 = typename vec2<T>::type;
    const int64_t items = 2 * nside * cw;
    auto run = [&](auto kernel, int J) {
        kernel<<<(unsigned)((items + J - 1) / J), fold_threads(J), 0, s>>>(
            nside, L, ncomp, cbeg, cw, (const Quad<T, WIDE> *)syn, (const Quad<T, WIDE> *)rhs_map, shifted,
            (Quad<T, WIDE> *)out, (T2 *)spec, sstride);
    };
    if (items >= 8 * 296) run(k_fold_lanes<T, 8, RESIDUAL, WIDE>, 8);
    else run(k_fold_lanes<T, 2, RESIDUAL, WIDE>, 2);
}

extern "C" int gm_fold_residual(int precision, int64_t nside, int64_t L, int64_t ncomp,
                                const void *syn, const void *rhs_map, const uint8_t *shifted,
                                void *rhs_out, void *stream)
{
    if (nside < 1 || L < 1 || ncomp < 1 || ncomp > 65535) return GM_ERR_BAD_SHAPE;
    if (!syn || !rhs_map || !shifted || !rhs_out) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    const bool wide = ((reinterpret_cast<uintptr_t>(syn) | reinterpret_cast<uintptr_t>(rhs_map) |
                        reinterpret_cast<uintptr_t>(rhs_out)) & 15) == 0;
    auto run = [&](auto fold) { fold(nside, L, ncomp, 0, ncomp, syn, rhs_map, shifted, rhs_out, nullptr, 0, s); };
    if (precision == GM_FP64) run(wide ? fold_lanes<double, true, true> : fold_lanes<double, true, false>);
    else if (precision == GM_MIXED) run(wide ? fold_lanes<float, true, true> : fold_lanes<float, true, false>);
    else return GM_ERR_UNSUPPORTED;
    return check_launch("gm_fold_residual");
}

extern "C" int gm_ring_synthesis_ws(int precision, int64_t nside, int64_t L, int64_t ncomp,
                                    const void *syn, const void *tw, const uint8_t *shifted,
                                    double *maps, void *scratch, int64_t scratch_bytes,
                                    int64_t hcap_max, int64_t bs_min, void *stream)
{
    const bool big = scratch != nullptr;
    if (nside < 1 || nside > 8192 || L < 1 || ncomp < 1 || ncomp > 65535) return GM_ERR_BAD_SHAPE;
    if (!big && !ring_shape_ok(precision, nside, L, ncomp)) return GM_ERR_BAD_SHAPE;
    if (!syn || !tw || !shifted || !maps) return GM_ERR_BAD_PTR;
    const int64_t nslots = big ? scratch_bytes / gm_ring_big_scratch_bytes(nside, 1) : 0;
    if (big && nslots < 1) return GM_ERR_BAD_SHAPE;
    const int64_t nring = 4 * nside - 1, cnt = gm_ring_twiddle_count(nside);
    int hcap = ring_hcap(precision, nside, big);
    if (big && hcap_max > 0 && hcap_max < hcap) hcap = (int)hcap_max;
    const int bsmin = big && precision == GM_MIXED ? (bs_min > 0 ? (int)bs_min : 8192) : 0;
    const size_t smem = 2 * (size_t)hcap * (precision == GM_FP64 ? sizeof(double2) : sizeof(float2));
    const int64_t slot = gm_ring_big_scratch_bytes(nside, 1);
    const unsigned gbig = (unsigned)(nslots < nring ? nslots : nring);
    int threads = nside >= 256 ? 512 : 128;
    dim3 grid((unsigned)nring, (unsigned)ncomp);
    cudaStream_t s = as_stream(stream);
    int st;
    if (precision == GM_FP64) {
        if ((st = allow_smem(k_ring_synthesis<double>, kRingSmem, "gm_ring_synthesis attr"))) return st;
        k_ring_synthesis<double><<<grid, threads, smem, s>>>(nside, L, ncomp, (const double *)syn,
                                                             tw, cnt, shifted, maps, hcap, 0);
        if (big)
            k_ring_synthesis_big<double><<<gbig, 512, 0, s>>>(nside, L, ncomp, (const double *)syn, tw, cnt,
                                                              shifted, maps, hcap, 0, scratch, slot);
    } else if (precision == GM_MIXED) {
        if ((st = allow_smem(k_ring_synthesis<float>, kRingSmem, "gm_ring_synthesis attr"))) return st;
        k_ring_synthesis<float><<<grid, threads, smem, s>>>(nside, L, ncomp, (const float *)syn,
                                                            tw, cnt, shifted, maps, hcap, bsmin);
        if (big)
            k_ring_synthesis_big<float><<<gbig, 512, 0, s>>>(nside, L, ncomp, (const float *)syn, tw, cnt,
                                                             shifted, maps, hcap, bsmin, scratch, slot);
    } else {
        return GM_ERR_UNSUPPORTED;
    }
    return check_launch("gm_ring_synthesis");
}

extern "C" int gm_ring_synthesis(int precision, int64_t nside, int64_t L, int64_t ncomp,
                                 const void *syn, const void *tw, const uint8_t *shifted,
                                 double *maps, void *stream)
{
    return gm_ring_synthesis_ws(precision, nside, L, ncomp, syn, tw, shifted, maps, nullptr, 0, 0, 0,
                                stream);
}

extern "C" int64_t gm_ring_fold_bytes(int precision, int64_t nside)
{
    if (nside < 1) return 0;
    return (4 * nside - 1) * (2 * nside + 1) * (int64_t)(precision == GM_FP64 ? sizeof(double2) : sizeof(float2));
}

template <typename T>
static int ring_synthesis_fold(int64_t nside, int64_t L, int64_t ncomp, const void *syn, const void *tw,
                               const uint8_t *shifted, double *maps, void *work, int64_t chunk, int hcap, int bsmin,
                               bool big, cudaStream_t s)
{
    using T2 = typename vec2<T>::type;
    const int64_t cnt = gm_ring_twiddle_count(nside), sstride = 2 * nside + 1;
    for (int64_t c0 = 0; c0 < ncomp; c0 += chunk) {
        const int64_t cw = ncomp - c0 < chunk ? ncomp - c0 : chunk;
        fold_lanes<T, false>(nside, L, ncomp, c0, cw, syn, nullptr, shifted, nullptr, work, sstride, s);
        int st = check_launch("gm_ring_synthesis_fold");
        if (st) return st;
        st = for_ring_classes<T>(nside, cw, hcap, big, [&](int64_t i0, int64_t n, int64_t rows, int buf, int nbuf,
                                                           int threads, int cpc, int mcap) {
            const size_t bytes = (size_t)nbuf * buf * sizeof(T2);
            auto kernel = nbuf == 3 ? k_ring_inverse<T, true> : k_ring_inverse<T, false>;
            const int e = allow_smem(kernel, kRingSmem, "gm_ring_synthesis_fold attr");
            if (e) return e;
            dim3 grid((unsigned)((cw + cpc - 1) / cpc), (unsigned)rows);
            kernel<<<grid, threads, bytes, s>>>(nside, cw, cpc, sstride, (const T2 *)work, tw, cnt, shifted, maps,
                                                           c0, i0, n, mcap, big ? hcap : 0, bsmin, buf);
            return check_launch("gm_ring_synthesis_fold");
        });
        if (st) return st;
    }
    return GM_OK;
}

extern "C" int gm_ring_synthesis_fold(int precision, int64_t nside, int64_t L, int64_t ncomp, const void *syn,
                                      const void *tw, const uint8_t *shifted, double *maps, void *work,
                                      int64_t work_bytes, void *scratch, int64_t scratch_bytes, int64_t hcap_max,
                                      int64_t bs_min, void *stream)
{
    if (nside < 1 || nside > 8192 || L < 1 || ncomp < 1 || ncomp > 65535) return GM_ERR_BAD_SHAPE;
    if (precision != GM_FP64 && precision != GM_MIXED) return GM_ERR_UNSUPPORTED;
    if (!syn || !tw || !shifted || !maps || !work || !scratch) return GM_ERR_BAD_PTR;
    if ((reinterpret_cast<uintptr_t>(maps) | reinterpret_cast<uintptr_t>(syn) | reinterpret_cast<uintptr_t>(work)) & 15)
        return GM_ERR_BAD_PTR;
    const int64_t per = gm_ring_fold_bytes(precision, nside), chunk = work_bytes / per;
    const int64_t slot = gm_ring_big_scratch_bytes(nside, 1), nslots = scratch_bytes / slot;
    if (chunk < 1 || nslots < 1) return GM_ERR_BAD_SHAPE;
    int hcap = ring_hcap(precision, nside, true);
    if (hcap_max > 0 && hcap_max < hcap) hcap = (int)hcap_max;
    const int bsmin = precision == GM_MIXED ? (bs_min > 0 ? (int)bs_min : 8192) : 0;
    const bool big = any_ring_big(nside, hcap, bsmin);
    cudaStream_t s = as_stream(stream);
    const int st = precision == GM_FP64
                       ? ring_synthesis_fold<double>(nside, L, ncomp, syn, tw, shifted, maps, work, chunk, hcap, bsmin, big, s)
                       : ring_synthesis_fold<float>(nside, L, ncomp, syn, tw, shifted, maps, work, chunk, hcap, bsmin, big, s);
    if (st || !big) return st;
    const int64_t nring = 4 * nside - 1, cnt = gm_ring_twiddle_count(nside);
    const unsigned gbig = (unsigned)(nslots < nring ? nslots : nring);
    if (precision == GM_FP64)
        k_ring_synthesis_big<double><<<gbig, 512, 0, s>>>(nside, L, ncomp, (const double *)syn, tw, cnt, shifted, maps,
                                                          hcap, 0, scratch, slot);
    else
        k_ring_synthesis_big<float><<<gbig, 512, 0, s>>>(nside, L, ncomp, (const float *)syn, tw, cnt, shifted, maps,
                                                         hcap, bsmin, scratch, slot);
    return check_launch("gm_ring_synthesis_fold");
}
