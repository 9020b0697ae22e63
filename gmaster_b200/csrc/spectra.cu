// Pseudo-C_ell, Wigner-3j coupling blocks, binning and the binned decouple (sm_100a).
//
// Replaces, from the reference (licongxu/GMaster):
//   gmaster/workspaces.py:86-95      `_compute_coupled_cell` (XLA segment_sum)
//   gmaster/workspaces.py:352-517    scalar coupling (threej closed form / GL quadrature)
//   gmaster/workspaces.py:682-924    spin-0/2 coupling by GL quadrature GEMMs
//   gmaster/_native/cuda/coupling_tt.cu:18-45  (FP32-product threej kernel, lmax < 48)
//   gmaster/workspaces.py:1570-1590, 292-310   binned MCM (cuBLAS GEMMs)
//   gmaster/workspaces.py:2146       decouple solve (cuSOLVER getrf/getrs)
#include <math.h>

#include "gm_common.cuh"

namespace gm {

__device__ __forceinline__ int64_t alm_idx(int64_t lmax, int64_t l, int64_t m)
{
    return m * (2 * lmax + 1 - m) / 2 + l;
}

// ---------------------------------------------------------------- pseudo-C_ell

constexpr int kPclThreads = 1024;
constexpr int kPclPairs = 64;    // field pairs of one launch

// Field pairs of a launch: pair p has the alms a (N1 rows of nelem) and b (N2 rows), spectra out
// (N1 N2 rows of L).
struct PclPairs {
    const double2 *a[kPclPairs], *b[kPclPairs];
    double *out[kPclPairs];
};

// grid (blocks of LANES degrees, the longest sums first; pairs), 1024 threads: a thread takes degree
// l and sums the orders m = w, w + 1024 / LANES, ... <= l of every component product (each alm read
// once); the partial sums are then added in a fixed order, so the result does not depend on
// scheduling (equal inputs give bit-equal spectra).  Bound by the latency of the order loop at small
// lmax and by memory at large: 32 warps keep it at lmax / 32 steps, and a batch of pairs is one
// launch.  32 pairs of (E, B) at lmax 767: 74 us (4.1 TB/s); 911 us in 32 launches of eight warps and
// one product a CTA.  LANES = 32 up to 512 degrees, 16 up to 1024, 8 above: one pair has few blocks of
// 32 (two (E, B) fields at lmax 767 / 3071 / 6143: 19 / 148 / 381 -> 13 / 74 / 251 us), where 32
// pairs at lmax 767 lose 5 % with 16 and 25 % with 8.
template <int N1, int N2, int LANES>
__global__ void __launch_bounds__(kPclThreads) k_pseudo_cl(int64_t lmax, const __grid_constant__ PclPairs p)
{
    constexpr int kGroups = kPclThreads / LANES, kOut = N1 * N2 * LANES;
    constexpr int kPer = kPclThreads / kOut < 32 ? kPclThreads / kOut : 32;   // threads per result
    __shared__ double part[N1 * N2][kGroups][LANES + 1];
    const int64_t L = lmax + 1, nelem = L * (L + 1) / 2;
    const int lane = threadIdx.x % LANES, w = threadIdx.x / LANES;
    const int64_t l = (int64_t)(gridDim.x - 1 - blockIdx.x) * LANES + lane;
    const double2 *a = p.a[blockIdx.y], *b = p.b[blockIdx.y];
    const bool same = N1 == N2 && a == b;
    double s[N1 * N2];
#pragma unroll
    for (int q = 0; q < N1 * N2; ++q) s[q] = 0.0;
    if (l < L) {
#pragma unroll 4
        for (int64_t m = w; m <= l; m += kGroups) {
            const int64_t k = alm_idx(lmax, l, m);
            double2 x[N1], y[N2];
#pragma unroll
            for (int i = 0; i < N1; ++i) x[i] = a[i * nelem + k];
#pragma unroll
            for (int j = 0; j < N2; ++j) y[j] = same ? x[j % N1] : b[j * nelem + k];
#pragma unroll
            for (int i = 0; i < N1; ++i)
#pragma unroll
                for (int j = 0; j < N2; ++j) {
                    const double re = x[i].x * y[j].x + x[i].y * y[j].y;
                    s[i * N2 + j] += m == 0 ? re : 2.0 * re;
                }
        }
    }
#pragma unroll
    for (int q = 0; q < N1 * N2; ++q) part[q][w][lane] = s[q];
    __syncthreads();
    // kPer neighbouring threads add a result's partial sums, always in the same order
    const int o = threadIdx.x / kPer, i = threadIdx.x % kPer, d = o % LANES;
    double t = 0.0;
    if (o < kOut) {
#pragma unroll
        for (int g = i; g < kGroups; g += kPer) t += part[o / LANES][g][d];
    }
#pragma unroll
    for (int h = kPer / 2; h >= 1; h >>= 1) t += __shfl_xor_sync(0xffffffffu, t, h);
    const int64_t lo = (int64_t)(gridDim.x - 1 - blockIdx.x) * LANES + d;
    if (o < kOut && i == 0 && lo < L) p.out[blockIdx.y][(o / LANES) * L + lo] = t / (2.0 * (double)lo + 1.0);
}

// ---------------------------------------------------------------- Wigner-3j coupling

// Work unit u -> (l1, l2 block) with l1 descending (longest recursions first):
// t = lmax - l1 has floor(t / 32) + 1 blocks of 32 columns l2 >= l1.
__device__ __forceinline__ bool unit_to_pair(int64_t u, int64_t lmax, int64_t &l1, int64_t &l2b)
{
    // cumulative units before t = 32 G + rr: 16 G (G + 1) + rr (G + 1)
    int64_t G = (int64_t)floor((sqrt(1.0 + (double)u / 4.0) - 1.0) / 2.0);
    if (G < 0) G = 0;
    while (16 * (G + 1) * (G + 2) <= u) ++G;
    while (G > 0 && 16 * G * (G + 1) > u) --G;
    const int64_t rem = u - 16 * G * (G + 1);
    const int64_t rr = rem / (G + 1), b = rem % (G + 1);
    const int64_t t = 32 * G + rr;
    if (t > lmax) return false;
    l1 = lmax - t;
    l2b = l1 + 32 * b;
    return true;
}

__host__ __device__ __forceinline__ int64_t total_units(int64_t lmax)
{
    // t in [0, lmax]: sum of floor(t/32) + 1
    const int64_t T = lmax + 1, G = T / 32, rr = T % 32;
    return 16 * G * (G + 1) + rr * (G + 1);
}

// Coupling sums of one pair (l1 <= l2): vals[x] = S_x(l1, l2) for x = tt, te, pp, mm,
// S_x = sum_l3 (2 l3 + 1) W_l3 / (4 pi) T_x(l1, l2, l3) (the blocks divided by 2 l2 + 1),
// with T_tt = (l1 l2 l3; 000)^2, T_te = (000)(2 -2 0), T_pp / T_mm = (2 -2 0)^2 on the
// l1 + l2 + l3 even / odd terms.
//
// Recurrences in j = l3 from j_min = l2 - l1 to j_max = l1 + l2 (Schulten & Gordon 1975,
// m3 = 0): with P(j) = (j^2 - d^2)(S^2 - j^2), d = l2 - l1, S = l1 + l2 + 1,
//   sqrt P(j+1) f_{j+1} = -sqrt P(j) f_{j-1}                    for (000)
//   sqrt P(j+1) g_{j+1} = 4 (2j+1) g_j - sqrt P(j) g_{j-1}      for (2 -2 0),
// both unnormalised from f = g = 1 at j_min and normalised by sum (2j+1) f^2 = 1.  The
// substitution f^_j = f_j s_j, g^_j = g_j s_j with s_j = prod_{i <= j} sqrt P(i) removes
// every square root and division:
//   f^_{j+1} = -P(j) f^_{j-1},   g^_{j+1} = 4 (2j+1) g^_j - P(j) g^_{j-1},
// and f^2, f g, g^2 become the hatted products over D_j = prod_{i <= j} P(i).  Each sum
// sum_j c_j X^_j / D_j is carried as A / D_j with A_j = A_{j-1} P(j) + c_j X^_j (Horner
// form); D cancels in every quotient of the results, so it is never formed.  The odd-offset
// (000) terms vanish, so the loop steps j by two.  The products grow by ~P^2 per step;
// whenever a normalising sum passes 2^512 its family is scaled down by an exact power of
// two (f^ or g^ by 2^-256, their squared sums by 2^-512).
// Scaling f^, g^ by 4^(j - j_min) takes the factor 4 into P / 16, formed exactly from j / 2, d / 2
// and S / 2; the window multiplies the terms (2j+1) X^2 of the normalising sums: 26 double-precision
// operations per two steps for M+ and M- (31 before: 1.64 ms for both at lmax 1535), at the rate of
// three-operand FMAs the register file sustains (about two thirds of the pipe).
template <bool TT, bool TE, bool PM>
__device__ __forceinline__ void coupling_sums(int64_t l1, int64_t l2, const double *__restrict__ window,
                                              int64_t nw, double (&vals)[4])
{
    constexpr bool F = TT || TE, G = TE || PM;
    const double inv4pi = 1.0 / (4.0 * M_PI);
    const int64_t d = l2 - l1, jmin = d, jmax = l1 + l2;
    const double S = 0.5 * (double)(l1 + l2 + 1), S2 = S * S, dh = 0.5 * (double)d, d2 = dh * dh;
    const double lo = 0x1p-256, lo2 = 0x1p-512;
    const int big = (1023 + 512) << 20;  // high word of 2^512
    double t0 = 2.0 * (double)jmin + 1.0;
    const double w0 = (jmin < nw ? __ldg(window + jmin) : 0.0) * t0;
    double f0 = 1.0, g0 = 1.0, gm1 = 0.0, P0 = 0.0;
    double an0 = t0, att = w0, an2 = t0, ate = w0, app = w0, amm = 0.0;
    double jh = dh;   // j / 2
    for (int64_t j = jmin; j < jmax; j += 2) {
        const double j1 = jh + 0.5, j2 = jh + 1.0;
        const double P1 = fma(j1, j1, -d2) * fma(-j1, j1, S2);   // P / 16
        const double P2 = fma(j2, j2, -d2) * fma(-j2, j2, S2);
        const double t1 = t0 + 2.0, t2 = t0 + 4.0;
        const double w2 = j + 2 < nw ? __ldg(window + j + 2) : 0.0;
        const double PP = P1 * P2;
        double f2 = 0.0, g2 = 0.0;
        if (F) {
            f2 = -P1 * f0;
            const double tf2 = t2 * (f2 * f2);
            an0 = fma(an0, PP, tf2);
            if (TT) att = fma(att, PP, w2 * tf2);
        }
        if (G) {
            const double g1 = fma(t0, g0, -P0 * gm1);
            g2 = fma(t1, g1, -P1 * g0);
            const double tg1 = t1 * (g1 * g1), tg2 = t2 * (g2 * g2);
            an2 = fma(fma(an2, P1, tg1), P2, tg2);
            if (PM) {
                const double w1 = j + 1 < nw ? __ldg(window + j + 1) : 0.0;
                app = fma(app, PP, w2 * tg2);
                amm = fma(amm, P1, w1 * tg1) * P2;
            }
            if (TE) ate = fma(ate, PP, w2 * (t2 * (f2 * g2)));
            gm1 = g1;
            g0 = g2;
        }
        f0 = f2;
        P0 = P2;
        jh = j2;
        t0 = t2;
        if (F && __double2hiint(an0) > big) {
            f0 *= lo;
            an0 *= lo2;
            att *= lo2;
            ate *= lo;
        }
        if (G && __double2hiint(an2) > big) {
            g0 *= lo;
            gm1 *= lo;
            an2 *= lo2;
            app *= lo2;
            amm *= lo2;
            ate *= lo;
        }
    }
    if (TT) vals[0] = inv4pi * att / an0;
    if (TE) {
        // (000) and (2 -2 0) both carry (-1)^(l1 - l2) at l3 = l1 + l2, so the relative
        // sign of the unnormalised product is sign(f g) there.
        const double sgn = (f0 * g0) < 0.0 ? -1.0 : 1.0;
        vals[1] = sgn * inv4pi * ate / (sqrt(an0) * sqrt(an2));
    }
    if (PM) {
        vals[2] = inv4pi * app / an2;
        vals[3] = inv4pi * amm / an2;
    }
}

// Coupling sums of the blocks `which` asks for (bit x = block x); the others are zero.
// Spin-2 sums vanish unless l1, l2 >= 2.
__device__ __forceinline__ void coupling_pair(int64_t l1, int64_t l2, const double *__restrict__ window,
                                              int64_t nw, int which, double (&vals)[4])
{
    vals[0] = vals[1] = vals[2] = vals[3] = 0.0;
    const bool s2ok = l1 >= 2 && l2 >= 2;
    const int w = s2ok ? which : (which & 1);
    if (w == 1) coupling_sums<true, false, false>(l1, l2, window, nw, vals);
    else if (w == 2) coupling_sums<false, true, false>(l1, l2, window, nw, vals);
    else if (w == 4 || w == 8 || w == 12) coupling_sums<false, false, true>(l1, l2, window, nw, vals);
    else if (w != 0) coupling_sums<true, true, true>(l1, l2, window, nw, vals);
}

__global__ void __launch_bounds__(128) k_coupling(int64_t lmax, const double *__restrict__ window,
                                                  int64_t nw, int which,
                                                  double *__restrict__ blocks,
                                                  unsigned long long *__restrict__ queue)
{
    const int64_t n = lmax + 1, nn = n * n;
    const int64_t nunits = total_units(lmax);
    const int lane = threadIdx.x & 31;
    for (;;) {
        unsigned long long u = 0;
        if (lane == 0) u = atomicAdd(queue, 1ull);
        u = __shfl_sync(0xffffffffu, u, 0);
        if ((int64_t)u >= nunits) break;
        int64_t l1, l2b;
        if (!unit_to_pair((int64_t)u, lmax, l1, l2b)) break;
        const int64_t l2 = l2b + lane;
        if (l2 <= lmax) {
            double vals[4];
            coupling_pair(l1, l2, window, nw, which, vals);
            const double c1 = 2.0 * (double)l1 + 1.0, c2 = 2.0 * (double)l2 + 1.0;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (!(which & (1 << x))) continue;
                double *bx = blocks + x * nn;
                bx[l1 * n + l2] = c2 * vals[x];
                bx[l2 * n + l1] = c1 * vals[x];
            }
        }
    }
}

// Many coupling matrices of different lmax in one persistent launch.  Job j is the row
// jobs[6 j .. 6 j + 5] = (lmax, window offset, nw, which, blocks offset, first unit); units
// are numbered consecutively over the jobs (job j owns [first_j, first_{j+1}) and
// nunits in total), the jobs being ordered by decreasing lmax so the longest recursions
// go first.  Each warp takes the next unit from the shared queue, finds its job by binary
// search and computes its pair block as k_coupling does.
__global__ void __launch_bounds__(128) k_coupling_multi(int64_t njobs, const int64_t *__restrict__ jobs,
                                                        int64_t nunits,
                                                        const double *__restrict__ windows,
                                                        double *__restrict__ blocks,
                                                        unsigned long long *__restrict__ queue)
{
    const int lane = threadIdx.x & 31;
    for (;;) {
        unsigned long long u = 0;
        if (lane == 0) u = atomicAdd(queue, 1ull);
        u = __shfl_sync(0xffffffffu, u, 0);
        if ((int64_t)u >= nunits) break;
        int64_t lo = 0, hi = njobs - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) / 2;
            if (jobs[6 * mid + 5] <= (int64_t)u) lo = mid;
            else hi = mid - 1;
        }
        const int64_t *jb = jobs + 6 * lo;
        const int64_t lmax = jb[0], n = lmax + 1, nn = n * n;
        const int which = (int)jb[3];
        int64_t l1, l2b;
        if (!unit_to_pair((int64_t)u - jb[5], lmax, l1, l2b)) continue;
        const int64_t l2 = l2b + lane;
        if (l2 <= lmax) {
            double vals[4];
            coupling_pair(l1, l2, windows + jb[1], jb[2], which, vals);
            const double c1 = 2.0 * (double)l1 + 1.0, c2 = 2.0 * (double)l2 + 1.0;
            double *bj = blocks + jb[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (!(which & (1 << x))) continue;
                double *bx = bj + x * nn;
                bx[l1 * n + l2] = c2 * vals[x];
                bx[l2 * n + l1] = c1 * vals[x];
            }
        }
    }
}

// Scalar coupling sums S_tt(l1, l2) of an explicit list of pairs, written symmetrically
// into the dense (lmax+1)^2 matrix S (entries not listed are left as they are).
__global__ void k_coupling_pairs_tt(int64_t lmax, const double *__restrict__ window, int64_t nw,
                                    const int32_t *__restrict__ pairs, int64_t npairs,
                                    double *__restrict__ S)
{
    const int64_t t = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= npairs) return;
    const int64_t a = pairs[2 * t], b = pairs[2 * t + 1], n = lmax + 1;
    const int64_t l1 = a < b ? a : b, l2 = a < b ? b : a;
    double vals[4];
    coupling_pair(l1, l2, window, nw, 1, vals);
    S[l1 * n + l2] = vals[0];
    S[l2 * n + l1] = vals[0];
}

// NaMaster's Toeplitz approximation of the scalar coupling (Louis et al. 2020), filled
// from the exact entries of S = M / (2 l' + 1) that it reads: the diagonal, column
// l_toeplitz, columns 0..l_exact and the dl_band sub-diagonals.  With d_l = |S_ll|, the
// correlation c_l = S(l, lt) / sqrt(d_l d_lt) and the column correlation
// e_l = S(l, le) / sqrt(d_l d_le) (zero where d vanishes), entry (r >= q) of the lower
// triangle is, by the first rule that applies:
//   le <= q <= lt and r >= n - 1 - lt + q :  e_{r - q + le} sqrt(d_q d_r)
//   1 <= r - q <= dl_band and q <= lt      :  S(q, r)
//   r == q                                  :  S(r, r)
//   r >= lt and q >= lt                     :  c_{(r - q + lt) mod n} sqrt(d_r d_q)
//   r - q <= dl_band                        :  S(q, r)
//   q <= le                                 :  S(r, q)
//   otherwise                               :  c_{(r - q + lt) mod n} sqrt(d_r d_q)
// and the matrix is symmetric; out(i, j) = T(i, j) (2 j + 1).
__global__ void k_toeplitz_fill(int64_t lmax, int64_t lt, int64_t le, int64_t dlb,
                                const double *__restrict__ S, double *__restrict__ out)
{
    const int64_t n = lmax + 1;
    const int64_t i = blockIdx.y, j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= n) return;
    const int64_t r = i > j ? i : j, q = i > j ? j : i;
    auto d = [&](int64_t l) { return fabs(S[l * n + l]); };
    auto corr = [&](int64_t l) {
        const double den = sqrt(d(l) * d(lt));
        return den > 0.0 ? S[l * n + lt] / den : 0.0;
    };
    auto pure = [&]() { return corr((r - q + lt) % n) * sqrt(d(r) * d(q)); };
    double v;
    if (q >= le && q <= lt && r >= n - 1 - lt + q) {
        const int64_t l = r - q + le;
        const double dl = d(l);
        const double e = dl > 0.0 ? S[l * n + le] / sqrt(dl * d(le)) : 0.0;
        v = e * sqrt(d(q) * d(r));
    } else if (r - q >= 1 && r - q <= dlb && q <= lt) {
        v = S[q * n + r];
    } else if (r == q) {
        v = S[r * n + r];
    } else if (r >= lt && q >= lt) {
        v = pure();
    } else if (r - q <= dlb) {
        v = S[q * n + r];
    } else if (q <= le) {
        v = S[r * n + q];
    } else {
        v = pure();
    }
    out[i * n + j] = v * (2.0 * (double)j + 1.0);
}

// ---------------------------------------------------------------- binning

// Binned block: out[b][b'] = sum_{l in b} wfl[l] sum_{l' in b'} M[l][l'] beam[l'] inv_fl[l'].  ROWS warps
// per pair of bands: lanes along l', every ROWS-th row of b in turn (several loads in flight),
// then a sum over the lanes and the warps.  Bound by the latency of the rows.  A CTA of 256 threads
// per pair, with a division per element and a tree in shared memory, took 38 us a block at lmax 1535
// with bands of ten; 16 us here with one warp.  Few or wide bands take eight: three bands of 50
// degrees at Nside 64 78 us a binned workspace with one warp, 56 with eight; one of 766, 2.2 and 0.39 ms.
constexpr int kBinWarps = 8;
template <int ROWS>
__global__ void __launch_bounds__(32 * kBinWarps) k_bin_block(
    int64_t lmax, int64_t nb, const double *__restrict__ M, const int32_t *__restrict__ band_ptr,
    const int32_t *__restrict__ band_ells, const double *__restrict__ wfl, const double *__restrict__ inv_fl,
    const double *__restrict__ beam, double *__restrict__ out)
{
    constexpr int kPairs = kBinWarps / ROWS;
    __shared__ double part[kBinWarps];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int64_t b = blockIdx.y, bp = (int64_t)blockIdx.x * kPairs + w / ROWS, n = lmax + 1;
    double s = 0.0;
    if (bp < nb) {
        const int i0 = band_ptr[b] + w % ROWS, i1 = band_ptr[b + 1], k0 = band_ptr[bp], k1 = band_ptr[bp + 1];
        for (int k = k0 + lane; k < k1; k += 32) {
            const int lp = band_ells[k];
            double t = 0.0;
#pragma unroll 4
            for (int i = i0; i < i1; i += ROWS) {
                const int l = band_ells[i];
                t = fma(wfl[l], M[(int64_t)l * n + lp], t);
            }
            s += t * beam[lp] * inv_fl[lp];
        }
    }
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if (ROWS == 1) {
        if (lane == 0 && bp < nb) out[b * nb + bp] = s;
        return;
    }
    if (lane == 0) part[w] = s;
    __syncthreads();
    if (threadIdx.x < kPairs) {
        const int64_t q = (int64_t)blockIdx.x * kPairs + threadIdx.x;
        double t = 0.0;
        for (int r = 0; r < ROWS; ++r) t += part[threadIdx.x * ROWS + r];
        if (q < nb) out[b * nb + q] = t;
    }
}

// Place binned blocks into the (ncls nb)^2 matrix, band-major channel-minor.
__global__ void k_place_binned(int64_t nb, int ncls, const double *__restrict__ bb,
                               double *__restrict__ out)
{
    const int64_t N = ncls * nb;
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= N * N) return;
    const int64_t row = idx / N, col = idx % N;
    const int64_t b = row / ncls, c1 = row % ncls, bp = col / ncls, c2 = col % ncls;
    const int64_t nb2 = nb * nb;
    double v = 0.0;
    if (ncls == 1) {
        v = bb[b * nb + bp];
    } else if (ncls == 2) {
        if (c1 == c2) v = bb[b * nb + bp];
    } else {
        if (c1 == c2) v = bb[b * nb + bp];                       // M+ on the diagonal slots
        else if (c1 + c2 == 3)                                   // M- on the anti-diagonal
            v = ((c1 == 1 || c1 == 2) ? -1.0 : 1.0) * bb[nb2 + b * nb + bp];
    }
    out[idx] = v;
}

__global__ void k_bin_cells(int64_t lmax, int64_t nb, int64_t ncls, const double *__restrict__ cls,
                            const int32_t *__restrict__ band_ptr,
                            const int32_t *__restrict__ band_ells, const double *__restrict__ wfl,
                            double *__restrict__ out)
{
    const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= nb * ncls) return;
    const int64_t c = idx / nb, b = idx % nb;
    double s = 0.0;
    for (int i = band_ptr[b]; i < band_ptr[b + 1]; ++i) {
        const int l = band_ells[i];
        s += wfl[l] * cls[c * (lmax + 1) + l];
    }
    out[c * nb + b] = s;
}

// ---------------------------------------------------------------- LU

// Order of pivot candidates: NaN, then by magnitude (zero is 1).
__device__ __forceinline__ unsigned long long pivot_key(double v)
{
    const double f = fabs(v);
    return f >= 0.0 ? (unsigned long long)__double_as_longlong(f) + 1ull : 0ull;
}

// The warp's largest key and its lowest row: the key's halves and the row one after the other
// through the integer reductions (a shuffle tree of (key, row) takes 15 steps).
__device__ __forceinline__ void best_pivot(unsigned long long &q, int &r)
{
    const unsigned hi = (unsigned)(q >> 32), lo = (unsigned)q;
    const unsigned mh = __reduce_max_sync(0xffffffffu, hi);
    const unsigned ml = __reduce_max_sync(0xffffffffu, hi == mh ? lo : 0u);
    const bool mine = hi == mh && lo == ml;
    r = __reduce_min_sync(0xffffffffu, mine ? r : 0x7fffffff);
    q = ((unsigned long long)mh << 32) | ml;
}

// Blocked LU, panel step in shared memory: columns [k0, k0 + kb) of rows k0..n-1 of the
// row-major (n, n) matrix, one CTA, partial pivoting (largest magnitude, lowest row on ties; a
// NaN is never chosen over a number).  Row interchanges are confined to the panel here; k_lu_rest
// applies them to the other columns.  piv[k] is the row exchanged with row k; *status receives
// k + 1 for the first column without a non-zero pivot.
//
// Bound by latency: two barriers, a warp reduction of the pivot candidates and kb - k
// multiply-adds a row per column.  The panel is read and written once; held in global memory it
// took 7 us a column, here 1.6 at 612 rows (bound by the shared-memory traffic of the update).
__global__ void __launch_bounds__(1024) k_lu_panel_smem(int n, int k0, int kb, double *__restrict__ a,
                                                        int32_t *__restrict__ piv, int32_t *__restrict__ status)
{
    extern __shared__ double pan[];   // [kb][ld], column c at pan + c * ld
    __shared__ unsigned long long skey[2][32];
    __shared__ int srow[2][32];
    const int rows = n - k0, ld = rows | 1;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    if (k0 == 0 && tid == 0) *status = 0;
    for (int64_t e = tid; e < (int64_t)rows * kb; e += blockDim.x) {
        const int i = (int)(e / kb), c = (int)(e % kb);
        pan[(int64_t)c * ld + i] = a[(int64_t)(k0 + i) * n + k0 + c];
    }
    __syncthreads();
    for (int k = 0; k < kb; ++k) {
        double *col = pan + (int64_t)k * ld;
        unsigned long long key = 0;
        int row = k;
        for (int i = k + tid; i < rows; i += blockDim.x) {
            const unsigned long long q = pivot_key(col[i]);
            if (q > key) {
                key = q;
                row = i;
            }
        }
        best_pivot(key, row);
        if (lane == 0) {
            skey[k & 1][warp] = key;
            srow[k & 1][warp] = row;
        }
        __syncthreads();
        key = lane < nw ? skey[k & 1][lane] : 0ull;
        row = lane < nw ? srow[k & 1][lane] : 0x7fffffff;
        best_pivot(key, row);
        if (key == 0ull) row = k;   // no number in the column
        if (tid == 0) {
            piv[k0 + k] = k0 + row;
            if (key == 1ull && *status == 0) *status = k0 + k + 1;
        }
        if (row != k)
            for (int c = tid; c < kb; c += blockDim.x) {
                const double t = pan[(int64_t)c * ld + k];
                pan[(int64_t)c * ld + k] = pan[(int64_t)c * ld + row];
                pan[(int64_t)c * ld + row] = t;
            }
        __syncthreads();
        const double d = col[k], inv = d != 0.0 ? 1.0 / d : 0.0;
        for (int i = k + 1 + tid; i < rows; i += blockDim.x) {
            const double l = col[i] * inv;
            col[i] = l;
#pragma unroll 4
            for (int c = k + 1; c < kb; ++c) {
                double *pc = pan + (int64_t)c * ld;
                pc[i] = fma(-l, pc[k], pc[i]);
            }
        }
        __syncthreads();
    }
    for (int64_t e = tid; e < (int64_t)rows * kb; e += blockDim.x) {
        const int i = (int)(e / kb), c = (int)(e % kb);
        a[(int64_t)(k0 + i) * n + k0 + c] = pan[(int64_t)c * ld + i];
    }
}

// The panel step with every row in the registers of a thread (rows <= NT, kb <= KB): the update of
// a column then reads only the pivot row from shared memory, where the form above moves two
// entries a row and column through it: panels of a 612 x 612 matrix 1.0 -> 0.66 ms.
template <int KB, int NT>
__global__ void __launch_bounds__(NT) k_lu_panel_reg(int n, int k0, int kb, double *__restrict__ a,
                                                     int32_t *__restrict__ piv, int32_t *__restrict__ status)
{
    __shared__ __align__(16) double prow[KB], krow[KB];
    __shared__ unsigned long long skey[32];
    __shared__ int srow[32];
    const int rows = n - k0, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    const bool mine = tid < rows;
    if (k0 == 0 && tid == 0) *status = 0;
    double x[KB];
    double *src = a + (int64_t)(k0 + tid) * n + k0;
#pragma unroll
    for (int c = 0; c < KB; ++c) x[c] = mine && c < kb ? src[c] : 0.0;
#pragma unroll
    for (int k = 0; k < KB; ++k) {
        if (k >= kb) break;
        unsigned long long key = mine && tid >= k ? pivot_key(x[k]) : 0ull;
        int row = mine && tid >= k ? tid : 0x7fffffff;
        best_pivot(key, row);
        if (lane == 0) {
            skey[warp] = key;
            srow[warp] = row;
        }
        __syncthreads();
        key = lane < nw ? skey[lane] : 0ull;
        row = lane < nw ? srow[lane] : 0x7fffffff;
        best_pivot(key, row);
        if (key == 0ull) row = k;   // no number in the column
        if (tid == 0) {
            piv[k0 + k] = k0 + row;
            if (key == 1ull && *status == 0) *status = k0 + k + 1;
        }
        if (tid == row)
#pragma unroll
            for (int c = 0; c < KB; ++c) prow[c] = x[c];
        if (tid == k && row != k)
#pragma unroll
            for (int c = 0; c < KB; ++c) krow[c] = x[c];
        __syncthreads();
        if (row != k) {
            if (tid == row)
#pragma unroll
                for (int c = 0; c < KB; ++c) x[c] = krow[c];
            if (tid == k)
#pragma unroll
                for (int c = 0; c < KB; ++c) x[c] = prow[c];
        }
        if (tid > k) {
            const double d = prow[k], inv = d != 0.0 ? 1.0 / d : 0.0;
            const double l = x[k] * inv;
            x[k] = l;
#pragma unroll
            for (int c = k + 1; c < KB; ++c) x[c] = fma(-l, prow[c], x[c]);
        }
    }
    if (mine)
#pragma unroll
        for (int c = 0; c < KB; ++c)
            if (c < kb) src[c] = x[c];
}

// Blocked LU, the columns outside the panel [k0, k0 + kb), kb <= 32: the panel's row
// interchanges as one permutation (every row read before any is written), and right of the panel
// the U rows, L11^-1 times themselves with L11 unit lower triangular; one thread per column.
constexpr int kLuPan = 32;
__global__ void __launch_bounds__(128) k_lu_rest(int n, int k0, int kb, double *__restrict__ a,
                                                 const int32_t *__restrict__ piv)
{
    __shared__ double l11[kLuPan][kLuPan];
    __shared__ int top[kLuPan], ext[kLuPan], dst[kLuPan];   // sources of the panel's rows and of the rows below
    __shared__ bool below[kLuPan];                          // dst is below the panel and named for the first time
    const int tid = threadIdx.x, k1 = k0 + kb;
    for (int e = tid; e < kb * kb; e += blockDim.x) l11[e / kb][e % kb] = a[(int64_t)(k0 + e / kb) * n + k0 + e % kb];
    if (tid < kb) {
        top[tid] = k0 + tid;
        const int p = piv[k0 + tid];
        dst[tid] = p;
        ext[tid] = p;
    }
    __syncthreads();
    if (tid < kb) {
        bool first = dst[tid] >= k1;
        for (int e = 0; e < tid && first; ++e) first = dst[e] != dst[tid];
        below[tid] = first;
    }
    if (tid == 0) {
        for (int i = 0; i < kb; ++i) {
            const int p = dst[i], t = top[i];
            if (p < k1) {
                top[i] = top[p - k0];
                top[p - k0] = t;
            } else {
                int e = 0;   // the first step that exchanged with row p holds its content
                while (dst[e] != p) ++e;
                top[i] = ext[e];
                ext[e] = t;
            }
        }
    }
    __syncthreads();
    int col = blockIdx.x * blockDim.x + tid;
    if (col >= n - kb) return;
    if (col >= k0) col += kb;
    double u[kLuPan], w[kLuPan];
#pragma unroll
    for (int i = 0; i < kLuPan; ++i) {
        if (i >= kb) break;
        u[i] = a[(int64_t)top[i] * n + col];
        w[i] = below[i] ? a[(int64_t)ext[i] * n + col] : 0.0;
    }
#pragma unroll
    for (int i = 0; i < kLuPan; ++i) {
        if (i >= kb) break;
        if (below[i]) a[(int64_t)dst[i] * n + col] = w[i];
        if (col >= k1) {
#pragma unroll
            for (int j = 0; j < kLuPan; ++j) {
                if (j >= i) break;
                u[i] = fma(-l11[i][j], u[j], u[i]);
            }
        }
        a[(int64_t)(k0 + i) * n + col] = u[i];
    }
}

// Blocked LU, panel step in global memory for matrices whose panels do not fit shared memory:
// columns [k0, k1) of the row-major (n, n) matrix, rows k0..n-1,
// one CTA.  Partial pivoting as in k_lu_panel_smem (the pivot swap moves whole rows, all n
// columns, so the left factor and the trailing part stay consistent); the rank-1 updates
// are confined to the panel's columns.  The caller then solves for the U rows right of
// the panel (k_lu_trsm) and updates the trailing matrix with one GEMM.
__global__ void __launch_bounds__(1024) k_lu_panel(int64_t n, int64_t k0, int64_t k1,
                                                   double *__restrict__ a, int32_t *__restrict__ piv,
                                                   int32_t *__restrict__ status)
{
    __shared__ double sval[32];
    __shared__ int sidx[32];
    __shared__ int pivot_row;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
    for (int64_t k = k0; k < k1; ++k) {
        double best = -1.0;
        int bi = (int)k;
        for (int64_t i = k + tid; i < n; i += blockDim.x) {
            const double v = fabs(a[i * n + k]);
            if (v > best) {
                best = v;
                bi = (int)i;
            }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ov = __shfl_down_sync(0xffffffffu, best, o);
            const int oi = __shfl_down_sync(0xffffffffu, bi, o);
            if (ov > best || (ov == best && oi < bi)) {
                best = ov;
                bi = oi;
            }
        }
        if (lane == 0) {
            sval[warp] = best;
            sidx[warp] = bi;
        }
        __syncthreads();
        if (tid == 0) {
            double bv = sval[0];
            int bix = sidx[0];
            for (int w = 1; w < nwarps; ++w)
                if (sval[w] > bv || (sval[w] == bv && sidx[w] < bix)) {
                    bv = sval[w];
                    bix = sidx[w];
                }
            pivot_row = bix;
            piv[k] = bix;
            if (bv == 0.0 && *status == 0) *status = (int32_t)(k + 1);
        }
        __syncthreads();
        const int64_t p = pivot_row;
        if (p != k)
            for (int64_t jj = tid; jj < n; jj += blockDim.x) {
                const double t = a[k * n + jj];
                a[k * n + jj] = a[p * n + jj];
                a[p * n + jj] = t;
            }
        __syncthreads();
        const double d = a[k * n + k];
        const double inv = d != 0.0 ? 1.0 / d : 0.0;
        for (int64_t i = k + 1 + tid; i < n; i += blockDim.x) a[i * n + k] *= inv;
        __syncthreads();
        for (int64_t i = k + 1 + warp; i < n; i += nwarps) {
            const double lik = a[i * n + k];
            if (lik != 0.0)
                for (int64_t jj = k + 1 + lane; jj < k1; jj += 32) a[i * n + jj] -= lik * a[k * n + jj];
        }
        __syncthreads();
    }
}

// Blocked LU, U rows right of the panel: rows [k0, k1), columns [k1, n) become
// L11^-1 times themselves (L11 unit lower triangular); one thread per column.
__global__ void k_lu_trsm(int64_t n, int64_t k0, int64_t k1, double *__restrict__ a)
{
    const int64_t col = k1 + (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (col >= n) return;
    for (int64_t i = k0 + 1; i < k1; ++i) {
        double s = a[i * n + col];
        for (int64_t j = k0; j < i; ++j) s -= a[i * n + j] * a[j * n + col];
        a[i * n + col] = s;
    }
}

// Blocked LU, trailing update: A[i][j] -= sum_{k in [k0, k1)} A[i][k] A[k][j] for i, j >= k1
// (the Schur complement of the panel).  One CTA per 64 x 64 tile of the trailing matrix;
// the panel width (<= 64) is taken in chunks of 32: the tile's rows of the left factor and
// columns of the U rows are staged in shared memory and each of the 256 threads
// accumulates a 4 x 4 block in FP64.
constexpr int kLuTile = 64;
constexpr int kLuK = 32;
__global__ void __launch_bounds__(256) k_lu_update(int64_t n, int64_t k0, int64_t k1,
                                                   double *__restrict__ a)
{
    __shared__ double sl[kLuTile][kLuK + 1];   // [row][k]
    __shared__ double su[kLuTile][kLuK + 1];   // [col][k]
    const int kw = (int)(k1 - k0);
    const int64_t r0 = k1 + (int64_t)blockIdx.y * kLuTile, c0 = k1 + (int64_t)blockIdx.x * kLuTile;
    const int tid = threadIdx.x;
    const int ty = tid / 16, tx = tid % 16;   // rows 4 ty + i, columns tx + 16 j
    double acc[4][4] = {};
    for (int kc = 0; kc < kw; kc += kLuK) {
        for (int e = tid; e < kLuTile * kLuK; e += 256) {
            // left factor: consecutive threads take consecutive k of a row
            const int r = e / kLuK, k = e % kLuK;
            const int64_t gr = r0 + r;
            sl[r][k] = (gr < n && kc + k < kw) ? a[gr * n + k0 + kc + k] : 0.0;
            // U rows: consecutive threads take consecutive columns of a row
            const int kk = e / kLuTile, c = e % kLuTile;
            const int64_t gc = c0 + c;
            su[c][kk] = (gc < n && kc + kk < kw) ? a[(k0 + kc + kk) * n + gc] : 0.0;
        }
        __syncthreads();
#pragma unroll 4
        for (int k = 0; k < kLuK; ++k) {
            double l[4], u[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) l[i] = sl[4 * ty + i][k];
#pragma unroll
            for (int j = 0; j < 4; ++j) u[j] = su[tx + 16 * j][k];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(l[i], u[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int64_t gr = r0 + 4 * ty + i;
        if (gr >= n) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int64_t gc = c0 + tx + 16 * j;
            if (gc < n) a[gr * n + gc] -= acc[i][j];
        }
    }
}

// One warp per right-hand-side column: P, then L (unit) forward, then U backward.
// b is (n, nrhs) row-major.
__global__ void k_lu_solve(int64_t n, const double *__restrict__ lu, const int32_t *__restrict__ piv,
                           int64_t nrhs, double *__restrict__ b)
{
    const int64_t col = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (col >= nrhs) return;
    if (lane == 0)
        for (int64_t k = 0; k < n; ++k) {
            const int64_t p = piv[k];
            if (p != k) {
                const double t = b[k * nrhs + col];
                b[k * nrhs + col] = b[p * nrhs + col];
                b[p * nrhs + col] = t;
            }
        }
    __syncwarp();
    for (int64_t i = 0; i < n; ++i) {
        double s = 0.0;
        for (int64_t jj = lane; jj < i; jj += 32) s += lu[i * n + jj] * b[jj * nrhs + col];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) b[i * nrhs + col] -= s;
        __syncwarp();
    }
    for (int64_t i = n - 1; i >= 0; --i) {
        double s = 0.0;
        for (int64_t jj = i + 1 + lane; jj < n; jj += 32) s += lu[i * n + jj] * b[jj * nrhs + col];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) b[i * nrhs + col] = (b[i * nrhs + col] - s) / lu[i * n + i];
        __syncwarp();
    }
}

// Blocked solve for many right-hand sides: one CTA per kLuCB columns of b, held in shared
// memory.  Rows go in blocks of 32: the contributions of the rows solved so far are summed
// by all 256 threads (thread = (row, one eighth of the columns j), partials added in a fixed
// order), then the 32 x 32 diagonal block is solved by one warp per column with shuffles.
// The same arithmetic as k_lu_solve up to the order of the sums.
constexpr int kLuCB = 4;      // right-hand sides per CTA
constexpr int kLuRB = 32;     // rows per block

__device__ __forceinline__ void lu_block_sums(int64_t n, const double *__restrict__ lu, const double *x,
                                              int64_t r0, int rows, int64_t jbeg, int64_t jend,
                                              double (*part)[kLuCB])
{
    const int tid = threadIdx.x, r = tid >> 3, pt = tid & 7;
    double acc[kLuCB];
#pragma unroll
    for (int c = 0; c < kLuCB; ++c) acc[c] = 0.0;
    if (r < rows) {
        const double *row = lu + (r0 + r) * n;
        for (int64_t j = jbeg + pt; j < jend; j += 8) {
            const double l = __ldg(row + j);
#pragma unroll
            for (int c = 0; c < kLuCB; ++c) acc[c] = fma(l, x[j * kLuCB + c], acc[c]);
        }
    }
#pragma unroll
    for (int c = 0; c < kLuCB; ++c)
        for (int o = 1; o < 8; o <<= 1) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], o);
    if (pt == 0 && r < rows)
#pragma unroll
        for (int c = 0; c < kLuCB; ++c) part[r][c] = acc[c];
}

__global__ void __launch_bounds__(256) k_lu_solve_blk(int64_t n, const double *__restrict__ lu,
                                                      const int32_t *__restrict__ piv, int64_t nrhs,
                                                      double *__restrict__ b)
{
    extern __shared__ double xs[];                   // [n][kLuCB]
    __shared__ double part[kLuRB][kLuCB];
    __shared__ double dg[kLuRB][kLuRB + 1];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * kLuCB;
    const int ncol = (int)(nrhs - c0 < kLuCB ? nrhs - c0 : kLuCB);
    for (int64_t i = tid; i < n * kLuCB; i += blockDim.x) {
        const int64_t r = i / kLuCB;
        const int c = (int)(i % kLuCB);
        xs[i] = c < ncol ? b[r * nrhs + c0 + c] : 0.0;
    }
    __syncthreads();
    if (tid < kLuCB)   // row interchanges, in order
        for (int64_t k = 0; k < n; ++k) {
            const int64_t p = piv[k];
            if (p != k) {
                const double t = xs[k * kLuCB + tid];
                xs[k * kLuCB + tid] = xs[p * kLuCB + tid];
                xs[p * kLuCB + tid] = t;
            }
        }
    const int64_t nblk = (n + kLuRB - 1) / kLuRB;
    // forward: L with unit diagonal
    for (int64_t I = 0; I < nblk; ++I) {
        const int64_t r0 = I * kLuRB;
        const int rows = (int)(n - r0 < kLuRB ? n - r0 : kLuRB);
        __syncthreads();
        lu_block_sums(n, lu, xs, r0, rows, 0, r0, part);
        for (int i = tid; i < kLuRB * kLuRB; i += blockDim.x) {
            const int rr = i / kLuRB, kk = i % kLuRB;
            dg[rr][kk] = (rr < rows && kk < rows) ? lu[(r0 + rr) * n + r0 + kk] : 0.0;
        }
        __syncthreads();
        if (warp < kLuCB) {
            const int c = warp;
            double v = lane < rows ? xs[(r0 + lane) * kLuCB + c] - part[lane][c] : 0.0;
            for (int k = 0; k < rows; ++k) {
                const double xk = __shfl_sync(0xffffffffu, v, k);
                if (lane > k) v = fma(-dg[lane][k], xk, v);
            }
            if (lane < rows) xs[(r0 + lane) * kLuCB + c] = v;
        }
    }
    // backward: U
    for (int64_t I = nblk - 1; I >= 0; --I) {
        const int64_t r0 = I * kLuRB;
        const int rows = (int)(n - r0 < kLuRB ? n - r0 : kLuRB);
        __syncthreads();
        lu_block_sums(n, lu, xs, r0, rows, r0 + rows, n, part);
        for (int i = tid; i < kLuRB * kLuRB; i += blockDim.x) {
            const int rr = i / kLuRB, kk = i % kLuRB;
            dg[rr][kk] = (rr < rows && kk < rows) ? lu[(r0 + rr) * n + r0 + kk] : 1.0;
        }
        __syncthreads();
        if (warp < kLuCB) {
            const int c = warp;
            double v = lane < rows ? xs[(r0 + lane) * kLuCB + c] - part[lane][c] : 0.0;
            for (int k = rows - 1; k >= 0; --k) {
                if (lane == k) v = v / dg[k][k];
                const double xk = __shfl_sync(0xffffffffu, v, k);
                if (lane < k) v = fma(-dg[lane][k], xk, v);
            }
            if (lane < rows) xs[(r0 + lane) * kLuCB + c] = v;
        }
    }
    __syncthreads();
    for (int64_t i = tid; i < n * kLuCB; i += blockDim.x) {
        const int64_t r = i / kLuCB;
        const int c = (int)(i % kLuCB);
        if (c < ncol) b[r * nrhs + c0 + c] = xs[i];
    }
}

// Prepared solves.  The row interchanges of the factorisation as one permutation, and the
// inverses of the 32 x 32 diagonal blocks of L and U (the last block padded with the identity):
// a solve then has no sequential chain inside a block, only a product of 32 x 32.
constexpr int kLuSB = 32;

// Block 0: perm (n rows: row perm[i] of b becomes row i); block 1 + i: the inverses of diagonal
// block i.  inv holds (block, L or U, row, column).
__global__ void __launch_bounds__(64) k_lu_prepare(int n, const double *__restrict__ lu,
                                                   const int32_t *__restrict__ piv, int32_t *__restrict__ perm,
                                                   double *__restrict__ inv)
{
    __shared__ double d[kLuSB][kLuSB + 1];
    extern __shared__ int32_t sidx[];   // n entries, then the interchanges
    const int tid = threadIdx.x;
    if (blockIdx.x == 0) {
        int32_t *sp = sidx + n;
        for (int i = tid; i < n; i += blockDim.x) {
            sidx[i] = i;
            sp[i] = piv[i];
        }
        __syncthreads();
        if (tid == 0)
            for (int k = 0; k < n; ++k) {
                const int32_t p = sp[k], t = sidx[k];
                sidx[k] = sidx[p];
                sidx[p] = t;
            }
        __syncthreads();
        for (int i = tid; i < n; i += blockDim.x) perm[i] = sidx[i];
        return;
    }
    const int blk = blockIdx.x - 1, r0 = blk * kLuSB, lane = tid & 31, upper = tid >> 5;
    for (int e = tid; e < kLuSB * kLuSB; e += blockDim.x) {
        const int i = e / kLuSB, k = e % kLuSB;
        d[i][k] = r0 + i < n && r0 + k < n ? lu[(int64_t)(r0 + i) * n + r0 + k] : (i == k ? 1.0 : 0.0);
    }
    __syncthreads();
    // one warp per triangle, one column of the inverse per lane
    double y[kLuSB];
    if (!upper) {
#pragma unroll
        for (int i = 0; i < kLuSB; ++i) {
            double v = i == lane ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < kLuSB; ++k)
                if (k < i) v = fma(-d[i][k], y[k], v);
            y[i] = v;
        }
    } else {
#pragma unroll
        for (int i = kLuSB - 1; i >= 0; --i) {
            double v = i == lane ? 1.0 : 0.0;
#pragma unroll
            for (int k = 0; k < kLuSB; ++k)
                if (k > i) v = fma(-d[i][k], y[k], v);
            y[i] = v / d[i][i];
        }
    }
    double *o = inv + ((int64_t)blk * 2 + upper) * kLuSB * kLuSB;
#pragma unroll
    for (int i = 0; i < kLuSB; ++i) o[i * kLuSB + lane] = y[i];
}

// x = A^-1 b with the prepared factors; b and x (n, nrhs) row-major.  One CTA per CB columns of
// b, held in shared memory; one warp per row of a 32-row block: the products with the rows solved
// so far and with the inverse of the diagonal block are each a sum over the lanes, so a column's
// arithmetic does not depend on CB or on its neighbours.  Bound by the latency of 2 n / 32 block
// steps (two barriers, a row read and two reductions each); with the interchanges applied one by
// one and 32-step substitutions inside a block a solve of n = 92 took 42 us, of 612 438
// us; here 6.8 and 77 us.
// Sums of CB values over the lanes: lane c < CB returns value c's (CB = 4: the lanes exchange halves
// of the values over their two low bits first, six shuffles instead of twenty).  The additions
// pair the lanes in the same order for every CB.
template <int CB>
__device__ __forceinline__ double lane_sums(const double (&v)[CB], int lane)
{
    static_assert(CB == 1 || CB == 4, "columns per CTA");
    double s;
    if constexpr (CB == 1) {
        s = v[0] + __shfl_xor_sync(0xffffffffu, v[0], 2);
        s += __shfl_xor_sync(0xffffffffu, s, 1);
    } else {
        const bool b1 = lane & 2, b0 = lane & 1;
        const double k0 = b1 ? v[2] : v[0], k1 = b1 ? v[3] : v[1];   // kept, and given to the partner
        const double g0 = b1 ? v[0] : v[2], g1 = b1 ? v[1] : v[3];
        const double h0 = k0 + __shfl_xor_sync(0xffffffffu, g0, 2), h1 = k1 + __shfl_xor_sync(0xffffffffu, g1, 2);
        s = (b0 ? h1 : h0) + __shfl_xor_sync(0xffffffffu, b0 ? h0 : h1, 1);
    }
    s += __shfl_xor_sync(0xffffffffu, s, 4);
    s += __shfl_xor_sync(0xffffffffu, s, 8);
    s += __shfl_xor_sync(0xffffffffu, s, 16);
    return s;
}

// load(row, column): entry of b.
template <int CB, class Load>
__device__ __forceinline__ void lu_solve_columns(int n, const double *__restrict__ lu,
                                                 const int32_t *__restrict__ perm, const double *__restrict__ inv,
                                                 int64_t nrhs, Load load, double *__restrict__ x)
{
    extern __shared__ double xs[];   // [n rounded up to 32][CB]
    __shared__ double part[kLuSB][CB];
    const int tid = threadIdx.x, lane = tid & 31, r = tid >> 5;
    const int64_t c0 = (int64_t)blockIdx.x * CB;
    const int ncol = (int)(nrhs - c0 < CB ? nrhs - c0 : CB);
    const int nblk = (n + kLuSB - 1) / kLuSB;
    for (int i = tid; i < nblk * kLuSB * CB; i += blockDim.x) {
        const int row = i / CB, c = i % CB;
        xs[i] = row < n && c < ncol ? load(perm[row], c0 + c) : 0.0;
    }
    __syncthreads();
    auto step = [&](int blk, int jbeg, int jend, int upper) {
        const int row = blk * kLuSB + r;
        const double di = inv[((int64_t)blk * 2 + upper) * kLuSB * kLuSB + r * kLuSB + lane];
        double acc[CB];
#pragma unroll
        for (int c = 0; c < CB; ++c) acc[c] = 0.0;
        if (row < n) {
            const double *src = lu + (int64_t)row * n;
#pragma unroll 4
            for (int j = jbeg + lane; j < jend; j += 32) {
                const double l = __ldg(src + j);
#pragma unroll
                for (int c = 0; c < CB; ++c) acc[c] = fma(l, xs[j * CB + c], acc[c]);
            }
        }
        const double sum = lane_sums<CB>(acc, lane);
        if (lane < CB) part[r][lane] = xs[row * CB + lane] - sum;
        __syncthreads();
#pragma unroll
        for (int c = 0; c < CB; ++c) acc[c] = di * part[lane][c];
        const double v = lane_sums<CB>(acc, lane);
        if (lane < CB) xs[row * CB + lane] = v;
        __syncthreads();
    };
    for (int blk = 0; blk < nblk; ++blk) step(blk, 0, blk * kLuSB, 0);
    for (int blk = nblk - 1; blk >= 0; --blk) step(blk, (blk + 1) * kLuSB, n, 1);
    for (int i = tid; i < n * CB; i += blockDim.x) {
        const int row = i / CB, c = i % CB;
        if (c < ncol) x[(int64_t)row * nrhs + c0 + c] = xs[i];
    }
}

template <int CB>
__global__ void __launch_bounds__(1024) k_lu_solve_prepared(int n, const double *__restrict__ lu,
                                                            const int32_t *__restrict__ perm,
                                                            const double *__restrict__ inv, int64_t nrhs,
                                                            const double *__restrict__ b, double *__restrict__ x)
{
    lu_solve_columns<CB>(n, lu, perm, inv, nrhs,
                         [&](int row, int64_t c) { return b[(int64_t)row * nrhs + c]; }, x);
}

// Binning and decoupling of many spectra in one launch: right-hand side c is the binned cell c,
// rows band-major with the ncls spectra of a band adjacent (k_bin_cells' sums, entry by entry as
// they are needed).  Cell c: ncls rows of stride ld.
constexpr int kDecoupleCells = 256;
struct Cells {
    const double *c[kDecoupleCells];
};
template <int CB>
__global__ void __launch_bounds__(1024) k_decouple(int n, int ncls, int64_t ld, const __grid_constant__ Cells cells,
                                                   const int32_t *__restrict__ band_ptr,
                                                   const int32_t *__restrict__ band_ells,
                                                   const double *__restrict__ wfl, const double *__restrict__ lu,
                                                   const int32_t *__restrict__ perm, const double *__restrict__ inv,
                                                   int64_t nrhs, double *__restrict__ x)
{
    lu_solve_columns<CB>(n, lu, perm, inv, nrhs,
                         [&](int row, int64_t c) {
                             const int b = row / ncls, q = row - b * ncls;
                             const double *src = cells.c[c] + q * ld;
                             double s = 0.0;
#pragma unroll 4
                             for (int i = band_ptr[b]; i < band_ptr[b + 1]; ++i) {
                                 const int l = band_ells[i];
                                 s += wfl[l] * src[l];
                             }
                             return s;
                         },
                         x);
}

}  // namespace gm

using namespace gm;

extern "C" int gm_pseudo_cl_pairs(int64_t lmax, int64_t npairs, int64_t n1, const double *const *alm1, int64_t n2,
                                  const double *const *alm2, double *const *cls, void *stream)
{
    if (lmax < 0 || npairs < 1 || n1 < 1 || n2 < 1 || n1 * n2 > 65535) return GM_ERR_BAD_SHAPE;
    if (!alm1 || !alm2 || !cls) return GM_ERR_BAD_PTR;
    for (int64_t i = 0; i < npairs; ++i)
        if (!alm1[i] || !alm2[i] || !cls[i]) return GM_ERR_BAD_PTR;
    const int64_t L = lmax + 1, nelem = L * (L + 1) / 2;
    cudaStream_t s = as_stream(stream);
    // fields of one or two components run all their products together; more components as
    // pairs of single rows
    const bool whole = n1 <= 2 && n2 <= 2;
    const int64_t per = whole ? 1 : n1 * n2, total = npairs * per;
    for (int64_t i0 = 0; i0 < total; i0 += kPclPairs) {
        const int64_t cnt = total - i0 < kPclPairs ? total - i0 : kPclPairs;
        PclPairs p;
        for (int64_t i = 0; i < cnt; ++i) {
            const int64_t f = (i0 + i) / per, q = (i0 + i) % per;
            p.a[i] = (const double2 *)alm1[f] + (whole ? 0 : q / n2) * nelem;
            p.b[i] = (const double2 *)alm2[f] + (whole ? 0 : q % n2) * nelem;
            p.out[i] = cls[f] + q * L;
        }
        const int lanes = L <= 512 ? 32 : (L <= 1024 ? 16 : 8);   // by lmax alone: a pair's sums do not depend on the batch
        const dim3 grid((unsigned)((L + lanes - 1) / lanes), (unsigned)cnt);
        auto run = [&](auto k32, auto k16, auto k8) {
            (lanes == 32 ? k32 : (lanes == 16 ? k16 : k8))<<<grid, kPclThreads, 0, s>>>(lmax, p);
        };
        if (!whole || (n1 == 1 && n2 == 1)) run(k_pseudo_cl<1, 1, 32>, k_pseudo_cl<1, 1, 16>, k_pseudo_cl<1, 1, 8>);
        else if (n1 == 1) run(k_pseudo_cl<1, 2, 32>, k_pseudo_cl<1, 2, 16>, k_pseudo_cl<1, 2, 8>);
        else if (n2 == 1) run(k_pseudo_cl<2, 1, 32>, k_pseudo_cl<2, 1, 16>, k_pseudo_cl<2, 1, 8>);
        else run(k_pseudo_cl<2, 2, 32>, k_pseudo_cl<2, 2, 16>, k_pseudo_cl<2, 2, 8>);
        const int st = check_launch("gm_pseudo_cl");
        if (st != GM_OK) return st;
    }
    return GM_OK;
}

extern "C" int gm_pseudo_cl(int64_t lmax, int64_t n1, const double *alm1, int64_t n2,
                            const double *alm2, double *cls, void *stream)
{
    if (!alm1 || !alm2 || !cls) return lmax < 0 || n1 < 1 || n2 < 1 || n1 * n2 > 65535 ? GM_ERR_BAD_SHAPE : GM_ERR_BAD_PTR;
    return gm_pseudo_cl_pairs(lmax, 1, n1, &alm1, n2, &alm2, &cls, stream);
}

extern "C" int gm_coupling_blocks(int64_t lmax, const double *window, int64_t nw, int which,
                                  double *blocks, int64_t *queue, void *stream)
{
    if (lmax < 0 || lmax > 65535 || nw < 0) return GM_ERR_BAD_SHAPE;
    if (which <= 0 || which > 15) return GM_ERR_UNSUPPORTED;
    if (!window || !blocks || !queue) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    const int64_t n = lmax + 1;
    cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(int64_t), s);
    if (e == cudaSuccess) e = cudaMemsetAsync(blocks, 0, sizeof(double) * 4 * n * n, s);
    if (e != cudaSuccess) {
        set_error("gm_coupling_blocks memset", e);
        return GM_ERR_LAUNCH;
    }
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    k_coupling<<<nsm * 8, 128, 0, s>>>(lmax, window, nw, which, blocks,
                                       reinterpret_cast<unsigned long long *>(queue));
    return check_launch("gm_coupling_blocks");
}

extern "C" int64_t gm_coupling_units(int64_t lmax) { return lmax < 0 ? 0 : total_units(lmax); }

extern "C" int gm_coupling_blocks_multi(int64_t njobs, const int64_t *jobs, int64_t nunits,
                                        const double *windows, double *blocks, int64_t *queue,
                                        void *stream)
{
    if (njobs < 1 || nunits < 1) return GM_ERR_BAD_SHAPE;
    if (!jobs || !windows || !blocks || !queue) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    cudaError_t e = cudaMemsetAsync(queue, 0, sizeof(int64_t), s);
    if (e != cudaSuccess) {
        set_error("gm_coupling_blocks_multi memset", e);
        return GM_ERR_LAUNCH;
    }
    int dev = 0, nsm = 148;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev);
    k_coupling_multi<<<nsm * 8, 128, 0, s>>>(njobs, jobs, nunits, windows, blocks,
                                             reinterpret_cast<unsigned long long *>(queue));
    return check_launch("gm_coupling_blocks_multi");
}

extern "C" int gm_coupling_pairs_tt(int64_t lmax, const double *window, int64_t nw,
                                    const int32_t *pairs, int64_t npairs, double *S, void *stream)
{
    if (lmax < 0 || nw < 0 || npairs < 0) return GM_ERR_BAD_SHAPE;
    if (npairs == 0) return GM_OK;
    if (!window || !pairs || !S) return GM_ERR_BAD_PTR;
    k_coupling_pairs_tt<<<(unsigned)((npairs + 127) / 128), 128, 0, as_stream(stream)>>>(
        lmax, window, nw, pairs, npairs, S);
    return check_launch("gm_coupling_pairs_tt");
}

extern "C" int gm_toeplitz_fill(int64_t lmax, int64_t l_toeplitz, int64_t l_exact, int64_t dl_band,
                                const double *S, double *out, void *stream)
{
    if (lmax < 1 || l_toeplitz < 1 || l_exact < 0 || dl_band < 0 || l_exact > l_toeplitz ||
        l_toeplitz >= lmax || dl_band >= lmax || lmax >= 65535)
        return GM_ERR_BAD_SHAPE;
    if (!S || !out) return GM_ERR_BAD_PTR;
    const int64_t n = lmax + 1;
    dim3 grid((unsigned)((n + 127) / 128), (unsigned)n);
    k_toeplitz_fill<<<grid, 128, 0, as_stream(stream)>>>(lmax, l_toeplitz, l_exact, dl_band, S, out);
    return check_launch("gm_toeplitz_fill");
}

// Binning operators are passed in CSR form to support any NmtBin.
extern "C" int gm_bin_coupling_csr(int64_t lmax, int64_t nbands, int ncls, const double *blocks,
                                   const int32_t *band_ptr, const int32_t *band_ells,
                                   const double *wfl, const double *inv_fl, const double *beam,
                                   double *scratch, double *out, void *stream)
{
    if (lmax < 0 || nbands < 1 || nbands > 65535 || (ncls != 1 && ncls != 2 && ncls != 4))
        return GM_ERR_BAD_SHAPE;
    if (!blocks || !band_ptr || !band_ells || !wfl || !inv_fl || !beam || !scratch || !out)
        return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    const int64_t n = lmax + 1, nn = n * n, nb2 = nbands * nbands;
    // eight warps a pair where one would leave the chip idle (nbands <= 48) or walk 64 rows and more
    const bool split = n >= 8 * nbands && (nbands <= 48 || n >= 64 * nbands);
    const int64_t pairs = split ? 1 : kBinWarps;
    const dim3 grid((unsigned)((nbands + pairs - 1) / pairs), (unsigned)nbands);
    auto bin = [&](const double *M, double *to) {
        (split ? k_bin_block<kBinWarps> : k_bin_block<1>)<<<grid, 32 * kBinWarps, 0, s>>>(
            lmax, nbands, M, band_ptr, band_ells, wfl, inv_fl, beam, to);
    };
    // block slots: tt 0, te 1, pp 2, mm 3
    if (ncls == 1) {
        bin(blocks, scratch);
    } else if (ncls == 2) {
        bin(blocks + nn, scratch);
    } else {
        bin(blocks + 2 * nn, scratch);
        bin(blocks + 3 * nn, scratch + nb2);
    }
    const int64_t N = ncls * nbands;
    k_place_binned<<<(unsigned)((N * N + 255) / 256), 256, 0, s>>>(nbands, ncls, scratch, out);
    return check_launch("gm_bin_coupling");
}

extern "C" int gm_bin_cells_csr(int64_t lmax, int64_t nbands, int64_t ncls, const double *cls,
                                const int32_t *band_ptr, const int32_t *band_ells,
                                const double *wfl, double *out, void *stream)
{
    if (lmax < 0 || nbands < 1 || ncls < 1) return GM_ERR_BAD_SHAPE;
    if (!cls || !band_ptr || !band_ells || !wfl || !out) return GM_ERR_BAD_PTR;
    const int64_t tot = nbands * ncls;
    k_bin_cells<<<(unsigned)((tot + 255) / 256), 256, 0, as_stream(stream)>>>(
        lmax, nbands, ncls, cls, band_ptr, band_ells, wfl, out);
    return check_launch("gm_bin_cells");
}

// Shared memory of a panel or of the right-hand sides of a CTA.
constexpr int kLuSmem = 200 * 1024;

// Panel width of the shared-memory panels: the widest of 32, 16, 8, 4 columns that fit (the
// whole matrix up to n = 159), 0 when none does.
static int lu_panel_width(int64_t n)
{
    const int64_t fit = kLuSmem / (8 * (n | 1));
    if (fit >= n) return (int)n;
    for (int kb = kLuPan; kb >= 4; kb /= 2)
        if (fit >= kb) return kb;
    return 0;
}

extern "C" int gm_lu_factor(int64_t n, double *a, int32_t *piv, int32_t *status, void *stream)
{
    if (n < 1 || n > 65535) return GM_ERR_BAD_SHAPE;
    if (!a || !piv || !status) return GM_ERR_BAD_PTR;
    cudaStream_t s = as_stream(stream);
    const int w = lu_panel_width(n);
    if (w == 0) {   // panels in global memory
        cudaError_t e = cudaMemsetAsync(status, 0, sizeof(int32_t), s);
        if (e != cudaSuccess) {
            set_error("gm_lu_factor memset", e);
            return GM_ERR_LAUNCH;
        }
        for (int64_t k0 = 0; k0 < n; k0 += kLuTile) {
            const int64_t k1 = k0 + kLuTile < n ? k0 + kLuTile : n;
            int st = gm_lu_panel(n, a, k0, k1, piv, status, stream);
            if (st == GM_OK && k1 < n) st = gm_lu_trsm(n, a, k0, k1, stream);
            if (st == GM_OK && k1 < n) st = gm_lu_update(n, a, k0, k1, stream);
            if (st != GM_OK) return st;
        }
        return GM_OK;
    }
    const size_t smem = (size_t)w * (n | 1) * sizeof(double);
    const int sa = allow_smem(k_lu_panel_smem, kLuSmem, "gm_lu_factor attr");
    if (sa != GM_OK) return sa;
    for (int64_t k0 = 0; k0 < n;) {
        const int64_t rows = n - k0;
        // one panel in shared memory where the whole matrix fits; else rows in registers, 32 columns
        // of up to 640 rows, 16 of up to 1024, or the widest panel that fits shared memory
        const bool whole = w == n;
        const int width = whole ? w : (rows <= 640 ? 32 : (rows <= 1024 ? 16 : w));
        const int kb = (int)(rows < width ? rows : width);
        const int64_t k1 = k0 + kb;
        const int threads = rows >= 1024 ? 1024 : (int)((rows + 31) / 32 * 32);
        if (!whole && rows <= 640)
            k_lu_panel_reg<32, 640><<<1, threads, 0, s>>>((int)n, (int)k0, kb, a, piv, status);
        else if (!whole && rows <= 1024)
            k_lu_panel_reg<16, 1024><<<1, threads, 0, s>>>((int)n, (int)k0, kb, a, piv, status);
        else
            k_lu_panel_smem<<<1, threads, smem, s>>>((int)n, (int)k0, kb, a, piv, status);
        if (n > kb) k_lu_rest<<<(unsigned)((n - kb + 127) / 128), 128, 0, s>>>((int)n, (int)k0, kb, a, piv);
        if (k1 < n) {
            const int st = gm_lu_update(n, a, k0, k1, stream);
            if (st != GM_OK) return st;
        }
        k0 = k1;
    }
    return check_launch("gm_lu_factor");
}

extern "C" int gm_lu_panel(int64_t n, double *a, int64_t k0, int64_t k1, int32_t *piv,
                           int32_t *status, void *stream)
{
    if (n < 1 || n > 65535 || k0 < 0 || k1 <= k0 || k1 > n) return GM_ERR_BAD_SHAPE;
    if (!a || !piv || !status) return GM_ERR_BAD_PTR;
    k_lu_panel<<<1, 1024, 0, as_stream(stream)>>>(n, k0, k1, a, piv, status);
    return check_launch("gm_lu_panel");
}

extern "C" int gm_lu_trsm(int64_t n, double *a, int64_t k0, int64_t k1, void *stream)
{
    if (n < 1 || n > 65535 || k0 < 0 || k1 <= k0 || k1 > n) return GM_ERR_BAD_SHAPE;
    if (!a) return GM_ERR_BAD_PTR;
    if (k1 == n) return GM_OK;
    k_lu_trsm<<<(unsigned)((n - k1 + 127) / 128), 128, 0, as_stream(stream)>>>(n, k0, k1, a);
    return check_launch("gm_lu_trsm");
}

extern "C" int gm_lu_update(int64_t n, double *a, int64_t k0, int64_t k1, void *stream)
{
    if (n < 1 || k0 < 0 || k1 <= k0 || k1 - k0 > kLuTile || k1 > n) return GM_ERR_BAD_SHAPE;
    if (!a) return GM_ERR_BAD_PTR;
    if (k1 == n) return GM_OK;
    const unsigned t = (unsigned)((n - k1 + kLuTile - 1) / kLuTile);
    k_lu_update<<<dim3(t, t), 256, 0, as_stream(stream)>>>(n, k0, k1, a);
    return check_launch("gm_lu_update");
}

extern "C" int gm_lu_solve(int64_t n, const double *lu, const int32_t *piv, int64_t nrhs,
                           double *b, void *stream)
{
    if (n < 1 || nrhs < 1) return GM_ERR_BAD_SHAPE;
    if (!lu || !piv || !b) return GM_ERR_BAD_PTR;
    const size_t smem = (size_t)n * kLuCB * sizeof(double);
    if (smem <= kLuSmem) {
        // the columns of b fit in shared memory: the blocked solve
        const int sa = allow_smem(k_lu_solve_blk, kLuSmem, "gm_lu_solve attr");
        if (sa != GM_OK) return sa;
        k_lu_solve_blk<<<(unsigned)((nrhs + kLuCB - 1) / kLuCB), 256, smem, as_stream(stream)>>>(n, lu, piv,
                                                                                                nrhs, b);
        return check_launch("gm_lu_solve");
    }
    const int64_t threads = 256, warps_per = threads / 32;
    k_lu_solve<<<(unsigned)((nrhs + warps_per - 1) / warps_per), (unsigned)threads, 0,
                 as_stream(stream)>>>(n, lu, piv, nrhs, b);
    return check_launch("gm_lu_solve");
}

extern "C" int64_t gm_lu_prepared_bytes(int64_t n)
{
    if (n < 1) return 0;
    const int64_t nblk = (n + kLuSB - 1) / kLuSB;
    return nblk * (2 * kLuSB * kLuSB * (int64_t)sizeof(double) + kLuSB * (int64_t)sizeof(int32_t));
}

// The columns of b in shared memory: 4 per CTA up to this many rows.
constexpr int64_t kLuPreparedMax = kLuSmem / (4 * 8);

extern "C" int gm_lu_prepare(int64_t n, const double *lu, const int32_t *piv, void *work, void *stream)
{
    if (n < 1 || n > kLuPreparedMax) return GM_ERR_BAD_SHAPE;
    if (!lu || !piv || !work) return GM_ERR_BAD_PTR;
    const int64_t nblk = (n + kLuSB - 1) / kLuSB;
    double *inv = (double *)work;
    int32_t *perm = (int32_t *)(inv + nblk * 2 * kLuSB * kLuSB);
    const size_t smem = 2 * (size_t)n * sizeof(int32_t);
    const int sa = allow_smem(k_lu_prepare, 2 * (int)kLuPreparedMax * (int)sizeof(int32_t), "gm_lu_prepare attr");
    if (sa != GM_OK) return sa;
    k_lu_prepare<<<(unsigned)(1 + nblk), 64, smem, as_stream(stream)>>>((int)n, lu, piv, perm, inv);
    return check_launch("gm_lu_prepare");
}

extern "C" int gm_lu_solve_prepared(int64_t n, const double *lu, const void *work, int64_t nrhs, const double *b,
                                    double *x, void *stream)
{
    if (n < 1 || n > kLuPreparedMax || nrhs < 1) return GM_ERR_BAD_SHAPE;
    if (!lu || !work || !b || !x || b == x) return GM_ERR_BAD_PTR;
    const int64_t nblk = (n + kLuSB - 1) / kLuSB;
    const double *inv = (const double *)work;
    const int32_t *perm = (const int32_t *)(inv + nblk * 2 * kLuSB * kLuSB);
    // four columns a CTA share every row of the factors; few columns spread over more CTAs
    const bool wide = nrhs > 2 * 148;
    auto kern = wide ? k_lu_solve_prepared<4> : k_lu_solve_prepared<1>;
    const int cb = wide ? 4 : 1;
    const size_t smem = (size_t)nblk * kLuSB * cb * sizeof(double);
    const int sa = allow_smem(kern, kLuSmem, "gm_lu_solve_prepared attr");
    if (sa != GM_OK) return sa;
    kern<<<(unsigned)((nrhs + cb - 1) / cb), 1024, smem, as_stream(stream)>>>((int)n, lu, perm, inv, nrhs, b, x);
    return check_launch("gm_lu_solve_prepared");
}

extern "C" int gm_decouple_cells(int64_t nbands, int64_t ncls, int64_t ncells, const double *const *cells, int64_t ld,
                                 const int32_t *band_ptr, const int32_t *band_ells, const double *wfl,
                                 const double *lu, const void *work, double *x, void *stream)
{
    const int64_t n = nbands * ncls;
    if (nbands < 1 || ncls < 1 || n > kLuPreparedMax || ncells < 1 || ncells > kDecoupleCells || ld < 1)
        return GM_ERR_BAD_SHAPE;
    if (!cells || !band_ptr || !band_ells || !wfl || !lu || !work || !x) return GM_ERR_BAD_PTR;
    Cells c;
    for (int64_t i = 0; i < ncells; ++i) {
        if (!cells[i]) return GM_ERR_BAD_PTR;
        c.c[i] = cells[i];
    }
    const int64_t nblk = (n + kLuSB - 1) / kLuSB;
    const double *inv = (const double *)work;
    const int32_t *perm = (const int32_t *)(inv + nblk * 2 * kLuSB * kLuSB);
    const bool wide = ncells > 148;   // four columns share the rows of the factors
    auto kern = wide ? k_decouple<4> : k_decouple<1>;
    const int cb = wide ? 4 : 1;
    const size_t smem = (size_t)nblk * kLuSB * cb * sizeof(double);
    const int sa = allow_smem(kern, kLuSmem, "gm_decouple_cells attr");
    if (sa != GM_OK) return sa;
    kern<<<(unsigned)((ncells + cb - 1) / cb), 1024, smem, as_stream(stream)>>>(
        (int)n, (int)ncls, ld, c, band_ptr, band_ells, wfl, lu, perm, inv, ncells, x);
    return check_launch("gm_decouple_cells");
}
