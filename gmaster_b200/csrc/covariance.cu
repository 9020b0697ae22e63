// Gaussian covariance of pseudo-C_ell bandpowers in the narrow-kernel approximation
// (gmaster/covariance.py:407-575): every output block X (a pair of spectrum components of
// the two power spectra) is a signed sum of terms
//     cov_X(l1, l2) = sum_t sign_t * (A_t(l1) B_t(l2) + A_t(l2) B_t(l1)) / 2 * Xi_{k_t}(l1, l2)
// with A_t, B_t rows of the best-guess spectra and Xi_k the coupling kernels of the mask
// products.  The host builds the term list from the spins (which kernel and which spectra
// each output block takes); these kernels evaluate it.
//
// k_cov_bands fuses the assembly with the binning of both sides: one CTA per pair of
// bands (p, q) reads the (l1 in p) x (l2 in q) tile of every kernel once and reduces the
// weighted sums of all output blocks, so the unbinned (L x L) blocks are never written.
// k_cov_coupled writes the unbinned blocks (the coupled covariance).

#include "gm_common.cuh"

namespace gm {
namespace {

constexpr int kCovMaxBlocks = 16;   // 4 x 4 components (spin 2 x spin 2)
constexpr int kCovThreads = 256;

struct CovTerms {
    const double *xi;        // (nk, L, L) kernels
    const double *spec;      // (nrows, L) best-guess spectra
    const int32_t *terms;    // (nterm, 3): kernel, row of A, row of B
    const double *signs;     // (nterm,)
    const int32_t *bptr;     // (nblocks + 1,) term range of each output block
};

__device__ __forceinline__ double block_value(const CovTerms &c, int64_t L, int x, int64_t l1,
                                              int64_t l2)
{
    double s = 0.0;
    const int t1 = c.bptr[x + 1];
    for (int t = c.bptr[x]; t < t1; ++t) {
        const int64_t k = c.terms[3 * t], ra = c.terms[3 * t + 1], rb = c.terms[3 * t + 2];
        const double *A = c.spec + ra * L, *B = c.spec + rb * L;
        const double sym = 0.5 * (A[l1] * B[l2] + A[l2] * B[l1]);
        s += c.signs[t] * sym * c.xi[(k * L + l1) * L + l2];
    }
    return s;
}

// Any term table and signs, the indices read on the device (the C entry gm_cov_binned; the
// package takes k_cov_bands).
__global__ void __launch_bounds__(kCovThreads) k_cov_binned(
    int64_t L, int nblocks, CovTerms c, const int32_t *__restrict__ ptr_a,
    const int32_t *__restrict__ ells_a, const double *__restrict__ w_a,
    const int32_t *__restrict__ ptr_b, const int32_t *__restrict__ ells_b,
    const double *__restrict__ w_b, int64_t nbb, double *__restrict__ out, int64_t nba)
{
    __shared__ double red[kCovThreads / 32][kCovMaxBlocks];
    const int64_t p = blockIdx.y, q = blockIdx.x;
    const int a0 = ptr_a[p], n1 = ptr_a[p + 1] - a0;
    const int b0 = ptr_b[q], n2 = ptr_b[q + 1] - b0;
    double acc[kCovMaxBlocks];
#pragma unroll
    for (int x = 0; x < kCovMaxBlocks; ++x) acc[x] = 0.0;
    const int64_t n = (int64_t)n1 * n2;
    for (int64_t e = threadIdx.x; e < n; e += kCovThreads) {
        const int64_t l1 = ells_a[a0 + (int)(e / n2)];
        const int64_t l2 = ells_b[b0 + (int)(e % n2)];
        const double w = w_a[l1] * w_b[l2];
#pragma unroll
        for (int x = 0; x < kCovMaxBlocks; ++x)
            if (x < nblocks) acc[x] += w * block_value(c, L, x, l1, l2);
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int x = 0; x < kCovMaxBlocks; ++x) {
        if (x >= nblocks) break;
        double v = acc[x];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[warp][x] = v;
    }
    __syncthreads();
    if (threadIdx.x < nblocks) {
        double v = 0.0;
#pragma unroll
        for (int w = 0; w < kCovThreads / 32; ++w) v += red[w][threadIdx.x];
        out[((int64_t)threadIdx.x * nba + p) * nbb + q] = v;
    }
}

// Binned covariance of one pair of bands (p, q).  With the band sums
//   T_k(r, s) = sum_{l1 in p, l2 in q} w_a(l1) A_r(l1) Xi_k(l1, l2) w_b(l2) A_s(l2)
// over the spectra rows r, s, output block X is the sum over its terms (k, ra, rb) of
// sign (T_k(ra, rb) + T_k(rb, ra)) / 2.  Per kernel: a kCovTile^2 tile of Xi in shared memory,
// Y(s, l1) = sum_l2 Xi(l1, l2) w_b A_s(l2) by one thread per (s, l1), then T(r, s) += w_a A_r(l1)
// Y(s, l1) by one thread per (r, s): 2 x rows multiply-adds per element of Xi, where evaluating
// every term at every element took up to 160 terms of seven loads each.  Bound by the latency of
// the tile steps (three barriers each).  Spin 2, lmax 1535, 95 bands: 907 us in that
// form, 86 us here.
constexpr int kCovRows = 16;    // spectra rows: four power spectra of up to four components
constexpr int kCovTile = 16;
constexpr int kCovKernels = 8;
constexpr int kCovTerms = 512;
struct CovKernels {
    const double *xi[kCovKernels];
};
struct CovTermTable {
    // kernel | ra << 4 | rb << 8 | negative << 12, by output block
    uint16_t term[kCovTerms];
    uint16_t bptr[kCovMaxBlocks + 1];
};

__global__ void __launch_bounds__(kCovThreads) k_cov_bands(
    int64_t L, int nblocks, int nk, int nrows, const __grid_constant__ CovKernels kern,
    const __grid_constant__ CovTermTable tab, const double *__restrict__ spec, const int32_t *__restrict__ ptr_a,
    const int32_t *__restrict__ ells_a, const double *__restrict__ w_a, const int32_t *__restrict__ ptr_b,
    const int32_t *__restrict__ ells_b, const double *__restrict__ w_b, int64_t nbb, double *__restrict__ out,
    int64_t nba)
{
    __shared__ double xt[kCovTile][kCovTile + 1];               // Xi(l1, l2)
    __shared__ double sa[kCovRows][kCovTile + 1], sb[kCovRows][kCovTile + 1];   // weighted rows at l1 / l2
    __shared__ double y[kCovRows][kCovTile + 1];
    __shared__ double T[kCovKernels][kCovRows][kCovRows];
    static_assert(kCovThreads == kCovTile * kCovTile && kCovThreads == kCovRows * kCovRows, "one thread per entry");
    const int64_t p = blockIdx.y, q = blockIdx.x;
    const int a0 = ptr_a[p], n1 = ptr_a[p + 1] - a0;
    const int b0 = ptr_b[q], n2 = ptr_b[q + 1] - b0;
    const int hi = threadIdx.x / kCovTile, lo = threadIdx.x % kCovTile;
    for (int k = 0; k < nk; ++k) {
        const double *xi = kern.xi[k];
        double t = 0.0;
        for (int i0 = 0; i0 < n1; i0 += kCovTile) {
            double acc = 0.0;
            for (int j0 = 0; j0 < n2; j0 += kCovTile) {
                const int64_t l1 = i0 + hi < n1 ? ells_a[a0 + i0 + hi] : -1, l2 = j0 + lo < n2 ? ells_b[b0 + j0 + lo] : -1;
                xt[hi][lo] = l1 >= 0 && l2 >= 0 ? xi[l1 * L + l2] : 0.0;
                sb[hi][lo] = hi < nrows && l2 >= 0 ? w_b[l2] * spec[hi * L + l2] : 0.0;
                if (j0 == 0) {
                    const int64_t la = i0 + lo < n1 ? ells_a[a0 + i0 + lo] : -1;
                    sa[hi][lo] = hi < nrows && la >= 0 ? w_a[la] * spec[hi * L + la] : 0.0;
                }
                __syncthreads();
#pragma unroll
                for (int e = 0; e < kCovTile; ++e) acc = fma(xt[hi][e], sb[lo][e], acc);   // (l1, s) = (hi, lo)
                __syncthreads();
            }
            y[lo][hi] = acc;
            __syncthreads();
#pragma unroll
            for (int e = 0; e < kCovTile; ++e) t = fma(sa[hi][e], y[lo][e], t);   // (r, s) = (hi, lo)
            __syncthreads();
        }
        T[k][hi][lo] = t;
    }
    __syncthreads();
    for (int x = threadIdx.x >> 5; x < nblocks; x += kCovThreads / 32) {
        // one warp per output block, its terms in a fixed order
        double v = 0.0;
        for (int e = tab.bptr[x] + (threadIdx.x & 31); e < tab.bptr[x + 1]; e += 32) {
            const unsigned d = tab.term[e];
            const unsigned k = d & 15, ra = (d >> 4) & 15, rb = (d >> 8) & 15;
            const double s = 0.5 * (T[k][ra][rb] + T[k][rb][ra]);
            v += d >> 12 ? -s : s;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if ((threadIdx.x & 31) == 0) out[((int64_t)x * nba + p) * nbb + q] = v;
    }
}

__global__ void __launch_bounds__(kCovThreads) k_cov_coupled(int64_t L, int nblocks, CovTerms c,
                                                             double *__restrict__ out)
{
    const int64_t l1 = blockIdx.y;
    const int64_t l2 = (int64_t)blockIdx.x * kCovThreads + threadIdx.x;
    if (l2 >= L) return;
    for (int x = 0; x < nblocks; ++x) out[((int64_t)x * L + l1) * L + l2] = block_value(c, L, x, l1, l2);
}

}  // namespace
}  // namespace gm

using namespace gm;

extern "C" int gm_cov_bands(int64_t lmax, int64_t nblocks, int64_t nk, const double *const *xi, int64_t nrows,
                             const double *spec, const int32_t *terms, const double *signs, const int32_t *block_ptr,
                             int64_t nbands_a, const int32_t *ptr_a, const int32_t *ells_a,
                             const double *w_a, int64_t nbands_b, const int32_t *ptr_b,
                             const int32_t *ells_b, const double *w_b, double *out, void *stream)
{
    if (lmax < 0 || nblocks < 1 || nblocks > kCovMaxBlocks || nbands_a < 1 || nbands_b < 1 ||
        nbands_a > 65535 || nbands_b > (int64_t)INT32_MAX || nk < 0 || nk > kCovKernels || nrows < 1 ||
        nrows > kCovRows)
        return GM_ERR_BAD_SHAPE;
    if (!xi || !spec || !terms || !signs || !block_ptr || !ptr_a || !ells_a || !w_a || !ptr_b ||
        !ells_b || !w_b || !out)
        return GM_ERR_BAD_PTR;
    CovKernels kern{};
    for (int64_t k = 0; k < nk; ++k) {
        if (!xi[k]) return GM_ERR_BAD_PTR;
        kern.xi[k] = xi[k];
    }
    CovTermTable tab{};
    if (block_ptr[0] != 0 || block_ptr[nblocks] > kCovTerms) return GM_ERR_BAD_SHAPE;
    for (int64_t x = 0; x < nblocks; ++x) {
        if (block_ptr[x + 1] < block_ptr[x]) return GM_ERR_BAD_SHAPE;
        tab.bptr[x + 1] = (uint16_t)block_ptr[x + 1];
    }
    for (int32_t t = 0; t < block_ptr[nblocks]; ++t) {
        const int32_t k = terms[3 * t], ra = terms[3 * t + 1], rb = terms[3 * t + 2];
        if (k < 0 || k >= nk || ra < 0 || ra >= nrows || rb < 0 || rb >= nrows) return GM_ERR_BAD_SHAPE;
        if (signs[t] != 1.0 && signs[t] != -1.0) return GM_ERR_UNSUPPORTED;
        tab.term[t] = (uint16_t)(k | ra << 4 | rb << 8 | (signs[t] < 0.0 ? 1 << 12 : 0));
    }
    const dim3 grid((unsigned)nbands_b, (unsigned)nbands_a);
    k_cov_bands<<<grid, kCovThreads, 0, as_stream(stream)>>>(lmax + 1, (int)nblocks, (int)nk, (int)nrows, kern, tab,
                                                              spec, ptr_a, ells_a, w_a, ptr_b, ells_b, w_b, nbands_b,
                                                              out, nbands_a);
    return check_launch("gm_cov_bands");
}

extern "C" int gm_cov_binned(int64_t lmax, int64_t nblocks, const double *xi, const double *spec,
                             const int32_t *terms, const double *signs, const int32_t *block_ptr,
                             int64_t nbands_a, const int32_t *ptr_a, const int32_t *ells_a,
                             const double *w_a, int64_t nbands_b, const int32_t *ptr_b,
                             const int32_t *ells_b, const double *w_b, double *out, void *stream)
{
    if (lmax < 0 || nblocks < 1 || nblocks > kCovMaxBlocks || nbands_a < 1 || nbands_b < 1 ||
        nbands_a > 65535 || nbands_b > (int64_t)INT32_MAX)
        return GM_ERR_BAD_SHAPE;
    if (!xi || !spec || !terms || !signs || !block_ptr || !ptr_a || !ells_a || !w_a || !ptr_b ||
        !ells_b || !w_b || !out)
        return GM_ERR_BAD_PTR;
    const CovTerms c{xi, spec, terms, signs, block_ptr};
    const dim3 grid((unsigned)nbands_b, (unsigned)nbands_a);
    k_cov_binned<<<grid, kCovThreads, 0, as_stream(stream)>>>(
        lmax + 1, (int)nblocks, c, ptr_a, ells_a, w_a, ptr_b, ells_b, w_b, nbands_b, out, nbands_a);
    return check_launch("gm_cov_binned");
}

extern "C" int gm_cov_coupled(int64_t lmax, int64_t nblocks, const double *xi, const double *spec,
                              const int32_t *terms, const double *signs, const int32_t *block_ptr,
                              double *out, void *stream)
{
    if (lmax < 0 || lmax + 1 > 65535 || nblocks < 1 || nblocks > kCovMaxBlocks)
        return GM_ERR_BAD_SHAPE;
    if (!xi || !spec || !terms || !signs || !block_ptr || !out) return GM_ERR_BAD_PTR;
    const CovTerms c{xi, spec, terms, signs, block_ptr};
    const int64_t L = lmax + 1;
    const dim3 grid((unsigned)((L + kCovThreads - 1) / kCovThreads), (unsigned)L);
    k_cov_coupled<<<grid, kCovThreads, 0, as_stream(stream)>>>(L, (int)nblocks, c, out);
    return check_launch("gm_cov_coupled");
}
