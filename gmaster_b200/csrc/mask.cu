// Mask apodisation on the GPU: exact distance from every pixel to the nearest masked pixel,
// then the C1 / C2 tapers or the zeroing step of the "Smooth" type (gmaster/utils.py:61-147,
// where a k-d tree over the masked pixels' unit vectors and healpy's query_disc do this on
// the host).
//
// The search walks HEALPix rings.  Within one ring the chord from a query q to a ring pixel
// grows with |phi - phi_q| (in [0, pi]), so the nearest masked pixel of that ring is the
// first masked pixel met going down from the pixel just below phi_q, or the first met going
// up from the pixel just above it.  k_ring_runs stores both for every pixel (cyclically
// within its ring): prev[p] = the masked pixel at or before p, next[p] = at or after p
// (ring-local indices, -1 for a ring without masked pixels).  k_mask_apodize then visits
// rings outwards from the query's own ring or the nearest one with a masked pixel (k_ring_gaps),
// alternating north and south, two candidates per ring, passing over rings without a masked pixel
// that could improve a pixel of the query's warp, until the latitude alone puts every later ring
// beyond the worst chord that the warp still has.  The result is the exact minimum over all masked pixels, like the
// k-d tree's.
//
// Chords are evaluated as |v_q - v_c|^2 = dz^2 + ds^2 + 4 s_q s_c sin^2(dphi / 2) with
// z = cos(theta), s = sin(theta): the same Euclidean distance between unit vectors, free of
// the cancellation of 2 - 2 v_q.v_c at small separations.

#include "gm_common.cuh"

namespace gm {
namespace {

constexpr int kRunThreads = 512;
constexpr int kApoThreads = 256;
constexpr int kGapThreads = 1024;
constexpr double kTwoPi = 6.283185307179586;   // 2 pi rounded to double, as numpy's 2*np.pi
constexpr double kInvTwoPi = 0.15915494309189535;

// For every word of bits the last non-empty word at or before it and the first at or after it (-1:
// none), by the first two warps of the CTA.
__device__ __forceinline__ void word_neighbours(const unsigned *bits, int nwords, int *before, int *after)
{
    if (threadIdx.x >= 64) return;
    const bool fwd = threadIdx.x < 32;
    const int lane = threadIdx.x & 31;
    int carry = -1;
    for (int base = 0; base < nwords; base += 32) {
        const int k = base + lane, w = fwd ? k : nwords - 1 - k;
        int v = k < nwords && bits[w] ? w : -1;
        for (int o = 1; o < 32; o <<= 1) {
            const int u = __shfl_up_sync(0xffffffffu, v, o);
            if (lane >= o && v < 0) v = u;
        }
        if (v < 0) v = carry;
        if (k < nwords) (fwd ? before : after)[w] = v;
        carry = __shfl_sync(0xffffffffu, v, 31);
    }
}

// One CTA per ring (grid-stride over rings).  The ring's masked pixels become one bit each (a
// ballot per 32 pixels, read coalesced and once); one warp then finds for every word the last
// non-empty word before it and the first after it, and every pixel takes its neighbours from
// its own word or from those two.  Bound by memory (8 bytes read, 8 written a pixel): 105 -> 53 us
// at Nside 1024 against block scans of per-thread chunks.
__global__ void __launch_bounds__(kRunThreads) k_ring_runs(int64_t nside,
                                                           const double *__restrict__ mask,
                                                           int32_t *__restrict__ prev,
                                                           int32_t *__restrict__ next)
{
    extern __shared__ unsigned bits[];   // words of the ring, then the two neighbour lists
    const int t = threadIdx.x, lane = t & 31;
    const int64_t nring = 4 * nside - 1;
    const int wmax = (int)((4 * nside + 31) / 32);
    int *before = reinterpret_cast<int *>(bits + wmax), *after = before + wmax;
    for (int64_t r = blockIdx.x; r < nring; r += gridDim.x) {
        const int n = (int)ring_nphi(nside, r), nwords = (n + 31) / 32;
        const int64_t off = ring_offset(nside, r);
        for (int i = t; i < nwords * 32; i += kRunThreads) {
            const unsigned w = __ballot_sync(0xffffffffu, i < n && mask[off + i] <= 0.0);
            if (lane == 0) bits[i >> 5] = w;
        }
        __syncthreads();
        word_neighbours(bits, nwords, before, after);
        __syncthreads();
        const int lastw = before[nwords - 1], firstw = after[0];
        const int ring_last = lastw < 0 ? -1 : 32 * lastw + 31 - __clz(bits[lastw]);
        const int ring_first = firstw < 0 ? -1 : 32 * firstw + __ffs(bits[firstw]) - 1;
        for (int i = t; i < n; i += kRunThreads) {
            const int w = i >> 5;
            const unsigned own = bits[w];
            const unsigned lo = own & (0xffffffffu >> (31 - (i & 31))), hi = own & (0xffffffffu << (i & 31));
            int p, q;
            if (lo) {
                p = 32 * w + 31 - __clz(lo);
            } else {
                const int u = w > 0 ? before[w - 1] : -1;
                p = u < 0 ? ring_last : 32 * u + 31 - __clz(bits[u]);   // wrap: the ring's last masked pixel
            }
            if (hi) {
                q = 32 * w + __ffs(hi) - 1;
            } else {
                const int u = w + 1 < nwords ? after[w + 1] : -1;
                q = u < 0 ? ring_first : 32 * u + __ffs(bits[u]) - 1;   // wrap: the ring's first masked pixel
            }
            prev[off + i] = p;
            next[off + i] = q;
        }
        __syncthreads();   // every thread has read the words before the next ring rewrites them
    }
}

// Rings from each ring to the nearest one with a masked pixel (0: itself, INT32_MAX: none), one CTA.
// Bound by the latency of the rings' first entries.
__global__ void __launch_bounds__(kGapThreads) k_ring_gaps(int64_t nside, const int32_t *__restrict__ prev,
                                                           int32_t *__restrict__ gaps)
{
    extern __shared__ unsigned bits[];
    const int nring = (int)(4 * nside - 1), nwords = (nring + 31) / 32, t = threadIdx.x;
    int *before = reinterpret_cast<int *>(bits + nwords), *after = before + nwords;
#pragma unroll 4
    for (int j = t; j < nwords * 32; j += kGapThreads) {
        const unsigned w = __ballot_sync(0xffffffffu, j < nring && prev[ring_offset(nside, min(j, nring - 1))] >= 0);
        if ((t & 31) == 0) bits[j >> 5] = w;
    }
    __syncthreads();
    word_neighbours(bits, nwords, before, after);
    __syncthreads();
    for (int j = t; j < nring; j += kGapThreads) {
        const int w = j >> 5;
        const unsigned own = bits[w];
        const unsigned lo = own & (0xffffffffu >> (31 - (j & 31))), hi = own & (0xffffffffu << (j & 31));
        const int wl = lo ? w : (w > 0 ? before[w - 1] : -1), wh = hi ? w : (w + 1 < nwords ? after[w + 1] : -1);
        int d = INT32_MAX;
        if (wl >= 0) d = j - (32 * wl + 31 - __clz(lo ? lo : bits[wl]));
        if (wh >= 0) d = min(d, 32 * wh + __ffs(hi ? hi : bits[wh]) - 1 - j);
        gaps[j] = d;
    }
}

// Ring table rows (each nring doubles): cos theta, sin theta, phi0, 2 pi / nphi, nphi / (2 pi).
struct Rings {
    const double *z, *s, *phi0, *step, *inv;
};

struct Query {
    double z, s, phi;
    double best;   // smallest chord^2 found so far (starts at the search radius, exclusive)
    bool found;
};

// Visit ring jj for query q: false once the ring's latitude alone is out of reach.
__device__ __forceinline__ bool probe(int64_t nside, int64_t jj, const Rings &rg,
                                      const int32_t *__restrict__ prev,
                                      const int32_t *__restrict__ next, Query &q)
{
    const double zc = rg.z[jj], sc = rg.s[jj];
    const double dz = q.z - zc, ds = q.s - sc;
    const double lb = dz * dz + ds * ds;   // chord^2 to the ring point at the same phi
    if (lb >= q.best) return false;
    const int64_t nn = ring_nphi(nside, jj);
    const int64_t off = ring_offset(nside, jj);
    const double phi0 = rg.phi0[jj], step = rg.step[jj];
    const double tpos = (q.phi - phi0) * rg.inv[jj];
    // phi_q < 2 pi + pi/4 and phi0 >= 0, so floor(tpos) lies in [-1, 9 nn / 8]
    int k = (int)floor(tpos);
    if (k < 0) k += (int)nn;
    if (k >= (int)nn) k -= (int)nn;
    k = min(max(k, 0), (int)nn - 1);
    const int32_t a = prev[off + k];
    if (a < 0) return true;   // no masked pixel on this ring
    const int32_t b = next[off + (k + 1 == nn ? 0 : k + 1)];
    const double w = 4.0 * q.s * sc;
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int32_t c = u == 0 ? a : b;
        double dphi = fma((double)c, step, phi0 - q.phi);
        dphi -= kTwoPi * rint(dphi * kInvTwoPi);   // into [-pi, pi]
        // sin(|x|/2) >= |x|/pi on [0, pi]: skip the sine when even that bound loses
        const double rough = lb + w * (dphi * dphi) * (1.0 / (M_PI * M_PI));
        if (rough >= q.best) continue;
        const double h = sin(0.5 * dphi);
        const double d2 = lb + w * h * h;
        if (d2 < q.best) {
            q.best = d2;
            q.found = true;
        }
    }
    return true;
}

// Whether ring jj has a masked pixel that some pixel of ring j between longitudes phi_a and phi_b
// could find within the radius: the longitudes within reach widen [phi_a, phi_b] by
// 2 asin x <= 2 (x + (pi / 2 - 1) x^3) on [0, 1], x^2 = (chord2_max - lb) / w, taken with a margin for its
// single-precision evaluation and one pixel each side.
__device__ __forceinline__ bool ring_in_reach(int64_t nside, int64_t jj, double lb, double w, const Rings &rg,
                                              const int32_t *__restrict__ prev, double phi_a, double phi_b,
                                              double chord2_max)
{
    const int nn = (int)ring_nphi(nside, jj);
    const int32_t *run = prev + ring_offset(nside, jj);
    const float x2 = (float)((chord2_max - lb) / fmax(w, 1e-300)) * 1.0001f;
    if (!(x2 < 1.0f)) return run[0] >= 0;   // the whole ring
    const float x = sqrtf(x2);
    const double reach = 2.0 * 1.0001 * (double)(x + 0.570797f * x * x2);
    const double inv = rg.inv[jj], phi0 = rg.phi0[jj];
    const double a = floor((phi_a - reach - phi0) * inv) - 1.0, b = ceil((phi_b + reach - phi0) * inv) + 1.0;
    if (b - a + 1.0 >= (double)nn) return run[0] >= 0;
    // a >= -2 nn and b <= 3 nn: both lie within a few turns
    int k = (int)b % nn;
    if (k < 0) k += nn;
    const int c = run[k];   // the last masked pixel at or before the right end, cyclically
    if (c < 0) return false;
    const int back = c <= k ? k - c : k - c + nn;
    return back <= (int)(b - a);
}

// mode 0: C1 taper, 1: C2 taper (out = mask * f(x) for unmasked pixels closer than the
// radius, x = sqrt(0.5 d^2 / threshold)); mode 2: zeroing step (out = 0 for masked pixels
// and for pixels closer than the radius to a masked one, else the mask value).
//
// Bound by the instructions of the probes.  A warp takes 32 neighbouring pixels of one ring at a
// time: its lanes first test 32 rings at a time, outwards from the nearest ring with a masked pixel
// (`gaps`, where given, else from the warp's own), for masked pixels within reach of the whole warp,
// and only the rings found are probed per pixel, in the same order.  Most pixels have none: at Nside
// 1024 with a radius of one degree (36 rings) every pixel probed them all, 2.29 ms; 0.38 ms here.
// After every four probes the rings that can no longer improve the worst of the warp's distances are
// dropped: a search on to the radius took 16.9 instead of 0.73 ms with every second pixel masked at
// random at 20 degrees, and one through the empty rings 2.9 instead of 0.12 ms without masked pixels.
// GROUPS pixels a thread: two from Nside 512 on, half the CTAs, 7 % (four: a quarter, 50 % slower, the
// rings' probes of a CTA one after the other).
// The warp's 32 pixels iw ... of ring j (n pixels, gap rings from the nearest one with a masked
// pixel); m: the mask of the thread's pixel i, p its place.
__device__ __forceinline__ void apodize_warp(int64_t nside, const Rings &rg, const int32_t *__restrict__ prev,
                                             const int32_t *__restrict__ next, double chord2_max, double threshold,
                                             int mode, double *__restrict__ out, int64_t j, int64_t n, int64_t iw,
                                             int gap, double m, int64_t p)
{
    const int lane = threadIdx.x & 31;
    const int64_t i = iw + lane, nring = 4 * nside - 1;
    const bool search = i < n && (mode == 2 ? !(m <= 0.0) : m > 0.0);
    if (i < n && !search) out[p] = mode == 2 ? 0.0 : m;
    if (!__any_sync(0xffffffffu, search)) return;
    Query q;
    q.z = rg.z[j];
    q.s = rg.s[j];
    q.phi = fma((double)i, rg.step[j], rg.phi0[j]);
    q.best = search ? chord2_max : 0.0;
    q.found = false;
    double limit = chord2_max;   // worst distance of the warp's pixels: rings beyond improve none
    const double phi_a = fma((double)iw, rg.step[j], rg.phi0[j]);
    const double phi_b = fma((double)(iw + 31 < n ? iw + 31 : n - 1), rg.step[j], rg.phi0[j]);
    // slot 2 d: ring j + d, slot 2 d + 1: ring j - 1 - d
    auto ring_of = [&](int64_t slot) { return (slot & 1) ? j - 1 - (slot >> 1) : j + (slot >> 1); };
    for (int64_t base = gap == 0 ? 0 : 2 * ((int64_t)gap - 1);; base += 32) {
        const int64_t jj = ring_of(base + lane);
        double lb = 5.0;   // beyond every chord
        bool hit = false;
        if (jj >= 0 && jj < nring) {
            const double dz = q.z - rg.z[jj], ds = q.s - rg.s[jj];
            lb = dz * dz + ds * ds;
            if (lb < limit) hit = ring_in_reach(nside, jj, lb, 4.0 * q.s * rg.s[jj], rg, prev, phi_a, phi_b, limit);
        }
        unsigned todo = __ballot_sync(0xffffffffu, hit);
        while (todo) {
            for (int e = 0; e < 4 && todo; ++e) {
                const int64_t ring = ring_of(base + __ffs(todo) - 1);
                todo &= todo - 1;
                if (search) probe(nside, ring, rg, prev, next, q);
            }
            limit = q.best;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) limit = fmax(limit, __shfl_xor_sync(0xffffffffu, limit, o));
            todo &= __ballot_sync(0xffffffffu, lb < limit);
        }
        // latitudes alone put every later ring out of reach (lb grows outwards)
        if (!__any_sync(0xffffffffu, lb < limit)) break;
    }
    if (!search) return;
    if (!q.found) {
        out[p] = m;
        return;
    }
    if (mode == 2) {
        out[p] = 0.0;
        return;
    }
    const double x = sqrt(fmax(0.5 * q.best, 0.0) / threshold);
    const double f = mode == 0 ? x - sin(kTwoPi * x) / kTwoPi : 0.5 * (1.0 - cos(M_PI * x));
    out[p] = m * f;
}

template <int GROUPS>
__global__ void __launch_bounds__(kApoThreads) k_mask_apodize(
    int64_t nside, Rings rg, const double *__restrict__ mask,
    const int32_t *__restrict__ prev, const int32_t *__restrict__ next, const int32_t *__restrict__ gaps,
    double chord2_max, double threshold, int mode, double *__restrict__ out)
{
    const int64_t j = blockIdx.y, n = ring_nphi(nside, j), off = ring_offset(nside, j);
    const int64_t i0 = (int64_t)blockIdx.x * GROUPS * kApoThreads + threadIdx.x;
    double m[GROUPS];
#pragma unroll
    for (int e = 0; e < GROUPS; ++e) m[e] = i0 + e * kApoThreads < n ? mask[off + i0 + e * kApoThreads] : 0.0;
    const int gap = gaps ? gaps[j] : 0;
#pragma unroll
    for (int e = 0; e < GROUPS; ++e) {
        const int64_t i = i0 + e * kApoThreads, iw = i - (threadIdx.x & 31);
        if (iw >= n) return;
        if (gap != INT32_MAX) apodize_warp(nside, rg, prev, next, chord2_max, threshold, mode, out, j, n, iw, gap, m[e], off + i);
        else if (i < n) out[off + i] = m[e];   // no masked pixel anywhere
    }
}

}  // namespace
}  // namespace gm

using namespace gm;

extern "C" int gm_mask_ring_runs(int64_t nside, const double *mask, int32_t *prev, int32_t *next,
                                 void *stream)
{
    if (nside < 1 || nside > 16384) return GM_ERR_BAD_SHAPE;
    if (!mask || !prev || !next) return GM_ERR_BAD_PTR;
    const int64_t nring = 4 * nside - 1;
    const int grid = (int)(nring < 592 ? nring : 592);
    const size_t smem = 3 * (size_t)((4 * nside + 31) / 32) * sizeof(int);   // 24 KB at Nside 16384
    k_ring_runs<<<grid, kRunThreads, smem, as_stream(stream)>>>(nside, mask, prev, next);
    return check_launch("gm_mask_ring_runs");
}

extern "C" int gm_mask_ring_gaps(int64_t nside, const int32_t *prev, int32_t *gaps, void *stream)
{
    if (nside < 1 || nside > 16384) return GM_ERR_BAD_SHAPE;
    if (!prev || !gaps) return GM_ERR_BAD_PTR;
    const size_t smem = 3 * (size_t)((4 * nside + 30) / 32) * sizeof(int);   // 24 KB at Nside 16384
    k_ring_gaps<<<1, kGapThreads, smem, as_stream(stream)>>>(nside, prev, gaps);
    return check_launch("gm_mask_ring_gaps");
}

extern "C" int gm_mask_apodize(int64_t nside, const double *ring_table, const double *mask,
                               const int32_t *prev, const int32_t *next, double chord2_max,
                               double threshold, int mode, double *out, void *stream)
{
    return gm_mask_apodize_gaps(nside, ring_table, mask, prev, next, nullptr, chord2_max, threshold, mode, out, stream);
}

extern "C" int gm_mask_apodize_gaps(int64_t nside, const double *ring_table, const double *mask,
                                    const int32_t *prev, const int32_t *next, int32_t *gaps,
                                    double chord2_max, double threshold, int mode, double *out, void *stream)
{
    if (nside < 1 || nside > 16384) return GM_ERR_BAD_SHAPE;
    if (!ring_table || !mask || !prev || !next || !out) return GM_ERR_BAD_PTR;
    if (mode < 0 || mode > 2) return GM_ERR_UNSUPPORTED;
    if (!(chord2_max > 0.0) || (mode != 2 && !(threshold > 0.0))) return GM_ERR_BAD_SHAPE;
    const int64_t nring = 4 * nside - 1;
    // below Nside 512 the table of the nearest rings (5 us) takes longer than the few rings that it
    // passes over, and half the CTAs would not fill the chip several times
    const bool large = nside >= 512;
    if (!large) gaps = nullptr;
    if (gaps) {
        const int st = gm_mask_ring_gaps(nside, prev, gaps, stream);
        if (st != GM_OK) return st;
    }
    const int64_t per = (large ? 2 : 1) * kApoThreads;
    const dim3 grid((unsigned)((4 * nside + per - 1) / per), (unsigned)nring);
    const Rings rg{ring_table, ring_table + nring, ring_table + 2 * nring, ring_table + 3 * nring,
                   ring_table + 4 * nring};
    (large ? k_mask_apodize<2> : k_mask_apodize<1>)<<<grid, kApoThreads, 0, as_stream(stream)>>>(nside, rg, mask, prev, next, gaps,
                                                                 chord2_max, threshold, mode, out);
    return check_launch("gm_mask_apodize");
}
