// One-field Legendre / Wigner-d passes in mixed precision, SIMT, sm_100a: spin 0 and spin 2
// rows in single precision restarted every 128 rows from the checkpoint tables of
// legendre_ck.cu, contracted against a few maps in registers.
//
// Rows.  With r_l = 1 / alpha_l the normalised three-term recurrence
//     v_{l+1} = alpha_{l+1} (x - c_{l+1}) v_l - (alpha_{l+1} / alpha_l) v_{l-1}
// (beta = alpha_{l+1} / alpha_l exactly) reads, with D_l = v_l - v_{l-1} = alpha_l d_l,
//     d_{l+1} = d_l + ((x - 1) + e_{l+1}) v_l,   e_l = 1 - r_{l-1} - r_l - c_l,
//     v_{l+1} = v_l + alpha_{l+1} d_{l+1}:
// the difference form of legendre_ck.cu (each rounding stays unamplified near the poles and
// turning points) in three operations a row instead of four, with two coefficients.  Both
// hemispheres come from the northern rows (the hemisphere fold of legendre.cu).
//
// Packing.  All arithmetic is on pairs of floats (fma.rn.f32x2: two FMAs per issue slot; the
// FMA rate is that of scalar code, 128 a clock and SM, but at half the issue slots, which the
// reduction's selects, adds and loads take).  A pair is two lanes of one warp for spin 0, and
// the two row variants s' = -2, +2 of one lane for spin 2.  There the contraction takes their
// sum F = v^- + v^+ and difference G = v^- - v^+ (two scalar additions a row and lane):
//     -2 E_l = sum  F Q_p + i G U_d,    -2 B_l = sum  F U_p - i G Q_d,
// p the hemispheres' sum and d their difference where l + m is even, the other way round where
// it is odd: four packed FMAs of (F, G), for odd rows of (G, F), whose two halves are added
// once per block of rows.  E and B are never formed from each other's rounded values: at m = 0
// (G = 0) E takes Q alone and B takes U alone, and elsewhere a B far below E carries the
// rounding of the products G Q only.  Summing 2a and -2a instead (P = Q + iU, M = Q - iU, no
// F and G) takes 3 % less time (field, spin 2, Nside 512: 6.8 against 7.0 ms) and leaves the
// rounding of E in B: with U = 1e-3 Q the error of B at m = 0, Nside 512, is 7e-5 of B there, 3e-7
// here.
//
// Bound and split.  The FMA pipe: (3 + 2 NC) packed FMAs per row and two lanes for spin 0, 7 and
// two additions per row and lane for spin 2, plus one shuffle per row, value and thread in the
// analysis (the shuffle unit takes one instruction a clock and SM, a quarter of the FMA issue
// rate, so a thread sums its 2R or R lanes first).  At Nside 512 the pipe is 56-62 % busy (a packed
// FMA of three different operands issues at 1.37 a clock and SM instead of 2: the register file's
// bandwidth), IPC 1.8-2.2.  Against the four-operation scalar rows with a warp tree per 32
// values: analysis / synthesis at Nside 2048 40.6 / 25.2 -> 17.0 / 14.0 ms (spin 0), at Nside
// 512 2.37 / 1.32 -> 1.04 / 0.77 ms (spin 2).  A CTA is up to eight warps of one order m; a warp's
// lanes are contiguous and it skips the segments whose checkpoint states are zero on all of
// them.
//
// Replaces gmaster/_native/cuda/march_v2.cu:155-407 for the one-field passes.
#include <math.h>

#include "gm_common.cuh"

namespace gm {
namespace rows {

using u64 = unsigned long long;

constexpr int kSeg = 128;      // rows per checkpoint segment

// Most warps of a CTA: four, and eight where they then hold every lane of Nside 512 (each alm
// receives one addition, in a fixed order).  Eight measured 5 to 9 % slower at Nside 1024 and
// 2048, where the lanes take several CTAs either way: rows_warps keeps to four there.
__host__ __device__ constexpr int max_warps(int spin, int r) { return spin == 2 && r == 4 ? 8 : 4; }

__device__ __forceinline__ u64 pack(float a, float b)
{
    u64 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack(u64 p, float &a, float &b)
{
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(p));
}
__device__ __forceinline__ u64 fma2(u64 a, u64 b, u64 c)
{
    u64 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ u64 add2(u64 a, u64 b)
{
    u64 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ u64 mul2(u64 a, u64 b)
{
    u64 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}

// Checkpoint tables: segment k of order m starts at row l0 + 128 k; per (segment, lane) the
// scaled pre-state (v_{l-1}, D_l) and its shift n (actual = stored * 2^(-64 n)).  Variant 0:
// s' = 0 (spin 0) or -2; variant 1: s' = +2.
struct Tab {
    const int64_t *segoff;
    const float2 *ck[2];
    const uint8_t *cn[2];
    // optional (NULL: every segment active): per segment, bit g set when a lane of the
    // 64-lane group g has a non-zero stored state (legendre_ck.cu:gm_ck_masks)
    const u64 *mask[2];
};

// Lane groups of segment `seg` with a non-zero state of either variant (all without masks;
// masks exist up to 4096 lanes).
__device__ __forceinline__ u64 active_groups(const Tab &tab, int nvar, int64_t seg)
{
    if (!tab.mask[0]) return ~0ull;
    u64 mk = __ldg(tab.mask[0] + seg);
    if (nvar > 1 && tab.mask[1]) mk |= __ldg(tab.mask[1] + seg);
    return mk;
}

// Mask bits of the 64-lane groups that lanes [j0, j1) touch; groups past 63 (no masks there)
// count as bit 63.
__device__ __forceinline__ u64 group_bits(int64_t j0, int64_t j1)
{
    if (j1 <= j0) return 0ull;
    const int g0 = (int)((j0 >> 6) < 63 ? j0 >> 6 : 63), g1 = (int)(((j1 - 1) >> 6) < 63 ? (j1 - 1) >> 6 : 63);
    const u64 hi = g1 >= 63 ? ~0ull : ((1ull << (g1 + 1)) - 1ull);
    return hi & ~((1ull << g0) - 1ull);
}

// r_l = 1 / alpha_l, zero at l = max(m, s).
__device__ __forceinline__ double inv_alpha(int l, int m, int s)
{
    const double dl = l, dm = m, ds = s;
    if (s == 0) return sqrt((dl * dl - dm * dm) / (4.0 * dl * dl - 1.0));
    return sqrt((dl * dl - dm * dm) * (dl * dl - ds * ds) / (4.0 * dl * dl - 1.0)) / dl;
}

// Coefficients of the step from row l to row l + 1: (e of s' = -s, e of s' = +s, alpha, alpha)
// (spin 0: the two e are equal, one for each lane of a pair).
__device__ __forceinline__ float4 step_coef(int l, int m, int s)
{
    const double r0 = inv_alpha(l, m, s), r1 = inv_alpha(l + 1, m, s);
    const double e = 1.0 - r0 - r1;
    const double c = s != 0 ? (double)s * m / ((double)l * (l + 1)) : 0.0;
    const float a = (float)(1.0 / r1);
    return make_float4((float)(e + c), (float)(e - c), a, a);
}

// Four floats of an array aligned to 16 bytes (wide) or to its elements.
__device__ __forceinline__ float4 load4(const float *p, bool wide)
{
    return wide ? *reinterpret_cast<const float4 *>(p) : make_float4(p[0], p[1], p[2], p[3]);
}
__device__ __forceinline__ void store4(float *p, float4 v, bool wide)
{
    if (wide) {
        *reinterpret_cast<float4 *>(p) = v;
    } else {
        p[0] = v.x;
        p[1] = v.y;
        p[2] = v.z;
        p[3] = v.w;
    }
}

__device__ __forceinline__ int64_t alm_index(int64_t lmax, int64_t l, int64_t m)
{
    return m * (2 * lmax + 1 - m) / 2 + l;
}

// The R packed row states of a thread: y = x - 1 rounded to single precision, the rows v and
// their scaled differences d.  The rounding of y is one direction for all rows of a lane (a
// shift of the lane by up to 2^-25 tan(theta / 2), the largest error of a 128-row segment):
// what it leaves off, eight rows' worth at a time, is added to d before every eighth row
// (`correct`, the factors in shared memory).  Lane of unit u, half h: spin 0
// jw + (2u + h) 32 + lane, spin 2 jw + 32 u + lane (the halves are the two variants).
template <int SPIN, int R> struct Rows {
    u64 y[R], v[R], d[R];
    int n[R];   // shifts of the two halves (low and high byte)

    static constexpr int kLanes = (SPIN == 0 ? 64 : 32) * R;   // lanes of a warp

    static __device__ __forceinline__ int64_t lane_of(int64_t jw, int u, int h, int lane)
    {
        return SPIN == 0 ? jw + (2 * u + h) * 32 + lane : jw + 32 * u + lane;
    }

    __device__ __forceinline__ void correct(const u64 *dy)
    {
#pragma unroll
        for (int u = 0; u < R; ++u) d[u] = fma2(dy[u * blockDim.x + threadIdx.x], v[u], d[u]);
    }

    // `dy` (R x blockDim pairs in shared memory) receives 8 (x - 1 - y).
    __device__ __forceinline__ void geometry(const double *__restrict__ geom, int64_t nlanes, int64_t jw, int lane,
                                             u64 *dy)
    {
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const int64_t j0 = lane_of(jw, u, 0, lane), j1 = lane_of(jw, u, 1, lane);
            const double x0 = j0 < nlanes ? geom[j0] - 1.0 : 0.0, x1 = j1 < nlanes ? geom[j1] - 1.0 : 0.0;
            const float y0 = (float)x0, y1 = (float)x1;
            y[u] = pack(y0, y1);
            dy[u * blockDim.x + threadIdx.x] = pack((float)(8.0 * (x0 - y0)), (float)(8.0 * (x1 - y1)));
        }
    }

    // State at the first row ls of segment seg (r = r_ls): v = v_pre + D, d = D r.  Returns
    // whether a lane of the warp is shifted.
    __device__ __forceinline__ bool start(const Tab &tab, int64_t seg, int64_t nlanes, int64_t jw, int lane, float r)
    {
        int any = 0;
#pragma unroll
        for (int u = 0; u < R; ++u) {
            float vv[2], dd[2];
            int nn[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int q = SPIN == 0 ? 0 : h;
                const int64_t j = lane_of(jw, u, h, lane);
                float2 st = make_float2(0.f, 0.f);
                nn[h] = 0;
                if (j < nlanes) {
                    st = __ldg(tab.ck[q] + seg * nlanes + j);
                    nn[h] = __ldg(tab.cn[q] + seg * nlanes + j);
                }
                vv[h] = st.x + st.y;
                dd[h] = st.y * r;
            }
            v[u] = pack(vv[0], vv[1]);
            d[u] = pack(dd[0], dd[1]);
            n[u] = nn[0] | (nn[1] << 8);
            any |= n[u];
        }
        return __any_sync(0xffffffffu, any != 0);
    }

    // Emission factors 2^(-64 n) of the shifted lanes (n >= 2: zero).
    __device__ __forceinline__ u64 factor(int u) const
    {
        auto f = [](int k) { return k == 0 ? 1.0f : (k == 1 ? 0x1p-64f : 0.0f); };
        return pack(f(n[u] & 255), f(n[u] >> 8));
    }

    // Shifted lanes past 2^48 move to the next shift (8 rows grow a value by at most 2^63:
    // alpha <= sqrt(2m) + 1 at Nside <= 8192).
    __device__ __forceinline__ void renormalise()
    {
#pragma unroll
        for (int u = 0; u < R; ++u) {
            if (n[u] == 0) continue;
            float a, b, da, db;
            unpack(v[u], a, b);
            unpack(d[u], da, db);
            if ((n[u] & 255) && fabsf(a) > 0x1p48f) {
                a *= 0x1p-64f;
                da *= 0x1p-64f;
                n[u] -= 1;
            }
            if ((n[u] >> 8) && fabsf(b) > 0x1p48f) {
                b *= 0x1p-64f;
                db *= 0x1p-64f;
                n[u] -= 256;
            }
            v[u] = pack(a, b);
            d[u] = pack(da, db);
        }
    }

    __device__ __forceinline__ bool shifted() const
    {
        int any = 0;
#pragma unroll
        for (int u = 0; u < R; ++u) any |= n[u];
        return __any_sync(0xffffffffu, any != 0);
    }

    // Spin 2: sum and difference of the two variants' values, in this order (even rows) or the
    // other (odd rows).
    static __device__ __forceinline__ u64 variant_sums(u64 val, bool odd)
    {
        float a, b;
        unpack(val, a, b);
        return odd ? pack(a - b, a + b) : pack(a + b, a - b);
    }

    __device__ __forceinline__ void step(int u, u64 e, u64 al)
    {
        const u64 C = add2(y[u], e);
        d[u] = fma2(C, v[u], d[u]);
        v[u] = fma2(al, d[u], v[u]);
    }
};

__device__ __forceinline__ void load_coef(const float4 *c, u64 &e, u64 &al)
{
    const ulonglong2 q = *reinterpret_cast<const ulonglong2 *>(c);
    e = q.x;
    al = q.y;
}

// Sum of each of the V values of all 32 threads: thread t returns value t % V.
template <int V>
__device__ __forceinline__ float reduce_scatter(float (&v)[V], int lane)
{
#pragma unroll
    for (int h = V / 2; h >= 1; h >>= 1) {
        const bool upper = (lane & h) != 0;
#pragma unroll
        for (int i = 0; i < h; ++i) {
            const float send = upper ? v[i] : v[i + h];
            const float keep = upper ? v[i + h] : v[i];
            v[i] = keep + __shfl_xor_sync(0xffffffffu, send, h);
        }
    }
    float r = v[0];
#pragma unroll
    for (int h = V; h < 32; h <<= 1) r += __shfl_xor_sync(0xffffffffu, r, h);
    return r;
}

// ---------------------------------------------------------------- analysis

// Eight rows of one warp: the row values times the right-hand sides, summed over the warp's
// lanes into red[8 NV] (value v of row s at s NV + v).  rh[u][.]: spin 0, per map Sum re, im
// and Diff re, im (each two lanes); spin 2, the factors of (F, G) that give E re, E im, B re,
// B im on even rows, and of (G, F) for -(B im), B re, E im, -(E re) on odd rows.
template <int SPIN, int NC, int R, bool SCALED>
__device__ __forceinline__ void ana8(Rows<SPIN, R> &w, const u64 (&rh)[R][4 * NC], const float4 *__restrict__ cf,
                                     float *__restrict__ red, int lane)
{
    using W = Rows<SPIN, R>;
    constexpr int NV = SPIN == 0 ? 2 * NC : 4;
    constexpr int V = NV == 16 ? 32 : 16;
    constexpr int RB = V / NV;
    static_assert(RB % 2 == 0 && 8 % RB == 0, "row parity is fixed by the row index");
    u64 sc[R];
    if (SCALED) {
#pragma unroll
        for (int u = 0; u < R; ++u) sc[u] = w.factor(u);
    }
#pragma unroll 1
    for (int i = 0; i < 8; i += RB) {
        u64 acc[V];
#pragma unroll
        for (int q = 0; q < V; ++q) acc[q] = 0ull;
#pragma unroll
        for (int s = 0; s < RB; ++s) {
            u64 e, al;
            load_coef(cf + i + s, e, al);
#pragma unroll
            for (int u = 0; u < R; ++u) {
                const u64 val = SCALED ? mul2(w.v[u], sc[u]) : w.v[u];
                if (SPIN == 0) {
#pragma unroll
                    for (int c = 0; c < NC; ++c) {
                        acc[s * NV + 2 * c] = fma2(val, rh[u][4 * c + 2 * (s & 1)], acc[s * NV + 2 * c]);
                        acc[s * NV + 2 * c + 1] = fma2(val, rh[u][4 * c + 2 * (s & 1) + 1], acc[s * NV + 2 * c + 1]);
                    }
                } else {
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        u64 &a = acc[s * 4 + ((s & 1) ? 3 - q : q)];
                        a = fma2(W::variant_sums(val, s & 1), rh[u][q], a);
                    }
                }
                w.step(u, e, al);
            }
        }
        float out[V];
#pragma unroll
        for (int q = 0; q < V; ++q) {
            float a, b;
            unpack(acc[q], a, b);
            const int s = q / NV, k = q % NV;
            out[q] = SPIN == 2 && (s & 1) && (k == 0 || k == 3) ? -a - b : a + b;
        }
        const float tot = reduce_scatter<V>(out, lane);
        if (lane < V) red[i * NV + lane] = tot;
    }
    if (SCALED) w.renormalise();
}

// Resident CTAs asked for: four of one spin-0 map at R = 4 (128 registers; 139 and three CTAs
// measured 18.0 instead of 16.9 ms at Nside 2048), two of eight warps of spin 2 at R = 4 (122
// registers; 172 and one CTA took 7.9 instead of 6.9 ms at Nside 1024, 1.31 instead of 1.04 at 512).
__host__ __device__ constexpr int ana_ctas(int spin, int nc, int r)
{
    return spin == 0 && nc == 1 && r == 4 ? 4 : (spin == 2 && r == 4 ? 2 : 1);
}

template <int SPIN, int NC, int R>
__global__ void __launch_bounds__(32 * max_warps(SPIN, R), ana_ctas(SPIN, NC, R)) k_rows_ana(int64_t nside, int64_t lmax, int64_t ncomp,
                                                          const double *__restrict__ geom,
                                                          const float *__restrict__ rhs, bool wide,
                                                          double *__restrict__ alm, double scale, Tab tab)
{
    constexpr int NV = SPIN == 0 ? 2 * NC : 4;
    constexpr int NVAR = SPIN == 0 ? 1 : 2;
    using W = Rows<SPIN, R>;
    __shared__ float4 cf[kSeg];
    __shared__ u64 sdy[R * 32 * max_warps(SPIN, R)];
    __shared__ float red[max_warps(SPIN, R)][kSeg * NV];
    const int64_t L = lmax + 1, nlanes = 2 * nside, nelem = L * (L + 1) / 2;
    const int m = blockIdx.y, l0 = m > SPIN ? m : SPIN;
    if (l0 > lmax) return;
    const int64_t c0 = (int64_t)blockIdx.z * (SPIN == 0 ? NC : 2);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t jb = (int64_t)blockIdx.x * nw * W::kLanes, jw = jb + warp * W::kLanes;

    W w;
    w.geometry(geom, nlanes, jw, lane, sdy);
    u64 rh[R][4 * NC];
#pragma unroll
    for (int u = 0; u < R; ++u) {
        if (SPIN == 0) {
            const int64_t j0 = W::lane_of(jw, u, 0, lane), j1 = W::lane_of(jw, u, 1, lane);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float4 a = make_float4(0.f, 0.f, 0.f, 0.f), b = a;
                if (c0 + c < ncomp) {
                    const float *src = rhs + 4 * ((int64_t)m * nlanes * ncomp + c0 + c);
                    if (j0 < nlanes) a = load4(src + 4 * j0 * ncomp, wide);
                    if (j1 < nlanes) b = load4(src + 4 * j1 * ncomp, wide);
                }
                rh[u][4 * c] = pack(a.x, b.x);
                rh[u][4 * c + 1] = pack(a.y, b.y);
                rh[u][4 * c + 2] = pack(a.z, b.z);
                rh[u][4 * c + 3] = pack(a.w, b.w);
            }
        } else {
            const int64_t j = W::lane_of(jw, u, 0, lane);
            float4 q = make_float4(0.f, 0.f, 0.f, 0.f), p = q;
            if (j < nlanes) {
                const float *src = rhs + 4 * (((int64_t)m * nlanes + j) * ncomp + c0);
                q = load4(src, wide);
                p = load4(src + 4, wide);
            }
            if ((l0 + m) & 1) {   // the segments' even rows have odd l + m: Sum and Diff change places
                q = make_float4(q.z, q.w, q.x, q.y);
                p = make_float4(p.z, p.w, p.x, p.y);
            }
            rh[u][0] = pack(q.x, -p.w);
            rh[u][1] = pack(q.y, p.z);
            rh[u][2] = pack(p.x, q.w);
            rh[u][3] = pack(p.y, -q.z);
        }
    }

    const int nseg = (int)((L - l0 + kSeg - 1) / kSeg);
    const int64_t s0 = tab.segoff[m];
    const u64 mine = group_bits(jw, jw + W::kLanes < nlanes ? jw + W::kLanes : nlanes);
    for (int k = 0; k < nseg; ++k) {
        const u64 act = active_groups(tab, NVAR, s0 + k);
        const int64_t je = jb + nw * W::kLanes < nlanes ? jb + nw * W::kLanes : nlanes;
        if (!(act & group_bits(jb, je))) continue;   // zero rows on all lanes of this CTA
        const int lb = l0 + kSeg * k;
        const int nrow = (int)(L - lb < kSeg ? L - lb : kSeg);
        __syncthreads();   // the previous segment's sums are read
        for (int i = threadIdx.x; i < kSeg; i += blockDim.x)
            cf[i] = i < nrow ? step_coef(lb + i, m, SPIN) : make_float4(0.f, 0.f, 0.f, 0.f);
        const bool on = (act & mine) != 0ull;
        bool scaled = false;
        if (on) scaled = w.start(tab, s0 + k, nlanes, jw, lane, (float)inv_alpha(lb, m, SPIN));
        __syncthreads();
        if (on) {
#pragma unroll 1
            for (int i = 0; i < nrow; i += 8) {
                w.correct(sdy);
                if (scaled) {
                    ana8<SPIN, NC, R, true>(w, rh, cf + i, red[warp] + i * NV, lane);
                    scaled = w.shifted();
                } else {
                    ana8<SPIN, NC, R, false>(w, rh, cf + i, red[warp] + i * NV, lane);
                }
            }
        }
        __syncthreads();
        for (int i = threadIdx.x; i < nrow; i += blockDim.x) {
            double sv[NV];
#pragma unroll
            for (int q = 0; q < NV; ++q) sv[q] = 0.0;
            for (int g = 0; g < nw; ++g) {
                const int64_t ja = jb + g * W::kLanes, jz = ja + W::kLanes < nlanes ? ja + W::kLanes : nlanes;
                if (!(act & group_bits(ja, jz))) continue;
#pragma unroll
                for (int q = 0; q < NV; ++q) sv[q] += (double)red[g][i * NV + q];
            }
            const int64_t idx = alm_index(lmax, lb + i, m);
            if (SPIN == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    if (c0 + c < ncomp) {
                        double *a = alm + 2 * ((c0 + c) * nelem + idx);
                        atomicAdd(a, scale * sv[2 * c]);
                        atomicAdd(a + 1, scale * sv[2 * c + 1]);
                    }
                }
            } else {
                double *e = alm + 2 * (c0 * nelem + idx), *b = e + 2 * nelem;
                const double hs = -0.5 * scale;
                atomicAdd(e, hs * sv[0]);
                atomicAdd(e + 1, hs * sv[1]);
                atomicAdd(b, hs * sv[2]);
                atomicAdd(b + 1, hs * sv[3]);
            }
        }
    }
}

// ---------------------------------------------------------------- synthesis

// Eight rows of one warp added to the accumulators.  aw[row][.]: spin 0, per map (re, re, im,
// im); spin 2, the factors of (F, G) in Q re, Q im and U re, U im (even rows; odd rows of (G, F)).
// acc of spin 2: (Sum, Diff) of Q re, Q im, U re, U im: F of an even row and G of an odd one go
// to the hemispheres' sum, the others to their difference.
template <int SPIN, int NC, int R, bool SCALED>
__device__ __forceinline__ void syn8(Rows<SPIN, R> &w, u64 (&acc)[R][4 * NC], const float4 *__restrict__ cf,
                                     const float4 *__restrict__ aw)
{
    using W = Rows<SPIN, R>;
    constexpr int NA = SPIN == 0 ? NC : 2;
    u64 sc[R];
    if (SCALED) {
#pragma unroll
        for (int u = 0; u < R; ++u) sc[u] = w.factor(u);
    }
#pragma unroll
    for (int s = 0; s < 8; ++s) {
        u64 e, al;
        load_coef(cf + s, e, al);
        u64 a[2 * NA];
#pragma unroll
        for (int c = 0; c < NA; ++c) load_coef(aw + s * NA + c, a[2 * c], a[2 * c + 1]);
#pragma unroll
        for (int u = 0; u < R; ++u) {
            const u64 val = SCALED ? mul2(w.v[u], sc[u]) : w.v[u];
            if (SPIN == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    u64 *o = &acc[u][4 * c + 2 * (s & 1)];   // even rows: Sum part, odd rows: Diff part
                    o[0] = fma2(val, a[2 * c], o[0]);
                    o[1] = fma2(val, a[2 * c + 1], o[1]);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) acc[u][q] = fma2(W::variant_sums(val, s & 1), a[q], acc[u][q]);
            }
            w.step(u, e, al);
        }
    }
    if (SCALED) w.renormalise();
}

template <int SPIN, int NC, int R>
__global__ void __launch_bounds__(32 * max_warps(SPIN, R)) k_rows_syn(int64_t nside, int64_t lmax, int64_t ncomp,
                                                          const double *__restrict__ geom,
                                                          const double *__restrict__ alm,
                                                          float *__restrict__ syn, bool wide, Tab tab)
{
    constexpr int NVAR = SPIN == 0 ? 1 : 2;
    constexpr int NA = SPIN == 0 ? NC : 2;
    using W = Rows<SPIN, R>;
    __shared__ float4 cf[kSeg];
    __shared__ u64 sdy[R * 32 * max_warps(SPIN, R)];
    __shared__ float4 aw[kSeg * NA];
    // Spin 2: the sums of the segments done, kept apart from the running one (F and G terms share
    // an accumulator: one over all rows would add twice as many terms as sums of F and G apart).
    // Nside 512, E = 1e3 B, orders 1 to 4: absolute error of U (5.6) 4.4e-6 without, 2.5e-6 here.
    __shared__ u64 done[SPIN == 2 ? R * 4 : 1][SPIN == 2 ? 32 * max_warps(SPIN, R) : 1];
    const int64_t L = lmax + 1, nlanes = 2 * nside, nelem = L * (L + 1) / 2;
    const int m = blockIdx.y, l0 = m > SPIN ? m : SPIN;
    const int64_t c0 = (int64_t)blockIdx.z * (SPIN == 0 ? NC : 2);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int64_t jb = (int64_t)blockIdx.x * nw * W::kLanes, jw = jb + warp * W::kLanes;

    W w;
    w.geometry(geom, nlanes, jw, lane, sdy);
    u64 acc[R][4 * NC];
#pragma unroll
    for (int u = 0; u < R; ++u)
#pragma unroll
        for (int q = 0; q < 4 * NC; ++q) {
            acc[u][q] = 0ull;
            if (SPIN == 2) done[u * 4 + q][threadIdx.x] = 0ull;
        }

    const int nseg = l0 <= lmax ? (int)((L - l0 + kSeg - 1) / kSeg) : 0;
    const int64_t s0 = tab.segoff[m];
    const u64 mine = group_bits(jw, jw + W::kLanes < nlanes ? jw + W::kLanes : nlanes);
    const int64_t je = jb + nw * W::kLanes < nlanes ? jb + nw * W::kLanes : nlanes;
    const u64 whole = group_bits(jb, je);
    for (int k = 0; k < nseg; ++k) {
        const u64 act = active_groups(tab, NVAR, s0 + k);
        if (!(act & whole)) continue;   // zero rows on all lanes of this CTA
        const int lb = l0 + kSeg * k;
        const int nrow = (int)(L - lb < kSeg ? L - lb : kSeg);
        __syncthreads();   // the previous segment's rows are done with
        for (int i = threadIdx.x; i < kSeg; i += blockDim.x) {
            const bool in = i < nrow;
            cf[i] = in ? step_coef(lb + i, m, SPIN) : make_float4(0.f, 0.f, 0.f, 0.f);
            const int64_t idx = in ? alm_index(lmax, lb + i, m) : 0;
            const double *src = alm + 2 * (c0 * nelem + idx);   // 8-byte aligned
            if (SPIN == 0) {
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    const bool have = in && c0 + c < ncomp;
                    const float re = have ? (float)src[2 * c * nelem] : 0.f, im = have ? (float)src[2 * c * nelem + 1] : 0.f;
                    aw[i * NC + c] = make_float4(re, re, im, im);
                }
            } else {
                // 2 Q = -F E - i G B, 2 U = -F B + i G E
                const float er = in ? (float)src[0] : 0.f, ei = in ? (float)src[1] : 0.f;
                const float br = in ? (float)src[2 * nelem] : 0.f, bi = in ? (float)src[2 * nelem + 1] : 0.f;
                aw[i * 2] = (i & 1) ? make_float4(bi, -er, -br, -ei) : make_float4(-er, bi, -ei, -br);
                aw[i * 2 + 1] = (i & 1) ? make_float4(-ei, -br, er, -bi) : make_float4(-br, -ei, -bi, er);
            }
        }
        const bool on = (act & mine) != 0ull;
        bool scaled = false;
        if (on) scaled = w.start(tab, s0 + k, nlanes, jw, lane, (float)inv_alpha(lb, m, SPIN));
        __syncthreads();
        if (on) {
#pragma unroll 1
            for (int i = 0; i < nrow; i += 8) {
                w.correct(sdy);
                if (scaled) {
                    syn8<SPIN, NC, R, true>(w, acc, cf + i, aw + i * NA);
                    scaled = w.shifted();
                } else {
                    syn8<SPIN, NC, R, false>(w, acc, cf + i, aw + i * NA);
                }
            }
            if (SPIN == 2) {
#pragma unroll
                for (int q = 0; q < R * 4; ++q) {
                    done[q][threadIdx.x] = add2(done[q][threadIdx.x], acc[q / 4][q % 4]);
                    acc[q / 4][q % 4] = 0ull;
                }
            }
        }
    }
    if (SPIN == 2) {
#pragma unroll
        for (int q = 0; q < R * 4; ++q) acc[q / 4][q % 4] = done[q][threadIdx.x];
    }

    float *out = syn + 4 * ((int64_t)m * nlanes * ncomp + c0);
#pragma unroll
    for (int u = 0; u < R; ++u) {
        if (SPIN == 0) {
            // l0 + m = 2m: even rows are the Sum part; north = even + odd, south = even - odd
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                if (c0 + c >= ncomp) continue;
                float e[2][4];
#pragma unroll
                for (int q = 0; q < 4; ++q) unpack(acc[u][4 * c + q], e[0][q], e[1][q]);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int64_t j = W::lane_of(jw, u, h, lane);
                    if (j < nlanes)
                        store4(out + 4 * (j * ncomp + c),
                               make_float4(e[h][0] + e[h][2], e[h][1] + e[h][3], e[h][0] - e[h][2], e[h][1] - e[h][3]), wide);
                }
            }
        } else {
            const int64_t j = W::lane_of(jw, u, 0, lane);
            if (j >= nlanes) continue;
            // north = Sum + Diff, south = Sum - Diff, the other way round where even rows have odd l + m
            const float hs = (l0 + m) & 1 ? -0.5f : 0.5f;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                float sr, dr, si, di;
                unpack(acc[u][2 * c], sr, dr);
                unpack(acc[u][2 * c + 1], si, di);
                store4(out + 4 * (j * ncomp + c),
                       make_float4(0.5f * (sr + dr), 0.5f * (si + di), hs * (sr - dr), hs * (si - di)), wide);
            }
        }
    }
}

}  // namespace rows
}  // namespace gm

using namespace gm;
using namespace gm::rows;

// Warps of a CTA: all lanes in one CTA while max_warps hold them, else four.
template <int SPIN, int R> static int rows_warps(int64_t nlanes)
{
    const int64_t per = Rows<SPIN, R>::kLanes, need = (nlanes + per - 1) / per;
    return (int)(need <= max_warps(SPIN, R) ? need : 4);
}

template <int SPIN, int NC, int R>
static int launch_rows_ana(int64_t nside, int64_t lmax, int64_t ncomp, const double *geom, const void *rhs,
                           double *alm, double scale, const Tab &tab, cudaStream_t s)
{
    const int64_t nlanes = 2 * nside;
    const int nw = rows_warps<SPIN, R>(nlanes), per = nw * Rows<SPIN, R>::kLanes, nc = SPIN == 0 ? NC : 2;
    dim3 grid((unsigned)((nlanes + per - 1) / per), (unsigned)(lmax + 1), (unsigned)((ncomp + nc - 1) / nc));
    k_rows_ana<SPIN, NC, R><<<grid, 32 * nw, 0, s>>>(nside, lmax, ncomp, geom, (const float *)rhs,
                                                        reinterpret_cast<uintptr_t>(rhs) % 16 == 0, alm, scale, tab);
    return check_launch("gm_legendre_analysis_ck");
}

template <int SPIN, int NC, int R>
static int launch_rows_syn(int64_t nside, int64_t lmax, int64_t ncomp, const double *geom, const double *alm,
                           void *syn, const Tab &tab, cudaStream_t s)
{
    const int64_t nlanes = 2 * nside;
    const int nw = rows_warps<SPIN, R>(nlanes), per = nw * Rows<SPIN, R>::kLanes, nc = SPIN == 0 ? NC : 2;
    dim3 grid((unsigned)((nlanes + per - 1) / per), (unsigned)(lmax + 1), (unsigned)((ncomp + nc - 1) / nc));
    k_rows_syn<SPIN, NC, R><<<grid, 32 * nw, 0, s>>>(nside, lmax, ncomp, geom, alm, (float *)syn,
                                                        reinterpret_cast<uintptr_t>(syn) % 16 == 0, tab);
    return check_launch("gm_legendre_synthesis_ck");
}

// The built-in tile (index into the list of gm_legendre_tiles), R by the number of lanes: the
// autotuner's choices at Nside 64 to 2048 within 10 %.
static int rows_default_tile(int spin, int64_t nside, int64_t ncomp)
{
    const int64_t nlanes = 2 * nside;
    const int r = nlanes >= 1024 ? 2 : (nlanes >= 512 ? 1 : 0);   // R = 4, 2, 1
    if (spin == 2) return r;
    if (ncomp == 1) return r;
    if (ncomp == 2) return 3 + r;
    return 6 + (r > 1 ? 1 : r);
}

static int rows_args(int spin, int64_t nside, int64_t lmax, int64_t ncomp, int &tile)
{
    if (nside < 1 || lmax < 2 || lmax + 1 > 65535 || ncomp < 1 || ncomp > 65535) return GM_ERR_BAD_SHAPE;
    if (spin != 0 && spin != 2) return GM_ERR_UNSUPPORTED;
    if (spin == 2 && (ncomp % 2)) return GM_ERR_BAD_SHAPE;
    if (tile < -1 || tile >= gm_legendre_tiles(spin, nullptr, 0)) return GM_ERR_BAD_SHAPE;
    if (tile < 0) tile = rows_default_tile(spin, nside, ncomp);
    return GM_OK;
}

static Tab rows_tab(const int64_t *segoff, const void *ck_a, const uint8_t *cn_a, const void *ck_b,
                    const uint8_t *cn_b, const uint64_t *mask_a, const uint64_t *mask_b, int64_t nside)
{
    Tab t;
    t.segoff = segoff;
    t.ck[0] = (const float2 *)ck_a;
    t.cn[0] = cn_a;
    t.ck[1] = (const float2 *)ck_b;
    t.cn[1] = cn_b;
    // both variants' masks or neither; 64 groups of 64 lanes
    const bool masked = mask_a && (mask_b || ck_b == nullptr) && 2 * nside <= 4096;
    t.mask[0] = masked ? (const u64 *)mask_a : nullptr;
    t.mask[1] = masked ? (const u64 *)mask_b : nullptr;
    return t;
}

extern "C" int gm_legendre_analysis_ck(int spin, int64_t nside, int64_t lmax, int64_t ncomp,
                                       const double *lane_geom, const void *rhs, double *alm,
                                       double scale, const int64_t *segoff, const void *ck_a,
                                       const uint8_t *cn_a, const void *ck_b, const uint8_t *cn_b,
                                       const uint64_t *mask_a, const uint64_t *mask_b, int tile, void *stream)
{
    const int st = rows_args(spin, nside, lmax, ncomp, tile);
    if (st != GM_OK) return st;
    if (!lane_geom || !rhs || !alm || !segoff || !ck_a || !cn_a || (spin == 2 && (!ck_b || !cn_b)))
        return GM_ERR_BAD_PTR;
    const Tab tab = rows_tab(segoff, ck_a, cn_a, spin == 2 ? ck_b : nullptr, cn_b, mask_a,
                             spin == 2 ? mask_b : nullptr, nside);
    cudaStream_t s = as_stream(stream);
#define GM_ANA(SP, NC, R) return launch_rows_ana<SP, NC, R>(nside, lmax, ncomp, lane_geom, rhs, alm, scale, tab, s)
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
        default: GM_ANA(0, 2, 8);
        }
    }
    switch (tile) {
    case 0: GM_ANA(2, 1, 1);
    case 1: GM_ANA(2, 1, 2);
    case 2: GM_ANA(2, 1, 4);
    default: GM_ANA(2, 1, 8);
    }
#undef GM_ANA
}

extern "C" int gm_legendre_synthesis_ck(int spin, int64_t nside, int64_t lmax, int64_t ncomp,
                                        const double *lane_geom, const double *alm, void *syn,
                                        const int64_t *segoff, const void *ck_a, const uint8_t *cn_a,
                                        const void *ck_b, const uint8_t *cn_b, const uint64_t *mask_a,
                                        const uint64_t *mask_b, int tile, void *stream)
{
    const int st = rows_args(spin, nside, lmax, ncomp, tile);
    if (st != GM_OK) return st;
    if (!lane_geom || !alm || !syn || !segoff || !ck_a || !cn_a || (spin == 2 && (!ck_b || !cn_b)))
        return GM_ERR_BAD_PTR;
    const Tab tab = rows_tab(segoff, ck_a, cn_a, spin == 2 ? ck_b : nullptr, cn_b, mask_a,
                             spin == 2 ? mask_b : nullptr, nside);
    cudaStream_t s = as_stream(stream);
#define GM_SYN(SP, NC, R) return launch_rows_syn<SP, NC, R>(nside, lmax, ncomp, lane_geom, alm, syn, tab, s)
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
        default: GM_SYN(0, 2, 8);
        }
    }
    switch (tile) {
    case 0: GM_SYN(2, 1, 1);
    case 1: GM_SYN(2, 1, 2);
    case 2: GM_SYN(2, 1, 4);
    default: GM_SYN(2, 1, 8);
    }
#undef GM_SYN
}
