// The area methods with the 4 x cubic-spline enlargement built in (spx_half_area_spline_cd,
// spx_tail_area_spline_cd): the outputs of k_half_area and k_tail_area (cd.cu), whose zoom operators a
// caller passes as dense matrices, for the operators measure_cds uses.
//
// That enlargement is scipy.ndimage.zoom(order 3, grid mode) of the cell in a wide zero border
// (subpx/_cpu/invariant_cd.py:424-444): the cubic B-spline of the samples, with zeros outside, taken
// at (X + 0.5) / 4 - 0.5. Here it stays in that form. The coefficients (the cell plus two on either
// side) come from Unser's two-pass recursion, which on a zero-extended line is exact, and live in
// shared memory; a sub-pixel is 4 x 4 taps of four fixed phases, evaluated where it is wanted. The
// enlargement itself (445 KB for a 59 px window, 74 KB for a 24 px cell) is never stored: with the dense
// operators it was written to and re-read from global scratch by every step, and its products took
// 59 multiply-adds per sub-pixel and axis instead of four.
//
// Bound: latency and issue of a chain of CTA-wide steps on one cell; several CTAs share an SM, which
// the smaller footprint allows. A thread owns a sub-pixel column: walking down it needs one new row
// combination (4 taps) and four column combinations (16 taps) per pixel, five multiply-adds per
// sub-pixel. The walk over the whole cell is done once per enlargement (and per threshold sum); it
// leaves, for every unit of 1 x 8 pixels (one word of sub-pixels, four rows), an upper bound of its
// values, so each later step evaluates only the units that can hold what it looks for.
//
// Measured on one B200 against the dense kernels: the five tail methods of 4,032 windows of 59 px (both
// passes) 80.3 -> 6.7 ms; half_area and half_area_min + _min_avg of the 7,225 cells of a 2047 x 2050 page
// (24 px) 5.47 -> 1.41 ms.

#include <algorithm>

#include "area.cuh"
#include "methods.cuh"
#include "select.cuh"

namespace spx {
namespace {

constexpr int kF = 4;                       // enlargement
constexpr double kPole = -0.2679491924311227;  // sqrt(3) - 2

// Six times the cubic B-spline weights of the four taps floor(x) - 1 .. floor(x) + 2 at the sub-pixels
// of a pixel, x = k - 3/8, k - 1/8, k + 1/8, k + 3/8 (the first two count from pixel k - 2, the others
// from k - 1). All are exact in binary; the recursion's gain of 6 per axis cancels their divisor, so
// neither is applied.
__constant__ double c_tap[4][4] = {{0.052734375, 2.388671875, 3.314453125, 0.244140625},
                                   {0.001953125, 1.416015625, 3.912109375, 0.669921875},
                                   {0.669921875, 3.912109375, 1.416015625, 0.001953125},
                                   {0.244140625, 3.314453125, 2.388671875, 0.052734375}};
// The same weights as compile-time constants, for the taps along y.
__device__ __forceinline__ double tap4(int phase, double a, double b, double c, double d) {
    switch (phase) {
        case 0: return fma(0.244140625, d, fma(3.314453125, c, fma(2.388671875, b, 0.052734375 * a)));
        case 1: return fma(0.669921875, d, fma(3.912109375, c, fma(1.416015625, b, 0.001953125 * a)));
        case 2: return fma(0.001953125, d, fma(1.416015625, c, fma(3.912109375, b, 0.669921875 * a)));
        default: return fma(0.052734375, d, fma(2.388671875, c, fma(3.314453125, b, 0.244140625 * a)));
    }
}

// Shared memory of an area CTA. Coefficients of pixel (y, x) at coef[(y + 2) * cp + x + 2], y = -2 ..
// hm + 1; the pitch is odd, so the threads of the row recursion (one row each) fall in different banks.
struct AreaMem {
    int hm, wm, cp, Hb, Wb, RW;  // cell, coefficient pitch, enlargement, words per sub-pixel row
    long long plane, list, tmp;  // words of a sub-pixel bit plane; doubles of the list and the outline
    __host__ __device__ AreaMem(int hm_, int wm_, int n_angles, int outlines, int threads)
        : hm(hm_), wm(wm_), cp((wm_ + 4) | 1), Hb(hm_ * kF), Wb(wm_ * kF), RW((wm_ * kF + 31) / 32) {
        plane = (long long)Hb * RW;
        const long long planes = (3 * plane + 1) / 2;  // in doubles
        list = planes > 8LL * threads ? planes : 8LL * threads;
        tmp = outlines ? 3LL * (n_angles + 1) : 0;
    }
    __host__ __device__ long long coefs() const { return (long long)(hm + 4) * cp; }
    // masks: per-pixel-row bit words (mask; for windows also the core and the core in the territory).
    __host__ __device__ long long bytes(int masks) const {
        return (coefs() + list + tmp) * 8 + (long long)(1 + masks) * hm * RW * 4;
    }
};

template <int NT>
struct AreaCta {
    const AreaMem g;
    double* coef;
    double* list;      // values near the peak; the bit planes take its place afterwards
    double* tmp;
    float* unit;       // upper bound of the masked values of each unit (pixel row, word)
    uint32_t* pmask;   // mask bits of each pixel row, one per sub-pixel column
    uint32_t *above, *reg, *reg2;
    __device__ AreaCta(const AreaMem& m, double* sm) : g(m) {
        coef = sm;
        list = coef + g.coefs();
        tmp = list + g.list;
        unit = reinterpret_cast<float*>(tmp + g.tmp);
        pmask = reinterpret_cast<uint32_t*>(unit + (long long)g.hm * g.RW);
        above = reinterpret_cast<uint32_t*>(list);
        reg = above + g.plane;
        reg2 = reg + g.plane;
    }
    __device__ __forceinline__ bool pixel(int y, int x) const {
        return (pmask[y * g.RW + (x >> 3)] >> ((x & 7) * kF)) & 1u;
    }
};

// The recursion over one line of n samples at c[0], c[stride], ... with the two coefficients before
// and after it: c+ [k] = x[k] + z c+[k-1], then c[k] = z (c[k+1] - c+[k]) from its infinite-tail value
// two samples past the end. Eight samples are loaded before their chain of multiply-adds.
__device__ __forceinline__ void spline_line0(double* c, int n, int stride) {
    double v = 0.0;
    int k = 0;
    for (; k + 8 <= n; k += 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = c[(k + u) * stride];
#pragma unroll
        for (int u = 0; u < 8; ++u) c[(k + u) * stride] = v = fma(kPole, v, x[u]);
    }
    for (; k < n; ++k) c[k * stride] = v = fma(kPole, v, c[k * stride]);
    const double v1 = kPole * v, v2 = kPole * v1;
    double r = -kPole / (1.0 - kPole * kPole) * v2;
    c[(n + 1) * stride] = r;
    r = kPole * (r - v1);
    c[n * stride] = r;
    k = n - 1;
    for (; k >= 7; k -= 8) {
        double x[8];
#pragma unroll
        for (int u = 0; u < 8; ++u) x[u] = kPole * c[(k - u) * stride];
#pragma unroll
        for (int u = 0; u < 8; ++u) c[(k - u) * stride] = r = fma(kPole, r, -x[u]);
    }
    for (; k >= 0; --k) c[k * stride] = r = kPole * (r - c[k * stride]);
    r *= kPole;
    c[-stride] = r;
    c[-2 * stride] = r * kPole;
}

// The cell's samples at their places in coef become its spline coefficients. Called by all threads
// after the samples were written; ends with a barrier.
template <int NT>
__device__ void spline_coefs(const AreaCta<NT>& h) {
    __syncthreads();
    for (int x = threadIdx.x; x < h.g.wm; x += NT) spline_line0(h.coef + 2 * h.g.cp + x + 2, h.g.hm, h.g.cp);
    __syncthreads();
    for (int r = threadIdx.x; r < h.g.hm + 4; r += NT) spline_line0(h.coef + (long long)r * h.g.cp + 2, h.g.wm, 1);
    __syncthreads();
}

// Row combinations of one sub-pixel column.
struct Column {
    const double* q;  // first tap in coefficient row 0
    double w0, w1, w2, w3;
    __device__ __forceinline__ Column(const double* coef, int X) {
        const int px = X & 3;
        q = coef + (X >> 2) + (px >> 1);
        w0 = c_tap[px][0];
        w1 = c_tap[px][1];
        w2 = c_tap[px][2];
        w3 = c_tap[px][3];
    }
    __device__ __forceinline__ double row(int off) const {
        const double* p = q + off;
        return fma(w3, p[3], fma(w2, p[2], fma(w1, p[1], w0 * p[0])));
    }
    // The same of the difference of the pixels right and left, and of the second difference.
    __device__ __forceinline__ double row_dx(int off) const {
        const double* p = q + off;
        return fma(w3, p[4] - p[2], fma(w2, p[3] - p[1], fma(w1, p[2] - p[0], w0 * (p[1] - p[-1]))));
    }
    __device__ __forceinline__ double row_dxx(int off) const {
        const double* p = q + off;
        return fma(w3, fma(-2.0, p[3], p[4] + p[2]),
                   fma(w2, fma(-2.0, p[2], p[3] + p[1]),
                       fma(w1, fma(-2.0, p[1], p[2] + p[0]), w0 * fma(-2.0, p[0], p[1] + p[-1]))));
    }
};

__device__ __forceinline__ void column_taps(const double* r, double* v) {
    v[0] = tap4(0, r[0], r[1], r[2], r[3]);
    v[1] = tap4(1, r[0], r[1], r[2], r[3]);
    v[2] = tap4(2, r[1], r[2], r[3], r[4]);
    v[3] = tap4(3, r[1], r[2], r[3], r[4]);
}

// The four sub-pixels of pixel row ky in sub-pixel column X.
__device__ __forceinline__ void unit_values(const double* coef, int cp, int ky, int X, double* v) {
    const Column c(coef, X);
    double r[5];
#pragma unroll
    for (int a = 0; a < 5; ++a) r[a] = c.row((ky + a) * cp);
    column_taps(r, v);
}

// fn(ky, v) for every pixel row of sub-pixel column X.
template <class F>
__device__ __forceinline__ void walk_column(const double* coef, int cp, int hm, int X, F&& fn) {
    const Column c(coef, X);
    double r[5];
#pragma unroll
    for (int a = 0; a < 4; ++a) r[a] = c.row(a * cp);
    for (int ky = 0; ky < hm; ++ky) {
        r[4] = c.row((ky + 4) * cp);
        double v[4];
        column_taps(r, v);
        fn(ky, v);
#pragma unroll
        for (int a = 0; a < 4; ++a) r[a] = r[a + 1];
    }
}

__device__ __forceinline__ unsigned float_key(float f) {
    const unsigned u = __float_as_uint(f);
    return (u >> 31) ? ~u : (u | 0x80000000u);
}
__device__ __forceinline__ float key_float(unsigned k) {
    return __uint_as_float((k >> 31) ? (k & 0x7fffffffu) : ~k);
}

// The highest masked sub-pixel's value and, in top->y, its place (-inf and 0 when the mask is empty), on every
// thread, and the units' upper bounds. top->x: the first sub-pixel in row-major order that reaches it to rounding (a
// margin of 2^-48, twice the sums' error): equal peaks of a cell (isolated pixels of one value, mirrored holes) differ
// in the last bits of the recursion's sums, and the reference takes the first of equal ones. It is looked up over the
// few units that reach the peak, each found by a lane (half_area 1.38 -> 1.41 ms, tail windows as before).
template <int NT>
__device__ void area_peak(const AreaCta<NT>& h, double* s_red, int* s_ired, double* top_v, int2* top) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, RW = h.g.RW;
    double best = -INFINITY;
    int best_i = 0x7fffffff;
    for (int w = warp; w < RW; w += NT / 32) {
        const int X = w * 32 + lane;
        walk_column(h.coef, h.g.cp, h.g.hm, min(X, h.g.Wb - 1), [&](int ky, const double* v) {
            const bool in = (h.pmask[ky * RW + w] >> lane) & 1u;
            double mx = -INFINITY;
            if (in) {
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    if (v[p] > best) {
                        best = v[p];
                        best_i = (kF * ky + p) * h.g.Wb + X;
                    }
                    mx = fmax(mx, v[p]);
                }
            }
            const unsigned key = __reduce_max_sync(0xffffffffu, float_key(__double2float_ru(mx)));
            if (lane == 0) h.unit[ky * RW + w] = key_float(key);
        });
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oi = __shfl_xor_sync(0xffffffffu, best_i, o);
        if (ob > best || (ob == best && oi < best_i)) {
            best = ob;
            best_i = oi;
        }
    }
    if (lane == 0) {
        s_red[warp] = best;
        s_ired[warp] = best_i;
    }
    __syncthreads();
    best = s_red[0];
    best_i = s_ired[0];
    for (int q = 1; q < NT / 32; ++q)
        if (s_red[q] > best || (s_red[q] == best && s_ired[q] < best_i)) {
            best = s_red[q];
            best_i = s_ired[q];
        }
    __syncthreads();
    const double reach = best - 0x1p-48 * best;
    int first = best_i;
    const int units = h.g.hm * RW;
    if (best > 0.0 && isfinite(best))
        for (int u0 = warp * 32; u0 < units; u0 += NT) {
            const bool reaches = u0 + lane < units && (double)h.unit[min(u0 + lane, units - 1)] >= reach;
            for (unsigned b = __ballot_sync(0xffffffffu, reaches); b; b &= b - 1) {
                const int u = u0 + __ffs(b) - 1, ky = u / RW, w = u - ky * RW;
                const int X = min(w * 32 + lane, h.g.Wb - 1);
                double v[4];
                unit_values(h.coef, h.g.cp, ky, X, v);
                const bool in = (h.pmask[u] >> lane) & 1u;
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (in && v[p] >= reach) first = min(first, (kF * ky + p) * h.g.Wb + X);
            }
        }
    first = __reduce_min_sync(0xffffffffu, first);
    if (lane == 0) s_ired[warp] = first;
    __syncthreads();
    for (int q = 0; q < NT / 32; ++q) first = min(first, s_ired[q]);
    *top_v = best;
    *top = best_i == 0x7fffffff ? make_int2(0, 0) : make_int2(first, best_i);
    __syncthreads();
}

struct SelectMem {
    int hist[2048];
    int warp_tot[32], s_pick[3];
    unsigned long long s_keys[2];
};

// Mean of the n_top highest masked sub-pixels, or -1 when it is not a positive signal's (no value above
// zero, fewer sub-pixels in the mask, not finite). The values above a fraction of the highest are
// listed, each warp's in its own part of the list in a fixed order, and the n_top-th highest found
// among them by the CTA select; when no fraction gives a list that holds them and fits, the select
// runs over every sub-pixel.
template <int NT>
__device__ double area_peak_mean(const AreaCta<NT>& h, double best, int n_top, int mask_subpx, SelectMem* sel,
                                 double* s_red, int* s_ired) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, RW = h.g.RW;
    const int N = h.g.Hb * h.g.Wb;
    if (!(best > 0.0) || n_top > mask_subpx) return -1.0;
    const int cap = (int)(h.g.list / (NT / 32));
    double* mine = h.list + (long long)warp * cap;
    auto finish = [&](auto&& for_keys, int k, unsigned long long kmin) {
        unsigned long long kth, kth2;
        cta_select<NT>(for_keys, k, false, kmin, order_key(best), sel->hist, sel->warp_tot, sel->s_pick, sel->s_keys,
                       &kth, &kth2);
        double sum = 0.0;
        int cnt = 0;
        for_keys([&](unsigned long long key) {
            if (key > kth) {
                sum += key_value(key);
                ++cnt;
            }
        });
        sum = warp_sum(sum);
        cnt = warp_sum_i(cnt);
        if (lane == 0) {
            s_red[warp] = sum;
            s_ired[warp] = cnt;
        }
        __syncthreads();
        double total = 0.0;
        int above = 0;
        for (int q = 0; q < NT / 32; ++q) {
            total += s_red[q];
            above += s_ired[q];
        }
        total += (double)(n_top - above) * key_value(kth);
        const double mean = total / n_top;
        __syncthreads();
        return isfinite(mean) ? mean : -1.0;
    };
    const double part[3] = {0.93, 0.8, 0.5};
#pragma unroll 1
    for (int attempt = 0; attempt < 3; ++attempt) {
        const double floor_v = part[attempt] * best;
        int cnt = 0;
        for (int ky = warp; ky < h.g.hm; ky += NT / 32)
            for (int w = 0; w < RW; ++w) {
                if ((double)h.unit[ky * RW + w] < floor_v) continue;
                double v[4];
                unit_values(h.coef, h.g.cp, ky, min(w * 32 + lane, h.g.Wb - 1), v);
                const bool in = (h.pmask[ky * RW + w] >> lane) & 1u;
#pragma unroll
                for (int p = 0; p < 4; ++p) {
                    const bool take = in && v[p] >= floor_v;
                    const unsigned b = __ballot_sync(0xffffffffu, take);
                    const int slot = cnt + __popc(b & ((1u << lane) - 1u));
                    if (take && slot < cap) mine[slot] = v[p];
                    cnt += __popc(b);
                }
            }
        if (lane == 0) s_ired[warp] = cnt;
        __syncthreads();
        int total = 0, most = 0;
        for (int q = 0; q < NT / 32; ++q) {
            total += s_ired[q];
            most = max(most, s_ired[q]);
        }
        __syncthreads();
        if (most > cap) break;
        if (total < n_top) continue;
        auto listed = [&](auto&& fn) {
            for (int q = lane; q < cnt; q += 32) fn(order_key(mine[q]));
        };
        return finish(listed, total - n_top, order_key(floor_v));
    }
    auto every = [&](auto&& fn) {
        for (int w = warp; w < RW; w += NT / 32) {
            const int X = w * 32 + lane;
            walk_column(h.coef, h.g.cp, h.g.hm, min(X, h.g.Wb - 1), [&](int ky, const double* v) {
                if (X >= h.g.Wb) return;
                const bool in = (h.pmask[ky * RW + w] >> lane) & 1u;
#pragma unroll
                for (int p = 0; p < 4; ++p) fn(order_key(in ? v[p] : -INFINITY));
            });
        }
    };
    return finish(every, N - n_top, order_key(-INFINITY));
}

// Sums over the set bits j of a word: count, j, j^2.
__device__ __forceinline__ void bit_moments(uint32_t b, int* s1, int* s2) {
    constexpr uint32_t M[5] = {0xaaaaaaaau, 0xccccccccu, 0xf0f0f0f0u, 0xff00ff00u, 0xffff0000u};
    int a1 = 0, a2 = 0;
#pragma unroll
    for (int p = 0; p < 5; ++p) {
        const int c = __popc(b & M[p]);
        a1 += c << p;
        a2 += c << (2 * p);
#pragma unroll
        for (int q = 0; q < p; ++q) a2 += __popc(b & M[p] & M[q]) << (p + q + 1);
    }
    *s1 = a1;
    *s2 = a2;
}

struct AreaOptions {
    int n_angles, n_top, outlines;
    double level;
};

// One output from the cell's coefficients: the region of sub-pixels above cut around the highest one,
// its metrics and outline (area_result). The region's count and moments are integer sums, exact
// whatever the order: centroid SX / n, spreads (n SXX - SX^2) / n^2.
template <int NT>
__device__ void area_output(const AreaCta<NT>& h, const AreaOptions& o, const MethodOut& out, int i, double b,
                            double peak, double cut, double steepest, int2 top, const AreaPlace& at,
                            unsigned long long* s_mom, double* s_red) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int hm = h.g.hm, Hb = h.g.Hb, Wb = h.g.Wb, RW = h.g.RW;
    const AreaShape shape{hm, h.g.wm, o.n_angles, kF, o.outlines};
    const bool signal = peak > 0.0 && isfinite(cut) && cut < peak;
    if (!signal) {
        area_result<NT>(shape, out, i, AreaFound{false, false, 0, 0, 0, 0, 0, 0, peak, cut, b, steepest}, h.above, RW,
                        h.tmp, s_red, at);
        return;
    }
    for (int ky = warp; ky < hm; ky += NT / 32)
        for (int w = 0; w < RW; ++w) {
            uint32_t word[4] = {0u, 0u, 0u, 0u};
            if ((double)h.unit[ky * RW + w] > cut) {
                double v[4];
                unit_values(h.coef, h.g.cp, ky, min(w * 32 + lane, Wb - 1), v);
                const uint32_t m = h.pmask[ky * RW + w];
#pragma unroll
                for (int p = 0; p < 4; ++p) word[p] = __ballot_sync(0xffffffffu, v[p] > cut) & m;
            }
            if (lane < 4) {
                const int t = (kF * ky + lane) * RW + w;
                h.above[t] = lane == 0 ? word[0] : lane == 1 ? word[1] : lane == 2 ? word[2] : word[3];
                h.reg[t] = 0u;
                h.reg2[t] = 0u;
            }
        }
    __syncthreads();
    // (A threshold within the margin of the peak can leave the first place below it.)
    auto is_above = [&](int t) { return (h.above[t / Wb * RW + t % Wb / 32] >> (t % Wb % 32)) & 1u; };
    const int start = is_above(top.x) ? top.x : top.y, top_row = start / Wb;
    if (tid == 0 && is_above(start)) h.reg[top_row * RW + start % Wb / 32] = 1u << (start % Wb % 32);
    __syncthreads();
    // Grown from the highest sub-pixel one 8-neighbour ring per step until it stops changing; step s + 1
    // only computes the rows within s + 1 of the start.
    const uint32_t last_bits = (Wb % 32) ? ((1u << (Wb % 32)) - 1u) : 0xffffffffu;
    uint32_t* cur = h.reg;
    uint32_t* nxt = h.reg2;
    auto vert = [&](const uint32_t* p, int Y, int w) {
        uint32_t v = p[Y * RW + w];
        if (Y > 0) v |= p[(Y - 1) * RW + w];
        if (Y < Hb - 1) v |= p[(Y + 1) * RW + w];
        return v;
    };
    auto dilate = [&](const uint32_t* p, int t) {
        const int Y = t / RW, w = t % RW;
        const uint32_t v = vert(p, Y, w);
        const uint32_t vp = w > 0 ? vert(p, Y, w - 1) : 0u, vn = w < RW - 1 ? vert(p, Y, w + 1) : 0u;
        uint32_t d = v | (v << 1) | (v >> 1) | (vp >> 31) | (vn << 31);
        if (w == RW - 1) d &= last_bits;
        return d;
    };
    int r0 = top_row, r1 = top_row;
    for (int step = 0; step < Hb * Wb; ++step) {
        int changed = 0;
        r0 = max(r0 - 1, 0);
        r1 = min(r1 + 1, Hb - 1);
        for (int t = r0 * RW + tid; t < (r1 + 1) * RW; t += NT) {
            const uint32_t a = h.above[t];
            const uint32_t nw = a ? dilate(cur, t) & a : 0u;
            nxt[t] = nw;
            changed |= nw != cur[t];
        }
        changed = __syncthreads_or(changed);
        uint32_t* sw = cur;
        cur = nxt;
        nxt = sw;
        if (!changed) break;
    }
    // Whether the region reaches outside the mask or the cell's edge, its count and moments.
    int touch = 0, cnt = 0, sx = 0, sy = 0;
    unsigned long long sxx = 0, syy = 0;
    for (int t = max(r0 - 1, 0) * RW + tid; t < (min(r1 + 1, Hb - 1) + 1) * RW; t += NT) {
        const int Y = t / RW, w = t - Y * RW;
        const uint32_t valid = w == RW - 1 ? last_bits : 0xffffffffu;
        touch |= (dilate(cur, t) & ~h.pmask[(Y >> 2) * RW + w] & valid) != 0u;
        const uint32_t c = cur[t];
        if (!c) continue;
        touch |= Y == 0 || Y == Hb - 1 || (w == 0 && (c & 1u)) ||
                 (w == (Wb - 1) / 32 && ((c >> ((Wb - 1) % 32)) & 1u));
        int s1, s2;
        bit_moments(c, &s1, &s2);
        const int p = __popc(c), x0 = 32 * w;
        cnt += p;
        sx += p * x0 + s1;
        sy += p * Y;
        sxx += (unsigned)(p * x0 * x0 + 2 * x0 * s1 + s2);
        syy += (unsigned)(p * Y * Y);
    }
    double sum = 0.0;  // the region's brightness
    for (int ky = (r0 >> 2) + warp; ky <= (r1 >> 2); ky += NT / 32)
        for (int w = 0; w < RW; ++w) {
            uint32_t c[4], any = 0u;
#pragma unroll
            for (int p = 0; p < 4; ++p) any |= c[p] = cur[(kF * ky + p) * RW + w];
            if (!any) continue;
            double v[4];
            unit_values(h.coef, h.g.cp, ky, min(w * 32 + lane, Wb - 1), v);
#pragma unroll
            for (int p = 0; p < 4; ++p)
                if ((c[p] >> lane) & 1u) sum += v[p];
        }
    touch = __syncthreads_or(touch);
    sum = warp_sum(sum);
    unsigned long long mom[5] = {(unsigned long long)cnt, (unsigned long long)sx, (unsigned long long)sy, sxx, syy};
#pragma unroll
    for (int q = 0; q < 5; ++q)
#pragma unroll
        for (int s = 16; s > 0; s >>= 1) mom[q] += __shfl_xor_sync(0xffffffffu, mom[q], s);
    if (lane == 0) {
        s_red[warp] = sum;
#pragma unroll
        for (int q = 0; q < 5; ++q) s_mom[5 * warp + q] = mom[q];
    }
    __syncthreads();
    sum = s_red[0];
#pragma unroll
    for (int q = 0; q < 5; ++q) mom[q] = s_mom[q];
    for (int u = 1; u < NT / 32; ++u) {
        sum += s_red[u];
#pragma unroll
        for (int q = 0; q < 5; ++q) mom[q] += s_mom[5 * u + q];
    }
    __syncthreads();
    const long long count = (long long)mom[0];
    const double weight = (double)(count > 1 ? count : 1), w2 = weight * weight;
    const double scale = 1.0 / (kF * kF);
    const double var_x = (double)(mom[0] * mom[3] - mom[1] * mom[1]) / w2 * scale;
    const double var_y = (double)(mom[0] * mom[4] - mom[2] * mom[2]) / w2 * scale;
    area_result<NT>(shape, out, i,
                    AreaFound{true, touch != 0, count, (double)mom[1] / weight, (double)mom[2] / weight, var_x, var_y,
                              sum / weight, peak, cut, b, steepest},
                    cur, RW, h.tmp, s_red, at);
}

// Mean of the middle value(s) by rank (ties by position) of n values, none of them NaN; NaN if there are none.
template <int NT>
__device__ double cta_median(const double* v, int n, double* s_mid) {
    const int k1 = (n - 1) / 2, k2 = n / 2;
    for (int t = threadIdx.x; t < n; t += NT) {
        const double x = v[t];
        int rank = 0;
        for (int q = 0; q < n; ++q) rank += v[q] < x || (v[q] == x && q < t);
        if (rank == k1) s_mid[0] = x;
        if (rank == k2) s_mid[1] = x;
    }
    __syncthreads();
    const double m = n ? __ddiv_rn(__dadd_rn(s_mid[0], s_mid[1]), 2.0) : dnan();
    __syncthreads();
    return m;
}

// ------------------------------------------------------------------------------ half_area family

struct HalfSplineArgs {
    const double* cleaned;
    const int* vor;
    const int4* boxes;
    const int* which;
    int n, hm, wm, W, median;
    AreaOptions o;
    MethodOut out[2];  // highest-pixel peak, averaged peak (status null: not wanted)
};

template <int NT>
__global__ void __launch_bounds__(NT, 640 / NT) k_half_area_spline(const __grid_constant__ HalfSplineArgs a) {
    extern __shared__ double sm[];
    __shared__ SelectMem sel;
    __shared__ double s_red[NT / 32], s_mid[2];
    __shared__ int s_ired[NT / 32], s_n[2];
    __shared__ unsigned long long s_mom[5 * (NT / 32)];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const AreaCta<NT> h(AreaMem(a.hm, a.wm, a.o.n_angles, a.o.outlines, NT), sm);
    const int hm = a.hm, wm = a.wm, RW = h.g.RW, area = hm * wm;
    for (int i = blockIdx.x; i < a.n; i += gridDim.x) {
        const int j = a.which ? a.which[i] : i;
        const CellView c{a.cleaned + (long long)i * area, a.vor, a.boxes[j], j, a.W, hm, wm};
        __syncthreads();  // the previous cell's shared-memory reads are done
        if (tid == 0) s_n[0] = s_n[1] = 0;
        __syncthreads();
        for (int t = warp; t < hm * RW; t += NT / 32) {
            const int y = t / RW, X = (t - y * RW) * 32 + lane;
            const uint32_t m = __ballot_sync(0xffffffffu, X < h.g.Wb && c.mask(y, X >> 2));
            if (lane == 0) {
                h.pmask[t] = m;
                if (m) atomicAdd(&s_n[1], __popc(m));
            }
        }
        __syncthreads();
        // Outermost mask pixels: a 4-neighbour outside the mask, or on the stack's edge.
        double lmin = INFINITY;
        double* ring = h.coef;  // their values, before the coefficients
        for (int k = tid; k < area; k += NT) {
            const int y = k / wm, x = k - y * wm;
            if (!h.pixel(y, x)) continue;
            const bool inner = y > 0 && x > 0 && y < hm - 1 && x < wm - 1 && h.pixel(y - 1, x) && h.pixel(y + 1, x) &&
                               h.pixel(y, x - 1) && h.pixel(y, x + 1);
            if (!inner) {
                const double v = c.roi[k];
                if (a.median && !isnan(v)) ring[atomicAdd(&s_n[0], 1)] = v;
                lmin = fmin(lmin, v);
            }
        }
        lmin = warp_min(lmin);
        if (lane == 0) s_red[warp] = lmin;
        __syncthreads();
        double b;
        if (a.median) {
            b = cta_median<NT>(ring, s_n[0], s_mid);
        } else {
            b = s_red[0];
            for (int q = 1; q < NT / 32; ++q) b = fmin(b, s_red[q]);
            __syncthreads();
        }
        for (int k = tid; k < area; k += NT) {
            const int y = k / wm, x = k - y * wm;
            h.coef[(y + 2) * h.g.cp + x + 2] = h.pixel(y, x) ? __dsub_rn(c.roi[k], b) : 0.0;
        }
        spline_coefs(h);
        double top_v;
        int2 top;
        area_peak(h, s_red, s_ired, &top_v, &top);
        const AreaPlace at{(double)c.box.x, (double)c.box.y, dnan(), dnan()};
        // The averaged peak reads the list that the bit planes of an output replace.
        double mean = -1.0;
        if (a.out[1].status && a.o.n_top <= h.g.Hb * h.g.Wb)
            mean = area_peak_mean(h, top_v, a.o.n_top, kF * s_n[1], &sel, s_red, s_ired);
#pragma unroll 1
        for (int m = 0; m < 2; ++m) {
            if (!a.out[m].status) continue;
            const double peak = m == 0 ? top_v : mean;
            area_output(h, a.o, a.out[m], i, b, peak, __dmul_rn(a.o.level, peak), dnan(), top, at, s_mom, s_red);
        }
    }
}

// ------------------------------------------------------------------------------ tail family

struct TailSplineArgs {
    const float* cells;      // (n, S, S) each hole's share of the light
    const uint8_t* inside;   // (n, S, S) the window inside the image: the mask
    const uint8_t* levelm;   // level pixels (tail_area's local level)
    const uint8_t* zone;     // own territory (foot_area)
    const int* win_org;      // (n, 2) window origins
    const int* cell_org;     // (n, 2) the holes' own cell origins (center_local)
    int n, S;
    AreaOptions o;
    const double* cuts;      // (n) foot_area_ratio's thresholds
    MethodOut out[5];        // tail_area, tail_area_norm, edge_area, foot_area, foot_area_ratio (status null: not wanted)
};

// Sums of four values over the CTA, on every thread.
template <int NT>
__device__ void cta_sum4(double* v, double* s4) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = warp_sum(v[q]);
    if (lane == 0)
#pragma unroll
        for (int q = 0; q < 4; ++q) s4[4 * warp + q] = v[q];
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        v[q] = s4[q];
        for (int u = 1; u < NT / 32; ++u) v[q] += s4[4 * u + q];
    }
    __syncthreads();
}

// One CTA per window. The threshold sums run over the core sub-pixels (inside the mask with the pixels
// above, below, left and right of theirs): those neighbours have the same phase one pixel away, so a
// central or second difference of the enlargement is the spline of the coefficients' difference, and
// a column walk carries the differences along with the values.
template <int NT>
__global__ void __launch_bounds__(NT, 640 / NT) k_tail_area_spline(const __grid_constant__ TailSplineArgs t) {
    extern __shared__ double sm[];
    __shared__ SelectMem sel;
    __shared__ double s_red[NT / 32], s_mid[2], s4[4 * (NT / 32)];
    __shared__ int s_ired[NT / 32], s_n[2];
    __shared__ unsigned long long s_mom[5 * (NT / 32)];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const AreaCta<NT> h(AreaMem(t.S, t.S, t.o.n_angles, t.o.outlines, NT), sm);
    const int S = t.S, RW = h.g.RW, cp = h.g.cp, area = S * S;
    uint32_t* core = h.pmask + S * RW;   // core sub-pixels, per pixel row
    uint32_t* zcore = core + S * RW;     // and inside the territory
    enum { kMed = 0, kNorm, kEdge, kFoot, kGiven };
    const bool want_edge = t.out[kEdge].status, want_foot = t.out[kFoot].status;
    const bool want_zero = t.out[kNorm].status || want_edge || want_foot || t.out[kGiven].status;
    for (int i = blockIdx.x; i < t.n; i += gridDim.x) {
        __syncthreads();  // the previous window's shared-memory reads are done
        if (tid == 0) s_n[0] = s_n[1] = 0;
        __syncthreads();
        const long long base = (long long)i * area;
        for (int u = warp; u < S * RW; u += NT / 32) {
            const int y = u / RW, X = (u - y * RW) * 32 + lane;
            const int k = y * S + (X >> 2);
            const bool in = X < h.g.Wb;
            const uint32_t m = __ballot_sync(0xffffffffu, in && t.inside[base + k]);
            const uint32_t z = __ballot_sync(0xffffffffu, in && (!t.zone || t.zone[base + k]));
            if (lane == 0) {
                h.pmask[u] = m;
                zcore[u] = z;
                if (m) atomicAdd(&s_n[1], __popc(m));
            }
        }
        __syncthreads();
        for (int u = tid; u < S * RW; u += NT) {
            const int y = u / RW, w = u - y * RW;
            uint32_t c = 0u;
            if (y > 0 && y < S - 1) {
                const uint32_t m = h.pmask[u];
                const uint32_t left = (m << 4) | (w > 0 ? h.pmask[u - 1] >> 28 : 0u);
                const uint32_t right = (m >> 4) | (w < RW - 1 ? h.pmask[u + 1] << 28 : 0u);
                c = m & left & right & h.pmask[u - RW] & h.pmask[u + RW];
            }
            core[u] = c;
            zcore[u] &= c;
        }
        const AreaPlace at{(double)t.win_org[2LL * i], (double)t.win_org[2LL * i + 1], (double)t.cell_org[2LL * i],
                           (double)t.cell_org[2LL * i + 1]};
#pragma unroll 1
        for (int kind = 0; kind < 2; ++kind) {
            if (kind == 0 ? !t.out[kMed].status : !want_zero) continue;
            double b = 0.0;
            __syncthreads();  // the masks are written; the previous kind's coefficient reads are done
            if (kind == 0) {
                // nanmedian of the level pixels inside the window (NaN if none).
                double* lv = h.coef;
                for (int k = tid; k < area; k += NT)
                    if (t.inside[base + k] && t.levelm[base + k] && !isnan(t.cells[base + k]))
                        lv[atomicAdd(&s_n[0], 1)] = (double)t.cells[base + k];
                __syncthreads();
                b = cta_median<NT>(lv, s_n[0], s_mid);
            }
            for (int k = tid; k < area; k += NT) {
                const int y = k / S, x = k - y * S;
                h.coef[(y + 2) * cp + x + 2] = t.inside[base + k] ? __dsub_rn((double)t.cells[base + k], b) : 0.0;
            }
            spline_coefs(h);
            double top_v;
            int2 top;
            area_peak(h, s_red, s_ired, &top_v, &top);
            double peak = -1.0;
            if (t.o.n_top <= h.g.Hb * h.g.Wb)
                peak = area_peak_mean(h, top_v, t.o.n_top, kF * s_n[1], &sel, s_red, s_ired);
            double edge_cut = 0.0, foot_cut = 0.0, steepest = dnan();
            if (kind == 1 && (want_edge || want_foot)) {
                // Steepness sqrt(gy^2 + gx^2) (central differences over two pixels): its sums, alone and
                // times the value, over the core and over the core in the territory.
                double s[4] = {0.0, 0.0, 0.0, 0.0};
                for (int w = warp; w < RW; w += NT / 32) {
                    const int X = w * 32 + lane, kx = X >> 2;
                    if (kx < 1 || kx > S - 2) continue;
                    const Column c(h.coef, X);
                    double r[6], d[5], gx[5];  // rows ky .. ky + 5; differences of the rows ky .. ky + 4
#pragma unroll
                    for (int a = 0; a < 5; ++a) r[a + 1] = c.row((a + 1) * cp);
                    double r0 = c.row(0);
#pragma unroll
                    for (int a = 1; a < 5; ++a) d[a] = r[a + 1] - (a == 1 ? r0 : r[a - 1]);
#pragma unroll
                    for (int a = 1; a < 5; ++a) gx[a] = c.row_dx(a * cp);
                    // Held before step ky: r[1..5] = rows ky .. ky + 4, d[1..4], gx[1..4] of rows ky .. ky + 3.
                    for (int ky = 1; ky < S - 1; ++ky) {
#pragma unroll
                        for (int a = 0; a < 5; ++a) r[a] = r[a + 1];
                        r[5] = c.row((ky + 5) * cp);
#pragma unroll
                        for (int a = 0; a < 4; ++a) {
                            d[a] = d[a + 1];
                            gx[a] = gx[a + 1];
                        }
                        d[4] = r[5] - r[3];
                        gx[4] = c.row_dx((ky + 4) * cp);
                        if (!((core[ky * RW + w] >> lane) & 1u)) continue;
                        const bool zoned = (zcore[ky * RW + w] >> lane) & 1u;
                        double v[4], vy[4], vx[4];
                        column_taps(r, v);
                        column_taps(d, vy);
                        column_taps(gx, vx);
#pragma unroll
                        for (int p = 0; p < 4; ++p) {
                            const double st = 0.5 * sqrt(fma(vy[p], vy[p], vx[p] * vx[p]));
                            s[0] += st;
                            s[1] = fma(st, v[p], s[1]);
                            if (zoned) {
                                s[2] += st;
                                s[3] = fma(st, v[p], s[3]);
                            }
                        }
                    }
                }
                cta_sum4<NT>(s, s4);
                edge_cut = s[0] > 0.0 ? __ddiv_rn(s[1], s[0]) : INFINITY;
                if (want_foot) {
                    const double total = s[2];
                    steepest = __ddiv_rn(s[3], total > 0.0 ? total : 1.0);
                    // Second difference (both axes) of the values below the steepest level.
                    double q[4] = {0.0, 0.0, 0.0, 0.0};
                    for (int w = warp; w < RW; w += NT / 32) {
                        const int X = w * 32 + lane, kx = X >> 2;
                        if (kx < 1 || kx > S - 2) continue;
                        const Column c(h.coef, X);
                        double r[6], l[5];
#pragma unroll
                        for (int a = 0; a < 5; ++a) r[a + 1] = c.row((a + 1) * cp);
                        const double r0 = c.row(0);
#pragma unroll
                        for (int a = 1; a < 5; ++a)
                            l[a] = fma(-2.0, r[a], r[a + 1] + (a == 1 ? r0 : r[a - 1])) + c.row_dxx(a * cp);
                        for (int ky = 1; ky < S - 1; ++ky) {
#pragma unroll
                            for (int a = 0; a < 5; ++a) r[a] = r[a + 1];
                            r[5] = c.row((ky + 5) * cp);
#pragma unroll
                            for (int a = 0; a < 4; ++a) l[a] = l[a + 1];
                            l[4] = fma(-2.0, r[4], r[5] + r[3]) + c.row_dxx((ky + 4) * cp);
                            if (!((zcore[ky * RW + w] >> lane) & 1u)) continue;
                            double v[4], lv[4];
                            column_taps(r, v);
                            column_taps(l, lv);
#pragma unroll
                            for (int p = 0; p < 4; ++p)
                                if (v[p] < steepest) {
                                    q[0] += lv[p];
                                    q[1] = fma(lv[p], v[p], q[1]);
                                }
                        }
                    }
                    cta_sum4<NT>(q, s4);
                    foot_cut = total > 0.0 && q[0] > 0.0 ? __ddiv_rn(q[1], q[0]) : INFINITY;
                }
            }
            const double at_level = __dmul_rn(t.o.level, peak);
#pragma unroll 1
            for (int m = kind == 0 ? kMed : kNorm; m <= (kind == 0 ? kMed : kGiven); ++m) {
                if (!t.out[m].status) continue;
                const double cut = m == kEdge ? edge_cut : m == kFoot ? foot_cut : m == kGiven ? t.cuts[i] : at_level;
                area_output(h, t.o, t.out[m], i, b, peak, cut, m == kFoot ? steepest : dnan(), top, at, s_mom, s_red);
            }
        }
    }
}

// Persistent CTAs of an area kernel, as its shared memory and registers allow per SM.
template <class K>
int area_ctas(K kernel, int threads, size_t smem) {
    if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 0;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess) return 0;
    return 148 * std::max(per_sm, 1);
}

}  // namespace
}  // namespace spx

using namespace spx;

// 128 threads for cells up to 32 px wide (one sub-pixel column each), 256 for wider ones and windows.
template <int NT>
static int launch_half(const HalfSplineArgs& a, cudaStream_t s) {
    const size_t smem = (size_t)AreaMem(a.hm, a.wm, a.o.n_angles, a.o.outlines, NT).bytes(1);
    SPX_REQUIRE(smem <= 200 * 1024, "cell stack too large for the half-area kernel");
    const int ctas = area_ctas(k_half_area_spline<NT>, NT, smem);
    SPX_REQUIRE(ctas > 0, "half-area kernel launch configuration failed");
    k_half_area_spline<NT><<<std::min(a.n, ctas), NT, smem, s>>>(a);
    return check_launch("k_half_area_spline");
}

template <int NT>
static int launch_tail(const TailSplineArgs& t, cudaStream_t s) {
    const size_t smem = (size_t)AreaMem(t.S, t.S, t.o.n_angles, t.o.outlines, NT).bytes(3);
    SPX_REQUIRE(smem <= 200 * 1024, "tail window too large for the tail kernel");
    const int ctas = area_ctas(k_tail_area_spline<NT>, NT, smem);
    SPX_REQUIRE(ctas > 0, "tail kernel launch configuration failed");
    k_tail_area_spline<NT><<<std::min(t.n, ctas), NT, smem, s>>>(t);
    return check_launch("k_tail_area_spline");
}

extern "C" {

int spx_half_area_spline_cd(const double* cleaned, const int* voronoi, const int* boxes, const int* which, int n, int hm,
                            int wm, int width, int n_angles, double level, int median, int n_top, int outlines,
                            const spx_method_out* single, const spx_method_out* averaged, void* stream) {
    SPX_REQUIRE(n >= 0 && n_angles >= 1 && hm >= 1 && wm >= 1 && n_top >= 1, "bad arguments");
    SPX_REQUIRE(level > 0.0 && level < 1.0, "level must be between 0 and 1");
    if (n == 0) return SPX_OK;
    SPX_REQUIRE(cleaned && voronoi && boxes && (single || averaged), "null pointer");
    for (const spx_method_out* o : {single, averaged})
        if (o) SPX_REQUIRE(o->centers && o->status && o->metrics && o->n_metrics >= 10, "null pointer or too few metric columns");
    // The cells spx_half_area_cd takes at this factor.
    SPX_REQUIRE((long long)hm * kF * wm * kF <= 32768 && half_area_bytes(hm, wm, kF, n_angles) <= 200 * 1024,
                "cell stack too large for the half-area kernel");
    HalfSplineArgs a{cleaned, voronoi, reinterpret_cast<const int4*>(boxes), which, n, hm, wm, width, median,
                     AreaOptions{n_angles, n_top, outlines, level}, {method_out(single), method_out(averaged)}};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return wm <= 32 ? launch_half<128>(a, s) : launch_half<256>(a, s);
}

int spx_tail_area_spline_cd(const float* cells, const uint8_t* inside, const uint8_t* level_pixels,
                            const uint8_t* territory, const int* window_origins, const int* cell_origins, int n, int side,
                            int n_angles, double level, int n_top, int outlines, const double* cuts,
                            const spx_method_out* tail, const spx_method_out* norm, const spx_method_out* edge,
                            const spx_method_out* foot, const spx_method_out* given, void* stream) {
    SPX_REQUIRE(n >= 0 && n_angles >= 1 && side >= 1 && n_top >= 1, "bad arguments");
    SPX_REQUIRE(level > 0.0 && level < 1.0, "level must be between 0 and 1");
    if (n == 0) return SPX_OK;
    SPX_REQUIRE(cells && inside && window_origins && cell_origins && (tail || norm || edge || foot || given),
                "null pointer");
    SPX_REQUIRE(!tail || level_pixels, "tail_area needs the level pixels");
    SPX_REQUIRE(!given || cuts, "foot_area_ratio needs its thresholds");
    for (const spx_method_out* o : {tail, norm, edge, given})
        if (o) SPX_REQUIRE(o->centers && o->status && o->metrics && o->n_metrics >= 10, "null pointer or too few metric columns");
    if (foot) SPX_REQUIRE(foot->centers && foot->status && foot->metrics && foot->n_metrics >= 11,
                          "null pointer or too few metric columns");
    // The windows spx_tail_area_cd takes at this factor.
    SPX_REQUIRE((long long)side * kF * side * kF <= 65536 && tail_smem_bytes(side, kF, n_angles) <= 200 * 1024,
                "tail window too large for the tail kernel");
    TailSplineArgs t{cells, inside, level_pixels, territory, window_origins, cell_origins, n, side,
                     AreaOptions{n_angles, n_top, outlines, level}, cuts,
                     {method_out(tail), method_out(norm), method_out(edge), method_out(foot), method_out(given)}};
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    return side <= 32 ? launch_tail<128>(t, s) : launch_tail<256>(t, s);
}

}  // extern "C"
