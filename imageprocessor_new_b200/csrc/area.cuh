// What the area methods (half_area and tail families) share: where an output's positions go, and an
// output's rows once its region is known.
#pragma once

#include "methods.cuh"

namespace spx {
namespace {

constexpr int kHalfLeavesMax = 1024;  // pairwise-sum leaves of one enlarged cell (<= 128 values each)

// Doubles before the zoom operators in a half-area CTA's shared memory: cell, ring, leaf sums and
// small arrays (doubles), four bit planes, row / column counts and leaves (ints), the mask bytes.
__host__ __device__ inline long long half_ops_offset(int hm, int wm, int f, int n_angles) {
    const long long Hb = (long long)hm * f, Wb = (long long)wm * f, RW = (Wb + 31) / 32, area = (long long)hm * wm;
    const long long tmpn = Hb + Wb > 3LL * (n_angles + 1) ? Hb + Wb : 3LL * (n_angles + 1);
    const long long bytes = (2 * area + kHalfLeavesMax + tmpn) * 8 + 4 * Hb * RW * 4 + (Hb + Wb + 2 * kHalfLeavesMax) * 4 +
                            area;
    return (bytes + 7) / 8;
}

// Shared memory of one half-area CTA (see the layout in k_half_area): the cell's arrays, then the
// two zoom operators and the first product.
inline size_t half_area_bytes(int hm, int wm, int f, int n_angles) {
    return (half_ops_offset(hm, wm, f, n_angles) + (size_t)hm * f * hm + (size_t)wm * f * wm + (size_t)hm * f * wm) *
           sizeof(double);
}

// Shared memory of a tail CTA: the window (doubles), leaf sums and small arrays, five bit planes,
// row / column counts, the three masks. The enlargement, its first product (whose space also holds
// the level pixels' values before it) and the pairwise-sum leaves live in the CTA's global scratch,
// so that two CTAs fit an SM for windows up to 59 px.
__host__ __device__ inline long long tail_smem_bytes(int S, int f, int n_angles) {
    const long long Hb = (long long)S * f, RW = (Hb + 31) / 32, area = (long long)S * S;
    const long long tmpn = 2 * Hb > 3LL * (n_angles + 1) ? 2 * Hb : 3LL * (n_angles + 1);
    return (area + 2 * kHalfLeavesMax + tmpn) * 8 + 5 * Hb * RW * 4 + 2 * Hb * 4 + 3 * area;
}

// Where an area output's positions go: centres and contours are the enlargement's local positions
// plus (ox, oy); center_local is the local position itself, or with a finite lx the global centre
// minus (lx, ly) (the tail windows report it relative to the hole's own cell).
struct AreaPlace {
    double ox, oy, lx, ly;
};

struct AreaShape {
    int hm, wm, n_angles, factor, outlines;
};

// A region grown on the enlargement: whether there was a signal, whether it reaches the mask's edge,
// its sub-pixel count, centroid and spreads (sub-pixels; spreads in pixels^2), mean value, the peak,
// threshold above the local level b, and foot_area's steepest level.
struct AreaFound {
    bool signal, touch;
    long long count;
    double cx, cy, var_x, var_y, mean_signal, peak, cut, b, steepest;
};

// The rows of one area output (centre, metrics, status) and its display outline, by a CTA of NT
// threads. cur: the region's bit rows (RW words each); tmp: 3 (n_angles + 1) doubles of shared
// memory when outlines are wanted; s_perim: one double of shared memory.
template <int NT>
__device__ void area_result(const AreaShape& a, const MethodOut& out, int i, const AreaFound& fd, const uint32_t* cur,
                            int RW, double* tmp, double* s_perim, const AreaPlace& at) {
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int Hb = a.hm * a.factor, Wb = a.wm * a.factor;
    const double cx = fd.cx, cy = fd.cy, var_x = fd.var_x, var_y = fd.var_y, mean_signal = fd.mean_signal;
    const double peak = fd.peak, cut = fd.cut, steepest = fd.steepest;
    const long long count = fd.count;
    const double sx = 1.0 / a.factor, sy = sx;
    const bool pow2 = (a.factor & (a.factor - 1)) == 0;
    const double shift = (double)(a.factor - 1) / (2.0 * a.factor);
    const double cxl = __dsub_rn(__dmul_rn(cx, sx), shift), cyl = __dsub_rn(__dmul_rn(cy, sy), shift);
    const bool signal = fd.signal, ok = fd.signal && !fd.touch;
    // Display outline: along each ray from the centroid, the last 1/8 px step still in the region.
    const int nv = a.n_angles + 1;
    double* vx = tmp;
    double* vy = tmp + nv;
    if (a.outlines && signal) {
        const int nr = (int)ceil(hypot((double)a.hm, (double)a.wm) / 0.125);
        const double ang_step = 2.0 * kPi / a.n_angles;
        for (int q = tid; q < a.n_angles; q += NT) {
            const double ang = __dmul_rn((double)q, ang_step);
            const double co = cos(ang), si = sin(ang);
            int first_out = nr;
            for (int s = 0; s < nr; ++s) {
                const double st = __dmul_rn((double)s, 0.125);
                // (cos x step) / sx, a multiplication by the factor when it is a power of two (exact).
                const double ox = pow2 ? __dmul_rn(__dmul_rn(co, st), (double)a.factor) : __ddiv_rn(__dmul_rn(co, st), sx);
                const double oy = pow2 ? __dmul_rn(__dmul_rn(si, st), (double)a.factor) : __ddiv_rn(__dmul_rn(si, st), sy);
                const double fx = rint(__dadd_rn(cx, ox));
                const double fy = rint(__dadd_rn(cy, oy));
                bool hit = fx >= 0.0 && fx < (double)Wb && fy >= 0.0 && fy < (double)Hb;
                if (hit) {
                    const int X = (int)fx, Y = (int)fy;
                    hit = (cur[Y * RW + X / 32] >> (X % 32)) & 1u;
                }
                if (!hit) {
                    first_out = s;
                    break;
                }
            }
            const double e = __dadd_rn(__dmul_rn((double)max(first_out - 1, 0), 0.125), 0.0625);
            if (out.edge_px) out.edge_px[(long long)i * a.n_angles + q] = e;
            vx[q] = __dadd_rn(__dadd_rn(cxl, __dmul_rn(e, co)), at.ox);
            vy[q] = __dadd_rn(__dadd_rn(cyl, __dmul_rn(e, si)), at.oy);
        }
        __syncthreads();
        if (tid == 0) {
            vx[a.n_angles] = vx[0];
            vy[a.n_angles] = vy[0];
        }
        __syncthreads();
        if (out.contours)
            for (int k = tid; k < nv; k += NT) {
                out.contours[((long long)i * nv + k) * 2] = vx[k];
                out.contours[((long long)i * nv + k) * 2 + 1] = vy[k];
            }
        // Perimeter: the closed polygon's side lengths, summed in numpy's order by one warp.
        double* side = tmp + 2 * nv;
        for (int q = tid; q < a.n_angles; q += NT) {
            const double dx = __dsub_rn(vx[q + 1], vx[q]), dy = __dsub_rn(vy[q + 1], vy[q]);
            side[q] = sqrt(__dadd_rn(__dmul_rn(dx, dx), __dmul_rn(dy, dy)));
        }
        __syncthreads();
        if (warp == 0) {
            const double v = warp_np_sum(side, a.n_angles);
            if (lane == 0) *s_perim = v;
        }
    } else {
        if (out.edge_px)
            for (int q = tid; q < a.n_angles; q += NT) out.edge_px[(long long)i * a.n_angles + q] = dnan();
        if (out.contours)
            for (int k = tid; k < 2 * nv; k += NT) out.contours[(long long)i * 2 * nv + k] = dnan();
    }
    __syncthreads();
    if (tid == 0) {
        const MetricRow m = out.row(i);
        for (int q = 0; q < out.n_metrics; ++q) m[q] = dnan();
        m[M_LOCAL_LEVEL] = fd.b;
        out.status[i] = (uint8_t)(!signal ? SPX_ST_NO_SIGNAL : fd.touch ? SPX_ST_REGION_AT_CELL_BORDER : SPX_ST_OK);
        const double nan = dnan();
        const double gcx = __dadd_rn(cxl, at.ox), gcy = __dadd_rn(cyl, at.oy);
        out.centers[2LL * i] = signal ? gcx : nan;
        out.centers[2LL * i + 1] = signal ? gcy : nan;
        if (out.center_local) {
            const bool rel = isfinite(at.lx);
            out.center_local[2LL * i] = signal ? (rel ? __dsub_rn(gcx, at.lx) : cxl) : nan;
            out.center_local[2LL * i + 1] = signal ? (rel ? __dsub_rn(gcy, at.ly) : cyl) : nan;
        }
        if (signal) {
            m[M_PEAK] = peak;
            m[M_THRESHOLD] = __dadd_rn(fd.b, cut);
            m[M_MEAN_SIGNAL] = mean_signal;
            if (out.n_metrics > M_STEEPEST) m[M_STEEPEST] = steepest;
        }
        if (ok) {
            const double area = __dmul_rn((double)count, __dmul_rn(sx, sy));
            const double cd_eq = __dmul_rn(2.0, sqrt(__ddiv_rn(area, kPi)));
            const double ratio = sqrt(sqrt(__ddiv_rn(fmax(var_x, 1e-12), fmax(var_y, 1e-12))));
            m[M_AREA] = area;
            m[M_CD_EQ] = cd_eq;
            m[M_CD_X] = __dmul_rn(cd_eq, ratio);
            m[M_CD_Y] = __ddiv_rn(cd_eq, ratio);
            if (a.outlines) m[M_PERIM] = *s_perim;
        }
    }
    __syncthreads();
}

}  // namespace
}  // namespace spx
