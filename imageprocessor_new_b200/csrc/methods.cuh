// What the CD method kernels share: the view of a deblended cell, the output slots of a method and
// numpy's pairwise sums.
#pragma once

#include "common.cuh"

namespace spx {
namespace {

constexpr double kPi = 3.141592653589793;

struct CellView {
    const double* roi;  // hm x wm cleaned cell (zero outside its mask)
    const int* vor;
    int4 box;
    int j;              // cell index in the Voronoi labels
    int W, hm, wm;
    __device__ __forceinline__ bool mask(int yy, int xx) const {
        return yy >= 0 && xx >= 0 && yy < box.w && xx < box.z && yy < hm && xx < wm &&
               vor[(long long)(box.y + yy) * W + (box.x + xx)] == j;
    }
};

// Output slots of one method (per cell arrays; null pointers are skipped).
struct MethodOut {
    double* centers;     // n x 2 global
    double* contours;    // n x (n_angles + 1) x 2 global, or null (metrics_only)
    uint8_t* status;     // n
    double* metrics;     // n x n_metrics, NaN where not measured
    double* center_local;  // n x 2 (radial, logquad)
    double* edge_px;     // n x n_angles (radial)
    double* eigenvalues; // n x 2 (ellipse methods)
    double* axes;        // n x 2 x 2 (ellipse methods)
    int n_metrics;
    long long col_stride;  // 0: row-major metrics; else metric q of cell i at metrics[i + q * col_stride]
    __device__ __forceinline__ struct MetricRow row(long long i) const;
};

// One cell's metrics, row-major or column-major.
struct MetricRow {
    double* p;
    long long step;
    __device__ __forceinline__ double& operator[](int q) const { return p[q * step]; }
};

__device__ __forceinline__ MetricRow MethodOut::row(long long i) const {
    return col_stride ? MetricRow{metrics + i, col_stride} : MetricRow{metrics + i * n_metrics, 1};
}

// Metric columns (same order as the Python side).
enum {
    M_AREA = 0, M_CD_EQ = 1, M_CD_X = 2, M_CD_Y = 3, M_PERIM = 4, M_BACKGROUND = 5, M_PEAK = 6,
    // ellipse methods
    M_SIG_MAJ = 7, M_SIG_MIN = 8, M_FWHM_MAJ = 9, M_FWHM_MIN = 10, M_ANGLE = 11, M_RMSE = 12,
    // area methods
    M_LOCAL_LEVEL = 7, M_THRESHOLD = 8, M_MEAN_SIGNAL = 9, M_STEEPEST = 10,
    // radial methods
    M_COVERAGE = 7
};

// numpy's sum of n values a[k * stride] along a contiguous axis (pairwise_sum): in order below 8
// values; up to 128, eight running sums (a[j], a[j + 8], ...) combined as ((r0 + r1) + (r2 + r3)) +
// ((r4 + r5) + (r6 + r7)), then the values past the last full eight in order; above 128, the two
// halves (the first a multiple of 8 long) summed that way and added.
__device__ double np_pairwise_sum(const double* a, int n, int stride) {
    if (n < 8) {
        double r = 0.0;
        for (int i = 0; i < n; ++i) r = __dadd_rn(r, a[i * stride]);
        return r;
    }
    if (n <= 128) {
        double r[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) r[j] = a[j * stride];
        int i = 8;
        for (; i < n - (n % 8); i += 8)
#pragma unroll
            for (int j = 0; j < 8; ++j) r[j] = __dadd_rn(r[j], a[(i + j) * stride]);
        double res = __dadd_rn(__dadd_rn(__dadd_rn(r[0], r[1]), __dadd_rn(r[2], r[3])),
                               __dadd_rn(__dadd_rn(r[4], r[5]), __dadd_rn(r[6], r[7])));
        for (; i < n; ++i) res = __dadd_rn(res, a[i * stride]);
        return res;
    }
    int n2 = n / 2;
    n2 -= n2 % 8;
    return __dadd_rn(np_pairwise_sum(a, n2, stride), np_pairwise_sum(a + n2 * stride, n - n2, stride));
}

// np_pairwise_sum by one warp (every lane calls it; all lanes return the sum): lanes 0-7 run the
// eight running sums of a block of up to 128 values, every lane combines them in numpy's tree and
// adds the tail; above 128 values the same halves as numpy's.
__device__ double warp_np_sum(const double* a, int n) {
    if (n > 128) {
        int n2 = n / 2;
        n2 -= n2 % 8;
        const double left = warp_np_sum(a, n2);
        return __dadd_rn(left, warp_np_sum(a + n2, n - n2));
    }
    if (n < 8) {
        double r = 0.0;
        for (int i = 0; i < n; ++i) r = __dadd_rn(r, a[i]);
        return r;
    }
    const int lane = threadIdx.x & 31, full = n - n % 8;
    double r = 0.0;
    if (lane < 8) {
        r = a[lane];
        for (int i = 8; i < full; i += 8) r = __dadd_rn(r, a[i + lane]);
    }
    double q[8];
#pragma unroll
    for (int j = 0; j < 8; ++j) q[j] = __shfl_sync(0xffffffffu, r, j);
    double res = __dadd_rn(__dadd_rn(__dadd_rn(q[0], q[1]), __dadd_rn(q[2], q[3])),
                           __dadd_rn(__dadd_rn(q[4], q[5]), __dadd_rn(q[6], q[7])));
    for (int i = full; i < n; ++i) res = __dadd_rn(res, a[i]);
    return res;
}

inline MethodOut method_out(const spx_method_out* o) {
    MethodOut m;
    if (!o) {
        m = MethodOut{nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, nullptr, 0, 0};
        return m;
    }
    m.centers = o->centers;
    m.contours = o->contours;
    m.status = o->status;
    m.metrics = o->metrics;
    m.center_local = o->center_local;
    m.edge_px = o->edge_px;
    m.eigenvalues = o->eigenvalues;
    m.axes = o->axes;
    m.n_metrics = o->n_metrics;
    m.col_stride = o->metric_col_stride;
    return m;
}

}  // namespace
}  // namespace spx
