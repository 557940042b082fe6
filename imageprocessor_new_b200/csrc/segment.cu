// Segmentation: Otsu threshold, binarisation and connected-component labelling with stats.
//
// Replaces, for the subpx hot path:
//   cv2.threshold(..., THRESH_OTSU)            subpx/_cpu/centers.py:247-266, subpx/_gpu/centers.py:1789-1796
//   cv2.connectedComponentsWithStats           subpx/_cpu/components.py:18-32
//
// Otsu: a shared-memory histogram over the occupied value range, then OpenCV's published Otsu scan
// (between-class variance q1*q2*(mu1-mu2)^2, first maximum, bins skipped while min(q1,q2) <
// FLT_EPSILON). The scan's running sums are rounded sequentially by one thread so that the chosen
// bin is the one OpenCV chooses.
//
// CCL: union-find in two levels. Parents live in a canonical-order array: for 8-connectivity the
// pixels of each 2x2 block are contiguous and blocks follow the row-pair scan, for 4-connectivity
// canonical order is raster order. Unions always link the larger id under the smaller, so the root
// of a component is its first pixel in that order, and OpenCV's label numbering is the rank of the
// root among all roots: a bitmap of roots plus a prefix count of its words.
//   k_local_ccl     one warp per 32x64 tile: binarise, union-find in shared memory, write parents
//   k_border_merge  unions across tile borders in global memory (lock-free atomicMin linking)
//   scan            popcount prefix of the root bitmap -> component count K
//   k_finish        final raster labels (rank of the root) + stats by run, one warp per 32x64 tile

#include "common.cuh"

#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <mutex>

namespace spx {

static thread_local char g_error[1024];
static unsigned long long g_launches = 0;  // kernel launches issued by this library (all threads)

void set_error(const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_error, sizeof(g_error), fmt, ap);
    va_end(ap);
}

Tuning& tuning() {
    static Tuning t;
    return t;
}

int check_launch(const char* what) {
    __atomic_add_fetch(&g_launches, 1ull, __ATOMIC_RELAXED);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) {
        set_error("%s launch failed: %s", what, cudaGetErrorString(e));
        return SPX_ERR_CUDA;
    }
    return SPX_OK;
}

namespace {

constexpr int kHistSmemBins = 16384;  // value ranges up to this use a shared-memory histogram
constexpr int kScanPerBlock = 4096;   // bitmap words per prefix block (1024 threads x 4)
constexpr int kTileH = 32;            // CCL tile (even height keeps 2x2 blocks inside one tile)
constexpr int kTileW = 64;

// ------------------------------------------------------------------------------------------ Otsu

__device__ __forceinline__ unsigned int px_u(const void* img, int dtype, long long i) {
    return dtype == SPX_U8 ? (unsigned int)static_cast<const uint8_t*>(img)[i]
                           : (unsigned int)static_cast<const uint16_t*>(img)[i];
}

// An empty histogram and its range preset, in one launch (a memset and an 8-byte copy from pageable memory cost
// the host 8 us more).
__global__ void k_hist_init(unsigned int* hist, int n, unsigned int* range, unsigned int lo, unsigned int hi) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) hist[i] = 0u;
    if (threadIdx.x == 0 && blockIdx.x == 0) {
        range[0] = lo;
        range[1] = hi;
    }
}

// range[0] = min, range[1] = max of the sampled pixels (range must be preset to {~0u, 0}).
__global__ void k_minmax(const void* img, int dtype, int height, int width, int step,
                         unsigned int* range) {
    const int hs = (int)(((long long)height + step - 1) / step), ws = (int)(((long long)width + step - 1) / step);
    const long long n = (long long)hs * ws;
    unsigned int lo = 0xffffffffu, hi = 0;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        int yi, xi;
        divmod_idx(k, ws, &yi, &xi);
        const long long y = yi, x = xi;
        const unsigned int v = px_u(img, dtype, y * step * (long long)width + x * step);
        lo = min(lo, v);
        hi = max(hi, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&range[0], lo);
        atomicMax(&range[1], hi);
    }
}

// k_minmax for a contiguous, 16-byte aligned uint16 image: eight pixels per 16-byte load.
__global__ void k_minmax_dense(const uint16_t* img, long long n, unsigned int* range) {
    unsigned int lo = 0xffffffffu, hi = 0;
    const uint4* v4 = reinterpret_cast<const uint4*>(img);
    const long long n8 = n / 8;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n8;
         k += (long long)gridDim.x * blockDim.x) {
        const uint4 q = __ldg(v4 + k);
        const unsigned int w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const unsigned int a = w[j] & 0xffffu, b = w[j] >> 16;
            lo = min(lo, min(a, b));
            hi = max(hi, max(a, b));
        }
    }
    for (long long k = n8 * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
         k += (long long)gridDim.x * blockDim.x) {
        const unsigned int v = img[k];
        lo = min(lo, v);
        hi = max(hi, v);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = min(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        hi = max(hi, __shfl_xor_sync(0xffffffffu, hi, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMin(&range[0], lo);
        atomicMax(&range[1], hi);
    }
}

// Histogram of the sampled pixels into hist[65536] (pre-zeroed, u32).
__global__ void k_histogram(const void* img, int dtype, int height, int width, int step,
                            int dense, const unsigned int* range, unsigned int* hist) {
    extern __shared__ unsigned int sh[];
    const unsigned int lo = range[0], hi = range[1];
    const unsigned int nb = hi >= lo ? hi - lo + 1 : 0;
    const bool in_smem = nb <= (unsigned int)kHistSmemBins;
    if (in_smem) {
        for (unsigned int i = threadIdx.x; i < nb; i += blockDim.x) sh[i] = 0;
        __syncthreads();
    }
    const int hs = (int)(((long long)height + step - 1) / step), ws = (int)(((long long)width + step - 1) / step);
    const long long n = (long long)hs * ws;
    if (dense) {
        // 16-byte loads of 8 pixels, then the ragged tail.
        const uint4* v4 = static_cast<const uint4*>(img);
        const long long n8 = n / 8;
        for (long long k = n8 * 8 + blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
             k += (long long)gridDim.x * blockDim.x) {
            const unsigned int v = static_cast<const uint16_t*>(img)[k];
            if (in_smem) atomicAdd(&sh[v - lo], 1u);
            else atomicAdd(&hist[v], 1u);
        }
        for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n8;
             k += (long long)gridDim.x * blockDim.x) {
            const uint4 q = __ldg(v4 + k);
            const unsigned int w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const unsigned int a = w[j] & 0xffffu, b = w[j] >> 16;
                if (in_smem) {
                    atomicAdd(&sh[a - lo], 1u);
                    atomicAdd(&sh[b - lo], 1u);
                } else {
                    atomicAdd(&hist[a], 1u);
                    atomicAdd(&hist[b], 1u);
                }
            }
        }
    } else {
        for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < n;
             k += (long long)gridDim.x * blockDim.x) {
            int yi, xi;
        divmod_idx(k, ws, &yi, &xi);
        const long long y = yi, x = xi;
            const unsigned int v = px_u(img, dtype, y * step * (long long)width + x * step);
            if (in_smem) atomicAdd(&sh[v - lo], 1u);
            else atomicAdd(&hist[v], 1u);
        }
    }
    if (in_smem) {
        __syncthreads();
        for (unsigned int i = threadIdx.x; i < nb; i += blockDim.x)
            if (sh[i]) atomicAdd(&hist[lo + i], sh[i]);
    }
}

// Certified parallel Otsu: the bin that OpenCV's sequential FP64 scan chooses, found without the
// scan whenever the exact rational between-class variances single it out.
//
// For bin i with integer prefix sums Q = sum_{j<=i} h_j and S = sum_{j<=i} j h_j (N pixels, grey
// sum M), the exact variance is sigma2 = (S N - Q M)^2 / (N^2 Q (N - Q)), and mu1 - mu2 =
// (S N - Q M) / (Q (N - Q)). OpenCV's loop computes q1 as a running FP64 sum of h_j / N (relative
// error <= (n + 2) u for n bins, u = 2^-53), mu1 by a recurrence whose product mu1 q1 is a running
// sum of j h_j / N (relative error <= 4 (n + 2) u), mu2 = (mu - q1 mu1) / q2 and sigma2 = q1 q2
// (mu1 - mu2)^2. From these error terms every bin gets an interval [lo, hi] that holds OpenCV's
// rounded sigma2 (each term inflated four times), and the skip test min(q1, q2) < FLT_EPSILON is
// decided on the exact q1 = Q / N unless q1 or q2 lies within 1e-9 of FLT_EPSILON or of
// 1 - FLT_EPSILON (a bin that might go either way). When the bin i* with the largest lo among the
// surely unskipped bins has lo > 0 and lo above every other not-surely-skipped bin's hi, OpenCV's
// strict-maximum scan must choose i*: returns true with the threshold. Otherwise (near-ties,
// ambiguous skips) returns false and the caller runs the sequential scan. Block-uniform result;
// needs blockDim.x == 1024 and 16 KB of shared memory at s_buf.
//
// Bound: one SM's FP64 rate. The intervals take five divisions and a 128-bit difference a bin, so they are
// computed for i* and for the few bins a coarser upper bound does not already rule out: i* is the bin
// with the largest D^2 / (Q R), D = S N - Q M in doubles, compared by cross products; any other bin with
// q1, q2 >= 1e-3 has hi < (1 + 2e-7) (|D| + E Q R)^2 / (N^2 Q R), where E = 3e4 g M_max bounds the
// interval's error of mu1 - mu2 (both means are at most M_max, the highest grey value, and mu / (q2 mu2)
// <= 1 / q2 <= 1e3), and is passed over when that is below i*'s lo. A 1024 x 1024 frame, with every
// interval in full twice: 35 us; now 18 us.
__device__ bool otsu_certified(const unsigned int* hist, int first, int n, long long total,
                               unsigned long long grey_sum, double* s_buf, double* threshold) {
    constexpr int T = 1024;
    unsigned long long *s_q = reinterpret_cast<unsigned long long*>(s_buf), *s_m = s_q + T;
    __shared__ double s_val[32];
    __shared__ int s_idx[32];
    __shared__ double s_best_lo;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int per = (n + T - 1) / T, b0 = min(n, t * per), b1 = min(n, b0 + per);
    unsigned long long cq = 0, cm = 0;
    for (int k = b0; k < b1; ++k) {
        const unsigned long long h = hist[first + k];
        cq += h;
        cm += h * (unsigned long long)(first + k);
    }
    s_q[t] = cq;
    s_m[t] = cm;
    __syncthreads();
    for (int o = 1; o < T; o <<= 1) {  // inclusive scan of the chunk totals
        const unsigned long long aq = t >= o ? s_q[t - o] : 0ull, am = t >= o ? s_m[t - o] : 0ull;
        __syncthreads();
        s_q[t] += aq;
        s_m[t] += am;
        __syncthreads();
    }
    const unsigned long long q_start = s_q[t] - cq, m_start = s_m[t] - cm;
    const double Nd = (double)total, invN = 1.0 / Nd;
    const double u = 1.1102230246251565e-16;
    const double eps = 1.1920928955078125e-07, win = 1e-9;
    const double g = (double)(n + 2) * u;
    const double mu = (double)grey_sum * invN;
    // cls: 0 surely skipped, 1 surely unskipped, 2 either. lo / hi: the interval of OpenCV's sigma2.
    auto eval = [&](unsigned long long Q, unsigned long long S, double* lo, double* hi) -> int {
        const unsigned long long R = (unsigned long long)total - Q;
        const double q1 = (double)Q * invN, q2 = (double)R * invN;
        const bool amb = fabs(q1 - eps) <= win || fabs(q2 - eps) <= win || fabs(q1 - (1.0 - eps)) <= win ||
                         fabs(q2 - (1.0 - eps)) <= win;
        const bool skip = fmin(q1, q2) < eps || fmax(q1, q2) > 1.0 - eps;
        if (skip && !amb) return 0;
        if (Q == 0 || R == 0) {  // q1 or q2 exactly 0 cannot be unskipped (amb never holds here)
            *lo = *hi = 0.0;
            return 0;
        }
        const __int128 D = (__int128)S * (__int128)total - (__int128)Q * (__int128)grey_sum;
        const double qr = (double)Q * (double)R;
        const double d = (double)D / qr;                  // mu1 - mu2
        const double ad = fabs(d);
        const double mu1 = (double)S / (double)Q;
        const double mu2 = (double)(grey_sum - S) / (double)R;
        const double rel_q1 = 4.0 * g;
        const double rel_q2 = 4.0 * (g * q1 + u) / q2;
        const double num = q2 * mu2;                      // mu - q1 mu1, > 0 here
        const double rel_mu2 = (5.0 * g + u) * mu / fmax(num, 1e-300) + (g * q1 + u) / q2 + u;
        const double err_d = 4.0 * (4.0 * g * mu1 + mu2 * rel_mu2 + u * ad);
        const double base = q1 * q2;
        *hi = base * (1.0 + rel_q1) * (1.0 + rel_q2) * (ad + err_d) * (ad + err_d) * (1.0 + 16.0 * u);
        const double dl = fmax(ad - err_d, 0.0);
        *lo = rel_q2 >= 1.0 ? 0.0 : base * (1.0 - rel_q1) * (1.0 - rel_q2) * dl * dl * (1.0 - 16.0 * u);
        return amb ? 2 : 1;
    };
    const double Md = (double)grey_sum;  // all sums are integers below 2^53
    // Pass 1: the surely unskipped bin with the largest exact variance, to rounding (lowest index on ties).
    double bn = 0.0, bd = 1.0;
    unsigned long long bQ = 0, bS = 0;
    int best = 0x7fffffff;
    {
        double Q = (double)q_start, S = (double)m_start;
        for (int k = b0; k < b1; ++k) {
            const double h = (double)hist[first + k];
            Q += h;
            S = __fma_rn(h, (double)(first + k), S);
            const double R = Nd - Q, q1 = Q * invN, q2 = R * invN;
            if (fmin(q1, q2) < eps + win || fmax(q1, q2) > 1.0 - eps - win) continue;
            const double D = S * Nd - Q * Md, num = D * D, den = Q * R;
            if (num * bd > bn * den) {
                bn = num;
                bd = den;
                best = k;
                bQ = (unsigned long long)Q;
                bS = (unsigned long long)S;
            }
        }
    }
    double score = bn / bd;
    int star = best;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, score, o);
        const int oi = __shfl_xor_sync(0xffffffffu, star, o);
        if (ov > score || (ov == score && oi < star)) { score = ov; star = oi; }
    }
    if (lane == 0) { s_val[warp] = score; s_idx[warp] = star; }
    __syncthreads();
    score = s_val[0];
    star = s_idx[0];
    for (int w = 1; w < T / 32; ++w)
        if (s_val[w] > score || (s_val[w] == score && s_idx[w] < star)) { score = s_val[w]; star = s_idx[w]; }
    if (star == 0x7fffffff) return false;
    if (best == star) {
        double lo, hi;
        s_best_lo = eval(bQ, bS, &lo, &hi) == 1 ? lo : -1.0;
    }
    __syncthreads();
    const double star_lo = s_best_lo;
    // Pass 2: the largest upper bound of the other bins that may be unskipped and reach star_lo.
    double other_hi = 0.0;
    if (star_lo > 0.0) {
        const double E = 3e4 * g * (double)(first + n - 1), floor_n2 = star_lo * Nd * Nd;
        unsigned long long Q = q_start, S = m_start;
        for (int k = b0; k < b1; ++k) {
            const unsigned long long h = hist[first + k];
            Q += h;
            S += h * (unsigned long long)(first + k);
            if (k == star) continue;
            const double Qd = (double)Q, R = Nd - Qd, sn = (double)S * Nd, qm = Qd * Md, qr = Qd * R;
            if (fmin(Qd, R) * invN >= 1e-3) {
                const double top_d = fabs(sn - qm) + 4.0 * u * (sn + qm) + E * qr;
                if (top_d * top_d * (1.0 + 2e-7) < floor_n2 * qr) continue;
            }
            double lo, hi;
            if (eval(Q, S, &lo, &hi) != 0) other_hi = fmax(other_hi, hi);
        }
    }
    other_hi = warp_max(other_hi);
    if (lane == 0) s_val[warp] = other_hi;
    __syncthreads();
    double top = 0.0;
    for (int w = 0; w < T / 32; ++w) top = fmax(top, s_val[w]);
    const bool ok = star_lo > 0.0 && star_lo > top;
    if (ok && t == 0) *threshold = (double)(first + star);
    return ok;
}

// OpenCV's Otsu scan (getThreshVal_Otsu) over bins [0, N), by one block; where the certified pick does not
// decide, 1,024 bins at a time in shared memory:
//   A  p_i = h[i] * scale (parallel), then q1_i = q1_{i-1} + p_i by one thread (additions only);
//   B  y_i = RN(1 / q1_i) and i p_i (parallel);
//   C  the mu1 recurrence by one thread: mu1 <- mu1 * q1_{i-1}; unless bin i is skipped,
//      mu1 <- RN((mu1 + i p_i) / q1_i), the quotient by Markstein's correction
//      (q = RN(a y); r = a - q q1 exactly by FMA; RN(q + r y) = RN(a / q1) when y = RN(1 / q1));
//   D  sigma_i = q1 q2 (mu1 - mu2)^2 for every unskipped bin and the first maximum (parallel).
// Every value is rounded exactly as OpenCV's sequential loop rounds it, so the chosen bin is OpenCV's.
//
// Bound: the latency of C's five dependent operations a bin. With the arrays in global memory, loaded at the
// head of each eight bins, the loads were most of it: 480 us on a
// panel's sample whose valley is empty; now 154 us.
__global__ void __launch_bounds__(1024) k_otsu_scan(const unsigned int* hist, int nbins,
                                                    const unsigned int* range, long long total,
                                                    double* threshold) {
    constexpr int kChunk = 1024, kUnroll = 8;
    __shared__ unsigned long long s_mu[32];
    __shared__ double s_best[32];
    __shared__ int s_arg[32];
    __shared__ double s_buf[4 * kChunk];
    double *s_p = s_buf, *s_q1 = s_p + kChunk, *s_y = s_q1 + kChunk, *s_mu1 = s_y + kChunk;
    const int t = threadIdx.x;
    int first = (int)range[0], last = (int)range[1];
    if (first < 0) first = 0;
    if (last > nbins - 1) last = nbins - 1;
    const int n = last - first + 1;
    unsigned long long mu_part = 0;
#pragma unroll 16
    for (int i = t; i < nbins; i += 1024) mu_part += (unsigned long long)i * hist[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mu_part += __shfl_xor_sync(0xffffffffu, mu_part, o);
    if ((t & 31) == 0) s_mu[t >> 5] = mu_part;
    const double scale = 1.0 / (double)total;
    __syncthreads();
    unsigned long long mu_int = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) mu_int += s_mu[w];
    if (n > 0 && otsu_certified(hist, first, n, total, mu_int, s_buf, threshold)) return;
    // The reference sums i*h[i] sequentially in double: every partial sum is an integer below 2^53,
    // hence exact, and equal to this integer sum.
    const double mu = __dmul_rn((double)mu_int, scale);
    const double eps = (double)1.1920928955078125e-07f;
    const double one_minus_eps = __dsub_rn(1.0, eps);
    // Bins below the first occupied one leave mu1 = q1 = 0 and are all skipped; bins above the last
    // occupied one have q2 < FLT_EPSILON and are skipped as well.
    double run_q1 = 0.0, run_mu1 = 0.0, q1_prev = 0.0;  // thread 0's recurrences
    double best = 0.0;
    int arg = 0x7fffffff;
    for (int c0 = 0; c0 < n; c0 += kChunk) {
        const int m = min(kChunk, n - c0);
        // Bins past the end are zero: they add nothing to q1 and are not read back.
        const double p = t < m ? __dmul_rn((double)hist[first + c0 + t], scale) : 0.0;
        s_p[t] = p;
        __syncthreads();
        if (t == 0) {
            for (int k = 0; k < m; k += kUnroll) {
#pragma unroll
                for (int j = 0; j < kUnroll; ++j) {
                    run_q1 = __dadd_rn(run_q1, s_p[k + j]);
                    s_q1[k + j] = run_q1;
                }
            }
        }
        __syncthreads();
        const double q1 = s_q1[t], q2 = __dsub_rn(1.0, q1);
        const bool skip = t >= m || fmin(q1, q2) < eps || fmax(q1, q2) > one_minus_eps;
        s_y[t] = skip ? dnan() : __drcp_rn(q1);
        s_p[t] = __dmul_rn((double)(first + c0 + t), p);
        __syncthreads();
        if (t == 0) {
            for (int k = 0; k < m; k += kUnroll) {
#pragma unroll
                for (int j = 0; j < kUnroll; ++j) {
                    const double qk = s_q1[k + j], y = s_y[k + j];
                    run_mu1 = __dmul_rn(run_mu1, q1_prev);
                    q1_prev = qk;
                    const double a = __dadd_rn(run_mu1, s_p[k + j]);
                    const double q = __dmul_rn(a, y);
                    const double r = __fma_rn(-q, qk, a);
                    const double v = __fma_rn(r, y, q);
                    s_mu1[k + j] = v;
                    run_mu1 = isnan(y) ? run_mu1 : v;  // a skipped bin
                }
            }
        }
        __syncthreads();
        if (!skip) {
            const double mu1 = s_mu1[t];
            const double mu2 = __ddiv_rn(__dsub_rn(mu, __dmul_rn(q1, mu1)), q2);
            const double d = __dsub_rn(mu1, mu2);
            const double sigma = __dmul_rn(__dmul_rn(__dmul_rn(q1, q2), d), d);
            // First maximum strictly above 0 (OpenCV starts from max_sigma = 0, bin 0).
            if (sigma > best) { best = sigma; arg = c0 + t; }
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double ob = __shfl_xor_sync(0xffffffffu, best, o);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
        if (ob > best || (ob == best && oa < arg)) { best = ob; arg = oa; }
    }
    if ((threadIdx.x & 31) == 0) { s_best[threadIdx.x >> 5] = best; s_arg[threadIdx.x >> 5] = arg; }
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        int a = 0x7fffffff;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w)
            if (s_best[w] > b || (s_best[w] == b && s_arg[w] < a)) { b = s_best[w]; a = s_arg[w]; }
        *threshold = (b > 0.0 && a != 0x7fffffff) ? (double)(first + a) : 0.0;
    }
}

// OpenCV's triangle threshold (getThreshVal_Triangle_8u) over a 256-bin histogram: the bin of
// maximum distance to the line from the histogram peak to the far end of the occupied range. One bin per
// thread; ends, peak and farthest bin by block reductions with the scan's tie rules (the lowest index wins
// everywhere; a distance counts above zero only). 256 threads.
__global__ void __launch_bounds__(256) k_triangle_scan(const unsigned int* hist, double* threshold) {
    constexpr int N = 256;
    __shared__ unsigned int h[N];
    __shared__ int s_left, s_right;
    __shared__ unsigned long long s_peak;
    __shared__ double s_dist[8];
    __shared__ int s_at[8];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    h[t] = hist[t];
    if (t == 0) {
        s_left = N;
        s_right = -1;
        s_peak = 0ull;
    }
    __syncthreads();
    if (h[t] > 0) {
        atomicMin(&s_left, t);
        if (t > 0) atomicMax(&s_right, t);
        atomicMax(&s_peak, ((unsigned long long)h[t] << 32) | (unsigned)(N - 1 - t));
    }
    __syncthreads();
    int left = s_left < N ? s_left : 0, right = s_right > 0 ? s_right : 0;
    if (left > 0) left--;
    if (right < N - 1) right++;
    const long long mx = (long long)(s_peak >> 32);
    int max_ind = mx > 0 ? N - 1 - (int)(s_peak & 0xffffffffu) : 0;
    const bool flipped = max_ind - left < right - max_ind;
    if (flipped) {
        left = N - 1 - right;
        max_ind = N - 1 - max_ind;
    }
    const double a = (double)mx, b = (double)(left - max_ind);
    double dist = 0.0;
    int at = N;
    if (t > left && t <= max_ind) {
        const double d = __dadd_rn(__dmul_rn(a, (double)t), __dmul_rn(b, (double)h[flipped ? N - 1 - t : t]));
        if (d > 0.0) {
            dist = d;
            at = t;
        }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double od = __shfl_xor_sync(0xffffffffu, dist, o);
        const int oa = __shfl_xor_sync(0xffffffffu, at, o);
        if (od > dist || (od == dist && oa < at)) {
            dist = od;
            at = oa;
        }
    }
    if (lane == 0) {
        s_dist[warp] = dist;
        s_at[warp] = at;
    }
    __syncthreads();
    if (t == 0) {
        for (int w = 1; w < 8; ++w)
            if (s_dist[w] > dist || (s_dist[w] == dist && s_at[w] < at)) {
                dist = s_dist[w];
                at = s_at[w];
            }
        double thresh = (at < N ? at : left) - 1.0;
        if (flipped) thresh = (N - 1) - thresh;
        *threshold = thresh;
    }
}

// -------------------------------------------------------------------------------------------- CCL

struct Geo {
    int H, W, Wb;   // image size; blocks per row pair (8-connectivity)
    int conn;       // 8 or 4
    __device__ __forceinline__ int canon(int y, int x) const {
        return conn == 8 ? ((((y >> 1) * Wb + (x >> 1)) << 2) | ((y & 1) << 1) | (x & 1)) : y * W + x;
    }
    // Foreground bitmap: bit x & 31 of word y * words_per_row + x / 32 (rows padded to 64 bits).
    // Only local roots and foreground pixels on tile edges have an entry in the parents array;
    // readers test the bitmap first.
    __device__ __forceinline__ int words_per_row() const { return (W + 63) / 64 * 2; }
    __device__ __forceinline__ bool fg(const unsigned* bits, int y, int x) const {
        return (bits[(long long)y * words_per_row() + (x >> 5)] >> (x & 31)) & 1u;
    }
};

__device__ __forceinline__ bool is_fg(double v, double t, int invert) { return invert ? v <= t : v > t; }

// Root of a, halving the path on the way (each visited node is re-pointed to its grandparent, an
// ancestor, so concurrent finds and unions stay valid).
__device__ __forceinline__ int find_root_volatile(volatile int* p, int a) {
    while (true) {
        const int b = p[a];
        if (b == a) return a;
        const int c = p[b];
        if (c == b) return b;
        p[a] = c;
        a = c;
    }
}

// Lock-free union (link the larger root under the smaller with atomicMin; retry from the value
// that was there when another thread won the race). Clears the root bit of a root that gets linked.
__device__ void unite(int* p, int a, int b, unsigned int* roots) {
    while (true) {
        a = find_root_volatile(p, a);
        b = find_root_volatile(p, b);
        if (a == b) return;
        if (a < b) {
            const int t = a;
            a = b;
            b = t;
        }
        const int old = atomicMin(&p[a], b);
        if (old == a) {
            if (roots) atomicAnd(&roots[a >> 5], ~(1u << (a & 31)));
            return;
        }
        a = old;
    }
}

// ---------------------------------------------------------------------- run-based tile union-find
//
// A 32 x 64 tile is 32 row masks (bit x of mask[r] = pixel (ty0 + r, tx0 + x) is foreground). The
// union-find runs over the row runs, lane r of a warp holding row r: runs touch when their columns overlap
// (widened by one for 8-connectivity). A run's node is 32 r + start / 2 (runs of a row start at least two
// apart), 4 KB a tile. Nodes follow the raster scan, so a run's first neighbour in the row above is a
// smaller node and its parent without any search; only a run that touches a second one needs a union.
// A component's canonical id is then the smallest of its runs' first pixels, which for 8-connectivity (2x2
// blocks in scan order) is a run of the root's row or, below an even row, of the next one. Both CCL kernels
// rebuild the same forest from the bitmap; the result does not depend on the order of the unions.

// One warp does a tile from its pixels to its labels: no barriers between its serial parts, and four
// tiles per block hide one another's latency.
constexpr int kCclWarps = 4;
constexpr int kCclThreads = 32 * kCclWarps;
constexpr int kTileNodes = kTileH * kTileW / 2;

__device__ __forceinline__ int tile_lidx(int conn, int yl, int xl) {
    return conn == 8 ? ((((yl >> 1) * (kTileW / 2) + (xl >> 1)) << 2) | ((yl & 1) << 1) | (xl & 1))
                     : yl * kTileW + xl;
}

// First column of the run of set bits of m that holds bit x.
__device__ __forceinline__ int run_first(unsigned long long m, int x) {
    const unsigned long long below = ~m & ((1ull << x) - 1ull);
    return below ? 64 - __clzll((long long)below) : 0;
}

// Last column of the run of set bits of m that holds bit x.
__device__ __forceinline__ int run_last(unsigned long long m, int x) {
    const unsigned long long above = ~m & ~((1ull << x) - 1ull);
    return above ? __ffsll((long long)above) - 2 : 63;
}

__device__ __forceinline__ int run_node(int r, int first) { return r * 32 + (first >> 1); }

// Every run's parent becomes its root (starts: this lane's run starts). Each entry is written by its own
// lane only, with an ancestor of every value it had. Full warp.
__device__ __forceinline__ void tile_flatten(unsigned long long starts, int* par, int lane) {
    bool changed;
    do {
        changed = false;
        for (unsigned long long s = starts; s; s &= s - 1) {
            const int l = run_node(lane, __ffsll((long long)s) - 1);
            const int p = par[l], q = par[p];
            if (q != p) {
                par[l] = q;
                changed = true;
            }
        }
        __syncwarp();
    } while (__any_sync(0xffffffffu, changed));
}

// Builds the tile forest in par[] (by run node; only run nodes are written) from the row masks: a run that
// is not a root points at its root, a root holds ~l, l the component's smallest local canonical id.
// Called by a full warp, lane r holding row r's mask.
__device__ void tile_forest(unsigned long long m, int conn, int* par, int lane) {
    const unsigned long long starts = m & ~(m << 1);
    const unsigned long long above = __shfl_up_sync(0xffffffffu, m, 1);
    const unsigned long long mp = lane > 0 ? above : 0ull;
    const unsigned long long reach = conn == 8 ? mp | (mp << 1) | (mp >> 1) : mp;
    // The runs of the row above that run a..b touches, as columns of mp.
    auto touched = [&](int a, int b) {
        const int lo = conn == 8 ? max(a - 1, 0) : a, hi = conn == 8 ? min(b + 1, 63) : b;
        return mp & ((2ull << hi) - 1ull) & ~((1ull << lo) - 1ull);
    };
    unsigned long long again = 0;  // starts of the runs that touch more than one
    for (unsigned long long s = starts; s; s &= s - 1) {
        const int a = __ffsll((long long)s) - 1;
        const int me = run_node(lane, a);
        int p = me;
        const int b = run_last(m, a);
        if (reach & ((2ull << b) - 1ull) & ~((1ull << a) - 1ull)) {
            const unsigned long long t = touched(a, b);
            const int c = __ffsll((long long)t) - 1, e = run_last(mp, c);
            p = run_node(lane - 1, run_first(mp, c));
            if (t & ~((2ull << e) - 1ull)) again |= s & (~s + 1ull);
        }
        par[me] = p;
    }
    __syncwarp();
    tile_flatten(starts, par, lane);
    if (__any_sync(0xffffffffu, again != 0ull)) {
        for (unsigned long long s = again; s; s &= s - 1) {
            const int a = __ffsll((long long)s) - 1;
            unsigned long long t = touched(a, run_last(m, a));
            while (true) {
                const int e = run_last(mp, __ffsll((long long)t) - 1);
                t &= ~((2ull << e) - 1ull);  // (2 << 63) - 1 wraps to all ones: nothing is left
                if (!t) break;
                unite(par, run_node(lane, a), run_node(lane - 1, run_first(mp, __ffsll((long long)t) - 1)), nullptr);
            }
        }
        __syncwarp();
        tile_flatten(starts, par, lane);
    }
    for (unsigned long long s = starts; s; s &= s - 1) {
        const int a = __ffsll((long long)s) - 1, l = run_node(lane, a);
        if (par[l] == l) par[l] = ~tile_lidx(conn, lane, a);
    }
    __syncwarp();
    if (conn == 8) {
        if (lane & 1)
            for (unsigned long long s = starts; s; s &= s - 1) {
                const int a = __ffsll((long long)s) - 1, p = par[run_node(lane, a)];
                if (p >= 0 && (p >> 5) == lane - 1) atomicMax(&par[p], ~tile_lidx(conn, lane, a));
            }
        __syncwarp();
    }
}

// What the root of a run holds (~ its component's local canonical id, or ~ its label).
__device__ __forceinline__ int root_code(const int* par, int node) {
    const int p = par[node];
    return p < 0 ? p : par[p];
}

// Global canonical id of local canonical id l of the tile at (ty0, tx0).
__device__ __forceinline__ int tile_gid(const Geo& g, int ty0, int tx0, int l) {
    int ry, rx;
    if (g.conn == 8) {
        const int b = l >> 2;
        ry = (b / (kTileW / 2)) * 2 + ((l >> 1) & 1);
        rx = (b % (kTileW / 2)) * 2 + (l & 1);
    } else {
        ry = l / kTileW;
        rx = l % kTileW;
    }
    return g.canon(ty0 + ry, tx0 + rx);
}

// Whether a pixel is foreground. Integer pixels are compared with the threshold's floor (v > t <=> v >
// floor(t), v <= t <=> v <= floor(t)); a NaN threshold has no foreground.
template <typename Px>
struct Foreground {
    double t;
    int ti, invert;
    __device__ Foreground(double thr, int inv) : t(thr), invert(inv) {
        ti = isnan(thr) ? (inv ? -1 : 70000) : (int)fmin(fmax(floor(thr), -1.0), 70000.0);
    }
    __device__ __forceinline__ bool operator()(Px v) const {
        if constexpr (sizeof(Px) <= 2) return invert ? (int)v <= ti : (int)v > ti;
        else return is_fg((double)v, t, invert);
    }
};

// The foreground mask of row ty0 + lane of a tile (0 past the image): one ballot per half-row of 32
// pixels, eight rows' loads in flight.
template <typename Px>
__device__ __forceinline__ unsigned long long tile_mask(const Px* img, const Geo& g, int ty0, int tx0,
                                                        const Foreground<Px>& fg, int lane) {
    unsigned long long m = 0;
    constexpr int kAhead = 8;
    for (int r0 = 0; r0 < kTileH; r0 += kAhead) {
        Px v[2 * kAhead];
#pragma unroll
        for (int u = 0; u < 2 * kAhead; ++u) {
            const int y = min(ty0 + r0 + (u >> 1), g.H - 1), x = min(tx0 + (u & 1) * 32 + lane, g.W - 1);
            v[u] = img[(long long)y * g.W + x];
        }
#pragma unroll
        for (int u = 0; u < kAhead; ++u) {
            const int r = r0 + u;
            const bool in = ty0 + r < g.H;
            const unsigned lo = __ballot_sync(0xffffffffu, in && tx0 + lane < g.W && fg(v[2 * u]));
            const unsigned hi = __ballot_sync(0xffffffffu, in && tx0 + 32 + lane < g.W && fg(v[2 * u + 1]));
            if (lane == r) m = (unsigned long long)lo | ((unsigned long long)hi << 32);
        }
    }
    return m;
}

// tile_mask of a full-width tile of 8- or 16-bit pixels whose rows start on 16 bytes: the whole tile in
// flight as 16-byte loads, each compared in its lane to 16 or 8 bits of its row; the bits change lanes
// through buf (256 bytes).
template <typename Px>
__device__ __forceinline__ unsigned long long tile_mask_wide(const Px* img, const Geo& g, int ty0, int tx0,
                                                             const Foreground<Px>& fg, int* buf, int lane) {
    constexpr int kPer = 16 / (int)sizeof(Px), kLanes = kTileW / kPer, kRows = 32 / kLanes, kLoads = kTileH / kRows;
    const int q = lane / kLanes, c = lane % kLanes;
    uint4 v[kLoads];
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
        const int y = min(ty0 + k * kRows + q, g.H - 1);
        v[k] = __ldg(reinterpret_cast<const uint4*>(img + (long long)y * g.W + tx0) + c);
    }
    const unsigned t = (unsigned)(fg.ti + 1);  // v > ti <=> v >= t
#pragma unroll
    for (int k = 0; k < kLoads; ++k) {
        const unsigned w[4] = {v[k].x, v[k].y, v[k].z, v[k].w};
        unsigned bits = 0;
#pragma unroll
        for (int j = 0; j < kPer; ++j) {
            constexpr int kInWord = 4 / (int)sizeof(Px), kBits = 8 * (int)sizeof(Px);
            const unsigned px = (w[j / kInWord] >> (j % kInWord * kBits)) & ((1u << kBits) - 1u);
            if (px >= t) bits |= 1u << j;
        }
        const int at = (k * kRows + q) * kLanes + c;
        if constexpr (kPer == 16) reinterpret_cast<uint16_t*>(buf)[at] = (uint16_t)bits;
        else reinterpret_cast<uint8_t*>(buf)[at] = (uint8_t)bits;
    }
    __syncwarp();
    const uint2 w = reinterpret_cast<const uint2*>(buf)[lane];
    const unsigned long long m = (unsigned long long)w.x | ((unsigned long long)w.y << 32);
    __syncwarp();  // buf is reused
    return ty0 + lane < g.H ? (fg.invert ? ~m : m) : 0ull;
}

// Binarises 32 x 64 tiles into the foreground bitmap and builds their forests. Writes parents only
// where the border merge reads them: each local root points at itself (and gets its root bit) and
// each foreground pixel on the tile's four edges points at its local root.
//
// Bound: the serial work of a warp's tile (about ten cycles an instruction where a frame gives an SM three
// tiles; on pages enough tiles per SM to hide it, hence the 4 KB a tile).
// The 8192 uint16 page: 259 us with a block per tile and the forest by one of its warps, 191 us with a warp per
// tile and a search per touching pair, now 97 us; a 1024 px frame 13 -> 10 us.
template <typename Px>
__global__ void __launch_bounds__(kCclThreads) k_local_ccl(const Px* img, Geo g, const double* thr_dev,
                                                           double thr_fixed, int invert, int wide, int tiles_x,
                                                           long long tiles, int* parents, unsigned int* roots,
                                                           unsigned int* fgbits) {
    __shared__ __align__(16) int par_all[kCclWarps][kTileNodes];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* par = par_all[warp];
    const long long tile = blockIdx.x * (long long)kCclWarps + warp;
    if (tile >= tiles) return;
    const int tx0 = (int)(tile % tiles_x) * kTileW, ty0 = (int)(tile / tiles_x) * kTileH;
    const Foreground<Px> fg(thr_dev ? *thr_dev : thr_fixed, invert);
    unsigned long long m;
    if constexpr (sizeof(Px) <= 2) {
        if (wide && tx0 + kTileW <= g.W) m = tile_mask_wide(img, g, ty0, tx0, fg, par, lane);
        else m = tile_mask(img, g, ty0, tx0, fg, lane);
    } else {
        m = tile_mask(img, g, ty0, tx0, fg, lane);
    }
    const int y = ty0 + lane;
    if (y < g.H)
        *reinterpret_cast<uint2*>(fgbits + (long long)y * g.words_per_row() + (tx0 >> 5)) =
            make_uint2((unsigned)m, (unsigned)(m >> 32));
    if (!__any_sync(0xffffffffu, m != 0ull)) return;
    tile_forest(m, g.conn, par, lane);
    for (unsigned long long s = m & ~(m << 1); s; s &= s - 1) {
        const int code = par[run_node(lane, __ffsll((long long)s) - 1)];
        if (code < 0) {
            const int gid = tile_gid(g, ty0, tx0, ~code);
            parents[gid] = gid;
            atomicOr(&roots[gid >> 5], 1u << (gid & 31));
        }
    }
    // Left and right edge pixels of this row.
    if (m & 1ull) parents[g.canon(y, tx0)] = tile_gid(g, ty0, tx0, ~root_code(par, run_node(lane, 0)));
    if (m >> 63)
        parents[g.canon(y, tx0 + 63)] = tile_gid(g, ty0, tx0, ~root_code(par, run_node(lane, run_first(m, 63))));
    // Top and bottom rows, lanes over the 64 columns.
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int r = e == 0 ? 0 : kTileH - 1;
        const unsigned long long row = __shfl_sync(0xffffffffu, m, r);
        for (int x = lane; x < kTileW; x += 32)
            if ((row >> x) & 1ull)
                parents[g.canon(ty0 + r, tx0 + x)] =
                    tile_gid(g, ty0, tx0, ~root_code(par, run_node(r, run_first(row, x))));
    }
}

// Unions across tile borders. One thread per border pixel of a tile: top row (neighbours above),
// left column (neighbours to the left), right column (the up-right neighbour in the next tile).
__global__ void k_border_merge(Geo g, int* parents, unsigned int* roots, const unsigned int* fgbits, int tiles_x,
                               int tiles_y) {
    const int per_tile = kTileW + 2 * kTileH;
    const long long total = (long long)tiles_x * tiles_y * per_tile;
    for (long long k = blockIdx.x * (long long)blockDim.x + threadIdx.x; k < total;
         k += (long long)gridDim.x * blockDim.x) {
        int tile, e;
        divmod_idx(k, per_tile, &tile, &e);
        const int tx0 = (tile % tiles_x) * kTileW, ty0 = (tile / tiles_x) * kTileH;
        int y, x;
        if (e < kTileW) { y = ty0; x = tx0 + e; }
        else if (e < kTileW + kTileH) { y = ty0 + (e - kTileW); x = tx0; }
        else { y = ty0 + (e - kTileW - kTileH); x = tx0 + kTileW - 1; }
        if (y >= g.H || x >= g.W) continue;
        if (!g.fg(fgbits, y, x)) continue;
        const int me = g.canon(y, x);
        auto link = [&](int yy, int xx) {
            if (yy < 0 || xx < 0 || xx >= g.W) return;
            // Only neighbours in another tile.
            if (yy >= ty0 && xx >= tx0 && xx < tx0 + kTileW) return;
            if (!g.fg(fgbits, yy, xx)) return;
            unite(parents, me, g.canon(yy, xx), roots);
        };
        if (e < kTileW) {  // top row: (y-1, x) and, for 8-connectivity, (y-1, x-1), (y-1, x+1)
            link(y - 1, x);
            if (g.conn == 8) { link(y - 1, x - 1); link(y - 1, x + 1); }
        } else if (e < kTileW + kTileH) {  // left column: (y, x-1) and (y-1, x-1)
            link(y, x - 1);
            if (g.conn == 8) link(y - 1, x - 1);
        } else {  // right column: (y-1, x+1) lies in the tile to the right (or up-right)
            if (g.conn == 8) link(y - 1, x + 1);
        }
    }
}

// ---------------------------------------------------------------------------- prefix of popcounts

__global__ void k_popc_block_sums(const unsigned int* words, long long n, int per_block,
                                  int* block_sums) {
    __shared__ int s[32];
    const long long start = (long long)blockIdx.x * per_block;
    int acc = 0;
    for (int i = threadIdx.x; i < per_block; i += blockDim.x) {
        const long long w = start + i;
        if (w < n) acc += __popc(words[w]);
    }
    acc = warp_sum_i(acc);
    if ((threadIdx.x & 31) == 0) s[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x < 32) {
        int v = threadIdx.x < (blockDim.x >> 5) ? s[threadIdx.x] : 0;
        v = warp_sum_i(v);
        if (threadIdx.x == 0) block_sums[blockIdx.x] = v;
    }
}

// Exclusive scan of block_sums in place by one block; writes the total to *total.
__global__ void k_scan_small(int* block_sums, int n, int* total) {
    __shared__ int s[1024];
    const int per = (n + blockDim.x - 1) / blockDim.x;
    const int b0 = threadIdx.x * per;
    int acc = 0;
    for (int i = 0; i < per; ++i)
        if (b0 + i < n) acc += block_sums[b0 + i];
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 1; o < (int)blockDim.x; o <<= 1) {
        const int v = threadIdx.x >= (unsigned)o ? s[threadIdx.x - o] : 0;
        __syncthreads();
        s[threadIdx.x] += v;
        __syncthreads();
    }
    int run = s[threadIdx.x] - acc;  // exclusive prefix of this thread's chunk
    for (int i = 0; i < per; ++i)
        if (b0 + i < n) {
            const int v = block_sums[b0 + i];
            block_sums[b0 + i] = run;
            run += v;
        }
    if (threadIdx.x == blockDim.x - 1) *total = s[threadIdx.x];
}

// prefix[w] = number of set bits in words[0..w).
__global__ void k_popc_prefix(const unsigned int* words, long long n, int per_block,
                              const int* block_offsets, int* prefix) {
    __shared__ int s[1024];
    const long long start = (long long)blockIdx.x * per_block;
    const int per = per_block / blockDim.x;  // words per thread (per_block is a multiple)
    const long long w0 = start + (long long)threadIdx.x * per;
    int acc = 0;
    for (int i = 0; i < per; ++i)
        if (w0 + i < n) acc += __popc(words[w0 + i]);
    s[threadIdx.x] = acc;
    __syncthreads();
    for (int o = 1; o < (int)blockDim.x; o <<= 1) {
        const int v = threadIdx.x >= (unsigned)o ? s[threadIdx.x - o] : 0;
        __syncthreads();
        s[threadIdx.x] += v;
        __syncthreads();
    }
    int run = block_offsets[blockIdx.x] + s[threadIdx.x] - acc;
    for (int i = 0; i < per; ++i)
        if (w0 + i < n) {
            prefix[w0 + i] = run;
            run += __popc(words[w0 + i]);
        }
}

// The three kernels above in one launch, for bitmaps of at most kScanDirect blocks: every block counts the
// words before its own itself (up to 512 KB from L2) instead of waiting for the others' sums. At 1024 x 1024 4.6
// instead of 11 us and two launches less; the counting grows with the square of the size: at 2048 x 2048 (32 blocks)
// 8.4 against 10.7 us for the three kernels at 2100 x 2100.
constexpr int kScanDirect = 33;
__global__ void __launch_bounds__(1024) k_popc_prefix_direct(const unsigned int* words, long long n, int* prefix,
                                                             int* total) {
    constexpr int kPer = kScanPerBlock / 1024;
    __shared__ int s_before[32], s_own[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const long long start = (long long)blockIdx.x * kScanPerBlock;
    int before = 0;
    const uint4* w4 = reinterpret_cast<const uint4*>(words);
#pragma unroll 8
    for (int i = t; i < (int)(start / 4); i += 1024) {
        const uint4 w = w4[i];
        before += __popc(w.x) + __popc(w.y) + __popc(w.z) + __popc(w.w);
    }
    unsigned w[kPer];
    int own = 0;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const long long i = start + kPer * t + j;
        w[j] = i < n ? words[i] : 0u;
        own += __popc(w[j]);
    }
    before = warp_sum_i(before);
    int incl = own;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    if (lane == 31) {
        s_before[warp] = before;
        s_own[warp] = incl;
    }
    __syncthreads();
    const int b = warp_sum_i(s_before[lane]), mine = s_own[lane];
    int run = b + warp_sum_i(lane < warp ? mine : 0) + incl - own;
#pragma unroll
    for (int j = 0; j < kPer; ++j) {
        const long long i = start + kPer * t + j;
        if (i < n) prefix[i] = run;
        run += __popc(w[j]);
    }
    if (blockIdx.x == gridDim.x - 1 && t == 1023) *total = run;
}

// --------------------------------------------------------------------------------------- finish

__global__ void k_stats_init(int* stats, unsigned long long* sums, int k1) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k1; i += gridDim.x * blockDim.x) {
        stats[i * 5 + 0] = 0x7fffffff;  // min x
        stats[i * 5 + 1] = 0x7fffffff;  // min y
        stats[i * 5 + 2] = -1;          // max x (turned into width)
        stats[i * 5 + 3] = -1;          // max y (turned into height)
        stats[i * 5 + 4] = 0;           // area
        sums[2 * i] = 0;
        sums[2 * i + 1] = 0;
    }
}

// Final labels and stats of 32 x 64 tiles. A tile's forest is rebuilt from the bitmap; each local root
// follows the merged parents to its global root once, whose label is the rank of that root among the
// roots (popcount prefix) + 1; every pixel then takes the label of its run.
//
// Bound: instructions and atomics. The background's statistics come from the row masks' complements and are
// kept by each lane over all its tiles (one set of atomics a block, not one a tile to the same seven words).
// Labels are written four to a lane. Measured on the 8192 page (116k holes): a block per tile, with run heads
// found per pixel, 523 us; a warp per tile, runs joined by label with masked reductions (one group of lanes after
// another), 223 us; joined along the lanes, 167 us. On a 1024 px frame 24 and 16 us.
constexpr int kFinishBlocks = 10;  // per SM
__global__ void __launch_bounds__(kCclThreads, kFinishBlocks) k_finish(Geo g, const int* parents, const unsigned int* roots,
                                                        const int* prefix, const unsigned int* fgbits, int tiles_x,
                                                        long long tiles, int* labels, int* stats,
                                                        unsigned long long* sums, int k1, const int* count) {
    if (count && *count >= k1) return;  // more components than the tables hold: the caller starts again
    __shared__ int par_all[kCclWarps][kTileNodes];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int* par = par_all[warp];
    int bx0 = 0x7fffffff, by0 = 0x7fffffff, bx1 = -1, by1 = -1;  // this lane's rows' background
    long long barea = 0, bsx = 0, bsy = 0;
    const bool vec = g.W % 4 == 0 && (reinterpret_cast<uintptr_t>(labels) & 15) == 0;
    for (long long tile = blockIdx.x * (long long)kCclWarps + warp; tile < tiles;
         tile += (long long)gridDim.x * kCclWarps) {
        const int tx0 = (int)(tile % tiles_x) * kTileW, ty0 = (int)(tile / tiles_x) * kTileH;
        const int y = ty0 + lane, cols = min(kTileW, g.W - tx0);
        unsigned long long m = 0;
        if (y < g.H) {
            const uint2 w = *reinterpret_cast<const uint2*>(fgbits + (long long)y * g.words_per_row() + (tx0 >> 5));
            m = (unsigned long long)w.x | ((unsigned long long)w.y << 32);
            const unsigned long long bg = ~m & (cols == 64 ? ~0ull : (1ull << cols) - 1ull);
            if (bg) {
                const unsigned lo = (unsigned)bg, hi = (unsigned)(bg >> 32);
                const int n = __popcll(bg);
                int pos = 32 * __popc(hi);
                constexpr unsigned M[5] = {0xaaaaaaaau, 0xccccccccu, 0xf0f0f0f0u, 0xff00ff00u, 0xffff0000u};
#pragma unroll
                for (int q = 0; q < 5; ++q) pos += (__popc(lo & M[q]) + __popc(hi & M[q])) << q;
                barea += n;
                bsx += (long long)tx0 * n + pos;
                bsy += (long long)y * n;
                bx0 = min(bx0, tx0 + __ffsll((long long)bg) - 1);
                bx1 = max(bx1, tx0 + 63 - __clzll((long long)bg));
                by0 = min(by0, y);
                by1 = max(by1, y);
            }
        }
        const bool any = __any_sync(0xffffffffu, m != 0ull);
        if (any) {
            tile_forest(m, g.conn, par, lane);
            // Roots get their label (its complement, in place of the canonical id's), four of a lane's at a time...
            unsigned long long s = m & ~(m << 1);
            while (__any_sync(0xffffffffu, s != 0ull)) {
                constexpr int kRoots = 4;
                int at[kRoots], p[kRoots], q[kRoots], n = 0;
#pragma unroll
                for (int u = 0; u < kRoots; ++u) at[u] = -1;
                for (; s && n < kRoots; s &= s - 1) {
                    const int l = run_node(lane, __ffsll((long long)s) - 1);
                    if (par[l] >= 0) continue;
#pragma unroll
                    for (int u = 0; u < kRoots; ++u)
                        if (u == n) at[u] = l;
                    ++n;
                }
#pragma unroll
                for (int u = 0; u < kRoots; ++u) {
                    p[u] = at[u] >= 0 ? tile_gid(g, ty0, tx0, ~par[at[u]]) : 0;
                    q[u] = at[u] >= 0 ? parents[p[u]] : 0;
                }
                bool up;
                do {
                    up = false;
                    int r[kRoots];
#pragma unroll
                    for (int u = 0; u < kRoots; ++u) r[u] = q[u] != p[u] ? parents[q[u]] : q[u];
#pragma unroll
                    for (int u = 0; u < kRoots; ++u) {
                        up |= r[u] != q[u];
                        p[u] = q[u];
                        q[u] = r[u];
                    }
                } while (up);
#pragma unroll
                for (int u = 0; u < kRoots; ++u)
                    if (at[u] >= 0)
                        par[at[u]] = ~(prefix[p[u] >> 5] + __popc(roots[p[u] >> 5] & ((1u << (p[u] & 31)) - 1u)) + 1);
            }
            __syncwarp();
            // ... the other runs take it from their root, and every run adds its statistics: the i-th runs of all
            // rows at a time, those of consecutive rows with one label joined.
            s = m & ~(m << 1);
            while (__any_sync(0xffffffffu, s != 0ull)) {
                int lab = 0;
                unsigned long long cols_of = 0, acc = 0;  // columns covered; area | sum of x << 16 | sum of y << 40
                if (s) {
                    const int a = __ffsll((long long)s) - 1, b = run_last(m, a);
                    const int l = run_node(lane, a), code = root_code(par, l);
                    par[l] = code;
                    lab = ~code;
                    const unsigned len = b - a + 1;
                    cols_of = ((2ull << b) - 1ull) & ~((1ull << a) - 1ull);
                    acc = len | ((unsigned long long)((a + b) * len / 2) << 16) | ((unsigned long long)(lane * len) << 40);
                    s &= s - 1;
                }
                const int prev = __shfl_up_sync(0xffffffffu, lab, 1);
                const bool head = lane == 0 || prev != lab;
                const unsigned later = __ballot_sync(0xffffffffu, head) & ~((2u << lane) - 1u);
                const int end = later ? __ffs(later) - 2 : 31;  // last row of this group
                for (int d = 1; __any_sync(0xffffffffu, lab > 0 && lane + d <= end); d <<= 1) {
                    const unsigned long long oc = __shfl_down_sync(0xffffffffu, cols_of, d);
                    const unsigned long long oa = __shfl_down_sync(0xffffffffu, acc, d);
                    if (lane + d <= end) {
                        cols_of |= oc;
                        acc += oa;
                    }
                }
                // (labels beyond the component count cannot occur, or are not counted in a capped table)
                if (head && lab > 0 && lab < k1) {
                    const int n = (int)(acc & 0xffff), px = (int)((acc >> 16) & 0xffffff), py = (int)(acc >> 40);
                    int* st = stats + (long long)lab * 5;
                    atomicMin(&st[0], tx0 + __ffsll((long long)cols_of) - 1);
                    atomicMin(&st[1], ty0 + lane);
                    atomicMax(&st[2], tx0 + 63 - __clzll((long long)cols_of));
                    atomicMax(&st[3], ty0 + end);
                    atomicAdd(&st[4], n);
                    atomicAdd(&sums[2LL * lab], (unsigned long long)((long long)tx0 * n + px));
                    atomicAdd(&sums[2LL * lab + 1], (unsigned long long)((long long)ty0 * n + py));
                }
            }
            __syncwarp();
        }
        // Labels: two rows of sixteen quads at a time. A quad has a run at its first pixel (which
        // may have begun earlier), runs that begin inside, or both.
        const int xq = (lane & 15) * 4;
        int* out = labels + (long long)(ty0 + (lane >> 4)) * g.W + (tx0 + xq);
        for (int r0 = 0; r0 < kTileH && ty0 + r0 < g.H; r0 += 2, out += 2LL * g.W) {
            const int r = r0 + (lane >> 4);
            const unsigned long long row = __shfl_sync(0xffffffffu, m, r);
            const unsigned nib = (unsigned)(row >> xq) & 15u;
            int4 lab = make_int4(0, 0, 0, 0);
            if (nib) {
                int first = 0, later = 0;
                if (nib & 1u) first = ~par[run_node(r, run_first(row, xq))];
                const unsigned begin = nib & ~(nib << 1) & 14u;        // runs that begin inside the quad
                if (begin) later = ~par[run_node(r, xq + __ffs(begin) - 1)];
                const unsigned old = nib & (nib ^ (nib + 1u));         // pixels of the run at pixel 0
                lab.x = nib & 1u ? first : 0;
                lab.y = nib & 2u ? (old & 2u ? first : later) : 0;
                lab.z = nib & 4u ? (old & 4u ? first : later) : 0;
                lab.w = nib & 8u ? (old & 8u ? first : later) : 0;
                if (nib == 10u) lab.w = ~par[run_node(r, xq + 3)];     // .x.x: two begin inside
            }
            if (ty0 + r < g.H && xq < cols) {
                if (vec) {  // every quad is whole and on 16 bytes
                    *reinterpret_cast<int4*>(out) = lab;
                } else {
                    out[0] = lab.x;
                    if (xq + 1 < cols) out[1] = lab.y;
                    if (xq + 2 < cols) out[2] = lab.z;
                    if (xq + 3 < cols) out[3] = lab.w;
                }
            }
        }
        __syncwarp();  // the next tile rewrites par
    }
    // The block's background.
    bx0 = __reduce_min_sync(0xffffffffu, bx0);
    by0 = __reduce_min_sync(0xffffffffu, by0);
    bx1 = __reduce_max_sync(0xffffffffu, bx1);
    by1 = __reduce_max_sync(0xffffffffu, by1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        barea += __shfl_xor_sync(0xffffffffu, barea, o);
        bsx += __shfl_xor_sync(0xffffffffu, bsx, o);
        bsy += __shfl_xor_sync(0xffffffffu, bsy, o);
    }
    __shared__ int s_box[4];
    __shared__ unsigned long long s_sum[3];
    if (threadIdx.x == 0) {
        s_box[0] = s_box[1] = 0x7fffffff;
        s_box[2] = s_box[3] = -1;
        s_sum[0] = s_sum[1] = s_sum[2] = 0ull;
    }
    __syncthreads();
    if (lane == 0 && barea != 0) {
        atomicMin(&s_box[0], bx0);
        atomicMin(&s_box[1], by0);
        atomicMax(&s_box[2], bx1);
        atomicMax(&s_box[3], by1);
        atomicAdd(&s_sum[0], (unsigned long long)barea);
        atomicAdd(&s_sum[1], (unsigned long long)bsx);
        atomicAdd(&s_sum[2], (unsigned long long)bsy);
    }
    __syncthreads();
    if (threadIdx.x < 7 && s_sum[0] != 0ull) {
        const int i = threadIdx.x;
        if (i < 2) atomicMin(&stats[i], s_box[i]);
        else if (i < 4) atomicMax(&stats[i], s_box[i]);
        else if (i == 4) atomicAdd(&stats[4], (int)s_sum[0]);
        else atomicAdd(&sums[i - 5], s_sum[i - 4]);
    }
}

// bbox max -> width/height; centroid = exact integer sum / area (as OpenCV).
__global__ void k_stats_final(int* stats, const unsigned long long* sums, double* centroids, int k1) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < k1; i += gridDim.x * blockDim.x) {
        int* st = stats + (long long)i * 5;
        const int area = st[4];
        const unsigned long long sx = sums[2 * i], sy = sums[2 * i + 1];
        if (area > 0) {
            st[2] = st[2] - st[0] + 1;
            st[3] = st[3] - st[1] + 1;
            centroids[2 * i] = (double)sx / (double)area;
            centroids[2 * i + 1] = (double)sy / (double)area;
        } else {
            st[0] = st[1] = st[2] = st[3] = 0;
            centroids[2 * i] = dnan();
            centroids[2 * i + 1] = dnan();
        }
    }
}

struct CclLayout {
    long long canon_n;   // entries of the canonical parents array
    long long words;     // root bitmap words
    int scan_blocks;     // blocks of the popcount prefix
    int* parents;
    unsigned int* roots;
    int* prefix;
    int* block_sums;
    int* scratch_count;
    unsigned int* fgbits;  // foreground bitmap, H x words-per-row
};

CclLayout ccl_layout(void* ws, int H, int W, size_t* bytes) {
    CclLayout L;
    const long long Hb = (H + 1) / 2, Wb = (W + 1) / 2;
    L.canon_n = Hb * Wb * 4;  // >= H*W; also covers raster order for 4-connectivity
    L.words = (L.canon_n + 31) / 32;
    L.scan_blocks = (int)((L.words + kScanPerBlock - 1) / kScanPerBlock);
    Arena a(ws);
    L.parents = a.take<int>(L.canon_n);
    L.roots = a.take<unsigned int>(L.words);
    L.prefix = a.take<int>(L.words);
    L.block_sums = a.take<int>(L.scan_blocks + 1);
    L.scratch_count = a.take<int>(4);
    L.fgbits = a.take<unsigned int>((long long)H * ((W + 63) / 64 * 2));
    if (bytes) *bytes = a.used;
    return L;
}

// ---------------------------------------------------------------------- allocation-free Otsu

// Scratch of spx_otsu_static: the same pieces as the Otsu workspace (histogram, value range), in one
// file-scope device array. Every GPU that loads this library holds it (0.25 MiB) until the process exits.
constexpr size_t kOtsuStaticBytes = 65536 * sizeof(unsigned int) + 2 * 256;
__device__ __align__(256) unsigned char g_otsu_static[kOtsuStaticBytes];

// Device address of g_otsu_static for the current device, looked up once per device and kept for the
// life of the process: a cudaDeviceReset (which unloads this module's device copy) invalidates it,
// so the library must not be used across one.
int otsu_static_scratch(void** out) {
    static std::mutex mu;
    static void* cache[128] = {};
    int dev = 0;
    SPX_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 128) {
        set_error("device index %d out of range", dev);
        return SPX_ERR_ARGUMENT;
    }
    std::lock_guard<std::mutex> lock(mu);
    if (!cache[dev]) {
        void* p = nullptr;
        const cudaError_t e = cudaGetSymbolAddress(&p, g_otsu_static);
        if (e != cudaSuccess || !p) {
            set_error("cudaGetSymbolAddress(g_otsu_static) failed: %s", cudaGetErrorString(e));
            return SPX_ERR_CUDA;
        }
        cache[dev] = p;
    }
    *out = cache[dev];
    return SPX_OK;
}


// ------------------------------------------------------------------------------ morphology

// bw = 255 where the pixel is foreground (img > t, or img <= t with invert), else 0: the 0/255
// image of cv2.threshold(THRESH_BINARY[_INV]).
__global__ void k_binarize(const void* img, int dtype, long long n, const double* t_dev, double t_fixed, int invert,
                           uint8_t* bw) {
    const double t = t_dev ? *t_dev : t_fixed;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        bw[i] = is_fg(load_px(img, dtype, i), t, invert) ? 255 : 0;
}

// One erosion (dilate = 0: minimum) or dilation (maximum) of a 0/255 image with the 3x3 cross
// (cv2.getStructuringElement(MORPH_ELLIPSE, (3, 3))); neighbours outside the image are ignored, as
// OpenCV's default morphology border does.
__global__ void k_morph_cross(const uint8_t* in, int H, int W, int dilate, uint8_t* out) {
    const long long total = (long long)H * W;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        int y, x;
        divmod_idx(i, W, &y, &x);
        unsigned v = in[i];
        if (dilate) {
            if (y > 0) v = max(v, (unsigned)in[i - W]);
            if (y < H - 1) v = max(v, (unsigned)in[i + W]);
            if (x > 0) v = max(v, (unsigned)in[i - 1]);
            if (x < W - 1) v = max(v, (unsigned)in[i + 1]);
        } else {
            if (y > 0) v = min(v, (unsigned)in[i - W]);
            if (y < H - 1) v = min(v, (unsigned)in[i + W]);
            if (x > 0) v = min(v, (unsigned)in[i - 1]);
            if (x < W - 1) v = min(v, (unsigned)in[i + 1]);
        }
        out[i] = (uint8_t)v;
    }
}

}  // namespace
}  // namespace spx

using namespace spx;

extern "C" {

const char* spx_last_error(void) { return spx::g_error; }

int spx_version(void) { return 1; }

int spx_tune_set(const char* knob, int value) {
    SPX_REQUIRE(knob, "null knob name");
    Tuning& t = tuning();
    if (!strcmp(knob, "fit_warps")) {
        SPX_REQUIRE(value == 2 || value == 4 || value == 8, "fit_warps must be 2, 4 or 8");
        t.fit_warps = value;
    } else if (!strcmp(knob, "fit_blocks_per_sm")) {
        SPX_REQUIRE(value >= 2 && value <= 32, "fit_blocks_per_sm must be in [2, 32]");
        t.fit_blocks_per_sm = value;
    } else if (!strcmp(knob, "render_tile")) {
        SPX_REQUIRE(value == 16 || value == 32 || value == 64, "render_tile must be 16, 32 or 64");
        t.render_tile = value;
    } else if (!strcmp(knob, "radial_rays")) {
        SPX_REQUIRE(value == 0 || value == 2, "radial_rays must be 0 or 2");
        t.radial_rays = value;
    } else {
        set_error("unknown tuning knob '%s'", knob);
        return SPX_ERR_ARGUMENT;
    }
    return SPX_OK;
}

int spx_tune_get(const char* knob, int* value) {
    SPX_REQUIRE(knob && value, "null pointer");
    const Tuning& t = tuning();
    if (!strcmp(knob, "fit_warps")) *value = t.fit_warps;
    else if (!strcmp(knob, "fit_blocks_per_sm")) *value = t.fit_blocks_per_sm;
    else if (!strcmp(knob, "render_tile")) *value = t.render_tile;
    else if (!strcmp(knob, "radial_rays")) *value = t.radial_rays;
    else {
        set_error("unknown tuning knob '%s'", knob);
        return SPX_ERR_ARGUMENT;
    }
    return SPX_OK;
}

unsigned long long spx_launch_count(void) { return __atomic_load_n(&spx::g_launches, __ATOMIC_RELAXED); }

}  // extern "C"

namespace spx {
namespace {
// Eight independent FP64 FMA chains per thread (no dependency between them, so the FP64 pipe, not
// the FMA latency, bounds the rate); the sums go to `sink` so nothing is optimised away.
__global__ void __launch_bounds__(256) k_fp64_fma_rate(int iters, double* sink) {
    double a[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) a[q] = 1.0 + 1e-3 * (threadIdx.x + q);
    const double b = 0.9999999, c = 1e-7;
    for (int i = 0; i < iters; ++i)
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = __fma_rn(a[q], b, c);
    double t = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) t += a[q];
    sink[blockIdx.x * blockDim.x + threadIdx.x] = t;
}
}  // namespace
}  // namespace spx

extern "C" {

int spx_fp64_fma_rate(int blocks, int iters, double* sink, double* flops, void* stream) {
    SPX_REQUIRE(blocks >= 1 && iters >= 1 && sink && flops, "bad arguments");
    k_fp64_fma_rate<<<blocks, 256, 0, static_cast<cudaStream_t>(stream)>>>(iters, sink);
    *flops = 2.0 * 8.0 * 256.0 * (double)blocks * (double)iters;
    return check_launch("k_fp64_fma_rate");
}

int spx_device_info(int* sm_count, int* is_sm100) {
    int dev = 0;
    SPX_CUDA(cudaGetDevice(&dev));
    cudaDeviceProp prop;
    SPX_CUDA(cudaGetDeviceProperties(&prop, dev));
    if (sm_count) *sm_count = prop.multiProcessorCount;
    if (is_sm100) *is_sm100 = prop.major == 10 ? 1 : 0;
    return SPX_OK;
}

size_t spx_otsu_workspace_bytes(int dtype) {
    (void)dtype;
    Arena a(nullptr);
    a.take<unsigned int>(65536);
    a.take<unsigned int>(2);
    return a.used;
}

static int launch_minmax(const void* img, int dtype, int height, int width, int step, long long n, unsigned int* range,
                         cudaStream_t s) {
    if (step == 1 && dtype == SPX_U16 && (reinterpret_cast<uintptr_t>(img) % 16) == 0) {
        k_minmax_dense<<<grid_for(n / 8 + 1, 256, 148 * 8), 256, 0, s>>>(static_cast<const uint16_t*>(img), n, range);
        return check_launch("k_minmax_dense");
    }
    k_minmax<<<grid_for(n, 256, 148 * 8), 256, 0, s>>>(img, dtype, height, width, step, range);
    return check_launch("k_minmax");
}

int spx_otsu(const void* img, int dtype, int height, int width, int step, double* threshold,
             void* workspace, size_t workspace_bytes, void* stream) {
    SPX_REQUIRE(dtype == SPX_U8 || dtype == SPX_U16, "Otsu thresholding needs a uint8 or uint16 image");
    SPX_REQUIRE(height > 0 && width > 0 && step >= 1, "bad image size or step");
    SPX_REQUIRE(img && threshold && workspace, "null pointer");
    SPX_REQUIRE(workspace_bytes >= spx_otsu_workspace_bytes(dtype), "workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Arena a(workspace);
    unsigned int* hist = a.take<unsigned int>(65536);
    unsigned int* range = a.take<unsigned int>(2);
    const int nbins = dtype == SPX_U8 ? 256 : 65536;
    k_hist_init<<<64, 256, 0, s>>>(hist, 65536, range, 0xffffffffu, 0u);
    if (int e = check_launch("k_hist_init")) return e;
    const int hs = (int)(((long long)height + step - 1) / step), ws = (int)(((long long)width + step - 1) / step);
    const long long n = (long long)hs * ws;
    if (int e = launch_minmax(img, dtype, height, width, step, n, range, s)) return e;
    const size_t smem = kHistSmemBins * sizeof(unsigned int);
    SPX_CUDA(cudaFuncSetAttribute(k_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int dense = step == 1 && dtype == SPX_U16 && (reinterpret_cast<uintptr_t>(img) % 16) == 0;
    k_histogram<<<grid_for(n / 8 + 1, 512, 148 * 3), 512, smem, s>>>(img, dtype, height, width, step,
                                                                     dense, range, hist);
    if (int e = check_launch("k_histogram")) return e;
    k_otsu_scan<<<1, 1024, 0, s>>>(hist, nbins, range, n, threshold);
    return check_launch("k_otsu_scan");
}

int spx_histogram(const void* img, int dtype, int height, int width, int step, unsigned int* hist,
                  unsigned int* range, void* stream) {
    SPX_REQUIRE(dtype == SPX_U8 || dtype == SPX_U16, "histograms need a uint8 or uint16 image");
    SPX_REQUIRE(height > 0 && width > 0 && step >= 1, "bad image size or step");
    SPX_REQUIRE(img && hist && range, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_hist_init<<<64, 256, 0, s>>>(hist, 65536, range, 0xffffffffu, 0u);
    if (int e = check_launch("k_hist_init")) return e;
    const int hs = (int)(((long long)height + step - 1) / step), ws = (int)(((long long)width + step - 1) / step);
    const long long n = (long long)hs * ws;
    if (int e = launch_minmax(img, dtype, height, width, step, n, range, s)) return e;
    const size_t smem = kHistSmemBins * sizeof(unsigned int);
    SPX_CUDA(cudaFuncSetAttribute(k_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int dense = step == 1 && dtype == SPX_U16 && (reinterpret_cast<uintptr_t>(img) % 16) == 0;
    k_histogram<<<grid_for(n / 8 + 1, 512, 148 * 3), 512, smem, s>>>(img, dtype, height, width, step, dense, range,
                                                                     hist);
    return check_launch("k_histogram");
}

int spx_otsu_from_histogram(const unsigned int* hist, int dtype, const unsigned int* range, long long total,
                            double* threshold, void* workspace, size_t workspace_bytes, void* stream) {
    SPX_REQUIRE(dtype == SPX_U8 || dtype == SPX_U16, "Otsu thresholding needs a uint8 or uint16 histogram");
    SPX_REQUIRE(total > 0, "empty histogram");
    SPX_REQUIRE(hist && range && threshold && workspace, "null pointer");
    SPX_REQUIRE(workspace_bytes >= spx_otsu_workspace_bytes(dtype), "workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_otsu_scan<<<1, 1024, 0, s>>>(hist, dtype == SPX_U8 ? 256 : 65536, range, total, threshold);
    return check_launch("k_otsu_scan");
}

int spx_otsu_static(const void* img, int dtype, int height, int width, int step, double* threshold, void* stream) {
    SPX_REQUIRE(dtype == SPX_U8 || dtype == SPX_U16, "Otsu thresholding needs a uint8 or uint16 image");
    SPX_REQUIRE(height > 0 && width > 0 && step >= 1, "bad image size or step");
    const long long hs = ((long long)height + step - 1) / step, ws = ((long long)width + step - 1) / step;
    SPX_REQUIRE(hs * ws <= 0xffffffffLL,
                "spx_otsu_static: %lld sampled pixels exceed the maximum of 4294967295 (32-bit histogram counts)",
                hs * ws);
    SPX_REQUIRE(img && threshold, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    void* scratch = nullptr;
    if (int e = otsu_static_scratch(&scratch)) return e;
    Arena a(scratch);
    unsigned int* hist = a.take<unsigned int>(65536);
    unsigned int* range = a.take<unsigned int>(2);
    SPX_REQUIRE(a.used <= kOtsuStaticBytes, "static Otsu scratch too small");
    const int nbins = dtype == SPX_U8 ? 256 : 65536;
    const long long n = hs * ws;
    // The array keeps the previous call's contents: clear the histogram and reset the range first.
    k_hist_init<<<64, 256, 0, s>>>(hist, 65536, range, 0xffffffffu, 0u);
    if (int e = check_launch("k_hist_init")) return e;
    if (int e = launch_minmax(img, dtype, height, width, step, n, range, s)) return e;
    const size_t smem = kHistSmemBins * sizeof(unsigned int);
    SPX_CUDA(cudaFuncSetAttribute(k_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int dense = step == 1 && dtype == SPX_U16 && (reinterpret_cast<uintptr_t>(img) % 16) == 0;
    k_histogram<<<grid_for(n / 8 + 1, 512, 148 * 3), 512, smem, s>>>(img, dtype, height, width, step, dense, range,
                                                                     hist);
    if (int e = check_launch("k_histogram")) return e;
    k_otsu_scan<<<1, 1024, 0, s>>>(hist, nbins, range, n, threshold);
    return check_launch("k_otsu_scan");
}

int spx_triangle(const void* img, int dtype, int height, int width, double* threshold,
                 void* workspace, size_t workspace_bytes, void* stream) {
    SPX_REQUIRE(dtype == SPX_U8, "the triangle threshold needs a uint8 image");
    SPX_REQUIRE(height > 0 && width > 0, "bad image size");
    SPX_REQUIRE(img && threshold && workspace, "null pointer");
    SPX_REQUIRE(workspace_bytes >= spx_otsu_workspace_bytes(dtype), "workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    Arena a(workspace);
    unsigned int* hist = a.take<unsigned int>(65536);
    unsigned int* range = a.take<unsigned int>(2);
    k_hist_init<<<1, 256, 0, s>>>(hist, 256, range, 0u, 255u);
    if (int e = check_launch("k_hist_init")) return e;
    const long long n = (long long)height * width;
    const size_t smem = kHistSmemBins * sizeof(unsigned int);
    SPX_CUDA(cudaFuncSetAttribute(k_histogram, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    k_histogram<<<grid_for(n, 512, 148 * 3), 512, smem, s>>>(img, dtype, height, width, 1, 0, range, hist);
    if (int e = check_launch("k_histogram")) return e;
    k_triangle_scan<<<1, 256, 0, s>>>(hist, threshold);
    return check_launch("k_triangle_scan");
}

size_t spx_ccl_workspace_bytes(int height, int width) {
    size_t b = 0;
    ccl_layout(nullptr, height, width, &b);
    return b;
}

int spx_binarize(const void* img, int dtype, int height, int width, const double* threshold_dev,
                 double fixed_threshold, int invert, uint8_t* out, void* stream) {
    SPX_REQUIRE(height > 0 && width > 0 && dtype >= SPX_U8 && dtype <= SPX_F64, "bad arguments");
    SPX_REQUIRE(img && out, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long long n = (long long)height * width;
    k_binarize<<<grid_for(n, 256), 256, 0, s>>>(img, dtype, n, threshold_dev, fixed_threshold, invert, out);
    return check_launch("k_binarize");
}

int spx_morphology(uint8_t* bw, int height, int width, int open_iterations, int close_iterations, uint8_t* tmp,
                   void* stream) {
    SPX_REQUIRE(height > 0 && width > 0 && open_iterations >= 0 && close_iterations >= 0, "bad arguments");
    SPX_REQUIRE(bw && tmp && bw != tmp, "null or aliased pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const long long n = (long long)height * width;
    // MORPH_OPEN: erode then dilate, `open` times each; MORPH_CLOSE: dilate then erode. The number
    // of passes is even, so the result ends in bw.
    uint8_t* cur = bw;
    uint8_t* nxt = tmp;
    auto pass = [&](int dilate, int times) -> int {
        for (int k = 0; k < times; ++k) {
            k_morph_cross<<<grid_for(n, 256), 256, 0, s>>>(cur, height, width, dilate, nxt);
            if (int e = check_launch("k_morph_cross")) return e;
            uint8_t* t = cur;
            cur = nxt;
            nxt = t;
        }
        return SPX_OK;
    };
    if (int e = pass(0, open_iterations)) return e;
    if (int e = pass(1, open_iterations)) return e;
    if (int e = pass(1, close_iterations)) return e;
    return pass(0, close_iterations);
}

int spx_ccl_label(const void* img, int dtype, int height, int width, const double* threshold_dev,
                  double fixed_threshold, int invert, int connectivity, int* labels, int* count,
                  void* workspace, size_t workspace_bytes, void* stream) {
    (void)labels;
    SPX_REQUIRE(height > 0 && width > 0, "bad image size");
    SPX_REQUIRE((long long)((height + 1) / 2) * ((width + 1) / 2) * 4 < 0x7fffffffLL,
                "image too large for 32-bit labels");
    SPX_REQUIRE(connectivity == 8 || connectivity == 4, "connectivity must be 4 or 8");
    SPX_REQUIRE(dtype >= SPX_U8 && dtype <= SPX_F64, "bad dtype");
    SPX_REQUIRE(img && count && workspace, "null pointer");
    SPX_REQUIRE(workspace_bytes >= spx_ccl_workspace_bytes(height, width), "workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CclLayout L = ccl_layout(workspace, height, width, nullptr);
    Geo g{height, width, (width + 1) / 2, connectivity};
    SPX_CUDA(cudaMemsetAsync(L.roots, 0, L.words * sizeof(unsigned int), s));
    const int tiles_x = (width + kTileW - 1) / kTileW, tiles_y = (height + kTileH - 1) / kTileH;
    const long long tiles = (long long)tiles_x * tiles_y;
    const int wide = (long long)width * (dtype == SPX_U8 ? 1 : 2) % 16 == 0 && (reinterpret_cast<uintptr_t>(img) & 15) == 0;
    auto local = [&](auto px) {
        using Px = decltype(px);
        k_local_ccl<Px><<<(unsigned)((tiles + kCclWarps - 1) / kCclWarps), kCclThreads, 0, s>>>(
            static_cast<const Px*>(img), g, threshold_dev, fixed_threshold, invert, wide, tiles_x, tiles, L.parents, L.roots,
            L.fgbits);
    };
    switch (dtype) {
        case SPX_U8: local(uint8_t{}); break;
        case SPX_U16: local(uint16_t{}); break;
        case SPX_F32: local(float{}); break;
        default: local(double{}); break;
    }
    if (int e = check_launch("k_local_ccl")) return e;
    const long long border = (long long)tiles_x * tiles_y * (kTileW + 2 * kTileH);
    k_border_merge<<<grid_for(border, 256), 256, 0, s>>>(g, L.parents, L.roots, L.fgbits, tiles_x, tiles_y);
    if (int e = check_launch("k_border_merge")) return e;
    SPX_REQUIRE(L.scan_blocks <= 1024 * 64, "image too large for the label prefix");
    if (L.scan_blocks <= kScanDirect) {
        k_popc_prefix_direct<<<L.scan_blocks, 1024, 0, s>>>(L.roots, L.words, L.prefix, count);
        return check_launch("k_popc_prefix_direct");
    }
    k_popc_block_sums<<<L.scan_blocks, 1024, 0, s>>>(L.roots, L.words, kScanPerBlock, L.block_sums);
    if (int e = check_launch("k_popc_block_sums")) return e;
    k_scan_small<<<1, 1024, 0, s>>>(L.block_sums, L.scan_blocks, count);
    if (int e = check_launch("k_scan_small")) return e;
    k_popc_prefix<<<L.scan_blocks, 1024, 0, s>>>(L.roots, L.words, kScanPerBlock, L.block_sums, L.prefix);
    return check_launch("k_popc_prefix");
}

static int ccl_finish(int* labels, int height, int width, int connectivity, int num_components, const int* count,
                      int* stats, double* centroids, void* workspace, size_t workspace_bytes, void* stream) {
    SPX_REQUIRE(labels && stats && centroids && workspace, "null pointer");
    SPX_REQUIRE(num_components >= 0, "bad component count");
    SPX_REQUIRE(workspace_bytes >= spx_ccl_workspace_bytes(height, width), "workspace too small");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    CclLayout L = ccl_layout(workspace, height, width, nullptr);
    Geo g{height, width, (width + 1) / 2, connectivity};
    const int k1 = num_components + 1;
    // The u64 coordinate sums live in the centroid array until the last kernel converts them.
    unsigned long long* sums = reinterpret_cast<unsigned long long*>(centroids);
    k_stats_init<<<grid_for(k1, 256), 256, 0, s>>>(stats, sums, k1);
    if (int e = check_launch("k_stats_init")) return e;
    const int tiles_x = (width + kTileW - 1) / kTileW;
    const long long tiles = (long long)tiles_x * ((height + kTileH - 1) / kTileH);
    // Warps enough to fill the chip, each with several tiles on large images.
    const int blocks = (int)std::min<long long>((tiles + kCclWarps - 1) / kCclWarps, 148 * kFinishBlocks);
    k_finish<<<blocks, kCclThreads, 0, s>>>(g, L.parents, L.roots, L.prefix, L.fgbits, tiles_x, tiles, labels, stats,
                                            sums, k1, count);
    if (int e = check_launch("k_finish")) return e;
    k_stats_final<<<grid_for(k1, 256), 256, 0, s>>>(stats, sums, centroids, k1);
    return check_launch("k_stats_final");
}

int spx_ccl_finish(int* labels, int height, int width, int connectivity, int num_components, int* stats,
                   double* centroids, void* workspace, size_t workspace_bytes, void* stream) {
    return ccl_finish(labels, height, width, connectivity, num_components, nullptr, stats, centroids, workspace,
                      workspace_bytes, stream);
}

int spx_ccl_finish_counted(int* labels, int height, int width, int connectivity, int capacity, const int* count,
                           int* stats, double* centroids, void* workspace, size_t workspace_bytes, void* stream) {
    SPX_REQUIRE(count, "null pointer");
    return ccl_finish(labels, height, width, connectivity, capacity, count, stats, centroids, workspace,
                      workspace_bytes, stream);
}

}  // extern "C"
