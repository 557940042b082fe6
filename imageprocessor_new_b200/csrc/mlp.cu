// The learned warm start of the LM fits: a 1024 -> 256 -> 256 -> 7 MLP on 32x32 cell patches.
//
// GEMMs run on the 5th-generation tensor cores: one CTA of 256 threads computes a 128 x BN tile of
// C = A B^T (A: M x K, B: N x K, both bf16 and K-contiguous) with the accumulator in TMEM. One thread
// brings 64-wide K-blocks of both operands into a ring of 128-byte-swizzled shared-memory tiles by TMA
// (zero past M, N and K), another issues four tcgen05.mma (K = 16 each) per block and commits them to
// the mbarrier that gives the stage back. The epilogue reads TMEM with tcgen05.ld (warps w and w + 4 own
// rows 32w..32w+31, every other 16 columns each) and applies scale, bias, ReLU or the ReLU derivative of
// a forward activation, and writes f32 and/or bf16 outputs, row-major or transposed (the transposed
// copies feed the weight-gradient GEMMs, whose reduction runs over the batch).
//
// Every element is accumulated over K in one order, whatever the tile (column_tile), so a product's bits
// do not depend on the number of rows. For that reason K is not split either: AdamW divides a gradient
// by its own size, and the sign of a gradient near zero is decided by the last bits of its sum.
//
// Bound: latency. A training step's products are small (batch 4096: 6 GFLOP in eight GEMMs, 4 us at the
// tensor cores' rate); what counts is how many CTAs share a product, that no thread stands between a copy
// and its MMA, and an epilogue of few instructions. With the K-blocks copied by 128 threads (cp.async,
// some 200 instructions a thread and block), 256-wide tiles (2 to 32 CTAs) and an element-wise epilogue
// (1 us per 16 columns) the eight took 443 us of a 506 us step; with TMA, tiles down to 16 columns,
// the vector epilogue, the weight gradients in one launch and each launch overlapping the one before the
// step takes 73 us (the GEMMs 60: 24 of them the weight gradients' chain of 256 dependent MMAs). 40,000
// cells' first layer (256-wide tiles): 60 -> 34 us.
//
// Every wait on an mbarrier is bounded; a wait that runs out sets the error flag, and the kernel still
// waits for its copies and frees its TMEM.

#include <cuda.h>
#include <cuda_bf16.h>

#include <algorithm>
#include <utility>

#include "umma.cuh"

namespace spx {
namespace {

constexpr int kGemmThreads = 256;
constexpr int kGemmBM = 128;
constexpr int kGemmBK = 64;
constexpr int kGemmStagesMax = 8;
constexpr long long kWaitLimit = 1ll << 24;

// A training step's kernels follow one another with small grids: each is launched while the one before
// still runs (programmatic dependent launch), sets itself up, and waits here, before its first access
// to global memory, until that one has finished and its writes are visible. Without the launch
// attribute both calls do nothing.
__device__ __forceinline__ void wait_for_previous() {
    cudaTriggerProgrammaticLaunchCompletion();
    cudaGridDependencySynchronize();
}

struct GemmEpi {
    float scale;
    const float* bias;
    int relu;
    const __nv_bfloat16* mask_act;
    int ld_mask;
    float* out_f32;
    int ld_f32;
    int accumulate;
    __nv_bfloat16* out_bf16;
    int ld_bf16;
    __nv_bfloat16* out_bf16_t;
    int ld_t;
};

// Sixteen columns nb .. nb + 15 of output row m from their accumulators.
__device__ __forceinline__ void store_columns(const GemmEpi& ep, const float* v, int m, int nb, int N) {
    const int cnt = min(16, N - nb);
    if (cnt <= 0) return;
    float x[16];
    if (cnt == 16 && (!ep.bias || (reinterpret_cast<uintptr_t>(ep.bias + nb) & 15) == 0) &&
        (!ep.mask_act || (reinterpret_cast<uintptr_t>(ep.mask_act + (long long)m * ep.ld_mask + nb) & 15) == 0)) {
        // A full chunk: each option tested once, bias and mask by 16-byte loads (the element-wise form below
        // is some 300 instructions a chunk, 1 us at one warp per scheduler).
#pragma unroll
        for (int i = 0; i < 16; ++i) x[i] = v[i] * ep.scale;
        if (ep.bias) {
            const float4* b4 = reinterpret_cast<const float4*>(ep.bias + nb);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 b = b4[q];
                x[4 * q] += b.x;
                x[4 * q + 1] += b.y;
                x[4 * q + 2] += b.z;
                x[4 * q + 3] += b.w;
            }
        }
        if (ep.mask_act) {
            const uint4* m4 = reinterpret_cast<const uint4*>(ep.mask_act + (long long)m * ep.ld_mask + nb);
            const uint4 a = m4[0], b = m4[1];
            const uint32_t w[8] = {a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w};
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                if (!(__uint_as_float(w[q] << 16) > 0.0f)) x[2 * q] = 0.0f;
                if (!(__uint_as_float(w[q] & 0xffff0000u) > 0.0f)) x[2 * q + 1] = 0.0f;
            }
        }
        if (ep.relu) {
#pragma unroll
            for (int i = 0; i < 16; ++i) x[i] = fmaxf(x[i], 0.0f);
        }
    } else
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        const int n = nb + i;
        float t = v[i] * ep.scale;
        if (i < cnt) {
            if (ep.bias) t += ep.bias[n];
            if (ep.mask_act && !(__bfloat162float(ep.mask_act[(long long)m * ep.ld_mask + n]) > 0.0f)) t = 0.0f;
        }
        if (ep.relu) t = fmaxf(t, 0.0f);
        x[i] = t;
    }
    // Row-major outputs: 16-byte vector stores for a full, aligned chunk of 16 columns.
    if (ep.out_f32) {
        float* o = ep.out_f32 + (long long)m * ep.ld_f32 + nb;
        if (cnt == 16 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
            float4* o4 = reinterpret_cast<float4*>(o);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                float4 w = make_float4(x[4 * q], x[4 * q + 1], x[4 * q + 2], x[4 * q + 3]);
                if (ep.accumulate) {
                    const float4 u = o4[q];
                    w.x += u.x; w.y += u.y; w.z += u.z; w.w += u.w;
                }
                o4[q] = w;
            }
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < cnt) o[i] = ep.accumulate ? o[i] + x[i] : x[i];
        }
    }
    if (ep.out_bf16) {
        __nv_bfloat16* o = ep.out_bf16 + (long long)m * ep.ld_bf16 + nb;
        if (cnt == 16 && (reinterpret_cast<uintptr_t>(o) & 15) == 0) {
            uint4 pk[2];
            uint32_t* w = reinterpret_cast<uint32_t*>(pk);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const __nv_bfloat162 h = __floats2bfloat162_rn(x[2 * q], x[2 * q + 1]);
                w[q] = *reinterpret_cast<const uint32_t*>(&h);
            }
            reinterpret_cast<uint4*>(o)[0] = pk[0];
            reinterpret_cast<uint4*>(o)[1] = pk[1];
        } else {
#pragma unroll
            for (int i = 0; i < 16; ++i)
                if (i < cnt) o[i] = __float2bfloat16_rn(x[i]);
        }
    }
    if (ep.out_bf16_t) {  // consecutive rows on consecutive lanes: coalesced per column
        __nv_bfloat16* o = ep.out_bf16_t + (long long)nb * ep.ld_t + m;
#pragma unroll
        for (int i = 0; i < 16; ++i, o += ep.ld_t)
            if (i < cnt) *o = __float2bfloat16_rn(x[i]);
    }
}

// P independent products in one launch: CTA b works on the product whose tiles hold b.
struct GemmProblem {
    CUtensorMap map_a, map_b;
    int M, N, K, BN, row_tiles, first;  // first: its first CTA
    uint32_t tmem_cols;
    GemmEpi ep;
};
template <int P>
struct GemmBatch {
    GemmProblem p[P];
    int stages;
    int* err;
};

template <int P>
__global__ void __launch_bounds__(kGemmThreads) k_gemm_bf16(const __grid_constant__ GemmBatch<P> batch) {
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t full[kGemmStagesMax], empty[kGemmStagesMax], finished;
    __shared__ uint32_t tmem_slot;
    int which = 0;
#pragma unroll
    for (int q = 1; q < P; ++q) which += (int)blockIdx.x >= batch.p[q].first;
    const GemmProblem& g = batch.p[which];
    const int M = g.M, N = g.N, K = g.K, BN = g.BN, stages = batch.stages;
    const int tile = (int)blockIdx.x - g.first;
    // 1024-byte aligned stages [A | B].
    uint8_t* base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int a_bytes = kGemmBM * 128, stage_bytes = a_bytes + BN * 128;
    const int warp = threadIdx.x >> 5;
    const int m0 = tile % g.row_tiles * kGemmBM, n0 = tile / g.row_tiles * BN;
    if (warp == 0) tmem_alloc(&tmem_slot, g.tmem_cols);
    if (threadIdx.x == 0) {
        for (int s = 0; s < stages; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(&finished, 1);
        fence_mbar_init();
    }
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;
    wait_for_previous();
    const int nk = (K + kGemmBK - 1) / kGemmBK;
    if (threadIdx.x == 0) {
        int issued = 0;
        bool ok = true;
        for (int kb = 0, s = 0, round = 0; kb < nk && ok; ++kb) {
            if (round > 0) ok = mbar_wait(&empty[s], (round - 1) & 1, kWaitLimit);
            if (ok) {
                uint8_t* stage = base + s * stage_bytes;
                mbar_expect_tx(&full[s], stage_bytes);
                tma_load_2d(stage, &g.map_a, kb * kGemmBK, m0, &full[s]);
                tma_load_2d(stage + a_bytes, &g.map_b, kb * kGemmBK, n0, &full[s]);
                ++issued;
            }
            if (++s == stages) {
                s = 0;
                ++round;
            }
        }
        // No copy into shared memory outlives the block (when nothing failed, the MMAs have waited for each).
        for (int kb = max(0, issued - stages); kb < issued; ++kb)
            mbar_wait(&full[kb % stages], (kb / stages) & 1, kWaitLimit);
    } else if (threadIdx.x == 32) {
        const uint32_t idesc = umma_idesc_bf16(kGemmBM, BN);
        bool ok = true;
        for (int kb = 0, s = 0, round = 0; kb < nk && ok; ++kb) {
            ok = mbar_wait(&full[s], round & 1, kWaitLimit);
            if (ok) {
                tc_fence_after();
                const uint8_t* stage = base + s * stage_bytes;
                const uint64_t ad = umma_desc_sw128(smem_u32(stage)), bd = umma_desc_sw128(smem_u32(stage + a_bytes));
#pragma unroll
                for (int k = 0; k < kGemmBK / 16; ++k)
                    umma_bf16(tmem, ad + (uint64_t)((k * 32) >> 4), bd + (uint64_t)((k * 32) >> 4), idesc,
                              (kb > 0 || k > 0) ? 1u : 0u);
                umma_commit(&empty[s]);
            }
            if (++s == stages) {
                s = 0;
                ++round;
            }
        }
        if (ok) umma_commit(&finished);  // covers every MMA of the tile
    }
    __syncwarp();
    // `ok` is block-uniform, so the warp-collective tcgen05.ld runs with whole warps or not at all.
    const bool ok = __syncthreads_and(mbar_wait(&finished, 0, kWaitLimit)) != 0;
    tc_fence_after();
    if (!ok && threadIdx.x == 0) atomicExch(batch.err, 1);
    if (ok) {
        const int quarter = warp & 3, m = m0 + quarter * 32 + (threadIdx.x & 31);
        const uint32_t lane_addr = tmem + ((uint32_t)(quarter * 32) << 16);
        for (int c0 = 16 * (warp >> 2); c0 < BN; c0 += 32) {
            float v[16];
            tmem_ld16(lane_addr + (uint32_t)c0, v);
            if (m < M) store_columns(g.ep, v, m, n0 + c0, N);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, g.tmem_cols);
}

// Weighted MSE gradient: dy = 2 w_j (y - t) / B as bf16, row-major (B x ldd, zero in the padding
// columns) and transposed (ldd x B); loss += sum w_j (y - t)^2 / B (f64 atomics per block).
__global__ void k_mse_grad(const float* y, const float* t, const float* w, int B, int nout, int ldd,
                           __nv_bfloat16* dy, __nv_bfloat16* dy_t, double* loss) {
    __shared__ double s_part[32];
    wait_for_previous();
    double part = 0.0;
    const long long total = (long long)B * ldd;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
         i += (long long)gridDim.x * blockDim.x) {
        int b, j;
        divmod_idx(i, ldd, &b, &j);
        float g = 0.0f;
        if (j < nout) {
            const float d = y[(long long)b * nout + j] - t[(long long)b * nout + j];
            part += (double)w[j] * d * d;
            g = 2.0f * w[j] * d / (float)B;
        }
        const __nv_bfloat16 gb = __float2bfloat16_rn(g);
        dy[i] = gb;
        dy_t[(long long)j * B + b] = gb;
    }
    part = warp_sum(part);
    if ((threadIdx.x & 31) == 0) s_part[threadIdx.x >> 5] = part;
    __syncthreads();
    if (threadIdx.x == 0) {
        double acc = 0.0;
        for (int i = 0; i < (int)(blockDim.x >> 5); ++i) acc += s_part[i];
        atomicAdd(loss, acc / (double)B);
    }
}

// Sum of one row of C bf16 values by a warp, f32 accumulation: eight values a lane and load where the
// row allows it (its start on 16 bytes).
__device__ __forceinline__ float row_sum_bf16(const __nv_bfloat16* src, int C, int lane) {
    float acc = 0.0f;
    int c = 0;
    if ((reinterpret_cast<uintptr_t>(src) & 15) == 0) {
        c = C & ~255;
        for (int k = lane * 8; k < c; k += 256) {
            const uint4 q = *reinterpret_cast<const uint4*>(src + k);
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int u = 0; u < 4; ++u)
                acc += __uint_as_float(w[u] << 16) + __uint_as_float(w[u] & 0xffff0000u);
        }
    }
    for (c += lane; c < C; c += 32) acc += __bfloat162float(src[c]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
    return acc;
}

// out[r] = sum over the row r of up to three bf16 matrices of C columns, one warp per row.
struct RowSums {
    const __nv_bfloat16* src[3];
    float* out[3];
    int rows[3];
};
__global__ void k_rowsum_bf16(RowSums a, int C) {
    wait_for_previous();
    const int lane = threadIdx.x & 31;
    const int total = a.rows[0] + a.rows[1] + a.rows[2];
    for (int t = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); t < total; t += gridDim.x * (blockDim.x >> 5)) {
        const int q = t < a.rows[0] ? 0 : t < a.rows[0] + a.rows[1] ? 1 : 2;
        const int r = t - (q > 0 ? a.rows[0] : 0) - (q > 1 ? a.rows[1] : 0);
        const __nv_bfloat16* src = q == 0 ? a.src[0] : q == 1 ? a.src[1] : a.src[2];
        float* out = q == 0 ? a.out[0] : q == 1 ? a.out[1] : a.out[2];
        const float acc = row_sum_bf16(src + (long long)r * C, C, lane);
        if (lane == 0) out[r] = acc;
    }
}

// AdamW on f32 parameters (rows x cols): m, v moments, bias-corrected step, decoupled decay; then
// the bf16 copy (row-major, padded to out_rows rows of zeros) and/or its transpose (cols x ld_t).
struct AdamParam {
    float* p;
    const float* g;
    float *m, *v;
    int rows, cols;
    float wd;
    __nv_bfloat16* out;
    int out_rows;
    __nv_bfloat16* out_t;
    int ld_t;
    __host__ __device__ long long total() const { return (long long)(rows > out_rows ? rows : out_rows) * cols; }
};
struct AdamRates {
    float lr, beta1, beta2, eps, c1, c2;
};

__device__ __forceinline__ void adamw_element(const AdamParam& a, const AdamRates& h, long long i) {
    int r, c;
    divmod_idx(i, a.cols, &r, &c);
    float w = 0.0f;
    if (r < a.rows) {
        const float gi = a.g[i];
        const float mi = h.beta1 * a.m[i] + (1.0f - h.beta1) * gi;
        const float vi = h.beta2 * a.v[i] + (1.0f - h.beta2) * gi * gi;
        a.m[i] = mi;
        a.v[i] = vi;
        const float mh = mi / h.c1, vh = vi / h.c2;
        w = a.p[i] - h.lr * (mh / (sqrtf(vh) + h.eps) + a.wd * a.p[i]);
        a.p[i] = w;
    }
    if (a.out && r < a.out_rows) a.out[i] = __float2bfloat16_rn(w);
    if (a.out_t && r < a.rows) a.out_t[(long long)c * a.ld_t + r] = __float2bfloat16_rn(w);
}

__global__ void k_adamw(AdamParam a, AdamRates h) {
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < a.total();
         i += (long long)gridDim.x * blockDim.x)
        adamw_element(a, h, i);
}

// The six parameters of the network in one launch.
struct AdamNet {
    AdamParam p[6];
};
__global__ void k_adamw_net(const __grid_constant__ AdamNet net, AdamRates h) {
    wait_for_previous();
    const long long stride = (long long)gridDim.x * blockDim.x;
    long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x;
#pragma unroll
    for (int q = 0; q < 6; ++q) {
        const long long n = net.p[q].total();
        for (; i < n; i += stride) adamw_element(net.p[q], h, i);
        i -= n;
    }
}

// dst (C x R) = src (R x C)^T for bf16, through 32 x 32 shared-memory tiles.
__global__ void k_transpose_bf16(const __nv_bfloat16* src, int R, int C, __nv_bfloat16* dst) {
    __shared__ __nv_bfloat16 tile[32][33];
    const int c0 = blockIdx.x * 32, r0 = blockIdx.y * 32;
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int r = r0 + i, c = c0 + threadIdx.x;
        if (r < R && c < C) tile[i][threadIdx.x] = src[(long long)r * C + c];
    }
    __syncthreads();
    for (int i = threadIdx.y; i < 32; i += blockDim.y) {
        const int c = c0 + i, r = r0 + threadIdx.x;
        if (r < R && c < C) dst[(long long)c * R + r] = tile[threadIdx.x][i];
    }
}

// Standardised MLP outputs -> ROI-local LM starting params: A = t0 amp, x0 = ox + 16 + t1 - box.x,
// y0 = oy + 16 + t2 - box.y, u = t3..t5 (t = y * std + mean); ok = finite and A > 0.
__global__ void k_outputs_to_params(const float* y, const double* mean, const double* stdv, const double* norm,
                                    const int4* boxes, int n, double* params, uint8_t* ok) {
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        double t[6];
#pragma unroll
        for (int j = 0; j < 6; ++j) t[j] = (double)y[7LL * i + j] * stdv[j] + mean[j];
        const double* nm = norm + 4LL * i;
        const int4 b = boxes[i];
        // Patch origin relative to the box first (exact integers), so the result does not depend on
        // where the box sits (a stack's rows).
        const double p[6] = {t[0] * nm[3], (nm[0] - b.x) + 16.0 + t[1], (nm[1] - b.y) + 16.0 + t[2], t[3], t[4],
                             t[5]};
        bool good = p[0] > 0.0;
#pragma unroll
        for (int j = 0; j < 6; ++j) {
            good = good && isfinite(p[j]);
            params[6LL * i + j] = p[j];
        }
        ok[i] = good;
    }
}

// Column tile of an M x N product: the widest tile (256, 128, .. 16 columns; all of a
// narrower N) that still gives nearly every SM a CTA, else 16. Measured at 4096 x 256 x 1024 (32 row tiles):
// 256 columns 13.3 us, 64 columns 9.9 us; at 256 x 1024 x 4096 (two row tiles): 256 columns 26.4 us, 64 columns
// 23.7 us, 16 columns 22.1 us.
int column_tile(int M, int N) {
    const long long mt = (M + kGemmBM - 1) / kGemmBM;
    int bn = 256;
    while (bn > 16 && mt * ((N + bn - 1) / bn) < 120) bn /= 2;
    return std::min(bn, (N + 15) / 16 * 16);
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_tiled() {
    static const EncodeTiled fn = [] {
        void* f = nullptr;
        cudaDriverEntryPointQueryResult found = cudaDriverEntryPointSymbolNotFound;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            f = nullptr;
        return reinterpret_cast<EncodeTiled>(f);
    }();
    return fn;
}

// Tensor map of a rows x K bf16 matrix (row stride ld) read in boxes of box_rows x 64, 128-byte swizzle.
bool tile_map(CUtensorMap* map, const void* p, int rows, int K, int ld, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)K, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)ld * 2};
    const cuuint32_t box[2] = {(cuuint32_t)kGemmBK, (cuuint32_t)box_rows};
    const cuuint32_t step[2] = {1, 1};
    return encode_tiled()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(p), dims, strides, box, step,
                          CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}

// One product of a launch.
struct GemmCall {
    const __nv_bfloat16* A;
    int lda;
    const __nv_bfloat16* B;
    int ldb, M, N, K;
    GemmEpi ep;
};

// Launches a kernel, `chained`: as the next of a training step (wait_for_previous).
template <class... Params, class... Args>
int launch(const char* what, void (*kernel)(Params...), int grid, int threads, size_t smem, cudaStream_t s, bool chained,
           Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = chained ? 1 : 0;
    SPX_CUDA(cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...));
    return check_launch(what);
}

template <int P>
int gemm(const GemmCall (&calls)[P], int* err, cudaStream_t s, bool chained = false) {
    SPX_REQUIRE(encode_tiled(), "the driver has no cuTensorMapEncodeTiled");
    GemmBatch<P> batch;
    int ctas = 0, widest = 0;
    for (int q = 0; q < P; ++q) {
        const GemmCall& c = calls[q];
        GemmProblem& g = batch.p[q];
        g.M = c.M;
        g.N = c.N;
        g.K = c.K;
        g.BN = column_tile(c.M, c.N);
        SPX_REQUIRE(tile_map(&g.map_a, c.A, c.M, c.K, c.lda, kGemmBM) && tile_map(&g.map_b, c.B, c.N, c.K, c.ldb, g.BN),
                    "cuTensorMapEncodeTiled refused the operands");
        g.row_tiles = (c.M + kGemmBM - 1) / kGemmBM;
        g.first = ctas;
        ctas += g.row_tiles * ((c.N + g.BN - 1) / g.BN);
        g.tmem_cols = 32;
        while ((int)g.tmem_cols < g.BN) g.tmem_cols <<= 1;
        g.ep = c.ep;
        widest = std::max(widest, g.BN);
    }
    // Rings take half an SM's shared memory, so that two CTAs share an SM and one's epilogue overlaps the
    // other's products.
    const int stage = kGemmBM * 128 + widest * 128;
    batch.stages = std::min(kGemmStagesMax, 100 * 1024 / stage);
    batch.err = err;
    const size_t smem = (size_t)batch.stages * stage + 1024;
    SPX_CUDA(cudaFuncSetAttribute(k_gemm_bf16<P>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    return launch("k_gemm_bf16", k_gemm_bf16<P>, ctas, kGemmThreads, smem, s, chained, batch);
}

// The warm-start network: inputs, hidden units, outputs and the padded outputs of its gradients.
constexpr int kMlpIn = 1024, kMlpHid = 256, kMlpOut = 7, kMlpOutPad = 16;

// Activations and their gradients of one training step, row-major and transposed.
struct TrainBuffers {
    float* y;
    __nv_bfloat16 *h1, *h1t, *h2, *h2t, *dy, *dyt, *dh2, *dh2t, *dh1t;
    size_t bytes;
    TrainBuffers(void* ws, int batch) {
        Arena a(ws);
        const size_t b = (size_t)batch;
        y = a.take<float>(b * kMlpOut);
        h1 = a.take<__nv_bfloat16>(b * kMlpHid);
        h1t = a.take<__nv_bfloat16>(b * kMlpHid);
        h2 = a.take<__nv_bfloat16>(b * kMlpHid);
        h2t = a.take<__nv_bfloat16>(b * kMlpHid);
        dy = a.take<__nv_bfloat16>(b * kMlpOutPad);
        dyt = a.take<__nv_bfloat16>(b * kMlpOutPad);
        dh2 = a.take<__nv_bfloat16>(b * kMlpHid);
        dh2t = a.take<__nv_bfloat16>(b * kMlpHid);
        dh1t = a.take<__nv_bfloat16>(b * kMlpHid);
        bytes = a.used;
    }
};

}  // namespace
}  // namespace spx

using namespace spx;

extern "C" {

int spx_gemm_bf16(const void* A, int lda, const void* B, int ldb, int M, int N, int K, const spx_gemm_epilogue* epi,
                  int* error_flag, void* stream) {
    SPX_REQUIRE(M > 0 && N > 0 && K > 0 && lda >= K && ldb >= K, "bad GEMM shape");
    SPX_REQUIRE(lda % 8 == 0 && ldb % 8 == 0, "lda and ldb must be multiples of 8 (16-byte rows)");
    SPX_REQUIRE(A && B && epi && error_flag, "null pointer");
    SPX_REQUIRE(reinterpret_cast<uintptr_t>(A) % 16 == 0 && reinterpret_cast<uintptr_t>(B) % 16 == 0,
                "operands must be 16-byte aligned");
    SPX_REQUIRE(epi->out_f32 || epi->out_bf16 || epi->out_bf16_t, "no output");
    const GemmEpi ep{epi->scale,
                     epi->bias,
                     epi->relu,
                     static_cast<const __nv_bfloat16*>(epi->mask_act),
                     epi->ld_mask,
                     epi->out_f32,
                     epi->ld_f32,
                     epi->accumulate,
                     static_cast<__nv_bfloat16*>(epi->out_bf16),
                     epi->ld_bf16,
                     static_cast<__nv_bfloat16*>(epi->out_bf16_t),
                     epi->ld_t};
    const GemmCall call[1] = {{static_cast<const __nv_bfloat16*>(A), lda, static_cast<const __nv_bfloat16*>(B), ldb, M, N, K, ep}};
    return gemm(call, error_flag, static_cast<cudaStream_t>(stream));
}

int spx_mlp_loss_grad(const float* y, const float* t, const float* weights, int batch, int n_out, int ld_grad,
                      void* dy, void* dy_t, double* loss, void* stream) {
    SPX_REQUIRE(batch > 0 && n_out > 0 && ld_grad >= n_out, "bad arguments");
    SPX_REQUIRE(y && t && weights && dy && dy_t && loss, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_mse_grad<<<grid_for((long long)batch * ld_grad, 256, 148 * 4), 256, 0, s>>>(
        y, t, weights, batch, n_out, ld_grad, static_cast<__nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(dy_t), loss);
    return check_launch("k_mse_grad");
}

int spx_rowsum_bf16(const void* src, int rows, int cols, float* out, void* stream) {
    SPX_REQUIRE(rows > 0 && cols > 0 && src && out, "bad arguments");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const RowSums a{{static_cast<const __nv_bfloat16*>(src), nullptr, nullptr}, {out, nullptr, nullptr}, {rows, 0, 0}};
    k_rowsum_bf16<<<grid_for(rows, 8, 148 * 8), 256, 0, s>>>(a, cols);
    return check_launch("k_rowsum_bf16");
}

int spx_adamw(float* param, const float* grad, float* m, float* v, int rows, int cols, int step, float lr, float beta1,
              float beta2, float eps, float weight_decay, void* out_bf16, int out_rows, void* out_bf16_t, int ld_t,
              void* stream) {
    SPX_REQUIRE(rows > 0 && cols > 0 && step >= 1 && out_rows >= 0 && (!out_bf16_t || ld_t >= rows),
                "bad arguments");
    SPX_REQUIRE(param && grad && m && v, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const float c1 = 1.0f - powf(beta1, (float)step), c2 = 1.0f - powf(beta2, (float)step);
    const AdamParam a{param, grad, m, v, rows, cols, weight_decay, static_cast<__nv_bfloat16*>(out_bf16), out_rows,
                      static_cast<__nv_bfloat16*>(out_bf16_t), ld_t};
    k_adamw<<<grid_for(a.total(), 256), 256, 0, s>>>(a, AdamRates{lr, beta1, beta2, eps, c1, c2});
    return check_launch("k_adamw");
}

size_t spx_mlp_train_workspace_bytes(int batch) { return batch > 0 ? TrainBuffers(nullptr, batch).bytes : 0; }

int spx_mlp_train_step(const spx_mlp_train* t, int batch, int step, float lr, float beta1, float beta2, float eps,
                       float weight_decay, void* workspace, size_t workspace_bytes, void* stream) {
    SPX_REQUIRE(t && batch > 0 && batch % 8 == 0 && step >= 1, "bad arguments (the batch is a multiple of 8)");
    SPX_REQUIRE(t->x && t->x_t && t->target && t->weights && t->loss && t->error_flag && t->w1 && t->w2 && t->w2_t &&
                    t->w3 && t->w3_t && workspace,
                "null pointer");
    for (int i = 0; i < 6; ++i) SPX_REQUIRE(t->param[i] && t->grad[i] && t->m[i] && t->v[i], "null pointer");
    SPX_REQUIRE(workspace_bytes >= spx_mlp_train_workspace_bytes(batch), "workspace too small");
    using bf = __nv_bfloat16;
    const bf *x = static_cast<const bf*>(t->x), *xt = static_cast<const bf*>(t->x_t);
    bf *w1 = static_cast<bf*>(t->w1), *w2 = static_cast<bf*>(t->w2), *w2t = static_cast<bf*>(t->w2_t);
    bf *w3 = static_cast<bf*>(t->w3), *w3t = static_cast<bf*>(t->w3_t);
    for (const void* q : {t->x, t->x_t, (const void*)w1, (const void*)w2, (const void*)w2t, (const void*)w3,
                          (const void*)w3t, (const void*)workspace})
        SPX_REQUIRE(reinterpret_cast<uintptr_t>(q) % 16 == 0, "operands must be 16-byte aligned");
    const TrainBuffers b(workspace, batch);
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    enum { W1 = 0, B1, W2, B2, W3, B3 };
    auto act = [&](const float* bias, bf* out, bf* out_t) {  // a hidden layer, row-major and transposed
        return GemmEpi{1.0f, bias, 1, nullptr, 0, nullptr, 0, 0, out, kMlpHid, out_t, batch};
    };
    auto grad_in = [&](const bf* mask, bf* out, bf* out_t) {  // a layer's input gradient through its ReLU
        return GemmEpi{1.0f, nullptr, 0, mask, kMlpHid, nullptr, 0, 0, out, kMlpHid, out_t, batch};
    };
    auto f32 = [&](const float* bias, float* out, int ld) {
        return GemmEpi{1.0f, bias, 0, nullptr, 0, out, ld, 0, nullptr, 0, nullptr, 0};
    };
    auto run = [&](const bf* A, int lda, const bf* B, int ldb, int M, int N, int K, const GemmEpi& ep) {
        const GemmCall call[1] = {{A, lda, B, ldb, M, N, K, ep}};
        return gemm(call, t->error_flag, s, true);
    };
    // Forward.
    if (int e = run(x, kMlpIn, w1, kMlpIn, batch, kMlpHid, kMlpIn, act(t->param[B1], b.h1, b.h1t))) return e;
    if (int e = run(b.h1, kMlpHid, w2, kMlpHid, batch, kMlpHid, kMlpHid, act(t->param[B2], b.h2, b.h2t))) return e;
    if (int e = run(b.h2, kMlpHid, w3, kMlpHid, batch, kMlpOut, kMlpHid, f32(t->param[B3], b.y, kMlpOut))) return e;
    if (int e = launch("k_mse_grad", k_mse_grad, grid_for((long long)batch * kMlpOutPad, 256, 148 * 4), 256, 0, s, true,
                       b.y, t->target, t->weights, batch, kMlpOut, kMlpOutPad, b.dy, b.dyt, t->loss))
        return e;
    // dH2 = (dY W3) (H2 > 0), dH1 = (dH2 W2) (H1 > 0); then the three weight gradients dH1^T X, dH2^T H1 and
    // dY^T H2 together: each is a chain of 4 x batch / 64 dependent MMAs on a few tiles (22 us at batch
    // 4096 whatever its width), so side by side they cost one chain.
    if (int e = run(b.dy, kMlpOutPad, w3t, kMlpOutPad, batch, kMlpHid, kMlpOutPad, grad_in(b.h2, b.dh2, b.dh2t)))
        return e;
    if (int e = run(b.dh2, kMlpHid, w2t, kMlpHid, batch, kMlpHid, kMlpHid, grad_in(b.h1, nullptr, b.dh1t))) return e;
    const GemmCall grads[3] = {{b.dh1t, batch, xt, batch, kMlpHid, kMlpIn, batch, f32(nullptr, t->grad[W1], kMlpIn)},
                               {b.dh2t, batch, b.h1t, batch, kMlpHid, kMlpHid, batch, f32(nullptr, t->grad[W2], kMlpHid)},
                               {b.dyt, batch, b.h2t, batch, kMlpOut, kMlpHid, batch, f32(nullptr, t->grad[W3], kMlpHid)}};
    if (int e = gemm(grads, t->error_flag, s, true)) return e;
    // The bias gradients, row sums of the transposed gradients.
    const RowSums sums{{b.dh1t, b.dh2t, b.dyt}, {t->grad[B1], t->grad[B2], t->grad[B3]}, {kMlpHid, kMlpHid, kMlpOut}};
    if (int e = launch("k_rowsum_bf16", k_rowsum_bf16, grid_for(2 * kMlpHid + kMlpOut, 4, 148 * 8), 128, 0, s, true, sums,
                       batch))
        return e;
    AdamNet net;
    auto set = [&](int i, int rows, int cols, float wd, bf* out, int out_rows, bf* out_t, int ld_t) {
        net.p[i] = AdamParam{t->param[i], t->grad[i], t->m[i], t->v[i], rows, cols, wd, out, out_rows, out_t, ld_t};
    };
    set(W1, kMlpHid, kMlpIn, weight_decay, w1, kMlpHid, nullptr, 0);
    set(B1, 1, kMlpHid, 0.0f, nullptr, 0, nullptr, 0);
    set(W2, kMlpHid, kMlpHid, weight_decay, w2, kMlpHid, w2t, kMlpHid);
    set(B2, 1, kMlpHid, 0.0f, nullptr, 0, nullptr, 0);
    set(W3, kMlpOut, kMlpHid, weight_decay, w3, kMlpOutPad, w3t, kMlpOutPad);
    set(B3, 1, kMlpOut, 0.0f, nullptr, 0, nullptr, 0);
    const AdamRates rates{lr, beta1, beta2, eps, 1.0f - powf(beta1, (float)step), 1.0f - powf(beta2, (float)step)};
    return launch("k_adamw_net", k_adamw_net, 148 * 4, 256, 0, s, true, net, rates);
}

int spx_transpose_bf16(const void* src, int rows, int cols, void* dst, void* stream) {
    SPX_REQUIRE(rows > 0 && cols > 0 && src && dst && src != dst, "bad arguments");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const dim3 grid((cols + 31) / 32, (rows + 31) / 32);
    k_transpose_bf16<<<grid, dim3(32, 8), 0, s>>>(static_cast<const __nv_bfloat16*>(src), rows, cols,
                                                 static_cast<__nv_bfloat16*>(dst));
    return check_launch("k_transpose_bf16");
}

int spx_mlp_outputs_to_params(const float* y, const double* out_mean, const double* out_std, const double* norm,
                              const int* boxes, int n, double* params, uint8_t* ok, void* stream) {
    SPX_REQUIRE(n >= 0, "bad arguments");
    if (n == 0) return SPX_OK;
    SPX_REQUIRE(y && out_mean && out_std && norm && boxes && params && ok, "null pointer");
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    k_outputs_to_params<<<grid_for(n, 256), 256, 0, s>>>(y, out_mean, out_std, norm,
                                                        reinterpret_cast<const int4*>(boxes), n, params, ok);
    return check_launch("k_outputs_to_params");
}

}  // extern "C"
