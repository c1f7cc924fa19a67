// apply.cu -- C-ABI entry points of the element stiffness apply y = D K(x) D p.
#include <float.h>

#include "apply_modal.cuh"
#include "internal.h"

namespace gbs {

template <typename Tile, typename T, typename KeT>
int launch_apply_plain(const gbsimp_ctx *ctx, int nx, int ny, int nz, const Law<T> &law, const KeT &ke,
                       const float *x, const T *p, T *y, const uint8_t *mask, cudaStream_t st) {
    TileArgs<T> A{nx, ny, nz, x, p, y, mask};
    PcgArgs pa{};
    const dim3 g = tile_grid<Tile>(nx, ny, nz), b = tile_block<Tile>();
    if (ctx->translation_free)
        apply_tile_kernel<T, KeT, Tile::X, Tile::Y, Tile::Z, true, MODE_PLAIN><<<g, b, 0, st>>>(A, law, ke, pa);
    else
        apply_tile_kernel<T, KeT, Tile::X, Tile::Y, Tile::Z, false, MODE_PLAIN><<<g, b, 0, st>>>(A, law, ke, pa);
    GBS_LAUNCH_CHECK("apply_tile_kernel");
    return GBS_OK;
}

int apply_f32(const gbsimp_ctx *ctx, int nx, int ny, int nz, const gbsimp_law *law, const float *x,
              const float *p, float *y, const uint8_t *mask, cudaStream_t st) {
    if (ctx->modal_ok && modal_fits(nz)) return apply_plain(ctx, nx, ny, nz, make_law<float>(*law), x, p, y, mask, st);
    return launch_apply_plain<TileF, float, KeF>(ctx, nx, ny, nz, make_law<float>(*law), ctx->kef, x, p, y, mask,
                                                 st);
}

int apply_f64(const gbsimp_ctx *ctx, int nx, int ny, int nz, const gbsimp_law *law, const float *x,
              const double *p, double *y, const uint8_t *mask, cudaStream_t st) {
    return launch_apply_plain<TileD, double, KeD>(ctx, nx, ny, nz, make_law<double>(*law), ctx->ked, x, p, y,
                                                  mask, st);
}

// ---- arbitrary edof table (drop-in for cuda_kernels.fused_spmv / simp_sensitivity) ----
// A block's rows of the table go through shared memory: a row is 96 or 192 bytes and a thread's, so that
// reading it straight took a sector per index and lane. Rows are padded by one index (no bank conflicts).
constexpr int kEdofNT = 128;
constexpr int kEdofRow = 25;
template <typename I>
__device__ __forceinline__ void edof_rows(const void *edof, int64_t e0, int64_t n_elem, I *rows) {
    const I *src = (const I *)edof + e0 * 24;
    const int n = 24 * (int)(n_elem - e0 < kEdofNT ? n_elem - e0 : kEdofNT);
#pragma unroll 8
    for (int q = threadIdx.x; q < n; q += kEdofNT) rows[q / 24 * kEdofRow + q % 24] = src[q];
    __syncthreads();
}

__global__ void zero_f32_kernel(float *y, int64_t n) {
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = 0.0f;
}

// One thread per element: gather p_e, y_e = E_e Ke p_e, scatter with atomics. Indices
// outside [0, n_dof) read as 0 and are not written (as the reference kernel clamps them,
// cuda_kernels/simp_sensitivity_ptx.cu:223-230).
// 65536 elements, 64-bit table: 6.9 us (9.7 without the staged rows).
template <typename I>
__global__ void __launch_bounds__(kEdofNT) apply_edof_kernel(int64_t n_elem, int64_t n_dof, const void *edof,
                                                             Law<float> law, const KeF ke, const float *x,
                                                             const float *p, float *y) {
    __shared__ I rows[kEdofNT * kEdofRow];
    const int64_t e0 = blockIdx.x * (int64_t)kEdofNT, e = e0 + threadIdx.x;
    edof_rows<I>(edof, e0, n_elem, rows);
    if (e >= n_elem) return;
    const I *idx = rows + threadIdx.x * kEdofRow;
    float pe[24];
#pragma unroll
    for (int q = 0; q < 24; ++q) {
        const int64_t d = (int64_t)idx[q];
        pe[q] = (d >= 0 && d < n_dof) ? p[d] : 0.0f;
    }
    const float E = modulus(law, x[e]);
#pragma unroll
    for (int r = 0; r < 24; ++r) {
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < 24; ++q) s = fmaf(ke.k[r * 24 + q], pe[q], s);
        const int64_t d = (int64_t)idx[r];
        if (d >= 0 && d < n_dof) atomicAdd(&y[d], E * s);
    }
}

// The energy's 24 products, exact to their rounding errors, are summed in FP32 pairs (2^-46); an FP64 sum,
// with its conversions, took half of the kernel's 16 us at 65536 elements (6.4 so). The displacements are
// scaled by a power of two to a largest component between 1 and 2, so that displacements of any size keep
// to the pairs (a call took 17 to 18 us at every size; unscaled, 15 to 19, and 23 at 1e-13 and below, where
// the sums ran in FP64). Where a pair does not hold the sum all the same (infinities, NaN, a stiffness near either end of the range) it runs in FP64.
template <typename I>
__global__ void __launch_bounds__(kEdofNT) sens_edof_kernel(int64_t n_elem, int64_t n_dof, const void *edof,
                                                            Law<float> law, const KeF ke, const float *x,
                                                            const float *u, float *dc) {
    __shared__ I rows[kEdofNT * kEdofRow];
    const int64_t e0 = blockIdx.x * (int64_t)kEdofNT, e = e0 + threadIdx.x;
    edof_rows<I>(edof, e0, n_elem, rows);
    if (e >= n_elem) return;
    float ue[24], most = 0.0f;
#pragma unroll
    for (int q = 0; q < 24; ++q) {
        const int64_t d = (int64_t)rows[threadIdx.x * kEdofRow + q];
        ue[q] = (d >= 0 && d < n_dof) ? u[d] : 0.0f;
        most = fmaxf(most, fabsf(ue[q]));
    }
    // the exponent of the largest component; 2^-ex as a product of two factors within the range
    const int ex = most > 0.0f && most <= FLT_MAX ? ilogbf(most) : 0;
    const float f1 = __int_as_float((127 - ex / 2) << 23), f2 = __int_as_float((127 - (ex - ex / 2)) << 23);
    float h = 0.0f, l = 0.0f, ws = 0.0f, ss = 0.0f;
#pragma unroll
    for (int q = 0; q < 24; ++q) ue[q] = ue[q] * f1 * f2;
#pragma unroll
    for (int r = 0; r < 24; ++r) {
        float s = 0.0f;
#pragma unroll
        for (int q = 0; q < 24; ++q) s = fmaf(ke.k[r * 24 + q], ue[q], s);
        const float w = __fmul_rn(ue[r], s);
        float d;
        l = __fadd_rn(l, __fmaf_rn(ue[r], s, -w));
        two_sum(h, w, h, d);
        l = __fadd_rn(l, d);
        ws = fmaxf(ws, fabsf(w));
        ss = fmaxf(ss, fabsf(s));
    }
    float ce = h + l;
    if (!(fabsf(ce) < 1e37f) || (ss > 0.0f && ws < 1e-25f)) {
        double c = 0.0;
#pragma unroll 1
        for (int r = 0; r < 24; ++r) {
            float s = 0.0f, ur = 0.0f;
            for (int q = 0; q < 24; ++q) {
                const int64_t d = (int64_t)rows[threadIdx.x * kEdofRow + q];
                const float uq = (d >= 0 && d < n_dof) ? u[d] : 0.0f;
                s = fmaf(ke.k[r * 24 + q], uq, s);
                if (q == r) ur = uq;
            }
            c += (double)ur * (double)s;
        }
        ce = (float)c;
    } else if (ex != 0) {
        ce = ldexpf(ce, 2 * ex);
    }
    dc[e] = -dmodulus(law, x[e]) * ce;
}

}  // namespace gbs

using namespace gbs;

extern "C" int gbsimp_apply_f32(gbsimp_ctx *ctx, int nx, int ny, int nz, const gbsimp_law *law, const float *x,
                                const float *p, float *y, const uint8_t *node_mask, void *stream) {
    if (!ctx || !law || !x || !p || !y || !grid_ok(nx, ny, nz))
        return set_error(GBS_EINVAL, "gbsimp_apply_f32: bad arguments");
    return apply_f32(ctx, nx, ny, nz, law, x, p, y, node_mask, (cudaStream_t)stream);
}

extern "C" int gbsimp_apply_path(const gbsimp_ctx *ctx, int nz) {
    if (!ctx) return -1;
    return (ctx->modal_ok && modal_fits(nz)) ? 1 : 0;
}

extern "C" int gbsimp_apply_f64(gbsimp_ctx *ctx, int nx, int ny, int nz, const gbsimp_law *law, const float *x,
                                const double *p, double *y, const uint8_t *node_mask, void *stream) {
    if (!ctx || !law || !x || !p || !y || !grid_ok(nx, ny, nz))
        return set_error(GBS_EINVAL, "gbsimp_apply_f64: bad arguments");
    return apply_f64(ctx, nx, ny, nz, law, x, p, y, node_mask, (cudaStream_t)stream);
}

extern "C" int gbsimp_apply_edof_f32(gbsimp_ctx *ctx, int64_t n_elem, int64_t n_dof, const void *edof,
                                     int edof_is_int64, const gbsimp_law *law, const float *x, const float *p,
                                     float *y, void *stream) {
    if (!ctx || !law || !edof || !x || !p || !y || n_elem < 0 || n_dof < 0)
        return set_error(GBS_EINVAL, "gbsimp_apply_edof_f32: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    if (n_dof > 0) {
        zero_f32_kernel<<<(unsigned)((n_dof + 255) / 256 < 65535 ? (n_dof + 255) / 256 : 65535), 256, 0, st>>>(y, n_dof);
        GBS_LAUNCH_CHECK("zero_f32_kernel");
    }
    if (n_elem == 0) return GBS_OK;
    const unsigned blocks = (unsigned)((n_elem + kEdofNT - 1) / kEdofNT);
    if (edof_is_int64)
        apply_edof_kernel<int64_t><<<blocks, kEdofNT, 0, st>>>(n_elem, n_dof, edof, make_law<float>(*law), ctx->kef, x, p, y);
    else
        apply_edof_kernel<int32_t><<<blocks, kEdofNT, 0, st>>>(n_elem, n_dof, edof, make_law<float>(*law), ctx->kef, x, p, y);
    GBS_LAUNCH_CHECK("apply_edof_kernel");
    return GBS_OK;
}

extern "C" int gbsimp_sensitivity_edof_f32(gbsimp_ctx *ctx, int64_t n_elem, int64_t n_dof, const void *edof,
                                           int edof_is_int64, const gbsimp_law *law, const float *x,
                                           const float *u, float *dc, void *stream) {
    if (!ctx || !law || !edof || !x || !u || !dc || n_elem < 0 || n_dof < 0)
        return set_error(GBS_EINVAL, "gbsimp_sensitivity_edof_f32: bad arguments");
    if (n_elem == 0) return GBS_OK;
    cudaStream_t st = (cudaStream_t)stream;
    const unsigned blocks = (unsigned)((n_elem + kEdofNT - 1) / kEdofNT);
    if (edof_is_int64)
        sens_edof_kernel<int64_t><<<blocks, kEdofNT, 0, st>>>(n_elem, n_dof, edof, make_law<float>(*law), ctx->kef, x, u, dc);
    else
        sens_edof_kernel<int32_t><<<blocks, kEdofNT, 0, st>>>(n_elem, n_dof, edof, make_law<float>(*law), ctx->kef, x, u, dc);
    GBS_LAUNCH_CHECK("sens_edof_kernel");
    return GBS_OK;
}
