// voxel.cu -- the evaluator's input step on the device.
//
// A decoded (D, H, W) density grid is resampled with linear interpolation, as
// scipy.ndimage.zoom(v, 0.5, order=1) does in VoxelFEMEvaluator.evaluate
// (fem/voxel_fem.py:457-459): output index o reads input coordinate o (n_in - 1) / (n_out - 1)
// (grid_mode off), weights (1 - w, w) on floor and floor + 1, nothing beyond the last input.
// It is then filtered as smooth_voxels does (pipeline_utils.py:55-76): a Gaussian of sigma
// voxels (radius int(4 sigma + 0.5), weights exp(-t^2 / (2 sigma^2)) normalised to sum 1,
// mirror boundary "reflect": d c b a | a b c d | d c b a), then the logistic
// 1 / (1 + exp(-sharpness (v - 0.5))).
//
// Both linear steps are separable, so each axis gets one banded n_out x n_in matrix
// A = G Z, built on the device in FP64, and a batch of volumes goes through three 1-D passes
// (z, y, x; FP32 between passes, like the reference's float32 intermediates); the last pass
// applies the logistic. The weights are kept as pairs of FP32 numbers (48 bits) and the sums of a
// pass run in such pairs on the FP32 pipe: 16 volumes of 64^3 -> 32^3 take 52 us (passes 15, 13 and 11,
// the table 6), where FP64 sums took 459 (FP64 issue, 64-bit index divisions, 32 predicated taps where
// 10 are nonzero, and 14 us for each axis's table). The results are the same to the last bit there.
#include <math.h>

#include "internal.h"

namespace gbs {

constexpr int kVoxBand = 32;      // nonzeros per row of A
constexpr int kVoxMaxExtent = 1024;

struct VoxRow {
    int start, count;      // inputs start .. start + count - 1, all within the axis
    float2 w[kVoxBand];    // (hi, lo)
};
static_assert(sizeof(VoxRow) == 8 + 8 * kVoxBand, "workspace layout");
constexpr int kVoxMaxRadius = 256;  // sigma <= 64

static size_t al256v(size_t b) { return (b + 255) & ~(size_t)255; }

static inline int vox_radius(double sigma) { return sigma > 0.0 ? (int)(4.0 * sigma + 0.5) : 0; }

// Input span of one row of G Z (host check of the band).
static int vox_span(int n_in, int n_out, double sigma) {
    const double s = n_out > 1 ? (double)(n_in - 1) / (double)(n_out - 1) : 0.0;
    return (int)ceil(2.0 * vox_radius(sigma) * s) + 3;
}

__device__ __forceinline__ int vox_reflect(int j, int n) {
    // half-sample symmetric extension, repeated for offsets longer than the axis
    const int period = 2 * n;
    j %= period;
    if (j < 0) j += period;
    return j < n ? j : period - 1 - j;
}

struct VoxAxes {
    int n_in[3], n_out[3];
};

// The rows of the three axes' matrices (axis blockIdx.y), in FP64: a warp per output row, a lane per
// weight, so that the taps are the only serial chain; the Gaussian's weights are formed once per block, a
// thread each. A thread per row with its own exponentials and 32 weights took 14 us per axis.
constexpr int kVoxTableNT = 128;
__global__ void __launch_bounds__(kVoxTableNT) vox_table_kernel(VoxAxes ax, double sigma, VoxRow *rows) {
    __shared__ double g[2 * kVoxMaxRadius + 1];
    __shared__ double s_norm;
    const int a = blockIdx.y, n_in = ax.n_in[a], n_out = ax.n_out[a];
    rows += a > 0 ? ax.n_out[0] : 0;
    rows += a > 1 ? ax.n_out[1] : 0;
    const int tid = threadIdx.x, lane = tid & 31, r = sigma > 0.0 ? (int)(4.0 * sigma + 0.5) : 0;
    for (int i = tid; i <= 2 * r; i += kVoxTableNT) {
        const int t = i - r;
        g[i] = r > 0 ? exp(-0.5 / (sigma * sigma) * (double)(t * t)) : 1.0;
    }
    __syncthreads();
    if (tid == 0) {
        double norm = 0.0;
        for (int i = 0; i <= 2 * r; ++i) norm += g[i];
        s_norm = norm;
    }
    __syncthreads();
    for (int i = tid; i <= 2 * r; i += kVoxTableNT) g[i] = g[i] / s_norm;
    __syncthreads();
    const int o = blockIdx.x * (kVoxTableNT / 32) + (tid >> 5);
    if (o >= n_out) return;
    const double s = n_out > 1 ? (double)(n_in - 1) / (double)(n_out - 1) : 0.0;
    // the taps visit output rows from the lowest to the highest of the mirrored window
    int jlo = n_out;
    for (int t = -r; t <= r; ++t) jlo = min(jlo, vox_reflect(o + t, n_out));
    const int lo = (int)floor((double)jlo * s);
    double acc = 0.0;
    for (int t = -r; t <= r; ++t) {
        const double p = (double)vox_reflect(o + t, n_out) * s;
        const int i0 = (int)floor(p), k0 = i0 - lo;
        const double w = p - (double)i0;
        if (lane == k0) acc += g[t + r] * (1.0 - w);
        if (lane == k0 + 1 && i0 + 1 < n_in) acc += g[t + r] * w;
    }
    const double w = lo + lane < n_in ? acc : 0.0;
    const float h = (float)w;
    rows[o].w[lane] = make_float2(h, (float)(w - (double)h));
    const unsigned nonzero = __ballot_sync(0xffffffffu, w != 0.0);
    if (lane == 0) {
        rows[o].start = lo;
        rows[o].count = 32 - __clz(nonzero);
    }
}
static_assert(kVoxBand == 32, "a lane per weight");

// s + e += w v: the product's rounding error from one fma, the sum's from a two-sum.
__device__ __forceinline__ void vox_add(float2 w, float v, float &s, float &e) {
    const float p = __fmul_rn(w.x, v);
    float d;
    e = __fmaf_rn(w.y, v, __fadd_rn(e, __fmaf_rn(w.x, v, -p)));
    two_sum(s, p, s, d);
    e = __fadd_rn(e, d);
}

// What the pair s + e cannot hold (an infinity or NaN among the inputs, an overflow on the way) is summed
// again in FP64, without the taps of weight zero. A sum so small that its errors fall below the FP32 range
// stays: the logistic takes 1/2 from every sum, beside which it is nothing to FP64 either. (Summed again,
// a void of 1e-35 took 567 us where 16 x 64^3 -> 32^3 of ordinary values takes 52.)
__device__ __forceinline__ bool vox_plain(float s) { return fabsf(s) < 1e38f; }
static __device__ __noinline__ double vox_sum64(const VoxRow *R, const float *src, long long stride) {
    double acc = 0.0;
    for (int k = 0; k < R->count; ++k) {
        const double w = (double)R->w[k].x + (double)R->w[k].y;
        if (w != 0.0) acc += w * (double)src[k * stride];
    }
    return acc;
}

// The last axis: out[row][o] = sum_k A[o][k] in[row][start_o + k]. A block takes 32 outputs (the lanes)
// of 8 rows per warp: the weights, lane by lane different, are read from shared memory once for 8 rows.
// 15 us for 65536 rows of 64 -> 32: half the FP32 issue of its sums, half waiting for rows.
constexpr int kVoxNT = 256;
constexpr int kVoxRows = 8;
__global__ void __launch_bounds__(kVoxNT) vox_last_kernel(long long nrows, int n_in, int n_out,
                                                          const float *__restrict__ in,
                                                          const VoxRow *__restrict__ rows, float *__restrict__ out) {
    __shared__ float2 w[kVoxBand][33];
    __shared__ int2 span[32];
    const int tid = threadIdx.x, lane = tid & 31, o0 = 32 * blockIdx.y, no = min(32, n_out - o0);
    for (int i = tid; i < 32 * kVoxBand; i += kVoxNT) {
        const int l = i / kVoxBand, k = i - l * kVoxBand;
        w[k][l] = l < no ? rows[o0 + l].w[k] : make_float2(0.0f, 0.0f);
    }
    if (tid < 32) span[tid] = tid < no ? make_int2(rows[o0 + tid].start, rows[o0 + tid].count) : make_int2(0, 0);
    __syncthreads();
    const long long r0 = ((long long)blockIdx.x * (kVoxNT / 32) + (tid >> 5)) * kVoxRows;
    if (r0 >= nrows || lane >= no) return;
    const int nr = (int)min((long long)kVoxRows, nrows - r0);
    const int2 sp = span[lane];
    const float *src = in + r0 * n_in + sp.x;
    float s[kVoxRows], e[kVoxRows];
    const float *at[kVoxRows];
#pragma unroll
    for (int q = 0; q < kVoxRows; ++q) {
        s[q] = e[q] = 0.0f;
        at[q] = src + (q < nr ? q : 0) * n_in;
    }
#pragma unroll 2
    for (int k = 0; k < sp.y; ++k) {
        const float2 wk = w[k][lane];
#pragma unroll
        for (int q = 0; q < kVoxRows; ++q) vox_add(wk, at[q][k], s[q], e[q]);
    }
#pragma unroll
    for (int q = 0; q < kVoxRows; ++q)
        if (q < nr) {
            float v = s[q] + e[q];
            if (!vox_plain(v)) v = (float)vox_sum64(rows + o0 + lane, src + (long long)q * n_in, 1);
            out[(r0 + q) * n_out + o0 + lane] = v;
        }
}

// exp(z) for |z| < 88: z = k ln 2 + r, Taylor's series of r (|r| <= 0.35: degree 12 leaves 7e-15), its
// terms from the seventh on in FP32.
__device__ __forceinline__ df32 vox_exp(df32 z) {
    const float k = rintf(z.hi * 1.44269504f);
    const df32 r = df_add(z, df_neg(df_mul(df32{k, 0.0f}, df_from(0.69314718055994530942))));
    float t = 1.0f / 479001600.0f;
    t = fmaf(t, r.hi, 1.0f / 39916800.0f);
    t = fmaf(t, r.hi, 1.0f / 3628800.0f);
    t = fmaf(t, r.hi, 1.0f / 362880.0f);
    t = fmaf(t, r.hi, 1.0f / 40320.0f);
    t = fmaf(t, r.hi, 1.0f / 5040.0f);
    df32 v{t, 0.0f};
    v = df_add(df_mul(v, r), df_from(1.0 / 720.0));
    v = df_add(df_mul(v, r), df_from(1.0 / 120.0));
    v = df_add(df_mul(v, r), df_from(1.0 / 24.0));
    v = df_add(df_mul(v, r), df_from(1.0 / 6.0));
    v = df_add(df_mul(v, r), df32{0.5f, 0.0f});
    v = df_add(df_mul(v, r), df32{1.0f, 0.0f});
    v = df_add(df_mul(v, r), df32{1.0f, 0.0f});
    const float scale = __int_as_float(((int)k + 127) << 23);
    return df32{v.hi * scale, v.lo * scale};
}
static __device__ __noinline__ float vox_logistic64(double v, double sharpness) {
    return (float)(1.0 / (1.0 + exp(-sharpness * (v - 0.5))));
}

// Another axis: out[a][o][c] = sum_k A[o][k] in[a][start_o + k][c], `outer` planes a (grid y), `inner`
// trailing extent, a thread per output. Bound by the latency of its loads (16 x 64 x 32 x 32 outputs
// 13 us, of which 4 are the sums' FP32 issue); four planes per thread took 21, twelve taps in flight 15. The
// last of the passes applies the logistic, double-float too: an FP64 exponential and division per output
// took as long as the sums.
template <bool kLogistic>
__global__ void __launch_bounds__(kVoxNT) vox_pass_kernel(long long outer, int n_in, int n_out, int inner, FastDiv fin,
                                                          const float *__restrict__ in,
                                                          const VoxRow *__restrict__ rows, float *__restrict__ out,
                                                          double sharpness, df32 sharp) {
    const int id = blockIdx.x * kVoxNT + threadIdx.x;
    if (id >= n_out * inner) return;
    const int o = (int)fdiv((uint32_t)id, fin), c = id - o * inner;
    const VoxRow &R = rows[o];
    const int start = R.start, count = R.count;
    for (long long a = blockIdx.y; a < outer; a += gridDim.y) {
        const float *src = in + (a * n_in + start) * inner + c;
        float s = 0.0f, e = 0.0f;
#pragma unroll 4
        for (int k = 0; k < count; ++k) vox_add(R.w[k], src[(long long)k * inner], s, e);
        float v = s + e;
        const bool plain = vox_plain(v);
        if (kLogistic) {
            const df32 y = df_mul(sharp, df_add(df_renorm(s, e), df32{-0.5f, 0.0f}));
            if (plain && fabsf(y.hi) < 80.0f) {
                const df32 l = df_div(df32{1.0f, 0.0f}, df_add(df32{1.0f, 0.0f}, vox_exp(df_neg(y))));
                v = l.hi + l.lo;
            } else {
                v = vox_logistic64(plain ? (double)s + (double)e : vox_sum64(&R, src, inner), sharpness);
            }
        } else if (!plain) {
            v = (float)vox_sum64(&R, src, inner);
        }
        out[a * n_out * inner + id] = v;
    }
}

static bool vox_dims_ok(int n_in, int n_out) {
    return n_in >= 1 && n_in <= kVoxMaxExtent && n_out >= 1 && n_out <= kVoxMaxExtent && (n_out >= 2 || n_in == 1);
}

static size_t vox_ws_bytes_impl(int batch, int D, int H, int W, int d, int h, int w) {
    return 256 + al256v(sizeof(VoxRow) * ((size_t)d + h + w)) + al256v(4 * (size_t)batch * D * H * w) +
           al256v(4 * (size_t)batch * D * h * w);
}

}  // namespace gbs

using namespace gbs;

extern "C" size_t gbsimp_voxel_prep_ws_bytes(int batch, int D, int H, int W, int d, int h, int w) {
    if (batch <= 0 || !vox_dims_ok(D, d) || !vox_dims_ok(H, h) || !vox_dims_ok(W, w)) return 0;
    return vox_ws_bytes_impl(batch, D, H, W, d, h, w);
}

extern "C" int gbsimp_voxel_prep(gbsimp_ctx *ctx, int batch, int D, int H, int W, const float *in, int d, int h,
                                 int w, float *out, double sigma, double sharpness, void *ws, size_t ws_bytes,
                                 void *stream) {
    if (!ctx || !in || !out || !ws || batch <= 0 || !vox_dims_ok(D, d) || !vox_dims_ok(H, h) ||
        !vox_dims_ok(W, w) || !(sigma >= 0.0) || !(sigma <= 64.0) || !isfinite(sharpness))
        return set_error(GBS_EINVAL, "gbsimp_voxel_prep: bad arguments");
    if (vox_span(D, d, sigma) > kVoxBand || vox_span(H, h, sigma) > kVoxBand || vox_span(W, w, sigma) > kVoxBand)
        return set_error(GBS_EINVAL, "gbsimp_voxel_prep: sigma %g with this zoom needs more than %d taps per row",
                         sigma, kVoxBand);
    if (ws_bytes < vox_ws_bytes_impl(batch, D, H, W, d, h, w))
        return set_error(GBS_EINVAL, "gbsimp_voxel_prep: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    char *p = (char *)(((uintptr_t)ws + 255) & ~(uintptr_t)255);
    VoxRow *rx = (VoxRow *)p, *ry = rx + d, *rz = ry + h;
    p += al256v(sizeof(VoxRow) * ((size_t)d + h + w));
    float *t1 = (float *)p;  // (batch, D, H, w)
    p += al256v(4 * (size_t)batch * D * H * w);
    float *t2 = (float *)p;  // (batch, D, h, w)
    const int most = d > h ? (d > w ? d : w) : (h > w ? h : w);
    const VoxAxes ax{{D, H, W}, {d, h, w}};
    vox_table_kernel<<<dim3((unsigned)((most + kVoxTableNT / 32 - 1) / (kVoxTableNT / 32)), 3), kVoxTableNT, 0, st>>>(ax, sigma, rx);
    GBS_LAUNCH_CHECK("vox_table_kernel");
    const long long B = batch, nrows = B * D * H, per = (kVoxNT / 32) * kVoxRows;
    vox_last_kernel<<<dim3((unsigned)((nrows + per - 1) / per), (unsigned)((w + 31) / 32)), kVoxNT, 0, st>>>(
        nrows, W, w, in, rz, t1);
    GBS_LAUNCH_CHECK("vox_last_kernel");
    auto grid = [](int n, long long outer) {
        return dim3((unsigned)((n + kVoxNT - 1) / kVoxNT), (unsigned)(outer < 65535 ? outer : 65535));
    };
    const df32 sharp = df_from(sharpness);
    const int plane = h * w;
    vox_pass_kernel<false><<<grid(plane, B * D), kVoxNT, 0, st>>>(B * D, H, h, w, fast_div((uint32_t)w), t1, ry, t2,
                                                                   0.0, df32{0.0f, 0.0f});
    GBS_LAUNCH_CHECK("vox_pass_kernel");
    vox_pass_kernel<true><<<grid(d * plane, B), kVoxNT, 0, st>>>(B, D, d, plane, fast_div((uint32_t)plane), t2,
                                                                     rx, out, sharpness, sharp);
    GBS_LAUNCH_CHECK("vox_pass_kernel");
    return GBS_OK;
}
