// elem.cu -- element-wise kernels: sensitivity/compliance, density filter, OC bisection,
// FP64 dot. All reductions: per-block partials (FP64; double-float in the OC multisection),
// summed in a fixed order by the last block to finish (deterministic for a given launch
// shape).
#include <math.h>
#include <string.h>

#include <atomic>

#include "internal.h"
#include "modal_dd.cuh"

namespace gbs {

// ---- last-block reduction helper -----------------------------------------------------
// Every block calls it with its partial(s); returns true in the last block, whose threads
// then see the K sums of all partials in out[0..K-1] (shared). counter is reset.
template <int K>
__device__ bool last_block_reduce(const double (&v)[K], double *partials, unsigned *counter, double *out,
                                  double *sred) {
    __shared__ bool last;
    const int nblk = gridDim.x;
    double bs[K];
#pragma unroll
    for (int k = 0; k < K; ++k) bs[k] = block_sum(v[k], sred);
    if (threadIdx.x == 0) {
#pragma unroll
        for (int k = 0; k < K; ++k) partials[k * nblk + blockIdx.x] = bs[k];
        __threadfence();
        last = (atomicAdd(counter, 1u) == (unsigned)(nblk - 1));
    }
    __syncthreads();
    if (!last) return false;
    __threadfence();
#pragma unroll
    for (int k = 0; k < K; ++k) {
        double s = 0.0;
        for (int i = threadIdx.x; i < nblk; i += blockDim.x) s += ((volatile double *)partials)[k * nblk + i];
        s = block_sum(s, sred);
        if (threadIdx.x == 0) out[k] = s;
    }
    __syncthreads();
    if (threadIdx.x == 0) *counter = 0;
    return true;
}

inline unsigned reduce_blocks(const gbsimp_ctx *ctx, int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = 4LL * (ctx->num_sms > 0 ? ctx->num_sms : 148);
    if (b > cap) b = cap;
    if (b < 1) b = 1;
    return (unsigned)b;
}

// ---- sensitivity ------------------------------------------------------------------------
// Thread per element: u_e gathered in FP64; ce = u_e^T Ke u_e through the modal form
// (q = T^T u_e, the 45 nonzeros of Km) when Ke has it, else the dense product (minus node 0's
// displacement when Ke annihilates translations); dc = -dE/dx ce, energy partial E ce.
__global__ void __launch_bounds__(128) sens_kernel(int nx, int ny, int nz, Law<double> law, const KeD ke, int sub,
                                                   int modal, const ModalKD kmd,
                                                   const float *__restrict__ x, const double *__restrict__ u,
                                                   float *dc, float *ce_out, double *partials, unsigned *counter,
                                                   double *energy_out) {
    __shared__ double sred[32];
    __shared__ double tot[1];
    const int64_t n_elem = (int64_t)nx * ny * nz;
    const int64_t NY = ny + 1, NZ = nz + 1;
    double part = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_elem; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / ((int64_t)ny * nz)), j = (int)((e / nz) % ny), k = (int)(e % nz);
        double ue[24];
#pragma unroll
        for (int b = 0; b < 8; ++b) {
            const int64_t m = ((int64_t)(i + corner_x(b)) * NY + (j + corner_y(b))) * NZ + (k + corner_z(b));
#pragma unroll
            for (int c = 0; c < 3; ++c) ue[3 * b + c] = u[3 * m + c];
        }
        double s = 0.0;
        if (modal) {
            // ce = q^T Km q with q = T^T u_e (Walsh-Hadamard of the corner values): the
            // translation modes drop out exactly and only the 45 nonzeros of Km are used.
            double q[8][3];
#pragma unroll
            for (int a = 0; a < 8; ++a) {
                const int b = corner_x(a) * 4 + corner_y(a) * 2 + corner_z(a);
#pragma unroll
                for (int c = 0; c < 3; ++c) q[b][c] = ue[3 * a + c];
            }
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int bit = 1 << d;
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    if (b & bit) continue;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double u0 = q[b][c], u1 = q[b | bit][c];
                        q[b][c] = u0 + u1;
                        q[b | bit][c] = u1 - u0;
                    }
                }
            }
#pragma unroll
            for (int t = 0; t < kModalNnz; ++t) {
                const int ro = modal_row(t), co = modal_col(t);
                s = fma(kmd.v[t] * q[ro / 3][ro % 3], q[co / 3][co % 3], s);
            }
        } else {
            if (sub) {
                const double c0 = ue[0], c1 = ue[1], c2 = ue[2];
#pragma unroll
                for (int b = 0; b < 8; ++b) {
                    ue[3 * b] -= c0;
                    ue[3 * b + 1] -= c1;
                    ue[3 * b + 2] -= c2;
                }
            }
#pragma unroll
            for (int r = 0; r < 24; ++r) {
                double t = 0.0;
#pragma unroll
                for (int q = 0; q < 24; ++q) t = fma(ke.k[r * 24 + q], ue[q], t);
                s = fma(ue[r], t, s);
            }
        }
        const double xe = (double)x[e];
        if (dc) dc[e] = (float)(-dmodulus(law, xe) * s);
        if (ce_out) ce_out[e] = (float)s;
        part += modulus(law, xe) * s;
    }
    if (energy_out) {
        const double v[1] = {part};
        if (last_block_reduce<1>(v, partials, counter, tot, sred) && threadIdx.x == 0) *energy_out = tot[0];
    }
}

// The same through the double-float modal form (modal_dd.cuh), from the split displacements:
// ce = q^T Km q accumulated in double-float, then dc, ce and the energy partial as above.
__global__ void __launch_bounds__(128) sens_dd_kernel(int nx, int ny, int nz, Law<double> law, const ModalKDD km,
                                                      const FastDiv fy, const FastDiv fz,
                                                      const float *__restrict__ x, const float2 *__restrict__ udd,
                                                      float *dc, float *ce_out, double *partials, unsigned *counter,
                                                      double *energy_out) {
    __shared__ double sred[32];
    __shared__ double tot[1];
    const int64_t n_elem = (int64_t)nx * ny * nz;
    double part = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_elem; e += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        unflatten3((uint32_t)e, fy, fz, i, j, k);
        ddv q[8][3], r[8][3];
        modal_fwd_dd(ny, nz, i, j, k, udd, q);
        modal_km_dd(km, q, r);
        ddv s{0.0f, 0.0f};
#pragma unroll
        for (int m = 1; m < 8; ++m)
#pragma unroll
            for (int c = 0; c < 3; ++c) s = dd_add(s, dd_mul(q[m][c].h, q[m][c].l, r[m][c]));
        const double ce = dd_value(s);
        const double xe = (double)x[e];
        if (dc) dc[e] = (float)(-dmodulus(law, xe) * ce);
        if (ce_out) ce_out[e] = (float)ce;
        part += modulus(law, xe) * ce;
    }
    if (energy_out) {
        const double v[1] = {part};
        if (last_block_reduce<1>(v, partials, counter, tot, sred) && threadIdx.x == 0) *energy_out = tot[0];
    }
}

// ---- density filter ---------------------------------------------------------------------
constexpr int kMaxStencil = 1024;
struct Stencil {
    int n;
    int r;
    int flat;              // 1: doff[] holds the flat offsets of this grid
    int off[kMaxStencil];  // dx, dy, dz packed as signed bytes
    float w[kMaxStencil];  // rmin - dist > 0
    int doff[kMaxStencil]; // (dx ny + dy) nz + dz: the element offset in x-y-z order
};

// The neighbourhood of simp_solver.py:1553-1565: offsets of the box of half-width
// ceil(rmin) with dist <= rmin; zero weights (dist == rmin) are dropped (they add nothing).
static int make_stencil(double rmin, Stencil *s) {
    if (!(rmin > 0.0) || rmin > 6.0) return set_error(GBS_EINVAL, "filter: rmin must be in (0, 6], got %g", rmin);
    const int r = (int)ceil(rmin);
    s->n = 0;
    s->r = r;
    s->flat = 0;
    for (int di = -r; di <= r; ++di)
        for (int dj = -r; dj <= r; ++dj)
            for (int dk = -r; dk <= r; ++dk) {
                const double d = sqrt((double)(di * di + dj * dj + dk * dk));
                if (d > rmin) continue;
                const double w = rmin - d;
                if (!(w > 0.0)) continue;
                if (s->n >= kMaxStencil) return set_error(GBS_EINVAL, "filter: stencil too large");
                s->off[s->n] = (int)(((unsigned)(uint8_t)(int8_t)di) | ((unsigned)(uint8_t)(int8_t)dj << 8) |
                                     ((unsigned)(uint8_t)(int8_t)dk << 16));
                s->w[s->n] = (float)w;
                ++s->n;
            }
    return GBS_OK;
}

// The flat element offsets of the stencil for a grid of ny x nz element rows, when every
// one fits in an int (s->flat = 1; otherwise the kernel uses the bounds-checked path only).
static void set_flat_offsets(int ny, int nz, Stencil *s) {
    const int64_t reach = (int64_t)s->r * ((int64_t)ny * nz + nz + 1);
    s->flat = reach < INT32_MAX ? 1 : 0;
    if (!s->flat) return;
    for (int q = 0; q < s->n; ++q) {
        const int o = s->off[q];
        const int di = (int)(int8_t)(o & 0xff), dj = (int)(int8_t)((o >> 8) & 0xff), dk = (int)(int8_t)((o >> 16) & 0xff);
        s->doff[q] = (int)(((int64_t)di * ny + dj) * nz + dk);
    }
}

__device__ __forceinline__ void neumaier_add(float &s, float &c, float v) {
    const float t = s + v;
    c += fabsf(s) >= fabsf(v) ? (s - t) + v : (v - t) + s;
    s = t;
}

__device__ __forceinline__ void unpack_off(int o, int &di, int &dj, int &dk) {
    di = (int)(int8_t)(o & 0xff);
    dj = (int)(int8_t)((o >> 8) & 0xff);
    dk = (int)(int8_t)((o >> 16) & 0xff);
}

// The stencil as columns along z, sorted by their half-extent h: weights w[0..h] of |dz|.
constexpr int kFilterR = 5;  // rmin <= 6, and a weight at distance 6 is zero
constexpr int kFilterCols = (2 * kFilterR + 1) * (2 * kFilterR + 1);
struct FilterCols {
    int start[kFilterR + 2];  // columns of half-extent h: start[h] .. start[h + 1] - 1
    short di[kFilterCols], dj[kFilterCols];
    float w[kFilterCols][kFilterR + 1];
};
static int filter_columns(const Stencil &st, FilterCols *F) {
    int half[2 * kFilterR + 1][2 * kFilterR + 1], R = 0, n = 0;
    float w[2 * kFilterR + 1][2 * kFilterR + 1][kFilterR + 1] = {};
    for (auto &row : half)
        for (int &h : row) h = -1;
    for (int q = 0; q < st.n; ++q) {
        const int di = (int8_t)(st.off[q] & 0xff), dj = (int8_t)((st.off[q] >> 8) & 0xff);
        const int dk = abs((int8_t)((st.off[q] >> 16) & 0xff));
        int &h = half[di + kFilterR][dj + kFilterR];
        h = dk > h ? dk : h;
        w[di + kFilterR][dj + kFilterR][dk] = st.w[q];
        R = std::max(R, std::max(abs(di), std::max(abs(dj), dk)));
    }
    memset(F, 0, sizeof *F);
    for (int h = 0; h <= kFilterR; ++h) {
        F->start[h] = n;
        if (h > R) continue;
        for (int i = kFilterR - R; i <= kFilterR + R; ++i)
            for (int j = kFilterR - R; j <= kFilterR + R; ++j) {
                if (half[i][j] != h) continue;
                F->di[n] = (short)(i - kFilterR);
                F->dj[n] = (short)(j - kFilterR);
                memcpy(F->w[n], w[i][j], sizeof F->w[n]);
                ++n;
            }
    }
    F->start[kFilterR + 1] = n;
    return R;
}

// A block's tile of outputs: ti x tj rows of kt threads, four elements along z each.
struct FilterTile {
    int ti, tj, kt, nbj, nbk;
    FastDiv fk, fj;  // by the tile's words per row and rows per plane, margins included
};

// s + c += the columns of half-extent H and above of the four elements whose window starts at t.
template <int R, int H>
__device__ __forceinline__ void filter_cols(const FilterCols &F, const float *t, int SJ, int SK, float (&s)[4],
                                            float (&c)[4]) {
#pragma unroll 1
    for (int q = F.start[H]; q < F.start[H + 1]; ++q) {
        constexpr int lo = (R - H) & ~3, n4 = (R + H + 4 - lo + 3) / 4;
        const float4 *row = (const float4 *)(t + (F.di[q] * SJ + F.dj[q]) * SK + lo);
        float v[4 * n4];
#pragma unroll
        for (int i = 0; i < n4; ++i) {
            const float4 x = row[i];
            v[4 * i] = x.x;
            v[4 * i + 1] = x.y;
            v[4 * i + 2] = x.z;
            v[4 * i + 3] = x.w;
        }
#pragma unroll
        for (int d = -H; d <= H; ++d) {
            const float w = F.w[q][d < 0 ? -d : d];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                float e;
                two_sum(s[m], __fmul_rn(w, v[m + R + d - lo]), s[m], e);
                c[m] += e;
            }
        }
    }
    if constexpr (H < R) filter_cols<R, H + 1>(F, t, SJ, SK, s, c);
}

// mode 0: out = (sum w v) / hs[e] (hs nullable: computed);  mode 1: out = sum w v/hs[e2];
// mode 2 (hs): out = sum w over in-bounds neighbours. preserved (mode 0): out = 1 there.
// A tap at a time, an element per thread, for small work (filter_tiled): nothing to load first, and a
// tap outside the grid costs its test only. FP32 products summed with their rounding errors (a few ulp
// whatever the stencil, up to ~900 terms at rmin 6).
__global__ void __launch_bounds__(256) filter_taps_kernel(int nx, int ny, int nz, const FastDiv fy, const FastDiv fz,
                                                     const Stencil st, int mode,
                                                     const float *__restrict__ hs, const float *__restrict__ in,
                                                     const uint8_t *__restrict__ preserved, float *out) {
    const int64_t n_elem = (int64_t)nx * ny * nz;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_elem; e += (int64_t)gridDim.x * blockDim.x) {
        int i, j, k;
        unflatten3((uint32_t)e, fy, fz, i, j, k);
        // FP32 with compensated (Neumaier) summation in the fixed stencil order: error of a
        // few ulp whatever the stencil size (up to ~900 terms at rmin 6).
        float s = 0.0f, sc = 0.0f, ws = 0.0f, wc = 0.0f;
        // Away from the x and y faces only z can leave the grid: the same terms in the same
        // order, with one z test and a precomputed flat offset per term (a warp's elements
        // lie in one or two z columns, so the branch rarely splits a warp).
        if (st.flat && i >= st.r && i < nx - st.r && j >= st.r && j < ny - st.r) {
            for (int q = 0; q < st.n; ++q) {
                const int k2 = k + (int)(int8_t)((st.off[q] >> 16) & 0xff);
                if (k2 < 0 || k2 >= nz) continue;
                const int64_t e2 = e + st.doff[q];
                const float w = st.w[q];
                neumaier_add(ws, wc, w);
                if (mode == 0) neumaier_add(s, sc, w * in[e2]);
                else if (mode == 1) neumaier_add(s, sc, w * (in[e2] / hs[e2]));
            }
        } else {
            for (int q = 0; q < st.n; ++q) {
                int di, dj, dk;
                unpack_off(st.off[q], di, dj, dk);
                const int i2 = i + di, j2 = j + dj, k2 = k + dk;
                if (i2 < 0 || i2 >= nx || j2 < 0 || j2 >= ny || k2 < 0 || k2 >= nz) continue;
                const int64_t e2 = ((int64_t)i2 * ny + j2) * nz + k2;
                const float w = st.w[q];
                neumaier_add(ws, wc, w);
                if (mode == 0) neumaier_add(s, sc, w * in[e2]);
                else if (mode == 1) neumaier_add(s, sc, w * (in[e2] / hs[e2]));
            }
        }
        s += sc;
        ws += wc;
        float o;
        if (mode == 0) {
            const float h = hs ? hs[e] : ws;
            o = s / h;
            if (preserved && preserved[e]) o = 1.0f;
        } else if (mode == 1) {
            o = (float)s;
        } else {
            o = (float)ws;
        }
        out[e] = o;
    }
}

// The same from a tile. FP32 products summed with their rounding errors. Bound by FP32 issue, eight
// operations per tap. v, v/hs or one (zero outside the grid) of the tile and its margin R goes to shared
// memory once, and a thread takes four elements along z, so that a column of taps costs it two or three
// 16-byte loads: 192x96x96 takes 58 us with rmin 3 where a tap at a time takes 173 (device time; rmin
// 1.5: 22 for 41). The tile's words are dealt to the threads one by one, eight loads in flight each; a warp
// per row left most lanes idle where rows are short and took 11.0 us at 32x8x8 with rmin 1.5, 5.4 so.
// Plain FP32 sums along a column would take a third of the operations, but moved the compliance of a
// twelve-step SIMP run at 20x8x8 by 7e-6.
template <int R>
__global__ void __launch_bounds__(256) filter_kernel(int nx, int ny, int nz, const __grid_constant__ FilterTile T,
                                                     const __grid_constant__ FilterCols F, int mode,
                                                     const float *__restrict__ hs, const float *__restrict__ in,
                                                     const uint8_t *__restrict__ preserved, float *__restrict__ out) {
    extern __shared__ float4 tile4[];
    float *tile = (float *)tile4;
    const int SK = (4 * T.kt + 2 * R + 3) & ~3, SJ = T.tj + 2 * R, rows = (T.ti + 2 * R) * SJ;
    const int bk = blockIdx.x % T.nbk, bij = blockIdx.x / T.nbk, bj = bij % T.nbj, bi = bij / T.nbj;
    const int i0 = bi * T.ti, j0 = bj * T.tj, k0 = bk * 4 * T.kt;
    const int tid = threadIdx.x, kt = tid % T.kt, ij = tid / T.kt, jl = ij % T.tj, il = ij / T.tj;
    float s[4], c[4], h[4] = {1.0f, 1.0f, 1.0f, 1.0f};
    const bool own = mode == 0 && hs == nullptr;  // the sums of weights first
    for (int pass = own ? 0 : 1; pass < 2; ++pass) {
        const bool ones = mode == 2 || pass == 0;
#pragma unroll 8
        for (int q = tid; q < rows * SK; q += blockDim.x) {
            const int r = (int)fdiv((uint32_t)q, T.fk), a = (int)fdiv((uint32_t)r, T.fj);
            const int i = i0 + a - R, j = j0 + (r - a * SJ) - R, k = k0 + (q - r * SK) - R;
            float v = 0.0f;
            if (i >= 0 && i < nx && j >= 0 && j < ny && k >= 0 && k < nz) {
                const int64_t e = ((int64_t)i * ny + j) * nz + k;
                if (ones) v = 1.0f;
                else if (mode == 1) v = in[e] / hs[e];
                else v = in[e];
            }
            tile[q] = v;
        }
        __syncthreads();
#pragma unroll
        for (int m = 0; m < 4; ++m) s[m] = c[m] = 0.0f;
        filter_cols<R, 0>(F, tile + ((il + R) * SJ + jl + R) * SK + 4 * kt, SJ, SK, s, c);
        if (pass == 0) {
#pragma unroll
            for (int m = 0; m < 4; ++m) h[m] = s[m] + c[m];
            __syncthreads();
        }
    }
    const int i = i0 + il, j = j0 + jl, k = k0 + 4 * kt;
    if (i >= nx || j >= ny || k >= nz) return;
    const int64_t e = ((int64_t)i * ny + j) * nz + k;
    float o[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        o[m] = s[m] + c[m];
        if (mode == 0 && k + m < nz) {
            o[m] = o[m] / (own ? h[m] : hs[e + m]);
            if (preserved && preserved[e + m]) o[m] = 1.0f;
        }
    }
    if ((nz & 3) == 0 && ((uintptr_t)out & 15) == 0) {
        *(float4 *)(out + e) = make_float4(o[0], o[1], o[2], o[3]);
    } else {
#pragma unroll
        for (int m = 0; m < 4; ++m)
            if (k + m < nz) out[e + m] = o[m];
    }
}

static unsigned elem_blocks(const gbsimp_ctx *ctx, int64_t n, int threads) {
    int64_t b = (n + threads - 1) / threads;
    const int64_t cap = 32LL * (ctx->num_sms > 0 ? ctx->num_sms : 148);
    if (b > cap) b = cap;
    return (unsigned)(b < 1 ? 1 : b);
}

// The tile: 4 kt elements along z (kt a power of two up to 8 that covers nz), then the split of the
// rows of 256, 128 or 64 threads with the fewest elements to load; the smaller blocks only where the
// larger would leave SMs without one.
static FilterTile filter_tile(const gbsimp_ctx *ctx, int nx, int ny, int nz, int R, int *threads) {
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    FilterTile T{1, 1, 1, 1, 1, {}, {}};
    while (T.kt < 8 && 4 * T.kt < nz) T.kt *= 2;
    T.nbk = up(nz, 4 * T.kt);
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 148;
    for (int nt = 256; nt >= 64; nt /= 2) {
        double best = 1e300;
        for (int ti = 1; ti <= nt / T.kt; ti *= 2) {
            const int tj = nt / T.kt / ti;
            const double rows = (double)(ti + 2 * R) * (tj + 2 * R);
            const double load = rows * up(nx, ti) * up(ny, tj);
            if (rows * ((4 * T.kt + 2 * R + 3) & ~3) * 4 > 48 * 1024 || load >= best) continue;
            best = load;
            T.ti = ti;
            T.tj = tj;
        }
        *threads = nt;
        T.nbj = up(ny, T.tj);
        if ((int64_t)up(nx, T.ti) * T.nbj * T.nbk >= sms) break;
    }
    T.fk = fast_div((uint32_t)((4 * T.kt + 2 * R + 3) & ~3));
    T.fj = fast_div((uint32_t)(T.tj + 2 * R));
    return T;
}

// Whether the tiled kernel takes the call. Device times, a tap at a time -> tiled, at the lines: seven
// taps (rmin up to sqrt 2) 48^3 3.7 -> 5.2 us, 256x256x100 67 -> 81; 19 taps 32^3 5.0 -> 6.2, 33^3
// 6.4 -> 5.8, 32x8x8 6.6 -> 5.4 but 3x60x60 5.1 -> 6.6; 81 taps 32^3 13.6 -> 12.0, 1x64x64 7.8 -> 9.5,
// 1x450x450 20.5 -> 13.0, 1x1x200000 17 -> 164 (the columns beyond the grid are all zeros); 93 taps
// 450x450x1 27 -> 34 (three of a thread's four elements lie outside); 485 taps
// 1x450x450 98 -> 61, 739 taps 146 -> 170.
// With the sums of weights to form as well (own), which the tile does one after the other: 81 taps 32^3
// 13.5 -> 17.7, 33^3 21.0 -> 16.0, 19 taps 64^3 9.4 -> 8.9, 256x256x100 142 -> 153, 895 taps 2x300x300
// 171 -> 207.
static bool filter_tiled(int nx, int ny, int nz, int taps, bool own) {
    const int64_t n = (int64_t)nx * ny * nz;
    const int lo = std::min(nx, std::min(ny, nz)), hi = std::max(nx, std::max(ny, nz));
    if (taps <= 7) return false;
    if (lo == 1) return !own && taps >= 60 && taps < 600 && n >= 100000 && n / hi >= 32 && nz >= 32;
    if (own) return taps >= 60 && n > 33000 && lo > 2;
    return taps >= 60 || n > 33000 || (nz < 16 && lo > 3);
}

int filter_launch(const gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, int mode, const float *hs,
                  const float *in, const uint8_t *preserved, float *out, cudaStream_t st) {
    Stencil s;
    int rc = make_stencil(rmin, &s);
    if (rc) return rc;
    if (!filter_tiled(nx, ny, nz, s.n, mode == 0 && !hs)) {
        const int64_t n = (int64_t)nx * ny * nz;
        set_flat_offsets(ny, nz, &s);
        filter_taps_kernel<<<elem_blocks(ctx, n, 256), 256, 0, st>>>(nx, ny, nz, fast_div(ny), fast_div(nz), s, mode, hs,
                                                                     in, preserved, out);
        GBS_LAUNCH_CHECK("filter_taps_kernel");
        return GBS_OK;
    }
    FilterCols F;
    const int R = filter_columns(s, &F);
    int nt = 256;
    const FilterTile T = filter_tile(ctx, nx, ny, nz, R, &nt);
    const unsigned blocks = (unsigned)(((nx + T.ti - 1) / T.ti) * T.nbj * T.nbk);
    const size_t smem = sizeof(float) * (size_t)(T.ti + 2 * R) * (T.tj + 2 * R) * ((4 * T.kt + 2 * R + 3) & ~3);
    static void (*const kern[])(int, int, int, FilterTile, FilterCols, int, const float *, const float *,
                                const uint8_t *, float *) = {filter_kernel<1>, filter_kernel<2>, filter_kernel<3>,
                                                             filter_kernel<4>, filter_kernel<5>};
    kern[R - 1]<<<blocks, nt, smem, st>>>(nx, ny, nz, T, F, mode, hs, in, preserved, out);
    GBS_LAUNCH_CHECK("filter_kernel");
    return GBS_OK;
}

// ---- OC bisection -----------------------------------------------------------------------
struct OcScalars {
    double l1, l2, lfinal, npres;
    int steps, done;
    unsigned counter;
    int status;  // GBS_ETIMEOUT when a wait of oc_coop_kernel ran out
};

struct OcParams {
    float move, sqrt_floor;
    double tol, tol_eps, volfrac, l1, l2;
    int max_bisect;
};

// Workspace: [OcScalars (256 B)] [hs: n floats] [w: n floats] [partials: kOcPartials bytes]
constexpr size_t kOcPartials = 4 * 4096 * sizeof(double) + 65536;
struct OcWs {
    OcScalars *sc;
    float *hs, *w;
    double *partials;
};

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

static size_t oc_ws_bytes(int64_t n) {
    return 256 + 2 * align256((size_t)n * sizeof(float)) + align256(kOcPartials);
}

static OcWs oc_ws(void *ws, int64_t n) {
    char *p = (char *)ws;
    OcWs w;
    w.sc = (OcScalars *)p;
    p += 256;
    w.hs = (float *)p;
    p += align256((size_t)n * sizeof(float));
    w.w = (float *)p;
    p += align256((size_t)n * sizeof(float));
    w.partials = (double *)p;
    return w;
}

// w_e = sum_{e1 in ball(e), e1 not preserved} H[e1,e] / Hs[e1];  npres = #preserved.
__global__ void oc_weights_kernel(int nx, int ny, int nz, const Stencil st, const float *__restrict__ hs,
                                  const uint8_t *__restrict__ preserved, float *w, double *partials, OcScalars *sc) {
    __shared__ double sred[32];
    __shared__ double tot[1];
    const int64_t n_elem = (int64_t)nx * ny * nz;
    double np = 0.0;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n_elem; e += (int64_t)gridDim.x * blockDim.x) {
        const int i = (int)(e / ((int64_t)ny * nz)), j = (int)((e / nz) % ny), k = (int)(e % nz);
        double s = 0.0;
        for (int q = 0; q < st.n; ++q) {
            int di, dj, dk;
            unpack_off(st.off[q], di, dj, dk);
            const int i2 = i + di, j2 = j + dj, k2 = k + dk;
            if (i2 < 0 || i2 >= nx || j2 < 0 || j2 >= ny || k2 < 0 || k2 >= nz) continue;
            const int64_t e2 = ((int64_t)i2 * ny + j2) * nz + k2;
            if (preserved && preserved[e2]) continue;
            s += (double)st.w[q] / (double)hs[e2];
        }
        w[e] = (float)s;
        if (preserved && preserved[e]) np += 1.0;
    }
    const double v[1] = {np};
    if (last_block_reduce<1>(v, partials, &sc->counter, tot, sred) && threadIdx.x == 0) sc->npres = tot[0];
}

__device__ __forceinline__ float oc_trial(float x, float dc, float inv_l, const OcParams &P, bool pres) {
    float t = -dc * inv_l;
    t = t > P.sqrt_floor ? t : P.sqrt_floor;
    float v = x * sqrtf(t);
    v = v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);
    const float lo = x - P.move, hi = x + P.move;
    v = v < lo ? lo : v;
    v = v > hi ? hi : v;
    return pres ? 1.0f : v;
}

__global__ void oc_init_kernel(int64_t n, const OcParams P, const float *__restrict__ dc, double *partials,
                               OcScalars *sc, uint4 *box, int packets) {
    sc->done = 0;  // every block writes the same values
    sc->steps = 0;
    sc->status = 0;
    // oc_coop_kernel's packets: none may carry an epoch of the rounds to come
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < packets; i += gridDim.x * blockDim.x)
        box[i] = make_uint4(0, 0, 0, 0);
    if (P.l2 >= 0.0) {
        if (blockIdx.x == 0 && threadIdx.x == 0) {
            sc->l1 = P.l1;
            sc->l2 = P.l2;
            sc->lfinal = 0.5 * (P.l1 + P.l2);
        }
        return;
    }
    // l2 = 2 * max(max(-dc), 1)  (simp_solver_gpu.py:813); max via a sum of per-block maxima
    // would lose the max, so partials carry maxima and the last block takes their max.
    float m = -INFINITY;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        m = fmaxf(m, -dc[e]);
    m = warp_max(m);
    __shared__ float wm[32];
    __shared__ bool last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (lane == 0) wm[wid] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        float b = -INFINITY;
        for (int i = 0; i < (int)((blockDim.x + 31) >> 5); ++i) b = fmaxf(b, wm[i]);
        partials[blockIdx.x] = (double)b;
        __threadfence();
        last = (atomicAdd(&sc->counter, 1u) == gridDim.x - 1);
    }
    __syncthreads();
    if (last && threadIdx.x == 0) {
        __threadfence();
        double mm = -INFINITY;
        for (unsigned i = 0; i < gridDim.x; ++i) mm = fmax(mm, ((volatile double *)partials)[i]);
        sc->counter = 0;
        sc->l1 = P.l1;
        sc->l2 = 2.0 * (mm > 1.0 ? mm : 1.0);
        sc->lfinal = 0.5 * (sc->l1 + sc->l2);
    }
}

// ---- multisection: kOcLevels bisection steps per launch ---------------------------------
// The bisection of simp_solver.py:229-247 visits one midpoint per step. One launch evaluates
// the volume at every midpoint the next kOcLevels steps could visit: the 2^kOcLevels - 1 nodes
// of the binary tree below (l1, l2), heap-ordered (node t: children 2t + 1 = [lo, mid] and
// 2t + 2 = [mid, hi]), each midpoint formed as bisection forms it, 0.5 (hi + lo) of its
// parent interval. The last block then walks the tree with bisection's tests (stop on
// (l2 - l1) / (l1 + l2 + eps) < tol, then vol > volfrac -> l1 = mid, else l2 = mid), so the
// sequence of intervals, lfinal and the step count are those of one launch per step (up to
// the rounding of the volume sums), in max_bisect / kOcLevels launches.
constexpr int kOcLevels = 5;
constexpr int kOcNodes = (1 << kOcLevels) - 1;
constexpr int kOcThreads = 256;

__global__ void __launch_bounds__(kOcThreads) oc_multi_kernel(int64_t n, const OcParams P, const float *__restrict__ x,
                                                              const float *__restrict__ dc,
                                                              const uint8_t *__restrict__ pres,
                                                              const float *__restrict__ w, float2 *partials,
                                                              OcScalars *sc) {
    __shared__ float s_sq[kOcNodes];    // sqrt(1 / mid) of node t
    __shared__ bool s_stop[kOcNodes];   // the stop test on node t's interval
    __shared__ double s_mid[kOcNodes];  // midpoint of node t
    __shared__ float s_part[kOcNodes][kOcThreads];
    __shared__ double s_tot[kOcNodes];
    __shared__ bool s_last;
    if (sc->done) return;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int nblk = gridDim.x;
    if (tid < kOcNodes) {  // node tid: follow its path from the root (bits of tid + 1 below the leading one)
        double lo = sc->l1, hi = sc->l2;
        const int path = tid + 1, depth = 31 - __clz(path);
        for (int i = depth - 1; i >= 0; --i) {
            const double m = 0.5 * (hi + lo);
            if ((path >> i) & 1)
                lo = m;
            else
                hi = m;
        }
        const double m = 0.5 * (hi + lo);
        s_mid[tid] = m;
        s_sq[tid] = (float)sqrt(1.0 / m);
        s_stop[tid] = (hi - lo) / (lo + hi + P.tol_eps) < P.tol;
    }
    __syncthreads();
    // trial density of node t: x sqrt(max(-dc / mid, floor)) clamped, written as
    // x max(sqrt(-dc) sqrt(1 / mid), sqrt(floor)) (sqrt is monotone: one square root per element)
    float sq[kOcNodes], v[kOcNodes];
#pragma unroll
    for (int t = 0; t < kOcNodes; ++t) {
        sq[t] = s_sq[t];
        v[t] = 0.0f;
    }
    const float sfloor = sqrtf(P.sqrt_floor);
    for (int64_t e = blockIdx.x * (int64_t)kOcThreads + tid; e < n; e += (int64_t)nblk * kOcThreads) {
        const float we = w[e];
        if (pres && pres[e]) {  // xnew = 1
#pragma unroll
            for (int t = 0; t < kOcNodes; ++t) v[t] += we;
            continue;
        }
        const float xe = x[e], s0 = sqrtf(fmaxf(-dc[e], 0.0f));
        const float lo = xe - P.move, hi = xe + P.move;
#pragma unroll
        for (int t = 0; t < kOcNodes; ++t) {
            float tv = xe * fmaxf(s0 * sq[t], sfloor);
            tv = fminf(fmaxf(tv, 0.0f), 1.0f);
            tv = fminf(fmaxf(tv, lo), hi);
            v[t] = fmaf(we, tv, v[t]);
        }
    }
    // block sums: warp wi sums nodes wi, wi + 8, ... over the block's threads in double-float
#pragma unroll
    for (int t = 0; t < kOcNodes; ++t) s_part[t][tid] = v[t];
    __syncthreads();
    for (int t = warp; t < kOcNodes; t += kOcThreads / 32) {
        df32 a{0.0f, 0.0f};
        for (int j = lane; j < kOcThreads; j += 32) a = df_add(a, df32{s_part[t][j], 0.0f});
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            a = df_add(a, df32{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)});
        if (lane == 0) partials[t * nblk + blockIdx.x] = make_float2(a.hi, a.lo);
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) s_last = atomicAdd(&sc->counter, 1u) == (unsigned)nblk - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    for (int t = warp; t < kOcNodes; t += kOcThreads / 32) {
        df32 a{0.0f, 0.0f};
        for (int b = lane; b < nblk; b += 32) {
            const float2 p = __ldcg(&partials[t * nblk + b]);
            a = df_add(a, df32{p.x, p.y});
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1)
            a = df_add(a, df32{__shfl_xor_sync(0xffffffffu, a.hi, o), __shfl_xor_sync(0xffffffffu, a.lo, o)});
        if (lane == 0) s_tot[t] = df_value(a);
    }
    __syncthreads();
    if (tid == 0) {
        double l1 = sc->l1, l2 = sc->l2, lfinal = sc->lfinal;
        int steps = sc->steps, done = 0, node = 0;
        const double target = P.volfrac * (double)n - sc->npres;  // vol > volfrac <=> sum > target
        for (int lvl = 0; lvl < kOcLevels; ++lvl) {
            const double m = s_mid[node];
            if (s_stop[node]) {
                lfinal = m;
                steps += 1;
                done = 1;
                break;
            }
            if (s_tot[node] > target) {
                l1 = m;
                node = 2 * node + 2;
            } else {
                l2 = m;
                node = 2 * node + 1;
            }
            lfinal = m;
            steps += 1;
            if (steps >= P.max_bisect) {
                done = 1;
                break;
            }
        }
        sc->l1 = l1;
        sc->l2 = l2;
        sc->lfinal = lfinal;
        sc->steps = steps;
        sc->done = done;
        sc->counter = 0;
    }
}

// ---- multisection in one cooperative launch ----------------------------------------------
// The rounds of oc_multi_kernel without a launch per round, one block per SM, six levels (63 midpoints) a
// round: with tol 1e-4 twelve steps follow the first one to the right, so that three rounds do (with five
// levels and 31 midpoints along the first path it took five). Per element a trial density is a clamp of a
// line in sqrt(1 / mid), a + d sat(p sqrt(1 / mid) + q): its numbers are formed once and kept in shared
// memory (the rest, beyond 2 M elements on 152 SMs, anew in every round), so that a trial takes two
// operations; half of a block's threads take 32 of the midpoints, half the others. A block's sums of
// the trial volumes and of w a go to the first block as packets; it adds them in block order, walks the
// tree and sends (l1, l2, lfinal, steps, done) back. Its polls are the only ones on the sums; one block (up
// to kOcShare elements) has no exchange. Bound by the latency of its rounds: 61x37x23 takes 24 us and
// 192x96x96 (1.8 M elements) 61, where a grid barrier, all blocks adding all sums, and trials of six
// operations from global memory took 50 and 125. A wait that runs out sets sc->status = GBS_ETIMEOUT
// and ends the rounds; the host reports it.
constexpr int kCoopLevels = 6;
constexpr int kCoopNodes = (1 << kCoopLevels) - 1;
constexpr int kCoopThreads = 512;
constexpr int kCoopRow = kCoopThreads / 2 + 8;  // a node's row of partial sums: four rows meet in no bank
constexpr int kCoopPoll = 10;                   // packets a lane of the first block polls at once
constexpr int kCoopBlocks = 160;
constexpr int kCoopCopies = 8;                // of the first block's answer
constexpr int kOcShare = 4 * kCoopThreads;    // elements per block below one block per SM
constexpr size_t kCoopBoxAt = 16384;          // bytes into the partials, behind oc_init_kernel's
constexpr size_t kCoopSums = sizeof(float) * ((kCoopNodes + 1) * kCoopRow + kCoopThreads / 2);
constexpr int kCoopKeep = (int)((220 * 1024 - kCoopSums) / (3 * sizeof(float) * kCoopThreads));
static_assert(kCoopNodes + 1 == 64 && kCoopThreads == 8 * 64, "eight lanes per node");
static_assert(kCoopBoxAt + 16 * ((size_t)64 * kCoopBlocks + 3 * kCoopCopies) <= kOcPartials, "room");
static int coop_packets(int nblk) { return nblk > 1 ? 64 * nblk + 3 * kCoopCopies : 0; }

// (float)sqrt(1 / m): the reciprocal square root of m's leading part, and one Newton step with m in
// full (1 - m y^2 to 1e-14), where the FP64 division and root take 1200 cycles.
__device__ __forceinline__ float oc_rsqrt(double m) {
    if (!(m > 1e-30 && m < 1e30)) return (float)sqrt(1.0 / m);
    const float h = (float)m, l = (float)(m - (double)h), y = rsqrtf(h), p = __fmul_rn(y, y);
    float e = __fmaf_rn(-h, p, 1.0f);
    e = __fmaf_rn(-h, __fmaf_rn(y, y, -p), e);
    e = __fmaf_rn(-l, p, e);
    return __fmaf_rn(0.5f * y, e, y);
}
// Bisection's test of an interval; the division only where the answer is not clear without.
__device__ __forceinline__ bool oc_stop(double lo, double hi, const OcParams &P) {
    const double d = hi - lo, s = lo + hi + P.tol_eps;
    if (d > 1.000001 * P.tol * s && s > 0.0) return false;
    return d / s < P.tol;
}

// p, q and w d of an element; base gains w a.
__device__ __forceinline__ float3 oc_line(float xe, float dce, float we, bool pre, const OcParams &P, float sfloor,
                                          float &base) {
    if (pre) {  // xnew = 1
        base += we;
        return make_float3(0.0f, 0.0f, 0.0f);
    }
    const float lo = xe - P.move, hi = xe + P.move, b = fminf(fmaxf(1.0f, lo), hi);
    const float a = fminf(fmaxf(xe * sfloor, fminf(fmaxf(0.0f, lo), hi)), b), d = b - a;
    base = fmaf(we, a, base);
    const float inv = d > 0.0f ? 1.0f / d : 0.0f;
    return make_float3(xe * sqrtf(fmaxf(-dce, 0.0f)) * inv, -a * inv, we * d);
}

__global__ void __launch_bounds__(kCoopThreads, 1)
    oc_coop_kernel(int64_t n, const OcParams P, const float *__restrict__ x, const float *__restrict__ dc,
                   const uint8_t *__restrict__ pres, const float *__restrict__ w, uint4 *box, OcScalars *sc,
                   float *xnew, int keep, unsigned polls) {
    extern __shared__ float coop_sh[];
    float *s_part = coop_sh, *kp = s_part + kCoopSums / sizeof(float), *kq = kp + keep, *kw = kq + keep;
    __shared__ float s_sq[kCoopNodes + 1];
    __shared__ int s_stop[kCoopNodes + 1];
    __shared__ double s_mid[kCoopNodes + 1];
    __shared__ double s_tot[kCoopNodes + 1];
    __shared__ double s_lim[3];  // l1, l2, lfinal
    __shared__ int s_steps, s_done, s_ok;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int half = tid >> 8, ht = tid & (kCoopThreads / 2 - 1);
    const int nblk = gridDim.x, bid = blockIdx.x;
    uint4 *answer = box + 64 * nblk;
    if (tid == 0) {
        s_lim[0] = sc->l1;
        s_lim[1] = sc->l2;
        s_lim[2] = sc->lfinal;
        s_steps = sc->steps;
        s_done = sc->done;
        s_ok = 1;
        s_sq[kCoopNodes] = 0.0f;
    }
    const float sfloor = sqrtf(P.sqrt_floor);
    const double target = P.volfrac * (double)n - sc->npres;  // vol > volfrac <=> sum > target
    const int64_t block0 = (int64_t)bid * kCoopThreads, stride = (int64_t)nblk * kCoopThreads;
    float kept = 0.0f;  // w a of the kept elements
    for (int k = tid; k < keep; k += kCoopThreads) {
        const int64_t e = block0 + tid + (int64_t)(k / kCoopThreads) * stride;
        float3 l = make_float3(0.0f, 0.0f, 0.0f);
        if (e < n) l = oc_line(x[e], dc[e], w[e], pres && pres[e], P, sfloor, kept);
        kp[k] = l.x;
        kq[k] = l.y;
        kw[k] = l.z;
    }
    __syncthreads();
    // Rounds have two shapes. While l1 is still 0 the bisection's midpoints are l2/2, l2/4, ...
    // for as long as every volume stays at or below the target (each step sets l2 = mid); a
    // chain round evaluates the next kCoopNodes midpoints of that all-left path, formed exactly
    // as bisection forms them (0.5 (hi + 0)), and ends at the first step that goes right. Once
    // l1 > 0, tree rounds evaluate the full kCoopLevels-level tree. Each round advances the
    // bisection by at least one step, so max_bisect rounds bound the loop.
    for (int round = 0; round < P.max_bisect; ++round) {
        // block-uniform: written before the last __syncthreads. Through a shuffle, so that the compiler
        // knows it uniform: in code it takes for divergent every shuffle costs about 250 cycles
        if (__shfl_sync(0xffffffffu, (int)(s_done != 0 || s_ok == 0), 0)) break;
        const bool chain = s_lim[0] == 0.0;
        const unsigned ep = (unsigned)round + 1;
        if (tid < 128 && (tid & 63) < kCoopNodes) {  // the midpoints by two warps, the stop tests by two
            const int node = tid & 63;
            double lo = s_lim[0], hi = s_lim[1];
            if (chain) {
                // halvings 0.5 (hi + 0) of the all-left path: exact, so the same bits as that
                // loop of dependent FP64 operations (l2 <= 1e9 stays far above the subnormals)
                hi = ldexp(hi, -node);
            } else {
                const int path = node + 1, depth = 31 - __clz(path);
                for (int i = depth - 1; i >= 0; --i) {
                    const double m = 0.5 * (hi + lo);
                    if ((path >> i) & 1)
                        lo = m;
                    else
                        hi = m;
                }
            }
            if (tid < 64) {
                const double m = 0.5 * (hi + lo);
                s_mid[node] = m;
                s_sq[node] = oc_rsqrt(m);
            } else {
                s_stop[node] = oc_stop(lo, hi, P);
            }
        }
        __syncthreads();
        float sq[32], v[32], base = kept;
#pragma unroll
        for (int t = 0; t < 32; ++t) {
            sq[t] = s_sq[32 * half + t];
            v[t] = 0.0f;
        }
        auto trials = [&](float p, float q, float wd) {
#pragma unroll
            for (int t = 0; t < 32; ++t) {
                float y;
                asm("fma.rn.sat.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(p), "f"(sq[t]), "f"(q));
                v[t] = fmaf(wd, y, v[t]);
            }
        };
#pragma unroll 2
        for (int k = ht; k < keep; k += kCoopThreads / 2) trials(kp[k], kq[k], kw[k]);
        for (int64_t e0 = block0 + (int64_t)(keep / kCoopThreads) * stride + ht; e0 < n; e0 += stride)
            for (int64_t e = e0; e < n && e <= e0 + kCoopThreads / 2; e += kCoopThreads / 2) {
                float a = 0.0f;
                const float3 l = oc_line(x[e], dc[e], w[e], pres && pres[e], P, sfloor, a);
                trials(l.x, l.y, l.z);
                if (half == 0) base += a;
            }
#pragma unroll
        for (int t = 0; t < 32; ++t)
            if (32 * half + t < kCoopNodes) s_part[(32 * half + t) * kCoopRow + ht] = v[t];
        s_part[kCoopNodes * kCoopRow + tid] = base;
        __syncthreads();
        // block sums: node t summed by 8 lanes (columns sub, sub + 8, ...), then across those lanes; the
        // sums' errors carried; every sum in a fixed order
        const int t = tid >> 3, sub = tid & 7, columns = t == kCoopNodes ? kCoopThreads : kCoopThreads / 2;
        ddv a{0.0f, 0.0f};
#pragma unroll 8
        for (int j = sub; j < columns; j += 8) {
            float e;
            two_sum(a.h, s_part[t * kCoopRow + j], a.h, e);
            a.l += e;
        }
        __syncwarp();
        auto across = [&]() {
#pragma unroll
            for (int o = 4; o > 0; o >>= 1)
                a = dd_add(a, ddv{__shfl_xor_sync(0xffffffffu, a.h, o), __shfl_xor_sync(0xffffffffu, a.l, o)});
        };
        across();
        bool ok = true;
        if (nblk > 1) {
            if (sub == 0) st_packet(box + t * nblk + bid, __float_as_uint(a.h), __float_as_uint(a.l), 0, ep);
            if (bid == 0) {
                // ten packets polled together, one round trip per sweep
                a = ddv{0.0f, 0.0f};
#pragma unroll 1
                for (int m0 = sub; m0 < nblk && ok; m0 += 8 * kCoopPoll) {
                    uint4 u[kCoopPoll];
#pragma unroll
                    for (int m = 0; m < kCoopPoll; ++m)
                        u[m] = make_uint4(0, 0, 0, m0 + 8 * m < nblk ? ep - 1 : ep);
                    bool all;
                    unsigned sweep = 0;
#pragma unroll 1
                    do {
                        all = true;
#pragma unroll
                        for (int m = 0; m < kCoopPoll; ++m)
                            if (u[m].w != ep) u[m] = ld_packet(box + t * nblk + m0 + 8 * m);
#pragma unroll
                        for (int m = 0; m < kCoopPoll; ++m) all = all && u[m].w == ep;
                    } while (!all && ++sweep < polls);
                    ok = all;
#pragma unroll
                    for (int m = 0; m < kCoopPoll; ++m)
                        a = dd_add(a, ddv{__uint_as_float(u[m].x), __uint_as_float(u[m].y)});
                }
                __syncwarp();
                across();
            } else if (tid < 3) {
                uint4 u = ld_packet(answer + 3 * (bid & (kCoopCopies - 1)) + tid);
                for (unsigned sweep = 0; u.w != ep; ++sweep) {
                    if (sweep >= polls) {
                        ok = false;
                        break;
                    }
                    u = ld_packet(answer + 3 * (bid & (kCoopCopies - 1)) + tid);
                }
                s_lim[tid] = __hiloint2double((int)u.y, (int)u.x);
                if (tid == 0) {
                    s_steps = (int)(u.z >> 1);
                    s_done = (int)(u.z & 1u);
                }
            }
            if (!ok) s_ok = 0;
        }
        if (bid == 0) {
            if (sub == 0) s_tot[t] = dd_value(a);
            __syncthreads();
            if (warp == 0) {  // bisection's tests along the chain or the tree (oc_multi_kernel's walk)
                unsigned long long right = 0, stop = 0;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int node = lane + 32 * h;
                    const bool is = node < kCoopNodes;
                    const unsigned r = __ballot_sync(0xffffffffu, is && s_tot[node] + s_tot[kCoopNodes] > target);
                    const unsigned st = __ballot_sync(0xffffffffu, is && s_stop[node]);
                    right |= (unsigned long long)r << (32 * h);
                    stop |= (unsigned long long)st << (32 * h);
                }
                // the nodes whose midpoints become l1, l2 and lfinal (-1: none)
                int steps = s_steps, done = 0, n1 = -1, n2 = -1, nf;
                if (chain) {
                    // left as far as the first stop or step to the right (tree rounds from there) goes
                    const int event = __ffsll((long long)(stop | right)) - 1;
                    const int left = event < 0 ? kCoopNodes : event, room = P.max_bisect - steps;
                    if (event >= 0 && left < room) {
                        steps += left + 1;
                        nf = left;
                        n2 = left - 1;
                        if ((stop >> left) & 1u) {
                            done = 1;
                        } else {
                            n1 = left;
                            done = steps >= P.max_bisect;
                        }
                    } else {
                        const int took = left < room ? left : room;
                        steps += took;
                        nf = n2 = took - 1;
                        done = steps >= P.max_bisect;
                    }
                } else {
                    int at = 0;
                    for (int lvl = 0; lvl < kCoopLevels; ++lvl) {
                        nf = at;
                        ++steps;
                        if ((stop >> at) & 1u) {
                            done = 1;
                            break;
                        }
                        const bool r = (right >> at) & 1u;
                        if (r)
                            n1 = at;
                        else
                            n2 = at;
                        at = 2 * at + (r ? 2 : 1);
                        if (steps >= P.max_bisect) {
                            done = 1;
                            break;
                        }
                    }
                }
                if (lane < 3) {
                    const int from = lane == 0 ? n1 : (lane == 1 ? n2 : nf);
                    if (from >= 0) s_lim[lane] = s_mid[from];
                }
                __syncwarp();
                // the next step's stop test spares the round that would only find it
                const double lo = s_lim[0], hi = s_lim[1];
                if (!done && lo > 0.0 && oc_stop(lo, hi, P)) {
                    done = 1;
                    ++steps;
                    if (lane == 2) s_lim[2] = 0.5 * (hi + lo);
                }
                if (lane == 0) {
                    s_steps = steps;
                    s_done = done;
                }
                __syncwarp();
                if (nblk > 1 && s_ok && lane < 3 * kCoopCopies) {
                    const double l = s_lim[lane % 3];
                    st_packet(answer + lane, (unsigned)__double2loint(l), (unsigned)__double2hiint(l),
                              (unsigned)steps << 1 | (unsigned)done, ep);
                }
            }
        }
        __syncthreads();
    }
    if (tid == 0 && !s_ok) atomicExch(&sc->status, (int)GBS_ETIMEOUT);
    if (bid == 0 && tid == 0) {
        sc->l1 = s_lim[0];
        sc->l2 = s_lim[1];
        sc->lfinal = s_lim[2];
        sc->steps = s_steps;
        sc->done = s_done;
    }
    const float inv_l = (float)(1.0 / s_lim[2]);
    for (int64_t e = block0 + tid; e < n; e += stride) xnew[e] = oc_trial(x[e], dc[e], inv_l, P, pres && pres[e]);
}

__global__ void oc_final_kernel(int64_t n, const OcParams P, const float *__restrict__ x,
                                const float *__restrict__ dc, const uint8_t *__restrict__ pres, const OcScalars *sc,
                                float *xnew) {
    const float inv_l = (float)(1.0 / sc->lfinal);
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        xnew[e] = oc_trial(x[e], dc[e], inv_l, P, pres && pres[e]);
}

// ---- FP64 dot ---------------------------------------------------------------------------
__global__ void dot_f64_kernel(int64_t n, const double *__restrict__ a, const double *__restrict__ b,
                               double *partials, unsigned *counter, double *out) {
    __shared__ double sred[32];
    __shared__ double tot[1];
    double s = 0.0;
    for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s = fma(a[i], b[i], s);
    const double v[1] = {s};
    if (last_block_reduce<1>(v, partials, counter, tot, sred) && threadIdx.x == 0) *out = tot[0];
}

}  // namespace gbs

using namespace gbs;

// ---- C ABI ------------------------------------------------------------------------------
static size_t reduce_ws_bytes(int64_t nblocks) { return 256 + ((size_t)nblocks * 8 * 4 + 255) / 256 * 256; }

// [counter][partials][the double-float split of u (modal Ke)]
extern "C" size_t gbsimp_sensitivity_ws_bytes(int nx, int ny, int nz) {
    if (!grid_ok(nx, ny, nz)) return reduce_ws_bytes(4096);
    const size_t nd = 3 * (size_t)(nx + 1) * (ny + 1) * (nz + 1);
    return reduce_ws_bytes(4096) + (nd * sizeof(float2) + 255) / 256 * 256;
}

extern "C" int gbsimp_sensitivity(gbsimp_ctx *ctx, int nx, int ny, int nz, const gbsimp_law *law, const float *x,
                                  const double *u, float *dc, float *ce, double *energy_out, void *ws,
                                  size_t ws_bytes, void *stream) {
    NvtxRange range("gbsimp_sensitivity");
    if (!ctx || !law || !x || !u || !grid_ok(nx, ny, nz))
        return set_error(GBS_EINVAL, "gbsimp_sensitivity: bad arguments");
    if (energy_out && (!ws || ws_bytes < reduce_ws_bytes(4096)))
        return set_error(GBS_EINVAL, "gbsimp_sensitivity: workspace too small");
    const int64_t n = (int64_t)nx * ny * nz;
    const unsigned blocks = reduce_blocks(ctx, n, 128);
    unsigned *counter = (unsigned *)ws;
    double *partials = (double *)((char *)ws + 256);
    cudaStream_t st = (cudaStream_t)stream;
    if (energy_out) GBS_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned), st));
    // The double-float element products need the split of u in the workspace; without room
    // for it (a workspace sized for the energy sum only, or none) the FP64 pass runs.
    if (ctx->modal_ok && ws && ws_bytes >= gbsimp_sensitivity_ws_bytes(nx, ny, nz)) {
        float2 *udd = (float2 *)((char *)ws + reduce_ws_bytes(4096));
        int rc = split_dd(ctx, 3 * (int64_t)(nx + 1) * (ny + 1) * (nz + 1), u, nullptr, udd, st);
        if (rc) return rc;
        sens_dd_kernel<<<blocks, 128, 0, st>>>(nx, ny, nz, make_law<double>(*law), modal_kdd(ctx->kmd),
                                               fast_div(ny), fast_div(nz), x, udd, dc,
                                               ce, partials, counter, energy_out);
        GBS_LAUNCH_CHECK("sens_dd_kernel");
        return GBS_OK;
    }
    sens_kernel<<<blocks, 128, 0, st>>>(nx, ny, nz, make_law<double>(*law), ctx->ked, ctx->translation_free ? 1 : 0,
                                        ctx->modal_ok ? 1 : 0, ctx->kmd, x, u, dc, ce, partials, counter, energy_out);
    GBS_LAUNCH_CHECK("sens_kernel");
    return GBS_OK;
}

extern "C" int gbsimp_filter_hs(gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, float *hs, void *stream) {
    if (!ctx || !hs || !grid_ok(nx, ny, nz)) return set_error(GBS_EINVAL, "gbsimp_filter_hs: bad arguments");
    return filter_launch(ctx, nx, ny, nz, rmin, 2, nullptr, nullptr, nullptr, hs, (cudaStream_t)stream);
}

extern "C" int gbsimp_filter(gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, const float *hs, const float *in,
                             float *out, int transpose, void *stream) {
    NvtxRange range("gbsimp_filter");
    if (!ctx || !in || !out || !grid_ok(nx, ny, nz))
        return set_error(GBS_EINVAL, "gbsimp_filter: bad arguments");
    if (transpose && !hs) return set_error(GBS_EINVAL, "gbsimp_filter: the transpose needs hs");
    return filter_launch(ctx, nx, ny, nz, rmin, transpose ? 1 : 0, hs, in, nullptr, out, (cudaStream_t)stream);
}

extern "C" size_t gbsimp_oc_ws_bytes(int nx, int ny, int nz) { return oc_ws_bytes((int64_t)nx * ny * nz); }

namespace gbs {

size_t oc_ws_bytes_impl(int64_t n) { return oc_ws_bytes(n); }

const float *oc_ws_hs(const void *ws, int64_t n) { return oc_ws(const_cast<void *>(ws), n).hs; }

int oc_prepare_impl(const gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, const uint8_t *preserved, void *ws,
                    cudaStream_t st) {
    const int64_t n = (int64_t)nx * ny * nz;
    OcWs w = oc_ws(ws, n);
    GBS_CUDA_TRY(cudaMemsetAsync(w.sc, 0, sizeof(OcScalars), st));
    int rc = filter_launch(ctx, nx, ny, nz, rmin, 2, nullptr, nullptr, nullptr, w.hs, st);
    if (rc) return rc;
    Stencil s;
    rc = make_stencil(rmin, &s);
    if (rc) return rc;
    oc_weights_kernel<<<reduce_blocks(ctx, n, 256), 256, 0, st>>>(nx, ny, nz, s, w.hs, preserved, w.w, w.partials, w.sc);
    GBS_LAUNCH_CHECK("oc_weights_kernel");
    return GBS_OK;
}

// Blocks of oc_coop_kernel that can be resident together on the context's device (cached per
// device): one per SM; 0 when cooperative launches are unavailable.
static int oc_coop_blocks(const gbsimp_ctx *ctx) {
    static std::atomic<int> cache[64];
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64) return 0;
    int v = cache[dev].load(std::memory_order_relaxed);
    if (v != 0) return v > 0 ? v : 0;
    int coop = 0, per_sm = 0;
    const int most = (int)(kCoopSums + 3 * sizeof(float) * kCoopThreads * kCoopKeep);
    if (cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) != cudaSuccess || !coop ||
        cudaFuncSetAttribute(oc_coop_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, oc_coop_kernel, kCoopThreads, most) != cudaSuccess ||
        per_sm < 1) {
        (void)cudaGetLastError();
        cache[dev].store(-1, std::memory_order_relaxed);
        return 0;
    }
    v = std::min(ctx->num_sms > 0 ? ctx->num_sms : 148, kCoopBlocks);
    cache[dev].store(v, std::memory_order_relaxed);
    return v;
}

int oc_run_impl(const gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, const gbsimp_oc_params *prm, const float *x,
                const float *dc, const uint8_t *preserved, float *xnew, float *xphys, void *ws, cudaStream_t st) {
    NvtxRange range("OC update");
    const int64_t n = (int64_t)nx * ny * nz;
    OcWs w = oc_ws(ws, n);
    OcParams P;
    P.move = (float)prm->move;
    P.sqrt_floor = (float)prm->sqrt_floor;
    P.tol = prm->tol;
    P.tol_eps = prm->tol_eps;
    P.volfrac = prm->volfrac;
    P.l1 = prm->l1;
    P.l2 = prm->l2;
    P.max_bisect = prm->max_bisect;
    const unsigned blocks = reduce_blocks(ctx, n, 256);
    // One cooperative launch for the multisection and xnew. A block takes kOcShare elements before there is
    // one on every SM: fewer blocks make the exchange cheaper than the trials get dearer.
    const int cb = oc_coop_blocks(ctx);
    const int nb = (int)std::min<int64_t>((n + kOcShare - 1) / kOcShare, cb);
    uint4 *box = (uint4 *)((char *)w.partials + kCoopBoxAt);
    oc_init_kernel<<<blocks, 256, 0, st>>>(n, P, dc, w.partials, w.sc, box, coop_packets(nb));
    GBS_LAUNCH_CHECK("oc_init_kernel");
    if (cb > 0) {
        const int64_t per = (n + (int64_t)nb * kCoopThreads - 1) / ((int64_t)nb * kCoopThreads);
        int keep = (int)std::min<int64_t>(per, kCoopKeep) * kCoopThreads;
        unsigned polls = wait_polls(ctx);
        void *args[] = {(void *)&n, (void *)&P, (void *)&x, (void *)&dc, (void *)&preserved, (void *)&w.w,
                        (void *)&box, (void *)&w.sc, (void *)&xnew, (void *)&keep, (void *)&polls};
        const cudaError_t e =
            ctx->diag[GBSIMP_DIAG_OC] == 1
                ? cudaErrorCooperativeLaunchTooLarge
                : cudaLaunchCooperativeKernel((void *)oc_coop_kernel, dim3((unsigned)nb), dim3(kCoopThreads), args,
                                              kCoopSums + 3 * sizeof(float) * keep, st);
        if (e == cudaSuccess) {
            GBS_LAUNCH_CHECK("oc_coop_kernel");
            return filter_launch(ctx, nx, ny, nz, rmin, 0, w.hs, xnew, preserved, xphys, st);
        }
        // refused: a context that may use fewer SMs than the device has, say, does not hold a block per SM
        (void)cudaGetLastError();
    }
    // a launch per round; kOcNodes double-float partials per block fit the 4 * 4096 doubles of the workspace
    int64_t mb = (n + kOcThreads - 1) / kOcThreads;
    const int64_t mcap = 2LL * (ctx->num_sms > 0 ? ctx->num_sms : 148);
    mb = mb > mcap ? mcap : (mb < 1 ? 1 : mb);
    if (mb * kOcNodes > 4 * 4096) mb = (4 * 4096) / kOcNodes;
    for (int k = 0; k < prm->max_bisect; k += kOcLevels) {
        oc_multi_kernel<<<(unsigned)mb, kOcThreads, 0, st>>>(n, P, x, dc, preserved, w.w, (float2 *)w.partials, w.sc);
        GBS_LAUNCH_CHECK("oc_multi_kernel");
    }
    oc_final_kernel<<<elem_blocks(ctx, n, 256), 256, 0, st>>>(n, P, x, dc, preserved, w.sc, xnew);
    GBS_LAUNCH_CHECK("oc_final_kernel");
    return filter_launch(ctx, nx, ny, nz, rmin, 0, w.hs, xnew, preserved, xphys, st);
}

int oc_check_args(const gbsimp_ctx *ctx, int nx, int ny, int nz, const gbsimp_oc_params *prm, const float *x,
                  const float *dc, const float *xnew, const float *xphys) {
    if (!ctx || !prm || !x || !dc || !xnew || !xphys || !grid_ok(nx, ny, nz))
        return set_error(GBS_EINVAL, "gbsimp_oc: bad arguments");
    if (prm->max_bisect <= 0 || prm->max_bisect > 1000)
        return set_error(GBS_EINVAL, "gbsimp_oc: max_bisect out of range");
    if (x == xnew) return set_error(GBS_EINVAL, "gbsimp_oc: x and xnew must not alias");
    return GBS_OK;
}

}  // namespace gbs

extern "C" int gbsimp_oc_prepare(gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, const uint8_t *preserved,
                                 void *ws, size_t ws_bytes, void *stream) {
    if (!ctx || !grid_ok(nx, ny, nz) || !ws) return set_error(GBS_EINVAL, "gbsimp_oc_prepare: bad arguments");
    if (ws_bytes < oc_ws_bytes((int64_t)nx * ny * nz)) return set_error(GBS_EINVAL, "gbsimp_oc_prepare: workspace too small");
    return oc_prepare_impl(ctx, nx, ny, nz, rmin, preserved, ws, (cudaStream_t)stream);
}

extern "C" int gbsimp_oc(gbsimp_ctx *ctx, int nx, int ny, int nz, double rmin, const gbsimp_oc_params *prm,
                         const float *x, const float *dc, const uint8_t *preserved, float *xnew, float *xphys,
                         void *ws, size_t ws_bytes, void *stream) {
    int rc = oc_check_args(ctx, nx, ny, nz, prm, x, dc, xnew, xphys);
    if (rc) return rc;
    if (!ws || ws_bytes < oc_ws_bytes((int64_t)nx * ny * nz)) return set_error(GBS_EINVAL, "gbsimp_oc: workspace too small");
    return oc_run_impl(ctx, nx, ny, nz, rmin, prm, x, dc, preserved, xnew, xphys, ws, (cudaStream_t)stream);
}

extern "C" int gbsimp_oc_result(gbsimp_ctx *ctx, const void *ws, double *lambda_out, int *steps_out, void *stream) {
    if (!ctx || !ws) return set_error(GBS_EINVAL, "gbsimp_oc_result: bad arguments");
    cudaStream_t st = (cudaStream_t)stream;
    OcScalars h;
    void *hp = thread_pinned();
    if (!hp) return set_error(GBS_ECUDA, "gbsimp_oc_result: no pinned staging buffer");
    GBS_CUDA_TRY(cudaMemcpyAsync(hp, ws, sizeof(OcScalars), cudaMemcpyDeviceToHost, st));
    GBS_CUDA_TRY(cudaStreamSynchronize(st));
    memcpy(&h, hp, sizeof h);
    if (lambda_out) *lambda_out = h.lfinal;
    if (steps_out) *steps_out = h.steps;
    if (h.status == GBS_ETIMEOUT)
        return set_error(GBS_ETIMEOUT, "gbsimp_oc_result: a wait of the OC update on another block ran out");
    return GBS_OK;
}

extern "C" int gbsimp_dot_f64(gbsimp_ctx *ctx, int64_t n, const double *a, const double *b, double *out, void *ws,
                              size_t ws_bytes, void *stream) {
    if (!ctx || !a || !b || !out || !ws || n < 0) return set_error(GBS_EINVAL, "gbsimp_dot_f64: bad arguments");
    if (ws_bytes < reduce_ws_bytes(4096)) return set_error(GBS_EINVAL, "gbsimp_dot_f64: workspace too small");
    cudaStream_t st = (cudaStream_t)stream;
    unsigned *counter = (unsigned *)ws;
    double *partials = (double *)((char *)ws + 256);
    GBS_CUDA_TRY(cudaMemsetAsync(counter, 0, sizeof(unsigned), st));
    dot_f64_kernel<<<reduce_blocks(ctx, n, 256), 256, 0, st>>>(n, a, b, partials, counter, out);
    GBS_LAUNCH_CHECK("dot_f64_kernel");
    return GBS_OK;
}
