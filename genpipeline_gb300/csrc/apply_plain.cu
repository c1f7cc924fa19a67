// apply_plain.cu -- y = D K(x) D p, the bare FP32 apply of a modal-form element stiffness.
//
// A (y, z) node plane is cut into flat tiles: thread t of a block stands for node f = F0 - H + t of the
// plane (row-major, H = nz + 2: a row and a node of halo) and for the element whose low corner that is,
// and marches along x. It takes two slabs of x at once, in the lanes of packed FP32x2
// instructions, and carries the (y, z)-transformed node plane and the cx = 1 half of the element plane
// before, so that a step transforms one plane. Node values reach shared memory a step ahead, one load
// per thread and component, and are read back as pairs; the contributions to the other three corners
// go to the threads of those nodes through shared memory, one barrier per step.
//
// Bound by the latency of its steps, sixteen warps between two barriers: 192x96x96 takes 37 us, its 51 MB
// 7, its FP32 operations 14. The pass that the PCG's iteration is made of (bulk copies of whole planes, two
// elements of one plane per thread) took 48 here with 1.8 times the instructions. A mask that is
// looked at when it arrives, rather than a step later, cost 2 us.
#include <atomic>

#include "apply_modal.cuh"
#include "internal.h"

namespace gbs {

constexpr int kPlainNT = 512;

struct PlainGeom {
    int nx, ny, nz;
    int planes, rem;  // node planes of a segment (one more in the first rem)
    FastDiv fz;       // by nz + 1
};

static size_t plain_smem(int nz) {
    return sizeof(float2) * (2 * 3 * (size_t)(kPlainNT + nz + 2) + 2 * 9 * (size_t)kPlainNT);
}

template <bool kMask>
__global__ void __launch_bounds__(kPlainNT, 1)
    apply_plain_kernel(const PlainGeom G, const float *__restrict__ x, const float *__restrict__ p,
                       float *__restrict__ y, const uint8_t *__restrict__ mask, const Law<float> law, const ModalK km) {
    extern __shared__ float2 plain_sh[];
    const int nx = G.nx, ny = G.ny, nz = G.nz, NZ = nz + 1, S = (ny + 1) * NZ, H = nz + 2, R = kPlainNT + H;
    float2 *U = plain_sh;            // [2][R][3] node values of two planes (slots alternate by step)
    float2 *Hs = plain_sh + 6 * R;   // [2][3 corners][3][NT] contributions to the nodes of other threads
    const int tid = threadIdx.x, f = (int)blockIdx.x * (kPlainNT - H) - H + tid, seg = blockIdx.y;
    const int xs = seg * G.planes + min(seg, G.rem), n = G.planes + (seg < G.rem ? 1 : 0), L = (n + 1) / 2;
    const int a0 = xs, a1 = xs + L;  // the slabs' first node planes (L planes each, the second up to xs + n)

    const int ey = f >= 0 ? (int)fdiv((uint32_t)f, G.fz) : 0, ez = f - ey * NZ;
    const bool element = f >= 0 && ey < ny && ez < nz;
    const bool owned = tid >= H && f < S;
    const float *xe = x + (element ? (int64_t)ey * nz + ez : 0);
    const int64_t ep = (int64_t)ny * nz;

    // Node values of plane j as they are in memory, and the node's mask: nothing waits for them before the
    // next step stores them.
    auto fetch = [&](int j, int node, float (&v)[3], unsigned &m) {
        v[0] = v[1] = v[2] = 0.0f;
        m = 0;
        if (j < 0 || j > nx || node < 0 || node >= S) return;
        const int64_t at = (int64_t)j * S + node;
        if (kMask) m = mask[at];
#pragma unroll
        for (int c = 0; c < 3; ++c) v[c] = p[3 * at + c];
    };
    // this thread's node, and node tid + NT of the tile for tid < H, in both slabs
    struct Nodes {
        float own[2][3], halo[2][3];
        unsigned mo[2], mh[2];
    };
    auto load = [&](int t, Nodes &q) {
        fetch(a0 - 1 + t, f, q.own[0], q.mo[0]);
        fetch(a1 - 1 + t, f, q.own[1], q.mo[1]);
        if (tid < H) {
            fetch(a0 - 1 + t, f + kPlainNT, q.halo[0], q.mh[0]);
            fetch(a1 - 1 + t, f + kPlainNT, q.halo[1], q.mh[1]);
        }
    };
    auto free_of = [&](float v, unsigned m, int c) { return kMask && ((m >> c) & 1u) ? 0.0f : v; };
    unsigned masks = 0;  // of this thread's node: a byte per plane stored, the latest lowest
    auto store = [&](int slot, const Nodes &q) {
        float2 *u = U + slot * 3 * R + 3 * tid;
#pragma unroll
        for (int c = 0; c < 3; ++c) u[c] = make_float2(free_of(q.own[0][c], q.mo[0], c), free_of(q.own[1][c], q.mo[1], c));
        if (kMask) masks = masks << 8 | (q.mo[0] & 7u) | (q.mo[1] & 7u) << 3;
        if (tid < H)
#pragma unroll
            for (int c = 0; c < 3; ++c)
                u[3 * kPlainNT + c] = make_float2(free_of(q.halo[0][c], q.mh[0], c), free_of(q.halo[1][c], q.mh[1], c));
    };
    // the four corners of the element in one plane, transformed along y and z
    auto corners = [&](int slot, float2 (&q)[4][3]) {
        const float2 *u = U + slot * 3 * R + 3 * tid;
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 3; ++c) q[b][c] = element ? u[3 * ((b >> 1) * NZ + (b & 1)) + c] : make_float2(0.0f, 0.0f);
#pragma unroll
        for (int d = 0; d < 2; ++d) {
            const int bit = 1 << d;
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (b & bit) continue;
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float2 u0 = q[b][c], u1 = q[b | bit][c];
                    q[b][c] = add2(u0, u1);
                    q[b | bit][c] = sub2(u1, u0);
                }
            }
        }
    };
    auto density = [&](int j) { return element && j >= 0 && j < nx ? xe[j * ep] : 0.0f; };
    auto moduli = [&](int j, float d) { return element && j >= 0 && j < nx ? modulus(law, d) : 0.0f; };

    Nodes q;
    load(0, q);
    store(0, q);
    load(1, q);
    store(1, q);
    load(2, q);
    float d0 = density(a0 - 1), d1 = density(a1 - 1);
    __syncthreads();
    float2 low[4][3], g1[4][3];
    corners(0, low);
#pragma unroll
    for (int b = 0; b < 4; ++b)
#pragma unroll
        for (int c = 0; c < 3; ++c) g1[b][c] = make_float2(0.0f, 0.0f);
    __syncthreads();  // slot 0 is read before step 0 stores to it

    // Step t: element planes a0 - 1 + t and a1 - 1 + t; node planes of the same numbers are complete and
    // go out (from t = 1 on: the first step is the element plane before the slab).
#pragma unroll 1
    for (int t = 0; t <= L; ++t) {
        const float2 E = make_float2(moduli(a0 - 1 + t, d0), moduli(a1 - 1 + t, d1));
        if (t < L) {
            d0 = density(a0 + t);
            d1 = density(a1 + t);
            store(t & 1, q);  // node plane t + 2; the slot's plane t was read in step t - 1
            if (t + 1 < L) load(t + 3, q);
        }
        float2 v[8][3];
        {
            float2 high[4][3];
            corners((t + 1) & 1, high);
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    v[b][c] = add2(low[b][c], high[b][c]);
                    v[4 + b][c] = sub2(high[b][c], low[b][c]);
                    low[b][c] = high[b][c];
                }
        }
        modal_rows2(v, E, km);
        float2 h[4][3];
#pragma unroll
        for (int b = 0; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                h[b][c] = add2(g1[b][c], sub2(v[b][c], v[4 + b][c]));
                g1[b][c] = add2(v[b][c], v[4 + b][c]);
            }
        yz_inverse2(h);
        float2 *hs = Hs + (t & 1) * 9 * kPlainNT;
#pragma unroll
        for (int b = 1; b < 4; ++b)
#pragma unroll
            for (int c = 0; c < 3; ++c) hs[(3 * (b - 1) + c) * kPlainNT + tid] = h[b][c];
        __syncthreads();
        if (t == 0 || !owned) continue;
        const int j0 = a0 - 1 + t, j1 = a1 - 1 + t;
        float2 s[3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
            s[c] = add2(add2(h[0][c], hs[c * kPlainNT + tid - 1]),
                        add2(hs[(3 + c) * kPlainNT + tid - NZ], hs[(6 + c) * kPlainNT + tid - NZ - 1]));
        // the mask of node plane t: stored two steps ago, one when nothing was stored in this one
        const unsigned m = kMask ? masks >> (t < L ? 16 : 8) : 0u;
        float *y0 = y + 3 * ((int64_t)j0 * S + f), *y1 = y + 3 * ((int64_t)j1 * S + f);
#pragma unroll
        for (int c = 0; c < 3; ++c) y0[c] = free_of(s[c].x, m, c);
        if (j1 < xs + n)
#pragma unroll
            for (int c = 0; c < 3; ++c) y1[c] = free_of(s[c].y, m >> 3, c);
    }
}

int apply_plain(const gbsimp_ctx *ctx, int nx, int ny, int nz, const Law<float> &law, const float *x, const float *p,
                float *y, const uint8_t *mask, cudaStream_t st) {
    const auto kern = mask ? apply_plain_kernel<true> : apply_plain_kernel<false>;
    const size_t smem = plain_smem(nz);
    // the shared-memory limit of the tallest z, once per device (every thread stores the same value)
    static std::atomic<bool> ready[64];
    const int dev = ctx->device;
    if (dev < 0 || dev >= 64 || !ready[dev].load(std::memory_order_relaxed)) {
        const int most = (int)plain_smem(kModalNT * kModalEPT - 64);
        GBS_CUDA_TRY(cudaFuncSetAttribute(apply_plain_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        GBS_CUDA_TRY(cudaFuncSetAttribute(apply_plain_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
        if (dev >= 0 && dev < 64) ready[dev].store(true, std::memory_order_relaxed);
    }
    const int F = kPlainNT - (nz + 2), tiles = ((ny + 1) * (nz + 1) + F - 1) / F;
    // as many segments of x as one wave of blocks has room for, of two node planes at least
    const int sms = ctx->num_sms > 0 ? ctx->num_sms : 148;
    int segs = sms / tiles;
    if (segs > (nx + 2) / 2) segs = (nx + 2) / 2;
    if (segs < 1) segs = 1;
    const PlainGeom G{nx, ny, nz, (nx + 1) / segs, (nx + 1) % segs, fast_div((uint32_t)(nz + 1))};
    kern<<<dim3((unsigned)tiles, (unsigned)segs), kPlainNT, smem, st>>>(G, x, p, y, mask, law, ctx->km);
    GBS_LAUNCH_CHECK("apply_plain_kernel");
    return GBS_OK;
}

}  // namespace gbs
