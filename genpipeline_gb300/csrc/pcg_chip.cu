// pcg_chip.cu -- the single-reduction Jacobi-PCG (apply_modal.cuh, CgPass) with every vector on
// the chip: one cooperative launch per inner solve, one CTA per SM, each CTA keeping its box of
// the grid in registers and shared memory for all iterations.
//
// Why. A PCG iteration of a grid whose vectors fit the chip is bound by latency when each
// iteration is its own launch: at 64^3 the streaming pass takes 11.4 us for 34 MB of L2 traffic
// (a serial march over node planes, each waiting for its copies) and 13.9 us with the fold of
// the partial sums and the launch gap, where its arithmetic takes 1.4 us of the SMs' FP32 rate.
// 152 SMs hold 34 MB of shared memory and 39 MB of registers; the PCG state of 64^3 is 20 MB.
// Here an iteration of 32^3 takes 4.1 us (streaming 8.4): march 1.4, exchange 2.2, sums 0.3,
// update 0.2; one of 64^3 8.8, of which 0.8 is its kernel's code not fitting the instruction cache
// (launches of 2000 iterations; with the loads and stores of one of 50 9.8 to 10.0 at 64^3).
// Split. The elements are cut into Px x Py x Pz boxes, one per CTA. A CTA holds all nodes of its
// box, so nodes on a face between boxes are held by both. The box's K u is a partial sum there;
// per iteration the CTAs exchange those partials (a node's 12 bytes) and three sums, and every
// holder of a node adds the partials in the same order, so that all copies of a node stay equal
// bit for bit and no vector is ever exchanged. r, s and p of a node live in registers of the thread
// that updates it; shared memory holds u = M r (the operand), the two halves of w, 1/diag and x.
//
// Exchange without a grid barrier. A packet is 16 bytes, three values and an epoch, stored and
// loaded as one access; a reader polls the packet itself until its epoch is the iteration's: one
// way through the L2 (500 cycles on a die, 880 across) where flag-after-data takes a fence and two.
// The sums go to the first CTA, which adds them in CTA order, takes the scalar step and sends
// alpha, beta and the verdict to all; the neighbours' packets arrive and are settled behind that.
// Measured per exchange of 128 CTAs with 300 node packets each: 2700 cycles; with a mailbox of all
// sums in every CTA 5200, with every CTA polling one set of packets 9000, with a counter and a
// fence 4600. Packets alternate between two copies by iteration parity: a CTA overwrites iteration
// k's packet in iteration k + 2, after it has the scalars of k + 1, which the first CTA sends after
// it has every CTA's sums of k + 1, which each CTA sends behind a block barrier that follows its
// reads of iteration k. Polls are bounded.
//
// The element pass. A lane owns a column of elements along x (lanes run along z, rows of a box
// packed into warps) and marches two slabs of it at once in the lanes of packed FP32x2
// instructions, carrying the (y, z)-transformed node plane and the cx = 1 half to the next step.
// The cz = 1 halves reach the lane above by a shuffle; the cy = 0 and cy = 1 sums go to two
// arrays (W0, W1) with one writer each, so the march needs no block barrier. The slabs' end planes
// are joined behind the march by the warps that have no sums to send: in the march's last step it
// took 0.2 us longer (two or three sets of loads, adds and stores at the end of its serial chain) and 4 KB
// of code.
#include <math.h>
#include <string.h>

#include <algorithm>
#include <atomic>
#include <vector>

#include "apply_modal.cuh"
#include "internal.h"
#include "pcg_chip.h"

namespace gbs {

constexpr int kChipNT = 256;
constexpr int kChipWarps = kChipNT / 32;
constexpr int kChipQ = 6;  // most node pairs per thread (their r, s and p in registers)
constexpr int kChipSmemMax = 224 * 1024;
constexpr int kChipCopies = 16;  // of the packet that carries an iteration's scalars

struct ChipDesign {
    ChipGeom g;
    int block0, nblk;
    ChipItem it;
};
struct ChipTable {
    int n, late;  // late: the block that reports a timeout at its end (diagnostics), 0: none
    ChipDesign d[kChipMaxDesigns];
};
static_assert(sizeof(ChipTable) + 128 <= 4096, "kernel parameters");

// Sums of (h, l) pairs whose leading parts are exact (two-sum) and whose low parts are carried in
// FP32: a level of a tree waits for one FP32 add, not for a renormalisation.
// (A rolled loop: the iteration's code has to stay in the instruction cache.)
__device__ __forceinline__ void sum_dd(ddv (&v)[3], int lanes) {
#pragma unroll 1
    for (int o = lanes >> 1; o > 0; o >>= 1)
#pragma unroll
        for (int k = 0; k < 3; ++k)
            v[k] = dd_add(v[k], ddv{__shfl_xor_sync(0xffffffffu, v[k].h, o), __shfl_xor_sync(0xffffffffu, v[k].l, o)});
}

// The scalars of a solve between two steps.
struct ChipScalars {
    df32 gamma, alpha, beta, rr, delta;
    float rr_stop;
    int done, status, max_iter, freeze;
    double tol, bnorm;
};

// The block's sums from its warps' partials, in every lane.
__device__ __forceinline__ void box_sums(const float2 (*red)[3], ddv (&v)[3]) {
    const int w = threadIdx.x & (kChipWarps - 1);
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float2 f = red[w][k];
        v[k] = ddv{f.x, f.y};
    }
    sum_dd(v, kChipWarps);
}

struct ChipSpan {
    int start, len;
};
// Elements of box a of n cut into P (the first n mod P boxes are one longer).
__host__ __device__ __forceinline__ ChipSpan chip_span(int n, int P, int a) {
    const int q = n / P, r = n - q * P;
    return ChipSpan{a * q + (a < r ? a : r), q + (a < r ? 1 : 0)};
}

// Places of a box whose nodes other boxes hold too, by number of shared axes, when it has
// neighbours on both sides wherever the cut has three boxes or more (the most any box of the cut
// has): NX planes of places along x, the last plane of the box twice among them when `twice`.
struct ChipShared {
    int one, two, three;
    // packets a box waits for, packets it sends, nodes of several neighbours, terms of their sums
    int items() const { return one + 3 * two + 7 * three; }
    int sends() const { return one + two + three; }
    int multi() const { return two + three; }
    int terms() const { return 4 * two + 8 * three; }
};
static ChipShared chip_shared(int NX, int NY, int NZ, int Px, int Py, int Pz, bool twice) {
    auto planes = [](int P) { return P == 1 ? 0 : (P == 2 ? 1 : 2); };
    const int a = Px == 1 ? 0 : planes(Px) + (twice ? 1 : 0), b = planes(Py), c = planes(Pz);
    return ChipShared{a * (NY - b) * (NZ - c) + b * (NX - a) * (NZ - c) + c * (NX - a) * (NY - b),
                      a * b * (NZ - c) + a * c * (NY - b) + b * c * (NX - a), a * b * c};
}

// Bytes of dynamic shared memory of a box: U, W0, W1, 1/diag and x (three float2 per node pair), the
// terms of the nodes of several neighbours, the element moduli (a pair per column and step), the
// lists of packets to wait for, of those nodes and of packets to send.
static size_t chip_smem(int slots, int esteps, const ChipShared &n) {
    return (size_t)5 * 24 * slots + 8 + 16 * (size_t)n.terms() + 8 * (size_t)esteps + 8 * (size_t)(n.items() + n.multi()) +
           4 * (size_t)n.sends();
}

// Bytes of a solve's exchange buffer: the first CTA's mailbox (two parities x a pair of packets from
// each CTA), the scalars' packets (two parities x copies, a 128-byte line each), then the node
// packets (two parities x CTAs x the largest box).
__host__ __device__ inline size_t chip_mail(int nblk) { return (((size_t)64 * nblk + 255) & ~(size_t)255) + 2 * kChipCopies * 128; }
// The launch's flag of a wait that ran out: a word of the first scalars' line that no packet uses.
__device__ __forceinline__ unsigned *chip_late(float4 *xch, int nblk) {
    return (unsigned *)((char *)xch + chip_mail(nblk) - 2 * kChipCopies * 128 + 64);
}
static size_t chip_xch(int nblk, int stride) {
    return nblk > 1 ? chip_mail(nblk) + 2 * (size_t)nblk * stride * sizeof(float4) : 0;
}

// A node's place among the boxes that share it, per axis: 0 its own, 1 shared with the box below,
// 2 with the box above.
__device__ __forceinline__ int chip_side(int i, int e, int a, int P) { return i == 0 ? (a > 0) : (i == e && a + 1 < P ? 2 : 0); }

// E (Ke u) of two elements (the two lanes) from their x-summed and x-differenced (y, z) modes, in
// place; dl gains u . E Ke u = q . r.
__device__ __forceinline__ void chip_element(float2 (&v)[8][3], float2 E, const ModalK &km, float2 &dl) {
#pragma unroll
    for (int bk = 0; bk < kModalBlocks; ++bk) {
        float2 t[3];
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int ro = modal_block(bk, a);
            if (ro < 0) continue;
            float2 s = make_float2(0.0f, 0.0f);
#pragma unroll
            for (int i = 0; i < kModalNnz; ++i) {
                if (modal_row(i) != ro) continue;
                const int co = modal_col(i);
                const float2 k = km.c[modal_class(i)];
                s = modal_row_first(i) ? __fmul2_rn(k, v[co / 3][co % 3]) : __ffma2_rn(k, v[co / 3][co % 3], s);
            }
            t[a] = __fmul2_rn(s, E);
        }
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const int ro = modal_block(bk, a);
            if (ro < 0) continue;
            dl = __ffma2_rn(v[ro / 3][ro % 3], t[a], dl);
            v[ro / 3][ro % 3] = t[a];
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) v[0][c] = make_float2(0.0f, 0.0f);
}

// (y, z) forward butterflies of one node plane's four corners (b = cy * 2 + cz).
__device__ __forceinline__ void chip_yz_forward(float2 (&q)[4][3]) {
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
}

template <int Q>
__global__ void __launch_bounds__(kChipNT, 1)
    pcg_chip_kernel(const ModalK km, unsigned polls, int budget, const __grid_constant__ ChipTable T) {
    extern __shared__ float4 smem4[];
    __shared__ float2 red[kChipWarps][3], red2[kChipWarps][3];
    __shared__ int kd[27];  // packet offset of the neighbour in direction (dx, dy, dz), 9 (dx+1) + 3 (dy+1) + dz+1
    __shared__ int s_ni, s_nm, s_nt, s_ns, s_fail, s_word;
    __shared__ float s_al, s_be;
    // The warp index and the loop's verdict through a shuffle, so that the compiler knows them uniform
    // over a warp: in code it takes for divergent every later shuffle costs about 250 cycles (a
    // three-level sum 4600 instead of 340).
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    int di = 0;
    while (di + 1 < T.n && (int)blockIdx.x >= T.d[di + 1].block0) ++di;
    // The geometry by value from the parameters (uniform), the pointers through shared memory: code that
    // picks one of several pointer members by their address (the right-hand side's three forms) must
    // not do so in parameter space.
    const ChipGeom g = T.d[di].g;
    const int bid = (int)blockIdx.x - T.d[di].block0, nblk = T.d[di].nblk;
    __shared__ ChipItem I;
    if (tid == 0) I = T.d[di].it;
    __syncthreads();
    PcgScalars *sc = I.sc;

    // ---- the box ---------------------------------------------------------------------------
    const int bz = bid % g.Pz, by = (bid / g.Pz) % g.Py, bx = bid / (g.Pz * g.Py);
    const ChipSpan X = chip_span(g.nx, g.Px, bx), Y = chip_span(g.ny, g.Py, by), Z = chip_span(g.nz, g.Pz, bz);
    const int ex = X.len, ey = Y.len, ez = Z.len;
    const int SZ = g.NZm, SY = g.NYm * g.NZm;  // node strides of a plane
    const int64_t NZg = g.nz + 1, Sg = (int64_t)(g.ny + 1) * NZg;
    // Slab s starts at plane s L; pair gp holds slabs gp (lane x) and gp + G (lane y), planes 0..L of
    // each. So the last plane of a slab and the first of the next are the same nodes twice: both
    // copies are kept (the same bits), the later slab's is the one that counts.
    const int L = (ex + 2 * g.G - 1) / (2 * g.G), NP = L + 1, slots = g.G * NP * SY;
    const int ncol = g.G * ey * ez;

    float2 *U = (float2 *)smem4, *W0 = U + 3 * slots, *W1 = W0 + 3 * slots, *Dv = W1 + 3 * slots, *Xs = Dv + 3 * slots;
    float4 *Tm = (float4 *)(Xs + 3 * slots + (slots & 1));  // terms of the nodes of several neighbours
    float2 *Es = (float2 *)(Tm + g.terms);
    uint2 *item = (uint2 *)(Es + L * ncol);  // packets to wait for
    uint2 *multi = item + g.items;           // nodes of several neighbours
    unsigned *sends = (unsigned *)(multi + g.multi);
    // word of component c of place d (node pair << 1 | lane) in the float view of an array
    auto word_of = [](int d, int c) { return 6 * (d >> 1) + (d & 1) + 2 * c; };

    if (tid == 0) s_ni = s_nm = s_nt = s_ns = s_fail = 0;
    if (tid < 27) {
        const int dx = tid / 9 - 1, dy = (tid / 3) % 3 - 1, dz = tid % 3 - 1;
        int o = ((dx * g.Py + dy) * g.Pz + dz) * g.stride;
        if (dx) o += (dx < 0 ? (bx > 0 ? chip_span(g.nx, g.Px, bx - 1).len : 0) : -ex) * SY;
        if (dy) o += (dy < 0 ? (by > 0 ? chip_span(g.ny, g.Py, by - 1).len : 0) : -ey) * SZ;
        if (dz) o += dz < 0 ? (bz > 0 ? chip_span(g.nz, g.Pz, bz - 1).len : 0) : -ez;
        kd[tid] = o;
    }
    // The node of lane h of pair n: plane, row, column, and whether it is the copy that counts; false
    // when there is none (a plane past the box, a row or column of a smaller box).
    auto node_at = [&](int n, int h, int &i, int &j, int &k, bool &counts) {
        const int pt = n / SY, jk = n - pt * SY, gp = pt / NP, t = pt - gp * NP, slab = gp + h * g.G;
        j = jk / SZ;
        k = jk - j * SZ;
        i = slab * L + t;
        counts = t < L || slab + 1 == 2 * g.G;
        return n < slots && i <= ex && j <= ey && k <= ez;
    };
    // ---- the vectors: thread tid holds node pairs tid, tid + 256, ... ---------------------------
    float2 r[Q][3], s[Q][3], p[Q][3];
    // The widest kernel's loop code outgrows the instruction cache (at 64^3 a warp waited for code 18 % of
    // the time): it takes the shorter forms of two parts, which the others are slower with (64^3 9.8 ->
    // 8.9 us, 60^3 7.6 -> 8.1 with both): two packets polled together instead of four, and x updated in
    // every iteration instead of in every other, for two.
    constexpr bool kTight = Q > 5;
    constexpr int kPoll = kTight ? 2 : 4;
    unsigned own = 0;  // bit 2 q + h: counts in this CTA's sums (one of a shared node's holders counts it)
    const bool fresh = I.fresh != 0;
    const volatile PcgScalars *vsc = sc;
    int it = fresh ? 0 : vsc->iter;
    const float bs = fresh && I.bdd ? (float)*I.bscale : 0.0f;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int n = tid + kChipNT * q;
        float rv[2][3] = {}, sv[2][3] = {}, pv[2][3] = {}, xv[2][3] = {}, dv[2][3] = {}, wv[2][3] = {};
        bool last_row = false;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int i, j, k;
            bool counts;
            if (!node_at(n, h, i, j, k, counts)) continue;
            last_row = j == ey;
            const int64_t g0 = 3 * ((X.start + i) * Sg + (Y.start + j) * NZg + (Z.start + k));
            if (counts && chip_side(i, ex, bx, g.Px) != 2 && chip_side(j, ey, by, g.Py) != 2 &&
                chip_side(k, ez, bz, g.Pz) != 2)
                own |= 1u << (2 * q + h);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const int64_t gw = g0 + c;
                dv[h][c] = I.dinv[gw];
                if (fresh) {
                    if (I.bdd) {
                        const float2 v = I.bdd[gw];
                        rv[h][c] = fmaf(v.x, bs, v.y * bs);
                    } else {
                        rv[h][c] = I.b[gw];
                    }
                } else {
                    rv[h][c] = I.r[gw];
                    wv[h][c] = I.w[gw];
                    xv[h][c] = I.u[gw];
                    if (it > 0) {
                        sv[h][c] = I.s[gw];
                        pv[h][c] = I.p[gw];
                    }
                }
                if (dv[h][c] == 0.0f) rv[h][c] = 0.0f;  // fixed DOFs: r stays zero, out of every sum
            }
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            r[q][c] = make_float2(rv[0][c], rv[1][c]);
            s[q][c] = make_float2(sv[0][c], sv[1][c]);
            p[q][c] = make_float2(pv[0][c], pv[1][c]);
            if (n >= slots) continue;
            // W0 holds rows j < ey, W1 row ey: the march rewrites exactly the words the sums use
            const float2 w = make_float2(wv[0][c], wv[1][c]), zero = make_float2(0.0f, 0.0f);
            W0[3 * n + c] = last_row ? zero : w;
            W1[3 * n + c] = last_row ? w : zero;
            U[3 * n + c] = zero;
            Dv[3 * n + c] = make_float2(dv[0][c], dv[1][c]);
            Xs[3 * n + c] = make_float2(xv[0][c], xv[1][c]);
        }
    }
    for (int e = tid; e < L * ncol; e += kChipNT) {
        const int t = e / ncol, col = e - t * ncol;
        const int gg = col / (ey * ez), jk = col - gg * ey * ez, j = jk / ez, k = jk - j * ez;
        float v[2];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int i = (gg + h * g.G) * L + t;
            v[h] = i < ex ? I.E[((int64_t)(X.start + i) * g.ny + Y.start + j) * g.nz + Z.start + k] : 0.0f;
        }
        Es[e] = make_float2(v[0], v[1]);
    }
    __syncthreads();
    // ---- shared nodes --------------------------------------------------------------------------
    // item.x: the packet's place relative to this box's packets; item.y: place | row-ey flag << 16
    // (a node of one neighbour), or term | 1 << 31. multi.x: place | row-ey flag << 16; multi.y: first
    // term | number << 16 | own term << 24. sends: packet | place << 16 (the copy that counts). The
    // order of the lists does not matter.
    if (nblk > 1) {
        for (int d = tid; d < 2 * slots; d += kChipNT) {
            int i, j, k;
            bool counts;
            if (!node_at(d >> 1, d & 1, i, j, k, counts)) continue;
            const int sd[3] = {chip_side(i, ex, bx, g.Px), chip_side(j, ey, by, g.Py), chip_side(k, ez, bz, g.Pz)};
            const int axes = (sd[0] != 0) + (sd[1] != 0) + (sd[2] != 0), o = i * SY + j * SZ + k;
            const unsigned place = (unsigned)d | (unsigned)(j == ey) << 16;
            if (axes == 0) continue;
            if (counts) sends[atomicAdd(&s_ns, 1)] = (unsigned)o | (unsigned)d << 16;
            int first = 0, at = 0, self = 0;
            if (axes > 1) first = atomicAdd(&s_nt, 1 << axes);
#pragma unroll 1
            for (int m = 0; m < 8; ++m) {  // the holders in the order of their boxes (x, y, z)
                int dir = 13;
                bool use = true;
#pragma unroll
                for (int a = 0; a < 3; ++a) {
                    const int hi = (m >> (2 - a)) & 1, me = sd[a] == 1;  // the higher box of the pair on axis a
                    use = use && !(sd[a] == 0 && hi);
                    if (sd[a] != 0 && hi != me) dir += (hi ? 1 : -1) * (a == 0 ? 9 : (a == 1 ? 3 : 1));
                }
                if (!use) continue;
                if (dir == 13) self = at;
                else item[atomicAdd(&s_ni, 1)] =
                        make_uint2((unsigned)(o + kd[dir]), axes == 1 ? place : (unsigned)(first + at) | 1u << 31);
                ++at;
            }
            if (axes > 1)
                multi[atomicAdd(&s_nm, 1)] =
                    make_uint2(place, (unsigned)first | (unsigned)at << 16 | (unsigned)self << 24);
        }
        __syncthreads();
    }
    const int ni = s_ni, nm = s_nm, ns = s_ns;

    // ---- the march's column ----------------------------------------------------------------------
    const int rpw = 32 / ez, groups = (ey + rpw - 1) / rpw;
    const bool task = warp < groups * g.G;
    const int gp = warp / groups, jrow = (warp - gp * groups) * rpw + lane / ez, kcol = lane - (lane / ez) * ez;
    const bool col_ok = task && lane < rpw * ez && jrow < ey;
    const int j0 = col_ok ? jrow : 0, k0 = col_ok ? kcol : 0;
    const int base = task ? 3 * (gp * NP * SY + j0 * SZ + k0) : 0, ecol = (gp * ey + j0) * ez + k0;
    const bool top = col_ok && kcol == ez - 1;
    const float lowf = col_ok && kcol > 0 ? 1.0f : 0.0f;  // a lane below in the same row

    // ---- scalars: the first warp's (of the first CTA), in shared memory between its steps -----------
    __shared__ ChipScalars S;
    if (tid == 0) {
        S = ChipScalars{};
        S.tol = fresh ? I.tol : vsc->tol;
        S.max_iter = fresh ? I.max_iter : vsc->max_iter;
        if (!fresh) {
            S.done = vsc->done;
            S.status = vsc->status;
            S.gamma = df_from(vsc->rz);
            S.alpha = df_from(vsc->alpha[0]);
            S.beta = df_from(vsc->beta);
            S.rr = df_from(vsc->rr);
            S.delta = df_from(vsc->pap);
            S.bnorm = vsc->bnorm;
            S.freeze = vsc->freeze;  // timing: every iteration with the scalars as they are
            const double stop = S.tol * S.bnorm;
            S.rr_stop = (float)(stop * stop);
        }
        s_al = S.alpha.hi;
        s_be = S.beta.hi;
        s_word = S.done | (S.status << 1);
    }
    __syncthreads();
    int done = s_word & 1, status = s_word >> 1;
    bool first = fresh;
    unsigned ep = 0;
    float alpha_prev = 0.0f;
    bool two = false;  // this iteration updates x, for the one before too
    // The scalar step of the iteration whose sums are v3 (the first warp of the design's first CTA;
    // the other threads get its alpha, beta and verdict).
    auto step = [&](const ddv (&v)[3]) {
        df32 t[3];
#pragma unroll
        for (int k = 0; k < 3; ++k) t[k] = df_renorm(v[k].h, v[k].l);
        ChipScalars c = S;
        __syncwarp();
        c.rr = t[2];
        c.delta = t[1];
        if (first) {
            c.bnorm = sqrt(df_value(c.rr));
            const double stop = c.tol * c.bnorm;
            c.rr_stop = (float)(stop * stop);
            cg_first_step_df(t[0], t[1], t[2], c.tol, c.done, c.status, c.gamma, c.alpha, c.beta);
        } else if (!c.freeze) {
            int its = it;
            cg_scalar_step_df(t[0], t[1], t[2], c.rr_stop, c.max_iter, its, c.done, c.status, c.gamma, c.alpha, c.beta);
        }
        if (lane == 0) {
            S = c;
            s_al = c.alpha.hi;
            s_be = c.beta.hi;
            s_word = c.done | (c.status << 1);
        }
        return c;
    };
    // The halves of w at the slabs' ends: a slab's last plane and the next slab's first are the same
    // nodes, and both copies take the sum (by all warps but the first, which has the sums to send).
    auto join = [&]() {
        float *f0 = (float *)W0, *f1 = (float *)W1;
#pragma unroll 1
        for (int e = tid - 32; e < (2 * g.G - 1) * SY; e += kChipNT - 32) {
            const int slab = e / SY, jk = e - slab * SY, next = slab + 1;
            const int hl = slab >= g.G, hn = next >= g.G;
            const int a = word_of((((slab - hl * g.G) * NP + L) * SY + jk) << 1 | hl, 0);
            const int b = word_of(((next - hn * g.G) * NP * SY + jk) << 1 | hn, 0);
#pragma unroll
            for (int c = 0; c < 6; c += 2) {
                f0[a + c] = f0[b + c] = f0[a + c] + f0[b + c];
                f1[a + c] = f1[b + c] = f1[a + c] + f1[b + c];
            }
        }
    };
    const int it_end = budget > 0 ? it + budget : 0x7fffffff;

    while (!done && (first || it < it_end)) {
        // ---- s, r, u, p, x of the box's nodes ---------------------------------------------------
        const float al = s_al, be = s_be;
        const float2 al2 = make_float2(al, al), na2 = make_float2(-al, -al), be2 = make_float2(be, be);
        // x takes two steps at once, every other iteration: x_{i+1} = x_{i-1} +
        // (alpha_{i-1} + alpha_i beta_i) p_{i-1} + alpha_i u_i
        const float c1 = fmaf(al, be, alpha_prev);
        const float2 c12 = make_float2(c1, c1), ap2 = make_float2(alpha_prev, alpha_prev);
        float2 g_ru = make_float2(0.0f, 0.0f), g_rr = g_ru;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int n3 = 3 * (tid + kChipNT * q);
            if (n3 >= 3 * slots) continue;
            float2 w[3], d[3], x[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                w[c] = add2(W0[n3 + c], W1[n3 + c]);
                d[c] = Dv[n3 + c];
                if (kTight || two) x[c] = Xs[n3 + c];
            }
            float2 ru = make_float2(0.0f, 0.0f), rr = ru;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float2 uo = __fmul2_rn(d[c], r[q][c]);
                if (kTight) Xs[n3 + c] = __ffma2_rn(ap2, p[q][c], x[c]);
                else if (two) Xs[n3 + c] = __ffma2_rn(c12, p[q][c], __ffma2_rn(al2, uo, x[c]));
                s[q][c] = __ffma2_rn(be2, s[q][c], w[c]);
                p[q][c] = __ffma2_rn(be2, p[q][c], uo);
                const float2 rn = __ffma2_rn(na2, s[q][c], r[q][c]);
                r[q][c] = make_float2(d[c].x != 0.0f ? rn.x : 0.0f, d[c].y != 0.0f ? rn.y : 0.0f);
                const float2 u = __fmul2_rn(d[c], r[q][c]);
                U[n3 + c] = u;
                ru = __ffma2_rn(r[q][c], u, ru);
                rr = __ffma2_rn(r[q][c], r[q][c], rr);
            }
            const float2 mine = make_float2((own >> (2 * q)) & 1u ? 1.0f : 0.0f, (own >> (2 * q + 1)) & 1u ? 1.0f : 0.0f);
            g_ru = __ffma2_rn(mine, ru, g_ru);
            g_rr = __ffma2_rn(mine, rr, g_rr);
        }
        __syncthreads();

        // ---- w = K u: the march ------------------------------------------------------------------
        float2 dl = make_float2(0.0f, 0.0f);
        if (task) {
            float2 g1[4][3], qp[4][3];
            auto load = [&](float2 (&v)[4][3], int t) {
                const float2 *u = U + base + 3 * SY * t, *u1 = u + 3 * SZ;
#pragma unroll
                for (int b = 0; b < 4; ++b)
#pragma unroll
                    for (int c = 0; c < 3; ++c) v[b][c] = ((b >> 1) ? u1 : u)[3 * (b & 1) + c];
            };
            load(qp, 0);
            chip_yz_forward(qp);
#pragma unroll
            for (int b = 0; b < 4; ++b)
#pragma unroll
                for (int c = 0; c < 3; ++c) g1[b][c] = make_float2(0.0f, 0.0f);
#pragma unroll 1
            for (int t = 0; t <= L; ++t) {
                float2 h[4][3];
                if (t < L) {
                    float2 v[8][3], qn[4][3];
                    const float2 E = col_ok ? Es[t * ncol + ecol] : make_float2(0.0f, 0.0f);
                    load(qn, t + 1);
                    chip_yz_forward(qn);
#pragma unroll
                    for (int b = 0; b < 4; ++b)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            v[b][c] = add2(qp[b][c], qn[b][c]);
                            v[4 + b][c] = sub2(qn[b][c], qp[b][c]);
                            qp[b][c] = qn[b][c];
                        }
                    chip_element(v, E, km, dl);
#pragma unroll
                    for (int b = 0; b < 4; ++b)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            h[b][c] = add2(g1[b][c], sub2(v[b][c], v[4 + b][c]));
                            g1[b][c] = add2(v[b][c], v[4 + b][c]);
                        }
                } else {
#pragma unroll
                    for (int b = 0; b < 4; ++b)
#pragma unroll
                        for (int c = 0; c < 3; ++c) h[b][c] = g1[b][c];
                }
                // node plane out: back to corner values, the cz = 1 corners to the lane above; rows to
                // W0 (cy = 0) and W1 (cy = 1)
                yz_inverse2(h);
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    const float2 lf = make_float2(lowf, lowf);
                    h[0][c] = __ffma2_rn(lf, shfl_up2(h[1][c]), h[0][c]);
                    h[2][c] = __ffma2_rn(lf, shfl_up2(h[3][c]), h[2][c]);
                }
                if (col_ok) {
                    const int n = base + 3 * SY * t;
                    float2 *w0 = W0 + n, *w1 = W1 + n + 3 * SZ;
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        w0[c] = h[0][c];
                        w1[c] = h[2][c];
                    }
                    if (top)
#pragma unroll
                        for (int c = 0; c < 3; ++c) {
                            w0[3 + c] = h[1][c];
                            w1[3 + c] = h[3][c];
                        }
                }
            }
        }

        // ---- sums, exchange ------------------------------------------------------------------------
        ddv v3[3];
        two_sum(g_ru.x, g_ru.y, v3[0].h, v3[0].l);
        two_sum(dl.x, dl.y, v3[1].h, v3[1].l);
        two_sum(g_rr.x, g_rr.y, v3[2].h, v3[2].l);
        sum_dd(v3, 32);
        if (lane == 0)
#pragma unroll
            for (int k = 0; k < 3; ++k) red[warp][k] = make_float2(v3[k].h, v3[k].l);
        __syncthreads();
        if (nblk > 1) {
            ++ep;
            const int par = (int)(ep & 1u);
            uint4 *mail = (uint4 *)I.xch + (size_t)par * nblk * 2;  // the first CTA's
            uint4 *word = (uint4 *)((char *)I.xch + chip_mail(nblk)) - (size_t)(2 - par) * kChipCopies * 8;
            float4 *xp = (float4 *)((char *)I.xch + chip_mail(nblk)) + ((size_t)par * nblk + bid) * g.stride;
            if (warp == 0) {
                box_sums(red, v3);
                if (lane == 0) {
                    st_packet(mail + 2 * bid, __float_as_uint(v3[0].h), __float_as_uint(v3[0].l), __float_as_uint(v3[1].h), ep);
                    st_packet(mail + 2 * bid + 1, __float_as_uint(v3[1].l), __float_as_uint(v3[2].h),
                              __float_as_uint(v3[2].l), ep);
                }
            } else {
                join();
            }
            __syncthreads();
            const float *f0 = (const float *)W0, *f1 = (const float *)W1;
#pragma unroll 2
            for (int e = tid; e < ns; e += kChipNT) {
                const unsigned y = sends[e];
                const int w = word_of((int)(y >> 16), 0);
                st_packet(xp + (y & 0xffffu), __float_as_uint(f0[w] + f1[w]), __float_as_uint(f0[w + 2] + f1[w + 2]),
                          __float_as_uint(f0[w + 4] + f1[w + 4]), ep);
            }
            for (int e = tid; e < nm; e += kChipNT) {
                const uint2 m = multi[e];
                const int w = word_of((int)(m.x & 0xffffu), 0);
                Tm[(m.y & 0xffffu) + (m.y >> 24)] =
                    make_float4(f0[w] + f1[w], f0[w + 2] + f1[w + 2], f0[w + 4] + f1[w + 4], 0.0f);
            }
            bool ok = true;
            if (bid == 0) {
                // The first CTA adds every CTA's sums (in CTA order within a warp, then by warps), takes
                // the scalar step and sends its result to all. One CTA polls the sums: 152 CTAs polling
                // the same packets took 7700 cycles per exchange, a mailbox each 6000, this 2900.
                const int per = (nblk + kChipWarps - 1) / kChipWarps, peer = warp * per + lane;
                const bool one = lane < per && peer < nblk;
                const uint4 *from = mail + 2 * (one ? peer : 0);
                uint4 ta = make_uint4(0, 0, 0, one ? ep - 1 : ep), tb = ta;
                for (unsigned sweep = 0; ta.w != ep || tb.w != ep; ++sweep) {
                    if (ta.w != ep) ta = ld_packet(from);
                    if (tb.w != ep) tb = ld_packet(from + 1);
                    if (sweep >= polls) {
                        ok = false;
                        break;
                    }
                }
                v3[0] = ddv{__uint_as_float(ta.x), __uint_as_float(ta.y)};
                v3[1] = ddv{__uint_as_float(ta.z), __uint_as_float(tb.x)};
                v3[2] = ddv{__uint_as_float(tb.y), __uint_as_float(tb.z)};
                sum_dd(v3, 32);
                if (lane == 0)
#pragma unroll
                    for (int k = 0; k < 3; ++k) red2[warp][k] = make_float2(v3[k].h, v3[k].l);
                if (!ok) s_fail = 1;
                __syncthreads();
                if (warp == 0 && !s_fail) {
                    box_sums(red2, v3);
                    const ChipScalars c = step(v3);
                    if (lane < kChipCopies)
                        st_packet(word + 8 * lane, __float_as_uint(c.alpha.hi), __float_as_uint(c.beta.hi),
                                  (unsigned)(c.done | (c.status << 1)), ep);
                }
            }
            // The neighbours' packets, a few polled together, one round trip per sweep. A node of one
            // neighbour is settled at once (two terms: the same sum in either order), the others once
            // all their terms are here.
            auto settle = [&](unsigned place, float a, float b, float c) {
                const int w = word_of((int)(place & 0xffffu), 0);
                const bool last_row = (place >> 16) & 1u;
                float *to = (float *)(last_row ? W1 : W0) + w, *no = (float *)(last_row ? W0 : W1) + w;
                to[0] = a;
                to[2] = b;
                to[4] = c;
                no[0] = no[2] = no[4] = 0.0f;
            };
            // Every packet is on its way before a word of W0 or W1 changes: the copies of a node are
            // sent by one thread and settled by others.
            __syncthreads();
#pragma unroll 1
            for (int e0 = tid; ok && e0 < ni; e0 += kPoll * kChipNT) {
                uint2 at[kPoll];
                uint4 v[kPoll];
#pragma unroll
                for (int m = 0; m < kPoll; ++m) {
                    const int e = e0 + m * kChipNT;
                    at[m] = item[e < ni ? e : e0];
                    v[m].w = e < ni ? ep - 1 : ep;
                }
                bool all;
                unsigned sweep = 0;
#pragma unroll 1
                do {
                    all = true;
#pragma unroll
                    for (int m = 0; m < kPoll; ++m)
                        if (v[m].w != ep) v[m] = ld_packet(xp + (int)at[m].x);
#pragma unroll
                    for (int m = 0; m < kPoll; ++m) all = all && v[m].w == ep;
                } while (!all && ++sweep < polls);
                ok = all;
#pragma unroll
                for (int m = 0; m < kPoll; ++m) {
                    if (e0 + m * kChipNT >= ni) continue;
                    const float x = __uint_as_float(v[m].x), y = __uint_as_float(v[m].y), z = __uint_as_float(v[m].z);
                    if (at[m].y >> 31) {
                        Tm[at[m].y & 0x7fffffffu] = make_float4(x, y, z, 0.0f);
                    } else {
                        const int w = word_of((int)(at[m].y & 0xffffu), 0);
                        settle(at[m].y, (f0[w] + f1[w]) + x, (f0[w + 2] + f1[w + 2]) + y, (f0[w + 4] + f1[w + 4]) + z);
                    }
                }
            }
            __syncthreads();
            for (int e = kChipNT - 1 - tid; e < nm; e += kChipNT) {
                // added in the order of their boxes, the same for every holder
                const uint2 m = multi[e];
                const float4 *t = Tm + (m.y & 0xffffu);
                float w[3] = {0.0f, 0.0f, 0.0f};
                const int nt = (int)(m.y >> 16) & 0xff;
#pragma unroll 4
                for (int k = 0; k < nt; ++k) {
                    const float4 v = t[k];
                    w[0] += v.x;
                    w[1] += v.y;
                    w[2] += v.z;
                }
                settle(m.x, w[0], w[1], w[2]);
            }
            if (bid != 0 && tid == 0 && ok) {
                uint4 v = ld_packet(word + 8 * (bid & (kChipCopies - 1)));
                for (unsigned k = 0; v.w != ep; ++k) {
                    if (k >= polls) {
                        ok = false;
                        break;
                    }
                    v = ld_packet(word + 8 * (bid & (kChipCopies - 1)));
                }
                s_al = __uint_as_float(v.x);
                s_be = __uint_as_float(v.y);
                s_word = (int)v.z;
            }
            if (!ok) s_fail = 1;
            __syncthreads();
            if (s_fail) {
                status = GBS_ETIMEOUT;
                break;
            }
        } else {
            if (warp == 0) {
                box_sums(red, v3);
                step(v3);
            } else {
                join();
            }
            __syncthreads();
        }
        const int verdict = __shfl_sync(0xffffffffu, s_word, 0);
        done = verdict & 1;
        status = verdict >> 1;
        // (the start pass and frozen passes leave x as it is: alpha = 0)
        alpha_prev = al;
        two = !two;
        if (!first) ++it;
        first = false;
    }
    // Whichever block's wait ran out, the solve's status is GBS_ETIMEOUT: the block raises the launch's
    // flag before it writes the status, the first block looks at the flag after it has written its own, so
    // that one of the two writes GBS_ETIMEOUT last. Its part of x stays as it came (nobody reads that of
    // a fresh solve).
    if (status == GBS_ETIMEOUT || (T.late > 0 && T.late == bid)) {
        if (tid == 0) {
            if (bid == 0) {
                sc->iter = it;
                sc->trips = 0;
            }
            atomicExch(chip_late(I.xch, nblk), 1u);
            __threadfence();
            atomicExch(&sc->status, (int)GBS_ETIMEOUT);
            atomicExch(&sc->done, 1);
        }
        return;
    }
    // ---- the iterate out; a paused solve's state too -------------------------------------------
    // x owes the last iteration's step when that one did not update it; x = 0 when D b = 0, whatever x0
    const float owed = kTight || two ? alpha_prev : 0.0f;
    const bool zero = !fresh && S.bnorm == 0.0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int n = tid + kChipNT * q;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            int i, j, k;
            bool counts;
            if (!node_at(n, h, i, j, k, counts) || !counts || chip_side(i, ex, bx, g.Px) == 2 ||
                chip_side(j, ey, by, g.Py) == 2 || chip_side(k, ez, bz, g.Pz) == 2)
                continue;
            const int64_t g0 = 3 * ((X.start + i) * Sg + (Y.start + j) * NZg + (Z.start + k));
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const float2 w = add2(W0[3 * n + c], W1[3 * n + c]), x = Xs[3 * n + c];
                I.u[g0 + c] = zero ? 0.0f : fmaf(owed, h ? p[q][c].y : p[q][c].x, h ? x.y : x.x);
                if (!done) {
                    I.r[g0 + c] = h ? r[q][c].y : r[q][c].x;
                    I.w[g0 + c] = h ? w.y : w.x;
                    I.s[g0 + c] = h ? s[q][c].y : s[q][c].x;
                    I.p[g0 + c] = h ? p[q][c].y : p[q][c].x;
                }
            }
        }
    }
    if (bid == 0 && tid == 0) {
        sc->iter = it;
        sc->max_iter = S.max_iter;
        sc->tol = S.tol;
        sc->done = done;
        sc->status = status;
        sc->bnorm = S.bnorm;
        sc->rz = df_value(S.gamma);
        sc->rr = df_value(S.rr);
        sc->pap = df_value(S.delta);
        sc->alpha[0] = df_value(S.alpha);
        sc->beta = df_value(S.beta);
        sc->trips = 0;
        sc->freeze = S.freeze;
        __threadfence();
        if (nblk > 1 && atomicAdd(chip_late(I.xch, nblk), 0u)) {
            atomicExch(&sc->status, (int)GBS_ETIMEOUT);
            atomicExch(&sc->done, 1);
        }
    }
}

// ---- plans ------------------------------------------------------------------------------------
// Modelled SM cycles of one iteration of a box, fitted to clock counts of its phases over boxes of
// 2x8x8 to 16x8x16 elements (within 10 %; over 190 grids 0.78 to 1.19 of it): the march's steps,
// dearer with a second warp on a scheduler and with several slabs (their planes meet in shared memory's
// banks; not in single steps of rows up to four); the update of q places per thread; the block's sums; the exchange; and what the widest
// kernel, whose iteration outgrows the instruction cache, takes longer.
static double chip_cost(int ex, int ez, int q, int warps, int G, int nblk, int items) {
    const int L = (ex + 2 * G - 1) / (2 * G);
    double c = 1560.0 + L * (650.0 + 55.0 * std::min(warps, 4) + (warps > 4 ? 370.0 : 0.0));
    if (G > 1) c += 100.0 + (ez > 4 || L > 1 ? 100.0 * warps * L : 0.0);
    c += 700.0 + 320.0 * q + (q > 5 ? 2500.0 : 0.0);
    return c + (nblk > 1 ? 4500.0 + 1.6 * items : 630.0);
}

// Every way to cut the grid into at most max_blocks boxes; f(geom, nblk, cost) for each that fits.
template <typename F>
static void chip_each(int nx, int ny, int nz, int max_blocks, F &&f) {
    auto up = [](int a, int b) { return (a + b - 1) / b; };
    for (int Pz = up(nz, 32); Pz <= nz && Pz <= max_blocks; ++Pz) {
        const int ez = up(nz, Pz), rpw = 32 / ez;
        if (Pz > 1 && up(nz, Pz - 1) == ez) continue;  // no smaller box for one more cut
        for (int Py = 1; Py <= ny && Pz * Py <= max_blocks; ++Py) {
            const int ey = up(ny, Py), groups = up(ey, rpw);
            if ((Py > 1 && up(ny, Py - 1) == ey) || groups > kChipWarps) continue;
            for (int Px = 1; Px <= nx && Pz * Py * Px <= max_blocks; ++Px) {
                const int ex = up(nx, Px);
                if (Px > 1 && up(nx, Px - 1) == ex) continue;
                const int64_t nodes = (int64_t)(ex + 1) * (ey + 1) * (ez + 1);
                if (nodes > 2 * kChipNT * kChipQ) continue;
                const int nblk = Px * Py * Pz;
                for (int G = 1; G <= kChipWarps / groups && 2 * G <= ex + 1; ++G) {
                    // places for the boxes of either length along x (the shorter may have more of a kind)
                    const int L = up(ex, 2 * G), slots = G * (L + 1) * (ey + 1) * (ez + 1);
                    if (slots > kChipNT * kChipQ) continue;
                    const ChipShared sh = chip_shared(ex + 2 * G, ey + 1, ez + 1, Px, Py, Pz, true);
                    if (chip_smem(slots, L * G * ey * ez, sh) > (size_t)kChipSmemMax) continue;
                    const int q = up(slots, kChipNT);
                    ChipGeom g{nx, ny, nz, Px, Py, Pz, G, ey + 1, ez + 1, (int)nodes, q, sh.items(), sh.multi(), sh.terms()};
                    f(g, nblk, chip_cost(ex, ez, q, groups * G, G, nblk, sh.items()));
                }
            }
        }
    }
}

using ChipKernel = void (*)(const ModalK, unsigned, int, const ChipTable);
// Places per thread of the largest box, rounded up to a kernel's: 95x47x33 (four) took 7.3 us per
// iteration in its own kernel and 11.4 in the one for six, 60^3 (five) 7.6 and 8.0; one for three measured
// no better than four's.
static const ChipKernel chip_kern[5] = {pcg_chip_kernel<1>, pcg_chip_kernel<2>, pcg_chip_kernel<4>, pcg_chip_kernel<5>,
                                        pcg_chip_kernel<kChipQ>};

// Sets the kernels' shared-memory limit once per device; false without cooperative launches or when a
// CTA does not fit an SM.
static bool chip_coop(const gbsimp_ctx *ctx) {
    static std::atomic<int> ready[128];  // every thread stores the same value
    const int dev = ctx->device >= 0 && ctx->device < 128 ? ctx->device : 0;
    if (ready[dev] == 0) {
        int coop = 0;
        bool ok = cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, dev) == cudaSuccess && coop;
        for (ChipKernel k : chip_kern) {
            int per_sm = 0;
            ok = ok && cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, kChipSmemMax) == cudaSuccess &&
                 cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, kChipNT, kChipSmemMax) == cudaSuccess &&
                 per_sm > 0;
        }
        (void)cudaGetLastError();
        ready[dev] = ok ? 1 : -1;
    }
    return ready[dev] > 0;
}

// A grid's plans: for each number of CTAs the cheapest cut into at most that many boxes (cost 1e300
// below the fewest that hold it). One search over all cuts takes about 10 us and a solve asks at
// every inner PCG, a batch for every design: each thread keeps its last few (a pure function of the
// arguments).
struct ChipPlans {
    int nx, ny, nz, sms;
    size_t xch_bytes;
    int least;  // fewest CTAs, 0: none
    struct {
        double cost;
        ChipGeom g;
    } at[kChipNT + 1];
};

static const ChipPlans &chip_plans(int nx, int ny, int nz, int sms, size_t xch_bytes) {
    constexpr size_t kKeep = 32;
    static thread_local std::vector<ChipPlans> known;
    static thread_local size_t next = 0;
    for (const ChipPlans &k : known)
        if (k.nx == nx && k.ny == ny && k.nz == nz && k.sms == sms && k.xch_bytes == xch_bytes)
            return k;
    known.resize(kKeep);
    ChipPlans &P = known[next];
    next = (next + 1) % kKeep;
    P.nx = nx;
    P.ny = ny;
    P.nz = nz;
    P.sms = sms;
    P.xch_bytes = xch_bytes;
    P.least = 0;
    for (int b = 0; b <= kChipNT; ++b) P.at[b].cost = 1e300;
    chip_each(nx, ny, nz, sms, [&](const ChipGeom &g, int nblk, double c) {
        if (c < P.at[nblk].cost && chip_xch(nblk, g.stride) <= xch_bytes) {
            P.at[nblk].cost = c;
            P.at[nblk].g = g;
        }
    });
    for (int b = 1; b <= sms; ++b) {
        if (P.least == 0 && P.at[b].cost < 1e300) P.least = b;
        if (P.at[b - 1].cost < P.at[b].cost) P.at[b] = P.at[b - 1];
    }
    return P;
}

static const ChipPlans &chip_plans(const gbsimp_ctx *ctx, const ChipItem &it) {
    return chip_plans(it.nx, it.ny, it.nz, std::min(ctx->num_sms, kChipNT), it.xch_bytes);
}

int chip_min_blocks(const gbsimp_ctx *ctx, const ChipItem &it) {
    // a cheap bound first: the boxes' nodes cover the grid's
    const int64_t room = (int64_t)std::min(ctx->num_sms, kChipNT) * 2 * kChipNT * kChipQ;
    if (!ctx->modal_ok || ctx->diag[GBSIMP_DIAG_CHIP] == 1 || (int64_t)it.nx * it.ny * it.nz > room || !chip_coop(ctx))
        return 0;
    return chip_plans(ctx, it).least;
}

// The cuts of n designs of one launch and their modelled cycles; false when they do not fit together.
static bool chip_allot(const gbsimp_ctx *ctx, const ChipItem *items, int n, ChipGeom *geo, double *cost) {
    if (n <= 0 || n > kChipMaxDesigns || !ctx->modal_ok || !chip_coop(ctx)) return false;
    const int sms = std::min(ctx->num_sms, kChipNT);
    auto blocks = [&](int i) { return geo[i].Px * geo[i].Py * geo[i].Pz; };
    // CTAs: the fewest that hold each design, then more to whichever has the longest iteration,
    // up to the next number of CTAs that shortens it, while that many are left
    int used = 0;
    for (int i = 0; i < n; ++i) {
        const ChipPlans &P = chip_plans(ctx, items[i]);
        if (P.least == 0) return false;
        const auto &a = P.at[n == 1 ? sms : P.least];
        geo[i] = a.g;
        cost[i] = a.cost;
        used += blocks(i);
    }
    if (used > sms) return false;
    bool stuck[kChipMaxDesigns] = {};
    while (n > 1) {
        int j = -1;
        for (int i = 0; i < n; ++i)
            if (!stuck[i] && (j < 0 || cost[i] > cost[j])) j = i;
        if (j < 0) break;
        const ChipPlans &P = chip_plans(ctx, items[j]);
        int c = blocks(j) + 1;
        while (c <= sms && used - blocks(j) + c <= sms && !(P.at[c].cost < cost[j])) ++c;
        if (c > sms || used - blocks(j) + c > sms) {
            stuck[j] = true;
            continue;
        }
        used -= blocks(j);
        geo[j] = P.at[c].g;
        cost[j] = P.at[c].cost;
        used += blocks(j);
    }
    return true;
}

// Shared memory of a cut's largest box.
static size_t chip_smem_of(const ChipGeom &g) {
    const int ex = (g.nx + g.Px - 1) / g.Px, L = (ex + 2 * g.G - 1) / (2 * g.G);
    return chip_smem(g.G * (L + 1) * g.NYm * g.NZm, L * g.G * (g.NYm - 1) * (g.NZm - 1),
                     chip_shared(ex + 2 * g.G, g.NYm, g.NZm, g.Px, g.Py, g.Pz, true));
}

bool chip_plan(int nx, int ny, int nz, int sms, size_t xch_bytes, ChipGeom *g, size_t *smem) {
    sms = std::min(sms, kChipNT);
    if ((int64_t)nx * ny * nz > (int64_t)sms * 2 * kChipNT * kChipQ) return false;
    const ChipPlans &P = chip_plans(nx, ny, nz, sms, xch_bytes);
    if (P.least == 0) return false;
    *g = P.at[sms].g;
    *smem = chip_smem_of(*g);
    return true;
}

double chip_cycles(const gbsimp_ctx *ctx, const ChipItem *items, int n) {
    ChipGeom geo[kChipMaxDesigns];
    double cost[kChipMaxDesigns];
    return chip_allot(ctx, items, n, geo, cost) ? *std::max_element(cost, cost + n) : 1e300;
}

int chip_run(const gbsimp_ctx *ctx, const ChipItem *items, int n, int budget, cudaStream_t st) {
    ChipGeom geo[kChipMaxDesigns] = {};
    double cost[kChipMaxDesigns];
    if (!chip_allot(ctx, items, n, geo, cost)) return kChipRefused;
    auto blocks = [&](int i) { return geo[i].Px * geo[i].Py * geo[i].Pz; };
    ChipTable T;
    memset(&T, 0, sizeof T);
    T.n = n;
    T.late = ctx->diag[GBSIMP_DIAG_TIMEOUT] > 1 ? (int)(ctx->diag[GBSIMP_DIAG_TIMEOUT] - 1) : 0;
    int block0 = 0, q = 0;
    size_t smem = 0;
    for (int i = 0; i < n; ++i) {
        ChipDesign &D = T.d[i];
        D.g = geo[i];
        D.it = items[i];
        D.block0 = block0;
        D.nblk = blocks(i);
        block0 += D.nblk;
        q = std::max(q, D.g.q);
        smem = std::max(smem, chip_smem_of(D.g));
    }
    const int v = q <= 1 ? 0 : (q <= 2 ? 1 : (q <= 4 ? 2 : (q <= 5 ? 3 : 4)));
    for (int i = 0; i < n; ++i) {
        // no packet of an earlier launch may carry an epoch of this one
        if (T.d[i].nblk > 1)
            GBS_CUDA_TRY(cudaMemsetAsync(items[i].xch, 0, chip_xch(T.d[i].nblk, T.d[i].g.stride), st));
    }
    ModalK km = ctx->km;
    unsigned polls = wait_polls(ctx);
    void *args[] = {&km, &polls, &budget, &T};
    const cudaError_t e =
        ctx->diag[GBSIMP_DIAG_CHIP] == 2
            ? cudaErrorCooperativeLaunchTooLarge
            : cudaLaunchCooperativeKernel((const void *)chip_kern[v], dim3((unsigned)block0), dim3(kChipNT), args, smem, st);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        return kChipRefused;
    }
    count_launches(1);
    return GBS_OK;
}

}  // namespace gbs
