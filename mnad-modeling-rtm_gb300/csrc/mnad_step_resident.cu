// step_resident: many time steps of a propagation in one launch, its whole
// state on chip.
//
// The grid of a propagation is cut into patches (mnad_resident.h), one per
// CTA and at most one CTA per SM.  A CTA loads both time levels of U, V, W,
// r and the CPML memory variables of its patch into shared memory once, runs
// every step of the launch from there, and writes the state back at the end.
// Between steps only the cells within two points of a patch edge leave the
// SM: the owner publishes them as 16-byte words {U, V, W, tag}, tag = the time
// level + 1, and a CTA that needs a cell polls its word until the tag is the
// one it waits for.  Data and tag travel in one 128-bit access, so the
// exchange needs no fence and no flag, and costs one trip through L2.
//
// One step of a CTA: the groups of 4 points at the patch edges first, each
// publishing its new cells at once, then the inner groups, then one CTA
// barrier.  The last warp or two do nothing but the exchange: they poll the
// cells of the next level while the others compute, sample the receivers and
// fetch the next step's injection amounts.  Where all patches are small
// (RES_SMALL) a lane takes one point instead of a group of 4.
//
// What bounds it: with a few thousand points per SM the shared-memory pipe
// (about 180 wavefronts per 128 points: the window of three columns, the old
// level, the strips' nine variables) and the FP32 pipe (about 450 cycles) at
// about equal weight; with a few hundred points the exchange, about 1 us from
// a published cell to its use.  Time per step of one propagation, on chip /
// the step-per-launch kernel it replaces (CUDA events, GB300):
//   96 x 112 1.7 / 4.1 us, 201 x 201 1.95 / 4.6, 381 x 681 3.3 / 8.7,
//   481 x 1281 5.1 / 16.9, 600 x 1200 (persistent kernel's rounding) 5.2 / 11.4,
//   eight of 256 x 256 0.65 / 1.74 each, eight of 321 x 641 2.0 / 3.3 each.
// Layouts that measured worse on 481 x 1281: one lane group per column with
// idle lanes at the column ends 6.7 us; a warp marching along x with the
// window in registers 7+; strips in a pass of their own 6.9; tasks claimed
// from a counter instead of dealt round 5.9; one point per lane 7.5.
//
// The words have one slot per cell and level parity.  A CTA writes level n+2
// over level n only after it has polled level n+1 of every neighbour, and a
// neighbour publishes level n+1 after the barrier that follows its own reads
// of level n, so no word is overwritten before it was read.
//
// CTAs wait for one another, so the launch is cooperative (all resident).
// Every wait is bounded (ResArgs::spin_limit polls, and the launch's status
// word is looked at on the way): a wait that runs out sets ST_TIMEOUT and the
// CTA leaves at its barrier, all threads together.
//
// Per point the arithmetic is bit for bit that of the kernel the launch would
// run on otherwise: the persistent kernels' (step_resident, step_resident_small)
// or the one-thread-per-point kernel's (..._point).
#include <cuda.h>

#include "mnad_resident.h"
#include "mnad_tile.cuh"

namespace mnad {

namespace {

using namespace tile;

constexpr int Q = TMA_PZ;
// Table entry of a group, or of a point of a small patch (offsets in floats):
//   x: its place in a staged field | flags
//   y: its place in r | in the x strips' arrays << 16
//   z: its place in the top strip's arrays | in the bottom strip's << 16
//   z of a point: its place in its z strip's arrays | its publication slot << 16
//   w: group row (4-row units; a point's row) | column << 8 | injection slot << 16
constexpr unsigned RQ_EDGE = 1u << 16;        // holds cells that other patches need
constexpr unsigned RQ_X = 1u << 17;           // in an x strip
constexpr unsigned RQ_RIGHT = 1u << 18;       // in the right one
constexpr unsigned RQ_TOP = 1u << 19;         // some rows in the top strip
constexpr unsigned RQ_BOTTOM = 1u << 20;      // ... in the bottom strip
constexpr unsigned RQ_SOURCE = 1u << 21;      // the source or a neighbour of it
constexpr unsigned RQ_INJECT = 1u << 22;      // an adjoint receiver
constexpr unsigned RQ_PAST = 1u << 23;        // rows past nz
constexpr unsigned RQ_GENERAL = 1u << 24;     // any of the seven above
constexpr unsigned RQ_UP = 1u << 25;          // the previous lane holds the group above
constexpr unsigned RQ_DOWN = 1u << 26;        // the next lane holds the group below
constexpr unsigned RQ_IMAGE = 1u << 27;       // in the image region (points)
// order of the groups: edges on the general path, plain edges, the others alike
constexpr int RES_CLASSES = 4;
constexpr unsigned RES_STAGGER = 600;         // cycles between the starts of a sub-partition's warps
static_assert(RES_RECS <= 4096, "injection slots fit the table entry");
static_assert(RES_MAX_ROWS / 4 <= 255 && RES_MAX_COLS <= 255, "group coordinates fit the table entry");

struct Cell {
    unsigned u, v, w, tag;
};

__device__ __forceinline__ void publish(uint4* slot, float u, float v, float w, unsigned tag)
{
    const unsigned long long lo = (unsigned long long)__float_as_uint(u) | ((unsigned long long)__float_as_uint(v) << 32);
    const unsigned long long hi = (unsigned long long)__float_as_uint(w) | ((unsigned long long)tag << 32);
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(slot),
                 "l"(lo), "l"(hi)
                 : "memory");
}

__device__ __forceinline__ Cell peek(const uint4* slot)
{
    unsigned long long lo, hi;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(lo), "=l"(hi)
                 : "l"(slot)
                 : "memory");
    return Cell{(unsigned)lo, (unsigned)(lo >> 32), (unsigned)hi, (unsigned)(hi >> 32)};
}

// A CTA's patch, in shared memory (registers are for the stencil).
struct PatchCtx {
    ResLayout L;                            // offsets into the CTA's dynamic shared memory
    int j0, nj, i0, ni;
    float ihx, ihz;                         // 1/dx, 1/dz
    int src_row, src_col;                   // the forward's source (-8: none)
    int inj_scan;                           // injection amounts are looked up in the receiver buckets
    int nhalo, nrec;                        // cells polled; receivers in the table
    int single;                             // the launch runs one step
    int ntask;                              // warp tasks of a step
    int vsx, vst, vsb;                      // strides of the strips' variables
    int s_end;                              // the launch's last step + 1 for this propagation
    uint4* words;                           // published cells of the propagation [parity][patch][slot]
    uint4* out;                             // this patch's, of parity 0 (null: nobody needs them)
    uint4* peaks;                           // the propagation's snapshot maxima [parity][patch]
    int me;                                 // number of the patch
    size_t plane;                           // words per parity
};

// One step of it.
struct StepCtx {
    const float* cur;                       // U of the current level (halo included)
    float* nxt;                             // U of the level written
    uint4* out;                             // publication slots of the new level (null: nobody needs them)
    unsigned tag;
    int tt, tq;
    int inj;                                // this step's injection amounts (offset)
    bool snap_step;
};

__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }

// Snapshot and illumination of a group's points inside the image region at a
// forward's snapshot step.
__device__ __forceinline__ void snapshot(const PropDesc& P, const StepCtx& S, int j, int i, const float2* su,
                                         const float4& uc4, const float4& pu4, float& peak)
{
    const int d = P.d, nz = P.nz, nx = P.nx, niz = nz - 2 * d;
    if (!(i >= d && i < nx - d)) return;
    const size_t nint = (size_t)niz * (nx - 2 * d);
    const long long q0 = (long long)(j - d) + (long long)(i - d) * niz;
    const float sus[Q] = {su[0].x, su[0].y, su[1].x, su[1].y};
    const float pus[Q] = {pu4.x, pu4.y, pu4.z, pu4.w};
    const float ucs[Q] = {uc4.x, uc4.y, uc4.z, uc4.w};
    const int slot = P.snap_stage ? 0 : S.tq - 1 - P.snap_col0;
    const bool keep = (P.snap_flags & SNAP_WRITE) && slot >= 0 && slot < P.snap_cols;
    float sq[Q] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const int jk = j + k;
        if (!(jk >= d && jk < nz - d)) continue;
        // fwd_PDE_exact_MNAD.m:128-141; nU - 2U + pU = su
        float d2u = sus[k];
        if (S.tt == 1) d2u = fmaf(2.0f, ucs[k], sus[k] - pus[k]);
        else if (S.tt == 2) d2u = sus[k] - pus[k];
        d2u *= P.inv_dt2;
        if (keep) {
            const size_t at = (size_t)slot * nint + (size_t)(q0 + k);
            if (P.codec == CODEC_BF16) static_cast<__nv_bfloat16*>(P.snap)[at] = __float2bfloat16_rn(d2u);
            else static_cast<float*>(P.snap)[at] = d2u;
            peak = fmaxf(peak, fabsf(d2u));
        }
        sq[k] = __fmul_rn(d2u, d2u);
    }
    if (P.snap_flags & SNAP_ILLUM) accumulate4(P.illum + q0, sq);
}

// Born_adj_MNAD.m:127-134: the snapshot column that an adjoint's step tt = tq T
// images with, from 0; -1 for none.
__device__ __forceinline__ int image_column(const PropDesc& P, int tq)
{
    const int col = (P.pairing == PAIR_REFERENCE ? P.ncols : P.nsnap) - (P.img_steps - tq) - 1;
    return col >= 0 && col < P.nsnap && col >= P.snap_col0 && col - P.snap_col0 < P.snap_cols ? col : -1;
}

// Adds the patch's image terms: U of the level at `level` (staged), snapshot
// column col.  Done by the warps of the step after the imaging step, as they run
// out of groups: along the columns, G at a time, all loads before the first
// store.  Inside the group's own update the loads were strided and their
// latency stood before the step's barrier (an adjoint of 481 x 1281 that images
// at every step 10.7 -> 7.7 us a step, at every eighth 6.05 -> 5.41).
template <int G, int CODEC>
__device__ __forceinline__ void add_image_as(const PropDesc& P, const PatchCtx& C, const float* level, int col, int warp, int warps)
{
    const int d = P.d, niz = P.nz - 2 * d, lane = threadIdx.x & 31;
    const size_t nint = (size_t)niz * (P.nx - 2 * d);
    const int ja = max(C.j0, d), n = min(C.j0 + C.nj, P.nz - d) - ja, ia = max(C.i0, d), m = min(C.i0 + C.ni, P.nx - d) - ia;
    const size_t q0 = (size_t)(ja - d) + (size_t)(ia - d) * niz, at = (size_t)(col - P.snap_col0) * nint;
    const float sc = CODEC == CODEC_F16 ? P.snap_scale[col] : 1.0f;
    const float* u0 = level + (ia - C.i0 + 2) * RES_PITCH + 4 + (ja - C.j0);
    constexpr int R = RES_MAX_ROWS / 32;
    const void* snap = P.snap;
    double* image = P.image;
    for (int c0 = warp; c0 < m; c0 += G * warps) {
        float p[G][R];
        double a[G][R];
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int c = c0 + g * warps, row = lane + 32 * r;
                const bool in = c < m && row < n;
                const size_t q = q0 + (size_t)c * niz + row;
                p[g][r] = in ? __fmul_rn(snap_decode(snap, CODEC, at + q, sc), u0[c * RES_PITCH + row]) : 0.0f;
                a[g][r] = in ? image[q] : 0.0;
            }
#pragma unroll
        for (int g = 0; g < G; ++g)
#pragma unroll
            for (int r = 0; r < R; ++r)
                if (p[g][r] != 0.0f)                      // as accumulate_product
                    image[q0 + (size_t)(c0 + g * warps) * niz + lane + 32 * r] = a[g][r] + widen_f32(p[g][r]);
    }
}
template <int G>
__device__ __forceinline__ void add_image(const PropDesc& P, const PatchCtx& C, const float* level, int col, int warp, int warps)
{
    if (P.codec == CODEC_BF16) add_image_as<G, CODEC_BF16>(P, C, level, col, warp, warps);
    else if (P.codec == CODEC_F16) add_image_as<G, CODEC_F16>(P, C, level, col, warp, warps);
    else add_image_as<G, CODEC_F32>(P, C, level, col, warp, warps);
}

// nF = F + ((F - pF) + sF) of a group.
__device__ __forceinline__ void advance4(const float4& f, const float4& p, const float2* s, float* o)
{
    const float2 a = padd(pr(f.x, f.y), padd(psub(pr(f.x, f.y), pr(p.x, p.y)), s[0]));
    const float2 b = padd(pr(f.z, f.w), padd(psub(pr(f.z, f.w), pr(p.z, p.w)), s[1]));
    o[0] = a.x; o[1] = a.y; o[2] = b.x; o[3] = b.y;
}

// Ux123_gen.m / Uz123_gen.m of one direction for the 4 points of a group
// (tile::cpml_vec with the fields in registers and the coefficients at hand).
// fd, f0, fa: U, V, W behind, at and ahead of the points; m: the points' m1 of
// U, variables vs apart (advanced in place if `store`); k: their coefficients.
// Adds F1 into c[field].
__device__ __forceinline__ void strip_step(const float (*fd)[Q], const float (*f0)[Q], const float (*fa)[Q], bool low,
                                           float inv_h, float* m, const float* k, int vs, bool store, float2 (*c)[2])
{
    const float2 ih = pr(inv_h, inv_h), ih2 = pmul(ih, ih);
    const float4 k1 = ld4(k), k2 = ld4(k + vs), k3 = ld4(k + 2 * vs);
    const CpmlC cc[2] = {{pr(k1.x, k1.y), pr(k2.x, k2.y), pr(k3.x, k3.y)}, {pr(k1.z, k1.w), pr(k2.z, k2.w), pr(k3.z, k3.w)}};
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        float* mf = m + 3 * f * vs;
        const float4 a = ld4(mf), b = ld4(mf + vs), g = ld4(mf + 2 * vs);
        float2 m1[2] = {pr(a.x, a.y), pr(a.z, a.w)}, m2[2] = {pr(b.x, b.y), pr(b.z, b.w)},
               m3[2] = {pr(g.x, g.y), pr(g.z, g.w)};
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 x0 = pr(f0[f][2 * h], f0[f][2 * h + 1]);
            const float dx = fd[f][2 * h], dy = fd[f][2 * h + 1], ax = fa[f][2 * h], ay = fa[f][2 * h + 1];
            const float2 gr = low ? pr(dx - ax, dy - ay) : pr(ax - dx, ay - dy);
            const float2 lap = psub(pr(dx + ax, dy + ay), padd(x0, x0));
            c[f][h] = padd(c[f][h], cpml_mem2(cc[h], ih, ih2, gr, lap, m1[h], m2[h], m3[h]));
        }
        if (store) {
            *reinterpret_cast<float4*>(mf) = make_float4(m1[0].x, m1[0].y, m1[1].x, m1[1].y);
            *reinterpret_cast<float4*>(mf + vs) = make_float4(m2[0].x, m2[0].y, m2[1].x, m2[1].y);
            *reinterpret_cast<float4*>(mf + 2 * vs) = make_float4(m3[0].x, m3[0].y, m3[1].x, m3[1].y);
        }
    }
}

// The register window of a group; the rows above and below it come from the
// neighbouring lanes where those hold the neighbouring groups of the column
// (a shuffle is one shared-memory wavefront, a load with 16 bytes between
// lanes four), from shared memory elsewhere.  All lanes of a warp together.
__device__ __forceinline__ void load_window(Window& w, const float* f0, int fs, unsigned flags)
{
    const unsigned all = 0xffffffffu;
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) {
        const float* f = f0 + (cc - 1) * RES_PITCH;
        ldv(f, &w.u[cc][1]);
        ldv(f + fs, &w.v[cc][1]);
        ldv(f + 2 * fs, &w.w[cc][1]);
    }
    ldv(f0 + fs - 2 * RES_PITCH, w.v2m);
    ldv(f0 + fs + 2 * RES_PITCH, w.v2p);
#pragma unroll
    for (int cc = 0; cc < 3; ++cc) {
        w.u[cc][0] = __shfl_up_sync(all, w.u[cc][4], 1);
        w.u[cc][5] = __shfl_down_sync(all, w.u[cc][1], 1);
        w.v[cc][0] = __shfl_up_sync(all, w.v[cc][4], 1);
        w.v[cc][5] = __shfl_down_sync(all, w.v[cc][1], 1);
        w.w[cc][0] = __shfl_up_sync(all, w.w[cc][4], 1);
        w.w[cc][5] = __shfl_down_sync(all, w.w[cc][1], 1);
    }
    w.wz[0] = __shfl_up_sync(all, w.w[1][3], 1);
    w.wz[1] = __shfl_down_sync(all, w.w[1][2], 1);
    const bool up = flags & RQ_UP, down = flags & RQ_DOWN;
    if (!up || !down) {
        // one side from shared memory (with both sides missing, the other too):
        // the two ends of a run share one set of loads
        const int o1 = up ? Q : -1, o2 = up ? Q + 1 : -2;
        float x[10];
#pragma unroll
        for (int cc = 0; cc < 3; ++cc) {
            const float* f = f0 + (cc - 1) * RES_PITCH + o1;
            x[3 * cc] = f[0];
            x[3 * cc + 1] = f[fs];
            x[3 * cc + 2] = f[2 * fs];
        }
        x[9] = f0[2 * fs + o2];
        if (up) {
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) w.u[cc][5] = x[3 * cc], w.v[cc][5] = x[3 * cc + 1], w.w[cc][5] = x[3 * cc + 2];
            w.wz[1] = x[9];
        } else {
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) w.u[cc][0] = x[3 * cc], w.v[cc][0] = x[3 * cc + 1], w.w[cc][0] = x[3 * cc + 2];
            w.wz[0] = x[9];
        }
        if (!up && !down) {
#pragma unroll
            for (int cc = 0; cc < 3; ++cc) {
                const float* f = f0 + (cc - 1) * RES_PITCH + Q;
                w.u[cc][5] = f[0];
                w.v[cc][5] = f[fs];
                w.w[cc][5] = f[2 * fs];
            }
            w.wz[1] = f0[2 * fs + Q + 1];
        }
    }
}

// One group of 4 points: the new U, V, W into S.nxt, and its edge cells out.
// All lanes of a warp together; those without `mine` write nothing.
template <bool POINT_ORDER, bool GENERAL>
__device__ __forceinline__ void group_step(const Coefs2& K, const PropDesc& P, const PatchCtx& C, const StepCtx& S,
                                           float* sm, int fs, const uint4 e, bool mine, float& peak)
{
    const int o = e.x & 0xffff;
    const float* f0 = S.cur + o;
    float* n0 = S.nxt + o;                                // holds the previous level
    float rr[Q];
    ldv(sm + C.L.r + (e.y & 0xffff), rr);
    float2 s[3][2];
    float4 uc, vc, wc;
    {
        Window win;
        load_window(win, f0, fs, e.x);
        mnad_update_pairs<POINT_ORDER>(K, win, rr, s[0], s[1], s[2]);
        uc = make_float4(win.u[1][1], win.u[1][2], win.u[1][3], win.u[1][4]);
        vc = make_float4(win.v[1][1], win.v[1][2], win.v[1][3], win.v[1][4]);
        wc = make_float4(win.w[1][1], win.w[1][2], win.w[1][3], win.w[1][4]);
        if constexpr (GENERAL) {
            if (e.x & (RQ_X | RQ_TOP | RQ_BOTTOM)) {
                float2 c[3][2];
#pragma unroll
                for (int f = 0; f < 3; ++f) c[f][0] = c[f][1] = pr(0.0f, 0.0f);
                // the CPML sees U before this step's injection
                // (fwd_PDE_exact_MNAD.m:95-111): the staged U already holds it
                int at = -1000;                           // the source's row in the group (0..3), its column
                int side = 9;
                float amp = 0.0f;
                if (e.x & RQ_SOURCE) {
                    const int zq = e.w & 0xff, col = (e.w >> 8) & 0xff;
                    at = C.src_row - (C.j0 + zq * Q);
                    side = C.src_col - (C.i0 + col);
                    amp = P.src_amp[S.tt - 1];
                }
                auto minus = [&](float (&x)[Q], int row, int column) {
#pragma unroll
                    for (int k = 0; k < Q; ++k)
                        if (side == column && at == k + row) x[k] -= amp;
                };
                auto rows = [](float (*d)[Q], const float* a, const float* b, const float* g) {
#pragma unroll
                    for (int k = 0; k < Q; ++k) d[0][k] = a[k], d[1][k] = b[k], d[2][k] = g[k];
                };
                float x0[3][Q], xa[3][Q], xd[3][Q];
                rows(x0, &win.u[1][1], &win.v[1][1], &win.w[1][1]);
                if (e.x & RQ_SOURCE) minus(x0[0], 0, 0);
                if (e.x & RQ_X) {
                    rows(xd, &win.u[0][1], &win.v[0][1], &win.w[0][1]);
                    rows(xa, &win.u[2][1], &win.v[2][1], &win.w[2][1]);
                    if (e.x & RQ_SOURCE) minus(xd[0], 0, -1), minus(xa[0], 0, 1);
                    const int at_x = e.y >> 16, vs = C.L.xcols * C.nj;
                    strip_step(xd, x0, xa, !(e.x & RQ_RIGHT), C.ihx, sm + C.L.xm + at_x, sm + C.L.xk + at_x,
                                            vs, mine, c);
                }
                if (e.x & (RQ_TOP | RQ_BOTTOM)) {
                    rows(xd, &win.u[1][0], &win.v[1][0], &win.w[1][0]);
                    rows(xa, &win.u[1][2], &win.v[1][2], &win.w[1][2]);
                    if (e.x & RQ_SOURCE) minus(xd[0], -1, 0), minus(xa[0], 1, 0);
                    if (e.x & RQ_TOP) {
                        const int at_z = e.z & 0xffff;
                        strip_step(xd, x0, xa, true, C.ihz, sm + C.L.ztm + at_z, sm + C.L.ztk + at_z,
                                                C.ni * C.L.zt, mine, c);
                    }
                    if (e.x & RQ_BOTTOM) {
                        const int at_z = e.z >> 16;
                        strip_step(xd, x0, xa, false, C.ihz, sm + C.L.zbm + at_z, sm + C.L.zbk + at_z,
                                                C.ni * C.L.zb, mine, c);
                    }
                }
                // sF -= r * (F1_x + F1_z), per point fmaf(-r, c, s)
#pragma unroll
                for (int f = 0; f < 3; ++f)
#pragma unroll
                    for (int h = 0; h < 2; ++h) s[f][h] = pfma(pr(-rr[2 * h], -rr[2 * h + 1]), c[f][h], s[f][h]);
            }
        }
    }
    const float4 pu = ld4(n0);
    float ou[Q], ov[Q], ow[Q];
    advance4(uc, pu, s[0], ou);
    advance4(vc, ld4(n0 + fs), s[1], ov);
    advance4(wc, ld4(n0 + 2 * fs), s[2], ow);
    const int zq = e.w & 0xff, c = (e.w >> 8) & 0xff;
    if constexpr (GENERAL) {
        const int j = C.j0 + zq * Q, i = C.i0 + c;
        if (P.mode == MODE_FWD) {
            // the next step's injection (fwd_PDE_exact_MNAD.m:111): stored U holds it
            if ((e.x & RQ_SOURCE) && i == C.src_col && S.tt < P.nt) {
                const float a = P.src_amp[S.tt];
                if (a != 0.0f) {
#pragma unroll
                    for (int k = 0; k < Q; ++k)
                        if (j + k == C.src_row) ou[k] += a;
                }
            }
        } else if ((e.x & RQ_INJECT) && S.tt < P.nt) {
            // Born_adj_MNAD.m:109-111: the residual of step tt+1 enters U after the update
            float inj[Q];
            if (C.inj_scan) {
#pragma unroll
                for (int k = 0; k < Q; ++k) inj[k] = 0.0f;
                injection(P, S.tt, (j / TMA_TZ) + (i / TMA_TX) * P.ntz, i % TMA_TX, (i + HX) * P.ld + (j + HZ), inj);
            } else {
                ldv(sm + S.inj + (e.w >> 16) * Q, inj);
            }
#pragma unroll
            for (int k = 0; k < Q; ++k) ou[k] -= inj[k];
        }
        if (e.x & RQ_PAST) {
#pragma unroll
            for (int k = 0; k < Q; ++k)
                if (j + k >= P.nz) ou[k] = ov[k] = ow[k] = 0.0f;   // rows past nz are the zero halo
        }
    }
    if (!mine) return;
    stv(n0, ou);
    stv(n0 + fs, ov);
    stv(n0 + 2 * fs, ow);
    if ((e.x & RQ_EDGE) && S.out) {
        if (c < 2 || c >= C.ni - 2) {
            uint4* w = S.out + (c < 2 ? c : c - C.ni + 4) * C.nj + zq * Q;
#pragma unroll
            for (int k = 0; k < Q; ++k) publish(w + k, ou[k], ov[k], ow[k], S.tag);
        } else {
            uint4* w = S.out + 4 * C.nj + c;
            if (zq == 0) {
                publish(w, ou[0], ov[0], ow[0], S.tag);
                publish(w + C.ni, ou[1], ov[1], ow[1], S.tag);
            }
            if (zq == C.nj / Q - 1) {
                publish(w + 2 * C.ni, ou[2], ov[2], ow[2], S.tag);
                publish(w + 3 * C.ni, ou[3], ov[3], ow[3], S.tag);
            }
        }
    }
    if (S.snap_step) snapshot(P, S, C.j0 + zq * Q, C.i0 + c, s[0], uc, pu, peak);
}

// mnad_update_pairs at one point.
template <bool POINT_ORDER>
__device__ __forceinline__ void update_point(const Coefs2& K, float r, const Hood& h, float* s)
{
    const float q = __fmul_rn(r, r);
    const float u2 = h.u00 + h.u00, v2 = h.v00 + h.v00, w2 = h.w00 + h.w00;
    const float dUz = (h.uzm + h.uzp) - u2, dUx = (h.uxm + h.uxp) - u2;
    const float dVz = (h.vzm + h.vzp) - v2, dVx = (h.vxm + h.vxp) - v2;
    const float dWz = (h.wzm + h.wzp) - w2, dWx = (h.wxm + h.wxp) - w2;
    const float uLx = h.uxm - h.uxp, uLz = h.uzm - h.uzp, nvX1 = h.vxm - h.vxp, vX2 = h.vxm2 - h.vxp2;
    const float wZ1 = h.wzp - h.wzm, wZ2 = h.wzm2 - h.wzp2;
    // row sums of the side columns
    const float su0 = h.umm + h.ump, su1 = h.upm + h.upp, sw0 = h.wmm + h.wmp, sw1 = h.wpm + h.wpp;
    const float uDz = su0 - su1, wDz = sw1 - sw0;
    float dUd, uDx, dVd, nvDx, vXZ, dWd, wXZ;
    if constexpr (POINT_ORDER) {
        dUd = ((h.umm + h.upp) + (h.upm + h.ump)) - (u2 + u2);
        uDx = (h.umm + h.upm) - (h.ump + h.upp);
        const float vA = h.vmm + h.vpp, vB = h.vpm + h.vmp, wA = h.wmm + h.wpp, wB = h.wpm + h.wmp;
        dVd = (vA + vB) - (v2 + v2);
        nvDx = (h.vmm + h.vpm) - (h.vmp + h.vpp);
        vXZ = vA - vB;
        dWd = (wA + wB) - (w2 + w2);
        wXZ = wA - wB;
    } else {
        const float dv0 = h.vmm - h.vmp, dv1 = h.vpm - h.vpp;
        dUd = (su0 + su1) - (u2 + u2);
        uDx = (h.umm - h.ump) + (h.upm - h.upp);
        dVd = ((h.vmm + h.vmp) + (h.vpm + h.vpp)) - (v2 + v2);
        nvDx = dv0 + dv1;
        vXZ = dv0 - dv1;
        dWd = (sw0 + sw1) - (w2 + w2);
        wXZ = (h.wmm - h.wmp) - (h.wpm - h.wpp);
    }
    auto al = [&](int k) { return K.alpha[k].x; };
    auto be = [&](int k) { return K.beta[k].x; };
    float a = __fmul_rn(al(K_UU_Z), dUz);
    a = fmaf(al(K_UU_X), dUx, a);
    a = fmaf(al(K_UV_X1), nvX1, a);
    a = fmaf(al(K_UV_X2), vX2, a);
    a = fmaf(al(K_UW_Z1), wZ1, a);
    a = fmaf(al(K_UW_Z2), wZ2, a);
    float b = __fmul_rn(be(K_UU_Z), dUz);
    b = fmaf(be(K_UU_X), dUx, b);
    b = fmaf(be(K_UU_D), dUd, b);
    b = fmaf(be(K_UV_X1), nvX1, b);
    b = fmaf(be(K_UV_D), nvDx, b);
    b = fmaf(be(K_UV_X2), vX2, b);
    b = fmaf(be(K_UW_Z1), wZ1, b);
    b = fmaf(be(K_UW_D), wDz, b);
    b = fmaf(be(K_UW_Z2), wZ2, b);
    s[0] = fmaf(q, b, __fmul_rn(r, a));
    a = __fmul_rn(al(K_VV_Z), dVz);
    a = fmaf(al(K_VV_X), dVx, a);
    a = fmaf(al(K_VV_R), h.v00, a);
    a = fmaf(al(K_VU_X1), uLx, a);
    a = fmaf(al(K_VU_D), uDx, a);
    a = fmaf(al(K_VW), wXZ, a);
    b = __fmul_rn(be(K_VV_Z), dVz);
    b = fmaf(be(K_VV_X), dVx, b);
    b = fmaf(be(K_VV_D), dVd, b);
    b = fmaf(be(K_VV_R), h.v00, b);
    b = fmaf(be(K_VU_X1), uLx, b);
    b = fmaf(be(K_VU_D), uDx, b);
    b = fmaf(be(K_VW), wXZ, b);
    s[1] = fmaf(q, b, __fmul_rn(r, a));
    a = __fmul_rn(al(K_WW_Z), dWz);
    a = fmaf(al(K_WW_X), dWx, a);
    a = fmaf(al(K_WW_R), h.w00, a);
    a = fmaf(al(K_WU_Z1), uLz, a);
    a = fmaf(al(K_WU_D), uDz, a);
    a = fmaf(al(K_WV), vXZ, a);
    b = __fmul_rn(be(K_WW_Z), dWz);
    b = fmaf(be(K_WW_X), dWx, b);
    b = fmaf(be(K_WW_D), dWd, b);
    b = fmaf(be(K_WW_R), h.w00, b);
    b = fmaf(be(K_WU_Z1), uLz, b);
    b = fmaf(be(K_WU_D), uDz, b);
    b = fmaf(be(K_WV), vXZ, b);
    s[2] = fmaf(q, b, __fmul_rn(r, a));
}

// One direction of the CPML of one field at one point (cpml_mem2 at a point):
// m1, m2, m3 at m, m + vs, m + 2 vs; returns the new m1.
__device__ __forceinline__ float strip_point(const float* c, float ih, float fd, float f0, float fa, bool low, float* m,
                                             int vs)
{
    const float gr = low ? fd - fa : fa - fd, lap = (fd + fa) - (f0 + f0), ih2 = __fmul_rn(ih, ih);
    const float g2 = __fmul_rn(__fmul_rn(c[1], ih), gr), hg = __fmul_rn(0.5f, g2);
    const float m3 = fmaf(c[0], m[2 * vs], hg);
    const float t2 = fmaf(lap, ih2, -m3), b2 = fmaf(c[0], m[vs], g2);
    const float m2 = fmaf(c[2], t2, b2);
    const float t1 = fmaf(2.0f * lap, ih2, -m2), b1 = fmaf(c[0], m[0], hg);
    const float m1 = fmaf(c[2], t1, b1);
    m[0] = m1;
    m[vs] = m2;
    m[2 * vs] = m3;
    return m1;
}

// One point: the new U, V, W into S.nxt, and the cell out if other patches need
// it.  Where everything of the point lies is in its table entry, built once: worked
// out in every step it cost more instructions than the stencil (197 integer to
// 131 FP32 per point; a step of 201 x 201 2.26 -> 2.16 us, of 300 x 300 2.87 -> 2.70).
template <bool POINT_ORDER>
__device__ __forceinline__ void point_step(const Coefs2& K, const PropDesc& P, const PatchCtx& C, const StepCtx& S,
                                           float* sm, const uint4 e, float& peak)
{
    constexpr int X = RES_PITCH;
    const int fs = C.L.fs, o = e.x & 0xffff;
    const float *u = S.cur + o, *v = u + fs, *w = v + fs;
    float* n = S.nxt + o;
    const float r = sm[C.L.r + (e.y & 0xffff)];
    Hood h;
    h.u00 = u[0]; h.uzm = u[-1]; h.uzp = u[1]; h.uxm = u[-X]; h.uxp = u[X];
    h.umm = u[-X - 1]; h.upm = u[-X + 1]; h.ump = u[X - 1]; h.upp = u[X + 1];
    h.v00 = v[0]; h.vzm = v[-1]; h.vzp = v[1]; h.vxm = v[-X]; h.vxp = v[X];
    h.vmm = v[-X - 1]; h.vpm = v[-X + 1]; h.vmp = v[X - 1]; h.vpp = v[X + 1]; h.vxm2 = v[-2 * X]; h.vxp2 = v[2 * X];
    h.w00 = w[0]; h.wzm = w[-1]; h.wzp = w[1]; h.wxm = w[-X]; h.wxp = w[X];
    h.wmm = w[-X - 1]; h.wpm = w[-X + 1]; h.wmp = w[X - 1]; h.wpp = w[X + 1]; h.wzm2 = w[-2]; h.wzp2 = w[2];
    float s[3];
    update_point<POINT_ORDER>(K, r, h, s);
    if (e.x & (RQ_X | RQ_TOP | RQ_BOTTOM)) {
        // the CPML sees U before this step's injection (fwd_PDE_exact_MNAD.m:95-111)
        float u0 = h.u00, uxm = h.uxm, uxp = h.uxp, uzm = h.uzm, uzp = h.uzp;
        if (e.x & RQ_SOURCE) {
            const float amp = P.src_amp[S.tt - 1];
            const int dj = C.src_row - C.j0 - (int)(e.w & 0xff), di = C.src_col - C.i0 - (int)((e.w >> 8) & 0xff);
            if (dj == 0 && di == 0) u0 -= amp;
            else if (di == -1) uxm -= amp;
            else if (di == 1) uxp -= amp;
            else if (dj == -1) uzm -= amp;
            else uzp -= amp;
        }
        float cp[3] = {0.0f, 0.0f, 0.0f};
        if (e.x & RQ_X) {
            const bool low = !(e.x & RQ_RIGHT);
            const int at = e.y >> 16, vs = C.vsx;
            const float* kc = sm + C.L.xk + at;
            const float k[3] = {kc[0], kc[vs], kc[2 * vs]};
            float* m = sm + C.L.xm + at;
            cp[0] += strip_point(k, C.ihx, uxm, u0, uxp, low, m, vs);
            cp[1] += strip_point(k, C.ihx, h.vxm, h.v00, h.vxp, low, m + 3 * vs, vs);
            cp[2] += strip_point(k, C.ihx, h.wxm, h.w00, h.wxp, low, m + 6 * vs, vs);
        }
        if (e.x & (RQ_TOP | RQ_BOTTOM)) {
            const bool low = e.x & RQ_TOP;
            const int at = e.z & 0xffff, vs = low ? C.vst : C.vsb;
            const float* kc = sm + (low ? C.L.ztk : C.L.zbk) + at;
            const float k[3] = {kc[0], kc[vs], kc[2 * vs]};
            float* m = sm + (low ? C.L.ztm : C.L.zbm) + at;
            cp[0] += strip_point(k, C.ihz, uzm, u0, uzp, low, m, vs);
            cp[1] += strip_point(k, C.ihz, h.vzm, h.v00, h.vzp, low, m + 3 * vs, vs);
            cp[2] += strip_point(k, C.ihz, h.wzm, h.w00, h.wzp, low, m + 6 * vs, vs);
        }
#pragma unroll
        for (int f = 0; f < 3; ++f) s[f] = fmaf(-r, cp[f], s[f]);
    }
    // nF = F + ((F - pF) + sF)
    const float pu = n[0];
    float ou = h.u00 + ((h.u00 - pu) + s[0]);
    float ov = h.v00 + ((h.v00 - n[fs]) + s[1]);
    float ow = h.w00 + ((h.w00 - n[2 * fs]) + s[2]);
    if (P.mode == MODE_FWD) {
        // the next step's injection (fwd_PDE_exact_MNAD.m:111): stored U holds it
        if ((e.x & RQ_SOURCE) && S.tt < P.nt && C.j0 + (int)(e.w & 0xff) == C.src_row &&
            C.i0 + (int)((e.w >> 8) & 0xff) == C.src_col)
            ou += P.src_amp[S.tt];
    } else if ((e.x & RQ_INJECT) && S.tt < P.nt) {
        // Born_adj_MNAD.m:109-111: the residual of step tt+1 enters U after the update
        const int j = C.j0 + (int)(e.w & 0xff), i = C.i0 + (int)((e.w >> 8) & 0xff);
        float inj = 0.0f;
        if (C.inj_scan) inj = adjoint_injection(P, S.tt, (j / TMA_TZ + (i / TMA_TX) * P.ntz) * TMA_TX + i % TMA_TX,
                                                (size_t)(i + HX) * P.ld + (j + HZ));
        else inj = sm[S.inj + (e.w >> 16)];
        ou -= inj;
    }
    if (e.x & RQ_PAST) ou = ov = ow = 0.0f;               // rows past nz are the zero halo
    n[0] = ou;
    n[fs] = ov;
    n[2 * fs] = ow;
    if (S.out && (e.x & RQ_EDGE)) publish(S.out + (e.z >> 16), ou, ov, ow, S.tag);
    if (S.snap_step && (e.x & RQ_IMAGE)) {
        const int d = P.d, j = C.j0 + (int)(e.w & 0xff), i = C.i0 + (int)((e.w >> 8) & 0xff), niz = P.nz - 2 * d;
        const size_t nint = (size_t)niz * (P.nx - 2 * d), q = (size_t)(j - d) + (size_t)(i - d) * niz;
        // fwd_PDE_exact_MNAD.m:128-141; nU - 2U + pU = su
        float d2u = s[0];
        if (S.tt == 1) d2u = fmaf(2.0f, h.u00, s[0] - pu);
        else if (S.tt == 2) d2u = s[0] - pu;
        d2u *= P.inv_dt2;
        const int slot = P.snap_stage ? 0 : S.tq - 1 - P.snap_col0;
        if ((P.snap_flags & SNAP_WRITE) && slot >= 0 && slot < P.snap_cols) {
            const size_t at = (size_t)slot * nint + q;
            if (P.codec == CODEC_BF16) static_cast<__nv_bfloat16*>(P.snap)[at] = __float2bfloat16_rn(d2u);
            else static_cast<float*>(P.snap)[at] = d2u;
            peak = fmaxf(peak, fabsf(d2u));
        }
        if (P.snap_flags & SNAP_ILLUM) accumulate_product(&P.illum[q], d2u, d2u);
    }
}

// Distance terms of 4 points in the x strip (C_cof.m), and in the z strip of a
// side: 0 for rows outside it, whose coefficients are then exactly (1, 0, 0).
__device__ __forceinline__ void x_distance(const PropDesc& P, int i, float* X)
{
    const float x = i < P.d ? float(P.d - i) * P.dx : float(i - (P.nx - P.d) + 1) * P.dx;
#pragma unroll
    for (int k = 0; k < Q; ++k) X[k] = x;
}
__device__ __forceinline__ void z_distance(const PropDesc& P, int side, int j, float* X)
{
#pragma unroll
    for (int k = 0; k < Q; ++k) {
        const int jk = j + k;
        X[k] = 0.0f;
        if (side == 0 && jk < P.d) X[k] = float(P.d - jk) * P.dz;
        if (side == 1 && jk >= P.nz - P.d && jk < P.nz) X[k] = float(jk - (P.nz - P.d) + 1) * P.dz;
    }
}

// Coefficients of a group's strip points from their r (time-invariant).
template <bool POINT_ORDER>
__device__ __forceinline__ void strip_coefs(const PropDesc& P, float K, const float* r, const float* X, float* out,
                                            int stride)
{
    float4 o[3];
    float* c1 = reinterpret_cast<float*>(&o[0]);
    float* c2 = reinterpret_cast<float*>(&o[1]);
    float* c3 = reinterpret_cast<float*>(&o[2]);
#pragma unroll
    for (int m = 0; m < 2; ++m) {
        const float2 r2 = pr(r[2 * m], r[2 * m + 1]), idt = pr(P.inv_dt, P.inv_dt);
        float2 v;
        if constexpr (POINT_ORDER) v = pmul(pr(__fsqrt_rn(r2.x), __fsqrt_rn(r2.y)), idt);
        else v = pmul(pmul(r2, pr(rsqrtf(r2.x), rsqrtf(r2.y))), idt);
        const CpmlC c = cpml_c2<POINT_ORDER>(K, v, pr(X[2 * m], X[2 * m + 1]), P.dt);
        c1[2 * m] = c.c1.x; c1[2 * m + 1] = c.c1.y;
        c2[2 * m] = c.c2.x; c2[2 * m + 1] = c.c2.y;
        c3[2 * m] = c.c3.x; c3[2 * m + 1] = c.c3.y;
    }
#pragma unroll
    for (int v = 0; v < 3; ++v) *reinterpret_cast<float4*>(out + v * stride) = o[v];
}

// The memory variables of a patch between global and shared memory.
template <bool STORE>
__device__ __forceinline__ void move_strips(const PropDesc& P, const ResPatch& p, const ResLayout& L, float* sm)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    const int nqz = p.nj / Q, nj = p.nj, ni = p.ni, i0 = p.i0, d = P.d, nx = P.nx;
    auto move = [&](float* s, float* g) {
        if (STORE) *reinterpret_cast<float4*>(g) = *reinterpret_cast<const float4*>(s);
        else *reinterpret_cast<float4*>(s) = __ldcg(reinterpret_cast<const float4*>(g));
    };
#pragma unroll 4
    for (int k = warp; k < 9 * L.xcols; k += nwarps) {
        const int v = k / L.xcols, xc = k - v * L.xcols, side = xc < L.xleft ? 0 : 1;
        const int kx = side ? max(i0, nx - d) - (nx - d) + (xc - L.xleft) : i0 + xc;
        if (lane < nqz)
            move(sm + L.xm + k * nj + 4 * lane, P.mx + ((size_t)(side * 9 + v) * d + kx) * P.ld + p.j0 + 4 * lane);
    }
    for (int side = 0; side < 2; ++side) {
        const int rows = side ? L.zb : L.zt, k0 = side ? L.zb_first - P.zb0 : p.j0;
        if (rows == 0) continue;
        float* base = sm + (side ? L.zbm : L.ztm);
        // lanes over (column, 4-row unit) of a variable
        const int nu = rows / Q, per = 32 / nu, sub = lane / nu, u = lane - sub * nu;
#pragma unroll 4
        for (int k = warp * per + sub; k < 9 * ni; k += nwarps * per) {
            const int v = k / ni, c = k - v * ni;
            if (sub < per)
                move(base + k * rows + 4 * u, P.mz + ((size_t)(side * 9 + v) * nx + i0 + c) * P.dpz + k0 + 4 * u);
        }
    }
}

// B halo cells per lane, from number k0 on, into the staged field `nxt`; false
// if a wait ran out.  The polls are unconditional and back to back (past the
// end the last cell again), so a round costs one trip through L2.
template <int B>
__device__ __forceinline__ bool collect(const uint4* in, const int2* halo, int nhalo, float* nxt, int fs, unsigned tag,
                                        int k0, int comm, const ResArgs& A)
{
    int at[B];
    const uint4* w[B];
#pragma unroll
    for (int m = 0; m < B; ++m) {
        const int2 h = halo[min(k0 + comm * m, nhalo - 1)];
        w[m] = in + h.x;
        at[m] = h.y;
    }
    for (unsigned it = 1;; ++it) {
        Cell x[B];
#pragma unroll
        for (int m = 0; m < B; ++m) x[m] = peek(w[m]);
        bool here = true;
#pragma unroll
        for (int m = 0; m < B; ++m) here &= x[m].tag == tag;
        if (here) {
#pragma unroll
            for (int m = 0; m < B; ++m) {
                nxt[at[m]] = __uint_as_float(x[m].u);
                nxt[fs + at[m]] = __uint_as_float(x[m].v);
                nxt[2 * fs + at[m]] = __uint_as_float(x[m].w);
            }
            return true;
        }
        if (it >= A.spin_limit || ((it & 1023u) == 0 && (*reinterpret_cast<volatile unsigned*>(A.status) & ST_TIMEOUT)))
            return false;
    }
}

// FP16 codec: encodes the patch's part of the staged snapshot number tq (from
// 1) with the scale that the largest |d2u| of all patches gives (f16_absmax and
// f16_encode); all threads together; false if a wait ran out.  A patch publishes
// maximum tq + 2 over tq only after it has encoded tq + 1, for which it polled
// every patch's maximum tq + 1, published after that patch had encoded tq.
__device__ __noinline__ bool encode(const PropDesc& P, const PatchCtx& C, float* sm, int tq, const ResArgs& A)
{
    const int tid = threadIdx.x, nthr = blockDim.x;
    unsigned* peak = reinterpret_cast<unsigned*>(sm + C.L.misc) + 6;
    bool bad = false;
    for (int k = tid; k < A.npatch && !bad; k += nthr) {
        const uint4* w = C.peaks + (size_t)(tq & 1) * A.npatch + k;
        for (unsigned it = 1;; ++it) {
            const Cell x = peek(w);
            if (x.tag == (unsigned)tq) {
                if (x.u > 0) atomicMax(peak, x.u);
                break;
            }
            if (it >= A.spin_limit || ((it & 1023u) == 0 && (*reinterpret_cast<volatile unsigned*>(A.status) & ST_TIMEOUT))) {
                bad = true;
                break;
            }
        }
    }
    if (__syncthreads_or(bad)) return false;
    float s, inv;
    f16_scale(__uint_as_float(*peak), s, inv);
    const int d = P.d, niz = P.nz - 2 * d;
    const size_t nint = (size_t)niz * (P.nx - 2 * d);
    const int ja = max(C.j0, d), n = min(C.j0 + C.nj, P.nz - d) - ja, ia = max(C.i0, d), m = min(C.i0 + C.ni, P.nx - d) - ia;
    if (tq <= P.nsnap && C.me == 0 && tid == 0) P.enc_scale[tq - 1] = s;
    if (tq <= P.nsnap && n > 0) {
        const int lane = tid & 31;
        for (int c = tid >> 5; c < m; c += nthr >> 5) {
            const size_t q = (size_t)(ja - d) + (size_t)(ia + c - d) * niz;
            const float* from = static_cast<const float*>(P.snap) + q;
            __half* to = static_cast<__half*>(P.enc) + (size_t)(tq - 1) * nint + q;
            for (int r = lane; r < n; r += 32) to[r] = __float2half_rn(__ldcg(from + r) * inv);
        }
    }
    __syncthreads();
    if (tid == 0) *peak = 0;
    return true;
}

template <bool POINT_ORDER, bool SMALL>
__device__ __forceinline__ void resident_body(const ResArgs& A)
{
    extern __shared__ __align__(128) float sm[];
    __shared__ __align__(16) PropDesc P;
    __shared__ PatchCtx C;
    static_assert(sizeof(PropDesc) + sizeof(PatchCtx) + 16 <= RES_SMEM_STATIC, "the dynamic part leaves no room for these");
    const int tid = threadIdx.x, nthr = blockDim.x, lane = tid & 31, warp = tid >> 5;
    const int pi = blockIdx.x / A.npatch, me = blockIdx.x - pi * A.npatch;
    {
        const int n = sizeof(PropDesc) / 8;
        const unsigned long long* src = reinterpret_cast<const unsigned long long*>(A.props + pi);
        for (int k = tid; k < n; k += nthr) reinterpret_cast<unsigned long long*>(&P)[k] = __ldg(src + k);
    }
    const int4 pq = __ldg(A.patches + me);
    const ResPatch patch{pq.x, pq.y, pq.z, pq.w};
    __syncthreads();
    // the steps of this launch in which the propagation advances
    const int sa = max(A.s0, max(P.s_begin, P.s_off)), sb = min(A.s1, min(P.s_end, P.s_off + P.nt));
    if (sa >= sb) return;
    const int nz = P.nz, nx = P.nx, d = P.d, ld = P.ld;
    const ResLayout L = res_layout(patch, nz, nx, d, SMALL);
    const int j0 = patch.j0, nj = patch.nj, i0 = patch.i0, ni = patch.ni, nqz = nj / Q;
    uint4* qtab = reinterpret_cast<uint4*>(sm + L.qtab);
    unsigned* qinj = reinterpret_cast<unsigned*>(sm + L.qinj);
    int2* halo = reinterpret_cast<int2*>(sm + L.halo);
    int2* recs = reinterpret_cast<int2*>(sm + L.recs);
    int* misc = reinterpret_cast<int*>(sm + L.misc);     // 0: halo cells, 1: receivers, 2: injection slots,
                                                         // 3: duplicate receivers, 4, 5: largest |d2u| of a
                                                         // snapshot by step parity, 6: of all patches, 8, 9: the
                                                         // step's image column by step parity, 16..: groups per warp and class
    // ---- load the patch: a warp per staged column, a few columns in flight ----
    const int nwarps = nthr >> 5;
    {
        const int nu = nqz + 2, cols = ni + 4;            // 16-byte units of a staged column
        const int c0 = sa & 1;
#pragma unroll 4
        for (int k = warp; k < 6 * cols; k += nwarps) {
            const int f6 = k / cols, c = k - f6 * cols, lvl = f6 >= 3, f = f6 - lvl * 3;
            const float* src = P.fld[lvl][f] + (size_t)(i0 + c) * ld + j0;
            for (int u = lane; u < nu; u += 32) {
                const bool own = c >= 2 && c < ni + 2 && u >= 1 && u <= nqz;
                // the previous level's halo is never read before it is written (zero outside the grid)
                float4 x = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
                if (own || lvl == c0) x = __ldcg(reinterpret_cast<const float4*>(src + 4 * u));
                *reinterpret_cast<float4*>(sm + f6 * L.fs + c * RES_PITCH + 4 * u) = x;
            }
        }
#pragma unroll 4
        for (int c = warp; c < ni; c += nwarps)
            if (lane < nqz)
                *reinterpret_cast<float4*>(sm + L.r + c * nj + 4 * lane) =
                    __ldg(reinterpret_cast<const float4*>(P.r + (size_t)(i0 + c + HX) * ld + j0 + HZ + 4 * lane));
    }
    move_strips<false>(P, patch, L, sm);
    // ---- tables --------------------------------------------------------------
    for (int k = tid; k < L.nquads; k += nthr) qinj[k] = 0;
    for (int k = tid; k < 2 * 4 * RES_RECS; k += nthr) sm[L.inj + k] = 0.0f;
    for (int k = tid; k < 128; k += nthr) misc[k] = 0;
    __syncthreads();
    // the strips' coefficients, once: they depend on the model only
    {
        float X[Q];
        for (int k = tid; k < L.xcols * nqz; k += nthr) {
            const int xc = k / nqz, u = k - xc * nqz;
            const int c = xc < L.xleft ? xc : max(i0, nx - d) - i0 + (xc - L.xleft);
            x_distance(P, i0 + c, X);
            strip_coefs<POINT_ORDER>(P, P.kx, sm + L.r + c * nj + 4 * u, X, sm + L.xk + xc * nj + 4 * u, L.xcols * nj);
        }
        for (int side = 0; side < 2; ++side) {
            const int rows = side ? L.zb : L.zt, nu = rows / Q, jf = side ? L.zb_first : j0;
            for (int k = tid; k < ni * nu; k += nthr) {
                const int c = k / nu, u = k - c * nu;
                z_distance(P, side, jf + 4 * u, X);
                strip_coefs<POINT_ORDER>(P, P.kz, sm + L.r + c * nj + (jf - j0) + 4 * u, X,
                                         sm + (side ? L.zbk : L.ztk) + c * rows + 4 * u, ni * rows);
            }
        }
    }
    // receivers of the patch: those beyond the table's size, or two at one
    // point of an adjoint, are looked up in the buckets at every step instead
    const bool fwd = P.mode == MODE_FWD;
    for (int k = tid; k < P.nr; k += nthr) {
        const int pt = __ldg(P.rec_pt + k), ic = pt / ld, lr = pt - ic * ld - HZ - j0, lc = ic - HX - i0;
        if (lr < 0 || lr >= nj || lc < 0 || lc >= ni) continue;
        const int n = atomicAdd(&misc[1], 1);
        if (n < RES_RECS) recs[n] = make_int2(k, lc << 16 | lr);
        if (!fwd) atomicOr(&qinj[lc * nqz + lr / Q], RQ_INJECT);
    }
    // halo cells: which published word each one is (the patch list, searched
    // for the owner of every cell, comes into the exchange area meanwhile)
    int4* const list = reinterpret_cast<int4*>(sm + L.inj);
    static_assert(2 * RES_RECS >= RES_MAX_PATCHES + RES_MAX_PATCHES / 4, "the patch list fits the injection area");
    int* const first = reinterpret_cast<int*>(list + RES_MAX_PATCHES);
    if (A.npatch > 1) {
        for (int k = tid; k < A.npatch; k += nthr) list[k] = __ldg(A.patches + k);
        for (int k = tid; k <= A.nbands; k += nthr) first[k] = __ldg(A.band_first + k);
        __syncthreads();
        for (int k = tid; k < L.nhalo; k += nthr) {
            int lr, lc;
            if (k < 4 * nj) {                             // two columns on each side
                const int s = k / nj;
                lr = k - s * nj;
                lc = s < 2 ? s - 2 : ni + s - 2;
            } else if (k < 4 * nj + 4 * ni) {             // two rows above and below
                const int s = (k - 4 * nj) / ni;
                lc = (k - 4 * nj) - s * ni;
                lr = s < 2 ? s - 2 : nj + s - 2;
            } else {                                      // the four diagonal neighbours
                const int s = k - 4 * nj - 4 * ni;
                lr = s & 1 ? nj : -1;
                lc = s & 2 ? ni : -1;
            }
            const int j = j0 + lr, i = i0 + lc;
            if (j < 0 || j >= nz || i < 0 || i >= nx) continue;
            int b = 0;                                    // the band of row j, then its patch of column i
            while (b + 1 < A.nbands && list[first[b + 1]].x <= j) ++b;
            int lo = first[b], hi = first[b + 1] - 1;
            while (lo < hi) {
                const int mid = (lo + hi + 1) / 2;
                if (list[mid].z <= i) lo = mid; else hi = mid - 1;
            }
            const int4 o = list[lo];
            halo[atomicAdd(&misc[0], 1)] = make_int2(lo * A.slots + res_slot(o.y, o.w, j - o.x, i - o.z),
                                                     (lc + 2) * RES_PITCH + lr + 4);
        }
        __syncthreads();
        for (int k = tid; k < 2 * 4 * RES_RECS; k += nthr) sm[L.inj + k] = 0.0f;
    }
    __syncthreads();
    const int nhalo = misc[0], nrec = min(misc[1], RES_RECS);
    if (!fwd && misc[1] <= RES_RECS)
        for (int k = tid; k < L.nquads; k += nthr)
            if (qinj[k] != 0) qinj[k] |= (unsigned)atomicAdd(&misc[2], 1);
    __syncthreads();
    if (!fwd && misc[1] <= RES_RECS) {
        for (int k = tid; k < nrec; k += nthr) {
            const int lc = recs[k].y >> 16, lr = recs[k].y & 0xffff;
            const int at = (int)(qinj[lc * nqz + lr / Q] & 0xffff) * Q + lr % Q;
            recs[k].y = at;
            if (atomicAdd(reinterpret_cast<int*>(sm + L.inj) + at, 1) > 0) misc[3] = 1;
        }
    } else if (fwd) {
        for (int k = tid; k < nrec; k += nthr) {
            const int lc = recs[k].y >> 16, lr = recs[k].y & 0xffff;
            recs[k] = make_int2(__ldg(P.rec_id + recs[k].x), (lc + 2) * RES_PITCH + lr + 4);
        }
    }
    __syncthreads();
    const bool scan = misc[1] > RES_RECS || misc[3] != 0;
    for (int k = tid; k < 2 * 4 * RES_RECS; k += nthr) sm[L.inj + k] = 0.0f;
    // the groups by class, each class column by column: each warp classifies a
    // run of groups, the counts per warp and class give every warp its places
    const int zs = P.src >= 0 ? P.src % ld - HZ : -8, xsrc = P.src >= 0 ? P.src / ld - HX : -8;
    const int run = (L.nquads + nwarps * 32 - 1) / (nwarps * 32) * 32, q0 = warp * run, q1 = min(q0 + run, L.nquads);
    if constexpr (SMALL)
        for (int n = tid; n < nj * ni; n += nthr) {
            const int c = n / nj, lr = n - c * nj, j = j0 + lr, i = i0 + c;
            const unsigned inj = qinj[c * nqz + lr / Q];
            unsigned fl = inj & RQ_INJECT;
            if (i < d) fl |= RQ_X;
            else if (i >= nx - d) fl |= RQ_X | RQ_RIGHT;
            if (j < d) fl |= RQ_TOP;
            else if (j >= nz - d && j < nz) fl |= RQ_BOTTOM;
            if (P.src >= 0 && abs(i - xsrc) + abs(j - zs) <= 1) fl |= RQ_SOURCE;
            if (j >= nz) fl |= RQ_PAST;
            if (i >= d && i < nx - d && j >= d && j < nz - d) fl |= RQ_IMAGE;
            const int slot = A.npatch > 1 ? res_slot(nj, ni, lr, c) : -1;
            if (slot >= 0) fl |= RQ_EDGE;
            const int xc = i < d ? c : L.xleft + (i - max(i0, nx - d));
            uint4 e;
            e.x = (unsigned)((c + 2) * RES_PITCH + 4 + lr) | fl;
            e.y = (unsigned)n | (fl & RQ_X ? (unsigned)(xc * nj + lr) << 16 : 0u);
            e.z = (fl & RQ_TOP ? (unsigned)(c * L.zt + lr) : fl & RQ_BOTTOM ? (unsigned)(c * L.zb + j - L.zb_first) : 0u) |
                  (slot >= 0 ? (unsigned)slot << 16 : 0u);
            e.w = (unsigned)lr | (unsigned)c << 8 | ((inj & 0xffff) * Q + lr % Q) << 16;
            qtab[n] = e;
        }
    for (int pass = 0; pass < 2 && !SMALL; ++pass) {
        int at[RES_CLASSES] = {0, 0, 0, 0};
        if (pass == 1) {
            int before = 0;
#pragma unroll
            for (int cls = 0; cls < RES_CLASSES; ++cls)
                for (int w = 0; w < nwarps; ++w) {
                    if (w == warp) at[cls] = before;
                    before += misc[16 + w * RES_CLASSES + cls];
                }
        }
        for (int k0 = q0; k0 < q1; k0 += 32) {
            const int k = k0 + lane;
            uint4 e = make_uint4(0, 0, 0, 0);
            int mine = -1;
            if (k < q1) {
                const int c = k / nqz, zq = k - c * nqz, j = j0 + zq * Q, i = i0 + c;
                unsigned fl = qinj[k] & RQ_INJECT;
                if (i < d) fl |= RQ_X;
                else if (i >= nx - d) fl |= RQ_X | RQ_RIGHT;
                if (j < d) fl |= RQ_TOP;
                if (d > 0 && j + Q - 1 >= nz - d) fl |= RQ_BOTTOM;
                if (j + Q > nz) fl |= RQ_PAST;
                if (P.src >= 0 && i >= xsrc - 1 && i <= xsrc + 1 && j + Q >= zs && j - 1 <= zs) fl |= RQ_SOURCE;
                if (fl) fl |= RQ_GENERAL;
                if (A.npatch > 1 && (c < 2 || c >= ni - 2 || zq == 0 || zq == nqz - 1)) fl |= RQ_EDGE;
                mine = (fl & RQ_EDGE ? 0 : 2) + (fl & RQ_GENERAL ? 0 : 1);
                const int xc = i < d ? c : L.xleft + (i - max(i0, nx - d));
                e.x = (unsigned)((c + 2) * RES_PITCH + 4 + zq * Q) | fl;
                e.y = (unsigned)(c * nj + zq * Q) | (fl & RQ_X ? (unsigned)(xc * nj + zq * Q) << 16 : 0u);
                e.z = (fl & RQ_TOP ? (unsigned)(c * L.zt + zq * Q) : 0u) |
                      (fl & RQ_BOTTOM ? (unsigned)(c * L.zb + j - L.zb_first) << 16 : 0u);
                e.w = (unsigned)zq | (unsigned)c << 8 | (qinj[k] & 0xffff) << 16;
            }
#pragma unroll
            for (int cls = 0; cls < RES_CLASSES; ++cls) {
                const unsigned m = __ballot_sync(0xffffffffu, mine == cls);
                if (pass == 1 && mine == cls) qtab[at[cls] + __popc(m & ((1u << lane) - 1u))] = e;
                at[cls] += __popc(m);
            }
        }
        // which neighbours a group has in its warp's lanes
        if (pass == 1) __syncthreads();
        for (int k = tid; pass == 1 && k < L.nquads; k += nthr) {
            const unsigned w = qtab[k].w & 0xffff;
            if ((k & 31) > 0 && (qtab[k - 1].w & 0xffff) + 1 == w) qtab[k].x |= RQ_UP;
            if ((k & 31) < 31 && k + 1 < L.nquads && (qtab[k + 1].w & 0xffff) == w + 1) qtab[k].x |= RQ_DOWN;
        }
        if (pass == 0 && lane < RES_CLASSES)
            misc[16 + warp * RES_CLASSES + lane] = lane == 0 ? at[0] : lane == 1 ? at[1] : lane == 2 ? at[2] : at[3];
        __syncthreads();
    }
    if (tid == 0) {
        misc[8] = misc[9] = -1;                           // no step before the first
        C.L = L;
        C.j0 = j0; C.nj = nj; C.i0 = i0; C.ni = ni;
        C.ihx = 1.0f / P.dx;
        C.ihz = 1.0f / P.dz;
        C.src_row = zs;
        C.src_col = xsrc;
        C.inj_scan = scan;
        C.nhalo = nhalo;
        C.nrec = nrec;
        C.single = sb - sa == 1;
        C.vsx = L.xcols * nj;
        C.vst = ni * L.zt;
        C.vsb = ni * L.zb;
        C.ntask = res_tasks(nj, ni, SMALL);
        C.s_end = sb;
        C.plane = (size_t)A.npatch * A.slots;
        C.words = A.words + (size_t)pi * C.plane * 2;
        C.peaks = A.peaks + (size_t)pi * A.npatch * 2;
        C.me = me;
        C.out = A.npatch > 1 ? C.words + (size_t)me * A.slots : nullptr;
    }
    __syncthreads();
    // injection amounts of step s
    auto fill_injection = [&](int s, int k) {
        const int tt = P.nt - (s - P.s_off);
        const int2* recs = reinterpret_cast<const int2*>(sm + C.L.recs);
        sm[C.L.inj + (s & 1) * 4 * RES_RECS + recs[k].y] = tt < P.nt ? __ldg(P.inj + (size_t)tt * P.nr + recs[k].x) : 0.0f;
    };
    if (!fwd && !scan)
        for (int k = tid; k < nrec; k += nthr) fill_injection(sa, k);
    __syncthreads();
    // ---- the steps ------------------------------------------------------------
    int staged = 0;                                       // number of the snapshot that is not encoded yet
    const bool staging = P.snap_stage != 0;
    for (int s = sa; s < C.s_end; ++s) {
        // words of the descriptor and the patch are read again in every step
        // (kept in registers they spill)
        asm volatile("" ::: "memory");
        const int cur = s & 1;
        const bool fwd = P.mode == MODE_FWD;
        const int fs = C.L.fs;
        const uint4* qtab = reinterpret_cast<const uint4*>(sm + C.L.qtab);
        const int2* halo = reinterpret_cast<const int2*>(sm + C.L.halo);
        const int2* recs = reinterpret_cast<const int2*>(sm + C.L.recs);
        StepCtx S;
        S.cur = sm + cur * 3 * fs;
        S.nxt = sm + (cur ^ 1) * 3 * fs;
        S.tt = fwd ? s - P.s_off + 1 : P.nt - (s - P.s_off);
        S.tag = (unsigned)(s + 2);
        bool bad = false;
        const int tid = threadIdx.x, lane = tid & 31;
        const int comm = A.comm, nwork = blockDim.x - comm;   // compute threads; the last warps do the exchange
        if (tid < nwork) {
            S.tq = (int)(((float)S.tt + 0.5f) * P.invT);
            S.snap_step = fwd && P.T > 0 && S.tt - S.tq * P.T == 0;
            S.inj = C.L.inj + (s & 1) * 4 * RES_RECS;
            S.out = C.out && s + 1 < C.s_end ? C.out + ((s + 1) & 1) * C.plane : nullptr;
            const int ntask = C.ntask, warps = nwork >> 5;
            if constexpr (!SMALL) {
                // The warps of an SM sub-partition start one after the other.
                // Released together by the barrier they load together and then
                // compute together, and each pipe idles through the other's
                // phase; staggered by a third of a task they overlap, and the
                // first four warps, which hold the edges, publish earlier.
                // 600 cycles: 481 x 1281 5.45 -> 5.10 us a step, 381 x 681 3.50
                // -> 3.30, 600 x 1200 5.69 -> 5.20 (300: 5.20, 3.38, 5.31; 900:
                // 5.25, 3.21, 5.28; turns passed by named barriers: 5.69, 3.45, 5.74).
                // All of these plans go round twice or more; one round was not measured.
                const unsigned t0 = clock(), wait = (tid >> 7) * RES_STAGGER;
                while ((unsigned)clock() - t0 < wait) {}
            }
            float peak = 0.0f;                                // largest |d2u| of a snapshot
            for (int k = tid >> 5; k < ntask; k += warps) {
                if constexpr (SMALL) {
                    const int n = 32 * k + lane;
                    if (n < C.nj * C.ni) point_step<POINT_ORDER>(A.coef2, P, C, S, sm, qtab[n], peak);
                } else {
                    // the general path if one of the warp's groups needs it
                    const int nquads = C.L.nquads;
                    const bool mine = 32 * k + lane < nquads;
                    const uint4 q = qtab[mine ? 32 * k + lane : nquads - 1];
                    if (__any_sync(0xffffffffu, q.x & RQ_GENERAL))
                        group_step<POINT_ORDER, true>(A.coef2, P, C, S, sm, fs, q, mine, peak);
                    else
                        group_step<POINT_ORDER, false>(A.coef2, P, C, S, sm, fs, q, mine, peak);
                }
            }
            if (S.snap_step && P.snap_stage) {
                const unsigned m = __reduce_max_sync(0xffffffffu, __float_as_uint(peak));
                if (lane == 0 && m > 0) atomicMax(reinterpret_cast<unsigned*>(sm + C.L.misc) + 4 + (s & 1), m);
            }
            // the image terms of the step before, whose U is the current level now
            const int image = reinterpret_cast<const int*>(sm + C.L.misc)[8 + ((s + 1) & 1)];
            if (image >= 0) add_image<SMALL ? 1 : 4>(P, C, S.cur, image, tid >> 5, warps);
        } else {
            // forward receivers (fwd_PDE_exact_MNAD.m:119-123): U after this
            // step's injection, before its update
            auto record = [&](int id, int off) {
                const size_t at = (size_t)id * P.nt + (S.tt - 1);
                const float x = S.cur[off];
                if (!isfinite(x)) atomicOr(P.status, ST_NONFINITE);
                P.data[at] = x;
                if (P.datav) P.datav[at] = S.cur[fs + off];
                if (P.dataw) P.dataw[at] = S.cur[2 * fs + off];
            };
            const int ct = tid - nwork;
            if (ct == 0) {
                const int tq = (int)(((float)S.tt + 0.5f) * P.invT);
                reinterpret_cast<int*>(sm + C.L.misc)[8 + (s & 1)] =
                    !fwd && P.T > 0 && S.tt - tq * P.T == 0 ? image_column(P, tq) : -1;
            }
            if (fwd && !C.inj_scan) {
                for (int k = ct; k < C.nrec; k += comm) record(recs[k].x, recs[k].y);
            } else if (fwd) {
                for (int k = ct; k < P.nr; k += comm) {
                    const int pt = __ldg(P.rec_pt + k), ic = pt / P.ld, lr = pt - ic * P.ld - HZ - C.j0, lc = ic - HX - C.i0;
                    if (lr >= 0 && lr < C.nj && lc >= 0 && lc < C.ni)
                        record(__ldg(P.rec_id + k), (lc + 2) * RES_PITCH + lr + 4);
                }
            }
            if (s + 1 < C.s_end) {
                if (!fwd && !C.inj_scan)
                    for (int k = ct; k < C.nrec; k += comm) fill_injection(s + 1, k);
                const uint4* in = C.words + ((s + 1) & 1) * C.plane;
                const int nhalo = C.nhalo;
                // all cells in one round of polls where 3 or 6 per lane do; more per
                // lane and round than 11 (12, 16, 20) measured the same
                if (nhalo <= 0) {
                } else if (nhalo <= 3 * comm) {
                    bad = !collect<3>(in, halo, nhalo, S.nxt, fs, S.tag, ct, comm, A);
                } else if (nhalo <= 6 * comm) {
                    bad = !collect<6>(in, halo, nhalo, S.nxt, fs, S.tag, ct, comm, A);
                } else {
                    for (int k0 = ct; k0 < nhalo && !bad; k0 += 11 * comm)
                        bad = !collect<11>(in, halo, nhalo, S.nxt, fs, S.tag, k0, comm, A);
                }
            }
        }
        if (__syncthreads_or(bad)) {
            if (tid == 0) atomicOr(A.status, ST_TIMEOUT);
            return;
        }
        if (staging) {
            // the patch's maximum goes out; the snapshot is encoded where all
            // patches' are due: before the next one, or after the last step
            const int tq = (int)(((float)S.tt + 0.5f) * P.invT);
            if (S.tt - tq * P.T == 0) {
                if (tid == 0) {
                    unsigned* m = reinterpret_cast<unsigned*>(sm + C.L.misc) + 4 + (s & 1);
                    publish(C.peaks + (size_t)(tq & 1) * A.npatch + C.me, __uint_as_float(*m), 0.0f, 0.0f, (unsigned)tq);
                    *m = 0;
                }
                staged = tq;
            }
            if (staged > 0 && (s + 1 >= C.s_end || (S.tt + 1) % P.T == 0)) {
                if (!encode(P, C, sm, staged, A)) {
                    if (tid == 0) atomicOr(A.status, ST_TIMEOUT);
                    return;
                }
                staged = 0;
            }
        }
    }
    // ---- write the state back (the layout from shared memory) --------------------
    asm volatile("" ::: "memory");
    const int image = reinterpret_cast<const int*>(sm + C.L.misc)[8 + ((C.s_end + 1) & 1)];
    if (image >= 0)
        add_image<SMALL ? 1 : 4>(P, C, sm + (C.s_end & 1) * 3 * C.L.fs, image, threadIdx.x >> 5, blockDim.x >> 5);
    {
        const ResPatch p{C.j0, C.nj, C.i0, C.ni};
        const int s0 = max(A.s0, max(P.s_begin, P.s_off)), nqe = p.nj / Q, nw = blockDim.x >> 5;
#pragma unroll 4
        for (int k = threadIdx.x >> 5; k < 6 * p.ni; k += nw) {
            const int f6 = k / p.ni, c = k - f6 * p.ni, lvl = f6 >= 3, f = f6 - lvl * 3, u = threadIdx.x & 31;
            // after a single step the current level is unchanged (and may still
            // be loaded by a neighbour)
            if (C.single && lvl == (s0 & 1)) continue;
            if (u < nqe)
                *reinterpret_cast<float4*>(P.fld[lvl][f] + (size_t)(p.i0 + c + HX) * P.ld + p.j0 + HZ + 4 * u) =
                    ld4(sm + f6 * C.L.fs + (c + 2) * RES_PITCH + 4 + 4 * u);
        }
        move_strips<true>(P, p, C.L, sm);
    }
}

}  // namespace

__global__ void __launch_bounds__(RES_THREADS, 1) step_resident(const __grid_constant__ ResArgs A)
{
    resident_body<false, false>(A);
}

__global__ void __launch_bounds__(RES_THREADS, 1) step_resident_point(const __grid_constant__ ResArgs A)
{
    resident_body<true, false>(A);
}

__global__ void __launch_bounds__(RES_POINT_THREADS, 1) step_resident_small(const __grid_constant__ ResArgs A)
{
    resident_body<false, true>(A);
}

__global__ void __launch_bounds__(RES_POINT_THREADS, 1)
step_resident_small_point(const __grid_constant__ ResArgs A)
{
    resident_body<true, true>(A);
}

}  // namespace mnad
