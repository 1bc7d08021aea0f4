// How the on-chip step kernel (step_resident) splits a grid into patches, one
// per CTA, and what a patch keeps in shared memory.  Plain host code apart
// from the layout, which the kernel evaluates too.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstddef>
#include <vector>

#ifdef __CUDACC__
#define MNAD_HD __host__ __device__ __forceinline__
#else
#define MNAD_HD inline
#endif

namespace mnad {

// A staged column: up to RES_MAX_ROWS rows with a 4-row halo above and below
// and 4 rows of padding, so that the pitch is an odd number of 16-byte units
// and lanes in neighbouring columns read different banks.
constexpr int RES_MAX_ROWS = 128;
constexpr int RES_PITCH = RES_MAX_ROWS + 12;
constexpr int RES_MAX_COLS = 255;       // quad table entries hold the column in 8 bits
constexpr int RES_THREADS = 384;        // per CTA at most: 168 registers each
constexpr int RES_POINT_THREADS = 512;  // the same for patches that go point by point: 128
constexpr int RES_RECS = 192;           // receivers of a patch kept in its own table (more: looked up every step)
constexpr int RES_SMALL = 1024;         // points of a patch that goes point by point, at most
constexpr int RES_MAX_PATCHES = 256;    // CTAs of a propagation at most
// a plan on the device, in 16-byte units: the patches, then the bands' first patches
constexpr int RES_TABLE = RES_MAX_PATCHES + (RES_MAX_PATCHES + 1 + 3) / 4;
// Shared memory of a CTA: what the device gives, less the kernel's own static
// part (the descriptor and the patch).
constexpr size_t RES_SMEM_STATIC = 1024;
constexpr size_t RES_SMEM_LIMIT = 227 * 1024 - RES_SMEM_STATIC;

// Rows j0 .. j0+nj-1 (a multiple of 4, rows past nz are zero) and columns
// i0 .. i0+ni-1 of the grid.
struct ResPatch {
    int j0, nj, i0, ni;
};

// Shared memory of a patch, offsets in floats: two time levels of U, V, W
// with halo; r; the CPML memory variables [var 9][column][row] and
// coefficients [3][column][row] of its columns in the x strips, of its rows in
// the top and in the bottom strip; tables.
struct ResLayout {
    int fs;                     // floats per field and level
    int xleft, xcols;           // its columns in the left strip, in both
    int zt, zb, zb_first;       // rows in the top strip, in the bottom strip; first row of those
    int nquads, nhalo;          // 4-row groups; halo cells at most
    int r, xm, ztm, zbm, xk, ztk, zbk, inj, qtab, qinj, halo, recs, misc, total;
};

// small: the patch goes point by point (a table entry per point instead of per group)
MNAD_HD ResLayout res_layout(const ResPatch& p, int nz, int nx, int d, bool small = false)
{
    ResLayout L;
    L.fs = (p.ni + 4) * RES_PITCH;
    const int le = p.i0 + p.ni < d ? p.i0 + p.ni : d, rb = p.i0 > nx - d ? p.i0 : nx - d;
    L.xleft = le > p.i0 ? le - p.i0 : 0;
    L.xcols = L.xleft + (d > 0 && p.i0 + p.ni > rb ? p.i0 + p.ni - rb : 0);
    // 4-row groups that overlap rows [0, d) and [nz - d, nz)
    const int top = d > p.j0 ? ((d - p.j0 + 3) & ~3) : 0;
    L.zt = top < p.nj ? top : p.nj;
    const int zb0 = (nz - d) & ~3;
    L.zb_first = p.j0 > zb0 ? p.j0 : zb0;
    L.zb = d > 0 && p.j0 + p.nj > L.zb_first ? p.j0 + p.nj - L.zb_first : 0;
    L.nquads = p.nj / 4 * p.ni;
    L.nhalo = 4 * p.nj + 4 * p.ni + 4;
    int o = 6 * L.fs;
    L.r = o;      o += p.ni * p.nj;
    L.xm = o;     o += 9 * L.xcols * p.nj;
    L.ztm = o;    o += 9 * p.ni * L.zt;
    L.zbm = o;    o += 9 * p.ni * L.zb;
    L.xk = o;     o += 3 * L.xcols * p.nj;
    L.ztk = o;    o += 3 * p.ni * L.zt;
    L.zbk = o;    o += 3 * p.ni * L.zb;
    L.inj = o;    o += 2 * 4 * RES_RECS;
    L.qtab = o;   o += (small ? 16 : 4) * L.nquads;
    L.qinj = o;   o += L.nquads;
    o = (o + 3) & ~3;
    L.halo = o;   o += 2 * L.nhalo;
    L.recs = o;   o += 2 * RES_RECS;
    L.misc = o;   o += 128;
    L.total = o;
    return L;
}

// Cells of a patch that other patches may need, in publication order: its two
// first and two last columns, then its two first and two last rows.
MNAD_HD int res_slots(int nj, int ni) { return 4 * nj + 4 * ni; }

// Publication slot of the patch's cell (row lr, column lc), -1 if it is not
// within two points of an edge.
MNAD_HD int res_slot(int nj, int ni, int lr, int lc)
{
    if (lc < 2) return lc * nj + lr;
    if (lc >= ni - 2) return (lc - (ni - 2) + 2) * nj + lr;
    if (lr < 2) return 4 * nj + lr * ni + lc;
    if (lr >= nj - 2) return 4 * nj + (lr - (nj - 2) + 2) * ni + lc;
    return -1;
}

struct ResPlan {
    std::vector<ResPatch> patches;      // band by band (z), along x within a band
    std::vector<int> band_first;        // first patch of each band, and the patch count
    size_t smem = 0;                    // bytes of the largest patch
    int slots = 0, threads = 0, comm = 0;  // comm: threads that do the exchange
    bool small = true;                  // all patches go point by point
    double cost = 0;                    // of the costliest patch, in plain quads
    bool ok() const { return !patches.empty() && smem <= RES_SMEM_LIMIT; }
};

// A step of a patch is a list of warp tasks.  If all patches of a plan are
// small they go point by point, 32 to a task: the least latency.  Else a task
// is 32 groups of 4 rows, the patch's edges first.
MNAD_HD int res_tasks(int nj, int ni, bool small)
{
    return ((small ? nj : nj / 4) * ni + 31) / 32;
}

// Cost of a 4-row group whose points lie in a strip, on top of the plain
// stencil's 1, per strip direction.
constexpr double RES_STRIP_COST = 1.0;
// The same where the patches hold RES_FEW points or fewer on average: a step is
// then one or two tasks per warp and the exchange, which a wider patch in the
// interior only lengthens.  201 x 201 2.18 -> 1.94 us a step, 250 x 220 2.38 ->
// 2.20, 300 x 300 2.69 -> 2.57, 96 x 112 1.69 -> 1.73 (350 x 420, 967 points per
// patch, 2.89 -> 2.96: not below RES_FEW).
constexpr double RES_STRIP_COST_FEW = 0.3;
constexpr int RES_FEW = 640;
// Fewer groups per CTA than this do not shorten a step, which then costs the
// exchange of the halo.
constexpr int RES_MIN_QUADS = 32;

// Splits an nz x nx grid (CPML width d) into at most `ncta` patches of about
// equal cost that each fit an SM: bands along z of equal height, each cut
// along x where the running cost reaches the smallest bound for which `ncta`
// patches suffice.  An empty plan if they do not fit.
inline ResPlan res_plan(int nz, int nx, int d, int ncta)
{
    const int nq = (nz + 3) / 4;
    ResPlan best;
    const double all = (double)nq * nx;
    ncta = std::min(ncta, RES_MAX_PATCHES);
    const double strip = (double)nz * nx <= (double)RES_FEW * ncta ? RES_STRIP_COST_FEW : RES_STRIP_COST;
    ncta = (int)std::min<double>(ncta, std::max(1.0, std::ceil(all / RES_MIN_QUADS)));
    const int nb0 = (nq + RES_MAX_ROWS / 4 - 1) / (RES_MAX_ROWS / 4);
    for (int nb = nb0; nb <= std::min(nb0 + 4, nq) && nb <= ncta; ++nb) {
        auto row0 = [&](int b) { return (int)((long long)nq * b / nb) * 4; };
        // cost of columns [0, x) of a band of nj rows
        auto strips = [&](int x) { return std::min(x, d) + std::max(0, x - std::max(nx - d, d)); };
        auto colcost = [&](int j0, int nj) {
            ResPatch p{j0, nj, 0, 1};
            const ResLayout L = res_layout(p, nz, nx, d);
            return nj / 4 + strip * (L.zt + L.zb) / 4;
        };
        auto cut = [&](double bound, std::vector<ResPatch>* out, std::vector<int>* first) {
            int count = 0;
            for (int b = 0; b < nb; ++b) {
                const int j0 = row0(b), nj = row0(b + 1) - j0;
                const double c = colcost(j0, nj), sx = strip * (nj / 4);
                if (first) first->push_back(count);
                int x = 0;
                while (x < nx) {
                    const double base = c * x + sx * strips(x);
                    int lo = x + 1, hi = std::min(nx, x + RES_MAX_COLS);     // largest end within the bounds
                    auto fits = [&](int e) {
                        const ResPatch p{j0, nj, x, e - x};
                        return c * e + sx * strips(e) - base <= bound &&
                               (size_t)res_layout(p, nz, nx, d).total * 4 <= RES_SMEM_LIMIT;
                    };
                    if (!fits(lo)) return -1;
                    while (lo < hi) {
                        const int mid = (lo + hi + 1) / 2;
                        if (fits(mid)) lo = mid; else hi = mid - 1;
                    }
                    if (out) out->push_back(ResPatch{j0, nj, x, lo - x});
                    x = lo;
                    if (++count > ncta) return -1;
                }
            }
            if (first) first->push_back(count);
            return count;
        };
        // bisection between the mean cost of a patch and the best split so far
        double all_cost = 0;
        for (int b = 0; b < nb; ++b)
            all_cost += colcost(row0(b), row0(b + 1) - row0(b)) * nx + strip * (row0(b + 1) - row0(b)) / 4 * strips(nx);
        double lo = all_cost / ncta, hi = best.ok() ? best.cost - 0.5 : all_cost;
        if (hi < lo || cut(hi, nullptr, nullptr) < 0) continue;   // no better, or does not fit at any cost
        for (double m = 2 * lo; !best.ok() && m < hi; m *= 2)
            if (cut(m, nullptr, nullptr) >= 0) hi = m;
        while (hi - lo > 0.5) {
            const double mid = 0.5 * (lo + hi);
            if (cut(mid, nullptr, nullptr) >= 0) hi = mid; else lo = mid;
        }
        ResPlan p;
        cut(hi, &p.patches, &p.band_first);
        p.cost = hi;
        for (const ResPatch& q : p.patches) {
            p.slots = std::max(p.slots, res_slots(q.nj, q.ni));
            // a table entry per point takes 48 bytes more per group than the
            // layout that the cut above was held to
            p.small &= q.nj * q.ni <= RES_SMALL && (size_t)res_layout(q, nz, nx, d, true).total * 4 <= RES_SMEM_LIMIT;
        }
        int tasks = 0;
        for (const ResPatch& q : p.patches) {
            tasks = std::max(tasks, res_tasks(q.nj, q.ni, p.small));
            p.smem = std::max(p.smem, (size_t)res_layout(q, nz, nx, d, p.small).total * 4);
        }
        // one warp does the exchange, two where the compute warps go round as
        // often without the second
        const int warps = (p.small ? RES_POINT_THREADS : RES_THREADS) / 32;
        const int one = (tasks + warps - 2) / (warps - 1), two = (tasks + warps - 3) / (warps - 2);
        p.comm = two == one ? 64 : 32;
        p.threads = 32 * std::max(4, (tasks + one - 1) / one) + p.comm;
        best = std::move(p);
    }
    return best;
}

// ---- on chip or a kernel launched once per step ------------------------------
// One propagation of a launch group over the steps between two returns to the
// host: its steps, the snapshots it takes in them, and what looking up its
// receivers adds to a step of the on-chip kernel (res_scan_us).
struct ResRun {
    int steps, snaps;
    bool f16;
    double scan_us;
};

// Linear fits of measured times (us, GB300), each over the ranges named; the
// terms are what a launch or a step has to do.
//
// On chip, 293 groups of 0.75 to 12 M points (33 x 2000 to 2000 x 100, strips of
// 0 to 40 points): a launch loads the state, builds its tables and stores the
// state (29 to 56 us; standard error of the fit 9 %); a step costs the exchange
// and the groups of the costliest patch (9 %).
inline double res_fixed_us(const ResPlan& p, int wave, int sms)
{
    return 10.5 + 0.154 * p.smem / 1000.0 * (double)p.patches.size() * wave / sms;
}
inline double res_step_us(const ResPlan& p) { return 1.44 + 0.003 * p.cost; }
// Receivers of a propagation beyond what a patch's own table holds (RES_RECS) are
// looked up among all nr of it by that patch's exchange warps at every step: 1024
// in one patch of 481 x 1281 5.4 -> 15.2 us a step, 4096 48.6; with two such warps
// (321 x 641) 3.4 -> 6.9 and 25.9; the first 1.7 us pass beside the other warps'
// work.  An adjoint looks them up where it injects: 1024 6.0 -> 9.7 us, 4096 22.9.
// Without the on-chip kernel they cost next to nothing (201 x 201, all 40,000 points
// of it: 7.5 instead of 0.34 ms for 60 steps).
inline double res_scan_us(int nr, int comm, bool forward)
{
    return forward ? std::max(0.0, 0.0105 * nr * 32 / comm - 1.7) : 0.0043 * nr;
}
// Receivers in the patch that holds the most of them (rows zr, columns xr, from 0).
inline int res_most_receivers(const ResPlan& p, const std::vector<int>& zr, const std::vector<int>& xr)
{
    std::vector<int> held(p.patches.size(), 0);
    int most = 0;
    for (size_t k = 0; k < zr.size(); ++k) {
        size_t b = 0;                                 // the band of the row, then the patch of the column
        while (b + 2 < p.band_first.size() && p.patches[p.band_first[b + 1]].j0 <= zr[k]) ++b;
        const auto first = p.patches.begin() + p.band_first[b], last = p.patches.begin() + p.band_first[b + 1];
        const auto o = std::upper_bound(first, last, xr[k], [](int x, const ResPatch& q) { return x < q.i0; }) - 1;
        most = std::max(most, ++held[o - p.patches.begin()]);
    }
    return most;
}
// A step of the persistent kernels (same groups, 11 %): the launch, the
// bytes of the tiles with their z halo, the strips along z and along x.  Of the
// one-thread-per-point kernel: 96 x 112 to 768 x 768.
constexpr double TMA_LAUNCH_US = 4.8, DIRECT_LAUNCH_US = 3.8;
inline double step_prop_us(int nz, int nx, int d, int tile_cols)
{
    const double m = 1e-6, z = 2.0 * d * nx, x = 2.0 * d * nz;
    if (tile_cols == 0) return m * (20.0 * nz * nx + 8.0 * (z + x));
    return m * (6.6 * ((nz + 63) / 64 * 64 + 22) * (double)((nx + tile_cols - 1) / tile_cols * tile_cols) + 10.5 * x + 18.8 * z);
}

// Whether the on-chip kernel is expected to run the group's propagations (the
// longest first, `wave` of them to a launch) faster than the persistent kernel on
// tiles of `tile_cols` columns (0: the one-thread-per-point kernel).  A state that
// is loaded and stored for a few steps only, or many propagations that each fill
// the SMs, are where it is not (time on chip / without):
//   600 x 1100 d 20, 16 propagations: 8 steps 1.64, 36 steps 1.04, 104 steps 0.90;
//   128 x 128 d 20, 256: 8 steps 1.54, 24 steps 1.05, 100 steps 0.85;
//   2000 x 100 d 40, 60: 104 steps 1.20, a step alone 1.11;
//   481 x 1281 d 40, 19: 104 steps 0.76; 2: 6 steps 1.02, 8 steps 0.9.
// FP16 snapshots at every step (600 x 1100 d 20, 32 forwards) 1.17, every fourth 1.03.
// The 5 % are held against the fits' error: of those 293 groups 4 run slower than
// without the on-chip kernel at 104 steps (by 8 % at most, 512 x 512 d 40), 29 without
// this rule (by 21 % at most); at 400 steps 1 (by 2 %).
inline bool res_pays(const ResPlan& p, int wave, int sms, int nz, int nx, int d, int tile_cols, const std::vector<ResRun>& runs)
{
    double chip = 0, other = 0;
    const double prop = step_prop_us(nz, nx, d, tile_cols), mpts = 1e-6 * nz * nx;
    for (size_t k0 = 0; k0 < runs.size(); k0 += wave) {
        double scan = 0, snaps = 0;
        for (size_t k = k0; k < std::min(runs.size(), k0 + wave); ++k) {
            const ResRun& r = runs[k];
            scan = std::max(scan, r.scan_us);
            // a snapshot: stored by the step itself; an FP16 one is read again and encoded
            snaps = std::max(snaps, r.snaps * (r.f16 ? 0.009 : 0.0028) * p.cost);
            other += r.steps * prop + r.snaps * (r.f16 ? 3.3 + 7.5 * mpts : 3.0 * mpts);
        }
        chip += res_fixed_us(p, wave, sms) + runs[k0].steps * (res_step_us(p) + scan) + snaps;
    }
    if (!runs.empty()) other += runs[0].steps * (tile_cols ? TMA_LAUNCH_US : DIRECT_LAUNCH_US);
    return chip <= 0.95 * other;
}

}  // namespace mnad
