// Line-scheduled exact triangular solves for matrices on structured grids.
//
// Replaces, like the box schedule (xs_trsv_tiles.cuh), the level-ordered
// sync-free solve that stands in for the reference's Lcsr_trsv_sync_free /
// Ucsc_trsv_sync_free (hip/Precond/gpuparilu.cpp:257-364), for triangles
// whose entries lie on at most 32 grid diagonals (7-point and 27-point
// ILU(0), ParILUT fill of a stencil).
//
// What bounds an exact solve on a grid is its dependency chain: 382 rows one
// after another at 128^3, 7-point.  The box schedule pays about three times
// that many steps (every box on the critical path walks all its levels) plus
// a staged wait per box.  Here a thread owns a whole grid line (all x of one
// (y, z)) and a CTA owns a patch of lines; the CTA marches over the linear
// schedule
//     step(x, Y, Z) = x + al*Y + be*Z,   Y = y + c*z,  Z = z
// (c, al, be: the smallest non-negative integers for which every dependency
// has Y and Z no larger and a smaller step), one step of all its lines
// between two barriers.  The chain is then the schedule's length, with no
// step walked twice, plus one hand-off latency per patch on the way.
//
//   compute threads   one line each (KC columns of one line with several
//                     right-hand sides); a step reads its dependencies from
//                     a shared-memory ring of the last RL steps, indexed
//                     [step][line] with the halo lines beside the patch's
//                     own, and sums its entries in the order and with the
//                     operations of the CPU reference's LUsolve
//                     (hip/HostMatrix/HostMatrixCSR.cpp:385-409): FP64
//                     results are bitwise those of the other exact solves
//   poller warps      read the halo lines' values from the exchange buffer
//                     that the owning patches publish into (a NaN bit
//                     pattern no arithmetic produces marks a value not yet
//                     published, every wait bounded) and run ahead of the
//                     compute threads as far as the ring allows
//   staging warps     bring the factor data NS stages ahead (one bulk copy
//                     each for values, diagonal and masks, stored in exactly
//                     the order they are used) and the right-hand side
//   draining warps    write finished steps to the output along x, so that
//                     vectors stay in natural order and accesses coalesce
//
// Measured on B200, an LU solve in FP64, boxes / lines: 128^3 7-point
// 932 / 317 us, 80^3 27-point 2006 / 568 us, 128^2 5-point 87 us (197 us in
// one CTA), eight right-hand sides at 96^3 919 / 397 us.  One patch alone
// (16*8 lines of 2000, 7-point) takes 392 cycles a step, of which the sums are
// 40 and storing, a barrier and reading back 67; a row of eight patches takes
// 6 us more per hand-off, and at 128^3 (22 hand-offs on the way, 128 CTAs) a
// step of the chain comes to 817 cycles, half of them hand-offs; DRAM stays
// below 10 % of its rate.
//
// Patches are taken by ticket in an order in which dependencies come first,
// so a CTA only waits on patches that running CTAs hold: no co-residency is
// needed.  The exchange buffer is doubled: a launch publishes into one half
// and re-arms the other for the next launch.
#pragma once
#include <climits>
#include <vector>
#include "xs_internal.cuh"
#include "xs_spmv.cuh"
#include "xs_trsv_tiles.cuh"

namespace xs {

constexpr int LINE_DIAG_MAX = 32;   // entries per row: bits of the row mask
// lines per patch for D diagonals: a compile-time constant of the kernels.
// Four warps hide each other's gaps where a step is a few sums; with more
// diagonals the step is bound by instructions and shared-memory traffic, and
// twice as many CTAs take it.
__host__ __device__ constexpr int line_patch(int D) { return D == 2 || D == 3 ? 128 : 64; }
constexpr int LINE_HALO_MAX = 64;   // halo lines per patch
constexpr int LINE_HELPERS = 128;   // staging threads, and as many draining threads
constexpr int LINE_WINDOW = 8;      // steps polled at once
constexpr int LINE_STEP = 8;        // steps per patch are a multiple of this (the longest stage)
constexpr size_t LINE_SMEM_MAX = 222 * 1024;

// Geometry of a line schedule (passed by value to the kernels).
struct LineGeo {
    int n = 0, nx = 0, ny = 0, nz = 0;
    int c = 0, al = 0, be = 0;
    int L = 0, ty = 0, tz = 0;       // lines per patch = ty * tz (Y fastest)
    int ry = 0, rz = 0, py = 0, npad = 0;  // reach, ring columns: (tz+rz) rows of py = ty+ry
    int npy = 0, npz = 0, npatch = 0, nsteps = 0;
    int D = 0, E = 0, nh = 0, maxd = 0;  // diagonals, exported lines, halo lines, longest step distance
    int delta[LINE_DIAG_MAX] = {}, shift[LINE_DIAG_MAX] = {}, offq[LINE_DIAG_MAX] = {};
    int back[LINE_DIAG_MAX] = {};  // ring distance of a diagonal's value: delta rows and shift columns
    // first logical index of line (Yl, Zl) of patch (pY, pZ), or -1 outside the grid
    __host__ __device__ int line_q0(int pY, int pZ, int Yl, int Zl) const
    {
        const int Z = pZ * tz + Zl, y = pY * ty + Yl - c * Z;
        if (Z < 0 || Z >= nz || y < 0 || y >= ny) return -1;
        return (Z * ny + y) * nx;
    }
    __host__ __device__ long slots() const { return (long)npatch * nsteps * L; }
    __host__ __device__ bool mask8() const { return D == 2 || D == 3; }
};

constexpr int LINE_NS_MAX = 8;  // most stages

// shared-memory layout of a CTA (byte offsets)
struct LineSmem {
    size_t ring, rhs, pv, dinv, mask, tab, total;
    int Ps, RS;  // ring columns per step (odd), right-hand-side columns per step (odd)
    // nv: values per row in the stream (the diagonals', or twice as many for the factorisation)
    static __host__ __device__ LineSmem of(const LineGeo &g, int nv, int S, int NS, int RL, int KC, size_t vb, size_t fb,
                                           size_t db, size_t mb)
    {
        auto al = [](size_t b) { return (b + 127) & ~(size_t)127; };
        LineSmem m;
        m.Ps = g.npad | 1;
        m.RS = (g.L * KC) | 1;
        m.ring = 0;
        m.rhs = m.ring + al((size_t)2 * RL * m.Ps * KC * vb);  // every step twice, RL rows apart
        m.pv = m.rhs + al((size_t)NS * S * m.RS * vb);
        m.dinv = m.pv + al((size_t)NS * S * nv * g.L * fb);
        m.mask = m.dinv + al((size_t)NS * S * g.L * db);
        m.tab = m.mask + al((size_t)NS * S * g.L * mb);
        m.total = m.tab + al((size_t)g.L * 4 * sizeof(int));
        return m;
    }
};

// Stage length, stage count and ring length that fit in shared memory: two
// CTAs per SM when there are more patches than SMs, stages as long as
// possible (fewer hand-offs between the warps), the ring long enough for the
// pollers to run ahead.
struct LineCfg {
    int S = 0, NS = 0, RL = 0;
    size_t smem = 0;
};
inline LineCfg line_cfg(const LineGeo &g, int nv, int items, int KC, size_t vb, size_t fb, size_t db, size_t mb, int sms)
{
    LineCfg c;
    int best = -1;
    for (size_t lim : {items > sms ? (size_t)112 * 1024 : LINE_SMEM_MAX, LINE_SMEM_MAX}) {
        for (int RL : {64, 32})
            for (int S = LINE_STEP; S >= 1; S /= 2)
                for (int NS = LINE_NS_MAX; NS >= 3; NS--) {
                    const int ahead = RL - g.maxd - S;  // steps the pollers run ahead
                    if (ahead < 8 || RL < 2 * S) continue;
                    const size_t b = LineSmem::of(g, nv, S, NS, RL, KC, vb, fb, db, mb).total;
                    if (b > lim) continue;
                    if (lim != LINE_SMEM_MAX && NS * S < 12) continue;  // too little in flight to share an SM
                    const int score = std::min(NS * S, 24) * 10000 + S * 1000 + std::min(ahead, 16) * 10 + (8 - NS);
                    if (score <= best) continue;
                    best = score;
                    c.S = S; c.NS = NS; c.RL = RL; c.smem = b;
                }
        if (best >= 0) break;
    }
    return c;
}

// device copy of a schedule's tables (in TriDev)
struct LinePlan {
    LineGeo g;
    // in one buffer: pY, pZ of each patch in ticket order; ticket rank of
    // patch (pY, pZ), -1: no lines; Yl, Zl of each halo line (relative to the
    // patch); per line of a patch its index among the exported lines, or -1
    DBuf<int> tab;
    const int *patch = nullptr, *rank_of = nullptr, *halo = nullptr, *exp_of = nullptr;
    DBuf<uint8_t> mask8;
    DBuf<uint32_t> mask32;
    int brk = -1;       // debugging: rank of a patch made to wait for a value of its own
};

// exchange buffer of one consumer (a preconditioner's own solves, or a batch)
template <typename VT>
struct LineXchg {
    DBuf<VT> x;  // two halves, and behind them the ticket and the current half
    size_t half = 0;
    unsigned *ctl() const { return (unsigned *)(x.p + 2 * half); }
};

// Host half of the plan from a detected grid.  False when the pattern does
// not qualify: more than 32 diagonals, over a quarter of padding, a reach
// beyond a patch, or lines too short for the schedule's skew (more than
// four slots per row).
struct LineHost {
    LineGeo g;
    std::vector<int> patch, rank_of, halo, exp_of;
    // the tables into the plan's buffer, in the order of its pointers
    void upload(LinePlan &P, cudaStream_t s) const
    {
        std::vector<int> all;
        const int **at[4] = {&P.patch, &P.rank_of, &P.halo, &P.exp_of};
        const std::vector<int> *v[4] = {&patch, &rank_of, &halo, &exp_of};
        size_t off[4];
        for (int k = 0; k < 4; k++) {
            off[k] = all.size();
            all.insert(all.end(), v[k]->begin(), v[k]->end());
        }
        P.g = g;
        P.tab.alloc(std::max<size_t>(all.size(), 1));
        P.tab.upload(all.data(), all.size(), s);
        XS_CUDA(cudaStreamSynchronize(s));  // `all` goes out of scope
        for (int k = 0; k < 4; k++) *at[k] = P.tab.p + off[k];
    }
};

inline bool line_layout(int n, long nnz, const TileGrid &G, int sms, LineHost &h)
{
    const int D = (int)(G.vecs.size() / 3);
    if (D < 1 || D > LINE_DIAG_MAX || (long)D * n > nnz + nnz / 4) return false;
    auto ceil_div = [](int a, int b) { return a >= 0 ? (a + b - 1) / b : -((-a) / b); };  // b > 0
    LineGeo g;
    g.n = n; g.nx = G.nx; g.ny = G.ny; g.nz = G.nz;
    g.D = D;
    std::vector<int> ord(D), dy(D), dz(D), dx(D);
    int c = 0;
    for (int k = 0; k < D; k++) {
        dx[k] = G.vecs[3 * k];
        dy[k] = G.vecs[3 * k + 1];
        dz[k] = G.vecs[3 * k + 2];
        ord[k] = k;
        if (dz[k] < 0) c = std::max(c, ceil_div(dy[k], -dz[k]));
    }
    g.c = c;
    auto dY = [&](int k) { return dy[k] + c * dz[k]; };
    int al = 0, be = 0;
    for (int k = 0; k < D; k++)
        if (dz[k] == 0 && dy[k] < 0) al = std::max(al, ceil_div(dx[k] + 1, -dy[k]));
    for (int k = 0; k < D; k++)
        if (dz[k] < 0) be = std::max(be, ceil_div(dx[k] + al * dY(k) + 1, -dz[k]));
    g.al = al;
    g.be = be;
    // diagonals in increasing logical offset: the order of a row's sum
    auto offq = [&](int k) { return dx[k] + dy[k] * g.nx + dz[k] * g.nx * g.ny; };
    std::sort(ord.begin(), ord.end(), [&](int a, int b) { return offq(a) < offq(b); });
    for (int k = 0; k < D; k++) {
        const int q = ord[k];
        if (k > 0 && offq(ord[k - 1]) == offq(q)) return false;
        g.offq[k] = offq(q);
        g.delta[k] = -(dx[q] + al * dY(q) + be * dz[q]);
        if (g.delta[k] < 1 || dY(q) > 0 || dz[q] > 0) return false;
        g.maxd = std::max(g.maxd, g.delta[k]);
        g.ry = std::max(g.ry, -dY(q));
        g.rz = std::max(g.rz, -dz[q]);
    }
    if (g.maxd > 32) return false;
    // patch shape: the cheapest of the power-of-two shapes by a model of the
    // chain (steps and hand-offs), the factor stream and the steps all
    // patches take on the GPU's SMs (microseconds; the constants are early
    // estimates that rank the shapes: a 7-point step takes 0.2 us alone, a
    // hand-off 4 to 6)
    const int Yext = g.ny + c * (g.nz - 1);
    double best = 1e300;
    {
        const int L = line_patch(D);
        for (int ty = 1; ty <= L; ty *= 2) {
            const double ts = (100.0 + 20.0 * D) / 1900.0, th = 0.6;
            const int tz = L / ty;
            if (ty < g.ry || tz < g.rz) continue;
            const int npy = (Yext + ty - 1) / ty, npz = (g.nz + tz - 1) / tz;
            // steps of a patch (a patch wider than the domain ends with its last line)
            const int ns = (g.nx + al * (std::min(ty, Yext) - 1) + be * (std::min(tz, g.nz) - 1) + LINE_STEP - 1) /
                           LINE_STEP * LINE_STEP;
            // patches that hold lines (the sheared domain is a parallelogram)
            long np = 0;
            for (int p = 0; p < npz; p++) {
                const int z0 = p * tz, z1 = std::min(g.nz, z0 + tz) - 1;
                np += (c * z1 + g.ny - 1) / ty - (c * z0) / ty + 1;
            }
            if (np * ns * L > 4L * n + 65536) continue;  // mostly padding
            const double chain = (g.nx + al * (double)(Yext - 1) + be * (double)(g.nz - 1)) * ts + (npy + npz - 2) * th;
            const double stream = (double)np * ns * L * (8.0 * D + 24.0) / 5.5e6;
            const double work = (double)np * ns * ts / sms;
            const double cost = std::max(chain, work) + 0.5 * stream;
            LineGeo t = g;
            t.L = L; t.ty = ty; t.tz = tz;
            t.npad = (ty + g.ry) * (tz + g.rz);
            if (cost < best && line_cfg(t, D, 0, 1, 8, 8, 8, g.mask8() ? 1 : 4, 1).S) {
                best = cost;
                g.L = L; g.ty = ty; g.tz = tz;
                g.npy = npy; g.npz = npz; g.nsteps = ns;
            }
        }
    }
    if (best >= 1e300) return false;
    g.py = g.ty + g.ry;
    g.npad = g.py * (g.tz + g.rz);
    for (int k = 0; k < D; k++) {
        g.shift[k] = -dY(ord[k]) - dz[ord[k]] * g.py;
        g.back[k] = g.delta[k] * (g.npad | 1) + g.shift[k];
    }
    // patches in ticket order: by the step they start at (dependencies start no later), then Z, Y
    std::vector<std::pair<long, int>> order;
    for (int pz = 0; pz < g.npz; pz++)
        for (int py = 0; py < g.npy; py++) {
            bool any = false;
            for (int l = 0; l < g.L && !any; l++) any = g.line_q0(py, pz, l % g.ty, l / g.ty) >= 0;
            if (any) order.push_back({(long)al * g.ty * py + (long)be * g.tz * pz, pz * g.npy + py});
        }
    std::sort(order.begin(), order.end());  // ties: smaller Z, then smaller Y first
    g.npatch = (int)order.size();
    h.patch.clear();
    h.rank_of.assign((size_t)g.npy * g.npz, -1);
    for (int t = 0; t < g.npatch; t++) {
        const int id = order[t].second;
        h.patch.push_back(id % g.npy);
        h.patch.push_back(id / g.npy);
        h.rank_of[id] = t;
    }
    // halo lines a patch reads, and the lines other patches read from it
    std::vector<char> need((size_t)g.npad, 0), exported(g.L, 0);
    for (int l = 0; l < g.L; l++)
        for (int k = 0; k < D; k++) {
            const int Y = l % g.ty + dY(k), Z = l / g.ty + dz[k];
            if (Y < 0 || Z < 0) need[(Z + g.rz) * g.py + Y + g.ry] = 1;
        }
    h.halo.clear();
    for (int p = 0; p < g.npad; p++)
        if (need[p]) {
            const int Y = p % g.py - g.ry, Z = p / g.py - g.rz;
            h.halo.push_back(Y);
            h.halo.push_back(Z);
            exported[((Z + g.tz) % g.tz) * g.ty + (Y + g.ty) % g.ty] = 1;
        }
    g.nh = (int)h.halo.size() / 2;
    if (g.nh > LINE_HALO_MAX) return false;
    h.exp_of.assign(g.L, -1);
    for (int l = 0; l < g.L; l++)
        if (exported[l]) h.exp_of[l] = g.E++;
    if (g.E == 0) g.E = 1;
    h.g = g;
    return true;
}

// ---------------------------------------------------------------- factor data in schedule order
// Slot (patch, step, line) of the schedule at (patch*nsteps + step)*L + line;
// its row's entry k at (patch*nsteps + step)*D*L + k*L + line.  One thread
// per slot, so the writes coalesce; a block covers consecutive steps, so the
// strided reads of consecutive rows of a line share cache lines.
template <bool UPPER>
__device__ __forceinline__ int line_slot_row(const LineGeo &g, const int *__restrict__ patch, long slot)
{
    const int l = (int)(slot % g.L);
    const long ps = slot / g.L;
    const int tau = (int)(ps % g.nsteps), p = (int)(ps / g.nsteps);
    const int Yl = l % g.ty, Zl = l / g.ty;
    const int q0 = g.line_q0(patch[2 * p], patch[2 * p + 1], Yl, Zl);
    const int x = tau - g.al * Yl - g.be * Zl;
    if (q0 < 0 || x < 0 || x >= g.nx) return -1;
    return UPPER ? g.n - 1 - (q0 + x) : q0 + x;
}

// row masks: bit k set when the row has an entry on diagonal k
template <bool UPPER, typename MK>
__global__ void k_line_masks(LineGeo g, const int *__restrict__ patch, const int *__restrict__ rp,
                             const int *__restrict__ ci, MK *mask)
{
    const long m = g.slots();
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < m; s += (long)gridDim.x * blockDim.x) {
        const int r = line_slot_row<UPPER>(g, patch, s);
        uint32_t b = 0;
        if (r >= 0)
            for (int e = rp[r]; e < rp[r + 1]; e++) {
                const int off = UPPER ? r - ci[e] : ci[e] - r;  // logical offset
                for (int k = 0; k < g.D; k++)
                    if (g.offq[k] == off) b |= 1u << k;
            }
        mask[s] = (MK)b;
    }
}

// values: the j-th set bit of a row's mask is its j-th entry in the order of
// the sum (L: increasing column; U: decreasing column)
template <bool UPPER, typename MK, typename FT>
__global__ void k_line_vals(LineGeo g, const int *__restrict__ patch, const MK *__restrict__ mask,
                            const int *__restrict__ rp, const long *__restrict__ src, const double *__restrict__ vals,
                            FT *__restrict__ dst)
{
    const long m = g.slots();
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < m; s += (long)gridDim.x * blockDim.x) {
        const int r = line_slot_row<UPPER>(g, patch, s);
        const uint32_t b = mask[s];
        long e = r >= 0 ? (UPPER ? (long)rp[r + 1] - 1 : (long)rp[r]) : 0;
        FT *o = dst + s / g.L * g.D * g.L + s % g.L;
        for (int k = 0; k < g.D; k++) {
            double v = 0.0;
            if ((b >> k) & 1u) {
                v = vals[src[e]];
                e += UPPER ? -1 : 1;
            }
            if constexpr (std::is_same<FT, double>::value) o[(long)k * g.L] = v;
            else if constexpr (std::is_same<FT, float>::value) o[(long)k * g.L] = (float)v;
            else if constexpr (std::is_same<FT, __nv_bfloat16>::value) o[(long)k * g.L] = __double2bfloat16(v);
            else o[(long)k * g.L] = __double2half(v);
        }
    }
}

template <typename DT>
__global__ void k_line_dinv(LineGeo g, const int *__restrict__ patch, const long *__restrict__ diagsrc,
                            const double *__restrict__ vals, DT *dst)
{
    const long m = g.slots();
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < m; s += (long)gridDim.x * blockDim.x) {
        const int r = line_slot_row<true>(g, patch, s);
        dst[s] = r >= 0 ? (DT)vals[diagsrc[r]] : (DT)0;
    }
}

// ---------------------------------------------------------------- kernel
template <typename VT, typename FT, typename DT>
struct LineArgs {
    const int *patch, *rank_of, *halo, *exp_of;
    const FT *pv;
    const void *mask;
    const DT *dinv;
    VT *xb;          // exchange buffer (two halves)
    long xb_half;
    unsigned *ctl;   // ticket, half
    int S, NS, RL, NP;  // stage length, stages, ring steps, poller warps
    int k, ngroups;  // right-hand sides, column groups (KC columns each)
    const VT *rhs;
    VT *out;
    VT *reset_other;  // a readiness buffer another kernel polls, re-armed row by row (or null)
    const int *done_flag;
    int *err;
    int brk;
};

__device__ __forceinline__ int ld_acquire_cta(const int *p)
{
    int v;
    asm volatile("ld.acquire.cta.shared::cta.b32 %0, [%1];" : "=r"(v) : "r"(smem_u32(p)) : "memory");
    return v;
}
__device__ __forceinline__ void st_release_cta(int *p, int v)
{
    asm volatile("st.release.cta.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(p)), "r"(v) : "memory");
}
// wait until the counter *p reaches target; its value.  Bounded: after 4 s,
// or with an error recorded, the wait is given up
__device__ __forceinline__ int line_wait(const int *p, int target, int *err, unsigned ns)
{
    int v = ld_acquire_cta(p);
    if (v >= target) return v;
    unsigned long long t0 = 0;
    for (long it = 1; (v = ld_acquire_cta(p)) < target; it++) {
        if (ns) __nanosleep(ns);
        if ((it & 4095) == 0) {
            const unsigned long long now = gtimer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > 4 * WAIT_LIMIT_NS) atomicOr(err, DEV_TRSV_TIMEOUT);
            if (*(volatile int *)err) return INT_MAX;
        }
    }
    return v;
}
// the same, but ended by its own limit only: twice that of any chain of waits
// the counter's owner can be in (false: given up, error recorded)
__device__ __forceinline__ bool line_wait_alone(const int *p, int target, int *err, unsigned ns)
{
    unsigned long long t0 = 0;
    for (long it = 1; ld_acquire_cta(p) < target; it++) {
        __nanosleep(ns);
        if ((it & 4095) == 0) {
            const unsigned long long now = gtimer();
            if (t0 == 0) t0 = now;
            else if (now - t0 > 16 * WAIT_LIMIT_NS) {
                atomicOr(err, DEV_TRSV_TIMEOUT);
                return false;
            }
        }
    }
    return true;
}
// loads and stores at 32-bit shared addresses, in program order with the barriers
template <typename T>
__device__ __forceinline__ T lds(uint32_t a)
{
    if constexpr (sizeof(T) == 8) {
        double v;
        asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
        return v;
    } else if constexpr (sizeof(T) == 4) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
        T o;
        memcpy(&o, &v, 4);
        return o;
    } else if constexpr (sizeof(T) == 2) {
        uint16_t v;
        asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a) : "memory");
        T o;
        memcpy(&o, &v, 2);
        return o;
    } else {
        uint32_t v;
        asm volatile("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a) : "memory");
        return (T)v;
    }
}
// the same for a stage's data, which nobody writes while it is read: free to
// move across the step barriers, but not above the wait for the stage, whose
// addresses come from after_wait
__device__ __forceinline__ uint32_t after_wait(uint32_t a)
{
    asm volatile("mov.u32 %0, %0;" : "+r"(a)::"memory");
    return a;
}
template <typename T>
__device__ __forceinline__ T lds_stage(uint32_t a)
{
    if constexpr (sizeof(T) == 8) {
        double v;
        asm("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a));
        return v;
    } else if constexpr (sizeof(T) == 4) {
        uint32_t v;
        asm("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
        T o;
        memcpy(&o, &v, 4);
        return o;
    } else if constexpr (sizeof(T) == 2) {
        uint16_t v;
        asm("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(a));
        T o;
        memcpy(&o, &v, 2);
        return o;
    } else {
        uint32_t v;
        asm("ld.shared.u8 %0, [%1];" : "=r"(v) : "r"(a));
        return (T)v;
    }
}
template <typename T>
__device__ __forceinline__ void sts(uint32_t a, T v)
{
    if constexpr (sizeof(T) == 8) asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
    else asm volatile("st.shared.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}
__device__ __forceinline__ void st_publish_if(bool on, double *p, double v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.relaxed.gpu.global.f64 [%0], %1;\n\t}" ::"l"(p),
                 "d"(v), "r"((uint32_t)on)
                 : "memory");
}
__device__ __forceinline__ void st_publish_if(bool on, float *p, float v)
{
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %2, 0;\n\t@p st.relaxed.gpu.global.f32 [%0], %1;\n\t}" ::"l"(p),
                 "f"(v), "r"((uint32_t)on)
                 : "memory");
}
__device__ __forceinline__ void line_bar(int id, int count)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// the mbarrier gets one (already counted) arrival when this thread's earlier cp.async have landed
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// poller warps for nh halo lines of KC columns (a lane each)
__host__ __device__ constexpr int line_poll_warps(int nh, int KC) { return nh * KC > 32 ? (nh * KC + 31) / 32 : 1; }
__host__ __device__ constexpr int line_threads_max(int KC, int W)
{
    return line_patch(W) * KC + 2 * LINE_HELPERS + 32 * line_poll_warps(LINE_HALO_MAX, KC);
}

// PIVOT: instead of solving, the pivots of an ILU(0) whose eliminations only
// reach the diagonal (see k_line_pairs): rhs and out are A's diagonal and the
// pivots, the stream holds a_ij and a_ji of the W lower entries, and the sum
// subtracts (a_ij / d_j) * a_ji in the order of the reference's IKJ update.
// SU: steps unrolled (a divisor of the stage length).
template <typename VT, typename FT, typename DT, bool UPPER, int KC, int W, bool PIVOT, int SU>
__global__ void __launch_bounds__(line_threads_max(KC, W))
    k_trsv_lines(const __grid_constant__ LineGeo G, const __grid_constant__ LineArgs<VT, FT, DT> A)
{
    using MK = typename std::conditional<(W == 2 || W == 3), uint8_t, uint32_t>::type;
    static_assert(!PIVOT || (W > 0 && !UPPER), "the pivots run on the lower triangle");
    constexpr int L = line_patch(W), T = L * KC, RS = T | 1;
    extern __shared__ __align__(128) unsigned char line_smem[];
    __shared__ __align__(8) uint64_t full[LINE_NS_MAX];
    __shared__ int s_item, s_stop, cdone, drained, hcnt[line_poll_warps(LINE_HALO_MAX, KC)];
    __shared__ unsigned s_half;
    const int D = W > 0 ? W : G.D, NV = PIVOT ? 2 * W : D;
    const int S = A.S, NS = A.NS, RL = A.RL, NP = A.NP;
    const LineSmem M = LineSmem::of(G, NV, S, NS, RL, KC, sizeof(VT), sizeof(FT), UPPER ? sizeof(DT) : 0, sizeof(MK));
    VT *ring = (VT *)(line_smem + M.ring);
    VT *s_rhs = (VT *)(line_smem + M.rhs);
    FT *s_pv = (FT *)(line_smem + M.pv);
    DT *s_dinv = (DT *)(line_smem + M.dinv);
    MK *s_mask = (MK *)(line_smem + M.mask);
    // per line: logical row of step 0 (first row - first active step), first
    // active step (out of reach: no line), ring column
    int4 *s_tab = (int4 *)(line_smem + M.tab);
    const int tid = threadIdx.x;
    const int PsK = M.Ps * KC;
    const int nst = G.nsteps / S;
    const int items = G.npatch * A.ngroups;
    pdl_trigger();
    if (tid == 0) {
        for (int q = 0; q < NS; q++) mbar_init(&full[q], 1 + LINE_HELPERS);
        fence_mbar_init();
    }
    pdl_wait();
    if (A.done_flag && *A.done_flag) return;
    if (tid == 0) {
        s_half = *(volatile unsigned *)(A.ctl + 1);
        s_stop = 0;
    }
    unsigned cnt0 = 0;  // stages consumed by earlier patches of this CTA
    while (true) {
        __syncthreads();  // the previous patch is finished
        if (tid == 0) {
            __threadfence();  // s_half was read before this CTA's ticket is drawn
            const unsigned t = atomicAdd(A.ctl, 1u);
            if (t == (unsigned)(items + gridDim.x - 1)) {  // every CTA has drawn its final ticket
                A.ctl[0] = 0u;
                A.ctl[1] = s_half ^ 1u;
            }
            s_item = (int)t;
            cdone = 0;
            drained = 0;
        }
        if (tid < NP) hcnt[tid] = -G.maxd;
        __syncthreads();
        const int item = s_item;
        if (item >= items) break;
        if (s_stop) continue;  // staging gave up: only the tickets are drawn to the end
        const int rank = item / A.ngroups, grp = item % A.ngroups;
        const int pY = A.patch[2 * rank], pZ = A.patch[2 * rank + 1];
        for (int l = tid; l < L; l += blockDim.x) {
            const int Yl = l % G.ty, Zl = l / G.ty;
            const int q0 = G.line_q0(pY, pZ, Yl, Zl), off = G.al * Yl + G.be * Zl;
            s_tab[l] = make_int4(q0 - off, q0 >= 0 ? off : (1 << 30), ((Zl + G.rz) * G.py + Yl + G.ry) * KC, 0);
        }
        __syncthreads();
        VT *xpub = A.xb + (s_half ? A.xb_half : 0);
        if (tid < T) {
            // ------------------------------------------------ compute
            // One warp per scheduler runs this loop, so a step costs its
            // instructions as much as its latencies: with the ring indexed
            // afresh for every entry through generic pointers a 7-point step
            // took 560 cycles, of which the sums are 40.  So every step is
            // stored twice, RL ring rows apart, an entry is read at a
            // constant distance from a moving row without a wrap (the row
            // returns to the lower copy between stages: RL is a multiple of
            // S), and all addresses are 32-bit shared ones that advance by
            // constants.
            const int l = tid / KC, c = tid % KC;
            const int4 tab = s_tab[l];
            const int e = __ldg(A.exp_of + l);
            const long pstep = (long)G.E * KC;
            VT *pub = xpub + ((long)item * G.nsteps * G.E + max(e, 0)) * KC + c;
            const int xlo = e >= 0 ? tab.y : INT_MAX;  // published steps [xlo, xlo + nx)
            const uint32_t rstep = (uint32_t)(PsK * sizeof(VT)), rlen = (uint32_t)RL * rstep;
            uint32_t row = smem_u32(ring) + rlen + (uint32_t)((tab.z + c) * sizeof(VT));  // in the upper copy
            const uint32_t row_end = row + rlen;
            int avail = -G.maxd;
            bool landed = true;
            int slot = (int)(cnt0 % (unsigned)NS);
            unsigned par = (cnt0 / (unsigned)NS) & 1u;
            uint32_t back[W > 0 ? W : 1];  // ring distance of each diagonal, in bytes
            if constexpr (W > 0) {
#pragma unroll
                for (int k = 0; k < W; k++) back[k] = (uint32_t)(G.back[k] * KC * (int)sizeof(VT));
            }
            const uint32_t a_pv = smem_u32(s_pv) + (uint32_t)(l * sizeof(FT)), a_mk = smem_u32(s_mask) + (uint32_t)(l * sizeof(MK));
            const uint32_t a_dv = smem_u32(s_dinv) + (uint32_t)(l * sizeof(DT)), a_rh = smem_u32(s_rhs) + (uint32_t)(tid * sizeof(VT));
            int tau = 0;
            for (int g = 0; g < nst; g++) {
                if (landed) landed = mbar_wait_bounded(&full[slot], par, A.err);
                line_wait(&drained, (g + 1) * S - RL, A.err, 0);
                const uint32_t first = (uint32_t)(slot * S);
                uint32_t pv = after_wait(a_pv + first * (uint32_t)(NV * L * sizeof(FT)));
                uint32_t mk = after_wait(a_mk + first * (uint32_t)(L * sizeof(MK)));
                uint32_t dv = after_wait(a_dv + first * (uint32_t)(L * sizeof(DT)));
                uint32_t rh = after_wait(a_rh + first * (uint32_t)(RS * sizeof(VT)));
                // a step's own data is loaded during the step before it
                VT rr[2], dd[2];
                uint32_t mm[2];
                constexpr int NVC = W > 0 ? (PIVOT ? 2 * W : W) : 1;
                FT vv[2][NVC];
                auto fetch = [&](int b, uint32_t u) {
                    rr[b] = lds_stage<VT>(rh + u * (uint32_t)(RS * sizeof(VT)));
                    mm[b] = lds_stage<MK>(mk + u * (uint32_t)(L * sizeof(MK)));
                    if constexpr (UPPER) dd[b] = (VT)lds_stage<DT>(dv + u * (uint32_t)(L * sizeof(DT)));
                    if constexpr (W > 0) {
#pragma unroll
                        for (int k = 0; k < NVC; k++)
                            vv[b][k] = lds_stage<FT>(pv + (u * (uint32_t)NVC + (uint32_t)k) * (uint32_t)(L * sizeof(FT)));
                    }
                };
                fetch(0, 0);
                for (int s = 0; s < S; s += SU) {
#pragma unroll
                    for (int u = 0; u < SU; u++) {
                        const int cb = SU > 1 ? (u & 1) : 0, nb = cb ^ 1;
                        // the halo values this step may read (steps before it)
                        if (avail < tau) {
                            avail = line_wait(&hcnt[0], tau, A.err, 0);
                            for (int w = 1; w < NP; w++) avail = min(avail, line_wait(&hcnt[w], tau, A.err, 0));
                        }
                        VT acc;
                        if constexpr (W > 0) {
                            VT y[W];
#pragma unroll
                            for (int k = 0; k < W; k++) y[k] = lds<VT>(row - back[k]);
                            if (u + 1 < SU || s + SU < S) fetch(nb, (uint32_t)(u + 1));
                            acc = rr[cb];
                            if constexpr (UPPER) acc = (VT)(acc * dd[cb]);
#pragma unroll
                            for (int k = 0; k < W; k++) {
                                if constexpr (PIVOT) {
                                    const VT q = vv[cb][k] / y[k];
                                    const VT t = q * vv[cb][W + k];
                                    if ((mm[cb] >> k) & 1u) acc = acc - t;
                                } else {
                                    const VT t = msub(acc, y[k], (VT)FVal<FT>::cvt(vv[cb][k]));
                                    if ((mm[cb] >> k) & 1u) acc = t;
                                }
                            }
                            if constexpr (PIVOT) {
                                if (fabs(acc) < 1e-20) acc = 1e-20;
                            }
                        } else {
                            // chunks of 8 entries, the next chunk's loads before
                            // this one's sum (k is a constant in every copy)
                            VT y[2][8];
                            FT e8[2][8];
                            auto chunk = [&](auto kb_, int b) {
                                constexpr int kb = decltype(kb_)::value;
#pragma unroll
                                for (int j = 0; j < 8; j++) {
                                    const int k = kb + j, kk = k < D ? k : 0;
                                    y[b][j] = lds<VT>(row - (uint32_t)(G.back[k] * KC * (int)sizeof(VT)));
                                    e8[b][j] = lds_stage<FT>(pv + (uint32_t)(kk * L * sizeof(FT)));
                                }
                            };
                            const uint32_t m = mm[cb];
                            auto sum = [&](auto kb_, int b) {
                                constexpr int kb = decltype(kb_)::value;
#pragma unroll
                                for (int j = 0; j < 8; j++) {
                                    const VT t = msub(acc, y[b][j], (VT)FVal<FT>::cvt(e8[b][j]));
                                    if ((m >> (kb + j)) & 1u) acc = t;
                                }
                            };
                            using std::integral_constant;
                            chunk(integral_constant<int, 0>(), 0);
                            acc = rr[cb];
                            if constexpr (UPPER) acc = (VT)(acc * dd[cb]);
                            if (D > 8) chunk(integral_constant<int, 8>(), 1);
                            sum(integral_constant<int, 0>(), 0);
                            if (D > 8) {
                                if (D > 16) chunk(integral_constant<int, 16>(), 0);
                                sum(integral_constant<int, 8>(), 1);
                                if (D > 16) {
                                    if (D > 24) chunk(integral_constant<int, 24>(), 1);
                                    sum(integral_constant<int, 16>(), 0);
                                    if (D > 24) sum(integral_constant<int, 24>(), 1);
                                }
                            }
                            if (s + SU < S) fetch(nb, 1);
                        }
                        // a step outside the line is stored too: no entry names it
                        sts<VT>(row, acc);
                        sts<VT>(row - rlen, acc);
                        st_publish_if((unsigned)(tau - xlo) < (unsigned)G.nx, pub, acc);
                        pub += pstep;
                        row += rstep;
                        tau++;
                        if constexpr (SU == 1) {
                            rr[0] = rr[1];
                            mm[0] = mm[1];
                            if constexpr (UPPER) dd[0] = dd[1];
#pragma unroll
                            for (int k = 0; k < NVC; k++) vv[0][k] = vv[1][k];
                        }
                        line_bar(1, T);
                    }
                    rh += (uint32_t)(SU * RS * sizeof(VT));
                    mk += (uint32_t)(SU * L * sizeof(MK));
                    if (UPPER) dv += (uint32_t)(SU * L * sizeof(DT));
                    pv += (uint32_t)(SU * NV * L * sizeof(FT));
                }
                if (row == row_end) row -= rlen;
                if (tid == 0) st_release_cta(&cdone, tau);
                if (++slot == NS) {
                    slot = 0;
                    par ^= 1u;
                }
            }
        } else if (tid < T + 2 * LINE_HELPERS) {
            // ------------------------------------------------ staging, draining
            const bool drain = tid >= T + LINE_HELPERS;
            const int h = tid - T - (drain ? LINE_HELPERS : 0);
            const long base = (long)rank * G.nsteps;
            const int lg = 31 - __clz(S);  // S is a power of two
            const int nel = T * S;
            // element i of a stage: column i % KC, step i / KC % S, line i / KC / S
            auto element = [&](int i, int tau0, int &l, int &s, int &c, long &o) {
                c = i % KC;
                s = (i / KC) & (S - 1);
                l = (i / KC) >> lg;
                const int4 t = s_tab[l];
                const int tau = tau0 + s, col = grp * KC + c;
                const int q = t.x + tau;
                const int row = UPPER ? G.n - 1 - q : q;
                o = (long)row * A.k + col;
                const bool in = (unsigned)(tau - t.y) < (unsigned)G.nx && (KC == 1 || col < A.k);
                return in ? t.z + c : -1;  // ring column
            };
            if (!drain) {
                auto stage = [&](int g) {
                    const unsigned st = cnt0 + (unsigned)g;
                    const int slot = (int)(st % (unsigned)NS);
                    if (h == 0) {
                        const uint32_t bv = (uint32_t)(S * NV * L * sizeof(FT)), bm = (uint32_t)(S * L * sizeof(MK));
                        const uint32_t bd = UPPER ? (uint32_t)(S * L * sizeof(DT)) : 0u;
                        mbar_expect_tx(&full[slot], bv + bm + bd);
                        bulk_g2s(s_pv + (size_t)slot * S * NV * L, A.pv + (base + (long)g * S) * NV * L, bv, &full[slot]);
                        bulk_g2s(s_mask + (size_t)slot * S * L, (const MK *)A.mask + (base + (long)g * S) * L, bm,
                                 &full[slot]);
                        if (UPPER)
                            bulk_g2s(s_dinv + (size_t)slot * S * L, A.dinv + (base + (long)g * S) * L, bd, &full[slot]);
                    }
                    VT *rb = s_rhs + (size_t)slot * S * RS;
#pragma unroll 4
                    for (int i = h; i < nel; i += LINE_HELPERS) {
                        int l, s, c;
                        long o;
                        if (element(i, g * S, l, s, c, o) >= 0)
                            cp_async_n<sizeof(VT)>(rb + s * RS + l * KC + c, A.rhs + o);
                    }
                    cp_async_mbar_arrive(&full[slot]);
                };
                // This wait does not end with an error of another one: the
                // compute threads go on to the last step with every wait of
                // theirs bounded, and take each stage that is brought, so
                // the barriers' phases stay in step with them.
                int g = 0;
                for (; g < NS && g < nst; g++) stage(g);
                for (; g < nst; g++) {
                    if (!line_wait_alone(&cdone, (g - NS + 1) * S, A.err, 100)) break;
                    stage(g);
                }
                if (g < nst) s_stop = 1;
                // no copy is in flight when the patch ends, whatever happened
                if (h == 0)
                    for (int q = max(0, g - NS); q < g; q++) {
                        const unsigned st = cnt0 + (unsigned)q;
                        if (!mbar_wait_bounded(&full[st % (unsigned)NS], (st / (unsigned)NS) & 1u, A.err)) s_stop = 1;
                    }
            } else {
                // re-arm this patch's part of the other half for the next launch
                VT *xr = A.xb + (s_half ? 0 : A.xb_half) + (long)item * G.nsteps * G.E * KC;
                for (int i = h; i < G.nsteps * G.E * KC; i += LINE_HELPERS) xr[i] = Sentinel<VT>::value();
                for (int g = 0; g < nst; g++) {
                    line_wait(&cdone, (g + 1) * S, A.err, 200);
                    for (int i0 = h; i0 < nel; i0 += 4 * LINE_HELPERS) {
                        VT v[4];
                        long o[4];
#pragma unroll
                        for (int u = 0; u < 4; u++) {
                            const int i = i0 + u * LINE_HELPERS;
                            o[u] = -1;
                            if (i < nel) {
                                int l, s, c;
                                long a;
                                const int rc = element(i, g * S, l, s, c, a);
                                if (rc >= 0) {
                                    v[u] = ring[((g * S + s) & (RL - 1)) * PsK + rc];
                                    o[u] = a;
                                }
                            }
                        }
#pragma unroll
                        for (int u = 0; u < 4; u++)
                            if (o[u] >= 0) {
                                A.out[o[u]] = v[u];
                                if (A.reset_other) A.reset_other[o[u]] = Sentinel<VT>::value();
                            }
                    }
                    line_bar(2, LINE_HELPERS);
                    if (h == 0) st_release_cta(&drained, (g + 1) * S);
                }
            }
        } else {
            // ------------------------------------------------ halo
            // each lane follows one halo line (a column of it): pos is the
            // first step whose value it does not have yet
            const int pw = (tid - T - 2 * LINE_HELPERS) / 32, lane = tid & 31;
            const VT *src = nullptr;  // the value of step pos
            int x1 = 0, pos = INT_MAX, rc = 0;
            const long pstep = (long)G.E * KC;
            {
                const int i = pw * 32 + lane;
                if (i < G.nh * KC) {
                    const int hl = i / KC, c = i % KC;
                    const int Yl = __ldg(A.halo + 2 * hl), Zl = __ldg(A.halo + 2 * hl + 1);
                    if (G.line_q0(pY, pZ, Yl, Zl) >= 0 && (KC == 1 || grp * KC + c < A.k)) {
                        const int dpY = Yl < 0 ? -1 : 0, dpZ = Zl < 0 ? -1 : 0;
                        const int Yo = Yl - dpY * G.ty, Zo = Zl - dpZ * G.tz;  // the line inside its own patch
                        const int ro = __ldg(A.rank_of + (pZ + dpZ) * G.npy + pY + dpY);
                        const int off_o = G.al * Yo + G.be * Zo, off_h = G.al * Yl + G.be * Zl;
                        const int eo = __ldg(A.exp_of + Zo * G.ty + Yo);
                        // active steps [off_h, off_h + nx) here are [off_o, off_o + nx) of the owner
                        src = xpub + (((long)ro * A.ngroups + grp) * G.nsteps + off_o) * pstep + eo * KC + c;
                        pos = off_h;
                        x1 = off_h + G.nx;
                        rc = ((Zl + G.rz) * G.py + Yl + G.ry) * KC + c;
                    }
                }
            }
            const bool brk = A.brk == rank && pw == 0 && lane == 0;  // debugging: a wait that never ends
            bool ok = true;
            int published = -G.maxd;
            unsigned long long t0 = 0;
            long spins = 0;
            while (published < G.nsteps) {
                const int lim = min(ld_acquire_cta(&cdone) + RL - G.maxd, G.nsteps);
                const int m = min(min(lim, x1) - pos, LINE_WINDOW);  // values this lane may take now
                if (m > 0 && ok) {
                    VT v[LINE_WINDOW];
                    const VT *q = src;
#pragma unroll
                    for (int u = 0; u < LINE_WINDOW; u++) {
                        v[u] = Sentinel<VT>::value();
                        if (u < m) v[u] = ld_poll(q);
                        q += pstep;
                    }
                    int r = 0;
#pragma unroll
                    for (int u = 0; u < LINE_WINDOW; u++)
                        if (r == u && !Sentinel<VT>::is(v[u])) r = u + 1;
#pragma unroll
                    for (int u = 0; u < LINE_WINDOW; u++)
                        if (u < r) {
                            VT *w = ring + ((pos + u) & (RL - 1)) * PsK + rc;
                            w[0] = v[u];
                            w[RL * PsK] = v[u];
                        }
                    pos += r;
                    src += r * pstep;
                }
                int mn = pos < x1 && ok ? min(pos, lim) : lim;
                if (brk && ok) mn = min(mn, 0);
                mn = __reduce_min_sync(0xffffffffu, mn);
                if (mn > published) {
                    published = mn;
                    __syncwarp();
                    if (lane == 0) st_release_cta(&hcnt[pw], mn);
                    t0 = 0;
                    spins = 0;
                } else if (mn >= lim) {
                    // the ring is full: the compute threads are behind (their waits are bounded)
                    line_wait(&cdone, lim + G.maxd - RL + 1, A.err, 40);
                    t0 = 0;
                } else if ((++spins & 63) == 0) {
                    const unsigned long long now = gtimer();
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > WAIT_LIMIT_NS) {
                        if (lane == 0) atomicOr(A.err, DEV_TRSV_TIMEOUT);
                        ok = false;
                    }
                    if (*(volatile int *)A.err) ok = false;
                    ok = __all_sync(0xffffffffu, ok);
                }
            }
        }
        cnt0 += (unsigned)nst;
    }
}

// ---------------------------------------------------------------- launch
// columns of one compute line for k right-hand sides: 1, or 2 when the patches
// of all columns would take the SMs several times over.  A line of one column
// has the shorter step; two columns read the factor once.  LU solve with 1 / 2
// columns per line, us: 7-point 48^3 k = 8 125 / 156; 64^3 k = 8 195 / 212, 12
// 247 / 234; 96^3 k = 2 240 / 308, 5 307 / 338, 6 339 / 345, 8 430 / 397; 128^3
// k = 3 389 / 457, 4 454 / 466, 6 599 / 558; 5-point 200^2 k = 16 234 / 316;
// 27-point 40^3 k = 16 310 / 373, 64^3 k = 12 595 / 633, 16 756 / 669, 80^3
// k = 8 712 / 790, 10 808 / 796, 16 1248 / 961.  (Four columns fit at 27
// points only, with stages of one step: 2731 at 80^3 for k = 4.)
// (4, 6 and 9 diagonals have no two-column instance of their own; with one
// column 19-point 60^3 k = 16 takes 553 us.)
constexpr bool line_two_columns(int D) { return D != 4 && D != 6 && D != 9; }
inline int line_kc(const LineGeo &g, int k)
{
    const long sms = geom().sms, most = g.mask8() ? 5 * sms / 2 : 7 * sms;
    if (k < 2 || (long)g.npatch * k <= most || !line_two_columns(g.D)) return 1;
    return line_cfg(g, g.D, 0, 2, sizeof(double), sizeof(double), sizeof(double), g.mask8() ? 1 : 4, 1).S ? 2 : 1;
}

template <typename VT>
inline void line_xchg_ensure(LineXchg<VT> &X, const LineGeo &g, int k, cudaStream_t s)
{
    const int kc = line_kc(g, k), ng = (k + kc - 1) / kc;
    const size_t half = (size_t)g.npatch * ng * g.nsteps * g.E * kc;
    if (X.half == half && X.x.p) return;
    X.x.alloc(2 * half, 2 * sizeof(unsigned) / sizeof(VT) + 1);  // zeroed
    X.half = half;
    k_fill_sentinel<VT><<<256, 256, 0, s>>>(X.x.p, (long)(2 * half));
    check_launch();
}
template <typename VT>
inline void line_xchg_rearm(LineXchg<VT> &X, cudaStream_t s)
{
    if (!X.x.p) return;
    k_fill_sentinel<VT><<<256, 256, 0, s>>>(X.x.p, (long)(2 * X.half));
    XS_CUDA(cudaMemsetAsync(X.ctl(), 0, sizeof(unsigned), s));
}

template <typename VT, typename FT, typename DT, bool UPPER, int KC, bool PIVOT = false>
inline void launch_trsv_lines(const LinePlan &P, const FT *pv, const uint8_t *mask8, const DT *dinv, LineXchg<VT> &X,
                              int k, const VT *rhs, VT *out, VT *reset_other, const int *done_flag, int *err,
                              cudaStream_t s)
{
    const LineGeo &g = P.g;
    const int ng = (k + KC - 1) / KC, items = g.npatch * ng, sms = geom().sms;
    const bool m8 = g.mask8();
    const LineCfg c = line_cfg(g, PIVOT ? 2 * g.D : g.D, items, KC, sizeof(VT), sizeof(FT), UPPER ? sizeof(DT) : 0,
                               m8 ? 1 : 4, sms);
    if (c.S == 0 || !X.x.p || X.half != (size_t)items * g.nsteps * g.E * KC) throw Status(XS_ERR_ORDER);
    LineArgs<VT, FT, DT> A;
    A.patch = P.patch; A.rank_of = P.rank_of; A.halo = P.halo; A.exp_of = P.exp_of;
    A.pv = pv;
    A.mask = m8 ? (const void *)mask8 : (const void *)P.mask32.p;
    A.dinv = dinv;
    A.xb = X.x.p; A.xb_half = (long)X.half; A.ctl = X.ctl();
    A.S = c.S; A.NS = c.NS; A.RL = c.RL;
    A.NP = line_poll_warps(g.nh, KC);
    A.k = k; A.ngroups = ng;
    A.rhs = rhs; A.out = out; A.reset_other = reset_other;
    A.done_flag = done_flag; A.err = err; A.brk = PIVOT ? -1 : P.brk;
    const int threads = line_patch(g.D) * KC + 2 * LINE_HELPERS + 32 * A.NP;
    const int per_sm = c.smem <= 112 * 1024 && 2 * threads <= 2048 ? 2 : 1;
    const int grid = std::min(items, sms * per_sm);
    auto go = [&](auto kern) {
        // the attribute is per function and idempotent: set on every launch (host-side only, no synchronisation)
        XS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LINE_SMEM_MAX));
        launch_pdl(kern, dim3(grid), dim3(threads), c.smem, s, g, A);
    };
    // The ILU(0) triangles of 9- and 13-point 2D and 19- and 27-point 3D
    // patterns (4, 6, 9 and 13 diagonals) have instances of their own, without
    // which the line schedule is behind one CTA up to about 10,000 rows.  LU
    // solve in one CTA / generic instance / its own, us: 9-point 100^2 267 /
    // 300 / 134, 13-point 100^2 293 / 300 / 155, 19-point 12^3 103 / 118 / 61,
    // 27-point 16^3 179 / 167 / 100; 80^3 - / 921 / 568.
    // Unrolled steps: 2 and 4 measured alike, 8 slower (instruction cache), 1
    // slower by a sixth (LU solve 128^3 7-point: 319, 318, 330 and 362 us)
    constexpr int SU = 4;
    const bool unrolled = c.S % SU == 0;
    if (g.D == 3 && unrolled) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 3, PIVOT, SU>);
    else if (g.D == 3) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 3, PIVOT, 1>);
    else if (g.D == 2 && unrolled) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 2, PIVOT, SU>);
    else if (g.D == 2) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 2, PIVOT, 1>);
    else if constexpr (PIVOT) throw Status(XS_ERR_UNSUPPORTED);
    else if (g.D == 13 && c.S % 2 == 0) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 13, false, 2>);
    else if constexpr (KC == 1) {
        if (g.D == 4 && c.S % 2 == 0) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 4, false, 2>);
        else if (g.D == 6 && c.S % 2 == 0) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 6, false, 2>);
        else if (g.D == 9 && c.S % 2 == 0) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 9, false, 2>);
        else go(k_trsv_lines<VT, FT, DT, UPPER, KC, 0, false, 1>);
    } else go(k_trsv_lines<VT, FT, DT, UPPER, KC, 0, false, 1>);
}

// ---------------------------------------------------------------- ILU(0) on the line schedule
// When the sum of a lower and an upper diagonal of A is the main diagonal or
// no diagonal at all (5- and 7-point stencils), an elimination of ILU(0)
// changes nothing but the pivot: u_ij = a_ij, l_ij = a_ij / d_j, and
//     d_i = a_ii - sum_j (a_ij / d_j) * a_ji,
// a recurrence over L's dependencies with one value per row.  It runs on the
// line schedule of the L solve (k_trsv_lines<PIVOT>), with the operations of
// the reference's ilu0_simple in its order, so the factors are bitwise the
// same; the rest of the factor is one elementwise pass (k_line_ilu_finish).
// The lane-group kernel pays a cross-SM hand-off per dependency level: 4.6 ms
// at 128^3 7-point against 0.67 here (pivots 0.40).
inline bool line_ilu_ok(const LinePlan &L, const LinePlan &U)
{
    const LineGeo &a = L.g, &b = U.g;
    if (!a.mask8()) return false;
    auto has = [&](int off) {
        for (int k = 0; k < a.D; k++)
            if (a.offq[k] == off) return true;
        for (int k = 0; k < b.D; k++)
            if (-b.offq[k] == off) return true;
        return false;
    };
    for (int j = 0; j < a.D; j++)
        for (int m = 0; m < b.D; m++) {
            const int s = a.offq[j] - b.offq[m];  // lower + upper (U's offsets are logical: reversed)
            if (s != 0 && has(s)) return false;
        }
    return line_cfg(a, 2 * a.D, 0, 1, 8, 8, 0, 1, 1).S != 0;
}

// the stream of the pivots: per slot a_ij and a_ji of each lower diagonal,
// and the mask of the ones that have both (rp/ci/v: A; uptr: its diagonal)
static __global__ void k_line_pairs(LineGeo g, const int *__restrict__ patch, const int *__restrict__ rp,
                                    const int *__restrict__ ci, const int *__restrict__ uptr,
                                    const double *__restrict__ v, double *__restrict__ pv, uint8_t *__restrict__ mask)
{
    const long m = g.slots();
    for (long s = blockIdx.x * (long)blockDim.x + threadIdx.x; s < m; s += (long)gridDim.x * blockDim.x) {
        const int r = line_slot_row<false>(g, patch, s);
        double *o = pv + s / g.L * (2 * g.D) * g.L + s % g.L;
        uint32_t b = 0;
        int e = r >= 0 ? rp[r] : 0;
        const int e1 = r >= 0 ? uptr[r] : 0;
        for (int k = 0; k < g.D; k++) {
            double a = 0.0, t = 0.0;
            if (e < e1 && ci[e] - r == g.offq[k]) {
                const int c = ci[e];
                a = v[e++];
                for (int q = uptr[c] + 1; q < rp[c + 1]; q++)
                    if (ci[q] == r) {
                        t = v[q];
                        b |= 1u << k;
                    }
            }
            o[(long)k * g.L] = a;
            o[(long)(g.D + k) * g.L] = t;
        }
        mask[s] = (uint8_t)b;
    }
}
static __global__ void k_line_diag(int n, const int *__restrict__ uptr, const double *__restrict__ v, double *d)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) d[i] = v[uptr[i]];
}
// luv (A's values): l_ij = a_ij / d_j, the pivots on the diagonal, U unchanged
static __global__ void k_line_ilu_finish(int n, const int *__restrict__ rp, const int *__restrict__ ci,
                                         const int *__restrict__ uptr, const double *__restrict__ d, double *luv)
{
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int up = uptr[i];
        for (int e = rp[i]; e < up; e++) luv[e] = luv[e] / __ldg(d + ci[e]);
        luv[up] = __ldg(d + i);
    }
}

}  // namespace xs
