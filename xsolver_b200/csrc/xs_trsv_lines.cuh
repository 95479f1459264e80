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
//   helper warps      stage the factor data NS stages ahead (one bulk copy
//                     each for values, diagonal and masks, stored in exactly
//                     the order they are used) and the right-hand side, and
//                     drain finished steps to the output along x, so that
//                     vectors stay in natural order and accesses coalesce
//
// Patches are taken by ticket in an order in which dependencies come first,
// so a CTA only waits on patches that running CTAs hold: no co-residency is
// needed.  The exchange buffer is doubled: a launch publishes into one half
// and re-arms the other for the next launch.
#pragma once
#include <vector>
#include "xs_internal.cuh"
#include "xs_spmv.cuh"
#include "xs_trsv_tiles.cuh"

namespace xs {

constexpr int LINE_DIAG_MAX = 32;   // entries per row: bits of the row mask
constexpr int LINE_PATCH = 128;       // lines per patch
constexpr int LINE_HALO_MAX = 64;   // halo lines per patch
constexpr int LINE_HELPERS = 128;   // staging / draining threads
constexpr int LINE_POLL_WARPS = 4;  // most poller warps
constexpr int LINE_ITEMS = 2;       // halo values polled per poller lane
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
    static __host__ __device__ LineSmem of(const LineGeo &g, int S, int NS, int RL, int KC, size_t vb, size_t fb,
                                           size_t db, size_t mb)
    {
        auto al = [](size_t b) { return (b + 127) & ~(size_t)127; };
        LineSmem m;
        m.Ps = g.npad | 1;
        m.RS = (g.L * KC) | 1;
        m.ring = 0;
        m.rhs = m.ring + al((size_t)RL * m.Ps * KC * vb);
        m.pv = m.rhs + al((size_t)NS * S * m.RS * vb);
        m.dinv = m.pv + al((size_t)NS * S * g.D * g.L * fb);
        m.mask = m.dinv + al((size_t)NS * S * g.L * db);
        m.tab = m.mask + al((size_t)NS * S * g.L * mb);
        m.total = m.tab + al((size_t)3 * g.L * sizeof(int));
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
inline LineCfg line_cfg(const LineGeo &g, int items, int KC, size_t vb, size_t fb, size_t db, size_t mb, int sms)
{
    LineCfg c;
    int best = -1;
    for (size_t lim : {items > sms ? (size_t)112 * 1024 : LINE_SMEM_MAX, LINE_SMEM_MAX}) {
        for (int RL : {64, 32})
            for (int S = LINE_STEP; S >= 1; S /= 2)
                for (int NS = LINE_NS_MAX; NS >= 3; NS--) {
                    const int ahead = RL - g.maxd - S;  // steps the pollers run ahead
                    if (ahead < LINE_WINDOW || RL < 2 * S) continue;
                    const size_t b = LineSmem::of(g, S, NS, RL, KC, vb, fb, db, mb).total;
                    if (b > lim) continue;
                    if (lim != LINE_SMEM_MAX && NS * S < 12) continue;  // too little in flight to share an SM
                    const int score = std::min(NS * S, 24) * 10000 + std::min(ahead, 24) * 100 + 10 * S + (8 - NS);
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
    DBuf<int> patch;    // pY, pZ of each patch in ticket order
    DBuf<int> rank_of;  // ticket rank of patch (pY, pZ), -1: no lines
    DBuf<int> halo;     // Yl, Zl of each halo line (relative to the patch)
    DBuf<int> exp_of;   // per line of a patch: index among the exported lines, or -1
    DBuf<uint8_t> mask8;
    DBuf<uint32_t> mask32;
    int brk = -1;       // debugging: rank of a patch made to wait for a value of its own
};

// exchange buffer of one consumer (a preconditioner's own solves, or a batch)
template <typename VT>
struct LineXchg {
    DBuf<VT> x;          // two halves
    DBuf<unsigned> ctl;  // ticket, current half
    size_t half = 0;
};

// Host half of the plan from a detected grid.  False when the pattern does
// not qualify: more than 32 diagonals, over a quarter of padding, a reach
// beyond a patch, or lines too short for the schedule's skew (more than
// four slots per row).
struct LineHost {
    LineGeo g;
    std::vector<int> patch, rank_of, halo, exp_of;
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
    // patches take on the GPU's SMs (microseconds; the constants are the
    // measured step and hand-off of the kernel below, to one digit)
    const int Yext = g.ny + c * (g.nz - 1);
    const double ts = 0.05 + 0.005 * D, th = 1.0;
    double best = 1e300;
    for (int L = 32; L <= LINE_PATCH; L *= 2)
        for (int ty = 1; ty <= L; ty *= 2) {
            const int tz = L / ty;
            if (ty < g.ry || tz < g.rz) continue;
            const int npy = (Yext + ty - 1) / ty, npz = (g.nz + tz - 1) / tz;
            const int ns = (g.nx + al * (ty - 1) + be * (tz - 1) + LINE_STEP - 1) / LINE_STEP * LINE_STEP;
            // patches that hold lines (the sheared domain is a parallelogram)
            long np = 0;
            for (int p = 0; p < npz; p++) {
                const int z0 = p * tz, z1 = std::min(g.nz, z0 + tz) - 1;
                np += (c * z1 + g.ny - 1) / ty - (c * z0) / ty + 1;
            }
            if (np * ns * L > 4L * n + 16384) continue;  // mostly padding
            const double chain = (g.nx + al * (double)(Yext - 1) + be * (double)(g.nz - 1)) * ts + (npy + npz - 2) * th;
            const double stream = (double)np * ns * L * (8.0 * D + 24.0) / 5.5e6;
            const double work = (double)np * ns * ts / sms;
            const double cost = std::max(chain, work) + 0.5 * stream;
            LineGeo t = g;
            t.L = L; t.ty = ty; t.tz = tz;
            t.npad = (ty + g.ry) * (tz + g.rz);
            if (cost < best && line_cfg(t, 0, 1, 8, 8, 8, g.mask8() ? 1 : 4, 1).S) {
                best = cost;
                g.L = L; g.ty = ty; g.tz = tz;
                g.npy = npy; g.npz = npz; g.nsteps = ns;
            }
        }
    if (best >= 1e300) return false;
    g.py = g.ty + g.ry;
    g.npad = g.py * (g.tz + g.rz);
    for (int k = 0; k < D; k++) g.shift[k] = -dY(ord[k]) - dz[ord[k]] * g.py;
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
struct LineSlot {
    int row;  // -1: no row
};
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
__device__ __forceinline__ void line_bar(int id, int count)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// the mbarrier gets one (already counted) arrival when this thread's earlier cp.async have landed
__device__ __forceinline__ void cp_async_mbar_arrive(uint64_t *bar)
{
    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

template <typename VT, typename FT, typename DT, bool UPPER, int KC, int W>
__global__ void __launch_bounds__(LINE_PATCH *KC + LINE_HELPERS + 32 * LINE_POLL_WARPS)
    k_trsv_lines(const __grid_constant__ LineGeo G, const __grid_constant__ LineArgs<VT, FT, DT> A)
{
    using MK = typename std::conditional<(W == 2 || W == 3), uint8_t, uint32_t>::type;
    extern __shared__ __align__(128) unsigned char line_smem[];
    __shared__ __align__(8) uint64_t full[LINE_NS_MAX];
    __shared__ int s_item, cdone, drained, hcnt[LINE_POLL_WARPS];
    __shared__ unsigned s_half;
    const int D = W > 0 ? W : G.D;
    const int L = G.L, T = L * KC, S = A.S, NS = A.NS, RM = A.RL - 1, NP = A.NP;
    const LineSmem M = LineSmem::of(G, S, NS, A.RL, KC, sizeof(VT), sizeof(FT), UPPER ? sizeof(DT) : 0, sizeof(MK));
    VT *ring = (VT *)(line_smem + M.ring);
    VT *s_rhs = (VT *)(line_smem + M.rhs);
    FT *s_pv = (FT *)(line_smem + M.pv);
    DT *s_dinv = (DT *)(line_smem + M.dinv);
    MK *s_mask = (MK *)(line_smem + M.mask);
    int *s_q0 = (int *)(line_smem + M.tab), *s_off = s_q0 + L, *s_pad = s_off + L;
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
    if (tid == 0) s_half = *(volatile unsigned *)(A.ctl + 1);
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
        if (tid < LINE_POLL_WARPS) hcnt[tid] = -G.maxd;
        __syncthreads();
        const int item = s_item;
        if (item >= items) break;
        const int rank = item / A.ngroups, grp = item % A.ngroups;
        const int pY = A.patch[2 * rank], pZ = A.patch[2 * rank + 1];
        for (int l = tid; l < L; l += blockDim.x) {
            const int Yl = l % G.ty, Zl = l / G.ty;
            s_q0[l] = G.line_q0(pY, pZ, Yl, Zl);
            s_off[l] = G.al * Yl + G.be * Zl;
            s_pad[l] = (Zl + G.rz) * G.py + Yl + G.ry;
        }
        __syncthreads();
        VT *xpub = A.xb + (s_half ? A.xb_half : 0);
        if (tid < T) {
            // ------------------------------------------------ compute
            const int l = tid / KC, c = tid % KC;
            const int q0 = s_q0[l], off = s_off[l];
            const int e = __ldg(A.exp_of + l);
            VT *pub = e >= 0 ? xpub + ((long)item * G.nsteps * G.E + e) * KC + c : nullptr;
            const long pstep = (long)G.E * KC;
            VT *rcol = ring + s_pad[l] * KC + c;
            int avail = -G.maxd;
            bool landed = true;
            for (int g = 0; g < nst; g++) {
                const unsigned st = cnt0 + (unsigned)g;
                const int slot = (int)(st % (unsigned)NS);
                if (landed) landed = mbar_wait_bounded(&full[slot], (st / (unsigned)NS) & 1u, A.err);
                line_wait(&drained, (g + 1) * S - A.RL, A.err, 0);
                const FT *pv = s_pv + (size_t)slot * S * D * L + l;
                const MK *mk = s_mask + (size_t)slot * S * L + l;
                const DT *dv = s_dinv + (size_t)slot * S * L + l;
                const VT *rh = s_rhs + (size_t)slot * S * M.RS + tid;
                for (int s = 0; s < S; s++) {
                    const int tau = g * S + s, x = tau - off;
                    VT acc = rh[s * M.RS];
                    const uint32_t m = mk[s * L];
                    if (UPPER) acc = (VT)(acc * (VT)dv[s * L]);
                    const FT *pvs = pv + (size_t)s * D * L;
                    FT v[W > 0 ? W : 1];
                    if constexpr (W > 0) {
#pragma unroll
                        for (int k = 0; k < W; k++) v[k] = pvs[k * L];
                    }
                    // the halo values this step may read (steps before it)
                    if (avail < tau) {
                        avail = line_wait(&hcnt[0], tau, A.err, 0);
                        for (int w = 1; w < NP; w++) avail = min(avail, line_wait(&hcnt[w], tau, A.err, 0));
                    }
                    if (q0 >= 0 && (unsigned)x < (unsigned)G.nx) {
                        if constexpr (W > 0) {
#pragma unroll
                            for (int k = 0; k < W; k++) {
                                const VT y = rcol[((tau - G.delta[k]) & RM) * PsK - G.shift[k] * KC];
                                const VT a2 = msub(acc, y, (VT)FVal<FT>::cvt(v[k]));
                                acc = (m >> k) & 1u ? a2 : acc;
                            }
                        } else {
#pragma unroll 4
                            for (int k = 0; k < D; k++) {
                                const VT y = rcol[((tau - G.delta[k]) & RM) * PsK - G.shift[k] * KC];
                                const VT a2 = msub(acc, y, (VT)FVal<FT>::cvt(pvs[k * L]));
                                acc = (m >> k) & 1u ? a2 : acc;
                            }
                        }
                        rcol[(tau & RM) * PsK] = acc;
                        if (pub) st_publish(pub + tau * pstep, acc);
                    }
                    line_bar(1, T);
                }
                if (tid == 0) st_release_cta(&cdone, (g + 1) * S);
            }
        } else if (tid < T + LINE_HELPERS) {
            // ------------------------------------------------ staging and draining
            const int h = tid - T;
            const long base = (long)rank * G.nsteps;
            const int per = S * KC;
            const int nel = L * per;
            auto stage = [&](int g) {
                const unsigned st = cnt0 + (unsigned)g;
                const int slot = (int)(st % (unsigned)NS);
                if (h == 0) {
                    const uint32_t bv = (uint32_t)(S * D * L * sizeof(FT)), bm = (uint32_t)(S * L * sizeof(MK));
                    const uint32_t bd = UPPER ? (uint32_t)(S * L * sizeof(DT)) : 0u;
                    mbar_expect_tx(&full[slot], bv + bm + bd);
                    bulk_g2s(s_pv + (size_t)slot * S * D * L, A.pv + (base + (long)g * S) * D * L, bv, &full[slot]);
                    bulk_g2s(s_mask + (size_t)slot * S * L, (const MK *)A.mask + (base + (long)g * S) * L, bm, &full[slot]);
                    if (UPPER)
                        bulk_g2s(s_dinv + (size_t)slot * S * L, A.dinv + (base + (long)g * S) * L, bd, &full[slot]);
                }
                VT *rb = s_rhs + (size_t)slot * S * M.RS;
                for (int i = h; i < nel; i += LINE_HELPERS) {
                    const int l = i / per, r = i % per, s = r / KC, c = r % KC;
                    const int q0 = s_q0[l], x = g * S + s - s_off[l], col = grp * KC + c;
                    if (q0 >= 0 && (unsigned)x < (unsigned)G.nx && (KC == 1 || col < A.k)) {
                        const long row = UPPER ? G.n - 1 - (q0 + x) : q0 + x;
                        cp_async_n<sizeof(VT)>(rb + s * M.RS + l * KC + c, A.rhs + (KC == 1 ? row : row * A.k + col));
                    }
                }
                cp_async_mbar_arrive(&full[slot]);
            };
            for (int g = 0; g < NS && g < nst; g++) stage(g);
            for (int g = 0; g < nst; g++) {
                line_wait(&cdone, (g + 1) * S, A.err, 40);
                if (g + NS < nst) stage(g + NS);
                for (int i = h; i < nel; i += LINE_HELPERS) {
                    const int l = i / per, r = i % per, s = r / KC, c = r % KC;
                    const int q0 = s_q0[l], tau = g * S + s, x = tau - s_off[l], col = grp * KC + c;
                    if (q0 >= 0 && (unsigned)x < (unsigned)G.nx && (KC == 1 || col < A.k)) {
                        const long row = UPPER ? G.n - 1 - (q0 + x) : q0 + x;
                        const long o = KC == 1 ? row : row * A.k + col;
                        A.out[o] = ring[(tau & RM) * PsK + s_pad[l] * KC + c];
                        if (A.reset_other) A.reset_other[o] = Sentinel<VT>::value();
                    }
                }
                line_bar(2, LINE_HELPERS);
                if (h == 0) st_release_cta(&drained, (g + 1) * S);
            }
            // re-arm this patch's part of the other half for the next launch
            VT *xr = A.xb + (s_half ? 0 : A.xb_half) + (long)item * G.nsteps * G.E * KC;
            for (int i = h; i < G.nsteps * G.E * KC; i += LINE_HELPERS) xr[i] = Sentinel<VT>::value();
        } else if ((tid - T - LINE_HELPERS) / 32 < NP) {
            // ------------------------------------------------ halo
            const int pw = (tid - T - LINE_HELPERS) / 32, lane = tid & 31;
            const VT *src[LINE_ITEMS];
            int x0[LINE_ITEMS], x1[LINE_ITEMS], pos[LINE_ITEMS], rc[LINE_ITEMS];
            const long pstep = (long)G.E * KC;
#pragma unroll
            for (int j = 0; j < LINE_ITEMS; j++) {
                const int i = (j * NP + pw) * 32 + lane;
                src[j] = nullptr;
                x0[j] = x1[j] = rc[j] = 0;
                pos[j] = -G.maxd;
                if (i < G.nh * KC) {
                    const int hl = i / KC, c = i % KC;
                    const int Yl = __ldg(A.halo + 2 * hl), Zl = __ldg(A.halo + 2 * hl + 1);
                    if (G.line_q0(pY, pZ, Yl, Zl) >= 0 && (KC == 1 || grp * KC + c < A.k)) {
                        const int dpY = Yl < 0 ? -1 : 0, dpZ = Zl < 0 ? -1 : 0;
                        const int Yo = Yl - dpY * G.ty, Zo = Zl - dpZ * G.tz;  // the line inside its own patch
                        const int ro = __ldg(A.rank_of + (pZ + dpZ) * G.npy + pY + dpY);
                        const int off_o = G.al * Yo + G.be * Zo, off_h = G.al * Yl + G.be * Zl;
                        const int eo = __ldg(A.exp_of + Zo * G.ty + Yo);
                        // value of step t here: step t + (off_o - off_h) of the owner
                        src[j] = xpub + (((long)ro * A.ngroups + grp) * G.nsteps + (off_o - off_h)) * pstep + eo * KC + c;
                        x0[j] = off_h;  // active steps [x0, x1)
                        x1[j] = off_h + G.nx;
                        rc[j] = ((Zl + G.rz) * G.py + Yl + G.ry) * KC + c;
                    }
                }
            }
            const bool brk = A.brk == rank && pw == 0 && lane == 0;  // debugging: a wait that never ends
            bool ok = true;
            int published = -G.maxd;
            unsigned long long t0 = 0;
            long spins = 0;
            while (published < G.nsteps) {
                const int lim = min(ld_acquire_cta(&cdone) + A.RL - G.maxd, G.nsteps);
                int mn = lim;
#pragma unroll
                for (int j = 0; j < LINE_ITEMS; j++) {
                    if (!src[j] || !ok) continue;
                    const int p = pos[j], m = min(lim - p, LINE_WINDOW);
                    VT v[LINE_WINDOW];
#pragma unroll
                    for (int u = 0; u < LINE_WINDOW; u++) {
                        v[u] = (VT)0;
                        if (u < m && p + u >= x0[j] && p + u < x1[j]) v[u] = ld_poll(src[j] + (p + u) * pstep);
                    }
                    int r = 0;
#pragma unroll
                    for (int u = 0; u < LINE_WINDOW; u++) {
                        if (r == u && u < m && !Sentinel<VT>::is(v[u])) {
                            if (p + u >= x0[j] && p + u < x1[j]) ring[((p + u) & RM) * PsK + rc[j]] = v[u];
                            r = u + 1;
                        }
                    }
                    pos[j] = p + r;
                    mn = min(mn, p + r);
                }
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
                    line_wait(&cdone, lim + G.maxd - A.RL + 1, A.err, 64);
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
// columns of one compute line for k right-hand sides: up to 4, fewer when
// their ring and stages do not fit in shared memory
inline int line_kc(const LineGeo &g, int k)
{
    for (int kc = k >= 3 ? 4 : k; kc > 1; kc = kc == 4 ? 2 : 1)
        if (line_cfg(g, 0, kc, sizeof(double), sizeof(double), sizeof(double), g.mask8() ? 1 : 4, 1).S) return kc;
    return 1;
}

template <typename VT>
inline void line_xchg_ensure(LineXchg<VT> &X, const LineGeo &g, int k, cudaStream_t s)
{
    const int kc = line_kc(g, k), ng = (k + kc - 1) / kc;
    const size_t half = (size_t)g.npatch * ng * g.nsteps * g.E * kc;
    if (X.half == half && X.x.p) return;
    X.x.alloc(2 * half);
    X.ctl.alloc(2);
    X.half = half;
    k_fill_sentinel<VT><<<256, 256, 0, s>>>(X.x.p, (int)(2 * half));
    check_launch();
}
template <typename VT>
inline void line_xchg_rearm(LineXchg<VT> &X, cudaStream_t s)
{
    if (!X.x.p) return;
    k_fill_sentinel<VT><<<256, 256, 0, s>>>(X.x.p, (int)(2 * X.half));
    XS_CUDA(cudaMemsetAsync(X.ctl.p, 0, sizeof(unsigned), s));
}

template <typename VT, typename FT, typename DT, bool UPPER, int KC>
inline void launch_trsv_lines(const LinePlan &P, const FT *pv, const DT *dinv, LineXchg<VT> &X, int k, const VT *rhs,
                              VT *out, VT *reset_other, const int *done_flag, int *err, cudaStream_t s)
{
    const LineGeo &g = P.g;
    const int ng = (k + KC - 1) / KC, items = g.npatch * ng, sms = geom().sms;
    const bool m8 = g.mask8();
    const LineCfg c = line_cfg(g, items, KC, sizeof(VT), sizeof(FT), UPPER ? sizeof(DT) : 0, m8 ? 1 : 4, sms);
    if (c.S == 0 || !X.x.p || X.half != (size_t)items * g.nsteps * g.E * KC) throw Status(XS_ERR_ORDER);
    LineArgs<VT, FT, DT> A;
    A.patch = P.patch.p; A.rank_of = P.rank_of.p; A.halo = P.halo.p; A.exp_of = P.exp_of.p;
    A.pv = pv;
    A.mask = m8 ? (const void *)P.mask8.p : (const void *)P.mask32.p;
    A.dinv = dinv;
    A.xb = X.x.p; A.xb_half = (long)X.half; A.ctl = X.ctl.p;
    A.S = c.S; A.NS = c.NS; A.RL = c.RL;
    A.NP = std::max(1, std::min(LINE_POLL_WARPS, (g.nh * KC + 31) / 32));
    A.k = k; A.ngroups = ng;
    A.rhs = rhs; A.out = out; A.reset_other = reset_other;
    A.done_flag = done_flag; A.err = err; A.brk = P.brk;
    const int threads = g.L * KC + LINE_HELPERS + 32 * A.NP;
    const int per_sm = c.smem <= 112 * 1024 && 2 * threads <= 2048 ? 2 : 1;
    const int grid = std::min(items, sms * per_sm);
    auto go = [&](auto kern) {
        // the attribute is per function and idempotent: set on every launch (host-side only, no synchronisation)
        XS_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)LINE_SMEM_MAX));
        launch_pdl(kern, dim3(grid), dim3(threads), c.smem, s, g, A);
    };
    if (g.D == 3) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 3>);
    else if (g.D == 2) go(k_trsv_lines<VT, FT, DT, UPPER, KC, 2>);
    else go(k_trsv_lines<VT, FT, DT, UPPER, KC, 0>);
}

}  // namespace xs
