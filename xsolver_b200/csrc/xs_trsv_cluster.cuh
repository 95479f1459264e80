// Exact LU solve on one thread-block cluster, for patterns without a grid.
//
// The level-ordered sync-free solve (k_trsv_syncfree, standing in for the
// reference's Lcsr_trsv_sync_free / Ucsc_trsv_sync_free,
// hip/Precond/gpuparilu.cpp:257-364) hands a value from row to row through
// L2: a store reaching it and a poll seeing it, about 1.9 us per dependency
// level, and an unstructured mesh of 100,000 rows has some 400 levels.  Here
// one cluster of up to 16 CTAs holds the whole solution vector in its
// distributed shared memory, so a hand-off is one shared-memory load.
//
// Each level's rows are cut into as many ranges as there are CTAs.  Rows
// keep their order within a level, so with a numbering of any locality a
// row's dependencies lie in the same CTA's part of the levels before, or its
// neighbour's: most hand-offs stay on the SM.  (Rows dealt to the CTAs in
// turn, every dependency remote and polled: 980 ns a level, the lanes that
// wait fill the SM-to-SM network; now 850 ns, of which a remote load is 117.
// LU solve of a mesh of 103,776 rows 677 us, 420,000 rows 1793 us against 2716
// for the sync-free solve.  Whole warps waiting together, 8 or 32 rows each:
// 1364 and 936 us.)  For the same reason a lane polls
// one dependency, the one of the latest level, and reads the others when
// that one is there.  A warp takes a chunk of up to 32 rows of one level at
// a time, the warps of a CTA the levels in turn, so the next levels' row
// data is loaded while the current one is solved.  A slot holds a NaN
// pattern no arithmetic produces until its row is solved; the sums run in
// the order and with the operations of the CPU reference's LUsolve
// (hip/HostMatrix/HostMatrixCSR.cpp:385-409), so FP64 results are bitwise
// those of the other exact solves.  All CTAs of a cluster run at once and
// every warp takes its chunks in level order, so each wait is for a row that
// is being worked on; every wait is bounded.  L and U run in one launch with
// a cluster barrier between them.
#pragma once
#include "xs_internal.cuh"

namespace xs {

constexpr int CLU_MAX = 16;                     // CTAs per cluster (8 where 16 are not available)
constexpr int CLU_WARPS_MAX = 16;               // warps per CTA
constexpr int CLU_CHUNK = 8;                    // entries of a row polled at once
constexpr int CLU_AHEAD = 12;                   // levels in flight
constexpr int CLU_MIN_ROWS = 4096;              // below, one CTA is as fast (lu_block_ok)
constexpr size_t CLU_SMEM_MAX = 224 * 1024;

__device__ __forceinline__ uint32_t clu_rank()
{
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ void clu_sync()
{
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// the address of this CTA's shared location `a` in CTA `cta` of the cluster
__device__ __forceinline__ uint32_t clu_map(uint32_t a, uint32_t cta)
{
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(cta));
    return r;
}
// a value at a mapped address (40 cycles when it is this CTA's own, 230 from
// another SM)
__device__ __forceinline__ double clu_ld(uint32_t a, double)
{
    double v;
    asm volatile("ld.relaxed.cluster.shared::cluster.f64 %0, [%1];" : "=d"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ float clu_ld(uint32_t a, float)
{
    float v;
    asm volatile("ld.relaxed.cluster.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
    return v;
}
__device__ __forceinline__ void clu_st(uint32_t a, double v)
{
    asm volatile("st.relaxed.cluster.shared::cta.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void clu_st(uint32_t a, float v)
{
    asm volatile("st.relaxed.cluster.shared::cta.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// where a position's value lives: CTA of the cluster and slot in its shared
// memory, packed
__host__ __device__ __forceinline__ uint32_t clu_pack(uint32_t cta, uint32_t slot) { return (cta << 16) | slot; }
constexpr uint32_t CLU_NONE = 0xffffffffu;

// a triangle's tables for a cluster of C CTAs (level layout)
struct CluArgs {
    int nlevels;
    const int *lstart;      // first position of each level (and n)
    const int *lslot;       // nlevels * C: first slot of each CTA's part of a level
    const uint32_t *dep;    // per entry: where its dependency's value lives
    const uint32_t *last;   // per position: the dependency of the latest level (CLU_NONE: no entries)
};
// first row of CTA c's part of a level of w rows
// (C = 8 or 16; w is at most the number of rows a cluster can hold)
__host__ __device__ __forceinline__ int clu_part(int w, int c, int C)
{
    return (c * w + C - 1) >> (C == 16 ? 4 : 3);
}

// mapped address of a packed place
template <typename VT>
__device__ __forceinline__ uint32_t clu_addr(uint32_t base, uint32_t where)
{
    return clu_map(base + (where & 0xffffu) * (uint32_t)sizeof(VT), where >> 16);
}

template <typename VT, typename FT, typename DT, bool UPPER>
__device__ __forceinline__ void clu_phase(const TrsvArgs<FT> &P, const CluArgs &Q, const DT *__restrict__ dinv,
                                          const VT *rhs, VT *out, uint32_t base, int C, uint32_t rank, int *err)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    bool ok = true;
    int first = warp;  // this warp's first chunk of the level: (warp - level) mod nw
    int p1 = __ldg(Q.lstart);
    for (int l = 0; l < Q.nlevels; l++, first = first ? first - 1 : nw - 1) {
        const int p0 = p1;
        p1 = __ldg(Q.lstart + l + 1);
        const int w = p1 - p0;
        const int ra = clu_part(w, (int)rank, C), rb = clu_part(w, (int)rank + 1, C);
        for (int j = ra + first * 32; j < rb; j += nw * 32) {
            const int p = p0 + j + lane;
            bool live = j + lane < rb;
            int row = 0, k = 0, k1 = 0;
            uint32_t last = CLU_NONE, own = 0;
            VT acc = (VT)0;
            if (live) {
                row = __ldg(P.perm + p);
                k = __ldg(P.prp + p);
                k1 = __ldg(P.prp + p + 1);
                last = __ldg(Q.last + p);
                acc = rhs[row];
                if (UPPER) acc = (VT)(acc * (VT)__ldg(dinv + p));
                own = base + (uint32_t)(__ldg(Q.lslot + (long)l * C + rank) + (j + lane - ra)) * (uint32_t)sizeof(VT);
            }
            uint32_t a[CLU_CHUNK];  // addresses in the cluster
            VT y[CLU_CHUNK], f[CLU_CHUNK];
            int cnt = 0;
            auto load = [&]() {  // the next entries of the row
                cnt = live ? min(CLU_CHUNK, k1 - k) : 0;
#pragma unroll
                for (int q = 0; q < CLU_CHUNK; q++) {
                    a[q] = base;
                    f[q] = (VT)0;
                    if (q < cnt) {
                        a[q] = clu_addr<VT>(base, __ldg(Q.dep + k + q));
                        f[q] = (VT)FVal<FT>::ld(P.pv, k + q);
                    }
                }
            };
            load();
            // entries read per chunk: the warp's longest row, not the full chunk
            int most = (int)__reduce_max_sync(0xffffffffu, (unsigned)cnt);
            uint32_t wait = last == CLU_NONE ? CLU_NONE : clu_addr<VT>(base, last);
            unsigned long long t0 = 0;
            for (int it = 1; __any_sync(0xffffffffu, live); it++) {
                if (wait != CLU_NONE && (!Sentinel<VT>::is(clu_ld(wait, (VT)0)) || !ok)) wait = CLU_NONE;
                if (live && wait == CLU_NONE) {
                    // all of them at once, then the checks: one latency
#pragma unroll
                    for (int q = 0; q < CLU_CHUNK; q++) {
                        if (q >= most) break;
                        y[q] = clu_ld(a[q], (VT)0);
                    }
                    bool pending = false;
#pragma unroll
                    for (int q = 0; q < CLU_CHUNK; q++) {
                        if (q >= most) break;
                        pending |= q < cnt && Sentinel<VT>::is(y[q]);
                    }
                    if (!pending || !ok) {
#pragma unroll
                        for (int q = 0; q < CLU_CHUNK; q++) {
                            if (q >= cnt) break;  // no sums of absent entries
                            acc = msub(acc, y[q], f[q]);
                        }
                        k += cnt;
                        if (k >= k1) {
                            clu_st(own, acc);
                            out[row] = acc;
                            live = false;
                        } else {
                            load();
                            most = CLU_CHUNK;
                        }
                    }
                }
                if ((it & 1023) == 0) {
                    const unsigned long long now = gtimer();
                    if (t0 == 0) t0 = now;
                    else if (now - t0 > WAIT_LIMIT_NS) {
                        if (lane == 0) atomicOr(err, DEV_TRSV_TIMEOUT);
                        ok = false;
                    }
                    if (*(volatile int *)err) ok = false;
                }
            }
        }
    }
}

template <typename VT, typename FT, typename DT>
__global__ void __launch_bounds__(32 * CLU_WARPS_MAX) k_lu_cluster(TrsvArgs<FT> L, CluArgs QL,
                                                                   TrsvArgs<FT> U, CluArgs QU,
                                                                   const DT *__restrict__ dinv, const VT *x, VT *y, VT *z,
                                                                   const int *done_flag, int *err, int C,
                                                                   int slots)
{
    extern __shared__ __align__(16) unsigned char clu_smem[];
    VT *sv = (VT *)clu_smem;
    pdl_trigger();
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sv), rank = clu_rank();
    for (int i = threadIdx.x; i < slots; i += blockDim.x) sv[i] = Sentinel<VT>::value();
    pdl_wait();
    if (done_flag && *done_flag) return;  // the same in every CTA
    clu_sync();
    clu_phase<VT, FT, DT, false>(L, QL, (const DT *)nullptr, x, y, base, C, rank, err);
    clu_sync();  // y is complete and no CTA reads L's slots any more
    for (int i = threadIdx.x; i < slots; i += blockDim.x) sv[i] = Sentinel<VT>::value();
    clu_sync();
    clu_phase<VT, FT, DT, true>(U, QU, dinv, y, z, base, C, rank, err);
    clu_sync();  // shared memory stays while other CTAs read it
}

// where each row's value lives, by row
static __global__ void k_clu_rows(int n, int nlevels, int C, const int *__restrict__ perm, const int *__restrict__ lstart,
                                  const int *__restrict__ lslot, uint32_t *where, int *level)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        int lo = 0, hi = nlevels - 1;  // the level that holds p
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (lstart[mid] <= p) lo = mid;
            else hi = mid - 1;
        }
        const int j = p - lstart[lo], w = lstart[lo + 1] - lstart[lo];
        const int c = (int)((long)j * C / w);
        where[perm[p]] = clu_pack((uint32_t)c, (uint32_t)(lslot[(long)lo * C + c] + j - clu_part(w, c, C)));
        level[perm[p]] = lo;
    }
}
// the entries' dependencies, and each position's one of the latest level
static __global__ void k_clu_entries(int n, const int *__restrict__ prp, const int *__restrict__ pci,
                                     const uint32_t *__restrict__ where, const int *__restrict__ level, uint32_t *dep,
                                     uint32_t *last)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) {
        int best = -1;
        uint32_t b = CLU_NONE;
        for (int e = prp[p]; e < prp[p + 1]; e++) {
            const int r = pci[e];
            dep[e] = where[r];
            if (level[r] > best) {
                best = level[r];
                b = where[r];
            }
        }
        last[p] = b;
    }
}

// the largest cluster this kernel can run as on the current device (16, else
// 8, else 0: none), with its shared memory enabled there.  Function
// attributes belong to one device, so the answer is kept for each.
template <typename VT, typename FT, typename DT>
inline int clu_size()
{
    static std::mutex mu;
    static signed char known[64] = {};  // by device: 0 not asked yet, else the size + 1
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64) return 0;
    std::lock_guard<std::mutex> lock(mu);
    if (known[dev]) return known[dev] - 1;
    const int c = [] {
        auto kern = k_lu_cluster<VT, FT, DT>;
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)CLU_SMEM_MAX) != cudaSuccess ||
            cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        for (int q = CLU_MAX; q >= 8; q /= 2) {
            cudaLaunchConfig_t cfg = {};
            cfg.gridDim = dim3(q);
            cfg.blockDim = dim3(32 * CLU_WARPS_MAX);
            cfg.dynamicSmemBytes = CLU_SMEM_MAX;
            cudaLaunchAttribute at[1];
            at[0].id = cudaLaunchAttributeClusterDimension;
            at[0].val.clusterDim.x = q;
            at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
            cfg.attrs = at;
            cfg.numAttrs = 1;
            int count = 0;
            if (cudaOccupancyMaxActiveClusters(&count, kern, &cfg) == cudaSuccess && count > 0) return q;
            cudaGetLastError();
        }
        return 0;
    }();
    known[dev] = (signed char)(c + 1);
    return c;
}

}  // namespace xs
