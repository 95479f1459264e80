// Exact LU solve on one thread-block cluster, for patterns without a grid.
//
// The level-ordered sync-free solve (k_trsv_syncfree, standing in for the
// reference's Lcsr_trsv_sync_free / Ucsc_trsv_sync_free,
// hip/Precond/gpuparilu.cpp:257-364) hands a value from row to row through
// L2: a store reaching it and a poll seeing it, about 1.9 us per dependency
// level, and an unstructured mesh of 100,000 rows has some 400 levels.  Here
// one cluster of up to 16 CTAs holds the whole solution vector in its
// distributed shared memory (a slot per position, spread over the CTAs in
// groups of 32), so a hand-off is one shared-memory load from a neighbouring
// SM.  Warps take groups of 32 consecutive positions of the level order in
// turn, a lane per row; a lane polls its pending dependencies until each
// slot holds something other than the NaN pattern it was filled with, then
// sums its entries in order with the operations of the CPU reference's
// LUsolve (hip/HostMatrix/HostMatrixCSR.cpp:385-409), so FP64 results are
// bitwise those of the other exact solves.  The number of warps is chosen so
// that only a few levels' rows are in flight: rows further ahead would only
// poll, while the ones in flight have their row data loaded long before
// their turn.  All CTAs of a cluster run at once and every warp takes its
// groups in increasing order, so each wait is for a row that is being worked
// on; every wait is bounded.  L and U run in one launch with a cluster
// barrier between them.
#pragma once
#include "xs_internal.cuh"

namespace xs {

constexpr int CLU_MAX = 16;                     // CTAs per cluster (8 where 16 are not available)
constexpr int CLU_WARPS_MAX = 16;               // warps per CTA
constexpr int CLU_CHUNK = 8;                    // entries of a row polled at once
constexpr int CLU_AHEAD = 6;                    // levels in flight
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
    asm volatile("st.relaxed.cluster.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void clu_st(uint32_t a, float v)
{
    asm volatile("st.relaxed.cluster.shared::cluster.f32 [%0], %1;" ::"r"(a), "f"(v) : "memory");
}

// one triangle: pci holds dependency positions.  Position p sits in CTA
// (p / 32) % C at slot (p / 32 / C) * 32 + p % 32.
template <typename VT, typename FT, typename DT, bool UPPER>
__device__ __forceinline__ void clu_phase(const TrsvArgs<FT> &P, const int *__restrict__ ppos, const DT *__restrict__ dinv,
                                          const VT *rhs, VT *out, uint32_t base, uint32_t C, uint32_t cshift,
                                          uint32_t rank, int *err)
{
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = blockDim.x >> 5;
    const int groups = (P.n + 31) / 32;
    bool ok = true;
    for (int g = warp * (int)C + (int)rank; g < groups; g += nw * (int)C) {
        const int p = g * 32 + lane;
        bool live = p < P.n;
        int row = 0, k = 0, k1 = 0;
        VT acc = (VT)0;
        if (live) {
            row = __ldg(P.perm + p);
            k = __ldg(P.prp + p);
            k1 = __ldg(P.prp + p + 1);
            acc = rhs[row];
            if (UPPER) acc = (VT)(acc * (VT)__ldg(dinv + p));
        }
        uint32_t a[CLU_CHUNK];
        VT y[CLU_CHUNK], f[CLU_CHUNK];
        unsigned pending = 0;
        int cnt = 0;
        auto load = [&]() {  // the next entries of the row
            cnt = live ? min(CLU_CHUNK, k1 - k) : 0;
            pending = (1u << cnt) - 1u;
#pragma unroll
            for (int j = 0; j < CLU_CHUNK; j++)
                if (j < cnt) {
                    const uint32_t q = (uint32_t)__ldg(ppos + k + j);
                    const uint32_t gq = q >> 5;
                    a[j] = clu_map(base + (((gq >> cshift) << 5) + (q & 31u)) * (uint32_t)sizeof(VT), gq & (C - 1));
                    f[j] = (VT)FVal<FT>::ld(P.pv, k + j);
                }
        };
        load();
        unsigned long long t0 = 0;
        for (long it = 1; __any_sync(0xffffffffu, live); it++) {
            if (live) {
                if (ok) {
#pragma unroll
                    for (int j = 0; j < CLU_CHUNK; j++)
                        if (pending & (1u << j)) {
                            y[j] = clu_ld(a[j], (VT)0);
                            if (!Sentinel<VT>::is(y[j])) pending &= ~(1u << j);
                        }
                } else {
                    pending = 0;
                }
                if (!pending) {
#pragma unroll
                    for (int j = 0; j < CLU_CHUNK; j++)
                        if (j < cnt) acc = msub(acc, y[j], f[j]);
                    k += cnt;
                    if (k >= k1) {
                        const uint32_t own = base + ((((uint32_t)g >> cshift) << 5) + (uint32_t)lane) * (uint32_t)sizeof(VT);
                        clu_st(clu_map(own, rank), acc);
                        out[row] = acc;
                        live = false;
                    } else {
                        load();
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

template <typename VT, typename FT, typename DT>
__global__ void __launch_bounds__(32 * CLU_WARPS_MAX) k_lu_cluster(TrsvArgs<FT> L, const int *__restrict__ lpos,
                                                                   TrsvArgs<FT> U, const int *__restrict__ upos,
                                                                   const DT *__restrict__ dinv, const VT *x, VT *y, VT *z,
                                                                   const int *done_flag, int *err, uint32_t C,
                                                                   uint32_t cshift, int slots)
{
    extern __shared__ __align__(16) unsigned char clu_smem[];
    VT *sv = (VT *)clu_smem;
    pdl_trigger();
    const uint32_t base = (uint32_t)__cvta_generic_to_shared(sv), rank = clu_rank();
    for (int i = threadIdx.x; i < slots; i += blockDim.x) sv[i] = Sentinel<VT>::value();
    pdl_wait();
    if (done_flag && *done_flag) return;  // the same in every CTA
    clu_sync();
    clu_phase<VT, FT, DT, false>(L, lpos, (const DT *)nullptr, x, y, base, C, cshift, rank, err);
    clu_sync();  // y is complete and no CTA reads L's slots any more
    for (int i = threadIdx.x; i < slots; i += blockDim.x) sv[i] = Sentinel<VT>::value();
    clu_sync();
    clu_phase<VT, FT, DT, true>(U, upos, dinv, y, z, base, C, cshift, rank, err);
    clu_sync();  // shared memory stays while other CTAs read it
}

// dependency positions of the level-ordered entries
static __global__ void k_inverse_perm(int n, const int *__restrict__ perm, int *pos_of)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < n; p += gridDim.x * blockDim.x) pos_of[perm[p]] = p;
}
static __global__ void k_entry_positions(long m, const int *__restrict__ pci, const int *__restrict__ pos_of, int *ppos)
{
    for (long e = blockIdx.x * (long)blockDim.x + threadIdx.x; e < m; e += (long)gridDim.x * blockDim.x)
        ppos[e] = pos_of[pci[e]];
}

// the largest cluster this kernel can run as (16, else 8, else 0: none),
// with its shared memory enabled
template <typename VT, typename FT, typename DT>
inline int clu_size()
{
    static const int c = [] {
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
    return c;
}

}  // namespace xs
