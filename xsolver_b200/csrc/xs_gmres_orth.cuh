// One GMRES step's orthogonalisation as one kernel.
//
// Modified Gram-Schmidt (intel/mpisolver-C-v1.cpp:982-1010) is a chain: the
// coefficient h_k = (w, v_k) needs w after the update with v_{k-1}.  As one
// vector kernel per coefficient a step i costs i + 3 launches, each with a
// grid-wide reduction and a pass over w, v_{k-1} and v_k.  Here one
// cooperative launch does the whole step: every thread keeps its elements of
// w in registers, a coefficient's block partials are exchanged through one
// grid barrier and summed by every block itself (in block order, so all
// blocks hold the same bits), and the next basis vector is loaded while the
// barrier is pending, so each basis vector is read once.  The last barrier's
// norm gives the Givens rotation (one thread, as the last block of the norm
// reduction did) and the scaled v_{i+1}.  Elements use the operations of the
// separate kernels; the dot products' partial sums follow this grid.
//
// The barrier is a monotonic counter, its waits bounded: a block that gives
// up records an error and every later wait ends at once.
#pragma once
#include "xs_solvers.cuh"

namespace xs {

constexpr int ORTH_THREADS = 1024;
constexpr int ORTH_BYTES = 64;  // of w per thread, at most

struct GridBar {
    unsigned *count;  // arrivals, then departures in count[1]
    int *err;
};
// all blocks of a cooperative launch; phase = 1, 2, ... in each launch
__device__ __forceinline__ void grid_barrier(const GridBar &B, unsigned phase)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        atomicAdd(B.count, 1u);
        const unsigned target = phase * gridDim.x;
        unsigned long long t0 = 0;
        for (long it = 1; (unsigned)ld_acquire((const int *)B.count) < target; it++) {
            if ((it & 1023) == 0) {
                const unsigned long long now = gtimer();
                if (t0 == 0) t0 = now;
                else if (now - t0 > WAIT_LIMIT_NS) atomicOr(B.err, DEV_TRSV_TIMEOUT);
                if (*(volatile int *)B.err) break;
            }
        }
    }
    __syncthreads();
}
// the last block to leave re-arms the counter for the next launch
__device__ __forceinline__ void grid_barrier_leave(const GridBar &B)
{
    __syncthreads();
    if (threadIdx.x == 0) {
        const unsigned t = atomicAdd(B.count + 1, 1u);
        if (t == gridDim.x - 1) {
            B.count[0] = 0u;
            B.count[1] = 0u;
        }
    }
}

// sum of a over the block in every thread of warp 0 (lane 0 publishes)
__device__ __forceinline__ double orth_block_sum(double a, double *s_warp)
{
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if ((threadIdx.x & 31) == 0) s_warp[threadIdx.x >> 5] = a;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32) {
        s = s_warp[threadIdx.x];
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    }
    return s;
}
// every block's partials, summed in block order by warp 0, to all threads
__device__ __forceinline__ double orth_total(const double *part, double *s_tot)
{
    if (threadIdx.x < 32) {
        double s = 0.0;
        for (int b = threadIdx.x; b < (int)gridDim.x; b += 32) s += __ldcg(part + b);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (threadIdx.x == 0) *s_tot = s;
    }
    __syncthreads();
    return *s_tot;
}

// w: the new direction A M^-1 v_i; V: the basis (v_k at V + k*n); step i.
// CH chunks of VW consecutive elements per thread.
template <typename VT, int CH, int VW>
__global__ void __launch_bounds__(ORTH_THREADS, 1) k_gm_orth(int n, KState *st, const VT *__restrict__ w, VT *V, GmDev g,
                                                             int i, int quirk, double *part, GridBar B)
{
    __shared__ double s_warp[32], s_tot;
    if (st->done) return;
    const int T = gridDim.x * ORTH_THREADS, t = blockIdx.x * ORTH_THREADS + threadIdx.x;
    VT wr[CH][VW], vr[CH][VW];
    auto load = [&](const VT *p, VT(&r)[CH][VW]) {
#pragma unroll
        for (int c = 0; c < CH; c++) {
            const long e = ((long)c * T + t) * VW;
#pragma unroll
            for (int q = 0; q < VW; q++) r[c][q] = (VT)0;
            if (e < n) {
                if constexpr (VW > 1) ld16<VT, VW>(p + e, r[c]);
                else r[c][0] = p[e];
            }
        }
    };
    load(w, wr);
    load(V, vr);
    unsigned phase = 0;
    for (int k = 0; k <= i; k++) {
        double a = 0.0;
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
            for (int q = 0; q < VW; q++) a += (double)wr[c][q] * (double)vr[c][q];
        double *pk = part + (size_t)(phase & 1u) * gridDim.x;  // the other half may still be read
        const double s = orth_block_sum(a, s_warp);
        if (threadIdx.x == 0) pk[blockIdx.x] = s;
        VT vn[CH][VW];
        if (k < i) load(V + (size_t)(k + 1) * n, vn);  // on its way during the barrier
        grid_barrier(B, ++phase);
        const double hk = orth_total(pk, &s_tot);
        if (blockIdx.x == 0 && threadIdx.x == 0) g.H[k * g.m + i] = hk;
        const VT minh = -(VT)hk;
#pragma unroll
        for (int c = 0; c < CH; c++)
#pragma unroll
            for (int q = 0; q < VW; q++) {
                wr[c][q] = wr[c][q] + minh * vr[c][q];
                vr[c][q] = vn[c][q];
            }
    }
    double a = 0.0;
#pragma unroll
    for (int c = 0; c < CH; c++)
#pragma unroll
        for (int q = 0; q < VW; q++) a += (double)wr[c][q] * (double)wr[c][q];
    double *pk = part + (size_t)(phase & 1u) * gridDim.x;
    const double s = orth_block_sum(a, s_warp);
    if (threadIdx.x == 0) pk[blockIdx.x] = s;
    grid_barrier(B, ++phase);
    const double tot = orth_total(pk, &s_tot);
    const VT inv = (VT)(1.0 / (sqrt(tot) + KSMALL));
    VT *vo = V + (size_t)(i + 1) * n;
#pragma unroll
    for (int c = 0; c < CH; c++) {
        const long e = ((long)c * T + t) * VW;
        if (e < n) {
            VT o[VW];
#pragma unroll
            for (int q = 0; q < VW; q++) o[q] = wr[c][q] * inv;
            if constexpr (VW > 1) st16<VT, VW>(vo + e, o);
            else vo[e] = o[0];
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) gm_norm_finish(st, g, i, quirk, tot);
    grid_barrier_leave(B);
}

// whether one launch serves vectors of n elements, and its shape
template <typename VT>
struct OrthShape {
    int grid = 0, ch = 0;
    bool vec = false;
};
template <typename VT>
inline OrthShape<VT> orth_shape(int n)
{
    OrthShape<VT> o;
    constexpr int VW = 16 / (int)sizeof(VT);
    o.vec = n % VW == 0;  // every basis vector then starts on a 16-byte boundary
    const int vw = o.vec ? VW : 1, most = ORTH_BYTES / (int)sizeof(VT) / vw;
    const long units = ((long)n + vw - 1) / vw;  // chunks to distribute
    o.grid = (int)std::min<long>(geom().sms, (units + ORTH_THREADS - 1) / ORTH_THREADS);
    const long per = (units + (long)o.grid * ORTH_THREADS - 1) / ((long)o.grid * ORTH_THREADS);
    if (per > most) return OrthShape<VT>();
    o.ch = 1;
    while (o.ch < per) o.ch *= 2;
    return o;
}

template <typename VT>
inline void launch_gm_orth(const OrthShape<VT> &o, int n, KState *st, const VT *w, VT *V, const GmDev &g, int i,
                           int quirk, double *part, const GridBar &B, cudaStream_t s)
{
    constexpr int VW = 16 / (int)sizeof(VT);
    auto go = [&](auto kern) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(o.grid);
        cfg.blockDim = dim3(ORTH_THREADS);
        cfg.stream = s;
        cudaLaunchAttribute at[1];
        at[0].id = cudaLaunchAttributeCooperative;
        at[0].val.cooperative = 1;
        cfg.attrs = at;
        cfg.numAttrs = 1;
        if (cudaLaunchKernelEx(&cfg, kern, n, st, w, V, g, i, quirk, part, B) != cudaSuccess) throw Status(XS_ERR_CUDA);
    };
    constexpr int MV = ORTH_BYTES / 16, MS = ORTH_BYTES / (int)sizeof(VT);
    if (o.vec) {
        if (o.ch == 1) go(k_gm_orth<VT, 1, VW>);
        else if (o.ch == 2) go(k_gm_orth<VT, 2, VW>);
        else if constexpr (MV >= 4) go(k_gm_orth<VT, 4, VW>);
    } else {
        if (o.ch == 1) go(k_gm_orth<VT, 1, 1>);
        else if (o.ch == 2) go(k_gm_orth<VT, 2, 1>);
        else if (o.ch == 4) go(k_gm_orth<VT, 4, 1>);
        else if (o.ch == 8) go(k_gm_orth<VT, 8, 1>);
        else if constexpr (MS >= 16) go(k_gm_orth<VT, 16, 1>);
    }
}

}  // namespace xs
