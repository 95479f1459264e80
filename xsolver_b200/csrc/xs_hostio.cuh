// Large copies between the device and a caller's pageable arrays.
//
// The C API takes plain host pointers (hip/xsolver_c.h:37-49), so most
// callers' arrays are pageable.  The driver copies such memory through its
// own staging buffer on one thread, about 10 GB/s, and a fresh result array
// is faulted in page by page on the way.  Here a few host threads each take
// a stripe of the array through a pinned double buffer of their own, so the
// copies, the page faults and the DMA of different stripes overlap.
// Measured (B200 host, a solve of one step: two arrays up, a fresh one down),
// milliseconds with the driver's path / with stripes, by the array's size:
// 8 MB 2.65 / 2.43, 16 MB 5.4 / 3.7, 32 MB 12.8 / 4.5, 128 MB 47 / 14.
//
// One HostIo belongs to one handle and is used by one call at a time, as the
// handle is; its pinned memory is bounded (HOSTIO_THREADS * 2 *
// HOSTIO_CHUNK), allocated at the first large copy and freed with the handle.
#pragma once
#include <cstring>
#include <thread>
#include <vector>
#include "xs_internal.cuh"

namespace xs {

constexpr int HOSTIO_THREADS = 8;
constexpr size_t HOSTIO_CHUNK = (size_t)2 << 20;
// below this the driver's own path is as fast (thread starts and two stream
// synchronisations; the figures above meet at 8 MB)
constexpr size_t HOSTIO_MIN = (size_t)8 << 20;

struct HostIo {
    char *pin = nullptr;
    cudaStream_t st[HOSTIO_THREADS] = {};
    cudaEvent_t ev[HOSTIO_THREADS][2] = {};
    HostIo() = default;
    HostIo(const HostIo &) = delete;
    HostIo &operator=(const HostIo &) = delete;
    ~HostIo()
    {
        for (int t = 0; t < HOSTIO_THREADS; t++) {
            for (cudaEvent_t e : ev[t])
                if (e) cudaEventDestroy(e);
            if (st[t]) cudaStreamDestroy(st[t]);
        }
        if (pin) cudaFreeHost(pin);
    }
    // streams, events and pinned memory, as far as they are not there yet
    bool create()
    {
        for (int t = 0; t < HOSTIO_THREADS; t++) {
            if (!st[t] && cudaStreamCreateWithFlags(&st[t], cudaStreamNonBlocking) != cudaSuccess) return false;
            for (cudaEvent_t &e : ev[t])
                if (!e && cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) return false;
        }
        if (cudaMallocHost((void **)&pin, HOSTIO_THREADS * 2 * HOSTIO_CHUNK) == cudaSuccess) return true;
        pin = nullptr;
        return false;
    }
    // whether a copy goes through the stripes: large, and not pinned already
    // (or managed: the driver copies those at full rate by itself)
    bool striped(const void *host, size_t bytes)
    {
        if (bytes < HOSTIO_MIN || std::thread::hardware_concurrency() < 4) return false;
        cudaPointerAttributes a;
        if (cudaPointerGetAttributes(&a, host) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        if (a.type != cudaMemoryTypeUnregistered) return false;
        if (!pin && !create()) {
            cudaGetLastError();
            return false;  // the driver's own path needs none of it
        }
        return true;
    }
    // fn(thread, first byte, last byte) for the stripes, on host threads of
    // the caller's device; the first CUDA error of any of them is thrown
    template <typename F>
    void stripes(size_t bytes, F fn)
    {
        int dev = 0;
        XS_CUDA(cudaGetDevice(&dev));
        cudaError_t err[HOSTIO_THREADS] = {};
        const size_t per = (bytes / HOSTIO_THREADS + 4095) / 4096 * 4096;
        std::vector<std::thread> th;
        auto run = [&](int t) {
            err[t] = cudaSetDevice(dev);
            const size_t a = std::min(bytes, t * per), b = t == HOSTIO_THREADS - 1 ? bytes : std::min(bytes, a + per);
            if (err[t] == cudaSuccess && a < b) err[t] = fn(t, a, b);
        };
        int started = 1;
        try {
            for (; started < HOSTIO_THREADS; started++) th.emplace_back(run, started);
        } catch (...) {  // no more threads to be had: the rest here
        }
        run(0);
        for (int t = started; t < HOSTIO_THREADS; t++) run(t);
        for (auto &x : th) x.join();
        for (cudaError_t e : err)
            if (e != cudaSuccess) throw Status(XS_ERR_CUDA);
    }
    char *chunk(int t, int q) const { return pin + (size_t)(2 * t + q) * HOSTIO_CHUNK; }

    // device -> host, ordered after stream s; complete when it returns
    void download(void *dst, const void *src, size_t bytes, cudaStream_t s)
    {
        if (!striped(dst, bytes)) {
            XS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s));
            XS_CUDA(cudaStreamSynchronize(s));
            return;
        }
        XS_CUDA(cudaStreamSynchronize(s));
        stripes(bytes, [&](int t, size_t a, size_t b) -> cudaError_t {
            size_t from[2] = {0, 0}, len[2] = {0, 0};
            size_t next = a;
            auto issue = [&](int q) -> cudaError_t {
                from[q] = next;
                len[q] = std::min(HOSTIO_CHUNK, b - next);
                next += len[q];
                cudaError_t e = cudaMemcpyAsync(chunk(t, q), (const char *)src + from[q], len[q], cudaMemcpyDeviceToHost, st[t]);
                return e == cudaSuccess ? cudaEventRecord(ev[t][q], st[t]) : e;
            };
            cudaError_t e = issue(0);
            for (int q = 0; e == cudaSuccess && len[q]; q ^= 1) {
                len[q ^ 1] = 0;
                if (next < b) e = issue(q ^ 1);
                if (e == cudaSuccess) e = cudaEventSynchronize(ev[t][q]);
                if (e == cudaSuccess) std::memcpy((char *)dst + from[q], chunk(t, q), len[q]);
                len[q] = 0;
            }
            return e;
        });
    }
    // host -> device, ordered after stream s.  In stripes it is complete when
    // it returns; otherwise it is a copy in the order of s, and a pinned
    // source has to stay as it is until s has been waited for
    void upload(void *dst, const void *src, size_t bytes, cudaStream_t s)
    {
        if (!striped(src, bytes)) {
            XS_CUDA(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, s));
            return;
        }
        XS_CUDA(cudaStreamSynchronize(s));  // earlier work may still use dst
        stripes(bytes, [&](int t, size_t a, size_t b) -> cudaError_t {
            cudaError_t e = cudaSuccess;
            int q = 0;
            for (size_t p = a, k = 0; e == cudaSuccess && p < b; p += HOSTIO_CHUNK, k++, q ^= 1) {
                const size_t len = std::min(HOSTIO_CHUNK, b - p);
                if (k >= 2) e = cudaEventSynchronize(ev[t][q]);  // the chunk's previous copy has left it
                if (e == cudaSuccess) {
                    std::memcpy(chunk(t, q), (const char *)src + p, len);
                    e = cudaMemcpyAsync((char *)dst + p, chunk(t, q), len, cudaMemcpyHostToDevice, st[t]);
                }
                if (e == cudaSuccess) e = cudaEventRecord(ev[t][q], st[t]);
            }
            const cudaError_t f = cudaStreamSynchronize(st[t]);
            return e == cudaSuccess ? f : e;
        });
    }
};

}  // namespace xs
