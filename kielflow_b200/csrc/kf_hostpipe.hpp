// kf_hostpipe.hpp -- copies between pageable host arrays and the device.
//
// cudaMemcpyAsync stages a pageable array through the driver's buffer on the
// calling thread: 10 GB/s in at 128^3 (16.8 MB), and 4 GB/s out into memory that is
// touched for the first time, as a fresh numpy array is, because the page faults
// are taken one by one there.  Here a few threads each take a range of the array,
// copy it through two pinned pieces of their own and queue their own transfers on
// the stream, so that the host copies, the faults and the transfers overlap.
// Page-locked or device-visible arrays, small ones and the per-thread default stream
// (whose handle names another stream in each thread) take cudaMemcpyAsync.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <exception>
#include <thread>
#include <vector>

namespace kf {

class HostPipe {
  public:
    static constexpr size_t kPiece = 256 << 10;  // bytes of a pinned piece
    static constexpr size_t kMin = 4 << 20;    // smaller arrays: one plain copy
    static constexpr int kThreads = 8;
    // Pageable bytes after which the pieces are made: allocating them takes 2 to 5 ms,
    // about what this many bytes lose by plain copies, so an object that is used
    // once does not pay for them.
    static constexpr size_t kAfter = 64 << 20;

    HostPipe() = default;
    HostPipe(const HostPipe &) = delete;
    HostPipe &operator=(const HostPipe &) = delete;
    ~HostPipe() {
        for (cudaEvent_t e : ev_)
            if (e) cudaEventDestroy(e);
        if (buf_) cudaFreeHost(buf_);
    }

    // As cudaMemcpyAsync on st: an upload's source may change on return, a
    // download's target is complete on return.
    cudaError_t copy(void *dst, const void *src, size_t bytes, bool up, cudaStream_t st) {
        const cudaMemcpyKind kind = up ? cudaMemcpyHostToDevice : cudaMemcpyDeviceToHost;
        if (bytes < kMin || st == cudaStreamPerThread || !pageable(up ? src : dst) || !ready(bytes))
            return cudaMemcpyAsync(dst, src, bytes, kind, st);
        int dev = 0;
        cudaError_t e = cudaGetDevice(&dev);
        if (e != cudaSuccess) return e;
        const int nt = (int)ev_.size() / 2;
        const size_t part = ((bytes + nt - 1) / nt + 4095) / 4096 * 4096;  // nt parts hold all of it
        std::vector<cudaError_t> err(nt, cudaSuccess);
        std::vector<std::thread> th;
        th.reserve(nt);
        int own = 0;  // ranges from here on are taken by this thread
        try {
            for (; own + 1 < nt; ++own)
                th.emplace_back([&, own, dev] {
                    err[own] = cudaSetDevice(dev);
                    if (err[own] == cudaSuccess) err[own] = range(own, part, dst, src, bytes, up, st);
                });
        } catch (const std::exception &) {  // no thread to be had: fewer do it
        }
        for (int k = own; k < nt; ++k) err[k] = range(k, part, dst, src, bytes, up, st);
        for (std::thread &t : th) t.join();
        for (cudaError_t x : err)
            if (x != cudaSuccess) return x;
        return cudaSuccess;
    }

  private:
    std::vector<cudaEvent_t> ev_;  // two per thread: its pieces' last transfers
    char *buf_ = nullptr;
    size_t seen_ = 0;  // pageable bytes asked for so far

    static bool pageable(const void *p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        return a.type == cudaMemoryTypeUnregistered;
    }

    // The pinned pieces and their events, before a copy of `bytes`; false: plain copies.
    bool ready(size_t bytes) {
        if (buf_) return true;
        if ((seen_ += bytes) <= kAfter) return false;
        const int nt = std::min(kThreads, (int)std::thread::hardware_concurrency() / 2);
        if (nt < 2) return false;
        if (cudaMallocHost(&buf_, 2 * kPiece * nt) != cudaSuccess) {
            cudaGetLastError();
            buf_ = nullptr;
            return false;
        }
        ev_.assign(2 * nt, nullptr);
        for (cudaEvent_t &e : ev_)
            if (cudaEventCreateWithFlags(&e, cudaEventDisableTiming) != cudaSuccess) {
                cudaGetLastError();
                for (cudaEvent_t x : ev_)
                    if (x) cudaEventDestroy(x);
                ev_.clear();
                cudaFreeHost(buf_);
                buf_ = nullptr;
                return false;
            }
        return true;
    }

    // Range k of `part` bytes through the two pieces of thread k.
    cudaError_t range(int k, size_t part, void *dst, const void *src, size_t bytes, bool up, cudaStream_t st) {
        const size_t lo = std::min(bytes, (size_t)k * part), hi = std::min(bytes, lo + part);
        char *piece[2] = {buf_ + (size_t)(2 * k) * kPiece, buf_ + (size_t)(2 * k + 1) * kPiece};
        cudaEvent_t *ev = &ev_[2 * k];
        cudaError_t e = cudaSuccess;
        auto len = [&](size_t o) { return std::min(kPiece, hi - o); };
        size_t done = lo;  // download: what has been handed to the caller's array
        int b = 0;
        for (size_t o = lo; o < hi && e == cudaSuccess; o += kPiece, b ^= 1) {
            if (up) {
                // the piece's last transfer (of an earlier copy, on whatever stream) has to be over
                if ((e = cudaEventSynchronize(ev[b])) != cudaSuccess) break;
                std::memcpy(piece[b], (const char *)src + o, len(o));
                if ((e = cudaMemcpyAsync((char *)dst + o, piece[b], len(o), cudaMemcpyHostToDevice, st)) != cudaSuccess) break;
                e = cudaEventRecord(ev[b], st);
            } else {
                if (o >= lo + 2 * kPiece) e = drain(dst, piece, ev, b, done, len(done));
                if (e != cudaSuccess) break;
                if (o < lo + 2 * kPiece && (e = cudaEventSynchronize(ev[b])) != cudaSuccess) break;
                if ((e = cudaMemcpyAsync(piece[b], (const char *)src + o, len(o), cudaMemcpyDeviceToHost, st)) != cudaSuccess) break;
                e = cudaEventRecord(ev[b], st);
            }
        }
        if (!up)
            for (int q = (int)((done - lo) / kPiece) & 1; done < hi && e == cudaSuccess; q ^= 1)
                e = drain(dst, piece, ev, q, done, len(done));
        return e;
    }
    static cudaError_t drain(void *dst, char *const *piece, const cudaEvent_t *ev, int b, size_t &done, size_t n) {
        const cudaError_t e = cudaEventSynchronize(ev[b]);
        if (e != cudaSuccess) return e;
        std::memcpy((char *)dst + done, piece[b], n);
        done += n;
        return cudaSuccess;
    }
};

}  // namespace kf
