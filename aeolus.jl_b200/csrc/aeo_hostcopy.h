// aeo_hostcopy.h -- copies between pageable host arrays and the device.
//
// A cudaMemcpyAsync on pageable memory goes through the driver's staging buffer
// on the calling thread, 11 GB/s on the hosts measured; the link does 50.  Here a
// few threads copy the array's chunks into pinned buffers (two a thread) and
// enqueue each chunk's transfer, so that the host copy runs at the memory's
// rate and overlaps the link.  Arrays that are small or already pinned take the
// plain call.
//
// The pinned buffers (LANES x 2 x CHUNK, 12 MiB) belong to the live handles
// together: the first one allocates them, the last one gives them back, and a
// mutex lets one copy at a time use them.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cstring>
#include <memory>
#include <mutex>
#include <new>
#include <system_error>
#include <thread>

class HostStage {
public:
    static constexpr size_t CHUNK = size_t(1) << 20, SMALL = size_t(2) << 20;
    static constexpr int LANES = 6;

    // the live handles' buffers
    static std::shared_ptr<HostStage> get(cudaError_t* e) {
        static std::mutex m;
        static std::weak_ptr<HostStage> live;
        std::lock_guard<std::mutex> lock(m);
        *e = cudaSuccess;
        std::shared_ptr<HostStage> s = live.lock();
        if (s) return s;
        try {
            s = std::make_shared<HostStage>();
        } catch (const std::bad_alloc&) {
            *e = cudaErrorMemoryAllocation;
            return nullptr;
        }
        *e = cudaHostAlloc(reinterpret_cast<void**>(&s->pin_), LANES * 2 * CHUNK, cudaHostAllocPortable);
        if (*e != cudaSuccess) { s->pin_ = nullptr; return nullptr; }
        live = s;
        return s;
    }
    ~HostStage() {
        if (pin_) cudaFreeHost(pin_);
    }

    // src (host) -> dst (device) on st; returns when src has been read
    cudaError_t upload(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
        if (bytes < SMALL || pinned(src)) return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
        return lanes(bytes, device, [=](char* pin, size_t at, size_t n, cudaEvent_t ev) -> cudaError_t {
            std::memcpy(pin, static_cast<const char*>(src) + at, n);
            cudaError_t e = cudaMemcpyAsync(static_cast<char*>(dst) + at, pin, n, cudaMemcpyHostToDevice, st);
            return e == cudaSuccess ? cudaEventRecord(ev, st) : e;
        }, [](char*, size_t, size_t) {});
    }
    // src (device) -> dst (host), ordered on st; returns when dst is complete
    cudaError_t download(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
        if (bytes < SMALL || pinned(dst)) {
            cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
            return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
        }
        return lanes(bytes, device, [=](char* pin, size_t at, size_t n, cudaEvent_t ev) -> cudaError_t {
            cudaError_t e = cudaMemcpyAsync(pin, static_cast<const char*>(src) + at, n, cudaMemcpyDeviceToHost, st);
            return e == cudaSuccess ? cudaEventRecord(ev, st) : e;
        }, [=](char* pin, size_t at, size_t n) { std::memcpy(static_cast<char*>(dst) + at, pin, n); });
    }

private:
    char* pin_ = nullptr;
    std::mutex use_;

    static bool pinned(const void* p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
        return a.type != cudaMemoryTypeUnregistered;
    }

    // Lane l takes the chunks l, l + nl, ... through its two buffers: go(buffer, offset,
    // bytes, event) starts a chunk, done(buffer, offset, bytes) runs once its event has
    // passed, before the buffer's next chunk and at the end.
    template <class Go, class Done>
    cudaError_t lanes(size_t bytes, int device, Go go, Done done) {
        std::lock_guard<std::mutex> lock(use_);
        const size_t nc = (bytes + CHUNK - 1) / CHUNK;
        const int hw = (int)std::max(1u, std::thread::hardware_concurrency());
        const int nl = (int)std::min<size_t>(nc, (size_t)std::min(LANES, std::max(1, hw / 2)));
        cudaError_t err[LANES];
        auto lane = [&](int l) {
            cudaError_t e = cudaSetDevice(device);
            cudaEvent_t ev[2] = {};
            for (int b = 0; b < 2 && e == cudaSuccess; ++b) e = cudaEventCreateWithFlags(&ev[b], cudaEventDisableTiming);
            size_t held[2] = {nc, nc};   // the chunk in each buffer
            auto finish = [&](int b) {
                if (held[b] == nc) return;
                if (e == cudaSuccess) e = cudaEventSynchronize(ev[b]);
                const size_t at = held[b] * CHUNK;
                if (e == cudaSuccess) done(pin_ + (size_t)(2 * l + b) * CHUNK, at, std::min(CHUNK, bytes - at));
                held[b] = nc;
            };
            int b = 0;
            for (size_t c = (size_t)l; c < nc && e == cudaSuccess; c += (size_t)nl, b ^= 1) {
                finish(b);
                if (e != cudaSuccess) break;
                const size_t at = c * CHUNK;
                e = go(pin_ + (size_t)(2 * l + b) * CHUNK, at, std::min(CHUNK, bytes - at), ev[b]);
                if (e == cudaSuccess) held[b] = c;
            }
            finish(b);
            finish(b ^ 1);
            for (int q = 0; q < 2; ++q)
                if (ev[q]) cudaEventDestroy(ev[q]);
            err[l] = e;
        };
        std::thread th[LANES];
        for (int l = 1; l < nl; ++l) {
            try {
                th[l] = std::thread(lane, l);
            } catch (const std::system_error&) {
                lane(l);   // no thread to be had: this one does the lane's chunks
            }
        }
        lane(0);
        for (int l = 1; l < nl; ++l)
            if (th[l].joinable()) th[l].join();
        for (int l = 0; l < nl; ++l)
            if (err[l] != cudaSuccess) return err[l];
        return cudaSuccess;
    }
};
