// aeo_hostcopy.h -- copies between pageable host arrays and the device.
//
// A cudaMemcpyAsync on pageable memory goes through the driver's staging buffer
// on the calling thread, 11 GB/s on the hosts measured; the link does 50.  Here a
// few threads copy the array's chunks into pinned buffers (two a thread) and
// enqueue each chunk's transfer, so that the host copy runs at the memory's
// rate and overlaps the link.  Arrays that are already pinned take the plain call,
// and so do those below SMALL, where starting the threads costs what they save: an
// apply of the network, two copies (ms, plain and by lanes), takes 0.63 and 0.74 on
// arrays of 2.1 MB, 1.43 and 1.47 on 6.3, 2.15 and 1.98 on 12.6, 3.98 and 3.15 on 25,
// 16.8 and 7.0 on 50.
//
// The pinned buffers (LANES x 2 x CHUNK, 12 MiB) belong together to the live handles
// that have use for them: the first such handle pins them, the last one gives them back,
// and one copy at a time uses them (a copy that finds them in use goes the plain way).
// Pinning huge pages and giving them back takes 3.0 ms (7.2 ms by cudaHostAlloc), what the
// lanes save on 30 to 80 MB of 50 MB arrays; a handle asks for them once its pageable
// copies come to PAYS.  So creating a handle pins nothing, one that copies little pays for
// nothing, and where pinned memory is refused the plain call serves.
#pragma once

#include <cuda_runtime.h>
#include <sys/mman.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <exception>
#include <memory>
#include <mutex>
#include <new>
#include <thread>

class HostStage {
public:
    static constexpr size_t CHUNK = size_t(1) << 20, SMALL = size_t(8) << 20, PAYS = size_t(40) << 20;
    static constexpr int LANES = 6;

    // src (host) -> dst (device) on st; returns when a pageable src has been read
    cudaError_t upload(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
        if (Turn turn{*this, src, bytes})
            return lanes(bytes, device, st, [=](char* pin, size_t at, size_t n, cudaEvent_t ev) -> cudaError_t {
                std::memcpy(pin, static_cast<const char*>(src) + at, n);
                cudaError_t e = cudaMemcpyAsync(static_cast<char*>(dst) + at, pin, n, cudaMemcpyHostToDevice, st);
                return e == cudaSuccess ? cudaEventRecord(ev, st) : e;
            }, [](char*, size_t, size_t) {});
        return cudaMemcpyAsync(dst, src, bytes, cudaMemcpyHostToDevice, st);
    }
    // src (device) -> dst (host), ordered on st; returns when dst is complete
    cudaError_t download(void* dst, const void* src, size_t bytes, int device, cudaStream_t st) {
        if (Turn turn{*this, dst, bytes})
            return lanes(bytes, device, st, [=](char* pin, size_t at, size_t n, cudaEvent_t ev) -> cudaError_t {
                cudaError_t e = cudaMemcpyAsync(pin, static_cast<const char*>(src) + at, n, cudaMemcpyDeviceToHost, st);
                return e == cudaSuccess ? cudaEventRecord(ev, st) : e;
            }, [=](char* pin, size_t at, size_t n) { std::memcpy(static_cast<char*>(dst) + at, pin, n); });
        cudaError_t e = cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, st);
        return e == cudaSuccess ? cudaStreamSynchronize(st) : e;
    }

private:
    struct Buffers {
        char* pin = nullptr;
        std::mutex use;
        ~Buffers() {
            if (!pin) return;
            cudaHostUnregister(pin);
            std::free(pin);
        }
    };
    std::shared_ptr<Buffers> buf_;
    size_t plain_ = 0;   // bytes of this handle's pageable copies so far

    // the live handles' buffers, where there are none made if `make`; null without, or where pinned
    // memory is refused
    static std::shared_ptr<Buffers> shared(bool make) {
        static std::mutex m;
        static std::weak_ptr<Buffers> live;
        std::lock_guard<std::mutex> lock(m);
        std::shared_ptr<Buffers> s = live.lock();
        if (s || !make) return s;
        try {
            s = std::make_shared<Buffers>();
        } catch (const std::bad_alloc&) {
            return nullptr;
        }
        const size_t n = LANES * 2 * CHUNK;
        void* p = std::aligned_alloc(size_t(2) << 20, n);
        if (!p) return nullptr;
        madvise(p, n, MADV_HUGEPAGE);
        if (cudaHostRegister(p, n, cudaHostRegisterPortable) != cudaSuccess) {
            cudaGetLastError();
            std::free(p);
            return nullptr;
        }
        s->pin = static_cast<char*>(p);
        live = s;
        return s;
    }
    // whether this copy takes the lanes (after a refusal the count starts again)
    bool buffers(size_t bytes) {
        if (buf_) return true;
        plain_ += bytes;
        const bool make = plain_ >= PAYS;
        if (make) plain_ = 0;
        buf_ = shared(make);
        return buf_ != nullptr;
    }

    // Whether a copy of the host array at p has the buffers: held while it runs, never waited for (another copy,
    // of another device perhaps, has them: the plain call is no slower than waiting).
    struct Turn {
        std::unique_lock<std::mutex> lock;
        Turn(HostStage& s, const void* p, size_t bytes) {
            if (bytes >= SMALL && !pinned(p) && s.buffers(bytes)) lock = std::unique_lock<std::mutex>(s.buf_->use, std::try_to_lock);
        }
        explicit operator bool() const { return lock.owns_lock(); }
    };

    static bool pinned(const void* p) {
        cudaPointerAttributes a{};
        if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return false; }
        return a.type != cudaMemoryTypeUnregistered;
    }

    // Lane l takes the chunks l, l + nl, ... through its two buffers: go(buffer, offset,
    // bytes, event) starts a chunk, done(buffer, offset, bytes) runs once its event has
    // passed, before the buffer's next chunk and at the end.  After an error what was already
    // enqueued on st is waited for: the buffers are the next copy's.
    template <class Go, class Done>
    cudaError_t lanes(size_t bytes, int device, cudaStream_t st, Go go, Done done) {
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
                if (e == cudaSuccess) done(buf_->pin + (size_t)(2 * l + b) * CHUNK, at, std::min(CHUNK, bytes - at));
                held[b] = nc;
            };
            int b = 0;
            for (size_t c = (size_t)l; c < nc && e == cudaSuccess; c += (size_t)nl, b ^= 1) {
                finish(b);
                if (e != cudaSuccess) break;
                const size_t at = c * CHUNK;
                e = go(buf_->pin + (size_t)(2 * l + b) * CHUNK, at, std::min(CHUNK, bytes - at), ev[b]);
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
            } catch (const std::exception&) {
                lane(l);   // no thread (or no memory for one) to be had: this one does the lane's chunks
            }
        }
        lane(0);
        for (int l = 1; l < nl; ++l)
            if (th[l].joinable()) th[l].join();
        for (int l = 0; l < nl; ++l)
            if (err[l] != cudaSuccess) {
                cudaStreamSynchronize(st);
                return err[l];
            }
        return cudaSuccess;
    }
};
