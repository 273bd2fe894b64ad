"""The pageable arrays' copies (aeo_hostcopy.h) on the host, against a stand-in of the CUDA runtime whose transfers
run only when something waits for them, and which refuses or fails calls on demand."""
import os
import shutil
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "aeolus.jl_b200", "csrc")

RUNTIME = r"""
#pragma once
#include <condition_variable>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <mutex>
#include <new>
#include <vector>
enum cudaError_t { cudaSuccess = 0, cudaErrorMemoryAllocation = 2, cudaErrorUnknown = 999 };
enum cudaMemcpyKind { cudaMemcpyHostToDevice = 1, cudaMemcpyDeviceToHost = 2 };
enum { cudaHostRegisterPortable = 1, cudaEventDisableTiming = 2 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes { cudaMemoryType type; };

namespace fake {
struct Transfer { void* dst; const void* src; size_t n; bool done = false; };
struct Stream { std::vector<Transfer> queue; };
struct Event { Stream* s = nullptr; size_t upto = 0; };
inline std::mutex m;
inline char* pin = nullptr;
inline size_t pin_bytes = 0;
inline int allocs = 0, frees = 0, copies = 0, plain = 0, records = 0;
inline bool refuse = false;
inline int fail_copy = -1, fail_record = -1, fail_create = -1, creates = 0;
inline std::function<void()> at_wait;
inline bool of_pin(const void* p) { return pin && p >= pin && p < pin + pin_bytes; }
inline void run(Stream* s, size_t upto) {
    for (size_t q = 0; q < upto; ++q) {
        Transfer& t = s->queue[q];
        if (!t.done) { std::memcpy(t.dst, t.src, t.n); t.done = true; }
    }
}
inline int in_flight(Stream* s) {
    int n = 0;
    for (auto& t : s->queue) n += !t.done && (of_pin(t.src) || of_pin(t.dst));
    return n;
}
}  // namespace fake
typedef fake::Stream* cudaStream_t;
typedef fake::Event* cudaEvent_t;

inline cudaError_t cudaGetLastError() { return cudaSuccess; }
inline cudaError_t cudaSetDevice(int) { return cudaSuccess; }
inline cudaError_t cudaHostRegister(void* p, size_t n, unsigned) {
    std::lock_guard<std::mutex> l(fake::m);
    if (fake::refuse) return cudaErrorMemoryAllocation;
    ++fake::allocs;
    fake::pin = static_cast<char*>(p);
    fake::pin_bytes = n;
    return cudaSuccess;
}
inline cudaError_t cudaHostUnregister(void*) {
    std::lock_guard<std::mutex> l(fake::m);
    ++fake::frees;
    fake::pin = nullptr;
    return cudaSuccess;
}
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    a->type = cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
// a pageable copy has read its source (or, to the host, is complete) when it returns; a pinned one is only queued
inline cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    std::lock_guard<std::mutex> l(fake::m);
    if (fake::copies++ == fake::fail_copy) return cudaErrorUnknown;
    st->queue.push_back({d, s, n});
    if (!fake::of_pin(d) && !fake::of_pin(s)) {
        ++fake::plain;
        fake::run(st, st->queue.size());
    }
    return cudaSuccess;
}
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    std::lock_guard<std::mutex> l(fake::m);
    if (fake::creates++ == fake::fail_create) return cudaErrorUnknown;
    *e = new (std::malloc(sizeof(fake::Event))) fake::Event;
    return cudaSuccess;
}
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return cudaSuccess; }
inline cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    std::lock_guard<std::mutex> l(fake::m);
    if (fake::records++ == fake::fail_record) return cudaErrorUnknown;
    e->s = s;
    e->upto = s->queue.size();
    return cudaSuccess;
}
inline cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    if (fake::at_wait) fake::at_wait();
    std::lock_guard<std::mutex> l(fake::m);
    fake::run(e->s, e->upto);
    return cudaSuccess;
}
inline cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    std::lock_guard<std::mutex> l(fake::m);
    fake::run(s, s->queue.size());
    return cudaSuccess;
}
"""

HEAD = r"""
#include "cuda_runtime.h"
#include "aeo_hostcopy.h"
#include <chrono>
#include <cstdio>
#include <future>
#include <atomic>
#define REQUIRE(x) do { if (!(x)) { std::printf("line %d: %s\n", __LINE__, #x); std::fflush(stdout); std::_Exit(1); } } while (0)
// in the place of the library's: one lane, or all of them
unsigned std::thread::hardware_concurrency() noexcept { return CORES; }
std::vector<char> bytes(size_t n, int seed) {
    std::vector<char> a(n);
    unsigned x = 2463534242u + seed;
    for (auto& c : a) { x ^= x << 13; x ^= x >> 17; x ^= x << 5; c = (char)x; }
    return a;
}
"""

PROGRAMS = {
    # a handle pins nothing until its pageable copies have paid for the buffers; the last one gives them back
    "kept": r"""
int main() {
    fake::Stream st;
    auto a = bytes(HostStage::PAYS + 12345, 1);
    std::vector<char> d(a.size()), b(a.size());
    {
        HostStage one, two;
        REQUIRE(fake::allocs == 0);
        const size_t small = (size_t(8) << 20) - 1, half = HostStage::PAYS / 2;   // below 8 MiB the plain call is faster
        for (int q = 0; q < 50; ++q) REQUIRE(one.upload(d.data(), a.data(), small, 0, &st) == cudaSuccess);
        REQUIRE(one.upload(d.data(), a.data(), half, 0, &st) == cudaSuccess && fake::allocs == 0);
        REQUIRE(one.upload(d.data(), a.data(), half, 0, &st) == cudaSuccess && fake::allocs == 1);
        const int plain = fake::plain;
        REQUIRE(one.upload(d.data(), a.data(), a.size(), 0, &st) == cudaSuccess);
        REQUIRE(two.download(b.data(), d.data(), a.size(), 0, &st) == cudaSuccess);
        REQUIRE(b == a && fake::allocs == 1 && fake::plain == plain && fake::in_flight(&st) == 0);
    }
    REQUIRE(fake::frees == 1);
    HostStage three;   // a first array of that size is worth them at once
    REQUIRE(three.download(b.data(), d.data(), a.size(), 0, &st) == cudaSuccess && fake::allocs == 2);
}
""",
    # a call that fails leaves no transfer under way through the buffers, which the next copy uses (on one core too,
    # where one thread has all chunks and no other one waits for them)
    "failed": r"""
int main() {
    auto a = bytes(HostStage::PAYS + 4321, 3);
    std::vector<char> d(a.size()), b(a.size());
    HostStage keep;
    fake::Stream st;
    REQUIRE(keep.upload(d.data(), a.data(), a.size(), 0, &st) == cudaSuccess && fake::allocs == 1);
    for (int which = 0; which < 3; ++which)
        for (int at : {0, 1, 5, 11, 20})
            for (bool up : {true, false}) {
                fake::Stream s1;
                if (which == 0) fake::fail_copy = fake::copies + at;
                if (which == 1) fake::fail_record = fake::records + at;
                if (which == 2) fake::fail_create = fake::creates + (at & 1);
                cudaError_t e = up ? keep.upload(d.data(), a.data(), a.size(), 0, &s1) : keep.download(b.data(), d.data(), a.size(), 0, &s1);
                REQUIRE(e == cudaErrorUnknown);
                REQUIRE(fake::in_flight(&s1) == 0);
                fake::fail_copy = fake::fail_record = fake::fail_create = -1;
                REQUIRE(keep.upload(d.data(), a.data(), a.size(), 0, &s1) == cudaSuccess);
                REQUIRE(keep.download(b.data(), d.data(), a.size(), 0, &s1) == cudaSuccess && b == a);
            }
}
""",
    # while one copy has the buffers, another handle's goes the plain way and does not wait for it
    "busy": r"""
int main() {
    fake::Stream s1, s2;
    auto a = bytes(HostStage::PAYS, 4), b = bytes(HostStage::PAYS, 5);
    std::vector<char> da(a.size()), db(a.size()), back(a.size());
    HostStage one, two;
    REQUIRE(one.upload(da.data(), a.data(), a.size(), 0, &s1) == cudaSuccess);
    REQUIRE(two.upload(db.data(), b.data(), b.size(), 0, &s2) == cudaSuccess && fake::allocs == 1);
    std::promise<void> go;
    auto gate = go.get_future().share();
    std::atomic<int> held{0};
    fake::at_wait = [&] { ++held; gate.wait(); };
    auto first = std::async(std::launch::async, [&] { return one.upload(da.data(), a.data(), a.size(), 0, &s1); });
    while (!held) std::this_thread::yield();
    std::fill(db.begin(), db.end(), 0);
    auto second = std::async(std::launch::async, [&] {
        cudaError_t e = two.upload(db.data(), b.data(), b.size(), 0, &s2);
        return e == cudaSuccess ? two.download(back.data(), db.data(), b.size(), 0, &s2) : e;
    });
    const bool through = second.wait_for(std::chrono::seconds(20)) == std::future_status::ready;
    go.set_value();
    REQUIRE(through && first.get() == cudaSuccess && second.get() == cudaSuccess && da == a && back == b);
}
""",
    # a lane whose thread cannot be had, for want of threads or of memory, runs on the calling one
    "threads": r"""
thread_local bool starved = false;
void* operator new(size_t n) {
    void* p = starved ? nullptr : std::malloc(n);
    if (!p) throw std::bad_alloc();
    return p;
}
void operator delete(void* p) noexcept { std::free(p); }
void operator delete(void* p, size_t) noexcept { std::free(p); }
int main() {
    fake::Stream st;
    st.queue.reserve(1 << 12);
    auto a = bytes(HostStage::PAYS + 99, 6);
    std::vector<char> d(a.size()), b(a.size());
    HostStage s;
    REQUIRE(s.upload(d.data(), a.data(), a.size(), 0, &st) == cudaSuccess);
    std::fill(d.begin(), d.end(), 0);
    starved = true;
    const cudaError_t up = s.upload(d.data(), a.data(), a.size(), 0, &st), down = s.download(b.data(), d.data(), a.size(), 0, &st);
    starved = false;
    REQUIRE(up == cudaSuccess && down == cudaSuccess && b == a);
}
""",
    # where pinned memory is refused the copies still work
    "refused": r"""
int main() {
    fake::Stream st;
    fake::refuse = true;
    auto a = bytes(HostStage::PAYS + 1, 2);
    std::vector<char> d(a.size()), b(a.size());
    HostStage s;
    for (int q = 0; q < 3; ++q) {
        REQUIRE(s.upload(d.data(), a.data(), a.size(), 0, &st) == cudaSuccess);
        REQUIRE(s.download(b.data(), d.data(), a.size(), 0, &st) == cudaSuccess);
    }
    REQUIRE(b == a && fake::allocs == 0);
    fake::refuse = false;
    REQUIRE(s.upload(d.data(), a.data(), a.size(), 0, &st) == cudaSuccess && fake::allocs == 1);
}
""",
}


@pytest.mark.parametrize("cores", [1, 12])
@pytest.mark.parametrize("name", sorted(PROGRAMS))
def test_host_copy(tmp_path, name, cores):
    if shutil.which("g++") is None:
        pytest.skip("no host compiler")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "main.cpp").write_text(HEAD + PROGRAMS[name])
    exe = str(tmp_path / "main")
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", f"-DCORES={cores}", "-I", str(tmp_path), "-I", CSRC, "-o", exe,
                    str(tmp_path / "main.cpp")], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=120)
    assert r.returncode == 0, r.stdout + r.stderr
