"""Which way an upload takes (tdi_stage.h), on the CPU with a stand-in for the CUDA runtime that records
every copy: staged through the pinned slots by several threads, or by plain copies from the calling thread
where the upload is small, the memory pinned, the slots busy or refused, or the stream is the per-thread
default stream (which names another stream in every thread, so that copies made by the staging threads
would not wait for the caller's earlier work). Every byte arrives in each of them."""
import ctypes
import os
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))

RUNTIME = r"""
#pragma once
#include <cstddef>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <thread>
typedef int cudaError_t;
typedef struct CUstream_st *cudaStream_t;
typedef struct { int x; } *cudaEvent_t;
enum { cudaSuccess = 0, cudaErrorMemoryAllocation = 2 };
enum { cudaMemcpyHostToDevice = 1, cudaEventDisableTiming = 2, cudaHostAllocPortable = 1 };
enum cudaMemoryType { cudaMemoryTypeUnregistered = 0, cudaMemoryTypeHost = 1 };
struct cudaPointerAttributes { cudaMemoryType type; };
#define cudaStreamLegacy ((cudaStream_t)0x1)
#define cudaStreamPerThread ((cudaStream_t)0x2)
struct Fake {
    std::mutex mu;
    std::thread::id caller;
    int pinned = 0, refuse = 0;                    // settings
    int copies = 0, elsewhere = 0, from_slots = 0; // all copies; from other threads; out of the pinned slots
    char *lo = nullptr, *hi = nullptr;             // the slots
    int allocs = 0, frees = 0;
};
inline Fake &fake() { static Fake f; return f; }
inline cudaError_t cudaGetLastError() { return 0; }
inline cudaError_t cudaGetDevice(int *d) { *d = 0; return 0; }
inline cudaError_t cudaSetDevice(int) { return 0; }
inline cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, int) { *e = (cudaEvent_t)std::malloc(8); return 0; }
inline cudaError_t cudaEventSynchronize(cudaEvent_t) { return 0; }
inline cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return 0; }
inline cudaError_t cudaEventDestroy(cudaEvent_t e) { std::free(e); return 0; }
inline cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *)
{ a->type = fake().pinned ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered; return 0; }
template <class T> inline cudaError_t cudaHostAlloc(T **p, size_t n, int)
{
    if (fake().refuse) return cudaErrorMemoryAllocation;
    *p = (T *)std::malloc(n);
    fake().lo = (char *)*p; fake().hi = fake().lo + n; ++fake().allocs;
    return 0;
}
inline cudaError_t cudaFreeHost(void *p) { std::free(p); fake().lo = fake().hi = nullptr; ++fake().frees; return 0; }
inline cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t rows, int, cudaStream_t)
{
    {
        std::lock_guard<std::mutex> lk(fake().mu);
        ++fake().copies;
        fake().elsewhere += std::this_thread::get_id() != fake().caller;
        fake().from_slots += (const char *)s >= fake().lo && (const char *)s < fake().hi;
    }
    for (size_t r = 0; r < rows; ++r) std::memcpy((char *)d + r * dp, (const char *)s + r * sp, w);
    return 0;
}
inline cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, int k, cudaStream_t st)
{ return cudaMemcpy2DAsync(d, n, s, n, n, 1, k, st); }
"""

HARNESS = r"""
#include "tdi_stage.h"
using namespace tdi;
// One upload of n windows [rows][width] (pitch apart on the host) on a stream; out: copies, those from other
// threads, those out of the slots, wrong bytes, allocations and releases of the slots so far.
extern "C" int upload(int n, long width, long pitch, long rows, long stream, int pinned, int refuse, int busy, int *out)
{
    Fake &f = fake();
    f.caller = std::this_thread::get_id();
    f.pinned = pinned; f.refuse = refuse;
    f.copies = f.elsewhere = f.from_slots = 0;
    std::vector<char> host((size_t)n * pitch * rows), dev((size_t)n * width * rows, 0);
    unsigned r = 12345;
    for (char &c : host) c = (char)((r = r * 1664525u + 1013904223u) >> 24);
    std::vector<StagePiece> pieces;
    for (int i = 0; i < n; ++i)
        pieces.push_back({host.data() + (size_t)i * pitch * rows, (size_t)pitch, (size_t)width, (size_t)rows,
                          dev.data() + (size_t)i * width * rows});
    cudaError_t e;
    if (busy) {                                         // another thread's upload holds the slots
        std::mutex go; go.lock();
        std::atomic<bool> held{false};
        std::thread other([&] { std::lock_guard<std::mutex> lk(stage_pool().mu); held = true; go.lock(); });
        while (!held) std::this_thread::yield();
        e = stage_upload(pieces, STAGE_MIN, (cudaStream_t)stream);
        go.unlock();
        other.join();
    } else {
        e = stage_upload(pieces, STAGE_MIN, (cudaStream_t)stream);
    }
    int wrong = 0;
    for (int i = 0; i < n; ++i)
        for (long y = 0; y < rows; ++y)
            wrong += std::memcmp(dev.data() + ((size_t)i * rows + y) * width, host.data() + ((size_t)i * rows + y) * pitch, width) != 0;
    const int o[6] = {f.copies, f.elsewhere, f.from_slots, wrong, f.allocs, f.frees};
    std::memcpy(out, o, sizeof(o));
    return e;
}
extern "C" void retain() { stage_pool().retain(); }
extern "C" void release() { stage_pool().release(); }
extern "C" void reset() { fake().allocs = fake().frees = 0; }
"""

LEGACY, PER_THREAD, OTHER = 0, 2, 0x1000


@pytest.fixture(scope="module")
def built(tmp_path_factory):
    tmp_path = tmp_path_factory.mktemp("stage")
    (tmp_path / "cuda_runtime.h").write_text(RUNTIME)
    (tmp_path / "h.cpp").write_text(HARNESS)
    so = str(tmp_path / "stage.so")
    subprocess.run(["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-pthread", f"-I{tmp_path}",
                    "-I" + os.path.join(ROOT, "3di_b200", "csrc"), "-o", so, str(tmp_path / "h.cpp")], check=True)
    return ctypes.CDLL(so)


@pytest.fixture()
def lib(built):
    built.reset()
    return built


def _upload(lib, n, width, pitch, rows, stream=OTHER, pinned=0, refuse=0, busy=0):
    out = (ctypes.c_int * 6)()
    c = ctypes.c_long
    assert lib.upload(n, c(width), c(pitch), c(rows), c(stream), pinned, refuse, busy, out) == 0
    copies, elsewhere, from_slots, wrong, allocs, frees = out
    assert wrong == 0
    return copies, elsewhere, from_slots, allocs, frees


@pytest.mark.parametrize("n,width,pitch,rows", [(3, 3000, 5760, 900), (1, 5 << 20, 5 << 20, 1), (2, (1 << 20) + 5, (1 << 20) + 9, 3),
                                                (13, 2401, 5760, 77)])
@pytest.mark.parametrize("stream", [LEGACY, OTHER])
def test_large_pageable_uploads_are_staged(lib, n, width, pitch, rows, stream):
    lib.retain()
    copies, _, from_slots, allocs, frees = _upload(lib, n, width, pitch, rows, stream)
    assert copies == from_slots > 0 and (allocs, frees) == (1, 0)
    assert _upload(lib, n, width, pitch, rows, stream)[3] == 1          # the slots are kept
    lib.retain()
    lib.release()
    assert _upload(lib, n, width, pitch, rows, stream)[4] == 0
    lib.release()                                                       # and given back with the last batch
    assert _upload(lib, 1, 100, 100, 1)[4] == 1


@pytest.mark.parametrize("n,width,pitch,rows", [(3, 3000, 5760, 900), (1, 5 << 20, 5 << 20, 1)])
@pytest.mark.parametrize("kw", [dict(stream=PER_THREAD), dict(pinned=1), dict(refuse=1), dict(busy=1)])
def test_other_uploads_are_plain_copies_of_the_caller(lib, n, width, pitch, rows, kw):
    lib.retain()
    for _ in range(2):
        copies, elsewhere, from_slots, allocs, _ = _upload(lib, n, width, pitch, rows, **kw)
        assert (copies, elsewhere, from_slots, allocs) == (n, 0, 0, 0), kw
    lib.release()


def test_small_uploads_are_plain_copies(lib):
    lib.retain()
    assert _upload(lib, 2, 1000, 3000, 100)[:4] == (2, 0, 0, 0)
    lib.release()
