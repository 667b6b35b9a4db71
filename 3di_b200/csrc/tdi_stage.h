// Large uploads of pageable host memory, staged through pinned slots by a few threads. A plain
// cudaMemcpyAsync of pageable memory is one thread copying through the driver's buffers (8-13 GB/s
// here); with STAGE_THREADS threads the pinned transfers (about 45 GB/s) are kept fed: the windows of
// 13 decoded 1080p frames, crops formed and read back, 7.1 -> 3.3 ms. Pinned memory and small copies go straight
// to cudaMemcpyAsync.
//
// The slots (8 MiB) are the process's: pinning memory takes 4-14 ms, which a batch must not pay for
// its first frames. They are allocated at the first staged upload of video frames, or of crops from
// STAGE_PIN bytes (24 frames' crops, 6 MB: 0.7 ms plain, 4.5 ms when the slots are pinned for them; a
// plain copy of 64 MB takes as long as pinning and staging it), and given back when the last
// batch is destroyed. One upload uses them at a time and has left them when it returns; an
// upload that finds them busy (another thread's batch), or is on the per-thread default stream, makes
// plain copies instead.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <mutex>
#include <thread>
#include <vector>

namespace tdi {

constexpr int STAGE_THREADS = 4;                        // threads of an upload, the caller included
constexpr size_t STAGE_SLOT = (size_t)1 << 20;          // bytes per slot, two slots per thread
constexpr size_t STAGE_MIN = (size_t)2 << 20;           // smaller uploads are not staged
constexpr size_t STAGE_PIN = (size_t)64 << 20;          // crops already formed: slots are pinned for them from here on

// A piece of an upload: rows of `width` bytes, `pitch` bytes apart on the host, packed on the device.
struct StagePiece {
    const char *host;
    size_t pitch, width, rows;
    char *dev;
};

struct StagePool {
    std::mutex mu;
    char *slots = nullptr;                              // [STAGE_THREADS][2][STAGE_SLOT], pinned, for every device
    int users = 0;                                      // live batches

    void retain()
    {
        std::lock_guard<std::mutex> lk(mu);
        ++users;
    }

    void release()
    {
        std::lock_guard<std::mutex> lk(mu);
        if (--users > 0 || !slots) return;
        cudaFreeHost(slots);
        slots = nullptr;
    }
};

inline StagePool &stage_pool()
{
    static StagePool *p = new StagePool();              // (never destroyed: no CUDA call at process exit)
    return *p;
}

inline bool stage_pageable(const void *p)
{
    cudaPointerAttributes a;
    if (cudaPointerGetAttributes(&a, p) != cudaSuccess) { cudaGetLastError(); return true; }
    return a.type == cudaMemoryTypeUnregistered;
}

// The pieces by plain copies.
inline cudaError_t stage_plain(const std::vector<StagePiece> &pieces, cudaStream_t s)
{
    for (const StagePiece &p : pieces) {
        const cudaError_t e = p.pitch == p.width || p.rows == 1
                                  ? cudaMemcpyAsync(p.dev, p.host, p.width * p.rows, cudaMemcpyHostToDevice, s)
                                  : cudaMemcpy2DAsync(p.dev, p.width, p.host, p.pitch, p.width, p.rows, cudaMemcpyHostToDevice, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Uploads the pieces on s; pins the slots, if no upload has, for pin_min bytes or more. Staged uploads
// are complete when it returns; plain ones are enqueued.
inline cudaError_t stage_upload(const std::vector<StagePiece> &pieces, size_t pin_min, cudaStream_t s)
{
    size_t total = 0;
    for (const StagePiece &p : pieces) total += p.width * p.rows;
    // (the per-thread default stream is another stream in each staging thread: their copies would not wait
    // for the caller's earlier work)
    if (total < STAGE_MIN || s == cudaStreamPerThread || !stage_pageable(pieces[0].host)) return stage_plain(pieces, s);
    StagePool &pool = stage_pool();
    std::unique_lock<std::mutex> lk(pool.mu, std::try_to_lock);
    if (!lk.owns_lock()) return stage_plain(pieces, s);
    if (!pool.slots && total < pin_min) return stage_plain(pieces, s);
    if (!pool.slots && cudaHostAlloc(&pool.slots, STAGE_THREADS * 2 * STAGE_SLOT, cudaHostAllocPortable) != cudaSuccess) {
        cudaGetLastError();
        pool.slots = nullptr;
        return stage_plain(pieces, s);
    }
    int device = 0;
    cudaError_t e0 = cudaGetDevice(&device);
    if (e0 != cudaSuccess) return e0;
    // pieces cut to the slots
    std::vector<StagePiece> cut;
    for (const StagePiece &p : pieces) {
        if (p.pitch == p.width || p.rows == 1) {
            for (size_t o = 0, n = p.width * p.rows; o < n; o += STAGE_SLOT)
                cut.push_back({p.host + o, 0, std::min(STAGE_SLOT, n - o), 1, p.dev + o});
        } else if (p.width > STAGE_SLOT) {
            for (size_t r = 0; r < p.rows; ++r)
                for (size_t o = 0; o < p.width; o += STAGE_SLOT)
                    cut.push_back({p.host + r * p.pitch + o, 0, std::min(STAGE_SLOT, p.width - o), 1, p.dev + r * p.width + o});
        } else {
            const size_t per = STAGE_SLOT / p.width;
            for (size_t r = 0; r < p.rows; r += per)
                cut.push_back({p.host + r * p.pitch, p.pitch, p.width, std::min(per, p.rows - r), p.dev + r * p.width});
        }
    }
    std::atomic<size_t> next{0};
    std::atomic<int> err{(int)cudaSuccess};
    auto work = [&](int t) {
        cudaEvent_t ev[2] = {nullptr, nullptr};
        auto ok = [&](cudaError_t e) { if (e != cudaSuccess) err = (int)e; return e == cudaSuccess; };
        bool good = (t == 0 || ok(cudaSetDevice(device))) && ok(cudaEventCreateWithFlags(&ev[0], cudaEventDisableTiming)) &&
                    ok(cudaEventCreateWithFlags(&ev[1], cudaEventDisableTiming));
        for (int q = 0; good && err == (int)cudaSuccess; q ^= 1) {
            const size_t i = next.fetch_add(1);
            if (i >= cut.size()) break;
            const StagePiece &p = cut[i];
            char *slot = pool.slots + ((size_t)t * 2 + q) * STAGE_SLOT;
            good = ok(cudaEventSynchronize(ev[q]));     // the slot's last transfer has left it
            if (!good) break;
            for (size_t r = 0; r < p.rows; ++r) std::memcpy(slot + r * p.width, p.host + r * p.pitch, p.width);
            good = ok(cudaMemcpyAsync(p.dev, slot, p.width * p.rows, cudaMemcpyHostToDevice, s)) && ok(cudaEventRecord(ev[q], s));
        }
        for (cudaEvent_t e : ev)
            if (e) { ok(cudaEventSynchronize(e)); cudaEventDestroy(e); }
    };
    std::vector<std::thread> th;
    th.reserve(STAGE_THREADS);
    try {
        for (int t = 1; t < (int)std::min<size_t>(STAGE_THREADS, cut.size()); ++t) th.emplace_back(work, t);
    } catch (...) {                                     // fewer threads: the others take their pieces
    }
    work(0);
    for (auto &t : th) t.join();
    return (cudaError_t)err.load();
}

}  // namespace tdi
