// Columns between pageable host arrays and the device, through a few small
// blocks of host memory (dsmc_upload_particles, dsmc_download_particles,
// dsmc_trace).
//
// A transfer is cut into blocks of kItems values, taken by up to kThreads
// host threads; each thread has two blocks of memory, so that the host copy
// (and with it the page faults of a fresh array) of one overlaps the transfer
// of the other. What a block's values become on the way, a conversion on the
// device or a gather on the host, is the caller's. A transfer allocates no
// device memory.
//
// The blocks, 6 MB, are freed with the handle. They are ordinary memory for
// the first kPlain bytes that a handle moves and page-locked after that, since
// page-locking them takes 2.6 to 7.5 ms: a handle that moves little (a few
// tracing checks, a small restart) does without, and one that moves more has
// by then gained about as much over the transfers it replaces. First tracing
// check on a handle, 5,000 / 50,000 / 200,000 particles on 6,080 cells: 0.6 / 3.1 /
// 9.6 ms (page-locked at once 8.3 / 9.2 / 13.4; a copy per column and array
// 1.3 / 4.0 / 14.3), later ones 0.3 / 1.4 / 4.8. With kPlain at 16 MB, checks of
// 50,000 were behind the copies by column until the sixth. Where none can be
// page-locked, ordinary memory does for good (the copies then wait for each
// other).
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cuda_runtime.h>
#include <thread>

namespace dsmc {

struct HostLink {
    static constexpr int kThreads = 6;
    static constexpr int kSlots = 2 * kThreads;
    static constexpr int64_t kItems = 65536;
    static constexpr size_t kBytes = (size_t)kItems * 8;   // of a block: values of at most 8 bytes

    static constexpr int64_t kPlain = 32 << 20;

    int device = 0;                  // set by the owner
    cudaStream_t stream = nullptr;
    char* blocks = nullptr;          // [kSlots][kBytes]
    bool pinned = false;             // whether they are page-locked
    int64_t plainLeft = kPlain;      // bytes still to be moved through ordinary memory
    char* staged = nullptr;          // the same on the device, for values converted there (the caller's)
    cudaEvent_t event[kSlots] = {};

    // A block of column `col`: values [off, off + len), with its memory.
    struct Block {
        int col;
        int64_t off, len;
        char* host;
        char* dev;
    };

    // Makes the blocks ready for a transfer of `bytes`.
    cudaError_t ready(int64_t bytes)
    {
        if (bytes <= plainLeft) {
            plainLeft -= bytes;
        } else if (!pinned && plainLeft >= 0) {
            plainLeft = -1;
            void* q = nullptr;
            if (cudaHostAlloc(&q, kSlots * kBytes, cudaHostAllocDefault) == cudaSuccess) {
                freeBlocks();
                blocks = static_cast<char*>(q);
                pinned = true;
            } else {
                (void)cudaGetLastError();
            }
        }
        if (!blocks && !(blocks = static_cast<char*>(std::malloc(kSlots * kBytes)))) return cudaErrorMemoryAllocation;
        cudaError_t e = cudaSuccess;
        for (cudaEvent_t& ev : event)
            if (e == cudaSuccess && !ev) e = cudaEventCreateWithFlags(&ev, cudaEventDisableTiming);
        if (e != cudaSuccess) (void)cudaGetLastError();   // reported here, not by a later launch
        return e;
    }
    void release()
    {
        freeBlocks();
        for (cudaEvent_t& ev : event)
            if (ev) { cudaEventDestroy(ev); ev = nullptr; }
    }

    // Host to device. fill(block) writes the block's values to block.host;
    // issue(block) enqueues what takes them from there (in stream order, from
    // any thread) and returns the CUDA status. All of it is enqueued on return,
    // and the sources have been read.
    template <class Fill, class Issue>
    cudaError_t in(int ncol, const int64_t* n, Fill fill, Issue issue)
    {
        return run(ncol, n, [&](int slot, const Block* b) {
            cudaError_t e = cudaSuccess;
            if (!b) return e;
            if ((e = cudaEventSynchronize(event[slot])) != cudaSuccess) return e;
            fill(*b);
            if ((e = issue(*b)) != cudaSuccess) return e;
            return cudaEventRecord(event[slot], stream);
        });
    }

    // Device to host. issue(block) enqueues what brings the block's values to
    // block.host; take(block) copies them out once they are there.
    template <class Issue, class Take>
    cudaError_t out(int ncol, const int64_t* n, Issue issue, Take take)
    {
        Block held[kSlots];
        bool has[kSlots] = {};
        return run(ncol, n, [&](int slot, const Block* b) {
            cudaError_t e = cudaSuccess;
            if (has[slot]) {
                if ((e = cudaEventSynchronize(event[slot])) != cudaSuccess) return e;
                take(held[slot]);
                has[slot] = false;
            }
            if (!b) return e;
            if ((e = issue(*b)) != cudaSuccess) return e;
            if ((e = cudaEventRecord(event[slot], stream)) != cudaSuccess) return e;
            held[slot] = *b;
            has[slot] = true;
            return e;
        });
    }

private:
    void freeBlocks()
    {
        for (cudaEvent_t ev : event)
            if (ev) cudaEventSynchronize(ev);   // the copies that read or write them
        if (pinned) cudaFreeHost(blocks);
        else std::free(blocks);
        blocks = nullptr;
        pinned = false;
    }

    // step(slot, block) for every block, a thread's two slots in turn, and at
    // the end step(slot, nullptr) for each of them, the older first.
    template <class Step>
    cudaError_t run(int ncol, const int64_t* n, Step step)
    {
        int64_t total = 0, items = 0;
        for (int c = 0; c < ncol; ++c) {
            total += (n[c] + kItems - 1) / kItems;
            items += n[c];
        }
        if (total == 0) return cudaSuccess;
        if (const cudaError_t e = ready(items * 8)) return e;
        std::atomic<int64_t> next{0};
        std::atomic<int> error{0};
        auto work = [&](int t) {
            cudaError_t e = cudaSetDevice(device);
            int b = 0;
            for (; e == cudaSuccess && error.load(std::memory_order_relaxed) == 0; b ^= 1) {
                int64_t q = next.fetch_add(1);
                if (q >= total) break;
                Block k{};
                for (int64_t m; q >= (m = (n[k.col] + kItems - 1) / kItems); ++k.col) q -= m;
                k.off = q * kItems;
                k.len = std::min(kItems, n[k.col] - k.off);
                const int slot = 2 * t + b;
                k.host = blocks + (size_t)slot * kBytes;
                k.dev = staged + (size_t)slot * kBytes;
                e = step(slot, &k);
            }
            for (int i = 0; i < 2 && e == cudaSuccess; ++i) e = step(2 * t + (b ^ i), nullptr);
            if (e != cudaSuccess) error.store((int)e);
        };
        const int hw = (int)std::thread::hardware_concurrency();
        // a thread for every block of values there are (starting one costs
        // about what a block does)
        const int threads = (int)std::min<int64_t>(items / kItems, std::min(kThreads, hw > 0 ? hw : 1));
        std::thread pool[kThreads];
        for (int t = 1; t < threads; ++t) {
            try {
                pool[t] = std::thread(work, t);
            } catch (...) {   // no thread to be had: the others take its blocks
                break;
            }
        }
        work(0);
        for (std::thread& th : pool)
            if (th.joinable()) th.join();
        return (cudaError_t)error.load();
    }
};

}  // namespace dsmc
