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
// The blocks, 1 MB a thread, are page-locked two threads' at a time when a
// transfer first gives those threads work, and given back with the handle. They
// lie in huge pages where the system gives any, one for two threads:
// page-locking one takes 0.4 to 0.7 ms, all three 0.6 to 1.4; in small pages 1 to 2.6
// and 2 to 7, and cudaHostAlloc of all 6 MB as much. A handle's first kPlain
// transfers of no more than one block's values, the one or two tracing checks of
// a few particles that a program may make, go through ordinary memory instead.
// First tracing check on a handle, 1 / 5,000 / 50,000 / 200,000 particles on 6,080
// cells: 0.4 / 0.7 / 3.4 / 7.8 ms, where all blocks allocated at once took 8.1 / 7.8 /
// 10 / 14, and a copy per column and array 0.5 / 1.3 / 3.9 / 14; later ones 0.2 / 0.4 /
// 1.5 / 4.6. Blocks that cannot be page-locked stay ordinary memory (their copies
// then wait).
#pragma once

#include <algorithm>
#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cuda_runtime.h>
#include <sys/mman.h>
#include <thread>

namespace dsmc {

struct HostLink {
    static constexpr int kThreads = 6;
    static constexpr int kSlots = 2 * kThreads;
    static constexpr int64_t kItems = 65536;
    static constexpr size_t kBytes = (size_t)kItems * 8;   // of a block: values of at most 8 bytes
    static constexpr size_t kHuge = 2 << 20;               // a huge page: the blocks of kUnit threads
    static constexpr int kUnit = (int)(kHuge / (2 * kBytes));
    static constexpr int kPlain = 6;
    static_assert(kUnit >= 1 && kThreads % kUnit == 0, "whole huge pages");

    int device = 0;                  // set by the owner
    cudaStream_t stream = nullptr;
    void* mapped = nullptr;          // kSlots * kBytes + kHuge
    char* blocks = nullptr;          // [kSlots][kBytes] in there, from a huge page's start
    int ready = 0;                   // threads whose blocks have been page-locked (or could not be)
    bool pinned[kThreads] = {};      // page-locked in one call from this thread's blocks on
    int plain = 0;                   // small transfers so far
    char* small = nullptr;           // [2][kBytes], theirs
    char* staged = nullptr;          // the same on the device, for values converted there (the caller's)
    cudaEvent_t event[kSlots] = {};

    // A block of column `col`: values [off, off + len), with its memory.
    struct Block {
        int col;
        int64_t off, len;
        char* host;
        char* dev;
    };

    void release()
    {
        if (blocks || small) cudaStreamSynchronize(stream);   // copies that a failed transfer left
        for (int t = 0; t < kThreads; ++t)
            if (pinned[t]) { cudaHostUnregister(blocks + 2 * t * kBytes); pinned[t] = false; }
        if (mapped) munmap(mapped, kSlots * kBytes + kHuge);
        std::free(small);
        mapped = nullptr;
        blocks = small = nullptr;
        ready = 0;
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
    // Blocks (at *at) and events for a transfer of `items` values by `threads` threads.
    cudaError_t prepare(int64_t items, int threads, char** at)
    {
        for (int s = 0; s < 2 * threads; ++s)
            if (!event[s]) {
                const cudaError_t e = cudaEventCreateWithFlags(&event[s], cudaEventDisableTiming);
                if (e != cudaSuccess) {
                    (void)cudaGetLastError();   // reported here, not by a later launch
                    return e;
                }
            }
        if (ready == 0 && items <= kItems && plain < kPlain) {
            ++plain;
            if (!small) small = static_cast<char*>(std::malloc(2 * kBytes));
            *at = small;
            return small ? cudaSuccess : cudaErrorMemoryAllocation;
        }
        if (!blocks) {
            void* q = mmap(nullptr, kSlots * kBytes + kHuge, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
            if (q == MAP_FAILED) return cudaErrorMemoryAllocation;
            mapped = q;
            blocks = static_cast<char*>(q) + (kHuge - (uintptr_t)q % kHuge) % kHuge;
            (void)madvise(blocks, kSlots * kBytes, MADV_HUGEPAGE);
            // a fork must not make the pages copy-on-write: this process's next
            // write would move them away from where the device was told they are
            (void)madvise(blocks, kSlots * kBytes, MADV_DONTFORK);
        }
        if (threads > ready) {
            const int upTo = std::min(kThreads, (threads + kUnit - 1) / kUnit * kUnit);
            pinned[ready] = cudaHostRegister(blocks + 2 * ready * kBytes, 2 * (upTo - ready) * kBytes,
                                             cudaHostRegisterDefault) == cudaSuccess;
            if (!pinned[ready]) (void)cudaGetLastError();
            ready = upTo;
        }
        *at = blocks;
        return cudaSuccess;
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
        const int hw = (int)std::thread::hardware_concurrency();
        // a thread for every block of values there are (starting one costs
        // about what a block does)
        const int threads = (int)std::max<int64_t>(1, std::min<int64_t>(items / kItems, std::min(kThreads, hw > 0 ? hw : 1)));
        char* at = nullptr;
        if (const cudaError_t e = prepare(items, threads, &at)) return e;
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
                k.host = at + (size_t)slot * kBytes;
                k.dev = staged + (size_t)slot * kBytes;
                e = step(slot, &k);
            }
            for (int i = 0; i < 2 && e == cudaSuccess; ++i) e = step(2 * t + (b ^ i), nullptr);
            if (e != cudaSuccess) error.store((int)e);
        };
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
