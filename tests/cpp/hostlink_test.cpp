// CPU check of dig-appolo_b200/csrc/dsmc_hostlink.h on a host stand-in for the
// CUDA runtime: what goes through the blocks comes out the same, at the ends
// of a block, through ordinary and page-locked memory and where none can be
// page-locked; a handle that moves little page-locks nothing, and all memory
// and events are given back. Prints "ok" and exits 0, or names what failed.
#include "dsmc_hostlink.h"

#include <cstdio>
#include <fstream>
#include <string>
#include <vector>

using dsmc::HostLink;

namespace {

int failures = 0;

void check(bool ok, const char* what, long long n)
{
    if (!ok && failures++ < 10) std::printf("failed: %s (%lld)\n", what, n);
}

// three columns of unlike length through the link to a "device" and back
bool round_trip(HostLink& L, int64_t n, int salt)
{
    const int64_t len[3] = {n, n / 2, n + 1};
    std::vector<std::vector<double>> src(3), dev(3), back(3);
    for (int c = 0; c < 3; ++c) {
        src[c].resize((size_t)len[c]);
        for (int64_t i = 0; i < len[c]; ++i) src[c][(size_t)i] = (double)(i * 3 + c) + 0.25 * salt;
        dev[c].assign((size_t)len[c], -1.0);
        back[c].assign((size_t)len[c], -2.0);
    }
    const cudaError_t in = L.in(
        3, len, [&](const HostLink::Block& b) { std::memcpy(b.host, src[b.col].data() + b.off, (size_t)b.len * 8); },
        [&](const HostLink::Block& b) {
            std::memcpy(dev[b.col].data() + b.off, b.host, (size_t)b.len * 8);
            return cudaSuccess;
        });
    const cudaError_t out = L.out(
        3, len,
        [&](const HostLink::Block& b) {
            std::memcpy(b.host, dev[b.col].data() + b.off, (size_t)b.len * 8);
            return cudaSuccess;
        },
        [&](const HostLink::Block& b) { std::memcpy(back[b.col].data() + b.off, b.host, (size_t)b.len * 8); });
    return in == cudaSuccess && out == cudaSuccess && dev == src && back == src;
}

// whether the mapping at p is left out of a fork
bool not_forked(const void* p)
{
    std::ifstream maps("/proc/self/smaps");
    std::string line;
    bool in = false;
    while (std::getline(maps, line)) {
        unsigned long a = 0, b = 0;
        if (std::sscanf(line.c_str(), "%lx-%lx ", &a, &b) == 2) in = (unsigned long)p >= a && (unsigned long)p < b;
        if (in && line.compare(0, 8, "VmFlags:") == 0) return line.find(" dc") != std::string::npos;
    }
    return false;
}

}  // namespace

int main()
{
    constexpr int64_t K = HostLink::kItems;
    for (bool fail : {false, true}) {
        fake::failRegister = fail;
        fake::registeredBytes = 0;
        HostLink L;
        check(L.in(0, nullptr, [](const HostLink::Block&) {}, [](const HostLink::Block&) { return cudaSuccess; }) ==
                      cudaSuccess && !L.blocks, "no columns, no memory", 0);
        // kPlain small transfers without page-locking, then what a thread needs
        int salt = 0;
        for (int k = 0; k < HostLink::kPlain / 2; ++k) check(round_trip(L, 1 + 7 * k, ++salt), "values", k);
        check(fake::registeredBytes == 0 && fake::lastError == cudaSuccess, "page-locked early", 0);
        check(round_trip(L, 5, ++salt), "values", 5);
        check(fake::registeredBytes == (fail ? 0 : HostLink::kHuge), "one huge page", (long long)fake::registeredBytes);
        for (int round = 0; round < 2; ++round)
            for (int64_t n : {int64_t(1), K / 3, K - 1, K, K + 1, 2 * K + 5, 5 * K + 3, int64_t(100)})
                check(round_trip(L, n, ++salt), "values", n);
        check(not_forked(L.blocks) && not_forked(L.blocks + HostLink::kSlots * HostLink::kBytes - 1), "left out of a fork", 0);
        check(fake::registeredBytes <= HostLink::kSlots * HostLink::kBytes, "each block once", (long long)fake::registeredBytes);
        check(fake::lastError == cudaSuccess, "no error left behind", fake::lastError);
        // an error of a copy ends the transfer and leaves the link usable
        const int64_t n = 3 * K;
        check(L.in(1, &n, [](const HostLink::Block&) {}, [](const HostLink::Block&) { return cudaErrorInvalidValue; }) ==
                  cudaErrorInvalidValue, "the copy's error", n);
        check(round_trip(L, 1000, ++salt), "values after an error", 1000);
        L.release();
        check(fake::registered == 0 && fake::events == 0 && !L.blocks, "given back", fake::registered);
        // a large first transfer page-locks at once, what it needs
        fake::registeredBytes = 0;
        check(round_trip(L, 6 * K, ++salt), "values", 6 * K);
        check(fail || (fake::registeredBytes >= HostLink::kHuge &&
                       fake::registeredBytes <= HostLink::kSlots * HostLink::kBytes), "page-locked", (long long)fake::registeredBytes);
        L.release();
        check(fake::registered == 0 && fake::events == 0, "given back", fake::registered);
    }
    if (failures) return 1;
    std::printf("ok\n");
    return 0;
}
