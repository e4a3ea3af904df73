// CPU check of dig-appolo_b200/csrc/dsmc_hostlink.h on a host stand-in for the
// CUDA runtime: what goes through the blocks comes out the same, at the ends
// of a block, through ordinary and page-locked memory and where none can be
// page-locked; a handle that moves little page-locks nothing, and all memory
// and events are given back. Prints "ok" and exits 0, or names what failed.
#include "dsmc_hostlink.h"

#include <cstdio>
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

}  // namespace

int main()
{
    for (bool fail : {false, true}) {
        fake::failHostAlloc = fail;
        fake::hostAllocs = fake::hostFrees = 0;
        {
            HostLink L;
            check(L.in(0, nullptr, [](const HostLink::Block&) {}, [](const HostLink::Block&) { return cudaSuccess; }) ==
                          cudaSuccess && !L.blocks, "no columns, no memory", 0);
            int64_t moved = 0;
            int salt = 0;
            const int64_t sizes[] = {1, 2, HostLink::kItems - 1, HostLink::kItems, HostLink::kItems + 1, 5 * HostLink::kItems + 3};
            for (int round = 0; round < 4; ++round)
                for (int64_t n : sizes) {
                    const int64_t one = (n + n / 2 + n + 1) * 8;
                    check(round_trip(L, n, ++salt), "values", n);
                    moved += 2 * one;
                    if (moved <= HostLink::kPlain) check(fake::hostAllocs == 0, "page-locked early", moved);
                }
            check(moved > HostLink::kPlain, "the sizes go past the ordinary blocks", moved);
            check(fake::hostAllocs == (fail ? 0 : 1) && L.pinned == !fail, "page-locked once", fake::hostAllocs);
            check(fake::lastError == cudaSuccess, "no error left behind", fake::lastError);
            // an error of a copy ends the transfer and leaves the link usable
            const int64_t n = 3 * HostLink::kItems;
            check(L.in(1, &n, [](const HostLink::Block&) {}, [](const HostLink::Block&) { return cudaErrorInvalidValue; }) ==
                      cudaErrorInvalidValue, "the copy's error", n);
            check(round_trip(L, 1000, 99), "values after an error", 1000);
            L.release();
        }
        check(fake::hostFrees == fake::hostAllocs && fake::events == 0, "given back", fake::hostFrees);
    }
    if (failures) return 1;
    std::printf("ok\n");
    return 0;
}
