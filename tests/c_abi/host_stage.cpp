// Transfers through the page-locked ring (z-ant_b200/csrc/host_stage.cuh) without a GPU.  The source of a transfer is made unreadable
// the moment the call returns, failed calls included: a copy thread that still reads it ends the program.  With the argument
// "streams": the ring's streams are left and destroyed between transfers of every kind.
#include "host_stage.cuh"

#include <sys/mman.h>

#include <cstdio>

static int streams() {
    zb::HostStage* st = zb::HostStage::create();
    std::vector<char> src((size_t)3 << 20, 7), dst(src.size());
    const zb::HostStage::Part parts[2] = {{src.data(), 100, 0}, {src.data(), 50, 256}};
    auto transfer = [&](int kind, cudaStream_t s) {
        switch (kind) {
            case 0: return st->to_device(dst.data(), src.data(), 1000, s);
            case 1: return st->to_device(dst.data(), parts, 2, 306, s);
            case 2: return st->to_device(dst.data(), src.data(), src.size(), s);
            default: return st->result_slot(4096, s) ? cudaSuccess : cudaErrorUnknown;
        }
    };
    size_t next = 1;
    for (int before = 0; before < 4; ++before)
        for (int after = 0; after < 4; ++after)
            for (int own = 0; own < 2; ++own) {
                cudaStream_t a = (cudaStream_t)next++, b = (cudaStream_t)next++;
                bool ok = transfer(before, a) == cudaSuccess && zb::leave_stream(st, a, own != 0) == cudaSuccess;
                if (!own) cudaStreamDestroy(a);                    // (its owner, once the context has left it)
                ok = ok && transfer(after, b) == cudaSuccess && transfer(0, b) == cudaSuccess && zb::leave_stream(st, b, true) == cudaSuccess;
                if (!ok || fake_dead_uses) { std::printf("transfer %d, then %d: %d uses of a destroyed stream\n", before, after, fake_dead_uses); return 1; }
            }
    delete st;
    return 0;
}

int main(int argc, char** argv) {
    if (argc > 1 && std::strcmp(argv[1], "streams") == 0) return streams();
    const int rounds = argc > 1 ? std::atoi(argv[1]) : 2000;
    const size_t room = (size_t)24 << 20;
    char* src = (char*)mmap(nullptr, room, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS, -1, 0);
    std::vector<char> dst(room);
    for (size_t i = 0; i < room; ++i) src[i] = (char)(i * 2654435761u >> 13);
    zb::HostStage* st = zb::HostStage::create();
    unsigned seed = 1;
    int failed = 0;
    for (int r = 0; r < rounds; ++r) {
        seed = seed * 1664525u + 1013904223u;
        const bool fails = r % 32 != 0;
        const size_t n = fails ? (size_t)2 << 20 : 1 + seed % room;
        fake_fail_at = fails ? (int)(seed >> 16) % 3 : -1;
        if (mprotect(src, room, PROT_READ) != 0) return 3;
        std::memset(dst.data(), 0, 4096);
        const cudaError_t e = st->to_device(dst.data(), src, n, nullptr);
        if (mprotect(src, room, PROT_NONE) != 0) return 3;
        if ((e != cudaSuccess) != fails) { std::printf("round %d: status %d\n", r, (int)e); return 1; }
        failed += fails;
        if (r % 3 == 0) st->drained();
        if (!fails) {
            mprotect(src, room, PROT_READ);
            if (std::memcmp(dst.data(), src, n) != 0) { std::printf("round %d: %zu bytes differ\n", r, n); return 1; }
        }
    }
    delete st;
    std::printf("%d transfers, %d of them failed on purpose\n", rounds, failed);
    return 0;
}
