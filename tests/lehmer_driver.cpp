// lehmer_driver.cpp -- lehmer.cuh's rounds in one block on the host
// (cta_host.h), for tests/test_lehmer_host.py.
#include "lehmer.cuh"

// order[16]: the warps, first come first run.  V: 4 W words (a, b, zeros), R: 8
// mw words with the identity in front, or null.  On return *va, *ra, *parity
// tell where the result is; -1 if the block stopped moving.
extern "C" int lehmer_host(u64 *V, u64 W, u64 *R, u64 mw, long long da, long long db, long long m,
                           const int *order, int *va, int *ra, int *parity, long long *rounds) {
    LehmerEnd end;
    const bool moved = cta::run(BASE_THREADS, std::vector<int>(order, order + BASE_THREADS / 32), [&] {
        const LehmerEnd E = R ? lehmer_cta<true>(V, W, R, mw, da, db, m)
                              : lehmer_cta<false>(V, W, nullptr, 0, da, db, m);
        if (threadIdx.x == 0) end = E;
    });
    if (!moved) return -1;
    *va = end.va;
    *ra = end.ra;
    *parity = end.parity;
    *rounds = end.rounds;
    return end.status;
}
