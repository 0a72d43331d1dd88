// slicefft_driver.cpp -- the bit-sliced product transform (slicefft.cuh) on the
// host, for tests/test_slicefft_host.py: its kernels' bodies step by step, each
// step for every thread in turn, on buffers of the sizes that the launches in
// slicefft.cu give them.
//
//   slicefft_driver IN OUT
//
// IN: records of 64-bit words: kind (0 separate launches, 1 one cluster), m,
// planes a Taylor block (log2), nchunks of a and b, xor of a's first chunk,
// output words, then the operands.  OUT: the products' words.
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "slicefft.cuh"

using namespace slice;

namespace {

constexpr int MIN_K = 10, IN_LOG = 7;       // as in slicefft.cu

struct HostEx {
    u32 threads;
    template <class F> void operator()(const F &f) const {
        for (u32 t = 0; t < threads; t++) f(t, threads);
    }
    template <class F> void warps(u32 n, const F &f) const {
        for (u32 w = 0; w < n; w++) f(w);
    }
    void pair() const {}
};
struct HostClusterEx {
    u32 threads;
    std::vector<std::vector<uint4>> *sm;
    uint4 *mem(u32 r) const { return (*sm)[r].data(); }
    template <class F> void block(const F &f) const {
        for (u32 r = 0; r < 8; r++)
            for (u32 t = 0; t < threads; t++) f(r, t, threads);
    }
    template <class F> void cluster(const F &f) const { block(f); }
    template <class F> void warps(const F &f) const {
        for (u32 r = 0; r < 8; r++)
            for (u32 w = 0; w < threads / 32; w++) f(r, w, threads / 32);
    }
};

int clog2(u64 v) {
    int k = 0;
    while (((u64)1 << k) < v) k++;
    return k;
}

template <bool FWD>
void taylor(int k, uint4 *f, u32 s0, int plog, u32 c0, u32 c_src, u32 reps, u32 rep_stride) {
    std::vector<u32> sm((size_t)((1 << (k - 5)) + 4) << plog);
    const HostEx ex{64};
    switch (k) {
#define TAYLOR(K) \
    case K: body_taylor<K, FWD>(ex, sm.data(), f, s0, plog, c0, c_src, reps, rep_stride); break;
    TAYLOR(10) TAYLOR(11) TAYLOR(12) TAYLOR(13) TAYLOR(14) TAYLOR(15) TAYLOR(16)
#undef TAYLOR
    default: abort();
    }
}
template <int RLOG, bool FWD>
void taylor_hi_r(const uint4 *src, uint4 *dst, u32 c_dst) {
    typedef Hi<RLOG> H;
    std::vector<u32> sm(H::WORDS);
    for (u32 c = 0; c < (FWD ? 8u : 16u); c += 1u << H::CL)
        for (u32 ct = 0; ct < (u32)H::TILES; ct++)
            body_taylor_hi<RLOG, FWD>(HostEx{64}, sm.data(), src, c, dst, c_dst + c, ct);
}
template <bool FWD> void taylor_hi(int rlog, const uint4 *src, uint4 *dst, u32 c_dst) {
    switch (rlog) {
    case 1: return taylor_hi_r<1, FWD>(src, dst, c_dst);
    case 2: return taylor_hi_r<2, FWD>(src, dst, c_dst);
    case 3: return taylor_hi_r<3, FWD>(src, dst, c_dst);
    case 4: return taylor_hi_r<4, FWD>(src, dst, c_dst);
    default: abort();
    }
}

// one tile of a butterfly pass by the two blocks of its cluster: both read all
// they need before either writes, so half 1 runs on a copy
template <int NQ, bool FWD>
void bfly_tile(uint4 *f, const Tile &T, int top, bool first, bool lowp) {
    const u32 ns = 1u << (T.rlog + T.clog);
    std::vector<uint4> sm(9 * ns), before(16 * ns), half1(16 * ns);
    const auto at = [&](u32 s) { return f + (u64)tile_gslice(T, s) * 16; };
    for (u32 s = 0; s < ns; s++) memcpy(&before[16 * s], at(s), 256);
    body_bfly<NQ, FWD>(HostEx{64}, sm.data(), f, T, 1, top, first, lowp);
    for (u32 s = 0; s < ns; s++) {
        memcpy(&half1[16 * s], at(s), 256);
        memcpy(at(s), &before[16 * s], 256);
    }
    body_bfly<NQ, FWD>(HostEx{64}, sm.data(), f, T, 0, top, first, lowp);
    for (u32 s = 0; s < ns; s++) memcpy(at(s) + 8, &half1[16 * s + 8], 128);
}
template <bool FWD> void bfly_pass(const Plan &P, int i, uint4 *f, int top, bool first) {
    const bool lowp = i == P.ntop;
    Tile T;
    T.m = P.m;
    T.llo = lowp ? 5 : P.top[i].llo;
    T.rlog = lowp ? P.low - 5 : P.top[i].rlog;
    T.clog = lowp ? 0 : P.top[i].clog;
    const int collog = T.llo - 5 - T.clog;
    for (u32 tile = 0; tile < 1u << (P.m - 5 - T.rlog - T.clog); tile++) {
        const u32 win = tile >> collog, col = tile & ((1u << collog) - 1);
        T.base = (win << (T.llo + T.rlog - 5)) + (col << T.clog);
        if (P.m <= 16) bfly_tile<1, FWD>(f, T, top, first && i == 0, lowp);
        else bfly_tile<2, FWD>(f, T, top, first && i == 0, lowp);
    }
}

void forward(const Plan &P, uint4 *f, const u32 *src, u64 nchunks, u32 xor0, int plog) {
    const int m = P.m, k = std::min(m, std::max(MIN_K, clog2(nchunks))), kt = std::min(k, 16);
    std::vector<u32> sm(33 << IN_LOG);
    const int nlog = std::min(k - 5, IN_LOG);
    for (u32 s0 = 0; s0 < 1u << (k - 5); s0 += 1u << nlog)
        body_slice_in(HostEx{64}, sm.data(), src, nchunks, xor0, f, s0, nlog);
    u32 c_src = 0;
    if (k > 16) {
        taylor_hi<true>(k - 16, f, f, 8);
        c_src = 8;
    }
    for (u32 b = 0; b < 1u << (k - kt); b++)
        for (u32 c = 0; c < 8; c += 1u << (plog - 2))
            taylor<true>(kt, f, b << (kt - 5), plog, c, c_src + c, 1u << (m - k), 1u << (k - 5));
    for (int i = 0; i <= P.ntop; i++) bfly_pass<true>(P, i, f, k, true);
}
void inverse(const Plan &P, uint4 *f, uint4 *tmp, u32 *out, u64 words, int plog) {
    const int m = P.m, kt = std::min(m, 16);
    for (int i = P.ntop; i >= 0; i--) bfly_pass<false>(P, i, f, m, false);
    for (u32 b = 0; b < 1u << (m - kt); b++)
        for (u32 c = 0; c < 16; c += 1u << (plog - 2))
            taylor<false>(kt, f, b << (kt - 5), plog, c, c, 1, 1u << (m - 5));
    if (m > 16) {
        taylor_hi<false>(m - 16, f, tmp, 0);
        f = tmp;
    }
    std::vector<uint4> tile(17 << IN_LOG);
    std::vector<u32> side((1 << IN_LOG) + 1);
    for (u32 s0 = 0; (u64)s0 * 32 < words; s0 += (1 << IN_LOG) - 1)
        body_slice_out(HostEx{64}, tile.data(), side.data(), f, 1u << (m - 5), out, words, s0, IN_LOG);
}

void product(int m, int plog, const u32 *a, u64 ca, u32 xor0, const u32 *b, u64 cb, u32 *out,
             u64 words) {
    const Plan P = make_plan(m, std::min(14, std::max(10, m - 7)), m >= 22 ? TILE_LOG : 0);
    const u32 ns = 1u << (m - 5);
    std::vector<uint4> fa(16 * ns), fb(16 * ns);
    memset(fa.data(), 0xAB, 256 * (size_t)ns);
    memset(fb.data(), 0xCD, 256 * (size_t)ns);
    forward(P, fa.data(), a, ca, xor0, plog);
    forward(P, fb.data(), b, cb, 0, plog);
    std::vector<uint4> ta(32 * 17), tb(32 * 17);
    for (u32 s0 = 0; s0 < ns; s0 += 32) {
        for (u32 i = 0; i < 32 * 16; i++) {
            Full{ta.data()}.chunk(i >> 4, i & 15) = fa[s0 * 16 + i];
            Full{tb.data()}.chunk(i >> 4, i & 15) = fb[s0 * 16 + i];
        }
        HostEx{64}([&](u32 t, u32 n) { mul_slices(Full{ta.data()}, Full{tb.data()}, 32, t, n); });
        for (u32 i = 0; i < 32 * 16; i++) fa[s0 * 16 + i] = Full{ta.data()}.chunk(i >> 4, i & 15);
    }
    inverse(P, fa.data(), fb.data(), out, words, plog);
}
void product_small(int m, const u32 *a, u64 ca, u32 xor0, const u32 *b, u64 cb, u32 *out,
                   u64 words) {
    std::vector<std::vector<uint4>> sm(8, std::vector<uint4>(small_chunks(m)));
    for (auto &v : sm) memset(v.data(), 0xAB, 16 * v.size());
    const auto k = [&](u64 n) { return std::min(m, std::max(MIN_K, clog2(n))); };
    body_small(HostClusterEx{m <= 12 ? 128u : 256u, &sm}, m, Operand{a, ca, xor0, k(ca)},
               Operand{b, cb, 0, k(cb)}, out, words);
}

}  // namespace

int main(int argc, char **argv) {
    FILE *in = argc == 3 ? fopen(argv[1], "rb") : nullptr, *out = argc == 3 ? fopen(argv[2], "wb") : nullptr;
    if (!in || !out) return 1;
    u64 h[7];
    while (fread(h, 8, 7, in) == 7) {
        std::vector<u64> a((h[3] + 1) / 2), b((h[4] + 1) / 2), p(h[6], 0xEEEEEEEEEEEEEEEEull);
        if (fread(a.data(), 8, a.size(), in) != a.size() || fread(b.data(), 8, b.size(), in) != b.size())
            return 1;
        const u32 *pa = reinterpret_cast<const u32 *>(a.data()), *pb = reinterpret_cast<const u32 *>(b.data());
        u32 *po = reinterpret_cast<u32 *>(p.data());
        if (h[0]) product_small((int)h[1], pa, h[3], (u32)h[5], pb, h[4], po, 2 * h[6]);
        else product((int)h[1], (int)h[2], pa, h[3], (u32)h[5], pb, h[4], po, 2 * h[6]);
        fwrite(p.data(), 8, p.size(), out);
    }
    fclose(in);
    return fclose(out) ? 1 : 0;
}
