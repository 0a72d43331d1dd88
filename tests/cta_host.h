// cta_host.h -- one CUDA block on the host: its threads are fibers, its warps
// run in a chosen order, and each runs as far as it can (to a block barrier)
// before the next one does.  A result that depends on one warp reading a
// shared word before another writes it, with no barrier between, then comes
// out wrong or as a block that no longer moves.  Stands in for
// gf2e_internal.cuh where device code with warp-wide steps and block barriers
// is compiled for the host.
#pragma once

#include <stdint.h>
#include <string.h>
#include <ucontext.h>

#include <algorithm>
#include <functional>
#include <vector>

#include "gf2e.h"

typedef uint64_t u64;
typedef uint32_t u32;
using std::max;
using std::min;
inline long long max(int a, long long b) { return a > b ? a : b; }
inline long long min(int a, long long b) { return a < b ? a : b; }

#define GF2E_DEV inline
#define __shared__ static

namespace cta {

struct Warp {
    int arrived = 0;
    long long gen = 0;
    u64 slot[2][32];
};
struct Fiber {
    ucontext_t ctx;
    std::vector<char> stack;
    int wait = 0;                    // 1: its warp's, 2: the block's step `gen`
    long long gen = 0;
    bool done = false;
};
struct Block {
    std::vector<Fiber> f;
    std::vector<Warp> w;
    int arrived = 0;
    long long gen = 0;
    int now = 0;
    ucontext_t sched;
    std::function<void()> body;
};
inline Block *&cur() { static Block *b = nullptr; return b; }

inline void yield_() {
    Block &b = *cur();
    swapcontext(&b.f[b.now].ctx, &b.sched);
}
inline void block_barrier() {
    Block &b = *cur();
    Fiber &f = b.f[b.now];
    f.wait = 2;
    f.gen = b.gen;
    if (++b.arrived == (int)b.f.size()) {
        b.arrived = 0;
        b.gen++;
    }
    yield_();
}
// every lane's value, after all 32 have come
inline const u64 *warp_values(u64 v) {
    Block &b = *cur();
    Fiber &f = b.f[b.now];
    Warp &w = b.w[b.now / 32];
    const int p = (int)(w.gen & 1);
    w.slot[p][b.now % 32] = v;
    f.wait = 1;
    f.gen = w.gen;
    if (++w.arrived == 32) {
        w.arrived = 0;
        w.gen++;
    } else {
        yield_();
    }
    return w.slot[p];
}
inline void entry() {
    Block &b = *cur();
    b.body();
    b.f[b.now].done = true;
    yield_();
}
// runs `body` on every thread; `order`: the warps, first come first run.
// false if the block stopped moving before every thread was through
inline bool run(int threads, const std::vector<int> &order, const std::function<void()> &body) {
    Block b;
    b.f.resize(threads);
    b.w.resize(threads / 32);
    b.body = body;
    cur() = &b;
    for (Fiber &f : b.f) {
        f.stack.resize(1 << 16);
        getcontext(&f.ctx);
        f.ctx.uc_stack.ss_sp = f.stack.data();
        f.ctx.uc_stack.ss_size = f.stack.size();
        f.ctx.uc_link = nullptr;
        makecontext(&f.ctx, entry, 0);
    }
    const auto can_run = [&](const Fiber &f, const Warp &w) {
        return !f.done && (f.wait == 0 || (f.wait == 1 && w.gen > f.gen) ||
                           (f.wait == 2 && b.gen > f.gen));
    };
    for (bool moved = true; moved;) {
        moved = false;
        for (int wi : order) {
            const long long gen = b.gen;
            for (bool again = true; again;) {
                again = false;
                for (int l = 32 * wi; l < 32 * wi + 32; l++)
                    if (can_run(b.f[l], b.w[wi])) {
                        b.f[l].wait = 0;
                        b.now = l;
                        swapcontext(&b.sched, &b.f[l].ctx);
                        again = moved = true;
                    }
                if (b.gen != gen) break;           // a barrier opened: from the first warp again
            }
            if (b.gen != gen) break;
        }
    }
    cur() = nullptr;
    for (const Fiber &f : b.f)
        if (!f.done) return false;
    return true;
}

struct ThreadIdx {
    struct X {
        operator int() const { return cur()->now; }
    } x;
};

}  // namespace cta

static const cta::ThreadIdx threadIdx;

inline void __syncthreads() { cta::block_barrier(); }
inline void __syncwarp() { cta::warp_values(0); }
inline int lane_() { return cta::cur()->now % 32; }
template <class T> T __shfl_sync(unsigned, T v, int lane) {
    return (T)cta::warp_values((u64)v)[lane & 31];
}
template <class T> T __shfl_xor_sync(unsigned, T v, int mask) {
    return (T)cta::warp_values((u64)v)[lane_() ^ mask];
}
template <class T> T __shfl_up_sync(unsigned, T v, int d) {
    const u64 *s = cta::warp_values((u64)v);
    return lane_() >= d ? (T)s[lane_() - d] : v;
}
template <class T> T __shfl_down_sync(unsigned, T v, int d) {
    const u64 *s = cta::warp_values((u64)v);
    return lane_() + d < 32 ? (T)s[lane_() + d] : v;
}
inline unsigned __ballot_sync(unsigned, bool p) {
    const u64 *s = cta::warp_values(p);
    unsigned r = 0;
    for (int i = 0; i < 32; i++) r |= (unsigned)(s[i] != 0) << i;
    return r;
}
inline int __ffs(unsigned v) { return __builtin_ffs((int)v); }
inline int __clz(unsigned v) { return v ? __builtin_clz(v) : 32; }
inline int __clzll(u64 v) { return v ? __builtin_clzll(v) : 64; }
inline u32 __funnelshift_r(u32 lo, u32 hi, unsigned sh) {
    return (u32)(((u64)hi << 32 | lo) >> (sh & 31));
}
inline long long clock64() { return 0; }

inline u64 funnel64(u64 lo, u64 hi, unsigned sh) {
    return sh ? ((lo >> sh) | (hi << (64 - sh))) : lo;
}
inline u64 clmul32(u32 a, u32 b) {
    u64 r = 0;
    for (int i = 0; i < 32; i++)
        if (b >> i & 1) r ^= (u64)a << i;
    return r;
}
