// frobenius.cu -- two squarings per pass over HBM: F -> F^4 mod T,
// T = x^r + x^s + 1 (r odd, 1 <= s, 2s < r), batched over many s.
//
// One squaring F -> F^2 mod T is linear over GF(2), and the derivation in
// trinomial.cu writes it as five windows: output bit j, for j in [lo, hi)
// and j = c (mod 2), is the XOR of input bits (j - c)/2 + K over the windows
// covering j (h = (r+1)/2):
//     spread(A_lo)            c = 0,           [0, r),       K = 0
//     S << 1                  c = 1,           [1, r-1),     K = h
//     S << (s+1) mod x^r      c = (s+1) & 1,   [s+1, r),     K = h - (s+1-c)/2
//     S >> (r-s-1)            c = s & 1,       [0, s-1),     K = h + (r-s-1+c)/2
//     (S >> (r-s-1)) << s     c = 0,           [s, 2s-1),    K = h + (r-2s-1)/2
// Composing two window maps gives windows of the same form with modulus
// M = 4: an outer window (2, ca, [loa, hia), Ka) applied to the output of an
// inner one (mB, cb, [lob, hib), Kb) reads the intermediate bit
// p = (j - ca)/2 + Ka, which lies in the inner window when
// j in [ca + 2 (lob - Ka), ca + 2 (hib - Ka)) and p = cb (mod mB), i.e.
//     j = c := ca + 2 ((cb - Ka) mod mB)   (mod 2 mB),
// and then reads input bit (p - cb)/mB + Kb = (j - c)/(2 mB) + K with
//     K = ((c - ca)/2 + Ka - cb)/mB + Kb.
// So F^4 mod T has at most 25 windows (out bit j = c mod 4 in [lo, hi) takes
// input bit (j - c)/4 + K); at r = 136279841 9 to 13 of them overlap a
// given output tile.  The squaring result is the same bits as two passes of
// the one-squaring kernel (the reference's k_square_fused twice,
// tsfactor.cu:128-186), read and written once instead of twice.
//
// Work unit: a lane's unit is two output words (128 bits).  Its bits of
// class c are j = 128 u + c + 4 t, t = 0..31, whose sources are the 32
// consecutive input bits 32 u + K + t: one funnel-shifted 32-bit read per
// window, XORed into the class accumulator C[c].  The unit's output is the
// 4-way bit interleave of C[0..3] (bit 4 t + c = bit t of C[c]): cross-
// register and in-register delta swaps, then a byte transpose by byte
// permutes.  Lanes own units u0 + lane + 32 q, q < 4, so
// loads and 16-byte stores are coalesced.
//
// Per warp tile of 128 units, one ballot lists the windows overlapping it and
// one those that cover all of it and read inside the state; the latter are
// applied class by class, two at a time (both windows' 16 loads issued before
// either is used) with no masks or bounds tests; the rest (windows that start
// or end inside the tile, a few tiles per state) with per-lane bit masks and
// bounds-tested loads.  The kernel is bound by memory latency: 7 of 17 cycles
// between a warp's instructions wait for loads, the integer pipe is 48 % busy
// and 53 % of the issue slots are used (8 states).  A pass of 64
// states at r = 136279841: windows one at a time with the high words by
// shuffle 1.06 ms, the per-tile list with two loads a unit 0.72 ms, two
// windows at a time 0.65 ms, fast windows listed by class 0.58 ms (1 state 29
// us, 256 states at 999961 46 us; the windows that end inside a tile without
// branches, their loads together, 15 and 27); staging
// each window's run in shared memory by cp.async first ran 1.5 ms (more issued
// instructions, fewer resident warps).  Each CTA composes its state's
// windows in warp 0 with shifts and masks (the moduli are powers of two).
#include "gf2e_internal.cuh"

#include <algorithm>
#include <atomic>
#include <cstdlib>
#include <cstring>

namespace {

constexpr int KL = 2;                 // squarings per pass
constexpr int M = 1 << KL;            // residue classes of output bits
constexpr int NCAND = 25;             // 5^KL composed candidates
constexpr u32 UBITS = 32 * M;         // output bits per unit (two words)

struct FWin {
    int lo, hi;       // output bits j in [lo, hi), lo = hi - 1 = c (mod M)
    int K;            // input bit (j - c) / M + K
    int c;
};

struct Win64 {
    int64_t m, c, lo, hi, K;
};

// a mod m in [0, m) for m a power of two (two's complement: the low bits)
GF2E_DEV int64_t mod_pos(int64_t a, int64_t m) { return a & (m - 1); }
GF2E_DEV int log2i(int64_t m) { return 63 - __clzll((unsigned long long)m); }

// window i (0..4) of one squaring; lo >= hi when empty
GF2E_DEV Win64 square_win(int i, int64_t r, int64_t s) {
    const int64_t h = (r + 1) >> 1;
    Win64 w{2, 0, 0, 0, 0};
    switch (i) {
        case 0: w.c = 0; w.lo = 0; w.hi = r; w.K = 0; break;
        case 1: w.c = 1; w.lo = 1; w.hi = r - 1; w.K = h; break;
        case 2: w.c = (s + 1) & 1; w.lo = s + 1; w.hi = r; w.K = h - ((s + 1 - w.c) >> 1); break;
        case 3: w.c = s & 1; w.lo = 0; w.hi = s - 1; w.K = h + ((r - s - 1 + w.c) >> 1); break;
        default: w.c = 0; w.lo = s; w.hi = 2 * s - 1; w.K = h + ((r - 2 * s - 1) >> 1); break;
    }
    return w;
}

// trim [lo, hi) to its first and last member of class c (mod m); the moduli
// are powers of two, so the divisions below are exact shifts
GF2E_DEV void trim(Win64 &w) {
    if (w.lo >= w.hi) return;
    w.lo += mod_pos(w.c - w.lo, w.m);
    if (w.lo < w.hi) w.hi = w.lo + ((w.hi - 1 - w.lo) & ~(w.m - 1)) + 1;
}

// outer window a (modulus 2) applied after inner window b
GF2E_DEV Win64 compose(const Win64 &a, const Win64 &b) {
    Win64 w;
    const int la = log2i(a.m), lb = log2i(b.m);
    w.m = a.m * b.m;
    w.c = a.c + a.m * mod_pos(b.c - a.K, b.m);
    const int64_t t = ((w.c - a.c) >> la) + a.K - b.c;    // a multiple of b.m
    w.K = (t >> lb) + b.K;                                 // exact: arithmetic shift
    w.lo = max(a.lo, a.c + a.m * (b.lo - a.K));
    w.hi = min(a.hi, a.c + a.m * (b.hi - a.K));
    trim(w);
    return w;
}

// candidate i = (outer digit i / 5, inner digit i % 5) for KL = 2
GF2E_DEV Win64 candidate(int i, int64_t r, int64_t s) {
    Win64 in = square_win(i % 5, r, s);
    if (in.lo >= in.hi) return in;
    trim(in);
    if (in.lo >= in.hi) return in;
    Win64 out = square_win(i / 5, r, s);
    if (out.lo >= out.hi) return out;
    return compose(out, in);
}

// 4-way bit interleave of one unit: bit 4 t + c of the 128-bit output is
// bit t of C[c].  Index bookkeeping (register index r1 r0, then bit position
// p4..p0): the input holds bit t of class c = (c1 c0) at register (c1 c0),
// position (t4 t3 t2 t1 t0).  Relabelling the registers (free) swaps r1 and
// r0; a cross-register delta swap exchanges r0 with p1, another r1 with p2,
// and one delta swap inside each register exchanges p0 with p2, which gives
// register (t2 t1), position (t4 t3 t0 c1 c0); a 4x4 byte transpose (8 byte
// permutes) then exchanges the register index with the byte index (p4 p3):
// register (t4 t3), position (t2 t1 t0 c1 c0), so register b holds output
// bits [32 b, 32 b + 32).  44 operations for 128 output bits.
GF2E_DEV void xswap(u32 &x, u32 &y, int sh, u32 m) {    // x[p + sh] <-> y[p], p in m
    const u32 t = ((x >> sh) ^ y) & m;
    y ^= t;
    x ^= t << sh;
}
GF2E_DEV u32 dswap(u32 x, int d, u32 m) {                // x[p] <-> x[p + d], p in m
    const u32 t = (x ^ (x >> d)) & m;
    return x ^ (t * (1u + (1u << d)));       // t and t << d are disjoint
}
GF2E_DEV ulonglong2 interleave4(u32 c0, u32 c1, u32 c2, u32 c3) {
    u32 r0 = c0, r1 = c2, r2 = c1, r3 = c3;              // r1 <-> r0 of the index
    xswap(r0, r1, 2, 0x33333333u);                       // r0 <-> p1
    xswap(r2, r3, 2, 0x33333333u);
    xswap(r0, r2, 4, 0x0F0F0F0Fu);                       // r1 <-> p2
    xswap(r1, r3, 4, 0x0F0F0F0Fu);
    r0 = dswap(r0, 3, 0x0A0A0A0Au);                      // p0 <-> p2
    r1 = dswap(r1, 3, 0x0A0A0A0Au);
    r2 = dswap(r2, 3, 0x0A0A0A0Au);
    r3 = dswap(r3, 3, 0x0A0A0A0Au);
    const u32 lo01 = __byte_perm(r0, r1, 0x5140), hi01 = __byte_perm(r0, r1, 0x7362);
    const u32 lo23 = __byte_perm(r2, r3, 0x5140), hi23 = __byte_perm(r2, r3, 0x7362);
    ulonglong2 v;
    v.x = ((u64)__byte_perm(lo01, lo23, 0x7632) << 32) | __byte_perm(lo01, lo23, 0x5410);
    v.y = ((u64)__byte_perm(hi01, hi23, 0x7632) << 32) | __byte_perm(hi01, hi23, 0x5410);
    return v;
}

// ---- the pass: per warp tile, the overlapping windows, two at a time
// units per lane per warp tile (256 words a tile) and resident CTAs per SM.
// A pass in us, units x CTAs an SM (64 states at r = 136279841, 64 at
// 10001567, 256 at 999961): 6 x 4 579 / 82 / 43, 4 x 5 582 / 63 / 36, 5 x 5
// 572 / 67 / 56, 3 x 6 594 / 63 / 34, 8 x 3 603 / 72 / 60
constexpr int LANE_UNITS = 4;
constexpr int MIN_CTAS = 5;

// A word of a state: by a read-only load, or by a plain one in a chained pass
// (read-only loads are for data that nobody writes while a CTA lives).
template <bool RO>
GF2E_DEV u32 state_word(const u32 *p) {
    return RO ? __ldg(p) : *p;
}

// A full window over all of the tile's units, every index inside the state:
// lane l's units u0 + l + 32 q read input words first + l + 32 q and the
// word after it (the high word of the funnel shift) with two plain loads.
template <int UL, bool RO>
GF2E_DEV void full_window(const u32 *in32, u32 first, u32 lane, u32 sh,
                          u32 (&acc)[UL]) {
    const u32 *p = in32 + (first + lane);
    u32 lo[UL], hi[UL];
#pragma unroll
    for (int q = 0; q < UL; q++) {
        lo[q] = state_word<RO>(p + 32 * q);
        hi[q] = state_word<RO>(p + 32 * q + 1);
    }
#pragma unroll
    for (int q = 0; q < UL; q++) acc[q] ^= __funnelshift_r(lo[q], hi[q], sh);
}

// Two full windows of one class, every load of both issued before use, so
// their memory latencies overlap.
template <int UL, bool RO>
GF2E_DEV void full_windows2(const u32 *in32, u32 first1, u32 sh1, u32 first2, u32 sh2,
                         u32 lane, u32 (&acc)[UL]) {
    const u32 *p1 = in32 + (first1 + lane);
    const u32 *p2 = in32 + (first2 + lane);
    u32 l1[UL], h1[UL], l2[UL], h2[UL];
#pragma unroll
    for (int q = 0; q < UL; q++) {
        l1[q] = state_word<RO>(p1 + 32 * q);
        h1[q] = state_word<RO>(p1 + 32 * q + 1);
        l2[q] = state_word<RO>(p2 + 32 * q);
        h2[q] = state_word<RO>(p2 + 32 * q + 1);
    }
#pragma unroll
    for (int q = 0; q < UL; q++)
        acc[q] ^= __funnelshift_r(l1[q], h1[q], sh1) ^ __funnelshift_r(l2[q], h2[q], sh2);
}

// Any other overlapping window: per unit the bits t whose output position
// 128 u + c + 4 t lies in [lo, hi), loads bounds-tested.  Positions are below
// 2^31 (r < 2^31 - 2^16 and a tile ends less than 2^15 bits past r), and
// lo, hi - 1 and j0 are all c mod 4, so the shifts are exact.  No branches:
// the loads of all units are issued together.
template <int UL, bool RO>
GF2E_DEV void part_window(const u32 *in32, u32 n32, u32 u0, u32 lane, const FWin &w,
                        u32 (&acc)[UL]) {
    u32 lo[UL], hi[UL];
#pragma unroll
    for (int q = 0; q < UL; q++) {
        const u32 i = u0 + lane + 32 * q + (u32)(w.K >> 5);     // negative: above any n32
        lo[q] = i < n32 ? state_word<RO>(in32 + i) : 0u;
        hi[q] = i + 1 < n32 ? state_word<RO>(in32 + i + 1) : 0u;
    }
#pragma unroll
    for (int q = 0; q < UL; q++) {
        const int j0 = (int)((u0 + lane + 32 * q) * UBITS) + w.c;
        const int tlo = max((w.lo - j0) >> KL, 0);
        const int thi = min(((w.hi - 1 - j0) >> KL) + 1, 32);
        const u32 mask = tlo < thi ? (0xffffffffu >> (32 - (thi - tlo))) << tlo : 0u;
        acc[q] ^= __funnelshift_r(lo[q], hi[q], (u32)w.K & 31u) & mask;
    }
}

// Warp-wide: compose the windows of F -> F^4 mod x^r + x^s + 1 into tab[]
// in class order; returns their number (lane 0's count, on every lane).
GF2E_DEV int compose_windows(u64 r, u64 s, FWin *tab, u32 lane) {
    Win64 w{};
    bool ok = false;
    if (lane < (u32)NCAND) {
        w = candidate((int)lane, (int64_t)r, (int64_t)s);
        ok = w.lo < w.hi;
    }
    int base = 0;
    for (int c = 0; c < M; c++) {
        const u32 b = __ballot_sync(0xffffffffu, ok && w.c == c);
        if (ok && w.c == c) {
            const int pos = base + __popc(b & ((1u << lane) - 1u));
            tab[pos] = FWin{(int)w.lo, (int)w.hi, (int)w.K, c};
        }
        base += __popc(b);
    }
    __syncwarp();
    return base;
}

// the fast windows of one class (bits of m), two at a time
template <int UL, bool RO>
GF2E_DEV void class_windows(const u32 *in32, const int *tabK, u32 m, int u0, u32 lane,
                            u32 (&acc)[UL]) {
    while (m) {
        const int K1 = tabK[__ffs(m) - 1];
        m &= m - 1;
        const u32 f1 = (u32)(u0 + (K1 >> 5));
        if (m) {
            const int K2 = tabK[__ffs(m) - 1];
            m &= m - 1;
            full_windows2<UL, RO>(in32, f1, (u32)K1, (u32)(u0 + (K2 >> 5)), (u32)K2, lane, acc);
        } else {
            full_window<UL, RO>(in32, f1, lane, (u32)K1, acc);
        }
    }
}

// One warp tile: the 32 UL units from u0 of one state.  Lane k holds window
// k of the state (`mine`, k < nwin), cls[c] the windows of class c.  One
// ballot lists the windows overlapping the tile and another the fast ones:
// those that cover all of it and read inside the state (the highest index is
// u0 + floor(K/32) + 32 UL, one past the last lane's last word), which are
// applied class by class with no masks, bounds tests or branches on the
// class (a loop over all windows with a test and a switch each took 180
// instructions a unit, 94 of them in the integer pipe).
template <int UL, bool RO>
GF2E_DEV void frob4_tile(const u32 *in32, ulonglong2 *o, u32 n32,
                         u32 nu, const FWin *tab, const int *tabK, int nwin, const FWin &mine,
                         const u32 (&cls)[M], u32 u0, u32 lane) {
    constexpr u32 TWL = 32 * UL;
    const int B0 = (int)(u0 * UBITS), B1 = B0 + (int)(TWL * UBITS);
    const bool over = lane < (u32)nwin && mine.hi > B0 && mine.lo < B1;
    const u32 act = __ballot_sync(0xffffffffu, over);
    const u32 fast = __ballot_sync(0xffffffffu,
                                   over && mine.lo <= B0 && mine.hi >= B1 &&
                                       (int)u0 + (mine.K >> 5) + (int)TWL + 1 < (int)n32);
    u32 C[M][UL];
#pragma unroll
    for (int c = 0; c < M; c++) {
#pragma unroll
        for (int q = 0; q < UL; q++) C[c][q] = 0;
        class_windows<UL, RO>(in32, tabK, fast & cls[c], (int)u0, lane, C[c]);
    }
    for (u32 m = act & ~fast; m; m &= m - 1) {     // windows that start or end in the tile
        const FWin w = tab[__ffs(m) - 1];
        switch (w.c) {
            case 0: part_window<UL, RO>(in32, n32, u0, lane, w, C[0]); break;
            case 1: part_window<UL, RO>(in32, n32, u0, lane, w, C[1]); break;
            case 2: part_window<UL, RO>(in32, n32, u0, lane, w, C[2]); break;
            default: part_window<UL, RO>(in32, n32, u0, lane, w, C[3]); break;
        }
    }
#pragma unroll
    for (int q = 0; q < UL; q++) {
        const u32 u = u0 + lane + 32 * q;
        if (u < nu) o[u] = interleave4(C[0][q], C[1][q], C[2][q], C[3][q]);
    }
}

// Batched F -> F^4 mod T (r < 2^31 - 2^16, even stride): blockIdx.y = state;
// warp 0 composes the state's windows for the CTA, the warps stride over
// its tiles.
// RO: every word read was written before this kernel's first CTA started (not a
// chained pass)
template <bool RO>
__global__ void __launch_bounds__(256, MIN_CTAS)
k_frob4_batch(const u64 *in, u64 *out, size_t stride, u64 r,
              const u64 *__restrict__ s_arr, u64 s_uniform) {
    __shared__ FWin tab[NCAND];
    __shared__ int tabK[NCAND];
    __shared__ int s_nwin;
    const int st = blockIdx.y;
    const u32 lane = threadIdx.x & 31;
    cudaTriggerProgrammaticLaunchCompletion();
    if (threadIdx.x < 32) {
        const int n = compose_windows(r, s_arr ? s_arr[st] : s_uniform, tab, lane);
        if (lane == 0) s_nwin = n;
        if (lane < (u32)n) tabK[lane] = tab[lane].K;
    }
    __syncthreads();
    // everything above reads only r and s; from here on the states, which the
    // previous pass of the same call may still have been writing
    if (!RO) cudaGridDependencySynchronize();
    const int nwin = s_nwin;
    const u32 nw = (u32)((r + 63) >> 6);
    const u32 n32 = 2 * nw, nu = (nw + 1) >> 1;
    const u32 *in32 = reinterpret_cast<const u32 *>(in + (size_t)st * stride);
    ulonglong2 *o = reinterpret_cast<ulonglong2 *>(out + (size_t)st * stride);
    const FWin mine = lane < (u32)nwin ? tab[lane] : FWin{0, 0, 0, 0};
    u32 cls[M];
#pragma unroll
    for (int c = 0; c < M; c++)
        cls[c] = __ballot_sync(0xffffffffu, lane < (u32)nwin && mine.c == c);
    constexpr u32 TWL = 32 * LANE_UNITS;
    const u32 ntiles = (nu + TWL - 1) / TWL;
    const u32 warps_total = (gridDim.x * blockDim.x) >> 5;
    for (u32 t = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; t < ntiles; t += warps_total)
        frob4_tile<LANE_UNITS, RO>(in32, o, n32, nu, tab, tabK, nwin, mine, cls, TWL * t, lane);
}

}  // namespace

namespace gf2e {

bool frob4_supported(u64 r, size_t stride) {
    return r < (1ull << 31) - (1ull << 16) && !(stride & 1);
}

// squarings fused per pass for the batched entry points, from
// GF2E_SQUARINGS_PER_PASS (read at each call): 1 keeps the one-squaring
// kernel throughout, 2 uses the fused pass wherever it applies; unset, the
// fused pass is used where it applies and pays.
int squarings_per_pass() {
    const char *e = getenv("GF2E_SQUARINGS_PER_PASS");
    if (!e) return 0;
    const int v = atoi(e);
    return v == 1 || v == 2 ? v : 0;
}

// fused pass for this batch: applies (r, stride), and not switched off.  Two
// squarings by one fused pass or two single ones, us: 607 / 797 (64 states at
// r = 136279841), 14 / 28 (1), 25 / 47 (256 at 999961), 7 / 17 (24 at 99767),
// 6 / 13 (16 at 4423)
bool use_frob4(u64 r, size_t stride) {
    return squarings_per_pass() != 1 && frob4_supported(r, stride);
}

// `chained`: the launch before this one on `st` was a pass of the same call,
// so this one's CTAs may start (and compose their windows) while its last
// ones drain; the kernel waits for it before it touches the states.  A pass
// without / with, us: 8.6 / 6.8 (32 states at r = 100003), 12.7 / 10.9 (64 at
// 999961), 27.9 / 25.5 (256), 14.8 / 13.9 (1 at 136279841).  Batches of many
// rounds gain nothing and keep read-only loads (582 us, plain 588, 64 states).
int launch_frob4(const u64 *in, u64 *out, size_t stride, int nstates, u64 r, const u64 *s_dev,
                 u64 s, cudaStream_t st, bool chained) {
    if (!frob4_supported(r, stride)) return invalid("launch_frob4: needs r < 2^31, even stride");
    const size_t nw = (size_t)((r + 63) >> 6);
    const size_t nu = (nw + 1) / 2;
    // Warp tiles a warp (the window set each CTA composes serves 8 times as
    // many): four when that leaves 16 rounds of the resident CTAs, three when
    // it leaves one, else as many as one round leaves.  A pass in us by tiles
    // a warp 1 / 2 / 3 / 4 / 6 / 8: 64 states at r = 136279841 690 / 626 / 607
    // / 602 / 634 / 652, 3 of them 39 / 38 / 38 / 45 / 40 / 43, 16 at 30000001
    // 45 / 44 / 43 / 48 / 48 / 51, 4 at 10001567 (0.9 rounds of one tile) 11 /
    // 13 / 17 / 19 / 27 / 33
    const size_t twl = 32 * (size_t)LANE_UNITS;
    const size_t ntile = (nu + twl - 1) / twl;
    const size_t slots = (size_t)MIN_CTAS * sm_count();
    auto ctas = [&](size_t t) { return (ntile + 8 * t - 1) / (8 * t); };
    const bool deep = ctas(4) * nstates >= 16 * slots;
    size_t bx = deep              ? ctas(4)
                : ctas(3) * nstates >= slots    ? ctas(3)
                                                : std::min(ctas(1), (slots + nstates - 1) / nstates);
    if (bx > 65535) bx = 65535;
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)bx, (unsigned)nstates);
    cfg.blockDim = dim3(256);
    cfg.stream = st;
    cfg.attrs = &attr;
    cfg.numAttrs = chained && !deep ? 1 : 0;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, cfg.numAttrs ? k_frob4_batch<false> : k_frob4_batch<true>,
                                             in, out, stride, r, s_dev, s);
    return e == cudaSuccess ? GF2E_OK : cuda_status(e, "k_frob4_batch");
}

int trin_square_any(const u64 *in, u64 *out, size_t stride, int nstates, u64 r,
                    const u64 *s_dev, u64 s, cudaStream_t st);

// k squarings of every state (s_dev[i] for state i, s_uniform for all when
// s_dev is null), alternating between a and b.  Squarings go two per pass
// where the fused kernel applies.  With `where` null the result is left in a:
// the passes are made even in number (one fused pass turned into two single
// ones when needed), so no copy is needed unless k = 1 or only single passes
// apply and k is odd.  Otherwise *where is the buffer that holds it.
int frobenius_states(u64 *a, u64 *b, size_t stride, int nstates, u64 r, const u64 *s_dev,
                     u64 k, cudaStream_t st, u64 s_uniform, u64 **where) {
    // the fused pass stores word pairs: both buffers on 16 bytes
    const bool fused = use_frob4(r, stride) && (((uintptr_t)a | (uintptr_t)b) & 15) == 0;
    u64 n4 = fused ? k / 2 : 0, n1 = k - 2 * n4;
    if (!where && ((n4 + n1) & 1) && n4 > 0) {
        n4--;
        n1 += 2;
    }
    u64 *x = a, *y = b;
    for (u64 i = 0; i < n4; i++) {
        GF2E_TRY(launch_frob4(x, y, stride, nstates, r, s_dev, s_uniform, st, i > 0));
        std::swap(x, y);
    }
    for (u64 i = 0; i < n1; i++) {
        GF2E_TRY(trin_square_any(x, y, stride, nstates, r, s_dev, s_uniform, st));
        std::swap(x, y);
    }
    if (where) {
        *where = x;
    } else if (x != a) {
        cudaError_t e = cudaMemcpyAsync(a, x, (size_t)nstates * stride * 8,
                                        cudaMemcpyDeviceToDevice, st);
        if (e != cudaSuccess) return cuda_status(e, "frobenius copy-back");
    }
    return GF2E_OK;
}

}  // namespace gf2e

extern "C" int gf2e_trin_squarings_per_pass(uint64_t r, size_t stride_words, int nstates) {
    // passes over HBM: states and scratch of at most 96 MB stay in L2
    const size_t n = nstates < 1 ? 1 : nstates;
    if (gf2e::squarings_per_pass() != 2 && n * stride_words * 16 <= ((size_t)96 << 20)) return 1;
    return gf2e::use_frob4(r, stride_words) ? 2 : 1;
}
