// lehmer.cuh -- Lehmer rounds of a GF(2)[x] gcd in one CTA, operands in shared
// memory: the half-gcd's base case (hgcd.cu, with the transition matrix) and
// the whole quadratic gcd of operands that fit (gcd.cu, without it).
#pragma once

#include "gf2e_internal.cuh"

namespace {

constexpr int BASE_THREADS = 512;

GF2E_DEV int deg64(u64 v) { return v ? 63 - __clzll(v) : -1; }

GF2E_DEV u64 win_at(const u64 *X, long long nw, long long pos) {   // bits pos..pos+63
    long long i = pos >> 6;
    unsigned sh = (unsigned)(pos & 63);
    u64 a = (i >= 0 && i < nw) ? X[i] : 0, b = (i + 1 < nw) ? X[i + 1] : 0;
    return funnel64(a, b, sh);
}

// warp-wide degree of X below word `top` (inclusive); all 32 lanes return it
GF2E_DEV long long warp_degree(const u64 *X, long long top) {
    const int lane = threadIdx.x & 31;
    for (long long base = top; base >= 0; base -= 32) {
        long long i = base - lane;
        u64 v = (i >= 0) ? X[i] : 0;
        unsigned ball = __ballot_sync(0xffffffffu, v != 0);
        if (ball) {
            int l = __ffs(ball) - 1;
            u64 vv = __shfl_sync(0xffffffffu, v, l);
            return (base - l) * 64 + 63 - __clzll(vv);
        }
    }
    return -1;
}

// One Lehmer round on 64-bit windows of A and B taken at bit `lo` (deg A = da
// >= deg B = db >= m): division steps one degree at a time, on windows kept
// left-aligned at the degree each is known to.  With f = (window, row) of the
// vector with its leading coefficient at bit 63 and g the other, s_f and s_g
// the places each has been shifted up: where g's top bit is set, and f is the
// longer (s_g > s_f), they swap; then g += f clears the bit, and g moves up one
// place.  The rows move with their windows, so the entries are the rows shifted
// down by s_f and s_g at the end, of degree at most s_g and s_f.  Every bit
// decided on is exact: a window shifted by s has 64 - s exact bits, and there
// are at most 62 steps.  A swap needs s_g <= 31 (entries of 32 bits) and deg g
// >= m (the half-gcd's stop: deg a' >= m).
//
// Each step is a dozen integer operations without a branch; the lanes of a
// warp hold the columns of the matrix by parity and run the windows side by
// side.  (62 steps take 3163 cycles; whole quotients, each a loop over its own
// degrees with a degree search and the role swap after it, took 3258 on one
// thread.)
struct Lehmer {
    u32 ef, eg;         // this lane's column of the rows of a' and b'
    long long k;
    int mode;           // 1: a gap of more than 31 degrees, A ^= B << k alone
};
GF2E_DEV Lehmer lehmer_round(u64 wa, u64 wb, long long da, long long db, long long lo,
                             long long m, int lane) {
    Lehmer L;
    L.k = da - db;
    L.mode = L.k > 31 ? 1 : 0;
    L.ef = L.eg = 0;
    if (L.mode) return L;
    const int dga = (int)(da - lo);
    const int lim = m > lo ? min(31, dga - (int)(m - lo)) : 31;
    u64 A = wa << (63 - dga), B = wb << (63 - dga);
    int N = 0;                                          // s_f - s_g
    int t = 0;                                          // s_f + s_g
    u64 p, q;
    {
        u32 p1 = (lane & 1) ^ 1, q1 = lane & 1;
        if (lim == 31) {
            // s_g <= t <= 31 and rows of 32 bits: no test
#pragma unroll
            for (int i = 0; i < 31; i++) {
                const int bh = (int)(B >> 32), c = bh >> 31, sw = (bh & N) >> 31;
                const u64 c64 = ((u64)(u32)c << 32) | (u32)c, s64 = ((u64)(u32)sw << 32) | (u32)sw;
                const u64 a = A;
                const u32 x = p1;
                A = (a & ~s64) | (B & s64);
                p1 = (x & ~(u32)sw) | (q1 & (u32)sw);
                B = (B ^ (a & c64)) << 1;
                q1 = (q1 ^ (x & (u32)c)) << 1;
                N = (N ^ sw) - 1 - sw;
            }
            t = 31;
        }
        p = p1;
        q = q1;
    }
    int R = 2 * lim - t;                                // R + N < 0: s_g > lim
#pragma unroll 4
    for (; t < 62; t++) {
        const int bh = (int)(B >> 32);
        if ((bh & N & (R + N)) < 0) break;              // a swap that is not allowed
        const int c = bh >> 31, sw = (bh & N) >> 31;
        const u64 c64 = ((u64)(u32)c << 32) | (u32)c, s64 = ((u64)(u32)sw << 32) | (u32)sw;
        const u64 a = A, x = p;
        A = (a & ~s64) | (B & s64);
        p = (x & ~s64) | (q & s64);
        B = (B ^ (a & c64)) << 1;
        q = (q ^ (x & c64)) << 1;
        N = (N ^ sw) - 1 - sw;
        R--;
    }
    const int sf = (t + N) >> 1;
    L.ef = (u32)(p >> sf);
    L.eg = (u32)(q >> (t - sf));
    return L;
}

// x * m_a and x * m_b as 96 bits each (lo: bits 0..63, hi: bits 64..95) by
// 16-entry tables T[v] = v * m (v a nibble, entries of up to 35 bits), one
// pass over x's nibbles for both: lookups, shifts and XORs, no multiplies
// (the 32 x 32 -> 64 multiplier of the bit-class product is the apply's
// bottleneck)
GF2E_DEV void mul96_tab2(u64 x, const u64 *Ta, const u64 *Tb, u64 &la, u64 &ha, u64 &lb,
                         u64 &hb) {
    la = ha = lb = hb = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        const unsigned v = (unsigned)(x >> (4 * i)) & 15u;
        const u64 ta = Ta[v], tb = Tb[v];
        la ^= ta << (4 * i);
        lb ^= tb << (4 * i);
        if (i >= 8) {                                  // entries reach bit 34
            ha ^= ta >> (64 - 4 * i);
            hb ^= tb >> (64 - 4 * i);
        }
    }
}
// word w of (X << k) for a vector X
GF2E_DEV u64 shl_word(const u64 *X, long long w, long long k) {
    const long long ks = k >> 6;
    const unsigned kb = (unsigned)(k & 63);
    u64 h = (w >= ks) ? X[w - ks] : 0, l = (w >= ks + 1) ? X[w - ks - 1] : 0;
    return kb ? ((h << kb) | (l >> (64 - kb))) : h;
}
// what the rounds ended with (thread 0's counters)
struct LehmerEnd {
    int parity = 0;              // which copy of the rows holds the result
    int va = 0, ra = 0;          // vector of a' (of the gcd without ROWS), row of a'
    int status = GF2E_OK;
    long long rounds = 0, cyc_serial = 0;
};

// (a', b') = M (a, b) with deg a' >= m > deg b'; with ROWS the matrix M in four
// arrays of mw words (row-major M00 M01 M10 M11).  Without, m = 0: the gcd, at
// b' = 0 or b' = 1.
//
// Lehmer rounds, pipelined: while warps 1..15 apply round r's matrix to the
// vectors A, B and to the accumulated rows (one output word per item, the
// carry from word w-1 recomputed, so no barrier inside the round), warp 0
// computes the six top 32-bit chunks of the new A and B itself, reads their
// degrees and 64-bit windows off them and runs round r+1's division steps.
// One barrier per round; when the new windows are not within
// those chunks (a large drop in degree), warp 0 scans the new vectors
// after the barrier instead.  Round state is double-buffered by parity.
// Shared memory: V[4][W] (two buffers of A, B), R[2][4][mw].
// The caller has put a and b (zeros above) into V[0 .. W), V[W .. 2 W) and, with
// ROWS, the identity into R[0], and passed a barrier; degrees da0 and db0.
template <bool ROWS>
GF2E_DEV LehmerEnd lehmer_cta(u64 *V, u64 W, u64 *R, u64 mw, long long da0, long long db0,
                              long long m) {
    LehmerEnd E;
    __shared__ int s_va[2], s_vb[2], s_ra[2], s_mode[2], s_done[2], s_slow[2];
    __shared__ long long s_k[2], s_top[2], s_md[2];
    __shared__ u32 s_m[2][4];
    __shared__ u64 s_tab[(BASE_THREADS / 32 / 4) * 3][64];   // per apply warp: v * m_e
    const int tid = threadIdx.x;
    const long long max_rounds = 2 * (max(da0, db0) + 2) + 16;

    // warp 0: publish round q's state from degrees/roles and windows
    auto publish = [&](int q, int va, int vb, int ra, long long da, long long db, u64 wa, u64 wb,
                       long long md, long long round) {
        if (da < db) {
            int x = va; va = vb; vb = x;
            ra ^= 1;
            long long t = da; da = db; db = t;
            u64 u = wa; wa = wb; wb = u;
        }
        // a gcd with 1 is 1: beside a long a each round would clear one
        // coefficient of it (a unit against 409000 bits: 200000 rounds)
        const bool unit = !ROWS && db == 0;
        const bool done = unit || db < m || round > max_rounds;
        if (tid == 0) {
            s_va[q] = unit ? vb : va;
            s_vb[q] = vb; s_ra[q] = ra;
            s_top[q] = da >> 6;
            s_md[q] = md;
            s_done[q] = done;
            if (round > max_rounds) E.status = GF2E_ERR_TIMEOUT;
            E.rounds = round;
        }
        if (done) return;
        const long long lo = da >= 63 ? da - 63 : 0;
        const long long c0 = clock64();
        const Lehmer L = lehmer_round(wa, wb, da, db, lo, m, tid);
        E.cyc_serial += clock64() - c0;
        if (tid < 2) {
            s_m[q][tid] = L.ef;
            s_m[q][2 + tid] = L.eg;
        }
        if (tid == 0) {
            s_mode[q] = L.mode;
            s_k[q] = L.k;
        }
    };
    // warp 0: degrees and windows of vectors va, vb read from shared memory
    auto publish_from_vectors = [&](int q, int va, int vb, int ra, long long da, long long db,
                                    long long md, long long round) {
        const long long dhi = max(da, db);
        const long long lo = dhi >= 63 ? dhi - 63 : 0;
        publish(q, va, vb, ra, da, db, win_at(V + (u64)va * W, (long long)W, lo),
                win_at(V + (u64)vb * W, (long long)W, lo), md, round);
    };
    if (tid < 32) publish_from_vectors(0, 0, 1, 0, da0, db0, 0, 0);
    __syncthreads();

    for (long long round = 0;; round++) {
        const int p = (int)(round & 1), q = p ^ 1;
        if (s_done[p]) {
            E.parity = p;
            E.va = s_va[p];
            E.ra = s_ra[p];
            break;
        }
        const int va = s_va[p], vb = s_vb[p], ra = s_ra[p], mode = s_mode[p];
        const long long top = s_top[p], md = s_md[p], k = s_k[p];
        // live words: vectors 0..top; rows 0..nwm (the growth of this round included)
        const long long nwv = top + 1;
        const long long nwm =
            ROWS ? min((long long)mw - 1, md + (mode == 1 ? (k >> 6) + 1 : 1)) : 0;
        int spare[2], ns = 0;
        for (int i = 0; i < 4 && ns < 2; i++)
            if (i != va && i != vb) spare[ns++] = i;
        const u64 *A = V + (u64)va * W, *B = V + (u64)vb * W;
        u64 *A2 = V + (u64)spare[0] * W, *B2 = V + (u64)spare[1] * W;
        const u64 *RA = R + (u64)(p * 4 + 2 * ra) * mw, *RB = R + (u64)(p * 4 + 2 * (ra ^ 1)) * mw;
        u64 *N = R + (u64)q * 4 * mw;
        const long long md_next =
            ROWS ? min((long long)mw - 2, md + (mode == 1 ? (k >> 6) + 1 : 1)) : 0;
        const int warp = tid >> 5;
        if (warp != 0 && (warp & 3) != 0) {
            // the apply runs on the warps of the other three schedulers, so
            // warp 0's serial chain keeps its scheduler (warp w is on w % 4).
            // Work in chunks of 31 output words of one pair of outputs: the
            // new vectors (A', B') from (A, B), or the new row entries
            // (N[col], N[2 + col]) from (RA[col], RB[col]).  Lane l takes
            // word 31 c + l - 1 of the inputs, computes its full products
            // (by the warp's nibble tables of the four matrix entries) and
            // passes their high words up one lane: lane 0's word only feeds
            // lane 1, so every input word is multiplied once.
            constexpr int APPLY_WARPS = (BASE_THREADS / 32 / 4) * 3;
            const int aw = warp - 1 - (warp >> 2), lane = tid & 31;
            u64 *T = s_tab[aw];                         // T[16 e + v] = v * m_e
            if (mode != 1) {
                for (int i = lane; i < 64; i += 32) {
                    const u64 me = s_m[p][i >> 4];
                    u64 t = 0;
#pragma unroll
                    for (int b = 0; b < 4; b++)
                        if ((i >> b) & 1) t ^= me << b;
                    T[i] = t;
                }
                __syncwarp();
            }
            const long long ncv = (nwv + 30) / 31, ncr = ROWS ? (nwm + 31) / 31 : 0;
            for (long long c = aw; c < ncv + 2 * ncr; c += APPLY_WARPS) {
                const bool vec = c < ncv;
                const long long cr = c - ncv;
                const int col = vec ? 0 : (int)(cr / ncr);
                const long long n = vec ? nwv : nwm + 1;
                const long long w = 31 * (vec ? c : cr - col * ncr) + lane - 1;
                const u64 *X = vec ? A : RA + (u64)col * mw, *Y = vec ? B : RB + (u64)col * mw;
                u64 *O0 = vec ? A2 : N + (u64)col * mw, *O1 = vec ? B2 : N + (u64)(2 + col) * mw;
                const bool in = w >= 0 && w < n;
                u64 o0 = 0, o1 = 0;
                if (mode == 1) {                        // (X ^ (Y << k), Y)
                    if (in) {
                        o0 = X[w] ^ shl_word(Y, w, k);
                        o1 = Y[w];
                    }
                } else {                                // (m0 X + m1 Y, m2 X + m3 Y)
                    u64 l0, h0, l1, h1, tl0, th0, tl1, th1;
                    mul96_tab2(in ? X[w] : 0, T, T + 32, l0, h0, l1, h1);        // x m0, x m2
                    mul96_tab2(in ? Y[w] : 0, T + 16, T + 48, tl0, th0, tl1, th1);  // y m1, y m3
                    l0 ^= tl0; h0 ^= th0;
                    l1 ^= tl1; h1 ^= th1;
                    o0 = l0 ^ __shfl_up_sync(0xffffffffu, h0, 1);
                    o1 = l1 ^ __shfl_up_sync(0xffffffffu, h1, 1);
                }
                if (lane >= 1 && in) {
                    O0[w] = o0;
                    O1[w] = o1;
                }
            }
            // stale words of the new vectors above the live range
            constexpr int APPLY_THREADS = APPLY_WARPS * 32;
            const int at = aw * 32 + lane;
            for (long long w = nwv + at; w < (long long)W; w += APPLY_THREADS) {
                A2[w] = 0;
                B2[w] = 0;
            }
        } else if (warp == 0) {
            // warp 0: the six top 32-bit chunks of the new A and B, then their
            // degrees and the next windows by ballot and shuffle
            const int lane = tid, r = lane >> 4, c = lane & 7;
            const long long g0 = 2 * top + 1;                 // chunk c is number g0 - c
            u32 ch = 0;
            if (mode != 1) {
                // lane (row r, vector, c < 7) multiplies one chunk of A or B by
                // its entry; the rows' sums, and the high half of the chunk below
                const u32 *X = reinterpret_cast<const u32 *>((lane & 8) ? B : A);
                const u32 x = c < 7 && g0 - c >= 0 ? X[g0 - c] : 0;
                u64 P = clmul32(x, s_m[p][2 * r + ((lane >> 3) & 1)]);
                P ^= __shfl_xor_sync(0xffffffffu, P, 8);
                const u32 up = __shfl_down_sync(0xffffffffu, (u32)(P >> 32), 1);
                ch = c < 6 ? (u32)P ^ up : 0;
            } else {
                const long long w = top - (c >> 1);
                u64 v = 0;
                if (c < 6 && w >= 0) v = r ? B[w] : A[w] ^ shl_word(B, w, k);
                ch = (u32)((c & 1) ? v : v >> 32);
            }
            const unsigned nz = __ballot_sync(0xffffffffu, ch != 0);
            const int fa = __ffs(nz & 63u) - 1, fb = __ffs((nz >> 16) & 63u) - 1;
            const u32 ta = __shfl_sync(0xffffffffu, ch, fa < 0 ? 0 : fa);
            const u32 tb = __shfl_sync(0xffffffffu, ch, fb < 0 ? 16 : 16 + fb);
            const long long dn0 = fa < 0 ? -1 : (g0 - fa) * 32 + 31 - __clz(ta);
            const long long dn1 = fb < 0 ? -1 : (g0 - fb) * 32 + 31 - __clz(tb);
            bool slow = dn0 < 0 || dn1 < 0;
            const long long dhi = max(dn0, dn1), lo = dhi >= 63 ? dhi - 63 : 0;
            slow = slow || (lo >> 5) < g0 - 5;
            // the windows' lowest chunk is chunk i0, the two above it i0 - 1, i0 - 2
            const int i0 = slow ? 2 : (int)(g0 - (lo >> 5));
            const int i1 = max(i0 - 1, 0), i2 = max(i0 - 2, 0);
            u32 x[2][3];
#pragma unroll
            for (int v = 0; v < 2; v++) {
                x[v][0] = __shfl_sync(0xffffffffu, ch, 16 * v + i0);
                x[v][1] = __shfl_sync(0xffffffffu, ch, 16 * v + i1);
                x[v][2] = __shfl_sync(0xffffffffu, ch, 16 * v + i2);
                if (i0 < 1) x[v][1] = 0;
                if (i0 < 2) x[v][2] = 0;
            }
            if (!slow) {
                const unsigned sb = (unsigned)(lo & 31);
                u64 win[2];
#pragma unroll
                for (int v = 0; v < 2; v++)
                    win[v] = ((u64)__funnelshift_r(x[v][1], x[v][2], sb) << 32) |
                             __funnelshift_r(x[v][0], x[v][1], sb);
                publish(q, spare[0], spare[1], 0, dn0, dn1, win[0], win[1], md_next, round + 1);
            }
            if (lane == 0) s_slow[p] = slow;
        }
        __syncthreads();
        // of its own parity too: warp 0 may be deciding the next round before
        // another warp has read this
        if (s_slow[p]) {                                // degrees from the full new vectors
            if (tid < 32) {
                const long long d0 = warp_degree(A2, top), d1 = warp_degree(B2, top);
                publish_from_vectors(q, spare[0], spare[1], 0, d0, d1, md_next, round + 1);
            }
            __syncthreads();
        }
    }
    __syncthreads();
    return E;
}

}  // namespace
