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

// one Lehmer round on exact 64-bit windows of A and B taken at bit `lo`
// (deg A = da >= deg B): whole quotients while every bit they depend on is
// exact (a row's window bits are exact above its matrix degree), the
// half-gcd stop (deg B < m) is not reached and the 2x2 matrix stays within
// degree 31; mode 1 (no quotient fits) is the single shift-XOR A ^= B << k.
struct Lehmer {
    u32 mt[4];
    long long k;
    int mode;
};
GF2E_DEV Lehmer lehmer_round(u64 wa, u64 wb, long long da, long long db, long long lo,
                             long long m) {
    Lehmer L;
    u32 ma0 = 1, ma1 = 0, mb0 = 0, mb1 = 1;
    int dga = (int)(da - lo), dgb = deg64(wb), dma = 0, dmb = 0, steps = 0;
    const bool exact = (lo == 0);
    const int dstop = (int)max(-1LL, m - lo);          // window degree of x^m
    // the windows left-aligned (leading coefficient at bit 63): the division
    // below then tests one bit and shifts, with no degree search per step
    u64 A = wa << (63 - dga);
    u64 B = dgb >= 0 ? wb << (63 - dgb) : 0;
    for (int it = 0; it < 64; it++) {
        if (dgb < 0 || dgb < dstop) break;              // b = 0 / half-gcd stop
        const int dq = dga - dgb;
        const int ndm = max(dma, dmb + dq);
        if (ndm > 31) break;                            // matrix degree bound
        if (!exact && dgb < ndm) break;                 // quotient not exact
        // a <- a mod b, row a += q row b: at each of the dq + 1 degrees from
        // the top, XOR in b (and x^(dq-j) row b) when a's leading bit is set,
        // then move one degree down.  Afterwards bit 63 of A is degree dgb.
        // At the top degree the bit is a's leading coefficient, always set.
        u32 s0 = mb0 << dq, s1 = mb1 << dq;
        A ^= B;
        ma0 ^= s0;
        ma1 ^= s1;
#pragma unroll 1
        for (int j = 1; j <= dq; j++) {
            A <<= 1;
            s0 >>= 1;
            s1 >>= 1;
            const u64 msk = (u64)((long long)A >> 63);
            A ^= B & msk;
            ma0 ^= s0 & (u32)msk;
            ma1 ^= s1 & (u32)msk;
        }
        const int c = A ? __clzll(A) : 64;
        const u64 Bn = A ? A << c : 0;
        const int dr = A ? dgb - c : -1;
        A = B;                                          // (a, b) <- (b, a mod b)
        B = Bn;
        dga = dgb;
        dgb = dr;
        u32 y = ma0; ma0 = mb0; mb0 = y;
        y = ma1; ma1 = mb1; mb1 = y;
        dma = dmb;
        dmb = ndm;
        steps++;
    }
    if (steps == 0) {
        L.mode = 1;
        L.k = da - db;
        L.mt[0] = L.mt[1] = L.mt[2] = L.mt[3] = 0;
    } else {
        L.mode = 0;
        L.k = 0;
        L.mt[0] = ma0; L.mt[1] = ma1; L.mt[2] = mb0; L.mt[3] = mb1;
    }
    return L;
}

// lo and hi parts of x (64 bits) times a 32-bit polynomial
GF2E_DEV u64 mul64x32_lo(u64 x, const Masked &m) {
    return clmul_masked(mask32((u32)x), m) ^ (clmul_masked(mask32((u32)(x >> 32)), m) << 32);
}
GF2E_DEV u64 mul64x32_hi(u64 x, const Masked &m) {
    return clmul_masked(mask32((u32)(x >> 32)), m) >> 32;
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
// word w of one new vector / row: mode 0: m0*X + m1*Y; mode 1 (row a): X ^ (Y << k)
GF2E_DEV u64 new_word(int mode, const u64 *X, const u64 *Y, long long w, const Masked &m0,
                      const Masked &m1, long long k, bool is_a) {
    if (mode == 1) return is_a ? (X[w] ^ shl_word(Y, w, k)) : Y[w];
    u64 v = mul64x32_lo(X[w], m0) ^ mul64x32_lo(Y[w], m1);
    if (w >= 1) v ^= mul64x32_hi(X[w - 1], m0) ^ mul64x32_hi(Y[w - 1], m1);
    return v;
}

// what the rounds ended with (thread 0's counters)
struct LehmerEnd {
    int parity = 0;              // which copy of the rows holds the result
    int va = 0, ra = 0;          // vector of a', row of a'
    int status = GF2E_OK;
    long long rounds = 0, cyc_serial = 0;
};

// (a', b') = M (a, b) with deg a' >= m > deg b'; with ROWS the matrix M in four
// arrays of mw words (row-major M00 M01 M10 M11).  m = 0 runs to b' = 0.
//
// Lehmer rounds, pipelined: while warps 1..15 apply round r's matrix to the
// vectors A, B and to the accumulated rows (one output word per item, the
// carry from word w-1 recomputed, so no barrier inside the round), warp 0
// computes the three top words of the new A and B itself, reads their
// degrees and 64-bit windows off them and runs round r+1's Euclid steps on
// thread 0.  One barrier per round; when the new windows are not within
// those three words (a large drop in degree), warp 0 scans the new vectors
// after the barrier instead.  Round state is double-buffered by parity.
// Shared memory: V[4][W] (two buffers of A, B), R[2][4][mw].
// The caller has put a and b (zeros above) into V[0 .. W), V[W .. 2 W) and, with
// ROWS, the identity into R[0], and passed a barrier; degrees da0 and db0.
template <bool ROWS>
GF2E_DEV LehmerEnd lehmer_cta(u64 *V, u64 W, u64 *R, u64 mw, long long da0, long long db0,
                              long long m) {
    LehmerEnd E;
    __shared__ int s_va[2], s_vb[2], s_ra[2], s_mode[2], s_done[2], s_slow;
    __shared__ long long s_k[2], s_top[2], s_md[2];
    __shared__ u32 s_m[2][4];
    __shared__ u64 s_tab[(BASE_THREADS / 32 / 4) * 3][64];   // per apply warp: v * m_e
    const int tid = threadIdx.x;
    const long long max_rounds = 2 * (max(da0, db0) + 2) + 16;

    // thread 0: publish round q's state from degrees/roles and windows
    auto publish = [&](int q, int va, int vb, int ra, long long da, long long db, u64 wa, u64 wb,
                       long long md, long long round) {
        if (da < db) {
            int x = va; va = vb; vb = x;
            ra ^= 1;
            long long t = da; da = db; db = t;
            u64 u = wa; wa = wb; wb = u;
        }
        s_va[q] = va; s_vb[q] = vb; s_ra[q] = ra;
        s_top[q] = da >> 6;
        s_md[q] = md;
        if (db < m || round > max_rounds) {
            s_done[q] = 1;
            if (round > max_rounds) E.status = GF2E_ERR_TIMEOUT;
            E.rounds = round;
            return;
        }
        s_done[q] = 0;
        const long long lo = da >= 63 ? da - 63 : 0;
        const long long c0 = clock64();
        Lehmer L = lehmer_round(wa, wb, da, db, lo, m);
        E.cyc_serial += clock64() - c0;
        s_mode[q] = L.mode;
        s_k[q] = L.k;
        for (int i = 0; i < 4; i++) s_m[q][i] = L.mt[i];
    };
    // thread 0: degrees and windows of vectors va, vb read from shared memory
    auto publish_from_vectors = [&](int q, int va, int vb, int ra, long long da, long long db,
                                    long long md, long long round) {
        const long long dhi = max(da, db);
        const long long lo = dhi >= 63 ? dhi - 63 : 0;
        publish(q, va, vb, ra, da, db, win_at(V + (u64)va * W, (long long)W, lo),
                win_at(V + (u64)vb * W, (long long)W, lo), md, round);
    };
    if (tid == 0) publish_from_vectors(0, 0, 1, 0, da0, db0, 0, 0);
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
        const Masked m0 = mask32(s_m[p][0]), m1 = mask32(s_m[p][1]), m2 = mask32(s_m[p][2]),
                     m3 = mask32(s_m[p][3]);
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
            // warp 0: the three top words of the new A (lanes 0-2) and B (3-5)
            // in one pass (each lane with its own matrix row), then their
            // degrees and the next windows by ballot and shuffle
            const int lane = tid;
            const bool vb = lane >= 3;
            const long long w = top - (lane % 3);
            u64 val = 0;
            if (lane < 6 && w >= 0)
                val = new_word(mode, A, B, w, vb ? m2 : m0, vb ? m3 : m1, k, !vb);
            const unsigned nz = __ballot_sync(0xffffffffu, lane < 6 && val != 0);
            const int fa = __ffs(nz & 7u) - 1, fb = __ffs((nz >> 3) & 7u) - 1;
            const u64 ta = __shfl_sync(0xffffffffu, val, fa < 0 ? 0 : fa);
            const u64 tb = __shfl_sync(0xffffffffu, val, fb < 0 ? 3 : 3 + fb);
            const long long dn0 = fa < 0 ? -1 : (top - fa) * 64 + 63 - __clzll(ta);
            const long long dn1 = fb < 0 ? -1 : (top - fb) * 64 + 63 - __clzll(tb);
            bool slow = dn0 < 0 || dn1 < 0;
            long long lo = 0;
            if (!slow) {
                const long long dhi = max(dn0, dn1);
                lo = dhi >= 63 ? dhi - 63 : 0;
                slow = (lo >> 6) < top - 2;
            }
            // the windows' low words are words lo/64 (lane top - lo/64) and
            // lo/64 + 1 (one lane lower) of the new vectors
            const int ia = slow ? 0 : (int)(top - (lo >> 6));
            const int ib = ia >= 1 ? ia - 1 : 0;
            const u64 x0a = __shfl_sync(0xffffffffu, val, ia), x1a = __shfl_sync(0xffffffffu, val, ib);
            const u64 x0b = __shfl_sync(0xffffffffu, val, 3 + ia), x1b = __shfl_sync(0xffffffffu, val, 3 + ib);
            if (lane == 0) {
                if (!slow) {
                    const unsigned sb = (unsigned)(lo & 63);
                    publish(q, spare[0], spare[1], 0, dn0, dn1, funnel64(x0a, ia >= 1 ? x1a : 0, sb),
                            funnel64(x0b, ia >= 1 ? x1b : 0, sb), md_next, round + 1);
                }
                s_slow = slow;
            }
        }
        __syncthreads();
        if (s_slow) {                                  // degrees from the full new vectors
            if (tid < 32) {
                const long long d0 = warp_degree(A2, top), d1 = warp_degree(B2, top);
                if (tid == 0) publish_from_vectors(q, spare[0], spare[1], 0, d0, d1, md_next, round + 1);
            }
            __syncthreads();
        }
    }
    __syncthreads();
    return E;
}

}  // namespace
