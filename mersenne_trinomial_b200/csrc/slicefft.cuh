// slicefft.cuh -- bit-sliced core of the products' Cantor transform
// (slicefft.cu launches it): field arithmetic, Taylor levels and butterfly
// passes as functions of (thread, thread count) on a shared-memory tile, so
// that each step is a plain loop between two barriers.
//
// A product needs no particular transform order or field representation
// between its forward and inverse transforms, so this one is laid out for
// the ALU.  A "slice" is 32 consecutive elements held as 64 bit planes of 32
// bits (bit e of plane p = coordinate p of element e), 256 bytes, the same
// place in memory as the 32 elements.  GF(2^64) is taken in the tower basis
// x_k^2 = x_k + x_0 .. x_(k-1) (the nim field: coordinate i is the product of
// the x_k over the set bits k of i), in which the subfields GF(2^8),
// GF(2^16), GF(2^32) are the low 8, 16, 32 coordinates.  The twiddle of
// butterfly level L is a sum of the Cantor basis elements 1 .. m-1-L, which
// lie in those subfields, so a multiply splits into 8 / 4 / 2 independent
// subfield multiplies, each a Karatsuba tree of AND-XORs over planes: 61,
// 211 and ~600 operations for 32 products, 15-38 a field product where a
// 64 x 64 carry-less multiply by integer multiplies takes ~200.
#pragma once

#include <stdint.h>
#include <utility>

#ifdef __CUDACC__
#define SL_HD __device__ __forceinline__
#else
#define SL_HD inline
struct uint4 { uint32_t x, y, z, w; };
#endif

namespace slice {

typedef uint64_t u64;
typedef uint32_t u32;

// ------------------------------------------------- tower-field constants
constexpr u64 c_delta(u64 a, int n) {            // a * v_(n-1) in GF(2^n)
    if (n == 1) return a;
    const int h = n / 2;
    const u64 lo = a & ((1ull << h) - 1), hi = a >> h;
    return c_delta(c_delta(hi, h), h) | (c_delta(lo ^ hi, h) << h);
}
constexpr u64 c_mul(u64 a, u64 b, int n) {
    if (!a || !b) return 0;
    if (n == 1) return a & b;
    const int h = n / 2;
    const u64 m = (1ull << h) - 1;
    const u64 p0 = c_mul(a & m, b & m, h), p1 = c_mul(a >> h, b >> h, h),
              p2 = c_mul((a & m) ^ (a >> h), (b & m) ^ (b >> h), h);
    return (p0 ^ c_delta(p1, h)) | ((p2 ^ p0) << h);
}
// image of x under an isomorphism from GF(2)[x]/(x^64 + x^4 + x^3 + x + 1):
// a root of the modulus in the tower field
constexpr u64 ROOT = 0x67b6b273eb5d60f6ull;

struct Phi {
    u64 to[64];        // to[i] = image of x^i
    u64 from[64];      // from[i] = the polynomial-basis element of coordinate i
};
constexpr Phi make_phi() {
    Phi p{};
    u64 v = 1;
    for (int i = 0; i < 64; i++) {
        p.to[i] = v;
        v = c_mul(v, ROOT, 64);
    }
    // Gauss-Jordan on (to[i], x^i)
    u64 a[64] = {}, b[64] = {};
    for (int i = 0; i < 64; i++) { a[i] = p.to[i]; b[i] = 1ull << i; }
    for (int c = 0; c < 64; c++) {
        int r = c;
        while (r < 64 && !((a[r] >> c) & 1)) r++;
        const u64 ta = a[r], tb = b[r];
        a[r] = a[c]; b[r] = b[c];
        a[c] = ta; b[c] = tb;
        for (int k = 0; k < 64; k++)
            if (k != c && ((a[k] >> c) & 1)) { a[k] ^= a[c]; b[k] ^= b[c]; }
    }
    for (int i = 0; i < 64; i++) p.from[i] = b[i];
    return p;
}
constexpr Phi PHI = make_phi();

// images of the Cantor basis elements 0 .. 24 (checked against the basis in
// the polynomial representation when a plan is made)
constexpr u32 CANTOR[25] = {
    0x1, 0x3, 0x6, 0xf, 0x1c, 0x30, 0x66, 0xf6, 0x1dd, 0x332, 0x604, 0xf95, 0x1c8e,
    0x305d, 0x6638, 0xf6ee, 0x1ddf7, 0x33229, 0x6048c, 0xf95ee, 0x1c8ed9, 0x305d3c,
    0x6638c6, 0xf6ee5d, 0x1dd773f};

// W[t] = XOR of CANTOR[j+1] over the set bits j of t, t < 2^24, by bytes of t
struct TwTab { u32 v[768]; };
constexpr TwTab make_twtab() {
    TwTab t{};
    for (int k = 0; k < 3; k++)
        for (int b = 0; b < 256; b++) {
            u32 w = 0;
            for (int j = 0; j < 8; j++)
                if ((b >> j) & 1) w ^= CANTOR[8 * k + j + 1];
            t.v[256 * k + b] = w;
        }
    return t;
}
// in levels 0..4 the 32 elements of a slice have different twiddles: bit b of
// a slice adds sum of CANTOR[5-L+k] over the set bits k of b; pat[L][i] = plane i
struct PatTab { u32 v[5][16]; };
constexpr PatTab make_pattab() {
    constexpr u32 P[5] = {0xAAAAAAAAu, 0xCCCCCCCCu, 0xF0F0F0F0u, 0xFF00FF00u, 0xFFFF0000u};
    PatTab t{};
    for (int L = 0; L < 5; L++)
        for (int i = 0; i < 16; i++)
            for (int k = 0; k < 5; k++)
                if ((CANTOR[5 - L + k] >> i) & 1) t.v[L][i] ^= P[k];
    return t;
}
#ifdef __CUDACC__
static __device__ const TwTab TWTAB = make_twtab();
static __device__ __constant__ const PatTab PATTAB = make_pattab();
#else
static const TwTab TWTAB = make_twtab();
static const PatTab PATTAB = make_pattab();
#endif

SL_HD u32 twiddle(u32 t) {
    return TWTAB.v[t & 255] ^ TWTAB.v[256 + ((t >> 8) & 255)] ^ TWTAB.v[512 + ((t >> 16) & 255)];
}

// ------------------------------------------------- bit-sliced field products
template <int N> SL_HD void t_delta(const u32 *a, u32 *c) {       // c = v_(N-1) a
    if constexpr (N == 1) {
        c[0] = a[0];
    } else {
        constexpr int H = N / 2;
        u32 s[H], u[H];
#pragma unroll
        for (int i = 0; i < H; i++) s[i] = a[i] ^ a[H + i];
        t_delta<H>(a + H, u);
        t_delta<H>(u, c);
        t_delta<H>(s, c + H);
    }
}
template <int N> SL_HD void t_mul(const u32 *a, const u32 *b, u32 *c) {
    if constexpr (N == 2) {
        const u32 p = a[0] & b[0];
        c[0] = p ^ (a[1] & b[1]);
        c[1] = p ^ ((a[0] ^ a[1]) & (b[0] ^ b[1]));
    } else {
        constexpr int H = N / 2;
        u32 p0[H], p1[H], sa[H], sb[H];
#pragma unroll
        for (int i = 0; i < H; i++) { sa[i] = a[i] ^ a[H + i]; sb[i] = b[i] ^ b[H + i]; }
        t_mul<H>(a, b, p0);
        t_mul<H>(a + H, b + H, p1);
        t_mul<H>(sa, sb, c + H);
        t_delta<H>(p1, c);
#pragma unroll
        for (int i = 0; i < H; i++) { c[H + i] ^= p0[i]; c[i] ^= p0[i]; }
    }
}

// ------------------------------------------------- linear maps on planes
// out[p] = XOR over i < NI of bit p of M[i], in[i]; four inputs at a time
// through their 16 XORs (NO outputs)
template <bool TO, int G, int P> struct Sel {
    static constexpr u64 at(int i) { return ((TO ? PHI.to[i] : PHI.from[i]) >> P) & 1; }
    static constexpr int v = (int)(at(G) | at(G + 1) << 1 | at(G + 2) << 2 | at(G + 3) << 3);
};
template <bool TO, int G, int... P>
SL_HD void lin_group(const u32 *in, u32 *out, std::integer_sequence<int, P...>) {
    u32 c[16];
    c[0] = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int v = 0; v < (1 << k); v++) c[(1 << k) + v] = c[v] ^ in[G + k];
    ((out[P] ^= c[Sel<TO, G, P>::v]), ...);
}
template <bool TO, int NO, int... G>
SL_HD void lin_groups(const u32 *in, u32 *out, std::integer_sequence<int, G...>) {
    (lin_group<TO, 4 * G>(in, out, std::make_integer_sequence<int, NO>{}), ...);
}
template <int NI, int NO, bool TO> SL_HD void lin_map(const u32 *in, u32 *out) {
#pragma unroll
    for (int p = 0; p < NO; p++) out[p] = 0;
    lin_groups<TO, NO>(in, out, std::make_integer_sequence<int, NI / 4>{});
}

// 32 x 32 bit transposition in registers: bit i of x[j] <-> bit j of x[i]
SL_HD void transpose32(u32 *x) {
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const int d = 16 >> k;
        const u32 m = d == 16 ? 0x0000FFFFu : d == 8 ? 0x00FF00FFu : d == 4 ? 0x0F0F0F0Fu
                    : d == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            if (j & d) continue;
            const u32 t = ((x[j] >> d) ^ x[j + d]) & m;
            x[j + d] ^= t;
            x[j] ^= t << d;
        }
    }
}

// ------------------------------------------------- shared-memory slices
// 16-byte chunks of a slice are XOR-swizzled by its number: any 8 slices that
// differ in three of its four low bits put one chunk in 8 different banks,
// which holds for the slices 8 lanes touch at every butterfly distance
SL_HD u32 swz(u32 s) { return (s ^ (0u - ((s >> 3) & 1))) & 7; }
SL_HD u32 chunk_at(u32 s, u32 c) { return (s << 4) + (c ^ swz(s)); }
SL_HD u32 word_at(u32 s, u32 p) { return (chunk_at(s, p >> 2) << 2) + (p & 3); }

template <int N> SL_HD void load_planes(const uint4 *tile, u32 s, u32 c0, u32 *v) {
#pragma unroll
    for (int k = 0; k < N / 4; k++) {
        const uint4 q = tile[chunk_at(s, c0 + k)];
        v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
    }
}
template <int N> SL_HD void store_planes(uint4 *tile, u32 s, u32 c0, const u32 *v) {
#pragma unroll
    for (int k = 0; k < N / 4; k++) {
        uint4 q;
        q.x = v[4 * k]; q.y = v[4 * k + 1]; q.z = v[4 * k + 2]; q.w = v[4 * k + 3];
        tile[chunk_at(s, c0 + k)] = q;
    }
}

// ------------------------------------------------- butterflies
// masks of the N bits of w from bit `sh` (all ones where set), XORed with the
// slice's pattern where its elements differ
template <int N> SL_HD void masks_of(u32 w, int sh, const u32 *pat, u32 *out) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        out[i] = (u32)((int)(w << (31 - (sh + i))) >> 31);
        if (pat) out[i] ^= pat[i];
    }
}

// one butterfly of a group of planes [c0, c0 + N/4 chunks): FWD: u += w v,
// v += u; inverse: v += u, u += w v.  mul(v, p): p = w v
template <int N, bool FWD, class Mul>
SL_HD void bfly_planes(uint4 *tile, u32 su, u32 sv, u32 c0, const Mul &mul) {
    u32 u[N], v[N], p[N];
    load_planes<N>(tile, sv, c0, v);
    load_planes<N>(tile, su, c0, u);
    if (FWD) {
        mul(v, p);
#pragma unroll
        for (int i = 0; i < N; i++) { u[i] ^= p[i]; v[i] ^= u[i]; }
    } else {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] ^= u[i];
        mul(v, p);
#pragma unroll
        for (int i = 0; i < N; i++) u[i] ^= p[i];
    }
    store_planes<N>(tile, sv, c0, v);
    store_planes<N>(tile, su, c0, u);
}

// the butterfly of one slice pair over `NQ` quarters (16 planes each) from
// quarter q0; nb = m - 1 - L bits of t decide the subfield
template <int NQ, bool FWD>
SL_HD void bfly_pair(uint4 *tile, u32 su, u32 sv, u32 q0, int nb, u32 w, const u32 *pat) {
    if (nb == 0) {                              // W[0] = 0
        for (int q = 0; q < NQ; q++)
            bfly_planes<16, FWD>(tile, su, sv, 4 * (q0 + q), [](const u32 *, u32 *p) {
#pragma unroll
                for (int i = 0; i < 16; i++) p[i] = 0;
            });
    } else if (nb <= 7) {
        u32 wm[8];
        masks_of<8>(w, 0, pat, wm);
#pragma unroll 1
        for (int q = 0; q < 2 * NQ; q += 2)
            bfly_planes<16, FWD>(tile, su, sv, 4 * q0 + 2 * q, [&](const u32 *v, u32 *p) {
                t_mul<8>(v, wm, p);
                t_mul<8>(v + 8, wm, p + 8);
            });
    } else if (nb <= 15) {
        u32 wm[16];
        masks_of<16>(w, 0, pat, wm);
#pragma unroll 1
        for (int q = 0; q < NQ; q++)
            bfly_planes<16, FWD>(tile, su, sv, 4 * (q0 + q),
                                 [&](const u32 *v, u32 *p) { t_mul<16>(v, wm, p); });
    } else if constexpr (NQ >= 2) {             // m > 16: two quarters a thread
        // w = w0 + w1 X with w1 in GF(2^8); (v0 + v1 X)(w0 + w1 X), X^2 = X + v_15
        u32 w0[16], ws[16], w1[8];
        masks_of<16>(w, 0, pat, w0);
        masks_of<8>(w, 16, nullptr, w1);
#pragma unroll
        for (int i = 0; i < 16; i++) ws[i] = i < 8 ? w0[i] ^ w1[i] : w0[i];
#pragma unroll 1
        for (int q = 0; q < NQ; q += 2)
            bfly_planes<32, FWD>(tile, su, sv, 4 * (q0 + q), [&](const u32 *v, u32 *p) {
                u32 a[16], b[16];
                t_mul<8>(v + 16, w1, a);
                t_mul<8>(v + 24, w1, a + 8);
                t_delta<16>(a, p);
                t_mul<16>(v, w0, a);
#pragma unroll
                for (int i = 0; i < 16; i++) { p[i] ^= a[i]; b[i] = v[i] ^ v[16 + i]; }
                t_mul<16>(b, ws, p + 16);
#pragma unroll
                for (int i = 0; i < 16; i++) p[16 + i] ^= a[i];
            });
    }
}

// geometry of a butterfly pass's tile: 2^rlog rows of 2^clog consecutive
// slices, rows 2^(llo - 5) slices apart (levels llo .. llo + rlog - 1)
struct Tile {
    int m, rlog, clog, llo;
    u32 base;                   // global slice number of row 0, column 0
};
SL_HD u32 tile_gslice(const Tile &T, u32 s) {
    return T.base + ((s >> T.clog) << (T.llo - 5)) + (s & ((1u << T.clog) - 1));
}

// level L >= 5 of the tile (slices hold 32 consecutive elements)
template <int NQ, bool FWD>
SL_HD void level_n(uint4 *tile, const Tile &T, int L, u32 tid, u32 nt) {
    const int lg = L - T.llo + T.clog;
    const u32 pairs = 1u << (T.rlog + T.clog - 1);
    const int pl = T.rlog + T.clog - 1;
    for (u32 i = tid; i < pairs * (4 / NQ); i += nt) {
        const u32 g = i & (pairs - 1), q0 = (i >> pl) * NQ;
        const u32 su = ((g >> lg) << (lg + 1)) | (g & ((1u << lg) - 1)), sv = su | (1u << lg);
        const u32 t = tile_gslice(T, su) >> (L - 4);
        bfly_pair<NQ, FWD>(tile, su, sv, q0, T.m - 1 - L, twiddle(t), nullptr);
    }
}

// level L <= 4 of a contiguous tile whose groups of 32 slices are transposed
// (slice s of a group holds the elements 32 b + s)
template <int NQ, bool FWD>
SL_HD void level_x(uint4 *tile, const Tile &T, int L, u32 tid, u32 nt) {
    const u32 pairs = 1u << (T.rlog + T.clog - 1);
    const int pl = T.rlog + T.clog - 1;
    for (u32 i = tid; i < pairs * (4 / NQ); i += nt) {
        const u32 g = i & (pairs - 1), q0 = (i >> pl) * NQ;
        const u32 su = ((g >> L) << (L + 1)) | (g & ((1u << L) - 1)), sv = su | (1u << L);
        const u32 G = (T.base + su) >> 5, s = su & 31;
        const u32 t = (G << (9 - L)) | (s >> (L + 1));
        bfly_pair<NQ, FWD>(tile, su, sv, q0, T.m - 1 - L, twiddle(t), PATTAB.v[L]);
    }
}

// elements of each group of 32 slices transposed (32 b + s <-> 32 s + b)
SL_HD void transpose_groups(uint4 *tile, u32 nslices, u32 tid, u32 nt) {
    u32 *w = reinterpret_cast<u32 *>(tile);
    for (u32 i = tid; i < nslices * 2; i += nt) {
        const u32 g = (i >> 6) << 5, p = i & 63;
        u32 x[32];
#pragma unroll
        for (int s = 0; s < 32; s++) x[s] = w[word_at(g + s, p)];
        transpose32(x);
#pragma unroll
        for (int s = 0; s < 32; s++) w[word_at(g + s, p)] = x[s];
    }
}

// 32 chunk planes -> 64 tower planes, and 64 tower -> 64 polynomial planes
SL_HD void phi_in(uint4 *tile, u32 nslices, u32 tid, u32 nt) {
    for (u32 s = tid; s < nslices; s += nt) {
        u32 a[32], b[64];
        load_planes<32>(tile, s, 0, a);
        lin_map<32, 64, true>(a, b);
        store_planes<64>(tile, s, 0, b);
    }
}
SL_HD void phi_out(uint4 *tile, u32 nslices, u32 tid, u32 nt) {
    for (u32 s = tid; s < nslices; s += nt) {
        u32 a[64], b[64];
        load_planes<64>(tile, s, 0, a);
        lin_map<64, 64, false>(a, b);
        store_planes<64>(tile, s, 0, b);
    }
}
SL_HD void mul_slices(uint4 *fa, const uint4 *fb, u32 nslices, u32 tid, u32 nt) {
    for (u32 s = tid; s < nslices; s += nt) {
        u32 a[64], b[64], c[64];
        load_planes<64>(fa, s, 0, a);
        load_planes<64>(fb, s, 0, b);
        t_mul<64>(a, b, c);
        store_planes<64>(fa, s, 0, c);
    }
}

// ------------------------------------------------- Taylor levels
// Conversion of 2^k coefficients (index bits [0, k), k <= 16) by levels at
// x^(2^h) + x: level (M, a) acts on blocks of 2^M coefficients in chunks of
// 2^a (forward: Hi[0..c) ^= Top, then A[c..) ^= Hi; the inverse in reverse).
// Levels with chunks of 256 coefficients and more, and those of a conversion
// split at 2^8 (M > 8), work on whole words in shared memory; the 8-bit
// conversions of each 256 consecutive coefficients run in 8 registers.
constexpr int MAX_LV = 32;
struct Levels {
    int n;
    signed char M[MAX_LV], a[MAX_LV];
};
inline void add_levels(Levels &lv, int lo, int hi) {
    const int m = hi - lo;
    if (m <= 1) return;
    int h = 1;
    while (2 * h < m) h *= 2;
    for (int M = m; M > h; M--) {
        lv.M[lv.n] = (signed char)(lo + M);
        lv.a[lv.n++] = (signed char)(lo + M - 1 - h);
    }
    add_levels(lv, lo + h, hi);
    if (hi > 8 && lo == 0 && h == 8) return;     // [0, 8) in registers
    add_levels(lv, lo, lo + h);
}

// one level on 8 words (256 coefficients), M <= 8
template <int M, int A, bool FWD> SL_HD void reg_level(u32 *x) {
    constexpr int c = 1 << A;
    if constexpr (M <= 5) {
        constexpr int half = 1 << (M - 1);
        constexpr u32 lowc = (1u << c) - 1;
        u32 lm = 0, cm = 0;                      // low halves, and their low chunks
        for (int b = 0; b < 32; b += 2 * half) {
            lm |= (u32)((1ull << half) - 1) << b;
            cm |= lowc << b;
        }
#pragma unroll
        for (int j = 0; j < 8; j++) {
            u32 h = (x[j] >> half) & lm, l = x[j] & lm;
            if (FWD) h ^= (h >> (half - c)) & cm;
            l ^= (h << c) & lm;
            if (!FWD) h ^= (h >> (half - c)) & cm;
            x[j] = l | (h << half);
        }
    } else {
        constexpr int hw = 1 << (M - 6);         // words of a half
#pragma unroll
        for (int b = 0; b < 8; b += 2 * hw) {
            u32 *a = x + b, *h = x + b + hw;
            if constexpr (A >= 5) {
                constexpr int cw = c / 32;
                if (FWD)
#pragma unroll
                    for (int j = 0; j < cw; j++) h[j] ^= h[hw - cw + j];
#pragma unroll
                for (int j = cw; j < hw; j++) a[j] ^= h[j - cw];
                if (!FWD)
#pragma unroll
                    for (int j = 0; j < cw; j++) h[j] ^= h[hw - cw + j];
            } else {
                if (FWD) h[0] ^= h[hw - 1] >> (32 - c);
#pragma unroll
                for (int j = hw - 1; j >= 0; j--)
                    a[j] ^= (h[j] << c) | (j ? h[j - 1] >> (32 - c) : 0);
                if (!FWD) h[0] ^= h[hw - 1] >> (32 - c);
            }
        }
    }
}
template <bool FWD> SL_HD void reg_taylor8(u32 *x) {
    if (FWD) {
        reg_level<8, 3, true>(x); reg_level<7, 2, true>(x); reg_level<6, 1, true>(x);
        reg_level<5, 0, true>(x);
        reg_level<8, 5, true>(x); reg_level<7, 4, true>(x);          // bits [4, 8)
        reg_level<8, 6, true>(x); reg_level<6, 4, true>(x);
        reg_level<4, 1, true>(x); reg_level<3, 0, true>(x);          // bits [0, 4)
        reg_level<4, 2, true>(x); reg_level<2, 0, true>(x);
    } else {
        reg_level<2, 0, false>(x); reg_level<4, 2, false>(x);
        reg_level<3, 0, false>(x); reg_level<4, 1, false>(x);
        reg_level<6, 4, false>(x); reg_level<8, 6, false>(x);
        reg_level<7, 4, false>(x); reg_level<8, 5, false>(x);
        reg_level<5, 0, false>(x); reg_level<6, 1, false>(x); reg_level<7, 2, false>(x);
        reg_level<8, 3, false>(x);
    }
}

// word j of plane p of a Taylor tile: at(j, p)
struct TaylorAddr {              // [word][2^plog planes]
    int plog;
    SL_HD u32 operator()(u32 j, u32 p) const { return (j << plog) + p; }
};
struct SliceAddr {               // a tile of slices
    int plog;
    SL_HD u32 operator()(u32 j, u32 p) const { return word_at(j, p); }
};

// level (M, a), M >= 9, of 2^k coefficients (2^(k-5) words) x 2^plog planes
template <bool FWD, class At>
SL_HD void taylor_level(u32 *sm, const At &at, int k, int M, int a, u32 tid, u32 nt) {
    const int hl = M - 6;                            // log2 words of a half
    const u32 hw = 1u << hl, np = 1u << at.plog;
    const u32 items = (1u << (k - 6)) << at.plog;
    for (u32 i = tid; i < items; i += nt) {
        const u32 p = i & (np - 1), g = i >> at.plog;
        const u32 j = g & (hw - 1), b = (g >> hl) << (hl + 1);
        const u32 ih = at(b + hw + j, p);
        u32 h = sm[ih];
        if (a >= 5) {
            const u32 cw = 1u << (a - 5);
            const u32 top = j < cw ? sm[at(b + hw + hw - cw + j, p)] : 0;
            if (FWD && j < cw) { h ^= top; sm[ih] = h; }
            if (j + cw < hw) sm[at(b + j + cw, p)] ^= h;
            if (!FWD && j < cw) sm[ih] = h ^ top;
        } else {
            // the top bits read from word j-1 are not the low bits word 0 changes
            const int c = 1 << a;
            const u32 prev = j ? sm[at(b + hw + j - 1, p)] : 0;
            const u32 top = j ? 0 : sm[at(b + 2 * hw - 1, p)] >> (32 - c);
            if (FWD && j == 0) { h ^= top; sm[ih] = h; }
            sm[at(b + j, p)] ^= (h << c) | (j ? prev >> (32 - c) : 0);
            if (!FWD && j == 0) sm[ih] = h ^ top;
        }
    }
}
template <bool FWD, class At>
SL_HD void taylor_regs(u32 *sm, const At &at, int k, u32 tid, u32 nt) {
    const u32 np = 1u << at.plog, items = (1u << (k - 8)) << at.plog;
    for (u32 i = tid; i < items; i += nt) {
        const u32 p = i & (np - 1), r = (i >> at.plog) << 3;
        u32 x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = sm[at(r + j, p)];
        reg_taylor8<FWD>(x);
#pragma unroll
        for (int j = 0; j < 8; j++) sm[at(r + j, p)] = x[j];
    }
}

// Levels of a conversion of 2^k > 2^16 coefficients above the split at 2^16:
// rows of 2^16 coefficients, a tile of 2^tlog words (columns) of every row
// with `halo` words to their left.  Row e with bit b set moves by 2^b
// coefficients into row e without it; what moves past a row's end is kept
// apart and folded once (x^65536 = y + x forward, the next row inverse).
struct HiGeom {
    int rlog;                    // rows 2^rlog, rlog = k - 16 (1 .. 8)
    int tlog, plog;              // words a tile, planes
    u32 halo;                    // words: at least 2^rlog - 1 coefficients
};
#ifdef __CUDACC__
__host__
#endif
SL_HD u32 hi_pitch(const HiGeom &G) { return (1u << G.tlog) + G.halo; }
SL_HD u32 hi_at(const HiGeom &G, u32 row, u32 col, u32 p) {
    return ((row * hi_pitch(G) + col) << G.plog) + p;
}
SL_HD void hi_shift(u32 *sm, const HiGeom &G, int b, u32 tid, u32 nt) {
    const u32 np = 1u << G.plog, W = hi_pitch(G);
    const u32 items = (W << (G.rlog - 1)) << G.plog;
    for (u32 i = tid; i < items; i += nt) {
        const u32 p = i & (np - 1), g = i >> G.plog, rr = g / W, col = g - rr * W;
        const u32 lo = ((rr >> b) << (b + 1)) | (rr & ((1u << b) - 1)), hi = lo | (1u << b);
        u32 v;
        if (b >= 5) {
            const u32 cw = 1u << (b - 5);
            if (col < cw) continue;
            v = sm[hi_at(G, hi, col - cw, p)];
        } else {
            const int c = 1 << b;
            v = sm[hi_at(G, hi, col, p)] << c;
            if (col) v |= sm[hi_at(G, hi, col - 1, p)] >> (32 - c);
        }
        sm[hi_at(G, lo, col, p)] ^= v;
    }
}
// level (M, a) of the conversion over the row index, columns from col0 on
template <bool FWD>
SL_HD void hi_rows(u32 *sm, const HiGeom &G, int M, int a, u32 col0, u32 tid, u32 nt) {
    const u32 np = 1u << G.plog, n = hi_pitch(G) - col0;
    const u32 half = 1u << (M - 1), c = 1u << a;
    const u32 items = (n << (G.rlog - 1)) << G.plog;
    for (u32 i = tid; i < items; i += nt) {
        const u32 p = i & (np - 1), g = i >> G.plog, rr = g / n, col = col0 + g - rr * n;
        const u32 j = rr & (half - 1), b = (rr >> (M - 1)) << M;
        const u32 ih = hi_at(G, b + half + j, col, p);
        u32 h = sm[ih];
        const u32 top = j < c ? sm[hi_at(G, b + 2 * half - c + j, col, p)] : 0;
        if (FWD && j < c) { h ^= top; sm[ih] = h; }
        if (j + c < half) sm[hi_at(G, b + j + c, col, p)] ^= h;
        if (!FWD && j < c) sm[ih] = h ^ top;
    }
}

// ------------------------------------------------- host-side pass planning
struct BflyPass { int llo, rlog, clog; };
struct Plan {
    int m = 0;
    int low = 0;                 // the last forward pass: levels low-1 .. 0
    int ntop = 0;
    BflyPass top[3];             // forward order
    Levels rows[9];              // rows[k-16]: conversions over k - 16 row bits
    Levels taylor[17];           // taylor[k]: smem levels of 2^k coefficients
};
constexpr int TILE_LOG = 9;      // at most 512 slices a tile
inline Plan make_plan(int m, int low, int clog) {
    Plan P;
    P.m = m;
    P.low = low < m ? low : m;
    int hi = m;
    int left = m - P.low;
    const int np = (left + TILE_LOG - 1) / TILE_LOG;
    for (int i = 0; i < np; i++) {
        const int take = (left + (np - i) - 1) / (np - i);
        hi -= take;
        left -= take;
        int c = clog;
        if (c > TILE_LOG - take) c = TILE_LOG - take;
        if (c > hi - 5) c = hi - 5;
        P.top[P.ntop++] = BflyPass{hi, take, c};
    }
    for (int k = 8; k <= 16; k++) {
        P.taylor[k].n = 0;
        if (k > 8) add_levels(P.taylor[k], 0, k);
    }
    for (int k = 0; k <= 8; k++) {
        P.rows[k].n = 0;
        add_levels(P.rows[k], 0, k);
    }
    return P;
}

// ------------------------------------------------- kernel bodies
// Each body is a sequence of steps ex([&](tid, nt) {...}) with a barrier
// after every step; `sm` is the block's shared memory.

// 32-bit chunks of an operand (chunk 0 XORed with xor0, zero from nchunks)
// into planes 0 .. 31 of the slices [s0, s0 + 2^nlog)
template <class Ex>
SL_HD void body_slice_in(Ex ex, u32 *sm, const u32 *src, u64 nchunks, u32 xor0, uint4 *f, u32 s0,
                         int nlog) {
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < (32u << nlog); i += nt) {
            const u64 k = (u64)s0 * 32 + i;
            u32 v = k < nchunks ? src[k] : 0;
            if (k == 0) v ^= xor0;
            sm[(i >> 5) * 33 + (i & 31)] = v;
        }
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 s = tid; s < (1u << nlog); s += nt) {
            u32 x[32];
#pragma unroll
            for (int j = 0; j < 32; j++) x[j] = sm[s * 33 + j];
            transpose32(x);
#pragma unroll
            for (int j = 0; j < 32; j++) sm[s * 33 + j] = x[j];
        }
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < (8u << nlog); i += nt) {
            const u32 *w = sm + (i >> 3) * 33 + 4 * (i & 7);
            uint4 q;
            q.x = w[0]; q.y = w[1]; q.z = w[2]; q.w = w[3];
            f[(u64)(s0 + (i >> 3)) * 16 + (i & 7)] = q;
        }
    });
}

// Taylor conversion of the 2^k coefficients from slice s0 on, planes
// [4 c0, 4 c0 + 2^plog), read at chunk offset c_src, written at chunk c0 of
// these slices and of `reps` - 1 copies rep_stride slices apart
template <bool FWD, class Ex>
SL_HD void body_taylor(Ex ex, u32 *sm, uint4 *f, u32 s0, int k, int plog, u32 c0, u32 c_src,
                       u32 reps, u32 rep_stride, const Levels &lv) {
    const TaylorAddr at{plog};
    const int cl = plog - 2;                         // log2 chunks a word
    const u32 items = 1u << (k - 5 + cl);
    uint4 *sm4 = reinterpret_cast<uint4 *>(sm);
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < items; i += nt)
            sm4[i] = f[(u64)(s0 + (i >> cl)) * 16 + c_src + (i & ((1u << cl) - 1))];
    });
    if (!FWD) ex([&](u32 tid, u32 nt) { taylor_regs<false>(sm, at, k, tid, nt); });
    for (int l = 0; l < lv.n; l++) {
        const int q = FWD ? l : lv.n - 1 - l;
        ex([&](u32 tid, u32 nt) { taylor_level<FWD>(sm, at, k, lv.M[q], lv.a[q], tid, nt); });
    }
    if (FWD) ex([&](u32 tid, u32 nt) { taylor_regs<true>(sm, at, k, tid, nt); });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < items; i += nt) {
            const uint4 q = sm4[i];
            for (u32 r = 0; r < reps; r++)
                f[(u64)(s0 + r * rep_stride + (i >> cl)) * 16 + c0 + (i & ((1u << cl) - 1))] = q;
        }
    });
}

// Taylor levels above 2^16 (HiGeom) of planes [4 c_src, ..) of `src` to
// chunk c_dst of `dst` (not the same chunks), column tile `ct`.  `side`
// holds the overflow of the first tile: 2^rlog rows x halo words x planes.
template <bool FWD, class Ex>
SL_HD void body_taylor_hi(Ex ex, u32 *sm, u32 *side, const uint4 *src, u32 c_src, uint4 *dst,
                          u32 c_dst, const HiGeom G, u32 ct, const Levels &rows) {
    const int cl = G.plog - 2;
    const u32 cm = (1u << cl) - 1, T = 1u << G.tlog, W = hi_pitch(G), R = 1u << G.rlog;
    uint4 *sm4 = reinterpret_cast<uint4 *>(sm);
    // col < halo: the words left of the tile; `tail`: those left of column 0
    // are the row's last words and the body is empty
    auto load = [&](bool tail) {
        ex([&](u32 tid, u32 nt) {
            for (u32 i = tid; i < ((R * W) << cl); i += nt) {
                const u32 c = i & cm, g = i >> cl, row = g / W, col = g - row * W;
                uint4 q;
                q.x = q.y = q.z = q.w = 0;
                const bool body = col >= G.halo;
                if (tail ? !body : (body || ct)) {
                    const u32 j = (ct * T + col - G.halo) & 2047;
                    q = src[(u64)(row * 2048 + j) * 16 + c_src + c];
                }
                sm4[i] = q;
            }
        });
    };
    auto shifts = [&]() {
        for (int l = 0; l < G.rlog; l++) {
            const int b = FWD ? G.rlog - 1 - l : l;
            ex([&](u32 tid, u32 nt) { hi_shift(sm, G, b, tid, nt); });
        }
    };
    auto inv_rows = [&]() {                       // before the shifts: the halo too
        if (FWD) return;
        for (int l = rows.n - 1; l >= 0; l--)
            ex([&](u32 tid, u32 nt) { hi_rows<false>(sm, G, rows.M[l], rows.a[l], 0, tid, nt); });
    };
    if (ct == 0) {
        load(true);
        inv_rows();
        shifts();
        ex([&](u32 tid, u32 nt) {
            const u32 n = (R * G.halo) << G.plog, np = 1u << G.plog;
            for (u32 i = tid; i < n; i += nt) {
                const u32 p = i & (np - 1), g = i >> G.plog, row = g / G.halo, q = g - row * G.halo;
                side[i] = sm[hi_at(G, row, G.halo + q, p)];
            }
        });
    }
    load(false);
    inv_rows();
    shifts();
    if (ct == 0) {
        ex([&](u32 tid, u32 nt) {
            const u32 n = (R * G.halo) << G.plog, np = 1u << G.plog;
            for (u32 i = tid; i < n; i += nt) {
                const u32 p = i & (np - 1), g = i >> G.plog, row = g / G.halo, q = g - row * G.halo;
                u32 v = 0;
                if (row) v = side[i - (G.halo << G.plog)];           // y, or the next row
                if (FWD) {                                           // and x
                    v ^= side[i] << 1;
                    if (q) v ^= side[i - np] >> 31;
                }
                sm[hi_at(G, row, G.halo + q, p)] ^= v;
            }
        });
    }
    if (FWD)
        for (int l = 0; l < rows.n; l++)
            ex([&](u32 tid, u32 nt) { hi_rows<true>(sm, G, rows.M[l], rows.a[l], G.halo, tid, nt); });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < ((R << G.tlog) << cl); i += nt) {
            const u32 c = i & cm, g = i >> cl, row = g >> G.tlog, col = g & (T - 1);
            dst[(u64)(row * 2048 + ct * T + col) * 16 + c_dst + c] =
                sm4[((row * W + G.halo + col) << cl) + c];
        }
    });
}

// one butterfly pass over a tile; FIRST (forward): planes 0..31 are chunk
// planes; LOWP: the pass that holds levels 4..0; LAST (inverse): back to
// polynomial planes.  Forward levels hi-1 .. lo, inverse lo .. hi-1, those
// at or above `top` (copies made by the Taylor step) left out.
template <int NQ, bool FWD, class Ex>
SL_HD void body_bfly(Ex ex, uint4 *tile, uint4 *f, const Tile T, int top, bool edge, bool lowp) {
    const u32 ns = 1u << (T.rlog + T.clog);
    const int hi = T.llo + T.rlog;
    const bool first = FWD && edge;
    ex([&](u32 tid, u32 nt) {
        const u32 n = ns * (first ? 8 : 16);
        for (u32 i = tid; i < n; i += nt) {
            const u32 s = first ? i >> 3 : i >> 4, c = first ? i & 7 : i & 15;
            tile[chunk_at(s, c)] = f[(u64)tile_gslice(T, s) * 16 + c];
        }
    });
    if (FWD) {
        if (first) ex([&](u32 tid, u32 nt) { phi_in(tile, ns, tid, nt); });
        for (int L = (hi < top ? hi : top) - 1; L >= T.llo; L--)
            ex([&](u32 tid, u32 nt) { level_n<NQ, true>(tile, T, L, tid, nt); });
        if (lowp) {
            ex([&](u32 tid, u32 nt) { transpose_groups(tile, ns, tid, nt); });
            for (int L = 4; L >= 0; L--)
                ex([&](u32 tid, u32 nt) { level_x<NQ, true>(tile, T, L, tid, nt); });
        }
    } else {
        if (lowp) {
            for (int L = 0; L <= 4; L++)
                ex([&](u32 tid, u32 nt) { level_x<NQ, false>(tile, T, L, tid, nt); });
            ex([&](u32 tid, u32 nt) { transpose_groups(tile, ns, tid, nt); });
        }
        for (int L = T.llo; L < hi; L++)
            ex([&](u32 tid, u32 nt) { level_n<NQ, false>(tile, T, L, tid, nt); });
        if (edge) ex([&](u32 tid, u32 nt) { phi_out(tile, ns, tid, nt); });
    }
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < ns * 16; i += nt)
            f[(u64)tile_gslice(T, i >> 4) * 16 + (i & 15)] = tile[chunk_at(i >> 4, i & 15)];
    });
}

// planes of slice s to its 32 output words (in chunks 0 .. 7): word e is the
// low half of coefficient e and the high half of coefficient e - 1, the last
// high half goes to side[s + 1]
SL_HD void slice_words(uint4 *tile, u32 *side, u32 s) {
    u32 lo[32], hi[32];
    load_planes<32>(tile, s, 0, lo);
    load_planes<32>(tile, s, 8, hi);
    transpose32(lo);
    transpose32(hi);
#pragma unroll
    for (int e = 31; e > 0; e--) lo[e] ^= hi[e - 1];
    store_planes<32>(tile, s, 0, lo);
    side[s + 1] = hi[31];
}

// 32-bit words 32 s0 .. of the overlap-add of the polynomial planes of a
// transform of nsl slices (64-bit coefficients at 32-bit steps); words from
// `words` on are not written.  side: 2^nlog + 1 words.
template <class Ex>
SL_HD void body_slice_out(Ex ex, uint4 *tile, u32 *side, const uint4 *f, u32 nsl, u32 *out,
                          u64 words, u32 s0, int nlog) {
    const u32 n = 1u << nlog;
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < n * 16; i += nt) {
            const u32 s = i >> 4;
            uint4 q;
            q.x = q.y = q.z = q.w = 0;
            if (s0 + s < nsl) q = f[(u64)(s0 + s) * 16 + (i & 15)];
            tile[chunk_at(s, i & 15)] = q;
        }
        if (tid == 0) {                          // high half of the coefficient before
            u32 v = 0;
            if (s0 && s0 - 1 < nsl) {
                const u32 *w = reinterpret_cast<const u32 *>(f + (u64)(s0 - 1) * 16) + 32;
                for (int p = 0; p < 32; p++) v |= (w[p] >> 31) << p;
            }
            side[0] = v;
        }
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 s = tid; s < n; s += nt) slice_words(tile, side, s);
    });
    ex([&](u32 tid, u32 nt) {
        const u32 *w = reinterpret_cast<const u32 *>(tile);
        for (u32 i = tid; i < 32 * n; i += nt) {
            const u64 k = (u64)s0 * 32 + i;
            if (k < words) out[k] = w[word_at(i >> 5, i & 31)] ^ ((i & 31) ? 0 : side[i >> 5]);
        }
    });
}

// a whole product of at most 2^m coefficients in one block (m <= SMALL_M)
constexpr int SMALL_M = 12;
struct Operand { const u32 *src; u64 nchunks; u32 xor0; };
template <class Ex>
SL_HD void body_small(Ex ex, uint4 *ta, uint4 *tb, u32 *side, int m, const Operand A,
                      const Operand B, int ka, int kb, const Levels &la, const Levels &lb,
                      const Levels &lm, u32 *out, u64 words) {
    const u32 ns = 1u << (m - 5);
    const Tile T{m, m - 5, 0, 5, 0};
    const SliceAddr at{5};
    // chunk words to planes 0 .. 31
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < 32 * ns; i += nt) {
            u32 va = i < A.nchunks ? A.src[i] : 0, vb = i < B.nchunks ? B.src[i] : 0;
            if (i == 0) { va ^= A.xor0; vb ^= B.xor0; }
            reinterpret_cast<u32 *>(ta)[word_at(i >> 5, i & 31)] = va;
            reinterpret_cast<u32 *>(tb)[word_at(i >> 5, i & 31)] = vb;
        }
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < 2 * ns; i += nt) {
            uint4 *t = i < ns ? ta : tb;
            u32 x[32];
            load_planes<32>(t, i & (ns - 1), 0, x);
            transpose32(x);
            store_planes<32>(t, i & (ns - 1), 0, x);
        }
    });
    u32 *wa = reinterpret_cast<u32 *>(ta), *wb = reinterpret_cast<u32 *>(tb);
    for (int l = 0; l < la.n || l < lb.n; l++)
        ex([&](u32 tid, u32 nt) {
            if (l < la.n) taylor_level<true>(wa, at, ka, la.M[l], la.a[l], tid, nt);
            if (l < lb.n) taylor_level<true>(wb, at, kb, lb.M[l], lb.a[l], tid, nt);
        });
    ex([&](u32 tid, u32 nt) {
        taylor_regs<true>(wa, at, ka, tid, nt);
        taylor_regs<true>(wb, at, kb, tid, nt);
    });
    // copies of the converted slices (through planes 32 .. 63), tower planes
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < 16 * ns; i += nt) {
            const bool b = i >= 8 * ns;
            uint4 *t = b ? tb : ta;
            const u32 s = (i >> 3) & (ns - 1), c = i & 7;
            const u32 from = s & ((1u << ((b ? kb : ka) - 5)) - 1);
            t[chunk_at(s, 8 + c)] = t[chunk_at(from, c)];
        }
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < 2 * ns; i += nt) {
            uint4 *t = i < ns ? ta : tb;
            u32 a[32], b[64];
            load_planes<32>(t, i & (ns - 1), 8, a);
            lin_map<32, 64, true>(a, b);
            store_planes<64>(t, i & (ns - 1), 0, b);
        }
    });
    for (int L = m - 1; L >= 5; L--)
        ex([&](u32 tid, u32 nt) {
            if (L < ka) level_n<1, true>(ta, T, L, tid, nt);
            if (L < kb) level_n<1, true>(tb, T, L, tid, nt);
        });
    ex([&](u32 tid, u32 nt) {
        transpose_groups(ta, ns, tid, nt);
        transpose_groups(tb, ns, tid, nt);
    });
    for (int L = 4; L >= 0; L--)
        ex([&](u32 tid, u32 nt) {
            level_x<1, true>(ta, T, L, tid, nt);
            level_x<1, true>(tb, T, L, tid, nt);
        });
    ex([&](u32 tid, u32 nt) { mul_slices(ta, tb, ns, tid, nt); });
    for (int L = 0; L <= 4; L++)
        ex([&](u32 tid, u32 nt) { level_x<1, false>(ta, T, L, tid, nt); });
    ex([&](u32 tid, u32 nt) { transpose_groups(ta, ns, tid, nt); });
    for (int L = 5; L < m; L++)
        ex([&](u32 tid, u32 nt) { level_n<1, false>(ta, T, L, tid, nt); });
    ex([&](u32 tid, u32 nt) { phi_out(ta, ns, tid, nt); });
    const SliceAddr at6{6};
    ex([&](u32 tid, u32 nt) { taylor_regs<false>(wa, at6, m, tid, nt); });
    for (int l = lm.n - 1; l >= 0; l--)
        ex([&](u32 tid, u32 nt) { taylor_level<false>(wa, at6, m, lm.M[l], lm.a[l], tid, nt); });
    ex([&](u32 tid, u32 nt) {
        if (tid == 0) side[0] = 0;
        for (u32 s = tid; s < ns; s += nt) slice_words(ta, side, s);
    });
    ex([&](u32 tid, u32 nt) {
        for (u64 k = tid; k < words; k += nt) {
            const u32 s = (u32)(k >> 5);
            u32 v = 0;
            if (s < ns) v = wa[word_at(s, (u32)k & 31)];
            if (!(k & 31) && s <= ns) v ^= side[s];
            out[k] = v;
        }
    });
}

}  // namespace slice
