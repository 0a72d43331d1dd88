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
// x_k^2 = x_(k-1) x_k + 1 (Wiedemann's tower; coordinate i is the product of the x_k over the
// set bits k of i), in which the subfields GF(2^8), GF(2^16), GF(2^32) are the
// low 8, 16, 32 coordinates.  The twiddle of butterfly level L is a sum of the
// Cantor basis elements 1 .. m-1-L, which lie in those subfields, so a
// multiply splits into 8 / 4 / 2 independent subfield multiplies, each a tree
// of three-way products down to AND-XORs over planes: 60, 204 and ~590
// operations for 32 products, 15-37 a field product where a 64 x 64
// carry-less multiply by integer multiplies takes ~200.
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

// a register of a warp: on the host the 32 lanes' values, so that the
// warp-wide steps below also run there
#ifdef __CUDACC__
typedef u32 V;
SL_HD V lane_id() { return threadIdx.x & 31; }
SL_HD V shfl(V x, V lane) { return __shfl_sync(0xFFFFFFFFu, x, lane); }
SL_HD V below(V a, u32 b) { return a < b ? 0xFFFFFFFFu : 0u; }      // masks
template <class F> SL_HD V lane_load(const u32 *sm, const F &at) { return sm[at(lane_id())]; }
template <class F> SL_HD void lane_store(u32 *sm, const F &at, V x) { sm[at(lane_id())] = x; }
// keeps shuffles (and the registers of their results) from moving up past it
SL_HD void warp_fence() { __syncwarp(); }
template <class P, class F> SL_HD V lane_load_if(const u32 *sm, const P &p, const F &at) {
    return p(lane_id()) ? sm[at(lane_id())] : 0;
}
template <class P, class F> SL_HD void lane_store_if(u32 *sm, const P &p, const F &at, V x) {
    if (p(lane_id())) sm[at(lane_id())] = x;
}
#else
struct V {
    u32 l[32];
    V(u32 x = 0) { for (u32 &v : l) v = x; }
};
#define SL_OP(op)                                                          \
    inline V operator op(const V &a, const V &b) {                         \
        V r;                                                               \
        for (int i = 0; i < 32; i++) r.l[i] = a.l[i] op b.l[i];            \
        return r;                                                          \
    }
SL_OP(^) SL_OP(&) SL_OP(|) SL_OP(+) SL_OP(-)
#undef SL_OP
inline V &operator^=(V &a, const V &b) { return a = a ^ b; }
inline V operator~(const V &a) { return a ^ V(0xFFFFFFFFu); }
inline V operator<<(const V &a, int s) { V r; for (int i = 0; i < 32; i++) r.l[i] = a.l[i] << s; return r; }
inline V operator>>(const V &a, int s) { V r; for (int i = 0; i < 32; i++) r.l[i] = a.l[i] >> s; return r; }
inline V lane_id() { V r; for (int i = 0; i < 32; i++) r.l[i] = i; return r; }
inline V shfl(const V &x, const V &lane) { V r; for (int i = 0; i < 32; i++) r.l[i] = x.l[lane.l[i] & 31]; return r; }
inline V below(const V &a, u32 b) { V r; for (int i = 0; i < 32; i++) r.l[i] = a.l[i] < b ? ~0u : 0u; return r; }
template <class F> inline V lane_load(const u32 *sm, const F &at) { V r; for (int i = 0; i < 32; i++) r.l[i] = sm[at(i)]; return r; }
template <class F> inline void lane_store(u32 *sm, const F &at, const V &x) { for (int i = 0; i < 32; i++) sm[at(i)] = x.l[i]; }
inline void warp_fence() {}
template <class P, class F> inline V lane_load_if(const u32 *sm, const P &p, const F &at) { V r; for (int i = 0; i < 32; i++) if (p(i)) r.l[i] = sm[at(i)]; return r; }
template <class P, class F> inline void lane_store_if(u32 *sm, const P &p, const F &at, const V &x) { for (int i = 0; i < 32; i++) if (p(i)) sm[at(i)] = x.l[i]; }
#endif

// ------------------------------------------------- tower-field constants
constexpr u64 c_mulx(u64 a, int n) {             // a times GF(2^n)'s own generator
    if (n == 1) return a;
    const int h = n / 2;
    const u64 lo = a & ((1ull << h) - 1), hi = a >> h;
    return hi | ((lo ^ c_mulx(hi, h)) << h);
}
constexpr u64 c_mul(u64 a, u64 b, int n) {
    if (!a || !b) return 0;
    if (n == 1) return a & b;
    const int h = n / 2;
    const u64 m = (1ull << h) - 1;
    const u64 p0 = c_mul(a & m, b & m, h), p1 = c_mul(a >> h, b >> h, h),
              p2 = c_mul((a & m) ^ (a >> h), (b & m) ^ (b >> h), h);
    return (p0 ^ p1) | ((p2 ^ p0 ^ p1 ^ c_mulx(p1, h)) << h);
}
// image of x under an isomorphism from GF(2)[x]/(x^64 + x^4 + x^3 + x + 1):
// a root of the modulus in the tower field
constexpr u64 ROOT = 0x4d12d23e481d71ddull;

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
    0x1, 0x3, 0xe, 0xb, 0x62, 0xd5, 0x8c, 0xf0, 0x1450, 0x3ce3, 0xefe9, 0xb2c2, 0x2e06,
    0x5025, 0xcf80, 0xff1, 0x110ecfb, 0x330a54a, 0xee04fec, 0xbb0ec09, 0x6236b7ac,
    0xd56d18a7, 0x8c2888b8, 0xf0bff8be, 0x50c1afc9};

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
// c = X a, X the generator of GF(2^N) over its half (1 for N = 1)
template <int N> SL_HD void t_mulx(const u32 *a, u32 *c) {
    if constexpr (N == 1) {
        c[0] = a[0];
    } else {
        constexpr int H = N / 2;
        u32 t[H];
        t_mulx<H>(a + H, t);
#pragma unroll
        for (int i = 0; i < H; i++) { c[H + i] = a[i] ^ t[i]; c[i] = a[H + i]; }
    }
}
// A multiplier b prepared for products in GF(2^N).  With X^2 = t X + 1 over
// the half field, b = b0 + b1 X acts on (a0, a1) as the matrix [b0 b1; b1 b0 +
// t b1], equal on its second diagonal, so three half products by b0 + b1, b1
// and b1 + b0 + t b1 make one and all else is done to b once.  The leaves are
// GF(2^4) elements, each with the 9 sums of its bits that its 4 x 4 matrix
// holds (3^(log2 N - 2) leaves).
template <int N> struct Prep {
    Prep<N / 2> p0, p1, p2;
    SL_HD void set(const u32 *b) {
        constexpr int H = N / 2;
        u32 s[H], t[H];
        t_mulx<H>(b + H, t);
#pragma unroll
        for (int i = 0; i < H; i++) { s[i] = b[i] ^ b[H + i]; t[i] ^= s[i]; }
        p0.set(s);
        p1.set(b + H);
        p2.set(t);
    }
};
template <> struct Prep<4> {
    u32 b0, b1, b2, b3, b01, b23, e0, e1, e01;
    SL_HD void set(const u32 *b) {
        b0 = b[0]; b1 = b[1]; b2 = b[2]; b3 = b[3];
        b01 = b0 ^ b1; b23 = b2 ^ b3; e0 = b0 ^ b3; e1 = b1 ^ b23; e01 = b01 ^ b2;
    }
};
// c ^= a b: every AND joins an XOR, 16 three-input operations a leaf; 60 in
// GF(2^8), 204 in GF(2^16)
template <int N> SL_HD void t_addmul(const u32 *a, const Prep<N> &b, u32 *c) {
    if constexpr (N == 4) {
        c[0] ^= a[0] & b.b0; c[0] ^= a[1] & b.b1; c[0] ^= a[2] & b.b2; c[0] ^= a[3] & b.b3;
        c[1] ^= a[0] & b.b1; c[1] ^= a[1] & b.b01; c[1] ^= a[2] & b.b3; c[1] ^= a[3] & b.b23;
        c[2] ^= a[0] & b.b2; c[2] ^= a[1] & b.b3; c[2] ^= a[2] & b.e0; c[2] ^= a[3] & b.e1;
        c[3] ^= a[0] & b.b3; c[3] ^= a[1] & b.b23; c[3] ^= a[2] & b.e1; c[3] ^= a[3] & b.e01;
    } else {
        constexpr int H = N / 2;
        u32 p[H], s[H];
#pragma unroll
        for (int i = 0; i < H; i++) { p[i] = 0; s[i] = a[i] ^ a[H + i]; }
        t_addmul<H>(s, b.p1, p);
        t_addmul<H>(a, b.p0, c);
        t_addmul<H>(a + H, b.p2, c + H);
#pragma unroll
        for (int i = 0; i < H; i++) { c[i] ^= p[i]; c[H + i] ^= p[i]; }
    }
}

// the same for a multiplier used once: its sums are made on the way down, so
// that few of them are held at a time
template <int N> SL_HD void t_addmul_once(const u32 *a, const u32 *b, u32 *c) {
    if constexpr (N == 4) {
        Prep<4> w;
        w.set(b);
        t_addmul<4>(a, w, c);
    } else {
        constexpr int H = N / 2;
        u32 p[H], s[H], t[H];
#pragma unroll
        for (int i = 0; i < H; i++) { p[i] = 0; s[i] = a[i] ^ a[H + i]; }
        t_addmul_once<H>(s, b + H, p);
#pragma unroll
        for (int i = 0; i < H; i++) { c[i] ^= p[i]; c[H + i] ^= p[i]; s[i] = b[i] ^ b[H + i]; }
        t_addmul_once<H>(a, s, c);
        t_mulx<H>(b + H, t);
#pragma unroll
        for (int i = 0; i < H; i++) t[i] ^= s[i];
        t_addmul_once<H>(a + H, t, c + H);
    }
}

// ------------------------------------------------- linear maps on planes
// out[p] = XOR over i < NI of bit p of M[i], in[i]; four inputs at a time
// through their 16 XORs (outputs P0 .. P0 + NO - 1)
template <bool TO, int G, int P> struct Sel {
    static constexpr u64 at(int i) { return ((TO ? PHI.to[i] : PHI.from[i]) >> P) & 1; }
    static constexpr int v = (int)(at(G) | at(G + 1) << 1 | at(G + 2) << 2 | at(G + 3) << 3);
};
template <bool TO, int G, int P0, int... P>
SL_HD void lin_group(const u32 *in, u32 *out, std::integer_sequence<int, P...>) {
    u32 c[16];
    c[0] = 0;
#pragma unroll
    for (int k = 0; k < 4; k++)
#pragma unroll
        for (int v = 0; v < (1 << k); v++) c[(1 << k) + v] = c[v] ^ in[G + k];
    ((out[P] ^= c[Sel<TO, G, P0 + P>::v]), ...);
}
template <bool TO, int NO, int P0, int... G>
SL_HD void lin_groups(const u32 *in, u32 *out, std::integer_sequence<int, G...>) {
    (lin_group<TO, 4 * G, P0>(in, out, std::make_integer_sequence<int, NO>{}), ...);
}
template <int NI, int NO, bool TO, int P0 = 0> SL_HD void lin_map(const u32 *in, u32 *out) {
#pragma unroll
    for (int p = 0; p < NO; p++) out[p] = 0;
    lin_groups<TO, NO, P0>(in, out, std::make_integer_sequence<int, NI / 4>{});
}

SL_HD u32 byte_perm(u32 a, u32 b, u32 sel) {
#ifdef __CUDACC__
    return __byte_perm(a, b, sel);
#else
    const u64 v = a | (u64)b << 32;
    u32 r = 0;
    for (int i = 0; i < 4; i++) r |= (u32)((v >> (8 * ((sel >> (4 * i)) & 7))) & 255) << (8 * i);
    return r;
#endif
}
// 32 x 32 bit transposition in registers: bit i of x[j] <-> bit j of x[i]
SL_HD void transpose32(u32 *x) {
#pragma unroll
    for (int k = 0; k < 5; k++) {
        const int d = 16 >> k;
        const u32 m = d == 4 ? 0x0F0F0F0Fu : d == 2 ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int j = 0; j < 32; j++) {
            if (j & d) continue;
            const u32 a = x[j], b = x[j + d];
            if (d == 16) {
                x[j] = byte_perm(a, b, 0x5410);
                x[j + d] = byte_perm(a, b, 0x7632);
            } else if (d == 8) {
                x[j] = byte_perm(a, b, 0x6240);
                x[j + d] = byte_perm(a, b, 0x7351);
            } else {
                const u32 t = ((a >> d) ^ b) & m;
                x[j + d] = b ^ t;
                x[j] = a ^ (t << d);
            }
        }
    }
}

// ------------------------------------------------- shared-memory slices
// slices PITCH 16-byte chunks apart, an odd number, so that one chunk of 8
// consecutive slices is in 8 different banks and every access of a thread is a
// constant offset from its slice (an XOR swizzle without padding cost 24
// address operations for 16 planes of a butterfly; the three smallest
// butterfly distances conflict two ways here)
template <int PITCH> struct Slab {
    uint4 *t;
    SL_HD uint4 &chunk(u32 s, u32 c) const { return t[s * PITCH + c]; }
    SL_HD u32 &word(u32 s, u32 p) const { return reinterpret_cast<u32 *>(t)[s * (4 * PITCH) + p]; }
};
typedef Slab<17> Full;           // all 64 planes
typedef Slab<9> Half;            // planes 0 .. 31 or 32 .. 63
typedef Slab<5> Quarter;         // 16 planes

// 16 bytes to shared memory, asynchronously on the device
SL_HD void copy16(uint4 *dst, const uint4 *src) {
#ifdef __CUDACC__
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(
                     (u32)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
#else
    *dst = *src;
#endif
}
SL_HD void copy_wait() {
#ifdef __CUDACC__
    asm volatile("cp.async.wait_all;\n" ::: "memory");
#endif
}

// store(i, load(i)) for i < n, B loads in flight a thread before the first
// store (global loads are not moved over shared stores otherwise: one at a
// time, 11 of 17 us of a block of the levels above 2^16 were load latency)
template <int B, class T, class L, class S>
SL_HD void staged(u32 n, u32 tid, u32 nt, const L &load, const S &store) {
    for (u32 i0 = tid; i0 < n; i0 += B * nt) {
        T q[B];
#pragma unroll
        for (int k = 0; k < B; k++)
            if (i0 + k * nt < n) q[k] = load(i0 + k * nt);
#pragma unroll
        for (int k = 0; k < B; k++)
            if (i0 + k * nt < n) store(i0 + k * nt, q[k]);
    }
}

template <int N, class S> SL_HD void load_planes(const S &tile, u32 s, u32 c0, u32 *v) {
#pragma unroll
    for (int k = 0; k < N / 4; k++) {
        const uint4 q = tile.chunk(s, c0 + k);
        v[4 * k] = q.x; v[4 * k + 1] = q.y; v[4 * k + 2] = q.z; v[4 * k + 3] = q.w;
    }
}
template <int N, class S> SL_HD void store_planes(const S &tile, u32 s, u32 c0, const u32 *v) {
#pragma unroll
    for (int k = 0; k < N / 4; k++) {
        uint4 q;
        q.x = v[4 * k]; q.y = v[4 * k + 1]; q.z = v[4 * k + 2]; q.w = v[4 * k + 3];
        tile.chunk(s, c0 + k) = q;
    }
}

// ------------------------------------------------- butterflies
// all ones where the top bit of byte b of w is set (a permute that repeats it)
SL_HD u32 sign_byte(u32 w, int b) {
#ifdef __CUDACC__
    u32 r;
    asm("prmt.b32 %0, %1, 0, %2;" : "=r"(r) : "r"(w), "r"((8 + b) * 0x1111));
    return r;
#else
    return (u32)((int)(w << (24 - 8 * b)) >> 31);
#endif
}
// masks of the N bits of w from bit `sh` (all ones where set), XORed with the
// slice's pattern where its elements differ
template <int N> SL_HD void masks_of(u32 w, int sh, const u32 *pat, u32 *out) {
#pragma unroll
    for (int i = 0; i < N; i++) {
        const int b = sh + i;
        out[i] = sign_byte(w << (7 - (b & 7)), b >> 3);
        if (pat) out[i] ^= pat[i];
    }
}

// butterflies of the N planes from chunk c0: DIR 1 (forward): u += w v, v += u;
// 0 (inverse): v += u, u += w v; 2: by `fwd`, all ones forward, else zero (one
// copy of the code for both).  addmul(v, u): u += w v
template <int N, int DIR, class S, class Mul>
SL_HD void bfly_planes(const S &tile, u32 su, u32 sv, u32 c0, u32 fwd, const Mul &addmul) {
    u32 u[N], v[N];
    load_planes<N>(tile, sv, c0, v);
    load_planes<N>(tile, su, c0, u);
    if (DIR != 1) {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] ^= DIR ? u[i] & ~fwd : u[i];
        if (DIR == 0) store_planes<N>(tile, sv, c0, v);
    }
    addmul(v, u);
    if (DIR != 0) {
#pragma unroll
        for (int i = 0; i < N; i++) v[i] ^= DIR == 2 ? u[i] & fwd : u[i];
        store_planes<N>(tile, sv, c0, v);
    }
    store_planes<N>(tile, su, c0, u);
}

// the butterfly of one slice pair over `NQ` quarters (16 planes each) from
// quarter q0; nb = m - 1 - L, the number of Cantor basis elements the level's
// twiddles are sums of, decides the subfield
template <int NQ, int DIR, class S>
SL_HD void bfly_pair(const S &tile, u32 su, u32 sv, u32 q0, int nb, u32 w, const u32 *pat,
                     u32 fwd) {
    if (DIR != 2 && nb == 0) {                  // W[0] = 0
#pragma unroll 1
        for (int q = 0; q < NQ; q++)
            bfly_planes<16, DIR>(tile, su, sv, 4 * (q0 + q), fwd, [](const u32 *, u32 *) {});
    } else if (DIR != 2 && nb <= 7) {
        u32 wm[8];
        Prep<8> b;
        masks_of<8>(w, 0, pat, wm);
        b.set(wm);
#pragma unroll 1
        for (int q = 0; q < NQ; q++)
            bfly_planes<16, DIR>(tile, su, sv, 4 * (q0 + q), fwd, [&](const u32 *v, u32 *u) {
                t_addmul<8>(v, b, u);
                t_addmul<8>(v + 8, b, u + 8);
            });
    } else if (nb <= 15) {
        u32 wm[16];
        Prep<16> b;
        masks_of<16>(w, 0, pat, wm);
        b.set(wm);
#pragma unroll 1
        for (int q = 0; q < NQ; q++)
            bfly_planes<16, DIR>(tile, su, sv, 4 * (q0 + q), fwd,
                                 [&](const u32 *v, u32 *u) { t_addmul<16>(v, b, u); });
    } else if constexpr (NQ >= 2) {             // m > 16: two quarters at a time
        // w = w0 + w1 X, w1 = b / t with b in GF(2^8), the high byte of w, as
        // elements past 16 of the basis are b_i X / t + ...: the half product
        // by w1 is one by b of (v0 + v1) / t, 1 / t = X' + t' one tower below
        const u32 w1 = w >> 16;
        u32 x[16];
        Prep<16> a0, a2;
        Prep<8> a1;
        masks_of<16>(w ^ w1, 0, pat, x);
        a0.set(x);
        masks_of<16>(w ^ w1 ^ (w >> 24), 0, pat, x);          // t w1 = b
        a2.set(x);
        masks_of<8>(w, 24, nullptr, x);
        a1.set(x);
#pragma unroll 1
        for (int q = 0; q < NQ; q += 2)
            bfly_planes<32, DIR>(tile, su, sv, 4 * (q0 + q), fwd, [&](const u32 *v, u32 *u) {
                u32 z[16], y[16], p[16];
#pragma unroll
                for (int i = 0; i < 16; i++) { y[i] = v[i] ^ v[16 + i]; p[i] = 0; }
                t_mulx<8>(y, z);                          // y / t = (y1 + t' y0) + y0 X'
#pragma unroll
                for (int i = 0; i < 8; i++) { z[i] ^= y[8 + i]; z[8 + i] = y[i]; }
                t_addmul<8>(z, a1, p);
                t_addmul<8>(z + 8, a1, p + 8);
                t_addmul<16>(v, a0, u);
                t_addmul<16>(v + 16, a2, u + 16);
#pragma unroll
                for (int i = 0; i < 16; i++) { u[i] ^= p[i]; u[16 + i] ^= p[i]; }
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

// the same for twiddles in GF(2^8) and 8 planes from chunk c0
template <int DIR, class S>
SL_HD void bfly_pair8(const S &tile, u32 su, u32 sv, u32 c0, u32 w, const u32 *pat, u32 fwd) {
    u32 wm[8];
    Prep<8> b;
    masks_of<8>(w, 0, pat, wm);
    b.set(wm);
    bfly_planes<8, DIR>(tile, su, sv, c0, fwd,
                        [&](const u32 *v, u32 *u) { t_addmul<8>(v, b, u); });
}

// level L >= 5 of the tile (slices hold 32 consecutive elements) on its NT
// quarters, NQ of a slice pair a thread
template <int NT, int NQ, int DIR, class S>
SL_HD void level_n(const S &tile, const Tile &T, int L, u32 tid, u32 nt, u32 fwd = 0) {
    const int lg = L - T.llo + T.clog;
    const u32 pairs = 1u << (T.rlog + T.clog - 1);
    const int pl = T.rlog + T.clog - 1;
    if (DIR == 2 && T.m - 1 - L <= 7) {          // few slices: 8 planes a thread
        for (u32 i = tid; i < 2 * NT * pairs; i += nt) {
            const u32 g = i & (pairs - 1);
            const u32 su = ((g >> lg) << (lg + 1)) | (g & ((1u << lg) - 1));
            bfly_pair8<DIR>(tile, su, su | (1u << lg), 2 * (i >> pl),
                            twiddle(tile_gslice(T, su) >> (L - 4)), nullptr, fwd);
        }
        return;
    }
    for (u32 i = tid; i < pairs * (NT / NQ); i += nt) {
        const u32 g = i & (pairs - 1), q0 = (i >> pl) * NQ;
        const u32 su = ((g >> lg) << (lg + 1)) | (g & ((1u << lg) - 1)), sv = su | (1u << lg);
        const u32 t = tile_gslice(T, su) >> (L - 4);
        bfly_pair<NQ, DIR>(tile, su, sv, q0, T.m - 1 - L, twiddle(t), nullptr, fwd);
    }
}

// level L <= 4 of a contiguous tile whose groups of 32 slices are transposed
// (slice s of a group holds the elements 32 b + s)
template <int NT, int NQ, int DIR, class S>
SL_HD void level_x(const S &tile, const Tile &T, int L, u32 tid, u32 nt, u32 fwd = 0) {
    const u32 pairs = 1u << (T.rlog + T.clog - 1);
    const int pl = T.rlog + T.clog - 1;
    const auto pair_of = [&](u32 g, u32 &su, u32 &t) {
        su = ((g >> L) << (L + 1)) | (g & ((1u << L) - 1));
        const u32 G = (T.base + su) >> 5, s = su & 31;
        t = (G << (9 - L)) | (s >> (L + 1));
    };
    u32 su, t;
    if (DIR == 2 && T.m - 1 - L <= 7) {
        for (u32 i = tid; i < 2 * NT * pairs; i += nt) {
            pair_of(i & (pairs - 1), su, t);
            bfly_pair8<DIR>(tile, su, su | (1u << L), 2 * (i >> pl), twiddle(t), PATTAB.v[L], fwd);
        }
        return;
    }
    for (u32 i = tid; i < pairs * (NT / NQ); i += nt) {
        const u32 q0 = (i >> pl) * NQ;
        pair_of(i & (pairs - 1), su, t);
        const u32 sv = su | (1u << L);
        bfly_pair<NQ, DIR>(tile, su, sv, q0, T.m - 1 - L, twiddle(t), PATTAB.v[L], fwd);
    }
}

// elements of each group of 32 slices transposed (32 b + s <-> 32 s + b),
// 16 NT planes
template <int NT, class S>
SL_HD void transpose_groups(const S &tile, u32 nslices, u32 tid, u32 nt) {
    for (u32 i = tid; i < nslices / 2 * NT; i += nt) {
        const u32 g = i / (16 * NT) << 5, p = i & (16 * NT - 1);
        u32 x[32];
#pragma unroll
        for (int s = 0; s < 32; s++) x[s] = tile.word(g + s, p);
        transpose32(x);
#pragma unroll
        for (int s = 0; s < 32; s++) tile.word(g + s, p) = x[s];
    }
}

// 32 chunk planes -> tower planes 32 H .. 32 H + 31, in place
template <int H> SL_HD void phi_in(const Half &tile, u32 nslices, u32 tid, u32 nt) {
    for (u32 s = tid; s < nslices; s += nt) {
        u32 a[32], b[32];
        load_planes<32>(tile, s, 0, a);
        lin_map<32, 32, true, 32 * H>(a, b);
        store_planes<32>(tile, s, 0, b);
    }
}
template <class S> SL_HD void phi_quarter(const S &dst, u32 s, u32 q, const u32 *a) {
    u32 b[16];
    switch (q) {
    case 0: lin_map<32, 16, true, 0>(a, b); break;
    case 1: lin_map<32, 16, true, 16>(a, b); break;
    case 2: lin_map<32, 16, true, 32>(a, b); break;
    default: lin_map<32, 16, true, 48>(a, b); break;
    }
    store_planes<16>(dst, s, 0, b);
}
SL_HD void mul_slices(const Full &fa, const Full &fb, u32 nslices, u32 tid, u32 nt) {
    for (u32 s = tid; s < nslices; s += nt) {
        u32 a[64], b[64], c[64];
        load_planes<64>(fa, s, 0, a);
        load_planes<64>(fb, s, 0, b);
#pragma unroll
        for (int i = 0; i < 64; i++) c[i] = 0;
        t_addmul_once<64>(a, b, c);
        store_planes<64>(fa, s, 0, c);
    }
}

// ------------------------------------------------- Taylor levels
// Conversion of 2^k coefficients (index bits [0, k), k <= 16) by levels at
// x^(2^h) + x: level (M, a) acts on blocks of 2^M coefficients in chunks of
// 2^a (forward: Hi[0..c) ^= Top, then A[c..) ^= Hi; the inverse in reverse).
// A conversion of m bits, h the largest power of two below m, is the levels
// (M, M - 1 - h), M = m .. h + 1, and the conversions of the upper m - h and
// the lower h bits.  The 8-bit conversions of each 256 consecutive
// coefficients run in 8 registers of a thread, the levels above them in the
// registers of a warp.
// one level inside a word, M <= 5: shifting right by half - c takes the top
// chunk to the lowest of the high half and the high half onto the low one
template <int M, int A, bool FWD, class V> SL_HD V word_level(V x) {
    constexpr int half = 1 << (M - 1), c = 1 << A;
    constexpr u32 lowc = (1u << c) - 1, halfm = (u32)((1ull << half) - 1);
    constexpr u32 ones = (u32)(0xFFFFFFFFull / ((1ull << (2 * half)) - 1));     // one a block
    constexpr u32 to_a = ones * (halfm & ~lowc), to_h = (ones * lowc) << half;
    if (!FWD) return x ^ ((x >> (half - c)) & (to_a | to_h));
    x = x ^ ((x >> (half - c)) & to_h);
    return x ^ ((x >> (half - c)) & to_a);
}
// one level on 8 words (256 coefficients), M <= 8
template <int M, int A, bool FWD> SL_HD void reg_level(u32 *x) {
    constexpr int c = 1 << A;
    if constexpr (M <= 5) {
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = word_level<M, A, FWD>(x[j]);
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

// the 8-bit conversions of 2^k coefficients; word j of plane p is at(j, p)
template <bool FWD, class At>
SL_HD void taylor_regs(u32 *sm, const At &at, int k, u32 tid, u32 nt) {
    const u32 nr = 1u << (k - 8), items = nr << at.plog;
    for (u32 i = tid; i < items; i += nt) {
        const u32 p = At::rows_first ? i >> (k - 8) : i & ((1u << at.plog) - 1);
        const u32 r = (At::rows_first ? i & (nr - 1) : i >> at.plog) << 3;
        u32 x[8];
#pragma unroll
        for (int j = 0; j < 8; j++) x[j] = sm[at(r + j, p)];
        reg_taylor8<FWD>(x);
#pragma unroll
        for (int j = 0; j < 8; j++) sm[at(r + j, p)] = x[j];
    }
}

// The same conversions in the registers of one warp, a plane each: word
// r * 32 + lane of 2^k coefficients in x[r] (k >= 10).  Words half a block
// apart are registers or lanes; a shift by less than 32 words takes the lane
// below's word by shuffle.  (In shared memory a level costs three accesses
// and a dozen address instructions a word: 2^16 coefficients of 32 planes of
// two operands took 328 us at 2^23 coefficients.)
template <int M, int A, bool FWD, int NR> SL_HD void warp_level(V (&x)[NR]) {
    const V lane = lane_id();
    constexpr int hw = M >= 6 ? 1 << (M - 6) : 0;          // words of a half
    constexpr int c = 1 << A, cw = c / 32;
    if constexpr (M <= 5) {
#pragma unroll
        for (int r = 0; r < NR; r++) x[r] = word_level<M, A, FWD>(x[r]);
    } else if constexpr (hw >= 32) {
        constexpr int hr = hw / 32;
#pragma unroll
        for (int b = 0; b < NR; b += 2 * hr) {
            V *a = x + b, *h = x + b + hr;
            if constexpr (cw >= 32) {
                constexpr int cr = cw / 32;
                if (FWD)
#pragma unroll
                    for (int j = 0; j < cr; j++) h[j] ^= h[hr - cr + j];
#pragma unroll
                for (int j = cr; j < hr; j++) a[j] ^= h[j - cr];
                if (!FWD)
#pragma unroll
                    for (int j = 0; j < cr; j++) h[j] ^= h[hr - cr + j];
            } else if constexpr (cw >= 1) {
                const V from = (lane - V(cw)) & V(31), low = below(lane, cw);
                if (FWD) h[0] ^= shfl(h[hr - 1], from) & low;
                V prev = V(0);
#pragma unroll
                for (int j = 0; j < hr; j++) {
                    const V t = shfl(h[j], from);
                    a[j] ^= (prev & low) | (t & ~low);
                    prev = t;
                }
                if (!FWD) h[0] ^= prev & low;
            } else {
                // the low c bits that the top chunk changes in word 0 are not
                // among the top ones the next word takes from it
                const V from = (lane - V(1)) & V(31), low = below(lane, 1);
                V prev = V(0);
                if (FWD) h[0] ^= (shfl(h[hr - 1], from) >> (32 - c)) & low;
#pragma unroll
                for (int j = 0; j < hr; j++) {
                    const V t = shfl(h[j], from), p = (prev & low) | (t & ~low);
                    a[j] ^= (h[j] << c) | (p >> (32 - c));
                    prev = t;
                }
                if (!FWD) h[0] ^= (prev >> (32 - c)) & low;
            }
        }
    } else {
        const V j = lane & V(hw - 1), lo = below(lane & V(hw), 1), hi = ~lo;
        if constexpr (cw >= 1) {
            const V from = (lane + V(hw - cw)) & V(31);
            const V top = hi & below(j, cw), to_a = lo & ~below(j, cw);
#pragma unroll
            for (int r = 0; r < NR; r++) {
                if (FWD) {
                    x[r] ^= shfl(x[r], from) & top;
                    x[r] ^= shfl(x[r], from) & to_a;
                } else {
                    x[r] ^= shfl(x[r], from) & (top | to_a);
                }
            }
        } else {
            const V from = (lane + V(hw)) & V(31), prev = (lane + V(hw - 1)) & V(31);
            const V first = below(j, 1), top = hi & first, to_a = lo & ~first;
#pragma unroll
            for (int r = 0; r < NR; r++) {
                const V p = shfl(x[r], prev) >> (32 - c);
                if (FWD) x[r] ^= p & top;
                const V h = shfl(x[r], from);
                x[r] ^= ((h << c) & lo) ^ (p & to_a);
                if (!FWD) x[r] ^= p & top;
            }
        }
    }
}

// the levels of a conversion over index bits [LO, HI) in forward or inverse
// order ([0, 8) of a split at 2^8 left out where Op::skip_low)
constexpr int split_of(int m) { int h = 1; while (2 * h < m) h *= 2; return h; }
template <bool FWD, int LO, int HI> struct Conv {
    static constexpr int m = HI - LO, h = split_of(m);
    template <class Op, int... I>
    static SL_HD void own(const Op &op, std::integer_sequence<int, I...>) {
        if (FWD) (op.template level<LO + m - I, LO + m - I - 1 - h>(), ...);
        else (op.template level<LO + h + 1 + I, LO + I>(), ...);
    }
    template <class Op> static SL_HD void lower(const Op &op) {
        if constexpr (!(LO == 0 && HI > 8 && h == 8 && Op::skip_low)) Conv<FWD, LO, LO + h>::run(op);
    }
    template <class Op> static SL_HD void run(const Op &op) {
        if constexpr (m > 1) {
            if constexpr (FWD) {
                own(op, std::make_integer_sequence<int, m - h>{});
                Conv<FWD, LO + h, HI>::run(op);
                lower(op);
            } else {
                lower(op);
                Conv<FWD, LO + h, HI>::run(op);
                own(op, std::make_integer_sequence<int, m - h>{});
            }
        }
    }
};
template <bool FWD, int NR> struct WarpLevels {
    static constexpr bool skip_low = true;
    V (&x)[NR];
    template <int M, int A> SL_HD void level() const { warp_level<M, A, FWD>(x); }
};

// a Taylor tile a plane after another: word j of plane p, swizzled so that
// 32 consecutive words, and word j of 32 consecutive groups of 8, are in
// different banks, and the stores of 16-byte chunks of 16 slices too
struct PlaneAddr {
    static constexpr bool rows_first = true;
    int plog, pitch;
    SL_HD u32 operator()(u32 j, u32 p) const { return p * pitch + (j ^ ((j >> 5) & 7)); }
};
template <int K, bool FWD, class At> SL_HD void taylor_warp(u32 *sm, const At &at, u32 p) {
    constexpr int NR = 1 << (K - 10);
    V x[NR];
#pragma unroll
    for (int r = 0; r < NR; r++)
        x[r] = lane_load(sm, [&](u32 l) { return at(r * 32 + l, p); });
    Conv<FWD, 0, K>::run(WarpLevels<FWD, NR>{x});
#pragma unroll
    for (int r = 0; r < NR; r++)
        lane_store(sm, [&](u32 l) { return at(r * 32 + l, p); }, x[r]);
}

// 32 elements (words lo, hi of each in order) to planes of the tower basis, and
// back
SL_HD void words_to_planes(const u32 *w, u32 *planes) {
    u32 a[64];
#pragma unroll
    for (int e = 0; e < 32; e++) { a[e] = w[2 * e]; a[32 + e] = w[2 * e + 1]; }
    transpose32(a);
    transpose32(a + 32);
    lin_map<64, 64, true>(a, planes);
}
SL_HD void planes_to_words(const u32 *planes, u32 *w) {
    u32 a[64];
    lin_map<64, 64, false>(planes, a);
    transpose32(a);
    transpose32(a + 32);
#pragma unroll
    for (int e = 0; e < 32; e++) { w[2 * e] = a[e]; w[2 * e + 1] = a[32 + e]; }
}

// ------------------------------------------------- host-side pass planning
struct BflyPass { int llo, rlog, clog; };
struct Plan {
    int m = 0;
    int low = 0;                 // the last forward pass: levels low-1 .. 0
    int ntop = 0;
    BflyPass top[3];             // forward order
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
    return P;
}

// ------------------------------------------------- kernel bodies
// Each body is a sequence of steps ex([&](tid, nt) {...}) with a barrier
// after every step; `sm` is the block's shared memory.

// 32-bit chunks of an operand of 64-bit words (chunk 0 XORed with xor0, zero from nchunks)
// into planes 0 .. 31 of the slices [s0, s0 + 2^nlog)
template <class Ex>
SL_HD void body_slice_in(Ex ex, u32 *sm, const u32 *src, u64 nchunks, u32 xor0, uint4 *f, u32 s0,
                         int nlog) {
    ex([&](u32 tid, u32 nt) {
        const u64 *src64 = reinterpret_cast<const u64 *>(src);
        staged<8, u64>(
            16u << nlog, tid, nt,
            [&](u32 i) {
                const u64 k = (u64)s0 * 32 + 2 * i;
                u64 v = k < nchunks ? src64[k >> 1] : 0;
                if (k + 1 == nchunks) v = (u32)v;
                return v;
            },
            [&](u32 i, u64 v) {
                if (i == 0 && s0 == 0) v ^= xor0;
                u32 *w = sm + (i >> 4) * 33 + 2 * (i & 15);
                w[0] = (u32)v;
                w[1] = (u32)(v >> 32);
            });
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

// Taylor conversion of the 2^K coefficients from slice s0 on, planes
// [4 c0, 4 c0 + 2^plog), read at chunk offset c_src, written at chunk c0 of
// these slices and of `reps` - 1 copies rep_stride slices apart
template <int K, bool FWD, class Ex>
SL_HD void body_taylor(Ex ex, u32 *sm, uint4 *f, u32 s0, int plog, u32 c0, u32 c_src, u32 reps,
                       u32 rep_stride) {
    const PlaneAddr at{plog, (1 << (K - 5)) + 4};
    const int cl = plog - 2;                         // log2 chunks a word
    const u32 items = 1u << (K - 5 + cl);
    ex([&](u32 tid, u32 nt) {
        staged<8, uint4>(
            items, tid, nt,
            [&](u32 i) {
                return f[(u64)(s0 + (i >> cl)) * 16 + c_src + (i & ((1u << cl) - 1))];
            },
            [&](u32 i, const uint4 &q) {
                const u32 j = i >> cl, c = i & ((1u << cl) - 1);
                sm[at(j, 4 * c)] = q.x;
                sm[at(j, 4 * c + 1)] = q.y;
                sm[at(j, 4 * c + 2)] = q.z;
                sm[at(j, 4 * c + 3)] = q.w;
            });
    });
    if (!FWD) ex([&](u32 tid, u32 nt) { taylor_regs<false>(sm, at, K, tid, nt); });
    ex.warps(1u << plog, [&](u32 p) { taylor_warp<K, FWD>(sm, at, p); });
    if (FWD) ex([&](u32 tid, u32 nt) { taylor_regs<true>(sm, at, K, tid, nt); });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < items; i += nt) {
            const u32 j = i >> cl, c = i & ((1u << cl) - 1);
            uint4 q;
            q.x = sm[at(j, 4 * c)];
            q.y = sm[at(j, 4 * c + 1)];
            q.z = sm[at(j, 4 * c + 2)];
            q.w = sm[at(j, 4 * c + 3)];
            for (u32 r = 0; r < reps; r++) f[(u64)(s0 + r * rep_stride + j) * 16 + c0 + c] = q;
        }
    });
}

// Taylor levels above 2^16: 2^RLOG rows of 2^16 coefficients.  Row e with bit
// b set moves by 2^b coefficients into row e without it; what moves past a
// row's end is kept apart and folded once (x^65536 = y + x forward, the next
// row inverse).  A warp holds one plane's rows in registers, 32 consecutive
// words in its lanes, the first HALO of them the words to the tile's left
// (at least 2^RLOG - 1 coefficients).
template <int RLOG> struct Hi {
    static constexpr int PLOG = RLOG >= 7 ? 2 : 3;         // planes a block: 4 of 128 rows
    static constexpr int CL = PLOG - 2;                    // log2 chunks a word
    static constexpr int R = 1 << RLOG, HALO = RLOG <= 5 ? 1 : 1 << (RLOG - 5), T = 32 - HALO;
    static constexpr int TILES = (2048 + T - 1) / T;
    static constexpr int PITCH = 36;             // words a row and plane
    static SL_HD u32 at(u32 row, u32 p, u32 col) { return ((row << PLOG) + p) * PITCH + col; }
    static constexpr int WORDS = (R << PLOG) * (PITCH + HALO);
};
template <bool FWD, int NR> struct RowLevels {
    static constexpr bool skip_low = false;
    V (&x)[NR];
    template <int M, int A> SL_HD void level() const {
        constexpr int half = 1 << (M - 1), c = 1 << A;
#pragma unroll
        for (int b = 0; b < NR; b += 2 * half) {
            V *a = x + b, *h = x + b + half;
            if (FWD)
#pragma unroll
                for (int j = 0; j < c; j++) h[j] ^= h[half - c + j];
#pragma unroll
            for (int j = c; j < half; j++) a[j] ^= h[j - c];
            if (!FWD)
#pragma unroll
                for (int j = 0; j < c; j++) h[j] ^= h[half - c + j];
        }
    }
};
template <int B, int NR> SL_HD void hi_shift(V (&x)[NR]) {
    const V lane = lane_id();
    const V from = (lane - V(B >= 5 ? 1 << (B >= 5 ? B - 5 : 0) : 1)) & V(31);
#pragma unroll
    for (int r = 0; r < NR; r++) {
        if (NR >= 128 && r % 16 == 0) warp_fence();
        if (r & (1 << B)) continue;
        const V h = x[r | (1 << B)], t = shfl(h, from);
        if constexpr (B >= 5) x[r] ^= t;
        else x[r] ^= (h << (1 << B)) | (t >> (32 - (1 << B)));
    }
}
template <bool FWD, int RLOG, int NR, int... I>
SL_HD void hi_shifts(V (&x)[NR], std::integer_sequence<int, I...>) {
    (hi_shift<FWD ? RLOG - 1 - I : I>(x), ...);
}

// planes [4 c_src, ..) of `src` to chunk c_dst of `dst` (not the same
// chunks), column tile ct; sm: Hi<RLOG>::WORDS
template <int RLOG, bool FWD, class Ex>
SL_HD void body_taylor_hi(Ex ex, u32 *sm, const uint4 *src, u32 c_src, uint4 *dst, u32 c_dst,
                          u32 ct) {
    typedef Hi<RLOG> H;
    constexpr int R = H::R, HALO = H::HALO, T = H::T, cl = H::CL, plog = H::PLOG;
    u32 *side = sm + (R << plog) * H::PITCH;     // overflow of the first tile
    // `tail`: the words left of column 0 are the row's last and the body is empty
    auto load = [&](bool tail) {
        ex([&](u32 tid, u32 nt) {
staged<8, uint4>(
                (u32)(R * 32) << cl, tid, nt,
                [&](u32 i) {
                    const u32 c = i & ((1u << cl) - 1), col = (i >> cl) & 31, row = i >> (cl + 5);
                    const u32 j = ct * T + col - HALO;
                    uint4 q;
                    q.x = q.y = q.z = q.w = 0;
                    if (tail ? col < HALO : (col >= HALO || ct) && (col < HALO || j < 2048))
                        q = src[(u64)(row * 2048 + (j & 2047)) * 16 + c_src + c];
                    return q;
                },
                [&](u32 i, const uint4 &q) {
                    const u32 c = i & ((1u << cl) - 1), col = (i >> cl) & 31, row = i >> (cl + 5);
                    sm[H::at(row, 4 * c, col)] = q.x;
                    sm[H::at(row, 4 * c + 1, col)] = q.y;
                    sm[H::at(row, 4 * c + 2, col)] = q.z;
                    sm[H::at(row, 4 * c + 3, col)] = q.w;
                });
        });
    };
    for (int run = ct == 0 ? 0 : 1; run < 2; run++) {
        const bool tail = run == 0;
        load(tail);
        ex.warps(1u << plog, [&](u32 p) {
            V x[R];
#pragma unroll
            for (int r = 0; r < R; r++)
                x[r] = lane_load(sm, [&](u32 l) { return H::at(r, p, l); });
            const auto over = [](u32 l) { return l >= (u32)H::HALO && l < 2u * H::HALO; };
            const V left = (lane_id() - V(1)) & V(31);
            if (!FWD) Conv<false, 0, RLOG>::run(RowLevels<false, R>{x});
            hi_shifts<FWD, RLOG>(x, std::make_integer_sequence<int, RLOG>{});
            if (tail) {
#pragma unroll
                for (int r = 0; r < R; r++)
                    lane_store_if(side, over, [&](u32 l) { return ((r << plog) + p) * HALO + l - HALO; },
                                  x[r]);
                return;
            }
            if (ct == 0) {
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const V o = lane_load_if(side, over, [&](u32 l) {
                        return ((r << plog) + p) * HALO + l - HALO;
                    });
                    if (r + 1 < R) x[r + 1] ^= o;                // y, or the next row
                    if (FWD) x[r] ^= (o << 1) | (shfl(o, left) >> 31);      // and x
                }
            }
            if (FWD) Conv<true, 0, RLOG>::run(RowLevels<true, R>{x});
#pragma unroll
            for (int r = 0; r < R; r++)
                lane_store(sm, [&](u32 l) { return H::at(r, p, l); }, x[r]);
        });
    }
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < ((u32)(R * 32) << cl); i += nt) {
            const u32 c = i & ((1u << cl) - 1), col = (i >> cl) & 31, row = i >> (cl + 5);
            const u32 j = ct * T + col - HALO;
            if (col < HALO || j >= 2048) continue;
            uint4 q;
            q.x = sm[H::at(row, 4 * c, col)];
            q.y = sm[H::at(row, 4 * c + 1, col)];
            q.z = sm[H::at(row, 4 * c + 2, col)];
            q.w = sm[H::at(row, 4 * c + 3, col)];
            dst[(u64)(row * 2048 + j) * 16 + c_dst + c] = q;
        }
    });
}

// one butterfly pass over half the planes of a tile (every twiddle product
// stays inside a half).  `first` (forward): planes 0 .. 31 are chunk planes,
// and both halves' blocks read them before either writes (ex.pair()); `lowp`:
// the pass that holds levels 4 .. 0.  Forward levels hi-1 .. lo, inverse lo ..
// hi-1, those at or above `top` (copies made by the Taylor step) left out.
template <int NQ, bool FWD, class Ex>
SL_HD void body_bfly(Ex ex, uint4 *sm, uint4 *f, const Tile T, u32 half, int top, bool first,
                     bool lowp) {
    const Half tile{sm};
    const u32 ns = 1u << (T.rlog + T.clog);
    const int hi = T.llo + T.rlog;
    ex([&](u32 tid, u32 nt) {
        const u32 c0 = first ? 0 : 8 * half;
        for (u32 i = tid; i < ns * 8; i += nt)
            copy16(&tile.chunk(i >> 3, i & 7), f + (u64)tile_gslice(T, i >> 3) * 16 + c0 + (i & 7));
        copy_wait();
    });
    if (FWD) {
        if (first) {
            ex.pair();
            ex([&](u32 tid, u32 nt) {
                if (half) phi_in<1>(tile, ns, tid, nt);
                else phi_in<0>(tile, ns, tid, nt);
            });
        }
        for (int L = (hi < top ? hi : top) - 1; L >= T.llo; L--)
            ex([&](u32 tid, u32 nt) { level_n<2, NQ, true>(tile, T, L, tid, nt); });
        if (lowp) {
            ex([&](u32 tid, u32 nt) { transpose_groups<2>(tile, ns, tid, nt); });
            for (int L = 4; L >= 0; L--)
                ex([&](u32 tid, u32 nt) { level_x<2, NQ, true>(tile, T, L, tid, nt); });
        }
    } else {
        if (lowp) {
            for (int L = 0; L <= 4; L++)
                ex([&](u32 tid, u32 nt) { level_x<2, NQ, false>(tile, T, L, tid, nt); });
            ex([&](u32 tid, u32 nt) { transpose_groups<2>(tile, ns, tid, nt); });
        }
        for (int L = T.llo; L < hi; L++)
            ex([&](u32 tid, u32 nt) { level_n<2, NQ, false>(tile, T, L, tid, nt); });
    }
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < ns * 8; i += nt)
            f[(u64)tile_gslice(T, i >> 3) * 16 + 8 * half + (i & 7)] = tile.chunk(i >> 3, i & 7);
    });
}

// tower planes of slice s to its 32 output words (in chunks 0 .. 7): word e is
// the low half of coefficient e and the high half of coefficient e - 1, the
// last high half goes to side[s + 1]
SL_HD void slice_words(const Full &tile, u32 *side, u32 s) {
    u32 a[64], b[64];
    load_planes<64>(tile, s, 0, a);
    lin_map<64, 64, false>(a, b);
    transpose32(b);
    transpose32(b + 32);
#pragma unroll
    for (int e = 31; e > 0; e--) b[e] ^= b[31 + e];
    store_planes<32>(tile, s, 0, b);
    side[s + 1] = b[63];
}

// 32-bit words 32 s0 .. of the overlap-add of a transform of nsl slices in
// tower planes (64-bit coefficients at 32-bit steps); words from `words` on
// are not written.  The block takes 2^nlog - 1 slices and the one before them
// for its last high half.  side: 2^nlog + 1 words.
template <class Ex>
SL_HD void body_slice_out(Ex ex, uint4 *sm, u32 *side, const uint4 *f, u32 nsl, u32 *out,
                          u64 words, u32 s0, int nlog) {
    const Full tile{sm};
    const u32 n = 1u << nlog;
    ex([&](u32 tid, u32 nt) {
        for (u32 i = tid; i < n * 16; i += nt) {
            const u32 s = s0 + (i >> 4) - 1;                 // the slice before s0 first
            if (s < nsl) {
                copy16(&tile.chunk(i >> 4, i & 15), f + (u64)s * 16 + (i & 15));
            } else {
                uint4 q;
                q.x = q.y = q.z = q.w = 0;
                tile.chunk(i >> 4, i & 15) = q;
            }
        }
        copy_wait();
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 s = tid; s < n; s += nt) slice_words(tile, side, s);
    });
    ex([&](u32 tid, u32 nt) {
        for (u32 i = 32 + tid; i < 32 * n; i += nt) {
            const u64 k = (u64)s0 * 32 + i - 32;
            if (k < words) out[k] = tile.word(i >> 5, i & 31) ^ ((i & 31) ? 0 : side[i >> 5]);
        }
    });
}

// Whole products of at most 2^m coefficients, 10 <= m <= 14, by a cluster of
// 8 blocks: block 4 o + q takes quarter q (16 planes) of operand o up to its
// transform (every twiddle is in GF(2^16) there, so quarters stay apart), the
// products are shared out by slices, blocks 0 .. 3 run the inverse of their
// quarters, and the slices are shared out again for the words.  ex.mem(r) is
// the shared memory of block r; ex.block(f) and ex.cluster(f) run f(rank, tid,
// threads) on every block, with a barrier of the block or the cluster after.
// (One block for a whole product took 72 us at m = 12, its levels bound by
// one SM; as separate launches 79 us at m = 13.)  Each line of code runs a few
// times a block, and on a cold start half of the stalls are instruction
// fetches, so both directions of the levels share one copy, as the three
// products of a slice do, and the map back from tower planes is by table
// (70001 x 51203 bits: 43.0 to 38.9 us).  The four blocks of an operand convert
// 8 of its 32 planes each, and the three half products of a slice run side by
// side (38.9 to 34.8 us).  What a block needs of the others is copied first,
// from another block each, instead of read where it is used by all from one (a
// product of 200001 x 200000 bits: 143 K cycles to 121 K); 32.8 us with the
// words' loads unconditional.
struct Operand { const u32 *src; u64 nchunks; u32 xor0; int k; };
struct RowAddr {                 // word j of plane p of slices PITCH words apart
    static constexpr bool rows_first = false;
    int plog, pitch;
    SL_HD u32 operator()(u32 j, u32 p) const { return j * pitch + p; }
};
// the map from tower planes by the 16 nibbles of a coefficient (entry v of
// nibble k at 16 k + v: the 16 entries fill the 32 banks once)
struct FromTable { u64 v[256]; };
constexpr FromTable make_from_table() {
    FromTable t{};
    for (int k = 0; k < 16; k++)
        for (int v = 0; v < 16; v++) {
            u64 x = 0;
            for (int b = 0; b < 4; b++)
                if (v >> b & 1) x ^= PHI.from[4 * k + b];
            t.v[16 * k + v] = x;
        }
    return t;
}
#ifdef __CUDACC__
__device__
#endif
static const FromTable FROM4 = make_from_table();
// 16-byte chunks a block: 32 planes, 16 planes
#ifdef __CUDACC__
__host__
#endif
SL_HD constexpr u32 small_chunks(int m) { return 14u << (m - 5); }
template <bool FWD, class At> SL_HD void taylor_warp_k(u32 *sm, const At &at, int k, u32 p) {
    switch (k) {
    case 10: taylor_warp<10, FWD>(sm, at, p); break;
    case 11: taylor_warp<11, FWD>(sm, at, p); break;
    case 12: taylor_warp<12, FWD>(sm, at, p); break;
    case 13: taylor_warp<13, FWD>(sm, at, p); break;
    default: taylor_warp<14, FWD>(sm, at, p); break;
    }
}
template <class Ex>
SL_HD void body_small(Ex ex, int m, const Operand &A, const Operand &B, u32 *out, u64 words) {
    const u32 ns = 1u << (m - 5), nb = ns / 8;
    const Tile T{m, m - 5, 0, 5, 0};
    const auto half = [&](u32 r) { return Half{ex.mem(r)}; };
    const auto quarter = [&](u32 r) { return Quarter{ex.mem(r) + 9 * ns}; };
    // in the space of the 32 planes, once those are used: the middle products,
    // later the words of nb + 1 slices, and the table at its end
    const auto words_of = [&](u32 r) { return Full{ex.mem(r)}; };
    const auto table = [&](u32 r) { return reinterpret_cast<u64 *>(ex.mem(r) + 9 * ns - 128); };
    const auto op = [&](u32 r) -> const Operand & { return r < 4 ? A : B; };
    const RowAddr at_half{3, 36}, at_quarter{4, 20};
    // chunk words, their planes, the conversion of 8 planes a block
    ex.block([&](u32 r, u32 tid, u32 nt) {
        const u32 nch = (u32)op(r).nchunks, xor0 = op(r).xor0;
        const u32 *src = nch ? op(r).src : reinterpret_cast<const u32 *>(FROM4.v);
        const Half h = half(r);
        staged<16, u32>(
            1u << op(r).k, tid, nt,
            // an unconditional load: behind a test they went one at a time
            // (10.4 K of 66 K cycles at m = 12)
            [&](u32 i) { return (src[i < nch ? i : 0] & (0u - (i < nch))) ^ (i == 0 ? xor0 : 0); },
            [&](u32 i, u32 v) { h.word(i >> 5, i & 31) = v; });
    });
    ex.block([&](u32 r, u32 tid, u32 nt) {
        const Half h = half(r);
        for (u32 i = tid; i < (1u << (op(r).k - 5)); i += nt) {
            u32 x[32];
            load_planes<32>(h, i, 0, x);
            transpose32(x);
            store_planes<32>(h, i, 0, x);
        }
    });
    ex.warps([&](u32 r, u32 w, u32 nw) {
        for (u32 p = w; p < 8; p += nw)
            taylor_warp_k<true>(&half(r).word(0, 8 * (r & 3)), at_half, op(r).k, p);
    });
    ex.block([&](u32 r, u32 tid, u32 nt) {
        taylor_regs<true>(&half(r).word(0, 8 * (r & 3)), at_half, op(r).k, tid, nt);
    });
    ex.cluster([](u32, u32, u32) {});
    // the planes of the other three blocks, each block beginning with another
    // one's (all reading one block's at a time took 11 K cycles at m = 14)
    ex.block([&](u32 r, u32 tid, u32 nt) {
        const int kl = op(r).k - 4;
        const auto from = [&](u32 i) { return (r + 1 + (i >> kl)) & 3; };
        staged<8, uint4>(
            3u << kl, tid, nt,
            [&](u32 i) {
                const u32 j = (i & ((1u << kl) - 1)) >> 1;
                return half((r & 4) + from(i)).chunk(j, 2 * from(i) + (i & 1));
            },
            [&](u32 i, const uint4 &q) {
                const u32 j = (i & ((1u << kl) - 1)) >> 1;
                half(r).chunk(j, 2 * from(i) + (i & 1)) = q;
            });
    });
    // tower planes of the quarter, copies included
    ex.block([&](u32 r, u32 tid, u32 nt) {
        for (u32 i = tid; i < ns; i += nt) {
            u32 a[32];
            load_planes<32>(half(r), i & ((1u << (op(r).k - 5)) - 1), 0, a);
            phi_quarter(quarter(r), i, r & 3, a);
        }
    });
#pragma unroll 1
    for (int pass = 0; pass < 2; pass++) {       // forward, inverse
        // levels m - 1 .. 5, the transposition, levels 4 .. 0, or back
#pragma unroll 1
        for (int i = 0; i <= m; i++)
            ex.block([&](u32 r, u32 tid, u32 nt) {
                const int j = pass ? m - i : i, L = j < m - 5 ? m - 1 - j : m - j;
                const u32 fwd = pass ? 0u : ~0u;
                if (pass ? r >= 4 : j < m - 5 && L >= op(r).k) return;
                if (j < m - 5) level_n<1, 1, 2>(quarter(r), T, L, tid, nt, fwd);
                else if (j > m - 5) level_x<1, 1, 2>(quarter(r), T, L, tid, nt, fwd);
                else transpose_groups<1>(quarter(r), ns, tid, nt);
            });
        if (pass) break;
        ex.cluster([](u32, u32, u32) {});
        // slices r nb .. r nb + nb - 1 of all quarters, after the space of 3 nb
        // products, each block beginning with another quarter
        const auto own = [&](u32 r, u32 q) { return Quarter{ex.mem(r) + (27 + 5 * q) * nb}; };
        const u32 nbl = (u32)(m - 8);
        ex.block([&](u32 r, u32 tid, u32 nt) {
            staged<8, uint4>(
                32 * nb, tid, nt,
                [&](u32 i) {
                    return quarter((r + (i >> (nbl + 2))) & 7)
                        .chunk(r * nb + ((i >> 2) & (nb - 1)), i & 3);
                },
                [&](u32 i, const uint4 &q) {
                    own(r, (r + (i >> (nbl + 2))) & 7).chunk((i >> 2) & (nb - 1), i & 3) = q;
                });
        });
        // their products (a0 + a1) b1, a0 (b0 + b1) and a1 (b0 + b1 + X b1),
        // then the first added to the other two
        ex.block([&](u32 r, u32 tid, u32 nt) {
            for (u32 i = tid; i < 3 * nb; i += nt) {
                const u32 join = i >= nb ? 1 : 0, h = i >= 2 * nb ? 1 : 0;
                const u32 s = i - (join + h) * nb;
                u32 a[32], b[32], c[32];
#pragma unroll
                for (int k = 0; k < 2; k++) load_planes<16>(own(r, 6 + k), s, 0, a + 16 * k);
                t_mulx<32>(a, c);
#pragma unroll
                for (int k = 0; k < 2; k++) load_planes<16>(own(r, 4 + k), s, 0, b + 16 * k);
#pragma unroll
                for (int k = 0; k < 32; k++)
                    b[k] = a[k] ^ (b[k] & (0u - join)) ^ (c[k] & (0u - h));
#pragma unroll
                for (int k = 0; k < 2; k++) load_planes<16>(own(r, 2 * h + k), s, 0, a + 16 * k);
#pragma unroll
                for (int k = 0; k < 2; k++) load_planes<16>(own(r, 2 + k), s, 0, c + 16 * k);
#pragma unroll
                for (int k = 0; k < 32; k++) { a[k] ^= c[k] & (join - 1u); c[k] = 0; }
                t_addmul_once<32>(a, b, c);
                store_planes<32>(half(r), i, 0, c);
            }
        });
        ex.block([&](u32 r, u32 tid, u32 nt) {
            for (u32 i = tid; i < 256; i += nt) table(r)[i] = FROM4.v[i];
            for (u32 i = tid; i < 16 * nb; i += nt) {
                const u32 h = (i >> 3) & 1, j = i >> 4, c = i & 7;
                uint4 x = half(r).chunk(j, c);
                const uint4 y = half(r).chunk((1 + h) * nb + j, c);
                x.x ^= y.x; x.y ^= y.y; x.z ^= y.z; x.w ^= y.w;
                quarter(2 * h + (c >> 2)).chunk(r * nb + j, c & 3) = x;
            }
        });
        ex.cluster([](u32, u32, u32) {});
    }
    ex.block([&](u32 r, u32 tid, u32 nt) {
        if (r < 4) taylor_regs<false>(&quarter(r).word(0, 0), at_quarter, m, tid, nt);
    });
    ex.warps([&](u32 r, u32 w, u32 nw) {
        if (r < 4)
            for (u32 p = w; p < 16; p += nw)
                taylor_warp_k<false>(&quarter(r).word(0, 0), at_quarter, m, p);
    });
    ex.cluster([](u32, u32, u32) {});
    // words of slices r nb .. and of the one before them: coefficients of 64
    // tower bits, the map, and the overlap-add of their halves
    ex.cluster([&](u32 r, u32 tid, u32 nt) {
        for (u32 i = tid; i < 2 * (nb + 1); i += nt) {
            const u32 h = i & 1, j = i >> 1, s = r * nb + j - 1;
            u32 a[32];
#pragma unroll
            for (int k = 0; k < 32; k++) a[k] = 0;
            if (s < ns) {                        // else before slice 0
#pragma unroll
                for (int k = 0; k < 2; k++) load_planes<16>(quarter(2 * h + k), s, 0, a + 16 * k);
                transpose32(a);
            }
            store_planes<32>(words_of(r), j, 8 * h, a);
        }
    });
    ex.block([&](u32 r, u32 tid, u32 nt) {
        const Full w = words_of(r);
        const u64 *t = table(r);
        for (u32 i = tid; i < 32 * (nb + 1); i += nt) {
            u32 &lo = w.word(i >> 5, i & 31), &hi = w.word(i >> 5, 32 + (i & 31));
            u64 x = 0;
#pragma unroll
            for (int k = 0; k < 8; k++)
                x ^= t[16 * k + (lo >> (4 * k) & 15)] ^ t[128 + 16 * k + (hi >> (4 * k) & 15)];
            lo = (u32)x;
            hi = (u32)(x >> 32);
        }
    });
    ex.block([&](u32 r, u32 tid, u32 nt) {
        const Full w = words_of(r);
        const u64 k0 = (u64)r * nb * 32;
        for (u32 i = tid; i < 32 * nb; i += nt)
            if (k0 + i < words)
                out[k0 + i] = w.word((i + 32) >> 5, i & 31) ^ w.word((i + 31) >> 5, 32 + ((i + 31) & 31));
        if (r == 7)
            for (u64 k = (u64)ns * 32 + tid; k < words; k += nt)
                out[k] = k == (u64)ns * 32 ? w.word(nb, 63) : 0;
    });
}

}  // namespace slice
