// slicefft.cu -- launches of the bit-sliced product transform
// (slicefft.cuh): products of up to 2^23 32-bit chunk coefficients.
//
// A product of 2^m coefficients is seven short passes over memory a side:
// chunk words to planes, Taylor levels above 2^16 (m > 16), the 2^16-chunk
// conversions in shared memory 4 or 8 planes at a time (planes are
// independent), then the butterflies in two passes over tiles of up to 512
// slices (128 KB): levels m-1 .. low over strided rows, low-1 .. 0 over
// consecutive slices.  Levels above an operand's own size are copies, made
// when its conversion is stored.  Between the transforms the values stay
// bit-sliced in the tower basis, in the order the last pass leaves them.
#include "gf2e_internal.cuh"
#include "slicefft.cuh"
#include "slicefft_api.cuh"

#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>

namespace {

using namespace slice;
using gf2e::SLICE_MAX_M;
using gf2e::SLICE_MIN_M;

struct DevEx {
    template <class F> GF2E_DEV void operator()(const F &f) const {
        f(threadIdx.x, blockDim.x);
        __syncthreads();
    }
    template <class F> GF2E_DEV void warps(u32 n, const F &f) const {
        if ((threadIdx.x >> 5) < n) f(threadIdx.x >> 5);
        __syncthreads();
    }
    GF2E_DEV void pair() const {             // the two blocks of a cluster
        asm volatile("barrier.cluster.arrive.release.aligned;\n"
                     "barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    }
};

constexpr int IN_LOG = 7;                    // slices a block of k_slice_in / out
constexpr int MIN_K = 10;                    // least conversion: 2^10 coefficients

// up to two operands, `batch` transforms each: blockIdx.y = operand * batch + i
struct In {
    const u32 *src[2];
    u64 sstride[2], nchunks[2];
    u32 xor0[2];
    uint4 *f[2];
    u64 fstride;                             // in 16-byte chunks
    int k[2];                                // 2^k slices' coefficients converted
    int batch;
};

__global__ void __launch_bounds__(1 << IN_LOG) k_slice_in(const In a) {
    __shared__ u32 sm[33 << IN_LOG];
    const int o = (int)blockIdx.y / a.batch, i = (int)blockIdx.y - o * a.batch;
    if ((blockIdx.x << (IN_LOG + 5)) >= (1u << a.k[o])) return;
    body_slice_in(DevEx{}, sm, a.src[o] + i * a.sstride[o], a.nchunks[o], a.xor0[o],
                  a.f[o] + i * a.fstride, blockIdx.x << IN_LOG,
                  a.k[o] - 5 < IN_LOG ? a.k[o] - 5 : IN_LOG);
}

// one operand's conversions of 2^K coefficients; blockIdx.x = block * groups
// + plane group, a warp a plane
struct TaylorArgs {
    uint4 *f;
    u64 fstride;
    int plog, groups;
    u32 c_src, reps, rep_stride;
};
template <int K, bool FWD>
__global__ void __launch_bounds__(256, 2) k_taylor(const TaylorArgs a) {
    extern __shared__ uint4 sm4[];
    const u32 b = blockIdx.x / a.groups, g = blockIdx.x - b * a.groups;
    const u32 c = g << (a.plog - 2);
    body_taylor<K, FWD>(DevEx{}, reinterpret_cast<u32 *>(sm4), a.f + blockIdx.y * a.fstride,
                        b << (K - 5), a.plog, c, a.c_src + c, a.reps, a.rep_stride);
}

struct HiArgs {
    const uint4 *src;
    uint4 *dst;
    u64 sstride, dstride;
    u32 c_dst;
    int groups;
};
template <int RLOG, bool FWD>
__global__ void __launch_bounds__(32 << Hi<RLOG>::PLOG, RLOG >= 7 ? 2 : 1)
k_taylor_hi(const HiArgs a) {
    extern __shared__ uint4 sm4[];
    const u32 ct = blockIdx.x / a.groups, g = blockIdx.x - ct * a.groups;
    const u32 c = g << Hi<RLOG>::CL;
    body_taylor_hi<RLOG, FWD>(DevEx{}, reinterpret_cast<u32 *>(sm4),
                              a.src + blockIdx.y * a.sstride, c, a.dst + blockIdx.y * a.dstride,
                              a.c_dst + c, ct);
}

struct BflyArgs {
    uint4 *f[2];
    u64 fstride;
    int m, rlog, clog, llo, collog;          // 2^collog column groups a window
    int top[2];
    int batch;
    bool first, lowp;
};
// blockIdx.x = 2 * tile + half, the halves of a tile one cluster; NQ quarters
// of a slice pair a thread (1 where the tiles leave SMs idle).  Two blocks of
// 256 threads an SM, so that one's loads and stores pass behind the other's
// products.
template <int NQ, bool FWD>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(NQ == 2 ? 256 : 512, NQ == 2 ? 2 : 1)
k_bfly(const BflyArgs a) {
    extern __shared__ uint4 sm4[];
    const int o = (int)blockIdx.y / a.batch, i = (int)blockIdx.y - o * a.batch;
    const u32 half = blockIdx.x & 1, tile = blockIdx.x >> 1;
    const u32 win = tile >> a.collog, col = tile & ((1u << a.collog) - 1);
    Tile T;
    T.m = a.m;
    T.rlog = a.rlog;
    T.clog = a.clog;
    T.llo = a.llo;
    T.base = (win << (a.llo + a.rlog - 5)) + (col << a.clog);
    body_bfly<NQ, FWD>(DevEx{}, sm4, a.f[o] + i * a.fstride, T, half, a.top[o], a.first, a.lowp);
}

// o = x1 y1 (+ x2 y2 where TWO) over 128 slices a block
template <bool TWO>
__global__ void __launch_bounds__(128, 2)
k_slice_mul(uint4 *o, const uint4 *x1, const uint4 *y1, const uint4 *x2, const uint4 *y2,
            u64 nslices, u64 fstride) {
    extern __shared__ uint4 sm4[];
    const u64 s0 = (u64)blockIdx.x * 128, y = blockIdx.y * fstride;
    o += y;
    x1 += y;
    y1 += y;
    if (TWO) {
        x2 += y;
        y2 += y;
    }
    const u32 n = (u32)min((u64)128, nslices - s0);
    const u32 tid = threadIdx.x;
    const Full ta{sm4}, tb{sm4 + 128 * 17}, tc{sm4 + 256 * 17};
    const bool same = x1 == y1;
    for (u32 i = tid; i < n * 16; i += 128) {
        copy16(&ta.chunk(i >> 4, i & 15), x1 + s0 * 16 + i);
        if (!same) copy16(&tb.chunk(i >> 4, i & 15), y1 + s0 * 16 + i);
    }
    copy_wait();
    __syncthreads();
    mul_slices(ta, same ? ta : tb, n, tid, 128);
    __syncthreads();
    if (TWO) {
        for (u32 i = tid; i < n * 16; i += 128) {
            copy16(&tb.chunk(i >> 4, i & 15), x2 + s0 * 16 + i);
            copy16(&tc.chunk(i >> 4, i & 15), y2 + s0 * 16 + i);
        }
        copy_wait();
        __syncthreads();
        mul_slices(tb, tc, n, tid, 128);
        __syncthreads();
    }
    for (u32 i = tid; i < n * 16; i += 128) {
        uint4 v = ta.chunk(i >> 4, i & 15);
        if (TWO) {
            const uint4 w = tb.chunk(i >> 4, i & 15);
            v.x ^= w.x; v.y ^= w.y; v.z ^= w.z; v.w ^= w.w;
        }
        o[s0 * 16 + i] = v;
    }
}

__global__ void __launch_bounds__(1 << IN_LOG)
k_slice_out(const uint4 *f, u64 fstride, u32 nsl, u32 *out, u64 ostride, u64 words) {
    __shared__ uint4 tile[17 << IN_LOG];
    __shared__ u32 side[(1 << IN_LOG) + 1];
    body_slice_out(DevEx{}, tile, side, f + blockIdx.y * fstride, nsl, out + blockIdx.y * ostride,
                   words, blockIdx.x * ((1 << IN_LOG) - 1), IN_LOG);
}

// 128 slices of natural words <-> tower planes, in place.  GROUPED: slice s of
// 32 takes the elements 32 b + s (the order of the last forward pass), else
// its own 32.
template <bool IN, bool GROUPED>
__global__ void __launch_bounds__(128, 2) k_slice_words(uint4 *f, u32 ns) {
    extern __shared__ uint4 sm4[];
    const Full src{sm4}, dst{sm4 + 128 * 17};
    f += (u64)blockIdx.x * 128 * 16;
    const u32 n = min(128u, ns), s = threadIdx.x, g = s & ~31u;
    for (u32 i = s; i < n * 16; i += 128) copy16(&src.chunk(i >> 4, i & 15), f + i);
    copy_wait();
    __syncthreads();
    if (s < n) {
        u32 a[64], b[64];
        if (IN && GROUPED) {
#pragma unroll
            for (int e = 0; e < 32; e++) {
                a[2 * e] = src.word(g + e, 2 * (s & 31));
                a[2 * e + 1] = src.word(g + e, 2 * (s & 31) + 1);
            }
        } else {
            load_planes<64>(src, s, 0, a);
        }
        if (IN) words_to_planes(a, b);
        else planes_to_words(a, b);
        if (!IN && GROUPED) {
#pragma unroll
            for (int e = 0; e < 32; e++) {
                dst.word(g + e, 2 * (s & 31)) = b[2 * e];
                dst.word(g + e, 2 * (s & 31) + 1) = b[2 * e + 1];
            }
        } else {
            store_planes<64>(dst, s, 0, b);
        }
    }
    __syncthreads();
    for (u32 i = s; i < n * 16; i += 128) f[i] = dst.chunk(i >> 4, i & 15);
}

struct SmallArgs {
    Operand op[2];
    u64 sstride[2];
    int m;
    u32 *out;
    u64 ostride, words;
};
struct ClusterEx {
    uint4 *sm;
    GF2E_DEV u32 rank() const { return blockIdx.x & 7; }
    GF2E_DEV uint4 *mem(u32 r) const {
        return r == rank() ? sm : cooperative_groups::this_cluster().map_shared_rank(sm, r);
    }
    template <class F> GF2E_DEV void block(const F &f) const {
        f(rank(), threadIdx.x, blockDim.x);
        __syncthreads();
    }
    template <class F> GF2E_DEV void warps(const F &f) const {
        f(rank(), threadIdx.x >> 5, blockDim.x >> 5);
        __syncthreads();
    }
    template <class F> GF2E_DEV void cluster(const F &f) const {
        f(rank(), threadIdx.x, blockDim.x);
        cooperative_groups::this_cluster().sync();
    }
};
// blockIdx.x = 8 * product + rank
__global__ void __cluster_dims__(8, 1, 1) __launch_bounds__(256, 2) k_small_mul(const SmallArgs a) {
    extern __shared__ uint4 sm4[];
    const u64 y = blockIdx.x >> 3;
    Operand A = a.op[0], B = a.op[1];
    A.src += y * a.sstride[0];
    B.src += y * a.sstride[1];
    body_small(ClusterEx{sm4}, a.m, A, B, a.out + y * a.ostride, a.words);
}

constexpr size_t SLICE_BYTES = 16 * 17, HALF_BYTES = 16 * 9;
constexpr size_t small_smem(int m) { return 16 * (size_t)small_chunks(m); }
constexpr size_t BFLY_SMEM = HALF_BYTES << TILE_LOG;

size_t taylor_smem(int k, int plog) { return (size_t)(4 * ((1 << (k - 5)) + 4)) << plog; }

int allow_smem() {
    // set once per device; two threads racing here both set the same values
    static std::atomic<bool> done[64];
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64 && done[dev].load(std::memory_order_acquire)) return GF2E_OK;
    cudaError_t e = cudaSuccess;
    auto allow = [&](const void *k, size_t n) {
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)n);
    };
#define GF2E_SL_ALLOW(K)                                             \
    allow((const void *)k_taylor<K, true>, taylor_smem(K, 3));       \
    allow((const void *)k_taylor<K, false>, taylor_smem(K, 3));
    GF2E_SL_ALLOW(15) GF2E_SL_ALLOW(16)
#undef GF2E_SL_ALLOW
#define GF2E_SL_ALLOW(R)                                                        \
    allow((const void *)k_taylor_hi<R, true>, 4 * Hi<R>::WORDS);    \
    allow((const void *)k_taylor_hi<R, false>, 4 * Hi<R>::WORDS);
    GF2E_SL_ALLOW(6) GF2E_SL_ALLOW(7)
#undef GF2E_SL_ALLOW
    allow((const void *)k_small_mul, small_smem(gf2e::SLICE_SMALL_MAX_M));
    allow((const void *)k_slice_words<true, true>, 2 * 128 * SLICE_BYTES);
    allow((const void *)k_slice_words<true, false>, 2 * 128 * SLICE_BYTES);
    allow((const void *)k_slice_words<false, true>, 2 * 128 * SLICE_BYTES);
    allow((const void *)k_slice_words<false, false>, 2 * 128 * SLICE_BYTES);
    allow((const void *)k_slice_mul<false>, 2 * 128 * SLICE_BYTES);
    allow((const void *)k_slice_mul<true>, 3 * 128 * SLICE_BYTES);
#define GF2E_SL_ALLOW(NQ)                                \
    allow((const void *)k_bfly<NQ, true>, BFLY_SMEM);    \
    allow((const void *)k_bfly<NQ, false>, BFLY_SMEM);
    GF2E_SL_ALLOW(1) GF2E_SL_ALLOW(2)
#undef GF2E_SL_ALLOW
    if (e != cudaSuccess) return gf2e::cuda_status(e, "sliced transform smem attribute");
    if (dev >= 0 && dev < 64) done[dev].store(true, std::memory_order_release);
    return GF2E_OK;
}

// a plan per size (host arithmetic only): the last pass holds the levels
// below m - 7 (10 to 14), so that 128 tiles and more keep the SMs busy from
// m = 17 on; the upper rows come one slice (256 bytes) wide until a tile of
// 512 slices is full
const Plan &plan_for(int m) {
    static const struct All {
        Plan p[SLICE_MAX_M + 1];
        All() {
            for (int m = SLICE_MIN_M; m <= SLICE_MAX_M; m++) {
                const int low = std::min(14, std::max(10, m - 7));
                p[m] = make_plan(m, low, m >= 22 ? TILE_LOG : 0);
            }
        }
    } all;
    return all.p[m];
}

int clog2(u64 v) {
    int k = 0;
    while (((u64)1 << k) < v) k++;
    return k;
}

// `chunks`: of a slice, 8 (the 32 chunk planes of an operand) or 16
template <bool FWD>
int launch_taylor(uint4 *f, u64 fstride, int batch, int m, int k, int chunks, u32 c_src,
                  cudaStream_t st) {
    TaylorArgs a;
    a.f = f;
    a.fstride = fstride;
    const int kt = std::min(k, 16);
    const u32 blocks = 1u << (k - kt);
    // 8 planes a block (whole 32-byte sectors) unless that leaves SMs idle
    a.plog = blocks * (chunks / 2) * (u32)batch >= (u32)gf2e::sm_count() ? 3 : 2;
    a.groups = chunks >> (a.plog - 2);
    a.c_src = c_src;
    a.reps = FWD ? 1u << (m - k) : 1u;
    a.rep_stride = 1u << (k - 5);
    const dim3 grid(blocks * a.groups, batch);
    const int threads = 32 << a.plog;
    const size_t smem = taylor_smem(kt, a.plog);
    switch (kt) {
    case 10: k_taylor<10, FWD><<<grid, threads, smem, st>>>(a); break;
    case 11: k_taylor<11, FWD><<<grid, threads, smem, st>>>(a); break;
    case 12: k_taylor<12, FWD><<<grid, threads, smem, st>>>(a); break;
    case 13: k_taylor<13, FWD><<<grid, threads, smem, st>>>(a); break;
    case 14: k_taylor<14, FWD><<<grid, threads, smem, st>>>(a); break;
    case 15: k_taylor<15, FWD><<<grid, threads, smem, st>>>(a); break;
    default: k_taylor<16, FWD><<<grid, threads, smem, st>>>(a); break;
    }
    GF2E_CHECK_LAUNCH("k_taylor");
    return GF2E_OK;
}

template <int RLOG, bool FWD>
int launch_hi_r(HiArgs a, int batch, cudaStream_t st) {
    typedef Hi<RLOG> H;
    a.groups = (FWD ? 8 : 16) >> H::CL;
    k_taylor_hi<RLOG, FWD><<<dim3(H::TILES * a.groups, batch), 32 << H::PLOG, 4 * H::WORDS, st>>>(a);
    GF2E_CHECK_LAUNCH("k_taylor_hi");
    return GF2E_OK;
}
template <bool FWD>
int launch_hi(const uint4 *src, u64 sstride, uint4 *dst, u64 dstride, u32 c_dst, int batch, int k,
              cudaStream_t st) {
    HiArgs a{src, dst, sstride, dstride, c_dst, 0};
    switch (k - 16) {
    case 1: return launch_hi_r<1, FWD>(a, batch, st);
    case 2: return launch_hi_r<2, FWD>(a, batch, st);
    case 3: return launch_hi_r<3, FWD>(a, batch, st);
    case 4: return launch_hi_r<4, FWD>(a, batch, st);
    case 5: return launch_hi_r<5, FWD>(a, batch, st);
    case 6: return launch_hi_r<6, FWD>(a, batch, st);
    default: return launch_hi_r<7, FWD>(a, batch, st);
    }
}

template <int NQ, bool FWD>
int launch_bfly(const BflyArgs &a, u32 tiles, int ny, cudaStream_t st) {
    const int tl = a.rlog + a.clog;
    const int threads = std::max(32, std::min(NQ == 2 ? 256 : 512, (1 << (tl - 1)) * (2 / NQ)));
    k_bfly<NQ, FWD><<<dim3(2 * tiles, ny), threads, HALF_BYTES << tl, st>>>(a);
    GF2E_CHECK_LAUNCH("k_bfly");
    return GF2E_OK;
}

// pass i of the butterflies (i = ntop: the low pass)
template <bool FWD>
int run_bfly(const Plan &P, int i, BflyArgs a, int nops, bool first, cudaStream_t st) {
    const bool lowp = i == P.ntop;
    a.m = P.m;
    a.llo = lowp ? 5 : P.top[i].llo;
    a.rlog = lowp ? P.low - 5 : P.top[i].rlog;
    a.clog = lowp ? 0 : P.top[i].clog;
    a.collog = a.llo - 5 - a.clog;
    const u32 tiles = 1u << (P.m - 5 - a.rlog - a.clog);
    const int ny = nops * a.batch;
    a.first = first && i == 0;
    a.lowp = lowp;
    // one quarter a thread while that fills idle SMs (m <= 16, where every
    // twiddle is in GF(2^16))
    if (P.m <= 16 && (u64)tiles * ny < (u64)gf2e::sm_count())
        return launch_bfly<1, FWD>(a, tiles, ny, st);
    return launch_bfly<2, FWD>(a, tiles, ny, st);
}

}  // namespace

namespace gf2e {

bool slice_selfcheck(const u64 *basis) {
    for (int i = 0; i < 25; i++) {
        u64 v = 0;
        for (int j = 0; j < 64; j++)
            if ((basis[i] >> j) & 1) v ^= PHI.to[j];
        if (v != CANTOR[i]) return false;
    }
    return true;
}

int slice_fwd(int m, const SliceOp *ops, int nops, u64 fstride, int batch, cudaStream_t st) {
    GF2E_TRY(allow_smem());
    const Plan &P = plan_for(m);
    In in;
    in.fstride = fstride / 2;
    in.batch = batch;
    u32 nx = 1;
    for (int o = 0; o < nops; o++) {
        in.src[o] = ops[o].src;
        in.sstride[o] = ops[o].stride;
        in.nchunks[o] = ops[o].nchunks;
        in.xor0[o] = ops[o].xor0;
        in.f[o] = reinterpret_cast<uint4 *>(ops[o].f);
        in.k[o] = std::min(m, std::max(MIN_K, clog2(ops[o].nchunks)));
        nx = std::max(nx, 1u << std::max(0, in.k[o] - 5 - IN_LOG));
    }
    k_slice_in<<<dim3(nx, nops * batch), 1 << IN_LOG, 0, st>>>(in);
    GF2E_CHECK_LAUNCH("k_slice_in");
    BflyArgs a;
    a.fstride = in.fstride;
    a.batch = batch;
    for (int o = 0; o < nops; o++) {
        u32 c = 0;
        if (in.k[o] > 16) {
            GF2E_TRY(launch_hi<true>(in.f[o], in.fstride, in.f[o], in.fstride, 8, batch, in.k[o], st));
            c = 8;
        }
        GF2E_TRY(launch_taylor<true>(in.f[o], in.fstride, batch, m, in.k[o], 8, c, st));
        a.f[o] = in.f[o];
        a.top[o] = in.k[o];
    }
    for (int i = 0; i <= P.ntop; i++) GF2E_TRY(run_bfly<true>(P, i, a, nops, true, st));
    return GF2E_OK;
}

int slice_pointwise(u64 *o, const u64 *x1, const u64 *y1, const u64 *x2, const u64 *y2, u64 n,
                    u64 fstride, int batch, cudaStream_t st) {
    GF2E_TRY(allow_smem());
    const u64 ns = n / 32, fs = fstride / 2;
    const dim3 grid((unsigned)((ns + 127) / 128), batch);
    auto p = [](const u64 *x) { return reinterpret_cast<const uint4 *>(x); };
    if (x2)
        k_slice_mul<true><<<grid, 128, 3 * 128 * SLICE_BYTES, st>>>(reinterpret_cast<uint4 *>(o), p(x1),
                                                            p(y1), p(x2), p(y2), ns, fs);
    else
        k_slice_mul<false><<<grid, 128, 2 * 128 * SLICE_BYTES, st>>>(reinterpret_cast<uint4 *>(o), p(x1),
                                                             p(y1), nullptr, nullptr, ns,
                                                             fs);
    GF2E_CHECK_LAUNCH("k_slice_mul");
    return GF2E_OK;
}

int slice_inv(int m, u64 *f, u64 *tmp, u64 fstride, int batch, u64 *out, u64 ostride, u64 ow,
              cudaStream_t st) {
    GF2E_TRY(allow_smem());
    const Plan &P = plan_for(m);
    uint4 *f4 = reinterpret_cast<uint4 *>(f);
    const u64 fs = fstride / 2;
    BflyArgs a;
    a.f[0] = a.f[1] = f4;
    a.top[0] = a.top[1] = m;
    a.fstride = fs;
    a.batch = batch;
    for (int i = P.ntop; i >= 0; i--) GF2E_TRY(run_bfly<false>(P, i, a, 1, false, st));
    GF2E_TRY(launch_taylor<false>(f4, fs, batch, m, m, 16, 0, st));
    if (m > 16) {
        uint4 *t4 = reinterpret_cast<uint4 *>(tmp);
        GF2E_TRY(launch_hi<false>(f4, fs, t4, fs, 0, batch, m, st));
        f4 = t4;
    }
    const u64 words = 2 * ow;
    const u64 per = 32 * ((1 << IN_LOG) - 1);
    const unsigned grid = (unsigned)((words + per - 1) / per);
    k_slice_out<<<dim3(grid, batch), 1 << IN_LOG, 0, st>>>(f4, fs, 1u << (m - 5),
                                                         reinterpret_cast<u32 *>(out),
                                                         2 * ostride, words);
    GF2E_CHECK_LAUNCH("k_slice_out");
    return GF2E_OK;
}

int slice_transform(int m, bool forward, u64 *f, cudaStream_t st) {
    GF2E_TRY(allow_smem());
    const Plan &P = plan_for(m);
    uint4 *f4 = reinterpret_cast<uint4 *>(f);
    const u32 ns = 1u << (m - 5);
    const u32 grid = (ns + 127) / 128;
    const size_t smem = 2 * 128 * SLICE_BYTES;
    BflyArgs a;
    a.f[0] = a.f[1] = f4;
    a.top[0] = a.top[1] = m;
    a.fstride = 0;
    a.batch = 1;
    if (forward) {
        k_slice_words<true, false><<<grid, 128, smem, st>>>(f4, ns);
        GF2E_CHECK_LAUNCH("k_slice_words");
        GF2E_TRY(launch_taylor<true>(f4, 0, 1, m, m, 16, 0, st));
        for (int i = 0; i <= P.ntop; i++) GF2E_TRY(run_bfly<true>(P, i, a, 1, false, st));
        k_slice_words<false, true><<<grid, 128, smem, st>>>(f4, ns);
    } else {
        k_slice_words<true, true><<<grid, 128, smem, st>>>(f4, ns);
        GF2E_CHECK_LAUNCH("k_slice_words");
        for (int i = P.ntop; i >= 0; i--) GF2E_TRY(run_bfly<false>(P, i, a, 1, false, st));
        GF2E_TRY(launch_taylor<false>(f4, 0, 1, m, m, 16, 0, st));
        k_slice_words<false, false><<<grid, 128, smem, st>>>(f4, ns);
    }
    GF2E_CHECK_LAUNCH("k_slice_words");
    return GF2E_OK;
}

int slice_transform_passes(int m) { return plan_for(m).ntop + 4; }

int slice_small(int m, const SliceOp &x, const SliceOp &y, int batch, u64 *out, u64 ostride,
                u64 ow, cudaStream_t st) {
    GF2E_TRY(allow_smem());
    SmallArgs a;
    const SliceOp *op[2] = {&x, &y};
    for (int o = 0; o < 2; o++) {
        a.op[o] = Operand{op[o]->src, op[o]->nchunks, op[o]->xor0,
                          std::min(m, std::max(MIN_K, clog2(op[o]->nchunks)))};
        a.sstride[o] = op[o]->stride;
    }
    a.m = m;
    a.out = reinterpret_cast<u32 *>(out);
    a.ostride = 2 * ostride;
    a.words = 2 * ow;
    // 128 threads up to m = 12 (64 slice pairs a level): four blocks an SM
    k_small_mul<<<8 * batch, m <= 12 ? 128 : 256, small_smem(m), st>>>(a);
    GF2E_CHECK_LAUNCH("k_small_mul");
    return GF2E_OK;
}

}  // namespace gf2e
