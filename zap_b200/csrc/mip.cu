// mip.cu - 2x2 box-filter mip generator (zap_tex.h:1358-1469), bit-exact, HBM-bound.
//
// RGBA8: with srgb, RGB goes through the sRGB->linear table, the four values are summed left to right and scaled
// by 0.25f, and the result maps back to sRGB as the first k whose threshold exceeds it (the reference's binary
// search; here one table word and no search, srgb_back below). Alpha (and RGB without srgb) is (a + b + c + d + 2) >> 2.
// Odd sizes drop the last row / column.
// A launch makes up to six levels of a chain: a CTA takes a 64x64 tile of the source level, from which every texel of
// levels 1..6 below the tile follows (odd sizes drop the last row or column at each level, and a side of 1 stays
// 1, so a tile never needs a neighbour's texels). Each thread averages a 4x4 source block to 2x2 texels of level 1 and
// one of level 2 in registers; levels 3..6 go through shared memory. So a 4096x4096 chain is two launches and one
// read of the source, instead of a launch per level that reads the level above back (sRGB 101.9 -> 46.8 us, linear 64.3 ->
// 28.3; 256x256 42.8 -> 12.8).
#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>

#include "ztc_common.cuh"
#include "ztc_internal.h"

namespace ztc {

// the bucket of a linear value: 0 below 2^-16 (and for negative values), else its exponent and top 6 mantissa bits
ZTC_DEV int srgb_bucket(float v) {
    const uint32_t u = f_as_u(v);
    if (u < 0x37800000u || (u & 0x80000000u)) return 0;
    const int q = (int)(u >> 17) - (0x37800000 >> 17);
    return q < kSrgbBuckets - 1 ? q : kSrgbBuckets - 1;
}
// first k with v < thr[k] (zap_tex.h:1429-1433), 255 when there is none: the reference's binary search finds it in
// eight steps; here the scan starts at the bucket's lower bound, one to three steps. It builds srgb_back's table.
ZTC_DEV uint32_t lin_to_srgb(const float *thr, const uint8_t *bucket, float v) {
    int k = bucket[srgb_bucket(v)];
    while (k < 255 && !(v < thr[k])) k++;
    return (uint32_t)k;
}

// The sRGB code of a quarter of s = the sum of four linear values, from one table word and no search. A bucket here is
// the exponent and the top 7 mantissa bits of s over [2^-11, 4] (its relative width, 2^-7 at most, is below the spacing
// of neighbouring thresholds, 0.89 % at its least, near 4, so a bucket holds at most one). With t the low 16 bits of 4 times
// the threshold inside the bucket (2^16 for none), the word is (code at the bucket's lowest value << 16) + 2^16 - t
// less the bucket's own high half, so adding s's bits leaves the code in bits 16..23, one more where s has reached the
// threshold. A quarter of s is exact. Sums below 2^-11 are 0 and 3.0e-4 (one texel of code 1), both below 4 times the
// least threshold (6.1e-4) like 2^-11 itself, whose code 0 they take.
template <typename Tables>
ZTC_DEV uint32_t srgb_back(const Tables &T, float s) {  // the code in bits 16..23
    const uint32_t u = f_as_u(fmaxf(s, u_as_f((uint32_t)kSrgbBackLow << 16)));
    return T.back(u >> 16) + u;
}

// The tables as box4_srgb reads them: in memory (host code), or a CTA's copy in shared memory by 32-bit address (one byte
// extraction and one multiply-add a lookup). One copy per CTA: 2 to 32 copies of the linear values in separate banks
// measured no faster on a texture (45.6 us at 1 and at 32 copies, 49.3 at 8: neighbouring lanes mostly share a code).
struct MipTables {
    const SrgbTables *t;
    ZTC_DEV float lin(uint32_t x, int c) const { return t->lin[chan(x, c)]; }
    ZTC_DEV uint32_t back(uint32_t hi) const { return t->back[hi - kSrgbBackLow]; }
};
struct MipShared {
    float lin[256];
    uint32_t back[kSrgbBack];
};
__device__ MipShared gSrgb;  // what the kernels read of the tables
struct MipSharedTables {
    uint32_t lin0, back0;  // shared-memory addresses of lin[0] and of back[-kSrgbBackLow]
#ifdef __CUDACC__
    __device__ __forceinline__ explicit MipSharedTables(const MipShared &S)
        : lin0((uint32_t)__cvta_generic_to_shared(S.lin)), back0((uint32_t)__cvta_generic_to_shared(S.back) - 4u * kSrgbBackLow) {}
    __device__ __forceinline__ static uint32_t ld(uint32_t a) {
        uint32_t v;
        asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(a));
        return v;
    }
    __device__ __forceinline__ float lin(uint32_t x, int c) const {
        return __uint_as_float(ld(__byte_perm(x, 0u, 0x4440u | (uint32_t)c) * 4u + lin0));
    }
    __device__ __forceinline__ uint32_t back(uint32_t hi) const { return ld(hi * 4u + back0); }
#endif
};

ZTC_DEV uint32_t box4_linear(uint32_t a, uint32_t b, uint32_t c, uint32_t d) {  // (a + b + c + d + 2) >> 2 per channel
    const uint32_t m = 0x00FF00FFu;  // two channels a word, as 16-bit fields: sums below 2^10
    const uint32_t rb = (a & m) + (b & m) + (c & m) + (d & m) + 0x00020002u;
    const uint32_t ga = ((a >> 8) & m) + ((b >> 8) & m) + ((c >> 8) & m) + ((d >> 8) & m) + 0x00020002u;
    return ((rb >> 2) & m) | ((ga << 6) & ~m);
}
template <typename Tables>
ZTC_DEV uint32_t box4_srgb(uint32_t a, uint32_t b, uint32_t c, uint32_t d, const Tables &T) {
    uint32_t r[3];
    #pragma unroll
    for (int k = 0; k < 3; k++) r[k] = srgb_back(T, T.lin(a, k) + T.lin(b, k) + T.lin(c, k) + T.lin(d, k));
    const uint32_t top = 0x01000000u;  // alpha: dot products take the top bytes' sum off the logic pipe
    const uint32_t al = (dot4(a, top) + dot4(b, top) + dot4(c, top) + dot4(d, top) + 2u) >> 2;
#ifdef __CUDA_ARCH__
    return __byte_perm(__byte_perm(r[0], r[1], 0x0062u), __byte_perm(r[2], al, 0x0042u), 0x5410u);
#else
    return ((r[0] >> 16) & 0xFFu) | ((r[1] >> 8) & 0xFF00u) | (r[2] & 0xFF0000u) | (al << 24);
#endif
}
// with the tables in memory: the form the host tests of the arithmetic call
ZTC_DEV uint32_t box4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, bool srgb, const SrgbTables &T) {
    return srgb ? box4_srgb(a, b, c, d, MipTables{&T}) : box4_linear(a, b, c, d);
}

ZTC_DEV uint32_t ld_texel(const uint8_t *p) {
    if ((((uintptr_t)p) & 3u) == 0) return ldg((const uint32_t *)p);
    return (uint32_t)ldg(p) | ((uint32_t)ldg(p + 1) << 8) | ((uint32_t)ldg(p + 2) << 16) | ((uint32_t)ldg(p + 3) << 24);
}
ZTC_DEV void st_texel(uint8_t *p, uint32_t v) {
    if ((((uintptr_t)p) & 3u) == 0) { *(uint32_t *)p = v; return; }
    p[0] = (uint8_t)v; p[1] = (uint8_t)(v >> 8); p[2] = (uint8_t)(v >> 16); p[3] = (uint8_t)(v >> 24);
}

// source texels a side, threads of a CTA (a 4x4 block each), resident CTAs per SM. 4 CTAs measured best: 46.8 / 47.6 / 50.7 /
// 56.5 us at 4 / 5 / 6 / 8 for a 4096x4096 sRGB chain (45 % ALU pipe, 50 % LSU; the read of the source alone takes 10.4);
// loading the next tile ahead did not help (49.9).
constexpr int kMipTile = 64, kMipThreads = 256, kMipCtas = 4;

// every thread of the CTA calls it; a barrier must follow before the tables are read
__device__ __forceinline__ void stage_mip_tables(MipShared &S, const MipShared *g) {
    for (int k = threadIdx.x; k < 256; k += kMipThreads) S.lin[k] = __ldg(g->lin + k);
    for (int k = threadIdx.x; k < kSrgbBack; k += kMipThreads) S.back[k] = __ldg(g->back + k);
}

struct NoTables {};  // of a linear chain
template <typename Tables>
__device__ __forceinline__ uint32_t mip_box(uint32_t a, uint32_t b, uint32_t c, uint32_t d, bool srgb, const Tables &T) {
    return srgb ? box4_srgb(a, b, c, d, T) : box4_linear(a, b, c, d);
}
__device__ __forceinline__ uint32_t mip_box(uint32_t a, uint32_t b, uint32_t c, uint32_t d, bool, const NoTables &) {
    return box4_linear(a, b, c, d);
}

struct MipScratch { uint32_t l2[256], l3[64], l4[16], l5[4]; };  // a tile's texels of levels 2..5

// One level of a tile by one warp, `side` x `side` texels from the level above: from (2 side x 2 side) to `to`.
template <int SIDE, typename Tables>
__device__ __forceinline__ void mip_tail_level(const uint32_t *from, uint32_t *to, uint8_t *dst, int tx, int ty, int w, int h, int nw, int nh,
                                               bool srgb, const Tables &T) {
    #pragma unroll 1
    for (int k = threadIdx.x & 31; k < SIDE * SIDE; k += 32) {
        const int sx = k & (SIDE - 1), sy = k / SIDE, x = tx * SIDE + sx, y = ty * SIDE + sy;
        if (x >= nw || y >= nh) continue;
        const uint32_t *p = from + 4 * sy * SIDE + 2 * sx;  // a side of 1 is averaged with itself
        const int c1 = 2 * x + 1 < w ? 1 : 0, r1 = 2 * y + 1 < h ? 2 * SIDE : 0;
        const uint32_t v = mip_box(p[0], p[c1], p[r1], p[r1 + c1], srgb, T);
        st_texel(dst + ((size_t)y * nw + x) * 4, v);
        to[k] = v;
    }
    __syncwarp();
}

// a thread's 4x4 source texels of tile (tx, ty); whole: they lie inside the level and were loaded (rows of 16 bytes, or of
// four words at a lesser alignment), else the edge code reads them texel by texel
struct MipSource {
    uint4 r[4];
    bool whole;
};
__device__ __forceinline__ MipSource mip_load(const MipChain &C, int tx, int ty) {
    MipSource m;
    const int x0 = tx * kMipTile + 4 * (int)(threadIdx.x & 15), y0 = ty * kMipTile + 4 * (int)(threadIdx.x >> 4);
    const uint32_t align = (uint32_t)((uintptr_t)C.src | C.pitch) & 15u;
    m.whole = x0 + 3 < C.w && y0 + 3 < C.h && (align & 3u) == 0;
    if (m.whole) {
        const uint8_t *p = C.src + (size_t)y0 * C.pitch + (size_t)x0 * 4;
        #pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t *q = (const uint32_t *)(p + (size_t)k * C.pitch);
            m.r[k] = align == 0 ? __ldg((const uint4 *)q) : make_uint4(__ldg(q), __ldg(q + 1), __ldg(q + 2), __ldg(q + 3));
        }
    }
    return m;
}

// Tile (tx, ty) of one chain: levels 1..C.levels below its 64x64 source texels m; n counts the CTA's tiles before it that
// have a second level. Every thread of the CTA calls it. Levels 3..6 are one warp's work (warp n modulo 8) while the
// others go on to the next tile. A tile with a second level writes S[n & 1] and meets one barrier; S[n & 1] is written
// again by the second such tile after it, behind the barrier of the first, which this tile's warp reaches only when it is
// done. A tile of one level has neither, and the chains of a batch differ, so n must not count it.
template <typename Tables>
__device__ __forceinline__ void mip_tile(const MipChain &C, const MipSource &m, int tx, int ty, int n, const Tables &T, MipScratch (&S)[2]) {
    const bool srgb = C.srgb != 0;
    const int lx = threadIdx.x & 15, ly = threadIdx.x >> 4, x0 = tx * kMipTile + 4 * lx, y0 = ty * kMipTile + 4 * ly;
    int w = C.w, h = C.h, nw = w > 1 ? w >> 1 : 1, nh = h > 1 ? h >> 1 : 1;
    uint32_t o[4] = {0u, 0u, 0u, 0u};  // the thread's 2x2 texels of level 1
    {
        const int x = x0 >> 1, y = y0 >> 1;
        uint8_t *d = C.dst[0] + (size_t)y * C.dst_pitch + (size_t)x * 4;
        if (m.whole) {
            #pragma unroll
            for (int k = 0; k < 2; k++) {
                o[2 * k] = mip_box(m.r[2 * k].x, m.r[2 * k].y, m.r[2 * k + 1].x, m.r[2 * k + 1].y, srgb, T);
                o[2 * k + 1] = mip_box(m.r[2 * k].z, m.r[2 * k].w, m.r[2 * k + 1].z, m.r[2 * k + 1].w, srgb, T);
            }
            if ((((uintptr_t)C.dst[0] | C.dst_pitch) & 7u) == 0) {
                *(uint2 *)d = make_uint2(o[0], o[1]);
                *(uint2 *)(d + C.dst_pitch) = make_uint2(o[2], o[3]);
            } else {
                st_texel(d, o[0]); st_texel(d + 4, o[1]);
                st_texel(d + C.dst_pitch, o[2]); st_texel(d + C.dst_pitch + 4, o[3]);
            }
        } else if (x < nw && y < nh) {
            #pragma unroll 1
            for (int k = 0; k < 4; k++) {  // a texel past the level's edge matters only where the side is 1: its one texel again
                const int xx = min(x + (k & 1), nw - 1), yy = min(y + (k >> 1), nh - 1);
                const uint8_t *r0 = C.src + (size_t)(2 * yy) * C.pitch, *r1 = C.src + (size_t)min(2 * yy + 1, h - 1) * C.pitch;
                const size_t c0 = (size_t)(2 * xx) * 4, c1 = (size_t)min(2 * xx + 1, w - 1) * 4;
                const uint32_t v = mip_box(ld_texel(r0 + c0), ld_texel(r0 + c1), ld_texel(r1 + c0), ld_texel(r1 + c1), srgb, T);
                if (xx == x + (k & 1) && yy == y + (k >> 1)) st_texel(d + (size_t)(k >> 1) * C.dst_pitch + 4 * (k & 1), v);
                #pragma unroll
                for (int q = 0; q < 4; q++) if (q == k) o[q] = v;
            }
        }
    }
    if (C.levels < 2) return;
    MipScratch &M = S[n & 1];
    w = nw; h = nh; nw = w > 1 ? w >> 1 : 1; nh = h > 1 ? h >> 1 : 1;
    {
        const int x = x0 >> 2, y = y0 >> 2;
        if (x < nw && y < nh) {
            const uint32_t v = mip_box(o[0], o[1], o[2], o[3], srgb, T);
            st_texel(C.dst[1] + ((size_t)y * nw + x) * 4, v);
            M.l2[threadIdx.x] = v;
        }
    }
    __syncthreads();
    if (C.levels < 3 || (int)(threadIdx.x >> 5) != (n & 7)) return;
    int pw = nw, ph = nh;
    nw = pw > 1 ? pw >> 1 : 1; nh = ph > 1 ? ph >> 1 : 1;
    mip_tail_level<8>(M.l2, M.l3, C.dst[2], tx, ty, pw, ph, nw, nh, srgb, T);
    if (C.levels < 4) return;
    pw = nw; ph = nh; nw = pw > 1 ? pw >> 1 : 1; nh = ph > 1 ? ph >> 1 : 1;
    mip_tail_level<4>(M.l3, M.l4, C.dst[3], tx, ty, pw, ph, nw, nh, srgb, T);
    if (C.levels < 5) return;
    pw = nw; ph = nh; nw = pw > 1 ? pw >> 1 : 1; nh = ph > 1 ? ph >> 1 : 1;
    mip_tail_level<2>(M.l4, M.l5, C.dst[4], tx, ty, pw, ph, nw, nh, srgb, T);
    if (C.levels < 6) return;
    pw = nw; ph = nh; nw = pw > 1 ? pw >> 1 : 1; nh = ph > 1 ? ph >> 1 : 1;
    mip_tail_level<1>(M.l5, M.l4, C.dst[5], tx, ty, pw, ph, nw, nh, srgb, T);  // l4 is free again
}

// the CTA's tiles k = blockIdx.x, + gridDim.x, ...; at(k): the chain and place of tile k
template <typename Tables, typename At>
__device__ __forceinline__ void mip_tiles_of_cta(int ntiles, const Tables &T, MipScratch (&S)[2], At &&at) {
    int n = 0;  // tiles with a second level so far (mip_tile)
    for (int k = blockIdx.x; k < ntiles; k += gridDim.x) {
        const MipChain *c;
        int x, y;
        at(k, c, x, y);
        const MipSource m = mip_load(*c, x, y);
        if (k == (int)blockIdx.x) __syncthreads();  // the tables are staged
        mip_tile(*c, m, x, y, n, T, S);
        n += c->levels > 1;
    }
}

template <bool SRGB>
__global__ void __launch_bounds__(kMipThreads, kMipCtas) mip_chain_kernel(const __grid_constant__ MipChain C, int tiles_x, int ntiles) {
    __shared__ MipShared s_tab;  // not referenced (and not allocated) without SRGB
    __shared__ MipScratch S[2];
    const auto at = [&](int k, const MipChain *&c, int &x, int &y) { c = &C; x = k % tiles_x; y = k / tiles_x; };
    if constexpr (SRGB) {
        stage_mip_tables(s_tab, &gSrgb);
        mip_tiles_of_cta(ntiles, MipSharedTables(s_tab), S, at);
    } else mip_tiles_of_cta(ntiles, NoTables{}, S, at);
}

// batched: tiles of many chains
__global__ void __launch_bounds__(kMipThreads, kMipCtas) batch_mip_kernel(const MipChain *__restrict__ chains, const MipTile *__restrict__ tiles, int ntiles) {
    __shared__ MipShared s_tab;
    __shared__ MipScratch S[2];
    stage_mip_tables(s_tab, &gSrgb);
    mip_tiles_of_cta(ntiles, MipSharedTables(s_tab), S, [&](int k, const MipChain *&c, int &x, int &y) {
        const MipTile t = tiles[k];
        c = chains + t.chain; x = t.x; y = t.y;
    });
}

// float RGBA (linear): 0.25f * (a + b + c + d) per channel (zap_tex.h:1460-1469)
__global__ void __launch_bounds__(256) mip_f32_kernel(const float *__restrict__ src, int w, int h, size_t stride,
                                                      float *__restrict__ dst, size_t dst_stride, int nw, int nh, int vec) {
    const long total = (long)nw * nh;
    for (long id = (long)blockIdx.x * blockDim.x + threadIdx.x; id < total; id += (long)gridDim.x * blockDim.x) {
        int y = (int)(id / nw), x = (int)(id % nw);
        int x0 = min(2 * x, w - 1), x1 = min(2 * x + 1, w - 1), y0 = min(2 * y, h - 1), y1 = min(2 * y + 1, h - 1);
        const float *a = src + (size_t)y0 * stride + (size_t)x0 * 4, *b = src + (size_t)y0 * stride + (size_t)x1 * 4;
        const float *c = src + (size_t)y1 * stride + (size_t)x0 * 4, *d = src + (size_t)y1 * stride + (size_t)x1 * 4;
        float *o = dst + (size_t)y * dst_stride + (size_t)x * 4;
        if (vec) {
            float4 A = __ldg((const float4 *)a), B = __ldg((const float4 *)b), C = __ldg((const float4 *)c), D = __ldg((const float4 *)d);
            *(float4 *)o = make_float4(0.25f * (A.x + B.x + C.x + D.x), 0.25f * (A.y + B.y + C.y + D.y),
                                       0.25f * (A.z + B.z + C.z + D.z), 0.25f * (A.w + B.w + C.w + D.w));
        } else {
            #pragma unroll
            for (int k = 0; k < 4; k++) o[k] = 0.25f * (__ldg(a + k) + __ldg(b + k) + __ldg(c + k) + __ldg(d + k));
        }
    }
}

// The reference's sRGB constants are the double-precision transfer function printed with 9 significant digits
// and read back as float (checked bit for bit against the reference's tables by the test suite).
static float srgb_to_linear_9g(double c) {
    double lin = c <= 0.04045 ? c / 12.92 : std::pow((c + 0.055) / 1.055, 2.4);
    char buf[64];
    std::snprintf(buf, sizeof buf, "%.9g", lin);
    return std::strtof(buf, nullptr);
}

void srgb_tables_host(SrgbTables &t) {
    for (int k = 0; k < 256; k++) t.lin[k] = srgb_to_linear_9g(k / 255.0);
    for (int k = 0; k < 255; k++) t.thr[k] = srgb_to_linear_9g((k + 0.5) / 255.0);
    t.thr[255] = INFINITY;
    for (int q = 0; q < kSrgbBuckets; q++) {  // the answer at the bucket's lowest value (0 for bucket 0)
        uint32_t u = q ? (uint32_t)(q + (0x37800000 >> 17)) << 17 : 0u;
        float lo;
        std::memcpy(&lo, &u, 4);
        int k = 0;
        while (k < 255 && !(lo < t.thr[k])) k++;
        t.bucket[q] = (uint8_t)k;
    }
    for (int q = 0; q < kSrgbBack; q++) {
        const uint32_t u = (uint32_t)(q + kSrgbBackLow) << 16;  // the bucket's lowest sum
        float lo, thr;
        std::memcpy(&lo, &u, 4);
        const uint32_t k = lin_to_srgb(t.thr, t.bucket, lo * 0.25f);
        thr = 4.0f * t.thr[k];
        const uint32_t tu = f_as_u(thr), in = (tu >> 16) == (u >> 16) ? tu & 0xFFFFu : 0x10000u;  // the bucket's threshold, or none
        t.back[q] = (k << 16) + 0x10000u - in - u;
    }
}

cudaError_t upload_mip_tables() {
    SrgbTables T;
    srgb_tables_host(T);
    MipShared D;
    std::memcpy(D.lin, T.lin, sizeof D.lin);
    std::memcpy(D.back, T.back, sizeof D.back);
    return cudaMemcpyToSymbol(gSrgb, &D, sizeof D);
}

static int grid_for(long work, int threads) {
    long g = (work + threads - 1) / threads;
    return (int)(g < 148L * 32 ? (g < 1 ? 1 : g) : 148L * 32);
}

int mip_tiles(int w, int h, int &tiles_x) {
    const int nw = w > 1 ? w / 2 : 1, nh = h > 1 ? h / 2 : 1, half = kMipTile / 2;
    tiles_x = (nw + half - 1) / half;
    return tiles_x * ((nh + half - 1) / half);
}

}  // namespace ztc

cudaError_t ztc_launch_mip_levels(const ztc::MipChain &chain, cudaStream_t stream) {
    int tiles_x = 1;
    const int ntiles = ztc::mip_tiles(chain.w, chain.h, tiles_x), sms = ztc_sm_count();
    ztc::TraceScope tr("mip_rgba8", stream);
    long units = 0;
    for (int l = 1; l <= chain.levels; l++) units += (long)std::max(1, chain.w >> l) * std::max(1, chain.h >> l);
    ztc::trace_units(units);
    const int grid = std::min(ntiles, sms * ztc::kMipCtas);
    if (chain.srgb) ztc::mip_chain_kernel<true><<<grid, ztc::kMipThreads, 0, stream>>>(chain, tiles_x, ntiles);
    else ztc::mip_chain_kernel<false><<<grid, ztc::kMipThreads, 0, stream>>>(chain, tiles_x, ntiles);
    return cudaGetLastError();
}

cudaError_t ztc_launch_mip(const uint8_t *src, int w, int h, size_t stride, int srgb, uint8_t *dst, size_t dst_stride,
                           cudaStream_t stream) {
    ztc::MipChain c{};
    c.src = src; c.pitch = stride; c.w = w; c.h = h; c.levels = 1; c.srgb = srgb ? 1 : 0;
    c.dst[0] = dst; c.dst_pitch = dst_stride;
    return ztc_launch_mip_levels(c, stream);
}

cudaError_t ztc_launch_mip_f(const float *src, int w, int h, size_t stride, float *dst, size_t dst_stride, cudaStream_t stream) {
    int nw = w > 1 ? w / 2 : 1, nh = h > 1 ? h / 2 : 1;
    int vec = ((((uintptr_t)src) | (stride * 4)) & 15u) == 0 && ((((uintptr_t)dst) | (dst_stride * 4)) & 15u) == 0;
    long work = (long)nw * nh;
    ztc::TraceScope tr("mip_f32", stream);
    ztc::trace_units((long)nw * nh);
    ztc::mip_f32_kernel<<<ztc::grid_for(work, 256), 256, 0, stream>>>(src, w, h, stride, dst, dst_stride, nw, nh, vec);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- batched: six levels of every texture per launch
cudaError_t ztc_launch_batch_mip(const ztc::MipChain *chains, const ztc::MipTile *tiles, int ntiles, cudaStream_t stream) {
    if (ntiles <= 0) return cudaSuccess;
    const int sms = ztc_sm_count();
    ztc::batch_mip_kernel<<<std::min(ntiles, sms * ztc::kMipCtas), ztc::kMipThreads, 0, stream>>>(chains, tiles, ntiles);
    return cudaGetLastError();
}
