// rdo.cu - rate-distortion encoding at lambda > 0 (zap_tex.h:223-306, :786-815) for sm_100a, bit-exact.
//
// The reference picks every sub-block among its own encoding and up to 48 candidates rebuilt from the 16 blocks
// chosen before it in the call's raster order (a neighbour's endpoints with refit indices, its indices with these
// endpoints, or the whole neighbour; for BC7: the whole neighbour, or for a mode-6 neighbour its endpoint bytes
// with refit indices or its index bytes with refit endpoints), minimising SSE + lambda * rate. The rate models
// zap's LZ on the split planes, per field: 0 if the field repeats the one at the current match distance,
// min(size, 3) for a new match in the window, its size in literals otherwise.
//
// Only that window makes the work serial. The base encodings do not depend on it, so the ordinary encoder kernels
// write them for every block first, in parallel. The chain then runs as one CTA per call (or per band of block
// rows: each band is its own call in the reference's banded callers; and per sub-block kind, whose chains are
// independent): per block, groups of lanes evaluate the candidates side by side, and a minimum of (cost, candidate
// order) picks the winner. That minimum is the
// reference's choice: its scan takes a candidate only if its cost is below the best so far (strict "<"), so it ends
// on the first candidate of the lowest cost, and its early "skip if SSE >= best" never changes that, because
// SSE + lambda * rate >= SSE in float arithmetic when lambda * rate >= 0 (finite lambda > 0: the entry points reject
// any other lambda). Costs are non-negative floats, whose bit patterns order like their values. The window of the
// last 16 chosen sub-blocks lives in shared memory; chosen blocks overwrite the base encodings in place.
#include "ztc_common.cuh"
#include "ztc_decode.cuh"
#include "ztc_internal.h"

namespace ztc {
namespace {

constexpr int kWindow = 16;          // ZAP_TEX_WINDOW (zap_tex.h:227)

enum SubType { kBc1 = 0, kBc4 = 1, kBc7 = 2 };
struct Sub {
    int type, chan, force4, off;  // chan: the BC4 channel; off: byte offset of the sub-block in the block
};
// the sub-blocks of a format's block, in the order the reference encodes them (zap_tex.h:1489-1503)
__host__ __device__ constexpr int sub_count(int fmt) { return fmt == ZTC_FMT_BC3 || fmt == ZTC_FMT_BC5 ? 2 : 1; }
__host__ __device__ constexpr Sub sub_of(int fmt, int s) {
    return fmt == ZTC_FMT_BC1   ? Sub{kBc1, 0, 0, 0}
           : fmt == ZTC_FMT_BC3 ? (s == 0 ? Sub{kBc4, 3, 0, 0} : Sub{kBc1, 0, 1, 8})
           : fmt == ZTC_FMT_BC4 ? Sub{kBc4, 0, 0, 0}
           : fmt == ZTC_FMT_BC5 ? (s == 0 ? Sub{kBc4, 0, 0, 0} : Sub{kBc4, 1, 0, 8})
                                : Sub{kBc7, 0, 0, 0};
}

// ---- BC4 sub-block (zap_tex.h:172-196): u8 a0, u8 a1, 3-bit indices; 6 values + 0 and 255 when a0 <= a1
ZTC_DEV int bc4_entry(int a0, int a1, int k) {
    // without branches on the entry (a warp's lanes build one each); the numerators are below 2^11
    const uint32_t n7 = (uint32_t)((8 - k) * a0 + (k - 1) * a1 + 3), n5 = (uint32_t)((6 - k) * a0 + (k - 1) * a1 + 2);
    const int six = k < 6 ? (int)(n5 / 5u) : k == 6 ? 0 : 255;
    return k == 0 ? a0 : k == 1 ? a1 : a0 > a1 ? (int)(n7 / 7u) : six;
}
// ---- BC7 mode-6 blocks (zap_tex.h:529)
ZTC_DEV bool is_mode6(uint64_t lo) { return (lo & 0x7Fu) == 0x40u; }
// mode-6 fields: q[e][c] 7 bits each (c-major), p-bits, 4-bit indices (texel 0: 3 bits) packed into idx, 4 bits each
__device__ __forceinline__ uint64_t key_of(float cost, int order) { return ((uint64_t)__float_as_uint(cost) << 32) | (uint32_t)order; }


// ---------------------------------------------------------------- BC7
// A BC7 candidate costs a whole palette search or least-squares solve, so this chain spreads each candidate over a
// group of L lanes: lane q takes texels q*T .. q*T + T - 1 (T = 16 / L), and the window slots at those distances
// minus one when the rate is counted. Groups 0-15 kind 1 (neighbour j = group + 1: its endpoints, refit indices),
// 16-31 kind 2 (its indices, refit endpoints), 32-47 kind 0 (the whole neighbour), 48 the base; a last warp loads the
// blocks ahead, software-pipelined like the BC1 / BC4 chains' loader (its own warp, so its global loads hold no
// candidate's minimum). Every chosen block enters the window with its decoded texels and, for mode 6, its palette
// (with 16 |p|^2 + k for entry k), indices and index weights, so no candidate decodes a block: kind 0 compares the
// texels with the stored decode, kind 1 searches the stored palette. The base encodings are decoded for every block
// by a parallel pass before the chains. Kind 2's least-squares sums are exact in the reference's float accumulation
// (weights k/64, texels integers: every partial sum is a multiple of 1/4096 below 2^17 of them), so they are integer
// dot products (the weights and the texels' channels a byte per texel), scaled, which gives the same floats in any
// order; its solve and quantisation are one (channel, endpoint) per lane, both p-bits.
//
// What bounds a chain is the length of a step, about 2200 cycles a block: kind 2 1900 of them, kind 1 1700, the others
// 1350-1500, the window's update 300. 512x512 in 8-row bands: the nearest values per parity by rule, end points and the
// first word gathered in two packed words instead of twelve exchanges, weights from the window (1531 -> 1395 us); the
// winner's window entries computed before the minimum and its group in the key, palette keys stored ready to subtract
// from (-> 1268); the collectives as below (-> 1213).

// Sums and ORs over a group of L lanes; gm: the lanes of the warp that meet them. In the BC7 chain that is every lane
// (the groups past the base's repeat it and never win), a mask known at compile time (512x512 in 8-row bands 1268 ->
// 1217 us, with one OR for both fields' match masks). In the BC1 / BC4 chains the idle groups do nothing: those two
// changes there measured BC1 726 -> 736 us next to BC3 1531 -> 1509. redux.sync for the group sums measured slower than
// shuffle trees (BC7 512x512 in one chain: 30.6 -> 47 ms). ZTC_RDO_MIN_REDUX selects redux.sync (1) or an xor-shuffle
// tree (0) for the warp-wide key minimum (BC7 as above: 1217 / 1365 us).
#ifndef ZTC_RDO_MIN_REDUX
#define ZTC_RDO_MIN_REDUX 1
#endif
constexpr unsigned kAll = 0xFFFFFFFFu;
template <int L> __device__ __forceinline__ int lsum(int v, unsigned gm = kAll) {
    #pragma unroll
    for (int m = L / 2; m >= 1; m >>= 1) v += __shfl_xor_sync(gm, v, m, L);
    return v;
}
template <int L> __device__ __forceinline__ uint32_t lor(uint32_t v, unsigned gm = kAll) {
    #pragma unroll
    for (int m = L / 2; m >= 1; m >>= 1) v |= __shfl_xor_sync(gm, v, m, L);
    return v;
}
// warp-wide minimum of 64-bit keys
__device__ __forceinline__ uint64_t warp_min_redux(uint64_t k) {
#if ZTC_RDO_MIN_REDUX  // the high words' minimum, then the low words' among the lanes holding it
    const uint32_t hi = __reduce_min_sync(0xFFFFFFFFu, (uint32_t)(k >> 32));
    const uint32_t lo = __reduce_min_sync(0xFFFFFFFFu, (uint32_t)(k >> 32) == hi ? (uint32_t)k : 0xFFFFFFFFu);
    return ((uint64_t)hi << 32) | lo;
#else  // xor-shuffle tree
    #pragma unroll
    for (int m = 16; m >= 1; m >>= 1) {
        const uint32_t lo = __shfl_xor_sync(0xFFFFFFFFu, (uint32_t)k, m), hi = __shfl_xor_sync(0xFFFFFFFFu, (uint32_t)(k >> 32), m);
        const uint64_t o = ((uint64_t)hi << 32) | lo;
        k = o < k ? o : k;
    }
    return k;
#endif
}
// squared RGBA difference (zap__sq4 over 4 channels) as |a|^2 + |b|^2 - 2 a.b, three dp4a; aa = |a|^2
ZTC_DEV int sq4px(uint32_t a, int aa, uint32_t b) { return aa + (int)dot4(b, b) - 2 * (int)dot4(a, b); }
ZTC_DEV uint32_t lerp_px(const int x0[4], const int x1[4], int w) {
    return pack_rgba(lerp64(x0[0], x1[0], w), lerp64(x0[1], x1[1], w), lerp64(x0[2], x1[2], w), lerp64(x0[3], x1[3], w));
}
// mode 6's first word from expanded endpoints, a byte per channel (the last bit of each byte is that endpoint's p-bit)
ZTC_DEV uint64_t mode6_lo(uint32_t X0, uint32_t X1) {
    const uint32_t a = (X0 >> 1) & 0x7F7F7F7Fu, b = (X1 >> 1) & 0x7F7F7F7Fu;
    const uint32_t rb = (a & 0x00FF00FFu) | ((b & 0x00FF00FFu) << 7), ga = ((a >> 8) & 0x00FF00FFu) | (((b >> 8) & 0x00FF00FFu) << 7);
    const uint32_t rg = (rb & 0xFFFFu) | ((ga & 0xFFFFu) << 14), ba = (rb >> 16) | ((ga >> 16) << 14);  // 28 bits each
    return ((uint64_t)((rg >> 25) | (ba << 3) | (X0 << 31)) << 32) | ((rg << 7) | 0x40u);
}
// mode 6 bit layout: mode bits 0-6, R0 R1 G0 G1 B0 B1 A0 A1 (7 bits each) from bit 7, P0 bit 63, P1 bit 64, then
// the indices (texel 0: 3 bits, the others 4) from bit 65
ZTC_DEV void mode6_ends_of(uint64_t lo, uint64_t hi, int x0[4], int x1[4]) {  // expanded endpoints
    const int p0 = (int)(lo >> 63), p1 = (int)(hi & 1u);
    #pragma unroll
    for (int c = 0; c < 4; c++) {
        x0[c] = (int)(((lo >> (7 + 14 * c)) & 0x7Fu) << 1) | p0;
        x1[c] = (int)(((lo >> (14 + 14 * c)) & 0x7Fu) << 1) | p1;
    }
}
ZTC_DEV uint64_t mode6_idx_of(uint64_t hi) { return ((hi >> 1) & 7u) | (hi & ~0xFull); }  // 4 bits per texel
ZTC_DEV uint64_t mode6_hi(int p1, uint64_t idx) { return (uint64_t)p1 | ((idx & 7u) << 1) | (idx & ~0xFull); }

// the base encodings of blocks [0, nblocks), decoded: 16 texels per block
__global__ void __launch_bounds__(128) bc7_decode_bases_kernel(const uint8_t *__restrict__ blocks, int nblocks, uint4 *__restrict__ dec) {
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    if (b >= nblocks) return;
    const uint4 v = *(const uint4 *)(blocks + (size_t)b * 16);
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    uint32_t px[16];
    dec::bc7_block(w, px);
    #pragma unroll
    for (int k = 0; k < 4; k++) dec[(size_t)b * 4 + k] = make_uint4(px[4 * k], px[4 * k + 1], px[4 * k + 2], px[4 * k + 3]);
}

// The loader warp's registers for one block: lane i < 16 its texel i and decoded base texel i, every lane the base.
struct Bc7Fetch {
    uint32_t tex = 0, dec = 0;
    uint64_t lo = 0, hi = 0;
    __device__ __forceinline__ void fetch(const SrcU8 &src, int bw, const uint8_t *out, const uint32_t *dec_base, int gk, int lane) {
        if (lane < 16) {
            tex = load_texel(src, min((gk % bw) * 4 + (lane & 3), src.w - 1), min((gk / bw) * 4 + (lane >> 2), src.h - 1));
            dec = dec_base[(size_t)gk * 16 + lane];
        }
        lo = *(const uint64_t *)(out + (size_t)gk * 16);
        hi = *(const uint64_t *)(out + (size_t)gk * 16 + 8);
    }
    // into slot ns: texels, decoded base, base, the base's mode-6 palette, and the texels by channel (byte i of
    // texc[c] is channel c of texel i, for the least-squares sums as dp4a)
    __device__ __forceinline__ void store(int lane, int ns, uint32_t (*s_tex)[16], uint32_t (*s_dbase)[16], uint64_t (*s_base)[2],
                                          uint32_t (*s_bpal)[16], uint32_t (*s_texc)[4][4]) const {
        if (lane < 16) {
            s_tex[ns][lane] = tex;
            s_dbase[ns][lane] = dec;
            int x0[4], x1[4];
            mode6_ends_of(lo, hi, x0, x1);
            s_bpal[ns][lane] = lerp_px(x0, x1, w4(lane));
            #pragma unroll
            for (int c = 0; c < 4; c++) ((uint8_t *)s_texc[ns][c])[lane] = (uint8_t)chan(tex, c);
        }
        if (lane < 2) s_base[ns][lane] = lane ? hi : lo;
    }
};

template <int L> struct B7Chain {  // kWc candidate warps, then the loader warp
    static constexpr int T = 16 / L, kWc = (49 * L + 31) / 32, kThreads = (kWc + 1) * 32;
};
#ifndef ZTC_RDO_BC7_LANES
#define ZTC_RDO_BC7_LANES 8
#endif

template <int L>
__global__ void __launch_bounds__(B7Chain<L>::kThreads, 1) rdo_bc7_chain_kernel(SrcU8 src, int bw, int nby, int chain_rows, uint8_t *__restrict__ out,
                                                                                const uint32_t *__restrict__ dec_base, float lambda) {
    static_assert(L >= 8, "a lane per (channel, endpoint) of a least-squares candidate");
    constexpr int T = B7Chain<L>::T, kW = B7Chain<L>::kWc;
    __shared__ uint64_t ring[kWindow][2];       // the last 16 chosen blocks, slot = block & 15
    __shared__ uint32_t ring_dec[kWindow][16];  // their decoded texels
    __shared__ __align__(16) uint32_t ring_pal[kWindow][16];  // mode 6: their palettes
    __shared__ __align__(16) int ring_pp[kWindow][16];        // and 16 |p|^2 + k for entry k
    __shared__ uint64_t ring_idx[kWindow];      // mode 6: their indices, 4 bits per texel
    __shared__ __align__(16) uint32_t ring_wp[kWindow][4];  // mode 6: their index weights w4(idx), a byte per texel
    __shared__ uint32_t s_tex[3][16], s_dbase[3][16];  // block cur in slot cur % 3, loaded two blocks ahead
    __shared__ uint64_t s_base[3][2];
    __shared__ uint32_t s_bpal[3][16];                 // the base's palette, if mode 6
    __shared__ __align__(16) uint32_t s_texc[3][4][4];  // the block's texels by channel, a byte per texel
    __shared__ uint64_t s_key[kW];
    __shared__ int s_dist[2];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = tid & (L - 1), grp = tid / L;
    const bool loader = warp == kW;
    // the warps of groups 0-47 hold one kind each; the groups from 48 on all evaluate the base, for group 48
    const int kind = loader ? -2 : grp < 16 ? 1 : grp < 32 ? 2 : grp < 48 ? 0 : -1, j = (grp & 15) + 1;
    const int row0 = blockIdx.x * chain_rows, rows = min(chain_rows, nby - row0);
    if (rows <= 0) return;
    const int first = row0 * bw, count = rows * bw;
    Bc7Fetch fb;
    if (loader) {
        for (int k = 0; k < 2 && k < count; k++) {
            fb.fetch(src, bw, out, dec_base, first + k, lane);
            fb.store(lane, k, s_tex, s_dbase, s_base, s_bpal, s_texc);
        }
        if (count > 2) fb.fetch(src, bw, out, dec_base, first + 2, lane);
    }
    if (tid == 0) { s_dist[0] = 1; s_dist[1] = 1; }
    __syncthreads();
    for (int cur = 0; cur < count; cur++) {
        const int g = first + cur, slot = cur % 3, d0 = s_dist[0], d1 = s_dist[1];
        uint64_t key = ~0ull, clo = 0, chi = 0, cidx = 0;
        uint32_t dec[T];  // the candidate's decode of this lane's texels
        int nd0 = 0, nd1 = 0;
        uint32_t pal[T], wt[T];  // entries q T + u of the candidate's mode-6 palette, and its texels' index weights
        const int r = (cur - j) & (kWindow - 1);
        if (kind >= -1) {
            uint32_t t[T];
            int tt[T];
            #pragma unroll
            for (int u = 0; u < T; u++) { t[u] = s_tex[slot][q * T + u]; tt[u] = (int)dot4(t[u], t[u]); }
            bool ok;
            int e = 0;
            if (kind == -1) {  // the base (its SSE: the one the reference's encoder returns)
                clo = s_base[slot][0]; chi = s_base[slot][1];
                #pragma unroll
                for (int u = 0; u < T; u++) { dec[u] = s_dbase[slot][q * T + u]; e += sq4px(t[u], tt[u], dec[u]); }
                e = lsum<L>(e);
                cidx = mode6_idx_of(chi);
                #pragma unroll
                for (int u = 0; u < T; u++) { pal[u] = s_bpal[slot][q * T + u]; wt[u] = (uint32_t)w4((int)((cidx >> (4 * (q * T + u))) & 15u)); }
                ok = true;
            } else if (kind == 0) {  // the whole neighbour (zap__bc7_err)
                clo = ring[r][0]; chi = ring[r][1]; cidx = ring_idx[r];
                #pragma unroll
                for (int u = 0; u < T; u++) {
                    dec[u] = ring_dec[r][q * T + u]; e += sq4px(t[u], tt[u], dec[u]);
                    pal[u] = ring_pal[r][q * T + u]; wt[u] = ((const uint8_t *)ring_wp[r])[q * T + u];
                }
                e = lsum<L>(e);
                ok = j <= cur;
            } else if (kind == 1) {  // its endpoints, best indices; texel 0 keeps to 0..7 (zap__bc7_fit6_idx)
                const uint64_t nlo = ring[r][0], nhi = ring[r][1];
                ok = j <= cur && is_mode6(nlo);
                uint64_t bits = 0;
                #pragma unroll
                for (int u = 0; u < T; u++) {
                    // key 16 (|p|^2 - 2 t.p) + k per entry (its minimum is the first nearest entry), minimised as a tree
                    const int i = q * T + u;
                    int kk[16];
                    #pragma unroll
                    for (int k4 = 0; k4 < 4; k4++) {
                        const uint4 pk = *(const uint4 *)&ring_pal[r][4 * k4];
                        const int4 pp = *(const int4 *)&ring_pp[r][4 * k4];
                        kk[4 * k4 + 0] = pp.x - 32 * (int)dot4(t[u], pk.x);
                        kk[4 * k4 + 1] = pp.y - 32 * (int)dot4(t[u], pk.y);
                        kk[4 * k4 + 2] = pp.z - 32 * (int)dot4(t[u], pk.z);
                        kk[4 * k4 + 3] = pp.w - 32 * (int)dot4(t[u], pk.w);
                    }
                    if (i == 0) {  // the anchor texel's index has 3 bits
                        #pragma unroll
                        for (int k = 8; k < 16; k++) kk[k] = 0x7FFFFFFF;
                    }
                    #pragma unroll
                    for (int h = 8; h >= 1; h >>= 1)
                        #pragma unroll
                        for (int k = 0; k < h; k++) kk[k] = min(kk[k], kk[k + h]);
                    dec[u] = ring_pal[r][kk[0] & 15];
                    e += (kk[0] >> 4) + tt[u];
                    bits |= (uint64_t)(kk[0] & 15) << (4 * i);
                    pal[u] = ring_pal[r][i]; wt[u] = (uint32_t)w4(kk[0] & 15);
                }
                e = lsum<L>(e);
                cidx = ((uint64_t)lor<L>((uint32_t)(bits >> 32)) << 32) | lor<L>((uint32_t)bits);
                clo = nlo; chi = mode6_hi((int)(nhi & 1u), cidx);
            } else {  // its indices, least-squares endpoints, each endpoint's own p-bit (zap__bc7_fit6_ep)
                const uint64_t nlo = ring[r][0], nhi = ring[r][1];
                ok = j <= cur && is_mode6(nlo);
                cidx = ring_idx[r];
                const int task = q & 7, ch = task >> 1, ep = task & 1;  // this lane's (channel, endpoint)
                // the neighbour's weights and this block's channel ch, a byte per texel: sum w, sum w^2 and sum w x
                // are four dp4a each; with u = 64 - w: sum u^2 = 16 * 4096 - 128 sum w + sum w^2,
                // sum u w = 64 sum w - sum w^2, sum u x = 64 sum x - sum w x
                const uint4 wp = *(const uint4 *)ring_wp[r], xc = *(const uint4 *)s_texc[slot][ch];
                const int W1 = (int)__dp4a(wp.w, 0x01010101u, __dp4a(wp.z, 0x01010101u, __dp4a(wp.y, 0x01010101u, dot4(wp.x, 0x01010101u))));
                const int W2 = (int)__dp4a(wp.w, wp.w, __dp4a(wp.z, wp.z, __dp4a(wp.y, wp.y, dot4(wp.x, wp.x))));
                const int SB = (int)__dp4a(wp.w, xc.w, __dp4a(wp.z, xc.z, __dp4a(wp.y, xc.y, dot4(wp.x, xc.x))));
                const int SX = (int)__dp4a(xc.w, 0x01010101u, __dp4a(xc.z, 0x01010101u, __dp4a(xc.y, 0x01010101u, dot4(xc.x, 0x01010101u))));
                const int AA = 16 * 4096 - 128 * W1 + W2, AB = 64 * W1 - W2, BB = W2, SA = 64 * SX - SB;
                const float aa = (float)AA / 4096.0f, ab = (float)AB / 4096.0f, bb = (float)BB / 4096.0f;
                const float ax = (float)SA / 64.0f, bx = (float)SB / 64.0f, det = aa * bb - ab * ab;
                float v;
                if (det < 1e-6f && det > -1e-6f) v = (ax + bx) / 16.0f;  // one index everywhere: flat
                else v = ep ? (bx * aa - ax * ab) / det : (ax * bb - bx * ab) / det;
                v = clamp255(v);
                // zap__bc7q for this (channel, endpoint), 7 bits + p, for both p-bits
                uint32_t bq[2][4];
                int be[2];
                quant8_pbits<1>(&v, bq, be);
                // each endpoint's errors over the four channels, both p-bits in one word (each below 2^16: a
                // candidate lies within 2 of v); the endpoint keeps the p-bit of the smaller sum, p = 0 on ties
                int s2 = be[0] | (be[1] << 16);
                s2 += __shfl_xor_sync(kAll, s2, 2, L);
                s2 += __shfl_xor_sync(kAll, s2, 4, L);
                const uint32_t pbm = (s2 >> 16) < (s2 & 0xFFFF) ? 1u : 0u, qm = (pbm ? bq[1][0] : bq[0][0]) & 127u;
                // the expanded endpoints gathered a byte per channel: X0 the first, X1 the second
                uint32_t X = ((qm << 1) | pbm) << (8 * ch);
                X |= __shfl_xor_sync(kAll, X, 2, L);
                X |= __shfl_xor_sync(kAll, X, 4, L);
                const uint32_t Y = __shfl_xor_sync(kAll, X, 1, L), X0 = ep ? Y : X, X1 = ep ? X : Y;
                const Lerp4 fit(X0, X1);
                #pragma unroll
                for (int u = 0; u < T; u++) {
                    wt[u] = ((const uint8_t *)ring_wp[r])[q * T + u];
                    dec[u] = fit.at((int)wt[u]); pal[u] = fit.at(w4(q * T + u));
                    e += sq4px(t[u], tt[u], dec[u]);
                }
                const uint32_t pb1 = X1 & 1u;
                const uint64_t lo = mode6_lo(X0, X1);
                e = lsum<L>(e);
                clo = lo; chi = (nhi & ~1ull) | pb1;
            }
            // rate (zap__bc7_rate): bit d - 1 of a mask says the field equals the window's at distance d
            uint32_t m2 = 0;  // the two fields' masks in one word's halves
            #pragma unroll
            for (int u = 0; u < T; u++) {
                const int d = q * T + u + 1, rw = (cur - d) & (kWindow - 1);
                if (d <= cur) m2 |= (((uint32_t)(ring[rw][0] == clo)) | ((uint32_t)((ring[rw][1] >> 8) == (chi >> 8)) << 16)) << (d - 1);
            }
            m2 = lor<L>(m2);
            const uint32_t mA = m2 & 0xFFFFu, mB = m2 >> 16;
            float fa = 8.0f, fb = 7.0f;
            nd0 = d0; nd1 = d1;
            if (d0 > 0 && d0 <= cur && ((mA >> (d0 - 1)) & 1u)) fa = 0.0f;
            else if (mA) { nd0 = __ffs((int)mA); fa = 3.0f; }
            if (d1 > 0 && d1 <= cur && ((mB >> (d1 - 1)) & 1u)) fb = 0.0f;
            else if (mB) { nd1 = __ffs((int)mB); fb = 3.0f; }
            // the order, then the group that holds the candidate
            if (ok) key = key_of((float)e + lambda * (fa + fb + 1.0f), (kind < 0 ? 0 : (j - 1) * 3 + kind + 1) << 8 | grp);
        } else if (loader) {  // block cur + 2 (fetched the iteration before) to shared memory; fetch block cur + 3
            if (cur + 2 < count) fb.store(lane, (cur + 2) % 3, s_tex, s_dbase, s_base, s_bpal, s_texc);
            if (cur + 3 < count) fb.fetch(src, bw, out, dec_base, g + 3, lane);
        }
        if (!loader) {
            const uint64_t wk = warp_min_redux(key);
            if (lane == 0) s_key[warp] = wk;
        }
        __syncthreads();
        const int won = loader ? -1 : (int)((uint32_t)warp_min_redux(lane < kW ? s_key[lane] : ~0ull) & 0xFFu);
        if (grp == won) {  // the winner enters the window (with j = 16 its slot is the one it read; all it writes was read before the barrier)
            const int ws = cur & (kWindow - 1);
            #pragma unroll
            for (int u = 0; u < T; u++) {
                const int i = q * T + u;
                ring_dec[ws][i] = dec[u];
                ring_pal[ws][i] = pal[u];
                ring_pp[ws][i] = 16 * (int)dot4(pal[u], pal[u]) + i;
                ((uint8_t *)ring_wp[ws])[i] = (uint8_t)wt[u];
            }
            if (q == 0) {
                ring[ws][0] = clo; ring[ws][1] = chi; ring_idx[ws] = cidx;
                s_dist[0] = nd0; s_dist[1] = nd1;
                if (kind >= 0) { *(uint64_t *)(out + (size_t)g * 16) = clo; *(uint64_t *)(out + (size_t)g * 16 + 8) = chi; }
            }
        }
        __syncthreads();
    }
}

// Word k of a sub-block's palette as the chain keeps it in shared memory: BC1 entries 0-3 as RGB texels (alpha
// byte 0), then words 4-7 their squared norms |p|^2, so a texel's squared distance to entry k is
// |t|^2 + |p_k|^2 - 2 t.p_k with t.p_k one dp4a; BC4 its 8 values. Each chosen sub-block enters the window with its
// palette and the loader builds each block's base palette two blocks ahead, so no candidate builds one.
ZTC_DEV int palette_word(const Sub &S, uint64_t v, int k) {
    if (S.type == kBc1) {  // (zap_tex.h:52-94: 3 colours and transparent when c0 <= c1) without branches on the entry: the loader's lanes build one word each
        const uint32_t c0 = (uint32_t)(v & 0xFFFFu), c1 = (uint32_t)((v >> 16) & 0xFFFFu);
        const bool four = S.force4 || c0 > c1;
        int a[3], b[3];
        unpack565(c0, a[0], a[1], a[2]); unpack565(c1, b[0], b[1], b[2]);
        const int e = k & 3, wa = e == 0 ? 6 : e == 1 ? 0 : four ? (e == 2 ? 4 : 2) : 3;  // sixths of the first endpoint
        uint32_t p = 0;
        #pragma unroll
        for (int c = 0; c < 3; c++) p |= (uint32_t)((a[c] * wa + b[c] * (6 - wa) + (e < 2 ? 0 : four ? 2 : 3)) / 6) << (8 * c);
        if (e == 3 && !four) p = 0;
        return k < 4 ? (int)p : (int)dot4(p, p);
    }
    return bc4_entry((int)(v & 0xFFu), (int)((v >> 8) & 0xFFu), k);
}

// ---------------------------------------------------------------- BC1 / BC4 sub-blocks
// One chain per CTA and sub-block kind, in two roles. The candidates of a block that do not involve the block
// chosen just before it (the base, and every neighbour at distance j >= 2) depend only on decisions at least two
// blocks back, so producer warps evaluate them one block ahead: while block b - 1 is being chosen, they compute
// block b's candidates (SSE, fields, and the match masks against window distances 2..16) into shared memory. The
// chooser then decides block b alone: three warps evaluate the three candidates of neighbour distance 1, one kind
// each, down to their costs (sub_near), while the deciding warp adds the distance-1 match bit to the 46 others and turns
// their masks into costs; a named barrier over the four joins them, and the deciding warp takes the minimum of (cost,
// candidate order). One barrier per block; no CTA-wide minimum. The producers' candidates are evaluated by groups of L
// lanes, lane q taking 16 / L texels and as many window distances. Producer groups: 0-15 kind 0 (neighbour j =
// (group & 15) + 2: its endpoints, fitted indices), 16-31 kind 1 (these endpoints, its indices), 32-47 kind 2 (the
// whole neighbour), the last group of each kind idle (it repeats j = 16 and keeps nothing), 48 the base; a last warp
// loads the blocks ahead (block b + 2 stored while block b + 4 is fetched into registers). The two sub-blocks of a
// BC3 or BC5 block are independent chains (each looks only at its own fields of earlier blocks, with its own match
// distances, zap_tex.h:1494-1501), so each runs in its own CTA (blockIdx.y) and writes its own 8 bytes of the blocks.
//
// What bounds a chain is the length of a step: with a 1021x767 BC3 texture in 8-row bands (2048 blocks a chain), 2100 cycles
// a block, the deciding warp's two keys per lane 1400 of them, next to one warp for two distance-1 kinds (1230 after the
// keys were shortened) and a loader that waited for its own load (1500). Now about 1350, producers, deciding warp and
// loader within a tenth of each other: field sizes known at compile time (-4 %), costs without the next match
// distances, distance-1 candidates on 16 lanes with one reduction or vote per sum and mask (-22 % more), a warp per kind
// and loads two blocks ahead (-9 %), palettes without branches on the entry (-5 %): 2.375 -> 1.53 ms.
// A chain's warps at L lanes per producer candidate: producers, then the deciding warp, the three distance-1 warps and the
// loader. BC1 chains take 4 lanes, launches with a BC4 chain 8: 512x512 in 8-row bands BC1 0.726 / 0.757 ms at 4 / 8, BC3
// 0.796 / 0.757.
template <int L>
struct SubRoles {
    static constexpr int kProducers = (49 * L + 31) / 32, kDecide = kProducers, kNear = kDecide + 1, kLoader = kNear + 3, kThreads = (kLoader + 1) * 32;
};

struct SubCand {
    int e;
    uint64_t cand;
    bool ok;
    uint32_t mA, mB;  // bit d - 1: the field equals the window's at distance d (from distance dlo on)
};

// One candidate of chain block b on a group of L lanes (gm: the lanes that meet its collectives). kind -1: the base;
// 0: neighbour j's endpoints with fitted indices; 1: the base's endpoints with neighbour j's indices; 2: the whole
// neighbour j. Its window masks cover distances dlo..16 (up to b).
template <bool bc1, int L>
__device__ __forceinline__ SubCand sub_candidate(const Sub &S, int kind, int j, int b, int q, unsigned gm, int dlo,
                                                 const uint32_t (*s_tex)[16], const uint64_t *s_base, const int (*s_bpal)[8],
                                                 const uint64_t *ring, const int (*ring_pal)[8]) {
    constexpr int T = 16 / L, nA = bc1 ? 4 : 2;
    constexpr uint64_t maskA = (1ull << (8 * nA)) - 1ull;
    const int slot = b % 3;
    uint32_t t[T];
    #pragma unroll
    for (int u = 0; u < T; u++) t[u] = s_tex[slot][q * T + u];
    const uint64_t base = s_base[slot], nb = ring[(b - j) & (kWindow - 1)];
    // kind 1 and the base: these endpoints (the base's palette); kinds 0 and 2: the neighbour's
    const bool own = kind == 1 || kind == -1;
    const int *P = own ? s_bpal[slot] : ring_pal[(b - j) & (kWindow - 1)];
    SubCand r;
    r.ok = kind == -1 || j <= b;
    int e = 0;
    if (bc1) {  // the CTA's sub-block type: uniform
        const uint32_t a = (uint32_t)((own ? base : nb) & 0xFFFFu), c = (uint32_t)(((own ? base : nb) >> 16) & 0xFFFFu);
        uint32_t idx;
        if (kind == 0) {  // zap__bc1_fit: best of the 4 (3 in 3-colour order) entries, first on ties
            const int4 pe = *(const int4 *)P, pn = *(const int4 *)(P + 4);
            const bool n4 = S.force4 || a > c;
            idx = 0;
            #pragma unroll
            for (int u = 0; u < T; u++) {
                const uint32_t tc = t[u] & 0xFFFFFFu;
                // 4 (|p|^2 - 2 t.p) + entry: its least is the first nearest entry
                const int k0 = 4 * (pn.x - 2 * (int)dot4(tc, (uint32_t)pe.x)), k1 = 4 * (pn.y - 2 * (int)dot4(tc, (uint32_t)pe.y)) + 1;
                const int k2 = 4 * (pn.z - 2 * (int)dot4(tc, (uint32_t)pe.z)) + 2, k3 = 4 * (pn.w - 2 * (int)dot4(tc, (uint32_t)pe.w)) + 3;
                int m = min(min(k0, k1), k2);
                if (n4) m = min(m, k3);
                e += (m >> 2) + (int)dot4(tc, tc);
                idx |= ((uint32_t)m & 3u) << (2 * (q * T + u));
            }
            e = lsum<L>(e, gm);
            idx = lor<L>(idx, gm);
        } else {  // zap__bc1_eval with the base's or the neighbour's indices
            idx = (uint32_t)((kind == -1 ? base : nb) >> 32);
            #pragma unroll
            for (int u = 0; u < T; u++) {
                const uint32_t tc = t[u] & 0xFFFFFFu;
                const int k = (int)((idx >> (2 * (q * T + u))) & 3u);
                e += P[4 + k] - 2 * (int)dot4(tc, (uint32_t)P[k]) + (int)dot4(tc, tc);
            }
            e = lsum<L>(e, gm);
        }
        r.cand = (uint64_t)a | ((uint64_t)c << 16) | ((uint64_t)idx << 32);
        // a 3-colour block may not use index 3 (transparent); the base is never checked
        if (kind >= 0 && !S.force4 && a <= c && (idx & (idx >> 1) & 0x55555555u)) r.ok = false;
    } else {
        const int a = (int)((own ? base : nb) & 0xFFu), c = (int)(((own ? base : nb) >> 8) & 0xFFu);
        uint64_t idx;
        if (kind == 0) {  // zap__bc4_fit
            const int4 p0 = *(const int4 *)P, p1 = *(const int4 *)(P + 4);
            const int pv[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
            uint32_t part = 0;  // this lane's T 3-bit indices
            #pragma unroll
            for (int u = 0; u < T; u++) {
                const int v = (int)chan(t[u], S.chan);
                int m = 0x7FFFFFFF;  // 8 squared distance + entry: its least is the first nearest entry
                #pragma unroll
                for (int k = 0; k < 8; k++) m = min(m, (v - pv[k]) * (v - pv[k]) * 8 + k);
                e += m >> 3;
                part |= ((uint32_t)m & 7u) << (3 * u);
            }
            e = lsum<L>(e, gm);
            // lane q's indices start at bit 3 q T: two 32-bit words of the 48
            const uint64_t mine = (uint64_t)part << (3 * q * T);
            idx = ((uint64_t)lor<L>((uint32_t)(mine >> 32), gm) << 32) | lor<L>((uint32_t)mine, gm);
        } else {  // zap__bc4_eval
            idx = (kind == -1 ? base : nb) >> 16;
            #pragma unroll
            for (int u = 0; u < T; u++) {
                const int d = (int)chan(t[u], S.chan) - P[(int)((idx >> (3 * (q * T + u))) & 7u)];
                e += d * d;
            }
            e = lsum<L>(e, gm);
        }
        r.cand = (uint64_t)a | ((uint64_t)c << 8) | (idx << 16);
    }
    r.e = e;
    // rate inputs (zap__field_rate per field): which window fields equal this candidate's
    uint32_t mA = 0, mB = 0;
    #pragma unroll
    for (int u = 0; u < T; u++) {
        const int d = q * T + u + 1;
        const uint64_t w = ring[(b - d) & (kWindow - 1)];
        if (d >= dlo && d <= b) {
            mA |= (uint32_t)((w & maskA) == (r.cand & maskA)) << (d - 1);
            mB |= (uint32_t)((w >> (8 * nA)) == (r.cand >> (8 * nA))) << (d - 1);
        }
    }
    r.mA = lor<L>(mA, gm);
    r.mB = lor<L>(mB, gm);
    return r;
}

// the rate of a candidate (zap__field_rate per field) and its cost's bits (non-negative floats order like them);
// mA, mB: its match masks, complete; d0, d1: the current match distances (bits past the window's blocks are never set)
template <bool bc1>
__device__ __forceinline__ uint32_t sub_cost(int e, uint32_t mA, uint32_t mB, int d0, int d1, float lambda) {
    constexpr float sizeA = bc1 ? 4.0f : 2.0f, sizeB = bc1 ? 4.0f : 6.0f, newA = bc1 ? 3.0f : 2.0f, newB = 3.0f;  // new: min(size, 3)
    const float fa = ((mA >> (d0 - 1)) & 1u) ? 0.0f : mA ? newA : sizeA, fb = ((mB >> (d1 - 1)) & 1u) ? 0.0f : mB ? newB : sizeB;
    return e >= 0 ? __float_as_uint((float)e + lambda * (fa + fb)) : ~0u;
}

// A candidate of neighbour distance 1 of chain block b on 16 lanes, one texel and one window distance each: the chain's
// longest path runs through it, so its sums and masks are one reduction or vote each instead of shuffle trees (lanes 0-15 of
// a warp, l the lane). Kinds as in sub_candidate; cost: see sub_cost.
template <bool bc1>
__device__ __forceinline__ void sub_near(const Sub &S, int kind, int b, int l, const uint32_t (*s_tex)[16], const uint64_t *s_base,
                                         const int (*s_bpal)[8], const uint64_t *ring, const int (*ring_pal)[8], int d0, int d1, float lambda,
                                         uint64_t &cand, uint32_t &cost, uint32_t &masks) {
    constexpr int nA = bc1 ? 4 : 2;
    constexpr uint64_t maskA = (1ull << (8 * nA)) - 1ull;
    constexpr unsigned gm = 0xFFFFu;
    const int slot = b % 3, d = l + 1;
    const uint32_t t = s_tex[slot][l];
    const uint64_t base = s_base[slot], nb = ring[(b - 1) & (kWindow - 1)], w = ring[(b - d) & (kWindow - 1)];
    const bool own = kind == 1;
    const int *P = own ? s_bpal[slot] : ring_pal[(b - 1) & (kWindow - 1)];
    bool ok = b >= 1;
    int e;
    if (bc1) {
        const uint32_t a = (uint32_t)((own ? base : nb) & 0xFFFFu), c = (uint32_t)(((own ? base : nb) >> 16) & 0xFFFFu), tc = t & 0xFFFFFFu;
        uint32_t idx = (uint32_t)(nb >> 32);
        if (kind == 0) {  // zap__bc1_fit
            const int4 pe = *(const int4 *)P, pn = *(const int4 *)(P + 4);
            const int k0 = 4 * (pn.x - 2 * (int)dot4(tc, (uint32_t)pe.x)), k1 = 4 * (pn.y - 2 * (int)dot4(tc, (uint32_t)pe.y)) + 1;
            const int k2 = 4 * (pn.z - 2 * (int)dot4(tc, (uint32_t)pe.z)) + 2, k3 = 4 * (pn.w - 2 * (int)dot4(tc, (uint32_t)pe.w)) + 3;
            int m = min(min(k0, k1), k2);
            if (S.force4 || a > c) m = min(m, k3);
            e = (m >> 2) + (int)dot4(tc, tc);
            idx = __reduce_or_sync(gm, ((uint32_t)m & 3u) << (2 * l));
        } else {  // zap__bc1_eval
            const int k = (int)((idx >> (2 * l)) & 3u);
            e = P[4 + k] - 2 * (int)dot4(tc, (uint32_t)P[k]) + (int)dot4(tc, tc);
        }
        cand = (uint64_t)a | ((uint64_t)c << 16) | ((uint64_t)idx << 32);
        if (!S.force4 && a <= c && (idx & (idx >> 1) & 0x55555555u)) ok = false;  // index 3 is transparent there
    } else {
        const int v = (int)chan(t, S.chan);
        const uint32_t ac = (uint32_t)(own ? base : nb) & 0xFFFFu;
        uint64_t idx = nb >> 16;
        if (kind == 0) {  // zap__bc4_fit
            const int4 p0 = *(const int4 *)P, p1 = *(const int4 *)(P + 4);
            const int pv[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
            int m = 0x7FFFFFFF;
            #pragma unroll
            for (int k = 0; k < 8; k++) m = min(m, (v - pv[k]) * (v - pv[k]) * 8 + k);
            e = m >> 3;
            const uint64_t mine = (uint64_t)((uint32_t)m & 7u) << (3 * l);
            idx = ((uint64_t)__reduce_or_sync(gm, (uint32_t)(mine >> 32)) << 32) | __reduce_or_sync(gm, (uint32_t)mine);
        } else {  // zap__bc4_eval
            const int x = v - P[(int)((idx >> (3 * l)) & 7u)];
            e = x * x;
        }
        cand = (uint64_t)ac | (idx << 16);
    }
    e = __reduce_add_sync(gm, e);
    const uint32_t mA = __ballot_sync(gm, d <= b && (w & maskA) == (cand & maskA)) & 0xFFFFu;
    const uint32_t mB = __ballot_sync(gm, d <= b && (w >> (8 * nA)) == (cand >> (8 * nA))) & 0xFFFFu;
    masks = mA | (mB << 16);
    cost = sub_cost<bc1>(ok ? e : -1, mA, mB, d0, d1, lambda);
}

// The deciding warp and the three distance-1 warps meet here, after branches that part a warp's lanes: the form that does not
// ask for converged warps (bar.sync is the aligned one, undefined where a warp's lanes arrive apart).
__device__ __forceinline__ void near_barrier() { asm volatile("barrier.sync 1, 128;" ::: "memory"); }

struct SubShared {
    uint64_t ring[kWindow];  // the sub-block of the last 16 chosen blocks, slot = block & 15
    __align__(16) int ring_pal[kWindow][8];  // their palettes (palette_word)
    __align__(16) uint32_t tex[3][16];  // block b in slot b % 3
    uint64_t base[3];
    __align__(16) int bpal[3][8];  // the base sub-block's palette
    // the candidates of block b by candidate order (0 the base, (j - 1) * 3 + kind + 1 the others), buffer b & 1
    uint64_t cand[2][49];
    uint64_t meta[2][49];  // SSE (bit 31 set: not allowed) | mA << 32 | mB << 48
    uint2 near_cost[3];    // the distance-1 candidates' costs and masks (mA | mB << 16)
    int dist[2];           // the current match distances (zap_tex.h:234)
};
// the chain of one sub-block kind, whose field sizes are known at compile time (the CTA's kind is uniform)
template <bool bc1, int L>
__device__ __forceinline__ void sub_chain(SubShared &M, const Sub S, const SrcU8 &src, int bw, int nby, int chain_rows, uint8_t *__restrict__ out, int bs,
                                          float lambda) {
    using R = SubRoles<L>;
    auto &ring = M.ring;
    auto &ring_pal = M.ring_pal;
    auto &s_tex = M.tex;
    auto &s_base = M.base;
    auto &s_bpal = M.bpal;
    auto &c_cand = M.cand;
    auto &c_meta = M.meta;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, q = tid & (L - 1), grp = tid / L;
    const int row0 = blockIdx.x * chain_rows, rows = min(chain_rows, nby - row0);
    if (rows <= 0) return;
    const int first = row0 * bw, count = rows * bw;
    // the loader warp: lane i < 16 fetches texel i of a block, every lane its base sub-block; a fetched block waits a whole
    // step in registers before it is stored, so a load has that long to arrive
    struct Fetched {
        uint32_t tex;
        uint64_t base;
    };
    int fx = 0, fy = 0;  // the block row and column of the next fetch
    auto fetch = [&]() {
        Fetched f{0u, 0ull};
        if (lane < 16) f.tex = load_texel(src, min(fx * 4 + (lane & 3), src.w - 1), min((row0 + fy) * 4 + (lane >> 2), src.h - 1));
        f.base = *(const uint64_t *)(out + (size_t)(first + fy * bw + fx) * bs + S.off);
        if (++fx == bw) { fx = 0; fy++; }
        return f;
    };
    auto store = [&](const Fetched &f, int ns) {  // the fetched block into slot ns, with the base's palette
        if (lane < 16) s_tex[ns][lane] = f.tex;
        if (lane < 8) s_bpal[ns][lane] = palette_word(S, f.base, lane);
        if (lane == 0) s_base[ns] = f.base;
    };
    Fetched f0{0u, 0ull}, f1{0u, 0ull};  // the next two blocks to store
    if (tid == 0) { M.dist[0] = 1; M.dist[1] = 1; }
    if (warp == R::kLoader) {
        store(fetch(), 0);
        if (count > 1) f0 = fetch();
        if (count > 2) f1 = fetch();
    }
    __syncthreads();
    // producers: kind and neighbour distance of the group (the idle groups repeat j = 16), which warps hold one kind
    const int pkind = grp < 48 ? grp >> 4 : grp == 48 ? -1 : -3, pj = min((grp & 15) + 2, 16);
    const unsigned pgm = warp < 48 * L / 32 ? kAll : ((1u << L) - 1u) << (lane & ~(L - 1));
    const bool pkeep = grp < 48 ? (grp & 15) < 15 : grp == 48;
    constexpr int nA = bc1 ? 4 : 2;
    constexpr uint64_t maskA = (1ull << (8 * nA)) - 1ull;
    int d0 = 1, d1 = 1;  // the deciding warp's current match distances (zap_tex.h:234)
    for (int it = -1; it < count; it++) {
        const int b = it + 1;  // the producers' block
        if (warp < R::kProducers) {
            if (pkind >= -1 && b < count) {
                const SubCand c = sub_candidate<bc1, L>(S, pkind, pj, b, q, pgm, 2, s_tex, s_base, s_bpal, ring, ring_pal);
                if (pkeep && q == 0) {
                    const int o = pkind < 0 ? 0 : (pj - 1) * 3 + pkind + 1;
                    c_cand[b & 1][o] = c.cand;
                    c_meta[b & 1][o] = (uint32_t)c.e | (c.ok ? 0u : 0x80000000u) | ((uint64_t)c.mA << 32) | ((uint64_t)c.mB << 48);
                }
            }
        } else if (warp >= R::kNear && warp < R::kNear + 3) {
            // the candidates of neighbour distance 1 (block it - 1, chosen in the previous step), down to their costs: one
            // kind per warp, on its lanes 0-15
            if (it >= 0) {
                const int ck = warp - R::kNear;
                if (lane < 16) {
                    uint64_t cand;
                    uint32_t cost, masks;
                    sub_near<bc1>(S, ck, it, lane, s_tex, s_base, s_bpal, ring, ring_pal, M.dist[0], M.dist[1], lambda, cand, cost, masks);
                    if (lane == 0) { c_cand[it & 1][ck + 1] = cand; M.near_cost[ck] = make_uint2(cost, masks); }
                }
                near_barrier();  // with the deciding warp
            }
        } else if (warp == R::kDecide) {
            if (it >= 0) {
                const int cur = it, bi = cur & 1;
                const uint64_t w1 = ring[(cur - 1) & (kWindow - 1)];  // the block chosen in the previous step
                // candidate o's cost, the window's distance-1 bits added to the producers' masks
                auto consider = [&](int o, uint32_t &masks) -> uint32_t {
                    const uint64_t cand = c_cand[bi][o], meta = c_meta[bi][o];
                    const uint32_t near_bits = cur < 1 ? 0u : (uint32_t)((w1 & maskA) == (cand & maskA)) | ((uint32_t)((w1 >> (8 * nA)) == (cand >> (8 * nA))) << 16);
                    masks = (uint32_t)(meta >> 32) | near_bits;
                    return sub_cost<bc1>((int)(uint32_t)meta, masks & 0xFFFFu, masks >> 16, d0, d1, lambda);
                };
                uint32_t masks, order = lane == 0 ? 0u : (uint32_t)lane + 3u;  // the base and orders 4..34
                uint32_t cost = consider((int)order, masks);
                if (lane + 35 < 49) {  // orders 35..48
                    uint32_t m2;
                    const uint32_t c2 = consider(lane + 35, m2);
                    if (c2 < cost) { cost = c2; masks = m2; order = (uint32_t)lane + 35u; }
                }
                near_barrier();  // the distance-1 candidates are in
                if (lane >= 1 && lane <= 3) {  // orders 1..3
                    const uint2 n = M.near_cost[lane - 1];
                    if (n.x <= cost) { cost = n.x; masks = n.y; order = (uint32_t)lane; }
                }
                const uint32_t least = __reduce_min_sync(0xFFFFFFFFu, cost);
                order = __reduce_min_sync(0xFFFFFFFFu, cost == least ? order : ~0u);
                const int win = order <= 3u ? (int)order : order <= 34u ? (int)order - 3 : (int)order - 35;  // the lane that has it
                masks = __shfl_sync(0xFFFFFFFFu, masks, win);
                const uint32_t mA = masks & 0xFFFFu, mB = masks >> 16;
                if (mA && !((mA >> (d0 - 1)) & 1u)) d0 = __ffs((int)mA);
                if (mB && !((mB >> (d1 - 1)) & 1u)) d1 = __ffs((int)mB);
                // the winner enters the window with its palette (the base's, or the neighbour's: with j = 16 the
                // neighbour's slot is this one, and each lane rewrites its own word)
                const int oc = (int)order - 1, wkind = oc % 3, wj = oc / 3 + 1;
                const uint64_t wc = c_cand[bi][order];
                if (lane < 8) {
                    const int *P = order == 0 || wkind == 1 ? s_bpal[cur % 3] : ring_pal[(cur - wj) & (kWindow - 1)];
                    ring_pal[cur & (kWindow - 1)][lane] = P[lane];
                }
                if (lane == 0) {
                    ring[cur & (kWindow - 1)] = wc;
                    M.dist[0] = d0; M.dist[1] = d1;
                    if (order != 0) *(uint64_t *)(out + (size_t)(first + cur) * bs + S.off) = wc;
                }
            }
        } else {  // the loader: block it + 2 to shared memory, block it + 4 fetched
            if (it + 2 < count) {
                store(f0, (it + 2) % 3);
                f0 = f1;
                if (it + 4 < count) f1 = fetch();
            }
        }
        __syncthreads();
    }
}

template <int L>
__global__ void __launch_bounds__(SubRoles<L>::kThreads, 1) rdo_sub_chain_kernel(SrcU8 src, int bw, int nby, int chain_rows, uint8_t *__restrict__ out,
                                                                      int bs, Sub S0, Sub S1, float lambda) {
    __shared__ SubShared M;
    const Sub S = blockIdx.y ? S1 : S0;
    if (S.type == kBc1) sub_chain<true, L>(M, S, src, bw, nby, chain_rows, out, bs, lambda);
    else sub_chain<false, L>(M, S, src, bw, nby, chain_rows, out, bs, lambda);
}

}  // namespace
}  // namespace ztc

// RDO pass over an image whose base encodings `out` holds (raster blocks): one chain per band of band_rows block
// rows (band_rows >= the block-row count: one chain, the reference's single call). lambda: finite, > 0.
cudaError_t ztc_launch_rdo(int fmt, const ztc::SrcU8 &src, uint8_t *out, float lambda, int band_rows, zap_tex_cuda_ctx *ctx, cudaStream_t stream) {
    const int bw = (src.w + 3) / 4, nby = (src.h + 3) / 4;
    if (band_rows <= 0 || band_rows > nby) band_rows = nby;
    const int chains = (nby + band_rows - 1) / band_rows;
    ztc::TraceScope tr("rdo_chain", stream);
    ztc::trace_units((long)bw * nby);
    if (fmt == ZTC_FMT_BC7) {
        const int nblocks = bw * nby;
        uint32_t *dec = nullptr;
        cudaError_t e = ztc_malloc_async((void **)&dec, (size_t)nblocks * 64, stream, ctx);
        if (e != cudaSuccess) return e;
        ztc::bc7_decode_bases_kernel<<<(nblocks + 127) / 128, 128, 0, stream>>>(out, nblocks, (uint4 *)dec);
        constexpr int L = ZTC_RDO_BC7_LANES;
        ztc::rdo_bc7_chain_kernel<L><<<chains, ztc::B7Chain<L>::kThreads, 0, stream>>>(src, bw, nby, band_rows, out, dec, lambda);
        e = cudaGetLastError();
        cudaFreeAsync(dec, stream);
        return e;
    }
    {
        const ztc::Sub S0 = ztc::sub_of(fmt, 0), S1 = ztc::sub_of(fmt, 1);
        const int ns = ztc::sub_count(fmt), bs = fmt == ZTC_FMT_BC1 || fmt == ZTC_FMT_BC4 ? 8 : 16;
        const dim3 grid(chains, ns);
        if (fmt < ZTC_FMT_BC1 || fmt > ZTC_FMT_BC5) return cudaErrorInvalidValue;
        // see SubRoles
        if (fmt == ZTC_FMT_BC1) ztc::rdo_sub_chain_kernel<4><<<grid, ztc::SubRoles<4>::kThreads, 0, stream>>>(src, bw, nby, band_rows, out, bs, S0, S1, lambda);
        else ztc::rdo_sub_chain_kernel<8><<<grid, ztc::SubRoles<8>::kThreads, 0, stream>>>(src, bw, nby, band_rows, out, bs, S0, S1, lambda);
        return cudaGetLastError();
    }
}
