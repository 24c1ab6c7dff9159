// bcn.cu - BC1 / BC3 / BC4 / BC5 block encoders for sm_100a, one thread per 4x4 block.
//
// Bit-exact with the reference encoder (zap_tex.h:39-213 at rdo = 0). The float part (PCA start, least-squares
// refits) keeps the reference's operation order; the palette searches are exact integer work arranged for the GPU:
// a texel's squared distance to palette entry k is |p|^2 + |c_k|^2 - 2 p.c_k, with p.c_k from one dp4a, and
// the key 4 * (|c_k|^2 - 2 p.c_k) + k orders candidates exactly like the reference's first-best scan.
#include "ztc_common.cuh"
#include "ztc_internal.h"

namespace ztc {

// ---------------------------------------------------------------- BC1 (zap_tex.h:39-168)
ZTC_DEV uint32_t pack565(float r, float g, float b) {  // zap_tex.h:45-49
    int R = f2i_x86(div255(r * 31.0f) + 0.5f), G = f2i_x86(div255(g * 63.0f) + 0.5f), B = f2i_x86(div255(b * 31.0f) + 0.5f);
    return ((uint32_t)clampi(R, 0, 31) << 11) | ((uint32_t)clampi(G, 0, 63) << 5) | (uint32_t)clampi(B, 0, 31);
}

// A 4-colour palette by channel: byte k of col[c] is channel c of entry k (0, 1: the endpoints; 2, 3: the thirds
// between them, zap_tex.h:52-62 with force4)
ZTC_DEV uint32_t bc1_column(uint32_t x0, uint32_t x1) {  // from the endpoints' 8-bit values; n / 3 = (683 n) >> 11 for n <= 766
    return x0 | (x1 << 8) | (((2u * x0 + x1 + 1u) * 683u >> 11) << 16) | (((x0 + 2u * x1 + 1u) * 683u >> 11) << 24);
}
ZTC_DEV uint32_t expand5(uint32_t v) { return (v << 3) | (v >> 2); }
ZTC_DEV uint32_t expand6(uint32_t v) { return (v << 2) | (v >> 4); }
ZTC_DEV void bc1_columns(uint32_t c0, uint32_t c1, uint32_t col[3]) {
    col[0] = bc1_column(expand5(c0 >> 11), expand5(c1 >> 11));
    col[1] = bc1_column(expand6((c0 >> 5) & 63u), expand6((c1 >> 5) & 63u));
    col[2] = bc1_column(expand5(c0 & 31u), expand5(c1 & 31u));
}
// sum over N texels p (alpha byte clear) of the greatest 2 p.c_k - |c_k|^2 over the palette: sum |p|^2 less it is
// the squared error of the best indices, without the indices
template <int N>
ZTC_DEV int bc1_match(const uint32_t p[N], const uint32_t col[3]) {
    uint32_t q[4];
    by_channel(col[0], col[1], col[2], 0u, q);
    int a[4], sum = 0;
    #pragma unroll
    for (int k = 0; k < 4; k++) a[k] = -(int)dot4(q[k], q[k]);
    #pragma unroll
    for (int i = 0; i < N; i++) {
        const int m = max3i((int)(dot4(p[i], q[0]) << 1) + a[0], (int)(dot4(p[i], q[1]) << 1) + a[1], (int)(dot4(p[i], q[2]) << 1) + a[2]);
        sum += max(m, (int)(dot4(p[i], q[3]) << 1) + a[3]);
    }
    return sum;
}
// the same with the first best indices, 2 bits a texel: the key 4 (2 p.c_k - |c_k|^2) - k orders entries like the
// reference's first-best scan
template <int N>
ZTC_DEV int bc1_match_idx(const uint32_t p[N], const uint32_t col[3], uint32_t &idx) {
    uint32_t q[4];
    by_channel(col[0], col[1], col[2], 0u, q);
    int a[4], sum = 0;
    uint32_t bits = 0;
    #pragma unroll
    for (int k = 0; k < 4; k++) a[k] = -4 * (int)dot4(q[k], q[k]) - k;
    #pragma unroll
    for (int i = 0; i < N; i++) {
        int m = max3i((int)(dot4(p[i], q[0]) << 3) + a[0], (int)(dot4(p[i], q[1]) << 3) + a[1], (int)(dot4(p[i], q[2]) << 3) + a[2]);
        m = -max(m, (int)(dot4(p[i], q[3]) << 3) + a[3]);
        sum += m;
        bits |= ((uint32_t)m & 3u) << (2 * i);
    }
    idx = bits;
    const int ksum = popc(bits & 0x55555555u) + 2 * popc(bits & 0xAAAAAAAAu);
    return -((sum - ksum) >> 2);
}

struct Bc1Texels {
    uint32_t p[16];  // r, g, b bytes; alpha byte cleared
    int pp;          // sum of |p|^2
};
ZTC_DEV void bc1_prepare(const uint32_t t[16], Bc1Texels &T) {
    T.pp = 0;
    #pragma unroll
    for (int i = 0; i < 16; i++) {
        T.p[i] = t[i] & 0x00FFFFFFu;
        T.pp = (int)dot4_add(T.p[i], T.p[i], (uint32_t)T.pp);
    }
}
// canonical order (c0 > c1, or solid c0 == c1 with indices 0), indices and SSE (zap_tex.h:90-94; a solid pair's four
// entries are equal, so the scan gives index 0)
ZTC_DEV int bc1_try(const Bc1Texels &T, uint32_t &c0, uint32_t &c1, uint32_t &idx) {
    if (c0 < c1) { uint32_t s = c0; c0 = c1; c1 = s; }
    uint32_t col[3];
    bc1_columns(c0, c1, col);
    return T.pp - bc1_match_idx<16>(T.p, col, idx);
}
ZTC_DEV uint32_t bc1_indices(const Bc1Texels &T, uint32_t b0, uint32_t b1) {
    uint32_t col[3], idx;
    bc1_columns(b0, b1, col);
    bc1_match_idx<16>(T.p, col, idx);
    return idx;
}

ZTC_DEV float bc1_lsw(uint32_t k) { return k == 0 ? 1.0f : k == 1 ? 0.0f : k == 2 ? 2.0f / 3.0f : 1.0f / 3.0f; }

// One step of the climb (zap_tex.h:146-165), step 0..11: endpoint step / 6, channel (step / 2) % 3, down or up one. False when
// the channel is at its limit; else the changed endpoint pair (not ordered) and the palette columns it gives: only
// one channel's column changes.
ZTC_DEV bool bc1_step(int step, uint32_t b0, uint32_t b1, const uint32_t col[3], uint32_t &n0, uint32_t &n1, uint32_t ncol[3]) {
    const int ep = step >= 6, ch = (step >> 1) - 3 * ep, d = (step & 1) ? 1 : -1;
    const int sh = ch == 0 ? 11 : ch == 1 ? 5 : 0, mx = ch == 1 ? 63 : 31;
    const int f = (int)((ep ? b1 : b0) >> sh) & mx;
    if (f + d < 0 || f + d > mx) return false;
    const uint32_t add = (uint32_t)d << sh;  // modulo 2^32; the field does not carry
    n0 = b0 + (ep ? 0u : add); n1 = b1 + (ep ? add : 0u);
    const uint32_t f0 = (n0 >> sh) & (uint32_t)mx, f1 = (n1 >> sh) & (uint32_t)mx;
    const uint32_t nc = ch == 1 ? bc1_column(expand6(f0), expand6(f1)) : bc1_column(expand5(f0), expand5(f1));
    #pragma unroll
    for (int c = 0; c < 3; c++) ncol[c] = c == ch ? nc : col[c];
    return true;
}
// the pair in canonical order, with its columns (entries 0 and 1, 2 and 3 change places)
ZTC_DEV void bc1_order(uint32_t &c0, uint32_t &c1, uint32_t col[3]) {
    if (c0 >= c1) return;
    const uint32_t s = c0; c0 = c1; c1 = s;
    #pragma unroll
    for (int c = 0; c < 3; c++) {
        const uint32_t x = col[c];
        col[c] = ((x >> 8) & 0x00FF00FFu) | ((x << 8) & 0xFF00FF00u);
    }
}

// +-1 climb passes [first, last) over the six 565 channels of the two endpoints, first improvement taken
// immediately (zap_tex.h:146-165); the climb stops early at SSE 0 or after a pass without improvement. Returns
// whether the last pass that ran improved. A step needs only the SSE (the order of the endpoints does not change it); the
// indices are found once, for the pair the climb ends on.
ZTC_DEV bool bc1_climb(const Bc1Texels &T, uint32_t &b0, uint32_t &b1, int &best, int first, int last) {
    bool improved = true;
    uint32_t col[3];
    bc1_columns(b0, b1, col);
    for (int pass = first; improved && pass < last && best > 0; pass++) {
        improved = false;
        #pragma unroll 1
        for (int step = 0; step < 12; step++) {
            uint32_t n0, n1, ncol[3];
            if (!bc1_step(step, b0, b1, col, n0, n1, ncol)) continue;
            const int ne = T.pp - bc1_match<16>(T.p, ncol);
            if (ne < best) {
                best = ne; b0 = n0; b1 = n1; improved = true;
                #pragma unroll
                for (int c = 0; c < 3; c++) col[c] = ncol[c];
                bc1_order(b0, b1, col);
            }
        }
    }
    return improved;
}

// the block's texel sums S and products Q (rr, rg, rb, gg, gb, bb) of N texels, N a multiple of 4
template <int N>
ZTC_DEV void bc1_moments(const uint32_t p[N], uint32_t S[3], uint32_t Q[6]) {
    #pragma unroll
    for (int k = 0; k < 3; k++) S[k] = 0u;
    #pragma unroll
    for (int k = 0; k < 6; k++) Q[k] = 0u;
    #pragma unroll
    for (int r = 0; r < N / 4; r++) {
        uint32_t x[4];
        by_channel(p[4 * r], p[4 * r + 1], p[4 * r + 2], p[4 * r + 3], x);
        #pragma unroll
        for (int c = 0; c < 3; c++) S[c] = dot4_add(x[c], 0x01010101u, S[c]);
        Q[0] = dot4_add(x[0], x[0], Q[0]); Q[1] = dot4_add(x[0], x[1], Q[1]); Q[2] = dot4_add(x[0], x[2], Q[2]);
        Q[3] = dot4_add(x[1], x[1], Q[3]); Q[4] = dot4_add(x[1], x[2], Q[4]); Q[5] = dot4_add(x[2], x[2], Q[5]);
    }
}
// covariance from the moments (each float sum of the reference is exact while the channels' sums of squares are below
// 2^16: see pca_endpoints); false for a wider block, whose sums must be taken in the reference's order
ZTC_DEV bool bc1_covariance(const uint32_t S[3], const uint32_t Q[6], float C[6]) {
    const int q[6] = {(int)(16u * Q[0] - S[0] * S[0]), (int)(16u * Q[1] - S[0] * S[1]), (int)(16u * Q[2] - S[0] * S[2]),
                      (int)(16u * Q[3] - S[1] * S[1]), (int)(16u * Q[4] - S[1] * S[2]), (int)(16u * Q[5] - S[2] * S[2])};
    #pragma unroll
    for (int k = 0; k < 6; k++) C[k] = small_i2f(q[k]) / 16.0f;
    return q[0] < (1 << 20) && q[3] < (1 << 20) && q[5] < (1 << 20);
}
// a term of the covariance sums
ZTC_DEV void bc1_cov_term(uint32_t x, const float mu[3], float C[6]) {
    const float r = texel_at_2p15(x, 0) - (mu[0] + 32768.0f), g = texel_at_2p15(x, 1) - (mu[1] + 32768.0f), b = texel_at_2p15(x, 2) - (mu[2] + 32768.0f);
    C[0] = C[0] + r * r; C[1] = C[1] + r * g; C[2] = C[2] + r * b; C[3] = C[3] + g * g; C[4] = C[4] + g * b; C[5] = C[5] + b * b;
}
ZTC_DEV float bc1_project(uint32_t x, const float mu[3], const float v[3]) {
    return (texel_at_2p15(x, 0) - (mu[0] + 32768.0f)) * v[0] + (texel_at_2p15(x, 1) - (mu[1] + 32768.0f)) * v[1] +
           (texel_at_2p15(x, 2) - (mu[2] + 32768.0f)) * v[2];
}
ZTC_DEV void bc1_axis(const float C[6], float v[3]) {  // six power-iteration steps
    v[0] = v[1] = v[2] = 1.0f;
    for (int it = 0; it < 6; it++) {
        float x = C[0] * v[0] + C[1] * v[1] + C[2] * v[2];
        float y = C[1] * v[0] + C[3] * v[1] + C[4] * v[2];
        float z = C[2] * v[0] + C[4] * v[1] + C[5] * v[2];
        float m = fabsf(x);
        if (fabsf(y) > m) m = fabsf(y);
        if (fabsf(z) > m) m = fabsf(z);
        if (m < 1e-6f) break;
        v[0] = x / m; v[1] = y / m; v[2] = z / m;
    }
}
// the endpoints of one start (zap_tex.h:118-124): start 0 inset by a sixteenth, start 1 the whole range
ZTC_DEV void bc1_start_ends(int start, const float mu[3], const float v[3], float n2, float tmin, float tmax, uint32_t &c0, uint32_t &c1) {
    const float inset = start ? 0.0f : (tmax - tmin) / 16.0f, lo = (tmin + inset) / n2, hi = (tmax - inset) / n2;
    c0 = pack565(mu[0] + v[0] * hi, mu[1] + v[1] * hi, mu[2] + v[2] * hi);
    c1 = pack565(mu[0] + v[0] * lo, mu[1] + v[1] * lo, mu[2] + v[2] * lo);
}

template <int UNROLL>
ZTC_DEV uint32_t bc1_texel(const Bc1Texels &T, TexRef tx, int i) { return UNROLL == 1 ? tx[i] : T.p[i]; }

// one start of the quality search (zap_tex.h:118-143): endpoints from the axis, then up to three least-squares refits
template <int UNROLL>
ZTC_DEV void bc1_one_start(const Bc1Texels &T, TexRef tx, int start, const float mu[3], const float v[3], float n2, float tmin, float tmax,
                           uint32_t &b0, uint32_t &b1, int &best) {
    uint32_t c0, c1, idx = 0;
    bc1_start_ends(start, mu, v, n2, tmin, tmax, c0, c1);
    int e = bc1_try(T, c0, c1, idx);
    for (int it = 0; it < 3 && e > 0; it++) {
        float aa = 0, ab = 0, bb = 0, sa0 = 0, sa1 = 0, sa2 = 0, sb0 = 0, sb1 = 0, sb2 = 0;
        for_texels<UNROLL>([&](int i) {
            float wa = bc1_lsw((idx >> (2 * i)) & 3u), wb = 1.0f - wa;
            aa = aa + wa * wa; ab = ab + wa * wb; bb = bb + wb * wb;
            const uint32_t x = bc1_texel<UNROLL>(T, tx, i);
            float r = byte_u2f(x, 0), g = byte_u2f(x, 1), b = byte_u2f(x, 2);
            sa0 = sa0 + wa * r; sa1 = sa1 + wa * g; sa2 = sa2 + wa * b;
            sb0 = sb0 + wb * r; sb1 = sb1 + wb * g; sb2 = sb2 + wb * b;
        });
        float det = aa * bb - ab * ab;
        if (det < 1e-6f && det > -1e-6f) break;
        uint32_t n0 = pack565((sa0 * bb - sb0 * ab) / det, (sa1 * bb - sb1 * ab) / det, (sa2 * bb - sb2 * ab) / det);
        uint32_t n1 = pack565((sb0 * aa - sa0 * ab) / det, (sb1 * aa - sa1 * ab) / det, (sb2 * aa - sa2 * ab) / det);
        // the accepted pair again (bc1_try orders it c0 >= c1): the same fit and SSE, which ends the refits
        if (max(n0, n1) == c0 && min(n0, n1) == c1) break;
        uint32_t ni = 0;
        int ne = bc1_try(T, n0, n1, ni);
        if (ne >= e) break;
        e = ne; c0 = n0; c1 = n1; idx = ni;
    }
    if (e < best) { best = e; b0 = c0; b1 = c1; }
}

// quality search up to the climb (zap_tex.h:97-145): PCA axis, two starts with least-squares refits (the colour
// channels of T.p are the texels' r, g, b)
// UNROLL 16: the texel loops unrolled over T.p (tx unused); UNROLL 1: rolled loops over tx, the block's texels in
// shared memory
template <int UNROLL = 16>
ZTC_DEV void bc1_start(const Bc1Texels &T, TexRef tx, uint32_t &b0, uint32_t &b1, int &best) {
    uint32_t S[3], Q[6];
    bc1_moments<16>(T.p, S, Q);
    // the reference's mean sums x / 16 in texel order; every term and every partial sum is exact (a multiple of 1/16
    // below 256), so the float sum is the channel's integer sum / 16
    const float mu[3] = {small_u2f(S[0]) / 16.0f, small_u2f(S[1]) / 16.0f, small_u2f(S[2]) / 16.0f};
    float C[6], v[3];
    if (!bc1_covariance(S, Q, C)) {
        #pragma unroll
        for (int k = 0; k < 6; k++) C[k] = 0.0f;
        for_texels<UNROLL>([&](int i) { bc1_cov_term(bc1_texel<UNROLL>(T, tx, i), mu, C); });
    }
    bc1_axis(C, v);
    float n2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2], tmin = 1e9f, tmax = -1e9f;
    for_texels<UNROLL>([&](int i) {
        const float s = bc1_project(bc1_texel<UNROLL>(T, tx, i), mu, v);
        if (s < tmin) tmin = s;
        if (s > tmax) tmax = s;
    });
    b0 = 0; b1 = 0;
    best = 1 << 30;
    #pragma unroll 1
    for (int start = 0; start < 2; start++) bc1_one_start<UNROLL>(T, tx, start, mu, v, n2, tmin, tmax, b0, b1, best);
}

// quality search (zap_tex.h:97-168), one thread
ZTC_DEV uint2 bc1_encode(const uint32_t t[16]) {
    Bc1Texels T;
    bc1_prepare(t, T);
    uint32_t b0, b1;
    int best;
    bc1_start(T, TexRef{nullptr, 0}, b0, b1, best);
    bc1_climb(T, b0, b1, best, 0, 8);
    return make_uint2(b0 | (b1 << 16), bc1_indices(T, b0, b1));
}

// The quality search for the CTA's blocks, one per thread, with the climb past its second pass compacted. Every
// thread runs the starts and the first two climb passes of its block; the blocks whose climb goes on (about a
// tenth on photographic content, yet nearly every warp holds one) are listed in shared memory, and the first
// threads of the CTA climb them on to the end from the owners' texels, so the long tail of the climb costs about
// a tenth of the warps. Same bytes as bc1_encode. Every thread of the CTA calls it (it synchronises); a `valid`
// thread's block is in t and in column threadIdx.x of s_tex.
// ROLLED: the starts' principal axis and least-squares sums run in rolled loops over s_tex (less code, more
// instructions): faster in launches of several waves, slower in a launch of less than one wave, where each
// thread's own chain of dependent instructions sets the time (512x512 BC1, one thread per block: 0.0415 -> 0.0441 ms).
template <int CTA, bool ROLLED>
__device__ __forceinline__ uint2 bc1_encode_cta(bool valid, const uint32_t t[16], uint32_t (*s_tex)[CTA]) {
    static_assert(CTA % 32 == 0 && CTA <= 256, "whole warps, owners fit a byte");
    __shared__ uint32_t s_ends[CTA];
    __shared__ int s_best[CTA], s_wcnt[CTA / 32];
    __shared__ uint8_t s_list[CTA];
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    Bc1Texels T;
    uint32_t b0 = 0, b1 = 0;
    int best = 0;
    if (valid) {
        bc1_prepare(t, T);
        if (ROLLED) bc1_start<1>(T, TexRef{&s_tex[0][tid], CTA}, b0, b1, best);
        else bc1_start(T, TexRef{nullptr, 0}, b0, b1, best);
    }
    bool active = valid;
    int owner = tid;
    #pragma unroll 1
    for (int round = 0; round < 2; round++) {
        bool more = false;
        if (active) more = bc1_climb(T, b0, b1, best, round ? 2 : 0, round ? 8 : 2) && best > 0;
        if (active) { s_ends[owner] = b0 | (b1 << 16); s_best[owner] = best; }
        if (round == 1) break;
        const unsigned bal = __ballot_sync(0xFFFFFFFFu, more);
        if (lane == 0) s_wcnt[warp] = __popc(bal);
        __syncthreads();
        int base = 0, total = 0;
        #pragma unroll
        for (int w = 0; w < CTA / 32; w++) { const int c = s_wcnt[w]; base += w < warp ? c : 0; total += c; }
        const int pos = base + __popc(bal & ((1u << lane) - 1u));
        if (more && ZTC_IN_BOUNDS(pos, CTA, 3)) s_list[pos] = (uint8_t)tid;
        __syncthreads();
        active = tid < total;
        if (active) owner = s_list[tid];
        if (active && !ZTC_IN_BOUNDS(owner, CTA, 8)) active = false;
        if (active) {
            uint32_t u[16];
            #pragma unroll
            for (int i = 0; i < 16; i++) u[i] = s_tex[i][owner];
            bc1_prepare(u, T);
            b0 = s_ends[owner] & 0xFFFFu; b1 = s_ends[owner] >> 16; best = s_best[owner];
        }
    }
    __syncthreads();
    if (!valid) return make_uint2(0u, 0u);
    uint32_t u[16];
    #pragma unroll
    for (int i = 0; i < 16; i++) u[i] = s_tex[i][tid];
    bc1_prepare(u, T);
    return make_uint2(s_ends[tid], bc1_indices(T, s_ends[tid] & 0xFFFFu, s_ends[tid] >> 16));
}

// ---------------------------------------------------------------- BC4 (zap_tex.h:170-213)
// round(a b) for |a b| < 2^22: the sum with 1.5 * 2^23 is rounded to an integer, and taking that away is exact
ZTC_DEV float bc4_rint_mul(float a, float b) { return fma_rn(a, b, 12582912.0f) - 12582912.0f; }

// Plus or minus the distance of a level v to the nearest of the eight palette levels a1 + round(m D / 7), m = 0..7
// (D = a0 - a1 > 0), from u = 7 (v - a1) and i7 = 1 / (7 D), without the palette. With r = u - m D the distance
// to level m is round(|r| / 7) (an integer over 7 never ties), so the nearest level is one of least |r|: m = round(u / D),
// clamped to 0..7 for a v outside [a1, a0]. u / D as computed is within 1e-5 of exact, and exactly it is either a
// half (both neighbours then have the same |r|) or at least 1 / (2 * 255) away from one, so the rounding is right
// for every i7 within a few ulp.
ZTC_DEV float bc4_distance(float u, float D, float i7) {
    const float m = bc4_rint_mul(saturate(u * i7), 7.0f);
    return bc4_rint_mul(fma_rn(-m, D, u), 1.0f / 7.0f);
}

// The reference scans the 8-level palettes of 9 inset endpoint pairs for all 16 texels, keeping the best pair's indices.
// Here a pair's SSE comes from bc4_distance (8 float operations per texel instead of a scan of about 28 integer
// ones; integer-valued float sums below 2^24 are exact), one minimum over (SSE, pair) picks the pair, and only that
// pair's palette is scanned for indices (the lower one on ties, as the reference's scan keeps).
// The SSE over N levels f (7 v) of the pairs (hi - k, lo + j), k = 0..2; D[k]: the pair's a0 - a1 (0 or less: no pair)
template <int N>
ZTC_DEV void bc4_pair_errors(const float f[N], float lo, float hi, int j, float D[3], float e[3]) {
    const float base = lo + 7.0f * (float)j;  // 7 a1
    float i7[3];
    #pragma unroll
    for (int k = 0; k < 3; k++) {
        const float d7 = hi - base - 7.0f * (float)k;  // 7 D
        D[k] = bc4_rint_mul(d7, 1.0f / 7.0f);
        i7[k] = d7 > 0.0f ? rcp_approx(d7) : 0.0f;
        e[k] = 0.0f;
    }
    #pragma unroll
    for (int i = 0; i < N; i++) {
        const float u = f[i] - base;
        #pragma unroll
        for (int k = 0; k < 3; k++) { const float d = bc4_distance(u, D[k], i7[k]); e[k] = fma_rn(d, d, e[k]); }
    }
}
// the chosen pair (key modulo 16 = 3 k + j) and 8 times its palette: a0, a1, then from a0 to a1
ZTC_DEV void bc4_palette(float key, float lo, float hi, int &ia0, int &ia1, float p[8]) {
    const int pair = trunc_i(key) & 15, pk = pair / 3, pj = pair - 3 * pk;
    const float a1 = lo * (1.0f / 7.0f), a0 = hi * (1.0f / 7.0f);  // within an ulp of an integer: rounded below
    ia0 = (int)(f_as_u(a0 + 8388608.0f) & 0xFFu) - pk; ia1 = (int)(f_as_u(a1 + 8388608.0f) & 0xFFu) + pj;
    #pragma unroll
    for (int k = 0; k < 8; k++) p[k] = small_u2f((uint32_t)(8 * (k == 0 ? ia0 : k == 1 ? ia1 : ((8 - k) * ia0 + (k - 1) * ia1 + 3) / 7)));
}
// the first nearest entry of the palette
ZTC_DEV uint32_t bc4_index(uint32_t t, int c, const float p[8]) {
    const float v = fma_rn(u_as_f(0x4B000000u | chan(t, c)), 8.0f, -67108864.0f);  // 8 times the level
    float m = fabsf(v - p[0]);  // 8 distance + index
    #pragma unroll
    for (int k = 1; k < 8; k++) m = fminf(m, fabsf(v - p[k]) + (float)k);
    return f_as_u(m + 8388608.0f) & 7u;
}
ZTC_DEV uint2 bc4_encode(const uint32_t t[16], int c) {
    float f[16], lo = 1785.0f, hi = 0.0f;  // 7 v
    #pragma unroll
    for (int i = 0; i < 16; i++) {
        f[i] = fma_rn(u_as_f(0x4B000000u | chan(t[i], c)), 7.0f, -58720256.0f);  // 7 (2^23 + v) - 7 * 2^23
        lo = fminf(lo, f[i]); hi = fmaxf(hi, f[i]);
    }
    float key = 3.0e38f;  // 16 SSE + pair < 2^24
    #pragma unroll 1
    for (int j = 0; j < 3; j++) {
        float D[3], e[3];
        bc4_pair_errors<16>(f, lo, hi, j, D, e);
        // a pair without a0 > a1 stands for (hi, lo) again, which is pair 0: left out, except pair 0 of a flat block,
        // whose distances are u = 0
        #pragma unroll
        for (int k = 0; k < 3; k++)
            if (D[k] > 0.0f || (k == 0 && j == 0)) key = fminf(key, fma_rn(e[k], 16.0f, (float)(3 * k + j)));
    }
    int ia0, ia1;
    float p[8];
    bc4_palette(key, lo, hi, ia0, ia1, p);
    uint32_t bits[2] = {0u, 0u};  // texels 0..7 and 8..15, 3 bits each
    #pragma unroll
    for (int i = 15; i >= 0; i--) bits[i >> 3] = bits[i >> 3] * 8u + bc4_index(t[i], c, p);
    return make_uint2((uint32_t)ia0 | ((uint32_t)ia1 << 8) | (bits[0] << 16), (bits[0] >> 16) | (bits[1] << 8));
}

// ---------------------------------------------------------------- small launches: eight threads per block
// With fewer blocks than the chip has room for threads, a launch takes as long as one thread's chain of dependent
// instructions (BC1: 38 us from 16x16 texels up, one warp per scheduler at 512x512). Here eight threads share a block.
// Thread r of each half holds row r: fits cover four texels and add their sums over the four threads, and in the
// least-squares sums, whose terms must be added in texel order, each thread runs one channel's (thread 3 the
// weights' own). The halves take the two starts, and in the climb the eight threads try the next eight steps at once.
// Integer sums, minima and maxima do not depend on their order, so every result is the one-thread code's. All loops
// run until no block of the warp needs them, and every thread meets every shuffle. 128x128 BC1 38.1 -> 14.2 us.
constexpr unsigned kAll = 0xFFFFFFFFu;
__device__ __forceinline__ int quad_sum(int v) {
    v += __shfl_xor_sync(kAll, v, 1);
    return v + __shfl_xor_sync(kAll, v, 2);
}
__device__ __forceinline__ uint32_t quad_or(uint32_t v) {
    v |= __shfl_xor_sync(kAll, v, 1);
    return v | __shfl_xor_sync(kAll, v, 2);
}
__device__ __forceinline__ float quad_sum(float v) {  // integer-valued, below 2^24: exact in any order
    v += __shfl_xor_sync(kAll, v, 1);
    return v + __shfl_xor_sync(kAll, v, 2);
}
__device__ __forceinline__ float quad_min(float v) {
    v = fminf(v, __shfl_xor_sync(kAll, v, 1));
    return fminf(v, __shfl_xor_sync(kAll, v, 2));
}
__device__ __forceinline__ float quad_max(float v) {
    v = fmaxf(v, __shfl_xor_sync(kAll, v, 1));
    return fmaxf(v, __shfl_xor_sync(kAll, v, 2));
}

// s_ch[c]: the block's channel c, a byte per texel (row r's word is written here by thread r); s_px: its 16 texels
__device__ __forceinline__ uint2 bc1_encode_group(const uint32_t t[4], uint4 *s_ch, uint32_t *s_px, int r) {
    uint32_t p[4], x[4], S[3], Q[6];
    #pragma unroll
    for (int i = 0; i < 4; i++) { p[i] = t[i] & 0x00FFFFFFu; s_px[4 * r + i] = p[i]; }
    by_channel(p[0], p[1], p[2], p[3], x);
    #pragma unroll
    for (int c = 0; c < 3; c++) ((uint32_t *)&s_ch[c])[r] = x[c];
    __syncwarp();
    bc1_moments<4>(p, S, Q);
    #pragma unroll
    for (int k = 0; k < 3; k++) S[k] = (uint32_t)quad_sum((int)S[k]);
    #pragma unroll
    for (int k = 0; k < 6; k++) Q[k] = (uint32_t)quad_sum((int)Q[k]);
    const int pp = (int)(Q[0] + Q[3] + Q[5]);
    const float mu[3] = {small_u2f(S[0]) / 16.0f, small_u2f(S[1]) / 16.0f, small_u2f(S[2]) / 16.0f};
    float C[6], v[3];
    if (!bc1_covariance(S, Q, C)) {  // the four threads of a block agree
        #pragma unroll
        for (int k = 0; k < 6; k++) C[k] = 0.0f;
        #pragma unroll 1
        for (int i = 0; i < 16; i++) bc1_cov_term(s_px[i], mu, C);
    }
    bc1_axis(C, v);
    const float n2 = v[0] * v[0] + v[1] * v[1] + v[2] * v[2];
    float tmin = 1e9f, tmax = -1e9f;
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        const float s = bc1_project(p[i], mu, v);
        if (s < tmin) tmin = s;
        if (s > tmax) tmax = s;
    }
    tmin = quad_min(tmin); tmax = quad_max(tmax);
    // this thread's channel (thread 3 follows channel 0 and adds nothing)
    const int ch = r < 3 ? r : 0, base = (threadIdx.x & 31) & ~3;
    const uint4 mine = s_ch[ch];
    const uint32_t y4[4] = {mine.x, mine.y, mine.z, mine.w};
    const float muc = ch == 0 ? mu[0] : ch == 1 ? mu[1] : mu[2], vc = ch == 0 ? v[0] : ch == 1 ? v[1] : v[2];
    const float scale = ch == 1 ? 63.0f : 31.0f;
    const int mx = ch == 1 ? 63 : 31, sh = ch == 0 ? 11 : ch == 1 ? 5 : 0;
    const auto pack = [&](float a, float b) -> uint32_t {  // both endpoints' fields of this channel, then all three
        const int f0 = clampi(f2i_x86(div255(a * scale) + 0.5f), 0, mx), f1 = clampi(f2i_x86(div255(b * scale) + 0.5f), 0, mx);
        return quad_or(r < 3 ? ((uint32_t)f0 << sh) | ((uint32_t)f1 << (sh + 16)) : 0u);
    };
    const auto fit = [&](uint32_t &c0, uint32_t &c1, uint32_t &idx) -> int {
        if (c0 < c1) { const uint32_t s = c0; c0 = c1; c1 = s; }
        uint32_t col[3], bits;
        bc1_columns(c0, c1, col);
        const int m = quad_sum(bc1_match_idx<4>(p, col, bits));
        idx = quad_or(bits << (8 * r));
        return pp - m;
    };
    // the two starts side by side, one per half of the eight threads
    uint32_t b0, b1, idx;
    int best;
    {
        const int start = (threadIdx.x >> 2) & 1;
        const float inset = start ? 0.0f : (tmax - tmin) / 16.0f, lo = (tmin + inset) / n2, hi = (tmax - inset) / n2;
        const uint32_t e2 = pack(muc + vc * hi, muc + vc * lo);
        b0 = e2 & 0xFFFFu; b1 = e2 >> 16;
        best = fit(b0, b1, idx);
        bool go = true;
        #pragma unroll 1
        for (int it = 0; it < 3; it++) {
            go = go && best > 0;
            if (!__any_sync(kAll, go)) break;
            float s1 = 0.0f, s2 = 0.0f, s3 = 0.0f;  // sum wa y, wb y, wb wb: y the channel, or wa in thread 3
            #pragma unroll
            for (int i = 0; i < 16; i++) {
                const float wa = bc1_lsw((idx >> (2 * i)) & 3u), wb = 1.0f - wa, y = r < 3 ? byte_u2f(y4[i >> 2], i & 3) : wa;
                s1 = s1 + wa * y; s2 = s2 + wb * y; s3 = s3 + wb * wb;
            }
            const float aa = __shfl_sync(kAll, s1, base + 3), ab = __shfl_sync(kAll, s2, base + 3), bb = s3;
            const float det = aa * bb - ab * ab;
            const bool singular = det < 1e-6f && det > -1e-6f;
            const uint32_t n = pack((s1 * bb - s2 * ab) / det, (s2 * aa - s1 * ab) / det);
            uint32_t n0 = n & 0xFFFFu, n1 = n >> 16, ni;
            // a singular system, or the accepted pair again: the refits end
            go = go && !singular && !(max(n0, n1) == b0 && min(n0, n1) == b1);
            const int ne = fit(n0, n1, ni);
            go = go && ne < best;
            if (go) { best = ne; b0 = n0; b1 = n1; idx = ni; }
        }
        // start 1 counts when its SSE is lower
        const int other = __shfl_xor_sync(kAll, best, 4);
        const uint32_t ends = __shfl_xor_sync(kAll, b0 | (b1 << 16), 4);
        if (start ? other <= best : other < best) { best = other; b0 = ends & 0xFFFFu; b1 = ends >> 16; }
    }
    // The climb, eight steps at a time: each thread tries one of the next eight on all 16 texels, the first that improves
    // is taken, and the steps after it are tried again from there, as the reference's step by step order has it.
    const int j = threadIdx.x & 7, base8 = (threadIdx.x & 31) & ~7;
    uint32_t px[16], col[3];
    #pragma unroll
    for (int i = 0; i < 16; i++) px[i] = s_px[i];
    bc1_columns(b0, b1, col);
    bool climbing = best > 0, improved = false;
    int pass = 0, step = 0;
    while (__any_sync(kAll, climbing)) {
        uint32_t n0 = b0, n1 = b1, ncol[3] = {col[0], col[1], col[2]};
        const bool can = step + j < 12 && bc1_step(step + j, b0, b1, col, n0, n1, ncol);
        const int ne = pp - bc1_match<16>(px, ncol);
        const unsigned won = (__ballot_sync(kAll, climbing && can && ne < best) >> base8) & 255u;
        const int w = won ? __ffs(won) - 1 : 0;
        const uint32_t ends = __shfl_sync(kAll, n0 | (n1 << 16), base8 + w);
        const int e = __shfl_sync(kAll, ne, base8 + w);
        #pragma unroll
        for (int c = 0; c < 3; c++) ncol[c] = __shfl_sync(kAll, ncol[c], base8 + w);
        if (won) {
            best = e; b0 = ends & 0xFFFFu; b1 = ends >> 16; improved = true;
            #pragma unroll
            for (int c = 0; c < 3; c++) col[c] = ncol[c];
            bc1_order(b0, b1, col);
        }
        step += won ? w + 1 : 8;
        if (step >= 12) {  // the pass ends
            pass++;
            climbing = climbing && improved && pass < 8 && best > 0;
            step = 0; improved = false;
        }
    }
    bc1_columns(b0, b1, col);
    bc1_match_idx<4>(p, col, idx);
    return make_uint2(b0 | (b1 << 16), quad_or(idx << (8 * r)));
}

// bc4_encode by four threads, thread r its row's four levels (bytes c of t)
__device__ __forceinline__ uint2 bc4_encode_quad(const uint32_t t[4], int c, int r) {
    float f[4], lo = 1785.0f, hi = 0.0f;
    #pragma unroll
    for (int i = 0; i < 4; i++) {
        f[i] = fma_rn(u_as_f(0x4B000000u | chan(t[i], c)), 7.0f, -58720256.0f);
        lo = fminf(lo, f[i]); hi = fmaxf(hi, f[i]);
    }
    lo = quad_min(lo); hi = quad_max(hi);
    float key = 3.0e38f;
    #pragma unroll 1
    for (int j = 0; j < 3; j++) {
        float D[3], e[3];
        bc4_pair_errors<4>(f, lo, hi, j, D, e);
        #pragma unroll
        for (int k = 0; k < 3; k++) {
            e[k] = quad_sum(e[k]);
            if (D[k] > 0.0f || (k == 0 && j == 0)) key = fminf(key, fma_rn(e[k], 16.0f, (float)(3 * k + j)));
        }
    }
    int a0, a1;
    float p[8];
    bc4_palette(key, lo, hi, a0, a1, p);
    uint32_t bits = 0u;
    #pragma unroll
    for (int i = 3; i >= 0; i--) bits = bits * 8u + bc4_index(t[i], c, p);
    const uint64_t all = (uint64_t)bits << (12 * r + 16);
    return make_uint2(quad_or((uint32_t)all) | (uint32_t)a0 | ((uint32_t)a1 << 8), quad_or((uint32_t)(all >> 32)));
}

constexpr int kGroupBlocks = 16;  // blocks of a 128-thread CTA, eight threads each
template <int FMT>
__global__ void __launch_bounds__(8 * kGroupBlocks) bcn_group_kernel(SrcU8 src, int bw, int by0, int nblocks, BlockOut out, size_t b0) {
    static_assert(FMT == ZTC_FMT_BC1 || FMT == ZTC_FMT_BC3, "colour blocks");
    __shared__ uint4 s_ch[kGroupBlocks][3];
    __shared__ uint32_t s_px[kGroupBlocks][17];
    const int slot = threadIdx.x >> 3, r = threadIdx.x & 3, bi = blockIdx.x * kGroupBlocks + slot;
    const int b = min(bi, nblocks - 1);  // threads past the last block repeat it and store nothing
    uint32_t t[4];
    gather_row(src, b % bw, by0 + b / bw, r, t);
    uint2 a = make_uint2(0u, 0u);
    if (FMT == ZTC_FMT_BC3) a = bc4_encode_quad(t, 3, r);
    const uint2 c = bc1_encode_group(t, s_ch[slot], s_px[slot], r);
    if ((threadIdx.x & 7) != 0 || bi >= nblocks) return;
    if (FMT == ZTC_FMT_BC1) put_block8(out, b0 + (size_t)b, c);
    else put_block16(out, b0 + (size_t)b, make_uint4(a.x, a.y, c.x, c.y));
}

// ---------------------------------------------------------------- kernel: one thread per block
// CTA sizes of the BC1-BC5 kernel. For BC1 / BC3 a larger CTA shares one list of compacted climbs among more
// blocks (2048x2048 BC1: 64 threads 0.217 ms, 128 0.189, 256 0.185; BC4 the same at all three); a launch smaller
// than one full wave of large CTAs takes the small size, which keeps more SMs busy. BC1 / BC3 take 224 threads at
// 4 CTAs per SM (72 registers; 2048x2048 BC1 fills 1.98 waves instead of 1.73: 0.172 -> 0.168 ms); BC4 / BC5 keep
// 256 (224 measured 0.0558 -> 0.0567 ms on BC4).
constexpr int kBcnSmall = 128;
template <int FMT>
constexpr int bcn_large() { return FMT == ZTC_FMT_BC1 || FMT == ZTC_FMT_BC3 ? 224 : 256; }
// Blocks per SM up to which a BC1 / BC3 launch takes eight threads per block (23680 blocks, 615x615 texels). One thread
// / eight threads per block: BC1 256x256 35.3 / 14.9 us, 512x512 35.3 / 27.1, 724x724 40.7 / 43.9, 1024x1024 55.1 /
// 77.7; BC3 36.0 / 15.8, 36.7 / 29.5, 42.8 / 52.7, 60.3 / 95.6.
constexpr int kGroupLimit = 160;
template <int FMT, int CTA>
__global__ void __launch_bounds__(CTA, ZTC_MINB_BCN * 128 / CTA) bcn_kernel(SrcU8 src, int bw, int by0, int nblocks, BlockOut out, size_t b0) {
    constexpr bool kColour = FMT == ZTC_FMT_BC1 || FMT == ZTC_FMT_BC3;
    __shared__ uint32_t s_tex[16][kColour ? CTA : 1];  // column threadIdx.x: this thread's block (BC1 / BC3)
    const int b = blockIdx.x * blockDim.x + threadIdx.x;
    const bool valid = b < nblocks;
    if (!kColour && !valid) return;  // BC4 / BC5 never synchronise
    uint32_t t[16];
    if (valid) {
        gather_block(src, b % bw, by0 + b / bw, t);
        if (kColour) {
            #pragma unroll
            for (int i = 0; i < 16; i++) s_tex[i][threadIdx.x] = t[i];
        }
    }
    const size_t ob = b0 + (size_t)b;  // the block's index in the output
    if (FMT == ZTC_FMT_BC1) {
        const uint2 c = bc1_encode_cta<CTA, CTA != kBcnSmall>(valid, t, (uint32_t(*)[CTA])s_tex);
        if (valid) put_block8(out, ob, c);
    } else if (FMT == ZTC_FMT_BC4) {
        put_block8(out, ob, bc4_encode(t, 0));
    } else if (FMT == ZTC_FMT_BC3) {
        uint2 a = valid ? bc4_encode(t, 3) : make_uint2(0u, 0u);
        const uint2 c = bc1_encode_cta<CTA, CTA != kBcnSmall>(valid, t, (uint32_t(*)[CTA])s_tex);
        if (valid) put_block16(out, ob, make_uint4(a.x, a.y, c.x, c.y));
    } else {  // BC5
        uint2 r = bc4_encode(t, 0), g = bc4_encode(t, 1);
        put_block16(out, ob, make_uint4(r.x, r.y, g.x, g.y));
    }
}

// the launch at the threads per block and CTA size that suit its block count
template <int F>
static void launch_bcn(const SrcU8 &src, int bw, int by0, int nblocks, const BlockOut &out, size_t b0, cudaStream_t stream) {
    if constexpr (F == ZTC_FMT_BC1 || F == ZTC_FMT_BC3) {
        if (nblocks <= ztc_sm_count() * kGroupLimit) {
            bcn_group_kernel<F><<<(nblocks + kGroupBlocks - 1) / kGroupBlocks, 8 * kGroupBlocks, 0, stream>>>(src, bw, by0, nblocks, out, b0);
            return;
        }
    }
    constexpr int kLarge = bcn_large<F>();
    const bool large = nblocks >= ztc_sm_count() * (ZTC_MINB_BCN * 128 / kLarge) * kLarge;
    const int cta = large ? kLarge : kBcnSmall, grid = (nblocks + cta - 1) / cta;
    if (large) bcn_kernel<F, kLarge><<<grid, cta, 0, stream>>>(src, bw, by0, nblocks, out, b0);
    else bcn_kernel<F, kBcnSmall><<<grid, cta, 0, stream>>>(src, bw, by0, nblocks, out, b0);
}

}  // namespace ztc

cudaError_t ztc_launch_bcn_to(int fmt, const ztc::SrcU8 &src, int by0, int nby, const ztc::BlockOut &out, size_t b0, cudaStream_t stream) {
    int bw = (src.w + 3) / 4, nblocks = bw * nby;
    if (nblocks <= 0) return cudaSuccess;
    static const char *names[4] = {"bc1_encode", "bc3_encode", "bc4_encode", "bc5_encode"};
    ztc::TraceScope tr(fmt >= 0 && fmt < 4 ? names[fmt] : "bcn_encode", stream);
    ztc::trace_units(nblocks);
    switch (fmt) {
    case ZTC_FMT_BC1: ztc::launch_bcn<ZTC_FMT_BC1>(src, bw, by0, nblocks, out, b0, stream); break;
    case ZTC_FMT_BC3: ztc::launch_bcn<ZTC_FMT_BC3>(src, bw, by0, nblocks, out, b0, stream); break;
    case ZTC_FMT_BC4: ztc::launch_bcn<ZTC_FMT_BC4>(src, bw, by0, nblocks, out, b0, stream); break;
    case ZTC_FMT_BC5: ztc::launch_bcn<ZTC_FMT_BC5>(src, bw, by0, nblocks, out, b0, stream); break;
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

cudaError_t ztc_launch_bcn(int fmt, const ztc::SrcU8 &src, int by0, int nby, uint8_t *out, cudaStream_t stream) {
    return ztc_launch_bcn_to(fmt, src, by0, nby, ztc::BlockOut{out, 0, fmt, 0}, 0, stream);
}

// ---------------------------------------------------------------- batched: one persistent launch over a tile queue
// A CTA takes one tile at a time and runs it in chunks of CTA blocks (a tile holds a multiple of the CTA's blocks:
// blocks per tile and CTA size are separate knobs of the batch autotuner, as are the tile's shape, a row strip or a
// 2-D tile, and MINB, the minimum resident CTAs of 128 threads per SM that sets the register cap).
namespace ztc {
template <int FMT, int CTA, int MINB>
__global__ void __launch_bounds__(CTA, MINB * 128 / CTA) batch_bcn_kernel(const BatchLevel *__restrict__ levels, const BatchTile *__restrict__ tiles,
                                                                         int ntiles, uint32_t *__restrict__ counter) {
    constexpr bool kColour = FMT == ZTC_FMT_BC1 || FMT == ZTC_FMT_BC3;
    __shared__ int s_tile;
    __shared__ uint32_t s_tex[16][kColour ? CTA : 1];  // column threadIdx.x: this thread's block (BC1 / BC3)
    for (;;) {
        if (threadIdx.x == 0) s_tile = (int)atomicAdd(counter, 1u);
        __syncthreads();
        const int tile = s_tile;
        __syncthreads();  // every thread has read s_tile before thread 0 overwrites it
        if (tile >= ntiles) break;
        const BatchTile T = tiles[tile];
        const BatchLevel L = levels[T.level];
        const SrcU8 src{L.src, L.pitch, L.w, L.h, 4, (((uintptr_t)L.src | L.pitch) & 15u) == 0};
        for (int j0 = 0; j0 < T.count; j0 += CTA) {  // the same trip count in every thread: barriers stay uniform
            const int j = j0 + (int)threadIdx.x;
            const bool valid = j < T.count;
            if (!kColour && !valid) continue;  // BC4 / BC5 never synchronise inside a tile
            const int b = tile_block(T, L.bw, j);
            uint32_t t[16];
            if (valid) {
                gather_block(src, b % L.bw, b / L.bw, t);
                if (kColour) {
                    #pragma unroll
                    for (int i = 0; i < 16; i++) s_tex[i][threadIdx.x] = t[i];
                }
            }
            if (FMT == ZTC_FMT_BC1) {
                const uint2 c = bc1_encode_cta<CTA, true>(valid, t, (uint32_t(*)[CTA])s_tex);
                if (valid) store_block8(L.dst + (size_t)b * 8, c);
            } else if (FMT == ZTC_FMT_BC4) store_block8(L.dst + (size_t)b * 8, bc4_encode(t, 0));
            else if (FMT == ZTC_FMT_BC3) {
                const uint2 a = valid ? bc4_encode(t, 3) : make_uint2(0u, 0u);
                const uint2 c = bc1_encode_cta<CTA, true>(valid, t, (uint32_t(*)[CTA])s_tex);
                if (valid) store_block16(L.dst + (size_t)b * 16, make_uint4(a.x, a.y, c.x, c.y));
            } else {
                uint2 r = bc4_encode(t, 0), g = bc4_encode(t, 1);
                store_block16(L.dst + (size_t)b * 16, make_uint4(r.x, r.y, g.x, g.y));
            }
            if (kColour) __syncthreads();  // the next chunk overwrites s_tex
        }
    }
}

template <int FMT, int MINB>
static const void *batch_fn_cap(int cta) {
    switch (cta) {
    case 64: return (const void *)batch_bcn_kernel<FMT, 64, MINB>;
    case 128: return (const void *)batch_bcn_kernel<FMT, 128, MINB>;
    case 256: return (const void *)batch_bcn_kernel<FMT, 256, MINB>;
    default: return nullptr;
    }
}
template <int FMT>
static const void *batch_fn(int cta, int regs) {
    return regs ? batch_fn_cap<FMT, ZTC_MINB_BCN_BATCH_LOOSE>(cta) : batch_fn_cap<FMT, ZTC_MINB_BCN_BATCH>(cta);
}
}  // namespace ztc

const void *ztc_batch_bcn_kernel_fn(int fmt, int cta, int regs) {
    switch (fmt) {
    case ZTC_FMT_BC1: return ztc::batch_fn<ZTC_FMT_BC1>(cta, regs);
    case ZTC_FMT_BC3: return ztc::batch_fn<ZTC_FMT_BC3>(cta, regs);
    case ZTC_FMT_BC4: return ztc::batch_fn<ZTC_FMT_BC4>(cta, regs);
    case ZTC_FMT_BC5: return ztc::batch_fn<ZTC_FMT_BC5>(cta, regs);
    default: return nullptr;
    }
}

cudaError_t ztc_launch_batch_bcn(int fmt, int cta, int regs, int grid, const ztc::BatchLevel *levels, const ztc::BatchTile *tiles, int ntiles,
                                 uint32_t *counter, cudaStream_t stream) {
    const void *fn = ztc_batch_bcn_kernel_fn(fmt, cta, regs);
    if (!fn) return cudaErrorInvalidValue;
    void *args[] = {(void *)&levels, (void *)&tiles, (void *)&ntiles, (void *)&counter};
    return cudaLaunchKernel(fn, dim3(grid), dim3(cta), args, 0, stream);
}
