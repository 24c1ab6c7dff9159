// ztc_decode.cuh - block decoders (zap_bc_decode, zap_tex.h:1508-1547; BC7 all modes, :367-417; BC6H mode 11,
// :933-943), host+device. Used by the device decode kernels and by the refinement statistics.
#pragma once
#include "ztc_common.cuh"

namespace ztc {
namespace dec {

// BC7 mode descriptors (format spec): subsets, partition bits, rotation bits, index-selector bits, colour bits,
// alpha bits, per-endpoint p-bit, shared p-bit, index bits, secondary index bits
struct Mode { uint8_t ns, pb, rb, isb, cb, ab, epb, spb, ib, ib2; };
ZTC_DEV Mode mode_info(int m) {
    switch (m) {
    case 0: return {3, 4, 0, 0, 4, 0, 1, 0, 3, 0};
    case 1: return {2, 6, 0, 0, 6, 0, 0, 1, 3, 0};
    case 2: return {3, 6, 0, 0, 5, 0, 0, 0, 2, 0};
    case 3: return {2, 6, 0, 0, 7, 0, 1, 0, 2, 0};
    case 4: return {1, 0, 2, 1, 5, 6, 0, 0, 2, 3};
    case 5: return {1, 0, 2, 0, 7, 8, 0, 0, 2, 2};
    case 6: return {1, 0, 0, 0, 7, 7, 1, 0, 4, 0};
    default: return {2, 6, 0, 0, 5, 5, 1, 0, 2, 0};
    }
}

constexpr uint32_t p3(const char *s) {
    uint32_t v = 0;
    for (int i = 0; i < 16; i++) v |= (uint32_t)(s[i] - '0') << (2 * i);
    return v;
}
// partitions (format spec): two-subset masks (bit i = subset 1) and three-subset rows (texel 0 first)
static __constant__ uint16_t kP2d[64] = {
    0xCCCC, 0x8888, 0xEEEE, 0xECC8, 0xC880, 0xFEEC, 0xFEC8, 0xEC80, 0xC800, 0xFFEC, 0xFE80, 0xE800, 0xFFE8, 0xFF00, 0xFFF0, 0xF000,
    0xF710, 0x008E, 0x7100, 0x08CE, 0x008C, 0x7310, 0x3100, 0x8CCE, 0x088C, 0x3110, 0x6666, 0x366C, 0x17E8, 0x0FF0, 0x718E, 0x399C,
    0xAAAA, 0xF0F0, 0x5A5A, 0x33CC, 0x3C3C, 0x55AA, 0x9696, 0xA55A, 0x73CE, 0x13C8, 0x324C, 0x3BDC, 0x6996, 0xC33C, 0x9966, 0x0660,
    0x0272, 0x04E4, 0x4E40, 0x2720, 0xC936, 0x936C, 0x39C6, 0x639C, 0x9336, 0x9CC6, 0x817E, 0xE718, 0xCCF0, 0x0FCC, 0x7744, 0xEE22};
static __constant__ uint32_t kP3d[64] = {
    p3("0011001102212222"), p3("0001001122112221"), p3("0000200122112211"), p3("0222002200110111"), p3("0000000011221122"),
    p3("0011001100220022"), p3("0022002211111111"), p3("0011001122112211"), p3("0000000011112222"), p3("0000111111112222"),
    p3("0000111122222222"), p3("0012001200120012"), p3("0112011201120112"), p3("0122012201220122"), p3("0011011211221222"),
    p3("0011200122002220"), p3("0001001101121122"), p3("0111001120012200"), p3("0000112211221122"), p3("0022002200221111"),
    p3("0111011102220222"), p3("0001000122212221"), p3("0000001101220122"), p3("0000110022102210"), p3("0122012200110000"),
    p3("0012001211222222"), p3("0110122112210110"), p3("0000011012211221"), p3("0022110211020022"), p3("0110011020022222"),
    p3("0011012201220011"), p3("0000200022112221"), p3("0000000211221222"), p3("0222002200120011"), p3("0011001200220222"),
    p3("0120012001200120"), p3("0000111122220000"), p3("0120120120120120"), p3("0120201212010120"), p3("0011220011220011"),
    p3("0011112222000011"), p3("0101010122222222"), p3("0000000021212121"), p3("0022112200221122"), p3("0022001100220011"),
    p3("0220122102201221"), p3("0101222222220101"), p3("0000212121212121"), p3("0101010101012222"), p3("0222011102220111"),
    p3("0002111200021112"), p3("0000211221122112"), p3("0222011101110222"), p3("0002111211120002"), p3("0110011001102222"),
    p3("0000000021122112"), p3("0110011022222222"), p3("0022001100110022"), p3("0022112211220022"), p3("0000000000002112"),
    p3("0002000100020001"), p3("0222122202221222"), p3("0101222222222222"), p3("0111201122012220")};
// anchor texels (format spec): subset 1 of two, subsets 1 and 2 of three
static __constant__ uint8_t kA2d[64] = {
    15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 2, 8, 2, 2, 8, 8, 15, 2, 8, 2, 2, 8, 8, 2, 2,
    15, 15, 6, 8, 2, 8, 15, 15, 2, 8, 2, 2, 2, 15, 15, 6, 6, 2, 6, 8, 15, 15, 2, 2, 15, 15, 15, 15, 15, 2, 2, 15};
static __constant__ uint8_t kA3ad[64] = {
    3, 3, 15, 15, 8, 3, 15, 15, 8, 8, 6, 6, 6, 5, 3, 3, 3, 3, 8, 15, 3, 3, 6, 10, 5, 8, 8, 6, 8, 5, 15, 15,
    8, 15, 3, 5, 6, 10, 8, 15, 15, 3, 15, 5, 15, 15, 15, 15, 3, 15, 5, 5, 5, 8, 5, 10, 5, 10, 8, 13, 15, 12, 3, 3};
static __constant__ uint8_t kA3bd[64] = {
    15, 8, 8, 3, 15, 15, 3, 8, 15, 15, 15, 15, 15, 15, 15, 8, 15, 8, 15, 3, 15, 8, 15, 8, 3, 15, 6, 10, 15, 15, 10, 8,
    15, 3, 15, 10, 10, 8, 9, 10, 6, 15, 8, 15, 3, 6, 6, 8, 15, 3, 15, 15, 15, 15, 15, 15, 15, 15, 15, 15, 3, 15, 15, 8};

// partition tables are device constants: the multi-subset modes decode on the device only
ZTC_DEV int subset_of(int ns, int part, int i) {
    if (ns == 1) return 0;
#ifdef __CUDA_ARCH__
    if (ns == 2) return (kP2d[part] >> i) & 1;
    return (int)((kP3d[part] >> (2 * i)) & 3u);
#else
    return 0;  // not used on the host
#endif
}
ZTC_DEV int anchor_of(int ns, int part, int s) {
#ifdef __CUDA_ARCH__
    return s == 0 ? 0 : ns == 2 ? kA2d[part] : s == 1 ? kA3ad[part] : kA3bd[part];
#else
    return 0;
#endif
}

// A BC7 block's fields (zap_tex.h:378-412): mode (8 = reserved), subsets, partition, rotation, whether alpha has
// its own bits (else it decodes to 255), the expanded 8-bit endpoints (endpoint 2s + k of subset s) and each
// texel's subset and colour / alpha interpolation weight (0..64). The decode of texel i is
// lerp64(ep[2s][c], ep[2s+1][c], w) per channel, then alpha swapped with channel rot - 1 when rot > 0; with the
// weights held fixed it is linear in the endpoints, which the differentiable decode builds on.
struct Bc7Fields {
    int mode, ns, part, rot, ab;
    int ep[6][4];
    uint8_t subset[16], cw[16], aw[16];
};
ZTC_DEV bool bc7_parse(const uint32_t w[4], Bc7Fields &F) {
    int mode = 0;
    while (mode < 8 && !((w[0] >> mode) & 1u)) mode++;
    F.mode = mode;
    F.ns = 1; F.part = 0; F.rot = 0; F.ab = 0;
    if (mode == 8) return false;
    const Mode M = mode_info(mode);
    int pos = mode + 1;
    const int part = (int)get_bits128(w, pos, M.pb); pos += M.pb;
    const int rot = (int)get_bits128(w, pos, M.rb); pos += M.rb;
    const int isb = (int)get_bits128(w, pos, M.isb); pos += M.isb;
    const int ne = 2 * M.ns;
    int cb = M.cb, ab = M.ab;
    for (int c = 0; c < 3; c++)
        for (int e = 0; e < ne; e++) { F.ep[e][c] = (int)get_bits128(w, pos, cb); pos += cb; }
    for (int e = 0; e < ne; e++) {
        if (ab) { F.ep[e][3] = (int)get_bits128(w, pos, ab); pos += ab; }
        else F.ep[e][3] = 255;
    }
    if (M.epb || M.spb) {
        for (int e = 0; e < ne; e++) {
            if (!M.epb && (e & 1)) continue;
            int p = (int)get_bits128(w, pos, 1); pos += 1;
            int last = M.epb ? e : e + 1;
            for (int k = e; k <= last; k++) {
                for (int c = 0; c < 3; c++) F.ep[k][c] = (F.ep[k][c] << 1) | p;
                if (ab) F.ep[k][3] = (F.ep[k][3] << 1) | p;
            }
        }
        cb++;
        if (ab) ab++;
    }
    for (int e = 0; e < ne; e++) {
        for (int c = 0; c < 3; c++) F.ep[e][c] = expand_bits(F.ep[e][c], cb);
        if (ab) F.ep[e][3] = expand_bits(F.ep[e][3], ab);
    }
    for (int e = ne; e < 6; e++)
        for (int c = 0; c < 4; c++) F.ep[e][c] = 0;
    int i1[16], i2[16];
    for (int i = 0; i < 16; i++) {
        int anchor = i == anchor_of(M.ns, part, subset_of(M.ns, part, i));
        i1[i] = (int)get_bits128(w, pos, M.ib - anchor); pos += M.ib - anchor;
    }
    for (int i = 0; i < 16; i++) {
        i2[i] = 0;
        if (M.ib2) { i2[i] = (int)get_bits128(w, pos, M.ib2 - (i == 0)); pos += M.ib2 - (i == 0); }
    }
    for (int i = 0; i < 16; i++) {
        F.subset[i] = (uint8_t)subset_of(M.ns, part, i);
        const int cw = (M.ib2 && isb) ? wbits(M.ib2, i2[i]) : wbits(M.ib, i1[i]);
        F.cw[i] = (uint8_t)cw;
        F.aw[i] = (uint8_t)(!M.ib2 ? cw : isb ? wbits(M.ib, i1[i]) : wbits(M.ib2, i2[i]));
    }
    F.ns = M.ns; F.part = part; F.rot = rot; F.ab = M.ab > 0;
    return true;
}

// ---------------------------------------------------------------- decode to texels
// The BC7 interpolation weights (wbits) as j shifted and multiplied: two or three operations.
template <int IB>
ZTC_DEV int weight_of(uint32_t j) {
    return (int)(IB == 2 ? 21u * j + (j >> 1) : IB == 3 ? 9u * j + (j >> 2) : 4u * j + ((j + 2u) >> 2));
}
// bits [pos, pos + n) of a block held as two 64-bit words (n <= 63; pos and n are compile-time where it is inlined)
ZTC_DEV uint64_t field64(uint64_t lo, uint64_t hi, int pos, int n) {
    const uint64_t v = pos >= 64 ? hi >> (pos - 64) : pos == 0 ? lo : (lo >> pos) | (hi << (64 - pos));
    return v & ((1ull << n) - 1ull);
}
// an index stream with the anchors' missing top bits put back as zeros (p: position of one, the lower ones already
// back): the bits from p up move up by one
ZTC_DEV uint64_t open_bit(uint64_t x, int p) { return x + (x & (~0ull << p)); }

// One BC7 block of a mode whose layout is known at compile time (zap_tex.h:378-417): every field at a fixed position,
// the indices as one 64-bit stream of equal widths, two channels per word in the interpolation. The fields never
// leave registers: a parse into arrays indexed by run-time field widths kept them in local memory and made a
// warp with any block outside mode 6 wait for it
// (2048x2048, 4 % such blocks: 34.3 -> 8.7 us, BC3 10.8 -> 6.7; 3.2 us is the copy bound).
template <int MODE, int NS, int PB, int RB, int ISB, int CB, int AB, int EPB, int SPB, int IB, int IB2>
ZTC_DEV void bc7_mode_block(uint64_t lo, uint64_t hi, uint32_t out[16]) {
    constexpr int kEnds = 2 * NS, kBase = MODE + 1 + PB + RB + ISB, kAlpha = kBase + 3 * kEnds * CB, kP = kAlpha + kEnds * AB;
    constexpr int kIdx = kP + (EPB ? kEnds : 0) + (SPB ? NS : 0), kIdx2 = kIdx + 16 * IB - NS, kPb = (EPB || SPB) ? 1 : 0;
    const int part = PB ? (int)field64(lo, hi, MODE + 1, PB) : 0;
    const uint32_t rot = RB ? (uint32_t)field64(lo, hi, MODE + 1 + PB, RB) : 0u;
    const bool swap = ISB && field64(lo, hi, MODE + 1 + PB + RB, 1) != 0;
    Lerp4 row[NS];
    #pragma unroll
    for (int s = 0; s < NS; s++) {
        int x[2][4];
        #pragma unroll
        for (int k = 0; k < 2; k++) {
            const int e = 2 * s + k;
            const int p = EPB ? (int)field64(lo, hi, kP + e, 1) : SPB ? (int)field64(lo, hi, kP + s, 1) : 0;
            #pragma unroll
            for (int c = 0; c < 4; c++) {
                if (c == 3 && !AB) { x[k][c] = 255; continue; }
                const int n = c < 3 ? CB : AB, pos = c < 3 ? kBase + (c * kEnds + e) * CB : kAlpha + e * AB;
                x[k][c] = expand_bits((int)(field64(lo, hi, pos, n) << kPb) | p, n + kPb);
            }
        }
        row[s] = Lerp4(x[0], x[1]);
    }
    uint32_t mask = 0;  // the texels' subsets, one or two bits a texel
    uint64_t i1 = field64(lo, hi, kIdx, 16 * IB - NS), i2 = 0;
    i1 = open_bit(i1, IB - 1);
#ifdef __CUDA_ARCH__
    if (NS == 2) {
        mask = kP2d[part];
        i1 = open_bit(i1, kA2d[part] * IB + IB - 1);
    } else if (NS == 3) {
        mask = kP3d[part];
        const int a = kA3ad[part], b = kA3bd[part];
        i1 = open_bit(i1, min(a, b) * IB + IB - 1);
        i1 = open_bit(i1, max(a, b) * IB + IB - 1);
    }
#endif
    if (IB2) i2 = open_bit(field64(lo, hi, kIdx2, 16 * IB2 - 1), IB2 - 1);
    // rotation: alpha and channel rot - 1 change places after the interpolation
    const uint32_t sel = rot == 0 ? 0x3210u : rot == 1 ? 0x0213u : rot == 2 ? 0x1230u : 0x2310u;
    #pragma unroll
    for (int i = 0; i < 16; i++) {
        const int w1 = weight_of<IB>((uint32_t)(i1 >> (IB * i)) & ((1u << IB) - 1u));
        if (IB2) {
            const int w2 = weight_of<IB2 ? IB2 : 2>((uint32_t)(i2 >> (IB2 * i)) & ((1u << IB2) - 1u));
            const uint32_t t = row[0].at2(swap ? w2 : w1, swap ? w1 : w2);
#ifdef __CUDA_ARCH__
            out[i] = __byte_perm(t, 0u, sel);
#else
            out[i] = chan(t, sel & 3) | (chan(t, (sel >> 4) & 3) << 8) | (chan(t, (sel >> 8) & 3) << 16) | (chan(t, (sel >> 12) & 3) << 24);
#endif
        } else if (NS == 1) {
            out[i] = row[0].at(w1);
        } else {
            const uint32_t s = NS == 2 ? (mask >> i) & 1u : (mask >> (2 * i)) & 3u;
            Lerp4 r = s == 0 ? row[0] : row[1];
            if (NS == 3 && s == 2) r = row[NS - 1];
            out[i] = r.at(w1);
        }
    }
}

// full BC7 decode, all 8 modes; reserved mode -> transparent black (zap_tex.h:378-417)
ZTC_DEV void bc7_block(const uint32_t w[4], uint32_t out[16]) {
    const uint64_t lo = w[0] | ((uint64_t)w[1] << 32), hi = w[2] | ((uint64_t)w[3] << 32);
    const uint32_t m = w[0] & 0xFFu;  // the mode is the place of the lowest set bit
    if ((m & 0x7Fu) == 0x40u) bc7_mode_block<6, 1, 0, 0, 0, 7, 7, 1, 0, 4, 0>(lo, hi, out);
    else if ((m & 0x3Fu) == 0x20u) bc7_mode_block<5, 1, 0, 2, 0, 7, 8, 0, 0, 2, 2>(lo, hi, out);
    else if ((m & 0x03u) == 0x02u) bc7_mode_block<1, 2, 6, 0, 0, 6, 0, 0, 1, 3, 0>(lo, hi, out);
    else if (m & 0x01u) bc7_mode_block<0, 3, 4, 0, 0, 4, 0, 1, 0, 3, 0>(lo, hi, out);
    else if (m & 0x04u) bc7_mode_block<2, 3, 6, 0, 0, 5, 0, 0, 0, 2, 0>(lo, hi, out);
    else if (m & 0x08u) bc7_mode_block<3, 2, 6, 0, 0, 7, 0, 1, 0, 2, 0>(lo, hi, out);
    else if (m & 0x10u) bc7_mode_block<4, 1, 0, 2, 1, 5, 6, 0, 0, 2, 3>(lo, hi, out);
    else if (m & 0x80u) bc7_mode_block<7, 2, 6, 0, 0, 5, 5, 1, 0, 2, 0>(lo, hi, out);
    else {
        #pragma unroll
        for (int i = 0; i < 16; i++) out[i] = 0u;
    }
}

// BC1 colour block; four_always: the BC3 colour half (zap_tex.h:1508-1517)
ZTC_DEV void bc1_block(uint2 v, bool four_always, uint32_t out[16]) {
    const uint32_t c0 = v.x & 0xFFFFu, c1 = v.x >> 16;
    int a[3], b[3], p2[3], p3[3];
    unpack565(c0, a[0], a[1], a[2]); unpack565(c1, b[0], b[1], b[2]);
    const bool four = four_always || c0 > c1;
    #pragma unroll
    for (int c = 0; c < 3; c++) {
        p2[c] = four ? (2 * a[c] + b[c] + 1) / 3 : (a[c] + b[c] + 1) / 2;
        p3[c] = four ? (a[c] + 2 * b[c] + 1) / 3 : 0;
    }
    const uint32_t q0 = pack_rgba(a[0], a[1], a[2], 255), q1 = pack_rgba(b[0], b[1], b[2], 255);
    const uint32_t q2 = pack_rgba(p2[0], p2[1], p2[2], 255), q3 = pack_rgba(p3[0], p3[1], p3[2], four ? 255 : 0);
    #pragma unroll
    for (int i = 0; i < 16; i++) {
        const bool b0 = (v.y >> (2 * i)) & 1u, b1 = (v.y >> (2 * i)) & 2u;
        const uint32_t lo = b0 ? q1 : q0, hi = b0 ? q3 : q2;
        out[i] = b1 ? hi : lo;
    }
}

// bytes 0..7 of (lo, hi) picked by four 3-bit indices in nibbles
ZTC_DEV uint32_t pick4(uint32_t lo, uint32_t hi, uint32_t nibbles) {
#ifdef __CUDA_ARCH__
    return __byte_perm(lo, hi, nibbles);
#else
    uint32_t r = 0;
    for (int k = 0; k < 4; k++) {
        const uint32_t j = (nibbles >> (4 * k)) & 7u;
        r |= (((j < 4 ? lo : hi) >> (8 * (j & 3))) & 0xFFu) << (8 * k);
    }
    return r;
#endif
}
// BC4 channel block (zap_tex.h:1519-1524): row r's four values in the bytes of out[r]
ZTC_DEV void bc4_block(uint2 v, uint32_t out[4]) {
    const int a0 = v.x & 0xFF, a1 = (v.x >> 8) & 0xFF;
    const bool eight = a0 > a1;
    uint32_t lo = (uint32_t)a0 | ((uint32_t)a1 << 8), hi = 0;
    #pragma unroll
    for (int i = 2; i < 8; i++) {
        const int p = eight ? ((8 - i) * a0 + (i - 1) * a1 + 3) / 7 : i < 6 ? ((6 - i) * a0 + (i - 1) * a1 + 2) / 5 : i == 6 ? 0 : 255;
        if (i < 4) lo |= (uint32_t)p << (8 * i); else hi |= (uint32_t)p << (8 * (i - 4));
    }
    const uint64_t idx = (uint64_t)(v.x >> 16) | ((uint64_t)v.y << 16);
    #pragma unroll
    for (int r = 0; r < 4; r++) {
        const uint32_t x = (uint32_t)(idx >> (12 * r));
        out[r] = pick4(lo, hi, (x & 7u) | ((x & 0x38u) << 1) | ((x & 0x1C0u) << 2) | ((x & 0xE00u) << 3));
    }
}

// A decoded 4x4 block of RGBA8 texels (px[i]: texel i, R in the low byte) into an image: each row of four texels
// inside the image as one 16-byte store when vec (the image and its pitch 16-byte aligned), texels past the right
// or bottom edge left out, a row the right edge cuts texel by texel (4-byte stores if aligned4, else bytes).
ZTC_DEV void store_block_rgba8(uint8_t *out, size_t stride, int w, int h, int bx, int by, const uint32_t px[16], bool vec,
                               bool aligned4) {
    #pragma unroll
    for (int r = 0; r < 4; r++) {
        const int y = by * 4 + r, x0 = bx * 4;
        if (y >= h) break;
        uint8_t *row = out + (size_t)y * stride + (size_t)x0 * 4;
        if (vec && x0 + 3 < w) {
            *(uint4 *)row = make_uint4(px[4 * r], px[4 * r + 1], px[4 * r + 2], px[4 * r + 3]);
            continue;
        }
        #pragma unroll
        for (int c = 0; c < 4; c++) {
            if (x0 + c >= w) break;
            const uint32_t v = px[4 * r + c];
            if (aligned4) *(uint32_t *)(row + 4 * c) = v;
            else { row[4 * c] = (uint8_t)v; row[4 * c + 1] = (uint8_t)(v >> 8); row[4 * c + 2] = (uint8_t)(v >> 16); row[4 * c + 3] = (uint8_t)(v >> 24); }
        }
    }
}

// one block of format FMT (0..4) to 16 RGBA8 texels (zap_tex.h:1526-1547)
template <int FMT>
ZTC_DEV void bcn_block(const uint8_t *b, uint32_t out[16]) {
    if (FMT == 0) {
        bc1_block(ldg((const uint2 *)b), false, out);
    } else if (FMT == 2) {
        uint32_t r[4];
        bc4_block(ldg((const uint2 *)b), r);
        #pragma unroll
        for (int i = 0; i < 16; i++) out[i] = chan(r[i >> 2], i & 3) | 0xFF000000u;
    } else {
        const uint4 v = ldg((const uint4 *)b);
        if (FMT == 4) {
            const uint32_t w[4] = {v.x, v.y, v.z, v.w};
            bc7_block(w, out);
        } else if (FMT == 1) {
            uint32_t a[4];
            bc1_block(make_uint2(v.z, v.w), true, out);
            bc4_block(make_uint2(v.x, v.y), a);
            #pragma unroll
            for (int i = 0; i < 16; i++) out[i] = (out[i] & 0x00FFFFFFu) | (chan(a[i >> 2], i & 3) << 24);
        } else {
            uint32_t r[4], g[4];
            bc4_block(make_uint2(v.x, v.y), r);
            bc4_block(make_uint2(v.z, v.w), g);
            #pragma unroll
            for (int i = 0; i < 16; i++) out[i] = chan(r[i >> 2], i & 3) | (chan(g[i >> 2], i & 3) << 8) | 0xFF000000u;
        }
    }
}

// BC6H mode 11 to half bits, alpha 1.0 (zap_tex.h:933-943): texel i in out[2 i] (R, G) and out[2 i + 1] (B, A); other
// modes decode to 0. A channel's lerp is affine in the weight: 64 a + 32 + (b - a) w, never negative.
ZTC_DEV void bc6h_block(const uint32_t w[4], uint32_t out[32]) {
    const uint64_t lo = w[0] | ((uint64_t)w[1] << 32), hi = w[2] | ((uint64_t)w[3] << 32);
    const bool ok = (w[0] & 31u) == 3u;
    int base[3], slope[3];
    #pragma unroll
    for (int c = 0; c < 3; c++) {
        int e[2];
        #pragma unroll
        for (int k = 0; k < 2; k++) {
            const int q = (int)field64(lo, hi, 5 + 10 * (3 * k + c), 10);
            e[k] = q == 0 ? 0 : q == 1023 ? 0xFFFF : ((q << 16) + 0x8000) >> 10;
        }
        base[c] = 64 * e[0] + 32;
        slope[c] = e[1] - e[0];
    }
    const uint64_t idx = open_bit(field64(lo, hi, 65, 63), 3);
    #pragma unroll
    for (int i = 0; i < 16; i++) {
        const int wt = weight_of<4>((uint32_t)(idx >> (4 * i)) & 15u);
        uint32_t h[3];
        #pragma unroll
        for (int c = 0; c < 3; c++) h[c] = ((uint32_t)((base[c] + slope[c] * wt) >> 6) * 31u) >> 6;
        out[2 * i] = ok ? h[0] | (h[1] << 16) : 0u;
        out[2 * i + 1] = ok ? h[2] | 0x3C000000u : 0u;
    }
}

}  // namespace dec
}  // namespace ztc
