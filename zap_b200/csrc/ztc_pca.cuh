// ztc_pca.cuh - principal-axis endpoint estimate over a texel subset (zap_tex.h:441-462), shared by the BC7 and
// ASTC kernels. The subset is a 16-bit mask (texel i selected when bit i is set); sums run over the selected
// texels in increasing texel order, exactly like the reference's sel[] lists.
#pragma once
#include "ztc_common.cuh"

namespace ztc {

// one power-iteration step on the axis ax; false (ax unchanged) when C ax vanishes
template <int NC>
ZTC_DEV bool pca_power_step(const float C[NC][NC], float ax[NC]) {
    float nv[NC], m = 0.0f;
    #pragma unroll
    for (int a = 0; a < NC; a++) {
        float s = 0.0f;
        #pragma unroll
        for (int b = 0; b < NC; b++) s = s + C[a][b] * ax[b];
        nv[a] = s;
        if (fabsf(s) > m) m = fabsf(s);
    }
    if (m < 1e-6f) return false;
    #pragma unroll
    for (int a = 0; a < NC; a++) ax[a] = nv[a] / m;
    return true;
}

// a byte or a small count as a float: a conversion, or (BITS) small_u2f's logic op and add; the same value either
// way, and which is faster depends on the kernel's other work
template <bool BITS>
ZTC_DEV float pca_u2f(uint32_t n) { return BITS ? small_u2f(n) : (float)n; }

// mean and covariance (upper triangle) of a whole block
template <int NC, int UNROLL, typename Tex>
ZTC_DEV void pca_whole_moments(const Tex &t, float mu[NC], float C[NC][NC]) {
    // The reference's mean sums x / 16 and its covariance d_a d_b over the texels, d = x - mean. d is a multiple of 1/16 below
    // 2^8, so each product is exact (24 bits), and so is every partial sum while it stays below 2^16; they all do
    // when each channel's sum of d^2 is below 2^16. Then the floats are the integer sums 16 sum x_a x_b - S_a S_b
    // over 16, whatever their order: 14 dot products per four texels instead of 20 float operations and 8
    // conversions per texel. Blocks with a wider channel (Q below 2^20 fails) take the sums as the reference does.
    uint32_t S[NC], Q[NC][NC];
    #pragma unroll
    for (int a = 0; a < NC; a++) {
        S[a] = 0u;
        #pragma unroll
        for (int b = a; b < NC; b++) Q[a][b] = 0u;
    }
    const auto row = [&](int r) {
        uint32_t x[4];
        by_channel(t[4 * r], t[4 * r + 1], t[4 * r + 2], t[4 * r + 3], x);
        #pragma unroll
        for (int a = 0; a < NC; a++) {
            S[a] = dot4_add(x[a], 0x01010101u, S[a]);
            #pragma unroll
            for (int b = a; b < NC; b++) Q[a][b] = dot4_add(x[a], x[b], Q[a][b]);
        }
    };
    if (UNROLL == 1) {
        #pragma unroll 1
        for (int r = 0; r < 4; r++) row(r);
    } else {
        #pragma unroll
        for (int r = 0; r < 4; r++) row(r);
    }
    bool exact = true;
    #pragma unroll
    for (int a = 0; a < NC; a++) {
        mu[a] = small_u2f(S[a]) / 16.0f;
        #pragma unroll
        for (int b = a; b < NC; b++) {
            const int q = (int)(16u * Q[a][b] - S[a] * S[b]);
            if (a == b) exact = exact && q < (1 << 20);
            C[a][b] = small_i2f(q) / 16.0f;
        }
    }
    if (!exact) {
        #pragma unroll
        for (int a = 0; a < NC; a++)
            #pragma unroll
            for (int b = a; b < NC; b++) C[a][b] = 0.0f;
        for_texels<UNROLL>([&](int i) {
            float d[NC];
            #pragma unroll
            for (int c = 0; c < NC; c++) d[c] = texel_at_2p15(t[i], c) - (mu[c] + 32768.0f);
            #pragma unroll
            for (int a = 0; a < NC; a++)
                #pragma unroll
                for (int b = a; b < NC; b++) C[a][b] = C[a][b] + d[a] * d[b];
        });
    }
}
// the axis by power iteration from the upper triangle of C
template <int NC, int UNROLL>
ZTC_DEV void pca_power(float C[NC][NC], float ax[NC]) {
    #pragma unroll
    for (int a = 0; a < NC; a++)
        #pragma unroll
        for (int b = 0; b < a; b++) C[a][b] = C[b][a];
    #pragma unroll
    for (int c = 0; c < NC; c++) ax[c] = 1.0f;
    constexpr int kSteps = UNROLL == 1 ? 1 : 6;
    #pragma unroll kSteps
    for (int it = 0; it < 6; it++)
        if (!pca_power_step<NC>(C, ax)) break;
}
// mean and axis of a whole block
template <int NC, int UNROLL, typename Tex>
ZTC_DEV void pca_axis(const Tex &t, float mu[NC], float ax[NC]) {
    float C[NC][NC];
    pca_whole_moments<NC, UNROLL>(t, mu, C);
    pca_power<NC, UNROLL>(C, ax);
}

// t: the texels in registers (uint32_t[16]) or a TexRef; UNROLL 1 rolls the texel loops and the power iteration
// (the same operations in the same order, in less code), UNROLL 16 unrolls them; U2F_BITS: pca_u2f's form
template <int NC, int UNROLL = 16, bool U2F_BITS = true, typename Tex>
ZTC_DEV void pca_endpoints(const Tex &t, uint32_t mask, float lo[4], float hi[4]) {
    const bool whole = mask == 0xFFFFu;  // a compile-time constant for whole-block calls
    float mu[NC], C[NC][NC];
    if (whole) {
        pca_whole_moments<NC, UNROLL>(t, mu, C);
    } else {
        const float cnt = pca_u2f<U2F_BITS>((uint32_t)popc(mask)), cnti = 1.0f / cnt;
        #pragma unroll
        for (int c = 0; c < NC; c++) mu[c] = 0.0f;
        for_texels<UNROLL>([&](int i) {
            if ((mask >> i) & 1u) {
                #pragma unroll
                for (int c = 0; c < NC; c++) mu[c] = mu[c] + div_small(pca_u2f<U2F_BITS>(chan(t[i], c)), cnt, cnti);
            }
        });
        // upper triangle only: cov[a][b] and cov[b][a] add bitwise-identical products in the same order
        #pragma unroll
        for (int a = 0; a < NC; a++)
            #pragma unroll
            for (int b = a; b < NC; b++) C[a][b] = 0.0f;
        for_texels<UNROLL>([&](int i) {
            if ((mask >> i) & 1u) {
                float d[NC];
                #pragma unroll
                for (int c = 0; c < NC; c++) d[c] = pca_u2f<U2F_BITS>(chan(t[i], c)) - mu[c];
                #pragma unroll
                for (int a = 0; a < NC; a++)
                    #pragma unroll
                    for (int b = a; b < NC; b++) C[a][b] = C[a][b] + d[a] * d[b];
            }
        });
    }
    float ax[NC];
    pca_power<NC, UNROLL>(C, ax);
    float n2 = 0.0f, tl = 1e9f, th = -1e9f;
    #pragma unroll
    for (int a = 0; a < NC; a++) n2 = n2 + ax[a] * ax[a];
    for_texels<UNROLL>([&](int i) {
        if ((mask >> i) & 1u) {
            float s = 0.0f;
            #pragma unroll
            for (int c = 0; c < NC; c++) {
                const float d = whole ? texel_at_2p15(t[i], c) - (mu[c] + 32768.0f) : pca_u2f<U2F_BITS>(chan(t[i], c)) - mu[c];
                s = s + d * ax[c];
            }
            if (s < tl) tl = s;
            if (s > th) th = s;
        }
    });
    #pragma unroll
    for (int c = 0; c < 4; c++) {
        if (c < NC) { lo[c] = mu[c] + ax[c] * tl / n2; hi[c] = mu[c] + ax[c] * th / n2; }
        else { lo[c] = 255.0f; hi[c] = 255.0f; }
    }
}

}  // namespace ztc
