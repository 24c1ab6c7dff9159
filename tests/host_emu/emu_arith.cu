// emu_arith.cu - TEST INFRASTRUCTURE: arithmetic shortcuts of the kernels, compiled for the host, against the rule they
// stand for, over their whole domains (tests/test_kernel_arithmetic.py).
#include "../../zap_b200/csrc/bcn.cu"
#include "../../zap_b200/csrc/mip.cu"

namespace ztc {
void trace_begin(const char *, cudaStream_t) {}
void trace_end(cudaStream_t) {}
void trace_units(long) {}
void trace_units_dev(const uint32_t *, cudaStream_t) {}
}  // namespace ztc
int ztc_set_error(int status, const char *) { return status; }
int ztc_sm_count() { return 148; }

using namespace ztc;
#define EMU extern "C" __attribute__((visibility("default")))

// sums s with bit patterns in [lo, hi) whose one-word sRGB search differs from the first k with s / 4 < thr[k]
EMU uint64_t emu_srgb_back_mismatches(uint64_t lo, uint64_t hi) {
    SrgbTables T;
    srgb_tables_host(T);
    uint64_t bad = 0;
    for (uint64_t b = lo; b < hi; b++) {
        const float s = u_as_f((uint32_t)b), v = s * 0.25f;
        int l = 0, h = 255;
        while (l < h) { const int mid = (l + h) >> 1; if (v < T.thr[mid]) h = mid; else l = mid + 1; }
        bad += ((srgb_back(MipTables{&T}, s) >> 16) & 0xFFu) != (uint32_t)l;
    }
    return bad;
}
EMU float emu_srgb_linear(int code) {
    SrgbTables T;
    srgb_tables_host(T);
    return T.lin[code];
}

// (a0, a1, v) with a1 < a0 and v up to 3 outside [a1, a0] for which bc4_distance is not the distance to the nearest of the
// eight palette levels, at a reciprocal `ulps` units off
EMU uint64_t emu_bc4_distance_mismatches(int ulps) {
    uint64_t bad = 0;
    for (int a1 = 0; a1 < 256; a1++)
        for (int a0 = a1 + 1; a0 < 256; a0++)
            for (int v = a1 > 3 ? a1 - 3 : 0; v <= a0 + 3 && v < 256; v++) {
                int best = 1 << 30;
                for (int k = 0; k < 8; k++) {
                    const int p = k == 0 ? a0 : k == 1 ? a1 : ((8 - k) * a0 + (k - 1) * a1 + 3) / 7, d = v > p ? v - p : p - v;
                    best = d < best ? d : best;
                }
                const float i7 = u_as_f(f_as_u(1.0f / (7.0f * (float)(a0 - a1))) + (uint32_t)ulps);
                const float d = bc4_distance(7.0f * (float)(v - a1), (float)(a0 - a1), i7);
                bad += (d < 0.0f ? -d : d) != (float)best;
            }
    return bad;
}

// floats v in [-512, 768] with bit patterns in [lo, hi) (either sign) for which quant8_pbits differs from quant_pbit
EMU uint64_t emu_quant8_mismatches(uint64_t lo, uint64_t hi) {
    uint64_t bad = 0;
    for (uint64_t b = lo; b < hi; b++) {
        const float v[4] = {u_as_f((uint32_t)b), 0.0f, 0.0f, 0.0f};
        if (!(v[0] >= -512.0f && v[0] <= 768.0f)) continue;
        uint32_t k[2][4];
        int err[2];
        quant8_pbits<1>(v, k, err);
        for (int p = 0; p < 2; p++) {
            int q[4], x8[4];
            const int e = quant_pbit<1>(v, 8, p, q, x8);
            const int got = (int)(k[p][0] & 127u);
            bad += e != err[p] || q[0] != got || x8[0] != 2 * got + p;
        }
    }
    return bad;
}
