// Double-float complex numbers of the complex128 tile sweeps (sweep_df.cu,
// sweep_cluster.cu): conversions and the complex multiply-accumulate.
#pragma once

#include "sweep_common.cuh"

namespace qgb {

struct dfc {  // one complex128 amplitude as two double-float numbers: 16 bytes, like double2
    float rh, rl, ih, il;
};

// x 2^(896 - bias) as a pair of floats (bias >= 1).
__device__ __forceinline__ void df_split(double x, float& h, float& l, int bias = 896) {
    const unsigned long long b = static_cast<unsigned long long>(__double_as_longlong(x));
    const uint32_t hw = uint32_t(b >> 32), lw = uint32_t(b);
    const uint32_t sign = hw & 0x80000000u;
    const int E = int((hw >> 20) & 0x7ffu);
    const int ef = E - bias;  // the float's biased exponent (1023 - 127 = 896)
    if (ef <= 0) {            // zero, and every |x| < 2^(bias - 1022)
        h = 0.f;
        l = 0.f;
        return;
    }
    // h: the significand rounded to 24 bits (half up); a carry out of the
    // significand moves into the exponent field, as it should
    const uint32_t up = (lw >> 28) & 1u;
    h = __uint_as_float(sign | (((uint32_t(ef) << 23) | ((hw & 0xfffffu) << 3) | (lw >> 29)) + up));
    // l = x - h: the 29 dropped bits (unit 2^(E - 1075)), less 2^29 when h was rounded up
    uint32_t r = lw & 0x1fffffffu;
    uint32_t lsign = sign;
    if (up) {
        r = 0x20000000u - r;
        lsign ^= 0x80000000u;
    }
    const int lz = __clz(r);
    const int el = ef - lz - 21;  // biased exponent of r's leading bit: (31 - lz) + (E - 1075) + bias - 769
    if (r == 0u || el <= 0) {
        l = 0.f;
        return;
    }
    uint32_t lb;
    if (lz >= 8) {
        lb = (uint32_t(el) << 23) | ((r << (lz - 8)) & 0x7fffffu);  // exact
    } else {  // leading bit to position 23, rounded half up (carry into the exponent field)
        const int sh = 8 - lz;
        lb = ((uint32_t(el) << 23) | ((r >> sh) & 0x7fffffu)) + ((r >> (sh - 1)) & 1u);
    }
    l = __uint_as_float(lsign | lb);
}

// A normal float (or zero) as a float64, exactly, from its bits; float
// subnormals (below 2^-126) become 0.
__device__ __forceinline__ double df_widen(float f) {
    const uint32_t b = __float_as_uint(f);
    const uint32_t e = (b >> 23) & 0xffu;
    if (e == 0u) return 0.0;
    const uint32_t hw = (b & 0x80000000u) | ((e + 896u) << 20) | ((b & 0x7fffffu) >> 3);
    return __hiloint2double(int(hw), int(b << 29));
}

__device__ __forceinline__ double df_join(float h, float l) { return df_widen(h) + df_widen(l); }

// (sh, sl) += (ah, al) * (bh, bl)
__device__ __forceinline__ void df_mac(float& sh, float& sl, float ah, float al, float bh, float bl) {
    const float p = __fmul_rn(ah, bh);
    float e = __fmaf_rn(ah, bh, -p);
    e = __fmaf_rn(ah, bl, e);
    e = __fmaf_rn(al, bh, e);
    const float t = __fadd_rn(sh, p);
    const float z = __fsub_rn(t, sh);
    const float err = __fadd_rn(__fsub_rn(sh, __fsub_rn(t, z)), __fsub_rn(p, z));
    sh = t;
    sl = __fadd_rn(sl, __fadd_rn(err, e));
}

// s = (re high, re low, im high, im low) += m * v
__device__ __forceinline__ void dfc_mac(float (&s)[4], const dfc& m, const dfc& v) {
    df_mac(s[0], s[1], m.rh, m.rl, v.rh, v.rl);
    df_mac(s[0], s[1], -m.ih, -m.il, v.ih, v.il);
    df_mac(s[2], s[3], m.rh, m.rl, v.ih, v.il);
    df_mac(s[2], s[3], m.ih, m.il, v.rh, v.rl);
}

__device__ __forceinline__ dfc dfc_finish(const float (&s)[4]) {
    dfc r;
    r.rh = __fadd_rn(s[0], s[1]);
    r.rl = __fsub_rn(s[1], __fsub_rn(r.rh, s[0]));
    r.ih = __fadd_rn(s[2], s[3]);
    r.il = __fsub_rn(s[3], __fsub_rn(r.ih, s[2]));
    return r;
}

}  // namespace qgb
