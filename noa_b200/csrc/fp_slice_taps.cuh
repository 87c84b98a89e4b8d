// What the windowed-sinc insertions evaluate per (sample, slice) pair: the window at the sample's distance
// to the slice, and the LINEAR interpolation of the slice. Shared by the gather, scatter and
// insert-and-extract kernels; both are written for few instructions, which is what bounds those kernels.
#pragma once

#include "fp_args.cuh"

namespace nb {

// Whether a call's slices can be read by interp_linear_slice: LINEAR, arrays, offsets within a slice in
// 32 bits (the slice's base pointer takes 64).
inline bool linear_slices(const ProjArgs& a) {
    return a.interp == I_LINEAR && a.in_slice_narrow && !a.in.is_value && !(a.in_w.present && a.in_w.is_value);
}

// interp_spectrum_2d<LINEAR> of one slice from its base pointer, without its branches: the same flip, taps,
// weights and order of the sum, a tap outside the slice reads as zero instead of being skipped.
struct LinearCell {
    float w00, w01, w10, w11;   // 1 - t and t, per axis
    int row0, row1, x;          // indices of the two rows and of the first column
    bool ok0, ok1, okx0, okx1, flip;

    __device__ __forceinline__ LinearCell(const Spectrum2& sp, float f0, float f1) {
        flip = f1 < 0.f;
        f0 = flip ? -f0 : f0;
        f1 = fabsf(f1);
        const float fl0 = floorf(f0), fl1 = floorf(f1);
        const int b0 = static_cast<int>(fl0);
        x = static_cast<int>(fl1);
        w01 = sub(f0, fl0);
        w11 = sub(f1, fl1);
        w00 = sub(1.f, w01);
        w10 = sub(1.f, w11);
        const int lo0 = -sp.n0 / 2, hi0 = (sp.n0 - 1) / 2, hi1 = sp.n1 / 2;
        ok0 = b0 >= lo0 && b0 <= hi0;
        ok1 = b0 + 1 >= lo0 && b0 + 1 <= hi0;
        okx0 = x <= hi1;   // x >= 0
        okx1 = x < hi1;
        row0 = frequency2index(sp.centered, b0, sp.n0);
        row1 = frequency2index(sp.centered, b0 + 1, sp.n0);
    }

    __device__ __forceinline__ float2 read(const float2* base, int s1, int s2) const {
        const int o0 = row0 * s1 + x * s2, o1 = row1 * s1 + x * s2;
        const auto at = [base](int off) { return __ldg(reinterpret_cast<const unsigned long long*>(base + off)); };
        const unsigned long long e00 = ok0 && okx0 ? at(o0) : 0ull, e01 = ok0 && okx1 ? at(o0 + s2) : 0ull;
        const unsigned long long e10 = ok1 && okx0 ? at(o1) : 0ull, e11 = ok1 && okx1 ? at(o1 + s2) : 0ull;
        const unsigned long long wa = pack2(w10, w10), wb = pack2(w11, w11);
        unsigned long long v0 = fma2(e00, wa, 0ull), v1 = fma2(e10, wa, 0ull);
        v0 = fma2(e01, wb, v0);
        v1 = fma2(e11, wb, v1);
        float2 v = unpack2(fma2(v1, pack2(w01, w01), fma2(v0, pack2(w00, w00), 0ull)));
        if (flip)
            v.y = -v.y;
        return v;
    }

    __device__ __forceinline__ float2 read(const float* base, int s1, int s2) const {
        const int o0 = row0 * s1 + x * s2, o1 = row1 * s1 + x * s2;
        const float e00 = ok0 && okx0 ? __ldg(base + o0) : 0.f, e01 = ok0 && okx1 ? __ldg(base + (o0 + s2)) : 0.f;
        const float e10 = ok1 && okx0 ? __ldg(base + o1) : 0.f, e11 = ok1 && okx1 ? __ldg(base + (o1 + s2)) : 0.f;
        const float v0 = fmaf(e01, w11, e00 * w10), v1 = fmaf(e11, w11, e10 * w10);
        return make_float2(fmaf(v1, w01, v0 * w00), 0.f);
    }
};

} // namespace nb
