// What the windowed-sinc insertions evaluate per (sample, slice) pair: the window at the sample's distance
// to the slice, and the LINEAR interpolation of the slice. Shared by the gather, scatter and
// insert-and-extract kernels; both are written for few instructions, which is what bounds those kernels.
#pragma once

#include "fp_args.cuh"

namespace nb {

// Whether a call's slices can be read by slice_value and LinearCell: LINEAR, arrays with adjacent columns;
// and whether WindowPair's phase stays in its range. The readers take offsets within a slice as Idx: 32-bit
// where they fit (in_slice_narrow), beside the slice's 64-bit base pointer.
inline bool linear_slices(const ProjArgs& a) {
    return a.interp == I_LINEAR && !a.in.is_value && a.in.s2 == 1 &&
           !(a.in_w.present && a.in_w.is_value) && a.fb * a.ifs < 2097152.f;
}

// windowed_sinc_fast of two distances of at most fftfreq_blackman, in packed operations. The distances get
// a term too small to change any but zero, where it makes the sinc's quotient 1.
struct WindowPair {
    unsigned long long pfs, ifs, pfb;

    __device__ __forceinline__ explicit WindowPair(const ProjArgs& a)
        : pfs(pack2(a.pfs, a.pfs)), ifs(pack2(a.ifs, a.ifs)), pfb(pack2(a.pfb, a.pfb)) {}

    __device__ __forceinline__ float2 operator()(unsigned long long z) const {
        constexpr float TINY = 1e-30f, PI_TINY = 3.1415926535897932384626433832795f * 1e-30f;
        const auto both = [](float v) { return pack2(v, v); };
        z &= 0x7fffffff7fffffffull;
        const unsigned long long xs = fma2(z, pfs, both(PI_TINY)), s = fma2(z, ifs, both(TINY));
        const unsigned long long t = add2(s, both(SINPI_ROUND));  // rounds to integers, as sinpi_reduced
        const unsigned long long r = fma2(add2(t, both(-SINPI_ROUND)), both(-1.f), s);
        const unsigned long long u = mul2(r, r);
        constexpr float C[5] = NB_SINPI;
        unsigned long long p = fma2(both(C[0]), u, both(C[1]));
#pragma unroll
        for (int k = 2; k < 5; ++k)
            p = fma2(p, u, both(C[k]));
        const float2 x = unpack2(xs), b = unpack2(mul2(z, pfb));
        float2 sn = unpack2(mul2(r, p)), inv;
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.x) : "f"(x.x));
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv.y) : "f"(x.y));
        sn.x = __uint_as_float(__float_as_uint(sn.x) ^ static_cast<unsigned>(t) << 31);
        sn.y = __uint_as_float(__float_as_uint(sn.y) ^ static_cast<unsigned>(t >> 32) << 31);
        const unsigned long long c = pack2(__cosf(b.x), __cosf(b.y));
        const unsigned long long blackman = fma2(c, fma2(c, both(0.16f), both(0.5f)), both(0.34f));
        return unpack2(mul2(mul2(pack2(sn.x, sn.y), pack2(inv.x, inv.y)), blackman));
    }
};

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

    template<typename Idx>
    __device__ __forceinline__ float2 read(const float2* base, Idx s1, Idx s2) const {
        const Idx o0 = row0 * s1 + x * s2, o1 = row1 * s1 + x * s2;
        const auto at = [base](Idx off) { return __ldg(reinterpret_cast<const unsigned long long*>(base + off)); };
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

    template<typename Idx>
    __device__ __forceinline__ float2 read(const float* base, Idx s1, Idx s2) const {
        const Idx o0 = row0 * s1 + x * s2, o1 = row1 * s1 + x * s2;
        const float e00 = ok0 && okx0 ? __ldg(base + o0) : 0.f, e01 = ok0 && okx1 ? __ldg(base + (o0 + s2)) : 0.f;
        const float e10 = ok1 && okx0 ? __ldg(base + o1) : 0.f, e11 = ok1 && okx1 ? __ldg(base + (o1 + s2)) : 0.f;
        const float v0 = fmaf(e01, w11, e00 * w10), v1 = fmaf(e11, w11, e10 * w10);
        return make_float2(fmaf(v1, w01, v0 * w00), 0.f);
    }
};

// LinearCell's value of a slice, for a cell whose taps all lie in the slice, on rows adjacent in memory,
// straight from the base; other cells go through LinearCell. q1 may be -0 (no flip).
template<typename T, typename Idx>
__device__ __forceinline__ T slice_value(const T* base, const Spectrum2& sp, Idx s1, float q0, float q1) {
    const unsigned sign = __float_as_uint(add(q1, 0.f)) & 0x80000000u;  // set if q1 < 0
    const float f0 = __uint_as_float(__float_as_uint(q0) ^ sign), f1 = fabsf(q1);
    const float fl0 = floorf(f0), fl1 = floorf(f1);
    const int b0 = static_cast<int>(fl0), x = static_cast<int>(fl1);
    const int c0 = b0 + sp.n0 / 2;
    if (static_cast<unsigned>(c0) < static_cast<unsigned>(sp.n0 - 1) && x < sp.n1 / 2 && (sp.centered || b0 != -1)) {
        const T* row0 = base + ((sp.centered ? c0 : b0 < 0 ? b0 + sp.n0 : b0) * s1 + x);
        const T* row1 = row0 + s1;
        const float t0 = sub(f0, fl0), t1 = sub(f1, fl1), u0 = sub(1.f, t0), u1 = sub(1.f, t1);
        if constexpr (sizeof(T) == 8) {
            const auto at = [](const T* p) { return __ldg(reinterpret_cast<const unsigned long long*>(p)); };
            const unsigned long long e00 = at(row0), e01 = at(row0 + 1), e10 = at(row1), e11 = at(row1 + 1);
            const unsigned long long wa = pack2(u1, u1), wb = pack2(t1, t1);
            const unsigned long long v0 = fma2(e01, wb, mul2(e00, wa)), v1 = fma2(e11, wb, mul2(e10, wa));
            const float2 v = unpack2(fma2(v1, pack2(t0, t0), mul2(v0, pack2(u0, u0))));
            return make_float2(v.x, __uint_as_float(__float_as_uint(v.y) ^ sign));
        } else {
            const float e00 = __ldg(row0), e01 = __ldg(row0 + 1), e10 = __ldg(row1), e11 = __ldg(row1 + 1);
            return fmaf(fmaf(e11, t1, e10 * u1), t0, fmaf(e01, t1, e00 * u1) * u0);
        }
    }
    const LinearCell cell(sp, q0, q1);
    if constexpr (sizeof(T) == 8)
        return cell.read(base, s1, Idx(1));
    else
        return cell.read(base, s1, Idx(1)).x;
}

} // namespace nb
