// Extraction with the interpolation windows of 4 taps and more (CUBIC, BSPLINE, LANCZOS4/6/8), shared by
// the per-call and batched kernels: a warp's 32 pixels, each interpolated by a group of lanes.
//
// Bound: the L1. A pixel reads SIZE x SIZE rows of SIZE consecutive voxels. With one lane per pixel a
// warp's load touches 32 unrelated places (19 sectors a request for LANCZOS8), each a pass of its own
// through the L1. Here the lanes of a group (4 for SIZE 4, else 8) read one row of one pixel together,
// consecutive in memory, so one request serves 4 pixels and touches their 4 rows: LANCZOS8, 500 slices of
// 192^2, 5180 us -> 2200 us (2286 us without the simple cells' path below).
//
// A warp works in three phases. (1) One lane per pixel: coordinates, cutoff, and the pixel's cell and
// three sets of tap weights into a shared slot; pixels outside the cutoff take none. (2) One group per
// slot: lane j of a group owns the x tap j, sums its SIZE x SIZE column of taps over y then z, applies
// its x weight and, for taps on the other side of x = 0, the Friedel conjugation (a tap's mirror depends
// on its x alone, so it is the same for a lane's whole column); then the group adds up. (3) One lane per
// pixel again: the store. The sum over x comes last instead of first, the terms are the same.
#pragma once

#include "fp_args.cuh"

#include <type_traits>

namespace nb {

template<int I>
struct WindowSlots {
    static constexpr int SIZE = InterpTraits<I>::SIZE;
    static constexpr int LANES = SIZE <= 4 ? 4 : 8;        // per pixel
    static constexpr int AXIS = LANES;                     // words of one axis' weights, padded
    static constexpr int WORDS = SIZE <= 4 ? 20 : 28;      // cell, three axes; multiple of 4, not of 32
    float slot[32][WORDS];                                 // of one warp
    float2 value[32];
};

// Whether the window kernels apply to an interpolation.
template<int I>
constexpr bool has_window() { return InterpTraits<I>::SIZE >= 4; }

// Adds up the lanes of each group; the first of them stores the value of slot `at`.
template<typename S, bool CPLX>
__device__ __forceinline__ void group_sum(S& s, float2 sum, int j, int at, int n) {
#pragma unroll
    for (int o = S::LANES / 2; o > 0; o /= 2) {
        sum.x += __shfl_xor_sync(0xffffffffu, sum.x, o);
        if constexpr (CPLX)
            sum.y += __shfl_xor_sync(0xffffffffu, sum.y, o);
    }
    if (j == 0 && at < n)
        s.value[at] = sum;
}

// Whether the taps b + [0, size) along an axis of n frequencies all exist and follow each other in memory.
__device__ __forceinline__ bool simple_axis(bool centered, int b, int size, int n) {
    return b >= -n / 2 && b <= (n - 1) / 2 - (size - 1) && (centered || b >= 0 || b <= -size);
}

// Values of `n` slots' samples of the volume `v`, into s.value. All lanes of the warp call it together.
template<int I, bool CPLX, typename Idx>
__device__ __forceinline__ void window_samples(const View3<Idx>& v, const Spectrum3& sp, WindowSlots<I>& s, int n) {
    using S = WindowSlots<I>;
    constexpr int SIZE = S::SIZE, LANES = S::LANES, START = -(SIZE - 1) / 2;
    using T = typename std::conditional<CPLX, float2, float>::type;
    const int lane = threadIdx.x & 31;
    const int j = lane % LANES;
    const int lo0 = -sp.n0 / 2, hi0 = (sp.n0 - 1) / 2;
    const int lo1 = -sp.n1 / 2, hi1 = (sp.n1 - 1) / 2;
    for (int first = 0; first < n; first += 32 / LANES) {
        const int at = first + lane / LANES;
        const float* slot = s.slot[at < n ? at : n - 1];  // groups past the end repeat the last slot
        const float4 cell = *reinterpret_cast<const float4*>(slot);
        const int b0 = __float_as_int(cell.x) + START, b1 = __float_as_int(cell.y) + START;
        const int x = __float_as_int(cell.z) + START + j;
        float w1[S::AXIS];
#pragma unroll
        for (int k = 0; k < S::AXIS; k += 4)
            *reinterpret_cast<float4*>(w1 + k) = *reinterpret_cast<const float4*>(slot + 4 + S::AXIS + k);
        float2 sum = make_float2(0.f, 0.f);
        unsigned long long sum2 = 0, w12[SIZE];
        if constexpr (CPLX) {
#pragma unroll
            for (int k = 0; k < SIZE; ++k)
                w12[k] = pack2(w1[k], w1[k]);
        }
        if (__all_sync(0xffffffffu, cell.w != 0.f)) {
            // Simple cells: one offset per pixel, rows and planes at the volume's strides from it. With 32-bit
            // byte offsets from the volume's base (Idx = uint32_t) a row costs one addition.
            const T* from = static_cast<const T*>(v.data);
            const Idx start = static_cast<Idx>(frequency2index(sp.centered, b0, sp.n0)) * v.s0 +
                              static_cast<Idx>(frequency2index(sp.centered, b1, sp.n1)) * v.s1 +
                              static_cast<Idx>(j < SIZE ? x : x - j) * v.s2;  // lanes past the window: its first column
            Idx plane = start * static_cast<Idx>(sizeof(T));
            const Idx to_plane = v.s0 * static_cast<Idx>(sizeof(T)), to_row = v.s1 * static_cast<Idx>(sizeof(T));
#pragma unroll 1
            for (int k0 = 0; k0 < SIZE; ++k0) {
                using E = typename std::conditional<CPLX, unsigned long long, float>::type;  // an element's bits
                E e[SIZE];
                Idx row = plane;
#pragma unroll
                for (int k = 0; k < SIZE; ++k) {
                    e[k] = __ldg(reinterpret_cast<const E*>(reinterpret_cast<const char*>(from) + row));
                    row += to_row;
                }
                const float w0 = slot[4 + k0];
                if constexpr (CPLX) {
                    unsigned long long az = 0;
#pragma unroll
                    for (int k = 0; k < SIZE; ++k)
                        az = fma2(e[k], w12[k], az);
                    sum2 = fma2(az, pack2(w0, w0), sum2);
                } else {
                    float az = 0.f;
#pragma unroll
                    for (int k = 0; k < SIZE; ++k)
                        az = fmaf(e[k], w1[k], az);
                    sum.x = fmaf(az, w0, sum.x);
                }
                plane += to_plane;
            }
            if constexpr (CPLX)
                sum = unpack2(sum2);
            sum = j < SIZE ? cmul(sum, slot[4 + 2 * S::AXIS + j]) : make_float2(0.f, 0.f);
            group_sum<S, CPLX>(s, sum, j, at, n);
            continue;
        }
        const bool mirror = x < 0;
        const int ix = mirror ? -x : x;
        const bool okx = j < SIZE && ix <= sp.n2 / 2;
        Idx oy[SIZE];
        unsigned oky = 0, okz = 0;
#pragma unroll
        for (int k = 0; k < SIZE; ++k) {
            const int y = mirror ? -(b1 + k) : b1 + k;
            const int z = mirror ? -(b0 + k) : b0 + k;
            const bool good = y >= lo1 && y <= hi1;
            oky |= good ? 1u << k : 0u;
            okz |= z >= lo0 && z <= hi0 ? 1u << k : 0u;
            oy[k] = good ? static_cast<Idx>(frequency2index(sp.centered, y, sp.n1)) * v.s1 : 0;
        }
        const T* column = static_cast<const T*>(v.data) + (okx ? static_cast<Idx>(ix) * v.s2 : 0);
#pragma unroll 1
        for (int k0 = 0; k0 < SIZE; ++k0) {
            const int z = mirror ? -(b0 + k0) : b0 + k0;
            const bool goodz = (okz >> k0) & 1u;
            const float w0 = slot[4 + k0];
            const T* row = column + (goodz ? static_cast<Idx>(frequency2index(sp.centered, z, sp.n0)) * v.s0 : 0);
            if constexpr (CPLX) {
                unsigned long long e[SIZE], az = 0;
#pragma unroll
                for (int k = 0; k < SIZE; ++k)
                    e[k] = goodz && ((oky >> k) & 1u)
                               ? __ldg(reinterpret_cast<const unsigned long long*>(row + oy[k])) : 0ull;
#pragma unroll
                for (int k = 0; k < SIZE; ++k)
                    az = fma2(e[k], w12[k], az);
                sum2 = fma2(az, pack2(w0, w0), sum2);
            } else {
                float az = 0.f;
#pragma unroll
                for (int k = 0; k < SIZE; ++k) {
                    const float e = goodz && ((oky >> k) & 1u) ? __ldg(row + oy[k]) : 0.f;
                    az = fmaf(e, w1[k], az);
                }
                sum.x = fmaf(az, w0, sum.x);
            }
        }
        if constexpr (CPLX)
            sum = unpack2(sum2);
        sum = okx ? cmul(sum, slot[4 + 2 * S::AXIS + j]) : make_float2(0.f, 0.f);
        if (mirror)
            sum.y = -sum.y;
        group_sum<S, CPLX>(s, sum, j, at, n);
    }
    __syncwarp();
}

// One pixel (b, y, u) per lane of slice extraction `a`: all lanes of the warp call it together, those
// without a pixel with valid = false. `table`: the first `table_size` w_sample values.
template<int I, bool IN_C, bool OUT_C, typename Idx>
__device__ __forceinline__ void extract_window_patch(const ProjArgs& a, int64_t b, int y, int u, bool valid,
                                                     WindowSlots<I>& s, const float2* table, int table_size) {
    using S = WindowSlots<I>;
    const Spectrum3 sp{a.vol_d, a.vol_h, a.vol_w, a.in_centered};
    const View3<Idx> vol{a.in.data, static_cast<Idx>(a.in.s0), static_cast<Idx>(a.in.s1), static_cast<Idx>(a.in.s2)};
    const View3<Idx> volw{a.in_w.data, static_cast<Idx>(a.in_w.s0), static_cast<Idx>(a.in_w.s1),
                          static_cast<Idx>(a.in_w.s2)};
    const bool has_out_w = a.out_w.present;
    const bool has_in_w = a.in_w.present;
    const int lane = threadIdx.x & 31;
    const float f0 = div(static_cast<float>(index2frequency(a.out_centered, y, a.slice_h)), a.f_slice0);
    const float f1 = div(static_cast<float>(u), a.f_slice1);
    float fz, fy, fx;
    slice2grid(f0, f1, a.scale, a.rot, b, a.ews, fz, fy, fx);

    float2 value = make_float2(0.f, 0.f);
    float weight = 0.f;
    const int steps = a.wsize > 1 ? a.wsize : 1;
    for (int w = 0; w < steps; ++w) {
        float gz = fz, cw = 1.f;
        if (a.wsize > 1) {
            const float2 offset = w < table_size ? table[w] : w_sample(a, w);
            gz = add(fz, offset.x);
            cw = offset.y;
        }
        const float sqd = dot3(gz, fy, fx, gz, fy, fx);
        const bool inside = valid && (a.wsize > 1 ? !(sqd > a.cutoff_sqd) : sqd <= a.cutoff_sqd);
        const unsigned mask = __ballot_sync(0xffffffffu, inside);
        if (mask == 0)
            continue;
        const int at = __popc(mask & ((1u << lane) - 1u));
        if (inside) {
            const float q[3] = {mul(gz, a.target0), mul(fy, a.target1), mul(fx, a.target2)};
            int cell[3];
            float ws[3][S::AXIS] = {};
#pragma unroll
            for (int k = 0; k < 3; ++k) {
                const float fl = floorf(q[k]);
                // Far outside (infinities included): no tap either way. NaN (which the w-window's cutoff test lets pass) meets
                // taps, whose weights carry it into the value, as in the other interpolations.
                cell[k] = fl != fl ? 0 : static_cast<int>(fminf(fmaxf(fl, -1e9f), 1e9f));
                interp_weights<I>(sub(q[k], fl), ws[k]);
            }
            float4* slot = reinterpret_cast<float4*>(s.slot[at]);
            constexpr int START = -(S::SIZE - 1) / 2;
            const bool simple = simple_axis(sp.centered, cell[0] + START, S::SIZE, sp.n0) &&
                                simple_axis(sp.centered, cell[1] + START, S::SIZE, sp.n1) &&
                                cell[2] >= -START && cell[2] <= sp.n2 / 2 - (S::SIZE - 1) - START;
            slot[0] = make_float4(__int_as_float(cell[0]), __int_as_float(cell[1]), __int_as_float(cell[2]), simple ? 1.f : 0.f);
#pragma unroll
            for (int k = 0; k < 3; ++k) {
#pragma unroll
                for (int e = 0; e < S::AXIS; e += 4)
                    slot[1 + (k * S::AXIS + e) / 4] = make_float4(ws[k][e], ws[k][e + 1], ws[k][e + 2], ws[k][e + 3]);
            }
        }
        __syncwarp();
        const int n = __popc(mask);
        window_samples<I, IN_C>(vol, sp, s, n);
        if (inside) {
            const float2 iv = to_output<IN_C, OUT_C>(s.value[at]);
            value = a.wsize > 1 ? cadd(value, cmul(iv, cw)) : iv;
        }
        if (has_out_w) {
            float iw = 1.f;
            if (has_in_w) {
                __syncwarp();
                window_samples<I, false>(volw, sp, s, n);
                if (inside)
                    iw = s.value[at].x;
            }
            if (inside)
                weight = a.wsize > 1 ? add(weight, mul(iw, cw)) : iw;
        }
        __syncwarp();  // the slots are written again
    }
    if (valid) {
        dst_store_stream<OUT_C>(a.out, b, y, u, value);
        if (has_out_w)
            store_real_stream(a.out_w, b, y, u, weight);
    }
}

} // namespace nb
