// Pair copy of a volume for LINEAR extraction, shared by the per-call and batched extraction kernels.
//
// Element (z, y, x) of the copy (D x H x W/2+1, strides pair_sz, pair_sy, 1) holds the two x-neighbours v[z][y][x] and
// v[z][y][x+1] (zero past the last column) as one float4, so the 2x2x2 trilinear cell is 4 aligned
// 16-byte loads instead of 8 scattered 8-byte ones. The taps, weights and summation order are those of
// interp_linear_3d, so results are bit-identical to the generic path.
#pragma once

#include "fp_args.cuh"
#include "fp_pool.cuh"

namespace nb {

__device__ __forceinline__ float2 interp_linear_pairs(const float4* __restrict__ pairs, int sz, int sy,
                                                      const Spectrum3& sp, float q0, float q1, float q2) {
    float conjugate = 1.f;
    if (q2 < 0.f) {
        q0 = -q0; q1 = -q1; q2 = -q2;
        conjugate = -1.f;
    }
    const float fl0 = floorf(q0), fl1 = floorf(q1), fl2 = floorf(q2);
    const int b0 = static_cast<int>(fl0), b1 = static_cast<int>(fl1), b2 = static_cast<int>(fl2);
    const float t0 = sub(q0, fl0), t1 = sub(q1, fl1), t2 = sub(q2, fl2);
    // Interior cells: the same terms in the same order, from one base offset, with the four loads issued
    // together.
    if (interior_cell(sp, b0, b1, b2)) {
        const float4* p = pairs + (frequency2index(sp.centered, b0, sp.n0) * sz +
                                   frequency2index(sp.centered, b1, sp.n1) * sy + b2);
        unsigned long long e[8];
        ldg_pair(p, e[0], e[1]);
        ldg_pair(p + sy, e[2], e[3]);
        ldg_pair(p + sz, e[4], e[5]);
        ldg_pair(p + sz + sy, e[6], e[7]);
        float2 value = trilinear(e, t0, t1, t2);
        value.y *= conjugate;
        return value;
    }
    const float w0[2] = {sub(1.f, t0), t0};
    const float w1[2] = {sub(1.f, t1), t1};
    const float w20 = sub(1.f, t2);
    const int lo0 = -sp.n0 / 2, hi0 = (sp.n0 - 1) / 2;
    const int lo1 = -sp.n1 / 2, hi1 = (sp.n1 - 1) / 2;
    const int hi2 = sp.n2 / 2;
    const bool okx0 = b2 >= 0 && b2 <= hi2;
    const bool okx1 = b2 + 1 >= 0 && b2 + 1 <= hi2;
    float2 value = make_float2(0.f, 0.f);
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        const int iz = b0 + z;
        const bool okz = iz >= lo0 && iz <= hi0;
        const int oz = frequency2index(sp.centered, iz, sp.n0) * sz;
        float2 vz = make_float2(0.f, 0.f);
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const int iy = b1 + y;
            const bool oky = iy >= lo1 && iy <= hi1;
            float2 vy = make_float2(0.f, 0.f);
            if (okz && oky && okx0) {
                const float4 p = ldg_evict_last_half(pairs + (oz + frequency2index(sp.centered, iy, sp.n1) * sy + b2));
                vy = cfma(make_float2(p.x, p.y), w20, vy);
                if (okx1)
                    vy = cfma(make_float2(p.z, p.w), t2, vy);
            }
            vz = cfma(vy, w1[y], vz);
        }
        value = cfma(vz, w0[z], value);
    }
    value.y *= conjugate;
    return value;
}

// The y and x part of interp_linear_pairs, for samples that share it: sum(iz) is the sum over the cell's
// y and x taps in the z plane iz (which lies inside the volume), in interp_linear_pairs' order. `q1` and
// `q2` are the coordinates after the Friedel flip (q2 >= 0).
struct PairPlane {
    const float4* pairs;
    const Spectrum3 sp;
    int sz, row0, row1;       // element offsets of the two y rows, at the x cell
    bool ok0, ok1, okx1;
    float w10, w11, w20, w21;

    __device__ __forceinline__ PairPlane(const float4* p, int stride_z, int stride_y, const Spectrum3& s, float q1, float q2)
        : pairs(p), sp(s), sz(stride_z) {
        const float fl1 = floorf(q1), fl2 = floorf(q2);
        const int b1 = static_cast<int>(fl1), b2 = static_cast<int>(fl2);
        w11 = sub(q1, fl1);
        w21 = sub(q2, fl2);
        w10 = sub(1.f, w11);
        w20 = sub(1.f, w21);
        const int lo1 = -sp.n1 / 2, hi1 = (sp.n1 - 1) / 2, hi2 = sp.n2 / 2;
        const bool okx0 = b2 >= 0 && b2 <= hi2;
        ok0 = okx0 && b1 >= lo1 && b1 <= hi1;
        ok1 = okx0 && b1 + 1 >= lo1 && b1 + 1 <= hi1;
        okx1 = b2 + 1 <= hi2;
        row0 = frequency2index(sp.centered, b1, sp.n1) * stride_y + b2;
        row1 = frequency2index(sp.centered, b1 + 1, sp.n1) * stride_y + b2;
    }

    __device__ __forceinline__ float2 row(const float4 p) const {
        float2 v = cfma(make_float2(p.x, p.y), w20, make_float2(0.f, 0.f));
        return okx1 ? cfma(make_float2(p.z, p.w), w21, v) : v;
    }

    __device__ __forceinline__ float2 sum(int iz) const {
        const int oz = frequency2index(sp.centered, iz, sp.n0) * sz;
        float4 p0 = make_float4(0.f, 0.f, 0.f, 0.f), p1 = p0;
        if (ok0)
            p0 = ldg_evict_last_half(pairs + (oz + row0));
        if (ok1)
            p1 = ldg_evict_last_half(pairs + (oz + row1));
        const float2 v = cfma(row(p0), w10, make_float2(0.f, 0.f));
        return cfma(row(p1), w11, v);
    }
};

// Strides of a pair copy. Dense for the copies that callers hold (nb_volume_pairs). Copies that the library
// makes for itself pad rows to 4 and planes to 2 elements past a multiple of 8: the L1 serves eight 16-byte
// lanes at a time, each element in one of eight bank groups, and with these strides the 2 x 4 pixels that
// share a pass fall on 1.96 lines of a group on average over orientations, against 2.69 for 1 x 8 pixels
// over dense planes of an even number of rows, all of which start on the same banks (replayed on the CPU; the
// best of the 64 pairs of strides modulo 8). The L1's wavefronts are what bounds the extraction: 4096 slices
// of 256^3 1165 us -> 1104 us, with the matrix read once per slice and column (LeanColumn).
inline void dense_pairs(ProjArgs& a) {
    a.pair_sy = a.vol_w / 2 + 1;
    a.pair_sz = static_cast<int>(static_cast<int64_t>(a.vol_h) * a.pair_sy);  // pairs_apply bounds it
}

inline void pad_pairs(ProjArgs& a) {
    const int64_t sy = (a.vol_w / 2 + 1 + 3) / 8 * 8 + 4;
    const int64_t sz = (a.vol_h * sy + 5) / 8 * 8 + 2;
    if (sz * a.vol_d < (int64_t(1) << 31)) {
        a.pair_sy = static_cast<int>(sy);
        a.pair_sz = static_cast<int>(sz);
    }
}

inline int64_t pair_elements(const ProjArgs& a) { return static_cast<int64_t>(a.vol_d) * a.pair_sz; }

// Row and column of a lane within its warp's 4 x 8 pixels: 2 x 4 per eight lanes.
__device__ __forceinline__ int pair_row(int lane) { return (lane >> 4) * 2 + ((lane >> 2) & 1); }
__device__ __forceinline__ int pair_column(int lane) { return ((lane >> 3) & 1) * 4 + (lane & 3); }

// slice2grid for a Mat33 rotation with no scaling and no Ewald curvature, when the slice's matrix
// column 0 is finite: rotate() computes ((m_k0 * 0) + (m_k1 * f0)) + (m_k2 * f1), and for finite m_k0
// the first product is a zero whose sign never reaches the result (the coordinates then decide the
// cutoff, the cell, its weights and the Friedel flip the same way), so it is left out. The products with
// f1 are those of a column of pixels.
struct LeanColumn {
    float z1, y1, x1, z2, y2, x2;

    // Whether slice b of `a` can take the lean form. The matrix is read once, 16 bytes at a time (its 48
    // bytes are aligned): read per pixel it cost as many L1 wavefronts as one of the four tap loads.
    __device__ __forceinline__ bool load(const ProjArgs& a, int64_t b, float f1) {
        if (a.rot.kind != 2 || a.scale.kind != 0 || a.ews.on)
            return false;
        const float* m = xform_ptr(a.rot, b, 12);
        float m0, m2, m3, m5, m6, m8;
        if (a.rot.data) {
            const float4* rows = reinterpret_cast<const float4*>(m);
            const float4 r0 = __ldg(rows), r1 = __ldg(rows + 1);
            m0 = r0.x; z1 = r0.y; m2 = r0.z; m3 = r0.w;
            y1 = r1.x; m5 = r1.y; m6 = r1.z; x1 = r1.w;
            m8 = __ldg(m + 8);
        } else {
            m0 = m[0]; z1 = m[1]; m2 = m[2]; m3 = m[3];
            y1 = m[4]; m5 = m[5]; m6 = m[6]; x1 = m[7];
            m8 = m[8];
        }
        z2 = mul(m2, f1);
        y2 = mul(m5, f1);
        x2 = mul(m8, f1);
        return isfinite(m0) && isfinite(m3) && isfinite(m6);
    }

    __device__ __forceinline__ void at(float f0, float& z, float& y, float& x) const {
        z = add(mul(z1, f0), z2);
        y = add(mul(y1, f0), y2);
        x = add(mul(x1, f0), x2);
    }
};

// Whether a call may read the pair copy: LINEAR, complex volume given as an array, no input weights,
// no w-window (per-call extractions take extract_pairs_w_kernel for that), a copy addressable in 32
// bits. Scaling and the Ewald-sphere curvature only change the coordinates (slice2grid), which the
// pair kernels compute as the generic ones do.
inline bool pairs_apply(const ProjArgs& a) {
    const int64_t vox = static_cast<int64_t>(a.vol_d) * a.vol_h * (a.vol_w / 2 + 1);
    return a.interp == I_LINEAR && a.in_cplx && !a.in_w.present && !a.in.is_value && a.wsize <= 1 &&
           vox < (int64_t(1) << 31);
}

// From how many output pixels on a LINEAR extraction is faster through a pair copy made for it: two per
// voxel, four where the copy is twice the L2 and more (2^24 voxels), and 2^21 for its allocation and launch;
// 3 * 2^17 in a stream capture, where the allocation is a node of the graph. Called one after another, us without and
// with: 64^3 x 384 slices (6 pixels per voxel) 18 and 19, x 512 (8) 21 and 20; 96^3 x 192 (2) 21 and 21, x 384 (4) 31 and 29;
// 128^3 x 192 (1.5) 28 and 27, x 256 (2) 33 and 31, x 512 (4) 57 and 48; 160^3 x 320 (2) 58 and 51; 256^3 x 512 (2) 196 and 187,
// x 768 (3) 276 and 243; 384^3 x 1152 (3) 959 and 962, x 1536 (4) 1328 and 1253; 512^3 x 1536 (3) 2489 and 2622, x 2048 (4) 3349 and
// 3390, x 4096 (8) 6778 and 6473. In a graph: 64^3 x 160 (2.5) 9.1 and 9.1, x 192 (3) 10.6 and 9.0; 96^3 x 192 (2) 19 and 16;
// 128^3 x 256 (2) 32 and 26; 384^3 x 960 (2.5) 812 and 823. A smaller cutoff leaves less to gain: 77^3 x 575 slices (1.7 M
// pixels) with a cutoff of 0.3 25 and 29.
inline bool pairs_pay(int64_t pixels, int64_t voxels, cudaStream_t stream) {
    return pixels >= (voxels < (int64_t(1) << 24) ? 2 : 4) * voxels && pixels >= 3 * (int64_t(1) << 17) &&
           (pixels >= int64_t(1) << 21 || stream_capturing(stream));
}

// The same of the w-windowed extraction, by samples: three per voxel (four), and 2 M.
inline bool pairs_pay_w(int64_t samples, int64_t voxels) {
    return samples >= (voxels < (int64_t(1) << 24) ? 3 : 4) * voxels && samples >= (int64_t(1) << 21);
}

// The per-call LINEAR extraction from the volume itself (no w-window).
cudaError_t launch_extract_volume(const ProjArgs& a, cudaStream_t stream);

// Writes the pair copy of a.in (a.vol_d x a.vol_h x a.vol_w/2+1 complex values) to `pairs`. With
// `priority`, the launch carries that scheduling priority (kept by a graph captured from it).
cudaError_t launch_make_pairs(const ProjArgs& a, float4* pairs, cudaStream_t stream, const int* priority = nullptr);

// The per-call LINEAR extraction over a pair copy of a.in: one grid of (slice tile, slices) CTAs
// (extract_linear_kernel, or extract_pairs_w_kernel with a w-window).
cudaError_t launch_extract_pairs(const ProjArgs& a, const float4* pairs, cudaStream_t stream);

} // namespace nb
