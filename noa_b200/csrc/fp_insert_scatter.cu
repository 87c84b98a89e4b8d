// Slice-major scatter form of insert_central_slices_3d (windowed sinc), nb_insert_central_slices_3d_scatter.
//
// The gather form (fp_insert.cu) sums, for every voxel, the terms of the slices whose slab
// |fz| <= fftfreq_blackman contains it (FourierInsertInterpolate, FourierProject.hpp:478-519). This form
// enumerates the same (voxel, slice) pairs from the slice side: slice i's slab is thin along the axis
// where its normal n_i (row 0 of the inverse rotation) has the largest component per voxel, so a thread
// owns one column of voxels along that axis, computes the k range the slab can cover there (widened
// by one voxel; the exact test below decides), and for each voxel of it evaluates the term exactly as
// the gather form does — same rounded coordinates, cutoff, window and 2-D interpolation — and adds it
// with one reduction (value and weight interleaved) into a dense accumulator. A finalize pass applies
// the output conversion (|z|^2 for complex -> real, to the sum, as the reference does) and adds the
// accumulator into the caller's grids. Every term is the gather form's; only the order of the sum over
// slices differs (float atomics).
//
// Not used with an Ewald-sphere curvature (the slab is curved) or when the accumulator cannot be
// allocated: both run the gather form.
#include "fp_args.cuh"
#include "fp_pool.cuh"
#include "fp_slice_taps.cuh"

#include <algorithm>
#include <type_traits>

namespace nb {
namespace {

constexpr int SCATTER_THREADS = 256;

template<bool IN_C, bool W> struct AccT;
template<> struct AccT<true, true> { using T = float4; };   // re, im, weight, -
template<> struct AccT<true, false> { using T = float2; };  // re, im
template<> struct AccT<false, true> { using T = float2; };  // value, weight
template<> struct AccT<false, false> { using T = float; };

template<bool IN_C, bool W>
__device__ __forceinline__ void acc_red(void* acc, int off, float2 v, float w) {
    auto* p = static_cast<typename AccT<IN_C, W>::T*>(acc) + off;
    if constexpr (IN_C && W)
        atomicAdd(p, make_float4(v.x, v.y, w, 0.f));
    else if constexpr (IN_C)
        atomicAdd(p, v);
    else if constexpr (W)
        atomicAdd(p, make_float2(v.x, w));
    else
        atomicAdd(p, v.x);
}

// Six CTAs per SM for the LINEAR and NEAREST instantiations (39 registers, no spills): 512^3 x 20,000
// slices, 378.6 -> 364.2-365.1 ms on one box (1000 slices: 19.32 -> 18.79-18.82 ms). Left to the compiler the
// wider windows take up to 96 registers (two CTAs): 400 slices into 256^3, CUBIC 2280 us and 1440 us with four CTAs asked
// for; LANCZOS6 4640 us and 3280 us, LANCZOS8 8070 us and 6430 us with three.
template<int I>
constexpr int scatter_min_ctas() { return I == I_LINEAR || I == I_NEAREST ? 6 : I == I_CUBIC || I == I_BSPLINE ? 4 : 3; }

template<int I, bool IN_C, bool W>
__global__ void __launch_bounds__(SCATTER_THREADS, scatter_min_ctas<I>())
insert_scatter_kernel(const __grid_constant__ ProjArgs a, void* __restrict__ acc) {
    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const bool vc = a.out_centered;
    const Spectrum2 sp{a.slice_h, a.slice_w, a.in_centered, a.in_slice_narrow != 0};
    const bool has_in_w = a.in_w.present;
    // Frequency ranges: z in [-D/2, (D-1)/2], y in [-H/2, (H-1)/2], x in [0, W/2].
    auto lo_of = [&](int axis) { return axis == 0 ? -D / 2 : axis == 1 ? -H / 2 : 0; };
    auto hi_of = [&](int axis) { return axis == 0 ? (D - 1) / 2 : axis == 1 ? (H - 1) / 2 : WP - 1; };
    auto pick = [](int axis, float v0, float v1, float v2) { return axis == 0 ? v0 : axis == 1 ? v1 : v2; };
    const int col = blockIdx.x * SCATTER_THREADS + threadIdx.x;

    for (int64_t i = blockIdx.y; i < a.n_slices; i += gridDim.y) {
        const float3 n = rotation_row0(a.rot, i);
        const float c0 = n.x / a.target0, c1 = n.y / a.target1, c2 = n.z / a.target2;  // slab per index step
        const int ax = fabsf(c0) >= fabsf(c1) ? (fabsf(c0) >= fabsf(c2) ? 0 : 2) : (fabsf(c1) >= fabsf(c2) ? 1 : 2);
        const int p = ax == 0 ? 1 : 0, q = ax == 2 ? 1 : 2;   // the column's axes, q fastest
        const int ep = hi_of(p) - lo_of(p) + 1, eq = hi_of(q) - lo_of(q) + 1;
        if (col >= ep * eq)
            continue;
        const int kp = lo_of(p) + col / eq, kq = lo_of(q) + col % eq;
        const float fp = div(static_cast<float>(kp), pick(p, a.target0, a.target1, a.target2));
        const float fq = div(static_cast<float>(kq), pick(q, a.target0, a.target1, a.target2));
        if (fp * fp + fq * fq > a.cutoff_sqd * 1.0001f)
            continue;  // every voxel of the column is outside the cutoff
        int k_lo = lo_of(ax), k_hi = hi_of(ax);
        const float ca = pick(ax, c0, c1, c2);
        if (fabsf(ca) > 1e-30f) {
            const float s = pick(p, n.x, n.y, n.z) * fp + pick(q, n.x, n.y, n.z) * fq;
            const float t0 = (-a.fb - s) / ca, t1 = (a.fb - s) / ca;
            const float r0 = floorf(fminf(t0, t1)) - 1.f, r1 = ceilf(fmaxf(t0, t1)) + 1.f;
            // clamped in float first: the range stays within the axis whatever r0, r1 are (NaN included)
            k_lo = static_cast<int>(fmaxf(r0, static_cast<float>(k_lo)));
            k_hi = static_cast<int>(fminf(r1, static_cast<float>(k_hi)));
        }
        for (int ka = k_lo; ka <= k_hi; ++ka) {
            const int kz = ax == 0 ? ka : kp;
            const int ky = ax == 0 ? kp : (ax == 1 ? ka : kq);
            const int kx = ax == 2 ? ka : kq;
            // The gather form's term for voxel (kz, ky, kx) and slice i (fp_insert.cu,
            // FourierProject.hpp:479-518).
            const float fz = div(static_cast<float>(kz), a.target0);
            const float fy = div(static_cast<float>(ky), a.target1);
            const float fx = div(static_cast<float>(kx), a.target2);
            if (dot3(fz, fy, fx, fz, fy, fx) > a.cutoff_sqd)
                continue;
            float f0, f1;
            const float zz = grid2slice(fz, fy, fx, a.scale, a.rot, i, a.ews, f0, f1);
            if (!(fabsf(zz) <= a.fb))
                continue;
            const float window = windowed_sinc_fast(zz, a.pfs, a.ifs, a.pfb);
            const float q0 = mul(f0, a.f_slice0), q1 = mul(f1, a.f_slice1);
            const float2 v = cmul(interp_spectrum_2d<I, IN_C>(a.in, sp, i, q0, q1), window);
            float w = 0.f;
            if constexpr (W)
                w = has_in_w ? mul(interp_spectrum_2d<I, false>(a.in_w, sp, i, q0, q1).x, window) : window;
            const int off = (frequency2index(vc, kz, D) * H + frequency2index(vc, ky, H)) * WP + kx;
            acc_red<IN_C, W>(acc, off, v, w);
        }
    }
}

// The LINEAR form for Mat33 rotations without scaling, from slices with adjacent columns:
// insert_scatter_kernel's terms for few instructions per (voxel, slice) pair, which is what bounds it:
// 500 slices into 256^3 with half-width 6 and weights 2620 us -> 1333 us (1676 us one voxel at a time).
//
// The axis that the columns run along is a compile-time constant (the slice picks one of three bodies), so
// the products of the matrix with the column's two fixed frequencies, and the accumulator offset, are
// computed once per column; the frequencies come from a table per CTA instead of divisions; and the k
// range is widened by its rounding error instead of a whole voxel each side.
template<int AX, bool IN_C, bool W, typename Idx>
__device__ __forceinline__ void scatter_column(const ProjArgs& a, void* acc, const float* freq, int col, int64_t slice,
                                               const float* m) {
    constexpr int P = AX == 0 ? 1 : 0, Q = AX == 2 ? 1 : 2;  // the column's fixed axes, Q fastest
    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const int extent[3] = {D, H, WP}, lo[3] = {-D / 2, -H / 2, 0}, table[3] = {0, D, D + H};
    const int stride[3] = {H * WP, WP, 1};
    if (col >= extent[P] * extent[Q])
        return;
    const int ip = col / extent[Q], iq = col - ip * extent[Q];
    const float fp = freq[table[P] + ip], fq = freq[table[Q] + iq];
    if (fp * fp + fq * fq > a.cutoff_sqd * 1.0001f)
        return;  // every voxel of the column is outside the cutoff
    const float* fa = freq + table[AX];
    const float target = AX == 0 ? a.target0 : AX == 1 ? a.target1 : a.target2;
    const float slope = m[AX] / target;  // of the distance to the slice, per index
    int first = 0, last = extent[AX] - 1;
    if (fabsf(slope) > 1e-30f) {
        const float s = m[P] * fp + m[Q] * fq;
        const float t0 = (-a.fb - s) / slope, t1 = (a.fb - s) / slope;
        // s and the exact test below are each off by a few 1e-7 of the sum of their terms' sizes.
        const float slack = 0.01f + 4e-6f * (fabsf(m[P] * fp) + fabsf(m[Q] * fq) + a.fb) / fabsf(slope);
        // clamped in float first: the range stays within the axis whatever t0, t1 are (NaN included)
        first = static_cast<int>(fmaxf(ceilf(fminf(t0, t1) - slack) - static_cast<float>(lo[AX]), 0.f));
        last = static_cast<int>(fminf(floorf(fmaxf(t0, t1) + slack) - static_cast<float>(lo[AX]), static_cast<float>(last)));
    }
    const Spectrum2 sp{a.slice_h, a.slice_w, a.in_centered, true};
    const bool vc = a.out_centered, has_in_w = a.in_w.present;
    const auto index = [vc](int k, int n) { return frequency2index(vc, k, n); };
    // Offset of the column; x frequencies are their indices.
    const int offset = index(lo[P] + ip, extent[P]) * stride[P] + (Q == 2 ? iq : index(lo[Q] + iq, extent[Q]) * stride[Q]);
    const Idx s1 = static_cast<Idx>(a.in.s1);
    const WindowPair window_of(a);
    using T = typename std::conditional<IN_C, float2, float>::type;
    const T* base = static_cast<const T*>(a.in.data) + slice * a.in.s0;
    const float* base_w = has_in_w ? static_cast<const float*>(a.in_w.data) + slice * a.in_w.s0 : nullptr;
    // v0 z + v1 y + v2 x summed in that order, the terms of the fixed axes given; for two voxels at a time.
    const auto both = [](float v) { return pack2(v, v); };
    const auto dot = [both](float c, float f0, float f1, float p, float q) {
        const unsigned long long run = pack2(mul(c, f0), mul(c, f1));
        return AX == 0 ? add2(add2(run, both(p)), both(q)) : AX == 1 ? add2(add2(both(p), run), both(q))
                                                                     : add2(both(add(p, q)), run);
    };
    const auto dot3_axis = [](float run, float p, float q) {
        return AX == 0 ? add(add(run, p), q) : AX == 1 ? add(add(p, run), q) : add(add(p, q), run);
    };
    const float pp = mul(fp, fp), qq = mul(fq, fq);
    const float p0 = mul(m[P], fp), q0 = mul(m[Q], fq), p1 = mul(m[3 + P], fp), q1 = mul(m[3 + Q], fq);
    const float p2 = mul(m[6 + P], fp), q2 = mul(m[6 + Q], fq);
    for (int k = first; k <= last; k += 2) {
        // The gather form's terms (fp_insert.cu, FourierProject.hpp:479-518).
        const float f0 = fa[k], f1 = fa[min(k + 1, last)];
        const unsigned long long zz = dot(m[AX], f0, f1, p0, q0);
        const float2 z = unpack2(zz);
        const float sqd0 = dot3_axis(mul(f0, f0), pp, qq), sqd1 = dot3_axis(mul(f1, f1), pp, qq);
        const bool in0 = fabsf(z.x) <= a.fb && !(sqd0 > a.cutoff_sqd);
        const bool in1 = k < last && fabsf(z.y) <= a.fb && !(sqd1 > a.cutoff_sqd);
        if (!in0 && !in1)
            continue;
        const float2 window = window_of(zz);
        const float2 c0 = unpack2(mul2(dot(m[3 + AX], f0, f1, p1, q1), both(a.f_slice0)));
        const float2 c1 = unpack2(mul2(dot(m[6 + AX], f0, f1, p2, q2), both(a.f_slice1)));
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            if (!(e ? in1 : in0))
                continue;
            float w = e ? window.y : window.x;
            const float s0 = e ? c0.y : c0.x, s1_ = e ? c1.y : c1.x;
            float2 v;
            if constexpr (IN_C)
                v = cmul(slice_value(base, sp, s1, s0, s1_), w);
            else
                v = make_float2(slice_value(base, sp, s1, s0, s1_) * w, 0.f);
            if (W && has_in_w) {
                const LinearCell cell(sp, s0, s1_);
                w = mul(cell.read(base_w, static_cast<Idx>(a.in_w.s1), static_cast<Idx>(a.in_w.s2)).x, w);
            }
            acc_red<IN_C, W>(acc, offset + (AX == 2 ? k + e : index(lo[AX] + k + e, extent[AX]) * stride[AX]), v, w);
        }
    }
}

// Frequencies of one CTA's table: all indices of the three axes.
constexpr int SCATTER_TABLE = 8192;

// Six CTAs per SM (40 registers): 1333 us against 1386 us with the compiler's five, 1448 us with four, 500
// slices into 256^3 with half-width 6.
template<bool IN_C, bool W, typename Idx>
__global__ void __launch_bounds__(SCATTER_THREADS, 6)
scatter_linear_kernel(const __grid_constant__ ProjArgs a, void* __restrict__ acc) {
    extern __shared__ float s_freq[];
    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    for (int i = threadIdx.x; i < D + H + WP; i += SCATTER_THREADS) {
        const int k = i < D ? i - D / 2 : i < D + H ? i - D - H / 2 : i - D - H;
        s_freq[i] = div(static_cast<float>(k), i < D ? a.target0 : i < D + H ? a.target1 : a.target2);
    }
    __syncthreads();
    const int col = blockIdx.x * SCATTER_THREADS + threadIdx.x;
    for (int64_t i = blockIdx.y; i < a.n_slices; i += gridDim.y) {
        const float* m = xform_ptr(a.rot, i, 12);
        const float c0 = fabsf(m[0] / a.target0), c1 = fabsf(m[1] / a.target1), c2 = fabsf(m[2] / a.target2);
        if (c0 >= c1 && c0 >= c2)
            scatter_column<0, IN_C, W, Idx>(a, acc, s_freq, col, i, m);
        else if (c1 >= c2)
            scatter_column<1, IN_C, W, Idx>(a, acc, s_freq, col, i, m);
        else
            scatter_column<2, IN_C, W, Idx>(a, acc, s_freq, col, i, m);
    }
}

// Whether scatter_linear_kernel applies.
bool use_linear_scatter(const ProjArgs& a) {
    return linear_slices(a) && a.rot.kind == 2 && a.scale.kind == 0 &&
           static_cast<int64_t>(a.vol_d) + a.vol_h + a.vol_w / 2 + 1 <= SCATTER_TABLE;
}

// Caller's grids += the accumulator (dense, the caller's index order), converted to the output type.
template<bool IN_C, bool OUT_C, bool W>
__global__ void scatter_finalize_kernel(const __grid_constant__ ProjArgs a, const void* __restrict__ acc) {
    using T = typename AccT<IN_C, W>::T;
    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const int64_t n = static_cast<int64_t>(D) * H * WP;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        const int x = static_cast<int>(i % WP);
        const int64_t zy = i / WP;
        const int y = static_cast<int>(zy % H), z = static_cast<int>(zy / H);
        const T s = static_cast<const T*>(acc)[i];
        float2 v;
        float w = 0.f;
        if constexpr (IN_C && W) { v = make_float2(s.x, s.y); w = s.z; }
        else if constexpr (IN_C) { v = s; }
        else if constexpr (W) { v = make_float2(s.x, 0.f); w = s.y; }
        else { v = make_float2(s, 0.f); }
        const float2 o = to_output<IN_C, OUT_C>(v);
        dst_store<OUT_C>(a.out, z, y, x, cadd(dst_load<OUT_C>(a.out, z, y, x), o));
        if constexpr (W)
            store_real(a.out_w, z, y, x, add(load_real(a.out_w, z, y, x), w));
    }
}

template<int I, bool IN_C, bool OUT_C, bool W>
cudaError_t launch_typed(const ProjArgs& a, cudaStream_t stream, bool& done) {
    done = false;
    using T = typename AccT<IN_C, W>::T;
    const int64_t D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const int64_t vox = D * H * WP;
    const size_t bytes = static_cast<size_t>(vox) * sizeof(T);
    void* acc = scratch_alloc(bytes, stream);
    if (!acc)
        return cudaSuccess;
    cudaError_t err = cudaMemsetAsync(acc, 0, bytes, stream);
    if (err == cudaSuccess) {
        const int64_t cols = std::max(H * WP, std::max(D * WP, D * H));
        const dim3 grid(static_cast<unsigned>((cols + SCATTER_THREADS - 1) / SCATTER_THREADS),
                        static_cast<unsigned>(a.n_slices < 65535 ? a.n_slices : 65535));
        if (I == I_LINEAR && use_linear_scatter(a)) {
            const size_t table = static_cast<size_t>(D + H + WP) * sizeof(float);
            if (a.in_slice_narrow)
                scatter_linear_kernel<IN_C, W, int><<<grid, SCATTER_THREADS, table, stream>>>(a, acc);
            else
                scatter_linear_kernel<IN_C, W, int64_t><<<grid, SCATTER_THREADS, table, stream>>>(a, acc);
        } else {
            insert_scatter_kernel<I, IN_C, W><<<grid, SCATTER_THREADS, 0, stream>>>(a, acc);
        }
        const int64_t blocks = (vox + 255) / 256;
        const int grid_f = static_cast<int>(blocks < static_cast<int64_t>(sm_count()) * 16 ? blocks : sm_count() * 16);
        scatter_finalize_kernel<IN_C, OUT_C, W><<<grid_f, 256, 0, stream>>>(a, acc);
        err = cudaGetLastError();
    }
    scratch_free(acc, stream);
    done = err == cudaSuccess;
    return err;
}

template<int I, bool IN_C, bool OUT_C>
cudaError_t launch_w(const ProjArgs& a, cudaStream_t stream, bool& done) {
    return a.out_w.present ? launch_typed<I, IN_C, OUT_C, true>(a, stream, done)
                           : launch_typed<I, IN_C, OUT_C, false>(a, stream, done);
}

template<int I>
cudaError_t launch_interp(const ProjArgs& a, cudaStream_t stream, bool& done) {
    if (a.in_cplx && a.out_cplx)
        return launch_w<I, true, true>(a, stream, done);
    if (a.in_cplx)
        return launch_w<I, true, false>(a, stream, done);
    return launch_w<I, false, false>(a, stream, done);
}

} // namespace

cudaError_t launch_insert_scatter(const ProjArgs& a, cudaStream_t stream) {
    const int64_t vox = static_cast<int64_t>(a.vol_d) * a.vol_h * (a.vol_w / 2 + 1);
    if (a.n_slices == 0 || a.ews.on || vox >= (int64_t(1) << 31))
        return launch_insert(a, stream);
    bool done = false;
    cudaError_t err;
    switch (a.interp) {
        case I_NEAREST: err = launch_interp<I_NEAREST>(a, stream, done); break;
        case I_LINEAR: err = launch_interp<I_LINEAR>(a, stream, done); break;
        case I_CUBIC: err = launch_interp<I_CUBIC>(a, stream, done); break;
        case I_BSPLINE: err = launch_interp<I_BSPLINE>(a, stream, done); break;
        case I_LANCZOS4: err = launch_interp<I_LANCZOS4>(a, stream, done); break;
        case I_LANCZOS6: err = launch_interp<I_LANCZOS6>(a, stream, done); break;
        case I_LANCZOS8: err = launch_interp<I_LANCZOS8>(a, stream, done); break;
        default: return cudaErrorInvalidValue;
    }
    if (err != cudaSuccess || done)
        return err;
    return launch_insert(a, stream);
}

} // namespace nb
