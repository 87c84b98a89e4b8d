// extract_central_slices_3d on sm_100a: one thread per output pixel, 3-D spectrum interpolation of
// the volume (FourierExtract, noa/xform/FourierProject.hpp:632-694).
//
// Work decomposition: a CTA owns a 16x16 tile of one slice (blockIdx.x = tile, blockIdx.y strides
// over slices), each warp a 4x8 sub-tile, so the rotation is uniform per CTA and a warp's taps fall on
// a compact patch of the volume; taps are read through the non-coherent L1 path. Volume offsets are
// 32-bit whenever the volume fits, and the LINEAR path resolves bounds and frequency2index once per
// axis rather than once per tap. LINEAR extraction of a complex volume with enough pixels first makes
// a pair copy of the volume (fp_pairs.cuh) and reads each trilinear cell as four 16-byte loads, four
// pixels per thread (extract_linear_kernel; extract_pairs_w_kernel with the w-window).
//
// The w-windowed form (wsize > 1) keeps the reference's semantics — outputs are the windowed sum over
// the w offsets of the z-shifted samples — but sums in registers, in w order, instead of zeroing the
// outputs and adding atomically, so it is deterministic and needs no extra pass.
#include "fp_args.cuh"
#include "fp_pairs.cuh"
#include "fp_pool.cuh"
#include "fp_window.cuh"

#include <climits>
#include <type_traits>

namespace nb {
namespace {

constexpr int TY = 16, TX = 16, EXTRACT_THREADS = TY * TX;

// ---------------------------------------------------------------------------------------------------
// Fast LINEAR path over a pair copy of the volume (fp_pairs.cuh). Each thread interpolates PPT
// pixels (rows y, y+16, ...) of one column, keeping more loads in flight.
// ---------------------------------------------------------------------------------------------------
constexpr int PPT = 4;

// The w-window's offsets and values do not depend on the pixel, so a CTA tabulates them once (the same
// expressions as the per-sample ones, hence the same bits) instead of dividing and evaluating the window
// for every pixel and offset. Windows of more than W_TABLE offsets evaluate the rest per sample.
constexpr int W_TABLE = 64;

// Called by every thread of the CTA before any of them returns (it synchronizes when wsize > 1).
__device__ __forceinline__ void fill_w_table(const ProjArgs& a, float2* table) {
    if (a.wsize <= 1)
        return;
    for (int w = threadIdx.x; w < a.wsize && w < W_TABLE; w += blockDim.x)
        table[w] = w_sample(a, w);
    __syncthreads();
}

// Idx: the type of the linear voxel index, 32-bit when the volume has fewer than 2^31 voxels (its
// divisions then cost a fifth of the 64-bit ones, which bounded the copy).
template<typename Idx>
__global__ void make_pairs(const __grid_constant__ ProjArgs a, float4* __restrict__ pairs) {
    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const Idx n = static_cast<Idx>(D) * H * WP;
    const float2* vol = static_cast<const float2*>(a.in.data);
    for (Idx i = blockIdx.x * static_cast<Idx>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<Idx>(gridDim.x) * blockDim.x) {
        const int x = static_cast<int>(i % static_cast<Idx>(WP));
        const Idx zy = i / static_cast<Idx>(WP);
        const int y = static_cast<int>(zy % static_cast<Idx>(H)), z = static_cast<int>(zy / static_cast<Idx>(H));
        const int64_t off = z * a.in.s0 + y * a.in.s1 + x * a.in.s2;
        const float2 v0 = vol[off];
        const float2 v1 = x + 1 < WP ? vol[off + a.in.s2] : make_float2(0.f, 0.f);
        pairs[z * static_cast<Idx>(a.pair_sz) + y * static_cast<Idx>(a.pair_sy) + x] = make_float4(v0.x, v0.y, v1.x, v1.y);
    }
}

// LINEAR extraction without a w-window: a CTA owns PPT tiles of TY x TX pixels of `per_cta` consecutive
// slices, a thread PPT pixels (rows y, y + TY, ...) of one column, so that what depends on the pixel alone
// (its 2-D frequency, its offset) is computed once for all slices, and what depends on the slice and the
// column once for PPT pixels. PAIRS: the taps come from a pair copy (four 16-byte loads per pixel), else
// from the volume (eight loads). Same bits
// as one slice per CTA and one pixel at a time: 4096 slices of 256^3 1195 us -> 1164 us with the copy
// (1104 us with the copy padded, pad_pairs); 150 slices of 200^3 without it 50.1 us -> 41.2 us.
template<bool PAIRS, bool IN_C, bool OUT_C, typename Idx>
__global__ void __launch_bounds__(EXTRACT_THREADS, 5)
extract_linear_kernel(const __grid_constant__ ProjArgs a, const float4* __restrict__ pairs, int ntx, int per_cta,
                      bool lanes_16) {
    const int wp = a.slice_w / 2 + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // A warp's pixels: 4 x 8, 2 x 4 per eight lanes, over a pair copy; else 4 x 8, or 2 x 16 (lanes_16).
    const int row = PAIRS ? (warp >> 1) * 4 + pair_row(lane) : lanes_16 ? warp * 2 + (lane >> 4) : (warp >> 1) * 4 + (lane >> 3);
    const int column = PAIRS ? (warp & 1) * 8 + pair_column(lane) : lanes_16 ? lane & 15 : (warp & 1) * 8 + (lane & 7);
    const int y0 = (blockIdx.x / ntx) * (TY * PPT) + row;
    const int u = (blockIdx.x % ntx) * TX + column;
    if (u >= wp || y0 >= a.slice_h)
        return;
    const Spectrum3 sp{a.vol_d, a.vol_h, a.vol_w, a.in_centered};
    const int sz = a.pair_sz, sy = a.pair_sy;
    const View3<Idx> vol{a.in.data, static_cast<Idx>(a.in.s0), static_cast<Idx>(a.in.s1), static_cast<Idx>(a.in.s2)};
    const bool has_out_w = a.out_w.present;
    const bool has_in_w = !PAIRS && a.in_w.present;
    const float f1 = div(static_cast<float>(u), a.f_slice1);
    float f0[PPT];
#pragma unroll
    for (int r = 0; r < PPT; ++r)
        f0[r] = div(static_cast<float>(index2frequency(a.out_centered, y0 + r * TY, a.slice_h)), a.f_slice0);
    const int64_t pixel = y0 * a.out.s1 + u * a.out.s2, pixel_w = y0 * a.out_w.s1 + u * a.out_w.s2;

    for (int64_t first = blockIdx.y * static_cast<int64_t>(per_cta); first < a.n_slices;
         first += static_cast<int64_t>(gridDim.y) * per_cta) {
        const int64_t end = first + per_cta < a.n_slices ? first + per_cta : a.n_slices;
        for (int64_t b = first; b < end; ++b) {
            LeanColumn column_of;
            const bool lean = column_of.load(a, b, f1);
            using T = typename std::conditional<OUT_C, float2, float>::type;
            T* out = static_cast<T*>(a.out.data) + (b * a.out.s0 + pixel);
            float* out_w = static_cast<float*>(a.out_w.data) + (b * a.out_w.s0 + pixel_w);
#pragma unroll
            for (int r = 0; r < PPT; ++r) {
                if (y0 + r * TY >= a.slice_h)
                    break;
                float fz, fy, fx;
                if (lean)
                    column_of.at(f0[r], fz, fy, fx);
                else
                    slice2grid(f0[r], f1, a.scale, a.rot, b, a.ews, fz, fy, fx);
                float2 value = make_float2(0.f, 0.f);
                float weight = 0.f;
                if (dot3(fz, fy, fx, fz, fy, fx) <= a.cutoff_sqd) {
                    const float q0 = mul(fz, a.target0), q1 = mul(fy, a.target1), q2 = mul(fx, a.target2);
                    if constexpr (PAIRS)
                        value = interp_linear_pairs(pairs, sz, sy, sp, q0, q1, q2);
                    else
                        value = interp_linear_3d<IN_C>(vol, sp, q0, q1, q2);
                    value = to_output<IN_C, OUT_C>(value);
                    weight = 1.f;
                    if (has_in_w && has_out_w) {
                        const View3<Idx> volw{a.in_w.data, static_cast<Idx>(a.in_w.s0), static_cast<Idx>(a.in_w.s1),
                                              static_cast<Idx>(a.in_w.s2)};
                        weight = interp_linear_3d<false>(volw, sp, q0, q1, q2).x;
                    }
                }
                if constexpr (OUT_C)
                    __stcs(out, value);
                else
                    __stcs(out, value.x);
                out += TY * a.out.s1;
                if (has_out_w) {
                    __stcs(out_w, weight);
                    out_w += TY * a.out_w.s1;
                }
            }
        }
    }
}

// Slices per CTA: as many (up to 8) as leave the launch 16 CTAs for each that the chip holds at a time.
int slices_per_cta(int64_t tiles, int64_t slices) {
    const int64_t s = tiles * slices / (static_cast<int64_t>(sm_count()) * 5 * 16);
    return static_cast<int>(s < 1 ? 1 : s > 8 ? 8 : s);
}

template<bool PAIRS, bool IN_C, bool OUT_C, typename Idx>
cudaError_t launch_linear(const ProjArgs& a, const float4* pairs, cudaStream_t stream) {
    const int wp = a.slice_w / 2 + 1;
    const int ntx = (wp + TX - 1) / TX, nty = (a.slice_h + TY * PPT - 1) / (TY * PPT);
    const int per_cta = slices_per_cta(static_cast<int64_t>(ntx) * nty, a.n_slices);
    const int64_t groups = (a.n_slices + per_cta - 1) / per_cta;
    const dim3 grid(static_cast<unsigned>(ntx * nty), static_cast<unsigned>(groups < 65535 ? groups : 65535));
    // Without a pair copy sixteen lanes share a pass of the L1, over 16 bank groups of 8 bytes. Planes that
    // all start on the same banks (boxes that are a multiple of 32) are read with 3.4 lines a group by lanes
    // in a row and 4.1 by lanes in two rows of 8, others with 2.5 and 2.3 (replayed on the CPU).
    const bool lanes_16 = !PAIRS && a.in.s0 % 16 == 0;
    extract_linear_kernel<PAIRS, IN_C, OUT_C, Idx><<<grid, EXTRACT_THREADS, 0, stream>>>(a, pairs, ntx, per_cta, lanes_16);
    return cudaGetLastError();
}

// Without a pair copy: whether the launch is large enough for four pixels per thread. One pixel per thread
// (extract_kernel) has four times the threads to hide the taps' latency with, up to so many rounds of the chip's
// 2048 threads per SM (303 k pixels): three, two in a batch, whose grids fill the chip together. us of
// extract_kernel and of extract_linear_kernel, means over boxes of 48 to 256: 0.65 M pixels 12.5 and 14.1, 1.3 M 21.9 and
// 21.9, 1.8 M 28.8 and 27.5; with weights 1.3 M 31.3 and 33.5, 1.8 M 41.4 and 41.8; real 0.65 M 11.4 and 12.1, 0.9 M 14.8
// and 15.2, 1.3 M 20.0 and 19.0. With a cutoff of 0.3 fewer taps are waited for: 1.1 M with weights 16.4 and 14.6. Batches
// by lines at five, at two and at none: 59 requests of 0.02 M to 1.2 M 352, 329 and 309, 41 of 0.06 M to 2.1 M 322, 291 and 276,
// but 49 of up to 0.2 M 48 at two and 57 at none, 29 of 30 k 27 and 33.
bool use_linear_kernel(const ProjArgs& a, int rounds) {
    const int64_t pixels = a.n_slices * a.slice_h * static_cast<int64_t>(a.slice_w / 2 + 1);
    return a.interp == I_LINEAR && a.wsize <= 1 && pixels >= static_cast<int64_t>(sm_count()) * 2048 * rounds;
}

// The w-windowed form over the pair copy: per pixel, the windowed sum over the w offsets of the
// z-shifted samples — extract_kernel's w loop step for step (same offsets, cutoff tests, window values
// and sum order), so the results are bit-identical to it. The offsets are whole z samples, so one
// sample's cell and the next one's share a z plane: its sum over y and x (the inner part of the sample's
// sum, in its order) is kept, and each sample but the first reads two pair rows instead of four.
// 1000 slices of 256^2 with 7 offsets and weights: 1417 us -> 1192 us (1113 us with the offsets tabulated
// beside their window values, 1067 us with the padded copy).
template<bool OUT_C>
__global__ void __launch_bounds__(EXTRACT_THREADS)
extract_pairs_w_kernel(const __grid_constant__ ProjArgs a, const float4* __restrict__ pairs, int ntx) {
    const int wp = a.slice_w / 2 + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y0 = (blockIdx.x / ntx) * (TY * PPT) + (warp >> 1) * 4 + pair_row(lane);
    const int u = (blockIdx.x % ntx) * TX + (warp & 1) * 8 + pair_column(lane);
    __shared__ float2 s_w[W_TABLE];
    fill_w_table(a, s_w);
    if (u >= wp)
        return;
    const Spectrum3 sp{a.vol_d, a.vol_h, a.vol_w, a.in_centered};
    const int sz = a.pair_sz, sy = a.pair_sy;
    const int lo0 = -sp.n0 / 2, hi0 = (sp.n0 - 1) / 2;
    const bool has_out_w = a.out_w.present;
    const float f1 = div(static_cast<float>(u), a.f_slice1);

    for (int64_t b = blockIdx.y; b < a.n_slices; b += gridDim.y) {
#pragma unroll 1
        for (int r = 0; r < PPT; ++r) {
            const int y = y0 + r * TY;
            if (y >= a.slice_h)
                break;
            const float f0 = div(static_cast<float>(index2frequency(a.out_centered, y, a.slice_h)), a.f_slice0);
            float fz, fy, fx;
            slice2grid(f0, f1, a.scale, a.rot, b, a.ews, fz, fy, fx);
            // What the samples share: the Friedel flip, the y and x cell and its weights.
            const float qx = mul(fx, a.target2);
            const bool flip = qx < 0.f;
            const PairPlane plane(pairs, sz, sy, sp, flip ? -mul(fy, a.target1) : mul(fy, a.target1), flip ? -qx : qx);
            const int step = flip ? -1 : 1;  // how the z cell moves with w
            int last_cell = INT_MIN / 2;
            float2 last = make_float2(0.f, 0.f);
            float2 value = make_float2(0.f, 0.f);
            float weight = 0.f;
            for (int w = 0; w < a.wsize; ++w) {
                const float2 offset = w < W_TABLE ? s_w[w] : w_sample(a, w);
                const float gz = add(fz, offset.x);
                if (dot3(gz, fy, fx, gz, fy, fx) > a.cutoff_sqd)
                    continue;
                const float cw = offset.y;
                const float qz = flip ? -mul(gz, a.target0) : mul(gz, a.target0);
                const float fl = floorf(qz);
                const int cell = static_cast<int>(fl);
                const float t = sub(qz, fl);
                // The plane the cell shares with the previous one, unless rounding moved it otherwise.
                const int shared = flip ? cell + 1 : cell, fresh = flip ? cell : cell + 1;
                if (cell - last_cell != step)
                    last = shared >= lo0 && shared <= hi0 ? plane.sum(shared) : make_float2(0.f, 0.f);
                const float2 next = fresh >= lo0 && fresh <= hi0 ? plane.sum(fresh) : make_float2(0.f, 0.f);
                float2 sample = cfma(flip ? next : last, sub(1.f, t), make_float2(0.f, 0.f));
                sample = cfma(flip ? last : next, t, sample);
                if (flip)
                    sample.y = -sample.y;
                last = next;
                last_cell = cell;
                const float2 iv = to_output<true, OUT_C>(sample);
                value = cadd(value, cmul(iv, cw));
                if (has_out_w)
                    weight = add(weight, mul(1.f, cw));
            }
            dst_store_stream<OUT_C>(a.out, b, y, u, value);
            if (has_out_w)
                store_real_stream(a.out_w, b, y, u, weight);
        }
    }
}

// Whether the per-call pair path applies: the pair copy is readable (pairs_apply) and there are enough
// pixels to amortise making it.
bool use_pairs(const ProjArgs& a, cudaStream_t stream) {
    const int64_t vox = static_cast<int64_t>(a.vol_d) * a.vol_h * (a.vol_w / 2 + 1);
    const int64_t pix = a.n_slices * a.slice_h * static_cast<int64_t>(a.slice_w / 2 + 1);
    ProjArgs plain = a;
    plain.wsize = 1;  // the w-windowed form reads the pair copy too (extract_pairs_w_kernel)
    if (!pairs_apply(plain))
        return false;
    return a.wsize > 1 ? pairs_pay_w(pix * a.wsize, vox) : pairs_pay(pix, vox, stream);
}

cudaError_t launch_pairs(const ProjArgs& call, cudaStream_t stream, bool& done) {
    done = false;
    ProjArgs a = call;
    pad_pairs(a);
    float4* pairs = static_cast<float4*>(scratch_alloc(static_cast<size_t>(pair_elements(a)) * sizeof(float4), stream));
    if (!pairs)
        return cudaSuccess; // no scratch: the caller takes the generic path
    launch_make_pairs(a, pairs, stream);
    const cudaError_t err = launch_extract_pairs(a, pairs, stream);
    scratch_free(pairs, stream);
    done = err == cudaSuccess;
    return err;
}

// NEAREST, and LINEAR from the volume in small launches or with a w-window: one pixel per thread.
template<int I, bool IN_C, bool OUT_C, typename Idx>
__global__ void __launch_bounds__(EXTRACT_THREADS)
extract_kernel(const __grid_constant__ ProjArgs a, int ntx) {
    const int wp = a.slice_w / 2 + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y = (blockIdx.x / ntx) * TY + (warp >> 1) * 4 + (lane >> 3);
    const int u = (blockIdx.x % ntx) * TX + (warp & 1) * 8 + (lane & 7);
    __shared__ float2 s_w[W_TABLE];
    fill_w_table(a, s_w);
    if (u >= wp || y >= a.slice_h)
        return;
    const Spectrum3 sp{a.vol_d, a.vol_h, a.vol_w, a.in_centered};
    const View3<Idx> vol{a.in.data, static_cast<Idx>(a.in.s0), static_cast<Idx>(a.in.s1), static_cast<Idx>(a.in.s2)};
    const View3<Idx> volw{a.in_w.data, static_cast<Idx>(a.in_w.s0), static_cast<Idx>(a.in_w.s1),
                          static_cast<Idx>(a.in_w.s2)};
    const bool has_out_w = a.out_w.present;
    const bool has_in_w = a.in_w.present;
    const int v = index2frequency(a.out_centered, y, a.slice_h);
    const float f0 = div(static_cast<float>(v), a.f_slice0);
    const float f1 = div(static_cast<float>(u), a.f_slice1);

    for (int64_t b = blockIdx.y; b < a.n_slices; b += gridDim.y) {
        float fz, fy, fx;
        slice2grid(f0, f1, a.scale, a.rot, b, a.ews, fz, fy, fx);

        float2 value = make_float2(0.f, 0.f);
        float weight = 0.f;
        if (a.wsize <= 1) {
            if (dot3(fz, fy, fx, fz, fy, fx) <= a.cutoff_sqd) {
                const float q0 = mul(fz, a.target0), q1 = mul(fy, a.target1), q2 = mul(fx, a.target2);
                value = to_output<IN_C, OUT_C>(interp_3d<I, IN_C>(vol, sp, q0, q1, q2));
                if (has_out_w)
                    weight = has_in_w ? interp_3d<I, false>(volw, sp, q0, q1, q2).x : 1.f;
            }
        } else {
            for (int w = 0; w < a.wsize; ++w) {
                const float2 offset = w < W_TABLE ? s_w[w] : w_sample(a, w);
                const float gz = add(fz, offset.x);
                if (dot3(gz, fy, fx, gz, fy, fx) > a.cutoff_sqd)
                    continue;
                const float q0 = mul(gz, a.target0), q1 = mul(fy, a.target1), q2 = mul(fx, a.target2);
                const float cw = offset.y;
                const float2 iv = to_output<IN_C, OUT_C>(interp_3d<I, IN_C>(vol, sp, q0, q1, q2));
                value = cadd(value, cmul(iv, cw));
                if (has_out_w) {
                    const float iw = has_in_w ? interp_3d<I, false>(volw, sp, q0, q1, q2).x : 1.f;
                    weight = add(weight, mul(iw, cw));
                }
            }
        }
        dst_store_stream<OUT_C>(a.out, b, y, u, value);
        if (has_out_w)
            store_real_stream(a.out_w, b, y, u, weight);
    }
}

// Windows of 4 taps and more (fp_window.cuh): each warp owns a 4x8 patch, as in extract_kernel.
template<int I, bool IN_C, bool OUT_C, typename Idx>
__global__ void __launch_bounds__(EXTRACT_THREADS, 3)
extract_window_kernel(const __grid_constant__ ProjArgs a, int ntx) {
    __shared__ __align__(16) WindowSlots<I> s_slots[EXTRACT_THREADS / 32];
    __shared__ float2 s_w[W_TABLE];
    fill_w_table(a, s_w);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int y = (blockIdx.x / ntx) * TY + (warp >> 1) * 4 + (lane >> 3);
    const int u = (blockIdx.x % ntx) * TX + (warp & 1) * 8 + (lane & 7);
    const bool valid = u < a.slice_w / 2 + 1 && y < a.slice_h;
    if (!__any_sync(0xffffffffu, valid))
        return;
    for (int64_t b = blockIdx.y; b < a.n_slices; b += gridDim.y)
        extract_window_patch<I, IN_C, OUT_C, Idx>(a, b, y, u, valid, s_slots[warp], s_w, W_TABLE);
}

template<int I, bool IN_C, bool OUT_C>
cudaError_t launch_typed(const ProjArgs& a, cudaStream_t stream, int rounds) {
    const int wp = a.slice_w / 2 + 1;
    const int ntx = (wp + TX - 1) / TX, nty = (a.slice_h + TY - 1) / TY;
    if (a.n_slices == 0)
        return cudaSuccess;
    const dim3 grid(static_cast<unsigned>(ntx * nty), static_cast<unsigned>(a.n_slices < 65535 ? a.n_slices : 65535));
    if constexpr (I == I_LINEAR) {
        if (use_linear_kernel(a, rounds))
            return a.wide_in ? launch_linear<false, IN_C, OUT_C, int64_t>(a, nullptr, stream)
                             : launch_linear<false, IN_C, OUT_C, int32_t>(a, nullptr, stream);
    }
    if constexpr (has_window<I>()) {
        if (a.in_bytes_narrow)
            extract_window_kernel<I, IN_C, OUT_C, uint32_t><<<grid, EXTRACT_THREADS, 0, stream>>>(a, ntx);
        else
            extract_window_kernel<I, IN_C, OUT_C, int64_t><<<grid, EXTRACT_THREADS, 0, stream>>>(a, ntx);
    } else {
        if (a.wide_in)
            extract_kernel<I, IN_C, OUT_C, int64_t><<<grid, EXTRACT_THREADS, 0, stream>>>(a, ntx);
        else
            extract_kernel<I, IN_C, OUT_C, int32_t><<<grid, EXTRACT_THREADS, 0, stream>>>(a, ntx);
    }
    return cudaGetLastError();
}

template<int I>
cudaError_t launch_interp(const ProjArgs& a, cudaStream_t stream, int rounds = 3) {
    if (a.in_cplx && a.out_cplx)
        return launch_typed<I, true, true>(a, stream, rounds);
    if (a.in_cplx)
        return launch_typed<I, true, false>(a, stream, rounds);
    return launch_typed<I, false, false>(a, stream, rounds);
}

} // namespace

cudaError_t launch_extract_pairs(const ProjArgs& a, const float4* pairs, cudaStream_t stream) {
    if (a.n_slices <= 0)
        return cudaSuccess;
    if (a.wsize <= 1)
        return a.out_cplx ? launch_linear<true, true, true, int>(a, pairs, stream)
                          : launch_linear<true, true, false, int>(a, pairs, stream);
    const int wp = a.slice_w / 2 + 1;
    const int ntx = (wp + TX - 1) / TX, nty = (a.slice_h + TY * PPT - 1) / (TY * PPT);
    const dim3 grid(static_cast<unsigned>(ntx * nty), static_cast<unsigned>(a.n_slices < 65535 ? a.n_slices : 65535));
    if (a.out_cplx)
        extract_pairs_w_kernel<true><<<grid, EXTRACT_THREADS, 0, stream>>>(a, pairs, ntx);
    else
        extract_pairs_w_kernel<false><<<grid, EXTRACT_THREADS, 0, stream>>>(a, pairs, ntx);
    return cudaGetLastError();
}

cudaError_t launch_make_pairs(const ProjArgs& a, float4* pairs, cudaStream_t stream, const int* priority) {
    const int64_t vox = static_cast<int64_t>(a.vol_d) * a.vol_h * (a.vol_w / 2 + 1);
    const int threads = 256;
    const int64_t blocks = (vox + threads - 1) / threads;
    const int grid = static_cast<int>(blocks < static_cast<int64_t>(sm_count()) * 16 ? blocks : sm_count() * 16);
    if (grid <= 0)
        return cudaSuccess;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(static_cast<unsigned>(grid));
    cfg.blockDim = dim3(threads);
    cfg.stream = stream;
    cudaLaunchAttribute attr{};
    if (priority) {
        attr.id = cudaLaunchAttributePriority;
        attr.val.priority = *priority;
        cfg.attrs = &attr;
        cfg.numAttrs = 1;
    }
    if (vox < (int64_t(1) << 31))
        return cudaLaunchKernelEx(&cfg, make_pairs<uint32_t>, a, pairs);
    return cudaLaunchKernelEx(&cfg, make_pairs<int64_t>, a, pairs);
}

cudaError_t launch_extract_volume(const ProjArgs& a, cudaStream_t stream) { return launch_interp<I_LINEAR>(a, stream, 2); }

cudaError_t launch_extract(const ProjArgs& a, cudaStream_t stream) {
    if (a.n_slices > 0 && use_pairs(a, stream)) {
        bool done = false;
        const cudaError_t err = launch_pairs(a, stream, done);
        if (err != cudaSuccess || done)
            return err;
    }
    switch (a.interp) {
        case I_NEAREST: return launch_interp<I_NEAREST>(a, stream);
        case I_LINEAR: return launch_interp<I_LINEAR>(a, stream);
        case I_CUBIC: return launch_interp<I_CUBIC>(a, stream);
        case I_BSPLINE: return launch_interp<I_BSPLINE>(a, stream);
        case I_LANCZOS4: return launch_interp<I_LANCZOS4>(a, stream);
        case I_LANCZOS6: return launch_interp<I_LANCZOS6>(a, stream);
        case I_LANCZOS8: return launch_interp<I_LANCZOS8>(a, stream);
        default: return cudaErrorInvalidValue;
    }
}

} // namespace nb
