// insert_central_slices_3d on sm_100a: deterministic gather-form windowed-sinc insertion
// (FourierInsertInterpolate, noa/xform/FourierProject.hpp:478-519).
//
// The reference visits every slice for every voxel, an O(voxels x slices) loop. Here a CTA owns a
// 4x8x8 brick of voxels and first culls the slices: slice i can only reach a voxel of the brick if
// the plane's normal n_i (row 0 of the inverse rotation) satisfies |n_i . c| <= blackman + |n_i| rho
// (+ a rounding margin), with c the brick's centre and rho its half-diagonal, all in fftfreq units.
// The surviving slice indices are compacted into shared memory IN INCREASING ORDER, and every thread
// then sums its voxel's contributions over that list. Skipped slices contribute exactly 0 in the
// reference (they fail |fz| <= blackman), so each voxel's sum sees the same terms in the same order.
// With an Ewald-sphere curvature the normal test is not conservative, and every slice is visited.
#include "fp_args.cuh"
#include "fp_slice_taps.cuh"

#include <type_traits>

namespace nb {
namespace {

constexpr int BZ = 4, BY = 8, BX = 8;
constexpr int INSERT_THREADS = BZ * BY * BX;

// CTAs per SM the LINEAR and NEAREST instantiations are compiled for (32 registers, small spills): the
// kernel is issue-bound and more resident warps hide its latencies: 512^3 x 20,000 slices, 328.9 ->
// 286.2-287.1 ms on one box (1000 slices: 16.13 -> 13.50-13.64 ms; six CTAs 13.80-13.86 ms). The
// wider windows keep the compiler's choice.
template<int I>
constexpr int insert_min_ctas() { return I == I_LINEAR || I == I_NEAREST ? 8 : 1; }

template<int I, bool IN_C, bool OUT_C>
__global__ void __launch_bounds__(INSERT_THREADS, insert_min_ctas<I>())
insert_kernel(const __grid_constant__ ProjArgs a, int nbz, int nby, int nbx) {
    __shared__ int s_list[INSERT_THREADS];
    __shared__ int s_warp_count[INSERT_THREADS / 32];
    __shared__ int s_count;
    // With a Mat33 rotation and neither scaling nor Ewald curvature, the kept slices' matrices are
    // staged here (in list order) so that the voxel loop reads them from shared memory, computes the
    // distance to the plane (row 0) first and the in-plane coordinates (rows 1 and 2) only inside the
    // window: the same products and sums as grid2slice, in the same order.
    __shared__ float s_mat[9][INSERT_THREADS];
    const bool lean = a.rot.kind == 2 && a.scale.kind == 0 && !a.ews.on;

    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const bool vc = a.out_centered;
    const Spectrum2 sp{a.slice_h, a.slice_w, a.in_centered, a.in_slice_narrow != 0};
    const bool has_out_w = a.out_w.present;
    const bool has_in_w = a.in_w.present;
    const int tid = threadIdx.x;
    const int tx = tid % BX, ty = (tid / BX) % BY, tz = tid / (BX * BY);
    const int lane = tid & 31, warp = tid >> 5;
    const int64_t n_bricks = static_cast<int64_t>(nbz) * nby * nbx;

    for (int64_t brick = blockIdx.x; brick < n_bricks; brick += gridDim.x) {
        const int bx = static_cast<int>(brick % nbx);
        const int by = static_cast<int>((brick / nbx) % nby);
        const int bz = static_cast<int>(brick / (static_cast<int64_t>(nbx) * nby));
        const int z0 = bz * BZ, y0 = by * BY, x0 = bx * BX;
        const int z = z0 + tz, y = y0 + ty, x = x0 + tx;
        const bool valid = z < D && y < H && x < WP;

        // This voxel's frequency (FourierProject.hpp:479-484).
        const float fz = div(static_cast<float>(index2frequency(vc, z, D)), a.target0);
        const float fy = div(static_cast<float>(index2frequency(vc, y, H)), a.target1);
        const float fx = div(static_cast<float>(x), a.target2);
        const bool active = valid && dot3(fz, fy, fx, fz, fy, fx) <= a.cutoff_sqd;
        if (!__syncthreads_or(active))
            continue;

        // Brick bounding box in fftfreq (per-axis min/max over the brick's valid indices; the
        // non-centered layout wraps, so scan rather than assume monotonic).
        float lo[3], hi[3];
        {
            const int n3[3] = {D, H, WP};
            const int s3[3] = {z0, y0, x0};
            const int e3[3] = {BZ, BY, BX};
            const float t3[3] = {a.target0, a.target1, a.target2};
            for (int ax = 0; ax < 3; ++ax) {
                float mn = 3.4e38f, mx = -3.4e38f;
                for (int k = 0; k < e3[ax]; ++k) {
                    const int idx = s3[ax] + k;
                    if (idx >= n3[ax])
                        break;
                    const int f = ax == 2 ? idx : index2frequency(vc, idx, n3[ax]);
                    const float ff = static_cast<float>(f) / t3[ax];
                    mn = fminf(mn, ff);
                    mx = fmaxf(mx, ff);
                }
                lo[ax] = mn;
                hi[ax] = mx;
            }
        }
        const float c0 = 0.5f * (lo[0] + hi[0]), c1 = 0.5f * (lo[1] + hi[1]), c2 = 0.5f * (lo[2] + hi[2]);
        const float h0 = 0.5f * (hi[0] - lo[0]), h1 = 0.5f * (hi[1] - lo[1]), h2 = 0.5f * (hi[2] - lo[2]);
        const float rho = sqrtf(h0 * h0 + h1 * h1 + h2 * h2);
        const float cn = sqrtf(c0 * c0 + c1 * c1 + c2 * c2);
        const float margin = 1e-5f * (cn + rho + 1.f);
        const bool cull = !a.ews.on;

        float2 value = make_float2(0.f, 0.f);
        float weights = 0.f;

        for (int64_t chunk = 0; chunk < a.n_slices; chunk += INSERT_THREADS) {
            const int64_t i = chunk + tid;
            bool keep = false;
            if (i < a.n_slices) {
                if (cull) {
                    const float3 n = rotation_row0(a.rot, i);
                    const float nn = sqrtf(n.x * n.x + n.y * n.y + n.z * n.z);
                    const float d = fabsf(n.x * c0 + n.y * c1 + n.z * c2);
                    keep = d <= a.fb + nn * rho + margin * (1.f + nn);
                } else {
                    keep = true;
                }
            }
            // Ordered compaction of the kept slice indices.
            const unsigned ballot = __ballot_sync(0xffffffffu, keep);
            if (lane == 0)
                s_warp_count[warp] = __popc(ballot);
            __syncthreads();
            int base = 0;
            for (int w = 0; w < warp; ++w)
                base += s_warp_count[w];
            if (keep) {
                const int slot = base + __popc(ballot & ((1u << lane) - 1u));
                s_list[slot] = static_cast<int>(i - chunk);
                if (lean) {
                    const float* m = xform_ptr(a.rot, i, 12);
#pragma unroll
                    for (int e = 0; e < 9; ++e)
                        s_mat[e][slot] = m[e];
                }
            }
            if (tid == INSERT_THREADS - 1)
                s_count = base + __popc(ballot);
            __syncthreads();
            const int count = s_count;

            if (active) {
                for (int k = 0; k < count; ++k) {
                    const int64_t si = chunk + s_list[k];
                    float f0, f1, zz;
                    if (lean) {
                        zz = dot3(s_mat[0][k], s_mat[1][k], s_mat[2][k], fz, fy, fx);
                        if (!(fabsf(zz) <= a.fb))
                            continue;
                        f0 = dot3(s_mat[3][k], s_mat[4][k], s_mat[5][k], fz, fy, fx);
                        f1 = dot3(s_mat[6][k], s_mat[7][k], s_mat[8][k], fz, fy, fx);
                    } else {
                        zz = grid2slice(fz, fy, fx, a.scale, a.rot, si, a.ews, f0, f1);
                    }
                    if (fabsf(zz) <= a.fb) {
                        const float window = windowed_sinc_fast(zz, a.pfs, a.ifs, a.pfb);
                        const float q0 = mul(f0, a.f_slice0), q1 = mul(f1, a.f_slice1);
                        value = cadd(value, cmul(interp_spectrum_2d<I, IN_C>(a.in, sp, si, q0, q1), window));
                        if (has_out_w) {
                            const float iw = has_in_w ?
                                mul(interp_spectrum_2d<I, false>(a.in_w, sp, si, q0, q1).x, window) : window;
                            weights = add(weights, iw);
                        }
                    }
                }
            }
            __syncthreads();
        }

        if (active) {
            const float2 o = to_output<IN_C, OUT_C>(value);
            dst_store<OUT_C>(a.out, z, y, x, cadd(dst_load<OUT_C>(a.out, z, y, x), o));
            if (has_out_w)
                store_real(a.out_w, z, y, x, add(load_real(a.out_w, z, y, x), weights));
        }
    }
}

// The LINEAR insertion of Mat33 rotations without scaling or curvature, from slices with adjacent columns:
// insert_kernel's sum, term for term in the same order, for few instructions per (voxel, slice)
// pair, which is what bounds it: 400 slices
// into 512^3 with half-width 6 and weights 6074 us -> 3083 us (insert_kernel issues at 87 % of its rate; 3803
// us with the window and the coordinates of one voxel at a time).
//
// A thread owns LIN_PZ voxels along z: the products of a slice's matrix with the voxels' y and x
// frequencies are shared by them, so a voxel costs one product and two sums per row of the matrix, and the
// sums and the window of two voxels run in packed operations. A
// slice's matrix and base pointer are staged as three 16-byte words, the test of the cull is the exact
// interval of n . f over the brick's box, and a chunk of the list holds twice as many slices as the CTA
// has threads (half the barriers).
constexpr int LIN_PZ = 4;                                    // voxels per thread, along z
constexpr int LIN_Z = 8, LIN_Y = 8, LIN_X = 8;               // brick
constexpr int LIN_THREADS = LIN_Z / LIN_PZ * LIN_Y * LIN_X;  // 128; a warp covers 4 x 4 x 8 voxels
constexpr int LIN_CHUNK = 2 * LIN_THREADS;                   // slices culled per pass
constexpr int LIN_WARPS = LIN_THREADS / 32;

template<bool IN_C, bool OUT_C, typename Idx>
__global__ void __launch_bounds__(LIN_THREADS, 8)
insert_linear_kernel(const __grid_constant__ ProjArgs a, int nbz, int nby, int nbx) {
    using T = typename std::conditional<IN_C, float2, float>::type;
    __shared__ float4 s_row[3][LIN_CHUNK];   // rows of the kept slices; .w: slice index, pointer low, high
    __shared__ int s_warp_count[2][LIN_WARPS];
    __shared__ float2 s_box[3];

    const int D = a.vol_d, H = a.vol_h, WP = a.vol_w / 2 + 1;
    const bool vc = a.out_centered;
    const Spectrum2 sp{a.slice_h, a.slice_w, a.in_centered, true};
    const bool has_out_w = a.out_w.present;
    const bool has_in_w = has_out_w && a.in_w.present;
    const Idx s1 = static_cast<Idx>(a.in.s1);
    const WindowPair window_of(a);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int tx = tid % LIN_X, ty = (tid / LIN_X) % LIN_Y, tz = tid / (LIN_X * LIN_Y) * LIN_PZ;
    const int64_t n_bricks = static_cast<int64_t>(nbz) * nby * nbx;

    for (int64_t brick = blockIdx.x; brick < n_bricks; brick += gridDim.x) {
        const int bx = static_cast<int>(brick % nbx);
        const int by = static_cast<int>((brick / nbx) % nby);
        const int bz = static_cast<int>(brick / (static_cast<int64_t>(nbx) * nby));
        const int z0 = bz * LIN_Z + tz, y = by * LIN_Y + ty, x = bx * LIN_X + tx;

        // The voxels' frequencies (FourierProject.hpp:479-484).
        const float fy = div(static_cast<float>(index2frequency(vc, y, H)), a.target1);
        const float fx = div(static_cast<float>(x), a.target2);
        float fz[LIN_PZ];
        unsigned active = 0;
#pragma unroll
        for (int k = 0; k < LIN_PZ; ++k) {
            fz[k] = div(static_cast<float>(index2frequency(vc, z0 + k, D)), a.target0);
            if (z0 + k < D && y < H && x < WP && dot3(fz[k], fy, fx, fz[k], fy, fx) <= a.cutoff_sqd)
                active |= 1u << k;
        }
        if (!__syncthreads_or(active))
            continue;

        // The brick's box, centre and half extent per axis; the non-centered layout wraps, so its extents
        // are the smallest and largest of the indices', 8 lanes per axis.
        if (warp == 0) {
            const int axis = lane >> 3, first = axis == 0 ? bz * LIN_Z : axis == 1 ? by * LIN_Y : bx * LIN_X;
            const int n = axis == 0 ? D : axis == 1 ? H : WP, i = min(first + (lane & 7), n - 1);
            const float f = static_cast<float>(axis < 2 ? index2frequency(vc, i, n) : i) /
                            (axis == 0 ? a.target0 : axis == 1 ? a.target1 : a.target2);
            float mn = f, mx = f;
#pragma unroll
            for (int o = 4; o > 0; o /= 2) {
                mn = fminf(mn, __shfl_xor_sync(0xffffffffu, mn, o));
                mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            }
            if ((lane & 7) == 0 && axis < 3)
                s_box[axis] = make_float2(0.5f * (mn + mx), 0.5f * (mx - mn));
        }
        __syncthreads();
        const float2 box0 = s_box[0], box1 = s_box[1], box2 = s_box[2];

        float2 value[LIN_PZ] = {};
        float weights[LIN_PZ] = {};

        for (int64_t chunk = 0; chunk < a.n_slices; chunk += LIN_CHUNK) {
            // Ordered compaction of the slices whose slab meets the box: |n . f| over it spans
            // |n . c| +- sum |n_k| h_k, the margin covers the rounding of the exact test.
            unsigned ballot[2];
            bool keep[2];
            const float* m[2];
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int64_t i = chunk + h * LIN_THREADS + tid;
                keep[h] = false;
                m[h] = xform_ptr(a.rot, i, 12);
                if (i < a.n_slices) {
                    const float n0 = m[h][0], n1 = m[h][1], n2 = m[h][2];
                    const float c = fabsf(n0 * box0.x + n1 * box1.x + n2 * box2.x);
                    const float r = fabsf(n0) * box0.y + fabsf(n1) * box1.y + fabsf(n2) * box2.y;
                    const float size = fabsf(n0) * fabsf(box0.x) + fabsf(n1) * fabsf(box1.x) + fabsf(n2) * fabsf(box2.x);
                    keep[h] = c <= a.fb + r + 1e-5f * (1.f + size + r);
                }
                ballot[h] = __ballot_sync(0xffffffffu, keep[h]);
                if (lane == 0)
                    s_warp_count[h][warp] = __popc(ballot[h]);
            }
            __syncthreads();
            int count = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
#pragma unroll
                for (int w = 0; w < LIN_WARPS; ++w) {
                    if (w == warp && keep[h]) {
                        const int slot = count + __popc(ballot[h] & ((1u << lane) - 1u));
                        const int i = static_cast<int>(chunk) + h * LIN_THREADS + tid;
                        const T* base = static_cast<const T*>(a.in.data) + i * a.in.s0;
                        const uint64_t p = reinterpret_cast<uint64_t>(base);
                        s_row[0][slot] = make_float4(m[h][0], m[h][1], m[h][2], __int_as_float(i));
                        s_row[1][slot] = make_float4(m[h][3], m[h][4], m[h][5], __uint_as_float(static_cast<uint32_t>(p)));
                        s_row[2][slot] = make_float4(m[h][6], m[h][7], m[h][8], __uint_as_float(static_cast<uint32_t>(p >> 32)));
                    }
                    count += s_warp_count[h][w];
                }
            }
            __syncthreads();

            if (active) {
                for (int s = 0; s < count; ++s) {
                    const float4 r0 = s_row[0][s];
                    const float y0 = mul(r0.y, fy), x0 = mul(r0.z, fx);
                    unsigned long long zz[LIN_PZ / 2];
                    unsigned near = 0;  // voxels within the window
#pragma unroll
                    for (int h = 0; h < LIN_PZ / 2; ++h) {
                        zz[h] = add2(add2(pack2(mul(r0.x, fz[2 * h]), mul(r0.x, fz[2 * h + 1])), pack2(y0, y0)), pack2(x0, x0));
                        const float2 z = unpack2(zz[h]);
                        near |= (fabsf(z.x) <= a.fb ? 1u << 2 * h : 0u) | (fabsf(z.y) <= a.fb ? 2u << 2 * h : 0u);
                    }
                    near &= active;
                    if (!near)
                        continue;
                    const float4 r1 = s_row[1][s], r2 = s_row[2][s];
                    const float y1 = mul(r1.y, fy), x1 = mul(r1.z, fx), y2 = mul(r2.y, fy), x2 = mul(r2.z, fx);
                    const T* base = reinterpret_cast<const T*>(static_cast<uint64_t>(__float_as_uint(r1.w)) |
                                                               static_cast<uint64_t>(__float_as_uint(r2.w)) << 32);
#pragma unroll
                    for (int h = 0; h < LIN_PZ / 2; ++h) {
                        if (!(near & (3u << 2 * h)))
                            continue;
                        const float2 window = window_of(zz[h]);
                        const float za = fz[2 * h], zb = fz[2 * h + 1];
                        const float2 q0 = unpack2(mul2(add2(add2(pack2(mul(r1.x, za), mul(r1.x, zb)), pack2(y1, y1)), pack2(x1, x1)),
                                                       pack2(a.f_slice0, a.f_slice0)));
                        const float2 q1 = unpack2(mul2(add2(add2(pack2(mul(r2.x, za), mul(r2.x, zb)), pack2(y2, y2)), pack2(x2, x2)),
                                                       pack2(a.f_slice1, a.f_slice1)));
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int k = 2 * h + e;
                            if (!((near >> k) & 1u))
                                continue;
                            const float w = e ? window.y : window.x;
                            const T v = slice_value(base, sp, s1, e ? q0.y : q0.x, e ? q1.y : q1.x);
                            if constexpr (IN_C)
                                value[k] = cfma(v, w, value[k]);
                            else
                                value[k].x = fmaf(v, w, value[k].x);
                            if (has_in_w) {
                                const float* base_w = static_cast<const float*>(a.in_w.data) + __float_as_int(r0.w) * a.in_w.s0;
                                const LinearCell cell(sp, e ? q0.y : q0.x, e ? q1.y : q1.x);
                                weights[k] = fmaf(cell.read(base_w, static_cast<Idx>(a.in_w.s1), static_cast<Idx>(a.in_w.s2)).x, w, weights[k]);
                            } else {
                                weights[k] += w;
                            }
                        }
                    }
                }
            }
            __syncthreads();
        }

#pragma unroll
        for (int k = 0; k < LIN_PZ; ++k) {
            if (!((active >> k) & 1u))
                continue;
            const int z = z0 + k;
            const float2 o = to_output<IN_C, OUT_C>(value[k]);
            dst_store<OUT_C>(a.out, z, y, x, cadd(dst_load<OUT_C>(a.out, z, y, x), o));
            if (has_out_w)
                store_real(a.out_w, z, y, x, add(load_real(a.out_w, z, y, x), weights[k]));
        }
    }
}

template<bool IN_C, bool OUT_C>
cudaError_t launch_linear(const ProjArgs& a, cudaStream_t stream) {
    const int WP = a.vol_w / 2 + 1;
    const int nbz = (a.vol_d + LIN_Z - 1) / LIN_Z, nby = (a.vol_h + LIN_Y - 1) / LIN_Y, nbx = (WP + LIN_X - 1) / LIN_X;
    const int64_t n = static_cast<int64_t>(nbz) * nby * nbx;
    if (n == 0)
        return cudaSuccess;
    const int64_t max_grid = int64_t(1) << 30;
    const unsigned grid = static_cast<unsigned>(n < max_grid ? n : max_grid);
    if (a.in_slice_narrow)
        insert_linear_kernel<IN_C, OUT_C, int><<<grid, LIN_THREADS, 0, stream>>>(a, nbz, nby, nbx);
    else
        insert_linear_kernel<IN_C, OUT_C, int64_t><<<grid, LIN_THREADS, 0, stream>>>(a, nbz, nby, nbx);
    return cudaGetLastError();
}

// Whether insert_linear_kernel applies, and pays: with a quarter of the threads it needs many bricks to fill the
// chip, and the slices through the brick at the origin, one after another, take it longer (1.15 us each against
// 0.67 us), so a launch has to hold 320 bricks for one slice, more for more slices, up to 12,000, from where on the
// other bricks' work outlasts that one. us of the general kernel and of this one, half-width 1 (6), with weights:
// one slice into 48^3 7.1 and 8.4, 80^3 11.6 and 8.7; 8 into 96^3 18 and 17 (21 and 18); 50 into 128^3 60 and 69 (74 and
// 76), 160^3 78 and 77 (106 and 88); 400 into 64^3 273 and 450, 176^3 441 and 538 (605 and 625), 224^3 613 and 635 (961
// and 770), 256^3 889 and 698 (1421 and 877).
bool use_linear(const ProjArgs& a) {
    const double bricks = static_cast<double>((a.vol_d + LIN_Z - 1) / LIN_Z) * ((a.vol_h + LIN_Y - 1) / LIN_Y) *
                          ((a.vol_w / 2 + LIN_X) / LIN_X);
    const double slices = static_cast<double>(a.n_slices);
    if (bricks < 12000. && bricks * bricks * bricks < 320. * 320. * 320. * slices * slices)
        return false;
    return linear_slices(a) && a.rot.kind == 2 && a.scale.kind == 0 && !a.ews.on && a.n_slices < (int64_t(1) << 31);
}

template<int I, bool IN_C, bool OUT_C>
cudaError_t launch_typed(const ProjArgs& a, cudaStream_t stream) {
    const int WP = a.vol_w / 2 + 1;
    const int nbz = (a.vol_d + BZ - 1) / BZ, nby = (a.vol_h + BY - 1) / BY, nbx = (WP + BX - 1) / BX;
    const int64_t n = static_cast<int64_t>(nbz) * nby * nbx;
    if (n == 0)
        return cudaSuccess;
    const int64_t max_grid = static_cast<int64_t>(sm_count()) * 8 * 16;
    const int grid = static_cast<int>(n < max_grid ? n : max_grid);
    insert_kernel<I, IN_C, OUT_C><<<grid, INSERT_THREADS, 0, stream>>>(a, nbz, nby, nbx);
    return cudaGetLastError();
}

template<int I>
cudaError_t launch_interp(const ProjArgs& a, cudaStream_t stream) {
    if (a.in_cplx && a.out_cplx)
        return launch_typed<I, true, true>(a, stream);
    if (a.in_cplx)
        return launch_typed<I, true, false>(a, stream);
    return launch_typed<I, false, false>(a, stream);
}

} // namespace

cudaError_t launch_insert(const ProjArgs& a, cudaStream_t stream) {
    if (use_linear(a)) {
        if (a.in_cplx && a.out_cplx)
            return launch_linear<true, true>(a, stream);
        if (a.in_cplx)
            return launch_linear<true, false>(a, stream);
        return launch_linear<false, false>(a, stream);
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
