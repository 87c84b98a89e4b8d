// insert_and_extract_central_slices_3d on sm_100a: every output pixel samples the virtual volume made
// of the input slices (FourierInsertExtract, noa/xform/FourierProject.hpp:858-977).
//
// A CTA owns a 16x16 tile of one output slice, each warp a 4x8 sub-tile. The input slices are culled
// twice: slice i can only contribute to a pixel whose 3-D frequency g satisfies |n_i . g| < blackman,
// and without curvature g is linear in the pixel's 2-D frequency, so n_i . g over a box of pixels is an
// interval known from two dot products (patch_reaches). The slices whose interval over the CTA's box
// meets the slab are compacted, in increasing order, into shared memory, 4096 at a time, each warp
// compacting its own range of slice indices so that building the list needs no barrier.
//
// Each warp then takes the list 32 slices at a time, one per lane, with no barrier until the next pass. Where
// slabs are about as thick as a patch is wide, or few slices meet a patch, it culls them over its own box and
// walks the rest, every lane evaluating its own pixel of one slice (WALK). Where they are thinner, that leaves half
// of the lanes idle (17 of 32 active with the default window), and it goes by a queue: fz is
// linear along a row of pixels, so a slice's slab covers an interval of each of the warp's four rows
// (widened by the rounding of the exact test): together a 32-bit mask of pixels. The warp walks the slices
// whose mask is not empty, queues their (pixel, slice) pairs and evaluates queued pairs 64 at a time, two per
// lane, whichever pixels they belong to: exact distance, window and interpolation run with all lanes busy.
// Each lane keeps the queue slots of its own pixel's pairs as a bit mask and adds their results in slot order.
// (Masks transposed so that each lane walks its own pixel's slices without a queue were 10 % slower, the
// longest list of 32 setting the pace.)
//
// The slices through a pixel grow as 1 / |f|, so the tiles around the origin hold up to 20 times the pairs
// of the others, and the warp at the origin works for a good part of the launch: in launches of several tiles
// per SM, tiles are taken in the order of their distance to it, those of all output slices together, so that the
// long ones start first. 2000 input to 64 output slices of 256^2, default window and weights: 3180 us ->
// 1837 us with a queue filled by exact tests and evaluated 32 pairs at a time -> 1253 us.
//
// Summation order per pixel is therefore the reference's (increasing slice index). With an Ewald
// sphere (curved slices) nothing is culled. The w-windowed form sums the w offsets in registers (in w order)
// rather than zero-filling and adding atomically; each offset re-samples the virtual volume at the
// z-shifted frequency.
#include "fp_args.cuh"
#include "fp_slice_taps.cuh"

#include <type_traits>

namespace nb {
namespace {

constexpr int IE_THREADS = 256;
constexpr int IE_TILE = 16;  // 16x16 pixels per CTA; warps own 4x8 sub-tiles
constexpr int IE_LIST = 4096;                           // input slices culled per pass (16 KB of indices)
constexpr int IE_REGION = IE_LIST / (IE_THREADS / 32);  // of which each warp compacts one range

// A box of 2-D output frequencies: centre and half-extent per axis.
struct Box2 {
    float c0, h0, c1, h1;
    __device__ static Box2 of(float lo0, float hi0, float lo1, float hi1) {
        return {0.5f * (lo0 + hi0), 0.5f * (hi0 - lo0), 0.5f * (lo1 + hi1), 0.5f * (hi1 - lo1)};
    }
};

// The 3-D frequencies of an output slice's unit 2-D steps (z, y, x).
struct Patch {
    float gv0, gv1, gv2, gu0, gu1, gu2;
};

// Whether input slice i (n = row 0 of its inverse rotation, so that its fz = n . g) can reach
// |fz| < blackman at a frequency g of the box, shifted along z by `off`: over the box, n . g spans
// centre +- (|n . Gv| h0 + |n . Gu| h1). The margin covers the rounding of the exact per-pixel test.
__device__ __forceinline__ bool patch_reaches(const float3 n, const Patch& p, const Box2& box, float off, float fb) {
    const float al = n.x * p.gv0 + n.y * p.gv1 + n.z * p.gv2;
    const float be = n.x * p.gu0 + n.y * p.gu1 + n.z * p.gu2;
    const float centre = al * box.c0 + be * box.c1 + n.x * off;
    const float half = fabsf(al) * box.h0 + fabsf(be) * box.h1;
    return fabsf(centre) <= fb + half + 1e-5f * (1.f + fabsf(centre) + half);
}

// Columns lo to hi (0 <= lo <= 8, -1 <= hi <= 7) of a row of 8 pixels; none if hi < lo.
__host__ __device__ constexpr unsigned row_columns(int lo, int hi) { return hi < lo ? 0u : (2u << hi) - (1u << lo); }
static_assert(row_columns(0, 7) == 0xffu && row_columns(3, 5) == 0x38u && row_columns(7, 7) == 0x80u, "");
static_assert(row_columns(0, -1) == 0u && row_columns(8, 7) == 0u && row_columns(8, -1) == 0u, "no shift is out of range");

// The pixels of a warp's 4 x 8 patch (bit 8 row + column) that slice n may reach, fz being linear along a row.
// `rows`: the rows' 2-D frequencies; `first`, `step`: the first column's frequency and the columns' spacing.
__device__ __forceinline__ unsigned patch_mask(const float3 n, const Patch& p, const float (&rows)[4], float first,
                                               float step, float off, float fb) {
    const float al = n.x * p.gv0 + n.y * p.gv1 + n.z * p.gv2;
    const float be = n.x * p.gu0 + n.y * p.gu1 + n.z * p.gu2;
    const float shift = n.x * off;
    const float reach = fb + 1e-5f * (1.f + fabsf(al) + fabsf(be) + fabsf(shift));
    const float inv = 1.f / (be * step);  // infinite for a slice parallel to the rows: all or nothing below
    unsigned mask = 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float start = al * rows[r] + be * first + shift;
        const float a = (-reach - start) * inv, b = (reach - start) * inv;
        // Clamped before the conversions (NaN included: then the whole row, and the exact test decides).
        const int lo = __float2int_ru(fminf(fmaxf(fminf(a, b) - 1e-3f, 0.f), 8.f));
        const int hi = __float2int_rd(fmaxf(fminf(fmaxf(a, b) + 1e-3f, 7.f), -1.f));
        mask |= row_columns(lo, hi) << 8 * r;
    }
    return mask;
}

// One warp's queue of (pixel, slice) pairs: a ring of two halves, evaluated half by half.
constexpr int IE_HALF = 64;
struct PairQueue {
    unsigned entry[2 * IE_HALF];   // slice index within the pass << 5 | pixel's lane
    float2 value[IE_HALF];         // of the half evaluated last
    float weight[IE_HALF];
};

// How a warp evaluates the pairs of a slice (form_of chooses).
enum Form {
    WALK,   // every lane evaluates its own pixel, one slice at a time
    QUEUE,  // by the queue, one pair per lane at a time
    LEAN,   // by the queue, for Mat33 rotations without scaling: LINEAR two pairs per lane in packed operations
};

// Resident CTAs per SM asked of the compiler. WALK: 5 (48 registers; with 6 3 % slower for quaternions and scaling,
// equal for matrices), 2 for the wider windows. The queue's wider windows ask for none: they stay within the 128
// registers of two, and with two asked for (104 registers) are 1.5 % slower on average, up to 7 %.
template<int I, Form FORM>
constexpr int insert_extract_min_ctas() {
    return FORM == WALK ? (I != I_LINEAR && I != I_NEAREST ? 2 : 5) : (I != I_LINEAR && I != I_NEAREST ? 1 : 4);
}

template<int I, bool IN_C, bool OUT_C, Form FORM, typename Idx = int>
__global__ void __launch_bounds__(IE_THREADS, insert_extract_min_ctas<I, FORM>())
insert_extract_kernel(const __grid_constant__ ProjArgs a, int ntx, int nty, int64_t n_tiles, bool by_place) {
    __shared__ int s_list[IE_LIST];
    __shared__ int s_warp_count[IE_THREADS / 32];
    __shared__ float s_box[4][IE_THREADS / 32];
    __shared__ PairQueue s_queue[FORM == WALK ? 1 : IE_THREADS / 32];

    const int wp = a.slice_w / 2 + 1;
    const Spectrum2 sp{a.in_h, a.in_w_, a.in_centered, a.in_slice_narrow != 0};
    const bool has_out_w = a.out_w.present;
    const bool has_in_w = a.in_w.present;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    PairQueue& queue = s_queue[FORM == WALK ? 0 : warp];
    const WindowPair window_of(a);
    const bool mat33 = a.rot.kind == 2 && a.scale.kind == 0 && !a.ews.on;

    // Where the sample (z, y, x) lies relative to input slice i: its distance and in-slice frequencies.
    const auto locate = [&](int64_t i, float z, float y, float x, float& q0, float& q1) {
        float f0, f1, fz;
        if (FORM == LEAN || mat33) {
            // grid2slice's Mat33 rows (same products and sums)
            const float* m = xform_ptr(a.rot, i, 12);
            fz = dot3(m[0], m[1], m[2], z, y, x);
            if (FORM == WALK && !(fabsf(fz) < a.fb))
                return fz;  // the in-plane rows are only needed inside the slab
            f0 = dot3(m[3], m[4], m[5], z, y, x);
            f1 = dot3(m[6], m[7], m[8], z, y, x);
        } else {
            fz = grid2slice(z, y, x, a.scale, a.rot, i, a.ews, f0, f1);
        }
        q0 = mul(f0, a.f_in0);
        q1 = mul(f1, a.f_in1);
        return fz;
    };
    // The term of input slice i there, inside its slab.
    const auto term = [&](int64_t i, float fz, float q0, float q1, float2& value, float& weight) {
        weight = windowed_sinc_fast(fz, a.pfs, a.ifs, a.pfb);
        value = cmul(interp_spectrum_2d<I, IN_C>(a.in, sp, i, q0, q1), weight);
        if (has_in_w)
            weight = mul(interp_spectrum_2d<I, false>(a.in_w, sp, i, q0, q1).x, weight);
    };

    for (int64_t tile = blockIdx.x; tile < n_tiles; tile += gridDim.x) {
        // by_place: the tile's place by distance to the origin (column of tiles, then rows alternately below and
        // above the origin's), all output slices of one place together.
        int64_t b;
        int tx, ty;
        if (by_place) {
            const int place = static_cast<int>(tile / a.n_slices);
            b = tile - place * a.n_slices;
            tx = place / nty;
            const int k_row = place - tx * nty;
            ty = (a.out_centered ? a.slice_h / 2 / IE_TILE : 0) + (k_row & 1 ? nty - (k_row + 1) / 2 : k_row / 2);
            ty -= ty < nty ? 0 : nty;
        } else {
            b = tile / (ntx * nty);
            const int t = static_cast<int>(tile - b * (ntx * nty));
            ty = t / ntx;
            tx = t - ty * ntx;
        }
        const int py = ty * IE_TILE + (warp >> 1) * 4 + (lane >> 3);
        const int pu = tx * IE_TILE + (warp & 1) * 8 + (lane & 7);
        const bool valid = py < a.slice_h && pu < wp;
        const int y = valid ? py : 0;
        const int u = valid ? pu : 0;
        const int v = index2frequency(a.out_centered, y, a.slice_h);
        const float pf0 = div(static_cast<float>(v), a.f_slice0), pf1 = div(static_cast<float>(u), a.f_slice1);
        float gz, gy, gx;
        slice2grid(pf0, pf1, a.scale2, a.rot2, b, a.ews, gz, gy, gx);

        // Without curvature a pixel's frequency is linear in its 2-D frequency: g = pf0 Gv + pf1 Gu.
        // Over a box of 2-D frequencies, n . g therefore spans an interval whose centre and half-width
        // follow from n . Gv and n . Gu (patch_reaches); the boxes are the warp's and the CTA's.
        Patch patch;
        slice2grid(1.f, 0.f, a.scale2, a.rot2, b, a.ews, patch.gv0, patch.gv1, patch.gv2);
        slice2grid(0.f, 1.f, a.scale2, a.rot2, b, a.ews, patch.gu0, patch.gu1, patch.gu2);
        float bmin[2] = {valid ? pf0 : 3.4e38f, valid ? pf1 : 3.4e38f};
        float bmax[2] = {valid ? pf0 : -3.4e38f, valid ? pf1 : -3.4e38f};
#pragma unroll
        for (int ax = 0; ax < 2; ++ax) {
            for (int o = 16; o > 0; o >>= 1) {
                bmin[ax] = fminf(bmin[ax], __shfl_xor_sync(0xffffffffu, bmin[ax], o));
                bmax[ax] = fmaxf(bmax[ax], __shfl_xor_sync(0xffffffffu, bmax[ax], o));
            }
            if (lane == 0) {
                s_box[ax][warp] = bmin[ax];
                s_box[2 + ax][warp] = bmax[ax];
            }
        }
        const bool warp_valid = __any_sync(0xffffffffu, valid);
        const Box2 wbox = Box2::of(bmin[0], bmax[0], bmin[1], bmax[1]);  // every lane holds its warp's
        // The warp's rows and columns (the non-centered layout wraps between rows, not along them).
        float rows[4] = {}, step = 0.f, first = 0.f;
        if constexpr (FORM != WALK) {
#pragma unroll
            for (int r = 0; r < 4; ++r)
                rows[r] = __shfl_sync(0xffffffffu, pf0, 8 * r);
            step = 1.f / a.f_slice1;
            first = __shfl_sync(0xffffffffu, static_cast<float>(pu), 0) * step;
        }
        __syncthreads();
        float lo[2], hi[2];
#pragma unroll
        for (int ax = 0; ax < 2; ++ax) {
            lo[ax] = 3.4e38f;
            hi[ax] = -3.4e38f;
            for (int w = 0; w < IE_THREADS / 32; ++w) {
                lo[ax] = fminf(lo[ax], s_box[ax][w]);
                hi[ax] = fmaxf(hi[ax], s_box[2 + ax][w]);
            }
        }
        const Box2 cbox = Box2::of(lo[0], hi[0], lo[1], hi[1]);
        const bool cull = !a.ews.on;

        // Accumulators: one (value, weight) per w offset would be needed for the windowed form, so
        // the windowed form keeps a running windowed sum per offset instead (registers, bounded).
        const int nw = a.wsize > 1 ? a.wsize : 1;
        float2 acc = make_float2(0.f, 0.f);
        float accw = 0.f;

        // Each w offset is a separate virtual-volume sample; process them one after another so the
        // per-sample sums over input slices keep the reference's order.
        for (int w = 0; w < nw; ++w) {
            const float off = a.wsize > 1 ? div(static_cast<float>(w - a.wsize / 2), a.vz) : 0.f;
            const float sz = a.wsize > 1 ? add(gz, off) : gz;
            const bool in_cut = valid && dot3(sz, gy, gx, sz, gy, gx) <= a.cutoff_sqd;
            const unsigned cut_mask = __ballot_sync(0xffffffffu, in_cut);
            float2 value = make_float2(0.f, 0.f);
            float weight = 0.f;

            for (int64_t super = 0; super < a.n_in; super += IE_LIST) {
                int cnt = 0;
                for (int r = 0; r < IE_REGION; r += 32) {
                    const int64_t i = super + warp * IE_REGION + r + lane;
                    if (super + warp * IE_REGION + r >= a.n_in)
                        break;
                    const bool keep = i < a.n_in &&
                                      (!cull || patch_reaches(rotation_row0(a.rot, i), patch, cbox, off, a.fb));
                    const unsigned ballot = __ballot_sync(0xffffffffu, keep);
                    if (keep)
                        s_list[warp * IE_REGION + cnt + __popc(ballot & ((1u << lane) - 1u))] =
                            static_cast<int>(i - super);
                    cnt += __popc(ballot);
                }
                if (lane == 0)
                    s_warp_count[warp] = cnt;
                __syncthreads();

                int filled = 0;                           // queued pairs, counted from the pass' start
                unsigned long long mine0 = 0, mine1 = 0;  // this lane's pixel's slots of the ring's two halves
                // Evaluates `n` pairs of a half and adds each pixel's.
                auto evaluate = [&](int half, int n) {
                    __syncwarp();
                    // Pair lane + 32 e of the half; past n the first one, outside every slab.
                    const auto prepare = [&](int e, int64_t& i, float& q0, float& q1) {
                        const int at = lane + 32 * e;
                        const unsigned entry = queue.entry[half * IE_HALF + (at < n ? at : 0)];
                        const int owner = static_cast<int>(entry & 31u);
                        const float z = __shfl_sync(0xffffffffu, sz, owner);
                        const float y = __shfl_sync(0xffffffffu, gy, owner);
                        const float x = __shfl_sync(0xffffffffu, gx, owner);
                        i = super + (entry >> 5);
                        const float fz = locate(i, z, y, x, q0, q1);
                        return at < n ? fz : 3.4e38f;
                    };
                    const auto keep = [&](int e, float2 v, float w1) {
                        if (lane + 32 * e < n) {
                            queue.value[lane + 32 * e] = v;
                            queue.weight[lane + 32 * e] = w1;
                        }
                    };
                    if constexpr (InterpTraits<I>::SIZE <= 4) {
                        // Both pairs' matrices and coordinates in flight together.
                        int64_t si[2];
                        float q0[2], q1[2], fz[2];
#pragma unroll
                        for (int e = 0; e < 2; ++e)
                            fz[e] = prepare(e, si[e], q0[e], q1[e]);
                        float2 iv[2] = {};
                        float iw[2] = {};
                        if constexpr (FORM == LEAN && I == I_LINEAR) {
                            using T = typename std::conditional<IN_C, float2, float>::type;
                            const float2 window = window_of(pack2(fz[0], fz[1]));
#pragma unroll
                            for (int e = 0; e < 2; ++e) {
                                if (!(fabsf(fz[e]) < a.fb))
                                    continue;
                                iw[e] = e ? window.y : window.x;
                                const T* base = static_cast<const T*>(a.in.data) + si[e] * a.in.s0;
                                if constexpr (IN_C)
                                    iv[e] = cmul(slice_value(base, sp, static_cast<Idx>(a.in.s1), q0[e], q1[e]), iw[e]);
                                else
                                    iv[e].x = slice_value(base, sp, static_cast<Idx>(a.in.s1), q0[e], q1[e]) * iw[e];
                                if (has_in_w) {
                                    const LinearCell cell(sp, q0[e], q1[e]);
                                    iw[e] = mul(cell.read(static_cast<const float*>(a.in_w.data) + si[e] * a.in_w.s0,
                                                          static_cast<Idx>(a.in_w.s1), static_cast<Idx>(a.in_w.s2)).x, iw[e]);
                                }
                            }
                        } else {
#pragma unroll 1
                            for (int e = 0; 32 * e < n; ++e) {
                                const float f = e ? fz[1] : fz[0];
                                if (!(fabsf(f) < a.fb))
                                    continue;
                                float2 v;
                                float w1;
                                term(e ? si[1] : si[0], f, e ? q0[1] : q0[0], e ? q1[1] : q1[0], v, w1);
                                (e ? iv[1] : iv[0]) = v;
                                (e ? iw[1] : iw[0]) = w1;
                            }
                        }
                        keep(0, iv[0], iw[0]);
                        keep(1, iv[1], iw[1]);
                    } else {
                        // The windows of 6 and 8 taps have no registers for a second pair (LANCZOS8 10 % slower).
#pragma unroll 1
                        for (int e = 0; 32 * e < n; ++e) {
                            int64_t i;
                            float q0, q1, w1 = 0.f;
                            float2 v = make_float2(0.f, 0.f);
                            const float f = prepare(e, i, q0, q1);
                            if (fabsf(f) < a.fb)
                                term(i, f, q0, q1, v, w1);
                            keep(e, v, w1);
                        }
                    }
                    __syncwarp();
                    unsigned long long slots = half ? mine1 : mine0;
                    while (slots) {
                        const int j = __ffsll(static_cast<long long>(slots)) - 1;
                        slots &= slots - 1;
                        value = cadd(value, queue.value[j]);
                        weight = add(weight, queue.weight[j]);
                    }
                    if (half)
                        mine1 = 0;
                    else
                        mine0 = 0;
                };

                for (int region = 0; warp_valid && region < IE_THREADS / 32; ++region) {
                    const int count = s_warp_count[region];
                    const int* list = s_list + region * IE_REGION;
                    for (int g = 0; g < count; g += 32) {
                        const int k = g + lane;
                        const int listed = k < count ? list[k] : 0;
                        unsigned mask = k < count ? cut_mask : 0u;
                        if (mask && cull && FORM == WALK)
                            mask = patch_reaches(rotation_row0(a.rot, super + listed), patch, wbox, off, a.fb) ? mask : 0u;
                        else if (mask && cull)
                            mask &= patch_mask(rotation_row0(a.rot, super + listed), patch, rows, first, step,
                                               off, a.fb);
                        unsigned todo = __ballot_sync(0xffffffffu, mask != 0);
                        while (todo) {
                            const int j = __ffs(todo) - 1;
                            todo &= todo - 1u;
                            const int index = __shfl_sync(0xffffffffu, listed, j);
                            const unsigned pixels = FORM == WALK ? cut_mask : __shfl_sync(0xffffffffu, mask, j);
                            if constexpr (FORM == WALK) {
                                if (in_cut) {
                                    float q0, q1;
                                    const float fz = locate(super + index, sz, gy, gx, q0, q1);
                                    if (fabsf(fz) < a.fb) {
                                        float2 v;
                                        float iw;
                                        term(super + index, fz, q0, q1, v, iw);
                                        value = cadd(value, v);
                                        weight = add(weight, iw);
                                    }
                                }
                                continue;
                            }
                            if ((pixels >> lane) & 1u) {
                                const int slot = (filled + __popc(pixels & ((1u << lane) - 1u))) & (2 * IE_HALF - 1);
                                queue.entry[slot] = static_cast<unsigned>(index) << 5 | static_cast<unsigned>(lane);
                                if (slot < IE_HALF)
                                    mine0 |= 1ull << slot;
                                else
                                    mine1 |= 1ull << (slot - IE_HALF);
                            }
                            const int before = filled / IE_HALF;
                            filled += __popc(pixels);
                            if (filled / IE_HALF != before)  // at most 32 pairs were added: one half is full
                                evaluate(before & 1, IE_HALF);
                        }
                    }
                }
                if (FORM != WALK && filled % IE_HALF)
                    evaluate(filled / IE_HALF & 1, filled % IE_HALF);
                __syncthreads();
            }

            if (a.wsize <= 1) {
                if (in_cut && a.correct_weights) {
                    const float fw = fmaxf(1.f, fabsf(weight));
                    value.x = div(value.x, fw);
                    value.y = div(value.y, fw);
                }
                acc = value;
                accw = weight;
            } else if (in_cut) {
                const float cw = windowed_sinc(off, a.efs, a.efb);
                acc = cadd(acc, cmul(to_output<IN_C, OUT_C>(value), cw));
                accw = add(accw, mul(weight, cw));
            }
        }

        if (!valid)
            continue;
        if (a.wsize <= 1) {
            const bool in_cut = dot3(gz, gy, gx, gz, gy, gx) <= a.cutoff_sqd;
            if (!in_cut) {
                if (!a.add_to_output) {
                    dst_store<OUT_C>(a.out, b, y, u, make_float2(0.f, 0.f));
                    if (has_out_w)
                        store_real(a.out_w, b, y, u, 0.f);
                }
                continue;
            }
            const float2 o = to_output<IN_C, OUT_C>(acc);
            if (a.add_to_output)
                dst_store<OUT_C>(a.out, b, y, u, cadd(dst_load<OUT_C>(a.out, b, y, u), o));
            else
                dst_store<OUT_C>(a.out, b, y, u, o);
            if (has_out_w) {
                if (a.add_to_output)
                    store_real(a.out_w, b, y, u, add(load_real(a.out_w, b, y, u), accw));
                else
                    store_real(a.out_w, b, y, u, accw);
            }
        } else {
            // Windowed form: the reference zero-fills (unless add_to_output) then adds every offset.
            float2 o = acc;
            float ow = accw;
            if (a.add_to_output) {
                o = cadd(dst_load<OUT_C>(a.out, b, y, u), acc);
                if (has_out_w)
                    ow = add(load_real(a.out_w, b, y, u), accw);
            }
            dst_store<OUT_C>(a.out, b, y, u, o);
            if (has_out_w)
                store_real(a.out_w, b, y, u, ow);
        }
    }
}

// The queue gathers the pixels that a slab covers only in part; it costs about 16 instructions per pair, and a
// half that is not full runs with idle lanes. It therefore pays for thin slabs and for warps that meet many
// pairs. `reach` is the slab's half-width in output pixels: within half a patch the lanes of WALK are mostly idle, from
// 2 pixels on (1.5 for the windows of 6 and 8 taps, whose taps neighbouring lanes share in WALK) they are not. 700
// slices of 64^2 to 8 of 64^2, us by WALK and by QUEUE (LINEAR by quaternions), half-widths of 1, 2, 3 and 6 pixels: 652 and
// 406, 642 and 540, 640 and 640, 640 and 768; the LEAN form against WALK 645 and 354, 645 and 458, 640 and 525, 621 and 629.
// A launch of many tiles that meet few slices each fills no halves: 64 slices to 48 of 256^2 take 88 us by WALK,
// 90 by LEAN and 102 by QUEUE. With a curvature nothing is culled and most of the queue would be pairs outside the slabs.
template<int I>
Form form_of(const ProjArgs& a, int64_t n_tiles) {
    const bool mat33 = a.rot.kind == 2 && a.scale.kind == 0, packed = I == I_LINEAR && mat33 && linear_slices(a);
    const float reach = a.fb * a.f_slice1;
    const float limit = packed ? 5.f : InterpTraits<I>::SIZE <= 4 ? 2.f : 1.5f;
    const bool few = n_tiles > static_cast<int64_t>(sm_count()) * 8 ? a.n_in * 3 < a.slice_w : !packed && a.n_in < 8;
    if (a.ews.on || reach > limit * 1.001f || few)
        return WALK;
    return packed || (I == I_NEAREST && mat33) ? LEAN : QUEUE;
}

template<int I, bool IN_C, bool OUT_C>
cudaError_t launch_typed(const ProjArgs& a, cudaStream_t stream) {
    const int wp = a.slice_w / 2 + 1;
    const int ntx = (wp + IE_TILE - 1) / IE_TILE, nty = (a.slice_h + IE_TILE - 1) / IE_TILE;
    const int64_t n_tiles = static_cast<int64_t>(ntx) * nty * a.n_slices;
    if (n_tiles == 0)
        return cudaSuccess;
    const int64_t max_grid = static_cast<int64_t>(sm_count()) * 8 * 16;
    const int grid = static_cast<int>(n_tiles < max_grid ? n_tiles : max_grid);
    // Few tiles are resident together in any order; those of one place next to each other, on the SMs of one TPC,
    // are then slower. By slices and by places: 64 slices to 8 of 128^2 (320 tiles), half-width 6, LANCZOS8 935 and 1006
    // us, CUBIC 183 and 181; 700 to 48 of 64^2 (576 tiles) LANCZOS8 20.3 and 18.9 ms, CUBIC 3.10 and 2.58, LINEAR 0.70
    // and 0.64.
    const bool by_place = n_tiles > static_cast<int64_t>(sm_count()) * 3;
    switch (form_of<I>(a, n_tiles)) {
        case LEAN:
            if constexpr (I == I_LINEAR || I == I_NEAREST) {
                if (I == I_NEAREST || a.in_slice_narrow)
                    insert_extract_kernel<I, IN_C, OUT_C, LEAN, int><<<grid, IE_THREADS, 0, stream>>>(a, ntx, nty, n_tiles, by_place);
                else if constexpr (I == I_LINEAR)
                    insert_extract_kernel<I, IN_C, OUT_C, LEAN, int64_t><<<grid, IE_THREADS, 0, stream>>>(a, ntx, nty, n_tiles, by_place);
            }
            break;
        case QUEUE:
            insert_extract_kernel<I, IN_C, OUT_C, QUEUE><<<grid, IE_THREADS, 0, stream>>>(a, ntx, nty, n_tiles, by_place);
            break;
        case WALK:
            insert_extract_kernel<I, IN_C, OUT_C, WALK><<<grid, IE_THREADS, 0, stream>>>(a, ntx, nty, n_tiles, by_place);
            break;
    }
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

cudaError_t launch_insert_extract(const ProjArgs& a, cudaStream_t stream) {
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
