// The step between insertion and the inverse FFT of a reconstruction, in one pass over the spectrum:
// value / max(weight, threshold), the remap from the inserted layout (centered "hc" or not "h") to the
// non-centered layout a c2r FFT reads, and the phase exp(-2 pi i k.c / n) with c = n / 2 per axis that
// puts the real-space origin at the volume's center (for even sizes, the factor (-1)^(kz+ky+kx)). After
// the c2r, fourier_interpolation_correction (fp_gridding.cu) finishes the reconstruction in real space.
// No function of the reference does this step; it replaces the elementwise ops, remap and fftshift a
// noa user would chain (fft/Remap.hpp).
#include "fp_args.cuh"

namespace nb {
namespace {

struct SpecArgs {
    const float2* values;
    const float* weights;      // may be null: no division
    float2* out;
    int64_t vs[3], ws[3];      // strides (d, h, w) of the inputs, in elements
    int d, h, wp, n_w;         // logical sizes; wp = n_w / 2 + 1
    bool centered;             // inputs are centered (hc)
    float threshold;
    float cz, cy, cx;          // phase centers (n / 2), as fractions of the sizes: c / n
};

// A block takes up to 256 columns of up to SPEC_ROWS consecutive rows (z, y) per thread row; a row's offsets and
// the z and y part of its phase are computed once, by one thread, and shared. One linear index per voxel,
// taken apart by 64-bit divisions, cost more than the arithmetic: 250^3, 65 us ->
// 45 us, against 24 us for its 156 MB.
constexpr int SPEC_ROWS = 4;
constexpr int SPEC_MAX_ROWS = SPEC_ROWS * 8;  // of a block: at most 256 / 32 thread rows

// Block: blockDim.x columns by blockDim.y thread rows; thread row y takes rows y, y + blockDim.y, ...
__global__ void __launch_bounds__(256) spectrum_kernel(const __grid_constant__ SpecArgs a, int rows_each) {
    __shared__ float s_turns[SPEC_MAX_ROWS];
    __shared__ int64_t s_value[SPEC_MAX_ROWS], s_weight[SPEC_MAX_ROWS];
    const int64_t rows = static_cast<int64_t>(a.d) * a.h;
    const int per_block = static_cast<int>(blockDim.y) * rows_each;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    const int x = blockIdx.x * blockDim.x + threadIdx.x;
    for (int64_t first = blockIdx.y * static_cast<int64_t>(per_block); first < rows;
         first += static_cast<int64_t>(gridDim.y) * per_block) {
        const int count = static_cast<int>(rows - first < per_block ? rows - first : per_block);
        __syncthreads();  // nobody still reads the previous rows
        if (tid < count) {
            const int z = static_cast<int>((first + tid) / a.h);
            const int y = static_cast<int>(first + tid - static_cast<int64_t>(z) * a.h);
            // Output row (z, y) is non-centered: its frequencies, then where they sit in the input.
            const int fz = index2frequency(false, z, a.d), fy = index2frequency(false, y, a.h);
            const int iz = frequency2index(a.centered, fz, a.d), iy = frequency2index(a.centered, fy, a.h);
            s_turns[tid] = fz * a.cz + fy * a.cy;
            s_value[tid] = iz * a.vs[0] + iy * a.vs[1];
            s_weight[tid] = iz * a.ws[0] + iy * a.ws[1];
        }
        __syncthreads();
        if (x >= a.wp)
            continue;
        const float2* values = a.values + x * a.vs[2];
        const float* weights = a.weights + x * a.ws[2];
        float2* out = a.out + first * a.wp + x;
#pragma unroll 4
        for (int r = threadIdx.y; r < count; r += blockDim.y) {
            float2 v = __ldcs(values + s_value[r]);
            if (a.weights) {
                const float w = fmaxf(__ldcs(weights + s_weight[r]), a.threshold);
                v = make_float2(v.x / w, v.y / w);
            }
            // exp(-2 pi i (fz cz + fy cy + fx cx)), the turns reduced to [-0.5, 0.5) before sincospi.
            float turns = s_turns[r] + x * a.cx;
            turns -= rintf(turns);
            float s, c;
            sincospif(-2.f * turns, &s, &c);
            __stcs(out + static_cast<int64_t>(r) * a.wp, make_float2(v.x * c - v.y * s, v.x * s + v.y * c));
        }
    }
}

} // namespace

cudaError_t launch_reconstruction_spectrum(const nb_array* values, const nb_array* weights,
                                           const int64_t shape[4], bool centered, float threshold,
                                           const nb_array* out, cudaStream_t stream) {
    SpecArgs a{};
    a.values = static_cast<const float2*>(values->data);
    a.weights = weights && weights->data ? static_cast<const float*>(weights->data) : nullptr;
    a.out = static_cast<float2*>(out->data);
    for (int k = 0; k < 3; ++k) {
        a.vs[k] = values->strides[k + 1];
        a.ws[k] = a.weights ? weights->strides[k + 1] : 0;
    }
    a.d = static_cast<int>(shape[1]);
    a.h = static_cast<int>(shape[2]);
    a.n_w = static_cast<int>(shape[3]);
    a.wp = a.n_w / 2 + 1;
    a.centered = centered;
    a.threshold = threshold;
    a.cz = static_cast<float>(a.d / 2) / static_cast<float>(a.d);
    a.cy = static_cast<float>(a.h / 2) / static_cast<float>(a.h);
    a.cx = static_cast<float>(a.n_w / 2) / static_cast<float>(a.n_w);
    const int64_t total = static_cast<int64_t>(a.d) * a.h * a.wp;
    if (total > 0) {
        // A block covers up to 256 columns; narrower rows, and rows that would leave a quarter of the
        // columns idle, get narrower blocks of several groups of rows.
        int bx = 256;
        while (bx > 32 && ((a.wp + bx - 1) / bx * bx - a.wp) * 4 > a.wp)
            bx /= 2;
        const dim3 block(static_cast<unsigned>(bx), static_cast<unsigned>(256 / bx));
        const int64_t rows = static_cast<int64_t>(a.d) * a.h;
        // Fewer rows per thread row where the launch would not give every SM its eight blocks.
        const int64_t cols = (a.wp + bx - 1) / bx;
        int rows_each = SPEC_ROWS;
        while (rows_each > 1 && (rows + block.y * rows_each - 1) / (block.y * rows_each) * cols < sm_count() * 8)
            rows_each /= 2;
        const int64_t groups = (rows + static_cast<int64_t>(block.y) * rows_each - 1) / (static_cast<int64_t>(block.y) * rows_each);
        const dim3 grid(static_cast<unsigned>(cols), static_cast<unsigned>(groups < 65535 ? groups : 65535));
        spectrum_kernel<<<grid, block, 0, stream>>>(a, rows_each);
    }
    return cudaGetLastError();
}

} // namespace nb
