// fourier_interpolation_correction on sm_100a (noa/xform/FourierProject.hpp:2062-2087, operator
// GriddingCorrection :1009-1061): the real-space correction of the trilinear gridding kernel. Per
// voxel (b, j, k, l): dist = ((j, k, l) - half) / shape, half = shape / 2 (0 where a size is 1),
// r = |dist|, sinc2 = sinc(pi r)^2 (noa::sinc is 1 at 0, base/Math.hpp:28-29); the output is
// value / sinc2 (post-correction) or value * sinc2. One read and one write per voxel, coalesced along l;
// in place is allowed. The coordinates are rounded like the reference's f32 operator (no contraction), so
// the factors differ from it only through sinf.
//
// A block takes up to 256 columns of up to GRID_ROWS consecutive rows (b, j, k) per thread row. What belongs to
// a row (its offsets and the j and k terms of the distance) is computed once per row, by one thread, and
// shared; what belongs to a column (the l term) once per thread. What is left per voxel is the square
// root, the sine and two divisions. One linear index per voxel, taken apart by 64-bit divisions, with
// the three coordinate divisions made the kernel bound by instructions: 250^3, 159 us (77 % of the issue
// rate) -> about 60 us, against 19 us for its 125 MB.
#include "fp_args.cuh"

namespace nb {
namespace {

struct Grid4 {
    const float* in;
    float* out;
    int64_t is[4], os[4];     // strides in elements (input strides are 0 along broadcast dimensions)
    int64_t n[4];             // output shape
    float f[3], half[3];
    float value;              // constant input when in == nullptr
    int post;
};

constexpr int GRID_ROWS = 8;
constexpr int GRID_MAX_ROWS = GRID_ROWS * 8;  // of a block: at most 256 / 32 thread rows

// Block: blockDim.x columns by blockDim.y thread rows; thread row y takes rows y, y + blockDim.y, ...
__global__ void __launch_bounds__(256) gridding_correction_kernel(const __grid_constant__ Grid4 g, int rows_each) {
    constexpr float PI = 3.1415926535897932384626433832795f;
    __shared__ float s_sqd[GRID_MAX_ROWS];
    __shared__ int64_t s_from[GRID_MAX_ROWS], s_to[GRID_MAX_ROWS];
    const int64_t rows = g.n[0] * g.n[1] * g.n[2];
    const int per_block = static_cast<int>(blockDim.y) * rows_each;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    for (int64_t first = blockIdx.y * static_cast<int64_t>(per_block); first < rows;
         first += static_cast<int64_t>(gridDim.y) * per_block) {
        const int count = static_cast<int>(rows - first < per_block ? rows - first : per_block);
        __syncthreads();  // nobody still reads the previous rows
        if (tid < count) {
            const int64_t t = (first + tid) / g.n[2];
            const int64_t k = first + tid - t * g.n[2];
            const int64_t b = t / g.n[1];
            const int64_t j = t - b * g.n[1];
            const float d0 = div(sub(static_cast<float>(j), g.half[0]), g.f[0]);
            const float d1 = div(sub(static_cast<float>(k), g.half[1]), g.f[1]);
            s_sqd[tid] = add(mul(d0, d0), mul(d1, d1));
            s_from[tid] = b * g.is[0] + j * g.is[1] + k * g.is[2];
            s_to[tid] = b * g.os[0] + j * g.os[1] + k * g.os[2];
        }
        __syncthreads();
        for (int64_t l = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; l < g.n[3];
             l += static_cast<int64_t>(gridDim.x) * blockDim.x) {
            const float d2 = div(sub(static_cast<float>(l), g.half[2]), g.f[2]);
            const float d2_sqd = mul(d2, d2);
            const float* in = g.in + l * g.is[3];
            float* out = g.out + l * g.os[3];
#pragma unroll 4
            for (int r = threadIdx.y; r < count; r += blockDim.y) {
                const float v = g.in ? in[s_from[r]] : g.value;
                const float radius = __fsqrt_rn(add(s_sqd[r], d2_sqd));
                const float x = mul(PI, radius);
                const float sinc = x == 0.f ? 1.f : div(sinf(x), x);
                const float sinc2 = mul(sinc, sinc);
                out[s_to[r]] = g.post ? div(v, sinc2) : mul(v, sinc2);
            }
        }
    }
}

} // namespace

cudaError_t launch_gridding_correction(const nb_array* input, const nb_array* output, bool post,
                                       cudaStream_t stream) {
    Grid4 g{};
    g.in = input->is_value ? nullptr : static_cast<const float*>(input->data);
    g.out = static_cast<float*>(output->data);
    g.value = static_cast<float>(input->value[0]);
    for (int d = 0; d < 4; ++d) {
        g.n[d] = output->shape[d];
        g.os[d] = output->strides[d];
        g.is[d] = input->is_value || input->shape[d] == 1 ? 0 : input->strides[d];
    }
    for (int d = 0; d < 3; ++d) {
        g.f[d] = static_cast<float>(output->shape[d + 1]);
        g.half[d] = output->shape[d + 1] == 1 ? 0.f : g.f[d] / 2.f;
    }
    g.post = post ? 1 : 0;
    const int64_t total = g.n[0] * g.n[1] * g.n[2] * g.n[3];
    if (total == 0)
        return cudaSuccess;
    // A block covers up to 256 columns; narrower rows, and rows that would leave a quarter of the columns
    // idle, get narrower blocks of several groups of rows.
    int bx = 256;
    while (bx > 32 && ((g.n[3] + bx - 1) / bx * bx - g.n[3]) * 4 > g.n[3])
        bx /= 2;
    const dim3 block(static_cast<unsigned>(bx), static_cast<unsigned>(256 / bx));
    const int64_t cols = (g.n[3] + bx - 1) / bx;
    const int64_t rows = g.n[0] * g.n[1] * g.n[2];
    // Fewer rows per thread row where the launch would not give every SM its eight blocks: a block is a serial
    // chain of its rows (33^3: 2.6 us with one voxel per thread, 6.4 us with eight).
    int rows_each = GRID_ROWS;
    while (rows_each > 1 && (rows + block.y * rows_each - 1) / (block.y * rows_each) * cols < sm_count() * 8)
        rows_each /= 2;
    const int64_t groups = (rows + static_cast<int64_t>(block.y) * rows_each - 1) / (static_cast<int64_t>(block.y) * rows_each);
    const dim3 grid(static_cast<unsigned>(cols < 65535 ? cols : 65535), static_cast<unsigned>(groups < 65535 ? groups : 65535));
    gridding_correction_kernel<<<grid, block, 0, stream>>>(g, rows_each);
    return cudaGetLastError();
}

} // namespace nb
