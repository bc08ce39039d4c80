// f32 glue operators of quantized graphs (the float islands between int8 contractions: softmax, LayerNorm,
// GELU, residual adds, dynamic activation scales) with the arithmetic of nGraph's reference kernels:
//
//   elementwise +, -, *, /, max, min, abs, neg, sqrt, relu   IEEE single, one rounding each, nothing contracted
//   exp, erf                                                   reference: std::exp / std::erf on float; here the double
//                                                              routine rounded to float (differs from a given libm in
//                                                              the last bit on a small share of inputs)
//   Sum          runtime/reference/sum.hpp:56-90     Kahan-compensated, inputs taken in row-major order
//   Max          runtime/reference/max.hpp:32-58     start at -inf, replace when x > max
//   Broadcast    runtime/reference/broadcast.hpp     output coordinate with the broadcast axes dropped
//   BatchMatMul  runtime/reference/batch_mat_mul.hpp -> dot.hpp:108-160: the sum over k runs in DOUBLE, in order,
//                over exact products, and is rounded to float once
//   Gather       runtime/reference/gather.hpp        rows of a matrix picked by an index vector
//   Reshape      runtime/reference/reshape.hpp       axis permutation followed by a free re-interpretation
//
// All are HBM-bound (or, for the reductions and the matrix product, latency-bound on purpose: they keep the
// reference's summation order so that results are identical, not merely close).
#include <cuda_runtime.h>
#include <math.h>
#include <algorithm>
#include <initializer_list>
#include "common.cuh"

namespace b200
{
    constexpr int MAX_RANK = 8;
    struct Dims
    {
        int rank;
        int64_t out_dim[MAX_RANK];    // shape of the tensor the thread index runs over
        int64_t in_stride[MAX_RANK];  // element stride in the other tensor for each of those axes (0: axis absent)
    };

    __device__ __forceinline__ int64_t mapped_offset(const Dims& d, int64_t idx)
    {
        int64_t off = 0;
#pragma unroll 1
        for (int a = d.rank - 1; a >= 0; --a)
        {
            const int64_t c = idx % d.out_dim[a];
            idx /= d.out_dim[a];
            off += c * d.in_stride[a];
        }
        return off;
    }

    template <int OP>
    __device__ __forceinline__ float binary_op(float a, float b)
    {
        switch (OP)
        {
        case B200_F32_ADD: return __fadd_rn(a, b);
        case B200_F32_SUB: return __fsub_rn(a, b);
        case B200_F32_MUL: return __fmul_rn(a, b);
        case B200_F32_DIV: return __fdiv_rn(a, b);
        case B200_F32_MAX: return a > b ? a : b; // reference::maximum
        default: return a < b ? a : b;           // reference::minimum
        }
    }

    template <int OP>
    __global__ void __launch_bounds__(256) binary_kernel(const float* __restrict__ a, const float* __restrict__ b,
                                                         float* __restrict__ out, int64_t n)
    {
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
            out[i] = binary_op<OP>(a[i], b[i]);
    }

    // One operand is a small tensor that op::v0::Broadcast would repeat along new leading axes (a bias row, a scalar
    // factor): element i of the large operand meets v[i % period] instead of a materialised copy.  V_LEFT: v is the
    // left-hand operand.  Four neighbours at a time when `period` allows it.
    template <int OP, bool V_LEFT, bool VEC>
    __global__ void __launch_bounds__(256) binary_periodic_kernel(const float* __restrict__ a, const float* __restrict__ v,
                                                                  float* __restrict__ out, int64_t n, int64_t period)
    {
        if (VEC)
        {
            const int64_t n4 = n >> 2, p4 = period >> 2; // period == 1: p4 == 0
            const float4* a4 = reinterpret_cast<const float4*>(a);
            const float s = p4 == 0 ? __ldg(v) : 0.0f;
            for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n4; i += int64_t(gridDim.x) * blockDim.x)
            {
                const float4 x = a4[i];
                const float4 y = p4 == 0 ? make_float4(s, s, s, s) : __ldg(reinterpret_cast<const float4*>(v) + i % p4);
                float4 r;
                r.x = V_LEFT ? binary_op<OP>(y.x, x.x) : binary_op<OP>(x.x, y.x);
                r.y = V_LEFT ? binary_op<OP>(y.y, x.y) : binary_op<OP>(x.y, y.y);
                r.z = V_LEFT ? binary_op<OP>(y.z, x.z) : binary_op<OP>(x.z, y.z);
                r.w = V_LEFT ? binary_op<OP>(y.w, x.w) : binary_op<OP>(x.w, y.w);
                reinterpret_cast<float4*>(out)[i] = r;
            }
        }
        else
            for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
            {
                const float x = a[i], y = __ldg(v + i % period);
                out[i] = V_LEFT ? binary_op<OP>(y, x) : binary_op<OP>(x, y);
            }
    }

    template <int OP>
    void launch_binary_periodic(const float* a, const float* v, float* out, int64_t n, int64_t period, bool v_left, cudaStream_t st)
    {
        const bool vec = n % 4 == 0 && (period == 1 || period % 4 == 0) &&
                         ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(out) | (period == 1 ? 0 : reinterpret_cast<uintptr_t>(v))) & 15) == 0;
        const int64_t work = vec ? n / 4 : n, blocks = (work + 255) / 256, cap = b200::sm_count() * 16;
        const unsigned g = unsigned(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
        if (vec && v_left) binary_periodic_kernel<OP, true, true><<<g, 256, 0, st>>>(a, v, out, n, period);
        else if (vec) binary_periodic_kernel<OP, false, true><<<g, 256, 0, st>>>(a, v, out, n, period);
        else if (v_left) binary_periodic_kernel<OP, true, false><<<g, 256, 0, st>>>(a, v, out, n, period);
        else binary_periodic_kernel<OP, false, false><<<g, 256, 0, st>>>(a, v, out, n, period);
    }

    template <int OP>
    __device__ __forceinline__ float unary_op(float x)
    {
        switch (OP)
        {
        case B200_F32_ABS: return fabsf(x);
        case B200_F32_NEG: return -x;
        case B200_F32_SQRT: return __fsqrt_rn(x);
        case B200_F32_EXP: return static_cast<float>(exp(static_cast<double>(x)));
        case B200_F32_ERF: return static_cast<float>(erf(static_cast<double>(x)));
        default: return x > 0.0f ? x : 0.0f; // reference::relu
        }
    }

    template <int OP>
    __global__ void __launch_bounds__(256) unary_kernel(const float* __restrict__ x, float* __restrict__ out, int64_t n)
    {
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
            out[i] = unary_op<OP>(x[i]);
    }

    // out[idx] = in[mapped(idx)] for 4-byte elements: Broadcast (stride 0 on the new axes) and axis permutations.
    // T: one element (uint32_t) or four neighbours along a last axis that both tensors share (uint4); IDX: 32-bit index
    // arithmetic when every index and offset fits (a 64-bit division costs several times a 32-bit one).
    template <typename T, typename IDX>
    __global__ void __launch_bounds__(256) remap_kernel(const T* __restrict__ in, T* __restrict__ out, Dims d, int64_t n)
    {
        IDX dim[MAX_RANK], stride[MAX_RANK];
#pragma unroll
        for (int a = 0; a < MAX_RANK; ++a)
        {
            dim[a] = a < d.rank ? IDX(d.out_dim[a]) : IDX(1);
            stride[a] = a < d.rank ? IDX(d.in_stride[a]) : IDX(0);
        }
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        {
            IDX idx = IDX(i), off = 0;
#pragma unroll
            for (int a = MAX_RANK - 1; a >= 0; --a)
                if (a < d.rank)
                {
                    const IDX q = idx / dim[a];
                    off += (idx - q * dim[a]) * stride[a];
                    idx = q;
                }
            out[i] = in[off];
        }
    }

    // Picks the widest form the tensors allow.  `d` describes the output axes and the input stride of each.
    static void launch_remap(const void* in, void* out, Dims d, int64_t n, int64_t in_elements, cudaStream_t st)
    {
        const int last = d.rank - 1;
        bool wide = d.rank >= 1 && d.in_stride[last] == 1 && d.out_dim[last] % 4 == 0 &&
                    ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(out)) & 15) == 0;
        for (int a = 0; wide && a < last; ++a)
            wide = d.in_stride[a] % 4 == 0;
        if (wide)
        {
            d.out_dim[last] /= 4;
            for (int a = 0; a < last; ++a)
                d.in_stride[a] /= 4;
            n /= 4;
            in_elements /= 4;
        }
        const bool small = n < (int64_t(1) << 31) && in_elements < (int64_t(1) << 31);
        const int64_t blocks = (n + 255) / 256, cap = b200::sm_count() * 16;
        const unsigned grid = unsigned(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
        if (wide && small)
            remap_kernel<uint4, uint32_t><<<grid, 256, 0, st>>>(static_cast<const uint4*>(in), static_cast<uint4*>(out), d, n);
        else if (wide)
            remap_kernel<uint4, int64_t><<<grid, 256, 0, st>>>(static_cast<const uint4*>(in), static_cast<uint4*>(out), d, n);
        else if (small)
            remap_kernel<uint32_t, uint32_t><<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out), d, n);
        else
            remap_kernel<uint32_t, int64_t><<<grid, 256, 0, st>>>(static_cast<const uint32_t*>(in), static_cast<uint32_t*>(out), d, n);
    }

    // One thread per output element; the reduced coordinates are walked in row-major order, as the reference does.
    // keep: the kept axes (thread index -> input offset); red: the reduced axes.
    // One step of the reference's compensated sum (runtime/reference/sum.hpp:56-90).
    __device__ __forceinline__ void kahan_step(float& z, float& c, float x)
    {
        if (isfinite(x) && isfinite(z))
        {
            const float y = __fsub_rn(x, c);
            const float t = __fadd_rn(z, y);
            c = __fsub_rn(__fsub_rn(t, z), y);
            z = t;
        }
        else
            z = __fadd_rn(z, x);
    }

    // Max, Min and Max over Abs.  The result does not depend on the order the inputs are taken in (a NaN never wins the strict
    // comparison, in any order), so these equal the sequential reference loops (max.hpp:32-58, min.hpp).
    template <int OP>
    __device__ __forceinline__ float extreme_of(float m, float x)
    {
        if (OP == B200_REDUCE_MAX_ABS)
            x = fabsf(x);
        return (OP == B200_REDUCE_MIN ? x < m : x > m) ? x : m;
    }
    template <int OP>
    __device__ __forceinline__ float extreme_start()
    {
        return OP == B200_REDUCE_MIN ? INFINITY : -INFINITY;
    }
    template <int OP> // b200_reduce_op
    __global__ void __launch_bounds__(128) reduce_kernel(const float* __restrict__ in, float* __restrict__ out, Dims keep, Dims red,
                                                         int64_t n_out, int64_t n_red)
    {
        for (int64_t o = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; o < n_out; o += int64_t(gridDim.x) * blockDim.x)
        {
            const float* base = in + mapped_offset(keep, o);
            if (OP == B200_REDUCE_SUM)
            {
                float z = 0.0f, c = 0.0f;
                for (int64_t r = 0; r < n_red; ++r)
                    kahan_step(z, c, base[mapped_offset(red, r)]);
                out[o] = z;
            }
            else
            {
                float m = extreme_start<OP>();
                for (int64_t r = 0; r < n_red; ++r)
                    m = extreme_of<OP>(m, base[mapped_offset(red, r)]);
                out[o] = m;
            }
        }
    }

    // of all threads of the block, in thread 0 (partial results meet without the absolute value: -inf is "nothing yet")
    template <int ELEMENT_OP>
    __device__ __forceinline__ float extreme_of_block(float m, float* partial)
    {
        constexpr int OP = ELEMENT_OP == B200_REDUCE_MAX_ABS ? int(B200_REDUCE_MAX) : ELEMENT_OP;
#pragma unroll
        for (int d = 16; d > 0; d >>= 1)
            m = extreme_of<OP>(m, __shfl_xor_sync(0xffffffffu, m, d));
        if ((threadIdx.x & 31) == 0)
            partial[threadIdx.x >> 5] = m;
        __syncthreads();
        if (threadIdx.x == 0)
            for (int w = 1; w < int(blockDim.x >> 5); ++w)
                m = extreme_of<OP>(m, partial[w]);
        return m;
    }
    // of a contiguous run, thread `t` of `threads`: 16-byte loads, four in flight
    template <int OP>
    __device__ __forceinline__ float extreme_of_run(const float* __restrict__ in, int64_t n, int64_t t, int64_t threads)
    {
        float m = extreme_start<OP>();
        const int64_t head = min(n, int64_t((16 - (reinterpret_cast<uintptr_t>(in) & 15)) & 15) / 4), n4 = (n - head) / 4;
        const float4* in4 = reinterpret_cast<const float4*>(in + head);
        for (int64_t i = t; i < n4; i += 4 * threads)
        {
            float4 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                v[j] = in4[min(i + j * threads, n4 - 1)]; // past the end: the last vector again
#pragma unroll
            for (int j = 0; j < 4; ++j)
                m = extreme_of<OP>(extreme_of<OP>(extreme_of<OP>(extreme_of<OP>(m, v[j].x), v[j].y), v[j].z), v[j].w);
        }
        if (t < head)
            m = extreme_of<OP>(m, in[t]);
        if (t < n - head - 4 * n4)
            m = extreme_of<OP>(m, in[head + 4 * n4 + t]);
        return m;
    }

    // few outputs, long reductions: one block per output
    template <int OP>
    __global__ void __launch_bounds__(256) reduce_extreme_block_kernel(const float* __restrict__ in, float* __restrict__ out, Dims keep,
                                                                       Dims red, int64_t n_red)
    {
        __shared__ float partial[8];
        const float* base = in + mapped_offset(keep, blockIdx.x);
        float m = extreme_start<OP>();
        for (int64_t r = threadIdx.x; r < n_red; r += blockDim.x)
            m = extreme_of<OP>(m, base[mapped_offset(red, r)]);
        m = extreme_of_block<OP>(m, partial);
        if (threadIdx.x == 0)
            out[blockIdx.x] = m;
    }

    // The whole of a tensor of up to a million elements (the dynamic activation scale of a layer): one cluster of eight
    // blocks, whose partial results meet in the first block's shared memory: one launch, no scratch, no atomics.
    // [128, 768]: 2.2 us, where the two launches of the form below took 4; fewer than 65536 elements used to run in one thread.
    constexpr int EXTREME_CLUSTER = 8;
    template <int OP>
    __global__ void __cluster_dims__(EXTREME_CLUSTER, 1, 1) __launch_bounds__(1024)
        reduce_extreme_cluster_kernel(const float* __restrict__ in, float* __restrict__ out, int64_t n)
    {
        __shared__ float partial[32];
        __shared__ float of_block[EXTREME_CLUSTER];
        asm volatile("barrier.cluster.arrive.relaxed.aligned;" ::: "memory"); // this block runs: its shared memory may be written
        const float m = extreme_of_block<OP>(extreme_of_run<OP>(in, n, int64_t(blockIdx.x) * 1024 + threadIdx.x, EXTREME_CLUSTER * 1024), partial);
        asm volatile("barrier.cluster.wait.aligned;" ::: "memory");
        if (threadIdx.x == 0)
        {
            uint32_t dst;
            asm volatile("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(dst) : "r"(uint32_t(__cvta_generic_to_shared(&of_block[blockIdx.x]))));
            asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(dst), "f"(m) : "memory");
        }
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        if (blockIdx.x == 0 && threadIdx.x == 0)
        {
            float r = of_block[0];
#pragma unroll
            for (int b = 1; b < EXTREME_CLUSTER; ++b)
                r = extreme_of<OP == B200_REDUCE_MAX_ABS ? int(B200_REDUCE_MAX) : OP>(r, of_block[b]);
            out[0] = r;
        }
    }

    // Larger tensors: many blocks, each over a slice, combined with an atomic on the ordered integer image of the float
    // (non-negative floats order like signed ints, negative ones like reversed unsigned ints); the output must hold the
    // starting value on entry.  Bound by HBM.
    template <int OP>
    __global__ void __launch_bounds__(256) reduce_extreme_all_kernel(const float* __restrict__ in, float* __restrict__ out, int64_t n)
    {
        __shared__ float partial[8];
        const float m = extreme_of_block<OP>(extreme_of_run<OP>(in, n, int64_t(blockIdx.x) * 256 + threadIdx.x, int64_t(gridDim.x) * 256), partial);
        if (threadIdx.x == 0)
        {
            int* const as_int = reinterpret_cast<int*>(out);
            unsigned int* const as_uint = reinterpret_cast<unsigned int*>(out);
            if (__float_as_int(m) < 0) // -0.0 included: below +0.0 in the image, equal as a value
                OP == B200_REDUCE_MIN ? atomicMax(as_uint, __float_as_uint(m)) : atomicMin(as_uint, __float_as_uint(m));
            else
                OP == B200_REDUCE_MIN ? atomicMin(as_int, __float_as_int(m)) : atomicMax(as_int, __float_as_int(m));
        }
    }

    __global__ void fill_f32_kernel(float* out, float value, int64_t n)
    {
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
            out[i] = value;
    }

    // Softmax and LayerNorm over the LAST axis of a [rows, L] matrix.  Their compensated sums have to walk a row in
    // order, so a row belongs to one thread; reading it straight from memory would make the 32 lanes of a warp touch 32
    // different rows per load.  A block therefore stages 32 rows in shared memory, lets all its threads do the
    // order-free parts (max, exp, normalise, divide) and one warp the 32 ordered sums, one row per lane.
    // VEC: L is a multiple of 4 and the pointers are 16-byte aligned, so rows move as float4 with eight loads in flight
    // per thread (row stride L + 4: the ordered walks then meet 4-way bank conflicts, hidden behind the dependent
    // additions); otherwise element by element with an odd row stride.
    constexpr int ROWS_PER_TILE = 32;
    __host__ __device__ inline int staged_row_stride(int L, bool vec) { return vec ? L + 4 : (L | 1); }

    // The elementwise op that produced the rows can be applied while they are staged (one rounding, the same value the
    // op's own kernel would have written): factor != nullptr multiplies by the scalar *factor (op::v1::Multiply by a
    // broadcast scalar), addend != nullptr adds the rows of a second tensor (op::v1::Add).
    template <bool VEC>
    __device__ __forceinline__ void stage_rows(const float* __restrict__ src, float* tile, int n_rows, int L, int stride,
                                               const float* __restrict__ factor, const float* __restrict__ addend)
    {
        const float f = factor ? __ldg(factor) : 1.0f;
        if (VEC)
        {
            const int L4 = L >> 2, total = n_rows * L4;
            const float4* src4 = reinterpret_cast<const float4*>(src);
            const float4* add4 = reinterpret_cast<const float4*>(addend);
            for (int i0 = threadIdx.x; i0 < total; i0 += blockDim.x * 8)
            {
                float4 v[8], w[8];
#pragma unroll
                for (int j = 0; j < 8; ++j)
                {
                    const int i = i0 + j * blockDim.x;
                    if (i < total)
                    {
                        v[j] = __ldg(src4 + i);
                        if (addend)
                            w[j] = __ldg(add4 + i);
                    }
                }
#pragma unroll
                for (int j = 0; j < 8; ++j)
                {
                    const int i = i0 + j * blockDim.x;
                    if (i < total)
                    {
                        float4 r = v[j];
                        if (factor)
                            r = make_float4(__fmul_rn(r.x, f), __fmul_rn(r.y, f), __fmul_rn(r.z, f), __fmul_rn(r.w, f));
                        if (addend)
                            r = make_float4(__fadd_rn(r.x, w[j].x), __fadd_rn(r.y, w[j].y), __fadd_rn(r.z, w[j].z), __fadd_rn(r.w, w[j].w));
                        *reinterpret_cast<float4*>(tile + (i / L4) * stride + 4 * (i % L4)) = r;
                    }
                }
            }
        }
        else
            for (int i = threadIdx.x; i < n_rows * L; i += blockDim.x)
            {
                float r = src[i];
                if (factor)
                    r = __fmul_rn(r, f);
                if (addend)
                    r = __fadd_rn(r, addend[i]);
                tile[(i / L) * stride + i % L] = r;
            }
    }

    template <bool VEC>
    __global__ void __launch_bounds__(128) softmax_rows_kernel(const float* __restrict__ in, const float* __restrict__ factor, float* __restrict__ out,
                                                               int64_t rows, int L)
    {
        extern __shared__ __align__(16) float tile[];
        __shared__ float row_max[ROWS_PER_TILE], row_sum[ROWS_PER_TILE];
        const int stride = staged_row_stride(L, VEC);
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int64_t n_tiles = (rows + ROWS_PER_TILE - 1) / ROWS_PER_TILE;
        for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x)
        {
            const int64_t row0 = t * ROWS_PER_TILE;
            const int n_rows = int(rows - row0 < ROWS_PER_TILE ? rows - row0 : ROWS_PER_TILE);
            stage_rows<VEC>(in + row0 * L, tile, n_rows, L, stride, factor, nullptr);
            __syncthreads();
            // softmax.hpp: max over the axis (the largest value whatever the order), then exp(x - max)
            for (int r = warp; r < n_rows; r += 4)
            {
                float m = -INFINITY;
                for (int c = lane; c < L; c += 32)
                {
                    const float x = tile[r * stride + c];
                    m = x > m ? x : m;
                }
                for (int d = 16; d; d >>= 1)
                {
                    const float o = __shfl_xor_sync(0xFFFFFFFFu, m, d);
                    m = o > m ? o : m;
                }
                // the same warp owns the row in the next step too, so no block-wide barrier is needed in between
                for (int c = lane; c < L; c += 32)
                {
                    float& v = tile[r * stride + c];
                    v = static_cast<float>(exp(static_cast<double>(__fsub_rn(v, m))));
                }
            }
            __syncthreads();
            if (warp == 0 && lane < n_rows)
            {
                const float* row = tile + lane * stride;
                float z = 0.0f, c = 0.0f;
                for (int k = 0; k < L; ++k)
                    kahan_step(z, c, row[k]);
                row_sum[lane] = z;
            }
            __syncthreads();
            float* dst = out + row0 * L;
            if (VEC)
            {
                const int L4 = L >> 2, total = n_rows * L4;
                for (int i = threadIdx.x; i < total; i += blockDim.x)
                {
                    const int r = i / L4;
                    float4 v = *reinterpret_cast<const float4*>(tile + r * stride + 4 * (i % L4));
                    const float sum = row_sum[r];
                    v.x = __fdiv_rn(v.x, sum), v.y = __fdiv_rn(v.y, sum), v.z = __fdiv_rn(v.z, sum), v.w = __fdiv_rn(v.w, sum);
                    reinterpret_cast<float4*>(dst)[i] = v;
                }
            }
            else
                for (int i = threadIdx.x; i < n_rows * L; i += blockDim.x)
                {
                    const int r = i / L;
                    dst[i] = __fdiv_rn(tile[r * stride + i % L], row_sum[r]);
                }
            __syncthreads();
        }
    }

    // op::v0::LayerNorm over the last axis with scale and bias, as ONE kernel with the rounding steps of its
    // decomposition (src/ngraph/op/layer_norm.cpp:68-150 with builder::mean / builder::variance,
    // src/ngraph/builder/reduce_ops.cpp:68-127), in that order:
    //   mean = KahanSum(x) / N;  var = KahanSum((x - mean) * (x - mean)) / N;  sd = sqrt(var + eps);
    //   y = ((x - mean) / sd) * gamma + beta          (every operation a separate IEEE rounding, no fused multiply-add)
    template <bool VEC>
    __global__ void __launch_bounds__(128) layer_norm_rows_kernel(const float* __restrict__ in, const float* __restrict__ addend,
                                                                  const float* __restrict__ gamma, const float* __restrict__ beta,
                                                                  float* __restrict__ out, int64_t rows, int L, float count, float eps)
    {
        extern __shared__ __align__(16) float tile[];
        __shared__ float row_mean[ROWS_PER_TILE], row_sd[ROWS_PER_TILE];
        const int stride = staged_row_stride(L, VEC);
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int64_t n_tiles = (rows + ROWS_PER_TILE - 1) / ROWS_PER_TILE;
        for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x)
        {
            const int64_t row0 = t * ROWS_PER_TILE;
            const int n_rows = int(rows - row0 < ROWS_PER_TILE ? rows - row0 : ROWS_PER_TILE);
            stage_rows<VEC>(in + row0 * L, tile, n_rows, L, stride, nullptr, addend ? addend + row0 * L : nullptr);
            __syncthreads();
            if (warp == 0 && lane < n_rows)
            {
                const float* row = tile + lane * stride;
                float z = 0.0f, c = 0.0f;
                for (int k = 0; k < L; ++k)
                    kahan_step(z, c, row[k]);
                const float mean = __fdiv_rn(z, count);
                z = 0.0f, c = 0.0f;
                for (int k = 0; k < L; ++k)
                {
                    const float d = __fsub_rn(row[k], mean);
                    kahan_step(z, c, __fmul_rn(d, d));
                }
                row_mean[lane] = mean;
                row_sd[lane] = __fsqrt_rn(__fadd_rn(__fdiv_rn(z, count), eps));
            }
            __syncthreads();
            float* dst = out + row0 * L;
            if (VEC)
            {
                const int L4 = L >> 2, total = n_rows * L4;
                for (int i = threadIdx.x; i < total; i += blockDim.x)
                {
                    const int r = i / L4, k4 = i % L4;
                    float4 v = *reinterpret_cast<const float4*>(tile + r * stride + 4 * k4);
                    const float4 g = __ldg(reinterpret_cast<const float4*>(gamma) + k4), b = __ldg(reinterpret_cast<const float4*>(beta) + k4);
                    const float mean = row_mean[r], sd = row_sd[r];
                    v.x = __fadd_rn(__fmul_rn(__fdiv_rn(__fsub_rn(v.x, mean), sd), g.x), b.x);
                    v.y = __fadd_rn(__fmul_rn(__fdiv_rn(__fsub_rn(v.y, mean), sd), g.y), b.y);
                    v.z = __fadd_rn(__fmul_rn(__fdiv_rn(__fsub_rn(v.z, mean), sd), g.z), b.z);
                    v.w = __fadd_rn(__fmul_rn(__fdiv_rn(__fsub_rn(v.w, mean), sd), g.w), b.w);
                    reinterpret_cast<float4*>(dst)[i] = v;
                }
            }
            else
                for (int i = threadIdx.x; i < n_rows * L; i += blockDim.x)
                {
                    const int r = i / L, k = i % L;
                    const float norm = __fdiv_rn(__fsub_rn(tile[r * stride + k], row_mean[r]), row_sd[r]);
                    dst[i] = __fadd_rn(__fmul_rn(norm, __ldg(gamma + k)), __ldg(beta + k));
                }
            __syncthreads();
        }
    }

    // op::v0::Gelu with the rounding steps of its decomposition (src/ngraph/op/gelu.cpp:46-60):
    //   (0.5 * x) * (1 + erf(x / float(sqrt(2.0))))
    __global__ void __launch_bounds__(256) gelu_kernel(const float* __restrict__ x, float* __restrict__ out, int64_t n)
    {
        const float sqrt_two = static_cast<float>(1.4142135623730951);
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < n; i += int64_t(gridDim.x) * blockDim.x)
        {
            const float v = x[i];
            const float e = static_cast<float>(erf(static_cast<double>(__fdiv_rn(v, sqrt_two))));
            out[i] = __fmul_rn(__fmul_rn(0.5f, v), __fadd_rn(1.0f, e));
        }
    }

    // Sum over the last axis for rows of any length: a warp owns 32 rows, one per lane, and walks them 64 columns at a
    // time; each 32 x 64 panel is fetched with coalesced loads into shared memory (row stride 65: the lanes' walks hit
    // 32 different banks) and then added in column order with the reference's compensated step.  Many one-warp blocks per
    // SM overlap one block's loads with another's additions.
    __global__ void __launch_bounds__(32) sum_rows_kernel(const float* __restrict__ in, float* __restrict__ out, int64_t rows, int64_t L)
    {
        constexpr int CH = 64;
        __shared__ float panel[32][CH + 1];
        const int lane = threadIdx.x;
        for (int64_t row0 = int64_t(blockIdx.x) * 32; row0 < rows; row0 += int64_t(gridDim.x) * 32)
        {
            const int n_rows = int(rows - row0 < 32 ? rows - row0 : 32);
            float z = 0.0f, c = 0.0f;
            for (int64_t col0 = 0; col0 < L; col0 += CH)
            {
                const int n_col = int(L - col0 < CH ? L - col0 : CH);
                // lane l fetches columns l and l + 32 of every row: 16 rows at a time, 32 loads in flight
#pragma unroll
                for (int r0 = 0; r0 < 32; r0 += 16)
                {
                    float v[16][2];
#pragma unroll
                    for (int r = 0; r < 16; ++r)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            v[r][h] = (r0 + r < n_rows && lane + 32 * h < n_col) ? in[(row0 + r0 + r) * L + col0 + lane + 32 * h] : 0.0f;
#pragma unroll
                    for (int r = 0; r < 16; ++r)
#pragma unroll
                        for (int h = 0; h < 2; ++h)
                            panel[r0 + r][lane + 32 * h] = v[r][h];
                }
                __syncwarp();
                if (lane < n_rows)
                    for (int cc = 0; cc < n_col; ++cc)
                        kahan_step(z, c, panel[lane][cc]);
                __syncwarp();
            }
            if (lane < n_rows)
                out[row0 + lane] = z;
        }
    }

    // Grid and shared memory of the two staged kernels: as many 32-row tiles per SM as fit.
    template <typename Kernel>
    bool staged_launch_shape(Kernel kernel, int64_t rows, int L, bool vec, unsigned& grid, size_t& bytes)
    {
        bytes = size_t(ROWS_PER_TILE) * staged_row_stride(L, vec) * sizeof(float);
        if (bytes > 48 * 1024 && // the attribute belongs to the current device's copy of the kernel: set it on each use
            cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024) != cudaSuccess)
            return false;
        const int64_t tiles = (rows + ROWS_PER_TILE - 1) / ROWS_PER_TILE;
        const int64_t per_sm = (200 * 1024) / int64_t(bytes) < 8 ? (200 * 1024) / int64_t(bytes) : 8;
        grid = unsigned(tiles < b200::sm_count() * per_sm ? tiles : b200::sm_count() * per_sm);
        return true;
    }

    inline bool all_aligned16(std::initializer_list<const void*> ptrs)
    {
        uintptr_t bits = 0;
        for (const void* p : ptrs)
            bits |= reinterpret_cast<uintptr_t>(p);
        return (bits & 15) == 0;
    }

    // out[b, m, n] = float(sum_k double(a[b, m, k]) * double(b[b, k, n])), k ascending, on the double-precision matrix
    // instruction (m8n8k4: each output receives its four exact products in ascending k, one rounding each, like the
    // reference's loop; B200 has no tcgen05 form of it).  A warp owns MT x NT tiles of 8 x 8 outputs, a block WM x WN warps.
    //
    // Bound by the double-precision pipe, 64 multiply-adds per clock and SM.  A matrix instruction issues 256 of them, so
    // the issue slots that scalar multiply-adds needed are free for the operands: panels of f32 in shared memory (filled by
    // cp.async while the previous panel is multiplied), converted to double as a warp picks up its fragments.  Scalar
    // multiply-adds on panels of doubles, 8 x 4 per thread, kept the pipe 49 % busy; measured before / after at
    // 768 x [384, 64] x [64, 384]: 756 -> 478 us, 768 x [384, 384] x [384, 64]: 725 -> 458 us (81-85 % of that pipe).
    constexpr int BMM_KC = 32;
    __device__ __forceinline__ void cp_async_4(uint32_t dst, const void* src, bool ok)
    {
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst), "l"(src), "r"(ok ? 4 : 0) : "memory");
    }
    __device__ __forceinline__ void cp_async_16(uint32_t dst, const void* src, bool ok)
    {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
    }
    __device__ __forceinline__ void dmma(double (&c)[2], double a, double b)
    {
        asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};" : "+d"(c[0]), "+d"(c[1]) : "d"(a), "d"(b));
    }

    template <int WM, int WN, int MT, int NT, bool VEC>
    __global__ void __launch_bounds__(WM* WN * 32) bmm_f32_kernel(const float* __restrict__ a, const float* __restrict__ bm, float* __restrict__ out,
                                                                  int M, int K, int N, uint32_t tiles_m, uint32_t tiles_n)
    {
        constexpr int TM = WM * MT * 8, TN = WN * NT * 8, KC = BMM_KC, THREADS = WM * WN * 32;
        constexpr int LDA = KC + 4, LDB = TN + 8; // fragment loads then touch 32 different banks
        extern __shared__ __align__(16) float panels[]; // two of { A [TM][LDA], B [KC][LDB] }
        const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, g = lane >> 2, t = lane & 3;
        const uint32_t tn = blockIdx.x % tiles_n, rest = blockIdx.x / tiles_n;
        const int m0 = int(rest % tiles_m) * TM, n0 = int(tn) * TN;
        const int64_t batch = rest / tiles_m;
        const float* ab = a + batch * int64_t(M) * K;
        const float* bb = bm + batch * int64_t(K) * N;
        const uint32_t base = uint32_t(__cvta_generic_to_shared(panels));
        auto fetch = [&](int k0, int buf) {
            // what lies beyond M, N or K is filled with zeros: fma(0, 0, acc) = acc
            const uint32_t as = base + uint32_t(buf) * (TM * LDA + KC * LDB) * 4, bs = as + TM * LDA * 4;
            if (VEC)
            {
                for (int i = tid; i < TM * KC / 4; i += THREADS)
                {
                    const int m = i / (KC / 4), k = (i % (KC / 4)) * 4;
                    const bool ok = m0 + m < M && k0 + k < K;
                    cp_async_16(as + (m * LDA + k) * 4, ok ? ab + int64_t(m0 + m) * K + k0 + k : ab, ok);
                }
                for (int i = tid; i < KC * TN / 4; i += THREADS)
                {
                    const int k = i / (TN / 4), n = (i % (TN / 4)) * 4;
                    const bool ok = k0 + k < K && n0 + n < N;
                    cp_async_16(bs + (k * LDB + n) * 4, ok ? bb + int64_t(k0 + k) * N + n0 + n : bb, ok);
                }
            }
            else
            {
                for (int i = tid; i < TM * KC; i += THREADS)
                {
                    const int m = i / KC, k = i % KC;
                    const bool ok = m0 + m < M && k0 + k < K;
                    cp_async_4(as + (m * LDA + k) * 4, ok ? ab + int64_t(m0 + m) * K + k0 + k : ab, ok);
                }
                for (int i = tid; i < KC * TN; i += THREADS)
                {
                    const int k = i / TN, n = i % TN;
                    const bool ok = k0 + k < K && n0 + n < N;
                    cp_async_4(bs + (k * LDB + n) * 4, ok ? bb + int64_t(k0 + k) * N + n0 + n : bb, ok);
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        double acc[MT][NT][2];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
                acc[i][j][0] = acc[i][j][1] = 0.0;
        const int wm = (warp / WN) * MT * 8, wn = (warp % WN) * NT * 8;
        if (K > 0)
            fetch(0, 0);
        for (int k0 = 0, buf = 0; k0 < K; k0 += KC, buf ^= 1)
        {
            if (k0 + KC < K)
            {
                fetch(k0 + KC, buf ^ 1);
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            }
            else
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            __syncthreads();
            const float* as = panels + buf * (TM * LDA + KC * LDB) + (wm + g) * LDA + t;
            const float* bs = panels + buf * (TM * LDA + KC * LDB) + TM * LDA + t * LDB + wn + g;
#pragma unroll
            for (int k = 0; k < KC; k += 4)
            {
                double x[MT], y[NT];
#pragma unroll
                for (int i = 0; i < MT; ++i)
                    x[i] = double(as[i * 8 * LDA + k]);
#pragma unroll
                for (int j = 0; j < NT; ++j)
                    y[j] = double(bs[k * LDB + 8 * j]);
#pragma unroll
                for (int i = 0; i < MT; ++i)
#pragma unroll
                    for (int j = 0; j < NT; ++j)
                        dmma(acc[i][j], x[i], y[j]);
            }
            __syncthreads(); // this panel's buffer is filled again in the next step
        }
        float* ob = out + batch * int64_t(M) * N;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
            {
                const int m = m0 + wm + 8 * i + g, n = n0 + wn + 8 * j + 2 * t;
                if (m < M)
                {
                    float* o = ob + int64_t(m) * N + n;
                    if (VEC && n + 1 < N) // N even: the pair is 8-byte aligned
                        *reinterpret_cast<float2*>(o) = make_float2(static_cast<float>(acc[i][j][0]), static_cast<float>(acc[i][j][1]));
                    else
                    {
                        if (n < N)
                            o[0] = static_cast<float>(acc[i][j][0]);
                        if (n + 1 < N)
                            o[1] = static_cast<float>(acc[i][j][1]);
                    }
                }
            }
    }

    // One tile shape of the product: what it would cost, and its launch.
    template <int WM, int WN, int MT, int NT>
    struct BmmShape
    {
        static constexpr int TM = WM * MT * 8, TN = WN * NT * 8;
        static int64_t tiles(int64_t batch, int64_t M, int64_t N) { return batch * ((M + TM - 1) / TM) * ((N + TN - 1) / TN); }
        // time in units of one 8 x 8 tile's walk over K: rounds of warps over the 4 x 148 scheduler partitions, each warp's
        // MT * NT tiles in turn (its operand loads weigh more the fewer tiles share them)
        static double cost(int64_t batch, int64_t M, int64_t N)
        {
            const double slots = 4.0 * sm_count(), warps = double(tiles(batch, M, N)) * WM * WN;
            const double rounds = warps <= slots ? 1.0 : warps / slots;
            return rounds * (MT * NT + 0.25 * (MT + NT));
        }
        static bool launch(const float* a, const float* b, float* out, int64_t batch, int M, int K, int N, cudaStream_t st)
        {
            constexpr size_t bytes = 2 * sizeof(float) * (TM * (BMM_KC + 4) + BMM_KC * (TN + 8));
            const int64_t blocks = tiles(batch, M, N);
            if (blocks > 0x7FFFFFFF)
                return false;
            const uint32_t tiles_m = uint32_t((M + TM - 1) / TM), tiles_n = uint32_t((N + TN - 1) / TN);
            const bool vec = K % 4 == 0 && N % 4 == 0 && all_aligned16({a, b, out});
            static std::atomic<uint64_t> told{0};
            int dev = 0;
            cudaGetDevice(&dev);
            if (bytes > 48 * 1024 && !((told.load(std::memory_order_relaxed) >> (dev & 63)) & 1))
            {
                if (cudaFuncSetAttribute(bmm_f32_kernel<WM, WN, MT, NT, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)) != cudaSuccess ||
                    cudaFuncSetAttribute(bmm_f32_kernel<WM, WN, MT, NT, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(bytes)) != cudaSuccess)
                    return false;
                told.fetch_or(uint64_t(1) << (dev & 63), std::memory_order_relaxed);
            }
            if (vec)
                bmm_f32_kernel<WM, WN, MT, NT, true><<<unsigned(blocks), WM * WN * 32, bytes, st>>>(a, b, out, M, K, N, tiles_m, tiles_n);
            else
                bmm_f32_kernel<WM, WN, MT, NT, false><<<unsigned(blocks), WM * WN * 32, bytes, st>>>(a, b, out, M, K, N, tiles_m, tiles_n);
            return true;
        }
    };

    template <typename I>
    __global__ void __launch_bounds__(256) gather_rows_kernel(const uint32_t* __restrict__ table, const I* __restrict__ idx,
                                                              uint32_t* __restrict__ out, int64_t n_idx, int64_t row_words,
                                                              int64_t n_rows)
    {
        const int64_t total = n_idx * row_words;
        for (int64_t i = int64_t(blockIdx.x) * blockDim.x + threadIdx.x; i < total; i += int64_t(gridDim.x) * blockDim.x)
        {
            const int64_t r = i / row_words, w = i - r * row_words;
            const int64_t src = int64_t(idx[r]);
            out[i] = (src >= 0 && src < n_rows) ? table[src * row_words + w] : 0u; // the reference does not check
        }
    }

    static unsigned grid_for(int64_t n, int threads)
    {
        int64_t blocks = (n + threads - 1) / threads;
        const int64_t cap = int64_t(b200::sm_count()) * 16;
        return unsigned(blocks < cap ? (blocks > 0 ? blocks : 1) : cap);
    }
}

extern "C" int b200_f32_binary(int op, const float* a, const float* b, float* out, int64_t n, void* stream)
{
    using namespace b200;
    if (n < 0 || op < B200_F32_ADD || op > B200_F32_MIN)
        return B200_ERR_INVALID_ARGUMENT;
    if (n == 0)
        return B200_OK;
    if (!a || !b || !out)
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned g = grid_for(n, 256);
    switch (op)
    {
    case B200_F32_ADD: binary_kernel<B200_F32_ADD><<<g, 256, 0, st>>>(a, b, out, n); break;
    case B200_F32_SUB: binary_kernel<B200_F32_SUB><<<g, 256, 0, st>>>(a, b, out, n); break;
    case B200_F32_MUL: binary_kernel<B200_F32_MUL><<<g, 256, 0, st>>>(a, b, out, n); break;
    case B200_F32_DIV: binary_kernel<B200_F32_DIV><<<g, 256, 0, st>>>(a, b, out, n); break;
    case B200_F32_MAX: binary_kernel<B200_F32_MAX><<<g, 256, 0, st>>>(a, b, out, n); break;
    default: binary_kernel<B200_F32_MIN><<<g, 256, 0, st>>>(a, b, out, n); break;
    }
    return after_launch("b200_f32_binary");
}

extern "C" int b200_f32_binary_periodic(int op, const float* a, const float* v, float* out, int64_t n, int64_t period, int v_is_left,
                                        void* stream)
{
    using namespace b200;
    if (n < 0 || period < 1 || op < B200_F32_ADD || op > B200_F32_MIN)
        return B200_ERR_INVALID_ARGUMENT;
    if (n == 0)
        return B200_OK;
    if (!a || !v || !out || n % period != 0)
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool left = v_is_left != 0;
    switch (op)
    {
    case B200_F32_ADD: launch_binary_periodic<B200_F32_ADD>(a, v, out, n, period, left, st); break;
    case B200_F32_SUB: launch_binary_periodic<B200_F32_SUB>(a, v, out, n, period, left, st); break;
    case B200_F32_MUL: launch_binary_periodic<B200_F32_MUL>(a, v, out, n, period, left, st); break;
    case B200_F32_DIV: launch_binary_periodic<B200_F32_DIV>(a, v, out, n, period, left, st); break;
    case B200_F32_MAX: launch_binary_periodic<B200_F32_MAX>(a, v, out, n, period, left, st); break;
    default: launch_binary_periodic<B200_F32_MIN>(a, v, out, n, period, left, st); break;
    }
    return after_launch("b200_f32_binary_periodic");
}

extern "C" int b200_f32_unary(int op, const float* x, float* out, int64_t n, void* stream)
{
    using namespace b200;
    if (n < 0 || op < B200_F32_ABS || op > B200_F32_RELU)
        return B200_ERR_INVALID_ARGUMENT;
    if (n == 0)
        return B200_OK;
    if (!x || !out)
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const unsigned g = grid_for(n, 256);
    switch (op)
    {
    case B200_F32_ABS: unary_kernel<B200_F32_ABS><<<g, 256, 0, st>>>(x, out, n); break;
    case B200_F32_NEG: unary_kernel<B200_F32_NEG><<<g, 256, 0, st>>>(x, out, n); break;
    case B200_F32_SQRT: unary_kernel<B200_F32_SQRT><<<g, 256, 0, st>>>(x, out, n); break;
    case B200_F32_EXP: unary_kernel<B200_F32_EXP><<<g, 256, 0, st>>>(x, out, n); break;
    case B200_F32_ERF: unary_kernel<B200_F32_ERF><<<g, 256, 0, st>>>(x, out, n); break;
    default: unary_kernel<B200_F32_RELU><<<g, 256, 0, st>>>(x, out, n); break;
    }
    return after_launch("b200_f32_unary");
}

namespace b200
{
    static bool valid_shape(const int64_t* shape, int rank)
    {
        if (rank < 0 || rank > MAX_RANK || (rank > 0 && !shape))
            return false;
        for (int i = 0; i < rank; ++i)
            if (shape[i] < 0)
                return false;
        return true;
    }
    static int64_t count_of(const int64_t* shape, int rank)
    {
        int64_t n = 1;
        for (int i = 0; i < rank; ++i)
            n *= shape[i];
        return n;
    }
}

extern "C" int b200_broadcast_b32(const void* in, void* out, const int64_t* out_shape, int rank, const int64_t* broadcast_axes,
                                  int n_axes, void* stream)
{
    using namespace b200;
    if (!valid_shape(out_shape, rank) || n_axes < 0 || n_axes > rank || (n_axes > 0 && !broadcast_axes))
        return B200_ERR_INVALID_ARGUMENT;
    bool is_new[MAX_RANK] = {false};
    for (int i = 0; i < n_axes; ++i)
    {
        if (broadcast_axes[i] < 0 || broadcast_axes[i] >= rank || is_new[broadcast_axes[i]])
            return B200_ERR_INVALID_ARGUMENT;
        is_new[broadcast_axes[i]] = true;
    }
    const int64_t n = count_of(out_shape, rank);
    if (n == 0)
        return B200_OK;
    if (!in || !out)
        return B200_ERR_INVALID_ARGUMENT;
    Dims d;
    d.rank = rank;
    int64_t stride = 1;
    for (int a = rank - 1; a >= 0; --a)
    {
        d.out_dim[a] = out_shape[a];
        d.in_stride[a] = is_new[a] ? 0 : stride;
        if (!is_new[a])
            stride *= out_shape[a];
    }
    launch_remap(in, out, d, n, stride, static_cast<cudaStream_t>(stream)); // stride: the input's element count by now
    return after_launch("b200_broadcast_b32");
}

extern "C" int b200_permute_b32(const void* in, void* out, const int64_t* in_shape, int rank, const int64_t* order, void* stream)
{
    using namespace b200;
    if (!valid_shape(in_shape, rank) || (rank > 0 && !order))
        return B200_ERR_INVALID_ARGUMENT;
    bool seen[MAX_RANK] = {false};
    for (int i = 0; i < rank; ++i)
    {
        if (order[i] < 0 || order[i] >= rank || seen[order[i]])
            return B200_ERR_INVALID_ARGUMENT;
        seen[order[i]] = true;
    }
    const int64_t n = count_of(in_shape, rank);
    if (n == 0)
        return B200_OK;
    if (!in || !out)
        return B200_ERR_INVALID_ARGUMENT;
    int64_t in_stride[MAX_RANK];
    int64_t s = 1;
    for (int a = rank - 1; a >= 0; --a)
    {
        in_stride[a] = s;
        s *= in_shape[a];
    }
    Dims d;
    d.rank = rank;
    for (int a = 0; a < rank; ++a)
    {
        d.out_dim[a] = in_shape[order[a]];
        d.in_stride[a] = in_stride[order[a]];
    }
    launch_remap(in, out, d, n, n, static_cast<cudaStream_t>(stream));
    return after_launch("b200_permute_b32");
}

extern "C" int b200_reduce_f32(int op, const float* in, float* out, const int64_t* shape, int rank, const int64_t* axes, int n_axes,
                               void* stream)
{
    using namespace b200;
    if (op < B200_REDUCE_SUM || op > B200_REDUCE_MAX_ABS || !valid_shape(shape, rank) || n_axes < 0 || n_axes > rank ||
        (n_axes > 0 && !axes))
        return B200_ERR_INVALID_ARGUMENT;
    bool reduced[MAX_RANK] = {false};
    for (int i = 0; i < n_axes; ++i)
    {
        if (axes[i] < 0 || axes[i] >= rank || reduced[axes[i]])
            return B200_ERR_INVALID_ARGUMENT;
        reduced[axes[i]] = true;
    }
    int64_t stride[MAX_RANK];
    int64_t s = 1;
    for (int a = rank - 1; a >= 0; --a)
    {
        stride[a] = s;
        s *= shape[a];
    }
    Dims keep, red;
    keep.rank = red.rank = 0;
    int64_t n_out = 1, n_red = 1;
    for (int a = 0; a < rank; ++a)
    {
        Dims& d = reduced[a] ? red : keep;
        d.out_dim[d.rank] = shape[a];
        d.in_stride[d.rank] = stride[a];
        ++d.rank;
        (reduced[a] ? n_red : n_out) *= shape[a];
    }
    if (n_out == 0)
        return B200_OK;
    if (!out || (!in && n_red > 0))
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (op != B200_REDUCE_SUM && n_out == 1 && n_red > 0)
    {
        // every axis reduced: the input is one contiguous run.  Up to a million elements one cluster reads it about as fast
        // as the extra launch of the atomic form takes.
        const bool small = n_red <= (int64_t(1) << 20);
        if (!small)
        {
            fill_f32_kernel<<<1, 32, 0, st>>>(out, op == B200_REDUCE_MIN ? INFINITY : -INFINITY, 1);
            g_launches.fetch_add(1, std::memory_order_relaxed);
        }
        const unsigned grid = small ? EXTREME_CLUSTER : unsigned(std::min<int64_t>((n_red + 8191) / 8192, sm_count() * 8));
        switch (op)
        {
        case B200_REDUCE_MAX:
            small ? reduce_extreme_cluster_kernel<B200_REDUCE_MAX><<<grid, 1024, 0, st>>>(in, out, n_red)
                  : reduce_extreme_all_kernel<B200_REDUCE_MAX><<<grid, 256, 0, st>>>(in, out, n_red);
            break;
        case B200_REDUCE_MIN:
            small ? reduce_extreme_cluster_kernel<B200_REDUCE_MIN><<<grid, 1024, 0, st>>>(in, out, n_red)
                  : reduce_extreme_all_kernel<B200_REDUCE_MIN><<<grid, 256, 0, st>>>(in, out, n_red);
            break;
        default:
            small ? reduce_extreme_cluster_kernel<B200_REDUCE_MAX_ABS><<<grid, 1024, 0, st>>>(in, out, n_red)
                  : reduce_extreme_all_kernel<B200_REDUCE_MAX_ABS><<<grid, 256, 0, st>>>(in, out, n_red);
        }
    }
    else if (op != B200_REDUCE_SUM && n_out <= 4096 && n_red >= 1024)
    {
        if (op == B200_REDUCE_MAX)
            reduce_extreme_block_kernel<B200_REDUCE_MAX><<<unsigned(n_out), 256, 0, st>>>(in, out, keep, red, n_red);
        else if (op == B200_REDUCE_MIN)
            reduce_extreme_block_kernel<B200_REDUCE_MIN><<<unsigned(n_out), 256, 0, st>>>(in, out, keep, red, n_red);
        else
            reduce_extreme_block_kernel<B200_REDUCE_MAX_ABS><<<unsigned(n_out), 256, 0, st>>>(in, out, keep, red, n_red);
    }
    else if (op == B200_REDUCE_SUM && n_axes == 1 && axes[0] == rank - 1 && n_out >= 64)
    {
        // the last axis of a matrix with many rows: panels staged through shared memory
        const int64_t warps = (n_out + 31) / 32, cap = b200::sm_count() * 16;
        sum_rows_kernel<<<unsigned(warps < cap ? warps : cap), 32, 0, st>>>(in, out, n_out, n_red);
    }
    else if (op == B200_REDUCE_SUM)
        reduce_kernel<B200_REDUCE_SUM><<<grid_for(n_out, 128), 128, 0, st>>>(in, out, keep, red, n_out, n_red);
    else if (op == B200_REDUCE_MAX)
        reduce_kernel<B200_REDUCE_MAX><<<grid_for(n_out, 128), 128, 0, st>>>(in, out, keep, red, n_out, n_red);
    else if (op == B200_REDUCE_MAX_ABS)
        reduce_kernel<B200_REDUCE_MAX_ABS><<<grid_for(n_out, 128), 128, 0, st>>>(in, out, keep, red, n_out, n_red);
    else
        reduce_kernel<B200_REDUCE_MIN><<<grid_for(n_out, 128), 128, 0, st>>>(in, out, keep, red, n_out, n_red);
    return after_launch("b200_reduce_f32");
}

extern "C" int b200_softmax_rows_f32(const float* x, float* out, int64_t rows, int64_t row_elements, void* stream)
{
    return b200_softmax_rows_scaled_f32(x, nullptr, out, rows, row_elements, stream);
}

extern "C" int b200_softmax_rows_scaled_f32(const float* x, const float* factor, float* out, int64_t rows, int64_t row_elements,
                                            void* stream)
{
    using namespace b200;
    if (rows < 0 || row_elements < 0)
        return B200_ERR_INVALID_ARGUMENT;
    if (rows * row_elements == 0)
        return B200_OK;
    if (!x || !out)
        return B200_ERR_INVALID_ARGUMENT;
    if (row_elements > 1535)
        return B200_ERR_UNSUPPORTED; // a row too long to stage: the caller composes the five steps instead
    const int L = int(row_elements);
    const bool vec = L % 4 == 0 && all_aligned16({x, out});
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    unsigned grid;
    size_t bytes;
    if (!(vec ? staged_launch_shape(softmax_rows_kernel<true>, rows, L, vec, grid, bytes)
              : staged_launch_shape(softmax_rows_kernel<false>, rows, L, vec, grid, bytes)))
        return B200_ERR_CUDA;
    if (vec)
        softmax_rows_kernel<true><<<grid, 128, bytes, st>>>(x, factor, out, rows, L);
    else
        softmax_rows_kernel<false><<<grid, 128, bytes, st>>>(x, factor, out, rows, L);
    return after_launch("b200_softmax_rows_f32");
}

extern "C" int b200_layer_norm_rows_f32(const float* x, const float* gamma, const float* beta, float* out, int64_t rows,
                                        int64_t row_elements, float epsilon, void* stream)
{
    return b200_layer_norm_rows_sum_f32(x, nullptr, gamma, beta, out, rows, row_elements, epsilon, stream);
}

extern "C" int b200_layer_norm_rows_sum_f32(const float* x, const float* addend, const float* gamma, const float* beta, float* out,
                                            int64_t rows, int64_t row_elements, float epsilon, void* stream)
{
    using namespace b200;
    if (rows < 0 || row_elements < 0)
        return B200_ERR_INVALID_ARGUMENT;
    if (rows * row_elements == 0)
        return B200_OK;
    if (!x || !gamma || !beta || !out)
        return B200_ERR_INVALID_ARGUMENT;
    if (row_elements > 1535)
        return B200_ERR_UNSUPPORTED; // a row too long to stage: the caller runs the decomposition
    const int L = int(row_elements);
    const bool vec = L % 4 == 0 && all_aligned16({x, addend, gamma, beta, out});
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const float count = static_cast<float>(row_elements);
    unsigned grid;
    size_t bytes;
    if (!(vec ? staged_launch_shape(layer_norm_rows_kernel<true>, rows, L, vec, grid, bytes)
              : staged_launch_shape(layer_norm_rows_kernel<false>, rows, L, vec, grid, bytes)))
        return B200_ERR_CUDA;
    if (vec)
        layer_norm_rows_kernel<true><<<grid, 128, bytes, st>>>(x, addend, gamma, beta, out, rows, L, count, epsilon);
    else
        layer_norm_rows_kernel<false><<<grid, 128, bytes, st>>>(x, addend, gamma, beta, out, rows, L, count, epsilon);
    return after_launch("b200_layer_norm_rows_f32");
}

extern "C" int b200_gelu_f32(const float* x, float* out, int64_t n, void* stream)
{
    using namespace b200;
    if (n < 0)
        return B200_ERR_INVALID_ARGUMENT;
    if (n == 0)
        return B200_OK;
    if (!x || !out)
        return B200_ERR_INVALID_ARGUMENT;
    gelu_kernel<<<grid_for(n, 256), 256, 0, static_cast<cudaStream_t>(stream)>>>(x, out, n);
    return after_launch("b200_gelu_f32");
}

extern "C" int b200_bmm_f32(const float* a, const float* b, float* out, int64_t batch, int64_t M, int64_t K, int64_t N, void* stream)
{
    using namespace b200;
    if (batch < 0 || M < 0 || K < 0 || N < 0 || M > 0x7FFFFFFF || K > 0x7FFFFFFF || N > 0x7FFFFFFF)
        return B200_ERR_INVALID_ARGUMENT;
    if (batch * M * N == 0)
        return B200_OK;
    if (!out || (K > 0 && (!a || !b)))
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    // the largest tile that spreads over the scheduler partitions: smaller ones load their operands more often, larger ones
    // leave partitions idle on small products (12 x [128, 128] x [128, 128] is 24 tiles of 128 x 64 for 148 SMs)
    using Big = BmmShape<4, 2, 4, 4>;
    using Mid = BmmShape<2, 2, 4, 4>;
    using Small = BmmShape<2, 2, 2, 2>;
    const double big = Big::cost(batch, M, N), mid = Mid::cost(batch, M, N), small = Small::cost(batch, M, N);
    const bool ok = big <= mid && big <= small ? Big::launch(a, b, out, batch, int(M), int(K), int(N), st)
                    : mid <= small             ? Mid::launch(a, b, out, batch, int(M), int(K), int(N), st)
                                               : Small::launch(a, b, out, batch, int(M), int(K), int(N), st);
    if (!ok)
        return B200_ERR_TOO_LARGE;
    return after_launch("b200_bmm_f32");
}

extern "C" int b200_gather_rows_b32(const void* table, int64_t n_rows, int64_t row_elements, const void* indices, int index_type,
                                    int64_t n_indices, void* out, void* stream)
{
    using namespace b200;
    if (n_rows < 0 || row_elements < 0 || n_indices < 0 || (index_type != B200_I32 && index_type != B200_I64))
        return B200_ERR_INVALID_ARGUMENT;
    const int64_t total = n_indices * row_elements;
    if (total == 0)
        return B200_OK;
    if (!table || !indices || !out)
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    if (index_type == B200_I32)
        gather_rows_kernel<int32_t><<<grid_for(total, 256), 256, 0, st>>>(static_cast<const uint32_t*>(table),
                                                                          static_cast<const int32_t*>(indices),
                                                                          static_cast<uint32_t*>(out), n_indices, row_elements, n_rows);
    else
        gather_rows_kernel<int64_t><<<grid_for(total, 256), 256, 0, st>>>(static_cast<const uint32_t*>(table),
                                                                          static_cast<const int64_t*>(indices),
                                                                          static_cast<uint32_t*>(out), n_indices, row_elements, n_rows);
    return after_launch("b200_gather_rows_b32");
}
