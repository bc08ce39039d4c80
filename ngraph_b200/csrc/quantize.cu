// Quantize / Dequantize: HBM-streaming kernels (5 bytes per element for 8-bit types).
//
// Arithmetic follows runtime::reference::quantize / dequantize
// (src/ngraph/runtime/reference/quantize.hpp:30-117, dequantize.hpp:32-52) exactly;
// the iteration order does not matter because every element is independent.
//
// Two launch shapes:
//   stream  - the tensor is viewed as [rows, inner] where every row has ONE scale / zero point (per-tensor: a single
//             row; per-axis on axis a: rows = prod(shape[0..a]), inner = prod(shape[a+1..])) but is walked as one flat
//             run of 16-byte vectors, wherever the rows start and end: 128-bit loads, packed 32-bit (or 128-bit) stores,
//             one to eight independent loads in flight per thread, by size.  The scales of the rows a block touches are looked up once per
//             block into a small shared-memory table while its loads are under way.
//   generic - one element per thread with the scale index recomputed from the
//             coordinates; any axis set, any alignment.
#include <type_traits>
#include "common.cuh"

namespace b200
{
    constexpr int QT = 256;                // threads per block
    constexpr int MIN_INNER = 16;          // shortest row the streaming kernels take

    struct ProjDims
    {
        int rank;
        int64_t shape[B200_MAX_RANK];
        int64_t sstride[B200_MAX_RANK]; // stride into scale/zero_point (0 for non-axes)
    };

    __device__ __forceinline__ int64_t project_index(const ProjDims& d, int64_t idx)
    {
        int64_t s = 0;
#pragma unroll 1
        for (int i = d.rank - 1; i >= 0; --i)
        {
            int64_t q = idx / d.shape[i];
            int64_t c = idx - q * d.shape[i];
            s += c * d.sstride[i];
            idx = q;
        }
        return s;
    }

    template <typename Q>
    __device__ __forceinline__ void store4(Q* p, Q a, Q b, Q c, Q d);
    template <>
    __device__ __forceinline__ void store4<uint8_t>(uint8_t* p, uint8_t a, uint8_t b, uint8_t c, uint8_t d)
    {
        *reinterpret_cast<uint32_t*>(p) = uint32_t(a) | (uint32_t(b) << 8) | (uint32_t(c) << 16) | (uint32_t(d) << 24);
    }
    template <>
    __device__ __forceinline__ void store4<int8_t>(int8_t* p, int8_t a, int8_t b, int8_t c, int8_t d)
    {
        *reinterpret_cast<uint32_t*>(p) = uint32_t(uint8_t(a)) | (uint32_t(uint8_t(b)) << 8) |
                                          (uint32_t(uint8_t(c)) << 16) | (uint32_t(uint8_t(d)) << 24);
    }
    template <>
    __device__ __forceinline__ void store4<int32_t>(int32_t* p, int32_t a, int32_t b, int32_t c, int32_t d)
    {
        *reinterpret_cast<int4*>(p) = make_int4(a, b, c, d);
    }

    // The [rows, inner] view of a tensor, with what replaces divisions by `inner` (see make_rows).
    struct RowMap
    {
        int64_t total, inner;
        FastDiv n_scales;
        uint64_t inner_inv64;  // ceil(2^64 / inner): row of a block's first element
        uint32_t inner_inv32;  // ceil(2^32 / inner): rows inside a block, for inner < the block's elements
    };

    // Where a block's first element lies: its row, and its offset inside that row.  The product with the rounded-up reciprocal is
    // the quotient or one more, whatever the sizes.
    __device__ __forceinline__ void block_row(const RowMap& m, int64_t base, uint32_t& row, int64_t& r0)
    {
        int64_t q = int64_t(__umul64hi(uint64_t(base), m.inner_inv64));
        if (q * m.inner > base)
            --q;
        row = uint32_t(q);
        r0 = base - q * m.inner;
    }

    // Row (counted from the block's first) of the element `off` = r0 + local, and the elements left in that row.
    __device__ __forceinline__ uint32_t local_row(const RowMap& m, uint32_t off, uint32_t& left)
    {
        const uint32_t r = __umulhi(off, m.inner_inv32);
        left = (r + 1) * uint32_t(m.inner) - off; // (rows shorter than a block)
        return r;
    }

    // Four elements with one scale.  FAST (8-bit outputs): the row's scale s is uniform, so y = RN(1/s) is computed once
    // (correctly rounded reciprocal) and each quotient is  q0 = RN(x*y);  e = x - q0*s (exact in one FMA);
    // q = RN(q0 + e*y), which is the correctly rounded x/s (Markstein's division theorem) whenever s is a normal number
    // whose significand is not all ones and nothing over/underflows.  y == 0 marks a scale that fails that test (or the
    // switched-off path): a block that meets one takes the IEEE division instead.  Quotients of magnitude >= 2^24, whose 8-bit result saturates
    // regardless of the last bit, skip the correction (see common.cuh).  Every output byte equals the plain
    // x / s -> rounding -> +zero_point -> clamp sequence of the reference.  An int32 output can be large enough for
    // the last bit of a quotient beyond 2^24 to matter, so it always divides.
    template <typename Q, int MODE, bool FAST>
    __device__ __forceinline__ void quantize4(const float4& v, float s, float y, int zi, Q (&r)[4])
    {
        if (FAST)
        {
            const int lo = int(QLimits<Q>::lo) - zi, hi = int(QLimits<Q>::hi) - zi;
            constexpr bool directed = MODE == B200_ROUND_TOWARD_INFINITY || MODE == B200_ROUND_TOWARD_ZERO || MODE == B200_ROUND_UP ||
                                      MODE == B200_ROUND_DOWN;
            int i[4];
            if (directed)
                quantize4_directed_fast<MODE>(v, s, y, __fmul_rn(fabsf(s), 5.9604644775390625e-8f) /* |s| * 2^-24 */, lo, hi, zi, i);
            else if (MODE == B200_ROUND_NEAREST_TOWARD_EVEN)
            {
                i[0] = quantize_rne_fast<Q>(v.x, s, y, lo, hi, zi), i[1] = quantize_rne_fast<Q>(v.y, s, y, lo, hi, zi);
                i[2] = quantize_rne_fast<Q>(v.z, s, y, lo, hi, zi), i[3] = quantize_rne_fast<Q>(v.w, s, y, lo, hi, zi);
            }
            else
            {
                i[0] = quantize_int_fast<Q, MODE>(v.x, s, y, lo, hi, zi), i[1] = quantize_int_fast<Q, MODE>(v.y, s, y, lo, hi, zi);
                i[2] = quantize_int_fast<Q, MODE>(v.z, s, y, lo, hi, zi), i[3] = quantize_int_fast<Q, MODE>(v.w, s, y, lo, hi, zi);
            }
#pragma unroll
            for (int j = 0; j < 4; ++j)
                r[j] = static_cast<Q>(i[j]);
        }
        else
        {
            const float z = static_cast<float>(static_cast<Q>(zi));
            r[0] = quantize_one<Q, MODE>(v.x, s, z), r[1] = quantize_one<Q, MODE>(v.y, s, z);
            r[2] = quantize_one<Q, MODE>(v.z, s, z), r[3] = quantize_one<Q, MODE>(v.w, s, z);
        }
    }

    // A row's scale as the kernels use it: {scale, reciprocal or 0, zero point}.
    struct RowScale
    {
        float s, y;
        int zp;
    };
    template <typename Q, bool FAST>
    __device__ __forceinline__ RowScale row_scale(const float* scale, const Q* zp, uint32_t i, bool fast)
    {
        RowScale e;
        e.s = __ldg(scale + i);
        e.zp = static_cast<int>(zp[i]);
        e.y = FAST && fast && scale_allows_fast_division(e.s) ? __frcp_rn(e.s) : 0.0f;
        return e;
    }

    // How a block finds the scale of an element, by the rows it can touch.
    enum Rows
    {
        ONE_ROW,  // per tensor: one scale
        TWO_ROWS, // rows at least as long as a block's elements: the scales of the block's first row and of the next one, in
                  // registers, and the place where the second begins
        MANY_ROWS // shorter ones: a table in shared memory, filled by as many threads as there are rows
    };
    template <typename Q, bool FAST, int ROWS, int CHUNK>
    struct BlockScales
    {
        RowScale e0, e1;
        uint32_t boundary; // TWO_ROWS: first element of the second row, CHUNK if there is none in the block
        uint32_t r0;
        RowScale* table;

        // true if every scale of the block admits the fast division
        __device__ __forceinline__ bool find(const RowMap& m, RowScale* shared, const float* scale, const Q* zp, int64_t base, uint32_t rem, bool fast)
        {
            boundary = CHUNK;
            if (ROWS == ONE_ROW)
            {
                e0 = e1 = row_scale<Q, FAST>(scale, zp, 0, fast);
                return e0.y != 0.0f;
            }
            uint32_t row;
            int64_t in_row;
            block_row(m, base, row, in_row);
            r0 = uint32_t(in_row); // (of rows shorter than a block)
            const uint32_t first = row - m.n_scales.div(row) * m.n_scales.d;
            if (ROWS == TWO_ROWS)
            {
                e0 = e1 = row_scale<Q, FAST>(scale, zp, first, fast);
                if (m.inner - in_row < int64_t(rem))
                {
                    boundary = uint32_t(m.inner - in_row);
                    e1 = row_scale<Q, FAST>(scale, zp, first + 1 == m.n_scales.d ? 0 : first + 1, fast);
                }
                return e0.y != 0.0f && e1.y != 0.0f;
            }
            table = shared;
            uint32_t left;
            const uint32_t n = local_row(m, r0 + rem - 1, left) + 1;
            bool ok = true;
            for (uint32_t i = threadIdx.x; i < n; i += QT)
            {
                const RowScale e = row_scale<Q, FAST>(scale, zp, row + i - m.n_scales.div(row + i) * m.n_scales.d, fast);
                ok = ok && e.y != 0.0f;
                shared[i] = e;
            }
            return __syncthreads_and(ok);
        }
        __device__ __forceinline__ RowScale of(const RowMap& m, uint32_t i) const
        {
            if (ROWS == ONE_ROW)
                return e0;
            if (ROWS == TWO_ROWS)
                return i >= boundary ? e1 : e0;
            uint32_t left;
            return table[local_row(m, r0 + i, left)];
        }
    };

    // U vectors of four elements per thread (see vectors_per_thread); blocks_for: what the registers are kept down for.
    constexpr int blocks_for(int u) { return u >= 8 ? 4 : 6; }
    // Bound by HBM for large tensors (f32 -> u8 at 1 GB: 6.3 TB/s in a half-way mode, a plain copy's rate) and by load latency below some 100 MB.  Walking the tensor
    // flat instead of row by row is what keeps odd row lengths on 128-bit accesses: [24, 64, 113, 113] per channel 182 -> 20 us,
    // [4000, 64, 15, 13] 458 -> 55 us.
    template <typename Q, int MODE, bool FAST, int ROWS, int U>
    __global__ void __launch_bounds__(QT, blocks_for(U)) quantize_stream_kernel(const float* __restrict__ x, const float* __restrict__ scale,
                                                                          const Q* __restrict__ zp, Q* __restrict__ out, RowMap m, bool fast)
    {
        after_earlier_kernels(x, scale, zp, out);
        constexpr int CHUNK = QT * U * 4;
        __shared__ RowScale table[ROWS == MANY_ROWS ? CHUNK / MIN_INNER + 2 : 1];
        const int64_t base = int64_t(blockIdx.x) * CHUNK;
        const uint32_t rem = uint32_t(min(m.total - base, int64_t(CHUNK)));
        x += base;
        out += base;
        float4 v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const uint32_t off = (u * QT + threadIdx.x) * 4;
            if (off + 4 <= rem)
                v[u] = *reinterpret_cast<const float4*>(x + off);
        }
        BlockScales<Q, FAST, ROWS, CHUNK> scales;
        const bool all_fast = scales.find(m, table, scale, zp, base, rem, fast);
        auto one = [&](uint32_t i, const RowScale& e) { out[i] = quantize_one<Q, MODE>(x[i], e.s, static_cast<float>(static_cast<Q>(e.zp))); };
        if (FAST && !all_fast)
        {
            for (uint32_t i = threadIdx.x; i < rem; i += QT)
                one(i, scales.of(m, i));
            return;
        }
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const uint32_t off = (u * QT + threadIdx.x) * 4;
            if (off + 4 > rem)
                break;
            Q r[4];
            if (ROWS == MANY_ROWS)
            {
                // four elements with the vector's row; where it runs into the next row, once more with that row's scale
                uint32_t left, lr = local_row(m, scales.r0 + off, left), done = 0;
#pragma unroll 1
                do
                {
                    Q t[4];
                    const RowScale e = table[lr++];
                    quantize4<Q, MODE, FAST>(v[u], e.s, e.y, e.zp, t);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
                        r[j] = j >= int(done) ? t[j] : r[j];
                    done = left;
                    left = 4;
                } while (done < 4);
            }
            else
            {
                const RowScale e = scales.of(m, off);
                quantize4<Q, MODE, FAST>(v[u], e.s, e.y, e.zp, r);
            }
            store4<Q>(out + off, r[0], r[1], r[2], r[3]);
        }
        // what the whole vectors leave: the elements that a vector of the first row has of the second (the thread that wrote
        // the vector writes them again), and the last, partial vector of the tensor
        if (ROWS == TWO_ROWS && (scales.boundary & 3) != 0 && threadIdx.x == (scales.boundary / 4) % QT)
            for (uint32_t i = scales.boundary; (i & 3) != 0 && i < rem; ++i)
                one(i, scales.e1);
        if ((rem & 3) != 0 && threadIdx.x == (rem / 4) % QT)
            for (uint32_t i = rem & ~3u; i < rem; ++i)
                one(i, scales.of(m, i));
    }

    template <typename Q, int MODE>
    __global__ void __launch_bounds__(QT) quantize_generic_kernel(const float* __restrict__ x,
                                                                  const float* __restrict__ scale,
                                                                  const Q* __restrict__ zp,
                                                                  Q* __restrict__ out,
                                                                  int64_t total,
                                                                  ProjDims dims)
    {
        for (int64_t i = int64_t(blockIdx.x) * QT + threadIdx.x; i < total; i += int64_t(gridDim.x) * QT)
        {
            int64_t sidx = project_index(dims, i);
            out[i] = quantize_one<Q, MODE>(x[i], scale[sidx], static_cast<float>(zp[sidx]));
        }
    }

    // out = (float)(in - zp) * scale   (dequantize.hpp:47-51; the subtraction is exact in int)
    template <typename Q>
    __device__ __forceinline__ float dequantize_one(Q v, int zp, float s)
    {
        return __fmul_rn(static_cast<float>(int(v) - zp), s);
    }
    template <>
    __device__ __forceinline__ float dequantize_one<int32_t>(int32_t v, int zp, float s)
    {
        // int32 - int32 as the reference computes it (wraps on overflow here; UB there)
        return __fmul_rn(static_cast<float>(int32_t(uint32_t(v) - uint32_t(zp))), s);
    }

    template <typename Q>
    struct Vec4;
    template <>
    struct Vec4<uint8_t>
    {
        uint32_t w;
        __device__ __forceinline__ void load(const uint8_t* p) { w = *reinterpret_cast<const uint32_t*>(p); }
        __device__ __forceinline__ uint8_t get(int i) const { return uint8_t(w >> (8 * i)); }
    };
    template <>
    struct Vec4<int8_t>
    {
        uint32_t w;
        __device__ __forceinline__ void load(const int8_t* p) { w = *reinterpret_cast<const uint32_t*>(p); }
        __device__ __forceinline__ int8_t get(int i) const { return int8_t(uint8_t(w >> (8 * i))); }
    };
    template <>
    struct Vec4<int32_t>
    {
        int4 w;
        __device__ __forceinline__ void load(const int32_t* p) { w = *reinterpret_cast<const int4*>(p); }
        __device__ __forceinline__ int32_t get(int i) const { return i == 0 ? w.x : i == 1 ? w.y : i == 2 ? w.z : w.w; }
    };

    // The same walk as quantize_stream_kernel.
    template <typename Q, int ROWS, int U>
    __global__ void __launch_bounds__(QT, blocks_for(U)) dequantize_stream_kernel(const Q* __restrict__ in, const float* __restrict__ scale,
                                                                            const Q* __restrict__ zp, float* __restrict__ out, RowMap m)
    {
        after_earlier_kernels(in, scale, zp, out);
        constexpr int CHUNK = QT * U * 4;
        __shared__ RowScale table[ROWS == MANY_ROWS ? CHUNK / MIN_INNER + 2 : 1];
        const int64_t base = int64_t(blockIdx.x) * CHUNK;
        const uint32_t rem = uint32_t(min(m.total - base, int64_t(CHUNK)));
        in += base;
        out += base;
        Vec4<Q> v[U];
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const uint32_t off = (u * QT + threadIdx.x) * 4;
            if (off + 4 <= rem)
                v[u].load(in + off);
        }
        BlockScales<Q, false, ROWS, CHUNK> scales;
        scales.find(m, table, scale, zp, base, rem, false);
#pragma unroll
        for (int u = 0; u < U; ++u)
        {
            const uint32_t off = (u * QT + threadIdx.x) * 4;
            if (off + 4 > rem)
                break;
            uint32_t left = 4;
            RowScale e, e2;
            if (ROWS == MANY_ROWS)
            {
                const uint32_t lr = local_row(m, scales.r0 + off, left);
                e = table[lr];
                e2 = left < 4 ? table[lr + 1] : e;
            }
            else
                e = e2 = scales.of(m, off);
            float4 r;
            r.x = dequantize_one<Q>(v[u].get(0), e.zp, e.s);
            r.y = dequantize_one<Q>(v[u].get(1), left > 1 ? e.zp : e2.zp, left > 1 ? e.s : e2.s);
            r.z = dequantize_one<Q>(v[u].get(2), left > 2 ? e.zp : e2.zp, left > 2 ? e.s : e2.s);
            r.w = dequantize_one<Q>(v[u].get(3), left > 3 ? e.zp : e2.zp, left > 3 ? e.s : e2.s);
            *reinterpret_cast<float4*>(out + off) = r;
        }
        if (ROWS == TWO_ROWS && (scales.boundary & 3) != 0 && threadIdx.x == (scales.boundary / 4) % QT)
            for (uint32_t i = scales.boundary; (i & 3) != 0 && i < rem; ++i)
                out[i] = dequantize_one<Q>(in[i], scales.e1.zp, scales.e1.s);
        if ((rem & 3) != 0 && threadIdx.x == (rem / 4) % QT)
            for (uint32_t i = rem & ~3u; i < rem; ++i)
            {
                const RowScale e = scales.of(m, i);
                out[i] = dequantize_one<Q>(in[i], e.zp, e.s);
            }
    }

    template <typename Q>
    __global__ void __launch_bounds__(QT) dequantize_generic_kernel(const Q* __restrict__ in,
                                                                    const float* __restrict__ scale,
                                                                    const Q* __restrict__ zp,
                                                                    float* __restrict__ out,
                                                                    int64_t total,
                                                                    ProjDims dims)
    {
        for (int64_t i = int64_t(blockIdx.x) * QT + threadIdx.x; i < total; i += int64_t(gridDim.x) * QT)
        {
            int64_t sidx = project_index(dims, i);
            out[i] = dequantize_one<Q>(in[i], static_cast<int>(zp[sidx]), scale[sidx]);
        }
    }

    // How the (shape, axes) pair maps onto the two launch shapes.
    struct QuantPlan
    {
        int64_t total;
        bool rows_ok;     // [rows, inner] view with one scale per row exists
        int64_t rows, inner, n_scales;
        ProjDims dims;
    };

    static int make_plan(const int64_t* shape, int rank, const int64_t* axes, int n_axes, QuantPlan& p)
    {
        if (rank < 0 || rank > B200_MAX_RANK || n_axes < 0 || n_axes > rank || (rank > 0 && !shape) ||
            (n_axes > 0 && !axes))
            return B200_ERR_INVALID_ARGUMENT;
        bool is_axis[B200_MAX_RANK] = {false};
        for (int i = 0; i < n_axes; ++i)
        {
            if (axes[i] < 0 || axes[i] >= rank || is_axis[axes[i]] || (i > 0 && axes[i] <= axes[i - 1]))
                return B200_ERR_INVALID_ARGUMENT;
            is_axis[axes[i]] = true;
        }
        p.total = 1;
        for (int i = 0; i < rank; ++i)
        {
            if (shape[i] < 0)
                return B200_ERR_INVALID_ARGUMENT;
            p.total *= shape[i];
        }
        p.dims.rank = rank;
        int64_t ss = 1;
        for (int i = rank - 1; i >= 0; --i)
        {
            p.dims.shape[i] = shape[i];
            p.dims.sstride[i] = is_axis[i] ? ss : 0;
            if (is_axis[i])
                ss *= shape[i];
        }
        p.n_scales = ss;
        // rows view: the axes are one contiguous run [a..b]; every dim before a only repeats the scales
        p.rows_ok = false;
        if (n_axes == 0)
        {
            p.rows_ok = true;
            p.rows = 1;
            p.inner = p.total;
        }
        else if (axes[n_axes - 1] - axes[0] == n_axes - 1)
        {
            int64_t inner = 1, rows = 1;
            for (int i = int(axes[n_axes - 1]) + 1; i < rank; ++i)
                inner *= shape[i];
            for (int i = 0; i <= int(axes[n_axes - 1]); ++i)
                rows *= shape[i];
            p.rows_ok = true;
            p.rows = rows;
            p.inner = inner;
        }
        return B200_OK;
    }

    // The streaming kernels take 16-byte aligned tensors whose rows are at least MIN_INNER long (shorter ones would need
    // more table entries per block than there are threads to fill them in one go).
    static bool make_rows(const QuantPlan& p, const void* a, const void* b, RowMap& m)
    {
        if (!p.rows_ok || ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b)) & 15))
            return false;
        if (p.rows > 1 && (p.inner < MIN_INNER || p.rows >= (int64_t(1) << 31)))
            return false;
        if (p.total / (QT * 4) >= (int64_t(1) << 31) - 1)
            return false;
        m.total = p.total;
        m.n_scales = p.rows > 1 ? FastDiv(uint32_t(p.n_scales)) : FastDiv(1);
        m.inner = p.rows > 1 ? p.inner : 0;
        m.inner_inv64 = p.rows > 1 ? ~uint64_t(0) / uint64_t(p.inner) + 1 : 0;
        m.inner_inv32 = p.rows > 1 ? uint32_t(0xFFFFFFFFull / uint64_t(p.inner) + 1) : 0;
        return true;
    }

    // Vectors per thread.  Few in small calls, which spread over the SMs that way: 1 MB of f32 in 1.2 us, 2 MB in 1.4 us (up to two
    // blocks of one or two vectors per SM; the line was drawn when only such grids were launched early, and has not moved since).
    // Eight in large Quantize calls, where the look-up of a block's scales weighs: per channel at 1 GB 225 us with four, 201 with
    // eight; 16 M elements 16.4 and 18.7 (fewer, longer blocks end less evenly).
    static int vectors_per_thread(int64_t total, bool quantize)
    {
        const int64_t early = int64_t(sm_count()) * 2 * QT * 4; // elements of two blocks per SM, one vector per thread
        if (quantize)
            return total <= 2 * early ? 2 : total < (int64_t(1) << 25) ? 4 : 8;
        return total <= early ? 1 : 4;
    }
    static unsigned stream_grid(int64_t total, int u) { return unsigned((total + QT * u * 4 - 1) / (QT * u * 4)); }

    static unsigned generic_grid(int64_t total)
    {
        int64_t b = (total + QT - 1) / QT;
        const int64_t cap = b200::sm_count() * 8 * 4;
        return unsigned(b < cap ? (b > 0 ? b : 1) : cap);
    }

    std::atomic<int> g_fast_division{1};

    template <typename Q, int MODE>
    static int launch_quantize(const float* x, const float* scale, const void* zp, void* out,
                               const QuantPlan& p, cudaStream_t st)
    {
        constexpr bool FAST = sizeof(Q) == 1;
        const Q* z = static_cast<const Q*>(zp);
        Q* o = static_cast<Q*>(out);
        RowMap m;
        if (make_rows(p, x, out, m))
        {
            const bool fast = g_fast_division.load(std::memory_order_relaxed) != 0;
            const int u = vectors_per_thread(p.total, true);
            const bool two = p.inner >= QT * 4 * u;
            auto go = [&](auto vectors) {
                constexpr int U = decltype(vectors)::value;
                launch(p.rows == 1 ? quantize_stream_kernel<Q, MODE, FAST, ONE_ROW, U>
                       : two       ? quantize_stream_kernel<Q, MODE, FAST, TWO_ROWS, U>
                                   : quantize_stream_kernel<Q, MODE, FAST, MANY_ROWS, U>,
                       stream_grid(p.total, U), QT, 0, st, x, scale, z, o, m, fast);
            };
            if (u == 2)
                go(std::integral_constant<int, 2>());
            else if (u == 4)
                go(std::integral_constant<int, 4>());
            else
                go(std::integral_constant<int, 8>());
        }
        else
            quantize_generic_kernel<Q, MODE><<<generic_grid(p.total), QT, 0, st>>>(x, scale, z, o, p.total, p.dims);
        return after_launch("b200_quantize");
    }

    template <typename Q>
    static int dispatch_quantize_mode(int mode, const float* x, const float* scale, const void* zp, void* out,
                                      const QuantPlan& p, cudaStream_t st)
    {
        switch (mode)
        {
        case 0: return launch_quantize<Q, 0>(x, scale, zp, out, p, st);
        case 1: return launch_quantize<Q, 1>(x, scale, zp, out, p, st);
        case 2: return launch_quantize<Q, 2>(x, scale, zp, out, p, st);
        case 3: return launch_quantize<Q, 3>(x, scale, zp, out, p, st);
        case 4: return launch_quantize<Q, 4>(x, scale, zp, out, p, st);
        case 5: return launch_quantize<Q, 5>(x, scale, zp, out, p, st);
        case 6: return launch_quantize<Q, 6>(x, scale, zp, out, p, st);
        case 7: return launch_quantize<Q, 7>(x, scale, zp, out, p, st);
        case 8: return launch_quantize<Q, 8>(x, scale, zp, out, p, st);
        default: return B200_ERR_INVALID_ARGUMENT;
        }
    }

    template <typename Q>
    static int launch_dequantize(const void* in, const float* scale, const void* zp, float* out,
                                 const QuantPlan& p, cudaStream_t st)
    {
        const Q *q = static_cast<const Q*>(in), *z = static_cast<const Q*>(zp);
        RowMap m;
        if (make_rows(p, in, out, m))
        {
            const int u = vectors_per_thread(p.total, false);
            const bool two = p.inner >= QT * 4 * u;
            auto go = [&](auto vectors) {
                constexpr int U = decltype(vectors)::value;
                launch(p.rows == 1 ? dequantize_stream_kernel<Q, ONE_ROW, U> : two ? dequantize_stream_kernel<Q, TWO_ROWS, U> : dequantize_stream_kernel<Q, MANY_ROWS, U>,
                       stream_grid(p.total, U), QT, 0, st, q, scale, z, out, m);
            };
            if (u == 1)
                go(std::integral_constant<int, 1>());
            else
                go(std::integral_constant<int, 4>());
        }
        else
            dequantize_generic_kernel<Q><<<generic_grid(p.total), QT, 0, st>>>(q, scale, z, out, p.total, p.dims);
        return after_launch("b200_dequantize");
    }
}

extern "C" int b200_set_fast_division(int enable)
{
    int old = b200::g_fast_division.exchange(enable ? 1 : 0);
    return old;
}

extern "C" int b200_quantize(const float* input, const float* scale, const void* zero_point, void* output,
                             int quant_type, const int64_t* shape, int rank, const int64_t* axes, int n_axes,
                             int round_mode, void* stream)
{
    using namespace b200;
    QuantPlan p;
    int rc = make_plan(shape, rank, axes, n_axes, p);
    if (rc != B200_OK)
        return rc;
    if (round_mode < 0 || round_mode > 8)
        return B200_ERR_INVALID_ARGUMENT;
    if (quant_type != B200_U8 && quant_type != B200_I8 && quant_type != B200_I32)
        return B200_ERR_INVALID_ARGUMENT;
    if (p.total == 0)
        return B200_OK;
    if (!input || !scale || !zero_point || !output)
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (quant_type)
    {
    case B200_U8: return dispatch_quantize_mode<uint8_t>(round_mode, input, scale, zero_point, output, p, st);
    case B200_I8: return dispatch_quantize_mode<int8_t>(round_mode, input, scale, zero_point, output, p, st);
    default: return dispatch_quantize_mode<int32_t>(round_mode, input, scale, zero_point, output, p, st);
    }
}

extern "C" int b200_dequantize(const void* input, const float* scale, const void* zero_point, float* output,
                               int quant_type, const int64_t* shape, int rank, const int64_t* axes, int n_axes,
                               void* stream)
{
    using namespace b200;
    QuantPlan p;
    int rc = make_plan(shape, rank, axes, n_axes, p);
    if (rc != B200_OK)
        return rc;
    if (quant_type != B200_U8 && quant_type != B200_I8 && quant_type != B200_I32)
        return B200_ERR_INVALID_ARGUMENT;
    if (p.total == 0)
        return B200_OK;
    if (!input || !scale || !zero_point || !output)
        return B200_ERR_INVALID_ARGUMENT;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    switch (quant_type)
    {
    case B200_U8: return launch_dequantize<uint8_t>(input, scale, zero_point, output, p, st);
    case B200_I8: return launch_dequantize<int8_t>(input, scale, zero_point, output, p, st);
    default: return launch_dequantize<int32_t>(input, scale, zero_point, output, p, st);
    }
}
