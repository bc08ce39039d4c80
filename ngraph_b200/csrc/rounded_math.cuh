// exp and erf on float: evaluated in double and rounded to float once, as std::exp / std::erf on double rounded to float.
//
// The general double routines cost some 40-100 instructions each; that, not memory, bounded Softmax and Gelu.  A float
// argument needs less: the value is a table entry at an equidistant point and a short Taylor step, about a dozen
// double-precision multiply-adds, with an error below 2^-47 of the result (2^-51 for erf).  All ends of the range (denormal and overflowing results, infinities,
// NaN) come out of the same instructions.
//
//   exp(x) = 2^(k >> 4) * 2^((k & 15) / 16) * e^r      k = rint(16 x / ln 2), |r| <= ln2 / 32, degree 6
//   erf(x) = E(g) + D(g) (d - g d^2 + ...)              g = rint(256 |x|) / 256, |d| <= 1 / 512, D = erf', degree 5
//
// The tables are constant-evaluated from the defining series (all terms positive: nothing cancels) and copied to shared memory
// by the kernels that use them.  Against the general double routines rounded to float, over all 2^32 arguments: exp never
// differs, erf for two of them (in the last bit).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <utility>

namespace b200
{
    namespace rounded
    {
        // e^x for x >= 0 by its Taylor series
        constexpr double exp_series(double x)
        {
            double term = 1.0, sum = 1.0;
            for (int n = 1; n < 90 && term > 1e-19 * sum; ++n)
            {
                term *= x / n;
                sum += term;
            }
            return sum;
        }
        // erf(x) for x >= 0: (2 / sqrt(pi)) e^(-x^2) sum_n 2^n x^(2n+1) / (1 3 5 ... (2n+1))
        constexpr double TWO_OVER_SQRT_PI = 1.1283791670955125739;
        constexpr double erf_series(double x)
        {
            double term = x, sum = x;
            for (int n = 1; n < 110 && term > 1e-19 * sum; ++n)
            {
                term *= 2.0 * x * x / (2 * n + 1);
                sum += term;
            }
            return TWO_OVER_SQRT_PI * sum / exp_series(x * x);
        }
        constexpr double LN2 = 0.69314718055994530942, LN2_LOW = 2.3190468138462996e-17; // ln 2 as the sum of two doubles

        constexpr int EXP_STEPS = 16 /* one double per pair of banks: lookups never conflict */, ERF_STEPS = 256, ERF_ENTRIES = 4 * ERF_STEPS + 1;
        struct ErfPoint
        {
            double e, d; // erf(g) and its derivative there
        };
        struct ExpTable
        {
            double v[EXP_STEPS];
        };
        struct ErfTable
        {
            ErfPoint v[ERF_ENTRIES];
        };
        // one constant expression per entry: a whole table at once exceeds the front end's evaluation limit
        template <int J>
        struct ExpEntry
        {
            static constexpr double v = exp_series(LN2 * J / EXP_STEPS);
        };
        template <int J>
        struct ErfEntry
        {
            static constexpr double g = double(J) / ERF_STEPS;
            static constexpr ErfPoint v{erf_series(g), TWO_OVER_SQRT_PI / exp_series(g * g)};
        };
        template <int... J>
        constexpr ExpTable make_exp_table(std::integer_sequence<int, J...>)
        {
            return ExpTable{{ExpEntry<J>::v...}};
        }
        template <int... J>
        constexpr ErfTable make_erf_table(std::integer_sequence<int, J...>)
        {
            return ErfTable{{ErfEntry<J>::v...}};
        }
        static __device__ const ExpTable g_exp_table = make_exp_table(std::make_integer_sequence<int, EXP_STEPS>());
        static __device__ const ErfTable g_erf_table = make_erf_table(std::make_integer_sequence<int, ERF_ENTRIES>());

        // Kernels call these with every thread of the block, then synchronise.
        __device__ __forceinline__ void load_exp_table(double* shared)
        {
            for (int i = threadIdx.x; i < EXP_STEPS; i += blockDim.x)
                shared[i] = g_exp_table.v[i];
        }
        __device__ __forceinline__ void load_erf_table(ErfPoint* shared)
        {
            for (int i = threadIdx.x; i < ERF_ENTRIES; i += blockDim.x)
                shared[i] = g_erf_table.v[i];
        }

        constexpr double ROUND_MAGIC = 6755399441055744.0; // 1.5 * 2^52: adding it rounds to an integer in the low word

        __device__ __forceinline__ float exp_rounded(float x, const double* table)
        {
            // beyond these the result is 0 or infinity like theirs; a NaN stays
            x = x < -110.0f ? -110.0f : x;
            x = x > 110.0f ? 110.0f : x;
            const double xd = x, m = fma(xd, EXP_STEPS / LN2, ROUND_MAGIC), k = m - ROUND_MAGIC;
            const int ki = __double2loint(m);
            const double t = table[ki & (EXP_STEPS - 1)];
            double r = fma(k, -LN2 / EXP_STEPS, xd);
            r = fma(k, -LN2_LOW / EXP_STEPS, r);
            double p = fma(r, 1.0 / 720.0, 1.0 / 120.0);
            p = fma(p, r, 1.0 / 24.0);
            p = fma(p, r, 1.0 / 6.0);
            p = fma(p, r, 0.5);
            p = fma(p, r * r, r);
            p = fma(t, p, t);
            return static_cast<float>(__hiloint2double(__double2hiint(p) + ((ki >> 4) << 20), __double2loint(p)));
        }

        // erf of |x| (arguments beyond 4 are taken as 4, whose result is 1; so is a NaN)
        __device__ __forceinline__ float erf_abs(float a, const ErfPoint* table)
        {
            a = fminf(a, 4.0f);
            constexpr float magic = 12582912.0f; // 1.5 * 2^23
            const float jm = __fmaf_rn(a, float(ERF_STEPS), magic), gf = __fmul_rn(__fsub_rn(jm, magic), 1.0f / ERF_STEPS);
            const ErfPoint t = table[__float_as_int(jm) & 2047];
            // the terms of d^4 and d^5 weigh less than 2^-27 of the result: single precision is enough for them
            const float df = __fsub_rn(a, gf), gf2 = gf * gf; // df is exact
            const float c4 = gf * fmaf(gf2, -1.0f / 3.0f, 0.5f), c5 = fmaf(gf2, fmaf(gf2, 2.0f / 15.0f, -0.4f), 0.1f);
            const double g = gf, d = df, c3 = fma(g * g, 2.0 / 3.0, -1.0 / 3.0);
            const double u = fma(d, fma(d, double(fmaf(df, c5, c4)), c3), -g);
            return static_cast<float>(fma(t.d, fma(d * d, u, d), t.e));
        }
        __device__ __forceinline__ float erf_rounded(float x, const ErfPoint* table)
        {
            return x == x ? copysignf(erf_abs(fabsf(x), table), x) : x;
        }
    }
}
