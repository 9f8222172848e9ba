// The last stages of a forward tensor-core transform, on the CUDA cores.
//
// On the tensor cores a group of stages with few index bits below it has one
// constant matrix per few elements (0.57 GB for the last three stages of 2^15
// coefficients at 8 limbs), a digit tile and an epilogue per matrix, and fills an
// SM's shared memory with one CTA whose nine warps wait on one another: 1001 us
// for 768 polynomials, a third of its HBM rate.  As butterflies the last w
// stages need w / 2 products per element, on a pipe the tensor-core groups
// leave idle.
//
// The groups before leave each value as biased base-256 digits of an integer
// congruent to the residue times 2^32 (the factor is in the constants of the
// group before this one): 4L + 2 balanced digits, so |v| < 1.01 * 2^(32L + 15).
// Adding a multiple of Q just above 2^(32L + 16) (and taking the digits' bias
// off: one constant) makes it positive and below 2^(32L + 17); one row of
// Montgomery reduction divides by 2^32 and leaves less than 2Q, for Q of at
// least 2^(32L - 15).
//
// A thread holds the two elements of a butterfly, as in pair.cuh; 2^(w-1) <= 32
// adjacent lanes share a tile of 2^w elements and trade by shuffles.
#pragma once

#include <cstdint>

#include "elementwise.cuh"
#include "limbs.cuh"
#include "ntt.cuh"

namespace hmpc_gb300
{
    struct TailParams
    {
        const uint32_t* digits;   // [L + 1][stride] words of four biased digits
        uint64_t stride;
        uint64_t elements;        // of one part
        uint64_t begin, end;      // the launch's elements of each part, whole tiles
        const uint32_t* twiddles;
        uint32_t log_n;
        uint32_t w;               // stages
        uint32_t offset[10];      // a multiple of Q minus the digits' bias, modulo 2^(32(L+1))
        uint32_t* out;            // plain: limb planes of `elements` words
        uint32_t* const* out_polys;  // or one buffer per polynomial
        const uint32_t* error;    // set by a group that gave up a wait, its digits incomplete
        // encryption: three parts u, x, w of `elements` each in the digit
        // planes; c0 = a * u + x, c1 = b * u + w
        const uint32_t* key_a;
        const uint32_t* key_b;
        uint32_t* c0;
        uint32_t* c1;
    };

    // Bound by the wide multiply-adds (their pipe 70 % busy): 1.5 products per
    // element at w = 3, and two more per ciphertext coefficient.  256 encryptions
    // of 2^15 at 8 limbs: 1050 us, against 1001 for the group on the tensor cores
    // and 355 for the combination after it.  24 warps per SM (80 registers, a few
    // spills) in blocks of 128: the encryption takes 2737 us, 2769 in blocks of
    // 256, 2765 at 32 warps, 2815 at 16.
    template<int L, bool Encrypt>
    __global__ void __launch_bounds__(128, 6) tc_tail_kernel(const TailParams p, const Modulus<L> m)
    {
        const uint32_t w = p.w;
        const uint64_t id = p.begin / 2 + static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
        const bool active = id < p.end / 2;
        const uint32_t r = static_cast<uint32_t>(id) & ((1u << (w - 1)) - 1u);
        const uint64_t first = (id >> (w - 1)) << w;  // the tile's first element
        const uint32_t coefficient = static_cast<uint32_t>(first) & ((1u << p.log_n) - 1u);
        const uint32_t twiddle_high = (1u << (p.log_n - w)) + (coefficient >> w);
        const uint32_t half_tile = 1u << (w - 1);
        uint32_t u[Encrypt ? 2 : 1][L];
        asm volatile("griddepcontrol.wait;" ::: "memory");
#pragma unroll 1
        for (uint32_t part = 0; part < (Encrypt ? 3u : 1u); ++part)
        {
            uint32_t x[2][L];
            const uint32_t gave_up = *p.error;  // on its way with the digits
#pragma unroll
            for (int k = 0; k < 2; ++k)
            {
                const uint32_t* d = p.digits + part * p.elements + first + r + k * half_tile;
                uint32_t v[L + 1];
#pragma unroll
                for (int j = 0; j < L + 1; ++j)
                {
                    v[j] = active ? d[static_cast<uint64_t>(j) * p.stride] : 0u;
                }
                v[0] = ptx::add_cc(v[0], p.offset[0]);
#pragma unroll
                for (int j = 1; j < L; ++j)
                {
                    v[j] = ptx::addc_cc(v[j], p.offset[j]);
                }
                v[L] = ptx::addc(v[L], p.offset[L]);
                redc<L, L + 1, 1>(x[k], v, m);
            }
            // Nothing is written from incomplete digits.  Looked at here, with the
            // digits, 256 encryptions take 10 us more than without; kept in a register
            // to the stores 90 us (spills).
            if (__any_sync(0xffffffffu, gave_up != 0))
            {
                return;
            }
#pragma unroll 1
            for (uint32_t j = 0; j < w; ++j)
            {
                uint32_t tw[L];
                load_twiddle<L>(tw, p.twiddles, (twiddle_high << j) + (r >> (w - 1 - j)));
                if (j > 0)
                {
                    const uint32_t bit = w - 1 - j;
                    const bool upper = (threadIdx.x >> bit) & 1u;
#pragma unroll
                    for (int k = 0; k < L; ++k)
                    {
                        const uint32_t v = __shfl_xor_sync(0xffffffffu, upper ? x[0][k] : x[1][k], 1 << bit);
                        x[0][k] = upper ? v : x[0][k];
                        x[1][k] = upper ? x[1][k] : v;
                    }
                }
                mont_mul<L>(x[1], x[1], tw, m);
                mod_add<L>(tw, x[0], x[1], m);
                mod_sub<L>(x[1], x[0], x[1], m);
#pragma unroll
                for (int k = 0; k < L; ++k)
                {
                    x[0][k] = tw[k];
                }
            }
            if (!active)
            {
                continue;
            }
            if constexpr (Encrypt)
            {
                if (part == 0)
                {
#pragma unroll
                    for (int k = 0; k < 2; ++k)
                    {
#pragma unroll
                        for (int j = 0; j < L; ++j)
                        {
                            u[k][j] = x[k][j];
                        }
                    }
                    continue;
                }
                const uint32_t* key = (part == 1 ? p.key_a : p.key_b) + coefficient + 2 * r;
                uint32_t* out = (part == 1 ? p.c0 : p.c1) + first + 2 * r;
#pragma unroll
                for (int k = 0; k < 2; ++k)
                {
                    uint32_t y[L];
                    load1<L>(y, key + k, 1ull << p.log_n, 0);
                    mont_mul<L>(y, y, u[k], m);
                    mod_add<L>(x[k], x[k], y, m);
                    store1<L>(out + k, p.elements, 0, x[k]);
                }
            }
            else
            {
                uint32_t* out = p.out_polys ? p.out_polys[first >> p.log_n] + coefficient : p.out + first;
                const uint64_t stride = p.out_polys ? 1ull << p.log_n : p.elements;
#pragma unroll
                for (int k = 0; k < 2; ++k)
                {
                    store1<L>(out + 2 * r + k, stride, 0, x[k]);
                }
            }
        }
    }
}
