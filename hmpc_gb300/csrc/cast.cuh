// Centred lift of residues between two moduli (hmpc/ints/mod.hpp:259-307):
// the source's canonical value v is shifted by `offset` when v > src/2 and is
// then converted into the target modulus as an unsigned integer -- directly
// (v*R^2, reduced) when it fits the target, otherwise with one reduction by
// R' = 2^(32 * words) followed by a product with R'*R^2 mod Q (mod.hpp:180-189).
//
// Both limb counts are compile-time values, so every value stays in registers
// (with a run-time source width they were arrays in local memory: 47 us for
// 33 * 2^14 residues from 6 limbs to 2).  Bound by HBM and the products.
#pragma once

#include <cstdint>

#include "elementwise.cuh"
#include "limbs.cuh"

namespace hmpc_gb300
{
    constexpr int max_device_limbs = 9;

    // constants of a centred lift from a source modulus into the target one
    // (hmpc/ints/mod.hpp:259-307)
    struct CastParams
    {
        uint32_t src_limbs;
        uint32_t src_ninv;
        uint32_t src_q[max_device_limbs];
        uint32_t src_half[max_device_limbs];
        uint32_t offset[max_device_limbs + 1];  // added when the value exceeds src/2
        uint32_t direct;                          // 1: value + offset < target Q
        uint32_t factor[max_device_limbs];        // R^2 (direct) or R'*R^2 mod Q
    };

    template<int L, int LS>
    __device__ __forceinline__ void cast_value(uint32_t (&y)[L], const uint32_t (&x)[LS], const CastParams& cp,
                                               const Modulus<L>& m)
    {
        constexpr int NW = (L > LS ? L : LS) + 1;  // words of value + offset
        Modulus<LS> src;
        uint32_t half[LS], f[L], v[LS], norm[NW];
#pragma unroll
        for (int j = 0; j < LS; ++j)
        {
            src.q[j] = cp.src_q[j];
            half[j] = cp.src_half[j];
        }
        src.ninv = cp.src_ninv;
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            f[j] = cp.factor[j];
        }
        redc<LS, LS>(v, x, src);
        const uint32_t mask = greater<LS>(v, half) ? 0xffffffffu : 0u;
        norm[0] = ptx::add_cc(v[0], cp.offset[0] & mask);
#pragma unroll
        for (int j = 1; j < NW; ++j)
        {
            norm[j] = ptx::addc_cc(j < LS ? v[j < LS ? j : 0] : 0u, cp.offset[j] & mask);
        }
        if (LS < L || (LS == L && cp.direct))
        {
#pragma unroll
            for (int j = 0; j < L; ++j)
            {
                y[j] = norm[j];
            }
        }
        else
        {
            redc<L, NW>(y, norm, m);
        }
        mont_mul<L>(y, f, y, m);
    }

    template<int L, int LS>
    __global__ void __launch_bounds__(256) cast_kernel(uint32_t* out, const uint32_t* in, uint64_t elements,
                                                       const CastParams cp, const Modulus<L> m)
    {
        for (uint64_t e = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; e < elements;
             e += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        {
            uint32_t x[LS], y[L];
            load1<LS>(x, in, elements, e);
            cast_value<L, LS>(y, x, cp, m);
            store1<L>(out, elements, e, y);
        }
    }
}
