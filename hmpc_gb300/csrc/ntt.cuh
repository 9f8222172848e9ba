// What feeds stage 0 of a forward transform, and the twiddle load.
//
// The samplers draw inside the transform's first stage: one generator per
// stage-0 pair, the lower element's value first
// (hmpc/expr/number_theoretic_transform.hpp:316-329).
#pragma once

#include <cstdint>

#include "chacha.cuh"
#include "limbs.cuh"

namespace hmpc_gb300
{
    enum ProducerKind : int
    {
        producer_tensor = 0,   // read `src` (or the output buffer when src == nullptr)
        producer_cbd = 1,      // centred binomial, 2V = vx2, NW words per sample
        producer_uniform = 2,  // uniform mod Q, W words per sample
        producer_parts = 3,    // the parts of an encryption or key pair (PairParts)
    };

    // One polynomial of a batch of independent requests: its RNG (the request's
    // nonce, the polynomial's index in the request and the request's polynomial
    // count), and where its coefficients are in the request's own buffers, limb
    // planes `stride` words apart.
    struct PolyRequest
    {
        uint32_t nonce[3];
        uint32_t index, count;
        const uint32_t* in;
        uint32_t* out[2];
        uint64_t stride;
    };

    // Generator key, nonce and counter of the stage-0 pair whose first element
    // is coefficient idx_u of polynomial `poly`.  With p.requests, polynomial i
    // draws with nonce = requests[i].nonce + slot * count * N and counter = index
    // * N + coefficient -- exactly what the request would draw alone with its own
    // nonce.
    template<class Params>
    __device__ __forceinline__ uint32_t pair_generator(const Params& p, uint64_t poly, uint64_t idx_u, uint32_t slot,
                                                       RngKey& rng)
    {
        rng = p.rng;
        if (p.requests)
        {
            const PolyRequest& d = p.requests[poly];
            const uint64_t add = static_cast<uint64_t>(slot) * d.count << p.log_n;
            uint64_t s = static_cast<uint64_t>(d.nonce[0]) + static_cast<uint32_t>(add);
            rng.nonce[0] = static_cast<uint32_t>(s);
            s = static_cast<uint64_t>(d.nonce[1]) + static_cast<uint32_t>(add >> 32) + (s >> 32);
            rng.nonce[1] = static_cast<uint32_t>(s);
            rng.nonce[2] = d.nonce[2] + static_cast<uint32_t>(s >> 32);
            return static_cast<uint32_t>((static_cast<uint64_t>(d.index) << p.log_n) + idx_u);
        }
        return static_cast<uint32_t>(poly * (1ull << p.log_n) + idx_u);
    }

    template<int L, int Kind, int NW, class Params>
    __device__ __forceinline__ void produce_pair(const Params& p, const Modulus<L>& m, uint64_t poly,
                                                 uint64_t idx_u, uint32_t (&u)[L], uint32_t (&v)[L])
    {
        if constexpr (Kind == producer_cbd)
        {
            // one generator per pair, counter = low word of the first element's
            // linear index; u draws first, v next (number_theoretic_transform.hpp
            // :316-329, comp/queue.hpp:191-212)
            uint32_t w[2 * NW];
            RngKey rng;
            const uint32_t counter = pair_generator(p, poly, idx_u, p.rng_slot, rng);
            chacha_stream<2 * NW>(rng, counter, w);
            int a = 0, b = 0;
            const int count = 2 * static_cast<int>(p.vx2);
#pragma unroll
            for (int i = 0; i < NW; ++i)
            {
                uint32_t mask = 0xffffffffu;
                if (i == NW - 1 && (count & 31))
                {
                    mask = (1u << (count & 31)) - 1u;
                }
                a += __popc(w[i] & mask);
                b += __popc(w[NW + i] & mask);
            }
            small_to_mont<L>(u, a - static_cast<int>(p.vx2), p.small_table, m);
            small_to_mont<L>(v, b - static_cast<int>(p.vx2), p.small_table, m);
        }
        else if constexpr (Kind == producer_uniform)
        {
            uint32_t w[2 * NW];
            RngKey rng;
            const uint32_t counter = pair_generator(p, poly, idx_u, p.rng_slot, rng);
            chacha_stream<2 * NW>(rng, counter, w);
            uniform_from_words<L, NW, 0, 2 * NW>(u, w, p.top_mask, m);
            uniform_from_words<L, NW, NW, 2 * NW>(v, w, p.top_mask, m);
        }
    }

    template<int L>
    __device__ __forceinline__ void load_twiddle(uint32_t (&t)[L], const uint32_t* table, uint32_t index)
    {
        const uint32_t* ptr = table + static_cast<size_t>(index) * L;
        if constexpr (L % 4 == 0)
        {
#pragma unroll
            for (int j = 0; j < L; j += 4)
            {
                const uint4 v = __ldg(reinterpret_cast<const uint4*>(ptr + j));
                t[j] = v.x;
                t[j + 1] = v.y;
                t[j + 2] = v.z;
                t[j + 3] = v.w;
            }
        }
        else if constexpr (L % 2 == 0)
        {
#pragma unroll
            for (int j = 0; j < L; j += 2)
            {
                const uint2 v = __ldg(reinterpret_cast<const uint2*>(ptr + j));
                t[j] = v.x;
                t[j + 1] = v.y;
            }
        }
        else
        {
#pragma unroll
            for (int j = 0; j < L; ++j)
            {
                t[j] = __ldg(ptr + j);
            }
        }
    }
}
