// Negacyclic NTT / INTT passes with one butterfly per thread and stage.
//
// Semantics are those of hmpc's stage-per-kernel transform
// (hmpc/expr/number_theoretic_transform.hpp:90-197,262-549):
//   forward stage s: length = 2^s, the lower element idx of a pair takes
//     psi = T[2^s + (idx >> (n - s))]; v *= psi; (u+v, u-v)
//   inverse stage s: psi = T[N/2^(s+1) + (idx >> (s+1))]; (u+v, (u-v)*psi); the
//     last stage multiplies u+v by T[0] = N^-1 and u-v by T[1]
//
// A pass covers w consecutive stages; the w element-index bits they touch are
// the rows of a tile, 2^c consecutive lower indices its columns (coalescing).
// A tile is 2^(w+c-1) threads, each holding the two elements of a butterfly.
// Between stages a thread keeps one of its two elements and trades the other
// with the thread whose index differs in one bit: by shuffles when that bit
// lies in the warp, through shared memory otherwise.
//
// Bound by the wide multiply-adds of the butterflies' products where the
// polynomials fill the SMs (256 of 2^15 at 8 limbs: 1154 us, 0.76 of the
// product rate), by the latency of the stages where they do not.  One
// butterfly per thread and one copy of the product's code in the stage loop:
// holding 8 elements in registers and unrolling three stages of butterflies
// touches shared memory a third as often, which the products hide anyway,
// but left a small transform with a quarter of the warps and about 150 KB of
// straight-line code to fetch.  Against that form, tuned: one polynomial of
// 2^15 at 8 limbs 55.8 -> 15.0 us, 3 of 2^13 49.2 -> 12.7, 33 of 2^14 at 6
// limbs 71 -> 54, 256 of 2^15 at 8 limbs 1334 -> 1154.
#pragma once

#include <cstdint>

#include "chacha.cuh"
#include "cast.cuh"
#include "elementwise.cuh"
#include "limbs.cuh"
#include "ntt.cuh"

namespace hmpc_gb300
{
    constexpr uint32_t pair_max_threads = 512;

    // Sampled transforms that run as one: part i is the polynomials
    // [i * polys, (i + 1) * polys) of the pass and has an output buffer of its
    // own.
    constexpr int pair_max_parts = 3;

    enum PairPartKind : uint32_t
    {
        part_ternary = 0,        // CBD(1/2)
        part_scaled = 1,         // p * CBD(10)
        part_scaled_message = 2, // p * CBD(10) + the centred lift of a residue mod p (one or two limbs)
    };

    struct PairParts
    {
        uint32_t kind[pair_max_parts];
        uint32_t nonce[pair_max_parts][3];
        const uint32_t* msg;           // msg_limbs planes of `elements` words, Montgomery form (nullptr: the
                                       // requests' inputs)
        uint32_t msg_limbs;
        uint32_t pq[2], phalf[2], pninv;
        uint32_t r2[9];                // R^2 mod Q
    };

    struct PairPassParams
    {
        uint32_t* out[pair_max_parts]; // per part: limb-planar, `elements` entries per limb
        uint64_t part_polys;           // polynomials of a part
        const uint32_t* src;           // tensor producer input (nullptr: read out)
        const uint32_t* twiddles;      // element-major [N][L]
        const uint32_t* small_table;   // Montgomery forms of 0..64, element-major
        uint64_t elements;             // of one part: polynomials * N
        uint64_t tiles;                // of all parts: polynomials * tiles per polynomial
        uint32_t log_n;
        uint32_t w, c;                 // stages of this pass, column bits
        uint32_t row_shift;            // element bit of the lowest row bit
        RngKey rng;
        uint32_t vx2;                  // 2V for the CBD producer
        uint32_t top_mask;             // uniform producer: mask of the top word
        const PolyRequest* requests;   // one per polynomial of a part (nullptr: none)
        uint32_t rng_slot;
        uint32_t dependent;            // host side: programmatic dependence on the kernel before
        PairParts parts;               // parts producer
    };

    // Canonical value of a residue mod p (one or two limbs, Montgomery form)
    // lifted to the centred integer in (-p/2, p/2] (hmpc/ints/mod.hpp:259-307).
    __device__ __forceinline__ int64_t centred_lift(const PairParts& p, uint32_t m0, uint32_t m1)
    {
        const uint64_t q = p.pq[0] | static_cast<uint64_t>(p.pq[1]) << 32;
        const uint64_t half = p.phalf[0] | static_cast<uint64_t>(p.phalf[1]) << 32;
        uint64_t v;
        if (p.msg_limbs > 1)
        {
            unsigned __int128 t = (static_cast<uint64_t>(m1) << 32) | m0;
            t += static_cast<unsigned __int128>(m0 * p.pninv) * q;  // the low word becomes 0
            t >>= 32;
            t += static_cast<unsigned __int128>(static_cast<uint32_t>(t) * p.pninv) * q;
            t >>= 32;  // < 2q
            v = static_cast<uint64_t>(t);
            v = (t >> 64) != 0 || v >= q ? v - q : v;
        }
        else
        {
            v = (static_cast<uint64_t>(m0 * p.pninv) * p.pq[0] + m0) >> 32;  // <= q
            v = v >= q ? v - q : v;
        }
        return v > half ? static_cast<int64_t>(v) - static_cast<int64_t>(q) : static_cast<int64_t>(v);
    }

    // r = x mod Q in Montgomery form, |x| < 2^70 < Q
    template<int L>
    __device__ __forceinline__ void int_to_mont(uint32_t (&r)[L], __int128 x, const uint32_t* r2, const Modulus<L>& m)
    {
        const bool negative = x < 0;
        const unsigned __int128 a = static_cast<unsigned __int128>(negative ? -x : x);
        uint32_t v[L], f[L];
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            v[j] = j < 3 ? static_cast<uint32_t>(a >> (32 * (j < 3 ? j : 0))) : 0u;
            f[j] = r2[j];
        }
        mont_mul<L>(r, f, v, m);
        if (negative)
        {
            mod_neg<L>(r, r, m);
        }
    }

    // The stage-0 pair of a part: one generator, the lower element's draw first
    // (number_theoretic_transform.hpp:316-329).  Both variances of BGV's
    // samplers consume words 0 and 1 or 0 to 3 of one block.
    template<int L>
    __device__ __forceinline__ void produce_part_pair(const PairPassParams& p, const Modulus<L>& m, uint32_t part,
                                                      uint64_t poly, uint32_t idx, uint32_t step, uint32_t (&u)[L],
                                                      uint32_t (&v)[L])
    {
        const uint32_t kind = p.parts.kind[part];
        uint32_t msg[2][2] = {};
        if (kind == part_scaled_message)
        {
            // issued before the keystream is computed: their latency hides behind it
            const uint32_t* at = p.parts.msg ? p.parts.msg + (poly << p.log_n) : p.requests[poly].in;
            const uint64_t plane = p.parts.msg ? p.elements : p.requests[poly].stride;
            at += idx;
            msg[0][0] = at[0];
            msg[1][0] = at[step];
            if (p.parts.msg_limbs > 1)
            {
                msg[0][1] = at[plane];
                msg[1][1] = at[plane + step];
            }
        }
        RngKey rng;
        const uint32_t counter = pair_generator(p, poly, idx, part, rng);
        if (!p.requests)
        {
            rng.nonce[0] = p.parts.nonce[part][0];
            rng.nonce[1] = p.parts.nonce[part][1];
            rng.nonce[2] = p.parts.nonce[part][2];
        }
        uint32_t w[4];
        chacha_stream<4>(rng, counter, w);
        if (kind == part_ternary)
        {
            small_to_mont<L>(u, __popc(w[0] & 3u) - 1, p.small_table, m);
            small_to_mont<L>(v, __popc(w[1] & 3u) - 1, p.small_table, m);
            return;
        }
        const uint64_t scale = p.parts.pq[0] | static_cast<uint64_t>(p.parts.pq[1]) << 32;
        __int128 x = static_cast<__int128>(scale) * (__popc(w[0]) + __popc(w[1] & 0xffu) - 20);
        __int128 y = static_cast<__int128>(scale) * (__popc(w[2]) + __popc(w[3] & 0xffu) - 20);
        if (kind == part_scaled_message)
        {
            x += centred_lift(p.parts, msg[0][0], msg[0][1]);
            y += centred_lift(p.parts, msg[1][0], msg[1][1]);
        }
        int_to_mont<L>(u, x, p.parts.r2, m);
        int_to_mont<L>(v, y, p.parts.r2, m);
    }

    // A thread's place in a tile.  Stage j of the pass pairs row bit w-1-j
    // (forward) or j (inverse).  The thread bits above that one stand for the
    // row bits above it, one to one, so both the twiddle and the rows follow from
    // r by shifts.
    struct PairTile
    {
        uint32_t w, c;
        uint32_t r;             // the row bits but the pair's
        uint32_t twiddle_high;  // from the index bits above the rows
        uint32_t* buffer;       // the exchange buffers, taking turns
        uint32_t* other;

        template<bool Inverse>
        __device__ __forceinline__ uint32_t twiddle_index(uint32_t j) const
        {
            return Inverse ? (twiddle_high << (w - 1 - j)) + (r >> j) : (twiddle_high << j) + (r >> (w - 1 - j));
        }
    };

    // The stages of a pass on the pair (lo, hi), tw the first stage's twiddle; by
    // every thread of the block.  last: the inverse transform's last stage is the
    // pass's last.
    // W: the pass's stages where the loop is unrolled, 0: as many as the tile says.
    template<int L, bool Inverse, int W>
    __device__ __forceinline__ void pair_stage_loop(uint32_t (&lo)[L], uint32_t (&hi)[L], uint32_t (&tw)[L],
                                                PairTile& tile, const uint32_t* twiddles, bool last,
                                                const Modulus<L>& m)
    {
        const uint32_t t = threadIdx.x;
        const uint32_t w = W ? W : tile.w;
#pragma unroll(W ? W : 1)
        for (uint32_t j = 0; j < w; ++j)
        {
            if (j > 0)
            {
                const uint32_t bit = tile.c + (Inverse ? j - 1 : w - 1 - j);
                const bool upper = (t >> bit) & 1u;
                if (bit < 5)
                {
#pragma unroll
                    for (int k = 0; k < L; ++k)
                    {
                        const uint32_t v = __shfl_xor_sync(0xffffffffu, upper ? lo[k] : hi[k], 1 << bit);
                        lo[k] = upper ? v : lo[k];
                        hi[k] = upper ? hi[k] : v;
                    }
                }
                else
                {
#pragma unroll
                    for (int k = 0; k < L; ++k)
                    {
                        tile.buffer[k * blockDim.x + t] = upper ? lo[k] : hi[k];
                    }
                    __syncthreads();
#pragma unroll
                    for (int k = 0; k < L; ++k)
                    {
                        const uint32_t v = tile.buffer[k * blockDim.x + (t ^ (1u << bit))];
                        lo[k] = upper ? v : lo[k];
                        hi[k] = upper ? hi[k] : v;
                    }
                    // the next exchange writes the other buffer: a thread gets
                    // there only after this barrier's readers of it are done
                    uint32_t* swap = tile.buffer;
                    tile.buffer = tile.other;
                    tile.other = swap;
                }
            }
            uint32_t next[L];
            load_twiddle<L>(next, twiddles, tile.twiddle_index<Inverse>(j + 1 < w ? j + 1 : j));
            if constexpr (!Inverse)
            {
                mont_mul<L>(hi, hi, tw, m);
                uint32_t sum[L];
                mod_add<L>(sum, lo, hi, m);
                mod_sub<L>(hi, lo, hi, m);
#pragma unroll
                for (int k = 0; k < L; ++k)
                {
                    lo[k] = sum[k];
                }
            }
            else
            {
                uint32_t sum[L];
                mod_add<L>(sum, lo, hi, m);
                mod_sub<L>(hi, lo, hi, m);
#pragma unroll
                for (int k = 0; k < L; ++k)
                {
                    lo[k] = sum[k];
                }
                if (last && j == w - 1)
                {
                    // the transform's last stage: tw is T[1], and u + v takes T[0] = N^-1
                    uint32_t scale[L];
                    load_twiddle<L>(scale, twiddles, 0u);
                    mont_mul<L>(lo, lo, scale, m);
                }
                mont_mul<L>(hi, hi, tw, m);
            }
#pragma unroll
            for (int k = 0; k < L; ++k)
            {
                tw[k] = next[k];
            }
        }
    }

    // One and two limbs: the stages' own code, their indices and exchanges, takes
    // more of the issue slots (80 % busy) than the products, so the loop is
    // unrolled, one copy for each number of stages.  128 of 2^15, forward and
    // inverse: 73 and 83 us -> 60 and 62 at one limb, 117 and 124 -> 107 and 108 at
    // two.  With more limbs the products hide that code, and copies of them would
    // outgrow the instruction cache.
    template<int L, bool Inverse>
    __device__ __forceinline__ void pair_stages(uint32_t (&lo)[L], uint32_t (&hi)[L], uint32_t (&tw)[L],
                                                PairTile& tile, const uint32_t* twiddles, bool last,
                                                const Modulus<L>& m)
    {
        if constexpr (L <= 2)
        {
            switch (tile.w)
            {
            case 3: return pair_stage_loop<L, Inverse, 3>(lo, hi, tw, tile, twiddles, last, m);
            case 4: return pair_stage_loop<L, Inverse, 4>(lo, hi, tw, tile, twiddles, last, m);
            case 5: return pair_stage_loop<L, Inverse, 5>(lo, hi, tw, tile, twiddles, last, m);
            case 6: return pair_stage_loop<L, Inverse, 6>(lo, hi, tw, tile, twiddles, last, m);
            case 7: return pair_stage_loop<L, Inverse, 7>(lo, hi, tw, tile, twiddles, last, m);
            case 8: return pair_stage_loop<L, Inverse, 8>(lo, hi, tw, tile, twiddles, last, m);
            case 9: return pair_stage_loop<L, Inverse, 9>(lo, hi, tw, tile, twiddles, last, m);
            case 10: return pair_stage_loop<L, Inverse, 10>(lo, hi, tw, tile, twiddles, last, m);
            default: break;
            }
        }
        pair_stage_loop<L, Inverse, 0>(lo, hi, tw, tile, twiddles, last, m);
    }

    // One pass over the tiles of block `block` of the pass's grid.  exchange
    // holds [2][L][blockDim.x] words.  load and store take the polynomial (within
    // its part), the index of the lower element of the thread's pair, the
    // distance to the upper one, and the pair.  Wait: whether the input may
    // still be being written by the kernel before this one in the stream.
    // after runs between the stages and the store, in every thread.
    template<int L, bool Inverse, bool Wait, class Load, class After, class Store>
    __device__ __forceinline__ void ntt_pair_process(const PairPassParams& p, const Modulus<L>& m, uint64_t block,
                                                     uint32_t* exchange, Load&& load, After&& after, Store&& store)
    {
        const uint32_t t = threadIdx.x;
        const uint32_t w = p.w, c = p.c;
        const uint32_t pair_bits = w + c - 1;
        const uint64_t number = block * (blockDim.x >> pair_bits) + (t >> pair_bits);
        const bool active = number < p.tiles;
        const uint32_t col = t & ((1u << c) - 1u);
        const uint32_t r = (t >> c) & ((1u << (w - 1)) - 1u);  // the row bits but the pair's
        const uint32_t tile_bits = p.log_n - w - c;
        uint64_t poly = number >> tile_bits;
        uint32_t part = 0;
#pragma unroll
        for (int i = 1; i < pair_max_parts; ++i)
        {
            if (poly >= p.part_polys)
            {
                poly -= p.part_polys;
                ++part;
            }
        }
        const uint32_t in_poly = static_cast<uint32_t>(number) & ((1u << tile_bits) - 1u);
        const uint32_t mid_bits = p.row_shift - c;
        const uint32_t high = in_poly >> mid_bits;  // index bits above the rows
        const uint32_t base = (high << (p.row_shift + w)) | ((in_poly & ((1u << mid_bits) - 1u)) << c) | col;
        PairTile tile{w, c, r, (1u << (p.log_n - p.row_shift - w)) + high, exchange, exchange + L * blockDim.x};
        uint32_t lo[L], hi[L], tw[L];
        load_twiddle<L>(tw, p.twiddles, tile.twiddle_index<Inverse>(0));
        if constexpr (Wait)
        {
            asm volatile("griddepcontrol.wait;" ::: "memory");
        }
        {
            const uint32_t row = Inverse ? r << 1 : r;
            const uint32_t idx = base | (row << p.row_shift);
            const uint32_t step = 1u << (p.row_shift + (Inverse ? 0u : w - 1));
            if (active)
            {
                load(part, poly, idx, step, lo, hi);
            }
            else
            {
                set_zero<L>(lo);
                set_zero<L>(hi);
            }
        }
        pair_stages<L, Inverse>(lo, hi, tw, tile, p.twiddles, p.row_shift + w == p.log_n, m);
        after(tile, lo, hi);
        // The next kernel's blocks may come in from here on.  Let in at this pass's
        // start they hold slots and issue while they wait: one 4096 pair 13.9 us,
        // a key pair of 2^15 25.4, decryption of 33 x 2^14 81.5; so 12.3, 23.5 and
        // 79.6.
        if constexpr (Wait)
        {
            asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
        }
        if (active)
        {
            const uint32_t row = Inverse ? r : r << 1;
            const uint32_t step = 1u << (p.row_shift + (Inverse ? w - 1 : 0u));
            store(part, poly, base | (row << p.row_shift), step, lo, hi);
        }
    }

    // the pass's own input (tensor or sampler) and output
    template<int L, int Kind, int NW, bool Inverse, bool Wait>
    __device__ __forceinline__ void ntt_pair_pass(const PairPassParams& p, const Modulus<L>& m, uint64_t block,
                                                  uint32_t* exchange)
    {
        ntt_pair_process<L, Inverse, Wait>(
            p, m, block, exchange,
            [&](uint32_t part, uint64_t poly, uint32_t idx, uint32_t step, uint32_t (&lo)[L], uint32_t (&hi)[L]) {
                if constexpr (Kind == producer_parts)
                {
                    produce_part_pair<L>(p, m, part, poly, idx, step, lo, hi);
                }
                else if constexpr (Kind != producer_tensor)
                {
                    produce_pair<L, Kind, NW>(p, m, poly, idx, lo, hi);
                }
                else
                {
                    const uint32_t* in = (p.src ? p.src : p.out[part]) + (poly << p.log_n) + idx;
                    load1<L>(lo, in, p.elements, 0);
                    load1<L>(hi, in + step, p.elements, 0);
                }
            },
            [](PairTile&, const uint32_t (&)[L], const uint32_t (&)[L]) {},
            [&](uint32_t part, uint64_t poly, uint32_t idx, uint32_t step, const uint32_t (&lo)[L],
                const uint32_t (&hi)[L]) {
                uint32_t* out = p.out[part] + (poly << p.log_n) + idx;
                store1<L>(out, p.elements, 0, lo);
                store1<L>(out + step, p.elements, 0, hi);
            });
    }

    // 64 registers at most (two blocks of 512 threads): at 8 limbs the inverse pass
    // would take 72 and leave a second wave to batches that just fill the SMs (12
    // of 2^13: 36.7 -> 25.0 us).  The parts' first pass, whose loads and keystream
    // want more, stays without: 3 encryptions of 2^13 20.8 us, 23.9 with the limit.
    template<int L, int Kind, int NW, bool Inverse>
    __global__ void __launch_bounds__(pair_max_threads, Kind == producer_parts ? 1 : 2)
        ntt_pair_kernel(const PairPassParams p, const Modulus<L> m)
    {
        extern __shared__ uint32_t exchange[];
        ntt_pair_pass<L, Kind, NW, Inverse, true>(p, m, blockIdx.x, exchange);
    }

    // Forward passes over the requests' own buffers: the first reads their
    // inputs, every one writes their outputs.
    template<int L, bool First>
    __global__ void __launch_bounds__(pair_max_threads, 2) ntt_request_kernel(const PairPassParams p,
                                                                              const Modulus<L> m)
    {
        extern __shared__ uint32_t exchange[];
        ntt_pair_process<L, false, true>(
            p, m, blockIdx.x, exchange,
            [&](uint32_t, uint64_t poly, uint32_t idx, uint32_t step, uint32_t (&lo)[L], uint32_t (&hi)[L]) {
                const PolyRequest& d = p.requests[poly];
                const uint32_t* in = (First ? d.in : d.out[0]) + idx;
                load1<L>(lo, in, d.stride, 0);
                load1<L>(hi, in + step, d.stride, 0);
            },
            [](PairTile&, const uint32_t (&)[L], const uint32_t (&)[L]) {},
            [&](uint32_t, uint64_t poly, uint32_t idx, uint32_t step, const uint32_t (&lo)[L],
                const uint32_t (&hi)[L]) {
                const PolyRequest& d = p.requests[poly];
                store1<L>(d.out[0] + idx, d.stride, 0, lo);
                store1<L>(d.out[0] + idx + step, d.stride, 0, hi);
            });
    }

    // Decryption's inverse transform: the first pass forms its input c0 - s * c1
    // (s broadcast over the batch; hmpc/expr/crypto/lhe/dec.hpp:29) as it loads,
    // and the last pass lifts its result to the plaintext modulus (1 or 2 limbs)
    // before it stores -- for NTT-form plaintexts after the forward transform's
    // first pass mod p, which works on the same tiles: it starts on the pair bit
    // that the inverse transform ends on.
    struct DecryptParams
    {
        const uint32_t* s;   // [L][N]
        const uint32_t* c0;
        const uint32_t* c1;
        uint32_t* out;       // residues mod p, limb planes of `elements`
        CastParams cast;
        uint32_t p[2], pninv;
        const uint32_t* p_twiddles;  // NTT-form plaintexts: the forward table mod p
    };

    // LP: limbs of p in the last pass, 0 in the passes before it
    template<int L, bool First, int LP>
    __global__ void __launch_bounds__(pair_max_threads, 2) ntt_decrypt_kernel(const PairPassParams p,
                                                                              const DecryptParams d,
                                                                              const Modulus<L> m)
    {
        extern __shared__ uint32_t exchange[];
        uint32_t y[2][LP > 0 ? LP : 1];
        Modulus<(LP > 0 ? LP : 1)> to;
        ntt_pair_process<L, true, true>(
            p, m, blockIdx.x, exchange,
            [&](uint32_t, uint64_t poly, uint32_t idx, uint32_t step, uint32_t (&lo)[L], uint32_t (&hi)[L]) {
                const uint64_t at = (poly << p.log_n) + idx;
                if constexpr (First)
                {
                    auto combine = [&](uint32_t (&x)[L], uint32_t offset) {
                        uint32_t t[L];
                        load1<L>(x, d.s, 1ull << p.log_n, idx + offset);
                        load1<L>(t, d.c1, p.elements, at + offset);
                        mont_mul<L>(t, t, x, m);
                        load1<L>(x, d.c0, p.elements, at + offset);
                        mod_sub<L>(x, x, t, m);
                    };
                    combine(lo, 0);
                    combine(hi, step);
                }
                else
                {
                    load1<L>(lo, p.out[0], p.elements, at);
                    load1<L>(hi, p.out[0], p.elements, at + step);
                }
            },
            [&](PairTile& tile, const uint32_t (&lo)[L], const uint32_t (&hi)[L]) {
                if constexpr (LP > 0)
                {
#pragma unroll
                    for (int j = 0; j < LP; ++j)
                    {
                        to.q[j] = d.p[j];
                    }
                    to.ninv = d.pninv;
                    cast_value<LP, L>(y[0], lo, d.cast, to);
                    cast_value<LP, L>(y[1], hi, d.cast, to);
                    if (d.p_twiddles)
                    {
                        uint32_t tw[LP];
                        load_twiddle<LP>(tw, d.p_twiddles, tile.template twiddle_index<false>(0));
                        pair_stage_loop<LP, false, 0>(y[0], y[1], tw, tile, d.p_twiddles, false, to);
                    }
                }
            },
            [&](uint32_t, uint64_t poly, uint32_t idx, uint32_t step, const uint32_t (&lo)[L],
                const uint32_t (&hi)[L]) {
                uint64_t at = (poly << p.log_n) + idx;
                if constexpr (LP > 0)
                {
                    if (d.p_twiddles)
                    {
                        // rows 2r and 2r + 1 in place of r and r + 2^(w-1)
                        const uint32_t r = (threadIdx.x >> p.c) & ((1u << (p.w - 1)) - 1u);
                        at += static_cast<uint64_t>(r) << p.row_shift;
                        step = 1u << p.row_shift;
                    }
                    store1<LP>(d.out, p.elements, at, y[0]);
                    store1<LP>(d.out, p.elements, at + step, y[1]);
                }
                else
                {
                    store1<L>(p.out[0], p.elements, at, lo);
                    store1<L>(p.out[0], p.elements, at + step, hi);
                }
            });
    }

    // ----------------------------------------------------------------------
    // Persistent transform over a batch of polynomials of uneven degree.
    // Work items are (pass of one polynomial, CTA tile group) in a list that
    // holds every first-pass item before any later-pass item; CTAs take items
    // in list order from an atomic counter.  An item of pass k of a
    // polynomial waits until all earlier-pass items of that polynomial have
    // signalled.  Every item it waits for was taken earlier by a running CTA
    // that never waits on later items, so the waits end; they are still
    // bounded, and a wait that runs out sets `error` and the kernel returns.
    struct BatchedControl
    {
        uint32_t next;      // work counter
        uint32_t error;     // nonzero: a wait ran out (value = item + 1)
        uint32_t done;      // items finished
        uint32_t pad;
    };

    struct BatchedParams
    {
        const PairPassParams* params;   // one per (polynomial, pass)
        const uint32_t* item_param;     // item -> params index
        const uint32_t* item_tile;      // item -> CTA tile group inside that pass
        const uint32_t* item_wait;      // item -> signals needed before it may start (0: none)
        const uint32_t* item_poly;      // item -> polynomial (counter index)
        const uint32_t* item_signal;    // item -> 1 when it must signal its polynomial
        uint32_t* counters;             // per polynomial
        BatchedControl* control;
        uint32_t items;
        uint32_t spin_limit;            // polls of 64 ns before a wait gives up
    };

    __device__ __forceinline__ uint32_t load_acquire(const uint32_t* ptr)
    {
        uint32_t v;
        asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(ptr) : "memory");
        return v;
    }

    template<int L, bool Inverse>
    __global__ void __launch_bounds__(pair_max_threads, 2) ntt_batched_kernel(const BatchedParams bp, const Modulus<L> m)
    {
        extern __shared__ uint32_t exchange[];
        __shared__ uint32_t item_s;
        __shared__ uint32_t abort_s;
        for (;;)
        {
            if (threadIdx.x == 0)
            {
                uint32_t item = atomicAdd(&bp.control->next, 1u);
                uint32_t abort = 0;
                if (item < bp.items)
                {
                    const uint32_t need = bp.item_wait[item];
                    if (need)
                    {
                        const uint32_t* counter = bp.counters + bp.item_poly[item];
                        uint32_t polls = 0;
                        while (load_acquire(counter) < need)
                        {
                            if (++polls > bp.spin_limit || load_acquire(&bp.control->error))
                            {
                                atomicCAS(&bp.control->error, 0u, item + 1u);
                                abort = 1;
                                break;
                            }
                            __nanosleep(64);
                        }
                    }
                }
                item_s = item;
                abort_s = abort;
            }
            __syncthreads();
            const uint32_t item = item_s;
            const uint32_t abort = abort_s;
            __syncthreads();
            if (item >= bp.items || abort)
            {
                return;
            }
            const PairPassParams& p = bp.params[bp.item_param[item]];
            ntt_pair_pass<L, producer_tensor, 1, Inverse, false>(p, m, bp.item_tile[item], exchange);
            __syncthreads();
            if (threadIdx.x == 0)
            {
                if (bp.item_signal[item])
                {
                    __threadfence();
                    atomicAdd(bp.counters + bp.item_poly[item], 1u);
                }
                atomicAdd(&bp.control->done, 1u);
            }
        }
    }
}
