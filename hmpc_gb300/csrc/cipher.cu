// ChaCha20 stream cipher over tensors (hmpc/expr/crypto/cipher.hpp:59-319,
// hmpc/crypto/cipher.hpp:29-44): element i's limbs are XORed with keystream
// words i*L .. i*L+L-1 of ChaCha20(key, nonce, counter from 0) -- the
// reference cuts the words into batches of lcm(16, L), starting batch b's
// generator at counter b * lcm(16, L) / 16, which is the same as word w using
// word w % 16 of block w / 16.  Encryption reads a limb-planar tensor and
// writes element-major words (the reference's [elements..., L] limb tensor);
// decryption is the reverse.
#include <cstdint>

#include "chacha.cuh"
#include "internal.hpp"

namespace
{
    using hmpc_gb300::RngKey;

    // Elements of a block of cipher_tile_kernel: 512 * L words are 32 * L
    // keystream blocks, one per thread.
    constexpr uint32_t tile_elements = 512;
    constexpr uint32_t tile_max_limbs = 16;  // 33 KB of shared memory, 512 threads
    constexpr uint32_t thread_words = 16;    // 512 * L words over 32 * L threads
    static_assert(tile_elements == 32 * thread_words, "one warp per limb plane, one keystream block per thread");

    __device__ __forceinline__ uint32_t padded(uint32_t w)
    {
        return w + (w >> 5);  // both the rows of a keystream block and strides of L words spread over the banks
    }

    // A tile's keystream goes through shared memory, so that the planes and
    // the element-major words are both read and written coalesced; the input
    // loads are issued before the keystream is computed.  Bound by the
    // keystream's integer arithmetic (one block of 16 words per thread).
    // 1,000,003 elements of 5 limbs: 27.5 us with a thread storing the 16 words
    // of its block one by one, 18.4 us so (4 limbs, 5,000,001: 84.8 and 58.4).
    __global__ void __launch_bounds__(32 * tile_max_limbs) cipher_tile_kernel(const RngKey rng, uint64_t elements,
                                                                              uint32_t limbs, const uint32_t* in,
                                                                              uint32_t* out, int decrypt)
    {
        extern __shared__ uint32_t tile[];
        const uint32_t t = threadIdx.x, lane = t & 31u;
        const uint64_t first = static_cast<uint64_t>(blockIdx.x) * tile_elements;
        const uint32_t count =
            elements - first < tile_elements ? static_cast<uint32_t>(elements - first) : tile_elements;
        const uint32_t words = count * limbs;
        // one warp per limb plane: its k-th access is element lane + 32 k; the
        // k-th element-major word of thread t is t + k * blockDim.x.  Both step
        // through the padded tile by 33 words per limb.
        const uint32_t step = 33 * limbs;
        const uint64_t plane = static_cast<uint64_t>(t >> 5) * elements + first + lane;
        const uint64_t flat = first * limbs + t;
        uint32_t* const at_plane = tile + padded(lane * limbs + (t >> 5));
        uint32_t* const at_flat = tile + padded(t);
        uint32_t data[thread_words];
#pragma unroll
        for (uint32_t k = 0; k < thread_words; ++k)
        {
            if (decrypt)
            {
                data[k] = t + k * blockDim.x < words ? in[flat + k * blockDim.x] : 0u;
            }
            else
            {
                data[k] = lane + 32 * k < count ? in[plane + 32 * k] : 0u;
            }
        }
        uint32_t ks[16];
        hmpc_gb300::chacha20_block(rng, static_cast<uint32_t>(first * limbs / 16 + t), ks);
        uint32_t* const at_block = tile + padded(16 * t);  // 16 words never cross a padding word
#pragma unroll
        for (uint32_t k = 0; k < 16; ++k)
        {
            at_block[k] = ks[k];
        }
        __syncthreads();
        if (decrypt)
        {
#pragma unroll
            for (uint32_t k = 0; k < thread_words; ++k)
            {
                at_flat[k * step] ^= data[k];
            }
            __syncthreads();
#pragma unroll
            for (uint32_t k = 0; k < thread_words; ++k)
            {
                if (lane + 32 * k < count)
                {
                    out[plane + 32 * k] = at_plane[k * step];
                }
            }
        }
        else
        {
#pragma unroll
            for (uint32_t k = 0; k < thread_words; ++k)
            {
                at_plane[k * step] ^= data[k];
            }
            __syncthreads();
#pragma unroll
            for (uint32_t k = 0; k < thread_words; ++k)
            {
                if (t + k * blockDim.x < words)
                {
                    out[flat + k * blockDim.x] = at_flat[k * step];
                }
            }
        }
    }

    // Any number of limbs (elements wider than a tile's shared memory): one
    // thread per keystream block, its 16 words read and written one by one.
    __global__ void __launch_bounds__(256) cipher_kernel(const RngKey rng, uint64_t elements, uint32_t limbs,
                                                         const uint32_t* in, uint32_t* out, int decrypt)
    {
        const uint64_t words = elements * limbs;
        const uint64_t blocks = (words + 15) / 16;
        for (uint64_t k = static_cast<uint64_t>(blockIdx.x) * blockDim.x + threadIdx.x; k < blocks;
             k += static_cast<uint64_t>(gridDim.x) * blockDim.x)
        {
            uint32_t ks[16];
            hmpc_gb300::chacha20_block(rng, static_cast<uint32_t>(k), ks);
            uint64_t w = k * 16;
            uint64_t i = w / limbs;
            uint32_t j = static_cast<uint32_t>(w - i * limbs);
#pragma unroll
            for (int t = 0; t < 16; ++t)
            {
                if (w + t < words)
                {
                    if (!decrypt)
                    {
                        out[w + t] = in[static_cast<uint64_t>(j) * elements + i] ^ ks[t];
                    }
                    else
                    {
                        out[static_cast<uint64_t>(j) * elements + i] = in[w + t] ^ ks[t];
                    }
                }
                if (++j == limbs)
                {
                    j = 0;
                    ++i;
                }
            }
        }
    }

    int run_cipher(hmpc_context* ctx, const uint32_t key[8], const uint32_t nonce[3], uint64_t elements,
                   int limbs, const uint32_t* in, uint32_t* out, int decrypt)
    {
        using namespace hmpc_gb300::detail;
        if (int rc = enter(ctx))
        {
            return rc;
        }
        if (!key || !nonce || limbs <= 0 || (elements && (!in || !out)))
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument or no limbs");
        }
        if (elements == 0)
        {
            return HMPC_OK;
        }
        const uint64_t blocks = (elements * static_cast<uint64_t>(limbs) + 15) / 16;
        if (blocks > (1ull << 32))
        {
            return fail(HMPC_ERROR_UNSUPPORTED, "more keystream blocks than the 32-bit block counter holds");
        }
        RngKey rng{};
        for (int i = 0; i < 8; ++i)
        {
            rng.key[i] = key[i];
        }
        for (int i = 0; i < 3; ++i)
        {
            rng.nonce[i] = nonce[i];
        }
        const uint64_t tiles = (elements + tile_elements - 1) / tile_elements;
        if (static_cast<uint32_t>(limbs) <= tile_max_limbs && tiles < (1ull << 31))
        {
            const uint32_t words = tile_elements * static_cast<uint32_t>(limbs);
            cipher_tile_kernel<<<static_cast<unsigned>(tiles), words / thread_words,
                                 (words + words / 32) * sizeof(uint32_t), ctx->stream>>>(
                rng, elements, static_cast<uint32_t>(limbs), in, out, decrypt);
        }
        else
        {
            const uint64_t grid = (blocks + 255) / 256;
            cipher_kernel<<<static_cast<unsigned>(grid < 152ull * 64 ? grid : 152ull * 64), 256, 0, ctx->stream>>>(
                rng, elements, static_cast<uint32_t>(limbs), in, out, decrypt);
        }
        const cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess)
        {
            return cuda_fail(e, "launching the cipher");
        }
        ++ctx->launches;
        return HMPC_OK;
    }
}

extern "C" {

int hmpc_cipher_enc(hmpc_context* ctx, const uint32_t key[8], const uint32_t nonce[3], uint64_t elements, int limbs,
                    const uint32_t* planar_in, uint32_t* flat_out)
{
    return run_cipher(ctx, key, nonce, elements, limbs, planar_in, flat_out, 0);
}

int hmpc_cipher_dec(hmpc_context* ctx, const uint32_t key[8], const uint32_t nonce[3], uint64_t elements, int limbs,
                    const uint32_t* flat_in, uint32_t* planar_out)
{
    return run_cipher(ctx, key, nonce, elements, limbs, flat_in, planar_out, 1);
}

}  // extern "C"
