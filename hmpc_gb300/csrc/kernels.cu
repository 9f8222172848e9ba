// Per-limb-count kernel instantiations and launchers.  Compiled once per L
// with -DHMPC_L=<L>; exports kernel_table_<L>().
#include <algorithm>
#include <type_traits>

#include "cast.cuh"
#include "dispatch.hpp"
#include "elementwise.cuh"
#include "linalg.cuh"
#include "ntt.cuh"
#include "pair.cuh"
#include "tail.cuh"

#ifndef HMPC_L
#error "compile with -DHMPC_L=<limbs>"
#endif

#define HMPC_CAT2(a, b) a##b
#define HMPC_CAT(a, b) HMPC_CAT2(a, b)

namespace hmpc_gb300
{
    namespace
    {
        constexpr int L = HMPC_L;

        Modulus<L> device_modulus(const HostModulus& h)
        {
            Modulus<L> m{};
            for (int j = 0; j < L; ++j)
            {
                m.q[j] = h.q[j];
                m.one[j] = h.one[j];
            }
            m.ninv = h.ninv;
            m.bits = static_cast<uint32_t>(h.bits);
            return m;
        }

        Modulus<L> holder(const uint32_t* words)
        {
            Modulus<L> m{};
            for (int j = 0; j < L; ++j)
            {
                m.one[j] = words[j];
            }
            return m;
        }

        unsigned grid_for(uint64_t work, unsigned block)
        {
            const uint64_t g = (work + block - 1) / block;
            return static_cast<unsigned>(std::max<uint64_t>(1, std::min<uint64_t>(g, 152ull * 64ull)));
        }

        // dependent: with programmatic dependence on the kernel before it in the
        // stream (the kernel waits for it by griddepcontrol.wait)
        template<class... Params, class... Args>
        cudaError_t launch(void (*kernel)(Params...), unsigned grid, unsigned block, size_t smem, bool dependent,
                           cudaStream_t stream, const Args&... args)
        {
            cudaLaunchConfig_t cfg{};
            cfg.gridDim = dim3(grid);
            cfg.blockDim = dim3(block);
            cfg.dynamicSmemBytes = smem;
            cfg.stream = stream;
            cudaLaunchAttribute attr[1];
            attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
            attr[0].val.programmaticStreamSerializationAllowed = 1;
            cfg.attrs = attr;
            cfg.numAttrs = dependent ? 1u : 0u;
            return cudaLaunchKernelEx(&cfg, kernel, args...);
        }

        template<int Kind, int NW, bool Inverse>
        cudaError_t launch_pair(const PairPassParams& p, const Modulus<L>& m, unsigned grid, unsigned block,
                                size_t smem, cudaStream_t stream)
        {
            return launch(ntt_pair_kernel<L, Kind, NW, Inverse>, grid, block, smem, p.dependent != 0, stream, p, m);
        }

        cudaError_t ntt_pair(const PairPassParams& p, int kind, int nw, bool inverse, const HostModulus& h,
                             unsigned grid, unsigned block, size_t smem, cudaStream_t stream)
        {
            const Modulus<L> m = device_modulus(h);
            if (inverse)
            {
                return launch_pair<producer_tensor, 1, true>(p, m, grid, block, smem, stream);
            }
            if (kind == producer_tensor)
            {
                return launch_pair<producer_tensor, 1, false>(p, m, grid, block, smem, stream);
            }
            if (kind == producer_cbd)
            {
                switch (nw)
                {
                case 1: return launch_pair<producer_cbd, 1, false>(p, m, grid, block, smem, stream);
                case 2: return launch_pair<producer_cbd, 2, false>(p, m, grid, block, smem, stream);
                case 3: return launch_pair<producer_cbd, 3, false>(p, m, grid, block, smem, stream);
                case 4: return launch_pair<producer_cbd, 4, false>(p, m, grid, block, smem, stream);
                default: return cudaErrorInvalidValue;
                }
            }
            if (kind == producer_parts)
            {
                return launch_pair<producer_parts, 1, false>(p, m, grid, block, smem, stream);
            }
            if (kind == producer_uniform && nw == L + 2)
            {
                return launch_pair<producer_uniform, L + 2, false>(p, m, grid, block, smem, stream);
            }
            if (kind == producer_uniform && nw == L + 3)
            {
                return launch_pair<producer_uniform, L + 3, false>(p, m, grid, block, smem, stream);
            }
            return cudaErrorInvalidValue;
        }

        cudaError_t fma(uint32_t* d, const uint32_t* a, const uint32_t* b, const uint32_t* c, uint64_t elements,
                        const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            // The widest access that the planes allow, up to two elements per
            // thread above 4 limbs, where four leave too few warps: 2^24
            // elements of 8 limbs 354.8 us with four, 313.3 with two, 356.3
            // with one; of 2 limbs 76.2, 75.9 and 86.1 and 1500008 of them 6.3,
            // 8.3 and 8.3.  Blocks of 128 threads there (8 limbs, two elements
            // per thread: 329.7 -> 313.3 us), of 256 below (6000000 elements of
            // one limb, two per thread: 16.4 -> 14.1 us).
            constexpr int widest = L <= 4 ? 4 : 2;
            constexpr unsigned block = L <= 4 ? 256 : 128;
            const uint64_t shape = reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) |
                                   reinterpret_cast<uintptr_t>(c) | reinterpret_cast<uintptr_t>(d) | elements * 4;
            auto launch = [&](auto width) {
                constexpr int V = decltype(width)::value;
                const uint64_t threads = elements / V;
                // only the kernel of single words loops
                const unsigned grid = L * V == 1 ? grid_for(threads, block)
                                                 : static_cast<unsigned>((threads + block - 1) / block);
                fma_kernel<L, V><<<grid, block, 0, stream>>>(d, a, b, c, elements, device_modulus(h));
            };
            if (shape % (4 * widest) == 0)
            {
                launch(std::integral_constant<int, widest>{});
            }
            else if (shape % 8 == 0)
            {
                launch(std::integral_constant<int, 2>{});
            }
            else
            {
                launch(std::integral_constant<int, 1>{});
            }
            return cudaGetLastError();
        }

        cudaError_t binary(uint32_t* out, const uint32_t* a, uint64_t a_elements, const uint32_t* b,
                           uint64_t b_elements, uint64_t elements, int op, const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            binary_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(out, a, a_elements, b, b_elements,
                                                                          elements, op, device_modulus(h));
            return cudaGetLastError();
        }

        cudaError_t lhe_combine(uint32_t* out, const uint32_t* k, uint64_t n, const uint32_t* u, const uint32_t* v,
                                const uint32_t* msg, uint64_t elements, const uint32_t* p_mont, const HostModulus& h,
                                cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            lhe_combine_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(out, k, n, u, v, msg, elements,
                                                                               device_modulus(h), holder(p_mont));
            return cudaGetLastError();
        }

        cudaError_t uniform(uint32_t* out, uint64_t elements, const RngKey& rng, int words, uint32_t top_mask,
                            const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            const unsigned grid = grid_for(elements, 256);
            if (words == L + 2)
            {
                uniform_kernel<L, L + 2><<<grid, 256, 0, stream>>>(out, elements, rng, top_mask, device_modulus(h));
            }
            else if (words == L + 3)
            {
                uniform_kernel<L, L + 3><<<grid, 256, 0, stream>>>(out, elements, rng, top_mask, device_modulus(h));
            }
            else
            {
                return cudaErrorInvalidValue;
            }
            return cudaGetLastError();
        }

        cudaError_t uniform_pairs(uint32_t* out, uint32_t log_n, uint64_t elements, const RngKey& rng, int words,
                                  uint32_t top_mask, const HostModulus& h, cudaStream_t stream)
        {
            if (elements < 2 || log_n < 1)
            {
                return elements ? cudaErrorInvalidValue : cudaSuccess;
            }
            const unsigned grid = grid_for(elements / 2, 256);
            if (words == L + 2)
            {
                uniform_pairs_kernel<L, L + 2><<<grid, 256, 0, stream>>>(out, log_n, elements, rng, top_mask,
                                                                         device_modulus(h));
            }
            else if (words == L + 3)
            {
                uniform_pairs_kernel<L, L + 3><<<grid, 256, 0, stream>>>(out, log_n, elements, rng, top_mask,
                                                                         device_modulus(h));
            }
            else
            {
                return cudaErrorInvalidValue;
            }
            return cudaGetLastError();
        }

        cudaError_t cbd(uint32_t* out, uint64_t elements, const RngKey& rng, uint32_t vx2, const uint32_t* table,
                        const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            const unsigned grid = grid_for(elements, 256);
            const Modulus<L> m = device_modulus(h);
            switch ((2 * vx2 + 31) / 32)
            {
            case 1: cbd_kernel<L, 1><<<grid, 256, 0, stream>>>(out, elements, rng, vx2, table, m); break;
            case 2: cbd_kernel<L, 2><<<grid, 256, 0, stream>>>(out, elements, rng, vx2, table, m); break;
            case 3: cbd_kernel<L, 3><<<grid, 256, 0, stream>>>(out, elements, rng, vx2, table, m); break;
            case 4: cbd_kernel<L, 4><<<grid, 256, 0, stream>>>(out, elements, rng, vx2, table, m); break;
            default: return cudaErrorInvalidValue;
            }
            return cudaGetLastError();
        }

        cudaError_t to_montgomery(uint32_t* out, const uint32_t* in, uint64_t elements, const HostModulus& h,
                                  cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            to_montgomery_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(out, in, elements, holder(h.r2),
                                                                                 device_modulus(h));
            return cudaGetLastError();
        }

        cudaError_t from_montgomery(uint32_t* out, const uint32_t* in, uint64_t elements, const HostModulus& h,
                                    cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            from_montgomery_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(out, in, elements,
                                                                                   device_modulus(h));
            return cudaGetLastError();
        }

        cudaError_t cast(uint32_t* out, const uint32_t* in, uint64_t elements, const CastParams& cp,
                         const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            const unsigned grid = grid_for(elements, 256);
            const Modulus<L> m = device_modulus(h);
            switch (cp.src_limbs)
            {
            case 1: cast_kernel<L, 1><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 2: cast_kernel<L, 2><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 3: cast_kernel<L, 3><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 4: cast_kernel<L, 4><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 5: cast_kernel<L, 5><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 6: cast_kernel<L, 6><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 7: cast_kernel<L, 7><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 8: cast_kernel<L, 8><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            case 9: cast_kernel<L, 9><<<grid, 256, 0, stream>>>(out, in, elements, cp, m); break;
            default: return cudaErrorInvalidValue;
            }
            return cudaGetLastError();
        }

        template<int Kind, int NW>
        cudaError_t launch_plain(const PlainStageParams& p, const Modulus<L>& m, cudaStream_t stream)
        {
            plain_stage_kernel<L, Kind, NW><<<grid_for(p.elements / 2, 256), 256, 0, stream>>>(p, m);
            return cudaGetLastError();
        }

        cudaError_t plain_stage(const PlainStageParams& p, int kind, int nw, const HostModulus& h, cudaStream_t stream)
        {
            const Modulus<L> m = device_modulus(h);
            if (kind == producer_tensor || p.stage != 0)
            {
                return launch_plain<producer_tensor, 1>(p, m, stream);
            }
            if (kind == producer_cbd)
            {
                switch (nw)
                {
                case 1: return launch_plain<producer_cbd, 1>(p, m, stream);
                case 2: return launch_plain<producer_cbd, 2>(p, m, stream);
                case 3: return launch_plain<producer_cbd, 3>(p, m, stream);
                case 4: return launch_plain<producer_cbd, 4>(p, m, stream);
                default: return cudaErrorInvalidValue;
                }
            }
            if (kind == producer_uniform)
            {
                if (nw == L + 2)
                {
                    return launch_plain<producer_uniform, L + 2>(p, m, stream);
                }
                if (nw == L + 3)
                {
                    return launch_plain<producer_uniform, L + 3>(p, m, stream);
                }
            }
            return cudaErrorInvalidValue;
        }

        cudaError_t ct_mul(uint32_t* d0, uint32_t* d1, uint32_t* d2, const uint32_t* a0, const uint32_t* a1,
                           const uint32_t* b0, const uint32_t* b1, uint64_t elements, const HostModulus& h,
                           cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            ct_mul_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(d0, d1, d2, a0, a1, b0, b1, elements,
                                                                          device_modulus(h));
            return cudaGetLastError();
        }

        cudaError_t dec_combine(uint32_t* x, const uint32_t* s, uint64_t n, const uint32_t* c0, const uint32_t* c1,
                                const uint32_t* c2, uint64_t elements, const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            dec_combine_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(x, s, n, c0, c1, c2, elements,
                                                                               device_modulus(h));
            return cudaGetLastError();
        }

        cudaError_t ntt_batched(const BatchedParams& bp, bool inverse, const HostModulus& h, unsigned grid,
                                unsigned block, size_t smem, cudaStream_t stream)
        {
            const Modulus<L> m = device_modulus(h);
            if (inverse)
            {
                ntt_batched_kernel<L, true><<<grid, block, smem, stream>>>(bp, m);
            }
            else
            {
                ntt_batched_kernel<L, false><<<grid, block, smem, stream>>>(bp, m);
            }
            return cudaGetLastError();
        }

        int ntt_batched_blocks_per_sm(bool inverse, unsigned block, size_t smem)
        {
            int blocks = 0;
            const cudaError_t e =
                inverse ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, ntt_batched_kernel<L, true>,
                                                                        static_cast<int>(block), smem)
                        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&blocks, ntt_batched_kernel<L, false>,
                                                                        static_cast<int>(block), smem);
            return e == cudaSuccess ? blocks : 0;
        }

        cudaError_t lhe_combine_pair(uint32_t* c0, uint32_t* c1, const PolyRequest* requests, const uint32_t* ka,
                                     const uint32_t* kb, uint64_t n, const uint32_t* u, const uint32_t* x, const uint32_t* w, uint64_t stride,
                                     uint64_t elements, bool dependent, const HostModulus& h, cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            return launch(requests ? lhe_combine_pair_kernel<L, true> : lhe_combine_pair_kernel<L, false>,
                          grid_for(elements, 256), 256, 0, dependent, stream, c0, c1, requests, ka, kb, n, u, x, w,
                          stride, elements, device_modulus(h));
        }

        cudaError_t lhe_key(uint32_t* a, uint32_t* b, const uint32_t* s, const uint32_t* x, uint64_t elements,
                            const RngKey& rng, int words, uint32_t top_mask, bool dependent, const HostModulus& h,
                            cudaStream_t stream)
        {
            const unsigned block = elements >= 152ull * 256 ? 256 : 128;
            const unsigned grid = static_cast<unsigned>((elements + block - 1) / block);
            const Modulus<L> m = device_modulus(h);
            if (words == L + 2)
            {
                return launch(lhe_key_kernel<L, L + 2>, grid, block, 0, dependent, stream, a, b, s, x, elements, rng,
                              top_mask, m);
            }
            if (words == L + 3)
            {
                return launch(lhe_key_kernel<L, L + 3>, grid, block, 0, dependent, stream, a, b, s, x, elements, rng,
                              top_mask, m);
            }
            return cudaErrorInvalidValue;
        }

        cudaError_t matvec(uint32_t* z, const uint32_t* mat, const uint32_t* x, const MatvecParams& p,
                           const HostModulus& h, cudaStream_t stream)
        {
            if (p.total == 0)
            {
                return cudaSuccess;
            }
            // 128 threads: 119 -> 115 us for 16 x (4 x 4) of degree 2^15 at 8 limbs (shorter last wave)
            const unsigned grid = grid_for(p.total, 128);
            // lazily where there are products to add up (figures at the kernel)
            if (L > 1 && p.cols > 1)
            {
                matvec_kernel<L, (L > 1)><<<grid, 128, 0, stream>>>(z, mat, x, p, device_modulus(h));
            }
            else
            {
                matvec_kernel<L, false><<<grid, 128, 0, stream>>>(z, mat, x, p, device_modulus(h));
            }
            return cudaGetLastError();
        }

        cudaError_t matvec_monomial(uint32_t* z, const int64_t* degrees, const uint32_t* x, const MatvecParams& p,
                                    const HostModulus& h, cudaStream_t stream)
        {
            if (p.total == 0)
            {
                return cudaSuccess;
            }
            matvec_monomial_kernel<L><<<grid_for(p.total, 256), 256, 0, stream>>>(z, degrees, x, p,
                                                                                device_modulus(h));
            return cudaGetLastError();
        }

        cudaError_t reduce(uint32_t* out, const uint32_t* in, uint64_t elements, int op, bool mod,
                           uint32_t top_mask, unsigned grid, const HostModulus& h, cudaStream_t stream)
        {
            const bool vectorised = elements % vec == 0 && reinterpret_cast<uintptr_t>(in) % 16 == 0;
            if (mod)
            {
                const Reducer<L, true> red{op, 0xffffffffu, device_modulus(h)};
                reduce_kernel<L, true><<<grid, 256, 0, stream>>>(out, grid, in, elements, vectorised, red);
            }
            else
            {
                const Reducer<L, false> red{op, top_mask, Modulus<L>{}};
                reduce_kernel<L, false><<<grid, 256, 0, stream>>>(out, grid, in, elements, vectorised, red);
            }
            return cudaGetLastError();
        }

        cudaError_t plane_sum(uint32_t* out, uint64_t* part, const uint32_t* in, uint64_t elements, unsigned chunks,
                              bool dependent, const HostModulus& h, cudaStream_t stream)
        {
            plane_sum_kernel<L><<<L * chunks, 256, 0, stream>>>(part, in, elements, chunks);
            cudaError_t e = cudaGetLastError();
            if (e != cudaSuccess)
            {
                return e;
            }
            return launch(plane_sum_finish_kernel<L>, 1, 32 * L, 0, dependent, stream, out, part, chunks,
                          holder(h.r2), device_modulus(h));
        }

        cudaError_t equal(uint32_t* out, const uint32_t* a, const uint32_t* b, uint64_t elements,
                          cudaStream_t stream)
        {
            if (elements == 0)
            {
                return cudaSuccess;
            }
            equal_kernel<L><<<grid_for(elements, 256), 256, 0, stream>>>(out, a, b, elements);
            return cudaGetLastError();
        }

        cudaError_t ntt_request(const PairPassParams& p, bool first, const HostModulus& h, unsigned grid,
                                unsigned block, size_t smem, cudaStream_t stream)
        {
            return launch(first ? ntt_request_kernel<L, true> : ntt_request_kernel<L, false>, grid, block, smem,
                          p.dependent != 0, stream, p, device_modulus(h));
        }

        cudaError_t ntt_decrypt(const PairPassParams& p, const DecryptParams& d, bool first, int p_limbs,
                                const HostModulus& h, unsigned grid, unsigned block, size_t smem, cudaStream_t stream)
        {
            const Modulus<L> m = device_modulus(h);
            void (*kernel)(PairPassParams, DecryptParams, Modulus<L>) = nullptr;
            switch (p_limbs)
            {
            case 0: kernel = first ? ntt_decrypt_kernel<L, true, 0> : ntt_decrypt_kernel<L, false, 0>; break;
            case 1: kernel = first ? ntt_decrypt_kernel<L, true, 1> : ntt_decrypt_kernel<L, false, 1>; break;
            case 2: kernel = first ? ntt_decrypt_kernel<L, true, 2> : ntt_decrypt_kernel<L, false, 2>; break;
            default: return cudaErrorInvalidValue;
            }
            return launch(kernel, grid, block, smem, p.dependent != 0, stream, p, d, m);
        }

        cudaError_t tc_tail(const TailParams& p, bool encrypt, bool dependent, const HostModulus& h,
                            cudaStream_t stream)
        {
            const unsigned grid = static_cast<unsigned>(((p.end - p.begin) / 2 + 127) / 128);
            const Modulus<L> m = device_modulus(h);
            return encrypt ? launch(tc_tail_kernel<L, true>, grid, 128, 0, dependent, stream, p, m)
                           : launch(tc_tail_kernel<L, false>, grid, 128, 0, dependent, stream, p, m);
        }

        cudaError_t ntt_cluster(const ClusterNttParams& p, uint64_t batch, const HostModulus& h, cudaStream_t stream)
        {
            if (batch == 0)
            {
                return cudaSuccess;
            }
            if (p.log_n < 10 || p.log_n > 14)
            {
                return cudaErrorInvalidValue;
            }
            const size_t smem = cl_smem_bytes<L>(p.log_n);
            static cudaError_t configured = cudaFuncSetAttribute(
                ntt_cluster_kernel<L>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cl_smem_bytes<L>(14)));
            if (configured != cudaSuccess)
            {
                return configured;
            }
            // one butterfly per thread and stage: N/16 per CTA
            const uint32_t work = 1u << (p.log_n - 4);
            const unsigned threads = std::min(256u, std::max(32u, work));
            ntt_cluster_kernel<L><<<static_cast<unsigned>(batch * cl_ctas), threads, smem, stream>>>(p, device_modulus(h));
            return cudaGetLastError();
        }

        const KernelTable table = {fma, binary, lhe_combine, uniform, cbd, to_montgomery,
                                   from_montgomery, cast, plain_stage, ct_mul, dec_combine, ntt_batched,
                                   ntt_batched_blocks_per_sm, lhe_combine_pair, lhe_key, matvec, matvec_monomial,
                                   reduce, plane_sum, equal, ntt_cluster, uniform_pairs, ntt_request, ntt_decrypt, tc_tail, ntt_pair};
    }

    const KernelTable* HMPC_CAT(kernel_table_, HMPC_L)()
    {
        return &table;
    }
}
