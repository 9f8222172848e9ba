// C-ABI layer: contexts (device, stream, RNG capability), registered moduli
// with their cached twiddle tables, the NTT pass planner and the launchers.
#include "../../include/hmpc_gb300.h"

#include <algorithm>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <string>
#include <vector>

#include <cuda_runtime.h>

#include "dispatch.hpp"
#include "host_math.hpp"
#include "internal.hpp"
#include "plan.hpp"

using namespace hmpc_gb300;

namespace hmpc_gb300::detail
{
    thread_local std::string last_error;

    int fail(int code, const std::string& message)
    {
        last_error = message;
        return code;
    }

    int cuda_fail(cudaError_t e, const char* what)
    {
        return fail(HMPC_ERROR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
    }

    void nonce_add(uint32_t nonce[3], uint64_t v)
    {
        uint64_t s = static_cast<uint64_t>(nonce[0]) + static_cast<uint32_t>(v);
        nonce[0] = static_cast<uint32_t>(s);
        s = static_cast<uint64_t>(nonce[1]) + static_cast<uint32_t>(v >> 32) + (s >> 32);
        nonce[1] = static_cast<uint32_t>(s);
        nonce[2] += static_cast<uint32_t>(s >> 32);
    }
}

using namespace hmpc_gb300::detail;

namespace
{
    host::words to_words(const uint32_t* p, int n)
    {
        return host::words(p, p + n);
    }
}

namespace hmpc_gb300::detail
{
    int check_degree(uint64_t n)
    {
        if (n < 4 || (n & (n - 1)) != 0 || n > (1ull << 30))
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "ring degree must be a power of two in [4, 2^30]");
        }
        return HMPC_OK;
    }

    int enter(hmpc_context* ctx)
    {
        if (!ctx)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null context");
        }
        HMPC_CUDA(cudaSetDevice(ctx->device), "cudaSetDevice");
        return HMPC_OK;
    }

    bool capturing(const hmpc_context* ctx)
    {
        cudaStreamCaptureStatus status = cudaStreamCaptureStatusNone;
        return cudaStreamIsCapturing(ctx->stream, &status) == cudaSuccess && status != cudaStreamCaptureStatusNone;
    }

    int run_transform(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t batch, bool inverse, int kind,
                      uint32_t vx2, uint32_t security, const uint32_t* src, uint32_t* out, const PolyRequest* requests,
                      uint32_t rng_slot, bool cuda_cores_only)
    {
        if (int rc = enter(ctx))
        {
            return rc;
        }
        if (!mod)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
        }
        if (int rc = check_degree(n))
        {
            return rc;
        }
        if (batch == 0)
        {
            return HMPC_OK;
        }
        if (!out)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null output");
        }
        Tables* t = nullptr;
        if (int rc = mod->prepare(n, &t))
        {
            return rc;
        }
        const int L = mod->c.limbs;
        int nw = 1;
        uint32_t top_mask = 0xffffffffu;
        if (kind == producer_cbd)
        {
            if (vx2 < 1 || vx2 > 64)
            {
                return fail(HMPC_ERROR_UNSUPPORTED, "centred binomial needs 1 <= 2V <= 64");
            }
            nw = static_cast<int>((2 * vx2 + 31) / 32);
        }
        else if (kind == producer_uniform)
        {
            const uint32_t bits = static_cast<uint32_t>(mod->c.bits) + security;
            nw = static_cast<int>((bits + 31) / 32);
            if (nw != L + 2 && nw != L + 3)
            {
                return fail(HMPC_ERROR_UNSUPPORTED, "uniform sampler supports statistical security 80");
            }
            if (bits % 32)
            {
                top_mask = (1u << (bits % 32)) - 1u;
            }
        }
        else if (kind != producer_tensor)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "unknown producer kind");
        }
        if (kind == producer_tensor && !src)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "tensor producer without source");
        }
        const int log_n = __builtin_ctzll(n);
        hmpc_modulus::TileChoice choice = mod->choice(n, inverse, batch);
        if (choice.radix_bits == 0)
        {
            // tensor-core engine; calls it does not cover run the default CUDA-core tiles
            if (!cuda_cores_only && tc_applicable(mod, log_n, kind, requests) &&
                (kind != producer_uniform || !inverse))
            {
                if (kind != producer_uniform)
                {
                    return run_tc_transform(ctx, mod, n, batch, inverse, kind, vx2, src, out, choice.local_bits);
                }
                // the engine's first group reads memory: the stage-0 pairs'
                // uniform draws go to `out` first, then the transform runs in place
                cudaError_t e = mod->kt->uniform_pairs(out, static_cast<uint32_t>(log_n), n * batch, ctx->rng(), nw,
                                                       top_mask, mod->h, ctx->stream);
                if (e != cudaSuccess)
                {
                    return cuda_fail(e, "launching the uniform pair sampler");
                }
                ++ctx->launches;
                if (int rc = run_tc_transform(ctx, mod, n, batch, false, producer_tensor, 0, out, out,
                                              choice.local_bits))
                {
                    return rc;
                }
                nonce_add(ctx->nonce, n * batch);
                return HMPC_OK;
            }
            choice = hmpc_modulus::TileChoice{};
        }
        if (choice.radix_bits == 1)
        {
            // one thread-block cluster per polynomial; calls it does not cover
            // run the default CUDA-core tiles
            if (kind == producer_tensor && !requests && log_n >= 10 && log_n <= 14)
            {
                ClusterNttParams cp{};
                cp.in = src;
                cp.out = out;
                cp.twiddles = inverse ? t->inverse : t->forward;
                cp.elements = n * batch;
                cp.log_n = static_cast<uint32_t>(log_n);
                cp.inverse = inverse ? 1u : 0u;
                cudaError_t e = mod->kt->ntt_cluster(cp, batch, mod->h, ctx->stream);
                if (e != cudaSuccess)
                {
                    return cuda_fail(e, "launching the cluster transform");
                }
                ++ctx->launches;
                return HMPC_OK;
            }
            choice = hmpc_modulus::TileChoice{};
        }
        // Every pass launches with programmatic dependence on the kernel before
        // it in the stream: its CTAs take the SMs' free slots and fetch their
        // first twiddles while that kernel drains, and wait for its completion
        // before reading an element.  Measured over the passes of one call:
        // 20.9 -> 14.9 us (one polynomial of 2^15 at 8 limbs), 18.8 -> 16.2 us
        // (12 of 2^13 at 6), 297.3 -> 295.2 us (64 of 2^15 at 8): never slower.
        // Ordinary launches while the stream is being captured.
        const bool dependent = !capturing(ctx);
        const std::vector<PairPlan> plan = plan_pairs(L, log_n, batch, inverse, choice.local_bits, choice.col_bits);
        for (size_t i = 0; i < plan.size(); ++i)
        {
            PairPassParams p = plan[i].params;
            p.dependent = dependent ? 1u : 0u;
            p.out[0] = out;
            p.src = i == 0 ? src : nullptr;
            p.twiddles = inverse ? t->inverse : t->forward;
            p.small_table = mod->small_table;
            p.elements = n * batch;
            p.rng = ctx->rng();
            p.vx2 = vx2;
            p.top_mask = top_mask;
            p.requests = requests;
            p.rng_slot = rng_slot;
            cudaError_t e = mod->kt->ntt_pair(p, i == 0 ? kind : producer_tensor, nw, inverse, mod->h, plan[i].grid,
                                              plan[i].block, plan[i].smem, ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching NTT pass");
            }
            ++ctx->launches;
        }
        if (kind != producer_tensor && !requests)
        {
            nonce_add(ctx->nonce, n * batch);
        }
        return HMPC_OK;
    }

    CastParams make_cast(const hmpc_modulus* dst, const hmpc_modulus* src)
    {
        CastParams cp{};
        const int ls = src->c.limbs;
        const int ld = dst->c.limbs;
        cp.src_limbs = static_cast<uint32_t>(ls);
        cp.src_ninv = src->c.ninv;
        for (int j = 0; j < ls; ++j)
        {
            cp.src_q[j] = src->c.q[static_cast<size_t>(j)];
            cp.src_half[j] = src->c.half[static_cast<size_t>(j)];
        }
        const int nw = std::max(ls, ld) + 1;
        host::words offset;
        if (host::compare(dst->c.q, src->c.q) > 0)
        {
            offset = host::sub(dst->c.q, src->c.q, nw);
            cp.direct = 1;
            for (int j = 0; j < ld; ++j)
            {
                cp.factor[j] = dst->c.r2[static_cast<size_t>(j)];
            }
        }
        else
        {
            const host::words rem = host::mod(src->c.q, dst->c.q);
            offset = host::bit_width(rem) == 0 ? host::words(static_cast<size_t>(nw), 0u) : host::sub(dst->c.q, rem, nw);
            cp.direct = 0;
            host::words wide(static_cast<size_t>(nw + ld), 0u);
            for (int j = 0; j < ld; ++j)
            {
                wide[static_cast<size_t>(nw + j)] = dst->c.r2[static_cast<size_t>(j)];
            }
            const host::words f = host::mod(wide, dst->c.q);
            for (int j = 0; j < ld; ++j)
            {
                cp.factor[j] = f[static_cast<size_t>(j)];
            }
        }
        offset = host::resize(offset, nw);
        for (int j = 0; j < nw; ++j)
        {
            cp.offset[j] = offset[static_cast<size_t>(j)];
        }
        return cp;
    }
}

namespace hmpc_gb300::detail
{
    bool overlap(const uint32_t* a, uint64_t a_words, const uint32_t* b, uint64_t b_words)
    {
        return a < b + b_words && b < a + a_words;
    }

    // the lift of INTT_q(c0 - s*c1) to p in the inverse transform's own passes
    int run_decrypt(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint64_t batch, const uint32_t* s,
                    const uint32_t* c0, const uint32_t* c1, uint32_t* x, uint32_t* out, bool ntt_form,
                    const hmpc_modulus::TileChoice& choice, const std::vector<PairPlan>& plan)
    {
        Tables* t = nullptr;
        Tables* pt = nullptr;
        if (int rc = q->prepare(n, &t))
        {
            return rc;
        }
        if (ntt_form)
        {
            if (int rc = p->prepare(n, &pt))
            {
                return rc;
            }
        }
        DecryptParams d{};
        d.s = s;
        d.c0 = c0;
        d.c1 = c1;
        d.out = out;
        d.cast = make_cast(p, q);
        std::copy(p->h.q, p->h.q + p->c.limbs, d.p);
        d.pninv = p->h.ninv;
        d.p_twiddles = ntt_form ? pt->forward : nullptr;
        const bool dependent = !capturing(ctx);
        for (size_t i = 0; i < plan.size(); ++i)
        {
            PairPassParams pp = plan[i].params;
            pp.out[0] = x;
            pp.twiddles = t->inverse;
            pp.elements = n * batch;
            pp.dependent = dependent ? 1u : 0u;
            const cudaError_t e = q->kt->ntt_decrypt(pp, d, i == 0, i + 1 == plan.size() ? p->c.limbs : 0, q->h,
                                                     plan[i].grid, plan[i].block, plan[i].smem, ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching decryption pass");
            }
            ++ctx->launches;
        }
        if (!ntt_form)
        {
            return HMPC_OK;
        }
        // the forward transform mod p from its second pass on, in the same tiles
        const std::vector<PairPlan> forward =
            plan_pairs(p->c.limbs, __builtin_ctzll(n), batch, false, choice.local_bits, choice.col_bits);
        for (size_t i = 1; i < forward.size(); ++i)
        {
            PairPassParams pp = forward[i].params;
            pp.out[0] = out;
            pp.twiddles = pt->forward;
            pp.elements = n * batch;
            pp.dependent = dependent ? 1u : 0u;
            const cudaError_t e = p->kt->ntt_pair(pp, producer_tensor, 1, false, p->h, forward[i].grid,
                                                  forward[i].block, forward[i].smem, ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching NTT pass");
            }
            ++ctx->launches;
        }
        return HMPC_OK;
    }

    // x = c0 - s*c1 (+ s^2*c2) -> INTT_q -> cast to p (-> NTT_p)
    int decrypt(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint64_t batch, const uint32_t* s,
                const uint32_t* c0, const uint32_t* c1, const uint32_t* c2, int plaintext_ntt, uint32_t* out)
    {
        if (int rc = enter(ctx))
        {
            return rc;
        }
        if (!q || !p || !s || !c0 || !c1 || !out)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
        }
        if (int rc = check_degree(n))
        {
            return rc;
        }
        if (batch == 0)
        {
            return HMPC_OK;
        }
        const uint64_t elements = n * batch;
        uint32_t* x = ctx->scratch(elements * static_cast<uint64_t>(q->c.limbs));
        if (!x)
        {
            return fail(HMPC_ERROR_OUT_OF_MEMORY, "allocating the decryption workspace");
        }
        const hmpc_modulus::TileChoice choice = q->choice(n, true, batch);
        if (!c2 && choice.radix_bits >= 2 && p->c.limbs <= 2 && host::compare(q->c.q, p->c.q) > 0)
        {
            const std::vector<PairPlan> plan =
                plan_pairs(q->c.limbs, __builtin_ctzll(n), batch, true, choice.local_bits, choice.col_bits);
            const uint64_t q_words = elements * static_cast<uint64_t>(q->c.limbs);
            const uint64_t s_words = n * static_cast<uint64_t>(q->c.limbs);
            const uint64_t out_words = elements * static_cast<uint64_t>(p->c.limbs);
            // one pass that reads and writes: not over its own operands
            if (plan.size() > 1 || !(overlap(out, out_words, c0, q_words) || overlap(out, out_words, c1, q_words) ||
                                     overlap(out, out_words, s, s_words)))
            {
                return run_decrypt(ctx, q, p, n, batch, s, c0, c1, x, out, plaintext_ntt != 0, choice, plan);
            }
        }
        cudaError_t e = q->kt->dec_combine(x, s, n, c0, c1, c2, elements, q->h, ctx->stream);
        if (e != cudaSuccess)
        {
            return cuda_fail(e, "launching decryption combine");
        }
        ++ctx->launches;
        int rc = run_transform(ctx, q, n, batch, true, producer_tensor, 0, 0, x, x);
        if (rc)
        {
            return rc;
        }
        e = p->kt->cast(out, x, elements, make_cast(p, q), p->h, ctx->stream);
        if (e != cudaSuccess)
        {
            return cuda_fail(e, "launching cast");
        }
        ++ctx->launches;
        if (plaintext_ntt)
        {
            rc = run_transform(ctx, p, n, batch, false, producer_tensor, 0, 0, out, out);
        }
        return rc;
    }

    bool parts_applicable(const hmpc_modulus* q, const hmpc_modulus* p)
    {
        // p times a sample plus a lifted residue stays below 2^70 < Q
        return p->c.limbs <= 2 && q->c.bits >= 72;
    }

    // Forward transforms of `count` parts of `batch` polynomials as one run of
    // passes: part i is drawn as kinds[i] with nonce ctx->nonce + slots[i] * n *
    // batch (or from the requests' with that slot) and goes to out[i].
    int run_parts(hmpc_context* ctx, hmpc_modulus* q, const hmpc_modulus* p, uint64_t n, uint64_t batch, int count,
                  const uint32_t* kinds, const uint32_t* slots, uint32_t* const* out, const uint32_t* msg,
                  const PolyRequest* requests, const hmpc_modulus::TileChoice& choice)
    {
        Tables* t = nullptr;
        if (int rc = q->prepare(n, &t))
        {
            return rc;
        }
        const std::vector<PairPlan> plan =
            plan_pairs(q->c.limbs, __builtin_ctzll(n), batch * count, false, choice.local_bits, choice.col_bits);
        const bool dependent = !capturing(ctx);
        for (size_t i = 0; i < plan.size(); ++i)
        {
            PairPassParams pp = plan[i].params;
            pp.part_polys = batch;
            pp.elements = n * batch;
            pp.twiddles = t->forward;
            pp.small_table = q->small_table;
            pp.rng = ctx->rng();
            pp.requests = requests;
            pp.dependent = dependent ? 1u : 0u;
            for (int j = 0; j < count; ++j)
            {
                pp.out[j] = out[j];
                pp.parts.kind[j] = kinds[j];
                std::copy(ctx->nonce, ctx->nonce + 3, pp.parts.nonce[j]);
                nonce_add(pp.parts.nonce[j], slots[j] * n * batch);
            }
            pp.parts.msg = msg;
            pp.parts.msg_limbs = static_cast<uint32_t>(p->c.limbs);
            for (int j = 0; j < p->c.limbs; ++j)
            {
                pp.parts.pq[j] = p->h.q[j];
                pp.parts.phalf[j] = p->h.half[j];
            }
            pp.parts.pninv = p->h.ninv;
            std::copy(q->h.r2, q->h.r2 + q->c.limbs, pp.parts.r2);
            cudaError_t e = q->kt->ntt_pair(pp, i == 0 ? producer_parts : producer_tensor, 1, false, q->h,
                                            plan[i].grid, plan[i].block, plan[i].smem, ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching NTT pass");
            }
            ++ctx->launches;
        }
        return HMPC_OK;
    }

    int run_requests(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t polys, const PolyRequest* requests)
    {
        hmpc_modulus::TileChoice choice = mod->choice(n, false, polys);
        if (choice.radix_bits < 2)
        {
            choice = hmpc_modulus::TileChoice{};
        }
        Tables* t = nullptr;
        if (int rc = mod->prepare(n, &t))
        {
            return rc;
        }
        const std::vector<PairPlan> plan =
            plan_pairs(mod->c.limbs, __builtin_ctzll(n), polys, false, choice.local_bits, choice.col_bits);
        const bool dependent = !capturing(ctx);
        for (size_t i = 0; i < plan.size(); ++i)
        {
            PairPassParams p = plan[i].params;
            p.dependent = dependent ? 1u : 0u;
            p.twiddles = t->forward;
            p.elements = n * polys;
            p.requests = requests;
            const cudaError_t e = mod->kt->ntt_request(p, i == 0, mod->h, plan[i].grid, plan[i].block, plan[i].smem,
                                                       ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching NTT pass");
            }
            ++ctx->launches;
        }
        return HMPC_OK;
    }

    int encrypt_cuda_cores(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint64_t batch,
                           const uint32_t* key_a, const uint32_t* key_b, const uint32_t* coefficients, uint32_t* c0,
                           uint32_t* c1, uint32_t* workspace, const PolyRequest* requests, bool cuda_cores_only)
    {
        const uint64_t elements = n * batch;
        const uint64_t poly_words = elements * static_cast<uint64_t>(q->c.limbs);
        uint32_t* u = workspace;
        uint32_t* v = u + poly_words;
        uint32_t* msg = v + poly_words;
        if (parts_applicable(q, p))
        {
            // linearity of the NTT: p*NTT(v) + NTT(lift(m)) = NTT(p*v + lift(m))
            // and p*NTT(w) = NTT(p*w), so three transforms run as one and one
            // kernel writes both halves.  Draws in the reference's order u, v, w
            // (expr/cache.hpp:226-271).
            const uint32_t kinds[3] = {part_ternary, part_scaled_message, part_scaled};
            const uint32_t slots[3] = {0, 1, 2};
            uint32_t* const outs[3] = {u, v, msg};
            // In the shape set or tuned for the transforms of (n, batch), three times
            // as many polynomials here: 16 of 2^14 at 8 limbs 152 us by the rule, 142
            // tuned; 8 of 2^13 43.5 and 45.7, the largest loss met.
            hmpc_modulus::TileChoice choice = q->choice(n, false, batch);
            if (choice.radix_bits < 2)
            {
                choice = hmpc_modulus::TileChoice{};
            }
            if (int rc = run_parts(ctx, q, p, n, batch, 3, kinds, slots, outs, coefficients, requests, choice))
            {
                return rc;
            }
            cudaError_t e = q->kt->lhe_combine_pair(c0, c1, c0 ? nullptr : requests, key_a, key_b, n, u, v, msg,
                                                    elements, elements,
                                                    !capturing(ctx), q->h, ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching combine");
            }
            ++ctx->launches;
            if (!requests)
            {
                nonce_add(ctx->nonce, 3 * elements);
            }
            return HMPC_OK;
        }
        // the reference's plan: NTT(u), NTT(v), NTT_q(msg), c0, NTT(w), c1
        int rc = run_transform(ctx, q, n, batch, false, producer_cbd, 1, 0, nullptr, u, requests, 0, cuda_cores_only);
        if (!rc)
        {
            rc = run_transform(ctx, q, n, batch, false, producer_cbd, 20, 0, nullptr, v, requests, 1, cuda_cores_only);
        }
        if (rc)
        {
            return rc;
        }
        cudaError_t e = q->kt->cast(msg, coefficients, elements, make_cast(q, p), q->h, ctx->stream);
        if (e != cudaSuccess)
        {
            return cuda_fail(e, "launching cast");
        }
        ++ctx->launches;
        if ((rc = run_transform(ctx, q, n, batch, false, producer_tensor, 0, 0, msg, msg, nullptr, 0,
                                cuda_cores_only)))
        {
            return rc;
        }
        const host::words pm = host::to_mont(q->c, p->c.q);
        if ((e = q->kt->lhe_combine(c0, key_a, n, u, v, msg, elements, pm.data(), q->h, ctx->stream)) != cudaSuccess)
        {
            return cuda_fail(e, "launching combine");
        }
        ++ctx->launches;
        // w reuses v's buffer
        if ((rc = run_transform(ctx, q, n, batch, false, producer_cbd, 20, 0, nullptr, v, requests, 2,
                                cuda_cores_only)))
        {
            return rc;
        }
        if ((e = q->kt->lhe_combine(c1, key_b, n, u, v, nullptr, elements, pm.data(), q->h, ctx->stream)) !=
            cudaSuccess)
        {
            return cuda_fail(e, "launching combine");
        }
        ++ctx->launches;
        return HMPC_OK;
    }

    // one launch per stage over global memory (plain.cuh)
    int run_plain(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t batch, bool inverse, int kind,
                  uint32_t vx2, uint32_t security, const uint32_t* src, uint32_t* out)
    {
        if (int rc = enter(ctx))
        {
            return rc;
        }
        if (!mod)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
        }
        if (int rc = check_degree(n))
        {
            return rc;
        }
        if (batch == 0)
        {
            return HMPC_OK;
        }
        if (!out)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "null output");
        }
        Tables* t = nullptr;
        if (int rc = mod->prepare(n, &t))
        {
            return rc;
        }
        const int L = mod->c.limbs;
        int nw = 1;
        uint32_t top_mask = 0xffffffffu;
        if (kind == producer_cbd)
        {
            if (vx2 < 1 || vx2 > 64)
            {
                return fail(HMPC_ERROR_UNSUPPORTED, "centred binomial needs 1 <= 2V <= 64");
            }
            nw = static_cast<int>((2 * vx2 + 31) / 32);
        }
        else if (kind == producer_uniform)
        {
            const uint32_t bits = static_cast<uint32_t>(mod->c.bits) + security;
            nw = static_cast<int>((bits + 31) / 32);
            if (nw != L + 2 && nw != L + 3)
            {
                return fail(HMPC_ERROR_UNSUPPORTED, "uniform sampler supports statistical security 80");
            }
            if (bits % 32)
            {
                top_mask = (1u << (bits % 32)) - 1u;
            }
        }
        else if (kind != producer_tensor || !src)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "bad producer");
        }
        PlainStageParams p{};
        p.out = out;
        p.src = src;
        p.twiddles = inverse ? t->inverse : t->forward;
        p.small_table = mod->small_table;
        p.elements = n * batch;
        p.log_n = static_cast<uint32_t>(__builtin_ctzll(n));
        p.inverse = inverse ? 1u : 0u;
        p.rng = ctx->rng();
        p.vx2 = vx2;
        p.top_mask = top_mask;
        for (uint32_t stage = 0; stage < p.log_n; ++stage)
        {
            p.stage = stage;
            cudaError_t e = mod->kt->plain_stage(p, kind, nw, mod->h, ctx->stream);
            if (e != cudaSuccess)
            {
                return cuda_fail(e, "launching plain stage");
            }
            ++ctx->launches;
        }
        if (kind != producer_tensor)
        {
            nonce_add(ctx->nonce, n * batch);
        }
        return HMPC_OK;
    }
}

extern "C" {

const char* hmpc_last_error(void)
{
    return last_error.c_str();
}

int hmpc_version(int* major, int* minor)
{
    if (major)
    {
        *major = 0;
    }
    if (minor)
    {
        *minor = 1;
    }
    return HMPC_OK;
}

int hmpc_context_create(int device, const uint32_t key[8], void* stream, hmpc_context** out)
{
    if (!out)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null output");
    }
    int count = 0;
    HMPC_CUDA(cudaGetDeviceCount(&count), "cudaGetDeviceCount");
    if (device < 0 || device >= count)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "no such CUDA device");
    }
    HMPC_CUDA(cudaSetDevice(device), "cudaSetDevice");
    auto* ctx = new hmpc_context;
    ctx->device = device;
    ctx->stream = static_cast<cudaStream_t>(stream);
    if (key)
    {
        std::memcpy(ctx->key, key, sizeof ctx->key);
    }
    *out = ctx;
    return HMPC_OK;
}

int hmpc_context_destroy(hmpc_context* ctx)
{
    if (!ctx)
    {
        return HMPC_OK;
    }
    cudaSetDevice(ctx->device);
    cudaStreamSynchronize(ctx->stream);
    for (auto* m : ctx->moduli)
    {
        delete m;
    }
    cudaFree(ctx->workspace);
    cudaFree(ctx->tc_workspace);
    cudaFree(ctx->tc_error);
    delete ctx;
    return HMPC_OK;
}

int hmpc_context_set_stream(hmpc_context* ctx, void* stream)
{
    if (!ctx)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null context");
    }
    ctx->stream = static_cast<cudaStream_t>(stream);
    return HMPC_OK;
}

int hmpc_context_get_nonce(const hmpc_context* ctx, uint32_t nonce[3])
{
    if (!ctx || !nonce)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    std::memcpy(nonce, ctx->nonce, sizeof ctx->nonce);
    return HMPC_OK;
}

int hmpc_context_set_nonce(hmpc_context* ctx, const uint32_t nonce[3])
{
    if (!ctx || !nonce)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    std::memcpy(ctx->nonce, nonce, sizeof ctx->nonce);
    return HMPC_OK;
}

int hmpc_context_launch_count(const hmpc_context* ctx, uint64_t* count)
{
    if (!ctx || !count)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    *count = ctx->launches;
    return HMPC_OK;
}

int hmpc_context_synchronize(hmpc_context* ctx)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    HMPC_CUDA(cudaStreamSynchronize(ctx->stream), "synchronizing");
    if (ctx->tc_error)
    {
        uint32_t code = 0;
        HMPC_CUDA(cudaMemcpy(&code, ctx->tc_error, sizeof code, cudaMemcpyDeviceToHost), "reading the error word");
        if (code)
        {
            HMPC_CUDA(cudaMemset(ctx->tc_error, 0, sizeof code), "clearing the error word");
            return fail(HMPC_ERROR_TIMEOUT, "a tensor-core transform gave up waiting for its tensor core or copy");
        }
    }
    return HMPC_OK;
}

int hmpc_modulus_create(hmpc_context* ctx, const uint32_t* q, int q_words, hmpc_modulus** out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!q || q_words <= 0 || !out)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus words");
    }
    auto m = std::make_unique<hmpc_modulus>();
    std::string error;
    if (!host::make_constants(to_words(q, q_words), m->c, error))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, error);
    }
    const int L = m->c.limbs;
    if (L > max_device_limbs)
    {
        return fail(HMPC_ERROR_UNSUPPORTED, "moduli up to 9 limbs (288 bits) are supported on the device");
    }
    m->ctx = ctx;
    m->kt = kernel_table(L);
    m->h.limbs = L;
    m->h.bits = m->c.bits;
    m->h.ninv = m->c.ninv;
    for (int j = 0; j < L; ++j)
    {
        m->h.q[j] = m->c.q[static_cast<size_t>(j)];
        m->h.one[j] = m->c.one[static_cast<size_t>(j)];
        m->h.r2[j] = m->c.r2[static_cast<size_t>(j)];
        m->h.half[j] = m->c.half[static_cast<size_t>(j)];
    }
    std::vector<uint32_t> small(static_cast<size_t>(65 * L));
    for (uint32_t v = 0; v <= 64; ++v)
    {
        const host::words mv = host::to_mont(m->c, host::words{v});
        std::copy(mv.begin(), mv.end(), small.begin() + static_cast<std::ptrdiff_t>(v * static_cast<uint32_t>(L)));
    }
    HMPC_CUDA(cudaMalloc(&m->small_table, small.size() * sizeof(uint32_t)), "allocating constants");
    HMPC_CUDA(cudaMemcpy(m->small_table, small.data(), small.size() * sizeof(uint32_t), cudaMemcpyHostToDevice),
              "uploading constants");
    ctx->moduli.push_back(m.get());
    *out = m.release();
    return HMPC_OK;
}

int hmpc_modulus_destroy(hmpc_modulus* mod)
{
    if (!mod)
    {
        return HMPC_OK;
    }
    auto& list = mod->ctx->moduli;
    list.erase(std::remove(list.begin(), list.end(), mod), list.end());
    cudaSetDevice(mod->ctx->device);
    cudaStreamSynchronize(mod->ctx->stream);
    delete mod;
    return HMPC_OK;
}

int hmpc_modulus_info(const hmpc_modulus* mod, int* limbs, int* bits, uint32_t* one)
{
    if (!mod)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
    }
    if (limbs)
    {
        *limbs = mod->c.limbs;
    }
    if (bits)
    {
        *bits = mod->c.bits;
    }
    if (one)
    {
        std::copy(mod->c.one.begin(), mod->c.one.end(), one);
    }
    return HMPC_OK;
}

int hmpc_modulus_prepare(hmpc_modulus* mod, uint64_t n)
{
    if (!mod)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    return mod->prepare(n, nullptr);
}

int hmpc_modulus_get_plan(hmpc_modulus* mod, uint64_t n, uint64_t batch, int inverse, int* radix_bits,
                          int* local_bits, int* col_bits)
{
    if (!mod || !radix_bits || !local_bits || !col_bits)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    const hmpc_modulus::TileChoice choice = mod->choice(n, inverse != 0, batch);
    *radix_bits = choice.radix_bits;
    *local_bits = choice.local_bits;
    *col_bits = choice.col_bits;
    return HMPC_OK;
}

int hmpc_modulus_tc_cost(hmpc_modulus* mod, uint64_t n, uint64_t batch, int inverse, int producer_kind, int splits,
                         hmpc_tc_cost* out)
{
    if (!mod || !out)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    return tc_cost(mod, n, batch, inverse != 0, producer_kind, splits, out);
}

int hmpc_modulus_tc_column_max(hmpc_modulus* mod, uint64_t n, int inverse, int splits, uint32_t* out)
{
    if (!mod || !out)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = enter(mod->ctx))
    {
        return rc;
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    return tc_column_max(mod->ctx, mod, n, inverse != 0, splits, out);
}

int hmpc_context_set_test_wait(hmpc_context* ctx, uint32_t polls, int stall)
{
    if (!ctx)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null context");
    }
    ctx->tc_spin_limit = polls ? polls : tc_default_spin_limit;
    ctx->tc_test_stall = stall ? 1u : 0u;
    return HMPC_OK;
}

int hmpc_context_set_tc_column_bound(hmpc_context* ctx, uint32_t bound)
{
    if (!ctx)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null context");
    }
    if (bound > tc_byte_carry_column_bound)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "the two-operation carry is exact up to a column bound of 32512");
    }
    ctx->tc_column_bound = bound;
    return HMPC_OK;
}

int hmpc_modulus_set_plan(hmpc_modulus* mod, uint64_t n, uint64_t batch, int inverse, int radix_bits,
                          int local_bits, int col_bits)
{
    if (!mod)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    if (radix_bits == 0)
    {
        if (local_bits < 0 || local_bits > 2)
        {
            return fail(HMPC_ERROR_INVALID_ARGUMENT, "the tensor-core engine splits its contiguous group 1 or 2 ways");
        }
        if (!tc_supported(mod))
        {
            return fail(HMPC_ERROR_UNSUPPORTED, "the tensor-core transform needs a 2- to 8-limb modulus below "
                                                "0.996 * 2^(32L) whose top limb is at least 32");
        }
    }
    else if (radix_bits == 1)
    {
        // the cluster engine has no tile shape
        local_bits = 0;
        col_bits = 0;
    }
    // Tiles of up to ten bits are what runs, and all of them fit; more bits run as
    // ten, and are refused where a tile that held as many in shared memory would
    // not have fitted, so that the statuses stay what they were.
    else if ((radix_bits != 2 && radix_bits != 3) || local_bits < 0 || local_bits > 13 || col_bits < 0 ||
             col_bits > 6 ||
             (local_bits && static_cast<uint64_t>(mod->c.limbs) * 4u * ((33u << local_bits) >> 5) > 200 * 1024))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "tile shape out of range");
    }
    std::lock_guard<std::mutex> lock(mod->tables_mutex);
    mod->tile_choices[std::make_tuple(__builtin_ctzll(n), inverse ? 1 : 0, batch)] = {radix_bits, local_bits,
                                                                                      col_bits};
    return HMPC_OK;
}

int hmpc_modulus_tune(hmpc_modulus* mod, uint64_t n, uint64_t batch, int inverse, float* best_ms)
{
    if (!mod)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
    }
    hmpc_context* ctx = mod->ctx;
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    if (batch == 0)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "empty batch");
    }
    if (int rc = mod->prepare(n, nullptr))
    {
        return rc;
    }
    const int L = mod->c.limbs;
    const uint64_t words = n * batch * static_cast<uint64_t>(L);
    uint32_t* buf = nullptr;
    if (cudaMalloc(&buf, words * sizeof(uint32_t)) != cudaSuccess)
    {
        return fail(HMPC_ERROR_OUT_OF_MEMORY, "allocating tuning scratch");
    }
    cudaMemsetAsync(buf, 0, words * sizeof(uint32_t), ctx->stream);
    cudaEvent_t t0, t1;
    cudaEventCreate(&t0);
    cudaEventCreate(&t1);
    const int log_n = __builtin_ctzll(n);
    const auto key = std::make_tuple(log_n, inverse ? 1 : 0, batch);
    float best = 1e30f;
    hmpc_modulus::TileChoice best_choice;
    auto time_choice = [&](const hmpc_modulus::TileChoice& choice) {
        {
            std::lock_guard<std::mutex> lock(mod->tables_mutex);
            mod->tile_choices[key] = choice;
        }
        float sample = 1e30f;
        for (int rep = 0; rep < 4; ++rep)
        {
            cudaEventRecord(t0, ctx->stream);
            if (run_transform(ctx, mod, n, batch, inverse, producer_tensor, 0, 0, buf, buf) != HMPC_OK)
            {
                return 1e30f;
            }
            cudaEventRecord(t1, ctx->stream);
            cudaEventSynchronize(t1);
            float ms = 0.f;
            cudaEventElapsedTime(&ms, t0, t1);
            if (rep)
            {
                sample = std::min(sample, ms);
            }
        }
        return sample;
    };
    if (log_n >= 4 && tc_supported(mod))
    {
        for (int splits : {1, 2})
        {
            hmpc_modulus::TileChoice tensor;
            tensor.radix_bits = 0;
            tensor.local_bits = splits;
            const float sample = time_choice(tensor);
            if (sample < best)
            {
                best = sample;
                best_choice = tensor;
            }
        }
    }
    // the cluster engine is no candidate: the tiles are ahead at every degree it
    // covers (one 4096 transform at 4 limbs 6.2 us, 12.3 on a cluster)
    for (int tile_bits = 7; tile_bits <= 10; ++tile_bits)
    {
        for (int c : {2, 3, 4})
        {
            const float sample = time_choice({3, tile_bits, c});
            if (sample < best)
            {
                best = sample;
                best_choice = {3, tile_bits, c};
            }
        }
    }
    {
        std::lock_guard<std::mutex> lock(mod->tables_mutex);
        mod->tile_choices[key] = best_choice;
    }
    cudaEventDestroy(t0);
    cudaEventDestroy(t1);
    cudaFree(buf);
    if (best_ms)
    {
        *best_ms = best;
    }
    return HMPC_OK;
}

int hmpc_modulus_root(hmpc_modulus* mod, uint64_t n, int inverse, uint32_t* root)
{
    if (!mod || !root)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    Tables* t = nullptr;
    if (int rc = mod->prepare(n, &t))
    {
        return rc;
    }
    const host::words& r = inverse ? t->inverse_root : t->root;
    std::copy(r.begin(), r.end(), root);
    return HMPC_OK;
}

int hmpc_modulus_twiddles(hmpc_modulus* mod, uint64_t n, int inverse, uint32_t* host_table)
{
    if (!mod || !host_table)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    Tables* t = nullptr;
    if (int rc = check_degree(n))
    {
        return rc;
    }
    if (int rc = mod->prepare(n, &t))
    {
        return rc;
    }
    HMPC_CUDA(cudaMemcpy(host_table, inverse ? t->inverse : t->forward,
                         n * static_cast<uint64_t>(mod->c.limbs) * sizeof(uint32_t), cudaMemcpyDeviceToHost),
              "downloading twiddles");
    return HMPC_OK;
}

int hmpc_tensor_alloc(hmpc_context* ctx, uint64_t words, uint32_t** out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!out)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null output");
    }
    if (cudaMalloc(out, std::max<uint64_t>(words, 1) * sizeof(uint32_t)) != cudaSuccess)
    {
        return fail(HMPC_ERROR_OUT_OF_MEMORY, "cudaMalloc failed");
    }
    return HMPC_OK;
}

int hmpc_tensor_free(hmpc_context* ctx, uint32_t* ptr)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    HMPC_CUDA(cudaFree(ptr), "cudaFree");
    return HMPC_OK;
}

int hmpc_tensor_upload(hmpc_context* ctx, uint32_t* dst, const uint32_t* host, uint64_t words)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    HMPC_CUDA(cudaMemcpyAsync(dst, host, words * sizeof(uint32_t), cudaMemcpyHostToDevice, ctx->stream), "upload");
    return HMPC_OK;
}

int hmpc_tensor_download(hmpc_context* ctx, uint32_t* host, const uint32_t* src, uint64_t words)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    HMPC_CUDA(cudaMemcpyAsync(host, src, words * sizeof(uint32_t), cudaMemcpyDeviceToHost, ctx->stream),
              "download");
    HMPC_CUDA(cudaStreamSynchronize(ctx->stream), "download");
    return HMPC_OK;
}

int hmpc_ntt_forward(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t batch, const hmpc_producer* producer,
                     uint32_t* out)
{
    if (!producer)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null producer");
    }
    return run_transform(ctx, mod, n, batch, false, producer->kind, producer->variance_x2, producer->security,
                         producer->src, out);
}

int hmpc_ntt_inverse(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t batch, const uint32_t* in,
                     uint32_t* out)
{
    return run_transform(ctx, mod, n, batch, true, producer_tensor, 0, 0, in, out);
}

int hmpc_fma(hmpc_context* ctx, hmpc_modulus* mod, uint64_t elements, const uint32_t* a, const uint32_t* b,
             const uint32_t* c, uint32_t* d)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!mod || (elements && (!a || !b || !c || !d)))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    cudaError_t e = mod->kt->fma(d, a, b, c, elements, mod->h, ctx->stream);
    ctx->launches += elements ? 1 : 0;
    return e == cudaSuccess ? HMPC_OK : cuda_fail(e, "launching fma");
}

int hmpc_binary(hmpc_context* ctx, hmpc_modulus* mod, int op, uint64_t elements, const uint32_t* a,
                uint64_t a_elements, const uint32_t* b, uint64_t b_elements, uint32_t* out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!mod || op < 0 || op > 2)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "bad modulus or operation");
    }
    if (elements == 0)
    {
        return HMPC_OK;
    }
    if (!a || !b || !out || a_elements == 0 || b_elements == 0 || elements % a_elements || elements % b_elements)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "operand sizes must divide the result size");
    }
    cudaError_t e = mod->kt->binary(out, a, a_elements, b, b_elements, elements, op, mod->h, ctx->stream);
    ++ctx->launches;
    return e == cudaSuccess ? HMPC_OK : cuda_fail(e, "launching binary op");
}

int hmpc_sample_uniform(hmpc_context* ctx, hmpc_modulus* mod, uint64_t elements, uint32_t security, uint32_t* out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!mod || (elements && !out))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    const uint32_t bits = static_cast<uint32_t>(mod->c.bits) + security;
    const int words = static_cast<int>((bits + 31) / 32);
    if (words != mod->c.limbs + 2 && words != mod->c.limbs + 3)
    {
        return fail(HMPC_ERROR_UNSUPPORTED, "uniform sampler supports statistical security 80");
    }
    const uint32_t top_mask = bits % 32 ? (1u << (bits % 32)) - 1u : 0xffffffffu;
    cudaError_t e = mod->kt->uniform(out, elements, ctx->rng(), words, top_mask, mod->h, ctx->stream);
    ctx->launches += elements ? 1 : 0;
    if (e != cudaSuccess)
    {
        return cuda_fail(e, "launching uniform sampler");
    }
    nonce_add(ctx->nonce, elements);
    return HMPC_OK;
}

int hmpc_sample_cbd(hmpc_context* ctx, hmpc_modulus* mod, uint64_t elements, uint32_t variance_x2, uint32_t* out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!mod || (elements && !out))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (variance_x2 < 1 || variance_x2 > 64)
    {
        return fail(HMPC_ERROR_UNSUPPORTED, "centred binomial needs 1 <= 2V <= 64");
    }
    cudaError_t e = mod->kt->cbd(out, elements, ctx->rng(), variance_x2, mod->small_table, mod->h, ctx->stream);
    ctx->launches += elements ? 1 : 0;
    if (e != cudaSuccess)
    {
        return cuda_fail(e, "launching binomial sampler");
    }
    nonce_add(ctx->nonce, elements);
    return HMPC_OK;
}

int hmpc_cast(hmpc_context* ctx, hmpc_modulus* dst, hmpc_modulus* src, uint64_t elements, const uint32_t* in,
              uint32_t* out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!dst || !src || (elements && (!in || !out)))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    cudaError_t e = dst->kt->cast(out, in, elements, make_cast(dst, src), dst->h, ctx->stream);
    ctx->launches += elements ? 1 : 0;
    return e == cudaSuccess ? HMPC_OK : cuda_fail(e, "launching cast");
}

int hmpc_to_montgomery(hmpc_context* ctx, hmpc_modulus* mod, uint64_t elements, const uint32_t* in, uint32_t* out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!mod)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
    }
    cudaError_t e = mod->kt->to_montgomery(out, in, elements, mod->h, ctx->stream);
    ctx->launches += elements ? 1 : 0;
    return e == cudaSuccess ? HMPC_OK : cuda_fail(e, "launching conversion");
}

int hmpc_from_montgomery(hmpc_context* ctx, hmpc_modulus* mod, uint64_t elements, const uint32_t* in, uint32_t* out)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!mod)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null modulus");
    }
    cudaError_t e = mod->kt->from_montgomery(out, in, elements, mod->h, ctx->stream);
    ctx->launches += elements ? 1 : 0;
    return e == cudaSuccess ? HMPC_OK : cuda_fail(e, "launching conversion");
}

int hmpc_lhe_enc(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint64_t batch,
                 const uint32_t* key_a, const uint32_t* key_b, const uint32_t* plaintext, int plaintext_ntt,
                 uint32_t* c0, uint32_t* c1)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!q || !p || !key_a || !key_b || !plaintext || !c0 || !c1)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    if (batch == 0)
    {
        return HMPC_OK;
    }
    const uint64_t elements = n * batch;
    const uint64_t lq = static_cast<uint64_t>(q->c.limbs);
    const uint64_t lp = static_cast<uint64_t>(p->c.limbs);
    const uint64_t poly_words = elements * lq;
    const int tc_splits = tc_plan_splits(q, n, batch);
    const bool tensor = tc_splits && n >= 16 && tc_supported(q) && p->c.limbs <= 2;
    // the tensor-core plan's last stages write the ciphertext themselves
    const uint64_t ws_words = tensor && tc_tail(q, n, false) ? 0 : 3 * poly_words;
    uint32_t* ws = ctx->scratch(std::max<uint64_t>(1, ws_words + (plaintext_ntt ? elements * lp : 0)));
    if (!ws)
    {
        return fail(HMPC_ERROR_OUT_OF_MEMORY, "allocating the encryption workspace");
    }
    uint32_t* coeff = ws + ws_words;
    const uint32_t* coefficients = plaintext;
    if (plaintext_ntt)
    {
        if (int rc = run_transform(ctx, p, n, batch, true, producer_tensor, 0, 0, plaintext, coeff))
        {
            return rc;
        }
        coefficients = coeff;
    }
    if (tensor)
    {
        // Tensor-core plan for q: the NTT is linear, so p*NTT(v) + NTT(lift(m))
        // is one transform of the small integers p*v + lift(m) drawn and lifted
        // in its first group, and p*NTT(w) one of p*w.  The three transforms
        // (u, p*v + lift(m), p*w) share every constant after their first
        // group, so they run stacked: three first-group launches, then the
        // other groups once over 3 * batch polynomials, the last stages'
        // kernel writing c0 and c1.  Every result is the reduced
        // representative, so the ciphertext is the reference's bit for bit.  RNG order as the
        // reference's plan: u, v, w (expr/cache.hpp:226-271).
        const TcSmallInput with_msg{coefficients, p};
        const TcSmallInput no_msg{nullptr, p};
        TcStackPart parts[3];
        parts[0].vx2 = 1;
        parts[1].vx2 = 20;
        parts[1].small = &with_msg;
        parts[2].vx2 = 20;
        parts[2].small = &no_msg;
        return run_tc_encrypt(ctx, q, n, batch, parts, TcCombine{key_a, key_b, c0, c1}, ws, tc_splits);
    }
    return encrypt_cuda_cores(ctx, q, p, n, batch, key_a, key_b, coefficients, c0, c1, ws, nullptr, false);
}

int hmpc_lhe_dec(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint64_t batch,
                 const uint32_t* s, const uint32_t* c0, const uint32_t* c1, int plaintext_ntt, uint32_t* out)
{
    return decrypt(ctx, q, p, n, batch, s, c0, c1, nullptr, plaintext_ntt, out);
}

int hmpc_lhe_dec2(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint64_t batch,
                  const uint32_t* s, const uint32_t* c0, const uint32_t* c1, const uint32_t* c2, int plaintext_ntt,
                  uint32_t* out)
{
    if (!c2)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null c2");
    }
    return decrypt(ctx, q, p, n, batch, s, c0, c1, c2, plaintext_ntt, out);
}

int hmpc_lhe_ct_mul(hmpc_context* ctx, hmpc_modulus* q, uint64_t elements, const uint32_t* a0, const uint32_t* a1,
                    const uint32_t* b0, const uint32_t* b1, uint32_t* d0, uint32_t* d1, uint32_t* d2)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!q || (elements && (!a0 || !a1 || !b0 || !b1 || !d0 || !d1 || !d2)))
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    cudaError_t e = q->kt->ct_mul(d0, d1, d2, a0, a1, b0, b1, elements, q->h, ctx->stream);
    if (e != cudaSuccess)
    {
        return cuda_fail(e, "launching ciphertext product");
    }
    ctx->launches += elements ? 1 : 0;
    return HMPC_OK;
}

int hmpc_ntt_forward_plain(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t batch,
                           const hmpc_producer* producer, uint32_t* out)
{
    if (!producer)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null producer");
    }
    return run_plain(ctx, mod, n, batch, false, producer->kind, producer->variance_x2, producer->security,
                     producer->src, out);
}

int hmpc_ntt_inverse_plain(hmpc_context* ctx, hmpc_modulus* mod, uint64_t n, uint64_t batch, const uint32_t* in,
                           uint32_t* out)
{
    return run_plain(ctx, mod, n, batch, true, producer_tensor, 0, 0, in, out);
}

int hmpc_lhe_keygen(hmpc_context* ctx, hmpc_modulus* q, hmpc_modulus* p, uint64_t n, uint32_t* s, uint32_t* a,
                    uint32_t* b)
{
    if (int rc = enter(ctx))
    {
        return rc;
    }
    if (!q || !p || !s || !a || !b)
    {
        return fail(HMPC_ERROR_INVALID_ARGUMENT, "null argument");
    }
    if (int rc = check_degree(n))
    {
        return rc;
    }
    uint32_t* e_poly = ctx->scratch(n * static_cast<uint64_t>(q->c.limbs));
    if (!e_poly)
    {
        return fail(HMPC_ERROR_OUT_OF_MEMORY, "allocating the key workspace");
    }
    const uint32_t bits = static_cast<uint32_t>(q->c.bits) + 80u;
    if (parts_applicable(q, p))
    {
        // s and p*e as one two-part transform, then b's draws and a in one
        // kernel; the nonces are b's, s's and e's in the reference's order
        const RngKey rng = ctx->rng();
        const uint32_t kinds[2] = {part_ternary, part_scaled};
        const uint32_t slots[2] = {1, 2};
        uint32_t* const outs[2] = {s, e_poly};
        // by the rule for two polynomials, whatever is set for one: the tiles that
        // spread one polynomial over the SMs are a pass too many for two (2^15 at 8
        // limbs 18.4 us by the rule, 24.6 in the shape tuned for one)
        if (int rc = run_parts(ctx, q, p, n, 1, 2, kinds, slots, outs, nullptr, nullptr, hmpc_modulus::TileChoice{}))
        {
            return rc;
        }
        const cudaError_t e = q->kt->lhe_key(a, b, s, e_poly, n, rng, static_cast<int>((bits + 31) / 32),
                                             bits % 32 ? (1u << (bits % 32)) - 1u : 0xffffffffu, !capturing(ctx),
                                             q->h, ctx->stream);
        if (e != cudaSuccess)
        {
            return cuda_fail(e, "launching the key combination");
        }
        ++ctx->launches;
        nonce_add(ctx->nonce, 3 * n);
        return HMPC_OK;
    }
    int rc = hmpc_sample_uniform(ctx, q, n, 80, b);
    if (!rc)
    {
        rc = run_transform(ctx, q, n, 1, false, producer_cbd, 1, 0, nullptr, s);
    }
    if (!rc)
    {
        rc = run_transform(ctx, q, n, 1, false, producer_cbd, 20, 0, nullptr, e_poly);
    }
    if (!rc)
    {
        const host::words pm = host::to_mont(q->c, p->c.q);
        cudaError_t e = q->kt->lhe_combine(a, b, n, s, e_poly, nullptr, n, pm.data(), q->h, ctx->stream);
        if (e != cudaSuccess)
        {
            return cuda_fail(e, "launching combine");
        }
        ++ctx->launches;
    }
    return rc;
}

}  // extern "C"
