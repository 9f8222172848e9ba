// Multi-limb modular arithmetic for sm_103a.
//
// Residues are L 32-bit limbs (least significant first) holding the fully
// reduced Montgomery representative x*R mod Q, R = 2^(32L) -- the same
// representation as hmpc's mod<Q> (hmpc/ints/mod.hpp:73-193), so any exact
// implementation of the operations below reproduces the reference bit for bit.
//
// Additions, subtractions and products use PTX carry chains
// (add.cc / addc / sub.cc / subc / mad.lo.cc / madc.hi.cc); each chain is a run
// of consecutive volatile asm statements with no other instruction between
// them touching the condition code.  The Montgomery product keeps its running
// value as two sums of 64-bit columns so that each word product is one wide
// multiply-add.
#pragma once

#include <cstdint>

namespace hmpc_gb300
{
    template<int L>
    struct Modulus
    {
        uint32_t q[L];
        uint32_t one[L];    // R mod Q (Montgomery one)
        uint32_t ninv;      // -Q^{-1} mod 2^32
        uint32_t bits;      // bit_width(Q - 1)
    };

    namespace ptx
    {
        __device__ __forceinline__ uint32_t add_cc(uint32_t a, uint32_t b)
        {
            uint32_t r;
            asm volatile("add.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
            return r;
        }
        __device__ __forceinline__ uint32_t addc_cc(uint32_t a, uint32_t b)
        {
            uint32_t r;
            asm volatile("addc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
            return r;
        }
        __device__ __forceinline__ uint32_t addc(uint32_t a, uint32_t b)
        {
            uint32_t r;
            asm volatile("addc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
            return r;
        }
        __device__ __forceinline__ uint32_t sub_cc(uint32_t a, uint32_t b)
        {
            uint32_t r;
            asm volatile("sub.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
            return r;
        }
        __device__ __forceinline__ uint32_t subc_cc(uint32_t a, uint32_t b)
        {
            uint32_t r;
            asm volatile("subc.cc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
            return r;
        }
        __device__ __forceinline__ uint32_t subc(uint32_t a, uint32_t b)
        {
            uint32_t r;
            asm volatile("subc.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(b));
            return r;
        }
        // d = lo(a*b) + c, sets carry
        __device__ __forceinline__ uint32_t mad_lo_cc(uint32_t a, uint32_t b, uint32_t c)
        {
            uint32_t r;
            asm volatile("mad.lo.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
            return r;
        }
        __device__ __forceinline__ uint32_t madc_lo_cc(uint32_t a, uint32_t b, uint32_t c)
        {
            uint32_t r;
            asm volatile("madc.lo.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
            return r;
        }
        __device__ __forceinline__ uint32_t mad_hi_cc(uint32_t a, uint32_t b, uint32_t c)
        {
            uint32_t r;
            asm volatile("mad.hi.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
            return r;
        }
        __device__ __forceinline__ uint32_t madc_hi_cc(uint32_t a, uint32_t b, uint32_t c)
        {
            uint32_t r;
            asm volatile("madc.hi.cc.u32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(c));
            return r;
        }
    }

    // r = (a + b) mod Q for a, b < Q (hmpc/ints/mod.hpp:17-34).
    template<int L>
    __device__ __forceinline__ void mod_add(uint32_t (&r)[L], const uint32_t (&a)[L], const uint32_t (&b)[L],
                                            const Modulus<L>& m)
    {
        uint32_t s[L];
        s[0] = ptx::add_cc(a[0], b[0]);
#pragma unroll
        for (int j = 1; j < L; ++j)
        {
            s[j] = ptx::addc_cc(a[j], b[j]);
        }
        uint32_t top = ptx::addc(0u, 0u);
        uint32_t d[L];
        d[0] = ptx::sub_cc(s[0], m.q[0]);
#pragma unroll
        for (int j = 1; j < L; ++j)
        {
            d[j] = ptx::subc_cc(s[j], m.q[j]);
        }
        uint32_t borrow = ptx::subc(top, 0u);  // 0xffffffff when s < Q
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            r[j] = borrow ? s[j] : d[j];
        }
    }

    // r = (a - b) mod Q for a, b < Q (hmpc/ints/mod.hpp:35-40).
    template<int L>
    __device__ __forceinline__ void mod_sub(uint32_t (&r)[L], const uint32_t (&a)[L], const uint32_t (&b)[L],
                                            const Modulus<L>& m)
    {
        uint32_t d[L];
        d[0] = ptx::sub_cc(a[0], b[0]);
#pragma unroll
        for (int j = 1; j < L; ++j)
        {
            d[j] = ptx::subc_cc(a[j], b[j]);
        }
        uint32_t mask = ptx::subc(0u, 0u);  // 0xffffffff on borrow
        r[0] = ptx::add_cc(d[0], m.q[0] & mask);
#pragma unroll
        for (int j = 1; j < L - 1; ++j)
        {
            r[j] = ptx::addc_cc(d[j], m.q[j] & mask);
        }
        if (L > 1)
        {
            r[L - 1] = ptx::addc(d[L - 1], m.q[L - 1] & mask);
        }
    }

    // r = -a mod Q (hmpc/ints/mod.hpp:327-341).
    template<int L>
    __device__ __forceinline__ void mod_neg(uint32_t (&r)[L], const uint32_t (&a)[L], const Modulus<L>& m)
    {
        uint32_t z[L];
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            z[j] = 0u;
        }
        mod_sub<L>(r, z, a, m);
    }

    // r = t mod Q for t = t[0..L] < 2Q: subtract Q once if t >= Q
    template<int L>
    __device__ __forceinline__ void reduce_once(uint32_t (&r)[L], const uint32_t (&t)[L + 1], const Modulus<L>& m)
    {
        uint32_t d[L];
        d[0] = ptx::sub_cc(t[0], m.q[0]);
#pragma unroll
        for (int j = 1; j < L; ++j)
        {
            d[j] = ptx::subc_cc(t[j], m.q[j]);
        }
        const uint32_t borrow = ptx::subc(t[L], 0u);
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            r[j] = borrow ? t[j] : d[j];
        }
    }

    // A value of L + 2 words held as two sums of 64-bit columns: `even` covers
    // words 0..EW-1 (columns at words 0, 2, ...), `odd` words 1..OW (columns
    // at words 1, 3, ...), EW and OW being L and L - 1 rounded up and down to
    // whole columns, and `top` is the count at word L + 1.  A word product
    // a_j * b lies exactly on one 64-bit column, so a row of products is two
    // chains of mad.lo.cc / madc.hi.cc pairs over adjacent words; each pair is
    // one wide multiply-add with carry in and out, where a single running sum
    // needs a further addition for each product.  Keeping the sums of even and odd
    // columns apart is a known way to whole carry chains (Emmart, Luitjens, Weems
    // and Woolley, "Optimizing Modular Multiplication for NVIDIA's Maxwell GPUs",
    // ARITH 2016, does it for 16-bit products).
    template<int L>
    struct Columns
    {
        static constexpr int EW = (L + 1) / 2 * 2;
        static constexpr int OW = L / 2 * 2;
        uint32_t even[EW];
        uint32_t odd[OW < 2 ? 2 : OW];
        uint32_t top;
        uint32_t pending;  // added at word 0 by the next row

        // even / odd = a * b
        __device__ __forceinline__ void set_product(const uint32_t (&a)[L], uint32_t b)
        {
#pragma unroll
            for (int j = 0; j < L; ++j)
            {
                const uint64_t w = static_cast<uint64_t>(a[j]) * b;
                uint32_t* column = j % 2 ? odd + (j - 1) : even + j;
                column[0] = static_cast<uint32_t>(w);
                column[1] = static_cast<uint32_t>(w >> 32);
            }
            top = 0u;
            pending = 0u;
        }

        // += a * b (+ pending at word 0 when First).  The odd chain goes first:
        // it starts at word 1, where the carry of the pending word's addition
        // belongs.
        template<bool First>
        __device__ __forceinline__ void add_product(const uint32_t (&a)[L], uint32_t b)
        {
            if constexpr (First)
            {
                even[0] = ptx::add_cc(even[0], pending);
            }
            if constexpr (L > 1)
            {
                odd[0] = First ? ptx::madc_lo_cc(a[1], b, odd[0]) : ptx::mad_lo_cc(a[1], b, odd[0]);
                odd[1] = ptx::madc_hi_cc(a[1], b, odd[1]);
#pragma unroll
                for (int j = 3; j < L; j += 2)
                {
                    odd[j - 1] = ptx::madc_lo_cc(a[j], b, odd[j - 1]);
                    odd[j] = ptx::madc_hi_cc(a[j], b, odd[j]);
                }
            }
            // the odd chain ends at word L + 1 (even L) or L (odd L)
            if constexpr (L % 2 == 0)
            {
                top = ptx::addc(top, 0u);
            }
            else if constexpr (L > 1 || First)
            {
                even[L] = ptx::addc_cc(even[L], 0u);
                top = ptx::addc(top, 0u);
            }
            even[0] = ptx::mad_lo_cc(a[0], b, even[0]);
            even[1] = ptx::madc_hi_cc(a[0], b, even[1]);
#pragma unroll
            for (int j = 2; j < L; j += 2)
            {
                even[j] = ptx::madc_lo_cc(a[j], b, even[j]);
                even[j + 1] = ptx::madc_hi_cc(a[j], b, even[j + 1]);
            }
            // the even chain ends at word L (even L) or L + 1 (odd L)
            if constexpr (L % 2 == 0)
            {
                odd[L - 1] = ptx::addc_cc(odd[L - 1], 0u);
            }
            top = ptx::addc(top, 0u);
        }

        // / 2^32, word 0 being zero: word k becomes word k - 1, so the two
        // column sums change places; the even sum's word 1 is left over
        __device__ __forceinline__ void shift()
        {
            uint32_t e[EW], o[OW < 2 ? 2 : OW];
            pending = even[1];
#pragma unroll
            for (int j = 0; j < EW; ++j)
            {
                e[j] = j < OW ? odd[j] : 0u;
            }
#pragma unroll
            for (int j = 0; j < OW; ++j)
            {
                o[j] = j + 2 < EW ? even[j + 2] : 0u;
            }
            (L % 2 == 0 ? o[L > 1 ? L - 1 : 0] : e[L % 2 ? L : 0]) = top;
            top = 0u;
#pragma unroll
            for (int j = 0; j < EW; ++j)
            {
                even[j] = e[j];
            }
#pragma unroll
            for (int j = 0; j < OW; ++j)
            {
                odd[j] = o[j];
            }
        }

        // words 0..L of the value, which is below 2^(32(L+1))
        __device__ __forceinline__ void value(uint32_t (&t)[L + 1]) const
        {
            t[0] = ptx::add_cc(even[0], pending);
#pragma unroll
            for (int j = 1; j < L; ++j)
            {
                t[j] = ptx::addc_cc(even[j], odd[j - 1]);
            }
            t[L] = ptx::addc(L % 2 ? even[L % 2 ? L : 0] : odd[L > 1 ? L - 1 : 0], 0u);
        }
    };

    // Montgomery product r = a*b*R^{-1} mod Q, a, b < Q, fully reduced, which is
    // what hmpc's schoolbook + separated REDC yields (hmpc/ints/mod.hpp:41-46,
    // hmpc/core/num/modulo.hpp:30-66): operand scanning, each row a * b_i and
    // the multiple of Q that clears word 0, on 64-bit columns (Columns).
    //
    // Bound by the wide integer multiply-add, of which it needs 2L^2 + L: on a
    // GB300 71.3 G products/s at L = 8 (9.7 T multiply-adds/s, 31 per SM and
    // clock), 249 G/s at L = 4.  The same rows as one running sum of 64-bit
    // multiply-adds reach 52.6 and 197 G/s: every product then needs two more
    // additions.  One limb has no chain to shorten and is slower on columns
    // (1.92 against 2.18 T/s), so it keeps the running sum.
    template<int L>
    __device__ __forceinline__ void mont_mul(uint32_t (&r)[L], const uint32_t (&a)[L], const uint32_t (&b)[L],
                                             const Modulus<L>& m)
    {
        uint32_t t[L + 1];
        if constexpr (L == 1)
        {
            const uint64_t ab = static_cast<uint64_t>(a[0]) * b[0];
            const uint32_t mq = static_cast<uint32_t>(ab) * m.ninv;
            const uint64_t c = (static_cast<uint64_t>(mq) * m.q[0] + static_cast<uint32_t>(ab)) >> 32;
            const uint64_t s = (ab >> 32) + c;
            t[0] = static_cast<uint32_t>(s);
            t[1] = static_cast<uint32_t>(s >> 32);
        }
        else
        {
            Columns<L> c;
            c.set_product(a, b[0]);
            c.template add_product<false>(m.q, c.even[0] * m.ninv);
            c.shift();
#pragma unroll
            for (int i = 1; i < L; ++i)
            {
                c.template add_product<true>(a, b[i]);
                c.template add_product<false>(m.q, c.even[0] * m.ninv);
                c.shift();
            }
            c.value(t);
        }
        reduce_once<L>(r, t, m);
    }

    // r = v * 2^(-32W) mod Q, fully reduced, for any W-word value: the reduction
    // with auxiliary power W (hmpc/core/num/modulo.hpp:30-66) -- W = L turns a
    // Montgomery form into the canonical value (hmpc/ints/mod.hpp:356-361), the
    // uniform sampler reduces W > L words (mod.hpp:210-215).  The rows of
    // mont_mul's reduction on a window of L + 2 words that takes in the value's
    // next word after each shift.  With fewer Rows, r = v * 2^(-32 Rows) mod Q
    // for v < Q * 2^(32 Rows).
    template<int L, int W, int Rows = W>
    __device__ __forceinline__ void redc(uint32_t (&r)[L], const uint32_t (&v)[W], const Modulus<L>& m)
    {
        uint32_t t[L + 1];
        if constexpr (L == 1)
        {
            // a running value of at most q that takes in one word a row, as in
            // mont_mul (10 M residues out of Montgomery form 16.4 us on columns, 14.4 so)
            static_assert(W - Rows <= 1);
            uint64_t s = 0;
#pragma unroll
            for (int i = 0; i < Rows; ++i)
            {
                s += v[i];
                const uint32_t low = static_cast<uint32_t>(s);
                s = (s >> 32) + ((static_cast<uint64_t>(low * m.ninv) * m.q[0] + low) >> 32);
            }
            s += Rows < W ? v[Rows < W ? Rows : 0] : 0u;
            t[0] = static_cast<uint32_t>(s);
            t[1] = static_cast<uint32_t>(s >> 32);
        }
        else
        {
            Columns<L> c;
            auto word = [&](int j) { return j < W ? v[j < W ? j : 0] : 0u; };
#pragma unroll
            for (int j = 0; j < Columns<L>::EW; ++j)
            {
                c.even[j] = word(j);
            }
#pragma unroll
            for (int j = 0; j < Columns<L>::OW; ++j)
            {
                c.odd[j] = j + 1 >= Columns<L>::EW ? word(j + 1) : 0u;
            }
            c.top = 0u;
            c.pending = 0u;
#pragma unroll
            for (int i = 0; i < Rows; ++i)
            {
                const uint32_t mq = (c.even[0] + c.pending) * m.ninv;
                c.template add_product<true>(m.q, mq);
                c.shift();
                if (i + 1 + L < W)
                {
                    uint32_t& last = L % 2 == 0 ? c.odd[L > 1 ? L - 1 : 0] : c.even[L % 2 ? L : 0];
                    last = ptx::add_cc(last, word(i + 1 + L));
                    c.top = ptx::addc(0u, 0u);
                }
            }
            c.value(t);
        }
        reduce_once<L>(r, t, m);
    }

    // t = (t + a * b) mod Q * R for t < Q * R and a, b < Q: one term of a sum of
    // products that is reduced once (redc<L, 2L, L>), so a term costs the L^2
    // wide multiply-adds of its product instead of a Montgomery product's
    // 2 L^2 + L.  The product is formed on two sums of 64-bit columns, as in
    // Columns, with every carry out of a row in the next column's low word.
    template<int L>
    __device__ __forceinline__ void add_product(uint32_t (&t)[2 * L], const uint32_t (&a)[L], const uint32_t (&b)[L],
                                                const Modulus<L>& m)
    {
        // [0]: columns at words 0, 2, ...; [1]: at words 1, 3, ...
        uint32_t columns[2][2 * L + 1];
#pragma unroll
        for (int k = 0; k < 2 * L + 1; ++k)
        {
            columns[0][k] = 0u;
            columns[1][k] = 0u;
        }
#pragma unroll
        for (int i = 0; i < L; ++i)
        {
#pragma unroll
            for (int parity = 0; parity < 2; ++parity)
            {
                uint32_t (&c)[2 * L + 1] = columns[parity];
                const int first = (i + parity) % 2;
#pragma unroll
                for (int j = first; j < L; j += 2)
                {
                    c[i + j] = j == first ? ptx::mad_lo_cc(a[j], b[i], c[i + j]) : ptx::madc_lo_cc(a[j], b[i], c[i + j]);
                    c[i + j + 1] = ptx::madc_hi_cc(a[j], b[i], c[i + j + 1]);
                    if (j + 2 >= L && i + j + 2 < 2 * L)
                    {
                        c[i + j + 2] = ptx::addc(c[i + j + 2], 0u);
                    }
                }
            }
        }
        t[0] = ptx::add_cc(t[0], columns[0][0]);
#pragma unroll
        for (int k = 1; k < 2 * L; ++k)
        {
            t[k] = ptx::addc_cc(t[k], columns[0][k]);
        }
        uint32_t high[L + 1];
        high[L] = ptx::addc(0u, 0u);
        t[1] = ptx::add_cc(t[1], columns[1][1]);
#pragma unroll
        for (int k = 2; k < 2 * L; ++k)
        {
            t[k] = ptx::addc_cc(t[k], columns[1][k]);
        }
        high[L] = ptx::addc(high[L], 0u);
        uint32_t r[L];
#pragma unroll
        for (int k = 0; k < L; ++k)
        {
            high[k] = t[L + k];
        }
        reduce_once<L>(r, high, m);
#pragma unroll
        for (int k = 0; k < L; ++k)
        {
            t[L + k] = r[k];
        }
    }

    template<int L>
    __device__ __forceinline__ void set_zero(uint32_t (&r)[L])
    {
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            r[j] = 0u;
        }
    }

    template<int L>
    __device__ __forceinline__ bool is_zero(const uint32_t (&a)[L])
    {
        uint32_t acc = 0u;
#pragma unroll
        for (int j = 0; j < L; ++j)
        {
            acc |= a[j];
        }
        return acc == 0u;
    }

    // a > b for L-limb unsigned integers
    template<int L>
    __device__ __forceinline__ bool greater(const uint32_t (&a)[L], const uint32_t (&b)[L])
    {
        // b - a borrows iff a > b
        uint32_t d = ptx::sub_cc(b[0], a[0]);
#pragma unroll
        for (int j = 1; j < L; ++j)
        {
            d = ptx::subc_cc(b[j], a[j]);
        }
        (void)d;
        return ptx::subc(0u, 0u) != 0u;
    }
}
