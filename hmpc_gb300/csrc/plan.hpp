// Pass planner of the one-butterfly-per-thread transform (pair.cuh).
#pragma once

#include <algorithm>
#include <cstdint>
#include <vector>

#include "pair.cuh"

namespace hmpc_gb300
{
    struct BitRange
    {
        int lo, hi, c;
    };

    struct PairPlan
    {
        PairPassParams params;
        unsigned grid = 0;
        unsigned block = 0;
        size_t smem = 0;
    };

    // Passes of the one-butterfly-per-thread transform (pair.cuh): the low
    // `tile_bits` index bits are one pass over contiguous elements, the bits
    // above them column passes of at least 2^col_bits consecutive elements.
    // tile_bits 0: the shape by the rule below, measured over 1 to 256
    // polynomials of 2^12..2^20, 2 to 8 limbs, all shapes of tile bits 6..10 and
    // column bits 2..5.  Fewest passes first: 2^13 takes two at tile bits 8,
    // 2^15 at 9, 2^16 at 9 with column bits 2 (127 against 135 us with a third
    // pass, 32 polynomials at 4 limbs), 2^17 at 10.  Above that the shapes are
    // within a few per cent of one another, except where there is at most one
    // warp per scheduler: then the smaller tile spreads it over twice the SMs
    // (one polynomial of 2^15 at 8 limbs: 15.0 us in three passes at tile bits
    // 8, 18.5 in two at 9; two polynomials: 24.6 and 18.4).
    // block: threads of every pass's blocks, at least 2^(tile_bits - 1) (0: by
    // the size).
    inline std::vector<PairPlan> plan_pairs(int limbs, int log_n, uint64_t batch, bool inverse, int tile_bits,
                                            int col_bits, unsigned block = 0)
    {
        if (tile_bits == 0)
        {
            // one warp per scheduler or less: small tiles spread over the SMs
            const bool sparse = (batch << (log_n - 1)) <= 152ull * 128;
            tile_bits = log_n <= 13 || (sparse && log_n <= 15) ? 8 : log_n <= 16 ? 9 : 10;
            col_bits = log_n == 16 ? 2 : 3;
        }
        tile_bits = std::min(tile_bits, 10);
        const int contiguous = std::min(log_n, tile_bits);
        const int rest = log_n - contiguous;
        const int widest = std::max(1, tile_bits - col_bits);
        const int columns = (rest + widest - 1) / widest;
        std::vector<BitRange> ranges;  // forward order: top bits first
        int hi = log_n;
        for (int i = 0; i < columns; ++i)
        {
            const int w = rest / columns + (i < rest % columns ? 1 : 0);
            ranges.push_back({hi - w, hi, std::max(0, std::min({tile_bits - w, hi - w, 5}))});
            hi -= w;
        }
        ranges.push_back({0, contiguous, 0});
        if (inverse)
        {
            std::reverse(ranges.begin(), ranges.end());
        }
        std::vector<PairPlan> out;
        for (const BitRange& rg : ranges)
        {
            PairPlan pp{};
            PairPassParams& p = pp.params;
            p.log_n = static_cast<uint32_t>(log_n);
            p.part_polys = batch;
            p.w = static_cast<uint32_t>(rg.hi - rg.lo);
            p.c = static_cast<uint32_t>(rg.c);
            p.row_shift = static_cast<uint32_t>(rg.lo);
            p.tiles = batch << (log_n - static_cast<int>(p.w + p.c));
            const unsigned tile_threads = 1u << (p.w + p.c - 1);
            pp.block = block ? block : std::max(tile_threads, p.tiles * tile_threads >= 152ull * 256 ? 128u : 32u);
            const uint64_t per_block = pp.block / tile_threads;
            pp.grid = static_cast<unsigned>((p.tiles + per_block - 1) / per_block);
            pp.smem = 2ull * static_cast<size_t>(limbs) * pp.block * sizeof(uint32_t);
            out.push_back(pp);
        }
        return out;
    }
}
