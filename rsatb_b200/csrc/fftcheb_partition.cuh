// How a transport call splits its workspace between the row stores of a section
// and the row stage's transform buffers.  Host arithmetic only.
#pragma once

#include <algorithm>
#include <cstddef>
#include <cstdint>

namespace rsatb_b200 {

struct FftchebSizes {
    size_t workspace;    // the call's bound
    size_t fixed;        // panels (and packed values) of the recurrence
    int64_t block_rows;
    int b;               // rows per block row
    int samples;
    int moments;
    size_t cplx;         // bytes of a stored complex value
    bool bastin;
    size_t part_bytes;   // fused Greenwood row stage: partial sums of one CTA; 0: cuFFT
    int max_ctas;        // and its CTAs where there is room for them
    int sections;        // at least this many (0: as few as fit)
};

struct FftchebPartition {
    int64_t sec_brows;   // block rows of a section
    int n_sections;
    int64_t chunk_rows;  // rows per cuFFT batch
    size_t e_bytes;      // transform buffer
    int ctas;            // of the fused stage
};

enum class FftchebFit { kFits, kNoSection, kNoRow };

// Bytes of a block row in the stores (both chains, 3 axes) and of a row in the
// cuFFT row stage (both sides' transform input, as much again for cuFFT's work
// area): M points of 16 bytes per sequence, Bastin two transforms of 2M.
inline size_t fftcheb_store_per_brow(const FftchebSizes& s) {
    return 2 * size_t(s.moments) * s.b * 3 * s.samples * s.cplx;
}
inline size_t fftcheb_row_points(const FftchebSizes& s) {
    return 2 * size_t(s.bastin ? 4 : 1) * size_t(s.moments) * 3 * s.samples;
}

// The cuFFT stage takes a quarter of what the fixed buffers leave, at most 2 GB
// (larger batches are no faster) but a whole row where the quarter holds one;
// the fused one a gathered chunk of up to 8,192 sequence pairs and partial sums
// for as many CTAs as an eighth holds (32 KB each: all of them from 80 MB up).
// The stores take the rest: fewer sections, each of which repeats the recurrence.
inline FftchebFit fftcheb_partition(const FftchebSizes& s, FftchebPartition* p) {
    const size_t store = fftcheb_store_per_brow(s);
    if (s.workspace <= s.fixed + store) return FftchebFit::kNoSection;
    const size_t avail = s.workspace - s.fixed;
    const size_t pair = 2 * size_t(s.moments) * s.cplx;  // one gathered pair of sequences
    const size_t per_row = fftcheb_row_points(s) * 16 * 2;
    const bool fused = s.part_bytes != 0;
    size_t budget = fused ? std::max(pair, std::min(avail / 4, 8192 * pair))
                          : std::min(avail / 4, std::max(size_t(2) << 30, per_row));
    p->chunk_rows = std::max<int64_t>(1, int64_t(budget / per_row));
    p->sec_brows = int64_t((avail - budget) / store);
    if (p->sec_brows < 1) return FftchebFit::kNoRow;
    p->ctas = 0;
    if (fused) {
        const auto ctas_in = [&](size_t bytes) {
            return int(std::max<size_t>(1, std::min(size_t(s.max_ctas), bytes / s.part_bytes)));
        };
        p->ctas = ctas_in(avail / 8);
        const size_t taken = budget + size_t(p->ctas) * s.part_bytes;
        if (taken + store <= avail) {
            p->sec_brows = int64_t((avail - taken) / store);
        } else {  // one block row of stores: the row stage takes what it leaves
            p->sec_brows = 1;
            const size_t room = avail - store;
            p->ctas = ctas_in(room / 2);
            const size_t part = size_t(p->ctas) * s.part_bytes;
            budget = std::max(pair, std::min(budget, room - std::min(room, part)));
        }
    }
    if (s.sections > 0)
        p->sec_brows = std::min(p->sec_brows, (s.block_rows + s.sections - 1) / s.sections);
    p->sec_brows = std::min(p->sec_brows, s.block_rows);
    p->n_sections = int((s.block_rows + p->sec_brows - 1) / p->sec_brows);
    // Balanced: the store is no larger than the section count needs.
    p->sec_brows = (s.block_rows + p->n_sections - 1) / p->n_sections;
    p->chunk_rows = std::min(p->chunk_rows, p->sec_brows * s.b);
    p->e_bytes = fused ? budget : fftcheb_row_points(s) * size_t(p->chunk_rows) * 16;
    return FftchebFit::kFits;
}

}  // namespace rsatb_b200
