// How the matrix kernel (umma_matmul.cu) splits a product over the SMs: a function of the descriptors alone, in plain C++, so that what it
// chooses can be checked without a GPU.
#pragma once

#include <algorithm>
#include <cmath>
#include <cstdint>

#include "dfgpu.h"

namespace dfgpu {
namespace {

constexpr int kRows = 128;            // rows of A per CTA and tile
constexpr int kRowBytes = 128;        // one swizzled shared-memory row: 64 16-bit values or 128 codes of K
constexpr int kABytes = kRows * kRowBytes;
constexpr int kStageBox = 128 * 128;  // one staging tile: 128 rows x 128 bytes of C
constexpr int kMaxStages = 16;
constexpr int kMaxSteps = DFGPU_MAX_EPILOGUE;
constexpr int kSmemBudget = 227 * 1024 - 1024;   // (1 KB of slack aligns the tiles)

enum Kind { kSixteen = 0, kCodes = 1, kScaled = 2, kPieces = 3, kSummed = 4, kScaledSummed = 5, kCodesSummed = 6, kPiecesSummed = 7 };

// One product as the kernel sees it; the descriptors alone decide everything but the pointers.
struct Problem {
    int kind;
    int64_t M, N, K;
    int64_t a_ld, b_ld, c_ld;
    bool b_mn_major;
    int in_bytes, out_bytes, out_dtype;
    bool direct_stores;       // C's rows are off the 16-byte boundaries, or E5M2: no TMA store
    int64_t a_rows, b_rows;   // rows the maps span (pieces: three matrices on top of one another)
};

// Few rows take little of a stage, so that more stages fit. (A product still reads 128 rows: ring_bytes() keeps the last
// stage's inside the allocation.)
inline int rows_of_a(const Problem& p, int cg) { return cg == 1 && p.M < kRows ? static_cast<int>((p.M + 7) / 8 * 8) : kRows; }
inline bool has_pieces(const Problem& p) { return p.kind == kPieces || p.kind == kPiecesSummed; }
inline bool in_registers(const Problem& p) { return p.kind == kSummed || p.kind == kCodesSummed; }
inline bool scaled(const Problem& p) { return p.kind == kScaled || p.kind == kScaledSummed; }
inline bool sixteen_bits(const Problem& p) { return p.kind == kSixteen || has_pieces(p) || p.kind == kSummed; }
// Columns of B that a CTA loads for bn / cg of its own: N-major copies come in whole boxes, so that 96 columns cost 128.
inline int loaded_columns(const Problem& p, int bn, int cg) {
    const int chunk = sixteen_bits(p) ? 64 : 128;
    return p.b_mn_major ? (bn / cg + chunk - 1) / chunk * chunk : bn / cg;
}
inline int stage_bytes(const Problem& p, int bn, int cg, int a_rows) { return (a_rows + loaded_columns(p, bn, cg)) * kRowBytes * (has_pieces(p) ? 3 : 1) + (scaled(p) ? 2048 : 0); }
inline int ring_bytes(int stages, int stage_size) { return (stages - 1) * stage_size + std::max(stage_size, kABytes); }
inline int stages_that_fit(int stage_size, int budget) {
    int stages = std::min(kMaxStages, budget / stage_size);
    while (stages > 2 && ring_bytes(stages, stage_size) > budget) --stages;
    return stages;
}

struct Shape {
    int cg, bn, splits, k_per_split;
    int64_t tiles;
    int64_t halved;   // tiles of the last round that are cut into halves
    double clocks;
};

// The shape with the fewest estimated clocks. One K block of a CTA costs the longest of
//   products       2.3 bn clocks (128 rows per SM, 16-bit and FP8 alike: a block is 128 bytes of K)
//   shared memory  every operand byte written and read once: 1.8 (rows of A + columns of B)
//   L2             the same bytes at 48 a clock and SM, 6300 for all SMs that fetch, or what the ring holds per 3400 clocks of latency
// and a round over the SMs costs its blocks (a last round that at most half fills the SMs is cut into half tiles: 4096^3 is 512
// tiles of 128 x 256 on 148 SMs, three rounds and 68 tiles, which become 136 halves) and, where there are several, an epilogue of 12 bn.
// Splitting K divides the blocks and adds an exchange that grows with the partial tile, 800 + 0.31 x rows x bn (1000 more with block
// scales, whose six loading warps also fall behind once they have more than a block each), and shares out the epilogue, which counts
// for every column that a group of its warps takes: 14 clocks for a full operand that is not loaded ahead (`operands` of them), 20 for E4M3 codes, and 300 in
// every round where a thread stores its row element by element, as K in splits is added up and stored by neighbouring threads side by side.
// Former costs -> these, in us: 777 x 4096 x 3072 bf16 [K, N] 26.9 (256 columns) -> 21.6 (192), 2050 x 1040 x 1040 13.0 -> 11.5, MXFP8
// 15 x 1632 x 816 7.7 -> 6.3 (more splits). Where an exchange of 230 split K: 1 x 136 x 3648 bf16 4.0 whole, 5.0 in two. With bias, ReLU and a
// full f32 operand, 128 x 384 x 384 f16: 6.0 in six, 7.5 whole; with a bf16 one 1059 x 368 x 104 6.4 and 7.7. With rows of C off the 16-byte boundaries 128 x 512 x 1280 f16 6.9 in splits, 12.9
// whole; FP8 128 x 1024 x 2688 to E5M2 10.2 and 29.2, 78 x 912 x 336 to E4M3 7.5 and 9.6.
// f32 results and f32 operands (pieces) keep the former costs. Those split K more often, and an accumulator is off by 2^-24 of its value
// for every block it takes, which a 16-bit result does not show and an f32 result does (128 x 640 x 3840 bf16 to f32: 1.7e-7 from
// 64 bits in four splits, 5.9e-7 in one; 128 x 3328 x 1536 4.0e-7 and 6.4e-7). For pieces they are the quicker too (25 x 6312 x 6632 165 us, 196).
// MATMUL_FP8's Amax_C is an f32 result beside a C of any type: new costs, but no accumulator of more blocks than by the former ones (956
// products, Amax_C 5.9e-8 from 64 bits in the root mean square that way, 6.2e-8 without).
inline Shape choose_shape(const Problem& p, int operands) {
    const int64_t blocks = (p.K * p.in_bytes + kRowBytes - 1) / kRowBytes;
    constexpr int clusters_at_once[9] = {0, 148, 74, 45, 33, 26, 22, 15, 15};   // (cudaOccupancyMaxActiveClusters, by CTAs per cluster)
    const int sms = 148;   // (a function of the shape alone: the count this library is built for)
    const bool former_only = p.out_dtype == DFGPU_F32 || has_pieces(p), both = p.kind == kCodes && !former_only;
    Shape best{0, 0, 0, 0, 0, 0, 0.0}, former_best = best, shapes[2 * 4 * 8];
    int count = 0;
    auto take = [](Shape& least, const Shape& shape) {
        if (least.cg == 0 || shape.clocks < least.clocks) least = shape;
    };
    for (int cg = 1; cg <= 2; ++cg)
        for (int bn = 64; bn <= 256; bn += 64) {
            const int chunk = sixteen_bits(p) ? 64 : 128;   // columns of one N-major copy
            if (p.b_mn_major && (bn / cg) % chunk != 0 && !(cg == 2 && bn == 192 && !scaled(p) && !former_only)) continue;
            if (p.out_dtype == DFGPU_E4M3 && bn % 128 != 0) continue;   // (whole 128-byte boxes)
            if (scaled(p) && bn % 128 != 0) continue;           // (whole chunks of column scales)
            if (cg == 2 && bn < 128) continue;
            if ((in_registers(p) || p.kind == kScaledSummed || p.kind == kPiecesSummed) && bn > 128) continue;   // (a row's sums live in registers, or beside two accumulators)
            if (bn > chunk && bn >= 2 * ((p.N + 63) / 64 * 64)) continue;  // (half the tile would be empty)
            const int64_t m_tiles = (p.M + kRows * cg - 1) / (kRows * cg), n_tiles = (p.N + bn - 1) / bn, tiles = m_tiles * n_tiles;
            const int rows = rows_of_a(p, cg), stage_size = stage_bytes(p, bn, cg, rows);
            if (2 * stage_size > kSmemBudget - 2 * kStageBox - 1024) continue;   // (pieces: a second stage has to fit)
            for (int splits = 1; splits <= (cg == 1 ? 8 : 1); ++splits) {
                if (splits > 1 && (bn > 128 || splits > blocks || tiles * splits > sms)) break;
                const int64_t k_per_split = (blocks + splits - 1) / splits;
                if (splits > 1 && k_per_split * (splits - 1) >= blocks) continue;   // (no CTA without a block)
                const int64_t slots = cg == 2 ? sms / 2 : clusters_at_once[splits];
                double rounds = static_cast<double>((tiles + slots - 1) / slots);
                int64_t halved = 0;
                const int half = bn / 2;
                const bool halves = splits == 1 && half / cg >= 64 && (!p.b_mn_major || half / cg % chunk == 0) && half % (scaled(p) || p.out_dtype == DFGPU_E4M3 ? 128 : 64) == 0;
                if (halves && tiles > slots && tiles % slots != 0 && 2 * (tiles % slots) <= slots) {
                    halved = tiles % slots;
                    rounds -= 0.45;
                }
                const double in_flight = static_cast<double>(stages_that_fit(stage_size, kSmemBudget - 2 * kStageBox)) * stage_size;
                Shape shape{cg, bn, splits, static_cast<int>(k_per_split), tiles, halved, 0.0};
                const bool whole_boxes = !p.b_mn_major || (bn / cg) % chunk == 0;
                if (former_only || (both && whole_boxes)) {
                    const double products = has_pieces(p) ? 6.0 : 1.0, pieces = has_pieces(p) ? 3.0 : 1.0;
                    const double summed = in_registers(p) ? 150.0 + 2.0 * bn : (p.kind == kScaledSummed ? 250.0 + 3.0 * bn : 0.0);   // the epilogue's loads and additions of a block
                    const double block = std::max({summed, products * 2.0 * bn, (products + pieces) * (rows + bn / cg), pieces * (rows + bn / cg) * kRowBytes / std::min(48.0, in_flight / 2300.0)});
                    shape.clocks = rounds * (k_per_split * block) + 2000.0 + bn * 6.0 + (splits > 1 ? (scaled(p) ? 5000.0 : 2500.0) : 0.0) + (cg == 2 ? 1500.0 : 0.0);
                    take(former_best, shape);
                }
                if (!former_only) {
                    const int columns = loaded_columns(p, bn, cg);
                    const double active = static_cast<double>(std::min<int64_t>(sms, tiles * cg * splits));
                    const double rate = std::min({48.0, 6300.0 / active, in_flight / 3400.0});
                    const double block = std::max({2.3 * bn, 0.9 * (2 * rows + bn / cg + columns), (rows + columns) * kRowBytes / rate});
                    const int box = p.direct_stores ? 32 : kRowBytes / p.out_bytes, serial = std::min(bn, (bn / box + 1) / 2 * box);   // (columns that one epilogue group takes)
                    const double exchange = splits > 1 ? 800.0 + 0.31 * std::min<double>(rows, static_cast<double>(p.M)) * bn + (scaled(p) ? 1000.0 : 0.0) : 0.0;
                    const double stores = p.direct_stores ? 300.0 * std::ceil(rounds) : (p.out_dtype == DFGPU_E4M3 ? 20.0 : 0.0);
                    const double epilogue = splits > 1 ? 0.0 : (14.0 * operands + stores) * serial;
                    shape.clocks = rounds * (k_per_split * block + (rounds > 1.0 ? 12.0 * bn : 0.0)) + 2000.0 + exchange + epilogue + (scaled(p) && k_per_split > 6 ? 450.0 : 0.0) + (cg == 2 ? 1480.0 : 0.0);
                    if (both) shapes[count++] = shape;
                    else take(best, shape);
                }
            }
        }
    if (former_only) return former_best;
    for (int i = 0; i < count; ++i)
        if (shapes[i].k_per_split <= former_best.k_per_split) take(best, shapes[i]);
    return best;
}

}  // namespace
}  // namespace dfgpu
