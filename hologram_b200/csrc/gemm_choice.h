// Which matmul kernel takes a product, its tile width and its K split: arithmetic on sizes alone, without CUDA, so that a test compiles it by
// itself. Tiles are 128 rows high, k-blocks 64 deep, a persistent CTA's tile is 256 columns wide.
#pragma once
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

namespace {
constexpr int BM = 128, BK = 64, PBN = 256;

// Which kernel takes a product of two row tiles or more: CTA pairs on 256 x 256 tiles (PAIRS), on 256 x 128 (HALF_PAIRS), 128 x 256 tiles
// walked by one CTA per SM (WALK), or a CTA per tile (tile_choice). What each takes, in ns, fitted to 249 shapes of 130 .. 4096 rows, each
// timed with all four: a start and, per round of items, an epilogue and what a k-block costs. Per SM and k-block a pair reads 32 KiB for
// 256 x 256 and 24 KiB for 256 x 128, CTAs with 128 x 64 tiles read 24 KiB each, two of them on an SM: that is why few tiles of a
// long k do better as halves on pairs (1024 x 8192 x 2048 43.7 -> 36.5 us, 446 x 2536 x 3440 31 -> 20, 1024 x 2048 x 2048 15.5 -> 14.8), and
// one round of whole tiles better than two of CTAs (2048 x 10240 x 2048 75 -> 63). Against a CTA per tile pairs have to gain 12 % of the
// estimate: between other kernels they lose what those gain by starting early (292 x 2048 x 512 in a bf16 encoder 17 -> 21 us; its block of
// 292 rows 180 us, 183 without the margin, 175 with it). `splits` is how many K slices a CTA per tile would take (linear_tile_choice):
// left out of the estimate, 256 x 8192 x 512 ran as four items on pairs in 34 us, its eight slices take 13. Over 583 Linear products of 130 ..
// 4096 rows, 407 of them with slices, each timed on all four, the choice is 1.0 % above the best on average (the worst 3410 x 2632 x 152, 31 us
// on CTAs, 20 on pairs); over the 407 it was 44 % without the slices' term.
// HOLO_GEMM_KERNEL names the kernel instead.
enum BigKernel { CTA_PER_TILE, WALK, PAIRS, HALF_PAIRS };
inline BigKernel big_choice(uint32_t sm_count, uint32_t m, uint32_t n, uint32_t kblocks, uint32_t splits) {
    const uint64_t sms = sm_count, pairs = sms / 2, kb = kblocks;
    const uint64_t mtiles = (m + BM - 1) / BM, ptiles = mtiles * ((n + PBN - 1) / PBN), quads = (uint64_t)((m + 255) / 256) * ((n + 255) / 256);
    const uint64_t halves = (uint64_t)((m + 255) / 256) * ((n + 127) / 128);
    if (mtiles < 2) return CTA_PER_TILE;
    if (const char* e = getenv("HOLO_GEMM_KERNEL")) {
        if (!strcmp(e, "tile")) return CTA_PER_TILE;
        if (!strcmp(e, "walk")) return WALK;
        if (!strcmp(e, "pairs")) return PAIRS;
        if (!strcmp(e, "halves")) return HALF_PAIRS;
    }
    auto up = [](uint64_t a, uint64_t b) { return (a + b - 1) / b; };
    const uint64_t grid = quads < pairs ? quads : pairs, rest = quads % grid;      // the last round's tiles run as halves where those fit one round
    const uint64_t tenths = quads / grid * 10 + (rest == 0 ? 0 : 2 * rest <= grid ? 6 : 10);
    const uint64_t whole_ns = 4500 + tenths * (3700 + 340 * kb) / 10, half_ns = 5200 + up(halves, pairs) * (1600 + 235 * kb);
    BigKernel best = CTA_PER_TILE;
    uint64_t best_ns;
    if (ptiles >= sms && quads >= pairs) {
        best = PAIRS;
        best_ns = whole_ns * 17 / 20;
    } else if (ptiles >= sms) {
        best = WALK;
        best_ns = 2700 + up(ptiles, sms) * (4250 + 366 * kb);
    } else {
        const uint64_t tiles128 = mtiles * ((n + 127) / 128), tiles64 = mtiles * ((n + 63) / 64);
        // K slices: fewer k-blocks each, then every warp of a CTA adds up 1 / (4 splits) of the tile's rows, a round trip to the peers a row
        if (splits > 1) best_ns = 5500 + 290 * up(kb, splits) + 530 * up(BM, 4 * splits);
        else best_ns = tiles128 < sms && tiles64 <= 2 * sms ? 5500 + (tiles64 <= sms ? 290 : 350) * kb : 6500 + up(tiles128, 2 * sms) * 480 * kb;
    }
    if (const char* e = getenv("HOLO_GEMM_PERSISTENT"))
        if (atoi(e) == 0) return CTA_PER_TILE;
    if (const char* e = getenv("HOLO_GEMM_PAIR"))
        if (atoi(e) == 0) return ptiles >= sms ? WALK : CTA_PER_TILE;
    // one CTA per tile starts beside the kernel before it, pairs with their whole shared memory do not
    const uint64_t of = best == CTA_PER_TILE ? 28 : 25;
    if (best != PAIRS && whole_ns * of / 25 < best_ns) best = PAIRS, best_ns = whole_ns * of / 25;
    return half_ns * of / 25 < best_ns ? HALF_PAIRS : best;
}

// Tile width and K split of the one-tile-per-CTA kernel. Compute-bound shapes (many row tiles) take 128-wide tiles, no split.
// One-row-tile shapes (decode) are HBM-bound: loaded HBM latency is 2-3 us, so 15-20 MB of
// weight bytes must be in flight across the chip. Measured on B200: with >= ~200 128-wide
// tiles, or >= one 64-wide tile per SM, no split is best (every CTA walks K in step with its
// neighbours, which keeps DRAM pages open); narrower outputs split K up to 8 ways inside a
// thread-block cluster, which reduces the slices through distributed shared memory.
inline void tile_choice(uint32_t sm_count, uint32_t m, uint32_t n, uint32_t kblocks, int* bn_out, uint32_t* splits_out) {
    const uint32_t mtiles = (m + BM - 1) / BM, slots = 2u * sm_count;
    int bn = 128;
    uint32_t splits = 1;
    const uint32_t tiles128 = mtiles * ((n + 127) / 128), tiles64 = mtiles * ((n + 63) / 64);
    if (mtiles == 1 && tiles128 < 200) {
        // 128-wide tiles read 256-byte weight rows instead of 128-byte ones; when two K slices of them still fit one
        // wave, that beats a 64-wide tile per SM (16 x 4096 x 14336: 26.0 -> 23.3 us)
        const uint32_t fit128 = tiles128 ? slots / tiles128 : 0;
        if (tiles64 >= sm_count && fit128 >= 2 && kblocks >= 8 && !getenv("HOLO_GEMM_OLD_NARROW")) {
            bn = 128;
            splits = 2;   // three slices (288 CTAs in clusters of 3) did not all become resident: 64 x 4096 x 12288 took 32.6 us against 25.3
        } else if (tiles64 >= sm_count) {
            bn = tiles64 > slots ? 128 : 64;   // 64-wide tiles that need a second wave lose to one wave of 128-wide ones
        } else {
            bn = tiles128 >= 16 ? 128 : 64;
            const uint32_t tiles = bn == 128 ? tiles128 : tiles64;
            uint32_t target = 240;   // CTAs aimed at; measured on the decoder step: 240 beats 192, 224 and 256 (1.735 / 1.745 / 1.741 / 1.779 ms)
            if (const char* e = getenv("HOLO_GEMM_CTA_TARGET")) target = (uint32_t)atoi(e) > 0 ? (uint32_t)atoi(e) : target;
            splits = (target + tiles - 1) / tiles;
            if (splits > 8) splits = 8;
            // k-blocks a slice keeps at least. Two: the 1/4 and 1/8 shards of the decoder's row-parallel products (K = 1024,
            // 512) then still spread over 64-128 CTAs; with eight they ran on 32 (measured on one GPU over a rank's shard of
            // the decoder step: 0.724 -> 0.648 ms at 1/8, 0.901 -> 0.822 ms at 1/4; one k-block per slice was no better)
            uint32_t min_kb = 2;
            if (const char* e = getenv("HOLO_GEMM_MIN_KB")) min_kb = (uint32_t)atoi(e) > 0 ? (uint32_t)atoi(e) : min_kb;
            if (splits > kblocks / min_kb) splits = kblocks / min_kb ? kblocks / min_kb : 1;
        }
    } else if (tiles128 < slots / 2) {
        bn = tiles64 <= slots ? 64 : 128;
    }
    *bn_out = bn;
    *splits_out = splits;
}
// A Linear product's: several row tiles of few columns (a router, an output product of a short prompt) split K as well, so that the slices
// fill the chip.
inline void linear_tile_choice(uint32_t sm_count, uint32_t m, uint32_t n, uint32_t kblocks, int* bn_out, uint32_t* splits_out) {
    tile_choice(sm_count, m, n, kblocks, bn_out, splits_out);
    const uint32_t mtiles = (m + BM - 1) / BM;
    if (mtiles < 2 || *splits_out != 1) return;
    uint32_t splits = sm_count / (mtiles * ((n + *bn_out - 1) / *bn_out));
    if (splits > kblocks / 4) splits = kblocks / 4;
    *splits_out = splits < 1 ? 1 : splits > 8 ? 8 : splits;
}
}  // namespace
