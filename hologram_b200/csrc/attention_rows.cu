// Attention of whole 16-bit sequences (the legacy Attention call: no cache, causal or not, grouped-query) on tcgen05.
//
// One CTA takes one or two tiles of 128 query rows of a head and walks the keys in tiles of 128:
//   warp 0     TMA producer: the query tiles once, K and V tiles through rings of two
//   warp 1     tcgen05.mma issuer: S = Q K^T, then O += P V with P read from TMEM, the two query tiles in turn
//   warps 2-9  softmax, one group of four warps per query tile, one thread per row: running maximum, exponentials, row sum;
//              a row's O is rescaled in TMEM only when its maximum grows by more than 2^GROWTH
// The weights are f32 values, and 16 bits of them would not do: each goes to the tensor core as two 16-bit terms, the rounded value
// and the rounded remainder, so O costs two products. That holds a weight to 2^-17 of itself in bf16 and to 2^-23 in f16 (f32: 2^-24),
// and the tensor core's sums over long sequences lose about 2^-18 more. It is less than the general routine keeps, whose weights and
// sums are f32; what shows is the output's own 16 bits. Error against 64 bits, here / there, normal inputs: bf16 16 keys 0.003279 /
// 0.003283, 512 causal 0.003178 / 0.003177, 2048 0.003321 / 0.003317; f16 0.0002061 / 0.0002061, 0.0001992 / 0.0001992, 0.0002077 /
// 0.0002076. Scores need no split: products of 16-bit values are exact in f32.
// TMEM (512 columns): S at 0 and 128, overwritten by its weights (first terms, then second terms), O at 256 and 384.
// Bound: three products per score on the tensor core (1536 cycles a 128 x 128 tile at dim 128) against 1024 cycles of ex2.
// What bounds it is the issuer: while it waits nothing is queued, so the next scores are issued right behind a product (on what that rests
// stands at product_ss; the scores' commit covers the product too) and the descriptors' words step by constants.
// 2048 rows, 32 heads over 8, dim 128, causal, bf16: one CTA per row on the CUDA cores took 48450 us, this 58.7 us (67.6 with a wait
// between a product and the next scores; the tensor core's share 24 us); all keys 122 -> 99.4, dim 64 108 -> 93. Error against 64 bits
// 0.0032 in all: the output's own 16 bits. Rounding the two terms with integer operations instead of conversions: 64.4 -> 68.9.
//
// A weight of zero times an infinite or NaN value is NaN, and so is the sum of an infinite value's two terms: a value that is not
// finite spoils its column of O in every row of the tile. compute_again sets that right.
#include "attention_tile.cuh"

namespace {

constexpr int ROWS_WARPS = 10;
constexpr float GROWTH = 8.0f;

struct RowsParams {
    HoloAttnArgs a;
    uint32_t* status;
    float to_log2;      // score to exponent of two
    uint32_t nq, chunks;
};

__device__ __forceinline__ uint32_t pack_f16(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}

__device__ __forceinline__ float2 widen_f16(uint32_t v) {
    float2 r;
    asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %2;\ncvt.f32.f16 %0, l;\ncvt.f32.f16 %1, h;\n}" : "=f"(r.x), "=f"(r.y) : "r"(v));
    return r;
}

// Two weights as a pair of 16-bit terms and the pair of their remainders
template <bool F16>
__device__ __forceinline__ void split_weights(float x, float y, uint32_t& first, uint32_t& second) {
    if (F16) {
        first = pack_f16(x, y);
        const float2 f = widen_f16(first);
        second = pack_f16(x - f.x, y - f.y);
    } else {
        first = pack_bf16(x, y);
        second = pack_bf16(x - __uint_as_float(first << 16), y - __uint_as_float(first & 0xffff0000u));
    }
}

template <bool F16>
__device__ __forceinline__ float2 widen_pair(uint32_t v) {
    return F16 ? widen_f16(v) : make_float2(__uint_as_float(v << 16), __uint_as_float(v & 0xffff0000u));
}

// Shared memory behind the tiles: barriers from `bars` on, flags, then what a row's weights refer to and what is to be computed again of it
struct RowsTail {
    uint32_t q, k, v, bars;     // offsets
    __device__ __forceinline__ RowsTail(uint32_t nq, uint32_t tile_bytes) : q(0), k(nq * tile_bytes), v(k + 2 * tile_bytes), bars(v + 2 * tile_bytes) {}
    static constexpr uint32_t AGAIN_BAR = 120, AGAIN_SCORES_BAR = 128, TMEM = 144, ABORT = 148, AGAIN = 152, SPOILT = 160, ROWS = 256, BYTES = 256 + 256 * 8;
};
enum { ROW_STAYS = 0, ROW_COLUMNS = 1, ROW_ALL = 2 };
constexpr float WILD = 0x1p22f;     // from here on rounding moves exponents of two by whole units: weights no longer have the range that the tiles count on

// Columns that are not finite in a row whose sum is, and whole rows with a sum that is not or with exponents beyond WILD: scores by
// another product, weights in f32, only the keys that a row sees, one thread a row. All threads come here, with every load and product
// at its end; nobody leaves early, they meet after each tile. One column of 2048 rows, 32 heads over 8, dim 128, causal: 285 us instead
// of 69, which is 59 by now (redoing the rows one after another 124000, the general routine 48400); 12 heads x 128 rows, dim 64 19 instead of 6.7 (1580,
// 90); 16 rows 12 instead of 5.7 (89, 9). That it can be reached costs finite inputs, in a loop that is the same, 0 to 2 % in bf16
// and 0 to 4 % in f16 (as measured at 67.4 and 70.0 us of this size), called or inlined: the registers are given out differently.
template <bool F16>
__device__ __noinline__ void compute_again(const CUtensorMap& map_k, const CUtensorMap& map_v, const RowsParams& p, uint8_t* sm, uint32_t tmem_base, uint32_t row0,
                                           uint32_t n0, uint32_t n1) {
    const HoloAttnArgs& a = p.a;
    const uint32_t tile_bytes = p.chunks * TILE_CHUNK, base = smem_u32(sm), warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const RowsTail at(p.nq, tile_bytes);
    const uint32_t bar = base + at.bars + RowsTail::AGAIN_BAR, bar_s = base + at.bars + RowsTail::AGAIN_SCORES_BAR;
    volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(sm + at.bars + RowsTail::ABORT);
    uint32_t* s_spoilt = reinterpret_cast<uint32_t*>(sm + at.bars + RowsTail::SPOILT);      // a bit per column
    const uint32_t plane = blockIdx.x, kv_plane = plane / a.h * a.hkv + plane % a.h / (a.h / a.hkv);
    const uint32_t q = warp < 2 ? 0u : (warp - 2) >> 2, quarter = warp & 3u, row = row0 + q * 128 + quarter * 32 + lane, n = warp < 2 ? 0u : q ? n1 : n0;
    const uint32_t limit = a.all_new ? a.m : min(row + 1, a.m), seen = a.all_new ? a.m : min(row - lane + 32, a.m);     // keys of this row, of any row of the warp
    const uint32_t tmem_s = tmem_base + q * 128 + ((quarter * 32u) << 16), tmem_o = tmem_s + 256;
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    float top = 0.0f, sum = 0.0f;
    uint32_t mine[4] = {0, 0, 0, 0};
    if (n) {
        const float2 about = reinterpret_cast<const float2*>(sm + at.bars + RowsTail::ROWS)[threadIdx.x - 64];
        top = about.x;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            if (16 * g >= a.d) break;
            uint32_t o[16], bits = 0;
            tmem_ld16(tmem_o + 16 * g, o);
#pragma unroll
            for (int x = 0; x < 16; ++x)
                if (about.y == ROW_ALL || !isfinite(__uint_as_float(o[x]))) bits |= 1u << x;
            if (about.y != ROW_STAYS) mine[g >> 1] |= bits << (16 * (g & 1));
        }
#pragma unroll
        for (int w = 0; w < 4; ++w)
            if (mine[w]) atomicOr(s_spoilt + w, mine[w]);
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    auto spoilt = [&](uint32_t g) { return (s_spoilt[g >> 1] >> (16 * (g & 1u)) & 0xffffu) != 0; };
#pragma unroll 1
    for (uint32_t t = 0; t < max(n0, n1); ++t) {
        if (threadIdx.x == 0 && !*s_abort) {
            mbar_arrive_expect_tx(bar, 2 * tile_bytes);
            for (uint32_t c = 0; c < p.chunks; ++c) {
                tma_load_3d(base + at.k + c * TILE_CHUNK, &map_k, (int)(64 * c), (int)(t * 128), (int)kv_plane, bar);
                tma_load_3d(base + at.v + c * TILE_CHUNK, &map_v, (int)(64 * c), (int)(t * 128), (int)kv_plane, bar);
            }
            if (mbar_wait(bar, t & 1u, s_abort, p.status)) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t idesc = (1u << 4) | (F16 ? 0u : (1u << 7) | (1u << 10)) | ((128u >> 3) << 17) | ((128u >> 4) << 24);
                const uint64_t dq = smem_desc(base + at.q, 16, 1024), dk = smem_desc(base + at.k, 16, 1024);
                for (uint32_t i = 0; i < 2; ++i)
                    for (uint32_t k = 0; t < (i ? n1 : n0) && k < a.d / 16; ++k) {
                        const uint32_t off = (k >> 2) * (TILE_CHUNK >> 4) + 2 * (k & 3u);
                        umma_bf16(tmem_base + i * 128, dq + i * (tile_bytes >> 4) + off, dk + off, idesc, k != 0);
                    }
                umma_commit(bar_s);
            } else {
                // nothing may still be on its way into this CTA's shared memory when it ends
                for (uint32_t it = 0; it < WAIT_LIMIT && !mbar_try_wait(bar, t & 1u); ++it) __nanosleep(64);
            }
        }
        __syncwarp();
        if (t < n) {
            bool ok = mbar_wait(bar, t & 1u, s_abort, p.status) && mbar_wait(bar_s, t & 1u, s_abort, p.status);
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
#pragma unroll 1
                for (uint32_t c = 0; c < 128; c += 16) {
                    uint32_t s[16];
                    tmem_ld16(tmem_s + c, s);
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        // `top` is at most GROWTH below the maximum: no weight is above 1. Not fused: a large exponent's rounding cancels
                        const float w = exp2f(__fsub_rn(__fmul_rn(__uint_as_float(s[x]), p.to_log2), top) - GROWTH);
                        s[x] = __float_as_uint(w);
                        if (t * 128 + c + x < limit) sum += w;
                    }
                    tmem_st16(tmem_s + c, s);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
#pragma unroll 1
                for (uint32_t g = 0; 16 * g < a.d; ++g) {
                    if (!spoilt(g)) continue;
                    uint32_t o[16];
                    if (t > 0) tmem_ld16(tmem_o + 16 * g, o);
                    float acc[16];
#pragma unroll
                    for (int x = 0; x < 16; ++x) acc[x] = t > 0 ? __uint_as_float(o[x]) : 0.0f;
                    const uint8_t* values = sm + at.v + (g >> 2) * TILE_CHUNK;
#pragma unroll 1
                    for (uint32_t c = 0; c < 128 && t * 128 + c < seen; c += 16) {
                        uint32_t w[16];
                        tmem_ld16(tmem_s + c, w);
#pragma unroll
                        for (int x = 0; x < 16; ++x) {
                            const uint32_t key = c + x;     // the row's 16-byte units stand at their number xor key % 8 (128-byte swizzle)
                            const uint4* v = reinterpret_cast<const uint4*>(values + key * 128);
                            const uint4 lo = v[(2 * (g & 3u)) ^ (key & 7u)], hi = v[(2 * (g & 3u) + 1) ^ (key & 7u)];
                            if (t * 128 + key < limit) {
                                const uint32_t e[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
                                for (int y = 0; y < 8; ++y) {
                                    const float2 f = widen_pair<F16>(e[y]);
                                    acc[2 * y] = fmaf(__uint_as_float(w[x]), f.x, acc[2 * y]);
                                    acc[2 * y + 1] = fmaf(__uint_as_float(w[x]), f.y, acc[2 * y + 1]);
                                }
                            }
                        }
                        __syncwarp();
                    }
#pragma unroll
                    for (int x = 0; x < 16; ++x) o[x] = __float_as_uint(acc[x]);
                    tmem_st16(tmem_o + 16 * g, o);
                }
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            }
        }
        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
        __syncthreads();
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    }
    if (n && !*s_abort) {
        uint16_t* out = (uint16_t*)a.out + ((uint64_t)plane * a.m + row) * a.d;
#pragma unroll
        for (int g = 0; g < 8; ++g) {
            if (16 * g >= a.d) break;
            if (!spoilt(g)) continue;
            uint32_t o[16];
            tmem_ld16(tmem_o + 16 * g, o);
#pragma unroll
            for (int x = 0; x < 16; ++x)
                if (mine[g >> 1] >> (16 * (g & 1) + x) & 1u) out[16 * g + x] = holo::narrow16(__fdiv_rn(__uint_as_float(o[x]), sum), F16 ? HOLO_DTYPE_F16 : HOLO_DTYPE_BF16);
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
}

template <bool F16>
__global__ void __launch_bounds__(ROWS_WARPS * 32, 1)
attention_rows_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                      const __grid_constant__ CUtensorMap map_v, const __grid_constant__ RowsParams p) {
    // f16 weights are kept 2^7 larger, so that their remainders stay above f16's smallest steps (2^GROWTH more still fits)
    constexpr float LIFT = F16 ? 7.0f : 0.0f;
    extern __shared__ uint8_t smem_raw[];
    const HoloAttnArgs& a = p.a;
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* sm = smem_raw + (base - raw);
    const uint32_t tile_bytes = p.chunks * TILE_CHUNK;
    const RowsTail at(p.nq, tile_bytes);
    const uint32_t s_q = base + at.q, s_k = base + at.k, s_v = base + at.v, off_bars = at.bars;
    const uint32_t bar_q = base + off_bars, bar_k_full = bar_q + 8, bar_k_empty = bar_k_full + 16, bar_v_full = bar_k_empty + 16,
                   bar_v_empty = bar_v_full + 16, bar_s = bar_v_empty + 16, bar_p = bar_s + 16, bar_pv = bar_p + 16;
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(sm + off_bars + RowsTail::TMEM);
    volatile uint32_t* s_abort = reinterpret_cast<volatile uint32_t*>(sm + off_bars + RowsTail::ABORT);
    volatile uint32_t* s_again = reinterpret_cast<volatile uint32_t*>(sm + off_bars + RowsTail::AGAIN);

    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t plane = blockIdx.x, kv_plane = plane / a.h * a.hkv + plane % a.h / (a.h / a.hkv);
    const uint32_t row0 = (gridDim.y - 1 - blockIdx.y) * p.nq * 128;   // causal: the tiles with the most keys first
    if (threadIdx.x == 0) {
        mbar_init(bar_q, 1);
        for (int s = 0; s < 2; ++s) {
            mbar_init(bar_k_full + 8 * s, 1);
            mbar_init(bar_k_empty + 8 * s, 1);
            mbar_init(bar_v_full + 8 * s, 1);
            mbar_init(bar_v_empty + 8 * s, 1);
            mbar_init(bar_s + 8 * s, 1);
            mbar_init(bar_p + 8 * s, 4);     // one arrival per softmax warp
            mbar_init(bar_pv + 8 * s, 1);
        }
        mbar_init(base + off_bars + RowsTail::AGAIN_BAR, 1);
        mbar_init(base + off_bars + RowsTail::AGAIN_SCORES_BAR, 1);
        *s_abort = 0;
        *s_again = 0;
        *reinterpret_cast<uint4*>(sm + off_bars + RowsTail::SPOILT) = make_uint4(0, 0, 0, 0);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    holo_pdl_wait();
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(s_tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    holo_pdl_trigger();
    const uint32_t tmem_base = *s_tmem;
    // key tiles of each query tile; the second has at least as many, or (past the end of the sequence) none
    auto keys_of = [&](uint32_t q) { return a.all_new ? a.m : min(row0 + (q + 1) * 128, a.m); };
    auto tiles_of = [&](uint32_t q) { return q < p.nq && row0 + q * 128 < a.m ? (keys_of(q) + 127) / 128 : 0u; };
    const uint32_t n0 = tiles_of(0), n1 = tiles_of(1), ntiles = max(n0, n1);

    if (warp == 0) {
        // ---------------- TMA producer ----------------
        if (lane == 0) {
            const uint32_t nq = n1 ? 2 : 1;
            mbar_arrive_expect_tx(bar_q, nq * tile_bytes);
            for (uint32_t i = 0; i < nq; ++i)
                for (uint32_t c = 0; c < p.chunks; ++c) tma_load_3d(s_q + i * tile_bytes + c * TILE_CHUNK, &map_q, (int)(64 * c), (int)(row0 + i * 128), (int)plane, bar_q);
            uint32_t kt = 0, vt = 0;
            bool ok = true;
            for (uint32_t t = 0; t < ntiles; ++t) {
                const uint32_t s = t & 1u, phase = ((t >> 1) - 1) & 1u;
                ok = t < 2 || mbar_wait(bar_k_empty + 8 * s, phase, s_abort, p.status);
                if (!ok) break;
                mbar_arrive_expect_tx(bar_k_full + 8 * s, tile_bytes);
                for (uint32_t c = 0; c < p.chunks; ++c) tma_load_3d(s_k + s * tile_bytes + c * TILE_CHUNK, &map_k, (int)(64 * c), (int)(t * 128), (int)kv_plane, bar_k_full + 8 * s);
                ++kt;
                ok = t < 2 || mbar_wait(bar_v_empty + 8 * s, phase, s_abort, p.status);
                if (!ok) break;
                mbar_arrive_expect_tx(bar_v_full + 8 * s, tile_bytes);
                for (uint32_t c = 0; c < p.chunks; ++c) tma_load_3d(s_v + s * tile_bytes + c * TILE_CHUNK, &map_v, (int)(64 * c), (int)(t * 128), (int)kv_plane, bar_v_full + 8 * s);
                ++vt;
            }
            if (!ok) {
                // nothing may still be on its way into this CTA's shared memory when it ends
                for (uint32_t it = 0; it < WAIT_LIMIT && !mbar_try_wait(bar_q, 0); ++it) __nanosleep(64);
                for (uint32_t t = kt > 2 ? kt - 2 : 0; t < kt; ++t)
                    for (uint32_t it = 0; it < WAIT_LIMIT && !mbar_try_wait(bar_k_full + 8 * (t & 1), (t >> 1) & 1); ++it) __nanosleep(64);
                for (uint32_t t = vt > 2 ? vt - 2 : 0; t < vt; ++t)
                    for (uint32_t it = 0; it < WAIT_LIMIT && !mbar_try_wait(bar_v_full + 8 * (t & 1), (t >> 1) & 1); ++it) __nanosleep(64);
            }
        }
    } else if (warp == 1) {
        // ---------------- MMA issuer ----------------
        if (lane == 0) {
            // D = f32, A and B of the call's type, M = 128; S: both operands K-major, N = 128; O: V is N-major, N = dim
            const uint32_t type = F16 ? 0u : (1u << 7) | (1u << 10);
            const uint32_t idesc_s = (1u << 4) | type | ((128u >> 3) << 17) | ((128u >> 4) << 24);
            const uint32_t idesc_o = (1u << 4) | type | (1u << 16) | ((a.d >> 3) << 17) | ((128u >> 4) << 24);
            const uint64_t first_q = smem_desc(s_q, 16, 1024), first_v = smem_desc(s_v, TILE_CHUNK, 1024);
            const uint32_t desc_q = (uint32_t)first_q, desc_k = (uint32_t)smem_desc(s_k, 16, 1024), high_s = (uint32_t)(first_q >> 32);
            const uint32_t desc_v = (uint32_t)first_v, high_v = (uint32_t)(first_v >> 32);
            const uint32_t step = tile_bytes >> 4, ksteps = a.d / 16;
            auto scores = [&](uint32_t q, uint32_t t) {
                const uint32_t dq = desc_q + q * step, dk = desc_k + (t & 1u) * step, d = tmem_base + q * 128;
                if (t == 0) {       // in a loop: the first tile is all of a short call, for which the steps below are code to fetch
                    for (uint32_t k = 0; k < ksteps; ++k) {
                        const uint32_t off = (k >> 2) * (TILE_CHUNK >> 4) + 2 * (k & 3u);
                        product_ss(d, dq + off, high_s, dk + off, high_s, idesc_s, k != 0);
                    }
                } else {
#pragma unroll
                    for (uint32_t k = 0; k < 8; ++k) {
                        const uint32_t off = (k >> 2) * (TILE_CHUNK >> 4) + 2 * (k & 3u);
                        if (k < ksteps) product_ss(d, dq + off, high_s, dk + off, high_s, idesc_s, k != 0);
                    }
                }
                umma_commit(bar_s + 8 * q);
            };
            bool ok = mbar_wait(bar_q, 0, s_abort, p.status) && mbar_wait(bar_k_full, 0, s_abort, p.status);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                scores(0, 0);
                if (n1) scores(1, 0);
                umma_commit(bar_k_empty);
            }
            for (uint32_t t = 0; t < ntiles && ok; ++t) {
                const uint32_t s = t & 1u, phase = (t >> 1) & 1u, next = t + 1;
                ok = mbar_wait(bar_v_full + 8 * s, phase, s_abort, p.status) &&
                     (next >= ntiles || mbar_wait(bar_k_full + 8 * (next & 1u), (next >> 1) & 1u, s_abort, p.status));
                for (uint32_t q = 0; q < 2 && ok; ++q) {
                    const uint32_t n = q ? n1 : n0;
                    if (t >= n) continue;
                    ok = mbar_wait(bar_p + 8 * q, t & 1u, s_abort, p.status);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    // keys past the last one any row of the tile sees have no weight: whole steps of them are left out
                    const uint32_t steps = min(8u, (keys_of(q) - t * 128 + 15) / 16);
                    const uint32_t tmem_p = tmem_base + q * 128, d = tmem_base + 256 + q * 128;
                    const uint32_t dv = desc_v + s * step;
                    if (steps == 8) {
#pragma unroll
                        for (uint32_t k = 0; k < 16; ++k) product_ts(d, tmem_p + k * 8, dv + 128 * (k & 7u), high_v, idesc_o, (k | t) != 0);
                    } else {
                        for (uint32_t k = 0; k < steps; ++k) product_ts(d, tmem_p + k * 8, dv + 128 * k, high_v, idesc_o, (k | t) != 0);
                        for (uint32_t k = 0; k < steps; ++k) product_ts(d, tmem_p + 64 + k * 8, dv + 128 * k, high_v, idesc_o, 1);
                    }
                    umma_commit(bar_pv + 8 * q);
                    // the next scores go where the weights are, behind the product that reads them (see product_ss)
                    if (next < n) scores(q, next);
                }
                if (!ok) break;
                umma_commit(bar_v_empty + 8 * s);
                if (next < ntiles) umma_commit(bar_k_empty + 8 * (next & 1u));
            }
        }
    } else {
        // ---------------- softmax (TMEM lane quarter = warp % 4), then the output ----------------
        const uint32_t q = (warp - 2) >> 2, quarter = warp & 3u, row = row0 + q * 128 + quarter * 32 + lane;
        const uint32_t n = q ? n1 : n0, lanes = (quarter * 32u) << 16;
        const uint32_t tmem_s = tmem_base + q * 128 + lanes, tmem_o = tmem_base + 256 + q * 128 + lanes;
        const uint32_t limit = a.all_new ? a.m : min(row + 1, a.m);          // keys this row sees
        const uint32_t common = a.all_new ? a.m : min(row - lane + 1, a.m);  // keys all rows of the warp see
        const uint64_t c2 = pair(p.to_log2, p.to_log2);
        float top = -INFINITY, sum = 0.0f;
        bool ok = true;
        for (uint32_t t = 0; t < n; ++t) {
            ok = mbar_wait(bar_s + 8 * q, t & 1u, s_abort, p.status) && !*s_abort;
            ok = __all_sync(0xffffffffu, ok);   // the TMEM accesses below are whole-warp instructions
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
            uint32_t v[4][32];
#pragma unroll
            for (int c = 0; c < 4; ++c) tmem_ld32_request(tmem_s + 32 * c, v[c]);
            tmem_ld32_wait(v[0]);
#pragma unroll
            for (int c = 1; c < 4; ++c) tmem_ld32_pass(v[c]);
            if (t * 128 + 128 > common) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int x = 0; x < 32; ++x)
                        if (t * 128 + c * 32 + x >= limit) v[c][x] = 0xff800000u;
            }
            float most[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
            for (int x = 0; x < 32; ++x)
#pragma unroll
                for (int c = 0; c < 4; ++c) most[c] = fmaxf(most[c], __uint_as_float(v[c][x]));
            const float here = fmaxf(fmaxf(most[0], most[1]), fmaxf(most[2], most[3])) * p.to_log2;
            const bool grows = here > top + GROWTH;
            if (__any_sync(0xffffffffu, grows)) {
                const float f = grows ? ex2(top - here) : 1.0f;      // 0 from the first scores on
                if (grows) top = here;
                sum *= f;
                if (t > 0) {    // the barrier of this tile's scores stands for the product before them too: O is at rest
                    const uint64_t f2 = pair(f, f);
                    for (uint32_t c = 0; c < a.d; c += 16) {
                        uint32_t o[16];
                        tmem_ld16(tmem_o + c, o);
#pragma unroll
                        for (int x = 0; x < 8; ++x) {
                            const float2 m = unpair(mul2(pair(__uint_as_float(o[2 * x]), __uint_as_float(o[2 * x + 1])), f2));
                            o[2 * x] = __float_as_uint(m.x);
                            o[2 * x + 1] = __float_as_uint(m.y);
                        }
                        tmem_st16(tmem_o + c, o);
                    }
                }
            }
            const float from = (top == -INFINITY ? 0.0f : top) - LIFT;
            const uint64_t from2 = pair(-from, -from);
            uint64_t s2[2] = {0, 0};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                uint32_t first[16], second[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    float2 e = unpair(fma2(pair(__uint_as_float(v[c][2 * x]), __uint_as_float(v[c][2 * x + 1])), c2, from2));
                    e.x = ex2(e.x);
                    e.y = ex2(e.y);
                    s2[x & 1] = add2(s2[x & 1], pair(e.x, e.y));
                    split_weights<F16>(e.x, e.y, first[x], second[x]);
                }
                tmem_st16(tmem_s + c * 16, first);
                tmem_st16(tmem_s + 64 + c * 16, second);
            }
            const float2 s0 = unpair(add2(s2[0], s2[1]));
            sum += s0.x + s0.y;
            asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
            __syncwarp();
            if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar_p + 8 * q) : "memory");
        }
        if (n) {
            ok = ok && mbar_wait(bar_pv + 8 * q, (n - 1) & 1u, s_abort, p.status) && !*s_abort;
            ok = __all_sync(0xffffffffu, ok);
            if (ok) {
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const float inv = __fdiv_rn(1.0f, sum);
                uint16_t* out = (uint16_t*)a.out + ((uint64_t)plane * a.m + row) * a.d;
                bool finite = true;
                for (uint32_t c = 0; c < a.d; c += 16) {
                    uint32_t o[16], w[8];
                    tmem_ld16(tmem_o + c, o);
#pragma unroll
                    for (int x = 0; x < 8; ++x) {
                        const float lo = __uint_as_float(o[2 * x]) * inv, hi = __uint_as_float(o[2 * x + 1]) * inv;
                        finite = finite && isfinite(lo) && isfinite(hi);
                        constexpr int DT = F16 ? HOLO_DTYPE_F16 : HOLO_DTYPE_BF16;
                        w[x] = (uint32_t)holo::narrow16(lo, DT) | ((uint32_t)holo::narrow16(hi, DT) << 16);
                    }
                    if (row < a.m) {
                        reinterpret_cast<uint4*>(out + c)[0] = make_uint4(w[0], w[1], w[2], w[3]);
                        reinterpret_cast<uint4*>(out + c)[1] = make_uint4(w[4], w[5], w[6], w[7]);
                    }
                }
                // a row whose maximum is +inf is NaN throughout
                const int what = row >= a.m || top == INFINITY ? ROW_STAYS : fabsf(top) >= WILD || !isfinite(inv) ? ROW_ALL : finite ? ROW_STAYS : ROW_COLUMNS;
                reinterpret_cast<float2*>(sm + off_bars + RowsTail::ROWS)[threadIdx.x - 64] = make_float2(top, (float)what);
                if (what != ROW_STAYS) *s_again = 1;
            }
        }
    }
    // everyone meets here, whatever happened above, so that TMEM is always released
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (*s_again && !*s_abort) compute_again<F16>(map_k, map_v, p, sm, tmem_base, row0, n0, n1);
    if (warp == 1) {
        asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(512u) : "memory");
    }
}

int32_t make_rows_map(CUtensorMap* map, const void* ptr, uint32_t d, uint32_t rows, uint32_t planes) {
    cuuint64_t dims[3] = {d, rows, planes};
    cuuint64_t strides[2] = {(cuuint64_t)d * 2, (cuuint64_t)rows * d * 2};
    cuuint32_t box[3] = {64, 128, 1};
    cuuint32_t es[3] = {1, 1, 1};
    const CUresult r = encode_tiled_fn()(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                                         CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return holo_fail(HOLO_ERR_DISPATCH, "dispatch failed: cuTensorMapEncodeTiled (attention) returned %d", (int)r);
    return HOLO_OK;
}

template <bool F16>
int32_t launch_rows(holo_b200_ctx* ctx, const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv, const RowsParams& p, dim3 grid, uint32_t smem) {
    static thread_local int configured_device = -1;
    if (configured_device != ctx->device) {
        HOLO_CUDA(cudaFuncSetAttribute(attention_rows_kernel<F16>, cudaFuncAttributeMaxDynamicSharedMemorySize, ctx->smem_optin));
        configured_device = ctx->device;
    }
    HOLO_CUDA(holo_launch_kernel(ctx, attention_rows_kernel<F16>, grid, dim3(ROWS_WARPS * 32), smem, 1, mq, mk, mv, p));
    ctx->launches++;
    return HOLO_OK;
}

}  // namespace

int32_t holo_try_attention_tile(holo_b200_ctx* ctx, const HoloAttnArgs& a, bool* taken) {
    *taken = false;
    // fewer than 16 rows would be nearly all padding; dims in whole steps of the product; TMA wants 16-byte aligned rows
    if (a.mask || a.quantized || a.dtype == HOLO_DTYPE_F32 || a.past != 0 || a.m != a.nnew || a.m < 16 || a.d % 16 != 0 || a.d > 128) return HOLO_OK;
    if ((((uintptr_t)a.q | (uintptr_t)a.k_new | (uintptr_t)a.v_new | (uintptr_t)a.out) & 15u) != 0) return HOLO_OK;
    const uint64_t planes = (uint64_t)a.b * a.h, tiles = ((uint64_t)a.m + 127) / 128;
    if (planes * a.m > 0x7fffffffull || tiles > 65535 || encode_tiled_fn() == nullptr) return HOLO_OK;
    RowsParams p;
    p.a = a;
    p.status = ctx->dev_status;
    p.to_log2 = LOG2E / a.scale_div;
    p.chunks = (a.d + 63) / 64;
    // two query tiles a CTA share what is read of K and V and hide each other's softmax, where that still gives every SM a CTA
    p.nq = tiles > 1 && planes * ((tiles + 1) / 2) >= (uint64_t)ctx->sm_count ? 2 : 1;
    CUtensorMap mq, mk, mv;
    HOLO_TRY(make_rows_map(&mq, a.q, a.d, a.m, (uint32_t)planes));
    HOLO_TRY(make_rows_map(&mk, a.k_new, a.d, a.m, a.b * a.hkv));
    HOLO_TRY(make_rows_map(&mv, a.v_new, a.d, a.m, a.b * a.hkv));
    const uint32_t smem = (p.nq + 4) * p.chunks * TILE_CHUNK + RowsTail::BYTES + 1024;   // barriers and rows, alignment slack
    const dim3 grid((uint32_t)planes, (uint32_t)((tiles + p.nq - 1) / p.nq));
    *taken = true;
    return a.dtype == HOLO_DTYPE_F16 ? launch_rows<true>(ctx, mq, mk, mv, p, grid, smem) : launch_rows<false>(ctx, mq, mk, mv, p, grid, smem);
}
