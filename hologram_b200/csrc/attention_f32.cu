// Attention of many f32 query rows (whole sequences, or a chunk after a cache) on the CUDA cores: f32 products and sums throughout.
//
// A CTA takes 16 * NR query rows of a head; NG groups of NR warps each take every NG-th tile of 64 keys and their results are
// added at the end, so that a short sequence still fills an SM. A warp holds 16 rows: a thread 4 rows x 8 keys of the scores and
// 4 rows x D / 8 columns of the context, all as packed pairs (fma.rn.f32x2). K arrives while the previous tile's context is added
// up, V while the scores are computed: one buffer each. Dot products are summed in runs of 32 elements and scaled by the divisor's
// rounded reciprocal; a row's context is one chain over a group's keys, so its error is up to 1.7 times that of the general routine's
// eight shorter ones (against 64 bits 64 keys 1.9e-7 and 1.3e-7, 1024 keys 4.4e-7 and 2.6e-7).
// Bound: the FMA rate, and beside it reads of shared memory (12 128-bit reads for 64 packed multiply-adds in the scores).
// Measured, us (one CTA per query row, before, in brackets): 381 rows, 12 heads, dim 64 20 [994]; 512 rows 44 [1720]; 1024 rows, 32
// heads over 8, dim 128, causal 272 [11461]; two such sequences, all keys 949 [47527] = 36 TFLOP/s of 74.
//
// A weight of zero times an infinite or NaN value is NaN: keys that only some rows of a warp see are added to those alone. The causal
// law's instances pay 2 % for that (381 rows 20.0 -> 20.3), those of 64-row blocks, short of registers, 4 to 8 % (1024 rows, 32 heads, dim 64
// 234 -> 244); the others have none of it.
#include "common.h"
#include "numerics.cuh"

namespace {

constexpr int TILE = 64;                 // keys
constexpr int P_LD = TILE + 8;           // weights: the four rows a warp writes together start 8 banks apart

__device__ __forceinline__ uint64_t both(float a) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ float2 unpair(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ uint64_t fma2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ uint64_t mul2(uint64_t a, uint64_t b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
// 16 bytes to shared memory, or 16 zero bytes when `take` is false (nothing is read then)
__device__ __forceinline__ void copy16(float* dst, const float* src, bool take) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(take ? 16u : 0u) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void arrived() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

template <int D, int NR, int NG>
struct Layout {
    static constexpr int ROWS = 16 * NR, WARPS = NR * NG, LD = D + 4;
    static constexpr int Q = ROWS * LD, GROUP = TILE * LD + TILE * D, P = WARPS * 16 * P_LD;
    static constexpr int FLOATS = Q + NG * GROUP + P;
    static_assert(NG * ROWS * (D + 2) <= NG * GROUP, "the groups' results fit in the tiles' memory");
};

template <int D, int NR, int NG, bool CAUSAL>
__global__ void __launch_bounds__(NR * NG * 32, NR * NG <= 4 ? 3 : 1)
attention_f32_kernel(const __grid_constant__ HoloAttnArgs a) {
    using L = Layout<D, NR, NG>;
    extern __shared__ __align__(16) float smem[];
    const uint32_t tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, group = warp / NR, wrow = warp % NR;
    // lanes' bits in the order column, row, column, column, row: 128-bit reads then take two wavefronts
    const uint32_t tx = (lane & 1) | ((lane >> 1) & 6), ty = ((lane >> 1) & 1) | ((lane >> 3) & 2);
    const uint32_t plane = blockIdx.x, kv_plane = plane / a.h * a.hkv + plane % a.h / (a.h / a.hkv);
    const uint32_t row0 = (gridDim.y - 1 - blockIdx.y) * L::ROWS;      // causal: the rows with the most keys first
    float *s_q = smem, *s_k = smem + L::Q + group * L::GROUP, *s_v = s_k + TILE * L::LD;
    float* s_p = smem + L::Q + NG * L::GROUP + warp * 16 * P_LD;
    holo_pdl_trigger();
    holo_pdl_wait();
    const uint32_t past = a.valid_len ? min(*a.valid_len, a.past) : a.past;
    auto limit_of = [&](uint32_t row) { return past + (a.all_new ? a.nnew : min(row + 1, a.nnew)); };
    const uint32_t keys = limit_of(min(row0 + L::ROWS, a.m) - 1), tiles = (keys + TILE - 1) / TILE, dvec = a.d / 4;
    {
        const float* q = (const float*)a.q + ((uint64_t)plane * a.m + row0) * a.d;
        for (uint32_t i = tid; i < L::ROWS * (D / 4); i += L::WARPS * 32) {
            const uint32_t r = i / (D / 4), c = i % (D / 4);
            const bool take = row0 + r < a.m && c < dvec;
            copy16(s_q + r * L::LD + 4 * c, take ? q + (uint64_t)r * a.d + 4 * c : q, take);
        }
    }
    const uint32_t gt = tid % (NR * 32);
    auto request = [&](float* dst, uint32_t ld, const void* old, const void* fresh, uint32_t tile) {
#pragma unroll 4
        for (uint32_t i = gt; i < TILE * (D / 4); i += NR * 32) {
            const uint32_t r = i / (D / 4), c = i % (D / 4), key = tile * TILE + r;
            const bool take = key < keys && c < dvec;
            const float* src = key < past ? (const float*)old + ((uint64_t)kv_plane * a.past + key) * a.d : (const float*)fresh + ((uint64_t)kv_plane * a.nnew + (key - past)) * a.d;
            copy16(dst + r * ld + 4 * c, take ? src + 4 * c : (const float*)fresh, take);
        }
    };
    auto meet = [&]() { asm volatile("bar.sync %0, %1;" ::"r"(group + 1), "n"(NR * 32) : "memory"); };
    if (group < tiles) request(s_k, L::LD, a.k_past, a.k_new, group);
    commit();
    arrived();
    __syncthreads();

    uint64_t o[4][D / 16];
    float top[4], sum[4];
    uint32_t limit[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        top[i] = -INFINITY;
        sum[i] = 0.0f;
        limit[i] = limit_of(min(row0 + wrow * 16 + ty + 4 * i, a.m - 1));
#pragma unroll
        for (int c = 0; c < D / 16; ++c) o[i][c] = 0;
    }
    const float* q = s_q + (wrow * 16 + ty) * L::LD;
    const float* k = s_k + tx * L::LD;
    const uint32_t runs = (a.d + 31) / 32;
    const float scale = __fdiv_rn(1.0f, a.scale_div);
#pragma unroll 1
    for (uint32_t t = group; t < tiles; t += NG) {
        arrived();
        meet();         // this tile's K is here, and everybody in the group has left the last tile's V
        request(s_v, D, a.v_past, a.v_new, t);
        commit();
        float s[4][8];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int x = 0; x < 8; ++x) s[i][x] = 0.0f;
#pragma unroll 1
        for (uint32_t run = 0; run < runs; ++run) {
            uint64_t acc[4][8];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int x = 0; x < 8; ++x) acc[i][x] = 0;
#pragma unroll 2
            for (uint32_t c = run * 32; c < run * 32 + 32; c += 4) {
                ulonglong2 qv[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) qv[i] = *reinterpret_cast<const ulonglong2*>(q + 4 * i * L::LD + c);
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const ulonglong2 kv = *reinterpret_cast<const ulonglong2*>(k + 8 * x * L::LD + c);
#pragma unroll
                    for (int i = 0; i < 4; ++i) acc[i][x] = fma2(qv[i].y, kv.y, fma2(qv[i].x, kv.x, acc[i][x]));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int x = 0; x < 8; ++x) {
                    const float2 e = unpair(acc[i][x]);
                    s[i][x] += e.x + e.y;
                }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float most = -INFINITY;
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                s[i][x] = t * TILE + tx + 8 * x < limit[i] ? s[i][x] * scale : -INFINITY;
                most = fmaxf(most, s[i][x]);
            }
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 1));
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 4));
            most = fmaxf(most, __shfl_xor_sync(0xffffffffu, most, 8));
            most = fmaxf(most, top[i]);
            const float f = top[i] == -INFINITY ? 0.0f : expf(top[i] - most);
            top[i] = most;
            float part = 0.0f;
#pragma unroll
            for (int x = 0; x < 8; ++x) {
                const float w = s[i][x] == -INFINITY ? 0.0f : expf(s[i][x] - most);
                s_p[(ty + 4 * i) * P_LD + tx + 8 * x] = w;
                part += w;
            }
            sum[i] = sum[i] * f + part;
            const uint64_t f2 = both(f);
#pragma unroll
            for (int c = 0; c < D / 16; ++c) o[i][c] = mul2(o[i][c], f2);
        }
        __syncwarp();
        arrived();
        meet();         // V is here, and everybody in the group has left K
        if (t + NG < tiles) request(s_k, L::LD, a.k_past, a.k_new, t + NG);
        commit();
        // Keys of this tile that all rows of the warp see (those of its first row, in lane 0) and that any of them does (its last row: ty
        // 3, lane 18); without the causal law all of them, rows of zeros behind the last one included.
        const uint32_t at = t * TILE;
        uint32_t common = TILE, end = TILE;
        if constexpr (CAUSAL) {
            const uint32_t all_see = __shfl_sync(0xffffffffu, limit[0], 0), one_sees = __shfl_sync(0xffffffffu, limit[3], 18);
            end = one_sees > at ? min(one_sees - at, (uint32_t)TILE) : 0u;
            common = all_see > at ? min(all_see - at, (uint32_t)TILE) & ~3u : 0u;
        }
#pragma unroll 1
        for (uint32_t j = 0; j < common; j += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(s_p + (ty + 4 * i) * P_LD + j);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ulonglong2 v[D / 32];
#pragma unroll
                for (int c = 0; c < D / 32; ++c) v[c] = *reinterpret_cast<const ulonglong2*>(s_v + (j + e) * D + 32 * c + 4 * tx);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const uint64_t w2 = both(e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w);
#pragma unroll
                    for (int c = 0; c < D / 32; ++c) {
                        o[i][2 * c] = fma2(w2, v[c].x, o[i][2 * c]);
                        o[i][2 * c + 1] = fma2(w2, v[c].y, o[i][2 * c + 1]);
                    }
                }
            }
        }
        if constexpr (CAUSAL)
#pragma unroll 1
        for (uint32_t j = common; j < end; j += 4) {
            float4 w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) w[i] = *reinterpret_cast<const float4*>(s_p + (ty + 4 * i) * P_LD + j);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                ulonglong2 v[D / 32];
#pragma unroll
                for (int c = 0; c < D / 32; ++c) v[c] = *reinterpret_cast<const ulonglong2*>(s_v + (j + e) * D + 32 * c + 4 * tx);
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    if (at + j + e < limit[i]) {
                        const uint64_t w2 = both(e == 0 ? w[i].x : e == 1 ? w[i].y : e == 2 ? w[i].z : w[i].w);
#pragma unroll
                        for (int c = 0; c < D / 32; ++c) {
                            o[i][2 * c] = fma2(w2, v[c].x, o[i][2 * c]);
                            o[i][2 * c + 1] = fma2(w2, v[c].y, o[i][2 * c + 1]);
                        }
                    }
            }
        }
        __syncwarp();   // the warp's weights have been read
    }
    // ---- add the groups up: each leaves its rows, maxima and sums in its own tiles' memory ----
    arrived();
    __syncthreads();
    float *s_o = smem + L::Q, *s_ml = s_o + NG * L::ROWS * D;      // [NG][ROWS][D], [NG][ROWS][2]
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 1);
        sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 4);
        sum[i] += __shfl_xor_sync(0xffffffffu, sum[i], 8);
        const uint32_t at = group * L::ROWS + wrow * 16 + ty + 4 * i;
#pragma unroll
        for (int c = 0; c < D / 32; ++c) *reinterpret_cast<ulonglong2*>(s_o + at * D + 32 * c + 4 * tx) = make_ulonglong2(o[i][2 * c], o[i][2 * c + 1]);
        if (tx == 0) {
            s_ml[2 * at] = top[i];
            s_ml[2 * at + 1] = sum[i];
        }
    }
    __syncthreads();
    float* out = (float*)a.out + ((uint64_t)plane * a.m + row0) * a.d;
    const uint32_t here = min((uint32_t)L::ROWS, a.m - row0);
    for (uint32_t i = tid; i < here * dvec; i += L::WARPS * 32) {
        const uint32_t r = i / dvec, c = 4 * (i % dvec);
        float most = -INFINITY, total = 0.0f;
#pragma unroll
        for (int g = 0; g < NG; ++g) most = fmaxf(most, s_ml[2 * (g * L::ROWS + r)]);
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int g = 0; g < NG; ++g) {
            const float m = s_ml[2 * (g * L::ROWS + r)], f = m == -INFINITY ? 0.0f : expf(m - most);
            const float4 v = *reinterpret_cast<const float4*>(s_o + (g * L::ROWS + r) * D + c);
            total = fmaf(f, s_ml[2 * (g * L::ROWS + r) + 1], total);
            acc = make_float4(fmaf(f, v.x, acc.x), fmaf(f, v.y, acc.y), fmaf(f, v.z, acc.z), fmaf(f, v.w, acc.w));
        }
        *reinterpret_cast<float4*>(out + (uint64_t)r * a.d + c) = make_float4(acc.x / total, acc.y / total, acc.z / total, acc.w / total);
    }
}

template <int D, int NR, int NG, bool CAUSAL>
int32_t launch_form(holo_b200_ctx* ctx, const HoloAttnArgs& a, uint32_t planes) {
    using L = Layout<D, NR, NG>;
    constexpr int SMEM = L::FLOATS * 4;
    static thread_local int configured_device = -1;
    if (configured_device != ctx->device) {
        HOLO_CUDA(cudaFuncSetAttribute(attention_f32_kernel<D, NR, NG, CAUSAL>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM));
        configured_device = ctx->device;
    }
    HOLO_CUDA(holo_launch_kernel(ctx, attention_f32_kernel<D, NR, NG, CAUSAL>, dim3(planes, (a.m + L::ROWS - 1) / L::ROWS), dim3(L::WARPS * 32), SMEM, 1, a));
    ctx->launches++;
    return HOLO_OK;
}
template <int D, int NR, int NG>
int32_t launch(holo_b200_ctx* ctx, const HoloAttnArgs& a, uint32_t planes) {
    return a.all_new ? launch_form<D, NR, NG, false>(ctx, a, planes) : launch_form<D, NR, NG, true>(ctx, a, planes);
}

}  // namespace

int32_t holo_try_attention_f32(holo_b200_ctx* ctx, const HoloAttnArgs& a, bool* taken) {
    *taken = false;
    if (a.mask || a.quantized || a.dtype != HOLO_DTYPE_F32 || a.m < 2 || a.m != a.nnew || a.d % 4 != 0 || a.d > 128) return HOLO_OK;
    const uintptr_t cache = a.past ? (uintptr_t)a.k_past | (uintptr_t)a.v_past : 0;
    if (((cache | (uintptr_t)a.q | (uintptr_t)a.k_new | (uintptr_t)a.v_new | (uintptr_t)a.out) & 15u) != 0) return HOLO_OK;
    const uint64_t planes = (uint64_t)a.b * a.h, blocks = ((uint64_t)a.m + 63) / 64;
    if (planes * a.m > 0x7fffffffull || 2 * blocks > 65535 || (uint64_t)a.past + a.nnew > 0x7fffffffull) return HOLO_OK;
    // where 64-row blocks leave SMs without one: 32-row blocks whose four groups share the keys
    const uint64_t sms = (uint64_t)ctx->sm_count, keys = (uint64_t)a.past + a.nnew, tiles = (keys + TILE - 1) / TILE;
    const bool small = a.d <= 64 && planes * blocks < sms;
    // Rows and keys are padded to whole tiles, so a few rows of a few keys are the general routine's. Measured, in ns: a wave of CTAs
    // and its first pass over a group's tile, then each further pass; dims up to 64 with every SM full, 31 a CTA and tile.
    auto waves = [&](uint64_t rows) { return (planes * ((a.m + rows - 1) / rows) + sms - 1) / sms; };
    const uint64_t ns = small ? waves(32) * (8300 + ((tiles + 3) / 4 - 1) * 9500) : a.d <= 64 ? 6000 + planes * blocks * tiles * 31 * 148 / sms
                              : a.d <= 96 ? waves(64) * (10300 + ((tiles + 1) / 2 - 1) * 12500) : waves(64) * (12500 + ((tiles + 1) / 2 - 1) * 15800);
    const uint64_t average = (uint64_t)a.past + (a.all_new ? a.m : (a.m + 1) / 2);
    // within 8 % the estimates do not tell which: this kernel
    if (ns * 25 > holo_general_attention_ns(planes * a.m, keys, average, a.d) * 27) return HOLO_OK;
    *taken = true;
    const uint32_t n = (uint32_t)planes;
    if (a.d <= 64) return small ? launch<64, 2, 4>(ctx, a, n) : launch<64, 4, 1>(ctx, a, n);
    return a.d <= 96 ? launch<96, 4, 2>(ctx, a, n) : launch<128, 4, 2>(ctx, a, n);
}
