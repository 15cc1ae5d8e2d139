// Single-token attention over a float cache (DecodeAttentionValid, f32 / f16 / bf16): keys split over the chip.
//
// Bound: every cached row is read once per kv head, so HBM (or L2, where the cache fits) at long caches and latency at short
// ones. All query rows of a kv head (up to RB of them) share the rows they read:
//   * LK lanes hold one key's row, E elements each, so a warp works on 32 / LK keys at a time. A lane copies just the 16-byte
//     pieces it will read itself through its own cp.async ring: nothing is synchronised inside the loop.
//   * The RB partial dot products are added across the LK lanes by halving: in each step a lane hands over half of the rows it
//     still has, and ends with one row's score. Division, exponential and running maximum are then done once per score.
//   * Groups of lanes, warps and CTAs each keep a (maximum, sum, context) triple; warps merge through shared memory, the CTAs of
//     a cluster through distributed shared memory (each CTA a slice of the cells), clusters through a buffer that the last one
//     to count in reads. Nobody waits for another cluster.
#include "common.h"
#include "numerics.cuh"

namespace {

constexpr int WARPS = 8;
constexpr uint32_t MAX_CLUSTER = 8;
constexpr uint32_t SLOT_FLOATS = 8 * 256 + MAX_CLUSTER * 8 * 2;   // cells, then (maximum, sum) per row for each CTA of the cluster
constexpr uint32_t SLOTS = HOLO_SPLIT_PARTIAL_BYTES / (SLOT_FLOATS * 4);

struct Params {
    HoloAttnArgs a;
    float* partials;
    uint32_t* arrivals;
    uint32_t rows, rowblocks, clusters, cluster;   // query rows of a kv head; clusters per (kv head, row block), CTAs per cluster
};

__device__ __forceinline__ uint64_t pair(float lo, float hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
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
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ float peer_read(uint32_t addr, uint32_t rank) {
    uint32_t at;
    float v;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(addr), "r"(rank));
    asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(at) : "memory");
    return v;
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}

// 16 bytes of a row as pairs of floats
template <int DT> struct Row;
template <> struct Row<HOLO_DTYPE_F32> {
    static constexpr int VEC = 4;
    static __device__ __forceinline__ void widen(const uint4& w, uint64_t* o) {
        o[0] = pair(__uint_as_float(w.x), __uint_as_float(w.y));
        o[1] = pair(__uint_as_float(w.z), __uint_as_float(w.w));
    }
};
template <> struct Row<HOLO_DTYPE_BF16> {
    static constexpr int VEC = 8;
    static __device__ __forceinline__ void widen(const uint4& w, uint64_t* o) {
        const uint32_t e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) o[i] = pair(__uint_as_float(e[i] << 16), __uint_as_float(e[i] & 0xffff0000u));
    }
};
template <> struct Row<HOLO_DTYPE_F16> {
    static constexpr int VEC = 8;
    static __device__ __forceinline__ void widen(const uint4& w, uint64_t* o) {
        const uint32_t e[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float lo, hi;
            asm("{\n.reg .b16 l, h;\nmov.b32 {l, h}, %2;\ncvt.f32.f16 %0, l;\ncvt.f32.f16 %1, h;\n}" : "=f"(lo), "=f"(hi) : "r"(e[i]));
            o[i] = pair(lo, hi);
        }
    }
};

// a triple's weight against the common maximum (an empty one has none)
__device__ __forceinline__ float share(float m, float common) { return m == -INFINITY ? 0.0f : expf(m - common); }

template <int DT, int RB, int E, int LK>
__global__ void __launch_bounds__(WARPS * 32, 1)
attention_split_kernel(const __grid_constant__ Params p) {
    constexpr int VEC = Row<DT>::VEC, NV = E / VEC, KEYS = 32 / LK, STAGES = NV >= 4 ? 4 : 8, SPREAD = LK / RB;
    static_assert(E % VEC == 0 && RB <= LK, "a lane holds whole vectors and ends with one row");
    extern __shared__ __align__(16) uint8_t sm[];
    __shared__ float s_ml[WARPS][RB][2], s_block[RB][2];
    __shared__ uint32_t s_last;
    const HoloAttnArgs& a = p.a;
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = lane / LK, j = lane % LK, mine = j / SPREAD;
    const uint32_t plane = blockIdx.y / p.rowblocks, row0 = blockIdx.y % p.rowblocks * RB, rows = min((uint32_t)RB, p.rows - row0);
    const uint32_t cl = blockIdx.x / p.cluster, rank = blockIdx.x % p.cluster;
    holo_pdl_trigger();
    holo_pdl_wait();
    const uint32_t vis_past = a.valid_len ? min(*a.valid_len, a.past) : a.past, vis = vis_past + a.nnew;
    // fewer visible keys than the cache has room for: fewer clusters, so that every warp has keys
    const uint32_t used = min(p.clusters, max(1u, vis / (p.cluster * WARPS * KEYS)));
    if (cl >= used) return;     // the whole cluster
    const uint32_t key0 = (uint32_t)((uint64_t)vis * blockIdx.x / (used * p.cluster)), key1 = (uint32_t)((uint64_t)vis * (blockIdx.x + 1) / (used * p.cluster));
    const uint32_t turns = (key1 - key0 + WARPS * KEYS - 1) / (WARPS * KEYS);
    const uint64_t row_bytes = (uint64_t)a.d * (16 / VEC);

    const uint32_t ring = smem_u32(sm) + (warp * STAGES * 2 * NV * 32 + lane) * 16;
    auto request = [&](uint32_t turn) {
        const uint32_t key = key0 + (turn * WARPS + warp) * KEYS + group, at = ring + (turn % STAGES) * 2 * NV * 512;
        const bool there = key < key1, past = key < vis_past;
        const uint64_t off = there ? (past ? (uint64_t)plane * a.past + key : (uint64_t)plane * a.nnew + (key - vis_past)) * row_bytes : 0;
        const uint8_t *k = (const uint8_t*)(past ? a.k_past : a.k_new) + off, *v = (const uint8_t*)(past ? a.v_past : a.v_new) + off;
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            const uint32_t at_vec = i * LK + j;
            const uint32_t take = there && at_vec * VEC < a.d ? 16 : 0;     // 0: sixteen zero bytes, nothing is read
            const uint32_t from = take ? at_vec * 16 : 0;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + i * 512), "l"(k + from), "r"(take) : "memory");
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + (NV + i) * 512), "l"(v + from), "r"(take) : "memory");
        }
    };
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        if ((uint32_t)s < turns) request(s);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    uint64_t q[RB][E / 2], o[RB][E / 2];
#pragma unroll
    for (int r = 0; r < RB; ++r)
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            uint4 w = make_uint4(0, 0, 0, 0);
            if ((uint32_t)r < rows && (i * LK + j) * VEC < a.d)
                w = *reinterpret_cast<const uint4*>((const uint8_t*)a.q + ((uint64_t)plane * p.rows + row0 + r) * row_bytes + (i * LK + j) * 16);
            Row<DT>::widen(w, &q[r][i * VEC / 2]);
#pragma unroll
            for (int e = 0; e < VEC / 2; ++e) o[r][i * VEC / 2 + e] = 0;
        }
    float top = -INFINITY, sum = 0.0f;      // of row `mine`, over this group's keys
#pragma unroll 1
    for (uint32_t turn = 0; turn < turns; ++turn) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        const uint32_t at = ring + (turn % STAGES) * 2 * NV * 512;
        uint64_t kv[E / 2];
        auto fetch = [&](uint32_t from) {
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                uint4 w;
                asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(from + i * 512) : "memory");
                Row<DT>::widen(w, &kv[i * VEC / 2]);
            }
        };
        fetch(at);
        float part[RB];
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            uint64_t acc = 0;
#pragma unroll
            for (int e = 0; e < E / 2; ++e) acc = fma2(q[r][e], kv[e], acc);
            const float2 s = unpair(acc);
            part[r] = s.x + s.y;
        }
#pragma unroll
        for (int n = RB / 2, step = LK / 2; step >= 1; step /= 2, n /= 2) {
            if (n >= 1) {
                const bool upper = (j & step) != 0;
#pragma unroll
                for (int i = 0; i < n; ++i) {
                    const float give = upper ? part[i] : part[i + n], keep = upper ? part[i + n] : part[i];
                    part[i] = keep + __shfl_xor_sync(0xffffffffu, give, step);
                }
            } else {
                part[0] += __shfl_xor_sync(0xffffffffu, part[0], step);
            }
        }
        const uint32_t key = key0 + (turn * WARPS + warp) * KEYS + group;
        const float s = key < key1 ? __fdiv_rn(part[0], a.scale_div) : -INFINITY;
        if (__any_sync(0xffffffffu, s > top)) {
            const float next = fmaxf(top, s), f = share(top, next);
            sum *= f;
            top = next;
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float fr = __shfl_sync(0xffffffffu, f, (lane & ~(LK - 1)) | r * SPREAD);
                const uint64_t f2 = pair(fr, fr);
#pragma unroll
                for (int e = 0; e < E / 2; ++e) o[r][e] = mul2(o[r][e], f2);
            }
        }
        const float w = s == -INFINITY ? 0.0f : expf(s - top);
        sum += w;
        fetch(at + NV * 512);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const float wr = __shfl_sync(0xffffffffu, w, (lane & ~(LK - 1)) | r * SPREAD);
            const uint64_t w2 = pair(wr, wr);
#pragma unroll
            for (int e = 0; e < E / 2; ++e) o[r][e] = fma2(w2, kv[e], o[r][e]);
        }
        // the stage read in the turn before this one is free: this lane alone uses it
        if (turn + STAGES - 1 < turns) request(turn + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // ---- groups of the warp ----
    {
        float common = top;
#pragma unroll
        for (int step = LK; step < 32; step *= 2) common = fmaxf(common, __shfl_xor_sync(0xffffffffu, common, step));
        const float f = share(top, common);
        sum *= f;
        top = common;
#pragma unroll
        for (int step = LK; step < 32; step *= 2) sum += __shfl_xor_sync(0xffffffffu, sum, step);
#pragma unroll
        for (int r = 0; r < RB; ++r) {
            const float fr = __shfl_sync(0xffffffffu, f, (lane & ~(LK - 1)) | r * SPREAD);
#pragma unroll
            for (int e = 0; e < E / 2; ++e) {
                float2 v = unpair(o[r][e]);
                v.x *= fr;
                v.y *= fr;
#pragma unroll
                for (int step = LK; step < 32; step *= 2) {
                    v.x += __shfl_xor_sync(0xffffffffu, v.x, step);
                    v.y += __shfl_xor_sync(0xffffffffu, v.y, step);
                }
                o[r][e] = pair(v.x, v.y);
            }
        }
    }
    __syncthreads();      // every ring has been read: the memory becomes [WARPS][RB][d]
    float* s_o = reinterpret_cast<float*>(sm);
    if (group == 0) {
#pragma unroll
        for (int r = 0; r < RB; ++r)
#pragma unroll
            for (int i = 0; i < NV; ++i)
                if ((i * LK + j) * VEC < a.d)
#pragma unroll
                    for (int e = 0; e < VEC / 2; ++e)
                        *reinterpret_cast<uint64_t*>(s_o + (warp * RB + r) * a.d + (i * LK + j) * VEC + 2 * e) = o[r][i * VEC / 2 + e];
        if (j % SPREAD == 0) {
            s_ml[warp][mine][0] = top;
            s_ml[warp][mine][1] = sum;
        }
    }
    __syncthreads();
    // ---- warps of the CTA: cell i into the first warp's place (only this thread touches cell i) ----
    const uint32_t cells = rows * a.d;
    for (uint32_t i = threadIdx.x; i < cells; i += WARPS * 32) {
        const uint32_t r = i / a.d;
        float common = -INFINITY, acc = 0.0f, total = 0.0f;
#pragma unroll
        for (int w = 0; w < WARPS; ++w) common = fmaxf(common, s_ml[w][r][0]);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) {
            const float f = share(s_ml[w][r][0], common);
            acc = fmaf(f, s_o[w * RB * a.d + i], acc);
            total = fmaf(f, s_ml[w][r][1], total);
        }
        s_o[i] = acc;
        if (i % a.d == 0) {
            s_block[r][0] = common;
            s_block[r][1] = total;
        }
    }
    const uint64_t out0 = ((uint64_t)plane * p.rows + row0) * a.d;
    auto finish = [&](uint32_t i, float common, float total, float acc) {
        holo::store_float(a.out, out0 + i, common == -INFINITY ? 0.0f : acc / fmaxf(total, 1e-30f), DT);
    };
    // ---- CTAs of the cluster: this one's slice of the cells ----
    if (p.cluster > 1) cluster_sync();
    else __syncthreads();
    const uint32_t begin = cells * rank / p.cluster, end = cells * (rank + 1) / p.cluster;
    float* part = p.partials + ((uint64_t)blockIdx.y * p.clusters + cl) * SLOT_FLOATS;
    for (uint32_t i = begin + threadIdx.x; i < end; i += WARPS * 32) {
        const uint32_t r = i / a.d;
        float common = s_block[r][0], total = s_block[r][1], acc = s_o[i];
        if (p.cluster > 1) {
            float m[MAX_CLUSTER], l[MAX_CLUSTER], v[MAX_CLUSTER];
#pragma unroll
            for (uint32_t c = 0; c < MAX_CLUSTER; ++c) {
                m[c] = c < p.cluster ? peer_read(smem_u32(&s_block[r][0]), c) : -INFINITY;
                l[c] = c < p.cluster ? peer_read(smem_u32(&s_block[r][1]), c) : 0.0f;
                v[c] = c < p.cluster ? peer_read(smem_u32(s_o + i), c) : 0.0f;
            }
            common = -INFINITY;
            total = acc = 0.0f;
#pragma unroll
            for (uint32_t c = 0; c < MAX_CLUSTER; ++c) common = fmaxf(common, m[c]);
#pragma unroll
            for (uint32_t c = 0; c < MAX_CLUSTER; ++c) {
                const float f = share(m[c], common);
                acc = c < p.cluster ? fmaf(f, v[c], acc) : acc;
                total = fmaf(f, l[c], total);
            }
        }
        if (used == 1) {
            finish(i, common, total, acc);
        } else {
            __stcg(part + i, acc);
            if (i == begin || i % a.d == 0) __stcg(reinterpret_cast<float2*>(part + 8 * 256) + rank * 8 + r, make_float2(common, total));
        }
    }
    if (p.cluster > 1) cluster_sync();     // the others have read this CTA's cells
    if (used == 1) return;
    // ---- clusters: the last one to count in adds them up, slice by slice ----
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) s_last = atomicAdd(p.arrivals + blockIdx.y * p.cluster + rank, 1u) == used - 1 ? 1u : 0u;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x == 0) p.arrivals[blockIdx.y * p.cluster + rank] = 0;
    const float* all = p.partials + (uint64_t)blockIdx.y * p.clusters * SLOT_FLOATS;
    for (uint32_t i = begin + threadIdx.x; i < end; i += WARPS * 32) {
        const uint32_t r = i / a.d;
        float common = -INFINITY, total = 0.0f, acc = 0.0f;
#pragma unroll 4
        for (uint32_t c = 0; c < used; ++c) {
            const float2 ml = __ldcg(reinterpret_cast<const float2*>(all + (uint64_t)c * SLOT_FLOATS + 8 * 256) + rank * 8 + r);
            const float v = __ldcg(all + (uint64_t)c * SLOT_FLOATS + i);
            const float next = fmaxf(common, ml.x), f = share(common, next), g = share(ml.x, next);
            acc = fmaf(acc, f, v * g);
            total = fmaf(total, f, ml.y * g);
            common = next;
        }
        finish(i, common, total, acc);
    }
}

template <int DT, int RB, int E, int LK>
int32_t launch(holo_b200_ctx* ctx, Params p, uint32_t items) {
    constexpr int NV = E / Row<DT>::VEC, STAGES = NV >= 4 ? 4 : 8;
    constexpr uint32_t RING = WARPS * STAGES * 2 * NV * 512, MERGE = WARPS * RB * E * LK * 4, SMEM = RING > MERGE ? RING : MERGE;
    auto kernel = attention_split_kernel<DT, RB, E, LK>;
    static thread_local int configured_device = -1;
    if (configured_device != ctx->device) {
        HOLO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
        configured_device = ctx->device;
    }
    // How many CTAs share a kv head: as many as shorten the longest SM's work, a CTA costing about as much as 64 keys per warp
    // group besides its keys. The largest cluster that wastes at most an eighth of them.
    const uint64_t keys = (uint64_t)p.a.past + p.a.nnew, sms = (uint64_t)ctx->sm_count;
    uint64_t want = 1, best = ~0ull;
    for (uint64_t w = 1; w <= 2 * sms && w * items <= 2 * sms + items && (w == 1 || w * WARPS * (32 / LK) <= keys); ++w) {
        const uint64_t cost = (items * w + sms - 1) / sms * ((keys + w - 1) / w + 64);
        if (cost < best) best = cost, want = w;
    }
    p.cluster = MAX_CLUSTER;
    while (p.cluster > 1 && (want / p.cluster) * p.cluster * 8 < want * 7) p.cluster /= 2;
    p.clusters = (uint32_t)(want / p.cluster);
    if (p.clusters > 1 && (uint64_t)items * p.clusters > SLOTS) p.clusters = items > SLOTS ? 1 : SLOTS / items;
    HOLO_CUDA(holo_launch_kernel_cluster(ctx, kernel, dim3(p.clusters * p.cluster, items), dim3(WARPS * 32), SMEM, p.cluster, 1u, p));
    ctx->launches++;
    return HOLO_OK;
}

// Rows of the block: one, up to four, up to eight; eight rows halve a lane's share of a row, so that q and the context stay in registers.
template <int DT>
int32_t launch_sized(holo_b200_ctx* ctx, Params p, uint64_t planes, bool* taken) {
    const uint32_t rb = p.rows == 1 ? 1 : p.rows <= 4 ? 4 : 8;
    p.rowblocks = (p.rows + rb - 1) / rb;
    if (planes * p.rowblocks > 65535) return HOLO_OK;
    const uint32_t items = (uint32_t)planes * p.rowblocks;
    *taken = true;
    if (p.a.d <= 64) return rb == 1 ? launch<DT, 1, 8, 8>(ctx, p, items) : rb == 4 ? launch<DT, 4, 8, 8>(ctx, p, items) : launch<DT, 8, 8, 8>(ctx, p, items);
    if (p.a.d <= 128) return rb == 1 ? launch<DT, 1, 16, 8>(ctx, p, items) : rb == 4 ? launch<DT, 4, 16, 8>(ctx, p, items) : launch<DT, 8, 8, 16>(ctx, p, items);
    return rb == 1 ? launch<DT, 1, 16, 16>(ctx, p, items) : rb == 4 ? launch<DT, 4, 16, 16>(ctx, p, items) : launch<DT, 8, 8, 32>(ctx, p, items);
}

}  // namespace

int32_t holo_try_attention_split(holo_b200_ctx* ctx, const HoloAttnArgs& a, bool* taken) {
    *taken = false;
    // every row must see the same keys: a weight of zero times an infinite value would not be zero
    if (a.mask || a.quantized || !(a.m == 1 || a.all_new) || a.nnew == 0) return HOLO_OK;
    const uint32_t vec = a.dtype == HOLO_DTYPE_F32 ? 4 : 8;
    const uint64_t rows = (uint64_t)(a.h / a.hkv) * a.m, keys = (uint64_t)a.past + a.nnew;
    if (a.d % vec != 0 || a.d > 256 || rows > 64 || keys > 0x7fffffffull) return HOLO_OK;
    const uintptr_t cache = a.past ? (uintptr_t)a.k_past | (uintptr_t)a.v_past : 0;
    if (((cache | (uintptr_t)a.q | (uintptr_t)a.k_new | (uintptr_t)a.v_new) & 15u) != 0) return HOLO_OK;
    Params p = {a, ctx->split_partials, ctx->attn_arrivals, (uint32_t)rows, 1, 1, 1};
    const uint64_t planes = (uint64_t)a.b * a.hkv;
    if (a.dtype == HOLO_DTYPE_F32) return launch_sized<HOLO_DTYPE_F32>(ctx, p, planes, taken);
    return a.dtype == HOLO_DTYPE_F16 ? launch_sized<HOLO_DTYPE_F16>(ctx, p, planes, taken) : launch_sized<HOLO_DTYPE_BF16>(ctx, p, planes, taken);
}
