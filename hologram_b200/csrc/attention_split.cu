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
//   * That buffer and its counters are the context's, and launches on its stream take turns with them. A graph that a caller
//     records may be replayed beside another one, on any stream: such a launch keeps to one cluster per kv head and touches
//     nothing but its operands (f32, 12 heads over 2, 8192 keys then 39 us instead of 14.6). So does a context without the buffer.
// Measured, us (one CTA per query row with a warp per key, before, in brackets): f32, 12 heads over 2, dim 128, 8192 keys 14.4 [2471];
// f32, 8 sequences, 32 over 8, 8192 keys 88 = 6.1 TB/s; bf16 the same 59 = 4.5 TB/s (two warps per scheduler, a turn's chain of
// product, halving, division and exponential); bf16, 8 sequences of 16 heads, dim 64 47 = 5.7 TB/s; 100 keys 5.3. The first figure
// was 18.8 with a rescaling at every new maximum and the parts' statistics and cells requested one after the other.
#include "common.h"
#include "numerics.cuh"

namespace {

constexpr int WARPS = 8;
constexpr float GROWTH = 8.0f;
constexpr uint32_t MAX_CLUSTER = 8, MAX_CLUSTERS = 16;            // CTAs of a cluster; clusters that share a kv head
constexpr uint32_t SLOT_CELLS = 8 * 256, SLOT_FLOATS = SLOT_CELLS + MAX_CLUSTER * 8 * 2;   // cells, then (maximum, sum) per row from each CTA of the cluster
constexpr uint32_t SLOTS = HOLO_SPLIT_PARTIAL_BYTES / (SLOT_FLOATS * 4);

struct Params {
    HoloAttnArgs a;
    float* partials;
    uint32_t* arrivals;
    uint32_t rows, rowblocks, clusters, cluster;   // query rows of a kv head; clusters per (kv head, row block), CTAs per cluster
    uint32_t max_clusters;                         // 1 where the partials may not be used
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
__device__ __forceinline__ uint32_t peer(const void* p, uint32_t rank) {
    uint32_t at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(at) : "r"(smem_u32(p)), "r"(rank));
    return at;
}
__device__ __forceinline__ float2 peer_read2(const void* p, uint32_t rank) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(peer(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ float4 peer_read4(const void* p, uint32_t rank) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(peer(p, rank)) : "memory");
    return v;
}
__device__ __forceinline__ void add_scaled(float4& acc, float f, const float4& v) {
    acc = make_float4(fmaf(f, v.x, acc.x), fmaf(f, v.y, acc.y), fmaf(f, v.z, acc.z), fmaf(f, v.w, acc.w));
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

// Keys a group of lanes takes per turn: their scores share the halving (KU * RB values over LK lanes), and two keys' chains hide
// each other's latency. Stages of the ring within 24 KB a warp.
template <int DT, int RB, int E, int LK>
struct Shape {
    static constexpr int VEC = Row<DT>::VEC, NV = E / VEC, GROUPS = 32 / LK;
    static constexpr int KU = RB == 8 && LK == 8 ? 1 : RB == 1 && NV <= 2 ? 4 : 2, SPREAD = LK / (RB * KU), KEYS = GROUPS * KU;
    static constexpr int LEVELS = LK == 8 ? 3 : LK == 16 ? 4 : 5;
    static constexpr int STAGE = KU * 2 * NV * 512, FIT = 24576 / STAGE, STAGES = FIT > 8 ? 8 : FIT;
    static constexpr int RING = WARPS * STAGES * STAGE, MERGE = WARPS * RB * E * LK * 4, SMEM = RING > MERGE ? RING : MERGE;
    static_assert(E % VEC == 0 && KU * RB <= LK && STAGES >= 3, "a lane holds whole vectors and ends with one score");
};

template <int DT, int RB, int E, int LK>
__global__ void __launch_bounds__(WARPS * 32, 1)
attention_split_kernel(const __grid_constant__ Params p) {
    using S = Shape<DT, RB, E, LK>;
    constexpr int VEC = S::VEC, NV = S::NV, KU = S::KU, KEYS = S::KEYS, STAGES = S::STAGES, SPREAD = S::SPREAD;
    extern __shared__ __align__(16) uint8_t sm[];
    __shared__ float s_ml[WARPS][RB][2], s_f[MAX_CLUSTERS][RB], s_sum[RB];
    __shared__ __align__(8) float s_block[RB][2];
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

    // key u of this lane's group in a turn
    auto key_of = [&](uint32_t turn, uint32_t u) { return key0 + ((turn * WARPS + warp) * KU + u) * S::GROUPS + group; };
    const uint32_t ring = smem_u32(sm) + warp * STAGES * S::STAGE + lane * 16;
    auto request = [&](uint32_t turn) {
#pragma unroll
        for (int u = 0; u < KU; ++u) {
            const uint32_t key = key_of(turn, u), at = ring + (turn % STAGES) * S::STAGE + u * NV * 512;
            const bool there = key < key1, past = key < vis_past;
            const uint64_t off = there ? (past ? (uint64_t)plane * a.past + key : (uint64_t)plane * a.nnew + (key - vis_past)) * row_bytes : 0;
            const uint8_t *k = (const uint8_t*)(past ? a.k_past : a.k_new) + off, *v = (const uint8_t*)(past ? a.v_past : a.v_new) + off;
#pragma unroll
            for (int i = 0; i < NV; ++i) {
                const uint32_t at_vec = i * LK + j;
                const uint32_t take = there && at_vec * VEC < a.d ? 16 : 0;     // 0: sixteen zero bytes, nothing is read
                const uint32_t from = take ? at_vec * 16 : 0;
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + i * 512), "l"(k + from), "r"(take) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(at + (KU * NV + i) * 512), "l"(v + from), "r"(take) : "memory");
            }
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
    // value v = u * RB + r of a group is in the lanes v * SPREAD ..: lane `mine` follows row mine % RB, over its own keys' share of the sum
    auto lane_of = [&](int v) { return (lane & ~(LK - 1)) | (v * SPREAD); };
    float top = -INFINITY, sum = 0.0f;
#pragma unroll 1
    for (uint32_t turn = 0; turn < turns; ++turn) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        const uint32_t at = ring + (turn % STAGES) * S::STAGE;
        uint64_t kv[KU][E / 2];
        auto fetch = [&](uint32_t from) {
#pragma unroll
            for (int u = 0; u < KU; ++u)
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    uint4 w;
                    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(w.x), "=r"(w.y), "=r"(w.z), "=r"(w.w) : "r"(from + (u * NV + i) * 512) : "memory");
                    Row<DT>::widen(w, &kv[u][i * VEC / 2]);
                }
        };
        fetch(at);
        float part[KU * RB];
#pragma unroll
        for (int u = 0; u < KU; ++u)
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                uint64_t acc = 0;
#pragma unroll
                for (int e = 0; e < E / 2; ++e) acc = fma2(q[r][e], kv[u][e], acc);
                const float2 s = unpair(acc);
                part[u * RB + r] = s.x + s.y;
            }
        fetch(at + KU * NV * 512);
#pragma unroll
        for (int level = 0; level < S::LEVELS; ++level) {
            const int n = (KU * RB / 2) >> level, step = (LK / 2) >> level;
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
        const float s = key_of(turn, mine / RB) < key1 ? __fdiv_rn(part[0], a.scale_div) : -INFINITY;
        // a row's context is rescaled only when its maximum has grown by more than e^GROWTH: weights stay far inside f32's range
        if (__any_sync(0xffffffffu, s > top + GROWTH)) {
            float next = fmaxf(top, s);
#pragma unroll
            for (int step = LK / 2; step > LK / 2 / KU; step /= 2) next = fmaxf(next, __shfl_xor_sync(0xffffffffu, next, step));
            const float f = share(top, next);
            sum *= f;
            top = next;
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float fr = __shfl_sync(0xffffffffu, f, lane_of(r));
                const uint64_t f2 = pair(fr, fr);
#pragma unroll
                for (int e = 0; e < E / 2; ++e) o[r][e] = mul2(o[r][e], f2);
            }
        }
        const float w = s == -INFINITY ? 0.0f : expf(s - top);
        sum += w;
#pragma unroll
        for (int u = 0; u < KU; ++u)
#pragma unroll
            for (int r = 0; r < RB; ++r) {
                const float wr = __shfl_sync(0xffffffffu, w, lane_of(u * RB + r));
                const uint64_t w2 = pair(wr, wr);
#pragma unroll
                for (int e = 0; e < E / 2; ++e) o[r][e] = fma2(w2, kv[u][e], o[r][e]);
            }
        // the stage read in the turn before this one is free: this lane alone uses it
        if (turn + STAGES - 1 < turns) request(turn + STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    // ---- groups of the warp ----
#pragma unroll
    for (int step = LK / 2; step > LK / 2 / KU; step /= 2) sum += __shfl_xor_sync(0xffffffffu, sum, step);
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
            const float fr = __shfl_sync(0xffffffffu, f, lane_of(r));
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
                    for (int e = 0; e < VEC / 2; e += 2)
                        *reinterpret_cast<ulonglong2*>(s_o + (warp * RB + r) * a.d + (i * LK + j) * VEC + 2 * e) = make_ulonglong2(o[r][i * VEC / 2 + e], o[r][i * VEC / 2 + e + 1]);
        if (j % SPREAD == 0 && mine < RB) {
            s_ml[warp][mine][0] = top;
            s_ml[warp][mine][1] = sum;
        }
    }
    __syncthreads();
    // One thread per row works out the parts' weights, then all threads add four cells at a time.
    const uint32_t vecs = rows * a.d / 4, tid = threadIdx.x;
    auto weigh = [&](uint32_t n, auto ml) {     // ml(part) -> (maximum, sum) of row `tid`, requested all at once
        float2 v[MAX_CLUSTERS];
        float common = -INFINITY, total = 0.0f;
#pragma unroll
        for (uint32_t c = 0; c < MAX_CLUSTERS; ++c) v[c] = c < n ? ml(c) : make_float2(-INFINITY, 0.0f);
#pragma unroll
        for (uint32_t c = 0; c < MAX_CLUSTERS; ++c) common = fmaxf(common, v[c].x);
#pragma unroll
        for (uint32_t c = 0; c < MAX_CLUSTERS; ++c) {
            if (c < n) {
                const float f = share(v[c].x, common);
                s_f[c][tid] = f;
                total = fmaf(f, v[c].y, total);
            }
        }
        return make_float2(common, total);
    };
    // ---- warps of the CTA: cells into the first warp's place (only this thread touches them there) ----
    if (tid < RB) {
        const float2 v = weigh(WARPS, [&](uint32_t c) { return make_float2(s_ml[c][tid][0], s_ml[c][tid][1]); });
        s_block[tid][0] = v.x;
        s_block[tid][1] = v.y;
    }
    __syncthreads();
    for (uint32_t i = tid; i < vecs; i += WARPS * 32) {
        const uint32_t r = 4 * i / a.d;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int w = 0; w < WARPS; ++w) add_scaled(acc, s_f[w][r], reinterpret_cast<const float4*>(s_o + w * RB * a.d)[i]);
        reinterpret_cast<float4*>(s_o)[i] = acc;
    }
    const uint64_t out0 = ((uint64_t)plane * p.rows + row0) * a.d;
    auto finish = [&](uint32_t i, float total, const float4& acc) {
        const float v[4] = {acc.x, acc.y, acc.z, acc.w};
#pragma unroll
        for (int e = 0; e < 4; ++e) holo::store_float(a.out, out0 + 4 * i + e, v[e] / fmaxf(total, 1e-30f), DT);
    };
    // ---- CTAs of the cluster: this one's slice of the cells ----
    const uint32_t begin = vecs * rank / p.cluster, end = vecs * (rank + 1) / p.cluster;
    float* part = p.partials + ((uint64_t)blockIdx.y * p.clusters + cl) * SLOT_FLOATS;
    if (p.cluster > 1) cluster_sync();
    else __syncthreads();
    if (tid < RB) {
        float2 v = make_float2(s_block[tid][0], s_block[tid][1]);
        if (p.cluster > 1) v = weigh(p.cluster, [&](uint32_t c) { return peer_read2(s_block[tid], c); });
        s_sum[tid] = v.y;
        if (used > 1) __stcg(reinterpret_cast<float2*>(part + SLOT_CELLS) + rank * 8 + tid, v);
    }
    __syncthreads();
    for (uint32_t i = begin + tid; i < end; i += WARPS * 32) {
        const uint32_t r = 4 * i / a.d;
        float4 acc = reinterpret_cast<const float4*>(s_o)[i];
        if (p.cluster > 1) {
            float4 v[MAX_CLUSTER];
#pragma unroll
            for (uint32_t c = 0; c < MAX_CLUSTER; ++c)
                if (c < p.cluster) v[c] = peer_read4(s_o + 4 * i, c);
            acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (uint32_t c = 0; c < MAX_CLUSTER; ++c)
                if (c < p.cluster) add_scaled(acc, s_f[c][r], v[c]);
        }
        if (used == 1) finish(i, s_sum[r], acc);
        else __stcg(reinterpret_cast<float4*>(part) + i, acc);
    }
    if (p.cluster > 1) cluster_sync();     // the others have read this CTA's cells
    if (used == 1) return;
    // ---- clusters: the last one to count in adds them up, slice by slice ----
    __syncthreads();
    if (tid == 0) {     // the barrier orders the others' stores before this fence
        __threadfence();
        s_last = atomicAdd(p.arrivals + blockIdx.y * p.cluster + rank, 1u) == used - 1 ? 1u : 0u;
        __threadfence();
    }
    __syncthreads();
    if (!s_last) return;
    if (tid == 0) p.arrivals[blockIdx.y * p.cluster + rank] = 0;
    const float* all = p.partials + (uint64_t)blockIdx.y * p.clusters * SLOT_FLOATS;
    // a thread's first cells are requested along with the weights
    float4 v[MAX_CLUSTERS];
    auto fetch = [&](uint32_t i) {
#pragma unroll
        for (uint32_t c = 0; c < MAX_CLUSTERS; ++c)
            v[c] = c < used && i < end ? __ldcg(reinterpret_cast<const float4*>(all + (uint64_t)c * SLOT_FLOATS) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    fetch(begin + tid);
    if (tid < RB) s_sum[tid] = weigh(used, [&](uint32_t c) { return __ldcg(reinterpret_cast<const float2*>(all + (uint64_t)c * SLOT_FLOATS + SLOT_CELLS) + rank * 8 + tid); }).y;
    __syncthreads();
    for (uint32_t i = begin + tid; i < end; i += WARPS * 32) {
        if (i != begin + tid) fetch(i);
        const uint32_t r = 4 * i / a.d;
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (uint32_t c = 0; c < MAX_CLUSTERS; ++c)
            if (c < used) add_scaled(acc, s_f[c][r], v[c]);
        finish(i, s_sum[r], acc);
    }
}

template <int DT, int RB, int E, int LK>
int32_t launch(holo_b200_ctx* ctx, Params p, uint32_t items) {
    using S = Shape<DT, RB, E, LK>;
    auto kernel = attention_split_kernel<DT, RB, E, LK>;
    static thread_local int configured_device = -1, resident[4];      // clusters of 1, 2, 4, 8 CTAs that run at a time
    if (configured_device != ctx->device) {
        HOLO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, S::SMEM));
        for (int i = 0; i < 4; ++i) {
            cudaLaunchConfig_t cfg = {};
            cudaLaunchAttribute attr;
            cfg.gridDim = dim3(1u << i);
            cfg.blockDim = dim3(WARPS * 32);
            cfg.dynamicSmemBytes = S::SMEM;
            attr.id = cudaLaunchAttributeClusterDimension;
            attr.val.clusterDim.x = 1u << i;
            attr.val.clusterDim.y = attr.val.clusterDim.z = 1;
            cfg.attrs = &attr;
            cfg.numAttrs = 1;
            HOLO_CUDA(cudaOccupancyMaxActiveClusters(&resident[i], kernel, &cfg));
            if (resident[i] < 1) resident[i] = 1;
        }
        configured_device = ctx->device;
    }
    // How many clusters of how many CTAs share a kv head: what the longest SM has to do, in keys. A CTA costs as much as about 64
    // keys besides its own, exchanging with its cluster and with other clusters as much again.
    const uint64_t keys = (uint64_t)p.a.past + p.a.nnew;
    uint64_t best = ~0ull;
    for (uint32_t i = 0; i < 4; ++i)
        for (uint32_t n = 1; n <= p.max_clusters; ++n) {
            const uint64_t ctas = (uint64_t)n << i, waves = ((uint64_t)items * n + resident[i] - 1) / resident[i];
            if (ctas > 1 && (ctas * WARPS * S::KEYS > keys || (n > 1 && (uint64_t)items * n > SLOTS))) break;
            const uint64_t cost = waves * ((keys + ctas - 1) / ctas + 64 + (i ? 64 : 0) + (n > 1 ? 64 + 4 * n : 0));
            if (cost < best) best = cost, p.cluster = 1u << i, p.clusters = n;
            if (waves > 4) break;
        }
    HOLO_CUDA(holo_launch_kernel_cluster(ctx, kernel, dim3(p.clusters * p.cluster, items), dim3(WARPS * 32), S::SMEM, p.cluster, 1u, p));
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
    // One CTA fits an SM (its ring takes 128 KB and more), so many sequences with a few keys each go round after round: 2.9 us a
    // round for one row, 3.6 to 4.5 for several. The general routine runs several CTAs an SM: 2048 heads of 4 keys, dim 64, 25 us
    // against 40 here; of 24 keys 45 against 41.
    const uint64_t keys = (uint64_t)p.a.past + p.a.nnew, rounds = (items + (uint64_t)ctx->sm_count - 1) / ctx->sm_count;
    const uint64_t ns = 400 + rounds * (p.rows == 1 ? 2900 : p.a.d <= 64 ? 3600 : 4300);
    if (ns > holo_general_attention_ns(planes * p.rows, keys, keys, p.a.d)) return HOLO_OK;
    *taken = true;
    if (p.a.d <= 64) return rb == 1 ? launch<DT, 1, 8, 8>(ctx, p, items) : rb == 4 ? launch<DT, 4, 8, 8>(ctx, p, items) : launch<DT, 8, 8, 8>(ctx, p, items);
    if (p.a.d <= 128) return rb == 1 ? launch<DT, 1, 16, 8>(ctx, p, items) : rb == 4 ? launch<DT, 4, 16, 8>(ctx, p, items) : launch<DT, 8, 8, 16>(ctx, p, items);
    return rb == 1 ? launch<DT, 1, 16, 16>(ctx, p, items) : rb == 4 ? launch<DT, 4, 16, 16>(ctx, p, items) : launch<DT, 8, 8, 32>(ctx, p, items);
}

}  // namespace

void holo_split_partials_create(holo_b200_ctx* ctx) {
    if (cudaMalloc(&ctx->split_partials, HOLO_SPLIT_PARTIAL_BYTES) == cudaSuccess) return;
    ctx->split_partials = nullptr;
    cudaGetLastError();
}

int32_t holo_try_attention_split(holo_b200_ctx* ctx, const HoloAttnArgs& a, bool* taken) {
    *taken = false;
    // every row must see the same keys: a weight of zero times an infinite value would not be zero
    if (a.mask || a.quantized || !(a.m == 1 || a.all_new) || a.nnew == 0) return HOLO_OK;
    const uint32_t vec = a.dtype == HOLO_DTYPE_F32 ? 4 : 8;
    const uint64_t rows = (uint64_t)(a.h / a.hkv) * a.m, keys = (uint64_t)a.past + a.nnew;
    if (a.d % vec != 0 || a.d > 256 || rows > 64 || keys > 0x7fffffffull) return HOLO_OK;
    const uintptr_t cache = a.past ? (uintptr_t)a.k_past | (uintptr_t)a.v_past : 0;
    if (((cache | (uintptr_t)a.q | (uintptr_t)a.k_new | (uintptr_t)a.v_new) & 15u) != 0) return HOLO_OK;
    cudaStreamCaptureStatus recording = cudaStreamCaptureStatusNone;
    if (!ctx->session_capture) HOLO_CUDA(cudaStreamIsCapturing(ctx->stream, &recording));
    const bool shared = ctx->split_partials && recording == cudaStreamCaptureStatusNone;
    Params p = {a, ctx->split_partials, ctx->attn_arrivals, (uint32_t)rows, 1, 1, 1, shared ? MAX_CLUSTERS : 1};
    const uint64_t planes = (uint64_t)a.b * a.hkv;
    if (a.dtype == HOLO_DTYPE_F32) return launch_sized<HOLO_DTYPE_F32>(ctx, p, planes, taken);
    return a.dtype == HOLO_DTYPE_F16 ? launch_sized<HOLO_DTYPE_F16>(ctx, p, planes, taken) : launch_sized<HOLO_DTYPE_BF16>(ctx, p, planes, taken);
}
