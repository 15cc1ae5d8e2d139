// The reference's own matmul recurrence on the CUDA cores: every output cell is one ascending-k chain of fused
// multiply-adds (multiply, then add, in the n % 8 column tail: cpu/simd.rs:746-799), bit-identical to the CPU kernel. Takes
// every f32 product, shapes the tensor-core path cannot take (row pitches that are not 16-byte multiples, unaligned bases)
// and tiny problems.
//
// A chain cannot be split, so the bound is the FMA rate over the cells that run at once: 74 TFLOP/s when every SM holds
// equally many. One thread keeps TM x TN cells in registers; tiles of A and B (BK deep, as f32) pass through a ring in shared
// memory, filled by cp.async (f32) or through registers (16-bit, widened once per tile instead of once per cell); the next
// depths' operands are read from shared memory while these are multiplied. What is left is reads of shared memory (8 bytes
// per lane and wavefront at most: 2.0 cycles for a warp's 16-byte read in both patterns below, 4.0 where no two lanes share an address. A 4 x 4
// thread needs as many cycles for them as for its multiply-adds, a 2 x 4 thread 1.5 times as many) and their latency.
// One thread per cell, before: 500 x 1000 x 771 f32 148 us, now 36 (21 TFLOP/s); 381 x 3072 x 768 462 us, now 81;
// 1000 x 2048 x 2048 now 209 (40 TFLOP/s).
#include "common.h"
#include "numerics.cuh"

namespace {

struct Params {
    const void *a, *b;
    void* out;
    const uint16_t* table;
    const void* residual;
    uint32_t m, k, n, n8;      // n8 = n - n % 8: columns of the fused chain
    uint32_t main_blocks;      // column blocks over the n8 columns; one more holds the tail
    int act, add_first;
    bool vec_a, vec_b;         // f32: rows of A / B may be copied 16 bytes at a time
};

// f32 activations are the scalar function itself (no table exists for 32-bit patterns). `add_first` (MatMulAddActivation,
// cpu/float_kernels.rs:899-938): the residual is added before the activation and nothing is narrowed between the two; for
// 16-bit dtypes the product itself is narrowed once, as the matmul stores it.
template <int DT>
__device__ __forceinline__ void store_cell(const Params& p, float acc, uint64_t idx) {
    if (DT == HOLO_DTYPE_F32) {
        const float* res = reinterpret_cast<const float*>(p.residual);
        if (p.add_first) acc = holo::lut_act_ref(p.act, __fadd_rn(acc, res[idx]));
        else {
            if (p.act >= 0) acc = holo::lut_act_ref(p.act, acc);
            if (res) acc = __fadd_rn(acc, res[idx]);
        }
        reinterpret_cast<float*>(p.out)[idx] = acc;
    } else {
        const uint16_t* res = reinterpret_cast<const uint16_t*>(p.residual);
        uint16_t h = holo::narrow16(acc, DT);
        if (p.add_first) h = holo::narrow16(holo::lut_act_ref(p.act, __fadd_rn(holo::widen16(h, DT), holo::widen16(res[idx], DT))), DT);
        else {
            if (p.table) h = __ldg(p.table + h);
            if (res) h = holo::narrow16(__fadd_rn(holo::widen16(h, DT), holo::widen16(__ldg(res + idx), DT)), DT);
        }
        reinterpret_cast<uint16_t*>(p.out)[idx] = h;
    }
}

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ uint64_t both(float a) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}

template <int DT> struct Element { typedef uint16_t type; };
template <> struct Element<HOLO_DTYPE_F32> { typedef float type; };

// ROWS x COLS words to shared memory (pitch LD), W words a copy; `rows` x `cols` of them exist in the source.
template <int ROWS, int COLS, int W, int LD, int THREADS>
__device__ __forceinline__ void copy_tile(float* dst, const float* src, uint32_t pitch, uint32_t rows, uint32_t cols) {
    constexpr int PER = COLS / W, STEP = THREADS / PER, N = (ROWS + STEP - 1) / STEP;
    static_assert(THREADS % PER == 0, "a pass is whole rows");
    const uint32_t c = (threadIdx.x % PER) * W, r = threadIdx.x / PER;
    src += (uint64_t)r * pitch + c;
    dst += r * LD + c;
    const int left = c < cols ? (int)rows - (int)r : 0;
    const uint64_t step = (uint64_t)STEP * pitch;
#pragma unroll
    for (int x = 0; x < N; ++x) {
        if (x * STEP < left) {
            if (W == 4) copy16(dst + x * STEP * LD, src);
            else copy4(dst + x * STEP * LD, src);
        }
        src += step;
    }
}

// A thread's share of a 16-bit tile on its way to shared memory
template <int DT, int ROWS, int COLS, int THREADS>
struct Held {
    static constexpr int STEP = THREADS / COLS, N = DT == HOLO_DTYPE_F32 ? 1 : (ROWS + STEP - 1) / STEP;
    uint16_t v[N];
    __device__ __forceinline__ void load(const uint16_t* src, uint32_t pitch, uint32_t rows, uint32_t cols) {
        const uint32_t c = threadIdx.x % COLS, r = threadIdx.x / COLS;
        src += (uint64_t)r * pitch + c;
        const int left = c < cols ? (int)rows - (int)r : 0;
        const uint64_t step = (uint64_t)STEP * pitch;
#pragma unroll
        for (int x = 0; x < N; ++x) {
            v[x] = x * STEP < left ? __ldg(src) : (uint16_t)0;
            src += step;
        }
    }
    template <int LD>
    __device__ __forceinline__ void store(float* dst) const {
        const uint32_t c = threadIdx.x % COLS, r = threadIdx.x / COLS;
        dst += r * LD + c;
#pragma unroll
        for (int x = 0; x < N; ++x)
            if (ROWS % STEP == 0 || r + x * STEP < ROWS) dst[x * STEP * LD] = holo::widen16(v[x], DT);
    }
};

// What a thread holds of KU depths: TM rows of A, TN columns of B. Two neighbouring columns are one operand of a packed
// multiply-add (fma.rn.f32x2 rounds each half by itself, as two fmaf do).
template <int TM, int TN, int KU>
struct Frag {
    float4 a[TM][KU / 4];
    union { float b[KU][TN]; uint64_t b2[KU][(TN + 1) / 2]; };
};

// One BM x BN tile whose first cell is (row0, col0); columns at or past col_end are not stored.
template <int DT, int BM, int BN, int BK, int TM, int TN, int KU, int THREADS, int STAGES, bool FUSED>
__device__ __forceinline__ void tile(const Params& p, float* smem, uint32_t row0, uint32_t col0, uint32_t col_end) {
    constexpr int TX = BN / TN, TY = THREADS / TX;
    constexpr int A_LD = BK + 4;   // rows of A 4 words further in the banks each: the rows a warp reads together do not meet
    constexpr int STAGE = BM * A_LD + BK * BN;
        constexpr bool PACKED = FUSED && TN % 2 == 0;
    // A warp is 8 x 4 threads, the lanes' bits in the order column, row, column, column, row: a 128-bit read of shared memory
    // takes two wavefronts instead of four only where lanes one or two apart ask for the same address
    constexpr bool WOVEN = TX % 8 == 0 && TY % 4 == 0;
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    const int tx = WOVEN ? (warp % (TX / 8 + (TX < 8))) * 8 + (lane & 1) + ((lane >> 1) & 6) : threadIdx.x % TX;
    const int ty = WOVEN ? (warp / (TX / 8 + (TX < 8))) * 4 + ((lane >> 1) & 1) + ((lane >> 3) & 2) : threadIdx.x / TX;
    const uint32_t tiles = (p.k + BK - 1) / BK;

    // Every thread brings the same places of each tile: row r0 + x * ROWS, columns from c0, `W` words wide. Rows past m, columns
    // past col_end and depths past k stay as they are in shared memory: no cell that is stored reads them.
    typedef typename Element<DT>::type E;
    const E *a = reinterpret_cast<const E*>(p.a) + (uint64_t)row0 * p.k, *b = reinterpret_cast<const E*>(p.b) + col0;
    const uint32_t rows_here = min((uint32_t)BM, p.m - row0), cols_here = min((uint32_t)BN, col_end - col0);
    // f32: copies in flight STAGES - 1 tiles ahead
    auto request = [&](uint32_t t) {
        float *sa = smem + (t % STAGES) * STAGE, *sb = sa + BM * A_LD;
        const uint32_t k0 = t * BK, depth = min((uint32_t)BK, p.k - k0);
        if (p.vec_a) copy_tile<BM, BK, 4, A_LD, THREADS>(sa, reinterpret_cast<const float*>(a) + k0, p.k, rows_here, depth);
        else copy_tile<BM, BK, 1, A_LD, THREADS>(sa, reinterpret_cast<const float*>(a) + k0, p.k, rows_here, depth);
        if (FUSED && p.vec_b) copy_tile<BK, BN, 4, BN, THREADS>(sb, reinterpret_cast<const float*>(b) + (uint64_t)k0 * p.n, p.n, depth, cols_here);
        else copy_tile<BK, BN, 1, BN, THREADS>(sb, reinterpret_cast<const float*>(b) + (uint64_t)k0 * p.n, p.n, depth, cols_here);
    };
    // 16-bit: the next tile waits in registers while this one is worked on
    Held<DT, BM, BK, THREADS> ra;
    Held<DT, BK, BN, THREADS> rb;
    auto fetch = [&](uint32_t t) {
        const uint32_t k0 = t * BK, depth = min((uint32_t)BK, p.k - k0);
        ra.load(reinterpret_cast<const uint16_t*>(a) + k0, p.k, rows_here, depth);
        rb.load(reinterpret_cast<const uint16_t*>(b) + (uint64_t)k0 * p.n, p.n, depth, cols_here);
    };
    auto put = [&](uint32_t t) {
        float* s = smem + (t % STAGES) * STAGE;
        ra.template store<A_LD>(s);
        rb.template store<BN>(s + BM * A_LD);
    };

    union { float f[TM][TN]; uint64_t two[TM][(TN + 1) / 2]; } acc;
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc.f[i][j] = 0.0f;
    // the row a thread's i-th cell lies in; tiles with fewer rows than thread rows repeat the last one (those cells are not stored)
    auto local_row = [&](int i) { const int r = ty + i * TY; return TM * TY > BM && r >= BM ? BM - 1 : r; };
    // the tile's column of a thread's j-th cell: groups of four (or two) a whole row of threads apart
    constexpr int TG = TN % 4 == 0 ? 4 : TN;
    auto local_col = [&](int j) { return (j / TG) * (TX * TG) + tx * TG + j % TG; };

    const float *sa = nullptr, *sb = nullptr;
    auto load = [&](Frag<TM, TN, KU>& f, int kk) {
#pragma unroll
        for (int i = 0; i < TM; ++i)
#pragma unroll
            for (int e = 0; e < KU / 4; ++e) f.a[i][e] = *reinterpret_cast<const float4*>(sa + local_row(i) * A_LD + kk + 4 * e);
#pragma unroll
        for (int e = 0; e < KU; ++e) {
            if (TN % 4 == 0) {
#pragma unroll
                for (int j = 0; j < TN / 4; ++j) *reinterpret_cast<ulonglong2*>(&f.b2[e][2 * j]) = *reinterpret_cast<const ulonglong2*>(sb + (kk + e) * BN + local_col(4 * j));
            } else if (TN == 2) {
                f.b2[e][0] = *reinterpret_cast<const uint64_t*>(sb + (kk + e) * BN + local_col(0));
            } else {
                f.b[e][0] = sb[(kk + e) * BN + local_col(0)];
            }
        }
    };
    auto add = [&](const Frag<TM, TN, KU>& f) {
#pragma unroll
        for (int e = 0; e < KU; ++e)
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 v = f.a[i][e / 4];
                const float a = e % 4 == 0 ? v.x : e % 4 == 1 ? v.y : e % 4 == 2 ? v.z : v.w;
                if (PACKED) {
                    const uint64_t aa = both(a);
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc.two[i][j]) : "l"(aa), "l"(f.b2[e][j]));
                } else {
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc.f[i][j] = FUSED ? __fmaf_rn(a, f.b[e][j], acc.f[i][j]) : __fadd_rn(acc.f[i][j], __fmul_rn(a, f.b[e][j]));
                }
            }
    };

    if (DT == HOLO_DTYPE_F32) {
#pragma unroll
        for (int s = 0; s < STAGES - 1; ++s) {
            if ((uint32_t)s < tiles) request(s);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
    } else {
        fetch(0);
    }
#pragma unroll 1
    for (uint32_t t = 0; t < tiles; ++t) {
        if (DT == HOLO_DTYPE_F32) {
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            __syncthreads();            // tile t is here for every thread, and everybody has left tile t - 1
            if (t + STAGES - 1 < tiles) request(t + STAGES - 1);
            asm volatile("cp.async.commit_group;" ::: "memory");
        } else {
            put(t);                     // two buffers: the last reads of this one ended before the barrier of tile t - 1
            __syncthreads();
            if (t + 1 < tiles) fetch(t + 1);
        }
        sa = smem + (t % STAGES) * STAGE;
        sb = sa + BM * A_LD;
        const int depth = min((uint32_t)BK, p.k - t * BK);
        // the next depths are on their way from shared memory while these are worked on
        Frag<TM, TN, KU> f0, f1;
        if (depth == BK) {
            static_assert(BK % (2 * KU) == 0, "a tile is a whole number of pairs of steps");
            load(f0, 0);
#pragma unroll 1
            for (int kk = 0; kk < BK; kk += 2 * KU) {
                load(f1, kk + KU);
                add(f0);
                if (kk + 2 * KU < BK) load(f0, kk + 2 * KU);
                add(f1);
            }
        } else {
            // no padded depths: a product of zeros would turn a chain's -0 into +0
            int kk = 0;
#pragma unroll 1
            for (; kk + KU <= depth; kk += KU) {
                load(f0, kk);
                add(f0);
            }
#pragma unroll 1
            for (; kk < depth; ++kk) {
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    const float b = sb[kk * BN + local_col(j)];
#pragma unroll
                    for (int i = 0; i < TM; ++i) {
                        const float a = sa[local_row(i) * A_LD + kk];
                        acc.f[i][j] = FUSED ? __fmaf_rn(a, b, acc.f[i][j]) : __fadd_rn(acc.f[i][j], __fmul_rn(a, b));
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const uint32_t r = ty + i * TY;
        if (r >= BM || row0 + r >= p.m) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const uint32_t c = col0 + local_col(j);
            if (c < col_end) store_cell<DT>(p, acc.f[i][j], (uint64_t)(row0 + r) * p.n + c);
        }
    }
}

// The multiply-then-add columns of the tail are a block of their own beside the last full one: two instructions per cell in
// a tile of the same width would make that block the longest of the launch.
template <int DT, int BM, int BN, int BK, int TM, int TN, int KU, int THREADS, int STAGES>
__global__ void __launch_bounds__(THREADS) matmul_cell_kernel(const Params p) {
    extern __shared__ __align__(16) float cell_smem[];
    holo_pdl_trigger();
    holo_pdl_wait();
    const uint32_t row0 = blockIdx.y * BM;
    if (blockIdx.x < p.main_blocks) {
        tile<DT, BM, BN, BK, TM, TN, KU, THREADS, STAGES, true>(p, cell_smem, row0, blockIdx.x * BN, p.n8);
    } else {
        constexpr int TAIL_TM = (BM * 8 + THREADS - 1) / THREADS;
        tile<DT, BM, 8, BK, TAIL_TM, 1, (TAIL_TM > 1 ? 4 : 8), THREADS, STAGES, false>(p, cell_smem, row0, p.n8, p.n);
    }
}

// One thread per cell, operands from global memory: nothing to fill or to wait for
constexpr uint32_t THREAD_COLS = 128;
template <int DT>
__global__ void __launch_bounds__(THREAD_COLS) matmul_thread_kernel(const Params p) {
    holo_pdl_trigger();
    holo_pdl_wait();
    const uint32_t j = blockIdx.x * THREAD_COLS + threadIdx.x, i = blockIdx.y;
    if (j >= p.n) return;
    const bool fused = j < p.n8;
    float acc = 0.0f;
    for (uint32_t kk = 0; kk < p.k; ++kk) {
        const float a = holo::load_float(p.a, (uint64_t)i * p.k + kk, DT), b = holo::load_float(p.b, (uint64_t)kk * p.n + j, DT);
        acc = fused ? __fmaf_rn(a, b, acc) : __fadd_rn(acc, __fmul_rn(a, b));
    }
    store_cell<DT>(p, acc, (uint64_t)i * p.n + j);
}

// Where that is the quicker one. Short chains do not pay for the ring: us, a thread per cell / tiles, f32 1 x 4 x 1001 1.4 / 1.8,
// 300 x 4 x 129 1.8 / 2.4, f16 300 x 1 x 2001 5.8 / 15; the lines are where enough cells or depth share a tile. With up to 8 rows the
// product is a pass over B, and the wider B is the deeper it may be before a 4 x 32 tile, three quarters of it idle for one row, is
// the better way to read it: f32 1 x 201 x 100001 15 / 32, 8 x 33 x 100001 10.6 / 16.4, 8 x 404 x 100001 131 / 121.
template <int DT>
bool thread_per_cell(const Params& p) {
    constexpr bool F16 = DT == HOLO_DTYPE_F16;      // widening f16 takes a dozen instructions, which a tile does once
    const uint64_t cells = (uint64_t)p.m * p.n;
    if (p.m <= 8) {
        if (F16) return p.k <= 10 + (p.m == 1 ? p.n / 2500 : min(p.n / 3500, 28u));
        if (p.m == 1 && p.n >= 100000) return true;
        return p.k <= 16 + (p.m <= 2 ? p.n / (700 * p.m) : min(p.n / 1500, 104u));
    }
    if (p.n < 8) return p.k <= 4 && p.m <= 1000;
    if (F16) return p.m <= 4000 && cells <= 800000 && p.k <= (cells >= 40000 ? 12u : 6u);
    if (DT == HOLO_DTYPE_BF16) return p.m <= 1200 && cells <= 800000 && p.k <= 20;
    return p.m <= 2001 && cells <= (p.m <= 64 ? 400000u : 200000u) && p.k <= 24;
}

template <int DT, int BM, int BN, int BK, int TM, int TN, int KU, int THREADS>
int32_t launch(holo_b200_ctx* ctx, Params p) {
    constexpr int STAGES = DT == HOLO_DTYPE_F32 ? 3 : 2;
    constexpr size_t SMEM = sizeof(float) * STAGES * (BM * (BK + 4) + BK * BN);
    auto kernel = matmul_cell_kernel<DT, BM, BN, BK, TM, TN, KU, THREADS, STAGES>;
    if (SMEM > 48 * 1024) {
        static thread_local int configured_device = -1;
        if (configured_device != ctx->device) {
            HOLO_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)SMEM));
            configured_device = ctx->device;
        }
    }
    p.main_blocks = (p.n8 + BN - 1) / BN;
    const dim3 grid(p.main_blocks + (p.n8 < p.n ? 1 : 0), (p.m + BM - 1) / BM);
    HOLO_CUDA(holo_launch_kernel(ctx, kernel, grid, dim3(THREADS), SMEM, 1, p));
    ctx->launches++;
    return HOLO_OK;
}

// Which kernel: see above; else which tile: few rows are bound by the chain's latency and by the weight's way to shared memory (4 rows, deep steps); up to
// one 16 x 32 tile per SM four warps share each; more of them fill an SM several deep with two warps each; large products
// spend fewest reads of shared memory in 64 x 32 tiles. Measured f32, us, in this order (the one taken in brackets):
// 1 x 1024 x 1024 [7.7] 12.1 14.0 25.3; 32 x 1000 x 771 21.9 [15.0] 17.5 26.3; 512^3 29.0 16.2 [16.0] 32.7;
// 500 x 1000 x 771 106 46.5 [35.9] 65.7; 381 x 768 x 3072 179 67.7 55.4 [50.6]; 1000 x 2048 x 2048 825 299 237 [209].
template <int DT>
int32_t launch_sized(holo_b200_ctx* ctx, const Params& p) {
    if (thread_per_cell<DT>(p)) {
        HOLO_CUDA(holo_launch_kernel(ctx, matmul_thread_kernel<DT>, dim3((p.n + THREAD_COLS - 1) / THREAD_COLS, p.m), dim3(THREAD_COLS), 0, 1, p));
        ctx->launches++;
        return HOLO_OK;
    }
    const uint64_t sms = (uint64_t)ctx->sm_count;
    auto tiles = [&](uint64_t bm, uint64_t bn) { return (p.m + bm - 1) / bm * ((p.n + bn - 1) / bn); };
    if (p.m <= 8) return launch<DT, 4, 32, 128, 1, 1, 16, 128>(ctx, p);
    if (tiles(16, 32) <= sms) return launch<DT, 16, 32, 64, 2, 2, 8, 128>(ctx, p);
    if (2 * tiles(64, 32) < 7 * sms) return launch<DT, 16, 32, 64, 2, 4, 8, 64>(ctx, p);
    return launch<DT, 64, 32, 32, 4, 4, 4, 128>(ctx, p);
}

}  // namespace

int32_t holo_launch_matmul_cell(holo_b200_ctx* ctx, const void* a, const void* b, void* out, const uint16_t* table, int act, const void* residual, uint32_t m,
                                uint32_t k, uint32_t n, uint8_t dtype, int add_first) {
    if (m > 65535) return holo_fail(HOLO_ERR_UNSUPPORTED_OP, "unsupported op: matmul m %u on the per-cell path", m);
    Params p = {a, b, out, table, residual, m, k, n, n - n % 8, 0, act, add_first, false, false};
    p.vec_a = (k % 4) == 0 && ((uintptr_t)a & 15u) == 0;
    p.vec_b = (n % 4) == 0 && ((uintptr_t)b & 15u) == 0;
    if (dtype == HOLO_DTYPE_F32) return launch_sized<HOLO_DTYPE_F32>(ctx, p);
    return dtype == HOLO_DTYPE_F16 ? launch_sized<HOLO_DTYPE_F16>(ctx, p) : launch_sized<HOLO_DTYPE_BF16>(ctx, p);
}
