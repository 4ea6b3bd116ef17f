// C = A · W^T in 32-bit on the FMA units, for inputs whose rows can be fetched 16 bytes at a time.  As in gemm_simt.cu
// every output element is one sequential sum of fused multiply-adds over k = 0..K-1, so the results of the three kernels
// are the same bits, whatever tile, batch or expert group a row was computed in.
//
//   gemm_f32_tile   many rows: a block of (BM / 8)(BN / 8) threads, 8 x 8 outputs a thread, the next slice of K on its way
//                   from global memory into registers while this one is multiplied out of shared memory.  Bound by the FMA
//                   pipe: 32 packed multiply-adds (fma.rn.f32x2, two rounded sums each) meet four 16-byte shared loads.
//   gemm_f32_few    few rows (a decode step, experts with a few rows each): bound by reading W once.  16 columns a block,
//                   so that even a product of 2,048 columns spreads over 128 multiprocessors, and a ring of asynchronous copies
//                   that keeps 32-48 KB a block in flight, 72-86 KB where there are at most two blocks a multiprocessor; a thread owns one column and RPT rows, and the only
//                   serial chain is the sum itself (4 clocks a k).
#include "api.h"
#include "common.cuh"
#include "gemm_internal.h"

namespace dlmk {

namespace {

struct F32Params {
    const float* a; int lda; const int32_t* a_rows;
    const float* w; int ldw; long long w_expert_stride;
    const int32_t* expert_offsets; int num_experts;
    const float* bias;
    float* out; int ldo;
    int M, N, K;
    int vec_out;
};

struct RowTile { int expert, begin, end; };

// Row tile `ty` when every expert's rows are cut into tiles of `rows`; asked by a whole warp.  expert < 0: there is none.
__device__ __forceinline__ RowTile find_row_tile(const int32_t* offsets, int E, int rows, int ty) {
    const int lane = threadIdx.x & 31;
    int acc = 0;
    for (int base = 0; base < E; base += 32) {
        const int e = base + lane;
        const int r0 = e < E ? offsets[e] : 0, r1 = e < E ? offsets[e + 1] : 0;
        const int tiles = (r1 - r0 + rows - 1) / rows;
        int upto = tiles;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, upto, o);
            if (lane >= o) upto += v;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, acc + upto > ty);
        if (hit != 0) {
            const int src = __ffs(hit) - 1;
            const int before = acc + __shfl_sync(0xffffffffu, upto - tiles, src);
            RowTile t;
            t.expert = base + src;
            t.begin = __shfl_sync(0xffffffffu, r0, src) + (ty - before) * rows;
            t.end = min(__shfl_sync(0xffffffffu, r1, src), t.begin + rows);
            return t;
        }
        acc += __shfl_sync(0xffffffffu, upto, 31);
    }
    return RowTile{-1, 0, 0};
}

// What a tile's block works on, told to every thread: expert (0 when dense), first row, end row.
__device__ __forceinline__ RowTile block_row_tile(const F32Params& p, int rows, int ty, int* shared3) {
    RowTile t{0, ty * rows, min(p.M, (ty + 1) * rows)};
    if (p.expert_offsets != nullptr) {
        if (threadIdx.x < 32) {
            const RowTile f = find_row_tile(p.expert_offsets, p.num_experts, rows, ty);
            if (threadIdx.x == 0) { shared3[0] = f.expert; shared3[1] = f.begin; shared3[2] = min(f.end, p.M); }
        }
        __syncthreads();
        t.expert = shared3[0];
        t.begin = shared3[1];
        t.end = shared3[2];
    }
    return t;
}

__device__ __forceinline__ unsigned long long pack_f32x2(float lo, float hi) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack_f32x2(unsigned long long v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// two fused multiply-adds, each rounded as fmaf rounds
__device__ __forceinline__ void fma_f32x2(unsigned long long& d, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}

// Four neighbouring columns (col % 4 == 0) of one row.
template <int EPI>
__device__ __forceinline__ void store4(const F32Params& p, int row, int col, const float (&v)[4]) {
    if (epi_is_glu(EPI)) {
        float* o = p.out + (long long)row * p.ldo;
#pragma unroll
        for (int j = 0; j < 4; j += 2)
            if (col + j + 1 < p.N) o[(col + j) >> 1] = glu_out<EPI, false>(v[j], v[j + 1], p.bias);
    } else {
        float* o = p.out + (long long)row * p.ldo + col;
        float r[4];
#pragma unroll
        for (int j = 0; j < 4; ++j)
            r[j] = EPI == EPI_ADD ? v[j] : epi_act<EPI>(v[j] + (p.bias != nullptr && col + j < p.N ? p.bias[col + j] : 0.f));
        if (p.vec_out && col + 3 < p.N) {
            float4 x = make_float4(r[0], r[1], r[2], r[3]);
            if (EPI == EPI_ADD) {
                const float4 old = *reinterpret_cast<const float4*>(o);
                x = make_float4(old.x + r[0], old.y + r[1], old.z + r[2], old.w + r[3]);
            }
            *reinterpret_cast<float4*>(o) = x;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (col + j < p.N) o[j] = EPI == EPI_ADD ? o[j] + r[j] : r[j];
        }
    }
}

// ------------------------------------------------------------------------------------------------ many rows
constexpr int TBK = 16;

// (512 threads a multiprocessor, 128 registers each: with the 130 the compiler takes by itself there is room for 256)
template <int BM, int BN, int EPI>
__global__ void __launch_bounds__((BM / 8) * (BN / 8), 512 / ((BM / 8) * (BN / 8))) gemm_f32_tile_kernel(F32Params p) {
    constexpr int TX = BN / 8, THREADS = (BM / 8) * TX;
    constexpr int PA = BM + 4, PB = BN + 4;
    constexpr int LA = BM * (TBK / 4) / THREADS, LB = BN * (TBK / 4) / THREADS;     // 16-byte loads a thread and slice
    static_assert(LA * THREADS == BM * (TBK / 4) && LB * THREADS == BN * (TBK / 4), "every thread loads the same");
    __shared__ __align__(16) float As[2][TBK][PA];
    __shared__ __align__(16) float Bs[2][TBK][PB];
    __shared__ int s_tile[3];

    const int tid = threadIdx.x;
    const int n0 = blockIdx.x * BN;
    const RowTile rt = block_row_tile(p, BM, blockIdx.y, s_tile);
    if (rt.expert < 0 || rt.begin >= rt.end) return;
    const float* w = p.w + (long long)rt.expert * p.w_expert_stride;

    const float* a_src[LA];
    const float* b_src[LB];
#pragma unroll
    for (int i = 0; i < LA; ++i) {
        const int idx = tid + i * THREADS, r = rt.begin + (idx >> 2);
        a_src[i] = r < rt.end ? p.a + (long long)(p.a_rows != nullptr ? p.a_rows[r] : r) * p.lda + (idx & 3) * 4 : nullptr;
    }
#pragma unroll
    for (int i = 0; i < LB; ++i) {
        const int idx = tid + i * THREADS, n = n0 + (idx >> 2);
        b_src[i] = n < p.N ? w + (long long)n * p.ldw + (idx & 3) * 4 : nullptr;
    }
    const int kq = (tid & 3) * 4;                 // THREADS is a multiple of 4: the same for every load of a thread
    float4 ra[LA], rb[LB];
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load = [&](int k0) {                     // K is a multiple of 4
        const bool in = k0 + kq < p.K;
#pragma unroll
        for (int i = 0; i < LA; ++i) ra[i] = in && a_src[i] != nullptr ? *reinterpret_cast<const float4*>(a_src[i] + k0) : zero;
#pragma unroll
        for (int i = 0; i < LB; ++i) rb[i] = in && b_src[i] != nullptr ? *reinterpret_cast<const float4*>(b_src[i] + k0) : zero;
    };
    auto put = [&](int s) {
#pragma unroll
        for (int i = 0; i < LA; ++i) {
            const int r = (tid + i * THREADS) >> 2;
            As[s][kq][r] = ra[i].x; As[s][kq + 1][r] = ra[i].y; As[s][kq + 2][r] = ra[i].z; As[s][kq + 3][r] = ra[i].w;
        }
#pragma unroll
        for (int i = 0; i < LB; ++i) {
            const int r = (tid + i * THREADS) >> 2;
            Bs[s][kq][r] = rb[i].x; Bs[s][kq + 1][r] = rb[i].y; Bs[s][kq + 2][r] = rb[i].z; Bs[s][kq + 3][r] = rb[i].w;
        }
    };

    const int ty = tid / TX, tx = tid % TX;
    unsigned long long acc[8][4];                 // rows x pairs of columns
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;

    load(0);
    put(0);
    __syncthreads();
    int s = 0;
    for (int k0 = 0; k0 < p.K; k0 += TBK, s ^= 1) {
        const bool more = k0 + TBK < p.K;
        if (more) load(k0 + TBK);
#pragma unroll
        for (int k = 0; k < TBK; ++k) {
            const float4 a0 = *reinterpret_cast<const float4*>(&As[s][k][ty * 4]);
            const float4 a1 = *reinterpret_cast<const float4*>(&As[s][k][BM / 2 + ty * 4]);
            const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(&Bs[s][k][tx * 4]);
            const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(&Bs[s][k][BN / 2 + tx * 4]);
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const unsigned long long aa = pack_f32x2(a[i], a[i]);
                fma_f32x2(acc[i][0], aa, b0.x);
                fma_f32x2(acc[i][1], aa, b0.y);
                fma_f32x2(acc[i][2], aa, b1.x);
                fma_f32x2(acc[i][3], aa, b1.y);
            }
        }
        if (more) {
            put(s ^ 1);                           // the slice before the last barrier's has been read by everyone
            __syncthreads();
        }
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int row = rt.begin + (i >> 2) * (BM / 2) + ty * 4 + (i & 3);
        if (row >= rt.end) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const float2 lo = unpack_f32x2(acc[i][2 * h]), hi = unpack_f32x2(acc[i][2 * h + 1]);
            const float v[4] = {lo.x, lo.y, hi.x, hi.y};
            const int col = n0 + h * (BN / 2) + tx * 4;
            if (col < p.N) store4<EPI>(p, row, col, v);
        }
    }
}

// ------------------------------------------------------------------------------------------------- few rows
constexpr int FBN = 16, FKC = 128, FPITCH = FKC + 4, FTHREADS = 128, FGROUPS = 8;

__device__ __forceinline__ void copy16(float* dst, const float* src, bool real) {
    const unsigned d = static_cast<unsigned>(__cvta_generic_to_shared(dst));
    const int bytes = real ? 16 : 0;              // the rest is filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(bytes) : "memory");
}

// DEEP: a launch of at most two blocks a multiprocessor; otherwise more blocks with shorter rings hide more of each other
template <int RPT, bool DEEP> constexpr int few_stages() { return DEEP ? (RPT == 1 ? 8 : (RPT == 2 ? 6 : 4)) : (RPT == 1 ? 4 : 3); }
template <int RPT, bool DEEP> constexpr size_t few_smem() {
    return (size_t)few_stages<RPT, DEEP>() * (FBN + FGROUPS * RPT) * FPITCH * sizeof(float);
}

// Lane = (column, one of two row groups); row r of the tile belongs to group r % 8, so few rows spread over the warps.
template <int RPT, bool DEEP, int EPI>
__global__ void __launch_bounds__(FTHREADS) gemm_f32_few_kernel(F32Params p) {
    constexpr int R = FGROUPS * RPT, STAGES = few_stages<RPT, DEEP>(), STAGE = (FBN + R) * FPITCH;
    extern __shared__ __align__(16) float sm[];   // [STAGES][16 rows of W | R rows of A][FPITCH]
    __shared__ int s_tile[3];
    __shared__ const float* s_row[R];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * FBN;
    const RowTile rt = block_row_tile(p, R, blockIdx.y, s_tile);
    if (rt.expert < 0 || rt.begin >= rt.end) return;
    const int n_rows = rt.end - rt.begin;
    const float* w = p.w + (long long)rt.expert * p.w_expert_stride + (long long)n0 * p.ldw;
    for (int r = tid; r < n_rows; r += FTHREADS) {
        const int row = rt.begin + r;
        s_row[r] = p.a + (long long)(p.a_rows != nullptr ? p.a_rows[row] : row) * p.lda;
    }
    __syncthreads();
    const int n_cols = min(FBN, p.N - n0);
    const int chunks = (p.K + FKC - 1) / FKC;
    auto fetch = [&](int c) {                     // (a chunk beyond the last: an empty group, so that the count holds)
        if (c < chunks) {
            float* dst = sm + (size_t)(c % STAGES) * STAGE;
            const int k0 = c * FKC + 4 * lane;    // a warp a row: 32 lanes x 16 bytes
            const bool in = k0 < p.K;
#pragma unroll
            for (int r = warp; r < FBN; r += 4) {
                const bool real = in && r < n_cols;
                copy16(dst + r * FPITCH + 4 * lane, real ? w + (long long)r * p.ldw + k0 : p.w, real);
            }
            for (int r = warp; r < n_rows; r += 4)
                copy16(dst + (FBN + r) * FPITCH + 4 * lane, in ? s_row[r] + k0 : p.a, in);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int col = lane & 15, group = warp * 2 + (lane >> 4);
    const bool busy = warp * 2 < n_rows;          // of a warp's two groups the first holds a row
    float acc[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) acc[i] = 0.f;
#pragma unroll
    for (int c = 0; c < STAGES - 1; ++c) fetch(c);
    for (int c = 0; c < chunks; ++c) {
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                          // chunk c is there, and everyone has left chunk c - 1's stage
        fetch(c + STAGES - 1);
        if (busy) {
            const float* st = sm + (size_t)(c % STAGES) * STAGE;
            const float* wr = st + col * FPITCH;
            const float* ar = st + (FBN + group) * FPITCH;
#pragma unroll 8
            for (int k = 0; k < FKC; k += 4) {
                const float4 wv = *reinterpret_cast<const float4*>(wr + k);
#pragma unroll
                for (int i = 0; i < RPT; ++i) {
                    const float4 av = *reinterpret_cast<const float4*>(ar + i * FGROUPS * FPITCH + k);
                    acc[i] = fmaf(av.x, wv.x, acc[i]);
                    acc[i] = fmaf(av.y, wv.y, acc[i]);
                    acc[i] = fmaf(av.z, wv.z, acc[i]);
                    acc[i] = fmaf(av.w, wv.w, acc[i]);
                }
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int r = group + FGROUPS * i;
        const int c = n0 + col;
        if (epi_is_glu(EPI)) {
            const float up = __shfl_down_sync(0xffffffffu, acc[i], 1);
            if (r < n_rows && (col & 1) == 0 && c + 1 < p.N)
                p.out[(long long)(rt.begin + r) * p.ldo + (c >> 1)] = glu_out<EPI, false>(acc[i], up, p.bias);
        } else if (r < n_rows && c < p.N) {
            float* o = p.out + (long long)(rt.begin + r) * p.ldo + c;
            *o = EPI == EPI_ADD ? *o + acc[i] : epi_act<EPI>(acc[i] + (p.bias != nullptr ? p.bias[c] : 0.f));
        }
    }
}

template <int EPI>
void launch_tile(const F32Params& p, bool big, int m_extra, cudaStream_t stream) {
    const int bm = big ? 128 : 64;
    const dim3 grid((p.N + 127) / 128, (p.M + bm - 1) / bm + m_extra);
    if (big) gemm_f32_tile_kernel<128, 128, EPI><<<grid, 256, 0, stream>>>(p);
    else gemm_f32_tile_kernel<64, 128, EPI><<<grid, 128, 0, stream>>>(p);
}

template <int EPI, int RPT, bool DEEP>
void launch_few_ring(const F32Params& p, const dim3& grid, cudaStream_t stream) {
    auto kern = gemm_f32_few_kernel<RPT, DEEP, EPI>;
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)few_smem<RPT, DEEP>());
    kern<<<grid, FTHREADS, few_smem<RPT, DEEP>(), stream>>>(p);
}
template <int EPI, int RPT>
void launch_few(const F32Params& p, int m_tiles, cudaStream_t stream) {
    const dim3 grid((p.N + FBN - 1) / FBN, m_tiles);
    if ((long long)grid.x * grid.y <= 2LL * sm_count()) launch_few_ring<EPI, RPT, true>(p, grid, stream);
    else launch_few_ring<EPI, RPT, false>(p, grid, stream);
}

// Which kernel: measured at K = 2,048 (all three grow with K alike), beside gemm_simt's 64 x 64 tiles.
//   few    up to 32 rows (2,048 / 11,264 / 32,768 columns, 32 rows: 29 / 105 / 249 us, gemm_simt 123 / 214 / 364) and up to 16
//          rows an expert on average (60 experts x 2,816 columns, 8 rows each: 647 us against 1,515; at 12 rows 1,072 against
//          some 900 of the tiles).  From 33 to 64 rows the weights are read twice: up to 640,000 outputs (64 rows of 6,144 columns:
//          111 us against 183 of the tiles; 64 rows of 32,768 columns: 488 us, where gemm_simt takes 391).
//   tile   where gemm_simt would have more than one tile a multiprocessor: its second wave starts there (512 x 2,048: 218 us
//          against 184; 65 x 6,144: 205 against 183; 2,048 x 2,048: 683 against 433).
//   none   fewer tiles than that: a thread's 64 sums are then too long a walk (65-256 rows of 2,048 columns: 183 us against 132
//          of gemm_simt; 128 x 256, K = 256: 27 against 19).
enum class Plan { none, few, tile };
Plan plan(int M, int N, int num_experts) {
    const int mean = num_experts > 0 ? (M + num_experts - 1) / num_experts : M;
    if (num_experts > 0 ? mean <= 16 : mean <= 32 || (mean <= 64 && (long long)M * N < 640000)) return Plan::few;
    const long long row_tiles = num_experts > 0 ? (long long)num_experts * (mean / 64 + 1) : (M + 63) / 64;
    return row_tiles * ((N + 63) / 64) > sm_count() ? Plan::tile : Plan::none;
}

template <int EPI>
void launch(const F32Params& p, cudaStream_t stream) {
    const bool grouped = p.expert_offsets != nullptr;
    const int mean = grouped ? (p.M + p.num_experts - 1) / p.num_experts : p.M;
    if (plan(p.M, p.N, grouped ? p.num_experts : 0) == Plan::few) {
        // an expert's rows vary about their mean: the tile holds twice the mean where it can
        const int want = grouped ? 2 * mean : mean;
        const int r = want <= 8 ? 8 : (want <= 16 ? 16 : 32);
        int tiles = (p.M + r - 1) / r + (grouped ? p.num_experts : 0);
        if (tiles > p.M) tiles = p.M;             // every tile holds at least one row
        if (r == 8) launch_few<EPI, 1>(p, tiles, stream);
        else if (r == 16) launch_few<EPI, 2>(p, tiles, stream);
        else launch_few<EPI, 4>(p, tiles, stream);
        return;
    }
    const long long big_blocks = (long long)((p.N + 127) / 128) * ((p.M + 127) / 128);
    launch_tile<EPI>(p, !grouped && big_blocks >= 2 * sm_count(), grouped ? p.num_experts : 0, stream);
}

}  // namespace

bool gemm_f32_takes(const void* a, int lda, const void* w, int ldw, long long w_expert_stride, int M, int N, int K, int num_experts) {
    return plan(M, N, num_experts) != Plan::none && K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && w_expert_stride % 4 == 0 &&
           ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) & 15) == 0;
}

void gemm_f32(const float* a, int lda, const int32_t* a_rows, const float* w, int ldw, long long w_expert_stride,
              const int32_t* expert_offsets, int num_experts, const float* bias, float* out, int ldo, int M, int N, int K,
              int epilogue, cudaStream_t stream) {
    const int vec_out = ldo % 4 == 0 && (reinterpret_cast<uintptr_t>(out) & 15) == 0 ? 1 : 0;
    const F32Params p{a, lda, a_rows, w, ldw, w_expert_stride, expert_offsets, num_experts, bias, out, ldo, M, N, K, vec_out};
    switch (epilogue) {
        case EPI_STORE: launch<EPI_STORE>(p, stream); break;
        case EPI_ADD: launch<EPI_ADD>(p, stream); break;
        case EPI_SWIGLU: launch<EPI_SWIGLU>(p, stream); break;
        case EPI_GELU: launch<EPI_GELU>(p, stream); break;
        case EPI_GELU_TANH: launch<EPI_GELU_TANH>(p, stream); break;
        case EPI_GEGLU_TANH: launch<EPI_GEGLU_TANH>(p, stream); break;
        case EPI_CLAMP_GLU: launch<EPI_CLAMP_GLU>(p, stream); break;
        default: DLM_CHECK(false, "gemm: unknown epilogue");
    }
    check_launch("gemm_f32");
}

}  // namespace dlmk
