// Paged causal attention in 32-bit on the FMA units for head sizes that are a multiple of four, up to 128: the sums of
// attention_simt.cu in the same order (a score is one chain over the head's entries, a tile's probabilities are added by the
// same tree over its 32 keys, an output entry is one chain over the keys), so the results are the same bits.
//
// What bound the kernel that serves any head size was its loads: one 4-byte load with its page look-up per element, two
// shared-memory reads per multiply-add, and nothing in flight while a tile was worked on.  Here a block of BQ queries of one
// head works in tiles of registers: scores 4 queries x KPT keys a thread out of 16-byte shared loads, the softmax step with a
// key a lane, then 4 queries x DPT entries of the output a thread; the next tile of keys and values arrives meanwhile by
// 16-byte asynchronous copies.  BQ = 32 for prompts, 16 where that leaves multiprocessors without a block.
#include "api.h"
#include "attention_internal.h"
#include "common.cuh"

namespace dlmk {

namespace {

constexpr int THREADS = 128, WARPS = 4, BKV = 32, PP = BKV + 4;

__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}

template <int HD, int BQ> constexpr size_t f32_smem() {
    return (size_t)(BQ * (HD + 4) + 2 * BKV * (HD + 4) + 2 * BKV * HD + BQ * PP + BQ) * sizeof(float);
}

// HD: the head size rounded up to 64 or 128 (entries beyond the head's own are zeros).
template <int HD, int BQ>
__global__ void __launch_bounds__(THREADS)
attention_f32_kernel(const float* __restrict__ q, const float* __restrict__ k_cache, const float* __restrict__ v_cache,
                     const int32_t* __restrict__ block_table, int table_width, const int32_t* __restrict__ cu_q,
                     const int32_t* __restrict__ kv_len, float* __restrict__ out, int R, int nh, int nkv, int hd,
                     int page_size, int total_pages, int window, Score scale, int skip_single, int* err) {
    constexpr int QG = BQ / 4, LANES = THREADS / QG;       // threads that share four queries
    constexpr int KPT = BKV / LANES;                       // keys a thread scores
    constexpr int DPT = HD / LANES;                        // output entries a thread owns, in runs of RUN
    constexpr int RUN = DPT < 4 ? DPT : 4, RUNS = DPT / RUN;
    constexpr int QP = HD + 4, ROWS = BQ / WARPS;          // rows of the softmax step a warp takes
    static_assert(KPT >= 1 && DPT >= 2, "tile too small for the block");
    extern __shared__ __align__(16) float smem[];
    float* Qs = smem;                                      // [BQ][QP]
    float* Ks = Qs + BQ * QP;                              // [2][BKV][QP]
    float* Vs = Ks + 2 * BKV * QP;                         // [2][BKV][HD]
    float* Ps = Vs + 2 * BKV * HD;                         // [BQ][PP] scores, then probabilities
    float* s_alpha = Ps + BQ * PP;                         // [BQ]; negative: the row saw nothing in the tile
    __shared__ int s_map[2];

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int head = blockIdx.y, kvh = head / (nh / nkv);
    const float slope = scale.slopes != nullptr ? scale.slopes[head] : 0.f;
    if (tid == 0) {
        int acc = 0;
        s_map[0] = -1;
        const int want = (int)gridDim.x - 1 - (int)blockIdx.x;       // late queries (most keys) first
        for (int r = 0; r < R; ++r) {
            const int ql = cu_q[r + 1] - cu_q[r];
            const int tiles = (skip_single && ql == 1) ? 0 : (ql + BQ - 1) / BQ;
            if (want < acc + tiles) {
                s_map[0] = r;
                s_map[1] = (want - acc) * BQ;
                break;
            }
            acc += tiles;
        }
    }
    __syncthreads();
    const int r = s_map[0];
    if (r < 0) return;
    const int q0 = s_map[1];
    const int q_begin = cu_q[r], q_len = cu_q[r + 1] - q_begin;
    const int n_q = min(BQ, q_len - q0);
    const int len = kv_len[r];
    const int pos0 = len - q_len + q0;
    const int Q = nh * hd;

    for (int idx = tid; idx < BQ * (HD / 4); idx += THREADS) {
        const int qi = idx / (HD / 4), d = 4 * (idx % (HD / 4));
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (qi < n_q && d < hd) v = *reinterpret_cast<const float4*>(q + (long long)(q_begin + q0 + qi) * Q + head * hd + d);
        *reinterpret_cast<float4*>(Qs + qi * QP + d) = v;
    }

    const int hi = pos0 + n_q - 1;
    int lo = 0;
    if (window > 0) lo = max(0, pos0 - window + 1);
    if (scale.chunk > 0) lo = max(lo, (pos0 / scale.chunk) * scale.chunk);
    const int keep = scale.keep;
    const KeyTiles<BKV> tiles(lo, hi, keep);
    const int* table = block_table + (long long)r * table_width;
    const int d_lo = scale.parts == 2 ? (head & 1) * (hd / 2) : 0, d_hi = scale.parts == 2 ? d_lo + hd / 2 : hd;

    auto fetch = [&](int it) {
        const int kv0 = tiles.at(it);
        float* kd = Ks + (it & 1) * BKV * QP;
        float* vd = Vs + (it & 1) * BKV * HD;
        for (int idx = tid; idx < BKV * (HD / 4); idx += THREADS) {
            const int jj = idx / (HD / 4), d = 4 * (idx % (HD / 4));
            const int j = kv0 + jj;
            const float* ks = nullptr;
            const float* vs = nullptr;
            if (j <= hi && (j >= lo || j < keep) && d < hd) {
                const int lp = j / page_size;
                const int page = lp < table_width ? table[lp] : -1;
                if (page >= 0 && page < total_pages) {
                    const long long off = (((long long)page * nkv + kvh) * page_size + (j - lp * page_size)) * hd + d;
                    ks = k_cache + off;
                    vs = v_cache + off;
                } else {
                    *err = 3;        // a visible key without a page: refuse to read, report
                }
            }
            if (ks != nullptr) {
                copy16(kd + jj * QP + d, ks);
                copy16(vd + jj * HD + d, vs);
            } else {
                *reinterpret_cast<float4*>(kd + jj * QP + d) = make_float4(0.f, 0.f, 0.f, 0.f);
                *reinterpret_cast<float4*>(vd + jj * HD + d) = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };

    const int qg = tid / LANES, ql = tid % LANES;
    float m[ROWS], l[ROWS];
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
    }
    float o[4][DPT];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int d = 0; d < DPT; ++d) o[i][d] = 0.f;

    fetch(0);
    for (int it = 0; it < tiles.n; ++it) {
        const int kv0 = tiles.at(it);
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();                                   // the tile is there; the tile before has been left by everyone
        if (it + 1 < tiles.n) fetch(it + 1);
        const float* kt = Ks + (it & 1) * BKV * QP;
        const float* vt = Vs + (it & 1) * BKV * HD;
        {
            float s[4][KPT];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < KPT; ++j) s[i][j] = 0.f;
#pragma unroll 4
            for (int d = d_lo; d < d_hi; d += 4) {
                float4 kv[KPT];
#pragma unroll
                for (int j = 0; j < KPT; ++j) kv[j] = *reinterpret_cast<const float4*>(kt + (ql + LANES * j) * QP + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 qv = *reinterpret_cast<const float4*>(Qs + (4 * qg + i) * QP + d);
#pragma unroll
                    for (int j = 0; j < KPT; ++j) {
                        s[i][j] = fmaf(qv.x, kv[j].x, s[i][j]);
                        s[i][j] = fmaf(qv.y, kv[j].y, s[i][j]);
                        s[i][j] = fmaf(qv.z, kv[j].z, s[i][j]);
                        s[i][j] = fmaf(qv.w, kv[j].w, s[i][j]);
                    }
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < KPT; ++j) Ps[(4 * qg + i) * PP + ql + LANES * j] = s[i][j];
        }
        __syncthreads();
        const int j = kv0 + lane;
#pragma unroll
        for (int i = 0; i < ROWS; ++i) {
            const int qi = warp * ROWS + i;
            float* row = Ps + qi * PP;
            if (qi >= n_q) {                                // uniform over the warp
                row[lane] = 0.f;
                if (lane == 0) s_alpha[qi] = -1.f;
                continue;
            }
            const int p = pos0 + qi;
            float s = row[lane];
            if (scale.softcap > 0.f) s = scale.softcap * tanhf((s * scale.scale) / scale.softcap) - slope * (float)(p - j);
            else s = s * scale.scale - slope * (float)(p - j);
            const bool visible = (j <= p) && (window <= 0 || p - j < window || j < keep) &&
                                 (scale.chunk <= 0 || j >= (p / scale.chunk) * scale.chunk);
            if (!visible) s = -INFINITY;
            const float m_new = fmaxf(m[i], warp_max(s));
            if (m_new == -INFINITY) {                       // this query sees nothing in the tile
                if (lane == 0) s_alpha[qi] = -1.f;
                continue;
            }
            const float pj = visible ? expf(s - m_new) : 0.f;
            const float alpha = expf(m[i] - m_new);         // exp(-inf) = 0 on the first tile with a visible key
            l[i] = l[i] * alpha + warp_sum(pj);
            m[i] = m_new;
            row[lane] = pj;
            if (lane == 0) s_alpha[qi] = alpha;
        }
        __syncthreads();
        bool sees[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float alpha = s_alpha[4 * qg + i];
            sees[i] = alpha >= 0.f;
            if (sees[i]) {
#pragma unroll
                for (int d = 0; d < DPT; ++d) o[i][d] *= alpha;
            }
        }
#pragma unroll 2
        for (int kk = 0; kk < BKV; kk += 4) {
            float pv[4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const float4 x = *reinterpret_cast<const float4*>(Ps + (4 * qg + i) * PP + kk);
                pv[i][0] = x.x; pv[i][1] = x.y; pv[i][2] = x.z; pv[i][3] = x.w;
            }
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                float v[DPT];
#pragma unroll
                for (int u = 0; u < RUNS; ++u) {
                    const float* src = vt + (kk + e) * HD + RUN * (ql + LANES * u);
                    if (RUN == 4) {
                        const float4 x = *reinterpret_cast<const float4*>(src);
                        v[4 * u] = x.x; v[4 * u + 1] = x.y; v[(4 * u + 2) % DPT] = x.z; v[(4 * u + 3) % DPT] = x.w;
                    } else {
                        const float2 x = *reinterpret_cast<const float2*>(src);
                        v[2 * u] = x.x; v[2 * u + 1] = x.y;
                    }
                }
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    if (sees[i]) {
#pragma unroll
                        for (int d = 0; d < DPT; ++d) o[i][d] = fmaf(pv[i][e], v[d], o[i][d]);
                    }
                }
            }
        }
    }

    // every row's 1 / denominator through shared memory to the threads that own its entries
#pragma unroll
    for (int i = 0; i < ROWS; ++i) {
        float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
        if (scale.sinks != nullptr && l[i] > 0.f) {
            const float sk = scale.sinks[head];
            const float M = fmaxf(m[i], sk);
            const float a = expf(m[i] - M);
            inv = a / (l[i] * a + expf(sk - M));
        }
        if (lane == 0) Ps[(warp * ROWS + i) * PP + BKV] = inv;      // (the padding of the row: nobody reads it)
    }
    __syncthreads();
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int qi = 4 * qg + i;
        if (qi >= n_q) continue;
        const float inv = Ps[qi * PP + BKV];
        float* orow = out + (long long)(q_begin + q0 + qi) * Q + head * hd;
#pragma unroll
        for (int u = 0; u < RUNS; ++u)
#pragma unroll
            for (int e = 0; e < RUN; ++e) {
                const int d = RUN * (ql + LANES * u) + e;
                if (d < hd) orow[d] = o[i][RUN * u + e] * inv;
            }
    }
}

template <int HD, int BQ>
void launch(const float* q, const float* k_cache, const float* v_cache, const int32_t* block_table, int table_width,
            const int32_t* cu_q, const int32_t* kv_len, float* out, int T, int R, int nh, int nkv, int hd, int page_size,
            int total_pages, int window, Score scale, int skip_single, cudaStream_t stream) {
    auto kern = attention_f32_kernel<HD, BQ>;
    constexpr size_t smem = f32_smem<HD, BQ>();
    cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<dim3(T / BQ + R, nh), THREADS, smem, stream>>>(q, k_cache, v_cache, block_table, table_width, cu_q, kv_len, out, R,
                                                          nh, nkv, hd, page_size, total_pages, window, scale, skip_single,
                                                          error_flag_ptr());
}

}  // namespace

bool attention_f32_takes(const void* q, const void* k_cache, const void* v_cache, int T, int R, int hd, Score scale) {
    // (a tile is 64 entries wide at least: with heads of 8 or 16 the kernel for any size is faster where most requests bring one
    // token, 8 such requests with 600 keys, heads of 8: 37 us against 56; prompts are not, 1,024 tokens, heads of 16: 207 against 132)
    if (hd <= 16 && T < 2 * R) return false;
    const uintptr_t all = reinterpret_cast<uintptr_t>(q) | reinterpret_cast<uintptr_t>(k_cache) | reinterpret_cast<uintptr_t>(v_cache);
    return hd % (scale.parts == 2 ? 8 : 4) == 0 && hd <= 128 && all % 16 == 0;
}

void attention_f32(const float* q, const float* k_cache, const float* v_cache, const int32_t* block_table, int table_width,
                   const int32_t* cu_q, const int32_t* kv_len, float* out, int T, int R, int nh, int nkv, int hd,
                   int page_size, int total_pages, int window, Score scale, int skip_single, cudaStream_t stream) {
    const bool small = (long long)(T / 32 + R) * nh < 2 * sm_count();
#define DLM_AF32(HD, BQ)                                                                                                \
    launch<HD, BQ>(q, k_cache, v_cache, block_table, table_width, cu_q, kv_len, out, T, R, nh, nkv, hd, page_size,      \
                   total_pages, window, scale, skip_single, stream)
    if (hd <= 64) { if (small) DLM_AF32(64, 16); else DLM_AF32(64, 32); }
    else { if (small) DLM_AF32(128, 16); else DLM_AF32(128, 32); }
#undef DLM_AF32
    check_launch("attention_f32");
}

}  // namespace dlmk
