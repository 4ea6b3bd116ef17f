// Kernels of mixers that run side by side and of the diagonal state-space scan:
//   * selective_scan: S[c, n] <- exp(dt_c A[c, n]) S[c, n] + dt_c x_c B_n, y_c = S[c, :] . C + D_c x_c, with the
//     step size dt_c = softplus(raw + bias) per channel and token, and the gate y silu(z) applied on the way out;
//   * qk_norm_write: RMS norm over the whole query and the whole key projection, a query temperature that grows
//     with the position, and the write of queries, keys and values in the layout of the attention kernels;
//   * rotate_heads: rotary positions applied in place to 32-bit rows (two runs of heads, each with a factor);
//   * branch_norm_add: resid += coef * sum_b rms_norm(branch_b) * w_b for one or two branch outputs;
//   * rmsnorm_pair: two RMS norms of the same rows (one statistic, two weights);
//   * concat_rows: [a | b] in the activation dtype (the input of a product that reads two residuals).
//
// Everything is computed in 32-bit whatever the activation dtype is; only what a kernel hands to a matrix product
// or to the cache is rounded.  A token's result depends on the tokens before it in its own request only, in an
// order that does not depend on how the request was cut into steps.
#include "api.h"
#include "common.cuh"

namespace dlmk {
namespace {

__device__ __forceinline__ float softplus_f(float z) { return z > 30.0f ? z : log1pf(expf(z)); }

__device__ __forceinline__ void copy4_async(float* dst_smem, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void copy16_async(float* dst_smem, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst_smem)), "l"(src)
                 : "memory");
}
template <int N> __device__ __forceinline__ void copies_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ------------------------------------------------------------------ selective scan
// A block owns (a run of channels, a request).  A walking warp holds 32 / PARTS channels; a channel's N <= 8 PARTS states lie in
// PARTS neighbouring lanes, eight a lane in registers, so that a token's B and C come from shared memory as 16-byte loads that
// meet eight states, and step size, input and gate are read once for all of them; what a lane does with a state is a product, an
// exponential and two multiply-adds, two states an instruction where there is such an instruction.  A token depends on the one
// before it only through the state's own multiply-add and nothing is stored to shared memory on the way, so neighbouring
// tokens overlap.  Helper warps bring the tokens' inputs by asynchronous copies, three tiles ahead, and turn a tile's raw
// step sizes into dt = softplus(raw + bias) and its z into silu(z) while the tile before it is walked.  The decay exp(dt A) is
// 2^(dt A log2 e) with A log2 e kept in registers; a channel's sum is added per lane in a fixed order, then by shuffles.
// Bound by the instructions issued per token.  Measured (4,096 channels of 16 states, requests of 1,101, 652 and 203 tokens): 368 us
// with two states a lane, a shared-memory store per token and three phases a tile, 343 us with four helpers that prepared four
// neighbouring channels a lane, about 143 us with eight.  (One request of 2,048 tokens: 439 us then, 197 now.)
constexpr int SCAN_WALKERS = 4, SCAN_HELPERS = 8, SCAN_STAGES = 4;

typedef unsigned long long f2;        // two floats, the lower one first
__device__ __forceinline__ f2 pack2(float lo, float hi) {
    f2 v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(lo), "f"(hi));
    return v;
}
__device__ __forceinline__ float2 unpack2(f2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
// 2^x on the special-function unit for x >= -126 (a result below that would become zero)
__device__ __forceinline__ float ex2_ftz(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// One token of a channel: the lane's eight states move on; returns the sum of s C over the channel's states (in every lane).
// TINY: a decay may lie below the smallest normal number; such tokens are rare, and ask the function that has such numbers.
template <int PARTS, bool TINY>
__device__ __forceinline__ float selective_token(f2 (&s)[4], const f2 (&a2)[4], const f2 (&bb)[4], const f2 (&cc)[4], float dt,
                                                 float xv) {
    const f2 dt2 = pack2(dt, dt), dx2 = pack2(dt * xv, dt * xv);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 w = unpack2(mul2(dt2, a2[i]));
        s[i] = fma2(TINY ? pack2(w.x < -126.f ? exp2f(w.x) : ex2_ftz(w.x), w.y < -126.f ? exp2f(w.y) : ex2_ftz(w.y))
                         : pack2(ex2_ftz(w.x), ex2_ftz(w.y)), s[i], mul2(dx2, bb[i]));
    }
    f2 u = mul2(s[0], cc[0]), v = mul2(s[1], cc[1]);
    u = fma2(s[2], cc[2], u);
    v = fma2(s[3], cc[3], v);
    const float2 uu = unpack2(u), vv = unpack2(v);
    float sum = (uu.x + uu.y) + (vv.x + vv.y);
#pragma unroll
    for (int o = 1; o < PARTS; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    return sum;
}

// A prepared tile of n tokens: rows of rl floats [B | C | dt | x | gate], o the channel's output of the first.
template <int PARTS, bool TINY, typename TOut>
__device__ __forceinline__ void selective_tile(const float* buf, int n, int rl, int cp, int part, int col, bool live, f2 (&s)[4],
                                               const f2 (&a2)[4], float d_c, TOut* o, int ldo) {
    constexpr int NP = 8 * PARTS;
#pragma unroll 4
    for (int tok = 0; tok < n; ++tok) {
        const float* row = buf + (size_t)tok * rl;
        const ulonglong2 b0 = *reinterpret_cast<const ulonglong2*>(row + 8 * part);
        const ulonglong2 b1 = *reinterpret_cast<const ulonglong2*>(row + 8 * part + 4);
        const ulonglong2 e0 = *reinterpret_cast<const ulonglong2*>(row + NP + 8 * part);
        const ulonglong2 e1 = *reinterpret_cast<const ulonglong2*>(row + NP + 8 * part + 4);
        const float dt = row[2 * NP + col], xv = row[2 * NP + cp + col], gate = row[2 * NP + 2 * cp + col];
        const f2 bb[4] = {b0.x, b0.y, b1.x, b1.y}, cc[4] = {e0.x, e0.y, e1.x, e1.y};
        const float sum = selective_token<PARTS, TINY>(s, a2, bb, cc, dt, xv);
        if (live && part == 0) o[(long long)tok * ldo] = from_f32<TOut>(fmaf(d_c, xv, sum) * gate);
    }
}

// (apart from the loop above, whose registers it would share)
template <int PARTS, typename TOut>
__device__ __noinline__ void selective_tile_tiny(const float* buf, int n, int rl, int cp, int part, int col, bool live, f2 (&s)[4],
                                                 const f2 (&a2)[4], float d_c, TOut* o, int ldo) {
    selective_tile<PARTS, true>(buf, n, rl, cp, part, col, live, s, a2, d_c, o, ldo);
}

struct SelectiveArgs {
    const float* x; int ldx;
    const float* dt_raw; int lddt;
    const float* bc; int ldbc;
    const float* z; int ldz;
    const float* dt_bias; const float* A_log; const float* D;
    float* state;
    const int32_t* cu_q; const int32_t* state_slot;
    int ldo, inner, N, wide_bc;          // wide_bc: the eights of a token's B and C start on 16-byte boundaries
};

// The lane's eight states of channel c and their A log2 e (zeros beyond N, and in lanes without a channel); returns the least
// of the latter.
template <int PARTS>
__device__ __forceinline__ float selective_load(const SelectiveArgs& p, const float* st, int c, int part, bool live, f2 (&s)[4],
                                                f2 (&a2)[4]) {
    float least = 0.f;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        float sv[2], av[2];
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int n = 8 * part + 2 * i + e;
            const bool ok = live && n < p.N;
            sv[e] = ok ? st[n] : 0.f;
            av[e] = ok ? -expf(p.A_log[(long long)c * p.N + n]) * 1.4426950408889634f : 0.f;
        }
        s[i] = pack2(sv[0], sv[1]);
        a2[i] = pack2(av[0], av[1]);
        least = fminf(least, fminf(av[0], av[1]));
    }
    return least;
}
__device__ __forceinline__ void selective_store(float* st, int N, int part, bool live, const f2 (&s)[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float2 two = unpack2(s[i]);
        const int n = 8 * part + 2 * i;
        if (live && n < N) st[n] = two.x;
        if (live && n + 1 < N) st[n + 1] = two.y;
    }
}

// Steps whose requests all have few tokens: no ring and no helpers.  Block = (a run of channels, request); every warp walks and
// loads what its channels and their states need of a token.  (64 requests of one token, 4,096 channels of 16 states: 72 us in
// the kernel below, whose blocks have a multiprocessor to themselves, 21 here; four tokens each: 41 and 17 for 32 requests.)
template <int PARTS, typename TOut>
__global__ void __launch_bounds__(32 * SCAN_WALKERS) selective_few_kernel(SelectiveArgs p, TOut* out) {
    dep_wait();          // nothing is read or written before the kernels before this one have ended
    const int r = blockIdx.y, lane = threadIdx.x & 31, part = lane % PARTS;
    const int c = (blockIdx.x * (blockDim.x >> 5) + (int)(threadIdx.x >> 5)) * (32 / PARTS) + lane / PARTS;
    const bool live = c < p.inner;
    const int N = p.N, ch = live ? c : 0;
    const int t0 = p.cu_q[r], t1 = p.cu_q[r + 1], slot = p.state_slot[r];
    const float d_c = p.D[ch], bias = p.dt_bias[ch];
    if (t0 >= t1) return;
    float* st = p.state + ((long long)slot * p.inner + ch) * N;
    f2 s[4], a2[4];
    selective_load<PARTS>(p, st, c, part, live, s, a2);
    for (long long t = t0; t < t1; ++t) {
        const float* row = p.bc + t * p.ldbc;
        f2 bb[4], cc[4];
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            f2 (&dst)[4] = h == 0 ? bb : cc;
            const float* src = row + h * N + 8 * part;
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                float v[4];
                if (p.wide_bc) {
                    const float4 w = 8 * part + 4 * g < N ? *reinterpret_cast<const float4*>(src + 4 * g)
                                                          : make_float4(0.f, 0.f, 0.f, 0.f);
                    v[0] = w.x; v[1] = w.y; v[2] = w.z; v[3] = w.w;
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e) v[e] = 8 * part + 4 * g + e < N ? src[4 * g + e] : 0.f;
                }
                dst[2 * g] = pack2(v[0], v[1]);
                dst[2 * g + 1] = pack2(v[2], v[3]);
            }
        }
        const float dt = softplus_f(p.dt_raw[t * p.lddt + ch] + bias), xv = p.x[t * p.ldx + ch], gate = silu_f(p.z[t * p.ldz + ch]);
        const float sum = selective_token<PARTS, true>(s, a2, bb, cc, dt, xv);
        if (live && part == 0) out[t * p.ldo + c] = from_f32<TOut>(fmaf(d_c, xv, sum) * gate);
    }
    selective_store(st, N, part, live, s);
}

template <int PARTS, typename TOut>
__global__ void __launch_bounds__(32 * (SCAN_WALKERS + SCAN_HELPERS), 1)
selective_scan_kernel(SelectiveArgs p, TOut* out, int walkers, int tile_tokens, int wide) {
    const float* x = p.x; const float* dt_raw = p.dt_raw; const float* bc = p.bc; const float* z = p.z;
    const int ldx = p.ldx, lddt = p.lddt, ldbc = p.ldbc, ldz = p.ldz, inner = p.inner, N = p.N;
    dep_wait();          // nothing is read or written before the kernels before this one have ended
    constexpr int NP = 8 * PARTS, CW = 32 / PARTS;        // states as stored; channels of a warp
    extern __shared__ __align__(16) float sm[];           // [STAGES][tile][B: NP | C: NP | dt | x | gate: cp each]
    __shared__ float s_least[SCAN_WALKERS * 32];          // a channel's most negative A log2 e
    __shared__ int s_tiny[SCAN_STAGES];                   // a decay of the tile may lie below the smallest normal number
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int chans = walkers * CW, cp = (chans + 3) & ~3, rl = 2 * NP + 3 * cp;
    const int c0 = blockIdx.x * chans, nch = min(chans, inner - c0);
    const int r = blockIdx.y;
    const int t0 = p.cu_q[r], t1 = p.cu_q[r + 1];
    const int n_tiles = (t1 - t0 + tile_tokens - 1) / tile_tokens;

    if (threadIdx.x < SCAN_STAGES) s_tiny[threadIdx.x] = 0;

    if (warp >= walkers) {
        const int helper = warp - walkers;
        // a warp a token; `wide`: every run of a token's inputs starts on a 16-byte boundary and is a multiple of four floats
        auto fetch = [&](int k) {         // (a tile beyond the last: an empty group, so that the count of groups holds)
            float* buf = sm + (size_t)(k % SCAN_STAGES) * tile_tokens * rl;
            const int first = t0 + k * tile_tokens, n = min(tile_tokens, t1 - first);
            for (int tok = helper; tok < n; tok += SCAN_HELPERS) {
                const long long t = first + tok;
                const float* src_bc = bc + t * ldbc;
                const float* src[3] = {dt_raw + t * lddt + c0, x + t * ldx + c0, z + t * ldz + c0};
                float* dst = buf + (size_t)tok * rl;
                if (wide) {
                    for (int i = 4 * lane; i < NP; i += 128) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (i < N) copy16_async(dst + h * NP + i, src_bc + h * N + i);
                            else *reinterpret_cast<float4*>(dst + h * NP + i) = make_float4(0.f, 0.f, 0.f, 0.f);
                        }
                    }
                    for (int i = 4 * lane; i < nch; i += 128)
#pragma unroll
                        for (int v = 0; v < 3; ++v) copy16_async(dst + 2 * NP + v * cp + i, src[v] + i);
                } else {
                    for (int i = lane; i < NP; i += 32) {
#pragma unroll
                        for (int h = 0; h < 2; ++h) {
                            if (i < N) copy4_async(dst + h * NP + i, src_bc + h * N + i);
                            else dst[h * NP + i] = 0.f;
                        }
                    }
                    for (int i = lane; i < nch; i += 32)
#pragma unroll
                        for (int v = 0; v < 3; ++v) copy4_async(dst + 2 * NP + v * cp + i, src[v] + i);
                }
            }
            copies_commit();
        };
        // (a warp touches only what it copied itself)
        auto prepare = [&](int k) {
            float* buf = sm + (size_t)(k % SCAN_STAGES) * tile_tokens * rl;
            const int n = min(tile_tokens, t1 - (t0 + k * tile_tokens));
            __syncwarp();                 // every lane has waited for its own copies
            bool tiny = false;
            for (int tok = helper; tok < n; tok += SCAN_HELPERS) {
                float* dt = buf + (size_t)tok * rl + 2 * NP;
                float* gate = dt + 2 * cp;
                for (int i = lane; i < nch; i += 32) {
                    const float step = softplus_f(dt[i] + p.dt_bias[c0 + i]);
                    dt[i] = step;
                    tiny = tiny || step * s_least[i] < -126.f;
                    gate[i] = silu_f(gate[i]);
                }
            }
            if (tiny) s_tiny[k % SCAN_STAGES] = 1;
        };
        for (int k = 0; k < SCAN_STAGES - 1; ++k) fetch(k);
        copies_wait<SCAN_STAGES - 2>();
        __syncthreads();                  // the channels' decays are known
        if (n_tiles > 0) prepare(0);
        __syncthreads();
        for (int k = 0; k < n_tiles; ++k) {              // the walkers are at tile k
            fetch(k + SCAN_STAGES - 1);                  // into the buffer of tile k - 1, which everyone has left
            copies_wait<SCAN_STAGES - 2>();
            if (k + 1 < n_tiles) prepare(k + 1);
            __syncthreads();
        }
        copies_wait<0>();
        return;
    }

    const int part = lane % PARTS, col = warp * CW + lane / PARTS, c = c0 + col;
    const bool live = c < inner;
    float* st = p.state + ((long long)p.state_slot[r] * inner + (live ? c : 0)) * N;
    f2 s[4], a2[4];
    float least = selective_load<PARTS>(p, st, c, part, live, s, a2);
#pragma unroll
    for (int o = 1; o < PARTS; o <<= 1) least = fminf(least, __shfl_xor_sync(0xffffffffu, least, o));
    if (part == 0) s_least[col] = least;
    const float d_c = live ? p.D[c] : 0.f;
    __syncthreads();
    __syncthreads();                      // tile 0 is prepared
    for (int k = 0; k < n_tiles; ++k) {
        const float* buf = sm + (size_t)(k % SCAN_STAGES) * tile_tokens * rl;
        const int first = t0 + k * tile_tokens, n = min(tile_tokens, t1 - first);
        TOut* o = out + (long long)first * p.ldo + c;
        if (s_tiny[k % SCAN_STAGES] != 0) {
            f2 kept[4] = {s[0], s[1], s[2], s[3]};
            selective_tile_tiny<PARTS, TOut>(buf, n, rl, cp, part, col, live, kept, a2, d_c, o, p.ldo);
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i] = kept[i];
        } else {
            selective_tile<PARTS, false>(buf, n, rl, cp, part, col, live, s, a2, d_c, o, p.ldo);
        }
        __syncthreads();
        // (nobody reads this tile's any more; it is set again for tile k + 4, after two more barriers)
        if (threadIdx.x == 0) s_tiny[k % SCAN_STAGES] = 0;
    }
    selective_store(st, N, part, live, s);
}

// ------------------------------------------------- whole-projection norms, temperature, cache write
// One block a token.  qkv f32 row: [q: nh * d | k: nkv * d | v: nkv * dv].  q and k are each divided by the root
// mean square of the WHOLE projection (all heads at once) and multiplied by a weight per entry; q also by the
// temperature 1 + coef * ln(floor((p + 1) / every) + 1) of its position p (every == 0: none).  Heads are written
// D wide (D >= d, dv; entries beyond a head's own size are zero) so that keys and values share one head size.
template <typename T>
__global__ void qk_norm_write_kernel(const float* qkv, int ld, const int32_t* __restrict__ positions,
                                     const float* __restrict__ qn_w, const float* __restrict__ kn_w, float eps,
                                     float temp_coef, int temp_every, const int32_t* __restrict__ slots, T* q_out,
                                     T* k_cache, T* v_cache, int nh, int nkv, int d, int dv, int D, int page_size,
                                     int total_pages, int* err) {
    __shared__ float s_part[32];
    dep_wait();
    dep_launch_next();
    const int t = blockIdx.x;
    const int Q = nh * d, K = nkv * d, V = nkv * dv;
    const float* row = qkv + (long long)t * ld;
    int in_page = 0, page = -1;
    if (slots != nullptr) {
        const int s = slots[t];
        if (s >= 0) {
            page = s / page_size;
            in_page = s % page_size;
            if (page >= total_pages) {
                if (threadIdx.x == 0) *err = 2;
                page = -1;
            }
        }
    }
    float pq = 0.f, pk = 0.f;
    for (int i = threadIdx.x; i < Q; i += blockDim.x) pq = fmaf(row[i], row[i], pq);
    for (int i = threadIdx.x; i < K; i += blockDim.x) pk = fmaf(row[Q + i], row[Q + i], pk);
    const float sq = block_sum(pq, s_part);
    const float sk = block_sum(pk, s_part);
    float fq = qn_w != nullptr ? 1.0f / sqrtf(sq / (float)Q + eps) : 1.0f;
    const float fk = kn_w != nullptr ? 1.0f / sqrtf(sk / (float)K + eps) : 1.0f;
    float temp = 1.0f;
    if (temp_every > 0) temp = 1.0f + temp_coef * logf((float)((positions[t] + 1) / temp_every) + 1.0f);
    for (int idx = threadIdx.x; idx < nh * D; idx += blockDim.x) {
        const int h = idx / D, i = idx - h * D;
        float v = 0.f;
        if (i < d) {
            const int e = h * d + i;
            v = (row[e] * fq) * (qn_w != nullptr ? qn_w[e] : 1.0f) * temp;
        }
        q_out[(long long)t * nh * D + idx] = from_f32<T>(v);
    }
    if (page >= 0) {
        for (int idx = threadIdx.x; idx < nkv * D; idx += blockDim.x) {
            const int h = idx / D, i = idx - h * D;
            float kv = 0.f, vv = 0.f;
            if (i < d) {
                const int e = h * d + i;
                kv = (row[Q + e] * fk) * (kn_w != nullptr ? kn_w[e] : 1.0f);
            }
            if (i < dv) vv = row[Q + K + h * dv + i];
            const long long o = (((long long)page * nkv + h) * page_size + in_page) * D + i;
            k_cache[o] = from_f32<T>(kv);
            v_cache[o] = from_f32<T>(vv);
        }
    }
    (void)V;
}

// ------------------------------------------------------------------ rotation in place
// One block a token.  x f32 rows; two runs of `heads` heads of `dim` entries start at columns off_a and off_b.
// In every head the first rot_dims entries are rotated (entry i with entry i + rot_dims / 2, angle
// position * inv_freq[i]); then the whole head is multiplied by the run's factor.
__global__ void rotate_heads_kernel(float* x, int ld, const int32_t* __restrict__ positions,
                                    const float* __restrict__ inv_freq, int rot_dims, int heads, int dim, int off_a,
                                    float scale_a, int off_b, float scale_b) {
    extern __shared__ float sc[];                  // [2][rot_dims / 2]: sines, cosines
    const int t = blockIdx.x;
    const int half = rot_dims / 2;
    const float pos = (float)positions[t];         // (positions and frequencies are the step's inputs)
    for (int i = threadIdx.x; i < half; i += blockDim.x) {
        float sn, cs;
        sincosf(pos * inv_freq[i], &sn, &cs);
        sc[i] = sn;
        sc[half + i] = cs;
    }
    dep_wait();
    dep_launch_next();
    __syncthreads();
    float* row = x + (long long)t * ld;
    const int per = heads * dim;
    for (int idx = threadIdx.x; idx < 2 * per; idx += blockDim.x) {
        const int run = idx / per, e = idx - run * per;
        const int h = e / dim, i = e - h * dim;
        float* head = row + (run ? off_b : off_a) + h * dim;
        const float f = run ? scale_b : scale_a;
        if (i < half) {
            const float u = head[i], v = head[i + half];
            const float sn = sc[i], cs = sc[half + i];
            head[i] = (u * cs - v * sn) * f;
            head[i + half] = (v * cs + u * sn) * f;
        } else if (i >= 2 * half && f != 1.0f) {
            head[i] *= f;
        }
    }
}

// --------------------------------------------------------- sum of normed branch outputs
// One block a token: resid[t] += coef * (a / rms(a) * wa + b / rms(b) * wb)   (b == nullptr: one branch).
__global__ void branch_norm_add_kernel(float* resid, const float* a, const float* __restrict__ wa, const float* b,
                                       const float* __restrict__ wb, float eps, float coef, int H) {
    __shared__ float s_part[32];
    dep_wait();
    dep_launch_next();
    const long long t = blockIdx.x;
    const float* ar = a + t * H;
    const float* br = b != nullptr ? b + t * H : nullptr;
    float pa = 0.f, pb = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        pa = fmaf(ar[i], ar[i], pa);
        if (br != nullptr) pb = fmaf(br[i], br[i], pb);
    }
    const float sa = block_sum(pa, s_part);
    const float sb = block_sum(pb, s_part);
    const float fa = 1.0f / sqrtf(sa / (float)H + eps), fb = 1.0f / sqrtf(sb / (float)H + eps);
    float* o = resid + t * H;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        float v = (ar[i] * fa) * wa[i];
        if (br != nullptr) v += (br[i] * fb) * wb[i];
        o[i] += coef * v;
    }
}

// ------------------------------------------------------------ two norms of the same rows
// One block a row: out_a = x / rms(x) * wa, out_b = x / rms(x) * wb (one statistic, two weights).
template <typename T>
__global__ void rmsnorm_pair_kernel(const float* x, const float* __restrict__ wa, const float* __restrict__ wb, T* out_a,
                                    T* out_b, int H, float eps) {
    __shared__ float s_part[32];
    dep_wait();
    dep_launch_next();
    const long long t = blockIdx.x;
    const float* row = x + t * H;
    float part = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) part = fmaf(row[i], row[i], part);
    const float inv = 1.0f / sqrtf(block_sum(part, s_part) / (float)H + eps);
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = row[i] * inv;
        out_a[t * H + i] = from_f32<T>(v * wa[i]);
        out_b[t * H + i] = from_f32<T>(v * wb[i]);
    }
}

// ------------------------------------------------------------------ two rows side by side
template <typename T>
__global__ void concat_rows_kernel(const float* a, const float* b, T* out, int H) {
    dep_wait();
    dep_launch_next();
    const long long t = blockIdx.x;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        out[t * 2 * H + i] = from_f32<T>(a[t * H + i]);
        out[t * 2 * H + H + i] = from_f32<T>(b[t * H + i]);
    }
}

}  // namespace

void selective_scan(const float* x, int ldx, const float* dt_raw, int lddt, const float* bc, int ldbc, const float* z,
                    int ldz, const float* dt_bias, const float* A_log, const float* D, float* state,
                    const int32_t* cu_q, const int32_t* state_slot, void* out, int ldo, int R, int inner, int N,
                    int out_dtype, int longest, cudaStream_t stream) {
    if (R <= 0 || inner <= 0) return;
    DLM_CHECK(N >= 1 && N <= 256, "selective_scan: state size 1..256");
    int parts = 1;
    while (8 * parts < N) parts *= 2;
    const int cw = 32 / parts;
    // four walkers a block, fewer where there would be a block for less than every other multiprocessor
    int walkers = SCAN_WALKERS;
    while (walkers > 1 && (long long)((inner + walkers * cw - 1) / (walkers * cw)) * R < sm_count() / 2) walkers /= 2;
    const int chans = walkers * cw;
    const dim3 grid((inner + chans - 1) / chans, R);
    const size_t row = (16 * parts + 3 * ((chans + 3) & ~3)) * sizeof(float);
    int tile = 16;
    while (tile > 1 && SCAN_STAGES * tile * row > 100 * 1024) tile /= 2;
    const size_t smem = SCAN_STAGES * tile * row;
    const int wide = (((reinterpret_cast<uintptr_t>(x) | reinterpret_cast<uintptr_t>(dt_raw) | reinterpret_cast<uintptr_t>(bc) |
                        reinterpret_cast<uintptr_t>(z)) & 15) == 0 && ldx % 4 == 0 && lddt % 4 == 0 && ldbc % 4 == 0 &&
                      ldz % 4 == 0 && N % 4 == 0 && chans % 4 == 0 && inner % 4 == 0) ? 1 : 0;
    const int wide_bc = (reinterpret_cast<uintptr_t>(bc) & 15) == 0 && ldbc % 4 == 0 && N % 4 == 0 ? 1 : 0;
    const SelectiveArgs args{x, ldx, dt_raw, lddt, bc, ldbc, z, ldz, dt_bias, A_log, D, state, cu_q, state_slot, ldo, inner, N, wide_bc};
    // One token a request, or up to four where the ring's kernel would need more than one wave of blocks
    const bool few = longest == 1 || (longest >= 1 && longest <= 4 && (long long)grid.x * grid.y > sm_count());
#define DLM_SEL(PARTS, TOUT)                                                                                         \
    do {                                                                                                             \
        if (few) {                                                                                                   \
            selective_few_kernel<PARTS, TOUT><<<grid, 32 * walkers, 0, stream>>>(args, static_cast<TOUT*>(out));     \
            break;                                                                                                   \
        }                                                                                                            \
        auto kern = selective_scan_kernel<PARTS, TOUT>;                                                              \
        if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);    \
        kern<<<grid, 32 * (walkers + SCAN_HELPERS), smem, stream>>>(args, static_cast<TOUT*>(out), walkers, tile,    \
                                                                    wide);                                           \
    } while (0)
#define DLM_SEL_T(PARTS)                                                                   \
    do {                                                                                   \
        if (out_dtype == F32) DLM_SEL(PARTS, float); else DLM_SEL(PARTS, __nv_bfloat16);   \
    } while (0)
    switch (parts) {
        case 1: DLM_SEL_T(1); break;
        case 2: DLM_SEL_T(2); break;
        case 4: DLM_SEL_T(4); break;
        case 8: DLM_SEL_T(8); break;
        case 16: DLM_SEL_T(16); break;
        default: DLM_SEL_T(32); break;
    }
#undef DLM_SEL_T
#undef DLM_SEL
    check_launch("selective_scan");
}

void qk_norm_write(const float* qkv, int ld, const int32_t* positions, const float* qn_w, const float* kn_w, float eps,
                   float temp_coef, int temp_every, const int32_t* slots, void* q_out, void* k_cache, void* v_cache,
                   int T, int nh, int nkv, int d, int dv, int D, int page_size, int total_pages, int dtype,
                   cudaStream_t stream) {
    if (T <= 0) return;
    DLM_CHECK(D >= d && D >= dv && d >= 1 && dv >= 1, "qk_norm_write: the stored head size must hold keys and values");
    DLM_CHECK(temp_every >= 0, "qk_norm_write: the temperature's period must not be negative");
    int* err = error_flag_ptr();
    if (dtype == F32)
        launch_dep(qk_norm_write_kernel<float>, dim3(T), dim3(256), 0, stream, qkv, ld, positions, qn_w, kn_w, eps,
                   temp_coef, temp_every, slots, static_cast<float*>(q_out), static_cast<float*>(k_cache),
                   static_cast<float*>(v_cache), nh, nkv, d, dv, D, page_size, total_pages, err);
    else
        launch_dep(qk_norm_write_kernel<__nv_bfloat16>, dim3(T), dim3(256), 0, stream, qkv, ld, positions, qn_w, kn_w,
                   eps, temp_coef, temp_every, slots, static_cast<__nv_bfloat16*>(q_out),
                   static_cast<__nv_bfloat16*>(k_cache), static_cast<__nv_bfloat16*>(v_cache), nh, nkv, d, dv, D,
                   page_size, total_pages, err);
    check_launch("qk_norm_write");
}

void rotate_heads(float* x, int ld, const int32_t* positions, const float* inv_freq, int rot_dims, int T, int heads,
                  int dim, int off_a, float scale_a, int off_b, float scale_b, cudaStream_t stream) {
    if (T <= 0) return;
    DLM_CHECK(rot_dims >= 0 && rot_dims % 2 == 0 && rot_dims <= dim, "rotate_heads: rot_dims must be even, at most dim");
    DLM_CHECK(rot_dims == 0 || inv_freq != nullptr, "rotate_heads: a rotation needs its frequencies");
    const int threads = 2 * heads * dim >= 1024 ? 256 : 128;
    launch_dep(rotate_heads_kernel, dim3(T), dim3(threads), sizeof(float) * (rot_dims > 0 ? rot_dims : 1), stream, x, ld,
               positions, inv_freq, rot_dims, heads, dim, off_a, scale_a, off_b, scale_b);
    check_launch("rotate_heads");
}

void branch_norm_add(float* resid, const float* a, const float* wa, const float* b, const float* wb, float eps,
                     float coef, int T, int H, cudaStream_t stream) {
    if (T <= 0) return;
    DLM_CHECK(a != nullptr && wa != nullptr && (b == nullptr || wb != nullptr), "branch_norm_add: a branch needs its weight");
    launch_dep(branch_norm_add_kernel, dim3(T), dim3(H >= 1024 ? 256 : 128), 0, stream, resid, a, wa, b, wb, eps, coef, H);
    check_launch("branch_norm_add");
}

void rmsnorm_pair(const float* x, const float* wa, const float* wb, void* out_a, void* out_b, int T, int H, float eps,
                  int out_dtype, cudaStream_t stream) {
    if (T <= 0) return;
    const int threads = H >= 1024 ? 256 : 128;
    if (out_dtype == F32)
        launch_dep(rmsnorm_pair_kernel<float>, dim3(T), dim3(threads), 0, stream, x, wa, wb, static_cast<float*>(out_a),
                   static_cast<float*>(out_b), H, eps);
    else
        launch_dep(rmsnorm_pair_kernel<__nv_bfloat16>, dim3(T), dim3(threads), 0, stream, x, wa, wb,
                   static_cast<__nv_bfloat16*>(out_a), static_cast<__nv_bfloat16*>(out_b), H, eps);
    check_launch("rmsnorm_pair");
}

void concat_rows(const float* a, const float* b, void* out, int T, int H, int out_dtype, cudaStream_t stream) {
    if (T <= 0) return;
    if (out_dtype == F32)
        launch_dep(concat_rows_kernel<float>, dim3(T), dim3(256), 0, stream, a, b, static_cast<float*>(out), H);
    else
        launch_dep(concat_rows_kernel<__nv_bfloat16>, dim3(T), dim3(256), 0, stream, a, b,
                   static_cast<__nv_bfloat16*>(out), H);
    check_launch("concat_rows");
}

}  // namespace dlmk
