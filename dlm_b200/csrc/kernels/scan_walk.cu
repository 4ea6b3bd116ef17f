// The walk of the linear recurrences: a state S [N rows, P columns] per head and request in 32-bit, one token after the
// other, for four ways the state moves on.
//
//   WALK_HEAD      S <- a S + k v^T with one decay a per head and token (state-space scan, retention);  o = S^T q + D v
//   WALK_CHANNEL   S <- diag(a) S + k v^T (gated linear attention);                                     o = S^T q
//   WALK_DELTA     S <- a S;  u = beta (v - S^T k);  S <- S + k u^T (gated delta rule);                 o = S^T q
//   WALK_REMOVE    S <- diag(a) S - (r u)(u^T S) + k v^T, u the unit key, r a rate per channel;         o = S^T q
//
// What bounds it is the chain of a token's steps (a request's tokens cannot overlap where a token reads the state the one
// before it left) and the instructions a warp issues per token, not memory.  So a lane keeps a tile of 8 rows x CPL columns of S
// in registers: a token's q, k and decays come from shared memory once for CPL columns (16-byte loads), the multiply-adds run
// two rows an instruction, and the sums over a column's rows, which lie in RL = N / 8 neighbouring lanes, meet in shuffles
// in a fixed order (it depends on N alone, so a result does not depend on how a request was cut into steps).  With the
// delta rules both read-outs are taken before the update, S'^T q = (a S)^T q + u (k . q), so that one set of shuffles is on the
// chain.  Beside the warps that walk, helper warps bring the tokens' inputs by asynchronous copies, three tiles ahead, and turn
// a tile's raw values into decays, rates and unit vectors while the tile before it is walked: done by the walking warps
// themselves that took two to four times as long as the walk.
//
// Measured, one request of 2,048 tokens, before (a lane one column, 4-16 rows, everything done by all warps) and now: state space, 64
// heads of 128 x 64: 824 -> 286 us; retention, 16 heads of 64 x 128: 534 -> 158; gated linear attention, 16 heads of 64 x 128:
// 577 -> 198; gated delta rule, 16 heads of 128 x 128: 754 -> 352; removal form, 32 heads of 64 x 64: 1,225 -> 319.
#include "api.h"
#include "common.cuh"
#include "scan_walk.h"

namespace dlmk {
namespace {

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
__device__ __forceinline__ float sum2(f2 v) {
    const float2 r = unpack2(v);
    return r.x + r.y;
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

__device__ __forceinline__ void copy4(float* dst, const float* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copy16(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
// neighbouring columns of a row (the address is a multiple of their size)
__device__ __forceinline__ void load_columns(const float* p, float (&v)[2]) {
    const float2 x = *reinterpret_cast<const float2*>(p);
    v[0] = x.x; v[1] = x.y;
}
__device__ __forceinline__ void load_columns(const float* p, float (&v)[4]) {
    const float4 x = *reinterpret_cast<const float4*>(p);
    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
}

__device__ __forceinline__ float sigmoid_w(float z) { return 1.0f / (1.0f + expf(-z)); }
__device__ __forceinline__ float softplus_w(float z) { return z > 20.0f ? z : log1pf(expf(z)); }

// four walking warps and eight helpers: with room for 20 warps a thread gets 96 registers instead of 168 and the walk of a
// state-space prompt (below) takes 500 us instead of 289
constexpr int STAGES = 4, MOST_WALKERS = 4, HELPERS = 8, MOST_WARPS = MOST_WALKERS + HELPERS;

template <int MODE> constexpr int walk_vectors() { return MODE == WALK_REMOVE ? 4 : (MODE == WALK_CHANNEL ? 3 : 2); }

// Row i = 0 .. 7 of a lane: two runs of four, so that a token's vectors come as 16-byte loads.
template <int RL> __device__ __forceinline__ int row_of(int rlane, int i) { return 4 * rlane + (i & 3) + 4 * RL * (i >> 2); }

// The lane's tile of a state [N, P]: rows (2 i, 2 i + 1) of CPL columns from c0 on.  `vec`: a row's columns come as one access.
template <int RL, int CPL>
__device__ __forceinline__ void load_state(const float* st, int N, int P, int rlane, int c0, bool vec, f2 (&s)[4][CPL]) {
    float raw[8][CPL];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int n = row_of<RL>(rlane, i);
        const float* src = st + (long long)n * P + c0;
#pragma unroll
        for (int c = 0; c < CPL; ++c) raw[i][c] = 0.f;
        if (n < N) {
            if (vec && c0 < P) {
                load_columns(src, raw[i]);
            } else {
#pragma unroll
                for (int c = 0; c < CPL; ++c)
                    if (c0 + c < P) raw[i][c] = src[c];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int c = 0; c < CPL; ++c) s[i][c] = pack2(raw[2 * i][c], raw[2 * i + 1][c]);
}

template <int RL, int CPL>
__device__ __forceinline__ void store_state(float* st, int N, int P, int rlane, int c0, bool vec, const f2 (&s)[4][CPL]) {
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int n = row_of<RL>(rlane, i);
        if (n >= N || c0 >= P) continue;
        float raw[CPL];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            const float2 two = unpack2(s[i >> 1][c]);
            raw[c] = i & 1 ? two.y : two.x;
        }
        float* dst = st + (long long)n * P + c0;
        if (vec) {
            if (CPL == 4) *reinterpret_cast<float4*>(dst) = make_float4(raw[0], raw[1 % CPL], raw[2 % CPL], raw[3 % CPL]);
            else *reinterpret_cast<float2*>(dst) = make_float2(raw[0], raw[1 % CPL]);
        } else {
#pragma unroll
            for (int c = 0; c < CPL; ++c)
                if (c0 + c < P) dst[c] = raw[c];
        }
    }
}

// One token: the lane's tile of the state moves on and the token's output goes to o (the lane's first column there, of which
// cols_left exist).  sc: the decay and what joins the columns' sums, as prepared.  Fused multiply-adds are spelled out, so that
// the two kernels that call this give the same bits.
template <int MODE, int RL, int CPL>
__device__ __forceinline__ void walk_token(f2 (&s)[4][CPL], const f2 (&q)[4], const f2 (&k)[4], const f2 (&a)[4],
                                           const f2 (&rr)[4], const float4& sc, const float (&v)[CPL], float dcoef, int rlane,
                                           int cols_left, float* o) {
    constexpr bool DELTA = MODE == WALK_DELTA || MODE == WALK_REMOVE;
    // what joins a column's sum: D v, or the update's share of a read-out taken before the update (u (k . q), or all of `with`)
    float out[CPL], with[CPL];
    auto joined = [&](float y, float x) {
        return MODE == WALK_HEAD ? fmaf(dcoef, x, y) : (MODE == WALK_DELTA ? fmaf(x, sc.z, y) : (MODE == WALK_REMOVE ? y + x : y));
    };
    if (!DELTA) {
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            const float x = MODE == WALK_HEAD ? sc.y * v[c] : v[c];
            const f2 xx = pack2(x, x);
#pragma unroll
            for (int i = 0; i < 4; ++i) s[i][c] = fma2(a[i], s[i][c], mul2(k[i], xx));
            f2 acc0 = mul2(s[0][c], q[0]), acc1 = mul2(s[1][c], q[1]);
            acc0 = fma2(s[2][c], q[2], acc0);
            acc1 = fma2(s[3][c], q[3], acc1);
            out[c] = sum2(acc0) + sum2(acc1);
            with[c] = v[c];
        }
    } else {
        float ks[CPL];
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            if (MODE == WALK_DELTA) {
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i][c] = mul2(s[i][c], a[i]);
            }
            f2 k0 = mul2(k[0], s[0][c]), k1 = mul2(k[1], s[1][c]);
            k0 = fma2(k[2], s[2][c], k0);
            k1 = fma2(k[3], s[3][c], k1);
            ks[c] = sum2(k0) + sum2(k1);
        }
#pragma unroll
        for (int o2 = 1; o2 < RL; o2 <<= 1)
#pragma unroll
            for (int c = 0; c < CPL; ++c) ks[c] += __shfl_xor_sync(0xffffffffu, ks[c], o2);
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            f2 q0 = mul2(q[0], s[0][c]), q1 = mul2(q[1], s[1][c]);
            q0 = fma2(q[2], s[2][c], q0);
            q1 = fma2(q[3], s[3][c], q1);
            out[c] = sum2(q0) + sum2(q1);
            if (MODE == WALK_DELTA) {
                const float u = sc.y * (v[c] - ks[c]);
                const f2 uu = pack2(u, u);
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i][c] = fma2(k[i], uu, s[i][c]);
                with[c] = u;
            } else {
                // (what is removed first, then k v^T: the other way round rounds the larger sum)
                const float us = ks[c] * sc.x;
                const f2 uu = pack2(us, us), vv = pack2(v[c], v[c]);
#pragma unroll
                for (int i = 0; i < 4; ++i) s[i][c] = fma2(k[i], vv, fma2(rr[i], uu, mul2(a[i], s[i][c])));
                with[c] = fmaf(v[c], sc.z, -(sc.y * us));
            }
        }
    }
    if (RL >= CPL) {
        // each stage of the sums over a column's row lanes hands half of the columns over, so that CPL columns cost little
        // more than one; lane `rlane` < CPL ends with column own_c
        float y;
        int own_c;
        if (CPL == 4) {
            const bool up = rlane & 1, up2 = rlane & 2;
            float k0 = up ? out[2 % CPL] : out[0], k1 = up ? out[3 % CPL] : out[1 % CPL];
            k0 += __shfl_xor_sync(0xffffffffu, up ? out[0] : out[2 % CPL], 1);
            k1 += __shfl_xor_sync(0xffffffffu, up ? out[1 % CPL] : out[3 % CPL], 1);
            y = (up2 ? k1 : k0) + __shfl_xor_sync(0xffffffffu, up2 ? k0 : k1, 2);
            own_c = (rlane & 1) << 1 | ((rlane >> 1) & 1);
        } else {
            const bool up = rlane & 1;
            y = (up ? out[1 % CPL] : out[0]) + __shfl_xor_sync(0xffffffffu, up ? out[0] : out[1 % CPL], 1);
            own_c = rlane & 1;
        }
#pragma unroll
        for (int o2 = CPL; o2 < RL; o2 <<= 1) y += __shfl_xor_sync(0xffffffffu, y, o2);
        y = joined(y, CPL == 4 ? (own_c & 2 ? (own_c & 1 ? with[3 % CPL] : with[2 % CPL]) : (own_c & 1 ? with[1 % CPL] : with[0]))
                               : (own_c ? with[1 % CPL] : with[0]));
        if (rlane < CPL && own_c < cols_left) o[own_c] = y;
    } else {
#pragma unroll
        for (int c = 0; c < CPL; ++c) {
            float y = out[c];
#pragma unroll
            for (int x = 1; x < RL; x <<= 1) y += __shfl_xor_sync(0xffffffffu, y, x);
            if (rlane == 0 && c < cols_left) o[c] = joined(y, with[c]);
        }
    }
}

// x[i] <- f(x[i], row of i) for the lane's eight rows.  The 32 / RL column lanes of a row group hold the same x, so each works out
// a share and hands it round.
template <int RL, typename F>
__device__ __forceinline__ void each_row(float (&x)[8], int lane, F f) {
    constexpr int G = 32 / RL < 8 ? 32 / RL : 8, E = 8 / G;
    const int rlane = lane & (RL - 1), g = (lane / RL) % G;
    float y[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
        float v = x[e];
#pragma unroll
        for (int j = 1; j < G; ++j) v = g == j ? x[j * E + e] : v;
        y[e] = f(v, row_of<RL>(rlane, g * E + e));
    }
#pragma unroll
    for (int i = 0; i < 8; ++i) x[i] = G == 1 ? y[i % E] : __shfl_sync(0xffffffffu, y[i % E], rlane + RL * (i / E));
}

// Steps whose requests all have few tokens: no ring and no helpers.  Block = (head, request, a run of columns); every warp walks,
// loads a token's raw values for its lanes' rows and columns and prepares them in registers, in the order of operations (and of
// the sums over N) of the helpers of the kernel below.  What bounds such a step is the latency of one block where there are
// few and the states' traffic where there are many: the kernel below has one block a multiprocessor and its ring to fill first.
// Measured, 64 requests of one token, in the kernel below and here: state space, 64 heads of 128 x 64: 159 and 91 us; retention,
// 16 heads of 64 x 128: 34 and 21; gated delta rule, 16 heads of 128 x 128: 87 and 48; removal form, 32 heads of 64 x 64: 54 and 26.
template <int MODE, int RL, int CPL>
__global__ void __launch_bounds__(32 * MOST_WALKERS, 3) scan_few_kernel(WalkParams p) {
    dep_wait();           // nothing is read or written before the kernels before this one have ended
    constexpr bool CHANNEL = MODE == WALK_CHANNEL || MODE == WALK_REMOVE;
    const int h = blockIdx.x, r = blockIdx.y, lane = threadIdx.x & 31, rlane = lane & (RL - 1);
    const int first = (blockIdx.z * p.walkers + (int)(threadIdx.x >> 5)) * (32 / RL * CPL), c0 = first + (lane / RL) * CPL;
    const int N = p.N, P = p.P, hq = h / p.q_div;
    if (first >= P) return;
    // (what does not depend on another load is asked for before anything is waited for)
    const bool fixed = MODE == WALK_HEAD && p.fixed_decay != nullptr, per_head = (MODE == WALK_HEAD && !fixed) || MODE == WALK_DELTA;
    const int t0 = p.cu_q[r], t1 = p.cu_q[r + 1], slot = p.state_slot[r];
    const float A_log = per_head ? p.A_log[h] : 0.f, fixed_a = fixed ? p.fixed_decay[h] : 0.f;
    const float bias = per_head && p.dec_bias != nullptr ? p.dec_bias[h] : 0.f;
    const float dcoef = MODE == WALK_HEAD && p.D != nullptr ? p.D[h] : 0.f;
    if (t0 >= t1) return;
    float* st = p.state + ((long long)slot * p.heads + h) * (long long)N * P;
    f2 s[4][CPL];
    load_state<RL, CPL>(st, N, P, rlane, c0, p.state_vec != 0, s);
    const float rate = per_head ? -expf(A_log) : 0.f;

    auto rows = [&](const float* src, float (&x)[8]) {     // the lane's entries of a vector of N, zeros beyond
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            const int at = 4 * rlane + 4 * RL * g;
            if (p.wide) {
                const float4 v = at < N ? *reinterpret_cast<const float4*>(src + at) : make_float4(0.f, 0.f, 0.f, 0.f);
                x[4 * g] = v.x; x[4 * g + 1] = v.y; x[4 * g + 2] = v.z; x[4 * g + 3] = v.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) x[4 * g + e] = at + e < N ? src[at + e] : 0.f;
            }
        }
    };
    // sum over N of x y, as the lanes of a helper add it up: one chain a four (RL = 32: one for both fours), then pairs of
    // neighbouring lanes, pairs of pairs, ...
    auto dot = [&](const float (&x)[8], const float (&y)[8]) {
        float part[2] = {0.f, 0.f};
#pragma unroll
        for (int i = 0; i < 8; ++i) part[RL == 32 ? 0 : i >> 2] = fmaf(x[i], y[i], part[RL == 32 ? 0 : i >> 2]);
#pragma unroll
        for (int o = 1; o < RL; o <<= 1) {
            part[0] += __shfl_xor_sync(0xffffffffu, part[0], o);
            if (RL < 32) part[1] += __shfl_xor_sync(0xffffffffu, part[1], o);
        }
        return RL == 32 ? part[0] : part[0] + part[1];
    };
    for (long long t = t0; t < t1; ++t) {
        float q[8], k[8], a[8], rr[8], v[CPL];
        float4 sc = make_float4(0.f, 0.f, 0.f, 0.f);
        rows(p.q + t * p.ldq + (long long)hq * N, q);
        rows(p.k + t * p.ldk + (long long)hq * N, k);
        if (CHANNEL) rows(p.dec + t * p.ldd + (long long)h * N, a);
        if (MODE == WALK_REMOVE) rows(p.rate + t * p.ldr + (long long)h * N, rr);
        const float* src = p.v + t * p.ldv + (long long)h * P + c0;
        if (p.wide && c0 < P) {
            load_columns(src, v);
        } else {
#pragma unroll
            for (int c = 0; c < CPL; ++c) v[c] = c0 + c < P ? src[c] : 0.f;
        }
        if (MODE == WALK_HEAD) {
            const float dt = fixed ? 1.0f : softplus_w(p.dec[t * p.ldd + h] + bias);
            sc.x = fixed ? fixed_a : expf(rate * dt);
            sc.y = dt;
            if (p.silu_inputs) {
                each_row<RL>(q, lane, [](float x, int) { return silu_f(x); });
                each_row<RL>(k, lane, [](float x, int) { return silu_f(x); });
#pragma unroll
                for (int c = 0; c < CPL; ++c) v[c] = silu_f(v[c]);
            }
        } else if (MODE == WALK_CHANNEL) {
#pragma unroll
            for (int i = 0; i < 8; ++i) q[i] *= p.q_scale;
            each_row<RL>(a, lane, [&](float x, int) { return expf(-softplus_w(-x) * p.inv_tau); });
        } else if (MODE == WALK_DELTA) {
            const float qq = dot(q, q), kk = dot(k, k), qk = dot(q, k);
            const float fq = p.unit ? p.q_scale * (1.0f / sqrtf(qq + p.unit_eps)) : p.q_scale;
            const float fk = p.unit ? 1.0f / sqrtf(kk + p.unit_eps) : 1.0f;
            sc.x = expf(rate * softplus_w(p.dec[t * p.ldd + h] + bias));
            sc.y = sigmoid_w(p.beta[t * p.ldb + h]);
            sc.z = qk * (fq * fk);
#pragma unroll
            for (int i = 0; i < 8; ++i) { q[i] *= fq; k[i] *= fk; }
        } else {
            each_row<RL>(a, lane, [&](float x, int n) { return n < N ? expf(-p.decay_coef * sigmoid_w(x)) : 0.f; });
            each_row<RL>(rr, lane, [&](float x, int n) { return n < N ? sigmoid_w(x + p.rate_bias[(long long)h * N + n]) : 0.f; });
#pragma unroll
            for (int i = 0; i < 8; ++i) rr[i] *= k[i];
            const float kk = dot(k, k), qk = dot(q, k), qr = dot(q, rr);
            const float inv = 1.0f / sqrtf(kk + p.unit_eps);
            sc.x = inv;
            sc.y = qr * inv;
            sc.z = qk;
#pragma unroll
            for (int i = 0; i < 8; ++i) { q[i] *= a[i]; rr[i] = -rr[i] * inv; }
        }
        f2 q2[4], k2[4], a2[4], r2[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            q2[i] = pack2(q[2 * i], q[2 * i + 1]);
            k2[i] = pack2(k[2 * i], k[2 * i + 1]);
            a2[i] = CHANNEL ? pack2(a[2 * i], a[2 * i + 1]) : pack2(sc.x, sc.x);
            if (MODE == WALK_REMOVE) r2[i] = pack2(rr[2 * i], rr[2 * i + 1]);
        }
        walk_token<MODE, RL, CPL>(s, q2, k2, a2, r2, sc, v, dcoef, rlane, P - c0, p.o + t * p.ldo + (long long)h * P + c0);
    }
    store_state<RL, CPL>(st, N, P, rlane, c0, p.state_vec != 0, s);
}

// RL: lanes that share a column's rows (N <= 8 RL).  Block = (head, request, a run of columns); the first p.walkers warps walk,
// CPL 32 / RL columns each, the others help.
template <int MODE, int RL, int CPL>
__global__ void __launch_bounds__(32 * MOST_WARPS, 1) scan_walk_kernel(WalkParams p) {
    dep_wait();           // nothing is read or written before the kernels before this one have ended
    constexpr int NP = 8 * RL, NV = walk_vectors<MODE>();
    constexpr int CL = 32 / RL, CW = CL * CPL;             // column lanes and columns of a warp
    constexpr int LT = 2 * RL < 32 ? 2 * RL : 32;          // lanes that fetch and prepare a token
    constexpr int QL = NP / 4 / LT;                        // fours of a vector a lane prepares
    constexpr int TPW = 32 / LT;                           // tokens a warp fetches at a time
    constexpr bool DELTA = MODE == WALK_DELTA || MODE == WALK_REMOVE;
    constexpr bool CHANNEL = MODE == WALK_CHANNEL || MODE == WALK_REMOVE;
    extern __shared__ __align__(16) float sm[];            // [STAGES][tile][q | k | decays | rates | v | 4 scalars]
    const int h = blockIdx.x, r = blockIdx.y;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, tile_tokens = p.tile;
    const int walkers = p.walkers, helpers = (int)(blockDim.x >> 5) - walkers;
    const int cols = walkers * CW, p0 = blockIdx.z * cols;
    const int off_v = NV * NP, off_s = off_v + ((cols + 3) & ~3), rl = off_s + 4;
    const int N = p.N, P = p.P;
    const int t0 = p.cu_q[r], t1 = p.cu_q[r + 1];
    const int n_tiles = (t1 - t0 + tile_tokens - 1) / tile_tokens;

    if (warp >= walkers) {
        const int ncols = min(cols, P - p0), hq = h / p.q_div;
        const bool fixed = MODE == WALK_HEAD && p.fixed_decay != nullptr;
        const float rate = (MODE == WALK_HEAD && !fixed) || MODE == WALK_DELTA ? -expf(p.A_log[h]) : 0.f;
        const float bias = ((MODE == WALK_HEAD && !fixed) || MODE == WALK_DELTA) && p.dec_bias != nullptr ? p.dec_bias[h] : 0.f;
        const float fixed_a = fixed ? p.fixed_decay[h] : 0.f;
        const int sub = lane / LT, lt = lane % LT, helper = warp - walkers;

        auto fetch = [&](int tile) {      // (a tile beyond the last: an empty group, so that the count of groups holds)
            float* buf = sm + (size_t)(tile % STAGES) * tile_tokens * rl;
            const int first = t0 + tile * tile_tokens, n = min(tile_tokens, t1 - first);
            for (int tok = helper * TPW + sub; tok < n; tok += helpers * TPW) {
                const long long t = first + tok;
                float* dst = buf + (size_t)tok * rl;
                const float* src[4] = {p.q + t * p.ldq + (long long)hq * N, p.k + t * p.ldk + (long long)hq * N,
                                       CHANNEL ? p.dec + t * p.ldd + (long long)h * N : nullptr,
                                       MODE == WALK_REMOVE ? p.rate + t * p.ldr + (long long)h * N : nullptr};
#pragma unroll
                for (int x = 0; x < NV; ++x)
#pragma unroll
                    for (int q = 0; q < QL; ++q) {
                        const int i = 4 * (lt + LT * q);
                        if (p.wide) {
                            if (i < N) copy16(dst + x * NP + i, src[x] + i);
                            else *reinterpret_cast<float4*>(dst + x * NP + i) = make_float4(0.f, 0.f, 0.f, 0.f);
                        } else {
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                if (i + e < N) copy4(dst + x * NP + i + e, src[x] + i + e);
                                else dst[x * NP + i + e] = 0.f;
                            }
                        }
                    }
                const float* srcv = p.v + t * p.ldv + (long long)h * P + p0;
                if (p.wide_v) for (int i = 4 * lt; i < ncols; i += 4 * LT) copy16(dst + off_v + i, srcv + i);
                else for (int i = lt; i < ncols; i += LT) copy4(dst + off_v + i, srcv + i);
                if (!CHANNEL && !fixed && lt == 0) copy4(dst + off_s, p.dec + t * p.ldd + h);
                if (MODE == WALK_DELTA && lt == 1) copy4(dst + off_s + 1, p.beta + t * p.ldb + h);
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        auto token_sum = [&](float v) {   // over the lanes of a token
#pragma unroll
            for (int o = 1; o < LT; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            return v;
        };
        // raw values of the tokens this warp fetched -> what the walk reads (a lane touches only what it copied itself)
        auto prepare = [&](int tile) {
            float* buf = sm + (size_t)(tile % STAGES) * tile_tokens * rl;
            const int first = t0 + tile * tile_tokens, n = min(tile_tokens, t1 - first);
            for (int tok0 = helper * TPW; tok0 < n; tok0 += helpers * TPW) {      // uniform over the warp
                const int tok = tok0 + sub;
                const bool mine = tok < n;
                float* row = buf + (size_t)(mine ? tok : 0) * rl;
                if (MODE == WALK_HEAD) {
                    if (mine && lt == 0) {
                        const float dt = fixed ? 1.0f : softplus_w(row[off_s] + bias);
                        row[off_s] = fixed ? fixed_a : expf(rate * dt);
                        row[off_s + 1] = dt;
                    }
                    if (p.silu_inputs && mine) {
#pragma unroll
                        for (int x = 0; x < 2; ++x)
#pragma unroll
                            for (int q = 0; q < QL; ++q)
#pragma unroll
                                for (int e = 0; e < 4; ++e) {
                                    float* v = row + x * NP + 4 * (lt + LT * q) + e;
                                    *v = silu_f(*v);
                                }
                        if (p.wide_v) {
                            for (int i = 4 * lt; i < ncols; i += 4 * LT)
                                for (int e = 0; e < 4; ++e) row[off_v + i + e] = silu_f(row[off_v + i + e]);
                        } else {
                            for (int i = lt; i < ncols; i += LT) row[off_v + i] = silu_f(row[off_v + i]);
                        }
                    }
                } else if (MODE == WALK_CHANNEL) {
                    if (mine) {
#pragma unroll
                        for (int q = 0; q < QL; ++q) {
                            const int i = 4 * (lt + LT * q);
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                row[i + e] *= p.q_scale;
                                float* a = row + 2 * NP + i + e;
                                *a = expf(-softplus_w(-*a) * p.inv_tau);
                            }
                        }
                    }
                } else {
                    float qv[4 * QL], kv[4 * QL], qq = 0.f, kk = 0.f, qk = 0.f, qr = 0.f;
                    float av[4 * QL], rv[4 * QL];
#pragma unroll
                    for (int q = 0; q < QL; ++q)
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const int i = 4 * (lt + LT * q) + e, x = 4 * q + e;
                            qv[x] = mine ? row[i] : 0.f;
                            kv[x] = mine ? row[NP + i] : 0.f;
                            qq = fmaf(qv[x], qv[x], qq);
                            kk = fmaf(kv[x], kv[x], kk);
                            qk = fmaf(qv[x], kv[x], qk);
                            if (MODE == WALK_REMOVE) {
                                av[x] = mine && i < N ? expf(-p.decay_coef * sigmoid_w(row[2 * NP + i])) : 0.f;
                                rv[x] = mine && i < N ? sigmoid_w(row[3 * NP + i] + p.rate_bias[(long long)h * N + i]) * kv[x] : 0.f;
                                qr = fmaf(qv[x], rv[x], qr);
                            }
                        }
                    kk = token_sum(kk);
                    qk = token_sum(qk);
                    if (MODE == WALK_DELTA) {
                        qq = token_sum(qq);
                        const float fq = p.unit ? p.q_scale * (1.0f / sqrtf(qq + p.unit_eps)) : p.q_scale;
                        const float fk = p.unit ? 1.0f / sqrtf(kk + p.unit_eps) : 1.0f;
                        if (mine) {
                            if (lt == 0) row[off_s] = expf(rate * softplus_w(row[off_s] + bias));
                            if (lt == 1) row[off_s + 1] = sigmoid_w(row[off_s + 1]);
                            if (lt == 0) row[off_s + 2] = qk * (fq * fk);
#pragma unroll
                            for (int q = 0; q < QL; ++q) {
                                const int i = 4 * (lt + LT * q);
                                *reinterpret_cast<float4*>(row + i) = make_float4(qv[4 * q] * fq, qv[4 * q + 1] * fq,
                                                                                  qv[4 * q + 2] * fq, qv[4 * q + 3] * fq);
                                *reinterpret_cast<float4*>(row + NP + i) = make_float4(kv[4 * q] * fk, kv[4 * q + 1] * fk,
                                                                                       kv[4 * q + 2] * fk, kv[4 * q + 3] * fk);
                            }
                        }
                    } else {
                        // k stays as it is (it carries v); the removal's r u u^T S = (r k / |k|)(k^T S / |k|): divided twice, so
                        // that nothing leaves the 32-bit range that u and r u do not leave; q meets the old state through
                        // the decays
                        qr = token_sum(qr);
                        const float inv = 1.0f / sqrtf(kk + p.unit_eps);
                        if (mine) {
                            if (lt == 0) row[off_s] = inv;
                            if (lt == 0) row[off_s + 1] = qr * inv;
                            if (lt == 1) row[off_s + 2] = qk;
#pragma unroll
                            for (int q = 0; q < QL; ++q) {
                                const int i = 4 * (lt + LT * q);
                                *reinterpret_cast<float4*>(row + i) = make_float4(qv[4 * q] * av[4 * q], qv[4 * q + 1] * av[4 * q + 1],
                                                                                  qv[4 * q + 2] * av[4 * q + 2], qv[4 * q + 3] * av[4 * q + 3]);
                                *reinterpret_cast<float4*>(row + 2 * NP + i) = make_float4(av[4 * q], av[4 * q + 1], av[4 * q + 2], av[4 * q + 3]);
                                *reinterpret_cast<float4*>(row + 3 * NP + i) = make_float4(-rv[4 * q] * inv, -rv[4 * q + 1] * inv,
                                                                                           -rv[4 * q + 2] * inv, -rv[4 * q + 3] * inv);
                            }
                        }
                    }
                }
            }
        };
        // one barrier a tile: while the walkers are at tile k, the helpers ask for tile k + 3 (into the buffer of tile k - 1,
        // which everyone has left) and prepare tile k + 1
        for (int k = 0; k < STAGES - 1; ++k) fetch(k);
        asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
        if (n_tiles > 0) prepare(0);
        __syncthreads();
        for (int k = 0; k < n_tiles; ++k) {
            fetch(k + STAGES - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(STAGES - 2) : "memory");
            if (k + 1 < n_tiles) prepare(k + 1);
            __syncthreads();
        }
        asm volatile("cp.async.wait_all;" ::: "memory");
        return;
    }

    const int rlane = lane & (RL - 1), c_local = warp * CW + (lane / RL) * CPL, c0 = p0 + c_local;
    const float dcoef = MODE == WALK_HEAD && p.D != nullptr ? p.D[h] : 0.f;
    float* st = p.state + ((long long)p.state_slot[r] * p.heads + h) * (long long)N * P;
    f2 s[4][CPL];
    load_state<RL, CPL>(st, N, P, rlane, c0, p.state_vec != 0, s);

    __syncthreads();
    for (int tile = 0; tile < n_tiles; ++tile) {
        const float* buf = sm + (size_t)(tile % STAGES) * tile_tokens * rl;
        const int first = t0 + tile * tile_tokens, n = min(tile_tokens, t1 - first);
#pragma unroll 4
        for (int tok = 0; tok < n; ++tok) {
            const float* row = buf + (size_t)tok * rl;
            const float4 sc = *reinterpret_cast<const float4*>(row + off_s);
            f2 q[4], k[4], a[4], rr[4];
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                const int at = 4 * rlane + 4 * RL * g;
                const ulonglong2 vq = *reinterpret_cast<const ulonglong2*>(row + at);
                const ulonglong2 vk = *reinterpret_cast<const ulonglong2*>(row + NP + at);
                q[2 * g] = vq.x; q[2 * g + 1] = vq.y;
                k[2 * g] = vk.x; k[2 * g + 1] = vk.y;
                if (CHANNEL) {
                    const ulonglong2 va = *reinterpret_cast<const ulonglong2*>(row + 2 * NP + at);
                    a[2 * g] = va.x; a[2 * g + 1] = va.y;
                } else {
                    a[2 * g] = a[2 * g + 1] = pack2(sc.x, sc.x);
                }
                if (MODE == WALK_REMOVE) {
                    const ulonglong2 vr = *reinterpret_cast<const ulonglong2*>(row + 3 * NP + at);
                    rr[2 * g] = vr.x; rr[2 * g + 1] = vr.y;
                }
            }
            float v[CPL];
            load_columns(row + off_v + c_local, v);
            walk_token<MODE, RL, CPL>(s, q, k, a, rr, sc, v, dcoef, rlane, P - c0,
                                      p.o + (long long)(first + tok) * p.ldo + (long long)h * P + c0);
        }
        __syncthreads();
    }
    store_state<RL, CPL>(st, N, P, rlane, c0, p.state_vec != 0, s);
}

template <int MODE, int RL, int CPL>
void launch_walk(WalkParams p, int R, int walkers, cudaStream_t stream) {
    constexpr int CW = 32 / RL * CPL;
    const int cols = walkers * CW;
    const int row = walk_vectors<MODE>() * 8 * RL + ((cols + 3) & ~3) + 4;
    p.walkers = walkers;
    p.state_vec = p.P % CPL == 0 && reinterpret_cast<uintptr_t>(p.state) % (CPL * sizeof(float)) == 0 ? 1 : 0;
    const dim3 grid(p.heads, R, (p.P + cols - 1) / cols);
    // One token a request, or two or three where the ring's kernel would need more than one wave (64 requests of three tokens,
    // gated delta rule, 16 heads of 128 x 128: 101 us there, 72 here; with four tokens the chain of loads a token costs as much
    // as it saves: 32 requests, gated linear attention, 16 heads of 64 x 128: 23 and 27).
    if (p.longest == 1 || (p.longest >= 1 && p.longest <= 3 && (long long)grid.x * grid.y * grid.z > sm_count())) {
        scan_few_kernel<MODE, RL, CPL><<<grid, 32 * walkers, 0, stream>>>(p);
        return;
    }
    p.wide_v = p.wide && cols % 4 == 0 ? 1 : 0;              // (a block's first column is a multiple of `cols`)
    p.tile = 16;
    while (p.tile > 1 && (size_t)STAGES * p.tile * row * sizeof(float) > 150 * 1024) p.tile /= 2;
    const size_t smem = (size_t)STAGES * p.tile * row * sizeof(float);
    auto kern = scan_walk_kernel<MODE, RL, CPL>;
    if (smem > 48 * 1024) cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    kern<<<grid, 32 * (walkers + HELPERS), smem, stream>>>(p);
}

template <int MODE, int RL>
void launch_rl(const WalkParams& p, int R, cudaStream_t stream) {
    constexpr int CL = 32 / RL;
    auto blocks = [&](int cpl, int walkers) { return (long long)p.heads * R * ((p.P + walkers * CL * cpl - 1) / (walkers * CL * cpl)); };
    // Four columns a lane where that still leaves three warps a multiprocessor (64 heads of 128 x 64, 2,048 tokens, 3.5 warps:
    // 289 us against 401 with two), two otherwise (32 heads of 64 x 64: 316 against 444; 16 heads of 128 x 128: 337 against 421).
    const int cpl = blocks(4, 1) >= 3LL * sm_count() ? 4 : 2;
    // Four walkers a block, which then share one preparation; two where there would be a block for less than every other
    // multiprocessor (32 heads of 64 x 64: 316 us against 346; 16 heads of 64 x 128 with a decay per channel: 180 against 212).
    int walkers = MOST_WALKERS;
    while (walkers > 1 && (blocks(cpl, walkers) < sm_count() / 2 || CL * cpl * walkers / 2 >= p.P)) walkers /= 2;
    if (cpl == 4) launch_walk<MODE, RL, 4>(p, R, walkers, stream);
    else launch_walk<MODE, RL, 2>(p, R, walkers, stream);
}

template <int MODE>
void launch_mode(const WalkParams& p, int R, cudaStream_t stream) {
    if (p.N <= 8) launch_rl<MODE, 1>(p, R, stream);
    else if (p.N <= 16) launch_rl<MODE, 2>(p, R, stream);
    else if (p.N <= 32) launch_rl<MODE, 4>(p, R, stream);
    else if (p.N <= 64) launch_rl<MODE, 8>(p, R, stream);
    else if (p.N <= 128) launch_rl<MODE, 16>(p, R, stream);
    else launch_rl<MODE, 32>(p, R, stream);
}

}  // namespace

bool scan_walk(int mode, WalkParams p, int R, cudaStream_t stream) {
    if (p.N > 256) return false;
    auto aligned = [](const float* x, int ld) { return reinterpret_cast<uintptr_t>(x) % 16 == 0 && ld % 4 == 0; };
    p.wide = p.N % 4 == 0 && p.P % 4 == 0 && aligned(p.q, p.ldq) && aligned(p.k, p.ldk) && aligned(p.v, p.ldv) &&
             (mode == WALK_HEAD || mode == WALK_DELTA || aligned(p.dec, p.ldd)) &&
             (mode != WALK_REMOVE || aligned(p.rate, p.ldr)) ? 1 : 0;
    switch (mode) {
        case WALK_HEAD: launch_mode<WALK_HEAD>(p, R, stream); break;
        case WALK_CHANNEL: launch_mode<WALK_CHANNEL>(p, R, stream); break;
        case WALK_DELTA: launch_mode<WALK_DELTA>(p, R, stream); break;
        default: launch_mode<WALK_REMOVE>(p, R, stream); break;
    }
    check_launch("scan_walk");
    return true;
}

}  // namespace dlmk
