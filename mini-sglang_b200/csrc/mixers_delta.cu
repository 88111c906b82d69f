// Kernels of softmax attention with a learned term in the denominator, of the gated delta rule and of the block
// arrangement with scaled sums and a per-layer token input (sm_100a; plain C entry points, loaded by ops.py as the
// library "mixers_delta", built only for models with such parts):
//
//   scaled_add_norm_kernel     res += x * s (s a float32 vector of the width), then y = rms(res) * w or y = res (or no y)
//   rotary_angles_kernel       cos | sin of position * frequency for the tokens of a step, in double precision
//   sink_qkv_prep_kernel       q and k heads RMS-normed, rotated in halves or in neighbouring pairs from the step's angles and
//                              brought to unit root mean square, heads of several maps laid out for one kv head, values
//                              blended with another layer's or brought to unit root mean square (each where asked), K and V
//                              rows (of head sizes of their own) into the paged cache; a 16-byte form where nothing is
//                              blended or rotated in halves
//   sink_attention_kernel      causal softmax attention within a window or a chunk over the paged cache, scores capped by a tanh
//                              where asked, with exp(sink_h) in the denominator and the output times a sigmoid gate per
//                              element where given; float32 arithmetic, any head size to 512
//   sink_attention_mma_kernel  the same for bfloat16 with both products on mma.sync tiles (64 rows a block, float32 scores,
//                              running maximum and sum), prompts, portions and decoded tokens
//   sink_merge_kernel          one-token steps cut a request's keys into pieces for blocks of their own: the pieces'
//                              (max, sum, weighted values) are joined, in the order of the pieces, with the sink
//   delta_prep_kernel          unit-length q and k, beta and g of the gated delta rule from their projections, all tokens
//   delta_rule_kernel          S <- g S; u = beta (v - S^T k); S <- S + k u^T; o = S^T q per head, token by token
//   delta_chunk_kernel, delta_chunk_scan_kernel   the same for runs of tokens, in chunks of 32
//   side_gate_mul_kernel       gelu_tanh(gate) times a slice of a per-token table's row
//
// Scores, weights, norms, angles, decays, states and everything that enters the recurrence are float32 (angles: double);
// T is the type of the activations between kernels (float or bfloat16).  Key chunks and pieces are anchored at absolute
// positions, so the order of a position's sums does not depend on how the tokens were cut into steps.
#include "common.cuh"
#include "tc_common.cuh"
#include <math.h>

namespace {
__device__ __forceinline__ float sigmoidf_(float x) { return 1.f / (1.f + expf(-x)); }
__device__ __forceinline__ float gelu_tanhf_(float z) {
    return 0.5f * z * (1.f + tanhf(0.7978845608028654f * (z + 0.044715f * z * z * z)));
}
__device__ __forceinline__ float softplusf_(float x) { return fmaxf(x, 0.f) + log1pf(expf(-fabsf(x))); }
}  // namespace

// ---------------------------------------------------------------------------------------
// res += x * s;  y = res / sqrt(mean(res^2) + eps) * w  (w given)  or  y = res  (y given, no w)
// One block per row; the sum of squares in float32.
// ---------------------------------------------------------------------------------------
template <typename A, typename O>
__global__ void __launch_bounds__(256) scaled_add_norm_kernel(const A* __restrict__ x, const float* __restrict__ s, float* __restrict__ res,
                                                              const float* __restrict__ w, float eps, O* __restrict__ y, int H) {
    __shared__ float scratch[32];
    const size_t row = (size_t)blockIdx.x * H;
    float ss = 0.f;
    for (int i = threadIdx.x; i < H; i += blockDim.x) {
        const float v = fmaf(to_f32<A>(x[row + i]), s[i], res[row + i]);
        res[row + i] = v;
        ss = fmaf(v, v, ss);
    }
    if (y == nullptr) return;
    float rs = 1.f;
    if (w != nullptr) rs = 1.f / sqrtf(block_sum(ss, scratch) / (float)H + eps);
    for (int i = threadIdx.x; i < H; i += blockDim.x) y[row + i] = from_f32<O>(w ? res[row + i] * rs * w[i] : res[row + i]);
}

// The same with four neighbouring columns a thread and turn (H a multiple of 4, rows 16-byte aligned); the row's new values stay
// in registers between the sum and the norm where the row has at most 4 * NV * blockDim columns.
template <typename A, typename O, int NV>
__global__ void __launch_bounds__(256) scaled_add_norm_vec_kernel(const A* __restrict__ x, const float* __restrict__ s, float* __restrict__ res,
                                                                  const float* __restrict__ w, float eps, O* __restrict__ y, int H) {
    __shared__ float scratch[32];
    const size_t row = (size_t)blockIdx.x * H;
    float v[NV][4];
    float ss = 0.f;
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        if (i < H) {
            const float4 r4 = *reinterpret_cast<const float4*>(res + row + i), s4 = *reinterpret_cast<const float4*>(s + i);
            float xv[4];
            if constexpr (sizeof(A) == 4) {
                const float4 x4 = *reinterpret_cast<const float4*>(reinterpret_cast<const float*>(x) + row + i);
                xv[0] = x4.x; xv[1] = x4.y; xv[2] = x4.z; xv[3] = x4.w;
            } else {
                const uint2 u = *reinterpret_cast<const uint2*>(reinterpret_cast<const __nv_bfloat16*>(x) + row + i);
                xv[0] = __uint_as_float(u.x << 16); xv[1] = __uint_as_float(u.x & 0xffff0000u);
                xv[2] = __uint_as_float(u.y << 16); xv[3] = __uint_as_float(u.y & 0xffff0000u);
            }
            v[k][0] = fmaf(xv[0], s4.x, r4.x); v[k][1] = fmaf(xv[1], s4.y, r4.y);
            v[k][2] = fmaf(xv[2], s4.z, r4.z); v[k][3] = fmaf(xv[3], s4.w, r4.w);
            *reinterpret_cast<float4*>(res + row + i) = make_float4(v[k][0], v[k][1], v[k][2], v[k][3]);
            ss += v[k][0] * v[k][0] + v[k][1] * v[k][1] + v[k][2] * v[k][2] + v[k][3] * v[k][3];
        }
    }
    if (y == nullptr) return;
    float rs = 1.f;
    if (w != nullptr) rs = 1.f / sqrtf(block_sum(ss, scratch) / (float)H + eps);
#pragma unroll
    for (int k = 0; k < NV; ++k) {
        const int i = (threadIdx.x + k * blockDim.x) * 4;
        if (i < H) {
            float o[4];
            if (w != nullptr) {
                const float4 w4 = *reinterpret_cast<const float4*>(w + i);
                o[0] = v[k][0] * rs * w4.x; o[1] = v[k][1] * rs * w4.y; o[2] = v[k][2] * rs * w4.z; o[3] = v[k][3] * rs * w4.w;
            } else {
                o[0] = v[k][0]; o[1] = v[k][1]; o[2] = v[k][2]; o[3] = v[k][3];
            }
            if constexpr (sizeof(O) == 4) {
                *reinterpret_cast<float4*>(reinterpret_cast<float*>(y) + row + i) = make_float4(o[0], o[1], o[2], o[3]);
            } else {
                const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
                *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(y) + row + i) =
                    make_uint2(*reinterpret_cast<const unsigned*>(&a), *reinterpret_cast<const unsigned*>(&b));
            }
        }
    }
}

MSGL_API int msgl_scaled_add_norm(const void* x, int x_is_f32, const float* s, float* res, const float* w, float eps, void* y,
                                  int y_dtype, int T_, int H, cudaStream_t stream) {
    if (T_ <= 0) return MSGL_OK;
    if (H <= 0) return MSGL_ERR_SIZE;
    if (y_dtype != MSGL_F32 && y_dtype != MSGL_BF16) return MSGL_ERR_DTYPE;
    const bool aligned = H % 4 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)res % 16) == 0 && ((uintptr_t)s % 16) == 0 &&
                         ((uintptr_t)w % 16) == 0 && ((uintptr_t)y % 16) == 0 && (x_is_f32 || H % 8 == 0);
    if (aligned && H <= 4 * 4 * 256) {
        const int vt = H <= 1024 ? 64 : (H <= 4096 ? 256 : 256);
        const int nv = (H / 4 + vt - 1) / vt;
#define SANV(A, O, NV) scaled_add_norm_vec_kernel<A, O, NV><<<T_, vt, 0, stream>>>((const A*)x, s, res, w, eps, (O*)y, H)
#define SANV_T(NV)                                                                                                           \
    do {                                                                                                                     \
        if (y_dtype == MSGL_F32) { if (x_is_f32) SANV(float, float, NV); else SANV(__nv_bfloat16, float, NV); }              \
        else { if (x_is_f32) SANV(float, __nv_bfloat16, NV); else SANV(__nv_bfloat16, __nv_bfloat16, NV); }                  \
    } while (0)
        if (nv <= 1) SANV_T(1); else if (nv <= 2) SANV_T(2); else SANV_T(4);
#undef SANV_T
#undef SANV
        return msgl_check_launch();
    }
    const int threads = H >= 1024 ? 256 : 128;
#define SAN(A, O) scaled_add_norm_kernel<A, O><<<T_, threads, 0, stream>>>((const A*)x, s, res, w, eps, (O*)y, H)
    if (y_dtype == MSGL_F32) { if (x_is_f32) SAN(float, float); else SAN(__nv_bfloat16, float); }
    else if (y_dtype == MSGL_BF16) { if (x_is_f32) SAN(float, __nv_bfloat16); else SAN(__nv_bfloat16, __nv_bfloat16); }
    else return MSGL_ERR_DTYPE;
#undef SAN
    return msgl_check_launch();
}

// ---------------------------------------------------------------------------------------
// out[t, i] = mag * cos(position_t * f_i),  out[t, half + i] = mag * sin(position_t * f_i),  i < half; double precision
// ---------------------------------------------------------------------------------------
__global__ void rotary_angles_kernel(const int* __restrict__ positions, const double* __restrict__ freq, double mag, float* __restrict__ out,
                                     int T_, int half) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= T_ * half) return;
    const int t = idx / half, i = idx - t * half;
    double s, c;
    sincos((double)positions[t] * freq[i], &s, &c);
    out[(size_t)t * 2 * half + i] = (float)(c * mag);
    out[(size_t)t * 2 * half + half + i] = (float)(s * mag);
}

MSGL_API int msgl_rotary_angles(const int* positions, const double* freq, double mag, float* out, int T_, int half, cudaStream_t stream) {
    if (T_ <= 0 || half <= 0) return MSGL_OK;
    const int n = T_ * half;
    rotary_angles_kernel<<<(n + 127) / 128, 128, 0, stream>>>(positions, freq, mag, out, T_, half);
    return msgl_check_launch();
}

// ---------------------------------------------------------------------------------------
// q, k, v of a packed projection row [q: n_q * d | k: n_kv * d | v: n_kv * dv]:
//   q and k heads: where weights are given (wq, wk [d], for all heads), x / sqrt(mean(x^2) + eps) * w first; then the first
//   `rot` elements turn by the token's angles (cs [T][rot] = cos | sin), in halves (element i with i + rot / 2) or, with
//   `interleaved`, in neighbouring pairs (2 i with 2 i + 1), the rest pass; with qk_unit then x / sqrt(mean(x^2) + eps)
//   v heads: v <- (1 - lam) v + lam v_first where another layer's values are given; with v_unit then v / sqrt(mean(v^2) + eps)
//   q -> q_out [T, n_q, d]; k, v -> the paged caches at token slot out_loc[t] (where given)
// With maps = M > 1 every q and kv head has M vectors of d elements side by side, each treated as a head of its own by all of
// the above: K rows are the M vectors of a kv head [M * d]; q comes out as n_q * M rows of M * d elements of which row
// (h, m) has its vector in place m and zeros in the others, so that its product with a K row is that of map m alone.
// One warp per (token, vector of q, k or v).
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void sk_load16(const float* p, float (&v)[4]) {
    const float4 a = *reinterpret_cast<const float4*>(p);
    v[0] = a.x; v[1] = a.y; v[2] = a.z; v[3] = a.w;
}
__device__ __forceinline__ void sk_load16(const __nv_bfloat16* p, float (&v)[8]) {
    const uint4 a = *reinterpret_cast<const uint4*>(p);
    const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&a);
#pragma unroll
    for (int k = 0; k < 4; ++k) { const float2 f = __bfloat1622float2(h[k]); v[2 * k] = f.x; v[2 * k + 1] = f.y; }
}
__device__ __forceinline__ void sk_store16(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void sk_store16(__nv_bfloat16* p, const float (&v)[8]) {
    uint4 a;
    __nv_bfloat162* h = reinterpret_cast<__nv_bfloat162*>(&a);
#pragma unroll
    for (int k = 0; k < 4; ++k) h[k] = __floats2bfloat162_rn(v[2 * k], v[2 * k + 1]);
    *reinterpret_cast<uint4*>(p) = a;
}

struct SinkPrepParams {
    const void* proj; long long stride;
    const float* cs; int rot;
    const void* v_first; long long vf_stride; float lam;
    const int* out_loc; void* q_out; void* k_cache; void* v_cache;
    int page_size, n_q, n_kv, d, dv, T;
    const float* wq; const float* wk; int v_unit; float eps;
    int interleaved, qk_unit, maps;
};

template <typename T>
__global__ void __launch_bounds__(128) sink_qkv_prep_kernel(const SinkPrepParams p) {
    const int t = blockIdx.x;
    const int slot = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    const int M = p.maps, nq = p.n_q * M, nk = p.n_kv * M;
    if (slot >= nq + nk + p.n_kv) return;
    const T* row = reinterpret_cast<const T*>(p.proj) + (size_t)t * p.stride;
    const int half = p.rot >> 1;
    const float* cs = p.cs ? p.cs + (size_t)t * p.rot : nullptr;
    if (slot < nq + nk) {
        const bool is_q = slot < nq;
        const int h = is_q ? slot : slot - nq, m = h % M;
        const T* src = row + (size_t)slot * p.d;
        T* dst;
        if (is_q) {
            dst = reinterpret_cast<T*>(p.q_out) + ((size_t)t * nq + h) * p.d * M;
            for (int e = lane; e < p.d * M; e += 32)
                if (e / p.d != m) dst[e] = from_f32<T>(0.f);
        } else {
            if (p.k_cache == nullptr) return;
            const int loc = p.out_loc[t];
            dst = reinterpret_cast<T*>(p.k_cache) + (((size_t)(loc / p.page_size) * p.n_kv + h / M) * p.page_size + loc % p.page_size) * p.d * M;
        }
        dst += m * p.d;
        const float* w = is_q ? p.wq : p.wk;
        float f = 1.f;
        if (w != nullptr) {
            float ss = 0.f;
            for (int e = lane; e < p.d; e += 32) { const float v = to_f32<T>(src[e]); ss = fmaf(v, v, ss); }
            f = 1.f / sqrtf(warp_sum(ss) / (float)p.d + p.eps);
        }
        auto elem = [&](int e) -> float { const float v = to_f32<T>(src[e]); return w != nullptr ? v * f * w[e] : v; };
        auto turned = [&](int e) -> float {
            const float v = elem(e);
            if (cs == nullptr || e >= p.rot) return v;
            if (p.interleaved) {
                const float c = cs[e >> 1], s = cs[half + (e >> 1)], o = elem(e ^ 1);
                return (e & 1) ? v * c + o * s : v * c - o * s;
            }
            return e < half ? v * cs[e] - elem(e + half) * cs[half + e] : v * cs[e - half] + elem(e - half) * cs[e];
        };
        float g = 1.f;
        if (p.qk_unit) {
            float ss = 0.f;
            for (int e = lane; e < p.d; e += 32) { const float v = turned(e); ss = fmaf(v, v, ss); }
            g = 1.f / sqrtf(warp_sum(ss) / (float)p.d + p.eps);
        }
        for (int e = lane; e < p.d; e += 32) dst[e] = from_f32<T>(turned(e) * g);
    } else {
        if (p.v_cache == nullptr) return;
        const int h = slot - nq - nk;
        const T* src = row + (size_t)(nq + nk) * p.d + (size_t)h * p.dv;
        const T* vf = p.v_first ? reinterpret_cast<const T*>(p.v_first) + (size_t)t * p.vf_stride + (size_t)h * p.dv : nullptr;
        const int loc = p.out_loc[t];
        T* dst = reinterpret_cast<T*>(p.v_cache) + (((size_t)(loc / p.page_size) * p.n_kv + h) * p.page_size + loc % p.page_size) * p.dv;
        auto elem = [&](int e) -> float {
            const float v = to_f32<T>(src[e]);
            return vf != nullptr ? (1.f - p.lam) * v + p.lam * to_f32<T>(vf[e]) : v;
        };
        float f = 1.f;
        if (p.v_unit) {
            float ss = 0.f;
            for (int e = lane; e < p.dv; e += 32) { const float v = elem(e); ss = fmaf(v, v, ss); }
            f = 1.f / sqrtf(warp_sum(ss) / (float)p.dv + p.eps);
        }
        for (int e = lane; e < p.dv; e += 32) dst[e] = from_f32<T>(elem(e) * f);
    }
}

// The same without blending or a rotation in halves, a lane 16 bytes of a vector (sizes that are multiples of the lane's share and
// at most 32 of them): one read of every element, norms and turned pairs from registers.  n_slots: the vectors of a token that
// are made (q alone where nothing is cached); their number in all fits 32 bits.
template <typename T>
__global__ void __launch_bounds__(128) sink_qkv_prep_vec_kernel(const SinkPrepParams p, int n_slots, int lg) {
    constexpr int V = 16 / sizeof(T);
    pdl_launch_dependents();
    const int M = p.maps, nq = p.n_q * M, nk = p.n_kv * M, lane = threadIdx.x & 31;
    // 2^lg lanes take a vector; vectors of 16 shares or less share a warp
    const int lanes = 1 << lg, l = lane & (lanes - 1);
    const unsigned job = ((blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5)) << (5 - lg)) + (unsigned)(lane >> lg);
    const bool live = job < (unsigned)p.T * (unsigned)n_slots;
    const int t = live ? (int)(job / (unsigned)n_slots) : 0, slot = live ? (int)job - t * n_slots : 0;
    const bool is_v = slot >= nq + nk, is_q = slot < nq;
    const int n = is_v ? p.dv : p.d;
    const T* row = reinterpret_cast<const T*>(p.proj) + (size_t)t * p.stride;
    const T* src = is_v ? row + (size_t)(nq + nk) * p.d + (size_t)(slot - nq - nk) * p.dv : row + (size_t)slot * p.d;
    const bool mine = live && l * V < n;
    float v[V];
#pragma unroll
    for (int k = 0; k < V; ++k) v[k] = 0.f;
    pdl_wait();
    pdl_after_wait();
    pdl_small();
    if (mine) sk_load16(src + l * V, v);
    const float* w = is_v ? nullptr : (is_q ? p.wq : p.wk);
    if (w != nullptr || (is_v && p.v_unit)) {           // (the lanes of one vector take the same branch: the shuffles stay among them)
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) ss = fmaf(v[k], v[k], ss);
        const unsigned mask = lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1u) << (lane - l);
        for (int o = lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(mask, ss, o);
        const float f = 1.f / sqrtf(ss / (float)n + p.eps);
        if (w != nullptr && mine) {
            const float4* w4 = reinterpret_cast<const float4*>(w + l * V);
#pragma unroll
            for (int k = 0; k < V / 4; ++k) {
                const float4 x = w4[k];
                v[4 * k] *= f * x.x; v[4 * k + 1] *= f * x.y; v[4 * k + 2] *= f * x.z; v[4 * k + 3] *= f * x.w;
            }
        } else {
#pragma unroll
            for (int k = 0; k < V; ++k) v[k] *= f;
        }
    }
    if (p.cs != nullptr && !is_v && mine) {             // neighbouring pairs lie within a lane
        const float* cs = p.cs + (size_t)t * p.rot;
        const int half = p.rot >> 1;
        float cv[V / 2], sv[V / 2];
        const int p0 = (l * V) >> 1;
        if (V == 8 && (half & 3) == 0) {                // a lane's pairs are turned together or not at all: 16 bytes of angles at once
            if (p0 < half) {
                const float4 c4 = *reinterpret_cast<const float4*>(cs + p0), s4 = *reinterpret_cast<const float4*>(cs + half + p0);
                cv[0] = c4.x; cv[1] = c4.y; sv[0] = s4.x; sv[1] = s4.y;
                if constexpr (V == 8) { cv[2] = c4.z; cv[3] = c4.w; sv[2] = s4.z; sv[3] = s4.w; }
            } else {
#pragma unroll
                for (int k = 0; k < V / 2; ++k) { cv[k] = 1.f; sv[k] = 0.f; }
            }
        } else {
#pragma unroll
            for (int k = 0; k < V / 2; ++k) { cv[k] = p0 + k < half ? cs[p0 + k] : 1.f; sv[k] = p0 + k < half ? cs[half + p0 + k] : 0.f; }
        }
#pragma unroll
        for (int k = 0; k < V / 2; ++k) {
            const float a = v[2 * k], b = v[2 * k + 1];
            if (p0 + k < half) { v[2 * k] = a * cv[k] - b * sv[k]; v[2 * k + 1] = b * cv[k] + a * sv[k]; }
        }
    }
    if (p.qk_unit && !is_v) {
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < V; ++k) ss = fmaf(v[k], v[k], ss);
        const unsigned mask = lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1u) << (lane - l);
        for (int o = lanes >> 1; o > 0; o >>= 1) ss += __shfl_xor_sync(mask, ss, o);
        const float f = 1.f / sqrtf(ss / (float)n + p.eps);
#pragma unroll
        for (int k = 0; k < V; ++k) v[k] *= f;
    }
    if (!mine) return;
    T* dst;
    if (is_q) {
        const int m = M == 1 ? 0 : (M == 2 ? slot & 1 : slot % M);
        dst = reinterpret_cast<T*>(p.q_out) + ((size_t)t * nq + slot) * n * M + l * V;
        float z[V];
#pragma unroll
        for (int k = 0; k < V; ++k) z[k] = 0.f;
        for (int o = 0; o < M; ++o)
            if (o != m) sk_store16(dst + o * n, z);
        dst += m * n;
    } else {
        const int loc = p.out_loc[t], h = is_v ? slot - nq - nk : slot - nq;
        const int mm = is_v ? 1 : M, hh = mm == 1 ? h : (mm == 2 ? h >> 1 : h / mm);
        const unsigned page = (unsigned)loc / (unsigned)p.page_size, at = (unsigned)loc - page * (unsigned)p.page_size;
        dst = reinterpret_cast<T*>(is_v ? p.v_cache : p.k_cache) + (((size_t)page * p.n_kv + hh) * p.page_size + at) * (size_t)(n * mm) +
              (h - hh * mm) * n + l * V;
    }
    sk_store16(dst, v);
}

MSGL_API int msgl_sink_qkv_prep(const void* proj, long long stride, const float* cs, int rot, const void* v_first, long long vf_stride,
                                float lam, const int* out_loc, void* q_out, void* k_cache, void* v_cache, int page_size, int n_q, int n_kv,
                                int d, int dv, int T_, int dtype, const float* wq, const float* wk, int v_unit, float eps,
                                int interleaved, int qk_unit, int maps, cudaStream_t stream) {
    if (T_ <= 0) return MSGL_OK;
    if (dtype != MSGL_F32 && dtype != MSGL_BF16) return MSGL_ERR_DTYPE;
    if (d <= 0 || dv <= 0 || n_q <= 0 || n_kv <= 0 || rot < 0 || rot > d || (rot & 1) || page_size < 1 || maps < 1 || (rot > 0 && cs == nullptr) ||
        (k_cache != nullptr && (out_loc == nullptr || v_cache == nullptr)))
        return MSGL_ERR_SIZE;
    SinkPrepParams p;
    p.proj = proj; p.stride = stride; p.cs = rot > 0 ? cs : nullptr; p.rot = rot; p.v_first = v_first; p.vf_stride = vf_stride; p.lam = lam;
    p.out_loc = out_loc; p.q_out = q_out; p.k_cache = k_cache; p.v_cache = v_cache; p.page_size = page_size; p.n_q = n_q; p.n_kv = n_kv;
    p.d = d; p.dv = dv; p.T = T_; p.wq = wq; p.wk = wk; p.v_unit = v_unit; p.eps = eps;
    p.interleaved = interleaved; p.qk_unit = qk_unit; p.maps = maps;
    const int V = dtype == MSGL_F32 ? 4 : 8;
    const uintptr_t all = (uintptr_t)proj | (uintptr_t)q_out | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)wq | (uintptr_t)wk;
    // vectors of a token: q, and where they are cached k and v
    const int n_slots = maps * n_q + (k_cache != nullptr ? (maps + 1) * n_kv : 0);
    if ((p.cs == nullptr || interleaved) && v_first == nullptr && d % V == 0 && dv % V == 0 && stride % V == 0 && max(d, dv) <= 32 * V && (all & 15) == 0 &&
        ((uintptr_t)cs & 15) == 0 && (long long)T_ * n_slots < (1ll << 30)) {
        const int widest = max(d, dv) / V, lg = widest <= 4 ? 2 : widest <= 8 ? 3 : widest <= 16 ? 4 : 5, per = 4 * (32 >> lg);
        const unsigned blocks = (unsigned)(((long long)T_ * n_slots + per - 1) / per);
        if (dtype == MSGL_F32) msgl_launch_pdl(sink_qkv_prep_vec_kernel<float>, dim3(blocks), dim3(128), 0, stream, p, n_slots, lg);
        else msgl_launch_pdl(sink_qkv_prep_vec_kernel<__nv_bfloat16>, dim3(blocks), dim3(128), 0, stream, p, n_slots, lg);
        return msgl_check_launch();
    }
    const dim3 grid(T_, (n_slots + 3) / 4);
    if (dtype == MSGL_F32) sink_qkv_prep_kernel<float><<<grid, 128, 0, stream>>>(p);
    else if (dtype == MSGL_BF16) sink_qkv_prep_kernel<__nv_bfloat16><<<grid, 128, 0, stream>>>(p);
    else return MSGL_ERR_DTYPE;
    return msgl_check_launch();
}

// ---------------------------------------------------------------------------------------
// Causal softmax attention within a window or a chunk over the paged cache, with a sink
//
//   s(i, j) = q[i, h] . k[j, g] * scale;   s <- cap * tanh(s / cap) (cap > 0);   j <= i and (no window or i - j < window) and
//   (no chunks or j / chunk_keys == i / chunk_keys)
//   o[i, h, :] = sum_j exp(s(i, j)) v[j, g, :] / (sum_j exp(s(i, j)) + exp(sink[h]))        (sink null: without that term)
//   o[i, h, e] <- o[i, h, e] * sigmoid(gate[i, h, e])   (where gates are given: rows of the activation type, one per output element)
//
// A block owns a tile of QT tokens x GH query heads of one kv head (SK_ROWS rows, one warp each) and walks the keys in
// chunks of 32 anchored at multiples of 32, with a running maximum and sum per row.  In the score phase lane l of a row's
// warp takes key l of the chunk, in the value phase lane l takes the output elements l, l + 32, ...  Cache rows behind the
// window of the tile's first token are never read (their pages may be gone).  With `splits` > 1 (steps in which every
// request brings one token) block z walks piece z of the request's keys, pieces of `split_keys` keys anchored at multiples
// of split_keys from the piece that holds the first key the token sees, and leaves (max, sum, weighted values) in `part`.
// ---------------------------------------------------------------------------------------
#define SK_ROWS 8
#define SK_KC 32
#define SK_MAX_DPL 16       // head sizes up to 512

struct SinkAttnParams {
    const void* q;            // [T, n_q, d]
    const void* k_cache; const void* v_cache;
    const int* q_start; const int* kv_len; const int* block_table; int bt_stride;
    int uniform;
    const float* sink;                            // [n_q] or null
    void* out; long long out_stride;              // [T rows][n_q * dv]
    float* part_o; float* part_ml; int splits, split_keys;      // [splits][T][n_q][dv], [splits][T][n_q][2]
    int T, B, n_q, n_kv, d, dv, page_size, QT, GH, window;
    float scale, softcap;
    const void* gate; long long gate_stride;      // [T rows][n_q * dv] or null
    int chunk_keys;                               // > 0 (without a window): keys are seen within chunks of the sequence only
};

// the first key that the query at position `pos` sees
__device__ __forceinline__ int sk_first_key(const SinkAttnParams& p, int pos) {
    if (p.window > 0) return max(0, pos - p.window + 1);
    return p.chunk_keys > 0 ? pos - pos % p.chunk_keys : 0;
}

template <typename T, int DPL>
__global__ void __launch_bounds__(SK_ROWS * 32) sink_attention_kernel(const SinkAttnParams p) {
    extern __shared__ float smem[];
    const int d = p.d, dv = p.dv;
    float* qs = smem;                                // [SK_ROWS][d]
    float* ks = qs + SK_ROWS * d;                    // [SK_KC][d + 1]
    float* vs = ks + SK_KC * (d + 1);                // [SK_KC][dv]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    __shared__ int tile_sh[2];
    int req, t0;
    if (p.uniform) {
        req = blockIdx.x; t0 = 0;
    } else {
        if (tid == 0) {
            int left = blockIdx.x, found = -1, at = 0;
            for (int r = 0; r < p.B; ++r) {
                const int nt = (p.q_start[r + 1] - p.q_start[r] + p.QT - 1) / p.QT;
                if (left < nt) { found = r; at = left * p.QT; break; }
                left -= nt;
            }
            tile_sh[0] = found; tile_sh[1] = at;
        }
        __syncthreads();
        req = tile_sh[0]; t0 = tile_sh[1];
    }
    if (req < 0 || req >= p.B) return;
    const int G = p.n_q / p.n_kv;
    const int n_chunks = (G + p.GH - 1) / p.GH;
    const int kvh = blockIdx.y / n_chunks, chunk = blockIdx.y - kvh * n_chunks;
    const int q_base = p.q_start[req], q_len = p.q_start[req + 1] - q_base, kv_len = p.kv_len[req];
    const int n_tok = min(p.QT, q_len - t0);
    if (n_tok <= 0) return;
    const int p_min = kv_len - q_len + t0, p_max = p_min + n_tok - 1;
    int key_lo = sk_first_key(p, p_min), key_hi = p_max + 1;      // keys this block walks: [key_lo, key_hi)
    if (p.splits > 1) {
        const int piece = key_lo / p.split_keys + blockIdx.z;
        key_lo = max(key_lo, piece * p.split_keys);
        key_hi = min(key_hi, (piece + 1) * p.split_keys);
    }

    const int tl = warp / p.GH, hl = warp - tl * p.GH;
    const int hg = chunk * p.GH + hl;
    const bool row_ok = tl < n_tok && hg < G && tl < p.QT;
    const int head = kvh * G + (row_ok ? hg : 0);
    const int tok = q_base + t0 + (row_ok ? tl : 0);
    const int pos = p_min + tl;
    const int first_seen = sk_first_key(p, pos);
    const T* qg = reinterpret_cast<const T*>(p.q);
    for (int e = lane; e < d; e += 32) qs[warp * d + e] = row_ok ? to_f32<T>(qg[((size_t)tok * p.n_q + head) * d + e]) : 0.f;
    const T* kc = reinterpret_cast<const T*>(p.k_cache);
    const T* vc = reinterpret_cast<const T*>(p.v_cache);
    const int* bt = p.block_table + (size_t)req * p.bt_stride;
    const float inv_cap = p.softcap > 0.f ? 1.f / p.softcap : 0.f;

    float o[DPL];
#pragma unroll
    for (int i = 0; i < DPL; ++i) o[i] = 0.f;
    float m_run = -INFINITY, l_run = 0.f;

    for (int key0 = key_lo - key_lo % SK_KC; key0 < key_hi; key0 += SK_KC) {
        __syncthreads();
        for (int idx = tid; idx < SK_KC * d; idx += SK_ROWS * 32) {
            const int kr = idx / d, e = idx - kr * d;
            const int key = key0 + kr;
            float kv = 0.f;
            if (key >= key_lo && key < key_hi) {
                const int page = bt[key / p.page_size];
                kv = to_f32<T>(kc[(((size_t)page * p.n_kv + kvh) * p.page_size + (key % p.page_size)) * d + e]);
            }
            ks[kr * (d + 1) + e] = kv;
        }
        for (int idx = tid; idx < SK_KC * dv; idx += SK_ROWS * 32) {
            const int kr = idx / dv, e = idx - kr * dv;
            const int key = key0 + kr;
            float vv = 0.f;
            if (key >= key_lo && key < key_hi) {
                const int page = bt[key / p.page_size];
                vv = to_f32<T>(vc[(((size_t)page * p.n_kv + kvh) * p.page_size + (key % p.page_size)) * dv + e]);
            }
            vs[kr * dv + e] = vv;
        }
        __syncthreads();
        const int key = key0 + lane;
        const bool vis = row_ok && key <= pos && key >= first_seen && key >= key_lo && key < key_hi;
        float sc = -INFINITY;
        if (vis) {
            float acc = 0.f;
            const float* qr = qs + warp * d;
            const float* kr = ks + lane * (d + 1);
            for (int e = 0; e < d; ++e) acc = fmaf(qr[e], kr[e], acc);
            sc = acc * p.scale;
            if (p.softcap > 0.f) sc = p.softcap * tanhf(sc * inv_cap);
        }
        const float cm = warp_max(sc);
        if (cm == -INFINITY) continue;                               // warp-uniform: no key of the chunk is seen by this row
        const float m_new = fmaxf(m_run, cm);
        const float corr = expf(m_run - m_new);                      // 0 at the first seen chunk (m_run = -inf)
        const float pr = vis ? expf(sc - m_new) : 0.f;
        l_run = l_run * corr + warp_sum(pr);
        m_run = m_new;
#pragma unroll
        for (int i = 0; i < DPL; ++i) o[i] *= corr;
        for (int j = 0; j < SK_KC; ++j) {
            const float pj = __shfl_sync(0xffffffffu, pr, j);
            if (pj == 0.f) continue;                                 // warp-uniform
            const float* vr = vs + j * dv;
#pragma unroll
            for (int i = 0; i < DPL; ++i) {
                const int e = lane + 32 * i;
                if (e < dv) o[i] = fmaf(pj, vr[e], o[i]);
            }
        }
    }
    if (!row_ok) return;
    if (p.splits > 1) {
        const size_t r = ((size_t)blockIdx.z * p.T + tok) * p.n_q + head;
        float* pg = p.part_o + r * dv;
#pragma unroll
        for (int i = 0; i < DPL; ++i) {
            const int e = lane + 32 * i;
            if (e < dv) pg[e] = o[i];
        }
        if (lane == 0) { p.part_ml[2 * r] = m_run; p.part_ml[2 * r + 1] = l_run; }
        return;
    }
    const float sk = p.sink ? p.sink[head] : -INFINITY;
    const float M = fmaxf(m_run, sk);
    const float f = expf(m_run - M);
    const float inv = f / (l_run * f + expf(sk - M));
    T* og = reinterpret_cast<T*>(p.out) + (size_t)tok * p.out_stride + (size_t)head * dv;
#pragma unroll
    for (int i = 0; i < DPL; ++i) {
        const int e = lane + 32 * i;
        if (e < dv) {
            float r = o[i] * inv;
            if (p.gate != nullptr) r *= sigmoidf_(to_f32<T>(reinterpret_cast<const T*>(p.gate)[(size_t)tok * p.gate_stride + (size_t)head * dv + e]));
            og[e] = from_f32<T>(r);
        }
    }
}

// the pieces of a one-token step joined, in the order of the pieces: one block per token, a thread per output element
template <typename T>
__global__ void __launch_bounds__(128) sink_merge_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                                         const float* __restrict__ sink, T* __restrict__ out, long long out_stride,
                                                         int T_, int n_q, int dv, int splits, const T* __restrict__ gate,
                                                         long long gate_stride) {
    const int t = blockIdx.x, head = blockIdx.y;
    const size_t r0 = (size_t)t * n_q + head, step = (size_t)T_ * n_q;
    const float sk = sink ? sink[head] : -INFINITY;
    float M = sk;
    for (int s = 0; s < splits; ++s) M = fmaxf(M, part_ml[2 * (r0 + s * step)]);
    float den = expf(sk - M);
    for (int s = 0; s < splits; ++s) den = fmaf(part_ml[2 * (r0 + s * step) + 1], expf(part_ml[2 * (r0 + s * step)] - M), den);
    const float inv = 1.f / den;
    for (int e = threadIdx.x; e < dv; e += blockDim.x) {
        float acc = 0.f;
        for (int s = 0; s < splits; ++s) {
            const float f = expf(part_ml[2 * (r0 + s * step)] - M);
            if (f != 0.f) acc = fmaf(part_o[(r0 + s * step) * dv + e], f, acc);
        }
        acc *= inv;
        if (gate != nullptr) acc *= sigmoidf_(to_f32<T>(gate[(size_t)t * gate_stride + (size_t)head * dv + e]));
        out[(size_t)t * out_stride + (size_t)head * dv + e] = from_f32<T>(acc);
    }
}

MSGL_API int msgl_sink_attention(const void* q, const void* k_cache, const void* v_cache, const int* q_start, const int* kv_len,
                                 const int* block_table, int bt_stride, int uniform, int n_tiles, const float* sink, void* out,
                                 long long out_stride, float* part_o, float* part_ml, int splits, int split_keys, int T_, int B, int n_q,
                                 int n_kv, int d, int dv, int page_size, int QT, int GH, int window, float scale, float softcap, int dtype,
                                 const void* gate, long long gate_stride, int chunk_keys, cudaStream_t stream) {
    if (n_tiles <= 0) return MSGL_OK;
    if (d <= 0 || dv <= 0 || dv > 32 * SK_MAX_DPL || d > 32 * SK_MAX_DPL || n_kv <= 0 || n_q % n_kv || QT < 1 || GH < 1 ||
        QT * GH > SK_ROWS || page_size < 1 || window < 0 || chunk_keys < 0 || (window > 0 && chunk_keys > 0) || splits < 1 ||
        (splits > 1 && (!uniform || part_o == nullptr || part_ml == nullptr || split_keys < SK_KC || split_keys % SK_KC)))
        return MSGL_ERR_SIZE;
    if (dtype != MSGL_F32 && dtype != MSGL_BF16) return MSGL_ERR_DTYPE;
    SinkAttnParams p;
    p.q = q; p.k_cache = k_cache; p.v_cache = v_cache; p.q_start = q_start; p.kv_len = kv_len; p.block_table = block_table;
    p.bt_stride = bt_stride; p.uniform = uniform; p.sink = sink; p.out = out; p.out_stride = out_stride; p.part_o = part_o;
    p.part_ml = part_ml; p.splits = splits; p.split_keys = split_keys; p.T = T_; p.B = B; p.n_q = n_q; p.n_kv = n_kv; p.d = d; p.dv = dv;
    p.page_size = page_size; p.QT = QT; p.GH = GH; p.window = window; p.scale = scale; p.softcap = softcap;
    p.gate = gate; p.gate_stride = gate_stride; p.chunk_keys = chunk_keys;
    const int G = n_q / n_kv;
    const dim3 grid(n_tiles, n_kv * ((G + GH - 1) / GH), splits);
    const size_t smem = ((size_t)SK_ROWS * d + (size_t)SK_KC * (d + 1) + (size_t)SK_KC * dv) * sizeof(float);
    const int dpl = (dv + 31) / 32;
#define SK_LAUNCH(N)                                                                                                         \
    do {                                                                                                                     \
        static MsglOncePerDevice once;                                                                                       \
        if (smem > 48 * 1024 && once.due()) {                                                                                \
            cudaFuncSetAttribute(sink_attention_kernel<float, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);  \
            cudaFuncSetAttribute(sink_attention_kernel<__nv_bfloat16, N>, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024); \
            once.mark();                                                                                                     \
        }                                                                                                                    \
        if (dtype == MSGL_F32) sink_attention_kernel<float, N><<<grid, SK_ROWS * 32, smem, stream>>>(p);                     \
        else sink_attention_kernel<__nv_bfloat16, N><<<grid, SK_ROWS * 32, smem, stream>>>(p);                               \
    } while (0)
    if (dpl <= 1) SK_LAUNCH(1);
    else if (dpl <= 2) SK_LAUNCH(2);
    else if (dpl <= 4) SK_LAUNCH(4);
    else if (dpl <= 8) SK_LAUNCH(8);
    else SK_LAUNCH(16);
#undef SK_LAUNCH
    int code = msgl_check_launch();
    if (code != MSGL_OK || splits <= 1) return code;
    const dim3 g2(T_, n_q);
    if (dtype == MSGL_F32) sink_merge_kernel<float><<<g2, 128, 0, stream>>>(part_o, part_ml, sink, (float*)out, out_stride, T_, n_q, dv, splits, (const float*)gate, gate_stride);
    else sink_merge_kernel<__nv_bfloat16><<<g2, 128, 0, stream>>>(part_o, part_ml, sink, (__nv_bfloat16*)out, out_stride, T_, n_q, dv, splits, (const __nv_bfloat16*)gate, gate_stride);
    return msgl_check_launch();
}

// ---------------------------------------------------------------------------------------
// The same attention on the tensor cores (bfloat16): S = Q K^T and O += P V by mma.sync m16n8k16 with float32 accumulators;
// scores, cap, running maximum and sum in float32 between them, the weights rounded to bfloat16 only as the operand of the
// value product.  A block owns 64 rows = 64 / G tokens x the G query heads of one kv head (so a key tile serves all its
// heads) and walks the key tiles of 64 anchored at multiples of 64 from the one that holds the first key its first token
// sees, two tiles in flight (cp.async).  Cache rows before that key and after the last token are not read (zero in shared
// memory).  Exponentials are 2^x of scores in log2 units.  DK, DV: the head sizes rounded up to a size the kernel is built
// for; columns beyond d, dv are zero in shared memory.
// ---------------------------------------------------------------------------------------
namespace {
__device__ __forceinline__ unsigned smem_u32(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void cp_async16_u32(unsigned s, const void* gmem, bool valid) {
    const int n = valid ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(s), "l"(gmem), "r"(n));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }
__device__ __forceinline__ void ldmatrix_x4_u32(unsigned (&r)[4], unsigned s) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void ldmatrix_x4_trans_u32(unsigned (&r)[4], unsigned s) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(s));
}
__device__ __forceinline__ void mma_bf16_16816(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ unsigned pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<unsigned*>(&v);
}
__device__ __forceinline__ float ex2_(float x) {          // 2^x on the special-function unit (-inf gives 0)
    float e;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(e) : "f"(x));
    return e;
}
// tanh(x) = 1 - 2 / (e^2x + 1), to about 1e-6 absolutely
__device__ __forceinline__ float fast_tanh(float x) { return 1.f - __fdividef(2.f, ex2_(2.8853900817779268f * x) + 1.f); }
}  // namespace

#define SKM_R 64            // rows of a block
#define SKM_KT 64           // keys of a tile
#define SKM_THREADS 128
#define LOG2E_F 1.4426950408889634f
#define LN2_F 0.6931471805599453f

template <int DK, int DV>
__global__ void __launch_bounds__(SKM_THREADS) sink_attention_mma_kernel(const SinkAttnParams p) {
    constexpr int LDK = DK + 8, LDV = DV + 8;           // padded rows (elements): ldmatrix without bank conflicts
    constexpr int NKB = SKM_KT / 8, NDB = DV / 8;
    constexpr int CHK = DK / 8, CHV = DV / 8;           // 16-byte pieces of a row
    extern __shared__ __align__(16) unsigned char smem_raw[];
    __nv_bfloat16* Qs = reinterpret_cast<__nv_bfloat16*>(smem_raw);                 // [64][LDK]
    __nv_bfloat16* KVs = Qs + SKM_R * LDK;                                          // [stage][K: 64 x LDK | V: 64 x LDV]
    __shared__ int tile_sh[2];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int G = p.n_q / p.n_kv;
    const int Gc = G <= SKM_R ? G : SKM_R;
    const int n_chunks = G <= SKM_R ? 1 : (G + SKM_R - 1) / SKM_R;
    const int QT = G <= SKM_R ? SKM_R / G : 1;
    const int kvh = blockIdx.y / n_chunks, chunk = blockIdx.y - kvh * n_chunks;
    if (tid == 0) {
        if (p.uniform) {
            tile_sh[0] = blockIdx.x; tile_sh[1] = 0;
        } else {
            int left = (int)gridDim.x - 1 - (int)blockIdx.x, found = -1, at = 0;      // heaviest tiles first
            for (int r = 0; r < p.B; ++r) {
                const int nt = (p.q_start[r + 1] - p.q_start[r] + QT - 1) / QT;
                if (left < nt) { found = r; at = left * QT; break; }
                left -= nt;
            }
            tile_sh[0] = found; tile_sh[1] = at;
        }
    }
    __syncthreads();
    const int req = tile_sh[0], t0 = tile_sh[1];
    if (req < 0 || req >= p.B) return;
    const int q_base = p.q_start[req], q_len = p.q_start[req + 1] - q_base, kv_len = p.kv_len[req];
    const int n_tok = min(QT, q_len - t0);
    if (n_tok <= 0) return;
    const int p_min = kv_len - q_len + t0, p_max = p_min + n_tok - 1;
    const int key_lo = sk_first_key(p, p_min);      // the first key any row of the block sees
    int kt_lo = key_lo / SKM_KT, kt_hi = p_max / SKM_KT + 1;
    if (p.splits > 1) {       // a piece is a whole number of tiles, counted from the piece that holds key_lo
        const int piece = key_lo / p.split_keys + (int)blockIdx.z;
        kt_lo = max(kt_lo, piece * (p.split_keys / SKM_KT));
        kt_hi = min(kt_hi, (piece + 1) * (p.split_keys / SKM_KT));
    }
    const int d = p.d, dv = p.dv;
    const __nv_bfloat16* qg = reinterpret_cast<const __nv_bfloat16*>(p.q);
    const __nv_bfloat16* kc = reinterpret_cast<const __nv_bfloat16*>(p.k_cache);
    const __nv_bfloat16* vc = reinterpret_cast<const __nv_bfloat16*>(p.v_cache);
    const int* bt = p.block_table + (size_t)req * p.bt_stride;
    const unsigned q_s = smem_u32(Qs), kv_s = smem_u32(KVs);
    constexpr unsigned K_BYTES = SKM_KT * LDK * 2u, STAGE_BYTES = K_BYTES + SKM_KT * LDV * 2u;

    const int row_base = warp * 16;
    const int r_lo = row_base + (lane >> 2), r_hi = r_lo + 8;
    const int tl_lo = r_lo / Gc, tl_hi = r_hi / Gc;
    const int hl_lo = r_lo - tl_lo * Gc, hl_hi = r_hi - tl_hi * Gc;
    const int pos_lo = p_min + tl_lo, pos_hi = p_min + tl_hi;
    const int first_lo = sk_first_key(p, pos_lo), first_hi = sk_first_key(p, pos_hi);
    float o[NDB][4];
#pragma unroll
    for (int i = 0; i < NDB; ++i) { o[i][0] = o[i][1] = o[i][2] = o[i][3] = 0.f; }
    float m_run[2] = {-INFINITY, -INFINITY}, l_run[2] = {0.f, 0.f};       // log2 units; l: this thread's share of the row's sum

    if (kt_lo < kt_hi) {
        // ---- the block's query rows (zero where the tile has no token or head, and beyond d)
        for (int idx = tid; idx < SKM_R * CHK; idx += SKM_THREADS) {
            const int r = idx / CHK, c = idx - r * CHK;
            const int tl = r / Gc, hl = r - tl * Gc, hg = chunk * SKM_R + hl;
            const bool valid = tl < n_tok && tl < QT && hg < G && c * 8 < d;
            const size_t tok = (size_t)(q_base + t0 + (valid ? tl : 0));
            const __nv_bfloat16* src = qg + (tok * p.n_q + (size_t)kvh * G + (valid ? hg : 0)) * d + (valid ? c * 8 : 0);
            cp_async16_u32(q_s + (unsigned)(r * LDK + c * 8) * 2u, src, valid);
        }
        // a thread copies half a row of K and of V per tile: row tid / 2, every second 16-byte piece
        const int ld_row = tid >> 1, ld_half = tid & 1;
        auto load_kv = [&](int stage, int kt) {
            const int key = kt * SKM_KT + ld_row;
            const bool live = key <= p_max && key >= key_lo;
            size_t row = 0;
            if (live) row = ((size_t)bt[key / p.page_size] * p.n_kv + kvh) * p.page_size + (key % p.page_size);
            const unsigned ks = kv_s + (unsigned)stage * STAGE_BYTES + (unsigned)(ld_row * LDK) * 2u;
            const unsigned vs = kv_s + (unsigned)stage * STAGE_BYTES + K_BYTES + (unsigned)(ld_row * LDV) * 2u;
#pragma unroll
            for (int c = ld_half; c < CHK; c += 2) {
                const bool ok = live && c * 8 < d;
                cp_async16_u32(ks + c * 16, kc + row * d + (ok ? c * 8 : 0), ok);
            }
#pragma unroll
            for (int c = ld_half; c < CHV; c += 2) {
                const bool ok = live && c * 8 < dv;
                cp_async16_u32(vs + c * 16, vc + row * dv + (ok ? c * 8 : 0), ok);
            }
        };
        load_kv(0, kt_lo);
        cp_async_commit();

        const bool warp_live = row_base / Gc < n_tok;       // else all 16 rows of the warp are empty: it copies, but multiplies nothing
        const int warp_pos_lo = p_min + row_base / Gc, warp_pos_hi = p_min + (row_base + 15) / Gc;
        const int warp_first_lo = sk_first_key(p, warp_pos_lo), warp_first_hi = sk_first_key(p, warp_pos_hi);
        const unsigned q_a = q_s + (unsigned)((row_base + (lane & 15)) * LDK + (lane >> 4) * 8) * 2u;
        const unsigned k_lane = (unsigned)(((lane & 7) + ((lane >> 4) & 1) * 8) * LDK + ((lane >> 3) & 1) * 8) * 2u;
        const unsigned v_lane = (unsigned)(((lane & 7) + ((lane >> 3) & 1) * 8) * LDV + ((lane >> 4) & 1) * 8) * 2u;
        const float scale2 = p.scale * LOG2E_F;
        const float inv_cap = p.softcap > 0.f ? 1.f / p.softcap : 0.f, cap2 = p.softcap * LOG2E_F;

        for (int kt = kt_lo; kt < kt_hi; ++kt) {
            const int stage = (kt - kt_lo) & 1;
            if (kt + 1 < kt_hi) {
                load_kv(stage ^ 1, kt + 1);
                cp_async_commit();
                cp_async_wait<1>();
            } else {
                cp_async_wait<0>();
            }
            __syncthreads();
            const int key0 = kt * SKM_KT;
            // no row of the warp sees a key of this tile: the tile lies behind its last token or before its first token's first key
            if (!warp_live || key0 > warp_pos_hi || key0 + SKM_KT - 1 < warp_first_lo) {
                __syncthreads();
                continue;
            }
            const unsigned ks_a = kv_s + (unsigned)stage * STAGE_BYTES + k_lane;
            const unsigned vs_a = kv_s + (unsigned)stage * STAGE_BYTES + K_BYTES + v_lane;

            float s[NKB][4];
#pragma unroll
            for (int i = 0; i < NKB; ++i) { s[i][0] = s[i][1] = s[i][2] = s[i][3] = 0.f; }
#pragma unroll
            for (int kk = 0; kk < DK / 16; ++kk) {
                unsigned a[4];
                ldmatrix_x4_u32(a, q_a + kk * 32);
#pragma unroll
                for (int nb2 = 0; nb2 < NKB / 2; ++nb2) {
                    unsigned b[4];
                    ldmatrix_x4_u32(b, ks_a + (unsigned)(nb2 * 16 * LDK + kk * 16) * 2u);
                    mma_bf16_16816(s[2 * nb2], a, b[0], b[1]);
                    mma_bf16_16816(s[2 * nb2 + 1], a, b[2], b[3]);
                }
            }
            // ---- scores in log2 units, capped, masked; the tile's maximum per row
            const bool need_mask = key0 + SKM_KT - 1 > warp_pos_lo || key0 < warp_first_hi;
            float tmax[2] = {-INFINITY, -INFINITY};
#pragma unroll
            for (int nb = 0; nb < NKB; ++nb) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    float v = s[nb][e] * scale2;
                    if (p.softcap > 0.f) v = cap2 * fast_tanh(s[nb][e] * p.scale * inv_cap);
                    if (need_mask) {
                        const int key = key0 + nb * 8 + (lane & 3) * 2 + (e & 1);
                        const int pos = (e < 2) ? pos_lo : pos_hi, first = (e < 2) ? first_lo : first_hi;
                        if (key > pos || key < first) v = -INFINITY;
                    }
                    s[nb][e] = v;
                    tmax[e >> 1] = fmaxf(tmax[e >> 1], v);
                }
            }
            float corr[2], m_use[2];
#pragma unroll
            for (int hf = 0; hf < 2; ++hf) {
                float t = tmax[hf];
                t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 1));
                t = fmaxf(t, __shfl_xor_sync(0xffffffffu, t, 2));
                const float m_new = fmaxf(m_run[hf], t);
                m_use[hf] = m_new == -INFINITY ? 0.f : m_new;            // a row that has seen no key yet: all weights 0
                corr[hf] = ex2_(m_run[hf] - m_use[hf]);                  // m_run = -inf gives 0
                m_run[hf] = m_new;
                l_run[hf] *= corr[hf];
            }
#pragma unroll
            for (int nb = 0; nb < NKB; ++nb) {
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const float w = ex2_(s[nb][e] - m_use[e >> 1]);
                    s[nb][e] = w;
                    l_run[e >> 1] += w;
                }
            }
#pragma unroll
            for (int nd = 0; nd < NDB; ++nd) { o[nd][0] *= corr[0]; o[nd][1] *= corr[0]; o[nd][2] *= corr[1]; o[nd][3] *= corr[1]; }
            // ---- O += P V
#pragma unroll
            for (int j = 0; j < NKB / 2; ++j) {
                unsigned a[4];
                a[0] = pack_bf16(s[2 * j][0], s[2 * j][1]);
                a[1] = pack_bf16(s[2 * j][2], s[2 * j][3]);
                a[2] = pack_bf16(s[2 * j + 1][0], s[2 * j + 1][1]);
                a[3] = pack_bf16(s[2 * j + 1][2], s[2 * j + 1][3]);
#pragma unroll
                for (int nd2 = 0; nd2 < DV / 16; ++nd2) {
                    unsigned b[4];
                    ldmatrix_x4_trans_u32(b, vs_a + (unsigned)(j * 16 * LDV + nd2 * 16) * 2u);
                    mma_bf16_16816(o[2 * nd2], a, b[0], b[1]);
                    mma_bf16_16816(o[2 * nd2 + 1], a, b[2], b[3]);
                }
            }
            __syncthreads();
        }
        cp_async_wait<0>();
    }

    __nv_bfloat16* og = reinterpret_cast<__nv_bfloat16*>(p.out);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int tl = half ? tl_hi : tl_lo, hl = half ? hl_hi : hl_lo, hg = chunk * SKM_R + hl;
        float l = l_run[half];
        l += __shfl_xor_sync(0xffffffffu, l, 1);
        l += __shfl_xor_sync(0xffffffffu, l, 2);
        if (!(tl < n_tok && tl < QT && hg < G)) continue;
        const int head = kvh * G + hg;
        const size_t tok = (size_t)(q_base + t0 + tl);
        if (p.splits > 1) {
            const size_t r = ((size_t)blockIdx.z * p.T + tok) * p.n_q + head;
            float* pg = p.part_o + r * dv;
#pragma unroll
            for (int nd = 0; nd < NDB; ++nd) {
                const int col = nd * 8 + (lane & 3) * 2;
                if (col < dv) *reinterpret_cast<float2*>(pg + col) = make_float2(o[nd][half * 2], o[nd][half * 2 + 1]);
            }
            if ((lane & 3) == 0) { p.part_ml[2 * r] = m_run[half] * LN2_F; p.part_ml[2 * r + 1] = l; }
            continue;
        }
        const float sk2 = p.sink ? p.sink[head] * LOG2E_F : -INFINITY;
        const float M = fmaxf(m_run[half], sk2);
        const float f = ex2_(m_run[half] - M);
        const float inv = __fdividef(f, l * f + ex2_(sk2 - M));
        __nv_bfloat16* dst = og + tok * p.out_stride + (size_t)head * dv;
        const __nv_bfloat16* gt = p.gate ? reinterpret_cast<const __nv_bfloat16*>(p.gate) + tok * p.gate_stride + (size_t)head * dv : nullptr;
#pragma unroll
        for (int nd = 0; nd < NDB; ++nd) {
            const int col = nd * 8 + (lane & 3) * 2;
            if (col < dv) {         // dv is a multiple of 8: a pair lies inside the row or outside it
                float a = o[nd][half * 2] * inv, b = o[nd][half * 2 + 1] * inv;
                if (gt != nullptr) {
                    const float2 g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(gt + col));
                    a *= sigmoidf_(g.x); b *= sigmoidf_(g.y);
                }
                *reinterpret_cast<__nv_bfloat162*>(dst + col) = __floats2bfloat162_rn(a, b);
            }
        }
    }
}

// The tensor-core launch: bfloat16, head sizes that are multiples of 8 up to 128, rows of `out` that pairs of elements can be
// stored into.  n_tiles: the sum over the requests of ceil(tokens / QT) with QT = 64 / (heads per kv head) (1 beyond 64), or
// with `uniform` (every request brings one token) the number of requests; then `splits` pieces of `split_keys` keys (a
// multiple of 64) go to blocks of their own, which leave (max, sum, weighted values) for sink_merge_kernel.
MSGL_API int msgl_sink_attention_mma(const void* q, const void* k_cache, const void* v_cache, const int* q_start, const int* kv_len,
                                     const int* block_table, int bt_stride, int uniform, int n_tiles, const float* sink, void* out,
                                     long long out_stride, float* part_o, float* part_ml, int splits, int split_keys, int T_, int B, int n_q,
                                     int n_kv, int d, int dv, int page_size, int window, float scale, float softcap, const void* gate,
                                     long long gate_stride, int chunk_keys, cudaStream_t stream) {
    if (n_tiles <= 0) return MSGL_OK;
    if (d <= 0 || dv <= 0 || d > 128 || dv > 128 || d % 8 || dv % 8 || n_kv <= 0 || n_q % n_kv || page_size < 1 ||
        window < 0 || chunk_keys < 0 || (window > 0 && chunk_keys > 0) || (out_stride & 1) || ((size_t)out & 3) || (gate_stride & 1) || ((size_t)gate & 3) || splits < 1 ||
        (splits > 1 && (!uniform || part_o == nullptr || part_ml == nullptr || split_keys < SKM_KT || split_keys % SKM_KT || ((size_t)part_o & 7))))
        return MSGL_ERR_SIZE;
    SinkAttnParams p;
    p.q = q; p.k_cache = k_cache; p.v_cache = v_cache; p.q_start = q_start; p.kv_len = kv_len; p.block_table = block_table;
    p.bt_stride = bt_stride; p.uniform = uniform; p.sink = sink; p.out = out; p.out_stride = out_stride; p.part_o = part_o;
    p.part_ml = part_ml; p.splits = splits; p.split_keys = split_keys; p.T = T_; p.B = B; p.n_q = n_q; p.n_kv = n_kv; p.d = d; p.dv = dv;
    p.page_size = page_size; p.QT = 0; p.GH = 0; p.window = window; p.scale = scale; p.softcap = softcap;
    p.gate = gate; p.gate_stride = gate_stride; p.chunk_keys = chunk_keys;
    const int G = n_q / n_kv;
    const dim3 grid(n_tiles, n_kv * (G <= SKM_R ? 1 : (G + SKM_R - 1) / SKM_R), splits);
#define SKM_LAUNCH(DK, DV)                                                                                                   \
    do {                                                                                                                     \
        const size_t smem = ((size_t)SKM_R * (DK + 8) + 2 * ((size_t)SKM_KT * (DK + 8) + (size_t)SKM_KT * (DV + 8))) * 2;    \
        static MsglOncePerDevice once;                                                                                       \
        if (once.due()) {                                                                                                    \
            cudaFuncSetAttribute(sink_attention_mma_kernel<DK, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
            once.mark();                                                                                                     \
        }                                                                                                                    \
        sink_attention_mma_kernel<DK, DV><<<grid, SKM_THREADS, smem, stream>>>(p);                                           \
    } while (0)
#define SKM_BY_DV(DK)                                                                                                        \
    do {                                                                                                                     \
        if (dv <= 64) SKM_LAUNCH(DK, 64);                                                                                    \
        else if (dv <= 96) SKM_LAUNCH(DK, 96);                                                                               \
        else SKM_LAUNCH(DK, 128);                                                                                            \
    } while (0)
    if (d <= 64) SKM_BY_DV(64);
    else if (d <= 96) SKM_BY_DV(96);
    else SKM_BY_DV(128);
#undef SKM_BY_DV
#undef SKM_LAUNCH
    int code = msgl_check_launch();
    if (code != MSGL_OK || splits <= 1) return code;
    const dim3 g2(T_, n_q);
    sink_merge_kernel<__nv_bfloat16><<<g2, 128, 0, stream>>>(part_o, part_ml, sink, (__nv_bfloat16*)out, out_stride, T_, n_q, dv, splits, (const __nv_bfloat16*)gate, gate_stride);
    return msgl_check_launch();
}

// ---------------------------------------------------------------------------------------
// The gated delta rule, token by token
//
//   per head h (q/k head g = h / (heads / kv_heads)), state S [d][dv] float32 per request, per token t:
//     qn = q / sqrt(sum q^2 + 1e-6) * d^-1/2,  kn = k / sqrt(sum k^2 + 1e-6)
//     beta = sigmoid(pb[t, h]);  g = exp(-exp(A_log[h]) * softplus(pa[t, h] + dt_bias[h]))
//     S <- g S;  u = beta (v - S^T kn);  S <- S + kn u^T;  o[t, h, :] = S^T qn
//   qkv row [T][kv_heads * d | kv_heads * d | heads * dv] (what the convolution left); pa, pb column ranges of the packed
//   projection.
// delta_prep_kernel makes what does not depend on the state, all tokens side by side: (kn, qn) pairs [T][kv_heads][d] and
// (beta, g, kn . qn) [T][heads], float32.  delta_rule_kernel then walks a request's tokens in order.  The columns of a state
// do not meet: a warp owns DR_WCOLS columns of one (request, head) state, DR_PARTS lanes share a column's rows (each keeps its
// RPT rows in registers), and a token costs the warp two shuffle rounds and no barrier.  Both products with the old state are
// taken in one pass, A = S^T kn and Q = S^T qn, and o = g Q + (kn . qn) u.  The tokens go through shared memory in batches
// of DR_TB, the next batch on its way (cp.async; the block's columns of v through registers) while the current one is walked:
// a barrier a batch.  Few columns in all (one request's prompt): blocks of DR_FEW_WARPS warps, so that more SMs take part;
// else DR_MANY_WARPS.
// ---------------------------------------------------------------------------------------
#define DR_WCOLS 4
#define DR_PARTS 8
#ifndef DR_TB
#define DR_TB 16
#endif
#ifndef DR_FEW_WARPS
#define DR_FEW_WARPS 4
#endif
#ifndef DR_MANY_WARPS
#define DR_MANY_WARPS 8
#endif

struct DeltaParams {
    const void* qkv; const void* proj; long long proj_stride; int a_off, b_off;
    const float* a_log; const float* dt_bias;
    float2* kq; float4* sc;                      // what delta_prep_kernel leaves
    float* state; const int* q_start; const int* slots; float* out;
    int heads, kv_heads, d, dv, T;
    int n_min, n_max;                            // the requests that a launch takes: those with n_min <= tokens <= n_max
};

template <typename T>
__global__ void __launch_bounds__(128) delta_prep_kernel(const DeltaParams p) {
    pdl_wait();
    pdl_small();
    const int t = blockIdx.x, lane = threadIdx.x & 31;
    const int g = blockIdx.y * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (g >= p.kv_heads) return;
    const int d = p.d, Ck = p.kv_heads * d, W = 2 * Ck + p.heads * p.dv;
    const T* rowp = reinterpret_cast<const T*>(p.qkv) + (size_t)t * W;
    float sq = 0.f, sk = 0.f;
    for (int e = lane; e < d; e += 32) {
        const float qe = to_f32<T>(rowp[(size_t)g * d + e]), ke = to_f32<T>(rowp[Ck + (size_t)g * d + e]);
        sq = fmaf(qe, qe, sq); sk = fmaf(ke, ke, sk);
    }
    sq = warp_sum(sq); sk = warp_sum(sk);
    const float rq = (1.f / sqrtf((float)d)) / sqrtf(sq + 1e-6f), rk = 1.f / sqrtf(sk + 1e-6f);
    float2* dst = p.kq + ((size_t)t * p.kv_heads + g) * d;
    float dot = 0.f;
    for (int e = lane; e < d; e += 32) {
        const float qe = to_f32<T>(rowp[(size_t)g * d + e]) * rq, ke = to_f32<T>(rowp[Ck + (size_t)g * d + e]) * rk;
        dst[e] = make_float2(ke, qe);
        dot = fmaf(ke, qe, dot);
    }
    dot = warp_sum(dot);
    const int per = p.heads / p.kv_heads;
    const T* proj = reinterpret_cast<const T*>(p.proj) + (size_t)t * p.proj_stride;
    for (int i = lane; i < per; i += 32) {
        const int h = g * per + i;
        const float pa = to_f32<T>(proj[p.a_off + h]), pb = to_f32<T>(proj[p.b_off + h]);
        p.sc[(size_t)t * p.heads + h] = make_float4(sigmoidf_(pb), expf(-expf(p.a_log[h]) * softplusf_(pa + p.dt_bias[h])), dot, 0.f);
    }
}

namespace {
__device__ __forceinline__ void cp_async8_(void* smem_dst, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)), "l"(gmem));
}
__device__ __forceinline__ void cp_async16_(void* smem_dst, const void* gmem) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"((unsigned)__cvta_generic_to_shared(smem_dst)), "l"(gmem));
}
}  // namespace

template <typename T, int RPT, bool EXACT /* d == RPT * DR_PARTS: no row of a thread lies beyond the state */>
__global__ void __launch_bounds__(DR_MANY_WARPS * 32) delta_rule_kernel(const DeltaParams p) {
    pdl_wait();
    pdl_small();
    extern __shared__ __align__(16) unsigned char dr_smem[];
    const int d = p.d, dv = p.dv;
    const int warps = blockDim.x >> 5, cols = warps * DR_WCOLS;
    constexpr int VPT = DR_TB * DR_WCOLS / 32;                          // values of v a thread brings per batch
    // per stage: sc [DR_TB] float4 | kq [DR_TB][d] float2 | v [DR_TB][cols] float
    const size_t stage_bytes = (size_t)DR_TB * 16 + (size_t)DR_TB * d * 8 + (size_t)DR_TB * cols * 4;
    const int h = blockIdx.x, r = blockIdx.y, c0 = blockIdx.z * cols;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int part = lane / DR_WCOLS, wc = lane % DR_WCOLS;             // lanes of a part read neighbouring columns
    const int g = h / (p.heads / p.kv_heads);
    const int t0 = p.q_start[r], n = p.q_start[r + 1] - t0;
    if (n < p.n_min || n > p.n_max) return;
    const int lcol = warp * DR_WCOLS + wc, col = c0 + lcol;
    const bool col_ok = col < dv;
    const int Ck = p.kv_heads * d, W = 2 * Ck + p.heads * dv;
    float* S = p.state + ((size_t)p.slots[r] * p.heads + h) * d * dv;
    float s_reg[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = part + DR_PARTS * i;
        s_reg[i] = ((EXACT || row < d) && col_ok) ? S[(size_t)row * dv + col] : 0.f;
    }
    const T* qkv = reinterpret_cast<const T*>(p.qkv);
    auto stage_sc = [&](int st) { return reinterpret_cast<float4*>(dr_smem + st * stage_bytes); };
    auto stage_kq = [&](int st) { return reinterpret_cast<float2*>(dr_smem + st * stage_bytes + DR_TB * 16); };
    auto stage_v = [&](int st) { return reinterpret_cast<float*>(dr_smem + st * stage_bytes + DR_TB * 16 + (size_t)DR_TB * d * 8); };
    auto issue = [&](int st, int b0) {           // the batch's (kn, qn) and (beta, g, kn . qn) on their way into a stage
        const int nb = min(DR_TB, n - b0);
        float2* kq = stage_kq(st);
        for (int j = 0; j < nb; ++j) {
            const float2* src = p.kq + ((size_t)(t0 + b0 + j) * p.kv_heads + g) * d;
            for (int e = tid; e < d; e += blockDim.x) cp_async8_(kq + j * d + e, src + e);
        }
        if (tid < nb) cp_async16_(stage_sc(st) + tid, p.sc + (size_t)(t0 + b0 + tid) * p.heads + h);
        asm volatile("cp.async.commit_group;\n" ::);
    };
    float vreg[VPT];
    const int vj = tid / cols, vc = tid - vj * cols, vstep = blockDim.x / cols;      // VPT * vstep = DR_TB
    auto load_v = [&](int b0) {                  // this block's columns of the batch's v into registers
        const int nb = min(DR_TB, n - b0);
#pragma unroll
        for (int k = 0; k < VPT; ++k) {
            const int j = vj + k * vstep;
            vreg[k] = (j < nb && c0 + vc < dv) ? to_f32<T>(qkv[(size_t)(t0 + b0 + j) * W + 2 * Ck + (size_t)h * dv + c0 + vc]) : 0.f;
        }
    };
    issue(0, 0);
    load_v(0);
    for (int b0 = 0, st = 0; b0 < n; b0 += DR_TB, st ^= 1) {
        const int nb = min(DR_TB, n - b0);
        float* vv = stage_v(st);
#pragma unroll
        for (int k = 0; k < VPT; ++k) vv[(vj + k * vstep) * cols + vc] = vreg[k];
        asm volatile("cp.async.wait_group 0;\n" ::);
        __syncthreads();                         // the batch lies in its stage; the other stage is no longer read
        if (b0 + DR_TB < n) {
            issue(st ^ 1, b0 + DR_TB);
            load_v(b0 + DR_TB);
        }
        const float2* kq = stage_kq(st) + part;
        const float4* sc = stage_sc(st);
        for (int j = 0; j < nb; ++j) {
            const float2* kqj = kq + j * d;
            float2 kr[RPT];                      // the thread's rows of (kn, qn): read once, used by both passes
            float A0 = 0.f, A1 = 0.f, Q0 = 0.f, Q1 = 0.f;
#pragma unroll
            for (int i = 0; i < RPT; ++i) {
                kr[i] = (EXACT || part + DR_PARTS * i < d) ? kqj[DR_PARTS * i] : make_float2(0.f, 0.f);
                if (i & 1) { A1 = fmaf(s_reg[i], kr[i].x, A1); Q1 = fmaf(s_reg[i], kr[i].y, Q1); }
                else { A0 = fmaf(s_reg[i], kr[i].x, A0); Q0 = fmaf(s_reg[i], kr[i].y, Q0); }
            }
            float A = A0 + A1, Q = Q0 + Q1;
#pragma unroll
            for (int o = DR_WCOLS; o < 32; o <<= 1) {
                A += __shfl_xor_sync(0xffffffffu, A, o);
                Q += __shfl_xor_sync(0xffffffffu, Q, o);
            }
            const float4 c4 = sc[j];             // beta, g, kn . qn
            const float u = c4.x * (vv[j * cols + lcol] - c4.y * A);
#pragma unroll
            for (int i = 0; i < RPT; ++i) s_reg[i] = fmaf(kr[i].x, u, c4.y * s_reg[i]);
            if (part == 0 && col_ok) p.out[((size_t)(t0 + b0 + j) * p.heads + h) * dv + col] = fmaf(c4.z, u, c4.y * Q);
        }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = part + DR_PARTS * i;
        if ((EXACT || row < d) && col_ok) S[(size_t)row * dv + col] = s_reg[i];
    }
}

// ---------------------------------------------------------------------------------------
// The same recurrence for a run of tokens in chunks of DC_C.  With the chunk's start state S0, its decays multiplied up, P_t = g_1 ... g_t and
// D_ts = g_(s+1) ... g_t:
//     x_t = beta_t (v_t - P_t S0^T k_t),     u_t + sum_{s < t} beta_t D_ts (k_t . k_s) u_s = x_t,     that is u = R x with R = (1 + L)^-1
//     o_t = P_t S0^T q_t + sum_{s <= t} D_ts (q_t . k_s) u_s = P_t S0^T q_t + (M R x)_t
//     S <- P_C S0 + sum_s D_Cs k_s u_s^T
// R and M R [C][C] and the factors of a token do not read the state: delta_chunk_kernel makes them for all chunks side by side.
// delta_chunk_scan_kernel walks a request's chunks in order with 16 columns of one state a block: S0^T k and S0^T q, then x, u and the new state.
// The decays are products of the g themselves, not differences of sums of logarithms, which would lose digits where they are small.
//
// Token by token the walk is a chain (a product with the state, two rounds of shuffles, the update) of 0.37 us a token whatever the number of
// SMs.  32 tokens: a row of the weights is a warp's width, and two blocks of the walk fit an SM.
//
// The walk's products go to the tensor cores, every float32 operand as the sum of three bfloat16 parts, which hold all of its 24 bits.  Keys and queries
// of bfloat16 activations need no parts: their rows go in as they came (one part, exactly) and the factors that make them unit vectors go to the other
// operand or the sum, as in the Gram products of the first kernel; float32 activations come as three parts of the unit rows.
// What the first kernel leaves is laid out chunk by chunk, rows at the pitch that the walk's shared memory has, tokens behind the request's
// last one as zeros: a stage of the walk is a straight copy.
// ---------------------------------------------------------------------------------------
constexpr int DC_C = 32, DC_COLS = 16, DC_THREADS = 256;
constexpr int DC_LDM = DC_C + 4;                 // pitch of the rows of R, M R and x
template <typename T, int D> struct DcSizes {
    static constexpr int PARTS = sizeof(T) == 2 ? 1 : 3;         // bfloat16 parts of a key or query row
    static constexpr int LDK = D + 8;            // pitch of such a row: ldmatrix's eight rows fall on different banks
    static constexpr int KQ = PARTS * DC_C * LDK * 2, M = DC_C * DC_LDM * 4;         // bytes of a chunk's keys (queries) and of R (M R)
};

struct DeltaChunkParams {
    const void* qkv; const void* proj; long long proj_stride; int a_off, b_off;
    const float* a_log; const float* dt_bias;
    unsigned char* K; unsigned char* Q;          // [chunk][kv_heads]: keys, queries [PARTS][C][LDK] bfloat16
    // [chunk][heads]: R, M R [C][LDM] float32, zeros behind the diagonal.  Behind row t of R: beta_t, beta_t P_t |k_t|^-1, D_Ct |k_t|^-1, P_t |q_t|^-1 d^-1/2 (the
    // norms of rows that are not unit rows yet); behind the first row of M R: P of the chunk's last token
    unsigned char* R; unsigned char* M;
    float* state; const int* q_start; const int* slots; float* out;
    int* status;                                 // word 1: a copy did not arrive
    int heads, kv_heads, dv, B, n_min, n_chunks;
};

namespace {
__device__ __forceinline__ void dc_ldmatrix4(unsigned (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void dc_ldmatrix4t(unsigned (&r)[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"((unsigned)__cvta_generic_to_shared(p)) : "memory");
}
__device__ __forceinline__ void dc_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// the next bfloat16 part of two floats, taken off them: cut off or (ROUND) rounded; three parts hold all 24 bits either way, rounded ones fall off faster
template <bool ROUND> __device__ __forceinline__ unsigned dc_part(float& x, float& y) {
    if (!ROUND) {
        const unsigned a = __float_as_uint(x), b = __float_as_uint(y);
        x -= __uint_as_float(a & 0xffff0000u); y -= __uint_as_float(b & 0xffff0000u);
        return __byte_perm(a, b, 0x7632);
    }
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const unsigned u = *reinterpret_cast<const unsigned*>(&h);
    x -= __uint_as_float(u << 16); y -= __uint_as_float(u & 0xffff0000u);
    return u;
}
// 8 elements of a row
__device__ __forceinline__ void dc_load8(const float* p, float* o) {
    const float4 a = *reinterpret_cast<const float4*>(p), b = *reinterpret_cast<const float4*>(p + 4);
    o[0] = a.x; o[1] = a.y; o[2] = a.z; o[3] = a.w; o[4] = b.x; o[5] = b.y; o[6] = b.z; o[7] = b.w;
}
__device__ __forceinline__ void dc_load8(const __nv_bfloat16* p, float* o) {
    const uint4 v = *reinterpret_cast<const uint4*>(p);
    const unsigned u[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
    for (int i = 0; i < 4; ++i) { o[2 * i] = __uint_as_float(u[i] << 16); o[2 * i + 1] = __uint_as_float(u[i] & 0xffff0000u); }
}
__device__ __forceinline__ float4 dc_load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 dc_load4(const __nv_bfloat16* p) {
    const uint2 v = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(v.x << 16), __uint_as_float(v.x & 0xffff0000u), __uint_as_float(v.y << 16), __uint_as_float(v.y & 0xffff0000u));
}
// the request and the place in it of the `left`-th chunk of the requests with n_min tokens or more (one warp); at < 0: there is none
__device__ __forceinline__ void dc_find(const int* q_start, int B, int n_min, int left, int& at, int& rest) {
    const int lane = threadIdx.x & 31;
    at = -1; rest = 0;
    for (int r0 = 0; r0 < B && at < 0; r0 += 32) {
        const int r = r0 + lane;
        const int n = r < B ? q_start[r + 1] - q_start[r] : 0;
        const int c = n >= n_min ? (n + DC_C - 1) / DC_C : 0;
        int sum = c;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
        const unsigned hit = __ballot_sync(0xffffffffu, left < sum);
        if (hit) {
            const int l = __ffs(hit) - 1;
            at = r0 + l;
            rest = left - __shfl_sync(0xffffffffu, sum - c, l);
        }
        left -= __shfl_sync(0xffffffffu, sum, 31);
    }
}
// the `nth` request with n_min tokens or more and the chunks of those before it (one warp); at < 0: there is none
__device__ __forceinline__ void dc_nth(const int* q_start, int B, int n_min, int nth, int& at, int& before) {
    const int lane = threadIdx.x & 31;
    int sum = 0;
    at = -1;
    for (int r0 = 0; r0 < B && at < 0; r0 += 32) {
        const int r = r0 + lane;
        const int n = r < B ? q_start[r + 1] - q_start[r] : 0;
        const unsigned hits = __ballot_sync(0xffffffffu, n >= n_min);
        const unsigned own = __ballot_sync(0xffffffffu, n >= n_min && __popc(hits & ((1u << lane) - 1u)) == nth);
        if (own) at = r0 + __ffs(own) - 1;
        else nth -= __popc(hits);
        if (n >= n_min && (at < 0 || r < at)) sum += (n + DC_C - 1) / DC_C;
    }
    before = __reduce_add_sync(0xffffffffu, sum);
}
}  // namespace

template <typename T, int D> struct DcPrep {     // shared memory of delta_chunk_kernel, in bytes
    using Z = DcSizes<T, D>;
    static constexpr int LDF = D + 4;            // pitch of float32 rows: 16 bytes apart in the banks
    static constexpr int KS = 0, QS = KS + (Z::PARTS == 1 ? DC_C * Z::LDK * 2 : DC_C * LDF * 4), KK = 2 * QS, QK = KK + DC_C * (DC_C + 1) * 4,
                         LS = QK + DC_C * (DC_C + 1) * 4, RS = LS + DC_C * DC_LDM * 4, TMP = RS + DC_C * DC_LDM * 4, TOTAL = TMP + 16 * 17 * 4;
};

// A block makes one head's chunk.  Latency decides, so several blocks share an SM.  R by halves: its two diagonal blocks of 16 rows by substitution, a lane a column of
// one of them, then R_21 = -R_22 L_21 R_11.  1,411 tokens of 16 heads: 15 us; with unit rows from a launch ahead (7.5 us), Gram products in multiply-adds and a
// substitution of all of beta v and beta P K (256 columns a head) it took 43.
// A sum takes rows of tokens up to its own only: a later token's row may be no number, and 0 times that is none either.  (What stands behind the diagonal of a row
// belongs to that row's token or earlier ones, and nobody reads it.)
template <typename T, int D>
__global__ void __launch_bounds__(DC_THREADS, 4) delta_chunk_kernel(const DeltaChunkParams p) {
    using Z = DcSizes<T, D>;
    using Sm = DcPrep<T, D>;
    constexpr int LDK = Z::LDK, LDF = Sm::LDF;
    constexpr bool RAW = Z::PARTS == 1;
    static_assert(D == 128 && DC_C == 32, "eight threads a row, two halves of 16");
    extern __shared__ __align__(16) unsigned char dc_smem[];
    float* Ks = reinterpret_cast<float*>(dc_smem + Sm::KS);              // float32: [C][LDF] unit keys, queries
    float* Qs = reinterpret_cast<float*>(dc_smem + Sm::QS);
    __nv_bfloat16* Kr = reinterpret_cast<__nv_bfloat16*>(dc_smem + Sm::KS);      // bfloat16: [2 C][LDK] rows as they came, keys then queries
    float* KK = reinterpret_cast<float*>(dc_smem + Sm::KK);              // [C][C + 1]
    float* QK = reinterpret_cast<float*>(dc_smem + Sm::QK);              // then M, in place
    float* Ls = reinterpret_cast<float*>(dc_smem + Sm::LS);              // [C][LDM]
    float* Rs = reinterpret_cast<float*>(dc_smem + Sm::RS);              // [C][LDM]
    float* tmp = reinterpret_cast<float*>(dc_smem + Sm::TMP);            // [16][17]
    __shared__ float beta_s[DC_C], g_s[DC_C], pre_s[DC_C], suf_s[DC_C], rk_s[DC_C], rq_s[DC_C];
    __shared__ int where_s[2];
    pdl_wait();
    pdl_small();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, h = blockIdx.y, per = p.heads / p.kv_heads, g = h / per;
    if (warp == 0) {
        int at, rest;
        dc_find(p.q_start, p.B, p.n_min, blockIdx.x, at, rest);
        if (lane == 0) { where_s[0] = at; where_s[1] = rest; }
    }
    __syncthreads();
    if (where_s[0] < 0) return;
    const int r = where_s[0], base = p.q_start[r] + where_s[1] * DC_C, nb = min(DC_C, p.q_start[r + 1] - base);
    const bool first = h == g * per;             // this head's block leaves keys and queries for the walk
    const int Ck = p.kv_heads * D, Wd = 2 * Ck + p.heads * p.dv;
    const T* qkv = reinterpret_cast<const T*>(p.qkv) + (size_t)base * Wd;
    const size_t chunk_h = (size_t)blockIdx.x * p.heads + h, chunk_g = (size_t)blockIdx.x * p.kv_heads + g;
    {   // a row's eight threads take elements 8 j .. and 64 + 8 j ..
        const int t = tid >> 3, j = tid & 7;
        float k[16] = {}, q[16] = {};
        if (t < nb) {
            const T* rowq = qkv + (size_t)t * Wd + (size_t)g * D + 8 * j;
            dc_load8(rowq, q); dc_load8(rowq + 64, q + 8); dc_load8(rowq + Ck, k); dc_load8(rowq + Ck + 64, k + 8);
        }
        if (tid < DC_C) {
            float beta = 0.f, gt = 1.f;
            if (tid < nb) {
                const T* proj = reinterpret_cast<const T*>(p.proj) + (size_t)(base + tid) * p.proj_stride;
                beta = sigmoidf_(to_f32<T>(proj[p.b_off + h]));
                gt = expf(-expf(p.a_log[h]) * softplusf_(to_f32<T>(proj[p.a_off + h]) + p.dt_bias[h]));
            }
            beta_s[tid] = beta; g_s[tid] = gt;
        }
        float sq = 0.f, sk = 0.f;
#pragma unroll
        for (int i = 0; i < 16; ++i) { sq = fmaf(q[i], q[i], sq); sk = fmaf(k[i], k[i], sk); }
#pragma unroll
        for (int o = 4; o > 0; o >>= 1) { sq += __shfl_xor_sync(0xffffffffu, sq, o); sk += __shfl_xor_sync(0xffffffffu, sk, o); }
        const float rq = (1.f / sqrtf((float)D)) / sqrtf(sq + 1e-6f), rk = 1.f / sqrtf(sk + 1e-6f);
        if (j == 0) { rk_s[t] = rk; rq_s[t] = rq; }
        unsigned char* kq[2] = {p.K + chunk_g * Z::KQ, p.Q + chunk_g * Z::KQ};
#pragma unroll
        for (int which = 0; which < 2; ++which) {
            float* v = which ? q : k;
            const float unit = which ? rq : rk;
            if (!RAW || unit == 0.f) {           // a norm beyond float32: zeros either way (an infinity: not a number)
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] *= unit;
            }
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int e = 64 * half + 8 * j;
                if (!RAW) {
                    float* dst = (which ? Qs : Ks) + t * LDF + e;
                    *reinterpret_cast<float4*>(dst) = make_float4(v[8 * half], v[8 * half + 1], v[8 * half + 2], v[8 * half + 3]);
                    *reinterpret_cast<float4*>(dst + 4) = make_float4(v[8 * half + 4], v[8 * half + 5], v[8 * half + 6], v[8 * half + 7]);
                }
#pragma unroll
                for (int part = 0; part < Z::PARTS; ++part) {
                    unsigned u[4];
#pragma unroll
                    for (int i = 0; i < 4; ++i) u[i] = dc_part<true>(v[8 * half + 2 * i], v[8 * half + 2 * i + 1]);
                    const uint4 w = make_uint4(u[0], u[1], u[2], u[3]);
                    if (RAW) *reinterpret_cast<uint4*>(Kr + (which * DC_C + t) * LDK + e) = w;
                    if (first) *reinterpret_cast<uint4*>(kq[which] + ((part * DC_C + t) * LDK + e) * 2) = w;
                }
            }
        }
    }
    __syncthreads();
    if constexpr (RAW) {                         // warp: 16 rows (of k or q) against 16 keys
        float acc[4][2][4] = {};                 // four sums each: less rounding than one over all of D
        const int m0 = (warp >> 1) * 16, n0 = (warp & 1) * 16;
        const __nv_bfloat16* ap = Kr + (m0 + (lane & 15)) * LDK + (lane >> 4) * 8;
        const __nv_bfloat16* bp = Kr + (n0 + (lane & 7) + (lane >> 4) * 8) * LDK + ((lane >> 3) & 1) * 8;
#pragma unroll
        for (int e = 0; e < D; e += 16) {
            unsigned a[4], b[4];
            dc_ldmatrix4(a, ap + e);
            dc_ldmatrix4(b, bp + e);
            dc_mma(acc[e / 16 % 4][0], a, b[0], b[1]);
            dc_mma(acc[e / 16 % 4][1], a, b[2], b[3]);
        }
        float* dst = warp < 4 ? KK : QK;
        const float* rr = warp < 4 ? rk_s : rq_s;
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int row = (m0 & 16) + (lane >> 2) + ((i >> 1) & 1) * 8, col = n0 + (i >> 2) * 8 + (lane & 3) * 2 + (i & 1);
            const float sum = (acc[0][i >> 2][i & 3] + acc[1][i >> 2][i & 3]) + (acc[2][i >> 2][i & 3] + acc[3][i >> 2][i & 3]);
            dst[row * (DC_C + 1) + col] = sum * rr[row] * rk_s[col];
        }
    } else {
        // k_t . k_s and q_t . k_s: rows ti, ti + 16 against columns tj, tj + 16
        const int ti = tid >> 4, tj = tid & 15;
        float kk[2][2][4] = {}, qk[2][2][4] = {};            // four partial sums each: less rounding than one over all of D
#pragma unroll 1
        for (int e = 0; e < D; e += 4) {
            float4 kt[2], qt[2], ks[2];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                kt[i] = *reinterpret_cast<const float4*>(Ks + (ti + 16 * i) * LDF + e);
                qt[i] = *reinterpret_cast<const float4*>(Qs + (ti + 16 * i) * LDF + e);
                ks[i] = *reinterpret_cast<const float4*>(Ks + (tj + 16 * i) * LDF + e);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    kk[i][j][0] = fmaf(kt[i].x, ks[j].x, kk[i][j][0]); kk[i][j][1] = fmaf(kt[i].y, ks[j].y, kk[i][j][1]);
                    kk[i][j][2] = fmaf(kt[i].z, ks[j].z, kk[i][j][2]); kk[i][j][3] = fmaf(kt[i].w, ks[j].w, kk[i][j][3]);
                    qk[i][j][0] = fmaf(qt[i].x, ks[j].x, qk[i][j][0]); qk[i][j][1] = fmaf(qt[i].y, ks[j].y, qk[i][j][1]);
                    qk[i][j][2] = fmaf(qt[i].z, ks[j].z, qk[i][j][2]); qk[i][j][3] = fmaf(qt[i].w, ks[j].w, qk[i][j][3]);
                }
        }
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int at = (ti + 16 * i) * (DC_C + 1) + tj + 16 * j;
                KK[at] = (kk[i][j][0] + kk[i][j][1]) + (kk[i][j][2] + kk[i][j][3]);
                QK[at] = (qk[i][j][0] + qk[i][j][1]) + (qk[i][j][2] + qk[i][j][3]);
            }
    }
    __syncthreads();
    {   // column s = lane: the decays from s on; a warp takes four rows
        const int s = lane, t_first = 4 * warp;
        float run = 1.f;
        for (int t = 1; t < t_first; ++t) run *= t > s ? g_s[t] : 1.f;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int t = t_first + i, at = t * (DC_C + 1) + s;
            if (t > s) run *= g_s[t];
            Ls[t * DC_LDM + s] = t > s ? beta_s[t] * run * KK[at] : 0.f;
            QK[at] = t >= s ? run * QK[at] : 0.f;
            if (s == 0) pre_s[t] = g_s[0] * run;
            if (t == nb - 1) suf_s[s] = run;
        }
    }
    __syncthreads();
    if (warp == 0) {                             // R_11 and R_22: half-warp b, column j of the block at b0; rows one after the other
        const int b0 = lane & 16, j = lane & 15;
        float x[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            float a = i == j ? 1.f : 0.f, a1 = 0.f;
#pragma unroll
            for (int s = 0; s < i; ++s) {
                const float l = Ls[(b0 + i) * DC_LDM + b0 + s];
                if (s & 1) a1 = fmaf(-l, x[s], a1); else a = fmaf(-l, x[s], a);
            }
            x[i] = a + a1;
            Rs[(b0 + i) * DC_LDM + b0 + j] = x[i];
        }
    } else if (warp == 1) {                      // the factors of the tokens
        const int t = lane;
        const float rk = RAW ? rk_s[t] : 1.f, rq = RAW ? rq_s[t] : 1.f, beta = beta_s[t];
        const bool in = t < nb;
        *reinterpret_cast<float4*>(p.R + chunk_h * Z::M + (t * DC_LDM + DC_C) * 4) =
            in ? make_float4(beta, beta * pre_s[t] * rk, suf_s[t] * rk, pre_s[t] * rq) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (t == 0) *reinterpret_cast<float*>(p.M + chunk_h * Z::M + DC_C * 4) = pre_s[nb - 1];
    } else if (tid >= 128) {
        const int i = (tid - 128) >> 3, j = (tid & 7) * 2;                   // R_12 = 0
        *reinterpret_cast<float2*>(Rs + i * DC_LDM + 16 + j) = make_float2(0.f, 0.f);
    }
    __syncthreads();
    const int ri = tid >> 4, rj = tid & 15;
    {   // L_21 R_11 (columns of R_11 begin at its diagonal)
        float a = 0.f, a1 = 0.f;
#pragma unroll
        for (int s = 0; s < 16; s += 2) {
            a = fmaf(Ls[(16 + ri) * DC_LDM + s], s >= rj ? Rs[s * DC_LDM + rj] : 0.f, a);
            a1 = fmaf(Ls[(16 + ri) * DC_LDM + s + 1], s + 1 >= rj ? Rs[(s + 1) * DC_LDM + rj] : 0.f, a1);
        }
        tmp[ri * 17 + rj] = a + a1;
    }
    __syncthreads();
    {
        float a = 0.f, a1 = 0.f;
#pragma unroll
        for (int s = 0; s < 16; s += 2) {        // rows behind ri are left out, not multiplied by zero: they may be no numbers
            if (s <= ri) a = fmaf(Rs[(16 + ri) * DC_LDM + 16 + s], tmp[s * 17 + rj], a);
            if (s + 1 <= ri) a1 = fmaf(Rs[(16 + ri) * DC_LDM + 17 + s], tmp[(s + 1) * 17 + rj], a1);
        }
        Rs[(16 + ri) * DC_LDM + rj] = -(a + a1);
    }
    __syncthreads();
    float* Rg = reinterpret_cast<float*>(p.R + chunk_h * Z::M);
    float* Mg = reinterpret_cast<float*>(p.M + chunk_h * Z::M);
#pragma unroll
    for (int i = 0; i < 4; ++i) {                // M R, row 8 i + warp, column lane
        const int t = 8 * i + warp;
        float a = 0.f, a1 = 0.f;
#pragma unroll 8
        for (int s = 0; s <= t; s += 2) {
            a = fmaf(QK[t * (DC_C + 1) + s], Rs[s * DC_LDM + lane], a);
            if (s < t) a1 = fmaf(QK[t * (DC_C + 1) + s + 1], Rs[(s + 1) * DC_LDM + lane], a1);
        }
        Mg[t * DC_LDM + lane] = a + a1;
        Rg[t * DC_LDM + lane] = Rs[t * DC_LDM + lane];
    }
}

// Shared memory of a block of the walk, in bytes: keys, queries and R of two chunks (the next one's on their way), M R of three (read last), the walkers'
// partial sums of K S and Q S, x, u in three bfloat16 parts.  100 KB for bfloat16 activations: two blocks an SM.
template <typename T, int D> struct DcStage {
    using Z = DcSizes<T, D>;
    static constexpr int K = 0, Q = K + Z::KQ, R = Q + Z::KQ, SIZE = R + Z::M;
    static constexpr int LDP = D + 8, LDU = DC_COLS + 8, PLANE = DC_C * LDU;
    static constexpr int M = 2 * SIZE, PK = M + 3 * Z::M, PQ = PK + DC_C * LDP * 4, XS = PQ + DC_C * LDP * 4, UP = XS + DC_COLS * DC_LDM * 4,
                         BAR = UP + 3 * PLANE * 2, TOTAL = BAR + 16;
};
constexpr int DC_WALKERS = 256, DC_READERS = 128;

// Two groups of warps.  The eight walkers carry the state from chunk to chunk, 16 of its rows each, in registers: partial sums of K S and Q S over their rows,
// then S <- P_C S + K^T (D u).  The four readers add the partial sums up, make x and u for the walkers and, while those go on, the outputs.
//
// The state lies in the accumulators' layout with its columns as rows, which is the layout of the other operand of K S and Q S, so it never goes through shared
// memory.  R x and M R x stay float32 multiply-adds over the tokens up to t only: a later token's infinity must not reach back (0 times infinity).
//
// Bound by the chain of a chunk (split, products, sums, R x, split, products): 1.7 us a chunk with one block an SM, 68 us for 1,111 + 300 tokens of 16 heads.  All
// products in multiply-adds were bound by their reads of shared memory (16 columns a block leave no room for more than 4 x 4 results a thread), 2.8-3.4 us
// a chunk, 121 us; tensor cores with W = R (beta P K) and U = R (beta v) from the first kernel in place of R, three times the copies and twice the
// products, took 85.  Errors against 64 bits there: outputs 2.0e-7 (multiply-adds 2.4e-7), states 1.8e-7 (2.0e-7).
//
// A block a long request, not a request: the blocks of the others, a hundred kilobytes of shared memory each, cost more than they look (one of 24 tokens beside 63 single ones, 16 heads:
// 73 -> 67 us, 32 heads: 148 -> 134).
//
// Named barriers (each side meets the other once a chunk, in turn): 1 the first chunk, 3 partial sums of K S, 4 u, 5 partial sums of Q S, 6 Q S read.
template <typename T, int D>
__global__ void __launch_bounds__(DC_WALKERS + DC_READERS, DcSizes<T, D>::PARTS == 1 ? 2 : 1) delta_chunk_scan_kernel(const DeltaChunkParams p) {
    static_assert(D == 128 && DC_C == 32 && DC_COLS == 16, "eight walkers of 16 rows");
    using St = DcStage<T, D>;
    using Z = DcSizes<T, D>;
    constexpr int LDK = Z::LDK, LDP = St::LDP, LDU = St::LDU, PARTS = Z::PARTS;
    extern __shared__ __align__(16) unsigned char dc_smem[];
    float* PK = reinterpret_cast<float*>(dc_smem + St::PK);                         // [C][LDP]: walker w's sums at 16 w
    float* PQ = reinterpret_cast<float*>(dc_smem + St::PQ);
    __nv_bfloat16* up = reinterpret_cast<__nv_bfloat16*>(dc_smem + St::UP);         // [3][C][LDU]
    __shared__ int where_s[2];
    const int h = blockIdx.x, c0 = blockIdx.y * DC_COLS;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = h / (p.heads / p.kv_heads), dv = p.dv;
    const unsigned bar = (unsigned)__cvta_generic_to_shared(dc_smem + St::BAR);     // a barrier a stage
    pdl_wait();
    pdl_small();
    if (warp == 0) {
        int at, before;
        dc_nth(p.q_start, p.B, p.n_min, blockIdx.z, at, before);
        if (lane == 0) {
            where_s[0] = at; where_s[1] = before;
            tc_mbar_init(bar, 1); tc_mbar_init(bar + 8u, 1);
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        }
    }
    __syncthreads();
    const int r = where_s[0];
    if (r < 0) return;
    const int t0 = p.q_start[r], n = p.q_start[r + 1] - t0;
    const size_t first = (size_t)where_s[1];
    const int n_chunks = min((n + DC_C - 1) / DC_C, p.n_chunks - where_s[1]);         // (no more than the host's count has room for)
    if (n_chunks <= 0) return;
    auto wait = [&](int c) {                                 // for the operands of chunk c: one thread, the others meet it at a barrier
        if (!tc_mbar_wait(bar + 8u * (c & 1), (unsigned)(c >> 1) & 1u)) atomicExch(p.status + 1, 1);
    };

    if (tid < DC_WALKERS) {
        const int gr = lane >> 2, gt = 2 * (lane & 3), k0 = 16 * warp;
        // s[j]: rows k0 + 8 j + gt and the next, columns gr (entries 0, 1) and gr + 8 (2, 3)
        float* S = p.state + ((size_t)p.slots[r] * p.heads + h) * D * dv + c0;
        auto copy = [&](int dst, const unsigned char* src, int bytes, unsigned b) {
            asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                         ::"r"((unsigned)__cvta_generic_to_shared(dc_smem + dst)), "l"(src), "r"(bytes), "r"(b) : "memory");
        };
        auto fetch = [&](int c) {
            const int st = (c & 1) * St::SIZE;
            const unsigned b = bar + 8u * (c & 1);
            const size_t ch = (first + c) * p.heads + h, cg = (first + c) * p.kv_heads + g;
            tc_mbar_expect_tx(b, 2 * Z::KQ + 2 * Z::M);
            copy(st + St::K, p.K + cg * Z::KQ, Z::KQ, b);
            copy(st + St::Q, p.Q + cg * Z::KQ, Z::KQ, b);
            copy(st + St::R, p.R + ch * Z::M, Z::M, b);
            copy(St::M + (c % 3) * Z::M, p.M + ch * Z::M, Z::M, b);
        };
        if (tid == 0) {
            fetch(0);
            if (n_chunks > 1) fetch(1);
            wait(0);
        }
        float s[2][4];
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) s[j][i] = S[(size_t)(k0 + 8 * j + gt + (i & 1)) * dv + gr + 8 * (i >> 1)];
        // products of one to three parts of a and three of b, to float32's precision: all but those below 2^-24 of the product, the small ones in a sum of
        // their own; two b side by side, so that one's latency passes beside the other's
        auto mma3 = [](float (&big)[2][4], float (&rest)[2][4], const unsigned (&a)[3][4], const unsigned (&b)[2][3][2], bool a_parts, bool b_parts) {
            constexpr int A[5] = {2, 0, 1, 1, 0}, B[5] = {0, 2, 1, 0, 1};
#pragma unroll
            for (int i = 0; i < 5; ++i)
                if ((A[i] == 0 || a_parts) && (B[i] == 0 || b_parts)) {
#pragma unroll
                    for (int j = 0; j < 2; ++j) dc_mma(rest[j], a[A[i]], b[j][B[i]][0], b[j][B[i]][1]);
                }
#pragma unroll
            for (int j = 0; j < 2; ++j) dc_mma(big[j], a[0], b[j][0][0], b[j][0][1]);
        };
        // this warp's share of A [C][D] times the state; groups of four columns change places in every second four rows, for the readers
        auto with_state = [&](int A, const unsigned (&b)[2][3][2], float* P) {
            const __nv_bfloat16* Ap = reinterpret_cast<const __nv_bfloat16*>(dc_smem + A) + (lane & 15) * LDK + k0 + (lane >> 4) * 8;
            float* dst = P + gr * LDP + k0 + (gt ^ (gr & 4));
#pragma unroll
            for (int m = 0; m < 2; ++m) {
                unsigned a[3][4];
                float big[2][4] = {}, rest[2][4] = {};
#pragma unroll
                for (int i = 0; i < PARTS; ++i) dc_ldmatrix4(a[i], Ap + (i * DC_C + 16 * m) * LDK);
                mma3(big, rest, a, b, PARTS > 1, true);
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    *reinterpret_cast<float2*>(dst + 16 * m * LDP + 8 * j) = make_float2(big[j][0] + rest[j][0], big[j][1] + rest[j][1]);
                    *reinterpret_cast<float2*>(dst + (16 * m + 8) * LDP + 8 * j) = make_float2(big[j][2] + rest[j][2], big[j][3] + rest[j][3]);
                }
            }
        };
        asm volatile("bar.sync 1, 256;\n" ::: "memory");
        for (int c = 0; c < n_chunks; ++c) {
            const int st = (c & 1) * St::SIZE;
            {
                unsigned b[2][3][2];
#pragma unroll
                for (int j = 0; j < 2; ++j)
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        float x = s[k][2 * j], y = s[k][2 * j + 1];
#pragma unroll
                        for (int i = 0; i < 3; ++i) b[j][i][k] = dc_part<(PARTS > 1)>(x, y);
                    }
                with_state(st + St::K, b, PK);
                asm volatile("bar.arrive 3, 384;\n" ::: "memory");
                with_state(st + St::Q, b, PQ);
                asm volatile("bar.arrive 5, 384;\n" ::: "memory");
            }
            const float decay = *reinterpret_cast<const float*>(dc_smem + St::M + (c % 3) * Z::M + DC_C * 4);
            // keys as [token][row]: turned on the way, both halves of the rows
            unsigned kb[2][2][3][2];
            {
                const __nv_bfloat16* Kp = reinterpret_cast<const __nv_bfloat16*>(dc_smem + st + St::K) + (lane & 15) * LDK + k0 + (lane >> 4) * 8;
#pragma unroll
                for (int k = 0; k < 2; ++k)
#pragma unroll
                    for (int i = 0; i < PARTS; ++i) {
                        unsigned v[4];
                        dc_ldmatrix4t(v, Kp + (i * DC_C + 16 * k) * LDK);
                        kb[k][0][i][0] = v[0]; kb[k][0][i][1] = v[1]; kb[k][1][i][0] = v[2]; kb[k][1][i][1] = v[3];
                    }
            }
            asm volatile("bar.sync 4, 384;\n" ::: "memory");         // u
            float big[2][2][4] = {}, rest[2][4] = {};
#pragma unroll
            for (int k = 0; k < 2; ++k) {                            // 16 tokens
                unsigned ua[3][4];
#pragma unroll
                for (int i = 0; i < 3; ++i) dc_ldmatrix4t(ua[i], up + i * St::PLANE + (16 * k + (lane & 7) + (lane >> 4) * 8) * LDU + ((lane >> 3) & 1) * 8);
                mma3(big[k], rest, ua, kb[k], true, PARTS > 1);
            }
#pragma unroll
            for (int j = 0; j < 2; ++j)
#pragma unroll
                for (int i = 0; i < 4; ++i) s[j][i] = fmaf(decay, s[j][i], (big[0][j][i] + big[1][j][i]) + rest[j][i]);
            asm volatile("bar.sync 6, 384;\n" ::: "memory");         // Q S is read, and the stage by every walker; the next chunk is there
            if (tid == 0 && c + 2 < n_chunks) fetch(c + 2);
        }
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
            for (int i = 0; i < 4; ++i) S[(size_t)(k0 + 8 * j + gt + (i & 1)) * dv + gr + 8 * (i >> 1)] = s[j][i];
    } else {
        const int w = warp - DC_WALKERS / 32, t = lane, cc = 4 * w;          // token t and columns cc .. cc + 3
        float* xs = reinterpret_cast<float*>(dc_smem + St::XS);      // [16][LDM]; a warp's columns are its own
        auto sums = [&](const float* P) {                            // of the eight walkers' shares, as a tree
            float4 v[8];
#pragma unroll
            for (int k = 0; k < 8; ++k) v[k] = *reinterpret_cast<const float4*>(P + t * LDP + 16 * k + (cc ^ (t & 4)));
#pragma unroll
            for (int o = 1; o < 8; o *= 2)
#pragma unroll
                for (int k = 0; k < 8; k += 2 * o) { v[k].x += v[k + o].x; v[k].y += v[k + o].y; v[k].z += v[k + o].z; v[k].w += v[k + o].w; }
            return v[0];
        };
        // row t of A [C][LDM] times x for this warp's columns: a thread sums four tokens over every fourth group of four tokens s, then the four lanes that share
        // them hand each other three quarters.  Tokens up to t only.
        auto below = [&](int A, float (&out)[4]) {
            float o[4][4] = {};
            const int ts = lane & ~3;
            const float* Ap = reinterpret_cast<const float*>(dc_smem + A) + ts * DC_LDM;
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int s4 = 16 * i + 4 * (lane & 3);
                if (s4 > ts) continue;
                float4 x[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) x[j] = *reinterpret_cast<const float4*>(xs + (cc + j) * DC_LDM + s4);
                const bool diag = s4 == ts;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 m = *reinterpret_cast<const float4*>(Ap + k * DC_LDM + s4);
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        o[k][j] = fmaf(m.x, x[j].x, o[k][j]);
                        if (k >= 1 || !diag) o[k][j] = fmaf(m.y, x[j].y, o[k][j]);
                        if (k >= 2 || !diag) o[k][j] = fmaf(m.z, x[j].z, o[k][j]);
                        if (k >= 3 || !diag) o[k][j] = fmaf(m.w, x[j].w, o[k][j]);
                    }
                }
            }
            __syncwarp();
            const bool b0 = lane & 1, b1 = lane & 2;
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const float y0 = (b1 ? o[2][j] : o[0][j]) + __shfl_xor_sync(0xffffffffu, b1 ? o[0][j] : o[2][j], 2);
                const float y1 = (b1 ? o[3][j] : o[1][j]) + __shfl_xor_sync(0xffffffffu, b1 ? o[1][j] : o[3][j], 2);
                out[j] = (b0 ? y1 : y0) + __shfl_xor_sync(0xffffffffu, b0 ? y0 : y1, 1);
            }
        };
        const int Wd = 2 * p.kv_heads * D + p.heads * dv;
        const T* vp = reinterpret_cast<const T*>(p.qkv) + (size_t)t0 * Wd + 2 * p.kv_heads * D + (size_t)h * dv + c0 + cc;
        auto value = [&](int c) { return c * DC_C + t < n ? dc_load4(vp + (size_t)(c * DC_C + t) * Wd) : make_float4(0.f, 0.f, 0.f, 0.f); };
        float4 v = value(0);
        for (int c = 0; c < n_chunks; ++c) {
            asm volatile("bar.sync 3, 384;\n" ::: "memory");         // K S
            const float4 f = *reinterpret_cast<const float4*>(dc_smem + (c & 1) * St::SIZE + St::R + (t * DC_LDM + DC_C) * 4);
            {
                const float4 ks = sums(PK);
                xs[cc * DC_LDM + t] = fmaf(f.x, v.x, -f.y * ks.x); xs[(cc + 1) * DC_LDM + t] = fmaf(f.x, v.y, -f.y * ks.y);
                xs[(cc + 2) * DC_LDM + t] = fmaf(f.x, v.z, -f.y * ks.z); xs[(cc + 3) * DC_LDM + t] = fmaf(f.x, v.w, -f.y * ks.w);
            }
            __syncwarp();
            float u[4];
            below((c & 1) * St::SIZE + St::R, u);
            {
                float x0 = f.z * u[0], y0 = f.z * u[1], x1 = f.z * u[2], y1 = f.z * u[3];
#pragma unroll
                for (int i = 0; i < 3; ++i) {
                    const unsigned lo = dc_part<(PARTS > 1)>(x0, y0), hi = dc_part<(PARTS > 1)>(x1, y1);
                    *reinterpret_cast<uint2*>(up + i * St::PLANE + t * LDU + cc) = make_uint2(lo, hi);
                }
            }
            asm volatile("bar.arrive 4, 384;\n" ::: "memory");
            if (c + 1 < n_chunks) v = value(c + 1);
            asm volatile("bar.sync 5, 384;\n" ::: "memory");         // Q S
            const float4 qs = sums(PQ);
            if (tid == DC_WALKERS && c + 1 < n_chunks) wait(c + 1);
            __syncwarp();
            asm volatile("bar.arrive 6, 384;\n" ::: "memory");
            float o[4];
            below(St::M + (c % 3) * Z::M, o);
            if (c * DC_C + t < n)
                *reinterpret_cast<float4*>(p.out + ((size_t)(t0 + c * DC_C + t) * p.heads + h) * dv + c0 + cc) =
                    make_float4(fmaf(f.w, qs.x, o[0]), fmaf(f.w, qs.y, o[1]), fmaf(f.w, qs.z, o[2]), fmaf(f.w, qs.w, o[3]));
        }
    }
}

// whether runs of tokens are taken in chunks for these sizes
static bool delta_chunks_ok(int d, int dv) { return d == 128 && dv % DC_COLS == 0; }
static long long delta_prep_floats(int T_, int heads, int kv_heads, int d) {
    return ((long long)T_ * kv_heads * d * 2 + (long long)T_ * heads * 4 + 3) & ~3LL;
}
// bytes that the chunks' parts take; every part is a whole number of 16 bytes
static long long delta_chunk_bytes(long long n_chunks, int heads, int kv_heads, int dtype) {
    const long long kq = dtype == MSGL_F32 ? DcSizes<float, 128>::KQ : DcSizes<__nv_bfloat16, 128>::KQ;
    return n_chunks * (2 * kq * kv_heads + heads * (2LL * DcSizes<float, 128>::M));
}

// floats of scratch memory that msgl_delta_rule wants for T tokens; n_chunks: chunks of the runs that are taken in chunks, n_short: whether there are
// requests that are not
MSGL_API long long msgl_delta_rule_scratch(int T_, int heads, int kv_heads, int d, int dv, int n_chunks, int n_short, int dtype) {
    if (n_chunks <= 0 || !delta_chunks_ok(d, dv)) return delta_prep_floats(T_, heads, kv_heads, d);
    return (n_short ? delta_prep_floats(T_, heads, kv_heads, d) : 0) + delta_chunk_bytes(n_chunks, heads, kv_heads, dtype) / 4;
}

template <typename T, int D>
static int delta_chunk_launch(DeltaChunkParams& p, unsigned char* scratch, int n_chunks, int n_long, cudaStream_t stream) {
    using Z = DcSizes<T, D>;
    constexpr int smem1 = DcPrep<T, D>::TOTAL, smem2 = DcStage<T, D>::TOTAL;
    static_assert(Z::PARTS > 1 || 2 * (smem2 + 1024 + 64) <= 228 * 1024, "two blocks of the walk an SM");
    static MsglOncePerDevice once;
    if (once.due()) {      // first call on this device, never inside a stream capture
        if (cudaFuncSetAttribute(delta_chunk_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem1) != cudaSuccess ||
            cudaFuncSetAttribute(delta_chunk_scan_kernel<T, D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem2) != cudaSuccess ||
            cudaFuncSetAttribute(delta_chunk_kernel<T, D>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess ||
            cudaFuncSetAttribute(delta_chunk_scan_kernel<T, D>, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared) != cudaSuccess)
            return msgl_check_launch();
        once.mark();
    }
    const size_t ch = (size_t)n_chunks * p.heads, cg = (size_t)n_chunks * p.kv_heads;
    p.n_chunks = n_chunks;
    p.K = scratch; p.Q = p.K + cg * Z::KQ; p.R = p.Q + cg * Z::KQ; p.M = p.R + ch * Z::M;
    msgl_launch_pdl(delta_chunk_kernel<T, D>, dim3(n_chunks, p.heads), dim3(DC_THREADS), smem1, stream, p);
    msgl_launch_pdl(delta_chunk_scan_kernel<T, D>, dim3(p.heads, p.dv / DC_COLS, n_long), dim3(DC_WALKERS + DC_READERS), smem2, stream, p);
    return msgl_check_launch();
}

// n_chunks, n_long, n_min: chunks of DC_C tokens and number of the requests with n_min tokens or more (host's count), which are taken in chunks; 0: none.
// n_short: whether requests with fewer tokens are in the step.
MSGL_API int msgl_delta_rule(const void* qkv, const void* proj, long long proj_stride, int a_off, int b_off, const float* a_log,
                             const float* dt_bias, float* state, const int* q_start, const int* slots, float* out, float* scratch,
                             int heads, int kv_heads, int d, int dv, int T_, int B, int dtype, int n_chunks, int n_long, int n_min, int n_short,
                             void* status, cudaStream_t stream) {
    if (B <= 0 || T_ <= 0) return MSGL_OK;
    if (n_chunks > 0 && (!delta_chunks_ok(d, dv) || n_min < 1 || n_long < 1 || n_long > B || B > 65535 || heads > 65535 || dv / DC_COLS > 65535)) return MSGL_ERR_SIZE;
    if (n_chunks > 0 && (((uintptr_t)qkv & 15) != 0 || status == nullptr)) return MSGL_ERR_ALIGN;
    if (heads <= 0 || kv_heads <= 0 || heads % kv_heads || d <= 0 || dv <= 0 || d > DR_PARTS * 64 || scratch == nullptr) return MSGL_ERR_SIZE;
    if (((uintptr_t)scratch & 15) != 0) return MSGL_ERR_ALIGN;
    if (dtype != MSGL_F32 && dtype != MSGL_BF16) return MSGL_ERR_DTYPE;
    DeltaParams p;
    p.qkv = qkv; p.proj = proj; p.proj_stride = proj_stride; p.a_off = a_off; p.b_off = b_off; p.a_log = a_log; p.dt_bias = dt_bias;
    p.sc = reinterpret_cast<float4*>(scratch);                                  // [T][heads] first: 16-byte rows stay aligned
    p.kq = reinterpret_cast<float2*>(scratch + (size_t)T_ * heads * 4);
    p.state = state; p.q_start = q_start; p.slots = slots; p.out = out; p.heads = heads; p.kv_heads = kv_heads; p.d = d; p.dv = dv; p.T = T_;
    p.n_min = 1; p.n_max = n_chunks > 0 ? n_min - 1 : 0x7fffffff;
    int code;
    if (n_chunks <= 0 || n_short) {
        const dim3 g0(T_, (kv_heads + 3) / 4);
        if (dtype == MSGL_F32) msgl_launch_pdl(delta_prep_kernel<float>, g0, dim3(128), 0, stream, p);
        else msgl_launch_pdl(delta_prep_kernel<__nv_bfloat16>, g0, dim3(128), 0, stream, p);
        code = msgl_check_launch();
        if (code != MSGL_OK) return code;
    }
    if (n_chunks > 0) {
        DeltaChunkParams c;
        c.qkv = qkv; c.proj = proj; c.proj_stride = proj_stride; c.a_off = a_off; c.b_off = b_off; c.a_log = a_log; c.dt_bias = dt_bias;
        c.state = state; c.q_start = q_start; c.slots = slots; c.out = out; c.status = (int*)status;
        c.heads = heads; c.kv_heads = kv_heads; c.dv = dv; c.B = B; c.n_min = n_min;
        unsigned char* rest = reinterpret_cast<unsigned char*>(scratch + (n_short ? delta_prep_floats(T_, heads, kv_heads, d) : 0));
        if (dtype == MSGL_F32) code = delta_chunk_launch<float, 128>(c, rest, n_chunks, n_long, stream);
        else code = delta_chunk_launch<__nv_bfloat16, 128>(c, rest, n_chunks, n_long, stream);
        if (code != MSGL_OK || !n_short) return code;
    }
    const int many_cols = DR_MANY_WARPS * DR_WCOLS;
    const long long blocks_many = (long long)heads * B * ((dv + many_cols - 1) / many_cols);
    const int warps = blocks_many >= 2LL * msgl_sm_count() ? DR_MANY_WARPS : DR_FEW_WARPS;
    const int cols = warps * DR_WCOLS;
    const dim3 grid(heads, B, (dv + cols - 1) / cols);
    const size_t smem = 2 * ((size_t)DR_TB * 16 + (size_t)DR_TB * d * 8 + (size_t)DR_TB * cols * 4);
    const int rpt = (d + DR_PARTS - 1) / DR_PARTS;
#define DR_LAUNCH_E(N, E)                                                                                                   \
    do {                                                                                                                    \
        static MsglOncePerDevice once;                                                                                      \
        if (smem > 48 * 1024 && once.due()) {                                                                               \
            cudaFuncSetAttribute(delta_rule_kernel<float, N, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024);  \
            cudaFuncSetAttribute(delta_rule_kernel<__nv_bfloat16, N, E>, cudaFuncAttributeMaxDynamicSharedMemorySize, 160 * 1024); \
            once.mark();                                                                                                    \
        }                                                                                                                   \
        if (dtype == MSGL_F32) msgl_launch_pdl(delta_rule_kernel<float, N, E>, grid, dim3(warps * 32), smem, stream, p);             \
        else msgl_launch_pdl(delta_rule_kernel<__nv_bfloat16, N, E>, grid, dim3(warps * 32), smem, stream, p);                      \
    } while (0)
#define DR_LAUNCH(N)                                                                                                        \
    do {                                                                                                                    \
        if (d == N * DR_PARTS) DR_LAUNCH_E(N, true); else DR_LAUNCH_E(N, false);                                            \
    } while (0)
    if (rpt <= 4) DR_LAUNCH(4);
    else if (rpt <= 8) DR_LAUNCH(8);
    else if (rpt <= 16) DR_LAUNCH(16);
    else if (rpt <= 32) DR_LAUNCH(32);
    else DR_LAUNCH(64);
#undef DR_LAUNCH
#undef DR_LAUNCH_E
    return msgl_check_launch();
}

// ---------------------------------------------------------------------------------------
// out[t, j] = gelu_tanh(gate[t, j]) * table[ids[t]][offset + j],  j < dim: a layer's slice of a per-token table, gated
// ---------------------------------------------------------------------------------------
template <typename T>
__global__ void side_gate_mul_kernel(const T* __restrict__ gate, long long gate_stride, const T* __restrict__ table, int columns, int offset,
                                     const int* __restrict__ ids, int vocab, T* __restrict__ out, int dim, long long n) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long t = i / dim;
    const int j = (int)(i - t * dim);
    int id = ids[t];
    id = id < 0 ? 0 : (id >= vocab ? vocab - 1 : id);
    const float e = to_f32<T>(table[(size_t)id * columns + offset + j]);
    out[i] = from_f32<T>(gelu_tanhf_(to_f32<T>(gate[t * gate_stride + j])) * e);
}

MSGL_API int msgl_side_gate_mul(const void* gate, long long gate_stride, const void* table, int columns, int offset, const int* ids,
                                int vocab, void* out, int dim, int T_, int dtype, cudaStream_t stream) {
    if (T_ <= 0) return MSGL_OK;
    if (dim <= 0 || offset < 0 || offset + dim > columns || vocab <= 0) return MSGL_ERR_SIZE;
    const long long n = (long long)T_ * dim;
    const unsigned blocks = (unsigned)((n + 255) / 256);
    if (dtype == MSGL_F32) side_gate_mul_kernel<float><<<blocks, 256, 0, stream>>>((const float*)gate, gate_stride, (const float*)table, columns, offset, ids, vocab, (float*)out, dim, n);
    else if (dtype == MSGL_BF16) side_gate_mul_kernel<__nv_bfloat16><<<blocks, 256, 0, stream>>>((const __nv_bfloat16*)gate, gate_stride, (const __nv_bfloat16*)table, columns, offset, ids, vocab, (__nv_bfloat16*)out, dim, n);
    else return MSGL_ERR_DTYPE;
    return msgl_check_launch();
}
