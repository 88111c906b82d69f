// Float32 matrix product on the 5th-generation tensor cores: out[M, N] = x[M, K] . W[N, K]^T (+ bias), all float32.
//
// A float32 number is the sum of three bfloat16 numbers that hold all of its 24 bits, and a product of two bfloat16 numbers is exact in
// float32.  So a product of two float32 numbers is nine products of parts, of which the three smallest lie below 2^-25 of it and are
// left out: six tcgen05.mma with float32 accumulation give what float32 multiply-adds give.  The tensor cores' own
// accumulation runs over 64 neighbouring terms only; those sums are added up in float32 registers.
//
// The weight rows sit on the M dimension of tcgen05.mma (128 a tile), the tokens on its N dimension (up to 128 a tile, in steps of 16).  A block owns one
// tile and one of `splits` equal ranges of K:
//
//     adders      (four warps for 64 tokens) take a slab's sums out of tensor memory and add them to theirs, a thread a weight row
//     loaders     (eight warps) load a slab of K (64 columns of the 128 weight rows and of the tokens) into registers a slab ahead, split it and store the
//                 parts as the operand tiles (128-byte swizzle) of a stage
//     last warp   one lane issues a slab's 24 products and commits the stage to the loaders and the accumulator to the adders
//     all         the blocks of a tile's ranges form a cluster: each sums its share of the tokens over the cluster's shared memories, in the order of
//                 one tree, then bias and store
//
// Numbers that three bfloat16 parts do not hold (infinities, NaN, the last 2^-8 below the largest number, and most of those below 2^-110 other than 0: bfloat16 ends at 2^-133)
// are seen on the way by what the split leaves.  The block then does the sums of the tokens and weight rows that have one again in plain multiply-adds, so they behave as in float32
// arithmetic, and all other sums keep their bits.  (The parts of a product may lie up to 2^-8 above it: a sum that close to the largest number can come out infinite.)  [4096, 1024], 247 tokens, such a number in none, one, every 64th, every token: 25, 40, 51, 208 us, in one weight row 39 (the
// library 48); [1024, 2048], 64 tokens: 12.5, 21, 25, 75 and 18 (37).
//
// Bound by the split (11 instructions a pair of numbers) and the stores of the parts to shared memory.  Against the library's float32 product:
// [4096, 1024] 247 tokens 45.1 -> 23.1 us (90 TFLOP/s of float32; multiply-adds give 74 at the most), 9 tokens 19.3 -> 9.8; [1024, 2048] 39.6 -> 17.1 and 19.6 -> 9.2.
// Errors against 64 bits 1e-7 with terms of both signs (the library's 2e-7 to 1e-6) and 0.9e-7 with terms of one (0.7e-7 to 6e-7).
#include "common.cuh"
#include "tc_common.cuh"
#include <math.h>

constexpr int GF_LOADERS = 256, GF_MAX_SPLITS = 8, GF_STAGES = 2, GF_ROWS = 128;
constexpr unsigned GF_HEAD_BYTES = 256u;
template <int BN> struct GfSizes {
    static constexpr int COLS = BN < 64 ? BN : 64, ADDERS = 128 * (BN / COLS), THREADS = ADDERS + GF_LOADERS + 32;       // tokens an adder sums
    static constexpr unsigned A = GF_ROWS * 128u, B = BN * 128u, STAGE = 3u * (A + B), TMEM = 2 * BN;
    static constexpr unsigned SMEM = GF_HEAD_BYTES + 1024u + GF_STAGES * STAGE;
    static_assert(GF_STAGES * STAGE >= BN * GF_ROWS * 4u, "the sums lie over the stages");
};

struct GemmF32Params {
    const float* W; const float* X; const float* bias; float* out;
    long long ldx, ldo;
    int M, N, K, splits, n_tiles, rows;      // n_tiles: tiles of weight rows; rows: tokens of a tile
    int* status;
};

__device__ __forceinline__ unsigned gf_part(float& x, float& y) {            // the next bfloat16 part of two floats, taken off them
    const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
    const unsigned u = *reinterpret_cast<const unsigned*>(&h);
    x -= __uint_as_float(u << 16); y -= __uint_as_float(u & 0xffff0000u);
    return u;
}
// The last part: what is left after two has no more than eight bits, so its upper half is all of it.  Bits in the lower half (`rest` gathers them) mean that three parts do
// not hold the number: an infinity, NaN, a number that rounds to one, or one so small that its last part falls below the smallest bfloat16.
__device__ __forceinline__ unsigned gf_last(float x, float y, unsigned& rest) {
    rest |= __float_as_uint(x) | __float_as_uint(y);
    return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632);
}

template <int BN>
__global__ void __launch_bounds__(GfSizes<BN>::THREADS, 1) gemm_f32_kernel(const GemmF32Params p) {
    using Z = GfSizes<BN>;
    constexpr int ADD_WARPS = Z::ADDERS / 32, LAST = ADD_WARPS + GF_LOADERS / 32;
    extern __shared__ __align__(16) unsigned char gf_smem[];
    const unsigned smem_base = tc_smem_u32(gf_smem);
    const unsigned ring = (smem_base + GF_HEAD_BYTES + 1023u) & ~1023u;
    float* sums = reinterpret_cast<float*>(gf_smem + (ring - smem_base));           // [BN][128], when the products are done
    unsigned& tmem_base_s = *reinterpret_cast<unsigned*>(gf_smem + 64);
    unsigned* odd_s = reinterpret_cast<unsigned*>(gf_smem + 96);                    // a bit a weight row (four words) and a token (four): has a number that its parts do not hold
    const unsigned bar_full = smem_base, bar_empty = smem_base + 16u, bar_acc = smem_base + 32u, bar_free = smem_base + 48u;     // two of each
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int splits = p.splits, range = blockIdx.x % splits, tile = blockIdx.x / splits;
    const int n0 = (tile % p.n_tiles) * GF_ROWS, m0 = (tile / p.n_tiles) * p.rows, n_tok = min(p.rows, p.M - m0), n16 = (n_tok + 15) & ~15;
    const int slabs_all = (p.K + 63) / 64;
    const int k_begin = (int)((long long)range * slabs_all / splits), n_slabs = (int)((long long)(range + 1) * slabs_all / splits) - k_begin;

    if (warp == LAST) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_base_s)), "r"(Z::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    } else if (tid == 0) {
        for (int i = 0; i < 2; ++i) {
            tc_mbar_init(bar_full + 8u * i, GF_LOADERS / 32); tc_mbar_init(bar_empty + 8u * i, 1);
            tc_mbar_init(bar_acc + 8u * i, 1); tc_mbar_init(bar_free + 8u * i, ADD_WARPS);
        }
        for (int i = 0; i < 8; ++i) odd_s[i] = 0u;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_base_s;
    int fail = 0, issued = 0;                                    // slabs whose products are under way or done
    float acc[Z::COLS];                                          // adders: a weight row's sums, tokens col0 ..
    const int col0 = (warp >> 2) * Z::COLS;

    if (warp < ADD_WARPS) {
#pragma unroll
        for (int i = 0; i < Z::COLS; ++i) acc[i] = 0.f;
        const unsigned src = tmem + ((unsigned)((warp & 3) * 32) << 16) + (unsigned)col0;
        for (int i = 0; i < n_slabs; ++i) {
            if (!fail && !tc_mbar_wait(bar_acc + 8u * (i & 1), (i >> 1) & 1)) fail = 1;         // (goes on, without waiting: the lanes stay together)
            tc_fence_after();
#pragma unroll
            for (int c = 0; c < Z::COLS; c += 16) {
                if (col0 + c >= n16) break;
                unsigned v[16];
                tc_ld16(src + (unsigned)((i & 1) * BN + c), v);
                tc_wait_ld16(v);
#pragma unroll
                for (int j = 0; j < 16; ++j) acc[c + j] += __uint_as_float(v[j]);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(bar_free + 8u * (i & 1));
        }
    } else if (warp < LAST) {
        // a thread takes 8 columns (16-byte piece c of a part's row) of rows r, r + 32, ...: 128 of weights, then the tokens
        constexpr int NA = GF_ROWS / 32, NB = (BN + 31) / 32, NI = NA + NB;
        const int l = tid - Z::ADDERS, c = l & 7, r = l >> 3;
        const float* row[NI];
        bool ok[NI];
#pragma unroll
        for (int i = 0; i < NI; ++i) {
            const int rr = r + 32 * (i < NA ? i : i - NA);
            ok[i] = i < NA ? n0 + rr < p.N : rr < n_tok;
            row[i] = i < NA ? p.W + (size_t)(ok[i] ? n0 + rr : 0) * p.K : p.X + (size_t)(m0 + (ok[i] ? rr : 0)) * p.ldx;
        }
        float4 buf[NI][2];
        auto load = [&](int s, int i) {
            const int k = (k_begin + s) * 64 + 8 * c;
            const bool in = ok[i] && k < p.K && s < n_slabs;
            buf[i][0] = in ? *reinterpret_cast<const float4*>(row[i] + k) : make_float4(0.f, 0.f, 0.f, 0.f);
            buf[i][1] = in ? *reinterpret_cast<const float4*>(row[i] + k + 4) : make_float4(0.f, 0.f, 0.f, 0.f);
        };
        unsigned rest = 0u;
        // Before the wait the weights are only asked into L2 (a lane a 128-byte line of the first two slabs): the kernel before this one may be the one that writes them, as
        // when one product's result is the next one's weight.
#pragma unroll
        for (int i = 0; i < NA; ++i) {
            const int s = c & 3, k = (k_begin + s) * 64 + 8 * (c & 4);
            if (s < min(2, n_slabs) && ok[i] && k < p.K) asm volatile("prefetch.global.L2 [%0];\n" ::"l"(row[i] + k));
        }
        pdl_wait();
#pragma unroll
        for (int i = 0; i < NI; ++i) load(0, i);
        for (int s = 0; s < n_slabs; ++s) {
            const int st = s & 1;
            // (Passes at once the first time round.)  A warp gives up as one, or goes on without waiting, whichever the compiler schedules better around: [4096, 1024] with 9 rows and
            // cold weights 10.2 / 10.8 us, with 600 rows 64 / 60.
            if (BN < 64) {
                if (!__all_sync(0xffffffffu, tc_mbar_wait(bar_empty + 8u * st, ((s >> 1) & 1) ^ 1))) { fail = 1; break; }
            } else if (!fail && !tc_mbar_wait(bar_empty + 8u * st, ((s >> 1) & 1) ^ 1)) fail = 1;
            const unsigned base = ring + (unsigned)st * Z::STAGE;
#pragma unroll
            for (int i = 0; i < NI; ++i) {
                const int rr = r + 32 * (i < NA ? i : i - NA);
                if (i >= NA && rr >= n16) continue;
                float v[8] = {buf[i][0].x, buf[i][0].y, buf[i][0].z, buf[i][0].w, buf[i][1].x, buf[i][1].y, buf[i][1].z, buf[i][1].w};
                load(s + 1, i);                                  // its registers are free again
                const unsigned dst = base + (i < NA ? 0u : 3u * Z::A) + (unsigned)rr * 128u + (unsigned)((c ^ (rr & 7)) << 4);
#pragma unroll
                for (int part = 0; part < 3; ++part) {
                    unsigned a[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) a[j] = part < 2 ? gf_part(v[2 * j], v[2 * j + 1]) : gf_last(v[2 * j], v[2 * j + 1], rest);
                    asm volatile("st.shared.v4.u32 [%0], {%1,%2,%3,%4};\n" ::"r"(dst + (unsigned)part * (i < NA ? Z::A : Z::B)), "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]) : "memory");
                }
            }
            tc_fence_async_smem();
            __syncwarp();
            if (lane == 0) tc_mbar_arrive(bar_full + 8u * st);
        }
        if ((rest & 0xffffu) != 0u) {                            // which of the thread's rows it was
#pragma unroll 1
            for (int i = 0; i < NI; ++i) {
                const int rr = r + 32 * (i < NA ? i : i - NA);
                if (i < NA ? n0 + rr >= p.N : rr >= n_tok) continue;
                const float* src = i < NA ? p.W + (size_t)(n0 + rr) * p.K : p.X + (size_t)(m0 + rr) * p.ldx;
                unsigned left = 0u;
                const int k1 = min(p.K, (k_begin + n_slabs) * 64);
                for (int k = k_begin * 64 + 8 * c; k < k1; k += 256) {
                    float4 v[4][2];
#pragma unroll
                    for (int j = 0; j < 8; ++j)
                        v[j >> 1][j & 1] = k + (j >> 1) * 64 < k1 ? *reinterpret_cast<const float4*>(src + k + (j >> 1) * 64 + (j & 1) * 4) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < 8; ++j) {
                        float4& u = v[j >> 1][j & 1];
                        gf_part(u.x, u.y); gf_part(u.x, u.y); gf_last(u.x, u.y, left);
                        gf_part(u.z, u.w); gf_part(u.z, u.w); gf_last(u.z, u.w, left);
                    }
                }
                if ((left & 0xffffu) != 0u) atomicOr(odd_s + (i < NA ? 0 : 4) + (rr >> 5), 1u << (rr & 31));
            }
        }
    } else if (lane == 0) {
        const unsigned idesc = tc_idesc(false, (unsigned)n16);
        const unsigned long long da0 = tc_desc(ring, 16, 1024), db0 = tc_desc(ring + 3u * Z::A, 16, 1024);
        for (int i = 0; i < n_slabs; ++i) {
            const int st = i & 1;
            if (!tc_mbar_wait(bar_full + 8u * st, (i >> 1) & 1) || !tc_mbar_wait(bar_free + 8u * st, ((i >> 1) & 1) ^ 1)) { fail = 1; break; }
            tc_fence_after();
            const unsigned long long da = da0 + (unsigned long long)st * (Z::STAGE >> 4), db = db0 + (unsigned long long)st * (Z::STAGE >> 4);
            const unsigned d = tmem + (unsigned)(st * BN);
            constexpr int PA[6] = {2, 0, 1, 1, 0, 0}, PB[6] = {0, 2, 1, 0, 1, 0};              // the small products first
#pragma unroll
            for (int q = 0; q < 6; ++q)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk)
                    tc_mma(d, da + (unsigned long long)(PA[q] * (Z::A >> 4) + 2 * kk), db + (unsigned long long)(PB[q] * (Z::B >> 4) + 2 * kk), idesc, (q > 0 || kk > 0) ? 1u : 0u);
            tc_commit(bar_empty + 8u * st);
            tc_commit(bar_acc + 8u * st);
            ++issued;
        }
    }
    tc_fence_before();
    __syncwarp();
    const bool failed = __syncthreads_or(fail) != 0;
    if (failed) {                                                // somebody gave up waiting: no product may be under way when the stages and the tensor memory are let go
        if (issued > 0) tc_mbar_wait(bar_acc + 8u * ((issued - 1) & 1), ((issued - 1) >> 1) & 1);
        __syncwarp();
        __syncthreads();
    }
    // every product is done: the stages become [token][weight row]
    tc_fence_after();
    if (warp < ADD_WARPS) {
#pragma unroll
        for (int t = 0; t < Z::COLS; ++t) sums[(col0 + t) * GF_ROWS + (tid & 127)] = acc[t];
    }
    pdl_wait();                                                  // (all of x has been seen by the loaders; the others wait here before they write)
    pdl_late();
    __syncthreads();
    unsigned odd = 0u;
#pragma unroll
    for (int i = 0; i < 8; ++i) odd |= odd_s[i];
    if (odd) {                                                   // plain multiply-adds over the block's range: a warp four tokens against four weight rows, its lanes along K
        const int k1 = min(p.K, (k_begin + n_slabs) * 64);
        for (int item = warp; item < ((n_tok + 3) >> 2) * (GF_ROWS / 4); item += Z::THREADS / 32) {
            const int t0 = (item / (GF_ROWS / 4)) * 4, j0 = (item % (GF_ROWS / 4)) * 4;
            const unsigned tokens = odd_s[4 + (t0 >> 5)] >> (t0 & 31) & 15u, rows = odd_s[j0 >> 5] >> (j0 & 31) & 15u;
            if (!(tokens | rows) || n0 + j0 >= p.N) continue;
            float a[4][4] = {};
#pragma unroll 1
            for (int k = k_begin * 64 + 4 * lane; k < k1; k += 128) {
                float4 x[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = *reinterpret_cast<const float4*>(p.X + (size_t)(m0 + min(t0 + i, n_tok - 1)) * p.ldx + k);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float4 w = *reinterpret_cast<const float4*>(p.W + (size_t)min(n0 + j0 + j, p.N - 1) * p.K + k);
#pragma unroll
                    for (int i = 0; i < 4; ++i) a[i][j] = fmaf(w.w, x[i].w, fmaf(w.z, x[i].z, fmaf(w.y, x[i].y, fmaf(w.x, x[i].x, a[i][j]))));
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    const float v = warp_sum(a[i][j]);
                    if (lane == 0 && t0 + i < n_tok && ((tokens >> i | rows >> j) & 1u)) sums[(t0 + i) * GF_ROWS + j0 + j] = v;
                }
        }
    }
    __syncwarp();                                                // the aligned barrier wants whole warps
    if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    else __syncthreads();
    {   // the block's share of the tokens: range, range + splits, ..., SIDE at a time
        constexpr int SIDE = Z::THREADS / 128;
        const int j = tid & 127, n = n0 + j;
        const unsigned mine = tc_smem_u32(sums) + (unsigned)j * 4u;
        const float b = p.bias != nullptr && n < p.N ? p.bias[n] : 0.f;
        if (tid < SIDE * 128 && n < p.N) {
            for (int t = range + (tid >> 7) * splits; t < n_tok; t += SIDE * splits) {
                float v[GF_MAX_SPLITS];
#pragma unroll
                for (int r = 0; r < GF_MAX_SPLITS; ++r) {
                    v[r] = 0.f;
                    if (r < splits) {
                        unsigned peer;
                        asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(peer) : "r"(mine + (unsigned)t * (GF_ROWS * 4u)), "r"(r));
                        asm volatile("ld.shared::cluster.f32 %0, [%1];\n" : "=f"(v[r]) : "r"(peer));
                    }
                }
#pragma unroll
                for (int o = 1; o < GF_MAX_SPLITS; o *= 2)
#pragma unroll
                    for (int r = 0; r < GF_MAX_SPLITS; r += 2 * o) v[r] += v[r + o];
                p.out[(size_t)(m0 + t) * p.ldo + n] = v[0] + b;
            }
        }
    }
    __syncwarp();                                                // the aligned barrier wants whole warps
    if (splits > 1) asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
    __syncthreads();
    if (failed && tid == 0) atomicExch(p.status + 2, 1);
    if (warp == LAST) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(Z::TMEM) : "memory");
}

template <int BN>
static int gf_launch(const GemmF32Params& p, int blocks, cudaStream_t stream) {
    static MsglOncePerDevice attr_set;
    if (attr_set.due()) {      // first call on this device, never inside a stream capture
        if (cudaFuncSetAttribute(gemm_f32_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)GfSizes<BN>::SMEM) != cudaSuccess) return msgl_check_launch();
        attr_set.mark();
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)blocks); cfg.blockDim = dim3(GfSizes<BN>::THREADS); cfg.dynamicSmemBytes = GfSizes<BN>::SMEM; cfg.stream = stream; cfg.attrs = attr;
    cfg.numAttrs = msgl_pdl_enabled() ? 2 : 1;
    cudaLaunchKernelEx(&cfg, gemm_f32_kernel<BN>, p);
    return msgl_check_launch();
}

// float32 operands; K and ldx multiples of 8 and 4, bases 16-byte aligned.
MSGL_API int msgl_gemm_f32(const float* W, const float* X, const float* bias, float* out, int M, int N, int K, long long ldx, long long ldo, void* status, cudaStream_t stream) {
    if (M <= 0) return MSGL_OK;
    if (N <= 0 || K <= 0 || (K & 7) || (ldx & 3) || status == nullptr) return MSGL_ERR_SIZE;
    if (((uintptr_t)W | (uintptr_t)X) & 15) return MSGL_ERR_ALIGN;
    const int slabs = (K + 63) / 64;
    GemmF32Params p;
    p.W = W; p.X = X; p.bias = bias; p.out = out; p.ldx = ldx; p.ldo = ldo; p.M = M; p.N = N; p.K = K; p.status = (int*)status;
    p.n_tiles = (N + GF_ROWS - 1) / GF_ROWS;
    // Tokens a tile (up to 128 or up to 64, the tiles alike) and ranges of K: what takes least by a block's rows a slab, counted with those of 128 weights, and some 600
    // rows for its start and end, as long as all blocks run at once (ranges, of four slabs or more each, are for launches that leave SMs idle).  Clusters of eight fill the chip's groups of SMs
    // badly: no more than half of it.  [1024, 2048], 247 tokens: 64 a tile and 4 ranges 16 us, 128 and 4 ranges 20.5; [4096, 1024]: 64 and 1 range 25.8, 128 and 2 24.7.
    const int sms = msgl_sm_count();
    int splits = 1;
    long long tiles = 0;
    double best = 0.0;
    for (int cap = 128; cap >= 64; cap /= 2) {
        const int m_tiles = (M + cap - 1) / cap, rows = ((M + m_tiles - 1) / m_tiles + 15) & ~15;
        const long long t = (long long)p.n_tiles * ((M + rows - 1) / rows);
        for (int sp = 1; sp <= GF_MAX_SPLITS; sp *= 2) {
            if (sp > 1 && (t * sp > (sp == 8 ? sms / 2 : sms) || slabs < 4 * sp)) break;
            const double cost = (double)((t * sp + sms - 1) / sms) * (600.0 + (double)((slabs + sp - 1) / sp) * (GF_ROWS + rows));
            if (tiles == 0 || cost < best) { best = cost; tiles = t; splits = sp; p.rows = rows; }
        }
    }
    const int rows = p.rows;
    if (tiles * splits > 0x7fffffff) return MSGL_ERR_SIZE;
    p.splits = splits;
    const int blocks = (int)(tiles * splits);
    return rows > 64 ? gf_launch<128>(p, blocks, stream) : rows > 32 ? gf_launch<64>(p, blocks, stream) : rows > 16 ? gf_launch<32>(p, blocks, stream) : gf_launch<16>(p, blocks, stream);
}
