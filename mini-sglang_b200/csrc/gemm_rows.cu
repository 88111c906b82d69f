// Matrix product for a decode batch on the 5th-generation tensor cores: out[M, N] = x[M, K] . W[N, K]^T in bfloat16 with
// float32 accumulation, for few enough tokens (M up to about 256) that reading W once is what the product costs; plain, with a
// bias, or with a gated activation in the epilogue.  The same kernel runs the products of routed experts ("grouped": every
// expert has rows of its own in x and a matrix of its own in the stacked W).
//
// The weight rows sit on the M dimension of tcgen05.mma (128 of them a tile) and the tokens on its N dimension (16 to 256, in
// steps of 16), so nothing is computed for padding beyond the last 16 tokens and a tile's weights pass through shared memory
// once.  A block owns one tile (128 output columns; gated: 64, with their 64 gate and 64 up rows) and one of `splits` equal
// ranges of K (grouped: or both of two, with an accumulator each):
//
//     warp 0    TMA: W tile [128 x 64] and x tile [tokens x 64] of a slab of K into a ring of stages; the first stages' weights
//               are asked for before the kernel before this one has finished (programmatic dependent launch), x after it
//     warp 1    one lane issues four tcgen05.mma 128 x tokens x 16 a slab and commits the stage back to the loader
//     warps 2-5 accumulator -> shared memory, [token][weight row] float32
//     all       the blocks of a tile's ranges form a cluster: each sums its share of the tokens over the cluster's shared
//               memories (in the order of one tree whatever the block, so the result depends on neither timing nor the row's place),
//               then bias / activation and one rounding
//
// The ranges' sums never touch global memory, so the kernel needs no scratch.  Two or three blocks share an SM where the stages
// allow it: one streams while another starts or drains.  Every wait for a copy or a product is bounded; a block that gives up
// sets status[2], meets the others all the same and frees its tensor memory (results are then invalid and the host raises).  The
// cluster's barriers and the allocation of tensor memory are not: they wait for blocks that always get there.
#include "common.cuh"
#include "tc_common.cuh"
#include <math.h>

constexpr int GR_THREADS = 192, GR_MAX_STAGES = 12, GR_MAX_SPLITS = 8;
constexpr unsigned GR_A_BYTES = 128u * 128u;                     // 128 weight rows x 64 elements
constexpr unsigned GR_HEAD_BYTES = 512u;                         // barriers and the tensor-memory address

enum { GR_PLAIN = 0, GR_SILU = 1, GR_RELU = 2, GR_CLAMPED = 3 };  // the first three are the GLU modes of common.cuh

struct GemmRowsParams {
    const __nv_bfloat16* bias;     // [n_valid], gated: [2 n_valid]; or null
    void* out;
    long long ldo;
    int M, n_valid, K;             // tokens (grouped: rows of x), output columns, inner size
    int up_off;                    // gated: how many rows of W an up row lies behind its gate row
    int expert_rows, experts;      // grouped: rows of W an expert has, how many there are
    const int* ends;               // grouped: [experts] running sum of the experts' rows in x
    int asked;                     // the kernel before this one may be the one that writes W: its first tiles are only asked into L2 ahead of the wait
    int apart;                     // grouped: the expert whose matrix is w2map's (one that all tokens use); -1: none
    int bn, stages, splits;        // tokens a pass (a multiple of 16), ring depth, blocks that share a tile's K
    int halves;                    // 2: a block has two ranges of K (splits is 1 then), an accumulator each
    unsigned tmem_cols;
    float limit;                   // GR_CLAMPED
    int* status;
};

__device__ __forceinline__ unsigned gr_peer(unsigned saddr, unsigned rank) {       // the same offset in block `rank` of the cluster
    unsigned r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;\n" : "=r"(r) : "r"(saddr), "r"(rank));
    return r;
}
__device__ __forceinline__ float2 gr_peer_load(unsigned cluster_addr) {
    float2 v;
    asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];\n" : "=f"(v.x), "=f"(v.y) : "r"(cluster_addr));
    return v;
}
__device__ __forceinline__ void gr_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\nbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void gr_ask(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];\n" ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(x), "r"(y) : "memory");
}

template <int MODE> __device__ __forceinline__ float gr_act(float g, float u, float limit) {
    if (MODE == GR_CLAMPED) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return g / (1.f + expf(-1.702f * g)) * (u + 1.f);
    }
    return glu_act<MODE>(g) * u;
}
__device__ __forceinline__ void gr_store2(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void gr_store2(__nv_bfloat16* p, float a, float b) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b); }
__device__ __forceinline__ void gr_store(float* p, float a) { *p = a; }
__device__ __forceinline__ void gr_store(__nv_bfloat16* p, float a) { *p = __float2bfloat16_rn(a); }

// Block `range` of a tile's SP blocks: tokens range, range + SP, ... of the pass, summed over the blocks' accumulators in shared
// memory as a balanced tree over the ranges, ((0 + 1) + (2 + 3)) + ..., then bias / activation and the store.  Every block starts at its own
// accumulator (they do not all read one) and goes on by the tree: its neighbour's, the neighbouring pair's ...  Only the two sides of an
// addition change places with the block, so a row's result does not depend on where in the batch it stands.  A thread takes two output
// columns of a token, four tokens at a time (two with eight ranges): the loads from the other blocks take a few hundred cycles each and have to be
// under way together, ahead of all additions (one token after the other they made the product of 128 rows of 24,576 x 4,096 44 us long; additions
// between the loads of eight ranges made that of 16 rows of 2,048 x 4,096 9.0 us long instead of 7.3).
template <int MODE, typename OutT, int SP>
__device__ __forceinline__ void gr_reduce(const GemmRowsParams& p, unsigned sums, int range, int tok0, int n_tok, int col0) {
    constexpr bool GLU = MODE != GR_PLAIN;
    constexpr int PER = GLU ? 32 : 64, SLOTS = GR_THREADS / PER, U = SP >= 8 ? 2 : 4;
    const int j = threadIdx.x % PER, col = col0 + 2 * j;
    if (col >= p.n_valid) return;
    const bool two = col + 1 < p.n_valid;
    float2 ba = make_float2(0.f, 0.f), bu = make_float2(0.f, 0.f);
    if (p.bias != nullptr) {
        ba.x = __bfloat162float(p.bias[col]);
        if (two) ba.y = __bfloat162float(p.bias[col + 1]);
        if (GLU) {
            bu.x = __bfloat162float(p.bias[p.n_valid + col]);
            if (two) bu.y = __bfloat162float(p.bias[p.n_valid + col + 1]);
        }
    }
    unsigned peer[SP];
#pragma unroll
    for (int r = 0; r < SP; ++r) peer[r] = gr_peer(sums + (unsigned)j * 8u, (unsigned)(range ^ r));
    OutT* out = reinterpret_cast<OutT*>(p.out) + col;
    for (int n0 = range + (int)(threadIdx.x / PER) * SP; n0 < n_tok; n0 += U * SLOTS * SP) {
        float2 a[SP][U], u[SP][U];
#pragma unroll
        for (int r = 0; r < SP; ++r)
#pragma unroll
            for (int i = 0; i < U; ++i) {
                const int n = n0 + i * SLOTS * SP;
                a[r][i] = u[r][i] = make_float2(0.f, 0.f);
                if (n >= n_tok) continue;
                a[r][i] = gr_peer_load(peer[r] + (unsigned)n * 512u);
                if (GLU) u[r][i] = gr_peer_load(peer[r] + (unsigned)n * 512u + 256u);
            }
#pragma unroll
        for (int step = 1; step < SP; step *= 2)
#pragma unroll
            for (int r = 0; r < SP; r += 2 * step)
#pragma unroll
                for (int i = 0; i < U; ++i) {
                    a[r][i].x += a[r + step][i].x; a[r][i].y += a[r + step][i].y;
                    if (GLU) { u[r][i].x += u[r + step][i].x; u[r][i].y += u[r + step][i].y; }
                }
#pragma unroll
        for (int i = 0; i < U; ++i) {
            const int n = n0 + i * SLOTS * SP;
            if (n >= n_tok) continue;
            float x = a[0][i].x + ba.x, y = a[0][i].y + ba.y;
            if (GLU) { x = gr_act<MODE>(x, u[0][i].x + bu.x, p.limit); y = gr_act<MODE>(y, u[0][i].y + bu.y, p.limit); }
            OutT* dst = out + (size_t)(tok0 + n) * p.ldo;
            if (two) gr_store2(dst, x, y);              // ldo and col are even, the base 16-byte aligned
            else gr_store(dst, x);
        }
    }
}

template <int MODE, typename OutT, bool GROUPED>
__global__ void __launch_bounds__(GR_THREADS) gemm_rows_kernel(const __grid_constant__ CUtensorMap xmap, const __grid_constant__ CUtensorMap wmap,
                                                               const __grid_constant__ CUtensorMap w2map, const GemmRowsParams p) {
    constexpr bool GLU = MODE != GR_PLAIN;
    extern __shared__ __align__(16) unsigned char gr_smem[];
    const unsigned smem_base = tc_smem_u32(gr_smem);
    const unsigned ring = (smem_base + GR_HEAD_BYTES + 1023u) & ~1023u;
    unsigned& tmem_base_s = *reinterpret_cast<unsigned*>(gr_smem + 280);
    auto bar_full = [&](int s) { return smem_base + 8u * (unsigned)s; };
    auto bar_empty = [&](int s) { return smem_base + 128u + 8u * (unsigned)s; };
    const unsigned bar_acc = smem_base + 256u;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int S = p.stages, splits = p.splits;
    const unsigned stage_bytes = GR_A_BYTES + (unsigned)p.bn * 128u;
    const int tile = blockIdx.x / splits, range = blockIdx.x - tile * splits;

    const int slabs_all = (p.K + 63) / 64;
    const int k_begin = (int)((long long)range * slabs_all / splits), k_end = (int)((long long)(range + 1) * slabs_all / splits);
    const int n_slabs = k_end - k_begin, n_first = p.halves == 2 ? slabs_all / 2 : n_slabs;        // slabs of the block's first accumulator
    const unsigned half_cols = p.tmem_cols / 2;
    const int col0 = tile * (GLU ? 64 : 128);

    // The tokens that this block multiplies: all of them, or (grouped) runs of up to bn rows of an expert, counted over the experts in order, from
    // the blockIdx.y-th on in steps of gridDim.y.  So a crowd at a few experts, whose rows a router may send there together, is worked on side by side.
    // 32 experts are looked at together, four looks' loads under way at once.  The blocks of a cluster share their runs.
    int expert = 0, tok0 = 0, n_tok = p.M, run = blockIdx.y, n_runs = 1;
    auto find_run = [&]() -> bool {
        int counted = 0;
        bool found = false;
        for (int e0 = 0; e0 < p.experts; e0 += 128) {
            int begin[4], end[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int e = min(e0 + 32 * i + lane, p.experts - 1);
                end[i] = p.ends[e];
                begin[i] = e > 0 ? p.ends[e - 1] : 0;
                if (e0 + 32 * i + lane >= p.experts) begin[i] = end[i];
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (e0 + 32 * i >= p.experts) break;
                const int rows = end[i] - begin[i];
                int runs = rows > 0 ? 1 : 0;
                if (__any_sync(0xffffffffu, rows > p.bn)) runs = (rows + p.bn - 1) / p.bn;
                const int total = __reduce_add_sync(0xffffffffu, runs);
                if (!found && run < counted + total) {           // this look's
                    int sum = runs;
#pragma unroll
                    for (int o = 1; o < 32; o <<= 1) { const int v = __shfl_up_sync(0xffffffffu, sum, o); if (lane >= o) sum += v; }
                    const int l = __ffs(__ballot_sync(0xffffffffu, run < counted + sum)) - 1;
                    expert = e0 + 32 * i + l;
                    tok0 = __shfl_sync(0xffffffffu, begin[i], l) + (run - counted - __shfl_sync(0xffffffffu, sum - runs, l)) * p.bn;
                    n_tok = min(p.bn, __shfl_sync(0xffffffffu, end[i], l) - tok0);
                    found = true;
                }
                counted += total;
            }
        }
        n_runs = counted;
        return found;
    };
    // the set-up goes on while the kernel before this one finishes, which `ends` comes from, but for blocks that a random choice of experts
    // leaves without a run
    const bool ahead = GROUPED && (int)blockIdx.y >= p.experts;
    if (ahead) {
        pdl_wait();
        if (!find_run()) return;
    }

    if (tid == 0) {
        for (int s = 0; s < S; ++s) { tc_mbar_init(bar_full(s), 1); tc_mbar_init(bar_empty(s), 1); }
        tc_mbar_init(bar_acc, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem_u32(&tmem_base_s)), "r"(p.tmem_cols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const unsigned tmem = tmem_base_s;

    if (GROUPED && !ahead) {
        pdl_wait();
        if (!find_run()) {
            if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
            return;
        }
    }
    int fail = 0, g0 = 0, pass = 0;                    // g0: slabs that went through the ring before this run
    for (;;) {
        const bool other = GROUPED && expert == p.apart;
        const CUtensorMap* wm = other ? &w2map : &wmap;
        const int w_row = (other ? 0 : expert * p.expert_rows) + col0, n16 = (n_tok + 15) & ~15;      // n16: tokens that are multiplied
        const unsigned x_bytes = (GROUPED ? (unsigned)n16 : (unsigned)p.bn) * 128u;
        const bool last = !GROUPED || run + (int)gridDim.y >= n_runs;
        if (warp == 0) {
            if (lane == 0) {
                auto load_w = [&](int k, unsigned a_s, unsigned bar) {
                    if (GLU) {
                        tc_tma_load(a_s, wm, k * 64, w_row, bar);
                        tc_tma_load(a_s + 64u * 128u, wm, k * 64, w_row + p.up_off, bar);
                    } else {
                        tc_tma_load(a_s, wm, k * 64, w_row, bar);
                    }
                };
                auto load_x = [&](int k, unsigned b_s, unsigned bar) {
                    if (GROUPED) {
                        for (int n = 0; n < n16; n += 16) tc_tma_load(b_s + (unsigned)n * 128u, &xmap, k * 64, tok0 + n, bar);
                    } else {
                        tc_tma_load(b_s, &xmap, k * 64, 0, bar);
                    }
                };
                int first = 0;
                if (!GROUPED) {                        // weights depend on no kernel: the ring's first round is under way before the wait
                    first = min(S, n_slabs);
                    auto first_w = [&]() {
                        for (int i = 0; i < first; ++i) {
                            tc_mbar_expect_tx(bar_full(i), GR_A_BYTES + x_bytes);
                            load_w(k_begin + i, ring + (unsigned)i * stage_bytes, bar_full(i));
                        }
                    };
                    if (!p.asked) {
                        first_w();
                    } else {
                        for (int i = 0; i < first; ++i) {
                            gr_ask(wm, (k_begin + i) * 64, w_row);
                            if (GLU) gr_ask(wm, (k_begin + i) * 64, w_row + p.up_off);
                        }
                    }
                    pdl_wait();
                    if (p.asked) first_w();
                    for (int i = 0; i < first; ++i) load_x(k_begin + i, ring + (unsigned)i * stage_bytes + GR_A_BYTES, bar_full(i));
                }
                for (int i = first; i < n_slabs; ++i) {
                    const int g = g0 + i, st = g % S;
                    if (!tc_mbar_wait(bar_empty(st), ((g / S) & 1) ^ 1)) { fail = 1; break; }       // (passes at once the first time round)
                    const unsigned a_s = ring + (unsigned)st * stage_bytes;
                    tc_mbar_expect_tx(bar_full(st), GR_A_BYTES + x_bytes);
                    load_w(k_begin + i, a_s, bar_full(st));
                    load_x(k_begin + i, a_s + GR_A_BYTES, bar_full(st));
                }
                if (last) pdl_late();                  // everything is asked for, and tensor memory is allocated: the next kernel may set itself up
            }
        } else if (warp == 1) {
            if (lane == 0) {
                const unsigned idesc = tc_idesc(false, (unsigned)n16);
                const unsigned long long da0 = tc_desc(ring, 16, 1024), db0 = tc_desc(ring + GR_A_BYTES, 16, 1024);
                const unsigned long long step = stage_bytes >> 4;
                for (int i = 0; i < n_slabs; ++i) {
                    const int g = g0 + i, st = g % S;
                    if (!tc_mbar_wait(bar_full(st), (g / S) & 1)) { fail = 1; break; }
                    tc_fence_after();
                    const unsigned long long da = da0 + (unsigned long long)st * step, db = db0 + (unsigned long long)st * step;
                    const unsigned acc = i < n_first ? tmem : tmem + half_cols;
#pragma unroll
                    for (int kk = 0; kk < 4; ++kk)
                        tc_mma(acc, da + (unsigned long long)(2 * kk), db + (unsigned long long)(2 * kk), idesc, ((i > 0 && i != n_first) || kk > 0) ? 1u : 0u);
                    tc_commit(bar_empty(st));
                }
                if (!fail) tc_commit(bar_acc);
            }
        } else {
            // accumulator (lane = weight row of the tile) -> [token][128 rows] over the ring, which nothing reads or fills any more
            if (!tc_mbar_wait(bar_acc, pass & 1)) fail = 1;
            tc_fence_after();
            if (!fail) {
                const int q = warp & 3;
                const unsigned src = tmem + ((unsigned)(q * 32) << 16), dst = ring + (unsigned)(q * 32 + lane) * 4u;
                for (int c = 0; c < n16; c += 16) {
                    unsigned v[16];
                    tc_ld16(src + (unsigned)c, v);
                    tc_wait_ld16(v);
                    if (p.halves == 2) {               // the sum that two blocks would make of their accumulators
                        unsigned w[16];
                        tc_ld16(src + half_cols + (unsigned)c, w);
                        tc_wait_ld16(w);
#pragma unroll
                        for (int j = 0; j < 16; ++j) v[j] = __float_as_uint(__uint_as_float(v[j]) + __uint_as_float(w[j]));
                    }
#pragma unroll
                    for (int j = 0; j < 16; ++j) asm volatile("st.shared.b32 [%0], %1;\n" ::"r"(dst + (unsigned)(c + j) * 512u), "r"(v[j]) : "memory");
                }
            }
        }
        tc_fence_before();
        __syncwarp();
        if (splits > 1) gr_cluster_sync();
        else __syncthreads();
        tc_fence_after();
        if (splits == 1) gr_reduce<MODE, OutT, 1>(p, ring, 0, tok0, n_tok, col0);
        else if (splits == 2) gr_reduce<MODE, OutT, 2>(p, ring, range, tok0, n_tok, col0);
        else if (splits == 4) gr_reduce<MODE, OutT, 4>(p, ring, range, tok0, n_tok, col0);
        else gr_reduce<MODE, OutT, 8>(p, ring, range, tok0, n_tok, col0);
        if (!last) tc_fence_async_smem();               // the next run's copies may overwrite what was read here
        __syncwarp();
        if (splits > 1) gr_cluster_sync();              // ... and the cluster's other blocks have read this block's sums
        else if (!last) __syncthreads();
        if (last) break;
        g0 += n_slabs;
        ++pass;
        run += (int)gridDim.y;
        find_run();
    }
    const bool failed = __syncthreads_or(fail) != 0;
    if (failed && p.status != nullptr && tid == 0) atomicExch(p.status + 2, 1);
    if (warp == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(p.tmem_cols) : "memory");
}

template <int MODE, typename OutT, bool GROUPED>
static int gr_launch(const CUtensorMap& xm, const CUtensorMap& wm, const CUtensorMap& w2m, const GemmRowsParams& p, int tiles, int runs, size_t smem, cudaStream_t stream) {
    auto* kernel = gemm_rows_kernel<MODE, OutT, GROUPED>;
    static MsglOncePerDevice attr_set;
    if (attr_set.due()) {      // first call on this device, never inside a stream capture
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return msgl_check_launch();
        attr_set.mark();
    }
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = p.splits; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.gridDim = dim3((unsigned)(tiles * p.splits), (unsigned)runs);
    cfg.blockDim = dim3(GR_THREADS); cfg.dynamicSmemBytes = smem; cfg.stream = stream; cfg.attrs = attr;
    cfg.numAttrs = msgl_pdl_enabled() ? 2 : 1;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, xm, wm, w2m, p);
    (void)e;
    return msgl_check_launch();
}

// How a product of `tiles` tiles of `slabs` slabs with bn tokens a pass is cut: ranges of K, blocks an SM, ring depth.
//
// Ranges: a block alone on an SM leaves the memory waiting (its stages are fetched, multiplied and drained one behind the other, and it starts and
// ends alone), so the launch should have two blocks an SM or more; ranges of fewer than four slabs cost more in their sum than they bring.  [24,576 x 4,096]
// gated, 48 rows: 1 range 38.7-41.0 us, 2 ranges 36.5, 4 ranges 43.0; [6,144 x 1,024] gated, 16 rows: 7.9 / 5.9 / 5.7 us.
// Blocks an SM: three where the shared memory allows it, two where they fill their last round better (32 experts of
// [2,048 x 1,536], 700 tokens, four experts each: 512 blocks, two an SM 46.5 us, three 52.5; [3,072 x 2,048]: 768 blocks, 85.3 / 79.0).
static void gr_plan(long long tiles, int slabs, int bn, int& splits, int& stages, int want_splits, int want_per_sm) {
    const unsigned stage_bytes = GR_A_BYTES + (unsigned)bn * 128u;
    const int sms = msgl_sm_count();
    splits = 1;
    if (want_splits > 0) splits = want_splits;
    else
        while (splits < GR_MAX_SPLITS && tiles * splits < 2 * sms && slabs >= splits * 2 * 4) splits *= 2;
    while (splits > slabs) splits /= 2;
    auto fill = [&](int per_sm) {              // how full the rounds of blocks are
        const long long slots = (long long)sms * per_sm, rounds = (tiles * splits + slots - 1) / slots;
        return (double)(tiles * splits) / (double)(rounds * slots);
    };
    int per_sm = want_per_sm > 0 ? want_per_sm : (fill(2) > 1.1 * fill(3) ? 2 : 3);
    for (;; --per_sm) {                        // (an SM has 228 KB, 1 KB of it taken by every block)
        const unsigned budget = (228u * 1024u) / (unsigned)per_sm - 1024u - GR_HEAD_BYTES - 1024u;
        stages = (int)(budget / stage_bytes);
        if (stages > GR_MAX_STAGES) stages = GR_MAX_STAGES;
        if (per_sm == 1 || (stages >= 2 && (unsigned)stages * stage_bytes >= (unsigned)bn * 512u)) break;      // the ring has to hold the sums as well
    }
    const int most = (slabs + splits - 1) / splits;
    if (stages > most && (unsigned)most * stage_bytes >= (unsigned)bn * 512u) stages = most;
}

// Grouped products: a tile's K is one range or two, added at the end, and which of them follows from the sizes alone, so that a token's results do not
// depend on how many tokens stand beside it.  Two where `experts` experts, the fewest that a step uses, give fewer than two blocks an SM (as
// above).  How two ranges are worked on does follow the tokens and changes no bit: by the two blocks of a cluster where the experts in use give too few blocks, else
// by one block with an accumulator each (up to 64 tokens: beyond, the accumulators of three blocks are more than an SM's tensor memory).
static int gr_ranges(long long tiles, long long experts, int slabs) { return tiles * experts < 2 * msgl_sm_count() && slabs >= 8 ? 2 : 1; }

// Whether the driver makes tensor maps, without which no product of this file runs.
MSGL_API int msgl_tensor_maps() { return tc_encoder() != nullptr; }

// mode 0: out[M, n_out] = x . W^T (+ bias); 1, 2: act(gate) * up with act = silu, relu, W = [gate; up] (n_out rows each); 3: the
// clamped form min(g, limit) * sigmoid(1.702 min(g, limit)) * (clamp(u, -limit, limit) + 1).
// experts > 0: W is [experts][n_out or 2 n_out][K], x holds M rows in the order of their experts, ends [experts] their running sum on
// the device; tokens: how many tokens brought the rows, M / tokens experts each.  Else M is at most 256.
// W2 (grouped; or null): one more expert that all tokens use, its matrix apart from W; its rows lie behind the others' in x and out (M counts them not), ends is [experts + 1].
// splits: ranges of K; 0 = chosen from the sizes, grouped: for steps that use all experts; -1 = grouped, for steps down to a single token.
// per_sm: 0 = chosen by gr_plan.
// bfloat16 operands; out bfloat16 or (mode 0) float32.  K, ldx multiples of 8, ldo even, bases 16-byte aligned.
static int gr_product(const void* W, const void* W2, const void* X, const void* bias, void* out, int M, int n_out, int K, long long ldx, long long ldo,
                      int mode, int out_f32, float limit, int experts, const int* ends, int tokens, int splits, int per_sm, bool asked, void* status, cudaStream_t stream) {
    if (M <= 0) return MSGL_OK;
    const bool glu = mode != GR_PLAIN, grouped = experts > 0;
    if (mode < 0 || mode > 3 || n_out <= 0 || K <= 0 || (K & 7) || (ldx & 7) || (ldo & 1) || status == nullptr || experts < 0 || experts > 65535 ||
        splits < -1 || (splits == -1 && !grouped) || splits > GR_MAX_SPLITS || (splits > 0 && (splits & (splits - 1))) || per_sm < 0 || per_sm > 3)
        return MSGL_ERR_SIZE;
    if (grouped ? (ends == nullptr || bias != nullptr || tokens <= 0) : M > 256) return MSGL_ERR_SIZE;
    if (W2 != nullptr && !grouped) return MSGL_ERR_SIZE;
    if (((uintptr_t)W | (uintptr_t)W2 | (uintptr_t)X | (uintptr_t)out) & 15) return MSGL_ERR_ALIGN;
    long long w_rows = glu ? 2 * (long long)n_out : n_out;
    int bn = (M + 15) & ~15;
    double live = 1.0;
    if (grouped) {
        // Room for the rows of an expert that the tokens favour: a little over what a random choice gives, and from 32 to 64 all of 64 (only
        // rows that are there are copied and multiplied, and three blocks an SM have three stages at 32 as at 64).  An expert with more has
        // its weights read by several blocks side by side; more room costs shared memory (700 tokens, 88 rows an expert in the mean: 112 rows 79 us,
        // 160 rows 85 us).
        const double mean = (double)M / experts, room = mean + 4.0 * sqrt(mean) + 2.0;
        bn = room >= 160.0 ? 160 : room > 16.0 && room <= 64.0 ? 64 : ((int)room + 15) & ~15;
        const int most = (tokens + 15) & ~15;
        if (bn > most) bn = most;
        live = experts * (1.0 - pow(1.0 - fmin(1.0, (double)M / tokens / experts), (double)tokens));       // experts that some token uses, in the mean
        if (live < 1.0) live = 1.0;
        if (W2 != nullptr) live += 1.0;
        w_rows *= experts;
    }
    CUtensorMap xm, wm, w2m;
    const int apart_rows = W2 != nullptr ? tokens : 0;
    if (!tc_matrix_map(X, (long long)M + apart_rows, K, ldx * 2, grouped ? 16 : bn, &xm) || !tc_matrix_map(W, w_rows, K, (long long)K * 2, glu ? 64 : 128, &wm)) return MSGL_ERR_SIZE;
    if (W2 == nullptr) w2m = wm;
    else if (!tc_matrix_map(W2, w_rows / experts, K, (long long)K * 2, glu ? 64 : 128, &w2m)) return MSGL_ERR_SIZE;
    GemmRowsParams p;
    p.asked = asked ? 1 : 0;
    p.bias = (const __nv_bfloat16*)bias; p.out = out; p.ldo = ldo; p.M = M; p.n_valid = n_out; p.K = K;
    p.up_off = n_out; p.expert_rows = grouped ? (glu ? 2 * n_out : n_out) : 0; p.experts = experts + (W2 != nullptr ? 1 : 0); p.apart = W2 != nullptr ? experts : -1; p.ends = ends; p.bn = bn; p.limit = limit; p.status = (int*)status;
    const int tiles = (n_out + (glu ? 63 : 127)) / (glu ? 64 : 128);
    const int slabs = (K + 63) / 64;
    p.halves = 1;
    if (grouped) {
        if (splits <= 0) splits = gr_ranges(tiles, splits < 0 ? (M + tokens - 1) / tokens : experts, slabs);
        if (splits == 2 && slabs >= 2 && bn <= 64 && tiles * live >= 2.0 * msgl_sm_count()) { p.halves = 2; splits = 1; }
    }
    // Blocks along y: no more than the runs of up to bn rows that the experts can have, and not many more than a random choice gives (one an
    // expert): blocks without a run are not free (128 experts, 8,192 rows: 73 rows of them added 12 us to 265).
    const long long most_runs = (long long)(M < experts ? M : experts) + M / bn, usual = experts + (experts > 128 ? experts / 16 : 8);
    const long long own_runs = !grouped ? 1 : most_runs < usual ? most_runs : usual < 65535 ? usual : 65535, runs = own_runs + (apart_rows + bn - 1) / bn;
    gr_plan((long long)(tiles * live), slabs, bn, p.splits, p.stages, splits, per_sm);
    p.tmem_cols = 32;
    while (p.tmem_cols < (unsigned)bn) p.tmem_cols *= 2;
    if (p.halves == 2) p.tmem_cols *= 2;
    const size_t smem = (size_t)p.stages * (GR_A_BYTES + (unsigned)bn * 128u) + GR_HEAD_BYTES + 1024u;
#define GR_GO(MODE, T) (grouped ? gr_launch<MODE, T, true>(xm, wm, w2m, p, tiles, (int)runs, smem, stream) : gr_launch<MODE, T, false>(xm, wm, w2m, p, tiles, 1, smem, stream))
    if (out_f32) return mode == GR_PLAIN ? GR_GO(GR_PLAIN, float) : MSGL_ERR_DTYPE;
    switch (mode) {
        case GR_PLAIN: return GR_GO(GR_PLAIN, __nv_bfloat16);
        case GR_SILU: return GR_GO(GR_SILU, __nv_bfloat16);
        case GR_RELU: return grouped ? MSGL_ERR_SIZE : gr_launch<GR_RELU, __nv_bfloat16, false>(xm, wm, w2m, p, tiles, 1, smem, stream);      // no experts with it
        default: return GR_GO(GR_CLAMPED, __nv_bfloat16);
    }
#undef GR_GO
}

MSGL_API int msgl_gemm_rows_apart(const void* W, const void* W2, const void* X, const void* bias, void* out, int M, int n_out, int K, long long ldx, long long ldo,
                                  int mode, int out_f32, float limit, int experts, const int* ends, int tokens, int splits, int per_sm, void* status, cudaStream_t stream) {
    return gr_product(W, W2, X, bias, out, M, n_out, K, ldx, ldo, mode, out_f32, limit, experts, ends, tokens, splits, per_sm, false, status, stream);
}
MSGL_API int msgl_gemm_rows(const void* W, const void* X, const void* bias, void* out, int M, int n_out, int K, long long ldx, long long ldo,
                            int mode, int out_f32, float limit, int experts, const int* ends, int tokens, int splits, int per_sm, void* status, cudaStream_t stream) {
    return gr_product(W, nullptr, X, bias, out, M, n_out, K, ldx, ldo, mode, out_f32, limit, experts, ends, tokens, splits, per_sm, false, status, stream);
}
// the plain product with weights that the launch before this one may write
MSGL_API int msgl_gemm_rows_plain(const void* W, const void* X, const void* bias, void* out, int M, int n_out, int K, long long ldx, long long ldo, int out_f32, void* status,
                                  cudaStream_t stream) {
    return gr_product(W, nullptr, X, bias, out, M, n_out, K, ldx, ldo, GR_PLAIN, out_f32, 0.f, 0, nullptr, 0, 0, 0, true, status, stream);
}
