// Weight-streaming matrix product for decode: out[M, N] = x[M, K] . W[N, K]^T with M <= 32 tokens, for weights of some size (gemm_small_m.cu has the others
// up to 8 tokens).
//
// With so few tokens the product is bound by reading W once from HBM, so the kernel is built around that stream:
//   * one block an SM takes an equal share of the output columns (rows of W) and all of K, in passes of up to 16 MT rows;
//   * a round of a pass is 576 elements of K: one TMA copy (W as [N][K / 64][64], boxes of rows x 9 x 64, 128-byte swizzle; gated: two) brings nine chunks
//     of 64 elements of every row, a chunk a warp.  With nine of them the rows of a chunk lie 1,152 bytes apart and change their place in the swizzle from row to row, so
//     that ldmatrix meets no bank twice.  The rounds of all passes are one stream through a ring of stages; one thread of a tenth warp asks for
//     a round as soon as the nine warps have read the stage's last one;
//   * up to 8 tokens weights are nobody's output, so the ring's first rounds are on their way before the wait for the kernel before this one (beyond, where products went to the
//     library, they are asked into L2), and the next kernel may
//     start behind that wait: of two products in a row the second has its first weights in shared memory when the first ends;
//   * x comes beside them by cp.async, a chunk a warp, on the same barriers; both go to mma.sync m16n8k16 by ldmatrix, the tokens on its n dimension (8 per n-block), fp32 accumulate;
//   * the warps' partial sums are added in warp order through shared memory (a fixed order, so
//     the result does not depend on timing), then bias / SwiGLU and one rounding to the output type.
//
// Gated modes (SwiGLU, ReGLU): W is [2I, K] with the gate rows first; a tile of 16 rows is 8 gate rows and the
// 8 up rows that belong to them, which land in the two row halves of the accumulator fragment, so
// out[M, I] = act(gate (+ bias)) * (up (+ bias)) is formed in registers and the [M, 2I] intermediate never exists.
//
// Which sizes come here is `_stream_rule` in ops.py, with the figures: not those where passes of few rounds, copies a chunk (K no multiple of 64) or, from 9 rows on, passes and the reads of x cost more
// than the kernels that have the others.
//
// What bounds it: the stream of W (8B, 1 token: gate/up and down 302 MB in 48.4 us, 6.2 TB/s; before, in blocks of 16 rows by cp.async of 16 bytes, 53.5), and with small weights the
// chain from the wait to the last store (0.6B feed-forward: 7.1 us a layer for 19 MB, before 8.2).  us of a product in a chain of them, before / now, 1 row: [4096, 4096] 8.0 / 7.3,
// [5120, 5120] 12.6 / 10.0 (320 blocks on 148 SMs before), [4096, 12288] 19.4 / 17.4, gated [24576, 4096] 35.9 / 33.5, [51200, 5120] 81.7 / 77.3; 8 rows: 8.5 / 7.9, 13.4 / 10.8, 20.2 / 18.0, 36.9 / 34.0,
// 84.8 / 84.0.  Tried: every warp copying for itself, a chunk of 64 elements a time (by cp.async of 16 bytes 35 % behind the old kernel: the copies' instructions; by TMA 2 to 8 %
// behind this one, x by TMA too 0.6 us a product); x straight into registers (28.2 -> 36.7 us for four 0.6B feed-forwards: the loads of later rounds come too late); tiles of 32 rows at most
// (28.2 -> 32.6: a pass more); rings of 104 and 144 KB (8B, 1 token: 109.7 and 104.6 us of two layers, 96.9 with 176 KB).
//
// Requirements (checked by the entry point, which returns MSGL_ERR_SIZE otherwise and the caller
// uses the library GEMM): bfloat16 inputs, K % 32 == 0, N % 16 == 0 (I % 8 == 0 in gated modes),
// 16-byte aligned rows.  Every wait for a copy is bounded; a block that gives up sets status[2] (the host raises) once its copies have landed.
#include "common.cuh"
#include "tc_common.cuh"

constexpr int GST_WARPS = 9, GST_THREADS = GST_WARPS * 32 + 32;      // a chunk a warp; lane 0 of the last warp asks for the copies
constexpr int GST_MAX_STAGES = 16;
constexpr int GST_RING = 176 * 1024;      // bytes of a block's ring at most
constexpr unsigned GST_ROW = GST_WARPS * 128u;
constexpr int GST_MAX_TILES = 3, GST_MAX_ROWS = 32;

__device__ __forceinline__ void gst_mma(float (&c)[4], const unsigned (&a)[4], unsigned b0, unsigned b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void gst_ldmatrix(unsigned (&r)[4], unsigned addr) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(addr) : "memory");
}
__device__ __forceinline__ void gst_load3(unsigned dst, const CUtensorMap* map, int chunk, int row, unsigned bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];\n"
                 ::"r"(dst), "l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(chunk), "r"(row), "r"(bar) : "memory");
}
__device__ __forceinline__ void gst_ask3(const CUtensorMap* map, int chunk, int row) {
    asm volatile("cp.async.bulk.prefetch.tensor.3d.L2.global.tile [%0, {%1, %2, %3}];\n" ::"l"(reinterpret_cast<unsigned long long>(map)), "r"(0), "r"(chunk), "r"(row) : "memory");
}
__device__ __forceinline__ void gst_consumers_sync() { asm volatile("bar.sync 1, %0;\n" ::"n"(GST_WARPS * 32) : "memory"); }

template <typename OutT> __device__ __forceinline__ void gst_store(OutT* p, float v);
template <> __device__ __forceinline__ void gst_store<float>(float* p, float v) { *p = v; }
template <> __device__ __forceinline__ void gst_store<__nv_bfloat16>(__nv_bfloat16* p, float v) { *p = __float2bfloat16_rn(v); }

struct StreamParams {
    const __nv_bfloat16* X;
    const __nv_bfloat16* bias;
    void* out;
    int* status;
    long long ldx, ldo;
    int M, N, K;                 // N: output columns
    int share, per_pass, passes; // output columns of a block, of a pass (of the last ones maybe fewer), passes of a block
    int stages;
    int bufs;                    // of the warps' sums
    int asked;                   // weights are only asked into L2 ahead of the wait: the kernel before this one may be the one that writes them
    int ragged;                  // K is no multiple of 64: the map is [rows][K] with boxes of rows x 64, a copy a chunk; the rows of a chunk lie back to back
    unsigned half;               // bytes of a stage, gated: of its gate rows and of its up rows; a multiple of 1,024
};

// a pass has up to 16 MT output columns (gated: 8 MT); up to 8 NB tokens
template <int NB, int MT, int GLU, typename OutT>
__global__ void __launch_bounds__(GST_THREADS) gemm_stream_kernel(const __grid_constant__ CUtensorMap wmap, const StreamParams p) {
    extern __shared__ __align__(1024) unsigned char gs_smem[];
    constexpr int PITCH = 16 * MT + 4;
    const unsigned base = tc_smem_u32(gs_smem), ring = (base + 1023u) & ~1023u, stage_bytes = GLU ? 2u * p.half : p.half;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, S = p.stages;
    const unsigned x_bytes = ((unsigned)(GST_WARPS * p.M) * 128u + 1023u) & ~1023u, x_ring = ring + (unsigned)S * stage_bytes, bars = x_ring + (unsigned)S * x_bytes;
    auto bar_full = [&](int s) { return bars + 16u * (unsigned)s; };
    auto bar_empty = [&](int s) { return bars + 16u * (unsigned)s + 8u; };
    const int o_begin = p.share * (int)blockIdx.x, chunks = (p.K + 63) / 64, rounds = (chunks + GST_WARPS - 1) / GST_WARPS, total = p.passes * rounds;

    if (warp == GST_WARPS) {
        int ld_round = 0, ld_row = o_begin;
        auto load = [&](int st) {
            const unsigned dst = ring + (unsigned)st * stage_bytes, b = bar_full(st);
            const unsigned rows = (GLU ? 2u : 1u) * (unsigned)p.per_pass;
            if (!p.ragged) {
                tc_mbar_expect_tx(b, rows * GST_ROW);
                gst_load3(dst, &wmap, ld_round * GST_WARPS, ld_row, b);
                if (GLU) gst_load3(dst + p.half, &wmap, ld_round * GST_WARPS, p.N + ld_row, b);
            } else {
                const int c0 = ld_round * GST_WARPS, n = min(GST_WARPS, chunks - c0);
                tc_mbar_expect_tx(b, rows * 128u * (unsigned)n);
                for (int c = 0; c < n; ++c) {
                    tc_tma_load(dst + (unsigned)(c * p.per_pass) * 128u, &wmap, (c0 + c) * 64, ld_row, b);
                    if (GLU) tc_tma_load(dst + p.half + (unsigned)(c * p.per_pass) * 128u, &wmap, (c0 + c) * 64, p.N + ld_row, b);
                }
            }
            if (++ld_round == rounds) { ld_round = 0; ld_row += p.per_pass; }
        };
        const int first = min(S, total);
        if (lane == 0) {
            for (int s = 0; s < S; ++s) { tc_mbar_init(bar_full(s), 1 + GST_WARPS * 32); tc_mbar_init(bar_empty(s), GST_WARPS); }
            asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
            if (!p.asked) {
                for (int i = 0; i < first; ++i) load(i);
            } else if (!p.ragged) {
                for (int i = 0, row = o_begin, r = 0; i < first; ++i) {
                    gst_ask3(&wmap, r * GST_WARPS, row);
                    if (GLU) gst_ask3(&wmap, r * GST_WARPS, p.N + row);
                    if (++r == rounds) { r = 0; row += p.per_pass; }
                }
            }
        }
        __syncthreads();
        if (lane == 0) {
            pdl_wait();
            if (p.asked)
                for (int i = 0; i < first; ++i) load(i);
            pdl_small();    // (not ahead of the wait: a kernel may then take for finished what was launched before this one)
            for (int i = first, st = 0, phase = 0; i < total; ++i) {
                if (!tc_mbar_wait(bar_empty(st), (unsigned)phase)) break;
                load(st);
                if (++st == S) { st = 0; phase ^= 1; }
            }
        }
        return;
    }
    float* red = reinterpret_cast<float*>(gs_smem + (bars - base) + GST_MAX_STAGES * 16);      // [bufs][GST_WARPS][M][PITCH]
    const int g = lane >> 2, t = lane & 3, r8 = lane & 7;
    __syncthreads();                                 // the barriers are there
    pdl_wait();

    // x of the warp's chunk of a round: 16 bytes a lane into the warp's place of the stage, on the stage's barrier as well; zeros behind the last element of K
    const int x_col = (lane & 7) * 8;
    const __nv_bfloat16* x_src = p.X + (size_t)(lane >> 3) * p.ldx;
    int x_round = 0;
    auto load_x = [&](int st) {
        const int k = (x_round * GST_WARPS + warp) * 64 + x_col, n16 = k < p.K ? 16 : 0;
        const unsigned to = x_ring + (unsigned)st * x_bytes + (unsigned)(warp * p.M) * 128u;
#pragma unroll
        for (int q = 0; q < 2 * NB; ++q) {
            const int tok = 4 * q + (lane >> 3);
            const unsigned at = to + (unsigned)tok * 128u;
            if (tok < p.M)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(at + (((unsigned)(lane & 7) ^ (at >> 7 & 7u)) << 4)), "l"(x_src + (size_t)(4 * q) * p.ldx + (n16 ? k : 0)), "r"(n16) : "memory");
        }
        tc_cp_async_arrive(bar_full(st));
        if (++x_round == rounds) x_round = 0;
    };
    for (int i = 0; i < min(S, total); ++i) load_x(i);

    // fragments: lane l gives row l % 8 of the matrix l / 8 of an ldmatrix.  Rows that a pass does not have are what lies behind, and reach no column that is stored.
    const unsigned up = (unsigned)((lane >> 3) & 1), piece = (unsigned)(lane >> 4);
    const unsigned pitch = p.ragged ? 128u : GST_ROW, tile = (GLU ? 8u : 16u) * pitch, first_row = (unsigned)(p.ragged ? warp * p.per_pass : warp);      // (row r in place first_row + r pitch / 128)
    const unsigned a_off = (unsigned)r8 * pitch + first_row * 128u + up * (GLU ? p.half : 8u * pitch) + ((piece ^ ((unsigned)r8 + first_row & 7u)) << 4);
    unsigned x_off[NB];                              // (tokens that are not there: the last one)
#pragma unroll
    for (int nb = 0; nb < NB; ++nb) {
        const unsigned row = (unsigned)(warp * p.M + min(nb * 8 + r8, p.M - 1));
        x_off[nb] = row * 128u + (((unsigned)(lane >> 3) ^ (row & 7u)) << 4);
    }
    int stage = 0, phase = 0, done = 0, fail = 0;
    for (int ps = 0; ps < p.passes; ++ps) {
        float c[NB][MT][4];
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int mt = 0; mt < MT; ++mt) c[nb][mt][0] = c[nb][mt][1] = c[nb][mt][2] = c[nb][mt][3] = 0.f;
        for (int i = 0; i < rounds && !fail; ++i) {
            if (!__all_sync(0xffffffffu, tc_mbar_wait(bar_full(stage), (unsigned)phase))) { fail = 1; break; }
            if (i * GST_WARPS + warp < chunks) {
                const unsigned at = ring + (unsigned)stage * stage_bytes + a_off, xt = x_ring + (unsigned)stage * x_bytes;
#pragma unroll
                for (int h = 0; h < 2; ++h) {        // 32 elements of K
                    unsigned b[NB][4];
#pragma unroll
                    for (int nb = 0; nb < NB; ++nb) gst_ldmatrix(b[nb], (xt + x_off[nb]) ^ (unsigned)(h << 6));
#pragma unroll
                    for (int kk = 0; kk < 2; ++kk)
#pragma unroll
                        for (int mt = 0; mt < MT; ++mt) {
                            unsigned a[4];
                            gst_ldmatrix(a, (at + (unsigned)mt * tile) ^ (unsigned)((2 * h + kk) << 5));
#pragma unroll
                            for (int nb = 0; nb < NB; ++nb) gst_mma(c[nb][mt], a, b[nb][2 * kk], b[nb][2 * kk + 1]);
                        }
                }
            }
            __syncwarp();                            // all lanes have read the stage
            if (lane == 0) tc_mbar_arrive(bar_empty(stage));
            if (done + S < total) load_x(stage);
            ++done;
            if (++stage == S) { stage = 0; phase ^= 1; }
        }
        // the warps' sums -> shared memory, [token][row of the pass]; accumulator layout: c0, c1 = (row g, tokens 2t, 2t + 1), c2, c3 = row g + 8.  Two buffers in
        // turn (a pass writes one when every thread has read it in the pass before the last), or one
        const int per_warp = p.M * PITCH, buf = p.bufs == 2 ? ps & 1 : 0;
        float* mine = red + (buf * GST_WARPS + warp) * per_warp;
#pragma unroll
        for (int nb = 0; nb < NB; ++nb)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int tok = nb * 8 + 2 * t + e;
                if (tok < p.M) {
#pragma unroll
                    for (int mt = 0; mt < MT; ++mt) {
                        mine[tok * PITCH + mt * 16 + g] = c[nb][mt][e];
                        mine[tok * PITCH + mt * 16 + g + 8] = c[nb][mt][2 + e];
                    }
                }
            }
        gst_consumers_sync();
        constexpr int COLS = GLU ? 8 * MT : 16 * MT;
        const int o0 = ps * p.per_pass, n = min(min(p.per_pass, p.share - o0), p.N - o_begin - o0);
        const float* sums = red + buf * GST_WARPS * per_warp;
        for (int idx = threadIdx.x; idx < p.M * COLS; idx += GST_WARPS * 32) {
            const int tok = idx / COLS, o = idx - tok * COLS, col = o_begin + o0 + o;
            if (o >= n) continue;
            const float* at = sums + tok * PITCH + (GLU ? (o >> 3) * 16 + (o & 7) : o);
            float acc = 0.f, gated = 0.f;
#pragma unroll
            for (int w = 0; w < GST_WARPS; ++w) {
                acc += at[w * per_warp];
                if (GLU) gated += at[w * per_warp + 8];
            }
            if (p.bias != nullptr) {
                acc += __bfloat162float(p.bias[col]);
                if (GLU) gated += __bfloat162float(p.bias[(size_t)p.N + col]);
            }
            gst_store<OutT>(reinterpret_cast<OutT*>(p.out) + (size_t)tok * p.ldo + col, GLU ? glu_act<GLU>(acc) * gated : acc);
        }
        if (p.bufs == 1 && ps + 1 < p.passes) gst_consumers_sync();
    }
    if (fail) {                                      // what is under way lands before the block lets go of its shared memory
        const int asked = min(total, done + S);
        for (int i = done; i < asked; ++i) {
            tc_mbar_wait(bar_full(stage), (unsigned)phase);
            if (++stage == S) { stage = 0; phase ^= 1; }
        }
        if (lane == 0 && p.status != nullptr) atomicExch(p.status + 2, 1);
    }
}

// the tensor map of [rows][K / 64][64] in boxes of box_rows x 9 x 64, made once per (matrix, size) and kept
static bool gst_map(const void* W, long long rows, int K, int box_rows, CUtensorMap* out) {
    static std::mutex mu;
    static std::map<std::tuple<const void*, long long, int, int>, CUtensorMap> maps;
    const tc_encode_fn encode = tc_encoder();
    if (encode == nullptr) return false;
    std::lock_guard<std::mutex> lock(mu);
    const auto key = std::make_tuple(W, rows, K, box_rows);
    auto it = maps.find(key);
    if (it != maps.end()) { *out = it->second; return true; }
    if (maps.size() > 4096) maps.clear();
    CUtensorMap m;
    const cuuint64_t dims[3] = {64, (cuuint64_t)(K / 64), (cuuint64_t)rows};
    const cuuint64_t strides[2] = {128, (cuuint64_t)K * 2};
    const cuuint32_t box[3] = {64, GST_WARPS, (cuuint32_t)box_rows}, estr[3] = {1, 1, 1};
    if (encode(&m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 3, const_cast<void*>(W), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
        return false;
    maps.emplace(key, m);
    *out = m;
    return true;
}

template <int NB, int MT, int GLU, typename OutT>
static int gst_launch(const void* W, StreamParams p, int grid, cudaStream_t stream) {
    constexpr int COLS = GLU ? 8 * MT : 16 * MT;
    constexpr size_t FIXED = 1024 + GST_MAX_STAGES * 16, RED = sizeof(float) * GST_WARPS * (16 * MT + 4);
    auto* kernel = gemm_stream_kernel<NB, MT, GLU, OutT>;
    static MsglOncePerDevice attr_set;
    if (attr_set.due()) {      // first call on this device, never inside a stream capture
        if (cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024) != cudaSuccess) return msgl_check_launch();
        cudaFuncSetAttribute(kernel, cudaFuncAttributePreferredSharedMemoryCarveout, cudaSharedmemCarveoutMaxShared);      // room for the next kernel's blocks
        attr_set.mark();
    }
    p.passes = (p.share + COLS - 1) / COLS;
    p.per_pass = (p.share + p.passes - 1) / p.passes;
    p.half = ((unsigned)p.per_pass * GST_ROW + 1023u) & ~1023u;
    p.ragged = p.K & 63 ? 1 : 0;
    CUtensorMap wm;
    const long long rows = GLU ? 2LL * p.N : p.N;
    if (!(p.ragged ? tc_matrix_map(W, rows, p.K, (long long)p.K * 2, p.per_pass, &wm) : gst_map(W, rows, p.K, p.per_pass, &wm))) return MSGL_ERR_SIZE;
    const int total = p.passes * (((p.K + 63) / 64 + GST_WARPS - 1) / GST_WARPS);
    const size_t stage = (GLU ? 2 : 1) * (size_t)p.half, x_stage = ((size_t)GST_WARPS * p.M * 128 + 1023) / 1024 * 1024;
    p.bufs = p.passes > 1 && p.M <= 8 ? 2 : 1;
    const size_t sums = p.bufs * RED * p.M, room = 227 * 1024 - FIXED - sums;
    p.stages = (int)((room < GST_RING ? room : GST_RING) / (stage + x_stage));
    if (p.stages > GST_MAX_STAGES) p.stages = GST_MAX_STAGES;
    // full passes of five to eight tokens: with two stages a round is asked for when the one before it is read.  us at 8 rows, two / three, blocks of 16 rows: [20480, 2560] 21.3 / 19.4, 20.4;
    // [32000, 2048] 25.1 / 23.3, 24.6; [65536, 2048] 46.7 / 44.3, 44.4
    if (p.stages < 3) p.stages = 3 * (stage + x_stage) <= room ? 3 : 2;
    if (p.stages > total) p.stages = total;
    // fragments of rows that a pass does not have are read behind the last stage
    const size_t reach = p.ragged ? (size_t)(GST_WARPS - 1) * p.per_pass * 128 + COLS * 128 : (size_t)COLS * GST_ROW, over = reach > p.half ? reach - p.half : 0;
    size_t smem = FIXED + p.stages * (stage + x_stage) + sums;
    if (smem < 1024 + p.stages * stage + over) smem = 1024 + p.stages * stage + over;
    if (smem > 227 * 1024) return MSGL_ERR_SIZE;
    msgl_launch_pdl(kernel, dim3(grid), dim3(GST_THREADS), smem, stream, wm, p);
    return msgl_check_launch();
}

// mode: 0 = plain (out [M, N]), 1 / 2 = SwiGLU / ReGLU (W [2I, K], bias [2I], out [M, I], N = 2I).  out_f32: output type.
MSGL_API int msgl_gemm_stream(const void* W, const void* X, const void* bias, void* out, int M, int N, int K,
                               long long ldx, long long ldo, int mode, int out_f32, void* status, cudaStream_t stream) {
    if (M <= 0) return MSGL_OK;
    if (M > GST_MAX_ROWS || K <= 0 || (K & 31) || N <= 0 || (N & 15)) return MSGL_ERR_SIZE;
    if (((uintptr_t)W | (uintptr_t)X) & 15) return MSGL_ERR_ALIGN;
    if ((ldx & 7) != 0) return MSGL_ERR_ALIGN;
    if (mode < 0 || mode > 2) return MSGL_ERR_SIZE;
    const bool glu = mode != MSGL_GLU_NONE;
    if (glu && out_f32) return MSGL_ERR_DTYPE;
    StreamParams p = {};
    p.X = (const __nv_bfloat16*)X; p.ldx = ldx; p.bias = (const __nv_bfloat16*)bias; p.out = out; p.status = (int*)status; p.ldo = ldo;
    p.M = M; p.N = glu ? N / 2 : N; p.K = K; p.asked = M > 8;
    const int sms = msgl_sm_count();
    p.share = (p.N + sms - 1) / sms;
    if (p.share < 4) p.share = p.N < 4 ? p.N : 4;
    const int grid = (p.N + p.share - 1) / p.share;
    int tiles = (p.share + (glu ? 7 : 15)) / (glu ? 8 : 16);
    if (tiles > GST_MAX_TILES) tiles = GST_MAX_TILES;
#define GST_MT(NB, GLU, T) \
    (tiles == 1 ? gst_launch<NB, 1, GLU, T>(W, p, grid, stream) : tiles == 2 ? gst_launch<NB, 2, GLU, T>(W, p, grid, stream) : gst_launch<NB, 3, GLU, T>(W, p, grid, stream))
#define GST_GO(GLU, T) (M <= 8 ? GST_MT(1, GLU, T) : M <= 16 ? GST_MT(2, GLU, T) : M <= 24 ? GST_MT(3, GLU, T) : GST_MT(4, GLU, T))
    for (;; --tiles) {           // (fewer rows a pass where the sums of many tokens leave no room for two stages)
        const int code = mode == MSGL_GLU_SILU ? GST_GO(1, __nv_bfloat16) : mode == MSGL_GLU_RELU ? GST_GO(2, __nv_bfloat16) : out_f32 ? GST_GO(0, float) : GST_GO(0, __nv_bfloat16);
        if (code != MSGL_ERR_SIZE || tiles == 1) return code;
    }
#undef GST_GO
#undef GST_MT
}
