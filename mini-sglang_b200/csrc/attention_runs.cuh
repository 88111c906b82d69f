// Decode attention (bfloat16, head size 128, one new token a request, up to eight query heads a kv head; MIXED: the requests of a step that bring one) in one launch: the keys
// of all requests dealt out evenly over one block an SM, partial results merged by the block that comes last.
//
// A segment is one request under one kv head, cut into units of 16 keys (anchored at absolute positions; a page holds whole
// units).  Every block works out from the requests' lengths alone which units are its own:
//   * few keys (all requests together fit the blocks in pieces of RUN_UNITS units or more): a segment of u units has
//     max(1, u / RUN_UNITS) equal pieces, a block a piece (or one, where whole segments fill the blocks nearly evenly);
//   * many short segments: a warp takes whole segments, and no two share one (a segment costs a block 1.1 us beside its stream, a warp 0.6 and
//     0.4 a unit);
//   * otherwise the units of all segments are laid end to end and cut into as many runs of equal length as there are blocks; a
//     cut within RUN_SNAP units of a segment's edge moves onto the edge.
// Pieces of a segment lie in consecutive blocks.  A segment within one block is written out by it; of the others every block leaves
// its partial result in scratch memory, and the one that raises the segment's counter to its number of pieces merges them in the
// order of the keys and clears the counter.
//
// A block's eight warps take the units of its run in turn.  Every warp keeps a ring of ST units in shared memory, 4 KB of keys and
// 4 KB of values each (a unit's rows of one kv head lie back to back in the cache), filled by cp.async whole units ahead and
// across the edges of segments, so the stream goes on while a segment's eight partial results are merged.  The arithmetic is that of
// decode_t_run: keys on the M dimension of the mma with the head's elements permuted (16 bytes a lane), P through movmatrix, the
// exponentials' reference moved only where a score lies DEC_LAZY above it.
//
// Bound by the stream of keys and values (8 requests of 4,096 keys, 134 MB: 21 of the launch's 28 us from the first units asked for to the latest block's last one, 6.4 TB/s, part of them asked into L2 before that), then by
// the cut at its start (1.3 us, under the kernels ahead of it as far as they last) and the exchange of partial results at its end (2 to 4 us).  An attention layer
// before / with it, us (kernels of four warps with kv splits from the host and a merge of their own): 8B, 8 x 4,096 keys 58.7 / 51.8;
// 4B, 40 of 64 ... 6,000 76.6 / 58.2; 8B, 64 x 2,000 133.6 / 113; 1.7B, one of 130 18.2 / 14.3, 16 x 512 32.9 / 25.2, 64 of 4 ... 64 23.2 / 22.5.
// Rings of two units and of three are level but for 64 x 2,000 (113.0 / 114.8), so it is two (58 KB of an SM are then free for a block behind: norms and small products, not a ring of gemm_stream.cu).  Without
// RUN_HEAD the mixed case takes 70.6: the block that gets the short requests runs 49 us, the others 34.  Decoded tokens among prompt portions, launched behind the prefill tiles and
// ahead of their merges, so that its blocks take the SMs that the last tiles leave free (8B, 1,500, 333, 65, 1, 1, 1 tokens behind 0, 700, 4,000, 2,047, 511, 37: the
// layer 223.8 -> 213.7 us; before, 18 us of decode attention ahead of the tiles and a merge over all tokens of 9).
// Against the kernels with kv splits over 837 steps (12 pairs of head counts, 1 to 256 requests, keys alike, spread and short, pages of 16): 1.58 times as fast in the mean, four behind by 4 to 6 % (64 x 128 keys on 7 of 7
// heads 10.7 / 11.4, 5 x 128 on 64 of 64 8.8 / 9.3, 8 x 128 on 40 of 40 8.9 / 9.3, 17 x 600 on 32 of 32 35.6 / 36.9); pages of 48, 132 steps: 1.55, none behind.
#pragma once

constexpr int RUN_NW = 8;            // warps of a block
constexpr int RUN_ST = 2;            // units of a warp's ring
constexpr int RUN_UNITS = 16;        // units of a piece at least, where segments are cut by themselves
constexpr int RUN_SNAP = 6;          // a cut this close to a segment's edge moves onto it
constexpr int RUN_HEAD = 6;          // what a segment costs beside its units (its queries, its merge), in units
constexpr int RUN_WARP_UNITS = 16;   // longest segment where a warp takes whole segments
constexpr int RUN_MAX_B = 256;       // a thread a request
constexpr int RUN_D = 128;
constexpr int RUN_OLD = RUN_D + 4;   // floats of a row of the merge buffer
constexpr int RUN_THREADS = RUN_NW * 32;

struct RunParams {
    const __nv_bfloat16* q;          // [B, n_q, 128]
    __nv_bfloat16* out;
    const __nv_bfloat16* k_cache;
    const __nv_bfloat16* v_cache;
    const int* kv_len;               // [B]
    const int* block_table;          // [B, bt_stride]
    float* part_o;                   // [2 * blocks][8][128]
    float* part_ml;                  // [2 * blocks][8][2]
    int* count;                      // [B * n_kv], zero before and after
    const int* q_start;              // MIXED: [B + 1]; the requests with one token are taken
    int wait_last;                   // MIXED: q and the cache are written by kernels that are done when this one starts; it waits for the one before it at its end
    int B, n_q, n_kv, page_size, page_shift, bt_stride;
    float scale;
};

constexpr size_t run_smem_bytes() {
    return (size_t)RUN_NW * RUN_ST * 2 * 16 * RUN_D * 2 + (size_t)RUN_NW * 8 * RUN_OLD * 4 + (size_t)RUN_NW * 8 * 2 * 4 + (4 * RUN_MAX_B + 4) * 4;
}

static_assert(run_smem_bytes() + 256 <= 227 * 1024, "one block an SM");

// which segment a unit lies in, walked forward
struct RunCursor {
    int r, kvh, c0, u;               // request, kv head, first unit of the segment among all, units
};

template <bool MIXED>
__global__ void __launch_bounds__(RUN_THREADS, 1) attn_decode_runs_kernel(const RunParams p) {
    extern __shared__ __align__(128) unsigned char run_smem[];
    constexpr int UNIT_BYTES = 16 * RUN_D * 2;
    float* Om = reinterpret_cast<float*>(run_smem + (size_t)RUN_NW * RUN_ST * 2 * UNIT_BYTES);      // [NW][8][RUN_OLD]
    float* Mm = Om + RUN_NW * 8 * RUN_OLD;                                                          // [NW][8]
    float* Lm = Mm + RUN_NW * 8;                                                                    // [NW][8]
    int* pre = reinterpret_cast<int*>(Lm + RUN_NW * 8);                                             // [B + 1] units of the requests before
    __shared__ int4 sh_sum[RUN_NW];
    __shared__ int2 sh_run;
    __shared__ int4 sh_seg;                              // request, kv head, (by_piece) pieces of the segment, this block's
    __shared__ int sh_last;

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int g = lane >> 2, t = lane & 3;
    const int G = p.n_q / p.n_kv, NB = (int)gridDim.x, j = (int)blockIdx.x;

    // ---- the requests that are taken (MIXED: numbered anew), their units and pieces and the sums, a request a thread (lengths and first tokens come from
    // the step's fields, not from the kernel before this one)
    int* lens = pre + RUN_MAX_B + 4;                     // MIXED: of request i here its length, its number in the step and its token
    int* number = lens + RUN_MAX_B;
    int* token = number + RUN_MAX_B;
    int B = p.B, my_len = 0;
    if (MIXED) {
        __shared__ int sh_taken[RUN_NW];
        const int first = tid < p.B ? p.q_start[tid] : 0, len = tid < p.B ? p.kv_len[tid] : 0;
        const bool taken = tid < p.B && p.q_start[tid + 1] - first == 1;
        const unsigned all = __ballot_sync(0xffffffffu, taken);
        if (lane == 0) sh_taken[warp] = __popc(all);
        __syncthreads();
        int at = __popc(all & ((1u << lane) - 1u));
        B = 0;
#pragma unroll
        for (int w = 0; w < RUN_NW; ++w) {
            if (w < warp) at += sh_taken[w];
            B += sh_taken[w];
        }
        if (taken) { lens[at] = len; number[at] = tid; token[at] = first; }
        __syncthreads();
        if (B == 0) { pdl_wait(); return; }
        if (tid < B) my_len = lens[tid];
    } else if (tid < p.B) {
        my_len = p.kv_len[tid];
    }
    auto leave = [&]() { if (MIXED && p.wait_last) pdl_wait(); };      // (whoever waits for this kernel counts on the one before it as well)
    auto len_of = [&](int r) { return MIXED ? lens[r] : p.kv_len[r]; };
    auto token_of = [&](int r) { return MIXED ? token[r] : r; };
    const int my_u = tid < B ? max(my_len + 15, 16) >> 4 : 0;
    int my_pre = my_u, my_pc = my_u > 0 ? max(1, my_u / RUN_UNITS) : 0, my_pcs = my_pc;                   // of the requests before this one, at last
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int v = __shfl_up_sync(0xffffffffu, my_pre, o), w = __shfl_up_sync(0xffffffffu, my_pcs, o);
        if (lane >= o) { my_pre += v; my_pcs += w; }
    }
    const int most_u = __reduce_max_sync(0xffffffffu, my_u);
    if (lane == 31) sh_sum[warp] = make_int4(my_pre, my_pcs, most_u, 0);
    __syncthreads();
    int U = 0, pieces_all = 0, longest = 0;
    my_pre -= my_u;
    my_pcs -= my_pc;
#pragma unroll
    for (int w = 0; w < RUN_NW; ++w) {
        const int4 v = sh_sum[w];
        if (w < warp) { my_pre += v.x; my_pcs += v.y; }
        U += v.x;
        pieces_all += v.y;
        longest = max(longest, v.z);
    }
    if (tid < B) pre[tid] = my_pre;
    if (tid == 0) pre[B] = U;
    const int S = B * p.n_kv;                          // segments
    if (pieces_all * p.n_kv > NB && S <= NB && 3 * longest * NB <= 4 * U * p.n_kv) {      // a block a segment is nearly even, and nothing is left to merge
        pieces_all = B;
        my_pcs = tid;
        my_pc = tid < B ? 1 : 0;
    }
    const bool by_piece = pieces_all * p.n_kv <= NB;
    const bool by_warp = !by_piece && longest <= RUN_WARP_UNITS && (4 * longest + 6) * NB < 11 * S;
    U *= p.n_kv;

    // ---- this block's run of units [lo, hi) of the segments laid end to end, and the segment it starts in
    const int V = U + RUN_HEAD * S, per = V / NB, rest = V - per * NB;      // with every segment's head ahead of its units
    if (by_piece) {
        if (j >= pieces_all * p.n_kv) { leave(); return; }
        const int in_r = j - my_pcs * p.n_kv;
        if (in_r >= 0 && in_r < my_pc * p.n_kv) {
            const int kvh = in_r / my_pc, piece = in_r - kvh * my_pc, c0 = my_pre * p.n_kv + kvh * my_u;
            sh_seg = make_int4(tid, kvh, my_pc, piece);
            sh_run = make_int2(c0 + my_u * piece / my_pc, c0 + my_u * (piece + 1) / my_pc);
        }
    } else if (!by_warp) {
        // the thread whose request holds the raw cut floor(V i / NB) finds the cut: a segment's edge or a unit within it
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int i = j + e, in_r = i * per + i * rest / NB - (my_pre + RUN_HEAD * tid) * p.n_kv;
            if (i == NB && tid == 0) sh_run.y = U;
            if (tid < B && in_r >= 0 && in_r < (my_u + RUN_HEAD) * p.n_kv) {
                const int kvh = in_r / (my_u + RUN_HEAD), off = in_r - kvh * (my_u + RUN_HEAD) - RUN_HEAD;
                const int unit = off <= RUN_SNAP ? 0 : my_u - off <= RUN_SNAP ? my_u : off, x = my_pre * p.n_kv + kvh * my_u + unit;
                if (e == 1) { sh_run.y = x; continue; }
                const bool next = unit == my_u, next_r = next && kvh + 1 == p.n_kv;      // a cut at the end: the run starts with the segment behind
                sh_run.x = x;
                sh_seg = make_int4(next_r ? tid + 1 : tid, next_r ? 0 : next ? kvh + 1 : kvh, 1, 0);
            }
        }
    }
    __syncthreads();
    int lo, hi, seg_pieces = 1, piece = 0;
    RunCursor seg;
    if (by_warp) {                                       // segments [s0, s1) in order are this warp's
        const int idx = warp * NB + j, W = NB * RUN_NW, s0 = S * idx / W, s1 = S * (idx + 1) / W;
        if (s0 >= s1) { leave(); return; }                     // (no barrier of the block lies behind)
        seg.r = s0 / p.n_kv;
        seg.kvh = s0 - seg.r * p.n_kv;
        const int r1 = (s1 - 1) / p.n_kv;
        hi = pre[r1] * p.n_kv + (s1 - r1 * p.n_kv) * (pre[r1 + 1] - pre[r1]);
    } else {
        lo = sh_run.x; hi = sh_run.y;
        seg_pieces = sh_seg.z; piece = sh_seg.w;
        if (lo >= hi) { leave(); return; }
        seg.r = sh_seg.x;
        seg.kvh = sh_seg.y;
    }
    seg.u = pre[seg.r + 1] - pre[seg.r];
    seg.c0 = pre[seg.r] * p.n_kv + seg.kvh * seg.u;
    if (by_warp) lo = seg.c0;

    // the warp's units: x0, x0 + 8, ... below hi (by_warp: every one)
    static_assert(RUN_NW == 8, "a shift below");
    const int x0 = by_warp ? lo : lo + warp, shift = by_warp ? 0 : 3, n_my = max(hi - x0 + (1 << shift) - 1, 0) >> shift;
    unsigned char* my_ring = run_smem + (size_t)warp * RUN_ST * 2 * UNIT_BYTES;
    const unsigned ring_u32 = smem_u32(my_ring);

    // ---- the warp's loader: unit i lies in the segment of `ld`; its page is looked up an iteration before it is asked for
    RunCursor ld = seg;
    struct Place { int page, slot, kvh, rows; };         // rows of the unit that hold keys the query sees
    auto place_of = [&](int i) -> Place {
        Place w;
        if (i >= n_my) { w.page = 0; w.slot = 0; w.kvh = 0; w.rows = 0; return w; }
        const int x = x0 + (i << shift);
        while (x >= ld.c0 + ld.u) {
            ld.c0 += ld.u;
            if (++ld.kvh == p.n_kv) { ld.kvh = 0; ++ld.r; ld.u = pre[ld.r + 1] - pre[ld.r]; }
        }
        const int key = (x - ld.c0) << 4;
        const int pi = p.page_shift >= 0 ? key >> p.page_shift : key / p.page_size;
        w.slot = key - pi * p.page_size;
        w.kvh = ld.kvh;
        w.rows = len_of(ld.r) - key;
        w.page = w.rows > 0 ? p.block_table[(size_t)(MIXED ? number[ld.r] : ld.r) * p.bt_stride + pi] : 0;
        return w;
    };
    auto offset_of = [&](const Place& w) -> size_t { return (((size_t)w.page * p.n_kv + w.kvh) * p.page_size + w.slot) * RUN_D; };
    auto load = [&](int i, const Place& w) {
        const unsigned st = ring_u32 + (unsigned)(i % RUN_ST) * 2 * UNIT_BYTES;
        const size_t off = offset_of(w) + lane * 8;
        const int c = lane & 15;
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int row = 2 * m + (lane >> 4);
            cp_async16_u32(st + row * (RUN_D * 2) + ((c ^ ((row & 1) << 2)) << 4), p.k_cache + off + m * 256, row < w.rows);
        }
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int row = 2 * m + (lane >> 4);
            cp_async16_u32(st + UNIT_BYTES + row * (RUN_D * 2) + ((c ^ (row & 7)) << 4), p.v_cache + off + m * 256, row < w.rows);
        }
    };
    auto ask_l2 = [&](const Place& w) {                   // the unit's 32 lines of keys and 32 of values
        if (w.rows <= (lane >> 1)) return;
        const size_t off = offset_of(w) + lane * 64;
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.k_cache + off));
        asm volatile("prefetch.global.L2 [%0];\n" ::"l"(p.v_cache + off));
    };
    Place at[RUN_ST];
#pragma unroll
    for (int i = 0; i < RUN_ST; ++i) at[i] = place_of(i);
#pragma unroll
    for (int i = 0; i < RUN_ST; ++i) ask_l2(at[i]);
    if (!MIXED || !p.wait_last) {
        pdl_wait();
        pdl_after_wait();
    }
#pragma unroll
    for (int i = 0; i < RUN_ST - 1; ++i) {
        if (i < n_my) load(i, at[i]);
        cp_async_commit();
    }
    Place next = at[RUN_ST - 1];

    // Q as B operand: lane (g, t) holds Q[head g of the group][32 m + 8 t .. + 7]
    uint4 qf[4];
    auto load_q = [&](int r, int kvh) {
        const __nv_bfloat16* src = p.q + ((size_t)token_of(r) * p.n_q + (size_t)kvh * G + (g < G ? g : 0)) * RUN_D + 8 * t;
#pragma unroll
        for (int m = 0; m < 4; ++m) qf[m] = g < G ? *reinterpret_cast<const uint4*>(src + 32 * m) : make_uint4(0u, 0u, 0u, 0u);
    };
    load_q(seg.r, seg.kvh);
    const float sc = p.scale * 1.4426950408889634f;
    int i = 0;
    bool first_segment = true;
    for (int begin = lo; begin < hi;) {
        const int end = min(hi, seg.c0 + seg.u);
        const int pos = len_of(seg.r) - 1;
        float o[8][4];
#pragma unroll
        for (int mt = 0; mt < 8; ++mt) o[mt][0] = o[mt][1] = o[mt][2] = o[mt][3] = 0.f;
        float m_c[2] = {-INFINITY, -INFINITY}, l_c[2] = {0.f, 0.f};

        for (; i < n_my; ++i) {
            const int x = x0 + (i << shift);
            if (x >= end) break;
            cp_async_wait<RUN_ST - 2>();
            __syncwarp();                     // unit i has come for all lanes, and all have left the stage that is filled next
            if (i + RUN_ST - 1 < n_my) load(i + RUN_ST - 1, next);
            cp_async_commit();
            next = place_of(i + RUN_ST);
            const unsigned st = ring_u32 + (unsigned)(i % RUN_ST) * 2 * UNIT_BYTES;
            // ---- S^T = K Q^T
            float s[4] = {0.f, 0.f, 0.f, 0.f}, s2[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                uint4 kl, kh;
                const unsigned a = st + g * (RUN_D * 2) + (((4 * m + t) ^ ((g & 1) << 2)) << 4);
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(kl.x), "=r"(kl.y), "=r"(kl.z), "=r"(kl.w) : "r"(a));
                asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(kh.x), "=r"(kh.y), "=r"(kh.z), "=r"(kh.w) : "r"(a + 8 * RUN_D * 2));
                mma_bf16_regs(s, kl.x, kh.x, kl.y, kh.y, qf[m].x, qf[m].y);
                mma_bf16_regs(s2, kl.z, kh.z, kl.w, kh.w, qf[m].z, qf[m].w);
            }
            const int key0 = (x - seg.c0) << 4;
            float v[4];
            bool behind = false;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                v[e] = (s[e] + s2[e]) * sc;
                if (key0 + 15 > pos && key0 + g + ((e & 2) ? 8 : 0) > pos) v[e] = -INFINITY;
                behind = behind || v[e] > m_c[e & 1] + DEC_LAZY;
            }
            if (__any_sync(0xffffffffu, behind)) {
                float alpha[2];
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    float mx = fmaxf(v[e], v[e + 2]);
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 4));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 8));
                    mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, 16));
                    const float mn = fmaxf(m_c[e], mx);
                    const float mu = (mn == -INFINITY) ? 0.f : mn;
                    alpha[e] = fast_exp2(m_c[e] - mu);
                    m_c[e] = mn;
                    l_c[e] *= alpha[e];
                }
#pragma unroll
                for (int mt = 0; mt < 8; ++mt) {
                    o[mt][0] *= alpha[0]; o[mt][1] *= alpha[1];
                    o[mt][2] *= alpha[0]; o[mt][3] *= alpha[1];
                }
            }
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const float mu = (m_c[e] == -INFINITY) ? 0.f : m_c[e];
                v[e] = fast_exp2(v[e] - mu);
                v[e + 2] = fast_exp2(v[e + 2] - mu);
                l_c[e] += v[e] + v[e + 2];
            }
            const unsigned pb0 = movmatrix_trans(pack_bf16(v[0], v[1])), pb1 = movmatrix_trans(pack_bf16(v[2], v[3]));
            // ---- O^T += V^T P^T
            const int vr = (lane & 7) + ((lane >> 4) & 1) * 8;
            const unsigned va = st + UNIT_BYTES + vr * (RUN_D * 2);
#pragma unroll
            for (int mt = 0; mt < 8; ++mt) {
                unsigned a[4];
                ldmatrix_x4_trans_u32(a, va + (((2 * mt + ((lane >> 3) & 1)) ^ (vr & 7)) << 4));
                mma_bf16_16816(o[mt], a, pb0, pb1);
            }
        }
        if (end >= hi) pdl_late();
        else load_q(seg.kvh + 1 < p.n_kv ? seg.r : seg.r + 1, seg.kvh + 1 < p.n_kv ? seg.kvh + 1 : 0);      // the next segment's

        // ---- the warps' results through shared memory, added in warp order
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            l_c[e] += __shfl_xor_sync(0xffffffffu, l_c[e], 4);
            l_c[e] += __shfl_xor_sync(0xffffffffu, l_c[e], 8);
            l_c[e] += __shfl_xor_sync(0xffffffffu, l_c[e], 16);
        }
        if (by_warp) __syncwarp();
        else if (!first_segment) __syncthreads();    // the segment before has been read
        first_segment = false;
#pragma unroll
        for (int mt = 0; mt < 8; ++mt)
#pragma unroll
            for (int e = 0; e < 4; ++e)
                Om[(warp * 8 + 2 * t + (e & 1)) * RUN_OLD + mt * 16 + g + ((e & 2) ? 8 : 0)] = o[mt][e];
        if (g == 0) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                Mm[warp * 8 + 2 * t + e] = m_c[e];
                Lm[warp * 8 + 2 * t + e] = l_c[e];
            }
        }
        const size_t row0 = (size_t)token_of(seg.r) * p.n_q + (size_t)seg.kvh * G;
        // pieces of this segment, this block's among them
        int pieces = seg_pieces, mine = piece;
        if (by_warp) {
            __syncwarp();
            for (int c = 0; c < G; ++c) {
                const float L = Lm[warp * 8 + c], inv = L > 0.f ? 1.f / L : 0.f;
                const float4 v = *reinterpret_cast<const float4*>(Om + (warp * 8 + c) * RUN_OLD + lane * 4);
                *reinterpret_cast<uint2*>(p.out + (row0 + c) * RUN_D + lane * 4) = make_uint2(pack_bf16(v.x * inv, v.y * inv), pack_bf16(v.z * inv, v.w * inv));
            }
        } else if (!by_piece) {
            pieces = 1; mine = 0;
            if (begin > seg.c0 || end < seg.c0 + seg.u) {      // the cuts inside are those of c + SNAP < floor(V i / NB) < c + u - SNAP; piece k in block first_cut - 1 + k
                const int c = seg.c0 + RUN_HEAD * (seg.r * p.n_kv + seg.kvh + 1);
                const int first_cut = (int)(((long long)(c + RUN_SNAP + 1) * NB + V - 1) / V), last_cut = (int)(((long long)(c + seg.u - RUN_SNAP) * NB + V - 1) / V) - 1;
                pieces = last_cut - first_cut + 2;
                mine = j - (first_cut - 1);
            }
        }
        if (!by_warp) {
            __syncthreads();
            const int slot = 2 * j + (mine == 0 ? 1 : 0);        // a run has at most one segment's first piece (its end) and one's later one (its start)
            for (int idx = tid; idx < G * 32; idx += RUN_THREADS) {
                const int c = idx >> 5, col = (idx & 31) * 4;
                float M = -INFINITY;
#pragma unroll
                for (int w = 0; w < RUN_NW; ++w) M = fmaxf(M, Mm[w * 8 + c]);
                const float Mu = (M == -INFINITY) ? 0.f : M;
                float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                float L = 0.f;
#pragma unroll
                for (int w = 0; w < RUN_NW; ++w) {
                    const float f = fast_exp2(Mm[w * 8 + c] - Mu);
                    const float4 ov = *reinterpret_cast<const float4*>(Om + (w * 8 + c) * RUN_OLD + col);
                    acc.x = fmaf(f, ov.x, acc.x); acc.y = fmaf(f, ov.y, acc.y);
                    acc.z = fmaf(f, ov.z, acc.z); acc.w = fmaf(f, ov.w, acc.w);
                    L += f * Lm[w * 8 + c];
                }
                if (pieces == 1) {
                    const float inv = L > 0.f ? 1.f / L : 0.f;
                    *reinterpret_cast<uint2*>(p.out + (row0 + c) * RUN_D + col) = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
                } else {
                    *reinterpret_cast<float4*>(p.part_o + ((size_t)slot * 8 + c) * RUN_D + col) = acc;
                    if (col == 0) *reinterpret_cast<float2*>(p.part_ml + ((size_t)slot * 8 + c) * 2) = make_float2(M, L);
                }
            }
            if (pieces > 1) {
                __syncthreads();
                int* count = p.count + (size_t)seg.r * p.n_kv + seg.kvh;
                if (tid == 0) {                          // the fence behind the barrier covers what the block's other threads wrote
                    __threadfence();
                    sh_last = atomicAdd(count, 1) == pieces - 1;
                    __threadfence();
                }
                __syncthreads();
                if (sh_last) {                           // all pieces are there: merged in the order of the keys
                    const int b0 = j - mine;             // the block of piece 0
                    if (tid == 0) *count = 0;
                    for (int c = warp; c < G; c += RUN_NW) {      // a warp a head: lane k knows the weight of piece k (of 32 at a time), four elements a lane
                        auto row_of = [&](int k) -> size_t { return (size_t)(2 * (b0 + k) + (k == 0 ? 1 : 0)) * 8 + c; };
                        float2 ml = make_float2(-INFINITY, 0.f);
                        if (lane < pieces) ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + row_of(lane) * 2));
                        float M = ml.x;
                        for (int k = lane + 32; k < pieces; k += 32) M = fmaxf(M, __ldcg(p.part_ml + row_of(k) * 2));
                        M = warp_max(M);
                        const float Mu = (M == -INFINITY) ? 0.f : M;
                        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
                        float L = 0.f;
                        for (int k0 = 0; k0 < pieces; k0 += 32) {
                            if (k0 > 0) ml = k0 + lane < pieces ? __ldcg(reinterpret_cast<const float2*>(p.part_ml + row_of(k0 + lane) * 2)) : make_float2(-INFINITY, 0.f);
                            const float w = exp2f(ml.x - Mu);
                            L = fmaf(w, ml.y, L);
                            const int n = min(pieces - k0, 32);
#pragma unroll 8
                            for (int k = 0; k < n; ++k) {
                                const float4 ov = __ldcg(reinterpret_cast<const float4*>(p.part_o + row_of(k0 + k) * RUN_D + lane * 4));
                                const float f = __shfl_sync(0xffffffffu, w, k);
                                acc.x = fmaf(f, ov.x, acc.x); acc.y = fmaf(f, ov.y, acc.y);
                                acc.z = fmaf(f, ov.z, acc.z); acc.w = fmaf(f, ov.w, acc.w);
                            }
                        }
                        L = warp_sum(L);
                        const float inv = L > 0.f ? 1.f / L : 0.f;
                        *reinterpret_cast<uint2*>(p.out + (row0 + c) * RUN_D + lane * 4) = make_uint2(pack_bf16(acc.x * inv, acc.y * inv), pack_bf16(acc.z * inv, acc.w * inv));
                    }
                }
            }
        }
        // ---- the next segment
        begin = end;
        if (begin < hi) {
            seg.c0 += seg.u;
            if (++seg.kvh == p.n_kv) { seg.kvh = 0; ++seg.r; seg.u = pre[seg.r + 1] - pre[seg.r]; }
        }
    }
    cp_async_wait<0>();
    leave();
}

// q_start null: every request has one token, request r token r.  Else the requests with one token are taken, and with wait_last the kernel reads what it is given without waiting
// for the one launched before it: for a launch behind the prefill kernels, whose launch waited for all that wrote it (and whose own rows nobody reads here).
MSGL_API int msgl_attention_decode_runs(const void* q, void* out, const void* k_cache, const void* v_cache, const int* kv_len, const int* block_table,
                                        float* part_o, float* part_ml, int* count, const int* q_start, int wait_last, int B, int n_q, int n_kv, int page_size,
                                        int bt_stride, float scale, int blocks, cudaStream_t stream) {
    if (B <= 0) return MSGL_OK;
    if (B > RUN_MAX_B || n_kv <= 0 || n_q % n_kv != 0 || n_q / n_kv > 8 || page_size <= 0 || page_size % 16 != 0 || bt_stride <= 0 || blocks <= 0 || blocks > 4096 ||
        (long long)B * n_kv * ((long long)bt_stride * (page_size / 16) + 1) > 0x7fffffffLL / 2)
        return MSGL_ERR_SIZE;
    if (((uintptr_t)q | (uintptr_t)k_cache | (uintptr_t)v_cache | (uintptr_t)out | (uintptr_t)part_o | (uintptr_t)part_ml) & 15) return MSGL_ERR_ALIGN;
    if (part_o == nullptr || part_ml == nullptr || count == nullptr) return MSGL_ERR_SIZE;
    static MsglOncePerDevice attr_set;
    if (attr_set.due()) {
        if (cudaFuncSetAttribute(attn_decode_runs_kernel<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)run_smem_bytes()) != cudaSuccess ||
            cudaFuncSetAttribute(attn_decode_runs_kernel<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)run_smem_bytes()) != cudaSuccess)
            return msgl_check_launch();
        attr_set.mark();
    }
    RunParams p;
    p.q = (const __nv_bfloat16*)q; p.out = (__nv_bfloat16*)out; p.k_cache = (const __nv_bfloat16*)k_cache; p.v_cache = (const __nv_bfloat16*)v_cache;
    p.kv_len = kv_len; p.block_table = block_table; p.part_o = part_o; p.part_ml = part_ml; p.count = count; p.q_start = q_start; p.wait_last = wait_last;
    p.B = B; p.n_q = n_q; p.n_kv = n_kv; p.page_size = page_size; p.bt_stride = bt_stride; p.scale = scale;
    p.page_shift = -1;
    if ((page_size & (page_size - 1)) == 0) { int sh = 0; while ((1 << sh) < page_size) ++sh; p.page_shift = sh; }
    if (q_start != nullptr) msgl_launch_pdl(attn_decode_runs_kernel<true>, dim3(blocks), dim3(RUN_THREADS), run_smem_bytes(), stream, p);
    else msgl_launch_pdl(attn_decode_runs_kernel<false>, dim3(blocks), dim3(RUN_THREADS), run_smem_bytes(), stream, p);
    return msgl_check_launch();
}
