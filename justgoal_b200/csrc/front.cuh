// Front end for small token counts (T <= FRONT_MAX_T): routing, histogram, scan, stable permutation and the
// expert-sorted activation gather in ONE launch (front_route_kernel; front_small_kernel is the same without the
// routing, for tokens that were routed elsewhere).
//
// With a few dozen tokens separate kernels are pure launch latency.  The tokens are routed one per warp over the CTAs;
// the CTAs meet once (the routing result of every token must be visible); then every CTA redoes the tiny integer
// work - histogram, scan, ranks - for ALL tokens in its own shared memory, so no CTA waits for another again, and
// copies its share of the rows.  One thread owns one (token, expert) pair: its rank inside its expert is its rank
// among the same-expert pairs of its warp (match.any) plus the counts of the warps before it, which keeps the rows of
// an expert in token order.  CTA 0 alone writes the tables that later kernels read (counts, row maps); all CTAs
// derive identical values.  Same results as count_kernel + permute_kernel + gather_kernel (permute.cuh).
// The next kernel (GEMM1) does not wait for this one to finish before it starts to work: it watches the count of the meeting
// (behind front_small_kernel a flag, ST_ROUTED) and FrontParams::copied, see GemmParams::routed.  The reference fuses the same stages for small batches
// (kda05_reproduction_full_shape/fable-5.1/moe_fp8_fwd/<def>/fable51_moe_v94/kernel.cu:724-806) and issues its first
// weight stages during the table build (its MOE_EARLY_W switch, same directory, main.py:50).
#pragma once
#include "permute.cuh"
#include "routing.cuh"

namespace b200moe {

constexpr int FRONT_MAX_T = 128;
constexpr int FRONT_MAX_ROWS = FRONT_MAX_T * 8 + ROW_ALIGN * MAX_LOCAL;   // worst case incl. segment padding
constexpr int FRONT_THREADS = 1024;

struct FrontParams {
    PlanParams plan;              // topk_idx / topk_w in, tables to publish (CTA 0) out
    const uint8_t* hidden;        // [T, H] fp8
    const float* hscale;          // [H/128, T]
    uint8_t* a_perm;              // [rows_cap, H]
    float* a_scale_perm;          // [H/128, rows_cap]
    int H;
    // `sync` (front_route_kernel only) is a word owned by the handle, zero between calls (the last kernel of the forward clears
    // it): CTAs that have arrived at the meeting.  `copied` lies in the workspace, whatever that held before, so that a routed
    // call keeps nothing in the handle: CTAs that have copied their share of the rows.  Behind a meeting it is one count, in the
    // head; without one (front_small_kernel) nobody could tell a CTA that the count is clear, so each has a byte, which it
    // clears itself before the next kernel can look.  Null: the next kernel waits for this one.  `head` is the part of the workspace that must be zero before the GEMMs
    // run (status, split-unit counters), in 16-byte units: CTA 0 clears it, so the forward needs no memset in front of the kernel.
    int* sync;
    int* copied;
    uint4* head;
    int head_vec;
};

struct FrontShared {
    int cnt[MAX_LOCAL];
    uint32_t wcnt_words[FRONT_THREADS / 32][MAX_LOCAL / 4];       // bytes: pairs of expert e among the 32 pairs of warp w
    int row0[MAX_LOCAL + 1], tiles[MAX_LOCAL + 1];
    int row_token[FRONT_MAX_ROWS];
};
__device__ __forceinline__ void front_clear(FrontShared& s) {
    constexpr int WORDS = MAX_LOCAL + FRONT_THREADS / 32 * (MAX_LOCAL / 4);         // cnt and the bytes behind it
    static_assert(offsetof(FrontShared, row0) == WORDS * 4, "cleared in one go");
    for (int i = threadIdx.x; i < WORDS; i += FRONT_THREADS) reinterpret_cast<uint32_t*>(&s)[i] = 0u;
}

// The body shared by the two entry kernels below, behind front_clear and a barrier.  FRESH: the routing result was written
// earlier in this same launch by other CTAs (read it past L1).
template <bool FRESH>
__device__ __forceinline__ void front_body(const FrontParams& fp, FrontShared& s) {
    int* const s_cnt = s.cnt; int* const s_row0 = s.row0; int* const s_tiles = s.tiles; int* const s_row_token = s.row_token;
    auto s_wcnt = reinterpret_cast<uint8_t(*)[MAX_LOCAL]>(s.wcnt_words);
    static_assert(FRONT_THREADS >= FRONT_MAX_T * 8, "one thread per (token, expert) pair");
    const PlanParams& pp = fp.plan;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int T = pp.T, K = pp.top_k, El = pp.num_local;
    const bool publish = blockIdx.x == 0;
    const int n = T * K;

    // ---- this thread's pair (pair i = tid, token-major), the histogram of the local experts, and the pair's rank
    // among the pairs of the same expert inside its warp (stable: pair order)
    const int tok = tid / K;
    const bool valid = tid < n;
    const size_t src = (size_t)tok * pp.pair_stride + (tid - tok * K);
    const int id = valid ? (FRESH ? __ldcg(pp.topk_idx + src) : pp.topk_idx[src]) : -1;
    const float wgt = valid ? (FRESH ? __ldcg(pp.topk_w + src) : pp.topk_w[src]) : 0.f;
    const int le = id - pp.local_offset;
    const bool local = valid && le >= 0 && le < El;
    const unsigned same = __match_any_sync(0xFFFFFFFFu, local ? le : -1 - lane);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (local && rank == 0) {
        s_wcnt[warp][le] = (uint8_t)__popc(same);
        atomicAdd(&s_cnt[le], __popc(same));
    }
    __syncthreads();

    // ---- scan
    if (warp == 0) scan_counts(s_cnt, El, pp.token_tile, pp.rows_cap, s_row0, s_tiles, publish ? pp.status : nullptr, lane);
    // pairs of the same expert in the warps before this one (independent byte loads, no second scan phase)
    int before = 0;
    if (local)
        for (int w2 = 0; w2 < warp; ++w2) before += s_wcnt[w2][le];
    __syncthreads();
    // more rows than the caller's capacity (see scan_counts): refuse, place and copy nothing
    const bool fits = s_row0[El] <= pp.rows_cap;
    const int total_rows = fits ? s_row0[El] : 0;
    if (publish) {
        for (int i = tid; i <= El; i += blockDim.x) {
            pp.expert_row0[i] = s_row0[i];
            pp.tile_prefix[i] = s_tiles[i];
            if (i < El) pp.counts[i] = s_cnt[i];
        }
    }
    for (int r = tid; r < total_rows; r += blockDim.x) s_row_token[r] = -1;
    __syncthreads();

    // ---- stable permutation: an expert's pairs take its rows in pair order
    if (local) {
        const int r = s_row0[le] + before + rank;
        if (fits) {
            s_row_token[r] = tok;
            if (publish) { pp.pair_row[tid] = r; pp.row_w[r] = wgt; }
        } else if (publish) {
            pp.pair_row[tid] = NO_ROW;
        }
    }
    __syncthreads();
    if (publish) {
        for (int r = tid; r < total_rows; r += blockDim.x) {
            const int t = s_row_token[r];
            pp.row_token[r] = t;
            if (t < 0) pp.row_w[r] = 0.f;
        }
    }

    // ---- gather: a row is cut into pieces, one warp per piece, dealt round-robin over all warps of the grid.  The
    // number of pieces grows until every warp has one (a few dozen rows: 16 pieces, one 16-byte load per lane); a
    // warp with more to copy keeps four loads in flight per lane.
    const int H = fp.H, KB = H >> 7, rows_cap = pp.rows_cap;
    const int chunks = H / 16;
    const int n_warps = (int)gridDim.x * (FRONT_THREADS / 32);
    int split = 1;
    while (split < 16 && total_rows * split * 2 <= n_warps) split *= 2;
    const int per_piece = (chunks + split - 1) / split;
    const int n_tasks = total_rows * split;
    for (int task = blockIdx.x * (FRONT_THREADS / 32) + warp; task < n_tasks; task += n_warps) {
        const int r = task / split, piece = task - r * split;
        const int t = s_row_token[r];
        if (t < 0) continue;     // padding rows stay unwritten: their columns are never stored by the GEMMs
        uint4* dst = reinterpret_cast<uint4*>(fp.a_perm + (size_t)r * H);
        const uint4* src = reinterpret_cast<const uint4*>(fp.hidden + (size_t)t * H);
        const int c_end = min(chunks, (piece + 1) * per_piece);
        for (int i = piece * per_piece + lane; i < c_end; i += 128) {
            uint4 v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + 32 * j < c_end) v[j] = __ldg(src + i + 32 * j);
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + 32 * j < c_end) dst[i + 32 * j] = v[j];
        }
        if (piece == split - 1) {
            // the row's block scales (KB <= 64 for every supported hidden size up to 8192: two loads per lane)
            for (int kb = lane; kb < KB; kb += 64) {
                const float s0 = __ldg(fp.hscale + (size_t)kb * T + t);
                const float s1 = kb + 32 < KB ? __ldg(fp.hscale + (size_t)(kb + 32) * T + t) : 0.f;
                fp.a_scale_perm[(size_t)kb * rows_cap + r] = s0;
                if (kb + 32 < KB) fp.a_scale_perm[(size_t)(kb + 32) * rows_cap + r] = s1;
            }
        }
    }
    // this CTA's rows are there for the GEMM that follows (GemmParams::copied)
    if (!fp.copied) return;
    __syncthreads();
    if (tid == 0) {
        if (FRESH) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(fp.copied) : "memory");
        else asm volatile("st.release.gpu.global.u8 [%0], %1;" ::"l"(reinterpret_cast<uint8_t*>(fp.copied) + blockIdx.x), "h"((uint16_t)1) : "memory");
    }
}


// Front end for tokens that were routed elsewhere (the expert-parallel receive side): no meeting, every CTA has the
// routing from the start.  CTA 0 clears the head of the workspace, announces the routing and only then lets GEMM1 start, which
// finds the word set and streams weights while the rows are copied.
// Against count + permute + gather behind a memset: see the rule in b200moe_forward_routed.
__global__ void __launch_bounds__(FRONT_THREADS, 1) front_small_kernel(const FrontParams fp) {
    __shared__ FrontShared s;
    front_clear(s);
    __syncthreads();
    pdl_wait();
    const int clears = FRONT_THREADS - 1;                      // its warp is the least likely to have a pair
    if (fp.copied && threadIdx.x == clears) reinterpret_cast<uint8_t*>(fp.copied)[blockIdx.x] = 0;
    if (blockIdx.x == 0) {
        for (int i = threadIdx.x; i < fp.head_vec; i += FRONT_THREADS) fp.head[i] = make_uint4(0u, 0u, 0u, 0u);
        __threadfence();
        __syncthreads();
        if (threadIdx.x == 0)
            asm volatile("st.release.gpu.global.s32 [%0], %1;" ::"l"(fp.plan.status + ST_ROUTED), "r"(1) : "memory");
        __syncthreads();
        pdl_launch();
    } else if (!fp.copied) {
        pdl_launch();
    } else if (threadIdx.x >= clears - 31) {
        // GEMM1 may start once every CTA has said so, and looks at this byte: one warp says it, behind a fence.  Kept in the
        // handle as a count, for which no CTA had to fence, us: 64 experts of 1024 x 512 64 tokens 38.5 / 39.0, 8 softmax experts of the
        // 4096-wide shape 128: 42.8 / 43.8, 16 of them 10: 39.4 / 40.6, 40: 57.7 / 58.0; 32 of 256 experts 2 tokens 55.5 / 55.7, 64: 134.4 /
        // 135.1 (the whole CTA behind a barrier: 42.1, 45.6, 39.8, 59.4; 55.3, 135.5).
        if (threadIdx.x == clears) asm volatile("fence.acq_rel.gpu;" ::: "memory");
        __syncwarp();
        pdl_launch();
    }
    front_body<false>(fp, s);
}

// Front end INCLUDING the routing (the operator's own forward for T <= FRONT_MAX_T): one launch, and nothing else on the
// stream before it (CTA 0 clears the head of the workspace itself), so the kernel may start while the caller's
// previous kernel still runs.  Before the wait for that kernel the CTAs pull the inputs into L2 (a prefetch returns
// no data, so it is harmless if the previous kernel is still writing them; it hides the first-touch latency of
// every input behind that kernel's tail).
// Phase A: the tokens are dealt over the CTAs (one warp per token) and routed; the CTAs then meet at a counter in
// device memory owned by the handle (all CTAs of this small grid are resident; the wait is bounded like every wait
// of the library); phase B is the common body, every CTA redoing the integer work for all tokens.
template <int VPT, int MODE>
__global__ void __launch_bounds__(FRONT_THREADS, 1) front_route_kernel(const FrontParams fp, const RouteParams rp) {
    __shared__ int s_go;
    __shared__ FrontShared s;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    {
        const size_t gtid = (size_t)blockIdx.x * FRONT_THREADS + threadIdx.x, gth = (size_t)gridDim.x * FRONT_THREADS;
        auto pull = [&](const void* base, size_t bytes) {
            for (size_t off = gtid * 128; off < bytes; off += gth * 128)
                asm volatile("prefetch.global.L2 [%0];" ::"l"(static_cast<const char*>(base) + off));
        };
        pull(rp.logits, (size_t)rp.T * rp.E * 4);
        pull(fp.hidden, (size_t)rp.T * fp.H);
        pull(fp.hscale, (size_t)(fp.H >> 7) * rp.T * 4);
        if (rp.bias) pull(rp.bias, (size_t)rp.E * 2);
    }
    front_clear(s);
    pdl_wait();
    // CTA 0 clears the head of the workspace.  Nothing flags an error in it before the meeting below, and CTA 0
    // arrives there only after its stores (its arrival releases them): whoever has seen all arrivals, the next kernel (GEMM1)
    // included, finds the zeros.
    // Its upper half does that, and alone lets GEMM1 start, while the lower half routes.
    constexpr int HALF = FRONT_THREADS / 2;
    if (blockIdx.x != 0) {
        pdl_launch();
    } else if (threadIdx.x >= HALF) {
        for (int i = threadIdx.x - HALF; i < fp.head_vec; i += HALF) fp.head[i] = make_uint4(0u, 0u, 0u, 0u);
        __threadfence();
        asm volatile("bar.sync 2, %0;" ::"n"(HALF) : "memory");
        pdl_launch();
    }
    for (int t = (int)blockIdx.x + (int)gridDim.x * warp; t < rp.T; t += (int)gridDim.x * (FRONT_THREADS / 32)) {
        int sel_id; float w;
        route_token<VPT, MODE>(rp, t, lane, sel_id, w);
        if (lane < rp.top_k) {
            rp.topk_idx[(size_t)t * rp.top_k + lane] = sel_id;
            rp.topk_w[(size_t)t * rp.top_k + lane] = w;
        }
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        // The meeting: one count, which GEMM1 watches too.  It builds its schedule from the routing and starts to stream weights
        // while this kernel still permutes and gathers.  Nobody clears the count before all that watch it are done: the last
        // kernel of the forward does, also of one that gave up.
        // An earlier form counted those that left as well, so that the last of them could clear both counts, and CTA 0 announced
        // the routing in a word of its own: two more round trips to L2 in front of GEMM1's first load.  With this one, `copied` and
        // eight CTAs up to eight tokens, start / now, us: 512-wide shape 1 token 20.6 / 19.1, 40: 22.4 / 21.6; 64 experts of
        // 1024 x 512 1 token 25.7 / 24.9, 64: 42.8 / 41.5; 32 of 256 experts 1 token 17.1 / 16.5; where the weight stream is long the
        // ring is full in time either way (64 tokens 131.7 / 131.9).
        int* const meet = fp.sync;
        asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(meet) : "memory");
        int go = 1;
        const unsigned long long t0 = globaltimer_ns();
        for (uint32_t it = 1;; ++it) {
            int v;
            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(meet) : "memory");
            if (v >= (int)gridDim.x) break;
            if ((it & 0xFFu) == 0 && globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
                atomicCAS(fp.plan.status + ST_ERR, 0, ERR_WAIT_GROUP); go = 0; break;
            }
        }
        s_go = go;
    }
    __syncthreads();
    if (!s_go) return;
    front_body<true>(fp, s);
}

}  // namespace b200moe

