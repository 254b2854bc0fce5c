// Grouped FP8 block-scale GEMMs on tcgen05 (sm_100a), weights on the M side ("swap-AB").
//
// One UNIT = (local expert, 128 weight rows, one tile of NTOK expert-sorted token rows), full K.
//   GEMM1 (G1): D_up[128, NTOK]   = W13[e, mt*128 .. +128, :]      . A_perm[rows]^T
//               D_gate[128, NTOK] = W13[e, I + mt*128 .. +128, :]  . A_perm[rows]^T
//               epilogue: c = silu(gate) * up, per-(row, 128 columns) amax -> scale = amax/448,
//               stored as TWO e4m3 values hi = rn(c/scale), lo = rn(c/scale - hi) under one scale.
//   GEMM2 (G2): D[128, NTOK] = W2[e, mt*128 .. +128, :] . (act_hi + act_lo)[rows]^T, two MMAs per
//               K step into the same accumulator; epilogue: y[row, h] = D as fp16 (weighted by the combine).
// Block scales change every 128 K, so each 128-K block is accumulated into a fresh TMEM region
// and promoted into fp32 registers: acc += part * (token_scale[kb] * weight_scale[kb]).
// The same arithmetic is stated by the reference's tcgen05 kernels
// (kda05_reproduction_full_shape/fable-5.1/moe_fp8_fwd/<def>/fable51_moe_v94/kernel.cu:3336,3441-3446
//  for the promotion, :3519-3584 for SwiGLU + requantisation,
//  goal_full_shape/fable-5.1/moe_fp8_fwd/<def>/moe_small.cuh:1-16 for the swap-AB orientation);
// unlike them the SwiGLU output keeps a second e4m3 term, because a single e4m3 per element
// does not meet an absolute/relative tolerance of 1e-2 against the unquantised definition.
//
// Schedule (of a kernel that does one GEMM): K is cut into GROUPS of KPB 128-K blocks (one TMEM hand-off per group).  The kernel is
// persistent.  Units are numbered so that the token tiles of one (expert, row tiles) are adjacent.  Every CTA
// first runs floor(U / grid) WHOLE units, round-robin (CTAs that run at the same time work on adjacent units, so
// a weight tile shared by several token tiles comes from HBM once).  The remaining U mod grid units stay
// whole or are cut along K into CHUNKS, whichever is done sooner (size_chunks), and the CTAs CLAIM them one at a time from a counter in
// global memory: SMs do not stream at the same rate under full load, and a CTA that finishes early simply takes more
// chunks (with equal static shares the finish times of the CTAs spread by 7-10 % of the kernel).  Every chunk stores
// its fp32 partial to its own slot and counts itself in; whoever arrives last adds the slots in a fixed order (results
// are bit-identical from run to run) and runs the epilogue, so nobody waits.  GEMM1 with narrow tiles cuts the remaining
// units into equal ranges instead (STATIC_TAIL): the piece that ends a unit waits (bounded) for pieces that their CTAs
// ran before everything else, so no cycle of waiting CTAs can form.
// Inside a CTA the producer claims the work and hands it to the MMA and promotion warps through a small queue
// in shared memory.
//
// Small token counts (GemmParams::routed): GEMM1 follows a front-end kernel that routes, permutes and gathers in one
// launch.  GEMM1's CTAs are resident while it runs; when it announces the routing result they build the expert tables
// themselves and the producer streams the first weight tiles before the front end has completed - only the token
// side of those stages waits for it.  GEMM2 does the same with the tables the front end left (GemmParams::tables_done), as
// soon as its CTA has an SM: the first weights travel under the tail of GEMM1 (T=64: 132 -> 130 us, T=7: 72 -> 70 us).  So does
// GEMM1 behind a separate gather: its tables come from the permutation before that.
// Optionally (FUSE) GEMM2's epilogue also does the combine.
//
// Both GEMMs in one launch (gemm_both_kernel, narrow tiles over weights that L2 cannot hold).  Such a call is two weight streams,
// and between them, with a kernel each, HBM stood idle for 8 to 14 us: the CTAs of GEMM1 end 7 to 15 us apart, a CTA of GEMM2
// takes 5 us from the end of the one before it to its first load, and all of them wait for GEMM1's last epilogue; the stage ring
// covers 4 us of that.  In one launch the producer goes on to GEMM2's weights with the next stage of the ring.  Everything is
// CLAIMED from one counter, in the order GEMM1's whole units, GEMM1's pieces, GEMM2's units and pieces: what a CTA waits for
// (partial sums, the rows of a token tile) has been claimed before its own item by a CTA that runs, so no cycle of waiting CTAs can form and no CTA
// has to be resident, whatever other streams run.  GEMM1's left-over units mostly stay whole, because the CTAs without one take up
// GEMM2's units of the experts that are done.  A token tile's rows are handed over by a counter (tile_done).  us, two launches / one:
// 32 of 256 experts 12 tokens 90 / 82, 64: 132 / 122, 128: 161 / 150, 200: 190 / 182; 128 of 256 experts 4: 136 / 127, 64: 450 / 440; 16
// experts of the 4096-wide shape 16: 62.5 / 54.5, 128: 70.5 / 67.5; 4 of 5120 x 8192 30: 117 / 106.  It is level with more units than a few per
// CTA (128 experts, 200 tokens 609 / 610) and with two to five experts in use (both sides at size_chunks).
//
// Warp roles: warp 0 = TMA producer, warp 1 = MMA issuer + TMEM owner (whole warps, one elected lane issues),
// warps 2-3: scales of 128-token tiles on their way into shared memory, otherwise idle (they complete the first warpgroup so register
// re-allocation is legal; with the fused combine they write the zero rows of tokens that have no pair on this rank),
// warps 4.. = promotion/epilogue (4 or 8 warps; warp % 4 selects the TMEM lane quarter).
// Every wait is bounded (common.cuh); no TMA load uses cluster multicast.
//
// Code size.  A forward runs five or six kernels in turn, and their code together decides whether an SM still holds this
// kernel's when the next forward comes.  With 90 + 63 KB (GEMM1 + GEMM2, 128-token tiles) it did not: the first epilogue of every
// launch, 40 KB of straight code, took 12-14 k cycles instead of 4 k (2048 tokens, 16 experts of the 4096-wide shape: 14.5 k).
// So the roles' loops stay rolled (`unroll 1`: their bodies hold whole waits) and partial sums move four at a time: 80 + 53 KB,
// 7.8 k cycles there; 300 tokens of a 1024-wide shape 60.6 -> 55.6 us, 901 tokens 255.4 -> 250.6 us.
#pragma once
#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include "common.cuh"
#include "permute.cuh"

namespace b200moe {

struct GemmParams {
    int* status;
    const int* counts;
    const int* expert_row0;
    const int* tile_prefix;
    int num_local;
    int KB;               // K blocks of 128
    int n_mtiles;         // 128-row weight tiles per expert that one unit family covers
    int rows_per_expert;  // rows of the weight matrix per expert (2I for GEMM1, H for GEMM2)
    int gate_offset;      // row offset of the unit's second weight tile (GEMM1: I, the gate half; GEMM2: 128)
    int unit_rows;        // weight rows one unit advances by (GEMM1: 128, GEMM2: 256)
    int valid_rows;       // GEMM2: output columns H (the last unit's second tile may lie beyond)
    int scale_rows;       // weight-scale rows per expert (rows_per_expert / 128)
    const float* w_scale; // [E_local, scale_rows, KB]
    const float* b_scale; // [KB, rows_cap] token-side scales
    int rows_cap;
    uint8_t* act_hi; uint8_t* act_lo; float* act_scale; int I;   // GEMM1 outputs
    const float* row_w; __half* y; int H;                         // GEMM2 output: y[row, h] = O[row, h] as fp16 (the routing
                                                                  // weight is applied by the combine, in fp32)
    int evict_first_weights;
    int* sk_count;        // [4 * gridDim.x + 4] zero at launch: [4 * ut ...] arrivals of split unit ut (claimed chunks: one byte
                          // per group of warps that arrives together), [4 * gridDim.x] the chunk claim counter
    float* sk_partial;    // [gridDim.x * chunks per unit] slots of SLOT_FLOATS floats: [NACCUM * NC / 4][NPT][4]
    long long* klog;      // [4][KLOG_N]: CTA 0's clock at its first KLOG_N K blocks: TMA issue, data seen by the
                          // MMA warp, group seen by the promotion warps, group folded (hand-back)
    long long* trace;     // [gridDim.x][TRACE_SLOTS]: slot 0 = %globaltimer at entry, others = SM clocks since entry
    // GEMM1 after a one-launch front end (small token counts), else null: the routing result of all tokens is visible when
    // *routed has reached routed_want (the CTAs that have routed their share, or a flag).  The CTAs then build the expert tables
    // themselves from topk_idx (the same histogram and scan as the front end) and the producer streams the first weight tiles
    // while the front end still permutes and gathers.  The token rows: with narrow tiles they are there when all
    // front_ctas CTAs of the front end have copied their share, by the count at `copied` or, with copied_bytes, a byte each -
    // earlier than the last of them has left and a waiting kernel has learned of it -, otherwise after the wait for the front end.
    const int* routed;
    const int* copied;
    int routed_want, front_ctas;
    bool copied_bytes;
    int* met;             // fused combine: the count of the front end's meeting, which the last kernel of a forward clears, and
                          // behind it, with both GEMMs in one launch, a count of the CTAs that are done
    // Both GEMMs in one launch: counter of every token tile, zero at launch; a warp that has stored its part of a GEMM1 unit's
    // rows counts in, and a unit of GEMM2 may read the tile when tile_want have.
    int* tile_done;
    int tile_want;
    int slots;                    // ... and this GEMM's share of the partial-sum slots, per CTA
    int next_mtiles, next_KB;     // GEMM1: units of GEMM2 per token tile, and their K blocks
    int tables_done;              // the expert tables are complete before this kernel can start (see the kernel's prologue)
    const int32_t* topk_idx;      // [n_pairs] global expert ids (pair_stride == top_k on this path)
    int n_pairs, local_offset;
    // GEMM1 with 128-token tiles reading the token rows straight from the caller's activations (no gather copy), else
    // g4_row_token == null: tm_b0 is then a map over the activations with one-row boxes, a stage's token tile is 32
    // four-row TMA gathers through row_token, and the scale warps copy their tokens' block scales from the
    // caller's scale tensor: scale(token, kb) = g4_scale[token * g4_tok_stride + kb * ts_stride].
    const int32_t* g4_row_token;
    const float* g4_scale;
    int g4_tok_stride;    // in floats
    int g4_T;
    int ts_stride;        // tokens-on-M tiles: floats between a row's token scales of consecutive K blocks (rows_cap for the
                          // gathered copy, the caller's K-block stride when g4_row_token is set); K blocks * ts_stride < 2^31
    // GEMM2 with the combine fused into its epilogue (FUSE: narrow token tiles of the operator's own forward).
    // Byte q of tok_count[t * n_mtiles + mt] (zero at launch) counts the rows of token t whose columns of unit mt that belong
    // to lane quarter q are stored; the warp that brings it to the number of the token's local pairs adds those columns
    // up (permute.cuh, combine_four_tokens) and writes the bf16 output.  Tokens without a local pair get their zero row
    // from the otherwise idle warps 2-3.
    __nv_bfloat16* fuse_out;
    int* tok_count;
    const int32_t* row_token; const int32_t* pair_row; const int32_t* c_topk;
    int c_stride, top_k, T, c_local_offset;
};

// BOTH: the GEMM is one of two in the same launch (gemm_both_kernel); the stages of both then have the same size.
template <int NTOK, bool G1, bool BOTH = false>
struct GemmCfg {
    static constexpr int NA = 2;                          // weight tiles per stage (GEMM1: up + gate rows; GEMM2: two row tiles)
    static constexpr int NB = G1 ? 1 : 2;                 // token tiles per stage
    static constexpr int A_BYTES = 128 * 128;
    static constexpr int B_BYTES = NTOK * 128;
    static constexpr int SC_OFF = NA * A_BYTES + (BOTH ? 2 : NB) * B_BYTES;
    static constexpr int STAGE_BYTES = SC_OFF + 1024;
    // tokens-on-M tiles get their (per-thread scalar) token scales through the scale warps; the others get the tile's
    // NTOK scales copied into the stage
    static constexpr bool SCALES_IN_STAGE = NTOK != 128;
    static constexpr int TX_BYTES = NA * A_BYTES + NB * B_BYTES + (SCALES_IN_STAGE ? NTOK * 4 : 0);
    // 128-token tiles: the rows of a part-full tile travel in boxes of BOX_ROWS, and only the boxes that hold rows of the unit.
    // What the stage held in the others is overwritten with zeros once: zero operands cost the tensor pipe less energy, and
    // the large forwards run into the power limit (8192 tokens, 256 experts: 5.55 -> 5.43 ms at more cycles; 4096 skewed tokens
    // 801 -> 792 us; 4201 routed tokens 743 -> 736 us).
    static constexpr bool BOXED = NTOK == 128;
    static constexpr int BOX_ROWS = BOXED ? 32 : NTOK;
    static constexpr int EMPTY_COUNT = 1 + (SCALES_IN_STAGE ? (NTOK >= 64 ? 8 : 4) : 0);   // MMA commit (+ promotion warps)
    static constexpr int STAGES_RAW = (208 * 1024) / STAGE_BYTES;
    static constexpr int STAGES = STAGES_RAW > 8 ? 8 : STAGES_RAW;
    static constexpr int NACCUM = 2;                      // one accumulator per weight tile
    // Orientation.  Narrow tiles put the weights on the MMA's M side (few tokens = few TMEM columns).
    // A full 128-token tile puts the TOKENS on M (TMEM lanes) and each weight tile's 128 rows on N:
    // a promotion thread then owns one token row, its scale is one scalar per K block (no per-column
    // scale loads or multiplies in the fold) and it stores 64 contiguous output columns as vectors.
    static constexpr bool TOK_ON_M = NTOK == 128;
    // Dependent MMAs into one accumulator serialise on the tensor pipe's latency, which dominates
    // for narrow token tiles; the MMAs of one K block are therefore spread over NSPLIT independent
    // partial accumulators (GEMM1: even/odd K step; GEMM2: hi / lo operand) that the promotion adds.
    static constexpr int NSPLIT = NTOK <= 32 ? 2 : 1;
    static constexpr int CPB = NACCUM * NSPLIT * NTOK;     // TMEM columns per K block
    static constexpr int KPB = (128 / CPB) < 1 ? 1 : (128 / CPB);
    static constexpr int BUFCOLS = KPB * CPB;               // TMEM columns per hand-off buffer
    static constexpr int NACC = (512 / BUFCOLS) > 4 ? 4 : (512 / BUFCOLS);
    static constexpr int TMEM_COLS = NACC * BUFCOLS;
    // Measured and dropped: handing a GEMM1 K block over as two 128-column halves (N = 128 MMAs, four
    // half-buffers in flight) - the N = 128 MMAs compete with the TMA fills for shared-memory bandwidth
    // and a K block took 750 ns instead of 570 ns.
    static constexpr int NTB = NACC;                        // TMEM hand-off barriers per direction
    // promotion warps: 4 (one per TMEM lane quarter) for narrow tiles, 8 (two column groups) from 64 tokens.
    // With tokens on M a thread folds 2 x 64 columns of a block through 64 staging registers; 16 warps of half the columns do not
    // fit the register pool with the same staging and were slower with half of it (700 against 526 cycles per block, no fills).
    static constexpr int NPW = NTOK >= 64 ? 8 : 4;
    static constexpr int NGRP = NPW / 4;                   // column groups (a group = 4 warps = all 128 lanes)
    static constexpr int NPT = 32 * NPW;                   // promotion threads
    static_assert(EMPTY_COUNT == 1 + (SCALES_IN_STAGE ? NPW : 0), "stage release count");
    static constexpr int NC = NTOK / (NPW / 4);            // token columns per promotion thread
    static constexpr int CH = (NACCUM * NC > 64) ? 16 : (NC < 32 ? NC : 32);   // columns per tcgen05.ld
    static constexpr int NTHREADS = 128 + NPT;
    // Register re-allocation (setmaxnreg).  The increase BLOCKS until the CTA's own pool holds enough
    // registers, and that pool is only what the control warps gave back from the allocation the CTA
    // was launched with - so the numbers below must add up exactly (checked here and, against the
    // register count ptxas actually chose, by the host before the first launch).
    static constexpr bool REALLOC_REGS = NPW >= 8;
    static constexpr int LAUNCH_REGS = (65536 / NTHREADS) / 8 * 8;          // what __launch_bounds__(NTHREADS, 1) yields
    static constexpr int CTRL_REGS = 56;      // 40/232 spills in the control warps (8192 tokens, 256 experts: 5.46 against 5.43 ms)
    static constexpr int PROMO_REGS = 224;
    static_assert(!REALLOC_REGS || 128 * CTRL_REGS + NPT * PROMO_REGS <= NTHREADS * LAUNCH_REGS,
                  "setmaxnreg.inc would wait forever: the control warps do not release enough registers");
    static_assert(!REALLOC_REGS || (CTRL_REGS <= LAUNCH_REGS && PROMO_REGS >= LAUNCH_REGS), "setmaxnreg direction");
    // narrow tiles: the promotion warps copy a group's token scales into registers as soon as the
    // stage has landed and release the stage at once, instead of holding it until the group is folded
    static constexpr bool EARLY_SCALES = KPB * NC <= 32 && NPW < 16;
    static constexpr int SLOT_FLOATS = NACCUM * NC * NPT;  // = NACCUM * 128 * NTOK
    // SMALLEST number of K blocks per claimed chunk of a split unit: what the partial-sum area is sized for (the producer decides how
    // many chunks there are).  A chunk streams CHUNK_BLOCKS * 32 KB of weights and leaves 1 KB * NTOK of partial sums.
    static constexpr int CHUNK_BLOCKS = NTOK / 8;
    static constexpr int CHUNK_GROUPS = (CHUNK_BLOCKS / KPB) < 1 ? 1 : (CHUNK_BLOCKS / KPB);
    // GEMM1 with narrow tiles has few, long units (decode: 256 units of 3.7 MB for 148 CTAs): there the units left
    // over after the whole rounds are cut into EQUAL contiguous ranges, one per CTA (or, few units, equal pieces of whole units).  A range touches at most two units, so a
    // CTA stores at most one partial sum, which it makes before anything else; the piece that ends a unit runs after the CTA's
    // whole units and waits for those other pieces (claimed chunks measured 5-15 us slower: every one of them costs a partial sum, late in the kernel).
    // Everywhere else the left-over units are cut into chunks that the CTAs claim as they go.
    static constexpr bool STATIC_TAIL = G1 && NTOK <= 32 && !BOTH;
    static constexpr int WQ = 4, WQ_INTS = 12;             // depth of the in-CTA work queue, words of an entry (WorkItem)
    static constexpr int BAR_BYTES = 320;                  // mbarriers + TMEM address word
    static constexpr int TABLE_INTS = 3 * (MAX_LOCAL + 1);
    static constexpr int RED_BYTES = 2 * (TOK_ON_M ? NGRP * 128 : NPW * NC) * 4;      // maxima, two halves used in turn
    // tokens-on-M: ring of the scales of TSD K blocks, a slot = 128 token scales | 2 weight scales | pad (see the scale warps)
    static constexpr int TSD = 8, TS_SLOT = 132, TS_AHEAD = 4;
    static_assert(TS_AHEAD + NACC <= TSD, "a slot is rewritten only when its block has been folded");
    static constexpr int TS_BYTES = TOK_ON_M ? TSD * TS_SLOT * 4 : 0;
    static constexpr int SMEM_BYTES = 1024 /*align slack*/ + STAGES * STAGE_BYTES + BAR_BYTES + WQ * WQ_INTS * 4 /*work queue*/ +
                                      TABLE_INTS * 4 + RED_BYTES + 80 + 16 + 512 /*token ids of the producer's unit, 16-byte aligned*/ + TS_BYTES;
    static_assert(NTOK % 16 == 0 && NTOK >= 16 && NTOK <= 128, "token tile");
    static_assert(TMEM_COLS >= 32 && TMEM_COLS <= 512 && (TMEM_COLS & (TMEM_COLS - 1)) == 0, "tmem");
    static_assert(STAGES >= KPB + 1, "a group must fit the stage ring with room to prefetch");
    static_assert(NC % CH == 0 && (CH == 8 || CH == 16 || CH == 32), "chunking");
    static_assert(SMEM_BYTES <= 227 * 1024, "shared memory");
};


// Per-CTA time line (SM clock cycles since kernel entry) written by whichever thread reaches the point.
enum : int { TR_ENTRY = 0, TR_PROLOGUE = 1, TR_TMA_FIRST = 2, TR_TMA_LAST = 3, TR_MMA_FIRST = 4, TR_MMA_LAST = 5,
             TR_PROMO_FIRST = 6, TR_PROMO_LAST = 7, TR_PARTIAL = 8, TR_REDUCED = 9, TR_EPILOGUE = 10, TR_EXIT = 11,
             TRACE_SLOTS = 16, KLOG_N = 64 };

struct Unit { int e, mt, row0, nvalid; };

// Unit number -> expert, weight tile, token tile, by a converged warp; the result is the same in all lanes and uniform for
// the compiler (see mbar_wait_warp).  The expert is the last one whose first unit is not beyond u: two rounds of one
// comparison per lane (a binary search was eight dependent shared-memory reads, ~500 cycles of every piece of work).
__device__ __forceinline__ bool decode_unit_warp(int u, int n_mtiles, int num_local, int ntok, const int* s_tiles,
                                                 const int* s_row0, const int* s_cnt, int lane, Unit& o) {
    const unsigned FULL = 0xFFFFFFFFu;
    const int per = (num_local + 31) >> 5;
    const int i1 = lane * per;
    const int base = (__popc(__ballot_sync(FULL, i1 < num_local && s_tiles[i1] * n_mtiles <= u)) - 1) * per;
    const int i2 = base + lane;
    const int e = base + __popc(__ballot_sync(FULL, lane < per && i2 < num_local && s_tiles[i2] * n_mtiles <= u)) - 1;
    if (u < 0 || e < 0) return false;
    const int t0 = s_tiles[e], ntt = s_tiles[e + 1] - t0;
    const int ul = u - t0 * n_mtiles;
    int mt = ul, tt = 0;
    if (ntt > 1) { mt = ul / ntt; tt = ul - mt * ntt; }
    auto uni = [&](int v) { return __shfl_sync(FULL, v, 0); };
    o.e = uni(e); o.mt = uni(mt);
    o.row0 = uni(s_row0[e] + tt * ntok); o.nvalid = uni(min(ntok, s_cnt[e] - tt * ntok));
    return __all_sync(FULL, ntt > 0 && o.mt < n_mtiles && o.nvalid > 0);
}

// One piece of work: unit u, K groups [gb, ge).  pieces == 1: the whole unit; otherwise piece number `piece` of the split
// unit number `ut`, whose partial sums live in the slots from `slot` on.  u < 0 ends the list.
struct WorkItem { int u, gb, ge, ut, piece, pieces, slot; Unit un; int tile; };
constexpr int GAVE_UP = -2;          // u of the item that ends a list because a wait of the producer ran out
constexpr int MAX_PIECES = 128;      // arrivals of a split unit are counted in bytes

// CTA that owns flat index x when `total` indices are cut into `parts` equal contiguous ranges (part c starts at
// c * total / parts)
// (32-bit arithmetic: total < #SMs * K groups, parts <= #SMs, so every product stays far below 2^31)
__device__ __forceinline__ int range_start(int c, int total, int parts) { return (int)((unsigned)c * (unsigned)total / (unsigned)parts); }
__device__ __forceinline__ int range_owner(int x, int total, int parts) {
    int c = (int)((unsigned)x * (unsigned)parts / (unsigned)total);
    while (c + 1 < parts && range_start(c + 1, total, parts) <= x) ++c;
    while (c > 0 && range_start(c, total, parts) > x) --c;
    return c;
}

// Chunks per chunked unit
__host__ __device__ inline int chunks_per_unit(int KB, int kpb, int chunk_groups) {
    const int NG = (KB + kpb - 1) / kpb;
    return (NG + chunk_groups - 1) / chunk_groups;
}

__device__ __forceinline__ float silu_f(float x) { return __fdividef(x, 1.0f + __expf(-x)); }

// N consecutive columns of one expert-output row, rounded to fp16 (the per-pair rows the combine weighs and adds
// up in fp32), as 32-byte stores
template <int N>
__device__ __forceinline__ void store_y_row(__half* dst, const float* acc) {
    static_assert(N % 16 == 0, "16 columns per store");
#pragma unroll
    for (int i = 0; i < N; i += 16) {
        uint32_t pk[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const __half2 h = __floats2half2_rn(acc[i + 2 * j], acc[i + 2 * j + 1]);
            pk[j] = *reinterpret_cast<const uint32_t*>(&h);
        }
        st_global_v8(dst + i, pk[0], pk[1], pk[2], pk[3], pk[4], pk[5], pk[6], pk[7]);
    }
}

template <int N>
__device__ __forceinline__ void tmem_ld_chunk(uint32_t taddr, float* v) {
    uint32_t r[N];
    if constexpr (N == 8) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
            : "r"(taddr) : "memory");
    } else if constexpr (N == 16) {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
            : "r"(taddr) : "memory");
    } else {
        asm volatile(
            "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
            "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"
            "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
            : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
              "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
              "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
              "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
            : "r"(taddr) : "memory");
    }
#pragma unroll
    for (int i = 0; i < N; ++i) v[i] = __uint_as_float(r[i]);
}

// What the roles of a CTA share, and what a warp carries from GEMM1 to GEMM2 where one launch does both.
struct GemmCta {
    uint8_t* smem;
    uint32_t smem_base, tmem_base;
    uint32_t bar_full, bar_empty, bar_tfull, bar_tempty, bar_red, bar_wqfull, bar_wqempty;
    uint32_t* s_tmem;
    int* s_wq; int* s_tiles; int* s_row0; int* s_cnt; uint32_t* s_red; int* s_flag; int* s_g4; float* s_ts;
    int warp, lane;
    long long t_entry;
    int stage; uint32_t phase;         // ring of stages
    int ab; uint32_t aphase;           // ring of accumulators
    uint32_t rphase; int rbuf;         // meetings in the epilogue, half of s_red the next one uses
    int n_item;                        // work queue
    int* claim; int claimed, claim_base;      // one launch for both GEMMs: the counter, lane 0's next claim, claims GEMM1 took
    bool fresh;                        // nothing of this launch has waited for the kernel before it or built the tables yet
    bool ok;
};

// Barriers, tensor memory, the carve-up of shared memory.
template <class C>
__device__ __forceinline__ void gemm_setup(GemmCta& x, uint8_t* smem_raw) {
    x.smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint8_t* tail = x.smem + C::STAGES * C::STAGE_BYTES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(tail);     // full[S], empty[S], tfull[NTB], tempty[NTB], red[4], wq_full[WQ], wq_empty[WQ]
    x.s_tmem = reinterpret_cast<uint32_t*>(tail + C::BAR_BYTES - 8);
    x.s_wq = reinterpret_cast<int*>(tail + C::BAR_BYTES);          // [WQ][WQ_INTS] work items, 16-byte aligned
    x.s_tiles = x.s_wq + C::WQ * C::WQ_INTS;
    x.s_row0 = x.s_tiles + (MAX_LOCAL + 1);
    x.s_cnt = x.s_row0 + (MAX_LOCAL + 1);
    x.s_red = reinterpret_cast<uint32_t*>(x.s_cnt + (MAX_LOCAL + 1));
    x.s_flag = reinterpret_cast<int*>(x.s_red + C::RED_BYTES / 4);   // 20 ints: [0] routing flag seen (early schedule), [4..5] the producer's chunk sizing, [8..11] pieces seen (s_last), [12..] s_filled
    // [128] token of every row of the producer's unit, 16-byte aligned (read and written as int4)
    x.s_g4 = reinterpret_cast<int*>((reinterpret_cast<uintptr_t>(x.s_flag + 20) + 15) & ~uintptr_t(15));
    x.s_ts = reinterpret_cast<float*>(x.s_g4 + 128);            // tokens-on-M: [TSD][TS_SLOT] scales of a K block
    x.warp = __shfl_sync(0xFFFFFFFFu, (int)(threadIdx.x >> 5), 0); x.lane = threadIdx.x & 31;   // uniform for the compiler too
    x.t_entry = clock64();
    x.bar_full = smem_u32(bars);
    x.bar_empty = x.bar_full + 8 * C::STAGES;
    x.bar_tfull = x.bar_empty + 8 * C::STAGES;
    x.bar_tempty = x.bar_tfull + 8 * C::NTB;
    // warps that meet in the epilogue (bounded): the 4 warps of a column group or, tokens on M, those of a lane quarter
    x.bar_red = x.bar_tempty + 8 * C::NTB;
    x.bar_wqfull = x.bar_red + 8 * 4;            // work queue: the producer has published item n
    x.bar_wqempty = x.bar_wqfull + 8 * C::WQ;  // ... and the MMA warp and every promotion warp have read it
    static_assert(8 * (2 * C::STAGES + 2 * C::NTB + 4 + 2 * C::WQ) <= C::BAR_BYTES - 8, "barrier area");
    x.stage = 0; x.phase = 0; x.ab = 0; x.aphase = 0; x.rphase = 0; x.rbuf = 0; x.n_item = 0;
    x.claim = nullptr; x.claimed = 0; x.claim_base = 0; x.fresh = true; x.ok = true;
}
template <class C, int NHELP>
__device__ __forceinline__ void gemm_init(GemmCta& x, const CUtensorMap& m0, const CUtensorMap& m1, const CUtensorMap& m2) {
    if (threadIdx.x == 0) {
        for (int s = 0; s < C::STAGES; ++s) { mbar_init(x.bar_full + 8 * s, 1); mbar_init(x.bar_empty + 8 * s, C::EMPTY_COUNT); }
        for (int b = 0; b < C::NTB; ++b) { mbar_init(x.bar_tfull + 8 * b, 1 + NHELP); mbar_init(x.bar_tempty + 8 * b, C::NPW); }
        for (int g = 0; g < 4; ++g) mbar_init(x.bar_red + 8 * g, C::TOK_ON_M ? C::NGRP : 4);
        for (int w = 0; w < C::WQ; ++w) { mbar_init(x.bar_wqfull + 8 * w, 1); mbar_init(x.bar_wqempty + 8 * w, 1 + NHELP + C::NPW); }
        mbar_fence_init();
        tma_prefetch_desc(&m0); tma_prefetch_desc(&m1); tma_prefetch_desc(&m2);
    }
    if (x.warp == 1) { tmem_alloc(smem_u32(x.s_tmem), C::TMEM_COLS); tmem_relinquish(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    x.tmem_base = *x.s_tmem;
    x.smem_base = smem_u32(x.smem);
}
template <class C>
__device__ __forceinline__ void gemm_teardown(GemmCta& x) {
    tc_fence_before();
    __syncthreads();
    if (x.warp == 1) { tc_fence_after(); tmem_dealloc(*x.s_tmem, C::TMEM_COLS); }
}
template <bool TOK_ON_M, bool G4>
__host__ __device__ constexpr int helper_warps() { return TOK_ON_M ? (G4 ? 2 : 1) : 0; }      // warps (2, 3) that fill the ring of scales

enum : int { SOLE = 0, FIRST = 1, SECOND = 2 };       // a launch's only GEMM; GEMM1, GEMM2 of a launch that does both

// G4 (GEMM1 with 128-token tiles only): the token rows come straight from the caller's activations by four-row TMA
// gathers (GemmParams::g4_row_token); a separate instantiation, so the plain kernel's code is unchanged by it.
// PART (128-token tiles): quarters of a token tile (32 rows, one warp's TMEM lanes) that hold no row of the unit are not
// folded.  With full tiles the extra path costs a few per cent of the promotion loop, so the host picks the instance by the
// expected number of rows per expert (both sides measured at the rule in b200moe.cu).
// FUSE (GEMM2, narrow tiles): with the combine in the epilogue (GemmParams::fuse_out); an instance of its own, so the plain
// kernel stays small.
template <int NTOK, bool G1, bool G4, bool PART, bool FUSE, int WHICH>
__device__ __forceinline__ void gemm_roles(GemmCta& x, const CUtensorMap& tm_w, const CUtensorMap& tm_b0, const CUtensorMap& tm_b1,
                                           const CUtensorMap& tm_s0, const CUtensorMap& tm_s1, const GemmParams& p) {
    constexpr bool BOTH = WHICH != SOLE;
    using C = GemmCfg<NTOK, G1, BOTH>;
    static_assert(!G4 || (C::TOK_ON_M && G1), "TMA-gathered token rows: GEMM1 with 128-token tiles");
    static_assert(!FUSE || (!G1 && !C::TOK_ON_M), "fused combine: GEMM2, narrow tiles");
    static_assert(!PART || (C::TOK_ON_M && !G4), "part-full tiles: tokens on M");
    static_assert(!BOTH || (!C::TOK_ON_M && C::EARLY_SCALES && G1 == (WHICH == FIRST)), "both GEMMs in one launch: narrow tiles");
    uint8_t* const smem = x.smem;
    int* const s_wq = x.s_wq; int* const s_tiles = x.s_tiles; int* const s_row0 = x.s_row0; int* const s_cnt = x.s_cnt;
    uint32_t* const s_red = x.s_red; int* const s_flag = x.s_flag; int* const s_g4 = x.s_g4; float* const s_ts = x.s_ts;
    constexpr int NHELP = helper_warps<C::TOK_ON_M, G4>();
    const int warp = x.warp, lane = x.lane;
    const long long t_entry = x.t_entry;
    long long* const trace = p.trace ? p.trace + (size_t)blockIdx.x * TRACE_SLOTS : nullptr;
    auto stamp = [&](int slot) { if (trace) trace[slot] = clock64() - t_entry; };
#ifdef B200MOE_ENABLE_KLOG
    long long* const klog = (p.klog && blockIdx.x == 0) ? p.klog : nullptr;
    auto klog_put = [&](int row, int n) { if (klog && n < KLOG_N) klog[row * KLOG_N + n] = clock64() - t_entry; };
#else
    auto klog_put = [&](int, int) {};      // the per-K-block log is a build option (-DB200MOE_ENABLE_KLOG)
#endif
    const uint32_t bar_full = x.bar_full, bar_empty = x.bar_empty, bar_tfull = x.bar_tfull, bar_tempty = x.bar_tempty;
    const uint32_t bar_red = x.bar_red, bar_wqfull = x.bar_wqfull, bar_wqempty = x.bar_wqempty;
    const uint32_t tmem_base = x.tmem_base, smem_base = x.smem_base;

    // Schedule (see the head of this file): q whole units per CTA, then chunks of the remaining units claimed
    // from a global counter.
    const int NG = (p.KB + C::KPB - 1) / C::KPB;
    int* const claim = WHICH == SECOND && !x.fresh ? x.claim : p.sk_count + 4 * (int)gridDim.x;

    // Consumer side of the work queue: item n sits in slot n % WQ.  Every lane of the calling warp waits and reads,
    // lane 0 then tells the producer that the warp has its copy.  false = list ended or a wait gave up.
    auto wq_fetch = [&](int n, WorkItem& w, bool& ok) -> bool {
        const int slot = n % C::WQ;
        if (!mbar_wait_warp(bar_wqfull + 8 * slot, (uint32_t)(n / C::WQ) & 1u, p.status, ERR_WAIT_GROUP)) { ok = false; return false; }
        // (the wait above and the arrival below are compiler barriers: plain loads)
        const int4* q = reinterpret_cast<const int4*>(s_wq + slot * C::WQ_INTS);
        const int4 q0 = q[0], q1 = q[1], q2 = q[2];
        auto uni = [](int v) { return __shfl_sync(0xFFFFFFFFu, v, 0); };                  // uniform for the compiler
        w.u = uni(q0.x); w.gb = uni(q0.y); w.ge = uni(q0.z); w.ut = uni(q0.w);
        w.piece = uni(q1.x); w.pieces = uni(q1.y); w.slot = uni(q1.z); w.un.e = uni(q1.w);
        w.un.mt = uni(q2.x); w.un.row0 = uni(q2.y); w.un.nvalid = uni(q2.z);
        if (BOTH && G1) w.tile = uni(q2.w);
        __syncwarp();
        if (lane == 0) mbar_arrive(bar_wqempty + 8 * slot);
        if (BOTH && w.u == GAVE_UP) ok = false;
        return w.u >= 0;
    };

    if (warp < 4) {
    // ================================================================ control warpgroup
    if (C::REALLOC_REGS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(C::CTRL_REGS));
    }
    // Expert tables, by the control warps (the others get decoded work items).  They are written by the kernels before this
    // one; three forms:
    //   GEMM1 after the fused front end (p.routed): built here from the routing result, while the front end still runs;
    //   GEMM2, and GEMM1 behind a gather (p.tables_done): written by a kernel that had completed before any CTA of the kernel
    //     before this one let this kernel start - read past L1, without a wait;
    //   otherwise: read after the wait for the kernel before this one.
    // In the first two forms the producer streams weights before that wait.
    const int ctid = threadIdx.x;
    auto ctrl_sync = []() { asm volatile("bar.sync 1, 128;" ::: "memory"); };
    bool early = false;             // the producer has not waited for the previous kernel yet
    if (WHICH != SECOND || x.fresh) {
    if (G1 && !G4 && p.routed) {
        if (ctid == 0) {
            int seen = 0;
            const unsigned long long t0 = globaltimer_ns();
#pragma unroll 1
            for (uint32_t it = 1;; ++it) {
                asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(seen) : "l"(p.routed) : "memory");
                seen = seen >= p.routed_want;
                if (seen) break;
                if ((it & 0xFFu) == 0 && globaltimer_ns() - t0 > WAIT_LIMIT_NS) break;     // fall back to the tables
            }
            *s_flag = seen;
            if (BOTH && seen) x.claimed = atomicAdd(claim, 1);       // cleared before the announcement; the answer travels under the scan
        }
#pragma unroll 1
        for (int i = ctid; i <= p.num_local; i += 128) s_cnt[i] = 0;
        ctrl_sync();
        early = *s_flag != 0;
    }
    if (early) {
#pragma unroll 1
        for (int i0 = ctid; i0 < p.n_pairs; i0 += 128 * 8) {
            int id[8];
#pragma unroll
            for (int j = 0; j < 8; ++j) id[j] = i0 + 128 * j < p.n_pairs ? __ldcg(p.topk_idx + i0 + 128 * j) - p.local_offset : -1;
#pragma unroll
            for (int j = 0; j < 8; ++j)
                if (id[j] >= 0 && id[j] < p.num_local) atomicAdd(&s_cnt[id[j]], 1);
        }
        ctrl_sync();
        if (warp == 0) scan_counts(s_cnt, p.num_local, NTOK, p.rows_cap, s_row0, s_tiles, nullptr, lane);
    } else {
        early = !G4 && p.tables_done;
        if (!early) pdl_wait();
        if (BOTH && ctid == 0) x.claimed = atomicAdd(claim, 1);
#pragma unroll 1
        for (int i = ctid; i <= p.num_local; i += 128) {
            s_tiles[i] = __ldcg(p.tile_prefix + i);
            s_row0[i] = __ldcg(p.expert_row0 + i);
            s_cnt[i] = i < p.num_local ? __ldcg(p.counts + i) : 0;
        }
    }
    ctrl_sync();
    // The producer (warp 0) waits after its first weight loads.  Nobody lets the next kernel start before having waited
    // for the previous one: the next kernel may rely on everything before this one (tables_done).
    // With `copied` only the idle warps 2-3 wait: all that the roles touch but the copied rows was done when the front end let this kernel start.
    const bool by_count = !C::TOK_ON_M && G1 && early && p.copied;
    if (by_count ? warp >= 2 : warp != 0) {
        if (early) pdl_wait();
        pdl_launch();
    }
    if (threadIdx.x == 0) stamp(TR_PROLOGUE);
    }
    if (warp == 0) {
        // ------------------------------------------------------------ TMA producer: the whole warp runs the loop, one
        // elected lane issues (see elect_one)
        {
            const uint64_t pol = policy_evict_first();
            const int total_units = s_tiles[p.num_local] * p.n_mtiles;
            const int sched_q = total_units / (int)gridDim.x;              // whole units per CTA
            const int sched_U0 = sched_q * (int)gridDim.x;                 // first chunked unit
            int stage = x.stage; uint32_t phase = x.phase;
            bool ok = true, issued = false;
            bool waited = !early || WHICH == SECOND;      // early schedule: has this thread waited for the previous kernel yet (GEMM2's
                                                          // rows behind GEMM1 in the same launch come with a counter)
            int nk = 0;
            // the producer decides what this CTA does next and publishes it to the other roles
            int n_item = x.n_item, n_whole = 0;
            constexpr bool BOXED = C::BOXED && !G4;
            volatile int* const s_filled = s_flag + 12;  // 128-token tiles: boxes of each stage whose rows are not zero
            if (BOXED && lane < C::STAGES) s_filled[lane] = 128 / C::BOX_ROWS;
            __syncwarp();
            auto publish = [&](const WorkItem& w) -> bool {
                const int slot = n_item % C::WQ;
                if (!mbar_wait_warp(bar_wqempty + 8 * slot, ((uint32_t)(n_item / C::WQ) & 1u) ^ 1u, p.status, ERR_WAIT_GROUP)) return false;
                if (lane == 0) {
                    int4* q = reinterpret_cast<int4*>(s_wq + slot * C::WQ_INTS);
                    q[0] = make_int4(w.u, w.gb, w.ge, w.ut);
                    q[1] = make_int4(w.piece, w.pieces, w.slot, w.un.e);
                    q[2] = make_int4(w.un.mt, w.un.row0, w.un.nvalid, w.tile);
                    mbar_arrive(bar_wqfull + 8 * slot);      // release: the item is visible to whoever sees the phase flip
                }
                __syncwarp();
                ++n_item;
                return true;
            };
            // Left-over units: `pieces` chunks of chunk_groups groups each, claimed one at a time (1: the units stay whole).  Of up to
            // MOST pieces the number for which the CTA that claims most is done first, by the length of its chunks and by what a
            // piece costs beside it, in K blocks: storing its partial sums, the meetings, the restart of the pipeline - 14-17 k
            // cycles measured for a full 128-token tile, hence 12 blocks there, 6 where most of the tile's rows are empty, 8 for narrow
            // tiles - and one more for every slot that the last piece adds up.  (6 or 12 goes by the instance, not by the tile: a full
            // tile of a call whose tiles are mostly part full is charged half of what it costs.)  The rule before this one, about two chunks per CTA
            // whatever a piece costs, made the tail longer than the whole units it cut up.  us, before / now: 32 of 256 experts 4
            // tokens 59.7 / 53.1, 16: 94.6 / 89.3, 128: 161.9 / 154.5, 257: 197.7 / 191, 901: 278 / 264; 16 experts of the 4096-wide
            // shape 16: 57.1 / 50.5, 128: 82.7 / 73.3, 2048: 129 / 112; K of 64 blocks in GEMM2 (4 experts, 5120 x 8192) 16: 57.2 / 49,
            // 400: 150 / 125.  The line is not sharp: 6 / 12 / 18 blocks with 128-token tiles 320 tokens 221 / 227 / 231, 600: 238 / 247 /
            // 248, 2048: 343 / 338 / 338; 4 / 8 / 12 / 20 blocks with narrow tiles differ by less than 1 us but for the shape of 64 blocks
            // (64 tokens 89.0 / 87.9 / 88.0 / 88.3) and 4 tokens of a 4096 x 4096 shape (40.0 / 40.0 / 40.0 / 44.4).
            // With both GEMMs in one launch: GEMM1's left-over units stay whole while the CTA that runs one more unit than the others,
            // and then one of GEMM2's, is done before all work is (F, in K blocks per CTA); else they are cut by the same cost at 4 blocks per
            // piece (the piece that ends a unit stores nothing, and the stream goes on meanwhile), not counting the CTAs that start late
            // because the front end runs on their SMs.  Pieces 1 / 2 / 3 / 4, us: 32 of 256 experts 2 tokens (32 units) 47 / 40 / 39 / 39, 4
            // (96) 65 / 68 / 63 / 68, 16 (160, of which 12 are left over; 8 pieces 83) 95 / 89 / 87 / 87, 128 (320) 152 / 153 / 153 / 157, 257 (400) 195 / 201 / 208 / 210;
            // 16 of the 4096-wide shape 1 (24) 33.9 / 30.3 / 29.6 / 28.7, 4 (72) 37.0 / 38.0 / 44.9 / 43.4.  GEMM2's are cut into pieces of 16 blocks
            // at most (K of 32, 8 of a 4096 x 4096 shape, 64 tokens, whole / cut 79.4 / 78.2; K of 64, 4 of 5120 x 8192, 30 tokens, two launches /
            // four pieces 117 / 106), and by the cost into smaller ones: 8 blocks a piece, but 5 where the whole launch has less than one of
            // its units per CTA and the CTAs without one would idle (1 expert of the DeepSeek-V3 shape, 28 units of 16 blocks, whole /
            // four pieces 32.4 / 30.3; 2 experts, 56 units, whole, which is what 7 blocks would do, / two pieces 35.9 / 34.5).
            // (Kept in shared memory between the rare claims rather than in registers for the whole loop.)
            volatile int* const s_sched = s_flag + 4;                      // [0] chunk_groups, or the number of ranges, [1] pieces, or 0
            bool sized = false;
            auto size_chunks = [&]() {
                constexpr int MOST = 8;
                const int PIECE_COST = C::TOK_ON_M ? (PART ? 6 : 12) : WHICH == FIRST ? 4 : WHICH == SECOND && sched_q == 0 ? 5 : 8;
                static_assert(MOST <= MAX_PIECES, "arrivals of a split unit");
                const int tail_units = total_units - sched_U0;
                const int slots = (int)gridDim.x * (BOTH ? p.slots : (NG + C::CHUNK_GROUPS - 1) / C::CHUNK_GROUPS);           // what sk_partial holds
                const int late = WHICH == FIRST && sched_q == 0 && p.routed ? p.front_ctas : 0;
                int best = NG * C::KPB, chunk_groups = NG;
                if (WHICH == FIRST && sched_q > 0 &&
                           (sched_q + 1) * p.KB + p.next_KB <= (total_units * p.KB + s_tiles[p.num_local] * p.next_mtiles * p.next_KB) / (int)gridDim.x) {
                    best = 0;
                }
#pragma unroll 1
                for (int n = 2; n <= MOST && tail_units * n <= slots; ++n) {
                    const int len = (NG + n - 1) / n;
                    const int cost = (tail_units * n + late + (int)gridDim.x - 1) / (int)gridDim.x * (len * C::KPB + PIECE_COST + n);
                    if (cost < best) { best = cost; chunk_groups = len; }
                }
                if (WHICH == SECOND) {
                    int n = min(max((p.KB + 8) / 16, 1), MOST);
                    while (n > 1 && tail_units * n > slots) --n;
                    chunk_groups = min(chunk_groups, (NG + n - 1) / n);
                }
                // Units between a third of the CTAs that can start at once and 5/8 of all are dealt out as one range per claim, which
                // may end one unit and start the next: equal pieces come out as half a unit each, or whole units, and leave a third of
                // the CTAs without loads.  Two launches / one with equal pieces or whole units / one with ranges, median us: DeepSeek-V3
                // shape, routed, 3 experts (48 units, 140 CTAs start at once) 38.0 / 39.6 / 38.8, 4 (64 units, 116 CTAs) 44.7 / 48.9 / 44.3,
                // 5 (80 units) 49.9 / 57.7 / 49.2; forward, 3 experts 43.1 / 42.4 / 41.0; 4 experts of the 4096-wide shape (48 units) routed
                // 30.8 / 32.3 / 31.8, forward 32.3 / 33.1 / 32.0.  Above the line 6 (96 units) 58.9 / 60.1 / 63.9, 7 (112) 64.1 / 63.8 / 68.7: GEMM2's loads
                // fill what whole units leave.  Below it 1 (16 units) 29.4 / 27.5 with pieces, 2 (32 units) 32.7 / 33.5 / 33.4: what is left
                // there is the claim that the start waits for.
                int pieces = (NG + chunk_groups - 1) / chunk_groups;
                const int ranges = (int)gridDim.x - late;
                if (WHICH == FIRST && sched_q == 0 && 3 * tail_units > ranges && 8 * tail_units <= 5 * (int)gridDim.x && tail_units <= ranges) {
                    chunk_groups = ranges; pieces = 0;
                }
                if (lane == 0) { s_sched[0] = chunk_groups; s_sched[1] = pieces; }       // no pieces: s_sched[0] ranges
                __syncwarp();
                sized = true;
            };
            // A claim is an atomic round trip (~1 us under load): it is sent while the piece before it is still being loaded.
            // Without whole units the first chunk is the CTA's own number, so that the start does not wait for one.
            // With both GEMMs in one launch everything is claimed, in the order GEMM1's whole units, its pieces, GEMM2's: a unit of
            // GEMM2 then waits only for work that CTAs that run have taken up, whatever other streams keep from running.
            int ahead = BOTH ? x.claimed : (int)blockIdx.x;                // lane 0's is the one that counts
            bool have_ahead = BOTH || sched_q == 0;
            const int claim0 = BOTH ? -x.claim_base : sched_q == 0 ? (int)gridDim.x : 0;
            auto claim_ahead = [&]() {
                if (!have_ahead && lane == 0) ahead = claim0 + atomicAdd(claim, 1);
                have_ahead = true;
            };
            // A range [t_lo, t_hi) of the flat (left-over unit, K group) space, number t_part of `ranges` equal ones: the end of one unit
            // and perhaps the start of the next.  What others wait for comes first, then the piece that ends a unit and waits itself.
            // A static tail has one range per CTA, numbered like the CTAs, and its whole units between the two (T=257: 214 ->
            // 209 us against running the waiting piece before the whole units); with both GEMMs in one launch a range is a claim of
            // GEMM1's, and what it waits for are claims before it.
            int t_lo = 0, t_hi = 0, t_unit = 0, t_part = (int)blockIdx.x;
            const int flat = (total_units - sched_U0) * NG;
            // Up to half as many units as CTAs are cut into the same number of pieces each, more into one range per CTA.  (A range
            // that crosses a unit's end leaves its CTA two pieces.  One range per CTA / equal pieces / equal pieces or whole units
            // whatever their number, us: 2 tokens 39.8 / 38.9 / 38.9, 16: 89.8 / 88.0 / 88.0, 24: 100.4 / 99.3 / 99.8, 128: 161.4 / 160.4 /
            // 160.0, 200: 185.1 / 186.1 / 182.2; 16 experts of the 4096-wide shape 64: 66.2 / 63.6 / 63.6; 8 of a 4096 x 4096 shape 128:
            // 83.5 / 83.7 / 85.7.)
            const int static_ranges = 2 * (total_units - sched_U0) > (int)gridDim.x || flat == 0
                                          ? min(flat, (int)gridDim.x)
                                          : (total_units - sched_U0) * min(NG, (int)gridDim.x / (total_units - sched_U0));
            auto take_range = [&](int part, int ranges) {
                t_part = part; t_lo = range_start(part, flat, ranges); t_hi = range_start(part + 1, flat, ranges);
                t_unit = t_lo / NG;
            };
            if (C::STATIC_TAIL && (int)blockIdx.x < static_ranges) take_range((int)blockIdx.x, static_ranges);
#pragma unroll 1
            while (ok) {
                WorkItem wi;
                wi.ut = wi.piece = wi.slot = 0; wi.pieces = 1; wi.un = Unit{0, 0, 0, 0}; wi.tile = 0;
                const int u_end = (t_unit + 1) * NG;
                const bool ends_unit = t_lo > t_unit * NG && t_hi == u_end;         // the rest of the range is such a piece
                if ((C::STATIC_TAIL || WHICH == FIRST) && t_lo < t_hi && !(C::STATIC_TAIL && ends_unit && n_whole < sched_q)) {
                    const int ranges = C::STATIC_TAIL ? static_ranges : s_sched[0];
                    if (t_hi > u_end) {                       // the start of the next unit
                        wi.ut = t_unit + 1; wi.gb = 0; wi.ge = t_hi - u_end;
                        t_hi = u_end;
                    } else {
                        wi.ut = t_unit; wi.gb = t_lo - t_unit * NG; wi.ge = t_hi - t_unit * NG;
                        t_lo = t_hi;
                    }
                    wi.u = sched_U0 + wi.ut;
                    if (wi.ge < NG) {                         // does not end its unit: leaves its partial sum in the range's slot
                        wi.slot = t_part; wi.pieces = 2;
                    } else if (wi.gb > 0) {
                        wi.slot = range_owner(wi.ut * NG, flat, ranges);       // range of the unit's first piece
                        wi.piece = t_part - wi.slot; wi.pieces = wi.piece + 1;
                    }
                } else if (BOTH) {
                    claim_ahead();
                    int c = __shfl_sync(0xFFFFFFFFu, ahead, 0);
                    if (c < sched_U0) {
                        wi.u = c; wi.gb = 0; wi.ge = NG;
                    } else {
                        if (!sized) size_chunks();
                        const int chunk_groups = s_sched[0], pieces = s_sched[1];
                        const int items = sched_U0 + (WHICH == FIRST && pieces == 0 ? chunk_groups : (total_units - sched_U0) * pieces);
                        if (c >= items) {                     // the claim carries over into GEMM2's list
                            x.claimed = ahead - items; x.claim_base += items; x.claim = claim;
                            wi.u = -1; wi.gb = wi.ge = 0; publish(wi); break;
                        }
                        c -= sched_U0;
                        if (WHICH == FIRST && pieces == 0) {
                            take_range(c, chunk_groups);
                            have_ahead = false;
                            continue;
                        }
                        wi.ut = c / pieces; wi.piece = c - wi.ut * pieces; wi.pieces = pieces;
                        wi.slot = wi.ut * pieces;
                        wi.u = sched_U0 + wi.ut;
                        wi.gb = wi.piece * chunk_groups; wi.ge = min(NG, wi.gb + chunk_groups);
                    }
                    have_ahead = false;
                } else if (n_whole < sched_q) {
                    wi.u = n_whole * (int)gridDim.x + (int)blockIdx.x; wi.gb = 0; wi.ge = NG;
                    ++n_whole;
                } else {
                    if (C::STATIC_TAIL || total_units == sched_U0) { wi.u = -1; wi.gb = wi.ge = 0; publish(wi); break; }
                    claim_ahead();
                    if (!sized) size_chunks();
                    const int chunk_groups = s_sched[0], pieces = s_sched[1];
                    const int c = __shfl_sync(0xFFFFFFFFu, ahead, 0);
                    have_ahead = false;
                    if (c >= (total_units - sched_U0) * pieces) { wi.u = -1; wi.gb = wi.ge = 0; publish(wi); break; }
                    wi.ut = c / pieces; wi.piece = c - wi.ut * pieces; wi.pieces = pieces;
                    wi.slot = wi.ut * pieces;
                    wi.u = sched_U0 + wi.ut;
                    wi.gb = wi.piece * chunk_groups; wi.ge = min(NG, wi.gb + chunk_groups);
                }
                if (!decode_unit_warp(wi.u, p.n_mtiles, p.num_local, NTOK, s_tiles, s_row0, s_cnt, lane, wi.un)) {
                    if (lane == 0) atomicCAS(p.status, 0, ERR_BAD_SCHEDULE);
                    ok = false; break;
                }
                if (BOTH) wi.tile = s_tiles[wi.un.e] + (wi.un.row0 - s_row0[wi.un.e]) / NTOK;
                // Are GEMM1's rows of the token tile there?
                const int* const done = WHICH == SECOND ? p.tile_done + wi.tile : nullptr;
                auto rows_done = [&]() -> bool {
                    int n = 0;
                    if (lane == 0) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(n) : "l"(done) : "memory");
                    n = __shfl_sync(0xFFFFFFFFu, n, 0);
                    __syncwarp();        // lane 0's acquire orders the loads of whichever lane issues them
                    return merged(n >= p.tile_want);
                };
                bool there = WHICH == SECOND && rows_done();
                if (!publish(wi)) { ok = false; break; }
                const int gb = wi.gb, ge = wi.ge;
                const Unit un = wi.un;
                const int wrow = un.e * p.rows_per_expert + un.mt * p.unit_rows;
                const int kb_end = min(p.KB, ge * C::KPB);
                const int boxes = BOXED ? (un.nvalid + C::BOX_ROWS - 1) / C::BOX_ROWS : 1;
                const uint32_t tx = BOXED ? (uint32_t)(C::NA * C::A_BYTES + C::NB * boxes * C::BOX_ROWS * 128) : (uint32_t)C::TX_BYTES;
                // zeros into the boxes of stage s_ that this unit leaves out and an earlier one filled; the stage is empty
                auto clear_dead_rows = [&](int s_) {
                    const int was = s_filled[s_];
                    if (was > boxes) {
                        uint8_t* st = smem + s_ * C::STAGE_BYTES + C::NA * C::A_BYTES;
#pragma unroll 1
                        for (int o = boxes * C::BOX_ROWS * 128 + lane * 16; o < was * C::BOX_ROWS * 128; o += 512) {
                            *reinterpret_cast<uint4*>(st + o) = make_uint4(0u, 0u, 0u, 0u);
                            if (!G1) *reinterpret_cast<uint4*>(st + C::B_BYTES + o) = make_uint4(0u, 0u, 0u, 0u);
                        }
                        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");      // the MMAs read through the async proxy
                    }
                    __syncwarp();
                    if (lane == 0) s_filled[s_] = boxes;
                };
                auto load_weights = [&](int s_, int kb) {
                    const uint32_t st = smem_base + s_ * C::STAGE_BYTES;
                    const uint32_t full = bar_full + 8 * s_;
                    mbar_arrive_expect_tx(full, tx);
                    if (p.evict_first_weights) {
                        tma_load_2d_hint(st, &tm_w, kb * 128, wrow, full, pol);
                        tma_load_2d_hint(st + C::A_BYTES, &tm_w, kb * 128, wrow + p.gate_offset, full, pol);
                    } else {
                        tma_load_2d(st, &tm_w, kb * 128, wrow, full);
                        tma_load_2d(st + C::A_BYTES, &tm_w, kb * 128, wrow + p.gate_offset, full);
                    }
                };
                constexpr bool g4 = G4;
                if (g4) {
                    // tokens of the unit's 128 rows (segments start at multiples of 16 rows: 16-byte loads; rows past
                    // the expert's own hold other tokens, -1 or stale values - their results are never stored, and a
                    // row index outside the tensor reads zeros)
                    const int4* src = reinterpret_cast<const int4*>(p.g4_row_token + un.row0);
#pragma unroll 1
                    for (int i = lane; i < 32; i += 32) reinterpret_cast<int4*>(s_g4)[i] = __ldg(src + i);
                    __syncwarp();
                }
                auto load_tokens = [&](int s_, int kb) {
                    const uint32_t st = smem_base + s_ * C::STAGE_BYTES;
                    const uint32_t full = bar_full + 8 * s_;
                    if (g4) {
#pragma unroll 1
                        for (int g = 0; g < 32; ++g) {
                            const int4 t = reinterpret_cast<const int4*>(s_g4)[g];
                            tma_gather4_2d(st + C::NA * C::A_BYTES + g * 512, &tm_b0, kb * 128, t.x, t.y, t.z, t.w, full);
                        }
                        return;
                    }
                    const uint32_t dst = st + C::NA * C::A_BYTES;
                    if (!BOXED || boxes == 128 / C::BOX_ROWS) {
                        tma_load_2d(dst, &tm_b0, kb * 128, un.row0, full);
                        if (!G1) tma_load_2d(dst + C::B_BYTES, &tm_b1, kb * 128, un.row0, full);
                    } else if constexpr (BOXED) {
#pragma unroll 1
                        for (int b = 0; b < boxes; ++b) {
                            tma_load_2d(dst + b * C::BOX_ROWS * 128, &tm_s0, kb * 128, un.row0 + b * C::BOX_ROWS, full);
                            if (!G1) tma_load_2d(dst + C::B_BYTES + b * C::BOX_ROWS * 128, &tm_s1, kb * 128, un.row0 + b * C::BOX_ROWS, full);
                        }
                    }
                    if (C::SCALES_IN_STAGE)
                        bulk_load(st + C::SC_OFF, p.b_scale + (size_t)kb * p.rows_cap + un.row0, NTOK * 4, full);
                };
                int kb_first = gb * C::KPB;
                // The clearing: in the first turn of the stage ring.  Not for a piece of a few K blocks, which is over before it pays: it
                // stands in front of the first loads.  (With 4, 5 and 8 K blocks it cost 1-2 us of a 34-55 us forward; pieces of 16
                // and 56 gain, see BOXED.)
                const bool clears = BOXED && kb_end - kb_first >= 3 * C::STAGES;
                const int kb_clear = clears ? kb_first + C::STAGES : kb_first;
                if (BOXED && !clears && lane < C::STAGES) s_filled[lane] = 128 / C::BOX_ROWS;
                __syncwarp();
                if constexpr (WHICH == SECOND) {
                    // where they are not, the stages take the weights first
                    if (!there) {
                        const int npre = min(C::STAGES, kb_end - kb_first);
                        int st_ = stage; uint32_t ph_ = phase;
#pragma unroll 1
                        for (int i = 0; i < npre; ++i) {
                            if (!mbar_wait_warp(bar_empty + 8 * st_, ph_ ^ 1, p.status, ERR_WAIT_SMEM_EMPTY)) { ok = false; break; }
                            if (elect_one()) load_weights(st_, kb_first + i);
                            __syncwarp();
                            if (++st_ == C::STAGES) { st_ = 0; ph_ ^= 1; }
                        }
                        if (!issued) { if (lane == 0) stamp(TR_TMA_FIRST); issued = true; }
                        const unsigned long long t0 = globaltimer_ns();
#pragma unroll 1
                        for (uint32_t it = 1; ok && !there; ++it) {
                            there = rows_done();
                            if (!there && (it & 0xFFu) == 0 && __any_sync(0xFFFFFFFFu, globaltimer_ns() - t0 > WAIT_LIMIT_NS)) {
                                if (lane == 0) atomicCAS(p.status, 0, ERR_WAIT_CHUNKS);
                                ok = false;
                            }
                        }
                        if (!ok) break;
                        asm volatile("fence.proxy.async.global;" ::: "memory");       // the rows were stored through the generic proxy
#pragma unroll 1
                        for (int i = 0; i < npre; ++i) {
                            if (elect_one()) load_tokens(stage, kb_first + i);
                            __syncwarp();
                            if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                        }
                        kb_first += npre;
                    } else {
                        asm volatile("fence.proxy.async.global;" ::: "memory");
                    }
                }
                if (!waited) {
                    // early schedule, first item: the (empty) stage ring takes weight tiles while the kernel before this one
                    // still runs, then the wait for it, then the token side of the same stages
                    const int npre = min(C::STAGES, kb_end - kb_first);
#pragma unroll 1
                    for (int i = 0; i < npre; ++i) {
                        if (clears) clear_dead_rows(i);
                        if (elect_one()) load_weights(i, kb_first + i);
                        __syncwarp();
                    }
                    if (lane == 0) stamp(TR_TMA_FIRST);
                    issued = true;
                    if (!C::TOK_ON_M && G1 && p.copied) {
                        const unsigned long long t0 = globaltimer_ns();
#pragma unroll 1
                        for (uint32_t it = 1;; ++it) {
                            // (as few requests as possible: every CTA polls the same few bytes)
                            bool mine = true;
                            if (!p.copied_bytes) {
                                int n = p.front_ctas;
                                if (lane == 0) asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(n) : "l"(p.copied) : "memory");
                                mine = n >= p.front_ctas;
                            } else if (16 * lane < p.front_ctas) {
                                uint32_t v[4];
                                asm volatile("ld.acquire.gpu.global.v4.u32 {%0,%1,%2,%3}, [%4];"
                                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]) : "l"(p.copied + 4 * lane) : "memory");
#pragma unroll
                                for (int j = 0; j < 4; ++j) {
                                    const int left = p.front_ctas - 16 * lane - 4 * j;           // bytes of this word that count
                                    const uint32_t set = left >= 4 ? 0x01010101u : left > 0 ? 0x01010101u >> (8 * (4 - left)) : 0u;
                                    mine = mine && (v[j] & (set * 255u)) == set;
                                }
                            }
                            mine = __all_sync(0xFFFFFFFFu, mine);
                            __syncwarp();        // the lanes' acquires order the loads of whichever lane issues them
                            if (merged(mine)) break;
                            if ((it & 0xFFu) == 0 && __any_sync(0xFFFFFFFFu, globaltimer_ns() - t0 > WAIT_LIMIT_NS)) { ok = false; break; }
                        }
                        if (!ok && lane == 0) atomicCAS(p.status, 0, ERR_WAIT_GROUP);
                        asm volatile("fence.proxy.async.global;" ::: "memory");
                    } else {
                        pdl_wait();
                    }
                    waited = true;
#pragma unroll 1
                    for (int i = 0; i < npre; ++i) {
                        if (elect_one()) load_tokens(i, kb_first + i);
                        __syncwarp();
                        if (lane == 0) klog_put(0, nk);
                        ++nk;
                    }
                    kb_first += npre;
                    stage = npre;
                    if (stage == C::STAGES) { stage = 0; phase ^= 1; }
                }
#pragma unroll 1
                for (int kb = kb_first; kb < kb_end; ++kb) {
                    if (!mbar_wait_warp(bar_empty + 8 * stage, phase ^ 1, p.status, ERR_WAIT_SMEM_EMPTY)) { ok = false; break; }
                    if (BOXED && kb < kb_clear) clear_dead_rows(stage);
                    if (elect_one()) { load_weights(stage, kb); load_tokens(stage, kb); }
                    __syncwarp();
                    if (!issued) { if (lane == 0) stamp(TR_TMA_FIRST); issued = true; }
                    if (lane == 0) klog_put(0, nk);
                    ++nk;
                    if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                    if (BOTH ? kb + 3 == kb_end : !C::STATIC_TAIL && kb + 3 == kb_end && n_whole == sched_q && total_units > sched_U0) claim_ahead();
                }
            }
            if (lane == 0) stamp(TR_TMA_LAST);
            x.stage = stage; x.phase = phase; x.n_item = n_item; x.ok = ok;
            if (!ok) {
                // gave up: end the list for the other roles (if the queue still moves), then give copies that are
                // still in flight time to land before the CTA's shared memory goes away
                WorkItem end_; end_.u = BOTH ? GAVE_UP : -1; end_.gb = end_.ge = end_.ut = end_.piece = end_.slot = 0; end_.pieces = 1; end_.un = Unit{0, 0, 0, 0}; end_.tile = 0;
                publish(end_);
                for (int i = 0; i < 64; ++i) __nanosleep(10000);
            }
        }
        __syncwarp();
    } else if (warp == 1) {
        // ------------------------------------------------------------ MMA issuer (whole warp, one elected lane issues)
        {
            constexpr uint32_t idesc = make_idesc_f8(128, NTOK);
            int stage = x.stage; uint32_t phase = x.phase;
            int ab = x.ab; uint32_t aphase = x.aphase;
            bool ok = true, seen = false;
            int nk = 0;
            int n_item = x.n_item;
            WorkItem wi;
#pragma unroll 1
            while (ok && wq_fetch(n_item++, wi, ok)) {
                const int gb = wi.gb, ge = wi.ge;
#pragma unroll 1
                for (int grp = gb; grp < ge; ++grp) {
                    const int nj = min(C::KPB, p.KB - grp * C::KPB);
#pragma unroll 1
                    for (int j = 0; j < nj; ++j) {
                        if (lane == 0) klog_put(6, nk);
                        // the group's accumulator buffer (first K block) and the stage, tried together: the tensor pipe's
                        // queue is only two or three MMAs deep, two waits in a row leave it idle
                        if (!(j == 0 ? mbar_wait_both(bar_tempty + 8 * ab, aphase ^ 1, ERR_WAIT_TMEM_EMPTY,
                                                      bar_full + 8 * stage, phase, ERR_WAIT_SMEM_FULL, p.status)
                                     : mbar_wait_warp(bar_full + 8 * stage, phase, p.status, ERR_WAIT_SMEM_FULL))) { ok = false; break; }
                        if (!seen) { if (lane == 0) stamp(TR_MMA_FIRST); seen = true; }
                        if (lane == 0) klog_put(1, nk);
                        ++nk;
                        tc_fence_after();
                        const uint32_t st = smem_base + stage * C::STAGE_BYTES;
                        const uint32_t d = tmem_base + ab * C::BUFCOLS + j * C::CPB;
                        // mm(D, weight tile, token tile): operand order follows the orientation
                        auto mm = [&](uint32_t dd, uint64_t wdesc, uint64_t tdesc, uint32_t accum) {
                            if (C::TOK_ON_M) umma_f8(dd, tdesc, wdesc, idesc, accum);
                            else umma_f8(dd, wdesc, tdesc, idesc, accum);
                        };
                        if (elect_one()) {
                        if (C::TOK_ON_M) {
                            // The two weight tiles of a stage are adjacent in shared memory (256 rows of 128 B)
                            // and so are their accumulators in TMEM: ONE N = 256 MMA per 32-byte K step covers
                            // both.  (An N = 128 MMA reads 8 KB of operands per 64 tensor-pipe cycles, all the
                            // shared-memory bandwidth of the SM: measured 75 cycles alone, slower beside TMA fills.)
                            constexpr uint32_t idesc2 = make_idesc_f8(128, 256);
                            const uint64_t w = make_smem_desc(st);
                            const uint64_t th = make_smem_desc(st + 2 * C::A_BYTES);
#pragma unroll
                            for (int k = 0; k < 4; ++k) umma_f8(d, th + 2 * k, w + 2 * k, idesc2, k > 0);
                            if (!G1) {      // GEMM2: the low-order term of the activation accumulates on top
                                const uint64_t tl = make_smem_desc(st + 2 * C::A_BYTES + C::B_BYTES);
#pragma unroll
                                for (int k = 0; k < 4; ++k) umma_f8(d, tl + 2 * k, w + 2 * k, idesc2, 1u);
                            }
                        } else if (G1) {
                            const uint64_t a_up = make_smem_desc(st);
                            const uint64_t a_gate = make_smem_desc(st + C::A_BYTES);
                            const uint64_t b = make_smem_desc(st + 2 * C::A_BYTES);
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int sp = k % C::NSPLIT;
                                mm(d + sp * NTOK, a_up + 2 * k, b + 2 * k, k >= C::NSPLIT);
                                mm(d + (C::NSPLIT + sp) * NTOK, a_gate + 2 * k, b + 2 * k, k >= C::NSPLIT);
                            }
                        } else {
                            const uint64_t a0 = make_smem_desc(st);
                            const uint64_t a1 = make_smem_desc(st + C::A_BYTES);
                            const uint64_t bh = make_smem_desc(st + 2 * C::A_BYTES);
                            if constexpr (C::NSPLIT == 2) {
                                // hi and lo token tiles are adjacent in the stage and their partial accumulators adjacent in
                                // TMEM: ONE N = 2 NTOK MMA per weight tile and K step covers both (an MMA this narrow costs
                                // its weight-operand read, ~60 cycles, whatever N is: 16 of them per block took 950 cycles)
                                constexpr uint32_t idesc2 = make_idesc_f8(128, 2 * NTOK);
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    umma_f8(d, a0 + 2 * k, bh + 2 * k, idesc2, k > 0);
                                    umma_f8(d + 2 * NTOK, a1 + 2 * k, bh + 2 * k, idesc2, k > 0);
                                }
                            } else {
                                // hi and lo accumulate on top of each other
                                const uint64_t bl = make_smem_desc(st + 2 * C::A_BYTES + C::B_BYTES);
#pragma unroll
                                for (int k = 0; k < 8; ++k) {
                                    mm(d, a0 + 2 * (k & 3), (k < 4 ? bh : bl) + 2 * (k & 3), k > 0);
                                    mm(d + NTOK, a1 + 2 * (k & 3), (k < 4 ? bh : bl) + 2 * (k & 3), k > 0);
                                }
                            }
                        }
                        umma_commit(bar_empty + 8 * stage);
                        if (j + 1 == nj) umma_commit(bar_tfull + 8 * ab);
                        }
                        __syncwarp();
                        if (++stage == C::STAGES) { stage = 0; phase ^= 1; }
                    }
                    if (!ok) break;
                    if (++ab == C::NACC) { ab = 0; aphase ^= 1; }
                }
            }
            if (lane == 0) stamp(TR_MMA_LAST);
            x.stage = stage; x.phase = phase; x.ab = ab; x.aphase = aphase; x.n_item = n_item; x.ok = ok;
        }
        __syncwarp();
    } else if constexpr (C::TOK_ON_M) {
        // ------------------------------------------------------------ scale warp (2; with gathered rows 2 and 3), tokens on M:
        // token and weight scales of every K block into the block's slot of the ring, by asynchronous copies TS_AHEAD blocks
        // ahead.  It counts in on the barrier of the MMAs' commit when the scales of the block AND of the one after it have
        // landed, so that the promotion warps read a block's scales while they fold the one before: a shared-memory load
        // beside full-rate MMAs takes ~150 cycles, and nothing in a promotion warp hides that in front of a block's first
        // FMA (in a loop without TMA fills: 526 cycles per block with the load ahead, 650 with the load in place).
        if (warp - 2 < NHELP) {
            const int h = threadIdx.x - 64;            // gathered rows: this thread copies the scales of rows h and h + 64
            int ab = 0; uint32_t aphase = 0;
            bool ok = true;
            int n_item = 0, blk = 0;
            WorkItem wi;
#pragma unroll 1
            while (ok && wq_fetch(n_item++, wi, ok)) {
                const int gb = wi.gb, ge = wi.ge;
                const Unit un = wi.un;
                // weight-scale rows of the unit's two tiles (the second one of GEMM2's last unit may not exist): lanes 0 and 1
                const int srow0 = un.mt * (p.unit_rows >> 7);
                const int srow = lane == 0 ? srow0 : min(srow0 + (p.gate_offset >> 7), p.scale_rows - 1);
                const float* const ws = p.w_scale + ((size_t)un.e * p.scale_rows + srow) * p.KB;
                const float* ts[2] = {p.b_scale + (size_t)un.row0 + 4 * lane, nullptr};
                if (G4) {
#pragma unroll
                    for (int r = 0; r < 2; ++r) {
                        const int tok = __ldg(p.g4_row_token + un.row0 + h + 64 * r);
                        ts[r] = p.g4_scale + (tok >= 0 && tok < p.g4_T ? (size_t)tok * (unsigned)p.g4_tok_stride : 0);   // any finite scale for a row of zeros
                    }
                }
                auto fetch = [&](int kb, int b) {
                    if (kb < ge) {                      // nothing past the piece's end: no copy is left in flight for the next piece
                        const uint32_t slot = smem_u32(s_ts) + (uint32_t)(b % C::TSD) * (C::TS_SLOT * 4);
                        if (G4) {
                            cp_async4(slot + 4 * h, ts[0] + (size_t)kb * p.ts_stride);
                            cp_async4(slot + 4 * h + 64 * 4, ts[1] + (size_t)kb * p.ts_stride);
                        } else {
                            cp_async16(slot + 16 * lane, ts[0] + (size_t)kb * p.rows_cap);      // segments start at multiples of 16 rows
                        }
                        if (warp == 2 && lane < 2) cp_async4(slot + 128 * 4 + 4 * lane, ws + kb);
                    }
                    cp_async_commit();
                };
#pragma unroll 1
                for (int i = 0; i < C::TS_AHEAD; ++i) fetch(gb + i, blk + i);
#pragma unroll 1
                for (int kb = gb; kb < ge; ++kb) {
                    cp_async_wait<C::TS_AHEAD - 2>();  // the scales of blocks kb and kb + 1 have landed
                    __syncwarp();
                    // the accumulator is free: block blk - NACC has been folded, and nobody reads its slot or one before it
                    if (!mbar_wait_warp(bar_tempty + 8 * ab, aphase ^ 1, p.status, ERR_WAIT_TMEM_EMPTY)) { ok = false; break; }
                    if (lane == 0) mbar_arrive(bar_tfull + 8 * ab);
                    fetch(kb + C::TS_AHEAD, blk + C::TS_AHEAD);
                    ++blk;
                    if (++ab == C::NACC) { ab = 0; aphase ^= 1; }
                }
            }
            cp_async_wait<0>();
        }
    } else if (FUSE) {
        // ------------------------------------------------------------ warps 2-3, fused combine: zero rows of the
        // tokens that have no pair on this rank (nobody else writes them)
#pragma unroll 1
        for (int t = (int)blockIdx.x * 2 + (warp - 2); t < p.T; t += (int)gridDim.x * 2) {
            bool local = false;
            if (lane < p.top_k) {
                const int le = __ldg(p.c_topk + (size_t)t * p.c_stride + lane) - p.c_local_offset;
                local = le >= 0 && le < p.num_local;
            }
            if (__any_sync(0xFFFFFFFFu, local)) continue;
            uint4* o = reinterpret_cast<uint4*>(p.fuse_out + (size_t)t * p.H);
#pragma unroll 1
            for (int i = lane; i < p.H / 8; i += 32) o[i] = make_uint4(0u, 0u, 0u, 0u);
        }
    }
    } else {
        // ------------------------------------------------------------ promotion + epilogue
        if (C::REALLOC_REGS) {
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(C::PROMO_REGS));
        }
        const int pw = warp - 4;
        const int quarter = warp & 3;                  // TMEM lanes [32*quarter, +32)
        const int grp_id = pw >> 2;                    // column group (0 when NPW == 4)
        const int c0 = grp_id * C::NC;
        const int m = quarter * 32 + lane;             // weight row inside the tile
        const int ptid = threadIdx.x - 128;
        const uint32_t tlane = (uint32_t)(quarter * 32) << 16;
        volatile int* const s_last = s_flag + 8;
        const uint32_t my_red = bar_red + 8 * (C::TOK_ON_M ? quarter : grp_id);
        int stage = x.stage; uint32_t phase = x.phase;
        int ab = x.ab; uint32_t aphase = x.aphase;
        uint32_t rphase = x.rphase;
        int rbuf = x.rbuf;                             // half of s_red the next epilogue uses
        bool ok = true, seen = false;
        int ng = 0, nu = 0;
        int blk = 0;                                   // tokens on M: K blocks folded so far
        float acc[C::NACCUM][C::NC];

        // the warps that share my_red meet (bounded); false = gave up
        auto group_sync = [&]() -> bool {
            __syncwarp();
            if (lane == 0) mbar_arrive(my_red);
            const bool r = mbar_wait_warp(my_red, rphase, p.status, ERR_WAIT_GROUP);
            rphase ^= 1;
            return r;
        };

        int n_item = x.n_item;
        WorkItem wi;
        if ((WHICH != SECOND || x.fresh) && !(!C::TOK_ON_M && G1 && p.copied)) { pdl_wait(); pdl_launch(); }
        if (FUSE && !BOTH && p.met && blockIdx.x == 0 && ptid == 0) *p.met = 0;
#pragma unroll 1
        while (ok && wq_fetch(n_item++, wi, ok)) {
            const int gb = wi.gb, ge = wi.ge;
            const Unit un = wi.un;
            if (PART && quarter * 32 >= un.nvalid) {
                // no row of the unit in this warp's lanes: only hand the buffers back (the warp it meets in the epilogue has
                // no row either, here and in the CTAs that run other pieces of the unit)
#pragma unroll 1
                for (int n = ge - gb; n > 0; --n) {
                    if (!mbar_wait_warp(bar_tfull + 8 * ab, aphase, p.status, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
                    if (lane == 0) mbar_arrive(bar_tempty + 8 * ab);
                    if (++ab == C::NACC) { ab = 0; aphase ^= 1; }
                }
                blk += ge - gb;
                continue;
            }
#pragma unroll
            for (int a = 0; a < C::NACCUM; ++a)
#pragma unroll
                for (int i = 0; i < C::NC; ++i) acc[a][i] = 0.f;
            // narrow tiles: the weight scales of a group are fetched one group ahead (the token scales travel in the
            // stage), so their global-load latency never sits between the TMEM hand-off and the first FMA
            const float* ws0 = nullptr; const float* ws1 = nullptr;
            float swn[C::KPB][C::NACCUM];
            if (!C::TOK_ON_M) {
                // weight-scale rows of the unit's two tiles (the second one of GEMM2's last unit may not exist)
                const int srow0 = un.mt * (p.unit_rows >> 7);
                const int srow1 = min(srow0 + (p.gate_offset >> 7), p.scale_rows - 1);
                ws0 = p.w_scale + ((size_t)un.e * p.scale_rows + srow0) * p.KB;
                ws1 = p.w_scale + ((size_t)un.e * p.scale_rows + srow1) * p.KB;
#pragma unroll
                for (int j = 0; j < C::KPB; ++j) {
                    const int kb = min(gb * C::KPB + j, p.KB - 1);
                    swn[j][0] = __ldg(ws0 + kb);
                    swn[j][1] = __ldg(ws1 + kb);
                }
            }
            if constexpr (C::TOK_ON_M) {
                // Tokens on M: this thread's row is one token, so a K block folds with ONE scalar per weight tile.  The
                // block is read as four 32-column chunks, two tcgen05.ld in flight per wait (a wait covers every
                // outstanding load).  256 cycles of packed FMAs per block and scheduler; what the loop adds to them are round
                // trips to shared memory beside full-rate MMAs (~100-150 cycles each), so a block has as few in a row as
                // possible: its scales were read during the block before, the barrier is looked at between the last two
                // chunks (the answer is there when they are folded), waits do not vote (the lanes meet behind them and vote
                // once per piece), and the buffer goes back before those two chunks are folded.  GEMM1 of 14107 tokens 925 k -> 815 k cycles against a loop that
                // waits, votes and reads its scales in place (under the power limit 690 -> 645 us).
                constexpr int QC = 32, QPA = C::NC / QC, NQ = C::NACCUM * QPA;
                static_assert(C::NC % QC == 0 && NQ == 4 && C::KPB == 1, "tokens-on-M chunking");
                float stg[2][QC];
                uint32_t tbuf;
                auto qload = [&](int q) { tmem_ld_chunk<QC>(tbuf + (q / QPA) * NTOK + (q % QPA) * QC, stg[q & 1]); };
                auto qfold = [&](int q, float sx) {
                    const float2 s2 = make_float2(sx, sx);
                    float* ac = &acc[q / QPA][(q % QPA) * QC];
                    const float* v = stg[q & 1];
#pragma unroll
                    for (int i = 0; i < QC; i += 2) {
                        const float2 r0 = __ffma2_rn(make_float2(v[i], v[i + 1]), s2, make_float2(ac[i], ac[i + 1]));
                        ac[i] = r0.x; ac[i + 1] = r0.y;
                    }
                };
                uint32_t landed = 1;
                bool ready = false;
                mbar_wait_flag(bar_tfull + 8 * ab, aphase, landed);
                const float* slot = s_ts + (blk % C::TSD) * C::TS_SLOT;
                float t = slot[m];
                float2 w2 = *reinterpret_cast<const float2*>(slot + 128);
                if (ptid == 0 && !seen) { stamp(TR_PROMO_FIRST); seen = true; }
#pragma unroll 1
                for (int n = ge - gb; n > 0; --n) {
                    if (!ready) mbar_wait_flag(bar_tfull + 8 * ab, aphase, landed);
                    __syncwarp();          // each lane has waited by itself, and the loads below take the whole warp (.aligned)
                    if (ptid == 0) klog_put(2, ng);
                    const float2 sx2 = make_float2(t * w2.x, t * w2.y);
                    tc_fence_after();
                    tbuf = tmem_base + tlane + ab * C::BUFCOLS + c0;
                    qload(0); qload(1);
                    tmem_wait_ld();
                    qfold(0, sx2.x); qload(2);
                    qfold(1, sx2.x); qload(3);
                    ++blk;
                    slot = s_ts + (blk % C::TSD) * C::TS_SLOT;         // the next block's (behind the last one nobody uses them)
                    t = slot[m];
                    w2 = *reinterpret_cast<const float2*>(slot + 128);
                    tmem_wait_ld();
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0 && landed) mbar_arrive(bar_tempty + 8 * ab);     // never a buffer whose wait gave up
                    if (++ab == C::NACC) { ab = 0; aphase ^= 1; }
                    qfold(2, sx2.y);
                    ready = mbar_test(bar_tfull + 8 * ab, aphase);
                    qfold(3, sx2.y);
                    if (ptid == 0) klog_put(3, ng++);
                }
                if (!__all_sync(0xFFFFFFFFu, landed != 0)) {
                    if (lane == 0) atomicCAS(p.status, 0, ERR_WAIT_TMEM_FULL);
                    ok = false; break;
                }
            } else
#pragma unroll 1
            for (int grp = gb; grp < ge; ++grp) {
                const int kb0 = grp * C::KPB;
                const int nj = min(C::KPB, p.KB - kb0);
                float sw[C::KPB][C::NACCUM];
#pragma unroll
                for (int j = 0; j < C::KPB; ++j) {
                    sw[j][0] = swn[j][0]; sw[j][1] = swn[j][1];
                    const int kb = min(kb0 + C::KPB + j, p.KB - 1);
                    swn[j][0] = __ldg(ws0 + kb);
                    swn[j][1] = __ldg(ws1 + kb);
                }
                const int st0 = stage;
                float scr[C::EARLY_SCALES ? C::KPB : 1][C::EARLY_SCALES ? C::NC : 1];
                if (C::EARLY_SCALES) {
#pragma unroll
                    for (int j = 0; j < C::KPB; ++j) {
                        if (j < nj) {
                            int sj = st0 + j; if (sj >= C::STAGES) sj -= C::STAGES;
                            const uint32_t ph = (st0 + j >= C::STAGES) ? (phase ^ 1) : phase;
                            if (!mbar_wait_warp(bar_full + 8 * sj, ph, p.status, ERR_WAIT_SMEM_FULL)) ok = false;
                            // (ld.shared: behind a load through a generic address the stage could be released, and its scales
                            // overwritten, while the load was still under way - 64-token tiles, a third of 901-token calls)
                            const uint32_t scp = smem_base + sj * C::STAGE_BYTES + C::SC_OFF + 4 * c0;
#pragma unroll
                            for (int i = 0; i < C::NC; i += 4) {
                                const float4 s4 = ld_shared_f4(scp + 4 * i);
                                scr[j][i] = s4.x; scr[j][i + 1] = s4.y; scr[j][i + 2] = s4.z; scr[j][i + 3] = s4.w;
                            }
                        }
                    }
                    if (!ok) break;
                    __syncwarp();
                    if (lane == 0) {
#pragma unroll 1
                        for (int j = 0; j < nj; ++j) {
                            int sj = st0 + j; if (sj >= C::STAGES) sj -= C::STAGES;
                            mbar_arrive(bar_empty + 8 * sj);
                        }
                    }
                }
                if (!mbar_wait_warp(bar_tfull + 8 * ab, aphase, p.status, ERR_WAIT_TMEM_FULL)) { ok = false; break; }
                if (ptid == 0 && !seen) { stamp(TR_PROMO_FIRST); seen = true; }
                if (ptid == 0) klog_put(2, ng);
                tc_fence_after();
                const uint32_t tbuf = tmem_base + tlane + ab * C::BUFCOLS + c0;

                // flattened chunk list (K block, column chunk, accumulator, partial); the tcgen05.ld of
                // chunk k+1 is in flight while chunk k is folded into the accumulators
                constexpr int NCH = C::NC / C::CH;
                constexpr int NK = C::KPB * NCH * C::NACCUM * C::NSPLIT;
                float part[2][C::CH];
                tmem_ld_chunk<C::CH>(tbuf, part[0]);
#pragma unroll
                for (int k = 0; k < NK; ++k) {
                    const int sp = k % C::NSPLIT;
                    const int a = (k / C::NSPLIT) % C::NACCUM;
                    const int ch = (k / (C::NSPLIT * C::NACCUM)) % NCH;
                    const int j = k / (C::NSPLIT * C::NACCUM * NCH);
                    if (j < nj) {
                        tmem_wait_ld();
                        if (k + 1 < NK) {
                            const int sp1 = (k + 1) % C::NSPLIT;
                            const int a1 = ((k + 1) / C::NSPLIT) % C::NACCUM;
                            const int ch1 = ((k + 1) / (C::NSPLIT * C::NACCUM)) % NCH;
                            const int j1 = (k + 1) / (C::NSPLIT * C::NACCUM * NCH);
                            if (j1 < nj)
                                tmem_ld_chunk<C::CH>(tbuf + j1 * C::CPB + (a1 * C::NSPLIT + sp1) * NTOK + ch1 * C::CH,
                                                     part[(k + 1) & 1]);
                        }
                        const float swa = sw[j][a];
                        if (C::EARLY_SCALES) {
#pragma unroll
                            for (int i = 0; i < C::CH; i += 2) {
                                const float2 mm = __fmul2_rn(make_float2(scr[j][ch * C::CH + i], scr[j][ch * C::CH + i + 1]),
                                                             make_float2(swa, swa));
                                float* ac = &acc[a][ch * C::CH + i];
                                const float2 r0 = __ffma2_rn(make_float2(part[k & 1][i], part[k & 1][i + 1]), mm,
                                                             make_float2(ac[0], ac[1]));
                                ac[0] = r0.x; ac[1] = r0.y;
                            }
                        } else {
                            int sj = st0 + j; if (sj >= C::STAGES) sj -= C::STAGES;
                            if (C::SCALES_IN_STAGE && ch == 0 && a == 0 && sp == 0) {
                                // token scales of this K block arrived with the stage's transaction barrier
                                const uint32_t ph = (st0 + j >= C::STAGES) ? (phase ^ 1) : phase;
                                if (!mbar_wait_warp(bar_full + 8 * sj, ph, p.status, ERR_WAIT_SMEM_FULL)) ok = false;
                            }
                            {
                                const uint32_t scp = smem_base + sj * C::STAGE_BYTES + C::SC_OFF + 4 * (c0 + ch * C::CH);
#pragma unroll
                                for (int i = 0; i < C::CH; i += 4) {
                                    const float4 s4 = ld_shared_f4(scp + 4 * i);
                                    const float2 m0 = __fmul2_rn(make_float2(s4.x, s4.y), make_float2(swa, swa));
                                    const float2 m1 = __fmul2_rn(make_float2(s4.z, s4.w), make_float2(swa, swa));
                                    float* ac = &acc[a][ch * C::CH + i];
                                    const float2 r0 = __ffma2_rn(make_float2(part[k & 1][i], part[k & 1][i + 1]), m0, make_float2(ac[0], ac[1]));
                                    const float2 r1 = __ffma2_rn(make_float2(part[k & 1][i + 2], part[k & 1][i + 3]), m1, make_float2(ac[2], ac[3]));
                                    ac[0] = r0.x; ac[1] = r0.y; ac[2] = r1.x; ac[3] = r1.y;
                                }
                            }
                        }
                    }
                }
                if (!ok) break;
                // all tcgen05.ld of this buffer have completed (the last wait above) and all scale reads are done
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(bar_tempty + 8 * ab);
                    if (C::SCALES_IN_STAGE && !C::EARLY_SCALES) {
#pragma unroll 1
                        for (int j = 0; j < nj; ++j) {
                            int sj = st0 + j; if (sj >= C::STAGES) sj -= C::STAGES;
                            mbar_arrive(bar_empty + 8 * sj);
                        }
                    }
                }
                if (ptid == 0) klog_put(3, ng++);
                stage += nj;
                if (stage >= C::STAGES) { stage -= C::STAGES; phase ^= 1; }
                if (++ab == C::NACC) { ab = 0; aphase ^= 1; }
            }
            if (!ok) break;
            if (ptid == 0) stamp(TR_PROMO_LAST);

            if (wi.pieces > 1) {
                // a slot holds four accumulators of a thread together: [NACCUM * NC / 4][NPT] of 16 bytes
                float4* const slots = reinterpret_cast<float4*>(p.sk_partial + (size_t)wi.slot * C::SLOT_FLOATS) + ptid;
                constexpr int SLOT_VECS = C::SLOT_FLOATS / 4, ACC_VECS = C::NACCUM * C::NC / 4;
                auto slot_of = [&](int c) -> float4* { return slots + (size_t)c * SLOT_VECS; };
                auto acc4 = [&](int k) -> float* { return &acc[4 * k / C::NC][4 * k % C::NC]; };
                auto store_partial = [&]() {
                    float4* slot = slot_of(wi.piece);
#pragma unroll
                    for (int k = 0; k < ACC_VECS; ++k) __stcg(slot + k * C::NPT, make_float4(acc4(k)[0], acc4(k)[1], acc4(k)[2], acc4(k)[3]));
                };
                int* const arrived = p.sk_count + 4 * wi.ut;
                constexpr bool ENDS = C::STATIC_TAIL || WHICH == FIRST;          // the piece that ends a unit finishes it
                if constexpr (ENDS) {
                    // ---- piece of a split unit, static ranges: the piece that ends the unit finishes it.  The others store
                    // their partial sums and count their warps in with a release - no meeting of the warps, no answer to
                    // wait for; the finisher waits (bounded) for that count.
                    if (wi.ge < NG) {
                        store_partial();
                        __syncwarp();        // orders the lanes' stores before lane 0's release below
                        if (lane == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(arrived) : "memory");
                        if (ptid == 0) stamp(TR_PARTIAL);
                        continue;
                    }
                    const int want = (wi.pieces - 1) * C::NPW;
                    bool here = true;
                    if (lane == 0) {
                        const unsigned long long t0 = globaltimer_ns();
#pragma unroll 1
                        for (uint32_t it = 1;; ++it) {
                            int v;
                            asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(arrived) : "memory");
                            if (v >= want) break;
                            if ((it & 0xFFu) == 0 && globaltimer_ns() - t0 > WAIT_LIMIT_NS) {
                                atomicCAS(p.status, 0, ERR_WAIT_CHUNKS); here = false; break;
                            }
                        }
                    }
                    here = __shfl_sync(0xFFFFFFFFu, here, 0);
                    __syncwarp();            // lane 0's acquire orders the other lanes' loads too (a shuffle orders nothing)
                    if (!here) { ok = false; break; }
                } else {
                    // ---- piece of a split unit, claimed chunks: every piece stores its partial sums; the warps that arrive
                    // last (a warp of GEMM2 by itself; those that meet in the epilogue, my_red, together in GEMM1) add all
                    // pieces in a fixed order - the last one in K, then the others from the first on - and run the epilogue.
                    // Nobody waits for another CTA.  (Waiting in the CTA that runs the last piece chained the waits: partial
                    // sums are stored only after the piece before them in the same CTA, which may be waiting itself.
                    // T=257, GEMM2: 81 -> 74 us.)
                    const int fld = G1 ? (C::TOK_ON_M ? quarter : grp_id) : pw;
                    store_partial();
                    __threadfence();
                    __syncwarp();
                    if (ptid == 0) stamp(TR_PARTIAL);
                    int seen_pieces = 0;
                    auto count_in = [&]() {
                        seen_pieces = (int)((unsigned)atomicAdd(arrived + (fld >> 2), 1 << (8 * (fld & 3))) >> (8 * (fld & 3))) & 0xFF;
                    };
                    if (G1) {
                        if (!group_sync()) { ok = false; break; }
                        const bool leader = C::TOK_ON_M ? grp_id == 0 : quarter == 0;
                        if (leader && lane == 0) { count_in(); s_last[fld] = seen_pieces; }
                        if (!group_sync()) { ok = false; break; }
                        seen_pieces = s_last[fld];
                    } else {
                        if (lane == 0) count_in();
                        seen_pieces = __shfl_sync(0xFFFFFFFFu, seen_pieces, 0);
                        __syncwarp();        // as above: before the fence of the lanes that read the other pieces
                    }
                    if (seen_pieces != wi.pieces - 1) continue;
                    __threadfence();
                }
                if (!ENDS && wi.piece != wi.pieces - 1) {
                    const float4* src = slot_of(wi.pieces - 1);
#pragma unroll
                    for (int k = 0; k < ACC_VECS; ++k) {
                        const float4 v = __ldcg(src + k * C::NPT);
                        acc4(k)[0] = v.x; acc4(k)[1] = v.y; acc4(k)[2] = v.z; acc4(k)[3] = v.w;
                    }
                }
                const int n_other = wi.pieces - 1;
                if constexpr (ACC_VECS <= 8) {
                    // narrow tiles: the next piece's slot is in flight while this one is added (same fixed order)
                    float4 nxt[ACC_VECS];
#pragma unroll
                    for (int k = 0; k < ACC_VECS; ++k) nxt[k] = __ldcg(slot_of(0) + k * C::NPT);
#pragma unroll 1
                    for (int c = 0; c < n_other; ++c) {
                        float4 cur[ACC_VECS];
#pragma unroll
                        for (int k = 0; k < ACC_VECS; ++k) cur[k] = nxt[k];
                        if (c + 1 < n_other) {
#pragma unroll
                            for (int k = 0; k < ACC_VECS; ++k) nxt[k] = __ldcg(slot_of(c + 1) + k * C::NPT);
                        }
#pragma unroll
                        for (int k = 0; k < ACC_VECS; ++k) {
                            acc4(k)[0] += cur[k].x; acc4(k)[1] += cur[k].y; acc4(k)[2] += cur[k].z; acc4(k)[3] += cur[k].w;
                        }
                    }
                } else {
#pragma unroll 1
                    for (int c = 0; c < n_other; ++c) {
                        const float4* src = slot_of(c);
#pragma unroll
                        for (int k = 0; k < ACC_VECS; ++k) {
                            const float4 v = __ldcg(src + k * C::NPT);
                            acc4(k)[0] += v.x; acc4(k)[1] += v.y; acc4(k)[2] += v.z; acc4(k)[3] += v.w;
                        }
                    }
                }
            }

            if (ptid == 0) { stamp(TR_REDUCED); klog_put(4, nu); }
            if (C::TOK_ON_M && G1) {
                // this thread: token row m, NC consecutive columns j of the 128-wide block -> SwiGLU, amax over
                // the block (own columns, then the other column groups' threads of the same row), two e4m3
                // terms, 16-byte stores
                float amax = 0.f;
#pragma unroll
                for (int i = 0; i < C::NC; ++i) {
                    const float v = silu_f(acc[1][i]) * acc[0][i];
                    acc[0][i] = v;
                    amax = fmaxf(amax, fabsf(v));
                }
                // [2][NGRP][128], used in turn: a warp is at most one meeting ahead of the one it meets
                float* redf = reinterpret_cast<float*>(s_red) + rbuf * (C::NGRP * 128);
                rbuf ^= 1;
                redf[grp_id * 128 + m] = amax;
                if (!group_sync()) { ok = false; break; }
#pragma unroll
                for (int g2 = 0; g2 < C::NGRP; ++g2) amax = fmaxf(amax, redf[g2 * 128 + m]);
                const float scale = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
                const float inv = amax > 0.f ? 448.0f / amax : 0.f;
                if (m < un.nvalid) {
                    const size_t row = (size_t)(un.row0 + m);
                    uint8_t* dhi = p.act_hi + row * p.I + (size_t)un.mt * 128 + c0;
                    uint8_t* dlo = p.act_lo + row * p.I + (size_t)un.mt * 128 + c0;
#pragma unroll
                    for (int v8 = 0; v8 < C::NC / 32; ++v8) {
                        uint32_t wh[8], wl[8];
#pragma unroll
                        for (int w4 = 0; w4 < 8; ++w4) {
                            const int i = v8 * 32 + w4 * 4;
                            const float q0 = acc[0][i] * inv, q1 = acc[0][i + 1] * inv;
                            const float q2 = acc[0][i + 2] * inv, q3 = acc[0][i + 3] * inv;
                            const uint16_t h01 = f32x2_to_e4m3x2(q0, q1), h23 = f32x2_to_e4m3x2(q2, q3);
                            const float2 f01 = e4m3x2_to_f32x2(h01), f23 = e4m3x2_to_f32x2(h23);
                            const uint16_t l01 = f32x2_to_e4m3x2(q0 - f01.x, q1 - f01.y);
                            const uint16_t l23 = f32x2_to_e4m3x2(q2 - f23.x, q3 - f23.y);
                            wh[w4] = (uint32_t)h01 | ((uint32_t)h23 << 16);
                            wl[w4] = (uint32_t)l01 | ((uint32_t)l23 << 16);
                        }
                        st_global_v8(dhi + v8 * 32, wh[0], wh[1], wh[2], wh[3], wh[4], wh[5], wh[6], wh[7]);
                        st_global_v8(dlo + v8 * 32, wl[0], wl[1], wl[2], wl[3], wl[4], wl[5], wl[6], wl[7]);
                    }
                    if (grp_id == 0) p.act_scale[(size_t)un.mt * p.rows_cap + row] = scale;
                }
            } else if (C::TOK_ON_M) {
                // 64 consecutive output columns of this thread's row per accumulator, as 256-bit stores.
                // A unit's rows drain at ~32 B per cycle per SM whatever the pattern (a shuffle transpose that
                // made every lane quad write 128 contiguous bytes was measured equal), so they leave as fp16.
                if (m < un.nvalid) {
                    const size_t row = (size_t)(un.row0 + m);
#pragma unroll
                    for (int a = 0; a < C::NACCUM; ++a) {
                        const int col0 = un.mt * p.unit_rows + a * p.gate_offset + c0;
                        if (col0 < p.valid_rows) store_y_row<C::NC>(p.y + row * p.H + col0, acc[a]);
                    }
                }
            } else if (G1) {
                // SwiGLU, then amax over the 128 rows of the tile for every token column.  A column's scale and reciprocal
                // are computed by one lane of every warp (lane i: column i) and handed out by shuffles; four columns'
                // bytes are transposed inside lane quads so that a store carries four weight rows of one token.  (Per
                // column and thread a division and two byte stores, with one warp per scheduler to hide nothing behind:
                // 6000 cycles for 16 columns at the end of every unit.)
                uint32_t* red = s_red + rbuf * (C::NPW * C::NC);
                rbuf ^= 1;
                uint32_t colmax = 0;
#pragma unroll
                for (int i = 0; i < C::NC; ++i) {
                    const float v = silu_f(acc[1][i]) * acc[0][i];
                    acc[0][i] = v;
                    const uint32_t wm = __reduce_max_sync(0xFFFFFFFFu, __float_as_uint(fabsf(v)));
                    if (lane == i) colmax = wm;
                }
                if (lane < C::NC) red[pw * C::NC + lane] = colmax;
                if (!group_sync()) { ok = false; break; }
                float inv = 0.f;
                if (lane < C::NC) {
                    const uint32_t* rg = red + grp_id * 4 * C::NC + lane;
                    const float amax = __uint_as_float(max(max(rg[0], rg[C::NC]), max(rg[2 * C::NC], rg[3 * C::NC])));
                    inv = amax > 0.f ? 448.0f / amax : 0.f;
                    if (quarter == 0 && c0 + lane < un.nvalid)
                        p.act_scale[(size_t)un.mt * p.rows_cap + un.row0 + c0 + lane] = amax > 0.f ? amax * (1.0f / 448.0f) : 1.0f;
                }
                const size_t out0 = (size_t)(un.row0 + c0 + (lane & 3)) * p.I + (size_t)un.mt * 128 + quarter * 32 + (lane & ~3);
                // 4 x 4 byte transpose inside a lane quad: in, byte j = column i + j of this lane's weight row; out, byte j =
                // weight row (lane & ~3) + j of column i + (lane & 3)
                auto quad_transpose = [&](uint32_t x) -> uint32_t {
                    const uint32_t y = __shfl_xor_sync(0xFFFFFFFFu, x, 1);
                    const uint32_t r = __byte_perm(x, y, (lane & 1) ? 0x3715 : 0x6240);
                    const uint32_t z = __shfl_xor_sync(0xFFFFFFFFu, r, 2);
                    return __byte_perm(r, z, (lane & 2) ? 0x3276 : 0x5410);
                };
#pragma unroll
                for (int i = 0; i < C::NC; i += 4) {
                    float q[4];
#pragma unroll
                    for (int j = 0; j < 4; ++j) q[j] = acc[0][i + j] * __shfl_sync(0xFFFFFFFFu, inv, i + j);
                    const uint16_t h01 = f32x2_to_e4m3x2(q[0], q[1]), h23 = f32x2_to_e4m3x2(q[2], q[3]);
                    const float2 f01 = e4m3x2_to_f32x2(h01), f23 = e4m3x2_to_f32x2(h23);
                    const uint16_t l01 = f32x2_to_e4m3x2(q[0] - f01.x, q[1] - f01.y), l23 = f32x2_to_e4m3x2(q[2] - f23.x, q[3] - f23.y);
                    const uint32_t hi = quad_transpose((uint32_t)h01 | ((uint32_t)h23 << 16));
                    const uint32_t lo = quad_transpose((uint32_t)l01 | ((uint32_t)l23 << 16));
                    if (c0 + i + (lane & 3) < un.nvalid) {
                        *reinterpret_cast<uint32_t*>(p.act_hi + out0 + (size_t)i * p.I) = hi;
                        *reinterpret_cast<uint32_t*>(p.act_lo + out0 + (size_t)i * p.I) = lo;
                    }
                }
            } else {
                const int col0 = un.mt * p.unit_rows + m;
                const bool second = col0 + p.gate_offset < p.valid_rows;
#pragma unroll
                for (int i = 0; i < C::NC; ++i) {
                    const int c = c0 + i;
                    if (c < un.nvalid) {
                        const size_t row = (size_t)(un.row0 + c);
                        p.y[row * p.H + col0] = __float2half_rn(acc[0][i]);
                        if (second) p.y[row * p.H + col0 + p.gate_offset] = __float2half_rn(acc[1][i]);
                    }
                }
                if (FUSE) {
                    // Fused combine.  This warp has stored its 64 of the unit's 256 columns (32 of either weight tile) of the
                    // column group's NC rows: fence, then count them in for every row's token (lane i: row i, all atomics in
                    // flight together; byte `quarter` of the token's word).  The warp that brings a token's byte to the number
                    // of its local pairs adds up those 64 columns of its rows, four tokens at a time.  (One warp for all 256
                    // columns of a token, one token after the other, left up to NC chains of dependent loads to the last of
                    // the four warps: 200 tokens of a 512-wide shape 66.5 us,
                    // now 42.7.)
                    __threadfence();
                    __syncwarp();
                    const int c = c0 + lane;
                    const bool mine = lane < C::NC && c < un.nvalid;
                    int t = -1;
                    bool last = false;
                    if (mine) {
                        t = __ldg(p.row_token + un.row0 + c);
                        int need = 0;
#pragma unroll 1
                        for (int k = 0; k < p.top_k; ++k) {
                            const int le = __ldg(p.c_topk + (size_t)t * p.c_stride + k) - p.c_local_offset;
                            need += le >= 0 && le < p.num_local;
                        }
                        const unsigned was = (unsigned)atomicAdd(p.tok_count + (size_t)t * p.n_mtiles + un.mt, 1 << (8 * quarter));
                        last = (int)((was >> (8 * quarter)) & 0xFFu) == need - 1;
                    }
                    unsigned todo = __ballot_sync(0xFFFFFFFFu, last);
                    __syncwarp();                       // as for the split units: the counting lane before the fence of all
                    if (todo) __threadfence();          // the other units' rows, counted in before this one, are visible
                    const int h = un.mt * p.unit_rows + ((lane & 4) ? p.gate_offset : 0) + quarter * 32 + (lane & 3) * 8;
                    while (todo) {
                        int src = -1;                   // lane that counted the token of this lane's group of eight
#pragma unroll
                        for (int g = 0; g < 4; ++g) {
                            if ((lane >> 3) == g) src = __ffs(todo) - 1;
                            todo &= todo - 1;
                        }
                        const int tt = __shfl_sync(0xFFFFFFFFu, t, max(src, 0));
                        combine_four_tokens(p.y, p.c_topk, p.pair_row, p.row_w, p.fuse_out, src < 0 ? -1 : tt, p.H, p.top_k, p.c_stride,
                                            p.c_local_offset, p.num_local, h, lane);
                    }
                }
            }
            if (WHICH == FIRST) {
                // this warp's part of the unit's rows is stored: other CTAs load them by TMA once every warp has counted in
                asm volatile("fence.proxy.async.global;" ::: "memory");
                __syncwarp();
                if (lane == 0) asm volatile("red.release.gpu.global.add.s32 [%0], 1;" ::"l"(p.tile_done + wi.tile) : "memory");
            }
            if (ptid == 0) klog_put(5, nu++);
        }
        x.stage = stage; x.phase = phase; x.ab = ab; x.aphase = aphase; x.rphase = rphase; x.rbuf = rbuf; x.n_item = n_item; x.ok = ok;
    }

    if (warp >= 4 && threadIdx.x == 128) stamp(TR_EPILOGUE);
}

template <int NTOK, bool G1, bool G4 = false, bool PART = false, bool FUSE = false>
__global__ void __launch_bounds__(GemmCfg<NTOK, G1>::NTHREADS, 1)
gemm_kernel(const __grid_constant__ CUtensorMap tm_w, const __grid_constant__ CUtensorMap tm_b0,
            const __grid_constant__ CUtensorMap tm_b1, const __grid_constant__ CUtensorMap tm_s0,
            const __grid_constant__ CUtensorMap tm_s1, const GemmParams p) {
    using C = GemmCfg<NTOK, G1>;
    extern __shared__ uint8_t smem_raw[];
    GemmCta x;
    gemm_setup<C>(x, smem_raw);
    if (p.trace && threadIdx.x == 0) p.trace[(size_t)blockIdx.x * TRACE_SLOTS + TR_ENTRY] = (long long)globaltimer_ns();
    gemm_init<C, helper_warps<C::TOK_ON_M, G4>()>(x, tm_w, tm_b0, G1 ? tm_b0 : tm_b1);
    gemm_roles<NTOK, G1, G4, PART, FUSE, SOLE>(x, tm_w, tm_b0, tm_b1, tm_s0, tm_s1, p);
    gemm_teardown<C>(x);
    if (p.trace && threadIdx.x == 0) p.trace[(size_t)blockIdx.x * TRACE_SLOTS + TR_EXIT] = clock64() - x.t_entry;
}

// parts: 1 GEMM1, 2 GEMM2, 3 both - in two launches for the stage times of the profile, with the same pieces and the same bits.
template <int NTOK, bool FUSE>
__global__ void __launch_bounds__(GemmCfg<NTOK, true, true>::NTHREADS, 1)
gemm_both_kernel(const __grid_constant__ CUtensorMap tm_w13, const __grid_constant__ CUtensorMap tm_a,
                 const __grid_constant__ CUtensorMap tm_w2, const __grid_constant__ CUtensorMap tm_hi,
                 const __grid_constant__ CUtensorMap tm_lo, const GemmParams p1, const GemmParams p2, const int parts) {
    using C = GemmCfg<NTOK, true, true>;
    using C2 = GemmCfg<NTOK, false, true>;
    static_assert(C::STAGE_BYTES == C2::STAGE_BYTES && C::SC_OFF == C2::SC_OFF && C::STAGES == C2::STAGES && C::SMEM_BYTES == C2::SMEM_BYTES &&
                  C::BUFCOLS == C2::BUFCOLS && C::NACC == C2::NACC && C::KPB == C2::KPB && C::NTHREADS == C2::NTHREADS &&
                  C::EMPTY_COUNT == C2::EMPTY_COUNT && C::RED_BYTES == C2::RED_BYTES, "the rings are carried over");
    extern __shared__ uint8_t smem_raw[];
    GemmCta x;
    gemm_setup<C>(x, smem_raw);
    if (threadIdx.x == 0) {                     // (trace is null for the GEMM that this launch does not do)
        const long long now = (long long)globaltimer_ns();
        if (p1.trace) p1.trace[(size_t)blockIdx.x * TRACE_SLOTS + TR_ENTRY] = now;
        if (p2.trace) p2.trace[(size_t)blockIdx.x * TRACE_SLOTS + TR_ENTRY] = now;
    }
    gemm_init<C, 0>(x, tm_w13, tm_a, tm_w2);
    if (parts & 1) {
        gemm_roles<NTOK, true, false, false, false, FIRST>(x, tm_w13, tm_a, tm_a, tm_a, tm_a, p1);
        x.fresh = false;
    }
    if (x.ok && (parts & 2)) gemm_roles<NTOK, false, false, false, FUSE, SECOND>(x, tm_w2, tm_hi, tm_lo, tm_hi, tm_lo, p2);
    gemm_teardown<C>(x);
    if (FUSE && p2.met && threadIdx.x == 0) {
        // The last kernel of the forward (met is null in another one) clears the count of the front end's meeting.  Every CTA comes by here, also one that gave up,
        // after its warps 2-3 have waited for the front end: behind the last of them nobody watches the count any more.
        __threadfence();
        if (atomicAdd(p2.met + 1, 1) == (int)gridDim.x - 1) { p2.met[0] = 0; p2.met[1] = 0; }
    }
    if (threadIdx.x == 0) {
        const long long cycles = clock64() - x.t_entry;
        if (p1.trace) p1.trace[(size_t)blockIdx.x * TRACE_SLOTS + TR_EXIT] = cycles;
        if (p2.trace) p2.trace[(size_t)blockIdx.x * TRACE_SLOTS + TR_EXIT] = cycles;
    }
}

}  // namespace b200moe
