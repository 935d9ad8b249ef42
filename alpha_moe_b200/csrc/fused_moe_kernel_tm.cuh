// Token-major variant of the fused W8A8 MoE kernel for large blocks (64 < block_m <= 128).
//
// Same operator and same work decomposition as fused_moe_kernel.cuh (which replaces
// csrc/kernels/fused_moe_w8a8/fused_moe_w8a8_up_down_acc.cu:654-1098), but with the operands the other
// way round: the block's tokens are the UMMA "M" operand (one token per TMEM lane, padded to 128) and
// the weight rows are the "N" operand (256 per instruction).  With a full block this runs the tensor
// pipe at its rated speed (an M=128, N=256, K=32 fp8 UMMA is compute-bound; the weight-major
// orientation is operand-fetch-bound at N <= 64), and everything the epilogue does becomes local to
// one thread = one token:
//   * scale promotion needs two scalars per chunk (token scale x gate / up block scale) instead of a
//     multiplication per column (reference :915-933);
//   * the interleaved gate/up rows arrive as interleaved accumulator columns (columns 16j..16j+7 gate,
//     16j+8..16j+15 up of the same intermediate columns), so SwiGLU needs no data movement
//     (reference :919-931, :945-946 obtains the same pairing inside a wgmma fragment);
//   * the fp8 intermediate is written as 16-byte vectors into the swizzled operand tile;
//   * each thread owns consecutive hidden columns of its token in the down-projection, so the
//     accumulation into `out` is done with 16-byte vector reductions (red.global.add.noftz.v4.bf16x2)
//     instead of one 4-byte reduction per pair of columns (reference :1085-1091 uses a 512-byte bulk
//     reduce per row).
//
// Ring slot: [256 weight rows x 128 B = 32 KB][128 token rows x 128 B = 16 KB]; slot contents as in
// fused_moe_kernel.cuh.  TMEM: up phase two buffers of 256 columns (one per K chunk in flight); down
// phase two buffers of 256 columns (SPC = 1: two hidden tiles; SPC = 2: the two slices' partial sums
// of one hidden tile, combined by the epilogue because each carries its own scales; SPC = 4: slices 0 and 1 of a
// hidden tile, then 2 and 3).
#pragma once

#include "fused_moe_kernel.cuh"

namespace amoe {

constexpr int kTmRows = 128;   // token rows of a block (TMEM lanes)
constexpr int kStgPitch = 144;                     // staging row pitch: 128 B + 16 B so that rows spread over the banks
constexpr int kStgWarpBytes = 32 * kStgPitch;      // one warp's staging tile
constexpr uint32_t kStgAliased = 0xFFFFFFFFu;      // SmemPlanTm::stage_out when the staging tiles alias the ring

struct SmemPlanTm {
    uint32_t stage_bytes, hq, stage_out, swg, swu, sw2, amaxx, xs, bars, misc, total;
};
// Row maxima of consecutive slices go to two sets of words in turn where nothing else keeps a warp from writing the next
// slice's before its partner has read this one's.  With two accumulator buffers a warp ends a slice only when every warp has
// released the slice's third chunk from the end, so from three chunks a slice on that is a chunk of the same slice, which the
// partner released after it read the maxima before.  (With two slices and more chunks a second set would be 1 KB that the
// largest accepted hidden size lacks.)
__host__ __device__ constexpr bool two_sets_of_maxima(int spc, int kc) { return spc == 4 || (spc == 2 && kc <= 2); }

__host__ __device__ inline SmemPlanTm smem_plan_tm(int s, int kc, int spc) {
    SmemPlanTm p;
    p.stage_bytes = 2 * kTileBytes + kTmRows * 128;
    uint32_t o = s * p.stage_bytes;
    p.hq = o;     o += spc * kTmRows * 128;
    // token scales [K chunk][token]; with four slices they start in the last slice's intermediate, which is written when
    // they are needed no more
    if (spc == 4) {
        p.xs = p.hq + 3 * kTmRows * 128;
        if (p.xs + kc * kTmRows * 4 > o) o = p.xs + kc * kTmRows * 4;
    }
    // per epilogue warp a staging tile of 32 rows x 128 B (+16 B pitch padding) for the down phase; with three
    // or more ring slots these live in the slots' token-row tiles, which that phase does not use
    if (s >= 3) { p.stage_out = kStgAliased; } else { p.stage_out = o;  o += 8 * kStgWarpBytes; }
    p.swg = o;    o += spc * kc * 4;
    p.swu = o;    o += spc * kc * 4;
    p.sw2 = o;    o += spc * kc * 4;
    o = (o + 15u) & ~15u;
    p.amaxx = o;  o += (two_sets_of_maxima(spc, kc) ? 4 : 2) * kTmRows * 4;
    if (spc < 4) { p.xs = o;  o += kc * kTmRows * 4; }
    p.bars = o;   o += (2 * s + (spc == 4 ? 11 : 7)) * 8;
    p.misc = o;   o += 16;
    p.total = o;
    return p;
}

// Token scales of one token into shared memory, xs[c * PITCH] for the K chunks of units first, first + step, ... (a unit is
// four chunks where the rows can be read as float4, else one).  All loads of a batch are in flight before the first store:
// this stands in front of the first promotion, and a load that waits for the one before costs a memory latency each.  With the
// sorted ids requested at kernel entry, calls in a row, DeepSeek-V3 TP8 shard, M = 4096 542 -> 535 us, M = 8192 (Zipf) 897 ->
// 887, Qwen3-Next shard M = 4096 235 -> 233.
template <int PITCH, int BATCH>
__device__ __forceinline__ void stage_token_scales(float* xs, const float* row, bool live, int first, int step, int units,
                                                   bool vec4) {
    if (vec4) {
        for (int u0 = first; u0 < units; u0 += BATCH * step) {
            float4 v[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int u = u0 + i * step;
                v[i] = live && u < units ? reinterpret_cast<const float4*>(row)[u] : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int u = u0 + i * step;
                if (u < units) {
                    xs[(4 * u) * PITCH] = v[i].x;
                    xs[(4 * u + 1) * PITCH] = v[i].y;
                    xs[(4 * u + 2) * PITCH] = v[i].z;
                    xs[(4 * u + 3) * PITCH] = v[i].w;
                }
            }
        }
    } else {
        for (int u0 = first; u0 < units; u0 += BATCH * step) {
            float v[BATCH];
#pragma unroll
            for (int i = 0; i < BATCH; ++i) {
                const int u = u0 + i * step;
                v[i] = live && u < units ? row[u] : 0.f;
            }
#pragma unroll
            for (int i = 0; i < BATCH; ++i)
                if (u0 + i * step < units) xs[(u0 + i * step) * PITCH] = v[i];
        }
    }
}

constexpr int kTmThreads = 512;     // 2 epilogue warpgroups + control warpgroup + gather warpgroup
constexpr int kTmGatherWarps = 5;   // one warp of the control warpgroup + the gather warpgroup

template <int SPC>
__global__ void __launch_bounds__(kTmThreads, 1)
fused_moe_w8a8_up_down_sm100_tokmajor_kernel(const __grid_constant__ CUtensorMap tm_w,
                                             const __grid_constant__ CUtensorMap tm_w2, const MoeParams p) {
    constexpr int EPI_THREADS = 256;
    // control warpgroup: weight TMA, gather, UMMA, one warp without a role; then four more gather warps.
    // A 128-row x 128-byte token tile is 32 cp.async of 32 lanes x 16 bytes.  A warp issues one in 7-15 cycles, but they are
    // in flight for several hundred (five warps x 16 of them are done in about 520): five warps bring a tile in about as
    // long as its UMMAs run.
    constexpr int W_TMA = 8, W_G0 = 9, W_MMA0 = 10, W_G1 = 12;
    constexpr int GATHER_THREADS = kTmGatherWarps * 32;
    constexpr uint32_t TMEM_COLS = 512;
    static_assert(SPC == 1 || SPC == 2 || SPC == 4, "slices per CTA");

    const int ngroups = (p.N >> 8) / SPC;
    const int mblock = blockIdx.x / ngroups;
    const int slice0 = (blockIdx.x - mblock * ngroups) * SPC;
    griddep_wait();      // the schedule, the activations and the cleared `out` may come from the kernel just before
    griddep_launch_dependents();   // a kernel behind this launch may be scheduled; it waits for our completion
    // What the rest of the prologue depends on is requested together, before the set-up: the schedule's length, this block's
    // expert and the sorted ids this thread will need (a gather thread those of its rows, an epilogue thread its token's).
    constexpr int GROUPS = kTmRows / 4, MAXG = (GROUPS + kTmGatherWarps - 1) / kTmGatherWarps;
    // (from lane 0: what depends on it is uniform in the warp for the compiler, too)
    const int warp = __shfl_sync(0xFFFFFFFFu, static_cast<int>(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int gather_warp = warp == W_G0 ? 0 : warp - W_G1 + 1;      // of the gather role only
    int pid_pre[MAXG];
    int expert;
    {
        const int npad_raw = ld_global_s32(p.num_tokens_post_padded);
        expert = ld_global_s32(p.expert_ids + mblock);
        const bool gather_role = warp == W_G0 || warp >= W_G1;
#pragma unroll
        for (int i = 0; i < MAXG; ++i) {
            const int grp = gather_warp + kTmGatherWarps * i;
            const int row = gather_role ? 4 * grp + (lane >> 3) : static_cast<int>(threadIdx.x & (kTmRows - 1));
            const int idx = mblock * p.block_m + row;
            pid_pre[i] = -1;
            if ((gather_role || (i == 0 && warp < W_TMA)) && row < p.block_m && idx < p.sorted_num)
                pid_pre[i] = ld_global_s32(p.sorted_token_ids + idx);
        }
        if (mblock * p.block_m >= min(npad_raw, p.sorted_num)) return;
        if (expert < 0 || expert >= p.E) return;
    }

    const int KC = p.K >> 7;
    const int UPI = SPC * KC;
    const int ND = SPC == 1 ? (KC + 1) >> 1 : SPC / 2 * KC;      // (SPC = 4: two iterations per hidden tile)
    const int NIT = UPI + ND;
    const int S = p.stages;

    // The operand tiles need 1024-byte alignment (128-byte swizzle atoms).  The dynamic shared memory
    // window is declared with that alignment; should a toolchain ever place it differently, the CTA
    // reports it and returns instead of computing on mis-swizzled tiles.
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw;
    if (smem_u32(smem_raw) & 1023u) {
        if (threadIdx.x == 0) atomicCAS(&p.status->code, ST_OK, ST_SMEM_MISALIGNED);
        return;
    }
    const SmemPlanTm L = smem_plan_tm(S, KC, SPC);
    uint8_t* hq = smem + L.hq;                                        // fp8 intermediate [SPC][128][128], swizzled
    float* swg = reinterpret_cast<float*>(smem + L.swg);
    float* swu = reinterpret_cast<float*>(smem + L.swu);
    float* sw2 = reinterpret_cast<float*>(smem + L.sw2);
    uint32_t* amaxx = reinterpret_cast<uint32_t*>(smem + L.amaxx);    // one or two sets of [2][128] per-thread |h| maxima of each column half
    float* xs = reinterpret_cast<float*>(smem + L.xs);                // [KC][128] token scales (0 for padding rows)
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + L.bars);
    uint64_t* empty = full + S;
    uint64_t* acc_full = empty + S;
    uint64_t* acc_empty = acc_full + 2;
    uint64_t* h_ready = acc_empty + 2;
    uint64_t* xchg = h_ready + 1;
    uint64_t* down_full = xchg + 2;      // (four slices) [warpgroup][buffer]: accumulators of a warpgroup's hidden tiles complete
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + L.misc);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + L.misc + 4);

    if (threadIdx.x == W_TMA * 32) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&full[i], 1 + GATHER_THREADS);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 2; ++i) {
            mbar_init(&acc_full[i], 1);
            mbar_init(&acc_empty[i], 8);
        }
        mbar_init(h_ready, 1);
        mbar_init(&xchg[0], 8);
        if (SPC == 4)
            for (int i = 0; i < 4; ++i) mbar_init(&down_full[i], 1);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == W_MMA0) {
        tmem_alloc(tmem_slot, TMEM_COLS);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;

    if (warp >= W_TMA) {
    // ====================================================================== control + gather warpgroups
    setmaxnreg_dec<40>();
    if (warp == W_MMA0 + 1) {
        // (no role: one warp issues a chunk's four or eight UMMAs faster than they run; setmaxnreg needs whole warpgroups)
    } else if (warp == W_MMA0) {
        // ------------------------------------------------------------------ UMMA issuer
        {
            constexpr uint32_t idesc256 = umma_idesc_e4m3(128, 256);
            constexpr uint32_t idesc128 = umma_idesc_e4m3(128, 128);
            const uint32_t st0 = smem_u32(smem);
            const uint32_t dstep = L.stage_bytes >> 4;
            const uint64_t w_0 = umma_desc_sw128(st0);                      // 256 weight rows of the slot (N operand)
            const uint64_t w_1 = umma_desc_sw128(st0 + kTileBytes);         // its second 128 rows
            const uint64_t x_0 = umma_desc_sw128(st0 + 2 * kTileBytes);     // gathered token rows (M operand)
            const uint64_t h0 = umma_desc_sw128(smem_u32(hq));
            const uint64_t h1 = umma_desc_sw128(smem_u32(hq + (SPC > 1 ? 1 : 0) * kTmRows * 128));
            int s = 0;
            uint32_t ph = 0;
            bool h_waited = false;
            for (int it = 0; it < NIT; ++it) {
                const int b = it & 1;
                const uint32_t aph = (it >> 1) & 1;
                const uint32_t d = tmem_base + b * 256;
                const bool up = it < UPI;
                if (!up && !h_waited) {
                    if (!mbar_wait_warp(h_ready, 0, abort_flag, p.status, 20, it)) break;
                    h_waited = true;
                }
                if (!mbar_wait_warp(&acc_empty[b], aph ^ 1, abort_flag, p.status, 21, it)) break;
                if (!mbar_wait_warp(&full[s], ph, abort_flag, p.status, 22, it)) break;
                tc_fence_after();
                const uint64_t off = static_cast<uint64_t>(s * dstep);
                if (elect_one()) {
                    fence_proxy_async_smem();  // token rows were written by cp.async, the UMMA reads them through the async proxy
                    if (up) {
                        umma_f8_chunk1(d, x_0 + off, w_0 + off, idesc256);           // D[token, 256 interleaved w rows]
                    } else if (SPC == 1) {
                        umma_f8_chunk1(d, h0, w_0 + off, idesc256);                  // D[token, 2 x 128 hidden rows]
                    } else {
                        const uint64_t two = SPC == 4 && b ? 2 * kTmRows * 128 / 16 : 0;      // (odd iterations: slices 2 and 3)
                        umma_f8_chunk2(d, d + 128, h0 + two, h1 + two, w_0 + off, w_1 + off, idesc128);   // per-slice partial sums
                    }
                    umma_commit(SPC == 4 && !up ? &down_full[((it - UPI) & 2) + b] : &acc_full[b]);
                    umma_commit(&empty[s]);    // the ring slot is free once these MMAs have read it
                }
                __syncwarp();
                if (++s == S) { s = 0; ph ^= 1; }
            }
        }
    } else if (warp == W_TMA) {
        // ------------------------------------------------------------------ weight TMA (one thread)
        if (lane == 0) {
            prefetch_tmap(&tm_w);
            prefetch_tmap(&tm_w2);
            int s = 0;
            uint32_t ph = 0;
            int kc = 0, sl = 0;
            for (int it = 0; it < NIT; ++it) {
                if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, 30, it)) break;
                uint8_t* st = smem + s * L.stage_bytes;
                mbar_arrive_expect_tx(&full[s], 2 * kTileBytes);
                if (it < UPI) {
                    tma_load_3d(st, &tm_w, &full[s], kc * 128, (slice0 + sl) * 256, expert);
                    if (++kc == KC) { kc = 0; ++sl; }
                } else {
                    // down phase: no token rows any more, so this thread also stands in for the gather threads
                    const int jt = it - UPI;
                    if (SPC == 1) {
                        tma_load_3d(st, &tm_w2, &full[s], slice0 * 128, (2 * jt) * 128, expert);
                        tma_load_3d(st + kTileBytes, &tm_w2, &full[s], slice0 * 128, (2 * jt + 1) * 128, expert);
                    } else {
                        const int tile = SPC == 4 ? jt >> 1 : jt, first = slice0 + (SPC == 4 ? 2 * (jt & 1) : 0);
                        tma_load_3d(st, &tm_w2, &full[s], first * 128, tile * 128, expert);
                        tma_load_3d(st + kTileBytes, &tm_w2, &full[s], (first + 1) * 128, tile * 128, expert);
                    }
                    mbar_arrive_n(&full[s], GATHER_THREADS);
                }
                if (++s == S) { s = 0; ph ^= 1; }
            }
        }
    } else {
        // ------------------------------------------------------------------ token-row gather (5 warps)
        // Row group j (4 token rows x 128 B, one cp.async of the warp) belongs to gather warp j % 5: 7 groups for
        // the first two warps, 6 for the others.  Lane l copies 16-byte piece l & 7 of row 4j + (l >> 3).
        const int gw = gather_warp;
        const int ch = lane & 7;
        uint32_t src16[MAXG];
        uint32_t dst[MAXG];
#pragma unroll
        for (int i = 0; i < MAXG; ++i) {
            const int grp = gw + kTmGatherWarps * i;
            const int row = 4 * grp + (lane >> 3);
            const int pid = pid_pre[i];            // requested at kernel entry; -1 for rows past the block
            src16[i] = 0xFFFFFFFFu;
            dst[i] = 0xFFFFFFFFu;                  // no such group for this warp
            if (grp < GROUPS) {
                dst[i] = row * 128 + ((ch ^ (row & 7)) << 4);
                if (pid >= 0 && pid < p.M * p.top_k)
                    src16[i] = static_cast<uint32_t>((static_cast<size_t>(pid / p.top_k) * p.K) >> 4);
            }
        }
        int s = 0;
        uint32_t ph = 0;
        int kc = 0;
        for (int it = 0; it < UPI; ++it) {
            if (!mbar_wait(&empty[s], ph ^ 1, abort_flag, p.status, 31, it)) break;
            const uint32_t base = smem_u32(smem + s * L.stage_bytes + 2 * kTileBytes);
            const uint8_t* col = p.x + kc * 128 + ch * 16;
#pragma unroll
            for (int i = 0; i < MAXG; ++i) {
                if (dst[i] != 0xFFFFFFFFu) {
                    const bool v = src16[i] != 0xFFFFFFFFu;
                    const uint8_t* src = v ? col + (static_cast<size_t>(src16[i]) << 4) : p.x;
                    cp_async_16(base + dst[i], src, v ? 16u : 0u);
                }
            }
            cp_async_mbar_arrive_noinc(&full[s]);      // arrives when this thread's copies have landed
            if (++s == S) { s = 0; ph ^= 1; }
            if (++kc == KC) kc = 0;
        }
        cp_async_wait_all();                        // nothing of this thread may still be in flight at exit
    }
    } else {
        // ====================================================================== epilogue: thread = token
        setmaxnreg_inc<216>();
        const int q = warp & 3;              // TMEM lane quarter
        const int hh = warp >> 2;            // column half handled by this warpgroup
        const int t = q * 32 + lane;         // token slot of the block = TMEM lane
        const int etid = threadIdx.x;
        int row = p.M;
        float tw = 0.f;
        {
            const int pid = pid_pre[0];
            if (pid >= 0 && pid < p.M * p.top_k) {
                row = pid / p.top_k;             // reference :757
                tw = p.topk_weights[pid];        // reference :761
            }
        }
        const bool valid = row < p.M;
        const bool warp_valid = __any_sync(0xFFFFFFFFu, valid);
        {
            const int nsr = p.N >> 7;
            const int isl = p.N >> 8;
            for (int i = etid; i < SPC * KC; i += EPI_THREADS) {
                const int sl = i / KC, c = i - sl * KC;
                const float* ws = p.w_scale + (static_cast<size_t>(expert) * nsr + 2 * (slice0 + sl)) * KC;
                swg[i] = ws[c];
                swu[i] = ws[KC + c];
                sw2[i] = p.w2_scale[(static_cast<size_t>(expert) * KC + c) * isl + slice0 + sl];
            }
        }
        // Token scales go to shared memory once (each warpgroup fetches one half of the K chunks of its tokens): the
        // chunk loop then holds no global load, whose latency a releasing hand-off would have to wait out.
        {
            const float* xs_row = p.x_scale + static_cast<size_t>(valid ? row : 0) * KC;
            stage_token_scales<kTmRows, 8>(xs + t, xs_row, valid, hh, 2, p.xs_vec4 ? KC >> 2 : KC, p.xs_vec4);
        }
        named_bar_sync(1, EPI_THREADS);

        // Accumulators of this token: 8 groups of (8 gate, 8 up) columns = 64 intermediate columns, as packed pairs.  In a row
        // of calls this kernel runs at the power limit, where an instruction saved counts even if its unit was not busy.  Packed
        // FMAs, the rows of the down phase's reductions in registers instead of a shuffle and a 64-bit multiplication for each,
        // no vote per chunk and one issuing warp instead of two that took turns: DeepSeek-V3 TP8 shard, M = 4096 531 -> 507 us,
        // M = 8192 (Zipf) 885 -> 854, unsharded M = 4096 3915 -> 3744, Qwen3-Next shard M = 4096 230 -> 220 (the rows alone
        // are two thirds of it).  For the same reason token rows of padding are zeroed: left as they are, M = 4096 is 3 % slower.
        f32x2 acc[64];
#pragma unroll
        for (int j = 0; j < 64; ++j) acc[j] = 0;
        float fac[SPC];                      // s_h * topk weight * scaling per slice (reference :997-1003)

        const uint32_t tlane = tmem_base + (static_cast<uint32_t>(q * 32) << 16);
        // A wait that runs out does not leave the loops of the up phase: with the abort flag raised every later wait returns after
        // one batch of polls (0.3 ms, so 70 ms for four slices of 56 chunks), and what was computed meanwhile is added nowhere
        // (see in front of the down phase).
        bool ok = true;
        uint32_t xph = 0;
        // ---- up-projection: promote each K chunk with its scales (reference :915-933).  The chunk loop is kept
        // small and contiguous (the slice-end code follows it instead of sitting inside it).
        for (int sl = 0, it = 0; sl < SPC; ++sl) {
#pragma unroll 1
        for (int kc = 0; kc < KC; ++kc, ++it) {
            const int b = it & 1;
            const uint32_t aph = (it >> 1) & 1;
            const float sx = xs[kc * kTmRows + t];
            const float fg = sx * swg[sl * KC + kc], fu = sx * swu[sl * KC + kc];
            if (!mbar_wait(&acc_full[b], aph, abort_flag, p.status, 40, it)) ok = false;
            tc_fence_after();
            // 64 columns are requested before the first is used (every wait lengthens the chain issue -> read-back -> hand-back
            // around the two accumulator buffers): against waits after every 32 columns, blocks of 128 at the DeepSeek-V3 TP8
            // shard, M = 4096 460 -> 449 us, M = 8192 (Zipf) 769 -> 754 us, unsharded M = 4096 3540 -> 3212 us.  TMEM loads do
            // not wait for UMMAs in flight: 16 columns and their FMAs take 40 cycles either way.
            const uint32_t tb = tlane + b * 256 + hh * 128;
            uint32_t v[4][16];
            const f32x2 fg2 = pack_f32x2(fg, fg), fu2 = pack_f32x2(fu, fu);
            auto request = [&](int c0) {
#pragma unroll
                for (int c = 0; c < 4; ++c) tmem_ld16(tb + c0 + 16 * c, v[c]);
                tmem_ld_wait();
            };
            auto promote = [&](int c0) {
#pragma unroll
                for (int c = 0; c < 4; ++c)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        const int j = (c0 + 16 * c) / 2 + e;
                        acc[j] = fma_f32x2(pack_u32x2(v[c][2 * e], v[c][2 * e + 1]), fg2, acc[j]);
                        acc[j + 4] = fma_f32x2(pack_u32x2(v[c][8 + 2 * e], v[c][9 + 2 * e]), fu2, acc[j + 4]);
                    }
            };
            if (warp_valid) {
                request(0);
                promote(0);
                request(64);
                promote(64);
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive_relaxed(&acc_empty[b]);
        }
            {
                // ---- end of a slice: SwiGLU, amax over the slice's 128 columns (64 here + 64 in the partner
                //      warpgroup's thread of the same token), fp8 re-quantisation (reference :936-1005)
                float amax = 0.f;
#pragma unroll
                for (int g8 = 0; g8 < 8; ++g8) {
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        float gv[2], uv[2], h[2];
                        unpack_f32x2(acc[8 * g8 + e], gv[0], gv[1]);
                        unpack_f32x2(acc[8 * g8 + 4 + e], uv[0], uv[1]);
#pragma unroll
                        for (int i = 0; i < 2; ++i) {
                            const float g = bf16_round(gv[i]), u = bf16_round(uv[i]);
                            h[i] = bf16_round(__fdividef(g, 1.0f + __expf(-g)) * u);
                            amax = fmaxf(amax, fabsf(h[i]));
                        }
                        acc[8 * g8 + e] = pack_f32x2(h[0], h[1]);
                    }
                }
                uint32_t* am = amaxx + (two_sets_of_maxima(SPC, KC) ? (sl & 1) * 2 * kTmRows : 0);
                am[hh * kTmRows + t] = __float_as_uint(amax);
                __syncwarp();
                if (lane == 0) mbar_arrive(&xchg[0]);
                if (!mbar_wait(&xchg[0], xph, abort_flag, p.status, 42, sl)) ok = false;
                xph ^= 1;
                amax = fmaxf(amax, __uint_as_float(am[(hh ^ 1) * kTmRows + t]));
                const float s_h = fmaxf(amax, 1e-10f) * (1.0f / 448.0f);
                uint8_t* hrow = hq + sl * kTmRows * 128 + t * 128;
#pragma unroll
                for (int i = 0; i < 4; ++i) {             // 16 intermediate columns = 16 bytes per store
                    uint32_t w4[4];
#pragma unroll
                    for (int k2 = 0; k2 < 4; ++k2) {
                        const int base = 8 * (2 * i + (k2 >> 1)) + 2 * (k2 & 1);
                        float qv[4];
                        unpack_f32x2(acc[base], qv[0], qv[1]);
                        unpack_f32x2(acc[base + 1], qv[2], qv[3]);
#pragma unroll
                        for (int e = 0; e < 4; ++e) qv[e] = fminf(fmaxf(__fdividef(qv[e], s_h), -448.0f), 448.0f);
                        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(qv[0], qv[1]), __NV_SATFINITE, __NV_E4M3);
                        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(qv[2], qv[3]), __NV_SATFINITE, __NV_E4M3);
                        w4[k2] = lo | (hi << 16);
                    }
                    const int chunk = (hh * 4 + i) ^ (t & 7);
                    *reinterpret_cast<uint4*>(hrow + chunk * 16) = make_uint4(w4[0], w4[1], w4[2], w4[3]);
                }
                // The loop over slices is not unrolled, and an index that varies puts the array on the stack: two are told apart
                // instead (DeepSeek-V3 TP8 shard, M = 4096 515 -> 513 us, M = 8192 (Zipf) 856 -> 847).  Four stay there, one
                // load each per hidden tile: kept in registers they make 176 bytes of spills out of 32.
                const float f = s_h * tw * p.scaling;
                if constexpr (SPC == 2) {
                    if (sl == 0) fac[0] = f;
                    else fac[SPC - 1] = f;
                } else {
                    fac[sl] = f;
                }
#pragma unroll
                for (int j = 0; j < 64; ++j) acc[j] = 0;
                fence_proxy_async_smem();
            }
        }
        named_bar_sync(1, EPI_THREADS);
        if (etid == 0) mbar_arrive(h_ready);

        // ---- down-projection epilogue (reference :1052-1094).  A thread holds 64 consecutive hidden columns
        // of its own token, but 32 lanes reducing into 32 different rows would make every reduction
        // instruction 32 separate half-sector requests.  So each warp turns its 32 x 128-byte block around in
        // a private staging tile: afterwards one instruction covers four token rows x 128 contiguous bytes
        // (whole lines), which is what the reduction path of the memory system handles best.  (Handing each
        // row to the bulk-copy engine instead - cp.reduce.async.bulk, 128 B per lane - measured 14 % slower.)
        // staging tiles: the token-row part of the ring slots is idle in this phase (three tiles per slot);
        // a ring of fewer than three slots has room for a dedicated area
        uint8_t* stg = L.stage_out != kStgAliased ? smem + L.stage_out + warp * kStgWarpBytes
                                                  : smem + (warp / 3) * L.stage_bytes + 2 * kTileBytes + (warp % 3) * kStgWarpBytes;
        // The flag has been raised in front of the barrier above by whoever gave up: no warp reduces anything then.
        ok = __all_sync(0xFFFFFFFFu, ok && !*abort_flag);
        // The rows that a lane reduces (token 4i + lane / 8 of its warp) stay the same for the whole phase.
        const int my_row = valid ? row : p.M;
        uint32_t red_row[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) red_row[i] = static_cast<uint32_t>(__shfl_sync(0xFFFFFFFFu, my_row, 4 * i + (lane >> 3)));
        auto pack2 = [](float lo, float hi) {
            const __nv_bfloat162 h2 = __floats2bfloat162_rn(lo, hi);
            return *reinterpret_cast<const uint32_t*>(&h2);
        };
        auto reduce_64 = [&](const uint32_t (&w)[32], int col0) {
#pragma unroll
            for (int g = 0; g < 8; ++g)
                *reinterpret_cast<uint4*>(stg + lane * kStgPitch + g * 16) = make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
            __syncwarp();
            uint4 vv[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) vv[i] = *reinterpret_cast<const uint4*>(stg + (4 * i + (lane >> 3)) * kStgPitch + (lane & 7) * 16);
            __nv_bfloat16* base = p.out + col0 + (lane & 7) * 8;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const bool live = red_row[i] < static_cast<uint32_t>(p.M);
                red_add_v4_bf16x2_raw_if(base + static_cast<size_t>(live ? red_row[i] : 0) * p.K, vv[i], live);
            }
            __syncwarp();
        };
        // The two warpgroups take alternate iterations: while one is held up issuing its reductions (an SM
        // passes only about 22 bytes of them per cycle) the other reads its accumulator and converts, so the
        // reduction path stays busy.  A warpgroup therefore handles all columns of its iteration, in parts of
        // 64 hidden columns: SPC = 2 -> 2 parts of hidden tile jt (columns [0,128) of the buffer are slice 0's
        // partial sums, [128,256) slice 1's); SPC = 1 -> 4 parts covering hidden tiles 2jt and 2jt+1.
        if constexpr (SPC == 4) {
            // A warpgroup takes both iterations of its hidden tile and adds the four slices' partial sums up in registers, so
            // that a (token, hidden column) is reduced into `out` once per four slices.  Both buffers serve both warpgroups in
            // turn, and a parity wait must not be two phases off its barrier: each warpgroup has barriers of its own.
            constexpr int COLS = 32;             // columns of both accumulators per wait (16: 3 % slower, 64 do not fit)
            for (int jt = hh; jt < KC && ok; jt += 2) {
                f32x2 y[64];
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const int it = UPI + 2 * jt + half;              // UPI is even: buffer `half`
                    ok = mbar_wait_warp(&down_full[2 * hh + half], (jt >> 1) & 1, abort_flag, p.status, 41, it);
                    if (!ok) break;
                    tc_fence_after();
                    if (warp_valid) {
                        const float fa = sw2[(2 * half) * KC + jt] * fac[2 * half], fb = sw2[(2 * half + 1) * KC + jt] * fac[2 * half + 1];
                        const f32x2 fa2 = pack_f32x2(fa, fa), fb2 = pack_f32x2(fb, fb);
#pragma unroll
                        for (int c0 = 0; c0 < 128; c0 += COLS) {
                            uint32_t va[COLS], vb[COLS];
                            const uint32_t tb = tlane + half * 256 + c0;
#pragma unroll
                            for (int c = 0; c < COLS; c += 16) {
                                tmem_ld16(tb + c, *reinterpret_cast<uint32_t(*)[16]>(&va[c]));
                                tmem_ld16(tb + 128 + c, *reinterpret_cast<uint32_t(*)[16]>(&vb[c]));
                            }
                            tmem_ld_wait();
#pragma unroll
                            for (int e = 0; e < COLS / 2; ++e) {
                                const f32x2 a = pack_u32x2(va[2 * e], va[2 * e + 1]), v = pack_u32x2(vb[2 * e], vb[2 * e + 1]);
                                f32x2& s = y[c0 / 2 + e];
                                s = half == 0 ? fma_f32x2(a, fa2, mul_f32x2(v, fb2)) : fma_f32x2(a, fa2, fma_f32x2(v, fb2, s));
                            }
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_relaxed_n(&acc_empty[half], 2);
                }
                if (ok && warp_valid) {
#pragma unroll
                    for (int part = 0; part < 2; ++part) {
                        uint32_t w[32];
#pragma unroll
                        for (int e = 0; e < 32; ++e) {
                            float lo, hi;
                            unpack_f32x2(y[32 * part + e], lo, hi);
                            w[e] = pack2(lo, hi);
                        }
                        reduce_64(w, jt * 128 + part * 64);
                    }
                }
            }
        } else {
        constexpr int PARTS = SPC == 1 ? 4 : 2;
        for (int jt = hh; jt < ND && ok; jt += 2) {
            const int it = UPI + jt;
            const int b = it & 1;
            const uint32_t aph = (it >> 1) & 1;
            ok = mbar_wait_warp(&acc_full[b], aph, abort_flag, p.status, 41, it);
            if (!ok) break;
            tc_fence_after();
            uint32_t va[64], vb[SPC == 2 ? 64 : 1];
            auto request = [&](int part) {
                const uint32_t tb = tlane + b * 256 + part * 64;
#pragma unroll
                for (int c0 = 0; c0 < 64; c0 += 16) {
                    tmem_ld16(tb + c0, *reinterpret_cast<uint32_t(*)[16]>(&va[c0]));
                    if constexpr (SPC == 2) tmem_ld16(tb + 128 + c0, *reinterpret_cast<uint32_t(*)[16]>(&vb[c0]));
                }
            };
#pragma unroll
            for (int part = 0; part < PARTS; ++part) {
                const int tile = SPC == 1 ? 2 * jt + (part >> 1) : jt;
                uint32_t w[32];
                if (warp_valid) {
                    request(part);
                    tmem_ld_wait();
                    if constexpr (SPC == 1) {
                        const float f = sw2[min(tile, KC - 1)] * fac[0];
                        const f32x2 f2 = pack_f32x2(f, f);
#pragma unroll
                        for (int e = 0; e < 32; ++e) {
                            float lo, hi;
                            unpack_f32x2(mul_f32x2(pack_u32x2(va[2 * e], va[2 * e + 1]), f2), lo, hi);
                            w[e] = pack2(lo, hi);
                        }
                    } else {
                        const float fa = sw2[jt] * fac[0], fb = sw2[KC + jt] * fac[SPC - 1];
                        const f32x2 fa2 = pack_f32x2(fa, fa), fb2 = pack_f32x2(fb, fb);
#pragma unroll
                        for (int e = 0; e < 32; ++e) {
                            float lo, hi;
                            unpack_f32x2(fma_f32x2(pack_u32x2(va[2 * e], va[2 * e + 1]), fa2,
                                                   mul_f32x2(pack_u32x2(vb[2 * e], vb[2 * e + 1]), fb2)), lo, hi);
                            w[e] = pack2(lo, hi);
                        }
                    }
                }
                if (part == PARTS - 1) {
                    // the buffer has been read completely: hand it back before the last reductions are issued
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive_relaxed_n(&acc_empty[b], 2);   // 4 warps stand in for the barrier's 8
                }
                if (warp_valid && tile < KC) reduce_64(w, SPC == 1 ? tile * 128 + (part & 1) * 64 : jt * 128 + part * 64);
            }
        }
        }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == W_MMA0) {
        tc_fence_after();
        tmem_dealloc(tmem_base, TMEM_COLS);
    }
}

}  // namespace amoe
