// Whole-sequence summaries of the tensor-core path (included by ssd_tc.cuh): what one contiguous piece of a
// sequence contributes to the state after it (forward) or to the gradient of the state before it (reverse),
// for a zero state on the other side.  These are the quantities the sequence-parallel schedule exchanges.
//
//   forward  F[n][p] = sum_j  B[j,n] * x[j,p] * dt_j * exp(sum of the log-decays AFTER position j)
//   reverse  D[n][p] = sum_i  C[i,n] * dy[i,p] *        exp(sum of the log-decays up to and including i)
//
// Neither is a recurrence: every tile adds one product to the same accumulator, so the kernel is a plain stream.
// One CTA per (batch entry, NH heads of a group): TMA loads (stages of the group's B or C panels + the x or dy panel of each
// head), eight warps per head scale the rows of their 64-wide panel in place, one lane of another warp issues eight tcgen05.mma per tile
// (N = 64 NH: the heads' panels side by side) that all accumulate into one TMEM accumulator, read once at the end.  With
// NH = 2 (heads per group even) the group's panels, two thirds of what a one-head CTA pulls in per tile, are fetched once
// for two heads; what one SM can pull in is what bounds this kernel.  The weights are <= 1 (dt aside), so nothing
// overflows; the forward walks the tiles from the last to the first (the decay after a tile is a running sum that starts
// at 0 where the weights are largest), the reverse from the first to the last.
//
// A given seed (initial state, or final-state gradient) enters as  exp(total log-decay) * seed.  blockIdx.z =
// (piece of `pt` tiles, part of `ps` tiles), each with its own out and logdecay (blockIdx.z, b, h, ...): the pieces of one
// sequence that the walks run side by side.
// mbarriers, per stage s (phase = turn of the stages): bar_ld[s] TMA bytes landed; bar_m[s] the products of the stage completed (the stage may be
// reloaded; the last one also releases the accumulator to the row warps).  Hardware barrier kSumBarU + s: rows scaled (row warps arrive, the
// products' warp waits; one per stage, since the row warps may be as many tiles ahead of the products as there are stages).
// Products and copies are issued by different warps, so that a stage is asked for again when its products are done and not a tile
// later: 64 heads of 131,072 positions, half of them forward 160 -> 130 us, three quarters of them in reverse 289 -> 211.
#pragma once

namespace ssd {
namespace tc {

template <int NH>
struct SumCfg {
    static constexpr int STAGES = NH == 1 ? 4 : 3;
    static constexpr uint32_t STAGE_BYTES = (2 + NH) * PANEL;  // V panels 0,1 | U of each head
    static constexpr size_t SMEM = (size_t)STAGES * STAGE_BYTES + 1024;
    static constexpr int THREADS = 256 * NH + 64;
};

struct SummaryParams {
    CUtensorMap mU;        // x (forward) or dy (reverse): 2D [b*T][h*64]
    CUtensorMap mV;        // B (forward) or C (reverse):  2D [b*T][g*128]
    const float* tcum;     // (b,h,T) tile-cumulative log2-decay
    const float* dtT;      // (b,h,T) dt (forward) or null
    const float* seed;     // (b,h,p,n) fp32 or null
    float* out;            // (z,b,h,p,n) fp32
    float* logdecay;       // (z,b,h) total log-decay of the part in natural-log units, or null
    int* status;
    int zero_status;      // see WalkParams
    int Tp, h, hpg, nt;   // Tp = nt * 128: stride of the per-position arrays
    int p, n;
    int pt, ps, parts;    // tiles of a piece and of a part, parts per piece
    int z0;               // piece of the blocks with blockIdx.z = 0
};

constexpr int kSumBarU = 1;  // one per stage
template <bool REV, int NH>
__global__ void __launch_bounds__(SumCfg<NH>::THREADS, 1) summary_kernel(const __grid_constant__ SummaryParams P) {
    dep_wait();
    if (P.zero_status) clear_status(P.status);
    using Cfg = SumCfg<NH>;
    constexpr int NS = Cfg::STAGES;
    constexpr int MMAW = 8 * NH, TMAW = MMAW + 1;  // control warps
    constexpr int BAR = 256 * NH + 32;             // row warps and the products' warp
    extern __shared__ uint8_t smem_raw[];
    uint8_t* sStage = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    __shared__ uint64_t bar_ld[4], bar_m[4];
    __shared__ uint32_t tmem_slot;
    __shared__ int alive;
    __shared__ int4 taken;  // see until_taken: .x kSumBarU

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hh0 = blockIdx.x * NH, bb = blockIdx.y;
    const int gg = hh0 / P.hpg;
    const int part = (int)blockIdx.z % P.parts, piece = P.z0 + (int)blockIdx.z / P.parts;
    const int k0 = piece * P.pt + part * P.ps, nt = min(min(P.ps, P.pt - part * P.ps), P.nt - k0);  // at least one (see Pieces)
    // forward: tiles nt-1 .. 0 of the part; reverse: 0 .. nt-1
    auto tile_of = [&](int it) { return k0 + (REV ? it : nt - 1 - it); };

    if (tid == 0) {
        alive = 1;
        taken = make_int4(NS, kTakenAll, kTakenAll, kTakenAll);
        for (int s = 0; s < NS; ++s) {
            mbar_init(&bar_ld[s], 1);
            mbar_init(&bar_m[s], 1);
        }
        mbar_fence_init();
    }
    if (warp == MMAW) {
        tmem_alloc(&tmem_slot, 64 * NH);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = tmem_slot;  // accumulator row = n, columns [64 hs, 64 hs + 64) = p of head hs

    if (warp == MMAW) {
        const uint32_t stMN = desc_lo(smem_u32(sStage), PANEL);
        int s = 0;
#pragma unroll 1
        for (int it = 0; it < nt; ++it) {
            __syncwarp();
            named_bar_sync(kSumBarU + s, BAR);
            if (lane == 0) {
                tc_fence_after();
                uint32_t v = stMN + (uint32_t)s * (Cfg::STAGE_BYTES >> 4);
                asm volatile("" : "+r"(v));
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)  // acc[n][p of every head] += V^T Uw : both MN-major, K = position
                    mma_ss_lo(tm, v + kk * 128, v + (2 * PANEL >> 4) + kk * 128, NH == 2 ? kIdescMM128 : kIdescMM, it > 0 || kk > 0);
                mma_commit(&bar_m[s]);
                set_taken(&taken.x, it + 1 + NS);
            }
            if (++s == NS) s = 0;
        }
    } else if (warp == TMAW) {
        if (lane == 0) {
            prefetch_tmap(&P.mU);
            prefetch_tmap(&P.mV);
            int s = 0;
            uint32_t ph = 1;  // (the first turn waits for nothing)
#pragma unroll 1
            for (int it = 0; it < nt; ++it) {
                uint8_t* st = sStage + (size_t)s * Cfg::STAGE_BYTES;
                const int pos = tile_of(it) * LT;
                mbar_wait(&bar_m[s], ph, &alive);  // the products of the stage's tile before are done
                mbar_expect_tx(&bar_ld[s], Cfg::STAGE_BYTES);
#pragma unroll
                for (int hs = 0; hs < NH; ++hs) tma_load_4d(st + (2 + hs) * PANEL, &P.mU, &bar_ld[s], 0, hh0 + hs, pos, bb);
                tma_load_4d(st, &P.mV, &bar_ld[s], 0, gg, pos, bb);
                tma_load_4d(st + PANEL, &P.mV, &bar_ld[s], 64, gg, pos, bb);
                if (++s == NS) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
        __syncwarp();
    } else {
        const int hs = tid >> 8;  // which of the CTA's heads
        const int hh = hh0 + hs;
        const size_t bh = (size_t)bb * P.h + hh;
        const int ht = tid & 255, row = ht & 127, hf = ht >> 7;  // scaling: position `row`, columns [32 hf, 32 hf + 32) of the panel
        const float* tcum = P.tcum + bh * P.Tp;
        const float* dtT = (!REV && P.dtT) ? P.dtT + bh * P.Tp : nullptr;
        float run = 0.f;  // forward: log2-decay of the tiles after this one; reverse: of the tiles before it
        const size_t o0 = (size_t)tile_of(0) * LT;
        float c_n = tcum[o0 + row];
        float S_n = tcum[o0 + LT - 1];
        float dt_n = dtT ? dtT[o0 + row] : 1.f;
        int s = 0;
        uint32_t ph = 0;
#pragma unroll 1
        for (int it = 0; it < nt; ++it) {
            const float c_i = c_n, Sk = S_n, dtv = dt_n;
            if (it + 1 < nt) {
                const size_t o = (size_t)tile_of(it + 1) * LT;
                c_n = tcum[o + row];
                S_n = tcum[o + LT - 1];
                dt_n = dtT ? dtT[o + row] : 1.f;
            }
            const float w = REV ? exp2f(run + c_i) : dtv * exp2f(run + (Sk - c_i));
            run += Sk;
            mbar_wait(&bar_ld[s], ph, &alive);
            const int late = gave_up(&alive);
            uint8_t* sU = sStage + (size_t)s * Cfg::STAGE_BYTES + (2 + hs) * PANEL;
            const __nv_bfloat162 w2 = __float2bfloat162_rn(w);
#pragma unroll
            for (int ch = 0; ch < 4; ++ch) {
                uint4* p = reinterpret_cast<uint4*>(sU + sw128(row, hf * 4 + ch));
                uint4 v = *p;
                uint32_t* u = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&u[q]), w2);
                    u[q] = *reinterpret_cast<uint32_t*>(&r);
                }
                *p = v;
            }
            fence_async_smem();
            until_taken(late, &taken, it);
            hand_over(kSumBarU + s, BAR);
            if (++s == NS) {
                s = 0;
                ph ^= 1;
            }
        }
        // `run` is now the total log2-decay of the piece
        const int last = nt - 1;
        uint32_t r[32];
        mbar_wait(&bar_m[last % NS], (last / NS) & 1, &alive);
        tc_fence_after();
        tmem_ld32(tm + lane_base(warp) + hs * 64 + hf * 32, r);
        tmem_ld_wait();
        const float dec = exp2f(run);
        float v[32];  // accumulator row = n, columns = p
        load_state_row(P.seed, bh, P.p, P.n, row, hf * 32, v);
#pragma unroll
        for (int q = 0; q < 32; ++q) v[q] = fmaf(dec, v[q], __uint_as_float(r[q]));
        const size_t zbh = (size_t)blockIdx.z * gridDim.y * P.h + bh;
        store_state_row(P.out, zbh, P.p, P.n, row, hf * 32, v);
        if (P.logdecay && ht == 0) P.logdecay[zbh] = run * 0.6931471805599453f;
    }
    tc_fence_before();
    __syncthreads();
    end_of_waits(&alive, P.status);
    if (warp == MMAW) tmem_dealloc(tm, 64 * NH);
}

}  // namespace tc
}  // namespace ssd
