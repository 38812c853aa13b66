// Reverse tile walk of the backward pass (included by ssd_tc.cuh after ssd_tc_walk.cuh).
//
// One CTA walks the 128-position tiles of NH heads of one group (same batch entry; or of a piece of the sequence, where
// a whole one per CTA would leave most of the chip idle) from the last tile to the first, with the gradient of each head's recurrent state Q (128 x 64, fp32) in the registers of that head's eight row
// warps.  Per tile k and head it
//   * stores Q as it leaves tile k (bf16, [n][p]) for the per-tile backward kernel,
//   * updates Q <- exp(S_k) Q + C^T (e . dY).
// It reads dY and C only (the terms of the decay gradient that need the forward state are evaluated by the tile
// kernel, which has that state on chip anyway).  Only the update is a recurrence, and it is a register update;
// everything else of tile k+1 (loads, the weighted rows, the MMA) is independent of tile k, so the kernel is a
// software pipeline: rings of C and dY, the accumulator double-buffered in TMEM, and the row warps prepare tile
// k+1 while the MMA of tile k runs.  The weighted rows e_i * dY[i,:] are written in place over the loaded dY panel.
// With NH = 2 the two heads share the C panels of a stage and one N = 128 product per tile
// (C^T [e dY_a | e dY_b]); their register chains are independent and run side by side on different warps.
// What bounds it: the row warps' steps of a tile where SMs are few (0.7 us with two blocks on the chip, 0.97 with 80, 1.22 for two heads), memory where all are busy: (16, 4096, 64 heads, 8 groups)
// 215 us, 5.0 TB/s (246 with copies and products on one lane, a block barrier on either side of every staged tile and log-decays asked for where they are
// used), one head per group 335 us, 6.4 TB/s (366).
//
// Threads: head hs = tid / 256 owns warps 8 hs .. 8 hs + 7 (thread = row, column half); one lane of the next warp issues the products, one of the
// last all copies.  The row warps hand over by hardware barriers and wait for mbarriers only (see the forward walk); a tile's log-decays are
// fetched two tiles before they are used.
// mbarriers:
//   bar_c[s], bar_u[s]   C / dY of the tile landed                    (rings of C_STAGES and U_STAGES tiles, phase = turn of the ring)
//   bar_m[b]   the MMA of the tile has completed, and the store of the state gradient of the tile before has read its panels, which the next one
//              overwrites (index tile parity b, phase (tile / 2) & 1; -> row warps, loads)
// Named barriers (row warps arrive, one control warp waits):
//   kRevBarU   weighted rows of the tile written, the accumulator of two tiles before read (-> products; two by tile parity: the row warps may
//              arrive once more before the products' warp has seen the last one)
//   kRevBarQ   state gradient leaving the tile staged                  (-> store)
#pragma once

namespace ssd {
namespace tc {

constexpr int kRevBarQ = 1, kRevBarU = 2 /* and 3 */;
template <int NH>
struct RevCfg {
    // dY is weighted a tile before its product, C wanted for the product only.  The state gradients are staged in two panels a head: with one
    // its store was part of every tile's chain (1.4 us a tile of two heads, 1.28 with two).
    static constexpr int C_STAGES = NH == 1 ? 3 : 2, U_STAGES = NH == 1 ? 4 : 3;
    static constexpr size_t SMEM = (size_t)(2 * C_STAGES + NH * U_STAGES + 2 * NH) * PANEL + 128;  // C (2 panels) | dY | sQ | barriers
    static constexpr int THREADS = 256 * NH + 64;
};

// CUT: in pieces.
template <int NH, bool CUT>
__global__ void __launch_bounds__(RevCfg<NH>::THREADS, 1) rev_walk_kernel(const __grid_constant__ WalkParams P) {
    dep_wait();
    if (P.zero_status) clear_status(P.status);
    using Cfg = RevCfg<NH>;
    // no static shared memory: the dynamic region starts at the CTA's shared-memory base
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int NC = Cfg::C_STAGES, NU = Cfg::U_STAGES;
    uint8_t* sC = smem_raw;                                // [NC][2 panels]
    uint8_t* sU0 = sC + (size_t)NC * 2 * PANEL;            // [NU][NH] dY, weighted in place
    uint8_t* sQ0 = sU0 + (size_t)NU * NH * PANEL;          // [2][NH] state gradient staged for its TMA store
    uint64_t* bars = reinterpret_cast<uint64_t*>(sQ0 + 2 * NH * PANEL);
    uint64_t* bar_c = bars;           // [NC]
    uint64_t* bar_u = bars + 3;       // [NU]
    uint64_t* bar_m = bars + 7;       // [2]
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 9);
    int& alive = *reinterpret_cast<int*>(bars + 10);
    int4& taken = *reinterpret_cast<int4*>(bars + 12);  // see until_taken: .x kRevBarU, .y kRevBarQ

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (smem_u32(smem_raw) & 1023u) {  // the swizzled panels need a 1024-byte aligned base: report instead of computing garbage
        if (tid == 0) atomicExch(P.status, 2);
        return;
    }
    constexpr int MMAW = 8 * NH, TMAW = MMAW + 1;  // control warps
    constexpr int BAR = 256 * NH + 32;             // row warps and one control warp
    const int hh0 = blockIdx.x * NH, bb = blockIdx.y;
    const int gg = hh0 / P.hpg;
    const int k0 = CUT ? (int)blockIdx.z * P.pt : 0, nt = CUT ? min(P.pt, P.nt - k0) : P.nt;  // the piece's tiles

    if (tid == 0) {
        alive = nt;  // until a wait gives up
        taken = make_int4(0, 0, kTakenAll, kTakenAll);
        for (int i = 0; i < 9; ++i) mbar_init(&bars[i], i < 7 ? 1 : 2);
        mbar_fence_init();
    }
    if (warp == MMAW) {
        tmem_alloc(&tmem_slot, 128 * NH);
        tmem_relinquish();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = tmem_slot;  // accumulator of tile parity b at columns [b * 64 NH, (b + 1) * 64 NH), head hs at + 64 hs

    if (warp == MMAW) {
        // ------------------------------------------------------------------ products
        const uint32_t cMN = desc_lo(smem_u32(sC), PANEL), uMN = desc_lo(smem_u32(sU0), PANEL);
        int sc = 0, su = 0;  // it % NC, it % NU
        uint32_t cph = 0;    // parity of the current turn of C's ring
#pragma unroll 1
        for (int it = 0; it < nt; ++it) {
            const int b = it & 1;
            if (lane == 0) mbar_wait(&bar_c[sc], cph, &alive);
            __syncwarp();
            named_bar_sync(kRevBarU + b, BAR);
            if (lane == 0) {
                tc_fence_after();
                uint32_t v = cMN + (uint32_t)sc * (2 * PANEL >> 4), u = uMN + (uint32_t)su * (NH * PANEL >> 4);
                asm volatile("" : "+r"(v), "+r"(u));
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)  // Hl = C^T [e . dY of each head] : both MN-major, K = position, N = 64 NH
                    mma_ss_lo(tm + b * 64 * NH, v + kk * 128, u + kk * 128, NH == 2 ? kIdescMM128 : kIdescMM, kk > 0);
                mma_commit(&bar_m[b]);
                set_taken(&taken.x, it + 1);
            }
            if (++sc == NC) {
                sc = 0;
                cph ^= 1;
            }
            if (++su == NU) su = 0;
        }
    } else if (warp == TMAW) {
        // ------------------------------------------------------------------ copies
        auto load_c = [&](int it) {
            uint8_t* st = sC + (size_t)(it % NC) * 2 * PANEL;
            uint64_t* bar = &bar_c[it % NC];
            const int pos = (k0 + nt - 1 - it) * LT;
            mbar_expect_tx(bar, 2 * PANEL);
            tma_load_4d(st, &P.mV, bar, 0, gg, pos, bb);
            tma_load_4d(st + PANEL, &P.mV, bar, 64, gg, pos, bb);
        };
        auto load_u = [&](int it) {
            uint8_t* st = sU0 + (size_t)(it % NU) * NH * PANEL;
            uint64_t* bar = &bar_u[it % NU];
            mbar_expect_tx(bar, NH * PANEL);
#pragma unroll
            for (int hs = 0; hs < NH; ++hs) tma_load_4d(st + hs * PANEL, &P.mU, bar, 0, hh0 + hs, (k0 + nt - 1 - it) * LT, bb);
        };
        if (lane == 0) {
            prefetch_tmap(&P.mU);
            prefetch_tmap(&P.mV);
#pragma unroll 1
            for (int it = 0; it < NU && it < nt; ++it) {
                load_u(it);
                if (it < NC) load_c(it);
            }
        }
#pragma unroll 1
        for (int it = 0; it < nt; ++it) {
            __syncwarp();
            named_bar_sync(kRevBarQ, BAR);  // the state gradient leaving tile nt-1-it is staged
            if (lane == 0) {
#pragma unroll
                for (int hs = 0; hs < NH; ++hs)
                    tma_store_2d(&P.mS, sQ0 + ((it & 1) * NH + hs) * PANEL, 0, (int)((((size_t)bb * P.nt + k0 + (nt - 1 - it)) * P.h + hh0 + hs) * DN));
                tma_store_commit();
                set_taken(&taken.y, it + 1);
                tma_store_wait_read<1>();
                mbar_arrive(&bar_m[it & 1]);  // the other panels may be rewritten
                mbar_wait(&bar_m[it & 1], (it >> 1) & 1, &alive);  // the MMA of the tile is done
                if (it + NC < nt) load_c(it + NC);
                if (it + NU < nt) load_u(it + NU);
            }
        }
        if (lane == 0) tma_store_wait_all();
    } else {
        // ------------------------------------------------------------------ row warps
        const int hs = tid >> 8;  // which of the CTA's heads
        const int hh = hh0 + hs;
        const int ht = tid & 255, row = ht & 127, hf = ht >> 7;
        const size_t bh = (size_t)bb * P.h + hh;
        const float* tcum = P.tcum + bh * P.Tp + (size_t)(k0 + nt - 1) * LT;  // of the walk's first tile; the next ones lie before it
        const uint32_t lanes = lane_base(warp);
        uint8_t* sQ = sQ0 + (size_t)hs * PANEL;  // of the even tiles; the odd ones' NH panels behind
        float H[32];  // state gradient row n = row, p in [hf*32, hf*32+32)
        if (CUT) load_piece_row<true>(P, bh, row, hf * 32, H);
        else load_state_row(P.seed, bh, P.p, P.n, row, hf * 32, H);
        float c0 = tcum[row], S0 = tcum[LT - 1], c1 = 0.f, S1 = 0.f;  // of the tile, and of the one behind
        if (nt > 1) {
            c1 = tcum[row - LT];
            S1 = tcum[-1];
        }
        int s = 0;         // stage of the tile that is weighed next
        uint32_t lph = 0;  // parity of the current turn of the ring
#pragma unroll 1
        for (int it = -1; it < nt; ++it) {
            // weighted copy of this thread's half row of dY of tile it + 1, in place
            if (it + 1 < nt) {
                mbar_wait(&bar_u[s], lph, &alive);
                uint8_t* sU = sU0 + (size_t)(s * NH + hs) * PANEL;
                const __nv_bfloat162 w2 = __float2bfloat162_rn(exp2f(it < 0 ? c0 : c1));
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
                tc_fence_before();
                fence_async_smem();
                hand_over(kRevBarU + ((it + 1) & 1), BAR);
                if (++s == NU) {
                    s = 0;
                    lph ^= 1;
                }
            }
            if (it >= 0) {
                const float dec = exp2f(S0);
                S0 = S1;
                if (it + 2 < nt) {
                    c1 = tcum[row - (it + 2) * LT];
                    S1 = tcum[LT - 1 - (it + 2) * LT];
                }
                mbar_wait(&bar_m[it & 1], (it >> 1) & 1, &alive);
                const int live = *(const volatile int*)&alive;
                tc_fence_after();
                uint32_t r[32];
                tmem_ld32(tm + (it & 1) * 64 * NH + hs * 64 + lanes + hf * 32, r);
                tmem_ld_wait();
                float2* H2 = reinterpret_cast<float2*>(H);
                const float2 d2 = make_float2(dec, dec);
#pragma unroll
                for (int q = 0; q < 16; ++q) H2[q] = fma2(d2, H2[q], reinterpret_cast<const float2*>(r)[q]);
                if (it + 1 >= live) {
                    if (it + 1 == nt) break;
                    until_taken(1, &taken, it);  // U and Q of the tile are behind what was waited for
                }
            }
            store_half_row(sQ + ((it + 1) & 1) * NH * PANEL, row, hf * 4, H);  // (the store of two tiles before has read it: bar_m)
            fence_async_smem();
            hand_over(kRevBarQ, BAR);
        }
        if (k0 == 0) store_state_row(P.out_state, bh, P.p, P.n, row, hf * 32, H);
    }
    tc_fence_before();
    __syncthreads();
    end_of_waits(&alive, P.status);
    if (warp == MMAW) tmem_dealloc(tm, 128 * NH);
}

}  // namespace tc
}  // namespace ssd
