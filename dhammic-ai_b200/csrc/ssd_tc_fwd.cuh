// Forward walk of the tensor-core path (included by ssd_tc.cuh).
//
// One CTA per (batch, head, piece of the sequence) walks the 128-position tiles in order with the recurrent state
// (64 x 128, fp32) in registers; more than one piece where (batch, head) pairs alone leave most of the chip idle (Pieces,
// ssd_tc_host.cuh).  Per tile k (V = B, U = x, C of the tile; H = state entering it; S_k = its total log2-decay):
//   S  = C V^T                     issued one tile ahead into a double-buffered TMEM accumulator
//   Hl = V^T (d dt o U)            the tile's contribution to the state, one tile ahead; the weighted copy of U is made by the rows
//   Yo = C H^T                     the entering state's part of the output
//   G' = S o L o dt  (bf16 pairs, written back to TMEM by the rows),  Yd = G' U   (A operand from TMEM)
//   y  = e o Yo + Yd + skip o x,   H <- 2^{S_k} H + Hl
// 16 row warps: thread = (row, column quarter).  A quarter is one 32-column block of the causal mask (active iff
// quarter <= row block), 16 columns of every 64-wide accumulator and 16 values of the row's state.  Four control warps: one lane of each issues
// copies or products.  The kernel starts at 96 registers per thread; the control warpgroup gives registers back and the
// row warps take them (setmaxnreg).
//
// What bounds it is the chain of a tile's steps and, with every SM busy, the clock, which falls from 1.9 to 1.6 GHz.  A tile's chain is
// mask -> state update, beside Yd -> output; everything else runs ahead:
//   * x has a ring of its own, three tiles deep; its weighted copy for tile k+1 is made while Yd of tile k runs, so that Hl and Yo of a tile are done
//     when its mask is.  B and C, whose last reader Yo runs early in their tile, have two stages that are refilled from there on.
//   * A lane that waits has to let the products it has issued drain first (some 300 cycles), so products that wait for different things are
//     issued by different warps; and an mbarrier arrive reaches a polling lane some 300 cycles later, a hardware barrier 30, so the row warps
//     hand over by bar.arrive.
//   * All loops that run at once (16 row warps, four control warps) have to fit the instruction cache: with the waits
//     unrolled by the compiler the pipeline above was slower than one without any of this, 315 us against 286 for 148 walks of 128 tiles.
// (16, 4096, 64 heads, 8 groups): 520 -> 424 us, 512 -> 384 without kept states; (8, 2048, 24) 85 -> 58, and 53 with the last walks cut; one walk of 128 tiles to every other SM
// 280 -> 184.  Tried and slower: the state on eight warps and mask and output on the other eight (500 us: the masks of the rows 96-127 take two
// warps 1,500 cycles and four 1,000); Yd in two halves as the masks complete (its lane drains in between).
//
// Shared memory: 2 stages of [V panels 0,1 | C panels 0,1] | x ring, y staged in place | weighted x | state (bf16 [n][p]) |
// per-position scalars of the ring's tiles, copied with x | column factors | barriers.  TMEM: S double-buffered [0,256), G' [256,320), Yd [320,384),
// Yo [384,448), Hl [448,512).
//
// mbarriers (s = tile & 1, phase = (tile / 2) & 1 unless noted):
//   bar_vc[s]  B and C of the tile landed
//   bar_mh[s]  Hl and Yo of the tile have completed, the store of its entering state has read sH, x of the next tile landed (-> row warps,
//              loads of B and C)
//   bar_m2[s]  Yd of the tile and S of the next have completed     (-> row warps)
//   bar_s0, bar_x0   S and x of the first tile
// Where several warps arrive at an mbarrier, none of them may arrive for a later tile before the others have for this one, or the phase completes without what it
// stands for.  bar_mh and bar_m2 are two each for that: a warp's next arrival at the same one is two tiles later, behind a hardware barrier that the row
// warps reach only when they have seen this phase complete.  bar_m2 of tile k: they wait for it ahead of kBarU of tile k + 2 (ahead of Hl, S and the last
// tile's arrival) and of kBarG (ahead of Yd), but behind kBarU of tile k + 1.  bar_mh of tile k: they wait for it ahead of kBarU of tile k + 1.
// Named barriers (row warps arrive, control warps wait):
//   kBarU   weighted rows of a tile and the state entering it written, Hl and Yo of the tile before read (-> Hl, Yo, store of the state)
//   kBarG   masked operand written                                  (-> Yd; two by tile parity: see until_taken)
//   kBarH   y staged over x, the tile's x and scalars no longer used (-> store of y, next load into the slot; two by tile parity: the row warps
//           may arrive once more before the store's warp has seen the last one)
// The per-half-row sums of y^2 keep their (b, T/128, h, 2, 128) layout: the odd quarter of each half leaves its partial
// in shared memory, the even quarter adds its own and writes the sum during the next tile.
//
// The diagonal block of the mask is evaluated entry by entry (one exponential each, by four of the ten warps that have a block to mask), which holds for any log-decay; below it
// the mask is the product of a row and a column factor, both at most 1.  (A second instantiation with factors in the diagonal block as well, and a
// flag that chose between the two on the device, was no faster, and the idle one of the two took 2.3 to 7 us a call.)
#pragma once

namespace ssd {
namespace tc {

constexpr int kFwdThreads = 640;
constexpr int kFwdRegsLaunch = 96, kFwdRegsRow = 104, kFwdRegsCtl = 64;
static_assert(512 * kFwdRegsRow + 128 * kFwdRegsCtl <= kFwdThreads * kFwdRegsLaunch, "register trade exceeds the CTA's pool");
constexpr uint32_t kFwdStageBytes = 4 * PANEL;  // V panels 0,1 | C panels 0,1
constexpr int kFwdStages = 2, kFwdRing = 3;
// stages | x ring (y staged in place) | weighted x, state | per ring slot: cumulative decay, dt, skip coefficient [128] each | column factors of
// each row warp [16][32] | partial sums of y^2 [2][2][128] | barriers
constexpr size_t kFwdSmem = kFwdStages * (size_t)kFwdStageBytes + (kFwdRing + 2) * (size_t)PANEL + (3 * kFwdRing + 4 + 4) * LT * 4 + 192;
// named barriers: all row warps arrive, one or three control warps wait
constexpr int kBarG = 1 /* and 2 */, kBarU = 3, kBarH = 4 /* and 5 */, kBarRows = 6, kBarLead = 7, kBarLeadU = 8 /* and 9 */;
constexpr int kLeadStages = 4;  // of [V panels 0,1 | x], over everything in front of the state
static_assert(kFwdSmem <= 227 * 1024, "more shared memory than a CTA can have");

// 16 fp32 values of (row, quarter) as two 16-byte chunks of a 128-byte-swizzled [row][64] bf16 panel
__device__ __forceinline__ void store_quarter_row(uint8_t* panel, int row, int chunk0, const float (&v)[16]) {
#pragma unroll
    for (int ch = 0; ch < 2; ++ch) {
        uint4 o;
        o.x = pack_bf16(v[ch * 8 + 0], v[ch * 8 + 1]);
        o.y = pack_bf16(v[ch * 8 + 2], v[ch * 8 + 3]);
        o.z = pack_bf16(v[ch * 8 + 4], v[ch * 8 + 5]);
        o.w = pack_bf16(v[ch * 8 + 6], v[ch * 8 + 7]);
        *reinterpret_cast<uint4*>(panel + sw128(row, chunk0 + ch)) = o;
    }
}

__global__ void __maxnreg__(kFwdRegsLaunch) fwd_walk_kernel(const __grid_constant__ WalkParams P) {
    dep_wait();
    if (P.zero_status) clear_status(P.status);
    // no static shared memory: the dynamic region starts at the CTA's shared-memory base
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* sStage = smem_raw;                            // per stage: V panels 0,1 | C panels 0,1
    uint8_t* sRing = sStage + kFwdStages * kFwdStageBytes; // x; y is staged over it
    uint8_t* sUd = sRing + kFwdRing * PANEL;               // weighted copy of x
    uint8_t* sH = sUd + PANEL;                             // state, bf16, [n][p]
    float* scum = reinterpret_cast<float*>(sH + PANEL);    // [ring][3][128] tile-cumulative log2-decay, dt, skip coefficient
    float* sf = scum + 3 * kFwdRing * LT;                  // [16][32] column factors dt_j 2^(cend - c_j) of each row warp's block
    float* sysq = sf + 4 * LT;                             // [2][2][128] partial sums of y^2 of the odd quarters
    uint64_t* bars = reinterpret_cast<uint64_t*>(sysq + 4 * LT);
    uint64_t *bar_vc = bars, *bar_mh = bars + 2, *bar_m2 = bars + 4, *bar_s0 = bars + 6, *bar_x0 = bars + 7, *lead_ld = bars + 8, *lead_m = bars + 12;
    uint32_t& tmem_slot = *reinterpret_cast<uint32_t*>(bars + 16);
    int& alive = *reinterpret_cast<int*>(bars + 17);
    int& rows_nt = *reinterpret_cast<int*>(bars + 18);  // (`alive` is the same until a wait gives up)
    // see until_taken: .x kBarG, .y kBarU and kBarH; kBarLeadU
    int4 &taken = *reinterpret_cast<int4*>(bars + 20), &taken_lead = *reinterpret_cast<int4*>(bars + 22);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (smem_u32(smem_raw) & 1023u) {  // the swizzled panels need a 1024-byte aligned base: report instead of computing garbage
        if (tid == 0) atomicExch(P.status, 2);
        return;
    }
    int hh = blockIdx.x, bb = blockIdx.y;
    int k0 = blockIdx.z * P.pt, nt = min(P.pt, P.nt - k0);  // the piece's tiles
    int lead = 0;                                           // tiles before them whose states this CTA walks for itself
    if (P.self.np > 1) {  // one-dimensional grid: whole walks, then pieces that find their own way (SelfCut)
        const int r = blockIdx.x - P.self.whole, pair = r < 0 ? (int)blockIdx.x : P.self.whole + r / P.self.np, z = r < 0 ? 0 : r % P.self.np;
        hh = pair % P.h;
        bb = pair / P.h;
        k0 = lead = r < 0 ? 0 : P.self.cut[z];
        nt = (r < 0 ? P.nt : P.self.cut[z + 1]) - k0;
    }
    const int gg = hh / P.hpg;
    const size_t bh = (size_t)bb * P.h + hh;

    if (tid == 0) {
        alive = nt;
        taken = make_int4(1, 0, kTakenAll, kTakenAll);
        taken_lead = make_int4(0, kTakenAll, kTakenAll, kTakenAll);
        rows_nt = nt;
        for (int i = 0; i < 16; ++i) mbar_init(&bars[i], i == 2 || i == 3 ? 4 : i == 4 || i == 5 ? 2 : 1);  // mh: Hl, Yo, the store of the state, the next tile's x; m2: Yd, the next S
        mbar_fence_init();
    }
    if (warp == 16) {
        tmem_alloc(&tmem_slot, 512);
        tmem_relinquish();
    }
    const int row = tid & 127, q = (tid >> 7) & 3;
    // state row of this thread: n = row, p in [16 q, 16 q + 16)
    float H[16];
    if (warp < 16) {
        if (!P.dtT)
            for (int i = tid; i < kFwdRing * LT; i += 512) scum[(3 * (i / LT) + 1) * LT + i % LT] = 1.f;
        load_piece_row<false>(P, bh, row, q * 16, H);
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tm = tmem_slot;
    // S double-buffered [0,256), masked operand (bf16 pairs) [256,320), Yd [320,384), Yo [384,448), Hl [448,512)
    const uint32_t tG = tm + 256, tYd = tm + 320, tYo = tm + 384, tHl = tm + 448;
    if (warp >= 16) {
        setmaxnreg_dec<kFwdRegsCtl>();
        const uint32_t stK = desc_lo(smem_u32(sStage), 16), stMN = desc_lo(smem_u32(sStage), PANEL);
        constexpr uint32_t PU = PANEL >> 4, SU = kFwdStageBytes >> 4;  // panel and stage pitch in 16-byte units
        auto offK = [](int kk) { return (uint32_t)(((kk >> 2) * (int)PANEL + (kk & 3) * 32) >> 4); };
        auto offMN = [](int kk) { return (uint32_t)(kk * 128); };
        auto fresh = [](uint32_t v) {  // keeps the descriptors from being hoisted out of the tile loop (64 registers here)
            asm volatile("" : "+r"(v));
            return v;
        };
        auto load_vc = [&](int it) {
            uint8_t* st = sStage + (size_t)(it & 1) * kFwdStageBytes;
            uint64_t* bar = &bar_vc[it & 1];
            mbar_expect_tx(bar, kFwdStageBytes);
            const int pos = (k0 + it) * LT;
            tma_load_4d(st, &P.mV, bar, 0, gg, pos, bb);
            tma_load_4d(st + PANEL, &P.mV, bar, 64, gg, pos, bb);
            tma_load_4d(st + 2 * PANEL, &P.mC, bar, 0, gg, pos, bb);
            tma_load_4d(st + 3 * PANEL, &P.mC, bar, 64, gg, pos, bb);
        };
        if (warp == 16) {
            // ------------------------------------------------------------------ products: Yd
            const uint32_t xMN = desc_lo(smem_u32(sRing), PANEL);
            int r = 0;  // it % 3
#pragma unroll 1
            for (int it = 0; it < nt; ++it) {
                __syncwarp();
                named_bar_sync(kBarG + (it & 1), 544);
                if (lane == 0) {
                    tc_fence_after();
                    const uint32_t uMN = fresh(xMN + (uint32_t)r * PU);
#pragma unroll
                    for (int kk = 0; kk < 8; ++kk)  // Yd = G' x : A in TMEM (K = j), B = x [j][p] MN-major
                        mma_ts_lo(tYd, tG + kk * 8, uMN + offMN(kk), kIdescKM, kk > 0);
                    mma_commit(&bar_m2[it & 1]);
                    set_taken(&taken.x, it + 2);
                }
                if (++r == kFwdRing) r = 0;
            }
        } else if (warp == 17) {
            // ------------------------------------------------------------------ TMA: x, every store
            const size_t t0 = bh * P.Tp + (size_t)k0 * LT;
            auto load_x = [&](int it) {  // and the tile's per-position scalars
                const int r = it % kFwdRing;
                uint64_t* bar = it > 0 ? &bar_mh[(it - 1) & 1] : bar_x0;
                mbar_expect_tx(bar, PANEL + LT * 4 * (1 + (P.dtT != nullptr) + (P.skipT != nullptr)));
                tma_load_4d(sRing + r * PANEL, &P.mU, bar, 0, hh, (k0 + it) * LT, bb);
                float* sc = scum + r * 3 * LT;
                const size_t o = t0 + (size_t)it * LT;
                bulk_load(sc, P.tcum + o, LT * 4, bar);
                if (P.dtT) bulk_load(sc + LT, P.dtT + o, LT * 4, bar);
                if (P.skipT) bulk_load(sc + 2 * LT, P.skipT + o, LT * 4, bar);
            };
            auto store_y = [&](int it) {
                tma_store_4d(&P.mY, sRing + (it % kFwdRing) * PANEL, 0, hh, (k0 + it) * LT, bb);
                tma_store_commit();
            };
            if (lane == 0) prefetch_tmap(&P.mU);
            if (lead > 0) {
                if (lane == 0) {
                    for (int it = 0; it < 2 && it < nt; ++it) {  // what the piece itself starts with comes to the L2 meanwhile
                        const int pos = (k0 + it) * LT;
                        tma_prefetch_4d(&P.mU, 0, hh, pos, bb);
                        for (int c = 0; c < 128; c += 64) {
                            tma_prefetch_4d(&P.mV, c, gg, pos, bb);
                            tma_prefetch_4d(&P.mC, c, gg, pos, bb);
                        }
                    }
#pragma unroll 1
                    for (int it = 0; it < lead; ++it) {
                        const int s = it % kLeadStages, pos = it * LT;
                        uint8_t* st = smem_raw + s * 3 * PANEL;
                        if (it >= kLeadStages) mbar_wait(&lead_m[s], (it / kLeadStages - 1) & 1, &alive);  // the stage's product before is done
                        mbar_expect_tx(&lead_ld[s], 3 * PANEL);
                        tma_load_4d(st + 2 * PANEL, &P.mU, &lead_ld[s], 0, hh, pos, bb);
                        tma_load_4d(st, &P.mV, &lead_ld[s], 0, gg, pos, bb);
                        tma_load_4d(st + PANEL, &P.mV, &lead_ld[s], 64, gg, pos, bb);
                    }
                }
                __syncwarp();
                named_bar_sync(kBarLead, 576);
            }
            if (lane == 0)
                for (int it = 0; it < kFwdRing && it < nt; ++it) load_x(it);
#pragma unroll 1
            for (int it = 0; it < nt; ++it) {
                __syncwarp();
                named_bar_sync(kBarU, 608);  // the entering state is in sH
                if (lane == 0 && P.save_states) {
                    tma_store_2d(&P.mS, sH, 0, (int)((((size_t)bb * P.nt + k0 + it) * P.h + hh) * DN));
                    tma_store_commit();
                }
                if (it > 0) {
                    __syncwarp();
                    named_bar_sync(kBarH + ((it - 1) & 1), 544);  // y of the tile before staged
                    if (lane == 0) store_y(it - 1);
                }
                if (lane == 0) {
                    set_taken(&taken.y, it + 1);
                    if (it > 0) tma_store_wait_read<1>();
                    else tma_store_wait_read();
                    mbar_arrive(&bar_mh[it & 1]);  // the store has read sH
                    if (it + 1 == nt) mbar_arrive(&bar_mh[it & 1]);  // (no x behind it)
                    if (it > 0 && it + 2 < nt) {
                        tma_store_wait_read();  // y
                        load_x(it + 2);
                    }
                }
            }
            __syncwarp();
            named_bar_sync(kBarH + ((nt - 1) & 1), 544);
            if (lane == 0) {
                store_y(nt - 1);
                tma_store_wait_all();
            }
        } else {
            // ------------------------------------------------------------------ products: Hl and S in one warp, Yo and the loads of B and C in another
            const bool hl = warp == 18;
            const uint32_t udMN = desc_lo(smem_u32(sUd), PANEL), hMN = desc_lo(smem_u32(sH), PANEL);
            auto issue_S = [&](int it) {  // S = C B^T of tile `it` into TMEM buffer it & 1, which the rows have masked two tiles before
                mbar_wait(&bar_vc[it & 1], (it >> 1) & 1, &alive);
                tc_fence_after();
                const uint32_t vK = fresh(stK + (uint32_t)(it & 1) * SU), cK = vK + 2 * PU, tS = tm + (it & 1) * 128;
#pragma unroll
                for (int kk = 0; kk < 8; ++kk) mma_ss_lo(tS, cK + offK(kk), vK + offK(kk), kIdescKK128, kk > 0);
                mma_commit(it > 0 ? &bar_m2[(it - 1) & 1] : bar_s0);
            };
            if (!hl && lead > 0) named_bar_sync(kBarLead, 576);
            if (hl) {
#pragma unroll 1
                for (int it = 0; it < lead; ++it) {
                    __syncwarp();
                    named_bar_sync(kBarLeadU + (it & 1), 544);
                    if (lane == 0) {
                        tc_fence_after();
                        const uint32_t st = fresh(stMN + (uint32_t)(it % kLeadStages) * 3 * PU);
#pragma unroll 2
                        for (int kk = 0; kk < 8; ++kk)  // V^T [d dt o x]
                            mma_ss_lo(tYo + (it & 1) * 64, st + offMN(kk), st + 2 * PU + offMN(kk), kIdescMM, kk > 0);
                        mma_commit(&lead_m[it % kLeadStages]);
                        set_taken(&taken_lead.x, it + 1);
                    }
                }
            }
            if (!hl && lane == 0) {
                prefetch_tmap(&P.mV);
                prefetch_tmap(&P.mC);
                load_vc(0);
                if (nt > 1) load_vc(1);
            }
            if (hl && lane == 0) issue_S(0);
#pragma unroll 1
            for (int it = 0; it < nt; ++it) {
                if (!hl && lane == 0) mbar_wait(&bar_vc[it & 1], (it >> 1) & 1, &alive);
                __syncwarp();
                named_bar_sync(kBarU, 608);  // weighted rows and entering state written, Hl and Yo of the tile before read
                if (lane == 0) {
                    tc_fence_after();
                    if (hl) {
                        const uint32_t vMN = fresh(stMN + (uint32_t)(it & 1) * SU), udMN_ = fresh(udMN);
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)  // Hl = V^T Ud : both MN-major, K = position
                            mma_ss_lo(tHl, vMN + offMN(kk), udMN_ + offMN(kk), kIdescMM, kk > 0);
                    } else {
                        const uint32_t cK = fresh(stK + (uint32_t)(it & 1) * SU + 2 * PU), hMN_ = fresh(hMN);
#pragma unroll
                        for (int kk = 0; kk < 8; ++kk)  // Yo = C H^T : A = C K-major, B = the running state in sH, [n][p] MN-major
                            mma_ss_lo(tYo, cK + offK(kk), hMN_ + offMN(kk), kIdescKM, kk > 0);
                    }
                    mma_commit(&bar_mh[it & 1]);
                    if (hl) {
                        if (it + 1 < nt) issue_S(it + 1);
                        else mbar_arrive(&bar_m2[it & 1]);  // (no S behind it)
                    } else if (it + 2 < nt) {
                        mbar_wait(&bar_mh[it & 1], (it >> 1) & 1, &alive);  // Hl and Yo (and S) of the tile, the readers of its stage, have completed
                        load_vc(it + 2);
                    }
                }
            }
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ row warps: thread = (row, column quarter)
        setmaxnreg_inc<kFwdRegsRow>();
        const int rb = row >> 5;  // row block, warp-uniform
        const bool active = q <= rb, diag = q == rb;
        const uint32_t lanes = lane_base(warp);
        const float Dhead = P.D ? P.D[hh] : 0.f;
        const bool has_skip = P.D || P.skipT;
        const int c0 = q * 32;  // this thread's 32 columns of S
        float* wsf = sf + warp * 32;
        float c_i, Sk = 0.f;  // of the tile that `weigh` has prepared
        uint32_t xw[8];     // its weighted x: this thread's quarter row
        // What a tile needs of x and the scalars before its own turn: the weighted copy, the column factors of this warp's block.
        auto weigh = [&](int r) {
            const float* sc = scum + r * 3 * LT;
            c_i = sc[row];
            Sk = sc[LT - 1];
            // the row weight as a bf16 pair: one packed multiply per two elements (the product is rounded to
            // bf16 for the MMA anyway; rounding the weight first costs at most one more ulp of bf16)
            const __nv_bfloat162 w2 = __float2bfloat162_rn(exp2f(Sk - c_i) * sc[LT + row]);
            const uint8_t* sU = sRing + r * PANEL;
#pragma unroll
            for (int ch = 0; ch < 2; ++ch) {
                const uint4 v = *reinterpret_cast<const uint4*>(sU + sw128(row, q * 2 + ch));
                const uint32_t* u = reinterpret_cast<const uint32_t*>(&v);
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    __nv_bfloat162 p = __hmul2(*reinterpret_cast<const __nv_bfloat162*>(&u[j]), w2);
                    xw[ch * 4 + j] = *reinterpret_cast<uint32_t*>(&p);
                }
            }
        };
        float rf = 0.f;  // row factor of this warp's block, relative to the block's last column
        auto factors = [&](int r) {
            if (active && !diag) {
                const float* sc = scum + r * 3 * LT;
                const float cend = sc[c0 + 31];
                wsf[lane] = sc[LT + c0 + lane] * exp2f(cend - sc[c0 + lane]);
                rf = exp2f(c_i - cend);
            }
        };
        auto put_weighted = [&]() {
            *reinterpret_cast<uint4*>(sUd + sw128(row, q * 2)) = make_uint4(xw[0], xw[1], xw[2], xw[3]);
            *reinterpret_cast<uint4*>(sUd + sw128(row, q * 2 + 1)) = make_uint4(xw[4], xw[5], xw[6], xw[7]);
            tc_fence_before();
            fence_async_smem();
            hand_over(kBarU, 608);
        };
        float ysq_own = 0.f;  // even quarters: own partial of the tile before
        if (lead > 0) {
            // the states of the tiles before the piece, as the walk itself makes them: weighted rows in place, one tile ahead of the product, whose
            // accumulator alternates between the columns of Yo and Hl
            const float *tc = P.tcum + bh * P.Tp, *dt = P.dtT ? P.dtT + bh * P.Tp : nullptr;
            float c = tc[row], S = tc[LT - 1], d = dt ? dt[row] : 1.f;
#pragma unroll 1
            for (int it = -1; it < lead; ++it) {
                const float dec = exp2f(it < 0 ? 0.f : Sk);
                if (it + 1 < lead) {
                    const int s = (it + 1) % kLeadStages;
                    mbar_wait(&lead_ld[s], ((it + 1) / kLeadStages) & 1, &alive);
                    uint8_t* sU = smem_raw + (s * 3 + 2) * PANEL;
                    const __nv_bfloat162 w2 = __float2bfloat162_rn(exp2f(S - c) * d);
#pragma unroll
                    for (int ch = 0; ch < 2; ++ch) {
                        uint4* p4 = reinterpret_cast<uint4*>(sU + sw128(row, q * 2 + ch));
                        uint4 v = *p4;
                        uint32_t* u = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            __nv_bfloat162 p = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&u[j]), w2);
                            u[j] = *reinterpret_cast<uint32_t*>(&p);
                        }
                        *p4 = v;
                    }
                    Sk = S;
                    tc_fence_before();
                    fence_async_smem();
                    hand_over(kBarLeadU + ((it + 1) & 1), 544);
                    if (it + 2 < lead) {
                        const int o = (it + 2) * LT;
                        c = tc[o + row];
                        S = tc[o + LT - 1];
                        d = dt ? dt[o + row] : 1.f;
                    }
                }
                if (it >= 0) {
                    mbar_wait(&lead_m[it % kLeadStages], (it / kLeadStages) & 1, &alive);
                    until_taken(gave_up(&alive), &taken_lead, it);
                    tc_fence_after();
                    uint32_t r[16];
                    tmem_ld16(tYo + (it & 1) * 64 + lanes + q * 16, r);
                    tmem_ld_wait();
                    float2* H2 = reinterpret_cast<float2*>(H);
                    const float2 d2 = make_float2(dec, dec);
#pragma unroll
                    for (int j = 0; j < 8; ++j) H2[j] = fma2(d2, H2[j], reinterpret_cast<const float2*>(r)[j]);
                }
            }
            hand_over(kBarLead, 576);  // the panels are free
        }
        store_quarter_row(sH, row, q * 2, H);
        mbar_wait(bar_x0, 0, &alive);
        weigh(0);
        put_weighted();
        factors(0);
        mbar_wait(bar_s0, 0, &alive);
        tc_fence_after();
        int ring = 0;  // it % 3

#pragma unroll 1
        for (int it = 0;;) {
            const uint32_t ph = it & 1;
            const float e = exp2f(c_i), dec = exp2f(Sk);
            const float* sc = scum + ring * 3 * LT;
            const uint32_t tS = tm + (it & 1) * 128 + lanes + c0;
            if (diag) {  // entry by entry
                const float4* C4 = reinterpret_cast<const float4*>(sc + c0);
                const float4* T4 = reinterpret_cast<const float4*>(sc + LT + c0);
#pragma unroll
                for (int sub = 0; sub < 2; ++sub) {
                    uint32_t r[16], packed[8];
                    tmem_ld16(tS + sub * 16, r);
                    float2 l[8];
#pragma unroll
                    for (int q4 = 0; q4 < 4; ++q4) {
                        const int j = sub * 16 + 4 * q4;
                        const float4 cj = C4[sub * 4 + q4], tj = T4[sub * 4 + q4];
                        l[2 * q4].x = (j > lane) ? 0.f : tj.x * ex2(c_i - cj.x);
                        l[2 * q4].y = (j + 1 > lane) ? 0.f : tj.y * ex2(c_i - cj.y);
                        l[2 * q4 + 1].x = (j + 2 > lane) ? 0.f : tj.z * ex2(c_i - cj.z);
                        l[2 * q4 + 1].y = (j + 3 > lane) ? 0.f : tj.w * ex2(c_i - cj.w);
                    }
                    tmem_ld_wait();
                    const float2* S2 = reinterpret_cast<const float2*>(r);
#pragma unroll
                    for (int q2 = 0; q2 < 8; ++q2) {
                        const float2 v = mul2(S2[q2], l[q2]);
                        packed[q2] = pack_bf16(v.x, v.y);
                    }
                    tmem_st8(tG + lanes + q * 16 + sub * 8, packed);
                }
                tmem_st_wait();
            } else if (active) {
                uint32_t r[32], packed[16];
                tmem_ld32(tS, r);
                __syncwarp();  // the warp's column factors
                const float2 rf2 = make_float2(rf, rf);
                const float4* F4 = reinterpret_cast<const float4*>(wsf);
                tmem_ld_wait();
                const float2* S2 = reinterpret_cast<const float2*>(r);
#pragma unroll
                for (int q4 = 0; q4 < 8; ++q4) {  // fp32 pairs: one instruction, two columns
                    const float4 f = F4[q4];
                    const float2 v = mul2(S2[2 * q4], mul2(rf2, make_float2(f.x, f.y))), w = mul2(S2[2 * q4 + 1], mul2(rf2, make_float2(f.z, f.w)));
                    packed[2 * q4] = pack_bf16(v.x, v.y);
                    packed[2 * q4 + 1] = pack_bf16(w.x, w.y);
                }
                tmem_st16(tG + lanes + q * 16, packed);
                tmem_st_wait();
            } else if (it == 0) {  // above the diagonal G' is zero in every tile: written once
                uint32_t packed[16];
#pragma unroll
                for (int j = 0; j < 16; ++j) packed[j] = 0u;
                tmem_st16(tG + lanes + q * 16, packed);
                tmem_st_wait();
            }
            tc_fence_before();
            hand_over(kBarG + ph, 544);

            // while Yd runs: what the next tile needs early, and the state update
            uint8_t* sU = sRing + ring * PANEL;
            const float Dh = P.skipT ? sc[2 * LT + row] : Dhead;
            if (++ring == kFwdRing) ring = 0;
            mbar_wait(&bar_mh[ph], (it >> 1) & 1, &alive);  // Hl and Yo have completed, so sH and sUd are free; the next tile's x is there
            tc_fence_after();
            if (P.ysq && it > 0 && !(q & 1))  // the sum of the half row of the tile before: own quarter + the odd one's (written before this tile's mask)
                P.ysq[((((size_t)bb * P.nt + k0 + (it - 1)) * P.h + hh) * 2 + (q >> 1)) * LT + row] =
                    ysq_own + sysq[(((it - 1) & 1) * 2 + (q >> 1)) * LT + row];
            uint32_t o[16];
            const int rnt = *(const volatile int*)&alive;  // tiles of the walk (the row warps have no register left for it), or zero
            {
                uint32_t r[16];
                tmem_ld16(tHl + lanes + q * 16, r);
                tmem_ld16(tYo + lanes + q * 16, o);
                if (it + 1 < rnt) weigh(ring);
                tmem_ld_wait();
                float2* H2 = reinterpret_cast<float2*>(H);
                const float2 d2 = make_float2(dec, dec);
#pragma unroll
                for (int j = 0; j < 8; ++j) H2[j] = fma2(d2, H2[j], reinterpret_cast<const float2*>(r)[j]);
            }
            if (it + 1 < rnt) {
                store_quarter_row(sH, row, q * 2, H);
                put_weighted();
                factors(ring);
            } else if (rnt <= 0) {
                until_taken(1, &taken, it);  // U of this tile, H and G of the one before are behind what was waited for
                if (it + 1 < rows_nt) hand_over(kBarU, 608);
            }
            {
                uint32_t a[16], xrow[8];
#pragma unroll
                for (int ch = 0; ch < 2; ++ch) {
                    const uint4 v = *reinterpret_cast<const uint4*>(sU + sw128(row, q * 2 + ch));
                    xrow[ch * 4 + 0] = v.x; xrow[ch * 4 + 1] = v.y; xrow[ch * 4 + 2] = v.z; xrow[ch * 4 + 3] = v.w;
                }
                mbar_wait(&bar_m2[ph], (it >> 1) & 1, &alive);
                tc_fence_after();
                tmem_ld16(tYd + lanes + q * 16, a);
                tmem_ld_wait();
                float y[16];
                const float2* A2 = reinterpret_cast<const float2*>(a);
                const float2* O2 = reinterpret_cast<const float2*>(o);
                float2* Y2 = reinterpret_cast<float2*>(y);
                const float2 e2 = make_float2(e, e), D2 = make_float2(Dh, Dh);
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    float2 v = fma2(e2, O2[j], A2[j]);
                    if (has_skip) v = fma2(D2, __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&xrow[j])), v);
                    Y2[j] = v;
                }
                store_quarter_row(sU, row, q * 2, y);  // over this thread's own values of x, which Yd has read
                if (P.ysq) {  // sum of squares of this quarter row, for the norm over all heads that follows the scan
                    float2 s2 = make_float2(0.f, 0.f);
#pragma unroll
                    for (int j = 0; j < 8; ++j) s2 = fma2(Y2[j], Y2[j], s2);
                    if (q & 1) sysq[((it & 1) * 2 + (q >> 1)) * LT + row] = s2.x + s2.y;
                    else ysq_own = s2.x + s2.y;
                }
            }
            tc_fence_before();
            fence_async_smem();
            hand_over(kBarH + ph, 544);
            if (++it >= *(const volatile int*)&alive && it >= rows_nt) break;
        }
        const int rnt = rows_nt;
        if (P.ysq) {
            named_bar_sync(kBarRows, 512);
            if (!(q & 1))
                P.ysq[((((size_t)bb * P.nt + k0 + (rnt - 1)) * P.h + hh) * 2 + (q >> 1)) * LT + row] =
                    ysq_own + sysq[(((rnt - 1) & 1) * 2 + (q >> 1)) * LT + row];
        }
        if (k0 + rnt == P.nt) store_state_row(P.out_state, bh, P.p, P.n, row, q * 16, H);
    }
    tc_fence_before();
    __syncthreads();
    end_of_waits(&alive, P.status);
    if (warp == 16) tmem_dealloc(tm, 512);
}

}  // namespace tc
}  // namespace ssd
