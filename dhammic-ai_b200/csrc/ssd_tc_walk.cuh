// State walk of the tensor-core path and what the walk kernels share (included by ssd_tc.cuh).
//
// states_walk_kernel: one CTA per (batch, head, piece of the sequence) walks the 128-position tiles in order with the recurrent state
// (64 x 128, fp32) in registers and stores the state entering every tile as bf16 — the recurrence of the forward without
// its output.  The backward uses it when the forward did not keep the states.  Ten warps:
//   warps 0-7  "row" warps: thread (row = tid & 127, half = tid >> 7) owns TMEM lane `row` and one half of the
//              columns of the accumulator; they weight the rows of x and update the state;
//   warp 8     one lane issues every tcgen05.mma (the issuing lane is held about as long as the products take,
//              so it does nothing else);
//   warp 9     one lane issues every TMA load and store.
// The forward itself is fwd_walk_kernel (ssd_tc_fwd.cuh), the reverse walk of the backward rev_walk_kernel
// (ssd_tc_revwalk.cuh).
//
// mbarriers (phase = tile parity unless noted):
//   bar_ld[s]  TMA bytes of stage s landed                        (phase = (tile / NST) & 1)
//   bar_u      weighted rows written, one arrival per warp         (row warps -> products)
//   bar_m2     Hl of the tile has completed                       (products -> row warps, TMA lane: stage free)
//   bar_h      accumulator read, new state written, one per warp  (row warps -> products, TMA lane)
//   bar_sr     the store of the tile before has read sH           (TMA lane -> products)
#pragma once

namespace ssd {
namespace tc {

// Write 32 fp32 values as bf16 into chunks [chunk0, chunk0+4) of this row of a swizzled panel.
__device__ __forceinline__ void store_half_row(uint8_t* panel, int row, int chunk0, const float (&v)[32]) {
#pragma unroll
    for (int ch = 0; ch < 4; ++ch) {
        uint4 o;
        o.x = pack_bf16(v[ch * 8 + 0], v[ch * 8 + 1]);
        o.y = pack_bf16(v[ch * 8 + 2], v[ch * 8 + 3]);
        o.z = pack_bf16(v[ch * 8 + 4], v[ch * 8 + 5]);
        o.w = pack_bf16(v[ch * 8 + 6], v[ch * 8 + 7]);
        *reinterpret_cast<uint4*>(panel + sw128(row, chunk0 + ch)) = o;
    }
}

// N values p0 .. p0+N-1 of row n of a (b,h,p,n) fp32 state, n and p below the tile's 128 x 64: what lies beyond the state's own
// size reads as zero and is not written.
template <int N>
__device__ __forceinline__ void load_state_row(const float* base, size_t bh, int p, int n, int row, int p0, float (&H)[N]) {
    const float* s = base ? base + bh * (size_t)p * n + (size_t)p0 * n + row : nullptr;
    if (s && p == HP && row < n) {
#pragma unroll
        for (int q = 0; q < N; ++q) H[q] = s[(size_t)q * n];
    } else {
#pragma unroll
        for (int q = 0; q < N; ++q) H[q] = (s && row < n && p0 + q < p) ? s[(size_t)q * n] : 0.f;
    }
}
// The same for the state entering this block's piece of a walk: the seed carried through the pieces before it (reverse walk:
// the state gradient leaving the piece, through the pieces behind it; the entries start with piece 1).
template <bool REV, int N>
__device__ __forceinline__ void load_piece_row(const WalkParams& P, size_t bh, int row, int p0, float (&H)[N]) {
    load_state_row(P.seed, bh, P.p, P.n, row, p0, H);
    const size_t nbh = (size_t)gridDim.y * P.h;
    const int passed = P.parts * (int)(REV ? gridDim.z - 1 - blockIdx.z : blockIdx.z), all = P.parts * (int)(gridDim.z - 1);
    for (int i = 0; i < passed; ++i) {
        const int j = REV ? all - 1 - i : i;
        const float dec = expf(P.piece_decay[j * nbh + bh]);
        float v[N];
        load_state_row(P.piece_sum, j * nbh + bh, P.p, P.n, row, p0, v);
#pragma unroll
        for (int q = 0; q < N; ++q) H[q] = fmaf(dec, H[q], v[q]);
    }
}
template <int N>
__device__ __forceinline__ void store_state_row(float* base, size_t bh, int p, int n, int row, int p0, const float (&H)[N]) {
    if (!base || row >= n) return;
    float* o = base + bh * (size_t)p * n + (size_t)p0 * n + row;
#pragma unroll
    for (int q = 0; q < N; ++q)
        if (p == HP || p0 + q < p) o[(size_t)q * n] = H[q];
}

struct WalkCfg {
    static constexpr int NST = 3;                      // load stages
    static constexpr uint32_t STAGE_BYTES = 3 * PANEL;  // V panels 0,1 | U
    static constexpr size_t SMEM = (size_t)NST * STAGE_BYTES + 2 * PANEL + 1024;  // stages | sUd | sH | alignment slack
};

constexpr int kWalkThreads = 320;  // 8 row warps, the product-issue warp, the TMA warp

__global__ void __launch_bounds__(kWalkThreads, 1) states_walk_kernel(const __grid_constant__ WalkParams P) {
    dep_wait();
    using Cfg = WalkCfg;
    constexpr int NST = Cfg::NST;
    extern __shared__ uint8_t smem_raw[];
    // 1024-byte alignment by an offset on the __shared__ array itself, so that every access below stays a
    // shared-memory instruction (a pointer rebuilt from an integer would be a generic-address access)
    uint8_t* sm = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* sStage = sm;                                  // per stage: V panels 0,1 | U
    uint8_t* sUd = sStage + (size_t)NST * Cfg::STAGE_BYTES;  // weighted copy of U
    uint8_t* sH = sUd + PANEL;                             // state, bf16, [n][p]
    __shared__ uint64_t bar_ld[3], bar_u, bar_m2, bar_h, bar_sr;
    __shared__ uint32_t tmem_slot;
    __shared__ int alive;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int hh = blockIdx.x, bb = blockIdx.y;
    const int gg = hh / P.hpg;
    const size_t bh = (size_t)bb * P.h + hh;
    const int k0 = blockIdx.z * P.pt, nt = min(P.pt, P.nt - k0);  // the piece's tiles

    if (tid == 0) {
        alive = 1;
        for (int s = 0; s < NST; ++s) mbar_init(&bar_ld[s], 1);
        mbar_init(&bar_u, 8);
        mbar_init(&bar_m2, 1);
        mbar_init(&bar_h, 8);
        mbar_init(&bar_sr, 1);
        mbar_fence_init();
    }
    if (warp == 8) {
        tmem_alloc(&tmem_slot, 64);
        tmem_relinquish();
    }
    const int row = tid & 127, hf = (tid >> 7) & 1;
    // state row of this thread: n = row, p in [hf*32, hf*32+32)
    float H[32];
    if (warp < 8) {
        load_piece_row<false>(P, bh, row, hf * 32, H);
        store_half_row(sH, row, hf * 4, H);
        fence_async_smem();
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tHl = tmem_slot;
    auto state_row = [&](int it) {  // row of tile `it` of this walk in the [b*nt*h*128][64] state tensor
        return (int)((((size_t)bb * P.nt + k0 + it) * P.h + hh) * DN);
    };
    if (warp == 8) {
        // ------------------------------------------------------------------ product lane
        if (lane == 0) {
            const uint32_t udMN = desc_lo(smem_u32(sUd), PANEL), stMN = desc_lo(smem_u32(sStage), PANEL);
            constexpr uint32_t SU = Cfg::STAGE_BYTES >> 4;  // stage pitch in 16-byte units
            for (int it = 0; it < nt; ++it) {
                const uint32_t ph = it & 1;
                const uint32_t vMN = stMN + (uint32_t)(it % NST) * SU;
                mbar_wait(&bar_ld[it % NST], (it / NST) & 1, &alive);
                if (it > 0) mbar_wait_spin(&bar_h, (it - 1) & 1, &alive);  // accumulator read
                mbar_wait_spin(&bar_u, ph, &alive);
                tc_fence_after();
#pragma unroll
                for (int kk = 0; kk < 8; ++kk)  // Hl = V^T Ud : both MN-major, K = position
                    mma_ss_lo(tHl, vMN + kk * 128, udMN + kk * 128, kIdescMM, kk > 0);
                // the rows rewrite sH after bar_m2: the store of the tile before must have read it
                mbar_wait_spin(&bar_sr, ph, &alive);
                mma_commit(&bar_m2);
            }
        }
        __syncwarp();
    } else if (warp == 9) {
        // ------------------------------------------------------------------ TMA lane
        if (lane == 0) {
            prefetch_tmap(&P.mU);
            prefetch_tmap(&P.mV);
            auto issue_loads = [&](int it) {
                const int s = it % NST;
                uint8_t* st = sStage + (size_t)s * Cfg::STAGE_BYTES;
                mbar_expect_tx(&bar_ld[s], Cfg::STAGE_BYTES);
                const int pos = (k0 + it) * LT;
                tma_load_4d(st, &P.mV, &bar_ld[s], 0, gg, pos, bb);
                tma_load_4d(st + PANEL, &P.mV, &bar_ld[s], 64, gg, pos, bb);
                tma_load_4d(st + 2 * PANEL, &P.mU, &bar_ld[s], 0, hh, pos, bb);
            };
            for (int it = 0; it < NST - 1 && it < nt; ++it) issue_loads(it);
            tma_store_2d(&P.mS, sH, 0, state_row(0));  // the seed is the state entering the first tile
            tma_store_commit();
            for (int it = 0; it < nt; ++it) {
                if (it + NST - 1 < nt) {
                    // the stage of tile it-1 is free once the product of that tile has completed
                    if (it > 0) mbar_wait(&bar_m2, (it - 1) & 1, &alive);
                    issue_loads(it + NST - 1);
                }
                if (it > 0) {
                    mbar_wait_spin(&bar_h, (it - 1) & 1, &alive);  // new state in sH
                    tma_store_2d(&P.mS, sH, 0, state_row(it));
                    tma_store_commit();
                }
                tma_store_wait_read();
                mbar_arrive(&bar_sr);  // sH may be rewritten
            }
            tma_store_wait_all();
        }
        __syncwarp();
    } else {
        // ------------------------------------------------------------------ row warps
        const float* tcum = P.tcum + bh * P.Tp + (size_t)k0 * LT;
        const float* dtT = P.dtT ? P.dtT + bh * P.Tp + (size_t)k0 * LT : nullptr;
        const uint32_t lanes = lane_base(warp);
        // per-tile scalars are fetched one tile ahead
        float c_n = tcum[row], S_n = tcum[LT - 1];
        float dt_n = dtT ? dtT[row] : 1.f;
        for (int it = 0; it < nt; ++it) {
            const int s = it % NST;
            const uint32_t ph = it & 1;
            const float c_i = c_n, dtv = dt_n, Sk = S_n;
            if (it + 1 < nt) {
                const size_t o = (size_t)(it + 1) * LT;
                c_n = tcum[o + row];
                S_n = tcum[o + LT - 1];
                dt_n = dtT ? dtT[o + row] : 1.f;
            }
            mbar_wait(&bar_ld[s], (it / NST) & 1, &alive);
            {
                // (sUd is free: this thread waited for the product of the tile before, its only reader, before the state update)
                // this thread's half row of U, weighted by d_j dt_j as a bf16 pair (one packed multiply per two elements)
                const uint8_t* sU = sStage + (size_t)s * Cfg::STAGE_BYTES + 2 * PANEL;
                const __nv_bfloat162 w2 = __float2bfloat162_rn(exp2f(Sk - c_i) * dtv);
#pragma unroll
                for (int ch = 0; ch < 4; ++ch) {
                    uint4 v = *reinterpret_cast<const uint4*>(sU + sw128(row, hf * 4 + ch));
                    uint32_t* u = reinterpret_cast<uint32_t*>(&v);
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        __nv_bfloat162 r = __hmul2(*reinterpret_cast<__nv_bfloat162*>(&u[q]), w2);
                        u[q] = *reinterpret_cast<uint32_t*>(&r);
                    }
                    *reinterpret_cast<uint4*>(sUd + sw128(row, hf * 4 + ch)) = v;
                }
            }
            fence_async_smem();
            mbar_arrive_warp(&bar_u);
            mbar_wait(&bar_m2, ph, &alive);
            tc_fence_after();
            {
                uint32_t r[32];
                tmem_ld32(tHl + lanes + hf * 32, r);
                const float dec = exp2f(Sk);
                tmem_ld_wait();
#pragma unroll
                for (int q = 0; q < 16; ++q) {
                    float2* H2 = reinterpret_cast<float2*>(H);
                    H2[q] = fma2(make_float2(dec, dec), H2[q], reinterpret_cast<const float2*>(r)[q]);
                }
                store_half_row(sH, row, hf * 4, H);
            }
            tc_fence_before();
            fence_async_smem();
            mbar_arrive_warp(&bar_h);
        }
        if (k0 + nt == P.nt) store_state_row(P.out_state, bh, P.p, P.n, row, hf * 32, H);
    }
    tc_fence_before();
    __syncthreads();
    end_of_waits(&alive, P.status);
    if (warp == 8) tmem_dealloc(tHl, 64);
}

}  // namespace tc
}  // namespace ssd
