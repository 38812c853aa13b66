// Tensor-core path of the SSD chunked scan for sm_100a: tcgen05.mma with TMEM accumulators,
// operands staged in 128-byte-swizzled shared memory by TMA (no cluster multicast).
//
// Covered shapes: bf16 storage, headdim up to 64, d_state up to 128 (see supported()), sequences and chunks of any
// length; chosen without being asked for where these fill whole tiles (whole_tiles()).  The kernels work on tiles of 128
// positions whatever the chunk size (the recurrence does not depend on where chunk boundaries fall); `tcum` is the inclusive
// cumulative log-decay inside each 128-tile.
//
// Kernels
//   tile_cumsum_kernel  a_cumsum (b,h,c,l) -> tcum (b,h,T), dt (b,T,h) -> dtT (b,h,T)
//   cumsum_tile_fused_kernel  the same together with the cumulative sums themselves
//   fwd_walk_kernel     one CTA per (batch, head) walks the tiles with the state (64 x 128 fp32) in registers:
//                       Y = ((C B^T) o L) X + diag(e) C H^T (+ D x);  H <- e^{S} H + X^T diag(d) B
//   states_walk_kernel  only the recurrence; stores H_k (state entering tile k) as bf16
//   summary_kernel      what a whole piece of the sequence adds to the state after it / to the state gradient
//                       before it (the quantities the sequence-parallel schedule exchanges): a stream, no recurrence
//   rev_walk_kernel     reverse walk of the backward pass, Q <- e^{S} Q + dY^T diag(e) C, software-pipelined
//                       over tiles; reads dY and C only, stores Q_k = dH_{k+1} as bf16
//   bwd_tile_kernel     persistent over (batch, tile, group) items, heads of the group in an inner loop so
//                       that dB and dC accumulate over heads in TMEM:
//        dG = dY X^T, dS = dG o L, dX = G^T dY + diag(d) B Q^T, dC += dS B + diag(e) dY H,
//        dB += dS^T C + diag(d) X Q, and the per-position decay-gradient terms.
//
// TMEM lane = tile row (tcgen05.ld 32x32b); the epilogues are the work of row warps, two or four threads to a row.  Products and TMA copies are issued by
// one lane each of other warps: products that wait for different things by different ones (fwd_walk_kernel, bwd_tile_kernel).
#pragma once
#include "ssd_common.cuh"
#include "ssd_cumsum.cuh"
#include "ssd_ptx.cuh"

namespace ssd {
namespace tc {

using namespace ssd::ptx;
using namespace ssd::cum;

constexpr int HP = 64;   // headdim
constexpr int DN = 128;  // d_state
constexpr int PANEL = 16384;  // bytes of one [128 rows][64 bf16] swizzled panel
// What the kernels can run: shapes below the tile's own size are padded on chip, TMA fills what lies behind the end of a
// sequence, or behind a head's last column, with zeros, and does not write it.  (A row of p or n bf16 values has to be a
// multiple of 16 bytes for that.)
inline bool supported(int dtype, int p, int n) {
    return dtype == 1 && p > HP / 2 && p <= HP && p % 8 == 0 && n > DN / 4 && n <= DN && n % 8 == 0;
}
// What they are chosen for.  Operands of the products (the masked scores, the weighted x, the states a tile starts from) are
// rounded to bf16 here and are fp32 in the kernels of ssd_mma.cuh and ssd_simt.cuh.  Calls that fill whole tiles take that rounding;
// for others it is the caller's choice (SSD_B200_PATH_TC): the final state of 320 positions in chunks of 80 is 2.4e-3 off
// the exact one on these kernels, 2.5e-7 in fp32 (and forward + backward of (4, 1984, 20 heads, 64), d_state 64, chunk 64
// take 125 us here, 303 us there).
inline bool whole_tiles(int T, int p, int n, int l) { return p == HP && n == DN && T % LT == 0 && (l % LT == 0 || LT % l == 0); }
inline int tiles_of(int T) { return (T + LT - 1) / LT; }

// ------------------------------------------------------------------------------------------
// Decay gradient of the tensor-core backward, one block per (128-tile, eight heads, batch): a head a warp and 32 registers.  (Blocks
// of 32 heads, four a warp, need 128: 18.5 us against 14.4 for 384 of them, 27.5 / 20.8 at (16, 4096, 64 heads), 176 / 145 at (4, 131072, 64).)
// Inputs in (b,h,T) layout (coalesced along t): the per-row gradients g w.r.t. the tile-cumulative
// log-decay, ddtx = sum_p dX x, dyx = sum_p dy x, and gS, the terms that act through the tile's last row.  Within a tile
//   dA[t] = sum_{t' >= t} g[t']      (a suffix sum, four 32-lane segments per warp and head)
// and  ddt = ddtx + dA A_head,  dA_head += dA dt,  dD += dyx.  dt is read and ddt / da written in the
// caller's (b,T,h) layout through a shared-memory transpose, so both sides are 128-byte rows.
struct DecayTileParams {
    const float* g;      // (b,h,T)
    const float* ddtx;   // (b,h,T)
    const float* dyx;    // (b,h,T) or null
    const float* gS;     // (b,h,nt,8) from the backward tile kernel: terms that act through the tile's last row
    const float* dt;     // (b,T,h) or null (operator form)
    const float* A_head; // (h) or null; null with dt given = scaled operator form (outputs ddt = ddtx, da, dskip = dyx)
    float* ddt;          // (b,T,h) or null
    float* da;           // (b,T,h) or null
    float* dskip;        // (b,T,h) or null (scaled operator form)
    float* dAh_part;     // (b*nt, h)
    float* dD_part;      // (b*nt, h) or null
    int b, T, Tp, h, nt;  // Tp = nt * 128: stride of g, ddtx and dyx
};

__global__ void __launch_bounds__(256) decay_tile_kernel(DecayTileParams P) {
    dep_wait();
    constexpr int HB = 8, R = 256 / HB;  // heads of a block, rows that its threads move at a time
    __shared__ float sdt[LT][HB + 1];
    __shared__ float sout[LT][HB + 1];
    const int k = blockIdx.x, bb = blockIdx.z, h0 = blockIdx.y * HB;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rl = threadIdx.x / HB, hcol = threadIdx.x % HB;
    const bool col_ok = h0 + hcol < P.h;
    const int rows = min(LT, P.T - k * LT);
    if (P.dt) {
#pragma unroll
        for (int t = rl; t < LT; t += R)
            sdt[t][hcol] = (col_ok && t < rows) ? P.dt[((size_t)bb * P.T + (size_t)k * LT + t) * P.h + h0 + hcol] : 0.f;
    }
    // every load of the warp's head is issued before any of them is used
    const bool scaled = P.dt && !P.A_head;  // scaled operator form: three per-position outputs
    const int hh = h0 + warp;
    const bool on = hh < P.h;  // warp-uniform
    float v[4], dxa[4], yxp[4], gs = 0.f;
#pragma unroll
    for (int s4 = 0; s4 < 4; ++s4) v[s4] = dxa[s4] = yxp[s4] = 0.f;
    if (on) {
        const size_t base = ((size_t)bb * P.h + hh) * P.Tp + (size_t)k * LT;
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4) {
            const int t = s4 * 32 + lane;
            v[s4] = P.g[base + t];
            dxa[s4] = P.ddtx[base + t];
            if (P.dyx) yxp[s4] = P.dyx[base + t];
        }
        if (lane < 8)  // the eight terms that act through the tile's last row, one per lane
            gs = P.gS[((((size_t)bb * P.h + hh) * P.nt) + k) * 8 + lane];
    }
    __syncthreads();
    if (on) {
        // fixed-order sum of the eight terms (the other lanes hold zero), result in every lane
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) gs += __shfl_xor_sync(0xffffffffu, gs, o);
        if (lane == 31) v[3] += gs;
        // suffix sums: inside each 32-lane segment by shuffles, then the totals of the later segments
        float tot[4];
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4) {
            float incl = v[s4];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const float u = __shfl_down_sync(0xffffffffu, incl, o);
                if (lane + o < 32) incl += u;
            }
            v[s4] = incl;
            tot[s4] = __shfl_sync(0xffffffffu, incl, 0);
        }
        v[2] += tot[3];
        v[1] += tot[3] + tot[2];
        v[0] += (tot[3] + tot[2]) + tot[1];  // v: d a[t] of this head and tile
        if (P.dt && !scaled) {
            float dAh = 0.f, yx = 0.f;
#pragma unroll
            for (int s4 = 0; s4 < 4; ++s4) {
                dAh += v[s4] * sdt[s4 * 32 + lane][warp];
                yx += yxp[s4];
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                dAh += __shfl_xor_sync(0xffffffffu, dAh, o);
                yx += __shfl_xor_sync(0xffffffffu, yx, o);
            }
            if (lane == 0) {
                const size_t po = ((size_t)bb * P.nt + k) * P.h + hh;
                P.dAh_part[po] = dAh;
                if (P.dD_part) P.dD_part[po] = yx;
            }
        }
    }
    // per-position outputs in the caller's (b,T,h) layout, one transpose through shared memory each:
    //   Mamba-2 form: ddt = ddtx + da A_head;  operator form: da;  scaled operator form: ddt = ddtx, da, dskip = dyx
    for (int pass = 0; pass < 3; ++pass) {
        float* out = nullptr;
        if (pass == 0) out = P.dt ? P.ddt : P.da;
        else if (pass == 1) out = scaled ? P.da : nullptr;
        else out = scaled ? P.dskip : nullptr;
        if (!out) continue;  // block-uniform
        __syncthreads();
        if (on) {
            const float Ah = (P.A_head && pass == 0) ? P.A_head[hh] : 0.f;
#pragma unroll
            for (int s4 = 0; s4 < 4; ++s4) {
                float val;
                if (pass == 0) val = P.dt ? dxa[s4] + v[s4] * Ah : v[s4];
                else if (pass == 1) val = v[s4];
                else val = yxp[s4];
                sout[s4 * 32 + lane][warp] = val;
            }
        }
        __syncthreads();
        if (col_ok) {
#pragma unroll
            for (int t = rl; t < rows; t += R) out[((size_t)bb * P.T + (size_t)k * LT + t) * P.h + h0 + hcol] = sout[t][hcol];
        }
    }
}

// out[hh] = sum_r part[r, hh] over `rows` rows, one block per head, fixed summation tree (deterministic).
// A second (part, out) pair, when given, is reduced by the blocks with blockIdx.y = 1 of the same launch.
__global__ void __launch_bounds__(256) reduce_rows_kernel(const float* __restrict__ part, float* __restrict__ out, int rows, int h,
                                                          const float* __restrict__ part2 = nullptr, float* __restrict__ out2 = nullptr) {
    dep_wait();
    __shared__ float red[8];
    const int hh = blockIdx.x;
    if (blockIdx.y) {
        part = part2;
        out = out2;
    }
    float s = 0.f;
    for (int r = threadIdx.x; r < rows; r += 256) s += part[(size_t)r * h + hh];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) out[hh] = ((red[0] + red[1]) + (red[2] + red[3])) + ((red[4] + red[5]) + (red[6] + red[7]));
}

// ------------------------------------------------------------------------------------------
// Self-test of the bounded wait: one warp waits (a few thousand polls) on an mbarrier that nothing ever arrives at,
// gives up, records it in the status word exactly as the tile kernels do, and returns.  The context stays usable.
__global__ void __launch_bounds__(32) bounded_wait_selftest_kernel(int* status, int polls) {
    __shared__ uint64_t bar;
    __shared__ int alive;
    if (threadIdx.x == 0) {
        alive = 1;
        mbar_init(&bar, 1);
        mbar_fence_init();
    }
    __syncwarp();
    mbar_wait(&bar, 0, &alive, (uint32_t)polls);
    __syncwarp();
    if (threadIdx.x == 0 && gave_up(&alive)) atomicExch(status, 1);
}

// ------------------------------------------------------------------------------------------
// Walks whose pieces find their own way (forward): the first `whole` (batch, head) pairs are walked whole, a CTA each, the others by np CTAs, of which CTA z
// walks the states of the tiles before cut[z] for itself, without their output (0.8 us a tile instead of 1.5), and then the tiles [cut[z], cut[z + 1]).
// Every state is made as a whole walk makes it, so the results have its bits.
struct SelfCut {
    int whole, np;
    int cut[5];
};
struct WalkParams {
    CUtensorMap mU;   // x, or dy (reverse walks): (b,T,h,p)
    CUtensorMap mV;   // B, or C (reverse walks): (b,T,g,n)
    CUtensorMap mC;   // C (forward)
    const float* tcum;
    const float* dtT;
    const float* D;
    const float* skipT;  // (b,h,T) per-position skip coefficient (replaces D), or null
    const float* seed;   // init (modes 0,1) or dfinal (reverse walks), (b,h,p,n) fp32, may be null
    float* out_state;    // final_state (modes 0,1) or dinit (reverse walks), may be null
    CUtensorMap mY;   // y store (mode 0)
    CUtensorMap mS;   // state store: 2D [b*nt*h*128][64]
    int save_states;  // store the state entering every tile of the walk through mS
    float* ysq;          // (b, T/128, h, 2, 128) per half row sum_p y^2 (forward only), or null
    int* status;
    int zero_status;     // this kernel is the pass's first: it clears the status word
    int Tp, h, hpg, nt;  // Tp = nt * 128: stride of the per-position arrays
    int p, n;            // headdim and d_state of the tensors (at most 64 and 128)
    // Pieces of the sequence (blockIdx.z; see Pieces): tiles of a piece, and what the parts of each piece but the last
    // (reverse walk: but the first) add to the state behind them (to the gradient of the state before them), (piece, part,
    // b, h, p, n), with their total log-decay (piece, part, b, h), from summary_kernel.
    int pt, parts;
    const float* piece_sum;
    const float* piece_decay;
    SelfCut self;  // forward walk, np > 1: one-dimensional grid
};

constexpr uint32_t kIdescKM = instr_desc(128, 64, false, true);     // A K-major, B MN-major, N = 64
constexpr uint32_t kIdescMM = instr_desc(128, 64, true, true);      // both MN-major, N = 64
constexpr uint32_t kIdescKK128 = instr_desc(128, 128, false, false); // K-major x K-major, N = 128
constexpr uint32_t kIdescKM128 = instr_desc(128, 128, false, true);  // A K-major, B MN-major, N = 128
constexpr uint32_t kIdescMM128 = instr_desc(128, 128, true, true);   // both MN-major, N = 128

__device__ __forceinline__ uint32_t lane_base(int warp) { return ((uint32_t)((warp & 3) * 32)) << 16; }

}  // namespace tc
}  // namespace ssd
#include "ssd_tc_walk.cuh"
#include "ssd_tc_fwd.cuh"
#include "ssd_tc_revwalk.cuh"
#include "ssd_tc_summary.cuh"
#include "ssd_tc_bwd.cuh"
