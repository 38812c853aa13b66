// Cumulative log-decays: within the caller's chunks (an output of the operator) and within the 128-position tiles
// the tensor-core kernels work on.
#pragma once
#include "ssd_common.cuh"

namespace ssd {
namespace cum {

constexpr int LT = 128;  // tile length

// The decay mask of a 32-column block is the product of a per-row and a per-column factor taken relative to the
// block's last column.  Below the diagonal both are <= 1.  Inside the diagonal block the row factor would be
// 2^(decay from the row to the block end) >= 1 and the column factor its inverse scale; beyond this many log2
// units across a block one of them would leave the fp32 range.  The forward evaluates diagonal blocks entry by entry (one exp2 per
// entry); the backward, which is 2 % slower that way, does where the flags of the kernels below, one word per block, ask for it.
constexpr float kMaskSafeLog2 = 100.f;
// Heads to a block of cumsum_tile_fused_kernel: 32, whose reads are whole 128-byte rows, or eight, a quarter of the loads and one head a warp instead of four, where
// blocks of eight are few (nine to an SM) or blocks of 32 are half empty (cumsum_blocks_of_eight).  Blocks of 32 / of eight, us, each after a
// write of 256 MB: 4 blocks of 32 heads, 24 of them heads, 8.2 / 6.4; 256, all heads, 10.2 / 10.3; 384 12.3 / 12.3; 512 14.3 / 14.4; 1024 18.4 / 22.5; 1024 with
// 8 heads each 14.4 / 10.2, with 16 14.6 / 14.4, with 24 17.4 / 17.8; log-decays given in bf16: 256, all heads, 12.3 / 10.2, 1024 20.5 / 22.5.
constexpr int kFewCumsumBlocks = 9 * 148;
constexpr int kFusedChunkMax = 1024;  // see cumsum_tile_fused_kernel

// The block's words of the flags (one per tile and eight heads; null: not wanted), from the threads' own; every thread of the block calls this.
template <int HB>
__device__ __forceinline__ void raise_flag(int* extreme, int beyond, int h) {
    if (!extreme) return;
    const int any = __syncthreads_or(beyond), words = (h + 7) / 8, w = blockIdx.y * (HB / 8) + threadIdx.x;
    if (threadIdx.x < HB / 8 && w < words) extreme[((size_t)blockIdx.z * words + w) * gridDim.x + blockIdx.x] = any;
}

// The first block of a pass clears the status word (a memset of its own is a gap of 1.2 us and more on the stream, and what follows one is not
// launched early).  What may be written there in the same kernel: what a block finds wrong at its start, which every block does and so this one too, behind its
// clearing; and that a bounded wait ran out, a tenth of a second later.
__device__ __forceinline__ void clear_status(int* status) {
    if (threadIdx.x == 0 && blockIdx.x == 0 && blockIdx.y == 0 && blockIdx.z == 0) *status = 0;
}

// ------------------------------------------------------------------------------------------
// Per-position arrays of the tile kernels from a given a_cumsum: the tile-cumulative log2 decay, dt and the skip coefficient in
// (b,h,Tp) order, Tp = T rounded up to whole tiles (behind the end of the sequence the decay stays at its last value and
// dt and skip are zero).  One block per (tile, eight heads, batch), a head a warp: dt arrives in the caller's (b,T,h) order and goes
// through a shared-memory transpose: reads of 32 bytes, writes of 128-byte rows.  (Blocks of 32 heads, four a warp, behind a call on the same inputs with chunks
// of 64: 12.4 us against 4.0 at (8, 2048, 32 heads), 23.5 / 15.7 at (16, 4096, 64), 59 / 55 at (4, 65536, 64), 105 / 108 at (4, 131072, 64).)  Chunks of any length: the cumulative
// decay from the tile's start is a difference inside the tile's first chunk plus the totals of the chunks that end in
// the tile.
__global__ void __launch_bounds__(256) tile_cumsum_kernel(const float* __restrict__ cum, const float* __restrict__ dt,
                                                          float* __restrict__ tcum, float* __restrict__ dtT,
                                                          const float* __restrict__ skip, float* __restrict__ skipT,
                                                          int* __restrict__ extreme, int* __restrict__ status, int T, int Tp, int h, int l) {
    dep_wait();
    clear_status(status);
    int beyond = 0;
    constexpr int HB = 8, R = 256 / HB;  // heads of a block, rows that its threads read at a time
    __shared__ float sdt[LT][HB + 1];
    __shared__ float ssk[LT][HB + 1];
    const int kt = blockIdx.x, h0 = blockIdx.y * HB, bb = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int rl = threadIdx.x / HB, hcol = threadIdx.x % HB;
    const int t0 = kt * LT, rows = min(LT, T - t0);
    const bool col_ok = h0 + hcol < h;
    if (dt) {
#pragma unroll
        for (int t = rl; t < LT; t += R)
            sdt[t][hcol] = (col_ok && t < rows) ? dt[((size_t)bb * T + t0 + t) * h + h0 + hcol] : 0.f;
    }
    if (skip) {  // per-position skip coefficient of the scaled operator form, same transpose
#pragma unroll
        for (int t = rl; t < LT; t += R)
            ssk[t][hcol] = (col_ok && t < rows) ? skip[((size_t)bb * T + t0 + t) * h + h0 + hcol] : 0.f;
    }
    __syncthreads();
    const int hh = h0 + warp;
    if (hh < h) {  // warp-uniform
        const int k0 = t0 / l, i0 = t0 - k0 * l;  // chunk of the tile's first position, position in it
        const bool one = i0 + rows <= l;           // the whole tile lies in that chunk
        const float* cu = cum + ((size_t)bb * h + hh) * T;  // (b,h,c,l): position t of the sequence at t
        const float before = i0 > 0 ? cu[t0 - 1] : 0.f;
        float v[4];
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4) v[s4] = cu[t0 + min(s4 * 32 + lane, rows - 1)];
        const size_t o = ((size_t)bb * h + hh) * Tp + t0;
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4) {
            const int tt = s4 * 32 + lane;
            float w = v[s4] - before;
            if (!one) {
                const int k = (t0 + min(tt, rows - 1)) / l;
                if (k != k0) {
                    w = v[s4] + (cu[(size_t)(k0 + 1) * l - 1] - before);
                    for (int kk = k0 + 1; kk < k; ++kk) w += cu[(size_t)(kk + 1) * l - 1];
                }
            }
            w *= 1.4426950408889634f;  // stored in log2 units: every consumer uses exp2
            tcum[o + tt] = w;
            // decay across this 32-position block (lane 0 to lane 31)
            const float span = __shfl_sync(0xffffffffu, w, 0) - __shfl_sync(0xffffffffu, w, 31);
            if (!(span <= kMaskSafeLog2)) beyond = 1;
            if (dtT) dtT[o + tt] = sdt[tt][warp];
            if (skipT) skipT[o + tt] = ssk[tt][warp];
        }
    }
    raise_flag<HB>(extreme, beyond, h);
}

// ------------------------------------------------------------------------------------------
// A thread's values of every `step`-th row, zeros from row `rows` on: a loop of its own, so that every load is issued before a value is used.  (Left to the
// compiler in one loop with the stores to shared memory, the loads went out one after the other or all at once as the rest of the kernel had it: 104 us or 123 at
// (4, 131072, 64 heads), 94 so.)
template <int N, class TV>
__device__ __forceinline__ void load_column(float (&v)[N], const TV* p, int step, int rows, int h) {
#pragma unroll
    for (int q = 0; q < N; ++q) v[q] = q * step < rows ? to_f(p[(size_t)q * step * h]) : 0.f;
}

// The same from the per-position log-decay itself (dt * A_head, or `a` as given, fp32 or bf16), which is read once in the
// caller's (b,T,h) layout through a shared-memory transpose and scanned inside each tile (warp per head, 32-lane segments
// scanned side by side); also writes a_cumsum (b,h,c,l) in natural-log units, where one is wanted (a backward without
// kept states runs this too, so that its per-position arrays have the forward's bits).  Chunks of any length: where one
// ends inside the tile its sums come from a second, segmented scan of the same values (CUT), so that they carry no
// rounding of the positions before the chunk; where a chunk began in an earlier tile, the block adds up the positions
// between (kFusedChunkMax bounds that second read, at most the chunk, against a launch and a pass over a_cumsum for the two
// kernels this replaces: 28 -> 7 us at (8, 2048, 24) with chunks of 64).  The skip array is transposed in a second round
// through the panel of the log-decay.
// HB heads to a block: see kFewCumsumBlocks.  Registers for five blocks on an SM, four with CUT: with six the loads no longer fit at once (92 -> 102 us at
// (4, 131072, 64 heads)), with CUT five are 121 us and four 117.
template <bool CUT, int HB>
__global__ void __launch_bounds__(256, CUT ? 4 : 5) cumsum_tile_fused_kernel(const void* __restrict__ a, int a_is_bf16,
                                                                const float* __restrict__ dt, const float* __restrict__ A_head,
                                                                float* __restrict__ cum, float* __restrict__ tcum,
                                                                float* __restrict__ dtT, const float* __restrict__ skip,
                                                                float* __restrict__ skipT, int* __restrict__ extreme,
                                                                int* __restrict__ status, int T, int Tp, int h, int l) {
    dep_wait();
    clear_status(status);
    int beyond = 0;
    constexpr int R = 256 / HB;  // rows that the block's threads read at a time
    __shared__ float sa[LT][HB + 1];
    __shared__ float sdt[LT][HB + 1];
    __shared__ float sbef[8][HB + 1];
    const int kt = blockIdx.x, hg = blockIdx.y, bb = blockIdx.z;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int h0 = hg * HB, rl = threadIdx.x / HB, hcol = threadIdx.x % HB;
    const int t0 = kt * LT, rows = min(LT, T - t0);
    const bool head_ok = h0 + hcol < h;
    const float Ah = (!a && head_ok) ? A_head[h0 + hcol] : 0.f;
    auto given = [&](size_t i) { return a_is_bf16 ? __bfloat162float(((const __nv_bfloat16*)a)[i]) : ((const float*)a)[i]; };
    auto log_decay = [&](size_t i, float d) { return a ? given(i) : d * Ah; };
    const size_t row0 = (size_t)bb * T;
    constexpr int N = LT / R;
    float dv[N], av[N];
    const size_t first = (row0 + t0 + rl) * h + h0 + hcol;
    const int mine = head_ok ? rows - rl : 0;
    if (a) {
        if (a_is_bf16) load_column(av, (const __nv_bfloat16*)a + first, R, mine, h);
        else load_column(av, (const float*)a + first, R, mine, h);
    }
    if (dt) load_column(dv, dt + first, R, mine, h);
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const int t = rl + q * R;
        sa[t][hcol] = a ? av[q] : q * R < mine ? dv[q] * Ah : 0.f;
        if (dt) sdt[t][hcol] = dv[q];
    }
    const int i0 = t0 % l;  // positions of the tile's first chunk that lie in earlier tiles
    if (i0 && rl < 8) {  // (eight sums whatever HB, so that they have the same bits)
        float s = 0.f;
#pragma unroll 8
        for (int t = rl; t < i0; t += 8) {
            const size_t i = (row0 + t0 - i0 + t) * h + h0 + hcol;
            if (head_ok) s += log_decay(i, dt && !a ? dt[i] : 0.f);
        }
        sbef[rl][hcol] = s;
    }
    __syncthreads();
#pragma unroll
    for (int i4 = 0; i4 < HB / 8; ++i4) {
        const int hl = warp * (HB / 8) + i4, hh = h0 + hl;
        if (hh >= h) break;  // warp-uniform
        const size_t o = ((size_t)bb * h + hh) * Tp + t0, oc = ((size_t)bb * h + hh) * T + t0;
        float before = 0.f;
        if (i0) {
#pragma unroll
            for (int w = 0; w < 8; ++w) before += sbef[w][hl];
        }
        float v[LT / 32], c[LT / 32];
#pragma unroll
        for (int s4 = 0; s4 < LT / 32; ++s4) v[s4] = c[s4] = sa[s4 * 32 + lane][hl];
        int pos[LT / 32];  // position inside its chunk
        if (CUT) {
#pragma unroll
            for (int s4 = 0; s4 < LT / 32; ++s4) pos[s4] = (t0 + s4 * 32 + lane) % l;
        }
#pragma unroll
        for (int of = 1; of < 32; of <<= 1) {
#pragma unroll
            for (int s4 = 0; s4 < LT / 32; ++s4) {
                const float u = __shfl_up_sync(0xffffffffu, v[s4], of);
                if (lane >= of) v[s4] += u;
                if (CUT) {
                    const float w = __shfl_up_sync(0xffffffffu, c[s4], of);
                    if (lane >= of && pos[s4] >= of) c[s4] += w;
                }
            }
        }
        float run = 0.f, runc = before;
#pragma unroll
        for (int s4 = 0; s4 < LT / 32; ++s4) {
            const int tt = s4 * 32 + lane;
            v[s4] += run;
            run = __shfl_sync(0xffffffffu, v[s4], 31);
            if (CUT) {
                if (pos[s4] > lane) c[s4] += runc;  // the chunk began before this segment
                runc = __shfl_sync(0xffffffffu, c[s4], 31);
            } else {
                c[s4] = v[s4] + before;
            }
            if (cum && tt < rows) cum[oc + tt] = c[s4];
            const float w = v[s4] * 1.4426950408889634f;
            tcum[o + tt] = w;
            const float span = __shfl_sync(0xffffffffu, w, 0) - __shfl_sync(0xffffffffu, w, 31);
            if (!(span <= kMaskSafeLog2)) beyond = 1;
            if (dtT) dtT[o + tt] = sdt[tt][hl];
        }
    }
    if (skip) {
        __syncthreads();
#pragma unroll
        for (int t = rl; t < LT; t += R)
            sa[t][hcol] = (head_ok && t < rows) ? skip[(row0 + t0 + t) * h + h0 + hcol] : 0.f;
        __syncthreads();
#pragma unroll
        for (int i4 = 0; i4 < HB / 8; ++i4) {
            const int hl = warp * (HB / 8) + i4, hh = h0 + hl;
            if (hh >= h) break;
            const size_t o = ((size_t)bb * h + hh) * Tp + t0;
#pragma unroll
            for (int s4 = 0; s4 < LT / 32; ++s4) skipT[o + s4 * 32 + lane] = sa[s4 * 32 + lane][hl];
        }
    }
    raise_flag<HB>(extreme, beyond, h);
}

// ------------------------------------------------------------------------------------------
// Chunk cumsum: a (b,T,h) -> cum (b,h,c,l), inclusive within each chunk.  One block per
// (chunk, batch); the [l][h] tile is staged through shared memory so that both the strided
// read (h contiguous) and the transposed write (l contiguous) are coalesced; each warp scans
// one head at a time with warp shuffles.  (SIMT path, and chunks beyond kFusedChunkMax.)
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) chunk_cumsum_kernel(const void* __restrict__ a, int a_is_bf16, const float* __restrict__ dt,
                                                           const float* __restrict__ A_head, float* __restrict__ cum, int T, int h, int l) {
    dep_wait();
    extern __shared__ float sm[];
    const int k = blockIdx.x, bb = blockIdx.y;
    const int ldh = h + 1;
    for (int idx = threadIdx.x; idx < l * h; idx += 256) {
        const int i = idx / h, hh = idx - i * h;
        const size_t o = ((size_t)bb * T + (size_t)k * l + i) * h + hh;
        sm[i * ldh + hh] = !a ? dt[o] * A_head[hh] : a_is_bf16 ? __bfloat162float(((const __nv_bfloat16*)a)[o]) : ((const float*)a)[o];
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // lane <-> position inside a 32-position segment (coalesced stores); segments in sequence with a running carry
    for (int hh = warp; hh < h; hh += 8) {
        float* out = cum + ((size_t)bb * h + hh) * T + (size_t)k * l;
        float carry = 0.f;
        for (int i0 = 0; i0 < l; i0 += 32) {
            const int i = i0 + lane;
            float incl = i < l ? sm[i * ldh + hh] : 0.f;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                float v = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += v;
            }
            incl += carry;
            if (i < l) out[i] = incl;
            carry = __shfl_sync(0xffffffffu, incl, 31);
        }
    }
}

// Total log-decay of every (batch, head) sequence from the within-chunk cumulative sums: sum of the chunks' last entries.
__global__ void logdecay_total_kernel(const float* __restrict__ cum, float* __restrict__ out, int bh, int c, int l) {
    dep_wait();
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= bh) return;
    float s = 0.f;
    for (int k = 0; k < c; ++k) s += cum[((size_t)m * c + k) * l + l - 1];
    out[m] = s;
}

}  // namespace cum
}  // namespace ssd
