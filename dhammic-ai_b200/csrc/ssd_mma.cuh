// Full-precision kernels on the tensor cores for bf16 calls that do not fill whole 128-position tiles.
//
// Such calls are computed in fp32: x, B, C and dy are bf16 as given, everything derived from them (masked scores, weighted rows,
// states) is fp32.  A product of a derived operand with a given one is three bf16 products: the fp32 value is cut into three bf16
// pieces of 8 significant bits each (cut8: hi + mid + lo is the value itself, no bit is lost), the given operand is bf16 already,
// and the tensor cores add the exact products up in fp32, small pieces first.  Products of two given operands (C B^T, dY x^T) need one.
//
// Why mma.sync: the pieces are made in the registers that hold the accumulator of the product before (the fragment of D is the
// fragment of A of the next product), so a masked score never leaves the registers; on tcgen05 every piece would go through TMEM and a
// barrier.  The rate of the products is not what bounds these kernels: the chain of the walk over the states is, and the latency of a head's
// loads and fragments.
//
// Tiles are 64 positions whatever the caller's chunk (the recurrence does not depend on where chunks end); what lies behind the
// end of a sequence is zero in shared memory.
//
//   state_kernel   one block per (batch, head, 32 columns of the state) walks the tiles with the state in registers and stores the state
//                  entering every tile, already cut into its three pieces, and the within-tile sums of the log-decay; a second
//                  set of blocks walks backwards with the state gradient.  One launch, or two, instead of a product per chunk and a
//                  pass over all of them.
//   scan_kernel    y of one tile and the heads of a group (or a part of them)
//   bwd_kernel     the row pass (dC, row sums) and the column pass (dx, dB, column sums) of one tile, as in chunk_bwd_kernel
//   decay_kernel   the decay gradient of a (head, batch), and dB and dC of a group whose heads several blocks share
//
// Forward + backward of (4, 1984, 20 heads, 64), d_state 64, chunk 64: 990 us of kernels in eleven launches with fp32 multiply-adds
// from shared memory, 303 us in seven now (states 131, backward 113, scan 42, decay 12); d dt is 4.0e-7 off the exact one (5.8e-7),
// dA_head 2.9e-6 (4.2e-6), the final state 1.1e-7 (2.8e-7).  At d_state 128 503 us a call; the backward has 255 registers there and spills.
#pragma once
#include <algorithm>
#include <cmath>

#include "ssd_common.cuh"
#include "ssd_ptx.cuh"

namespace ssd {
namespace mma {

constexpr int MT = 64;     // positions of a tile
constexpr int NTHR = 128;  // four warps, 16 rows of every product each
constexpr int XP = 72;     // pitch of an x-like panel [64][64]: an odd number of 16-byte units, so that eight rows hit different banks
template <int NN> constexpr int kBP = NN + 8;                // pitch of a B-like panel or a state piece [64][NN]
template <int NN> constexpr int kBPanel = MT * kBP<NN>;      // elements
constexpr int kXPanel = MT * XP;

struct Params {
    Dims d;
    int nt, splits;        // tiles; blocks that share the heads of a group
    const __nv_bfloat16 *x, *B, *C, *dy;
    const void* a;         // (b,T,h) log-decays, or null: dt * A_head
    int a_is_bf16;
    const float* cum;      // (b,h,T) their sums within each chunk, given in their place (cached calls), or null
    const float *dt, *A_head, *D, *init, *dfinal;
    __nv_bfloat16 *H, *Q;  // (b,nt,h,3,p,n): pieces of the state entering each tile, of the gradient of the state leaving it
    float* sums;           // (b,nt,h,3,64): sums of the log-decay of a tile up to each position, dt (1 without dt, 0 behind the end), sums behind it
    int per, np;           // tiles of a piece of the walk over the states, pieces
    int summary;           // the pieces' own sums are made, without a state before them: into part, for all but the last
    float *part, *part_logdecay;  // (dir,b,h,n / 32,np - 1,4,128,4): fragments of a piece's sum, (dir,b,h,n / 32,np - 1): log-decay over it
    float *final_state, *dinit;
    __nv_bfloat16 *y, *dx, *dB, *dC;
    float *g_row, *g_col, *ddtx, *dyx;   // (b,h,T)
    float* carry;          // (b,nt,h,2,4): per strip of a tile, the state's part of its sums g_row and g_col
    float *da, *ddt, *dAh_part, *dD_part;  // (b,T,h), (b,T,h), (b,h), (b,h)
    float *dB_part, *dC_part;            // (b,T,g*splits,n) when splits > 1
};

// Which calls these kernels can run.
inline bool supported(int dtype, int p, int n) { return dtype == 1 && p > 32 && p <= 64 && p % 8 == 0 && n > 32 && n <= 128 && n % 8 == 0; }
inline int tiles(int T) { return (T + MT - 1) / MT; }
// Tiles of a piece of the walk over the states, which has `blocks` blocks in one piece; nt for a walk in one piece.  As many pieces as the chip
// holds blocks at a time (three an SM), but no more than sqrt(6 nt), where the sums of the pieces before a block cost what its own
// steps do, and at least three, since every step but the last piece's is made twice.  Forward / forward and backward, us:
//   63 tiles, 2 / 4 blocks    80 / 178 in one piece, 43 / 100 in 4, 23 / 60 in 16, 22 / 57 in 32, 25 / 66 in 96
//   255 tiles, 32 / 64 blocks 350 / 885, 226 / 684 in 3, 186 / 612 in 4, 152 / 584 in 8, 149 / 556 in 12, 158 / 577 in 16, 178 / 649 in 64
//   63 tiles, 64 / 128 blocks 107 / 304, 90 / 294 in 3, 82 / 291 in 4, 80 / 291 in 6, 84 / 301 in 16
//   9 tiles, 2 / 4 blocks     20.6 / 47, 18.5 / 41 in 3, 16.5 / 39 in 5, 16.5 / 39 in 9
// Fewer than seven tiles gain nothing.
inline int piece_tiles(int nt, long long blocks) {
    const int want = (int)std::min<long long>(3 * 148 / blocks, (long long)std::sqrt(6.0 * nt));
    return nt < 7 || want < 3 ? nt : (nt + want - 1) / want;
}

// ---------------------------------------------------------------- fragments
using ptx::smem_u32;
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], uint32_t a) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void mma16816(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Address of a lane's row for the four 8 x 8 matrices of an ldmatrix.x4 whose upper-left element is (r0, c0):
// matrices in the order (rows 0-7, rows 8-15) x (columns 0-7, columns 8-15), columns slowest ...
__device__ __forceinline__ uint32_t at_rc(uint32_t base, int pitch, int r0, int c0) {
    const int l = threadIdx.x & 31;
    return base + (uint32_t)(((r0 + ((l >> 3) & 1) * 8 + (l & 7)) * pitch + c0 + (l >> 4) * 8) * 2);
}
// ... or rows slowest.
__device__ __forceinline__ uint32_t at_cr(uint32_t base, int pitch, int r0, int c0) {
    const int l = threadIdx.x & 31;
    return base + (uint32_t)(((r0 + (l >> 4) * 8 + (l & 7)) * pitch + c0 + ((l >> 3) & 1) * 8) * 2);
}
// A (16 x 16) of a matrix stored [m][k]: at_rc, ldsm4.  Of one stored [k][m]: at_cr, ldsm4t.
// B (16 x 16: two n tiles, registers {0,1} and {2,3}) of a matrix stored [n][k]: at_cr, ldsm4.  Of one stored [k][n]: at_rc, ldsm4t.

// A pair of fp32 values as three pairs of bf16 pieces: hi + mid + lo is the value (below 2^-110 in magnitude to 2^-133).  A piece is cut
// off the fp32 number before the value, and no further than the largest finite one: so each remainder of a value that is not zero is not
// zero either and has the value's sign, and an infinite value is finite pieces and an infinite lo.  Sums of the three products
// are then infinite where the product of the values is, on either side.  (Cut off the value itself, an infinite value left NaN as its
// remainder, and a piece of zero made NaN of an infinite given operand.)  The conversion cuts and packs at once: against masking the bits
// of each value, forward of (4, 1984, 20 heads, 64) 102.7 -> 100.6 us at d_state 64, forward and backward 300 -> 300; at d_state 128, where the
// backward has no register left, 496 -> 503.
__device__ __forceinline__ void cut8(float v0, float v1, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    const float2 minus = make_float2(-1.f, -1.f), before = make_float2(0x1.fffffep-1f, 0x1.fffffep-1f);
    auto head = [&](float2 v) {
        uint32_t r;
        v = ptx::mul2(v, before);
        asm("cvt.rz.satfinite.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
        return r;
    };
    auto floats = [](uint32_t u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); };
    float2 v = make_float2(v0, v1);
    hi = head(v);
    v = ptx::fma2(floats(hi), minus, v);
    mid = head(v);
    v = ptx::fma2(floats(mid), minus, v);
    lo = __byte_perm(__float_as_uint(v.x), __float_as_uint(v.y), 0x7632);
}
// The two accumulator tiles of 16 columns as the pieces of an A operand (k = those columns): f[0] = lo, f[1] = mid, f[2] = hi.
__device__ __forceinline__ void cut_tiles(const float (&t0)[4], const float (&t1)[4], uint32_t (&f)[3][4]) {
    cut8(t0[0], t0[1], f[2][0], f[1][0], f[0][0]);
    cut8(t0[2], t0[3], f[2][1], f[1][1], f[0][1]);
    cut8(t1[0], t1[1], f[2][2], f[1][2], f[0][2]);
    cut8(t1[2], t1[3], f[2][3], f[1][3], f[0][3]);
}
template <int N>
__device__ __forceinline__ void zero(float (&acc)[N][4]) {
#pragma unroll
    for (int i = 0; i < N; ++i)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
}
// (As __expf, without the instructions that keep results below 2^-126.)
__device__ __forceinline__ float exp_(float v) {
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v * 1.4426950408889634f));
    return r;
}
__device__ __forceinline__ float2 unpack(uint32_t u) { return make_float2(__uint_as_float(u << 16), __uint_as_float(u & 0xffff0000u)); }
__device__ __forceinline__ uint32_t pack(float a, float b) {
    const __nv_bfloat162 v = __floats2bfloat162_rn(a, b);
    return *reinterpret_cast<const uint32_t*>(&v);
}
__device__ __forceinline__ float quad_sum(float v) {
    v += __shfl_xor_sync(0xffffffffu, v, 1);
    return v + __shfl_xor_sync(0xffffffffu, v, 2);
}

// ---------------------------------------------------------------- loads
__device__ __forceinline__ void cp16(uint32_t dst, const void* src, bool ok) {  // 16 bytes, zeros where not ok
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }
// A panel of 64 rows x COLS columns; rows >= `rows` and columns >= `cols` (a multiple of 8) become zero.  WIDE: every tensor
// starts on a 16-byte boundary; else the values are fetched one by one (a kernel of its own: as a switch it cost 8 %).
template <int COLS, bool WIDE>
__device__ __forceinline__ void load_panel(uint32_t dst, int pitch, const __nv_bfloat16* src, size_t stride, int rows, int cols) {
    constexpr int Q = COLS / 8, RSTEP = NTHR / Q;  // 16-byte units of a row, rows of a round
    const unsigned r0 = threadIdx.x / Q, q = (threadIdx.x % Q) * 8;
    const __nv_bfloat16* p = src + (size_t)r0 * stride + q;
    uint32_t o = dst + (r0 * pitch + q) * 2;
#pragma unroll
    for (int r = 0; r < MT; r += RSTEP) {
        const bool ok = (int)(r0 + r) < rows && (int)q < cols;
        if (WIDE) {
            cp16(o, ok ? p : src, ok);
        } else {
            const unsigned short* e = reinterpret_cast<const unsigned short*>(p);
            uint32_t v[4] = {0u, 0u, 0u, 0u};
            if (ok)
#pragma unroll
                for (int i = 0; i < 4; ++i) v[i] = e[2 * i] | (uint32_t)e[2 * i + 1] << 16;
            asm volatile("st.shared.v4.b32 [%0], {%1,%2,%3,%4};" ::"r"(o), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]) : "memory");
        }
        p += RSTEP * stride;
        o += RSTEP * pitch * 2;
    }
}
// A pair of results as bf16.
template <bool WIDE>
__device__ __forceinline__ void store_pair(__nv_bfloat16* o, float a, float b) {
    if (WIDE) {
        *reinterpret_cast<uint32_t*>(o) = pack(a, b);
    } else {
        o[0] = __float2bfloat16_rn(a);
        o[1] = __float2bfloat16_rn(b);
    }
}
__device__ __forceinline__ size_t tile_off(const Dims& d, int nt, int bb, int k, int hh) { return ((size_t)bb * nt + k) * d.h + hh; }
template <int NN>
__device__ __forceinline__ void load_pieces(uint32_t dst, const __nv_bfloat16* src, const Dims& d) {
#pragma unroll
    for (int q = 0; q < 3; ++q) load_panel<NN, true>(dst + q * kBPanel<NN> * 2, kBP<NN>, src + (size_t)q * d.p * d.n, d.n, d.p, d.n);
}
// The first ROWS rows of the sums of a tile and head (cum[64], dt[64], behind[64]), in units of 16 bytes.
template <int ROWS>
__device__ __forceinline__ void load_sums(uint32_t dst, const Params& P, size_t tile) {
    if (threadIdx.x < ROWS * 16) cp16(dst + threadIdx.x * 16, P.sums + tile * 3 * MT + threadIdx.x * 4, true);
}

// The log-decay and dt of position t of the sequence (nothing behind its end); the load does not wait for a branch.
struct Decay {
    float v, dt;
};
__device__ __forceinline__ Decay fetch_decay(const Params& P, int bb, int hh, int t) {
    const size_t i = ((size_t)bb * P.d.T + min(t, P.d.T - 1)) * P.d.h + hh;
    Decay r{0.f, 1.f};
    if (P.dt) r.dt = P.dt[i];
    if (P.cum) {  // the differences: exact, or nearly so
        const int tt = min(t, P.d.T - 1);
        const float* c = P.cum + ((size_t)bb * P.d.h + hh) * P.d.T + tt;
        r.v = tt % P.d.l ? c[0] - c[-1] : c[0];
    } else if (P.a) r.v = P.a_is_bf16 ? __bfloat162float(((const __nv_bfloat16*)P.a)[i]) : ((const float*)P.a)[i];
    return r;
}
// A log-decay as it enters the sums of a tile.  exp_ is zero below -87.4, so nothing passes a position of -90 either; lower values, down to a
// type's lowest for a cut, would only take their bits from the sums of the positions behind, which may lie in other chunks of the caller's.
__device__ __forceinline__ float cut_off(float a) { return a < -90.f ? -90.f : a; }
// Inclusive sums over the 64 positions of a tile: lane l holds positions l and l + 32.  The whole warp.
__device__ __forceinline__ void tile_sums(float& c0, float& c1) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u0 = __shfl_up_sync(0xffffffffu, c0, o), u1 = __shfl_up_sync(0xffffffffu, c1, o);
        if (lane >= o) {
            c0 += u0;
            c1 += u1;
        }
    }
    c1 += __shfl_sync(0xffffffffu, c0, 31);
}
// The sums behind the positions.  (As the sum of the tile less the sum up to a position they would carry the rounding of the former: the final
// state of 640 positions with log-decays of -8 was 1.9e-6 off, 1.9e-7 so.)
__device__ __forceinline__ void tile_sums_behind(float& c0, float& c1) {
    const int lane = threadIdx.x & 31;
    const float n0 = __shfl_down_sync(0xffffffffu, c0, 1), n1 = __shfl_down_sync(0xffffffffu, c1, 1), m1 = __shfl_sync(0xffffffffu, c1, 0);
    c0 = lane < 31 ? n0 : m1;
    c1 = lane < 31 ? n1 : 0.f;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const float u0 = __shfl_down_sync(0xffffffffu, c0, o), u1 = __shfl_down_sync(0xffffffffu, c1, o);
        if (lane + o < 32) {
            c0 += u0;
            c1 += u1;
        }
    }
    c0 += __shfl_sync(0xffffffffu, c1, 0);
}
// ------------------------------------------------------------------------------------------
// The recurrence over the tiles.  Direction 0: H <- e^S H + sum_j x_j (w_j B_j), w_j = e^(sum behind j) dt_j, the state entering tile k
// stored before it; direction 1, from the last tile to the first: Q <- e^S Q + sum_i dy_i (e^(cum_i) C_i).  One block per
// (head, 32 columns of the state), batch, direction.  Four warps: a warp has all rows of 8 columns, so the weighted operand, which is
// the one that is cut, is cut once and used where it is cut, and the given one is read as it is; a fifth makes the weights
// of the next tile.  The state leaves through shared memory in 16-byte stores.
//
// Bound by the chain of its T / 64 steps, and within a step by shared memory and issue slots where an SM has two or three blocks.
// 31 steps of (4, 1984, 20 heads), d_state 64: 75 us with 32 x 16 of the state per warp (the cut operand was then read back
// by four warps) and 4-byte stores of the fragments (20 us of them).
//
// Where few blocks would walk far (piece_tiles), the walk is cut into pieces that run side by side: a first launch makes each piece's own
// sum, without a state before it, and in the second a block folds the sums of the pieces before its own into the state it starts from.
// ------------------------------------------------------------------------------------------
constexpr int kStateThreads = 160, kStateCols = 32;
struct StateCfg {
    static constexpr int ST = 3;   // load stages
    static constexpr int VP = kStateCols + 8;
    static constexpr int STAGE = kXPanel + MT * VP;  // elements: x or dy | 32 columns of B or C
    static constexpr int OUT = 3 * MT * VP;          // elements: the pieces of the state on their way out
    static constexpr size_t SMEM = ((size_t)ST * STAGE + 2 * OUT) * 2 + (2 * MT + 4) * 4;
};
// CUT: in pieces (a kernel of its own: with the bounds of a piece the walk of one piece took 2 % longer).
template <bool WIDE, bool CUT>
__global__ void __launch_bounds__(kStateThreads, 3) state_kernel(Params P) {
    dep_wait();
    using Cfg = StateCfg;
    extern __shared__ __align__(16) __nv_bfloat16 sh[];
    __nv_bfloat16* out = sh + Cfg::ST * Cfg::STAGE;          // [2][3][64][VP]
    float* w = reinterpret_cast<float*>(out + 2 * Cfg::OUT);  // [2][64] weights, [2] decay of the tile
    float* dec = w + 2 * MT;
    const Dims& d = P.d;
    const int nb = (d.n + kStateCols - 1) / kStateCols;
    const int piece = CUT ? blockIdx.x / (d.h * nb) : 0, hh = CUT ? blockIdx.x / nb % d.h : blockIdx.x / nb, col0 = (blockIdx.x % nb) * kStateCols, bb = blockIdx.y, dir = blockIdx.z;
    const int gg = hh / d.hpg, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool summary = CUT && P.summary;
    const int it0 = CUT ? piece * P.per : 0, steps = CUT ? min(P.per, P.nt - it0) : P.nt;
    const size_t slot = ((((size_t)dir * d.b + bb) * d.h + hh) * nb + col0 / kStateCols) * (P.np - 1);  // of the first piece
    auto tile_of = [&](int it) { return dir ? P.nt - 1 - it0 - it : it0 + it; };
    if (warp == 4) {  // the weights, and the arrays the other kernels read
        const bool given = P.a || P.cum;
        const float Ah = given ? 0.f : P.A_head[hh];
        const bool keep = dir == 0 && col0 == 0 && !summary;
        float total = 0.f;
        Decay f0, f1;
        auto fetch = [&](int it) {
            if (it >= steps) return;
            f0 = fetch_decay(P, bb, hh, tile_of(it) * MT + lane);
            f1 = fetch_decay(P, bb, hh, tile_of(it) * MT + 32 + lane);
        };
        auto weights = [&](int it) {
            if (it >= steps) return;
            const int left = d.T - tile_of(it) * MT - lane;  // positions left from this lane's first
            const float d0 = left > 0 ? f0.dt : 0.f, d1 = left > 32 ? f1.dt : 0.f;
            float a0 = left > 0 ? cut_off(given ? f0.v : f0.dt * Ah) : 0.f, a1 = left > 32 ? cut_off(given ? f1.v : f1.dt * Ah) : 0.f;
            fetch(it + 1);
            float b0 = a0, b1 = a1;
            if (!dir) tile_sums_behind(b0, b1);
            tile_sums(a0, a1);
            const float S = __shfl_sync(0xffffffffu, a1, 31);
            float* o = w + (it & 1) * MT;
            o[lane] = dir ? exp_(a0) : exp_(b0) * d0;
            o[32 + lane] = dir ? exp_(a1) : exp_(b1) * d1;
            if (lane == 0) dec[it & 1] = exp_(S);
            total += S;
            if (keep) {
                float* k = P.sums + tile_off(d, P.nt, bb, tile_of(it), hh) * 3 * MT;
                k[lane] = a0;
                k[32 + lane] = a1;
                k[MT + lane] = d0;
                k[MT + 32 + lane] = d1;
                k[2 * MT + lane] = b0;
                k[2 * MT + 32 + lane] = b1;
            }
        };
        fetch(0);
        weights(0);
        for (int it = 0; it < steps; ++it) {
            __syncthreads();
            weights(it + 1);
        }
        if (summary && lane == 0) P.part_logdecay[slot + piece] = total;
        return;
    }
    const __nv_bfloat16* U = (dir ? P.dy : P.x) + ((size_t)bb * d.T * d.h + hh) * d.p;
    const __nv_bfloat16* V = (dir ? P.C : P.B) + ((size_t)bb * d.T * d.g + gg) * d.n + col0;
    __nv_bfloat16* pieces = summary ? nullptr : dir ? P.Q : P.H;
    const uint32_t base = smem_u32(sh);
    auto stage = [&](int it) { return base + (it % Cfg::ST) * Cfg::STAGE * 2; };
    auto load = [&](int it) {  // one group of copies per tile, empty behind the last
        if (it < steps) {
            const int t0 = tile_of(it) * MT, rows = min(MT, d.T - t0);
            load_panel<64, WIDE>(stage(it), XP, U + (size_t)t0 * d.h * d.p, (size_t)d.h * d.p, rows, d.p);
            load_panel<kStateCols, WIDE>(stage(it) + kXPanel * 2, Cfg::VP, V + (size_t)t0 * d.g * d.n, (size_t)d.g * d.n, rows, d.n - col0);
        }
        cp_commit();
    };
    load(0);
    load(1);
    float H[4][4];  // rows 16 q + g (+ 8), columns 2 t, 2 t + 1 of the warp's eight
    const float* seed = summary ? nullptr : dir ? P.dfinal : P.init;
    const size_t bh = ((size_t)bb * d.h + hh) * d.p * d.n;
    const int nn0 = col0 + warp * 8 + 2 * t;
#pragma unroll
    for (int q = 0; q < 4; ++q)
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int pp = q * 16 + g + (c >> 1) * 8, nn = nn0 + (c & 1);
            H[q][c] = (seed && pp < d.p && nn < d.n) ? seed[bh + (size_t)pp * d.n + nn] : 0.f;
        }
    if (CUT && !summary)  // the pieces before this one
#pragma unroll 4
        for (int k = 0; k < piece; ++k) {
            const float4* f = reinterpret_cast<const float4*>(P.part) + (slot + k) * 512 + threadIdx.x;
            const float decay = exp_(P.part_logdecay[slot + k]);
            // (an infinite state lasts, also where the decay over a whole piece is too small for a number)
            auto step = [&](float h, float v) { return fmaf(isinf(h) ? 1.f : decay, h, v); };
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const float4 v = f[q * 128];
                H[q][0] = step(H[q][0], v.x);
                H[q][1] = step(H[q][1], v.y);
                H[q][2] = step(H[q][2], v.z);
                H[q][3] = step(H[q][3], v.w);
            }
        }
    auto stage_state = [&](int it) {  // the state before tile `it`, cut, on its way out
        uint32_t* o = reinterpret_cast<uint32_t*>(out + (it & 1) * Cfg::OUT + g * Cfg::VP + warp * 8 + 2 * t);
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                uint32_t hi, mid, lo;
                cut8(H[q][2 * c], H[q][2 * c + 1], hi, mid, lo);
                uint32_t* e = o + (q * 16 + c * 8) * Cfg::VP / 2;
                e[0] = hi;
                e[MT * Cfg::VP / 2] = mid;
                e[MT * Cfg::VP] = lo;
            }
    };
    if (pieces) stage_state(0);
    for (int it = 0; it < steps; ++it) {
        cp_wait<1>();
        __syncthreads();  // there: the tile, its weights, the state before it.  Free: the stage of the last tile
        load(it + 2);
        const uint32_t sU = stage(it), sV = sU + kXPanel * 2;
        const float* wt = w + (it & 1) * MT + 2 * t;
        uint32_t f[3][4][2];  // (w V), cut: B operands of the four k steps
#pragma unroll
        for (int k2 = 0; k2 < 2; ++k2) {
            uint32_t r[4];  // 32 positions x 8 columns
            ldsm4t(r, sV + (uint32_t)(((k2 * 32 + lane) * Cfg::VP + warp * 8) * 2));
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float2 v = unpack(r[c]), ww = *reinterpret_cast<const float2*>(wt + k2 * 32 + c * 8);
                const int kk = k2 * 2 + (c >> 1);
                cut8(v.x * ww.x, v.y * ww.y, f[2][kk][c & 1], f[1][kk][c & 1], f[0][kk][c & 1]);
            }
        }
        if (pieces) {
            __nv_bfloat16* o = pieces + tile_off(d, P.nt, bb, tile_of(it), hh) * 3 * d.p * d.n + col0;
            const __nv_bfloat16* from = out + (it & 1) * Cfg::OUT;
            const int r0 = threadIdx.x / 4, q = threadIdx.x % 4 * 8;
            if (col0 + q < d.n)
#pragma unroll
                for (int i = 0; i < 6; ++i) {
                    const int s = i / 2, r = r0 + (i & 1) * 32;
                    if (r < d.p) *reinterpret_cast<uint4*>(o + ((size_t)s * d.p + r) * d.n + q) = *reinterpret_cast<const uint4*>(from + (s * MT + r) * Cfg::VP + q);
                }
        }
        const float decay = dec[it & 1];
        float acc[4][4], small[4][4];  // the large pieces' part of the product, and the others'
        zero(acc);
        zero(small);
#pragma unroll
        for (int kk = 0; kk < MT / 16; ++kk)
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t a[4];
                ldsm4t(a, at_cr(sU, XP, kk * 16, q * 16));
                mma16816(small[q], a, f[0][kk][0], f[0][kk][1]);
                mma16816(acc[q], a, f[2][kk][0], f[2][kk][1]);
                mma16816(small[q], a, f[1][kk][0], f[1][kk][1]);
            }
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 4; ++c) H[q][c] = fmaf(decay, H[q][c], acc[q][c] + small[q][c]);
        if (pieces && it + 1 < steps) stage_state(it + 1);
    }
    if (summary) {
        float4* o = reinterpret_cast<float4*>(P.part) + (slot + piece) * 512 + threadIdx.x;
#pragma unroll
        for (int q = 0; q < 4; ++q) o[q * 128] = make_float4(H[q][0], H[q][1], H[q][2], H[q][3]);
        return;
    }
    if (float* o = CUT && piece + 1 < P.np ? nullptr : dir ? P.dinit : P.final_state)
#pragma unroll
        for (int q = 0; q < 4; ++q)
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int pp = q * 16 + g + (c >> 1) * 8;
                if (pp < d.p && nn0 < d.n) o[bh + (size_t)pp * d.n + nn0 + (c & 1)] = H[q][c];
            }
}

// Which rows a block works on: tile k of batch bb, heads h0 .. h0 + hps - 1 of group gg.  Causal rows are the longer the later
// they lie in the tile, so every other block hands its 16-row strips to the warps in the opposite order.
struct Where {
    int k, bb, gg, sp, h0, hps, t0, rows, strip;
};
__device__ __forceinline__ Where where(const Params& P) {
    Where w;
    w.k = blockIdx.x % P.nt;
    w.bb = blockIdx.x / P.nt;
    w.gg = blockIdx.y / P.splits;
    w.sp = blockIdx.y % P.splits;
    w.hps = P.d.hpg / P.splits;
    w.h0 = w.gg * P.d.hpg + w.sp * w.hps;
    w.t0 = w.k * MT;
    w.rows = min(MT, P.d.T - w.t0);
    const int warp = threadIdx.x >> 5;
    w.strip = ((blockIdx.x + blockIdx.y + blockIdx.z) & 1) ? 3 - warp : warp;
    return w;
}

// S[2 q], S[2 q + 1] = the 16 columns q of the strip's rows of A B^T (both [64][NN] panels), for q in [lo, hi)
template <int NN>
__device__ __forceinline__ void scores(float (&S)[8][4], uint32_t sA, uint32_t sB, int strip, int lo, int hi) {
    zero(S);
#pragma unroll
    for (int kk = 0; kk < NN / 16; ++kk) {
        uint32_t a[4];
        ldsm4(a, at_rc(sA, kBP<NN>, strip * 16, kk * 16));
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (q < lo || q >= hi) continue;
            uint32_t b[4];
            ldsm4(b, at_cr(sB, kBP<NN>, q * 16, kk * 16));
            mma16816(S[2 * q], a, b[0], b[1]);
            mma16816(S[2 * q + 1], a, b[2], b[3]);
        }
    }
}

// acc (8 column tiles from c0) += A pieces x B stored [k][n], 16 rows k from k0
__device__ __forceinline__ void mma_cut(float (*acc)[4], const uint32_t (&f)[3][4], uint32_t sB, int pitch, int k0, int c0) {
#pragma unroll
    for (int q = 0; q < 8; q += 2) {
        uint32_t b[4];
        ldsm4t(b, at_rc(sB, pitch, k0, c0 + q * 8));
#pragma unroll
        for (int s = 0; s < 3; ++s) {
            mma16816(acc[q], f[s], b[0], b[1]);
            mma16816(acc[q + 1], f[s], b[2], b[3]);
        }
    }
}

// Scores of the strip's own positions are zero behind each row, which on the tensor cores makes NaN of a row before an infinite value.
// So where rows k0 .. k0 + 15 of such a product's B (COLS columns) hold an infinite value or none ...  The look costs 0.2 us of 100.6 (forward of
// (4, 1984, 20 heads, 64), d_state 64), 1.7 of 150 at d_state 128; in the backward, once for all heads of a block, nothing that shows.
template <int COLS>
__device__ __forceinline__ bool all_finite(uint32_t sB, int pitch, int k0) {
    uint32_t z = 0u;  // 0 times every value
#pragma unroll
    for (int q = 0; q < COLS / 8; q += 2) {
        uint32_t b[4];
        ldsm4t(b, at_rc(sB, pitch, k0, q * 8));
#pragma unroll
        for (int i = 0; i < 4; ++i) asm("fma.rn.bf16x2 %0, %1, %2, %0;" : "+r"(z) : "r"(b[i]), "r"(0u));
    }
    return !__any_sync(0xffffffffu, (z & 0x7fff7fffu) != 0u);
}
// ... the products are made one by one, up to each row: v (rows g, g + 8 of the strip, its columns 8 u + 2 t, + 1) times eight columns of B
// (`row`: row k0, this thread's first column), the four values of this thread.  A call, so that the common path keeps its registers.
__device__ __noinline__ float4 own_positions(float4 v0, float4 v1, const __nv_bfloat16* row, int pitch) {
    const int lane = threadIdx.x & 31, g = lane >> 2;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = 0; j < 16; ++j, row += pitch) {
        const float4 v = j < 8 ? v0 : v1;
        const int from = (lane & ~3) | (j >> 1 & 3);
        const float w0 = __shfl_sync(0xffffffffu, j & 1 ? v.y : v.x, from), w1 = __shfl_sync(0xffffffffu, j & 1 ? v.w : v.z, from);
        const float2 b = unpack(*reinterpret_cast<const uint32_t*>(row));
        if (j <= g) {
            s.x = fmaf(w0, b.x, s.x);
            s.y = fmaf(w0, b.y, s.y);
        }
        if (j <= g + 8) {
            s.z = fmaf(w1, b.x, s.z);
            s.w = fmaf(w1, b.y, s.w);
        }
    }
    return s;
}
template <int N>
__device__ __forceinline__ void add_own_positions(float (&acc)[N][4], const float (&v)[2][4], const __nv_bfloat16* B, int pitch, int k0) {
    const __nv_bfloat16* row = B + k0 * pitch + 2 * (threadIdx.x & 3);
#pragma unroll
    for (int q = 0; q < N; ++q) {
        const float4 s = own_positions(make_float4(v[0][0], v[0][1], v[0][2], v[0][3]), make_float4(v[1][0], v[1][1], v[1][2], v[1][3]), row + q * 8, pitch);
        acc[q][0] += s.x;
        acc[q][1] += s.y;
        acc[q][2] += s.z;
        acc[q][3] += s.w;
    }
}

// ------------------------------------------------------------------------------------------
// y of one tile.
// ------------------------------------------------------------------------------------------
template <int NN>
struct ScanCfg {
    static constexpr size_t SMEM = (size_t)(5 * kBPanel<NN> + kXPanel) * 2 + 2 * MT * 4;  // C, B, three pieces of H | x | cum, dt
};
template <int NN, bool WIDE>
__global__ void __launch_bounds__(NTHR, NN == 64 ? 3 : 2) scan_kernel(Params P) {
    dep_wait();
    extern __shared__ __align__(16) __nv_bfloat16 sh[];
    const Dims& d = P.d;
    const Where w = where(P);
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    __nv_bfloat16* xs = sh + 5 * kBPanel<NN>;
    float* cum = reinterpret_cast<float*>(xs + kXPanel);
    float* dts = cum + MT;
    const uint32_t sC = smem_u32(sh), sB = sC + kBPanel<NN> * 2, sH = sB + kBPanel<NN> * 2, sX = smem_u32(xs);
    const size_t bc = (((size_t)w.bb * d.T + w.t0) * d.g + w.gg) * d.n;
    load_panel<NN, WIDE>(sC, kBP<NN>, P.C + bc, (size_t)d.g * d.n, w.rows, d.n);
    load_panel<NN, WIDE>(sB, kBP<NN>, P.B + bc, (size_t)d.g * d.n, w.rows, d.n);
    const int r0 = w.strip * 16 + g;  // this thread's rows: r0, r0 + 8
    float S[8][4];
    for (int hl = 0; hl < w.hps; ++hl) {
        const int hh = w.h0 + hl;
        const size_t xo = (((size_t)w.bb * d.T + w.t0) * d.h + hh) * d.p;
        if (hl) __syncthreads();
        load_panel<64, WIDE>(sX, XP, P.x + xo, (size_t)d.h * d.p, w.rows, d.p);
        const size_t tile = tile_off(d, P.nt, w.bb, w.k, hh);
        load_sums<2>(smem_u32(cum), P, tile);
        load_pieces<NN>(sH, P.H + tile * 3 * d.p * d.n, d);
        cp_commit();
        cp_wait<0>();
        __syncthreads();
        if (hl == 0) scores<NN>(S, sC, sB, w.strip, 0, w.strip + 1);
        const float c0 = cum[r0], c1 = cum[r0 + 8];
        float acc[8][4];
        zero(acc);
#pragma unroll
        for (int kk = 0; kk < NN / 16; ++kk) {  // the state entering the tile: C H^T
            uint32_t a[4];
            ldsm4(a, at_rc(sC, kBP<NN>, w.strip * 16, kk * 16));
#pragma unroll
            for (int s = 2; s >= 0; --s)
#pragma unroll
                for (int q = 0; q < 8; q += 2) {
                    uint32_t b[4];
                    ldsm4(b, at_cr(sH + s * kBPanel<NN> * 2, kBP<NN>, q * 8, kk * 16));
                    mma16816(acc[q], a, b[0], b[1]);
                    mma16816(acc[q + 1], a, b[2], b[3]);
                }
        }
        {
            const float e0 = exp_(c0), e1 = exp_(c1);
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                acc[q][0] *= e0;
                acc[q][1] *= e0;
                acc[q][2] *= e1;
                acc[q][3] *= e1;
            }
        }
        const bool finite = all_finite<64>(sX, XP, w.strip * 16);
        float vo[2][4];  // the strip's own positions, where not
#pragma unroll
        for (int kb = 0; kb < 4; ++kb) {  // the masked scores, 16 columns at a time
            if (kb > w.strip) continue;
            float v[2][4];
#pragma unroll
            for (int u = 0; u < 2; ++u) {
                const int j0 = kb * 16 + u * 8 + 2 * t;
                const float2 cj = *reinterpret_cast<const float2*>(cum + j0), dj = *reinterpret_cast<const float2*>(dts + j0);
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[u][c] = S[2 * kb + u][c] * ((c & 1 ? dj.y : dj.x) * exp_((c < 2 ? c0 : c1) - (c & 1 ? cj.y : cj.x)));
                    if (kb == w.strip && r0 + (c >> 1) * 8 < j0 + (c & 1)) v[u][c] = 0.f;
                    vo[u][c] = v[u][c];
                }
            }
            if (kb == w.strip && !finite) continue;
            uint32_t f[3][4];
            cut_tiles(v[0], v[1], f);
            mma_cut(acc, f, sX, XP, kb * 16, 0);
        }
        if (!finite) add_own_positions(acc, vo, xs, XP, w.strip * 16);
        const float Dh = P.D ? P.D[hh] : 0.f;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const int pp = q * 8 + 2 * t;
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                const int i = r0 + c * 8;
                if (i >= w.rows || pp >= d.p) continue;
                float y0 = acc[q][2 * c], y1 = acc[q][2 * c + 1];
                if (P.D) {
                    const float2 xv = unpack(*reinterpret_cast<const uint32_t*>(xs + i * XP + pp));
                    y0 = fmaf(Dh, xv.x, y0);
                    y1 = fmaf(Dh, xv.y, y1);
                }
                store_pair<WIDE>(P.y + xo + (size_t)i * d.h * d.p + pp, y0, y1);
            }
        }
    }
}

// ------------------------------------------------------------------------------------------
// Backward of one tile.  blockIdx.z = 0, rows i of the tile:
//   dC_i = sum_h [ sum_j dS_ij B_j + e_i dY_i H ],  g_row[i] = rowsum_i(dS o S) + <e_i dY_i H, C_i> per head
// and blockIdx.z = 1, rows j:
//   dX_j = sum_i G_ij^T dY_i + d_j B_j Q^T,  dB_j = sum_h [ sum_i dS_ij^T C_i + d_j dt_j x_j Q ],
//   g_col[j] = colsum_j(dS o S) + d_j dt_j <x_j, B_j Q^T>,  dx = dX dt + D dy,  ddtx[j] = <dX_j, x_j>,  dyx[j] = <dy_j, x_j>
// with dS_ij = dY_i x_j dt_j L_ij, G = (C B^T) o L.  Both make S and dY x^T for themselves (one product each, exact operands); the
// transposed operands of the column pass would otherwise go through shared memory in three pieces.
// ------------------------------------------------------------------------------------------
template <int NN>
struct BwdCfg {
    static constexpr size_t SMEM = (size_t)(5 * kBPanel<NN> + 2 * kXPanel) * 2 + 3 * MT * 4;  // own, other, three pieces | x, dy | cum, dt, behind
};
template <int NN, bool WIDE>
__device__ __forceinline__ void store_bc(const Params& P, const Where& w, const float (&acc)[NN / 8][4], float* part, __nv_bfloat16* out) {
    const Dims& d = P.d;
    const int lane = threadIdx.x & 31, r0 = w.strip * 16 + (lane >> 2);
#pragma unroll
    for (int q = 0; q < NN / 8; ++q) {
        const int nn = q * 8 + 2 * (lane & 3);
#pragma unroll
        for (int c = 0; c < 2; ++c) {
            const int i = r0 + c * 8;
            if (i >= w.rows || nn >= d.n) continue;
            const size_t row = ((size_t)w.bb * d.T + w.t0 + i) * d.g + w.gg;
            if (part) *reinterpret_cast<float2*>(part + (row * P.splits + w.sp) * d.n + nn) = make_float2(acc[q][2 * c], acc[q][2 * c + 1]);
            else store_pair<WIDE>(out + row * d.n + nn, acc[q][2 * c], acc[q][2 * c + 1]);
        }
    }
}
// o (8 column tiles) = A rows (fragments of the strip, k = headdim) x pieces stored [p][n], columns from c0, small pieces first
template <int NN>
__device__ __forceinline__ void rows_by_pieces(float (&o)[8][4], const uint32_t (&a)[4][4], uint32_t sW, int c0) {
    zero(o);
#pragma unroll
    for (int s = 2; s >= 0; --s)
#pragma unroll
        for (int kk = 0; kk < 4; ++kk)
#pragma unroll
            for (int q = 0; q < 8; q += 2) {
                uint32_t b[4];
                ldsm4t(b, at_rc(sW + s * kBPanel<NN> * 2, kBP<NN>, kk * 16, c0 + q * 8));
                mma16816(o[q], a[kk], b[0], b[1]);
                mma16816(o[q + 1], a[kk], b[2], b[3]);
            }
}

template <int NN, bool WIDE>
__global__ void __launch_bounds__(NTHR, NN == 64 ? 3 : 2) bwd_kernel(Params P) {
    dep_wait();
    extern __shared__ __align__(16) __nv_bfloat16 sh[];
    const Dims& d = P.d;
    const Where w = where(P);
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const bool row_pass = blockIdx.z == 0;
    __nv_bfloat16* own = sh;                   // C (row pass) or B: the rows of the block
    __nv_bfloat16* xs = sh + 5 * kBPanel<NN>;
    __nv_bfloat16* ys = xs + kXPanel;
    float* cum = reinterpret_cast<float*>(ys + kXPanel);
    float* dts = cum + MT;
    const uint32_t sOwn = smem_u32(sh), sOther = sOwn + kBPanel<NN> * 2, sW = sOther + kBPanel<NN> * 2, sX = smem_u32(xs), sY = smem_u32(ys);
    const size_t bc = (((size_t)w.bb * d.T + w.t0) * d.g + w.gg) * d.n;
    load_panel<NN, WIDE>(sOwn, kBP<NN>, (row_pass ? P.C : P.B) + bc, (size_t)d.g * d.n, w.rows, d.n);
    load_panel<NN, WIDE>(sOther, kBP<NN>, (row_pass ? P.B : P.C) + bc, (size_t)d.g * d.n, w.rows, d.n);
    const int r0 = w.strip * 16 + g;
    float acc[NN / 8][4];     // dC or dB
    zero(acc);
    uint32_t rows[NN / 16][4];  // the strip's rows of C or B
    bool finite = true;         // row pass: the strip's rows of B
    auto scores16 = [&](float (&S)[2][4], int kb) {  // 16 columns of the strip's scores (transposed in the column pass)
        zero(S);
#pragma unroll
        for (int kk = 0; kk < NN / 16; ++kk) {
            uint32_t b[4];
            ldsm4(b, at_cr(sOther, kBP<NN>, kb * 16, kk * 16));
            mma16816(S[0], rows[kk], b[0], b[1]);
            mma16816(S[1], rows[kk], b[2], b[3]);
        }
    };
    auto store_carry = [&](float v, size_t tile) {  // v: sum of a thread's two rows, the same in all lanes of a quad
#pragma unroll
        for (int o = 4; o < 32; o <<= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) P.carry[tile * 8 + (row_pass ? 0 : 4) + w.strip] = v;
    };
    for (int hl = 0; hl < w.hps; ++hl) {
        const int hh = w.h0 + hl;
        const size_t xo = (((size_t)w.bb * d.T + w.t0) * d.h + hh) * d.p;
        if (hl) __syncthreads();
        load_panel<64, WIDE>(sX, XP, P.x + xo, (size_t)d.h * d.p, w.rows, d.p);
        load_panel<64, WIDE>(sY, XP, P.dy + xo, (size_t)d.h * d.p, w.rows, d.p);
        const size_t tile = tile_off(d, P.nt, w.bb, w.k, hh);
        load_sums<3>(smem_u32(cum), P, tile);
        cp_commit();
        load_pieces<NN>(sW, (row_pass ? P.H : P.Q) + tile * 3 * d.p * d.n, d);
        cp_commit();
        cp_wait<1>();
        __syncthreads();
        if (hl == 0)
#pragma unroll
            for (int kk = 0; kk < NN / 16; ++kk) ldsm4(rows[kk], at_rc(sOwn, kBP<NN>, w.strip * 16, kk * 16));
        const float c0 = cum[r0], c1 = cum[r0 + 8];
        uint32_t a[4][4];  // rows of dy (row pass) or x
#pragma unroll
        for (int kk = 0; kk < 4; ++kk) ldsm4(a[kk], at_rc(row_pass ? sY : sX, XP, w.strip * 16, kk * 16));
        float sum0 = 0.f, sum1 = 0.f;  // of the rows r0, r0 + 8
        if (row_pass) {
            if (hl == 0) finite = all_finite<NN>(sOther, kBP<NN>, w.strip * 16);
            float vo[2][4];
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                if (kb > w.strip) continue;
                float v[2][4], S[2][4];
                zero(v);
                scores16(S, kb);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t b[4];
                    ldsm4(b, at_cr(sX, XP, kb * 16, kk * 16));
                    mma16816(v[0], a[kk], b[0], b[1]);
                    mma16816(v[1], a[kk], b[2], b[3]);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int j0 = kb * 16 + u * 8 + 2 * t;
                    const float2 cj = *reinterpret_cast<const float2*>(cum + j0), dj = *reinterpret_cast<const float2*>(dts + j0);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        v[u][c] *= (c & 1 ? dj.y : dj.x) * exp_((c < 2 ? c0 : c1) - (c & 1 ? cj.y : cj.x));
                        if (kb == w.strip && r0 + (c >> 1) * 8 < j0 + (c & 1)) v[u][c] = 0.f;
                        float& s = c < 2 ? sum0 : sum1;
                        s = fmaf(v[u][c], S[u][c], s);
                        vo[u][c] = v[u][c];
                    }
                }
                if (kb == w.strip && !finite) continue;
                uint32_t f[3][4];
                cut_tiles(v[0], v[1], f);
#pragma unroll
                for (int q = 0; q < NN / 8; q += 8) mma_cut(acc + q, f, sOther, kBP<NN>, kb * 16, q * 8);
            }
            if (!finite) add_own_positions(acc, vo, own + kBPanel<NN>, kBP<NN>, w.strip * 16);
            cp_wait<0>();
            __syncthreads();
            const float e0 = exp_(c0), e1 = exp_(c1);
            float st0 = 0.f, st1 = 0.f;  // the state's part
#pragma unroll
            for (int q0 = 0; q0 < NN / 8; q0 += 8) {
                float o[8][4];
                rows_by_pieces<NN>(o, a, sW, q0 * 8);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const __nv_bfloat16* cr = own + r0 * kBP<NN> + (q0 + q) * 8 + 2 * t;
                    const float2 k0 = unpack(*reinterpret_cast<const uint32_t*>(cr)), k1 = unpack(*reinterpret_cast<const uint32_t*>(cr + 8 * kBP<NN>));
                    const float v0 = e0 * o[q][0], v1 = e0 * o[q][1], v2 = e1 * o[q][2], v3 = e1 * o[q][3];
                    acc[q0 + q][0] += v0;
                    acc[q0 + q][1] += v1;
                    acc[q0 + q][2] += v2;
                    acc[q0 + q][3] += v3;
                    st0 = fmaf(v1, k0.y, fmaf(v0, k0.x, st0));
                    st1 = fmaf(v3, k1.y, fmaf(v2, k1.x, st1));
                }
            }
            st0 = quad_sum(st0);
            st1 = quad_sum(st1);
            if (r0 >= w.rows) st0 = 0.f;  // behind the end: no number where the state is infinite
            if (r0 + 8 >= w.rows) st1 = 0.f;
            store_carry(st0 + st1, tile);
            sum0 = quad_sum(sum0) + st0;
            sum1 = quad_sum(sum1) + st1;
            if (t == 0) {
                float* o = P.g_row + ((size_t)w.bb * d.h + hh) * d.T + w.t0 + r0;
                if (r0 < w.rows) o[0] = sum0;
                if (r0 + 8 < w.rows) o[8] = sum1;
            }
        } else {
            const float dt0 = dts[r0], dt1 = dts[r0 + 8], behind0 = dts[MT + r0], behind1 = dts[MT + r0 + 8];
            float a1[8][4];
            zero(a1);
#pragma unroll
            for (int kb = 0; kb < 4; ++kb) {
                if (kb < w.strip) continue;
                float v[2][4], gv[2][4], S[2][4];
                zero(v);
                scores16(S, kb);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t b[4];
                    ldsm4(b, at_cr(sY, XP, kb * 16, kk * 16));
                    mma16816(v[0], a[kk], b[0], b[1]);
                    mma16816(v[1], a[kk], b[2], b[3]);
                }
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    const int i0 = kb * 16 + u * 8 + 2 * t;
                    const float2 ci = *reinterpret_cast<const float2*>(cum + i0);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float L = exp_((c & 1 ? ci.y : ci.x) - (c < 2 ? c0 : c1));
                        gv[u][c] = S[u][c] * L;
                        v[u][c] *= (c < 2 ? dt0 : dt1) * L;
                        if (kb == w.strip && i0 + (c & 1) < r0 + (c >> 1) * 8) gv[u][c] = v[u][c] = 0.f;
                        float& s = c < 2 ? sum0 : sum1;
                        s = fmaf(v[u][c], S[u][c], s);
                    }
                }
                uint32_t f[3][4];
                cut_tiles(gv[0], gv[1], f);
                mma_cut(a1, f, sY, XP, kb * 16, 0);
                cut_tiles(v[0], v[1], f);
#pragma unroll
                for (int q = 0; q < NN / 8; q += 8) mma_cut(acc + q, f, sOther, kBP<NN>, kb * 16, q * 8);
            }
            cp_wait<0>();
            __syncthreads();
            const float w0 = r0 < w.rows ? exp_(behind0) : 0.f, w1 = r0 + 8 < w.rows ? exp_(behind1) : 0.f;
            // d_j dt_j x_j Q, to dB
#pragma unroll
            for (int q0 = 0; q0 < NN / 8; q0 += 8) {
                float o[8][4];
                rows_by_pieces<NN>(o, a, sW, q0 * 8);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    acc[q0 + q][0] = fmaf(w0 * dt0, o[q][0], acc[q0 + q][0]);
                    acc[q0 + q][1] = fmaf(w0 * dt0, o[q][1], acc[q0 + q][1]);
                    acc[q0 + q][2] = fmaf(w1 * dt1, o[q][2], acc[q0 + q][2]);
                    acc[q0 + q][3] = fmaf(w1 * dt1, o[q][3], acc[q0 + q][3]);
                }
            }
            // B_j Q^T, to dX
            float a2[8][4];
            zero(a2);
#pragma unroll
            for (int s = 2; s >= 0; --s)
#pragma unroll
                for (int kk = 0; kk < NN / 16; ++kk)
#pragma unroll
                    for (int q = 0; q < 8; q += 2) {
                        uint32_t b[4];
                        ldsm4(b, at_cr(sW + s * kBPanel<NN> * 2, kBP<NN>, q * 8, kk * 16));
                        mma16816(a2[q], rows[kk], b[0], b[1]);
                        mma16816(a2[q + 1], rows[kk], b[2], b[3]);
                    }
            const float Dh = P.D ? P.D[hh] : 0.f;
            float ddt[2] = {0.f, 0.f}, yx[2] = {0.f, 0.f}, st[2] = {0.f, 0.f};
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const int pp = q * 8 + 2 * t;
#pragma unroll
                for (int c = 0; c < 2; ++c) {
                    const int j = r0 + c * 8;
                    const float2 xv = unpack(*reinterpret_cast<const uint32_t*>(xs + j * XP + pp));
                    const float2 yv = unpack(*reinterpret_cast<const uint32_t*>(ys + j * XP + pp));
                    const float wj = c ? w1 : w0, dtj = c ? dt1 : dt0;
                    const float e0 = fmaf(wj, a2[q][2 * c], a1[q][2 * c]), e1 = fmaf(wj, a2[q][2 * c + 1], a1[q][2 * c + 1]);
                    ddt[c] = fmaf(e1, xv.y, fmaf(e0, xv.x, ddt[c]));
                    st[c] = fmaf(a2[q][2 * c + 1], xv.y, fmaf(a2[q][2 * c], xv.x, st[c]));
                    yx[c] = fmaf(yv.y, xv.y, fmaf(yv.x, xv.x, yx[c]));
                    if (j < w.rows && pp < d.p)
                        store_pair<WIDE>(P.dx + xo + (size_t)j * d.h * d.p + pp, fmaf(Dh, yv.x, e0 * dtj), fmaf(Dh, yv.y, e1 * dtj));
                }
            }
            st[0] = w0 * dt0 * quad_sum(st[0]);
            st[1] = w1 * dt1 * quad_sum(st[1]);
            if (r0 >= w.rows) st[0] = 0.f;
            if (r0 + 8 >= w.rows) st[1] = 0.f;
            store_carry(st[0] + st[1], tile);
            sum0 = quad_sum(sum0) + st[0];
            sum1 = quad_sum(sum1) + st[1];
#pragma unroll
            for (int c = 0; c < 2; ++c) {
                ddt[c] = quad_sum(ddt[c]);
                yx[c] = quad_sum(yx[c]);
                const int j = r0 + c * 8;
                if (t == 0 && j < w.rows) {
                    const size_t o = ((size_t)w.bb * d.h + hh) * d.T + w.t0 + j;
                    P.g_col[o] = c ? sum1 : sum0;
                    P.ddtx[o] = ddt[c];
                    if (P.dyx) P.dyx[o] = yx[c];
                }
            }
        }
    }
    store_bc<NN, WIDE>(P, w, acc, row_pass ? P.dC_part : P.dB_part, row_pass ? P.dC : P.dB);
}

// ------------------------------------------------------------------------------------------
// What the backward's blocks left in parts.  Blocks [0, b h): the decay gradient of one (head, batch),
//   d a_t = (sum over s >= t in its tile of g_row - g_col) + R,   R = sum over the later tiles of their state terms (+ <dfinal, final>):
// what a tile's own scores add to g_row and to g_col is the same in total, so it takes no part in the sum over the tiles, and its
// rounding stays in the tile.  (Summed over everything behind t, as on the SIMT kernels, d dt had 1.2 times the error at
// 31 tiles.)  Four tiles a step, the next values on their way meanwhile.  The blocks behind them: dB and dC of a split group.
// ------------------------------------------------------------------------------------------
constexpr int kDecayThreads = 256;
template <bool WIDE>
__global__ void __launch_bounds__(kDecayThreads) decay_kernel(Params P) {
    dep_wait();
    __shared__ float red[kDecayThreads / 32];
    const Dims& d = P.d;
    if ((int)blockIdx.x >= d.b * d.h) {
        const size_t e = ((size_t)(blockIdx.x - d.b * d.h) * kDecayThreads + threadIdx.x) * 2, total = (size_t)d.b * d.T * d.g * d.n;
        if (e >= total) return;
        const size_t o = (e / d.n) * P.splits * d.n + e % d.n;
        float2 sb = make_float2(0.f, 0.f), sc = sb;
#pragma unroll 4
        for (int s = 0; s < P.splits; ++s) {
            const float2 vb = *reinterpret_cast<const float2*>(P.dB_part + o + (size_t)s * d.n), vc = *reinterpret_cast<const float2*>(P.dC_part + o + (size_t)s * d.n);
            sb.x += vb.x;
            sb.y += vb.y;
            sc.x += vc.x;
            sc.y += vc.y;
        }
        store_pair<WIDE>(P.dB + e, sb.x, sb.y);
        store_pair<WIDE>(P.dC + e, sc.x, sc.y);
        return;
    }
    const int hh = blockIdx.x % d.h, bb = blockIdx.x / d.h, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const size_t pn = (size_t)d.p * d.n, bh = (size_t)bb * d.h + hh;
    float R = 0.f;
    if (P.dfinal) {
        float v = 0.f;
#pragma unroll 8
        for (size_t e = threadIdx.x; e < pn; e += kDecayThreads) v += P.dfinal[bh * pn + e] * P.final_state[bh * pn + e];
        R = block_sum<kDecayThreads>(v, red);
    }
    const bool form2 = P.dt != nullptr;
    const float Ah = form2 ? P.A_head[hh] : 0.f;
    const size_t base = bh * d.T;
    float dAh = 0.f, yx = 0.f;
    float n_g = 0.f, n_dx = 0.f, n_dt = 0.f, n_yx = 0.f;
    float4 n_c0, n_c1;  // thread 0 of a warp pair (tile): the state terms of its tile
    auto fetch = [&](int t, int k) {
        n_g = n_dx = n_dt = n_yx = 0.f;
        if (t >= 0 && t < d.T) {
            n_g = P.g_row[base + t] - P.g_col[base + t];
            if (form2) {
                n_dx = P.ddtx[base + t];
                n_dt = P.dt[((size_t)bb * d.T + t) * d.h + hh];
                if (P.dyx) n_yx = P.dyx[base + t];
            }
        }
        n_c0 = n_c1 = make_float4(0.f, 0.f, 0.f, 0.f);
        if (k >= 0 && k < P.nt) {
            const float4* c = reinterpret_cast<const float4*>(P.carry + tile_off(d, P.nt, bb, k, hh) * 8);
            n_c0 = c[0];
            n_c1 = c[1];
        }
    };
    // thread q handles position hi - 1 - q, so sums run toward smaller positions; two warps to a tile
    const int top = P.nt * MT;
    fetch(top - 1 - (int)threadIdx.x, P.nt - 1 - warp / 2);
    __shared__ float half[kDecayThreads / 32], state[kDecayThreads / 64];
    for (int hi = top; hi > 0; hi -= kDecayThreads) {
        const int t = hi - 1 - (int)threadIdx.x;
        const float v = n_g, dxv = n_dx, dtv = n_dt;
        const float st = ((n_c0.x + n_c0.y) + (n_c0.z + n_c0.w)) - ((n_c1.x + n_c1.y) + (n_c1.z + n_c1.w));
        yx += n_yx;
        fetch(t - kDecayThreads, (hi - kDecayThreads) / MT - 1 - warp / 2);
        float incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const float u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        __syncthreads();
        if (lane == 31) {
            half[warp] = incl;
            if (!(warp & 1)) state[warp >> 1] = st;
        }
        __syncthreads();
        float before = R;
#pragma unroll
        for (int k = 0; k < kDecayThreads / 64; ++k) {
            if (k < warp / 2) before += state[k];
            R += state[k];
        }
        const float dA = before + ((warp & 1 ? half[warp - 1] : 0.f) + incl);
        if (t >= 0 && t < d.T) {
            const size_t o = ((size_t)bb * d.T + t) * d.h + hh;
            if (form2) {
                P.ddt[o] = dxv + dA * Ah;
                dAh += dA * dtv;
            } else if (P.da) {
                P.da[o] = dA;
            }
        }
    }
    if (form2) {
        const float s = block_sum<kDecayThreads>(dAh, red);
        if (threadIdx.x == 0) P.dAh_part[bh] = s;
        if (P.dyx) {
            const float sd = block_sum<kDecayThreads>(yx, red);
            if (threadIdx.x == 0) P.dD_part[bh] = sd;
        }
    }
}

}  // namespace mma
}  // namespace ssd
