// fp32-accumulate SIMT kernels for the SSD chunked scan, forward and backward.
//
// This is the full-precision path (fp32 storage, 1e-4 parity) and the path for shapes that neither the
// tensor-core kernels nor those of ssd_mma.cuh cover.  Everything is computed in fp32 whatever the storage type.
// The algorithm per (batch, head), chunk k, in-chunk positions i, j (l per chunk):
//
//   cum_i = sum_{m<=i} a_m          S_k = cum_{l-1}
//   G     = (C B^T) o L,  L_ij = exp(cum_i - cum_j) for i >= j, 0 above      Y_diag = G X
//   Hloc  = X^T diag(exp(S_k - cum_j)) B                                      (p x n)
//   H_{k+1} = exp(S_k) H_k + Hloc_k       (H_0 = initial state)
//   Y     = Y_diag + diag(exp(cum_i)) C H_k^T   (+ D x)
//
// which restates src/kernels/ssd_scan.py:364-418 of the reference with the dense O(c^2) state
// passing (:408) replaced by the recurrence it equals, exact zeros above the diagonal instead
// of the reference's exp(-20), and no clamp (all log-decays here are <= 0).
//
// Backward (dY, dfinal given), with Q_k = dH_{k+1}:
//   dH_k = exp(S_k) Q_k + dY_k^T diag(e) C_k                 (reverse recurrence, dH_c = dfinal)
//   dG = dY X^T ; dS = dG o L ; M = dS o (C B^T)
//   dX = G^T dY + diag(d) B Q^T ;  dC = dS B + diag(e) dY H_k ;  dB = dS^T C + diag(d) X Q
//   g_t = rowsum_t(M) - colsum_t(M) + <dC_off_t, C_t> - <dB_st_t, B_t>  (+ <dfinal, final> at T-1)
//   d a_t = sum_{s >= t} g_s                                  (reverse cumsum over the sequence)
// This closed form replaces the reference's autograd re-run (src/kernels/ssd_scan.py:468-533)
// and its O(l^3)-traffic segsum backward (:123-198).
//
// What bounds these kernels at the sizes the path is used at is the number of blocks and the chain of launches, then shared
// memory.  So a block of the forward and of the backward takes as few heads of a group as it needs to fill the chip (dB and dC of a
// group are then summed over its blocks), the row and the column pass of the backward are one launch, states are kept from the forward,
// and the products read shared memory 16 bytes at a time without bank conflicts.  Forward + backward of (2, 512, 8 heads, 64,
// d_state 64, chunk 64): 665 us of kernels with one block per group and 4-byte reads, 82 us now.
//
// The decay gradient is a small difference of large row and column sums; its rounding (about 1e-5 of dA_head) follows from the
// order in which each element is summed.  That order is the same for any thread layout here: products run through k one by
// one, row and column sums through quads of columns, then a tree over the sixteen quads.
#pragma once
#include "ssd_common.cuh"

namespace ssd {
namespace simt {

constexpr int TS = 64;    // output tile edge of every block-level product
constexpr int NTHR = 256; // threads per block: 16 x 16, each owning a 4 x 4 micro-tile (rows 4 ty + r, columns 4 tx + c)

struct Params {
    Dims d;
    int lb;               // 64-row blocks per chunk
    int splits;           // blocks that share the heads of a group
    int share_ws;         // backward: the state panel takes the place of M0 and M1 (shapes that would not fit otherwise)
    const void* x;
    const float* dt;      // (b,T,h) or null
    const float* A_head;  // (h) or null
    const float* D;       // (h) or null
    const void* B;
    const void* C;
    const void* dy;
    const float* init;    // (b,h,p,n) or null
    const float* dfinal;  // (b,h,p,n) or null
    const float* cum;     // (b,h,c,l)
    float* states;        // (b,c,h,p,n): local chunk states, then states entering each chunk
    float* dstates;       // (b,c,h,p,n): local state gradients, then dH_{k+1} per chunk
    float* final_state;   // (b,h,p,n)
    float* final_keep;    // (b,h,p,n) second copy kept for the backward, or null
    float* dinit;         // (b,h,p,n) or null
    void* y;
    void* dx;
    void* dB;
    void* dC;
    float* g_row;         // (b,h,T)
    float* g_col;         // (b,h,T)
    float* ddtx;          // (b,h,T)  sum_p dX * x
    float* dyx;           // (b,h,T)  sum_p dy * x, or null
    float* da;            // (b,T,h)
    float* ddt;           // (b,T,h)
    float* dAh_part;      // (b,h)
    float* dD_part;       // (b,h)
    float* dB_part;       // (b,T,g*splits,n) fp32 when splits > 1, else null
    float* dC_part;
};

// ------------------------------------------------------------------------------------------
// Shared-memory tiles: rows of `ld` floats, ld a multiple of 32, in units of four floats; unit q of row r sits at q ^ ((r / 4) % 8), so
// that sixteen threads reading the same columns of rows 4 t + c hit different banks, and so do sixteen threads reading
// neighbouring units of one row.
// ------------------------------------------------------------------------------------------
__host__ __device__ __forceinline__ int ld_of(int cols) { return (cols + 31) / 32 * 32; }
__device__ __forceinline__ int sw(int r, int q, int ld) { return r * ld + ((q ^ ((r >> 2) & 7)) << 2); }
__device__ __forceinline__ float4 ld4(const float* t, int r, int q, int ld) { return *reinterpret_cast<const float4*>(t + sw(r, q, ld)); }
__device__ __forceinline__ float& at(float* t, int r, int c, int ld) { return t[sw(r, c >> 2, ld) + (c & 3)]; }

#define SSD_FMA4(acc, av, b)                 \
    do {                                     \
        (acc)[0] = fmaf(av, (b).x, (acc)[0]); \
        (acc)[1] = fmaf(av, (b).y, (acc)[1]); \
        (acc)[2] = fmaf(av, (b).z, (acc)[2]); \
        (acc)[3] = fmaf(av, (b).w, (acc)[3]); \
    } while (0)

// acc[r][c] += sum_k A[a0 + r][k] B[b0 + c][k], k in [ka, ka + K) of A and [0, K) of B (multiples of 4)
__device__ __forceinline__ void mma_nt(float (&acc)[4][4], const float* A, int a0, int lda, int ka, const float* B, int b0, int ldb, int K) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 a[4], b[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = ld4(A, a0 + r, (ka + k) >> 2, lda);
#pragma unroll
        for (int c = 0; c < 4; ++c) b[c] = ld4(B, b0 + c, k >> 2, ldb);
#pragma unroll
        for (int r = 0; r < 4; ++r)
#pragma unroll
            for (int c = 0; c < 4; ++c)
                acc[r][c] = fmaf(a[r].w, b[c].w, fmaf(a[r].z, b[c].z, fmaf(a[r].y, b[c].y, fmaf(a[r].x, b[c].x, acc[r][c]))));
    }
}
// acc[r][c] += sum_{k < K} A[a0 + r][k] B[k][4 bq + c]
__device__ __forceinline__ void mma_nn(float (&acc)[4][4], const float* A, int a0, int lda, const float* B, int bq, int ldb, int K) {
#pragma unroll 2
    for (int k = 0; k < K; k += 4) {
        float4 a[4];
#pragma unroll
        for (int r = 0; r < 4; ++r) a[r] = ld4(A, a0 + r, k >> 2, lda);
        const float* Bk = B + k * ldb + ((bq ^ ((k >> 2) & 7)) << 2);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 b = *reinterpret_cast<const float4*>(Bk + q * ldb);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float av = q == 0 ? a[r].x : q == 1 ? a[r].y : q == 2 ? a[r].z : a[r].w;
                SSD_FMA4(acc[r], av, b);
            }
        }
    }
}
// acc[r][c] += sum_{k0 <= k < K} A[k][4 aq + r] B[k][4 bq + c]   (k0 and K multiples of 4)
__device__ __forceinline__ void mma_tn(float (&acc)[4][4], const float* A, int aq, int lda, const float* B, int bq, int ldb, int k0, int K) {
#pragma unroll 2
    for (int k = k0; k < K; k += 4) {
        const int f = (k >> 2) & 7;
        const float* Ak = A + k * lda + ((aq ^ f) << 2);
        const float* Bk = B + k * ldb + ((bq ^ f) << 2);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const float4 a = *reinterpret_cast<const float4*>(Ak + q * lda), b = *reinterpret_cast<const float4*>(Bk + q * ldb);
            SSD_FMA4(acc[0], a.x, b);
            SSD_FMA4(acc[1], a.y, b);
            SSD_FMA4(acc[2], a.z, b);
            SSD_FMA4(acc[3], a.w, b);
        }
    }
}

__device__ __forceinline__ void zero(float (&acc)[4][4]) {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c < 4; ++c) acc[r][c] = 0.f;
}

// Four consecutive elements as floats (one wide access).
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 u = *reinterpret_cast<const uint2*>(p);
    const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.x));
    const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&u.y));
    return make_float4(a.x, a.y, b.x, b.y);
}
__device__ __forceinline__ void store4(float* p, const float (&v)[4]) { *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(__nv_bfloat16* p, const float (&v)[4]) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v[0], v[1]), b = __floats2bfloat162_rn(v[2], v[3]);
    uint2 u;
    u.x = *reinterpret_cast<const uint32_t*>(&a);
    u.y = *reinterpret_cast<const uint32_t*>(&b);
    *reinterpret_cast<uint2*>(p) = u;
}
// Whether rows of `cols` values (at a pitch of `stride`) can be moved four at a time.
template <class T>
__device__ __forceinline__ bool wide(const T* base, int cols, size_t stride) {
    return cols % 4 == 0 && stride % 4 == 0 && ((uintptr_t)base & (4 * sizeof(T) - 1)) == 0;
}
// Up to `n` of the four values v to o[0..3].
template <class T>
__device__ __forceinline__ void store_upto4(T* o, const float (&v)[4], int n, bool vec) {
    if (vec) {
        store4(o, v);
    } else {
#pragma unroll
        for (int c = 0; c < 4; ++c)
            if (c < n) o[c] = from_f<T>(v[c]);
    }
}
template <class T>
__device__ __forceinline__ float4 load_upto4(const T* p, int n, bool vec) {
    if (vec) return load4(p);
    return make_float4(n > 0 ? to_f(p[0]) : 0.f, n > 1 ? to_f(p[1]) : 0.f, n > 2 ? to_f(p[2]) : 0.f, n > 3 ? to_f(p[3]) : 0.f);
}

// `rows` rows of `cols` values (row r at src + r * stride, times scale[r] where given) into a shared tile; rows >= valid and the
// columns up to the next multiple of 4 become zero.
template <class T>
__device__ __forceinline__ void load_tile(float* dst, int ld, const T* src, size_t stride, int rows, int valid, int cols,
                                          const float* scale = nullptr) {
    const int q4 = (cols + 3) / 4;
    const bool vec = wide(src, cols, stride);
#pragma unroll 4
    for (int i = threadIdx.x; i < rows * q4; i += NTHR) {
        const int r = i / q4, q = i - r * q4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < valid) v = load_upto4(src + (size_t)r * stride + q * 4, cols - q * 4, vec);
        if (scale) {
            const float w = scale[r];
            v.x *= w; v.y *= w; v.z *= w; v.w *= w;
        }
        *reinterpret_cast<float4*>(dst + sw(r, q, ld)) = v;
    }
}

// Sum over the 16 threads (tx) that share a row; result valid in every lane of the group.
__device__ __forceinline__ float row_reduce16(float v) {
#pragma unroll
    for (int o = 8; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// ------------------------------------------------------------------------------------------
// Weighted outer-product accumulation over a chunk:
//   out[b,k,h][pp][nn] = sum_j w_j U[j,pp] V[j,nn]
// mode 0: U = x, V = B, w_j = exp(S_k - cum_j) * dt_j      (local chunk states)
// mode 1: U = dy, V = C, w_j = exp(cum_j)                  (local state gradients)
// ------------------------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(NTHR) chunk_state_kernel(Params P, int mode) {
    dep_wait_early();
    __shared__ __align__(16) float Us[TS * TS];
    __shared__ __align__(16) float Vs[TS * TS];
    __shared__ float w[TS];
    const Dims& d = P.d;
    const int ntn = (d.n + TS - 1) / TS;
    const int k = blockIdx.x % d.c, bb = blockIdx.x / d.c, hh = blockIdx.y;
    const int p0 = (blockIdx.z / ntn) * TS, n0 = (blockIdx.z % ntn) * TS;
    const int gg = hh / d.hpg;
    const T* U = (const T*)(mode == 0 ? P.x : P.dy);
    const T* V = (const T*)(mode == 0 ? P.B : P.C);
    const float* cum = P.cum + cum_off(d, bb, hh, k);
    const float S = cum[d.l - 1];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    float acc[4][4];
    zero(acc);
    for (int j0 = 0; j0 < d.l; j0 += TS) {
        const int rows = min(TS, d.l - j0), t0 = k * d.l + j0;
        if (j0) __syncthreads();
        if (threadIdx.x < TS) {
            const int j = j0 + threadIdx.x;
            float wv = 0.f;
            if (j < d.l) {
                if (mode == 0) {
                    wv = __expf(S - cum[j]);
                    if (P.dt) wv *= P.dt[((size_t)bb * d.T + k * d.l + j) * d.h + hh];
                } else {
                    wv = __expf(cum[j]);
                }
            }
            w[threadIdx.x] = wv;
        }
        load_tile(Vs, TS, V + bc_off(d, bb, t0, gg) + n0, (size_t)d.g * d.n, TS, rows, min(TS, d.n - n0));
        __syncthreads();
        load_tile(Us, TS, U + x_off(d, bb, t0, hh) + p0, (size_t)d.h * d.p, TS, rows, min(TS, d.p - p0), w);
        __syncthreads();
        mma_tn(acc, Us, ty, TS, Vs, tx, TS, 0, (rows + 3) / 4 * 4);
    }
    float* out = (mode == 0 ? P.states : P.dstates) + st_off(d, bb, k, hh);
    const int nn = n0 + tx * 4;
    const bool vec = d.n % 4 == 0;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int pp = p0 + ty * 4 + r;
        if (pp < d.p && nn < d.n) store_upto4(out + (size_t)pp * d.n + nn, acc[r], d.n - nn, vec);
    }
}

// ------------------------------------------------------------------------------------------
// Inter-chunk state passing, one thread per state element, sequential over chunks; eight chunks' values are fetched ahead
// of the chain of multiply-adds.
// forward : slot k <- H_k (state entering chunk k), H_{k+1} = exp(S_k) H_k + local_k ; final = H_c
// reverse : slot k <- Q_k = dH_{k+1},               dH_k   = exp(S_k) Q_k + local_k ; dinit = dH_0
// ------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(NTHR) state_passing_kernel(Params P, int reverse) {
    if (reverse) dep_wait_early();
    else dep_wait();  // blocks of the forward scan that come while this kernel's hold the SMs are spread unevenly
    const Dims& d = P.d;
    const size_t pn = (size_t)d.p * d.n;
    const size_t e = (size_t)blockIdx.x * NTHR + threadIdx.x;
    if (e >= pn) return;
    const int hh = blockIdx.y, bb = blockIdx.z;
    float* buf = (reverse ? P.dstates : P.states) + e;
    const float* seed = reverse ? P.dfinal : P.init;
    const size_t o = ((size_t)bb * d.h + hh) * pn + e;
    float H = seed ? seed[o] : 0.f;
    constexpr int BATCH = 8;
    for (int s0 = 0; s0 < d.c; s0 += BATCH) {
        float loc[BATCH], S[BATCH];
#pragma unroll
        for (int j = 0; j < BATCH; ++j)
            if (s0 + j < d.c) {
                const int k = reverse ? d.c - 1 - (s0 + j) : s0 + j;
                loc[j] = buf[st_off(d, bb, k, hh)];
                S[j] = P.cum[cum_off(d, bb, hh, k) + d.l - 1];
            }
#pragma unroll
        for (int j = 0; j < BATCH; ++j)
            if (s0 + j < d.c) {
                const int k = reverse ? d.c - 1 - (s0 + j) : s0 + j;
                buf[st_off(d, bb, k, hh)] = H;
                H = __expf(S[j]) * H + loc[j];
            }
    }
    float* out = reverse ? P.dinit : P.final_state;
    if (out) out[o] = H;
    if (!reverse && P.final_keep) P.final_keep[o] = H;
}

// Which rows a block of the forward or the backward works on: 64-row block `ib` of chunk k, heads h0 .. h0 + hps - 1 of group gg.
struct Where {
    int k, ib, bb, gg, sp, h0, hps;
};
__device__ __forceinline__ Where where(const Params& P) {
    Where w;
    int z = blockIdx.x;
    w.ib = z % P.lb;
    z /= P.lb;
    w.k = z % P.d.c;
    w.bb = z / P.d.c;
    w.gg = blockIdx.y / P.splits;
    w.sp = blockIdx.y % P.splits;
    w.hps = P.d.hpg / P.splits;
    w.h0 = w.gg * P.d.hpg + w.sp * w.hps;
    return w;
}
// cum of the 64 positions from j0 of a chunk, and dt of the same positions (1 without dt, 0 behind the chunk)
__device__ __forceinline__ void load_scalars(const Params& P, int bb, int hh, int k, int j0, float* cum64, float* dt64) {
    const Dims& d = P.d;
    if (threadIdx.x < TS) {
        const int j = j0 + threadIdx.x;
        const bool ok = j < d.l;
        cum64[threadIdx.x] = ok ? P.cum[cum_off(d, bb, hh, k) + j] : 0.f;
        if (dt64) dt64[threadIdx.x] = (ok && P.dt) ? P.dt[((size_t)bb * d.T + k * d.l + j) * d.h + hh] : 1.f;
    }
}

// ------------------------------------------------------------------------------------------
// Chunk scan output.  Block = 64 rows i of one (batch, chunk, split of a group); per head it loops the causal column
// blocks j <= i:  Y_i = sum_j ((C_i B_j^T) o L_ij) X_j  +  diag(e_i) C_i H_k^T  (+ D x_i).
// ------------------------------------------------------------------------------------------
template <class T, int PT>
__global__ void __launch_bounds__(NTHR) chunk_scan_kernel(Params P) {
    dep_wait_early();
    extern __shared__ __align__(16) float sm[];
    const Dims& d = P.d;
    const Where w = where(P);
    const int bb = w.bb, k = w.k, ldn = ld_of(d.n), ldp = ld_of(d.p), n4 = (d.n + 3) / 4 * 4;
    float* Cs = sm;                    // [64][ldn]
    float* Bs = Cs + TS * ldn;         // [64][ldn]
    float* Xs = Bs + TS * ldn;         // [64][ldp]
    float* Gs = Xs + TS * ldp;         // [64][64]
    float* Hs = Gs + TS * TS;          // [p][64]: 64 columns of the entering state
    float* cum_i = Hs + PT * TS * TS;  // [64] each
    float* cum_j = cum_i + TS;
    float* dt_j = cum_j + TS;
    const T* x = (const T*)P.x;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int i0 = w.ib * TS, t_i0 = k * d.l + i0;
    const int rows_i = min(TS, d.l - i0);
    load_tile(Cs, ldn, (const T*)P.C + bc_off(d, bb, t_i0, w.gg), (size_t)d.g * d.n, TS, rows_i, d.n);
    float s[4][4];
    for (int hl = 0; hl < w.hps; ++hl) {
        const int hh = w.h0 + hl;
        const float* H = P.states + st_off(d, bb, k, hh);
        float acc[PT][4][4];
#pragma unroll
        for (int q = 0; q < PT; ++q) zero(acc[q]);
        if (hl) __syncthreads();
        load_scalars(P, bb, hh, k, i0, cum_i, nullptr);
        load_tile(Hs, TS, H, d.n, d.p, d.p, min(TS, d.n));
        for (int jb = 0; jb <= w.ib; ++jb) {
            const int j0 = jb * TS, t_j0 = k * d.l + j0;
            const int rows_j = min(TS, d.l - j0);
            if (jb) __syncthreads();
            if (hl == 0 || w.ib) load_tile(Bs, ldn, (const T*)P.B + bc_off(d, bb, t_j0, w.gg), (size_t)d.g * d.n, TS, rows_j, d.n);
            load_tile(Xs, ldp, x + x_off(d, bb, t_j0, hh), (size_t)d.h * d.p, TS, rows_j, d.p);
            load_scalars(P, bb, hh, k, j0, cum_j, dt_j);
            __syncthreads();
            if (hl == 0 || w.ib) {  // a chunk of one block: C B^T serves every head of this block
                zero(s);
                mma_nt(s, Cs, ty * 4, ldn, 0, Bs, tx * 4, ldn, n4);
            }
            if (jb == 0) {  // state -> output, while the scalars of this head are fresh
                for (int n0 = 0; n0 < d.n; n0 += TS) {
                    if (n0) {
                        __syncthreads();
                        load_tile(Hs, TS, H + n0, d.n, d.p, d.p, min(TS, d.n - n0));
                        __syncthreads();
                    }
#pragma unroll
                    for (int q = 0; q < PT; ++q) mma_nt(acc[q], Cs, ty * 4, ldn, n0, Hs, q * TS + tx * 4, TS, min(TS, n4 - n0));
                }
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float e = __expf(cum_i[ty * 4 + r]);
#pragma unroll
                    for (int q = 0; q < PT; ++q)
#pragma unroll
                        for (int c = 0; c < 4; ++c) acc[q][r][c] *= e;
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float g[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int il = ty * 4 + r, jl = tx * 4 + c;
                    const bool ok = (i0 + il >= j0 + jl) && il < rows_i && jl < rows_j;
                    g[c] = ok ? s[r][c] * __expf(cum_i[il] - cum_j[jl]) * dt_j[jl] : 0.f;
                }
                *reinterpret_cast<float4*>(Gs + sw(ty * 4 + r, tx, TS)) = make_float4(g[0], g[1], g[2], g[3]);
            }
            __syncthreads();
            const int kend = jb == w.ib ? ty * 4 + 4 : TS;  // on the diagonal only the columns up to the row
#pragma unroll
            for (int q = 0; q < PT; ++q) mma_nn(acc[q], Gs, ty * 4, TS, Xs, q * 16 + tx, ldp, kend);
        }
        T* y = (T*)P.y + x_off(d, bb, t_i0, hh);
        const bool vec = wide(y, d.p, (size_t)d.h * d.p);
        const float Dh = P.D ? P.D[hh] : 0.f;
#pragma unroll
        for (int q = 0; q < PT; ++q) {
            const int pp = q * TS + tx * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int il = ty * 4 + r;
                if (il >= rows_i || pp >= d.p) continue;
                if (P.D) {  // Xs holds the block's own rows (the last column block)
                    const float4 xv = ld4(Xs, il, pp >> 2, ldp);
                    SSD_FMA4(acc[q][r], Dh, xv);
                }
                store_upto4(y + (size_t)il * d.h * d.p + pp, acc[q][r], d.p - pp, vec);
            }
        }
    }
}
__host__ inline size_t chunk_scan_smem(const Dims& d, int pt) {
    return ((size_t)2 * TS * ld_of(d.n) + TS * ld_of(d.p) + TS * TS + (size_t)pt * TS * TS + 3 * TS) * 4;
}

// ------------------------------------------------------------------------------------------
// Backward of 64 positions of one (batch, chunk, split of a group); the heads in an inner loop.  blockIdx.z = 0 is the row
// pass over the causal column blocks j <= i:
//   dC_i = sum_h [ sum_j dS_ij B_j + diag(e) dY_i H_k ],   g_row[i] = rowsum_i(M) + <dC_off_i, C_i> per head
// and blockIdx.z = 1 the column pass over the row blocks i >= j:
//   dX_j = sum_i G_ij^T dY_i + diag(d) B_j Q^T,  dB_j = sum_h [ sum_i dS_ij^T C_i + diag(d) X_j Q ],
//   g_col[j] = colsum_j(M) + <dB_st_j, B_j>,  dx = dX * dt + D * dy,  ddtx[j] = <dX_j, x_j>,  dyx[j] = <dy_j, x_j>.
// The panel Ws holds 64 columns of H (row pass) or Q (column pass) at a time.
// ------------------------------------------------------------------------------------------
template <int NTN, class T>
__device__ __forceinline__ void store_bc(const Params& P, const Where& w, int t0, int rows, const float (&acc)[NTN][4][4], float* part, T* out) {
    const Dims& d = P.d;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
#pragma unroll
    for (int q = 0; q < NTN; ++q) {
        const int nn = q * TS + tx * 4;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int il = ty * 4 + r;
            if (il >= rows || nn >= d.n) continue;
            if (part) {
                float* o = part + ((((size_t)w.bb * d.T + t0 + il) * d.g + w.gg) * P.splits + w.sp) * d.n + nn;
                store_upto4(o, acc[q][r], d.n - nn, d.n % 4 == 0);
            } else {
                T* o = out + bc_off(d, w.bb, t0 + il, w.gg) + nn;
                store_upto4(o, acc[q][r], d.n - nn, wide(o, d.n, 4));
            }
        }
    }
}

template <class T, int PT, int NTN>
__global__ void __launch_bounds__(NTHR, PT * NTN == 1 ? 2 : 1) chunk_bwd_kernel(Params P) {
    dep_wait_early();
    extern __shared__ __align__(16) float sm[];
    const Dims& d = P.d;
    const Where w = where(P);
    const int bb = w.bb, k = w.k, ldn = ld_of(d.n), ldp = ld_of(d.p), n4 = (d.n + 3) / 4 * 4, p4 = (d.p + 3) / 4 * 4;
    float* Rn = sm;                    // [64][ldn]  C_i (row pass) or B_j (column pass): the block's own positions
    float* On = Rn + TS * ldn;         // [64][ldn]  B_j or C_i: the positions it loops over
    float* Rp = On + TS * ldn;         // [64][ldp]  dY_i or X_j
    float* Op = Rp + TS * ldp;         // [64][ldp]  X_j or dY_i
    float* M0 = Op + TS * ldp;         // [64][64]   dS (row pass), dS^T (column pass)
    float* M1 = M0 + TS * TS;          // [64][64]   G^T (column pass)
    float* Ws = P.share_ws ? M0 : M1 + TS * TS;  // [p4][64]
    float* cum_r = M1 + TS * TS + (P.share_ws ? 0 : PT * TS * TS);  // [64] each: own positions, and the ones looped over
    float* dt_r = cum_r + TS;
    float* cum_o = dt_r + TS;
    float* dt_o = cum_o + TS;
    const T* x = (const T*)P.x;
    const T* dy = (const T*)P.dy;
    const T* Bp = (const T*)P.B;
    const T* Cp = (const T*)P.C;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int r0 = w.ib * TS, t_r0 = k * d.l + r0;
    const int rows_r = min(TS, d.l - r0);
    const bool row_pass = blockIdx.z == 0;
    const size_t xs = (size_t)d.h * d.p, bs = (size_t)d.g * d.n;
    float acc[NTN][4][4];  // dC_i or dB_j
#pragma unroll
    for (int q = 0; q < NTN; ++q) zero(acc[q]);
    load_tile(Rn, ldn, (row_pass ? Cp : Bp) + bc_off(d, bb, t_r0, w.gg), bs, TS, rows_r, d.n);
    float s[4][4];

    if (row_pass) {
        for (int hl = 0; hl < w.hps; ++hl) {
            const int hh = w.h0 + hl;
            const float* H = P.states + st_off(d, bb, k, hh);
            float rowacc[4] = {0.f, 0.f, 0.f, 0.f};
            if (hl) __syncthreads();
            load_tile(Rp, ldp, dy + x_off(d, bb, t_r0, hh), xs, TS, rows_r, d.p);
            if (!P.share_ws) load_tile(Ws, TS, H, d.n, p4, d.p, min(TS, d.n));
            load_scalars(P, bb, hh, k, r0, cum_r, nullptr);
            for (int jb = 0; jb <= w.ib; ++jb) {
                const int j0 = jb * TS, t_j0 = k * d.l + j0;
                const int rows_j = min(TS, d.l - j0);
                if (jb) __syncthreads();
                load_scalars(P, bb, hh, k, j0, cum_o, dt_o);
                if (hl == 0 || w.ib) load_tile(On, ldn, Bp + bc_off(d, bb, t_j0, w.gg), bs, TS, rows_j, d.n);
                __syncthreads();
                load_tile(Op, ldp, x + x_off(d, bb, t_j0, hh), xs, TS, rows_j, d.p, P.dt ? dt_o : nullptr);
                if (hl == 0 || w.ib) {
                    zero(s);
                    mma_nt(s, Rn, ty * 4, ldn, 0, On, tx * 4, ldn, n4);
                }
                __syncthreads();
                float dg[4][4];
                zero(dg);
                mma_nt(dg, Rp, ty * 4, ldp, 0, Op, tx * 4, ldp, p4);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    float v[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const int il = ty * 4 + r, jl = tx * 4 + c;
                        const bool ok = (r0 + il >= j0 + jl) && il < rows_r && jl < rows_j;
                        v[c] = ok ? dg[r][c] * __expf(cum_r[il] - cum_o[jl]) : 0.f;
                        rowacc[r] = fmaf(v[c], s[r][c], rowacc[r]);
                    }
                    *reinterpret_cast<float4*>(M0 + sw(ty * 4 + r, tx, TS)) = make_float4(v[0], v[1], v[2], v[3]);
                }
                __syncthreads();
                const int kend = jb == w.ib ? ty * 4 + 4 : TS;  // on the diagonal only the columns up to the row
#pragma unroll
                for (int q = 0; q < NTN; ++q)
                    if (q * TS < d.n) mma_nn(acc[q], M0, ty * 4, TS, On, q * 16 + tx, ldn, kend);
            }
            // state term: dC_off = diag(e) dY_i H_k
#pragma unroll
            for (int q = 0; q < NTN; ++q) {
                if (q * TS >= d.n) break;
                if (q || P.share_ws) {
                    __syncthreads();
                    load_tile(Ws, TS, H + q * TS, d.n, p4, d.p, min(TS, d.n - q * TS));
                    __syncthreads();
                }
                float o[4][4];
                zero(o);
                mma_nn(o, Rp, ty * 4, ldp, Ws, tx, TS, p4);
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const float e = __expf(cum_r[ty * 4 + r]);
                    const float4 cv = ld4(Rn, ty * 4 + r, q * 16 + tx, ldn);
                    const float cc[4] = {cv.x, cv.y, cv.z, cv.w};
#pragma unroll
                    for (int c = 0; c < 4; ++c)
                        if (q * TS + tx * 4 + c < d.n) {
                            const float v = e * o[r][c];
                            acc[q][r][c] += v;
                            rowacc[r] = fmaf(v, cc[c], rowacc[r]);
                        }
                }
            }
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float v = row_reduce16(rowacc[r]);
                const int il = ty * 4 + r;
                if (tx == 0 && il < rows_r) P.g_row[((size_t)bb * d.h + hh) * d.T + t_r0 + il] = v;
            }
        }
        store_bc<NTN, T>(P, w, t_r0, rows_r, acc, P.dC_part, (T*)P.dC);
        return;
    }

    for (int hl = 0; hl < w.hps; ++hl) {
        const int hh = w.h0 + hl;
        const float* Q = P.dstates + st_off(d, bb, k, hh);
        const float S = P.cum[cum_off(d, bb, hh, k) + d.l - 1];
        float colacc[4] = {0.f, 0.f, 0.f, 0.f};
        float a1[PT][4][4];
#pragma unroll
        for (int q = 0; q < PT; ++q) zero(a1[q]);
        if (hl) __syncthreads();
        load_scalars(P, bb, hh, k, r0, cum_r, dt_r);
        if (!P.share_ws) load_tile(Ws, TS, Q, d.n, p4, d.p, min(TS, d.n));
        __syncthreads();
        load_tile(Rp, ldp, x + x_off(d, bb, t_r0, hh), xs, TS, rows_r, d.p, P.dt ? dt_r : nullptr);
        for (int ib = w.ib; ib < P.lb; ++ib) {
            const int i0 = ib * TS, t_i0 = k * d.l + i0;
            const int rows_i = min(TS, d.l - i0);
            if (ib > w.ib) __syncthreads();
            if (hl == 0 || P.lb > 1) load_tile(On, ldn, Cp + bc_off(d, bb, t_i0, w.gg), bs, TS, rows_i, d.n);
            load_tile(Op, ldp, dy + x_off(d, bb, t_i0, hh), xs, TS, rows_i, d.p);
            load_scalars(P, bb, hh, k, i0, cum_o, nullptr);
            __syncthreads();
            if (hl == 0 || P.lb > 1) {  // transposed: rows j, columns i
                zero(s);
                mma_nt(s, Rn, ty * 4, ldn, 0, On, tx * 4, ldn, n4);
            }
            float dg[4][4];
            zero(dg);
            mma_nt(dg, Rp, ty * 4, ldp, 0, Op, tx * 4, ldp, p4);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                float gv[4], v[4];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const int jl = ty * 4 + r, il = tx * 4 + c;
                    const bool ok = (i0 + il >= r0 + jl) && il < rows_i && jl < rows_r;
                    const float L = ok ? __expf(cum_o[il] - cum_r[jl]) : 0.f;
                    v[c] = dg[r][c] * L;
                    colacc[r] = fmaf(v[c], s[r][c], colacc[r]);
                    gv[c] = s[r][c] * L;
                }
                *reinterpret_cast<float4*>(M0 + sw(ty * 4 + r, tx, TS)) = make_float4(v[0], v[1], v[2], v[3]);
                *reinterpret_cast<float4*>(M1 + sw(ty * 4 + r, tx, TS)) = make_float4(gv[0], gv[1], gv[2], gv[3]);
            }
            __syncthreads();
#pragma unroll
            for (int q = 0; q < PT; ++q) mma_nn(a1[q], M1, ty * 4, TS, Op, q * 16 + tx, ldp, TS);
#pragma unroll
            for (int q = 0; q < NTN; ++q)
                if (q * TS < d.n) mma_nn(acc[q], M0, ty * 4, TS, On, q * 16 + tx, ldn, TS);
        }
        // state terms with Q_k = dH_{k+1}
        float dj[4], a2[PT][4][4];
#pragma unroll
        for (int q = 0; q < PT; ++q) zero(a2[q]);
#pragma unroll
        for (int r = 0; r < 4; ++r) dj[r] = (ty * 4 + r) < rows_r ? __expf(S - cum_r[ty * 4 + r]) : 0.f;
#pragma unroll
        for (int q = 0; q < NTN; ++q) {
            if (q * TS >= d.n) break;
            if (q || P.share_ws) {
                __syncthreads();
                load_tile(Ws, TS, Q + q * TS, d.n, p4, d.p, min(TS, d.n - q * TS));
                __syncthreads();
            }
#pragma unroll
            for (int pq = 0; pq < PT; ++pq) mma_nt(a2[pq], Rn, ty * 4, ldn, q * TS, Ws, pq * TS + tx * 4, TS, min(TS, n4 - q * TS));
            float o[4][4];
            zero(o);
            mma_nn(o, Rp, ty * 4, ldp, Ws, tx, TS, p4);
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const float4 bv = ld4(Rn, ty * 4 + r, q * 16 + tx, ldn);
                const float bc[4] = {bv.x, bv.y, bv.z, bv.w};
#pragma unroll
                for (int c = 0; c < 4; ++c)
                    if (q * TS + tx * 4 + c < d.n) {
                        const float v = dj[r] * o[r][c];
                        acc[q][r][c] += v;
                        colacc[r] = fmaf(v, bc[c], colacc[r]);
                    }
            }
        }
        // per-head outputs; x and dy come back from memory as they were given (Rp holds x dt)
        const size_t xo = x_off(d, bb, t_r0, hh);
        T* dxo = (T*)P.dx + xo;
        const float Dh = P.D ? P.D[hh] : 0.f;
        const bool vec = wide(dxo, d.p, xs) && wide(x + xo, d.p, xs) && wide(dy + xo, d.p, xs);
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int jl = ty * 4 + r;
            float ddt = 0.f, yx = 0.f;
            const float dtj = dt_r[jl];
#pragma unroll
            for (int q = 0; q < PT; ++q) {
                const int pp = q * TS + tx * 4;
                if (jl >= rows_r || pp >= d.p) continue;
                const size_t o = (size_t)jl * xs + pp;
                const float4 xv = load_upto4(x + xo + o, d.p - pp, vec);
                const float xc[4] = {xv.x, xv.y, xv.z, xv.w};
                float yc[4] = {0.f, 0.f, 0.f, 0.f}, v[4];
                if (P.D) {
                    const float4 yv = load_upto4(dy + xo + o, d.p - pp, vec);
                    yc[0] = yv.x; yc[1] = yv.y; yc[2] = yv.z; yc[3] = yv.w;
                }
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    v[c] = 0.f;
                    if (pp + c < d.p) {
                        const float e = fmaf(dj[r], a2[q][r][c], a1[q][r][c]);
                        ddt = fmaf(e, xc[c], ddt);
                        yx = fmaf(yc[c], xc[c], yx);
                        v[c] = fmaf(Dh, yc[c], e * dtj);
                    }
                }
                store_upto4(dxo + o, v, d.p - pp, vec);
            }
            const float gc = row_reduce16(colacc[r]);
            ddt = row_reduce16(ddt);
            yx = row_reduce16(yx);
            if (tx == 0 && jl < rows_r) {
                const size_t o = ((size_t)bb * d.h + hh) * d.T + t_r0 + jl;
                P.g_col[o] = gc;
                P.ddtx[o] = ddt;
                if (P.dyx) P.dyx[o] = yx;
            }
        }
    }
    store_bc<NTN, T>(P, w, t_r0, rows_r, acc, P.dB_part, (T*)P.dB);
}
__host__ inline size_t chunk_bwd_smem(const Dims& d, int pt, bool share_ws) {
    return ((size_t)2 * TS * ld_of(d.n) + 2 * TS * ld_of(d.p) + 2 * TS * TS + (size_t)(share_ws ? 0 : pt) * TS * TS + 4 * TS) * 4;
}

// ------------------------------------------------------------------------------------------
// What the backward's blocks left in parts.  Blocks [0, b h): the decay gradient of one (head, batch),
// g = g_row - g_col (+ <dfinal, final> at T-1), d a_t = reverse inclusive cumsum of g over the whole sequence (tiles of 256
// with a carry, warp-shuffle scan inside a tile; the next tile's values are on their way meanwhile).  Operator form writes da;
// Mamba-2 form writes ddt = ddtx + da * A_head and the per-(batch, head) partials of dA_head and dD.  The blocks behind them:
// dB and dC summed over the splits of a group, four elements per thread, in a fixed order.
// ------------------------------------------------------------------------------------------
template <class T>
__global__ void __launch_bounds__(NTHR) decay_grad_kernel(Params P) {
    dep_wait_early();
    __shared__ float red[NTHR / 32];
    __shared__ float wsum[NTHR / 32];
    const Dims& d = P.d;
    if ((int)blockIdx.x >= d.b * d.h) {
        const size_t e = ((size_t)(blockIdx.x - d.b * d.h) * NTHR + threadIdx.x), total = (size_t)d.b * d.T * d.g * d.n;
        if (e >= total) return;
        const size_t o = (e / d.n) * P.splits * d.n + e % d.n;
        float sb = 0.f, sc = 0.f;
#pragma unroll 4
        for (int s = 0; s < P.splits; ++s) {
            sb += P.dB_part[o + (size_t)s * d.n];
            sc += P.dC_part[o + (size_t)s * d.n];
        }
        ((T*)P.dB)[e] = from_f<T>(sb);
        ((T*)P.dC)[e] = from_f<T>(sc);
        return;
    }
    const int hh = blockIdx.x % d.h, bb = blockIdx.x / d.h;
    const size_t pn = (size_t)d.p * d.n;
    float gfin = 0.f;
    if (P.dfinal) {
        const float* a = P.dfinal + ((size_t)bb * d.h + hh) * pn;
        const float* f = P.final_state + ((size_t)bb * d.h + hh) * pn;
        float v = 0.f;
#pragma unroll 8
        for (size_t e = threadIdx.x; e < pn; e += NTHR) v += a[e] * f[e];
        gfin = block_sum<NTHR>(v, red);
    }
    const size_t base = ((size_t)bb * d.h + hh) * d.T;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float carry = 0.f, dAh = 0.f, yx = 0.f;
    const float Ah = P.dt ? P.A_head[hh] : 0.f;
    const bool form2 = P.dt != nullptr;
    float n_row = 0.f, n_col = 0.f, n_dx = 0.f, n_dt = 0.f, n_yx = 0.f;
    auto fetch = [&](int t) {
        if (t < 0) return;
        n_row = P.g_row[base + t];
        n_col = P.g_col[base + t];
        if (form2) {
            n_dx = P.ddtx[base + t];
            n_dt = P.dt[((size_t)bb * d.T + t) * d.h + hh];
            if (P.dyx) n_yx = P.dyx[base + t];
        }
    };
    fetch(d.T - 1 - (int)threadIdx.x);
    for (int hi = d.T; hi > 0; hi -= NTHR) {
        // thread q handles t = hi-1-q, so the scan runs toward smaller t
        const int t = hi - 1 - (int)threadIdx.x;
        const float dxv = n_dx, dtv = n_dt;
        float v = 0.f;
        if (t >= 0) {
            v = n_row;
            v -= n_col;
            if (t == d.T - 1) v += gfin;
            yx += n_yx;
        }
        fetch(t - NTHR);
        float incl = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            float u = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= o) incl += u;
        }
        __syncthreads();
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        float pre = 0.f, tot = 0.f;
        for (int w = 0; w < NTHR / 32; ++w) {
            if (w < warp) pre += wsum[w];
            tot += wsum[w];
        }
        const float dA = carry + pre + incl;
        carry += tot;
        if (t >= 0) {
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
        const float s = block_sum<NTHR>(dAh, red);
        if (threadIdx.x == 0) P.dAh_part[(size_t)bb * d.h + hh] = s;
        if (P.dyx) {
            const float sd = block_sum<NTHR>(yx, red);
            if (threadIdx.x == 0) P.dD_part[(size_t)bb * d.h + hh] = sd;
        }
    }
}

// out[hh] = sum_b part[b,hh]   (fixed order: deterministic); dA_head, and dD by the blocks with blockIdx.y = 1
__global__ void reduce_batch_kernel(const float* part, float* out, const float* part2, float* out2, int b, int h) {
    dep_wait_early();
    int hh = blockIdx.x * blockDim.x + threadIdx.x;
    if (hh >= h) return;
    if (blockIdx.y) {
        part = part2;
        out = out2;
    }
    float s = 0.f;
    for (int bb = 0; bb < b; ++bb) s += part[(size_t)bb * h + hh];
    out[hh] = s;
}

// ------------------------------------------------------------------------------------------
// The reference's cache tensors, rebuilt from the chunk cumsum on request
// (src/kernels/ssd_scan.py:53-55, :371-382, :399-406): masked entries are exp(-20) there.
// ------------------------------------------------------------------------------------------
template <class T>
__global__ void cache_L_kernel(const float* cum, T* L, size_t chunks, int l) {
    const size_t m = blockIdx.x;  // (b,h,c) flattened
    if (m >= chunks) return;
    const float* cu = cum + m * l;
    T* out = L + m * (size_t)l * l;
    for (int idx = threadIdx.x; idx < l * l; idx += blockDim.x) {
        int i = idx / l, j = idx - i * l;
        float v = i >= j ? fminf(fmaxf(cu[i] - cu[j], -20.f), 20.f) : -20.f;
        out[idx] = from_f<T>(__expf(v));
    }
}

template <class T>
__global__ void cache_decay_chunk_kernel(const float* cum, T* dc, int c, int l) {
    const size_t m = blockIdx.x;  // (b,h) flattened
    const float* cu = cum + m * (size_t)c * l;
    T* out = dc + m * (size_t)(c + 1) * (c + 1);
    const int z = blockIdx.y;  // row
    // padded totals Z_0 = 0, Z_m = S_{m-1};  entry (z,k) = sum_{m=k+1..z} Z_m for z >= k
    for (int kk = threadIdx.x; kk <= c; kk += blockDim.x) {
        float v;
        if (z >= kk) {
            float s = 0.f;
            for (int mm = kk + 1; mm <= z; ++mm) s += cu[(size_t)(mm - 1) * l + l - 1];
            v = fminf(fmaxf(s, -20.f), 20.f);
        } else {
            v = -20.f;
        }
        out[(size_t)z * (c + 1) + kk] = from_f<T>(__expf(v));
    }
}

// Sequence-parallel prefix over per-piece summaries (all in this GPU's memory).  The sequence is cut into
// R * S consecutive pieces, piece index g = r * S + s (rank r, segment s of that rank).  Rank r's summaries sit at
// pieces + r * rank_stride as (b, S, h, pn) and its total log-decays at logp + r * logp_stride as (b, S, h).
// One launch writes, for the S pieces of `rank`, the state entering each piece (forward) or the state gradient
// leaving it (reverse) into out (b, S, h, pn); every piece is read once:
//     forward   acc = edge;  for g = 0 ..        : out[g] = acc;  acc = exp(logp[g]) acc + pieces[g]
//     reverse   acc = edge;  for g = R S - 1 .. : out[g] = acc;  acc = exp(logp[g]) acc + pieces[g]
// `edge` (b, h, pn) or null: the state before the first piece / the gradient behind the last one.  With `outer` given the
// walk is preceded by the slice summaries of the other ranks (one per rank, `outer_n` of them, this rank at `outer_rank`),
// so that the rank-level and the segment-level prefix of the sequence split are one launch.  `total` (b, h, pn)
// or null receives acc after the last of rank's pieces has been folded in (the summary of everything walked so far)
// and `total_logp` (b, h) or null the sum of the log-decays of rank's own S pieces.
__global__ void __launch_bounds__(256) state_prefix_all_kernel(const float* __restrict__ pieces, const float* __restrict__ logp,
                                        const float* __restrict__ edge, float* __restrict__ out, float* __restrict__ total,
                                        float* __restrict__ total_logp, int R, int rank, int S, int h, size_t pn,
                                        size_t rank_stride, size_t logp_stride, int reverse,
                                        const float* __restrict__ outer, const float* __restrict__ outer_logp, int outer_n,
                                        int outer_rank, size_t outer_stride, size_t outer_logp_stride) {
    const size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int m = blockIdx.y;  // (b,h)
    if (e >= pn) return;
    const int bb = m / h, hh = m - bb * h;
    float acc = edge ? edge[(size_t)m * pn + e] : 0.f;
    if (outer) {
        // first the summaries of the other ranks' whole slices (one (b, h, pn) block and one (b, h) log-decay per rank):
        // forward those before `outer_rank`, reverse those behind it; `edge` lies beyond all of them
        const int n = reverse ? outer_n - 1 - outer_rank : outer_rank;
        for (int i = 0; i < n; ++i) {
            const size_t q = (size_t)(reverse ? outer_n - 1 - i : i);
            acc = __expf(outer_logp[q * outer_logp_stride + m]) * acc + outer[q * outer_stride + (size_t)m * pn + e];
        }
    }
    const int lo = rank * S, hi = lo + S;
    float lsum = 0.f;
    // pieces walked: forward 0 .. hi-1, reverse R S - 1 .. lo.  (r, sg) = rank and segment of the piece of a step, kept
    // incrementally (no division in the loop); a piece's (b, S, h) record inside its rank's block is (bb S + sg) h + hh.
    const int steps = reverse ? R * S - lo : hi;
    const size_t rec0 = (size_t)bb * S * h + hh;
    int r = reverse ? R - 1 : 0, sg = reverse ? S - 1 : 0;
    // The recurrence is a chain of dependent multiply-adds, but its operands are not: they are fetched a batch at a
    // time (eight loads in flight per thread) before the chain consumes them.
    constexpr int BATCH = 8;
    for (int i0 = 0; i0 < steps; i0 += BATCH) {
        float v[BATCH], lp[BATCH];
        int rr = r, ss = sg;
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            if (i0 + j < steps) {
                const size_t rc = rec0 + (size_t)ss * h;
                lp[j] = logp[(size_t)rr * logp_stride + rc];
                v[j] = pieces[(size_t)rr * rank_stride + rc * pn + e];
                if (reverse) { if (--ss < 0) { ss = S - 1; --rr; } } else { if (++ss == S) { ss = 0; ++rr; } }
            }
        }
#pragma unroll
        for (int j = 0; j < BATCH; ++j) {
            if (i0 + j < steps) {
                const bool own = r == rank;
                if (own && out) out[(rec0 + (size_t)sg * h) * pn + e] = acc;
                if (own) lsum += lp[j];
                acc = __expf(lp[j]) * acc + v[j];
                if (reverse) { if (--sg < 0) { sg = S - 1; --r; } } else { if (++sg == S) { sg = 0; ++r; } }
            }
        }
    }
    if (total) total[(size_t)m * pn + e] = acc;
    if (total_logp && e == 0) total_logp[m] = lsum;
}

// ------------------------------------------------------------------------------------------
// Exchange of the per-rank summaries by direct stores into the other GPUs' memory (NVLink peer access), for the
// sequence-parallel schedule: every rank owns a receive buffer with one slot per source rank and a row of arrival
// counters; `bufs[q]` / `flags[q]` are rank q's buffer and counters as mapped into this process.
//
// push:    copy the local block into slot `rank` of every rank's buffer (plain 16-byte stores; own buffer included).
// arrive:  one thread per peer: after a system-wide fence (the push kernel before it on the stream has completed, so
//          its stores are performed), store this step's epoch into counter `rank` of peer q, then wait until peer q's
//          epoch shows up in the local counter q.  The wait is bounded; when it runs out the kernel records it in
//          `status` and returns (the gathered data is then invalid, nothing hangs).
__global__ void __launch_bounds__(256) exchange_push_kernel(const float4* __restrict__ src, size_t n4, float* const* bufs, int R,
                                                            size_t dst_offset) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n4) return;
    const float4 v = src[i];
    for (int q = 0; q < R; ++q) reinterpret_cast<float4*>(bufs[q] + dst_offset)[i] = v;
}

__global__ void __launch_bounds__(32) exchange_arrive_kernel(unsigned int* const* flags, int rank, int R, unsigned int epoch,
                                                             int* status, unsigned int max_polls) {
    const int q = threadIdx.x;
    if (q >= R) return;
    __threadfence_system();
    volatile unsigned int* theirs = flags[q] + rank;
    *theirs = epoch;
    __threadfence_system();
    volatile unsigned int* mine = flags[rank] + q;
    bool ok = false;
    for (unsigned int i = 0; i < max_polls; ++i) {
        // epochs only grow; a later one means the peer is already a step ahead, which also covers this step
        if ((int)(*mine - epoch) >= 0) { ok = true; break; }
        __nanosleep(64);
    }
    if (!ok) atomicExch(status, 3);
    __threadfence_system();
}

}  // namespace simt
}  // namespace ssd
