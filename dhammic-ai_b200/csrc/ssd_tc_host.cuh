// Host side of the tensor-core path: tensor maps, workspace layout and launches.
#pragma once
#include <atomic>
#include <climits>
#include <cmath>
#include <cstdio>

#include "../../include/ssd_b200.h"
#include "ssd_tc.cuh"

namespace ssd {
namespace tc {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

// The driver entry point is looked up at run time so that the library links against the CUDA
// runtime only and loads on machines without a driver.
inline EncodeTiledFn encode_fn() {
    static EncodeTiledFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess) p = nullptr;
        return (EncodeTiledFn)p;
    }();
    return fn;
}

// A bf16 tensor map with boxes of 128-byte rows, 128-byte swizzle.  The encoder belongs to the driver and wants a current context, which a
// thread that has not called the runtime yet does not have (autograd's, where the map is the first thing that a backward asks for).  Setting the
// device that is set makes its context current, and is allowed while a stream is captured.
inline bool encode_map(CUtensorMap* m, const void* base, cuuint32_t rank, const cuuint64_t* dims, const cuuint64_t* strides, const cuuint32_t* box) {
    EncodeTiledFn enc = encode_fn();
    if (!enc) return false;
    const cuuint32_t es[4] = {1, 1, 1, 1};
    auto encode = [&] {
        return enc(m, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                   CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    };
    CUresult r = encode();
    int dev = 0;
    if (r == CUDA_ERROR_INVALID_CONTEXT && cudaGetDevice(&dev) == cudaSuccess && cudaSetDevice(dev) == cudaSuccess) r = encode();
    return r == CUDA_SUCCESS;
}

// 2D bf16 tensor [rows][cols] (the saved states), box 64 columns x 128 rows, 128-byte swizzle.
inline bool make_map(CUtensorMap* m, const void* base, uint64_t rows, uint64_t cols) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, 128};
    return encode_map(m, base, 2, dims, strides, box);
}

// A (b, T, heads, inner) bf16 tensor as the tile kernels see it: boxes of 64 columns of one head x 128 positions of one
// sequence.  Keeping the dimensions apart is what makes a box that reaches behind the end of a sequence, or behind a head's
// last column, read zeros instead of the neighbour's values.
inline bool make_map4(CUtensorMap* m, const void* base, const Dims& d, int heads, int inner) {
    const cuuint64_t dims[4] = {(cuuint64_t)inner, (cuuint64_t)heads, (cuuint64_t)d.T, (cuuint64_t)d.b};
    const cuuint64_t strides[3] = {(cuuint64_t)inner * 2, (cuuint64_t)heads * inner * 2, (cuuint64_t)d.T * heads * inner * 2};
    const cuuint32_t box[4] = {64, 1, 128, 1};
    return encode_map(m, base, 4, dims, strides, box);
}

struct Ws {
    size_t status, tcum, dtT, skipT, Hst, Qst, final_state, dinit, g, ddtx, dyx, gS, dAh_part, dD_part, piece_sum, piece_decay, base, total;
};

constexpr int kPieceSms = 148, kMaxEntries = 16, kWholeWalks = 75;  // SMs; see Pieces
// The forward walks of a call's last round over the SMs (of all its pairs, where there are no more pairs than SMs), where they leave at least half the SMs idle and
// no walk is summarised (Pieces): as many CTAs a walk as there are SMs for, up to four, each of which walks the states before its own tiles for itself.  These
// take 0.8 us a tile and the piece's own 1.5, so pieces shrink by a constant factor.  Only where that saves a tenth of the walk.
// Whole -> cut, us: 44 walks behind 148 whole ones, of 4 tiles 22.8 -> 22.5, 16 tiles 58.3 -> 52.8, 64 tiles 195 -> 172, 256 tiles 742 -> 657; 72 of 16 tiles behind 148
// 60.0 -> 56.2, 4 of 256 739 -> 605; all of a call's: 24 of 2 tiles 8.1 -> 8.0, 4 tiles 10.7 -> 10.0, 8 tiles 16.2 -> 12.8, 64 of 4 tiles 11.8 -> 11.4, 16 tiles 29.0 -> 23.4.
constexpr double kTileUs = 1.5, kLeadUs = 0.8;
inline SelfCut self_cut(const Dims& d) {
    const int nt = tiles_of(d.T);
    const long long bh = (long long)d.b * d.h, rest = bh % kPieceSms;
    SelfCut best{(int)bh, 1, {0, nt}};
    if (rest == 0 || bh > INT_MAX / 4) return best;
    const double f = 1.0 - kLeadUs / kTileUs;
    double cost = 0.9 * kTileUs * nt;
    for (int np = 2; np <= 4 && np * rest <= kPieceSms && np <= nt; ++np) {
        SelfCut c{(int)(bh - rest), np, {0}};
        double len = nt * (1.0 - f) / (1.0 - std::pow(f, np)), at = 0, longest = 0;
        bool ok = true;
        for (int z = 0; z < np; ++z, len *= f) {
            at += len;
            c.cut[z + 1] = z + 1 == np ? nt : (int)(at + 0.5);
            ok = ok && c.cut[z + 1] > c.cut[z];
            longest = std::max(longest, kTileUs * (c.cut[z + 1] - c.cut[z]) + (z ? kLeadUs * c.cut[z] + 0.7 : 0.0));
        }
        if (ok && longest < cost) {
            cost = longest;
            best = c;
        }
    }
    return best;
}

// The pieces that a walk over one sequence is cut into.  A walk has one CTA per (batch, head), which is reckoned with 1.5 us per tile forward
// and 1.1 us in reverse (1.3 for two heads of a group in one CTA; 1.4, 0.97 and 1.22 with 80 CTAs); with few of them most SMs idle.  Pieces run side by side: every piece but the
// walk's last is first summarised (0.7 us per tile, 1.05 for two heads of a group, no chain, in parts that fill the chip), and a piece's CTA
// folds the summaries before its own into its seed.  Only while all CTAs fit on the chip at once, and where the tiles taken off the chain
// outweigh the summary and its launch (10 us) by a tenth.  A function of the shape alone: the workspace's size follows from it.
// No walk is cut from kWholeWalks pairs on, although reverse walks of up to 148 pairs with two heads per CTA would still gain by it ((1, 24576, 80 heads) forward and
// backward 1,157 us cut, 1,197 whole; (2, 16384, 64) 1,017, 1,019): a cut changes the order of the state gradient's sums, and a call of
// that many pairs has the same bits alone as a micro-batch of a larger one.
// One prompt of 16,384 positions and 64 heads (128 tiles): 184 us in one piece, 126 in two, 141 in two that find their own way (self_cut).
struct Pieces {
    int pt, np, ps, parts;  // tiles of a piece, pieces, tiles of a summarised part, parts of a piece
    int heads, sum_heads;   // of a group per CTA of the walk (reverse), of the summary
};
inline Pieces pieces_of(const Dims& d, bool reverse) {
    const int nt = tiles_of(d.T);
    const long long bh = (long long)d.b * d.h;
    const bool even = d.hpg % 2 == 0;
    // in one piece: two heads per CTA (shared C panels, one N = 128 product per tile) only where one head per CTA would not fit on the chip at once
    Pieces best{nt, 1, nt, 1, reverse && even && bh > kPieceSms ? 2 : 1, 1};
    double cost = 0.9 * (reverse ? 1.1 : kTileUs) * nt;
    if (bh >= kWholeWalks) return best;
    for (int heads = 1; heads <= (reverse && even ? 2 : 1); ++heads)
        for (int P = 2; P <= kMaxEntries && P * bh <= kPieceSms * heads && P <= nt; ++P)
            for (int sum_heads = 1; sum_heads <= (even ? 2 : 1); ++sum_heads) {
                const int pt = (nt + P - 1) / P, np = (nt + pt - 1) / pt;
                const long long ctas = bh / sum_heads * (np - 1);  // of the summary, for one part
                const int want = (int)std::max(1LL, std::min({(long long)pt, kPieceSms / ctas, (long long)kMaxEntries / (np - 1)}));
                const int ps = (pt + want - 1) / want, parts = (pt + ps - 1) / ps;
                if (reverse && nt - (np - 1) * pt <= (parts - 1) * ps) continue;  // the short last piece would have an empty part
                const double rounds = (double)((ctas * parts + kPieceSms - 1) / kPieceSms);
                const double c = (!reverse ? kTileUs : heads == 2 ? 1.3 : 1.1) * pt + (sum_heads == 2 ? 1.05 : 0.7) * rounds * ps + 10.0 + 0.6 * parts * (np - 1);
                if (c < cost) {
                    cost = c;
                    best = {pt, np, ps, parts, heads, sum_heads};
                }
            }
    return best;
}

// Words of the extreme-decay flags: one per tile and eight heads.
inline size_t flags_of(const Dims& d) { return (size_t)d.b * ((d.h + 7) / 8) * tiles_of(d.T); }

inline Ws ws_layout(const Dims& d, int pass) {
    Ws w{};
    size_t off = 0;
    auto take = [&](size_t bytes) {
        size_t o = off;
        off += (bytes + 255) / 256 * 256;
        return o;
    };
    const int nt = tiles_of(d.T);
    const size_t bht = (size_t)d.b * d.h * nt * LT * 4;
    const size_t bhpn = (size_t)d.b * d.h * d.p * d.n * 4;
    const size_t st = (size_t)d.b * tiles_of(d.T) * d.h * DN * HP * 2;
    w.status = take(256);
    w.tcum = take(bht);
    w.dtT = take(bht);
    w.skipT = take(bht);
    if (pass == SSD_B200_PASS_BWD) {
        w.Hst = take(st);
        w.Qst = take(st);
        w.final_state = take(bhpn);
        w.dinit = take(bhpn);
        w.g = take(bht);
        w.ddtx = take(bht);
        w.dyx = take(bht);
        w.gS = take((size_t)d.b * d.h * nt * 8 * 4);
        w.dAh_part = take((size_t)d.b * nt * d.h * 4);
        w.dD_part = take((size_t)d.b * nt * d.h * 4);
    }
    w.base = off;  // enough for a walk in one piece
    auto entries = [&](bool reverse) {
        const Pieces pc = pieces_of(d, reverse);
        return (size_t)(pc.np - 1) * pc.parts;
    };
    const size_t ne = pass == SSD_B200_PASS_BWD ? std::max(entries(false), entries(true)) : entries(false);
    if (ne > 0) {
        w.piece_sum = take(ne * bhpn);
        w.piece_decay = take(ne * d.b * d.h * 4);
    }
    w.total = off;
    return w;
}

inline size_t workspace_bytes(const Dims& d, int pass) { return ws_layout(d, pass).total; }
// The `states` buffer a forward call may fill for the backward call of the same inputs: the bf16 state entering
// every tile, followed by the three (b,h,Tp) fp32 arrays the tile kernels read (tile-cumulative log2 decay, dt and
// the per-position skip coefficient in (b,h,T) order) and the extreme-decay flags, so that the backward neither walks the states
// nor rebuilds those arrays.
inline size_t tile_states_bytes(const Dims& d) { return (size_t)d.b * tiles_of(d.T) * d.h * DN * HP * 2; }
inline size_t states_bytes(const Dims& d) { return tile_states_bytes(d) + 3 * ((size_t)d.b * d.h * tiles_of(d.T) * LT * 4) + flags_of(d) * 4; }

#define SSD_TC_FAIL(code, ...)              \
    do {                                    \
        snprintf(err, errn, __VA_ARGS__);   \
        return code;                        \
    } while (0)

#define SSD_TC_CHECK(what)                                                                        \
    do {                                                                                          \
        cudaError_t e_ = cudaGetLastError();                                                      \
        if (e_ != cudaSuccess) SSD_TC_FAIL(SSD_B200_ECUDA, "%s: %s", what, cudaGetErrorString(e_)); \
    } while (0)

inline int sm_count() {  // SMs of the current device (one persistent CTA each)
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n <= 0)
        return 148;
    return n;
}

// Opt-in shared-memory sizes of the tensor-core kernels: set once per device and process (a function attribute
// lives as long as the device's context; after cudaDeviceReset a launch fails with an error code, it does not misbehave).
inline int set_walk_attrs(char* err, size_t errn) {
    static std::atomic<unsigned long long> done{0};
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) dev = 0;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done.load(std::memory_order_acquire) & bit) return 0;
    const auto attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    cudaError_t e = cudaFuncSetAttribute(fwd_walk_kernel, attr, (int)kFwdSmem);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(states_walk_kernel, attr, (int)WalkCfg::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(rev_walk_kernel<1, false>, attr, (int)RevCfg<1>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(rev_walk_kernel<1, true>, attr, (int)RevCfg<1>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(rev_walk_kernel<2, false>, attr, (int)RevCfg<2>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(rev_walk_kernel<2, true>, attr, (int)RevCfg<2>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(summary_kernel<false, 1>, attr, (int)SumCfg<1>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(summary_kernel<true, 1>, attr, (int)SumCfg<1>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(summary_kernel<false, 2>, attr, (int)SumCfg<2>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(summary_kernel<true, 2>, attr, (int)SumCfg<2>::SMEM);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(bwd_tile_kernel, attr, (int)kBwdSmem);
    if (e != cudaSuccess) SSD_TC_FAIL(SSD_B200_ECUDA, "set shared memory size: %s", cudaGetErrorString(e));
    done.fetch_or(bit, std::memory_order_release);
    return 0;
}

inline bool cumsum_blocks_of_eight(const Dims& d) {  // see kFewCumsumBlocks
    const int eights = (d.h + 7) / 8;
    return (long long)tiles_of(d.T) * eights * d.b <= kFewCumsumBlocks || eights <= 2 * ((d.h + 31) / 32);
}

inline int launch_tile_cumsum(bool after, const Dims& d, const float* cum, const float* dt, float* tcum, float* dtT, const float* skip,
                              float* skipT, int* extreme, int* status, cudaStream_t st, char* err, size_t errn) {
    const int nt = tiles_of(d.T);
    SSD_LAUNCH(prof::K_TC_AUX, st, launch_dep(after, tile_cumsum_kernel, dim3(nt, (d.h + 7) / 8, d.b), 256, 0, st, cum, dt, tcum, dtT, skip, skipT, extreme, status, d.T,
                                              nt * LT, d.h, d.l));
    SSD_TC_CHECK("tile_cumsum");
    return 0;
}

// The same from the log-decays (`args` of a forward or a backward), and a_cumsum unless `cum` is null.
template <class Args>
inline int launch_cumsum_tile_fused(const Args* a, const Dims& d, float* cum, float* tcum, float* dtT, float* skipT, int* extreme, int* status, cudaStream_t st,
                                    char* err, size_t errn) {
    const int nt = tiles_of(d.T);
    const bool few = cumsum_blocks_of_eight(d), cut = d.l % LT != 0;  // cut: a chunk ends inside a tile
    const auto kernel = few ? (cut ? cumsum_tile_fused_kernel<true, 8> : cumsum_tile_fused_kernel<false, 8>)
                            : (cut ? cumsum_tile_fused_kernel<true, 32> : cumsum_tile_fused_kernel<false, 32>);
    SSD_LAUNCH(prof::K_CUMSUM, st, launch_dep(false, kernel, dim3(nt, few ? (d.h + 7) / 8 : (d.h + 31) / 32, d.b), 256, 0, st,
        a->a, a->shape.a_dtype == SSD_B200_BF16, a->dt, a->A_head, cum, tcum, dtT, a->skip, skipT, extreme, status, d.T, nt * LT, d.h, d.l));
    SSD_TC_CHECK("cumsum_tile_fused");
    return 0;
}

// Cuts the walk of P into pieces where that pays and the workspace has the room, and summarises them.  `after`: see launch_dep.
template <bool REV>
inline int split_walk(WalkParams& P, const Dims& d, const Ws& w, void* workspace, size_t bytes, int* pieces, bool* after, cudaStream_t st, char* err, size_t errn) {
    P.pt = P.nt;
    *pieces = 1;
    const Pieces pc = pieces_of(d, REV);
    if (pc.np == 1 || bytes < w.total || overlap(P.seed, P.out_state, (size_t)d.b * d.h * d.p * d.n * 4)) return 0;
    SummaryParams S{};
    S.mU = P.mU; S.mV = P.mV; S.tcum = P.tcum; S.dtT = P.dtT; S.out = (float*)((char*)workspace + w.piece_sum);
    S.logdecay = (float*)((char*)workspace + w.piece_decay); S.status = P.status; S.zero_status = P.zero_status; S.Tp = P.Tp; S.h = P.h; S.hpg = P.hpg; S.nt = P.nt;
    S.p = P.p; S.n = P.n; S.pt = pc.pt; S.ps = pc.ps; S.parts = pc.parts; S.z0 = REV ? 1 : 0;
    const int z = (pc.np - 1) * pc.parts;
    if (pc.sum_heads == 2)
        SSD_LAUNCH(prof::K_TC_SUMMARY, st, (launch_dep(*after, summary_kernel<REV, 2>, dim3(d.h / 2, d.b, z), SumCfg<2>::THREADS, SumCfg<2>::SMEM, st, S)));
    else
        SSD_LAUNCH(prof::K_TC_SUMMARY, st, (launch_dep(*after, summary_kernel<REV, 1>, dim3(d.h, d.b, z), SumCfg<1>::THREADS, SumCfg<1>::SMEM, st, S)));
    SSD_TC_CHECK("tc_summary_pieces");
    P.pt = pc.pt; P.parts = pc.parts; P.piece_sum = S.out; P.piece_decay = S.logdecay;
    *pieces = pc.np;
    *after = true;
    P.zero_status = 0;
    return 0;
}

inline int forward(const ssd_b200_fwd_args* a, const Dims& d, cudaStream_t st, char* err, size_t errn) {
    Ws w = ws_layout(d, SSD_B200_PASS_FWD);
    if (a->workspace_bytes < w.base) SSD_TC_FAIL(SSD_B200_EWORKSPACE, "workspace %zu < %zu", a->workspace_bytes, w.base);
    if (!encode_fn()) SSD_TC_FAIL(SSD_B200_ECUDA, "cuTensorMapEncodeTiled is not available");
    const bool states_only = (a->flags & SSD_B200_FWD_STATES_ONLY) != 0;
    for (const void* p : {a->x, a->B, a->C, (const void*)a->y})
        if ((uintptr_t)p & 15) SSD_TC_FAIL(SSD_B200_EINVAL, "tensor-core path needs 16-byte aligned tensors");
    const int nt = tiles_of(d.T), Tp = nt * LT;
    const size_t bht = (size_t)d.b * d.h * Tp;
    char* ws = (char*)a->workspace;
    int* status = (int*)(ws + w.status);
    float* tcum = (float*)(ws + w.tcum);
    float* dtT = a->dt ? (float*)(ws + w.dtT) : nullptr;
    float* skipT = a->skip ? (float*)(ws + w.skipT) : nullptr;
    int* extreme = nullptr;  // flags for the backward (see kMaskSafeLog2)
    const bool aux_valid = (a->flags & SSD_B200_FWD_AUX_VALID) != 0;
    if (aux_valid && !a->states) SSD_TC_FAIL(SSD_B200_EINVAL, "SSD_B200_FWD_AUX_VALID needs the `states` buffer that holds the arrays");
    if (a->states) {  // the per-position arrays live behind the tile states, kept for later calls on the same inputs
        tcum = (float*)((char*)a->states + tile_states_bytes(d));
        if (a->dt) dtT = tcum + bht;
        if (a->skip) skipT = tcum + 2 * bht;
        extreme = (int*)(tcum + 3 * bht);
    }
    if (!a->cumsum_is_input && !aux_valid && d.l <= kFusedChunkMax) {
        // the within-chunk cumulative sums, the tile-cumulative log2 copies, the transposes and the flags in one kernel
        if (int rc = launch_cumsum_tile_fused(a, d, a->a_cumsum, tcum, dtT, skipT, extreme, status, st, err, errn)) return rc;
    } else {
        if (!a->cumsum_is_input) {
            const size_t sm = (size_t)d.l * (d.h + 1) * 4;
            if (sm > 227 * 1024)  // (with a_cumsum given, a chunk can have any length)
                SSD_TC_FAIL(SSD_B200_EUNSUPPORTED, "chunk * nheads too large for the cumsum tile");
            if (sm > 48 * 1024 &&
                cudaFuncSetAttribute(chunk_cumsum_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) != cudaSuccess)
                SSD_TC_FAIL(SSD_B200_ECUDA, "chunk_cumsum: set shared memory size failed");
            SSD_LAUNCH(prof::K_CUMSUM, st, launch_dep(false, chunk_cumsum_kernel, dim3(d.c, d.b), 256, sm, st, 
                a->a, a->shape.a_dtype == SSD_B200_BF16, a->dt, a->A_head, a->a_cumsum, d.T, d.h, d.l));
            SSD_TC_CHECK("chunk_cumsum");
        }
        if (!aux_valid)
            if (int rc = launch_tile_cumsum(!a->cumsum_is_input, d, a->a_cumsum, a->dt, tcum, dtT, a->skip, skipT, extreme, status, st, err, errn)) return rc;
    }
    if (int rc = set_walk_attrs(err, errn)) return rc;
    bool after = !aux_valid;  // the cumulative sums are on the stream (and have cleared the status word)
    WalkParams P{};
    P.zero_status = aux_valid;
    P.skipT = skipT;
    P.ysq = a->ysq;
    bool ok = make_map4(&P.mU, a->x, d, d.h, d.p) && make_map4(&P.mV, a->B, d, d.g, d.n) && make_map4(&P.mC, a->C, d, d.g, d.n) &&
              make_map4(&P.mY, states_only ? a->x : (const void*)a->y, d, d.h, d.p);
    if (a->states && ((uintptr_t)a->states & 15)) SSD_TC_FAIL(SSD_B200_EINVAL, "`states` must be 16-byte aligned");
    if (ok && a->states && !states_only) {
        ok = make_map(&P.mS, a->states, (uint64_t)d.b * nt * d.h * DN, HP);
        P.save_states = 1;
    } else {
        P.mS = P.mY;
    }
    if (!ok) SSD_TC_FAIL(SSD_B200_ECUDA, "tensor map encoding failed");
    P.tcum = tcum; P.dtT = dtT; P.D = a->D; P.seed = a->init; P.out_state = a->final_state; P.status = status;
    P.Tp = Tp; P.h = d.h; P.hpg = d.hpg; P.nt = nt; P.p = d.p; P.n = d.n;
    if (states_only) {  // what this piece of the sequence adds to the state after it (plus the decayed seed)
        SummaryParams S{};
        S.mU = P.mU; S.mV = P.mV; S.tcum = tcum; S.dtT = dtT; S.seed = a->init; S.out = a->final_state;
        S.logdecay = a->logdecay_total; S.status = status; S.zero_status = aux_valid; S.Tp = Tp; S.h = d.h; S.hpg = d.hpg; S.nt = S.pt = S.ps = nt; S.parts = 1;
        S.p = d.p; S.n = d.n;
        if (d.hpg % 2 == 0)  // two heads of a group per CTA share the group's panels
            SSD_LAUNCH(prof::K_TC_SUMMARY, st, (launch_dep(after, summary_kernel<false, 2>, dim3(d.h / 2, d.b), SumCfg<2>::THREADS, SumCfg<2>::SMEM, st, S)));
        else
            SSD_LAUNCH(prof::K_TC_SUMMARY, st, (launch_dep(after, summary_kernel<false, 1>, dim3(d.h, d.b), SumCfg<1>::THREADS, SumCfg<1>::SMEM, st, S)));
        SSD_TC_CHECK("tc_summary_fwd");
        return 0;
    }
    int pieces;
    if (int rc = split_walk<false>(P, d, w, ws, a->workspace_bytes, &pieces, &after, st, err, errn)) return rc;
    dim3 grid(d.h, d.b, pieces);
    // (x is read again by the pieces behind, so it must not be written to either)
    if (pieces == 1 && !overlap(a->init, a->final_state, (size_t)d.b * d.h * d.p * d.n * 4) && !overlap(a->x, a->y, (size_t)d.b * d.T * d.h * d.p * 2)) {
        P.self = self_cut(d);
        if (P.self.np > 1) grid = dim3((unsigned)(P.self.whole + (d.b * d.h - P.self.whole) * P.self.np));
    }
    SSD_LAUNCH(prof::K_TC_FWD, st, launch_dep(after, fwd_walk_kernel, grid, kFwdThreads, kFwdSmem, st, P));
    SSD_TC_CHECK("tc_fwd_walk");
    if (a->logdecay_total) {
        SSD_LAUNCH(prof::K_CUMSUM, st, launch_dep(true, logdecay_total_kernel, (d.b * d.h + 127) / 128, 128, 0, st, a->a_cumsum, a->logdecay_total, d.b * d.h, d.c, d.l));
        SSD_TC_CHECK("logdecay_total");
    }
    return 0;
}

inline int backward(const ssd_b200_bwd_args* a, const Dims& d, cudaStream_t st, char* err, size_t errn) {
    Ws w = ws_layout(d, SSD_B200_PASS_BWD);
    if (a->workspace_bytes < w.base) SSD_TC_FAIL(SSD_B200_EWORKSPACE, "workspace %zu < %zu", a->workspace_bytes, w.base);
    if (!encode_fn()) SSD_TC_FAIL(SSD_B200_ECUDA, "cuTensorMapEncodeTiled is not available");
    for (const void* p : {a->x, a->B, a->C, a->dy, (const void*)a->dx, (const void*)a->dB, (const void*)a->dC})
        if ((uintptr_t)p & 15) SSD_TC_FAIL(SSD_B200_EINVAL, "tensor-core path needs 16-byte aligned tensors");
    const int nt = tiles_of(d.T), Tp = nt * LT;
    const size_t bht = (size_t)d.b * d.h * Tp;
    char* ws = (char*)a->workspace;
    int* status = (int*)(ws + w.status);
    float* tcum = (float*)(ws + w.tcum);
    float* dtT = a->dt ? (float*)(ws + w.dtT) : nullptr;
    const void* Hst = a->states ? a->states : (const void*)(ws + w.Hst);
    if ((uintptr_t)Hst & 15) SSD_TC_FAIL(SSD_B200_EINVAL, "`states` must be 16-byte aligned");
    void* Qst = ws + w.Qst;
    float* fin = (float*)(ws + w.final_state);
    float* dinit = a->dinit ? a->dinit : (float*)(ws + w.dinit);
    int* extreme = (int*)(ws + w.dAh_part);  // (written again behind the kernels that read the flags)
    float* skipT = a->skip ? (float*)(ws + w.skipT) : nullptr;
    if (a->states) {  // the forward left the arrays and the flags behind the tile states
        tcum = (float*)((uintptr_t)a->states + tile_states_bytes(d));
        dtT = a->dt ? tcum + bht : nullptr;
        skipT = a->skip ? tcum + 2 * bht : nullptr;
        extreme = (int*)(tcum + 3 * bht);
    } else {  // as the forward made them: from the log-decays, or from the sums it was given
        const bool decays = !a->cumsum_is_input && d.l <= kFusedChunkMax && (a->a || (a->dt && a->A_head));
        if (int rc = decays ? launch_cumsum_tile_fused(a, d, nullptr, tcum, dtT, skipT, extreme, status, st, err, errn)
                            : launch_tile_cumsum(false, d, a->a_cumsum, a->dt, tcum, dtT, a->skip, skipT, extreme, status, st, err, errn))
            return rc;
    }
    if (int rc = set_walk_attrs(err, errn)) return rc;
    bool after = !a->states;  // the cumulative sums are on the stream (and have cleared the status word)
    const uint64_t srows = (uint64_t)d.b * nt * d.h * DN;
    if (a->flags & SSD_B200_BWD_DINIT_ONLY) {  // d(initial state) of this piece for the given (or a zero) dfinal
        SummaryParams S{};
        if (!(make_map4(&S.mU, a->dy, d, d.h, d.p) && make_map4(&S.mV, a->C, d, d.g, d.n)))
            SSD_TC_FAIL(SSD_B200_ECUDA, "tensor map encoding failed");
        S.tcum = tcum; S.dtT = nullptr; S.seed = a->dfinal; S.out = a->dinit; S.logdecay = nullptr; S.status = status; S.zero_status = !after;
        S.Tp = Tp; S.h = d.h; S.hpg = d.hpg; S.nt = S.pt = S.ps = nt; S.parts = 1; S.p = d.p; S.n = d.n;
        if (d.hpg % 2 == 0)
            SSD_LAUNCH(prof::K_TC_SUMMARY, st, (launch_dep(after, summary_kernel<true, 2>, dim3(d.h / 2, d.b), SumCfg<2>::THREADS, SumCfg<2>::SMEM, st, S)));
        else
            SSD_LAUNCH(prof::K_TC_SUMMARY, st, (launch_dep(after, summary_kernel<true, 1>, dim3(d.h, d.b), SumCfg<1>::THREADS, SumCfg<1>::SMEM, st, S)));
        SSD_TC_CHECK("tc_summary_rev");
        return 0;
    }
    CUtensorMap mX, mdY, mB, mC, mH, mQ, mdX, mdB, mdC;
    bool ok = make_map4(&mX, a->x, d, d.h, d.p) && make_map4(&mdY, a->dy, d, d.h, d.p) && make_map4(&mB, a->B, d, d.g, d.n) &&
              make_map4(&mC, a->C, d, d.g, d.n) && make_map(&mH, Hst, srows, HP) && make_map(&mQ, Qst, srows, HP) &&
              make_map4(&mdX, a->dx, d, d.h, d.p) && make_map4(&mdB, a->dB, d, d.g, d.n) && make_map4(&mdC, a->dC, d, d.g, d.n);
    if (!ok) SSD_TC_FAIL(SSD_B200_ECUDA, "tensor map encoding failed");
    if (!a->states) {  // states entering every tile (skipped when the forward saved them)
        WalkParams P{};
        P.mU = mX; P.mV = mB; P.mC = mC; P.mY = mdX; P.mS = mH; P.save_states = 1;
        P.tcum = tcum; P.dtT = dtT; P.D = nullptr; P.seed = a->init; P.out_state = fin; P.status = status;
        P.Tp = Tp; P.h = d.h; P.hpg = d.hpg; P.nt = nt; P.p = d.p; P.n = d.n;
        int pieces;  // the same as the forward's: the states have the same bits
        if (int rc = split_walk<false>(P, d, w, ws, a->workspace_bytes, &pieces, &after, st, err, errn)) return rc;
        SSD_LAUNCH(prof::K_TC_BWD_STATE, st, (launch_dep(after, states_walk_kernel, dim3(d.h, d.b, pieces), kWalkThreads, WalkCfg::SMEM, st, P)));
        SSD_TC_CHECK("tc_bwd_state");
        after = true;
    }
    {   // reverse walk: gradient of the state leaving every tile, and d(initial state)
        WalkParams P{};
        P.mU = mdY; P.mV = mC; P.mC = mC; P.mY = mdX; P.mS = mQ; P.save_states = 1;
        P.tcum = tcum; P.dtT = nullptr; P.D = nullptr; P.seed = a->dfinal; P.out_state = dinit; P.status = status; P.zero_status = !after;
        P.Tp = Tp; P.h = d.h; P.hpg = d.hpg; P.nt = nt; P.p = d.p; P.n = d.n;
        int pieces;
        if (int rc = split_walk<true>(P, d, w, ws, a->workspace_bytes, &pieces, &after, st, err, errn)) return rc;
        const Pieces pc = pieces_of(d, true);
        const bool cut = pieces > 1, two = pc.heads == 2 && pieces == pc.np;  // (in one piece for want of room: one head per CTA)
        const auto kernel = two ? (cut ? rev_walk_kernel<2, true> : rev_walk_kernel<2, false>) : (cut ? rev_walk_kernel<1, true> : rev_walk_kernel<1, false>);
        SSD_LAUNCH(prof::K_TC_BWD_STATE, st, launch_dep(after, kernel, dim3(two ? d.h / 2 : d.h, d.b, pieces), two ? RevCfg<2>::THREADS : RevCfg<1>::THREADS,
                                                        two ? RevCfg<2>::SMEM : RevCfg<1>::SMEM, st, P));
        SSD_TC_CHECK("tc_bwd_dstate");
    }
    {
        BwdParams P{};
        P.mX = mX; P.mdY = mdY; P.mB = mB; P.mC = mC; P.mH = mH; P.mQ = mQ; P.mdX = mdX; P.mdB = mdB; P.mdC = mdC;
        P.tcum = tcum; P.dtT = dtT; P.D = a->D; P.skipT = skipT; P.g = (float*)(ws + w.g); P.ddtx = (float*)(ws + w.ddtx);
        P.dyx = (float*)(ws + w.dyx); P.status = status; P.Tp = Tp; P.h = d.h; P.n = d.n;
        P.hpg = d.hpg; P.nt = nt; P.b = d.b; P.gS = (float*)(ws + w.gS);
        P.items = nt * d.g * d.b;
        P.extreme = extreme;
        P.flags = (int)flags_of(d);
        const dim3 grid(std::min(P.items, sm_count()));
        SSD_LAUNCH(prof::K_TC_BWD, st, launch_dep(true, bwd_tile_kernel, grid, kBwdThreads, kBwdSmem, st, P));
        SSD_TC_CHECK("tc_bwd_walk");
    }
    {
        DecayTileParams P{};
        P.g = (const float*)(ws + w.g); P.ddtx = (const float*)(ws + w.ddtx); P.gS = (const float*)(ws + w.gS);
        P.dyx = (a->dt && (a->D || a->skip)) ? (const float*)(ws + w.dyx) : nullptr;
        P.dt = a->dt; P.A_head = a->A_head; P.ddt = a->ddt; P.da = a->cumsum_is_input ? nullptr : a->da;
        P.dskip = a->skip ? a->dskip : nullptr;
        P.dAh_part = (float*)(ws + w.dAh_part); P.dD_part = P.dyx ? (float*)(ws + w.dD_part) : nullptr;
        P.b = d.b; P.T = d.T; P.Tp = Tp; P.h = d.h; P.nt = nt;
        SSD_LAUNCH(prof::K_DECAY, st, launch_dep(true, decay_tile_kernel, dim3(nt, (d.h + 7) / 8, d.b), 256, 0, st, P));
        SSD_TC_CHECK("decay_grad");
        if (a->dt && a->A_head) {
            SSD_LAUNCH(prof::K_REDUCE, st, launch_dep(true, reduce_rows_kernel, dim3(d.h, a->D ? 2 : 1), 256, 0, st, 
                P.dAh_part, a->dA_head, d.b * nt, d.h, P.dD_part, a->dD));
            SSD_TC_CHECK("reduce_batch");
        }
    }
    return 0;
}

}  // namespace tc
}  // namespace ssd
