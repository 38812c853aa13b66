// Thin wrappers over the sm_100a PTX used by the tensor-core kernels: mbarrier, TMA
// (cp.async.bulk.tensor, no cluster multicast anywhere), tcgen05 MMA / TMEM, and the
// shared-memory / instruction descriptors of tcgen05.mma.
//
// Every wait for an mbarrier is bounded: one that runs out clears a word of the block (`alive`), on which all others give up too, and which the block turns into
// an error status at its end (no trap, no endless spin).  Hardware barriers know no limit; until_taken keeps them from waiting for good in such a block.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ssd {
namespace ptx {

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---------------------------------------------------------------- mbarrier
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_fence_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Arrive from the threads whose `pred` is set, as a predicated instruction: no branch, so a warp in which one lane
// arrives for all stays converged (a divergent arrive may be scheduled long after the other lanes have moved on).
__device__ __forceinline__ void mbar_arrive_if(uint64_t* bar, bool pred) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %1, 0;\n\t"
        "@p mbarrier.arrive.shared::cta.b64 _, [%0];\n\t}"
        ::"r"(smem_u32(bar)), "r"((uint32_t)pred)
        : "memory");
}
// One arrival for the whole (converged) warp: every lane has fenced its own writes, the warp meets, lane 0 arrives.
__device__ __forceinline__ void mbar_arrive_warp(uint64_t* bar) {
    __syncwarp();
    mbar_arrive_if(bar, (threadIdx.x & 31) == 0);
}
// Bounded waits: they give up when the limit is reached or when another wait of this block has given up (*alive, in shared memory and above zero until
// then, is zero), so a broken pipeline drains quickly instead of spinning.  Written out because their size counts: left to the compiler a wait is four polls
// and 50 instructions, and the tile kernels, whose warps run some ten loops at once, no longer fit the instruction cache.
constexpr uint32_t kSpinLimit = 4u << 20;
#define SSD_MBAR_WAIT(poll)                                                                 \
    asm volatile(                                                                           \
        "{\n\t.reg .pred p;\n\t.reg .b32 n, f;\n\t"                                         \
        "mov.b32 n, %3;\n"                                                                  \
        "WAIT:\n\t"                                                                         \
        "mbarrier." poll ".parity.shared::cta.b64 p, [%0], %1;\n\t"                         \
        "@p bra DONE;\n\t"                                                                  \
        "ld.volatile.shared.b32 f, [%2];\n\t"                                               \
        "setp.le.s32 p, f, 0;\n\t"                                                          \
        "@p bra DONE;\n\t"                                                                  \
        "add.s32 n, n, -1;\n\t"                                                             \
        "setp.ne.b32 p, n, 0;\n\t"                                                          \
        "@p bra WAIT;\n\t"                                                                  \
        "mov.b32 f, 0;\n\t"                                                                 \
        "st.volatile.shared.b32 [%2], f;\n"                                                 \
        "DONE:\n\t}"                                                                        \
        ::"r"(smem_u32(bar)), "r"(parity), "r"(smem_u32((const void*)alive)), "r"(limit)    \
        : "memory")
__device__ __forceinline__ void mbar_wait(uint64_t* bar, uint32_t parity, volatile int* alive, uint32_t limit = kSpinLimit) {
    SSD_MBAR_WAIT("try_wait");
}
// The same for phases that other threads complete with mbarrier.arrive: polls without suspending.  (try_wait may suspend the thread for a
// system-chosen time while the phase is open; a waiter that polled just before the last arrive of OTHER THREADS saw the phase about
// 0.75 us late, while completions by tcgen05.commit or TMA bytes woke it at once.)
__device__ __forceinline__ void mbar_wait_spin(uint64_t* bar, uint32_t parity, volatile int* alive, uint32_t limit = 16u * kSpinLimit) {
    SSD_MBAR_WAIT("test_wait");
}
#undef SSD_MBAR_WAIT
__device__ __forceinline__ bool gave_up(const volatile int* alive) { return *alive <= 0; }
// The end of a block, every thread's: what it reports; and where a wait gave up, a millisecond in which copies that are still on their way land before its
// shared memory is another block's.
__device__ __forceinline__ void end_of_waits(const volatile int* alive, int* status) {
    if (!gave_up(alive)) return;
    if (threadIdx.x == 0) atomicExch(status, 1);
#pragma unroll 1
    for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

// ---------------------------------------------------------------- proxy fences
__device__ __forceinline__ void fence_async_smem() {  // generic-proxy smem writes -> visible to TMA / tcgen05
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

// ---------------------------------------------------------------- TMA (tiled, no multicast)
// [rows][64] tensors (the saved states)
__device__ __forceinline__ void tma_load_2d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int x, int y) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(x), "r"(y)
        : "memory");
}
// [batch][position][head][column] tensors: a box is 64 columns of one head and 128 positions of one sequence; positions
// behind the end of the sequence and columns behind the head's last read as zero.
__device__ __forceinline__ void tma_load_4d(void* smem_dst, const CUtensorMap* map, uint64_t* bar, int col, int head, int pos, int batch) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], [%2];"
        ::"r"(smem_u32(smem_dst)), "l"(map), "r"(smem_u32(bar)), "r"(col), "r"(head), "r"(pos), "r"(batch)
        : "memory");
}
// Such a box into the L2 only.
__device__ __forceinline__ void tma_prefetch_2d(const CUtensorMap* map, int x, int y) {
    asm volatile("cp.async.bulk.prefetch.tensor.2d.L2.global.tile [%0, {%1, %2}];" ::"l"(map), "r"(x), "r"(y) : "memory");
}
__device__ __forceinline__ void tma_prefetch_4d(const CUtensorMap* map, int col, int head, int pos, int batch) {
    asm volatile("cp.async.bulk.prefetch.tensor.4d.L2.global.tile [%0, {%1, %2, %3, %4}];" ::"l"(map), "r"(col), "r"(head), "r"(pos), "r"(batch) : "memory");
}
// `bytes` of contiguous memory, both addresses and the size multiples of 16.
__device__ __forceinline__ void bulk_load(void* smem_dst, const void* gsrc, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(smem_u32(smem_dst)), "l"(gsrc), "r"(bytes),
                 "r"(smem_u32(bar))
                 : "memory");
}
// The store of such a box; what lies outside the tensor is not written.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap* map, const void* smem_src, int col, int head, int pos, int batch) {
    asm volatile("cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
                 "r"(smem_u32(smem_src)), "r"(col), "r"(head), "r"(pos), "r"(batch)
                 : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, const void* smem_src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%2, %3}], [%1];" ::"l"(map),
                 "r"(smem_u32(smem_src)), "r"(x), "r"(y)
                 : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
template <int N = 0>
__device__ __forceinline__ void tma_store_wait_read() {  // smem source of all but the last N groups may be reused
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void tma_store_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Per-thread register budget of the calling warpgroup (4 consecutive warps, all of which must execute it): release
// registers to the pool / take them from it.  The kernel needs a compile-time register cap (__maxnreg__).
template <int R>
__device__ __forceinline__ void setmaxnreg_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(R));
}
template <int R>
__device__ __forceinline__ void setmaxnreg_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(R));
}

// Barrier among `count` threads (a multiple of 32) of the CTA; id 0 is __syncthreads.
__device__ __forceinline__ void named_bar_sync(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// Hand-over by a hardware barrier: the warps that make something are counted in without waiting, the few that go on with it wait in named_bar_sync.
// A maker must not be counted twice in one turn of a barrier.  The waits between two hand-overs see to that, since they stand for what the takers do behind
// their barrier, until one gives up: then they stand for nothing.  So the takers keep count of the turns that are over, and every maker looks once a round,
// behind the wait that its next hand-overs rely on, whether a wait has given up (nothing had then, in the whole block, if not), and if so waits until those
// turns are over.  A block whose warps reach its barriers in one order, each warp some of them, comes to its end with this whatever wait runs out: the
// first barrier in that order that is not over lacks only warps that no later one holds back.
__device__ __forceinline__ void hand_over(int id, int count) {
    __syncwarp();
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}
// taken: the takers' counts, four words, of which each says how many rounds may begin, and which start where the makers' first round needs them (what is not
// used at kTakenAll).  Bounded all the same.
constexpr int kTakenAll = 0x7fffffff;
__device__ __forceinline__ void until_taken(int late, const int4* taken, int round) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b32 n, a, b, c, d;\n\t"
        "setp.eq.s32 p, %0, 0;\n\t"
        "@p bra DONE;\n\t"
        "mov.b32 n, %3;\n"
        "AGAIN:\n\t"
        "ld.volatile.shared.v4.b32 {a, b, c, d}, [%1];\n\t"
        "min.s32 a, a, b;\n\t"
        "min.s32 c, c, d;\n\t"
        "min.s32 a, a, c;\n\t"
        "setp.gt.s32 p, a, %2;\n\t"
        "@p bra DONE;\n\t"
        "add.s32 n, n, -1;\n\t"
        "setp.ne.b32 p, n, 0;\n\t"
        "@p bra AGAIN;\n"
        "DONE:\n\t}"
        ::"r"(late), "r"(smem_u32(taken)), "r"(round), "r"(16u * kSpinLimit)
        : "memory");
}
__device__ __forceinline__ void set_taken(int* count, int rounds) { *(volatile int*)count = rounds; }

__device__ __forceinline__ void prefetch_tmap(const CUtensorMap* map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---------------------------------------------------------------- TMEM allocation (one full warp)
__device__ __forceinline__ void tmem_alloc(uint32_t* smem_result, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(smem_result)),
                 "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------- descriptors
// Shared-memory matrix descriptor of tcgen05.mma for a 128-byte-swizzled tile whose rows are 128
// bytes (64 bf16) at a 128-byte pitch and whose base is 1024-byte aligned.
//   bits [0,14)  start address >> 4        bits [16,30) leading-dimension byte offset >> 4
//   bits [32,46) stride byte offset >> 4   bits [46,48) version = 1      bits [61,64) layout = 2 (SWIZZLE_128B)
// K-major operand (the 64 contiguous elements run along K): stride offset = 1024 (eight rows); the
// leading offset is unused.  MN-major operand (the 64 contiguous elements run along M or N, rows are
// K): stride offset = 1024 (eight K rows), leading offset = distance between 64-wide MN panels.
// The high word is the same for every operand of these kernels; an issuing thread derives the low word of each K step with one integer add.
constexpr uint32_t kDescHi = (1024u >> 4) | (1u << 14) | (2u << 29);
__device__ __forceinline__ uint32_t desc_lo(uint32_t saddr, uint32_t lbo_bytes) {
    return ((saddr >> 4) & 0x3FFFu) | ((lbo_bytes >> 4) << 16);
}
// Instruction descriptor, kind::f16, bf16 x bf16 -> fp32, dense.
//   [4,6) D format (1 = f32)  [7,10) A format (1 = bf16)  [10,13) B format (1 = bf16)
//   bit 15 A major (1 = MN)   bit 16 B major (1 = MN)     [17,23) N >> 3     [24,29) M >> 4
__host__ __device__ constexpr uint32_t instr_desc(int M, int N, bool a_mn_major, bool b_mn_major) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((a_mn_major ? 1u : 0u) << 15) | ((b_mn_major ? 1u : 0u) << 16) |
           ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// D[tmem] (+)= A[smem] * B[smem], operands by the low words of their descriptors; issued by ONE thread.
template <bool ACC>
__device__ __forceinline__ void mma_ss_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "n"(ACC ? 1 : 0), "r"(kDescHi)
        : "memory");
}
__device__ __forceinline__ void mma_ss_lo(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 da, {%1, %5};\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_lo), "r"(b_lo), "r"(idesc), "r"((uint32_t)accumulate), "r"(kDescHi)
        : "memory");
}
// D[tmem] (+)= A[tmem] * B[smem]; A holds bf16 pairs packed in 32-bit TMEM columns.
__device__ __forceinline__ void mma_ts_lo(uint32_t d_tmem, uint32_t a_tmem, uint32_t b_lo, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 db;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "mov.b64 db, {%2, %5};\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], db, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "r"(b_lo), "r"(idesc), "r"((uint32_t)accumulate), "r"(kDescHi)
        : "memory");
}
// mbarrier arrives once all tcgen05.mma issued so far by this thread have completed.
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// ---------------------------------------------------------------- TMEM <-> registers
// 32x32b shape: thread i of warp w (w = warp index mod 4) addresses TMEM lane 32*w + i; x32 moves
// 32 consecutive 32-bit columns starting at the column in taddr.
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,"
        "%29,%30,%31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]), "=r"(r[16]),
          "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]),
          "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
          "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// x16: 16 consecutive 32-bit columns.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%16], {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15};"
        ::"r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
          "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(taddr)
        : "memory");
}
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%8], {%0,%1,%2,%3,%4,%5,%6,%7};" ::"r"(r[0]), "r"(r[1]), "r"(r[2]),
                 "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 2^x in one instruction; what lies below 2^-126 comes out as zero.
__device__ __forceinline__ float ex2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// Packed fp32 pairs (sm_100): one instruction, two lanes.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    unsigned long long d;
    asm("mul.f32x2 %0, %1, %2;" : "=l"(d) : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)));
    return *reinterpret_cast<float2*>(&d);
}
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(d)
        : "l"(*reinterpret_cast<unsigned long long*>(&a)), "l"(*reinterpret_cast<unsigned long long*>(&b)),
          "l"(*reinterpret_cast<unsigned long long*>(&c)));
    return *reinterpret_cast<float2*>(&d);
}

// Byte offset of (row, 16-byte chunk) inside a 128-byte-swizzled tile with 128-byte rows.
__device__ __forceinline__ uint32_t sw128(uint32_t row, uint32_t chunk16) {
    return row * 128u + ((chunk16 ^ (row & 7u)) << 4);
}

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
}

}  // namespace ptx
}  // namespace ssd
