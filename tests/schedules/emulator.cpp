// The tile kernels on the CPU, from their own source: every thread of a block is a fiber, every copy and every group of products an agent of its own, and the one
// that runs next is chosen at random.  What the source does not order can so come in any order: a value that is read before the product or the copy it comes
// from, or overwritten while one still reads it, shows as other bits than those of another schedule; a barrier that a warp reaches twice in one
// turn, an arrival that no phase waits for and a block that cannot go on are counted.
// One block after the other, two products of one thread in order, those of different threads in any.  A wait can be made to run out.
#include <algorithm>
#include <array>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <deque>
#include <functional>
#include <random>
#include <unordered_map>
#include <vector>
#include <ucontext.h>

#include <cuda.h>
#include <cuda_runtime.h>
#include <cuda_bf16.h>
#undef __shared__
#define __shared__ static
#undef __launch_bounds__
#define __launch_bounds__(...)
#undef __maxnreg__
#define __maxnreg__(...)
#undef __grid_constant__
#define __grid_constant__
using std::max;
using std::min;

namespace emu {
constexpr int kPanel = 16384, kStack = 96 * 1024;
struct Mbar { int count = 0, pending = 0; long long bytes = 0; uint32_t phase = 0; };
struct HwBar { int expected = 0, arrived = 0; uint32_t turn = 0; uint32_t warps = 0; };
enum Why { kReady, kMbar, kHw, kWarp, kStores, kPoll, kDone };
struct Fiber {
    ucontext_t ctx;
    Why why = kReady;
    const void* bar = nullptr;
    uint32_t parity = 0, turn = 0;
    volatile int* alive = nullptr;
    int stores = 0;  // groups that may still read; what the counts have to pass
    bool expired = false;
};
struct Agent { double at; int kind; int index; };  // kind 0: warp, 1: products of a thread, 2: copy
struct Copy { std::function<void()> move; double at; bool store; int thread; };

struct State {
    int threads = 0, current = -1;
    std::vector<Fiber> fibers;
    std::vector<char> stacks;
    ucontext_t home;
    std::unordered_map<const void*, Mbar> mbars;
    HwBar hw[16];
    std::vector<HwBar> warp_bar;
    std::vector<double> warp_at;
    std::unordered_map<int, std::deque<std::function<void()>>> products;  // by issuing thread; a commit is one of them
    std::unordered_map<int, double> products_at;
    std::vector<Copy> copies;
    std::vector<int> uncommitted, reading;  // stores of a thread: of the open group, per group still reading
    std::unordered_map<int, std::deque<int>> groups;  // by thread: stores of each group that have not read yet
    std::unordered_map<int, int> open_group;
    std::mt19937 rng;
    uint32_t tmem[128][512];
    uint32_t shfl[2048];
    int overruns = 0, underflows = 0, hung = 0, expiries = 0, lose_copy = -1, copy_no = 0;
    bool in_order = false, expire = false;
    std::function<void()> body;
} S;

inline double dice() { return S.rng() / 4294967296.0; }
inline void leave() { swapcontext(&S.fibers[S.current].ctx, &S.home); }
inline void pause() {  // others may come in between
    if (!S.in_order && (S.rng() & 7) == 0) { S.fibers[S.current].why = kReady; leave(); }
}
inline Mbar& mbar(const void* p) { return S.mbars[p]; }
inline void settle(Mbar& b) {
    if (b.pending == 0 && b.bytes == 0) { b.phase ^= 1; b.pending = b.count; }
}
inline void arrive(const void* p) {
    Mbar& b = mbar(p);
    if (b.pending == 0) { ++S.underflows; return; }  // (the phase lacks bytes only)
    --b.pending;
    settle(b);
}
inline void wait(const void* p, uint32_t parity, volatile int* alive) {
    Fiber& f = S.fibers[S.current];
    pause();
    f.why = kMbar; f.bar = p; f.parity = parity; f.alive = alive; f.expired = false;
    leave();
    if (f.expired) *alive = 0;
}
// Every lane of the warp; `last` runs in the last of them to come.
inline void warp_meet(const std::function<void()>& last = {}) {
    const int w = S.current / 32;
    HwBar& b = S.warp_bar[w];
    if (++b.arrived == 32) {
        if (last) last();
        b.arrived = 0;
        ++b.turn;
        return;
    }
    Fiber& f = S.fibers[S.current];
    f.why = kWarp; f.turn = b.turn;
    leave();
}
inline void count_in(int id, int count) {
    HwBar& b = S.hw[id];
    const uint32_t bit = 1u << (S.current / 32);
    if (b.warps & bit || (b.arrived && b.expected != count)) ++S.overruns;
    b.warps |= bit;
    b.expected = count;
    if ((b.arrived += 32) >= count) { b.arrived -= count; b.warps = 0; ++b.turn; }
}
inline void hw_sync(int id, int count) {
    pause();
    const int w = S.current / 32;
    static uint32_t turn[64];
    warp_meet([&] { turn[w] = S.hw[id].turn; count_in(id, count); });
    Fiber& f = S.fibers[S.current];
    f.why = kHw; f.bar = &S.hw[id]; f.turn = turn[w];
    leave();
}
inline void hw_arrive(int id, int count) {
    pause();
    warp_meet([&] { count_in(id, count); });
}
inline void poll(const void* counts, int more_than) {
    Fiber& f = S.fibers[S.current];
    f.why = kPoll; f.bar = counts; f.stores = more_than;
    leave();
}
inline bool can_go(Fiber& f, int i) {
    switch (f.why) {
        case kReady: return true;
        case kMbar: return f.expired || mbar(f.bar).phase != f.parity || *f.alive <= 0;
        case kHw: return ((const HwBar*)f.bar)->turn != f.turn;
        case kWarp: return S.warp_bar[i / 32].turn != f.turn;
        case kPoll: {
            const volatile int* t = (const volatile int*)f.bar;
            return min(min(t[0], t[1]), min(t[2], t[3])) > f.stores;
        }
        case kStores: {
            int open = 0;
            auto& g = S.groups[i];
            for (size_t k = 0; k + f.stores < g.size(); ++k) open += g[k];
            return open == 0;
        }
        default: return false;
    }
}
inline bool run_warp(int w) {
    bool any = false;
    for (int i = w * 32; i < w * 32 + 32; ++i) {
        Fiber& f = S.fibers[i];
        if (f.why == kDone || !can_go(f, i)) continue;
        any = true;
        f.why = kReady;
        S.current = i;
        swapcontext(&S.home, &f.ctx);
    }
    return any;
}
inline void entry() {
    S.body();
    S.fibers[S.current].why = kDone;
    leave();
}
inline void block(int threads) {
    S.threads = threads;
    S.fibers.assign(threads, Fiber{});
    S.stacks.resize((size_t)threads * kStack);
    S.mbars.clear();
    for (auto& b : S.hw) b = HwBar{};
    const int warps = threads / 32;
    S.warp_bar.assign(warps, HwBar{});
    S.warp_at.resize(warps);
    for (auto& a : S.warp_at) a = dice();
    S.products.clear(); S.products_at.clear(); S.copies.clear(); S.groups.clear(); S.open_group.clear();
    for (int i = 0; i < 128 * 512; ++i) S.tmem[i / 512][i % 512] = 0x7fc00000u;
    for (int i = 0; i < threads; ++i) {
        getcontext(&S.fibers[i].ctx);
        S.fibers[i].ctx.uc_stack.ss_sp = S.stacks.data() + (size_t)i * kStack;
        S.fibers[i].ctx.uc_stack.ss_size = kStack;
        S.fibers[i].ctx.uc_link = nullptr;
        makecontext(&S.fibers[i].ctx, entry, 0);
    }
    std::vector<Agent> order;
    for (;;) {
        order.clear();
        for (int w = 0; w < warps; ++w) order.push_back({S.in_order ? 2.0 + w : S.warp_at[w], 0, w});
        for (auto& q : S.products)
            if (!q.second.empty()) order.push_back({S.in_order ? 1.0 : S.products_at[q.first], 1, q.first});
        for (size_t c = 0; c < S.copies.size(); ++c) order.push_back({S.in_order ? 0.0 : S.copies[c].at, 2, (int)c});
        std::sort(order.begin(), order.end(), [](const Agent& a, const Agent& b) { return a.at < b.at; });
        bool moved = false;
        for (auto& a : order) {
            if (a.kind == 0) {
                moved = run_warp(a.index);
                if (moved && S.rng() % 64 == 0) S.warp_at[a.index] = dice();
            } else if (a.kind == 1) {
                auto& q = S.products[a.index];
                q.front()();
                q.pop_front();
                S.products_at[a.index] = dice();
                moved = true;
            } else {
                auto move = S.copies[a.index].move;
                S.copies.erase(S.copies.begin() + a.index);
                move();
                moved = true;
            }
            if (moved) break;
        }
        auto expire = [&] {
            std::vector<int> at;
            for (int i = 0; i < threads; ++i)
                if (S.fibers[i].why == kMbar && mbar(S.fibers[i].bar).phase == S.fibers[i].parity) at.push_back(i);
            if (at.empty()) return false;
            S.fibers[at[S.rng() % at.size()]].expired = true;
            ++S.expiries;
            return true;
        };
        if (moved) {
            if (S.expire && S.rng() % 2048 == 0) expire();
            continue;
        }
        bool done = true;
        for (auto& f : S.fibers) done = done && f.why == kDone;
        if (done) return;
        if ((S.expire || S.lose_copy >= 0) && expire()) continue;
        ++S.hung;
        return;
    }
}
}  // namespace emu

struct ThreadIdx { struct X { operator int() const { return emu::S.current; } } x; };
static ThreadIdx threadIdx;
struct Three { int x = 0, y = 0, z = 0; };
static Three blockIdx, gridDim;
inline void __syncwarp(unsigned = ~0u) { emu::warp_meet(); }
inline void __syncthreads() { emu::hw_sync(0, emu::S.threads); }
inline int __syncthreads_or(int v) {
    static int any[2], turn[2048];
    const int t = turn[emu::S.current]++ & 1;
    any[t] |= v;
    __syncthreads();
    const int r = any[t];
    __syncthreads();
    any[t] = 0;
    return r;
}
template <class F> inline uint32_t exchange(uint32_t v, F from) {
    emu::S.shfl[emu::S.current] = v;
    emu::warp_meet();
    const int lane = emu::S.current & 31, base = emu::S.current & ~31, src = from(lane);
    const uint32_t r = emu::S.shfl[base + (src >= 0 && src < 32 ? src : lane)];
    emu::warp_meet();
    return r;
}
inline uint32_t bits_of(float v) { uint32_t u; memcpy(&u, &v, 4); return u; }
inline float float_of(uint32_t u) { float v; memcpy(&v, &u, 4); return v; }
#define __uint_as_float float_of
#define __float_as_uint bits_of
inline float __shfl_xor_sync(unsigned, float v, int o) { return float_of(exchange(bits_of(v), [o](int l) { return l ^ o; })); }
inline float __shfl_down_sync(unsigned, float v, int o) { return float_of(exchange(bits_of(v), [o](int l) { return l + o; })); }
inline float __shfl_sync(unsigned, float v, int s) { return float_of(exchange(bits_of(v), [s](int) { return s; })); }
inline int __any_sync(unsigned, int p) {
    emu::S.shfl[emu::S.current] = p != 0;
    emu::warp_meet();
    int r = 0;
    for (int i = 0; i < 32; ++i) r |= (int)emu::S.shfl[(emu::S.current & ~31) + i];
    emu::warp_meet();
    return r;
}
inline int atomicExch(int* p, int v) { const int o = *p; *p = v; return o; }

namespace ssd {
struct Dims { int b, T, h, p, n, g, l, c, hpg; };
inline void dep_wait() {}
namespace cum {
constexpr int LT = 128;
inline void clear_status(int* s) { if (threadIdx.x == 0) *s = 0; }
}
namespace tc { alignas(1024) extern uint8_t smem_raw[232 * 1024]; uint8_t smem_raw[232 * 1024]; }
namespace ptx {
using emu::S;
inline uint32_t smem_u32(const void* p) { return (uint32_t)((const uint8_t*)p - tc::smem_raw); }
inline void mbar_init(uint64_t* b, uint32_t n) { auto& m = emu::mbar(b); m = emu::Mbar{}; m.count = m.pending = (int)n; }
inline void mbar_fence_init() {}
inline void mbar_arrive(uint64_t* b) { emu::pause(); emu::arrive(b); }
inline void mbar_arrive_warp(uint64_t* b) { emu::pause(); emu::warp_meet([&] { emu::arrive(b); }); }
inline void mbar_expect_tx(uint64_t* b, uint32_t n) {
    emu::mbar(b).bytes += n;
    emu::arrive(b);
}
constexpr uint32_t kSpinLimit = 1;
inline void mbar_wait(uint64_t* b, uint32_t ph, volatile int* alive, uint32_t = 0) { emu::wait(b, ph, alive); }
inline void mbar_wait_spin(uint64_t* b, uint32_t ph, volatile int* alive, uint32_t = 0) { emu::wait(b, ph, alive); }
inline void fence_async_smem() { emu::pause(); }
inline void tc_fence_before() { emu::pause(); }
inline void tc_fence_after() {}
struct Map { const uint8_t* base; int64_t dim[4], pitch[4]; int rank; };
inline uint32_t swizzle(uint32_t a) { return a ^ ((a >> 7 & 7) << 4); }
// 64 columns x 128 rows between memory and a swizzled panel; at[d] the first index of dimension d, the rows along `rows`
inline void box(const CUtensorMap* m, uint8_t* smem, std::array<int64_t, 4> at, int rows, bool store) {
    Map t;
    memcpy(&t, m, sizeof t);
    for (int r = 0; r < 128; ++r, ++at[rows])
        for (int c = 0; c < 64; ++c) {
            uint16_t* s = (uint16_t*)(tc::smem_raw + swizzle((uint32_t)(smem - tc::smem_raw) + r * 128 + c * 2));
            bool in = at[0] + c < t.dim[0];
            int64_t o = (at[0] + c) * 2;
            for (int d = 1; d < t.rank; ++d) { in = in && at[d] < t.dim[d]; o += at[d] * t.pitch[d]; }
            if (store && in) *(uint16_t*)(t.base + o) = *s;
            if (!store) *s = in ? *(const uint16_t*)(t.base + o) : 0;
        }
}
inline void load(uint64_t* bar, uint32_t bytes, std::function<void()> move) {
    if (S.copy_no++ == S.lose_copy) return;
    S.copies.push_back({[=] { move(); auto& b = emu::mbar(bar); b.bytes -= bytes; emu::settle(b); }, emu::dice(), false, 0});
    emu::pause();
}
inline void store(std::function<void()> move) {
    const int me = S.current;
    auto& open = S.open_group[me];
    const int group = (int)S.groups[me].size();
    ++open;
    S.copies.push_back({[=] { move(); auto& g = S.groups[me]; if ((int)g.size() > group) --g[group]; else --S.open_group[me]; }, emu::dice(), true, me});
}
inline void tma_load_2d(void* d, const CUtensorMap* m, uint64_t* bar, int x, int y) { load(bar, emu::kPanel, [=] { box(m, (uint8_t*)d, {x, y, 0, 0}, 1, false); }); }
inline void tma_load_4d(void* d, const CUtensorMap* m, uint64_t* bar, int c, int h, int p, int b) { load(bar, emu::kPanel, [=] { box(m, (uint8_t*)d, {c, h, p, b}, 2, false); }); }
inline void bulk_load(void* d, const void* s, uint32_t n, uint64_t* bar) { load(bar, n, [=] { memcpy(d, s, n); }); }
inline void tma_store_2d(const CUtensorMap* m, const void* s, int x, int y) { store([=] { box(m, (uint8_t*)s, {x, y, 0, 0}, 1, true); }); }
inline void tma_store_4d(const CUtensorMap* m, const void* s, int c, int h, int p, int b) { store([=] { box(m, (uint8_t*)s, {c, h, p, b}, 2, true); }); }
inline void tma_prefetch_2d(const CUtensorMap*, int, int) {}
inline void tma_prefetch_4d(const CUtensorMap*, int, int, int, int) {}
inline void tma_store_commit() { S.groups[S.current].push_back(S.open_group[S.current]); S.open_group[S.current] = 0; }
template <int N = 0> inline void tma_store_wait_read() {
    auto& f = S.fibers[S.current];
    f.why = emu::kStores; f.stores = N;
    emu::leave();
}
inline void tma_store_wait_all() { tma_store_wait_read<0>(); }
template <int R> inline void setmaxnreg_dec() {}
template <int R> inline void setmaxnreg_inc() {}
inline void named_bar_sync(int id, int n) { emu::hw_sync(id, n); }
inline bool gave_up(const volatile int* alive) {
    const int a = *alive;
    emu::pause();
    return a <= 0;
}
inline void end_of_waits(const volatile int* alive, int* status) { if (gave_up(alive) && threadIdx.x == 0) *status = 1; }
inline void hand_over(int id, int n) { emu::hw_arrive(id, n); }
constexpr int kTakenAll = 0x7fffffff;
inline void until_taken(int late, const int4* taken, int round) { if (late) emu::poll(&taken->x, round); }
inline void set_taken(int* count, int rounds) { *(volatile int*)count = rounds; emu::pause(); }
inline void prefetch_tmap(const CUtensorMap*) {}
inline void tmem_alloc(uint32_t* p, uint32_t) { *p = 0; }
inline void tmem_relinquish() {}
inline void tmem_dealloc(uint32_t, uint32_t) {}
constexpr uint32_t instr_desc(int M, int N, bool a, bool b) { return (a ? 1u << 15 : 0) | (b ? 1u << 16 : 0) | (uint32_t)(N >> 3) << 17 | (uint32_t)(M >> 4) << 24; }
inline uint32_t desc_lo(uint32_t s, uint32_t lbo) { return (s >> 4 & 0x3FFF) | (lbo >> 4) << 16; }
inline float bf(uint32_t u) { return float_of(u << 16); }
// element (row of M or N, k) of an operand in shared memory
inline float element(uint32_t lo, bool mn_major, int r, int k) {
    const uint32_t at = (lo & 0x3FFF) << 4, lead = (lo >> 16) << 4;
    const uint32_t a = mn_major ? at + (r / 64) * lead + (k / 8) * 1024 + (k % 8) * 128 + (r % 64) * 2 : at + (r / 8) * 1024 + (r % 8) * 128 + k * 2;
    return bf(*(const uint16_t*)(tc::smem_raw + swizzle(a)));
}
inline void product(uint32_t d, bool a_tmem, uint32_t a, uint32_t b, uint32_t idesc, bool acc) {
    const int M = (idesc >> 24 & 31) << 4, N = (idesc >> 17 & 63) << 3;
    float A[128][16], B[128][16];
    for (int m = 0; m < M; ++m)
        for (int k = 0; k < 16; ++k) A[m][k] = a_tmem ? bf(S.tmem[m][(a & 0xffff) + k / 2] >> (k & 1) * 16 & 0xffff) : element(a, idesc >> 15 & 1, m, k);
    for (int n = 0; n < N; ++n)
        for (int k = 0; k < 16; ++k) B[n][k] = element(b, idesc >> 16 & 1, n, k);
    for (int m = 0; m < M; ++m)
        for (int n = 0; n < N; ++n) {
            float s = 0.f;
            for (int k = 0; k < 16; ++k) s += A[m][k] * B[n][k];
            uint32_t& t = S.tmem[m][(d & 0xffff) + n];
            t = bits_of(acc ? float_of(t) + s : s);
        }
}
inline void issue(std::function<void()> f) {
    if (S.products[S.current].empty()) S.products_at[S.current] = emu::dice();
    S.products[S.current].push_back(std::move(f));
}
inline void mma_ss_lo(uint32_t d, uint32_t a, uint32_t b, uint32_t i, bool acc) { issue([=] { product(d, false, a, b, i, acc); }); }
template <bool ACC> inline void mma_ss_lo(uint32_t d, uint32_t a, uint32_t b, uint32_t i) { mma_ss_lo(d, a, b, i, ACC); }
inline void mma_ts_lo(uint32_t d, uint32_t a, uint32_t b, uint32_t i, bool acc) { issue([=] { product(d, true, a, b, i, acc); }); }
inline void mma_commit(uint64_t* bar) { issue([=] { emu::arrive(bar); }); emu::pause(); }
template <int N> inline void tmem_get(uint32_t a, uint32_t (&r)[N]) {
    emu::pause();
    for (int i = 0; i < N; ++i) r[i] = S.tmem[(a >> 16) + (S.current & 31)][(a & 0xffff) + i];
}
template <int N> inline void tmem_put(uint32_t a, const uint32_t (&r)[N]) {
    emu::pause();
    for (int i = 0; i < N; ++i) S.tmem[(a >> 16) + (S.current & 31)][(a & 0xffff) + i] = r[i];
}
inline void tmem_ld32(uint32_t a, uint32_t (&r)[32]) { tmem_get(a, r); }
inline void tmem_ld16(uint32_t a, uint32_t (&r)[16]) { tmem_get(a, r); }
inline void tmem_st16(uint32_t a, const uint32_t (&r)[16]) { tmem_put(a, r); }
inline void tmem_st8(uint32_t a, const uint32_t (&r)[8]) { tmem_put(a, r); }
inline void tmem_ld_wait() {}
inline void tmem_st_wait() {}
inline float ex2(float x) { return exp2f(x); }
inline float2 mul2(float2 a, float2 b) { return make_float2(a.x * b.x, a.y * b.y); }
inline float2 fma2(float2 a, float2 b, float2 c) { return make_float2(fmaf(a.x, b.x, c.x), fmaf(a.y, b.y, c.y)); }
inline uint32_t sw128(uint32_t r, uint32_t c) { return r * 128u + ((c ^ (r & 7u)) << 4); }
inline uint32_t pack_bf16(float lo, float hi) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    uint32_t u;
    memcpy(&u, &v, 4);
    return u;
}
}  // namespace ptx
}  // namespace ssd

#include "ssd_tc.cuh"

// ------------------------------------------------------------------------------------------ one launch
namespace {
using namespace ssd::tc;
CUtensorMap map_of(void* base, std::vector<int64_t> dims) {  // innermost first
    CUtensorMap m{};
    ssd::ptx::Map t{(uint8_t*)base, {1, 1, 1, 1}, {2, 0, 0, 0}, (int)dims.size()};
    int64_t pitch = 2;
    for (size_t d = 0; d < dims.size(); ++d) { t.dim[d] = dims[d]; t.pitch[d] = pitch; pitch *= dims[d]; }
    static_assert(sizeof t <= sizeof m, "");
    memcpy(&m, &t, sizeof t);
    return m;
}
template <class K, class P> void launch(K kernel, const P& p, int gx, int gy, int gz, int threads) {
    gridDim.x = gx; gridDim.y = gy; gridDim.z = gz;
    emu::S.body = [&] { kernel(p); };
    for (int z = gz - 1; z >= 0; --z)
        for (int y = 0; y < gy; ++y)
            for (int x = 0; x < gx && !emu::S.hung; ++x) {
                blockIdx.x = x; blockIdx.y = y; blockIdx.z = z;
                for (size_t i = 0; i < sizeof smem_raw; i += 2) *(uint16_t*)(smem_raw + i) = 0x7fc0;
                emu::block(threads);
            }
}
}  // namespace

struct Args {  // every pointer (b, T, ...) as the entry points have them, bf16 as 16-bit words
    int b, T, h, g, p, n;
    uint16_t *x, *B, *C, *y, *dy, *dx, *dB, *dC, *states, *dstates;
    float *tcum, *dtT, *skipT, *D, *seed, *out_state, *ysq, *g_, *ddtx, *dyx, *gS;
    int *status, *extreme;
    int flags, whole, np, cut[5], ctas;
    unsigned seed_of_schedule;
    int in_order, expire, lose_copy;
    int overruns, underflows, hung, expiries;  // results
};

template <class K> void run(Args* a, K&& go) {
    auto& S = emu::S;
    S.rng.seed(a->seed_of_schedule);
    S.in_order = a->in_order; S.expire = a->expire; S.lose_copy = a->lose_copy;
    S.copy_no = S.overruns = S.underflows = S.hung = S.expiries = 0;
    *a->status = 0;
    go();
    a->overruns = S.overruns; a->underflows = S.underflows; a->hung = S.hung; a->expiries = S.expiries;
}
static WalkParams walk(Args* a, uint16_t* u, uint16_t* v) {
    WalkParams P{};
    const int nt = (a->T + 127) / 128;
    P.mU = map_of(u, {a->p, a->h, a->T, a->b});
    P.mV = map_of(v, {a->n, a->g, a->T, a->b});
    P.mC = map_of(a->C, {a->n, a->g, a->T, a->b});
    P.mY = map_of(a->y, {a->p, a->h, a->T, a->b});
    P.mS = map_of(a->states, {64, (int64_t)a->b * nt * a->h * 128});
    P.save_states = a->states != nullptr;
    P.tcum = a->tcum; P.dtT = a->dtT; P.D = a->D; P.skipT = a->skipT; P.seed = a->seed; P.out_state = a->out_state; P.ysq = a->ysq; P.status = a->status;
    P.Tp = nt * 128; P.h = a->h; P.hpg = a->h / a->g; P.nt = P.pt = nt; P.p = a->p; P.n = a->n;
    return P;
}
extern "C" void forward(Args* a) {
    WalkParams P = walk(a, a->x, a->B);
    int grid = a->h;
    if (a->np > 1) {
        P.self.whole = a->whole; P.self.np = a->np;
        memcpy(P.self.cut, a->cut, sizeof a->cut);
        grid = a->whole + (a->b * a->h - a->whole) * a->np;
    }
    run(a, [&] { launch(fwd_walk_kernel, P, grid, a->np > 1 ? 1 : a->b, 1, kFwdThreads); });
}
extern "C" void states(Args* a) {
    WalkParams P = walk(a, a->x, a->B);
    run(a, [&] { launch(states_walk_kernel, P, a->h, a->b, 1, kWalkThreads); });
}
extern "C" void reverse(Args* a, int heads) {
    WalkParams P = walk(a, a->dy, a->C);
    P.mS = map_of(a->dstates, {64, (int64_t)a->b * P.nt * a->h * 128});
    P.dtT = nullptr;
    run(a, [&] {
        if (heads == 2) launch(rev_walk_kernel<2, false>, P, a->h / 2, a->b, 1, RevCfg<2>::THREADS);
        else launch(rev_walk_kernel<1, false>, P, a->h, a->b, 1, RevCfg<1>::THREADS);
    });
}
extern "C" void summary(Args* a, int heads, int rev) {
    const WalkParams W = walk(a, rev ? a->dy : a->x, rev ? a->C : a->B);
    SummaryParams P{};
    P.mU = W.mU; P.mV = W.mV; P.tcum = W.tcum; P.dtT = rev ? nullptr : W.dtT; P.seed = W.seed; P.out = W.out_state; P.status = W.status; P.Tp = W.Tp; P.h = W.h;
    P.hpg = W.hpg; P.nt = P.pt = P.ps = W.nt; P.parts = 1; P.p = W.p; P.n = W.n;
    run(a, [&] {
        if (heads == 2 && rev) launch(summary_kernel<true, 2>, P, a->h / 2, a->b, 1, SumCfg<2>::THREADS);
        else if (heads == 2) launch(summary_kernel<false, 2>, P, a->h / 2, a->b, 1, SumCfg<2>::THREADS);
        else if (rev) launch(summary_kernel<true, 1>, P, a->h, a->b, 1, SumCfg<1>::THREADS);
        else launch(summary_kernel<false, 1>, P, a->h, a->b, 1, SumCfg<1>::THREADS);
    });
}
extern "C" void backward(Args* a) {  // of given states and state gradients
    const WalkParams W = walk(a, a->x, a->B);
    BwdParams P{};
    P.mX = W.mU; P.mB = W.mV; P.mC = W.mC; P.mH = W.mS;
    P.mdY = map_of(a->dy, {a->p, a->h, a->T, a->b});
    P.mQ = map_of(a->dstates, {64, (int64_t)a->b * W.nt * a->h * 128});
    P.mdX = map_of(a->dx, {a->p, a->h, a->T, a->b});
    P.mdB = map_of(a->dB, {a->n, a->g, a->T, a->b});
    P.mdC = map_of(a->dC, {a->n, a->g, a->T, a->b});
    P.tcum = W.tcum; P.dtT = W.dtT; P.D = W.D; P.skipT = W.skipT; P.g = a->g_; P.ddtx = a->ddtx; P.dyx = a->dyx; P.gS = a->gS; P.extreme = a->extreme; P.flags = a->flags;
    P.status = W.status; P.Tp = W.Tp; P.h = W.h; P.hpg = W.hpg; P.nt = W.nt; P.b = a->b; P.n = a->n; P.items = W.nt * a->g * a->b;
    run(a, [&] { launch(bwd_tile_kernel, P, min(P.items, a->ctas), 1, 1, kBwdThreads); });
}
