// Host run of one warp of the search kernel (csrc/search_warp.cuh), for CPU tests only.  The 32 lanes
// are fibers; a warp intrinsic is an exchange that every lane has to reach at the same line, so a
// divergent one aborts.  The table is all zeros (no child is pruned), which fills the node pool, the
// stashes and the spill list; pool and stash can be built small (CCS_WARP_POOL, CCS_WARP_STACK).
#include <ucontext.h>

#include <algorithm>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <memory>
#include <string>
#include <type_traits>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __global__
#define __restrict__
#define __launch_bounds__(...)
#define __grid_constant__
#define __shared__
#define CCS_HOST_EMULATION 1
using std::max;
using std::min;

static inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {  // prmt: selector bit 3 replicates the sign
    const uint64_t x = ((uint64_t)b << 32) | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) {
        const uint32_t n = (s >> (4 * i)) & 15u, byte = (uint32_t)(x >> (8 * (n & 7u))) & 0xFFu;
        r |= (n & 8u ? (byte & 0x80u ? 0xFFu : 0u) : byte) << (8 * i);
    }
    return r;
}
static inline int __popc(uint32_t v) { return __builtin_popcount(v); }
static inline int __ffs(uint32_t v) { return v ? __builtin_ctz(v) + 1 : 0; }
static inline uint32_t __funnelshift_r(uint32_t lo, uint32_t hi, uint32_t s) {
    return (uint32_t)((((uint64_t)hi << 32) | lo) >> (s & 31u));
}
static inline uint32_t __dp4a(uint32_t a, uint32_t b, uint32_t c) {
    for (int i = 0; i < 4; ++i) c += ((a >> (8 * i)) & 0xFFu) * ((b >> (8 * i)) & 0xFFu);
    return c;
}
template <typename T>
static inline T __ldg(const T* p) { return *p; }
template <typename T>
static inline T __ldcg(const T* p) { return *p; }

struct Dim { unsigned x; };
static int cur;
static ucontext_t main_ctx, ctx[32];
static bool gone[32];
static std::vector<char> stacks[32];
static unsigned long long arrived[32], value[2][32];
static int site[32];
#define threadIdx (Dim{(unsigned)cur})
static Dim blockIdx{0}, blockDim{32}, gridDim{1};

static void next_fiber() {
    const int me = cur;
    for (int i = 1; i < 32; ++i)
        if (const int t = (me + i) & 31; !gone[t]) {
            cur = t;
            swapcontext(&ctx[me], &ctx[t]);
            cur = me;
            return;
        }
}
static const unsigned long long* exchange(unsigned long long v, int line) {
    const int me = cur;
    const unsigned long long turn = ++arrived[me];
    value[turn & 1][me] = v;
    site[me] = line;
    for (;;) {
        bool all = true;
        for (int i = 0; i < 32 && all; ++i) {
            if (arrived[i] < turn && gone[i]) std::fprintf(stderr, "lane %d left the warp\n", i), std::abort();
            all = arrived[i] >= turn;
        }
        if (all) break;
        next_fiber();
    }
    for (int i = 0; i < 32; ++i)
        if (arrived[i] == turn && site[i] != line) std::fprintf(stderr, "divergent at %d / %d\n", line, site[i]), std::abort();
    return value[turn & 1];
}
static uint32_t ballot(bool p, int line) {
    const unsigned long long* v = exchange(p, line);
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= (uint32_t)(v[i] & 1u) << i;
    return r;
}
template <class T>
static T shuffle(T x, uint32_t from, int line) {
    unsigned long long bits = 0;
    std::memcpy(&bits, &x, sizeof x);
    const unsigned long long* v = exchange(bits, line);
    T r;
    std::memcpy(&r, &v[from & 31u], sizeof r);
    return r;
}
template <class F>
static uint32_t reduce(uint32_t x, F f, int line) {
    const unsigned long long* v = exchange(x, line);
    uint32_t r = (uint32_t)v[0];
    for (int i = 1; i < 32; ++i) r = f(r, (uint32_t)v[i]);
    return r;
}
#define __ballot_sync(m, p) ballot((p), __LINE__)
#define __shfl_sync(m, v, s) shuffle((v), (s), __LINE__)
#define __all_sync(m, p) (ballot((p), __LINE__) == 0xFFFFFFFFu)
#define __syncwarp() (void)exchange(0, __LINE__)
#define __reduce_or_sync(m, v) reduce((v), [](uint32_t a, uint32_t b) { return a | b; }, __LINE__)
#define __reduce_add_sync(m, v) reduce((v), [](uint32_t a, uint32_t b) { return a + b; }, __LINE__)
#define __reduce_min_sync(m, v) reduce((v), [](uint32_t a, uint32_t b) { return min(a, b); }, __LINE__)
#define __reduce_max_sync(m, v) reduce((v), [](uint32_t a, uint32_t b) { return max(a, b); }, __LINE__)
static void __nanosleep(unsigned) {}
static void __threadfence() {}
static void __threadfence_system() {}
template <class T, class U> static T atomicAdd(T* p, U v) { T o = *p; *p = o + (T)v; return o; }
template <class T, class U> static T atomicSub(T* p, U v) { T o = *p; *p = o - (T)v; return o; }
template <class T, class U> static T atomicExch(T* p, U v) { T o = *p; *p = (T)v; return o; }
template <class T, class U> static T atomicMax(T* p, U v) { T o = *p; if ((T)v > o) *p = (T)v; return o; }
template <class T, class U> static T atomicOr(T* p, U v) { T o = *p; *p = o | (T)v; return o; }
template <class T, class U, class V> static T atomicCAS(T* p, U c, V v) { T o = *p; if (o == (T)c) *p = (T)v; return o; }

#include "../../cuda-cube-solver_b200/csrc/warp_tables.cuh"
namespace ccs {
Word4 pool_smem[1 << 14];
template <class Tables>
static void stage_tables(Tables& dst, const Tables* src) { std::memcpy(&dst, src, sizeof dst); }
void cube_frames(const uint32_t state[5], uint32_t out[30]);
std::vector<uint32_t> canonical_prefixes(int length);
}  // namespace ccs
#include "../../cuda-cube-solver_b200/csrc/search_warp.cuh"

using namespace ccs;

static std::function<void()> body;
static void fiber() {
    body();
    gone[cur] = true;
    for (int i = 1; i < 32; ++i)
        if (const int t = (cur + i) & 31; !gone[t]) {
            cur = t;
            setcontext(&ctx[t]);
        }
    setcontext(&main_ctx);
}

template <typename F>
static void with_kind(const KindDesc& d, F&& f) {
    using std::integral_constant;
    if (d.mode == KIND_304) f(integral_constant<int, KIND_304>{}, integral_constant<int, 1>{});
    else if (d.nec == 8) f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 8>{});
    else if (d.nec == 12) f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 12>{});
    else if (d.nec == 16) f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 16>{});
    else f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 24>{});
}

extern "C" {

// Table index of each state after move `m` on a forward (left = 0) or an inverse (1) frame 0.
int emul_warp_index(const char* name, const uint32_t* w, int n, int m, int left, uint64_t* out) {
    KindDesc kd;
    if (!preset_kind(name, &kd)) return -1;
    auto T = std::make_unique<DevImage>();
    build_dev_tables(kd, &T->t);
    build_warp_tables(T->t, &T->w);
    const uint32_t* classidx = corner_classes().classidx.data();
    with_kind(kd, [&](auto M, auto N) {
        constexpr int MODE = decltype(M)::value, NEC = decltype(N)::value;
        for (int i = 0; i < n; ++i) {
            State s{w[5 * i], w[5 * i + 1], w[5 * i + 2], w[5 * i + 3], w[5 * i + 4]};
            if (m >= 0) s = left ? warp_left(T->w, s, m) : warp_right(T->w, s, m);
            const uint32_t packed = classidx[warp_corner_raw(T->w, s.c0, s.c1)];
            out[i] = (uint64_t)(packed >> 4) * KindTraits<MODE, NEC>::N_EDGE +
                     warp_edge_coord<MODE, NEC>(T->w, s, packed & 15u, (i & 1) != 0);  // (both tables hold the same kind)
        }
    });
    return 0;
}

void emul_warp_decode(const uint32_t* sectors, const uint32_t* entry, int n, uint32_t* out) {
    for (int i = 0; i < n; ++i) out[i] = warp_decode<FMT_BLOCK>(sectors + 8 * i, entry[i]);
}

void emul_warp_decode_b3(const uint32_t* sectors, const uint32_t* entry, int n, uint32_t* out) {
    for (int i = 0; i < n; ++i) out[i] = warp_decode<FMT_B3>(sectors + 8 * i, entry[i]);
}

// Warp intrinsics that the last emul_warp_solve ran: its length in steps of the warp.
uint64_t emul_warp_turns() { return arrived[0]; }

// Searches n cubes (at most 8) with one warp on an all-zero table; `starving`: 1: with shorter prefixes,
// donating all the time, 2: in items of one move, without donations.  status[n]; lengths[n]; nodes[24 n]: per cube and bound.  Returns the error bits.
int emul_warp_search(const char* name, const uint32_t* words, int n, int starving, uint32_t* status, uint32_t* lengths,
                     uint8_t* moves, uint64_t* nodes, uint64_t* donated) {
    KindDesc kd;
    if (!preset_kind(name, &kd)) return -2;
    auto T = std::make_unique<DevImage>();
    build_dev_tables(kd, &T->t);
    build_warp_tables(T->t, &T->w);
    std::unique_ptr<uint32_t, decltype(&std::free)> table((uint32_t*)std::calloc((kd.n_entries + 123) / 124 * 32, 1), &std::free);
    std::vector<Slot> slots(n);
    std::vector<DonationCell> cells(64);
    QueueState q;
    std::memset(&q, 0, sizeof q);
    std::memset(cells.data(), 0, sizeof(DonationCell) * cells.size());
    q.starving = starving == 1;
    constexpr uint32_t CAP = 64;
    std::vector<unsigned long long> ring(5 * CAP + 64, ~0ull);
    std::vector<std::vector<uint32_t>> prefixes;
    SearchParams P;
    std::memset(&P, 0, sizeof P);
    for (int L = 0; L <= MAX_PLEN; ++L) {
        prefixes.push_back(L <= 4 ? canonical_prefixes(L) : std::vector<uint32_t>());
        P.n_prefix[L] = (uint32_t)prefixes[L].size();
    }
    for (int L = 0; L <= MAX_PLEN; ++L) P.prefixes[L] = prefixes[L].data();
    P.slots = slots.data(), P.q = &q, P.n_slots = (uint32_t)n;
    P.ring = ring.data(), P.ring_cap = 4 * CAP + 64, P.admit = ring.data() + P.ring_cap, P.admit_cap = CAP;
    P.classidx = corner_classes().classidx.data(), P.table = P.table2 = table.get();
    P.base_plen = starving == 2 ? 1 : starving ? 3 : 4, P.max_plen = 4, P.few_divisor = 1, P.few_max_active = 4, P.shallow_min_active = 32;
    P.deeper_at[0] = P.deeper_at[1] = P.warp_many_at[0] = P.warp_many_at[1] = ~0ull;
    P.warp_items = 1, P.warp_at[0] = 200, P.warp_at[1] = 20000;  // prefixes two shorter, one, the base's
    if (starving == 2) P.warp_at[0] = P.warp_at[1] = ~0ull;
    P.idle_limit = 1000, P.spread = 64;
    P.don = cells.data(), P.don_cap = 64, P.don_target = 8, P.don_min_depth = 2, P.don_period = 16;
    for (int i = 0; i < n; ++i) {
        std::memset(&slots[i], 0, sizeof(Slot));
        cube_frames(words + 5 * i, slots[i].frame);
        slots[i].status = SLOT_ACTIVE;
        slots[i].ticket = TICKET_IDLE;
        P.admit[i] = (unsigned long long)i;
    }
    q.admit_tail = (unsigned long long)n;
    body = [&] {
        with_kind(kd, [&](auto M, auto N) {
            search_kernel_warp<decltype(M)::value, decltype(N)::value, FMT_BLOCK, 32, 1>(&T->w, P);
        });
    };
    std::memset(arrived, 0, sizeof arrived);
    for (int i = 0; i < 32; ++i) {
        gone[i] = false;
        stacks[i].resize(1 << 18);
        getcontext(&ctx[i]);
        ctx[i].uc_stack.ss_sp = stacks[i].data();
        ctx[i].uc_stack.ss_size = stacks[i].size();
        ctx[i].uc_link = nullptr;
        makecontext(&ctx[i], fiber, 0);
    }
    cur = 0;
    swapcontext(&main_ctx, &ctx[0]);
    for (int i = 0; i < n; ++i) {
        status[i] = slots[i].status;
        lengths[i] = slots[i].sol_len;
        std::memcpy(moves + 24 * i, slots[i].sol, 24);
        for (int b = 0; b < 24; ++b) nodes[24 * i + b] = slots[i].iter_nodes[b];
    }
    *donated = q.donated;
    return (int)q.error;
}
// The same for cubes that it is to solve (-1: one is unfinished).
int emul_warp_solve(const char* name, const uint32_t* words, int n, int starving, uint32_t* lengths, uint8_t* moves,
                    uint64_t* nodes, uint64_t* donated) {
    std::vector<uint32_t> status(n);
    const int error = emul_warp_search(name, words, n, starving, status.data(), lengths, moves, nodes, donated);
    for (int i = 0; i < n; ++i)
        if (status[i] != SLOT_SOLVED) return -1;
    return error;
}
}
