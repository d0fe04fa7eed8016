// Host build of the breadth-first search's structure kernels (csrc/bfs_rows.cuh), for CPU tests only:
// the blocks, rows and columns that a pass takes an entry's neighbours from, entry by entry.
#include <algorithm>
#include <cstdint>
#include <cstring>
#include <map>
#include <memory>
#include <string>
#include <vector>

#define __device__
#define __host__
#define __forceinline__ inline
#define __global__
#define __restrict__
#define __launch_bounds__(...)
#define __shared__ static
#define CCS_HOST_EMULATION 1
using std::max;
using std::min;

struct uint2 { uint32_t x, y; };
struct uint4 { uint32_t x, y, z, w; };
static inline uint2 make_uint2(uint32_t x, uint32_t y) { return {x, y}; }
static inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }
static inline uint32_t __byte_perm(uint32_t a, uint32_t b, uint32_t s) {
    const uint64_t x = ((uint64_t)b << 32) | a;
    uint32_t r = 0;
    for (int i = 0; i < 4; ++i) r |= (uint32_t)((x >> (8 * ((s >> (4 * i)) & 7u))) & 0xFFu) << (8 * i);
    return r;
}
static inline int __popc(uint32_t v) { return __builtin_popcount(v); }
static inline int __ffs(uint32_t v) { return v ? __builtin_ctz(v) + 1 : 0; }
static inline uint32_t __brev(uint32_t v) {
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= ((v >> i) & 1u) << (31 - i);
    return r;
}
static inline uint32_t __dp4a(uint32_t a, uint32_t b, uint32_t c) {
    for (int i = 0; i < 4; ++i) c += ((a >> (8 * i)) & 0xFFu) * ((b >> (8 * i)) & 0xFFu);
    return c;
}
template <typename T>
static inline T __ldg(const T* p) { return *p; }
static uint32_t thread_no;
struct Dim { uint32_t x; };
#define threadIdx (Dim{thread_no % 256u})
#define blockIdx (Dim{thread_no / 256u})
static Dim blockDim{256}, gridDim{1};
static void __syncthreads() {}
static void __syncwarp() {}
template <class T> static T __shfl_down_sync(uint32_t, T, int) { return T{}; }
template <class T> static T __shfl_sync(uint32_t, T v, int) { return v; }
static uint32_t __ballot_sync(uint32_t, bool p) { return p; }
static bool __any_sync(uint32_t, bool p) { return p; }
template <class T, class U> static T atomicAdd(T* p, U v) { T o = *p; *p = o + (T)v; return o; }
template <class T, class U> static T atomicAnd(T* p, U v) { T o = *p; *p = o & (T)v; return o; }
template <class T, class U> static T atomicOr(T* p, U v) { T o = *p; *p = o | (T)v; return o; }

#include "../../cuda-cube-solver_b200/csrc/dev_tables.h"
namespace ccs {
template <class Tables>
static void stage_tables(Tables& dst, const Tables* src) {
    if (thread_no == 0u) std::memcpy(&dst, src, sizeof dst);  // (static: the threads run one after another)
}
}  // namespace ccs
#include "../../cuda-cube-solver_b200/csrc/bfs_rows.cuh"

using namespace ccs;

namespace {
struct Structure {
    std::vector<uint32_t> cmove, lut;
    std::vector<uint4> desc;
};

template <int MODE, int NEC>
void neighbours(const DevTables& T, const uint64_t* idx, int n, int m, uint64_t* out, std::map<std::string, Structure>& memo, const char* name) {
    using RT = Rows<MODE, NEC>;
    Structure& s = memo[name];
    if (s.desc.empty()) {
        RowsParams P{};
        P.classidx = corner_classes().classidx.data();
        P.class_rep = corner_classes().rep.data();
        s.cmove.resize(N_CLASSES * 18u);
        s.desc.resize(N_SLICE * 18u * 16u);
        s.lut.resize(RT::N_LUT * RT::LUT);
        for (thread_no = 0; thread_no < s.cmove.size(); ++thread_no) rows_cmove(&T, P, s.cmove.data());
        for (thread_no = 0; thread_no < s.desc.size(); ++thread_no) rows_desc<MODE>(&T, s.desc.data());
        for (thread_no = 0; thread_no < s.lut.size(); ++thread_no) rows_lut<MODE, NEC>(&T, s.lut.data());
    }
    for (int i = 0; i < n; ++i) {
        const uint64_t row_no = idx[i] / RT::C, blk = row_no / RT::R;
        const uint32_t col = (uint32_t)(idx[i] % RT::C), row = (uint32_t)(row_no % RT::R);
        const uint32_t cls = (uint32_t)(blk / N_SLICE), slice = (uint32_t)(blk % N_SLICE);
        const uint32_t cm = s.cmove[cls * 18u + m];
        const uint4 d = s.desc[(slice * 18u + m) * 16u + (cm & 15u)];
        uint32_t id = (d.x >> 9) & 0x1FFFu, to;
        if (MODE == KIND_304) {
            to = T.ccomb_rank[permute8(row_bytes(T.ccomb_unrank[row]), d.y, d.z) ^ (d.x >> 24)];
        } else {
            to = permute8(row_bytes(row), d.y, d.z) ^ (d.x >> 24);
            id = id * 2u + (__popc(row) & 1u);
        }
        uint32_t from = ~0u, hits = 0;  // the one column whose bit comes to `col`
        for (uint32_t c = 0; c < RT::C; ++c)
            if ((s.lut[id * RT::LUT + ((c / RT::CB) << RT::CB) + (1u << (c % RT::CB))] >> col) & 1u) from = c, ++hits;
        out[i] = hits == 1u ? (((uint64_t)(cm >> 4) * N_SLICE + (d.x & 511u)) * RT::R + to) * RT::C + from : ~0ull;
    }
}

// Encoders on given distances: the planes of the first rows of the kind's array.
template <int MODE, int NEC>
void encode(const uint8_t* dist, uint64_t n, int late, uint32_t* blk, uint32_t* b3, uint32_t* mod3) {
    using RT = Rows<MODE, NEC>;
    const uint64_t rows = n / RT::C + 40;  // (the encoders look a few rows past the entries)
    std::vector<uint32_t> codes(rows * RT::QW, ~0u);
    std::vector<typename RT::Word> fifth(rows, 0);
    for (uint64_t i = 0; i < n; ++i) {
        uint32_t p[4];
        load_codes<RT>(codes.data(), i / RT::C, p);
        for (int b = 0; b < 4; ++b)
            if (!((dist[i] >> b) & 1u)) p[b] &= ~(1u << (i % RT::C));
        store_codes<RT>(codes.data(), i / RT::C, p);
        if (dist[i] & 16u) fifth[i / RT::C] |= (typename RT::Word)(1u << (i % RT::C));
    }
    RowsParams P{};
    P.codes = codes.data();
    if (late) P.late = reinterpret_cast<uint32_t*>(fifth.data());
    const uint64_t nb = (n + 123) / 124, n3 = (n + 154) / 155, nm = (n + 15) / 16;
    for (thread_no = 0; thread_no < nb; ++thread_no) encode_block<MODE, NEC>(P, n, nb, blk);
    for (thread_no = 0; thread_no < 32u; ++thread_no) {  // (stages the table of powers)
        encode_b3<MODE, NEC>(P, blk, n, thread_no < n3 ? n3 : 0u, b3);
    }
    for (thread_no = 0; thread_no < n3; ++thread_no) encode_b3<MODE, NEC>(P, blk, n, n3, b3);
    for (thread_no = 0; thread_no < nm; ++thread_no) encode_mod3<MODE, NEC>(P, n, nm, mod3);
}

// Frontier bits of distance d on given distances, of whole rows (n: a multiple of the kind's columns), and the
// flags of their blocks.
template <int MODE, int NEC>
void mark(const uint8_t* dist, uint64_t n, uint32_t d, uint8_t* bits, uint8_t* flags) {
    using RT = Rows<MODE, NEC>;
    const uint64_t rows = n / RT::C;
    std::vector<uint32_t> codes(rows * RT::QW, ~0u);
    std::vector<typename RT::Word> next(rows, 0);
    for (uint64_t i = 0; i < n; ++i) {
        uint32_t p[4];
        load_codes<RT>(codes.data(), i / RT::C, p);
        for (int b = 0; b < 4; ++b)
            if (!((dist[i] >> b) & 1u)) p[b] &= ~(1u << (i % RT::C));
        store_codes<RT>(codes.data(), i / RT::C, p);
    }
    RowsParams P{};
    P.codes = codes.data(), P.next = next.data(), P.next_flag = flags;
    for (thread_no = 0; thread_no < 256u; ++thread_no) rows_mark<MODE, NEC>(P, rows, d);
    for (uint64_t i = 0; i < n; ++i) bits[i] = (uint8_t)((next[i / RT::C] >> (i % RT::C)) & 1u);
}

template <typename F>
int with_kind(const char* name, F&& f) {
    using std::integral_constant;
    static std::map<std::string, std::pair<KindDesc, std::unique_ptr<DevTables>>> kinds;
    auto& k = kinds[name];
    if (!k.second) {
        if (!preset_kind(name, &k.first)) return -1;
        k.second = std::make_unique<DevTables>();
        build_dev_tables(k.first, k.second.get());
    }
    if (k.first.mode == KIND_304) f(integral_constant<int, KIND_304>{}, integral_constant<int, 1>{}, *k.second);
    else if (k.first.nec == 8) f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 8>{}, *k.second);
    else if (k.first.nec == 12) f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 12>{}, *k.second);
    else if (k.first.nec == 16) f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 16>{}, *k.second);
    else f(integral_constant<int, KIND_GEN>{}, integral_constant<int, 24>{}, *k.second);
    return 0;
}
}  // namespace

extern "C" {
int emul_rows_neighbours(const char* name, const uint64_t* idx, int n, int m, uint64_t* out) {
    static std::map<std::string, Structure> memo;
    return with_kind(name, [&](auto M, auto N, const DevTables& T) {
        neighbours<decltype(M)::value, decltype(N)::value>(T, idx, n, m, out, memo, name);
    });
}
int emul_rows_mark(const char* name, const uint8_t* dist, uint64_t n, uint32_t d, uint8_t* bits, uint8_t* flags) {
    return with_kind(name, [&](auto M, auto N, const DevTables&) {
        mark<decltype(M)::value, decltype(N)::value>(dist, n, d, bits, flags);
    });
}
int emul_rows_encode(const char* name, const uint8_t* dist, uint64_t n, int late, uint32_t* blk, uint32_t* b3, uint32_t* mod3) {
    return with_kind(name, [&](auto M, auto N, const DevTables&) {
        encode<decltype(M)::value, decltype(N)::value>(dist, n, late, blk, b3, mod3);
    });
}
}
