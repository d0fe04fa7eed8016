// GPU breadth-first search of a coset table, and the encoders of its files.
//
// What is computed is the reference's (table.py:82-129, kernels.cu:485-624,1839-1869): the exact
// distance of every entry from the solved coset, and files that are pure functions of it.
//
// The search rests on how the index factors.  Entry = corner class, slice (which positions hold E
// edges), row, column; row = flips of the other eight edges (304: the layout of the U edges among
// them), column = class of the E edges' content (304: their flips).  A move takes class -> (class',
// symmetry) whatever the edges are, and given the symmetry (slice, move) -> slice', the row to a
// fixed permutation of its eight bits (and a constant), and the column to a fixed permutation that
// depends on the row's parity alone.  So the neighbours of a (class, slice) block under one move are
// one other block, whole, with rows and columns permuted: a pass reads 18 contiguous blocks of
// frontier bits per block (a row is one word, a bit per column), permutes each row's bits with a few
// table lookups and ORs them, instead of unranking, moving and indexing every entry.
//
// A distance is four bits, one bit per column in each of four words of the row (1111: not reached);
// kinds deeper than 14 get a fifth word (`late`).  While the frontier is small it is a list, expanded
// forward entry by entry.  The encoders work on the bit planes, 32 entries at a time.
//
// Bound: a dense pass moves the distances once (20 GB for 24 classes) and 18 frontier blocks per block
// through L2; the lookups of the column permutations take the shared/L1 pipe.
// What it measured against the byte-per-entry form it replaces stands at rows_pull.
#pragma once

#include <type_traits>

#include "cube_dev.cuh"

namespace ccs {

template <int MODE, int NEC>
struct Rows {
    static constexpr uint32_t C = MODE == KIND_304 ? 16u : (uint32_t)NEC;  // columns
    static constexpr uint32_t R = MODE == KIND_304 ? 70u : 256u;           // rows of a block
    using Word = std::conditional_t<(C > 16), uint32_t, std::conditional_t<(C > 8), uint16_t, uint8_t>>;
    static constexpr uint32_t QW = sizeof(Word);                  // 32-bit words of a row's four planes
    static constexpr uint32_t ALL = C == 32 ? ~0u : (1u << C) - 1u;
    static constexpr uint32_t CB = C > 16 ? 5u : 4u;              // columns per lookup
    static constexpr uint32_t NCH = (C + CB - 1) / CB;
    static constexpr uint32_t LUT = NCH << CB;                    // words of a column permutation's tables
    static constexpr uint32_t N_LUT = MODE == KIND_304 ? 24u * 16u : 24u * 16u * 16u * 2u;
    static constexpr uint32_t LANE_ROWS = MODE == KIND_304 ? 3u : 8u;
    static constexpr uint64_t N_BLOCKS = (uint64_t)N_CLASSES * N_SLICE;
    static constexpr uint64_t N_ROWS = N_BLOCKS * R;
};

struct RowsParams {
    uint32_t* codes;                 // distances: Rows::QW words per row
    uint32_t* late;                  // fifth plane (Rows::Word per row), or null
    void* cur;                       // frontier bits (Rows::Word per row)
    void* next;
    uint8_t* cur_flag;               // per block: the frontier has entries in it
    uint8_t* next_flag;
    const uint32_t* classidx;
    const uint32_t* class_rep;
    const uint16_t* class_stab;
    const uint32_t* cmove;           // (class, move) -> class' << 4 | symmetry
    const uint4* desc;               // (slice, move, symmetry): see rows_desc
    const uint32_t* lut;             // column permutations: see rows_lut
    unsigned long long* counter;     // [0] entries found, [1] 32-byte sectors read at random, [2] claims
};

// The four planes of a row, as words.
template <class RT>
__device__ __forceinline__ void load_codes(const uint32_t* codes, uint64_t row, uint32_t p[4]) {
    if constexpr (RT::QW == 4) {
        const uint4 v = reinterpret_cast<const uint4*>(codes)[row];
        p[0] = v.x, p[1] = v.y, p[2] = v.z, p[3] = v.w;
    } else if constexpr (RT::QW == 2) {
        const uint2 v = reinterpret_cast<const uint2*>(codes)[row];
        p[0] = v.x & 0xFFFFu, p[1] = v.x >> 16, p[2] = v.y & 0xFFFFu, p[3] = v.y >> 16;
    } else {
        const uint32_t v = codes[row];
        p[0] = v & 0xFFu, p[1] = (v >> 8) & 0xFFu, p[2] = (v >> 16) & 0xFFu, p[3] = v >> 24;
    }
}

template <class RT>
__device__ __forceinline__ void store_codes(uint32_t* codes, uint64_t row, const uint32_t p[4]) {
    if constexpr (RT::QW == 4) reinterpret_cast<uint4*>(codes)[row] = make_uint4(p[0], p[1], p[2], p[3]);
    else if constexpr (RT::QW == 2) reinterpret_cast<uint2*>(codes)[row] = make_uint2(p[0] | (p[1] << 16), p[2] | (p[3] << 16));
    else codes[row] = p[0] | (p[1] << 8) | (p[2] << 16) | (p[3] << 24);
}

template <class RT>
__device__ __forceinline__ uint32_t unreached(const RowsParams& P, uint64_t row, const uint32_t p[4]) {
    uint32_t u = p[0] & p[1] & p[2] & p[3] & RT::ALL;
    if (P.late) u &= reinterpret_cast<const typename RT::Word*>(P.late)[row];
    return u;
}

__device__ __forceinline__ void add_count(unsigned long long* counter, unsigned long long local) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) local += __shfl_down_sync(0xFFFFFFFFu, local, o);
    if ((threadIdx.x & 31u) == 0 && local) atomicAdd(counter, local);
}

// ---- the structure of a kind --------------------------------------------------------------------

__global__ void __launch_bounds__(256) rows_cmove(const DevTables* __restrict__ gT, RowsParams P, uint32_t* __restrict__ cmove) {
    __shared__ DevTables T;
    stage_tables(T, gT);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N_CLASSES * 18u) return;
    State s;
    unrank_dev<KIND_304, 1>(T, P.class_rep, (uint64_t)(i / 18u) * KindTraits<KIND_304, 1>::N_EDGE, s);  // (the corners alone)
    corners_right(T, s.c0, s.c1, (int)(i % 18u));
    cmove[i] = P.classidx[corner_raw_words(T, s.c0, s.c1)];
}

// What a move and a symmetry do to the edges of a slice: x = slice' | column permutation << 9 | the
// row's constant << 24; y, z = a byte for each of the row's eight bits, with the bit it goes to set.  Found
// by moving states that carry one flip.  A column permutation is known by the order and flips that identity
// content comes to (and the symmetry, which relabels it: rows_lut).
template <int MODE>
__global__ void __launch_bounds__(256) rows_desc(const DevTables* __restrict__ gT, uint4* __restrict__ desc) {
    __shared__ DevTables T;
    stage_tables(T, gT);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= N_SLICE * 18u * 16u) return;
    const uint32_t sym = i & 15u, m = (i >> 4) % 18u, emask0 = T.slice_unrank[(i >> 4) / 18u];
    uint32_t base = 0, perm[2] = {0, 0}, slice = 0, order = 0, flips = 0;
    for (int mark = -1; mark < 8; ++mark) {
        uint32_t e[3] = {0, 0, 0}, ne = 0, no = 0;
        for (int q = 0; q < 12; ++q) {
            uint32_t b;
            if ((emask0 >> q) & 1u) b = 8u | ne++;
            else b = no | ((int)no == mark ? 16u : 0u), ++no;
            e[q >> 2] |= b << ((q & 3) * 8);
        }
        State s{0, 0, e[0], e[1], e[2]};
        move_right(T, s, (int)m);
        const uint32_t p0 = prmt(s.e0, s.e1, T.sy_psel[sym][0]), p1 = prmt(s.e0, s.e1, T.sy_psel[sym][1]),
                       p2 = prmt(s.e2, s.e2, T.sy_psel[sym][2]);
        const uint32_t em0 = gather4(p0, 3), em1 = gather4(p1, 3), em2 = gather4(p2, 3), emask = em0 | (em1 << 4) | (em2 << 8);
        uint32_t omask = gather4(p0, 4) | (gather4(p1, 4) << 4) | (gather4(p2, 4) << 8);
        omask ^= (0xF00u ^ emask) & (0u - (uint32_t)T.sy_fx[sym]);
        const uint32_t n0 = __popc(em0), n1 = __popc(em1);
        const uint32_t f0 = T.flp[(em0 << 4) | (omask & 15u)], f1 = T.flp[(em1 << 4) | ((omask >> 4) & 15u)],
                       f2 = T.flp[(em2 << 4) | (omask >> 8)];
        const uint32_t row = (f0 >> 4) | ((f1 >> 4) << (4 - n0)) | ((f2 >> 4) << (8 - n0 - n1));
        if (mark < 0) {
            base = row;
            slice = T.slice_rank[emask];
            flips = (f0 & 15u) | ((f1 & 15u) << n0) | ((f2 & 15u) << (n0 + n1));
            order = T.cmp4[em0][labels8(p0)] | ((uint32_t)T.cmp4[em1][labels8(p1)] << (2 * n0)) |
                    ((uint32_t)T.cmp4[em2][labels8(p2)] << (2 * (n0 + n1)));
        } else {
            perm[mark >> 2] |= (row ^ base) << (8 * (mark & 3));
        }
    }
    const uint32_t kind = (uint32_t)T.eorder_rank[order] * 16u + flips;
    if (MODE == KIND_304) base = T.sy_swap[sym] ? 0xFFu : 0u;  // (the row holds U edges: positions move, U and D may swap)
    desc[i] = make_uint4(slice | ((MODE == KIND_304 ? kind : kind * 16u + sym) << 9) | (base << 24), perm[0], perm[1], 0u);
}

// Lookup tables of the column permutations: of NCH groups of CB columns, the columns that the group's
// bits come from.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) rows_lut(const DevTables* __restrict__ gT, uint32_t* __restrict__ lut) {
    using RT = Rows<MODE, NEC>;
    __shared__ DevTables T;
    stage_tables(T, gT);
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= RT::N_LUT * RT::LUT) return;
    const uint32_t id = i / RT::LUT, chunk = (i % RT::LUT) >> RT::CB, bits = i & ((1u << RT::CB) - 1u);
    const uint32_t par = id & 1u, sym = (id >> 1) & 15u, kind = MODE == KIND_304 ? id : id >> 5;
    const uint32_t order = T.eorder_unrank[kind >> 4], toggle = kind & 15u;
    uint32_t out = 0;
    for (uint32_t col = 0; col < RT::C; ++col) {
        const uint32_t content = MODE == KIND_304 ? col : T.gen_rep[par][col];
        uint32_t flips = toggle, labels = 0;
        for (uint32_t j = 0; j < 4; ++j) {  // slot j takes what was in slot `from`
            const uint32_t from = (order >> (2 * j)) & 3u;
            flips ^= ((content >> from) & 1u) << j;
            if (MODE != KIND_304) labels |= ((T.eorder_unrank[content >> 4] >> (2 * from)) & 3u) << (2 * j);
        }
        const uint32_t to = MODE == KIND_304 ? flips : T.genc[((uint32_t)T.sy_lab[sym][labels] << 4) | flips];
        if (to / RT::CB == chunk && ((bits >> (to % RT::CB)) & 1u)) out |= 1u << col;
    }
    lut[i] = out;
}

// ---- forward passes: a listed frontier -----------------------------------------------------------

// Gives entry idx distance d if it has none: true for the one claim that did.
template <int MODE, int NEC>
__device__ __forceinline__ bool claim_entry(const RowsParams& P, uint64_t idx, uint32_t d, uint32_t& claims) {
    using RT = Rows<MODE, NEC>;
    const uint64_t row = idx / RT::C;
    const uint32_t col = (uint32_t)(idx - row * RT::C);
    constexpr uint32_t W = 8u * sizeof(typename RT::Word);  // bits of a plane's word
    volatile uint32_t* q = P.codes + row * RT::QW;
    uint32_t have = 0;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k) have |= ((q[k * W / 32u] >> (k * W % 32u + col)) & 1u) << k;
    if (have != 15u) return false;
    ++claims;
    bool first = true, won = false;
#pragma unroll
    for (uint32_t k = 0; k < 4; ++k)  // (distances below 15 have a 0 bit: the first one decides)
        if (!((d >> k) & 1u) && (first || won)) {
            const uint32_t bit = 1u << (k * W % 32u + col);
            const uint32_t old = atomicAnd(P.codes + row * RT::QW + k * W / 32u, ~bit);
            if (first) won = (old & bit) != 0u, first = false;
        }
    return won;
}

// Claims the coset of state n and its images under the symmetries that fix its corner class
// representative (kernels.cu:507-528), and lists what was claimed (or sets its frontier bits).
template <int MODE, int NEC>
__device__ __forceinline__ uint32_t claim_state(const DevTables& T, const RowsParams& P, const State& n, uint32_t d,
                                                uint64_t* list, uint32_t cap, uint32_t& reads, uint32_t& claims) {
    using RT = Rows<MODE, NEC>;
    const uint32_t packed = __ldg(P.classidx + corner_raw_dev(T, n)), cls = packed >> 4, sym = packed & 15u;
    uint32_t stab = __ldg(P.class_stab + cls), found = 0;
    while (stab) {
        const uint32_t t = __ffs(stab) - 1;
        stab &= stab - 1;
        const uint64_t idx = (uint64_t)cls * KindTraits<MODE, NEC>::N_EDGE + edge_coord_sym<MODE, NEC>(T, n, T.sym_mul[t][sym]);
        ++reads;
        if (!claim_entry<MODE, NEC>(P, idx, d, claims)) continue;
        ++found;
        if (list) {
            const unsigned long long at = atomicAdd(P.counter + 3, 1ull);
            if (at < cap) list[at] = idx;
        } else {
            const uint64_t row = idx / RT::C, bit = row * (8u * sizeof(typename RT::Word)) + (idx - row * RT::C);
            atomicOr(reinterpret_cast<uint32_t*>(P.next) + bit / 32u, 1u << (bit % 32u));
            P.next_flag[row / RT::R] = 1u;
        }
    }
    return found;
}

template <int MODE, int NEC>
__global__ void rows_seed(const DevTables* __restrict__ gT, RowsParams P, uint64_t* list, uint32_t cap) {
    __shared__ DevTables T;
    stage_tables(T, gT);
    if (threadIdx.x) return;
    uint32_t reads = 0, claims = 0;
    const State s{0x03020100u, 0x07060504u, 0x03020100u, 0x07060504u, 0x0B0A0908u};
    atomicAdd(P.counter, (unsigned long long)claim_state<MODE, NEC>(T, P, s, 0u, list, cap, reads, claims));
}

// One listed entry and move per thread.  out null: the claimed entries go to the frontier bits.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) rows_push(const DevTables* __restrict__ gT, RowsParams P, const uint64_t* __restrict__ in,
                                                 uint32_t n, uint64_t* out, uint32_t cap, uint32_t d) {
    __shared__ DevTables T;
    stage_tables(T, gT);
    unsigned long long found = 0;
    uint32_t reads = 0, claims = 0;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n * 18u; i += gridDim.x * blockDim.x) {
        State s;
        unrank_dev<MODE, NEC>(T, P.class_rep, in[i / 18u], s);
        move_right(T, s, (int)(i % 18u));
        found += claim_state<MODE, NEC>(T, P, s, d, out, cap, reads, claims);
    }
    add_count(P.counter, found);
    add_count(P.counter + 1, reads);
    add_count(P.counter + 2, claims);
}

// The frontier bits of distance d (at most 14), read off the planes: for a frontier that outgrew its list,
// whose claims past the list's end were given their distance but not listed.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) rows_mark(RowsParams P, uint64_t n_rows, uint32_t d) {
    using RT = Rows<MODE, NEC>;
    for (uint64_t row = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; row < n_rows; row += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t p[4], eq = RT::ALL;
        load_codes<RT>(P.codes, row, p);
#pragma unroll
        for (uint32_t j = 0; j < 4; ++j) eq &= (d >> j) & 1u ? p[j] : ~p[j];
        reinterpret_cast<typename RT::Word*>(P.next)[row] = (typename RT::Word)eq;
        if (eq) P.next_flag[row / RT::R] = 1u;
    }
}

// ---- dense passes: unreached entries look for a neighbour in the frontier --------------------------

// The lane's k-th row of a block.  Group kinds: rows k = 0..3 have even flip parity, 4..7 odd, so
// that a warp's lookup uses one column permutation.
template <int MODE>
__device__ __forceinline__ uint32_t lane_row(uint32_t lane, uint32_t k) {
    if (MODE == KIND_304) return lane + 32u * k;
    const uint32_t x = lane | ((k & 3u) << 5);
    return (x << 1) | ((__popc(x) & 1u) ^ (k >> 2));
}

// A row's bits as byte masks, and their permutation by rows_desc's bytes (they set different bits, so
// their sum, in the top byte of the product, is their union).
__device__ __forceinline__ uint2 row_bytes(uint32_t row) {
    return make_uint2((((row & 15u) * 0x00204081u) & 0x01010101u) * 255u, (((row >> 4) * 0x00204081u) & 0x01010101u) * 255u);
}
__device__ __forceinline__ uint32_t permute8(uint2 row, uint32_t y, uint32_t z) {
    return (((y & row.x) + (z & row.y)) * 0x01010101u) >> 24;
}

// A warp takes a (class, slice) block.  Blocks go slice by slice, so the warps of an SM work on
// neighbouring classes of one slice and share the lookups of its moves in L1.  A row's bits are
// permuted by lookups of CB bits: a group's 32 (16) entries lie in different banks, so 32 lanes with any
// groups read them at once.
//
// Bound by issue (59%, 32 warps per SM) and the lookups, not by memory: of a dense pass of 304 (5.5 G
// entries, 15-19 ms) DRAM moves 21 GB.  Measured on B200, whole builds on the device before (a byte per
// entry; every neighbour unranked, moved and indexed) and now: 304 0.46 -> 0.068 s, s4 base 3 1.34 ->
// 0.13, d4t 2.41 -> 0.20; its dense passes 129 / 396 / 1,086 / 586 -> 29 / 48 / 49 / 32 ms.  Held to 5 or
// 6 blocks an SM the rows of the group kinds spill: s4 33 and 36 ms a pass against 29.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256, 4) rows_pull(RowsParams P, uint32_t d) {
    using RT = Rows<MODE, NEC>;
    using Word = typename RT::Word;
    constexpr uint32_t K = RT::LANE_ROWS, FULL = 0xFFFFFFFFu;
    __shared__ uint8_t urank[256];   // 304: U layouts
    __shared__ uint8_t ulayout[72];
    if (MODE == KIND_304) {
        for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x) {
            uint32_t rank = 0;  // of the 4-bit masks in the order of the sorted positions
            if (__popc(i) == 4) {
                for (uint32_t j = 0; j < 256u; ++j)
                    if (__popc(j) == 4 && __brev(j) > __brev(i)) ++rank;
                ulayout[rank] = (uint8_t)i;
            }
            urank[i] = (uint8_t)rank;
        }
        __syncthreads();
    }
    const uint32_t lane = threadIdx.x & 31u;
    const Word* const cur = reinterpret_cast<const Word*>(P.cur);
    Word* const next = reinterpret_cast<Word*>(P.next);
    const uint32_t n_warps = gridDim.x * (blockDim.x >> 5);
    uint2 bytes[MODE == KIND_304 ? K : 1u];  // of the lane's rows (group kinds: its first one)
#pragma unroll
    for (uint32_t k = 0; k < (MODE == KIND_304 ? K : 1u); ++k) {
        const uint32_t r = lane_row<MODE>(lane, k);
        bytes[k] = row_bytes(MODE != KIND_304 ? r : r < RT::R ? ulayout[r] : 0u);
    }
    unsigned long long found = 0, read = 0;
    for (uint32_t b = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); b < (uint32_t)RT::N_BLOCKS; b += n_warps) {
        const uint32_t slice = b / N_CLASSES, cls = b - slice * N_CLASSES, blk = cls * N_SLICE + slice;
        const uint64_t row0 = (uint64_t)blk * RT::R;
        uint32_t rem[K], any = 0;
#pragma unroll
        for (uint32_t k = 0; k < K; ++k) {
            const uint32_t r = lane_row<MODE>(lane, k);
            rem[k] = 0;
            if (r < RT::R) {
                uint32_t p[4];
                load_codes<RT>(P.codes, row0 + r, p);
                rem[k] = unreached<RT>(P, row0 + r, p);
            }
            any |= rem[k];
        }
        uint32_t got = 0;
        if (__any_sync(FULL, any != 0u)) {
            // lane m: the block that move m leads to
            uint4 ds = make_uint4(0u, 0u, 0u, 0u);
            uint32_t nb = 0, busy = 0;
            if (lane < 18u) {
                const uint32_t cm = __ldg(P.cmove + cls * 18u + lane);
                ds = __ldg(P.desc + (slice * 18u + lane) * 16u + (cm & 15u));
                nb = (cm >> 4) * N_SLICE + (ds.x & 511u);
                busy = P.cur_flag[nb];
            }
            for (uint32_t left = __ballot_sync(FULL, busy != 0u); left; left &= left - 1u) {
                const int m = __ffs(left) - 1;
                const uint32_t dx = __shfl_sync(FULL, ds.x, m), y = __shfl_sync(FULL, ds.y, m), z = __shfl_sync(FULL, ds.z, m);
                const Word* const f = cur + (uint64_t)__shfl_sync(FULL, nb, m) * RT::R;
                const uint32_t flip = dx >> 24, id = (dx >> 9) & 0x1FFFu;
                ++read;
                uint32_t w[K];
                if constexpr (MODE == KIND_304) {
#pragma unroll
                    for (uint32_t k = 0; k < K; ++k) {
                        const uint32_t r = lane_row<MODE>(lane, k);
                        w[k] = r < RT::R ? f[urank[permute8(bytes[k], y, z) ^ flip]] : 0u;
                    }
                } else {
                    // (row k differs from row 0 in bits 6 and 7, k's, and in bit 0, which the parity sets)
                    const uint32_t mine = permute8(bytes[0], y, z) ^ flip;
                    const uint32_t b0 = y & 0xFFu, b6 = (z >> 16) & 0xFFu, b7 = z >> 24;
#pragma unroll
                    for (uint32_t k = 0; k < K; ++k) {
                        const uint32_t r = lane_row<MODE>(0u, k);
                        w[k] = f[mine ^ (r & 1u ? b0 : 0u) ^ (r & 64u ? b6 : 0u) ^ (r & 128u ? b7 : 0u)];
                    }
                }
                any = 0;
#pragma unroll
                for (uint32_t k = 0; k < K; ++k) {
                    if (__any_sync(FULL, w[k] && rem[k])) {
                        const uint32_t* t = P.lut + (MODE == KIND_304 ? id : id * 2u + (k >> 2)) * RT::LUT;
                        uint32_t hit = 0;
#pragma unroll
                        for (uint32_t c = 0; c < RT::NCH; ++c)
                            hit |= __ldg(t + (c << RT::CB) + ((w[k] >> (c * RT::CB)) & ((1u << RT::CB) - 1u)));
                        rem[k] &= ~hit;
                    }
                    any |= rem[k];
                }
                if (!__any_sync(FULL, any != 0u)) break;
            }
            // what went from unreached to reached
#pragma unroll
            for (uint32_t k = 0; k < K; ++k) {
                const uint32_t r = lane_row<MODE>(lane, k);
                if (r >= RT::R) continue;
                uint32_t p[4];
                load_codes<RT>(P.codes, row0 + r, p);
                const uint32_t hit = unreached<RT>(P, row0 + r, p) & ~rem[k];
                rem[k] = hit;
                if (hit) {
#pragma unroll
                    for (uint32_t j = 0; j < 4; ++j)
                        if (!((d >> j) & 1u)) p[j] &= ~hit;
                    store_codes<RT>(P.codes, row0 + r, p);
                    if (P.late && !((d >> 4) & 1u)) reinterpret_cast<Word*>(P.late)[row0 + r] &= (Word)~hit;
                    found += __popc(hit);
                    got = 1;
                }
            }
        } else {
#pragma unroll
            for (uint32_t k = 0; k < K; ++k) rem[k] = 0;
        }
        // the next frontier (its buffer holds the one before the current)
        got = __any_sync(FULL, got != 0u);
        if (got || P.next_flag[blk]) {
#pragma unroll
            for (uint32_t k = 0; k < K; ++k) {
                const uint32_t r = lane_row<MODE>(lane, k);
                if (r < RT::R) next[row0 + r] = (Word)rem[k];
            }
            __syncwarp();
            if (lane == 0u) P.next_flag[blk] = (uint8_t)got;
        }
    }
    add_count(P.counter, found);
    add_count(P.counter + 1, lane == 0u ? read * (RT::R * sizeof(Word) / 32u) : 0ull);
}

// The fifth plane when distances pass 14: set for every entry not yet reached, so that 1111 with it is
// "not reached" and 1111 without it is distance 15.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) rows_late(RowsParams P, void* late) {
    using RT = Rows<MODE, NEC>;
    for (uint64_t row = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; row < RT::N_ROWS; row += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t p[4];
        load_codes<RT>(P.codes, row, p);
        reinterpret_cast<typename RT::Word*>(late)[row] = (typename RT::Word)(p[0] & p[1] & p[2] & p[3] & RT::ALL);
    }
}

// Entries per distance (31: not reached), for the build's self-check.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) rows_histogram(RowsParams P, unsigned long long* __restrict__ hist) {
    using RT = Rows<MODE, NEC>;
    __shared__ unsigned long long sh[32];
    if (threadIdx.x < 32u) sh[threadIdx.x] = 0;
    __syncthreads();
    uint32_t local[16] = {}, deep[16] = {};
    for (uint64_t row = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; row < RT::N_ROWS; row += (uint64_t)gridDim.x * blockDim.x) {
        uint32_t p[4];
        load_codes<RT>(P.codes, row, p);
        const uint32_t late = P.late ? reinterpret_cast<const typename RT::Word*>(P.late)[row] : p[0] & p[1] & p[2] & p[3];
#pragma unroll
        for (uint32_t v = 0; v < 16; ++v) {
            const uint32_t eq = (v & 1u ? p[0] : ~p[0]) & (v & 2u ? p[1] : ~p[1]) & (v & 4u ? p[2] : ~p[2]) &
                                (v & 8u ? p[3] : ~p[3]) & RT::ALL;
            local[v] += __popc(eq & ~late);
            deep[v] += __popc(eq & late);
        }
    }
#pragma unroll
    for (uint32_t v = 0; v < 16; ++v) {
        if (local[v]) atomicAdd(&sh[v], (unsigned long long)local[v]);
        if (deep[v]) atomicAdd(&sh[16u + v], (unsigned long long)deep[v]);
    }
    __syncthreads();
    if (threadIdx.x < 32u && sh[threadIdx.x]) atomicAdd(&hist[threadIdx.x], sh[threadIdx.x]);
}

// ---- encoders: 32 entries at a time, a word per bit of the distance --------------------------------

// The distances of entries e0 .. e0 + 32 NW as NW words per bit (entries past the end: all ones).
template <int MODE, int NEC, int NW>
__device__ __forceinline__ void fetch_planes(const RowsParams& P, uint64_t e0, uint32_t v[5][NW]) {
    using RT = Rows<MODE, NEC>;
    uint64_t row = e0 / RT::C;
    const uint32_t skip = (uint32_t)(e0 - row * RT::C);
    unsigned long long acc[5];
    uint32_t fill = 0;
#pragma unroll
    for (int b = 0; b < 5; ++b) acc[b] = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        while (fill < 32u) {
            uint32_t p[4] = {RT::ALL, RT::ALL, RT::ALL, RT::ALL}, late = 0;
            if (row < RT::N_ROWS) {
                load_codes<RT>(P.codes, row, p);
                if (P.late) late = reinterpret_cast<const typename RT::Word*>(P.late)[row];
            }
            const uint32_t cut = fill == 0u && w == 0 ? skip : 0u;
#pragma unroll
            for (int b = 0; b < 4; ++b) acc[b] |= (unsigned long long)((p[b] & RT::ALL) >> cut) << fill;
            acc[4] |= (unsigned long long)(late >> cut) << fill;
            fill += RT::C - cut;
            ++row;
        }
#pragma unroll
        for (int b = 0; b < 5; ++b) v[b][w] = (uint32_t)acc[b], acc[b] >>= 32;
        fill -= 32u;
    }
}

// Smallest distance among the entries of `valid`; then distance - that minimum, as bit planes.
template <int NW>
__device__ __forceinline__ uint32_t minimum_and_offsets(uint32_t v[5][NW], const uint32_t valid[NW]) {
    uint32_t cand[NW], m = 0;
#pragma unroll
    for (int w = 0; w < NW; ++w) cand[w] = valid[w];
#pragma unroll
    for (int b = 4; b >= 0; --b) {
        uint32_t low[NW], any = 0;
#pragma unroll
        for (int w = 0; w < NW; ++w) low[w] = cand[w] & ~v[b][w], any |= low[w];
        if (!any) m |= 1u << b;
#pragma unroll
        for (int w = 0; w < NW; ++w) cand[w] = any ? low[w] : cand[w];
    }
#pragma unroll
    for (int w = 0; w < NW; ++w) {
        uint32_t borrow = 0;
#pragma unroll
        for (int b = 0; b < 5; ++b) {
            const uint32_t mb = 0u - ((m >> b) & 1u), x = v[b][w];
            v[b][w] = x ^ mb ^ borrow;
            borrow = (~x & (mb | borrow)) | (mb & borrow);
        }
    }
    return m;
}

__device__ __forceinline__ uint32_t spread16(uint32_t x) {  // bit i of 16 to bit 2i
    x = (x | (x << 8)) & 0x00FF00FFu;
    x = (x | (x << 4)) & 0x0F0F0F0Fu;
    x = (x | (x << 2)) & 0x33333333u;
    return (x | (x << 1)) & 0x55555555u;
}

template <int NW>
__device__ __forceinline__ void valid_mask(uint32_t n, uint32_t valid[NW]) {
#pragma unroll
    for (int w = 0; w < NW; ++w) valid[w] = n >= 32u * (w + 1) ? ~0u : n > 32u * w ? (1u << (n - 32u * w)) - 1u : 0u;
}

// 2-bit block file: per 124-entry block, u8 minimum then offsets min(distance - minimum, 3) at bit
// 8 + 2j; entries past the end keep offset 0 (kernels.cu:396-434, 485-503).
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) encode_block(RowsParams P, uint64_t n_entries, uint64_t n_blocks, uint32_t* __restrict__ out) {
    const uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (b >= n_blocks) return;
    uint32_t v[5][4], valid[4];
    fetch_planes<MODE, NEC, 4>(P, b * 124u, v);
    valid_mask<4>((uint32_t)min((uint64_t)124u, n_entries - b * 124u), valid);
    const uint32_t m = minimum_and_offsets<4>(v, valid);
    uint32_t o[8], carry = m;  // (the minimum takes the place of the bits shifted in)
#pragma unroll
    for (int w = 0; w < 4; ++w) {
        const uint32_t big = v[2][w] | v[3][w] | v[4][w], lo = (v[0][w] | big) & valid[w], hi = (v[1][w] | big) & valid[w];
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const uint32_t x = spread16((lo >> (16 * half)) & 0xFFFFu) | (spread16((hi >> (16 * half)) & 0xFFFFu) << 1);
            o[2 * w + half] = (x << 8) | carry;
            carry = x >> 24;
        }
    }
    uint4* dst = reinterpret_cast<uint4*>(out + b * 8u);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// Base-3 code of a 155-entry block whose entries' value - m is given as bit planes: header m | cut <<
// 6, the cut in 0..3 that maximises the sum of the encoded bounds (the lowest on ties), then five base-3
// digits per byte, least significant first: 0 up to m + cut, 1 at m + cut + 1, 2 above.
__device__ __forceinline__ void write_b3(uint32_t v[5][5], const uint32_t valid[5], uint32_t m, const uint8_t* three, uint32_t* __restrict__ out) {
    uint32_t count[5] = {0, 0, 0, 0, 0}, total = 0;  // entries at m + 0 .. m + 4
#pragma unroll
    for (int w = 0; w < 5; ++w) {
        const uint32_t small = ~(v[3][w] | v[4][w]) & valid[w];
        count[0] += __popc(small & ~v[2][w] & ~v[1][w] & ~v[0][w]);
        count[1] += __popc(small & ~v[2][w] & ~v[1][w] & v[0][w]);
        count[2] += __popc(small & ~v[2][w] & v[1][w] & ~v[0][w]);
        count[3] += __popc(small & ~v[2][w] & v[1][w] & v[0][w]);
        count[4] += __popc(small & v[2][w] & ~v[1][w] & ~v[0][w]);
        total += __popc(valid[w]);
    }
    uint32_t best = 0, best_score = 0, upto = 0;
#pragma unroll
    for (uint32_t c = 0; c < 4; ++c) {
        upto += count[c];
        const uint32_t score = total * m + count[c + 1] * (c + 1u) + (total - upto - count[c + 1]) * (c + 2u);
        if (score > best_score) best_score = score, best = c;
    }
    unsigned long long d1[3], d2[3];  // digit 1 and digit 2 of the entries, 64 a word
    const uint32_t t = best + 1u;
#pragma unroll
    for (int w = 0; w < 6; ++w) {
        uint32_t is1 = 0, is2 = 0;
        if (w < 5) {
            const uint32_t eq0 = v[0][w] ^ (0u - (~t & 1u)), eq1 = v[1][w] ^ (0u - (~(t >> 1) & 1u)), eq2 = v[2][w] ^ (0u - (~(t >> 2) & 1u));
            const uint32_t high = v[3][w] | v[4][w];
            is1 = eq0 & eq1 & eq2 & ~high & valid[w];
            // above t, of 1..4: by comparing three bits
            const uint32_t t0 = 0u - (t & 1u), t1 = 0u - ((t >> 1) & 1u), t2 = 0u - ((t >> 2) & 1u);
            const uint32_t gt = (v[2][w] & ~t2) | (~(v[2][w] ^ t2) & ((v[1][w] & ~t1) | (~(v[1][w] ^ t1) & (v[0][w] & ~t0))));
            is2 = (gt | high) & valid[w];
        }
        if (w & 1) d1[w / 2] |= (unsigned long long)is1 << 32, d2[w / 2] |= (unsigned long long)is2 << 32;
        else d1[w / 2] = is1, d2[w / 2] = is2;
    }
    uint32_t o[8];
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        uint32_t byte;
        if (i == 0) {
            byte = m | (best << 6);
        } else {
            const int bit = 5 * (i - 1), k = bit / 64, s = bit % 64;
            uint32_t a = (uint32_t)(d1[k] >> s), c = (uint32_t)(d2[k] >> s);
            if (s > 59) a |= (uint32_t)(d1[k + 1 < 3 ? k + 1 : 2] << (64 - s)), c |= (uint32_t)(d2[k + 1 < 3 ? k + 1 : 2] << (64 - s));
            byte = three[a & 31u] + 2u * three[c & 31u];
        }
        if (i % 4 == 0) o[i / 4] = byte;
        else o[i / 4] |= byte << (8 * (i % 4));
    }
    uint4* dst = reinterpret_cast<uint4*>(out);
    dst[0] = make_uint4(o[0], o[1], o[2], o[3]);
    dst[1] = make_uint4(o[4], o[5], o[6], o[7]);
}

// Sum of 3^k over the set bits k of a five-bit mask.
__device__ __forceinline__ void stage_three(uint8_t three[32]) {
    if (threadIdx.x < 32u) {
        const uint32_t x = threadIdx.x;
        three[x] = (uint8_t)((x & 1u) + 3u * ((x >> 1) & 1u) + 9u * ((x >> 2) & 1u) + 27u * ((x >> 3) & 1u) + 81u * (x >> 4));
    }
    __syncthreads();
}

// Base-3 file (kernels.cu:1839-1869).  The value of an entry is what the reference recovers from its
// 2-bit block and mod-3 tables: exact up to the 124-block minimum + 5, otherwise the smallest value >=
// minimum + 3 with the right residue -- which only lowers entries 6 or more above their 124-block's
// minimum (rare: such a block holds an entry within 8 moves of solved), one at a time below.
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) encode_b3(RowsParams P, const uint32_t* __restrict__ blk, uint64_t n_entries,
                                                 uint64_t n_blocks, uint32_t* __restrict__ out) {
    __shared__ uint8_t three[32];
    stage_three(three);
    const uint64_t b = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (b >= n_blocks) return;
    const uint64_t first = b * 155u;
    const uint32_t n = (uint32_t)min((uint64_t)155u, n_entries - first);
    uint32_t v[5][5], valid[5];
    fetch_planes<MODE, NEC, 5>(P, first, v);
    valid_mask<5>(n, valid);
    for (uint64_t s = first / 124u; s * 124u < first + n; ++s) {  // the 124-blocks of these entries
        const uint32_t m124 = __ldg(blk + s * 8u) & 0xFFu;
        uint32_t mask[5], high[5], any = 0;
        const uint32_t lo = s * 124u > first ? (uint32_t)(s * 124u - first) : 0u;
        const uint32_t hi = (uint32_t)min((uint64_t)n, (s + 1u) * 124u - first);
        uint32_t below[5];
        valid_mask<5>(hi, mask);
        valid_mask<5>(lo, below);
#pragma unroll
        for (int w = 0; w < 5; ++w) {
            mask[w] &= ~below[w];
            // distance >= m124 + 6, bit by bit from the top
            uint32_t ge = ~0u;
            const uint32_t t = m124 + 6u;
#pragma unroll
            for (int k = 0; k < 5; ++k) {
                const uint32_t tb = 0u - ((t >> k) & 1u), x = v[k][w];
                ge = (x & ~tb) | (~(x ^ tb) & ge);
            }
            high[w] = t > 31u ? 0u : ge & mask[w];
            any |= high[w];
        }
        if (!any) continue;
#pragma unroll
        for (int w = 0; w < 5; ++w)
            for (uint32_t h = high[w]; h; h &= h - 1u) {
                const int j = __ffs(h) - 1;
                uint32_t x = 0;
#pragma unroll
                for (int k = 0; k < 5; ++k) x |= ((v[k][w] >> j) & 1u) << k;
                x = m124 + 3u + (x - m124 - 3u) % 3u;
#pragma unroll
                for (int k = 0; k < 5; ++k) v[k][w] = (v[k][w] & ~(1u << j)) | (((x >> k) & 1u) << j);
            }
    }
    const uint32_t m = minimum_and_offsets<5>(v, valid);
    write_b3(v, valid, m, three, out + b * 8u);
}

// Mod-3 file: per little-endian uint32 sixteen entries, two bits each, distance mod 3 (3 past the end,
// as the reference's table starts all ones; table.py:94-95).
template <int MODE, int NEC>
__global__ void __launch_bounds__(256) encode_mod3(RowsParams P, uint64_t n_entries, uint64_t n_words, uint32_t* __restrict__ out) {
    const uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x;
    if (i >= n_words) return;
    uint32_t v[5][1], valid[1], r0 = 0, r1 = 0;
    fetch_planes<MODE, NEC, 1>(P, i * 16u, v);
    valid_mask<1>((uint32_t)min((uint64_t)16u, n_entries - i * 16u), valid);
#pragma unroll
    for (int b = 0; b < 5; ++b) {  // add 1, 2, 1, 2, 1 (2^b mod 3) where the bit is set
        const uint32_t x = v[b][0], zero = ~(r0 | r1);
        const uint32_t n0 = b & 1 ? r1 : zero, n1 = b & 1 ? zero : r0;
        r0 = (x & n0) | (~x & r0);
        r1 = (x & n1) | (~x & r1);
    }
    out[i] = spread16((r0 | ~valid[0]) & 0xFFFFu) | (spread16((r1 | ~valid[0]) & 0xFFFFu) << 1);
}

}  // namespace ccs
