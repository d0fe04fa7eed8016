// Constant tables of the warp search kernel and the probe arithmetic on them: the same index and
// bound as probe_dev (cube_dev.cuh), from rows that one 128-bit shared load brings and with the masks
// of a word's four edges gathered in one multiply.
#pragma once

#include "cube_dev.cuh"

namespace ccs {

__device__ __forceinline__ uint32_t prmt_raw(uint32_t a, uint32_t b, uint32_t s) {
#ifdef CCS_HOST_EMULATION
    return __byte_perm(a, b, s);
#else
    uint32_t r;
    asm("prmt.b32 %0, %1, %2, %3;" : "=r"(r) : "r"(a), "r"(b), "r"(s));
    return r;
#endif
}

struct alignas(16) Word4 {
    uint32_t x, y, z, w;
};

// s * m by a row of right-move selectors.
__device__ __forceinline__ State warp_right(const WarpTables& T, const State& s, uint32_t m) {
    const Word4* r = reinterpret_cast<const Word4*>(T.right[m]);
    const Word4 a = r[0], b = r[1], c = r[2], d = r[3];
    State o;
    o.c0 = wrap_twist(prmt_raw(s.c0, s.c1, a.x) + a.z);
    o.c1 = wrap_twist(prmt_raw(s.c0, s.c1, a.y) + a.w);
    o.e0 = ((prmt_raw(s.e0, s.e1, b.x) & ~c.z) | (prmt_raw(s.e2, s.e2, b.w) & c.z)) ^ d.y;
    o.e1 = ((prmt_raw(s.e0, s.e1, b.y) & ~c.w) | (prmt_raw(s.e2, s.e2, c.x) & c.w)) ^ d.z;
    o.e2 = ((prmt_raw(s.e0, s.e1, b.z) & ~d.x) | (prmt_raw(s.e2, s.e2, c.y) & d.x)) ^ d.w;
    return o;
}

// m * s by a row of renamed cubies.
__device__ __forceinline__ State warp_left(const WarpTables& T, const State& s, uint32_t m) {
    const Word4* r = reinterpret_cast<const Word4*>(T.left[m]);
    const Word4 a = r[0];
    const uint32_t r2 = T.left[m][4];
    State o;
    o.c0 = wrap_twist(prmt_raw(a.x, a.y, nib_sel(s.c0 & 0x07070707u)) + (s.c0 & 0x18181818u));
    o.c1 = wrap_twist(prmt_raw(a.x, a.y, nib_sel(s.c1 & 0x07070707u)) + (s.c1 & 0x18181818u));
    const uint32_t e[3] = {s.e0, s.e1, s.e2};
    uint32_t n[3];
#pragma unroll
    for (int w = 0; w < 3; ++w) {
        const uint32_t v = e[w], sel = nib_sel(v & 0x07070707u), hi = prmt_raw(v << 4, 0u, 0xBA98u);  // cubies 8..11: 0xFF
        n[w] = ((prmt_raw(a.z, a.w, sel) & ~hi) | (prmt_raw(r2, r2, sel) & hi)) ^ (v & 0x10101010u);
    }
    o.e0 = n[0];
    o.e1 = n[1];
    o.e2 = n[2];
    return o;
}

// Move `m` of the cube on frame k: right multiplication in the forward frames, left in the inverse.
__device__ __forceinline__ State warp_step(const WarpTables& T, const State& s, uint32_t k, uint32_t m) {
    const uint32_t a = T.act[k][m];
    return k < 3u ? warp_right(T, s, a) : warp_left(T, s, a);
}

// One bit of each byte of a (bit 0) and of b (bit 4, masked by the caller's shift), as 4 + 4 bits.
__device__ __forceinline__ uint32_t gather8(uint32_t lo, uint32_t hi) {
    return (((lo & 0x01010101u) | (hi & 0x10101010u)) * 0x01020408u) >> 24;
}

__device__ __forceinline__ uint32_t warp_corner_raw(const WarpTables& T, uint32_t c0, uint32_t c1) {
    const uint32_t twist = __dp4a((c0 >> 3) & 0x03030303u, 0x1B090301u, 81u * __dp4a((c1 >> 3) & 0x00030303u, 0x00090301u, 0u));
    return twist * 70u + T.ccomb_rank[gather8(c0 >> 2, c1 << 2)];
}

// Edge coordinate of M_sym g M_sym^-1 (edge_coord_sym's).  A word's E mask and flips come from one
// gather, and its row of `flp` -- chosen by whether the symmetry flips E positions and E cubies --
// gives the flips compacted over the E positions (bits 0-3) and over the others (4-7) and how many
// E positions there are (8-10).
template <int MODE, int NEC>
__device__ __forceinline__ uint32_t warp_edge_coord(const WarpTables& T, const State& s, uint32_t sym, bool second) {
    const Word4 y = *reinterpret_cast<const Word4*>(T.sym[sym]);
    const uint32_t p0 = prmt_raw(s.e0, s.e1, y.x), p1 = prmt_raw(s.e0, s.e1, y.y), p2 = prmt_raw(s.e2, s.e2, y.z);
    const uint32_t i0 = gather8(p0 >> 3, p0), i1 = gather8(p1 >> 3, p1), i2 = gather8(p2 >> 3, p2);
    const uint16_t* row = T.flp[0] + (y.w & 0xFFFFu);
    const uint32_t f0 = row[i0], f1 = row[i1], f2 = T.flp[0][(y.w >> 16) + i2];
    const uint32_t m0 = i0 & 15u, m1 = i1 & 15u, m2 = i2 & 15u;
    const uint32_t n0 = f0 >> 8, n01 = n0 + (f1 >> 8);
    const uint32_t slice = T.slice_rank[m0 | (m1 << 4) | (m2 << 8)];
    const uint32_t eflips = (f0 & 15u) | ((f1 & 15u) << n0) | ((f2 & 15u) << n01);
    if (MODE == KIND_304) {
        const uint32_t u0 = gather8(p0 >> 3, ~(p0 | (p0 >> 1)) << 2), u1 = gather8(p1 >> 3, ~(p1 | (p1 >> 1)) << 2),
                       u2 = gather8(p2 >> 3, ~(p2 | (p2 >> 1)) << 2);
        const uint8_t* ump = T.ump[T.swap[sym]];
        const uint32_t u = ump[u0] | ((uint32_t)ump[u1] << (4u - n0)) | ((uint32_t)ump[u2] << (8u - n01));
        return (slice * 70u + T.ccomb_rank[u]) * 16u + eflips;
    } else {
        const uint32_t nflips = ((f0 >> 4) & 15u) | (((f1 >> 4) & 15u) << (4u - n0)) | (((f2 >> 4) & 15u) << (8u - n01));
        const uint32_t eord = T.cmp4[m0][labels8(p0)] | ((uint32_t)T.cmp4[m1][labels8(p1)] << (2u * n0)) |
                              ((uint32_t)T.cmp4[m2][labels8(p2)] << (2u * n01));
        return (slice * 256u + nflips) * (uint32_t)NEC + T.genc[second][((uint32_t)T.lab[sym][eord] << 4) | eflips];
    }
}

// The same bound as decode_sector.  The word is found in three halvings.  A base-3 digit k of a byte is
// the integer part of 3 x the fraction of byte / 3^(k + 1), that fraction being byte * 3^(4 - k) times
// 1/243 as a 32-bit fraction (rounded up: off by less than 2^-17, digits are 1/243 apart): two
// multiplies where a division by a power chosen at run time took a loop of them.
template <int FMT>
__device__ __forceinline__ uint32_t warp_decode(const uint32_t w[8], uint32_t j) {
    const uint32_t q5 = j / 5u;                                           // (base 3: byte 1 + q5, digit j % 5)
    const uint32_t q = FMT == FMT_B3 ? (q5 + 1u) >> 2 : (j + 4u) >> 4;    // word
    const bool b0 = q & 1u, b1 = q & 2u, b2 = q & 4u;
    const uint32_t a = b0 ? w[1] : w[0], b = b0 ? w[3] : w[2], c = b0 ? w[5] : w[4], d = b0 ? w[7] : w[6];
    const uint32_t e = b1 ? b : a, f = b1 ? d : c, v = b2 ? f : e;
    if (FMT == FMT_B3) {
        const uint32_t byte = (v >> ((8u * q5 + 8u) & 31u)) & 0xFFu;
        const uint32_t power = prmt_raw(0x03091B51u, 1u, (j - 5u * q5) | 0x7770u);  // 81, 27, 9, 3, 1
        const uint32_t digit = (uint32_t)(((unsigned long long)(byte * power * 17674763u) * 3u) >> 32);
        const uint32_t m = w[0] & 63u;
        return digit ? m + ((w[0] >> 6) & 3u) + digit : m;
    }
    return (w[0] & 0xFFu) + ((v >> ((2u * j + 8u) & 31u)) & 3u);
}

// The bound of one state (admission).
template <int MODE, int NEC, int FMT>
__device__ __forceinline__ uint32_t warp_probe(const WarpTables& T, const uint32_t* __restrict__ classidx,
                                               const uint32_t* __restrict__ tab, const State& s, bool second) {
    const uint32_t packed = __ldg(classidx + warp_corner_raw(T, s.c0, s.c1));
    uint32_t sector, j, w[8];
    split_sector<FMT, KindTraits<MODE, NEC>::N_EDGE>(packed >> 4, warp_edge_coord<MODE, NEC>(T, s, packed & 15u, second), sector, j);
    load_sector(tab + (uint64_t)sector * 8u, w);
    return warp_decode<FMT>(w, j);
}

}  // namespace ccs
