// Expansion of packed bfloat8_b / bfloat4_b tiles into tensor memory as the bf16 A operand of tcgen05.mma, for matmul_rows.cu.
// (matmul_decode_tmem.cu has an expansion of its own, for activations that tensor maps deliver in order.)
//
// A warp expands one 32x32 packed tile into the 32 TMEM lanes of its quadrant (lane = weight column) and 16 TMEM columns (two
// K values each): two 16x256b.x2 stores, one (bfloat4_b) or two transposing loads and the scale shuffles, all of them through
// the same memory pipe, next to byte permutes, masks and multiplies.
#pragma once
#include "epilogue.cuh"
#include "sm100_ptx.cuh"

namespace ttb {

__device__ __forceinline__ void ldmatrix_x2_trans_b8(uint32_t addr, uint32_t (&r)[4]) {
    asm volatile("ldmatrix.sync.aligned.m16n16.x2.trans.shared.b8 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(addr));
}
// Lanes +0..15, columns +0..15 of tensor memory: registers 0-3 hold columns 0-7, registers 4-7 columns 8-15.
__device__ __forceinline__ void tmem_st_16x256b_x2(uint32_t taddr, const uint32_t (&v)[8]) {
    asm volatile("tcgen05.st.sync.aligned.16x256b.x2.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]),
                 "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_st_wait() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// D[tmem] (+)= A[tmem] * B[smem]
__device__ __forceinline__ void mma_bf16_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, bool accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t"
        "}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"((uint32_t)accumulate)
        : "memory");
}

__device__ __forceinline__ uint32_t mul2(uint32_t a, uint32_t b) {
    __nv_bfloat162 v = __hmul2(*reinterpret_cast<__nv_bfloat162 *>(&a), *reinterpret_cast<__nv_bfloat162 *>(&b));
    return *reinterpret_cast<uint32_t *>(&v);
}
// Four codes (consecutive K of one column) -> two packed bf16 pairs, each multiplied by its pair of row scales.
__device__ __forceinline__ void expand4(uint32_t codes, uint32_t s01, uint32_t s23, uint32_t &o01, uint32_t &o23) {
    o01 = mul2(__byte_perm(codes, 0u, 0x1100u) & 0x807f807fu, s01);
    o23 = mul2(__byte_perm(codes, 0u, 0x3322u) & 0x807f807fu, s23);
}

// Where a lane's row address of the transposing load points, relative to the tile.
// bfloat8_b: lanes 0-15 give the rows of the left face, 16-31 of the right face.
__device__ __forceinline__ uint32_t expand_ld_offset8(int lane) { return 64u + (uint32_t)(lane >> 4) * 256u + (uint32_t)(lane & 15) * 16u; }
// bfloat4_b: a 16-byte row of the transposing load is a pair of K rows of one face (8 bytes = 16 nibbles each). Lanes 0-15 give the
// rows of the left faces (0 and 2), lanes 16-31 of the right faces; row r of the 16 is K row pair sigma(r) of the upper
// (sigma < 8) or lower face, with sigma chosen such that the four rows a lane receives (4q .. 4q+3, q = lane % 4) are K rows
// 4q..4q+3 of the upper and 4(q^2)..4(q^2)+3 of the lower face. (The same K rows of both faces would put the eight addresses of
// a phase on 64 bytes of banks twice.) K 16..31 of a block therefore stand in tensor memory with their halves of eight exchanged,
// and the activations' copies exchange theirs (expand_b_swap).
__device__ __forceinline__ uint32_t expand_ld_offset4(int lane) {
    const int r16 = lane & 15;
    const int pair = (r16 >> 2) * 2 + (r16 & 1);   // rows 4q, 4q+1: pairs 2q, 2q+1 above; rows 4q+2, 4q+3: pairs 2(q^2), 2(q^2)+1 below
    const uint32_t row = ((r16 >> 1) & 1) ? 256u + (uint32_t)(pair ^ 4) * 16u : (uint32_t)pair * 16u;
    return 64u + (uint32_t)(lane >> 4) * 128u + row;
}
// What to exclusive-or into the shared-memory address of a 16-byte chunk of the activation (operand B) whose K lies in the
// second half of a K block.
template <int FMT>
constexpr uint32_t expand_b_swap = FMT == TTB_BFLOAT4_B ? 16u : 0u;
template <int FMT>
__device__ __forceinline__ uint32_t expand_ld_offset(int lane) { return FMT == TTB_BFLOAT8_B ? expand_ld_offset8(lane) : expand_ld_offset4(lane); }
// Which of its quadrant's 32 weight columns a TMEM lane holds. bfloat8_b: the lane's own. bfloat4_b: a code byte carries two
// neighbouring columns, and the transposing load hands the even one to lanes 0..7 and the odd one to lanes 8..15 of every
// 16-lane half.
template <int FMT>
__device__ __forceinline__ int expand_column_of_lane(int lane) { return FMT == TTB_BFLOAT8_B ? lane : (lane & 16) + ((lane & 7) << 1) + ((lane >> 3) & 1); }

// The tile's 64 exponents as [e0, 0, e1, 0]: exponent bytes 2 * lane and 2 * lane + 1 (face order, 16 per face).
__device__ __forceinline__ uint32_t expand_exponents(uint32_t tile, int lane) {
    uint32_t e;
    asm volatile("ld.shared.u16 %0, [%1];" : "=r"(e) : "r"(tile + 2u * lane));
    return __byte_perm(e, 0u, 0x4140u);
}
__device__ __forceinline__ uint32_t expand_scale(uint32_t eh) { return (__vminu2(eh, 0x007f007fu) + 0x007f007fu) << 7; }   // 2^min(E, 127) per half

// The packed codes of one tile as a lane holds them: bfloat8_b two transposing loads (K 0..15: faces 0 and 1, K 16..31: faces 2
// and 3), bfloat4_b one.
template <int FMT>
struct TileCodes {
    uint32_t r[FMT == TTB_BFLOAT8_B ? 2 : 1][4];
    __device__ __forceinline__ void load(uint32_t addr) {
        ldmatrix_x2_trans_b8(addr, r[0]);
        if (FMT == TTB_BFLOAT8_B) ldmatrix_x2_trans_b8(addr + 512u, r[FMT == TTB_BFLOAT8_B ? 1 : 0]);
    }
};

// The lane whose scale pair belongs to this lane's first two K rows of face 2 * kh + nh (the next lane has the other two).
template <int FMT>
__device__ __forceinline__ int expand_scale_lane(int nh, int kh, int sh0) { return 8 * (2 * kh + nh) + (FMT == TTB_BFLOAT4_B && kh ? sh0 ^ 4 : sh0); }

// Column half `nh` (16 TMEM lanes) and K half `kh` of a tile: four registers of products.
template <int FMT>
__device__ __forceinline__ void expand_quarter(const TileCodes<FMT> &c, int nh, int kh, uint32_t s01, uint32_t s23, uint32_t *o) {
    if (FMT == TTB_BFLOAT8_B) {
        // face 2 * kh + nh; registers {2*nh, 2*nh+1} of the kh-th load: columns lane/4 and lane/4 + 8
        const uint32_t *const q = c.r[FMT == TTB_BFLOAT8_B ? kh : 0];
        expand4(q[2 * nh], s01, s23, o[0], o[1]);
        expand4(q[2 * nh + 1], s01, s23, o[2], o[3]);
    } else {
        // registers {2*nh, 2*nh+1}: four bytes of even and four of odd K rows, each byte the codes of columns 2p (low nibble) and
        // 2p + 1 (high nibble), p = lane / 4; bytes 2*kh and 2*kh+1 are this lane's four K rows of the kh-th face. (sign << 15) | (mantissa
        // << 4) is the weight divided by a power of two: the same subnormal trick and the same row scales as for bfloat8_b
        const uint32_t e = c.r[0][2 * nh], d = c.r[0][2 * nh + 1];
        const uint32_t lo_e = (e << 4) & 0xf0f0f0f0u, lo_o = (d << 4) & 0xf0f0f0f0u, hi_e = e & 0xf0f0f0f0u, hi_o = d & 0xf0f0f0f0u;
        const uint32_t sel0 = kh ? 0x6622u : 0x4400u, sel1 = kh ? 0x7733u : 0x5511u;
        o[0] = mul2(__byte_perm(lo_e, lo_o, sel0) & 0x80708070u, s01);   // column 2p: the first two K rows
        o[1] = mul2(__byte_perm(lo_e, lo_o, sel1) & 0x80708070u, s23);   //            the other two
        o[2] = mul2(__byte_perm(hi_e, hi_o, sel0) & 0x80708070u, s01);   // column 2p + 1
        o[3] = mul2(__byte_perm(hi_e, hi_o, sel1) & 0x80708070u, s23);
    }
}

// One packed tile (shared address `tile`) -> the 32 TMEM lanes of this warp's quadrant, 16 columns at a_col. `sh0`: 2 * (lane % 4),
// within a face's 8 scale pairs those of this lane's K rows.
// BIG: some exponent of the tile exceeds 127 (a row maximum of 2 or more), whose power of two needs a second factor.
template <int FMT, bool BIG>
__device__ __forceinline__ void expand_tile(uint32_t tile, uint32_t a_col, uint32_t ld_off, uint32_t eh, int sh0) {
    const uint32_t my_scale = expand_scale(eh);
    const uint32_t my_t = BIG ? (__vmaxu2(__vminu2(eh, 0x00fe00feu), 0x007f007fu) << 7) : 0u;
    TileCodes<FMT> c;
    c.load(tile + ld_off);
#pragma unroll
    for (int nh = 0; nh < 2; ++nh) {
        uint32_t o[8];
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) {
            const int f = expand_scale_lane<FMT>(nh, kh, sh0);
            expand_quarter<FMT>(c, nh, kh, __shfl_sync(0xffffffffu, my_scale, f), __shfl_sync(0xffffffffu, my_scale, f + 1), o + 4 * kh);
            if (BIG) {
                const uint32_t t01 = __shfl_sync(0xffffffffu, my_t, f), t23 = __shfl_sync(0xffffffffu, my_t, f + 1);
                o[4 * kh] = mul2(o[4 * kh], t01); o[4 * kh + 1] = mul2(o[4 * kh + 1], t23);
                o[4 * kh + 2] = mul2(o[4 * kh + 2], t01); o[4 * kh + 3] = mul2(o[4 * kh + 3], t23);
            }
        }
        // TMEM lanes 32*quad + 16*nh + {lane/4, lane/4 + 8}; columns: stage base + 8*kh + 2*(lane%4) + {0, 1}
        tmem_st_16x256b_x2(a_col + ((uint32_t)(nh * 16) << 16), o);
    }
}
template <int FMT>
__device__ __noinline__ void expand_tile_big(uint32_t tile, uint32_t a_col, uint32_t ld_off, uint32_t eh, int sh0) {
    expand_tile<FMT, true>(tile, a_col, ld_off, eh, sh0);
}

// Two tiles at once (the common case: no exponent above 127): the transposing loads of both go out first and the faces
// are expanded alternately, so that one tile's shuffles and stores wait behind the other's arithmetic.
template <int FMT>
__device__ __forceinline__ void expand_pair(uint32_t tile0, uint32_t tile1, uint32_t a_col0, uint32_t a_col1, uint32_t ld_off, uint32_t eh0, uint32_t eh1,
                                            int sh0) {
    TileCodes<FMT> c, d;
    c.load(tile0 + ld_off);
    d.load(tile1 + ld_off);
    const uint32_t scale0 = expand_scale(eh0), scale1 = expand_scale(eh1);
#pragma unroll
    for (int nh = 0; nh < 2; ++nh) {
        uint32_t o[8], w[8];
#pragma unroll
        for (int kh = 0; kh < 2; ++kh) {
            const int f = expand_scale_lane<FMT>(nh, kh, sh0);
            const uint32_t p01 = __shfl_sync(0xffffffffu, scale0, f), p23 = __shfl_sync(0xffffffffu, scale0, f + 1);
            const uint32_t q01 = __shfl_sync(0xffffffffu, scale1, f), q23 = __shfl_sync(0xffffffffu, scale1, f + 1);
            expand_quarter<FMT>(c, nh, kh, p01, p23, o + 4 * kh);
            expand_quarter<FMT>(d, nh, kh, q01, q23, w + 4 * kh);
        }
        tmem_st_16x256b_x2(a_col0 + ((uint32_t)(nh * 16) << 16), o);
        tmem_st_16x256b_x2(a_col1 + ((uint32_t)(nh * 16) << 16), w);
    }
}

// `count` (1 or 2) consecutive tiles `stride` bytes apart.
template <int FMT>
__device__ __forceinline__ void expand_tiles(uint32_t tile, uint32_t stride, uint32_t a_col, uint32_t a_stride, int count, uint32_t ld_off, int sh0, int lane) {
    const uint32_t eh0 = expand_exponents(tile, lane), eh1 = count > 1 ? expand_exponents(tile + stride, lane) : 0u;
    if (count > 1 && !__any_sync(0xffffffffu, ((eh0 | eh1) & 0x00800080u) != 0u)) {
        expand_pair<FMT>(tile, tile + stride, a_col, a_col + a_stride, ld_off, eh0, eh1, sh0);
    } else {
        // a lone last tile, or an exponent above 127 somewhere (a row maximum of 2 or more): one tile at a time
        for (int t = 0; t < count; ++t) {
            const uint32_t e = t ? eh1 : eh0;
            if (__any_sync(0xffffffffu, (e & 0x00800080u) != 0u))
                expand_tile_big<FMT>(tile + t * stride, a_col + t * a_stride, ld_off, e, sh0);
            else
                expand_tile<FMT, false>(tile + t * stride, a_col + t * a_stride, ld_off, e, sh0);
        }
    }
}

}  // namespace ttb
