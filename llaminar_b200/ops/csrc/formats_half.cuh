// Dequantisation of half a weight chunk (128 rows x 128 of its 256 columns) from registers: the two 64-column atoms 2H and 2H + 1 of one
// row (lane == row inside the 32-row group g), for the warps that feed tensor memory.
//     Regs r = HalfChunk<FMT>::load(chunk, g, lane, H)       the packed bytes, from global memory
//     HalfChunk<FMT>::atom<K>(r, H, o, grid)                 atom 2H + K: 64 bf16 as 32 packed pairs, columns in order
// H is the same in all lanes.  Values are those of DequantBlock (formats.cuh), bit for bit; Q4_K for scales below 0.5 (DequantAtomQ4KRt:
// GEMMs of matrices with larger ones do not come here).
#pragma once
#include "formats_smem.cuh"

namespace llm {

template <int F> struct HalfChunk;

// Byte k (0 or 1) of `pair` times f, without the conversion unit: the byte under the exponent of 2^23.  Exact: the product has few bits.
template <int K> LLM_DEVICE float byte_times(uint32_t pair, float f) {
    return fmaf(__uint_as_float(__byte_perm(pair, 0x4b000000u, 0x7650 + K)), f, -8388608.0f * f);
}

template <> struct HalfChunk<FMT_Q4_K> {
    using T = FmtTraits<FMT_Q4_K>;
    struct Regs { uint4 meta, q[4]; };
    LLM_DEVICE static Regs load(const uint8_t* chunk, int g, int lane, int H) {
        Regs r;
        r.meta = ldg_nc_v4(chunk + T::P_META + ((g * 32 + lane) << 4));
#pragma unroll
        for (int u = 0; u < 4; ++u) r.q[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QS, 8, g, 4 * H + u, lane));
        return r;
    }
    template <int K> LLM_DEVICE static void atom(const Regs& r, int H, uint32_t (&o)[32], const uint32_t*) {
        DequantAtomQ4KRt::Regs q;
        q.q0 = r.q[2 * K]; q.q1 = r.q[2 * K + 1];
        DequantAtomQ4KRt::scales(r.meta, 2 * H + K, q);
        DequantAtomQ4KRt::convert(q, o);
    }
};

template <> struct HalfChunk<FMT_Q5_K> {
    using T = FmtTraits<FMT_Q5_K>;
    struct Regs { uint4 meta, q[4], h[2]; };
    LLM_DEVICE static Regs load(const uint8_t* chunk, int g, int lane, int H) {
        Regs r;
        r.meta = ldg_nc_v4(chunk + T::P_META + ((g * 32 + lane) << 4));
#pragma unroll
        for (int u = 0; u < 4; ++u) r.q[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QS, 8, g, 4 * H + u, lane));
#pragma unroll
        for (int u = 0; u < 2; ++u) r.h[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QH, 2, g, u, lane));
        return r;
    }
    template <int K> LLM_DEVICE static void atom(const Regs& r, int H, uint32_t (&o)[32], const uint32_t*) {
        const float d = half_bits_to_float(r.meta.x & 0xffff), ndmin = -half_bits_to_float(r.meta.x >> 16);
        // 6-bit scales and minima of sub-blocks 2A and 2A + 1, A = 2H + K (the packing of unpack_k4_scales)
        const uint32_t a = r.meta.y >> (16 * K), b = r.meta.z >> (16 * K), c = r.meta.w >> (16 * K);
        const uint32_t sc = H == 0 ? a & 0x3f3fu : (c & 0x0f0fu) | ((a >> 2) & 0x3030u);
        const uint32_t mn = H == 0 ? b & 0x3f3fu : ((c >> 4) & 0x0f0fu) | ((b >> 2) & 0x3030u);
        const __nv_bfloat162 off = __float2bfloat162_rn(128.0f);
        const __nv_bfloat162 s_lo = __float2bfloat162_rn(byte_times<0>(sc, d)), s_hi = __float2bfloat162_rn(byte_times<1>(sc, d));
        const __nv_bfloat162 b_lo = __float2bfloat162_rn(byte_times<0>(mn, ndmin)), b_hi = __float2bfloat162_rn(byte_times<1>(mn, ndmin));
        const int sh = 4 * H + 2 * K;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const uint32_t ws[4] = {r.q[2 * K + h].x, r.q[2 * K + h].y, r.q[2 * K + h].z, r.q[2 * K + h].w};
            const uint32_t hs[4] = {r.h[h].x, r.h[h].y, r.h[h].z, r.h[h].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t t = hs[i] >> sh;
                uint32_t *lo = o + 8 * h + 2 * i, *hi = lo + 16;
                affine4((ws[i] & 0x0f0f0f0fu) | ((t << 4) & 0x10101010u), off, s_lo, b_lo, lo[0], lo[1]);
                affine4(((ws[i] >> 4) & 0x0f0f0f0fu) | ((t << 3) & 0x10101010u), off, s_hi, b_hi, hi[0], hi[1]);
            }
        }
    }
};

template <> struct HalfChunk<FMT_Q6_K> {
    using T = FmtTraits<FMT_Q6_K>;
    struct Regs { uint2 sc; uint32_t d; uint4 ql[4], qh[2]; };
    LLM_DEVICE static Regs load(const uint8_t* chunk, int g, int lane, int H) {
        const int row = g * 32 + lane;
        Regs r;
        r.sc = ldg_nc_v2(chunk + T::P_SC + (row << 4) + 8 * H);
        r.d = ldg_nc_u16(chunk + T::P_D + (row << 1));
#pragma unroll
        for (int u = 0; u < 4; ++u) r.ql[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QL, 8, g, 4 * H + u, lane));
#pragma unroll
        for (int u = 0; u < 2; ++u) r.qh[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QH, 4, g, 2 * H + u, lane));
        return r;
    }
    template <int K> LLM_DEVICE static void atom(const Regs& r, int, uint32_t (&o)[32], const uint32_t*) {
        const float d = half_bits_to_float((uint16_t)r.d);
        const __nv_bfloat162 off = __float2bfloat162_rn(160.0f), zero = __float2bfloat162_rn(0.0f);
        const uint32_t sc = K ? r.sc.y : r.sc.x;             // scales of 16 columns, in order: units 0 and 1, then 2 and 3
#pragma unroll
        for (int lh = 0; lh < 2; ++lh) {
            const __nv_bfloat162 f0 = __float2bfloat162_rn(d * static_cast<int8_t>(sc >> (8 * lh))), f1 = __float2bfloat162_rn(d * static_cast<int8_t>(sc >> (8 * lh + 16)));
            const uint32_t as[4] = {r.ql[lh].x, r.ql[lh].y, r.ql[lh].z, r.ql[lh].w}, bs[4] = {r.ql[2 + lh].x, r.ql[2 + lh].y, r.ql[2 + lh].z, r.ql[2 + lh].w};
            const uint32_t hs[4] = {r.qh[lh].x, r.qh[lh].y, r.qh[lh].z, r.qh[lh].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t qa = ((K ? as[i] >> 4 : as[i]) & 0x0f0f0f0fu) | ((K ? hs[i] : hs[i] << 4) & 0x30303030u);
                const uint32_t qb = ((K ? bs[i] >> 4 : bs[i]) & 0x0f0f0f0fu) | ((K ? hs[i] >> 2 : hs[i] << 2) & 0x30303030u);
                uint32_t *a = o + 8 * lh + 2 * i, *b = a + 16;
                affine4(qa, off, f0, zero, a[0], a[1]);
                affine4(qb, off, f1, zero, b[0], b[1]);
            }
        }
    }
};

template <> struct HalfChunk<FMT_Q8_0> {
    using T = FmtTraits<FMT_Q8_0>;
    struct Regs { uint2 d; uint4 q[8]; };
    LLM_DEVICE static Regs load(const uint8_t* chunk, int g, int lane, int H) {
        Regs r;
        r.d = ldg_nc_v2(chunk + T::P_D + ((g * 32 + lane) << 4) + 8 * H);
#pragma unroll
        for (int u = 0; u < 8; ++u) r.q[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QS, 16, g, 8 * H + u, lane));
        return r;
    }
    // byte ^ 0x80 under the exponent of 2^23 is 2^23 + 128 + value: one exact addition, one rounded product, two values at a time (the
    // conversion unit has a quarter of the additions' rate)
    template <int K> LLM_DEVICE static void atom(const Regs& r, int, uint32_t (&o)[32], const uint32_t*) {
        const uint32_t dw = K ? r.d.y : r.d.x;
        const float2 off = make_float2(-8388736.0f, -8388736.0f);
#pragma unroll
        for (int u = 0; u < 4; ++u) {
            const float d = half_bits_to_float((dw >> (16 * (u >> 1))) & 0xffff);
            const float2 dd = make_float2(d, d);
            const uint32_t ws[4] = {r.q[4 * K + u].x, r.q[4 * K + u].y, r.q[4 * K + u].z, r.q[4 * K + u].w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const uint32_t w = ws[i] ^ 0x80808080u;
                const float2 lo = __fmul2_rn(__fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7650)), __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7651))), off), dd);
                const float2 hi = __fmul2_rn(__fadd2_rn(make_float2(__uint_as_float(__byte_perm(w, 0x4b000000u, 0x7652)), __uint_as_float(__byte_perm(w, 0x4b000000u, 0x7653))), off), dd);
                o[8 * u + 2 * i] = pack_bf16(lo.x, lo.y);
                o[8 * u + 2 * i + 1] = pack_bf16(hi.x, hi.y);
            }
        }
    }
};

template <> struct HalfChunk<FMT_Q4_0> {
    using T = FmtTraits<FMT_Q4_0>;
    struct Regs { uint2 d; uint4 q[4]; };
    LLM_DEVICE static Regs load(const uint8_t* chunk, int g, int lane, int H) {
        Regs r;
        r.d = ldg_nc_v2(chunk + T::P_D + ((g * 32 + lane) << 4) + 8 * H);
#pragma unroll
        for (int u = 0; u < 4; ++u) r.q[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QS, 8, g, 4 * H + u, lane));
        return r;
    }
    template <int K> LLM_DEVICE static void atom(const Regs& r, int, uint32_t (&o)[32], const uint32_t*) {
        const __nv_bfloat162 off = __float2bfloat162_rn(136.0f), zero = __float2bfloat162_rn(0.0f);
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const __nv_bfloat162 s = __float2bfloat162_rn(half_bits_to_float(((K ? r.d.y : r.d.x) >> (16 * b)) & 0xffff));
            const uint4 q = r.q[2 * K + b];
            const uint32_t ws[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                uint32_t *lo = o + 16 * b + 2 * i, *hi = lo + 8;
                affine4(ws[i] & 0x0f0f0f0fu, off, s, zero, lo[0], lo[1]);
                affine4((ws[i] >> 4) & 0x0f0f0f0fu, off, s, zero, hi[0], hi[1]);
            }
        }
    }
};

template <> struct HalfChunk<FMT_IQ3_S> {
    using T = FmtTraits<FMT_IQ3_S>;
    struct Regs { uint32_t qh, sc, d; uint4 sg, qs[2]; };
    LLM_DEVICE static Regs load(const uint8_t* chunk, int g, int lane, int H) {
        const int row = g * 32 + lane;
        Regs r;
        r.qh = ldg_nc_u32(chunk + T::P_QH + (row << 3) + 4 * H);
        r.sc = ldg_nc_u32(chunk + T::P_SC + (row << 2));
        r.d = ldg_nc_u16(chunk + T::P_D + (row << 1));
        r.sg = ldg_nc_v4(unit_ptr(chunk + T::P_SIGNS, 2, g, H, lane));
#pragma unroll
        for (int u = 0; u < 2; ++u) r.qs[u] = ldg_nc_v4(unit_ptr(chunk + T::P_QS, 4, g, 2 * H + u, lane));
        return r;
    }
    // `grid`: the 512-entry codebook
    template <int K> LLM_DEVICE static void atom(const Regs& r, int H, uint32_t (&o)[32], const uint32_t* grid) {
        const float d = half_bits_to_float((uint16_t)r.d);
        const __nv_bfloat162 off = __float2bfloat162_rn(128.0f), zero = __float2bfloat162_rn(0.0f);
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            const int ib = 2 * K + k;                            // of this half's four blocks of 32 columns
            const uint32_t hb = (r.qh >> (8 * ib)) & 0xff, sw = ib == 0 ? r.sg.x : ib == 1 ? r.sg.y : ib == 2 ? r.sg.z : r.sg.w;
            const __nv_bfloat162 db = __float2bfloat162_rn(d * (1 + 2 * ((r.sc >> (16 * H + 4 * ib)) & 0xf)));
#pragma unroll
            for (int l = 0; l < 4; ++l) {
                const uint32_t q = k ? (l < 2 ? r.qs[K].z : r.qs[K].w) : (l < 2 ? r.qs[K].x : r.qs[K].y);
                const uint32_t pair = q >> (16 * (l & 1)), sb = (sw >> (8 * l)) & 0xff;
                uint32_t* v = o + 16 * k + 4 * l;
                affine4(grid[(pair & 0xff) | ((hb << (8 - 2 * l)) & 256)], off, db, zero, v[0], v[1]);
                affine4(grid[((pair >> 8) & 0xff) | ((hb << (7 - 2 * l)) & 256)], off, db, zero, v[2], v[3]);
                v[0] ^= ((sb & 1) << 15) | ((sb & 2) << 30);          // sign bit k of sb flips value k
                v[1] ^= ((sb & 4) << 13) | ((sb & 8) << 28);
                v[2] ^= ((sb & 16) << 11) | ((sb & 32) << 26);
                v[3] ^= ((sb & 64) << 9) | ((sb & 128) << 24);
            }
        }
    }
};

}  // namespace llm
