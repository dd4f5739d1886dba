// BF16 / FP16 storage of fields: conversions to and from FP32 (round to
// nearest even, or stochastic for the _SR types) and 8-element vector loads
// and stores.  Bits are handled as unsigned short.
#pragma once
#include <type_traits>

#include "olc_device.cuh"
#include "olc_stencil.cuh"
#include "../../include/olc.h"

namespace olc {

template <int ST>
struct Store16;

template <>
struct Store16<OLC_FIELD_BF16> {
    static __device__ __forceinline__ float to_f(unsigned short h) { return __uint_as_float((olc_u32)h << 16); }
    // round to nearest even on the FP32 bit pattern (values here are finite)
    static __device__ __forceinline__ unsigned short from_f(float f) {
        unsigned short h;
        asm("cvt.rn.bf16.f32 %0, %1;" : "=h"(h) : "f"(f));
        return h;
    }
};

template <>
struct Store16<OLC_FIELD_F16> {
    static __device__ __forceinline__ float to_f(unsigned short h) {
        float f;
        asm("{ .reg .b16 t; mov.b16 t, %1; cvt.f32.f16 %0, t; }" : "=f"(f) : "h"(h));
        return f;
    }
    static __device__ __forceinline__ unsigned short from_f(float f) {
        unsigned short h;
        asm("{ .reg .b16 t; cvt.rn.f16.f32 t, %1; mov.b16 %0, t; }" : "=h"(h) : "f"(f));
        return h;
    }
};

// BF16 / FP16 with stochastic rounding in the substeps: same storage
template <>
struct Store16<OLC_FIELD_BF16_SR> : Store16<OLC_FIELD_BF16> {};
template <>
struct Store16<OLC_FIELD_F16_SR> : Store16<OLC_FIELD_F16> {};

template <int ST>
struct IsSR {
    static constexpr bool value = ST == OLC_FIELD_BF16_SR || ST == OLC_FIELD_F16_SR;
};

// Stochastic BF16 rounding of a finite non-negative value with 32 random bits:
// the low 16 bits of the FP32 pattern plus 16 random bits carry into the kept
// half with probability equal to the discarded fraction.
__device__ __forceinline__ unsigned short olc_bf16_sr(float f, olc_u32 rnd) {
    return (unsigned short)((__float_as_uint(f) + (rnd & 0xffffu)) >> 16);
}


// Random bits for one substep: `key` mixes the step, substep and field
// (fmix32, once per launch); voxels 2p and 2p+1 of a grid share one 32-bit
// word x = ((p ^ key) * 0x9E3779B1) ^ (x >> 15) (a multiplicative hash with
// one xorshift), voxel 2p taking its low and voxel 2p+1 its high 16 bits.
__device__ __forceinline__ olc_u32 olc_sr_key(olc_u32 step, int sub, int field) {
    return olc_fmix32((step << 8) ^ (olc_u32)sub ^ ((olc_u32)field << 24));
}
__device__ __forceinline__ olc_u32 olc_sr_pair(unsigned long long pair, olc_u32 key) {
    olc_u32 x = ((olc_u32)pair ^ key) * 0x9E3779B1u;
    return x ^ (x >> 15);
}

// Two FP32 values -> one word of two 16-bit values (a in the low half, b in
// the high half).  cvt.*x2 converts its first source into the high half.
template <int ST>
__device__ __forceinline__ olc_u32 pack2(float a, float b) {
    olc_u32 d;
    if (ST == OLC_FIELD_BF16 || ST == OLC_FIELD_BF16_SR)
        asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
    else
        asm("cvt.rn.f16x2.f32 %0, %1, %2;" : "=r"(d) : "f"(b), "f"(a));
    return d;
}

// The same with stochastic rounding, by the conversion's random-bits form:
// the low half (a) takes bits 15..0 of rnd (BF16) or 12..0 (FP16), the high
// half (b) bits 31..16 or 28..16; a value rounds away from zero when the top
// of its discarded bits plus those random bits carries (olc_bf16_sr for BF16).
template <int ST>
__device__ __forceinline__ olc_u32 pack2_sr(float a, float b, olc_u32 rnd) {
    olc_u32 d;
    if (ST == OLC_FIELD_BF16_SR)
        asm("cvt.rs.bf16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(b), "f"(a), "r"(rnd));
    else
        asm("cvt.rs.f16x2.f32 %0, %1, %2, %3;" : "=r"(d) : "f"(b), "f"(a), "r"(rnd));
    return d;
}

// ------------------------------------------------------------------ encodings
// What a 16-bit element holds (OLC_ENC_*, olc.h).  Kernels work on the
// "working" value of an element: the deficit b - f for OLC_ENC_DEFICIT (the
// 7-point update is linear, so substeps and residuals stay in that domain),
// the field value f otherwise.  `Codec` gathers the per-encoding steps.
struct EncConst {
    float b, half_b, quarter_b, upper_q;
};

template <int ST, int EN>
struct Codec {
    // working value of one element
    static __device__ __forceinline__ float work(unsigned short h, const EncConst& k) {
        if (EN != OLC_ENC_OFFSET3) return Store16<ST>::to_f(h);
        // magnitude with the sign (bit 15) kept and bit 14 cleared, plus
        // (b/2) x (bit 15 + bit 14): codes 00 -> m, 01 -> b/2 + m,
        // 10 -> b/2 - m, 11 -> b - m
        // The offset (b/2 per set flag bit; both products and their sum are
        // exact) is formed with selects: an integer-to-float conversion runs
        // on the quarter-rate conversion pipe and bounded the substep.
        const float m = Store16<ST>::to_f((unsigned short)(h & 0xBFFFu));
        const float o15 = (h & 0x8000u) ? k.half_b : 0.0f;
        const float o14 = (h & 0x4000u) ? k.half_b : 0.0f;
        return __fadd_rn(m, __fadd_rn(o15, o14));
    }
    // field value from a working value
    static __device__ __forceinline__ float phys_of_work(float w, const EncConst& k) {
        return EN == OLC_ENC_DEFICIT ? __fsub_rn(k.b, w) : w;
    }
    static __device__ __forceinline__ float phys(unsigned short h, const EncConst& k) {
        return phys_of_work(work(h, k), k);
    }
    // OLC_ENC_OFFSET3: magnitude to round and the code bits of a value f,
    // clamped to [0, b]; every subtraction is exact (Sterbenz)
    static __device__ __forceinline__ float split3(float f, const EncConst& k, olc_u32* code) {
        f = fminf(fmaxf(f, 0.0f), k.b);
        if (f < k.quarter_b) {
            *code = 0u;
            return fabsf(f);
        }
        if (f > k.upper_q) {
            *code = 0xC000u;
            return __fsub_rn(k.b, f);
        }
        const float d = __fsub_rn(f, k.half_b);
        *code = d < 0.0f ? 0x8000u : 0x4000u;
        return fabsf(d);
    }
    // OLC_ENC_OFFSET3, two working values >= 0 (no NaN) at once.  The integer and
    // select work of split3 saturated the ALU pipe (77 % busy, the FP32 pipe 23 %),
    // so the offsets are found with multiply-adds: the signs of f - b/4 and
    // f - (b - b/4) (exact differences, so the signs are exact) saturate to 0 or 1,
    // their sum n counts the offset in units of b/2, and f - n b/2 is split3's
    // difference.  n then becomes code bits 14 (n = 1) and 15 (n = 2).
    static __device__ __forceinline__ olc_u32 pack3(float f0, float f1, const EncConst& k, bool sr, olc_u32 rnd) {
        const float huge = __uint_as_float(0x7f000000u);  // 2^127: twice, any nonzero difference exceeds 1
        const f32x2 f = pk2(fminf(f0, k.b), fminf(f1, k.b)), huge2 = pk2(huge, huge);
        const float2 lo = upk2(mul2(sub2(f, pk2(k.quarter_b, k.quarter_b)), huge2));
        const float2 hi = upk2(mul2(sub2(f, pk2(k.upper_q, k.upper_q)), huge2));
        const f32x2 n = add2(pk2(__saturatef(__fmaf_rn(lo.x, huge, 1.0f)), __saturatef(__fmaf_rn(lo.y, huge, 1.0f))),
                             pk2(__saturatef(__fmul_rn(hi.x, huge)), __saturatef(__fmul_rn(hi.y, huge))));
        const float2 d = upk2(fma2(n, pk2(-k.half_b, -k.half_b), f)), nn = upk2(n);
        const olc_u32 w = sr ? pack2_sr<ST>(d.x, d.y, rnd) : pack2<ST>(d.x, d.y);
        // n0 and n1 in the halves' bits 0..1, from the mantissa of 2^23 + n0 + 2^16 n1
        const olc_u32 m = __float_as_uint(__fadd_rn(__fmaf_rn(nn.y, 65536.0f, nn.x), 8388608.0f));
        const olc_u32 c14 = m * 0x4000u, c13 = m * 0x2000u;  // bit 14: n = 1, bit 15: n = 2; the same one bit lower
        // bit 15: the distance is negative or n = 2; bit 14: n = 2, or n = 1 and it is not negative
        const olc_u32 t = (c14 & ~(w >> 1)) | c13;
        return w | ((c14 & 0x80008000u) | (t & 0x40004000u));
    }
    // two working values, >= 0 and no NaN -> one word (a low, b high), nearest
    // or stochastic (a magnitude rounds alike under either sign)
    static __device__ __forceinline__ olc_u32 pack(float a, float b, const EncConst& k, bool sr, olc_u32 rnd) {
        if (EN != OLC_ENC_OFFSET3) return sr ? pack2_sr<ST>(a, b, rnd) : pack2<ST>(a, b);
        return pack3(a, b, k, sr, rnd);
    }
    // the working values of a word's two elements
    static __device__ __forceinline__ float2 work2(olc_u32 w, const EncConst& k) {
        if (EN != OLC_ENC_OFFSET3)
            return make_float2(Store16<ST>::to_f((unsigned short)(w & 0xffffu)), Store16<ST>::to_f((unsigned short)(w >> 16)));
        // the offset's count n = floor(2 u + 1/2), u the element's 16 bits as a
        // fraction: the high word of a 64-bit multiply-add, which adds the bits of
        // 2^23 too, so that it reads as the float 2^23 + n (the compiler makes
        // shifts and carries of it; kept a multiply by a hidden 2, a substep of
        // 256^3 took 31.1 us instead of 29.2)
        const olc_u64 half = ((olc_u64)0x4B000000u << 32) | 0x80000000u;
        const olc_u32 n0 = (olc_u32)(((olc_u64)(w << 16) * 2u + half) >> 32);
        const olc_u32 n1 = (olc_u32)(((olc_u64)w * 2u + half) >> 32);
        const olc_u32 m = w & 0xBFFFBFFFu;
        const f32x2 n = add2(pk2(__uint_as_float(n0), __uint_as_float(n1)), pk2(-8388608.0f, -8388608.0f));
        return upk2(fma2(n, pk2(k.half_b, k.half_b),
                         pk2(Store16<ST>::to_f((unsigned short)(m & 0xffffu)), Store16<ST>::to_f((unsigned short)(m >> 16)))));
    }
    // one working value -> one element, to nearest
    static __device__ __forceinline__ unsigned short enc_rn(float w, const EncConst& k) {
        if (EN != OLC_ENC_OFFSET3) return Store16<ST>::from_f(w);
        olc_u32 c;
        const float m = split3(w, k, &c);
        return (unsigned short)(Store16<ST>::from_f(m) | c);
    }
};

// Eight elements (16 bytes) to working values.
template <int ST, int EN>
__device__ __forceinline__ void load8w(const unsigned short* p, float (&f)[8], const EncConst& k) {
    const uint4 raw = *reinterpret_cast<const uint4*>(p);
    const olc_u32 w[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const float2 v = Codec<ST, EN>::work2(w[q], k);
        f[2 * q] = v.x;
        f[2 * q + 1] = v.y;
    }
}

// Eight working values stored at voxel index vi (a multiple of 8).
template <int ST, int EN>
__device__ __forceinline__ void store8w_at(unsigned short* p, const float (&v)[8], unsigned long long vi,
                                           olc_u32 key, const EncConst& k) {
    olc_u32 w[4];
#pragma unroll
    for (int q = 0; q < 4; ++q)
        w[q] = Codec<ST, EN>::pack(v[2 * q], v[2 * q + 1], k, IsSR<ST>::value,
                                   IsSR<ST>::value ? olc_sr_pair((vi >> 1) + q, key) : 0u);
    *reinterpret_cast<uint4*>(p) = make_uint4(w[0], w[1], w[2], w[3]);
}

// Four elements (8 bytes) to working values.
template <int ST, int EN>
__device__ __forceinline__ float4 load4w(const unsigned short* p, const EncConst& k) {
    const uint2 w = *reinterpret_cast<const uint2*>(p);
    const float2 a = Codec<ST, EN>::work2(w.x, k), b = Codec<ST, EN>::work2(w.y, k);
    return make_float4(a.x, a.y, b.x, b.y);
}

// Four working values stored; `pair` is half the first one's voxel index (a multiple of 4).
template <int ST, int EN>
__device__ __forceinline__ void store4w_at(unsigned short* p, const float4& v, olc_u32 pair, olc_u32 key,
                                           const EncConst& k) {
    const olc_u32 r0 = IsSR<ST>::value ? olc_sr_pair(pair, key) : 0u;
    const olc_u32 r1 = IsSR<ST>::value ? olc_sr_pair(pair + 1, key) : 0u;
    *reinterpret_cast<uint2*>(p) = make_uint2(Codec<ST, EN>::pack(v.x, v.y, k, IsSR<ST>::value, r0),
                                              Codec<ST, EN>::pack(v.z, v.w, k, IsSR<ST>::value, r1));
}

// The per-step reaction of one interior voxel (FS: a FieldStep): working value
// w = work(h) + residual; the uptake f <- f / (1 + K dt) and the step's decay
// f <- f * decay_step (round-to-nearest storages; 1 otherwise), rounded to
// nearest with the new residual kept.  For OLC_ENC_DEFICIT (w = b - f) the
// same maps are w <- (w + b K dt) / (1 + K dt), w <- w * decay_step +
// b (1 - decay_step), which leave a voxel with K = 0 and no decay unchanged.
template <int ST, int EN, class FS>
__device__ __forceinline__ void react_voxel(unsigned short& h, float& comp, float kv, const FS& fs,
                                            const EncConst& k) {
    float val = __fadd_rn(Codec<ST, EN>::work(h, k), comp);
    if (EN == OLC_ENC_DEFICIT) {
        if (kv != 0.0f) {
            const float kd = __fmul_rn(kv, fs.sink_dt);
            val = __fdiv_rn(__fadd_rn(val, __fmul_rn(k.b, kd)), __fadd_rn(1.0f, kd));
        }
        val = __fmaf_rn(val, fs.decay_step, fs.dec_step);
    } else {
        if (kv != 0.0f) val = __fdiv_rn(val, __fadd_rn(1.0f, __fmul_rn(kv, fs.sink_dt)));
        val = __fmul_rn(val, fs.decay_step);
    }
    h = Codec<ST, EN>::enc_rn(val, k);
    comp = __fsub_rn(val, Codec<ST, EN>::work(h, k));
}

// A voxel's field value with its residual (reductions, metrics).
template <int ST, int EN>
__device__ __forceinline__ float phys_with_residual(unsigned short h, float comp, const EncConst& k) {
    return Codec<ST, EN>::phys_of_work(__fadd_rn(Codec<ST, EN>::work(h, k), comp), k);
}

// Host side: calls f(storage, encoding) with both as std::integral_constant,
// for the runtime 16-bit storage type and encoding of a field.
template <class F>
inline void with_storage16(int storage, int encoding, F&& f) {
    auto by_enc = [&](auto st) {
        if (encoding == OLC_ENC_DEFICIT)
            f(st, std::integral_constant<int, OLC_ENC_DEFICIT>{});
        else if (encoding == OLC_ENC_OFFSET3)
            f(st, std::integral_constant<int, OLC_ENC_OFFSET3>{});
        else
            f(st, std::integral_constant<int, OLC_ENC_VALUE>{});
    };
    if (storage == OLC_FIELD_BF16)
        by_enc(std::integral_constant<int, OLC_FIELD_BF16>{});
    else if (storage == OLC_FIELD_BF16_SR)
        by_enc(std::integral_constant<int, OLC_FIELD_BF16_SR>{});
    else if (storage == OLC_FIELD_F16_SR)
        by_enc(std::integral_constant<int, OLC_FIELD_F16_SR>{});
    else
        by_enc(std::integral_constant<int, OLC_FIELD_F16>{});
}

// The reaction and the reductions round to nearest: a stochastic-rounding
// storage type shares its base type's kernels there.
template <int ST>
struct BaseOf {
    static constexpr int value = ST == OLC_FIELD_BF16_SR ? OLC_FIELD_BF16 : ST == OLC_FIELD_F16_SR ? OLC_FIELD_F16 : ST;
};

}  // namespace olc
