// The resident field kernel (olc_resident.cuh) on one 16-bit storage type.
#pragma once
#include "olc_resident.cuh"

namespace olc {

namespace {

// 16-bit elements holding values or deficits (rows are whole groups: the x
// extent is a multiple of 8 and the buffers are 16-byte aligned).
template <int ST, int EN>
struct Resident16 {
    static_assert(EN != OLC_ENC_OFFSET3, "three-offset elements have no free bit");
    typedef uint2 Raw;
    static constexpr bool GROUPS = true;
    static constexpr olc_u32 PHASE = 0x80008000u;
    static constexpr olc_u32 POLLS = OLC_SPIN_LIMIT;
    static __device__ __forceinline__ Raw load(const void* f, olc_u32 v, int, olc_u32) {
        uint2 q;
        asm volatile("ld.relaxed.gpu.global.v2.u32 {%0, %1}, [%2];"
                     : "=r"(q.x), "=r"(q.y)
                     : "l"(static_cast<const unsigned short*>(f) + v)
                     : "memory");
        return q;
    }
    static __device__ __forceinline__ void store(void* f, olc_u32 v, int, Raw q) {
        asm volatile("st.relaxed.gpu.global.v2.u32 [%0], {%1, %2};" ::"l"(static_cast<unsigned short*>(f) + v), "r"(q.x),
                     "r"(q.y)
                     : "memory");
    }
    static __device__ __forceinline__ bool ready(Raw q, olc_u32 phase) {
        return (((q.x ^ phase) | (q.y ^ phase)) & PHASE) == 0u;
    }
    static __device__ __forceinline__ float4 value(Raw q) {
        const olc_u32 x = q.x & ~PHASE, y = q.y & ~PHASE;
        return make_float4(Store16<ST>::to_f((unsigned short)(x & 0xffffu)), Store16<ST>::to_f((unsigned short)(x >> 16)),
                           Store16<ST>::to_f((unsigned short)(y & 0xffffu)), Store16<ST>::to_f((unsigned short)(y >> 16)));
    }
    // v holds values that were rounded to storage: the conversion is exact
    static __device__ __forceinline__ Raw bits(float4 v, olc_u32 phase) {
        return make_uint2(pack2<ST>(v.x, v.y) | phase, pack2<ST>(v.z, v.w) | phase);
    }
    static __device__ __forceinline__ olc_u32 load_word(const void*, olc_u32) { return 0u; }
    static __device__ __forceinline__ float word(olc_u32) { return 0.0f; }
    static constexpr bool ROUNDS = true;
    // the working value of the faces: the boundary as stored, or a deficit of 0
    static __device__ __forceinline__ float face(float bval) {
        return EN == OLC_ENC_DEFICIT ? 0.0f : Store16<ST>::to_f(Store16<ST>::from_f(bval));
    }
    // rounded to storage (voxel index vox) and back
    static __device__ __forceinline__ float4 round(float4 v, olc_u32 vox, olc_u32 key) {
        if (IsSR<ST>::value)
            return value(make_uint2(pack2_sr<ST>(v.x, v.y, olc_sr_pair(vox >> 1, key)),
                                    pack2_sr<ST>(v.z, v.w, olc_sr_pair((vox >> 1) + 1, key))));
        return value(make_uint2(pack2<ST>(v.x, v.y), pack2<ST>(v.z, v.w)));
    }
    struct Update {
        f32x2 r2, idl, idr, dsl, dsr;
        float4 lo;
        float b;
        __device__ __forceinline__ Update(const ResidentArgs& a, float bval, const bool (&f)[4]) {
            const float ds = EN == OLC_ENC_DEFICIT ? a.dec_sub : 0.0f;
            r2 = pk2(a.r, a.r);
            idl = pk2(f[0] ? 0.0f : a.inv_decay, f[1] ? 0.0f : a.inv_decay);
            idr = pk2(f[2] ? 0.0f : a.inv_decay, f[3] ? 0.0f : a.inv_decay);
            dsl = pk2(f[0] ? 0.0f : ds, f[1] ? 0.0f : ds);
            dsr = pk2(f[2] ? 0.0f : ds, f[3] ? 0.0f : ds);
            lo = make_float4(f[0] ? bval : 0.0f, f[1] ? bval : 0.0f, f[2] ? bval : 0.0f, f[3] ? bval : 0.0f);
            b = a.bval;
        }
        __device__ __forceinline__ float4 operator()(float xl, float xr, const float4& c, const float4& ym,
                                                     const float4& yp, const float4& zm, const float4& zp) const {
            const float4 v = stencil_update4h<EN>(xl, xr, c, ym, yp, zm, zp, r2, idl, idr, dsl, dsr);
            const float4 w = make_float4(fmaxf(v.x, lo.x), fmaxf(v.y, lo.y), fmaxf(v.z, lo.z), fmaxf(v.w, lo.w));
            if (EN != OLC_ENC_DEFICIT) return w;
            return make_float4(fminf(w.x, b), fminf(w.y, b), fminf(w.z, b), fminf(w.w, b));
        }
    };
};

}  // namespace

// The variants of storage type ST, instantiated in a source file of their own.  The
// device code of a source file is loaded as a whole when the first of its kernels is
// launched, and a large one is stored compressed: with all 65 variants in one file
// that took 18 ms of a process's first field step, with the 25 of FP32 or the 10 of
// a storage type alone 2.
template <int ST>
cudaError_t launch_resident16(int encoding, const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s) {
    return encoding == OLC_ENC_DEFICIT ? launch_resident<Resident16<ST, OLC_ENC_DEFICIT>>(a, p, s)
                                       : launch_resident<Resident16<ST, OLC_ENC_VALUE>>(a, p, s);
}

}  // namespace olc
