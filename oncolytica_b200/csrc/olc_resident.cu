// The resident field kernel (olc_resident.cuh): its plans, its FP32 variants and the
// entries that launch it.
#include "olc_resident.cuh"

#include <algorithm>
#include <cmath>

namespace olc {

namespace {

// FP32 elements.  VEC: rows of whole, 16-byte aligned groups; else a row's last
// group may pass its end (those words read as `fill` and are not written).
template <bool VEC>
struct ResidentF32 {
    typedef uint4 Raw;
    static constexpr bool GROUPS = VEC;  // the ring is read by groups (else by words)
    static __device__ __forceinline__ Raw load(const void* f, olc_u32 v, int left, olc_u32 fill) {
        const olc_u32* w = static_cast<const olc_u32*>(f) + v;
        uint4 q = make_uint4(0u, fill, fill, fill);
        if (VEC) {
            asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                         : "=r"(q.x), "=r"(q.y), "=r"(q.z), "=r"(q.w)
                         : "l"(w)
                         : "memory");
            return q;
        }
        q.x = olc_ld_relaxed(w);
        if (left > 1) q.y = olc_ld_relaxed(w + 1);
        if (left > 2) q.z = olc_ld_relaxed(w + 2);
        if (left > 3) q.w = olc_ld_relaxed(w + 3);
        return q;
    }
    static __device__ __forceinline__ void store(void* f, olc_u32 v, int left, Raw q) {
        olc_u32* w = static_cast<olc_u32*>(f) + v;
        if (VEC) {
            asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(w), "r"(q.x), "r"(q.y), "r"(q.z),
                         "r"(q.w)
                         : "memory");
            return;
        }
        olc_st_relaxed(w, q.x);
        if (left > 1) olc_st_relaxed(w + 1, q.y);
        if (left > 2) olc_st_relaxed(w + 2, q.z);
        if (left > 3) olc_st_relaxed(w + 3, q.w);
    }
    static constexpr olc_u32 PHASE = 0x80000000u;
    static constexpr olc_u32 POLLS = OLC_SPIN_LIMIT;  // of one exchange; an argument cost 64^3 3 % of its time
    static __device__ __forceinline__ olc_u32 load_word(const void* f, olc_u32 v) {
        return olc_ld_relaxed(static_cast<const olc_u32*>(f) + v);
    }
    static __device__ __forceinline__ float word(olc_u32 w) { return __uint_as_float(w & 0x7fffffffu); }
    static constexpr bool ROUNDS = false;
    static __device__ __forceinline__ float face(float bval) { return bval; }
    static __device__ __forceinline__ float4 round(float4 v, olc_u32, olc_u32) { return v; }
    struct Update {
        f32x2 r2, idl, idr, nz2;
        float4 lo;
        // f[e]: voxel e is a face (or lies beyond the row): a factor 0 and a
        // lower bound bval in the clamp that every voxel has
        __device__ __forceinline__ Update(const ResidentArgs& a, float bval, const bool (&f)[4]) {
            r2 = pk2(a.r, a.r);
            nz2 = pk2(a.neg_zero, a.neg_zero);
            idl = pk2(f[0] ? 0.0f : a.inv_decay, f[1] ? 0.0f : a.inv_decay);
            idr = pk2(f[2] ? 0.0f : a.inv_decay, f[3] ? 0.0f : a.inv_decay);
            lo = make_float4(f[0] ? bval : 0.0f, f[1] ? bval : 0.0f, f[2] ? bval : 0.0f, f[3] ? bval : 0.0f);
        }
        __device__ __forceinline__ float4 operator()(float xl, float xr, const float4& c, const float4& ym,
                                                     const float4& yp, const float4& zm, const float4& zp) const {
            const float4 v = stencil_update4u(xl, xr, c, ym, yp, zm, zp, r2, idl, idr, nz2);
            return make_float4(fmaxf(v.x, lo.x), fmaxf(v.y, lo.y), fmaxf(v.z, lo.z), fmaxf(v.w, lo.w));
        }
    };
    static __device__ __forceinline__ bool ready(Raw q, olc_u32 phase) {
        return (((q.x ^ phase) | (q.y ^ phase) | (q.z ^ phase) | (q.w ^ phase)) & PHASE) == 0u;
    }
    static __device__ __forceinline__ float4 value(Raw q) {
        return make_float4(__uint_as_float(q.x & 0x7fffffffu), __uint_as_float(q.y & 0x7fffffffu),
                           __uint_as_float(q.z & 0x7fffffffu), __uint_as_float(q.w & 0x7fffffffu));
    }
    static __device__ __forceinline__ Raw bits(float4 v, olc_u32 phase) {
        return make_uint4(__float_as_uint(v.x) | phase, __float_as_uint(v.y) | phase, __float_as_uint(v.z) | phase,
                          __float_as_uint(v.w) | phase);
    }
};

int device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

// Tile of the field's rows and planes: at most one tile per SM, the least
// arithmetic and exchange per tile (a ring row costs about as much as two
// rows of arithmetic: it is published, polled and staged).
bool make_resident_plan(const int dims[3], bool groups, ResidentPlan* best) {
    const int nx = dims[0], ny = dims[1], nz = dims[2], sms = device_sms();
    const int G = (nx + 3) / 4;
    double best_cost = 1e30;
    // at most one tile per SM along y, and 512 groups in a tile's plane
    for (int By = (ny + sms - 1) / sms; By <= std::min(ny, 512 / G); ++By) {
        const int ty = (ny + By - 1) / By;
        const int tz_max = sms / ty;
        const int Bz = (nz + tz_max - 1) / tz_max;
        const int tz = (nz + Bz - 1) / Bz;
        const int cols = G * By;
        for (int K = 1; K <= 8; K *= 2) {
            const int runs = (Bz + K - 1) / K;
            const int threads = cols * runs;
            if (threads > 512) continue;
            const int nt = K == 1 && threads <= 256 ? 256 : 512;
            // ring groups per thread, or 128-word chunks of ring rows per warp
            const int ring = 2 * (By + Bz) * (groups ? G : (nx + 127) / 128), takers = groups ? nt : nt / 32;
            if (ring > RING_ITEMS * takers) continue;
            // the last run's loop reads past the tile where it has fewer planes
            const int L = (Bz + runs - 1) / runs;
            const size_t smem = (size_t)(By + 2) * (2 * (Bz + 2) + runs * L - Bz) * G * 16;
            if (smem > RES_SMEM_MAX) continue;
            const double cost = By * Bz + 4.0 * (By + Bz) + 0.5 * K;
            if (cost < best_cost) {
                best_cost = cost;
                best->By = By;
                best->Bz = Bz;
                best->ty = ty;
                best->tz = tz;
                best->K = K;
                best->runs = runs;
                best->L = L;
                best->NT = nt;
                best->RI = ring <= takers ? 1 : RING_ITEMS;
                best->smem = smem;
            }
            break;  // fewer planes per thread fill the SM better
        }
    }
    return best_cost < 1e30;
}

// Whether a field's substeps are worth the resident launch.  Six are the fewest it has
// been measured at, and it is faster there: us in passes and here 64^3 22.0 and 15.2,
// 96^3 26.9 and 19.0, 128^3 33.9 and 27.3, 33 x 35 x 47 (no tensor maps) 49.4 and 26.9.
bool resident_fits(const FieldStep& fs) {
    // faces get their value as the clamp's lower bound, which needs bval >= +0
    if (fs.substeps < RESIDENT_LEAD + 4 || !(fs.bval >= 0.0f) || std::signbit(fs.bval)) return false;
    ResidentPlan p;
    return make_resident_plan(fs.dims, (fs.dims[0] & 3) == 0, &p);
}

void fill_resident_args(ResidentArgs* a, void* in, void* other, const FieldStep& fs, const ResidentPlan& p, int substeps,
                        olc_u32* status) {
    *a = ResidentArgs{};
    a->in = in;
    a->other = other;
    a->nx = fs.dims[0];
    a->ny = fs.dims[1];
    a->nz = fs.dims[2];
    a->G = (a->nx + 3) / 4;
    a->By = p.By;
    a->Bz = p.Bz;
    a->ty = p.ty;
    a->runs = p.runs;
    a->L = p.L;
    a->substeps = substeps;
    a->r = fs.r;
    a->inv_decay = fs.inv_decay;
    a->bval = fs.bval;
    a->neg_zero = -0.0f;
    a->status = status;
    a->dec_sub = fs.dec_sub;
}

// `substeps` substeps from `in` (both buffers hold substep results: clear sign
// bits); returns the buffer holding the result, or null when the launch was
// not possible.
float* run_resident(float* in, float* other, const FieldStep& fs, int substeps, olc_u32* status, cudaStream_t s) {
    const bool vec =
        (fs.dims[0] & 3) == 0 && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(other)) & 15u) == 0;
    ResidentPlan p;
    if (substeps < 1 || !make_resident_plan(fs.dims, vec, &p)) return nullptr;
    ResidentArgs a;
    fill_resident_args(&a, in, other, fs, p, substeps, status);
    const cudaError_t e = vec ? launch_resident<ResidentF32<true>>(a, p, s) : launch_resident<ResidentF32<false>>(a, p, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return (substeps & 1) ? other : in;
}

// A 16-bit substep is shorter in passes and longer here than an FP32 one.  From a
// million voxels on, where they fill the passes' tiles (at least four fifths), the
// launch's fixed cost, about 10 us, is made up only at 10 substeps.  us in passes and
// here, 6, 8 and 10 substeps: 128^3 30.2 and 33.2, 37.5 and 38.2, 48.5 and 45.4;
// 256 x 64 x 64 24.8 and 29.0, 32.1 and 33.1, 38.3 and 37.2.  Else 6 are enough: 96^3
// 24.9 and 22.9, 64^3 24.7 and 18.8, 64 x 24 x 900 (tiles three quarters full) 28.1
// and 27.9.
bool resident_fits16(const FieldStep& fs) {
    auto tiles = [&](int axis, int size) { return (long long)((fs.dims[axis] + size - 1) / size) * size; };
    const long long voxels = (long long)fs.dims[0] * fs.dims[1] * fs.dims[2];
    const bool late = voxels >= 1000000 &&
                      5 * voxels >= 4 * tiles(0, BATCH_T16_TX) * tiles(1, BATCH_T16_TY) * tiles(2, BATCH_T16_TZ);
    return fs.encoding != OLC_ENC_OFFSET3 && fs.substeps >= (late ? 10 : 0) && resident_fits(fs);
}

// olc_resident16.cuh, a source file per storage type
template <int ST>
cudaError_t launch_resident16(int encoding, const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s);

// run_resident for 16-bit storage: substeps sub0 .. sub0 + substeps - 1.
void* run_resident16(void* in, void* other, const FieldStep& fs, int substeps, olc_u32* status, const olc_u32* step_ctr,
                     olc_u32 step_host, int sub0, int field, cudaStream_t s) {
    ResidentPlan p;
    if (substeps < 1 || fs.encoding == OLC_ENC_OFFSET3 || !make_resident_plan(fs.dims, true, &p))
        return nullptr;
    ResidentArgs a;
    fill_resident_args(&a, in, other, fs, p, substeps, status);
    a.step_ctr = step_ctr;
    a.step_host = step_host;
    a.sub0 = sub0;
    a.field = field;
    const cudaError_t e = fs.storage == OLC_FIELD_BF16      ? launch_resident16<OLC_FIELD_BF16>(fs.encoding, a, p, s)
                          : fs.storage == OLC_FIELD_F16     ? launch_resident16<OLC_FIELD_F16>(fs.encoding, a, p, s)
                          : fs.storage == OLC_FIELD_BF16_SR ? launch_resident16<OLC_FIELD_BF16_SR>(fs.encoding, a, p, s)
                                                            : launch_resident16<OLC_FIELD_F16_SR>(fs.encoding, a, p, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return (substeps & 1) ? other : in;
}

}  // namespace olc

// A field of two tiles of which only the first is launched: its exchange with the
// second waits for words that nobody publishes, gives up and reports it.
namespace {
constexpr int SELFTEST_DIMS[3] = {16, 8, 4};
__device__ __align__(16) float g_selftest_field[2][16 * 8 * 4];
}  // namespace

namespace olc {
namespace {
struct ResidentSelftest : ResidentF32<true> {
    static constexpr olc_u32 POLLS = 1000;
};
}  // namespace
}  // namespace olc

extern "C" int olc_selftest_exchange_wait(void* stream) {
    using namespace olc;
    cudaStream_t st = reinterpret_cast<cudaStream_t>(stream);
    void* buf = nullptr;
    olc_u32* status = stage_status_word();
    cudaError_t e = cudaGetSymbolAddress(&buf, g_selftest_field);
    if (e != cudaSuccess || !status) return cuda_status(cudaErrorSymbolNotFound, "olc_selftest_exchange_wait");
    e = cudaMemsetAsync(buf, 0, sizeof(g_selftest_field), st);
    if (e != cudaSuccess) return cuda_status(e, "olc_selftest_exchange_wait: clear");
    FieldStep fs = {};
    for (int i = 0; i < 3; ++i) fs.dims[i] = SELFTEST_DIMS[i];
    fs.r = 0.1f;
    fs.inv_decay = 1.0f;
    ResidentPlan p;
    p.By = p.Bz = p.runs = 4;
    p.ty = 2;
    p.tz = p.K = p.RI = p.L = 1;
    p.NT = 256;
    p.smem = (size_t)(p.By + 2) * 2 * (p.Bz + 2) * (SELFTEST_DIMS[0] / 4) * 16;
    ResidentArgs a;
    float* f = static_cast<float*>(buf);
    fill_resident_args(&a, f, f + sizeof(g_selftest_field) / 8, fs, p, 3, status);
    p.ty = 1;  // the launch's share of them
    return cuda_status(launch_resident_t<1, 256, 1, false, ResidentSelftest>(a, p, st), "olc_selftest_exchange_wait");
}
