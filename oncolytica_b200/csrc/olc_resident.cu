// FP32 fields small enough to stay on chip: all the remaining substeps of a
// field step in one launch.
//
// A substep of a small field is a fraction of a microsecond of arithmetic; as
// one launch each, the launches bound it (64^3: 2.96 us per substep, 96^3: 5.2,
// and 9.7 at 117 x 75 x 131, whose rows no tensor map describes).  Here each
// CTA of a cooperative grid (one per SM) keeps a tile of full rows in shared
// memory, and the CTAs exchange only the tiles' outer rows after each substep
// (whole field steps of 79, 88 and 21 substeps: 235 -> 112 us, 452 -> 193,
// 203 -> 120).
//
// Exchange without flags, fences or barriers: a substep's results are never
// negative (the clamp), so the sign bit of a published word is free and carries
// the exchange's phase.  A CTA publishes its outer rows in one of the field's
// two buffers (exchange e in buffer e & 1) with the phase flipped at each use
// of the buffer; a reader polls a word until it carries the expected phase.
//   * Every word validates itself, so relaxed loads and stores are enough.
//   * A buffer is written again two exchanges later.  A CTA gets there only
//     after it has read exchange e+1 of all its neighbours, and each of them
//     published e+1 after it had read exchange e (its block-wide barrier).
//   * Both buffers must start with clear sign bits: the two buffers then hold
//     earlier substeps' results, so the launch follows at least two ordinary
//     substeps, which also take care of whatever the caller's faces held.
// All waits are bounded: a thread that gives up records OLC_ST_TIMEOUT and
// polls no more, so the grid always ends.
//
// Per voxel the update is stencil_update4, so the result equals the
// one-launch-per-substep kernels bit for bit.
#include "olc_internal.h"
#include "olc_stencil.cuh"

#include <algorithm>

namespace olc {

namespace {

constexpr int RING_ITEMS = 4;  // ring groups per thread, at most

struct ResidentArgs {
    float* in;      // the field: substep input, and every second exchange
    float* other;   // the other buffer: first exchange
    int nx, ny, nz;
    int G;          // groups of four voxels per row
    int By, Bz;     // rows and planes of a tile
    int ty;         // tiles along y
    int runs;       // z runs per column of a tile
    int substeps;   // >= 1
    float r, inv_decay, bval;
    olc_u32* status;
};

__device__ __forceinline__ uint4 ld_relaxed4(const float* p) {
    uint4 v;
    asm volatile("ld.relaxed.gpu.global.v4.u32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
                 : "l"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void st_relaxed4(float* p, uint4 v) {
    asm volatile("st.relaxed.gpu.global.v4.u32 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(v.x), "r"(v.y), "r"(v.z),
                 "r"(v.w)
                 : "memory");
}

// Four voxels of a row at x (x + 3 may pass the row's end: those words read as
// `fill` and are not written).
template <bool VEC>
__device__ __forceinline__ uint4 ld_group(const float* row, int x, int nx, olc_u32 fill) {
    if (VEC) return ld_relaxed4(row + x);
    const olc_u32* w = reinterpret_cast<const olc_u32*>(row + x);
    uint4 v = make_uint4(olc_ld_relaxed(w), fill, fill, fill);
    if (x + 1 < nx) v.y = olc_ld_relaxed(w + 1);
    if (x + 2 < nx) v.z = olc_ld_relaxed(w + 2);
    if (x + 3 < nx) v.w = olc_ld_relaxed(w + 3);
    return v;
}
template <bool VEC>
__device__ __forceinline__ void st_group(float* row, int x, int nx, uint4 v) {
    if (VEC) {
        st_relaxed4(row + x, v);
        return;
    }
    olc_u32* w = reinterpret_cast<olc_u32*>(row + x);
    olc_st_relaxed(w, v.x);
    if (x + 1 < nx) olc_st_relaxed(w + 1, v.y);
    if (x + 2 < nx) olc_st_relaxed(w + 2, v.z);
    if (x + 3 < nx) olc_st_relaxed(w + 3, v.w);
}

__device__ __forceinline__ float4 as_f4(uint4 v) {
    return make_float4(__uint_as_float(v.x), __uint_as_float(v.y), __uint_as_float(v.z), __uint_as_float(v.w));
}
__device__ __forceinline__ uint4 with_phase(float4 v, olc_u32 phase) {
    return make_uint4((__float_as_uint(v.x) & 0x7fffffffu) | phase, (__float_as_uint(v.y) & 0x7fffffffu) | phase,
                      (__float_as_uint(v.z) & 0x7fffffffu) | phase, (__float_as_uint(v.w) & 0x7fffffffu) | phase);
}

// One tile per CTA; a thread owns up to K consecutive planes of four voxels of
// one row, in registers, and shares them with its neighbours through shared
// memory (two copies of the tile and its ring of one row and one plane).
template <int K, int NT, bool VEC>
__global__ void __launch_bounds__(NT, 1) k_resident(const ResidentArgs a) {
    extern __shared__ __align__(16) float s_tile[];
    const int P = a.G * 4;                 // row pitch
    const int Y2 = a.By + 2;               // rows held per plane, ring included
    const int plane = Y2 * P;
    const int copy = (a.Bz + 2) * plane;
    const int y0 = (blockIdx.x % a.ty) * a.By, z0 = (blockIdx.x / a.ty) * a.Bz;
    const int rows = min(a.By, a.ny - y0), planes = min(a.Bz, a.nz - z0);
    const size_t sy = (size_t)a.nx, sz = (size_t)a.nx * a.ny;
    const int tid = threadIdx.x, lane = tid & 31;

    // this thread's column
    const int per_run = a.G * a.By;
    const int run = tid / per_run, col = tid - run * per_run;
    const int ry = col / a.G, g = col - ry * a.G;
    const int kz0 = run * K;
    const int kn = (run < a.runs && ry < rows) ? min(K, planes - kz0) : 0;  // planes owned (<= 0: none)
    const int x = 4 * g, y = y0 + ry;
    const bool y_face = y == 0 || y >= a.ny - 1;
    const int xe = a.nx - 1 - x;  // element of the row's last voxel, when within 0..3
    float4 c[K];
    const float4 b4 = make_float4(a.bval, a.bval, a.bval, a.bval);

    // the ring's groups are dealt to the threads: rows below and above the
    // tile (planes x 2), then planes below and above (rows x 2)
    const int ring_rows = 2 * planes + 2 * rows;
    const int ring_items = ring_rows * a.G;

    // A ring group is read only where it and the own voxels next to it are
    // inside the grid's faces (elsewhere bval stands in, and only face voxels
    // see it), so two tiles always read each other or neither does.
    int ring_so[RING_ITEMS], ring_gx[RING_ITEMS];  // place in shared memory (< 0: nothing to read), x
    olc_u32 ring_go[RING_ITEMS];                   // first voxel of its row in the grid
    auto interior = [&](int yy, int zz) {
        const int Y = y0 + yy, Z = z0 + zz;
        return Y > 0 && Y < a.ny - 1 && Z > 0 && Z < a.nz - 1;
    };
    auto fix_x = [&](float4 v, int gx) {
        if (gx == 0) v.x = a.bval;
        const int e = a.nx - 1 - gx;
        if (e <= 0) v.x = a.bval;
        if (e <= 1) v.y = a.bval;
        if (e <= 2) v.z = a.bval;
        if (e <= 3) v.w = a.bval;
        return v;
    };

    // own voxels and the ring of the launch's input; the ring's face groups in both copies
    const int own = (kz0 + 1) * plane + (ry + 1) * P + x;
#pragma unroll
    for (int k = 0; k < K; ++k) {
        c[k] = b4;
        if (k < kn) {
            const int z = z0 + kz0 + k;
            if (!y_face && z > 0 && z < a.nz - 1)
                c[k] = fix_x(as_f4(ld_group<VEC>(a.in + (size_t)z * sz + (size_t)y * sy, x, a.nx, 0u)), x);
            *reinterpret_cast<float4*>(s_tile + own + k * plane) = c[k];
        }
    }
#pragma unroll
    for (int t = 0; t < RING_ITEMS; ++t) {
        const int i = tid + t * NT;
        ring_so[t] = -1;
        ring_gx[t] = 0;
        ring_go[t] = 0u;
        if (i >= ring_items) continue;
        const int rr = i / a.G;
        const int gx = 4 * (i - rr * a.G);
        int yy, zz, iy, iz;
        if (rr < 2 * planes) {
            iz = zz = rr >> 1;
            yy = (rr & 1) ? rows : -1;
            iy = (rr & 1) ? rows - 1 : 0;
        } else {
            const int q = rr - 2 * planes;
            iy = yy = q >> 1;
            zz = (q & 1) ? planes : -1;
            iz = (q & 1) ? planes - 1 : 0;
        }
        const int so = (zz + 1) * plane + (yy + 1) * P + gx;
        float4 v = b4;
        if (interior(yy, zz) && interior(iy, iz)) {
            ring_so[t] = so;
            ring_gx[t] = gx;
            ring_go[t] = (olc_u32)((size_t)(z0 + zz) * sz + (size_t)(y0 + yy) * sy);
            v = fix_x(as_f4(ld_group<VEC>(a.in + ring_go[t], gx, a.nx, 0u)), gx);
        } else {
            *reinterpret_cast<float4*>(s_tile + copy + so) = b4;
        }
        *reinterpret_cast<float4*>(s_tile + so) = v;
    }
    __syncthreads();

    bool gave_up = false;
    for (int e = 0;; ++e) {
        const float* cur = s_tile + (e & 1) * copy;
        float* nxt = s_tile + ((e & 1) ^ 1) * copy;
        const bool last = e == a.substeps - 1;
        float* out = (e & 1) ? a.in : a.other;
        const olc_u32 phase = (e & 2) ? 0u : 0x80000000u;
        // ---- one substep of the own column
        float4 prev = b4;
        if (kn > 0) prev = *reinterpret_cast<const float4*>(cur + own - plane);
#pragma unroll
        for (int k = 0; k < K; ++k) {
            const float* pc = cur + own + k * plane;
            float xl = __shfl_up_sync(0xffffffffu, c[k].w, 1);
            float xr = __shfl_down_sync(0xffffffffu, c[k].x, 1);
            if (k < kn) {
                // a warp's first and last lanes: the neighbour group is another warp's
                if (lane == 0 && x > 0) xl = pc[-1];
                if (lane == 31 && xe > 3) xr = pc[4];
                const float4 ym = *reinterpret_cast<const float4*>(pc - P);
                const float4 yp = *reinterpret_cast<const float4*>(pc + P);
                float4 zp;
                if (k + 1 < K && k + 1 < kn)
                    zp = c[k + 1 < K ? k + 1 : k];
                else
                    zp = *reinterpret_cast<const float4*>(pc + plane);
                const int z = z0 + kz0 + k;
                float4 v = stencil_update4(xl, xr, c[k], ym, yp, prev, zp, a.r, a.inv_decay);
                if (y_face || z == 0 || z == a.nz - 1) {
                    v = b4;
                } else {
                    if (x == 0) v.x = a.bval;
                    if (xe <= 3) {
                        if (xe <= 0) v.x = a.bval;
                        if (xe <= 1) v.y = a.bval;
                        if (xe <= 2) v.z = a.bval;
                        v.w = a.bval;
                    }
                }
                if (last) {
                    float* row = out + (size_t)z * sz + (size_t)y * sy;
                    st_group<VEC>(row, x, a.nx, make_uint4(__float_as_uint(v.x), __float_as_uint(v.y),
                                                           __float_as_uint(v.z), __float_as_uint(v.w)));
                } else {
                    *reinterpret_cast<float4*>(nxt + own + k * plane) = v;
                    if (ry == 0 || ry == rows - 1 || kz0 + k == 0 || kz0 + k == planes - 1)
                        st_group<VEC>(out + (size_t)z * sz + (size_t)y * sy, x, a.nx, with_phase(v, phase));
                }
                prev = c[k];
                c[k] = v;
            }
        }
        if (last) return;
        // ---- the neighbours' outer rows
        uint4 w[RING_ITEMS];
#pragma unroll
        for (int t = 0; t < RING_ITEMS; ++t)
            if (ring_so[t] >= 0) w[t] = ld_group<VEC>(out + ring_go[t], ring_gx[t], a.nx, phase);
#pragma unroll
        for (int t = 0; t < RING_ITEMS; ++t) {
            if (ring_so[t] < 0) continue;
            olc_u32 spins = 0;
            while (!gave_up &&
                   (((w[t].x ^ phase) | (w[t].y ^ phase) | (w[t].z ^ phase) | (w[t].w ^ phase)) & 0x80000000u)) {
                if (++spins > OLC_SPIN_LIMIT) {
                    atomicOr(a.status, OLC_ST_TIMEOUT);
                    gave_up = true;
                }
                w[t] = ld_group<VEC>(out + ring_go[t], ring_gx[t], a.nx, phase);
            }
            const uint4 v = make_uint4(w[t].x & 0x7fffffffu, w[t].y & 0x7fffffffu, w[t].z & 0x7fffffffu,
                                       w[t].w & 0x7fffffffu);
            *reinterpret_cast<float4*>(nxt + ring_so[t]) = fix_x(as_f4(v), ring_gx[t]);
        }
        __syncthreads();
    }
}

struct ResidentPlan {
    int By = 0, Bz = 0, ty = 0, tz = 0, K = 0, NT = 0, runs = 0;
    size_t smem = 0;
};

int device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

constexpr size_t RES_SMEM_MAX = 225 * 1024;

// Tile of the field's rows and planes: at most one tile per SM, the least
// arithmetic and exchange per tile (a ring row costs about as much as two
// rows of arithmetic: it is published, polled and staged).
bool make_resident_plan(const int dims[3], int sms, ResidentPlan* best) {
    const int nx = dims[0], ny = dims[1], nz = dims[2];
    const int G = (nx + 3) / 4;
    double best_cost = 1e30;
    for (int By = 1; By <= ny; ++By) {
        const int ty = (ny + By - 1) / By;
        if (ty > sms) continue;
        const int tz_max = sms / ty;
        const int Bz = (nz + tz_max - 1) / tz_max;
        const int tz = (nz + Bz - 1) / Bz;
        const size_t smem = 2 * (size_t)(By + 2) * (Bz + 2) * G * 16;
        if (smem > RES_SMEM_MAX) continue;
        const int cols = G * By;
        for (int K = 1; K <= 8; K *= 2) {
            const int runs = (Bz + K - 1) / K;
            const int threads = cols * runs;
            if (threads > 512) continue;
            const int nt = threads <= 256 ? 256 : 512;
            if (2 * (By + Bz) * G > RING_ITEMS * nt) continue;
            const double cost = By * Bz + 4.0 * (By + Bz) + 0.5 * K;
            if (cost < best_cost) {
                best_cost = cost;
                best->By = By;
                best->Bz = Bz;
                best->ty = ty;
                best->tz = tz;
                best->K = K;
                best->runs = runs;
                best->NT = nt;
                best->smem = smem;
            }
            break;  // fewer planes per thread fill the SM better
        }
    }
    return best_cost < 1e30;
}

template <int K, int NT, bool VEC>
cudaError_t launch_resident(const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s) {
    static int configured_mask = 0;  // per device (up to 32)
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 32 && !(configured_mask & (1 << dev))) {
        cudaFuncSetAttribute(k_resident<K, NT, VEC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)RES_SMEM_MAX);
        configured_mask |= 1 << dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(p.ty * p.tz);
    cfg.blockDim = dim3(NT);
    cfg.dynamicSmemBytes = p.smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_resident<K, NT, VEC>, a);
}

template <bool VEC>
cudaError_t launch_resident_k(const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s) {
#define OLC_RES_CASE(k, nt) \
    if (p.K == k && p.NT == nt) return launch_resident<k, nt, VEC>(a, p, s);
    OLC_RES_CASE(1, 256)
    OLC_RES_CASE(1, 512)
    OLC_RES_CASE(2, 256)
    OLC_RES_CASE(2, 512)
    OLC_RES_CASE(4, 256)
    OLC_RES_CASE(4, 512)
    OLC_RES_CASE(8, 256)
    OLC_RES_CASE(8, 512)
#undef OLC_RES_CASE
    return cudaErrorInvalidValue;
}

}  // namespace

// Whether a field's substeps are worth the resident launch.
bool resident_fits(const FieldStep& fs) {
    if (fs.substeps < RESIDENT_LEAD + 4) return false;
    ResidentPlan p;
    return make_resident_plan(fs.dims, device_sms(), &p);
}

// `substeps` substeps from `in` (both buffers hold substep results: clear sign
// bits); returns the buffer holding the result, or null when the launch was
// not possible.
float* run_resident(float* in, float* other, const FieldStep& fs, int substeps, olc_u32* status, cudaStream_t s) {
    ResidentPlan p;
    if (substeps < 1 || !make_resident_plan(fs.dims, device_sms(), &p)) return nullptr;
    ResidentArgs a;
    a.in = in;
    a.other = other;
    a.nx = fs.dims[0];
    a.ny = fs.dims[1];
    a.nz = fs.dims[2];
    a.G = (a.nx + 3) / 4;
    a.By = p.By;
    a.Bz = p.Bz;
    a.ty = p.ty;
    a.runs = p.runs;
    a.substeps = substeps;
    a.r = fs.r;
    a.inv_decay = fs.inv_decay;
    a.bval = fs.bval;
    a.status = status;
    const bool vec = (a.nx & 3) == 0 && ((reinterpret_cast<uintptr_t>(in) | reinterpret_cast<uintptr_t>(other)) & 15u) == 0;
    const cudaError_t e = vec ? launch_resident_k<true>(a, p, s) : launch_resident_k<false>(a, p, s);
    if (e != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    return (substeps & 1) ? other : in;
}

}  // namespace olc
