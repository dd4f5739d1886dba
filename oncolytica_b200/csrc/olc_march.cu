// Two substeps of a large FP32 field per pass over memory.
//
// A one-substep pass over 256^3 voxels runs at the copy rate (20.7 us for 134
// MB), so only fewer passes make it faster.  Here a CTA marches along z over a
// tile of rows: input planes arrive by TMA in a ring of shared-memory slots,
// and each step computes one plane of the intermediate field and one plane of
// results from it.  A lane holds four consecutive x voxels of R rows of two
// intermediate planes in registers; what bounds the pass is the L1 data pipe,
// instruction issue and the FP32 pipe (74, 57 and 47 % busy, 18.1 M warp instructions
// per pass on 256^3 against 21.3 M for two one-substep passes), so:
//   * R = 4 rows per lane: a row's y neighbours are the lane's own registers,
//     but for the group's outer rows, which go through shared memory (one
//     barrier per step, which also frees the oldest input slot).  Recomputing
//     them instead cost 16 % more row updates and more registers.
//   * The rows' x neighbours come from the neighbour lanes.  At the ends of a
//     tile, the intermediate column just outside is computed by lanes of the
//     same warp, one voxel per row.
//   * Face voxels cost nothing: a factor 0 and a lower bound bval in the clamp
//     that every voxel has (hence bval >= 0).  Tiles along y and chunks along z
//     are laid over the interior; their face rows are fixed up in a branch that
//     only the outermost groups take.
//   * Two copies of the step per loop and no more: a larger body missed the
//     instruction cache (2.1 stalls per instruction with six copies).
// Measured (us per substep, before -> after): 256^3 20.9 -> 15.6, 192^3 9.1 ->
// 7.6, 128^3 5.2 -> 3.8 (a size that stays on chip unless pairs are asked for),
// 100 x 100 x 256 6.1 -> 4.8.
// Alternate passes march in opposite directions, so a pass starts on the planes
// that the previous one wrote last, while they are in L2.
#include "olc_internal.h"
#include "olc_stencil.cuh"

#include <algorithm>
#include <cmath>
#include <type_traits>

namespace olc {

namespace {

constexpr int MARCH_R = 4;  // rows per lane

// LX lanes per row, R rows per lane, W warps per CTA on adjacent rows.
template <int LX, int R, int W>
struct MarchShape {
    static constexpr int SLOTS = W == 8 ? 5 : 4;    // ring slots (planes): three in use, the rest in flight
    static constexpr int GRP = 32 / LX;             // row groups per warp
    static constexpr int UNITS = W * GRP;
    static constexpr int TX = 4 * LX;               // columns
    static constexpr int TYM = UNITS * R;           // intermediate rows (output rows: all but the outer two)
    static constexpr int WX = TX + 8, WY = TYM + 2;  // TMA box of one plane
    static constexpr unsigned BYTES = WX * WY * 4;
    static constexpr unsigned SLOT = (BYTES + 127) / 128 * 128;
    static constexpr unsigned EXCH = 2 * UNITS * 2 * TX * 4;  // groups' outer intermediate rows, two planes
    static constexpr unsigned SMEM = SLOTS * (SLOT + 8) + EXCH + 128;
};

struct MarchArgs {
    float* out;
    int nx, ny, nz;
    int zl;      // output planes per CTA
    int down;    // march towards smaller z
    float r, inv_decay, bval;
    float neg_zero;  // -0.0f, where the compiler does not see it (stencil_update4x)
    olc_u32* status;
};

__device__ __forceinline__ olc_u32 march_smem(const void* p) { return static_cast<olc_u32>(__cvta_generic_to_shared(p)); }

// EDGE: several tiles along x (a row's end lanes then need the column outside).
template <int LX, int R, int W, bool EDGE>
__global__ void __launch_bounds__(32 * W, 16 / W) k_march2(const __grid_constant__ CUtensorMap in_map,
                                                                        const MarchArgs a) {
    using S = MarchShape<LX, R, W>;
    extern __shared__ unsigned char march_raw[];
    const olc_u32 pad = (128u - (march_smem(march_raw) & 127u)) & 127u;
    unsigned char* ring = march_raw + pad;
    float* exch = reinterpret_cast<float*>(ring + S::SLOTS * S::SLOT);
    const olc_u32 ring_a = march_smem(ring);
    const olc_u32 full0 = ring_a + S::SLOTS * S::SLOT + S::EXCH;
    asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
    if (threadIdx.x == 0) {
        for (int k = 0; k < S::SLOTS; ++k)
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(full0 + 8 * k) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    __syncthreads();
    asm volatile("griddepcontrol.wait;" ::: "memory");

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int gl = lane / LX, lx = lane - gl * LX;
    const int unit = warp * S::GRP + gl;
    // the last tile along y ends at the last row; rows that two tiles share get
    // the same values from both
    const int x0 = blockIdx.y * S::TX, cy0 = min((int)blockIdx.x * (S::TYM - 2), a.ny - S::TYM);
    const int z0 = 1 + blockIdx.z * a.zl, z1 = min(z0 + a.zl, a.nz - 1);
    // plane q of the march is input plane first + dir * q
    const int dir = a.down ? -1 : 1;
    const int first = a.down ? z1 + 1 : z0 - 2;
    const int nq = z1 - z0 + 4;
    // planes first + dir and first + dir (nq - 2) are the intermediate field's
    // first and last; either may be a face of the grid
    const int zi0 = first + dir, zi1 = first + dir * (nq - 2);
    const bool face0 = zi0 == 0 || zi0 == a.nz - 1, face1 = zi1 == 0 || zi1 == a.nz - 1;
    // Steps below this one compute their intermediate plane.  Planes below it are
    // loaded, and every one of them is waited for: the block's shared memory goes
    // to another block when it ends.
    const int n_full = face1 ? nq - 1 : nq;
    auto issue = [&](int q, int slot) {
        const olc_u32 bar = full0 + 8 * slot;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(S::BYTES) : "memory");
        asm volatile(
            "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes "
            "[%0], [%1, {%2, %3, %4}], [%5];" ::"r"(ring_a + slot * S::SLOT),
            "l"(reinterpret_cast<unsigned long long>(&in_map)), "r"(x0 - 4), "r"(cy0 - 1), "r"(first + dir * q),
            "r"(bar)
            : "memory");
    };
    if (threadIdx.x == 0)
        for (int q = 0; q < S::SLOTS && q < n_full; ++q) issue(q, q);

    const int x = x0 + 4 * lx;
    const int yr = cy0 + unit * R;  // the group's first row
    const bool lane_l = lx == 0, lane_r = lx == LX - 1;
    const bool top = yr == 0, bottom = yr + R == a.ny, in_x = x < a.nx;
    // the tile's outer rows are no results (where they are faces, the face block writes them)
    const bool put0 = in_x && unit > 0, putR = in_x && unit < S::UNITS - 1;
    const olc_u32 szv = (olc_u32)a.nx * (olc_u32)a.ny;
    const int row0 = unit * R * S::WX + 4 + 4 * lx;  // this lane's four voxels of the input row above the group's first
    // one column outside each end of the tile that is no face.  eoff: the input
    // column there; lanes 0..GRP*R-1 compute the left intermediate column, lanes
    // 16..16+GRP*R-1 the right one
    const int eoff = unit * R * S::WX + (lx == 0 ? 3 : S::TX + 4);
    const int xq = min(lane & 15, S::GRP * R - 1);
    const int xoff = (warp * S::GRP * R + xq + 1) * S::WX + ((lane & 16) ? S::TX + 4 : 3);
    const int xy = cy0 + warp * S::GRP * R + xq;
    const bool x_face = xy == 0 || xy == a.ny - 1;
    const int xsrc = (lx == 0 ? 0 : 16) + gl * R;
    const float bval = a.bval;
    const float4 b4 = make_float4(bval, bval, bval, bval);
    // Face voxels of a row (x = 0, x = nx - 1): their factor is 0 and their lower
    // bound bval >= 0, so the clamp that every voxel has gives bval, whatever
    // the update made of them; the others keep inv_decay and 0.
    const f32x2 r2 = pk2(a.r, a.r), nz2 = pk2(a.neg_zero, a.neg_zero);
    const bool ex0 = x == 0, ex3 = x + 3 == a.nx - 1;
    const f32x2 idl = pk2(ex0 ? 0.0f : a.inv_decay, a.inv_decay), idr = pk2(a.inv_decay, ex3 ? 0.0f : a.inv_decay);
    const float lo_l = ex0 ? bval : 0.0f, lo_r = ex3 ? bval : 0.0f;
    auto v4 = [](const float* p) { return *reinterpret_cast<const float4*>(p); };

    // the z faces next to this chunk
    if (in_x) {
        for (int f = 0; f < 2; ++f) {
            if (f ? z1 != a.nz - 1 : z0 != 1) continue;
            float* o = a.out + ((f ? (olc_u32)(a.nz - 1) * szv : 0u) + (olc_u32)yr * (olc_u32)a.nx + (olc_u32)x);
            for (int m = 0; m < R; ++m) *reinterpret_cast<float4*>(o + (size_t)m * a.nx) = b4;
        }
    }

    float4 M0[R], M1[R];  // own rows of two consecutive intermediate planes, by turns the older one
    float X0 = 0.0f, X1 = 0.0f;  // the extra column of those planes
#pragma unroll
    for (int m = 0; m < R; ++m) M0[m] = M1[m] = b4;
    // this group's outer rows in the exchange, and the neighbours' (the tile's
    // outermost groups read their own: their outer rows are no results)
    float* ex_own = exch + unit * 2 * S::TX + 4 * lx;
    const int ex_up = unit > 0 ? -S::TX : 0, ex_dn = unit < S::UNITS - 1 ? 2 * S::TX : S::TX;
    constexpr int EXP = S::UNITS * 2 * S::TX;  // floats per plane of the exchange
    olc_u32 ov = (olc_u32)first * szv + (olc_u32)yr * (olc_u32)a.nx + (olc_u32)x;  // first voxel of output plane q - 2
    const olc_u32 ostep = a.down ? 0u - szv : szv;
    const bool face_rows = top || bottom;

    // One step: plane q of the input has arrived; intermediate plane q - 1 from
    // planes q - 2 .. q (ZF: it is the far z face, and plane q is not read), output
    // plane q - 2 from mz, mc and it; it replaces mz.
    auto step = [&](auto zface, auto odd, int q, float4 (&mz)[R], const float4 (&mc)[R], float& xmz, const float xmc) {
        constexpr bool ZF = decltype(zface)::value;
        constexpr bool ODD = decltype(odd)::value;  // parity of q
        const float *pp = reinterpret_cast<const float*>(ring + (q % S::SLOTS) * S::SLOT),
                    *pc = reinterpret_cast<const float*>(ring + ((q + S::SLOTS - 1) % S::SLOTS) * S::SLOT),
                    *pm = reinterpret_cast<const float*>(ring + ((q + S::SLOTS - 2) % S::SLOTS) * S::SLOT);
        const bool put = q >= 4;
        const float* ex_in = ex_own + (ODD ? 0 : EXP);
        float* ex_out = ex_own + (ODD ? EXP : 0);
        float4 up = v4(ex_in + ex_up);  // intermediate row above the group, plane q - 2
        const float4 dn = v4(ex_in + ex_dn);
        float4 cp = v4(pc + row0), cc = v4(pc + row0 + S::WX);
#pragma unroll
        for (int m = 0; m < R; ++m) {
            const float4 cn = v4(pc + row0 + (m + 2) * S::WX);
            float xl = __shfl_up_sync(0xffffffffu, cc.w, 1, LX);
            float xr = __shfl_down_sync(0xffffffffu, cc.x, 1, LX);
            if (EDGE) {
                const float e = pc[eoff + (m + 1) * S::WX];
                xl = lane_l ? e : xl;
                xr = lane_r ? e : xr;
            }
            float4 v = ZF ? b4
                          : stencil_update4f(xl, xr, cc, cp, cn, v4(pm + row0 + (m + 1) * S::WX),
                                             v4(pp + row0 + (m + 1) * S::WX), r2, idl, idr, lo_l, lo_r, nz2);
            if (m == 0) *reinterpret_cast<float4*>(ex_out) = v;
            if (m == R - 1) *reinterpret_cast<float4*>(ex_out + S::TX) = v;
            cp = cc;
            cc = cn;
            float yl = __shfl_up_sync(0xffffffffu, mc[m].w, 1, LX);
            float yh = __shfl_down_sync(0xffffffffu, mc[m].x, 1, LX);
            if (EDGE) {
                const float e = __shfl_sync(0xffffffffu, xmc, xsrc + m);
                yl = lane_l ? e : yl;
                yh = lane_r ? e : yh;
            }
            const float4 w = stencil_update4f(yl, yh, mc[m], up, m == R - 1 ? dn : mc[m < R - 1 ? m + 1 : 0], mz[m], v, r2,
                                              idl, idr, lo_l, lo_r, nz2);
            up = mc[m];
            if (put && (m == 0 ? put0 : m == R - 1 ? putR : in_x))
                *reinterpret_cast<float4*>(a.out + (ov + (olc_u32)m * (olc_u32)a.nx)) = w;
            mz[m] = v;
        }
        if (face_rows) {
            asm volatile("");  // a branch of its own, rarely taken
            if (top) {
                mz[0] = b4;
                *reinterpret_cast<float4*>(ex_out) = b4;
                if (put && in_x) *reinterpret_cast<float4*>(a.out + ov) = b4;
            }
            if (bottom) {
                mz[R - 1] = b4;
                *reinterpret_cast<float4*>(ex_out + S::TX) = b4;
                if (put && in_x) *reinterpret_cast<float4*>(a.out + (ov + (olc_u32)(R - 1) * (olc_u32)a.nx)) = b4;
            }
        }
        ov += ostep;
        if (EDGE && !ZF) {  // no step follows the one of the far z face
            const float v = stencil_update(pc[xoff - 1], pc[xoff + 1], pc[xoff - S::WX], pc[xoff + S::WX], pm[xoff],
                                           pp[xoff], pc[xoff], a.r, a.inv_decay);
            xmz = x_face ? bval : v;
        }
    };

    auto wait_plane = [&](int q) {
        return olc_mbar_wait_bounded(full0 + 8 * (q % S::SLOTS), (olc_u32)((q / S::SLOTS) & 1), a.status);
    };
    // every warp is done with plane q - 2 and its outer rows are in the exchange:
    // the plane's slot is refilled; false when a plane never arrived
    auto end_step = [&](int q, bool ok) {
        if (__syncthreads_or(!ok)) return false;
        if (threadIdx.x == 0 && q - 2 + S::SLOTS < n_full) {
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            issue(q - 2 + S::SLOTS, (q - 2) % S::SLOTS);
        }
        return true;
    };
    bool ok = wait_plane(0) && wait_plane(1);
    int q = 2;
#pragma unroll 1
    for (; q < n_full; q += 2) {
        ok = ok && wait_plane(q);
        step(std::false_type{}, std::false_type{}, q, M0, M1, X0, X1);
        if (face0 && q == 2) {
            *reinterpret_cast<float4*>(ex_own) = b4;
            *reinterpret_cast<float4*>(ex_own + S::TX) = b4;
#pragma unroll
            for (int m = 0; m < R; ++m) M0[m] = b4;
            X0 = bval;
        }
        ok = end_step(q, ok);
        if (!ok || q + 1 >= n_full) break;
        ok = wait_plane(q + 1);
        step(std::false_type{}, std::true_type{}, q + 1, M1, M0, X1, X0);
        ok = end_step(q + 1, ok);
        if (!ok) break;
    }
    if (ok && face1) {  // the last step, next to the far z face
        if (n_full & 1)
            step(std::true_type{}, std::true_type{}, n_full, M1, M0, X1, X0);
        else
            step(std::true_type{}, std::false_type{}, n_full, M0, M1, X0, X1);
    }
    // a plane never arrived: let the copies in flight land before the block ends
    if (!ok && threadIdx.x == 0)
        for (int k = 0; k < 2 * S::SLOTS; ++k)
            olc_mbar_wait_bounded(full0 + 8 * (k % S::SLOTS), (olc_u32)((k / S::SLOTS) & 1), a.status, 1u << 16);
}

template <int LX, int R, int W, bool EDGE>
void launch_march_t(const CUtensorMap& map, const MarchArgs& a, dim3 grid, cudaStream_t s) {
    using S = MarchShape<LX, R, W>;
    static int configured_mask = 0;  // per device (up to 32)
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 32 && !(configured_mask & (1 << dev))) {
        cudaFuncSetAttribute(k_march2<LX, R, W, EDGE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)S::SMEM);
        configured_mask |= 1 << dev;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(32 * W);
    cfg.dynamicSmemBytes = S::SMEM;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, k_march2<LX, R, W, EDGE>, map, a);
}


int sm_count() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

// From a million voxels on, a pass's fixed cost (its launch and first planes) is
// below what it saves: 112^3 5.7 -> 3.8 us per substep, 300 x 300 x 40 6.2 ->
// 5.6.  Smaller fields mostly stay on chip (olc_resident.cu), which is faster.
bool march_pays(const int dims[3]) { return (long long)dims[0] * dims[1] * dims[2] >= 1000000; }

// The march of a field (lx 0: it does not apply) and the TMA box of one plane.
// Lanes per row and warps per CTA are those with the least row updates per CTA
// slot, idle columns, shared rows and the chunks' extra planes included.
bool make_march_plan(const int dims[3], float bval, int planes, MarchPlan* p, cuuint32_t box[3]) {
    p->lx = 0;
    // faces get their value as the clamp's lower bound, which needs bval >= +0
    if (dims[0] % 4 != 0 || dims[2] < 8 || !(bval >= 0.0f) || std::signbit(bval)) return false;
    if ((double)dims[0] * dims[1] * dims[2] >= 4294967296.0) return false;  // 32-bit voxel indices
    const int slots_sm = sm_count();
    double best = 1e30;
    for (int lx = 32; lx >= 16; lx /= 2) {
        for (int w = 8; w >= 4; w /= 2) {
            const int TX = 4 * lx, TYM = 32 / lx * MARCH_R * w;
            if (dims[1] < TYM) continue;
            MarchPlan c;
            c.lx = lx;
            c.w = w;
            c.gx = (dims[1] - 2 + TYM - 3) / (TYM - 2);
            c.gy = (dims[0] + TX - 1) / TX;
            if (c.gy > 65535) continue;  // the grid's limit; single passes have the columns in grid x
            const int nz = dims[2] - 2;  // interior planes
            const int resident = slots_sm * (16 / w);
            const int chunks = std::max(1, std::min(resident / (c.gx * c.gy), nz / 2));
            c.zl = planes > 0 ? std::min(planes, nz) : (nz + chunks - 1) / chunks;
            c.gz = (nz + c.zl - 1) / c.zl;
            const int waves = (c.gx * c.gy * c.gz + resident - 1) / resident;
            const double cost = (double)waves * (c.zl + 3) * w;
            if (cost < best) {
                best = cost;
                *p = c;
                box[0] = TX + 8;
                box[1] = TYM + 2;
                box[2] = 1;
            }
        }
    }
    return p->lx != 0;
}

void launch_march(const MarchPlan& p, const CUtensorMap& map, float* out, const FieldStep& fs, olc_u32* status, int down,
                  cudaStream_t s) {
    MarchArgs a;
    a.out = out;
    a.nx = fs.dims[0];
    a.ny = fs.dims[1];
    a.nz = fs.dims[2];
    a.zl = p.zl;
    a.down = down;
    a.r = fs.r;
    a.inv_decay = fs.inv_decay;
    a.bval = fs.bval;
    a.neg_zero = -0.0f;
    a.status = status;
    const dim3 grid(p.gx, p.gy, p.gz);
#define OLC_MARCH_CASE(L, W)                                                  \
    if (p.lx == L && p.w == W) {                                              \
        if (p.gy > 1) launch_march_t<L, MARCH_R, W, true>(map, a, grid, s);   \
        else launch_march_t<L, MARCH_R, W, false>(map, a, grid, s);           \
    }
    OLC_MARCH_CASE(32, 8)
    OLC_MARCH_CASE(32, 4)
    OLC_MARCH_CASE(16, 8)
    OLC_MARCH_CASE(16, 4)
#undef OLC_MARCH_CASE
}

}  // namespace olc
