// Fields small enough to stay on chip: all the remaining substeps of a
// field step in one launch.
//
// A substep of a small field is a fraction of a microsecond of arithmetic; as
// one launch each, the launches bound it (64^3: 2.96 us per substep, 96^3: 5.2,
// and 9.7 at 117 x 75 x 131, whose rows no tensor map describes).  Here each
// CTA of a cooperative grid (one per SM) keeps a tile of full rows in shared
// memory, and the CTAs exchange only the tiles' outer rows after each substep
// (whole field steps of 79, 88 and 21 substeps: 232 -> 97 us, 451 -> 170,
// 216 -> 100).
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
// Per voxel the update, and the rounding of 16-bit storage, are those of the
// one-launch-per-substep kernels, so the results equal theirs bit for bit.
// 16-bit fields keep FP32 working values on chip: each is decoded once per
// substep instead of at each of its neighbours (3.25 times).  Their exchange
// needs the element's sign bit too, which values and deficits leave clear;
// three-offset elements use all their bits and are left to single passes.
#pragma once
#include "olc_internal.h"
#include "olc_stencil.cuh"
#include "olc_store16.cuh"

namespace olc {

constexpr int RING_ITEMS = 4;  // ring groups per thread, or row chunks of 128 words per warp, at most

struct ResidentArgs {
    void* in;       // the field: substep input, and every second exchange
    void* other;    // the other buffer: first exchange
    int nx, ny, nz;
    int G;          // groups of four voxels per row
    int By, Bz;     // rows and planes of a tile
    int ty;         // tiles along y
    int runs, L;    // z runs per column of a tile, planes per run
    int substeps;   // >= 1
    float r, inv_decay;
    float bval;     // the boundary value
    float neg_zero;  // -0.0f, where the compiler does not see it (stencil_update4f)
    olc_u32* status;
    // 16-bit storage: the deficits' decay term, and what salts
    // the stochastic rounding (the step from step_ctr, else step_host)
    float dec_sub;
    const olc_u32* step_ctr;
    olc_u32 step_host;
    int sub0, field;
};

struct ResidentPlan {
    int By = 0, Bz = 0, ty = 0, tz = 0, K = 0, NT = 0, RI = 0, runs = 0, L = 0;
    size_t smem = 0;
};

constexpr size_t RES_SMEM_MAX = 225 * 1024;

bool make_resident_plan(const int dims[3], bool groups, ResidentPlan* best);
void fill_resident_args(ResidentArgs* a, void* in, void* other, const FieldStep& fs, const ResidentPlan& p, int substeps,
                        olc_u32* status);

namespace {

__device__ __forceinline__ float4 lds4(olc_u32 p) {
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "r"(p)
                 : "memory");
    return v;
}
__device__ __forceinline__ void sts4(olc_u32 p, float4 v) {
    asm volatile("st.shared.v4.f32 [%0], {%1, %2, %3, %4};" ::"r"(p), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// One tile per CTA; a thread owns up to K consecutive planes of four voxels of
// one row, in registers, and shares them with its neighbours through shared
// memory (two copies of the tile and its ring of one row and one plane).  The same
// words are reached by plain accesses and by the asm ones above, whose "memory"
// clobbers keep the compiler from reordering the two.  What
// bounds it is latency (the exchange: a substep of 8^3 takes 0.65 us) and, on larger tiles,
// instruction issue: the threads' addresses, faces and publications are worked
// out once, before the substeps.
template <int K, int NT, int RI, bool WRAP, class E>
__global__ void __launch_bounds__(NT, 1) k_resident(const ResidentArgs a) {
    extern __shared__ __align__(16) float s_tile[];
    const int P = a.G * 4;                 // row pitch
    const int plane = (a.By + 2) * P;
    const int copy = (a.Bz + 2) * plane;
    const int y0 = (blockIdx.x % a.ty) * a.By, z0 = (blockIdx.x / a.ty) * a.Bz;
    const int rows = min(a.By, a.ny - y0), planes = min(a.Bz, a.nz - z0);
    const olc_u32 sy = (olc_u32)a.nx, sz = (olc_u32)a.nx * (olc_u32)a.ny;
    const int tid = threadIdx.x, lane = tid & 31;
    const float bval = E::face(a.bval);  // what the faces hold
    const float4 b4 = make_float4(bval, bval, bval, bval);

    // this thread's column of the tile; threads without one work on some other
    // column's place and keep nothing
    const int per_run = a.G * a.By;
    const int run = min(tid / per_run, a.runs - 1), col = tid % per_run;
    const int ry = col / a.G, g = col - ry * a.G;
    const int kz0 = run * a.L;
    const int x = 4 * g, y = y0 + ry, left = a.nx - x;
    const bool has = tid < per_run * a.runs && ry < rows;
    const int kn = min(a.L, planes - kz0);  // planes of the run (the last run may have fewer, or none)
    const int own = (kz0 + 1) * plane + (ry + 1) * P + x;
    const olc_u32 vox = (olc_u32)(z0 + kz0) * sz + (olc_u32)y * sy + (olc_u32)x;
    // bit k: plane k is computed here; is published after each substep
    olc_u32 work = 0, publish = 0;
    for (int k = 0; k < kn; ++k) {
        const int z = z0 + kz0 + k;
        const bool inner = has && y > 0 && y < a.ny - 1 && z > 0 && z < a.nz - 1;
        work |= inner ? 1u << k : 0u;
        publish |= inner && (ry == 0 || ry == rows - 1 || kz0 + k == 0 || kz0 + k == planes - 1) ? 1u << k : 0u;
    }
    const bool face[4] = {x == 0 || left <= 1, left <= 2, left <= 3, left <= 4};  // x faces, and beyond the row's end
    const typename E::Update update(a, bval, face);
    // WRAP: rows go on in the next warp; its first and last lanes read their x
    // neighbours from shared memory
    const olc_u32 need_l = WRAP && lane == 0 && x > 0, need_r = WRAP && lane == 31 && left > 4;
    const olc_u32 own_a = static_cast<olc_u32>(__cvta_generic_to_shared(s_tile + own));
    const olc_u32 row_b = 4u * (olc_u32)P, plane_b = 4u * (olc_u32)plane;
    const bool busy = __any_sync(0xffffffffu, work != 0u) != 0;

    float4 c[K];
#pragma unroll
    for (int k = 0; k < K; ++k) {
        c[k] = b4;
        if (k < kn && has) {
            if (work >> k & 1u) c[k] = E::value(E::load(a.in, vox + (olc_u32)k * sz, left, 0u));
            *reinterpret_cast<float4*>(s_tile + own + k * plane) = c[k];
            *reinterpret_cast<float4*>(s_tile + copy + own + k * plane) = c[k];
        }
    }
    // The ring: rows below and above the tile (planes x 2), then planes below and
    // above (rows x 2).  A ring row is read only where it and the own row next to
    // it are inside the grid's faces (elsewhere bval stands in, and only face
    // voxels see it), so two tiles always read each other or neither does.
    const int ring_rows = 2 * planes + 2 * rows;
    auto ring_row = [&](int rr, int& so, olc_u32& go) {
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
        so = (zz + 1) * plane + (yy + 1) * P;
        const int Y = y0 + yy, Z = z0 + zz;
        go = (olc_u32)Z * sz + (olc_u32)Y * sy;
        iy += y0;
        iz += z0;
        return Y > 0 && Y < a.ny - 1 && Z > 0 && Z < a.nz - 1 && iy > 0 && iy < a.ny - 1 && iz > 0 && iz < a.nz - 1;
    };
    // by groups: dealt to the threads once; by words: a row per warp
    int ring_so[RI];        // place in shared memory
    olc_u32 ring_go[RI];    // voxel
    olc_u32 ring_mask = 0;  // bit t: item t is read (by words: bit 4 t + j its word 32 j)
    if (E::GROUPS) {
#pragma unroll
        for (int t = 0; t < RI; ++t) {
            const int i = tid + t * NT;
            ring_so[t] = 0;
            ring_go[t] = 0u;
            if (i >= ring_rows * a.G) continue;
            const int rr = i / a.G;
            const int gx = 4 * (i - rr * a.G);
            int so;
            olc_u32 go;
            float4 v = b4;
            const bool read = ring_row(rr, so, go);
            so += gx;
            if (read) {
                ring_mask |= 1u << t;
                ring_so[t] = so;
                ring_go[t] = go + (olc_u32)gx;
                v = E::value(E::load(a.in, ring_go[t], 4, 0u));
            } else {
                *reinterpret_cast<float4*>(s_tile + copy + so) = b4;
            }
            *reinterpret_cast<float4*>(s_tile + so) = v;
        }
    } else {
        for (int rr = tid >> 5; rr < ring_rows; rr += NT / 32) {
            int so;
            olc_u32 go;
            const bool read = ring_row(rr, so, go);
            for (int xx = lane; xx < P; xx += 32) {
                s_tile[so + xx] = read && xx < a.nx ? E::word(E::load_word(a.in, go + (olc_u32)xx)) : bval;
                s_tile[copy + so + xx] = bval;
            }
        }
        const int chunks = (a.nx + 127) / 128;  // of 128 words
#pragma unroll
        for (int t = 0; t < RI; ++t) {
            const int i = (tid >> 5) + t * (NT / 32), rr = i / chunks;
            ring_so[t] = 0;
            ring_go[t] = 0u;
            if (i >= ring_rows * chunks || !ring_row(rr, ring_so[t], ring_go[t])) continue;
            const int xx = lane + 128 * (i - rr * chunks);
            ring_so[t] += xx;
            ring_go[t] += (olc_u32)xx;
            for (int j = 0; j < 4; ++j) ring_mask |= xx + 32 * j < a.nx ? 1u << (4 * t + j) : 0u;
        }
    }
    __syncthreads();

    const olc_u32 step = E::ROUNDS ? (a.step_ctr ? *a.step_ctr : a.step_host) : 0u;
    bool gave_up = false;
    olc_u32 spins = 0;
    for (int e = 0;; ++e) {
        const int from = (e & 1) * copy, to = copy - from;
        const bool last = e == a.substeps - 1;
        void* out = (e & 1) ? a.in : a.other;
        const olc_u32 phase = (e & 2) ? 0u : E::PHASE;
        const olc_u32 publish_now = last ? 0u : publish;
        const olc_u32 key = E::ROUNDS ? olc_sr_key(step, a.sub0 + e, a.field) : 0u;
        spins = 0;
        // ---- one substep of the own column
        if (busy) {
            olc_u32 pc = own_a + 4u * (olc_u32)from;  // the plane's own group, and the groups around it
            olc_u32 pm = pc - row_b, pp = pc + row_b, pz = pc + plane_b, pn = own_a + 4u * (olc_u32)to;
            olc_u32 vo = vox;
            float4 prev = lds4(pc - plane_b);
#pragma unroll
            for (int k = 0; k < K; ++k) {
                if (k >= a.L) break;  // the same for every thread: lanes of one warp may belong to different runs
                float xl = __shfl_up_sync(0xffffffffu, c[k].w, 1);
                float xr = __shfl_down_sync(0xffffffffu, c[k].x, 1);
                if (WRAP) {
                    asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; @p ld.shared.f32 %0, [%1 + -4]; }"
                                 : "+f"(xl) : "r"(pc), "r"(need_l) : "memory");
                    asm volatile("{ .reg .pred p; setp.ne.u32 p, %2, 0; @p ld.shared.f32 %0, [%1 + 16]; }"
                                 : "+f"(xr) : "r"(pc), "r"(need_r) : "memory");
                }
                float4 v = update(xl, xr, c[k], lds4(pm), lds4(pp), prev, lds4(pz));
                if (E::ROUNDS) v = E::round(v, vo, key);
                prev = c[k];
                if (work >> k & 1u) {
                    c[k] = v;
                    sts4(pn, v);
                }
                if (publish_now >> k & 1u) E::store(out, vo, left, E::bits(v, phase));
                pc += plane_b;
                pm += plane_b;
                pp += plane_b;
                pz += plane_b;
                pn += plane_b;
                vo += sz;
            }
        }
        if (last) {
#pragma unroll
            for (int k = 0; k < K; ++k)
                if (k < kn && has) E::store(out, vox + (olc_u32)k * sz, left, E::bits(c[k], 0u));
            return;
        }
        // ---- the neighbours' outer rows.  Few polls are in flight at a time: the
        // tiles still computing would wait behind them.
        auto wait_more = [&]() {
            if (gave_up) return false;
            if (++spins <= E::POLLS) return true;
            atomicOr(a.status, OLC_ST_TIMEOUT);
            gave_up = true;
            return false;
        };
        if (E::GROUPS) {
            typename E::Raw w[RI];
#pragma unroll
            for (int t = 0; t < RI; ++t)
                if (ring_mask >> t & 1u) w[t] = E::load(out, ring_go[t], 4, phase);
#pragma unroll
            for (int t = 0; t < RI; ++t) {
                if (!(ring_mask >> t & 1u)) continue;
                while (!E::ready(w[t], phase) && wait_more()) w[t] = E::load(out, ring_go[t], 4, phase);
                *reinterpret_cast<float4*>(s_tile + to + ring_so[t]) = E::value(w[t]);
            }
        } else {
            olc_u32 w[4 * RI];
            olc_u32 missing = ring_mask;
            while (missing) {
#pragma unroll
                for (int t = 0; t < 4 * RI; ++t)
                    if (missing >> t & 1u) w[t] = E::load_word(out, ring_go[t >> 2] + 32u * (t & 3));
                const bool more = wait_more();
#pragma unroll
                for (int t = 0; t < 4 * RI; ++t) {
                    if (!(missing >> t & 1u) || (more && ((w[t] ^ phase) & E::PHASE))) continue;
                    missing &= ~(1u << t);
                    s_tile[to + ring_so[t >> 2] + 32 * (t & 3)] = E::word(w[t]);
                }
            }
        }
        __syncthreads();
    }
}

template <int K, int NT, int RI, bool WRAP, class E>
cudaError_t launch_resident_t(const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s) {
    static int configured_mask = 0;  // per device (up to 32)
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev < 32 && !(configured_mask & (1 << dev))) {
        cudaFuncSetAttribute(k_resident<K, NT, RI, WRAP, E>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                             (int)RES_SMEM_MAX);
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
    return cudaLaunchKernelEx(&cfg, k_resident<K, NT, RI, WRAP, E>, a);
}

template <int K, int NT, class E>
cudaError_t launch_resident_k(const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s) {
    // one variant serves rows read by words, and 16-bit storage
    if (!E::GROUPS || E::ROUNDS) return launch_resident_t<K, NT, RING_ITEMS, true, E>(a, p, s);
    const bool wrap = a.G > 32 || (32 % a.G) != 0;
    if (p.RI == 1)
        return wrap ? launch_resident_t<K, NT, 1, true, E>(a, p, s) : launch_resident_t<K, NT, 1, false, E>(a, p, s);
    return wrap ? launch_resident_t<K, NT, RING_ITEMS, true, E>(a, p, s)
                : launch_resident_t<K, NT, RING_ITEMS, false, E>(a, p, s);
}

template <class E>
cudaError_t launch_resident(const ResidentArgs& a, const ResidentPlan& p, cudaStream_t s) {
    if (p.NT == 256) return launch_resident_k<1, 256, E>(a, p, s);
    if (p.K == 1) return launch_resident_k<1, 512, E>(a, p, s);
    if (p.K == 2) return launch_resident_k<2, 512, E>(a, p, s);
    if (p.K == 4) return launch_resident_k<4, 512, E>(a, p, s);
    return launch_resident_k<8, 512, E>(a, p, s);
}

}  // namespace

}  // namespace olc
