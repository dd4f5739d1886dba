// The two contact walks of the solo and the batched kernels: one thread per agent
// (contact_force_thread) and one warp per eight (contact_force_warp).  Both first
// list the candidates near enough and then compute the force law for the listed
// ones with all lanes busy.  Of ~90 candidates ~15 touch; with one of 32 lanes
// nearly always among them, a walk that computes the law where it finds a pair
// spends its square roots and division (about 80 instructions) on every candidate.
#pragma once
#include "olc_device.cuh"
#include "olc_internal.h"

namespace olc {

// One listed candidate: the pair law of k_contact, its part of the force or 0.
// Where a test of it fails, the roots and the quotient are taken of 1 (no lane
// leaves, and none takes their slow paths for the agent itself).
__device__ __forceinline__ float3 contact_pair(const float4& p, const float4& q, olc_u32 i, olc_u32 j,
                                               float stiffness) {
    const float ddx = __fsub_rn(p.x, q.x);
    const float ddy = __fsub_rn(p.y, q.y);
    const float ddz = __fsub_rn(p.z, q.z);
    const float d2 = __fadd_rn(__fadd_rn(__fmul_rn(ddx, ddx), __fmul_rn(ddy, ddy)), __fmul_rn(ddz, ddz));
    const float rsum = __fadd_rn(p.w, q.w);
    const bool in = j != i && !(q.w < 0.0f) && !(d2 > __fmul_rn(__fmul_rn(rsum, rsum), 1.00000095367431640625f));
    const float dist = sqrtf(in ? d2 : 1.0f);
    const bool touch = in && dist < rsum;
    const float ov = touch ? __fsub_rn(rsum, dist) : 1.0f;
    const float f = __fmul_rn(__fmul_rn(stiffness, ov), sqrtf(ov));
    const bool apart = touch && !(dist < 1e-5f);
    const float sc = __fdiv_rn(f, apart ? dist : 1.0f);
    return make_float3(apart ? __fmul_rn(ddx, sc) : touch ? (i < j ? -f : f) : 0.0f, apart ? __fmul_rn(ddy, sc) : 0.0f,
                       apart ? __fmul_rn(ddz, sc) : 0.0f);
}

// Whether contact_pair could find more than nothing: false only where one of its
// distance tests fails (also for NaN).  The products are fused here, so the limit
// has a margin: 2^-18 of itself against roundings, 1e-30 against underflow.
__device__ __forceinline__ bool contact_near(const float4& p, const float4& q) {
    const float ddx = __fsub_rn(p.x, q.x), ddy = __fsub_rn(p.y, q.y), ddz = __fsub_rn(p.z, q.z);
    const float d2 = __fmaf_rn(ddz, ddz, __fmaf_rn(ddy, ddy, __fmul_rn(ddx, ddx)));
    const float rsum = __fadd_rn(p.w, q.w);
    return d2 <= __fmaf_rn(__fmul_rn(rsum, rsum), 1.0000038146972656f, 1e-30f);
}


// The rows of a bin; none outside the grid.
__device__ __forceinline__ uint2 contact_rows(const uint2* __restrict__ ranges, const int* tdims, int cx, int cy, int cz) {
    if ((unsigned)cx >= (unsigned)tdims[0] || (unsigned)cy >= (unsigned)tdims[1] || (unsigned)cz >= (unsigned)tdims[2])
        return make_uint2(0u, 0u);
    return __ldg(ranges + olc_tissue_key(cx, cy, cz));
}

__device__ __forceinline__ int3 contact_bin(const float4& p, float tvs, const int* tdims) {
    return make_int3(olc_bin_coord(p.x, tvs, tdims[0]), olc_bin_coord(p.y, tvs, tdims[1]),
                     olc_bin_coord(p.z, tvs, tdims[2]));
}

// The move of agent i under force f (as k_contact), clamped into lo .. hi.
__device__ __forceinline__ void contact_move(const float4& p, const float3& f, olc_u32 i, const ContactDev& c,
                                             const float* lo, const float* hi, float* __restrict__ xo,
                                             float* __restrict__ yo, float* __restrict__ zo) {
    const float md = __fmul_rn(c.mobility, c.dt);
    float mx = __fmul_rn(f.x, md), my = __fmul_rn(f.y, md), mz = __fmul_rn(f.z, md);
    const float len = sqrtf(__fadd_rn(__fadd_rn(__fmul_rn(mx, mx), __fmul_rn(my, my)), __fmul_rn(mz, mz)));
    if (len > c.max_disp) {
        const float sc = __fdiv_rn(c.max_disp, len);
        mx = __fmul_rn(mx, sc);
        my = __fmul_rn(my, sc);
        mz = __fmul_rn(mz, sc);
    }
    xo[i] = fminf(fmaxf(__fadd_rn(p.x, mx), lo[0]), hi[0]);
    yo[i] = fminf(fmaxf(__fadd_rn(p.y, my), lo[1]), hi[1]);
    zo[i] = fminf(fmaxf(__fadd_rn(p.z, mz), lo[2]), hi[2]);
}

// A run: rows x .. y of the candidates (the last one included).  Two bins of
// adjacent keys hold one run, so the three bins of a line along x hold at most two.
constexpr int CONTACT_RUNS = 18;

// The force on agent i, record p (active: it has one), from the rows of its 27
// Moore bins: x fastest, then y, then z, rows ascending, added in that order.
// c is its bin in the grid tdims, `ranges` the grid's table.  Every lane of the warp
// calls it.
//
// A thread lists its runs, walks their rows two at a time (four loads in flight)
// and lists the near rows; when a lane's list may overflow, and at the end, the
// warp computes the listed pairs together.  Bound by the L1 data pipe (70 % busy:
// the records of ~10 bins per load) and the latency behind it; every byte of shared
// memory per thread costs threads and L1.  1 M agents: 273 us, with 27 runs per
// thread 306, with two-row loads of 32 bytes 323, computing the law in the walk 347.
template <int NT, int HITS>
__device__ __forceinline__ float3 contact_force_thread(const float4* __restrict__ posr, olc_u32 n, const float4& p,
                                                       olc_u32 i, bool active, const int3& c, float stiffness,
                                                       const uint2* __restrict__ ranges, const int* tdims,
                                                       uint2 (*s_runs)[NT], olc_u32 (*s_hits)[NT]) {
    const int t = threadIdx.x;
    float3 f = make_float3(0.0f, 0.0f, 0.0f);
    auto add = [&](const float3& v) {
        f.x = __fadd_rn(f.x, v.x);
        f.y = __fadd_rn(f.y, v.y);
        f.z = __fadd_rn(f.z, v.z);
    };
    int nb = 0;
    if (active) {
        // per-axis key terms of the neighbour coordinates (olc_tissue_axis)
        olc_u32 kx[3], ky[3], kz[3];
        bool vx[3], vy[3], vz[3];
#pragma unroll
        for (int d = 0; d < 3; ++d) {
            kx[d] = olc_tissue_axis(c.x + d - 1, 0);
            ky[d] = olc_tissue_axis(c.y + d - 1, 1);
            kz[d] = olc_tissue_axis(c.z + d - 1, 2);
            vx[d] = (unsigned)(c.x + d - 1) < (unsigned)tdims[0];
            vy[d] = (unsigned)(c.y + d - 1) < (unsigned)tdims[1];
            vz[d] = (unsigned)(c.z + d - 1) < (unsigned)tdims[2];
        }
        olc_u32 last = 0xffffffffu, first = 0;
#pragma unroll
        for (int dz = 0; dz < 3; ++dz) {
            uint2 rg[9];
#pragma unroll
            for (int e = 0; e < 9; ++e) {
                rg[e] = make_uint2(0u, 0u);
                if (vz[dz] && vy[e / 3] && vx[e % 3]) rg[e] = __ldg(ranges + (kx[e % 3] | ky[e / 3] | kz[dz]));
            }
#pragma unroll
            for (int e = 0; e < 9; ++e) {
                if (rg[e].y > rg[e].x) {
                    if (rg[e].x != last) {
                        first = rg[e].x;
                        ++nb;
                    }
                    last = rg[e].y;
                    if (nb <= CONTACT_RUNS) s_runs[nb - 1][t] = make_uint2(first, last - 1);
                }
            }
        }
        if (nb > CONTACT_RUNS) {  // a table whose bins do not follow one another by key
            for (int e = 0; e < 27; ++e) {
                const uint2 rg =
                    contact_rows(ranges, tdims, c.x + e % 3 - 1, c.y + e / 3 % 3 - 1, c.z + e / 9 - 1);
                for (olc_u32 j = rg.x; j < rg.y; ++j) add(contact_pair(p, __ldg(posr + j), i, j, stiffness));
            }
            nb = 0;
        }
    }
    olc_u32* const hits = &s_hits[0][t];
    olc_u32* hp = hits;
    auto drain = [&]() {
        for (const olc_u32* h = hits; h < hp; h += NT) {
            const olc_u32 j = *h;
            add(contact_pair(p, __ldg(posr + j), i, j, stiffness));
        }
        hp = hits;
        __syncwarp();
    };
    // A lane that has no rows (left) reads its last one again, from a place that is
    // near nothing.
    const uint2* rp = &s_runs[0][t];
    const uint2* const rend = rp + nb * NT;
    olc_u32 j = min(i, n - 1), e1 = j;
    float px = __int_as_float(0x7fffffff);
    if (nb > 0) {
        const uint2 r = *rp;
        j = r.x;
        e1 = r.y;
        px = p.x;
    }
    while (__any_sync(0xffffffffu, rp < rend)) {
        // four rows: j and j + 1 (the second only if it is in the run), twice
        olc_u32 jj[2];
        bool two[2];
        float pv[2];
        float4 q[4];
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            jj[u] = j;
            two[u] = j < e1;
            pv[u] = px;
            q[2 * u] = __ldg(posr + j);
            q[2 * u + 1] = __ldg(posr + min(j + 1, e1));
            j += 2;
            if (j > e1) {
                rp += NT;
                j = e1;
                px = __int_as_float(0x7fffffff);
                if (rp < rend) {
                    const uint2 r = *rp;
                    j = r.x;
                    e1 = r.y;
                    px = p.x;
                }
            }
        }
#pragma unroll
        for (int u = 0; u < 2; ++u) {
            const float4 pu = make_float4(pv[u], p.y, p.z, p.w);
            *hp = jj[u];
            if (contact_near(pu, q[2 * u])) hp += NT;
            *hp = jj[u] + 1;
            if (contact_near(pu, q[2 * u + 1]) && two[u]) hp += NT;
        }
        if (__any_sync(0xffffffffu, hp > hits + (HITS - 5) * NT)) drain();
    }
    drain();
    return f;
}

// What a warp of contact_force_warp keeps in shared memory: AG agents, a chunk of candidate
// rows, and listed pairs (row, agent), which their parts of the force replace.
constexpr int CONTACT_CHUNK = 128;
template <int AG, int CAP>
struct ContactWarp {
    float4 p[AG];
    olc_u32 row[CONTACT_CHUNK];
    uint2 hit[CAP];
    float fz[CAP];
};

// The force on agents base .. base + AG - 1 (lane a has agent base + a: its record
// p, a bin coordinate c and whether it is `active`), each from the rows of its 27
// Moore bins: x fastest, then y, then z, rows ascending, added in that order.  The
// sum for agent a returns in lane a.  `ranges` and tdims as above.
//
// The agents of one bin (2 to 3 of the eight) share its candidates: lanes look up
// the 27 bins, spread their rows over the lanes and test 32 at a time against each
// agent.  The listed pairs of all eight are computed 32 at a time, and three lanes
// per agent add them up in order.  A warp's chain of loads is short, so a small
// population, too few threads to hide latency, takes 13 us where one thread per
// agent takes 25 (10,000 agents; 37 computing the law in the walk), but it needs
// twice the instructions per agent: 375 us against 273 for 1 M.
template <int AG, int CAP>
__device__ __forceinline__ float3 contact_force_warp(const float4* __restrict__ posr, olc_u32 base, const float4& p,
                                                const int3& c, bool active, float stiffness,
                                                const uint2* __restrict__ ranges, const int* tdims,
                                                     ContactWarp<AG, CAP>& s) {
    static_assert(AG <= 10 && CAP >= 64, "a lane per agent and component");
    const olc_u32 all = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const olc_u32 below = (1u << lane) - 1u;
    if (lane < AG) s.p[lane] = p;
    __syncwarp();
    // lane 3 a + e sums component e of agent a: its listed parts are hits beg .. end - 1
    float f = 0.0f;
    int cnt = 0, beg = 0, end = 0;
    const int own = lane / 3, comp = lane - 3 * own;
    auto drain = [&]() {
        __syncwarp();  // the lanes' listed pairs are visible to one another
        for (int h = lane; h < cnt; h += 32) {
            const uint2 hit = s.hit[h];
            const float3 v = contact_pair(s.p[hit.y], __ldg(posr + hit.x), base + hit.y, hit.x, stiffness);
            s.hit[h] = make_uint2(__float_as_uint(v.x), __float_as_uint(v.y));
            s.fz[h] = v.z;
        }
        __syncwarp();
        const float* src = comp == 2 ? s.fz : reinterpret_cast<const float*>(s.hit) + comp;
        const int step = comp == 2 ? 1 : 2;
        for (int h = beg; h < end; ++h) f = __fadd_rn(f, src[h * step]);
        __syncwarp();
        cnt = beg = end = 0;
    };
    const olc_u32 group = olc_tissue_key(c.x, c.y, c.z);
    olc_u32 todo = __ballot_sync(all, active && lane < AG);
    while (todo) {
        // the agents of one bin share its candidates
        const int lead = __ffs(todo) - 1;
        const olc_u32 same = __ballot_sync(all, group == __shfl_sync(all, group, lead)) & todo;
        todo &= ~same;
        const int cx = __shfl_sync(all, c.x, lead) + lane % 3 - 1;
        const int cy = __shfl_sync(all, c.y, lead) + lane / 3 % 3 - 1;
        const int cz = __shfl_sync(all, c.z, lead) + lane / 9 - 1;
        const uint2 rg = lane < 27 ? contact_rows(ranges, tdims, cx, cy, cz) : make_uint2(0u, 0u);
        const olc_u32 len = rg.y > rg.x ? rg.y - rg.x : 0u;
        olc_u32 at = len;
#pragma unroll
        for (int d = 1; d < 32; d *= 2) {
            const olc_u32 v = __shfl_up_sync(all, at, d);
            if (lane >= d) at += v;
        }
        const olc_u32 total = __shfl_sync(all, at, 31);
        at -= len;  // place of this bin's first row among the candidates
        for (olc_u32 c0 = 0; c0 < total; c0 += CONTACT_CHUNK) {
            if (c0 > 0) drain();  // an agent's listed pairs are one piece of the list
            const olc_u32 have = min(total - c0, (olc_u32)CONTACT_CHUNK);
            for (olc_u32 k = at < c0 ? c0 - at : 0u; k < len && at + k - c0 < have; ++k) s.row[at + k - c0] = rg.x + k;
            __syncwarp();
            olc_u32 j[CONTACT_CHUNK / 32];
            float4 q[CONTACT_CHUNK / 32];
#pragma unroll
            for (int r = 0; r < CONTACT_CHUNK / 32; ++r) {
                q[r] = make_float4(__int_as_float(0x7fffffff), 0.0f, 0.0f, 0.0f);  // near nothing
                j[r] = 0;
                if (32 * r + lane < have) {
                    j[r] = s.row[32 * r + lane];
                    q[r] = __ldg(posr + j[r]);
                }
            }
            for (olc_u32 m = same; m; m &= m - 1) {
                const int a = __ffs(m) - 1;
                const float4 pa = s.p[a];
                if (own == a) beg = cnt;
#pragma unroll
                for (int r = 0; r < CONTACT_CHUNK / 32; ++r) {
                    if (32 * r >= have) break;
                    const bool near = contact_near(pa, q[r]);
                    const olc_u32 nm = __ballot_sync(all, near);
                    if (cnt + __popc(nm) > CAP) {
                        if (own == a) end = cnt;
                        drain();
                    }
                    if (near) s.hit[cnt + __popc(nm & below)] = make_uint2(j[r], (olc_u32)a);
                    cnt += __popc(nm);
                }
                if (own == a) end = cnt;
            }
            __syncwarp();
        }
    }
    drain();
    const int src = lane < AG ? 3 * lane : 0;
    return make_float3(__shfl_sync(all, f, src), __shfl_sync(all, f, src + 1), __shfl_sync(all, f, src + 2));
}

}  // namespace olc
