// FLIP water step of the reference engine (NeonEngine/shaders/water_grid.comp, passes 0-8, in the
// dispatch order of NeonEngine/src/water_physics.cpp:164-430) as CUDA kernels behind the C ABI of
// include/neon_water.h.  This translation unit is compiled with -fmad=false: every kernel uses
// the shader's 32-bit float operations in the shader's order, so the results equal the CPU
// restatement bit for bit.  No CPU fallback exists.
//
// Redesign relative to the shader (results unchanged):
//  * pass 1 (all-pairs particle separation) runs one WARP per particle over the particles of the 27
//    cells around it (linked lists, built by the kernel that wrote the positions); the close ones are
//    applied one by one in ascending index, each time re-testing the later ones with the moved
//    position, which is exactly the sequential loop's arithmetic;
//  * passes 0 and 2-4 (reset, scatter with float compare-and-swap loops, normalising pass) become one
//    gather: one thread per node collects the particles of the 27 bins around it, orders them by id
//    and adds their contributions to its three velocity components and its density in that order -
//    no float atomics, deterministic;
//  * all pressure iterations run in one thread-block cluster with the field in shared memory;
//  * one step is a CUDA graph.
#include "../../include/neon_water.h"

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <new>
#include <string>
#include <utility>

namespace {

constexpr unsigned kFluid = 1u, kSolid = 2u;

struct WP {  // parameters every kernel takes by value
    int N, nx, ny, nz, C;
    float cs, orx, rd, damp, mass, dt;
    float bmin[3], bmax[3], g[3];
};

struct Stencil {
    int base[3];
    float frac[3];
};

__device__ __forceinline__ Stencil make_stencil(const WP& q, const float4& pos, float ox, float oy, float oz) {
    Stencil s;
    const float p[3] = {pos.x, pos.y, pos.z}, off[3] = {ox, oy, oz};
    const int dim[3] = {q.nx, q.ny, q.nz};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float local = (p[a] - q.bmin[a]) / q.cs;
        const float l = local - off[a];
        s.base[a] = min(max((int)floorf(l), 0), dim[a] - 2);
        s.frac[a] = l - (float)s.base[a];
    }
    return s;
}

__device__ __forceinline__ float corner_weight(const Stencil& s, int ix, int iy, int iz) {
    return (ix == 0 ? (1.0f - s.frac[0]) : s.frac[0]) * (iy == 0 ? (1.0f - s.frac[1]) : s.frac[1]) *
           (iz == 0 ? (1.0f - s.frac[2]) : s.frac[2]);
}

__device__ __forceinline__ int corner_cell(const WP& q, const Stencil& s, int ix, int iy, int iz) {
    return (s.base[0] + ix) + (s.base[1] + iy) * q.nx + (s.base[2] + iz) * (q.nx * q.ny);
}

// staggering of grid g: 0 = u faces, 1 = v faces, 2 = w faces, 3 = cell centres (density)
__device__ __forceinline__ Stencil grid_stencil(const WP& q, const float4& pos, int g) {
    return make_stencil(q, pos, g == 0 ? 0.0f : 0.5f, g == 1 ? 0.0f : 0.5f, g == 2 ? 0.0f : 0.5f);
}

// ---- particle lists ---------------------------------------------------------------------------------
// Linked lists of particle ids (-1 ends one): head[cell], next[particle].  A list's order is whatever the atomic
// exchanges made it; every reader orders what it takes by id.  Heads are cleared by an earlier kernel.
struct SepGrid {  // the separation pass's cells, at least its reach wide
    float inv;
    int n[3], M;
};

__device__ __forceinline__ int sep_axis(const WP& q, const SepGrid& sg, float p, int a) {
    return min(max((int)floorf((p - q.bmin[a]) * sg.inv), 0), sg.n[a] - 1);
}
__device__ __forceinline__ int sep_cell(const WP& q, const SepGrid& sg, float x, float y, float z) {
    return sep_axis(q, sg, x, 0) + sg.n[0] * (sep_axis(q, sg, y, 1) + sg.n[1] * sep_axis(q, sg, z, 2));
}

// A particle as the particles-to-grid gather wants it: its position in cells and the next particle of its bin.
__device__ __forceinline__ void put_in_bin(const WP& q, int i, float x, float y, float z, int* bin_head, float4* bin_rec) {
    const float l[3] = {(x - q.bmin[0]) / q.cs, (y - q.bmin[1]) / q.cs, (z - q.bmin[2]) / q.cs};
    const int dim[3] = {q.nx, q.ny, q.nz};
    int b[3];
#pragma unroll
    for (int a = 0; a < 3; ++a) b[a] = min(max((int)floorf(l[a]), 0), dim[a] - 1);
    const int next = atomicExch(bin_head + b[0] + q.nx * (b[1] + q.ny * b[2]), i);
    bin_rec[i] = make_float4(l[0], l[1], l[2], __int_as_float(next));
}

// The first sub-step's lists (start positions); without sub-steps the bins.
__global__ void k_sep_lists(WP q, SepGrid sg, const float4* __restrict__ pos, int* head, int* next) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.N) return;
    const float4 p = pos[i];
    next[i] = atomicExch(head + sep_cell(q, sg, p.x, p.y, p.z), i);
}
__global__ void k_bins(WP q, const float4* __restrict__ pos, int* bin_head, float4* bin_rec) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.N) return;
    const float4 p = pos[i];
    put_in_bin(q, i, p.x, p.y, p.z, bin_head, bin_rec);
}

// ---- pass 1 (water_grid.comp:721-744) on a snapshot: src -> dst ---------------------------------
// One warp per particle.  It collects, around its current position, the particles within the separation distance
// plus kSlack cells (27 lanes walk the lists of the 27 cells around it), then repeats: the lowest index beyond the
// last applied one that is closer than the separation distance is applied.  Between two applications the position
// stands still, so this visits the same neighbours with the same positions as the loop over all indices; and as long
// as the particle has moved less than the slack since the collection, every neighbour that can be close is in it -
// after that it collects again around where it is.  More than kSepCap candidates: all particles in order.
// The kernel ends with the lists its reader wants: the next sub-step's cells, or (LAST) the gather's bins.
// Bound by the latency of a few dependent L2 reads and of the chain of square roots and divisions; before, with
// boxes of 32 consecutive indices instead of cells, a sub-step of 8000 particles took 30 us.
constexpr int kSepWarps = 8, kSepCap = 128;
constexpr float kSlack = 0.5f;  // in grid cells
__host__ __device__ inline float sep_reach(float cs) { return cs * 1.5f + cs * kSlack; }

template <bool LAST>
__global__ void __launch_bounds__(kSepWarps * 32) k_separate(WP q, SepGrid sg, const float4* __restrict__ src, const int* __restrict__ head,
                                                             const int* __restrict__ next, float4* __restrict__ dst, int* head_out,
                                                             int* next_out, float4* bin_rec, int* __restrict__ head_clear) {
    __shared__ float4 found[kSepWarps][kSepCap];  // {position, id}
    constexpr unsigned all = 0xffffffffu;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < sg.M; c += gridDim.x * blockDim.x) head_clear[c] = -1;
    const int i = blockIdx.x * kSepWarps + warp;
    if (i >= q.N) return;
    float4* mine = found[warp];
    const float min_dist = q.cs * 1.5f, min_dist2 = min_dist * min_dist;
    const float reach = sep_reach(q.cs), reach2 = reach * reach * 1.0002f, slack = q.cs * kSlack, slack2 = slack * slack * 0.9998f;
    const float4 me = src[i];
    float px = me.x, py = me.y, pz = me.z;
    auto apply = [&](float ax, float ay, float az, float a2) {
        const float d = sqrtf(a2);
        const float f = 0.5f * (min_dist - d) / d;
        px += ax * f;
        py += ay * f;
        pz += az * f;
    };
    int after = -1;  // the last index applied
    bool again = true;
    while (again) {
        again = false;
        const float gx = px, gy = py, gz = pz;
        int j = -1, n = 0;
        if (lane < 27) {
            const int cx = sep_axis(q, sg, gx, 0) + lane % 3 - 1, cy = sep_axis(q, sg, gy, 1) + lane / 3 % 3 - 1, cz = sep_axis(q, sg, gz, 2) + lane / 9 - 1;
            if (cx >= 0 && cx < sg.n[0] && cy >= 0 && cy < sg.n[1] && cz >= 0 && cz < sg.n[2]) j = __ldg(head + cx + sg.n[0] * (cy + sg.n[1] * cz));
        }
        __syncwarp();
        int hops = 0;
        for (; hops < q.N && n <= kSepCap && __any_sync(all, j >= 0); ++hops) {
            bool take = false;
            float4 o = make_float4(0.f, 0.f, 0.f, 0.f);
            int then = -1;
            if (j >= 0) {
                o = src[j];
                then = __ldg(next + j);
                const float dx = gx - o.x, dy = gy - o.y, dz = gz - o.z;
                take = j > after && j != i && !(dx * dx + dy * dy + dz * dz > reach2);
            }
            const unsigned who = __ballot_sync(all, take);
            const int slot = n + __popc(who & ((1u << lane) - 1u));
            if (take && slot < kSepCap) mine[slot] = make_float4(o.x, o.y, o.z, __int_as_float(j));
            n += __popc(who);
            j = then;
        }
        __syncwarp();
        // Crowded beyond the list, or so that walking again (after every sixth application or so, of which there are about
        // 0.4 n; a hop waits for its predecessor) costs more than looking at every later index: those in order, 32 at a time.
        // 8000 particles at 4.6 a cell, us a sub-step: 168 by this rule, 370 by the lists alone.
        if (n > kSepCap || 3 * (n / 16 + 1) * min(hops, 1 << 20) > (q.N - after) / 32) {
            for (int base = (after + 1) & ~31; base < q.N; base += 32) {
                const int k = base + lane;
                const bool valid = k < q.N && k != i && k > after;
                const float4 o = k < q.N ? src[k] : make_float4(0.f, 0.f, 0.f, 0.f);
                float dx = px - o.x, dy = py - o.y, dz = pz - o.z;
                float d2 = dx * dx + dy * dy + dz * dz;
                unsigned mask = __ballot_sync(all, valid && !(d2 >= min_dist2 || d2 == 0.0f));
                while (mask) {
                    const int l = __ffs(mask) - 1;
                    apply(__shfl_sync(all, dx, l), __shfl_sync(all, dy, l), __shfl_sync(all, dz, l), __shfl_sync(all, d2, l));
                    dx = px - o.x; dy = py - o.y; dz = pz - o.z;
                    d2 = dx * dx + dy * dy + dz * dz;
                    mask = __ballot_sync(all, lane > l && valid && !(d2 >= min_dist2 || d2 == 0.0f));
                }
            }
            break;
        }
        while (true) {
            int key = 0x7fffffff;
            float ax = 0.f, ay = 0.f, az = 0.f, a2 = 0.f;
            for (int k = lane; k < n; k += 32) {
                const float4 o = mine[k];
                const int id = __float_as_int(o.w);
                const float dx = px - o.x, dy = py - o.y, dz = pz - o.z;
                const float d2 = dx * dx + dy * dy + dz * dz;
                if (id > after && id < key && !(d2 >= min_dist2 || d2 == 0.0f)) { key = id; ax = dx; ay = dy; az = dz; a2 = d2; }
            }
            const int lowest = __reduce_min_sync(all, key);
            if (lowest == 0x7fffffff) break;
            const int l = __ffs(__ballot_sync(all, key == lowest)) - 1;
            apply(__shfl_sync(all, ax, l), __shfl_sync(all, ay, l), __shfl_sync(all, az, l), __shfl_sync(all, a2, l));
            after = lowest;
            const float mx = px - gx, my = py - gy, mz = pz - gz;
            if (mx * mx + my * my + mz * mz > slack2) { again = true; break; }
        }
    }
    if (lane == 0) {
        dst[i] = make_float4(px, py, pz, me.w);
        if (LAST) put_in_bin(q, i, px, py, pz, head_out, bin_rec);
        else next_out[i] = atomicExch(head_out + sep_cell(q, sg, px, py, pz), i);
    }
}

// ---- passes 0 and 2-4 as one gather ----------------------------------------------------------------
// One thread per node.  A particle contributes to the two nodes per axis around its (staggered) position, which lie
// at most one bin from its own on every axis: the 27 bins around the node hold all its contributors, for all four
// grids.  Their ids are put in order, then added in that order (water_grid.comp:288-349 for the velocities, :695-720
// for the density) and normalised (:352-379).  Up to gather_alone(N) particles in the bins (a fluid has about four): the
// thread orders them in shared memory, kGatherCap at a time, one walk of the lists for each.  More, and the warp looks at
// all particles in the order of their ids, 32 at a time, and its crowded nodes take what lies near them, side by side; that
// costs by the number of all particles what ordering costs by the square of those in the bins.  (A walk of the lists for
// every id took 28 ms a step for 1000 particles within 0.2 cells and 135 for 1000 in one place; now 0.27 and 0.29.)
// zero_a / zero_b: pressure buffers to clear, where the pressure passes run from global memory; bar: their barrier counter.
constexpr int kGatherThreads = 128, kGatherCap = 32;
__device__ __forceinline__ int gather_alone(int N) { return max(kGatherCap, (int)sqrtf(0.05f * (float)N)); }

// What the particle of a record adds at a node: bit g of the result where it contributes to grid g (3: density), wg[g] its weight.
__device__ __forceinline__ unsigned node_weights(const WP& q, const float4& r, int gx, int gy, int gz, float (&wg)[4]) {
    // per axis: distance of the node from the stencil's base and the weight there, for faces (0) and centres (1)
    const float l[3] = {r.x, r.y, r.z};
    const int at[3] = {gx, gy, gz}, dim[3] = {q.nx, q.ny, q.nz};
    bool in[2][3];
    float wt[2][3];
#pragma unroll
    for (int o = 0; o < 2; ++o)
#pragma unroll
        for (int a = 0; a < 3; ++a) {
            const float lo = l[a] - (o ? 0.5f : 0.0f);
            const int base = min(max((int)floorf(lo), 0), dim[a] - 2), i = at[a] - base;
            const float frac = lo - (float)base;
            in[o][a] = i == 0 || i == 1;
            wt[o][a] = i == 0 ? (1.0f - frac) : frac;
        }
    unsigned grids = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        wg[g] = wt[g != 0][0] * wt[g != 1][1] * wt[g != 2][2];
        if (in[g != 0][0] && in[g != 1][1] && in[g != 2][2]) grids |= 1u << g;
    }
    return grids;
}
// False only for a particle that contributes to no node from `lo` to `hi` of an axis with n nodes: clamped to the grid as
// the stencil is, it lies from one cell before a node to one and a half behind it (and a little, for the rounding here).
__device__ __forceinline__ bool in_reach(float p, int n, int lo, int hi) {
    const float c = fminf(fmaxf(p, 0.0f), (float)(n - 1));
    return c >= (float)lo - 1.0001f && c <= (float)hi + 1.5001f;
}
__device__ __forceinline__ int bin_around(const WP& q, int node, int k) {  // the k-th of the 27 bins around a node
    return node + (k % 3 - 1) + (k / 3 % 3 - 1) * q.nx + (k / 9 - 1) * (q.nx * q.ny);
}

__global__ void __launch_bounds__(kGatherThreads, 9) k_p2g_gather(WP q, const float4* __restrict__ vel, const int* __restrict__ bin_head,
                                                               const float4* __restrict__ bin_rec, unsigned* flags, float* u, float* v,
                                                               float* w, float* pu, float* pv, float* pw, float* density,
                                                               float* zero_a, float* zero_b, unsigned* bar) {
    __shared__ int ids[kGatherCap][kGatherThreads];
    constexpr unsigned all = 0xffffffffu;
    const int tid = threadIdx.x, lane = tid & 31, node = blockIdx.x * kGatherThreads + tid;
    if (node == 0) *bar = 0u;
    if (node - lane >= q.C) return;  // whole warps: a crowded node takes all lanes
    const int nx = q.nx, ny = q.ny, nz = q.nz;
    const int gz = node / (nx * ny), rem = node - gz * (nx * ny), gy = rem / nx, gx = rem - gy * nx;
    // solid: takes nothing (nor does a lane beyond the grid)
    const bool border = gx == 0 || gx == nx - 1 || gy == 0 || gy == ny - 1 || gz == 0 || gz >= nz - 1;
    float acc[3] = {0.f, 0.f, 0.f}, wsum[3] = {0.f, 0.f, 0.f}, dens = 0.f;
    bool fluid = false, crowded = false;
    auto add = [&](const float4& r, const float4& pv4) {
        float wg[4];
        const unsigned grids = node_weights(q, r, gx, gy, gz, wg);
#pragma unroll
        for (int g = 0; g < 3; ++g) {
            if (!(grids >> g & 1u)) continue;
            const float comp = g == 0 ? pv4.x : (g == 1 ? pv4.y : pv4.z);
            acc[g] += comp * wg[g];
            wsum[g] += wg[g];
            fluid = true;
        }
        if (grids & 8u) dens += wg[3] * q.mass;
    };
    if (!border) {  // so all 27 bins exist
        int heads[27];
#pragma unroll
        for (int k = 0; k < 27; ++k) heads[k] = __ldg(bin_head + bin_around(q, node, k));
        const int alone = gather_alone(q.N);
        int m = 0, n = 0;  // ids kept (the lowest ones seen, ascending), particles in the bins
        auto keep = [&](int j) {
            int b = m - 1;
            if (m < kGatherCap) ++m;
            else if (ids[b][tid] < j) return;
            else --b;
            while (b >= 0 && ids[b][tid] > j) { ids[b + 1][tid] = ids[b][tid]; --b; }
            ids[b + 1][tid] = j;
        };
#pragma unroll
        for (int k = 0; k < 27; ++k)
            for (int j = heads[k]; j >= 0 && n <= alone; ++n) {
                keep(j);
                j = __float_as_int(__ldg(&bin_rec[j].w));
            }
        crowded = n > alone;
        for (int left = crowded ? 0 : n; left > 0;) {
            for (int k = 0; k < m; ++k) {
                const int id = ids[k][tid];
                add(__ldg(bin_rec + id), __ldg(vel + id));
            }
            left -= m;
            if (left <= 0) break;
            const int last = ids[m - 1][tid];
            m = 0;
            int hops = 0;
            for (int c = 0; c < 27; ++c)
                for (int j = __ldg(bin_head + bin_around(q, node, c)); j >= 0 && hops < n; ++hops) {
                    if (j > last) keep(j);
                    j = __float_as_int(__ldg(&bin_rec[j].w));
                }
            if (!m) break;
        }
    }
    if (__any_sync(all, crowded)) {
        // the box of the crowded nodes
        const int big = 0x7fffffff;
        const int x0 = __reduce_min_sync(all, crowded ? gx : big), x1 = __reduce_max_sync(all, crowded ? gx : -1);
        const int y0 = __reduce_min_sync(all, crowded ? gy : big), y1 = __reduce_max_sync(all, crowded ? gy : -1);
        const int z0 = __reduce_min_sync(all, crowded ? gz : big), z1 = __reduce_max_sync(all, crowded ? gz : -1);
        float4 next = lane < q.N ? __ldg(bin_rec + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        for (int first = 0; first < q.N; first += 32) {
            const int id = first + lane;
            const float4 r = next;
            if (id + 32 < q.N) next = __ldg(bin_rec + id + 32);
            unsigned who = __ballot_sync(all, id < q.N && in_reach(r.x, nx, x0, x1) && in_reach(r.y, ny, y0, y1) && in_reach(r.z, nz, z0, z1));
            if (!who) continue;
            const float4 pv4 = who >> lane & 1u ? __ldg(vel + id) : r;
            for (; who; who &= who - 1) {
                const int l = __ffs(who) - 1;
                const float4 one = make_float4(__shfl_sync(all, r.x, l), __shfl_sync(all, r.y, l), __shfl_sync(all, r.z, l), 0.f);
                const float4 its = make_float4(__shfl_sync(all, pv4.x, l), __shfl_sync(all, pv4.y, l), __shfl_sync(all, pv4.z, l), 0.f);
                if (crowded) add(one, its);
            }
        }
    }
    if (node >= q.C) return;
    if (zero_a) { zero_a[node] = 0.f; zero_b[node] = 0.f; }
    flags[node] = border ? kSolid : (fluid ? kFluid : 0u);
    const float eps = 1e-6f;
    float val[3];
#pragma unroll
    for (int g = 0; g < 3; ++g) val[g] = wsum[g] > eps ? acc[g] / wsum[g] : 0.0f;
    u[node] = val[0]; v[node] = val[1]; w[node] = val[2];
    pu[node] = val[0]; pv[node] = val[1]; pw[node] = val[2];
    density[node] = dens;
}

// The border's solidity, which no step changes.
__global__ void k_solidity(WP q, float* s) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= q.C) return;
    const int gz = idx / (q.nx * q.ny), rem = idx - gz * (q.nx * q.ny), gy = rem / q.nx, gx = rem - gy * q.nx;
    s[idx] = gx == 0 || gx == q.nx - 1 || gy == 0 || gy == q.ny - 1 || gz == 0 || gz == q.nz - 1 ? 0.0f : 1.0f;
}

// ---- pass 5 (water_grid.comp:382-488) ----------------------------------------------------------------
__global__ void k_jacobi(WP q, const unsigned* __restrict__ flags, const float* __restrict__ s, const float* __restrict__ u,
                         const float* __restrict__ v, const float* __restrict__ w, const float* __restrict__ density,
                         const float* __restrict__ p_read, float* __restrict__ p_write) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    if (idx >= q.C) return;
    const int nx = q.nx, ny = q.ny, nz = q.nz;
    const int gz = idx / (nx * ny), rem = idx - gz * (nx * ny), gy = rem / nx, gx = rem - gy * nx;
    const float here = p_read[idx];
    if (gx == 0 || gx == nx - 1 || gy == 0 || gy == ny - 1 || gz == 0 || gz == nz - 1 || (flags[idx] & kFluid) == 0u) {
        p_write[idx] = here;
        return;
    }
    const int left = idx - 1, right = idx + 1, bottom = idx - nx, top = idx + nx, back = idx - nx * ny, front = idx + nx * ny;
    const float sx0 = s[left], sx1 = s[right], sy0 = s[bottom], sy1 = s[top], sz0 = s[back], sz1 = s[front];
    const float s_sum = sx0 + sx1 + sy0 + sy1 + sz0 + sz1;
    if (s_sum <= 1e-9f) {
        p_write[idx] = here;
        return;
    }
    const float sum_p = sx0 * p_read[left] + sx1 * p_read[right] + sy0 * p_read[bottom] + sy1 * p_read[top] +
                        sz0 * p_read[back] + sz1 * p_read[front];
    float div = ((u[right] - u[idx]) + (v[top] - v[idx]) + (w[front] - w[idx]));
    const float pd = density[idx];
    if (q.rd > 0.0f && pd > 0.0f) {
        const float compression = pd - q.rd;
        if (compression > 0.0f) div -= compression;
    }
    const float dt_safe = fmaxf(q.dt, 1e-6f), cs_safe = fmaxf(q.cs, 1e-6f), rd_safe = fmaxf(q.rd, 1e-6f);
    const float cp = rd_safe * cs_safe * cs_safe / dt_safe;
    const float div_safe = fminf(fmaxf(div, -1e6f), 1e6f);
    const float p_new = (sum_p - cp * div_safe) / fmaxf(s_sum, 1e-6f);
    p_write[idx] = here + q.orx * (p_new - here);
}

// All Jacobi iterations in ONE cooperative launch: every thread keeps the iteration-invariant
// terms of its (at most two) cells in registers - neighbour solidities, cp * div and the
// denominator, formed by the same float operations as k_jacobi - and an iteration is seven L2
// loads, one store and a grid-wide barrier.  Cells that only copy their pressure never leave
// the zero pass 0 gave both buffers, so they are not touched.  The barrier is a counter in
// global memory with a bounded spin: on a timeout the status word is set and every CTA leaves.
constexpr int kFusedThreads = 1024;
__global__ void __launch_bounds__(kFusedThreads, 1)
k_jacobi_fused(WP q, const unsigned* __restrict__ flags, const float* __restrict__ s, const float* __restrict__ u,
               const float* __restrict__ v, const float* __restrict__ w, const float* __restrict__ density, float* pa, float* pb,
               int iterations, unsigned* bar, int* status) {
    const int T = gridDim.x * kFusedThreads, t = blockIdx.x * kFusedThreads + threadIdx.x;
    const int nx = q.nx, ny = q.ny, nz = q.nz;
    int cell[2];
    bool upd[2];
    float B[2], D[2], sn[2][6];
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        const int idx = t + k * T;
        cell[k] = idx;
        upd[k] = false;
        B[k] = 0.0f; D[k] = 1.0f;
#pragma unroll
        for (int a = 0; a < 6; ++a) sn[k][a] = 0.0f;
        if (idx >= q.C) continue;
        const int gz = idx / (nx * ny), rem = idx - gz * (nx * ny), gy = rem / nx, gx = rem - gy * nx;
        if (gx == 0 || gx == nx - 1 || gy == 0 || gy == ny - 1 || gz == 0 || gz == nz - 1 || (flags[idx] & kFluid) == 0u) continue;
        const int left = idx - 1, right = idx + 1, bottom = idx - nx, top = idx + nx, back = idx - nx * ny, front = idx + nx * ny;
        sn[k][0] = s[left]; sn[k][1] = s[right]; sn[k][2] = s[bottom]; sn[k][3] = s[top]; sn[k][4] = s[back]; sn[k][5] = s[front];
        const float s_sum = sn[k][0] + sn[k][1] + sn[k][2] + sn[k][3] + sn[k][4] + sn[k][5];
        if (s_sum <= 1e-9f) continue;
        float div = ((u[right] - u[idx]) + (v[top] - v[idx]) + (w[front] - w[idx]));
        const float pd = density[idx];
        if (q.rd > 0.0f && pd > 0.0f) {
            const float compression = pd - q.rd;
            if (compression > 0.0f) div -= compression;
        }
        const float dt_safe = fmaxf(q.dt, 1e-6f), cs_safe = fmaxf(q.cs, 1e-6f), rd_safe = fmaxf(q.rd, 1e-6f);
        const float cp = rd_safe * cs_safe * cs_safe / dt_safe;
        const float div_safe = fminf(fmaxf(div, -1e6f), 1e6f);
        B[k] = cp * div_safe;
        D[k] = fmaxf(s_sum, 1e-6f);
        upd[k] = true;
    }
    __shared__ int give_up;
    if (threadIdx.x == 0) give_up = 0;
    __syncthreads();
    for (int it = 0; it < iterations; ++it) {
        const float* p_read = (it % 2 == 0) ? pa : pb;
        float* p_write = (it % 2 == 0) ? pb : pa;
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (!upd[k]) continue;
            const int idx = cell[k];
            const float here = __ldcg(p_read + idx);
            const float sum_p = sn[k][0] * __ldcg(p_read + idx - 1) + sn[k][1] * __ldcg(p_read + idx + 1) +
                                sn[k][2] * __ldcg(p_read + idx - nx) + sn[k][3] * __ldcg(p_read + idx + nx) +
                                sn[k][4] * __ldcg(p_read + idx - nx * ny) + sn[k][5] * __ldcg(p_read + idx + nx * ny);
            const float p_new = (sum_p - B[k]) / D[k];
            __stcg(p_write + idx, here + q.orx * (p_new - here));
        }
        if (it + 1 == iterations) break;
        // grid barrier number it + 1: all CTAs have added 1 when the counter reaches (it + 1) * gridDim.x
        __syncthreads();
        if (threadIdx.x == 0) {
            // arrive with release semantics (orders this CTA's stores, made visible to thread 0 by the
            // barrier above, before the count), then poll with acquire loads
            asm volatile("red.release.gpu.global.add.u32 [%0], 1;" ::"l"(bar) : "memory");
            const unsigned target = (unsigned)(it + 1) * gridDim.x;
            long long spins = 0;
            for (;;) {
                unsigned seen;
                asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(seen) : "l"(bar) : "memory");
                if (seen >= target) break;
                if (++spins > 2000000ll || *reinterpret_cast<volatile int*>(status) != 0) {
                    atomicExch(status, 1);
                    give_up = 1;
                    break;
                }
            }
        }
        __syncthreads();
        if (give_up) return;
    }
}

// The same iterations in ONE thread-block cluster, for grids whose pressure field fits its shared memory twice.  CTA r
// owns L consecutive cells and keeps them between copies of the P = nx * ny cells before and after them (one layer of
// the grid, as far as a neighbour can lie); who writes a cell that a neighbouring CTA keeps a copy of writes the copy
// too, through distributed shared memory, and the cluster's barrier ends an iteration.  The cells that are updated at
// all (interior, fluid, not walled in) are listed once, so that a thread's share is of work and not of space; the
// terms that no iteration changes stay in registers.  Border cells are walls of pressure zero, so the solidity factors
// of the shader's sum (0 or 1) need no multiplication: the sum's terms and their order are the same.
// The shader's last iteration writes a buffer that nothing reads; it is not run.
// (The whole step of 8000 particles in 99 x 37 x 44 cells: 152 us, with the separation, gather and grid-wide
// pressure kernels before it 261 us.)
constexpr int kClusterThreads = 1024, kClusterCells = 12;
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release;\n\tbarrier.cluster.wait.acquire;" ::: "memory");
}
size_t cluster_smem(int L, int P) { return (size_t)2 * (L + 2 * P) * 4 + (size_t)L * 2; }

__global__ void __launch_bounds__(kClusterThreads, 1)
k_jacobi_cluster(WP q, const unsigned* __restrict__ flags, const float* __restrict__ u, const float* __restrict__ v, const float* __restrict__ w,
                 const float* __restrict__ density, float* __restrict__ p_out, int L, int updates) {
    extern __shared__ __align__(16) unsigned char cluster_mem[];
    __shared__ int n_list;
    const int nx = q.nx, ny = q.ny, nz = q.nz, P = nx * ny, span = L + 2 * P;
    float* buf = reinterpret_cast<float*>(cluster_mem);  // [2][span]
    uint16_t* list = reinterpret_cast<uint16_t*>(buf + 2 * span);
    unsigned rank, size;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    asm("mov.u32 %0, %%cluster_nctarank;" : "=r"(size));
    const int tid = threadIdx.x, lane = tid & 31, first = (int)rank * L;
    for (int i = tid; i < 2 * span; i += kClusterThreads) buf[i] = 0.0f;
    if (tid == 0) n_list = 0;
    __syncthreads();
    for (int o0 = 0; o0 < L; o0 += kClusterThreads) {
        const int o = o0 + tid, idx = first + o;
        bool upd = false;
        if (o < L && idx < q.C && (flags[idx] & kFluid)) {  // solid cells are never fluid
            const int gz = idx / P, rem = idx - gz * P, gy = rem / nx, gx = rem - gy * nx;
            // some neighbour is no border cell
            upd = gx > 1 || gx < nx - 2 || gy > 1 || gy < ny - 2 || gz > 1 || gz < nz - 2;
        }
        const unsigned who = __ballot_sync(0xffffffffu, upd);
        int at = 0;
        if (lane == 0 && who) at = atomicAdd(&n_list, __popc(who));
        at = __shfl_sync(0xffffffffu, at, 0);
        if (upd) list[at + __popc(who & ((1u << lane) - 1u))] = (uint16_t)o;
    }
    __syncthreads();
    const int n = n_list;
    int at[kClusterCells];
    float B[kClusterCells], D[kClusterCells];
#pragma unroll
    for (int k = 0; k < kClusterCells; ++k) {
        at[k] = -1;
        B[k] = 0.0f; D[k] = 1.0f;
        if (k * kClusterThreads + tid < n) {
            const int o = list[k * kClusterThreads + tid], idx = first + o;
            const int gz = idx / P, rem = idx - gz * P, gy = rem / nx, gx = rem - gy * nx;
            const float s_sum = (gx > 1 ? 1.f : 0.f) + (gx < nx - 2 ? 1.f : 0.f) + (gy > 1 ? 1.f : 0.f) + (gy < ny - 2 ? 1.f : 0.f) +
                                (gz > 1 ? 1.f : 0.f) + (gz < nz - 2 ? 1.f : 0.f);
            float div = ((u[idx + 1] - u[idx]) + (v[idx + nx] - v[idx]) + (w[idx + P] - w[idx]));
            const float pd = density[idx];
            if (q.rd > 0.0f && pd > 0.0f) {
                const float compression = pd - q.rd;
                if (compression > 0.0f) div -= compression;
            }
            const float dt_safe = fmaxf(q.dt, 1e-6f), cs_safe = fmaxf(q.cs, 1e-6f), rd_safe = fmaxf(q.rd, 1e-6f);
            const float cp = rd_safe * cs_safe * cs_safe / dt_safe;
            const float div_safe = fminf(fmaxf(div, -1e6f), 1e6f);
            at[k] = P + o;
            B[k] = cp * div_safe;
            D[k] = s_sum;
        }
    }
    const unsigned base = (unsigned)__cvta_generic_to_shared(buf);
    unsigned left = 0, right = 0;
    if (rank > 0) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(left) : "r"(base), "r"(rank - 1));
    if (rank + 1 < size) asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(right) : "r"(base), "r"(rank + 1));
    cluster_sync_all();  // everybody's buffers are cleared
    for (int it = 0; it < updates; ++it) {
        const float* now = buf + (it & 1) * span;
        float* then = buf + ((it & 1) ^ 1) * span;
        const unsigned then_off = (unsigned)(((it & 1) ^ 1) * span);
#pragma unroll
        for (int k = 0; k < kClusterCells; ++k) {
            if (k * kClusterThreads >= n) break;
            const int i = at[k];
            if (i < 0) continue;
            const float here = now[i];
            const float sum_p = now[i - 1] + now[i + 1] + now[i - nx] + now[i + nx] + now[i - P] + now[i + P];
            const float p_new = (sum_p - B[k]) / D[k];
            const float value = here + q.orx * (p_new - here);
            then[i] = value;
            if (left && i < 2 * P) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(left + (then_off + (unsigned)(i + L)) * 4u), "f"(value) : "memory");
            if (right && i >= L) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(right + (then_off + (unsigned)(i - L)) * 4u), "f"(value) : "memory");
        }
        cluster_sync_all();
    }
    const float* last = buf + (updates & 1) * span;
    for (int o = tid; o < L; o += kClusterThreads)
        if (first + o < q.C) p_out[first + o] = last[P + o];
}

// ---- pass 6 (water_grid.comp:491-560) ----------------------------------------------------------------
// Also clears the particle lists' heads that this step is done with: the bins, and the separation cells [0, n_sep).
__global__ void k_pressure_apply(WP q, const unsigned* __restrict__ flags, const float* __restrict__ p, float* u, float* v,
                                 float* w, int* bin_head, int* sep_head, int n_sep) {
    const int idx = blockIdx.x * blockDim.x + threadIdx.x;
    for (int c = idx; c < n_sep; c += gridDim.x * blockDim.x) sep_head[c] = -1;
    if (idx >= q.C) return;
    bin_head[idx] = -1;
    const int nx = q.nx, ny = q.ny, nz = q.nz;
    const int gz = idx / (nx * ny), rem = idx - gz * (nx * ny), gy = rem / nx, gx = rem - gy * nx;
    if (gx == 0 || gy == 0 || gz == 0 || gx >= nx - 1 || gy >= ny - 1 || gz >= nz - 1) return;
    if ((flags[idx] & kFluid) == 0u) return;
    const float inv_cp = q.dt / (q.rd * q.cs);
    const float p0 = p[idx];
    const int left = idx - 1, right = idx + 1, bot = idx - nx, top = idx + nx, back = idx - nx * ny, front = idx + nx * ny;
    u[idx] = (flags[left] & kSolid) ? 0.0f : u[idx] - (p0 - p[left]) * inv_cp;
    v[idx] = (flags[bot] & kSolid) ? 0.0f : v[idx] - (p0 - p[bot]) * inv_cp;
    w[idx] = (flags[back] & kSolid) ? 0.0f : w[idx] - (p0 - p[back]) * inv_cp;
    // faces of solid neighbours: those cells are border cells, whose own threads returned above
    if (flags[right] & kSolid) u[right] = 0.0f;
    if (flags[top] & kSolid) v[top] = 0.0f;
    if (flags[front] & kSolid) w[front] = 0.0f;
}

// ---- passes 7 and 8 (water_grid.comp:574-693), one thread per particle ----------------------------------
// pos_in: where the separation left the positions; head, next: the next step's first separation lists (nullptr: none).
__global__ void k_g2p_integrate(WP q, SepGrid sg, const unsigned* __restrict__ flags, const float* __restrict__ u, const float* __restrict__ v,
                                const float* __restrict__ w, const float* __restrict__ pu, const float* __restrict__ pv,
                                const float* __restrict__ pw, const float4* pos_in, float4* pos, float4* vel, int* head, int* next) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= q.N) return;
    const float4 p = pos_in[i];
    const float4 pv4 = vel[i];
    const float old[3] = {pv4.x, pv4.y, pv4.z};
    float nv[3] = {pv4.x, pv4.y, pv4.z};
    const float flip = fminf(fmaxf(q.damp, 0.0f), 1.0f);
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float* grid = a == 0 ? u : (a == 1 ? v : w);
        const float* prev = a == 0 ? pu : (a == 1 ? pv : pw);
        const Stencil st = grid_stencil(q, p, a);
        float pic = 0.0f, fl = 0.0f, tw = 0.0f;
#pragma unroll
        for (int c = 0; c < 8; ++c) {
            const int ix = c & 1, iy = (c >> 1) & 1, iz = c >> 2;
            const float wt = corner_weight(st, ix, iy, iz);
            const int cell = corner_cell(q, st, ix, iy, iz);
            if (flags[cell] & kSolid) continue;
            const float val = grid[cell];
            pic += val * wt;
            fl += (val - prev[cell]) * wt;
            tw += wt;
        }
        if (tw > 0.01f) {
            pic /= tw;
            fl /= tw;
            nv[a] = (1.0f - flip) * pic + flip * (old[a] + fl);
        }
    }
    // pass 8
    const float restitution = 0.3f, friction = 0.9f, margin = q.cs;
    float np[3] = {p.x, p.y, p.z};
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        nv[a] = nv[a] + q.g[a] * q.dt;
        np[a] = np[a] + nv[a] * q.dt;
    }
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        const float lo = q.bmin[a] + margin, hi = q.bmax[a] - margin;
        const int b = (a + 1) % 3, c = (a + 2) % 3;
        if (np[a] < lo) { np[a] = lo; nv[a] = fabsf(nv[a]) * restitution; nv[b] *= friction; nv[c] *= friction; }
        if (np[a] > hi) { np[a] = hi; nv[a] = -fabsf(nv[a]) * restitution; nv[b] *= friction; nv[c] *= friction; }
    }
    pos[i] = make_float4(np[0], np[1], np[2], 0.1f);
    vel[i] = make_float4(nv[0], nv[1], nv[2], pv4.w);
    if (head) next[i] = atomicExch(head + sep_cell(q, sg, np[0], np[1], np[2]), i);
}

thread_local std::string g_water_create_error;

}  // namespace

struct neon_water_handle {
    neon_water_config cfg{};
    WP q{};
    std::string err;
    float4 *pos = nullptr, *pos_tmp = nullptr, *vel = nullptr;
    float *u = nullptr, *v = nullptr, *w = nullptr, *pu = nullptr, *pv = nullptr, *pw = nullptr, *s = nullptr, *pa = nullptr,
          *pb = nullptr, *density = nullptr;
    unsigned* flags = nullptr;
    SepGrid sg{};
    int *sep_head = nullptr, *sep_next[2] = {nullptr, nullptr};  // three sets of heads in turn; lists of pos / pos_tmp
    int* bin_head = nullptr;                                     // the gather's bins; clear between steps
    float4* bin_rec = nullptr;
    int cluster = 0, cluster_cells = 0;  // CTAs of the pressure cluster (0: the grid does not fit one), cells of each
    unsigned* bar = nullptr;  // [0] grid-barrier counter, [1] status word (non-zero: a barrier wait gave up)
    int n_sms = 0, fused_jacobi = 1;
    bool coop = false;  // cooperative launches exist here
    const float* p_final = nullptr;
    int64_t launches = 0;
    int launches_per_step = 0;
    int use_graphs = 1;
    cudaStream_t own_stream = nullptr, last_stream = nullptr;
    cudaGraphExec_t graph = nullptr;
};

namespace {

int wfail(neon_water_handle* h, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (h) h->err = buf; else g_water_create_error = buf;
    return code;
}

#define WCU(h, call)                                                                                       \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) return wfail(h, NEON_MOE_ECUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

// the kernels of one step, in the reference's dispatch order; ev (optional) gets 5 event marks.
// Separation heads: sub-step s reads set s % 3, fills set (s + 1) % 3 and clears set (s + 2) % 3; a step starts with
// set 0 filled (by the last step's final kernel, or with the start positions) and set 1 clear.
int record_step(neon_water_handle* h, cudaStream_t st, cudaEvent_t* ev = nullptr) {
    const WP& q = h->q;
    const int cb = (q.C + 255) / 256, S = h->cfg.collision_substeps, M = h->sg.M, iters = h->cfg.jacobi_iterations;
    const bool in_cluster = h->fused_jacobi && h->cluster && iters > 1;
    int n = 0;
    if (ev) cudaEventRecord(ev[0], st);
    float4 *src = h->pos, *dst = h->pos_tmp;
    int *nsrc = h->sep_next[0], *ndst = h->sep_next[1];
    for (int i = 0; i < S; ++i) {
        const int *head = h->sep_head + (size_t)(i % 3) * M;
        int *fill = h->sep_head + (size_t)((i + 1) % 3) * M, *clear = h->sep_head + (size_t)((i + 2) % 3) * M;
        const int grid = (q.N + kSepWarps - 1) / kSepWarps;
        if (i + 1 < S) k_separate<false><<<grid, kSepWarps * 32, 0, st>>>(q, h->sg, src, head, nsrc, dst, fill, ndst, nullptr, clear);
        else k_separate<true><<<grid, kSepWarps * 32, 0, st>>>(q, h->sg, src, head, nsrc, dst, h->bin_head, nullptr, h->bin_rec, clear);
        ++n;
        std::swap(src, dst);
        std::swap(nsrc, ndst);
    }
    if (!S) { k_bins<<<(q.N + 127) / 128, 128, 0, st>>>(q, src, h->bin_head, h->bin_rec); ++n; }
    if (ev) cudaEventRecord(ev[1], st);
    k_p2g_gather<<<(q.C + kGatherThreads - 1) / kGatherThreads, kGatherThreads, 0, st>>>(
        q, h->vel, h->bin_head, h->bin_rec, h->flags, h->u, h->v, h->w, h->pu, h->pv, h->pw, h->density, in_cluster ? nullptr : h->pa, h->pb, h->bar); ++n;
    if (ev) cudaEventRecord(ev[2], st);
    const float* p_read = h->pa;
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute attr[1];
    cfg.stream = st;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (in_cluster) {
        cfg.gridDim = dim3(h->cluster);
        cfg.blockDim = dim3(kClusterThreads);
        cfg.dynamicSmemBytes = cluster_smem(h->cluster_cells, q.nx * q.ny);
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = h->cluster;
        attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
        WCU(h, cudaLaunchKernelEx(&cfg, k_jacobi_cluster, q, (const unsigned*)h->flags, (const float*)h->u, (const float*)h->v,
                                  (const float*)h->w, (const float*)h->density, h->pa, h->cluster_cells, iters - 1));
        ++n;
    } else if (h->fused_jacobi && h->coop && iters > 1 && q.C <= 2 * h->n_sms * kFusedThreads) {
        // one cooperative launch (all CTAs co-resident, one per SM) instead of `iters` launches
        cfg.gridDim = dim3(h->n_sms);
        cfg.blockDim = dim3(kFusedThreads);
        attr[0].id = cudaLaunchAttributeCooperative;
        attr[0].val.cooperative = 1;
        WCU(h, cudaLaunchKernelEx(&cfg, k_jacobi_fused, q, (const unsigned*)h->flags, (const float*)h->s, (const float*)h->u,
                                  (const float*)h->v, (const float*)h->w, (const float*)h->density, h->pa, h->pb, iters, h->bar,
                                  reinterpret_cast<int*>(h->bar + 1)));
        ++n;
        p_read = ((iters - 1) % 2 == 0) ? h->pa : h->pb;
    } else {
        for (int it = 0; it < iters; ++it) {
            p_read = (it % 2 == 0) ? h->pa : h->pb;
            float* p_write = (it % 2 == 0) ? h->pb : h->pa;
            k_jacobi<<<cb, 256, 0, st>>>(q, h->flags, h->s, h->u, h->v, h->w, h->density, p_read, p_write); ++n;
        }
    }
    // the reference leaves the last iteration's descriptor set bound: passes 6-8 read what it read
    h->p_final = p_read;
    if (ev) cudaEventRecord(ev[3], st);
    k_pressure_apply<<<cb, 256, 0, st>>>(q, h->flags, p_read, h->u, h->v, h->w, h->bin_head, h->sep_head, S ? 2 * M : 0); ++n;
    k_g2p_integrate<<<(q.N + 63) / 64, 64, 0, st>>>(q, h->sg, h->flags, h->u, h->v, h->w, h->pu, h->pv, h->pw, src, h->pos, h->vel,
                                                    S ? h->sep_head : nullptr, h->sep_next[0]); ++n;
    if (ev) cudaEventRecord(ev[4], st);
    h->launches_per_step = n;
    WCU(h, cudaGetLastError());
    return NEON_MOE_OK;
}

// the first sub-step's lists for positions that arrived from outside, in stream order
int record_lists(neon_water_handle* h, cudaStream_t st) {
    const WP& q = h->q;
    WCU(h, cudaMemsetAsync(h->bin_head, 0xff, (size_t)q.C * 4, st));
    if (!h->cfg.collision_substeps) return NEON_MOE_OK;
    WCU(h, cudaMemsetAsync(h->sep_head, 0xff, (size_t)2 * h->sg.M * 4, st));
    k_sep_lists<<<(q.N + 127) / 128, 128, 0, st>>>(q, h->sg, h->pos, h->sep_head, h->sep_next[0]);
    h->launches++;
    WCU(h, cudaGetLastError());
    return NEON_MOE_OK;
}

// cells of the separation pass: at least its reach wide (with a margin for the rounding of the cell index), at most
// 1024 per axis and 2^20 in all
SepGrid make_sep_grid(const WP& q) {
    SepGrid sg{};
    for (float width = sep_reach(q.cs) * 1.002f;; width *= 1.25f) {
        sg.inv = 1.0f / width;
        long long m = 1;
        bool fits = true;
        for (int a = 0; a < 3; ++a) {
            const float extent = q.bmax[a] - q.bmin[a];
            sg.n[a] = 1;  // also for a box that is not finite along an axis
            if (!std::isfinite(extent)) continue;
            const double cells = std::floor((double)extent * sg.inv) + 1.0;
            fits = fits && cells <= 1024.0;
            if (cells >= 1.0) sg.n[a] = (int)std::min(cells, 1024.0);
            m *= sg.n[a];
        }
        sg.M = (int)m;
        if (fits && m <= (1 << 20)) return sg;
    }
}

}  // namespace

extern "C" {

const char* neon_water_last_error(const neon_water_handle* h) { return h ? h->err.c_str() : g_water_create_error.c_str(); }
int64_t neon_water_launch_count(const neon_water_handle* h) { return h ? h->launches : 0; }

int neon_water_destroy(neon_water_handle* h) {
    if (!h) return NEON_MOE_OK;
    cudaSetDevice(h->cfg.device);
    cudaDeviceSynchronize();
    if (h->graph) cudaGraphExecDestroy(h->graph);
    for (void* p : {(void*)h->pos, (void*)h->pos_tmp, (void*)h->vel, (void*)h->u, (void*)h->v, (void*)h->w, (void*)h->pu,
                    (void*)h->pv, (void*)h->pw, (void*)h->s, (void*)h->pa, (void*)h->pb, (void*)h->density, (void*)h->flags,
                    (void*)h->sep_head, (void*)h->sep_next[0], (void*)h->sep_next[1], (void*)h->bin_head, (void*)h->bin_rec, (void*)h->bar})
        if (p) cudaFree(p);
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    cudaGetLastError();
    delete h;
    return NEON_MOE_OK;
}

int neon_water_create(const neon_water_config* cfg, const float* pos4, int on_device, neon_water_handle** out) {
    if (!cfg || !out) return wfail(nullptr, NEON_MOE_EINVAL, "null argument");
    *out = nullptr;
    const auto& c = *cfg;
    if (c.n_particles <= 0 || c.n_particles > (1 << 27)) return wfail(nullptr, NEON_MOE_EINVAL, "particle count %d out of range", c.n_particles);
    if (c.nx < 2 || c.ny < 2 || c.nz < 2 || (long long)c.nx * c.ny * c.nz > (1ll << 27))
        return wfail(nullptr, NEON_MOE_EINVAL, "grid %d x %d x %d out of range (at least 2 cells per axis)", c.nx, c.ny, c.nz);
    if (!(c.cell_size > 0.f) || !(c.dt > 0.f) || c.collision_substeps < 0 || c.jacobi_iterations < 0)
        return wfail(nullptr, NEON_MOE_EINVAL, "cell size and time step must be positive, loop counts non-negative");
    if (!pos4) return wfail(nullptr, NEON_MOE_EINVAL, "null start positions");
    if (cudaSetDevice(c.device) != cudaSuccess) {
        cudaGetLastError();
        return wfail(nullptr, NEON_MOE_ECUDA, "cudaSetDevice(%d) failed", c.device);
    }
    auto* h = new (std::nothrow) neon_water_handle;
    if (!h) return wfail(nullptr, NEON_MOE_ECUDA, "out of host memory");
    h->cfg = c;
    WP& q = h->q;
    q.N = c.n_particles; q.nx = c.nx; q.ny = c.ny; q.nz = c.nz; q.C = c.nx * c.ny * c.nz;
    q.cs = c.cell_size; q.orx = c.over_relaxation; q.rd = c.rest_density; q.damp = c.damping; q.mass = c.mass; q.dt = c.dt;
    for (int a = 0; a < 3; ++a) { q.bmin[a] = c.box_min[a]; q.bmax[a] = c.box_max[a]; q.g[a] = c.gravity[a]; }
    const size_t C = (size_t)q.C, N = (size_t)q.N;
    bool ok = true;
    auto alloc = [&](auto& ptr, size_t bytes) {
        if (ok && cudaMalloc(reinterpret_cast<void**>(&ptr), bytes) != cudaSuccess) ok = false;
        if (ok && cudaMemset(ptr, 0, bytes) != cudaSuccess) ok = false;
    };
    alloc(h->pos, N * 16); alloc(h->pos_tmp, N * 16); alloc(h->vel, N * 16);
    alloc(h->u, C * 4); alloc(h->v, C * 4); alloc(h->w, C * 4); alloc(h->pu, C * 4); alloc(h->pv, C * 4); alloc(h->pw, C * 4);
    alloc(h->s, C * 4); alloc(h->pa, C * 4); alloc(h->pb, C * 4); alloc(h->density, C * 4); alloc(h->flags, C * 4);
    h->sg = make_sep_grid(q);
    alloc(h->sep_head, (size_t)3 * h->sg.M * 4); alloc(h->sep_next[0], N * 4); alloc(h->sep_next[1], N * 4);
    alloc(h->bin_head, C * 4); alloc(h->bin_rec, N * 16); alloc(h->bar, 16);
    if (ok && cudaDeviceGetAttribute(&h->n_sms, cudaDevAttrMultiProcessorCount, c.device) != cudaSuccess) ok = false;
    int coop = 0;
    if (ok && cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, c.device) == cudaSuccess && coop) h->coop = true;
    if (ok) {
        k_solidity<<<(unsigned)((C + 255) / 256), 256>>>(q, h->s);
        ok = cudaGetLastError() == cudaSuccess;
    }
    // the pressure cluster: the most CTAs (of the sizes 16 ... 1) whose own cells reach one grid layer - so that copies
    // come from the next CTA alone -, fit a thread's registers and, with the copies, shared memory
    if (ok && cudaFuncSetAttribute(k_jacobi_cluster, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess) {
        const int P = q.nx * q.ny;
        for (int size = 16; size >= 1 && !h->cluster; size /= 2) {
            const long long L = ((long long)C + size - 1) / size;
            if ((size > 1 && P > L) || L > kClusterCells * kClusterThreads || P > (1 << 15) || cluster_smem((int)L, P) > 220 * 1024) continue;
            cudaLaunchConfig_t lc{};
            cudaLaunchAttribute attr[1];
            lc.gridDim = dim3(size);
            lc.blockDim = dim3(kClusterThreads);
            lc.dynamicSmemBytes = cluster_smem((int)L, P);
            attr[0].id = cudaLaunchAttributeClusterDimension;
            attr[0].val.clusterDim.x = size;
            attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
            lc.attrs = attr;
            lc.numAttrs = 1;
            int most = 0;
            // 220 KB for every handle of the process: the attribute is the kernel's, not the handle's
            if (cudaFuncSetAttribute(k_jacobi_cluster, cudaFuncAttributeMaxDynamicSharedMemorySize, 220 * 1024) == cudaSuccess &&
                cudaOccupancyMaxActiveClusters(&most, k_jacobi_cluster, &lc) == cudaSuccess && most >= 1) {
                h->cluster = size;
                h->cluster_cells = (int)L;
            }
        }
    }
    cudaGetLastError();
    if (ok && cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking) != cudaSuccess) ok = false;
    if (!ok) {
        cudaGetLastError();
        neon_water_destroy(h);
        return wfail(nullptr, NEON_MOE_ECUDA, "device allocation failed");
    }
    h->p_final = h->pa;
    int rc = neon_water_set_particles(h, pos4, nullptr, on_device);
    if (rc) {
        g_water_create_error = h->err;
        neon_water_destroy(h);
        return rc;
    }
    *out = h;
    return NEON_MOE_OK;
}

int neon_water_set_particles(neon_water_handle* h, const float* pos4, const float* vel4, int on_device) {
    if (!h) return NEON_MOE_EINVAL;
    if (!pos4) return wfail(h, NEON_MOE_EINVAL, "null positions");
    WCU(h, cudaSetDevice(h->cfg.device));
    const size_t bytes = (size_t)h->q.N * 16;
    const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    WCU(h, cudaDeviceSynchronize());
    WCU(h, cudaMemcpy(h->pos, pos4, bytes, kind));
    if (vel4) WCU(h, cudaMemcpy(h->vel, vel4, bytes, kind));
    else WCU(h, cudaMemset(h->vel, 0, bytes));
    if (int rc = record_lists(h, nullptr)) return rc;
    WCU(h, cudaDeviceSynchronize());
    return NEON_MOE_OK;
}

int neon_water_step(neon_water_handle* h, int n_steps, void* cuda_stream) {
    if (!h) return NEON_MOE_EINVAL;
    if (n_steps < 0) return wfail(h, NEON_MOE_EINVAL, "negative step count");
    WCU(h, cudaSetDevice(h->cfg.device));
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    h->last_stream = st;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    const bool capturing = cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone;
    cudaGetLastError();
    if (h->use_graphs && !capturing && !h->graph) {
        WCU(h, cudaStreamBeginCapture(h->own_stream, cudaStreamCaptureModeThreadLocal));
        int rc = record_step(h, h->own_stream);
        cudaGraph_t graph = nullptr;
        cudaError_t ce = cudaStreamEndCapture(h->own_stream, &graph);
        if (!rc && ce == cudaSuccess && graph) ce = cudaGraphInstantiate(&h->graph, graph, 0);
        if (graph) cudaGraphDestroy(graph);
        if (rc || ce != cudaSuccess) {
            h->graph = nullptr;
            h->use_graphs = 0;  // capture is not available here: stay eager
            cudaGetLastError();
        }
    }
    for (int i = 0; i < n_steps; ++i) {
        if (h->use_graphs && !capturing && h->graph) {
            WCU(h, cudaGraphLaunch(h->graph, st));
        } else {
            int rc = record_step(h, st);
            if (rc) return rc;
        }
        h->launches += h->launches_per_step;
    }
    return NEON_MOE_OK;
}

int neon_water_step_host(neon_water_handle* h, float* pos4, float* vel4, int n_steps, void* cuda_stream) {
    if (!h) return NEON_MOE_EINVAL;
    if (!pos4 || !vel4) return wfail(h, NEON_MOE_EINVAL, "null particle arrays");
    WCU(h, cudaSetDevice(h->cfg.device));
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    const size_t bytes = (size_t)h->q.N * 16;
    WCU(h, cudaMemcpyAsync(h->pos, pos4, bytes, cudaMemcpyHostToDevice, st));
    WCU(h, cudaMemcpyAsync(h->vel, vel4, bytes, cudaMemcpyHostToDevice, st));
    int rc = record_lists(h, st);
    if (rc) return rc;
    rc = neon_water_step(h, n_steps, st);
    if (rc) return rc;
    WCU(h, cudaMemcpyAsync(pos4, h->pos, bytes, cudaMemcpyDeviceToHost, st));
    WCU(h, cudaMemcpyAsync(vel4, h->vel, bytes, cudaMemcpyDeviceToHost, st));
    WCU(h, cudaStreamSynchronize(st));
    return NEON_MOE_OK;
}

int neon_water_particles_device(neon_water_handle* h, float** pos4, float** vel4) {
    if (!h) return NEON_MOE_EINVAL;
    if (pos4) *pos4 = reinterpret_cast<float*>(h->pos);
    if (vel4) *vel4 = reinterpret_cast<float*>(h->vel);
    return NEON_MOE_OK;
}

int neon_water_read_particles(neon_water_handle* h, float* pos4, float* vel4) {
    if (!h) return NEON_MOE_EINVAL;
    WCU(h, cudaSetDevice(h->cfg.device));
    WCU(h, cudaStreamSynchronize(h->last_stream));
    const size_t bytes = (size_t)h->q.N * 16;
    if (pos4) WCU(h, cudaMemcpy(pos4, h->pos, bytes, cudaMemcpyDeviceToHost));
    if (vel4) WCU(h, cudaMemcpy(vel4, h->vel, bytes, cudaMemcpyDeviceToHost));
    return NEON_MOE_OK;
}

int neon_water_read_grid(neon_water_handle* h, const char* name, void* dst, uint64_t bytes) {
    if (!h || !name || !dst) return NEON_MOE_EINVAL;
    const void* src = nullptr;
    if (!strcmp(name, "u")) src = h->u;
    else if (!strcmp(name, "v")) src = h->v;
    else if (!strcmp(name, "w")) src = h->w;
    else if (!strcmp(name, "pressure")) src = h->p_final;
    else if (!strcmp(name, "density")) src = h->density;
    else if (!strcmp(name, "flags")) src = h->flags;
    else return wfail(h, NEON_MOE_EINVAL, "unknown grid '%s'", name);
    if (bytes > (uint64_t)h->q.C * 4) return wfail(h, NEON_MOE_EINVAL, "'%s' holds %d bytes", name, h->q.C * 4);
    WCU(h, cudaSetDevice(h->cfg.device));
    WCU(h, cudaStreamSynchronize(h->last_stream));
    WCU(h, cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost));
    return NEON_MOE_OK;
}

int neon_water_status(neon_water_handle* h, int* word) {
    if (!h || !word) return NEON_MOE_EINVAL;
    WCU(h, cudaSetDevice(h->cfg.device));
    WCU(h, cudaStreamSynchronize(h->last_stream));
    WCU(h, cudaMemcpy(word, h->bar + 1, sizeof(int), cudaMemcpyDeviceToHost));
    WCU(h, cudaMemset(h->bar + 1, 0, sizeof(int)));
    return *word ? NEON_MOE_EDEVICE : NEON_MOE_OK;
}

int neon_water_profile_step(neon_water_handle* h, double* ms4, void* cuda_stream) {
    if (!h || !ms4) return NEON_MOE_EINVAL;
    WCU(h, cudaSetDevice(h->cfg.device));
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    h->last_stream = st;
    cudaEvent_t ev[5];
    for (auto& e : ev) WCU(h, cudaEventCreate(&e));
    int rc = record_step(h, st, ev);
    cudaError_t ce = cudaStreamSynchronize(st);
    if (!rc && ce == cudaSuccess) {
        for (int i = 0; i < 4; ++i) {
            float t = 0.f;
            cudaEventElapsedTime(&t, ev[i], ev[i + 1]);
            ms4[i] = t;
        }
        h->launches += h->launches_per_step;
    }
    for (auto& e : ev) cudaEventDestroy(e);
    if (rc) return rc;
    if (ce != cudaSuccess) return wfail(h, NEON_MOE_ECUDA, "profile step: %s", cudaGetErrorString(ce));
    return NEON_MOE_OK;
}

int neon_water_set_option(neon_water_handle* h, const char* name, int64_t value) {
    if (!h || !name) return NEON_MOE_EINVAL;
    if (!strcmp(name, "use_graphs")) {
        h->use_graphs = (int)value;
        if (!value && h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    } else if (!strcmp(name, "fused_jacobi")) {
        h->fused_jacobi = (int)value;
        if (h->graph) { cudaGraphExecDestroy(h->graph); h->graph = nullptr; }
    } else {
        return wfail(h, NEON_MOE_EINVAL, "unknown option '%s'", name);
    }
    return NEON_MOE_OK;
}

}  // extern "C"
