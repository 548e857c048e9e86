// A layer pass of ONE token as three kernels that stream its experts' weights through a small ring of shared memory per
// warp.
//
// At one token the layer is a stream over top_k experts' weights (53 MB at the 20b shape, 8 us at the HBM rate); what
// counts is how early and how evenly it runs.  The one-launch kernel (decode_fused.cuh) hands partial sums across the
// grid three times, the grouped GEMM needs seven launches; here
//
//   route     one cluster: router dot products, top k, softmax, the selected experts, and the hidden state as f16;
//   gate_up   an item is 32 weight rows (16 gate rows and their 16 linear rows) of one expert over the whole depth: 720
//             equal items at the 20b shape, five per SM, and no partial sum leaves a CTA; its four warps share the
//             depth.  The epilogue applies bias and SwiGLU and writes the down product's operand;
//   down      a CTA owns 16 output rows of ALL experts, its warps share the flat sequence of (expert, 128-column chunk)
//             steps; weighting, bias and the sum over the experts happen in the CTA: no combine pass.
//
// The product runs on mma.sync.m16n8k16 (f16 x f16, f32 accumulation): 8 columns are plenty for one token, where tcgen05
// would need 128-row tiles in shared memory and a trip through tensor memory.  e2m1 codes become f16 exactly, by one
// conversion instruction per two codes.  A lane holds 16 bytes: the 32 codes of ONE row in ONE scale block; the four lanes
// of a row hold the four blocks of a 128-column chunk.  So that each block keeps a sum of its own (its scale is a factor
// of that sum, not of the operands), the token occupies four columns, one per block, and lane t supplies its values only
// to column t: the other three columns multiply by zero.  Scales are then one f32 multiply-add per row, block and chunk.
//
// Precision.  The hidden state is bf16, scaled by one power of two so that its largest value lies in [2^14, 2^15): f16
// holds it exactly down to 2^-28 of the largest (and to 2^-39 of it absolutely).  The f32 SwiGLU outputs enter the down
// product as two f16 terms (22 bits), in columns 0-3 and 4-7.  Sums are f32 throughout.
//
// Measured per pass at the 20b shape: 27.6 to 28.0 us, one launch 36.2, seven launches 37.9 (128 experts: 34.4, 40.3, 45.8).
// From two tokens on the grouped GEMM wins (two: 49.9 here against 46.1; eight: 148 against 72): a step's 300
// instructions are a chain that 20 warps per SM do not hide at more bytes per SM (ncu: 1.9 instructions per clock, 54 % of
// the DRAM rate), so the rule is one token.
#pragma once
#include <cuda_fp16.h>

#include "decode_fused.cuh"

namespace neon {

constexpr int kStrCluster = 8;     // CTAs of the routing cluster (the portable size)
constexpr int kStrRouteThreads = 1024;
constexpr int kStrSlicesMax = 8;   // K slices of a router dot product
constexpr int kStrGuWarps = 4, kStrDnWarps = 16;
constexpr float kStrLoScale = 2048.f;  // the second f16 term holds the remainder times 2^11

struct StreamTables {  // written by the routing kernel
    int exp[kMaxTopK];   // expert of every slot
    float w[kMaxTopK];   // its routing weight
    float x_scale;       // power of two that undoes the hidden state's scaling
};

struct StreamParams {
    const uint16_t *x, *wr, *br;
    const float* logit_bias;
    int H, I, E, k, kp_h, kp_i, dn_tiles;
    float limit, alpha;
    const uint8_t *gu_w, *gu_sfa, *dn_w, *dn_sfa;
    const uint16_t *gu_bias, *dn_bias;
    int n_slices;
    float a_inv;       // power of two that scales SwiGLU outputs into f16's range
    __half* xt;        // [kp_h]
    __half* at;        // [slot][2 terms][kp_i]
    StreamTables* tab;
    float* out;
    int32_t* idx;
    float* route_w;
    DispatchArrays d;
};

// 8 e2m1 codes -> 8 f16, in column order
__device__ __forceinline__ void unpack_f16(uint32_t w, uint32_t (&r)[4]) {
    asm("{\n\t.reg .b8 b0, b1, b2, b3;\n\tmov.b32 {b0, b1, b2, b3}, %4;\n\t"
        "cvt.rn.f16x2.e2m1x2 %0, b0;\n\tcvt.rn.f16x2.e2m1x2 %1, b1;\n\tcvt.rn.f16x2.e2m1x2 %2, b2;\n\tcvt.rn.f16x2.e2m1x2 %3, b3;\n\t}"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
        : "r"(w));
}
// two E8M0 bytes -> their f32 values
__device__ __forceinline__ float2 unpack_scales(uint32_t two) {
    uint32_t r;
    asm("cvt.rn.bf16x2.ue8m0x2 %0, %1;" : "=r"(r) : "h"((uint16_t)two));
    return make_float2(__uint_as_float(r << 16), __uint_as_float(r & 0xffff0000u));
}
__device__ __forceinline__ void mma_f16_16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void copy16(unsigned dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy4(unsigned dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copy_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// One 16-row tile of a chunk times the eight columns: rows g and g + 8 (a lane's 16 bytes of each), two chains of products.
__device__ __forceinline__ void tile_mma(float (&c)[4], const uint4& ra, const uint4& rb, const uint4 (&b)[4]) {
    const uint32_t wa[4] = {ra.x, ra.y, ra.z, ra.w}, wb[4] = {rb.x, rb.y, rb.z, rb.w};
    float d[4] = {0.f, 0.f, 0.f, 0.f};
    c[0] = c[1] = c[2] = c[3] = 0.f;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        uint32_t fa[4], fb[4];
        unpack_f16(wa[j], fa);
        unpack_f16(wb[j], fb);
        mma_f16_16816(c, fa[0], fb[0], fa[1], fb[1], b[j].x, b[j].y);
        mma_f16_16816(d, fa[2], fb[2], fa[3], fb[3], b[j].z, b[j].w);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) c[i] += d[i];
}

// A warp's ring: what one step (a 128-column chunk of its weight rows) needs, several steps deep.  Weights: TILES 16-row
// tiles, for each rows g and g + 8 of lane (g, t) 16 bytes - every lane copies what it will read itself; one word of four
// scales per row; the 128 f16 of the token's TERMS terms.  Deep enough that an SM keeps 120 KB (gate_up, five CTAs) and
// 50 to 100 KB (down, one or two CTAs) of weights in flight: 2 us at its share of the HBM rate need 90 KB.
template <int TILES, int TERMS>
struct StreamRing {
    static constexpr int kScales = TILES * 1024, kRows = kScales + TILES * 64, kStage = kRows + TERMS * 256;
};
constexpr int kStrGuStages = 4, kStrDnStages = 4;
constexpr int kStrGuSmem = kStrGuWarps * kStrGuStages * StreamRing<2, 1>::kStage, kStrDnSmem = kStrDnWarps * kStrDnStages * StreamRing<1, 2>::kStage;

// ---- routing ------------------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(kStrRouteThreads) stream_route_kernel(const StreamParams p) {
    __shared__ float part[kMaxExperts * kStrSlicesMax], lg[kMaxExperts];  // CTA 0: the shares of the logits, the logits
    __shared__ unsigned amax;
    __shared__ int s_idx[kMaxTopK];
    __shared__ float s_w[kMaxTopK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int H = p.H, E = p.E, k = p.k, nvec = H / 8;
    unsigned rank;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(rank));
    pdl_launch_dependents();
    if (tid == 0) amax = 0u;
    unsigned remote;
    asm("mapa.shared::cluster.u32 %0, %1, 0;" : "=r"(remote) : "r"((unsigned)__cvta_generic_to_shared(part)));
    // (the barrier: everybody has started, remote stores may go out); the router weights of the first unit are on their
    // way before the predecessor has finished
    const int vps = (nvec + p.n_slices - 1) / p.n_slices, units = E * p.n_slices, step = kStrCluster * (kStrRouteThreads / 32);
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    int unit = (int)rank * (kStrRouteThreads / 32) + warp;
    auto wrow = [&](int u, int i) {
        const int v = (u / E) * vps + i * 32 + lane, v1 = min(nvec, (u / E + 1) * vps);
        return v < v1 ? __ldg(reinterpret_cast<const uint4*>(p.wr + (size_t)(u % E) * H) + v) : make_uint4(0u, 0u, 0u, 0u);
    };
    uint4 wv = unit < units ? wrow(unit, 0) : make_uint4(0u, 0u, 0u, 0u);
    pdl_wait();
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    for (; unit < units; unit += step) {
        const int e = unit % E, sl = unit / E, v0 = sl * vps, v1 = min(nvec, v0 + vps);
        float acc = 0.f;
        for (int i = 0; v0 + i * 32 < v1; ++i) {
            const int v = v0 + i * 32 + lane;
            const uint4 xv = v < v1 ? __ldcg(reinterpret_cast<const uint4*>(p.x) + v) : make_uint4(0u, 0u, 0u, 0u);
            const uint4 nw = wrow(unit, i + 1);
            const uint32_t wa[4] = {wv.x, wv.y, wv.z, wv.w}, xa[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc = fmaf(__uint_as_float(xa[j] << 16), __uint_as_float(wa[j] << 16), acc);
                acc = fmaf(__uint_as_float(xa[j] & 0xffff0000u), __uint_as_float(wa[j] & 0xffff0000u), acc);
            }
            wv = nw;
        }
        if (unit + step < units) wv = wrow(unit + step, 0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(remote + (unsigned)((e * p.n_slices + sl) * 4)), "f"(acc) : "memory");
    }
    asm volatile("barrier.cluster.arrive.release;" ::: "memory");
    // meanwhile, in the last CTA: the hidden state as f16
    if (rank == kStrCluster - 1) {
        const uint4* xr = reinterpret_cast<const uint4*>(p.x);
        unsigned m = 0u;
        for (int v = tid; v < nvec; v += kStrRouteThreads) {
            const uint4 xv = __ldcg(xr + v);
            const uint32_t a[4] = {xv.x, xv.y, xv.z, xv.w};
#pragma unroll
            for (int j = 0; j < 4; ++j) m = max(m, max(a[j] & 0x7fffu, (a[j] >> 16) & 0x7fffu));
        }
        m = __reduce_max_sync(0xffffffffu, m);
        if (lane == 0 && m) atomicMax(&amax, m);
        __syncthreads();
        // exponent field of the factor: the largest value goes to [2^14, 2^15); kept where it and its inverse are normal
        const int ef = (int)(amax >> 7), inv_f = amax ? min(max(268 - ef, 1), 253) : 127;
        const float inv = __uint_as_float((uint32_t)inv_f << 23);
        if (tid == 0) p.tab->x_scale = __uint_as_float((uint32_t)(254 - inv_f) << 23);
        for (int v = tid; v < nvec; v += kStrRouteThreads) {
            const uint4 xv = __ldcg(xr + v);
            const uint32_t a[4] = {xv.x, xv.y, xv.z, xv.w};
            uint32_t o[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const __half2 h = __floats2half2_rn(__uint_as_float(a[j] << 16) * inv, __uint_as_float(a[j] & 0xffff0000u) * inv);
                o[j] = *reinterpret_cast<const uint32_t*>(&h);
            }
            *reinterpret_cast<uint4*>(p.xt + v * 8) = make_uint4(o[0], o[1], o[2], o[3]);
        }
    }
    asm volatile("barrier.cluster.wait.acquire;" ::: "memory");
    if (rank) return;
    for (int e = tid; e < E; e += kStrRouteThreads) {
        float v = part[e * p.n_slices];
        for (int i = 1; i < p.n_slices; ++i) v += part[e * p.n_slices + i];
        v += bf16_bits_to_float(p.br[e]);
        if (p.logit_bias) v += p.logit_bias[e];
        lg[e] = v;
    }
    __syncthreads();
    if (warp == 0) topk_warp(lg, E, k, lane, s_idx, s_w);
    __syncthreads();
    if (tid < k) {
        const int e = s_idx[tid];
        int pos = 0;  // place in the order of expert ids
        for (int s = 0; s < k; ++s) pos += s_idx[s] < e;
        p.tab->exp[tid] = e;
        p.tab->w[tid] = s_w[tid];
        p.idx[tid] = e;
        p.route_w[tid] = s_w[tid];
        p.d.perm[pos] = tid;
        p.d.inv[tid] = pos;
    }
    for (int e = tid - 32; e >= 0 && e <= E; e += kStrRouteThreads - 32) {  // histogram and offsets, as the dispatch kernels write them
        int c = 0, below = 0;
        for (int s = 0; s < k; ++s) {
            c += s_idx[s] == e;
            below += s_idx[s] < e;
        }
        if (e < E) p.d.count[e] = c;
        p.d.offset[e] = below;
    }
}

__device__ __forceinline__ void load_tables(StreamTables* tab, const StreamTables* src) {
    for (int i = threadIdx.x; i < (int)(sizeof(StreamTables) / 4); i += blockDim.x) reinterpret_cast<int*>(tab)[i] = __ldcg(reinterpret_cast<const int*>(src) + i);
}

// ---- gate_up ------------------------------------------------------------------------------------------------------
// Item = (slot, weight tile m, quarter q): gate channels 64 m + 16 q + 0..15 and their linear rows, 2 KB in a row of every
// weight box.
__global__ void __launch_bounds__(kStrGuWarps * 32, 5) stream_gate_up_kernel(const StreamParams p) {
    constexpr int D = kStrGuStages;
    using Ring = StreamRing<2, 1>;
    extern __shared__ __align__(128) unsigned char ring_mem[];
    __shared__ StreamTables tab;
    __shared__ float red[kStrGuWarps][2][16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int n_chunks = p.kp_h / kChunkK, m_tiles = 2 * p.I / 128, per_exp = m_tiles * 4, n_items = p.k * per_exp;
    const int c0 = warp * n_chunks / kStrGuWarps, c1 = (warp + 1) * n_chunks / kStrGuWarps;
    unsigned char* ring = ring_mem + (size_t)warp * D * Ring::kStage;
    const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
    pdl_wait();
    pdl_launch_dependents();  // the routing is complete: a down CTA that starts early may already read it
    load_tables(&tab, p.tab);
    __syncthreads();
    // the next step to copy: item, chunk, ring stage, and this lane's addresses
    int p_item = c0 < c1 ? (int)blockIdx.x : n_items, p_c = c0, p_s = 0;
    const uint8_t *pw = nullptr, *ps = nullptr;
    const __half* px = nullptr;
    auto start_item = [&]() {
        if (p_item >= n_items) return;
        const int s = p_item / per_exp, rem = p_item - s * per_exp, m = rem >> 2, q = rem & 3;
        const size_t box = ((size_t)tab.exp[s] * m_tiles + m) * n_chunks + c0;
        pw = p.gu_w + box * 8192 + (q * 32 + g) * 64 + t * 16;
        ps = p.gu_sfa + box * 512 + lane * 16 + q * 4;
        px = p.xt + c0 * kChunkK + lane * 8;
    };
    start_item();
    auto copy_next = [&]() {
        if (p_item < n_items) {
            const unsigned dst = ring_at + (unsigned)(p_s * Ring::kStage);
#pragma unroll
            for (int r = 0; r < 4; ++r) copy16(dst + r * 512 + lane * 16, pw + r * 512);  // rows g, g + 8 of the gate tile, then of the linear tile
            copy4(dst + Ring::kScales + lane * 4, ps);
            if (lane < 16) copy16(dst + Ring::kRows + lane * 16, px);
            pw += 8192;
            ps += 512;
            px += kChunkK;
            if (++p_s == D) p_s = 0;
            if (++p_c == c1) { p_c = c0; p_item += gridDim.x; start_item(); }
        }
        copy_commit();
    };
#pragma unroll
    for (int i = 0; i < D - 1; ++i) copy_next();
    int stage = 0;
    const bool feeds = g == t;  // this lane supplies its column's values (columns 4..7 stay empty)
    // every warp of the CTA walks the same items and meets the others at each one's end
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        float acc[2][2] = {{0.f, 0.f}, {0.f, 0.f}};  // [tile][row g, g + 8]
#pragma unroll 1
        for (int c = c0; c < c1; ++c) {
            __syncwarp();  // the stage that is copied into next has been read by every lane
            copy_next();
            copy_wait<D - 1>();
            __syncwarp();
            const unsigned char* st = ring + stage * Ring::kStage;
            if (++stage == D) stage = 0;
            uint4 w[4], b[4];
            uint32_t sw[4];
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                w[r] = *reinterpret_cast<const uint4*>(st + r * 512 + lane * 16);
                sw[r] = *reinterpret_cast<const uint16_t*>(st + Ring::kScales + (r * 8 + g) * 4 + 2 * (t & 1));
                b[r] = make_uint4(0u, 0u, 0u, 0u);
                if (feeds) b[r] = *reinterpret_cast<const uint4*>(st + Ring::kRows + t * 64 + r * 16);
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {  // this lane's columns 2 t, 2 t + 1: blocks 2 t, 2 t + 1 (t < 2)
                float v[4];
                tile_mma(v, w[2 * i], w[2 * i + 1], b);
                const float2 s0 = unpack_scales(sw[2 * i]), s1 = unpack_scales(sw[2 * i + 1]);
                acc[i][0] = fmaf(v[1], s0.y, fmaf(v[0], s0.x, acc[i][0]));
                acc[i][1] = fmaf(v[3], s1.y, fmaf(v[2], s1.x, acc[i][1]));
            }
        }
        // ---- the warps' shares of the depth, bias, SwiGLU, the down product's operand
        const int s = item / per_exp, rem = item - s * per_exp, m = rem >> 2, q = rem & 3, e = tab.exp[s];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const float sum = acc[i][j] + __shfl_xor_sync(0xffffffffu, acc[i][j], 1);
                if (t == 0) red[warp][i][g + 8 * j] = sum;
            }
        __syncthreads();
        if (tid < 16) {
            const int ch = 64 * m + 16 * q + tid;
            float gate = ((red[0][0][tid] + red[1][0][tid]) + red[2][0][tid]) + red[3][0][tid];
            float lin = ((red[0][1][tid] + red[1][1][tid]) + red[2][1][tid]) + red[3][1][tid];
            const uint32_t bias = __ldg(reinterpret_cast<const uint32_t*>(p.gu_bias + (size_t)e * 2 * p.I) + ch);  // gate row 2 ch, linear row 2 ch + 1
            gate = fmaf(gate, tab.x_scale, __uint_as_float(bias << 16));
            lin = fmaf(lin, tab.x_scale, __uint_as_float(bias & 0xffff0000u));
            const float gg = fminf(gate, p.limit), ll = fminf(fmaxf(lin, -p.limit), p.limit);
            const float a = gg / (1.f + expf(-p.alpha * gg)) * (ll + 1.f) * p.a_inv;
            const __half hi = __float2half_rn(a);
            __half* dst = p.at + (size_t)s * 2 * p.kp_i + ch;
            dst[0] = hi;
            dst[p.kp_i] = __float2half_rn((a - __half2float(hi)) * kStrLoScale);
        }
        __syncthreads();
    }
}

// ---- down ---------------------------------------------------------------------------------------------------------
// CTA = (weight tile m, i8): output rows 128 m + 16 i8 + 0..15, 1 KB in a row of every weight box.
__global__ void __launch_bounds__(kStrDnWarps * 32, 2) stream_down_kernel(const StreamParams p) {
    constexpr int D = kStrDnStages;
    using Ring = StreamRing<1, 2>;
    extern __shared__ __align__(128) unsigned char ring_mem[];
    __shared__ StreamTables tab;
    __shared__ float sum[kStrDnWarps][16];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    const int n_chunks = p.kp_i / kChunkK, m = blockIdx.x >> 3, i8 = blockIdx.x & 7;
    const int total = p.k * n_chunks, s0 = warp * total / kStrDnWarps, s1 = (warp + 1) * total / kStrDnWarps;
    unsigned char* ring = ring_mem + (size_t)warp * D * Ring::kStage;
    const unsigned ring_at = (unsigned)__cvta_generic_to_shared(ring);
    // launched when the gate_up kernel's CTAs have all seen the routing complete: the tables and the weights may be read
    // before that kernel ends
    load_tables(&tab, p.tab);
    if (tid < kStrDnWarps * 16) (&sum[0][0])[tid] = 0.f;
    __syncthreads();
    auto copy_weights = [&](int s, int st) {
        const int slot = s / n_chunks, c = s - slot * n_chunks;
        const size_t box = ((size_t)tab.exp[slot] * p.dn_tiles + m) * n_chunks + c;
        const unsigned dst = ring_at + (unsigned)(st * Ring::kStage);
        const uint8_t* w = p.dn_w + box * 8192 + (16 * i8 + g) * 64 + t * 16;
        copy16(dst + lane * 16, w);
        copy16(dst + 512 + lane * 16, w + 512);
        if (lane < 16)  // scale word of tile row 16 i8 + lane
            copy4(dst + Ring::kScales + lane * 4, p.dn_sfa + box * 512 + (16 * (i8 & 1) + lane) * 16 + (i8 >> 1) * 4);
    };
    auto copy_rows = [&](int s, int st) {  // 16 lanes copy the chunk of one term, 16 of the other
        const int slot = s / n_chunks, c = s - slot * n_chunks;
        copy16(ring_at + (unsigned)(st * Ring::kStage) + Ring::kRows + lane * 16, p.at + ((size_t)slot * 2 + (lane >> 4)) * p.kp_i + c * kChunkK + (lane & 15) * 8);
    };
#pragma unroll 1
    for (int i = 0; i < D - 1; ++i)
        if (s0 + i < s1) copy_weights(s0 + i, i);
    pdl_wait();
    pdl_launch_dependents();
#pragma unroll 1
    for (int i = 0; i < D - 1; ++i) {
        if (s0 + i < s1) copy_rows(s0 + i, i);
        copy_commit();
    }
    float acc[2] = {0.f, 0.f};
    // term of this lane's accumulator columns 2 t, 2 t + 1, and the factor that undoes the operand's scaling
    const float factor = (t >> 1 ? 1.f / kStrLoScale : 1.f) / p.a_inv;
    const bool feeds = t == (g & 3);  // this lane supplies its column's values: term g / 4, block g % 4
    int stage = 0, ahead = D - 1;
#pragma unroll 1
    for (int s = s0; s < s1; ++s) {
        __syncwarp();  // the stage that is copied into next has been read by every lane
        if (s + D - 1 < s1) { copy_weights(s + D - 1, ahead); copy_rows(s + D - 1, ahead); }
        copy_commit();
        if (++ahead == D) ahead = 0;
        copy_wait<D - 1>();
        __syncwarp();
        const unsigned char* st = ring + stage * Ring::kStage;
        if (++stage == D) stage = 0;
        const uint4 wa = *reinterpret_cast<const uint4*>(st + lane * 16), wb = *reinterpret_cast<const uint4*>(st + 512 + lane * 16);
        uint4 b[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            b[j] = make_uint4(0u, 0u, 0u, 0u);
            if (feeds) b[j] = *reinterpret_cast<const uint4*>(st + Ring::kRows + (g >> 2) * 256 + t * 64 + j * 16);
        }
        float v[4];
        tile_mma(v, wa, wb, b);
        const float2 sa = unpack_scales(*reinterpret_cast<const uint16_t*>(st + Ring::kScales + g * 4 + 2 * (t & 1)));
        const float2 sb = unpack_scales(*reinterpret_cast<const uint16_t*>(st + Ring::kScales + (g + 8) * 4 + 2 * (t & 1)));
        acc[0] = fmaf(v[1], sa.y, fmaf(v[0], sa.x, acc[0]));
        acc[1] = fmaf(v[3], sb.y, fmaf(v[2], sb.x, acc[1]));
        if ((s + 1) % n_chunks == 0 || s + 1 == s1) {  // the warp's share of this expert, weighted, into its own sums
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float x = acc[r] * factor;
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                x += __shfl_xor_sync(0xffffffffu, x, 2);
                if (t == 0) sum[warp][g + 8 * r] += tab.w[s / n_chunks] * x;
                acc[r] = 0.f;
            }
        }
    }
    __syncthreads();
    if (tid < 16) {
        const int row = 128 * m + 16 * i8 + tid;
        if (row < p.H) {
            float v = 0.f;
#pragma unroll
            for (int x = 0; x < kStrDnWarps; ++x) v += sum[x][tid];
            for (int s = 0; s < p.k; ++s) v = fmaf(tab.w[s], bf16_bits_to_float(p.dn_bias[(size_t)tab.exp[s] * p.H + row]), v);
            p.out[row] = v;
        }
    }
}

}  // namespace neon
