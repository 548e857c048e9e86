// The reference engine's denoiser (NeonEngine/shaders/raytracing_pp.comp: temporal accumulation;
// NeonEngine/shaders/raytracing_atrous.comp: edge-avoiding a-trous filter) as CUDA kernels behind
// the C ABI of include/neon_svgf.h, scheduled per frame as NeonEngine/src/raytracing_app.cpp:735-765
// and NeonEngine/src/raytracing_rast.cpp:325-428 schedule the two shaders.  This translation unit is
// compiled with -fmad=false: every kernel uses the shaders' 32-bit float operations in the shaders'
// order (the only fused multiply-adds are the explicit ones of exp2_poly), so the results equal the
// CPU restatement bit for bit.  No CPU fallback exists.
//
// Redesign relative to the shaders (results unchanged):
//  * the moments image is held as two planes, {history length, second moment} and {first moment,
//    variance}, each double-buffered, so a pass never reads what it writes (the shaders update the
//    image in place while neighbours read it) and the filter moves only the plane it changes;
//  * every filter pass reads one of the two history images, none reads the storage image: what all
//    but the last pass write there is overwritten unseen, so only the last pass sums colours;
//  * the temporal pass leaves {normal, depth} as one 16-byte vector per pixel for the filter's taps;
//  * the copy of the storage image into the history image (the shaders' "iteration 98" dispatch) is
//    done by the last filter pass itself whenever that pass does not read the image being replaced
//    (always the case for an odd iteration count, the reference's 3);
//  * one frame is a CUDA graph.
#include "../../include/neon_svgf.h"

#include <cuda_fp16.h>
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdio>
#include <cstring>
#include <memory>
#include <new>
#include <string>
#include <vector>

namespace {

__device__ __forceinline__ float dot3(float ax, float ay, float az, float bx, float by, float bz) { return ax * bx + ay * by + az * bz; }
__device__ __forceinline__ float len3(float x, float y, float z) { return sqrtf(x * x + y * y + z * z); }
__device__ __forceinline__ float max_glsl(float a, float b) { return a < b ? b : a; }
__device__ __forceinline__ float min_glsl(float a, float b) { return b < a ? b : a; }
__device__ __forceinline__ float mixf(float x, float y, float a) { return x * (1.0f - a) + y * a; }

// Two floats in one 64-bit register: one instruction works on both, each rounded as the scalar operation rounds it.
// The assembler contracts a packed multiplication and the packed addition of its result into one fused operation, .rn
// and -fmad=false notwithstanding; a product that is added is therefore formed as a fused multiply-add of -0 (the same
// value, and nothing left to fuse), the -0 coming from a kernel argument so that it is not folded away.
using F2 = unsigned long long;
constexpr F2 kNegZero2 = 0x8000000080000000ull;
__device__ __forceinline__ F2 pack2(float a, float b) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void unpack2(F2 v, float& a, float& b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v)); }
__device__ __forceinline__ F2 add2(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 mul2(F2 a, F2 b) {
    F2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
// max_glsl(v, 0) up to the sign of a zero: a NaN stays a NaN
__device__ __forceinline__ float max0_nan(float v) {
    float r;
    asm("max.NaN.f32 %0, %1, 0f00000000;" : "=f"(r) : "f"(v));
    return r;
}

// 2^x for two x <= 0 (or NaN): nearest-integer split, degree-7 polynomial of 2^f on [-0.5, 0.5], exact scaling by 2^n;
// 0 for x <= -126.  The nearest integer (ties to even) comes from adding and subtracting 1.5 * 2^23, whose sum also
// carries that integer in its low mantissa bits: two additions on the main pipes instead of a rounding and a
// conversion instruction, same values.
__device__ __forceinline__ F2 exp2_poly2(F2 x) {
    const F2 shifted = add2(x, pack2(12582912.0f, 12582912.0f));
    const F2 n = add2(shifted, pack2(-12582912.0f, -12582912.0f));
    const F2 f = fma2(n, pack2(-1.0f, -1.0f), x);  // x - n: the product is exact
    F2 p = pack2(1.5252734e-5f, 1.5252734e-5f);
    p = fma2(p, f, pack2(1.5403530e-4f, 1.5403530e-4f));
    p = fma2(p, f, pack2(1.3333558e-3f, 1.3333558e-3f));
    p = fma2(p, f, pack2(9.6181291e-3f, 9.6181291e-3f));
    p = fma2(p, f, pack2(5.5504109e-2f, 5.5504109e-2f));
    p = fma2(p, f, pack2(2.4022651e-1f, 2.4022651e-1f));
    p = fma2(p, f, pack2(6.9314718e-1f, 6.9314718e-1f));
    p = fma2(p, f, pack2(1.0f, 1.0f));
    float x0, x1, s0, s1;
    unpack2(x, x0, x1);
    unpack2(shifted, s0, s1);
    // (n + 127) << 23 with n = bits(shifted) - bits(1.5 * 2^23), whose low nine bits are zero
    const F2 scale = pack2(__uint_as_float((__float_as_uint(s0) << 23) + 0x3F800000u), __uint_as_float((__float_as_uint(s1) << 23) + 0x3F800000u));
    float r0, r1;
    unpack2(mul2(p, scale), r0, r1);
    return pack2(x0 <= -126.0f ? 0.0f : r0, x1 <= -126.0f ? 0.0f : r1);
}

__device__ __forceinline__ unsigned to_unorm8(float v) {
    if (v != v) v = 0.0f;
    v = v < 0.0f ? 0.0f : (v > 1.0f ? 1.0f : v);
    return (unsigned)__float2int_rn(v * 255.0f);
}
__device__ __forceinline__ uchar4 pack_rgb8(float r, float g, float b) {
    return make_uchar4((unsigned char)to_unorm8(r), (unsigned char)to_unorm8(g), (unsigned char)to_unorm8(b), 255);
}
__device__ __forceinline__ float3 load_rgb16(const uint2* __restrict__ im, size_t i) {
    const uint2 v = __ldg(im + i);
    const __half2 lo = *reinterpret_cast<const __half2*>(&v.x), hi = *reinterpret_cast<const __half2*>(&v.y);
    return make_float3(__low2float(lo), __high2float(lo), __low2float(hi));
}
__device__ __forceinline__ uint2 pack_rgba16(float r, float g, float b, float a) {
    const __half2 lo = __halves2half2(__float2half_rn(r), __float2half_rn(g)), hi = __halves2half2(__float2half_rn(b), __float2half_rn(a));
    uint2 v;
    v.x = *reinterpret_cast<const unsigned*>(&lo);
    v.y = *reinterpret_cast<const unsigned*>(&hi);
    return v;
}

struct Frame {  // the caller's images of one frame
    const float4 *pos, *nrm, *bary, *mot;
    uchar4* image;
};

constexpr int kBlockX = 32, kBlockY = 8;

// ---- temporal accumulation (raytracing_pp.comp:35-247, display mode 5) ---------------------------
// a = {history length, second moment}, b = {first moment, variance}.  Also leaves what the filter passes read of the
// G-buffer: guide = {normal, depth} and whether the pixel shows a surface.
__global__ void __launch_bounds__(kBlockX* kBlockY) k_temporal(int w, int h, Frame fr, const uint2* __restrict__ hist_prev,
                                                               uint2* __restrict__ hist_next, const float2* __restrict__ a_in,
                                                               const float2* __restrict__ b_in, float2* __restrict__ a_out,
                                                               float2* __restrict__ b_out, float4* __restrict__ guide,
                                                               uint8_t* __restrict__ surface) {
    const int x = blockIdx.x * kBlockX + threadIdx.x, y = blockIdx.y * kBlockY + threadIdx.y;
    if (x >= w || y >= h) return;
    const size_t idx = (size_t)y * w + x;
    const uchar4 c8 = fr.image[idx];
    const float cr = c8.x / 255.0f, cg = c8.y / 255.0f, cb = c8.z / 255.0f;

    // LoadPreviousData (raytracing_pp.comp:35-140)
    float pr = 0.0f, pg = 0.0f, pb = 0.0f, hl = 0.0f, pm0 = 0.0f, pm1 = 0.0f;
    bool ok = false;
    const float4 cp = __ldg(fr.pos + idx), cn = __ldg(fr.nrm + idx);
    const bool none = dot3(cp.x, cp.y, cp.z, cp.x, cp.y, cp.z) < 1e-6f;
    if (!none) {
        const float4 cbary = __ldg(fr.bary + idx), m = __ldg(fr.mot + idx);
        const int cur_mesh = (int)roundf(cn.w);
        const float uvx = ((float)x + 0.5f) / (float)w, uvy = ((float)y + 0.5f) / (float)h;
        const float pux = uvx - m.x, puy = uvy - m.y;
        if (!(pux < 0.0f || puy < 0.0f || pux > 1.0f || puy > 1.0f)) {
            const float ppx = pux * (float)w - 0.5f, ppy = puy * (float)h - 0.5f;
            const float flx = floorf(ppx), fly = floorf(ppy);
            const int bx = (int)flx, by = (int)fly;
            const float fx = ppx - flx, fy = ppy - fly;
            const float weights[4] = {(1.0f - fx) * (1.0f - fy), fx * (1.0f - fy), (1.0f - fx) * fy, fx * fy};
            const float dist = len3(cp.x, cp.y, cp.z);
            const float pos_threshold = max_glsl(0.01f * dist, 0.005f);
            float ar = 0.0f, ag = 0.0f, ab = 0.0f, ah = 0.0f, am0 = 0.0f, am1 = 0.0f, aw = 0.0f;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int tx = bx + (i & 1), ty = by + (i >> 1);
                if (tx < 0 || ty < 0 || tx >= w || ty >= h) continue;
                const size_t t = (size_t)ty * w + tx;
                const float4 tp = __ldg(fr.pos + t);
                if (dot3(tp.x, tp.y, tp.z, tp.x, tp.y, tp.z) < 1e-6f) continue;
                const float4 tn = __ldg(fr.nrm + t);
                if (cur_mesh != (int)roundf(tn.w)) continue;
                const float tap_depth = len3(tp.x, tp.y, tp.z);
                if (fabsf(dist - tap_depth) > 0.02f * dist) continue;
                if (len3(cp.x - tp.x, cp.y - tp.y, cp.z - tp.z) > pos_threshold) continue;
                if (dot3(cn.x, cn.y, cn.z, tn.x, tn.y, tn.z) < 0.9f) continue;
                const float4 tb = __ldg(fr.bary + t);
                if (len3(cbary.x - tb.x, cbary.y - tb.y, cbary.z - tb.z) > 0.2f) continue;
                const float wt = weights[i];
                const float3 hc = load_rgb16(hist_prev, t);
                ar += hc.x * wt; ag += hc.y * wt; ab += hc.z * wt;
                const float2 ta = __ldg(a_in + t);
                ah += ta.x * wt;
                am0 += __ldg(&b_in[t].x) * wt;
                am1 += ta.y * wt;
                aw += wt;
            }
            if (!(aw < 0.5f)) {
                const float inv = 1.0f / aw;
                pr = ar * inv; pg = ag * inv; pb = ab * inv;
                hl = ah * inv;
                pm0 = am0 * inv;
                pm1 = am1 * inv;
                ok = true;
            }
        }
    }
    float alpha;
    if (ok) {
        hl = hl + 1.0f;
        alpha = 1.0f / hl;
        alpha = min_glsl(max_glsl(alpha, 0.0f), 1.0f);
    } else {
        alpha = 1.0f;
        hl = 1.0f;
    }
    const float br = ok ? pr : cr, bg = ok ? pg : cg, bb = ok ? pb : cb;
    const float nr = mixf(br, cr, alpha), ng = mixf(bg, cg, alpha), nb = mixf(bb, cb, alpha);
    float m0 = 0.2126f * cr + 0.7152f * cg + 0.0722f * cb;
    float m1 = m0 * m0;
    m0 = mixf(pm0, m0, alpha);
    m1 = mixf(pm1, m1, alpha);
    const float variance = max_glsl(0.0f, m1 - m0 * m0);
    hist_next[idx] = pack_rgba16(nr, ng, nb, 1.0f);
    a_out[idx] = make_float2(hl, m1);
    b_out[idx] = make_float2(m0, variance);
    guide[idx] = make_float4(cn.x, cn.y, cn.z, cp.z);
    surface[idx] = none ? 0 : 1;
}

// ---- a-trous filter pass (raytracing_atrous.comp:59-160, iteration < 98) -------------------------
// One CTA filters a tile of 32 x 16 pixels from shared memory, where the tile and its halo of two steps on each side
// lie with the image's edges already repeated; a thread filters two pixels eight rows apart, so that everything after
// the differences of a tap is one packed instruction for both.  Bound by instruction issue (25 taps of about 40
// instructions; issue slots 68 to 73 % active, the multiply-add pipe 41 %); a 1080p frame with 3 passes takes 332 us
// against 558 us with one pixel a thread, separate taps of 44 bytes through L1 and colours summed in every pass.  STEP 0:
// any step, taps from global memory (steps beyond 8, whose halo no longer fits).
// LAST: also the colour sums, the storage image and (copy_to != nullptr) its conversion back to floats in that
// history image (the shaders' separate copy dispatch, raytracing_atrous.comp:66-70).
constexpr int kTileX = 32, kTileY = 16, kFilterThreads = 256;
constexpr size_t tile_bytes(int step, bool last) { return (size_t)(kTileX + 4 * step) * (kTileY + 4 * step) * (last ? 32 : 24); }

template <int STEP, bool LAST>
__global__ void __launch_bounds__(kFilterThreads, STEP ? 3 : 2)
k_atrous(int w, int h, int any_step, const float4* __restrict__ guide, const uint8_t* __restrict__ surface, const float2* __restrict__ b_in,
         float2* __restrict__ b_out, const uint2* __restrict__ colour, uchar4* __restrict__ image, uint2* __restrict__ copy_to, F2 neg_zero) {
    constexpr int pitch = kTileX + 4 * STEP, rows = kTileY + 4 * STEP, cells = pitch * rows;
    extern __shared__ __align__(16) unsigned char tile[];
    float4* tg = reinterpret_cast<float4*>(tile);
    float2* tb = reinterpret_cast<float2*>(tile + (size_t)cells * 16);
    uint2* tc = reinterpret_cast<uint2*>(tile + (size_t)cells * 24);
    const int tid = threadIdx.x, lx = tid & 31, ly = tid >> 5;
    const int x0 = blockIdx.x * kTileX, y0 = blockIdx.y * kTileY;
    const int step = STEP ? STEP : any_step;
    if (STEP) {
        for (int i = tid; i < cells; i += kFilterThreads) {
            const int r = i / pitch, c = i - r * pitch;
            const int qx = min(max(x0 + c - 2 * STEP, 0), w - 1), qy = min(max(y0 + r - 2 * STEP, 0), h - 1);
            const size_t q = (size_t)qy * w + qx;
            const unsigned s16 = (unsigned)__cvta_generic_to_shared(tg + i), s8 = (unsigned)__cvta_generic_to_shared(tb + i);
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(s16), "l"(guide + q) : "memory");
            asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(s8), "l"(b_in + q) : "memory");
            if (LAST) asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"((unsigned)__cvta_generic_to_shared(tc + i)), "l"(colour + q) : "memory");
        }
        asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory");
        __syncthreads();
    }
    const int x = x0 + lx;
    const int ya = y0 + ly, yb = ya + 8;
    if (x >= w || ya >= h) return;
    const bool have_b = yb < h;
    const size_t ia = (size_t)ya * w + x, ib = have_b ? (size_t)yb * w + x : ia;
    // tap (yy, xx) of the pixel `down` rows below this thread's first one
    auto cell = [&](int yy, int xx, int down) -> size_t {
        if (STEP) return (size_t)((ly + down + (yy + 2) * STEP) * pitch + lx + (xx + 2) * STEP);
        // in 64 bits: rows * steps of a large image leave 32
        const long long ty = (long long)(ya + down) + (long long)yy * step, tx = (long long)x + (long long)xx * step;
        const int qy = (int)min(max(ty, 0ll), (long long)(h - 1)), qx = (int)min(max(tx, 0ll), (long long)(w - 1));
        return (size_t)qy * w + qx;
    };
    const float4* gp = STEP ? tg : guide;
    const float2* bp = STEP ? tb : b_in;
    const uint2* cp = STEP ? tc : colour;
    const float eps = 1e-6f, log2e = 1.4426950408889634f, inv256 = 1.0f / 256.0f;
    const size_t ca = cell(0, 0, 0), cb = cell(0, 0, 8);
    const float4 ga = gp[ca], gb = gp[cb];
    const float2 ba = bp[ca], bb = bp[cb];
    const float step_f = (float)step;
    const float inv_za = 1.0f / max_glsl(fabsf(ga.w) * step_f, eps), inv_zb = 1.0f / max_glsl(fabsf(gb.w) * step_f, eps);
    const float inv_la = 1.0f / max_glsl(1.0f * sqrtf(max_glsl(max_glsl(ba.y, 0.0f), 1e-10f)), eps);
    const float inv_lb = 1.0f / max_glsl(1.0f * sqrtf(max_glsl(max_glsl(bb.y, 0.0f), 1e-10f)), eps);
    const bool on_a = surface[ia] != 0, on_b = have_b && surface[ib] != 0;
    F2 sum_r = 0, sum_g = 0, sum_b = 0, sum_w = 0, sum_var = 0, sum_wvar = 0;  // bits of two zeros
    if (on_a || on_b) {
        const F2 log2e2 = pack2(log2e, log2e);
#pragma unroll 1
        for (int yy = -2; yy <= 2; ++yy) {
            const float ky = yy == 0 ? 6.0f : ((yy == 1 || yy == -1) ? 4.0f : 1.0f);
#pragma unroll
            for (int xx = -2; xx <= 2; ++xx) {
                const float kx = xx == 0 ? 6.0f : ((xx == 1 || xx == -1) ? 4.0f : 1.0f);
                const float wk = kx * ky * inv256;
                const size_t qa = cell(yy, xx, 0), qb = cell(yy, xx, 8);
                const float4 sa = gp[qa], sb = gp[qb];
                const float2 va = bp[qa], vb = bp[qb];
                F2 wn = pack2(max0_nan(dot3(ga.x, ga.y, ga.z, sa.x, sa.y, sa.z)), max0_nan(dot3(gb.x, gb.y, gb.z, sb.x, sb.y, sb.z)));
#pragma unroll
                for (int i = 0; i < 7; ++i) wn = mul2(wn, wn);
                float wna, wnb;
                unpack2(wn, wna, wnb);
                const bool skip_a = wna <= eps, skip_b = wnb <= eps;  // such a tap adds nothing, whatever its values
                const F2 wd = exp2_poly2(fma2(pack2(-fabsf(ga.w - sa.w) * inv_za, -fabsf(gb.w - sb.w) * inv_zb), log2e2, neg_zero));
                const F2 wl = exp2_poly2(fma2(pack2(-fabsf(ba.x - va.x) * inv_la, -fabsf(bb.x - vb.x) * inv_lb), log2e2, neg_zero));
                float wta, wtb;
                unpack2(mul2(mul2(mul2(pack2(wk, wk), wn), wd), wl), wta, wtb);
                const F2 wt = pack2(skip_a ? 0.0f : wta, skip_b ? 0.0f : wtb);
                // variances are never negative (a NaN stays one), so the shader's max(variance, 0) changes nothing
                const F2 sv = pack2(skip_a ? 0.0f : va.y, skip_b ? 0.0f : vb.y);
                if (LAST) {
                    uint2 pa = cp[qa], pb = cp[qb];
                    if (skip_a) pa = make_uint2(0u, 0u);
                    if (skip_b) pb = make_uint2(0u, 0u);
                    const __half2 la = *reinterpret_cast<const __half2*>(&pa.x), lb = *reinterpret_cast<const __half2*>(&pb.x);
                    const __half2 ha = *reinterpret_cast<const __half2*>(&pa.y), hb = *reinterpret_cast<const __half2*>(&pb.y);
                    sum_r = add2(sum_r, fma2(pack2(__low2float(la), __low2float(lb)), wt, neg_zero));
                    sum_g = add2(sum_g, fma2(pack2(__high2float(la), __high2float(lb)), wt, neg_zero));
                    sum_b = add2(sum_b, fma2(pack2(__low2float(ha), __low2float(hb)), wt, neg_zero));
                    sum_w = add2(sum_w, wt);
                }
                const F2 w2 = fma2(wt, wt, neg_zero);
                sum_var = add2(sum_var, fma2(sv, w2, neg_zero));
                sum_wvar = add2(sum_wvar, w2);
            }
        }
    }
    float sv[2], swv[2];
    unpack2(sum_var, sv[0], sv[1]);
    unpack2(sum_wvar, swv[0], swv[1]);
    float sr[2], sg[2], sb[2], sw[2];
    unpack2(sum_r, sr[0], sr[1]);
    unpack2(sum_g, sg[0], sg[1]);
    unpack2(sum_b, sb[0], sb[1]);
    unpack2(sum_w, sw[0], sw[1]);
#pragma unroll
    for (int k = 0; k < 2; ++k) {
        if (k && !have_b) break;
        const size_t idx = k ? ib : ia;
        const float2 centre = k ? bb : ba;
        const bool on = k ? on_b : on_a;  // no surface: colour and variance pass through
        b_out[idx] = make_float2(centre.x, on ? sv[k] * (1.0f / max_glsl(swv[k], eps)) : centre.y);
        if (LAST) {
            uchar4 result;
            if (on) {
                const float inv_w = 1.0f / max_glsl(sw[k], eps);
                result = pack_rgb8(sr[k] * inv_w, sg[k] * inv_w, sb[k] * inv_w);
            } else {
                const float3 s = load_rgb16(colour, idx);
                result = pack_rgb8(s.x, s.y, s.z);
            }
            image[idx] = result;
            if (copy_to) copy_to[idx] = pack_rgba16(result.x / 255.0f, result.y / 255.0f, result.z / 255.0f, result.w / 255.0f);
        }
    }
}

// ---- copy pass (raytracing_atrous.comp:66-70, iteration 98) ---------------------------------------
__global__ void k_copy(size_t n, const uchar4* __restrict__ image, uint2* __restrict__ dst) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uchar4 c = image[i];
    dst[i] = pack_rgba16(c.x / 255.0f, c.y / 255.0f, c.z / 255.0f, c.w / 255.0f);
}

// ---- the moments image {history length, first moment, second moment, variance} -> its two planes ----
__global__ void k_split_moments(size_t n, const float4* __restrict__ m, float2* __restrict__ a, float2* __restrict__ b) {
    const size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const float4 v = m[i];
    a[i] = make_float2(v.x, v.z);
    b[i] = make_float2(v.y, v.w);
}

thread_local std::string g_svgf_create_error;

}  // namespace

struct neon_svgf_handle {
    neon_svgf_config cfg{};
    std::string err;
    uint2 *colour_a = nullptr, *colour_b = nullptr;  // rgba16f history images
    float2* mom_a[2] = {nullptr, nullptr};           // {history length, second moment}: mom_a[cur_a] holds the state between frames
    float2* mom_b[2] = {nullptr, nullptr};           // {first moment, variance}: mom_b[0] holds the state between frames
    float4* guide = nullptr;                         // {normal, depth} of the frame being filtered
    uint8_t* surface = nullptr;                      // whether its pixels show a surface
    int ping_pong = 0, cur_a = 0;
    bool settle = false;  // a caller has captured frames, whose graphs name the buffers: every frame leaves the state in mom_a[cur_a]
    float4* stage[4] = {nullptr, nullptr, nullptr, nullptr};  // device copies of host G-buffers (denoise_host)
    uchar4* stage_image = nullptr;
    int64_t launches = 0;
    int launches_per_frame = 0;
    int use_graphs = 1;
    cudaStream_t own_stream = nullptr, last_stream = nullptr;
    struct Cached {
        Frame fr;
        int ping_pong, cur_a;
        bool settle;
        cudaGraphExec_t exec;
    };
    std::vector<Cached> graphs;
};

namespace {

int sfail(neon_svgf_handle* h, int code, const char* fmt, ...) {
    char buf[512];
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(buf, sizeof buf, fmt, ap);
    va_end(ap);
    if (h) h->err = buf; else g_svgf_create_error = buf;
    return code;
}

#define SCU(h, call)                                                                                       \
    do {                                                                                                   \
        cudaError_t e_ = (call);                                                                           \
        if (e_ != cudaSuccess) return sfail(h, NEON_MOE_ECUDA, "%s: %s", #call, cudaGetErrorString(e_)); \
    } while (0)

void drop_graphs(neon_svgf_handle* h) {
    for (auto& g : h->graphs)
        if (g.exec) cudaGraphExecDestroy(g.exec);
    h->graphs.clear();
}

template <int STEP, bool LAST>
void launch_atrous(neon_svgf_handle* h, int step, int from, const uint2* src, uchar4* image, uint2* copy_to, cudaStream_t st) {
    const dim3 grid((h->cfg.width + kTileX - 1) / kTileX, (h->cfg.height + kTileY - 1) / kTileY);
    k_atrous<STEP, LAST><<<grid, kFilterThreads, STEP ? tile_bytes(STEP, LAST) : 0, st>>>(
        h->cfg.width, h->cfg.height, step, h->guide, h->surface, h->mom_b[from], h->mom_b[from ^ 1], src, image, copy_to, kNegZero2);
}
template <bool LAST>
void launch_atrous(neon_svgf_handle* h, int step, int from, const uint2* src, uchar4* image, uint2* copy_to, cudaStream_t st) {
    switch (step) {
        case 1: launch_atrous<1, LAST>(h, step, from, src, image, copy_to, st); break;
        case 2: launch_atrous<2, LAST>(h, step, from, src, image, copy_to, st); break;
        case 4: launch_atrous<4, LAST>(h, step, from, src, image, copy_to, st); break;
        case 8: launch_atrous<8, LAST>(h, step, from, src, image, copy_to, st); break;
        default: launch_atrous<0, LAST>(h, step, from, src, image, copy_to, st);
    }
}
// tiles above 48 KB of shared memory have to be asked for
template <int STEP>
bool allow_tile() {
    return cudaFuncSetAttribute(k_atrous<STEP, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_bytes(STEP, false)) == cudaSuccess &&
           cudaFuncSetAttribute(k_atrous<STEP, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tile_bytes(STEP, true)) == cudaSuccess;
}

// the kernels of one frame in the reference's dispatch order; ev (optional) gets 3 event marks.
// ping_pong is the flag's value BEFORE the frame (RayTracingRast::renderCompute flips it), cur_a that of h->cur_a; the
// frame leaves the state in mom_a[cur_a ^ 1], with h->settle in mom_a[cur_a].
int record_frame(neon_svgf_handle* h, const Frame& fr, int ping_pong, int cur_a, cudaStream_t st, cudaEvent_t* ev = nullptr) {
    const int w = h->cfg.width, ht = h->cfg.height, iters = h->cfg.atrous_iterations;
    const dim3 grid((w + kBlockX - 1) / kBlockX, (ht + kBlockY - 1) / kBlockY), block(kBlockX, kBlockY);
    // set 1 binds {5: colour_a, 7: colour_b}, set 2 the two swapped; the temporal pass takes set 1 when the flag is set
    uint2* prev = ping_pong ? h->colour_a : h->colour_b;
    uint2* next = ping_pong ? h->colour_b : h->colour_a;
    int n = 0, cur = 0;  // mom_b[cur] is read, mom_b[cur ^ 1] written
    if (ev) cudaEventRecord(ev[0], st);
    k_temporal<<<grid, block, 0, st>>>(w, ht, fr, prev, next, h->mom_a[cur_a], h->mom_b[0], h->mom_a[cur_a ^ 1], h->mom_b[1], h->guide,
                                       h->surface); ++n;
    cur ^= 1;
    if (ev) cudaEventRecord(ev[1], st);
    // filter passes: even ones read the image the temporal pass wrote, odd ones the older one; the
    // even-count extra pass runs on the second set at step 1 (raytracing_rast.cpp:390-411).  Their number
    // is odd, so the variances end in mom_b[0].
    const int passes = iters + (iters % 2 == 0 ? 1 : 0);
    bool copied = false;
    for (int i = 0; i < passes; ++i) {
        const bool extra = i == iters;
        const uint2* src = extra ? prev : ((i % 2 == 0) ? next : prev);
        const bool last = i == passes - 1;
        uint2* copy_to = (last && src != prev) ? prev : nullptr;
        const int step = extra ? 1 : (1 << i);
        if (last) launch_atrous<true>(h, step, cur, src, fr.image, copy_to, st);
        else launch_atrous<false>(h, step, cur, src, nullptr, nullptr, st);
        ++n;
        cur ^= 1;
        copied = copy_to != nullptr;
    }
    if (!copied) {
        const size_t px = (size_t)w * ht;
        k_copy<<<(unsigned)((px + 255) / 256), 256, 0, st>>>(px, fr.image, prev); ++n;
    }
    if (h->settle && cudaMemcpyAsync(h->mom_a[cur_a], h->mom_a[cur_a ^ 1], (size_t)w * ht * sizeof(float2), cudaMemcpyDeviceToDevice, st) != cudaSuccess)
        return -1;
    if (ev) cudaEventRecord(ev[2], st);
    h->launches_per_frame = n;
    return cudaGetLastError() == cudaSuccess ? n : -1;
}

int check_frame_args(neon_svgf_handle* h, const void* a, const void* b, const void* c, const void* d, const void* e) {
    if (!a || !b || !c || !d || !e) return sfail(h, NEON_MOE_EINVAL, "null image pointer");
    return 0;
}

}  // namespace

extern "C" {

int neon_svgf_create(const neon_svgf_config* cfg, neon_svgf_handle** out) {
    if (!cfg || !out) return NEON_MOE_EINVAL;
    *out = nullptr;
    if (cfg->width < 1 || cfg->height < 1 || (int64_t)cfg->width * cfg->height > (int64_t)1 << 28)
        return sfail(nullptr, NEON_MOE_EINVAL, "bad image size %d x %d", cfg->width, cfg->height);
    if (cfg->atrous_iterations < 0 || cfg->atrous_iterations > 16)
        return sfail(nullptr, NEON_MOE_EINVAL, "atrous_iterations=%d outside [0, 16]", cfg->atrous_iterations);
    int n_dev = 0;
    if (cudaGetDeviceCount(&n_dev) != cudaSuccess || cfg->device < 0 || cfg->device >= n_dev) {
        cudaGetLastError();
        return sfail(nullptr, NEON_MOE_ECUDA, "no CUDA device %d", cfg->device);
    }
    neon_svgf_handle* h = new (std::nothrow) neon_svgf_handle;
    if (!h) return NEON_MOE_ECUDA;
    h->cfg = *cfg;
    const size_t px = (size_t)cfg->width * cfg->height;
    bool ok = cudaSetDevice(cfg->device) == cudaSuccess && cudaMalloc(&h->colour_a, px * 8) == cudaSuccess &&
              cudaMalloc(&h->colour_b, px * 8) == cudaSuccess && cudaMalloc(&h->guide, px * 16) == cudaSuccess &&
              cudaMalloc(&h->surface, px) == cudaSuccess && allow_tile<4>() && allow_tile<8>() &&
              cudaStreamCreateWithFlags(&h->own_stream, cudaStreamNonBlocking) == cudaSuccess;
    ok = ok && cudaMemset(h->colour_a, 0, px * 8) == cudaSuccess && cudaMemset(h->colour_b, 0, px * 8) == cudaSuccess;
    for (int i = 0; i < 2; ++i)
        for (float2** m : {&h->mom_a[i], &h->mom_b[i]})
            ok = ok && cudaMalloc(m, px * 8) == cudaSuccess && cudaMemset(*m, 0, px * 8) == cudaSuccess;
    if (!ok) {
        const cudaError_t e = cudaGetLastError();
        neon_svgf_destroy(h);
        return sfail(nullptr, NEON_MOE_ECUDA, "device allocation failed: %s", cudaGetErrorString(e));
    }
    *out = h;
    return NEON_MOE_OK;
}

int neon_svgf_destroy(neon_svgf_handle* h) {
    if (!h) return NEON_MOE_OK;
    cudaSetDevice(h->cfg.device);
    if (h->last_stream) cudaStreamSynchronize(h->last_stream);
    drop_graphs(h);
    cudaFree(h->colour_a); cudaFree(h->colour_b); cudaFree(h->guide); cudaFree(h->surface);
    for (int i = 0; i < 2; ++i) { cudaFree(h->mom_a[i]); cudaFree(h->mom_b[i]); }
    for (auto* p : h->stage) cudaFree(p);
    cudaFree(h->stage_image);
    if (h->own_stream) cudaStreamDestroy(h->own_stream);
    cudaGetLastError();
    delete h;
    return NEON_MOE_OK;
}

const char* neon_svgf_last_error(const neon_svgf_handle* h) { return h ? h->err.c_str() : g_svgf_create_error.c_str(); }

int neon_svgf_set_history(neon_svgf_handle* h, const uint16_t* colour_a, const uint16_t* colour_b, const float* moments,
                          int ping_pong, int on_device) {
    if (!h) return NEON_MOE_EINVAL;
    SCU(h, cudaSetDevice(h->cfg.device));
    SCU(h, cudaStreamSynchronize(h->last_stream));  // also the NULL stream
    const size_t px = (size_t)h->cfg.width * h->cfg.height;
    const cudaMemcpyKind kind = on_device ? cudaMemcpyDeviceToDevice : cudaMemcpyHostToDevice;
    if (colour_a) SCU(h, cudaMemcpy(h->colour_a, colour_a, px * 8, kind)); else SCU(h, cudaMemset(h->colour_a, 0, px * 8));
    if (colour_b) SCU(h, cudaMemcpy(h->colour_b, colour_b, px * 8, kind)); else SCU(h, cudaMemset(h->colour_b, 0, px * 8));
    if (moments) {
        // through the guide image, which every frame writes before it reads it, and on the copy's own stream: a
        // device-to-device or pageable copy may still be under way when its call returns
        SCU(h, cudaMemcpy(h->guide, moments, px * 16, kind));
        k_split_moments<<<(unsigned)((px + 255) / 256), 256, 0, nullptr>>>(px, h->guide, h->mom_a[h->cur_a], h->mom_b[0]);
        SCU(h, cudaGetLastError());
    } else {
        SCU(h, cudaMemset(h->mom_a[h->cur_a], 0, px * 8));
        SCU(h, cudaMemset(h->mom_b[0], 0, px * 8));
    }
    SCU(h, cudaStreamSynchronize(nullptr));  // the next frame may run on a stream that the NULL stream does not order
    h->ping_pong = ping_pong != 0;
    return NEON_MOE_OK;
}

int neon_svgf_denoise(neon_svgf_handle* h, const float* position, const float* normal, const float* barycentric,
                      const float* motion, uint8_t* image, void* cuda_stream) {
    if (!h) return NEON_MOE_EINVAL;
    if (int rc = check_frame_args(h, position, normal, barycentric, motion, image)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    SCU(h, cudaSetDevice(h->cfg.device));
    const Frame fr{reinterpret_cast<const float4*>(position), reinterpret_cast<const float4*>(normal),
                   reinterpret_cast<const float4*>(barycentric), reinterpret_cast<const float4*>(motion),
                   reinterpret_cast<uchar4*>(image)};
    const int pp = h->ping_pong, ca = h->cur_a;
    cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
    bool graphs = h->use_graphs != 0;
    if (cudaStreamIsCapturing(st, &cs) != cudaSuccess || cs != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        graphs = false;  // inside the caller's own capture: record the kernels directly
        if (cs != cudaStreamCaptureStatusNone) h->settle = true;
    }
    if (graphs) {
        neon_svgf_handle::Cached* hit = nullptr;
        for (auto& g : h->graphs)
            if (g.ping_pong == pp && g.cur_a == ca && g.settle == h->settle && !memcmp(&g.fr, &fr, sizeof fr)) { hit = &g; break; }
        if (!hit) {
            if (h->graphs.size() >= 32) drop_graphs(h);
            SCU(h, cudaStreamBeginCapture(h->own_stream, cudaStreamCaptureModeThreadLocal));
            const int n = record_frame(h, fr, pp, ca, h->own_stream);
            cudaGraph_t graph = nullptr;
            cudaError_t ce = cudaStreamEndCapture(h->own_stream, &graph);
            cudaGraphExec_t exec = nullptr;
            if (n >= 0 && ce == cudaSuccess && graph) ce = cudaGraphInstantiate(&exec, graph, 0);
            if (graph) cudaGraphDestroy(graph);
            if (n < 0 || ce != cudaSuccess || !exec) {
                cudaGetLastError();
                h->use_graphs = 0;  // capture is not available here: stay eager
                graphs = false;
            } else {
                h->graphs.push_back({fr, pp, ca, h->settle, exec});
                hit = &h->graphs.back();
            }
        }
        if (hit) {
            SCU(h, cudaGraphLaunch(hit->exec, st));
            h->launches += h->launches_per_frame;
        }
    }
    if (!graphs) {
        const int n = record_frame(h, fr, pp, ca, st);
        if (n < 0) return sfail(h, NEON_MOE_ECUDA, "kernel launch failed: %s", cudaGetErrorString(cudaGetLastError()));
        h->launches += n;
    }
    h->ping_pong = !pp;
    if (!h->settle) h->cur_a = ca ^ 1;
    h->last_stream = st;
    return NEON_MOE_OK;
}

int neon_svgf_denoise_host(neon_svgf_handle* h, const float* position, const float* normal, const float* barycentric,
                           const float* motion, uint8_t* image, void* cuda_stream) {
    if (!h) return NEON_MOE_EINVAL;
    if (int rc = check_frame_args(h, position, normal, barycentric, motion, image)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    SCU(h, cudaSetDevice(h->cfg.device));
    const size_t px = (size_t)h->cfg.width * h->cfg.height;
    if (!h->stage_image) {
        for (auto& p : h->stage) SCU(h, cudaMalloc(&p, px * 16));
        SCU(h, cudaMalloc(&h->stage_image, px * 4));
    }
    const float* src[4] = {position, normal, barycentric, motion};
    for (int i = 0; i < 4; ++i) SCU(h, cudaMemcpyAsync(h->stage[i], src[i], px * 16, cudaMemcpyHostToDevice, st));
    SCU(h, cudaMemcpyAsync(h->stage_image, image, px * 4, cudaMemcpyHostToDevice, st));
    if (int rc = neon_svgf_denoise(h, reinterpret_cast<const float*>(h->stage[0]), reinterpret_cast<const float*>(h->stage[1]),
                                   reinterpret_cast<const float*>(h->stage[2]), reinterpret_cast<const float*>(h->stage[3]),
                                   reinterpret_cast<uint8_t*>(h->stage_image), st))
        return rc;
    SCU(h, cudaMemcpyAsync(image, h->stage_image, px * 4, cudaMemcpyDeviceToHost, st));
    SCU(h, cudaStreamSynchronize(st));
    return NEON_MOE_OK;
}

int neon_svgf_read(neon_svgf_handle* h, const char* name, void* dst, uint64_t bytes) {
    if (!h || !name || !dst) return NEON_MOE_EINVAL;
    SCU(h, cudaSetDevice(h->cfg.device));
    SCU(h, cudaStreamSynchronize(h->last_stream));  // also the NULL stream
    const size_t px = (size_t)h->cfg.width * h->cfg.height;
    const void* src = nullptr;
    size_t need = 0;
    if (!strcmp(name, "colour_a")) { src = h->colour_a; need = px * 8; }
    else if (!strcmp(name, "colour_b")) { src = h->colour_b; need = px * 8; }
    else if (!strcmp(name, "moments")) need = px * 16;
    else if (!strcmp(name, "ping_pong")) {
        if (bytes != 4) return sfail(h, NEON_MOE_EINVAL, "ping_pong is 4 bytes");
        const int32_t v = h->ping_pong;
        memcpy(dst, &v, 4);
        return NEON_MOE_OK;
    } else return sfail(h, NEON_MOE_EINVAL, "unknown buffer '%s'", name);
    if (bytes != need) return sfail(h, NEON_MOE_EINVAL, "%s is %zu bytes, not %llu", name, need, (unsigned long long)bytes);
    if (!src) {  // the moments: joined from their planes on the host
        std::unique_ptr<float[]> planes(new (std::nothrow) float[4 * px]);
        if (!planes) return sfail(h, NEON_MOE_ECUDA, "out of host memory");
        const float *a = planes.get(), *b = a + 2 * px;
        SCU(h, cudaMemcpy(planes.get(), h->mom_a[h->cur_a], px * 8, cudaMemcpyDeviceToHost));
        SCU(h, cudaMemcpy(planes.get() + 2 * px, h->mom_b[0], px * 8, cudaMemcpyDeviceToHost));
        for (size_t i = 0; i < px; ++i) {
            const float m[4] = {a[2 * i], b[2 * i], a[2 * i + 1], b[2 * i + 1]};
            memcpy(static_cast<char*>(dst) + 16 * i, m, 16);
        }
        return NEON_MOE_OK;
    }
    SCU(h, cudaMemcpy(dst, src, need, cudaMemcpyDeviceToHost));
    return NEON_MOE_OK;
}

int neon_svgf_profile_frame(neon_svgf_handle* h, const float* position, const float* normal, const float* barycentric,
                            const float* motion, uint8_t* image, double* ms2, void* cuda_stream) {
    if (!h || !ms2) return NEON_MOE_EINVAL;
    if (int rc = check_frame_args(h, position, normal, barycentric, motion, image)) return rc;
    cudaStream_t st = static_cast<cudaStream_t>(cuda_stream);
    SCU(h, cudaSetDevice(h->cfg.device));
    const Frame fr{reinterpret_cast<const float4*>(position), reinterpret_cast<const float4*>(normal),
                   reinterpret_cast<const float4*>(barycentric), reinterpret_cast<const float4*>(motion),
                   reinterpret_cast<uchar4*>(image)};
    cudaEvent_t ev[3];
    for (auto& e : ev) SCU(h, cudaEventCreate(&e));
    const int n = record_frame(h, fr, h->ping_pong, h->cur_a, st, ev);
    int rc = NEON_MOE_OK;
    if (n < 0 || cudaStreamSynchronize(st) != cudaSuccess) rc = sfail(h, NEON_MOE_ECUDA, "profiled frame failed: %s", cudaGetErrorString(cudaGetLastError()));
    else {
        h->launches += n;
        h->ping_pong = !h->ping_pong;
        if (!h->settle) h->cur_a ^= 1;
        h->last_stream = st;
        for (int i = 0; i < 2; ++i) {
            float ms = 0.0f;
            cudaEventElapsedTime(&ms, ev[i], ev[i + 1]);
            ms2[i] = ms;
        }
    }
    for (auto& e : ev) cudaEventDestroy(e);
    return rc;
}

int neon_svgf_set_option(neon_svgf_handle* h, const char* name, int64_t value) {
    if (!h || !name) return NEON_MOE_EINVAL;
    if (!strcmp(name, "use_graphs")) {
        h->use_graphs = (int)value;
        if (!value) drop_graphs(h);
    } else return sfail(h, NEON_MOE_EINVAL, "unknown option '%s'", name);
    return NEON_MOE_OK;
}

int64_t neon_svgf_launch_count(const neon_svgf_handle* h) { return h ? h->launches : 0; }

}  // extern "C"
