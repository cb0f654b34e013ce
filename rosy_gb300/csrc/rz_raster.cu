// Geometry kernels of the shadow depth pass and the camera (visibility) pass.
//
// Reference path: the shadow draw loop (src/Engine/Graphics.cpp:5268-5288)
// running shadowVertexMain (src/shaders/shadow.slang:6-19), and the opaque
// scene draw loop (5631-5653) running the position part of vertexMain
// (src/shaders/basic.slang:116), followed by Vulkan's fixed-function clip,
// viewport, rasterisation, depth bias and GREATER_OR_EQUAL depth test with
// depth write (state at 4989-5040, 5222-5242).
//
// GB300 design:
//  * k_prep: per-draw MVP = P * W (one thread per draw).
//  * k_setup: one thread per triangle pulls its three positions, transforms,
//    clips (guard band + near/far), snaps to 8-bit sub-pixels, culls, and emits
//    64-byte records with the depth plane and bounding box. Records are
//    compacted and their 8x4-pixel stamp counts prefix-summed in the same pass
//    with a decoupled look-back across CTAs; each record also marks the work
//    chunks (kChunkStamps stamps) that start inside it.
//  * k_raster: persistent warps take chunks of stamps, so tiny and huge
//    triangles are balanced alike. A lane prepares a stamp (edges, bounds), then
//    the warp takes those that are left with a lane per pixel; coverage is
//    the integer edge-function test with the top-left rule, and the depth test
//    is a 64-bit atomicMax on (depth_bits << 32 | id). Because depths are
//    non-negative floats their bit patterns order like the values, so the max
//    key is exactly what a sequential GREATER_OR_EQUAL test leaves: the largest
//    depth, and among equal depths the last triangle submitted. The shadow map
//    is a 32-bit atomicMax on the depth bits.
#include <algorithm>
#include <type_traits>
#include <cstdio>

#include "rz_device.cuh"

namespace rz {

// ---------------------------------------------------------------------------
// per-draw matrices
// ---------------------------------------------------------------------------

// Also zeroes the clear list L (the pass's header and look-back words), so that
// the two need one launch.
__global__ void k_prep(const DrawRec* __restrict__ draws, uint32_t n, const rz_object* __restrict__ objects,
                       const ViewRec* __restrict__ views, float* __restrict__ out, ClearList L) {
    pdl_allow_next();
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    clear_share(L);
    if (d >= n) return;
    const float* P = views[draws[d].view].scene->shadow_projection_near;
    float A[16], B[16], C[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) A[i] = P[i];
    // cascade k: the light's orthographic extent times 2^k, i.e. clip x and y scaled by 2^-k (exact)
    const float s = ldexpf(1.0f, -(int)draws[d].cascade);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
        A[c * 4 + 0] *= s;
        A[c * 4 + 1] *= s;
    }
    const float* W = objects[draws[d].object].transform;
#pragma unroll
    for (int i = 0; i < 16; ++i) B[i] = W[i];
    mat4_mul(A, B, C);
#pragma unroll
    for (int i = 0; i < 16; ++i) out[16 * d + i] = C[i];
}

namespace {
thread_local uint32_t t_launches = 0;
}  // namespace

void note_launch() { ++t_launches; }

uint32_t take_launches() {
    const uint32_t n = t_launches;
    t_launches = 0;
    return n;
}

void launch_prep(const DrawRec* draws, uint32_t n, const rz_object* objects, const ViewRec* views, float* out_mvp,
                 cudaStream_t stream, const ClearList* clear, int sm_count) {
    const ClearList none{};
    const ClearList& L = clear ? *clear : none;
    const unsigned blocks = std::max((n + 127) / 128, clear_blocks(L, sm_count, 128));
    if (blocks == 0) return;
    k_prep<<<blocks, 128, 0, stream>>>(draws, n, objects, views, out_mvp, L);
    note_launch();
}

// ---------------------------------------------------------------------------
// clears (the load-op CLEAR of the depth attachments, scratch headers)
// ---------------------------------------------------------------------------

__global__ void __launch_bounds__(256) k_clear(ClearList L) { clear_share(L); }

unsigned clear_blocks(const ClearList& list, int sm_count, unsigned threads) {
    size_t most = 0;
    for (int b = 0; b < list.count; ++b) most = list.bytes[b] > most ? list.bytes[b] : most;
    if (most == 0) return 0;
    size_t blocks = (most / 16 + threads - 1) / threads;
    const size_t cap = (size_t)sm_count * 8 * (256 / threads);
    if (blocks > cap) blocks = cap;
    return blocks ? (unsigned)blocks : 1u;
}

void launch_clear(const ClearList& list, int sm_count, cudaStream_t stream) {
    const unsigned blocks = clear_blocks(list, sm_count, 256);
    if (blocks == 0) return;
    k_clear<<<blocks, 256, 0, stream>>>(list);
    note_launch();
}

// ---------------------------------------------------------------------------
// triangle setup
// ---------------------------------------------------------------------------

struct CV {
    float x, y, z, w;
};

__device__ __forceinline__ float plane_dist(const CV& c, int p) {
    switch (p) {
        case 0: return c.z;
        case 1: return c.w - c.z;
        case 2: return fmaf(kGuardBand, c.w, c.x);
        case 3: return fmaf(kGuardBand, c.w, -c.x);
        case 4: return fmaf(kGuardBand, c.w, c.y);
        default: return fmaf(kGuardBand, c.w, -c.y);
    }
}

__device__ __forceinline__ unsigned outcode(const CV& c) {
    unsigned m = 0;
#pragma unroll
    for (int p = 0; p < 6; ++p)
        if (!(plane_dist(c, p) >= 0.0f)) m |= 1u << p;
    return m;
}

// Whether outcode(c) is 0.
__device__ __forceinline__ bool inside_all(const CV& c) {
    bool in = true;
#pragma unroll
    for (int p = 0; p < 6; ++p) in = in && plane_dist(c, p) >= 0.0f;
    return in;
}

// Sutherland-Hodgman against the planes in `any` (rare path).
__device__ __noinline__ int clip_polygon(CV* poly, unsigned any) {
    CV buf[9];
    int n = 3;
    for (int p = 0; p < 6 && n > 0; ++p) {
        if (!(any & (1u << p))) continue;
        int m = 0;
        for (int i = 0; i < n; ++i) {
            const CV a = poly[i];
            const CV b = poly[(i + 1) % n];
            const float da = plane_dist(a, p);
            const float db = plane_dist(b, p);
            const bool ia = da >= 0.0f, ib = db >= 0.0f;
            if (ia) buf[m++] = a;
            if (ia != ib) {
                const float t = da / (da - db);
                CV c;
                c.x = fmaf(t, b.x - a.x, a.x);
                c.y = fmaf(t, b.y - a.y, a.y);
                c.z = fmaf(t, b.z - a.z, a.z);
                c.w = fmaf(t, b.w - a.w, a.w);
                buf[m++] = c;
            }
        }
        n = m;
        for (int i = 0; i < n; ++i) poly[i] = buf[i];
    }
    return n >= 3 ? n : 0;
}

struct SV {
    int32_t X, Y;
    float z;
};

// Window position (1/256 pixel) of a clip vertex. `unit`: w is 1, as under an
// orthographic light, and x / 1 is x.
__device__ __forceinline__ SV to_screen_xy(const CV& c, float hw, float hh, bool unit) {
    const float xn = unit ? c.x : c.x / c.w;
    const float yn = unit ? c.y : c.y / c.w;
    const float xs = fmaf(xn, hw, hw);
    const float ys = fmaf(yn, hh, hh);
    SV s;
    s.X = (int32_t)rintf(xs * 256.0f);
    s.Y = (int32_t)rintf(ys * 256.0f);
    s.z = 0.0f;
    return s;
}

__device__ __forceinline__ SV to_screen(const CV& c, float hw, float hh) {
    SV s = to_screen_xy(c, hw, hh, false);
    s.z = c.z / c.w;
    return s;
}

__device__ __forceinline__ int64_t area2(const SV& a, const SV& b, const SV& c) {
    return (int64_t)(b.X - a.X) * (int64_t)(c.Y - a.Y) - (int64_t)(c.X - a.X) * (int64_t)(b.Y - a.Y);
}

// Whether a record's stamps lie on the grid of the target's 8x4 blocks, so that each has a
// block's depth to be tested against (see raster_front): in the opaque camera pass, the one
// unordered pass with triangle references and the one that k_raster takes with ids
// (launch_raster sees to it), where the row and the column that this may add are few of many. (24x12
// or 16x8 pixels gain nothing on deep overdraw and cost a mesh scene up to 0.4 % more; 64x32
// lose 3 % of a soup's frame. Shadow passes have no grid: what they gained was within the noise,
// and scene-scale frames lost 2 %.)
constexpr int kGridW = 32, kGridH = 16;
__device__ __forceinline__ bool on_grid(bool camera, int px0, int py0, int px1, int py1) {
    return camera && px1 - px0 >= kGridW - 1 && py1 - py0 >= kGridH - 1;
}

// A record's stamps: how many in a row (nsx) and in all.
__device__ __forceinline__ uint32_t record_stamps(const TriRecord& r, bool camera, uint32_t& nsx) {
    const int px0 = r.p0 & 0xffff, py0 = r.p0 >> 16, px1 = r.p1 & 0xffff, py1 = r.p1 >> 16;
    const int m = on_grid(camera, px0, py0, px1, py1) ? -1 : 0;
    nsx = (uint32_t)((px1 - px0 + (px0 & m & (kStampW - 1))) / kStampW + 1);
    return nsx * (uint32_t)((py1 - py0 + (py0 & m & (kStampH - 1))) / kStampH + 1);
}

// The raster facts of a large record (packed by the setup, decoded by the raster):
// the edges' top-left bias, whether the stamps may be taken together (near: float
// offsets from vertex 0 are exact over the box, and edges are below 2^26 so that a
// stamp's edge values fit 32 bits), whether its edge functions themselves fit 32
// bits (small: an extent of at most 90 pixels each way), whether the viewport cut its
// box, and its stamps per row. Pixels past an uncut box edge lie outside the triangle's extent, so the
// edge test alone rejects the stamps' overhang there; only a cut box needs the check.
constexpr uint32_t kFactNear = 8u, kFactCut = 16u, kFactSmall = 32u;
// every edge value over the box plus a stamp of overhang is below 2 * ((90 + 8) * 256)^2 < 2^31
constexpr int kSmallEdges = 90;

__device__ __forceinline__ uint32_t large_facts(const TriRecord& r, int32_t bb_hi) {
    const int32_t X[3] = {r.X0, r.X1, r.X2}, Y[3] = {r.Y0, r.Y1, r.Y2};
    const int px0 = (int)(r.p0 & 0xffff), py0 = (int)(r.p0 >> 16), px1 = (int)(r.p1 & 0xffff), py1 = (int)(r.p1 >> 16);
    uint32_t flags = 0;
    bool near_origin = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = (i + 1) % 3, b = (i + 2) % 3;
        const int32_t dx = X[b] - X[a], dy = Y[b] - Y[a];
        if (!(dy < 0 || (dy == 0 && dx > 0))) flags |= 1u << i;
        near_origin = near_origin && abs(dx) < (1 << 26) && abs(dy) < (1 << 26);
    }
    const int32_t lo_x = px0 * 256 - X[0] - kStampW * 256, hi_x = px1 * 256 + 256 - X[0] + kStampW * 256;
    const int32_t lo_y = py0 * 256 - Y[0] - kStampH * 256, hi_y = py1 * 256 + 256 - Y[0] + kStampH * 256;
    const int32_t lim = 1 << 23;
    near_origin = near_origin && lo_x > -lim && hi_x < lim && lo_y > -lim && hi_y < lim;
    const int32_t max_x = max(X[0], max(X[1], X[2])), max_y = max(Y[0], max(Y[1], Y[2]));
    const bool cut = ((max_x - bb_hi) >> 8) > px1 || ((max_y - bb_hi) >> 8) > py1;
    const bool small = max_x - min(X[0], min(X[1], X[2])) <= kSmallEdges * 256 && max_y - min(Y[0], min(Y[1], Y[2])) <= kSmallEdges * 256;
    return flags | (small ? kFactSmall : 0u) | (near_origin ? kFactNear : 0u) | (cut ? kFactCut : 0u);
}


// Viewport and fixed-function state of the view a triangle belongs to.
struct ViewState {
    int width, height;
    int bb_lo, bb_hi;  // largest and smallest sample offset (1/256 pixel) of the pass: box of pixels any sample may hit
    int cull_front, ccw_front;
    int bias_enabled;
    float bias_constant, bias_clamp, bias_slope;
    uint32_t view;
};

// Builds the record of a triangle ordered with S > 0. Returns 0 if its pixel
// bounding box is empty, 2 for a small triangle (extent at most kSmallExtent
// pixels each way, rasterised by one lane), 1 otherwise.
__device__ __forceinline__ int make_record(const SV& v0, const SV& v1, const SV& v2, int64_t S, const ViewState& P,
                                           bool ordered, uint32_t small_extent, uint32_t id, TriRecord& r) {
    const int32_t minX = min(v0.X, min(v1.X, v2.X)), maxX = max(v0.X, max(v1.X, v2.X));
    const int32_t minY = min(v0.Y, min(v1.Y, v2.Y)), maxY = max(v0.Y, max(v1.Y, v2.Y));
    // pixels p with minX <= 256 p + o <= maxX for some sample offset o in [bb_hi, bb_lo]
    const int px0 = max((minX - P.bb_lo + 255) >> 8, 0), px1 = min((maxX - P.bb_hi) >> 8, P.width - 1);
    const int py0 = max((minY - P.bb_lo + 255) >> 8, 0), py1 = min((maxY - P.bb_hi) >> 8, P.height - 1);
    if (px0 > px1 || py0 > py1) return 0;
    const float fX1 = (float)(v1.X - v0.X), fY1 = (float)(v1.Y - v0.Y);
    const float fX2 = (float)(v2.X - v0.X), fY2 = (float)(v2.Y - v0.Y);
    const float fS = (float)S;
    const float dz1 = v1.z - v0.z, dz2 = v2.z - v0.z;
    const float dzdx = fmaf(dz1, fY2, -(dz2 * fY1)) / fS;
    const float dzdy = fmaf(dz2, fX1, -(dz1 * fX2)) / fS;
    float o = 0.0f;
    if (P.bias_enabled) {
        // Vulkan depth bias for floating-point depth: m * slope + r * constant,
        // r = 2^(e_max - 23), then clamped.
        const float m = fmaxf(fabsf(dzdx), fabsf(dzdy)) * 256.0f;
        uint32_t e = max((__float_as_uint(fabsf(v0.z)) >> 23) & 0xffu,
                         max((__float_as_uint(fabsf(v1.z)) >> 23) & 0xffu, (__float_as_uint(fabsf(v2.z)) >> 23) & 0xffu));
        const float rr = (e >= 24u) ? __uint_as_float((e - 23u) << 23) : 0.0f;
        o = fmaf(m, P.bias_slope, rr * P.bias_constant);
        if (P.bias_clamp > 0.0f) o = fminf(o, P.bias_clamp);
        else if (P.bias_clamp < 0.0f) o = fmaxf(o, P.bias_clamp);
    }
    r.X0 = v0.X;
    r.Y0 = v0.Y;
    r.X1 = v1.X;
    r.Y1 = v1.Y;
    r.X2 = v2.X;
    r.Y2 = v2.Y;
    r.z0 = v0.z;
    r.dzdx = dzdx;
    r.dzdy = dzdy;
    r.bias = o + 0.0f;  // -0 -> +0 (biased_depth relies on it; the sums are unchanged)
    r.p0 = (uint32_t)px0 | ((uint32_t)py0 << 16);
    r.p1 = (uint32_t)px1 | ((uint32_t)py1 << 16);
    r.id = id;
    r.view = P.view;
    r.stamp_offset = 0;
    const bool small = !ordered && (maxX - minX) <= (int32_t)small_extent * 256 && (maxY - minY) <= (int32_t)small_extent * 256;
    return small ? 2 : 1;
}

// Runs the fixed-function front end for one triangle and hands each record to `emit`.
template <bool kOrdered, class Emit>
__device__ __forceinline__ void setup_triangle(const PassParams& P, uint32_t tri, Emit& emit) {
    const uint32_t d = draw_from(P.draws, P.draw_count, P.draw_table, tri);
    const DrawRec dr = P.draws[d];
    const uint32_t t = tri - dr.tri_base;
    const uint32_t ib = dr.first_index + 3u * t;
    uint32_t vi[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) vi[k] = __ldg(&P.indices[ib + k]) + dr.vertex_base;
    if (vi[0] >= P.vertex_count || vi[1] >= P.vertex_count || vi[2] >= P.vertex_count) {
        atomicOr(P.error_flags, kErrBadIndex);
        return;
    }
    emit.source((uint32_t)dr.material, vi[0] - dr.vertex_base + dr.varying_base, vi[1] - dr.vertex_base + dr.varying_base,
                vi[2] - dr.vertex_base + dr.varying_base);
    const ViewRec& VR = P.views[dr.view];
    ViewState V;
    V.view = dr.view | (dr.cascade << kViewBits);
    V.width = P.write_id ? VR.width : VR.shadow_w;
    V.height = P.write_id ? VR.height : VR.shadow_h;
    const bool msaa = P.write_id && VR.samples > 1;
    V.bb_lo = msaa ? 224 : 128;
    V.bb_hi = msaa ? 32 : 128;
    V.cull_front = kOrdered ? 0 : VR.cull_front;
    V.ccw_front = VR.ccw_front;
    V.bias_enabled = P.write_id ? 0 : VR.bias_enabled;
    V.bias_constant = VR.bias_constant;
    V.bias_clamp = VR.bias_clamp;
    V.bias_slope = VR.bias_slope;
    const float4* M = reinterpret_cast<const float4*>(P.mvp + (size_t)P.mvp_stride * d);  // 16-byte aligned
    float Mr[16];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float4 m = __ldg(&M[i]);
        Mr[4 * i] = m.x;
        Mr[4 * i + 1] = m.y;
        Mr[4 * i + 2] = m.z;
        Mr[4 * i + 3] = m.w;
    }
    CV v[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 p = __ldg(&P.pos[vi[k]]);
        const float4 c = transform_point(Mr, p.x, p.y, p.z);
        v[k] = CV{c.x, c.y, c.z, c.w};
    }
    // the planes a vertex violates, worked out only if one of them does
    unsigned o0 = 0, o1 = 0, o2 = 0;
    if (!(inside_all(v[0]) && inside_all(v[1]) && inside_all(v[2]))) {
        o0 = outcode(v[0]);
        o1 = outcode(v[1]);
        o2 = outcode(v[2]);
        if (o0 & o1 & o2) return;
    }
    const float hw = (float)V.width * 0.5f, hh = (float)V.height * 0.5f;
    const uint32_t id = P.write_id ? (tri + 1u) : 0u;
    if (!(o0 | o1 | o2)) {
        if (!(v[0].w > 0.0f) || !(v[1].w > 0.0f) || !(v[2].w > 0.0f)) return;
        SV a, b, c;
        const bool unit = v[0].w == 1.0f && v[1].w == 1.0f && v[2].w == 1.0f;
        if (unit) {
            a = to_screen_xy(v[0], hw, hh, true);
            b = to_screen_xy(v[1], hw, hh, true);
            c = to_screen_xy(v[2], hw, hh, true);
        } else {
            a = to_screen_xy(v[0], hw, hh, false);
            b = to_screen_xy(v[1], hw, hh, false);
            c = to_screen_xy(v[2], hw, hh, false);
        }
        const int64_t S = area2(a, b, c);
        if (S == 0) return;
        const bool front = V.ccw_front ? (S < 0) : (S > 0);
        if (V.cull_front && front) return;
        if (unit) {
            a.z = v[0].z;
            b.z = v[1].z;
            c.z = v[2].z;
        } else {
            a.z = v[0].z / v[0].w;
            b.z = v[1].z / v[1].w;
            c.z = v[2].z / v[2].w;
        }
        TriRecord r;
        const int kind = S > 0 ? make_record(a, b, c, S, V, kOrdered, P.small_extent, id, r) : make_record(a, c, b, -S, V, kOrdered, P.small_extent, id, r);
        if (kind) emit(r, kind == 2);
        return;
    }
    // rare path: clip against the planes the vertices violate, fan-triangulate
    CV poly[9];
    poly[0] = v[0];
    poly[1] = v[1];
    poly[2] = v[2];
    const int n = clip_polygon(poly, o0 | o1 | o2);
    if (n < 3) return;
    for (int i = 0; i < n; ++i)
        if (!(poly[i].w > 0.0f)) return;
    SV sv[9];
    for (int i = 0; i < n; ++i) sv[i] = to_screen(poly[i], hw, hh);
    int64_t S = 0;
    for (int i = 1; i + 1 < n; ++i) S += area2(sv[0], sv[i], sv[i + 1]);
    if (S == 0) return;
    const bool front = V.ccw_front ? (S < 0) : (S > 0);
    if (V.cull_front && front) return;
    for (int i = 1; i + 1 < n; ++i) {
        const int64_t si = area2(sv[0], sv[i], sv[i + 1]);
        if (si == 0 || ((si > 0) != (S > 0))) continue;
        TriRecord r;
        const int kind = si > 0 ? make_record(sv[0], sv[i], sv[i + 1], si, V, kOrdered, P.small_extent, id, r)
                                : make_record(sv[0], sv[i + 1], sv[i], -si, V, kOrdered, P.small_extent, id, r);
        if (kind) emit(r, kind == 2);
    }
}

__device__ __forceinline__ void store_record(TriRecord* dst, const TriRecord& r) {
    const int4* s4 = reinterpret_cast<const int4*>(&r);
    int4* d4 = reinterpret_cast<int4*>(dst);
#pragma unroll
    for (int i = 0; i < 4; ++i) d4[i] = s4[i];
}

// Phase A: count the records (small and large) a triangle produces.
template <bool kOrdered>
struct CountEmit {
    uint32_t recs = 0;     // large
    uint64_t stamps = 0;   // of the large ones
    uint32_t small = 0;
    TriRecord first;       // the first record, kept for the common case of exactly one
    bool first_small = false;
    uint4* refs = nullptr; // camera passes: where the triangle's material and vertex records go
    uint32_t tri = 0;
    // every triangle with valid indices stores its material and the varying records
    // of its vertices: a triangle that owns a pixel of the visibility buffer is one of
    // them, and the shading finds them here (one load instead of a search of the
    // draw list and the index buffer, and no dependent load of the draw's material)
    __device__ void source(uint32_t material, uint32_t v0, uint32_t v1, uint32_t v2) {
        if (refs) refs[tri] = make_uint4(material, v0, v1, v2);
    }
    __device__ void operator()(const TriRecord& r, bool is_small) {
        if (recs + small == 0) {
            first = r;
            first_small = is_small;
        }
        if (is_small) {
            ++small;
            return;
        }
        ++recs;
        uint32_t nsx;
        stamps += record_stamps(r, !kOrdered && refs != nullptr, nsx);
    }
};

// Phase B: large records at their compacted index with their stamp offsets,
// small records at their slot in the small list (whose order does not matter:
// the depth test is an atomic max).
template <bool kOrdered>
struct WriteEmit {
    const PassParams* P;
    uint32_t rec;
    uint64_t stamp;
    uint32_t small;
    __device__ void source(uint32_t, uint32_t, uint32_t, uint32_t) {}
    __device__ void operator()(TriRecord& r, bool is_small) {
        if (is_small) {
            if (small < P->small_capacity) store_record(P->small_records + small, r);
            else atomicOr(P->error_flags, kErrRecordOverflow);
            ++small;
            return;
        }
        if (rec >= P->record_capacity) {
            atomicOr(P->error_flags, kErrRecordOverflow);
            return;
        }
        uint32_t nsx;
        const uint64_t end = stamp + record_stamps(r, !kOrdered && P->tri_refs != nullptr, nsx);
        r.view |= large_facts(r, P->bb_hi) << kRecFlagShift;
        r.stamp_offset = stamp | ((uint64_t)nsx << kStampOffsetBits);
        store_record(P->records + rec, r);
        // chunks whose first stamp lies inside this record start here
        const uint64_t cs = P->chunk_stamps;
        uint64_t k = (stamp + cs - 1) / cs;
        for (; k * cs < end; ++k) {
            if (k >= P->chunk_capacity) {
                atomicOr(P->error_flags, kErrStampOverflow);
                break;
            }
            P->chunk_map[k] = rec;
        }
        ++rec;
        stamp = end;
    }
};

// Packed scan value: records in bits 40..63, stamps in bits 0..39.
constexpr int kStampBits = 40;
constexpr uint64_t kStampMask = (1ull << kStampBits) - 1;
// Look-back status word: flag (2 bits) | records (24 bits) | stamps (38 bits).
constexpr uint64_t kFlagAgg = 1ull << 62;
constexpr uint64_t kFlagIncl = 2ull << 62;
constexpr int kStatusStampBits = 38;
constexpr uint64_t kStatusStampMask = (1ull << kStatusStampBits) - 1;
constexpr uint64_t kStatusRecMask = (1ull << 24) - 1;

__device__ __forceinline__ uint64_t to_status(uint64_t recs, uint64_t stamps) {
    return (recs << kStatusStampBits) | stamps;
}

// Bound by instruction issue and the latency of its chain (draw, indices, positions,
// slots): 46 % issue active, 5.7 of 12 cycles between a warp's instructions on memory.
// 4.2 million triangle instances in 1,024 shadow draws took 855 instructions a warp
// and 188 us with a binary search of the draws, nine divisions by w and 64-bit scans;
// with the draw table, w known to be 1 under the orthographic light, depths divided
// after culling and ballots for the counts it is 624 instructions and 148 us.
template <bool kOrdered>
__global__ void __launch_bounds__(kSetupThreads) k_setup(PassParams P) {
    __shared__ uint32_t s_tile;
    __shared__ uint64_t s_warp[kSetupThreads / 32];
    __shared__ uint64_t s_base_recs, s_base_stamps;
    __shared__ uint32_t s_small_warp[kSetupThreads / 32];
    __shared__ uint32_t s_small_base;
    // the pass's depth target is zeroed by the same launch: its stores overlap the
    // setup arithmetic, and the raster (the next launch) sees it cleared. The frames
    // that used it are done when the launch before this one starts.
    for (uint32_t b = 0; b < P.clear_count; ++b)
        zero_share(P.clear_ptr[b], P.clear_bytes[b], (size_t)blockIdx.x * blockDim.x + threadIdx.x,
                   (size_t)gridDim.x * blockDim.x);
    pdl_wait_previous();
    // The ordered list's look-back needs tiles numbered in the order the CTAs
    // start (a CTA only waits on tiles that have started); the unordered passes
    // wait on nobody and use the block index, sparing one same-address atomic
    // per CTA.
    if (kOrdered && threadIdx.x == 0) s_tile = atomicAdd(&P.header->ticket, 1u);
    const uint32_t tri_ctas = (P.tri_total + kSetupThreads - 1) / kSetupThreads;
    // CTAs launched only to share the zeroing hold no triangles: done
    if (!kOrdered && blockIdx.x >= tri_ctas) return;
    __syncthreads();
    const uint32_t tile = kOrdered ? s_tile : blockIdx.x;
    const uint32_t local = tile * kSetupThreads + threadIdx.x;
    const uint32_t tri = P.tri_offset + local;

    CountEmit<kOrdered> cnt;
    cnt.refs = P.tri_refs;
    cnt.tri = tri;
    if (local < P.tri_total) setup_triangle<kOrdered>(P, tri, cnt);

    // CTA-wide inclusive scan of (records, stamps) packed in one 64-bit word, and of the
    // small records. Nearly every triangle gives none or one, so that within a warp the
    // records are counted by ballots (only clipped ones fan out); the stamps of 32
    // triangles fit 32 bits.
    const uint64_t mine = ((uint64_t)cnt.recs << kStampBits) | cnt.stamps;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t recs_incl, small_incl, stamps_incl = (uint32_t)cnt.stamps;
    if (__any_sync(0xffffffffu, cnt.recs + cnt.small > 1)) {
        recs_incl = cnt.recs;
        small_incl = cnt.small;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t r = __shfl_up_sync(0xffffffffu, recs_incl, o), v = __shfl_up_sync(0xffffffffu, small_incl, o);
            if (lane >= o) {
                recs_incl += r;
                small_incl += v;
            }
        }
    } else {
        const uint32_t up_to = 0xffffffffu >> (31 - lane);
        recs_incl = __popc(__ballot_sync(0xffffffffu, cnt.recs != 0) & up_to);
        small_incl = __popc(__ballot_sync(0xffffffffu, cnt.small != 0) & up_to);
    }
    if (__any_sync(0xffffffffu, cnt.recs != 0)) {
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, stamps_incl, o);
            if (lane >= o) stamps_incl += v;
        }
    }
    const uint64_t incl = ((uint64_t)recs_incl << kStampBits) | stamps_incl;
    if (lane == 31) {
        s_warp[warp] = incl;
        s_small_warp[warp] = small_incl;
    }
    __syncthreads();
    uint64_t warp_prefix = 0, total = 0;
#pragma unroll
    for (int w = 0; w < kSetupThreads / 32; ++w) {
        if (w < warp) warp_prefix += s_warp[w];
        total += s_warp[w];
    }
    const uint64_t excl = warp_prefix + incl - mine;
    uint32_t small_prefix = 0, small_total = 0;
#pragma unroll
    for (int w = 0; w < kSetupThreads / 32; ++w) {
        if (w < warp) small_prefix += s_small_warp[w];
        small_total += s_small_warp[w];
    }
    const uint32_t small_excl = small_prefix + small_incl - cnt.small;
    if (threadIdx.x == 32) s_small_base = small_total ? atomicAdd(&P.header->small_records, small_total) : 0u;

    // Unordered passes (shadow, opaque camera pass): the depth test is an atomic
    // max, so records may land in any order; one 64-bit atomicAdd per CTA
    // allocates its record slots and its stamp range. The ordered blended list
    // keeps submission order with a decoupled look-back instead.
    if (!kOrdered) {
        if (threadIdx.x == 0) {
            const uint64_t old =
                total ? atomicAdd(reinterpret_cast<unsigned long long*>(&P.header->alloc), (unsigned long long)total) : 0ull;
            s_base_recs = old >> kStampBits;
            s_base_stamps = old & kStampMask;
            __threadfence();
            if (atomicAdd(&P.header->done, 1u) == tri_ctas - 1) {
                // last CTA: publish the totals for the raster and the host
                const uint64_t fin = atomicAdd(reinterpret_cast<unsigned long long*>(&P.header->alloc), 0ull);
                const uint64_t recs = fin >> kStampBits, st = fin & kStampMask;
                uint64_t chunks = (st + P.chunk_stamps - 1) / P.chunk_stamps;
                if (chunks > P.chunk_capacity) {
                    chunks = P.chunk_capacity;
                    atomicOr(P.error_flags, kErrStampOverflow);
                }
                P.header->records = (uint32_t)(recs < (uint64_t)P.record_capacity ? recs : (uint64_t)P.record_capacity);
                P.header->stamps = st;
                P.header->chunks = (uint32_t)chunks;
                P.header->records_needed = recs > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)recs;
            }
        }
    }
    // Decoupled look-back (warp 0): publish this tile's aggregate, then sum the
    // predecessors' values 32 at a time until an inclusive prefix is found.
    if (kOrdered && warp == 0) {
        const uint64_t agg_recs = total >> kStampBits, agg_stamps = total & kStampMask;
        volatile unsigned long long* status = reinterpret_cast<volatile unsigned long long*>(P.tile_status);
        uint64_t pre_recs = 0, pre_stamps = 0;
        if (tile == 0) {
            if (lane == 0) status[0] = kFlagIncl | to_status(agg_recs, agg_stamps);
        } else {
            if (lane == 0) status[tile] = kFlagAgg | to_status(agg_recs, agg_stamps);
            int64_t base = (int64_t)tile - 1;
            uint32_t spins = 0;
            for (;;) {
                const int64_t p = base - lane;
                const uint64_t sv = p >= 0 ? (uint64_t)status[p] : kFlagIncl;
                const uint64_t flag = sv & (3ull << 62);
                const unsigned incl = __ballot_sync(0xffffffffu, flag == kFlagIncl);
                const unsigned zero = __ballot_sync(0xffffffffu, flag == 0);
                const unsigned last = incl ? (unsigned)(__ffs(incl) - 1) : 31u;
                const unsigned need = last == 31u ? 0xffffffffu : ((2u << last) - 1u);
                if (zero & need) {
                    if (++spins > P.lookback_spins) {
                        if (lane == 0) atomicOr(P.error_flags, kErrLookbackTimeout);
                        break;
                    }
                    __nanosleep(32);
                    continue;
                }
                uint64_t rr = (unsigned)lane <= last ? (sv >> kStatusStampBits) & kStatusRecMask : 0;
                uint64_t ss = (unsigned)lane <= last ? sv & kStatusStampMask : 0;
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    rr += __shfl_xor_sync(0xffffffffu, rr, o);
                    ss += __shfl_xor_sync(0xffffffffu, ss, o);
                }
                pre_recs += rr;
                pre_stamps += ss;
                if (incl) break;
                base -= 32;
            }
            if (lane == 0) {
                __threadfence();
                status[tile] = kFlagIncl | to_status(pre_recs + agg_recs, pre_stamps + agg_stamps);
            }
        }
        if (lane == 0) {
            if (pre_recs + agg_recs > kStatusRecMask || pre_stamps + agg_stamps > kStatusStampMask)
                atomicOr(P.error_flags, kErrStampOverflow);
            s_base_recs = pre_recs;
            s_base_stamps = pre_stamps;
            if (tile == gridDim.x - 1) {
                const uint64_t st = pre_stamps + agg_stamps;
                uint64_t chunks = (st + P.chunk_stamps - 1) / P.chunk_stamps;
                if (chunks > P.chunk_capacity) chunks = P.chunk_capacity;
                P.header->records = (uint32_t)((pre_recs + agg_recs) < (uint64_t)P.record_capacity
                                                   ? (pre_recs + agg_recs) : (uint64_t)P.record_capacity);
                P.header->stamps = st;
                P.header->chunks = (uint32_t)chunks;
                const uint64_t need = pre_recs + agg_recs;
                P.header->records_needed = need > 0xFFFFFFFFull ? 0xFFFFFFFFu : (uint32_t)need;
            }
        }
    }
    __syncthreads();
    if (cnt.recs + cnt.small == 0) return;
    WriteEmit<kOrdered> w{&P, (uint32_t)(s_base_recs + (excl >> kStampBits)), s_base_stamps + (excl & kStampMask),
                s_small_base + small_excl};
    if (cnt.recs + cnt.small == 1) w(cnt.first, cnt.first_small);
    else setup_triangle<kOrdered>(P, tri, w);
}

int setup_ctas(uint32_t tri_total) { return (int)((tri_total + kSetupThreads - 1) / kSetupThreads); }

void launch_setup(const PassParams& p, cudaStream_t stream, bool next) {
    int ctas = setup_ctas(p.tri_total);
    if (ctas == 0) return;
    if (!p.ordered && p.clear_count) {
        // the depth target zeroed by this launch wants more CTAs than few triangles give
        // (about 32 KB each); the extra CTAs, past the last triangle tile, only zero
        // (the ordered list's look-back has one status word per triangle tile)
        size_t most = 0;
        for (uint32_t b = 0; b < p.clear_count; ++b) most = p.clear_bytes[b] > most ? p.clear_bytes[b] : most;
        const size_t want = std::min<size_t>(most / 32768, 4096);
        if ((size_t)ctas < want) ctas = (int)want;
    }
    void (*const kernel)(PassParams) = p.ordered ? k_setup<true> : k_setup<false>;
    if (next) launch_next(kernel, ctas, kSetupThreads, 0, stream, p);
    else kernel<<<ctas, kSetupThreads, 0, stream>>>(p);
    note_launch();
}

// ---------------------------------------------------------------------------
// raster
// ---------------------------------------------------------------------------

// Edge e (from vertex a to vertex b of the S>0-ordered triangle) at sample P:
//   E = dx*(PY - ay) - dy*(PX - ax),   dx = bx - ax, dy = by - ay,
// covered iff E > 0, or E == 0 on a top-left edge (dy < 0, or dy == 0 and dx > 0).
// With the top-left decision folded into the constant (E' = E - 1 on the other
// edges) the test is E' >= 0 on all three edges.

// The target of a view: visibility (camera pass; of a multisampled view, its first
// sample plane) or shadow map, and its row pitch.
struct Target {
    void* ptr;
    int pitch;
};

template <bool kWriteId>
__device__ __forceinline__ Target view_target(const PassParams& P, uint32_t view) {
    const ViewRec& V = P.views[view & kViewMask];
    if (kWriteId) return Target{V.vis, V.width};
    return Target{V.shadow + (size_t)((view >> kViewBits) & kCascadeMask) * (size_t)V.shadow_w * (size_t)V.shadow_h,
                  V.shadow_w};
}

// Words between the sample planes of a multisampled view's visibility.
__device__ __forceinline__ size_t plane_words(const PassParams& P, uint32_t view) {
    const ViewRec& V = P.views[view & kViewMask];
    return (size_t)V.width * (size_t)V.height;
}

// The stored depth of a fragment: the interpolated z plus the record's depth bias
// (+0 in the camera pass), saturated to [0, 1] in the same instruction. The
// saturation maps NaN and every value <= 0 to +0 and every value >= 1 to 1; the
// sum is never -0 because the bias is never -0 (make_record), so this equals
// adding the bias and then clamping with NaN -> 0.
__device__ __forceinline__ float biased_depth(float z, float bias) {
    float r;
    asm("add.rn.sat.f32 %0, %1, %2;" : "=f"(r) : "f"(z), "f"(bias));
    return r;
}

// The pixel's word of the target: u64 visibility key or u32 depth bits.
template <bool kWriteId>
using TargetWord = typename std::conditional<kWriteId, unsigned long long, unsigned int>::type;

template <bool kWriteId>
__device__ __forceinline__ TargetWord<kWriteId>* target_word(const Target& T, int px, int py) {
    return reinterpret_cast<TargetWord<kWriteId>*>(T.ptr) + ((size_t)py * (size_t)T.pitch + (size_t)px);
}

// The depth test and write: atomicMax of the fragment's key (z = biased_depth).
template <bool kWriteId>
__device__ __forceinline__ void write_word(TargetWord<kWriteId>* w, float z, uint32_t id) {
    if (kWriteId) {
        const unsigned long long key = ((unsigned long long)__float_as_uint(z) << 32) | id;
        atomicMax(reinterpret_cast<unsigned long long*>(w), key);
    } else {
        atomicMax(reinterpret_cast<unsigned int*>(w), __float_as_uint(z));
    }
}

template <bool kWriteId>
__device__ __forceinline__ void write_fragment(const Target& T, int px, int py, float z, uint32_t id) {
    write_word<kWriteId>(target_word<kWriteId>(T, px, py), z, id);
}

// One lane rasterises one small triangle: its extent is at most the pass's
// small_extent (<= kMaxSmallExtent = 16 pixels = 4096 sub-pixels) each way, so
// every edge value and product stays below 2^26 and fits in 32 bits.
template <bool kWriteId, bool kMsaa>
__device__ __forceinline__ void raster_small(const PassParams& P, const TriRecord* rec) {
    const int4* src = reinterpret_cast<const int4*>(rec);
    const int4 q0 = __ldg(src), q1 = __ldg(src + 1), q2 = __ldg(src + 2), q3 = __ldg(src + 3);
    const int32_t X[3] = {q0.x, q0.z, q1.x}, Y[3] = {q0.y, q0.w, q1.y};
    const float z0 = __int_as_float(q1.z), dzdx = __int_as_float(q1.w), dzdy = __int_as_float(q2.x);
    const float bias = __int_as_float(q2.y);
    const int px0 = q2.z & 0xffff, py0 = (uint32_t)q2.z >> 16, px1 = q2.w & 0xffff, py1 = (uint32_t)q2.w >> 16;
    const uint32_t id = (uint32_t)q3.x;
    const Target T = view_target<kWriteId>(P, (uint32_t)q3.y);
    // edge constants relative to vertex 0 (all values < 2^12 sub-pixels, products < 2^24)
    int32_t dx[3], dy[3], c[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = (i + 1) % 3, b = (i + 2) % 3;
        dx[i] = X[b] - X[a];
        dy[i] = Y[b] - Y[a];
        const bool tl = dy[i] < 0 || (dy[i] == 0 && dx[i] > 0);
        // E' at (PX, PY) = c + dx*(PY - Y0) - dy*(PX - X0)
        c[i] = dy[i] * (X[a] - X[0]) - dx[i] * (Y[a] - Y[0]) - (tl ? 0 : 1);
    }
    if (kMsaa) {
        // the four samples of a pixel: the edges at its corner plus constant offsets
        int32_t off[kMsaaSamples][3];
#pragma unroll
        for (int k = 0; k < kMsaaSamples; ++k)
#pragma unroll
            for (int i = 0; i < 3; ++i) off[k][i] = dx[i] * msaa_y(k) - dy[i] * msaa_x(k);
        const size_t plane = plane_words(P, (uint32_t)q3.y);
        for (int py = py0; py <= py1; ++py) {
            const int32_t ry = py * 256 - Y[0];
            for (int px = px0; px <= px1; ++px) {
                const int32_t rx = px * 256 - X[0];
                const int32_t e0 = c[0] + dx[0] * ry - dy[0] * rx;
                const int32_t e1 = c[1] + dx[1] * ry - dy[1] * rx;
                const int32_t e2 = c[2] + dx[2] * ry - dy[2] * rx;
#pragma unroll
                for (int k = 0; k < kMsaaSamples; ++k) {
                    if (((e0 + off[k][0]) | (e1 + off[k][1]) | (e2 + off[k][2])) >= 0) {
                        const float fx = (float)(rx + msaa_x(k)), fy = (float)(ry + msaa_y(k));
                        const float z = biased_depth(fmaf(dzdx, fx, fmaf(dzdy, fy, z0)), bias);
                        write_word<kWriteId>(target_word<kWriteId>(T, px, py) + k * plane, z, id);
                    }
                }
            }
        }
    } else {
        for (int py = py0; py <= py1; ++py) {
            const int32_t ry = py * 256 + kCentre - Y[0];
            for (int px = px0; px <= px1; ++px) {
                const int32_t rx = px * 256 + kCentre - X[0];
                const int32_t e0 = c[0] + dx[0] * ry - dy[0] * rx;
                const int32_t e1 = c[1] + dx[1] * ry - dy[1] * rx;
                const int32_t e2 = c[2] + dx[2] * ry - dy[2] * rx;
                if ((e0 | e1 | e2) >= 0) {
                    const float z = biased_depth(fmaf(dzdx, (float)rx, fmaf(dzdy, (float)ry, z0)), bias);
                    write_fragment<kWriteId>(T, px, py, z, id);
                }
            }
        }
    }
}


struct LargeRecord {
    int32_t X[3], Y[3];
    int32_t dx[3], dy[3];
    uint32_t tl_bias[3];  // 0 on top-left edges, 1 otherwise
    bool near_origin, cut, small;  // see large_facts
    bool grid;            // see on_grid
    float z0, dzdx, dzdy, bias;
    int px0, py0, px1, py1;  // first pixel of the first stamp, last pixel of the box
    uint32_t id, nsx, view;
    uint64_t begin, end;
};

// Decodes a large record from its four 16-byte words.
template <bool kCamera>
__device__ __forceinline__ void decode_large(const int4 q0, const int4 q1, const int4 q2, const int4 q3, LargeRecord& L) {
    L.X[0] = q0.x;
    L.Y[0] = q0.y;
    L.X[1] = q0.z;
    L.Y[1] = q0.w;
    L.X[2] = q1.x;
    L.Y[2] = q1.y;
    L.z0 = __int_as_float(q1.z);
    L.dzdx = __int_as_float(q1.w);
    L.dzdy = __int_as_float(q2.x);
    L.bias = __int_as_float(q2.y);
    L.px0 = q2.z & 0xffff;
    L.py0 = (uint32_t)q2.z >> 16;
    L.px1 = q2.w & 0xffff;
    L.py1 = (uint32_t)q2.w >> 16;
    L.id = (uint32_t)q3.x;
    L.grid = on_grid(kCamera, L.px0, L.py0, L.px1, L.py1);
    if (L.grid) {
        L.px0 &= -kStampW;
        L.py0 &= -kStampH;
    }
    const uint32_t flags = (uint32_t)q3.y >> kRecFlagShift;
    L.view = (uint32_t)q3.y & kRecViewMask;
    L.begin = (uint64_t)(uint32_t)q3.z | ((uint64_t)((uint32_t)q3.w & 0xffu) << 32);
    L.nsx = (uint32_t)q3.w >> (kStampOffsetBits - 32);
    L.end = L.begin + (uint64_t)L.nsx * (uint32_t)((L.py1 - L.py0) / kStampH + 1);
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = (i + 1) % 3, b = (i + 2) % 3;
        L.dx[i] = L.X[b] - L.X[a];
        L.dy[i] = L.Y[b] - L.Y[a];
        L.tl_bias[i] = (flags >> i) & 1u;
    }
    L.near_origin = (flags & kFactNear) != 0;
    L.cut = (flags & kFactCut) != 0;
    L.small = (flags & kFactSmall) != 0;
}

template <bool kCamera>
__device__ __forceinline__ void load_large(const TriRecord* rec, LargeRecord& L) {
    const int4* src = reinterpret_cast<const int4*>(rec);
    decode_large<kCamera>(__ldg(src), __ldg(src + 1), __ldg(src + 2), __ldg(src + 3), L);
}

// Record staging of the chunk walk: a warp copies the records a chunk starts
// with (one per lane, the first few of them) into shared memory with cp.async
// while it rasterises the chunk before, so that a segment finds its record
// there instead of waiting for a dependent global load.
constexpr int kRasterThreads = 256;
constexpr int kStageRecordsMax = 16;  // a chunk of 32 stamps rarely holds more; 8 where the stamps take more room (4x samples)

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem) : "memory");
}

// Lane `lane` copies record r0 + lane when it exists (below n_rec); one commit
// group per call, also when it copies nothing.
template <int kRecords>
__device__ __forceinline__ void stage_records(int4 (*buf)[4], const TriRecord* records, uint32_t r0, uint32_t n_rec,
                                              int lane) {
    if (lane < kRecords && (uint64_t)r0 + (uint64_t)lane < (uint64_t)n_rec) {
        const int4* src = reinterpret_cast<const int4*>(records + r0 + lane);
#pragma unroll
        for (int i = 0; i < 4; ++i) cp_async16(&buf[lane][i], src + i);
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

// Up to 32 stamps as the lanes of a warp (their pixels) read them from shared memory.
// A 16-byte broadcast takes four cycles of the shared-memory return path, so a stamp
// is kept to its own values, and its record's are read when the record changes.
template <int kSamples>
struct StampWork {
    int4 e[kSamples][32];  // per sample: floor(E' / 256) of the three edges at the stamp's first pixel, clamped;
                           // [0].w: the first pixel's word in the target
    float2 at[32];         // offset of the first pixel's sample from vertex 0
    int4 edges[32];        // the record's dx and -dy of edges 0 and 1 (edge 2's are minus their sums)
    int4 plane[32];        // the record's z0, dz/dx, dz/dy, and its id (camera) or depth bias (shadow)
    uint2 box[32];         // the lanes whose pixel lies in the record's box; the record's view field
};

constexpr uint32_t kAllLanes = 0xffffffffu;

// The edges of stamp (sx, sy) of a record whose stamps may be taken together, per
// sample, at its first pixel: floor(E' / 256), clamped. Returns false if no pixel of
// the stamp passes all three edges' bounds.
//
// The edge function of a pixel lx right of and ly below the stamp's first pixel is
// E' = E0 + 256 (dx ly - dy lx), so E' >= 0 exactly when floor(E0 / 256) + dx ly -
// dy lx >= 0. Edges are below 2^26, so the lane term stays below 2^30 in size, and
// the 64-bit floor may be clamped to +-2^30 without a change of that sign.
template <int kSamples, class Int>  // Int: the type that holds the record's edge values
__device__ __forceinline__ bool stamp_edges(const LargeRecord& L, int32_t PX, int32_t PY, int32_t (&q)[kSamples][3]) {
    uint32_t rejected = 0;  // samples
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = (i + 1) % 3;
        const int32_t dx = L.dx[i], dy = L.dy[i];
        const Int E = (Int)dx * (PY - L.Y[a]) - (Int)dy * (PX - L.X[a]) - (Int)L.tl_bias[i];
        const int32_t most = max(dx, 0) * (kStampH - 1) + max(-dy, 0) * (kStampW - 1);  // of the lane term
#pragma unroll
        for (int k = 0; k < kSamples; ++k) {
            Int f = (kSamples > 1 ? E + (Int)dx * msaa_y(k) - (Int)dy * msaa_x(k) : E) >> 8;
            if (sizeof(Int) > 4) f = max(min(f, (Int)1 << 30), -((Int)1 << 30));
            q[k][i] = (int32_t)f;
            if (q[k][i] + most < 0) rejected |= 1u << k;
        }
    }
    return rejected != (1u << kSamples) - 1u;
}

// Where the depth of the 8x4 block at (sx0, sy0) of a record's target is kept.
__device__ __forceinline__ uint32_t* front_of(const PassParams& P, uint32_t view, int sx0, int sy0) {
    const ViewRec& V = P.views[view & kViewMask];
    const uint32_t tile = V.shade_block_base + (uint32_t)(sy0 / 16) * (uint32_t)((V.width + 15) / 16) + (uint32_t)(sx0 / 16);
    return P.front + (size_t)tile * kTileBlocks + (uint32_t)((sy0 / kStampH) % 4) * 2u + (uint32_t)((sx0 / kStampW) % 2);
}

// Whether a stamp that lies on the grid has a pixel to draw, given the depth `front` that
// every pixel of its block reaches; and where it covers the block whole, its own least depth
// raises that depth. What a stamp draws is always written, so the block reaches the depth
// at the end whichever stamp is drawn first, and a stamp whose greatest depth stays below it
// draws nothing that is seen. A lane does this for the stamp it prepares, so a hidden stamp
// costs a thirty-second of one that is drawn. Frames of 4,096 random triangles over one
// another: 640x360 44 -> 31.6 us, 960x540 with its network 147 -> 127 us; scenes of
// small triangles are within 0.3 %. The greatest and least depth are the plane's at the corners:
// its two sums round monotonically.
template <int kSamples>
__device__ __forceinline__ bool raster_front(const LargeRecord& L, int32_t PX, int32_t PY, const int32_t (&q)[kSamples][3],
                                             uint32_t front, uint32_t* cell) {
    const float x0 = (float)(PX - L.X[0]), y0 = (float)(PY - L.Y[0]);
    const float x1 = x0 + (float)((kStampW - 1) * 256 + (kSamples > 1 ? 256 : 0)), y1 = y0 + (float)((kStampH - 1) * 256 + (kSamples > 1 ? 256 : 0));
    if (!(fabsf(L.dzdx) + fabsf(L.dzdy) < INFINITY)) return true;
    const bool rx = L.dzdx > 0.0f, ry = L.dzdy > 0.0f;
    const float far_z = biased_depth(fmaf(L.dzdx, rx ? x0 : x1, fmaf(L.dzdy, ry ? y0 : y1, L.z0)), 0.0f);
    const float near_z = biased_depth(fmaf(L.dzdx, rx ? x1 : x0, fmaf(L.dzdy, ry ? y1 : y0, L.z0)), 0.0f);
    if (__float_as_uint(near_z) < front) return false;
    if (__float_as_uint(far_z) <= front) return true;
    bool whole = true;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int32_t least = min(L.dx[i], 0) * (kStampH - 1) + min(-L.dy[i], 0) * (kStampW - 1);
#pragma unroll
        for (int k = 0; k < kSamples; ++k) whole = whole && q[k][i] + least >= 0;
    }
    if (whole) atomicMax(cell, __float_as_uint(far_z));
    return true;
}

// Leaves the stamp at (sx0, sy0) with edges q as entry i of w.
template <bool kWriteId, int kSamples>
__device__ __forceinline__ void put_stamp(const PassParams& P, const LargeRecord& L, int sx0, int sy0, int32_t PX, int32_t PY,
                                          const int32_t (&q)[kSamples][3], int i, StampWork<kSamples>& w) {
    const int pitch = kWriteId ? P.views[L.view & kViewMask].width : P.views[L.view & kViewMask].shadow_w;
#pragma unroll
    for (int k = 0; k < kSamples; ++k) w.e[k][i] = make_int4(q[k][0], q[k][1], q[k][2], sy0 * pitch + sx0);
    w.at[i] = make_float2((float)(PX - L.X[0]), (float)(PY - L.Y[0]));
    w.edges[i] = make_int4(L.dx[0], L.dx[1], -L.dy[0], -L.dy[1]);
    w.plane[i] = make_int4(__float_as_int(L.z0), __float_as_int(L.dzdx), __float_as_int(L.dzdy),
                           kWriteId ? (int)L.id : __float_as_int(L.bias));
    const int nx = min(L.px1 - sx0, kStampW - 1), ny = min(L.py1 - sy0, kStampH - 1);  // last column and row in the box
    w.box[i] = make_uint2(((0xffu >> (kStampW - 1 - nx)) * 0x01010101u) & (kAllLanes >> (8 * (kStampH - 1 - ny))), L.view);
}

// The n stamps of w, one after the other, a pixel per lane (column lx, row ly). Bit i
// of `heads`: stamp i is the first of its record; of `cut`: its record's box is cut.
// Offsets from vertex 0 are integers below 2^24, so their float sums are exact.
template <bool kWriteId, int kSamples, bool kCut>
__device__ __forceinline__ void raster_stamps(const PassParams& P, const StampWork<kSamples>& w, int n, uint32_t heads,
                                              uint32_t cut, int lane, int lx, int ly) {
    uint32_t cur_view = kAllLanes;  // the view whose target is held
    int32_t l0 = 0, l1 = 0, lane_word = 0;
    int4 plane{};
    size_t sample_words = 0;
    TargetWord<kWriteId>* base = nullptr;
    const float fx = (float)(lx * 256), fy = (float)(ly * 256);
    for (int i = 0; i < n; ++i, heads >>= 1, cut >>= 1) {
        if (heads & 1u) {
            const int4 d = w.edges[i];
            l0 = d.x * ly + d.z * lx;
            l1 = d.y * ly + d.w * lx;
            plane = w.plane[i];
            const uint32_t view = w.box[i].y;
            if (view != cur_view) {
                cur_view = view;
                const Target T = view_target<kWriteId>(P, view);
                base = reinterpret_cast<TargetWord<kWriteId>*>(T.ptr);
                lane_word = ly * T.pitch + lx;
                if (kSamples > 1) sample_words = plane_words(P, view);
            }
        }
        const float2 at = w.at[i];
        int4 e = w.e[0][i];
        auto* const word = base + (e.w + lane_word);
        if (kCut && (cut & 1u) && !((w.box[i].x >> lane) & 1u)) continue;
#pragma unroll
        for (int k = 0; k < kSamples; ++k) {
            if (k) e = w.e[k][i];
            // the third edge's lane term is minus the sum of the others'
            if (((e.x + l0) | (e.y + l1) | (e.z - l0 - l1)) < 0) continue;
            const float px = at.x + (kSamples > 1 ? fx + (float)msaa_x(k) : fx);
            const float py = at.y + (kSamples > 1 ? fy + (float)msaa_y(k) : fy);
            const float z = fmaf(__int_as_float(plane.y), px, fmaf(__int_as_float(plane.z), py, __int_as_float(plane.x)));
            write_word<kWriteId>(word + k * sample_words, biased_depth(z, kWriteId ? 0.0f : __int_as_float(plane.w)),
                                 kWriteId ? (uint32_t)plane.w : 0u);
        }
    }
}

// A pixel of a stamp of any record: 64-bit edge functions, float offsets rounded once.
template <bool kWriteId>
__device__ __forceinline__ void raster_far_pixel(const Target& T, const LargeRecord& L, int px, int py, int32_t ox, int32_t oy) {
    if (px > L.px1 || py > L.py1) return;
    const int32_t PX = px * 256 + ox, PY = py * 256 + oy;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = (i + 1) % 3;
        if ((int64_t)L.dx[i] * ((int64_t)PY - L.Y[a]) - (int64_t)L.dy[i] * ((int64_t)PX - L.X[a]) - (int64_t)L.tl_bias[i] < 0) return;
    }
    const float z = fmaf(L.dzdx, (float)(PX - L.X[0]), fmaf(L.dzdy, (float)(PY - L.Y[0]), L.z0));
    write_fragment<kWriteId>(T, px, py, biased_depth(z, L.bias), L.id);
}

// Persistent raster: each warp first takes batches of 32 small records (one per
// lane), then chunks of chunk_stamps stamps of the large records, both in a fixed
// grid-stride order. (A shared cursor that every warp bumps with an atomic
// serialises on one L2 line: a raster launch with its work skipped took 12 us that
// way on the 4096^2 shadow pass of 262,144 triangles, 6 us without.)
//
// A chunk goes 32 stamps at a time, of as many records as they belong to. Each lane
// first prepares one stamp: finds its record, evaluates the edges at the stamp's
// first pixel, drops it if an edge rejects it whole, and leaves what the pixels need
// in shared memory. Then the warp takes the stamps that are left one after the
// other, a pixel per lane. What is the same for all pixels of a stamp is so computed
// once instead of by 32 lanes, a record costs nothing beyond its stamps (the chunks
// of a shadow pass of 262,144 triangles hold 3.4 records each, 100-odd instructions
// to decode and start), and an empty stamp (over a third of a triangle's box) costs
// a thirty-second of its preparation. Against one lane per pixel throughout, with
// 64-bit edges for triangles above 90 pixels: 640x360 triangle soup frame 89 -> 43
// us, 3840x2160 with a million triangles and four cascades 975 -> 856 us, 1080p
// scene-scale shadow raster 70 -> 62 us (now the shared-memory path is 76 % busy:
// broadcasts, then the atomics). Four CTAs per SM were slower (62 -> 69 us).
template <bool kWriteId, bool kMsaa>
__global__ void __launch_bounds__(kRasterThreads, 3) k_raster(PassParams P) {
    constexpr int kSamples = kMsaa ? kMsaaSamples : 1;
    constexpr int kStageRecords = kMsaa ? kStageRecordsMax / 2 : kStageRecordsMax;
    __shared__ int4 s_stage[kRasterThreads / 32][2][kStageRecords][4];
    __shared__ StampWork<kSamples> s_work[kRasterThreads / 32];
    const int lane = threadIdx.x & 31;
    const int lx = lane & (kStampW - 1), ly = lane >> 3;
    // a multisampled pass's launches number their warps together
    const uint32_t warps = ((gridDim.x * blockDim.x) >> 5) * (kMsaa ? kMsaaSamples : 1u);
    const uint32_t warp_id = ((blockIdx.x * blockDim.x + threadIdx.x) >> 5) * (kMsaa ? kMsaaSamples : 1u) + (kMsaa ? P.part : 0u);
    pdl_wait_previous();
    const uint64_t n_small = min(P.header->small_records, P.small_capacity);
    for (uint64_t base = (uint64_t)warp_id * 32u; base < n_small; base += (uint64_t)warps * 32u)
        if (base + lane < n_small) raster_small<kWriteId, kMsaa>(P, P.small_records + base + lane);
    const uint32_t chunks = P.header->chunks;
    const uint64_t total = P.header->stamps;
    const uint32_t n_rec = min(P.header->records, P.record_capacity);  // records the setup wrote
    StampWork<kSamples>& work = s_work[threadIdx.x >> 5];
    // chunk k's first record (r_cur, staged in buffer cb), the next chunk's (r_next)
    int cb = 0;
    uint32_t r_cur = warp_id < chunks ? P.chunk_map[warp_id] : n_rec;
    stage_records<kStageRecords>(s_stage[threadIdx.x >> 5][0], P.records, r_cur, n_rec, lane);
    uint32_t r_next = (uint64_t)warp_id + warps < chunks ? P.chunk_map[warp_id + warps] : n_rec;
    for (uint32_t k = warp_id; k < chunks; k += warps) {
        const uint64_t s0 = (uint64_t)k * P.chunk_stamps;
        const uint64_t s_end = (s0 + P.chunk_stamps < total) ? (s0 + P.chunk_stamps) : total;
        // stage the next chunk's records while this one is rasterised, and fetch
        // the chunk map entry of the one after
        stage_records<kStageRecords>(s_stage[threadIdx.x >> 5][cb ^ 1], P.records, r_next, n_rec, lane);
        const uint64_t k_after = (uint64_t)k + 2u * (uint64_t)warps;
        const uint32_t r_after = k_after < chunks ? P.chunk_map[k_after] : n_rec;
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");  // this lane's copies of chunk k
        __syncwarp();                                          // and every other lane's
        const int4 (*const st)[4] = s_stage[threadIdx.x >> 5][cb];
        uint32_t r_first = r_cur;  // the record of the first of the 32 stamps
        for (uint64_t s = s0; s < s_end; s += 32) {
            // the stamps' records: lane l looks where record r_first + l starts, and each
            // stamp's record is the last that starts at or before it (a record has a stamp)
            uint32_t starts = 0;
            if (lane > 0 && (uint64_t)r_first + lane < n_rec) {
                const uint32_t j = r_first - r_cur + lane;
                const int4 q3 = j < (uint32_t)kStageRecords ? st[j][3] : __ldg(reinterpret_cast<const int4*>(P.records + r_first + lane) + 3);
                const uint64_t begin = (uint64_t)(uint32_t)q3.z | ((uint64_t)((uint32_t)q3.w & 0xffu) << 32);
                if (begin > s && begin < s + 32) starts = 1u << (uint32_t)(begin - s);
            }
            starts = __reduce_or_sync(kAllLanes, starts);
            const uint32_t r = r_first + __popc(starts & (kAllLanes >> (31 - lane)));
            uint32_t r_after_this = r;  // the record of the stamp after this one
            bool live = false, far = false;
            int sx0 = 0, sy0 = 0;
            int32_t PX = 0, PY = 0;  // the sample of the stamp's first pixel (its corner with 4x samples)
            int32_t q[kSamples][3];
            uint32_t* cell = nullptr;  // its block's depth
            uint32_t front = 0;
            LargeRecord L;
            if (s + lane < s_end && r < n_rec) {
                const uint32_t j = r - r_cur;
                if (j < (uint32_t)kStageRecords) decode_large<kWriteId>(st[j][0], st[j][1], st[j][2], st[j][3], L);
                else load_large<kWriteId>(P.records + r, L);
                if (s + lane >= L.begin && s + lane < L.end) {
                    // stamp i of the record, below 2^24: the quotient by stamps per row, off by one at most
                    const int i = (int)(s + lane - L.begin), nsx = (int)L.nsx;
                    int sy = (int)__fdividef((float)i, (float)nsx), sx = i - sy * nsx;
                    if (sx < 0) {
                        --sy;
                        sx += nsx;
                    } else if (sx >= nsx) {
                        ++sy;
                        sx -= nsx;
                    }
                    sx0 = L.px0 + sx * kStampW;
                    sy0 = L.py0 + sy * kStampH;
                    PX = sx0 * 256 + (kMsaa ? 0 : kCentre);
                    PY = sy0 * 256 + (kMsaa ? 0 : kCentre);
                    if (s + lane + 1 == L.end) ++r_after_this;
                    far = !L.near_origin;
                    live = !far;
                    if (kWriteId && live && L.grid) {
                        cell = front_of(P, L.view, sx0, sy0);
                        front = __ldcg(cell);
                    }
                } else {  // cannot happen with a consistent chunk map
                    atomicOr(P.error_flags, kErrStampOverflow);
                }
            }
            if (__all_sync(kAllLanes, !live || L.small)) live = live && stamp_edges<kSamples, int32_t>(L, PX, PY, q);
            else live = live && stamp_edges<kSamples, int64_t>(L, PX, PY, q);
            if (kWriteId && cell && live) live = raster_front<kSamples>(L, PX, PY, q, front, cell);
            // the stamps that are left, in order: entry `at`; the first one of its record is a head
            const uint32_t left = __ballot_sync(kAllLanes, live), below = left & ((1u << lane) - 1u);
            const int at = __popc(below);
            uint32_t head = 0, cut = 0;
            if (live) {
                put_stamp<kWriteId, kSamples>(P, L, sx0, sy0, PX, PY, q, at, work);
                // record starts after the stamp left before this one
                const uint32_t since = below ? starts & (kAllLanes >> (31 - lane)) & ~(kAllLanes >> __clz(below)) : kAllLanes;
                head = since ? 1u << at : 0u;
                cut = L.cut ? 1u << at : 0u;
            }
            const uint32_t heads = __reduce_or_sync(kAllLanes, head), cuts = __reduce_or_sync(kAllLanes, cut);
            __syncwarp();
            if (cuts) raster_stamps<kWriteId, kSamples, true>(P, work, __popc(left), heads, cuts, lane, lx, ly);
            else raster_stamps<kWriteId, kSamples, false>(P, work, __popc(left), heads, 0u, lane, lx, ly);
            for (uint32_t m = __ballot_sync(kAllLanes, far); m; m &= m - 1) {
                const int j = __ffs(m) - 1;
                load_large<kWriteId>(P.records + __shfl_sync(kAllLanes, r, j), L);
                const int px = __shfl_sync(kAllLanes, sx0, j) + lx, py = __shfl_sync(kAllLanes, sy0, j) + ly;
                const Target T = view_target<kWriteId>(P, L.view);
                const size_t plane = kMsaa ? plane_words(P, L.view) : 0;
#pragma unroll 1
                for (int i = 0; i < kSamples; ++i) {
                    const Target Ti{reinterpret_cast<TargetWord<kWriteId>*>(T.ptr) + i * plane, T.pitch};
                    raster_far_pixel<kWriteId>(Ti, L, px, py, kMsaa ? msaa_x(i) : kCentre, kMsaa ? msaa_y(i) : kCentre);
                }
            }
            r_first = __shfl_sync(kAllLanes, r_after_this, 31);
            __syncwarp();  // every lane is done with the stamps (and, at the chunk's end, its records)
        }
        r_cur = r_next;
        r_next = r_after;
        cb ^= 1;
    }
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

void launch_raster(const PassParams& p, int sm_count, cudaStream_t stream, int share, bool next) {
    // with ids it is the opaque camera pass, whose large stamps were counted on the block grid (on_grid)
    if (p.write_id && (p.ordered || !p.tri_refs || !p.front)) return;
    // persistent grid: as many CTAs as can be resident at once, with the launches beside this one
    static int occ[3] = {0, 0, 0};
    const int t = !p.write_id ? 0 : p.msaa ? 2 : 1;
    void (*const kernel)(PassParams) = t == 0 ? k_raster<false, false> : t == 1 ? k_raster<true, false> : k_raster<true, true>;
    if (!occ[t]) {
        int n = 0;
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kernel, kRasterThreads, 0);
        occ[t] = n > 0 ? n : 1;
    }
    const int ctas = (sm_count * occ[t] + share - 1) / share;
    if (next) launch_next(kernel, ctas, kRasterThreads, 0, stream, p);
    else kernel<<<ctas, kRasterThreads, 0, stream>>>(p);
    note_launch();
}

// ---------------------------------------------------------------------------
// debug-line overlay: vertex stage, clipping and viewport of each segment
// ---------------------------------------------------------------------------

// M * (x, y, z, w) as the chain M0r*x -> fma(M1r, y) -> fma(M2r, z) -> fma(M3r, w).
__device__ __forceinline__ CV transform4(const float* __restrict__ M, const float* v) {
    CV o;
    o.x = fmaf(M[12], v[3], fmaf(M[8], v[2], fmaf(M[4], v[1], M[0] * v[0])));
    o.y = fmaf(M[13], v[3], fmaf(M[9], v[2], fmaf(M[5], v[1], M[1] * v[0])));
    o.z = fmaf(M[14], v[3], fmaf(M[10], v[2], fmaf(M[6], v[1], M[2] * v[0])));
    o.w = fmaf(M[15], v[3], fmaf(M[11], v[2], fmaf(M[7], v[1], M[3] * v[0])));
    return o;
}

// debugVertMain (src/shaders/debug.slang:5-35): flags select the space by equality.
__device__ CV debug_vertex(const rz_scene_data& sd, const rz_debug_object& d, const float* v) {
    float M[16];
    CV c;
    if (d.flags == RZ_DEBUG_TRANSFORM_IS_POINTS) return transform4(sd.view_projection, v);
    if (d.flags == RZ_DEBUG_SCREEN_SPACE) {
        const float aspect = sd.draw_extent[0] / sd.draw_extent[1];
        const float q[4] = {v[0], v[1] * aspect, v[2], v[3]};
        c = transform4(d.transform, q);
        c.z = c.w = 1.0f;
        return c;
    }
    if (d.flags == RZ_DEBUG_VIEW_SPACE) {
        mat4_mul(sd.proj, d.transform, M);
        c = transform4(M, v);
        c.z = c.w = 1.0f;
        return c;
    }
    mat4_mul(sd.view_projection, d.transform, M);
    return transform4(M, v);
}

// One thread per (view, segment). The segment is clipped against the triangle
// planes in order (an end outside one plane is replaced by the crossing
// fma(t, b-a, a), t = da/(da-db)), mapped to the viewport and snapped to
// 1/256 pixel; its pixel box is widened by half the line width.
__global__ void __launch_bounds__(128) k_debug_prep(const DebugPair* __restrict__ pairs, uint32_t count,
                                                    const rz_debug_object* __restrict__ objects,
                                                    const ViewRec* __restrict__ views, uint32_t view_count,
                                                    DebugSeg* __restrict__ out, uint2* __restrict__ boxes) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (uint64_t)count * view_count) return;
    const uint32_t v = (uint32_t)(i / count), k = (uint32_t)(i % count);
    const DebugPair pr = pairs[k];
    const rz_debug_object& d = objects[pr.object];
    const ViewRec& VR = views[v];
    DebugSeg s{};
    uint2 box = make_uint2(kDebugNoBox, 0u);
    s.rgb[0] = d.color[0];
    s.rgb[1] = d.color[1];
    s.rgb[2] = d.color[2];
    CV a = debug_vertex(*VR.scene, d, pr.a), b = debug_vertex(*VR.scene, d, pr.b);
    bool live = true;
    for (int p = 0; p < 6 && live; ++p) {
        const float da = plane_dist(a, p), db = plane_dist(b, p);
        const bool ia = da >= 0.0f, ib = db >= 0.0f;
        if (!ia && !ib) {
            live = false;
        } else if (ia != ib) {
            const float t = da / (da - db);
            CV c;
            c.x = fmaf(t, b.x - a.x, a.x);
            c.y = fmaf(t, b.y - a.y, a.y);
            c.z = fmaf(t, b.z - a.z, a.z);
            c.w = fmaf(t, b.w - a.w, a.w);
            if (ia) b = c;
            else a = c;
        }
    }
    live = live && a.w > 0.0f && b.w > 0.0f;
    if (live) {
        const float hw = (float)VR.width * 0.5f, hh = (float)VR.height * 0.5f;
        const SV sa = to_screen(a, hw, hh), sb = to_screen(b, hw, hh);
        s.X0 = sa.X;
        s.Y0 = sa.Y;
        s.X1 = sb.X;
        s.Y1 = sb.Y;
        s.z0 = sa.z;
        s.z1 = sb.z;
        const float dx = (float)((int64_t)sb.X - sa.X), dy = (float)((int64_t)sb.Y - sa.Y);
        // an end whose w nearly vanishes can land far out, where the products of debug_meets may wrap
        const bool far = fmaxf(fmaxf(fabsf((float)sa.X), fabsf((float)sa.Y)), fmaxf(fabsf((float)sb.X), fabsf((float)sb.Y))) > 1.0e8f;
        s.reach = far ? INFINITY : (float)kDebugHalfWidth * sqrtf(dx * dx + dy * dy) * 1.00001f;
        const int x0 = max(0, (min(sa.X, sb.X) - kDebugHalfWidth) >> 8);
        const int x1 = min(VR.width - 1, (max(sa.X, sb.X) + kDebugHalfWidth) >> 8);
        const int y0 = max(0, (min(sa.Y, sb.Y) - kDebugHalfWidth) >> 8);
        const int y1 = min(VR.height - 1, (max(sa.Y, sb.Y) + kDebugHalfWidth) >> 8);
        if (x0 <= x1 && y0 <= y1)
            box = make_uint2((uint32_t)x0 | ((uint32_t)y0 << 16), (uint32_t)x1 | ((uint32_t)y1 << 16));
    }
    out[i] = s;
    boxes[i] = box;
}

void launch_debug_prep(const DebugPair* pairs, uint32_t count, const rz_debug_object* objects, const ViewRec* views,
                       uint32_t view_count, DebugSeg* out, uint2* boxes, cudaStream_t stream) {
    const uint64_t n = (uint64_t)count * view_count;
    if (n == 0) return;
    k_debug_prep<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(pairs, count, objects, views, view_count, out, boxes);
    note_launch();
}

}  // namespace rz
