// Deferred-style shading of the camera pass.
//
// Reference path: vertexMain (src/shaders/basic.slang:16-119) and fragmentMain
// (137-344) with pcf (src/shaders/pcf.slang:1-11) and the BRDF helpers
// (src/shaders/lighting.slang:5-43), evaluated once per pixel for the triangle
// that won the depth test, then the RGBA16F draw image (Graphics.cpp:1905-1908)
// and the blit to the sRGB swapchain (5845-5879).
//
// The vertex stage runs once per (draw, mesh vertex) in k_vertex, pulling the
// 64-byte vertex records as the reference does through buffer device addresses,
// and writes a 128-byte varying record. k_shade then shades each pixel once for
// the triangle that won its depth test: it gathers the three varying records
// and interpolates them with perspective-correct barycentrics computed from the
// clip positions in 2D homogeneous form. Texture level selection uses the
// derivative of the interpolated uv across the pixel's 2x2 quad (the value at
// the quad's top-left, right and lower neighbours, which is what a helper
// invocation would compute).
//
// The file is built with -fmad=false. Everything that feeds a discrete
// decision - barycentrics, the interpolated uv and its quad derivatives, level
// selection, texel addresses and filter weights, the shadow-map coordinate and
// depth compared in PCF - follows the oracle's fp32 operation order and is
// bit-identical to it (log2f of the trilinear fraction aside). The lighting
// arithmetic downstream is continuous and uses reciprocal square roots and
// approximate division; its output stays within the 1/255 bound.
#include <cuda_fp16.h>

#include <algorithm>

#include "rz_device.cuh"

namespace rz {

struct V3 {
    float x, y, z;
};
__device__ __forceinline__ V3 operator+(V3 a, V3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ V3 operator-(V3 a, V3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ V3 operator*(V3 a, float s) { return {a.x * s, a.y * s, a.z * s}; }
__device__ __forceinline__ V3 mul3(V3 a, V3 b) { return {a.x * b.x, a.y * b.y, a.z * b.z}; }
__device__ __forceinline__ float dot(V3 a, V3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ V3 cross(V3 a, V3 b) { return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x}; }
__device__ __forceinline__ V3 normalize(V3 a) {
    const float l = sqrtf(dot(a, a));
    return {a.x / l, a.y / l, a.z / l};
}
__device__ __forceinline__ float clamp01(float x) { return fminf(fmaxf(x, 0.0f), 1.0f); }
// Lighting-only forms (continuous quantities graded within 1/255): reciprocal
// square root and approximate division instead of IEEE sqrt/div.
__device__ __forceinline__ V3 fnormalize(V3 a) {
    const float r = rsqrtf(dot(a, a));
    return {a.x * r, a.y * r, a.z * r};
}
__device__ __forceinline__ float fdiv(float a, float b) { return __fdividef(a, b); }
__device__ __forceinline__ V3 mulm3v(const float* N, V3 v) {
    return {N[0] * v.x + N[3] * v.y + N[6] * v.z, N[1] * v.x + N[4] * v.y + N[7] * v.z, N[2] * v.x + N[5] * v.y + N[8] * v.z};
}

__device__ __forceinline__ F2 mix2(F2 x, F2 y, F2 w) { return x + w * (y - x); }

// ---------------------------------------------------------------------------
// per-draw constants
// ---------------------------------------------------------------------------

// Also zeroes the clear list L (the camera pass's headers and look-back words),
// so that the two need one launch.
__global__ void k_prep_camera(const DrawRec* __restrict__ draws, uint32_t n, const rz_object* __restrict__ objects,
                              const ViewRec* __restrict__ views, DrawConsts* __restrict__ out, ClearList L) {
    pdl_allow_next();
    const uint32_t d = blockIdx.x * blockDim.x + threadIdx.x;
    clear_share(L);
    if (d >= n) return;
    const rz_scene_data* sd = views[draws[d].view].scene;
    const rz_object& gd = objects[draws[d].object];
    float W[16], VP[16], C[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) {
        W[i] = gd.transform[i];
        VP[i] = sd->view_projection[i];
    }
    mat4_mul(VP, W, C);
    DrawConsts& o = out[d];
#pragma unroll
    for (int i = 0; i < 16; ++i) o.mvp[i] = C[i];
    // (ndc_to_tc * shadowProjNear) * W, ndc_to_tc rows (0.5,0,0,0.5) (0,0.5,0,0.5) (0,0,1,0) (0,0,0,1)
    float A[16];
    const float* P = sd->shadow_projection_near;
#pragma unroll
    for (int col = 0; col < 4; ++col) {
        const float x = P[col * 4 + 0], y = P[col * 4 + 1], z = P[col * 4 + 2], w = P[col * 4 + 3];
        A[col * 4 + 0] = 0.5f * x + 0.5f * w;
        A[col * 4 + 1] = 0.5f * y + 0.5f * w;
        A[col * 4 + 2] = z;
        A[col * 4 + 3] = w;
    }
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int r = 0; r < 4; ++r)
            o.csm[c * 4 + r] = A[0 * 4 + r] * W[c * 4 + 0] + A[1 * 4 + r] * W[c * 4 + 1] + A[2 * 4 + r] * W[c * 4 + 2] +
                               A[3 * 4 + r] * W[c * 4 + 3];
    const float* T = gd.to_object_space_transform;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        o.cam_obj[r] = T[0 * 4 + r] * sd->camera_position[0] + T[1 * 4 + r] * sd->camera_position[1] +
                       T[2 * 4 + r] * sd->camera_position[2] + T[3 * 4 + r] * sd->camera_position[3];
        o.sun_obj[r] = T[0 * 4 + r] * sd->sun_position[0] + T[1 * 4 + r] * sd->sun_position[1] +
                       T[2 * 4 + r] * sd->sun_position[2] + T[3 * 4 + r] * sd->sun_position[3];
    }
}

void launch_prep_camera(const DrawRec* draws, uint32_t n, const rz_object* objects, const ViewRec* views,
                        DrawConsts* out, cudaStream_t stream, const ClearList* clear, int sm_count) {
    const ClearList none{};
    const ClearList& L = clear ? *clear : none;
    const unsigned blocks = std::max((n + 127) / 128, clear_blocks(L, sm_count, 128));
    if (blocks == 0) return;
    k_prep_camera<<<blocks, 128, 0, stream>>>(draws, n, objects, views, out, L);
    note_launch();
}

// ---------------------------------------------------------------------------
// vertex stage
// ---------------------------------------------------------------------------

struct VsOut {
    V3 normal, worldNormal, viewDir, lightDir, tangent, bitangent;
    float color[4];
    float uv[2];
    float sigma;
    float csm[4];
};

// vertexMain, src/shaders/basic.slang:16-119 (outputs used by fragmentMain).
__device__ __forceinline__ void vertex_main(const rz_scene_data& sd, const rz_object& gd, const DrawConsts& dc,
                                            bool has_material, bool material_has_normal_map, const rz_vertex& v, VsOut& o) {
    float nt[4] = {v.tangent[0], v.tangent[1], v.tangent[2], v.tangent[3]};
    if (sd.ignore_asset_tangent_sign == 1) nt[3] = 1.0f;
    if (sd.flip_tangents[0] == 1) nt[0] = nt[0] * -1.0f;
    if (sd.flip_tangents[1] == 1) nt[1] = nt[1] * -1.0f;
    if (sd.flip_tangents[2] == 1) nt[2] = nt[2] * -1.0f;
    if (sd.flip_tangents[3] == 1) nt[3] = nt[3] * -1.0f;
    bool tse = sd.tangent_space_enabled == 1;
    if (has_material && !material_has_normal_map) tse = false;
    const V3 vpos{v.position[0], v.position[1], v.position[2]};
    V3 normal{v.normal[0], v.normal[1], v.normal[2]};
    V3 tangent{nt[0], nt[1], nt[2]};
    V3 bitangent = cross(normal, tangent) * nt[3];
    if (sd.ensure_orthogonal_bitangent == 1) {
        const V3 normal_projection = bitangent * dot(normal, bitangent);
        const V3 ortho_n = normalize(normal - normal_projection);
        const V3 tangent_projection = normal_projection - bitangent * dot(tangent, bitangent);
        const V3 ortho_t = normalize(tangent - tangent_projection);
        bitangent = cross(ortho_n, ortho_t) * nt[3];
    }
    V3 viewDir, lightDir;
    if (tse) {
        viewDir = V3{dc.cam_obj[0], dc.cam_obj[1], dc.cam_obj[2]} - vpos;
        lightDir = V3{dc.sun_obj[0], dc.sun_obj[1], dc.sun_obj[2]} - vpos;
    } else {
        const float* M = gd.transform;
        float wp[3];
#pragma unroll
        for (int r = 0; r < 3; ++r) wp[r] = M[0 * 4 + r] * vpos.x + M[1 * 4 + r] * vpos.y + M[2 * 4 + r] * vpos.z + M[3 * 4 + r] * 1.0f;
        viewDir = V3{sd.camera_position[0] - wp[0], sd.camera_position[1] - wp[1], sd.camera_position[2] - wp[2]};
        lightDir = V3{sd.sun_position[0] - wp[0], sd.sun_position[1] - wp[1], sd.sun_position[2] - wp[2]};
        normal = normalize(mulm3v(gd.normal_transform, V3{v.normal[0], v.normal[1], v.normal[2]}));
        tangent = normalize(mulm3v(gd.normal_transform, V3{nt[0], nt[1], nt[2]}));
        tangent = normalize(tangent - normal * dot(normal, tangent));
    }
    if (sd.flip_lights[0] == 1) lightDir.x = lightDir.x * -1.0f;
    if (sd.flip_lights[1] == 1) lightDir.y = lightDir.y * -1.0f;
    if (sd.flip_lights[2] == 1) lightDir.z = lightDir.z * -1.0f;
    o.normal = normal;
    o.worldNormal = mulm3v(gd.normal_transform, V3{v.normal[0], v.normal[1], v.normal[2]});
#pragma unroll
    for (int k = 0; k < 4; ++k) o.color[k] = v.color[k];
    o.tangent = V3{nt[0], nt[1], nt[2]};
    o.bitangent = bitangent;
    o.viewDir = viewDir;
    o.lightDir = lightDir;
    o.sigma = nt[3];
    o.uv[0] = v.uv[0];
    o.uv[1] = v.uv[1];
    const float* B = dc.csm;
#pragma unroll
    for (int r = 0; r < 4; ++r)
        o.csm[r] = B[0 * 4 + r] * vpos.x + B[1 * 4 + r] * vpos.y + B[2 * 4 + r] * vpos.z + B[3 * 4 + r];
}

// Perspective-correct barycentrics at pixel centre (px, py), 2D homogeneous form.
// Normalised device coordinate of pixel centre i of an extent of n pixels.
__device__ __forceinline__ float ndc(int i, int n) { return (float)(2 * i + 1 - n) / (float)n; }

// The normalised coordinates a pixel's barycentrics use: its centre (xp, yp) and
// its quad's (xq, yq), (xq1 = column + 1, yq1 = row + 1).
struct PixelNdc {
    float xp, yp, xq, yq, xq1, yq1;
};

__device__ __forceinline__ void barycentrics_n(const float4& c0, const float4& c1, const float4& c2, float xn, float yn,
                                               float b[3]) {
    const V3 v0{c0.x, c0.y, c0.w}, v1{c1.x, c1.y, c1.w}, v2{c2.x, c2.y, c2.w};
    const V3 p{xn, yn, 1.0f};
    const float b0 = dot(cross(v1, v2), p), b1 = dot(cross(v2, v0), p), b2 = dot(cross(v0, v1), p);
    const float inv = 1.0f / (b0 + b1 + b2);
    b[0] = b0 * inv;
    b[1] = b1 * inv;
    b[2] = b2 * inv;
}

__device__ __forceinline__ void barycentrics(const float4& c0, const float4& c1, const float4& c2, int px, int py, int W,
                                             int H, float b[3]) {
    barycentrics_n(c0, c1, c2, ndc(px, W), ndc(py, H), b);
}

struct Frag {
    V3 normal, worldNormal, viewDir, lightDir, tangent, bitangent;
    float color[4];
    float uv[2];
    float sigma;
    float csm[4];
    float duvdx[2], duvdy[2];
};

// ---------------------------------------------------------------------------
// textures
// ---------------------------------------------------------------------------

__device__ __forceinline__ int wrap_coord(int i, int size, int mode) {
    if (mode == 0) return min(max(i, 0), size - 1);
    if (mode == 2 && (size & (size - 1)) == 0) return i & (size - 1);  // == i mod size for powers of two
    if (mode == 2) {
        int m = i % size;
        return m < 0 ? m + size : m;
    }
    int t = i % (2 * size);
    if (t < 0) t += 2 * size;
    int a = t - size;
    a = a >= 0 ? a : -(1 + a);
    return size - 1 - a;
}

// Where a texture.Sample call reads: the level(s), their wrapped texels and the
// filter weights. It depends only on the texture's size and
// level count, the sampler and the uv/derivatives, so textures that share those
// share one SampleCoords (the three material textures usually do).
struct LevelCoords {
    uint32_t i00, i10, i01, i11;  // the texels, from the texture's first
    float a, b;                   // bilinear weights (unused for nearest)
};

struct SampleCoords {
    uint32_t width, height, levels;
    SamplerBits st;
    bool valid;
    bool linear;    // filter within the level(s)
    bool two;       // blend two levels
    float delta;
    LevelCoords l0, l1;
};

__device__ __forceinline__ void level_coords(const TexDesc& t, int level, bool linear, SamplerBits st, float u, float v,
                                             LevelCoords& c) {
    const int w = max(1, (int)(t.width >> level)), h = max(1, (int)(t.height >> level));
    const uint32_t off = t.level_off[level];
    const int wu = (st >> 4) & 3, wv = (st >> 6) & 3;
    if (!linear) {
        const int i = (int)floorf(u * (float)w), j = (int)floorf(v * (float)h);
        c.i00 = off + (uint32_t)wrap_coord(j, h, wv) * (uint32_t)w + (uint32_t)wrap_coord(i, w, wu);
        c.i10 = c.i01 = c.i11 = c.i00;
        c.a = c.b = 0.0f;
        return;
    }
    const float uu = u * (float)w - 0.5f, vv = v * (float)h - 0.5f;
    const float fi = floorf(uu), fj = floorf(vv);
    c.a = uu - fi;
    c.b = vv - fj;
    const int i0 = (int)fi, j0 = (int)fj;
    const uint32_t x0 = (uint32_t)wrap_coord(i0, w, wu), x1 = (uint32_t)wrap_coord(i0 + 1, w, wu);
    const uint32_t r0 = off + (uint32_t)wrap_coord(j0, h, wv) * (uint32_t)w, r1 = off + (uint32_t)wrap_coord(j0 + 1, h, wv) * (uint32_t)w;
    c.i00 = r0 + x0;
    c.i10 = r0 + x1;
    c.i01 = r1 + x0;
    c.i11 = r1 + x1;
}

// Level selection of texture.Sample with implicit derivatives (Vulkan LOD rules).
__device__ __forceinline__ void sample_coords(const TexDesc& t, SamplerBits st, const float uv[2], const float duvdx[2],
                                              const float duvdy[2], SampleCoords& c) {
    c.width = t.width;
    c.height = t.height;
    c.levels = t.levels;
    c.st = st;
    c.valid = true;
    const float w0 = (float)t.width, h0 = (float)t.height;
    const float ax = duvdx[0] * w0, ay = duvdx[1] * h0, bx = duvdy[0] * w0, by = duvdy[1] * h0;
    const float rx2 = ax * ax + ay * ay, ry2 = bx * bx + by * by;
    const float rho2 = fmaxf(rx2, ry2);
    const int q = (int)t.levels - 1;
    c.two = false;
    c.delta = 0.0f;
    if (!(rho2 > 1.0f)) {  // magnification: level 0
        c.linear = (st & 2u) != 0;
        level_coords(t, 0, c.linear, st, uv[0], uv[1], c.l0);
        return;
    }
    c.linear = (st & 1u) != 0;
    if (!(st & 4u)) {  // nearest mip: d = ceil(lambda + 0.5) - 1
        int d = 0;
        float thr = 2.0f;
        while (d < q && rho2 > thr) {
            ++d;
            thr = thr * 4.0f;
        }
        level_coords(t, d, c.linear, st, uv[0], uv[1], c.l0);
        return;
    }
    const float lambda = 0.5f * log2f(rho2);
    const float dp = fminf(lambda, (float)q);
    const int dlo = (int)floorf(dp);
    const int dhi = min(dlo + 1, q);
    const float delta = dp - (float)dlo;
    level_coords(t, dlo, c.linear, st, uv[0], uv[1], c.l0);
    if (delta > 0.0f && dhi != dlo) {
        c.two = true;
        c.delta = delta;
        level_coords(t, dhi, c.linear, st, uv[0], uv[1], c.l1);
    }
}

// byte / 255 rounded to nearest: the reciprocal as two floats, the small part's
// product in the addend of the large one's; exact for every byte (it equals the IEEE
// quotient, as a table of (float)b / 255.0f would, without the shared-memory lookup
// and its bank conflicts).
__device__ __forceinline__ float unorm8(uint32_t b) {
    const float x = (float)b, r = 1.0f / 255.0f;
    const float rest = (float)(1.0 / 255.0 - (double)r);
    return fmaf(x, r, x * rest);
}

__device__ __forceinline__ F2 unorm8x2(uint32_t lo, uint32_t hi) {
    const float r = 1.0f / 255.0f, rest = (float)(1.0 / 255.0 - (double)r);
    const F2 x = pack2((float)lo, (float)hi);
    return fma2(x, both(r), x * both(rest));
}

struct Sampler {
    const ShadeParams* P;
    const float* srgb;   // shared-memory table: sRGB byte -> linear

    // The channels of a texel that a caller reads: G and B always, R (and alpha) on demand.
    enum { kGB = 0, kRGB = 1, kRGBA = 2 };
    struct Texel {
        F2 gb, ra;
    };

    template <int kChannels>
    __device__ __forceinline__ Texel decode(bool is_srgb, uint32_t v) const {
        const uint32_t r = v & 0xffu, g = (v >> 8) & 0xffu, b = (v >> 16) & 0xffu, a = v >> 24;
        Texel o;
        o.ra.v = 0;
        if (is_srgb) {
            o.gb = pack2(srgb[g], srgb[b]);
            if (kChannels == kRGB) o.ra = both(srgb[r]);
            if (kChannels == kRGBA) o.ra = pack2(srgb[r], unorm8(a));
        } else {
            o.gb = unorm8x2(g, b);
            if (kChannels == kRGB) o.ra = both(unorm8(r));
            if (kChannels == kRGBA) o.ra = unorm8x2(r, a);
        }
        return o;
    }

    __device__ __forceinline__ void load_level(const TexDesc& t, const LevelCoords& c, uint32_t q[4]) const {
        const uint32_t* p = reinterpret_cast<const uint32_t*>(t.base);
        q[0] = __ldg(p + c.i00);
        q[1] = __ldg(p + c.i10);
        q[2] = __ldg(p + c.i01);
        q[3] = __ldg(p + c.i11);
    }

    template <int kChannels>
    __device__ __forceinline__ Texel filter_level(bool is_srgb, const LevelCoords& c, bool linear, const uint32_t q[4]) const {
        Texel o = decode<kChannels>(is_srgb, q[0]);
        if (!linear) return o;
        const Texel t10 = decode<kChannels>(is_srgb, q[1]), t01 = decode<kChannels>(is_srgb, q[2]), t11 = decode<kChannels>(is_srgb, q[3]);
        const F2 a = both(c.a), b = both(c.b);
        o.gb = mix2(mix2(o.gb, t10.gb, a), mix2(t01.gb, t11.gb, a), b);
        if (kChannels != kGB) o.ra = mix2(mix2(o.ra, t10.ra, a), mix2(t01.ra, t11.ra, a), b);
        return o;
    }

    // texture.Sample(sampler, uv) with implicit derivatives. `cache` holds the
    // coordinates of the previous call and is reused when the texture's size,
    // levels and sampler match. Channels that the caller does not read are 0.
    template <int kChannels>
    __device__ __forceinline__ void sample(uint32_t tex_index, uint32_t sampler_index, const Frag& f, SampleCoords& cache,
                                           float out[4]) const {
        out[0] = out[1] = out[2] = out[3] = 0.0f;
        if (tex_index >= P->texture_count) return;  // absent image: robust null descriptor reads 0
        const TexDesc& t = P->textures[tex_index];
        const SamplerBits st = P->samplers[min(sampler_index, P->sampler_count)];
        if (!(cache.valid && cache.width == t.width && cache.height == t.height && cache.levels == t.levels &&
              cache.st == st))
            sample_coords(t, st, f.uv, f.duvdx, f.duvdy, cache);
        const bool is_srgb = t.srgb != 0;
        uint32_t q0[4], q1[4];  // both levels' texels before either is filtered: one trip to memory, not two
        load_level(t, cache.l0, q0);
        if (cache.two) load_level(t, cache.l1, q1);
        Texel o = filter_level<kChannels>(is_srgb, cache.l0, cache.linear, q0);
        if (cache.two) {
            const Texel hi = filter_level<kChannels>(is_srgb, cache.l1, cache.linear, q1);
            const F2 d = both(cache.delta);
            o.gb = mix2(o.gb, hi.gb, d);
            if (kChannels != kGB) o.ra = mix2(o.ra, hi.ra, d);
        }
        unpack2(o.gb, out[1], out[2]);
        float alpha;
        if (kChannels != kGB) unpack2(o.ra, out[0], alpha);
        if (kChannels == kRGBA) out[3] = alpha;
    }
};

// SampleCmpLevelZero, linear, clamp-to-edge, GREATER_OR_EQUAL (Graphics.cpp:2697-2725).
__device__ __forceinline__ float sample_cmp(const float* __restrict__ shadow, int S, float u, float v, float dref) {
    const float uu = u * (float)S - 0.5f, vv = v * (float)S - 0.5f;
    const float fi = floorf(uu), fj = floorf(vv);
    const float a = uu - fi, b = vv - fj;
    const int i0 = (int)fmaxf(fminf(fi, (float)(S + 1)), -2.0f), j0 = (int)fmaxf(fminf(fj, (float)(S + 1)), -2.0f);
    const int x0 = min(max(i0, 0), S - 1), x1 = min(max(i0 + 1, 0), S - 1);
    const int y0 = min(max(j0, 0), S - 1), y1 = min(max(j0 + 1, 0), S - 1);
    const float c00 = dref >= __ldg(&shadow[(size_t)y0 * S + x0]) ? 1.0f : 0.0f;
    const float c10 = dref >= __ldg(&shadow[(size_t)y0 * S + x1]) ? 1.0f : 0.0f;
    const float c01 = dref >= __ldg(&shadow[(size_t)y1 * S + x0]) ? 1.0f : 0.0f;
    const float c11 = dref >= __ldg(&shadow[(size_t)y1 * S + x1]) ? 1.0f : 0.0f;
    const float top = c00 + a * (c10 - c00);
    const float bot = c01 + a * (c11 - c01);
    return top + b * (bot - top);
}

// 3x3 PCF: nine bilinear compare taps one texel apart. The taps' texel
// positions are computed one by one (as the single-tap path would), and when
// they fall on consecutive columns/rows - the usual case - the 16 compares of
// the shared 4x4 block are done once; otherwise each tap reads its own texels.
// Away from the map's border the block is four row pointers and constant offsets,
// and where it is all lit or all in shadow, as in most of a frame, the taps are
// what their sums would be: 9 ones or 9 zeros. (A block beyond float range is not
// consecutive, so the weights here are in [0, 1).)
__device__ float pcf3x3(const float* __restrict__ shadow, int S, const float csm[4]) {
    const float o = 1.0f / (float)S;
    int xi[3], yj[3];
    float a[3], b[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float uu = (csm[0] + (float)(k - 1) * o) * (float)S - 0.5f;
        const float vv = (csm[1] + (float)(k - 1) * o) * (float)S - 0.5f;
        const float fi = floorf(uu), fj = floorf(vv);
        a[k] = uu - fi;
        b[k] = vv - fj;
        xi[k] = (int)fmaxf(fminf(fi, (float)(S + 1)), -2.0f);
        yj[k] = (int)fmaxf(fminf(fj, (float)(S + 1)), -2.0f);
    }
    const float dref = csm[2];
    float result = 0.0f;
    if (xi[1] == xi[0] + 1 && xi[2] == xi[0] + 2 && yj[1] == yj[0] + 1 && yj[2] == yj[0] + 2) {
        float c[4][4];
        if (xi[0] >= 0 && yj[0] >= 0 && xi[0] + 3 < S && yj[0] + 3 < S) {
            const float* row = shadow + (yj[0] * S + xi[0]);  // S <= 16384
#pragma unroll
            for (int y = 0; y < 4; ++y, row += S) {
#pragma unroll
                for (int x = 0; x < 4; ++x) c[y][x] = dref >= __ldg(row + x) ? 1.0f : 0.0f;
            }
        } else {
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const int row = min(max(yj[0] + y, 0), S - 1) * S;
#pragma unroll
                for (int x = 0; x < 4; ++x) c[y][x] = dref >= __ldg(shadow + (row + min(max(xi[0] + x, 0), S - 1))) ? 1.0f : 0.0f;
            }
        }
        float lit = 0.0f;
#pragma unroll
        for (int y = 0; y < 4; ++y) lit += (c[y][0] + c[y][1]) + (c[y][2] + c[y][3]);
        if (lit == 16.0f) return 9.0f * (1.0f / 9.0f);
        if (lit == 0.0f) return 0.0f;
#pragma unroll
        for (int j = 0; j < 3; ++j) {
#pragma unroll
            for (int i = 0; i < 3; ++i) {
                const float top = c[j][i] + a[i] * (c[j][i + 1] - c[j][i]);
                const float bot = c[j + 1][i] + a[i] * (c[j + 1][i + 1] - c[j + 1][i]);
                result += top + b[j] * (bot - top);
            }
        }
        return result * (1.0f / 9.0f);
    }
    for (int j = -1; j <= 1; ++j)
        for (int i = -1; i <= 1; ++i)
            result += sample_cmp(shadow, S, csm[0] + (float)i * o, csm[1] + (float)j * o, csm[2]);
    return result * (1.0f / 9.0f);
}

// pcf.slang:1-11 (5 taps) and the 3x3 option.
__device__ float pcf(const float* __restrict__ shadow, int S, const float csm[4], uint32_t mode) {
    float result = 0.0f;
    if (mode == RZ_PCF_3X3) return pcf3x3(shadow, S, csm);
    const float o = 0.00025f;
    result += sample_cmp(shadow, S, csm[0] - o, csm[1] - o, csm[2]);
    result += sample_cmp(shadow, S, csm[0] + o * 2.0f, csm[1], csm[2]);
    result += sample_cmp(shadow, S, csm[0], csm[1] + o * 2.0f, csm[2]);
    result += sample_cmp(shadow, S, csm[0] + o * 2.0f, csm[1] + o * 2.0f, csm[2]);
    result += sample_cmp(shadow, S, csm[0] - o * 2.0f, csm[1] - o * 2.0f, csm[2]);
    return result * (1.0f / 5.0f);
}

// lighting.slang:5-43
__device__ __forceinline__ V3 schlick_fresnel(float vDotH, V3 f0) {
    const float x = clamp01(1.0f - vDotH);
    const float x2 = x * x;
    const float p = x2 * x2 * x;  // pow(x, 5)
    return {f0.x + (1.0f - f0.x) * p, f0.y + (1.0f - f0.y) * p, f0.z + (1.0f - f0.z) * p};
}
__device__ __forceinline__ float distribution_ggx(V3 N, V3 H, float roughness) {
    const float PI = 3.14159265359f;
    const float a = roughness * roughness;
    const float a2 = a * a;
    const float NdotH = fmaxf(dot(N, H), 0.0f);
    const float NdotH2 = NdotH * NdotH;
    float denom = (NdotH2 * (a2 - 1.0f) + 1.0f);
    denom = PI * denom * denom;
    return fdiv(a2, denom);
}
__device__ __forceinline__ float geometry_schlick_ggx(float NdotV, float roughness) {
    const float r = roughness + 1.0f;
    const float k = (r * r) * 0.125f;
    return fdiv(NdotV, NdotV * (1.0f - k) + k);
}
__device__ __forceinline__ float geometry_smith(V3 N, V3 V, V3 L, float roughness) {
    const float NdotV = fmaxf(dot(N, V), 0.0f);
    const float NdotL = fmaxf(dot(N, L), 0.0f);
    return geometry_schlick_ggx(NdotL, roughness) * geometry_schlick_ggx(NdotV, roughness);
}

// The shadow map a fragment samples: with one cascade the view's map and csm
// unchanged; with n > 1 the finest cascade k whose coordinates
// (csm.xy - 0.5) * 2^-k + 0.5 keep the PCF footprint (2 texels) inside the map,
// else the coarsest. Writes the coordinates in that cascade to cc.
__device__ __forceinline__ const float* select_cascade(const ViewRec& VR, const float csm[4], float cc[4]) {
#pragma unroll
    for (int i = 0; i < 4; ++i) cc[i] = csm[i];
    const float* base = reinterpret_cast<const float*>(VR.shadow);
    const int n = VR.cascades;
    if (n <= 1) return base;
    const float m = 2.0f / (float)VR.shadow_w;
    const float hi = 1.0f - m;
    int k = 0;
    for (; k < n; ++k) {
        float x = csm[0], y = csm[1];
        if (k > 0) {
            const float sc = ldexpf(1.0f, -k);
            x = (csm[0] - 0.5f) * sc + 0.5f;
            y = (csm[1] - 0.5f) * sc + 0.5f;
        }
        if ((x >= m && x <= hi && y >= m && y <= hi) || k == n - 1) {
            cc[0] = x;
            cc[1] = y;
            break;
        }
    }
    return base + (size_t)k * (size_t)VR.shadow_w * (size_t)VR.shadow_h;
}

// fragmentMain, src/shaders/basic.slang:137-344. Returns false on discard.
// kLit: the caller has checked that the view renders the default output
// (fragment_output 0) with the light, its shadow and the BRDF on, so those
// branches are taken without testing them and the debug outputs are not
// compiled into this copy. A view takes the same branches at every pixel, and
// the shading kernel runs the specialised copy for such views: the code its
// warps execute is then smaller (fewer instruction-fetch stalls).
// `late` interpolates the rest of bv (all but uv, its derivatives and csm) once the
// shadow and the textures have been read: while they are, few values are held. (With the
// other copy's shadow read among the lighting, its values were spilled around the 16 reads:
// 1280x720 with the BRDF off 52.2 us a frame instead of 49.4, 400 large blended triangles
// at 640x360 546 instead of 494.)
template <bool kLit, class Late>
__device__ __forceinline__ bool fragment_main(const ViewRec& VR, const rz_scene_data& sd, const GpuMaterial* md, Frag& bv, Late late,
                                              const Sampler& smp, float out[4], float* albedo = nullptr) {
    float shadowFactor = 1.0f;
    if (kLit || (sd.light_enabled > 0 && sd.shadows_enabled == 1)) {
        float cc[4];
        const float* map = select_cascade(VR, bv.csm, cc);
        shadowFactor = pcf(map, VR.shadow_w, cc, VR.pcf_mode);
    }
    float sampledRoughness = 0.0f, sampledMetallic = 0.0f;
    float normalTexel[4], colorTexel[4];
    bool has_normal = false, has_color = false;
    if (md) {
        SampleCoords cache;
        cache.valid = false;
        has_normal = sd.normal_maps_enabled == 1 && md->tex[1] != RZ_INVALID_INDEX;
        has_color = md->tex[0] != RZ_INVALID_INDEX;
        if (has_normal) smp.sample<Sampler::kRGB>(md->tex[1], md->sampler[1], bv, cache, normalTexel);
        if (has_color) smp.sample<Sampler::kRGBA>(md->tex[0], md->sampler[0], bv, cache, colorTexel);
        float s[4];
        const int mr = md->tex[3] != RZ_INVALID_INDEX ? 3 : 2;  // the mixmap, else the metallic-roughness texture
        smp.sample<Sampler::kGB>(md->tex[mr], md->sampler[mr], bv, cache, s);
        sampledRoughness = s[1];
        sampledMetallic = s[2];
    }
    late(bv);
    const V3 ambientLight{sd.ambient_color[0], sd.ambient_color[1], sd.ambient_color[2]};
    float outFragColor[4] = {bv.color[0], bv.color[1], bv.color[2], bv.color[3]};
    float imageTextureColor[4] = {outFragColor[0], outFragColor[1], outFragColor[2], outFragColor[3]};
    float alpha = bv.color[3];
    V3 lightNormal = fnormalize(bv.normal);
    const V3 lightDir = fnormalize(bv.lightDir);
    const V3 bitangent = bv.bitangent;
    if (md) {
#pragma unroll
        for (int k = 0; k < 4; ++k) outFragColor[k] = md->color[k];
#pragma unroll
        for (int k = 0; k < 4; ++k) imageTextureColor[k] = outFragColor[k];
        alpha = fminf(md->color[3], alpha);
        if (has_normal) {
            const V3 m{normalTexel[0] * 2.0f - 1.0f, normalTexel[1] * 2.0f - 1.0f, normalTexel[2] * 2.0f - 1.0f};
            const V3 n = fnormalize(bv.normal);
            const V3 t = fnormalize(bv.tangent - n * dot(bv.tangent, n));
            const V3 b = fnormalize(cross(bv.normal, bv.tangent) * bv.sigma);
            lightNormal = fnormalize(t * m.x + b * m.y + n * m.z);
        }
        if (has_color) {
#pragma unroll
            for (int k = 0; k < 4; ++k) imageTextureColor[k] = colorTexel[k];
            alpha = fminf(imageTextureColor[3], alpha);
        }
    }
    if (albedo) {
#pragma unroll
        for (int k = 0; k < 3; ++k) albedo[k] = imageTextureColor[k];
    }
    const V3 V = fnormalize(bv.viewDir);
    const V3 L = lightDir;
    const V3 N = lightNormal;
    const V3 H = fnormalize(L + V);
    const float cosTheta = clamp01(dot(L, N));
    const float cosPhi = clamp01(dot(H, N));
    const float lDotN = cosTheta;
    const float lDotH = clamp01(dot(L, H));
    const float nDotV = clamp01(dot(N, V));
    V3 c3;
    bool set = true;
    switch (kLit ? 0u : sd.fragment_output) {
        case 0: c3 = V3{imageTextureColor[0], imageTextureColor[1], imageTextureColor[2]}; break;
        case 1: c3 = fnormalize(bv.worldNormal) * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 2: c3 = fnormalize(bv.tangent) * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 3: c3 = fnormalize(bv.lightDir) * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 4: c3 = fnormalize(bv.viewDir) * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 5: c3 = V3{bv.color[0], bv.color[1], bv.color[2]}; break;
        case 6: c3 = lightNormal * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 7: c3 = bitangent * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 8: c3 = V3{cosTheta, cosTheta, cosTheta} * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 9: c3 = V3{cosPhi, cosPhi, cosPhi} * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 10: c3 = V3{lDotH, lDotH, lDotH} * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 11: c3 = V3{nDotV, nDotV, nDotV} * 0.5f + V3{0.5f, 0.5f, 0.5f}; break;
        case 12: c3 = V3{bv.uv[0], bv.uv[1], 0.0f}; break;
        case 13: c3 = V3{sampledRoughness, 0.05f, 0.05f}; break;
        case 14: c3 = V3{sampledMetallic, 0.05f, 0.05f}; break;
        case 15: c3 = V3{1.0f - alpha, 0.05f, 0.05f}; break;
        default: set = false; break;
    }
    if (set) {
        outFragColor[0] = c3.x;
        outFragColor[1] = c3.y;
        outFragColor[2] = c3.z;
        outFragColor[3] = alpha;
    }
    if (kLit || sd.light_enabled > 0) {
        if (!kLit && sd.brdf_lighting_enabled == 0) {
            const float ml = fmaxf(cosTheta, 0.0f);
            const V3 sunLight{sd.sunlight_color[0] * ml, sd.sunlight_color[1] * ml, sd.sunlight_color[2] * ml};
            outFragColor[0] = outFragColor[0] * fmaxf(ambientLight.x, sunLight.x * shadowFactor);
            outFragColor[1] = outFragColor[1] * fmaxf(ambientLight.y, sunLight.y * shadowFactor);
            outFragColor[2] = outFragColor[2] * fmaxf(ambientLight.z, sunLight.z * shadowFactor);
            outFragColor[3] = outFragColor[3] * alpha;
        } else {
            const float roughness = sampledRoughness;
            const float metallic = sampledMetallic;
            const float f04 = 0.04f;
            const V3 f0{f04 * (1.0f - metallic) + outFragColor[0] * metallic, f04 * (1.0f - metallic) + outFragColor[1] * metallic,
                        f04 * (1.0f - metallic) + outFragColor[2] * metallic};
            const float ndf = distribution_ggx(N, H, roughness);
            const float g = geometry_smith(N, V, L, roughness);
            const V3 f = schlick_fresnel(fmaxf(dot(H, V), 0.0f), f0);
            V3 kD{1.0f - f.x, 1.0f - f.y, 1.0f - f.z};
            kD = kD * (1.0f - metallic);
            const V3 numerator = f * (ndf * g);
            const float denominator = 4.0f * nDotV * lDotN + 0.0001f;
            const float inv_den = fdiv(1.0f, denominator);
            const V3 specular{numerator.x * inv_den, numerator.y * inv_den, numerator.z * inv_den};
            const float inv_pi = 1.0f / 3.14159265f;
            const V3 diffuse{outFragColor[0] * inv_pi, outFragColor[1] * inv_pi, outFragColor[2] * inv_pi};
            const float li = sd.light_intensity;
            const V3 sunLight{sd.sunlight_color[0] * li, sd.sunlight_color[1] * li, sd.sunlight_color[2] * li};
            V3 brdf = mul3(mul3(kD, diffuse) + specular, sunLight) * lDotN;
            brdf = V3{fmaxf(ambientLight.x * diffuse.x, brdf.x * shadowFactor), fmaxf(ambientLight.y * diffuse.y, brdf.y * shadowFactor),
                      fmaxf(ambientLight.z * diffuse.z, brdf.z * shadowFactor)};
            outFragColor[0] = brdf.x;
            outFragColor[1] = brdf.y;
            outFragColor[2] = brdf.z;
            outFragColor[3] = alpha;
        }
    }
    if (md) {
        if (md->alpha_mode == 1 && alpha < md->alpha_cutoff) return false;
        outFragColor[3] = alpha;
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = outFragColor[k];
    return true;
}

__device__ __forceinline__ uint32_t encode_srgb8(float c) {
    if (!(c > 0.0f)) c = 0.0f;
    if (c > 1.0f) c = 1.0f;
    const float s = c <= 0.0031308f ? c * 12.92f : 1.055f * __powf(c, 1.0f / 2.4f) - 0.055f;
    return (uint32_t)floorf(s * 255.0f + 0.5f);
}
__device__ __forceinline__ uint32_t encode_unorm8(float c) {
    if (!(c > 0.0f)) c = 0.0f;
    if (c > 1.0f) c = 1.0f;
    return (uint32_t)floorf(c * 255.0f + 0.5f);
}
__device__ __forceinline__ float half_round(float x) { return __half2float(__float2half_rn(x)); }

// A value of the RGBA16F draw image.
__device__ __forceinline__ uint2 pack_rgba16(float r, float g, float b, float a) {
    const __half2 rg = __floats2half2_rn(r, g), ba = __floats2half2_rn(b, a);
    return make_uint2(*reinterpret_cast<const uint32_t*>(&rg), *reinterpret_cast<const uint32_t*>(&ba));
}
__device__ __forceinline__ float4 unpack_rgba16(uint2 v) {
    const float2 rg = __half22float2(*reinterpret_cast<const __half2*>(&v.x)), ba = __half22float2(*reinterpret_cast<const __half2*>(&v.y));
    return make_float4(rg.x, rg.y, ba.x, ba.y);
}

// Varying record of one (draw, vertex): the vertex-stage outputs the fragment
// stage reads plus the clip position, 32 floats:
//   0-2 normal, 3-5 viewDir, 6-8 lightDir, 9-11 tangent, 12 sigma, 13 color.a,
//   14-16 color.rgb, 17 csm.near.w (not read), 18-19 uv, 20-22 csm.near.xyz, 23-25 worldNormal,
//   26-28 bitangent, 29-31 clip x, y, w.
// The fragment stage interpolates it two floats at a time.
constexpr int kVaryingF4 = 8;

// The vertex stage, once per (draw, mesh vertex): records [first, varying_count).
// Bound by the memory path: 64 bytes read and 128 written a vertex. A lane's record is
// 128 bytes, so its 16-byte words go through shared memory (swizzled: no bank
// conflicts) and leave 512 contiguous bytes at a time; stored by each lane they were
// half-filled sectors, 32 to an instruction (549,120 vertices: 36 -> 22 us).
__global__ void __launch_bounds__(256) k_vertex(ShadeParams P, uint32_t first) {
    __shared__ float4 s_rec[256 / 32][32][kVaryingF4];
    const uint32_t i = first + blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t lane = threadIdx.x & 31u;
    float4 (*const rec)[kVaryingF4] = s_rec[threadIdx.x >> 5];
    if (i < P.varying_count) {
        const uint32_t d = draw_in_table(i, [&](uint32_t g) { return __ldg(&P.varying_table[g]); },
                                         [&](uint32_t k) { return __ldg(&P.draws[k].varying_base); });
        const DrawRec dr = P.draws[d];
        const DrawConsts& dc = P.consts[d];
        const rz_object& gd = P.objects[dr.object];
        const GpuMaterial* md = dr.material >= 0 ? &P.materials[dr.material] : nullptr;
        const bool has_nm = md ? (md->tex[1] != RZ_INVALID_INDEX) : false;
        // the 64-byte vertex record as four 16-byte loads
        const float4* vp = reinterpret_cast<const float4*>(P.vertices + dr.vertex_base + (i - dr.varying_base));
        const float4 q0 = __ldg(vp), q1 = __ldg(vp + 1), q2 = __ldg(vp + 2), q3 = __ldg(vp + 3);
        rz_vertex v;
        v.position[0] = q0.x; v.position[1] = q0.y; v.position[2] = q0.z;
        v.normal[0] = q0.w; v.normal[1] = q1.x; v.normal[2] = q1.y;
        v.tangent[0] = q1.z; v.tangent[1] = q1.w; v.tangent[2] = q2.x; v.tangent[3] = q2.y;
        v.color[0] = q2.z; v.color[1] = q2.w; v.color[2] = q3.x; v.color[3] = q3.y;
        v.uv[0] = q3.z; v.uv[1] = q3.w;
        VsOut o;
        vertex_main(*P.views[dr.view].scene, gd, dc, md != nullptr, has_nm, v, o);
        const float4 clip = transform_point(dc.mvp, v.position[0], v.position[1], v.position[2]);
        const uint32_t x = lane & 7u;
        rec[lane][0 ^ x] = make_float4(o.normal.x, o.normal.y, o.normal.z, o.viewDir.x);
        rec[lane][1 ^ x] = make_float4(o.viewDir.y, o.viewDir.z, o.lightDir.x, o.lightDir.y);
        rec[lane][2 ^ x] = make_float4(o.lightDir.z, o.tangent.x, o.tangent.y, o.tangent.z);
        rec[lane][3 ^ x] = make_float4(o.sigma, o.color[3], o.color[0], o.color[1]);
        rec[lane][4 ^ x] = make_float4(o.color[2], o.csm[3], o.uv[0], o.uv[1]);
        rec[lane][5 ^ x] = make_float4(o.csm[0], o.csm[1], o.csm[2], o.worldNormal.x);
        rec[lane][6 ^ x] = make_float4(o.worldNormal.y, o.worldNormal.z, o.bitangent.x, o.bitangent.y);
        rec[lane][7 ^ x] = make_float4(o.bitangent.z, clip.x, clip.y, clip.w);
    }
    __syncwarp();
    const uint32_t i0 = i - lane;  // the warp's first record
    float4* dst = P.varyings + (size_t)i0 * kVaryingF4;
#pragma unroll
    for (int j = 0; j < kVaryingF4; ++j) {
        const uint32_t k = (uint32_t)j * 32u + lane, r = k / kVaryingF4, w = k % kVaryingF4;
        if (i0 + r < P.varying_count) dst[k] = rec[r][w ^ (r & 7u)];
    }
}
static_assert(kVaryingF4 == 8, "eight words to a record: the swizzle");

void launch_vertex(const ShadeParams& p, cudaStream_t stream) {
    if (p.varying_count == 0 || p.draw_count == 0) return;
    k_vertex<<<(p.varying_count + 255) / 256, 256, 0, stream>>>(p, 0u);
    note_launch();
}

void launch_vertex_range(const ShadeParams& p, uint32_t first, cudaStream_t stream) {
    if (p.varying_count <= first || p.draw_count == 0) return;
    k_vertex<<<(p.varying_count - first + 255) / 256, 256, 0, stream>>>(p, first);
    note_launch();
}

// Shade triangle `tri` (pass-global id) at pixel (px, py) from the varying
// records of its three vertices.
// With `aux` non-null it also returns the G-buffer values: albedo (the sampled
// base colour, rgb) and the interpolated world-space normal (normalised, xyz).
// With `pn` non-null the pixel-centre coordinates come from there (see pixel_ndc).
template <bool kLit = false>
__device__ bool shade_pixel(const ShadeParams& P, const ViewRec& VR, const rz_scene_data& sd, const Sampler& smp, uint32_t tri,
                            int px, int py, float out[4], float* aux = nullptr, const PixelNdc* pn = nullptr) {
    // the camera setup recorded the material and the vertices
    const uint4 ref = __ldg(&P.tri_refs[tri]);
    const float4* const rec[3] = {P.varyings + (size_t)ref.y * kVaryingF4, P.varyings + (size_t)ref.z * kVaryingF4,
                                  P.varyings + (size_t)ref.w * kVaryingF4};
    const int32_t material = (int32_t)ref.x;
    const GpuMaterial* md = material >= 0 ? &P.materials[material] : nullptr;
    float4 clip[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 q = __ldg(rec[k] + 7);
        clip[k] = make_float4(q.y, q.z, 0.0f, q.w);
    }
    float b[3], bq0[3], bqx[3], bqy[3];
    const int qx = px & ~1, qy = py & ~1;
    float xp, yp, xq, yq, xq1, yq1;  // ndc of px, py, qx, qy, qx + 1, qy + 1
    if (pn) {
        xp = pn->xp;
        yp = pn->yp;
        xq = pn->xq;
        yq = pn->yq;
        xq1 = pn->xq1;
        yq1 = pn->yq1;
    } else {
        xp = ndc(px, VR.width);
        yp = ndc(py, VR.height);
        xq = ndc(qx, VR.width);
        yq = ndc(qy, VR.height);
        xq1 = ndc(qx + 1, VR.width);
        yq1 = ndc(qy + 1, VR.height);
    }
    barycentrics_n(clip[0], clip[1], clip[2], xp, yp, b);
    barycentrics_n(clip[0], clip[1], clip[2], xq, yq, bq0);
    barycentrics_n(clip[0], clip[1], clip[2], xq1, yq, bqx);
    barycentrics_n(clip[0], clip[1], clip[2], xq, yq1, bqy);
    const bool debug_extra = (!kLit && (sd.fragment_output == 1 || sd.fragment_output == 7)) || aux != nullptr;
    // what the shadow and the textures need: uv here and at the quad's pixels, csm
    Frag f;
    F2 uv{}, uv0{}, uvx{}, uvy{}, csm_xy{};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const float4 q5 = __ldg(rec[k] + 5);
        const F2 tex{__ldg(reinterpret_cast<const ulonglong2*>(rec[k] + 4)).y}, xy = pack2(q5.x, q5.y);
        const F2 w = both(b[k]), wq = both(bq0[k]), wx = both(bqx[k]), wy = both(bqy[k]);
        uv = k == 0 ? tex * w : uv + tex * w;
        uv0 = k == 0 ? tex * wq : uv0 + tex * wq;
        uvx = k == 0 ? tex * wx : uvx + tex * wx;
        uvy = k == 0 ? tex * wy : uvy + tex * wy;
        csm_xy = k == 0 ? xy * w : csm_xy + xy * w;
        f.csm[2] = k == 0 ? q5.z * b[k] : f.csm[2] + q5.z * b[k];
    }
    unpack2(uv, f.uv[0], f.uv[1]);
    unpack2(uvx - uv0, f.duvdx[0], f.duvdx[1]);
    unpack2(uvy - uv0, f.duvdy[0], f.duvdy[1]);
    unpack2(csm_xy, f.csm[0], f.csm[1]);
    f.csm[3] = 0.0f;  // not read
    auto late = [&](Frag& v) {
        F2 acc[8], extra[2];
        float wnx = 0.0f, bz = 0.0f, c2 = 0.0f;
        extra[0].v = extra[1].v = 0;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            const F2 w = both(b[k]);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2*>(rec[k] + i));
                acc[2 * i] = k == 0 ? F2{q.x} * w : acc[2 * i] + F2{q.x} * w;
                acc[2 * i + 1] = k == 0 ? F2{q.y} * w : acc[2 * i + 1] + F2{q.y} * w;
            }
            const float blue = __ldg(&rec[k][4].x);
            c2 = k == 0 ? blue * b[k] : c2 + blue * b[k];
            if (debug_extra) {
                const float wx = __ldg(&rec[k][5].w), z = __ldg(&rec[k][7].x);
                const ulonglong2 q = __ldg(reinterpret_cast<const ulonglong2*>(rec[k] + 6));
                wnx = k == 0 ? wx * b[k] : wnx + wx * b[k];
                extra[0] = k == 0 ? F2{q.x} * w : extra[0] + F2{q.x} * w;
                extra[1] = k == 0 ? F2{q.y} * w : extra[1] + F2{q.y} * w;
                bz = k == 0 ? z * b[k] : bz + z * b[k];
            }
        }
        unpack2(acc[0], v.normal.x, v.normal.y);
        unpack2(acc[1], v.normal.z, v.viewDir.x);
        unpack2(acc[2], v.viewDir.y, v.viewDir.z);
        unpack2(acc[3], v.lightDir.x, v.lightDir.y);
        unpack2(acc[4], v.lightDir.z, v.tangent.x);
        unpack2(acc[5], v.tangent.y, v.tangent.z);
        unpack2(acc[6], v.sigma, v.color[3]);
        unpack2(acc[7], v.color[0], v.color[1]);
        v.color[2] = c2;
        v.worldNormal.x = wnx;
        unpack2(extra[0], v.worldNormal.y, v.worldNormal.z);
        unpack2(extra[1], v.bitangent.x, v.bitangent.y);
        v.bitangent.z = bz;
        if (aux) {
            const V3 n = fnormalize(v.worldNormal);
            aux[3] = n.x;
            aux[4] = n.y;
            aux[5] = n.z;
        }
    };
    return fragment_main<kLit>(VR, sd, md, f, late, smp, out, aux);
}

// Whether a view renders the default output with the light, its shadow and the
// BRDF on (the branches fragment_main<true> takes without testing).
__device__ __forceinline__ bool lit_view(const rz_scene_data& sd) {
    return sd.fragment_output == 0 && sd.light_enabled > 0 && sd.shadows_enabled == 1 && sd.brdf_lighting_enabled != 0;
}

// Octahedral encoding of a unit vector into two f16 (x in the low half).
__device__ __forceinline__ uint32_t encode_octahedral(float x, float y, float z) {
    const float s = fabsf(x) + fabsf(y) + fabsf(z);
    float u = 0.0f, v = 0.0f;
    if (s > 0.0f) {
        u = x / s;
        v = y / s;
        if (z < 0.0f) {
            const float au = 1.0f - fabsf(v), av = 1.0f - fabsf(u);
            u = u >= 0.0f ? au : -au;
            v = v >= 0.0f ? av : -av;
        }
    }
    const __half2 h = __floats2half2_rn(u, v);
    return *reinterpret_cast<const uint32_t*>(&h);
}

// The view a 16x16 shading tile belongs to (tiles are numbered view by view).
__device__ __forceinline__ uint32_t tile_view(const ViewRec* __restrict__ views, uint32_t n, uint32_t tile) {
    uint32_t lo = 0, hi = n;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (__ldg(&views[mid].shade_block_base) <= tile) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Average of four RGBA16F sample values ((s0 + s1) + (s2 + s3)) / 4, rounded
// to RGBA16F: the AVERAGE resolve of the multisampled draw image
// (src/Engine/Graphics.cpp:5571-5572).
__device__ __forceinline__ float resolve4(float a, float b, float c, float d) {
    return half_round(((a + b) + (c + d)) * 0.25f);
}

// The pixel (px, py) of this thread in the block's 16x16 tile, and its
// pixel-centre coordinates. Each lane of a warp (16 columns, 2 rows) computes its
// column's and its row's coordinate (the values ndc() gives) and takes its quad's
// from the lanes of its quad's first column and of the two rows, so the tile needs
// no shared table and no second block barrier. All lanes take part (shuffles).
__device__ __forceinline__ PixelNdc pixel_ndc(const ShadeParams& P, const ViewRec& VR, int& px, int& py) {
    const uint32_t lt = blockIdx.x + P.block_offset - VR.shade_block_base;
    const uint32_t tiles_x = ((uint32_t)VR.width + 15) / 16;
    px = (int)(lt % tiles_x) * 16 + (int)threadIdx.x;
    py = (int)(lt / tiles_x) * 16 + (int)threadIdx.y;
    const int lane = (int)(threadIdx.x + 16 * (threadIdx.y & 1));
    PixelNdc pn;
    pn.xp = ndc(px, VR.width);
    pn.yp = ndc(py, VR.height);
    pn.xq = __shfl_sync(0xffffffffu, pn.xp, lane & 14);
    pn.xq1 = __shfl_sync(0xffffffffu, pn.xp, (lane & 14) + 1);
    pn.yq = __shfl_sync(0xffffffffu, pn.yp, lane & 15);
    pn.yq1 = __shfl_sync(0xffffffffu, pn.yp, (lane & 15) + 16);
    return pn;
}

// Bound by instruction issue and the latency of its dependent reads (visibility,
// vertex records, texels, shadow map) about alike: 55 % issue active, 5.4 of 11
// cycles between a warp's instructions on memory. So the fragment stage reads the
// shadow and the textures while it holds little, interpolates the rest after them
// (two floats per instruction), and six CTAs of 42 registers hide more latency than
// four of 64 did when everything was interpolated first (then five were no faster).
// 1080p scene-scale frame: 166 -> 155 us with the kernel so, 4x MSAA 278 -> 256,
// 32 views 171 -> 154.
__global__ void __launch_bounds__(256, 6) k_shade(ShadeParams P) {
    __shared__ float s_srgb[256];
    __shared__ uint32_t s_view;
    {
        const int t = threadIdx.y * blockDim.x + threadIdx.x;
        s_srgb[t] = P.srgb_table[t];
        if (t == 0) s_view = tile_view(P.views, P.view_count, blockIdx.x + P.block_offset);
    }
    __syncthreads();
    const ViewRec& VR = P.views[s_view];
    int px, py;
    const PixelNdc pn = pixel_ndc(P, VR, px, py);
    if (px >= VR.width || py >= VR.height) return;
    const size_t p = (size_t)py * VR.width + px;
    const unsigned long long key = VR.vis[p];
    const uint32_t id = (uint32_t)key;
    float col[4] = {0.0f, 0.05f, 0.1f, 1.0f};  // clear colour, src/Engine/Graphics.cpp:5416-5419
    const bool gbuffer = VR.gb_albedo != nullptr;
    float aux[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
    if (id != 0) {
        const Sampler smp{&P, s_srgb};
        float o[4];
        const rz_scene_data& sd = *VR.scene;
        float* const ax = gbuffer ? aux : nullptr;
        if (lit_view(sd) ? shade_pixel<true>(P, VR, sd, smp, id - 1u, px, py, o, ax, &pn)
                         : shade_pixel<false>(P, VR, sd, smp, id - 1u, px, py, o, ax, &pn)) {
#pragma unroll
            for (int k = 0; k < 4; ++k) col[k] = o[k];
        }
    }
    if (gbuffer) {
        VR.gb_albedo[p] = encode_srgb8(half_round(aux[0])) | (encode_srgb8(half_round(aux[1])) << 8) |
                          (encode_srgb8(half_round(aux[2])) << 16) | ((id != 0 ? 255u : 0u) << 24);
        VR.gb_normal[p] = encode_octahedral(aux[3], aux[4], aux[5]);
    }
    VR.depth[p] = __uint_as_float((uint32_t)(key >> 32));
    if (P.blended) {  // blended surfaces follow: keep the RGBA16F draw image
        const __half2 rg = __floats2half2_rn(col[0], col[1]), ba = __floats2half2_rn(col[2], col[3]);
        VR.color16[p] = make_uint2(*reinterpret_cast<const uint32_t*>(&rg), *reinterpret_cast<const uint32_t*>(&ba));
        return;
    }
    const uint32_t r = encode_srgb8(half_round(col[0]));
    const uint32_t g = encode_srgb8(half_round(col[1]));
    const uint32_t b = encode_srgb8(half_round(col[2]));
    const uint32_t a = encode_unorm8(half_round(col[3]));
    VR.color[p] = r | (g << 8) | (b << 16) | (a << 24);
}

// k_shade for 4x multisampled views. Each distinct triangle among a pixel's
// samples is shaded once at the pixel centre (no sample shading, as the
// reference's pipeline), its colour is rounded to RGBA16F and given to the samples
// it covers; uncovered samples keep the clear colour. Without blended surfaces the
// samples are resolved and encoded here; with them they go to the RGBA16F sample
// planes for k_blend. The depth output is sample 0's.
//
// Bound by the instruction issue of the fragment stage, like k_shade, times the
// distinct triangles a warp meets: a pixel inside a triangle shows one, a pixel on
// an edge two to four, and with triangles of a few pixels almost every warp holds
// one with three or four. So the tile's (pixel, triangle) pairs are listed in
// shared memory first - every pixel's first triangle in pixel order, then the
// second ones, and so on, so that neighbours stay neighbours - and the block's
// threads shade the list, all lanes busy, in one copy of the fragment stage.
// 1920x1080, 262,144 triangles of a median 4 square pixels: the frame went from
// 527 to 307 us against four conditional copies of the stage per pixel.
constexpr int kMsaaItems = 256 * kMsaaSamples;  // (pixel, triangle) pairs of a tile, at most

// A tile's pixel-centre coordinates (the values ndc() gives): its columns and rows.
struct TileNdc {
    float x[16], y[16];
};

// Shades the listed pairs of the tile at (tx0, ty0): item i is the triangle
// item_id[i] (id + 1) at pixel item_px[i] (row * 16 + column). Writes its RGBA16F
// colour to item_col[i] and, with a G-buffer, its six values to item_aux + 6 i.
template <bool kLit, bool kAux>
__device__ __forceinline__ void shade_items(const ShadeParams& P, const ViewRec& VR, const float* s_srgb, const TileNdc& tn,
                                            int tx0, int ty0, int tid, int total, const uint32_t* item_id,
                                            const uint8_t* item_px, uint2* item_col, float* item_aux) {
    const Sampler smp{&P, s_srgb};
#pragma unroll 1
    for (int i = tid; i < total; i += 256) {
        const int t = item_px[i], lx = t & 15, ly = t >> 4;
        const PixelNdc pn{tn.x[lx], tn.y[ly], tn.x[lx & ~1], tn.y[ly & ~1], tn.x[lx | 1], tn.y[ly | 1]};
        float c[4] = {0.0f, 0.05f, 0.1f, 1.0f};  // clear colour, src/Engine/Graphics.cpp:5416-5419
        float aux[6] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        float o[4];
        if (shade_pixel<kLit>(P, VR, *VR.scene, smp, item_id[i] - 1u, tx0 + lx, ty0 + ly, o, kAux ? aux : nullptr, &pn)) {
#pragma unroll
            for (int k = 0; k < 4; ++k) c[k] = o[k];
        }
        const __half2 rg = __floats2half2_rn(c[0], c[1]), ba = __floats2half2_rn(c[2], c[3]);
        item_col[i] = make_uint2(*reinterpret_cast<const uint32_t*>(&rg), *reinterpret_cast<const uint32_t*>(&ba));
        if (kAux) {
#pragma unroll
            for (int k = 0; k < 6; ++k) item_aux[6 * i + k] = aux[k];
        }
    }
}

template <bool kAux>  // the views have a G-buffer
__global__ void __launch_bounds__(256, 5) k_shade_msaa(ShadeParams P) {
    __shared__ float s_srgb[256];
    __shared__ uint32_t s_view;
    __shared__ TileNdc s_ndc;
    __shared__ uint32_t s_count[kMsaaSamples][8];  // per rank and warp: pixels with that many distinct triangles
    __shared__ uint32_t s_id[kMsaaItems];
    __shared__ uint8_t s_px[kMsaaItems];
    __shared__ uint2 s_col[kMsaaItems];
    extern __shared__ float s_aux[];  // kMsaaItems x 6, with a G-buffer
    const int tid = threadIdx.y * 16 + threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    s_srgb[tid] = P.srgb_table[tid];
    if (tid == 0) s_view = tile_view(P.views, P.view_count, blockIdx.x + P.block_offset);
    __syncthreads();
    const ViewRec& VR = P.views[s_view];
    const uint32_t lt = blockIdx.x + P.block_offset - VR.shade_block_base;
    const uint32_t tiles_x = ((uint32_t)VR.width + 15) / 16;
    const int tx0 = (int)(lt % tiles_x) * 16, ty0 = (int)(lt / tiles_x) * 16;
    const int px = tx0 + (int)threadIdx.x, py = ty0 + (int)threadIdx.y;
    const bool inside = px < VR.width && py < VR.height;
    const size_t plane = (size_t)VR.width * VR.height;
    const size_t p = inside ? (size_t)py * VR.width + px : 0;
    if (tid < 16) s_ndc.x[tid] = ndc(tx0 + tid, VR.width);
    else if (tid < 32) s_ndc.y[tid - 16] = ndc(ty0 + tid - 16, VR.height);
    // the pixel's distinct triangles: sample k shows the rank[k]-th one
    uint32_t ids[kMsaaSamples], distinct[kMsaaSamples];
#pragma unroll
    for (int k = 0; k < kMsaaSamples; ++k) ids[k] = 0u;
    if (inside) {
#pragma unroll
        for (int k = 0; k < kMsaaSamples; ++k) {
            const unsigned long long key = VR.vis[p + k * plane];
            if (k == 0) VR.depth[p] = __uint_as_float((uint32_t)(key >> 32));
            ids[k] = (uint32_t)key;
        }
    }
    uint32_t n = 0, ranks = 0;
#pragma unroll
    for (int k = 0; k < kMsaaSamples; ++k) {
        distinct[k] = 0u;
        uint32_t r = n;
#pragma unroll
        for (int j = k - 1; j >= 0; --j)
            if (ids[j] == ids[k]) r = (ranks >> (4 * j)) & 7u;
        if (ids[k] == 0u) {
            r = 7u;  // not covered
        } else if (r == n) {
#pragma unroll
            for (int j = 0; j < kMsaaSamples; ++j)
                if ((uint32_t)j == n) distinct[j] = ids[k];
            ++n;
        }
        ranks |= r << (4 * k);
    }
    uint32_t before[kMsaaSamples];  // lanes before this one in the warp with a triangle of that rank
#pragma unroll
    for (int r = 0; r < kMsaaSamples; ++r) {
        const uint32_t m = __ballot_sync(0xffffffffu, n > (uint32_t)r);
        before[r] = __popc(m & ((1u << lane) - 1u));
        if (lane == 0) s_count[r][warp] = __popc(m);
    }
    __syncthreads();
    uint64_t slots = 0;  // where the pixel's triangles sit in the list, 16 bits per rank
    uint32_t total = 0;
#pragma unroll
    for (int r = 0; r < kMsaaSamples; ++r) {
        uint32_t at = total + before[r];
        for (int w = 0; w < 8; ++w) {
            if (w < warp) at += s_count[r][w];
            total += s_count[r][w];
        }
        slots |= (uint64_t)at << (16 * r);
        if (n > (uint32_t)r) {
            s_id[at] = distinct[r];
            s_px[at] = (uint8_t)tid;
        }
    }
    __syncthreads();
    if (lit_view(*VR.scene)) shade_items<true, kAux>(P, VR, s_srgb, s_ndc, tx0, ty0, tid, (int)total, s_id, s_px, s_col, s_aux);
    else shade_items<false, kAux>(P, VR, s_srgb, s_ndc, tx0, ty0, tid, (int)total, s_id, s_px, s_col, s_aux);
    __syncthreads();
    if (!inside) return;
    float cs[kMsaaSamples][4];
#pragma unroll
    for (int k = 0; k < kMsaaSamples; ++k) {
        const uint32_t r = (ranks >> (4 * k)) & 7u;
        cs[k][0] = half_round(0.0f);  // clear colour, src/Engine/Graphics.cpp:5416-5419
        cs[k][1] = half_round(0.05f);
        cs[k][2] = half_round(0.1f);
        cs[k][3] = half_round(1.0f);
        if (r != 7u) {
            const uint2 c = s_col[(slots >> (16 * r)) & 0xffffu];
            const __half2 rg = *reinterpret_cast<const __half2*>(&c.x), ba = *reinterpret_cast<const __half2*>(&c.y);
            cs[k][0] = __low2float(rg);
            cs[k][1] = __high2float(rg);
            cs[k][2] = __low2float(ba);
            cs[k][3] = __high2float(ba);
        }
    }
    if (kAux) {
        // G-buffer of a multisampled pixel: albedo and normal averaged over the samples,
        // coverage = covered samples / 4 in the albedo's alpha
        float gs[kMsaaSamples][6], g[6];
        uint32_t covered = 0;
#pragma unroll
        for (int k = 0; k < kMsaaSamples; ++k) {
            const uint32_t r = (ranks >> (4 * k)) & 7u;
            covered += r != 7u ? 1u : 0u;
#pragma unroll
            for (int i = 0; i < 6; ++i) gs[k][i] = r != 7u ? s_aux[6 * ((slots >> (16 * r)) & 0xffffu) + i] : 0.0f;
        }
#pragma unroll
        for (int i = 0; i < 6; ++i) g[i] = ((gs[0][i] + gs[1][i]) + (gs[2][i] + gs[3][i])) * 0.25f;
        VR.gb_albedo[p] = encode_srgb8(half_round(g[0])) | (encode_srgb8(half_round(g[1])) << 8) |
                          (encode_srgb8(half_round(g[2])) << 16) | (encode_unorm8((float)covered * 0.25f) << 24);
        const float len2 = g[3] * g[3] + g[4] * g[4] + g[5] * g[5];
        const float inv = len2 > 0.0f ? rsqrtf(len2) : 0.0f;
        VR.gb_normal[p] = encode_octahedral(g[3] * inv, g[4] * inv, g[5] * inv);
    }
    if (P.blended) {
#pragma unroll
        for (int k = 0; k < kMsaaSamples; ++k) {
            const __half2 rg = __floats2half2_rn(cs[k][0], cs[k][1]), ba = __floats2half2_rn(cs[k][2], cs[k][3]);
            VR.color16[p + k * plane] =
                make_uint2(*reinterpret_cast<const uint32_t*>(&rg), *reinterpret_cast<const uint32_t*>(&ba));
        }
        return;
    }
    float c4[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) c4[i] = resolve4(cs[0][i], cs[1][i], cs[2][i], cs[3][i]);
    VR.color[p] = encode_srgb8(c4[0]) | (encode_srgb8(c4[1]) << 8) | (encode_srgb8(c4[2]) << 16) | (encode_unorm8(c4[3]) << 24);
}

void launch_shade(const ShadeParams& p, cudaStream_t stream) {
    if (p.shade_blocks == 0) return;
    note_launch();
    if (p.samples > 1) {
        // the G-buffer values of the listed pairs: 24 KB, within the default limit with the static arrays
        if (p.gbuffer) k_shade_msaa<true><<<p.shade_blocks, dim3(16, 16), kMsaaItems * 6 * sizeof(float), stream>>>(p);
        else k_shade_msaa<false><<<p.shade_blocks, dim3(16, 16), 0, stream>>>(p);
        return;
    }
    k_shade<<<p.shade_blocks, dim3(16, 16), 0, stream>>>(p);
}

// ---------------------------------------------------------------------------
// sub-pixel sources of the learned half-resolution path (G-buffer)
// ---------------------------------------------------------------------------

// Screen position (pixels) and NDC depth of the three vertices of an opaque
// triangle: the clip position the vertex stage computes (the draw's MVP times
// the mesh position), divided by w.
struct SubTri {
    float X[3], Y[3], Z[3];
    float inv_area;  // 1 / twice the signed screen area (0 when degenerate)
    bool valid;      // every w > 0
};

__device__ __forceinline__ SubTri sub_triangle(const ShadeParams& P, uint32_t id, float hw, float hh) {
    const uint32_t tri = id - 1u;
    const uint32_t d = draw_from(P.draws, P.draw_count, P.draw_table, tri);
    const DrawRec dr = P.draws[d];
    const uint32_t t = tri - dr.tri_base;
    const float* M = P.consts[d].mvp;
    SubTri g;
    g.valid = true;
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const uint32_t vi = __ldg(&P.indices[dr.first_index + 3u * t + k]) + dr.vertex_base;
        const float* pos = P.vertices[vi].position;
        const float4 c = transform_point(M, __ldg(pos), __ldg(pos + 1), __ldg(pos + 2));
        g.valid = g.valid && c.w > 0.0f;
        const float rw = 1.0f / c.w;
        g.X[k] = (c.x * rw) * hw + hw;
        g.Y[k] = (c.y * rw) * hh + hh;
        g.Z[k] = c.z * rw;
    }
    const float area = (g.X[1] - g.X[0]) * (g.Y[2] - g.Y[0]) - (g.X[2] - g.X[0]) * (g.Y[1] - g.Y[0]);
    g.inv_area = area != 0.0f ? 1.0f / area : 0.0f;
    return g;
}

// Shared-memory table of a tile's distinct triangles (open addressing, 128
// slots): each triangle's geometry is computed once per tile, not once per
// pixel that considers it. Key 0 marks an empty slot (ids are >= 1).
constexpr int kSubSlots = 128;

__device__ __forceinline__ uint32_t sub_slot(uint32_t id) { return (id * 2654435761u) >> 25; }

// The slot of triangle `id` (entered if it is new), kSubSlots where the table is full:
// pixels that need such a triangle compute its geometry themselves.
__device__ __forceinline__ uint32_t sub_insert(uint32_t* keys, uint32_t id) {
    uint32_t h = sub_slot(id);
    for (int i = 0; i < kSubSlots; ++i) {
        const uint32_t prev = atomicCAS(&keys[h], 0u, id);
        if (prev == 0u || prev == id) return h;
        h = (h + 1) & (kSubSlots - 1);
    }
    return kSubSlots;
}

// For the x2 reconstruction of the learned path: which triangle is in front at
// each of the four points (x + 0.25 / 0.75, y + 0.25 / 0.75) that the pixel's
// four full-resolution pixels sample, among the triangles visible at the 3x3
// neighbourhood's pixel centres (covered by the float edge functions, front-most
// by the depth plane through the vertices' z / w, larger nearer as in the depth
// test), and which of each point's bilinear sources (own, horizontal, vertical,
// diagonal neighbour, clamped at the borders) show it: bit 4k + s,
// k = 2 * (y half) + (x half). A pixel whose neighbourhood shows one triangle
// (or none) keeps every source (0xFFFF). The arithmetic is plain float without
// contraction, restated by the oracle bit for bit. The reference has no learned
// path; nothing here follows a reference file.
//
// Bound by latency: five dependent reads lead to a triangle's geometry, and the
// pixels' candidates differ in number (17 of 32 lanes busy). So a triangle is looked
// up once per cell of the tile that needs it, not once per pixel that considers it,
// and a pixel keeps its distinct neighbours as bits, not as an indexed list:
// 960x540 learned frame of 4,096 random triangles 154 -> 150 us, 229 -> 223 alone.
// More CTAs per SM (5, 6 or 8 instead of 4) were no faster or slower.
__global__ void __launch_bounds__(256) k_subpixel_sources(ShadeParams P) {
    __shared__ uint32_t s_view;
    __shared__ uint32_t s_ids[18][18];  // the tile's triangle ids with a one-pixel border (clamped)
    __shared__ uint8_t s_slot[18][18];  // their slots in the table; before, 1 where an edge pixel considers the cell
    __shared__ uint32_t s_keys[kSubSlots];
    __shared__ SubTri s_geo[kSubSlots];
    __shared__ uint32_t s_edge_count;
    __shared__ uint8_t s_edges[256];  // the tile's pixels whose neighbourhood shows more than one triangle
    const int tid = threadIdx.y * 16 + threadIdx.x;
    if (tid == 0) {
        s_view = tile_view(P.views, P.view_count, blockIdx.x + P.block_offset);
        s_edge_count = 0u;
    }
    if (tid < kSubSlots) s_keys[tid] = 0u;
    __syncthreads();
    const ViewRec& VR = P.views[s_view];
    if (!VR.gb_sources) return;  // uniform over the block
    const uint32_t lt = blockIdx.x + P.block_offset - VR.shade_block_base;
    const uint32_t tiles_x = ((uint32_t)VR.width + 15) / 16;
    const int x0 = (int)(lt % tiles_x) * 16, y0 = (int)(lt / tiles_x) * 16;
    const int W = VR.width, H = VR.height;
    const float hw = (float)W * 0.5f, hh = (float)H * 0.5f;
    for (int i = tid; i < 18 * 18; i += 256) {
        const int yy = min(max(y0 + i / 18 - 1, 0), H - 1), xx = min(max(x0 + i % 18 - 1, 0), W - 1);
        s_ids[i / 18][i % 18] = (uint32_t)VR.vis[(size_t)yy * W + xx];
        s_slot[i / 18][i % 18] = 0;
    }
    __syncthreads();
    {
        const int x = x0 + threadIdx.x, y = y0 + threadIdx.y;
        bool same = true;
#pragma unroll
        for (int dy = 0; dy < 3; ++dy)
#pragma unroll
            for (int dx = 0; dx < 3; ++dx) same = same && s_ids[threadIdx.y + dy][threadIdx.x + dx] == s_ids[threadIdx.y + 1][threadIdx.x + 1];
        if (x < W && y < H) {
            if (same) {
                VR.gb_sources[(size_t)y * W + x] = 0xFFFFu;
            } else {  // the cells the edge pixels consider, and the pixel
#pragma unroll
                for (int dy = 0; dy < 3; ++dy)
#pragma unroll
                    for (int dx = 0; dx < 3; ++dx) s_slot[threadIdx.y + dy][threadIdx.x + dx] = 1;
                s_edges[atomicAdd(&s_edge_count, 1u)] = (uint8_t)tid;
            }
        }
    }
    __syncthreads();
    for (int i = tid; i < 18 * 18; i += 256) {
        const uint32_t id = s_ids[i / 18][i % 18];
        if (s_slot[i / 18][i % 18] != 0 && id != 0u) s_slot[i / 18][i % 18] = (uint8_t)sub_insert(s_keys, id);
    }
    __syncthreads();
    if (tid < kSubSlots && s_keys[tid] != 0u) s_geo[tid] = sub_triangle(P, s_keys[tid], hw, hh);
    __syncthreads();
    // the edge pixels, packed onto the first lanes of the block
    const uint32_t n_edges = s_edge_count;
    if ((uint32_t)tid >= n_edges) return;
    const int ex = s_edges[tid] & 15, ey = s_edges[tid] >> 4;
    const int x = x0 + ex, y = y0 + ey;
    uint32_t nb[9], candidates = 0u;  // bit ci: nb[ci] is a triangle no earlier one is
#pragma unroll
    for (int dy = 0; dy < 3; ++dy)
#pragma unroll
        for (int dx = 0; dx < 3; ++dx) nb[dy * 3 + dx] = s_ids[ey + dy][ex + dx];
#pragma unroll
    for (int ci = 0; ci < 9; ++ci) {
        bool seen = nb[ci] == 0u;
#pragma unroll
        for (int j = 0; j < ci; ++j) seen = seen || nb[j] == nb[ci];
        candidates |= seen ? 0u : 1u << ci;
    }
    const uint32_t own = nb[4];
    uint32_t mask;
    {
        uint32_t best[4] = {0u, 0u, 0u, 0u};
        float best_z[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
        for (; candidates != 0u; candidates &= candidates - 1u) {  // in neighbourhood order
            const int ci = __ffs((int)candidates) - 1, cy = ey + ci / 3, cx = ex + ci % 3;
            const uint32_t id = s_ids[cy][cx], slot = s_slot[cy][cx];
            const SubTri g = slot < kSubSlots ? s_geo[slot] : sub_triangle(P, id, hw, hh);
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const float sx = (float)x + ((k & 1) ? 0.75f : 0.25f), sy = (float)y + ((k >> 1) ? 0.75f : 0.25f);
                bool inside;
                float z;
                if (!g.valid) {  // a vertex behind the eye: only the pixel's own triangle, behind every other
                    inside = id == own;
                    z = -3.0e38f;
                } else {
                    const float e0 = (g.X[2] - g.X[1]) * (sy - g.Y[1]) - (g.Y[2] - g.Y[1]) * (sx - g.X[1]);
                    const float e1 = (g.X[0] - g.X[2]) * (sy - g.Y[2]) - (g.Y[0] - g.Y[2]) * (sx - g.X[2]);
                    const float e2 = (g.X[1] - g.X[0]) * (sy - g.Y[0]) - (g.Y[1] - g.Y[0]) * (sx - g.X[0]);
                    inside = g.inv_area != 0.0f &&
                             ((e0 >= 0.0f && e1 >= 0.0f && e2 >= 0.0f) || (e0 <= 0.0f && e1 <= 0.0f && e2 <= 0.0f));
                    z = ((e0 * g.Z[0] + e1 * g.Z[1]) + e2 * g.Z[2]) * g.inv_area;
                }
                if (inside && z > best_z[k]) {
                    best[k] = id;
                    best_z[k] = z;
                }
            }
        }
        mask = 0u;
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            // sources of point k: own, horizontal, vertical and diagonal neighbour (the 3x3 entries)
            const int hx = (k & 1) ? 2 : 0, vy = (k >> 1) ? 2 : 0;
            const uint32_t src[4] = {own, nb[3 + hx], nb[vy * 3 + 1], nb[vy * 3 + hx]};
#pragma unroll
            for (int s = 0; s < 4; ++s)
                if (src[s] == best[k]) mask |= 1u << (4 * k + s);
        }
    }
    VR.gb_sources[(size_t)y * W + x] = (uint16_t)mask;
}

void launch_subpixel_sources(const ShadeParams& p, cudaStream_t stream) {
    if (p.shade_blocks == 0 || p.samples > 1) return;
    k_subpixel_sources<<<p.shade_blocks, dim3(16, 16), 0, stream>>>(p);
    note_launch();
}

// ---------------------------------------------------------------------------
// blended list
// ---------------------------------------------------------------------------

// One CTA per 16x16 tile. The blended records overlapping the tile are listed in
// shared memory in submission order; every pixel takes from them, in that order, the
// fragments that cover it (the raster's integer edge test) and pass the
// GREATER_OR_EQUAL test against the opaque depth (no write); fragmentMain (discard
// honoured); then SRC_ALPHA / ONE_MINUS_SRC_ALPHA on colour, ONE / ZERO on alpha,
// rounded to the RGBA16F draw image after each blend
// (src/Engine/Graphics.cpp:5654-5691). Then the sRGB blit.
//
// Blending keeps the order; finding and shading the fragments does not need it.
// * A tile does not look at every record: k_blend_boxes gives each group of 32
//   consecutive records its box, a tile reads the boxes and then the records of the
//   groups that meet it. Neighbours in the list are mostly neighbours on the screen
//   (a mesh's triangles). Where they are not, every group meets every tile, and the
//   tile tests the records it tested without the boxes, and 1/32 as many boxes.
// * A tile's records are prepared once, a thread each (blend_prepare: edges relative to
//   the tile in 32 bits, records that miss it left out), and each warp keeps those that
//   meet its two rows. A pixel then tests a record with six multiplications and no branch;
//   reading the record and its 64-bit edges pixel by pixel was a serial chain, 620 cycles
//   a record, so that the fullest tile (318 records) ran 125 us.
// * The fragments are shaded together: a pixel collects up to kBlendRound of them,
//   the tile lists them (the first ones of all pixels, the second ones, ...), the
//   block shades the list with all lanes busy, and each pixel blends its own in
//   order. Shaded where they are met, a triangle of a few pixels ran the fragment
//   stage for a few lanes of a warp.
// * The overlay's segments are tested by their boxes (8 bytes each, read in a row; the
//   64-byte segments cost 118 MB a frame) and then against the tile itself, and a tile
//   that meets nothing of either list finishes after one test.
// 1279x717, 12,288 blended triangles (a median 4 square pixels) of 49,152 and 24 overlay
// objects: the frame went from 636 us to 125 us with the boxes and the shading together,
// to 113 us with the cheaper fragment stage, and to 91 us with the prepared records and
// the overlay's boxes. What is left is the latency of the fullest tiles and of the
// five loads that a tile waits for one after the other.
// A pixel's values are held packed as they are stored, and a CTA has 64 registers a thread,
// four to an SM (80 and three with 4 samples). With five of 48 the fragment stage spilled, and
// deep overdraw was slower than fragments shaded where they are met: 100 triangles across
// 640x360 376 us a frame, 471 without the BRDF, 496 with 4 samples, against 294, 287 and 355;
// now 289, 339 and 321. Three per SM would take 274 and 286 for the first two, but the tiles
// that meet little want more of them: 3840x2160 with 640 blended triangles 271 us, 249 with
// four, 260 with five. (The frame above: 87, 85 and 87.)
// Without a blended list only the overlay is compiled in, 40 registers and six CTAs: 900
// overlay objects at 1080p 737 -> 595 us.
constexpr int kBlendBatch = 512;   // group boxes (or overlay segments) tested at a time
constexpr int kBlendList = 256;    // records of a tile prepared at a time
constexpr int kBlendRound = 4;     // fragments a pixel collects before the tile shades them
constexpr int kBlendGroup = 32;    // records of a group box
constexpr int kBlendItems = 256 * kBlendRound;

// Ordered compaction of the items [start, min(start + kBlendBatch, n)) that `hit`
// selects (kPer consecutive items per thread) into s_list, in item order; returns
// their count. Every thread of the 256-thread CTA calls it.
template <int kPer, class Hit>
__device__ __forceinline__ uint32_t compact_batch(uint32_t start, uint32_t n, int tid, uint32_t* s_list,
                                                  uint32_t* s_count, Hit hit) {
    const int lane = tid & 31, warp = tid >> 5;
    uint32_t mask = 0;
#pragma unroll
    for (int k = 0; k < kPer; ++k) {
        const uint32_t r = start + kPer * tid + k;
        if (r < n && hit(r)) mask |= 1u << k;
    }
    const uint32_t cnt = __popc(mask);
    uint32_t incl = cnt;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += v;
    }
    __syncthreads();
    if (lane == 31) s_count[warp] = incl;
    __syncthreads();
    uint32_t base = 0, total = 0;
    for (int w = 0; w < 8; ++w) {
        if (w < warp) base += s_count[w];
        total += s_count[w];
    }
    uint32_t pos = base + incl - cnt;
#pragma unroll
    for (int k = 0; k < kPer; ++k)
        if (mask & (1u << k)) s_list[pos++] = start + kPer * tid + k;
    __syncthreads();
    return total;
}

// Whether the 5-pixel line `s` can cover a sample of the 16x16 tile at pixel (tx0, ty0):
// over the tile, `along` and `perp` of debug_covers differ from their values at its centre
// by at most 8 pixels times |dx| + |dy|. Most tiles in the box of a long slanted line are
// not met by the line.
__device__ __forceinline__ bool debug_meets(const DebugSeg& s, int tx0, int ty0) {
    if (s.reach > 1.0e30f) return true;
    const long long dx = (long long)s.X1 - s.X0, dy = (long long)s.Y1 - s.Y0;
    const long long ex = (long long)(tx0 + 8) * 256 - s.X0, ey = (long long)(ty0 + 8) * 256 - s.Y0;
    const long long slack = 2048 * (llabs(dx) + llabs(dy)), along = ex * dx + ey * dy;
    if (along + slack < 0 || along - slack >= dx * dx + dy * dy) return false;
    return (float)(llabs(dx * ey - dy * ex) - slack) <= s.reach;
}

// Whether the 5-pixel line `s` covers the sample at (PX, PY) (1/256 pixel), and
// its depth there: the rectangle 0 <= along < |d|^2, -(w/2)|d| < perp <= (w/2)|d|
// in exact integers; depth fma(along/|d|^2, z1 - z0, z0) clamped to [0, 1].
__device__ __forceinline__ bool debug_covers(const DebugSeg& s, int32_t PX, int32_t PY, float& z) {
    const long long dx = (long long)s.X1 - s.X0, dy = (long long)s.Y1 - s.Y0;
    const long long len2 = dx * dx + dy * dy;
    if (len2 == 0) return false;
    const long long ex = (long long)PX - s.X0, ey = (long long)PY - s.Y0;
    const long long perp = dx * ey - dy * ex;
    if ((float)llabs(perp) > s.reach) return false;  // further than the half width by more than a rounding
    const long long along = ex * dx + ey * dy;
    if (along < 0 || along >= len2) return false;
    const __int128 lhs = (__int128)perp * perp, rhs = (__int128)kDebugHalfWidth2 * len2;
    if (perp >= 0 ? lhs > rhs : lhs >= rhs) return false;
    const float t = (float)along / (float)len2;
    float zz = fmaf(t, s.z1 - s.z0, s.z0);
    if (!(zz > 0.0f)) zz = 0.0f;
    if (zz > 1.0f) zz = 1.0f;
    z = zz;
    return true;
}

// The box (pixels, inclusive) and the first and last view of every group of
// kBlendGroup records: (x0 | y0 << 16, x1 | y1 << 16, view, view). One warp per group.
__global__ void __launch_bounds__(256) k_blend_boxes(const TriRecord* __restrict__ records, const PassHeader* __restrict__ header,
                                                     uint32_t capacity, uint4* __restrict__ boxes) {
    const uint32_t n = min(header->records, capacity), groups = (n + kBlendGroup - 1) / kBlendGroup;
    const uint32_t lane = threadIdx.x & 31u, warps = (gridDim.x * blockDim.x) >> 5;
    for (uint32_t g = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; g < groups; g += warps) {
        const uint32_t r = g * kBlendGroup + lane;
        uint32_t x0 = 0xffffu, y0 = 0xffffu, x1 = 0u, y1 = 0u, v0 = 0xffffffffu, v1 = 0u;
        if (r < n) {
            const TriRecord& rec = records[r];
            x0 = rec.p0 & 0xffffu;
            y0 = rec.p0 >> 16;
            x1 = rec.p1 & 0xffffu;
            y1 = rec.p1 >> 16;
            v0 = v1 = rec.view & kViewMask;
        }
        x0 = __reduce_min_sync(0xffffffffu, x0);
        y0 = __reduce_min_sync(0xffffffffu, y0);
        x1 = __reduce_max_sync(0xffffffffu, x1);
        y1 = __reduce_max_sync(0xffffffffu, y1);
        v0 = __reduce_min_sync(0xffffffffu, v0);
        v1 = __reduce_max_sync(0xffffffffu, v1);
        if (lane == 0) boxes[g] = make_uint4(x0 | (y0 << 16), x1 | (y1 << 16), v0, v1);
    }
}

__device__ __forceinline__ bool box_meets(uint32_t p0, uint32_t p1, int tx0, int ty0) {
    const int x0 = p0 & 0xffff, y0 = p0 >> 16, x1 = p1 & 0xffff, y1 = p1 >> 16;
    return x1 >= tx0 && x0 <= tx0 + 15 && y1 >= ty0 && y0 <= ty0 + 15;
}

// The samples of pixel (px, py) (bits; bit 0 without multisampling) that a blended
// record covers and whose opaque depth it passes.
template <bool kMsaa>
__device__ __forceinline__ uint32_t blend_samples(const TriRecord& rec, int px, int py, const float* dst_depth) {
    const int4* src = reinterpret_cast<const int4*>(&rec);
    const int4 q0 = __ldg(src), q1 = __ldg(src + 1);
    const float dzdy = __int_as_float(__ldg(reinterpret_cast<const int*>(src + 2)));
    const int32_t X[3] = {q0.x, q0.z, q1.x}, Y[3] = {q0.y, q0.w, q1.y};
    const float z0 = __int_as_float(q1.z), dzdx = __int_as_float(q1.w);
    uint32_t pass = 0;
#pragma unroll
    for (int k = 0; k < (kMsaa ? kMsaaSamples : 1); ++k) {
        const int32_t PX = px * 256 + (kMsaa ? msaa_x(k) : 128), PY = py * 256 + (kMsaa ? msaa_y(k) : 128);
        bool in = true;
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            const int a = (i + 1) % 3, b = (i + 2) % 3;
            const int32_t dx = X[b] - X[a], dy = Y[b] - Y[a];
            const bool tl = dy < 0 || (dy == 0 && dx > 0);
            const int64_t E = (int64_t)dx * (int64_t)(PY - Y[a]) - (int64_t)dy * (int64_t)(PX - X[a]);
            in = in && (E > 0 || (E == 0 && tl));
        }
        if (!in) continue;
        float z = fmaf(dzdx, (float)(PX - X[0]), fmaf(dzdy, (float)(PY - Y[0]), z0));
        if (!(z > 0.0f)) z = 0.0f;
        if (z > 1.0f) z = 1.0f;
        if (z >= dst_depth[k]) pass |= 1u << k;
    }
    return pass;
}

// A record as a tile's pixels read it: edge i at (ux, uy) 1/256 pixels from the tile's
// corner is e[i] + a[i] * ux + b[i] * uy, the top-left rule folded into e, and a sample is
// covered where no edge is negative.
struct BlendTri {
    int32_t e[3], a[3], b[3];
    int32_t X0, Y0;
    uint32_t id;
    float z0, dzdx, dzdy;
    uint32_t wide;  // record + 1 where an edge does not fit 32 bits over the tile, else 0
};
static_assert(sizeof(BlendTri) == 64, "four 16-byte reads");

// Prepares record r for the tile at pixel (tx0, ty0); false where an edge leaves the whole
// tile outside. The values are blend_samples' own: an edge that is negative nowhere in the
// tile becomes zero, and one that changes sign there is small unless the triangle is huge.
__device__ __forceinline__ bool blend_prepare(const TriRecord& rec, uint32_t r, int tx0, int ty0, BlendTri& t) {
    const int4* src = reinterpret_cast<const int4*>(&rec);
    const int4 q0 = __ldg(src), q1 = __ldg(src + 1);
    const int32_t X[3] = {q0.x, q0.z, q1.x}, Y[3] = {q0.y, q0.w, q1.y};
    bool meets = true, wide = false;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        const int a = (i + 1) % 3, b = (i + 2) % 3;
        const int32_t dx = X[b] - X[a], dy = Y[b] - Y[a];
        const bool tl = dy < 0 || (dy == 0 && dx > 0);
        const int64_t e = (int64_t)dx * ((int64_t)ty0 * 256 - Y[a]) - (int64_t)dy * ((int64_t)tx0 * 256 - X[a]) - (tl ? 0 : 1);
        const int64_t lo = e + 4096 * ((int64_t)min(dx, 0) - (int64_t)max(dy, 0));
        const int64_t hi = e + 4096 * ((int64_t)max(dx, 0) - (int64_t)min(dy, 0));
        meets = meets && hi >= 0;
        const bool cuts = lo < 0;
        wide = wide || (cuts && (lo < -2147483647LL || hi > 2147483647LL));
        t.e[i] = cuts ? (int32_t)e : 0;
        t.a[i] = cuts ? -dy : 0;
        t.b[i] = cuts ? dx : 0;
    }
    t.X0 = X[0];
    t.Y0 = Y[0];
    t.id = rec.id;
    t.z0 = __int_as_float(q1.z);
    t.dzdx = __int_as_float(q1.w);
    t.dzdy = rec.dzdy;
    t.wide = wide ? r + 1u : 0u;
    return meets;
}

// blend_samples from a prepared record of the tile at (tx0, ty0), without a branch.
template <bool kMsaa>
__device__ __forceinline__ uint32_t blend_pass(const BlendTri& t, int px, int py, int tx0, int ty0, const float* dst_depth) {
    const int4* q = reinterpret_cast<const int4*>(&t);
    const int4 q0 = q[0], q1 = q[1], q2 = q[2], q3 = q[3];  // e, a0 | a1 a2, b0 b1 | b2, X0, Y0, id | z0, dzdx, dzdy, wide
    uint32_t pass = 0;
#pragma unroll
    for (int k = 0; k < (kMsaa ? kMsaaSamples : 1); ++k) {
        const int32_t PX = px * 256 + (kMsaa ? msaa_x(k) : 128), PY = py * 256 + (kMsaa ? msaa_y(k) : 128);
        const uint32_t ux = (uint32_t)(PX - tx0 * 256), uy = (uint32_t)(PY - ty0 * 256);
        const uint32_t E0 = (uint32_t)q0.x + (uint32_t)q0.w * ux + (uint32_t)q1.z * uy;
        const uint32_t E1 = (uint32_t)q0.y + (uint32_t)q1.x * ux + (uint32_t)q1.w * uy;
        const uint32_t E2 = (uint32_t)q0.z + (uint32_t)q1.y * ux + (uint32_t)q2.x * uy;
        float z = fmaf(__int_as_float(q3.y), (float)(PX - q2.y), fmaf(__int_as_float(q3.z), (float)(PY - q2.z), __int_as_float(q3.x)));
        z = z > 0.0f ? z : 0.0f;
        z = z > 1.0f ? 1.0f : z;
        if ((int32_t)(E0 | E1 | E2) >= 0 && z >= dst_depth[k]) pass |= 1u << k;
    }
    return pass;
}

// Shades the listed fragments: item i is the triangle item_id[i] (id + 1) at pixel
// item_px[i] (row * 16 + column) of the tile; its colour goes to item_out[i], and
// item_id[i] becomes 0 where it is discarded.
template <bool kLit>
__device__ __forceinline__ void shade_fragments(const ShadeParams& P, const ViewRec& VR, const float* s_srgb, const TileNdc& tn,
                                                int tx0, int ty0, int tid, int total, uint32_t* item_id,
                                                const uint8_t* item_px, float4* item_out) {
    const Sampler smp{&P, s_srgb};
#pragma unroll 1
    for (int i = tid; i < total; i += 256) {
        const int t = item_px[i], lx = t & 15, ly = t >> 4;
        const PixelNdc pn{tn.x[lx], tn.y[ly], tn.x[lx & ~1], tn.y[ly & ~1], tn.x[lx | 1], tn.y[ly | 1]};
        float o[4];
        if (shade_pixel<kLit>(P, VR, *VR.scene, smp, item_id[i] - 1u, tx0 + lx, ty0 + ly, o, nullptr, &pn))
            item_out[i] = make_float4(o[0], o[1], o[2], o[3]);
        else
            item_id[i] = 0u;
    }
}

template <bool kMsaa, bool kList>  // kList: there is a blended list (else only the overlay)
__global__ void __launch_bounds__(256, !kList ? 6 : kMsaa ? 3 : 4) k_blend(const __grid_constant__ BlendParams B) {
    constexpr int kSamples = kMsaa ? kMsaaSamples : 1;
    __shared__ float s_srgb[256];
    __shared__ uint32_t s_list[kBlendBatch];  // groups (or overlay segments) that meet the tile
    __shared__ alignas(16) BlendTri s_tri[kBlendList];
    __shared__ uint8_t s_rows[kBlendList];           // first and last row of a prepared record in the tile
    __shared__ uint8_t s_mine[256 / 32][kBlendList]; // the prepared records that meet a warp's two rows
    __shared__ uint32_t s_count[kBlendRound][256 / 32];
    __shared__ TileNdc s_ndc;
    __shared__ uint32_t s_id[kBlendItems];
    __shared__ uint8_t s_px[kBlendItems];
    __shared__ float4 s_out[kBlendItems];
    __shared__ uint32_t s_view;
    const ShadeParams& P = B.sh;
    const int tid = threadIdx.y * blockDim.x + threadIdx.x;
    // a pass whose look-back gave up has records at unreliable slots: blend none of them
    const bool records_ok = !B.error_flags || !(*B.error_flags & kErrLookbackTimeout);
    const uint32_t n = kList && records_ok ? min(B.header->records, B.record_capacity) : 0u;
    const uint32_t groups = (n + kBlendGroup - 1) / kBlendGroup;
    const float srgb = P.srgb_table[tid];
    uint32_t view = 0;
    if (P.view_count > 1) {
        if (tid == 0) s_view = tile_view(P.views, P.view_count, blockIdx.x + P.block_offset);
        __syncthreads();
        view = s_view;
    }
    const ViewRec& VR = P.views[view];
    const uint32_t lt = blockIdx.x + P.block_offset - VR.shade_block_base;
    const uint32_t tiles_x = ((uint32_t)VR.width + 15) / 16;
    const int tx0 = (int)(lt % tiles_x) * 16, ty0 = (int)(lt / tiles_x) * 16;
    const int px = tx0 + threadIdx.x, py = ty0 + threadIdx.y;
    const bool inside = px < VR.width && py < VR.height;
    const size_t p = inside ? (size_t)py * VR.width + px : 0;
    const size_t plane = (size_t)VR.width * VR.height;
    // per coverage sample: the RGBA16F value and the opaque depth it is tested against
    uint2 held[kSamples];
    float dst_depth[kSamples];
#pragma unroll
    for (int k = 0; k < kSamples; ++k) {
        held[k] = inside ? VR.color16[p + k * plane] : make_uint2(0u, 0u);
        dst_depth[k] = !inside ? 0.0f : kMsaa ? __uint_as_float((uint32_t)(VR.vis[p + k * plane] >> 32)) : VR.depth[p];
    }
    const int lane = tid & 31, warp = tid >> 5;
    // Most tiles meet nothing of the list or the overlay: they are known by one test of the boxes
    bool any = groups > kBlendBatch || B.debug_count > kBlendBatch;
#pragma unroll
    for (int k = 0; k < kBlendBatch / 256; ++k) {
        const uint32_t i = tid + 256 * k;
        if (i < groups) {
            const uint4 b = __ldg(&B.boxes[i]);
            any = any || (b.z <= view && view <= b.w && box_meets(b.x, b.y, tx0, ty0));
        }
        if (i < B.debug_count) {
            const uint2 b = __ldg(&B.debug_boxes[(size_t)view * B.debug_count + i]);
            any = any || box_meets(b.x, b.y, tx0, ty0);
        }
    }
    s_srgb[tid] = srgb;
    if (tid < 16) s_ndc.x[tid] = ndc(tx0 + tid, VR.width);
    else if (tid < 32) s_ndc.y[tid - 16] = ndc(ty0 + tid - 16, VR.height);
    any = __syncthreads_or(any) != 0;
    const bool lit = kList && any && lit_view(*VR.scene);
    for (uint32_t first = 0; kList && any && first < groups; first += kBlendBatch) {
        const uint32_t ngroups = compact_batch<kBlendBatch / 256>(first, groups, tid, s_list, s_count[0], [&](uint32_t g) {
            const uint4 b = __ldg(&B.boxes[g]);
            return b.z <= view && view <= b.w && box_meets(b.x, b.y, tx0, ty0);
        });
        for (uint32_t gs = 0, listed = 0; gs < ngroups;) {
            // the groups' records that meet the tile, in order, until the list is full: a group per warp, a record per lane
            for (; gs < ngroups; gs += 256 / kBlendGroup) {
                BlendTri t;
                uint32_t rows = 0;
                bool hit = false;
                if (gs + warp < ngroups) {
                    const uint32_t r = s_list[gs + warp] * kBlendGroup + lane;
                    if (r < n) {
                        const TriRecord& rec = B.records[r];
                        const uint32_t p0 = rec.p0, p1 = rec.p1;
                        hit = (rec.view & kViewMask) == view && box_meets(p0, p1, tx0, ty0);
                        if (hit) hit = blend_prepare(rec, r, tx0, ty0, t);
                        rows = (uint32_t)(max((int)(p0 >> 16) - ty0, 0) | (min((int)(p1 >> 16) - ty0, 15) << 4));
                    }
                }
                // of a scattered list mostly none of 256 records: one barrier instead of two (60,000 small
                // triangles in random order at 1080p: 1,276 -> 1,066 us a frame)
                if (__syncthreads_or(hit) == 0) continue;
                const uint32_t hits = __ballot_sync(0xffffffffu, hit);
                if (lane == 0) s_count[0][warp] = __popc(hits);
                __syncthreads();
                uint32_t at = listed, total = 0;
                for (int w = 0; w < 8; ++w) {
                    if (w < warp) at += s_count[0][w];
                    total += s_count[0][w];
                }
                const bool full = listed + total > kBlendList;  // they wait for the next list
                if (hit && !full) {
                    at += __popc(hits & ((1u << lane) - 1u));
                    s_tri[at] = t;
                    s_rows[at] = (uint8_t)rows;
                }
                __syncthreads();
                if (full) break;
                listed += total;
            }
            uint32_t mine = 0, far = 0;
            for (uint32_t base = 0; base < listed; base += 32) {
                const uint32_t i = base + lane, rows = i < listed ? s_rows[i] : 15u;  // 15: none
                const bool hit = (int)(rows & 15u) <= 2 * warp + 1 && (int)(rows >> 4) >= 2 * warp;
                const uint32_t m = __ballot_sync(0xffffffffu, hit);
                if (hit) s_mine[warp][mine + __popc(m & ((1u << lane) - 1u))] = (uint8_t)i;
                far |= __ballot_sync(0xffffffffu, hit && s_tri[i].wide != 0u);
                mine += __popc(m);
            }
            __syncwarp();
            uint32_t next = 0, open = 0;  // the warp's next record; the pixel's fragments of the last ones, not yet taken
            bool more = listed != 0;
            listed = 0;
            while (more) {
                // up to kBlendRound fragments of the pixel, in order. The warp tests kLook records at a time,
                // and stops at the first that leave a pixel of it with more fragments than it can take.
                constexpr uint32_t kLook = 32 / kSamples;
                uint32_t frag[kBlendRound], pass_of = 0, nf = 0;
#pragma unroll
                for (int r = 0; r < kBlendRound; ++r) frag[r] = 0u;
                for (;;) {
                    while (open != 0u && nf < kBlendRound) {
                        const uint32_t at = (uint32_t)(__ffs((int)open) - 1) / kSamples;
                        const uint32_t id = s_tri[s_mine[warp][next - kLook + at]].id;
#pragma unroll
                        for (int r = 0; r < kBlendRound; ++r)
                            if (nf == (uint32_t)r) frag[r] = id;
                        constexpr uint32_t kAll = (1u << kSamples) - 1u;
                        pass_of |= ((open >> (kSamples * at)) & kAll) << (4 * nf);
                        open &= ~(kAll << (kSamples * at));
                        ++nf;
                    }
                    if (next >= mine || __any_sync(0xffffffffu, open != 0u)) break;
                    const uint32_t look = min(mine - next, kLook);
                    if (far == 0u) {
#pragma unroll 4
                        for (uint32_t q = 0; q < look; ++q)
                            open |= blend_pass<kMsaa>(s_tri[s_mine[warp][next + q]], px, py, tx0, ty0, dst_depth) << (kSamples * q);
                    } else {
#pragma unroll 1
                        for (uint32_t q = 0; q < look; ++q) {
                            const BlendTri& t = s_tri[s_mine[warp][next + q]];
                            open |= (t.wide ? blend_samples<kMsaa>(B.records[t.wide - 1u], px, py, dst_depth)
                                            : blend_pass<kMsaa>(t, px, py, tx0, ty0, dst_depth)) << (kSamples * q);
                        }
                    }
                    if (!inside) open = 0u;
                    next += kLook;
                }
                uint32_t before[kBlendRound];
#pragma unroll
                for (int r = 0; r < kBlendRound; ++r) {
                    const uint32_t m = __ballot_sync(0xffffffffu, nf > (uint32_t)r);
                    before[r] = __popc(m & ((1u << lane) - 1u));
                    if (lane == 0) s_count[r][warp] = __popc(m);
                }
                __syncthreads();
                uint64_t slots = 0;  // where the pixel's fragments sit in the list, 16 bits each
                uint32_t items = 0;
#pragma unroll
                for (int r = 0; r < kBlendRound; ++r) {
                    uint32_t i = items + before[r];
                    for (int w = 0; w < 8; ++w) {
                        if (w < warp) i += s_count[r][w];
                        items += s_count[r][w];
                    }
                    slots |= (uint64_t)i << (16 * r);
                    if (nf > (uint32_t)r) {
                        s_id[i] = frag[r];
                        s_px[i] = (uint8_t)tid;
                    }
                }
                __syncthreads();
                if (lit) shade_fragments<true>(P, VR, s_srgb, s_ndc, tx0, ty0, tid, (int)items, s_id, s_px, s_out);
                else shade_fragments<false>(P, VR, s_srgb, s_ndc, tx0, ty0, tid, (int)items, s_id, s_px, s_out);
                __syncthreads();
                for (uint32_t r = 0; r < nf; ++r) {
                    const uint32_t i = (uint32_t)(slots >> (16 * r)) & 0xffffu;
                    if (s_id[i] == 0u) continue;  // discarded
                    const float4 o = s_out[i];
                    const float a = o.w;
#pragma unroll
                    for (int k = 0; k < kSamples; ++k) {
                        if (!((pass_of >> (4 * r + k)) & 1u)) continue;
                        const float4 d = unpack_rgba16(held[k]);
                        held[k] = pack_rgba16(o.x * a + d.x * (1.0f - a), o.y * a + d.y * (1.0f - a), o.z * a + d.z * (1.0f - a), a);
                    }
                }
                more = __syncthreads_or(open != 0u || next < mine) != 0;
            }
        }
    }
    // Debug-line overlay after the blended list (src/Engine/Graphics.cpp:5694-5738): the same
    // blend state and depth test, depth writes off; a covered sample in front of the opaque
    // depth takes the line's colour (SRC_ALPHA with alpha 1 keeps only the source).
    if (any && B.debug_count) {
        const DebugSeg* __restrict__ segs = B.debug + (size_t)view * B.debug_count;
        const uint2* __restrict__ boxes = B.debug_boxes + (size_t)view * B.debug_count;
        for (uint32_t start = 0; start < B.debug_count; start += kBlendBatch) {
            const uint32_t total = compact_batch<kBlendBatch / 256>(start, B.debug_count, tid, s_list, s_count[0], [&](uint32_t r) {
                const uint2 b = __ldg(&boxes[r]);
                return box_meets(b.x, b.y, tx0, ty0) && debug_meets(segs[r], tx0, ty0);
            });
            if (inside) {
                for (uint32_t j = 0; j < total; ++j) {
                    const DebugSeg& sg = segs[s_list[j]];
                    const uint2 b = __ldg(&boxes[s_list[j]]);
                    if (px < (int)(b.x & 0xffffu) || px > (int)(b.y & 0xffffu) || py < (int)(b.x >> 16) || py > (int)(b.y >> 16)) continue;
                    uint32_t pass = 0;  // samples covered and in front of the opaque depth
#pragma unroll
                    for (int k = 0; k < kSamples; ++k) {
                        const int32_t PX = px * 256 + (kMsaa ? msaa_x(k) : 128);
                        const int32_t PY = py * 256 + (kMsaa ? msaa_y(k) : 128);
                        float z;
                        if (debug_covers(sg, PX, PY, z) && z >= dst_depth[k]) pass |= 1u << k;
                    }
                    if (!pass) continue;
#pragma unroll
                    for (int k = 0; k < kSamples; ++k) {
                        if (!(pass & (1u << k))) continue;
                        held[k] = pack_rgba16(sg.rgb[0], sg.rgb[1], sg.rgb[2], 1.0f);
                    }
                }
            }
            __syncthreads();
        }
    }
    if (!inside) return;
    float4 o = unpack_rgba16(held[0]);
    if constexpr (kMsaa) {
        const float4 o1 = unpack_rgba16(held[1]), o2 = unpack_rgba16(held[2]), o3 = unpack_rgba16(held[3]);
        o = make_float4(resolve4(o.x, o1.x, o2.x, o3.x), resolve4(o.y, o1.y, o2.y, o3.y), resolve4(o.z, o1.z, o2.z, o3.z),
                        resolve4(o.w, o1.w, o2.w, o3.w));
    }
    VR.color[p] = encode_srgb8(o.x) | (encode_srgb8(o.y) << 8) | (encode_srgb8(o.z) << 16) | (encode_unorm8(o.w) << 24);
}

void launch_blend_boxes(const TriRecord* records, const PassHeader* header, uint32_t capacity, uint4* boxes,
                        cudaStream_t stream) {
    const uint32_t groups = (capacity + kBlendGroup - 1) / kBlendGroup;
    if (groups == 0) return;
    k_blend_boxes<<<std::min((groups + 7) / 8, 1024u), 256, 0, stream>>>(records, header, capacity, boxes);
    note_launch();
}

size_t blend_box_count(uint32_t capacity) { return (capacity + (size_t)kBlendGroup - 1) / kBlendGroup; }

void launch_blend(const BlendParams& p, cudaStream_t stream) {
    if (p.sh.shade_blocks == 0) return;
    void (*const kernel)(BlendParams) = p.list ? (p.sh.samples > 1 ? k_blend<true, true> : k_blend<false, true>)
                                               : (p.sh.samples > 1 ? k_blend<true, false> : k_blend<false, false>);
    kernel<<<p.sh.shade_blocks, dim3(16, 16), 0, stream>>>(p);
    note_launch();
}

}  // namespace rz
