// Device helpers shared by the raster and shading kernels. These implement the
// renderer's fp32 geometry contract; the translation units that include this
// file are compiled with -fmad=false so that every fused multiply-add is an
// explicit fmaf() and every other product and sum rounds on its own.
#pragma once

#include "rz_internal.h"

namespace rz {

// C = A * B for column-major 4x4 matrices; element (c, r) is the fma chain
// A[0][r]*B[c][0] -> +A[1][r]*B[c][1] -> +A[2][r]*B[c][2] -> +A[3][r]*B[c][3].
// (mul(sd.viewproj, worldMat) of src/shaders/basic.slang:116 and
//  mul(sd.shadowProjNear, worldMat) of src/shaders/shadow.slang:17.)
__device__ __forceinline__ void mat4_mul(const float* __restrict__ A, const float* __restrict__ B, float* __restrict__ C) {
#pragma unroll
    for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            float acc = A[0 * 4 + r] * B[c * 4 + 0];
            acc = fmaf(A[1 * 4 + r], B[c * 4 + 1], acc);
            acc = fmaf(A[2 * 4 + r], B[c * 4 + 2], acc);
            acc = fmaf(A[3 * 4 + r], B[c * 4 + 3], acc);
            C[c * 4 + r] = acc;
        }
    }
}

// clip = M * (x, y, z, 1): fma(M0r, x, M3r) -> fma(M1r, y, .) -> fma(M2r, z, .).
__device__ __forceinline__ float4 transform_point(const float* __restrict__ M, float x, float y, float z) {
    float4 o;
    o.x = fmaf(M[8], z, fmaf(M[4], y, fmaf(M[0], x, M[12])));
    o.y = fmaf(M[9], z, fmaf(M[5], y, fmaf(M[1], x, M[13])));
    o.z = fmaf(M[10], z, fmaf(M[6], y, fmaf(M[2], x, M[14])));
    o.w = fmaf(M[11], z, fmaf(M[7], y, fmaf(M[3], x, M[15])));
    return o;
}

// The draw that holds triangle `tri`, from the list's table; null: of the list's n draws.
__device__ __forceinline__ uint32_t draw_from(const DrawRec* __restrict__ draws, uint32_t n, const uint32_t* __restrict__ table,
                                              uint32_t tri) {
    const auto base = [&](uint32_t d) { return __ldg(&draws[d].tri_base); };
    if (!table) return draw_between(0u, n - 1u, tri, base);
    return draw_in_table(tri, [&](uint32_t g) { return __ldg(&table[g]); }, base);
}

// Thread `tid` of `stride` threads' share of zeroing n bytes at ptr: 16-byte
// stores on the 16-byte-aligned body, byte stores on the unaligned head and
// tail, so any start address and size is safe.
__device__ __forceinline__ void zero_share(void* ptr, size_t n, size_t tid, size_t stride) {
    unsigned char* base = static_cast<unsigned char*>(ptr);
    size_t head = (16 - ((size_t)base & 15)) & 15;
    if (head > n) head = n;
    if (tid < head) base[tid] = 0;
    const size_t n16 = (n - head) / 16;
    uint4* body = reinterpret_cast<uint4*>(base + head);
    for (size_t i = tid; i < n16; i += stride) body[i] = make_uint4(0u, 0u, 0u, 0u);
    const size_t done = head + n16 * 16;
    if (tid < n - done) base[done + tid] = 0;
}

// This thread's share of zeroing every range of L (all threads of the grid).
__device__ __forceinline__ void clear_share(const ClearList& L) {
    const size_t tid = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    const size_t stride = (size_t)gridDim.x * blockDim.x;
    for (int b = 0; b < L.count; ++b) zero_share(L.ptr[b], L.bytes[b], tid, stride);
}

// Two floats in a register pair, and the packed operations on them: each half rounds
// as the scalar operation does, in one instruction instead of two (kernels that are
// short of issue slots, not of multipliers).
struct F2 {
    unsigned long long v;
};
__device__ __forceinline__ F2 pack2(float lo, float hi) {
    F2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ F2 both(float x) { return pack2(x, x); }
__device__ __forceinline__ void unpack2(F2 p, float& lo, float& hi) { asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(p.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) {
    F2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 operator-(F2 a, F2 b) {
    F2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v));
    return r;
}
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) {
    F2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v));
    return r;
}
// The products: a * b - 0, whose sums round like a * b. The assembler contracts a packed
// multiply and the add after it into one multiply-add (whatever -fmad says, and with a
// literal -0 too), which rounds once; it does not know this value.
static __constant__ unsigned long long c_minus_zeros = 0x8000000080000000ull;
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { return fma2(a, b, F2{c_minus_zeros}); }

// Programmatic dependent launch. A kernel launched with launch_next may start once every
// CTA of the kernel before it in the stream has started and called pdl_allow_next (or is
// done): its CTAs then take the SMs as that one's leave them, and set up what does not
// depend on it. It waits in pdl_wait_previous for the one before to be complete and its
// writes visible, before it touches what that one computes. Where every kernel of a chain
// waits so, one that gets past this point comes after all the earlier ones. The first
// kernel of a chain is launched normally, after all that the stream holds. A kernel that
// allocates tensor memory lets the next one in after that, and the wait comes later still. (957x539
// upsampler inference, five kernels: 78 -> 64 us; a training step of two 960x540 frames:
// 555 -> 494. Frames: see chained in rz_api.cu.)
__device__ __forceinline__ void pdl_allow_next() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait_previous() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

template <class... P, class... A>
inline bool launch_next(void (*kernel)(P...), int grid, int threads, uint32_t smem, cudaStream_t s, const A&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3((unsigned)threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr{};
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...) == cudaSuccess;
}

}  // namespace rz
