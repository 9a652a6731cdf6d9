// fzb_common.cuh -- device helpers shared by the sm_100a hot-path kernels.
//
// Dependent launches, rounding, code mapping, block scans, the 16x16 in-register
// bit transpose used by Bitshuffle, and byte-mask helpers used by RZE.
#pragma once

#include <cstdint>
#include <utility>

#include <cuda_runtime.h>

namespace fzb {

// Launches `kernel` as a programmatic dependent of the previous kernel on
// `s` (it may start before that kernel ends and must wait with
// griddepcontrol.wait before reading its results, see follow()); a plain launch
// when the attribute is refused.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_dependent(void (*kernel)(KArgs...), dim3 grid, unsigned block, size_t smem,
                                    cudaStream_t s, Args&&... args) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(block);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        kernel<<<grid, block, smem, s>>>(std::forward<Args>(args)...);
        e = cudaGetLastError();
    }
    return e;
}

// First statement of a kernel that is launched by launch_dependent: waits for the
// kernels before it, then lets the next one be placed as soon as this grid's last
// blocks are (an empty statement in a plain launch).  The blocks of the next
// kernel are in place and waiting when this one ends: 64^3 both ways 84 us
// against 96 with plain launches, 3600 x 1800 118 against 133.
__device__ __forceinline__ void follow() {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    asm volatile("griddepcontrol.launch_dependents;");
}

constexpr int kThreads = 256;            // threads per chunk CTA
constexpr uint32_t kCtrlWords = 64;      // control words at the head of a workspace, zero when a call begins
constexpr int kChunkBytes = 16384;       // Bitshuffle block == RZE chunk
constexpr int kChunkCodes = kChunkBytes / 2;  // u16 codes per chunk
constexpr int kRzeAvail = kChunkBytes - 2;    // rze_stage.cu:369

// Device error word bits (workspace[0]); read by the host after the launch.
constexpr uint32_t kErrLookbackTimeout = 1u;  // reported for it; no kernel sets it
constexpr uint32_t kErrMalformed = 2u;
constexpr uint32_t kErrInexact = 4u;      // fused inverse left the exact-integer regime
constexpr uint32_t kErrUnsorted = 8u;     // outlier indices not ascending
constexpr uint32_t kErrTmaTimeout = 16u;  // a TMA copy did not complete within its bound

// Round half away from zero (the float overload of `round` that the
// reference applies to x * ebx2_r).  v - trunc(v) is exact in FP32.
__device__ __forceinline__ float round_half_away(float v) {
    float t = truncf(v);
    float d = __fsub_rn(v, t);
    float s = __int_as_float((__float_as_int(v) & 0x80000000) | 0x3f800000);  // +-1
    return (fabsf(d) >= 0.5f) ? __fadd_rn(t, s) : t;
}

// Delta of a code, plain int16 or zigzag (zigzag.h:80-84).
__device__ __forceinline__ float decode_code(uint32_t u, bool zigzag) {
    if (zigzag) {
        int s = (int)((u >> 1) ^ (0u - (u & 1u)));
        return (float)(int16_t)s;
    }
    return (float)(int16_t)u;
}

// ---------------------------------------------------------------- scans

__device__ __forceinline__ uint32_t warp_incl_scan(uint32_t v) {
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t n = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= d) v += n;
    }
    return v;
}

// Block-wide exclusive scan for kThreads threads.  `ws` needs 9 u32 of smem.
// Returns the exclusive prefix; *total receives the block sum.
__device__ __forceinline__ uint32_t block_excl_scan(uint32_t v, uint32_t* ws, uint32_t* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    uint32_t inc = warp_incl_scan(v);
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    if (warp == 0) {
        uint32_t t = (lane < kThreads / 32) ? ws[lane] : 0u;
        uint32_t ti = warp_incl_scan(t);
        if (lane < kThreads / 32) ws[lane] = ti - t;  // exclusive warp offsets
        if (lane == kThreads / 32 - 1) ws[8] = ti;
    }
    __syncthreads();
    uint32_t r = ws[warp] + inc - v;
    *total = ws[8];
    __syncthreads();
    return r;
}

// ---------------------------------------------------------------- bit transpose

// In-place transpose of two 16x16 bit matrices held in the low and high
// halves of x[0..15]: afterwards bit i of x[j] (per half) is what bit j of
// x[i] was.  With x[l] = code[l] | code[l+16] << 16 the result is
// x[b] = plane word of bit b over the 32 codes, i.e. exactly the word the
// reference's ballot bitshuffle (bitshuffle_stage.cu:299-323) stores at
// plane (15-b).  The transform is its own inverse.
__device__ __forceinline__ void transpose16x2(uint32_t (&x)[16]) {
    // 8x8 block swap: exchange byte 1 of x[i] with byte 0 of x[i+8] in both
    // halves (one byte permute per output word).
#pragma unroll
    for (int i = 0; i < 8; i++) {
        uint32_t a = x[i], b = x[i + 8];
        x[i] = __byte_perm(a, b, 0x6240);      // a.b0, b.b0, a.b2, b.b2
        x[i + 8] = __byte_perm(a, b, 0x7351);  // a.b1, b.b1, a.b3, b.b3
    }
#pragma unroll
    for (int s = 4; s >= 1; s >>= 1) {
        const uint32_t m = (s == 4) ? 0x0f0f0f0fu : (s == 2) ? 0x33333333u : 0x55555555u;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            if (i & s) continue;
            uint32_t t = ((x[i] >> s) ^ x[i + s]) & m;
            x[i + s] ^= t;
            x[i] ^= t << s;
        }
    }
}

// ---------------------------------------------------------------- byte masks

// 4-bit mask of the nonzero bytes of w (bit k <-> byte k).
__device__ __forceinline__ uint32_t nz_nibble(uint32_t w) {
    uint32_t hi = (((w & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w) & 0x80808080u;
    return (hi * 0x00204081u) >> 28;
}

__device__ __forceinline__ uint32_t nz_byte_mask64(uint64_t w) {
    return nz_nibble((uint32_t)w) | (nz_nibble((uint32_t)(w >> 32)) << 4);
}

}  // namespace fzb
