// fzb_codeload.cuh -- rows of 16-bit codes as packed pairs, at any alignment.
//
// Src is the array of codes: from(g) is the array from element g on, u16 / u32 /
// u64 / u128 load from element i (`once`: not read again), and shift(lo, hi, bits)
// is the low word of hi:lo shifted right.  The functions compile on the host too,
// where a Src checks the bounds.
#pragma once

#include <cstdint>

#include <cuda_runtime.h>

#ifdef __CUDA_ARCH__
#define FZB_UNROLL _Pragma("unroll")
#else
#define FZB_UNROLL
#endif

namespace fzb {

constexpr int kWords8 = 2;  // load8 by 4-byte words

// load8's mode for a tile, given the field's: 4-byte words end on an even element, so
// the tile with the last of an odd number of codes, whose word ends past the array,
// takes single ones.
__host__ __device__ __forceinline__ int end_mode(int mode, bool last_tile, uint32_t n_codes) {
    return mode == kWords8 && last_tile && (n_codes & 1u) ? mode + 1 : mode;
}

// Four codes from element g on (`valid` of them, the rest zero) as two packed
// pairs; mode 0: element g is 8-byte aligned and valid is 0 or 4; 1: the array is
// 4-byte aligned, g even and valid 4; 2: single codes.
template <class Src>
__host__ __device__ __forceinline__ uint2 load4(const Src& src, uint32_t g, int valid, int mode) {
    if (valid <= 0) return make_uint2(0u, 0u);
    const Src c = src.from(g);
    if (mode == 0) return c.u64_once(0);
    uint2 w = make_uint2(0u, 0u);
    if (mode == 1) {
        w.x = c.u32(0);
        w.y = c.u32(2);
    } else {
        w.x = c.u16(0);
        if (valid > 1) w.x |= c.u16(1) << 16;
        if (valid > 2) w.y = c.u16(2);
        if (valid > 3) w.y |= c.u16(3) << 16;
    }
    return w;
}

// Eight codes from element g on (`valid` of them, the rest zero) as four packed
// pairs.  mode 0: element g is 16-byte aligned, 1: 8-byte aligned (and valid a
// multiple of 4), 2 (kWords8): the array is 4-byte aligned, 3: single codes.
template <class Src>
__host__ __device__ __forceinline__ void load8(const Src& src, uint32_t g, int valid, int mode, uint32_t (&w)[4]) {
FZB_UNROLL
    for (int i = 0; i < 4; i++) w[i] = 0u;
    if (valid <= 0) return;
    if (mode == 0 && valid == 8) {
        const uint4 q = src.from(g).u128_once(0);
        w[0] = q.x, w[1] = q.y, w[2] = q.z, w[3] = q.w;
        return;
    }
    if (mode <= 1) {
        const Src c = src.from(g);
        const uint2 q = c.u64(0);
        w[0] = q.x, w[1] = q.y;
        if (valid > 4) {
            const uint2 h = c.u64(4);
            w[2] = h.x, w[3] = h.y;
        }
        return;
    }
    if (mode == kWords8) {
        const uint32_t odd = g & 1u;
        const Src c = src.from(g - odd);
        uint32_t v[5];
FZB_UNROLL
        for (int i = 0; i < 5; i++) v[i] = 2 * i < valid + (int)odd ? c.u32(2 * i) : 0u;
FZB_UNROLL
        for (int i = 0; i < 4; i++) w[i] = c.shift(v[i], v[i + 1], 16u * odd);
    } else {
        const Src c = src.from(g);
FZB_UNROLL
        for (int i = 0; i < 8; i++)
            if (i < valid) w[i >> 1] |= c.u16(i) << (16 * (i & 1));
    }
    if (valid < 8) {
FZB_UNROLL
        for (int i = 0; i < 4; i++) {
            if (2 * i >= valid) w[i] = 0u;
            else if (2 * i + 1 >= valid) w[i] &= 0xffffu;
        }
    }
}

}  // namespace fzb
