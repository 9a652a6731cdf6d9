// fzb_lqinv.cu -- tile-local Lorenzo inverse from codes (1-D 1024-element,
// 2-D 32x32 and 3-D 8x8x8 tiles; lorenzo_quant.cu:155-244,
// lorenzo_quant_nd.cu:112-190, :281-364), any extents.
//
// A delta is the decoded code plus, where the outlier bitmap has its bit set,
// the outlier value that mark_outliers_kernel left at the element's place in
// the output.  The reference sums with fixed add trees in FP32; when the
// deltas' magnitudes add up to no more than 2^24 in a tile every partial sum of
// any order is an exactly represented integer, so the tile is summed in the
// cheapest order.  2-D / 3-D: a warp takes 1024 / 2048 elements (a 32x32 tile,
// four 8x8x8 tiles).  A lane loads 8 consecutive codes of a row (8 rows of one
// plane in 3-D, 4 rows in 2-D, all loads ahead of their use), prefixes them
// along x in registers (2-D: with the row's other three lanes by shuffles),
// 3-D also down its rows, and stores the sums to shared memory; then the lanes
// change places, sum along the remaining axis (2-D: y, 3-D: z) with packed
// f32x2 adds and store 16 bytes each, or, where rows are not 16-byte aligned,
// one column each, so the stores stay coalesced.
// mark_outliers_kernel also leaves, per tile, the sum of the outliers'
// magnitudes (infinite for a non-integral one) and the rows that hold any, so a
// tile without outliers is known by one load, and rows without them take no
// extra work.  The condition then follows from that sum and a bound on the
// codes (in 3-D without outliers 512 deltas of at most 2^15 always meet it); a
// tile where it fails takes the reference's add tree, in a function of its own
// (inlined it cost registers): in 3-D from the deltas in shared memory, in 1-D and
// 2-D from the codes, loaded again by rows.  Read code by code from memory, with the
// bitmap for each, the trees took 283 us where 500 x 500 x 100 has 0.65 % outliers
// of up to 4e7 (now 79; 109 when every tile took them by CTAs), and 93
// for 4096 x 4096 codes of all 16 bits (now 42; 65).
//
// Bound by HBM in 2-D (2 B of code read, 4 B written an element: 8192 x 8192 in
// 87 us, 4.6 TB/s) and by load latency at the warps that 80 registers and the
// shared bricks leave (24 an SM) in 3-D.  The kernels these replaced added up
// floats with five shuffle-adds an element, and read an outlier plane of 4 B an
// element that had to be zeroed first: 8192 x 8192 177 us and 46 of zeroing,
// 3600 x 1800 15 and 9 (now 8.6), 500 x 500 x 100 with 0.8 % outliers 80 and 23
// (now 52 and 5 for the records).  Summing whole tiles in one lane's registers
// (no shared memory) left too few warps: 21 us for 3600 x 1800, 70 for
// 500 x 500 x 100.
#include "fzb_codeload.cuh"
#include "fzb_rzedec.cuh"

namespace fzb {
namespace {

constexpr float kIntSum = 16777216.0f;      // 2^24
constexpr float kSumSlack = 16700000.0f;    // a rounded sum of 1024 magnitudes below this is below 2^24
constexpr int kFewOutliers = 128;           // outliers of a warp's 2048 elements loaded one by one
constexpr int kWarps = 4;                   // warps a CTA

// The field's codes as load4 / load8 read them.
struct GlobalCodes {
    const uint16_t* p;
    __device__ __forceinline__ GlobalCodes from(uint32_t g) const { return {p + g}; }
    __device__ __forceinline__ uint32_t u16(int i) const { return __ldg(p + i); }
    __device__ __forceinline__ uint32_t u32(int i) const { return __ldg(reinterpret_cast<const uint32_t*>(p + i)); }
    __device__ __forceinline__ uint2 u64(int i) const { return __ldg(reinterpret_cast<const uint2*>(p + i)); }
    __device__ __forceinline__ uint2 u64_once(int i) const { return __ldcs(reinterpret_cast<const uint2*>(p + i)); }
    __device__ __forceinline__ uint4 u128_once(int i) const { return __ldcs(reinterpret_cast<const uint4*>(p + i)); }
    __device__ __forceinline__ uint32_t shift(uint32_t lo, uint32_t hi, uint32_t bits) const {
        return __funnelshift_r(lo, hi, bits);
    }
};

// The deltas of two packed code pairs (u - 32768 through 1.5 * 2^23 + u).
template <bool ZZ>
__device__ __forceinline__ float4 deltas4(uint2 w) {
    const uint32_t p0 = biased_pair<ZZ>(w.x), p1 = biased_pair<ZZ>(w.y);
    const float2 nb = f2(-(kMagic + 32768.0f), -(kMagic + 32768.0f));
    const float2 a = __fadd2_rn(f2(__uint_as_float(__byte_perm(p0, 0x4b400000u, 0x7610)),
                                   __uint_as_float(__byte_perm(p0, 0x4b400000u, 0x7632))), nb);
    const float2 b = __fadd2_rn(f2(__uint_as_float(__byte_perm(p1, 0x4b400000u, 0x7610)),
                                   __uint_as_float(__byte_perm(p1, 0x4b400000u, 0x7632))), nb);
    return make_float4(a.x, a.y, b.x, b.y);
}

__device__ __forceinline__ float4 add4(float4 a, float4 b) {
    const float2 x = __fadd2_rn(f2(a.x, a.y), f2(b.x, b.y)), y = __fadd2_rn(f2(a.z, a.w), f2(b.z, b.w));
    return make_float4(x.x, x.y, y.x, y.y);
}

__device__ __forceinline__ float4 mul4(float4 a, float s) {
    const float2 x = __fmul2_rn(f2(a.x, a.y), f2(s, s)), y = __fmul2_rn(f2(a.z, a.w), f2(s, s));
    return make_float4(x.x, x.y, y.x, y.y);
}

// Inclusive prefix of a row's deltas over the W lanes of a tile (W a power of
// two, aligned groups of lanes).
template <int W>
__device__ __forceinline__ float4 row_prefix(float4 v) {
    v.y = __fadd_rn(v.y, v.x);
    v.z = __fadd_rn(v.z, v.y);
    v.w = __fadd_rn(v.w, v.z);
    float inc = v.w;
#pragma unroll
    for (int d = 1; d < W; d <<= 1) {
        const float n = __shfl_up_sync(0xffffffffu, inc, d, W);
        if ((int)(threadIdx.x & (W - 1)) >= d) inc = __fadd_rn(inc, n);
    }
    const float ex = __fsub_rn(inc, v.w);  // exact: integers
    return add4(v, make_float4(ex, ex, ex, ex));
}

// A pair of codes as two words whose highest set bit grows with the delta's
// magnitude: the zigzag codes themselves, or those of plain int16 deltas.
template <bool ZZ>
__device__ __forceinline__ uint32_t abs_bits(uint32_t w) {
    if (ZZ) return w;
    const uint32_t neg = ((w >> 15) & 0x00010001u) * 0xffffu;
    return ((w << 1) & 0xfffefffeu) ^ neg;
}

// Outlier bits of elements g .. g + valid - 1, valid <= 8 (bit i: element g + i).
__device__ __forceinline__ uint32_t outlier_bits(const uint32_t* __restrict__ bits, uint32_t g, int valid) {
    if (valid <= 0) return 0u;
    const uint32_t w = g >> 5, s = g & 31u;
    uint32_t m = __ldg(bits + w) >> s;
    if (s + (uint32_t)valid > 32u) m |= __ldg(bits + w + 1) << (32u - s);
    return m & ((1u << valid) - 1u);
}

// Adds the outliers of elements g .. g + valid - 1 to their deltas: predicated
// loads, in flight together.
__device__ __forceinline__ float4 with_outliers(float4 d, const InvArgs& a, uint32_t g, int valid) {
    const uint32_t m = outlier_bits(a.obits, g, valid);
    const float* o = a.out + g;
    return add4(d, make_float4((m & 1u) ? __ldcg(o) : 0.0f, (m & 2u) ? __ldcg(o + 1) : 0.0f,
                               (m & 4u) ? __ldcg(o + 2) : 0.0f, (m & 8u) ? __ldcg(o + 3) : 0.0f));
}

// Upper bound of the magnitudes of deltas whose zigzag codes OR to `any`.
__device__ __forceinline__ float code_bound(uint32_t any) {
    any = (any | any >> 16) & 0xffffu;           // u < 2^b: |delta| <= 2^(b-1)
    return any ? (float)(1u << (31 - __clz(any))) : 0.0f;
}

// Whether magnitudes that add up to at most `bound` (a power of two) and the
// outliers' `osum` stay within 2^24.  A running sum that ever reached 2^24 cannot
// read below it, so `osum` is exact where it counts; false for infinite ones.
__device__ __forceinline__ bool sums_exact(float bound, float osum) {
    return osum < kIntSum && bound <= kIntSum - osum;
}

// Sum of four deltas' magnitudes.
template <bool ZZ>
__device__ __forceinline__ float magnitudes(uint2 w) {
    const float4 d = deltas4<ZZ>(w);
    return (fabsf(d.x) + fabsf(d.y)) + (fabsf(d.z) + fabsf(d.w));
}

// The reference's add trees, a warp one tile (in 3-D four).  rows: the steps of 128
// elements that hold outliers; mode: load4's.
template <bool ZZ>
__device__ __noinline__ void exact_tile_1d(const InvArgs& a, uint32_t base, uint32_t rows, int mode, float ebx2) {
    const uint32_t lane = threadIdx.x & 31u;
    auto deltas = [&](int vw) {
        const uint32_t g = base + 128u * vw + 4u * lane;
        const int valid = g < a.nfield ? (int)min(4u, a.nfield - g) : 0;
        float4 d = deltas4<ZZ>(load4(GlobalCodes{a.codes}, g, valid, valid != 4 ? 2 : mode));
        if ((rows >> vw) & 1u) d = with_outliers(d, a, g, valid);
        return d;
    };
    float tot[8];
    float4 next = deltas(0);
#pragma unroll
    for (int vw = 0; vw < 8; vw++) {  // the reference's eight warps of four elements a thread
        const uint32_t g0 = base + 128u * vw + 4u * lane;
        float v[4] = {next.x, next.y, next.z, next.w};
        if (vw < 7) next = deltas(vw + 1);  // loaded before this step's stores
#pragma unroll
        for (int i = 1; i < 4; i++) v[i] = __fadd_rn(v[i], v[i - 1]);
        float ts = v[3];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const float n = __shfl_up_sync(0xffffffffu, ts, d);
            if ((int)lane >= d) ts = __fadd_rn(ts, n);
        }
        const float pre = __shfl_up_sync(0xffffffffu, ts, 1);
        if (lane > 0) {
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = __fadd_rn(v[i], pre);
        }
        tot[vw] = __shfl_sync(0xffffffffu, v[3], 31);
        if (vw > 0) {
            // Hillis-Steele over the warp totals; entry vw - 1 depends on the totals before it only
            float w[8];
#pragma unroll
            for (int i = 0; i < 8; i++) w[i] = i < vw ? tot[i] : 0.0f;
#pragma unroll
            for (int d = 1; d < 8; d <<= 1)
#pragma unroll
                for (int i = 7; i >= 1; i--)
                    if (i >= d) w[i] = __fadd_rn(w[i], w[i - d]);
            const float add = w[vw - 1];
#pragma unroll
            for (int i = 0; i < 4; i++) v[i] = __fadd_rn(v[i], add);
        }
#pragma unroll
        for (int i = 0; i < 4; i++)
            if (g0 + i < a.nfield) a.out[g0 + i] = __fmul_rn(v[i], ebx2);
    }
}

// 1-D: one warp a tile, 8 steps of 128 elements.
template <bool ZZ>
__global__ void __launch_bounds__(32 * kWarps) lq_inverse_1d_kernel(const __grid_constant__ InvArgs a, int mode) {
    follow();
    if (inv_gated_off(a)) return;
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu;
    const float ebx2 = inv_ebx2(a);
    const bool has = a.obits != nullptr && *a.out_count != 0;
    const bool vec = (reinterpret_cast<uintptr_t>(a.out) & 15u) == 0;
    const uint32_t ntiles = (a.nfield + 1023u) / 1024u;
    for (uint32_t tile = blockIdx.x * kWarps + (threadIdx.x >> 5); tile < ntiles; tile += gridDim.x * kWarps) {
        const uint32_t base = tile * 1024u, g0 = base + 4u * lane;
        const float osum = has ? __uint_as_float(__ldg(a.otiles + 3u * tile)) : 0.0f;
        const uint32_t rows = has ? __ldg(a.otiles + 3u * tile + 1) : 0u;
        uint2 w[8];
        uint32_t ors = 0;
        auto valid = [&](int k) { return g0 + 128u * k < a.nfield ? (int)min(4u, a.nfield - (g0 + 128u * k)) : 0; };
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const int v = valid(k);
            w[k] = load4(GlobalCodes{a.codes}, g0 + 128u * k, v, v != 4 ? 2 : mode);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) ors |= abs_bits<ZZ>(w[k].x) | abs_bits<ZZ>(w[k].y);
        ors = __reduce_or_sync(full, ors);
        if (!sums_exact(1024.0f * code_bound(ors), osum)) {
            float s = 0.0f;  // the deltas' own magnitudes instead of their bound
#pragma unroll
            for (int k = 0; k < 8; k++) s += magnitudes<ZZ>(w[k]);
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) s += __shfl_xor_sync(full, s, d);
            if (!(s + osum < kSumSlack)) {
                exact_tile_1d<ZZ>(a, base, rows, mode, ebx2);
                continue;
            }
        }
        float carry = 0.0f;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            float4 d = deltas4<ZZ>(w[k]);
            const int v = valid(k);
            if ((rows >> k) & 1u) d = with_outliers(d, a, g0 + 128u * k, v);
            d = add4(row_prefix<32>(d), make_float4(carry, carry, carry, carry));
            carry = __shfl_sync(full, d.w, 31);
            const float4 y = mul4(d, ebx2);
            float* o = a.out + g0 + 128u * k;
            if (vec && v == 4) {
                *reinterpret_cast<float4*>(o) = y;
            } else {
                if (v > 0) o[0] = y.x;
                if (v > 1) o[1] = y.y;
                if (v > 2) o[2] = y.z;
                if (v > 3) o[3] = y.w;
            }
        }
    }
}

// The outliers of four 3-D tiles with many: a lane a column, row after row, so that a
// load takes a line of the field and not eight floats of each of 32 rows.  m: byte y
// flags those of row y of the lane's plane and tile (plane lane / 4, tile lane % 4);
// out: the lane's tile's first element.
__device__ __noinline__ void stage_columns(const float* out, uint32_t nx, uint32_t plane, uint64_t m, float* brick) {
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu, t = lane >> 3, x = lane & 7u;
    const float* col = reinterpret_cast<const float*>(__shfl_sync(full, reinterpret_cast<uint64_t>(out), t)) + x;
    __syncwarp();  // the rows' zeros are in place
    for (uint32_t z = 0; z < 8; z++, col += plane) {
        const uint32_t lo = __shfl_sync(full, (uint32_t)m, 4 * z + t) >> x,
                       hi = __shfl_sync(full, (uint32_t)(m >> 32), 4 * z + t) >> x;
        float v[8];
#pragma unroll
        for (uint32_t y = 0; y < 8; y++) v[y] = ((y < 4 ? lo : hi) >> (8u * (y & 3u))) & 1u ? __ldcg(col + y * nx) : 0.0f;
#pragma unroll
        for (uint32_t y = 0; y < 8; y++) brick[260u * z + 32u * y + lane] = v[y];
    }
    __syncwarp();
}

// Places the outliers of this lane's rows into its own part of the shared tile:
// row i's eight floats at p + pitch * i, written for the rows flagged in `rows`
// only.  The bitmap words and then the values of all rows are in flight
// together (their latencies one after another were most of the time of a field
// with 0.8 % outliers).  In 3-D, where a warp has more than kFewOutliers, it loads
// none and returns their bits, for stage_columns (500 x 500 x 100 with 12 % outliers
// 163 us for the inverse, now 105, but 91 instead of 84 with 3 % by columns; in 2-D such
// a call cost registers).
template <int ROWS>
__device__ __forceinline__ uint64_t stage_outliers(const InvArgs& a, uint32_t g0, uint32_t step, int valid,
                                                   uint32_t rows, float* p, uint32_t pitch) {
    uint64_t m = 0;
#pragma unroll
    for (int i = 0; i < ROWS; i++) {
        if ((rows >> i) & 1u) {
            m |= (uint64_t)outlier_bits(a.obits, g0 + i * step, valid) << (8 * i);
            *reinterpret_cast<float4*>(p + pitch * i) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
            *reinterpret_cast<float4*>(p + pitch * i + 4) = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    if (ROWS == 8 && __reduce_add_sync(0xffffffffu, __popcll(m)) > kFewOutliers) return m;
    while (__any_sync(0xffffffffu, m != 0)) {
        float v[4];
        int at[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            at[k] = __ffsll((long long)m) - 1;
            m &= m - 1;
            v[k] = at[k] >= 0 ? __ldcg(a.out + g0 + (at[k] >> 3) * step + (at[k] & 7)) : 0.0f;
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (at[k] >= 0) p[pitch * (at[k] >> 3) + (at[k] & 7)] = v[k];
    }
    return 0;
}

// Bit k: row r + 8k of a 2-D tile holds outliers.
__device__ __forceinline__ uint32_t lane_rows(uint32_t rows, uint32_t r) {
    return ((rows >> r) & 1u) | ((rows >> (r + 7u)) & 2u) | ((rows >> (r + 14u)) & 4u) | ((rows >> (r + 21u)) & 8u);
}

// Eight deltas, with the outliers staged at p when the row has any.
template <bool ZZ>
__device__ __forceinline__ void deltas8(const uint32_t (&w)[4], bool row, const float* p, float4& lo, float4& hi) {
    lo = deltas4<ZZ>(make_uint2(w[0], w[1]));
    hi = deltas4<ZZ>(make_uint2(w[2], w[3]));
    if (row) {
        lo = add4(lo, *reinterpret_cast<const float4*>(p));
        hi = add4(hi, *reinterpret_cast<const float4*>(p + 4));
    }
}

// Their x prefix.
template <bool ZZ>
__device__ __forceinline__ void prefix8(const uint32_t (&w)[4], bool row, const float* p, float4& lo, float4& hi) {
    deltas8<ZZ>(w, row, p, lo, hi);
    lo.y = __fadd_rn(lo.y, lo.x);
    lo.z = __fadd_rn(lo.z, lo.y);
    lo.w = __fadd_rn(lo.w, lo.z);
    hi.x = __fadd_rn(hi.x, lo.w);
    hi.y = __fadd_rn(hi.y, hi.x);
    hi.z = __fadd_rn(hi.z, hi.y);
    hi.w = __fadd_rn(hi.w, hi.z);
}

// The add trees of a 2-D tile: its deltas go to the strip first (36 floats a row).
template <bool ZZ>
__device__ __noinline__ void exact_tile_2d(const InvArgs& a, float* strip, uint32_t x0, uint32_t y0, uint32_t rows,
                                           int mode, float ebx2) {
    const uint32_t lane = threadIdx.x & 31u, r = lane >> 2, x = x0 + 8u * (lane & 3u);
    const int nv = x < a.nx ? (int)min(8u, a.nx - x) : 0, ny = (int)min(32u, a.ny - y0);
    const uint32_t g0 = (y0 + r) * a.nx + x;
    float* mine = strip + 36u * r + 8u * (lane & 3u);
    const uint32_t lrows = lane_rows(rows, r);
    if (rows) stage_outliers<4>(a, g0, 8u * a.nx, nv, lrows, mine, 36u * 8u);
#pragma unroll
    for (int k = 0; k < 4; k++) {
        uint32_t w[4];
        load8(GlobalCodes{a.codes}, g0 + 8 * k * a.nx, (int)r + 8 * k < ny ? nv : 0, mode, w);
        float4 lo, hi;
        float* p = mine + 36 * 8 * k;
        deltas8<ZZ>(w, (lrows >> k) & 1u, p, lo, hi);
        *reinterpret_cast<float4*>(p) = lo;
        *reinterpret_cast<float4*>(p + 4) = hi;
    }
    __syncwarp();
    float* out = a.out + (size_t)y0 * a.nx + x0 + lane;  // the lane's column
    float tot[4];
#pragma unroll
    for (int wy = 0; wy < 4; wy++) {  // the reference's four groups of 8 rows
        float v[8];
#pragma unroll
        for (int i = 0; i < 8; i++) v[i] = strip[36 * (8 * wy + i) + lane];
#pragma unroll
        for (int i = 1; i < 8; i++) v[i] = __fadd_rn(v[i], v[i - 1]);
        tot[wy] = v[7];
        if (wy > 0) {
            float add = tot[0];
            if (wy > 1) add = __fadd_rn(add, tot[1]);
            if (wy > 2) add = __fadd_rn(add, tot[2]);
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = __fadd_rn(v[i], add);
        }
#pragma unroll
        for (int d = 1; d < 32; d <<= 1)
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const float n = __shfl_up_sync(0xffffffffu, v[i], d);
                if ((int)lane >= d) v[i] = __fadd_rn(v[i], n);
            }
#pragma unroll
        for (int i = 0; i < 8; i++)
            if (x0 + lane < a.nx && 8 * wy + i < ny) out[(size_t)(8 * wy + i) * a.nx] = __fmul_rn(v[i], ebx2);
    }
    __syncwarp();
}

// The add trees of four 3-D tiles, whose deltas are in the brick (260 floats a
// plane); tile lane % 4 starts at element base and has nv x ny x nz elements.
__device__ __noinline__ void exact_brick_3d(const InvArgs& a, const float* brick, uint32_t base, int nv, int ny,
                                            int nz, float ebx2) {
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu;
    const uint32_t t = lane >> 3;  // the tile of the lane's column
    float* out = a.out + __shfl_sync(full, base, t) + (lane & 7u);
    const bool in = (int)(lane & 7u) < __shfl_sync(full, nv, t);
    const int tny = __shfl_sync(full, ny, t), tnz = __shfl_sync(full, nz, t);
    float run[8];
#pragma unroll
    for (int y = 0; y < 8; y++) {
        float w[8];
#pragma unroll
        for (int k = 0; k < 8; k++) {
            const float v = brick[260 * k + 32 * y + lane];
            run[k] = y == 0 ? v : __fadd_rn(v, run[k]);
            w[k] = run[k];
        }
#pragma unroll
        for (int d = 1; d < 8; d <<= 1)
#pragma unroll
            for (int k = 0; k < 8; k++) {
                const float n = __shfl_up_sync(full, w[k], d, 8);
                if ((int)(lane & 7u) >= d) w[k] = __fadd_rn(w[k], n);
            }
#pragma unroll
        for (int d = 1; d < 8; d <<= 1)
#pragma unroll
            for (int k = 7; k >= 1; k--)
                if (k >= d) w[k] = __fadd_rn(w[k], w[k - d]);
#pragma unroll
        for (int k = 0; k < 8; k++)
            if (in && y < tny && k < tnz) out[(size_t)k * a.plane + y * a.nx] = __fmul_rn(w[k], ebx2);
    }
    __syncwarp();
}

// 2-D: a warp a 32x32 tile.  Rows of the shared tile are padded to 36 floats,
// so that the 16-byte stores of eight lanes (two rows) fall on all banks.
template <bool ZZ, bool AL>
__global__ void __launch_bounds__(32 * kWarps)
    lq_inverse_2d_kernel(const __grid_constant__ InvArgs a, int mode) {
    __shared__ __align__(16) float strips[kWarps][32 * 36];
    follow();
    if (inv_gated_off(a)) return;
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu, r = lane >> 2, c = lane & 3u;
    float* strip = strips[threadIdx.x >> 5];
    const float ebx2 = inv_ebx2(a);
    const bool has = a.obits != nullptr && *a.out_count != 0;
    const uint32_t tx = (a.nx + 31u) / 32u, ntiles = tx * ((a.ny + 31u) / 32u);
    for (uint32_t tile = blockIdx.x * kWarps + (threadIdx.x >> 5); tile < ntiles; tile += gridDim.x * kWarps) {
        const uint32_t x0 = (tile % tx) * 32u, y0 = (tile / tx) * 32u, x = x0 + 8u * c;
        const int nv = x < a.nx ? (int)min(8u, a.nx - x) : 0;
        const uint32_t ny = min(32u, a.ny - y0), g0 = (y0 + r) * a.nx + x;
        const float osum = has ? __uint_as_float(__ldg(a.otiles + 3u * tile)) : 0.0f;
        const uint32_t rows = has ? __ldg(a.otiles + 3u * tile + 1) : 0u;
        const int tmode = AL ? mode : end_mode(mode, tile + 1u == ntiles, a.n_codes);  // AL: even rows
        uint32_t w[4][4], ors = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) load8(GlobalCodes{a.codes}, g0 + 8 * k * a.nx, r + 8 * k < ny ? nv : 0, tmode, w[k]);
#pragma unroll
        for (int k = 0; k < 4; k++)
#pragma unroll
            for (int i = 0; i < 4; i++) ors |= abs_bits<ZZ>(w[k][i]);
        ors = __reduce_or_sync(full, ors);
        if (!sums_exact(1024.0f * code_bound(ors), osum)) {
            float s = 0.0f;  // the deltas' own magnitudes instead of their bound
#pragma unroll
            for (int k = 0; k < 4; k++)
                s += magnitudes<ZZ>(make_uint2(w[k][0], w[k][1])) + magnitudes<ZZ>(make_uint2(w[k][2], w[k][3]));
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) s += __shfl_xor_sync(full, s, d);
            if (!(s + osum < kSumSlack)) {
                exact_tile_2d<ZZ>(a, strip, x0, y0, rows, tmode, ebx2);
                continue;
            }
        }
        float* mine = strip + 36u * r + 8u * c;
        const uint32_t lrows = lane_rows(rows, r);
        if (rows) stage_outliers<4>(a, g0, 8u * a.nx, nv, lrows, mine, 36u * 8u);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            float4 lo, hi;
            float* p = mine + 36u * 8u * k;
            prefix8<ZZ>(w[k], (lrows >> k) & 1u, p, lo, hi);
            float inc = hi.w;
            float n = __shfl_up_sync(full, inc, 1, 4);
            if (c >= 1) inc = __fadd_rn(inc, n);
            n = __shfl_up_sync(full, inc, 2, 4);
            if (c >= 2) inc = __fadd_rn(inc, n);
            const float ex = __fsub_rn(inc, hi.w);  // exact: integers
            const float4 e4 = make_float4(ex, ex, ex, ex);
            *reinterpret_cast<float4*>(p) = add4(lo, e4);
            *reinterpret_cast<float4*>(p + 4) = add4(hi, e4);
        }
        __syncwarp();
        if (AL) {  // a lane four columns of eight rows
            const uint32_t q = lane >> 3, x4 = 4u * (lane & 7u);
            const float* p = strip + 36u * 8u * q + x4;
            float4 v[8];
            v[0] = *reinterpret_cast<const float4*>(p);
#pragma unroll
            for (int i = 1; i < 8; i++) v[i] = add4(v[i - 1], *reinterpret_cast<const float4*>(p + 36 * i));
            float4 t = v[7];
#pragma unroll
            for (int d = 8; d <= 16; d <<= 1) {
                const float4 n = make_float4(__shfl_up_sync(full, t.x, d), __shfl_up_sync(full, t.y, d),
                                             __shfl_up_sync(full, t.z, d), __shfl_up_sync(full, t.w, d));
                if ((int)lane >= d) t = add4(t, n);
            }
            const float4 ex = make_float4(__fsub_rn(t.x, v[7].x), __fsub_rn(t.y, v[7].y), __fsub_rn(t.z, v[7].z),
                                          __fsub_rn(t.w, v[7].w));
            if (x0 + x4 < a.nx) {
                float* o = a.out + (size_t)(y0 + 8u * q) * a.nx + x0 + x4;
#pragma unroll
                for (int i = 0; i < 8; i++)
                    if (8u * q + i < ny) *reinterpret_cast<float4*>(o + (size_t)i * a.nx) = mul4(add4(v[i], ex), ebx2);
            }
        } else if (x0 + lane < a.nx) {  // a lane one column
            float run = 0.0f;
            float* o = a.out + (size_t)y0 * a.nx + x0 + lane;
#pragma unroll 8
            for (int i = 0; i < 32; i++, o += a.nx) {
                run = __fadd_rn(run, strip[36 * i + lane]);
                if (i < (int)ny) *o = __fmul_rn(run, ebx2);
            }
        }
        __syncwarp();
    }
}

// 3-D: a warp four 8x8x8 tiles (consecutive in the field's numbering of tiles),
// lane = plane * 4 + tile.  Planes of the shared brick are padded to 260 floats,
// so that the 16-byte stores of eight lanes (two planes) fall on all banks.
template <bool ZZ, bool AL>
__global__ void __launch_bounds__(32 * kWarps)
    lq_inverse_3d_kernel(const __grid_constant__ InvArgs a, int mode) {
    __shared__ __align__(16) float bricks[kWarps][8 * 260];
    follow();
    if (inv_gated_off(a)) return;
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu, z = lane >> 2, c = lane & 3u;
    float* brick = bricks[threadIdx.x >> 5];
    const float ebx2 = inv_ebx2(a);
    const bool has = a.obits != nullptr && *a.out_count != 0;
    const uint32_t tx = (a.nx + 7u) / 8u, ty = (a.ny + 7u) / 8u, ntiles = tx * ty * ((a.nz + 7u) / 8u);
    for (uint32_t wt = 4u * (blockIdx.x * kWarps + (threadIdx.x >> 5)); wt < ntiles; wt += 4u * gridDim.x * kWarps) {
        const uint32_t tile = wt + c;
        const uint32_t x0 = (tile % tx) * 8u, y0 = ((tile / tx) % ty) * 8u, z0 = (tile / (tx * ty)) * 8u;
        const uint32_t base = (z0 * a.ny + y0) * a.nx + x0, g0 = base + z * a.plane;
        const bool in = tile < ntiles;
        const int nv = in ? (int)min(8u, a.nx - x0) : 0, ny = in ? (int)min(8u, a.ny - y0) : 0;
        const int nz = in ? (int)min(8u, a.nz - z0) : 0;
        const int nvz = (int)z < nz ? nv : 0;
        float osum = 0.0f;
        uint32_t rows = 0;  // of this lane's plane
        if (has && in) {
            osum = __uint_as_float(__ldg(a.otiles + 3u * tile));
            rows = (__ldg(a.otiles + 3u * tile + 1 + (z >> 2)) >> (8u * (z & 3u))) & 0xffu;
        }
        const int tmode = AL ? mode : end_mode(mode, wt + 4u >= ntiles, a.n_codes);
        uint32_t w[8][4];
#pragma unroll
        for (int i = 0; i < 8; i++) load8(GlobalCodes{a.codes}, g0 + i * a.nx, i < ny ? nvz : 0, tmode, w[i]);
        bool exact = true;
        if (__any_sync(full, osum != 0.0f)) {  // NaN counts
            uint32_t ors = 0;
#pragma unroll
            for (int i = 0; i < 8; i++)
#pragma unroll
                for (int j = 0; j < 4; j++) ors |= abs_bits<ZZ>(w[i][j]);
            ors = __reduce_or_sync(full, ors);
            exact = !__any_sync(full, osum != 0.0f && !sums_exact(512.0f * code_bound(ors), osum));
            if (!exact) {
                float s = 0.0f;
#pragma unroll
                for (int i = 0; i < 8; i++)
                    s += magnitudes<ZZ>(make_uint2(w[i][0], w[i][1])) + magnitudes<ZZ>(make_uint2(w[i][2], w[i][3]));
#pragma unroll
                for (int d = 16; d >= 4; d >>= 1) s += __shfl_xor_sync(full, s, d);
                exact = !__any_sync(full, osum != 0.0f && !(s + osum < kSumSlack));
            }
        }
        float* p = brick + 260u * z + 8u * c;
        if (__any_sync(full, rows != 0u)) {
            const uint64_t many = stage_outliers<8>(a, g0, a.nx, nvz, rows, p, 32u);
            if (__any_sync(full, many != 0)) stage_columns(a.out + base, a.nx, a.plane, many, brick);
        }
        if (!exact) {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float4 lo, hi;
                deltas8<ZZ>(w[i], (rows >> i) & 1u, p + 32 * i, lo, hi);
                *reinterpret_cast<float4*>(p + 32 * i) = lo;
                *reinterpret_cast<float4*>(p + 32 * i + 4) = hi;
            }
            __syncwarp();
            exact_brick_3d(a, brick, base, nv, ny, nz, ebx2);
            continue;
        }
        {
            float4 ylo = make_float4(0.0f, 0.0f, 0.0f, 0.0f), yhi = ylo;
#pragma unroll
            for (int i = 0; i < 8; i++) {
                float4 lo, hi;
                prefix8<ZZ>(w[i], (rows >> i) & 1u, p + 32 * i, lo, hi);
                ylo = add4(ylo, lo);
                yhi = add4(yhi, hi);
                *reinterpret_cast<float4*>(p + 32 * i) = ylo;
                *reinterpret_cast<float4*>(p + 32 * i + 4) = yhi;
            }
        }
        __syncwarp();
        if (AL) {  // a lane four columns of two rows, all planes
            const uint32_t q = lane >> 3, x4 = lane & 7u, t = x4 >> 1;  // rows 2q, 2q + 1 of tile t
            const uint32_t ob = __shfl_sync(full, base, t) + 4u * (x4 & 1u);
            const int tnv = __shfl_sync(full, nv, t), tny = __shfl_sync(full, ny, t), tnz = __shfl_sync(full, nz, t);
            if ((int)(4u * (x4 & 1u)) < tnv) {
#pragma unroll
                for (int h = 0; h < 2; h++) {
                    const uint32_t y = 2u * q + h;
                    if ((int)y >= tny) break;
                    const float* p = brick + 32u * y + 4u * x4;
                    float* o = a.out + ob + y * a.nx;
                    float4 acc = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        acc = add4(acc, *reinterpret_cast<const float4*>(p + 260 * k));
                        if (k < tnz) *reinterpret_cast<float4*>(o + (size_t)k * a.plane) = mul4(acc, ebx2);
                    }
                }
            }
        } else {  // a lane one column
            const uint32_t t = lane >> 3;
            const uint32_t ob = __shfl_sync(full, base, t) + (lane & 7u);
            const int tnv = __shfl_sync(full, nv, t), tny = __shfl_sync(full, ny, t), tnz = __shfl_sync(full, nz, t);
            if ((int)(lane & 7u) < tnv) {
                for (int y = 0; y < tny; y++) {
                    float acc = 0.0f;
                    float* o = a.out + ob + y * a.nx;
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        acc = __fadd_rn(acc, brick[260 * k + 32 * y + lane]);
                        if (k < tnz) o[(size_t)k * a.plane] = __fmul_rn(acc, ebx2);
                    }
                }
            }
        }
        __syncwarp();
    }
}

}  // namespace

// Leaves each outlier at its index of the output, sets its bit in the zeroed
// bitmap (lorenzo_quant_kernels.cuh:23-40) and adds it to its tile's three
// zeroed words: the sum of the magnitudes (infinite for a non-integer) and the
// rows (1-D: steps of 128) that hold outliers.
__global__ void mark_outliers_kernel(InvArgs a) {
    follow();
    if (inv_gated_off(a)) return;
    const uint32_t n = min(*a.out_count, a.cap), lane = threadIdx.x & 31u, full = 0xffffffffu;
    for (uint32_t i0 = blockIdx.x * blockDim.x + threadIdx.x - lane; i0 < n; i0 += gridDim.x * blockDim.x) {
        const uint32_t i = i0 + lane, k = i < n ? a.out_idx[i] : a.n_total;
        const float o = i < n ? a.out_err[i] : 0.0f;
        if (k < a.n_total) a.out[k] = o;
        const bool in = k < a.nfield;
        uint32_t tile = 0xffffffffu, row = 0;
        if (in) {
            if (a.nz > 1) {
                const uint32_t z = k / a.plane, r = k - z * a.plane, y = r / a.nx, x = r - y * a.nx;
                tile = ((z >> 3) * ((a.ny + 7u) >> 3) + (y >> 3)) * ((a.nx + 7u) >> 3) + (x >> 3);
                row = 8u * (z & 7u) + (y & 7u);
            } else if (a.ny > 1) {
                const uint32_t y = k / a.nx, x = k - y * a.nx;
                tile = (y >> 5) * ((a.nx + 31u) >> 5) + (x >> 5);
                row = y & 31u;
            } else {
                tile = k >> 10;
                row = (k >> 7) & 7u;
            }
        }
        // runs of lanes whose outliers are in one tile row add up first (a sorted list of
        // many a tile: every one by itself took 21 us for 16.8 M values with 4 %)
        const uint32_t before = __shfl_up_sync(full, tile, 1), brow = __shfl_up_sync(full, row, 1);
        const uint32_t heads = __ballot_sync(full, lane == 0 || before != tile || brow != row);
        const uint32_t later = lane < 31 ? heads >> (lane + 1) : 0u;
        const uint32_t end = later ? lane + (uint32_t)__ffs(later) : 32u;  // the run's last lane + 1
        const bool whole = fabsf(o) <= kIntSum && truncf(o) == o;          // false for NaN
        uint32_t sum = in ? (whole ? (uint32_t)fabsf(o) : 1u << 25) : 0u;   // 2^25: past exactness
#pragma unroll
        for (uint32_t d = 1; d < 32; d <<= 1) {
            const uint32_t s = __shfl_down_sync(full, sum, d);
            if (lane + d < end) sum += s;
        }
        if (!in) continue;
        atomicOr(a.obits + (k >> 5), 1u << (k & 31u));
        if ((heads >> lane) & 1u) {
            atomicAdd(reinterpret_cast<float*>(a.otiles + 3u * tile), (float)sum);
            atomicOr(a.otiles + 3u * tile + 1 + (row >> 5), 1u << (row & 31u));
        }
    }
}

// Words of the outlier bitmap and, after it, of the tiles' outlier records.
uint64_t lq_inverse_outlier_words(int ndim, uint32_t nx, uint32_t ny, uint32_t nz, uint64_t* bit_words) {
    const uint64_t n = (uint64_t)nx * ny * nz;
    *bit_words = (n + 31u) / 32u + 1;
    const uint64_t tiles = ndim == 1 ? (n + 1023u) / 1024u
                         : ndim == 2 ? (uint64_t)((nx + 31u) / 32u) * ((ny + 31u) / 32u)
                                     : (uint64_t)((nx + 7u) / 8u) * ((ny + 7u) / 8u) * ((nz + 7u) / 8u);
    return *bit_words + 3 * tiles;
}

int launch_lq_inverse(const InvArgs& a, int ndim, unsigned max_grid, cudaStream_t s) {
    const uintptr_t pc = reinterpret_cast<uintptr_t>(a.codes), po = reinterpret_cast<uintptr_t>(a.out);
    auto grid = [&](uint64_t tiles, uint64_t per_warp) {
        const uint64_t g = (tiles + per_warp * kWarps - 1) / (per_warp * kWarps);
        return (unsigned)(g < max_grid ? (g ? g : 1) : max_grid);
    };
    if (ndim == 1) {
        const unsigned g = grid(((uint64_t)a.nfield + 1023u) / 1024u, 1);
        const int m1 = (pc & 7u) == 0 ? 0 : (pc & 3u) == 0 ? 1 : 2;
        return (int)launch_dependent(a.zigzag ? lq_inverse_1d_kernel<true> : lq_inverse_1d_kernel<false>, g, 32 * kWarps, 0,
                                     s, a, m1);
    }
    // the widest loads and stores that the rows' alignment allows
    const int mode = (pc & 15u) == 0 && a.nx % 8u == 0 ? 0 : (pc & 7u) == 0 && a.nx % 4u == 0 ? 1 : (pc & 3u) == 0 ? 2 : 3;
    const bool al = (po & 15u) == 0 && a.nx % 4u == 0;
    if (ndim == 2) {
        const unsigned g = grid((uint64_t)((a.nx + 31u) / 32u) * ((a.ny + 31u) / 32u), 1);
        auto k = a.zigzag ? (al ? lq_inverse_2d_kernel<true, true> : lq_inverse_2d_kernel<true, false>)
                          : (al ? lq_inverse_2d_kernel<false, true> : lq_inverse_2d_kernel<false, false>);
        return (int)launch_dependent(k, g, 32 * kWarps, 0, s, a, mode);
    } else {
        const unsigned g = grid((uint64_t)((a.nx + 7u) / 8u) * ((a.ny + 7u) / 8u) * ((a.nz + 7u) / 8u), 4);
        auto k = a.zigzag ? (al ? lq_inverse_3d_kernel<true, true> : lq_inverse_3d_kernel<true, false>)
                          : (al ? lq_inverse_3d_kernel<false, true> : lq_inverse_3d_kernel<false, false>);
        return (int)launch_dependent(k, g, 32 * kWarps, 0, s, a, mode);
    }
}

}  // namespace fzb
