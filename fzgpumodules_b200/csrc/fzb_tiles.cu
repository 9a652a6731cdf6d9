// fzb_tiles.cu -- Lorenzo codes of 2-D and 3-D fields of any extents, tile by
// tile (2-D 32x32, 3-D 8x8x8; lorenzo_quant_nd.cu:40-120, :200-280).
//
// The prediction never leaves a tile, so a warp takes 1024 / 2048 elements
// (one 2-D tile, four 3-D tiles consecutive in the field's numbering) with no
// halo: a lane loads 8 consecutive values of a row, rounds them with packed
// adds, takes the x differences in registers (2-D: one shuffle for the left
// neighbour), the y difference from the lane above by shuffles (2-D: in
// registers for three of its four rows) and, in 3-D, the z difference against
// the plane before, kept in registers.  Rows that are not 16-byte aligned go
// through a shared strip in both directions, so that loads and stores stay
// coalesced.  Codes leave in 16-byte stores: for the fused chain into the
// chunk's 16 KiB slot of the workspace, where the chunk kernel
// (code_chunk_kernel, fzb_forward.cu) picks them up.  Outliers get the code 0
// and a bit in a.obits; their values are recomputed there.
//
// Bound by HBM on large 3-D fields (4 B read, 2 B written an element) and by
// the latency of each warp's few loads on small 2-D ones.  The chunk kernel that
// this one replaced quantized 8192 consecutive elements at a time, with up to
// four windows of neighbours staged in shared memory and divisions for every
// element's place: 500 x 500 x 100 with outliers 243 us, now 31 and 62 for the
// chunks' encoding; 3600 x 1800 28.7 us, now 11.5 and 11.9; 20 fields of 1 to
// 256 MB in one batch 1012 us, now 134 and 539.
#include "fzb_slab.cuh"

namespace fzb {
namespace {

constexpr int kTileWarps = 4;  // warps a CTA

// Marks the outliers m (bit i: element g + i) of a field's bitmap.
__device__ __forceinline__ void mark_bits(uint32_t* bits, uint32_t g, uint32_t m) {
    const uint32_t s = g & 31u;
    atomicOr(bits + (g >> 5), m << s);
    if (s > 24u && (m >> (32u - s))) atomicOr(bits + (g >> 5) + 1, m >> (32u - s));
}

// Eight codes to dst + g; smode 0: 16-byte aligned, 1: 8-byte aligned and nv a
// multiple of 4.
__device__ __forceinline__ void store8(uint16_t* dst, uint32_t g, int nv, int smode, uint2 lo, uint2 hi) {
    if (nv <= 0) return;
    if (smode == 0 && nv == 8) {
        *reinterpret_cast<uint4*>(dst + g) = make_uint4(lo.x, lo.y, hi.x, hi.y);
    } else {
        *reinterpret_cast<uint2*>(dst + g) = lo;
        if (nv > 4) *reinterpret_cast<uint2*>(dst + g + 4) = hi;
    }
}

struct TileSmem {
    __align__(16) float v[32 * 36];  // a 2-D tile's (3-D: a plane's) values, rows padded to 36
};

// left: x predecessor of q.a.x (0 at a tile's start: x - 0 is exact)
__device__ __forceinline__ Q4 xdiff(Q4 v, float left) {
    return {sub2(v.a, f2(left, v.a.x)), sub2(v.b, f2(v.a.y, v.b.x))};
}

// One 32x32 tile; lane = row group of four rows * 4 + column group.  AL: rows
// start on 16-byte boundaries of the input and smode <= 1.
template <bool ZZ, bool AL>
__device__ __forceinline__ void tile_2d(const FwdArgs& a, uint32_t tile, float r, TileSmem& sm, int smode) {
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu, rg = lane >> 2, c = lane & 3u;
    const uint32_t tx = (a.nx + 31u) / 32u;
    const uint32_t x0 = (tile % tx) * 32u, y0 = (tile / tx) * 32u, x = x0 + 8u * c, y = y0 + 4u * rg;
    const int nv = x < a.nx ? (int)min(8u, a.nx - x) : 0;
    const int ny = y < a.ny ? (int)min(4u, a.ny - y) : 0;
    const uint32_t g0 = y * a.nx + x;
    float4 lo[4], hi[4];
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (AL) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4* p = reinterpret_cast<const float4*>(a.in + g0 + k * a.nx);
            lo[k] = (k < ny && nv > 0) ? __ldg(p) : zero;
            hi[k] = (k < ny && nv > 4) ? __ldg(p + 1) : zero;
        }
    } else {
        const uint32_t rows = min(32u, a.ny - y0);
        const float* p = a.in + (size_t)y0 * a.nx + x0 + lane;
        const bool col = x0 + lane < a.nx;
#pragma unroll
        for (int h = 0; h < 4; h++) {
            float e[8];
#pragma unroll
            for (int k = 0; k < 8; k++) e[k] = (col && 8u * h + k < rows) ? __ldg(p + (size_t)(8 * h + k) * a.nx) : 0.0f;
#pragma unroll
            for (int k = 0; k < 8; k++) sm.v[36 * (8 * h + k) + lane] = e[k];
        }
        __syncwarp();
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const float4* q = reinterpret_cast<const float4*>(sm.v + 36u * (4u * rg + k) + 8u * c);
            lo[k] = q[0];
            hi[k] = q[1];
        }
        __syncwarp();  // the strip takes the codes below
    }
    Q4 ql[4], qh[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        ql[k] = quant4(lo[k], r);
        qh[k] = quant4(hi[k], r);
    }
    Q4 ul, uh;  // the row above: the upper lane's last row, zero at the tile's top
    ul.a.x = __shfl_up_sync(full, ql[3].a.x, 4);
    ul.a.y = __shfl_up_sync(full, ql[3].a.y, 4);
    ul.b.x = __shfl_up_sync(full, ql[3].b.x, 4);
    ul.b.y = __shfl_up_sync(full, ql[3].b.y, 4);
    uh.a.x = __shfl_up_sync(full, qh[3].a.x, 4);
    uh.a.y = __shfl_up_sync(full, qh[3].a.y, 4);
    uh.b.x = __shfl_up_sync(full, qh[3].b.x, 4);
    uh.b.y = __shfl_up_sync(full, qh[3].b.y, 4);
    if (rg == 0) ul = uh = Q4{f2(0.0f, 0.0f), f2(0.0f, 0.0f)};
    uint32_t* codes = reinterpret_cast<uint32_t*>(sm.v);  // code rows of 16 words, padded to 20
#pragma unroll
    for (int k = 0; k < 4; k++) {
        // y, then x (lorenzo_quant_nd.cu:72-77)
        const Q4 vl = {sub2(ql[k].a, ul.a), sub2(ql[k].b, ul.b)}, vh = {sub2(qh[k].a, uh.a), sub2(qh[k].b, uh.b)};
        const float n = __shfl_up_sync(full, vh.b.y, 1);
        uint32_t ml, mh;
        const uint2 pl = codes4<ZZ>(xdiff(vl, c ? n : 0.0f), a.radius, ml);
        const uint2 ph = codes4<ZZ>(xdiff(vh, vl.b.y), a.radius, mh);
        const int w = k < ny ? nv : 0;
        const uint32_t m = (ml | mh << 4) & ((1u << w) - 1u);
        if (m) mark_bits(a.obits, g0 + k * a.nx, m);
        if (AL) store8(a.tcodes, g0 + k * a.nx, w, smode, pl, ph);
        else *reinterpret_cast<uint4*>(codes + 20u * (4u * rg + k) + 4u * c) = make_uint4(pl.x, pl.y, ph.x, ph.y);
        ul = ql[k];
        uh = qh[k];
    }
    if (!AL) {
        __syncwarp();
        const uint32_t rows = min(32u, a.ny - y0);
        if (x0 + lane < a.nx) {
            const uint16_t* h = reinterpret_cast<const uint16_t*>(codes) + lane;
            uint16_t* o = a.tcodes + (size_t)y0 * a.nx + x0 + lane;
#pragma unroll 8
            for (uint32_t i = 0; i < 32; i++, o += a.nx)
                if (i < rows) *o = h[40 * i];
        }
        __syncwarp();
    }
}

// Four 8x8x8 tiles from `wt`; lane = row * 4 + tile, marching along z.
template <bool ZZ, bool AL>
__device__ __forceinline__ void tiles_3d(const FwdArgs& a, uint32_t wt, uint32_t ntiles, float r, TileSmem& sm,
                                         int smode) {
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu, row = lane >> 2;
    const uint32_t tx = (a.nx + 7u) / 8u, ty = (a.ny + 7u) / 8u;
    auto place = [&](uint32_t t, uint32_t& base, int& nv, int& ny, int& nz) {
        const uint32_t tile = wt + t;
        const uint32_t x0 = (tile % tx) * 8u, y0 = ((tile / tx) % ty) * 8u, z0 = (tile / (tx * ty)) * 8u;
        base = (z0 * a.ny + y0) * a.nx + x0;
        const bool in = tile < ntiles;
        nv = in ? (int)min(8u, a.nx - x0) : 0;
        ny = in ? (int)min(8u, a.ny - y0) : 0;
        nz = in ? (int)min(8u, a.nz - z0) : 0;
    };
    uint32_t base, sbase = 0;   // this lane's tile, and the one whose column it moves (not AL)
    int nv, ny, nz, snv = 0, sny = 0, snz = 0;
    place(lane & 3u, base, nv, ny, nz);
    const uint32_t g0 = base + row * a.nx;
    if ((int)row >= ny) nv = 0;
    if (!AL) {
        place(lane >> 3, sbase, snv, sny, snz);
        sbase += lane & 7u;
        if ((int)(lane & 7u) >= snv) sny = 0;
    }
    const float4 zero = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    Q4 pl = {f2(0.0f, 0.0f), f2(0.0f, 0.0f)}, ph = pl;  // the plane before
    float4 lo[2], hi[2];
    float e[8];
    auto load = [&](int z, float4& l, float4& h) {
        const float4* p = reinterpret_cast<const float4*>(a.in + g0 + (size_t)z * a.plane);
        l = (z < nz && nv > 0) ? __ldg(p) : zero;
        h = (z < nz && nv > 4) ? __ldg(p + 1) : zero;
    };
    auto load_cols = [&](int z) {
        const float* p = a.in + sbase + (size_t)z * a.plane;
#pragma unroll
        for (int k = 0; k < 8; k++) e[k] = (z < snz && k < sny) ? __ldg(p + (size_t)k * a.nx) : 0.0f;
    };
    if (AL) {
        load(0, lo[0], hi[0]);
        load(1, lo[1], hi[1]);
    } else {
        load_cols(0);
    }
    uint32_t* codes = reinterpret_cast<uint32_t*>(sm.v + 8 * 36);  // code rows of 16 words, padded to 20
#pragma unroll
    for (int z = 0; z < 8; z++) {
        float4 vl, vh;
        if (AL) {
            vl = lo[z & 1];
            vh = hi[z & 1];
            if (z < 6) load(z + 2, lo[z & 1], hi[z & 1]);
        } else {
#pragma unroll
            for (int k = 0; k < 8; k++) sm.v[36 * k + lane] = e[k];
            __syncwarp();
            const float4* q = reinterpret_cast<const float4*>(sm.v + 36u * row + 8u * (lane & 3u));
            vl = q[0];
            vh = q[1];
            if (z < 7) load_cols(z + 1);
        }
        const Q4 ql = quant4(vl, r), qh = quant4(vh, r);
        // z, x, y (lorenzo_quant_nd.cu:234-246)
        const Q4 zl = {sub2(ql.a, pl.a), sub2(ql.b, pl.b)}, zh = {sub2(qh.a, ph.a), sub2(qh.b, ph.b)};
        pl = ql;
        ph = qh;
        const Q4 bl = xdiff(zl, 0.0f), bh = xdiff(zh, zl.b.y);
        Q4 ul, uh;
        ul.a.x = __shfl_up_sync(full, bl.a.x, 4);
        ul.a.y = __shfl_up_sync(full, bl.a.y, 4);
        ul.b.x = __shfl_up_sync(full, bl.b.x, 4);
        ul.b.y = __shfl_up_sync(full, bl.b.y, 4);
        uh.a.x = __shfl_up_sync(full, bh.a.x, 4);
        uh.a.y = __shfl_up_sync(full, bh.a.y, 4);
        uh.b.x = __shfl_up_sync(full, bh.b.x, 4);
        uh.b.y = __shfl_up_sync(full, bh.b.y, 4);
        if (row == 0) ul = uh = Q4{f2(0.0f, 0.0f), f2(0.0f, 0.0f)};
        uint32_t ml, mh;
        const uint2 cl = codes4<ZZ>(Q4{sub2(bl.a, ul.a), sub2(bl.b, ul.b)}, a.radius, ml);
        const uint2 ch = codes4<ZZ>(Q4{sub2(bh.a, uh.a), sub2(bh.b, uh.b)}, a.radius, mh);
        const int w = z < nz ? nv : 0;
        const uint32_t m = (ml | mh << 4) & ((1u << w) - 1u);
        const uint32_t g = g0 + z * a.plane;
        if (m) mark_bits(a.obits, g, m);
        if (AL) {
            store8(a.tcodes, g, w, smode, cl, ch);
        } else {
            *reinterpret_cast<uint4*>(codes + 20u * row + 4u * (lane & 3u)) = make_uint4(cl.x, cl.y, ch.x, ch.y);
            __syncwarp();
            const uint16_t* h = reinterpret_cast<const uint16_t*>(codes) + lane;
            uint16_t* o = a.tcodes + sbase + (size_t)z * a.plane;
            if (z < snz) {
#pragma unroll
                for (int k = 0; k < 8; k++)
                    if (k < sny) o[(size_t)k * a.nx] = h[40 * k];
            }
        }
    }
    if (!AL) __syncwarp();
}

// How a field's rows are read and written: bit 0 aligned input rows, bits 1-2
// the store mode (0: 16 bytes, 1: 8 bytes, else single codes).
__device__ __host__ __forceinline__ int tile_modes(const FwdArgs& a) {
    const bool r4 = a.nx % 4u == 0;
    const uintptr_t po = reinterpret_cast<uintptr_t>(a.tcodes);
    const int smode = (po & 15u) == 0 && a.nx % 8u == 0 ? 0 : (po & 7u) == 0 && r4 ? 1 : 2;
    return ((reinterpret_cast<uintptr_t>(a.in) & 15u) == 0 && r4 && smode < 2 ? 1 : 0) | smode << 1;
}

template <bool ZZ>
__device__ __forceinline__ void tile_block(const FwdArgs& a, uint32_t block, TileSmem& sm) {
    const uint32_t warp = block * kTileWarps + (threadIdx.x >> 5);
    const float r = *a.ebx2_r;
    const int modes = tile_modes(a), smode = modes >> 1;
    if (a.nz > 1) {
        const uint32_t n = ((a.nx + 7u) / 8u) * ((a.ny + 7u) / 8u) * ((a.nz + 7u) / 8u), wt = 4u * warp;
        if (wt >= n) return;
        if (modes & 1) tiles_3d<ZZ, true>(a, wt, n, r, sm, smode);
        else tiles_3d<ZZ, false>(a, wt, n, r, sm, smode);
    } else {
        if (warp >= ((a.nx + 31u) / 32u) * ((a.ny + 31u) / 32u)) return;
        if (modes & 1) tile_2d<ZZ, true>(a, warp, r, sm, smode);
        else tile_2d<ZZ, false>(a, warp, r, sm, smode);
    }
}

__global__ void __launch_bounds__(32 * kTileWarps, 8) lq_tiles_kernel(const __grid_constant__ FwdArgs a) {
    follow();
    __shared__ TileSmem sm[kTileWarps];
    if (a.zigzag) tile_block<true>(a, blockIdx.x, sm[threadIdx.x >> 5]);
    else tile_block<false>(a, blockIdx.x, sm[threadIdx.x >> 5]);
}

// The tiles of a batch's 2-D and 3-D fields (eight CTAs an SM: 127 us for twenty
// fields of 0.96 GB, 134 with six): CTAs [tile_begin[i], tile_begin[i + 1])
// belong to the field of slot i of unit_order.
__global__ void __launch_bounds__(32 * kTileWarps, 8) batch_tiles_kernel(BatchArgs b) {
    __shared__ TileSmem sm[kTileWarps];
    uint32_t lo = 0, hi = b.nfields;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (b.tile_begin[mid] <= blockIdx.x) lo = mid;
        else hi = mid;
    }
    const FwdArgs& a = b.fields[b.unit_order[lo]].a;
    const uint32_t block = blockIdx.x - b.tile_begin[lo];
    if (a.zigzag) tile_block<true>(a, block, sm[threadIdx.x >> 5]);
    else tile_block<false>(a, block, sm[threadIdx.x >> 5]);
}

}  // namespace

uint32_t lq_tile_blocks(const FwdArgs& a) {
    const uint64_t warps = a.nz > 1 ? ((uint64_t)((a.nx + 7u) / 8u) * ((a.ny + 7u) / 8u) * ((a.nz + 7u) / 8u) + 3) / 4
                                    : (uint64_t)((a.nx + 31u) / 32u) * ((a.ny + 31u) / 32u);
    return (uint32_t)((warps + kTileWarps - 1) / kTileWarps);
}

int launch_lq_tiles(const FwdArgs& a, cudaStream_t s) {
    return (int)launch_dependent(lq_tiles_kernel, lq_tile_blocks(a), 32 * kTileWarps, 0, s, a);
}

int launch_batch_tiles(const BatchArgs& b, uint32_t blocks, cudaStream_t s) {
    batch_tiles_kernel<<<blocks, 32 * kTileWarps, 0, s>>>(b);
    return (int)cudaGetLastError();
}

}  // namespace fzb
