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
// (lq_chunk_kernel, fzb_forward.cu) picks them up.  Outliers get the code 0
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

// A field whose tiles are mostly empty (lq_cells: a few columns, rows or planes in
// tiles of 32 or 8), where tile_2d and tiles_3d leave their lanes idle: a warp takes
// kCellRun consecutive elements, W a lane and step, and forms each delta from the
// element and its neighbours above and in the plane before, loaded as they are
// (mostly from L1); the x difference is against the lane before.  A neighbour of
// another tile counts as 0 (q - 0 is exact).  W = 4 where rows are a multiple of
// four elements and 16-byte aligned, else 1.
//
// Bound by instruction issue.  16.8 M elements with the chunks' encoding behind (us,
// tiles -> cells): 2-D 1 wide 629 -> 72, 4 wide 119 -> 57, 7 wide 125 -> 72, 8 wide
// 78 -> 57, two rows 195 -> 60; 3-D 1 x 1 1368 -> 98, 2 x 500 136 -> 93, 1000 x 1
// 127 -> 69.  The line lies where both meet: in 2-D at 9/16 of the tiles filled (16
// wide 59.7 and 57.0, 33 wide 75 and 72, but 40 wide, 10/16, 57.3 and 57.5), in 3-D,
// where the cells read up to four elements for one, at 3/8 (1000 x 3 69.8 and 69.8,
// 3 x 300 105 and 93, but 4 x 256, 4/8, 61 and 67).
constexpr uint32_t kCellRun = 1024;

// k / d and k % d for k < 2^31, m = 0xffffffff / d: the estimate is at most one
// too small.
__device__ __forceinline__ uint32_t split(uint32_t k, uint32_t d, uint32_t m, uint32_t& rem) {
    uint32_t q = __umulhi(k, m);
    rem = k - q * d;
    if (rem >= d) {
        rem -= d;
        q++;
    }
    return q;
}

// W elements from k on and their neighbours (0 outside the tile or the field);
// tx: the first one has an x predecessor in its tile.
template <int W>
struct Cells {
    float v[W], up[W], back[W], upback[W];
    bool tx;
};

template <int W>
__device__ __forceinline__ void load_cells(const float* p, bool in, float (&v)[W]) {
    if (W == 4) {
        const float4 q = in ? __ldg(reinterpret_cast<const float4*>(p)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        v[0] = q.x, v[1 % W] = q.y, v[2 % W] = q.z, v[3 % W] = q.w;
    } else {
        v[0] = in ? __ldg(p) : 0.0f;
    }
}

// The differences along z (3-D) or y (2-D).
template <int W>
__device__ __forceinline__ void quant_sub(const float (&v)[W], const float (&w)[W], float r, float (&d)[W]) {
    if (W == 4) {
        const Q4 a = quant4(make_float4(v[0], v[1 % W], v[2 % W], v[3 % W]), r);
        const Q4 b = quant4(make_float4(w[0], w[1 % W], w[2 % W], w[3 % W]), r);
        const float2 x = sub2(a.a, b.a), y = sub2(a.b, b.b);
        d[0] = x.x, d[1 % W] = x.y, d[2 % W] = y.x, d[3 % W] = y.y;
    } else {
        auto q = [&](float u) { return truncf(__fadd_rn(__fmul_rn(u, r), __uint_as_float(half_bits(u)))); };
        d[0] = __fsub_rn(q(v[0]), q(w[0]));
    }
}

template <int NDIM, bool ZZ, int W>
__device__ __forceinline__ void cells(const FwdArgs& a, uint32_t warp, float r) {
    constexpr uint32_t kIn = NDIM == 3 ? 7u : 31u;  // a place in the tile: its low bits
    constexpr int U = W == 4 ? 2 : 4;               // steps with their loads in flight together
    const uint32_t lane = threadIdx.x & 31u, full = 0xffffffffu, n = a.nfield, k0 = warp * kCellRun;
    if (k0 >= n) return;
    const uint32_t my = ~0u / a.nx, mz = NDIM == 3 ? ~0u / a.plane : 0u;
    auto load = [&](uint32_t k, Cells<W>& c) {
        uint32_t rem = k, x;
        const bool in = k < n, tz = NDIM == 3 && in && (split(k, a.plane, mz, rem) & kIn) != 0;
        const bool ty = (split(rem, a.nx, my, x) & kIn) != 0 && in;
        c.tx = (x & kIn) != 0;
        const float* p = a.in + k;
        load_cells<W>(p, in, c.v);
        load_cells<W>(p - a.nx, ty, c.up);
        if (NDIM == 3) {
            load_cells<W>(p - a.plane, tz, c.back);
            load_cells<W>(p - a.plane - a.nx, ty && tz, c.upback);
        }
    };
    auto first = [&](const Cells<W>& c, float (&d)[W], float (&du)[W]) {
        quant_sub<W>(c.v, NDIM == 3 ? c.back : c.up, r, d);
        if (NDIM == 3) quant_sub<W>(c.up, c.upback, r, du);
    };
    float cd = 0.0f, cu = 0.0f;  // of the element before the run
    if (k0) {
        Cells<W> c;
        float d[W], du[W];
        load(k0 - W, c);
        first(c, d, du);
        cd = d[W - 1];
        if (NDIM == 3) cu = du[W - 1];
    }
    for (uint32_t b = k0; b < min(n, k0 + kCellRun); b += 32u * W * U) {
        Cells<W> c[U];
#pragma unroll
        for (int i = 0; i < U; i++) load(b + W * (32u * i + lane), c[i]);
#pragma unroll
        for (int i = 0; i < U; i++) {
            float d[W], du[W];
            first(c[i], d, du);
            const float nd = __shfl_up_sync(full, d[W - 1], 1), ld = lane ? nd : cd;
            cd = __shfl_sync(full, d[W - 1], 31);
            float lu = 0.0f;
            if (NDIM == 3) {
                const float nu = __shfl_up_sync(full, du[W - 1], 1);
                lu = lane ? nu : cu;
                cu = __shfl_sync(full, du[W - 1], 31);
            }
            // 2-D: y, x (lorenzo_quant_nd.cu:72-77); 3-D: z, x, y (:234-246)
            const uint32_t k = b + W * (32u * i + lane);
            if (W == 4) {
                Q4 e = xdiff(Q4{f2(d[0], d[1 % W]), f2(d[2 % W], d[3 % W])}, c[i].tx ? ld : 0.0f);
                if (NDIM == 3) {
                    const Q4 u = xdiff(Q4{f2(du[0], du[1 % W]), f2(du[2 % W], du[3 % W])}, c[i].tx ? lu : 0.0f);
                    e = Q4{sub2(e.a, u.a), sub2(e.b, u.b)};
                }
                uint32_t m;
                const uint2 p = codes4<ZZ>(e, a.radius, m);
                if (k < n) {
                    *reinterpret_cast<uint2*>(a.tcodes + k) = p;
                    if (m) mark_bits(a.obits, k, m);
                }
            } else {
                float e = __fsub_rn(d[0], c[i].tx ? ld : 0.0f);
                if (NDIM == 3) e = __fsub_rn(e, __fsub_rn(du[0], c[i].tx ? lu : 0.0f));
                const bool in = fabsf(e) < a.radius;
                const uint32_t m = __ballot_sync(full, !in && k < n);
                if (k < n) a.tcodes[k] = (uint16_t)code_pair<ZZ>(f2(in ? e : 0.0f, 0.0f));
                if (m && lane == 0) a.obits[(b >> 5) + i] = m;
            }
        }
    }
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

template <bool ZZ>
__device__ __forceinline__ void cells_block(const FwdArgs& a, uint32_t block) {
    const uint32_t warp = block * kTileWarps + (threadIdx.x >> 5);
    const float r = *a.ebx2_r;
    if (tile_modes(a) & 1) a.nz > 1 ? cells<3, ZZ, 4>(a, warp, r) : cells<2, ZZ, 4>(a, warp, r);
    else a.nz > 1 ? cells<3, ZZ, 1>(a, warp, r) : cells<2, ZZ, 1>(a, warp, r);
}

// Eight CTAs an SM leave 64 registers, 40 bytes of which the compiler spills.
__global__ void __launch_bounds__(32 * kTileWarps, 8) lq_tiles_kernel(const __grid_constant__ FwdArgs a) {
    follow();
    __shared__ TileSmem sm[kTileWarps];
    if (a.zigzag) tile_block<true>(a, blockIdx.x, sm[threadIdx.x >> 5]);
    else tile_block<false>(a, blockIdx.x, sm[threadIdx.x >> 5]);
}

// A kernel of its own: beside the tiles' code the tiles of 501 x 500 x 99 took 3 us
// longer.
__global__ void __launch_bounds__(32 * kTileWarps, 8) lq_cells_kernel(const __grid_constant__ FwdArgs a) {
    follow();
    if (a.zigzag) cells_block<true>(a, blockIdx.x);
    else cells_block<false>(a, blockIdx.x);
}

// The tiles of a batch's 2-D and 3-D fields (eight CTAs an SM: 127 us for twenty
// fields of 0.96 GB, 134 with six), or the elements of those that take cells():
// block b of [tile_begin[i], tile_begin[i + 1]), `first` being the grid's, belongs to
// the field of slot i of unit_order.
template <bool CELLS>
__global__ void __launch_bounds__(32 * kTileWarps, 8) batch_tiles_kernel(BatchArgs b, uint32_t first) {
    __shared__ TileSmem sm[CELLS ? 1 : kTileWarps];
    uint32_t lo = 0, hi = b.nfields;
    while (hi - lo > 1) {
        const uint32_t mid = (lo + hi) >> 1;
        if (b.tile_begin[mid] <= first + blockIdx.x) lo = mid;
        else hi = mid;
    }
    const FwdArgs& a = b.fields[b.unit_order[lo]].a;
    const uint32_t block = first + blockIdx.x - b.tile_begin[lo];
    if (CELLS) {
        if (a.zigzag) cells_block<true>(a, block);
        else cells_block<false>(a, block);
    } else {
        if (a.zigzag) tile_block<true>(a, block, sm[threadIdx.x >> 5]);
        else tile_block<false>(a, block, sm[threadIdx.x >> 5]);
    }
}

}  // namespace

bool lq_cells(uint32_t ndim, uint32_t nx, uint32_t ny, uint32_t nz) {
    auto up = [](uint32_t v, uint32_t to) { return (uint64_t)((v + to - 1) / to * to); };
    const uint64_t n = (uint64_t)nx * ny * nz;
    return ndim == 2 ? 16 * n <= 9 * up(nx, 32) * up(ny, 32) : 8 * n <= 3 * up(nx, 8) * up(ny, 8) * up(nz, 8);
}

uint32_t lq_tile_blocks(const FwdArgs& a) {
    const uint64_t warps = a.cells ? (a.nfield + kCellRun - 1u) / kCellRun
                         : a.nz > 1 ? ((uint64_t)((a.nx + 7u) / 8u) * ((a.ny + 7u) / 8u) * ((a.nz + 7u) / 8u) + 3) / 4
                                    : (uint64_t)((a.nx + 31u) / 32u) * ((a.ny + 31u) / 32u);
    return (uint32_t)((warps + kTileWarps - 1) / kTileWarps);
}

int launch_lq_tiles(const FwdArgs& a, cudaStream_t s) {
    return (int)launch_dependent(a.cells ? lq_cells_kernel : lq_tiles_kernel, lq_tile_blocks(a), 32 * kTileWarps, 0, s, a);
}

int launch_batch_tiles(const BatchArgs& b, uint32_t tiles, uint32_t cells, cudaStream_t s) {
    if (tiles) batch_tiles_kernel<false><<<tiles, 32 * kTileWarps, 0, s>>>(b, 0);
    if (cells) batch_tiles_kernel<true><<<cells, 32 * kTileWarps, 0, s>>>(b, tiles);
    return (int)cudaGetLastError();
}

}  // namespace fzb
