// fzb_coders.cu -- RLE and Bitpack coders plus the device-wide scan they use.
//
// RLE wire format (modules/coders/rle/rle.h:22, rle.cu:119-148):
//   [u32 runs][values T x runs, padded to 4 bytes with zeros][u32 lengths x runs]
// Bitpack (modules/coders/bitpack/bitpack_stage.cu:30-124): low nbits of each
// element, LSB-first inside a byte for nbits < 8, little-endian bytes above.
//
// Every element count that is only known on the device (run count, detected
// nbits) is read by the kernels from device memory, so no call needs a host
// round trip.
#include "fzb_kernels.cuh"

namespace fzb {

constexpr int kScanTile = 4096;  // elements per CTA in the scan passes

// ---------------------------------------------------------------------------
// Exclusive scan of u32 values, three passes: tile sums, one-CTA scan of
// the tile sums, tile scan + offset.  The count is given or read from *cptr.
// ---------------------------------------------------------------------------
__device__ __forceinline__ const uint32_t* scan_src(const ScanSrc& a, uint32_t* cnt) {
    *cnt = a.cptr ? min(*a.cptr, a.n) : a.n;
    return a.base;
}

__global__ void __launch_bounds__(256) scan_tile_sums(ScanSrc a, uint32_t* __restrict__ tsum) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    uint32_t cnt;
    const uint32_t* in = scan_src(a, &cnt);
    const uint32_t b = blockIdx.x * kScanTile;
    uint32_t s = 0;
    for (uint32_t i = b + threadIdx.x; i < min(cnt, b + kScanTile); i += 256) s += in[i];
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) s += __shfl_xor_sync(0xffffffffu, s, d);
    __shared__ uint32_t w[8];
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = s;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0;
        for (int i = 0; i < 8; i++) t += w[i];
        tsum[blockIdx.x] = t;
    }
    asm volatile("griddepcontrol.launch_dependents;");
}

// Exclusive scan of the ntiles sums in place, one CTA.  runs (null: all): the run count
// of an RLE stream of at most n runs, whose tiles of kRunTile runs are the ones to scan.
// Eight sums a thread are in flight at a time, and tiles that hold no runs are left out:
// with one load after another over all n / 1024 tiles a run of 33.5 M bytes took 97 us
// to decode.
constexpr uint32_t kRunTile = 1024;

__global__ void __launch_bounds__(1024) scan_tile_offsets(uint32_t* __restrict__ tsum, uint32_t ntiles,
                                                          uint32_t* __restrict__ total,
                                                          const uint32_t* __restrict__ runs, uint32_t n) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ uint32_t s[1024];
    if (runs) ntiles = (min(*runs, n) + kRunTile - 1) / kRunTile;
    const uint32_t t = threadIdx.x, per = ((ntiles + 1023) / 1024 + 3) & ~3u;
    const uint32_t b = min(ntiles, t * per), e = min(ntiles, b + per);
    // sums i .. i + 7 of this thread's, 16 bytes at a time (the scratch is 16-byte
    // aligned and goes on past the last one), zero from e on
    auto load = [&](uint32_t i, uint32_t (&v)[8]) {
#pragma unroll
        for (int q = 0; q < 2; q++) {
            const uint4 w = i + 4 * q < e ? *reinterpret_cast<const uint4*>(tsum + i + 4 * q) : make_uint4(0u, 0u, 0u, 0u);
            v[4 * q] = w.x;
            v[4 * q + 1] = i + 4 * q + 1 < e ? w.y : 0u;
            v[4 * q + 2] = i + 4 * q + 2 < e ? w.z : 0u;
            v[4 * q + 3] = i + 4 * q + 3 < e ? w.w : 0u;
        }
    };
    uint32_t sum = 0;
    for (uint32_t i = b; i < e; i += 8) {
        uint32_t v[8];
        load(i, v);
#pragma unroll
        for (int k = 0; k < 8; k++) sum += v[k];
    }
    s[t] = sum;
    __syncthreads();
    for (int d = 1; d < 1024; d <<= 1) {
        uint32_t v = (t >= (unsigned)d) ? s[t - d] : 0u;
        __syncthreads();
        s[t] += v;
        __syncthreads();
    }
    uint32_t run = s[t] - sum;
    for (uint32_t i = b; i < e; i += 8) {
        uint32_t v[8];
        load(i, v);
#pragma unroll
        for (int k = 0; k < 8; k++) {
            if (i + k < e) tsum[i + k] = run;
            run += v[k];
        }
    }
    if (t == 1023 && total) *total = s[1023];
    asm volatile("griddepcontrol.launch_dependents;");
}

__global__ void __launch_bounds__(256) scan_tile_apply(ScanSrc a, const uint32_t* __restrict__ toff,
                                                       uint32_t* __restrict__ out) {
    asm volatile("griddepcontrol.wait;" ::: "memory");
    __shared__ uint32_t ws[16];
    uint32_t cnt;
    const uint32_t* in = scan_src(a, &cnt);
    const uint32_t b = blockIdx.x * kScanTile + threadIdx.x * 16;
    uint32_t v[16], s = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        v[i] = (b + i < cnt) ? in[b + i] : 0u;
        s += v[i];
    }
    uint32_t tot;
    uint32_t run = toff[blockIdx.x] + block_excl_scan(s, ws, &tot);
#pragma unroll
    for (int i = 0; i < 16; i++) {
        if (b + i < cnt) out[b + i] = run;
        run += v[i];
    }
    asm volatile("griddepcontrol.launch_dependents;");
}

int launch_scan_u32(const ScanSrc& a, uint32_t* out, uint32_t* tile_scratch, uint32_t* total,
                    cudaStream_t s) {
    if (a.n == 0) return 0;
    const uint32_t ntiles = (a.n + kScanTile - 1) / kScanTile;
    // programmatic dependents: each waits for the kernel before it (the
    // first for whatever produced the input) and lets the next one launch
    cudaError_t e = launch_dependent(scan_tile_sums, ntiles, 256, 0, s, a, tile_scratch);
    if (e == cudaSuccess) e = launch_dependent(scan_tile_offsets, 1, 1024, 0, s, tile_scratch, ntiles, total, nullptr, 0u);
    if (e == cudaSuccess) e = launch_dependent(scan_tile_apply, ntiles, 256, 0, s, a, (const uint32_t*)tile_scratch, out);
    return (int)e;
}

// ---------------------------------------------------------------------------
// RLE encode.  Pass 1 counts the runs that start in each 4096-element tile and
// notes the first start; the counts are scanned; pass 2 compacts a tile's runs
// in shared memory and writes their values and lengths in order (the last run
// of a tile ends at the first start of the next tile that has one).
//
// Bound by HBM: the input is read twice (2 B an element, the second time
// mostly from L2) and sizeof(T) + 4 B written a run.  Before, each thread
// wrote its 16 elements' runs one by one, with their starts, and a third
// kernel turned starts into lengths: 6.5 M elements in nearly as many runs took
// 9.6 + 65 + 15 us, now 4 + 17.
// ---------------------------------------------------------------------------

// The tile's elements 16t .. 16t + 15 (t the thread) and their run-start bits.
template <typename T>
__device__ __forceinline__ uint32_t run_starts16(const T* __restrict__ in, uint32_t n, uint32_t b, bool vec,
                                                 T (&v)[16]) {
    constexpr int kQ = 16 * sizeof(T) / 16;  // 16-byte granules a thread
    union {
        uint4 q[kQ];
        T e[16];
    } u;
    if (vec && b + 16 <= n) {
#pragma unroll
        for (int i = 0; i < kQ; i++) u.q[i] = __ldg(reinterpret_cast<const uint4*>(in + b) + i);
    } else {
#pragma unroll
        for (int i = 0; i < 16; i++) u.e[i] = b + i < n ? in[b + i] : T(0);
    }
    T prev = (b > 0 && b <= n) ? __ldg(in + b - 1) : T(0);
    uint32_t m = 0;
#pragma unroll
    for (int i = 0; i < 16; i++) {
        v[i] = u.e[i];
        m |= ((v[i] != prev || b + i == 0) ? 1u : 0u) << i;
        prev = v[i];
    }
    return b + 16 <= n ? m : b < n ? m & ((1u << (n - b)) - 1u) : 0u;
}

template <typename T>
__global__ void __launch_bounds__(256) rle_count_kernel(const T* __restrict__ in, uint32_t n, int vec,
                                                        uint32_t* __restrict__ tcnt, uint32_t* __restrict__ tfirst) {
    __shared__ uint32_t w[8], f[8];
    follow();
    T v[16];
    const uint32_t b = blockIdx.x * kScanTile + threadIdx.x * 16;
    const uint32_t m = run_starts16(in, n, b, vec != 0, v);
    const uint32_t s = __reduce_add_sync(0xffffffffu, __popc(m));
    const uint32_t first = __reduce_min_sync(0xffffffffu, m ? b + __ffs(m) - 1 : 0xffffffffu);
    if ((threadIdx.x & 31) == 0) {
        w[threadIdx.x >> 5] = s;
        f[threadIdx.x >> 5] = first;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t t = 0, g = 0xffffffffu;
        for (int i = 0; i < 8; i++) {
            t += w[i];
            g = min(g, f[i]);
        }
        tcnt[blockIdx.x] = t;
        tfirst[blockIdx.x] = g;
    }
}

template <typename T>
__global__ void __launch_bounds__(256) rle_emit_kernel(const T* __restrict__ in, uint32_t n, int vec,
                                                       const uint32_t* __restrict__ toff,
                                                       const uint32_t* __restrict__ tfirst,
                                                       const uint32_t* __restrict__ total, uint8_t* __restrict__ out,
                                                       unsigned long long* __restrict__ out_size) {
    __shared__ uint32_t ws[16];
    __shared__ uint32_t s_start[kScanTile + 1];
    __shared__ T s_val[kScanTile];
    follow();
    const uint32_t R = *total, t = threadIdx.x;
    const uint32_t vbytes = R * (uint32_t)sizeof(T), valigned = (vbytes + 3u) & ~3u;
    T* values = reinterpret_cast<T*>(out + 4);
    uint32_t* lens = reinterpret_cast<uint32_t*>(out + 4 + valigned);
    if (blockIdx.x == 0 && t == 0) {
        reinterpret_cast<uint32_t*>(out)[0] = R;
        for (uint32_t i = vbytes; i < valigned; i++) out[4 + i] = 0;
        *out_size = 4ull + valigned + 4ull * R;
    }
    const uint32_t r0 = toff[blockIdx.x];
    const uint32_t r1 = blockIdx.x + 1 < gridDim.x ? toff[blockIdx.x + 1] : R;
    if (r0 == r1) return;
    T v[16];
    const uint32_t b = blockIdx.x * kScanTile + t * 16;
    const uint32_t m = run_starts16(in, n, b, vec != 0, v);
    uint32_t tot;
    uint32_t r = block_excl_scan(__popc(m), ws, &tot);
#pragma unroll
    for (int i = 0; i < 16; i++) {
        if ((m >> i) & 1u) {
            s_start[r] = b + i;
            s_val[r] = v[i];
            r++;
        }
    }
    if (t == 0) {  // the first start after the tile: of the first later tile with more runs before its end
        uint32_t next = n;
        if (r1 < R) {
            uint32_t lo = blockIdx.x + 1, hi = gridDim.x - 1;  // tile lo .. hi holds run r1
            if (lo < hi && toff[lo + 1] > r1) hi = lo;         // mostly the next one (3600 x 1800: 15 us, 17 without)
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (toff[mid + 1] > r1) hi = mid;
                else lo = mid + 1;
            }
            next = tfirst[lo];
        }
        s_start[tot] = next;
    }
    __syncthreads();
    for (uint32_t i = t; i < tot; i += 256) {
        values[r0 + i] = s_val[i];
        lens[r0 + i] = s_start[i + 1] - s_start[i];
    }
}

// ---------------------------------------------------------------------------
// RLE decode.  The run lengths are summed per 1024 runs and the sums scanned;
// then each 4096-element output tile finds its first tile of runs, scans the
// lengths of the tiles of runs that overlap it and places their values.
//
// It replaced a scan that wrote every run's offset and a binary search for every
// element: the same stream took 5 + 37 + 50 us, now 5 + 26.
// ---------------------------------------------------------------------------
// Exclusive scan over 256 threads of values up to `top` (below 2^31), the sums
// saturating at it (a malformed stream's lengths may add up past 32 bits).
__device__ __forceinline__ uint32_t block_excl_scan_sat(uint32_t v, uint32_t top, uint32_t* ws, uint32_t* total) {
    const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
    uint32_t inc = v;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t o = __shfl_up_sync(0xffffffffu, inc, d);
        if (lane >= (uint32_t)d) inc = min(inc + o, top);
    }
    uint32_t ex = __shfl_up_sync(0xffffffffu, inc, 1);
    if (lane == 0) ex = 0;
    if (lane == 31) ws[warp] = inc;
    __syncthreads();
    uint32_t base = 0, all = 0;
#pragma unroll
    for (uint32_t w = 0; w < 8; w++) {
        if (w == warp) base = all;
        all = min(all + ws[w], top);
    }
    *total = all;
    return min(base + ex, top);
}

__device__ __forceinline__ uint32_t rle_runs(const uint8_t* in, uint32_t n) {
    return min(*reinterpret_cast<const uint32_t*>(in), n);  // at most n runs in a valid stream
}
__device__ __forceinline__ const uint32_t* rle_lens(const uint8_t* in, uint32_t elem) {
    const uint32_t R = *reinterpret_cast<const uint32_t*>(in);
    return reinterpret_cast<const uint32_t*>(in + 4 + ((R * elem + 3u) & ~3u));
}

// Sum of each tile of runs, a warp a tile.
__global__ void __launch_bounds__(256) rle_sums_kernel(const uint8_t* __restrict__ in, uint32_t n, uint32_t elem,
                                                       uint32_t* __restrict__ tsum, uint32_t ntiles) {
    follow();
    const uint32_t R = rle_runs(in, n), lane = threadIdx.x & 31u;
    const uint32_t* lens = rle_lens(in, elem);
    ntiles = min(ntiles, (R + kRunTile - 1) / kRunTile);
    for (uint32_t tile = blockIdx.x * 8 + (threadIdx.x >> 5); tile < ntiles; tile += gridDim.x * 8) {
        uint32_t s = 0;
        const uint32_t b = tile * kRunTile;
#pragma unroll 8
        for (uint32_t i = b + lane; i < b + kRunTile; i += 32)
            if (i < R) s += lens[i];
        s = __reduce_add_sync(0xffffffffu, s);
        if (lane == 0) tsum[tile] = s;
    }
}

// A tile of outputs: its runs' values and a flag go where the runs start, a max scan
// of the flagged places tells each thread which run covers its 16 outputs' first, and
// the flags the rest, so the work does not depend on the runs' lengths.
//
// Bound by the latency of a tile's steps (search, a barrier a tile of runs, scan).
// Each thread filling its runs output by output, long ones by the whole block, with a
// binary search: 3600 x 1800 33 us (now 26), 4000 x 4000 72 (59), 1000 x 500 9.8 (5.5).
template <typename T>
__global__ void __launch_bounds__(256) rle_expand_kernel(const uint8_t* __restrict__ in,
                                                         const uint32_t* __restrict__ toff,
                                                         const uint32_t* __restrict__ total, uint32_t n,
                                                         T* __restrict__ out, uint32_t* err) {
    static_assert(kScanTile == 16 * 256, "16 outputs a thread");
    __shared__ __align__(16) T s_out[kScanTile];      // a run's value where it starts
    __shared__ uint32_t s_flag[kScanTile / 32], ws[16];
    follow();
    const uint32_t R = rle_runs(in, n), t = threadIdx.x, lane = t & 31u, warp = t >> 5, full = 0xffffffffu;
    const uint32_t* lens = rle_lens(in, sizeof(T));
    const T* values = reinterpret_cast<const T*>(in + 4);
    const uint32_t t0 = blockIdx.x * kScanTile, t1 = min(n, t0 + kScanTile);
    if (blockIdx.x == 0 && t == 0 && (R == 0 || *total != n)) atomicOr(err, kErrMalformed);
    if (t < kScanTile / 32) s_flag[t] = 0u;
    // the last tile of runs starting at or before t0: every warp cuts [lo, hi) to a
    // 32nd at a time (the lane's candidates ascend, lane 0's always qualifies)
    uint32_t lo = 0, hi = (R + kRunTile - 1) / kRunTile;
    while (lo + 1 < hi) {
        const uint32_t step = (hi - lo + 31) / 32, mid = lo + step * lane;
        const uint32_t le = __ballot_sync(full, mid == lo || (mid < hi && toff[mid] <= t0));
        lo += step * (31u - __clz(le));
        hi = min(hi, lo + step);
    }
    uint32_t pos = R ? toff[lo] : t1;  // output position of the tile of runs
    uint32_t nlen[4];                  // the next tile's runs, in flight while this one is placed
    T nval[4];
    auto load = [&](uint32_t r0) {
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t r = r0 + 4 * t + k;
            nlen[k] = r < R ? lens[r] : 0u;
            nval[k] = r < R ? values[r] : T(0);
        }
    };
    load(lo * kRunTile);
    __syncthreads();
    auto start = [&](uint32_t i, T v) {
        s_out[i] = v;
        atomicOr(&s_flag[i >> 5], 1u << (i & 31u));
    };
    uint32_t half = 0;  // the scans' workspace alternates, so that one barrier a tile suffices
    for (uint32_t r0 = lo * kRunTile; r0 < R && pos < t1; r0 += kRunTile, half ^= 8u) {
        uint32_t len[4], sum = 0;
        T val[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            len[k] = min(nlen[k], n);
            val[k] = nval[k];
            sum = min(sum + len[k], n);
        }
        load(r0 + kRunTile);
        uint32_t tot;
        uint32_t e = min(pos + block_excl_scan_sat(sum, n, ws + half, &tot), n);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t a0 = max(e, t0);
            e = min(e + len[k], n);
            if (a0 < min(e, t1)) start(a0 - t0, val[k]);
        }
        pos = min(pos + tot, n);
    }
    if (t == 0 && pos < t1) start(max(pos, t0) - t0, T(0));  // a stream that ends early
    __syncthreads();
    // the last start at or before each of the thread's 16 outputs
    const uint32_t m = (s_flag[t >> 1] >> (16u * (t & 1u))) & 0xffffu;
    uint32_t last = m ? 16u * t + 32u - __clz(m) : 0u;  // place + 1
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) last = max(last, __shfl_up_sync(full, last, d));
    const uint32_t before = __shfl_up_sync(full, last, 1);
    if (lane == 31) ws[warp] = last;
    __syncthreads();
    uint32_t carry = lane ? before : 0u;
    for (uint32_t w = 0; w < warp; w++) carry = max(carry, ws[w]);
    T cur = carry ? s_out[carry - 1] : T(0);
    constexpr int kQuads = (int)sizeof(T);  // 16-byte words of the thread's outputs
    union {
        uint4 q[kQuads];
        T v[16];
    } o;
#pragma unroll
    for (int k = 0; k < kQuads; k++) o.q[k] = reinterpret_cast<const uint4*>(s_out)[kQuads * t + k];
#pragma unroll
    for (int k = 0; k < 16; k++) {
        cur = (m >> k) & 1u ? o.v[k] : cur;
        o.v[k] = cur;
    }
    const uint32_t i0 = t0 + 16u * t;
    if (i0 + 16u <= t1 && (reinterpret_cast<uintptr_t>(out) & 15u) == 0) {
#pragma unroll
        for (int k = 0; k < kQuads; k++) reinterpret_cast<uint4*>(out + i0)[k] = o.q[k];
    } else {
#pragma unroll
        for (int k = 0; k < 16; k++)
            if (i0 + k < t1) out[i0 + k] = o.v[k];
    }
}

template <typename T>
int launch_rle_encode_t(const T* in, uint32_t n, uint8_t* out, unsigned long long* out_size,
                        uint32_t* tcnt, uint32_t* tfirst, uint32_t* runs_total, cudaStream_t s) {
    const uint32_t ntiles = (n + kScanTile - 1) / kScanTile;
    const int vec = (reinterpret_cast<uintptr_t>(in) & 15u) == 0;
    rle_count_kernel<T><<<ntiles, 256, 0, s>>>(in, n, vec, tcnt, tfirst);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_dependent(scan_tile_offsets, 1, 1024, 0, s, tcnt, ntiles, runs_total, nullptr, 0u);
    if (e == cudaSuccess)
        e = launch_dependent(rle_emit_kernel<T>, ntiles, 256, 0, s, in, n, vec, tcnt, tfirst, runs_total, out, out_size);
    return (int)e;
}

int launch_rle_encode(const void* in, uint32_t n, int elem, uint8_t* out, unsigned long long* out_size,
                      uint32_t* tcnt, uint32_t* tfirst, uint32_t* runs_total, cudaStream_t s) {
    if (elem == 1) return launch_rle_encode_t<uint8_t>((const uint8_t*)in, n, out, out_size, tcnt, tfirst, runs_total, s);
    if (elem == 2) return launch_rle_encode_t<uint16_t>((const uint16_t*)in, n, out, out_size, tcnt, tfirst, runs_total, s);
    return launch_rle_encode_t<uint32_t>((const uint32_t*)in, n, out, out_size, tcnt, tfirst, runs_total, s);
}

int launch_rle_decode(const uint8_t* in, uint32_t n, int elem, void* out, uint32_t* tsum, uint32_t* total,
                      uint32_t* err, cudaStream_t s) {
    const uint32_t nrt = (n + kRunTile - 1) / kRunTile;  // tiles of runs, at most n runs
    rle_sums_kernel<<<min((nrt + 7) / 8, 1184u), 256, 0, s>>>(in, n, (uint32_t)elem, tsum, nrt);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_dependent(scan_tile_offsets, 1, 1024, 0, s, tsum, nrt, total,
                                               reinterpret_cast<const uint32_t*>(in), n);
    if (e != cudaSuccess) return (int)e;
    const uint32_t ntiles = (n + kScanTile - 1) / kScanTile;
    auto expand = [&](auto* kernel, auto* o) {
        return (int)launch_dependent(kernel, ntiles, 256, 0, s, in, tsum, total, n, o, err);
    };
    if (elem == 1) return expand(rle_expand_kernel<uint8_t>, (uint8_t*)out);
    if (elem == 2) return expand(rle_expand_kernel<uint16_t>, (uint16_t*)out);
    return expand(rle_expand_kernel<uint32_t>, (uint32_t*)out);
}

// ---------------------------------------------------------------------------
// Bitpack.  nbits may be detected on the device (smallest power of two whose
// range holds the maximum, bitpack_stage.cu:118-124); kernels read it there.
// ---------------------------------------------------------------------------
template <typename T>
__global__ void __launch_bounds__(256) bitpack_max_kernel(const T* __restrict__ in, uint64_t n,
                                                          uint32_t* __restrict__ pmax,
                                                          unsigned int* __restrict__ done,
                                                          uint8_t* __restrict__ nbits_out) {
    uint32_t m = 0;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x)
        m = max(m, (uint32_t)in[i]);
#pragma unroll
    for (int d = 16; d >= 1; d >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, d));
    __shared__ uint32_t w[8];
    __shared__ bool s_last;
    if ((threadIdx.x & 31) == 0) w[threadIdx.x >> 5] = m;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 0; i < 8; i++) m = max(m, w[i]);
        pmax[blockIdx.x] = m;
        __threadfence();
        s_last = atomicAdd(done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!s_last || threadIdx.x != 0) return;
    __threadfence();
    m = 0;
    for (unsigned b = 0; b < gridDim.x; b++) m = max(m, __ldcg(pmax + b));
    const int full = 8 * (int)sizeof(T);
    int nb = full;
    for (int b = 1; b < full; b *= 2)
        if ((uint64_t)m < (1ull << b)) { nb = b; break; }
    *nbits_out = (uint8_t)nb;
    *done = 0;
}

template <typename T>
__global__ void bitpack_encode_kernel(const T* __restrict__ in, uint64_t n,
                                      const uint8_t* __restrict__ nbits_ptr, uint8_t* __restrict__ out,
                                      unsigned long long* __restrict__ out_size) {
    const int nbits = *nbits_ptr;
    const uint64_t nout = (n * (uint64_t)nbits + 7) / 8;
    const uint64_t tid = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    if (tid == 0 && out_size) *out_size = nout;
    if (nbits < 8) {
        const int per = 8 / nbits;
        const uint32_t mask = (1u << nbits) - 1u;
        for (uint64_t b = tid; b < nout; b += stride) {
            uint32_t packed = 0;
            for (int k = 0; k < per; k++) {
                const uint64_t e = b * per + k;
                if (e < n) packed |= ((uint32_t)in[e] & mask) << (k * nbits);
            }
            out[b] = (uint8_t)packed;
        }
    } else {
        const int bytes = nbits / 8;
        for (uint64_t i = tid; i < n; i += stride) {
            uint32_t v = (uint32_t)in[i];
            if (nbits < 32) v &= (1u << nbits) - 1u;
            for (int b = 0; b < bytes; b++) out[i * bytes + b] = (uint8_t)(v >> (8 * b));
        }
    }
}

template <typename T>
__global__ void bitpack_decode_kernel(const uint8_t* __restrict__ in, uint64_t n, int nbits,
                                      T* __restrict__ out) {
    const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
    for (uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        uint32_t v = 0;
        if (nbits < 8) {
            const int per = 8 / nbits;
            v = (in[i / per] >> ((i % per) * nbits)) & ((1u << nbits) - 1u);
        } else {
            for (int b = 0; b < nbits / 8; b++) v |= (uint32_t)in[i * (nbits / 8) + b] << (8 * b);
        }
        out[i] = (T)v;
    }
}

__global__ void set_byte_kernel(uint8_t* p, uint8_t v) { *p = v; }

int launch_bitpack_encode(const void* in, uint64_t n, int elem, int nbits, uint8_t* nbits_dev,
                          uint8_t* out, unsigned long long* out_size, uint32_t* pmax,
                          unsigned int* done, cudaStream_t s) {
    const unsigned grid = 1184;
    if (nbits == 0) {
        if (elem == 1) bitpack_max_kernel<uint8_t><<<grid, 256, 0, s>>>((const uint8_t*)in, n, pmax, done, nbits_dev);
        else if (elem == 2) bitpack_max_kernel<uint16_t><<<grid, 256, 0, s>>>((const uint16_t*)in, n, pmax, done, nbits_dev);
        else bitpack_max_kernel<uint32_t><<<grid, 256, 0, s>>>((const uint32_t*)in, n, pmax, done, nbits_dev);
    } else {
        set_byte_kernel<<<1, 1, 0, s>>>(nbits_dev, (uint8_t)nbits);
    }
    if (elem == 1) bitpack_encode_kernel<uint8_t><<<grid, 256, 0, s>>>((const uint8_t*)in, n, nbits_dev, out, out_size);
    else if (elem == 2) bitpack_encode_kernel<uint16_t><<<grid, 256, 0, s>>>((const uint16_t*)in, n, nbits_dev, out, out_size);
    else bitpack_encode_kernel<uint32_t><<<grid, 256, 0, s>>>((const uint32_t*)in, n, nbits_dev, out, out_size);
    return (int)cudaGetLastError();
}

int launch_bitpack_decode(const uint8_t* in, uint64_t n, int elem, int nbits, void* out, cudaStream_t s) {
    const unsigned grid = 1184;
    if (elem == 1) bitpack_decode_kernel<uint8_t><<<grid, 256, 0, s>>>(in, n, nbits, (uint8_t*)out);
    else if (elem == 2) bitpack_decode_kernel<uint16_t><<<grid, 256, 0, s>>>(in, n, nbits, (uint16_t*)out);
    else bitpack_decode_kernel<uint32_t><<<grid, 256, 0, s>>>(in, n, nbits, (uint32_t*)out);
    return (int)cudaGetLastError();
}

}  // namespace fzb
