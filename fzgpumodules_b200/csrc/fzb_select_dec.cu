// fzb_select_dec.cu -- decoding a selector container: one kernel finds every
// chunk's payload, then every chunk is decoded at once, a CTA per 16 KiB block
// of a Bitshuffle+RZE or Bitpack chunk, one per RLE chunk, and one of 512
// threads per Huffman chunk (fzb_huffman.cu).
//
// The chunks are independent, so the whole container is a few waves of CTAs;
// decoded one after another from the host (five launches and two host waits a
// chunk) 2048 chunks took 77 ms, all but about 0.1 ms of it waiting.  Each coder's bytes
// mean what its stage's decoder makes of them (rze_stage.cu:846-994,
// rle.cu:196-259, bitpack_stage.cu:30-124, hf_kernels.cu:258-312).
#include "fzb_rzedec.cuh"

namespace fzb {
namespace {

constexpr uint32_t kRleTile = 1024;  // runs expanded at a time

// Checks the container's header and scans the chunk sizes (each padded to 4
// bytes) into payload offsets, one CTA.
__global__ void __launch_bounds__(1024) sel_offsets_kernel(SelDec a) {
    __shared__ uint32_t ws[66];
    const uint32_t* h = reinterpret_cast<const uint32_t*>(a.in);
    const uint32_t t = threadIdx.x;
    if (h[0] != 0x43535A46u || h[1] != a.nch || h[2] != (uint32_t)a.n || h[3] != (uint32_t)kSelCodes) return;
    const uint64_t in_words = a.in_bytes / 4;
    uint64_t base = (16 + 2 * (uint64_t)((a.nch + 3u) & ~3u) + 4 * (uint64_t)a.nch) / 4;
    for (uint32_t c0 = 0; c0 < a.nch; c0 += 1024u) {
        const uint32_t c = c0 + t;
        const uint32_t sz = c < a.nch ? sel_size(a, c) : 0u;
        // words by low and high halves, so that the sums of 1024 of any size fit
        const uint32_t words = (uint32_t)(((uint64_t)sz + 3) / 4);
        uint32_t e0, e1, t0, t1;
        block_scan2_1024(words & 0xffffu, words >> 16, e0, e1, t0, t1, ws);
        if (c < a.nch) {
            const uint64_t o = base + e0 + ((uint64_t)e1 << 16);
            a.offs[c] = (uint32_t)min(min(o, in_words), (uint64_t)0xffffffffu);
            // (a payload that starts past 2^32 words is refused with those past the input)
            if (4 * o + sz > a.in_bytes || o > 0xffffffffu || sel_tag(a, c) > 3u) sel_fail(a, c, kSelMalformed);
        }
        base = min(base + t0 + ((uint64_t)t1 << 16), in_words);
    }
    if (t == 0) *a.state = 1u;
}

// One block of the chunk's RZE stream [u32 bytes][u32 blocks][u32 size each]
// [payloads], then the bitshuffle inverse of a full block.
__device__ __forceinline__ void decode_rze(const SelDec& a, uint32_t c, uint64_t off, uint32_t sz, uint32_t cnt,
                                           RzeDecSmem& sm) {
    const uint32_t j = blockIdx.x & 3u, t = threadIdx.x;
    const uint32_t bytes = 2 * cnt, nsub = (bytes + kChunkBytes - 1) / kChunkBytes;
    const uint32_t* h = reinterpret_cast<const uint32_t*>(a.in + off);
    if (sz < 8 + 4 * nsub || h[0] != bytes || h[1] != nsub) {
        if (t == 0 && j == 0) sel_fail(a, c, kSelMalformed);
        return;
    }
    if (j >= nsub) return;
    uint64_t o = 8 + 4 * nsub, end = o;
    for (uint32_t k = 0; k < nsub; k++) {
        const uint32_t b = h[2 + k] & 0x7fffffffu;
        if (k < j) o += b;
        end += b;
    }
    if (end > sz && t == 0 && j == 0) sel_fail(a, c, kSelMalformed);
    __shared__ uint32_t s_err;
    if (t == 0) s_err = 0;
    rze_decode_init(sm);
    __syncthreads();
    const int osz = (int)min((uint32_t)kChunkBytes, bytes - j * kChunkBytes);
    uint32_t x[16];
    rze_decode_words(a.in, off + sz, off + o, h[2 + j], osz, sm, &s_err, x);
    uint16_t* dst = a.out + (size_t)c * kSelCodes + (size_t)j * kChunkCodes;
    if (osz == kChunkBytes) {
        uint32_t w[16];
        codes_from_planes(x, w);
        if ((reinterpret_cast<uintptr_t>(dst) & 15u) == 0) {
            uint4* d4 = reinterpret_cast<uint4*>(dst + 32 * t);
#pragma unroll
            for (int v = 0; v < 4; v++) d4[v] = make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
        } else {
#pragma unroll
            for (int l = 0; l < 16; l++) {
                dst[32 * t + 2 * l] = (uint16_t)w[l];
                dst[32 * t + 2 * l + 1] = (uint16_t)(w[l] >> 16);
            }
        }
    } else {  // a block shorter than 16 KiB is stored unshuffled
#pragma unroll
        for (int b = 0; b < 16; b++) {
            const uint32_t e = 2 * ((15 - b) * 256 + t);
            if (2 * e + 2 <= (uint32_t)osz) dst[e] = (uint16_t)x[b];
            if (2 * e + 4 <= (uint32_t)osz) dst[e + 1] = (uint16_t)(x[b] >> 16);
        }
    }
    __syncthreads();
    if (t == 0 && s_err) sel_fail(a, c, kSelMalformed);
}

// [u32 runs][u16 values, padded to 4 bytes][u32 lengths]: tiles of runs are
// scanned into output ranges; a thread finds the run of its first code by a
// binary search and walks on.
__device__ __forceinline__ void decode_rle(const SelDec& a, uint32_t c, uint64_t off, uint32_t cnt, uint32_t* s_off,
                                           uint16_t* s_val, uint32_t* ws) {
    const uint32_t t = threadIdx.x;
    uint16_t* out = a.out + (size_t)c * kSelCodes;
    const uint32_t runs = off + 4 <= a.in_bytes ? *reinterpret_cast<const uint32_t*>(a.in + off) : 0u;
    const uint32_t R = min(runs, cnt);
    const uint64_t vbytes = ((uint64_t)runs * 2 + 3) & ~3ull;
    if (R == 0 || off + 4 + vbytes + 4ull * R > a.in_bytes) {
        if (t == 0) sel_fail(a, c, kSelMalformed);
        return;
    }
    const uint16_t* vals = reinterpret_cast<const uint16_t*>(a.in + off + 4);
    const uint32_t* lens = reinterpret_cast<const uint32_t*>(a.in + off + 4 + vbytes);
    uint32_t pos = 0;  // codes before the tile of runs
    for (uint32_t r0 = 0; r0 < R; r0 += kRleTile) {
        const uint32_t nr = min(kRleTile, R - r0);
        uint32_t l[4], sum = 0;
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t r = 4 * t + k;
            l[k] = r < nr ? min(lens[r0 + r], cnt + 1) : 0u;  // sums below 2^26
            sum += l[k];
        }
        uint32_t total;
        uint32_t e = pos + block_excl_scan(sum, ws, &total);
#pragma unroll
        for (int k = 0; k < 4; k++) {
            const uint32_t r = 4 * t + k;
            s_off[r] = e;
            if (r < nr) s_val[r] = vals[r0 + r];
            e += l[k];
        }
        if (t == kThreads - 1) s_off[kRleTile] = e;
        __syncthreads();
        const uint32_t end = min(pos + total, cnt);
        for (uint32_t i = pos + 8 * t; i < end; i += 8 * kThreads) {
            uint32_t lo = 0, hi = nr;  // the last run starting at or before i
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (s_off[mid] <= i) lo = mid;
                else hi = mid;
            }
            for (uint32_t k = i; k < min(i + 8, end); k++) {
                while (lo + 1 < nr && s_off[lo + 1] <= k) lo++;
                out[k] = s_val[lo];
            }
        }
        pos = min(pos + total, 1u << 30);
        __syncthreads();
    }
    if (t == 0 && pos != cnt) sel_fail(a, c, kSelMalformed);
}

// Quarter blockIdx.x % 4 of a Bitpack chunk (LSB-first below 8 bits).
__device__ __forceinline__ void decode_bitpack(const SelDec& a, uint32_t c, uint64_t off, uint32_t cnt) {
    const uint32_t nbits = sel_param(a, c), t = threadIdx.x;
    if (nbits == 0 || nbits > 16 || (nbits & (nbits - 1)) != 0) {
        if (t == 0 && (blockIdx.x & 3u) == 0) sel_fail(a, c, kSelInvalid);
        return;
    }
    if (off + ((uint64_t)cnt * nbits + 7) / 8 > a.in_bytes) {
        if (t == 0 && (blockIdx.x & 3u) == 0) sel_fail(a, c, kSelMalformed);
        return;
    }
    const uint8_t* in = a.in + off;
    uint16_t* out = a.out + (size_t)c * kSelCodes;
    const uint32_t j = blockIdx.x & 3u, end = min(cnt, (j + 1) * (uint32_t)kChunkCodes);
    for (uint32_t i = j * (uint32_t)kChunkCodes + t; i < end; i += kThreads) {
        uint32_t v;
        if (nbits < 8) {
            const uint32_t bit = i * nbits;
            v = (in[bit >> 3] >> (bit & 7u)) & ((1u << nbits) - 1u);
        } else {
            v = nbits == 8 ? in[i] : ((uint32_t)in[2 * i] | (uint32_t)in[2 * i + 1] << 8);
        }
        out[i] = (uint16_t)v;
    }
}

// Four CTAs a chunk: everything but the Huffman chunks.  Six CTAs an SM (134 MB of
// codes: 100 us, 106 with four).  Launched as a dependent of the Huffman decoder,
// beside whose last CTAs it runs: the offsets that both read were complete when the
// first of them began.  Only the last block awaits that kernel, so that what follows
// comes after both.
__global__ void __launch_bounds__(kThreads, 6) sel_decode_kernel(SelDec a) {
    __shared__ RzeDecSmem sm;
    __shared__ uint32_t s_ws[16];
    if (blockIdx.x == gridDim.x - 1) asm volatile("griddepcontrol.wait;" ::: "memory");
    if (*a.state == 0u) return;
    const uint32_t c = blockIdx.x >> 2, tag = sel_tag(a, c), sz = sel_size(a, c);
    const uint64_t off = 4ull * a.offs[c];
    if (off + sz > a.in_bytes) return;  // reported by the offsets kernel
    const uint32_t cnt = (uint32_t)min((uint64_t)kSelCodes, a.n - (uint64_t)c * kSelCodes);
    if (tag == 0) {
        decode_rze(a, c, off, sz, cnt, sm);
    } else if (tag == 1) {
        // the RZE decoder's staging buffer holds a tile of runs
        if ((blockIdx.x & 3u) == 0)
            decode_rle(a, c, off, cnt, sm.C, reinterpret_cast<uint16_t*>(sm.C + kRleTile + 1), s_ws);
    } else if (tag == 2) {
        decode_bitpack(a, c, off, cnt);
    }
}

}  // namespace

int launch_sel_decode(const SelDec& a, cudaStream_t s) {
    sel_offsets_kernel<<<1, 1024, 0, s>>>(a);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = launch_sel_hf_decode(a, s);
    if (e == cudaSuccess) e = launch_dependent(sel_decode_kernel, 4 * a.nch, kThreads, 0, s, a);
    return (int)e;
}

}  // namespace fzb
