// fzb_rze.cuh -- block-level RZE chunk encoder (256 threads; the decoder is in
// fzb_rzedec.cuh).
//
// Format of one chunk (modules/coders/rze/rze_stage.cu:324-445):
//   [nonzero bytes][non-repeated bm1 bytes][non-repeated bm2 bytes]
//   [non-repeated bm3 bytes][bm4, 4 bytes][u16 input size]
// bmL+1 marks the bytes of bmL that differ from their predecessor (byte 0
// compared with 0); bm1 marks nonzero input bytes.  An all-zero chunk is the
// 2-byte size tag alone; a chunk that overflows any level is stored raw and
// its header size word carries bit 31.
//
// Work split: thread t owns input bytes [64t, 64t+64) (bm1 bytes 8t..8t+7 =
// bm2 byte t); levels 3 and 4 run in warp 0.
#pragma once

#include "fzb_common.cuh"

namespace fzb {

// Compaction selectors of a 4-bit mask: __byte_perm(w, 0, kRzeSel[m]) moves the
// bytes of w flagged in m to the low end, in order, zero-filled.
__constant__ static uint32_t kRzeSel[16] = {0x4444, 0x4440, 0x4441, 0x4410, 0x4442, 0x4420, 0x4421, 0x4210,
                                            0x4443, 0x4430, 0x4431, 0x4310, 0x4432, 0x4320, 0x4321, 0x3210};

// Compaction selectors of a word pair's 8-bit mask: __byte_perm(w0, w1, x) and
// (w0, w1, y) give the pair's flagged bytes in order, then copies of an
// unflagged byte (a zero byte, where the mask flags the nonzero ones).
struct RzePairSel {
    uint2 v[256];
};
constexpr RzePairSel rze_pair_sel() {
    RzePairSel t{};
    for (uint32_t m = 0; m < 256; m++) {
        uint32_t sel = 0, k = 0, zb = 0;
        for (uint32_t b = 8; b-- > 0;)
            if (!((m >> b) & 1u)) zb = b;
        for (uint32_t b = 0; b < 8; b++)
            if ((m >> b) & 1u) sel |= b << (4 * k++);
        for (; k < 8; k++) sel |= zb << (4 * k);
        t.v[m].x = sel & 0xffffu;
        t.v[m].y = sel >> 16;
    }
    return t;
}
__device__ static const RzePairSel kRzePairSel = rze_pair_sel();

constexpr int kRzeEncSmem = 2 * kChunkBytes + 16 + 256 + 2048;  // bytes of the encoder's shared memory

// Shared memory of one encoder, carved from kRzeEncSmem bytes.
struct RzeSmem {
    uint32_t* S;    // 4096 words: chunk bytes (zero past in_size), 16-byte granules swizzled (rze_granule)
    uint8_t* O;     // kChunkBytes + 16 bytes: encoded chunk
    uint8_t* bm2;   // 256 bytes
    uint2* sel8;    // 256: kRzePairSel
    uint32_t* ws;   // 16 words scan workspace
};
__device__ __forceinline__ RzeSmem rze_smem(void* base, uint32_t* ws) {
    uint8_t* p = static_cast<uint8_t*>(base);
    RzeSmem sm;
    sm.S = reinterpret_cast<uint32_t*>(p);
    sm.O = p + kChunkBytes;
    sm.bm2 = p + 2 * kChunkBytes + 16;
    sm.sel8 = reinterpret_cast<uint2*>(p + 2 * kChunkBytes + 16 + 256);
    sm.ws = ws;
    return sm;
}

// Place of granule g in S: eight threads' reads of their own four granules each
// (stride 64 bytes) then fall on all banks.
__device__ __forceinline__ uint32_t rze_granule(uint32_t g) { return g ^ ((g >> 3) & 7u); }

// Fills S from the thread's plane words x[b] = word (15 - b) * 256 + t.
__device__ __forceinline__ void rze_put_planes(const RzeSmem& sm, const uint32_t (&x)[16]) {
    const uint32_t t = threadIdx.x, at = 4u * rze_granule(t >> 2) + (t & 3u);  // 256 words: whole swizzle groups
#pragma unroll
    for (int b = 0; b < 16; b++) sm.S[(15 - b) * 256 + at] = x[b];
}

// Fills S from the thread's words 16t .. 16t + 15 in order.
__device__ __forceinline__ void rze_put_words(const RzeSmem& sm, const uint32_t (&w)[16]) {
#pragma unroll
    for (int v = 0; v < 4; v++)
        reinterpret_cast<uint4*>(sm.S)[rze_granule(4 * threadIdx.x + v)] =
            make_uint4(w[4 * v], w[4 * v + 1], w[4 * v + 2], w[4 * v + 3]);
}

// Granule i of the encoded chunk whose size word is sw.
__device__ __forceinline__ uint4 rze_payload(const RzeSmem& sm, uint32_t sw, uint32_t i) {
    return (sw >> 31) ? reinterpret_cast<const uint4*>(sm.S)[rze_granule(i)] : reinterpret_cast<const uint4*>(sm.O)[i];
}

// ORs the low bytes of `packed` into the zeroed byte stream at byte offset pos.
__device__ __forceinline__ void rze_or_bytes(uint32_t* Ow, uint32_t pos, uint32_t packed) {
    const uint32_t sh = (pos & 3u) * 8u;
    atomicOr(&Ow[pos >> 2], packed << sh);
    atomicOr(&Ow[(pos >> 2) + 1], __funnelshift_l(packed, 0u, sh));
}

// Encodes the chunk held in sm.S (in_size bytes, rest zero).  Returns the
// header size word (bit 31 = stored raw; then the payload is S itself).
// Uniform across the block; ends with a barrier.
//
// Thread t takes S words 16t..16t+15 (bytes 64t..64t+63): their nonzero-byte
// nibbles are bm1 bytes 8t..8t+7, so levels 1 and 2 need one packed warp scan
// of both byte counts and one barrier for the per-warp totals.  Nonzero bytes
// are compacted per word pair by two byte permutes and OR-ed into the zeroed
// output with three shared atomics (an output word can straddle two threads);
// warp 0 codes levels 3 and 4 beside that, its bytes ORed in as well.  Same
// bytes and raw decisions as rze_stage.cu:324-445.
//
// Bound by instruction issue on dense chunks and by the barriers and the serial
// level code on sparse ones.  Per word instead of per pair, with unswizzled
// reads (four-way bank conflicts) and levels 3 and 4 behind a barrier of their
// own the chunks of 500 x 500 x 100 took 62.6 us (now 56.4), those of 3600 x 1800
// 11.9 (9.8), the selector's blocks of 134 MB of codes 87 (71).
__device__ static uint32_t rze_encode_chunk(const RzeSmem& sm, int in_size) {
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5;
    const uint32_t full = 0xffffffffu;
    const uint32_t raw_word = 0x80000000u | (uint32_t)in_size;
    const int b1 = (in_size + 7) >> 3, b2 = (b1 + 7) >> 3, b3 = (b2 + 7) >> 3;
    uint32_t* Ow = reinterpret_cast<uint32_t*>(sm.O);
    // output zeroed for the atomics: payloads stay below kRzeAvail, so the last
    // word of an atomic stays below kChunkBytes + 16
    for (uint32_t i = t; i < (kChunkBytes + 16) / 16; i += kThreads)
        reinterpret_cast<uint4*>(sm.O)[i] = make_uint4(0u, 0u, 0u, 0u);
    sm.sel8[t] = __ldg(&kRzePairSel.v[t]);
    uint32_t w[16];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint4 q = reinterpret_cast<const uint4*>(sm.S)[rze_granule(4 * t + i)];
        w[4 * i] = q.x;
        w[4 * i + 1] = q.y;
        w[4 * i + 2] = q.z;
        w[4 * i + 3] = q.w;
    }
    uint32_t nlo = 0, nhi = 0;
    {
        uint32_t o = 0;
#pragma unroll
        for (int i = 0; i < 16; i++) o |= w[i];
        if (__any_sync(full, o != 0u)) {
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const uint32_t hb = (((w[i] & 0x7f7f7f7fu) + 0x7f7f7f7fu) | w[i]) & 0x80808080u;
                const uint32_t nb = ((hb * 0x00204081u) >> (28 - 4 * (i & 7))) & (15u << (4 * (i & 7)));
                if (i < 8) nlo |= nb;
                else nhi |= nb;
            }
        }
    }
    // level 2: the bm1 bytes (< b1) that differ from their predecessor
    uint32_t prev = __shfl_up_sync(full, nhi, 1) >> 24;
    if (lane == 0) {
        prev = 0u;
        if (t) {  // words 16t - 2 and 16t - 1
            const uint2 p = *reinterpret_cast<const uint2*>(sm.S + 4 * rze_granule(4 * t - 1) + 2);
            prev = nz_nibble(p.x) | (nz_nibble(p.y) << 4);
        }
    }
    const uint64_t M = ((uint64_t)nhi << 32) | nlo;
    uint32_t m2 = nz_byte_mask64(M ^ ((M << 8) | prev));
    {
        const int valid = b1 - 8 * (int)t;
        m2 &= (valid >= 8) ? 0xffu : (valid <= 0 ? 0u : ((1u << valid) - 1u));
    }
    const uint32_t v12 = (uint32_t)(__popc(nlo) + __popc(nhi)) | ((uint32_t)__popc(m2) << 16);
    const uint32_t inc12 = warp_incl_scan(v12);
    if (lane == 31) sm.ws[warp] = inc12;
    sm.bm2[t] = (uint8_t)m2;
    __syncthreads();
    uint32_t tot12 = 0, pre12 = inc12 - v12;
#pragma unroll
    for (uint32_t w8 = 0; w8 < kThreads / 32; w8++) {
        const uint32_t v = sm.ws[w8];
        tot12 += v;
        if (w8 < warp) pre12 += v;
    }
    const uint32_t nzT = tot12 & 0xffffu, n2T = tot12 >> 16;
    if (nzT == 0) {  // all-zero chunk: the 2-byte size tag alone
        if (t == 0) {
            sm.O[0] = (uint8_t)(in_size & 0xff);
            sm.O[1] = (uint8_t)((in_size >> 8) & 0xff);
        }
        __syncthreads();
        return 2u;
    }
    const uint32_t wpos = nzT + n2T;
    if ((int)nzT >= kRzeAvail || (int)nzT > kRzeAvail - b1 || (int)wpos >= kRzeAvail ||
        (int)wpos > kRzeAvail - b2) {
        __syncthreads();
        return raw_word;
    }
    {   // level-1 payload: nonzero bytes in byte order; level-2: non-repeated bm1 bytes
        uint32_t pos = pre12 & 0xffffu;
#pragma unroll
        for (int i = 0; i < 8; i++) {
            const uint32_t m8 = ((i < 4 ? nlo : nhi) >> (8 * (i & 3))) & 0xffu;
            if (m8) {
                const uint2 sel = sm.sel8[m8];
                const uint32_t lo = __byte_perm(w[2 * i], w[2 * i + 1], sel.x);
                const uint32_t hi = __byte_perm(w[2 * i], w[2 * i + 1], sel.y);
                const uint32_t sh = (pos & 3u) * 8u;
                uint32_t* dst = Ow + (pos >> 2);
                atomicOr(dst, lo << sh);
                atomicOr(dst + 1, __funnelshift_l(lo, hi, sh));
                atomicOr(dst + 2, __funnelshift_l(hi, 0u, sh));
            }
            pos += __popc(m8);
        }
        const uint32_t q = nzT + (pre12 >> 16);
        if (m2 & 15u) rze_or_bytes(Ow, q, __byte_perm(nlo, 0u, kRzeSel[m2 & 15u]));
        if (m2 >> 4) rze_or_bytes(Ow, q + __popc(m2 & 15u), __byte_perm(nhi, 0u, kRzeSel[m2 >> 4]));
    }
    // levels 3 and 4, trailer (warp 0): bm2 and the payload end are known since
    // the barrier
    if (warp == 0) {
        const uint2 mw = reinterpret_cast<const uint2*>(sm.bm2)[lane];
        const uint64_t M3 = ((uint64_t)mw.y << 32) | mw.x;
        uint32_t p3 = __shfl_up_sync(full, mw.y, 1) >> 24;
        if (lane == 0) p3 = 0;
        uint32_t m3 = nz_byte_mask64(M3 ^ ((M3 << 8) | p3));  // bm3 byte `lane`
        {
            const int valid = b2 - 8 * (int)lane;
            m3 &= (valid >= 8) ? 0xffu : (valid <= 0 ? 0u : ((1u << valid) - 1u));
        }
        const uint32_t n3 = __popc(m3), inc = warp_incl_scan(n3);
        const uint32_t n3T = __shfl_sync(full, inc, 31);
        {
            uint32_t p = wpos + inc - n3, m = m3;
            while (m) {
                const uint32_t b = __ffs(m) - 1;
                m &= m - 1;
                atomicOr(&Ow[p >> 2], (uint32_t)(uint8_t)(M3 >> (8 * b)) << (8 * (p & 3u)));
                p++;
            }
        }
        uint32_t pb = __shfl_up_sync(full, m3, 1);
        if (lane == 0) pb = 0;
        const bool nr4 = ((int)lane < b3) && (m3 != pb);
        const uint32_t bm4 = __ballot_sync(full, nr4);
        uint32_t wp = wpos + n3T;
        uint32_t sw = raw_word;
        if (!((int)wp >= kRzeAvail || (int)wp >= kRzeAvail - 4 || (int)wp > (kRzeAvail - 4) - b3)) {
            if (nr4) {
                const uint32_t q = wp + __popc(bm4 & ((1u << lane) - 1u));
                atomicOr(&Ow[q >> 2], (m3 & 0xffu) << (8 * (q & 3u)));
            }
            wp += __popc(bm4);
            if ((int)wp < kRzeAvail - 4) {
                if (lane == 0) {  // bm4 and the original size, six bytes
                    const uint32_t sh = 8 * (wp & 3u), hi = (uint32_t)in_size & 0xffffu;
                    atomicOr(&Ow[wp >> 2], bm4 << sh);
                    atomicOr(&Ow[(wp >> 2) + 1], __funnelshift_l(bm4, hi, sh));
                    atomicOr(&Ow[(wp >> 2) + 2], __funnelshift_l(hi, 0u, sh));
                }
                sw = wp + 6;
            }
        }
        if (lane == 0) sm.ws[12] = sw;
    }
    __syncthreads();
    return sm.ws[12];
}

}  // namespace fzb
