// fzb_rzedec.cuh -- block-level RZE chunk decoder (256 threads), and the staging of
// a chunk and the pairing of codes, which it shares with the inverse slab kernel
// (fzb_slab_inv.cu; that kernel decodes the levels in its own pipeline).
//
// Format of a chunk: fzb_rze.cuh (modules/coders/rze/rze_stage.cu:324-445;
// decoding :871-994).  The decoder hands thread t the sixteen words
// {(15 - b) * 256 + t : b = 0..15} of the chunk in registers: for a
// bitshuffled chunk of 2-byte codes these are the plane words of codes
// 32t..32t+31, ready for the bit transpose, so the decoded bytes never pass
// through shared memory.
#pragma once

#include "fzb_slab.cuh"

namespace fzb {
namespace {

constexpr int kCBytes = kChunkBytes + 64;  // one staged chunk (+ lead bytes and a slack word)

// Expansion selectors: __byte_perm(v, 0, kExpandInit[m]) moves the low
// popc(m) bytes of v to the byte positions flagged in the 4-bit mask m.
__constant__ uint32_t kExpandInit[16] = {
    0x4444, 0x4440, 0x4404, 0x4410, 0x4044, 0x4140, 0x4104, 0x4210,
    0x0444, 0x1440, 0x1404, 0x2410, 0x1044, 0x2140, 0x2104, 0x3210};

__device__ __forceinline__ void cp_async4(uint32_t* dst, const uint32_t* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async16s(uint32_t* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_u32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_group 0;" ::: "memory"); }

// Stages a chunk's payload (`e`: its header word, `off`: its offset in the
// stream of `rze_bytes` bytes at `rze`) from the 16-byte boundary at or below
// its first byte when the stream is 16-byte aligned, else the 4-byte one, into
// Cw.  Returns the first byte's offset from that boundary in lead, and ok =
// the payload lies inside the stream.
__device__ __forceinline__ void stage_payload(const uint8_t* rze, uint64_t rze_bytes, uint64_t off, uint32_t e,
                                              uint32_t* Cw, uint32_t& lead, bool& ok) {
    const uint32_t comp = e & 0x7fffffffu;
    ok = off + comp <= rze_bytes;
    const uint8_t* src = rze + (ok ? off : 0);
    const uint32_t ncopy = ok ? min(comp, (uint32_t)kChunkBytes) : 0u;
    const uint8_t* end = rze + rze_bytes;
    if ((reinterpret_cast<uintptr_t>(rze) & 15u) == 0) {
        // a 16-byte aligned stream: 16-byte copies from the 16-byte boundary
        // at or below the first byte (never below the stream's start)
        lead = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 15u);
        const uint32_t ng = (lead + ncopy + 15) >> 4;
        const uint8_t* g0 = src - lead;
        for (uint32_t i = threadIdx.x; i < ng; i += kThreads) {
            const uint8_t* p = g0 + 16u * i;
            if (p + 16 <= end) {
                cp_async16s(Cw + 4u * i, p);
            } else {  // the stream's last bytes: only those inside it
#pragma unroll
                for (int w = 0; w < 4; w++) {
                    uint32_t v = 0;
                    for (int b = 0; b < 4; b++)
                        if (p + 4 * w + b < end) v |= (uint32_t)p[4 * w + b] << (8 * b);
                    Cw[4u * i + w] = v;
                }
            }
        }
        cp_async_commit();
        return;
    }
    lead = (uint32_t)(reinterpret_cast<uintptr_t>(src) & 3u);
    const uint32_t nw = (lead + ncopy + 3) >> 2;
    const uint32_t* gw = reinterpret_cast<const uint32_t*>(src - lead);
    for (uint32_t i = threadIdx.x; i < nw; i += kThreads) {
        const uint8_t* p = reinterpret_cast<const uint8_t*>(gw + i);
        if (p + 4 <= end) {
            cp_async4(Cw + i, gw + i);
        } else {  // last word of the stream: only the bytes inside it
            uint32_t v = 0;
            for (int b = 0; b < 4; b++)
                if (p + b < end) v |= (uint32_t)p[b] << (8 * b);
            Cw[i] = v;
        }
    }
    cp_async_commit();
}

// 4 bytes of the staged chunk starting at payload byte q (lead included).
__device__ __forceinline__ uint32_t staged_word(const uint32_t* Cw, uint32_t q) {
    return __funnelshift_r(Cw[q >> 2], Cw[(q >> 2) + 1], 8u * (q & 3u));
}

__device__ __forceinline__ uint32_t staged_byte(const uint32_t* Cw, uint32_t q) {
    return (Cw[q >> 2] >> (8u * (q & 3u))) & 0xffu;
}

// Packed code pair -> two biased 16-bit values u = s + 32768 (s the signed
// delta): zigzag inverse (zigzag.h:80-84) or plain int16.
template <bool ZZ>
__device__ __forceinline__ uint32_t biased_pair(uint32_t x) {
    if (ZZ) {
        const uint32_t nb = 0x80008000u - (x & 0x00010001u);  // per half: bit0 ? 0x7fff : 0x8000
        return ((x >> 1) & 0x7fff7fffu) ^ nb;
    }
    return x ^ 0x80008000u;
}

// Shared memory of one decoder (about 20 KB: four to six CTAs an SM).
struct __align__(16) RzeDecSmem {
    uint32_t C[kCBytes / 4];
    uint32_t bm1[512];
    uint8_t bm2[256];
    uint32_t pfx2[256];     // bm2 bits before each bm2 byte
    uint32_t tot[8][4];     // per warp: inclusive plane counts, 8-bit fields
    uint32_t base[8][16];   // per warp, per plane: level-1 byte offset
    uint32_t exp[16];       // expansion selectors
    uint32_t misc[2];       // level-1 size, malformed flag
};

// Once per CTA, before the first rze_decode_words.
__device__ __forceinline__ void rze_decode_init(RzeDecSmem& sm) {
    if (threadIdx.x < 16) sm.exp[threadIdx.x] = kExpandInit[threadIdx.x];
}

// Decodes one chunk (header word `e`, payload at `off`, `osz` original bytes)
// into x[b] = word (15 - b) * 256 + t of the chunk (bytes past osz zero).
// Sets kErrMalformed on an inconsistent chunk (and leaves zeros).  All 256
// threads call it; a caller that decodes several chunks puts a barrier between
// the calls.
//
// Bound by instruction issue and the latency of the levels' serial part (the
// payload is a fraction of the output), so the levels run in registers and
// warp shuffles: warp 0 rebuilds levels 4 to 2 from one bm3 byte a lane, all
// threads rebuild eight bm1 bytes each, an 8-lane byte transpose turns bm1
// words into a thread's sixteen plane nibbles, packed warp scans give the
// level-1 offsets, and each word is one funnel shift and one byte permute
// (planes that are empty across the warp are skipped).  The decoder it
// replaced staged and expanded single bytes: decode to codes of 25 M codes
// (500 x 500 x 100) 71 -> 44 us, the pfpl preset's decode of 67 M values 359 ->
// 269 us (62 % of the issue slots busy, the largest stall the barriers).
__device__ __forceinline__ void rze_decode_words(const uint8_t* rze, uint64_t rze_bytes, uint64_t off, uint32_t e,
                                                 int osz, RzeDecSmem& sm, uint32_t* err, uint32_t (&x)[16]) {
    const uint32_t t = threadIdx.x, lane = t & 31u, warp = t >> 5, full = 0xffffffffu;
    const uint32_t comp = e & 0x7fffffffu;
    uint32_t lead = 0;
    bool ok;
    stage_payload(rze, rze_bytes, off, e, sm.C, lead, ok);
    cp_async_wait_all();
    __syncthreads();
    // 0: RZE levels, 1: zeros, 2: stored raw (rze_stage.cu:904-930 cases)
    int kind;
    bool bad = !ok;
    if (bad) kind = 1;
    else if (e >> 31) {
        kind = 2;
        bad = (int)min(comp, (uint32_t)kChunkBytes) < osz;  // the bytes there are kept
    } else if (comp <= 2) kind = 1;
    else if (comp > (uint32_t)kChunkBytes || comp < 7u) {
        bad = true;
        kind = 1;
    } else kind = 0;
    const uint32_t* Cw = sm.C;
    const int b1 = (osz + 7) >> 3, b2 = (b1 + 7) >> 3, b3 = (b2 + 7) >> 3;
#pragma unroll
    for (int b = 0; b < 16; b++) x[b] = 0u;
    if (kind == 0) {
        if (warp == 0) {  // levels 4 -> 2
            const uint32_t bm4 = staged_word(Cw, lead + comp - 6);
            const int t3 = (int)comp - 6 - __popc(bm4);
            bool b = t3 < 0;
            const uint32_t r3 = __popc(bm4 & (full >> (31 - lane)));
            const uint32_t v3 = (r3 && !b && (int)lane < b3) ? staged_byte(Cw, lead + (uint32_t)t3 + r3 - 1) : 0u;
            const uint32_t p3 = __popc(v3);
            const uint32_t i3 = warp_incl_scan(p3);
            const int t2 = t3 - (int)__shfl_sync(full, i3, 31);
            b = b || t2 < 0;
            // bm2 bytes 8*lane .. 8*lane+7 from bm3 byte `lane`
            uint32_t w2[2] = {0u, 0u}, q2[8];
            uint32_t run = 0;
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint32_t rk = i3 - p3 + __popc(v3 & (0xffu >> (7 - j)));
                const uint32_t v = (rk && !b && (int)(8 * lane + j) < b2)
                                       ? staged_byte(Cw, lead + (uint32_t)t2 + rk - 1) : 0u;
                w2[j >> 2] |= v << (8 * (j & 3));
                q2[j] = run;
                run += __popc(v);
            }
            const uint32_t i2 = warp_incl_scan(run);
            const int t1 = t2 - (int)__shfl_sync(full, i2, 31);
            b = b || t1 < 0;
            reinterpret_cast<uint2*>(sm.bm2)[lane] = make_uint2(w2[0], w2[1]);
#pragma unroll
            for (int j = 0; j < 8; j++) sm.pfx2[8 * lane + j] = i2 - run + q2[j];
            if (lane == 0) {
                sm.misc[0] = b ? 0u : (uint32_t)t1;
                sm.misc[1] = b ? 1u : 0u;
            }
        }
        __syncthreads();
        const uint32_t s1 = sm.misc[0];
        if (sm.misc[1]) {
            bad = true;
            kind = 1;
        }
        if (kind == 0) {  // bm1 bytes 8t .. 8t+7
            const uint32_t m2 = sm.bm2[t], ex = sm.pfx2[t];
            uint32_t w1[2] = {0u, 0u};
#pragma unroll
            for (int j = 0; j < 8; j++) {
                const uint32_t rk = ex + __popc(m2 & (0xffu >> (7 - j)));
                const uint32_t v = (rk && (int)(8 * t + j) < b1) ? staged_byte(Cw, lead + s1 + rk - 1) : 0u;
                w1[j >> 2] |= v << (8 * (j & 3));
            }
            reinterpret_cast<uint2*>(sm.bm1)[t] = make_uint2(w1[0], w1[1]);
        }
        __syncthreads();
        // this thread's 16 plane nibbles and the per-plane level-1 offsets
        uint64_t nib64 = 0;
        uint32_t pm = 0, KX[4] = {0u, 0u, 0u, 0u};
        if (kind == 0) {
            const uint32_t j = lane & 7u;
            nib64 = nibs_from_bm1(sm.bm1[(15 - 2 * j) * 32 + (t >> 3)], sm.bm1[(14 - 2 * j) * 32 + (t >> 3)], lane);
            uint32_t K[4] = {0u, 0u, 0u, 0u}, mine = 0;
#pragma unroll
            for (int b = 0; b < 16; b++) {
                const uint32_t nb = (uint32_t)(nib64 >> (4 * b)) & 15u;
                K[b >> 2] += (uint32_t)__popc(nb) << (8 * (b & 3));
                mine |= (nb ? 1u : 0u) << b;
            }
            pm = __reduce_or_sync(full, mine);
            uint32_t act = 0;
#pragma unroll
            for (int jj = 0; jj < 4; jj++) act |= (((pm >> (4 * jj)) & 15u) ? 1u : 0u) << jj;
            warp_scan4(K, act, KX);
            if (lane == 31) {
#pragma unroll
                for (int jj = 0; jj < 4; jj++) sm.tot[warp][jj] = ((act >> jj) & 1u) ? KX[jj] : 0u;
            }
#pragma unroll
            for (int jj = 0; jj < 4; jj++) KX[jj] = ((act >> jj) & 1u) ? KX[jj] - K[jj] : 0u;
        }
        __syncthreads();
        if (kind == 0 && warp == 0) {
            const uint32_t b = lane & 15u, h = lane >> 4;
            uint32_t cnt[4];
#pragma unroll
            for (int i = 0; i < 4; i++) cnt[i] = (sm.tot[4 * h + i][b >> 2] >> (8 * (b & 3u))) & 0xffu;
            const uint32_t gs = cnt[0] + cnt[1] + cnt[2] + cnt[3];
            const uint32_t other = __shfl_xor_sync(full, gs, 16);
            const uint32_t T = gs + other;
            uint32_t suf = T;  // planes >= b come first (plane 15 leads)
#pragma unroll
            for (uint32_t d = 1; d < 16; d <<= 1) {
                const uint32_t n = __shfl_down_sync(full, suf, d, 16);
                if (b + d < 16) suf += n;
            }
            uint32_t o = suf - T + (h ? other : 0u);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                sm.base[4 * h + i][b] = o;
                o += cnt[i];
            }
            if (lane == 0 && suf != s1) sm.misc[1] = 1u;  // bitmap and payload disagree
        }
        __syncthreads();
        if (kind == 0 && sm.misc[1]) {
            bad = true;
            kind = 1;
        }
        if (kind == 0) {
#pragma unroll
            for (int b = 0; b < 16; b++) {
                if ((pm >> b) & 1u) {
                    const uint32_t nb = (uint32_t)(nib64 >> (4 * b)) & 15u;
                    const uint32_t pos = sm.base[warp][b] + ((KX[b >> 2] >> (8 * (b & 3))) & 0xffu);
                    x[b] = __byte_perm(staged_word(Cw, lead + pos), 0u, sm.exp[nb]);
                }
            }
        }
    } else if (kind == 2) {
        const int n = min((int)min(comp, (uint32_t)kChunkBytes), osz);
#pragma unroll
        for (int b = 0; b < 16; b++) {
            const int p = 4 * ((15 - b) * 256 + (int)t);
            const int have = n - p;  // bytes of this word inside the chunk
            if (have > 0) {
                const uint32_t w = staged_word(Cw, lead + (uint32_t)p);
                x[b] = have >= 4 ? w : (w & ((1u << (8 * have)) - 1u));
            }
        }
    }
    if (bad && t == 0) atomicOr(err, kErrMalformed);
}

// The bitshuffle inverse of a thread's plane words (its own inverse, see
// transpose16x2) followed by the pairing of codes 2l, 2l+1 of the thread's 32
// codes into c[l].
__device__ __forceinline__ void codes_from_planes(uint32_t (&x)[16], uint32_t (&c)[16]) {
    transpose16x2(x);
#pragma unroll
    for (int l = 0; l < 8; l++) {
        c[l] = __byte_perm(x[2 * l], x[2 * l + 1], 0x5410);
        c[l + 8] = __byte_perm(x[2 * l], x[2 * l + 1], 0x7632);
    }
}

}  // namespace
}  // namespace fzb
