// BGZF compression on the device: the write side of the path.
//
// The reference's DeviceBlockCompressor (crates/fritillaria-core/src/device.rs:
// 326-372) compresses device-resident chunks into framed BGZF blocks that come
// back to the host (the small side), one block per chunk, no EOF block; its
// only implementation hands the deflate to nvCOMP and frames the result with
// kernels/bgzf_frame.cu, choosing the framing on the host
// (choose_framing/framed_size, crates/fritillaria-core/src/compress.rs:
// 100-142).  DeviceBgzfWriter (crates/fritillaria-bgzf/src/device_write.rs)
// batches chunks through it and appends the EOF block at the end.  The
// contract is a round trip, not byte identity: inflating the output must give
// back the input, block for block.
//
// Here the deflate is this library's own, a CTA per chunk:
//   * CRC-32 of the chunk first, each thread over a slice from zero (thread 0
//     from the initial register), combined by linearity (crc_shift);
//   * greedy LZ77 over a 32 KiB window: a step looks at 32 positions, and the
//     first that matches the latest position before the step with its 3-byte
//     prefix's 11-bit hash ends a run of literals;
//   * the symbols counted, from which one warp builds length-limited Huffman
//     codes (RFC 1951 3.2.7) and keeps them when they beat the fixed codes
//     (3.2.6) header included; then one final block with the winner, each
//     thread's codes at the place a sum of their lengths gives it.
// A stream longer than a BGZF block can carry stops early; the host then
// stores the chunk, as choose_framing does.

#include <cstring>
#include <mutex>
#include <vector>

#include "common.cuh"
#include "runtime.h"

using namespace frt;

namespace {

constexpr u32 kMaxBlock = 65536;                         // MAX_BLOCK_SIZE
constexpr u32 kHeader = 18, kTrailer = 8, kStoredHeader = 5;
constexpr u32 kMaxDeflate = kMaxBlock - kHeader - kTrailer; // MAX_DEFLATE_STREAM
constexpr u32 kMaxPayload = kMaxDeflate - kStoredHeader;    // MAX_COMPRESSIBLE_PAYLOAD
constexpr u32 kSlot = 65536;                              // a chunk's deflate slot (bytes)
constexpr u32 kTooBig = 0xffffffffu;                      // a stream past kMaxDeflate
constexpr int kHashBits = 11;
constexpr u32 kWindow = 32768;
constexpr u32 kRing = 128;  // words of the bit-packing ring
constexpr u32 kFlush = 64;  // words flushed at a time

enum Framing : u8 { FRAMING_DEFLATED = 0, FRAMING_STORED = 1, FRAMING_EMPTY = 2 };

struct ByteCrc {
    u32 t[256];
};
constexpr ByteCrc make_byte_crc()
{
    ByteCrc c{};
    for (u32 i = 0; i < 256; ++i) {
        u32 v = i;
        for (int k = 0; k < 8; ++k) v = (v >> 1) ^ (0xEDB88320u & (0u - (v & 1u)));
        c.t[i] = v;
    }
    return c;
}
__device__ const ByteCrc g_bcrc = make_byte_crc();

constexpr u32 kScratch = 2048; // keys, weights, parents
struct TreeState {
    u32 table[kScratch]; // the CRC's byte table, then the Huffman builder's scratch
    u32 ring[kRing];
    u32 lf[286], df[30]; // literal/length and distance symbol counts of the parse
    u16 lcode[286], dcode[30], ccode[19]; // codes, reversed as they are packed
    u8 llen[286], dlen[30], clen[19];
    u16 items[320]; // the code lengths, run-length coded: symbol | extra value << 5
    u32 cf[19];     // counts of the code-length code's symbols
    u32 n_items, hlit, hdist, hclen, dynamic;
};
static_assert(sizeof(u32) * kScratch >= 4u * (512 + 1024) + 2u * 1024, "the builder's scratch fits");

__device__ __forceinline__ u32 prefix_hash(u32 b0, u32 b1, u32 b2)
{
    return (((b0 << 16) | (b1 << 8) | b2) * 2654435761u) >> (32 - kHashBits);
}

// A Huffman code as it is packed: the code reversed (deflate sends Huffman
// codes most significant bit first into a stream filled from the least
// significant bit), in the low bits.
__device__ __forceinline__ u32 rev(u32 code, u32 len) { return len ? __brev(code) >> (32u - len) : 0u; }

// Fixed literal/length code of symbol s (RFC 1951 3.2.6): (packed bits, length).
__device__ __forceinline__ void fixed_lit(u32 s, u32 *v, u32 *n)
{
    if (s < 144) *v = rev(0x30u + s, 8), *n = 8;
    else if (s < 256) *v = rev(0x190u + (s - 144u), 9), *n = 9;
    else if (s < 280) *v = rev(s - 256u, 7), *n = 7;
    else *v = rev(0xC0u + (s - 280u), 8), *n = 8;
}

// The length symbol of a match length (3..258) with its extra bits (RFC 1951 3.2.5).
__device__ __forceinline__ void len_sym(u32 L, u32 *sym, u32 *ex, u32 *nb)
{
    if (L == 258) {
        *sym = 285, *ex = 0, *nb = 0;
    } else if (L <= 10) {
        *sym = 254u + L, *ex = 0, *nb = 0;
    } else {
        const u32 x = L - 3u, k = 31u - __clz(x), hi = (x >> (k - 2u)) & 3u;
        *sym = 257u + 4u * (k - 1u) + hi;
        *nb = k - 2u;
        *ex = L - (3u + ((4u | hi) << (k - 2u)));
    }
}

// The distance symbol of a distance (1..32768) with its extra bits.
__device__ __forceinline__ void dist_sym(u32 d, u32 *sym, u32 *ex, u32 *nb)
{
    const u32 y = d - 1u;
    if (y < 4u) {
        *sym = y, *ex = 0, *nb = 0;
    } else {
        const u32 k = 31u - __clz(y), hi = (y >> (k - 1u)) & 1u;
        *sym = 2u * k + hi;
        *nb = k - 1u;
        *ex = d - (1u + ((2u | hi) << (k - 1u)));
    }
}

// Adds each lane's (v, n), n <= 31, at bit `bitpos` + the bits of the lanes
// below it; returns the new bit position (warp-uniform).
__device__ __forceinline__ u32 pack(TreeState *ws, u32 bitpos, u32 v, u32 n, u32 lane)
{
    u32 x = n;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 y = __shfl_up_sync(FRT_FULL_MASK, x, d);
        if (lane >= (u32)d) x += y;
    }
    const u32 total = __shfl_sync(FRT_FULL_MASK, x, 31);
    if (n) {
        const u32 o = bitpos + x - n, w = o >> 5, sh = o & 31u;
        atomicOr(&ws->ring[w % kRing], v << sh);
        if (sh + n > 32u) atomicOr(&ws->ring[(w + 1u) % kRing], v >> (32u - sh));
    }
    __syncwarp();
    return bitpos + total;
}

// Writes the ring's words [from, to) to the slot and clears them.
__device__ __forceinline__ void flush(TreeState *ws, u32 *slot, u32 from, u32 to, u32 lane)
{
    for (u32 w = from + lane; w < to; w += 32u) {
        slot[w] = ws->ring[w % kRing];
        ws->ring[w % kRing] = 0;
    }
    __syncwarp();
}

enum PassMode { EMIT_FIXED = 1, EMIT_DYNAMIC = 2 };

// Code lengths of a Huffman code for freq[0, n), at most maxlen bits: the
// used symbols (at least two; the lowest unused ones get a count of 1) sorted
// by (count, symbol) with a warp bitonic sort, a two-queue Huffman merge,
// the lengths past maxlen folded in by the Kraft sum (each excess leaf moves
// one shorter code a level down), and the shortest codes to the most frequent
// symbols.  Scratch: keys[512], wt[1024], parent[1024] (u16).
__device__ __forceinline__ void huff_lengths(u32 *freq, u32 n, u32 maxlen, u8 *lens, u32 *keys, u32 *wt, u16 *parent, u32 lane)
{
    u32 used = 0;
    for (u32 b = 0; b < n; b += 32u) used += __popc(__ballot_sync(FRT_FULL_MASK, b + lane < n && freq[b + lane]));
    const u32 m = max(used, 2u);
    if (lane == 0)
        for (u32 s = 0; s < n && used < 2u; ++s)
            if (!freq[s]) freq[s] = 1u, ++used;
    __syncwarp();
    const u32 most = n <= 32u ? 32u : 512u; // keys sorted
    for (u32 i = lane; i < most; i += 32u) keys[i] = i < n && freq[i] ? (freq[i] << 9) | i : 0xffffffffu;
    for (u32 i = lane; i < n; i += 32u) lens[i] = 0;
    __syncwarp();
    for (u32 size = 2; size <= most; size <<= 1)
        for (u32 stride = size >> 1; stride; stride >>= 1) {
            for (u32 t = lane; t < most / 2u; t += 32u) {
                const u32 i = 2u * t - (t & (stride - 1u)), j = i + stride;
                const bool up = (i & size) == 0;
                const u32 a = keys[i], b = keys[j];
                if ((a > b) == up) keys[i] = b, keys[j] = a;
            }
            __syncwarp();
        }
    for (u32 i = lane; i < m; i += 32u) wt[i] = keys[i] >> 9;
    __syncwarp();
    if (lane == 0) {
        // two queues, the leaves and the inner nodes, their heads in registers
        constexpr u32 NONE = 0xffffffffu;
        u32 li = 0, ii = m, leaf = wt[0], inner = NONE;
        for (u32 nxt = m; nxt < 2u * m - 1u; ++nxt) {
            u32 sum = 0;
#pragma unroll
            for (int t = 0; t < 2; ++t) {
                if (leaf != NONE && leaf <= inner) {
                    sum += leaf;
                    parent[li++] = (u16)nxt;
                    leaf = li < m ? wt[li] : NONE;
                } else {
                    sum += inner;
                    parent[ii++] = (u16)nxt;
                    inner = ii < nxt ? wt[ii] : NONE;
                }
            }
            wt[nxt] = sum;
            if (inner == NONE) inner = wt[ii]; // the node just made heads the empty queue
        }
    }
    __syncwarp();
    // depths: each leaf counts the links to the root; lane L has the leaves at L
    const u32 root = 2u * m - 2u;
    u32 cnt = 0;
    for (u32 b = 0; b < m; b += 32u) {
        const u32 i = b + lane;
        u32 d = 0;
        if (i < m)
            for (u32 at = i; at != root; at = parent[at]) ++d;
        d = min(d, maxlen);
        for (u32 L = 1; L <= maxlen; ++L) {
            const u32 here = __popc(__ballot_sync(FRT_FULL_MASK, i < m && d == L));
            if (lane == L) cnt += here;
        }
    }
    u32 total = __reduce_add_sync(FRT_FULL_MASK, lane >= 1u && lane <= maxlen ? cnt << (maxlen - lane) : 0u);
    while (total > (1u << maxlen)) { // one leaf of the deepest level goes beside one moved a level down
        const u32 over = __ballot_sync(FRT_FULL_MASK, lane >= 1u && lane < maxlen && cnt) , L = 31u - __clz(over);
        if (lane == maxlen) --cnt;
        if (lane == L) --cnt;
        if (lane == L + 1u) cnt += 2u;
        --total;
    }
    // the shortest codes to the most frequent symbols (keys[m - 1] the most)
    u32 upto = lane >= 1u && lane <= maxlen ? cnt : 0u;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 y = __shfl_up_sync(FRT_FULL_MASK, upto, d);
        if (lane >= (u32)d) upto += y;
    }
    for (u32 b = 0; b < m; b += 32u) {
        const u32 i = b + lane;
        u32 L = 1;
        for (u32 l = 1; l < maxlen; ++l) L += i >= __shfl_sync(FRT_FULL_MASK, upto, l) ? 1u : 0u;
        if (i < m) lens[keys[m - 1u - i] & 511u] = (u8)L;
    }
    __syncwarp();
}

// Canonical codes of lens[0, n) (RFC 1951 3.2.2), reversed for packing.
// By a warp: lane L keeps the next code of length L.
__device__ __forceinline__ void canonical(const u8 *lens, u32 n, u16 *codes, u32 lane)
{
    u32 cnt = 0;
    for (u32 b = 0; b < n; b += 32u) {
        const u32 l = b + lane < n ? lens[b + lane] : 0u;
        for (u32 L = 1; L < 16u; ++L) {
            const u32 here = __popc(__ballot_sync(FRT_FULL_MASK, l == L));
            if (lane == L) cnt += here;
        }
    }
    u32 next = 0, code = 0;
    for (u32 L = 1; L < 16u; ++L) {
        code = (code + __shfl_sync(FRT_FULL_MASK, cnt, L - 1u)) << 1;
        if (lane == L) next = code;
    }
    for (u32 b = 0; b < n; b += 32u) {
        const u32 l = b + lane < n ? lens[b + lane] : 0u;
        for (u32 L = 1; L < 16u; ++L) {
            const u32 here = __ballot_sync(FRT_FULL_MASK, l == L);
            const u32 base = __shfl_sync(FRT_FULL_MASK, next, L);
            if (l == L) codes[b + lane] = (u16)rev(base + __popc(here & lanemask_lt()), L);
            if (lane == L) next += __popc(here);
        }
    }
    __syncwarp();
}

__device__ const u8 kClOrder[19] = {16, 17, 18, 0, 8, 7, 9, 6, 10, 5, 11, 4, 12, 3, 13, 2, 14, 1, 15};

__device__ __forceinline__ u32 fixed_len(u32 s) { return s < 144 ? 8u : s < 256 ? 9u : s < 280 ? 7u : 8u; }
__device__ __forceinline__ u32 cl_extra(u32 sym) { return sym == 16 ? 2u : sym == 17 ? 3u : sym == 18 ? 7u : 0u; }

// The dynamic trees from the counts (lf[256] counts the end of block), and
// whether they beat the fixed codes, their header included (the extra bits
// of lengths and distances are the same either way).
__device__ __forceinline__ void build_trees(TreeState *ws, u32 lane)
{
    u32 *keys = ws->table, *wt = ws->table + 512;
    u16 *parent = (u16 *)(ws->table + 1536);
    huff_lengths(ws->lf, 286, 15, ws->llen, keys, wt, parent, lane);
    huff_lengths(ws->df, 30, 15, ws->dlen, keys, wt, parent, lane);
    u32 hlit = 257, hdist = 1; // up to the last symbols with a code
    if (lane < 29u && ws->llen[257u + lane]) hlit = 258u + lane;
    if (lane < 30u && ws->dlen[lane]) hdist = 1u + lane;
    hlit = __reduce_max_sync(FRT_FULL_MASK, hlit);
    hdist = __reduce_max_sync(FRT_FULL_MASK, hdist);
    // run-length code the lengths (RFC 1951 3.2.7): 16 repeats the previous
    // length 3-6 times, 17 and 18 are runs of 3-10 and 11-138 zeros.  The warp
    // marks where runs begin, one lane goes from mark to mark.
    const u32 total = hlit + hdist;
    u32 *const begins = keys; // a bit a length, one past the last set too
    for (u32 b = 0; b <= total; b += 32u) {
        const u32 i = b + lane;
        const u32 cur = i < hlit ? ws->llen[i] : (i < total ? ws->dlen[i - hlit] : 0u);
        const u32 before = i == 0 || i > total ? 0u : (i - 1u < hlit ? ws->llen[i - 1u] : ws->dlen[i - 1u - hlit]);
        const u32 m = __ballot_sync(FRT_FULL_MASK, i == 0 || i == total || (i < total && cur != before));
        if (lane == 0) begins[b >> 5] = m;
    }
    __syncwarp();
    if (lane == 0) {
        u32 n = 0, i = 0;
        while (i < total) {
            const u32 v = i < hlit ? ws->llen[i] : ws->dlen[i - hlit];
            u32 w = (i + 1u) >> 5, m = begins[w] & (0xffffffffu << ((i + 1u) & 31u));
            while (!m) m = begins[++w];
            const u32 j = 32u * w + (u32)__ffs(m) - 1u;
            u32 run = j - i;
            if (v == 0) {
                while (run >= 11) {
                    const u32 r = min(run, 138u);
                    ws->items[n++] = (u16)(18u | ((r - 11u) << 5));
                    run -= r;
                }
                if (run >= 3) {
                    ws->items[n++] = (u16)(17u | ((run - 3u) << 5));
                    run = 0;
                }
                while (run--) ws->items[n++] = 0;
            } else {
                ws->items[n++] = (u16)v;
                --run;
                while (run >= 3) {
                    const u32 r = min(run, 6u);
                    ws->items[n++] = (u16)(16u | ((r - 3u) << 5));
                    run -= r;
                }
                while (run--) ws->items[n++] = (u16)v;
            }
            i = j;
        }
        ws->n_items = n;
        ws->hlit = hlit;
        ws->hdist = hdist;
        for (u32 t = 0; t < 19; ++t) ws->cf[t] = 0;
        for (u32 t = 0; t < n; ++t) ++ws->cf[ws->items[t] & 31u];
    }
    __syncwarp();
    huff_lengths(ws->cf, 19, 7, ws->clen, keys, wt, parent, lane);
    canonical(ws->llen, 286, ws->lcode, lane);
    canonical(ws->dlen, 30, ws->dcode, lane);
    canonical(ws->clen, 19, ws->ccode, lane);
    // bits of the two forms; sums of at most 65,505 symbols' bits fit 32 bits
    u32 dyn = 0, fix = 0;
    for (u32 t = lane; t < ws->n_items; t += 32u) {
        const u32 sym = ws->items[t] & 31u;
        dyn += ws->clen[sym] + cl_extra(sym);
    }
    for (u32 sy = lane; sy < 286; sy += 32u) {
        dyn += ws->lf[sy] * ws->llen[sy];
        fix += ws->lf[sy] * fixed_len(sy);
    }
    if (lane < 30u) {
        dyn += ws->df[lane] * ws->dlen[lane];
        fix += ws->df[lane] * 5u;
    }
    dyn = __reduce_add_sync(FRT_FULL_MASK, dyn);
    fix = __reduce_add_sync(FRT_FULL_MASK, fix);
    if (lane == 0) {
        u32 hclen = 19;
        while (hclen > 4 && !ws->clen[kClOrder[hclen - 1]]) --hclen;
        ws->hclen = hclen;
        ws->dynamic = dyn + 17u + 3u * hclen < fix + 3u ? 1u : 0u;
    }
    __syncwarp();
}

__device__ __forceinline__ void flush_some(TreeState *ws, u32 *slot, u32 bitpos, u32 &flushed, u32 lane)
{
    if ((bitpos >> 5) - flushed >= kFlush) {
        flush(ws, slot, flushed, flushed + kFlush, lane);
        flushed += kFlush;
    }
}

constexpr u32 kWarm = 512; // bytes a warp parses before its part
constexpr u32 kOthers = 40;

// A chunk's state, of at most MAX bytes, for a CTA of THREADS; LINKS of its
// warps link the prefixes.
template <u32 THREADS, u32 LINKS, u32 MAX> struct ChunkState {
    static constexpr u32 kThreads = THREADS, kWarps = THREADS / 32, kLinkWarps = LINKS, kMax = MAX;
    // The latest position + 1 before each one with the same prefix hash (0 none).
    u16 prev[MAX];
    union {
        u8 match[MAX];                    // match length with it, less 2, 255 for 257 and 258; 0: no match
        u16 last[LINKS][1u << kHashBits]; // while prev is built: each warp's last position + 1 of a hash
    };
    u32 inside[MAX / 32]; // positions inside a match, but its first
    u32 first[MAX / 32];  // first positions of matches
    u32 end[kWarps], sums[kWarps], head_bits; // where the warps' parts end; the block header's bits
    u32 other[kWarps][kOthers]; // a warp's matches with a candidate that is not prev: position | candidate << 16
    TreeState tree;
};

// The shapes a chunk is compressed in.
using Large = ChunkState<1024, 16, 65536>; // all of an SM's shared memory; 16 parts of a parse took half as long again
using Medium = ChunkState<256, 4, 8192>;   // four to an SM
using Small = ChunkState<128, 2, 4096>;    // seven

// Four bytes at p[i], all of them inside the chunk.
__device__ __forceinline__ u32 load4(const u8 *p, u32 i)
{
    const u64 a = (u64)(p + i);
    const u32 *w = (const u32 *)(a & ~3ull), sh = 8u * ((u32)a & 3u);
    const u32 lo = __ldg(w);
    return sh ? __funnelshift_r(lo, __ldg(w + 1), sh) : lo;
}

__device__ __forceinline__ u32 hash_at(const u8 *p, u32 q) { return prefix_hash(p[q], p[q + 1u], p[q + 2u]); }

// Bytes, at most `most`, in which position q and the earlier c agree, which are
// known to be i at least.
__device__ __forceinline__ u32 bytes_alike(const u8 *p, u32 q, u32 c, u32 len, u32 i, u32 most)
{
    const u32 cap = min(most, len - q);
    while (i + 4u <= cap) {
        const u32 x = load4(p, q + i) ^ load4(p, c + i);
        if (x) return i + (((u32)__ffs(x) - 1u) >> 3);
        i += 4;
    }
    while (i < cap && p[q + i] == p[c + i]) ++i;
    return i;
}

// Length of the match of position q with the earlier c (0: their first three
// bytes differ), for q + 3 <= len.
__device__ __forceinline__ u32 match_length(const u8 *p, u32 q, u32 c, u32 len)
{
    const u32 i = bytes_alike(p, q, c, len, 0, 258);
    return i >= 3u ? i : 0u;
}

constexpr u32 kNear = 32; // bytes every position compares (64: 1.09 and 1.83 ms below)

// match for the whole chunk, from prev.  All threads compare up to kNear bytes of
// each position first.  Where they all agree, most often the positions after do
// too at the same distance, and two of those no further apart than kNear end
// their matches at the same byte: so a warp goes over its part from the end and
// compares further only where the distance is a new one.  (By itself each
// position of a run or a repeated block takes 65 loads: 450 chunks of zeros 2.06
// ms, now 0.93, and of a block of 5,000 bytes over and over 2.58, now 1.78.)
template <class CS> __device__ __forceinline__ void match_all(CS *cs, const u8 *p, u32 len)
{
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
    for (u32 q = threadIdx.x; q < len; q += CS::kThreads) {
        const u32 c = q + 3u <= len ? cs->prev[q] : 0u;
        const u32 L = c && q - (c - 1u) <= kWindow ? bytes_alike(p, q, c - 1u, len, 0, kNear) : 0u;
        cs->match[q] = (u8)(L >= 3u ? L - 2u : 0u);
    }
    __syncthreads();
    const u32 part = (len + 32u * CS::kWarps - 1) / (32u * CS::kWarps) * 32u, from = warp * part, to = min(len, from + part);
    u32 last_d = 0, last_q = 0, last = 0; // the first such position of the turn before, and its length
    for (u32 n = from < to ? (to - from + 31u) / 32u : 0u; n--;) {
        const u32 q = from + 32u * n + lane;
        const bool open = q < to && cs->match[q] == kNear - 2u;
        const u32 some = __ballot_sync(FRT_FULL_MASK, open);
        if (!some) continue;
        const u32 d = open ? q + 1u - cs->prev[q] : 0x10000u + lane;
        const u32 peers = __match_any_sync(FRT_FULL_MASK, d), top = 31u - __clz(peers);
        u32 L = 0;
        if (open && lane == top)
            L = d == last_d && last_q - q <= kNear ? last + (last_q - q) : bytes_alike(p, q, q - d, len, kNear, 258);
        L = min(__shfl_sync(FRT_FULL_MASK, L, top) + (top - lane), 258u);
        if (open) cs->match[q] = (u8)min(L - 2u, 255u);
        const u32 first = __ffs(some) - 1u;
        last_d = __shfl_sync(FRT_FULL_MASK, d, first);
        last_q = __shfl_sync(FRT_FULL_MASK, q, first);
        last = __shfl_sync(FRT_FULL_MASK, L, first);
    }
}

// prev for the whole chunk: each warp goes over a part 32 positions at a time
// with a table of its own (lanes of one hash find each other by match_any);
// then each hash's last position before every part, and the positions their
// part had no earlier one for.
template <class CS> __device__ __forceinline__ void link_prefixes(CS *cs, const u8 *p, u32 len)
{
    constexpr u32 kThreads = CS::kThreads, kLinkWarps = CS::kLinkWarps;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
    const u32 part = (len + 32u * kLinkWarps - 1) / (32u * kLinkWarps) * 32u;
    u16 *last = cs->last[warp % kLinkWarps];
    for (u32 i = tid; i < kLinkWarps << (kHashBits - 1); i += kThreads) ((u32 *)cs->last)[i] = 0;
    __syncthreads();
    const u32 to = warp < kLinkWarps ? min(len, (warp + 1) * part) : 0u;
    for (u32 b = warp * part; b < to; b += 32) {
        const u32 q = b + lane;
        const bool in = q < to && q + 3u <= len;
        const u32 h = in ? hash_at(p, q) : 0u;
        u32 before = in ? last[h] : 0u;
        __syncwarp();
        if (in) last[h] = (u16)(q + 1u);
        __syncwarp();
        // lanes of one hash: one of them has written (seen without match_any,
        // whose 32 distinct values cost more than the rest of the turn)
        if (__any_sync(FRT_FULL_MASK, in && last[h] != (u16)(q + 1u))) {
            const u32 peers = __match_any_sync(FRT_FULL_MASK, in ? h : 0x10000u + lane), below = peers & lanemask_lt();
            if (below) before = b + 32u - __clz(below);
            __syncwarp();
            if (in && (peers >> lane) == 1u) last[h] = (u16)(q + 1u);
        }
        if (q < to) cs->prev[q] = (u16)(in ? before : 0u);
        __syncwarp();
    }
    __syncthreads();
    for (u32 h = tid; h < (1u << kHashBits); h += kThreads) {
        u16 run = 0;
        for (u32 w = 0; w < kLinkWarps; ++w) {
            const u16 t = cs->last[w][h];
            cs->last[w][h] = run;
            if (t) run = t;
        }
    }
    __syncthreads();
    for (u32 q = tid; q + 3u <= len; q += kThreads)
        if (cs->prev[q] == 0) cs->prev[q] = cs->last[q / part][hash_at(p, q)];
    __syncthreads();
}

// One step of the greedy parse at `pos`, by a warp (uniform result): the first
// of the next 32 positions that matches the latest position before `pos` with
// its hash ends a run of literals.  Returns where the step ends; `m`, `L` and
// `c` are its match (L 0: none), `again` whether c is not prev.  It depends on `pos` alone, so parts of the
// chunk can be parsed apart.  That candidate is prev, or, where prev lies in
// the step itself, further back along prev (rare: looked at by its bytes).
template <class CS>
__device__ __forceinline__ u32 parse_step(const CS *cs, const u8 *p, u32 len, u32 pos, u32 &m, u32 &L, u32 &c, bool &again)
{
    const u32 lane = lane_id(), q = pos + lane;
    const bool in = q + 3u <= len;
    const u32 pv = in ? cs->prev[q] : 0u, got = in ? cs->match[q] : 0u;
    const u32 hits = __ballot_sync(FRT_FULL_MASK, pv && pv <= pos && got);
    u32 k = hits ? (u32)__ffs(hits) - 1u : 32u;
    const u32 late = __ballot_sync(FRT_FULL_MASK, pv > pos) & (k < 32u ? (1u << k) - 1u : 0xffffffffu);
    u32 at = pv;
    again = false;
    if (late) {
        const bool mine = (late >> lane) & 1u;
        while (__any_sync(FRT_FULL_MASK, mine && at > pos))
            if (mine && at > pos) at = cs->prev[at - 1u];
        const bool ok = mine && at && q - (at - 1u) <= kWindow && p[at - 1u] == p[q] && p[at] == p[q + 1u] && p[at + 1u] == p[q + 2u];
        const u32 more = __ballot_sync(FRT_FULL_MASK, ok);
        if (more) {
            k = (u32)__ffs(more) - 1u;
            again = true;
        }
    }
    L = 0;
    if (k == 32u) return min(pos + 32u, len);
    m = pos + k;
    c = __shfl_sync(FRT_FULL_MASK, at, k) - 1u;
    if (again) {
        L = match_length(p, m, c, len);
    } else {
        L = __shfl_sync(FRT_FULL_MASK, got, k) + 2u;
        if (L == 257u && len - m >= 258u && p[m + 257u] == p[c + 257u]) L = 258u;
    }
    return m + L;
}

// Marks the match of L bytes at m in `first` and `inside`, by a warp.
template <class CS> __device__ __forceinline__ void mark_match(CS *cs, u32 m, u32 L)
{
    // lane 31 marks the first byte, the others the words of [m + 1, m + L): at
    // most 10, most often one
    const u32 lane = lane_id(), a = m + 1u, e = m + L, w = lane == 31u ? m >> 5 : (a >> 5) + lane;
    const u32 lo = max(a, 32u * w) & 31u, hi = min(e - 32u * w, 32u);
    const u32 bits = lane == 31u ? 1u << (m & 31u) : (0xffffffffu << lo) & (hi == 32u ? 0xffffffffu : (1u << (hi & 31u)) - 1u);
    if (lane == 31u || 32u * w < e) atomicOr((lane == 31u ? cs->first : cs->inside) + w, bits);
}

template <class CS> __device__ __forceinline__ void clear_marks(CS *cs)
{
    for (u32 i = threadIdx.x; i < CS::kMax / 32; i += CS::kThreads) cs->inside[i] = cs->first[i] = 0;
    __syncthreads();
}

// The parse of the chunk: its matches marked in `first` and `inside`, with
// prev and match their candidates and lengths.  Each warp parses and marks a
// part from where a parse begun kWarm bytes before it first reaches it.  Where
// a part then does not start where the one before ended (rare), the marks go,
// the starts are found, each such part again from its right place, and all
// parts are marked anew.
template <class CS> __device__ __forceinline__ void parse(CS *cs, const u8 *p, u32 len)
{
    constexpr u32 kWarps = CS::kWarps;
    const u32 lane = threadIdx.x & 31u, warp = threadIdx.x / 32;
    const u32 part = (len + kWarps - 1) / kWarps, from = min(len, warp * part), to = min(len, from + part);
    bool again;
    u32 m, L, c, pos = from > kWarm ? from - kWarm : 0u, others = 0;
    clear_marks(cs);
    while (pos < from) pos = parse_step(cs, p, len, pos, m, L, c, again);
    u32 start = pos;
    while (pos < to) {
        pos = parse_step(cs, p, len, pos, m, L, c, again);
        if (L) {
            mark_match(cs, m, L);
            if (again) { // prev stays as it is until the parse is proven
                if (lane == 0 && others < kOthers) cs->other[warp][others] = m | (c << 16);
                ++others;
            }
        }
    }
    if (lane == 0) cs->end[warp] = pos;
    __syncthreads();
    if (!__syncthreads_or(start != (warp ? cs->end[warp - 1] : 0u) || others > kOthers)) {
        for (u32 i = lane; i < others; i += 32u) {
            const u32 q = cs->other[warp][i] & 0xffffu, at = cs->other[warp][i] >> 16;
            cs->prev[q] = (u16)(at + 1u);
            cs->match[q] = (u8)min(match_length(p, q, at, len) - 2u, 255u);
        }
        __syncthreads();
        return;
    }
    while (true) {
        const u32 before = warp ? cs->end[warp - 1] : 0u;
        const bool go = start != before;
        start = before;
        if (!__syncthreads_or(go)) break;
        if (go) {
            pos = start;
            while (pos < to) pos = parse_step(cs, p, len, pos, m, L, c, again);
            if (lane == 0) cs->end[warp] = pos;
        }
        __syncthreads();
    }
    clear_marks(cs);
    for (pos = start; pos < to;) {
        pos = parse_step(cs, p, len, pos, m, L, c, again);
        if (L) {
            if (lane == 0) {
                cs->prev[m] = (u16)(c + 1u);
                cs->match[m] = (u8)min(L - 2u, 255u);
            }
            mark_match(cs, m, L);
            __syncwarp();
        }
    }
    __syncthreads();
}

// The symbols and extra bits of the match that starts at q.
template <class CS>
__device__ __forceinline__ void match_symbols(const CS *cs, const u8 *p, u32 len, u32 q, u32 &ls, u32 &lex, u32 &lnb,
                                              u32 &ds, u32 &dex, u32 &dnb)
{
    const u32 c = cs->prev[q] - 1u;
    u32 L = cs->match[q] + 2u;
    if (L == 257u && len - q >= 258u && p[q + 257u] == p[c + 257u]) L = 258u;
    len_sym(L, &ls, &lex, &lnb);
    dist_sym(q - c, &ds, &dex, &dnb);
}

// A symbol's code and extra bits (at most 20, a distance's 28 after them) and
// their lengths: the match that starts at q, or the literal `byte`.
template <int MODE, class CS>
__device__ __forceinline__ void symbol_bits(const CS *cs, const u8 *p, u32 len, u32 q, bool match, u32 byte, u32 &v, u32 &nb,
                                            u32 &v2, u32 &nb2)
{
    const TreeState *ws = &cs->tree;
    nb2 = 0;
    if (!match) {
        if (MODE == EMIT_FIXED) fixed_lit(byte, &v, &nb);
        else v = ws->lcode[byte], nb = ws->llen[byte];
        return;
    }
    u32 ls, lex, lnb, ds, dex, dnb;
    match_symbols(cs, p, len, q, ls, lex, lnb, ds, dex, dnb);
    if (MODE == EMIT_FIXED) {
        fixed_lit(ls, &v, &nb);
        v2 = rev(ds, 5), nb2 = 5;
    } else {
        v = ws->lcode[ls], nb = ws->llen[ls];
        v2 = ws->dcode[ds], nb2 = ws->dlen[ds];
    }
    v |= lex << nb;
    nb += lnb;
    v2 |= dex << nb2;
    nb2 += dnb;
}

// Writes a thread's run of bits: whole words by plain stores, the words it
// shares with the runs beside it by atomicOr (cleared beforehand).
struct BitRun {
    u32 *slot;
    u64 acc = 0;
    u32 have, word;
    bool shared = true; // the word at `word` holds earlier runs' bits too
    __device__ BitRun(u32 *s, u32 bit) : slot(s), have(bit & 31u), word(bit >> 5) {}
    __device__ __forceinline__ void put(u32 v, u32 n)
    {
        acc |= (u64)v << have;
        have += n;
        if (have >= 32u) {
            if (shared) atomicOr(&slot[word], (u32)acc);
            else slot[word] = (u32)acc;
            shared = false;
            ++word;
            acc >>= 32;
            have -= 32u;
        }
    }
    __device__ __forceinline__ void done()
    {
        if (have) atomicOr(&slot[word], (u32)acc);
    }
};

// Calls f(v, nb, v2, nb2) for each symbol of positions [from, to), in order;
// `from` is a multiple of 32.
template <int MODE, class CS, class F>
__device__ __forceinline__ void each_symbol(const CS *cs, const u8 *p, u32 len, u32 from, u32 to, F f)
{
    for (u32 b = from; b < to; b += 32) {
        u32 m = ~cs->inside[b >> 5];
        if (to - b < 32u) m &= (1u << (to - b)) - 1u;
        const u32 first = cs->first[b >> 5];
        u32 at = 0xffffffffu, four = 0;
        for (; m; m &= m - 1) {
            const u32 k = (u32)__ffs(m) - 1u, q = b + k;
            if ((k >> 2) != at && !((first >> k) & 1u)) {
                at = k >> 2;
                if (b + 4u * at + 4u <= len) four = load4(p, b + 4u * at);
                else
                    for (u32 i = four = 0; b + 4u * at + i < len; ++i) four |= (u32)p[b + 4u * at + i] << (8u * i);
            }
            u32 v, nb, v2, nb2;
            symbol_bits<MODE>(cs, p, len, q, (first >> k) & 1u, (four >> (8u * (k & 3u))) & 0xffu, v, nb, v2, nb2);
            f(v, nb, v2, nb2);
        }
    }
}

// The chunk's symbols as bits from `bit` on in the slot: each thread takes a
// run of positions, its place from a sum over the team.  Returns the bit past
// the last, the same in every thread, or 0 where the block with its
// end-of-block code of `eob` bits would outgrow a BGZF block.
template <int MODE, class CS>
__device__ __forceinline__ u32 emit(CS *cs, const u8 *p, u32 len, u32 *slot, u32 bit, u32 eob)
{
    constexpr u32 kThreads = CS::kThreads, kWarps = CS::kWarps;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32;
    // whole words of marks a thread; the chunk's bytes four at a time
    const u32 per = (len + 32u * kThreads - 1) / (32u * kThreads) * 32u, from = min(len, tid * per), to = min(len, from + per);
    u32 sum = 0;
    each_symbol<MODE>(cs, p, len, from, to, [&](u32, u32 nb, u32, u32 nb2) { sum += nb + nb2; });
    u32 x = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const u32 y = __shfl_up_sync(FRT_FULL_MASK, x, d);
        if (lane >= (u32)d) x += y;
    }
    if (lane == 31) cs->sums[warp] = x;
    __syncthreads();
    u32 before = bit, total = bit;
    for (u32 w = 0; w < kWarps; ++w) {
        if (w < warp) before += cs->sums[w];
        total += cs->sums[w];
    }
    if (((total + eob + 7u) >> 3) > kMaxDeflate) return 0;
    const u32 clear = (total + eob + 31u) >> 5;
    for (u32 w = ((bit + 31u) >> 5) + tid; w < clear; w += kThreads) slot[w] = 0;
    __syncthreads();
    BitRun run(slot, before + x - sum);
    each_symbol<MODE>(cs, p, len, from, to, [&](u32 v, u32 nb, u32 v2, u32 nb2) {
        run.put(v, nb);
        if (nb2) run.put(v2, nb2);
    });
    run.done();
    return total;
}

// A CTA per chunk, in one of the three shapes (by_shape).
//
// A warp per chunk walked the parse with its hash table, twice: each step a
// chain of dependent loads through L2, 2,000 cycles, 20 ms for a 64 KiB chunk
// whatever the number of chunks.  What a step does depends only on where it
// starts, once every position's earlier positions of its hash are linked: so
// the links and every position's match length are made by all threads at once,
// the warps parse as many parts (parses from different starts fall into
// step within a few matches), and counts and codes are taken position by
// position.  The stream is bit for bit the one-warp form's.  Measured on GB300
// through compress_batch_device: 454 chunks of short reads (29.6 MB) 19.8 ->
// 1.64 ms.
template <class CS>
__global__ void __launch_bounds__(CS::kThreads, 227u * 1024u / (sizeof(CS) + 1024u))
k_deflate_chunks(const u8 *data, const u64 *bounds, const u32 *which, u8 *slots, u32 *deflate_len, u32 *crcs)
{
    constexpr u32 kThreads = CS::kThreads, kWarps = CS::kWarps;
    extern __shared__ __align__(16) unsigned char smem[];
    CS *cs = (CS *)smem;
    TreeState *ws = &cs->tree;
    const u32 tid = threadIdx.x, lane = tid & 31u, warp = tid / 32, chunk = which ? which[blockIdx.x] : blockIdx.x;
    const u8 *p = data + bounds[chunk];
    const u32 len = (u32)(bounds[chunk + 1] - bounds[chunk]);

    // CRC-32: thread slices of whole words from zero, shifted past the bytes
    // after them; the byte table in the tree builder's scratch
    {
        u32 *t = ws->table;
        for (u32 i = tid; i < 256u; i += kThreads) t[i] = g_bcrc.t[i];
        __syncthreads();
        const u32 head = min(len, (4u - (u32)((u64)p & 3u)) & 3u), words = (len - head) / 4u;
        const u32 per = (words + kThreads - 1) / kThreads, w0 = min(words, tid * per), w1 = min(words, w0 + per);
        const u32 *w = (const u32 *)(p + head);
        u32 c = 0, end = head + 4u * w1;
        if (tid == 0) {
            c = 0xffffffffu;
            for (u32 i = 0; i < head; ++i) c = t[(c ^ p[i]) & 0xffu] ^ (c >> 8);
        }
        for (u32 i = w0; i < w1; ++i) {
            c ^= __ldg(w + i);
#pragma unroll
            for (int b = 0; b < 4; ++b) c = t[c & 0xffu] ^ (c >> 8);
        }
        if (w1 == words && (w0 < words || tid == 0))
            for (; end < len; ++end) c = t[(c ^ p[end]) & 0xffu] ^ (c >> 8);
        if (c) c = crc_shift(c, len - end);
        c = __reduce_xor_sync(FRT_FULL_MASK, c);
        if (lane == 0) cs->sums[warp] = c;
        __syncthreads();
        if (tid == 0) {
            for (u32 k = 1; k < kWarps; ++k) c ^= cs->sums[k];
            crcs[chunk] = ~c;
        }
        __syncthreads();
    }
    if (len == 0) {
        if (tid == 0) deflate_len[chunk] = 0;
        return;
    }
    link_prefixes(cs, p, len);
    match_all(cs, p, len);
    for (u32 i = tid; i < kRing; i += kThreads) ws->ring[i] = 0;
    for (u32 i = tid; i < 286u; i += kThreads) ws->lf[i] = i == 256u ? 1u : 0u; // the end of block
    if (tid < 30u) ws->df[tid] = 0;
    __syncthreads();
    parse(cs, p, len);
    for (u32 q = tid; q < len; q += kThreads) {
        if ((cs->inside[q >> 5] >> (q & 31u)) & 1u) continue;
        if ((cs->first[q >> 5] >> (q & 31u)) & 1u) {
            u32 ls, lex, lnb, ds, dex, dnb;
            match_symbols(cs, p, len, q, ls, lex, lnb, ds, dex, dnb);
            atomicAdd(&ws->lf[ls], 1u);
            atomicAdd(&ws->df[ds], 1u);
        } else {
            atomicAdd(&ws->lf[p[q]], 1u);
        }
    }
    __syncthreads();
    u32 *slot = (u32 *)(slots + (size_t)chunk * kSlot);
    if (warp == 0) {
        build_trees(ws, lane);
        u32 bitpos = 0, flushed = 0;
        if (!ws->dynamic) {
            bitpos = pack(ws, 0, 3u, lane == 0 ? 3u : 0u, lane); // BFINAL 1, BTYPE 01
        } else {
            // BFINAL 1, BTYPE 10, HLIT, HDIST, HCLEN; the code-length code's lengths
            // in their permuted order; the run-length coded lengths
            const u32 h = 1u | (2u << 1) | ((ws->hlit - 257u) << 3) | ((ws->hdist - 1u) << 8) | ((ws->hclen - 4u) << 13);
            bitpos = pack(ws, 0, lane == 0 ? h : 0u, lane == 0 ? 17u : 0u, lane);
            bitpos = pack(ws, bitpos, lane < ws->hclen ? ws->clen[kClOrder[lane]] : 0u, lane < ws->hclen ? 3u : 0u, lane);
            for (u32 base = 0; base < ws->n_items; base += 32u) {
                const u32 i = base + lane;
                u32 v = 0, nb = 0;
                if (i < ws->n_items) {
                    const u32 it = ws->items[i], sym = it & 31u;
                    v = ws->ccode[sym] | ((it >> 5) << ws->clen[sym]);
                    nb = ws->clen[sym] + cl_extra(sym);
                }
                bitpos = pack(ws, bitpos, v, nb, lane);
                flush_some(ws, slot, bitpos, flushed, lane);
            }
        }
        flush(ws, slot, flushed, (bitpos + 31u) >> 5, lane);
        if (lane == 0) cs->head_bits = bitpos;
    }
    __syncthreads();
    const u32 bit = cs->head_bits;
    const bool dyn = ws->dynamic != 0;
    const u32 eob_bits = dyn ? ws->llen[256] : 7u;
    const u32 end = dyn ? emit<EMIT_DYNAMIC>(cs, p, len, slot, bit, eob_bits) : emit<EMIT_FIXED>(cs, p, len, slot, bit, eob_bits);
    if (tid == 0) {
        if (end) {
            BitRun run(slot, end);
            run.put(dyn ? ws->lcode[256] : 0u, eob_bits);
            run.done();
        }
        deflate_len[chunk] = end ? (end + eob_bits + 7u) >> 3 : kTooBig;
    }
}

// One CTA per block: the gzip header with the BC subfield, the body
// (deflated, stored or the empty stream) and CRC32 + ISIZE, at out_offsets[i].
__global__ void k_frame_blocks(const u8 *slots, const u32 *deflate_len, const u8 *data, const u64 *bounds,
                               const u32 *crcs, const u8 *framing, const u64 *out_offsets, u8 *out, u32 n)
{
    const u32 i = blockIdx.x;
    if (i >= n) return;
    u8 *b = out + out_offsets[i];
    const u32 size = (u32)(out_offsets[i + 1] - out_offsets[i]);
    const u32 raw = (u32)(bounds[i + 1] - bounds[i]);
    const u8 how = framing[i];
    if (threadIdx.x == 0) {
        const u8 h[16] = {0x1f, 0x8b, 8, 4, 0, 0, 0, 0, 0, 0xff, 6, 0, 'B', 'C', 2, 0};
        for (int k = 0; k < 16; ++k) b[k] = h[k];
        b[16] = (u8)((size - 1u) & 0xffu);
        b[17] = (u8)((size - 1u) >> 8);
        u8 *t = b + size - kTrailer;
        const u32 c = crcs[i];
        for (int k = 0; k < 4; ++k) t[k] = (u8)(c >> (8 * k));
        for (int k = 0; k < 4; ++k) t[4 + k] = (u8)(raw >> (8 * k));
        if (how == FRAMING_EMPTY) {
            b[kHeader] = 0x03;
            b[kHeader + 1] = 0x00;
        } else if (how == FRAMING_STORED) {
            u8 *s = b + kHeader;
            s[0] = 0x01; // BFINAL 1, BTYPE 00
            s[1] = (u8)(raw & 0xffu);
            s[2] = (u8)(raw >> 8);
            s[3] = (u8)(~raw & 0xffu);
            s[4] = (u8)((~raw >> 8) & 0xffu);
        }
    }
    if (how == FRAMING_DEFLATED) {
        const u8 *src = slots + (size_t)i * kSlot;
        const u32 dl = deflate_len[i];
        for (u32 k = threadIdx.x; k < dl; k += blockDim.x) b[kHeader + k] = src[k];
    } else if (how == FRAMING_STORED) {
        const u8 *src = data + bounds[i];
        for (u32 k = threadIdx.x; k < raw; k += blockDim.x) b[kHeader + kStoredHeader + k] = src[k];
    }
}

} // namespace

struct frt_compressor {
    int device = 0;
    SharedStream *shared = nullptr;
    cudaStream_t stream = nullptr;
    std::mutex mu;
};

extern "C" int frt_compressor_create(int device, void *stream, frt_compressor **out, frt_error *err)
{
    if (!out) return FRT_ERR_INVALID_ARGUMENT;
    int rc = check_device(device, err);
    if (rc) return rc;
    DeviceGuardLite g(device);
    configure_pool(device);
    SharedStream *ss = stream_create(device, stream, err);
    if (!ss) return FRT_ERR_CUDA;
    frt_compressor *c = new frt_compressor;
    c->device = device;
    c->shared = ss;
    c->stream = ss->s;
    *out = c;
    return FRT_OK;
}

extern "C" void frt_compressor_destroy(frt_compressor *c)
{
    if (!c) return;
    stream_release(c->shared);
    delete c;
}

extern "C" const char *frt_compressor_name(const frt_compressor *) { return "gb300-deflate"; }

extern "C" int frt_compressor_device_ordinal(const frt_compressor *c) { return c ? c->device : -1; }

// choose_framing (compress.rs:115-128) and framed_size (compress.rs:134-142).
extern "C" int frt_choose_framing(size_t payload_len, size_t deflate_len)
{
    if (payload_len == 0) return FRAMING_EMPTY;
    if (deflate_len > kMaxDeflate || deflate_len > payload_len + kStoredHeader) return FRAMING_STORED;
    return FRAMING_DEFLATED;
}

extern "C" size_t frt_framed_size(size_t payload_len, size_t deflate_len)
{
    const int how = frt_choose_framing(payload_len, deflate_len);
    const size_t body = how == FRAMING_DEFLATED ? deflate_len : how == FRAMING_STORED ? payload_len + kStoredHeader : 2;
    return kHeader + body + kTrailer;
}

extern "C" size_t frt_compress_bound(size_t n_chunks) { return n_chunks * (size_t)kMaxBlock; }

namespace {
constexpr int kShapes = 3;

template <class CS>
cudaError_t launch_shape(u32 n, const u8 *data, const u64 *bounds, const u32 *which, u8 *slots, u32 *len, u32 *crc, cudaStream_t st)
{
    const cudaError_t e = cudaFuncSetAttribute(k_deflate_chunks<CS>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(CS));
    if (e != cudaSuccess) return e;
    k_deflate_chunks<CS><<<n, CS::kThreads, sizeof(CS), st>>>(data, bounds, which, slots, len, crc);
    return cudaGetLastError();
}

cudaError_t launch_deflate(int shape, u32 n, const u8 *data, const u64 *bounds, const u32 *which, u8 *slots, u32 *len, u32 *crc,
                           cudaStream_t st)
{
    if (shape == 0) return launch_shape<Large>(n, data, bounds, which, slots, len, crc, st);
    if (shape == 1) return launch_shape<Medium>(n, data, bounds, which, slots, len, crc, st);
    return launch_shape<Small>(n, data, bounds, which, slots, len, crc, st);
}

// The chunks by shape (Large, Medium, Small), counts[] of each; an empty list
// where all are of one.
//
// A chunk of the Large shape has an SM to itself, the quickest for up to one a
// SM; more of them wait in line, and a short chunk spends most of its time in
// one warp's tree builder.  Four Medium CTAs or seven Small ones run side by
// side on an SM.  Measured through compress_batch_device, a warp per chunk /
// Large / Medium / Small, us:
//                    152 chunks           500               1,000                20,000
//     100 bytes  170 116 113 117   177 278 116 118    191  468 182 136    1676  7718 2112 1683
//   1,000        336 156 151 162   338 442 167 171    360  741 284 190    3230 12916 3758 2530
//   4,096       1075 207 209 244  1138 617 256 272   1175 1037 417 328   11273 18484 6184 4987
//   8,192       2244 237 271   -  2247 736 339   -   2452 1245 570   -    (5,000: 7786 5632 2345)
// so Medium from one chunk a SM on, Small from four.
std::vector<u32> by_shape(const uint64_t *bounds, size_t n, u32 counts[kShapes])
{
    int dev = 0, sms = 1;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    size_t up_to[kShapes] = {0, 0, 0}; // chunks that fit each shape and no smaller one
    auto smallest = [&](size_t i) {
        const u64 len = bounds[i + 1] - bounds[i];
        return len <= Small::kMax ? 2 : len <= Medium::kMax ? 1 : 0;
    };
    for (size_t i = 0; i < n; ++i) ++up_to[smallest(i)];
    const size_t wave = (size_t)sms, fit = up_to[1] + up_to[2];
    int shape_of[kShapes] = {0, 0, 0}; // of the chunks counted in up_to
    shape_of[2] = up_to[2] > 4 * wave ? 2 : fit > wave ? 1 : 0;
    shape_of[1] = (shape_of[2] == 2 ? up_to[1] : fit) > wave ? 1 : 0;
    counts[0] = counts[1] = counts[2] = 0;
    for (int k = 0; k < kShapes; ++k) counts[shape_of[k]] += (u32)up_to[k];
    std::vector<u32> which;
    if (counts[0] == n || counts[1] == n || counts[2] == n) return which;
    which.resize(n);
    u32 at[kShapes] = {0, counts[0], counts[0] + counts[1]};
    for (size_t i = 0; i < n; ++i) which[at[shape_of[smallest(i)]]++] = (u32)i;
    return which;
}
} // namespace

// DeviceBlockCompressor::compress_batch_device (device.rs:357-371): each
// range bounds[i]..bounds[i + 1] of the device bytes becomes one framed block,
// written to the host buffer `out` (out_offsets[i] .. out_offsets[i + 1]); no
// EOF block.  The ranges need not cover the buffer.
extern "C" int frt_compress_batch_device(frt_compressor *cp, const uint8_t *data, size_t data_len,
                                         const uint64_t *bounds, size_t n_bounds, uint8_t *out, size_t out_cap,
                                         uint64_t *out_offsets, size_t *out_len, frt_error *err)
{
    if (!cp || !bounds || n_bounds == 0 || (n_bounds > 1 && (!data || !out || !out_offsets))) {
        set_error(err, FRT_ERR_INVALID_ARGUMENT, 0, 0, 0, 0, nullptr, "null argument or no bounds");
        return FRT_ERR_INVALID_ARGUMENT;
    }
    const size_t n = n_bounds - 1;
    for (size_t i = 0; i < n; ++i) {
        if (bounds[i + 1] < bounds[i] || bounds[i + 1] > data_len || bounds[i + 1] - bounds[i] > kMaxPayload) {
            set_error(err, FRT_ERR_MALFORMED, 0, 0, 0, bounds[i], "bgzf",
                      "chunk %zu is [%llu, %llu): bounds must rise, stay within the %zu device bytes and hold at "
                      "most %u bytes",
                      i, (unsigned long long)bounds[i], (unsigned long long)bounds[i + 1], data_len, kMaxPayload);
            return FRT_ERR_MALFORMED;
        }
    }
    if (out_offsets) out_offsets[0] = 0;
    if (out_len) *out_len = 0;
    if (n == 0) return FRT_OK;
    if (n >= 0xffffffffull) {
        set_error(err, FRT_ERR_INVALID_ARGUMENT, 0, 0, 0, 0, nullptr, "too many chunks");
        return FRT_ERR_INVALID_ARGUMENT;
    }
    DeviceGuardLite g(cp->device);
    std::lock_guard<std::mutex> lk(cp->mu);
    cudaStream_t st = cp->stream;
    u32 counts[kShapes];
    const std::vector<u32> which = by_shape(bounds, n, counts);
    const size_t work = 8 * (n + 1) + 4 * n + 4 * n + 4 * which.size() + (size_t)kSlot * n;
    u8 *w = nullptr;
    int rc = dev_alloc((void **)&w, work + 64, st, err);
    if (rc) return rc;
    u64 *d_bounds = (u64 *)w;
    u32 *d_len = (u32 *)(w + 8 * (n + 1));
    u32 *d_crc = d_len + n;
    u32 *d_which = which.empty() ? nullptr : d_crc + n;
    u8 *d_slots = (u8 *)(d_crc + n + which.size());
    d_slots += (64 - ((uintptr_t)d_slots & 63)) & 63;
    std::vector<u32> lens(n);
    cudaError_t e;
    auto fail = [&](cudaError_t ce, const char *what) {
        dev_free(w, st);
        return cuda_fail(err, ce, what);
    };
    if ((e = cudaMemcpyAsync(d_bounds, bounds, 8 * (n + 1), cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return fail(e, "uploading the chunk bounds");
    if (d_which && (e = cudaMemcpyAsync(d_which, which.data(), 4 * which.size(), cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return fail(e, "uploading the chunks' shapes");
    u32 at = 0;
    for (int shape = 0; shape < kShapes; ++shape) {
        const u32 k = counts[shape];
        const u32 *list = d_which ? d_which + at : nullptr;
        if (k && (e = launch_deflate(shape, k, data, d_bounds, list, d_slots, d_len, d_crc, st)) != cudaSuccess)
            return fail(e, "launching the deflate");
        at += k;
    }
    if ((e = cudaMemcpyAsync(lens.data(), d_len, 4 * n, cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return fail(e, "reading the deflate sizes");
    // the framing and the dense layout, decided on the host as the reference does
    std::vector<u64> offs(n + 1, 0);
    std::vector<u8> framing(n);
    for (size_t i = 0; i < n; ++i) {
        const size_t raw = bounds[i + 1] - bounds[i];
        const size_t dl = lens[i] == kTooBig ? (size_t)kMaxDeflate + 1 : lens[i];
        framing[i] = (u8)frt_choose_framing(raw, dl);
        offs[i + 1] = offs[i] + frt_framed_size(raw, dl);
    }
    if (offs[n] > out_cap) {
        dev_free(w, st);
        set_error(err, FRT_ERR_INVALID_ARGUMENT, 0, offs[n], out_cap, 0, nullptr,
                  "the %zu framed blocks take %llu bytes; the output holds %zu", n, (unsigned long long)offs[n],
                  out_cap);
        return FRT_ERR_INVALID_ARGUMENT;
    }
    u8 *d_out = nullptr, *d_meta = nullptr;
    if ((rc = dev_alloc((void **)&d_out, offs[n] + 16, st, err)) ||
        (rc = dev_alloc((void **)&d_meta, 8 * (n + 1) + n + 16, st, err))) {
        dev_free(d_out, st);
        dev_free(w, st);
        return rc;
    }
    u64 *d_offs = (u64 *)d_meta;
    u8 *d_framing = d_meta + 8 * (n + 1);
    auto fail2 = [&](cudaError_t ce, const char *what) {
        dev_free(d_meta, st);
        dev_free(d_out, st);
        return fail(ce, what);
    };
    if ((e = cudaMemcpyAsync(d_offs, offs.data(), 8 * (n + 1), cudaMemcpyHostToDevice, st)) != cudaSuccess ||
        (e = cudaMemcpyAsync(d_framing, framing.data(), n, cudaMemcpyHostToDevice, st)) != cudaSuccess)
        return fail2(e, "uploading the framing");
    k_frame_blocks<<<(unsigned)n, 256, 0, st>>>(d_slots, d_len, data, d_bounds, d_crc, d_framing, d_offs, d_out,
                                                (u32)n);
    if ((e = cudaGetLastError()) != cudaSuccess) return fail2(e, "launching the framing");
    if ((e = cudaMemcpyAsync(out, d_out, offs[n], cudaMemcpyDeviceToHost, st)) != cudaSuccess ||
        (e = cudaStreamSynchronize(st)) != cudaSuccess)
        return fail2(e, "reading the blocks back");
    dev_free(d_meta, st);
    dev_free(d_out, st);
    dev_free(w, st);
    std::memcpy(out_offsets, offs.data(), 8 * (n + 1));
    if (out_len) *out_len = offs[n];
    return FRT_OK;
}

// ---- DeviceBgzfWriter (crates/fritillaria-bgzf/src/device_write.rs) ----------

namespace {
// The 28-byte BGZF end-of-file block (crates/fritillaria-bgzf/src/block.rs:40-43).
const uint8_t kEofBlock[28] = {0x1f, 0x8b, 8, 4, 0, 0, 0, 0, 0, 0xff, 6, 0, 'B', 'C', 2, 0,
                               0x1b, 0, 3, 0, 0, 0, 0, 0, 0, 0, 0, 0};
} // namespace

struct frt_bgzf_writer {
    frt_write_fn write = nullptr;
    void *ctx = nullptr;
    frt_compressor *compressor = nullptr;
    size_t chunks_per_batch = 1024; // DEFAULT_CHUNKS_PER_BATCH
    size_t payload_size = 65280;    // DEFAULT_PAYLOAD_SIZE
    uint64_t blocks = 0, batches = 0, compressed = 0, uncompressed = 0;
    bool finished = false;
    std::vector<uint8_t> buf;
    std::vector<uint64_t> offs;
};

extern "C" int frt_bgzf_writer_open(frt_write_fn write, void *ctx, frt_compressor *c, frt_bgzf_writer **out,
                                    frt_error *err)
{
    if (!write || !c || !out) {
        set_error(err, FRT_ERR_INVALID_ARGUMENT, 0, 0, 0, 0, nullptr, "null argument");
        return FRT_ERR_INVALID_ARGUMENT;
    }
    frt_bgzf_writer *w = new frt_bgzf_writer;
    w->write = write;
    w->ctx = ctx;
    w->compressor = c;
    *out = w;
    return FRT_OK;
}

extern "C" void frt_bgzf_writer_set_chunks_per_batch(frt_bgzf_writer *w, size_t chunks)
{
    if (w) w->chunks_per_batch = chunks ? chunks : 1;
}

extern "C" void frt_bgzf_writer_set_payload_size(frt_bgzf_writer *w, size_t size)
{
    if (w) w->payload_size = size < 1 ? 1 : (size > kMaxPayload ? kMaxPayload : size);
}

namespace {
int writer_emit(frt_bgzf_writer *w, const uint8_t *p, size_t n, frt_error *err)
{
    while (n) {
        const int64_t k = w->write(w->ctx, p, n);
        if (k <= 0) {
            set_error(err, FRT_ERR_IO, 0, 0, 0, 0, nullptr, "the sink refused %zu bytes", n);
            return FRT_ERR_IO;
        }
        p += k;
        n -= (size_t)k;
    }
    return FRT_OK;
}
} // namespace

// write_batch (device_write.rs:106-141): the chunks bounds[i]..bounds[i + 1]
// of the device bytes, compressed chunks_per_batch at a time and written out.
extern "C" int frt_bgzf_writer_write_batch(frt_bgzf_writer *w, const uint8_t *data, size_t len, const uint64_t *bounds,
                                           size_t n_bounds, frt_error *err)
{
    if (!w || (!bounds && n_bounds) || w->finished) {
        set_error(err, FRT_ERR_INVALID_ARGUMENT, 0, 0, 0, 0, nullptr, "null argument, or the writer is finished");
        return FRT_ERR_INVALID_ARGUMENT;
    }
    if (n_bounds == 0) {
        set_error(err, FRT_ERR_MALFORMED, 0, 0, 0, w->compressed, "bgzf", "bounds must have at least one entry");
        return FRT_ERR_MALFORMED;
    }
    if (bounds[n_bounds - 1] > len) {
        set_error(err, FRT_ERR_MALFORMED, 0, 0, 0, w->compressed, "bgzf", "bounds reach byte %llu of %zu device bytes",
                  (unsigned long long)bounds[n_bounds - 1], len);
        return FRT_ERR_MALFORMED;
    }
    size_t start = 0;
    while (start + 1 < n_bounds) {
        const size_t end = start + w->chunks_per_batch + 1 < n_bounds ? start + w->chunks_per_batch + 1 : n_bounds;
        const size_t k = end - start - 1;
        w->buf.resize(frt_compress_bound(k));
        w->offs.resize(k + 1);
        size_t got = 0;
        int rc = frt_compress_batch_device(w->compressor, data, len, bounds + start, end - start, w->buf.data(),
                                           w->buf.size(), w->offs.data(), &got, err);
        if (rc) return rc;
        if ((rc = writer_emit(w, w->buf.data(), got, err))) return rc;
        w->uncompressed += bounds[end - 1] - bounds[start];
        w->compressed += got;
        w->blocks += k;
        ++w->batches;
        start = end - 1;
    }
    return FRT_OK;
}

// The device bytes in payload_size chunks (the write path of a caller that
// holds one contiguous buffer).
extern "C" int frt_bgzf_writer_write_device(frt_bgzf_writer *w, const uint8_t *data, size_t len, frt_error *err)
{
    if (!w) return FRT_ERR_INVALID_ARGUMENT;
    std::vector<uint64_t> b(1, 0);
    for (size_t at = 0; at < len;) {
        at = at + w->payload_size < len ? at + w->payload_size : len;
        b.push_back(at);
    }
    return frt_bgzf_writer_write_batch(w, data, len, b.data(), b.size(), err);
}

// finish: the EOF block, once.
extern "C" int frt_bgzf_writer_finish(frt_bgzf_writer *w, frt_error *err)
{
    if (!w) return FRT_ERR_INVALID_ARGUMENT;
    if (w->finished) return FRT_OK;
    int rc = writer_emit(w, kEofBlock, sizeof kEofBlock, err);
    if (rc) return rc;
    w->compressed += sizeof kEofBlock;
    w->finished = true;
    return FRT_OK;
}

extern "C" void frt_bgzf_writer_stats(const frt_bgzf_writer *w, uint64_t *blocks, uint64_t *batches,
                                      uint64_t *compressed, uint64_t *uncompressed)
{
    if (!w) return;
    if (blocks) *blocks = w->blocks;
    if (batches) *batches = w->batches;
    if (compressed) *compressed = w->compressed;
    if (uncompressed) *uncompressed = w->uncompressed;
}

extern "C" void frt_bgzf_writer_destroy(frt_bgzf_writer *w) { delete w; }
